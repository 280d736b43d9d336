// gtb_seq_gemm_plan.h -- what the tensor-core kernels of the layer-list library share on the host: the tensor-map encoder and the status word.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>

namespace gtb {
namespace seq {

typedef CUresult (*PFN_tmapEncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                        const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                        CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

struct SeqGemmPlan {
    PFN_tmapEncodeTiled enc = nullptr;
    int* d_status = nullptr;
    bool attr[2][2][4] = {};
    bool sk_attr[3][4] = {};
};

}  // namespace seq
}  // namespace gtb
