"""What is timed: the calls that programs make of this framework, over the sizes that they make them with.

Two libraries, seven kinds of call:

  llama_decode   one row of the order-exact TinyLlama path behind a context (Engine.logits): the step of a chat
  llama_prefill  an exact prompt pass (Engine.prefill): the same bits as the reference's row loop
  llama_fast     the batched prompt pass on the tensor cores (Engine.prefill_fast), one layer and the head
  llama_batch    several sequences: exact prompts into slots, then shared decode steps (Engine.batch_*)
  prefill        layer-list models (SeqModel.step): prompts of one or several sequences, the logits of some positions
  mix            continuous batching: a step of prompts, a step of decode rows beside another prompt, a step of decode rows
  generate       greedy generation: prompts, device-side decode steps (SeqModel.decode), one more step for its logits

The families of the layer-list library are built at the layer sizes of their own benchmarks, scaled with the width:
"attention" = Vulosun's gated attention with a dense feed-forward, "reninex", "nanotar", "siladra"."""
import math
import random
import zlib

import numpy as np
import torch

import gtb  # noqa: F401  (registers tinyllama_cpp_b200)
from tinyllama_cpp_b200 import capi, nanotar, reninex, seq, siladra, vulosun
from tinyllama_cpp_b200 import weights as gten

LLAMA_DTYPES = {"f16": gten.F16, "q8": gten.Q8, "q4": gten.Q4}
LLAMA_KINDS = ("llama_decode", "llama_prefill", "llama_fast", "llama_batch")


def listed():
    return [
        # chat with the 1.1 B Q4 model near the end of its context: the latency of one exact token
        {"name": "llama_q4_decode", "kind": "llama_decode", "dtype": "q4", "layers": 22, "n": 1999},
        # a medium prompt of the same model, with the reference's own bits
        {"name": "llama_q4_prefill", "kind": "llama_prefill", "dtype": "q4", "layers": 22, "n": 511},
        # a full-context prompt of the Q8 model where tolerance-level parity is enough
        {"name": "llama_q8_fast_prefill", "kind": "llama_fast", "dtype": "q8", "layers": 1, "n": 2047},
        # a small batch job on the Q4 model: ragged short prompts, then shared steps
        {"name": "llama_q4_batch", "kind": "llama_batch", "dtype": "q4", "layers": 22, "lens": "40,17,33,8,25,39,12,30", "new": 12},
        # an ordinary prompt through attention layers with a dense feed-forward
        {"name": "attention_prefill", "kind": "prefill", "family": "attention", "width": 2048, "layers": 2, "vocab": 2048, "dtype": "bf16", "lens": "2048"},
        # a long document, in passes of 2048 rows: attention over a long context
        {"name": "attention_long", "kind": "prefill", "family": "attention", "width": 1024, "layers": 1, "vocab": 2048, "dtype": "bf16", "lens": "8001"},
        # sigmoid attention beside retention, full prompt
        {"name": "reninex_prefill", "kind": "prefill", "family": "reninex", "width": 2048, "layers": 2, "vocab": 2048, "dtype": "bf16", "lens": "2048"},
        # the float32 mode, which users take to check a model: a paragraph
        {"name": "reninex_f32", "kind": "prefill", "family": "reninex", "width": 1024, "layers": 2, "vocab": 2048, "dtype": "f32", "lens": "300"},
        # a whole recurrent model (mLSTM, attention beside a selective scan, delta rule, experts) on a full prompt
        {"name": "siladra_prefill", "kind": "prefill", "family": "siladra", "width": 2048, "layers": 3, "vocab": 32000, "dtype": "bf16", "lens": "2048"},
        # what a server's scheduler does: ragged prompts, decode rows beside a new prompt, latent attention
        {"name": "nanotar_mix", "kind": "mix", "family": "nanotar", "width": 2048, "layers": 2, "vocab": 2048, "dtype": "bf16", "lens": "731,402,65", "more": 333},
        # the smallest request: a short question, a short answer, one sequence
        {"name": "attention_generate", "kind": "generate", "family": "attention", "width": 1024, "layers": 4, "vocab": 32000, "dtype": "bf16", "lens": "37", "new": 16},
        # a busy server: 24 sequences decode together
        {"name": "siladra_generate_24", "kind": "generate", "family": "siladra", "width": 1024, "layers": 3, "vocab": 8192, "dtype": "bf16",
         "lens": ",".join(str(16 + 7 * i) for i in range(24)), "new": 12},
    ]


def draw(rng: random.Random):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(("llama_decode", "llama_prefill", "llama_fast", "llama_batch", "prefill", "prefill", "prefill", "mix", "generate", "generate"))
    if kind == "llama_decode":
        return {"kind": kind, "dtype": rng.choice(("q4", "q8", "f16")), "layers": rng.choice((6, 22)), "n": log(32, 2040)}
    if kind == "llama_prefill":
        return {"kind": kind, "dtype": rng.choice(("q4", "q8")), "layers": rng.choice((6, 12)), "n": log(48, 900)}
    if kind == "llama_fast":
        return {"kind": kind, "dtype": rng.choice(("q4", "q8", "f16")), "layers": 1, "n": log(64, 2047)}
    if kind == "llama_batch":
        n = rng.randint(2, 12)
        return {"kind": kind, "dtype": rng.choice(("q4", "q8")), "layers": rng.choice((4, 8)), "lens": ",".join(str(log(6, 40)) for _ in range(n)), "new": rng.randint(3, 12)}
    family, width = rng.choice(("attention", "reninex", "nanotar", "siladra")), rng.choice((1024, 1280, 1536, 2048))
    c = {"kind": kind, "family": family, "width": width, "layers": 3 if family == "siladra" else 2, "vocab": rng.choice((2048, 5003)), "dtype": "bf16"}
    if kind == "prefill":
        if rng.random() < 0.2:
            c.update(dtype="f32", width=1024, lens=str(log(20, 300)))
        else:
            c["lens"] = ",".join(str(log(20, 3000 if s == 0 else 500)) for s in range(rng.choice((1, 1, 2, 4))))
    elif kind == "mix":
        c.update(lens=",".join(str(log(10, 800)) for _ in range(rng.randint(1, 4))), more=log(10, 500))
    else:
        c.update(lens=",".join(str(log(8, 400)) for _ in range(log(1, 32))), new=rng.randint(4, 14))
    return c


# ------------------------------------------------------------------------------------------------ inputs
def generator(seed, name):
    g = torch.Generator(device="cuda")
    g.manual_seed((seed * 1000003 + zlib.crc32(name.encode())) & 0x7FFFFFFF)
    return g


def lens_of(case):
    return [int(n) for n in case["lens"].split(",")]


def tokens_of(seed, name, n, vocab):
    return torch.randint(0, vocab, (n,), generator=generator(seed, name), device="cuda").cpu().numpy().astype(np.int32)


def llama_config(case):
    return gten.ModelConfig(n_layers=case["layers"])


def llama_payload(seed, dtype, layer, tid, rows, cols):
    """The bytes of one tensor of a checkpoint, on the GPU: Gaussian weights in the converter's block formats."""
    x = torch.randn(rows, cols, generator=generator(seed, f"{layer}.{tid}"), device="cuda")
    if gten.is_norm(tid):
        return (1.0 + 0.1 * x).half().view(torch.uint8).reshape(-1)
    x = 0.02 * x
    if dtype == gten.F16:
        return x.half().view(torch.uint8).reshape(-1)
    x = x.reshape(-1, 32)
    step = x.abs().amax(1, keepdim=True) / (127.0 if dtype == gten.Q8 else 7.0)
    q = torch.round(x / step).to(torch.int16)
    if dtype == gten.Q8:
        codes = (q & 255).to(torch.uint8)
    else:
        codes = (((q[:, :16] + 7) << 4) | (q[:, 16:] + 7)).to(torch.uint8)
    return torch.cat([step.half().view(torch.uint8).reshape(-1, 2), codes], 1).reshape(-1)


def llama_dequant(payload, dtype, tid, rows, cols):
    if gten.is_norm(tid) or dtype == gten.F16:
        return payload.view(torch.float16).double().reshape(rows, cols)
    b = payload.reshape(-1, 34 if dtype == gten.Q8 else 18)
    step = b[:, :2].contiguous().view(torch.float16).double()
    if dtype == gten.Q8:
        return (b[:, 2:].contiguous().view(torch.int8).double() * step).reshape(rows, cols)
    return (torch.cat([(b[:, 2:] >> 4).double() - 7, (b[:, 2:] & 15).double() - 7], 1) * step).reshape(rows, cols)


def family_config(case):
    W, n, V = case["width"], case["layers"], case["vocab"]
    f = case["family"]
    if f == "attention":
        lay = vulosun.gated_attention_layer(heads=W // 64, kv_heads=4, dim=64, vdim=64, rot_dims=64, rot_base=250000.0, mlp=vulosun.dense_mlp(11 * W // 4))
        return vulosun, vulosun.make_config(vocab=V, width=W, layers=[lay] * n, eps=1e-6)
    if f == "reninex":
        return reninex, reninex.make_config(vocab=V, width=W, n_layers=n, ff=11 * W // 4, taps=4, l_heads=W // 64, l_kv=4, l_dim=64, l_vdim=64, r_heads=W // 128, r_dim=128,
                                            r_vdim=128, rot_dims=64, bigram=(4093, 31, 17), loop=None)
    if f == "nanotar":
        att = dict(heads=W // 128, dim=96, rot_dim=32, vdim=128, kv_rank=W // 4, rot_base=500000.0)
        lays = [nanotar.latent_layer(mlp=nanotar.dense_mlp(11 * W // 4), **att),
                nanotar.latent_layer(q_rank=3 * W // 8, window=W // 2, mlp=nanotar.moe_mlp(experts=16, top=2, ff=11 * W // 16, shared_ff=11 * W // 16), **att)]
        return nanotar, nanotar.make_config(vocab=V, width=W, streams=2, layers=[lays[i % 2] for i in range(n)], eps=1e-6, logit_softcap=30.0)
    moe = siladra.moe_mlp(ff=11 * W // 16, experts=16, top=2)
    lays = [siladra.mlstm_layer(heads=W // 256, dim=128, vdim=256, gate_cap=15.0, mlp=moe),
            siladra.parallel_layer(heads=W // 128, kv_heads=4 if W % 512 == 0 else 2, dim=64, vdim=64, rot_dims=64, rot_base=10000.0, yarn=(8.0, 4096.0, 32.0, 1.0),
                                   inner=2 * W, state=16, dt_rank=W // 16, conv=4, mlp=moe),
            siladra.delta_layer(heads=W // 128, kv_heads=W // 256, dim=128, vdim=128, conv=4, mlp=moe)]
    return siladra, siladra.make_config(vocab=V, width=W, layers=[lays[i % 3] for i in range(n)], eps=1e-6, embed_scale=float(W) ** 0.5)


def tensor(case, seed, name, shape, scale):
    """One tensor of a checkpoint as bfloat16 on the GPU.  Token t's embedding carries the directions of two experts and the head
    carries the embedding of the token before: routing and greedy choices are as decided as those of a trained model."""
    W = case["width"]
    g = generator(seed, name)
    normal = lambda s: torch.randn(s, generator=g, device="cuda")
    uniform = lambda lo, hi: lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda")
    leaf = name.split(".")[-1]
    last = shape[-1] if shape else 1
    signs = lambda: torch.sign(torch.randn((16, W), generator=generator(seed, "experts"), device="cuda"))
    if name in ("embed", "head"):
        a = torch.randn(shape, generator=generator(seed, "embed"), device="cuda")
        if case["family"] in ("nanotar", "siladra"):
            t, d = torch.arange(shape[0], device="cuda"), signs()
            a += 0.6 * d[t % 16] + 0.45 * d[(5 * t + 3 + t // 16) % 16]
        a = a / scale if name == "embed" else normal(shape) / W ** 0.5 + torch.roll(a, 1, 0) * (40.0 / W)
    elif leaf == "router":
        a = signs() * (0.5 / W ** 0.5)
    elif leaf == "alpha":
        a = uniform(0.4, 0.6)
    elif ".hc" in name:
        S = last
        a = {"in": torch.full(shape, 1.0 / S), "out": torch.ones(shape), "mix": torch.eye(S).reshape(shape) if leaf == "mix" else None}[leaf].cuda() + 0.1 * normal(shape)
    elif leaf == "b" and len(shape) == 1:
        a = uniform(1.0, 5.0) if name.endswith(".f.b") else uniform(-4.5, -1.0) if name.endswith(".dt.b") else 0.1 * normal(shape)
    elif leaf.startswith("norm") or leaf == "out":
        a = 1.0 + 0.1 * normal(shape)
    elif leaf in ("sink", "pb"):
        a = normal(shape) - (1.0 if leaf == "pb" else 0.0)
    elif leaf.startswith("canon"):
        a = 0.3 * normal(shape)
    elif leaf == "conv":
        a = 0.4 * normal(shape)
        a[:, -1] += 0.8
    elif leaf == "A_log":
        a = torch.log(torch.arange(1, last + 1, device="cuda").float()) + 0.1 * normal(shape) if len(shape) == 2 else uniform(-1.0, 1.5)
    elif leaf == "dt_bias":
        a = uniform(-5.0, -1.0)
    elif leaf == "D":
        a = 1.0 + 0.2 * normal(shape)
    else:
        a = normal(shape) / (1.0 if name == "bigram" else last ** 0.5)
    return a.to(torch.bfloat16)


def prepare(case, seed):
    if case["kind"] in LLAMA_KINDS:
        capi.init(0)
        cfg, dt = llama_config(case), LLAMA_DTYPES[case["dtype"]]
        e = capi.Engine(cfg, 2048, dt)
        for layer, tid, _, rows, cols in gten.tensor_list(cfg):
            e.set_weight(layer, tid, llama_payload(seed, dt, layer, tid, rows, cols).cpu().numpy())
        st = {"case": case, "engine": e}
        if case["kind"] == "llama_batch":
            st["prompts"] = [tokens_of(seed, f"prompt{i}", n, 32000) for i, n in enumerate(lens_of(case))]
            e.batch_create(len(st["prompts"]))
        else:
            st["tokens"] = tokens_of(seed, "prompt", case["n"], 32000)
            if case["kind"] == "llama_decode":
                e.prefill(st["tokens"][:-1])
        return st
    seq.init(0)
    fam, cfg = family_config(case)
    desc = fam.describe(cfg)
    lens = lens_of(case) + ([case["more"]] if "more" in case else [])
    m = seq.SeqModel(desc, seq.F32 if case["dtype"] == "f32" else seq.BF16, len(lens), max(lens) + 64, max_rows=2048)
    scale = desc.get("embed_scale", 1.0)
    m.load({k: tensor(case, seed, k, s, scale).view(torch.int16).cpu().numpy().view(np.uint16) for k, s in fam.tensor_shapes(desc).items()})
    return {"case": case, "model": m, "prompts": [tokens_of(seed, f"prompt{i}", n, case["vocab"]) for i, n in enumerate(lens)], "fed": tokens_of(seed, "fed", 2 * len(lens), case["vocab"])}


# ------------------------------------------------------------------------------------------------ one pass
def wanted(total):
    """16 positions of a step spread over its rows, the last one among them."""
    return sorted({(i * (total - 1)) // 15 for i in range(16)})


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "llama_decode":
        return st["engine"].logits(st["tokens"], case["n"] - 1)
    if kind == "llama_prefill":
        st["engine"].prefill(st["tokens"])
        return {"logits": st["engine"].read_logits(), "next": st["engine"].read_tokens(case["n"], 1)}
    if kind == "llama_fast":
        st["engine"].prefill_fast(st["tokens"])
        return st["engine"].read_logits()
    if kind == "llama_batch":
        e = st["engine"]
        for s, p in enumerate(st["prompts"]):
            e.batch_prefill(s, p)
        e.batch_decode(case["new"])
        return {"tokens": [e.batch_read_tokens(s, len(p), case["new"] + 1) for s, p in enumerate(st["prompts"])],
                "logits": np.stack([e.batch_read_logits(s) for s in range(len(st["prompts"]))])}
    m, prompts, n = st["model"], st["prompts"], len(st["prompts"])
    for s in range(n):
        m.reset(s)
    if kind == "prefill":
        return m.step(list(enumerate(prompts)), wanted(sum(len(p) for p in prompts)))
    if kind == "mix":
        ends = np.cumsum([len(p) for p in prompts[:-1]]) - 1
        one = m.step(list(enumerate(prompts[:-1])), ends)
        rows = [(s, [t]) for s, t in enumerate(st["fed"][:n - 1])]
        two = m.step(rows + [(n - 1, prompts[-1])], list(range(n - 1)) + [n - 2 + len(prompts[-1])])
        return [one, two, m.step([(s, [t]) for s, t in enumerate(st["fed"][n:2 * n])], range(n))]
    first = m.step_greedy(list(enumerate(prompts)))
    toks = m.decode(range(n), case["new"])
    return {"first": first, "tokens": toks, "logits": m.step([(s, [t]) for s, t in enumerate(toks[:, -1])], range(n))}


# ------------------------------------------------------------------------------------------------ what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind in LLAMA_KINDS:
        cfg, dt = llama_config(case), LLAMA_DTYPES[case["dtype"]]
        per_layer = 2 * cfg.n_embd * (cfg.n_embd + cfg.kv_dim) + 3 * cfg.n_embd * cfg.n_ffn
        head = cfg.n_vocab * cfg.n_embd
        kv, wb, att = cfg.kv_bytes_per_pos(dt), cfg.weight_bytes_per_token(dt) + cfg.norm_bytes_per_token(), 4.0 * cfg.n_embd * cfg.n_layers
        if kind == "llama_decode":
            return {"bytes": wb + kv * case["n"] + 4 * cfg.n_vocab, "flops": 2.0 * (per_layer * cfg.n_layers + head) + att * case["n"]}
        if kind != "llama_batch":
            n = case["n"]
            return {"bytes": wb + kv * n + 4 * cfg.n_vocab, "flops": 2.0 * (per_layer * cfg.n_layers * n + head) + att * n * (n + 1) / 2}
        lens, new = lens_of(case), case["new"]
        rows = sum(lens) + new * len(lens)
        return {"bytes": (len(lens) + new) * wb + kv * sum(new * n + n for n in lens) + 4 * cfg.n_vocab * len(lens),
                "flops": 2.0 * (per_layer * cfg.n_layers * rows + head * (new + 1) * len(lens)) + att * sum((n + new) * (n + new + 1) / 2 for n in lens)}
    fam, cfg = family_config(case)
    desc = fam.describe(cfg)
    el, W, V = (4 if case["dtype"] == "f32" else 2), case["width"], case["vocab"]
    shapes = fam.tensor_shapes(desc)
    expert = sum(math.prod(s) for k, s in shapes.items() if ".mlp.e" in k)
    dense = sum(math.prod(s) for k, s in shapes.items() if len(s) == 2 and k not in ("embed", "bigram", "head") and ".mlp.e" not in k)

    def step(rows, outs, ctx):        # rows of one step, rows with logits, keys seen by all rows together
        touched = min(1.0, rows * 2 / 16)                                    # experts that the rows reach
        by = 2 * (dense + expert * touched + (V * W if outs else 0)) + el * W * rows + 4 * V * outs
        fl = 2.0 * (dense + expert * 2 / 16) * rows + 2.0 * V * W * outs
        for l in desc["layers"]:
            for b in l["branches"]:
                if b["kind"] in (seq.MIX_SIGMOID_ATTN, seq.MIX_SOFTMAX_ATTN, seq.MIX_LATENT_ATTN):
                    fl += 2.0 * b["heads"] * (b["dim"] + b.get("rope_dim", 0) + b["vdim"]) * ctx
                elif b["kind"] == seq.MIX_SSM:
                    fl += 6.0 * b["inner"] * b["state"] * rows
                else:
                    fl += (6.0 if b["kind"] == seq.MIX_DELTA else 4.0) * b["heads"] * b["dim"] * b["vdim"] * rows
        return by, fl
    lens = lens_of(case)
    tri = lambda n: n * (n + 1) / 2
    if kind == "prefill":
        parts = [step(sum(lens), 16, sum(map(tri, lens)))]
    elif kind == "mix":
        parts = [step(sum(lens), len(lens), sum(map(tri, lens))), step(len(lens) + case["more"], len(lens) + 1, sum(lens) + tri(case["more"])),
                 step(len(lens) + 1, len(lens) + 1, sum(lens) + case["more"])]
    else:
        parts = [step(sum(lens), len(lens), sum(map(tri, lens)))] + [step(len(lens), len(lens), sum(lens) + i * len(lens)) for i in range(case["new"] + 1)]
    return {"bytes": sum(p[0] for p in parts), "flops": sum(p[1] for p in parts)}


def tolerance(case):
    # the order-exact path of TinyLlama is defined bit by bit
    if case["kind"] in ("llama_decode", "llama_prefill", "llama_batch"):
        return "exact"
    # every operation re-encodes its row as Q8 blocks or halves: a last-bit difference becomes a step of a code
    if case["kind"] == "llama_fast":
        return {"rel": 0.03 if case["dtype"] != "f16" else 0.01}
    if case["dtype"] == "f32":
        return {"rel": 1e-5}
    # bf16 operands through two to four layers; greedy tokens are whole values
    return {"rel": 0.02, "differ": 0.01}


# ------------------------------------------------------------------------------------------------ the same in 64 bits
def rms(x, eps, w=1.0):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps) * w


def layer_norm(x, w, b, eps):
    x = x - x.mean(-1, keepdim=True)
    return rms(x, eps, w) + b


def silu(z):
    return z * torch.sigmoid(z)


def gelu_tanh(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def turn(x, freqs, pairs, amp=1.0):
    """Rotary positions on [T, heads, n]: pairs (2i, 2i + 1) or (i, i + len(freqs))."""
    half = len(freqs)
    f = torch.as_tensor(freqs, device=x.device, dtype=torch.float64)
    ang = torch.arange(x.shape[0], device=x.device, dtype=torch.float64)[:, None] * f
    c, s = torch.cos(ang)[:, None] * amp, torch.sin(ang)[:, None] * amp
    u, w = (x[..., 0:2 * half:2], x[..., 1:2 * half:2]) if pairs else (x[..., :half], x[..., half:2 * half])
    a, b = u * c - w * s, w * c + u * s
    return torch.cat([torch.stack([a, b], -1).flatten(-2) if pairs else torch.cat([a, b], -1), x[..., 2 * half:]], -1)


def freqs(dims, base):
    return [base ** (-2.0 * i / dims) for i in range(dims // 2)]


def causal(T, window=0):
    i = torch.arange(T, device="cuda")
    see = i[:, None] >= i[None]
    return see & (i[:, None] - i[None] < window) if window else see


def softmax_heads(q, k, v, scale, see, sink=None):
    """q [T, H, d], k [T, G, d], v [T, G, e] -> [T, H, e]"""
    out = []
    per = q.shape[1] // k.shape[1]
    for h in range(q.shape[1]):
        s = (q[:, h] @ k[:, h // per].T * scale).masked_fill(~see, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].expand(s.shape[0], 1)], 1)
        out.append(torch.softmax(s, 1)[:, :v.shape[0]] @ v[:, h // per])
    return torch.stack(out, 1)


def conv(u, w):
    y = torch.zeros_like(u)
    taps = w.shape[1]
    for j in range(taps):
        back = taps - 1 - j
        y[back:] += w[:, j] * u[:u.shape[0] - back]
    return y


def attention_model(c, P, x):
    eps, m = 1e-6, c["layers"][0]["mixer"]
    H, G, D = m["heads"], m["kv_heads"], m["dim"]
    ln = lambda v, n: layer_norm(v, P(n), P(n + ".b"), eps)
    T, see, fr = x.shape[0], causal(x.shape[0]), freqs(m["rot"]["dims"], m["rot"]["base"])
    for i in range(len(c["layers"])):
        p = f"l{i}."
        h = ln(x, p + "norm1")
        q = turn(rms(h @ P(p + "mix.q").T, eps, P(p + "mix.q.norm")).reshape(T, H, D), fr, True)
        k = turn(rms(h @ P(p + "mix.k").T, eps, P(p + "mix.k.norm")).reshape(T, G, D), fr, True)
        o = softmax_heads(q, k, (h @ P(p + "mix.v").T).reshape(T, G, D), m["scale"], see) * torch.sigmoid(h @ P(p + "mix.g").T)[..., None]
        x = x + ln(o.reshape(T, H * D) @ P(p + "mix.o").T, p + "norm1b")
        h = ln(x, p + "norm2")
        x = x + ln((silu(h @ P(p + "mlp.gate").T) * (h @ P(p + "mlp.up").T)) @ P(p + "mlp.down").T, p + "norm2b")
    return ln(x, "final.norm")


def reninex_model(c, P, x):
    eps, m = c["norm"]["eps"], c["layers"][0]["mixer"]
    le, ri, T, see = m["left"], m["right"], x.shape[0], causal(x.shape[0])
    for i in range(len(c["layers"])):
        p = f"l{i}."
        h = rms(x, eps, P(p + "norm1"))
        a, f = h + conv(h, P(p + "canon1")), h + conv(h, P(p + "canon2"))
        w = lambda t: P(p + "mix." + t)
        q = rms((a @ w("left.q").T).reshape(T, le["heads"], -1), eps)
        k = rms((a @ w("left.k").T).reshape(T, le["kv_heads"], -1), eps)
        v = (a @ w("left.v").T).reshape(T, le["kv_heads"], -1)
        per = le["heads"] // le["kv_heads"]
        att = torch.stack([(torch.sigmoid(q[:, g] @ k[:, g // per].T * le["scale"] + w("left.pb")[g]) * see) @ v[:, g // per] for g in range(le["heads"])], 1)
        H, D, fr = ri["heads"], ri["dim"], freqs(ri["rot"]["dims"], ri["rot"]["base"])
        q = turn((a @ w("right.q").T).reshape(T, H, D), fr, False)
        k = turn((a @ w("right.k").T).reshape(T, H, D), fr, False) * D ** -0.5
        v, dec = (a @ w("right.v").T).reshape(T, H, -1), torch.as_tensor(ri["decay"], device="cuda").double()
        gap = (torch.arange(T, device="cuda")[:, None] - torch.arange(T, device="cuda")[None]).clamp(min=0).double()
        ret = torch.stack([((q[:, g] @ k[:, g].T) * dec[g] ** gap * see) @ v[:, g] for g in range(H)], 1)
        y = m["left_scale"] * att.reshape(T, -1) @ w("left.o").T + m["right_scale"] * (rms(ret, eps).reshape(T, -1) * silu(a @ w("right.g").T)) @ w("right.o").T
        x = x + y + (gelu_tanh(f @ P(p + "mlp.gate").T) * (f @ P(p + "mlp.up").T)) @ P(p + "mlp.down").T
    return rms(x, eps, P("final.norm"))


def experts(h, P, p, top, softmax):
    s = h @ P(p + "router").T
    if not softmax:
        s = torch.sigmoid(s)
    w, idx = torch.topk(s, top, 1)
    w = torch.softmax(w, 1) if softmax else w / (w.sum(1, keepdim=True) + 1e-20)
    out = torch.zeros_like(h)
    for e in range(s.shape[1]):
        r, j = torch.where(idx == e)
        if len(r):
            out[r] += w[r, j, None] * ((silu(h[r] @ P(f"{p}e{e}.gate").T) * (h[r] @ P(f"{p}e{e}.up").T)) @ P(f"{p}e{e}.down").T)
    return out


def nanotar_model(c, P, x):
    eps, T = c["norm"]["eps"], x.shape[0]
    dyt = lambda v, n: torch.tanh(P(n + ".alpha") * v) * P(n) + P(n + ".b")
    xs = torch.stack([x] * c["streams"])

    def sub(xs, hc, f):
        y = f(torch.einsum("s,stw->tw", P(hc + ".in"), xs))
        return torch.einsum("sr,stw->rtw", P(hc + ".mix"), xs) + P(hc + ".out")[:, None, None] * y
    for i, lay in enumerate(c["layers"]):
        p, m = f"l{i}.", lay["mixer"]
        w = lambda t: P(p + "mix." + t)

        def latent(u):
            h, H, dn, dr, rank = dyt(u, p + "norm1"), m["heads"], m["dim"], m["rot_dim"], m["kv_rank"]
            q = (rms(h @ w("dq").T, eps, w("dq.norm")) @ w("uq").T if "q_rank" in m else h @ w("q").T).reshape(T, H, dn + dr)
            dkv, fr = h @ w("dkv").T, freqs(m["rot"]["dims"], m["rot"]["base"])
            lat = rms(dkv[:, :rank], eps, w("dkv.norm"))
            kr = turn(dkv[:, None, rank:], fr, True).expand(T, H, dr)
            q = torch.cat([q[..., :dn], turn(q[..., dn:], fr, True)], -1)
            k = torch.cat([(lat @ w("uk").T).reshape(T, H, dn), kr], -1)
            o = softmax_heads(q, k, (lat @ w("uv").T).reshape(T, H, -1), m["scale"], causal(T, (m.get("mask") or {}).get("size", 0)), w("sink") if "q_rank" in m else None)
            return (o * torch.sigmoid(h @ w("g").T)[..., None]).reshape(T, -1) @ w("o").T

        def ff(u):
            h, q = dyt(u, p + "norm2"), p + "mlp."
            if lay["mlp"]["kind"] == "dense":
                return (gelu_tanh(h @ P(q + "gate").T) * (h @ P(q + "up").T)) @ P(q + "down").T
            sh = (silu(h @ P(q + "shared.gate").T) * (h @ P(q + "shared.up").T)) @ P(q + "shared.down").T
            return experts(h, P, q, 2, False) + torch.sigmoid(h @ P(q + "shared.sg").T) * sh
        xs = sub(xs, p + "hc1", latent)
        xs = sub(xs, p + "hc2", ff)
    return dyt(xs.sum(0), "final.norm")


def siladra_model(c, P, x):
    eps, T = c["norm"]["eps"], x.shape[0]

    def mlstm(h, w, m):
        H, cap = m["heads"], m["gate_cap"]
        q, k, v = ((h @ w(t).T).reshape(T, H, -1) for t in "qkv")
        q = q * m["dim"] ** -0.5
        soft = lambda z: cap * torch.tanh(z / cap)
        i, f = soft(h @ w("i").T + w("i.b")), torch.nn.functional.logsigmoid(soft(h @ w("f").T + w("f.b")))
        S, n, r, out = torch.zeros(H, m["dim"], m["vdim"] + 1, device="cuda").double(), None, torch.zeros(H, device="cuda").double(), []
        v = torch.cat([v, torch.ones(T, H, 1, device="cuda").double()], -1)
        for t in range(T):
            new = torch.maximum(f[t] + r, i[t])
            S = torch.exp(f[t] + r - new)[:, None, None] * S + (torch.exp(i[t] - new)[:, None] * k[t])[..., None] * v[t][:, None]
            r = new
            o = torch.einsum("hdv,hd->hv", S, q[t])
            out.append(o[:, :-1] / (torch.maximum(o[:, -1].abs(), torch.exp(-r)) + 1e-6)[:, None])
        return rms(torch.stack(out), eps).reshape(T, -1) * w("norm") * torch.sigmoid(h @ w("g").T) @ w("o").T

    def delta(h, w, m):
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k, v = (silu(conv(h @ w(t).T, w(t + ".conv"))) for t in "qkv")
        unit = lambda z: z / torch.sqrt((z * z).sum(-1, keepdim=True) + 1e-6)
        wide = lambda z: unit(z.reshape(T, G, D)).repeat_interleave(H // G, 1)
        q, k, v = wide(q) * D ** -0.5, wide(k), v.reshape(T, H, -1)
        beta, g = torch.sigmoid(h @ w("b").T), torch.exp(-torch.exp(w("A_log")) * torch.nn.functional.softplus(h @ w("a").T + w("dt_bias")))
        S, out = torch.zeros(H, D, m["vdim"], device="cuda").double(), []
        for t in range(T):
            S = g[t][:, None, None] * S
            S = S + k[t][..., None] * (beta[t][:, None] * (v[t] - torch.einsum("hdv,hd->hv", S, k[t])))[:, None]
            out.append(torch.einsum("hdv,hd->hv", S, q[t]))
        return (rms(torch.stack(out), eps, w("norm")) * silu(h @ w("g").T).reshape(T, H, -1)).reshape(T, -1) @ w("o").T

    def left(h, w, m):
        H, G, D = m["heads"], m["kv_heads"], m["dim"]
        q, k = rms((h @ w("q").T + w("q.b")).reshape(T, H, D), eps, w("q.norm")), rms((h @ w("k").T + w("k.b")).reshape(T, G, D), eps, w("k.norm"))
        sc, n, base = m["rot"]["scaling"], m["rot"]["dims"], m["rot"]["base"]
        at = lambda turns: n * math.log(sc["original"] / (2.0 * math.pi * turns)) / (2.0 * math.log(base))
        lo, hi = max(math.floor(at(sc["fast"])), 0), min(math.ceil(at(sc["slow"])), n - 1)
        ramp = [min(1.0, max(0.0, (j - lo) / max(hi - lo, 0.001))) for j in range(n // 2)]
        fr, amp = [f / sc["factor"] * r + f * (1.0 - r) for f, r in zip(freqs(n, base), ramp)], 0.1 * math.log(sc["factor"]) + 1.0
        o = softmax_heads(turn(q, fr, True, amp), turn(k, fr, True, amp), (h @ w("v").T + w("v.b")).reshape(T, G, -1), m["scale"], causal(T))
        return o.reshape(T, -1) @ w("o").T

    def right(h, w, m):
        n, N, rank = m["inner"], m["state"], m["dt_rank"]
        xz = h @ w("in").T
        u, z = silu(conv(xz[:, :n], w("conv")) + w("conv.b")), xz[:, n:]
        d = u @ w("x").T
        dt, A = torch.nn.functional.softplus(d[:, :rank] @ w("dt").T + w("dt.b")), -torch.exp(w("A_log"))
        S, out = torch.zeros(n, N, device="cuda").double(), []
        for t in range(T):
            S = torch.exp(dt[t][:, None] * A) * S + (dt[t] * u[t])[:, None] * d[t, rank:rank + N]
            out.append(S @ d[t, rank + N:] + w("D") * u[t])
        return torch.stack(out) * silu(z) @ w("o").T
    for i, lay in enumerate(c["layers"]):
        p, m = f"l{i}.", lay["mixer"]
        w = lambda t: P(p + "mix." + t)
        h = rms(x, eps, P(p + "norm1"))
        if lay["type"] == "mlstm":
            y = mlstm(h, w, m)
        elif lay["type"] == "delta":
            y = delta(h, w, m)
        else:
            y = 0.5 * (rms(left(h, lambda t: w("left." + t), m["left"]), eps, w("left.out")) + rms(right(h, lambda t: w("right." + t), m["right"]), eps, w("right.out")))
        x = x + rms(y, eps, P(p + "norm1b"))
        x = x + rms(experts(rms(x, eps, P(p + "norm2")), P, p + "mlp.", 2, True), eps, P(p + "norm2b"))
    return rms(x, eps, P("final.norm"))


MODELS = {"attention": attention_model, "reninex": reninex_model, "nanotar": nanotar_model, "siladra": siladra_model}


def llama_exact(case, seed):
    """One layer and the head of the Q8 / FP16 activations' arithmetic: 64-bit sums between the re-encodings that define the format."""
    cfg, dt = llama_config(case), LLAMA_DTYPES[case["dtype"]]
    shape = {(layer, tid): (rows, cols) for layer, tid, _, rows, cols in gten.tensor_list(cfg)}
    P = lambda tid, layer=0: llama_dequant(llama_payload(seed, dt, layer, tid, *shape[layer, tid]), dt, tid, *shape[layer, tid])
    n, H, G, D = case["n"], cfg.n_heads, cfg.n_groups, cfg.d_head

    def enc(x):
        if dt == gten.F16:
            return x.half().double()
        pad = -x.shape[-1] % 32
        b = torch.nn.functional.pad(x, (0, pad)).unflatten(-1, (-1, 32))
        step = b.abs().amax(-1, keepdim=True) / 127.0
        q = torch.where(step > 0, torch.sign(b) * torch.floor(b.abs() / step.clamp(min=1e-300) + 0.5), 0.0)
        return (q * step.half().double()).flatten(-2)[..., :x.shape[-1]]
    toks = torch.as_tensor(tokens_of(seed, "prompt", n, 32000), device="cuda").long()
    x = P(gten.T_EMBED)[toks]
    x = enc(x) if dt == gten.Q4 else x
    for i in range(cfg.n_layers):
        a = enc(rms(x, 1e-5, P(gten.T_ATTN_NORM, i)))
        q, k, v = (enc(a @ P(t, i).T) for t in (gten.T_Q, gten.T_K, gten.T_V))
        fr = freqs(D, 10000.0)
        q, k = enc(turn(q.reshape(n, H, D), fr, False).reshape(n, -1)), enc(turn(k.reshape(n, G, D), fr, False).reshape(n, -1))
        q, k, v, see, out = q.reshape(n, H, D), k.reshape(n, G, D), v.reshape(n, G, D), causal(n), []
        for h in range(H):
            s = (q[:, h] @ k[:, h // (H // G)].T / D ** 0.5).masked_fill(~see, -math.inf)
            out.append(enc(torch.softmax(s, 1)) @ v[:, h // (H // G)])
        x = enc(x + enc(enc(torch.stack(out, 1).reshape(n, -1)) @ P(gten.T_O, i).T))
        f = enc(rms(x, 1e-5, P(gten.T_FFN_NORM, i)))
        x = enc(x + enc(enc(enc(silu(enc(f @ P(gten.T_GATE, i).T))) * enc(f @ P(gten.T_UP, i).T)) @ P(gten.T_DOWN, i).T))
    return (enc(rms(x[-1:], 1e-5, P(gten.T_FINAL_NORM))) @ P(gten.T_LM_HEAD).T)[0]


@torch.no_grad()
def exact(case, seed):
    if case["kind"] in ("llama_decode", "llama_prefill", "llama_batch"):
        return None            # the values of these calls are those of one order of 32-bit sums, to the last bit; no 64-bit result stands for them
    if case["kind"] == "llama_fast":
        return llama_exact(case, seed)
    fam, cfg = family_config(case)
    desc = fam.describe(cfg)
    shapes, scale, V = fam.tensor_shapes(desc), desc.get("embed_scale", 1.0), case["vocab"]
    P = lambda name: tensor(case, seed, name, shapes[name], scale).double()
    embed, head = P("embed") * scale, P("head")
    prompts = [tokens_of(seed, f"prompt{i}", n, V) for i, n in enumerate(lens_of(case) + ([case["more"]] if "more" in case else []))]
    fed = tokens_of(seed, "fed", 2 * len(prompts), V)

    def logits(toks, rows):
        t = torch.as_tensor(np.asarray(toks), device="cuda").long()
        x = embed[t]
        if case["family"] == "reninex":
            bg = cfg["embedding"]["bigram"]
            at = (torch.roll(t, 1) * bg["mul_prev"] + t * bg["mul_cur"]) % bg["buckets"]
            at[0] = bg["buckets"]
            x = x + P("bigram")[at]
        y = MODELS[case["family"]](cfg, P, x)[rows] @ head.T
        return 30.0 * torch.tanh(y / 30.0) if case["family"] == "nanotar" else y
    if case["kind"] == "prefill":
        want, out, base = wanted(sum(map(len, prompts))), [], 0
        for p in prompts:
            out.append(logits(p, [w - base for w in want if base <= w < base + len(p)]))
            base += len(p)
        return torch.cat(out)
    if case["kind"] == "mix":
        n = len(prompts)
        runs = [np.concatenate([p] + ([fed[s:s + 1]] if s < n - 1 else []) + [fed[n + s:n + s + 1]]) for s, p in enumerate(prompts)]
        y = [logits(r, list(range(len(p) - 1, len(r)))) for r, p in zip(runs, prompts)]
        return [torch.stack([y[s][0] for s in range(n - 1)]), torch.stack([y[s][1] for s in range(n - 1)] + [y[n - 1][0]]), torch.stack([v[-1] for v in y])]
    if case["family"] == "siladra" and sum(len(p) + case["new"] for p in prompts) > 4096:
        return None            # token-by-token recurrences over this many positions take too long
    first, toks, last = [], [], []
    for p in prompts:
        ids = list(p) + [0] * (case["new"] + 1)
        for i in range(len(p), len(ids)):
            ids[i] = (ids[i - 1] + 1) % V           # the head's preference; checked against the logits below
        while True:
            y = logits(ids, list(range(len(p) - 1, len(ids))))
            best = y[:-1].argmax(1).tolist()
            wrong = [i for i, b in enumerate(best) if ids[len(p) + i] != b]
            if not wrong:
                break
            ids[len(p) + wrong[0]] = best[wrong[0]]
        first.append(ids[len(p)])
        toks.append(ids[len(p) + 1:])
        last.append(y[-1])
    return {"first": np.asarray(first, np.int32), "tokens": np.asarray(toks, np.int32), "logits": torch.stack(last)}
