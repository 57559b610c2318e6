"""The work that a host program has this library do, as measurable cases.

A case is one routed-MoE layer (or a short stack of them) called through the public entry points of the package: the
expert bank resident in HBM, a batch of token rows in, the layer's rows out.  The shapes are the benchmark's (bench.py)
and the tests': the DeepSeek-V4.1-Flash-shaped layer over an EXL3 bank (3 bits per weight, and the 2-bit layers of the
same bank), the GLM-Flash-shaped EXL3 layer, the MiMo-shaped MXFP4 layer and the GLM-shaped NVFP4 layer.

Fields of a case:
  bank     "exl3" | "exl3_k2" | "mxfp4" | "nvfp4": how the experts are stored
  hidden, inter, experts, top_k, shared: the layer's geometry; shared = a bf16 dense shared expert is added
  layers   layers called back to back, each on the rows the one before it wrote
  tokens   rows of one call (1 = a single sequence's decode step, thousands = a prefill chunk)
  routing  "normal": N(0,1) logits; "zipf": the same plus a popularity ~ rank^-1.1 per layer (a few hot experts)
  entry    what the host holds and asks for:
             "forward"    x and the router's logits -> y (MoE.forward)
             "forward_x"  x alone, the router's weight is resident -> y (MoE.forward_x)
             "experts"    x, expert ids and weights (the host routes) -> y (MoE.experts)
             "routed"     x and ids -> the unweighted rows of every routed expert (MoE.routed)
             "host"       x and logits in pinned host memory -> y in pinned host memory (MoE.forward_host)
"""
import functools
import math

import numpy as np
import torch

from __graft_entry__ import load_package

GEOMETRY = {
    # bank kind, (hidden, inter), shared expert, scoring, routed scale, activation limit, combine in bf16 steps
    "dsv": dict(hidden=5120, inter=2304, shared=True, scoring="sqrtsoftplus", scale=1.5, limit=10.0, chain=False),
    "glm_exl3": dict(hidden=4096, inter=2048, shared=True, scoring="sigmoid", scale=2.5, limit=10.0, chain=False),
    "mimo": dict(hidden=4096, inter=2048, shared=False, scoring="softmax", scale=1.0, limit=0.0, chain=True),
    "glm": dict(hidden=6144, inter=2048, shared=True, scoring="sigmoid", scale=1.0, limit=10.0, chain=True),
}


def _case(model, bank, tokens, entry, routing="normal", layers=1, experts=256, **more):
    g = GEOMETRY[model]
    return dict(more, model=model, bank=bank, hidden=g["hidden"], inter=g["inter"], shared=g["shared"], experts=experts,
                top_k=8, layers=layers, tokens=tokens, routing=routing, entry=entry)


def listed():
    return [
        # one sequence decoding, the whole layer from x: latency and launches count as much as the weight stream
        _case("dsv", "exl3", 1, "forward_x", name="exl3_token"),
        _case("mimo", "mxfp4", 1, "forward", name="mxfp4_token"),
        # a few sequences decoding together
        _case("glm", "nvfp4", 7, "forward_x", name="nvfp4_batch7"),
        # a small server batch whose rows live on the host, over a 2-bit layer
        _case("dsv", "exl3_k2", 16, "host", name="exl3_k2_host16"),
        # the benchmark's default: a full decode batch, 3-bit trellis
        _case("dsv", "exl3", 64, "forward", name="exl3_batch64"),
        # a decode batch that is not a round number, MXFP4
        _case("mimo", "mxfp4", 61, "forward", name="mxfp4_batch61"),
        # consecutive layers of a model under skewed routing: hot experts with many rows beside experts with one
        _case("dsv", "exl3", 64, "forward", routing="zipf", layers=4, name="exl3_stack64_zipf"),
        # a short prompt (or speculative rows), routed by the host
        _case("glm_exl3", "exl3", 300, "experts", routing="zipf", name="exl3_chunk300_zipf"),
        # prefill chunks
        _case("dsv", "exl3", 2048, "forward_x", name="exl3_prefill2048"),
        _case("glm", "nvfp4", 4093, "forward", name="nvfp4_prefill4093"),
        _case("dsv", "exl3", 8192, "forward", name="exl3_prefill8192"),
        # the largest call the reference admits
        _case("mimo", "mxfp4", 16384, "forward", name="mxfp4_prefill16384"),
    ]


def draw(rng):
    model, bank, most = rng.choice([("dsv", "exl3", 8192), ("dsv", "exl3_k2", 8192), ("glm_exl3", "exl3", 8192),
                                    ("mimo", "mxfp4", 16384), ("glm", "nvfp4", 8192)])
    tokens = int(round(math.exp(rng.uniform(0.0, math.log(most)))))
    layers = 4 if bank.startswith("exl3") and tokens <= 64 and rng.random() < 0.25 else 1
    entries = ["forward", "forward_x", "experts"] + (["host", "routed"] if tokens <= 256 else [])
    entry = "forward" if layers > 1 else rng.choice(entries)
    # from x the logits are what the router's product gives: no popularity is added to them
    routing = "normal" if entry == "forward_x" else rng.choice(["normal", "zipf"])
    return _case(model, bank, tokens, entry, routing=routing, layers=layers, experts=rng.choice([256, 256, 256, 128, 64]))


# ------------------------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------------------------
def _popularity(experts, layer):
    """ln p of a layer's experts: p ~ rank^-1.1 over a permutation that belongs to the layer."""
    perm = np.random.default_rng(4242 + layer).permutation(experts)
    p = np.arange(1, experts + 1, dtype=np.float64) ** -1.1
    return np.log(p / p.sum())[np.argsort(perm)].astype(np.float32)


def _exl3_records(case, n, gen, dev):
    """n expert records: per projection the trellis code (every bit pattern is a valid code), then the sign / scale
    vectors of its outputs and inputs as f16."""
    H, I, bits = case["hidden"], case["inter"], 2 if case["bank"] == "exl3_k2" else 3
    code = (H // 16) * (I // 16) * 32 * bits
    parts = []
    for n_out, n_in in ((I, H), (I, H), (H, I)):
        parts.append(torch.randint(0, 256, (n, code), dtype=torch.uint8, device=dev, generator=gen))
        for width, size in ((n_out, 0.02), (n_in, 1.0)):
            v = torch.rand((n, width), device=dev, generator=gen) + 0.5
            sign = torch.where(torch.rand((n, width), device=dev, generator=gen) < 0.5, -size, size)
            parts.append((v * sign).to(torch.float16).view(torch.uint8))
    return torch.cat(parts, dim=1)


def _fp4_records(case, n, gen, dev):
    """n expert records: N(0, 0.02) weights rounded to e2m1 codes with a block scale per 32 (MXFP4, power of two) or per
    16 inputs (NVFP4, E4M3 and one f32 per projection)."""
    H, I, nv = case["hidden"], case["inter"], case["bank"] == "nvfp4"
    parts = []
    for rows, cols in ((I, H), (I, H), (H, I)):
        bs = 16 if nv else 32
        blk = (torch.randn((n, rows * cols // bs, bs), device=dev, generator=gen) * 0.02)
        amax = blk.abs().amax(dim=2, keepdim=True).clamp_min(1e-30)
        if nv:
            g = amax.amax(dim=1)                                             # [n, 1]
            inv = (g / 2688.0).unsqueeze(2)
            sc8 = (amax / (6.0 * inv)).clamp(max=448.0).to(torch.float8_e4m3fn)
            scale = (sc8.to(torch.float32) * inv).clamp_min(1e-30)
            sbytes = sc8.view(torch.uint8)
        else:
            ex = torch.floor(torch.log2(amax)) - 2
            scale, sbytes = torch.exp2(ex), (ex + 127).to(torch.uint8)
        v = blk / scale
        a = v.abs()
        # nearest e2m1 magnitude: 0, .5, 1, 1.5 in steps of a half, then 2, 3, 4, 6
        c = torch.where(a < 1.75, torch.round(a * 2), torch.where(a < 3.5, torch.round(a) + 2, 6 + (a >= 5.0).float()))
        code = c.to(torch.uint8) | ((v < 0).to(torch.uint8) << 3)
        code = code.view(n, -1, 2)
        parts += [code[:, :, 0] | (code[:, :, 1] << 4), sbytes.reshape(n, -1)]
        if nv:
            parts.append(g.to(torch.float32).contiguous().view(torch.uint8))
    return torch.cat(parts, dim=1)


def _load_bank(moe, case, gen, dev):
    make = _exl3_records if case["bank"].startswith("exl3") else _fp4_records
    batch = 8
    for layer in range(case["layers"]):
        for e0 in range(0, case["experts"], batch):
            recs = make(case, batch, gen, dev)
            torch.cuda.current_stream().synchronize()
            for j in range(batch):
                moe.load_expert(layer, e0 + j, recs[j].data_ptr(), recs.shape[1], on_device=True)


def prepare(case, seed):
    pkg = load_package()
    dev = torch.device("cuda", torch.cuda.current_device())
    g = GEOMETRY[case["model"]]
    H, I, E, K, T, L = (case[k] for k in ("hidden", "inter", "experts", "top_k", "tokens", "layers"))
    kind = {"exl3": pkg.BANK_EXL3_K3_MUL1, "exl3_k2": pkg.BANK_EXL3_K2_MUL1, "mxfp4": pkg.BANK_MXFP4, "nvfp4": pkg.BANK_NVFP4}[case["bank"]]
    scoring = {"sqrtsoftplus": pkg.SCORE_SQRTSOFTPLUS, "sigmoid": pkg.SCORE_SIGMOID, "softmax": pkg.SCORE_SOFTMAX}[g["scoring"]]
    moe = pkg.MoE(pkg.make_config(
        H, I, E, K, n_layers=L, bank_kind=kind, act=pkg.ACT_SWIGLU_CLAMPED if g["limit"] > 0 else pkg.ACT_SWIGLU,
        act_limit=g["limit"], scoring=scoring, norm_topk=True, routed_scale=g["scale"], shared_expert=case["shared"],
        combine=pkg.COMBINE_CHAIN if g["chain"] else pkg.COMBINE_F32, max_tokens=max(T, 64), device=dev.index))
    gen = torch.Generator(device=dev)
    gen.manual_seed(seed)
    _load_bank(moe, case, gen, dev)

    def dense(*shape, std):
        return (torch.randn(shape, device=dev, generator=gen) * std).to(torch.bfloat16)

    if case["shared"]:
        for layer in range(L):
            w1, w3, w2 = dense(I, H, std=0.02), dense(I, H, std=0.02), dense(H, I, std=0.02)
            torch.cuda.current_stream().synchronize()
            moe.set_shared(layer, w1.data_ptr(), w3.data_ptr(), w2.data_ptr(), on_device=True)
    st = {"moe": moe, "case": case, "x": dense(T, H, std=1.0), "stream": torch.cuda.current_stream().cuda_stream}
    logits = []
    for layer in range(L):
        lg = torch.randn((T, E), device=dev, generator=gen)
        if case["routing"] == "zipf":
            lg = lg + torch.from_numpy(_popularity(E, layer)).to(dev)
        logits.append(lg)
    st["logits"] = logits
    entry = case["entry"]
    if entry == "forward_x":
        # W ~ N(0, 1/H): the logits of N(0,1) rows are N(0,1)
        w = dense(E, H, std=H ** -0.5)
        torch.cuda.current_stream().synchronize()
        moe.set_router_weight(0, w.data_ptr(), on_device=True)
    if entry in ("experts", "routed"):
        top, ids = torch.topk(torch.sigmoid(logits[0]), K, dim=1)
        st["ids"] = ids.to(torch.int32).contiguous()
        st["weights"] = (top / top.sum(dim=1, keepdim=True) * g["scale"]).contiguous()
    if entry == "routed":
        st["rows"] = torch.empty((T, K, H), dtype=torch.float32, device=dev)
    elif entry == "host":
        st["x"], st["logits"] = st["x"].cpu().pin_memory(), [logits[0].cpu().pin_memory()]
        st["y"] = torch.empty((T, H), dtype=torch.bfloat16).pin_memory()
    else:
        st["y"] = [torch.empty((T, H), dtype=torch.bfloat16, device=dev) for _ in range(min(L, 2))]
    return st


def run(st):
    moe, case, s = st["moe"], st["case"], st["stream"]
    T, entry, x = case["tokens"], case["entry"], st["x"]
    if entry == "routed":
        moe.routed(0, x.data_ptr(), st["ids"].data_ptr(), T, st["rows"].data_ptr(), s)
        return st["rows"]
    if entry == "host":
        moe.forward_host(0, x.data_ptr(), st["logits"][0].data_ptr(), T, st["y"].data_ptr(), s)
        return st["y"]
    if entry == "forward_x":
        moe.forward_x(0, x.data_ptr(), T, st["y"][0].data_ptr(), s)
        return st["y"][0]
    if entry == "experts":
        moe.experts(0, x.data_ptr(), st["ids"].data_ptr(), st["weights"].data_ptr(), T, st["y"][0].data_ptr(), s)
        return st["y"][0]
    for layer in range(case["layers"]):
        y = st["y"][layer % 2]
        moe.forward(layer, x.data_ptr(), st["logits"][layer].data_ptr(), T, y.data_ptr(), s)
        x = y
    return x


# ------------------------------------------------------------------------------------------------------------
# what a pass cannot do without
# ------------------------------------------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _distinct(experts, top_k, tokens, routing, layer):
    """Distinct experts that a call's tokens touch, from logits of the same distribution (all of them once the call is
    large)."""
    lg = np.random.default_rng(77).standard_normal((min(tokens, 2048), experts)).astype(np.float32)
    if routing == "zipf":
        lg += _popularity(experts, layer)
    return len(np.unique(np.argpartition(-lg, top_k, axis=1)[:, :top_k]))


def work(case):
    H, I, E, K, T, L = (case[k] for k in ("hidden", "inter", "experts", "top_k", "tokens", "layers"))
    weights = 3 * H * I
    expert = {"exl3": weights * 3 / 8 + 6 * H + 6 * I, "exl3_k2": weights * 2 / 8 + 6 * H + 6 * I,
              "mxfp4": weights * (1 / 2 + 1 / 32), "nvfp4": weights * (1 / 2 + 1 / 16) + 12}[case["bank"]]
    rows = T * (K + (1 if case["shared"] else 0))
    out = T * K * H * 4 if case["entry"] == "routed" else T * H * 2
    if case["entry"] == "routed":
        rows = T * K
    shared = 2 * weights if case["shared"] and case["entry"] != "routed" else 0
    router = 2 * E * H if case["entry"] == "forward_x" else T * K * 8 if case["entry"] in ("experts", "routed") else T * E * 4
    total = sum(_distinct(E, K, T, case["routing"], layer) * expert for layer in range(L))
    flops = L * rows * 6 * H * I + (2 * T * E * H if case["entry"] == "forward_x" else 0)
    return {"bytes": total + L * (shared + router + T * H * 2 + out), "flops": flops}


def tolerance(case):
    if case["entry"] == "routed":
        # f32 rows; the products' inputs are f16 (EXL3) or go through the bf16 rounding steps of the activation (FP4)
        return {"rel": 1e-3} if case["bank"].startswith("exl3") else {"rel": 5e-3}
    return {"rel": 1e-2}                # rows of bf16; a stack rounds between its layers
