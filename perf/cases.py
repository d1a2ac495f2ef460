"""The work that users of this library have it do, as measured cases: decode matvecs, routed-expert layers from one
token to a full decode batch, prefill products, each through the C ABI (libosmos_b200/api.py) on synthetic weights with
the distributions of libosmos_b200/synth.py.

Kinds of case, and what each stands for:
  q8        a dense projection of a decode step on int8 activations: q8_round + q8_run
  mv        a dense projection of a decode step on F32 activations (1 .. 8 tokens: mv_strided; more tokens than one are
            a speculative or a small-batch step)
  lane      a routed-expert layer on the int8 lane, router to combine, as one ep_layer_step on one GPU (with a shared
            expert on every token where the model has one: shared_ffn before it)
  lane_f32  a routed-expert layer whose types have no int8 form: q4x_route + lane_ffn_f32
  moe_f16   a routed-expert layer over a prompt's tokens: q4x_moe (the grouped f16 product)
  mm        a dense projection over a prompt's tokens on f16 operands: mm_tokens
  mmq       the same on int8 activations in the reference's order of sums: mmq_x8_rows + mmq_group
  fp4       an NVFP4 projection over a prompt's tokens, W4A4: mm_fp4_act + mm_fp4
"""
import math

import torch

import libosmos_b200
from libosmos_b200 import api, synth

ROUTERS = {"softmax": 0, "sqrt_softplus": 1}


def listed():
    return [
        # the smallest call: one token through a 7 MB attention-sized matrix; launch latency counts
        {"name": "decode_q8_q4_0_6144x2048_b1", "kind": "q8", "type": "Q4_0", "rows": 6144, "cols": 2048, "n": 1},
        # a decode step's largest dense matrix, an output head of 49152 rows, in the type heads are usually kept in
        {"name": "decode_mv_q6_k_49152x2048_b1", "kind": "mv", "type": "Q6_K", "rows": 49152, "cols": 2048, "n": 1},
        # a few tokens at once (speculative decoding) through a shared-expert-sized matrix with long rows
        {"name": "decode_mv_q4_k_2048x7168_b5", "kind": "mv", "type": "Q4_K", "rows": 2048, "cols": 7168, "n": 5},
        # one user's decode token through a layer of 512 small experts
        {"name": "moe_iq3_xxs_512e_top10_b1", "kind": "lane", "type": "IQ3_XXS", "n_exp": 512, "k": 10, "dim": 2048, "ff": 512,
         "n": 1, "router": "softmax", "shared": ""},
        # a serving batch of 64 decode tokens through the same layer (the benchmark's default workload)
        {"name": "moe_iq3_xxs_512e_top10_b64", "kind": "lane", "type": "IQ3_XXS", "n_exp": 512, "k": 10, "dim": 2048, "ff": 512,
         "n": 64, "router": "softmax", "shared": ""},
        # one decode token, and a batch of 32, through a layer of 256 large experts with a shared expert beside them
        {"name": "moe_iq1_m_256e_top8_shared_b1", "kind": "lane", "type": "IQ1_M", "n_exp": 256, "k": 8, "dim": 7168, "ff": 2048,
         "n": 1, "router": "sqrt_softplus", "shared": "Q4_K"},
        {"name": "moe_iq1_m_256e_top8_shared_b32", "kind": "lane", "type": "IQ1_M", "n_exp": 256, "k": 8, "dim": 7168, "ff": 2048,
         "n": 32, "router": "sqrt_softplus", "shared": "Q4_K"},
        # a decode batch through MXFP4 experts (no int8 form: F32 activations)
        {"name": "moe_mxfp4_128e_top4_b32", "kind": "lane_f32", "type": "MXFP4", "n_exp": 128, "k": 4, "dim": 4096, "ff": 1536, "n": 32},
        # a 2048-token prompt through the same experts
        {"name": "moe_mxfp4_128e_top4_b2048", "kind": "moe_f16", "type": "MXFP4", "n_exp": 128, "k": 4, "dim": 4096, "ff": 1536, "n": 2048},
        # a prompt of no particular length through a dense matrix
        {"name": "prefill_mm_q4_k_4096x4096_b777", "kind": "mm", "type": "Q4_K", "rows": 4096, "cols": 4096, "n": 777},
        # a 512-token prompt through the same matrix on the int8 path
        {"name": "prefill_mmq_q4_k_4096x4096_b512", "kind": "mmq", "type": "Q4_K", "rows": 4096, "cols": 4096, "n": 512},
        # a full chunk of a long prompt through an FFN-sized NVFP4 matrix
        {"name": "prefill_fp4_nvfp4_17408x5120_b2048", "kind": "fp4", "type": "NVFP4", "rows": 17408, "cols": 5120, "n": 2048},
    ]


def _log(rng, lo, hi, step=1):
    """a multiple of `step` from lo to hi, spread over the logarithm"""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return int(min(hi, max(lo, round(v / step) * step)))


# no drawn case moves or computes more than the largest listed one does
_MAX_BYTES, _MAX_FLOPS = 1.6e9, 3.7e11


def draw(rng):
    while True:
        kind = rng.choice(["q8", "mv", "mv", "lane", "lane", "lane", "lane_f32", "moe_f16", "mm", "mm", "mmq", "fp4"])
        if kind == "q8":
            c = {"kind": kind, "type": rng.choice(["Q4_0", "Q8_0"]), "rows": _log(rng, 1024, 49152, rng.choice([1, 16, 128])),
                 "cols": _log(rng, 1024, 8192, 256), "n": rng.choice([1, 1, 1, 2])}
        elif kind == "mv":
            c = {"kind": kind, "type": rng.choice(["Q4_0", "Q8_0", "Q4_K", "Q5_K", "Q6_K", "IQ4_XS", "MXFP4"]),
                 "rows": _log(rng, 1024, 49152, rng.choice([8, 16, 128])), "cols": _log(rng, 1024, 8192, 256),
                 "n": rng.choice([1, 1, 2, 3, 4, 5, 8])}
        elif kind == "lane":  # (rows of 512 values up to 4096, of 1024 from there)
            dim = rng.choice([1024, 1536, 2048, 4096, 5120, 7168])
            shared = rng.choice(["", "", "Q4_K"])
            c = {"kind": kind, "type": rng.choice(["IQ3_XXS", "IQ3_XXS", "IQ2_XXS", "IQ1_S", "IQ1_M"]), "n_exp": _log(rng, 32, 512, 8),
                 "k": rng.randint(2, 10), "dim": dim, "ff": rng.choice([512, 1024, 1536, 2048]), "n": _log(rng, 1, 96),
                 "router": rng.choice(["softmax", "sqrt_softplus"]), "shared": shared}
            if c["n"] * c["k"] > 1024:
                continue
        elif kind == "lane_f32":
            c = {"kind": kind, "type": rng.choice(["MXFP4", "MXFP4", "Q4_K"]), "n_exp": _log(rng, 16, 128, 4), "k": rng.randint(2, 6),
                 "dim": rng.choice([2048, 2560, 4096]), "ff": rng.choice([768, 1536, 2048]), "n": _log(rng, 1, 64)}
        elif kind == "moe_f16":
            c = {"kind": kind, "type": rng.choice(["MXFP4", "MXFP4", "Q4_K"]), "n_exp": _log(rng, 16, 128, 4), "k": rng.randint(2, 6),
                 "dim": rng.choice([2048, 2560, 4096]), "ff": rng.choice([768, 1536, 2048]), "n": _log(rng, 65, 2048)}
        elif kind == "mm":
            c = {"kind": kind, "type": rng.choice(["Q4_K", "Q4_K", "Q8_0", "Q6_K", "Q5_K", "Q4_0", "MXFP4"]),
                 "rows": _log(rng, 1024, 17408, rng.choice([16, 128])), "cols": _log(rng, 1024, 8192, 256), "n": _log(rng, 9, 2048)}
        elif kind == "mmq":
            c = {"kind": kind, "type": "Q4_K", "rows": _log(rng, 1024, 17408, rng.choice([16, 128])), "cols": _log(rng, 1024, 8192, 256),
                 "n": _log(rng, 9, 2048)}
            if c["rows"] * c["cols"] * c["n"] > 3e10:  # (its F32 chain a group is work of its own: kept to a listed case's time)
                continue
        else:
            c = {"kind": kind, "type": "NVFP4", "rows": _log(rng, 1024, 17408, 128), "cols": _log(rng, 1024, 8192, 256),
                 "n": _log(rng, 16, 2048)}
        w = work(c)
        if w["bytes"] <= _MAX_BYTES and w["flops"] <= _MAX_FLOPS:
            return c


# ---- synthetic weights on the GPU: synth.py's recipe, a tensor at a time ---------------------------------------------------
_SIGMA = {"IQ3_XXS": 0.005, "IQ2_XXS": 0.005}
_SHARED_SIGMA = 1e-4  # (the shared expert's: its output then is of the routed experts' size, not a multiple that hides them)


def _halves(gen, n, sigma):
    d = torch.randn(n, generator=gen, device="cuda").abs_().mul_(sigma).to(torch.float16)
    return d.clamp_(min=6e-5).view(torch.int16)


def _tensor(gen, kind, rows, cols, sigma=None):
    """a row-major rows x cols tensor of blocks of type `kind` as flat bytes"""
    tid = synth.TYPE_ID[kind]
    values, nbytes = synth.BLOCK[tid]
    n = rows * (cols // values)
    words = torch.randint(-2 ** 31, 2 ** 31 - 1, ((n * nbytes + 3) // 4,), generator=gen, dtype=torch.int32, device="cuda")
    raw = words.view(torch.uint8)[:n * nbytes].view(n, nbytes)
    sigma = sigma or _SIGMA.get(kind, 0.01)
    if kind == "MXFP4":
        raw[:, 0] = torch.randint(117, 124, (n,), generator=gen, dtype=torch.int32, device="cuda").to(torch.uint8)
    elif kind == "NVFP4":
        raw[:, :4] = torch.randint(0x20, 0x48, (n, 4), generator=gen, dtype=torch.int32, device="cuda").to(torch.uint8)
    elif kind == "IQ1_M":  # the f16 scale lies in the top nibbles of the four scale words
        d = _halves(gen, n, sigma).to(torch.int32) & 0xFFFF
        for k in range(4):
            at = 48 + 2 * k + 1
            raw[:, at] = (raw[:, at] & 0x0F) | (((d >> (4 * k)) & 0x0F) << 4).to(torch.uint8)
    elif kind == "Q6_K":
        raw[:, 208:210] = _halves(gen, n, sigma).view(torch.uint8).view(n, 2)
    else:
        raw[:, 0:2] = _halves(gen, n, sigma).view(torch.uint8).view(n, 2)
        if kind in ("Q4_K", "Q5_K"):
            raw[:, 2:4] = _halves(gen, n, sigma).view(torch.uint8).view(n, 2)
    return raw.reshape(-1)


def _zeros(n, dtype):
    return torch.zeros(n, dtype=dtype, device="cuda")


def _scratch(nbytes):
    """(the tensor, its first 256-byte aligned address)"""
    assert nbytes, "the library refused the layer"
    t = _zeros(nbytes + 256, torch.uint8)
    return t, (t.data_ptr() + 255) // 256 * 256


def _experts(gen, c):
    """gate, up, down of all experts, each tensor's experts one after another, and an expert's bytes in each"""
    shapes = ((c["ff"], c["dim"]), (c["ff"], c["dim"]), (c["dim"], c["ff"]))
    w = [_tensor(gen, c["type"], c["n_exp"] * r, k) for r, k in shapes]
    return w, [t.numel() // c["n_exp"] for t in w]


def _lane_layer(c, w, per, lim):
    tid = synth.TYPE_ID[c["type"]]
    layer = api.LaneLayer(tid, tid, c["dim"], c["ff"], c["n_exp"], c["k"], lim, api.LaneExperts())
    for j in range(3):
        layer.experts.base[j], layer.experts.bytes[j] = w[j].data_ptr(), per[j]
    return layer


def prepare(case, seed):
    c = dict(case)
    lib = libosmos_b200.load()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    s = {"c": c, "lib": lib, "kind": c["kind"], "tid": synth.TYPE_ID[c["type"]]}
    n = c["n"]
    if c["kind"] in ("q8", "mv", "mm", "mmq", "fp4"):
        rows, cols = c["rows"], c["cols"]
        s["w"] = _tensor(gen, c["type"], rows, cols)
        s["x"] = torch.randn((n, cols), generator=gen, device="cuda")
        ys = (rows + 7) // 8 * 8  # (rows of y start on 32 bytes)
        s["y_mem"], s["ys"] = _zeros((n, ys), torch.float32), ys
        s["y"] = s["y_mem"][:, :rows]
    if c["kind"] == "q8":
        s["q"], s["d"] = _zeros((n, cols), torch.int8), _zeros((n, cols // 32), torch.float32)
    elif c["kind"] == "mm":
        n16 = (n + 15) // 16 * 16
        s["x16"], s["overflow"] = _zeros(n16 * cols, torch.float16), _zeros(1, torch.int32)
    elif c["kind"] == "mmq":
        n16 = (n + 15) // 16 * 16
        s["x8"] = _zeros(n16 * cols, torch.int8)
        s["dx"], s["sx"] = _zeros(n16 * cols // 32, torch.float32), _zeros(n16 * cols // 32, torch.float32)
        s["idx"], s["zero"] = torch.arange(n, dtype=torch.int32, device="cuda"), _zeros(1, torch.int32)
        s["cnt"] = torch.full((1,), n, dtype=torch.int32, device="cuda")
        s["tab"] = torch.tensor([s["w"].data_ptr()], dtype=torch.int64, device="cuda")
    elif c["kind"] == "fp4":
        s["xq"], s["xsc"] = _zeros((n, cols // 2), torch.uint8), _zeros((n, cols // 16), torch.uint8)
        s["gs"] = 5.0 / (6.0 * 448.0)  # a calibrated input scale: N(0, 1) activations reach about 5
    elif c["kind"] in ("lane", "lane_f32", "moe_f16"):
        dim, ff, k, n_exp = c["dim"], c["ff"], c["k"], c["n_exp"]
        s["w"], per = _experts(gen, c)
        s["x"] = torch.randn((n, dim), generator=gen, device="cuda")
        s["logits"] = torch.randn((n, n_exp), generator=gen, device="cuda")
        s["y"] = _zeros((n, dim), torch.float32)
        if c["kind"] == "lane":
            layer = _lane_layer(c, s["w"], per, 10.0 if c["shared"] else 1e30)
            s["mem"], at = _scratch(lib.lane_scratch_bytes(layer, n))
            scratch, lay, p = api.LaneScratch(), api.EpLayout(), api.EpPlan()
            assert lib.lane_scratch_bind(layer, n, at, s["mem"].numel() - 256, scratch)
            assert lib.ep_layout(1, n, k, dim, lay)
            s["exchange"], p.peer[0] = _scratch(lay.bytes)
            s["sync"], s["rows"] = _zeros(4, torch.int32), _zeros(2 * n * k, torch.int64)
            s["bias"] = torch.randn(n_exp, generator=gen, device="cuda").mul_(0.1)
            p.rank, p.n_ranks, p.n_tok, p.expert0, p.expert1, p.lay = 0, 1, n, 0, n_exp, lay
            p.sync, p.rows, p.layer, p.scratch = s["sync"].data_ptr(), s["rows"].data_ptr(), layer, scratch
            p.router, p.route_bias, p.route_scale = ROUTERS[c["router"]], s["bias"].data_ptr(), 2.5
            assert lib.ep_plan_ok(p), "the fused step does not take this layer"
            s["plan"], s["add"] = p, None
            if c["shared"]:
                st = synth.TYPE_ID[c["shared"]]
                s["shared_w"] = [_tensor(gen, c["shared"], r, q, _SHARED_SIGMA) for r, q in ((ff, dim), (ff, dim), (dim, ff))]
                e = api.SharedExpert(st, st, dim, ff, 10.0, *[t.data_ptr() for t in s["shared_w"]])
                s["shared_mem"], at = _scratch(lib.shared_scratch_bytes(e, n))
                sc = api.SharedScratch()
                assert lib.shared_scratch_bind(e, n, at, s["shared_mem"].numel() - 256, sc)
                s["shared"], s["shared_scratch"], s["add"] = e, sc, _zeros((n, dim), torch.float32)
        elif c["kind"] == "lane_f32":
            s["x"] = s["x"].to(torch.bfloat16).to(torch.float32)  # (activations out of a bf16 model)
            s["layer"] = layer = _lane_layer(c, s["w"], per, 7.0)
            s["mem"], at = _scratch(lib.lane_f32_scratch_bytes(layer, n))
            s["scratch"] = api.LaneScratchF32()
            assert lib.lane_f32_scratch_bind(layer, n, at, s["mem"].numel() - 256, s["scratch"])
            s["ids"], s["rows"] = _zeros(n * k, torch.int32), _zeros(n * k, torch.int32)
            s["wts"] = _zeros(n * k, torch.float32)
        else:
            s["x"] = s["x"].to(torch.bfloat16).to(torch.float32)
            s["layer"] = layer = api.Q4xMoeLayer()
            layer.dim, layer.ff, layer.n_exp, layer.k = dim, ff, n_exp, k
            for j in range(3):
                layer.type[j], layer.base[j], layer.bytes[j] = s["tid"], s["w"][j].data_ptr(), per[j]
            s["mem"], at = _scratch(lib.q4x_moe_scratch_bytes(layer, n))
            s["scratch"] = api.Q4xMoeScratch()
            assert lib.q4x_moe_scratch_bind(layer, n, at, s["mem"].numel() - 256, s["scratch"])
            s["shared"] = torch.randn((n, dim), generator=gen, device="cuda")
            s["shared_logit"] = torch.randn(n, generator=gen, device="cuda")
    return s


def run(s):
    c, lib, kind, x, y = s["c"], s["lib"], s["kind"], s["x"], s["y"]
    n = c["n"]
    if kind == "q8":
        rows, cols = c["rows"], c["cols"]
        ok = lib.q8_round(x.data_ptr(), n, cols, cols, s["q"].data_ptr(), s["d"].data_ptr(), 0)
        ok = ok and lib.q8_run(s["tid"], s["w"].data_ptr(), rows, cols, s["q"].data_ptr(), s["d"].data_ptr(), n,
                               s["y_mem"].data_ptr(), s["ys"], 0)
    elif kind == "mv":
        ok = lib.mv_strided(s["tid"], s["w"].data_ptr(), c["rows"], c["cols"], x.data_ptr(), c["cols"], n, s["y_mem"].data_ptr(),
                            s["ys"], 0)
    elif kind == "mm":
        ok = lib.mm_tokens(s["tid"], s["w"].data_ptr(), c["rows"], s["y_mem"].data_ptr(), s["ys"], None, 0, None, 0, c["cols"],
                           x.data_ptr(), c["cols"], n, s["x16"].data_ptr(), s["overflow"].data_ptr(), False, 0)
    elif kind == "mmq":
        ok = lib.mmq_x8_rows(x.data_ptr(), c["cols"], s["idx"].data_ptr(), n, c["cols"], s["x8"].data_ptr(), s["dx"].data_ptr(),
                             s["sx"].data_ptr(), 0)
        ok = ok and lib.mmq_group(s["tid"], s["tab"].data_ptr(), s["cnt"].data_ptr(), 1, n, c["rows"], c["cols"], s["x8"].data_ptr(),
                                  s["dx"].data_ptr(), s["sx"].data_ptr(), s["zero"].data_ptr(), s["y_mem"].data_ptr(),
                                  s["zero"].data_ptr(), s["ys"], 0)
    elif kind == "fp4":
        ok = lib.mm_fp4_act(x.data_ptr(), c["cols"], n, c["cols"], s["gs"], s["xq"].data_ptr(), s["xsc"].data_ptr(), 0)
        ok = ok and lib.mm_fp4(s["w"].data_ptr(), c["rows"], c["cols"], s["xq"].data_ptr(), s["xsc"].data_ptr(), n, s["gs"],
                               s["y_mem"].data_ptr(), s["ys"], 0)
    elif kind == "lane":
        add, ok = None, True
        if s["add"] is not None:
            add = s["add"].data_ptr()
            ok = lib.shared_ffn(s["shared"], s["shared_scratch"], x.data_ptr(), n, add, 0)
        ok = ok and lib.ep_layer_step(s["plan"], x.data_ptr(), s["logits"].data_ptr(), add, y.data_ptr(), 0)
    elif kind == "lane_f32":
        ok = lib.q4x_route(s["logits"].data_ptr(), n, c["n_exp"], c["k"], s["ids"].data_ptr(), s["wts"].data_ptr(), s["rows"].data_ptr(), 0)
        ok = ok and lib.lane_ffn_f32(s["layer"], s["scratch"], x.data_ptr(), s["ids"].data_ptr(), s["wts"].data_ptr(), n, None,
                                     y.data_ptr(), 0)
    else:
        ok = lib.q4x_moe(s["layer"], s["scratch"], x.data_ptr(), s["logits"].data_ptr(), s["shared"].data_ptr(),
                         s["shared_logit"].data_ptr(), n, y.data_ptr(), 0)
    if not ok:
        raise RuntimeError("libosmos_b200 refused a call")
    return y


def work(case):
    c = case
    n = c["n"]
    tb = lambda kind, r, k: synth.tensor_bytes(synth.TYPE_ID[kind], r, k)  # noqa: E731
    if c["kind"] in ("q8", "mv", "mm", "mmq", "fp4"):
        return {"bytes": tb(c["type"], c["rows"], c["cols"]) + 4 * n * (c["cols"] + c["rows"]), "flops": 2 * n * c["rows"] * c["cols"]}
    dim, ff = c["dim"], c["ff"]
    expert = 2 * tb(c["type"], ff, dim) + tb(c["type"], dim, ff)
    touched = c["n_exp"] * (1 - (1 - c["k"] / c["n_exp"]) ** n)  # distinct experts of n tokens' picks, on average
    w = {"bytes": touched * expert + 4 * n * (2 * dim + c["n_exp"]), "flops": 6 * n * c["k"] * dim * ff}
    if c.get("shared"):
        w["bytes"] += 2 * tb(c["shared"], ff, dim) + tb(c["shared"], dim, ff)
        w["flops"] += 6 * n * dim * ff
    if c["kind"] == "moe_f16":
        w["bytes"] += 4 * n * (dim + 1)
    return w


def tolerance(case):
    """The int8 lane, the F32 matvecs and mmq fix every sum's order: their bits are part of the interface. The f16 and FP4
    products accumulate in F32 in the tensor core's order: about four times their distance from 64-bit sums over the same
    operands at the listed sizes (mm 4.9e-6, fp4 2.6e-8, moe_f16 3.2e-5 and the shared expert 2.3e-5 with an activation next to a rounding boundary of f16
    falling either way)."""
    c = case
    if c["kind"] == "mm":
        return {"rel": 2e-5, "max": 2e-4}
    if c["kind"] == "fp4":
        return {"rel": 1e-6, "max": 1e-5}
    if c["kind"] == "moe_f16" or (c.get("shared") and c["n"] > 8):
        return {"rel": 1.3e-4, "max": 5e-3}
    return "exact"
