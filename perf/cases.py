"""What a user of the package has it do, as measurable cases: decode GEMVs (raw k-quant blocks, merged planes + units,
generic planes; one row, a few rows, ragged MoE), prefill GEMMs (dense, ragged prompt, grouped MoE), the dequantiser and
the load-time repacking of a weight.

A case is a dict of plain values.  `listed()` are the named ones, `draw(rng)` gives more of the same kinds and ranges:

    raw        gguf_vecdot_dense (one row) / gguf_vecdot_rows (2..8 rows) over raw blocks, every k-quant
    merged     gguf_gemv_bc, planes + packed units, one row, every k-quant
    plane      gemv_plane, W4 / W2 / W1 with fp16 scale and zero planes, 1..8 rows, fp16 or bf16; with a "qtype" instead
               of "bits": gguf_gemv_scale_first over that k-quant's planes
    plane_moe  gemv_plane with row offsets: decode MoE, offsets on the device, the token count as the row bound
    raw_moe    gguf_vecdot_moe over raw blocks, offsets on the device
    gemm       gemm_plane, dense, fp16 or bf16
    gemm_moe   gemm_plane with row offsets: prefill MoE, ragged rows
    fq         gguf_dense_fully_quantized: the GEMM that reads planes + packed units; with "experts" > 0 the grouped form
    dequantize gguf_dequantize
    pack       gguf_prepare_fully_quantized_dense: host blocks in, host planes + units out (what loading a weight pays)

Everything but `pack` works on device tensors.
"""
import numpy as np
import torch

import quactlize_b200 as qb
from quactlize_b200 import synth

Q2_K, Q3_K, Q4_K, Q5_K, Q6_K = 10, 11, 12, 13, 14
DEV = "cuda:0"


def listed():
    return [
        # one token through a key/value projection of an 8B-sized decoder: the smallest launch of a decode step
        {"name": "raw_q4k_m1_4096to1024", "kind": "raw", "qtype": Q4_K, "m": 1, "n": 1024, "k": 4096},
        # one token through the FFN gate or up projection: the bulk of a decode step
        {"name": "raw_q4k_m1_4096to14336", "kind": "raw", "qtype": Q4_K, "m": 1, "n": 14336, "k": 4096},
        # four concurrent sequences (or draft tokens) through the FFN down projection
        {"name": "raw_q4k_m4_14336to4096", "kind": "raw", "qtype": Q4_K, "m": 4, "n": 4096, "k": 14336},
        # one token over the merged artifact that also serves the GEMMs, in the widest format
        {"name": "merged_q6k_m1_4096to14336", "kind": "merged", "qtype": Q6_K, "n": 14336, "k": 4096},
        # one token over a generic group-quantised weight (GPTQ-like, group 128)
        {"name": "plane_w4_m1_4096to4096", "kind": "plane", "bits": 4, "group": 128, "m": 1, "n": 4096, "k": 4096, "bf16": False},
        # decode MoE, 128 experts top-8, a batch of eight tokens through gate+up
        {"name": "plane_moe_w2_t8", "kind": "plane_moe", "bits": 2, "group": 64, "experts": 128, "top_k": 8, "tokens": 8,
         "n": 1536, "k": 2048, "bf16": True},
        # decode MoE over raw blocks, 8 experts top-2, three tokens
        {"name": "raw_moe_q4k_t3", "kind": "raw_moe", "qtype": Q4_K, "experts": 8, "top_k": 2, "tokens": 3, "n": 14336, "k": 4096},
        # prefill of 2048 tokens through a square projection
        {"name": "gemm_w4_m2048_4096to4096", "kind": "gemm", "bits": 4, "group": 32, "m": 2048, "n": 4096, "k": 4096, "bf16": False},
        # prefill MoE, 8 experts top-2, 4096 tokens on a skewed router, FFN gate
        {"name": "gemm_moe_w4_t4096", "kind": "gemm_moe", "bits": 4, "group": 128, "experts": 8, "top_k": 2, "tokens": 4096,
         "n": 14336, "k": 4096, "bf16": True},
        # a prompt of odd length through the FFN, on the bytes that the decode step uses too
        {"name": "fq_q4k_m333_4096to14336", "kind": "fq", "qtype": Q4_K, "experts": 0, "m": 333, "n": 14336, "k": 4096},
        # the weight written out in fp16 for a library GEMM
        {"name": "dequantize_q4k_14336x4096", "kind": "dequantize", "qtype": Q4_K, "n": 14336, "k": 4096},
        # loading: raw blocks of one weight on the host into the planes + units artifact
        {"name": "pack_q4k_14336x4096", "kind": "pack", "qtype": Q4_K, "n": 14336, "k": 4096},
    ]


def _log(rng, lo, hi, step=1):
    """An integer of lo..hi, uniform over the logarithm, a multiple of `step`."""
    v = lo * (hi / lo) ** rng.random()
    return min(hi // step * step, max(-(-lo // step) * step, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["raw", "raw", "raw", "merged", "plane", "plane_moe", "raw_moe", "gemm", "gemm_moe", "fq", "dequantize", "pack"])
    qt = rng.choice([Q2_K, Q3_K, Q4_K, Q4_K, Q5_K, Q6_K])
    if kind == "raw":
        return {"kind": kind, "qtype": qt, "m": rng.choice([1, 1, 1, 2, 3, 4, 5, 8]), "n": _log(rng, 500, 16384), "k": _log(rng, 1024, 14336, 256)}
    if kind == "merged":
        return {"kind": kind, "qtype": qt, "n": _log(rng, 512, 16384, 256), "k": _log(rng, 1024, 14336, 512)}
    if kind == "plane":
        if rng.random() < 0.4:
            return {"kind": kind, "qtype": qt, "m": rng.choice([1, 1, 2, 3, 6]), "n": _log(rng, 512, 16384, 256),
                    "k": _log(rng, 1024, 14336, 256), "bf16": False}
        return {"kind": kind, "bits": rng.choice([4, 4, 2, 1]), "group": rng.choice([32, 64, 128]), "m": rng.choice([1, 1, 2, 3, 6, 8]),
                "n": _log(rng, 512, 16384, 8), "k": _log(rng, 1024, 14336, 256), "bf16": rng.random() < 0.5}
    if kind == "plane_moe":
        bits = rng.choice([2, 1, 4])
        return {"kind": kind, "bits": bits, "group": 64, "experts": rng.choice([32, 64, 128]), "top_k": rng.choice([4, 6, 8]),
                "tokens": _log(rng, 1, 64), "n": _log(rng, 512, 2816, 8), "k": _log(rng, 768, 2816, 256), "bf16": rng.random() < 0.7}
    if kind == "raw_moe":
        return {"kind": kind, "qtype": qt, "experts": rng.choice([8, 16, 32]), "top_k": rng.choice([1, 2, 4]), "tokens": _log(rng, 1, 12),
                "n": _log(rng, 1024, 8192), "k": _log(rng, 1024, 4096, 256)}
    if kind == "gemm":
        return {"kind": kind, "bits": rng.choice([4, 4, 2]), "group": rng.choice([32, 64, 128]), "m": _log(rng, 17, 4096),
                "n": _log(rng, 1024, 14336, 128), "k": _log(rng, 1024, 8192, 256), "bf16": rng.random() < 0.5}
    if kind == "gemm_moe":
        return {"kind": kind, "bits": 4, "group": rng.choice([64, 128]), "experts": rng.choice([8, 16]), "top_k": 2, "tokens": _log(rng, 100, 4096),
                "n": _log(rng, 1024, 8192, 128), "k": _log(rng, 1024, 4096, 256), "bf16": True}
    if kind == "fq":
        experts = rng.choice([0, 0, 8])
        return {"kind": kind, "qtype": qt, "experts": experts, "m": _log(rng, 2, 2048), "n": _log(rng, 1024, 8192, 256), "k": _log(rng, 1024, 8192, 512)}
    return {"kind": kind, "qtype": qt, "n": _log(rng, 512, 14336, 256), "k": _log(rng, 1024, 4096, 512)}


# ---------------------------------------------------------------------------------------------------------------------
# inputs: uniform codes and sub-scales, |N(0, 0.01)| super-block headers, |N(0, 0.02)| / 7 group scales with the zero at
# half the code range, N(0, 1) activations -- the distributions of `quactlize_b200.synth`, made on the device

_HEADERS = {Q2_K: (80, 82), Q3_K: (108,), Q4_K: (0, 2), Q5_K: (0, 2), Q6_K: (208,)}       # fp16 fields of a raw block


def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _bytes(shape, g):
    return torch.randint(0, 256, shape, dtype=torch.uint8, device=DEV, generator=g)


def _put_headers(rows, offsets, g):
    """|N(0, 0.01)| in fp16 at the byte `offsets` of every row of `rows` [R, bytes]."""
    for o in offsets:
        d = (torch.randn(rows.shape[0], device=DEV, generator=g).abs() * 0.01).to(torch.float16)
        rows[:, o:o + 2] = d.view(torch.uint8).view(-1, 2)


def _raw_blocks(qtype, count, g):
    b = _bytes((count, qb.kquant_geometry(qtype).block_bytes), g)
    _put_headers(b, _HEADERS[qtype], g)
    return b


def _artifact(qtype, experts, n, k, g):
    """(low, high, units) of the merged / fully-quantized artifact: [E,n,..], [E,n,..] or empty, [E,U,n,bytes]."""
    q = qb.kquant_geometry(qtype)
    low = _bytes((experts, n, k * q.lo_bits // 8), g)
    high = _bytes((experts, n, k * q.hi_bits // 8), g) if q.hi_bits else torch.empty((0,), dtype=torch.uint8, device=DEV)
    units = _bytes((experts, k // 256 // q.sb_per_unit, n, q.unit_total), g)
    _put_headers(units.view(-1, q.sb_bytes), (0, 2) if q.has_min else (0,), g)
    return low, high, units


def _scale_zero(experts, n, k, group, zero_point, g):
    s = (torch.randn((experts, k // group, n), device=DEV, generator=g).abs() * (0.02 / 7)).to(torch.float16)
    return s, (-zero_point * s.float()).to(torch.float16)


def _activations(rows, k, bf16, g):
    return torch.randn((rows, k), device=DEV, generator=g).to(torch.bfloat16 if bf16 else torch.float16)


def _routed(case, seed):
    """Rows per expert of one step: uniform routing for decode, a Zipf-skewed router for prefill."""
    t, e, k = case["tokens"], case["experts"], case["top_k"]
    if case["kind"] == "gemm_moe":
        return synth.zipf_rows_per_expert(t, e, k, seed=seed)
    return np.bincount(synth.uniform_routes(t, e, k, seed=seed).reshape(-1), minlength=e)


def _offsets(counts):
    return torch.from_numpy(np.concatenate([[0], np.cumsum(counts)]).astype(np.int32)).to(DEV)


def prepare(case, seed):
    g, kind = _generator(seed), case["kind"]
    n, k, qt = case["n"], case["k"], case.get("qtype")
    s = dict(case)
    if kind == "raw":
        s.update(blocks=_raw_blocks(qt, n * k // 256, g), x=_activations(case["m"], k, False, g))
    elif kind == "merged":
        low, high, units = _artifact(qt, 1, n, k, g)
        s.update(low=low, high=high, units=units[0], x=_activations(1, k, False, g))
    elif kind == "plane" and qt is not None:
        q = qb.kquant_geometry(qt)
        low, high, _ = _artifact(qt, 1, n, k, g)
        scale, zero = _scale_zero(1, n, k, q.group_size, float(1 << (q.lo_bits + q.hi_bits - 1)), g)
        s.update(low=low, high=high, scale=scale, zero=zero, x=_activations(case["m"], k, False, g))
    elif kind in ("plane", "plane_moe", "gemm", "gemm_moe"):
        e, bits = case.get("experts", 1), case["bits"]
        low = _bytes((e, n, k * bits // 8), g)
        scale, zero = _scale_zero(e, n, k, case["group"], float(1 << (bits - 1)), g)
        rows = case["tokens"] * case["top_k"] if "tokens" in case else case["m"]
        s.update(low=low, scale=scale, zero=zero, x=_activations(rows, k, case["bf16"], g))
        if "tokens" in case:
            s.update(offsets=_offsets(_routed(case, seed)))
    elif kind == "raw_moe":
        e = case["experts"]
        blocks = _raw_blocks(qt, e * n * k // 256, g).view(e, n * k // 256, -1)
        s.update(blocks=blocks, x=_activations(case["tokens"] * case["top_k"], k, False, g), offsets=_offsets(_routed(case, seed)))
    elif kind == "fq":
        e = case["experts"]
        low, high, units = _artifact(qt, max(e, 1), n, k, g)
        s.update(low=low, high=high, units=units if e else units[0], x=_activations(case["m"], k, False, g))
        if e:                                       # the router's counts, on the host as the grouped entry takes them
            pick = np.random.default_rng(seed).integers(0, e, size=case["m"])
            s.update(rows=torch.from_numpy(np.bincount(pick, minlength=e).astype(np.int32)))
    elif kind == "dequantize":
        s.update(blocks=_raw_blocks(qt, n * k // 256, g))
    else:
        s.update(blocks=_raw_blocks(qt, n * k // 256, g).cpu())
    return s


def run(s):
    kind = s["kind"]
    if kind == "raw":
        if s["m"] == 1:
            return qb.gguf_vecdot_dense(s["blocks"], s["x"], s["n"], s["k"], s["qtype"])
        return qb.gguf_vecdot_rows(s["blocks"], s["x"], s["n"], s["k"], s["qtype"])
    if kind == "merged":
        return qb.gguf_gemv_bc(s["x"], s["low"], s["high"], s["units"], s["qtype"])
    if kind == "plane":
        if "qtype" in s:
            return qb.gguf_gemv_scale_first(s["x"], s["low"], s["high"], s["scale"], s["zero"], s["qtype"])
        return qb.gemv_plane(s["x"], s["low"], None, s["scale"], s["zero"], s["bits"], 0, s["group"])
    if kind == "plane_moe":                         # an expert gets at most every token once
        return qb.gemv_plane(s["x"], s["low"], None, s["scale"], s["zero"], s["bits"], 0, s["group"],
                             row_offsets=s["offsets"], max_rows=s["tokens"])
    if kind == "raw_moe":
        return qb.gguf_vecdot_moe(s["blocks"], s["x"], s["offsets"], s["qtype"])
    if kind == "gemm":
        return qb.gemm_plane(s["x"], s["low"], None, s["scale"], s["zero"], s["bits"], 0, s["group"])
    if kind == "gemm_moe":
        return qb.gemm_plane(s["x"], s["low"], None, s["scale"], s["zero"], s["bits"], 0, s["group"], row_offsets=s["offsets"])
    if kind == "fq":
        if s["experts"]:
            return qb.gguf_grouped_fully_quantized(s["x"], s["low"], s["high"], s["units"], s["rows"], s["qtype"])
        return qb.gguf_dense_fully_quantized(s["x"], s["low"], s["high"], s["units"], s["qtype"])
    if kind == "dequantize":
        return qb.gguf_dequantize(s["blocks"], s["qtype"])
    return qb.gguf_prepare_fully_quantized_dense(s["blocks"], s["n"], s["k"], s["qtype"])


def _touched(case):
    """Experts that a pass has rows for, on average, and its rows."""
    e = case["experts"]
    if "tokens" in case:
        return e * (1.0 - (1.0 - case["top_k"] / e) ** case["tokens"]), case["tokens"] * case["top_k"]
    return e * (1.0 - (1.0 - 1.0 / e) ** case["m"]), case["m"]


def work(case):
    kind, n, k, qt = case["kind"], case["n"], case["k"], case.get("qtype")
    experts, rows = _touched(case) if case.get("experts") else (1.0, case.get("m", 1))
    out = 4 if kind in ("raw", "merged", "raw_moe") else 2
    if kind == "plane" and qt is not None:
        q = qb.kquant_geometry(qt)
        weight = n * k * (q.lo_bits + q.hi_bits) / 8 + 4 * (k // q.group_size) * n
    elif qt is not None:                            # raw blocks, or the same bytes as planes + units
        weight = n * k // 256 * qb.kquant_geometry(qt).block_bytes
    else:
        weight = n * k * case["bits"] / 8 + 4 * (k // case["group"]) * n
    if kind == "dequantize":
        return {"bytes": weight + 2 * n * k, "flops": 0}
    if kind == "pack":
        return {"bytes": 2 * weight, "flops": 0}
    return {"bytes": experts * weight + rows * k * 2 + rows * n * out, "flops": 2.0 * rows * n * k}


def tolerance(case):
    """Bytes and decoded weights are exact.  The GEMVs multiply fp16 operands and may add a few products in fp16 before
    the fp32 sum (unit roundoff 4.9e-4, a handful of roundings); fp16 results of the GEMMs round weights and outputs once
    each; bf16 has eight times the roundoff."""
    if case["kind"] in ("dequantize", "pack"):
        return "exact"
    return {"rel": 1e-2} if case.get("bf16") else {"rel": 2e-3}
