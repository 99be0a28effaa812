"""The work this library is used for, as cases that can be timed and compared.

Every case goes through the public entry points of bare_metal_b200.igemm, the way a program that serves
or checks a quantised model calls them: weights, scales, metadata and output buffers exist before the
call, activations arrive on the GPU.

Kinds
  gemm_i32        raw int32 accumulators of a dense int8 GEMM (correctness runs, further epilogues)
  linear          one W8A8 linear with fp16 output, activations already quantised
  layer           the four linears of a transformer layer (QKV, output, gate + up, down) for a batch of
                  tokens: fp16 activations are quantised per token, then multiplied.  Few tokens =
                  decoding, many = prefill.
  perchannel      reference ABI, B[K x N], fp32 output with per-channel scale and zero point
  pertensor       reference ABI, B[K x N], fp32 output with one scale
  sparse_left     reference ABI, 2:4-sparse operand on the left, metadata in the reference's words
  sparse_linear   2:4-sparse weights with tiled metadata, int32 or fp16 output (prefill)
  sparse_decode   2:4-sparse weights in packed form, fp16 output, at most 64 tokens (decoding)
  online_quant    fp16 operands quantised inside the call, fp32 output
  hgemm_sparse    fp16 2:4-sparse operand on the left, fp32 output, metadata tiled once
"""
import math

import torch

from bare_metal_b200 import igemm as ig

# Tolerances are about four times what two correct evaluations on a CPU differ by (K = 512, 4096, 8192).
# fp16 results of exact integer sums: float(acc) * (sa * sw) against (float(acc) * sa) * sw and against 64 bits,
# both rounded to half: up to 9e-6 in the 2-norm, one unit in the last place (9.2e-4) of single values.
_F16_OUT = {"rel": 3.5e-5, "max": 4e-3}
# the same behind the per-token quantiser: x * (1 / scale) against x / scale in 64 bits moves about one quantised
# value in 20000 by one step: up to 2.8e-4 in the 2-norm, 4.8e-3 for a single value.
_F16_LAYER = {"rel": 1e-3, "max": 2e-2}
# fp32 results of integer sums (reference ABI): one or two fp32 roundings, 3.7e-8 and 1.1e-7 against 64 bits.
_F32_SCALED = {"rel": 1.5e-7, "max": 4.5e-7}
# fp16 operands quantised inside the call: one scaling of the exact sum against one fp32 addition per 32 of K, as
# the reference does: up to 2.9e-7 and 1.6e-6.
_F32_ONLINE = {"rel": 1.2e-6, "max": 6.5e-6}
# fp16 x fp16 products added in fp32: added one by one against 64 bits, up to 1.2e-6 and 8.2e-6.
_F32_SUMS = {"rel": 5e-6, "max": 3.5e-5}


def listed():
    return [
        # a small GEMM called on its own: latency and launch cost count
        dict(name="gemm_i32_1024", kind="gemm_i32", m=1024, n=1024, k=1024, layout="kn"),
        # decoding with a batch of 16 sequences: every weight is read once for 16 tokens
        dict(name="layer_16_tokens", kind="layer", m=16, hidden=4096, ffn=11008),
        # a prompt of odd length: ragged token tiles, a few waves at most
        dict(name="layer_777_tokens", kind="layer", m=777, hidden=4096, ffn=11008),
        # a full prefill batch of the same layer
        dict(name="layer_8192_tokens", kind="layer", m=8192, hidden=4096, ffn=11008),
        # the library's headline product
        dict(name="linear_4096", kind="linear", m=4096, n=4096, k=4096),
        # reference ABI with every dimension off the tile grid
        dict(name="perchannel_ragged", kind="perchannel", m=2500, n=2256, k=2064),
        # the reference's sparse bench: sparse operand left, reference metadata on every call
        dict(name="sparse_left_4096", kind="sparse_left", m=4096, n=4096, k=4096),
        # sparse weights, many tokens
        dict(name="sparse_linear_4096", kind="sparse_linear", m=4096, n=4096, k=4096, out="i32"),
        # sparse weights, decoding one sequence and a batch of 64
        dict(name="sparse_decode_1", kind="sparse_decode", m=1, n=28672, k=8192),
        dict(name="sparse_decode_64", kind="sparse_decode", m=64, n=28672, k=8192),
        # fp16 in, quantised per tile inside the call, fp32 out
        dict(name="online_quant_4096", kind="online_quant", m=4096, n=4096, k=4096, col_block=128),
        # fp16 2:4 GEMM of the reference's hgemm_sparse family
        dict(name="hgemm_sparse_4096", kind="hgemm_sparse", m=4096, n=4096, k=4096),
    ]


def _log_int(rng, lo, hi, step=1):
    """An integer in [lo, hi], a multiple of `step`, spread evenly over its logarithm."""
    v = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(lo, min(hi, int(round(v / step)) * step))


def draw(rng):
    kind = rng.choice(["gemm_i32", "linear", "layer", "layer", "perchannel", "pertensor", "sparse_left",
                       "sparse_linear", "sparse_decode", "online_quant", "hgemm_sparse"])
    case = dict(kind=kind)
    if kind == "layer":
        case["m"] = _log_int(rng, 1, 8192)
        case["hidden"] = _log_int(rng, 1024, 4096, 16)
        case["ffn"] = min(11008, int(round(case["hidden"] * rng.uniform(2.0, 3.0) / 16)) * 16)
        return case
    if kind == "sparse_decode":
        case.update(m=rng.randint(1, 64), n=_log_int(rng, 2048, 28672, 8), k=_log_int(rng, 1024, 8192, 32))
        return case
    # an 8192-sized operand on two sides and up to 8192 on the third: below the largest listed layer
    if kind in ("gemm_i32", "linear"):
        case["m"] = _log_int(rng, 1, 8192)
        case["n"] = _log_int(rng, 512, 8192, 16)
        case["k"] = _log_int(rng, 512, 8192, 16)
        if kind == "gemm_i32":
            case["layout"] = rng.choice(["kn", "nk"])
    elif kind == "sparse_linear":
        case.update(m=_log_int(rng, 65, 8192), n=_log_int(rng, 512, 8192, 16), k=_log_int(rng, 512, 8192, 32),
                    out=rng.choice(["i32", "f16"]))
    else:                                   # reference ABI: rows in multiples of 16 for its metadata words
        step_m = 1 if kind in ("perchannel", "pertensor", "online_quant") else 16
        case.update(m=_log_int(rng, 256, 8192, step_m), n=_log_int(rng, 256, 8192, 16),
                    k=_log_int(rng, 256, 8192, 32))
        if kind == "online_quant":
            case["col_block"] = rng.choice([128, 256])
    return case


def _layer_shapes(case):
    h, f = case["hidden"], case["ffn"]
    return [("qkv", 3 * h, h), ("out", h, h), ("gate_up", 2 * f, h), ("down", h, f)]


# ---- inputs --------------------------------------------------------------------------------------
class _Inputs:
    """Seeded draws on the GPU: int8 values uniform on [-127, 127], scales uniform on [1e-3, 2e-2]."""

    def __init__(self, seed):
        self.dev = torch.device("cuda", torch.cuda.current_device())
        self.gen = torch.Generator(device=self.dev)
        self.gen.manual_seed(seed)

    def int8(self, *shape):
        return torch.randint(-127, 128, shape, dtype=torch.int8, device=self.dev, generator=self.gen)

    def scales(self, n):
        return torch.rand(n, device=self.dev, generator=self.gen) * 0.019 + 0.001

    def activations(self, m, k):
        """fp16 activations whose tokens differ in magnitude."""
        x = torch.randn((m, k), device=self.dev, dtype=torch.float16, generator=self.gen)
        return x.mul_((torch.rand((m, 1), device=self.dev, generator=self.gen) * 3.5 + 0.5).half())

    def uniform_f16(self, *shape):
        return torch.rand(shape, device=self.dev, dtype=torch.float16, generator=self.gen).mul_(2).sub_(1)

    def nibbles(self, count):
        """2:4 position nibbles (idx1 << 2) | idx0, the six patterns equally likely."""
        table = torch.tensor([0x4, 0x8, 0xC, 0x9, 0xD, 0xE], dtype=torch.int32, device=self.dev)
        return table[torch.randint(0, 6, (count,), device=self.dev, generator=self.gen)]

    def ref_meta_words(self, rows, k_steps, nibbles_per_word):
        """Reference metadata words [rows/16][k steps][8]: rows r and r + 8 of a 16-row tile share one."""
        words = self.nibbles((rows // 16) * k_steps * 8 * nibbles_per_word).view(-1, nibbles_per_word).long()
        shifts = torch.arange(0, 4 * nibbles_per_word, 4, device=self.dev)
        w = (words << shifts).sum(1)
        if nibbles_per_word == 4:
            w = w | (w << 16)
        return torch.where(w >= 2 ** 31, w - 2 ** 32, w).to(torch.int32)

    def empty(self, dtype, *shape):
        return torch.empty(shape, dtype=dtype, device=self.dev)


def prepare(case, seed):
    g = _Inputs(seed)
    kind, m = case["kind"], case["m"]
    st = {"case": dict(case)}
    if kind == "layer":
        st["parts"] = []
        for _, n, k in _layer_shapes(case):
            st["parts"].append(dict(x=g.activations(m, k), w=g.int8(n, k), sw=g.scales(n),
                                    d=g.empty(torch.float16, m, n), n=n, k=k))
        return st
    n, k = case["n"], case["k"]
    if kind in ("gemm_i32", "linear"):
        st["a"] = g.int8(m, k)
        if kind == "gemm_i32" and case["layout"] == "kn":
            st["b"], st["layout"] = g.int8(k, n), ig.BM_B_KN
        else:
            st["b"], st["layout"] = g.int8(n, k), ig.BM_B_NK
        if kind == "linear":
            st["sa"], st["sw"] = g.scales(m), g.scales(n)
            st["out"] = g.empty(torch.float16, m, n)
        else:
            st["out"] = g.empty(torch.int32, m, n)
    elif kind in ("perchannel", "pertensor"):
        st["a"], st["b"] = g.int8(m, k), g.int8(k, n)
        st["out"] = g.empty(torch.float32, m, n)
        if kind == "perchannel":
            st["scale"] = g.scales(n) * 1e-2
            st["zero"] = torch.randint(-8, 9, (n,), dtype=torch.int32, device=g.dev, generator=g.gen)
    elif kind == "sparse_left":
        st["comp"], st["b"] = g.int8(m, k // 2), g.int8(k, n)
        st["meta"] = g.ref_meta_words(m, k // 32, 8)
        st["out"] = g.empty(torch.float32, m, n)
    elif kind == "sparse_linear":
        st["x"] = g.int8(m, k)
        # a dense layer pruned by magnitude, then tiled: what a user does once per weight matrix
        st["comp"], nib = ig.prune_2_4(g.int8(n, k), n, k)
        st["meta"] = ig.sp_pack_meta(nib, ig.BM_META_ROWS, n, k)
        if case["out"] == "f16":
            st["sa"], st["sw"] = g.scales(m), g.scales(n)
            st["out"] = g.empty(torch.float16, m, n)
        else:
            st["out"] = g.empty(torch.int32, m, n)
    elif kind == "sparse_decode":
        st["x"] = g.int8(m, k)
        comp, nib = ig.prune_2_4(g.int8(n, k), n, k)
        st["packed"] = ig.sp_pack_weights(comp, nib, ig.BM_META_ROWS, n, k)
        st["sa"], st["sw"] = g.scales(m), g.scales(n)
        st["out"] = g.empty(torch.float16, m, n)
    elif kind == "online_quant":
        st["a"], st["b"] = g.uniform_f16(m, k), g.uniform_f16(k, n)
        st["out"] = g.empty(torch.float32, m, n)
    elif kind == "hgemm_sparse":
        st["comp"], st["b"] = g.uniform_f16(m, k // 2), g.uniform_f16(k, n)
        st["meta"] = ig.sp_pack_meta(g.ref_meta_words(m, k // 16, 4), ig.BM_META_REF_F16, m, k)
        st["out"] = g.empty(torch.float32, m, n)
    else:
        raise ValueError(kind)
    return st


# ---- one pass ------------------------------------------------------------------------------------
def run(st):
    case = st["case"]
    kind, m = case["kind"], case["m"]
    if kind == "layer":
        outs = []
        for p in st["parts"]:
            q, s = ig.quantize_rows(p["x"], m, p["k"])
            outs.append(ig.w8a8_linear(q, p["w"], p["d"], s, p["sw"], m, p["n"], p["k"]))
        return outs
    n, k = case["n"], case["k"]
    if kind == "gemm_i32":
        return ig.igemm_i32(st["a"], st["b"], st["out"], m, n, k, st["layout"])
    if kind == "linear":
        return ig.w8a8_linear(st["a"], st["b"], st["out"], st["sa"], st["sw"], m, n, k)
    if kind == "perchannel":
        return ig.igemm_pipelined_cpasync_perchannel(st["a"], st["b"], st["out"], m, n, k, st["scale"], st["zero"])
    if kind == "pertensor":
        return ig.igemm_wmma(st["a"], st["b"], st["out"], m, n, k, 0.011, 0.007)
    if kind == "sparse_left":
        return ig.igemm_sparse_tiled(st["comp"], st["b"], st["out"], st["meta"], m, n, k, 1 / 127, 1 / 127)
    if kind == "sparse_linear":
        if case["out"] == "f16":
            return ig.w8a8_sparse_linear(st["x"], st["comp"], st["meta"], st["out"], st["sa"], st["sw"], m, n, k)
        return ig.w8a8_sparse_i32(st["x"], st["comp"], st["meta"], st["out"], m, n, k)
    if kind == "sparse_decode":
        return ig.w8a8_sparse_linear_packed(st["x"], st["packed"], st["out"], st["sa"], st["sw"], m, n, k)
    if kind == "online_quant":
        return ig.igemm_online_quant(st["a"], st["b"], st["out"], m, n, k, case["col_block"])
    return ig.hgemm_sparse_tiled(st["comp"], st["b"], st["out"], st["meta"], m, n, k, ig.BM_META_TILED)


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    kind, m = case["kind"], case["m"]
    if kind == "layer":
        bytes_, flops = 0, 0
        for _, n, k in _layer_shapes(case):
            bytes_ += 2 * m * k + n * k + 4 * n + 2 * m * n
            flops += 2 * m * n * k
        return {"bytes": bytes_, "flops": flops}
    n, k = case["n"], case["k"]
    dense, sparse = 2 * m * n * k, m * n * k          # 2:4: half of the products are known to be zero
    if kind == "gemm_i32":
        return {"bytes": m * k + n * k + 4 * m * n, "flops": dense}
    if kind == "linear":
        return {"bytes": m * k + n * k + 2 * m * n + 4 * (m + n), "flops": dense}
    if kind == "perchannel":
        return {"bytes": m * k + n * k + 4 * m * n + 8 * n, "flops": dense}
    if kind == "pertensor":
        return {"bytes": m * k + n * k + 4 * m * n, "flops": dense}
    if kind == "sparse_left":                           # the reference's words serve two rows each
        return {"bytes": m * k // 2 + m * k // 16 + n * k + 4 * m * n, "flops": sparse}
    if kind == "sparse_linear":
        return {"bytes": n * k // 2 + n * k // 8 + m * k + (2 if case["out"] == "f16" else 4) * m * n, "flops": sparse}
    if kind == "sparse_decode":
        return {"bytes": n * k // 2 + n * k // 8 + m * k + 2 * m * n + 4 * (m + n), "flops": sparse}
    if kind == "online_quant":
        return {"bytes": 2 * (m * k + n * k) + 4 * m * n, "flops": dense}
    return {"bytes": m * k + m * k // 8 + 2 * n * k + 4 * m * n, "flops": sparse}


def tolerance(case):
    kind = case["kind"]
    if kind == "gemm_i32" or (kind == "sparse_linear" and case["out"] == "i32"):
        return "exact"                                  # int32 sums
    if kind == "layer":
        return dict(_F16_LAYER)
    if kind in ("linear", "sparse_linear", "sparse_decode"):
        return dict(_F16_OUT)
    if kind in ("perchannel", "pertensor", "sparse_left"):
        return dict(_F32_SCALED)
    if kind == "online_quant":
        return dict(_F32_ONLINE)
    return dict(_F32_SUMS)
