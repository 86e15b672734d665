"""Timing cases of the block-FP8 path: the calls a user's program makes, from the public package.

A case names one entry point and its sizes:

    op = "matmul"        w8a8_block_fp8_matmul on activations quantised beforehand
    op = "linear"        fp8_linear: bf16 activations in, quantised and multiplied
    op = "rowscale"      deep_gemm.gemm_fp8_fp8_bf16_nt: one weight scale per row
    op = "act_quant"     fp8_act_quant, per token and 128-wide group
    op = "weight_quant"  fp8_weight_quant, per 128 x 128 block

M tokens, N weight rows (output features), K input features; "fp32" asks for an fp32 result where the
entry point has the choice (its default), otherwise the result is bf16. Activations are N(0, 1),
weights N(0, 0.02), both bf16 before quantisation.
"""
import math

import torch

import hf_kernels_helion_b200 as pkg
from hf_kernels_helion_b200 import deep_gemm

BLOCK = [128, 128]
# The ranges that the listed cases stand for: one token to a prefill batch, a narrow projection to the
# 28672-wide MLP up-projection, and the products of both up to the 8192 x 18432 x 7168 MLP.
MAX_M, MIN_N, MAX_N, MIN_K, MAX_K = 8192, 128, 28672, 256, 8192
MAX_MNK = 8192 * 18432 * 7168


def listed():
    return [
        # one decoded token through a small layer: launches and host work are all there is
        {"name": "linear_m4_small", "op": "linear", "M": 4, "N": 2560, "K": 2048, "fp32": False},
        # one decoded token through a 70B-class MLP up-projection: the weight is read once, from HBM
        {"name": "linear_m1_mlp", "op": "linear", "M": 1, "N": 28672, "K": 8192, "fp32": False},
        # the same layer for an odd decode batch, activations quantised by an earlier layer
        {"name": "matmul_m37_mlp", "op": "matmul", "M": 37, "N": 28672, "K": 8192, "fp32": False},
        # a large decode batch (or a short prompt): between bandwidth and tensor bound
        {"name": "matmul_m256_mlp", "op": "matmul", "M": 256, "N": 28672, "K": 8192, "fp32": False},
        # the smallest benchmark shape, with the entry point's default fp32 result
        {"name": "matmul_512_fp32", "op": "matmul", "M": 512, "N": 512, "K": 2048, "fp32": True},
        # medium square shape: less than one wave of large tiles
        {"name": "matmul_2048", "op": "matmul", "M": 2048, "N": 2048, "K": 4096, "fp32": False},
        # a prompt of odd length, feature counts that no tile divides, a short last K block
        {"name": "matmul_ragged", "op": "matmul", "M": 1611, "N": 7000, "K": 4208, "fp32": False},
        # the compute-bound benchmark shape
        {"name": "matmul_4096", "op": "matmul", "M": 4096, "N": 4096, "K": 8192, "fp32": False},
        # a whole prefill step of a wide MLP, bf16 activations in
        {"name": "linear_prefill_mlp", "op": "linear", "M": 8192, "N": 18432, "K": 7168, "fp32": False},
        # the row-scaled weight layout at the same shape as matmul_4096
        {"name": "rowscale_4096", "op": "rowscale", "M": 4096, "N": 4096, "K": 8192, "fp32": False},
        # the quantiser in front of a prefill matmul
        {"name": "act_quant_4096", "op": "act_quant", "M": 4096, "N": 0, "K": 8192, "fp32": False},
        # converting one weight at load time
        {"name": "weight_quant_mlp", "op": "weight_quant", "M": 0, "N": 18432, "K": 7168, "fp32": False},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _multiple(n, of, lo):
    return max(lo, n // of * of)


def draw(rng):
    op = rng.choice(["matmul"] * 4 + ["linear"] * 3 + ["rowscale", "act_quant", "weight_quant"])
    while True:
        m = _log(rng, 1, MAX_M)
        # feature counts: mostly multiples of 128, some of 16 (sharded or pruned layers)
        n = _multiple(_log(rng, MIN_N, MAX_N), rng.choice([128, 128, 16]), MIN_N)
        k = _multiple(_log(rng, MIN_K, MAX_K), rng.choice([128, 128, 16]), MIN_K)
        if m * n * k <= MAX_MNK:
            break
    if op == "act_quant":
        n = 0
    if op == "weight_quant":
        m = 0
    return {"op": op, "M": m, "N": n, "K": k, "fp32": op == "matmul" and rng.random() < 0.25}


def prepare(case, seed):
    op, m, n, k = case["op"], case["M"], case["N"], case["K"]
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(seed)
    state = {"op": op, "dtype": torch.float32 if case["fp32"] else torch.bfloat16}
    if op != "weight_quant":
        x = torch.randn(m, k, generator=g, device=dev, dtype=torch.bfloat16)
        if op in ("act_quant", "linear"):
            state["x"] = x
        else:
            state["A"], state["As"] = pkg.fp8_act_quant(x)
    if op != "act_quant":
        w = torch.randn(n, k, generator=g, device=dev, dtype=torch.bfloat16).mul_(0.02)
        if op == "weight_quant":
            state["w"] = w
        elif op == "rowscale":
            state["B"], state["Bs"] = pkg.fp8_act_quant(w)
        else:
            state["B"], state["Bs"] = pkg.fp8_weight_quant(w)
    return state


def run(state):
    op = state["op"]
    if op == "matmul":
        return pkg.w8a8_block_fp8_matmul(state["A"], state["B"], state["As"], state["Bs"], BLOCK, state["dtype"])
    if op == "linear":
        return pkg.fp8_linear(state["x"], state["B"], state["Bs"])
    if op == "rowscale":
        return deep_gemm.gemm_fp8_fp8_bf16_nt(state["A"], state["B"], state["As"], state["Bs"])
    if op == "act_quant":
        return pkg.fp8_act_quant(state["x"])
    return pkg.fp8_weight_quant(state["w"])


def _groups(x):
    """[rows, K] bf16 -> (e4m3 values, fp32 scale) per 128-wide group, as [rows, groups, 128] and [rows, groups, 1]."""
    rows, k = x.shape
    x = torch.nn.functional.pad(x.float(), (0, -k % 128)).view(rows, -1, 128)
    s = x.abs().amax(2, keepdim=True)
    s = s / torch.full_like(s, 448.0)   # (a scalar divisor would become a multiplication by its reciprocal)
    return torch.where(s > 0, x / s, torch.zeros_like(x)).to(torch.float8_e4m3fn), s


def _blocks(w):
    """[N, K] bf16 -> (e4m3 values, fp32 scale) per 128 x 128 block, as [Nb, 128, Kb, 128] and [Nb, 1, Kb, 1]."""
    n, k = w.shape
    w = torch.nn.functional.pad(w.float(), (0, -k % 128, 0, -n % 128)).view(-(-n // 128), 128, -(-k // 128), 128)
    s = w.abs().amax((1, 3), keepdim=True)
    s = s / torch.full_like(s, 448.0)
    return torch.where(s > 0, w / s, torch.zeros_like(w)).to(torch.float8_e4m3fn), s


def exact(case, seed):
    op, m, n, k = case["op"], case["M"], case["N"], case["K"]
    dev = torch.device("cuda", 0)
    g = torch.Generator(device=dev).manual_seed(seed)
    if op != "weight_quant":
        qx, sx = _groups(torch.randn(m, k, generator=g, device=dev, dtype=torch.bfloat16))
        if op == "act_quant":
            return None, sx.double()[:, :, 0]   # the bytes are compared as such
    w = torch.randn(n, k, generator=g, device=dev, dtype=torch.bfloat16).mul_(0.02)
    qw, sw = _groups(w) if op == "rowscale" else _blocks(w)
    if op == "weight_quant":
        return None, sw.double()[:, 0, :, 0]
    a = (qx.double() * sx.double()).view(m, -1)
    b = (qw.double() * sw.double()).view(-1, a.shape[1])[:n]
    return a @ b.T


def work(case):
    op, m, n, k = case["op"], case["M"], case["N"], case["K"]
    kb, nb = -(-k // 128), -(-n // 128)
    if op == "act_quant":
        return {"bytes": m * (3 * k + 4 * kb), "flops": 0}
    if op == "weight_quant":
        return {"bytes": 3 * n * k + 4 * nb * kb, "flops": 0}
    activations = 2 * m * k if op == "linear" else m * (k + 4 * kb)
    weight = n * k + 4 * kb * (n if op == "rowscale" else nb)
    return {"bytes": activations + weight + m * n * (4 if case["fp32"] else 2), "flops": 2 * m * n * k}


def tolerance(case):
    if case["op"] in ("act_quant", "weight_quant"):
        return "exact"
    if case["fp32"]:
        # against the same products summed in fp64: rel 0.8e-7 .. 1.5e-7, max 0.5e-6 .. 1.2e-6
        return {"rel": 6e-7, "max": 5e-6}
    # a bf16 result rounds each element once: rel 1.66e-3, max 3.9e-3 (2^-8) against fp64
    return {"rel": 6.6e-3, "max": 1.6e-2}
