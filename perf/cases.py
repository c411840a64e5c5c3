"""What the W4A4 linear is timed on: the calls a user's program makes, over the sizes and options it makes them with.

Shapes are those of the benchmark configurations and small-row workloads of svdquant_kernels_b200/workloads.py, and
ragged sizes between them.  Values follow the same distributions: Gaussian activations (GELU'd in front of a down
projection) with a few outlier columns, smooth = sqrt(column amax), weights N(0, 0.02) / smooth, LoRA factors
N(0, 1/sqrt(K)) and N(0, 0.01).

Kinds of a case:
  linear      x on the GPU -> quantize_w4a4_act_fuse_lora -> gemm_w4a4: one layer's forward pass ("api": the Python
              operators, or the registered torch.ops.svdq_b200 ones a serving stack calls)
  next        the same, with the GEMM also packing the next layer's activations (smooth_next)
  pack        quantize_nvfp4_rows of a weight matrix, as at model load
  host        LinearPlan.forward_host: x and y in pinned host memory
"""
import math

import torch

import svdquant_kernels_b200 as svdq
from svdquant_kernels_b200 import torch_ops  # noqa: F401  (registers torch.ops.svdq_b200)

DT = {"f16": torch.float16, "bf16": torch.bfloat16, "f32": torch.float32}
MAX_M, MAX_K, MAX_N = 4352, 15360, 15360
MAX_MKN = 4352 * 3840 * 15360
MAX_PACK = 15360 * 3840


def _linear(name, M, K, N, R, dtype, **more):
    case = {"name": name, "kind": "linear", "M": M, "K": K, "N": N, "R": R, "dtype": dtype, "act": "gauss", "smooth": True,
            "wcscales": True, "bias": True, "api": "python"}
    case.update(more)
    return case


def listed():
    return [
        # the smallest layer of the test configurations: latency and launches
        _linear("tiny-64x128x128-f16", 64, 128, 128, 16, "f16"),
        # a few hundred rows (a text prompt's tokens, a small image): short K, and a long-K down projection
        _linear("rows256-3840x3072-f16", 256, 3840, 3072, 128, "f16"),
        _linear("rows256-15360x3840-bf16", 256, 15360, 3840, 128, "bf16", act="gelu"),
        # the same through the dispatcher, as a serving stack that resolves kernels by name calls it
        _linear("rows256-10240x3072-ops-f16", 256, 10240, 3072, 32, "f16", api="ops"),
        # a ragged number of rows, no bias, a rank between the usual ones
        _linear("ragged-1003x3840x3072-bf16", 1003, 3840, 3072, 64, "bf16", bias=False),
        # the four benchmark layers: attention projection, up and down projection, long-K projection
        _linear("proj-4352x3840x3072-f16", 4352, 3840, 3072, 128, "f16"),
        _linear("up-4352x3840x15360-bf16", 4352, 3840, 15360, 128, "bf16"),
        _linear("down-4352x15360x3840-bf16", 4352, 15360, 3840, 128, "bf16", act="gelu"),
        _linear("long-4352x10240x3072-f16", 4352, 10240, 3072, 32, "f16"),
        # two linears in a row: the first one's GEMM packs the second one's activations
        _linear("next-4352x3840x3072-f16", 4352, 3840, 3072, 128, "f16", kind="next"),
        # packing the largest weight matrix from the fp32 it is trained or smoothed in
        {"name": "pack-15360x3840-f32", "kind": "pack", "rows": 15360, "K": 3840, "dtype": "f32"},
        # activations that live on the host
        _linear("host-4352x3840x3072-f16", 4352, 3840, 3072, 128, "f16", kind="host"),
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choices(["linear", "next", "pack", "host"], [7, 1, 1, 1])[0]
    if kind == "pack":
        rows = _log_int(rng, 128, MAX_N)
        K = 16 * _log_int(rng, 8, min(MAX_K, MAX_PACK // rows) // 16)
        return {"kind": kind, "rows": rows, "K": K, "dtype": rng.choice(["f32", "bf16", "f16"])}
    M = _log_int(rng, 1, MAX_M)
    K = 64 * _log_int(rng, 2, MAX_K // 64)
    N = 128 * _log_int(rng, 1, MAX_N // 128)
    if kind != "linear":                       # at most what the largest such case above moves and computes
        K, N = min(K, 3840), min(N, 3072)
    while _padded(M) * K * N > MAX_MKN:
        if K > N:
            K = max(128, K // 2 // 64 * 64)
        else:
            N = max(128, N // 2 // 128 * 128)
    return {"kind": kind, "M": M, "K": K, "N": N, "R": rng.choice([16, 32, 48, 64, 96, 128, 128, 256]),
            "dtype": rng.choice(["f16", "bf16"]), "act": rng.choice(["gauss", "gelu"]),
            "smooth": kind == "host" or rng.random() < 0.9, "wcscales": rng.random() < 0.8, "bias": rng.random() < 0.7,
            "api": rng.choice(["python", "python", "ops"]) if kind == "linear" else "python"}


def _padded(M):
    return -(-M // 256) * 256


def prepare(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    dtype = DT[case["dtype"]]

    def randn(*shape):
        return torch.randn(*shape, generator=g, device="cuda", dtype=torch.float32)

    if case["kind"] == "pack":
        w = randn(case["rows"], case["K"]) * 0.02
        w /= torch.rand(case["K"], generator=g, device="cuda") + 0.5
        return {"kind": "pack", "w": w.to(dtype)}

    M, K, N, R = case["M"], case["K"], case["N"], case["R"]
    outliers = torch.randperm(K, generator=g, device="cuda")[:4]

    def activations(rows):
        x = randn(rows, K)
        if case["act"] == "gelu":
            x = torch.nn.functional.gelu(x)
        x[:, outliers] *= 20.0
        return x

    x = activations(M).to(dtype)
    smooth = activations(256).abs().amax(0).sqrt().clamp_min(1e-2)
    w = randn(N, K) * 0.02
    if case["smooth"]:
        w /= smooth
    wgt, wscales = svdq.quantize_nvfp4_rows(w, pad_size=1)
    del w
    s = {"kind": case["kind"], "api": case["api"], "dtype": dtype, "x": x, "wgt": wgt, "wscales": wscales,
         "lora_down": (randn(K, R) / K ** 0.5).to(dtype), "lora_up": (randn(N, R) * 0.01).to(dtype),
         "smooth": smooth.to(dtype) if case["smooth"] else None,
         "wcscales": (torch.rand(N, generator=g, device="cuda") + 0.5).to(dtype) if case["wcscales"] else None,
         "bias": (randn(N) * 0.01).to(dtype) if case["bias"] else None}
    if case["kind"] == "next":
        s["smooth_next"] = (torch.rand(N, generator=g, device="cuda") * 1.5 + 0.25).to(dtype)
    if case["kind"] == "host":
        plan = svdq.LinearPlan(M, K, N, R, dtype, wgt=wgt, wscales=wscales, lora_down=s["lora_down"], lora_up=s["lora_up"],
                               smooth=s["smooth"], wcscales=s["wcscales"], bias=s["bias"])
        x_host = torch.empty(M, K, dtype=dtype, pin_memory=True)
        x_host.copy_(x)
        s = {"kind": "host", "plan": plan, "x": x_host, "y": torch.empty(M, N, dtype=dtype, pin_memory=True)}
    return s


def run(s):
    kind = s["kind"]
    if kind == "pack":
        packed, scales = svdq.quantize_nvfp4_rows(s["w"], pad_size=1)
        return {"packed": packed, "scales": scales}
    if kind == "host":
        return {"y": s["plan"].forward_host(s["x"], s["y"])}
    if s["api"] == "ops":
        act, ascales, lora_act = torch.ops.svdq_b200.quantize_w4a4_act_fuse_lora(s["x"], s["lora_down"], s["smooth"])
        y = torch.ops.svdq_b200.gemm_w4a4(act, s["wgt"], ascales, s["wscales"], lora_act, s["lora_up"], s["wcscales"],
                                          s["bias"], s["dtype"])
        return {"act": act, "ascales": ascales, "lora_act": lora_act, "y": y}
    act, ascales, lora_act = svdq.quantize_w4a4_act_fuse_lora(s["x"], s["lora_down"], s["smooth"])
    if kind == "next":
        y, qout, oscales = svdq.gemm_w4a4(act, s["wgt"], ascales, s["wscales"], lora_act, s["lora_up"], s["wcscales"],
                                          s["bias"], s["dtype"], smooth_next=s["smooth_next"])
        return {"act": act, "ascales": ascales, "lora_act": lora_act, "y": y, "qout": qout, "oscales": oscales}
    y = svdq.gemm_w4a4(act, s["wgt"], ascales, s["wscales"], lora_act, s["lora_up"], s["wcscales"], s["bias"], s["dtype"])
    return {"act": act, "ascales": ascales, "lora_act": lora_act, "y": y}


def work(case):
    """Each input read once, each output written once; products at their unpadded sizes."""
    if case["kind"] == "pack":
        rows, K = case["rows"], case["K"]
        return {"bytes": rows * K * DT[case["dtype"]].itemsize + rows * K // 2 + rows * K // 16, "flops": rows * K}
    M, K, N, R = case["M"], case["K"], case["N"], case["R"]
    Mp = _padded(M)
    weights = N * K // 2 + N * K // 16 + (K + N) * R * 2
    columns = 2 * K * case["smooth"] + 2 * N * (case["wcscales"] + case["bias"] + (case["kind"] == "next"))
    flops = 2 * M * K * N + 2 * M * K * R + 2 * M * N * R
    if case["kind"] == "host":                       # codes, scales and lora_act stay inside; weights stay resident
        return {"bytes": weights + columns + M * K * 2 + M * N * 2, "flops": flops}
    outputs = Mp * K // 2 + Mp * K // 16 + Mp * R * 4 + Mp * N * 2
    if case["kind"] == "next":
        outputs += Mp * N // 2 + Mp * N // 16
    return {"bytes": weights + columns + M * K * 2 + outputs, "flops": flops}


def tolerance(case):
    """Codes and scales of the quantizer are exact; lora_act is an fp32 sum, y an fp32 sum rounded to 16 bits: a sum in
    another order moves some values by one unit in the last place (2^-10 for f16, 2^-7 for bf16 at most)."""
    if case["kind"] == "pack":
        return "exact"
    t = {"rel": 5e-4, "max": 4e-3} if case["dtype"] == "f16" else {"rel": 3e-3, "max": 2e-2}
    if case["kind"] == "next":
        # qout / oscales are packed from that fp32 sum: a value next to a rounding bound may take the neighbouring code,
        # and a scale the neighbouring e4m3 value (an eighth away)
        t = {"rel": 3e-3, "max": 0.2, "differ": 1e-3}
    return t
