"""The work that a user has this framework do, as cases that can be prepared, run and checked.

Two entry points are covered, each forward alone (inference) and forward with backward (training):
`flash_nystrom_attention` on (B, H, N, D) tensors and the `FlashNystromAttention` module on (B, N, dim)
activations.  The ranges: sequences of 128 to 65536 rows, one to 512 (batch, head) slices, head
sizes 32, 64 and 128, 16 to 128 landmarks, 4 to 8 Newton-Schulz iterations, with and without the ridge,
fp16, bf16 and fp32.  Sizes come from the repository's configurations, tests and benchmark.

    listed()             the named cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  inputs (and the module) on the GPU, from the seed alone
    run(state)           one pass, returning everything it computes
    work(case)           bytes and operations the pass cannot do without
    tolerance(case)      how far another correct implementation may be off
"""
import math

import torch

from flashnystrom_b200 import FlashNystromAttention, NystromConfig, flash_nystrom_attention

DTYPES = {"fp16": torch.float16, "bf16": torch.bfloat16, "fp32": torch.float32}
BYTES = {"fp16": 2, "bf16": 2, "fp32": 4}


def _op(name, dtype, train, B, H, N, D, m, J=6, kappa=0.0, qk_scale=1.0):
    return {"name": name, "path": "op", "dtype": dtype, "train": train, "B": B, "H": H, "N": N, "D": D, "m": m,
            "J": J, "kappa": kappa, "qk_scale": qk_scale}


def _module(name, dtype, train, B, heads, N, D, m, J=6, kappa=0.0, conv=3):
    return {"name": name, "path": "module", "dtype": dtype, "train": train, "B": B, "H": heads, "N": N, "D": D, "m": m,
            "J": J, "kappa": kappa, "conv": conv}


def listed():
    return [
        # one short prompt through a small model: launches and host time are all there is
        _op("infer_small", "fp16", False, 1, 2, 256, 64, 32),
        # the smallest training step, full precision (the CPU-runnable configuration)
        _op("train_small_fp32", "fp32", True, 1, 4, 1024, 64, 32, qk_scale=64 ** -0.25),
        # an ordinary training batch
        _op("train_4k", "fp16", True, 4, 8, 4096, 64, 64),
        # the same inside the attention block: projections and the depthwise residual around it
        _module("module_train_4k", "fp16", True, 4, 8, 4096, 64, 64),
        # serving the block on one document of odd length
        _module("module_infer_ragged", "bf16", False, 1, 8, 9999, 64, 64),
        # a large batch of short sequences, no multiple of a tile or of the landmark count
        _op("train_many_short", "bf16", True, 32, 16, 2000, 64, 64),
        # the long-sequence configuration, the benchmark's workload
        _op("train_64k", "fp16", True, 1, 16, 65536, 64, 64),
        # encoding one long sequence of odd length, odd numbers of heads and landmarks
        _op("infer_long_ragged", "bf16", False, 1, 7, 50001, 64, 33),
        # the large-landmark configuration: wide heads, 128 landmarks, eight iterations, ridge
        _op("train_128_landmarks", "fp16", True, 2, 8, 16384, 128, 128, J=8, kappa=5.0),
        # wide heads at the size of the reference's latency table, with its ridge
        _op("train_wide_heads", "fp16", True, 4, 16, 16384, 128, 64, kappa=5.0),
        # full precision at length
        _op("train_fp32", "fp32", True, 1, 16, 16384, 64, 64),
        # the usual head size with the largest landmark count
        _op("train_d64_128_landmarks", "bf16", True, 2, 8, 8192, 64, 128),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# a drawn case stays below the largest listed ones: elements of one (B, H, N, D) tensor, and elements times
# landmarks for full precision, whose products count for more
_MAX_ELEMENTS = 4 * 16 * 16384 * 128
_MAX_FP32_PRODUCT = 16 * 16384 * 64 * 64


def draw(rng):
    train = rng.random() < 0.65
    if rng.random() < 0.25:
        heads = rng.choice([4, 8, 12, 16])
        D = rng.choice([64, 64, 128])
        N = _log_int(rng, 256, 16384)
        B = _log_int(rng, 1, min(16, max(1, (1 << 25) // (heads * N * D))))
        m = rng.choice([32, 64, 64, rng.randint(16, 64)])
        return {k: v for k, v in _module("", rng.choice(["fp16", "bf16"]), train, B, heads, N, D, min(m, N), rng.randint(4, 8),
                                         rng.choice([0.0, 0.0, 5.0]), rng.choice([0, 3, 3, 7, 33])).items() if k != "name"}
    dtype = rng.choice(["fp16", "fp16", "fp16", "bf16", "bf16", "fp32"])
    D = rng.choice([64, 64, 64, 128, 128, 32])
    m = rng.choice([64, 64, 32, rng.randint(16, 64), rng.randint(65, 128), 128])
    while True:
        N = _log_int(rng, 128, 65536)
        N -= rng.choice([0, 0, N % 64])     # two of three as they fall, one a multiple of 64
        B, H = _log_int(rng, 1, 32), _log_int(rng, 1, 16)
        elements = B * H * N * D
        if N >= m and elements <= _MAX_ELEMENTS and (dtype != "fp32" or elements * m <= _MAX_FP32_PRODUCT):
            break
    case = _op("", dtype, train, B, H, N, D, m, rng.randint(4, 8), rng.choice([0.0, 0.0, 5.0]))
    del case["name"]
    return case


def prepare(case, seed):
    dev, dtype = torch.device("cuda", torch.cuda.current_device()), DTYPES[case["dtype"]]
    gen = torch.Generator(device=dev).manual_seed(seed)

    def normal(*shape, scale=1.0):
        return (torch.randn(*shape, generator=gen, device=dev) * scale).to(dtype)

    B, H, N, D, train = case["B"], case["H"], case["N"], case["D"], case["train"]
    if case["path"] == "op":
        s = case["qk_scale"]
        q, k, v = normal(B, H, N, D, scale=s), normal(B, H, N, D, scale=s), normal(B, H, N, D)
        if train:
            q, k, v = (t.requires_grad_(True) for t in (q, k, v))
        options = {"num_landmarks": case["m"], "newton_iter": case["J"], "kappa_star": case["kappa"]}
        return {"case": case, "q": q, "k": k, "v": v, "options": options, "d_out": normal(B, H, N, D) if train else None}
    dim = H * D
    config = NystromConfig(num_landmarks=case["m"], newton_iter=case["J"], kappa_star=case["kappa"],
                           conv_kernel_size=case["conv"], use_conv_residual=case["conv"] > 0)
    with torch.device(dev):
        module = FlashNystromAttention(dim, heads=H, config=config).to(dtype)
    with torch.no_grad():
        for name, p in module.named_parameters():
            p.copy_(normal(*p.shape, scale=0.02 if name == "conv_weight" else dim ** -0.5))
    x = normal(B, N, dim)
    if train:
        x.requires_grad_(True)
    return {"case": case, "module": module, "x": x, "d_out": normal(B, N, dim) if train else None}


def run(state):
    case = state["case"]
    if case["path"] == "op":
        q, k, v = state["q"], state["k"], state["v"]
        if not case["train"]:
            with torch.no_grad():
                return flash_nystrom_attention(q, k, v, **state["options"])
        q.grad = k.grad = v.grad = None
        out = flash_nystrom_attention(q, k, v, **state["options"])
        out.backward(state["d_out"])
        return out.detach(), q.grad, k.grad, v.grad
    module, x = state["module"], state["x"]
    if not case["train"]:
        with torch.no_grad():
            return module(x)
    module.zero_grad(set_to_none=True)
    x.grad = None
    y = module(x)
    y.backward(state["d_out"])
    return [y.detach(), x.grad] + [p.grad for p in module.parameters()]


def work(case):
    """Each input read once, each output written once; the products of the three softmaxes and of the
    pseudoinverse, forward and (with the scores formed again) backward; the projections of the module."""
    B, H, N, D, m, J, train = case["B"], case["H"], case["N"], case["D"], case["m"], case["J"], case["train"]
    size, BH = BYTES[case["dtype"]], case["B"] * case["H"]
    # S1 = Q Kt^T, S3 = Qt K^T, P3 V, P1 step2; backward: S1, S3, dP1, dP3, dstep2, dKt, dQ, dV, dK, dQt
    flops = BH * 2.0 * N * m * D * (14 if train else 4)
    # four products of m^3 per iteration; about eight more in its backward
    flops += BH * 2.0 * m ** 3 * J * (12 if train else 4)
    if case["path"] == "op":
        return {"bytes": size * BH * N * D * (8 if train else 4), "flops": flops}
    dim = H * D
    weights = 4 * dim * dim + H * case["conv"]
    flops += 2.0 * B * N * dim * (4 * dim + case["conv"]) * (3 if train else 1)
    return {"bytes": size * (B * N * dim * (4 if train else 2) + weights * (2 if train else 1)), "flops": flops}


# The largest relative error (2-norm) of any output against the CPU oracle evaluated in 64 bits on the same
# inputs, over the listed and some ninety drawn cases on a B200, was 1.9e-3 in fp16 (a weight gradient of the
# module), 8.2e-3 in bf16 (dQ, whose softmax Jacobians are rounded to the inputs' type) and 3.1e-6 in fp32 (dQ).
# Stated is about four times that.
_REL = {"fp16": 8e-3, "bf16": 3.2e-2, "fp32": 1.2e-5}


def tolerance(case):
    return {"rel": _REL[case["dtype"]]}
