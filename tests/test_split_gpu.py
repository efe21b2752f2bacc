"""The split-precision tensor-core passes (fp32 with up to 64 landmarks; 16-bit inputs of head_dim 16 / 32, and of
head_dim 64 with more than 64 landmarks) against the float64 oracle, with the FP32 CUDA-core kernels
as the yardstick: the same calls are made through both, and the split kernels may not be further
from the oracle than the CUDA-core ones by more than what the pseudoinverse (condition number up to a few tens
here, on other kernels too when the CUDA cores are forced) makes of the last places: bound 1.5 x yardstick + 1e-6.  16-bit
inputs: the results' own rounding (2^-12, 2^-9 relative at most) dominates both sides: bound 1.05 x yardstick + 5e-5.  What
these bounds cannot see, the exactness of the passes themselves, has tests of its own below."""
import pytest
import torch

from oracle import nystrom_oracle as O
from tests._util import run_cuda, run_oracle

pytestmark = pytest.mark.gpu

F32, F16, BF16 = torch.float32, torch.float16, torch.bfloat16

CASES = [
    # tile edges, one tile and a remainder, smallest landmark counts
    (1, 2, 127, 64, 1, 6, 0.0, F32), (1, 2, 128, 64, 64, 6, 0.0, F32), (1, 2, 129, 32, 63, 6, 5.0, F32), (1, 2, 257, 16, 5, 6, 0.0, F32),
    (1, 2, 128, 64, 65, 6, 0.0, F16), (1, 2, 129, 64, 128, 6, 5.0, BF16), (1, 2, 255, 32, 64, 6, 0.0, BF16), (1, 2, 300, 32, 65, 4, 0.0, F16),
    (1, 1, 128, 16, 128, 6, 0.0, F16), (1, 1, 16, 16, 16, 6, 0.0, BF16),
    # more slices than SMs, so that one CTA walks every tile of its slice: the running sums over many tiles
    (1, 150, 2500, 64, 64, 6, 0.0, F32), (3, 50, 1300, 64, 100, 6, 0.0, BF16), (3, 50, 1300, 32, 40, 6, 0.0, F16),
]


def _rel(a, b):
    a, b = a.detach().double().cpu(), b.double()
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("case", CASES, ids=lambda c: "x".join(str(x) for x in c[:7]) + str(c[7])[6:])
def test_split_precision_against_fp32_kernels(cuda_device, case):
    from flashnystrom_b200 import _C
    B, H, N, D, m, J, kappa, dtype = case
    q, k, v, dO = O.make_inputs(B, H, N, D, seed=9, dtype=dtype)
    got = run_cuda(q, k, v, dO, m, J, kappa)
    _C.set_force_generic(True)
    try:
        ref = run_cuda(q, k, v, dO, m, J, kappa)
    finally:
        _C.set_force_generic(False)
    slices = [0, B * H // 2, B * H - 1]
    pick = lambda t: t.reshape(1, B * H, *t.shape[2:])[:, slices]
    want = run_oracle(pick(q), pick(k), pick(v), pick(dO), m, J, kappa)
    factor, extra = (1.5, 1e-6) if dtype == F32 else (1.05, 5e-5)
    for key in ("out", "dq", "dk", "dv", "bmat", "step2", "lse1", "lse3"):
        a, b = _rel(pick(got[key]), want[key]), _rel(pick(ref[key]), want[key])
        print(key, f"{a:.2e} {b:.2e}")
        assert a <= factor * b + extra, (key, a, b)


def test_moving_reference(cuda_device):
    """Scores that grow along the sequence: the reference of the forward column pass moves in most tiles, and what has
    been summed is rescaled each time."""
    B, H, N, D, m = 1, 2, 2048, 64, 16
    q, k, v, dO = O.make_inputs(B, H, N, D, seed=2, dtype=torch.float32)
    k = k * torch.linspace(0.1, 12.0, N)[None, None, :, None]
    got = run_cuda(q, k, v, dO, m, 6, 0.0)
    want = run_oracle(q, k, v, dO, m, 6, 0.0)
    for key in ("out", "dq", "dk", "dv", "bmat", "lse3"):
        # scores of about 100: 2^-24 of them is an error of 6e-6 in a probability, several of which meet in a gradient
        assert _rel(got[key], want[key]) <= 1e-4, (key, _rel(got[key], want[key]))


@pytest.mark.parametrize("case", [
    (1, 2, 128, 64, 65, 6, 0.0, 1.0, F16), (2, 4, 2000, 64, 128, 6, 0.0, 1.0, BF16), (1, 4, 2000, 64, 128, 6, 5.0, 3.0, F16),
    (1, 4, 1500, 32, 100, 6, 0.0, 2.0, F16), (1, 4, 1000, 32, 64, 6, 0.0, 4.0, F16), (1, 4, 1500, 16, 64, 6, 0.0, 4.0, BF16),
], ids=lambda c: "x".join(str(x) for x in c[:8]) + str(c[8])[6:])
def test_16bit_inputs_keep_fp32_operands(cuda_device, case):
    """The FP32 results of the forward passes (16-bit outputs would hide a loss) for 16-bit inputs, large scores among
    them: no further from the oracle than the CUDA-core kernels, which multiply in FP32.  Every operand has 24 bits on
    both sides; what differs is the order and rounding of the sums: bound 1.15 x yardstick, for the spread of a few slices;
    2 x for step2, whose pseudoinverse comes from other kernels too when the CUDA cores are forced.  (Operands of 16 bits are
    4 to 18 x off, at scores of about 30 an error of 1e-4 in single probabilities.)"""
    from flashnystrom_b200 import _C
    B, H, N, D, m, J, kappa, qk, dtype = case
    q, k, v, dO = O.make_inputs(B, H, N, D, seed=4, dtype=torch.float32)
    q, k, v, dO = (q * qk).to(dtype), (k * qk).to(dtype), v.to(dtype), dO.to(dtype)
    got = run_cuda(q, k, v, dO, m, J, kappa)
    _C.set_force_generic(True)
    try:
        ref = run_cuda(q, k, v, dO, m, J, kappa)
    finally:
        _C.set_force_generic(False)
    want = run_oracle(q, k, v, dO, m, J, kappa)
    for key in ("bmat", "step2", "lse1", "lse3"):
        a, b = _rel(got[key], want[key]), _rel(ref[key], want[key])
        print(key, f"{a:.2e} {b:.2e}")
        assert a <= (2 if key == "step2" else 1.15) * b, (key, a, b)


@pytest.mark.parametrize("B,H,N,D,m", [(1, 4, 1024, 64, 32), (2, 2, 4096, 64, 64), (1, 8, 2000, 16, 64), (1, 4, 3000, 32, 33)])
def test_fp32_row_sums(cuda_device, B, H, N, D, m):
    """lse1 of fp32 inputs, over three seeds, at the CUDA-core kernels' error: both round it once more than the sum and the
    scores it comes from.  The bound, 1.15 x, is for the spread of a few thousand rows; with scores in units of log 2 and
    ex2.approx it was 1.23 to 1.53 x."""
    from flashnystrom_b200 import _C
    err = {False: 0.0, True: 0.0}
    for seed in range(3):
        q, k, v, _ = O.make_inputs(B, H, N, D, seed=seed, dtype=F32)
        want = O.forward(q.double(), k.double(), v.double(), m, 6)["lse1"]
        for generic in err:
            _C.set_force_generic(generic)
            try:
                got = _C.forward(q.cuda(), k.cuda(), v.cuda(), m, 6)[7]
            finally:
                _C.set_force_generic(False)
            err[generic] += _rel(got, want) ** 2
    print(err)
    assert err[False] <= 1.15 ** 2 * err[True]


def test_fp32_values_past_the_largest_bf16(cuda_device):
    """A value that rounds to infinity in bf16, under a weight of e^-60: finite on the CUDA cores, and here."""
    from flashnystrom_b200 import _C
    N, D, m, n = 256, 64, 8, 77
    q, k, v, dO = O.make_inputs(1, 1, N, D, seed=3, dtype=torch.float32)
    q = 0.1 * q + 0.5
    k = 0.1 * k
    k[0, 0, n] -= 15.0                       # scores of about -60 with every landmark query
    v[0, 0, n, ::2], v[0, 0, n, 1::2] = 3.4e38, -3.4e38
    got = run_cuda(q, k, v, dO, m, 6, 0.0)
    _C.set_force_generic(True)
    try:
        ref = run_cuda(q, k, v, dO, m, 6, 0.0)
    finally:
        _C.set_force_generic(False)
    want = run_oracle(q, k, v, dO, m, 6, 0.0)
    for key in ("bmat", "out"):
        assert torch.isfinite(ref[key]).all() and torch.isfinite(got[key]).all()
        # a score of 60 is off by about 60 * 2^-22, which the pseudoinverse amplifies some tens of times
        assert _rel(got[key], want[key]) <= 1e-3, key


@pytest.mark.parametrize("bad", [float("inf"), float("-inf"), float("nan")])
@pytest.mark.parametrize("dtype,D,m", [(F32, 64, 32), (F16, 32, 64), (BF16, 64, 100)])
def test_infinities_and_nan_stay_where_the_fp32_kernels_have_them(cuda_device, bad, dtype, D, m):
    """One bad element of V reaches its own column of the output and no other; one of Q or K reaches every output of its
    slice and nothing of the next slice.  What is finite on the CUDA cores is finite here, and the other way round."""
    from flashnystrom_b200 import _C
    for which in range(3):
        t = list(O.make_inputs(1, 2, 300, D, seed=13, dtype=F32))
        t[which][0, 0, 150, 5] = bad
        q, k, v, _ = (x.to(dtype).cuda() for x in t)
        got = _C.forward(q, k, v, m, 6)[0]
        _C.set_force_generic(True)
        try:
            ref = _C.forward(q, k, v, m, 6)[0]
        finally:
            _C.set_force_generic(False)
        assert torch.equal(torch.isfinite(got), torch.isfinite(ref))
        assert torch.isfinite(got[0, 1]).all()
        assert torch.isfinite(got[0, 0]).all(0).sum() == (D - 1 if which == 2 else 0)
    torch.cuda.synchronize()
    _C.check_device_status()


@pytest.mark.parametrize("B,H,N,D,m,qk", [(1, 4, 1024, 64, 32, 64 ** -0.25), (2, 2, 4096, 64, 64, 1.0), (1, 4, 3000, 32, 33, 1.0), (1, 8, 700, 64, 48, 2.0),
                                           (1, 8, 2000, 16, 64, 1.0), (4, 16, 128, 64, 64, 1.0), (1, 2, 20000, 64, 64, 1.0)])
def test_fp32_passes_are_as_exact_as_the_cuda_cores(cuda_device, B, H, N, D, m, qk):
    """What the passes make of the landmark tensors that the call itself saved, against the same in 64 bits, so that the
    pseudoinverse's error is no part of it; four seeds.  Bound 1.15 x the CUDA-core kernels' error, for the spread between
    seeds.  (With each product in one accumulator of the tensor core, which truncates, the output and dV are 1.2 to 1.4 x
    as far off.)"""
    from flashnystrom_b200 import _C
    s = float(torch.tensor(D ** -0.25, dtype=F32))
    err = {}
    for seed in range(4):
        q, k, v, dO = (t.cuda() for t in O.make_inputs(B, H, N, D, seed=seed, dtype=F32))
        q, k = q * qk, k * qk
        for generic in (False, True):
            _C.set_force_generic(generic)
            try:
                got = run_cuda(q, k, v, dO, m, 6)
            finally:
                _C.set_force_generic(False)
            x = {key: t.double() for key, t in got.items()}
            s1, s3 = (q.double() * s) @ x["kt"].transpose(-2, -1), x["qt"] @ (k.double() * s).transpose(-2, -1)
            p1, p3 = torch.softmax(s1, -1), torch.softmax(s3, -1)
            d_o3 = x["k2inv"].transpose(-2, -1) @ (p1.transpose(-2, -1) @ dO.double())
            want = dict(lse1=torch.logsumexp(s1, -1), lse3=torch.logsumexp(s3, -1), bmat=p3 @ v.double(), out=p1 @ x["step2"],
                        dv=p3.transpose(-2, -1) @ d_o3)
            for key, w in want.items():
                err[key, generic] = err.get((key, generic), 0.0) + float((x[key] - w).norm() / w.norm()) ** 2
    for key in want:
        print(key, f"{(err[key, False] / 4) ** 0.5:.2e} {(err[key, True] / 4) ** 0.5:.2e} {(err[key, False] / err[key, True]) ** 0.5:.2f}")
    for key in want:
        assert err[key, False] <= 1.15 ** 2 * err[key, True], key
