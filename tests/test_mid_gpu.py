"""The landmark-sized stages for more than 64 landmarks on the tensor cores, against the float64 oracle with the
CUDA-core kernels as the yardstick.  FP32 inputs run the same streaming passes on both sides, so only these stages
differ.  Operands keep 24 bits in three bf16 terms.  The accumulator truncates: the eight K steps of a product lose up
to 8 * 2^-24, all in one direction, where the yardstick's 128 rounded additions lose about sqrt(128) / 2 * 2^-24
= 6 * 2^-24 in either direction; both are amplified alike by the iterations, but a bias adds up over the terms of the
sums that follow (up to sqrt(64) = 8 times) where rounding averages out: bound 8 x yardstick + 1e-6."""
import pytest
import torch

from oracle import nystrom_oracle as O
from tests._util import run_cuda, run_oracle

pytestmark = pytest.mark.gpu


def _rel(a, b):
    a, b = a.detach().double().cpu(), b.double()
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("B,H,N,D,m,J,kappa", [
    (1, 2, 65, 16, 65, 1, 0.0), (1, 2, 200, 32, 96, 6, 0.0), (1, 3, 257, 64, 127, 6, 5.0), (1, 2, 300, 128, 128, 8, 0.0),
    (1, 1, 131, 128, 66, 20, 1e3),      # the largest iteration count
    (2, 50, 150, 64, 100, 4, 5.0),      # more slices than run at once
])
def test_against_cuda_core_stages(cuda_device, B, H, N, D, m, J, kappa):
    from flashnystrom_b200 import _C
    q, k, v, dO = O.make_inputs(B, H, N, D, seed=3, dtype=torch.float32)
    got = run_cuda(q, k, v, dO, m, J, kappa)
    _C.set_force_generic(True)
    try:
        ref = run_cuda(q, k, v, dO, m, J, kappa)
    finally:
        _C.set_force_generic(False)
    slices = [0, B * H - 1]
    pick = lambda t: t.reshape(1, B * H, *t.shape[2:])[:, slices]
    want = run_oracle(pick(q), pick(k), pick(v), pick(dO), m, J, kappa)
    for key in ("K2", "lse2", "k2inv", "step2", "out", "dq", "dk", "dv"):
        a, b = _rel(pick(got[key]), want[key]), _rel(pick(ref[key]), want[key])
        print(key, f"{a:.2e} {b:.2e}")
        assert a <= 8 * b + 1e-6, (key, a, b)


@pytest.mark.parametrize("BH", [2, 37, 38])     # beside the column passes up to a quarter of 148 SMs, in line above
@pytest.mark.parametrize("D", [64, 128])
def test_beside_the_column_passes(cuda_device, BH, D):
    """The same slice comes out the same whatever runs beside it; fp16 results are within one rounding of the sums."""
    m, J, N = 96, 6, 700
    q, k, v, dO = O.make_inputs(1, BH, N, D, seed=11, dtype=torch.float16)
    got = run_cuda(q, k, v, dO, m, J, 5.0)
    again = run_cuda(q, k, v, dO, m, J, 5.0)
    want = run_oracle(q[:, -1:], k[:, -1:], v[:, -1:], dO[:, -1:], m, J, 5.0)
    for key, bound in (("out", 2e-3), ("dq", 1e-2), ("dk", 1e-2), ("dv", 1e-2)):
        assert torch.equal(got[key], again[key]), key
        assert O.rel_max(got[key][:, -1:].cpu(), want[key]) <= bound, key
