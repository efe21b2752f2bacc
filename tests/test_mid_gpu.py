"""The landmark-sized stages for more than 64 landmarks on the tensor cores, against the float64 oracle with the
CUDA-core kernels as the yardstick.  FP32 inputs run the same streaming passes on both sides, so only these stages
differ.  Operands keep 24 bits in three bf16 terms.  The accumulator truncates: the eight K steps of a product lose up
to 8 * 2^-24, all in one direction, where the yardstick's 128 rounded additions lose about sqrt(128) / 2 * 2^-24
= 6 * 2^-24 in either direction; both are amplified alike by the iterations: bound 2 x yardstick for what these stages
form.  A bias adds up over the terms of the sums that follow (up to sqrt(64) = 8 times) where rounding averages out:
bound 8 x yardstick for the outputs and gradients."""
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
        assert a <= (2 if key in ("K2", "lse2", "k2inv", "step2") else 8) * b, (key, a, b)


@pytest.mark.parametrize("D,m,dtype", [(64, 96, torch.float16), (128, 96, torch.float16), (64, 65, torch.bfloat16), (32, 128, torch.float16)])
def test_beside_the_column_passes(cuda_device, D, m, dtype):
    """Up to a quarter of the SMs' worth of slices the pseudoinverse kernels run beside the column passes, above in line, and
    with more slices than clusters a cluster walks several.  The FP32 matrices of a slice do not depend on any of it,
    bit for bit; what the column passes make of them differs by the order of their chunks, one rounding of the result."""
    from flashnystrom_b200 import _C
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    J, N, few = 6, 700, sms // 4
    q, k, v, dO = O.make_inputs(1, sms + 5, N, D, seed=11, dtype=dtype)
    runs = [run_cuda(*(t[:, :BH] for t in (q, k, v, dO)), m, J, 5.0) for BH in (few, few, few + 1, sms + 5)]
    want = run_oracle(q[:, few - 1:few], k[:, few - 1:few], v[:, few - 1:few], dO[:, few - 1:few], m, J, 5.0)
    eps = 2.0 ** -10 if dtype == torch.float16 else 2.0 ** -7
    for r in runs[1:]:
        for key in ("qt", "kt", "K2", "lse2", "iterates", "k2inv"):
            assert torch.equal(r[key][:, :few], runs[0][key]), key
        for key in ("out", "dq", "dk", "dv"):
            a, b = r[key][:, :few].float(), runs[0][key].float()
            assert float((a - b).norm() / b.norm()) <= eps, key
            assert O.rel_max(r[key][:, few - 1:few].cpu(), want[key]) <= (2 if key == "out" else 10) * eps, key
    for key in ("out", "dq", "dk", "dv"):
        assert torch.equal(runs[0][key], runs[1][key]), key
