"""Isolation tests of the Newton-Schulz pseudoinverse kernels through the C-ABI debug hooks,
against the oracle's restatement of the same algebra (the role of the reference's
tests/test_ns_bwd_kernel.py and tests/test_ns_bwd_graph.py)."""
import pytest
import torch

from oracle import nystrom_oracle as O

pytestmark = pytest.mark.gpu


def _softmax_matrix(BH, m, seed):
    g = torch.Generator().manual_seed(seed)
    return torch.softmax(torch.randn(BH, m, m, generator=g) * 1.5, dim=-1)


def _oracle_pinv(k2, J, kappa):
    k2 = k2.double().unsqueeze(0)
    if kappa > 0:
        lam = O.ridge_lambda(k2, kappa)
        A = k2.transpose(-2, -1) @ k2 + lam * torch.eye(k2.shape[-1], dtype=k2.dtype)
        its = O.newton_schulz(A, J)
        inv = its[-1] @ k2.transpose(-2, -1)
    else:
        A = k2
        its = O.newton_schulz(A, J)
        inv = its[-1]
    return A, torch.stack(its, dim=2), inv


@pytest.mark.parametrize("m", [1, 7, 16, 33, 64, 100, 128])
@pytest.mark.parametrize("J,kappa", [(6, 0.0), (3, 1e3), (8, 5.0), (12, 0.0)])
def test_pinv_forward_and_backward(cuda_device, m, J, kappa):
    from flashnystrom_b200 import _C
    BH = 3
    k2 = _softmax_matrix(BH, m, seed=m + J)
    G = torch.randn(BH, m, m, generator=torch.Generator().manual_seed(99))
    iters, inv = _C.debug_pinv_forward(k2.cuda(), J, kappa)
    A, ref_its, ref_inv = _oracle_pinv(k2, J, kappa)
    assert O.rel_max(inv.cpu(), ref_inv[0]) < 2e-4, "k2_inv"
    assert O.rel_max(iters.cpu(), ref_its[0]) < 2e-4, "iterates"

    # backward: hand algebra of the oracle in float64 on the iterates the kernel itself saved
    dk2 = _C.debug_pinv_backward(k2.cuda(), iters, G.cuda(), kappa).cpu()
    its64 = iters.cpu().double().unsqueeze(0)
    k64, G64 = k2.double().unsqueeze(0), G.double().unsqueeze(0)
    if kappa > 0:
        ZJ = its64[:, :, -1]
        dA, _ = O.ns_backward(A, its64, G64 @ k64)
        ref = G64.transpose(-2, -1) @ ZJ + k64 @ (dA + dA.transpose(-2, -1))
    else:
        ref, _ = O.ns_backward(A, its64, G64)
    if kappa == 0:
        # K2 is row-stochastic, so its row sums tie at 1 and the argmax row of ||K2||_inf is
        # decided by round-off.  The term it steers is constant along a row and vanishes under
        # the softmax Jacobian that always follows, so compare after that projection.
        def jac(d):
            return k64[0] * (d - (d * k64[0]).sum(-1, keepdim=True))
        assert O.rel_max(jac(dk2.double()), jac(ref[0])) < 5e-4, "d_k2 (after softmax Jacobian)"
    else:
        assert O.rel_max(dk2, ref[0]) < 5e-4, "d_k2"


@pytest.mark.parametrize("m", [33, 65, 127, 128])
@pytest.mark.parametrize("J,kappa", [(1, 0.0), (2, 0.0), (3, 0.0), (1, 5.0), (2, 5.0)])
def test_pinv_few_iterations(cuda_device, m, J, kappa):
    """One to three iterations: the backward forms R, W and Y one iterate ahead and (past 64 landmarks) rotates three images
    of the iterates.  Bounds as in test_pinv_forward_and_backward."""
    test_pinv_forward_and_backward(cuda_device, m, J, kappa)


@pytest.mark.parametrize("D", [16, 64, 128])
@pytest.mark.parametrize("m", [15, 17, 31, 32, 47, 48, 49, 63, 64])
@pytest.mark.parametrize("kappa", [0.0, 5.0])
def test_tensor_core_pinv_no_less_precise_than_cuda_cores(cuda_device, m, D, kappa):
    """Edges of the 16-wide K steps and of the 32 x 32 blocks, the three head_dim forms of the scores and of the landmark
    gradients.  Both kernels against the oracle in float64 on the same landmarks and incoming gradients; the bound is the CUDA
    cores' own error plus the rounding of an FP32 result, half a unit in the last place (measured: K2inv 0.50 times the CUDA cores'
    error in the mean and 0.91 at most, dQ 0.56 and 0.92, dK 0.57 and 0.94; K2, whose error is that rounding, 1.08 and 1.30)."""
    from flashnystrom_b200 import _C
    q, k, v, dO = (t.cuda() for t in O.make_inputs(1, 3, 4 * m + 5, D, seed=m + D, dtype=torch.float32))
    err = {}
    for generic in (False, True):
        _C.set_force_generic(generic)
        try:
            r = _C.forward(q, k, v, m, 6, kappa)
            g = _C.backward(dO, *r[1:13], v, r[0], m, 6, True, kappa)
        finally:
            _C.set_force_generic(False)
        _C.check_device_status()
        with torch.device("cuda"):
            d = [t.double() for t in (q, k, v, dO)]
            f = O.forward(*d[:3], m, 6, kappa)
            f.update(O.backward(*d, m, 6, kappa, fwd=f))
        got = {"K2": r[11], "k2inv": r[5], "dq": g[0], "dk": g[1]}
        err[generic] = {n: float((t.double() - f[n]).norm() / f[n].norm()) for n, t in got.items()}
    for n in err[True]:
        assert err[False][n] <= err[True][n] + 2.0 ** -24, (n, err)


def test_pinv_same_call_twice_is_bit_identical(cuda_device):
    from flashnystrom_b200 import _C
    k2 = _softmax_matrix(4, 64, seed=1).cuda()
    a = _C.debug_pinv_forward(k2, 6, 5.0)
    b = _C.debug_pinv_forward(k2, 6, 5.0)
    assert torch.equal(a[0], b[0]) and torch.equal(a[1], b[1])
    G = torch.randn(4, 64, 64, device="cuda")
    assert torch.equal(_C.debug_pinv_backward(k2, a[0], G, 5.0), _C.debug_pinv_backward(k2, a[0], G, 5.0))


def test_ns_bwd_step_hook(cuda_device):
    """One backward iteration on the product's kernel against the oracle's algebra
    (the reference's tests/test_ns_bwd_kernel.py:49-119 does this for its per-step kernel)."""
    from flashnystrom_b200 import _C
    BH, m = 3, 48
    k2 = _softmax_matrix(BH, m, seed=5)
    its = torch.stack(O.newton_schulz(k2.double(), 3), dim=1)          # (BH, 4, m, m)
    Zj = its[:, 2].float()
    g = torch.Generator().manual_seed(6)
    dZn = torch.randn(BH, m, m, generator=g)
    dZ_out, dK2_acc = _C.debug_ns_bwd_step(k2.cuda(), Zj.cuda(), dZn.cuda())
    A, Z, dZ = k2.double(), Zj.double(), dZn.double()
    I = torch.eye(m, dtype=torch.float64)
    M = A @ Z; U = 7 * I - M; V = 15 * I - M @ U; T = 13 * I - M @ V
    Mt = M.transpose(-2, -1)
    dT = 0.25 * Z.transpose(-2, -1) @ dZ
    dV = -Mt @ dT
    dM = -dT @ V.transpose(-2, -1) - dV @ U.transpose(-2, -1) + Mt @ dV
    ref_dA = dM @ Z.transpose(-2, -1)
    ref_dZ = 0.25 * dZ @ T.transpose(-2, -1) + A.transpose(-2, -1) @ dM
    assert O.rel_max(dZ_out.cpu(), ref_dZ) < 2e-5
    assert O.rel_max(dK2_acc.cpu(), ref_dA) < 2e-5


def test_ns_bwd_final_hook(cuda_device):
    """The tail (Z0 norm terms, softmax-2 Jacobian, landmark gradients) against autograd through the
    same algebra (the reference's tests/test_ns_bwd_kernel.py:134-229)."""
    from flashnystrom_b200 import _C
    BH, m, D = 2, 40, 64
    g = torch.Generator().manual_seed(8)
    qt = torch.randn(BH, m, D, generator=g) * 0.3
    kt = torch.randn(BH, m, D, generator=g) * 0.3
    dZ0 = torch.randn(BH, m, m, generator=g)
    dK2_in = torch.randn(BH, m, m, generator=g)
    q64, k64 = qt.double().requires_grad_(True), kt.double().requires_grad_(True)
    K2 = torch.softmax(q64 @ k64.transpose(-2, -1), dim=-1)
    n1, _, ninf, _ = O.norms_1_inf(K2)
    Z0 = K2.transpose(-2, -1) / (n1 * ninf)[..., None, None]
    loss = (Z0 * dZ0.double()).sum() + (K2 * dK2_in.double()).sum()
    loss.backward()
    dq, dk, dk2 = _C.debug_ns_bwd_final(qt.cuda(), kt.cuda(), K2.detach().float().cuda(), dZ0.cuda(), dK2_in.cuda())
    assert O.rel_max(dq.cpu(), q64.grad) < 2e-4
    assert O.rel_max(dk.cpu(), k64.grad) < 2e-4


def test_probe_occupancy_lists_the_kernels(cuda_device):
    from flashnystrom_b200 import _C
    rep = _C.probe_occupancy(0)
    names = {r["name"] for r in rep}
    assert {"tc_fwd_b<half,64,64>", "tc_rows_inplace<half,64,64>", "ns_bwd_tc", "tc_bwd_a<half,128,64>"} <= names
    by = {r["name"]: r for r in rep}
    print("\n".join(f"{r['name']:32s} regs {r['registers']:3d}  smem {r['static_smem_bytes'] + r['dynamic_smem_bytes']:6d}  "
                    f"local {r['local_bytes_per_thread']:3d}  CTAs/SM {r['blocks_per_sm']}" for r in rep))
    # (blocks_per_sm is what cudaOccupancyMaxActiveBlocksPerMultiprocessor answers; for the 320-thread
    # tensor-core kernels of head_dim 64 it says 1 although two CTAs are co-resident in practice, as
    # per-CTA SM ids and lifetimes show, so it is only checked for sanity)
    assert all(r["registers"] > 0 and r["threads"] > 0 and r["blocks_per_sm"] >= 1 for r in rep)
    assert by["tc_fwd_c<half,64,64>"]["dynamic_smem_bytes"] * 2 < 227 * 1024
    assert by["tc_fwd_c<half,64,64>"]["registers"] * 320 * 2 <= 65536


def test_probe_occupancy_leaves_the_kernels_usable(cuda_device):
    """The report asks for the shared memory of the 64-landmark / 3-tap instances; a call that needs more
    of the same kernels (128 landmarks, a 33-tap convolution) has to work before and after it."""
    from flashnystrom_b200 import _C
    q, k, v, dO = O.make_inputs(1, 2, 1024, 128, seed=11, dtype=torch.float16)
    q, k, v = q.cuda(), k.cuda(), v.cuda()
    w = torch.randn(2, 33, device="cuda")
    first = _C.forward(q, k, v, 128, 6)[0]
    conv_first = _C.conv_residual(v, w)
    _C.probe_occupancy(0)
    again = _C.forward(q, k, v, 128, 6)[0]
    conv_again = _C.conv_residual(v, w)
    torch.cuda.synchronize()
    assert torch.equal(first, again) and torch.equal(conv_first, conv_again)


@pytest.mark.parametrize("dtype,m", [(torch.float16, 64), (torch.bfloat16, 63), (torch.float32, 49), (torch.float32, 33), (torch.float16, 30)])
def test_k2_is_the_same_with_and_without_the_ridge(cuda_device, dtype, m):
    """The forward kernel copies the softmaxed matrix out of a buffer that the ridge's Gram matrix takes next; scores and softmax
    do not depend on the ridge, so both calls give the same bits.  Two slices per SM, several times, 4-byte copies (m not a
    multiple of four) and 16-byte ones."""
    from flashnystrom_b200 import _C
    q, k, v, _ = (t.cuda() for t in O.make_inputs(37, 8, 2 * m + 1, 64, seed=m, dtype=dtype))
    want = _C.forward(q, k, v, m, 4, 0.0)
    for _ in range(8):
        got = _C.forward(q, k, v, m, 4, 5.0)
        assert torch.equal(got[11], want[11])
        assert torch.equal(got[8], want[8])
    _C.check_device_status()


@pytest.mark.parametrize("m", [17, 64])
def test_first_iterate_is_the_rounded_quotient(cuda_device, m):
    """Z0 = A^T / (||A||_1 ||A||_inf) against torch's division on the same bits, values over 40 powers of two.  The kernel adds the norms
    up in its own order, at most 19 additions each, and rounds their product: the divisor is within 24 units in the last place
    of the one in float64, and one of these has to give all quotients of a matrix."""
    from flashnystrom_b200 import _C
    g = torch.Generator().manual_seed(m)
    a = (torch.randn(24, m, m, generator=g) * torch.exp2(torch.rand(24, m, m, generator=g) * 40 - 30)).cuda()
    z0 = _C.debug_pinv_forward(a, 1)[0][:, 0]
    c = (a.abs().double().sum(1).amax(1) * a.abs().double().sum(2).amax(1)).float()
    steps = (c.view(torch.int32)[:, None] + torch.arange(-24, 25, device="cuda", dtype=torch.int32)).view(torch.float32)
    same = (a.transpose(1, 2)[:, None] / steps[:, :, None, None] == z0[:, None]).flatten(2).all(2)
    assert same.any(1).all()


@pytest.mark.parametrize("m", [17, 64])
def test_infinite_divisor(cuda_device, m):
    """An infinite entry, and finite ones whose norms' product overflows: zeros, and NaN for inf / inf."""
    from flashnystrom_b200 import _C
    a = _softmax_matrix(2, m, seed=m).cuda()
    a[0, 3, 5] = float("inf")
    a[1] *= 1e25
    z0 = _C.debug_pinv_forward(a, 1)[0][:, 0]
    assert torch.equal(z0.nan_to_num(nan=7.0), (a.transpose(1, 2) / float("inf")).nan_to_num(nan=7.0))


@pytest.mark.parametrize("dtype,m", [(torch.float32, 17), (torch.float16, 64), (torch.float32, 64)])
@pytest.mark.parametrize("kappa", [1e-25, 3e-20])
def test_ridge_whose_norms_overflow(cuda_device, dtype, m, kappa):
    """Condition numbers so small that the product of A's norms overflows: Z0 = A^T / inf = 0, and so are the other iterates and the
    output.  What is finite of the gradients on the CUDA cores, which divide, is finite here."""
    from flashnystrom_b200 import _C
    q, k, v, dO = (t.cuda() for t in O.make_inputs(1, 2, 300, 64, seed=9, dtype=dtype))
    finite = []
    for generic in (False, True):
        _C.set_force_generic(generic)
        try:
            r = _C.forward(q, k, v, m, 4, kappa)
            assert not r[10].any() and not r[5].any() and not r[0].any()
            finite.append([t.isfinite() for t in _C.backward(dO, *r[1:13], v, r[0], m, 4, True, kappa)])
        finally:
            _C.set_force_generic(False)
    for a, b in zip(*finite):
        assert torch.equal(a, b)


@pytest.mark.parametrize("ms,bound", [((16, 17, 33, 48, 49, 63, 64), 1.5), ((100, 128), 1.1)])
@pytest.mark.parametrize("J", [4, 6, 8])
def test_pinv_backward_is_about_as_precise_as_fp32_sums(cuda_device, ms, bound, J):
    """dL/dK2 (after the softmax Jacobian) against 64 bits, by the kernels and by FP32 sums in torch on the same iterates; the mean of
    the quotients of their errors.  The kernels' sums are truncated and given back what that costs on the average, by the number
    of additions: measured 1.17, 1.23 and 1.32 for J = 4, 6 and 8, past 64 landmarks 1.00, 0.99 and 0.96.  Where the products that
    share an accumulator got one product's share they were 1.62, 1.87 and 2.15, and 1.22, 1.27 and 1.27."""
    from flashnystrom_b200 import _C
    quotients = []
    for m in ms:
        g = torch.Generator().manual_seed(m + J)
        k2 = torch.softmax(torch.randn(8, m, m, generator=g) * 1.5, -1).cuda()
        G = torch.randn(8, m, m, generator=g).cuda()
        iterates, _ = _C.debug_pinv_forward(k2, J)
        got = _C.debug_pinv_backward(k2, iterates, G)
        with torch.device("cuda"):
            fp32, _ = O.ns_backward(k2[None], iterates[None], G[None])
            exact, _ = O.ns_backward(k2.double()[None], iterates.double()[None], G.double()[None])
        k64 = k2.double()
        want, a, b = (k64 * (d - (d * k64).sum(-1, keepdim=True)) for d in (exact[0], got.double(), fp32[0].double()))
        quotients.append(float((a - want).norm() / (b - want).norm()))
    assert sum(quotients) / len(quotients) <= bound, quotients
