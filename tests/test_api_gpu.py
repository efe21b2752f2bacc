"""Public Python API on the GPU: functional entry point, autograd Function, module, conv residual,
error behaviour.  Mirrors the reference's tests/test_flash_nystrom_cov.py and
tests/test_precision_config.py against the CPU oracle."""
import pytest
import torch

from oracle import nystrom_oracle as O

pytestmark = pytest.mark.gpu


def test_function_apply_eight_args_and_grads(cuda_device):
    from flashnystrom_b200 import FlashNystromFunction
    q, k, v, dO = O.make_inputs(1, 2, 384, 64, seed=0, dtype=torch.float16)
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    out = FlashNystromFunction.apply(qd, kd, vd, 32, 6, True, 0.0, False)
    out.backward(dO.cuda())
    ref = O.forward_backward_autograd(q.double(), k.double(), v.double(), dO.double(), 32, 6)
    assert O.rel_max(out.detach().cpu(), ref[0]) <= 2e-3
    for got, want in zip((qd.grad, kd.grad, vd.grad), ref[1:]):
        assert O.rel_max(got.cpu(), want) <= 1e-2


def test_conv_residual_matches_oracle(cuda_device):
    from flashnystrom_b200 import flash_nystrom_attention
    q, k, v, dO = O.make_inputs(2, 2, 200, 64, seed=1, dtype=torch.float32)
    w = torch.randn(2, 5, generator=torch.Generator().manual_seed(3)) * 0.3
    qd, kd, vd, wd = (t.cuda().requires_grad_(True) for t in (q, k, v, w))
    out = flash_nystrom_attention(qd, kd, vd, 16, 6, conv_weight=wd, conv_kernel_size=5)
    out.backward(dO.cuda())
    q2, k2, v2, w2 = (t.double().requires_grad_(True) for t in (q, k, v, w))
    ref = O.attention(q2, k2, v2, 16, 6, w2, 5)
    ref.backward(dO.double())
    assert O.rel_max(out.detach().cpu(), ref.detach()) <= 2e-4
    assert O.rel_max(vd.grad.cpu(), v2.grad) <= 2e-3
    assert O.rel_max(wd.grad.cpu(), w2.grad) <= 2e-3


def test_ridge_changes_output_and_matches(cuda_device):
    from flashnystrom_b200 import flash_nystrom_attention
    q, k, v, _ = O.make_inputs(1, 2, 1024, 64, seed=0, dtype=torch.float16)
    a = flash_nystrom_attention(q.cuda(), k.cuda(), v.cuda(), 64, 6, kappa_star=0.0)
    b = flash_nystrom_attention(q.cuda(), k.cuda(), v.cuda(), 64, 6, kappa_star=5.0)
    assert O.rel_max(a.cpu(), b.cpu()) > 1e-2
    ref = O.attention(q.double(), k.double(), v.double(), 64, 6, kappa_star=5.0)
    assert O.rel_max(b.cpu(), ref) <= 2e-3


def test_module_forward_backward_vs_cpu_module(cuda_device):
    """FlashNystromAttention (dim 128, 2 heads) against the same module evaluated on CPU in
    float64 with the oracle in place of the kernels and the same state_dict."""
    from flashnystrom_b200 import FlashNystromAttention, NystromConfig
    torch.manual_seed(0)
    cfg = NystromConfig(num_landmarks=16, newton_iter=6, conv_kernel_size=3)
    mod = FlashNystromAttention(128, heads=2, config=cfg)
    x = torch.randn(2, 256, 128)
    sd = {k_: v_.double() for k_, v_ in mod.state_dict().items()}

    def cpu_forward(xx):
        B, N, _ = xx.shape
        proj = lambda w: (xx @ w.t()).view(B, N, 2, 64).transpose(1, 2)
        q, k, v = proj(sd["q_proj.weight"]), proj(sd["k_proj.weight"]), proj(sd["v_proj.weight"])
        o = O.attention(q, k, v, 16, 6, sd["conv_weight"], 3)
        return o.transpose(1, 2).reshape(B, N, 128) @ sd["out_proj.weight"].t()

    xc = x.double().requires_grad_(True)
    yc = cpu_forward(xc)
    yc.sum().backward()
    modg = mod.cuda()
    xg = x.cuda().requires_grad_(True)
    yg = modg(xg)
    yg.sum().backward()
    assert O.rel_max(yg.detach().cpu(), yc.detach()) <= 1e-3
    assert O.rel_max(xg.grad.cpu(), xc.grad) <= 5e-3
    assert set(mod.state_dict()) == {"q_proj.weight", "k_proj.weight", "v_proj.weight", "out_proj.weight",
                                     "conv_weight"}


def test_module_fp16_runs(cuda_device):
    from flashnystrom_b200 import FlashNystromAttention
    mod = FlashNystromAttention(512, heads=8).cuda().half()
    x = torch.randn(2, 1024, 512, device="cuda", dtype=torch.float16, requires_grad=True)
    y = mod(x)
    y.sum().backward()
    assert torch.isfinite(y).all() and torch.isfinite(x.grad).all()


@pytest.mark.parametrize("bad,msg", [
    (dict(m=200), "num_landmarks must be in"),
    (dict(J=0), "newton_iter must be in"),
    (dict(kappa=-1.0), "kappa_star"),
    (dict(N=8, m=16), "must be >="),
])
def test_errors_are_runtime_errors(cuda_device, bad, msg):
    from flashnystrom_b200 import _C
    N, m, J, kappa = bad.get("N", 128), bad.get("m", 16), bad.get("J", 6), bad.get("kappa", 0.0)
    q = torch.zeros(1, 1, N, 64, device="cuda", dtype=torch.float16)
    with pytest.raises(RuntimeError, match=msg):
        _C.forward(q, q, q, m, J, kappa)
    with pytest.raises(RuntimeError, match="contiguous"):
        _C.forward(q.transpose(2, 3), q.transpose(2, 3), q.transpose(2, 3), 16, 6)
    with pytest.raises(RuntimeError, match="dtypes must match"):
        _C.forward(q, q.float(), q, 16, 6)


def test_backward_on_autograd_thread_and_no_status_error(cuda_device):
    from flashnystrom_b200 import flash_nystrom_attention, _C
    q, k, v, dO = O.make_inputs(1, 4, 2048, 64, seed=2, dtype=torch.bfloat16)
    qd, kd, vd = (t.cuda().requires_grad_(True) for t in (q, k, v))
    with torch.autograd.set_multithreading_enabled(False):
        flash_nystrom_attention(qd, kd, vd, 64, 6).backward(dO.cuda())
    torch.cuda.synchronize()
    _C.check_device_status()
    assert torch.isfinite(qd.grad).all()


def test_profile_lists_kernels(cuda_device):
    from flashnystrom_b200 import _C
    q, k, v, _ = O.make_inputs(1, 2, 512, 64, seed=0, dtype=torch.float16)
    _C.set_profiling(True)
    try:
        _C.forward(q.cuda(), k.cuda(), v.cuda(), 64, 6)
        prof = _C.last_profile()
    finally:
        _C.set_profiling(False)
    names = [n for n, _ in prof]
    assert "landmark_partial" in names and "tc_fwd_b" in names and "tc_fwd_c" in names
    assert all(ms >= 0 for _, ms in prof)
    caps = _C.query_sm_limits(0)
    assert caps["cc_major"] == 10 and caps["sm_count"] > 0


def test_cuda_graph_capture_and_replay(cuda_device):
    """A forward + backward captured once into a CUDA graph (the library allocates nothing, never
    synchronises and forks its side streams with events) replays to the same bits, also after the
    inputs were overwritten in place."""
    from flashnystrom_b200 import flash_nystrom_attention, _C
    q, k, v, dO = (t.cuda() for t in O.make_inputs(1, 4, 4096, 64, seed=12, dtype=torch.float16))
    q.requires_grad_(True), k.requires_grad_(True), v.requires_grad_(True)

    def step():
        q.grad = k.grad = v.grad = None
        out = flash_nystrom_attention(q, k, v, num_landmarks=64, newton_iter=6)
        out.backward(dO)
        return out

    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        for _ in range(3):
            eager = step()
    torch.cuda.current_stream().wait_stream(side)
    torch.cuda.synchronize()
    want = [eager.clone(), q.grad.clone(), k.grad.clone(), v.grad.clone()]
    g = torch.cuda.CUDAGraph()
    q.grad = k.grad = v.grad = None
    with torch.cuda.graph(g):
        gout = flash_nystrom_attention(q, k, v, num_landmarks=64, newton_iter=6)
        gout.backward(dO)
    g.replay()
    torch.cuda.synchronize()
    _C.check_device_status()
    for a, b in zip([gout, q.grad, k.grad, v.grad], want):
        assert torch.equal(a, b)
    # new data through the same graph: matches a fresh eager call
    with torch.no_grad():
        q.mul_(0.5)
        dO.mul_(2.0)
    g.replay()
    torch.cuda.synchronize()
    got = [gout.clone(), q.grad.clone(), k.grad.clone(), v.grad.clone()]
    eager = step()
    torch.cuda.synchronize()
    for a, b in zip(got, [eager, q.grad, k.grad, v.grad]):
        assert torch.equal(a, b)


def test_head_split_layout_matches_contiguous(cuda_device):
    """q, k, v given as head-split views of (B, N, H*D) tensors (what the projections of the module
    produce) go through strided tensor maps, without transposing copies: same bits as the contiguous
    call, and the output and the gradients come back in that layout too."""
    from flashnystrom_b200 import _C, flash_nystrom_attention
    B, H, N, D, m = 2, 3, 1500, 64, 48
    q, k, v, dO = (t.cuda() for t in O.make_inputs(B, H, N, D, seed=13, dtype=torch.float16))
    a = [t.clone().requires_grad_(True) for t in (q, k, v)]
    flash_nystrom_attention(*a, num_landmarks=m).backward(dO)
    want_out = flash_nystrom_attention(q, k, v, num_landmarks=m)
    # the same values stored as (B, N, H, D)
    b = [t.transpose(1, 2).contiguous().transpose(1, 2).detach().requires_grad_(True) for t in (q, k, v)]
    assert all(_C.layout_of(t) == 1 for t in b)
    out = flash_nystrom_attention(*b, num_landmarks=m)
    assert _C.layout_of(out) == 1 and torch.equal(out, want_out)
    out.backward(dO.transpose(1, 2).contiguous().transpose(1, 2))
    for x, y in zip(a, b):
        assert _C.layout_of(y.grad) == 1 and torch.equal(x.grad, y.grad)
    # head_dim 128 as well
    q, k, v, dO = (t.cuda() for t in O.make_inputs(1, 2, 700, 128, seed=14, dtype=torch.bfloat16))
    want = flash_nystrom_attention(q, k, v, num_landmarks=40)
    got = flash_nystrom_attention(*(t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v)), num_landmarks=40)
    assert torch.equal(got, want)
    # fp32 (CUDA-core path): the view is accepted by the module only through a copy; the op itself refuses it
    with pytest.raises(RuntimeError, match="contiguous"):
        _C.forward(*(t.float().transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v)), 40, 6)


def _shifted(t):
    """A contiguous copy of t that starts four bytes past a 16-byte boundary."""
    buf = torch.empty(t.numel() + 4, dtype=t.dtype, device=t.device)
    assert buf.data_ptr() % 16 == 0
    return buf[1:1 + t.numel()].view(t.shape).copy_(t)


@pytest.mark.parametrize("dtype,D,m,names", [
    (torch.float16, 64, 100, ("qt", "kt", "step2", "bmat")), (torch.bfloat16, 32, 128, ("qt", "kt", "step2", "bmat")),
    (torch.float32, 128, 70, ("qt", "kt", "step2", "bmat")), (torch.float32, 64, 64, ("step2",)), (torch.float16, 32, 40, ("step2",)),
])
def test_saved_tensors_need_only_their_types_alignment(cuda_device, dtype, D, m, names):
    """FP32 saved tensors that the backward took at any four-byte boundary (views into a larger buffer, say)."""
    from flashnystrom_b200 import _C
    q, k, v, dO = (t.cuda() for t in O.make_inputs(1, 2, 300, D, seed=5, dtype=dtype))
    res = _C.forward(q, k, v, m, 4)
    place = dict(qt=3, kt=4, step2=6, bmat=12)
    want = _C.backward(dO, *res[1:13], v, res[0], m, 4)
    for n in names:
        res[place[n]] = _shifted(res[place[n]])
    got = _C.backward(dO, *res[1:13], v, res[0], m, 4)
    for a, b in zip(got, want):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,D,m", [(torch.float16, 64, 100), (torch.float32, 32, 70), (torch.bfloat16, 16, 65)])
def test_landmark_outputs_need_only_their_types_alignment(cuda_device, dtype, D, m):
    """The same for the landmarks that a forward call of the C ABI writes (more than 64 of them)."""
    import ctypes
    from flashnystrom_b200 import _C, _lib
    q, k, v, _ = (t.cuda() for t in O.make_inputs(1, 2, 300, D, seed=6, dtype=dtype))
    lib, dev, J = _lib.load(), q.device, 4
    want = _C.forward(q, k, v, m, J)
    t = [torch.empty_like(x) for x in (want[0], want[7])] + [_shifted(want[i]) for i in (3, 4)]
    t[2].zero_(), t[3].zero_()
    t += [torch.empty_like(want[i]) for i in (11, 8, 10, 5, 12, 9, 6)]
    shape = _C._shape_struct(1, 2, 300, D, m, J, dtype, 0.0)
    ws = torch.empty(lib.fnb_fwd_workspace_bytes(ctypes.byref(shape)), dtype=torch.uint8, device=dev)
    args = _lib.FwdArgs(shape, *[x.data_ptr() for x in (q, k, v, *t)], ws.data_ptr(), ws.numel(), dev.index,
                        torch.cuda.current_stream(dev).cuda_stream, _C._status(dev).data_ptr())
    _lib.check(lib.fnb_forward(ctypes.byref(args)))
    torch.cuda.synchronize()
    _C.check_device_status()
    for a, b in zip(t, [want[i] for i in (0, 7, 3, 4, 11, 8, 10, 5, 12, 9, 6)]):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,D,m", [(torch.bfloat16, 32, 64), (torch.float16, 64, 100), (torch.float16, 128, 100), (torch.float32, 64, 64),
                                       (torch.float32, 64, 100)])
@pytest.mark.parametrize("split_heads", [False, True])
def test_autograd_function_matches_the_extension_calls(cuda_device, dtype, D, m, split_heads):
    """What users call keeps its FP32 tensors in one buffer; the extension's forward() and backward() have one each."""
    from flashnystrom_b200 import _C, flash_nystrom_attention
    q, k, v, dO = (t.cuda() for t in O.make_inputs(2, 3, 300, D, seed=7, dtype=dtype))
    res = _C.forward(q, k, v, m, 5, 5.0)
    want = [res[0], *_C.backward(dO, *res[1:13], v, res[0], m, 5, True, 5.0)]
    x = [q.clone(), k.clone(), v.clone()]
    if split_heads and _C.tc_eligible(dtype, D, m):
        x = [t.transpose(1, 2).contiguous().transpose(1, 2) for t in x]
    x = [t.requires_grad_(True) for t in x]
    out = flash_nystrom_attention(*x, num_landmarks=m, newton_iter=5, kappa_star=5.0)
    out.backward(dO)
    for a, b in zip([out, *(t.grad for t in x)], want):
        assert torch.equal(a, b)


def test_saved_tensor_hooks_may_move_the_buffer(cuda_device):
    """Saved tensors that come back from a hook at another address, and not 16-byte aligned."""
    from flashnystrom_b200 import flash_nystrom_attention
    q, k, v, dO = (t.cuda() for t in O.make_inputs(1, 2, 300, 64, seed=8, dtype=torch.float32))
    grads = []
    for unpack in (lambda t: t, lambda t: _shifted(t) if t.dim() == 1 else t.clone()):
        x = [t.clone().requires_grad_(True) for t in (q, k, v)]
        with torch.autograd.graph.saved_tensors_hooks(lambda t: t, unpack):
            out = flash_nystrom_attention(*x, num_landmarks=32)
        out.backward(dO)
        grads.append([t.grad for t in x])
    for a, b in zip(*grads):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dtype,D,m,kappa", [(torch.float16, 64, 64, 5.0), (torch.float16, 64, 64, 0.0), (torch.bfloat16, 128, 32, 5.0),
                                             (torch.float32, 64, 36, 5.0), (torch.float32, 32, 33, 5.0)])
def test_softmaxed_matrix_and_iterates_need_only_their_types_alignment(cuda_device, dtype, D, m, kappa):
    """Up to 64 landmarks: K2 and the iterates at any four-byte boundary, written by a forward call of the C ABI (which reads K2
    back for the ridge) and read by the backward."""
    import ctypes
    from flashnystrom_b200 import _C, _lib
    q, k, v, dO = (t.cuda() for t in O.make_inputs(1, 2, 300, D, seed=6, dtype=dtype))
    lib, dev, J = _lib.load(), q.device, 4
    want = _C.forward(q, k, v, m, J, kappa)
    got = [t if i in (1, 2) else torch.zeros_like(t) for i, t in enumerate(want)]
    for i in (10, 11):
        got[i] = _shifted(got[i])
    shape = _C._shape_struct(1, 2, 300, D, m, J, dtype, kappa)
    ws = torch.empty(lib.fnb_fwd_workspace_bytes(ctypes.byref(shape)), dtype=torch.uint8, device=dev)
    outputs = [got[i].data_ptr() for i in (0, 7, 3, 4, 11, 8, 10, 5, 12, 9, 6)]
    args = _lib.FwdArgs(shape, *[x.data_ptr() for x in (q, k, v)], *outputs, ws.data_ptr(), ws.numel(), dev.index,
                        torch.cuda.current_stream(dev).cuda_stream, _C._status(dev).data_ptr())
    _lib.check(lib.fnb_forward(ctypes.byref(args)))
    _C.check_device_status()
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    for a, b in zip(_C.backward(dO, *got[1:13], v, got[0], m, J, True, kappa), _C.backward(dO, *want[1:13], v, want[0], m, J, True, kappa)):
        assert torch.equal(a, b)


@pytest.mark.parametrize("m,kappa", [(64, 5.0), (64, 0.0), (36, 5.0), (33, 5.0), (100, 5.0)])
def test_pseudoinverse_entries_need_only_their_types_alignment(cuda_device, m, kappa):
    import ctypes
    from flashnystrom_b200 import _C, _lib
    k2 = torch.softmax(torch.randn(2, m, m, device="cuda", generator=torch.Generator("cuda").manual_seed(m)), -1)
    G = torch.randn(2, m, m, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    iterates, inv = _C.debug_pinv_forward(k2, 4, kappa)
    dk2 = _C.debug_pinv_backward(k2, iterates, G, kappa)
    lib, dev, t = _lib.load(), k2.device, {}
    for name, x in (("k2", k2), ("G", G)):
        t[name] = _shifted(x)
    for name, x in (("iterates", iterates), ("inv", inv), ("dk2", dk2)):
        t[name] = _shifted(torch.zeros_like(x))
    ws = torch.empty(lib.fnb_debug_pinv_workspace_bytes(2, m) + 4, dtype=torch.uint8, device=dev)[4:]
    stream, p = ctypes.c_void_p(torch.cuda.current_stream(dev).cuda_stream), {n: x.data_ptr() for n, x in t.items()}
    _lib.check(lib.fnb_debug_pinv_forward(2, m, 4, kappa, p["k2"], p["iterates"], p["inv"], ws.data_ptr(), ws.numel(), dev.index, stream))
    _lib.check(lib.fnb_debug_pinv_backward(2, m, 4, kappa, p["k2"], p["iterates"], p["G"], p["dk2"], ws.data_ptr(), ws.numel(), dev.index, stream))
    for name, x in (("iterates", iterates), ("inv", inv), ("dk2", dk2)):
        assert torch.equal(t[name], x), name
    if m <= 64:
        z, da = (_shifted(torch.zeros_like(k2)) for _ in range(2))
        want = _C.debug_ns_bwd_step(k2, inv, G)
        _lib.check(lib.fnb_debug_ns_bwd_step(2, m, p["k2"], p["inv"], p["G"], z.data_ptr(), da.data_ptr(), dev.index, stream))
        assert torch.equal(z, want[0]) and torch.equal(da, want[1])
