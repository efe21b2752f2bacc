"""The C++ module of the eager path against the autograd functions that it stands for: every form that it accepts (layouts, dtypes,
odd sizes, which inputs need gradients), and what it leaves to them."""
import pytest
import torch

from oracle import nystrom_oracle as O

pytestmark = pytest.mark.gpu


def _functions(q, k, v, m, J, kappa, w=None):
    from flashnystrom_b200.flash_nystrom import FlashNystromFunction, _ConvResidualFunction
    out = FlashNystromFunction.apply(q, k, v, m, J, True, kappa, False)
    return out if w is None else _ConvResidualFunction.apply(out, v, w)


def _inputs(B, H, N, D, dtype, split_heads, seed=3):
    q, k, v, dO = (t.cuda() for t in O.make_inputs(B, H, N, D, seed=seed, dtype=dtype))
    if split_heads:
        q, k, v, dO = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v, dO))
    return q, k, v, dO


@pytest.mark.parametrize("B,H,N,D,m,dtype,split_heads,ks", [
    (1, 2, 256, 64, 32, torch.float16, False, 0), (2, 3, 301, 64, 33, torch.bfloat16, True, 3), (1, 1, 130, 128, 128, torch.float16, True, 33),
    (2, 1, 99, 16, 7, torch.float32, False, 1), (1, 5, 64, 64, 64, torch.float32, False, 5), (3, 1, 200, 32, 100, torch.bfloat16, False, 7),
    (1, 1, 65, 64, 1, torch.float16, True, 0),
])
def test_same_as_the_autograd_functions(cuda_device, B, H, N, D, m, dtype, split_heads, ks):
    """Outputs and gradients bit for bit, but for the gradient of v with a convolution: that is added up in FP32 and rounded
    once instead of three times, so it may differ by two units of the dtype's rounding of its two summands."""
    from flashnystrom_b200 import _C, flash_nystrom_attention
    q, k, v, dO = _inputs(B, H, N, D, dtype, split_heads)
    w = (torch.randn(H, ks, device="cuda", generator=torch.Generator("cuda").manual_seed(1)) * 0.3).to(dtype) if ks else None
    for needs in ((True, True, True, True), (False, False, False, False), (False, False, True, False), (True, False, False, False),
                  (False, False, False, True)):
        grads = []
        for native in (True, False):
            x = [t.detach().requires_grad_(n) for t, n in zip((q, k, v), needs)]
            ww = w.detach().requires_grad_(needs[3]) if ks else None
            if native:
                out = _C.attention(*x, m, 4, 5.0, ww)
                assert out is not None and _C.layout_of(out) == _C.layout_of(q)
                assert torch.equal(out, flash_nystrom_attention(*x, num_landmarks=m, newton_iter=4, conv_weight=ww, conv_kernel_size=ks, kappa_star=5.0))
            else:
                out = _functions(*x, m, 4, 5.0, ww)
            assert out.requires_grad == any(needs[:3] + ((needs[3],) if ks else ()))
            if out.requires_grad:
                out.backward(dO)
            grads.append([out.detach()] + [t.grad for t in x] + ([ww.grad] if ks else []))
        for i, (a, b) in enumerate(zip(*grads)):
            assert (a is None) == (b is None)
            if a is not None and i == 3 and ks:
                unit = torch.finfo(dtype).eps
                assert (a.double() - b.double()).abs().max() <= 2 * unit * b.double().abs().max()
            elif a is not None:
                assert a.dtype == b.dtype and a.stride() == b.stride() and torch.equal(a, b), i


def test_gradient_of_v_with_convolution_is_rounded_once(cuda_device):
    """Against float64: no further off than the sum of two rounded gradients."""
    from flashnystrom_b200 import _C
    q, k, v, dO = _inputs(1, 2, 500, 64, torch.float16, False)
    w = torch.randn(2, 3, device="cuda").half()
    with torch.device("cuda"):
        d = [t.double().requires_grad_(True) for t in (q, k, v, w)]
        O.attention(*d[:3], 32, 6, d[3], 3).backward(dO.double())
    err = []
    for f in (_C.attention, _functions):
        x = v.detach().requires_grad_(True)
        f(q, k, x, 32, 6, 0.0, w).backward(dO)
        err.append(float((x.grad.double() - d[2].grad).norm()))
    assert err[0] <= err[1]


def test_left_to_the_autograd_functions(cuda_device):
    from flashnystrom_b200 import _C, flash_nystrom_attention
    q, k, v, dO = _inputs(1, 2, 256, 64, torch.float16, False)
    w = torch.randn(2, 3, device="cuda").half()
    assert _C.attention(q, k, v, 32, 6, 0.0, w) is not None
    noncontiguous = q.transpose(2, 3).contiguous().transpose(2, 3)
    for args in ((noncontiguous, k, v, 32, 6, 0.0), (q, k.float(), v, 32, 6, 0.0), (q, k, v[:, :, :128], 32, 6, 0.0), (q, k, v, 300, 6, 0.0),
                 (q, k, v, 32, 0, 0.0), (q, k, v, 32, 6, float("nan")), (q, k, v, 32, 6, "5"), (q, k, v, 32.0, 6, 0.0), (q, k, v, 32, 6, 0.0, w.cpu()),
                 (q, k, v, 32, 6, 0.0, w[:, :2]), (q, k, v, 32, 6, 0.0, w[:1]), (q, k, v, 2 ** 40, 6, 0.0)):
        assert _C.attention(*args) is None, args[3:]
    # head-split views of shapes whose kernels want contiguous tensors are refused as before
    with pytest.raises(RuntimeError, match="contiguous"):
        flash_nystrom_attention(*(t.float().transpose(1, 2).contiguous().transpose(1, 2) for t in (q, k, v)), num_landmarks=32)
    # weights on the host were brought to the device
    a = flash_nystrom_attention(q, k, v, 32, 6, conv_weight=w.cpu(), conv_kernel_size=3)
    assert torch.equal(a, flash_nystrom_attention(q, k, v, 32, 6, conv_weight=w, conv_kernel_size=3))
    with pytest.raises(ValueError):
        flash_nystrom_attention(q, k, v, 32, 6, conv_weight=w[:, :2], conv_kernel_size=2)


def test_transforms_and_tracing_go_to_the_autograd_functions(cuda_device):
    from flashnystrom_b200 import _C, flash_nystrom_attention
    q, k, v, _ = _inputs(1, 2, 256, 64, torch.float16, False)
    call = lambda a: flash_nystrom_attention(a, k, v, num_landmarks=32)
    with pytest.raises(RuntimeError):                 # no vmap rule, no forward-mode formula
        torch.func.vmap(call)(torch.stack([q, q]))
    with torch.autograd.forward_ad.dual_level(), torch.no_grad():
        dual = torch.autograd.forward_ad.make_dual(q, torch.ones_like(q))
        assert _C.attention(dual, k, v, 32, 6, 0.0) is None
    with pytest.raises(TypeError):                    # (a trace would take the output for a constant)
        torch.jit.trace(call, (q,), check_trace=False)
    want = call(q)
    with torch.inference_mode():
        assert torch.equal(call(q), want)


def test_backward_on_the_stream_of_the_forward(cuda_device):
    """Forward and backward on a side stream while the caller's stream is busy: copies of the results that the side stream takes at once
    are right, and the side stream is through before the caller's, so that nothing was launched on that one."""
    from flashnystrom_b200 import flash_nystrom_attention
    host = [t.cpu().pin_memory() for t in _inputs(1, 4, 2048, 64, torch.bfloat16, False)]
    taps = torch.randn(4, 3, dtype=torch.bfloat16).pin_memory()

    def step():
        q, k, v, dO = (t.to(cuda_device, non_blocking=True) for t in host)
        w = taps.to(cuda_device, non_blocking=True)
        x = [t.requires_grad_(True) for t in (q, k, v, w)]
        out = flash_nystrom_attention(q, k, v, num_landmarks=64, conv_weight=w, conv_kernel_size=3)
        out.backward(dO)
        return [t.clone() for t in [out.detach()] + [t.grad for t in x]]
    want = step()
    caller, side = torch.cuda.current_stream(), torch.cuda.Stream()
    with torch.cuda.stream(side):
        held = [step() for _ in range(8)]             # (the side stream's memory, so that nothing is allocated below)
        del held
    torch.cuda.synchronize()
    torch.cuda._sleep(400_000_000)                    # about 0.2 s of one thread
    busy, done = torch.cuda.Event(), torch.cuda.Event()
    busy.record(caller)
    with torch.cuda.stream(side):
        got = [step() for _ in range(8)]
        done.record(side)
    done.synchronize()
    assert not busy.query()
    for g in got:
        assert all(torch.equal(a, b) for a, b in zip(g, want))
    caller.synchronize()


def test_debug_statistics_are_printed(cuda_device, monkeypatch, capfd):
    from flashnystrom_b200 import flash_nystrom_attention
    q, k, v, dO = _inputs(1, 2, 256, 64, torch.float16, False)
    monkeypatch.setenv("FNB_BWD_DEBUG", "1")
    flash_nystrom_attention(q.requires_grad_(True), k, v, num_landmarks=32).backward(dO)
    torch.cuda.synchronize()
    assert "[FNB_BWD_DEBUG] dQ" in capfd.readouterr().out


def _module(dtype, dim=128, heads=2, conv=3, m=32):
    from flashnystrom_b200 import FlashNystromAttention, NystromConfig
    torch.manual_seed(0)
    cfg = NystromConfig(num_landmarks=m, newton_iter=5, conv_kernel_size=conv, use_conv_residual=conv > 0)
    mod = FlashNystromAttention(dim, heads=heads, config=cfg).cuda().to(dtype)
    with torch.no_grad():
        for p in mod.parameters():
            p.mul_(3.0)
    return mod


@pytest.mark.parametrize("dtype,dim,heads,conv,B,N", [(torch.float16, 128, 2, 3, 2, 301), (torch.bfloat16, 256, 2, 0, 1, 130), (torch.float16, 64, 1, 7, 3, 64)])
def test_module_same_as_four_linears_around_the_op(cuda_device, dtype, dim, heads, conv, B, N):
    """A forward hook on a projection sends the module the long way.  Same output bit for bit; gradients differ by the roundings
    that are left out (x's three summands, v's two), so by a few units of the dtype of the largest value."""
    mod = _module(dtype, dim, heads, conv)
    x0 = torch.randn(B, N, dim, device="cuda").to(dtype)
    dy = torch.randn(B, N, dim, device="cuda").to(dtype)
    for frozen in ((), ("q_proj.weight",), ("q_proj.weight", "k_proj.weight", "v_proj.weight", "conv_weight"), ("x",)):
        res = []
        for native in (True, False):
            calls = []
            h = None if native else mod.q_proj.register_forward_hook(lambda *a: calls.append(1))
            x = x0.detach().requires_grad_("x" not in frozen)
            for n, p in mod.named_parameters():
                p.grad = None
                p.requires_grad_(n not in frozen)
            assert (mod._native_forward(x) is not None) == native
            y = mod(x)
            y.backward(dy)
            res.append([y.detach(), x.grad] + [p.grad for p in mod.parameters()])
            if h:
                assert len(calls) == 1
                h.remove()
        assert torch.equal(res[0][0], res[1][0])
        for a, b in zip(*res):
            assert (a is None) == (b is None)
            if a is not None:
                assert a.shape == b.shape and a.dtype == b.dtype
                assert (a.double() - b.double()).abs().max() <= 4 * torch.finfo(dtype).eps * b.double().abs().max()
    with torch.no_grad():
        y = mod(x0)
    assert torch.equal(y, res[1][0]) and not y.requires_grad


def test_module_left_to_the_linears(cuda_device):
    mod = _module(torch.float16)
    x = torch.randn(1, 100, 128, device="cuda").half()
    assert mod._native_forward(x) is not None
    with torch.autocast("cuda", dtype=torch.bfloat16):
        assert mod._native_forward(x) is None
    assert mod._native_forward(x.float()) is None and _module(torch.float32)._native_forward(x.float()) is None
    assert mod._native_forward(x.transpose(0, 1).contiguous().transpose(0, 1).expand(2, 100, 128)) is None
    assert mod._native_forward(x[:, :16]) is None            # fewer rows than landmarks: refused further on
    with pytest.raises(RuntimeError, match="must be >="):
        mod(x[:, :16])

    class Lora(torch.nn.Linear):
        def forward(self, x):
            return super().forward(x) * 2
    other = Lora(128, 128, bias=False, device="cuda", dtype=torch.float16)
    mod.v_proj, plain = other, mod.v_proj
    assert mod._native_forward(x) is None and torch.isfinite(mod(x)).all()
    mod.v_proj = plain
    torch.nn.utils.parametrize.register_parametrization(mod.out_proj, "weight", torch.nn.Identity())
    assert mod._native_forward(x) is None


def test_module_backward_with_create_graph(cuda_device):
    """The projections can be differentiated twice, as torch's linears can."""
    mod = _module(torch.float16)
    got = []
    for native in (True, False):
        h = None if native else mod.k_proj.register_forward_hook(lambda *a: None)
        x = torch.randn(1, 100, 128, device="cuda", generator=torch.Generator("cuda").manual_seed(2)).half().requires_grad_(True)
        dx, = torch.autograd.grad(mod(x).float().square().sum() * 1e-3, x, create_graph=True)
        dw, = torch.autograd.grad(dx.float().sum(), mod.q_proj.weight)
        got.append(dw.double())
        if h:
            h.remove()
    assert (got[0] - got[1]).abs().max() <= 1e-2 * got[1].abs().max()


def test_taps_alone_run_no_attention_backward(cuda_device, monkeypatch, capfd):
    """Only the convolution's weights want a gradient: the attention's backward does not run (it would print its statistics) and
    nothing is kept for it."""
    from flashnystrom_b200 import flash_nystrom_attention
    q, k, v, dO = _inputs(1, 2, 256, 64, torch.float16, False)
    w0 = torch.randn(2, 3, device="cuda", generator=torch.Generator("cuda").manual_seed(1)).half()
    monkeypatch.setenv("FNB_BWD_DEBUG", "1")
    kept, grads = [], []
    for native in (True, False):
        w = w0.clone().requires_grad_(True)
        with torch.autograd.graph.saved_tensors_hooks(lambda t: kept.append(tuple(t.shape)) or t, lambda t: t):
            out = flash_nystrom_attention(q, k, v, 32, 6, conv_weight=w, conv_kernel_size=3) if native else _functions(q, k, v, 32, 6, 0.0, w)
        out.backward(dO)
        grads.append(w.grad)
    assert kept == [tuple(v.shape), (2, 3)] * 2
    assert torch.equal(*grads)
    torch.cuda.synchronize()
    assert "[FNB_BWD_DEBUG]" not in capfd.readouterr().out


@pytest.mark.parametrize("changed", ["x", "projections", "out_proj"])
def test_module_keeps_only_what_its_gradients_take(cuda_device, changed):
    """What no wanted gradient takes may be changed in place between forward and backward, as with four linears: x under frozen
    projections, the projections' weights for an x without a gradient, the output's weight where it alone is trained."""
    x0 = torch.randn(2, 100, 128, device="cuda", generator=torch.Generator("cuda").manual_seed(4)).half()
    grads = []
    for native in (True, False):
        mod = _module(torch.float16)
        h = None if native else mod.q_proj.register_forward_hook(lambda *a: None)
        x = x0.clone()
        if changed == "x":
            for p in (mod.q_proj, mod.k_proj, mod.v_proj):
                p.weight.requires_grad_(False)
            leaf = x.requires_grad_(True)
            x = leaf * 1
        elif changed == "out_proj":
            for n, p in mod.named_parameters():
                p.requires_grad_(n == "out_proj.weight")
        y = mod(x)
        with torch.no_grad():
            for t in {"x": [x], "projections": [mod.q_proj.weight, mod.k_proj.weight, mod.v_proj.weight], "out_proj": [mod.out_proj.weight]}[changed]:
                t.add_(1)
        y.backward(torch.ones_like(y))
        grads.append([leaf.grad if changed == "x" else None] + [p.grad for p in mod.parameters()])
    for a, b in zip(*grads):
        assert (a is None) == (b is None)
        if a is not None:
            assert (a.double() - b.double()).abs().max() <= 4 * torch.finfo(torch.float16).eps * b.double().abs().max()


def test_module_is_handed_back_before_anything_is_formed(cuda_device):
    """What the attention would not take is seen before the projections run: more slices than the convolution has, taps of
    another device, fewer rows than landmarks, a number of iterations out of range."""
    from flashnystrom_b200 import _C
    mod, many = _module(torch.float16), _module(torch.float16, m=1)
    x = torch.randn(1, 100, 128, device="cuda").half()
    assert mod._native_forward(x) is not None
    host = _module(torch.float16)
    host.conv_weight = torch.nn.Parameter(host.conv_weight.detach().cpu())
    odd = _module(torch.float16)
    odd.config.newton_iter = 21
    for refused, y in ((many, torch.zeros(32768, 1, 128, device="cuda", dtype=torch.float16)), (host, x), (mod, x[:, :31]), (odd, x)):
        torch.cuda.synchronize()
        before = torch.cuda.memory_stats()["allocation.all.allocated"]
        assert refused._native_forward(y) is None
        assert torch.cuda.memory_stats()["allocation.all.allocated"] == before
    _C.check_device_status()
