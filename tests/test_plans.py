"""The plans of the autograd function's path: what is kept between calls, and for whom.  No GPU: the library is a stub."""
import torch
import pytest

from flashnystrom_b200 import _C


class _Library:
    """Workspace sizes follow the device that is current, as in the library (SM count)."""
    def __init__(self):
        self.current, self.asked = 0, 0

    def fnb_check_shape(self, shape):
        return 0

    def fnb_fwd_workspace_bytes(self, shape):
        self.asked += 1
        return 1000 * (self.current + 1)

    def fnb_bwd_workspace_bytes(self, shape):
        return 2000 * (self.current + 1)


@pytest.fixture
def library(monkeypatch):
    lib = _Library()

    class On:
        def __init__(self, dev):
            self.dev = dev

        def __enter__(self):
            self.before, lib.current = lib.current, self.dev.index

        def __exit__(self, *exc):
            lib.current = self.before
    monkeypatch.setattr(_C, "_on_device", On)
    monkeypatch.setattr(_C, "_plans", {})
    return lib


def _plan(lib, index, N=256, kappa=0.0):
    return _C._plan(lib, torch.device("cuda", index), 1, 2, N, 64, 32, 6, torch.float16, kappa, 0)


@pytest.mark.parametrize("first", [0, 1])
def test_every_device_has_its_own_sizes(library, first):
    for index in (first, 1 - first, first):
        plan = _plan(library, index)
        assert (plan.fwd_ws, plan.bwd_ws) == (1000 * (index + 1), 2000 * (index + 1))
    assert library.asked == 2


def test_plans_are_bounded(library):
    for N in range(256, 256 + 2 * _C._MAX_PLANS):
        _plan(library, 0, N=N)
        assert len(_C._plans) <= _C._MAX_PLANS
    assert _plan(library, 0, N=256).shape.seq_len == 256


def test_flags_have_plans_of_their_own(library, monkeypatch):
    plain = _plan(library, 0)
    monkeypatch.setattr(_C, "_flags", 1)
    forced = _plan(library, 0)
    assert (plain.shape.flags, forced.shape.flags) == (0, 1)
    monkeypatch.setattr(_C, "_flags", 0)
    assert _plan(library, 0) is plain


def test_other_numbers_than_floats_are_not_kept(library):
    class K(float):
        pass
    a, b = _plan(library, 1, kappa=K(5.0)), _plan(library, 1, kappa=5.0)
    assert a is not b and a.shape.kappa_star == b.shape.kappa_star == 5.0 and a.fwd_ws == 2000
    with pytest.raises(RuntimeError):
        _plan(library, 0, kappa=float("nan"))
    with pytest.raises(RuntimeError):
        _plan(library, 0, kappa="5")
