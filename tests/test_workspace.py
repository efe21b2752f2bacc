"""Workspace sizes through the C ABI (no GPU: without a device the library sizes for 148 SMs)."""
import ctypes

import pytest
import torch

from flashnystrom_b200 import _C, _lib

GENERIC = _lib.FNB_FLAG_FORCE_GENERIC


def _bytes(BH, N, D, m, flags=0):
    lib = _lib.load()
    shape = _C._shape_struct(1, BH, N, D, m, 6, torch.float16, 0.0)
    shape.flags = flags
    return lib.fnb_fwd_workspace_bytes(ctypes.byref(shape)), lib.fnb_bwd_workspace_bytes(ctypes.byref(shape))


@pytest.mark.parametrize("m", [65, 128])
def test_scratch_of_the_pseudoinverse_does_not_grow_with_the_slices(m):
    """More than 64 landmarks: at most one scratch area per pair of SMs.  What a slice adds beyond that is its landmark-sized
    tensors, the same as with 64 landmarks but for their size."""
    areas = 74 if not torch.cuda.is_available() else torch.cuda.get_device_properties(0).multi_processor_count // 2
    for few, many in ((areas, 4 * areas),):
        for k in (0, 1):
            per_slice = (_bytes(many, 256, 64, m)[k] - _bytes(few, 256, 64, m)[k]) / (many - few)
            assert per_slice < 0.4e6, per_slice       # (an area is 0.75 MB forward, 1.5 MB backward)


@pytest.mark.parametrize("BH", [1, 16, 512])
def test_no_more_than_the_cuda_core_kernels_at_many_slices(BH):
    plain, generic = _bytes(BH, 256, 64, 128), _bytes(BH, 256, 64, 128, GENERIC)
    if BH == 512:
        assert plain[0] < generic[0] and plain[1] < generic[1]
    assert plain[0] < generic[0] + 0.76e6 * min(BH, 80) and plain[1] < generic[1] + 1.6e6 * min(BH, 80)
