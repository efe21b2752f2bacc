"""The landmarks and the softmax-2 matrix bit for bit: the order in which their sums are formed is part of the result,
whichever kernel of a size range forms them."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _segment_sums(x, m, elems):
    """(BH, N, D) values -> the FP32 segment sums in the order of the pooling pass: of the rows that eight warps load at
    once, warp w holds the w-th group; a lane adds its rows in order, lanes of the same columns are added by doubling
    distance, then the eight groups in order."""
    BH, N, D = x.shape
    x = x.astype(np.float32)
    seg, rpw = N // m, 32 // (D // elems)
    out = np.zeros((BH, m, D), np.float32)
    for last in (False, True):
        ls = [m - 1] if last else list(range(m - 1))
        n = N - seg * (m - 1) if last else seg
        if not ls:
            continue
        rows = np.stack([x[:, seg * l:seg * l + n] for l in ls], 1)
        steps = -(-n // (8 * rpw))
        rows = np.concatenate([rows, np.zeros((BH, len(ls), steps * 8 * rpw - n, D), np.float32)], 2)
        rows = rows.reshape(BH, len(ls), steps, 8, rpw, D)
        acc = np.zeros((BH, len(ls), 8, rpw, D), np.float32)
        for s in range(steps):
            acc = acc + rows[:, :, s]
        o = 1
        while o < rpw:
            acc = acc + acc[:, :, :, np.arange(rpw) ^ o]
            o *= 2
        t = np.zeros((BH, len(ls), D), np.float32)
        for w in range(8):
            t = t + acc[:, :, w, 0]
        out[:, ls] = t
    return out


@pytest.mark.parametrize("BH,N,D,m,dtype,split_heads", [
    # at least 24 items per SM, so that a segment is one item.  By single warps: one load and its remainders, one
    # step, several steps, the longest; a last segment almost twice as long
    (2, 64, 64, 64, torch.float16, False), (28, 2000, 64, 64, torch.float16, True), (30, 6437, 64, 64, torch.bfloat16, False),
    (60, 33 * 31 + 30, 128, 33, torch.float16, True), (28, 64 * 60, 128, 64, torch.float32, False), (64, 700, 32, 33, torch.float32, False),
    (64, 5000, 16, 30, torch.bfloat16, False),
    # by whole CTAs
    (28, 64 * 300, 64, 64, torch.float16, True), (60, 32 * 200, 128, 32, torch.float32, False),
])
def test_segment_sums(cuda_device, BH, N, D, m, dtype, split_heads):
    from flashnystrom_b200 import _C
    gen = torch.Generator().manual_seed(N + D)
    q, k = (torch.randn(1, BH, N, D, generator=gen).to(dtype) for _ in range(2))
    qd, kd = (t.cuda() for t in (q, k))
    if split_heads and _C.tc_eligible(dtype, D, m):      # the head-split view of a (B, N, H * D) tensor
        qd, kd = (t.transpose(1, 2).contiguous().transpose(1, 2) for t in (qd, kd))
    res = _C.forward(qd, kd, kd, m, 1)
    elems = 4 if dtype == torch.float32 else 8
    length = np.full((m, 1), N // m, np.float32)
    length[-1] = N - (N // m) * (m - 1)
    f = np.float32(D ** -0.25) / length
    for got, x in ((res[3], q), (res[4], k)):
        want = _segment_sums(x[0].float().numpy(), m, elems) * f
        assert np.array_equal(got[0].cpu().numpy(), want)


@pytest.mark.parametrize("m", [1, 3, 31, 33, 62, 64])
def test_softmax2_rows(cuda_device, m):
    """Scores that every product forms exactly (one dimension, few bits), so that K2 and lse2 follow from expf, logf
    and the order of the row sum: columns 32, 16, 8, 4, 2 and 1 apart."""
    from flashnystrom_b200 import _C
    D, scale = 64, np.float32(64 ** -0.25)

    def preimage(t):                         # the float x with fl(x * scale) == t
        x = np.float32(t / float(scale))
        for y in (x, np.nextafter(x, np.float32(np.inf)), np.nextafter(x, np.float32(-np.inf))):
            if np.float32(y * scale) == t:
                return y
        return None
    rng = np.random.RandomState(m)
    exact = [t for t in (np.arange(-96, 97) / 32).astype(np.float32) if preimage(t) is not None]
    a, b = rng.choice(exact, m), rng.choice(exact, m)
    q, k = torch.zeros(1, 1, m, D), torch.zeros(1, 1, m, D)
    q[0, 0, :, 0] = torch.tensor([preimage(t) for t in a])
    k[0, 0, :, 0] = torch.tensor([preimage(t) for t in b])
    res = _C.forward(q.cuda(), k.cuda(), k.cuda(), m, 1)
    s = torch.zeros(m, 64, device="cuda")
    s[:, :m] = torch.tensor(np.outer(a, b), device="cuda")
    live = torch.arange(64, device="cuda") < m
    mx = torch.where(live, s, s.new_tensor(float("-inf"))).max(1, keepdim=True).values
    e = torch.where(live, torch.exp(s - mx), s.new_zeros(()))
    t = e
    for o in (32, 16, 8, 4, 2, 1):
        t = t[:, :o] + t[:, o:2 * o]
    assert torch.equal(res[11][0, 0], (e / t)[:, :m])
    assert torch.equal(res[8][0, 0], (mx + torch.log(t))[:, 0])
