"""s1b_stitch at the sizes where its passes change form: overlaps of one
pixel, of odd and even counts, of equal angles, larger than the cluster's
shared memory holds, tables of more bursts than a launch takes by value, and
bursts given as separate tensors, views and conjugates."""
import numpy as np
import pytest
import torch

from oracle import stitch as ost
from sentinel_gpu_processor_b200 import formats
from sentinel_gpu_processor_b200.stitch import stitch_bursts

pytestmark = pytest.mark.gpu


def _column(n, h, w, overlap, seed, equal=False, shift=0):
    """n bursts of h x w below one another, each overlapping the one above by `overlap` rows."""
    rng = np.random.default_rng(seed)
    nrow0, ncol0 = (h - overlap) * (n - 1) + h + 3, w + shift * n + 4
    out = []
    for k in range(n):
        t, l = 2 + k * (h - overlap), 1 + shift * k
        a = np.exp(1j * 0.37 * k) * np.ones((h, w))
        if not equal:
            a = a * rng.rayleigh(1.0, (h, w)) * np.exp(1j * rng.normal(0, 0.3, (h, w)))
            a[rng.random((h, w)) < 0.03] = 0
        out.append((formats.make_header(nrow0, ncol0, l, t, l + w, t + h), a.astype(np.complex64), 1, k))
    return out, nrow0, ncol0


# h, w, overlap, bursts: 1 and 2 overlap pixels, odd and even counts, a whole row of
# threads, more overlap than 16 x 40960 kept angles, 97 bursts (a table in the workspace)
@pytest.mark.parametrize("n,h,w,overlap,shift", [
    (2, 5, 1, 1, 0), (2, 5, 2, 1, 0), (3, 9, 7, 3, 1), (3, 40, 1024, 16, 0), (4, 33, 517, 31, 2),
    (2, 800, 900, 760, 0), (97, 6, 40, 2, 0), (2, 7, 11, 0, 0)])
@pytest.mark.parametrize("out_float", [False, True])
def test_stitch_sizes(cuda, n, h, w, overlap, shift, out_float):
    bursts, nrow0, ncol0 = _column(n, h, w, overlap, seed=n * 1000 + w, shift=shift)
    if out_float:
        bursts = [(hd, np.where(d != 0, np.angle(d), 0).astype(np.float32), s, g) for hd, d, s, g in bursts]
    _compare(cuda, bursts, nrow0, ncol0, out_float)


def test_stitch_equal_angles(cuda):
    bursts, nrow0, ncol0 = _column(3, 20, 64, 8, seed=5, equal=True)
    _compare(cuda, bursts, nrow0, ncol0, False)


def _compare(cuda, bursts, nrow0, ncol0, out_float):
    want = ost.stitch(bursts, nrow0, ncol0, out_float)
    dev = [(tuple(int(v) for v in hd[2:6]), torch.from_numpy(d).to(cuda), s, g) for hd, d, s, g in bursts]
    got = stitch_bursts(dev, nrow0, ncol0, out_float).cpu().numpy()
    assert np.array_equal(got != 0, want != 0)
    # offsets add up down the column: float32 angles, one rounding (6e-8 of pi) per burst
    tol = 1e-6 * len(bursts)
    d = np.angle(np.exp(1j * (got.astype(np.float64) - want))) if out_float else got - want
    assert np.abs(d).max() <= tol * (1.0 if out_float else np.abs(want).max())


def test_stitch_views(cuda):
    bursts, nrow0, ncol0 = _column(3, 30, 50, 10, seed=9)
    want = stitch_bursts([(tuple(int(v) for v in hd[2:6]), torch.from_numpy(d).to(cuda), s, g)
                          for hd, d, s, g in bursts], nrow0, ncol0)
    views = []
    for k, (hd, d, s, g) in enumerate(bursts):
        z = torch.from_numpy(d).to(cuda)
        if k == 0:
            z = z.conj().resolve_conj().conj()           # a lazily conjugated tensor
        elif k == 1:
            z = z.t().contiguous().t()                   # column-major
        else:
            big = torch.zeros((32, 61), dtype=z.dtype, device=cuda)
            big[1:31, 5:55] = z
            z = big[1:31, 5:55]                          # a window
        views.append((tuple(int(v) for v in hd[2:6]), z, s, g))
    got = stitch_bursts(views, nrow0, ncol0)
    assert torch.equal(torch.view_as_real(got), torch.view_as_real(want))
    with pytest.raises(ValueError):
        stitch_bursts([(views[0][0], views[0][1].cpu(), 1, 0)], nrow0, ncol0)
