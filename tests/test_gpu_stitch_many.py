"""s1b_stitch where more bursts lie over one another than its kernels list (32
under one overlap or in one block of the frame), in one and in several
subswaths, with empty pixels so that an overlap's pixels belong to several
earlier bursts, against the oracle; and an overlap larger than 16 blocks keep
in shared memory (16 x 22528 products)."""
import numpy as np
import pytest
import torch

from oracle import stitch as ost
from sentinel_gpu_processor_b200 import formats
from sentinel_gpu_processor_b200.stitch import stitch_bursts

pytestmark = pytest.mark.gpu


def _pile(n, h, w, step, swaths, seed, holes=0.3):
    """n bursts a subswath, h x w, each `step` rows below the one before, a share of the pixels empty."""
    rng = np.random.default_rng(seed)
    nrow0, ncol0 = h + step * (n - 1) + 3, w + 15 * (swaths - 1) + 4
    out = []
    for s in range(swaths):
        for k in range(n):
            t, l = 1 + k * step, 2 + 15 * s
            a = rng.rayleigh(1.0, (h, w)) * np.exp(1j * (0.37 * k + 0.2 * s + rng.normal(0, 0.3, (h, w))))
            a[rng.random((h, w)) < holes] = 0
            out.append((formats.make_header(nrow0, ncol0, l, t, l + w, t + h), a.astype(np.complex64), s + 1,
                        100 * s + k))
    return out, nrow0, ncol0


# 33 and 40 bursts over one another: one more than is listed, and well above; 80: a
# table in the workspace; two and three subswaths: the frame's blocks fill with the first
@pytest.mark.parametrize("n,h,w,step,swaths,holes", [
    (33, 60, 40, 1, 1, 0.3), (40, 60, 37, 1, 1, 0.9), (40, 60, 300, 1, 2, 0.3), (80, 90, 21, 1, 1, 0.3),
    (20, 60, 50, 1, 3, 0.5), (36, 48, 70, 1, 3, 0.97), (3, 700, 600, 20, 1, 0.3)])
@pytest.mark.parametrize("out_float", [False, True])
def test_many_over_one_another(cuda, n, h, w, step, swaths, holes, out_float):
    bursts, nrow0, ncol0 = _pile(n, h, w, step, swaths, n + w, holes)
    if out_float:
        bursts = [(hd, np.where(d != 0, np.angle(d), 0).astype(np.float32), s, g) for hd, d, s, g in bursts]
    want = ost.stitch(bursts, nrow0, ncol0, out_float)
    dev = [(tuple(int(v) for v in hd[2:6]), torch.from_numpy(d).to(cuda), s, g) for hd, d, s, g in bursts]
    got = stitch_bursts(dev, nrow0, ncol0, out_float).cpu().numpy()
    assert np.array_equal(got != 0, want != 0)
    # offsets add up burst by burst: float32 angles, one rounding (6e-8 of pi) each
    tol = 1e-6 * n
    d = np.angle(np.exp(1j * (got.astype(np.float64) - want))) if out_float else got - want
    assert np.abs(d).max() <= tol * (1.0 if out_float else np.abs(want).max())
