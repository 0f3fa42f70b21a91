"""s1b_geo2rdr_offsets on rasters with pixels that are no point: a NaN or an
infinity in latitude, longitude or height makes that pixel's offsets (and
sensitivities) no number and leaves every other pixel as it is without it,
wherever it lies in the kernel's tiles (32 columns by up to 64 rows, solved
about the middle pixel): at the middle, all around it, in whole rows, columns
and tiles."""
import numpy as np
import pytest
import torch

from helpers import oracle_radar
from oracle import radargrid as orr
from sentinel_gpu_processor_b200 import kernels, plan as P, synth

pytestmark = pytest.mark.gpu

LINES, SAMPLES = 160, 400
BAD = {
    "middles": lambda y, x: (x % 32 == 16) & (y % 4 == 0),
    "rows": lambda y, x: (y % 16 == 8) | (y % 16 == 0),
    "columns": lambda y, x: x % 3 == 1,
    "tiles": lambda y, x: ((x // 32 + y // 64) % 2 == 0) & ~((x == 70) & (y == 63)),
    "all but one": lambda y, x: ~((x == 45) & (y == 7)),
    "edges": lambda y, x: (x >= 384) | (y >= 144) | (x == 0),
}


@pytest.fixture(scope="module")
def scene(cuda):
    sc = synth.make_radar_pair("c0", seed=3, device=cuda, lines=LINES, samples=SAMPLES)
    a, r = sc.sec, sc.ref
    pl = P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], None)
    rp = P.burst_plan(r.radar, r.orbit, r.fm, r.dc, r.bursts[0], None)
    llh = [t.contiguous() for t in (sc.lat, sc.lon, sc.hgt)]
    want = orr.offsets(*(t.cpu().numpy() for t in llh), oracle_radar(a.radar), a.orbit, a.bursts[0].azimuth_time)
    sens = kernels.geo2rdr_offsets_dh(pl, rp, *llh)[2:]
    return pl, rp, llh, want, sens


@pytest.mark.parametrize("value", [float("nan"), float("inf"), float("-inf")])
@pytest.mark.parametrize("which", [0, 1, 2])
@pytest.mark.parametrize("where", sorted(BAD))
def test_other_pixels_keep_their_offsets(scene, where, which, value):
    pl, rp, llh, want, sens = scene
    y, x = np.mgrid[:LINES, :SAMPLES]
    bad = BAD[where](y, x)
    llh = [t.clone() for t in llh]
    llh[which][torch.from_numpy(bad).to(llh[0].device)] = value
    got = [t.cpu().numpy() for t in kernels.geo2rdr_offsets(pl, *llh)]
    got_dh = [t.cpu().numpy() for t in kernels.geo2rdr_offsets_dh(pl, rp, *llh)]
    for g in got + got_dh:
        assert np.all(np.isnan(g[bad])) and np.all(np.isfinite(g[~bad]))
    # the bounds of the finite rasters: the oracle stops within 2.5e-7 lines of
    # the root, float32 rounds the residual by 6e-8 of it, FP64 range by 4e-9
    for g in (got, got_dh):
        for v, w, base in zip(g, want, (3e-7, 1e-8)):
            assert np.all(np.abs(v - w)[~bad] <= base + 6.1e-8 * np.abs(w[~bad]))
    # a float32 rounding on either side
    for v, s in zip(got_dh[2:], sens):
        s = s.cpu().numpy()
        assert np.all(np.abs(v - s)[~bad] <= 1.3e-7 * np.abs(s[~bad]) + 1e-12)


def test_no_point_at_all(scene):
    pl, rp, llh, _, _ = scene
    for g in kernels.geo2rdr_offsets_dh(pl, rp, llh[0], llh[1], torch.full_like(llh[2], float("nan"))):
        assert bool(torch.isnan(g).all())
