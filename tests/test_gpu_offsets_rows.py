"""s1b_geo2rdr_offsets over the widths at which a block takes 4, 8, 16, 32 and 64
rows (its height-sensitivity form the same or fewer), with and without pixels
that are no point at the middles of the tiles: a small scene side by side many
times, against its float64 oracle."""
import numpy as np
import pytest
import torch

from helpers import oracle_radar
from oracle import radargrid as orr
from sentinel_gpu_processor_b200 import kernels, plan as P, synth

pytestmark = pytest.mark.gpu

LINES, SAMPLES = 161, 400


@pytest.fixture(scope="module")
def scene(cuda):
    sc = synth.make_radar_pair("c0", seed=3, device=cuda, lines=LINES, samples=SAMPLES)
    a, r = sc.sec, sc.ref
    pl = P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], None)
    rp = P.burst_plan(r.radar, r.orbit, r.fm, r.dc, r.bursts[0], None)
    llh = [t.contiguous() for t in (sc.lat, sc.lon, sc.hgt)]
    _, _, az, rg = orr.offsets(*(t.cpu().numpy() for t in llh), oracle_radar(a.radar), a.orbit,
                               a.bursts[0].azimuth_time)
    sens = [t.cpu().numpy() for t in kernels.geo2rdr_offsets_dh(pl, rp, *llh)[2:]]
    return pl, rp, llh, az, rg, sens


@pytest.mark.parametrize("holes", [False, True])
@pytest.mark.parametrize("lines,columns", [(160, 900), (160, 3000), (161, 6000), (159, 12800), (160, 17001),
                                           (130, 24000), (161, 40000)])
def test_rows_per_block(scene, lines, columns, holes):
    pl, rp, llh, az, rg, sens = scene
    n = -(-columns // SAMPLES)
    llh = [t[:lines].repeat(1, n)[:, :columns].contiguous() for t in llh]
    az, rg, s0, s1 = (np.tile(v[:lines], (1, n))[:, :columns] for v in (az, rg, *sens))
    y, x = np.arange(lines)[:, None], np.arange(columns)[None, :]
    bad = (x % 32 == 16) & (y % 2 == 0) & holes
    if holes:
        llh[2][torch.from_numpy(bad).to(llh[2].device)] = float("nan")
    got = [t.cpu().numpy() for t in kernels.geo2rdr_offsets(pl, *llh)]
    got_dh = [t.cpu().numpy() for t in kernels.geo2rdr_offsets_dh(pl, rp, *llh)]
    for g in got + got_dh:
        assert np.array_equal(np.isnan(g), bad)
    # the oracle stops within 2.5e-7 lines of the root, float32 rounds the
    # residual by 6e-8 of it, FP64 time and range by 4e-9
    for g in (got, got_dh):
        for v, w, base in zip(g, (az - y, rg - x), (3e-7, 1e-8)):
            assert np.all((np.abs(v - w) <= base + 6.1e-8 * np.abs(w))[~bad])
    # sensitivities of the same points: a float32 rounding on either side (the
    # reference's line, and with it the time it is seen at, is the same)
    for v, w in zip(got_dh[2:], (s0, s1)):
        assert np.all((np.abs(v - w) <= 1.3e-7 * np.abs(w) + 1e-12)[~bad])
