"""s1b_geo2rdr_offsets at the edges of its tiles and off its fast path: grids of
one pixel, odd sizes around the 128 columns and 64 rows of a CTA, rows of the
rasters permuted (angles beyond the Taylor range, seeds far from their roots)
and columns moved minutes along the orbit (off the patch), against the float64
oracle; the height-sensitivity form gives the same offsets."""
import numpy as np
import pytest
import torch

from helpers import oracle_radar
from oracle import radargrid as orr
from sentinel_gpu_processor_b200 import kernels, plan as P, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def scene(cuda):
    return synth.make_radar_pair("c0", seed=3, device=cuda, lines=160, samples=400)


def _check(sc, lat, lon, hgt):
    a, r = sc.sec, sc.ref
    pl = P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], None)
    rp = P.burst_plan(r.radar, r.orbit, r.fm, r.dc, r.bursts[0], None)
    lat, lon, hgt = (t.contiguous() for t in (lat, lon, hgt))
    az, rg = kernels.geo2rdr_offsets(pl, lat, lon, hgt)
    want = orr.offsets(*(t.cpu().numpy() for t in (lat, lon, hgt)), oracle_radar(a.radar), a.orbit,
                       a.bursts[0].azimuth_time)
    # the oracle stops within 5e-9 s x 0.1 (its linear rate) of the root: 2.5e-7
    # lines; float32 rounds the residual by 6e-8 of it; FP64 time and range by 4e-9
    for got, w, base in ((az, want[0], 3e-7), (rg, want[1], 1e-8)):
        assert np.all(np.abs(got.cpu().numpy() - w) <= base + 6.1e-8 * np.abs(w))
    az2, rg2, _, _ = kernels.geo2rdr_offsets_dh(pl, rp, lat, lon, hgt)
    for x, y in ((az, az2), (rg, rg2)):
        assert torch.allclose(x, y, rtol=1.2e-7, atol=4e-9)


@pytest.mark.parametrize("lines,samples", [(1, 1), (1, 33), (2, 128), (3, 129), (63, 40), (64, 127), (65, 257),
                                           (129, 400), (160, 1)])
def test_sizes(scene, lines, samples):
    _check(scene, *(t[:lines, :samples] for t in (scene.lat, scene.lon, scene.hgt)))


def test_rough_rasters(scene):
    p = torch.randperm(160, generator=torch.Generator().manual_seed(1)).to(scene.lat.device)
    _check(scene, *(t[p] for t in (scene.lat, scene.lon, scene.hgt)))


def test_off_the_patch(scene):
    lat = scene.lat.clone()
    lat[:, ::3] += 0.4  # 6 s along the orbit
    lat[70:80] -= 0.02
    _check(scene, lat, scene.lon, scene.hgt)
