"""Resampling where consecutive tiles of a block read far-apart samples: the
offsets jump from tile to tile (16 x 64 outputs each), some tiles spread over
more than the staged window holds and some leave the burst altogether, so each
tile must be staged from its own coordinate range; against the float64 oracle,
and the same bits from run to run."""
import numpy as np
import pytest
import torch

from helpers import oracle_burst, oracle_radar, rel_err
from oracle import geo2rdr as og2
from oracle import radargrid as orr
from sentinel_gpu_processor_b200 import kernels, plan as P, synth

pytestmark = pytest.mark.gpu

TH, TW = 16, 64


@pytest.mark.parametrize("lines,samples", [(160, 640), (523, 2050)])
def test_tiles_of_different_ranges(cuda, lines, samples):
    sc = synth.make_radar_pair("c0", seed=17, device=cuda, lines=lines, samples=samples)
    a = sc.sec
    pl = P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], None)
    rng = np.random.default_rng(5)
    shape = (-(-lines // TH), -(-samples // TW))
    az = np.kron(rng.uniform(-40, 40, shape), np.ones((TH, TW)))[:lines, :samples]
    rg = np.kron(rng.uniform(-90, 90, shape), np.ones((TH, TW)))[:lines, :samples]
    kind = np.kron(rng.integers(0, 4, shape), np.ones((TH, TW), int))[:lines, :samples]
    az = np.where(kind == 1, az + 0.6 * (np.arange(lines) % TH)[:, None], az)  # beyond 32 staged rows in places
    rg = np.where(kind == 2, rg + 1.3 * (np.arange(samples) % TW)[None, :], rg)  # beyond 96 staged columns
    rg = np.where(kind == 3, rg + rng.choice([0, 1e5], size=shape).repeat(TH, 0).repeat(TW, 1)[:lines, :samples], rg)
    az, rg = (x.astype(np.float32) for x in (az, rg))
    taz, trg = (torch.from_numpy(x).to(cuda) for x in (az, rg))
    status = torch.full((1,), 7, dtype=torch.int32, device=cuda)
    got = kernels.resample(pl, sc.sec_slc, taz, trg, status=status)
    again = kernels.resample(pl, sc.sec_slc, taz, trg, status=status)
    assert status.item() == 0
    assert torch.equal(got, again)
    co = og2.burst_coefficients(oracle_radar(a.radar), a.orbit, a.fm, a.dc, oracle_burst(a.bursts[0]))
    want, ok = orr.resample(sc.sec_slc.cpu().numpy(), oracle_radar(a.radar), co,
                            np.arange(lines)[:, None] + az.astype(np.float64),
                            np.arange(samples)[None, :] + rg.astype(np.float64), "sinc8")
    got = got.cpu().numpy()
    assert ok.any() and not ok.all()
    assert np.array_equal(np.abs(got) > 0, np.abs(want) > 0)
    # as the other sinc comparisons: float32 weights, sums and phasors
    assert rel_err(got, want) < 2e-5
