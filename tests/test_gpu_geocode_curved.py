"""s1b_geocode where the TOPS terms bend from column to column: bursts of few
samples and many lines, whose FM rate and Doppler centroid change as much as a
whole swath's, and steeper and bent ones, against the general path (s1b_deramp
+ s1b_geo2rdr, which evaluates the terms at every pixel's own sample)."""
import copy

import pytest
import torch

from sentinel_gpu_processor_b200 import kernels, plan as P, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lines,samples", [(1530, 640), (1100, 400), (1500, 2600)])
@pytest.mark.parametrize("slope,bend", [(1.0, 0.0), (6.0, 0.0), (2.0, 30.0)])
@pytest.mark.parametrize("ci16", [False, True])
def test_terms_that_bend(cuda, lines, samples, slope, bend, ci16):
    sc = synth.make_pair("c1", seed=3, device=cuda, lines=lines, samples=samples)
    a = sc.ref[0]
    pl = copy.copy(P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], sc.rsc))
    swath = samples / a.radar.range_sampling_rate
    pl.fm[2] *= slope
    pl.fm[3] += bend * 0.02 * pl.fm[1] / swath ** 2 / 8
    pl.dc[3] += bend * 2.0 / swath ** 2
    slc = synth.cint16(sc.ref_slc[0]) if ci16 else sc.ref_slc[0]
    flat = slc.reshape(-1, 2) if ci16 else slc.reshape(-1)
    got, rows = kernels.geocode(pl, slc, sc.dem)
    want, wrows = kernels.geo2rdr(pl, sc.dem, kernels.deramp(pl, flat))
    assert torch.equal(rows, wrows) and torch.equal(got == 0, want == 0)
    got, want = got.to(torch.complex128), want.to(torch.complex128)
    # each path is within 2.1e-7 (2-norm) of float64
    assert float(torch.linalg.vector_norm(got - want)) <= 4.2e-7 * float(torch.linalg.vector_norm(want))
    # float32 roundings are as often up as down: the phases agree in the mean to
    # within a rounding of the phasors' (6e-8)
    m = want.abs() > 0.2 * want.abs().max()
    assert abs(float(torch.angle(got[m] * want[m].conj()).mean())) <= 6e-8
