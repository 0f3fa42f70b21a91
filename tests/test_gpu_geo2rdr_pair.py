"""s1b_geo2rdr_pair against s1b_deramp + s1b_geo2rdr of one burst after the
other: the same bits, for bursts of different sizes (odd and even widths, so
wide and narrow loads), windows of remainders, and a whole or windowed DEM."""
import pytest
import torch

from sentinel_gpu_processor_b200 import kernels, plan as P, synth

pytestmark = pytest.mark.gpu


def _burst(lines, samples, cuda, seed):
    sc = synth.make_pair("c0", seed=seed, device=cuda, lines=lines, samples=samples)
    a = sc.ref[0]
    return P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], sc.rsc), sc.ref_slc[0], sc


@pytest.mark.parametrize("sizes", [((96, 320), (96, 320)), ((331, 1187), (331, 1187)), ((160, 640), (333, 1031))])
def test_pair_equals_burst_by_burst(cuda, sizes):
    b = [_burst(*sizes[0], cuda, 3), _burst(*sizes[1], cuda, 3)]
    sc = b[1][2]
    plans = []
    for i, (lines, samples) in enumerate(sizes):  # both on the larger scene's grid
        a = sc.ref[0] if i == 1 else b[0][2].ref[0]
        plans.append(P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], sc.rsc))
    slcs = [b[0][1], b[1][1]]
    der = [torch.empty(p.lines * p.samples, dtype=torch.complex64, device=cuda) for p in plans]
    out = [torch.empty((p.nrow, p.ncol), dtype=torch.complex64, device=cuda) for p in plans]
    rows = torch.full((4,), 77, dtype=torch.int32, device=cuda)
    kernels.geo2rdr_pair(plans, slcs, sc.dem, der, out, rows)
    for i, p in enumerate(plans):
        d = kernels.deramp(p, slcs[i].reshape(-1))
        want, wrows = kernels.geo2rdr(p, sc.dem, d)
        assert torch.equal(torch.view_as_real(d), torch.view_as_real(der[i]))
        assert torch.equal(torch.view_as_real(want), torch.view_as_real(out[i]))
        assert torch.equal(wrows, rows[2 * i:2 * i + 2])


def test_bad_arguments(cuda):
    p, slc, sc = _burst(96, 320, cuda, 3)
    der = [torch.empty(p.lines * p.samples, dtype=torch.complex64, device=cuda) for _ in range(2)]
    out = [torch.empty((p.nrow, p.ncol), dtype=torch.complex64, device=cuda) for _ in range(2)]
    rows = torch.empty(4, dtype=torch.int32, device=cuda)
    for bad in ((slc, slc[:-1]), (slc, slc.to(torch.complex128))):
        with pytest.raises(ValueError):
            kernels.geo2rdr_pair([p, p], bad, sc.dem, der, out, rows)
    with pytest.raises(ValueError):
        kernels.geo2rdr_pair([p, p], (slc, slc), sc.dem.to(torch.int32), der, out, rows)
    with pytest.raises(ValueError):
        kernels.geo2rdr_pair([p, p], (slc, slc), sc.dem, der, out, rows[:3])
