"""s1b_geocode where the two columns of a gathered line turn against each other
by up to a third of a half-cycle (few samples, many lines, an FM rate three
times as steep), against the general path (s1b_deramp + s1b_geo2rdr)."""
import copy

import pytest
import torch

from sentinel_gpu_processor_b200 import kernels, plan as P, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lines,samples", [(1530, 640), (1100, 400)])
def test_turns_between_columns(cuda, lines, samples):
    sc = synth.make_pair("c1", seed=3, device=cuda, lines=lines, samples=samples)
    a = sc.ref[0]
    pl = copy.copy(P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], sc.rsc))
    pl.fm[2] *= 3.0
    slc = sc.ref_slc[0]
    got, _ = kernels.geocode(pl, slc, sc.dem)
    want, _ = kernels.geo2rdr(pl, sc.dem, kernels.deramp(pl, slc.reshape(-1)))
    d = (got - want).to(torch.complex128)
    # bursts whose columns do not turn differ by 1.5e-7 (2-norm); a turn of up to
    # 0.33 half-cycles rounded to float32 in each of four operations adds 0.33 pi
    # 2^-25 sqrt(12) = 1.1e-7 at most: 1.85e-7
    assert float(torch.linalg.vector_norm(d)) <= 1.85e-7 * float(torch.linalg.vector_norm(want.to(torch.complex128)))
