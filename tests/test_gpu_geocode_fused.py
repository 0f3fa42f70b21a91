"""s1b_geocode (deramp fused into the gathers) against the general path
(s1b_deramp + s1b_geo2rdr) over the forms it accepts: both sample types, odd
widths, windows of few tiles (8 rows) and of many (32 rows) with remainders,
culling on and off, validity limits beyond the raster, no valid pixel, a DEM
given whole or as the window."""
import copy

import numpy as np
import pytest
import torch

from sentinel_gpu_processor_b200 import _lib, geo2rdr, kernels, plan as P, synth

pytestmark = pytest.mark.gpu

# both paths are within 2.1e-7 (2-norm) of float64 at these sizes: the sum of
# the two, rounded up
TOL = 5e-7


def _scene(lines, samples, cuda, seed=3):
    sc = synth.make_pair("c1" if lines > 700 else "c0", seed=seed, device=cuda, lines=lines, samples=samples)
    a = sc.ref[0]
    return sc, P.burst_plan(a.radar, a.orbit, a.fm, a.dc, a.bursts[0], sc.rsc)


def _general(pl, slc, dem):
    flat = slc.reshape(-1, 2) if slc.dtype == torch.int16 else slc.reshape(-1)
    return kernels.geo2rdr(pl, dem, kernels.deramp(pl, flat))


def _check(pl, slc, dem):
    got, rows = kernels.geocode(pl, slc, dem)
    want, wrows = _general(pl, slc, dem)
    assert torch.equal(rows, wrows)
    assert torch.equal(got == 0, want == 0)
    n = torch.linalg.vector_norm(want.to(torch.complex128))
    assert float(torch.linalg.vector_norm((got - want).to(torch.complex128))) <= TOL * float(n)
    return got, rows


@pytest.mark.parametrize("lines,samples", [(96, 321), (160, 640), (331, 1187), (512, 2048), (901, 9001)])
@pytest.mark.parametrize("ci16", [False, True])
def test_matches_general_path(cuda, lines, samples, ci16):
    sc, pl = _scene(lines, samples, cuda)
    slc = synth.cint16(sc.ref_slc[0]) if ci16 else sc.ref_slc[0]
    got, rows = _check(pl, slc, sc.dem)
    assert int(rows[1]) > int(rows[0]) >= 0
    win = sc.dem[pl.win_top:pl.win_bottom, pl.win_left:pl.win_right]
    again, _ = kernels.geocode(pl, slc, win)
    assert torch.equal(torch.view_as_real(again), torch.view_as_real(got))
    kernels.set_geocode_culling(False)
    try:
        off, orows = kernels.geocode(pl, slc, sc.dem)
    finally:
        kernels.set_geocode_culling(True)
    assert torch.equal(torch.view_as_real(off), torch.view_as_real(got)) and torch.equal(orows, rows)


@pytest.mark.parametrize("limits", [(-20, 10 ** 6, -5, 10 ** 6), (0, 331, 0, 1187), (150, 170, 500, 503),
                                    (200, 190, 40, 1100), (24, 300, 1186, 1187)])
def test_validity_limits(cuda, limits):
    sc, pl = _scene(331, 1187, cuda)
    pl = copy.copy(pl)
    pl.first_valid_line, pl.last_valid_line, pl.first_valid_sample, pl.last_valid_sample = limits
    _check(pl, sc.ref_slc[0], sc.dem)


def test_geocode_burst_keeps_a_given_deramp_buffer(cuda):
    sc, pl = _scene(160, 640, cuda)
    buf = torch.zeros(160 * 640, dtype=torch.complex64, device=cuda)
    a = geo2rdr.geocode_burst(pl, sc.ref_slc[0], sc.dem, deramped=buf)
    assert torch.equal(torch.view_as_real(buf), torch.view_as_real(kernels.deramp(pl, sc.ref_slc[0].reshape(-1))))
    b = geo2rdr.geocode_burst(pl, sc.ref_slc[0], sc.dem)
    assert np.array_equal(a[0], b[0]) and a[1].shape == b[1].shape


def test_bad_arguments(cuda):
    sc, pl = _scene(96, 320, cuda)
    with pytest.raises(ValueError):
        kernels.geocode(pl, sc.ref_slc[0][:-1], sc.dem)
    with pytest.raises(ValueError):
        kernels.geocode(pl, sc.ref_slc[0].to(torch.complex128), sc.dem)
    with pytest.raises(ValueError):
        kernels.geocode(pl, sc.ref_slc[0], sc.dem.to(torch.int32))
    assert _lib.load().s1b_geocode_scratch_bytes(pl) == 24 * pl.samples
