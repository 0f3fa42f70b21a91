"""The adjoint at the look sizes where a tile's window sums change form (one
row per window up to all 16, one column per window up to the tile's 64, more
windows than threads, look columns that do not divide the tile, grids that end
inside a tile) against the float64 torch.autograd restatement
(oracle/adjoint.py), and a window too large for the stage."""
import numpy as np
import pytest
import torch

from helpers import oracle_burst, oracle_radar
from oracle import adjoint as oa
from oracle import geo2rdr as og2
from sentinel_gpu_processor_b200 import synth
from sentinel_gpu_processor_b200.refine import CoregProblem

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def stack(cuda):
    return synth.make_refine_stack(n_bursts=2, config="tiny", seed=6, device=cuda, margin=12)


def _oracle(stack, az0):
    acq = stack.sec_acq
    radar = oracle_radar(acq.radar)
    co = og2.burst_coefficients(radar, acq.orbit, acq.fm, acq.dc, oracle_burst(acq.bursts[0]))
    n = [t.cpu().numpy() for t in (stack.ref, stack.sec, az0, stack.rg0, stack.daz_dh, stack.drg_dh)]
    return [oa.AdjBurst(ref=n[0][b], sec=n[1][b], radar=radar, co=co, az0=n[2][b], rg0=n[3][b], daz_dh=n[4][b],
                        drg_dh=n[5][b]) for b in range(n[0].shape[0])]


def _check(stack, az0, rowlook, collook):
    dev = stack.ref.device
    p = CoregProblem(stack.sec_plans, stack.ref, stack.sec, az0, stack.rg0, stack.daz_dh, stack.drg_dh, rowlook, collook)
    rng = np.random.default_rng(3)
    params = torch.tensor(rng.normal(0, 0.03, (2, 6)), dtype=torch.float32, device=dev)
    dh = (2.0 * synth.gaussian_smooth(torch.randn(stack.dh_true.shape, generator=torch.Generator(dev).manual_seed(4),
                                                  device=dev), 5.0)).contiguous()
    J0 = float(p.objective(params, dh))
    J, gp, gh = p.gradient(params, dh)
    want, wp, wh = oa.torch_gradient(_oracle(stack, az0), params.cpu().numpy(), dh.cpu().numpy(), rowlook, collook)
    assert float(J) == J0
    assert abs(J0 - want) < 2e-6  # the objective's stated tolerance
    rel = lambda a, b: np.linalg.norm(a.double().cpu().numpy() - b) / np.linalg.norm(b)
    assert rel(gp, wp) < 1e-3 and rel(gh, wh) < 1e-3  # the gradient's


@pytest.mark.parametrize("rowlook,collook", [(1, 2), (2, 7), (4, 20), (8, 33), (16, 64), (1, 64), (16, 3)])
def test_looks(stack, rowlook, collook):
    _check(stack, stack.az0, rowlook, collook)


def test_window_beyond_the_stage(stack):
    """Offsets that jump by 20 lines inside a tile: its window exceeds the
    stage and every sample is read by itself."""
    az0 = stack.az0.clone()
    az0[:, :, 100:150] -= 20.0
    az0[:, :, 150:] += 15.0
    _check(stack, az0.contiguous(), 4, 20)
