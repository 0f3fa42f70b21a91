"""The timing hooks of the pair chains time the calls that the chain makes
without them: the same entry points in the same order, the same bits."""
import contextlib

import pytest
import torch

from sentinel_gpu_processor_b200 import chain, kernels, synth

pytestmark = pytest.mark.gpu


def _names(call, collect):
    seen, lib_call = [], kernels._call

    def record(name, fn, *args):
        seen.append((name, fn.__name__))
        return lib_call(name, fn, *args)

    timed = []

    @contextlib.contextmanager
    def timer(name):
        timed.append(name)
        yield

    kernels._call, kernels.timer = record, timer if collect else None
    try:
        out = call()
    finally:
        kernels._call, kernels.timer = lib_call, None
    return seen, timed, out


@pytest.mark.parametrize("frame", [False, True])
def test_timed_chain_is_the_chain(cuda, frame):
    sc = synth.make_pair("c0", seed=5, device=cuda, lines=331, samples=1187)
    ref, sec = sc.ref_slc[0], sc.sec_slc[0]
    if frame:
        ch = chain.FrameChain([sc.ref[0]], [sc.sec[0]], sc.rsc, sc.rowlook, sc.collook, sc.alpha, device=cuda)
        step = lambda: ch.run([ref], [sec], sc.dem)[0]  # noqa: E731
    else:
        ch = chain.PairChain(sc.ref[0], sc.sec[0], sc.rsc, sc.rowlook, sc.collook, sc.alpha, device=cuda)
        step = lambda: ch.run(ref, sec, sc.dem)  # noqa: E731
    plain, _, a = _names(step, False)
    ifg, filt, coh = a.ifg.clone(), a.filt.clone(), a.coh.clone()
    with_timer, timed, b = _names(step, True)
    assert with_timer == plain and timed == [n for n, _ in plain]
    for x, y in ((ifg, b.ifg), (filt, b.filt), (coh, b.coh)):
        assert torch.equal(x, y)
    ch.geo_events = []
    with_events, _, _ = _names(step, False)
    torch.cuda.synchronize()
    assert with_events == plain
    assert len(ch.geo_events) == 1 and ch.geo_events[0][0].elapsed_time(ch.geo_events[0][1]) > 0
