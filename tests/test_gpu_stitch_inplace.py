"""s1b_stitch with a frame that lies over the bursts it is made of: the same
frame, bit by bit, as one beside them, from a call and from a captured graph."""
import ctypes

import numpy as np
import pytest
import torch

from sentinel_gpu_processor_b200 import _lib

pytestmark = pytest.mark.gpu

H, W, N = 40, 300, 6


def _bursts(out_float):
    rng = np.random.default_rng(4)
    step, table, data = H - 9, [], []
    for k in range(N):
        sw, row = 1 + k // 3, k % 3
        l, t = 2 + 250 * (sw - 1), 1 + row * step
        a = rng.rayleigh(1.0, (H, W)) * np.exp(1j * (0.6 * k + rng.normal(0, 0.3, (H, W))))
        a[rng.random((H, W)) < 0.05] = 0
        data.append(np.where(a != 0, np.angle(a), 0).astype(np.float32) if out_float else a.astype(np.complex64))
        table.append(_lib.StitchBurst(k * H * W, l, t, l + W, t + H, sw, k))
    return np.concatenate([d.ravel() for d in data]), (_lib.StitchBurst * N)(*table), 2 * step + H + 5, 250 + W + 6


def _stitch(arr, data_ptr, out_float, nrow, ncol, frame_ptr, ws):
    _lib.check(_lib.load().s1b_stitch(arr, N, ctypes.c_void_p(data_ptr), int(out_float), nrow, ncol,
                                      ctypes.c_void_p(frame_ptr), None, _lib.dptr(ws), ws.numel(),
                                      _lib.stream_ptr()), "s1b_stitch")


# the frame's start against the bursts': at them, inside them, over their last element, over their first
@pytest.mark.parametrize("where", ["start", "inside", "last", "first"])
@pytest.mark.parametrize("captured", [False, True])
@pytest.mark.parametrize("out_float", [False, True])
def test_frame_over_the_bursts(cuda, where, captured, out_float):
    host, arr, nrow, ncol = _bursts(out_float)
    n, m = host.size, nrow * ncol
    ws = torch.empty(int(_lib.load().s1b_stitch_workspace_bytes(arr, N, int(out_float))), dtype=torch.uint8,
                     device=cuda)
    data = torch.from_numpy(host).to(cuda)
    want = torch.full((m,), 7.0, dtype=data.dtype, device=cuda)
    _stitch(arr, data.data_ptr(), out_float, nrow, ncol, want.data_ptr(), ws)
    buf = torch.zeros(n + 2 * m, dtype=data.dtype, device=cuda)
    at = {"start": m, "inside": m + n // 3, "last": m + n - 1, "first": 1}[where]
    es = buf.element_size()
    args = (arr, buf.data_ptr() + m * es, out_float, nrow, ncol, buf.data_ptr() + at * es, ws)
    if captured:
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            _stitch(*args)
    for _ in range(2):  # the bursts anew: the frame has replaced some of them
        buf[m:m + n] = data
        if captured:
            g.replay()
        else:
            _stitch(*args)
        assert torch.equal(buf[at:at + m], want)
        rest = torch.cat([buf[m:max(m, min(at, m + n))], buf[max(m, at + m):m + n] if at + m < m + n else buf[:0]])
        kept = torch.cat([data[:max(0, min(at - m, n))], data[max(0, at):] if at + m < m + n else data[:0]])
        assert torch.equal(rest, kept)
