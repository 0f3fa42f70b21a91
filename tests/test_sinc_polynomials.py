"""The polynomials of the 8-tap windowed-sinc weights and their derivatives
(csrc/s1b_sinc.cuh), evaluated in float32 as the kernels do, against the
definition in float64: within the bounds that the header states, and in the
mean square no farther than a table of 1024 bins with linear interpolation.  The
derivatives go with weights from such a table: no bias against a table of
derivatives."""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "sentinel_gpu_processor_b200", "csrc",
                   "s1b_sinc.cuh")


def _table(text, name):
    n, body = re.search(name + r"\[4 \* (\d)\] = \{(.*?)\};", text, re.S).groups()
    return np.array([float(x) for x in re.findall(r"-?\d\.\d+e[+-]\d+", body)], dtype=np.float32).reshape(4, int(n), 2)


def _definition(f):
    """Normalised weights [8, n] of the taps -3 .. 4 at the fractions f, and their derivatives."""
    x = np.arange(-3, 5)[:, None] - f[None, :]
    px = np.pi * x
    safe = np.where(np.abs(x) < 1e-5, 1.0, x)
    s = np.sinc(x)
    ds = np.where(np.abs(x) < 1e-5, -np.pi ** 2 / 3 * x, (np.cos(px) - s) / safe)
    c, dc = 0.5 + 0.5 * np.cos(px / 4), -np.pi / 8 * np.sin(px / 4)
    u, du = s * c, -(ds * c + s * dc)
    su, sdu = u.sum(0), du.sum(0)
    return u / su, (du * su - u * sdu) / su ** 2


def _fma(a, b, c):
    return (a.astype(np.float64) * b.astype(np.float64) + c).astype(np.float32)  # exact product, one sum


def _evaluate(table, f, even):
    """Taps 4 + j: p + t q, taps 3 - j: +-(p - t q), p and q by Horner's rule in v = t^2."""
    t = f - np.float32(0.5)
    v = t * t
    out = [None] * 8
    for j in range(4):
        p, q = (np.full_like(f, table[j, -1, i]) for i in (0, 1))
        for k in range(table.shape[1] - 2, -1, -1):
            p, q = _fma(p, v, table[j, k, 0]), _fma(q, v, table[j, k, 1])
        out[4 + j] = _fma(t, q, p)
        out[3 - j] = _fma(-t, q, p) if even else _fma(t, q, -p)
    return np.array(out)


@pytest.fixture(scope="module")
def text():
    with open(SRC) as fh:
        return fh.read()


@pytest.mark.parametrize("name,which", [("c_sinc8", 0), ("c_dsinc8", 1)])
def test_within_the_stated_bound(text, name, which):
    flat = " ".join(line.lstrip("/ ") for line in text.splitlines())
    bound = float(re.search((r"the weights are within (\S+);", r"From w' itself they are within (\S+) ")[which],
                            flat).group(1))
    f = np.append(np.arange(1 << 17) / (1 << 17), 1 - 2.0 ** -24).astype(np.float32)
    got = _evaluate(_table(text, name), f, even=which == 0)
    assert np.abs(got - _definition(f.astype(np.float64))[which]).max() <= bound


def _lerp_table(which, f):
    bins = _definition(np.arange(1025) / 1024)[which].astype(np.float32)
    pos = f * np.float32(1024)
    b = pos.astype(np.int64)
    return _fma(pos - b.astype(np.float32), bins[:, b + 1] - bins[:, b], bins[:, b])


@pytest.mark.parametrize("name,which", [("c_sinc8", 0), ("c_dsinc8", 1)])
def test_no_farther_than_a_table(text, name, which):
    f = ((np.arange(1 << 16) + 0.5) / (1 << 16)).astype(np.float32)
    want = _definition(f.astype(np.float64))[which]
    rms = lambda e: np.sqrt((e ** 2).mean(1))  # noqa: E731
    assert np.all(rms(_evaluate(_table(text, name), f, even=which == 0) - want) <= rms(_lerp_table(which, f) - want))


def test_slopes_as_the_table_in_the_mean(text):
    f = ((np.arange(1 << 16) + 0.5) / (1 << 16)).astype(np.float32)
    got = _evaluate(_table(text, "c_dsinc8"), f, even=False).astype(np.float64)
    # a sixth of the float32 spacing below 1
    assert np.abs((got - _lerp_table(1, f)).mean(1)).max() <= 1e-8
