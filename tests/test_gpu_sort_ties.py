"""Sort and argsort where many values share the bits that are sorted first, bit for
bit against the C oracle: floating-point values close to one another (their own range
is then taken), a close cluster among values spread over the whole range, and 64-bit
keys whose runs of ties are split once and twice."""

import numpy as np
import pytest

from test_gpu_sort_large import _gpu_sort, _oracle_sort, _same

pytestmark = pytest.mark.gpu

LENGTHS = {
    "short": [0, 1, 2, 3, 5, 8, 8, 7, 16, 15, 9, 24, 17, 32, 31, 25] * 30,
    "tiles": [33, 40, 2048, 700, 64, 100] * 3,
    "runs": [2049, 16_384, 40_000],
}


def _values(how, tname, n, rng):
    t = np.dtype(tname)
    if t.kind == "f":
        z = rng.standard_normal(n)
        if how == "close":
            x = 91.2 * (1 + z * 2.0**-20)
        elif how == "close to zero":  # the smallest numbers, of both signs, and zeros
            tiny = np.finfo(t).smallest_subnormal
            x = rng.integers(-40, 41, n) * tiny
        elif how == "mixed":
            x = np.where(rng.random(n) < 0.5, 91.2 * (1 + z * 2.0**-20), z * 1e4)
            x[rng.random(n) < 0.01] = np.nan
            x[rng.random(n) < 0.01] = -np.inf
            x[rng.random(n) < 0.02] = -0.0
        else:  # equal but for a few
            x = np.where(rng.random(n) < 0.9, 1.7e9, 1.7e9 + z * 1e-3)
        return x.astype(t)
    if how == "close":
        return (2**40 + rng.integers(0, 50, n)).astype(t)
    if how == "close to zero":
        return rng.integers(0, 3, n).astype(t)
    # runs of 50 to 100 equal upper bits; only the lowest 6 or 8 differ inside them
    groups, low = (300, 8) if how == "mixed" else (60, 6)
    return ((rng.integers(0, groups, n) << 54) + rng.integers(0, 1 << low, n)).astype(t)


@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("how", ["close", "close to zero", "mixed", "runs"])
@pytest.mark.parametrize("tname", ["float64", "float32", "int64", "uint64"])
def test_ties(lengths, how, tname):
    rng = np.random.default_rng(len(lengths) + 10 * len(tname) + len(how))
    off = np.concatenate([[0], np.cumsum(LENGTHS[lengths])]).astype(np.int64)
    x = _values(how, tname, int(off[-1]), rng)
    for arg in (True, False):
        for asc in (True, False):
            _same(_gpu_sort(arg, tname, "int64", x, off, len(x), asc),
                  _oracle_sort(arg, tname, "int64", x, off, len(x), asc))
