"""Sort and argsort at the edges of the GPU path's classes, bit for bit against
the C oracle: 32 elements (counted in a warp; 32 such lists are two halves of
its stage), 2048 (tiles of whole lists), 16384 (one run) and whole numbers of
runs and merge tiles; with 64-bit keys that share the 32 bits the radix sort
and the merges work on -- a cluster of close values beside far ones, in long
and in short groups of ties."""

import numpy as np
import pytest

from test_gpu_sort_large import _gpu_sort, _oracle_sort, _same

pytestmark = pytest.mark.gpu

LENGTHS = {
    "warp": [32] * 70 + [0, 1, 31, 16, 17] * 20 + [33, 32, 34],
    "tile": [33, 2048, 2047, 40, 64, 2048, 100, 0, 7] * 5,
    "run": [2049, 16_384, 16_385, 4096, 16_383],
    "merge": [32_768, 32_769, 36_864, 20_481, 70_000, 50],
}


def _values(tname, how, n, rng):
    if tname == "float64":
        if how == "cluster":
            x = 1.7e9 + rng.integers(0, 50_000, n) * 1e-3
            x[rng.random(n) < 0.01] = 0.0
            x[rng.random(n) < 0.01] = -1e300
            return x
        return rng.standard_normal(n)
    if tname in ("int64", "uint64"):
        info = np.iinfo(tname)
        x = rng.integers(info.min, info.max, n, dtype=tname, endpoint=True)
        if how == "cluster":
            x[rng.random(n) < 0.9] = 1 << 40
            near = rng.random(n) < 0.5
            x[near] = (1 << 41) + rng.integers(0, 100, int(near.sum())).astype(tname)
        return x
    if how == "cluster":
        return rng.integers(0, 3, n).astype(tname)
    return (rng.standard_normal(n) * 1000).astype(tname)


@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("how", ["spread", "cluster"])
@pytest.mark.parametrize("tname", ["float64", "int64", "uint64", "float32", "int16"])
def test_class_edges(lengths, how, tname):
    rng = np.random.default_rng(len(lengths) + 10 * len(tname) + len(how))
    off = np.concatenate([[0], np.cumsum(LENGTHS[lengths])]).astype(np.int64)
    x = _values(tname, how, int(off[-1]), rng)
    for arg in (True, False):
        for asc in (True, False):
            _same(_gpu_sort(arg, tname, "int64", x, off, len(x), asc),
                  _oracle_sort(arg, tname, "int64", x, off, len(x), asc))
