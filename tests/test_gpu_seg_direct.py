"""Lists of 8-byte elements that the reducers take 32 at a time straight from memory
(a mean of at least 96, none above 288): the edges of that rule, groups of four that
are not full, empty lists among them, values outside the sums' window, zeros and NaN
that win, and the same list beside different neighbours."""

import math

import numpy as np
import pytest

import oracle
from test_gpu_seg_tile import _call, _values

pytestmark = pytest.mark.gpu

LENGTHS = {
    "96": [96] * 33,
    "just below": [96] * 31 + [95] + [96] * 40,
    "288": [288] * 70,
    "289 among them": ([288] * 20 + [289]) * 4 + [200] * 37,
    "empty": [0, 288, 288, 0, 250, 0, 288] * 12,
    "few": [150, 97, 103],
    "one": [288],
    "mixed": [1, 280, 7, 260, 33, 120, 288, 0, 2, 250] * 17 + [8] * 50 + [130] * 41 + [300] * 3,
}
SHIFTS = (0, 1)


@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("tname,dtype", [("float64", np.float64), ("int64", np.int64),
                                         ("uint64", np.uint64)])
def test_extrema(lengths, tname, dtype):
    import torch

    rng = np.random.default_rng(len(lengths))
    L, lib = LENGTHS[lengths], oracle.load()
    for shift in SHIFTS:
        off = (shift + np.concatenate([[0], np.cumsum(L)])).astype(np.int64)
        x = _values(dtype, int(off[-1]), rng)
        n = len(L)
        if tname == "float64":
            for i in range(0, n, 5):  # zeros, a NaN at the start, all NaN, the identity
                a, b = off[i], off[i + 1]
                x[a:b] = [-0.0, 0.0, x[a:b], np.nan, -np.inf][i // 5 % 5]
                if i // 5 % 5 == 2 and b > a:
                    x[a] = np.nan
        else:
            x[off[0]:off[1]] = np.iinfo(dtype).min
            x[off[-2]:off[-1]] = np.iinfo(dtype).max
        d_off, d_x = torch.from_numpy(off).cuda(), torch.from_numpy(x).cuda()
        for which in ("max", "min"):
            ident = (-np.inf if which == "max" else np.inf) if tname == "float64" else int(
                getattr(np.iinfo(dtype), "min" if which == "max" else "max"))
            exp = np.zeros(n, dtype)
            oracle.call(lib, f"awkward_reduce_{which}_{tname}_{tname}_64", toptr=exp, fromptr=x,
                        offsets=off, outlength=n, identity=ident)
            got = _call(f"awkward_reduce_{which}_{tname}_{tname}_64", (d_x, d_off, n, ident),
                        torch.empty(n, dtype=d_x.dtype, device="cuda"))
            np.testing.assert_array_equal(got.view(np.uint8), exp.view(np.uint8))
            exp = np.zeros(n, np.int64)
            oracle.call(lib, f"awkward_reduce_arg{which}_{tname}_64", toptr=exp, fromptr=x,
                        offsets=off, starts=off[:-1].copy(), outlength=n)
            got = _call(f"awkward_reduce_arg{which}_{tname}_64", (d_x, d_off, d_off[:-1], n),
                        torch.empty(n, dtype=torch.int64, device="cuda"))
            np.testing.assert_array_equal(got, exp)


def _sums(x, off, dtype):
    import torch

    t = np.dtype(dtype).name
    return _call(f"awkward_reduce_sum_{t}_{t}_64",
                 (torch.from_numpy(x).cuda(), torch.from_numpy(off).cuda(), len(off) - 1),
                 torch.empty(len(off) - 1, dtype=torch.from_numpy(x[:0]).dtype, device="cuda"))


@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("how", ["normal", "small beside large", "window", "outside", "integers"])
def test_sums(lengths, how):
    rng = np.random.default_rng(len(lengths) + 2)
    L = np.array(LENGTHS[lengths])
    for shift in SHIFTS:
        off = (shift + np.concatenate([[0], np.cumsum(L)])).astype(np.int64)
        n = int(off[-1])
        if how == "integers":
            x = rng.integers(-2**62, 2**62, n)
            want = [int(x[a:b].sum()) for a, b in zip(off, off[1:])]
            np.testing.assert_array_equal(_sums(x, off, np.int64), want)
            continue
        x = rng.standard_normal(n)
        if how == "small beside large":  # each list within the window, its neighbours not
            scale = np.repeat(np.where(np.arange(len(L)) % 3 == 0, 1e30, 1e-30), L)
            x *= np.concatenate([np.ones(shift), scale])
        elif how == "window":
            x = np.ldexp(1 + rng.random(n), rng.integers(0, 25, n)) * rng.choice([-1, 1], n)
        elif how == "outside":
            x = np.ldexp(1 + rng.random(n), rng.integers(-500, 500, n)) * rng.choice([-1, 1], n)
        got = _sums(x, off, np.float64)
        exact = np.array([math.fsum(x[a:b]) for a, b in zip(off, off[1:])])
        if how != "outside":
            np.testing.assert_array_equal(got, exact)
        else:
            size = np.array([math.fsum(abs(x[a:b])) for a, b in zip(off, off[1:])])
            assert (abs(got - exact) <= np.maximum(L, 1) * np.finfo(np.float64).eps * size).all()


@pytest.mark.parametrize("how", ["normal", "outside"])
def test_float64_sums_do_not_depend_on_the_neighbours(how):
    """One list of 200 doubles among short lists, among lists of its own size and beside
    a giant: the same bits, in the sums' window and outside it."""
    rng = np.random.default_rng(7)
    mine = rng.standard_normal(200)
    if how == "outside":
        mine = np.ldexp(1 + rng.random(200), rng.integers(-300, 300, 200)) * rng.choice([-1, 1], 200)
    seen = set()
    for L in ([200], [3] * 40 + [200] + [3] * 40, [200] * 40, [250] * 5 + [200] + [250] * 30,
              [20_000, 200, 5], [60] * 7 + [200] + [90] * 9, [280, 200, 280]):
        off = np.concatenate([[0], np.cumsum(L)]).astype(np.int64)
        x = rng.standard_normal(int(off[-1]))
        at = [i for i, n in enumerate(L) if n == 200]
        for i in at:
            x[off[i]:off[i + 1]] = mine
        got = _sums(x, off, np.float64)
        seen.update(got[at].view(np.int64).tolist())
    assert len(seen) == 1


def test_float32_sums_beside_different_neighbours():
    """A list of floats may be added in another order beside other neighbours; its sum
    stays within the bound of any order of its additions, n - 1 of them."""
    rng = np.random.default_rng(9)
    for n in (5, 16, 17, 60, 200, 500):
        mine = (rng.standard_normal(n) + 0.5).astype(np.float32)
        part = mine.astype(np.float64)
        bound = (n - 1) * 2.0**-24 * 1.0001 * abs(part).sum()
        for L in ([n], [3] * 40 + [n] + [3] * 40, [n] * 40, [250] * 5 + [n] + [250] * 30, [20_000, n, 5]):
            off = np.concatenate([[0], np.cumsum(L)]).astype(np.int64)
            x = rng.standard_normal(int(off[-1])).astype(np.float32)
            at = [i for i, m in enumerate(L) if m == n]
            for i in at:
                x[off[i]:off[i + 1]] = mine
            got = _sums(x, off, np.float32)[at].astype(np.float64)
            assert (abs(got - math.fsum(part)) <= bound).all()
