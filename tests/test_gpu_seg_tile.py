"""The element-parallel reducer walk at its edges, against the C oracle (extrema
and integer sums bit for bit) and the exactly rounded sum of doubles
(math.fsum): lists of 0..3 elements, rounds of exactly 32 * K elements, one
element more than a round holds (288, or 544), lists beside ones that are reduced by
the whole warp, content that does not start on a 16-byte line, and doubles
whose exponents leave the fixed point's window."""

import math

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

LENGTHS = {  # (a round holds 288 elements of 8 bytes, 544 of 4)
    "tiny": [0, 1, 2, 3, 1, 0, 0, 2] * 40,
    "full9": [9] * 97,
    "full11": [11] * 64 + [12, 10] * 40,
    "span": [288, 287, 289, 1, 0, 288, 288, 700, 5, 144, 144, 145],
    "long": [4096, 3, 4097, 0, 20_000, 1, 289, 2],
    "few": [100, 100, 88, 50, 144, 140, 5, 288, 1, 200, 90, 96, 97, 95],
    "span4": [544, 543, 545, 1, 0, 544, 544, 272, 272, 273, 20, 288, 30, 27],
    "whole": [289, 4096, 0, 300, 1000, 5, 290],
    "mixed": [0, 40, 3, 120, 8, 8, 8, 200, 31, 32, 33, 64, 1, 0, 7] * 30,
}
SHIFTS = (0, 1, 3)


def _call(name, key_args, out):
    import awkward_gb300

    be = awkward_gb300.backend()
    be.by_name(name)(out, *key_args)
    be.synchronize()
    return out.cpu().numpy()


def _values(dtype, n, rng):
    if np.dtype(dtype).kind != "f":
        info = np.iinfo(dtype)
        return rng.integers(info.min, info.max, n, dtype=dtype, endpoint=True)
    x = rng.standard_normal(n).astype(dtype)
    k = rng.random(n)
    x[k < 0.2] = 0.0
    x[(k >= 0.2) & (k < 0.25)] = -0.0
    x[(k >= 0.25) & (k < 0.28)] = np.nan
    x[(k >= 0.28) & (k < 0.29)] = -np.inf
    return x


@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("tname,dtype", [("float64", np.float64), ("float32", np.float32),
                                         ("int64", np.int64), ("uint32", np.uint32)])
def test_extrema(lengths, tname, dtype):
    import torch

    rng = np.random.default_rng(len(lengths))
    L = LENGTHS[lengths]
    lib = oracle.load()
    for shift in SHIFTS:
        off = (shift + np.concatenate([[0], np.cumsum(L)])).astype(np.int64)
        x = _values(dtype, int(off[-1]), rng)
        d_off, d_x, n = torch.from_numpy(off).cuda(), torch.from_numpy(x).cuda(), len(L)
        for which in ("max", "min"):
            low = np.dtype(dtype).kind == "f"
            ident = (-np.inf if which == "max" else np.inf) if low else int(
                getattr(np.iinfo(dtype), "min" if which == "max" else "max"))
            exp = np.zeros(n, dtype)
            oracle.call(lib, f"awkward_reduce_{which}_{tname}_{tname}_64", toptr=exp, fromptr=x,
                        offsets=off, outlength=n, identity=ident)
            got = _call(f"awkward_reduce_{which}_{tname}_{tname}_64", (d_x, d_off, n, ident),
                        torch.empty(n, dtype=d_x.dtype, device="cuda"))
            np.testing.assert_array_equal(got.view(np.uint8), exp.view(np.uint8))
            exp = np.zeros(n, np.int64)
            starts = off[:-1].copy()
            oracle.call(lib, f"awkward_reduce_arg{which}_{tname}_64", toptr=exp, fromptr=x,
                        offsets=off, starts=starts, outlength=n)
            got = _call(f"awkward_reduce_arg{which}_{tname}_64", (d_x, d_off, d_off[:-1], n),
                        torch.empty(n, dtype=torch.int64, device="cuda"))
            np.testing.assert_array_equal(got, exp)


@pytest.mark.parametrize("lengths", list(LENGTHS))
@pytest.mark.parametrize("tname,dtype", [("int64", np.int64), ("float32", np.float32)])
def test_plain_sums(lengths, tname, dtype):
    import torch

    rng = np.random.default_rng(len(lengths) + 1)
    L = LENGTHS[lengths]
    for shift in SHIFTS:
        off = (shift + np.concatenate([[0], np.cumsum(L)])).astype(np.int64)
        x = (rng.standard_normal(int(off[-1])) * 100).astype(dtype)
        got = _call(f"awkward_reduce_sum_{tname}_{tname}_64",
                    (torch.from_numpy(x).cuda(), torch.from_numpy(off).cuda(), len(L)),
                    torch.empty(len(L), dtype=torch.from_numpy(x).dtype, device="cuda"))
        exact = [math.fsum(x[a:b]) for a, b in zip(off, off[1:])]
        size = [math.fsum(abs(x[a:b])) for a, b in zip(off, off[1:])]
        if np.dtype(dtype).kind == "i":
            np.testing.assert_array_equal(got, exact)
        else:  # any order of n - 1 additions
            bound = np.array(L) * np.finfo(dtype).eps * size
            assert (abs(got - exact) <= bound).all()


@pytest.mark.parametrize("lengths", ["tiny", "full9", "full11", "span", "mixed", "few", "whole"])
@pytest.mark.parametrize("how", ["normal", "zeros", "only zeros", "small beside large", "window", "outside"])
def test_exact_sums(lengths, how):
    import torch

    rng = np.random.default_rng(len(lengths) + 2)
    L = np.array(LENGTHS[lengths])
    for shift in SHIFTS:
        off = (shift + np.concatenate([[0], np.cumsum(L)])).astype(np.int64)
        n = int(off[-1])
        x = rng.standard_normal(n)
        if how == "zeros":
            x[rng.random(n) < 0.5] = 0.0
        elif how == "only zeros":
            x[:] = 0.0
        elif how == "small beside large":  # each list within the window, the round not
            x *= np.repeat(np.where(np.arange(len(L)) % 3 == 0, 1e30, 1e-30), L)[:n] if shift == 0 else 1
        elif how == "window":  # exponents over 24 binades in every list
            x = np.ldexp(1 + rng.random(n), rng.integers(0, 25, n)) * rng.choice([-1, 1], n)
        elif how == "outside":
            x = np.ldexp(1 + rng.random(n), rng.integers(-500, 500, n)) * rng.choice([-1, 1], n)
            x[rng.random(n) < 0.05] = 5e-324
        got = _call("awkward_reduce_sum_float64_float64_64",
                    (torch.from_numpy(x).cuda(), torch.from_numpy(off).cuda(), len(L)),
                    torch.empty(len(L), dtype=torch.float64, device="cuda"))
        exact = np.array([math.fsum(x[a:b]) for a, b in zip(off, off[1:])])
        if how != "outside":
            np.testing.assert_array_equal(got, exact)  # correctly rounded
        else:
            size = np.array([math.fsum(abs(x[a:b])) for a, b in zip(off, off[1:])])
            assert (abs(got - exact) <= np.maximum(L, 1) * np.finfo(np.float64).eps * size).all()


@pytest.mark.parametrize("n", [545, 767, 800, 4096, 4097, 70_000, 300_001])
@pytest.mark.parametrize("shift", SHIFTS)
def test_float32_sums_of_long_runs(n, shift):
    """A lane's chain has an eighth of its elements: at most n/256 + 1 additions, three
    inside a block of eight, five between lanes and the partials of at most n/256
    ranges, 32 at a time with five between lanes."""
    import torch

    rng = np.random.default_rng(n)
    off = np.array([0, 2, 2 + n, 2 + n, 7 + n], dtype=np.int64) + shift
    x = (rng.standard_normal(int(off[-1])) + 1).astype(np.float32)
    out = torch.empty(4, dtype=torch.float32, device="cuda")
    got = _call("awkward_reduce_sum_float32_float32_64",
                (torch.from_numpy(x).cuda(), torch.from_numpy(off).cuda(), 4), out)
    for i in range(4):
        part = x[off[i]:off[i + 1]].astype(np.float64)
        k = n / 256 + n / 8192 + 24
        assert abs(float(got[i]) - math.fsum(part)) <= 1.01 * k * 2.0**-24 * abs(part).sum()
