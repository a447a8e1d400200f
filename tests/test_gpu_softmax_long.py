"""Jagged softmax where long and short lists meet: lists of more than 192 elements in a
round of short ones, lists the whole CTA takes (more than 1024), and the numbers of
lists a CTA is given by their number and mean length.  Bounds as in
test_gpu_softmax_rounds.py."""

import numpy as np
import pytest
import torch

from test_gpu_softmax_rounds import test_softmax_lengths as check

pytestmark = pytest.mark.gpu


def _many(n, mean, longs):
    """n lists of 0..2*mean elements with `longs` spread among them."""
    L = np.random.default_rng(n).integers(0, 2 * mean + 1, n)
    L[np.linspace(0, n - 1, len(longs)).astype(int)] = longs
    return L.tolist()


CASES = {
    "one long in a round": [4] * 31 + [193] + [4] * 32,
    "long ones in many rounds": _many(45_000, 3, [193, 1024, 1025, 3000, 500, 192, 200] * 3),
    "few lists, mixed": [1, 1025, 0, 7, 192, 193, 1024, 30, 4000, 2],
    "mean above 192": [200, 193, 400, 0, 1, 250, 192, 1024] * 90,
    "16 to a CTA": [1000, 1100, 900] * 7,
    "2 to a CTA": [6000, 5000, 8192, 1],
    "one to a CTA": [30_000, 0, 3, 20_001, 17_000],
    "odd number": [600] * 45,
}


@pytest.mark.parametrize("dtype", [torch.float32, torch.float64])
@pytest.mark.parametrize("case", list(CASES))
def test_long_lists(case, dtype):
    check(CASES[case], dtype)
