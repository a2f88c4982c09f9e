"""Draws from blocks whose weights are at the ends of the FP64 range, and ties decided by the sequential CDF."""
import math
from fractions import Fraction

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [1, 4, 9, 12])
@pytest.mark.parametrize("exponent", [-534, -520, -514, -480, 0, 480, 500])
def test_grid_distance_at_the_ends_of_the_range(exponent, k):
    """The 53-bit distance and the sum of squares do not depend on a power of two in the amplitudes (whole numbers
    below 10, so that every weight is exact), down to totals whose reciprocal is infinite."""
    import torch

    from dcs245_classical_sampling_b200.sampling import draw_many
    n = 1 << k
    a = np.random.default_rng(k).integers(1, 10, n)
    w = [int(v) ** 2 for v in a]
    total = sum(w)
    tv, run, prev = [], 0, 0
    for i, wi in enumerate(w):
        run += wi
        end = math.ceil(float(Fraction(run, total)) * 2.0 ** 53) if i < n - 1 else 2 ** 53
        tv.append(abs(Fraction(end - prev, 2 ** 53) - Fraction(wi, total)))
        prev = end
    want = float(sum(tv) / 2)
    r = draw_many(torch.from_numpy(a * 2.0 ** exponent + 0j).cuda(), [0.4])[0]
    assert r["status"] == 0 and float(r["total_exact"]) == total * 2.0 ** (2 * exponent)
    # one unit of the grid per edge whose quotient rounds the other way, and the roundings of the n differences
    assert abs(float(r["tv53"]) - want) <= n * 2.0 ** -53 + 4 * 2.0 ** -53
    assert abs(float(r["weight_l2"]) - float(sum(Fraction(v, total) ** 2 for v in w))) <= 4 * 2.0 ** -53
    run, i = 0, 0
    while Fraction(run + w[i], total) <= Fraction(0.4):
        run, i = run + w[i], i + 1
    assert int(r["index"]) == i
