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


def _reference(w, u):
    """numpy's CDF and index, and whether the reference's independent check of the interval accepts u."""
    sums = np.cumsum(w)
    cdf = sums / sums[-1]
    cdf[-1] = 1.0
    i = int(np.searchsorted(cdf, u, side="right"))
    total = math.fsum(w)
    ok = w[i] > 0 and math.fsum(w[:i]) / total <= u < math.fsum(w[: i + 1]) / total
    return sums, cdf, i, ok


@pytest.mark.parametrize("k", [6, 8, 13])
@pytest.mark.parametrize("low,high", [(-537, -533), (-537, -500), (-520, -510), (-512, -505), (-456, -450), (-537, 0)])
def test_sequential_cdf_of_tiny_weights(low, high, k):
    """numpy's sequential CDF bit for bit where the sum is subnormal, leaves the subnormal numbers, or stays tiny."""
    import torch

    from dcs245_classical_sampling_b200.sampling import draw_many
    rng = np.random.default_rng([k, -low])
    a = rng.standard_normal(1 << k) * np.exp2(np.sort(rng.uniform(low, high, 1 << k)))
    a[: len(a) // 8] = 0.0
    w = a * a
    for u in (0.0, 0.25, 0.9):
        sums, cdf, i, ok = _reference(w, u)
        r = draw_many(torch.from_numpy(a + 0j).cuda(), [u], exact_cdf=True)[0]
        assert float(r["total_cdf"]) == float(sums[-1]) and float(r["total_exact"]) == math.fsum(w)
        assert (r["status"] == 0) == ok
        if ok:
            assert (int(r["index"]), float(r["cdf_upper"]), float(r["selected_weight"])) == (i, float(cdf[i]), float(w[i]))
            assert float(r["cdf_lower"]) == (float(cdf[i - 1]) if i else 0.0)


def test_tiny_weights_cost_no_walk():
    """A block far below 1 takes the time of any other, not an addition after the other for every entry."""
    import torch

    from dcs245_classical_sampling_b200.sampling import draw_many
    a = np.random.default_rng(3).random(1 << 18)
    times = []
    for scale in (1.0, 1e-140, 1e-158):  # weights near 1, near 2^-930, subnormal
        v = torch.from_numpy(a * scale + 0j).cuda()
        for _ in range(3):
            t0, t1 = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            t0.record()
            draw_many(v, [0.4], exact_cdf=True)
            t1.record()
            torch.cuda.synchronize()
        times.append(t0.elapsed_time(t1))
    assert max(times) < 8 * times[0] + 1.0  # (milliseconds; one by one: 33 against 0.1)


@pytest.mark.parametrize("k", [4, 11, 14, 17])
def test_ties_are_decided_as_the_reference_does(k):
    """u on an edge of numpy's CDF, and one place beside it: numpy's index where the reference's compensated check
    accepts it, an error where it does not, by a sequential pass that makes its maps itself."""
    import torch

    from dcs245_classical_sampling_b200.sampling import draw_many
    rng = np.random.default_rng(k)
    v = rng.standard_normal(1 << k) + 1j * rng.standard_normal(1 << k)
    w = v.real * v.real + v.imag * v.imag
    cdf = np.cumsum(w) / np.cumsum(w)[-1]
    accepted = 0
    for at in (0.1, 0.4, 0.7):
        edge = cdf[int(at * len(v))]
        for u in (edge, np.nextafter(edge, 0), np.nextafter(edge, 1)):
            sums, want, i, ok = _reference(w, u)
            r = draw_many(torch.from_numpy(v).cuda(), [u])[0]
            assert r["tie"] and float(r["total_cdf"]) == float(sums[-1])
            assert (r["status"] == 0) == ok
            if ok:
                assert (int(r["index"]), float(r["cdf_upper"])) == (i, float(want[i]))
            accepted += ok
    assert accepted
