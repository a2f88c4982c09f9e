"""The device draw's sequential CDF (integer maps of stretches of additions) against numpy's cumsum,
bit for bit: block sizes around the sub-chunk (128) and chunk (2048) edges, weights that tie (sums that
end in exactly half an ulp), zeros, and weights that cross many binades."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _weights(kind, n, rng):
    """Amplitudes whose weights are exact squares where ties are wanted."""
    if kind == "gauss":
        return rng.standard_normal(n) + 1j * rng.standard_normal(n)
    if kind == "equal":
        return np.full(n, 2.0 ** -8) + 0j
    if kind == "ties":  # odd multiples of 2^-52 .. 2^-50 below sums near 1, and a few large ones
        a = rng.choice([1.0, 3.0, 5.0, 7.0], n) * 2.0 ** -26
        a[0] = 1.0
        a[n // 3] = 1.5
        return a + 0j
    if kind == "zeros":  # zero chunks at the start, the middle and the end
        a = rng.standard_normal(n) + 1j * rng.standard_normal(n)
        a[: n // 3] = 0
        a[n // 2: 3 * n // 4] = 0
        a[-max(1, n // 8):] = 0
        a[n // 3] = 1.0
        return a
    return np.exp(np.linspace(-180.0, 0.0, n)) * (rng.standard_normal(n) + 1j)  # grows through 500 binades


@pytest.mark.parametrize("k", [0, 1, 5, 6, 7, 8, 10, 11, 12, 13, 16, 20])
@pytest.mark.parametrize("kind", ["gauss", "equal", "ties", "zeros", "growing"])
def test_sequential_cdf_is_numpys(kind, k):
    import torch

    from dcs245_classical_sampling_b200.sampling import draw_many
    n = 1 << k
    rng = np.random.default_rng([k, len(kind)])
    blocks = np.stack([_weights(kind, n, rng) for _ in range(3)]).astype(np.complex128)
    us = np.array([0.0, 0.61803398875, 1 - 2.0 ** -53])
    rec = draw_many(torch.from_numpy(blocks).cuda(), us, exact_cdf=True)
    for v, u, r in zip(blocks, us, rec):
        w = v.real * v.real + v.imag * v.imag
        sums = np.cumsum(w)
        cdf = sums / sums[-1]
        cdf[-1] = 1.0
        i = int(np.searchsorted(cdf, u, side="right"))
        if w[i] > 0 and r["status"] == 0:
            assert (int(r["index"]), float(r["cdf_upper"])) == (i, float(cdf[i]))
            assert float(r["cdf_lower"]) == (float(cdf[i - 1]) if i else 0.0)
            assert float(r["selected_weight"]) == float(w[i])
        else:  # the reference's independent check rejects what the compensated interval does not confirm
            total = math.fsum(w)
            low = math.fsum(w[:i]) / total
            assert r["status"] != 0 and not (w[i] > 0 and low <= u < math.fsum(w[: i + 1]) / total)
        assert float(r["total_cdf"]) == float(sums[-1])
        assert float(r["total_exact"]) == math.fsum(w)


@pytest.mark.parametrize("k", [4, 11, 14])
def test_tie_takes_the_sequential_cdf(k):
    """u on an edge of numpy's CDF cannot be certified: the exact pass decides without being asked for."""
    import torch

    from dcs245_classical_sampling_b200.sampling import draw_many
    rng = np.random.default_rng(k)
    v = rng.standard_normal(1 << k) + 1j * rng.standard_normal(1 << k)
    sums = np.cumsum(v.real * v.real + v.imag * v.imag)
    cdf = sums / sums[-1]
    i = int(0.7 * len(v))
    for u in (cdf[i], np.nextafter(cdf[i], 0), np.nextafter(cdf[i], 1)):
        r = draw_many(torch.from_numpy(v).cuda(), [u])[0]
        assert r["tie"] and float(r["total_cdf"]) == float(sums[-1])
        assert int(r["index"]) == int(np.searchsorted(cdf, u, side="right")) or r["status"] != 0
