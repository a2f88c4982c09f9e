"""Stretches of gather steps in shared memory on maxima at the lower end of the FP64 range."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("exponent", [-505, -518, -521, -522, -530, -534])
def test_least_maxima(exponent):
    """A step whose weight takes |entry|^2 to 2^-1010 .. 2^-1068: as one launch per step, not a zero table."""
    from dcs245_classical_sampling_b200.gather import ConditionalBlockGPU
    leaves = 6  # reference vertices on one open vertex
    A = np.zeros((1 + leaves, 1 + leaves), np.uint8)
    A[0, 1:] = A[1:, 0] = 1
    U = np.stack([np.eye(2, dtype=complex)] * (1 + leaves))
    order = list(range(1, 1 + leaves)) + [0]
    w = {q: np.array([1.0, 0.5]) for q in range(1, 1 + leaves)}
    plain = ConditionalBlockGPU(A, U, 1, order, [], [0])
    plain.alloc(np.complex128)
    want = plain.block(np.zeros(1, np.uint8), w)[0].cpu().numpy()
    w[3] = w[3] * 2.0 ** exponent  # a power of two: every other number of the contraction is the same
    got = plain.block(np.zeros(1, np.uint8), w)[0].cpu().numpy()
    # entries are normal numbers all along; the factor e^logscale of the block is rounded (logscale near -370)
    assert np.linalg.norm(want) > 0
    assert np.abs(got * 2.0 ** -exponent - want).max() <= 400 * 2.0 ** -52 * np.abs(want).max()
