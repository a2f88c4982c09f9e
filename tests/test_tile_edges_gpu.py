"""Tile groups at the edges of their range: tiles of one entry, tables whose maximum leaves the range of its
square in storage precision, step weights at the ends of what they take, single steps where they cannot run."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(graph, unitaries, n, order, opened, dtype=np.complex64, **kw):
    from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU
    eng = InplaceConditionalBlockGPU(np.asarray(graph, np.uint8), np.asarray(unitaries, complex), n, order, [], opened)
    eng.alloc(dtype, mode="device", **kw)
    return eng


def _random_case(seed, p):
    """A random graph state with Clifford-like and diagonal frames: tiles of one entry where `p` is small."""
    rng = np.random.default_rng(seed)
    n = int(rng.integers(2, 10))
    N = n + int(rng.integers(0, 10))
    A = np.triu(rng.random((N, N)) < p, 1).astype(np.uint8)
    U = [np.eye(2) if rng.random() < 0.3 else np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))[0]
         for _ in range(N)]
    opened = sorted(rng.choice(n, int(rng.integers(0, n)), replace=False).tolist())
    order = [int(v) for v in rng.permutation(N) if v not in opened] + opened
    return (A + A.T, np.stack(U).astype(complex), n, order, opened), rng.integers(0, 2, n).astype(np.uint8)


@pytest.mark.parametrize("storage", [None, "float16"])
@pytest.mark.parametrize("p", [0.0, 0.1, 0.3])
def test_small_tiles(p, storage):
    """Tables of one, two and a few entries (a group of isolated or fixed vertices has tiles of one): the bits of
    one launch per step, and in complex64 the oracle's block."""
    from oracle.block_ref import OracleEngine
    one_entry = 0
    for seed in range(12):
        (A, U, n, order, opened), x = _random_case(seed, p)
        eng = _engine(A, U, n, order, opened, storage=storage)
        one_entry += sum(int(g["tile_dim"]) == 0 for g in eng.tplan.groups)
        got = eng.block(x)[0].cpu().numpy()
        eng.tplan = None
        assert np.array_equal(got, eng.block(x)[0].cpu().numpy()), seed
        if storage:
            continue
        want, _ = OracleEngine(A, U, n, order, [], opened).block(x)
        # a step rounds weights, products and sums (5 roundings of 2^-24 of the largest entry that it can have, a
        # factor |f0| + |f1| <= sqrt 2 (data rows) or 2 (bras) per step, less the block's factor 2^(-1/2) per bra)
        largest = 2.0 ** ((len(A) - len(opened)) / 2)
        assert np.abs(got - want).max() <= 5 * 2.0 ** -24 * eng.nsteps * largest, seed
    assert one_entry or p


def _star(leaves):
    """Reference vertices on one open vertex: a growing step, then diagonal ones, which multiply an entry by f0 + f1."""
    A = np.zeros((1 + leaves, 1 + leaves), np.uint8)
    A[0, 1:] = A[1:, 0] = 1
    return A, np.stack([np.eye(2, dtype=complex)] * (1 + leaves)), 1, list(range(1, 1 + leaves)) + [0], [0]


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("leaves", [5, 24, 30, 60])
@pytest.mark.parametrize("weight", [0.125, 3.0, 4.0])
def test_weights_at_the_ends_of_the_range(weight, leaves, dtype):
    """Entries grow by up to 8 a step (2^72 in a group of 24): squares past the FP32 range, the block is right."""
    from oracle.block_ref import OracleEngine
    args, x, w = _star(leaves), np.zeros(1, np.uint8), np.array([weight, weight])
    eng = _engine(*args, dtype=dtype)
    assert all(eng.prepare([x], w)["unit_ok"]) == (dtype == np.complex128 or weight < 3.1 or leaves < 24)
    want, _ = OracleEngine(*args[:4], [], args[4]).block(x, w)
    got = eng.block(x, w)[0].cpu().numpy()
    assert np.linalg.norm(got - want) <= 4 * leaves * 2.0 ** -24 * np.linalg.norm(want)
