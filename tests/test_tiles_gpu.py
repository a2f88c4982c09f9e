"""Tile groups (csrc/tiles.cu) against one launch per step on the same prefixes: the same bits in
complex64, the same but for the rounding of the scale factor in complex128."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# qubits, depth, T gates, open bits, parity slices: tables of 2 to 2^19 entries, one tile to many
CIRCUITS = [(3, 3, 2, 1, 0), (6, 6, 9, 3, 0), (10, 12, 30, 4, 1), (14, 15, 50, 5, 0), (18, 20, 60, 7, 1),
            (24, 27, 100, 8, 2), (30, 33, 120, 10, 0), (34, 38, 150, 11, 0)]


def _engine(shape, dtype, items, **kw):
    from dcs245_classical_sampling_b200.circuits import build_ring_instance
    from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU
    from dcs245_classical_sampling_b200.workloads import choose_reference_slices, sweep_order
    n, depth, t, k, slices = shape
    inst = build_ring_instance(n, depth, t, 7)
    opened = list(range(n - k, n))
    order = sweep_order(inst, opened)
    ops = choose_reference_slices(inst["graph"], n, order, slices, opened)
    eng = InplaceConditionalBlockGPU(inst["graph"], inst["unitaries"], n, order, [list(o) for o in ops], opened)
    eng.alloc(dtype, mode="device", items=items, **kw)
    return eng


def _both(eng, xs, w=None):
    plan = eng.tplan
    assert plan is not None
    got = eng.blocks(xs, w).cpu().numpy()
    eng.tplan = None
    want = eng.blocks(xs, w).cpu().numpy()
    eng.tplan = plan
    return got, want


@pytest.mark.parametrize("items", [1, 5])
@pytest.mark.parametrize("shape", CIRCUITS, ids=lambda s: f"{s[0]}q")
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
def test_tile_groups_equal_steps(shape, dtype, items):
    eng = _engine(shape, dtype, items)
    rng = np.random.default_rng(shape[0])
    xs = [rng.integers(0, 2, shape[0]).astype(np.uint8) for _ in range(4)]
    plans = [eng.tplan] + [eng._build_tplan(dim, low) for dim, low in ((4, 1), (7, 0), (9, 2), (12, 5))]
    for plan in plans:
        eng.tplan = plan
        got, want = _both(eng, xs)
        if dtype == np.complex64:
            assert np.array_equal(got, want)
        for g, v in zip(got, want):
            # complex128: up to 40 steps' e ln 2 (below 100 together) summed per group, 100 ulps of exp's
            # argument; products and sums are the same, so a block that cancels to rounding noise is, too
            assert np.linalg.norm(g - v) <= 1e-12 * np.linalg.norm(v)


@pytest.mark.parametrize("items", [1, 5])
@pytest.mark.parametrize("shape", CIRCUITS, ids=lambda s: f"{s[0]}q")
def test_half_tiles_equal_steps(shape, items):
    """Binary16 tables: stretches of steps on one tile in one launch, the same bits (every step rounds)."""
    eng = _engine(shape, np.complex64, items, storage="float16")
    rng = np.random.default_rng(shape[0])
    xs = [rng.integers(0, 2, shape[0]).astype(np.uint8) for _ in range(4)]
    for plan in (eng.tplan, eng._build_tplan(6, 2), eng._build_tplan(11, 1)):
        assert plan.spans[-1][0] + plan.spans[-1][1] == eng.nsteps
        eng.tplan = plan
        got, want = _both(eng, xs)
        assert np.array_equal(got, want)


def test_weights_outside_the_range_take_single_steps():
    eng = _engine(CIRCUITS[4], np.complex64, 2)
    x = np.zeros(18, np.uint8)
    assert all(eng.prepare([x])["unit_ok"])
    for w in (np.array([1e-3, 2e-3]), np.array([1e6, 1.0]), np.array([1.0, np.nan])):
        assert not any(eng.prepare([x], w)["unit_ok"])
    got, want = _both(eng, [x], np.array([300.0, 200.0]))
    assert np.array_equal(got, want)
