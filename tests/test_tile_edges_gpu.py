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


def _with_isolated(shape, before, factors, seed=3):
    """A ring circuit's graph with isolated reference vertices, which multiply the table by f0 + f1, in the middle of
    the order: a product of small factors, as an improbable outcome of many vertices gives one."""
    from dcs245_classical_sampling_b200.circuits import build_ring_instance
    from dcs245_classical_sampling_b200.workloads import sweep_order
    n, depth, t, k = shape
    inst = build_ring_instance(n, depth, t, seed)
    opened = list(range(n - k, n))
    order = [int(v) for v in sweep_order(inst, opened)]
    g = np.asarray(inst["graph"], np.uint8)
    N, m = len(g), len(factors)
    A = np.zeros((N + m, N + m), np.uint8)
    A[:N, :N] = g
    # the default bra takes the first row: f = (1, factor - 1), exact for the factors used here
    rows = np.array([[[1, f - 1], [0, 0]] for f in factors], complex).reshape(m, 2, 2)
    U = np.concatenate([np.asarray(inst["unitaries"], complex), rows])
    at = int(before * (len(order) - k))
    return A, U, n, order[:at] + list(range(N, N + m)) + order[at:], opened


SMALL, GROW = 2.0 ** -7, 2.0  # f0 + f1
# 2^-49 .. 2^-280: squares normal, below the normal range, zero; zero inside a group and then not; one group and more
FACTORS = {"7": [SMALL] * 7, "9": [SMALL] * 9, "10": [SMALL] * 10, "11": [SMALL] * 11, "20": [SMALL] * 20,
           "40": [SMALL] * 40, "12 and back": [SMALL] * 12 + [GROW] * 10, "10 and back": [SMALL] * 10 + [GROW] * 3}


@pytest.mark.parametrize("factors", FACTORS)
@pytest.mark.parametrize("shape,before", [((6, 6, 9, 3), 0.0), ((6, 6, 9, 3), 1.0), ((14, 15, 50, 5), 0.5), ((34, 38, 150, 11), 0.4)])
def test_small_products_are_not_lost(shape, before, factors):
    """Maxima whose squares leave the FP32 range inside a group: the block of a launch per step, not zero."""
    args = _with_isolated(shape, before, FACTORS[factors])
    x = np.random.default_rng(shape[0]).integers(0, 2, shape[0]).astype(np.uint8)
    eng = _engine(*args, items=2)
    got = eng.blocks([x, x]).cpu().numpy()
    plan, eng.tplan = eng.tplan, None
    want = eng.blocks([x, x]).cpu().numpy()
    eng.tplan = plan
    assert np.linalg.norm(want) > 0 and np.array_equal(got, want)
    one = eng.block(x)[0].cpu().numpy()
    assert np.array_equal(one, want[0])
    ref = _engine(*args, dtype=np.complex128).block(x)[0].cpu().numpy()
    assert np.linalg.norm(one - ref) <= 1e-5 * np.linalg.norm(ref)  # complex64 against complex128 tables


@pytest.mark.parametrize("count", [24, 30])
def test_small_products_in_complex128(count):
    """24 factors of 2^-22 (2^-528) leave the range of an FP64 square."""
    args = _with_isolated((14, 15, 50, 5), 0.5, [2.0 ** -22] * count)
    x = np.random.default_rng(14).integers(0, 2, 14).astype(np.uint8)
    eng = _engine(*args, dtype=np.complex128)
    got = eng.block(x)[0].cpu().numpy()
    eng.tplan = None
    want = eng.block(x)[0].cpu().numpy()
    size = np.abs(want).max()
    assert size > 0 and np.abs(got - want).max() <= 1e-12 * size


def test_zero_tables_take_no_second_run(monkeypatch):
    """A table that is zero (f0 + f1 = 0 exactly) stays a zero block, and is not taken for a lost one."""
    from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU
    args = _with_isolated((14, 15, 50, 5), 0.5, [0.0] * 3)
    again = []
    monkeypatch.setattr(InplaceConditionalBlockGPU, "single_steps", staticmethod(lambda prep: again.append(1)))
    for dtype in (np.complex64, np.complex128):
        assert not _engine(*args, dtype=dtype).block(np.zeros(14, np.uint8))[0].cpu().numpy().any()
    assert not again


def _spy(monkeypatch):
    from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU
    calls, plain = [], InplaceConditionalBlockGPU.single_steps
    monkeypatch.setattr(InplaceConditionalBlockGPU, "single_steps", staticmethod(lambda prep: calls.append(1) or plain(prep)))
    return calls


def test_checked_samples_and_enqueue_of_small_products(monkeypatch):
    import torch

    from dcs245_classical_sampling_b200.sampling import sample_checked
    args = _with_isolated((14, 15, 50, 5), 0.5, [SMALL] * 20)
    rng = np.random.default_rng(5)
    xs, us = [rng.integers(0, 2, 14).astype(np.uint8) for _ in range(5)], rng.random(5).tolist()
    eng = _engine(*args)
    calls = _spy(monkeypatch)
    recs, blocks = sample_checked(eng, xs, us, keep_host_blocks=True)
    assert len(calls) == 5
    plain = _engine(*args, dtype=np.complex64)
    plain.tplan = None
    recs2, blocks2 = sample_checked(plain, xs, us, keep_host_blocks=True)
    assert recs == recs2 and all(np.array_equal(a, b) for a, b in zip(blocks, blocks2))
    prep, out = eng.prepare([xs[0]]), torch.empty((1, 32), dtype=torch.complex128, device="cuda")
    eng.enqueue(prep, out)  # nobody looks at flags: single steps
    assert np.array_equal(out[0].cpu().numpy(), blocks[0])
    flags = torch.zeros(eng.items, dtype=torch.int64, device="cuda")
    eng.enqueue(prep, out, flags)
    assert eng.out_of_range(prep, flags.cpu().numpy())


@pytest.mark.parametrize("tables", ["owned", "graphs", "pool"])
def test_served_samples_of_small_products(tables):
    from dcs245_classical_sampling_b200.sampling import draw_many
    from dcs245_classical_sampling_b200.serve import CircuitRunner, Request, Server, TablePool
    A, U, n, order, opened = _with_isolated((14, 15, 50, 5), 0.5, [SMALL] * 20)
    w = {"graph": A, "unitaries": U, "n": n, "order": order, "parity_operations": [], "open_vertices": opened}
    pool = TablePool(1 << 20, "cuda:0") if tables == "pool" else None
    run = CircuitRunner("c", w, 11, 4, graphs=tables == "graphs", pool=pool)
    again, launch = [], run.launch

    def spy(samples, region=(), tiles=None):
        again.extend([1] if tiles is False else [])
        return launch(samples, region, tiles)
    run.launch = spy
    reqs = Server({"c": run}, pool).run([Request(i, "c", 3, 0.0) for i in range(4)], realtime=False)
    assert again and (pool is None or pool.free_bytes() == pool.nbytes)
    ref = _engine(A, U, n, order, opened, dtype=np.complex128)
    for r in reqs:
        for i in range(3):
            rec, mask = r.records[i]
            x = np.array([mask >> q & 1 for q in range(n)], np.uint8)
            want = draw_many(ref.block(x)[0], [float(rec["uniform"])])[0]
            assert rec["status"] == 0 and rec["total_exact"] > 0
            assert abs(rec["total_exact"] / want["total_exact"] - 1) <= 2e-5  # squares of amplitudes within 1e-5


@pytest.mark.parametrize("shape,tiles", [((6, 6, 9, 3), False), ((30, 33, 120, 15), True)])
@pytest.mark.parametrize("storage", [None, "float16"])
def test_overflow_in_the_last_step_is_reported(shape, tiles, storage):
    """A weight past the storage's range at the last vertex: no block with infinities in it, on one tile or many."""
    A, U, n, order, opened = _with_isolated(shape, 0.5, [])
    x = np.random.default_rng(1).integers(0, 2, n).astype(np.uint8)
    eng = _engine(A, U, n, order, opened, storage=storage)
    assert (int(eng.tplan.groups[-1]["coset_m"]) > 0) == tiles
    last = int(eng.params.keep[eng.plan.steps[-1].v])
    eng.block(x)
    U[last] *= 1e6 if storage else 1e30  # entries up to 65504, |entry|^2 up to 3.4e38
    with pytest.raises(ArithmeticError):
        _engine(A, U, n, order, opened, storage=storage).block(x)


@pytest.mark.parametrize("storage,weight", [(None, 1e36), ("float16", 1e6)])
def test_overflow_in_the_last_step_shows_in_the_block(storage, weight):
    """A caller that takes no flags does not get a finite block without the overflowed table."""
    import torch
    A, U, n, order, opened = _with_isolated((14, 15, 50, 5), 0.5, [])
    xs = np.random.default_rng(1).integers(0, 2, (3, n)).astype(np.uint8)
    eng = _engine(A, U, n, order, opened, storage=storage)
    last = int(eng.params.keep[eng.plan.steps[-1].v])
    U[last] *= weight  # |entry|^2 past FP32, entries past binary16
    eng = _engine(A, U, n, order, opened, storage=storage, items=2)
    out = torch.zeros((3, 32), dtype=torch.complex128, device="cuda")
    flags = torch.zeros(2, dtype=torch.int64, device="cuda")
    eng.enqueue(eng.prepare(list(xs)), out, flags)
    got = out.cpu().numpy()
    assert np.all(flags.cpu().numpy() & 1)
    if storage:  # infinite entries
        assert not np.isfinite(got).all(axis=1).any()
    else:  # entries whose squares are infinite: the block itself is right
        want = _engine(A, U, n, order, opened, dtype=np.complex128).blocks(list(xs)).cpu().numpy()
        assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("w", [[300.0, 200.0], [1e-3, 2e-3], [2.0 ** 20, 1.0]])
def test_weights_outside_the_range(w):
    """Bras that tile groups do not take: single steps, and the block of complex128 tables."""
    A, U, n, order, opened = _with_isolated((18, 20, 60, 7), 0.5, [])
    x = np.random.default_rng(2).integers(0, 2, n).astype(np.uint8)
    eng = _engine(A, U, n, order, opened)
    assert not any(eng.prepare([x], np.array(w))["unit_ok"])
    got = eng.block(x, np.array(w))[0].cpu().numpy()
    ref = _engine(A, U, n, order, opened, dtype=np.complex128)
    ref.tplan = None
    want = ref.block(x, np.array(w))[0].cpu().numpy()
    if w[0] == 2.0 ** 20:  # the amplitudes themselves are past the FP64 range
        assert not np.isfinite(want).any() and not np.isfinite(got).any()
    else:
        assert np.linalg.norm(got - want) <= 1e-5 * np.linalg.norm(want)


@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("w", [[0.3, 0.125], [0.2, 0.2j], [2.5, 1.5j], [1.0, 1e-3]])
def test_other_bras_inside_the_range(w, dtype):
    """Bras other than the default, towards both ends of what tile groups take: one launch per step's bits."""
    A, U, n, order, opened = _with_isolated((18, 20, 60, 7), 0.5, [])
    U[n:] = np.eye(2)  # the bras are the references' weights
    x = np.random.default_rng(2).integers(0, 2, n).astype(np.uint8)
    eng = _engine(A, U, n, order, opened, dtype=dtype)
    assert all(eng.prepare([x], np.array(w))["unit_ok"])
    got = eng.block(x, np.array(w))[0].cpu().numpy()
    eng.tplan = None
    want = eng.block(x, np.array(w))[0].cpu().numpy()
    assert np.linalg.norm(want) > 0
    if dtype == np.complex64:
        assert np.array_equal(got, want)
    assert np.linalg.norm(got - want) <= 1e-12 * np.linalg.norm(want)  # the scale factor's rounding
