"""Work items built on the device (engine.device_batch) against the host bookkeeping: the same step
weights, coefficients, scatter offsets and chunks, and the same calls accepted and refused."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _workload(name):
    from dcs245_classical_sampling_b200.workloads import build_workload, choose_reference_slices, sweep_order
    if isinstance(name, str):
        return build_workload(name)
    from dcs245_classical_sampling_b200.circuits import build_ring_instance  # weights with negative zeros
    inst, opened = build_ring_instance(33, 40, 120, 947276), list(range(23, 33))
    order = sweep_order(inst, opened)
    ops = choose_reference_slices(inst["graph"], 33, order, 1, opened)
    return {"graph": inst["graph"], "unitaries": inst["unitaries"], "n": 33, "order": order,
            "parity_operations": [list(op) for op in ops], "open_vertices": opened}


def _engine(name="ring24_d24_t60_k10", items=3, **kw):
    from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU
    w = _workload(name)
    eng = InplaceConditionalBlockGPU(w["graph"], w["unitaries"], w["n"], w["order"], w["parity_operations"],
                                     w["open_vertices"])
    eng.alloc(items=items, **kw)
    return eng


@pytest.mark.parametrize("name", ["ring16_d20_t24_k8", "ring24_d24_t60_k10", "ring32_d37_t79_k14", "ring40_d45_t190_k16", 33])
@pytest.mark.parametrize("count,items", [(1, 1), (1, 8), (5, 3), (7, 4), (64, 256)])
def test_items_equal_the_hosts(name, count, items):
    from dcs245_classical_sampling_b200 import _lib
    eng = _engine(name, items)
    rng = np.random.default_rng(count)
    xs = [rng.integers(0, 2, eng.n).astype(np.uint8) for _ in range(count)]
    got = eng.prepare(xs)
    dc, eng.dc = eng.dc, None
    want = eng.prepare(xs)
    eng.dc = dc
    assert got["chunks"] == want["chunks"] and got["counts"] == want["counts"] and got["unit_ok"] == want["unit_ok"]
    assert (got["n_items"], got["nblocks"]) == (want["n_items"], want["nblocks"])
    a, b = (p["params"].cpu().numpy().view(_lib.PARAM_DTYPE) for p in (got, want))
    for f in _lib.PARAM_DTYPE.names:
        assert a[f].tobytes() == b[f].tobytes(), f  # the signs of zeros, too
    for key in ("coefs", "xors"):
        assert np.array_equal(got[key].cpu().numpy(), want[key].cpu().numpy())
    n = sum(1 + c[3] for c in want["chunks"])
    assert np.array_equal(got["begin"].cpu().numpy()[:n], want["begin"].cpu().numpy()[:n])


def test_prefix_forms():
    """Forms of a prefix that the host bookkeeping takes, and what it refuses."""
    eng = _engine()
    rng = np.random.default_rng(2)
    x = rng.integers(0, 2, eng.n).astype(np.uint8)
    want = eng.block(x)[0].cpu().numpy()
    longer = np.concatenate([x, [7, 9]])
    for form in (x.tolist(), tuple(int(v) for v in x), x.astype(bool), x.astype(np.int64), x.astype(float), longer,
                 x[::-1][::-1], np.stack([x, 1 - x], 1)[:, 0]):
        assert np.array_equal(eng.block(form)[0].cpu().numpy(), want)
    negative = x.astype(int)
    negative[x == 1] = -1  # an index from the end: the same row
    assert np.array_equal(eng.block(negative)[0].cpu().numpy(), want)
    two = x.astype(int)
    two[3] = 2
    for bad in (two, x[:-1], 5):
        with pytest.raises((IndexError, ValueError)):
            eng.block(bad)
    parts = sum(eng.block(x, part=p, parts=4)[0].cpu().numpy() for p in range(4))
    assert np.linalg.norm(parts - want) <= 1e-13 * np.linalg.norm(want)


def test_gather_engine_prefix_forms():
    from dcs245_classical_sampling_b200.gather import ConditionalBlockGPU
    from dcs245_classical_sampling_b200.workloads import build_workload
    w = build_workload("ring24_d24_t60_k10")
    eng = ConditionalBlockGPU(w["graph"], w["unitaries"], w["n"], w["order"], w["parity_operations"], w["open_vertices"])
    for items in (1, 3, 4):
        eng.alloc(np.complex128, items=items)
        x = np.random.default_rng(items).integers(0, 2, w["n"]).astype(np.uint8)
        got, meta = eng.block(x)
        dc, eng.dc = eng.dc, None
        want, meta2 = eng.block(x)
        eng.dc = dc
        assert np.array_equal(got.cpu().numpy(), want.cpu().numpy())
        assert meta["slices_evaluated"] == meta2["slices_evaluated"] == 4
