"""Engines with many slices: a part of a block needs no tables of all of them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["inplace", "half", "gather"])
def test_parts_and_whole_blocks(kind, monkeypatch):
    from dcs245_classical_sampling_b200 import engine as E
    from dcs245_classical_sampling_b200.circuits import build_ring_instance
    from dcs245_classical_sampling_b200.gather import ConditionalBlockGPU
    from dcs245_classical_sampling_b200.workloads import choose_reference_slices, sweep_order
    n, opened = 24, list(range(16, 24))
    inst = build_ring_instance(n, 27, 100, 7)
    order = sweep_order(inst, opened)
    ops = choose_reference_slices(inst["graph"], n, order, 6, opened)
    made, of = [], E.DeviceCircuit.of
    monkeypatch.setattr(E.DeviceCircuit, "of", classmethod(lambda cls, e: made.append(1) or of(e)))
    args = (inst["graph"], inst["unitaries"], n, order, [list(o) for o in ops], opened)
    cls = {"inplace": E.InplaceConditionalBlockGPU, "half": E.HalfConditionalBlockGPU, "gather": ConditionalBlockGPU}[kind]
    eng = cls(*args)
    eng.alloc()
    x = np.random.default_rng(0).integers(0, 2, n).astype(np.uint8)
    parts = [eng.block(x, part=p, parts=8) for p in range(8)]
    assert not made and [m["slices_evaluated"] for _, m in parts] == [8] * 8
    total = sum(v.cpu().numpy() for v, _ in parts)
    whole = eng.block(x)[0].cpu().numpy()
    assert made == [1]
    assert np.linalg.norm(whole - total) <= 1e-13 * np.linalg.norm(whole)  # another order of the slices' sums
