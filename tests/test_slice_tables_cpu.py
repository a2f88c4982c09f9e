"""The slices' tables of DeviceCircuit against the host bookkeeping, and when they are made."""
import time

import numpy as np
import pytest
import torch

from dcs245_classical_sampling_b200 import engine as E
from dcs245_classical_sampling_b200.circuits import build_ring_instance
from dcs245_classical_sampling_b200.workloads import choose_reference_slices, sweep_order


def _engine(n, depth, t, k, slices, seed=7):
    inst = build_ring_instance(n, depth, t, seed)
    opened = list(range(n - k, n))
    order = sweep_order(inst, opened)
    ops = choose_reference_slices(inst["graph"], n, order, slices, opened)
    eng = E.InplaceConditionalBlockGPU(inst["graph"], inst["unitaries"], n, order, [list(o) for o in ops], opened)
    eng.mode, eng.tplan, eng.device = "device", None, torch.device("cpu")
    return eng


@pytest.mark.parametrize("shape", [(6, 6, 9, 3, 0), (14, 15, 50, 5, 1), (24, 27, 100, 8, 3), (30, 33, 120, 10, 7)])
def test_tables_equal_the_items(shape):
    eng = _engine(*shape)
    dc = E.DeviceCircuit.of(eng)
    _, items = eng.params.items(np.zeros(shape[0], np.uint8))
    assert dc.nslices == len(items) == 1 << shape[4]
    coef = dc.coef.numpy().reshape(-1, 2)
    first = items[0][1]
    for i, (c, params, xo) in enumerate(items):
        assert (coef[i, 0], coef[i, 1]) == (c.real, c.imag)
        flipped = (params["f1r"] != first["f1r"]) | (params["f1i"] != first["f1i"])  # slice 0 flips nothing
        moves = (first["f1r"] != 0) | (first["f1i"] != 0)
        assert np.array_equal(flipped, (dc.flip.numpy()[i] != 0) & moves)
        assert int(dc.freeflip.numpy().view(np.uint64)[i]) == xo ^ items[0][2] ^ int(dc.freeflip.numpy().view(np.uint64)[0])
    assert np.array_equal(dc.flip_host.numpy(), dc.flip.numpy() | 0x80)


def test_many_slices_wait_for_a_whole_batch(monkeypatch):
    eng = _engine(30, 33, 120, 10, 11)
    made, of = [], E.DeviceCircuit.of
    monkeypatch.setattr(E.DeviceCircuit, "of", classmethod(lambda cls, e: made.append(1) or of(e)))
    eng._plan_items()
    assert not made
    t0 = time.perf_counter()
    assert eng.dc.nslices == 1 << 11 and made == [1] and eng.dc is eng.dc
    t1 = time.perf_counter()
    eng.params.items(np.zeros(30, np.uint8))
    t2 = time.perf_counter()
    assert made == [1]
    assert t1 - t0 < t2 - t1  # less than one host pass over the items
    eng.dc = None  # the host's items
    assert eng.dc is None and made == [1]
    few = _engine(14, 15, 50, 5, 2)
    few._plan_items()
    assert made == [1, 1]
