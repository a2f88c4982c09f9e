"""Host rules of device mode's tile groups: which step weights they take, and the groups they make."""
import numpy as np
import pytest

from dcs245_classical_sampling_b200 import _lib
from dcs245_classical_sampling_b200.engine import TILE_STEPS, InplaceConditionalBlockGPU, tile_dim
from dcs245_classical_sampling_b200.workloads import build_workload


@pytest.mark.parametrize("name", ["ring16_d20_t24_k8", "ring24_d24_t60_k10", "ring32_d37_t79_k14", "ring40_d45_t190_k16"])
def test_groups_and_weights(name):
    w = build_workload(name)
    eng = InplaceConditionalBlockGPU(w["graph"], w["unitaries"], w["n"], w["order"], w["parity_operations"],
                                     w["open_vertices"])
    fp = eng._build_tplan()
    assert sum(int(g["count"]) for g in fp.groups) == len(eng.plan.steps)
    assert all(1 <= int(g["count"]) <= TILE_STEPS for g in fp.groups)
    assert max(fp.dims) <= max(tile_dim(eng.plan.maxslots), 4) <= 12
    from dcs245_classical_sampling_b200.engine import device_steps
    eng.dsteps = device_steps(eng.plan.steps)
    eng.free_steps = ~np.isin(eng.dsteps["kind"], (4, 5))
    rng = np.random.default_rng(0)
    for _ in range(8):
        for _, params, _ in eng.params.items(rng.integers(0, 2, w["n"]))[1]:
            assert eng.tile_weights_ok(params)
    fixed, free = np.flatnonzero(~eng.free_steps), np.flatnonzero(eng.free_steps)
    for j in free[:3]:
        for f0, f1, ok in ((0.0, 0.125, True), (4.0, 0.0, True), (0.0, 0.1, False), (4.1, 1.0, False),
                           (np.nan, 1.0, False), (np.inf, 1.0, False), (0.0, 0.0, False)):
            p = params.copy()
            p["f0r"][j], p["f0i"][j], p["f1r"][j], p["f1i"][j] = f0, 0.0, f1, 0.0
            assert eng.tile_weights_ok(p) == ok, (f0, f1)
    for j in fixed[:3]:  # only the weight that the step's value selects counts
        for y, f0, f1, ok in ((0, 1.0, 1e-30, True), (1, 1e-30, 1.0, True), (0, 1e-30, 1.0, False), (1, 1.0, 1e-30, False)):
            p = params.copy()
            p["y"][j], p["f0r"][j], p["f0i"][j], p["f1r"][j], p["f1i"][j] = y, f0, 0.0, f1, 0.0
            assert eng.tile_weights_ok(p) == ok
    assert params.dtype == _lib.PARAM_DTYPE
