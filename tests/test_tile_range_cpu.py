"""Which step weights complex64 tile groups take: no group may let an entry's square leave the FP32 range."""
import numpy as np
import pytest

from dcs245_classical_sampling_b200 import _lib
from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU, device_steps
from dcs245_classical_sampling_b200.workloads import build_workload


def _star(leaves):
    """Reference vertices that all hang on one open vertex: one growing step, then diagonal ones."""
    n, N = 1, 1 + leaves
    A = np.zeros((N, N), np.uint8)
    A[0, 1:] = A[1:, 0] = 1
    return A, np.stack([np.eye(2, dtype=complex)] * N), n, list(range(1, N)) + [0], [], [0]


def _host_engine(*args):
    eng = InplaceConditionalBlockGPU(*args)
    eng.mode, eng.use_fp64 = "device", False
    eng.dsteps = device_steps(eng.plan.steps)
    eng.free_steps = ~np.isin(eng.dsteps["kind"], (4, 5))
    eng.tplan = eng._build_tplan()
    return eng


@pytest.mark.parametrize("weight,ok", [(1.0, True), (3.0, True), (3.2, False), (4.0, False)])
def test_growth_of_a_group(weight, ok):
    eng = _host_engine(*_star(30))
    assert eng.tplan.spans[0] == (0, 24)  # entries reach weight (2 weight)^23: 2^63 from weight 3.13 on
    params = eng.params.items(np.zeros(1, np.uint8), np.array([weight, weight]))[1][0][1]
    assert eng.tile_weights_ok(params)  # every step by itself is inside the range
    assert eng.weights_ok(params) == ok
    assert eng.weights_ok(np.stack([params, params])) == ok
    small = eng.params.items(np.zeros(1, np.uint8))[1][0][1]
    rows = np.stack([small, params])
    assert eng.weights_ok(rows, any_row=True) == ok
    rows[:, 1::2] = rows[::-1, 1::2].copy()  # either row's steps anywhere
    assert eng.weights_ok(rows, any_row=True) == ok
    eng.use_fp64 = True  # FP64 squares hold the whole range
    assert eng.weights_ok(params)


@pytest.mark.parametrize("name", ["ring16_d20_t24_k8", "ring40_d45_t190_k16", "ring48_d55_t177_k17"])
def test_growth_bounds_the_steps(name):
    """The default weights stay below 2^2 per step, and the bound holds for entries at each step's worst signs."""
    w = build_workload(name)
    eng = _host_engine(w["graph"], w["unitaries"], w["n"], w["order"], w["parity_operations"], w["open_vertices"])
    params = eng.params.items(np.random.default_rng(1).integers(0, 2, w["n"]))[1][0][1]
    growth = eng.step_growth(params)
    assert growth.max() <= 4 * (1 + 1e-12) and eng.weights_ok(params)
    f0 = params["f0r"] + 1j * params["f0i"]
    f1 = params["f1r"] + 1j * params["f1i"]
    for j, kind in enumerate(eng.dsteps["kind"]):
        a, b = f0[j], f1[j]
        worst = {0: max(abs(a), abs(b)), 1: abs(a) + abs(b), 2: max(abs(a + b), abs(a - b)), 3: 2 * max(abs(a), abs(b)),
                 4: abs(b if params["y"][j] else a), 5: 2 * abs(b if params["y"][j] else a), 6: 2 * (abs(a) + abs(b)),
                 7: max(abs(a + b) + abs(a - b), 2 * abs(a + b), 2 * abs(a - b))}[int(kind)]
        assert worst <= growth[j] * (1 + 1e-12)
    assert params.dtype == _lib.PARAM_DTYPE
