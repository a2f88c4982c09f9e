"""What dcs_tile_groups refuses before it touches a device."""
import numpy as np
import pytest

from dcs245_classical_sampling_b200 import _lib
from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU, device_steps
from dcs245_classical_sampling_b200.workloads import build_workload


@pytest.mark.parametrize("address,stride,nitems", [(1 << 30 | 8, 1 << 10, 1), (1 << 30, (1 << 10) + 1, 2)])
def test_tables_off_the_16_byte_words_of_a_row(address, stride, nitems):
    w = build_workload("ring16_d20_t24_k8")
    eng = InplaceConditionalBlockGPU(w["graph"], w["unitaries"], w["n"], w["order"], w["parity_operations"],
                                     w["open_vertices"])
    plan, steps, S = eng._build_tplan(), device_steps(eng.plan.steps), len(eng.plan.steps)
    assert any(int(g["low_bits"]) >= 1 for g in plan.groups)
    p = np.zeros(1, _lib.PARAM_DTYPE).ctypes.data  # (addresses that nothing reads)
    rc = _lib.load().dcs_tile_groups(_lib.C64, address, stride, steps.ctypes.data, S, plan.groups.ctypes.data, len(plan.groups),
                                     plan.tile_steps.ctypes.data, p, S, p, S + 1, p, nitems, None)
    assert rc == _lib.E_ARG
    assert b"16-byte" in _lib.load().dcs_last_error()
