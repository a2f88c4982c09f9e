"""Every kind of vertex step with general complex weights: the tile kernels' table against k_step's, bit for bit."""
import collections

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ("grow", "mix", "diag", "replace", "fixed", "fixed shrink", "shrink4", "shrink2")


def _case(seed):
    rng = np.random.default_rng(seed)
    n = int(rng.integers(1, 16))
    N = n + int(rng.integers(0, 22))
    A = np.triu(rng.random((N, N)) < rng.choice([0.08, 0.2, 0.5]), 1).astype(np.uint8)
    U = np.stack([np.linalg.qr(rng.standard_normal((2, 2)) + 1j * rng.standard_normal((2, 2)))[0] for _ in range(N)])
    for q in range(n):
        if rng.random() < 0.4:  # fixed by its outcome, with a phase
            U[q] = np.diag(np.exp(1j * rng.uniform(0, 2 * np.pi, 2)))
    opened = sorted(rng.choice(n, int(rng.integers(0, n)), replace=False).tolist())
    order = [int(v) for v in rng.permutation(N) if v not in opened] + opened
    return (A + A.T, U, n, order, [], opened), rng.integers(0, 2, n)


@pytest.mark.parametrize("storage", ["complex64", "complex128", "float16"])
def test_steps_round_alike(storage):
    import torch

    from dcs245_classical_sampling_b200 import _lib
    from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU, device_steps
    from dcs245_classical_sampling_b200.fused import build_fused_plan
    from dcs245_classical_sampling_b200.plan import BlockPlan
    lib, st = _lib.load(), torch.cuda.current_stream().cuda_stream
    half = storage == "float16"
    seen = collections.Counter()
    for seed in range(40):
        args, x = _case(seed)
        eng = InplaceConditionalBlockGPU(*args)
        if not len(eng.plan.steps):
            continue
        eng.alloc(np.complex64 if half else storage, mode="device", items=1, storage=storage if half else None)
        S, size = eng.nsteps, 1 << eng.plan.maxslots
        prm = eng.params.items(x)[1][0][1]
        d_prm = torch.from_numpy(prm.view(np.int64).copy()).cuda()
        eng._reset_items(1)
        for s, step in enumerate(eng.plan.steps):
            mine, before = eng.table.clone(), eng.maxbits[s].clone()
            _lib.check(lib.dcs_slice_steps_batched(eng.dcode, _lib.ptr(eng.table), size, eng.dsteps.ctypes.data, _lib.ptr(d_prm), S, S,
                                                   s, 1, _lib.ptr(eng.maxbits), _lib.ptr(eng.scale), 1, st))
            plan = build_fused_plan(BlockPlan(**{**eng.plan.__dict__, "steps": [step]}), max_dim=13 if half else 9, low=2,
                                    max_steps=1)
            one = device_steps([step])
            maxima = torch.zeros(2, dtype=torch.int64, device="cuda")
            maxima[0] = before
            scale = torch.zeros(_lib.SCALE_DTYPE.itemsize // 8, dtype=torch.int64, device="cuda")
            _lib.check(lib.dcs_tile_groups(eng.dcode, _lib.ptr(mine), size, one.ctypes.data, 1, plan.groups.ctypes.data, 1,
                                           plan.tile_steps.ctypes.data, _lib.ptr(d_prm) + s * _lib.PARAM_DTYPE.itemsize, 1,
                                           _lib.ptr(maxima), 2, _lib.ptr(scale), 1, st))
            entries = np.zeros(1, np.int64)
            for q in step.active_out:
                entries = np.concatenate([entries, entries | 1 << q])
            at = torch.from_numpy(entries).cuda()
            a, b = ((t.view(-1, 2) if half else t)[at].cpu().numpy() for t in (mine, eng.table))
            kind = KINDS[int(eng.dsteps["kind"][s])]
            assert np.array_equal(a, b), (kind, seed, s)
            if storage != "complex128":  # (FP64 maxima: of the group, by another formula's rounding)
                assert int(maxima[1]) == int(eng.maxbits[s + 1]), (kind, seed, s)
            seen[kind] += 1
    assert min(seen[k] for k in KINDS) >= 8, seen
