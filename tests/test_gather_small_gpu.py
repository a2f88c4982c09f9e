"""Stretches of gather steps in shared memory (one launch) against one launch per step: the same tables,
maxima and scale for plans below, at and above the size that fits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("items", [1, 3])
@pytest.mark.parametrize("dtype", [np.complex64, np.complex128])
@pytest.mark.parametrize("n,depth,t,k,slices", [(3, 3, 2, 1, 0), (8, 9, 20, 3, 0), (16, 20, 60, 6, 1), (22, 25, 80, 8, 0),
                                                (28, 32, 90, 9, 1), (34, 38, 150, 11, 0)])
def test_stretches_equal_single_steps(n, depth, t, k, slices, dtype, items):
    import torch

    from dcs245_classical_sampling_b200 import _lib
    from dcs245_classical_sampling_b200.circuits import build_ring_instance
    from dcs245_classical_sampling_b200.gather import ConditionalBlockGPU
    from dcs245_classical_sampling_b200.workloads import choose_reference_slices, sweep_order
    inst = build_ring_instance(n, depth, t, 5)
    opened = list(range(n - k, n))
    order = sweep_order(inst, opened)
    ops = choose_reference_slices(inst["graph"], n, order, slices, opened)
    eng = ConditionalBlockGPU(inst["graph"], inst["unitaries"], n, order, [list(o) for o in ops], opened)
    eng.alloc(dtype, items=items)
    x = np.random.default_rng(n).integers(0, 2, n).astype(np.uint8)
    count, chunks, keep = eng._prepare(x, None, 0, 1)
    S, lib, st = len(eng.steps), eng.lib, eng._stream()
    cn, d_params = chunks[0][:2]

    def run(spans):
        for t_ in eng.tab:
            t_.zero_()
        _lib.check(lib.dcs_begin_items(eng.dcode, _lib.ptr(eng.tab[0]), eng.stride, _lib.ptr(eng.maxbits), eng.nm,
                                       _lib.ptr(eng.scale), cn, st))
        for s, c in spans:
            a, b = (eng.tab[s & 1], eng.tab[(s & 1) ^ 1])
            _lib.check(lib.dcs_gather_steps(eng.dcode, _lib.ptr(a), _lib.ptr(b), eng.stride, eng.dsteps.ctypes.data,
                                            _lib.ptr(eng.words), d_params, S, s, c, _lib.ptr(eng.maxbits), eng.nm,
                                            _lib.ptr(eng.scale), cn, st))
        torch.cuda.synchronize()
        r = eng.steps[-1].r_out
        out = eng.tab[S & 1].view(eng.items, eng.stride)[:cn, :1 << r].cpu().numpy()
        return out, eng.scale.cpu().numpy().copy(), eng.maxbits.cpu().numpy().copy()

    want = run([(s, 1) for s in range(S)])  # a stretch of one step is a launch of k_gather
    for spans in ([(0, S)], [(0, S // 2), (S // 2, S - S // 2)], [(0, 1), (1, S - 1)]):
        got = run(spans)
        assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
        a, b = (m.view(np.uint64) for m in (got[2], want[2]))
        high = np.uint64(32 if dtype == np.complex128 else 0)  # complex128 stretches keep a maximum's high half
        assert np.array_equal(a >> high, b >> high)
