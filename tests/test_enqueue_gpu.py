"""What enqueue takes for its blocks and flags."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _engine(items, **kw):
    from dcs245_classical_sampling_b200.engine import InplaceConditionalBlockGPU
    from dcs245_classical_sampling_b200.workloads import build_workload
    w = build_workload("ring24_d24_t60_k10")
    eng = InplaceConditionalBlockGPU(w["graph"], w["unitaries"], w["n"], w["order"], w["parity_operations"],
                                     w["open_vertices"])
    eng.alloc(np.complex64, items=items, **kw)
    xs = [np.random.default_rng(i).integers(0, 2, w["n"]).astype(np.uint8) for i in range(3)]
    return eng, xs


def _overflowing(eng, x):
    """A batch whose last step's weights make every table nonfinite."""
    import torch

    from dcs245_classical_sampling_b200 import _lib
    prep = eng.single_steps(eng.prepare([x]))
    p = prep["params"].cpu().numpy().view(_lib.PARAM_DTYPE).reshape(-1, eng.nsteps)
    for f in ("f0r", "f0i", "f1r", "f1i"):
        p[f][:, -1] = 1e38
    prep["params"].copy_(torch.from_numpy(p.reshape(-1).view(np.int64)))
    return prep


@pytest.mark.parametrize("items", [4, 3])
def test_forms_of_the_flags(items):
    import torch
    eng, xs = _engine(items)
    out = torch.zeros((1, 1 << eng.k), dtype=torch.complex128, device="cuda")
    want = torch.zeros(items, dtype=torch.int64, device="cuda")
    prep = _overflowing(eng, xs[0])
    eng.enqueue(prep, out, want)
    assert (want & 1).all() and int(want.max()) < 32
    forms = [torch.zeros(items, dtype=d, device="cuda") for d in (torch.int32, torch.int16, torch.uint8)]
    forms += [torch.zeros((items, 2), dtype=torch.int64, device="cuda")[:, 1], torch.zeros(2 * items, dtype=torch.int64,
                                                                                           device="cuda")[::2],
              torch.zeros(items + 3, dtype=torch.int64, device="cuda")]
    for flags in forms:
        eng.enqueue(prep, out, flags)
        assert torch.equal(flags[:items].long(), want), flags.dtype
    with pytest.raises(Exception):
        eng.enqueue(prep, out, torch.zeros(items - 2, dtype=torch.int64, device="cuda"))


@pytest.mark.parametrize("items", [4, 1])
def test_forms_of_the_blocks(items):
    import torch
    eng, xs = _engine(items)
    n = 1 << eng.k
    want = eng.block(xs[0])[0].cpu().numpy()
    prep = eng.prepare([xs[0]])
    roomy = torch.full((3, n), 7.0, dtype=torch.complex128, device="cuda")
    eng.enqueue(prep, roomy, eng._flags_tensor())  # the rows that the batch does not have are zero
    assert np.array_equal(roomy[0].cpu().numpy(), want) and not roomy[1:].cpu().numpy().any()
    flat = torch.full((1, 2 * n), 7.0, dtype=torch.float64, device="cuda")
    eng.enqueue(prep, flat, eng._flags_tensor())
    assert np.array_equal(torch.view_as_complex(flat.view(n, 2)).cpu().numpy(), want)
    strided = torch.zeros((1, 2 * n), dtype=torch.complex128, device="cuda")
    with pytest.raises(RuntimeError):
        eng.enqueue(prep, strided[:, ::2], eng._flags_tensor())
    torch.cuda.synchronize()
    assert not strided.cpu().numpy().any()
