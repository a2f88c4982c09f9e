"""The block tail (Walsh-Hadamard, open-edge phase, U_open) against the same transforms in FP64 torch, for
every split of the bits that the passes use."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nblocks", [1, 3])
@pytest.mark.parametrize("k", [1, 2, 3, 4, 5, 7, 8, 9, 11, 12, 13, 14, 16, 17, 20, 21])
def test_tail(k, nblocks):
    import torch

    from dcs245_classical_sampling_b200 import _lib
    if k > 17 and nblocks > 1:
        nblocks = 2
    lib = _lib.load()
    rng = np.random.default_rng(k)
    g = torch.Generator(device="cuda")
    g.manual_seed(k)
    v = torch.view_as_complex(torch.randn((nblocks, 1 << k, 2), generator=g, dtype=torch.float64, device="cuda"))
    u = np.linalg.qr(rng.standard_normal((k, 2, 2)) + 1j * rng.standard_normal((k, 2, 2)))[0]
    edges = [(a, b) for a in range(k) for b in range(a + 1, k) if rng.random() < 0.4]
    adj = np.zeros(k, np.uint32)
    for a, b in edges:
        adj[a] |= np.uint32(1 << b)
    rows = np.ascontiguousarray(u.reshape(k, 4)).view(np.float64)
    want = v.clone()
    for j in range(k):
        w = want.view(nblocks, -1, 2, 1 << j)
        want = torch.stack([w[:, :, 0] + w[:, :, 1], w[:, :, 0] - w[:, :, 1]], 2).reshape(nblocks, -1)
    y = torch.arange(1 << k, device="cuda")
    odd = torch.zeros_like(y)
    for a, b in edges:
        odd ^= (y >> a) & (y >> b) & 1
    want = torch.where(odd.bool(), -want, want)
    for j in range(k):
        w = want.view(nblocks, -1, 2, 1 << j)
        c = [complex(z) for z in u[j].reshape(4)]
        want = torch.stack([w[:, :, 0] * c[0] + w[:, :, 1] * c[1], w[:, :, 0] * c[2] + w[:, :, 1] * c[3]],
                           2).reshape(nblocks, -1)
    _lib.check(lib.dcs_block_tail(_lib.ptr(v), k, adj.ctypes.data, rows.ctypes.data, nblocks,
                                  torch.cuda.current_stream().cuda_stream))
    # 2k stages of unitary 2x2 transforms (up to a factor), a few roundings of 2^-53 each
    assert float(torch.linalg.norm(v - want) / torch.linalg.norm(want)) <= 8 * k * 2.0 ** -53
    bad = np.zeros(1, np.float64)
    assert lib.dcs_block_tail(_lib.ptr(v), 22, adj.ctypes.data, bad.ctypes.data, 0, None) != 0
