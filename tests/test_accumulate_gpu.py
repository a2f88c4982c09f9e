"""The two accumulation entry points against the sum that their header states, with a scale record whose table_exp
a caller of the step kernels never set."""
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", ["c64", "c128", "h16"])
@pytest.mark.parametrize("tr,k,items", [(0, 0, [1]), (3, 3, [2, 1]), (4, 6, [0, 3]), (9, 11, [70])])
def test_accumulate(tr, k, items, dtype):
    import torch

    from dcs245_classical_sampling_b200 import _lib
    lib = _lib.load()
    rng = np.random.default_rng([tr, k])
    n, stride, mstride = sum(items), 1 << (tr + 1), 3
    dcode = {"c64": _lib.C64, "c128": _lib.C128, "h16": _lib.H16}[dtype]
    table = rng.standard_normal((n, stride)) + 1j * rng.standard_normal((n, stride))
    if dtype == "h16":
        half = np.stack([table.real, table.imag], -1).astype(np.float16)
        table, dev = half[..., 0].astype(float) + 1j * half[..., 1].astype(float), torch.from_numpy(half).cuda()
    else:
        table = table.astype(np.complex64 if dtype == "c64" else np.complex128)
        dev = torch.from_numpy(table).cuda()
    slots = np.array([0 | 1 << 8 | tr << 16], np.uint32)  # the index sits in slots 1 .. tr
    while True:  # independent vectors
        basis = rng.integers(1, 1 << max(k, 1), tr).astype(np.uint64)
        span = {0}
        for b in basis:
            span |= {s ^ int(b) for s in span}
        if len(span) == 1 << tr:
            break
    xors = rng.integers(0, 1 << k, n).astype(np.uint64)
    coefs = rng.standard_normal((n, 2))
    scale = np.zeros(n, _lib.SCALE_DTYPE)
    scale["logscale"], scale["phase"] = rng.standard_normal(n), rng.standard_normal(n)
    scale["table_exp"] = 7
    word = (np.array(1.5, np.float32).view(np.uint32) if dtype == "c64" else np.array(1.5).view(np.uint64))
    final = np.full((n, mstride), int(word), np.int64)
    if n > 1:
        scale["flags"][0], final[1, 0] = 2, 0  # a zero table on the way, and after the last step
    begin = np.concatenate([[0], np.cumsum(items)]).astype(np.int32)
    shift = 0.25
    want = np.zeros((len(items), 1 << k), np.complex128)
    for b in range(len(items)):
        for it in range(begin[b], begin[b + 1]):
            if scale["flags"][it] & 3 or not final[it, 0]:
                continue
            c = (coefs[it, 0] + 1j * coefs[it, 1]) * math.exp(scale["logscale"][it] - shift) * np.exp(1j * scale["phase"][it])
            for i in range(1 << tr):
                s = 0
                for j in range(tr):
                    s ^= int(basis[j]) if i >> j & 1 else 0
                want[b, s ^ int(xors[it])] += table[it, i << 1] * c
    d = lambda a: torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).cuda()
    args = [d(xors), d(coefs), d(begin), d(scale), d(final)]
    st = torch.cuda.current_stream().cuda_stream

    def call(ex, flags=0):
        out = torch.full((len(items), 1 << k), 3.0 if flags else 0.0, dtype=torch.complex128, device="cuda")
        head = (dcode, dev.data_ptr(), stride, tr, slots.ctypes.data, 1 if tr else 0, basis.ctypes.data, *[a.data_ptr() for a in args[:3]],
                len(items), shift, args[3].data_ptr(), args[4].data_ptr(), mstride, out.data_ptr(), k, n)
        _lib.check(lib.dcs_accumulate_ex(*head, flags, st) if ex else lib.dcs_accumulate_batched(*head, st))
        return out.cpu().numpy()

    # per term: a product of three rounded factors and a sum, a few 2^-53 of the terms' sizes
    bound = 64 * 2.0 ** -53 * max(1.0, np.abs(want).max()) * max(items)
    plain = call(False)
    assert np.abs(plain - want).max() <= bound
    for flags in (0, _lib.ACCUMULATE_FRESH):
        assert np.array_equal(call(True, flags), plain * 2.0 ** -7)
