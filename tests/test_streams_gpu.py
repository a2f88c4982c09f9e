"""Audits and draws that run at the same time on several streams of one GPU: no workspace is shared."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


class _Recorder:
    """The library with one entry point's calls recorded."""

    def __init__(self, lib, name, arg):
        self.lib, self.name, self.arg, self.seen = lib, name, arg, []

    def __getattr__(self, attr):
        fn = getattr(self.lib, attr)
        if attr != self.name:
            return fn

        def call(*args):
            self.seen.append(args[self.arg])
            return fn(*args)
        return call


def _pairs(count, bits):
    import torch
    g = torch.Generator(device="cuda")
    g.manual_seed(bits)
    v = torch.view_as_complex(torch.randn((count, 2, 1 << bits, 2), generator=g, dtype=torch.float64, device="cuda"))
    torch.cuda.synchronize()
    return v


def _in_streams(run, count):
    """run(i) on a stream and a thread of its own, all at once, twenty times each; the last results."""
    import torch
    out, errors = [None] * count, []
    gate = threading.Barrier(count)

    def work(i):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                gate.wait()
                for _ in range(20):
                    got = run(i)
                    assert out[i] is None or repr(out[i]) == repr(got)
                    out[i] = got
        except Exception as e:  # a thread's failure fails the test
            errors.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    return out


def test_audits_on_streams(monkeypatch):
    import torch

    from dcs245_classical_sampling_b200 import _lib, audit
    rec = _Recorder(_lib.load(), "dcs_overlap", 4)
    monkeypatch.setattr(audit._lib, "load", lambda: rec)
    pairs = _pairs(4, 17)
    want = [audit.overlap_sums(p[0], p[1]) for p in pairs]
    with torch.cuda.stream(torch.cuda.Stream()):
        audit.overlap_sums(pairs[0][0], pairs[0][1])
    assert abs(rec.seen[-1] - rec.seen[0]) >= 16384
    assert repr(_in_streams(lambda i: audit.overlap_sums(pairs[i][0], pairs[i][1]), 4)) == repr(want)


@pytest.mark.parametrize("exact_cdf", [False, True])
def test_draws_on_streams(monkeypatch, exact_cdf):
    import torch

    from dcs245_classical_sampling_b200 import _lib, sampling
    rec = _Recorder(_lib.load(), "dcs_draw_ex", 5)
    monkeypatch.setattr(sampling._lib, "load", lambda: rec)
    blocks = [p.contiguous() for p in _pairs(4, 14)]

    def draw(i):
        return sampling.draw_many(blocks[i], [0.3, 0.7], exact_cdf=exact_cdf).tolist()

    want = [draw(i) for i in range(4)]
    with torch.cuda.stream(torch.cuda.Stream()):
        draw(0)
    assert abs(rec.seen[-1] - rec.seen[0]) >= rec.lib.dcs_draw_scratch_bytes(14, 2)
    assert repr(_in_streams(draw, 4)) == repr(want)


def test_kept_workspaces_are_bounded():
    import torch

    from dcs245_classical_sampling_b200.sampling import Workspaces
    ws, dev = Workspaces(), torch.device("cuda", 0)
    first = ws.get(dev, 1, 1 << 20)
    assert ws.get(dev, 1, 1 << 10) is first and ws.get(dev, 2, 1 << 10) is not first
    big = ws.get(dev, 1, ws.KEEP_BYTES + 1)
    assert big.numel() > ws.KEEP_BYTES and ws.get(dev, 1, 1 << 20) is first
    for stream in range(3, 20):
        ws.get(dev, stream, 1 << 10)
    assert len(ws.buf) <= ws.KEEP
    seen = []
    t = threading.Thread(target=lambda: seen.append(ws.get(dev, 19, 1 << 10)))
    t.start()
    t.join()
    assert seen[0] is not ws.get(dev, 19, 1 << 10)
