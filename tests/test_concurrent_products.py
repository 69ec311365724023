"""Products issued at the same time by several threads, on one stream or several, keep their partial sums apart."""
import threading

import pytest
import torch

from cme213_final_project_b200 import ops


def test_calls_in_flight_have_scratch_of_their_own(monkeypatch):
    """Two threads are held inside the native call together: the scratch ranges that they passed must not overlap."""
    together, ranges = threading.Barrier(2, timeout=30), []

    class Lib:
        @staticmethod
        def cme_gemm(desc, backend, stream):
            g = desc._obj
            ranges.append((g.workspace, g.workspace + g.workspace_bytes))
            together.wait()
            return 0

    monkeypatch.setattr(ops, "lib", lambda: Lib)
    monkeypatch.setattr(ops, "_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "_st", lambda: 0)
    a, b = torch.zeros(64, 512), torch.zeros(512, 64)
    threads = [threading.Thread(target=ops.gemm, args=(a, b)) for _ in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(60)
    assert len(ranges) == 2
    (lo0, hi0), (lo1, hi1) = sorted(ranges)
    assert lo0 < hi0 <= lo1 < hi1


def test_a_full_device_does_without_scratch(monkeypatch):
    seen = []

    class Lib:
        @staticmethod
        def cme_gemm(desc, backend, stream):
            seen.append((desc._obj.workspace, desc._obj.workspace_bytes))
            return 0

    a, b = torch.zeros(64, 512), torch.zeros(512, 64)
    empty = torch.empty

    def full(*size, **kwargs):
        if size == (16 << 20,):
            raise torch.OutOfMemoryError("no memory left")
        return empty(*size, **kwargs)

    monkeypatch.setattr(ops, "lib", lambda: Lib)
    monkeypatch.setattr(ops, "_cuda", lambda *t: None)
    monkeypatch.setattr(ops, "_st", lambda: 0)
    monkeypatch.setattr(torch, "empty", full)
    ops.gemm(a, b)
    assert seen == [(None, 0)]


@pytest.mark.gpu
@pytest.mark.parametrize("kw", [dict(), dict(force_splits=3), dict(backend="simt")])
@pytest.mark.parametrize("M,N,K", [(2048, 512, 2048), (512, 2048, 2048), (1024, 512, 2048)])
def test_split_products_on_two_streams(M, N, K, kw):
    """Shapes whose reduction the plan splits, on two streams issued by two threads: bit for bit the serial results."""
    gen = torch.Generator(device="cuda").manual_seed(1)
    pairs = [[torch.randn(s, generator=gen, device="cuda").to(torch.bfloat16) for s in ((M, K), (K, N))] for _ in range(2)]
    want = [ops.gemm(a, b, **kw) for a, b in pairs]
    torch.cuda.synchronize()
    got = [[], []]

    def work(i):
        with torch.cuda.stream(torch.cuda.Stream()):
            got[i] = [ops.gemm(*pairs[i], **kw) for _ in range(12)]
            torch.cuda.current_stream().synchronize()

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    assert all(len(g) == 12 for g in got)
    assert all(torch.equal(x, want[i]) for i in range(2) for x in got[i])
