"""Small decodes and line calls by several callers at once: results, capture beside running calls, and
the time of many streams together."""
import ctypes as C
import threading
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 4, 20, 2, 75, 9, 1, 33, 300, 17, 3, 150]


def _callers(torch, sg, form):
    """(stream, call) for every size; the calls own their outputs and, in the batched form, their handle."""
    from sogrand_b200.batch import Batch

    _, llr = sg.gen_llr(21, 0, max(SIZES), ebn0_range=(1.0, 3.0), device="cuda")
    p = sg.params(Imax=5)
    xs = [llr[:n].contiguous() for n in SIZES]
    handles = [Batch() for _ in SIZES]
    calls = [(lambda x=x, b=b: (b.decode if form == "batch" else sg.decode)(x, p, want_lapp=True))
             for x, b in zip(xs, handles)]
    torch.cuda.synchronize()
    return [torch.cuda.Stream() for _ in SIZES], calls


@pytest.mark.parametrize("form", ["plain", "batch"])
def test_streams_and_threads_give_the_same_results(cuda, sg, form):
    torch = cuda
    streams, calls = _callers(torch, sg, form)
    want = []
    for c in calls:
        want.append([t.clone() for t in c()])
        torch.cuda.synchronize()
    got = [None] * len(calls)

    def work(i):
        with torch.cuda.stream(streams[i]):
            for _ in range(3):
                got[i] = calls[i]()
        streams[i].synchronize()

    for i in range(len(calls)):  # one thread, all streams in flight together
        with torch.cuda.stream(streams[i]):
            got[i] = calls[i]()
    torch.cuda.synchronize()
    assert all(torch.equal(a, b) for g, w in zip(got, want) for a, b in zip(g, w))
    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(calls))]
    [t.start() for t in threads]
    [t.join() for t in threads]
    assert all(torch.equal(a, b) for g, w in zip(got, want) for a, b in zip(g, w))


def test_capture_beside_running_calls(cuda, sg):
    """While one stream is under capture, calls on it are recorded and calls on another stream run."""
    torch = cuda
    from sogrand_b200 import _lib

    lib = _lib.load()
    n = 6
    _, llr = sg.gen_llr(23, 0, n, ebn0_db=2.0, device="cuda")
    p = sg.params()
    want, raw, _ = sg.decode(llr, p)
    out = [(torch.zeros_like(want), torch.zeros_like(raw)) for _ in range(2)]
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()

    def call(o, st):
        _lib.check(lib.sg_decode_device(llr.data_ptr(), n, C.byref(p), o[0].data_ptr(), None, o[1].data_ptr(),
                                        st.cuda_stream))

    call(out[1], b)
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=a, capture_error_mode="global"):
        call(out[0], a)
        for _ in range(3):
            call(out[1], b)
    b.synchronize()
    assert torch.equal(out[1][0], want) and torch.equal(out[1][1], raw) and not out[0][0].any()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(out[0][0], want) and torch.equal(out[0][1], raw)


@pytest.mark.parametrize("form", ["plain", "batch"])
def test_many_streams_share_the_sms(cuda, sg, form):
    """64 streams of 4 codewords each take no longer than the one-CTA forms take over them (half as
    much again allowed); as if each were alone they take 2.2 times as long."""
    torch = cuda
    from sogrand_b200 import autotune, batch

    _, llr = sg.gen_llr(3, 0, 256, ebn0_db=2.0, device="cuda")
    streams = [torch.cuda.Stream() for _ in range(64)]
    handles = [batch.Batch() for _ in streams]
    mod, other = (autotune, "w16-gmem") if form == "plain" else (batch, "p32x3")

    def run():
        for i, s in enumerate(streams):
            with torch.cuda.stream(s):
                (handles[i].decode if form == "batch" else sg.decode)(llr[4 * i : 4 * i + 4])
        torch.cuda.synchronize()

    def best():
        run()
        t = []
        for _ in range(5):
            t0 = time.perf_counter()
            run()
            t.append(time.perf_counter() - t0)
        return min(t)

    got = best()
    before = mod.get_variant()
    try:
        mod.set_variant(other)
        ref = best()
    finally:
        mod.set_variant(before)
    [b.close() for b in handles]
    assert got <= 1.5 * ref, (got, ref)


def test_line_calls_from_threads(cuda, sg):
    """sg_bitso_host from several threads at once, and from new threads after those have ended (each
    thread stages small calls in pinned memory of its own)."""
    _, llr = sg.gen_llr(25, 0, 8, ebn0_db=2.0)
    parts = [np.ascontiguousarray(c) for c in np.array_split(llr.reshape(-1, 16), 16)]
    want = [sg.bitso(p) for p in parts]
    for _ in range(2):
        got = [None] * len(parts)

        def work(i):
            for _ in range(20):
                got[i] = sg.bitso(parts[i])

        threads = [threading.Thread(target=work, args=(i,)) for i in range(len(parts))]
        [t.start() for t in threads]
        [t.join() for t in threads]
        assert all(np.array_equal(a, b) for g, w in zip(got, want) for a, b in zip(g, w))
