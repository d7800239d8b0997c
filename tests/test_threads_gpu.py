"""Calls from several threads, each with its own (default) handle."""
import threading
import time

import numpy as np
import pytest

import uvatrmm_gb300 as u
from oracle import oracle as orc
from tests.helpers import COL, EPS, LEFT, LOWER, NONUNIT, NOTRANS, rel_fro

pytestmark = pytest.mark.gpu


def in_threads(count, work):
    errors = []

    def guarded(k):
        try:
            work(k)
        except Exception as e:  # noqa: BLE001
            errors.append(e)

    threads = [threading.Thread(target=guarded, args=(k,)) for k in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors


def free_bytes():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def gives_back(before, room=64 << 20, seconds=10.0):
    """Free memory is back to `before` but for `room` (a joined Python thread
    may still be ending)."""
    until = time.monotonic() + seconds
    while before - free_bytes() > room and time.monotonic() < until:
        time.sleep(0.01)
    return before - free_bytes() <= room


def test_a_threads_default_handle_gives_its_memory_back(built):
    """Threads that called cblas_dtrmm on the lossless route (a gigabyte of
    scratch each at this size) and ended hold no device memory."""
    n = 2000
    rng = np.random.default_rng(1)
    A, B = rng.uniform(-1, 1, n * n), rng.uniform(-1, 1, n * n)
    want = []

    def work(k):
        C = B.copy()
        u.lib().cblas_dtrmm(COL, LEFT, LOWER, NOTRANS, NONUNIT, n, n, 1.0, A.ctypes.data, n, C.ctypes.data, n)
        assert u.lib().uvatrmm_last_status() == u.OK
        want.append(C)

    in_threads(1, work)  # (loads the kernels)
    time.sleep(0.5)
    before = free_bytes()
    in_threads(4, work)
    assert gives_back(before)
    assert all(np.array_equal(x, want[0]) for x in want)
    cols = orc.dtrmm_dd(COL, LEFT, LOWER, NOTRANS, NONUNIT, n, n, 1.0, A, n, B, n, cols=(7, 8))[:, 0]
    assert np.array_equal(want[0].reshape(n, n)[7], cols)


def test_what_outlives_the_thread_that_made_it(built):
    """A group and a captured call made with a thread's default handle work on
    after the thread has ended; so does a thread whose stream is gone."""
    import ctypes as C

    import torch
    n = 512
    A, B = (torch.rand(n, n, dtype=torch.float64, device="cuda") * 2 - 1 for _ in range(2))
    X, Y, Z = (torch.zeros_like(B) for _ in range(3))
    h = u.Handle()
    args = (COL, LEFT, LOWER, NOTRANS, NONUNIT, n, n, 1.0, A.data_ptr(), n)
    torch.cuda.synchronize()
    h.dtrmm_device_oop(*args[:8], A, n, B, n, Z, n)
    h.sync()
    made, st = {}, torch.cuda.Stream()
    # A first call that is captured takes no workspace: the tile kernel with the handle's control words.
    pinned = u.Handle(engine=u.ENGINE_DFMA)
    wide = torch.rand(100000, 64, dtype=torch.float64, device="cuda")
    out = torch.zeros_like(wide)
    torch.cuda.synchronize()
    pinned.dtrmm_device_oop(*args[:5], 64, 100000, 1.0, A, n, wide, 64, out, 64)
    pinned.sync()
    pinned.close()
    wanted = out.clone()

    class Default:  # a NULL handle: the calling thread's own
        h = None

    def work(k):
        L = u.lib()
        if k == 0:
            X.copy_(B)
            torch.cuda.synchronize()
            made["group"] = u.Group(Default, [dict(layout=COL, side=LEFT, uplo=LOWER, transa=NOTRANS, diag=NONUNIT, m=n,
                                                   n=n, alpha=1.0, A=A, lda=n, B=X, ldb=n)])
        elif k == 1:
            u.check(L.uvatrmm_set_stream(None, C.c_void_p(st.cuda_stream)))
            with torch.cuda.stream(st):
                call = (*args, B.data_ptr(), n, Y.data_ptr(), n)
                u.check(L.uvatrmm_dtrmm_device_oop(None, *call))
                u.check(L.uvatrmm_sync(None))
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=st, capture_error_mode="thread_local"):
                    u.check(L.uvatrmm_dtrmm_device_oop(None, *call))
                made["graph"] = graph
        else:
            u.check(L.uvatrmm_set_stream(None, C.c_void_p(st.cuda_stream)))
            with torch.cuda.stream(st):
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=st, capture_error_mode="thread_local"):
                    u.check(L.uvatrmm_dtrmm_device_oop(None, *args[:5], 64, 100000, 1.0, A.data_ptr(), n,
                                                       wide.data_ptr(), 64, out.data_ptr(), 64))
                made["tile graph"] = graph

    for k in range(3):
        t = threading.Thread(target=work, args=(k,))
        t.start()
        t.join()
    time.sleep(0.5)  # (the threads have ended)
    held = [torch.full((1 << 22,), 7.0, dtype=torch.float64, device="cuda") for _ in range(16)]
    Y.zero_()
    out.zero_()
    torch.cuda.synchronize()
    made["group"].run()
    made["graph"].replay()
    made["tile graph"].replay()
    torch.cuda.synchronize()
    assert torch.equal(X, Z) and torch.equal(Y, Z) and torch.equal(out, wanted)
    assert all(bool((x == 7.0).all()) for x in held)
    made["group"].close()
    h.close()


def test_a_thread_may_end_during_another_threads_capture(built):
    """Its default handle is given back without ending the capture."""
    import torch
    n = 512
    A, B = (torch.rand(n, n, dtype=torch.float64, device="cuda") for _ in range(2))
    X, x = torch.zeros_like(B), torch.zeros(100, device="cuda")
    torch.cuda.synchronize()
    called, end, errors = threading.Event(), threading.Event(), []

    def work():
        try:
            u.check(u.lib().uvatrmm_dtrmm_device_oop(None, COL, LEFT, LOWER, NOTRANS, NONUNIT, n, n, 1.0, A.data_ptr(),
                                                     n, B.data_ptr(), n, X.data_ptr(), n))
            u.check(u.lib().uvatrmm_sync(None))
        except Exception as e:  # noqa: BLE001
            errors.append(e)
        called.set()
        end.wait(30)

    before = free_bytes()
    t = threading.Thread(target=work)
    t.start()
    called.wait(30)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=torch.cuda.Stream(), capture_error_mode="global"):
        x.add_(1)
        end.set()
        t.join()
        time.sleep(0.5)  # (the thread has ended)
        x.add_(1)
    graph.replay()
    torch.cuda.synchronize()
    assert not errors and float(x[0]) == 2.0
    assert gives_back(before)


def test_calls_from_several_threads(built):
    """Six threads with a handle and stream each, sizes of every route, device
    and host calls: each result is the one of a thread alone, bit by bit."""
    import torch
    shapes = [(64, 64), (300, 300), (500, 333), (1000, 5), (700, 650), (129, 1000)]
    inputs, alone = [], []
    h = u.Handle()
    gen = torch.Generator(device="cuda").manual_seed(2)
    for m, n in shapes:
        A = torch.rand(m, m, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
        B = torch.rand(n, m, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1
        C = torch.zeros_like(B)
        torch.cuda.synchronize()
        h.dtrmm_device_oop(COL, LEFT, LOWER, NOTRANS, NONUNIT, m, n, 1.0, A, m, B, m, C, m)
        h.sync()
        inputs.append((A, B, A.cpu().numpy().ravel(), B.cpu().numpy().ravel()))
        alone.append(C.cpu().numpy())
        ref = inputs[-1][3].copy()
        orc.blas_dtrmm(COL, LEFT, LOWER, NOTRANS, NONUNIT, m, n, 1.0, inputs[-1][2], m, ref, m)
        assert rel_fro(alone[-1].ravel(), ref) <= 8 * m * EPS

    def work(k):
        st = torch.cuda.Stream()
        own = u.Handle(stream=st)
        with torch.cuda.stream(st):
            for i in range(40):
                j = (i + k) % len(shapes)
                m, n = shapes[j]
                A, B, hA, hB = inputs[j]
                if i % 4 == 3:
                    C = hB.copy()
                    own.dtrmm(COL, LEFT, LOWER, NOTRANS, NONUNIT, m, n, 1.0, hA, m, C, m)
                    got = C.reshape(n, m)
                else:
                    C = torch.zeros_like(B) if i % 2 else B.clone()
                    if i % 2:
                        own.dtrmm_device_oop(COL, LEFT, LOWER, NOTRANS, NONUNIT, m, n, 1.0, A, m, B, m, C, m)
                    else:
                        own.dtrmm_device(COL, LEFT, LOWER, NOTRANS, NONUNIT, m, n, 1.0, A, m, C, m)
                    own.sync()
                    got = C.cpu().numpy()
                assert np.array_equal(got, alone[j]), (k, i, shapes[j])
        own.close()

    in_threads(6, work)
    h.close()


def test_small_calls_beside_another_streams_long_kernel(built):
    """Calls whose scaling is one launch with an exchange between its blocks,
    while a pinned handle's tile kernel (some 0.2 s) holds the SMs."""
    import torch
    n, big = 512, 6000
    A, B = (torch.rand(n, n, dtype=torch.float64, device="cuda") for _ in range(2))
    X, Y = (torch.rand(big, big, dtype=torch.float64, device="cuda") for _ in range(2))
    Z, want = torch.zeros_like(Y), torch.zeros_like(B)
    one, two = torch.cuda.Stream(), torch.cuda.Stream()
    h, pinned = u.Handle(stream=one), u.Handle(stream=two, engine=u.ENGINE_DFMA)
    out = [torch.zeros_like(B) for _ in range(30)]
    torch.cuda.synchronize()
    h.dtrmm_device_oop(COL, LEFT, LOWER, NOTRANS, NONUNIT, n, n, 1.0, A, n, B, n, want, n)
    h.sync()
    pinned.dtrmm_device_oop(COL, LEFT, LOWER, NOTRANS, NONUNIT, big, big, 1.0, X, big, Y, big, Z, big)
    for C in out:
        h.dtrmm_device_oop(COL, LEFT, LOWER, NOTRANS, NONUNIT, n, n, 1.0, A, n, B, n, C, n)
    h.sync()
    pinned.sync()
    assert all(torch.equal(C, want) for C in out)
    h.close()
    pinned.close()
