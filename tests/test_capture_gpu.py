"""Device calls captured into CUDA graphs: a replay gives what the call gives,
also after later, larger calls have made the handle's workspace grow."""
import numpy as np
import pytest

import uvatrmm_gb300 as u
from tests.helpers import COL, LEFT, LOWER, NONUNIT, NOTRANS, RIGHT, TRANS, UPPER

pytestmark = pytest.mark.gpu


def rand(seed, *shape):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand(*shape, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1


def trmm_oop(m, n):
    def call(h, A, B, C):
        h.dtrmm_device_oop(COL, LEFT, LOWER, NOTRANS, NONUNIT, m, n, 1.5, A, m, B, m, C, m)
    return call, (m, m), (n, m)


def trmm_in_place(m, n):
    def call(h, A, B, C):
        C.copy_(B)
        h.dtrmm_device(COL, RIGHT, UPPER, TRANS, NONUNIT, m, n, -0.5, A, n, C, m)
    return call, (n, n), (n, m)


def gemm(m, n, k):
    def call(h, A, B, C):
        h.dgemm_device(COL, NOTRANS, NOTRANS, m, n, k, 1.0, A, m, B, k, 0.0, C, m)
    return call, (k, m), (n, k)


def emulated(m, n):
    def call(h, A, B, C):
        C.copy_(B)
        h.ozaki_device(COL, LEFT, UPPER, NOTRANS, NONUNIT, m, n, 1.0, A, m, C, m)
    return call, (m, m), (n, m)


# The lossless route (scaled in one launch and in two), the small kernel split
# along K, the staged copy of B, and the emulated tier.
@pytest.mark.parametrize("make", [lambda: trmm_oop(512, 500), lambda: trmm_oop(900, 700), lambda: trmm_oop(1000, 5),
                                  lambda: trmm_in_place(333, 500), lambda: gemm(900, 640, 520),
                                  lambda: emulated(600, 400)])
def test_replays_survive_a_larger_call_on_the_handle(built, make):
    import torch
    call, shape_a, shape_b = make()
    m_out = shape_b[1] if call.__qualname__.split(".")[0] != "gemm" else shape_a[1]
    st = torch.cuda.Stream()
    h, other = u.Handle(stream=st), u.Handle(stream=st)
    A, C, want = rand(1, *shape_a), torch.zeros(shape_b[0], m_out, dtype=torch.float64, device="cuda"), None
    B = rand(2, *shape_b)
    want = torch.zeros_like(C)
    torch.cuda.synchronize()
    try:
        with torch.cuda.stream(st):
            call(h, A, B, C)  # takes the workspace, which a capture could not
            h.sync()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=st):
                call(h, A, B, C)
            # Every workspace slot grows; what a freed one left is handed out and filled.
            n = 2304
            big, right, out = rand(3, n, n), rand(4, n, n), torch.zeros(n, n, dtype=torch.float64, device="cuda")
            h.dtrmm_device(COL, LEFT, LOWER, NOTRANS, NONUNIT, n, n, 1.0, big, n, right, n)
            h.dtrmm_device_oop(COL, LEFT, LOWER, NOTRANS, NONUNIT, 2500 - 196, 2, 1.0, big, n, right, n, out, n)
            h.dtrmm_device_oop(COL, LEFT, LOWER, NOTRANS, NONUNIT, 600, 28, 1.0, big, n, right, n, out, n)
            h.ozaki_device(COL, LEFT, LOWER, NOTRANS, NONUNIT, n, n, 1.0, big, n, out, n)
            h.sync()
            held = [torch.full((1 << 18,), 7.0, dtype=torch.float64, device="cuda") for _ in range(64)]
            held += [torch.full((1 << 24,), 7.0, dtype=torch.float64, device="cuda") for _ in range(8)]
            for seed in (5, 6):
                B.copy_(rand(seed, *shape_b))
                C.zero_()
                graph.replay()
                call(other, A, B, want)
                other.sync()
                assert torch.equal(C, want)
            assert all(bool((x == 7.0).all()) for x in held)
            assert np.isfinite(C.cpu().numpy()).all()
    finally:
        torch.cuda.synchronize()
        h.close()
        other.close()


@pytest.mark.parametrize("make", [lambda: trmm_oop(512, 500), lambda: trmm_oop(1000, 5), lambda: gemm(900, 640, 520)])
@pytest.mark.parametrize("outgrown", [False, True])
def test_growing_a_workspace_does_not_end_another_threads_capture(built, make, outgrown):
    """A call allocates its workspace, and frees the smaller one it had, while
    another thread captures in CUDA's global mode: both come out right."""
    import threading

    import torch
    call, shape_a, shape_b = make()
    A, B = rand(1, *shape_a), rand(2, *shape_b)
    m_out = shape_b[1] if call.__qualname__.split(".")[0] != "gemm" else shape_a[1]
    want = torch.zeros(shape_b[0], m_out, dtype=torch.float64, device="cuda")
    got, x = torch.zeros_like(want), torch.zeros(1000, device="cuda")
    st, warm = torch.cuda.Stream(), u.Handle()
    torch.cuda.synchronize()
    call(warm, A, B, want)  # (loads the kernels, too)
    warm.sync()
    fresh = u.Handle(stream=st)
    if outgrown:
        for m, n in ((300, 300), (86, 1)):
            trmm_oop(m, n)[0](fresh, rand(3, m, m), rand(4, n, m), torch.zeros(n, m, dtype=torch.float64, device="cuda"))
        fresh.sync()
    torch.cuda.synchronize()
    began, called, seen = threading.Event(), threading.Event(), {}

    def capture():
        try:
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=torch.cuda.Stream(), capture_error_mode="global"):
                x.add_(1)
                began.set()
                called.wait(30)
                x.add_(1)
            graph.replay()
            torch.cuda.synchronize()
            seen["x"] = float(x[0])
        except Exception as e:  # noqa: BLE001
            seen["error"] = e
        finally:
            began.set()

    t = threading.Thread(target=capture)
    t.start()
    began.wait(30)
    try:
        call(fresh, A, B, got)
    finally:
        called.set()
        t.join()
    fresh.sync()
    torch.cuda.synchronize()
    assert seen == {"x": 2.0}
    assert torch.equal(got, want)
    fresh.close()
    warm.close()
