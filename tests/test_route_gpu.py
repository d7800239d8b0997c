"""The lossless route of the FP64 calls at its edges: waits that run out, calls
it declines, handles and options that keep it off or bound it."""
import numpy as np
import pytest

import uvatrmm_gb300 as u
from oracle import oracle as orc
from tests.helpers import COL, EPS, LEFT, LOWER, NONUNIT, NOTRANS, RIGHT, TRANS, UPPER
from tests.test_exact_gpu import operands, run

pytestmark = pytest.mark.gpu


def oracle_dd(side, uplo, trans, m, n, alpha, A, lda, B, ldb):
    return orc.dtrmm_dd(COL, side, uplo, trans, NONUNIT, m, n, alpha, A.cpu().numpy().ravel(), lda,
                        B.cpu().numpy().ravel(), ldb)


def assert_fp64_tier(got, want, k):
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= 8 * k * EPS, err


@pytest.mark.parametrize("side,m,n", [(LEFT, 400, 300), (RIGHT, 129, 512), (LEFT, 512, 700)])
def test_an_exchange_that_runs_out_leaves_the_call_to_the_fp64_kernels(built, side, m, n):
    """One block of the one-launch scaling gives up its wait: it has cut no
    residues, so the call is the FP64 kernels', right and reported as
    ETIMEOUT; the calls after it take the route again."""
    h = u.Handle()
    ka = m if side == LEFT else n
    try:
        A0, lda, B0, ldb = operands(side, UPPER, m, n, "normal", pad=1)
        run(h, side, UPPER, NOTRANS, NONUNIT, m, n, 1.0, A0, lda, B0, ldb, in_place=True)  # other planes
        A, lda, B, ldb = operands(side, UPPER, m, n, "uniform", pad=1)
        want = oracle_dd(side, UPPER, NOTRANS, m, n, 1.5, A, lda, B, ldb)
        for _ in range(2):
            for in_place in (True, False):
                h.set_option("exchange_expiry_test", 1000)
                out = B.clone()
                if in_place:
                    h.dtrmm_device(COL, side, UPPER, NOTRANS, NONUNIT, m, n, 1.5, A, lda, out, ldb)
                else:
                    h.dtrmm_device_oop(COL, side, UPPER, NOTRANS, NONUNIT, m, n, 1.5, A, lda, B, ldb, out, ldb)
                with pytest.raises(u.UvatrmmError) as ei:
                    h.sync()
                assert ei.value.status == u.ETIMEOUT
                h.set_option("exchange_expiry_test", 0)
                assert_fp64_tier(out.cpu().numpy()[:, :m].T, want, ka)
                one = oracle_dd(side, UPPER, NOTRANS, m, n, 1.0, A, lda, B, ldb)
                got = run(h, side, UPPER, NOTRANS, NONUNIT, m, n, 1.0, A, lda, B, ldb, in_place)
                assert np.array_equal(got[:, :m].T, one)
    finally:
        h.close()


@pytest.mark.parametrize("side,m,n", [(LEFT, 400, 400), (LEFT, 1000, 1000), (RIGHT, 900, 1500), (LEFT, 300, 5000)])
def test_the_scratch_option_bounds_the_route(built, side, m, n):
    """With 64 MiB a call goes in panels and passes that fit, in place and out
    of place, with the same results; the handle takes no more than that."""
    import torch
    h, warm = u.Handle(), u.Handle()
    try:
        h.set_option("ozaki_scratch_mb", 64)
        A, lda, B, ldb = operands(side, LOWER, m, n, "wide")
        want = run(warm, side, LOWER, TRANS, NONUNIT, m, n, 1.0, A, lda, B, ldb, in_place=False)
        one = oracle_dd(side, LOWER, TRANS, m, n, 1.0, A, lda, B, ldb) if m * n <= 200000 else None
        out = B.clone()
        h.sync()
        torch.cuda.synchronize()
        free, _ = torch.cuda.mem_get_info()
        h.dtrmm_device_oop(COL, side, LOWER, TRANS, NONUNIT, m, n, 1.0, A, lda, B, ldb, out, ldb)
        h.sync()
        # (The scales' few hundred kilobytes, and 2 MiB steps of three blocks.)
        assert free - torch.cuda.mem_get_info()[0] <= (64 + 16) << 20
        assert np.array_equal(out.cpu().numpy(), want)
        assert one is None or np.array_equal(want[:, :m].T, one)
        got = run(h, side, LOWER, TRANS, NONUNIT, m, n, 1.0, A, lda, B, ldb, in_place=True)
        assert np.array_equal(got, want)
    finally:
        h.close()
        warm.close()


def test_a_groups_waves_fit_the_scratch_option(built):
    """FP64 problems join waves that fit the option; one that does not fit by
    itself (900 x 1500) runs on the tile kernel."""
    import torch
    h = u.Handle()
    try:
        h.set_option("ozaki_scratch_mb", 64)
        probs, staged = [], 0
        for i, (side, m, n) in enumerate([(LEFT, 400, 400), (RIGHT, 300, 450), (LEFT, 900, 1500), (RIGHT, 333, 512)]):
            A, lda, B, ldb = operands(side, UPPER, m, n, "uniform")
            probs.append(dict(layout=COL, side=side, uplo=UPPER, transa=NOTRANS, diag=NONUNIT, m=m, n=n, alpha=1.0, A=A,
                              lda=lda, B=B.clone(), B0=B, ldb=ldb, tier=u.TIER_FP64, moduli=0))
            staged += 8 * (m + 15) // 16 * 16 * n + 8 * (lda + 15) // 16 * 16 * lda
        torch.cuda.synchronize()
        g = u.Group(h, probs)
        st = g.stats()
        g.run()
        h.sync()
        g.close()
        assert st["arena_bytes"] <= (64 << 20) + staged + (1 << 20)
        assert st["ozaki_waves"] == 3
        for i, p in enumerate(probs):
            m, n = p["m"], p["n"]
            want = oracle_dd(p["side"], UPPER, NOTRANS, m, n, 1.0, p["A"], p["lda"], p["B0"], p["ldb"])
            got = p["B"].cpu().numpy()[:, :m].T
            if i == 2:
                assert_fp64_tier(got, want, m)
            else:
                assert np.array_equal(got, want)
    finally:
        h.close()


@pytest.mark.parametrize("option", [("schedule", u.SCHED_REG), ("shape", u.SHAPE_BOXES), ("tile", 64)])
def test_a_pinned_handles_gemm_stage_and_product_stay_on_the_tile_kernel(built, option):
    """A handle whose schedule, shape or tile was set keeps its GEMMs, stages
    and products on the FP64 tile kernel: bit by bit those of a handle whose
    engine was."""
    import torch
    h, pinned = u.Handle(**dict([option])), u.Handle(engine=u.ENGINE_DFMA)
    pinned.set_option(*option)
    n, w, b, hr = 900, 700, 300, 500
    gen = torch.Generator(device="cuda").manual_seed(9)
    A, B = (torch.rand(n, n, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1 for _ in range(2))
    torch.cuda.synchronize()
    out = []
    try:
        for hh in (h, pinned):
            C = [torch.zeros(n, n, dtype=torch.float64, device="cuda") for _ in range(3)]
            torch.cuda.synchronize()
            hh.dgemm_device(COL, NOTRANS, TRANS, n, n, n, -0.5, A, n, B, n, 0.0, C[0], n)
            hh.stage(n, w, b, hr, A[b:], n, B, n, C[1], n)
            hh.product(n, u.SCHED_DYNAMIC, u.SHAPE_TRAPEZOID, A, B, C[2])
            hh.sync()
            out.append(C)
        for x, y in zip(*out):
            assert bool(x.any()) and torch.equal(x, y)
    finally:
        h.close()
        pinned.close()


@pytest.mark.parametrize("n", [270, 1000, 4096])
def test_a_products_time_holds_no_allocation(built, n):
    """uvatrmm_product's seconds on a new handle, whose workspace it takes, are
    those of its next products (within a factor of two; the allocations take
    0.2 ms and more)."""
    import torch
    A, B = (torch.rand(n, n, dtype=torch.float64, device="cuda") for _ in range(2))
    C = torch.zeros(n, n, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    warm = u.Handle()
    for _ in range(3):  # (loads the kernels)
        warm.product(n, u.SCHED_DYNAMIC, u.SHAPE_TRAPEZOID, A, B, C)
    first, later = [], []
    for _ in range(5):
        h = u.Handle()
        first.append(h.product(n, u.SCHED_DYNAMIC, u.SHAPE_TRAPEZOID, A, B, C))
        later += [h.product(n, u.SCHED_DYNAMIC, u.SHAPE_TRAPEZOID, A, B, C) for _ in range(3)]
        h.close()
    warm.close()
    assert np.median(first) <= 2 * np.median(later), (first, later)


def triangle(A, uplo, trans):
    """op(A) as a host matrix from the column-major device tensor."""
    x = A.cpu().numpy().T
    x = np.tril(x) if uplo == LOWER else np.triu(x)
    return x.T if trans == TRANS else x


def assert_within_fp64(got, side, T, B, alpha, want, where):
    """Entry by entry within 8 k eps of |alpha| |op(A)| |B| of the double-double oracle."""
    k = T.shape[0]
    room = 8 * k * EPS * abs(alpha) * (np.abs(T) @ np.abs(B) if side == LEFT else np.abs(B) @ np.abs(T))
    assert np.all(np.abs(got - want)[where] <= room[where])


# (By the repository's rule the small kernel stands behind the route at these
# sizes, split along K at the first three.)
@pytest.mark.parametrize("ka,vecs", [(300, 300), (217, 401), (2500, 12), (700, 300)])
@pytest.mark.parametrize("side,uplo,trans", [(LEFT, LOWER, NOTRANS), (LEFT, UPPER, TRANS), (RIGHT, UPPER, NOTRANS),
                                             (RIGHT, LOWER, TRANS), (LEFT, UPPER, NOTRANS)])
@pytest.mark.parametrize("what", ["span", "nan"])
def test_declined_calls_are_right(built, ka, vecs, side, uplo, trans, what):
    """Operands that the route cannot hold, at sizes where a split kernel
    computes the call: in place, out of place and on host memory."""
    h = u.Handle()
    m, n = (ka, vecs) if side == LEFT else (vecs, ka)
    try:
        A, lda, B, ldb = operands(side, uplo, m, n, "uniform", pad=1)
        row, col = m // 3, n // 2
        B[col, row] = 2.0 ** 300 if what == "span" else float("nan")
        T = triangle(A, uplo, trans)
        hB = B.cpu().numpy()[:, :m].T.copy()
        where = np.ones((m, n), bool)
        if what == "nan":  # the line that holds it
            where[(slice(None), col) if side == LEFT else (row, slice(None))] = False
        # (The oracle multiplies by the zeros of the triangle: a zero in place of the NaN.)
        want = oracle_dd(side, uplo, trans, m, n, -0.75, A, lda, B.nan_to_num(0.0), ldb)
        got = [run(h, side, uplo, trans, NONUNIT, m, n, -0.75, A, lda, B, ldb, in_place) for in_place in (True, False)]
        host = B.cpu().numpy().ravel().copy()
        h.dtrmm(COL, side, uplo, trans, NONUNIT, m, n, -0.75, A.cpu().numpy().ravel(), lda, host, ldb)
        got.append(host.reshape(n, ldb))
        hB[np.isnan(hB)] = 0.0
        for x in got:
            assert np.all(x[:, m:] == -7.0), "padding was written"
            C = x[:, :m].T
            assert_within_fp64(C, side, T, hB, -0.75, want, where)
            if what == "nan":
                # Its line: not a number where the entry takes part, right away from there.
                line = C[:, col] if side == LEFT else C[row, :]
                true, at = (want[:, col], row) if side == LEFT else (want[row, :], col)
                takes = T[:, at] != 0.0 if side == LEFT else T[at, :] != 0.0
                assert not np.isfinite(line[takes]).any()
                far = ~takes & (np.abs(np.arange(ka) - at) >= 64)
                assert np.allclose(line[far], true[far], rtol=0, atol=8 * ka * EPS * ka)
    finally:
        h.close()


@pytest.mark.parametrize("entry", [float("nan"), float("inf"), 2.0 ** 300])
@pytest.mark.parametrize("layout,ta,tb", [(COL, NOTRANS, NOTRANS), (COL, TRANS, NOTRANS), (101, NOTRANS, TRANS)])
def test_declined_gemms_and_host_calls_equal_the_pinned_handles(built, layout, ta, tb, entry):
    """A GEMM whose operands the route cannot hold, odd leading dimensions and
    beta, and a host TRMM (1100 x 901): the tile kernel's finite results, bit
    by bit."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(5)
    h, pinned = u.Handle(), u.Handle(engine=u.ENGINE_DFMA)
    m, n, k = 700, 651, 903

    def store(rows, cols):  # (lines of the layout, one entry longer: odd where the length is even)
        lines, length = (cols, rows) if layout == COL else (rows, cols)
        ld = length + 1 + length % 2
        return torch.rand(lines, ld, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1, ld

    A, lda = store(k, m) if ta == TRANS else store(m, k)
    B, ldb = store(n, k) if tb == TRANS else store(k, n)
    C, ldc = store(m, n)
    B[40, 30] = entry
    try:
        out = []
        for hh in (h, pinned):
            X = C.clone()
            torch.cuda.synchronize()
            hh.dgemm_device(layout, ta, tb, m, n, k, -0.5, A, lda, B, ldb, 2.0, X, ldc)
            hh.sync()
            host = np.random.default_rng(1).uniform(-1, 1, 1100 * 901)
            T = np.random.default_rng(2).uniform(-1, 1, 1100 * 1100)
            host[5000] = entry
            hh.dtrmm(COL, LEFT, LOWER, ta, NONUNIT, 1100, 901, 1.25, T, 1100, host, 1100)
            out.append((X.cpu().numpy(), host))
        for x, y in zip(*out):
            fine = np.isfinite(y)  # (the tile kernel also multiplies by zeros beside the diagonal)
            assert np.array_equal(x[fine], y[fine])
            assert fine.mean() > 0.9
    finally:
        h.close()
        pinned.close()


@pytest.mark.parametrize("on_device", [True, False])
def test_a_server_reserves_the_moduli_that_fit_and_gives_back_the_rest(built, on_device):
    """Under 2 GiB a 1500 x 1500 request has planes for 16 moduli: uniform
    entries (14) take the route, as single calls do; entries of wide spans (some
    24) and a request too large for any planes run as tiles.  More are sent at
    once than 2 GiB hold planes for."""
    import torch
    h = u.Handle()
    srv = u.Server(h, hbm_budget_bytes=2 << 30)
    try:
        probs = []
        for i, (n, data) in enumerate([(1500, "uniform")] * 9 + [(1500, "wide"), (5200, "uniform"), (1500, "uniform")]):
            side = [LEFT, RIGHT][i % 2]
            A, lda, B, ldb = operands(side, LOWER, n, n, data)
            probs.append(dict(layout=COL, side=side, uplo=LOWER, transa=NOTRANS, diag=NONUNIT, m=n, n=n, alpha=1.0, A=A,
                              lda=lda, B=B.clone(), B0=B, ldb=ldb, tier=u.TIER_FP64, moduli=0, data=data))
        want = [run(h, p["side"], LOWER, NOTRANS, NONUNIT, p["m"], p["m"], 1.0, p["A"], p["lda"], p["B0"], p["ldb"],
                    in_place=False) for p in probs]
        torch.cuda.synchronize()
        for _ in range(2):
            for p in probs:
                p["B"].copy_(p["B0"])
            torch.cuda.synchronize()
            sent = probs if on_device else [dict(p, A=p["A"].cpu().numpy(), B=p["B0"].cpu().numpy()) for p in probs]
            for rid in [srv.submit(p, on_device=on_device) for p in sent]:
                assert srv.wait(rid) == 0
            for p, q, w in zip(probs, sent, want):
                got = q["B"].cpu().numpy() if on_device else q["B"]
                if p["m"] == 1500 and p["data"] == "uniform":
                    assert np.array_equal(got, w)
                else:
                    assert not np.array_equal(got, w)
                    assert np.linalg.norm(got - w) <= 8 * p["m"] * EPS * np.linalg.norm(w)
        assert srv.stats()["peak_bytes"] <= 2 << 30
    finally:
        srv.close()
        h.close()


@pytest.mark.parametrize("side,ka,vecs", [(LEFT, 5000, 60), (RIGHT, 3293, 135), (LEFT, 65, 30730), (RIGHT, 768, 2564),
                                          (LEFT, 120, 14785)])
def test_declined_calls_take_little_longer_than_the_tile_kernel(built, side, ka, vecs):
    """At most 30 % (the scaling and the launches that return at once are 30 us
    of 275 at the smallest; kernels that found the chip unevenly occupied, or
    the slower of the two, took 40 to 70 % more)."""
    import torch
    m, n = (ka, vecs) if side == LEFT else (vecs, ka)
    A, lda, B, ldb = operands(side, LOWER, m, n, "uniform")
    B[n // 2, m // 2] = float("nan")
    out = torch.zeros_like(B)
    took = []
    for options in ({}, {"engine": u.ENGINE_DFMA}):
        h = u.Handle(**options)
        times = []
        for _ in range(7):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            for _ in range(5):
                h.dtrmm_device_oop(COL, side, LOWER, NOTRANS, NONUNIT, m, n, 1.0, A, lda, B, ldb, out, ldb)
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        h.close()
        took.append(np.median(times[2:]))
    assert took[0] <= 1.3 * took[1], took


@pytest.mark.parametrize("m,n,k", [(4, 87428, 452), (1, 37864, 4631), (3, 14222, 412), (2, 13501, 510)])
def test_thin_gemms_are_not_slower_than_the_tile_kernel(built, m, n, k):
    """GEMMs of a few rows and many columns, whose tiles cost what their rows do
    (they took up to 70 % longer on the lossless route): at most 10 % over a
    pinned handle, and right."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(4)
    A, B = (torch.rand(s, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1 for s in ((k, m), (k, n)))
    C = torch.zeros(n, m, dtype=torch.float64, device="cuda")  # column-major: C = A (m x k) * B (n x k)^T
    took = []
    for options in ({}, {"engine": u.ENGINE_DFMA}):
        h = u.Handle(**options)
        times = []
        for _ in range(7):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            torch.cuda.synchronize()
            e0.record()
            for _ in range(5):
                h.dgemm_device(COL, NOTRANS, TRANS, m, n, k, 1.0, A, m, B, n, 0.0, C, m)
            e1.record()
            torch.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        if not options:
            want = (A.t().double() @ B).t()
            room = 8 * k * EPS * (A.t().abs() @ B.abs()).t()
            assert bool(((C - want).abs() <= room).all())
        h.close()
        took.append(np.median(times[2:]))
    assert took[0] <= 1.1 * took[1], took
