"""FP64 calls on the lossless integer route (the residue GEMMs of the tensor
cores, with every bit of every entry kept): each result is the exact product
rounded once, so it equals the double-double oracle's rounding (cblas_dtrmm
semantics, as the reference calls it at UVaTRMM/src/mm_triangular.c:374-387)
entry by entry; operands it cannot hold go to the FP64 kernels, whose finite results are
those of a handle pinned to the tile kernel, bit by bit."""
# (Bit by bit where the small kernel is not split along K: test_route_gpu.py has the split sizes.)
import numpy as np
import pytest

import uvatrmm_gb300 as u
from oracle import oracle as orc
from tests.helpers import COL, LEFT, LOWER, NONUNIT, NOTRANS, RIGHT, TRANS, UNIT, UPPER

pytestmark = pytest.mark.gpu


def operands(side, uplo, m, n, data, pad=0):
    """Column-major device A (NaN in the unreferenced triangle) and B with `pad` unused entries per column."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(3)
    ka = m if side == LEFT else n

    def values(cols, rows):
        x = torch.randn(cols, rows, dtype=torch.float64, device="cuda", generator=gen)
        if data == "integers":
            return torch.round(100 * x)
        x = torch.rand(cols, rows, dtype=torch.float64, device="cuda", generator=gen) * 2 - 1 if data != "normal" else x
        if data == "wide":
            x = torch.ldexp(x, torch.randint(-20, 21, (cols, rows), device="cuda", generator=gen))
        return x

    A, B = values(ka, ka), values(n, m)  # rows of the tensor are the matrix's columns
    keep = torch.ones(ka, ka, dtype=torch.bool, device="cuda")
    keep = torch.triu(keep) if uplo == LOWER else torch.tril(keep)
    A = torch.where(keep, A, torch.full_like(A, float("nan")))
    sB = torch.full((n, m + pad), -7.0, dtype=torch.float64, device="cuda")
    sB[:, :m] = B
    return A.contiguous(), ka, sB, m + pad


def run(h, side, uplo, trans, diag, m, n, alpha, A, lda, B, ldb, in_place):
    import torch
    out = B.clone()
    if in_place:
        h.dtrmm_device(COL, side, uplo, trans, diag, m, n, alpha, A, lda, out, ldb)
    else:
        out[:, :m] = 0
        h.dtrmm_device_oop(COL, side, uplo, trans, diag, m, n, alpha, A, lda, B, ldb, out, ldb)
    h.sync()
    torch.cuda.synchronize()
    return out.cpu().numpy()


SIZES = [(513, 600), (640, 640), (1100, 1531), (2311, 1029)]


@pytest.mark.parametrize("data", ["uniform", "normal", "wide", "integers"])
@pytest.mark.parametrize("side,uplo,trans,diag", [(LEFT, LOWER, NOTRANS, NONUNIT), (LEFT, UPPER, TRANS, UNIT),
                                                  (RIGHT, LOWER, NOTRANS, UNIT), (RIGHT, UPPER, TRANS, NONUNIT),
                                                  (LEFT, LOWER, TRANS, UNIT), (RIGHT, UPPER, NOTRANS, NONUNIT)])
def test_every_result_is_the_exact_product_rounded_once(handle, side, uplo, trans, diag, data):
    for k, (m, n) in enumerate(SIZES):
        A, lda, B, ldb = operands(side, uplo, m, n, data, pad=k)
        got = run(handle, side, uplo, trans, diag, m, n, 1.0, A, lda, B, ldb, in_place=k != 1)
        assert np.all(got[:, m:] == -7.0), "padding was written"
        hA, hB = A.cpu().numpy().ravel(), B.cpu().numpy().ravel()
        lines = n if side == LEFT else m
        for j in (0, 1, lines // 2, lines - 1):
            if side == LEFT:
                want = orc.dtrmm_dd(COL, side, uplo, trans, diag, m, n, 1.0, hA, lda, hB, ldb, cols=(j, j + 1))[:, 0]
                have = got[j, :m]
            else:
                want = orc.dtrmm_dd(COL, side, uplo, trans, diag, m, n, 1.0, hA, lda, hB, ldb, rows=(j, j + 1))[0, :]
                have = got[:, j]
            assert np.array_equal(have, want), (m, n, j, np.max(np.abs(have - want)))


@pytest.mark.parametrize("what", ["nan in B", "inf in A", "span beyond the CRT sets", "subnormal products"])
def test_operands_the_route_cannot_hold_take_the_fp64_kernels(handle, what):
    m, n = SIZES[2]
    A, lda, B, ldb = operands(LEFT, LOWER, m, n, "uniform", pad=1)
    if what == "nan in B":
        B[7, 5] = float("nan")
    elif what == "inf in A":
        A[3, 900] = float("inf")
    elif what == "span beyond the CRT sets":
        B[11, 20] = 2.0 ** 300
    else:
        A *= 2.0 ** -540
        B[:, :m] *= 2.0 ** -500
    pinned = u.Handle()
    try:
        pinned.set_option("engine", u.ENGINE_DFMA)
        for in_place in (True, False):
            got = run(handle, LEFT, LOWER, NOTRANS, NONUNIT, m, n, -0.75, A, lda, B, ldb, in_place)
            want = run(pinned, LEFT, LOWER, NOTRANS, NONUNIT, m, n, -0.75, A, lda, B, ldb, in_place)
            fine = np.isfinite(want)
            assert np.array_equal(got[fine], want[fine])
            if what == "nan in B":  # (the tile kernel also multiplies it by zeros beside the diagonal)
                assert not np.isfinite(got[7, 5:m]).any() and np.isfinite(got[:7, :m]).all()
            elif what == "inf in A":
                assert not np.isfinite(got[:, 900]).any() and np.isfinite(got[:, 901:m]).all()
            else:
                assert fine.all()
    finally:
        pinned.close()


def test_zero_operands_and_zero_lines(handle):
    m, n = SIZES[1]
    A, lda, B, ldb = operands(LEFT, UPPER, m, n, "uniform")
    B[5] = 0.0
    got = run(handle, LEFT, UPPER, NOTRANS, NONUNIT, m, n, -2.0, A, lda, B, ldb, True)
    assert np.all(got[5] == 0.0) and np.all(got[6] != 0.0)
    B.zero_()
    assert np.all(run(handle, LEFT, UPPER, NOTRANS, NONUNIT, m, n, 1.0, A, lda, B, ldb, True) == 0.0)


VARIANTS = [(side, uplo, trans, diag) for side in (LEFT, RIGHT) for uplo in (LOWER, UPPER)
            for trans in (NOTRANS, TRANS) for diag in (NONUNIT, UNIT)]


@pytest.mark.parametrize("ka,vecs", [(1, 1), (31, 5), (32, 4), (33, 130), (65, 3), (85, 2), (128, 1000)])
def test_small_products_equal_the_tile_kernel(built, ka, vecs):
    """The small kernel's row blocks (32), vector groups (4), clusters (in
    place) and K chunks (32), all variants: unsplit, the sums run in the tile
    kernel's order, so the results are its own, bit by bit."""
    h, pinned = u.Handle(), u.Handle()
    pinned.set_option("engine", u.ENGINE_DFMA)
    try:
        for side, uplo, trans, diag in VARIANTS:
            m, n = (ka, vecs) if side == LEFT else (vecs, ka)
            A, lda, B, ldb = operands(side, uplo, m, n, "normal", pad=1)
            for in_place in (True, False):
                got = run(h, side, uplo, trans, diag, m, n, 1.5, A, lda, B, ldb, in_place)
                want = run(pinned, side, uplo, trans, diag, m, n, 1.5, A, lda, B, ldb, in_place)
                assert np.array_equal(got, want), (side, uplo, trans, diag, in_place)
    finally:
        h.close()
        pinned.close()


@pytest.mark.parametrize("ka,vecs", [(86, 1), (200, 64), (257, 2), (600, 1), (1000, 5), (2500, 2)])
def test_small_products_split_along_k(built, ka, vecs):
    """Too few outputs for the chip: K is split into chunks and the partial
    sums are added in order.  Within 8 k eps of the double-double oracle (the
    FP64 tier's bound), in place and out of place alike, bit by bit."""
    h = u.Handle()
    try:
        for side, uplo, trans, diag in VARIANTS[::3]:
            m, n = (ka, vecs) if side == LEFT else (vecs, ka)
            A, lda, B, ldb = operands(side, uplo, m, n, "normal", pad=1)
            got = run(h, side, uplo, trans, diag, m, n, 1.5, A, lda, B, ldb, True)
            assert np.all(got[:, m:] == -7.0), "padding was written"
            assert np.array_equal(got[:, :m], run(h, side, uplo, trans, diag, m, n, 1.5, A, lda, B, ldb, False)[:, :m])
            want = orc.dtrmm_dd(COL, side, uplo, trans, diag, m, n, 1.5, A.cpu().numpy().ravel(), lda,
                                B.cpu().numpy().ravel(), ldb)
            err = np.linalg.norm(got[:, :m].T - want) / np.linalg.norm(want)
            assert err <= 8 * ka * np.finfo(np.float64).eps, err
    finally:
        h.close()


def mixed(seed, count=14):
    """FP64 and Ozaki problems on both sides of the route's threshold, one of
    them with a NaN in B and one with an entry no CRT set spans."""
    import torch
    rng = np.random.default_rng(seed)
    out = []
    for i in range(count):
        m, n = int(rng.integers(100, 1300)), int(rng.integers(40, 1300))
        if i in (4, 5):  # (large enough for the route)
            m, n = m + 700, n + 700
        side, uplo = [LEFT, RIGHT][i % 2], [LOWER, UPPER][(i // 2) % 2]
        A, lda, B, ldb = operands(side, uplo, m, n, ["uniform", "wide"][i % 3 == 0], pad=i % 2)
        if i == 4:
            B[3, 2] = float("nan")
        if i == 5:
            B[1, 1] = 2.0 ** 250
        out.append(dict(layout=COL, side=side, uplo=uplo, transa=[NOTRANS, TRANS][(i // 4) % 2], diag=NONUNIT, m=m,
                        n=n, alpha=[1.0, -0.5][i % 2], A=A, lda=lda, B=B.clone(), B0=B, ldb=ldb,
                        tier=u.TIER_OZAKI if i in (2, 9) else u.TIER_FP64, moduli=0))
    torch.cuda.synchronize()
    return out


def singles(h, probs):
    res = []
    for p in probs:
        B = p["B0"].clone()
        call = h.ozaki_device if p["tier"] == u.TIER_OZAKI else h.dtrmm_device
        call(p["layout"], p["side"], p["uplo"], p["transa"], p["diag"], p["m"], p["n"], p["alpha"], p["A"], p["lda"],
             B, p["ldb"])
        h.sync()
        res.append(B.cpu().numpy())
    return res


def test_groups_take_the_same_routes_as_single_calls(built):
    h = u.Handle()
    try:
        probs = mixed(1)
        want = singles(h, probs)
        g = u.Group(h, probs)
        for _ in range(2):  # the captured graph decides anew on every run
            for p in probs:
                p["B"].copy_(p["B0"])
            g.run()
            h.sync()
            for p, r in zip(probs, want):
                assert np.array_equal(p["B"].cpu().numpy(), r, equal_nan=True), (p["m"], p["n"], p["tier"])
        g.close()
    finally:
        h.close()


@pytest.mark.parametrize("on_device", [True, False])
def test_served_requests_take_the_same_routes_as_single_calls(built, on_device):
    import torch
    h = u.Handle()
    srv = u.Server(h, hbm_budget_bytes=24 << 30)
    try:
        probs = mixed(2)
        want = singles(h, probs)
        for _ in range(2):
            for p in probs:
                p["B"].copy_(p["B0"])
            torch.cuda.synchronize()
            sent = probs if on_device else [dict(p, A=p["A"].cpu().numpy(), B=p["B0"].cpu().numpy()) for p in probs]
            ids = [srv.submit(p, on_device=on_device) for p in sent]
            for i in ids:
                assert srv.wait(i) == 0
            for p, q, r in zip(probs, sent, want):
                got = q["B"].cpu().numpy() if on_device else q["B"]
                assert np.array_equal(got, r, equal_nan=True), (p["m"], p["n"], p["tier"])
    finally:
        srv.close()
        h.close()


@pytest.mark.parametrize("layout,ta,tb", [(101, NOTRANS, NOTRANS), (102, TRANS, NOTRANS), (101, NOTRANS, TRANS)])
def test_gemm_is_exact_up_to_its_last_rounding(built, layout, ta, tb):
    """alpha * A * B + beta * C with integer entries: every product is exact."""
    import torch
    h = u.Handle()
    m, n, k = 700, 651, 903
    gen = torch.Generator(device="cuda").manual_seed(5)
    A, B, C = (torch.randint(-2000, 2001, s, device="cuda", generator=gen).to(torch.float64)
               for s in ((k, m) if ta == TRANS else (m, k), (n, k) if tb == TRANS else (k, n), (m, n)))
    want = -0.5 * ((A.t() if ta == TRANS else A) @ (B.t() if tb == TRANS else B)) + 2.0 * C
    store = (lambda x: x.contiguous()) if layout == 101 else (lambda x: x.t().contiguous())
    sA, sB, sC = store(A), store(B), store(C)
    h.dgemm_device(layout, ta, tb, m, n, k, -0.5, sA, sA.shape[1], sB, sB.shape[1], 2.0, sC, sC.shape[1])
    h.sync()
    assert torch.equal(sC if layout == 101 else sC.t(), want)
    h.close()


@pytest.mark.parametrize("side,m,n,data", [(LEFT, 600, 230000, "uniform"), (RIGHT, 230000, 600, "normal"),
                                           (LEFT, 20000, 300, "wide")])
def test_panels_and_passes(built, side, m, n, data):
    """Products whose residues exceed the route's scratch: panels of the
    dimension without the triangle (the first two), passes over the moduli (the
    last), in place; sampled columns or rows against the double-double oracle."""
    h = u.Handle()
    try:
        A, lda, B, ldb = operands(side, LOWER, m, n, data)
        hB = B.cpu().numpy().ravel()
        h.dtrmm_device(COL, side, LOWER, NOTRANS, NONUNIT, m, n, 1.0, A, lda, B, ldb)
        h.sync()
        hA, got = A.cpu().numpy().ravel(), B.cpu().numpy()
        del A, B
        lines = n if side == LEFT else m
        for j in (0, lines // 2 + 1, lines - 1):
            if side == LEFT:
                want = orc.dtrmm_dd(COL, side, LOWER, NOTRANS, NONUNIT, m, n, 1.0, hA, lda, hB, ldb,
                                    cols=(j, j + 1))[:, 0]
                have = got[j]
            else:
                want = orc.dtrmm_dd(COL, side, LOWER, NOTRANS, NONUNIT, m, n, 1.0, hA, lda, hB, ldb,
                                    rows=(j, j + 1))[0, :]
                have = got[:, j]
            assert np.array_equal(have, want), (j, np.max(np.abs(have - want)))
    finally:
        h.close()


@pytest.mark.parametrize("data", ["uniform", "wide"])
@pytest.mark.parametrize("side,uplo,trans,diag", [(LEFT, LOWER, NOTRANS, UNIT), (LEFT, LOWER, TRANS, NONUNIT),
                                                  (RIGHT, UPPER, NOTRANS, UNIT), (RIGHT, LOWER, NOTRANS, NONUNIT)])
def test_scales_and_residues_in_one_launch(built, side, uplo, trans, diag, data):
    """The lossless route's sizes whose operands lie in shared memory (an order
    of 512 and 152 blocks of eight rows and columns at most, the third size)
    and the next ones up, against the double-double oracle; then a NaN."""
    h = u.Handle()
    try:
        for ka, vecs in ((300, 300), (449, 513), (512, 704), (512, 712), (513, 600)):
            m, n = (ka, vecs) if side == LEFT else (vecs, ka)
            A, lda, B, ldb = operands(side, uplo, m, n, data, pad=3)
            got = run(h, side, uplo, trans, diag, m, n, 1.0, A, lda, B, ldb, in_place=False)
            hA, hB = A.cpu().numpy().ravel(), B.cpu().numpy().ravel()
            for j in (0, vecs // 2 + 1, vecs - 1):
                if side == LEFT:
                    want = orc.dtrmm_dd(COL, side, uplo, trans, diag, m, n, 1.0, hA, lda, hB, ldb, cols=(j, j + 1))[:, 0]
                    have = got[j, :m]
                else:
                    want = orc.dtrmm_dd(COL, side, uplo, trans, diag, m, n, 1.0, hA, lda, hB, ldb, rows=(j, j + 1))[0, :]
                    have = got[:, j]
                assert np.array_equal(have, want), (m, n, j, np.max(np.abs(have - want)))
            B[n - 1, m - 1] = float("nan")
            got = run(h, side, uplo, trans, diag, m, n, 1.0, A, lda, B, ldb, in_place=True)
            assert np.isnan(got[n - 1, :m]).any() if side == LEFT else np.isnan(got[:, m - 1]).any()
            assert np.isfinite(got[:n - 1, :m - 1]).all()
    finally:
        h.close()


@pytest.mark.parametrize("moduli", [0, 2, 20])
@pytest.mark.parametrize("side,uplo,trans,diag", [(LEFT, LOWER, NOTRANS, UNIT), (LEFT, UPPER, NOTRANS, NONUNIT),
                                                  (RIGHT, LOWER, TRANS, NONUNIT), (RIGHT, UPPER, TRANS, UNIT)])
def test_emulated_tier_in_one_launch_equals_two(built, side, uplo, trans, diag, moduli):
    """The emulated tier's small sizes: bit by bit what the scaling and slicing
    kernels give (which run when stage times are taken)."""
    one, two = u.Handle(), u.Handle()
    try:
        two.set_option("stage_timing", 1)
        for ka, vecs in ((1, 1), (7, 9), (8, 8), (65, 255), (257, 300), (512, 704), (513, 703), (700, 450), (1024, 8)):
            m, n = (ka, vecs) if side == LEFT else (vecs, ka)
            A, lda, B, ldb = operands(side, uplo, m, n, "wide", pad=1)
            B[0, :m] = 0.0
            got, want = B.clone(), B.clone()
            one.ozaki_device(COL, side, uplo, trans, diag, m, n, 1.5, A, lda, got, ldb, moduli=moduli)
            two.ozaki_device(COL, side, uplo, trans, diag, m, n, 1.5, A, lda, want, ldb, moduli=moduli)
            one.sync()
            two.sync()
            assert np.array_equal(got.cpu().numpy(), want.cpu().numpy()), (m, n)
    finally:
        one.close()
        two.close()


@pytest.mark.parametrize("vecs", [262140, 262141, 262144, 262145])
def test_small_products_at_the_grid_limit(built, vecs):
    """As many vectors as the small kernel's grid holds, and more, in place."""
    h = u.Handle()
    try:
        A, lda, B, ldb = operands(LEFT, LOWER, 1, vecs, "uniform")
        want = (A.cpu().numpy() * B.cpu().numpy())[:, :1]
        got = run(h, LEFT, LOWER, NOTRANS, NONUNIT, 1, vecs, 1.0, A, lda, B, ldb, in_place=True)
        assert np.array_equal(got[:, :1], want)
    finally:
        h.close()


@pytest.mark.parametrize("side,m,n", [(LEFT, 600, 230000), (RIGHT, 230000, 600)])
def test_panels_left_to_the_fp64_kernel_in_place(built, side, m, n):
    """In place and with a NaN, the route's kernels copy each panel of B for the
    FP64 kernel behind them: its results are those of a pinned handle."""
    import torch
    h, pinned = u.Handle(), u.Handle()
    try:
        pinned.set_option("engine", u.ENGINE_DFMA)
        A, lda, B, ldb = operands(side, LOWER, m, n, "uniform", pad=1)
        B[n - 2, m - 3] = float("nan")
        out = []
        for hh in (h, pinned):
            C = B.clone()
            hh.dtrmm_device(COL, side, LOWER, NOTRANS, NONUNIT, m, n, 1.0, A, lda, C, ldb)
            hh.sync()
            out.append(C)
        got, want = out
        fine = torch.isfinite(want)
        assert fine.sum() > 0.99 * m * n
        assert torch.equal(got[fine], want[fine])
    finally:
        h.close()
        pinned.close()
