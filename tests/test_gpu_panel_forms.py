"""Where a rule of the panel, the triangular solves, the small GEMM tiles, the
residual pass or the generator changes form: both sides of each line and ragged
remainders, against the launch-per-step panel, LAPACK or the oracle."""
import numpy as np
import pytest

from gpu_util import from_dev

pytestmark = pytest.mark.gpu
EPS = 2.0 ** -53


def _panel(hlib, oracle, n, jb, nbmin, rfact, kind, zero_col=None):
    import torch

    from rochpl_b200.hpl import Algo
    from rochpl_b200.lib import LEAF_AUTO

    ld = oracle.default_ld(n)
    dA = torch.empty(ld * jb, dtype=torch.float64, device="cuda")
    hlib.matgen_block(n, n, 0, 0, n, jb, 7, dA.data_ptr(), ld)
    if zero_col is not None:
        dA.view(jb, ld)[zero_col].zero_()
    piv = torch.zeros(jb, dtype=torch.int32, device="cuda")
    try:
        hlib.set_leaf(kind)
        info = hlib.panel_factor(Algo(jb, nbmin, 2, 2, rfact, 1, 0).c(), n, 0, jb, dA.data_ptr(),
                                 ld, 0, piv.data_ptr())
    finally:
        hlib.set_leaf(LEAF_AUTO)
    return dA.view(jb, ld)[:, :n].clone(), piv, info


# Rows a cluster holds with 1, 2 and 3 rows of 32 columns per thread, 4 and 6 of
# 16, 8 of 8, and none; CTA counts below 16; leaves of every width in a panel.
@pytest.mark.parametrize("n,jb,nbmin,rfact", [
    (40, 40, 32, 2), (65, 64, 8, 2), (129, 96, 16, 1), (1025, 100, 32, 0), (4096, 64, 32, 2),
    (4097, 70, 16, 2), (8192, 256, 32, 2), (8193, 33, 32, 2), (12288, 64, 32, 1),
    (12289, 64, 32, 2), (16384, 48, 32, 2), (16385, 64, 32, 0), (24576, 32, 32, 2),
    (24577, 72, 32, 2), (32768, 40, 16, 2), (32769, 40, 32, 2)])
def test_panel_forms_match_the_launch_per_step_panel(hlib, oracle, n, jb, nbmin, rfact):
    """The cluster panel against the panel of one launch per step: identical
    pivots; identical bits where the leaves are not split (rows <= 12288), else
    every entry within its summation error (jb products of |l| <= 1 and u)."""
    from rochpl_b200.lib import LEAF_AUTO, LEAF_REGISTERS

    a, pa, ia = _panel(hlib, oracle, n, jb, nbmin, rfact, LEAF_AUTO)
    b, pb, ib = _panel(hlib, oracle, n, jb, nbmin, rfact, LEAF_REGISTERS)
    assert ia == ib == 0 and pa.tolist() == pb.tolist()
    if n <= 12288:
        assert bool((a == b).all())
    else:
        umax = float(b[:, :jb].abs().max())
        # Backward error of both orders, carried through the jb x jb unit-lower
        # solve of a panel whose multipliers partial pivoting keeps below 1.
        assert float((a - b).abs().max()) <= 64 * jb * jb * EPS * max(umax, 1.0)


def _scaled(n, cols, shifts, seed):
    """Random entries times powers of two from `shifts`, an exponent per row."""
    rng = np.random.default_rng(seed)
    A = rng.random((n, cols)) - 0.5
    return np.ldexp(A, rng.choice(shifts, size=n)[:, None])


@pytest.mark.parametrize("shifts", [
    [-400, -399, -398], [-402, -401, -400, -399], [498, 499, 500], [499, 500, 501, 502],
    [-401, 0, 499], [-1050, -1022, -900, 0], [-700, 0, 700]])
def test_panel_quotients_at_the_exponent_limits(hlib, oracle, shifts):
    """Multipliers by reciprocal and correction are exact only between 2^-400 and
    2^500; the rest divide: the bits of the panel that always divides (in global
    memory: the one across the GPU's registers underflows to +0 whatever the sign)."""
    import torch

    from rochpl_b200.hpl import Algo
    from rochpl_b200.lib import LEAF_AUTO, LEAF_GLOBAL

    for n, jb in ((300, 64), (5000, 40)):
        ld = oracle.default_ld(n)
        A = torch.zeros((jb, ld), dtype=torch.float64, device="cuda")
        A[:, :n] = torch.from_numpy(np.ascontiguousarray(_scaled(n, jb, shifts, n).T))
        out = []
        for kind in (LEAF_AUTO, LEAF_GLOBAL):
            B, piv = A.clone(), torch.zeros(jb, dtype=torch.int32, device="cuda")
            try:
                hlib.set_leaf(kind)
                hlib.panel_factor(Algo(jb, 32, 2, 2, 2, 1, 0).c(), n, 0, jb, B.data_ptr(), ld, 0,
                                  piv.data_ptr())
            finally:
                hlib.set_leaf(LEAF_AUTO)
            out.append((B.view(torch.int64), piv))
        assert torch.equal(out[0][1], out[1][1])
        assert torch.equal(out[0][0], out[1][0])


@pytest.mark.parametrize("shifts", [[-62, -61, -60, -59], [57, 58, 59, 60], [-61, 0, 59]])
def test_fp32_panel_quotients_at_the_exponent_limits(hlib, shifts):
    """The same for the mixed form's FP32 panels (2^-60 to 2^60), by its pivots and
    solution."""
    import torch

    from rochpl_b200.hpl import Algo
    from rochpl_b200.lib import LEAF_AUTO, LEAF_GLOBAL, PREC_FP16X3

    n = 400
    A = torch.from_numpy(np.ascontiguousarray(_scaled(n, n + 1, shifts, 5).T)).cuda()
    out = []
    for kind in (LEAF_AUTO, LEAF_GLOBAL):
        x = torch.zeros(n, dtype=torch.float64, device="cuda")
        piv = torch.zeros(n, dtype=torch.int32, device="cuda")
        try:
            hlib.set_leaf(kind)
            hlib.pdgesv_mixed(Algo(64, 32, 2, 2, 2, 1, 0).c(), n, x.data_ptr(), A=A.data_ptr(), ld=n,
                              precision=PREC_FP16X3, ipiv=piv.data_ptr(), max_outer=1)
        finally:
            hlib.set_leaf(LEAF_AUTO)
        out.append((piv, x.view(torch.int64)))
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])


def test_panel_zero_pivot(hlib, oracle):
    from rochpl_b200.lib import LEAF_AUTO

    for n in (100, 5000, 13000):
        assert _panel(hlib, oracle, n, 64, 32, 2, LEAF_AUTO, zero_col=37)[2] == 38


def _unit_lower(hlib, oracle, jb):
    """The factored LCG panel of 2048 rows and its unit-lower block."""
    import torch

    from rochpl_b200.hpl import Algo

    n = 2048
    ld = oracle.default_ld(n)
    W = torch.zeros((2 * jb, ld), dtype=torch.float64, device="cuda")
    hlib.matgen_block(n, n, 0, 0, n, jb, 7, W.data_ptr(), ld)
    piv = torch.zeros(jb, dtype=torch.int32, device="cuda")
    assert hlib.panel_factor(Algo(jb, min(32, jb), 2, 2, 2, 1, 0).c(), n, 0, jb, W.data_ptr(),
                             ld, 0, piv.data_ptr()) == 0
    return n, ld, W, np.tril(W[:jb, :jb].cpu().numpy().T, -1) + np.eye(jb)


def _residual(L, X):
    """|L X - I| in the Frobenius norm; X has L's shape."""
    assert np.array_equal(np.triu(X, 1), np.zeros_like(X))
    wide = np.float64 if X.dtype == np.float32 else np.longdouble
    return float(np.linalg.norm((L.astype(wide) @ X.astype(wide) - np.eye(len(L))).astype(float)))


# L11^-1 leaves no larger a residual L X - I, which is what U12 = L11^-1 A12 sees,
# than the blocked substitution on the identity.  Both are norms of jb^2 / 2
# rounding errors of the same size, so they agree closely; doubling without a
# correction is at 1.5 times at jb = 128 and 5 at 512.
SLACK = 1.25


@pytest.mark.parametrize("jb", [33, 64, 65, 128, 200, 255, 257, 400, 512, 513])
def test_unit_lower_inverse_residual(hlib, oracle, jb):
    """hplb_panel_update on the identity against hplb_laswp_trsm on it."""
    import torch

    n, ld, W, L = _unit_lower(hlib, oracle, jb)
    eye = torch.eye(jb, dtype=torch.float64, device="cuda")
    X = torch.zeros((jb, ld), dtype=torch.float64, device="cuda")
    X[:, :jb] = eye
    W[jb:, :jb] = eye
    own = torch.arange(jb, dtype=torch.int32, device="cuda")  # no interchanges
    hlib.panel_update(n, 0, jb, W.data_ptr(), ld, own.data_ptr(), X.data_ptr(), ld, 0, jb)
    hlib.laswp_trsm(W.data_ptr(), ld, 0, jb, 0, range(jb), jb, jb)
    new, sub = (_residual(L, T[:, :jb].cpu().numpy().T) for T in (X, W[jb:]))
    assert new <= SLACK * sub, (new / EPS, sub / EPS)
    assert torch.equal(X[:, :jb], W[jb:, :jb])  # substitution as well, in the same order


@pytest.mark.parametrize("jb", [96, 256, 300, 512, 600])
def test_unit_lower_inverse_residual_fp32(hlib, oracle, jb):
    """The mixed form's FP32 inverse, called by its C++ symbol, against the
    substitution in FP32 on the host."""
    import ctypes

    import torch

    _, _, _, L = _unit_lower(hlib, oracle, jb)
    L = L.astype(np.float32)
    dL = torch.from_numpy(np.ascontiguousarray(L.T)).cuda()
    dinv = torch.zeros((jb // 32 + 1) * 1024, dtype=torch.float32, device="cuda")
    X = torch.full((jb, jb), np.nan, dtype=torch.float32, device="cuda")
    P, q, i = ctypes.c_void_p, ctypes.c_int64, ctypes.c_int
    sym = "_ZN4hplb{}IfEE9cudaError{}P11CUstream_st"
    diag = getattr(hlib.L, sym.format("15launch_diag_inv", "PKT_liiiPS2_"))
    diag.argtypes = [P, q, i, i, i, P, P]
    inv = getattr(hlib.L, sym.format("25launch_unit_lower_inverse", "PKT_liS4_PS2_l") + "Pi")
    inv.argtypes = [P, q, i, P, P, q, P, P]
    torch.cuda.synchronize()
    assert diag(dL.data_ptr(), jb, 0, 0, jb, dinv.data_ptr(), None) == 0
    assert inv(dL.data_ptr(), jb, jb, dinv.data_ptr(), X.data_ptr(), jb, None,
               ctypes.byref(i(0))) == 0
    torch.cuda.synchronize()
    ref = np.eye(jb, dtype=np.float32)
    for b in range(0, jb, 32):  # 32 rows by their block's inverse, as on the GPU
        e = min(b + 32, jb)
        D = np.eye(e - b, dtype=np.float32)
        for r in range(1, e - b):
            D[r] -= L[b + r, b:b + r] @ D[:r]
        ref[b:e] = D @ (ref[b:e] - L[b:e, :b] @ ref[:b])
    new, sub = _residual(L, X.cpu().numpy().T), _residual(L, ref)
    assert new <= SLACK * sub, (new * 2 ** 24, sub * 2 ** 24)


@pytest.mark.parametrize("n,nb,nrhs", [(1, 1, 1), (63, 64, 7), (64, 64, 8), (65, 64, 9),
                                       (130, 65, 33), (200, 200, 31), (257, 48, 40),
                                       (300, 33, 128), (300, 64, 129)])
@pytest.mark.parametrize("trans", [0, 1])
def test_getrs_block_edges(hlib, oracle, n, nb, nrhs, trans):
    import torch

    from rochpl_b200.hpl import Algo

    M = oracle.matgen(n, n + nrhs, 11)
    A, B = np.array(M[:n, :n]), np.array(M[:n, n:])
    LU = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
    X = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")
    nbe = min(nb, n)
    assert hlib.getrf(Algo(nbe, min(16, nbe), 2, 2, 2, 1, 0).c(), n, LU.data_ptr(), n,
                      piv.data_ptr()) == 0
    hlib.getrs(trans, n, nbe, nrhs, LU.data_ptr(), n, piv.data_ptr(), X.data_ptr(), n)
    ref = np.linalg.solve(A.T if trans else A, B)
    tol = 64 * n * EPS * np.linalg.cond(A, np.inf)
    err = np.max(np.abs(X.cpu().numpy().T - ref)) / np.max(np.abs(ref))
    assert err <= tol, (err, tol)


@pytest.mark.parametrize("nrhs", [2, 8, 9, 130])
@pytest.mark.parametrize("n", [1, 15, 16, 17, 31, 32, 33, 48, 63, 64, 65, 97, 161])
def test_trsm_upper_block_edges(hlib, n, nrhs):
    """Diagonal blocks of 64 are inverted in two halves of 32, ragged ones to their
    own size: U X = B with |U X - B| within n + 64 roundings of |U| |U^-1| |U| |X|
    (a sum of n products, and one of 64 with a block's inverse, whose own error is
    a sum of 64 more)."""
    import torch

    rng = np.random.default_rng(100 * n + nrhs)
    ld = n + n % 2
    U = np.triu(rng.random((n, n)) - 0.5) + 2.0 * np.eye(n)
    B = rng.random((n, nrhs)) - 0.5
    dU = torch.full((n, ld), np.nan, dtype=torch.float64, device="cuda")
    low = rng.random((n, n))  # what stands below the diagonal is not U's
    dU[:, :n] = torch.from_numpy(np.ascontiguousarray((U + np.tril(low, -1)).T))
    dB = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
    dX = torch.full_like(dB, np.nan)
    hlib.trsm_upper(n, nrhs, dU.data_ptr(), ld, dB.data_ptr(), n, dX.data_ptr(), n)
    X = dX.cpu().numpy().T
    A = np.abs(U)
    bound = 2 * (n + 64) * EPS * (A @ np.abs(np.linalg.inv(U)) @ A @ np.abs(X))
    assert np.all(np.abs(U @ X - B) <= bound)


@pytest.mark.parametrize("n,nb", [(200, 64), (400, 128)])
def test_transposed_getrs_residual_of_the_block_solve(hlib, oracle, n, nb):
    """|A^T x - b| of random systems against LAPACK's, in the geometric mean over 24 of
    them.  With unit-lower blocks applied as two inverses of 32 rows, as the blocked
    substitution does, 1.15 and 1.11 times LAPACK's; with one inverse of 64 rows 1.40
    and 1.28.  The logarithms spread by about 0.3 (0.06 in the mean)."""
    import torch

    from rochpl_b200.hpl import Algo

    logs = []
    for seed in range(24):
        g = np.random.default_rng(seed)
        A, B = g.random((n, n)) - 0.5, g.random((n, 3)) - 0.5
        LU = torch.from_numpy(np.ascontiguousarray(A.T)).cuda()
        X = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
        piv = torch.zeros(n, dtype=torch.int32, device="cuda")
        assert hlib.getrf(Algo(nb, 32, 2, 2, 2, 1, 0).c(), n, LU.data_ptr(), n,
                          piv.data_ptr()) == 0
        hlib.getrs(1, n, nb, 3, LU.data_ptr(), n, piv.data_ptr(), X.data_ptr(), n)
        M, ml = A.T, A.T.astype(np.longdouble)
        ours, ref = (np.linalg.norm((ml @ x - B).astype(float)) / np.linalg.norm(x)
                     for x in (X.cpu().numpy().T, np.linalg.solve(M, B)))
        logs.append(np.log(ours / ref))
    assert np.exp(np.mean(logs)) <= 1.25


@pytest.mark.parametrize("n,row", [(40, 7), (64, 33), (100, 70), (200, 90)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_trsm_upper_non_finite_rows(hlib, n, row, bad):
    """An infinity or NaN in y reaches the rows above its own and its own column;
    the rows below, and the other right-hand sides, are what they are without it, to
    a sum of n products in another order."""
    import torch

    rng = np.random.default_rng(n)
    U = np.triu(rng.random((n, n)) - 0.5) + 2.0 * np.eye(n)
    B = rng.random((n, 8)) - 0.5
    dU = torch.from_numpy(np.ascontiguousarray(U.T)).cuda()
    out = []
    for y in (None, bad):
        dX = torch.from_numpy(np.ascontiguousarray(B.T)).cuda()
        if y is not None:
            dX[3, row] = y
        hlib.trsm_upper(n, 8, dU.data_ptr(), n, dX.data_ptr(), n, dX.data_ptr(), n)
        out.append(dX.cpu().numpy().T)
    clean, got = out
    assert not np.any(np.isfinite(got[: row + 1, 3]))
    got[: row + 1, 3] = clean[: row + 1, 3]
    bound = 2 * (n + 64) * EPS * (np.abs(np.linalg.inv(U)) @ np.abs(U) @ np.abs(clean))
    assert np.all(np.abs(got - clean) <= bound)


@pytest.mark.parametrize("trans", [0, 1])
def test_getrs_launches_do_not_grow_with_right_hand_sides(hlib, oracle, trans):
    """Up to 128 right-hand sides a triangular solve is one launch: a chain of row
    blocks per 32 of them in turn made 64 take 1.5 to 1.8 times as long."""
    import torch

    from rochpl_b200.hpl import Algo

    n, nb = 300, 64
    M = oracle.matgen(n, n + 128, 11)
    LU = torch.from_numpy(np.ascontiguousarray(M[:n, :n].T)).cuda()
    piv = torch.zeros(n, dtype=torch.int32, device="cuda")
    hlib.getrf(Algo(nb, 16, 2, 2, 2, 1, 0).c(), n, LU.data_ptr(), n, piv.data_ptr())
    launches, cols = [], []
    for nrhs in (8, 33, 64, 128):
        X = torch.from_numpy(np.ascontiguousarray(M[:n, n:n + nrhs].T)).cuda()
        hlib.getrs(trans, n, nb, nrhs, LU.data_ptr(), n, piv.data_ptr(), X.data_ptr(), n)
        launches.append(hlib.last_timing()["kernel_launches"])
        cols.append(X[:8].clone())
    assert len(set(launches)) == 1, launches
    assert all(torch.equal(c, cols[0]) for c in cols)  # a group's sums are its own


@pytest.mark.parametrize("n", [1, 255, 257, 512, 2047, 2049])
def test_residual_pass_edges(hlib, oracle, n):
    """One read of the stored matrix: the regenerated check's bits, the oracle's
    norms."""
    import torch

    ld = oracle.default_ld(n)
    dA = torch.empty(ld * (n + 1), dtype=torch.float64, device="cuda")
    hlib.matgen(n, n + 1, 100, dA.data_ptr(), ld)
    x = (np.arange(n) % 7 - 3.0) / 5
    dX = torch.from_numpy(x).cuda()
    d1 = hlib.residual(n, dA.data_ptr(), ld, dX.data_ptr())
    d2 = hlib.residual_lcg(n, 100, dX.data_ptr())
    o = oracle.residual(oracle.matgen(n, n + 1, 100, ld=ld), n, x)
    assert d1 == d2
    for k in ("rnorm_inf", "anorm_1", "anorm_inf", "xnorm_1", "bnorm_inf"):
        assert d1[k] == pytest.approx(o[k], rel=4 * n * EPS, abs=1e-300), k


def test_residual_in_bands(hlib):
    """A stored matrix of more than 102400 rows is read in bands of rows (84 GB: its
    check against the regenerated one's bits)."""
    import torch

    n = 102657  # 402 row groups: six bands of 67, the last group of one row
    ld = n + (-n) % 32
    if torch.cuda.mem_get_info()[0] < 8 * ld * (n + 1) + (1 << 31):
        pytest.skip("needs 86 GB of device memory")
    dA = torch.empty(ld * (n + 1), dtype=torch.float64, device="cuda")
    hlib.matgen(n, n + 1, 100, dA.data_ptr(), ld)
    dX = (torch.arange(n, device="cuda") % 7 - 3.0).double() / 5
    d1 = hlib.residual(n, dA.data_ptr(), ld, dX.data_ptr())
    assert d1 == hlib.residual_lcg(n, 100, dX.data_ptr())
    del dA
    torch.cuda.empty_cache()


def test_matgen_long_runs(hlib, oracle):
    """Tall matrices take 64-row runs; the last run of a column is ragged."""
    import torch

    m, n = 5001, 3400
    ld = oracle.default_ld(m)
    dA = torch.full((ld * n,), np.nan, dtype=torch.float64, device="cuda")
    hlib.matgen(m, n, 3, dA.data_ptr(), ld)
    got = from_dev(dA, ld, n)
    assert np.array_equal(got[:m].view(np.uint64), oracle.matgen(m, n, 3, ld=ld)[:m].view(np.uint64))
    assert np.all(np.isnan(got[m:]))


@pytest.mark.parametrize("m,n,k", [(1400, 1250, 40), (1408, 1536, 96), (129, 63, 17)])
def test_dgemm_tiles_agree(hlib, m, n, k):
    """Tiles of 128 and of 64 sum in the same order: a product of many tiles and
    the same product by blocks small enough for the small ones, bit for bit."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(m + n + k)
    rnd = lambda *s: torch.rand(*s, generator=g, dtype=torch.float64, device="cuda") - 0.5
    ld, k2 = m + 32 - m % 32, k + k % 2
    A, B, C0 = rnd(k, ld), rnd(n, k2), rnd(n, ld)
    whole, parts = C0.clone(), C0.clone()
    hlib.dgemm_sub(m, n, k, A.data_ptr(), ld, B.data_ptr(), k2, whole.data_ptr(), ld)
    for c in range(0, n, 128):
        w = min(128, n - c)
        hlib.dgemm_sub(m, w, k, A.data_ptr(), ld, B.data_ptr() + 8 * c * k2, k2,
                       parts.data_ptr() + 8 * c * ld, ld)
    assert torch.equal(whole, parts)
    ref = C0[:, :m] - B[:, :k] @ A[:, :m]
    assert float((whole[:, :m] - ref).abs().max()) <= 2 * k * EPS * (1 + 0.25 * k)
    assert torch.equal(whole[:, m:], C0[:, m:])


@pytest.mark.parametrize("n,nb", [(4500, 256), (17000, 512), (25000, 512)])
def test_mixed_tall_panels(hlib, n, nb):
    """FP32 panels of 2, 4, 6 and 8 rows per thread."""
    import torch

    from rochpl_b200.hpl import Algo
    from rochpl_b200.lib import PREC_FP16X3

    x = torch.zeros(n, dtype=torch.float64, device="cuda")
    r = hlib.pdgesv_mixed(Algo(nb, 32, 2, 2, 2, 1, 0).c(), n, x.data_ptr(), seed=5,
                          precision=PREC_FP16X3)
    assert r["converged"] == 1 and r["gmres_iters"] <= 10
    assert hlib.residual_lcg(n, 5, x.data_ptr())["resid"] < 16.0


@pytest.mark.parametrize("trans", [0, 1])
def test_batch_getrs_with_recursive_factors(hlib, trans):
    """Stored factors of a recursive plan: LAPACK's, whatever made them."""
    import torch

    from rochpl_b200.batch import BatchPlan
    from rochpl_b200.lib import HPLB_BATCH_RECURSIVE

    sizes, nrhs = np.array([33, 64, 97, 250], dtype=np.int32), 5
    plan = BatchPlan(hlib, sizes, nrhs, [HPLB_BATCH_RECURSIVE] * 6)
    g = torch.Generator(device="cuda").manual_seed(3)
    rnd = lambda k: torch.rand(k, generator=g, dtype=torch.float64, device="cuda") - 0.5
    A0, B0 = rnd(plan.a_elems), rnd(plan.b_elems)
    A, B = A0.clone(), B0.clone()
    P = torch.zeros(plan.p_elems, dtype=torch.int32, device="cuda")
    info = torch.zeros(plan.count, dtype=torch.int32, device="cuda")
    plan.gesv(A.data_ptr(), B.data_ptr(), P.data_ptr(), info.data_ptr())
    X = B0.clone()
    plan.getrs(trans, A.data_ptr(), P.data_ptr(), X.data_ptr())
    for n, a, b in zip(map(int, sizes), plan.a_off, plan.b_off):
        M = A0[a:a + n * n].view(n, n).t().cpu().numpy()
        R = B0[b:b + n * nrhs].view(nrhs, n).t().cpu().numpy()
        ref = np.linalg.solve(M.T if trans else M, R)
        got = X[b:b + n * nrhs].view(nrhs, n).t().cpu().numpy()
        tol = 64 * n * EPS * np.linalg.cond(M, np.inf)
        assert np.max(np.abs(got - ref)) / np.max(np.abs(ref)) <= tol
    plan.close()
