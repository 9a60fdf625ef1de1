"""The FP64 tensor-core forms of the factorization, the solves and the batched kernel at the
sizes where they can go wrong: edges of the 8-, 16-, 64- and 128-wide tiles, odd leading
dimensions and bases that are only 8-byte aligned, failed pivots on both sides of every tile
edge, and the FP32 tile products with and without TMA.

Bounds: a Cholesky factor satisfies |A - L L^T| <= (n + 1) u |L||L^T| entrywise (Higham,
Accuracy and Stability, theorem 10.3); the products here sum in blocks and by reciprocal pivots
and inverted tiles, each an operation or two more per step, hence the factor 4."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = {"s": float(np.finfo(np.float32).eps), "d": float(np.finfo(np.float64).eps)}
NP = {"s": np.float32, "d": np.float64}


def _torch():
    import torch

    return torch


def spd(n, seed):
    g = np.random.default_rng(seed).standard_normal((n, n))
    return g @ g.T / max(n, 1) + np.eye(n)


def device(host, lda, p, shift=0):
    """Column-major copy with leading dimension lda, its first word `shift` words into the allocation."""
    torch = _torch()
    n, m = host.shape
    flat = np.full(shift + lda * m, np.nan, dtype=NP[p])
    flat[shift:].reshape(m, lda)[:, :n] = host.T
    t = torch.from_numpy(flat).cuda()
    return t, t.data_ptr() + shift * t.element_size()


def host(t, n, m, lda, shift=0):
    return t.cpu().numpy()[shift:].reshape(m, lda)[:, :n].T


def potrf(handle, p, uplo, n, ptr, lda):
    torch = _torch()
    from libddla_b200 import ddla

    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ddla.potrf(handle, p, uplo, n, ptr, lda, info.data_ptr())
    handle.synchronize()
    return int(info[0])


def check_factor(a, out, uplo, p):
    n = a.shape[0]
    low = np.tril(out) if uplo == "L" else np.triu(out).T
    low = low.astype(np.float64)
    bound = 4 * (n + 1) * EPS[p] * (np.abs(low) @ np.abs(low.T)) + np.abs(a) * EPS[p]
    i = np.tril_indices(n)
    diff = np.abs(a - low @ low.T)
    assert np.all(diff[i] <= bound[i]), np.max(diff[i] / bound[i])


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("n", [1, 7, 8, 9, 16, 17, 127, 128, 129, 136, 193, 257, 700])
def test_factor_tile_edges(handle, p, uplo, n):
    a = spd(n, n).astype(NP[p]).astype(np.float64)
    for pad, shift in ((0, 0), (1, 0), (2, 1), (5, 3)):
        poisoned = a.copy()
        poisoned[np.triu_indices(n, 1) if uplo == "L" else np.tril_indices(n, -1)] = np.nan
        t, ptr = device(poisoned, n + pad, p, shift)
        assert potrf(handle, p, uplo, n, ptr, n + pad) == 0
        out = host(t, n, n, n + pad, shift)
        other = np.triu_indices(n, 1) if uplo == "L" else np.tril_indices(n, -1)
        assert np.all(np.isnan(out[other]))
        check_factor(a, out, uplo, p)


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("group,n,pad", [(2, 1500, 0), (2, 1501, 0), (4, 1500, 0), (4, 1499, 0), (8, 1500, 2), (8, 1501, 0),
                                         (1, 2433, 0), (2, 2433, 0), (1, 2432, 0), (4, 2433, 0)])
def test_super_steps(handle, p, uplo, group, n, pad):
    """Updates with K up to 1024 (several turns of the stage ring), look-ahead and left-looking regions,
    and regions of 148 or more 128 x 128 tiles (from n - 128 (1 + group) = 2049), all with and without
    TMA.  Bound as check_factor's."""
    torch = _torch()
    from libddla_b200.ddla import _c_api as C

    g = torch.randn(n, n, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(n))
    a = (g @ g.T / n + torch.eye(n, device="cuda", dtype=torch.float64)).cpu().numpy().astype(NP[p]).astype(np.float64)
    a = np.tril(a) + np.tril(a, -1).T
    lda = n + pad
    t, ptr = device(a, lda, p)
    f = C.lib.ddlak_potrf_grouped
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_char, ctypes.c_char, ctypes.c_int, ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong,
                  ctypes.c_void_p, ctypes.c_void_p]
    info = torch.full((1,), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    assert f(p.encode(), uplo.encode(), group, n, ptr, lda, info.data_ptr(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert int(info[0]) == 0
    out = t.view(n, lda)[:, :n].T
    low = (torch.tril(out) if uplo == "L" else torch.triu(out).T).double()
    am = torch.from_numpy(a).cuda()
    bound = 4 * (n + 1) * EPS[p] * (low.abs() @ low.abs().T) + am.abs() * EPS[p]
    diff = torch.tril((am - low @ low.T).abs() - bound)
    assert float(diff.max()) <= 0.0


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("bad", [0, 6, 7, 8, 63, 64, 127, 128, 199])
def test_failed_pivot(handle, p, uplo, bad):
    """info is the failed pivot's order and the columns before it are final."""
    n = 200
    a = spd(n, 3).astype(NP[p]).astype(np.float64)
    want = np.linalg.cholesky(a)
    b = a.copy()
    b[bad, bad] = -1.0
    t, ptr = device(b, n + 1, p)
    assert potrf(handle, p, uplo, n, ptr, n + 1) == bad + 1
    out = host(t, n, n, n + 1).astype(np.float64)
    low = np.tril(out) if uplo == "L" else np.triu(out).T
    # the block that fails is final in its own rows; the blocks before it in every row
    rows = n if bad % 128 == 0 else min(n, (bad // 128 + 1) * 128)
    got, ref = low[:rows, :bad], want[:rows, :bad]
    keep = np.tril_indices(rows, 0, bad)
    ok = ref.copy()
    # row `bad` differs only through the changed diagonal entry, which no earlier column holds
    assert np.allclose(got[keep], ok[keep], rtol=0, atol=50 * n * EPS[p])


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("n,nrhs", [(1, 1), (63, 8), (64, 9), (65, 16), (129, 17), (700, 3), (701, 33)])
def test_solve_edges(handle, p, uplo, side, n, nrhs):
    from libddla_b200 import ddla

    a = spd(n, 5).astype(NP[p]).astype(np.float64)
    rng = np.random.default_rng(7)
    b = rng.standard_normal((n, nrhs) if side == "L" else (nrhs, n)).astype(NP[p])
    ta, pa = device(a, n + 1, p)
    assert potrf(handle, p, uplo, n, pa, n + 1) == 0
    ldb = b.shape[0] + 2
    tb, pb = device(b, ldb, p)
    wrap = ddla.DistributedMatrix.wrap
    dA = wrap(handle, pa, n, n, n + 1, NP[p])
    dB = wrap(handle, pb, b.shape[0], b.shape[1], ldb, NP[p])
    ddla.ppotrs(dA, dB, uplo=uplo, side=side)
    x = host(tb, b.shape[0], b.shape[1], ldb).astype(np.float64)
    res = a @ x - b if side == "L" else x @ a - b
    # the factor's backward error and that of the two triangular solves, condition number about 5
    assert np.max(np.abs(res)) <= 40 * (n + 1) * EPS[p] * np.linalg.norm(a, 2) * np.max(np.abs(x))


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo,side", [("L", "L"), ("U", "R")])
@pytest.mark.parametrize("n,nrhs", [(2240, 33), (2497, 40)])
def test_solve_many_blocks(handle, p, uplo, side, n, nrhs):
    """Block rows with more than 32 others before them, a last chunk of one right-hand side."""
    from libddla_b200 import ddla

    a = spd(n, 21).astype(NP[p]).astype(np.float64)
    b = np.random.default_rng(8).standard_normal((n, nrhs) if side == "L" else (nrhs, n)).astype(NP[p])
    ta, pa = device(a, n, p)
    assert potrf(handle, p, uplo, n, pa, n) == 0
    tb, pb = device(b, b.shape[0] + 1, p)
    wrap = ddla.DistributedMatrix.wrap
    dA = wrap(handle, pa, n, n, n, NP[p])
    ddla.ppotrs(dA, wrap(handle, pb, b.shape[0], b.shape[1], b.shape[0] + 1, NP[p]), uplo=uplo, side=side)
    x = host(tb, b.shape[0], b.shape[1], b.shape[0] + 1).astype(np.float64)
    res = a @ x - b if side == "L" else x @ a - b
    # as test_solve_edges
    assert np.max(np.abs(res)) <= 40 * (n + 1) * EPS[p] * np.linalg.norm(a, 2) * np.max(np.abs(x))


@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("n,noise", [(64, 1e-12), (256, 1e-8), (256, 1e-12), (700, 1e-10)])
def test_solve_is_backward_stable(handle, uplo, side, n, noise):
    """Substitution solves with |b - L L^T x| <= 2 (n + 1) u |L||L^T||x| whatever the condition number
    (Higham, theorem 8.5 for each triangle), here up to 1e14; twice that for sums in blocks and
    inverted 8 x 8 tiles.  Inverting whole 64 x 64 diagonal blocks misses it a hundredfold."""
    from libddla_b200 import ddla

    x = np.sort(np.random.default_rng(n).random(n))
    a = np.exp(-((x[:, None] - x[None]) ** 2) / 0.18) + noise * np.eye(n)
    ta, pa = device(a, n + 1, "d")
    assert potrf(handle, "d", uplo, n, pa, n + 1) == 0
    f = host(ta, n, n, n + 1)
    low = (np.tril(f) if uplo == "L" else np.triu(f).T).astype(np.longdouble)
    rng = np.random.default_rng(13)
    b = rng.standard_normal((n, 5))
    b[:, 1] = a @ b[:, 1]
    tb, pb = device(b if side == "L" else b.T, n if side == "L" else 5, "d")
    wrap = ddla.DistributedMatrix.wrap
    dA = wrap(handle, pa, n, n, n + 1, np.float64)
    dB = wrap(handle, pb, n, 5, n, np.float64) if side == "L" else wrap(handle, pb, 5, n, 5, np.float64)
    ddla.ppotrs(dA, dB, uplo=uplo, side=side)
    got = host(tb, n, 5, n) if side == "L" else host(tb, 5, n, 5).T
    got = got.astype(np.longdouble)
    res = np.abs(low @ (low.T @ got) - b)
    bound = 2 * (n + 1) * EPS["d"] * (np.abs(low) @ (np.abs(low.T) @ np.abs(got)))
    assert np.all(res <= bound), float(np.max(res / bound))


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("value", [np.nan, np.inf])
@pytest.mark.parametrize("r,c", [(5, 2), (14, 3), (100, 50), (127, 126), (128, 5), (190, 63)])
def test_entries_that_are_not_finite_stay_behind_their_column(handle, p, uplo, value, r, c):
    """A NaN or infinite entry (r, c) fails the pivot of row r; what substitution computes before it,
    row r's columns before c among them, is what it is without the entry."""
    n = 200
    a = spd(n, 3).astype(NP[p]).astype(np.float64)
    want = np.linalg.cholesky(a)
    b = a.copy()
    b[r, c] = b[c, r] = value
    t, ptr = device(b, n + 1, p)
    assert potrf(handle, p, uplo, n, ptr, n + 1) == r + 1
    out = host(t, n, n, n + 1).astype(np.float64)
    low = np.tril(out) if uplo == "L" else np.triu(out).T
    tol = 50 * n * EPS[p]
    assert np.allclose(low[r, :c], want[r, :c], rtol=0, atol=tol)
    assert not np.isfinite(low[r, c])
    # the other rows of the blocks that were finished, and of the failed block
    rows = np.array([i for i in range(n if r >= 128 else 128) if i != r])
    cols = 128 if r >= 128 else r
    keep = rows[:, None] >= np.arange(cols)[None]
    assert np.allclose(low[rows][:, :cols][keep], want[rows][:, :cols][keep], rtol=0, atol=tol)


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("side", ["L", "R"])
@pytest.mark.parametrize("row", [0, 6, 33, 63, 64, 77, 129])
def test_forward_solve_leaves_the_rows_before_a_nan(handle, p, uplo, side, row):
    torch = _torch()
    from libddla_b200.ddla import _c_api as C

    n, nrhs = 130, 11
    a = spd(n, 4)
    low = np.linalg.cholesky(a).astype(NP[p])
    b = np.random.default_rng(row).standard_normal((n, nrhs)).astype(NP[p])
    want = np.linalg.solve(low.astype(np.float64), b.astype(np.float64))
    b[row, 9] = np.nan
    b[row, 2] = np.inf
    ta, pa = device(low if uplo == "L" else low.T, n + 1, p)
    tb, pb = device(b if side == "L" else b.T, n if side == "L" else nrhs, p)
    C.lib.ddlak_potrs_workspace.restype = ctypes.c_ulonglong
    work = torch.zeros(int(C.lib.ddlak_potrs_workspace(n, nrhs)), dtype=torch.uint8, device="cuda")
    f = C.lib.ddlak_forward_solve
    f.restype = ctypes.c_int
    f.argtypes = ([ctypes.c_char] * 3 + [ctypes.c_int] * 2 +
                  [ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p,
                   ctypes.c_ulonglong, ctypes.c_void_p])
    torch.cuda.synchronize()
    assert f(p.encode(), uplo.encode(), side.encode(), n, nrhs, pa, n + 1, pb, n if side == "L" else nrhs,
             work.data_ptr(), work.numel(), torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    x = host(tb, n, nrhs, n) if side == "L" else host(tb, nrhs, n, nrhs).T
    tol = 50 * n * EPS[p] * np.max(np.abs(want))
    whole = [k for k in range(nrhs) if k not in (2, 9)]
    assert np.allclose(x[:, whole], want[:, whole], rtol=0, atol=tol)
    assert np.allclose(x[:row, [2, 9]], want[:row, [2, 9]], rtol=0, atol=tol)
    assert not np.any(np.isfinite(x[row, [2, 9]]))


def batched_run(p, variant, mats, ldas, shifts, rhs):
    """ddlak_posv_vbatched with one variant for all: (factors, solutions, info, logdet); rhs None: no solve."""
    torch = _torch()
    from libddla_b200.ddla import _c_api as C

    up = lambda v, dt: torch.tensor(np.array(v, dtype=dt), device="cuda")  # noqa: E731
    count, orders = len(mats), [m.shape[0] for m in mats]
    ta = [device(m, lda, p, s) for m, lda, s in zip(mats, ldas, shifts)]
    tb = [device(b, b.shape[0], p) for b in rhs] if rhs is not None else []
    dn, dl, da = up(orders, np.int32), up(ldas, np.int32), up([x[1] for x in ta], np.int64)
    db = up([x[1] for x in tb], np.int64) if rhs is not None else None
    logdet = torch.zeros(count, dtype=torch.float64, device="cuda")
    info = torch.full((count,), -5, dtype=torch.int32, device="cuda")
    sel = torch.full((count,), variant, dtype=torch.uint8, device="cuda")
    counters = torch.zeros(2, dtype=torch.int32, device="cuda")
    f = C.lib.ddlak_posv_vbatched
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_char, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 9 + [ctypes.c_int, ctypes.c_void_p]
    torch.cuda.synchronize()
    rc = f(p.encode(), 512, count, dn.data_ptr(), da.data_ptr(), dl.data_ptr(), db.data_ptr() if db is not None else None,
           logdet.data_ptr(), info.data_ptr(), None, sel.data_ptr(), counters.data_ptr(), 7,
           torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    outs = [host(t, n, n, lda, s).astype(np.float64) for (t, _), n, lda, s in zip(ta, orders, ldas, shifts)]
    xs = [host(t, n, 1, n).astype(np.float64) for (t, _), n in zip(tb, orders)]
    return outs, xs, info.cpu().numpy(), logdet.cpu().numpy()


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("value", [np.nan, np.inf])
def test_batched_entries_that_are_not_finite(handle, p, variant, value):
    """As above for the batched kernel: inside the diagonal block, below it, in a later round of rows."""
    n = 230
    places = [(5, 2), (20, 11), (40, 5), (63, 62), (100, 45), (200, 70), (229, 30)]
    a = [spd(n, 31 + i).astype(NP[p]).astype(np.float64) for i in range(len(places))]
    bad = [m.copy() for m in a]
    for m, (r, c) in zip(bad, places):
        m[r, c] = m[c, r] = value
    outs, xs, info, logdet = batched_run(p, variant, bad, [n + 1] * len(a), [0] * len(a), [np.ones((n, 1))] * len(a))
    width = (32, 64)[variant]
    for i, (r, c) in enumerate(places):
        assert info[i] == r + 1 and np.isnan(logdet[i]) and np.all(xs[i] == 1.0)
        low, want = np.tril(outs[i]), np.linalg.cholesky(a[i])
        tol = 50 * n * EPS[p]
        assert np.allclose(low[r, :c], want[r, :c], rtol=0, atol=tol) and not np.isfinite(low[r, c])
        done = r // width * width  # the block columns before the failed one are finished
        rows = np.arange(n) != r
        assert np.allclose(low[rows][:, :done], np.tril(want)[rows][:, :done], rtol=0, atol=tol)


@pytest.mark.parametrize("variant", [0, 1])
def test_pivot_helpers_over_the_exponent_range(handle, variant):
    """sqrt(d) and b / sqrt(d) of a tile, against correctly rounded ones: d from the smallest subnormal
    to the largest double, powers of two and values between.  2 u for the root (one rounding after the
    correction), 4 u for the quotient (reciprocal root and product)."""
    rng = np.random.default_rng(9)
    exps = np.unique(np.concatenate([np.arange(-1074, -1000, 7), np.arange(-1074, 1024, 61), [-1023, -1022, -1021, 1023]]))
    d = np.ldexp(1.0, exps)
    d = np.concatenate([d, [v for v in d * rng.uniform(1, 2, d.size) if np.isfinite(v)], [np.finfo(np.float64).max]])
    # b = 0.75 sqrt(d), the last pivot 1 - 0.75^2
    mats = [np.array([[v, 0.75 * np.sqrt(v)], [0.75 * np.sqrt(v), 1.0]]) for v in d] + [np.array([[v]]) for v in d]
    outs, _, info, logdet = batched_run("d", variant, mats, [m.shape[0] for m in mats], [0] * len(mats), None)
    assert np.all(info == 0) and np.all(np.isfinite(logdet))
    u = EPS["d"] / 2
    for m, out in zip(mats, outs):
        root = np.sqrt(m[0, 0])
        assert abs(out[0, 0] - root) <= 2 * u * root
        if m.shape[0] == 2:
            assert abs(out[1, 0] - m[1, 0] / root) <= 4 * u * 0.75


@pytest.mark.parametrize("uplo", ["L", "U"])
def test_panel_over_the_exponent_range(handle, uplo):
    """A diagonal block of pivots from 1e-320 to 1e300, one row below it: b / sqrt(d) within 6 u."""
    n = 129
    d = 10.0 ** np.random.default_rng(2).permutation(np.linspace(-320, 300, 128))
    a = np.diag(np.append(d, 1.0))
    a[128, :128] = a[:128, 128] = np.sqrt(d) / 16
    t, ptr = device(a, n, "d")
    assert potrf(handle, "d", uplo, n, ptr, n) == 0
    out = host(t, n, n, n)
    low = np.tril(out) if uplo == "L" else np.triu(out).T
    u = EPS["d"] / 2
    assert np.all(np.abs(np.diag(low)[:128] - np.sqrt(d)) <= 2 * u * np.sqrt(d))
    want = a[128, :128] / np.sqrt(d)
    assert np.all(np.abs(low[128, :128] - want) <= 6 * u * want)


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("uplo", ["L", "U"])
@pytest.mark.parametrize("k", [0, 7, 100, 127, 150, 199])
def test_infinite_pivot(handle, p, uplo, k):
    """As sqrt and division give it: an infinite diagonal entry, zeros below it, the rest as without
    that row and column."""
    n = 200
    a = spd(n, 6).astype(NP[p]).astype(np.float64)
    b = a.copy()
    b[k, k] = np.inf
    t, ptr = device(b, n, p)
    assert potrf(handle, p, uplo, n, ptr, n) == 0
    out = host(t, n, n, n).astype(np.float64)
    low = np.tril(out) if uplo == "L" else np.triu(out).T
    assert low[k, k] == np.inf and np.all(low[k + 1:, k] == 0)
    rest = np.delete(np.arange(n), k)
    want = np.linalg.cholesky(a[np.ix_(rest, rest)])
    assert np.allclose(low[np.ix_(rest, rest)], want, rtol=0, atol=50 * n * EPS[p])


@pytest.mark.parametrize("p", ["s", "d"])
@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("solve", [False, True])
def test_batched_variants(handle, p, variant, solve):
    """Both block-column widths over every tile edge, odd and padded leading dimensions, matrices that
    fail on both sides of the edges among them."""
    torch = _torch()
    from libddla_b200.ddla import _c_api as C

    orders = [1, 7, 8, 9, 31, 32, 33, 63, 64, 65, 127, 128, 129, 159, 160, 191, 192, 193, 320, 511, 512]
    fails = [(64, 0), (65, 64), (129, 63), (129, 128), (200, 71), (320, 256), (512, 511)]
    cases = [(n, None) for n in orders] + fails
    mats, store, ptrs, rhs, bptr, ldas = [], [], [], [], [], []
    for i, (n, bad) in enumerate(cases):
        a = spd(n, 11 + i).astype(NP[p]).astype(np.float64)
        if bad is not None:
            a[bad, bad] = -2.0
        lda = n + i % 4
        t, ptr = device(a, lda, p, shift=i % 3)
        b = np.random.default_rng(i).standard_normal((n, 1))
        tb, pb = device(b, n, p)
        mats.append(a), store.append(t), ptrs.append(ptr), rhs.append((b, tb)), bptr.append(pb), ldas.append(lda)
    count = len(cases)
    up = lambda v, dt: torch.tensor(np.array(v, dtype=dt), device="cuda")
    dn, dl = up([n for n, _ in cases], np.int32), up(ldas, np.int32)
    da, db = up(ptrs, np.int64), up(bptr, np.int64)
    logdet = torch.zeros(count, dtype=torch.float64, device="cuda")
    info = torch.full((count,), -5, dtype=torch.int32, device="cuda")
    sel = torch.full((count,), variant, dtype=torch.uint8, device="cuda")
    counters = torch.zeros(2, dtype=torch.int32, device="cuda")
    f = C.lib.ddlak_posv_vbatched
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_char, ctypes.c_int, ctypes.c_int] + [ctypes.c_void_p] * 9 + [ctypes.c_int, ctypes.c_void_p]
    torch.cuda.synchronize()
    rc = f(p.encode(), 512, count, dn.data_ptr(), da.data_ptr(), dl.data_ptr(), db.data_ptr() if solve else None,
           logdet.data_ptr(), info.data_ptr(), None, sel.data_ptr(), counters.data_ptr(), 7,
           torch.cuda.current_stream().cuda_stream)
    assert rc == 0
    torch.cuda.synchronize()
    for i, (n, bad) in enumerate(cases):
        out = host(store[i], n, n, ldas[i], i % 3).astype(np.float64)
        b, tb = rhs[i]
        x = host(tb, n, 1, n).astype(np.float64)
        if bad is not None:
            assert int(info[i]) == bad + 1 and np.isnan(float(logdet[i]))
            assert np.array_equal(x, b.astype(NP[p]).astype(np.float64))
            fixed = mats[i].copy()
            fixed[bad, bad] = 1e3  # any positive definite completion has the same columns before `bad`
            low = np.linalg.cholesky(fixed)
            assert np.allclose(np.tril(out)[:, :bad], low[:, :bad], rtol=0, atol=50 * n * EPS[p])
            continue
        assert int(info[i]) == 0
        check_factor(mats[i], out, "L", p)
        assert np.array_equal(np.triu(out, 1), np.triu(mats[i], 1))
        want = np.linalg.slogdet(mats[i])[1]
        # the stored factor is that of A + E, |E| <= 4 (n + 1) u |A|; log det moves by at most
        # trace |A^-1 E| <= n cond(A) 4 (n + 1) u, cond(A) about 5
        assert abs(float(logdet[i]) - want) <= 20 * n * (n + 1) * EPS[p] + 1e-12
        if solve:
            res = mats[i] @ x - b.astype(NP[p])
            assert np.max(np.abs(res)) <= 40 * (n + 1) * EPS[p] * np.linalg.norm(mats[i], 2) * np.max(np.abs(x))


@pytest.mark.parametrize("p,n", [("s", 1), ("s", 65), ("s", 1025), ("s", 3799), ("s", 3800), ("s", 3801), ("s", 4097),
                                 ("d", 1), ("d", 65), ("d", 1025)])
def test_inverse_of_a_large_factor(handle, p, n):
    """Both sides of the order from which FP32 inverts by doubling, leading dimensions with TMA and
    without, a last leaf of one row.  Substitution and products alike give |L W - I| <= c n u |L||W|
    with c a small constant (Higham, section 14.2); 4 here."""
    torch = _torch()
    from libddla_b200.ddla import _c_api as C

    dt = torch.float32 if p == "s" else torch.float64
    g = torch.randn(n, n, device="cuda", dtype=torch.float64, generator=torch.Generator(device="cuda").manual_seed(n))
    low = torch.linalg.cholesky(g @ g.T / n + torch.eye(n, device="cuda", dtype=torch.float64)).to(dt)
    store, w = low.T.contiguous(), torch.full((n, n), float("nan"), device="cuda", dtype=dt)
    C.lib.ddlak_potrs_workspace.restype = ctypes.c_ulonglong
    work = torch.zeros(int(C.lib.ddlak_potrs_workspace(n, n)), dtype=torch.uint8, device="cuda")
    f = C.lib.ddlak_trtri_blocked
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_char, ctypes.c_int, ctypes.c_void_p, ctypes.c_longlong, ctypes.c_void_p, ctypes.c_longlong,
                  ctypes.c_void_p, ctypes.c_ulonglong, ctypes.c_void_p]
    assert f(p.encode(), n, store.data_ptr(), n, w.data_ptr(), n, work.data_ptr(), work.numel(),
             torch.cuda.current_stream().cuda_stream) == 0
    torch.cuda.synchronize()
    assert int(work[:4].view(torch.int32)[0]) == 0
    inv = torch.tril(w.T).double()
    low = low.double()
    res = (low @ inv - torch.eye(n, device="cuda", dtype=torch.float64)).abs()
    bound = 4 * n * EPS[p] / 2 * (low.abs() @ inv.abs())
    assert bool(torch.all(res <= bound)), float((res / bound).nan_to_num().max())


@pytest.mark.parametrize("n", [1025, 1101, 1536, 3801])
def test_large_fp32_gradient(handle, n):
    """The FP32 inversion and the contraction: leading dimensions with TMA (a multiple of 4) and without."""
    torch = _torch()
    from libddla_b200.ddla import autograd as ag

    g = torch.Generator(device="cuda").manual_seed(n)
    x = torch.rand(1, n, 2, generator=g, device="cuda", dtype=torch.float32)
    y = torch.randn(1, n, generator=g, device="cuda", dtype=torch.float32)
    th = torch.tensor([0.3, 1.0, 0.5], dtype=torch.float64, device="cuda", requires_grad=True)
    loss = ag.gp_nll(x, y, th, handle)
    (got,) = torch.autograd.grad(loss.sum(), th)
    t = th.detach().clone().requires_grad_()
    xd, yd = x[0].double(), y[0].double()
    k = t[1] * torch.exp(-torch.cdist(xd, xd).square() / (2 * t[0] ** 2)) + t[2] * torch.eye(n, device="cuda")
    low = torch.linalg.cholesky(k)
    want_loss = 0.5 * (yd @ torch.cholesky_solve(yd[:, None], low)[:, 0]) + low.diagonal().log().sum()
    (want,) = torch.autograd.grad(want_loss, t)
    # condition number of K + 0.5 I up to about n; errors of n u relative to the largest component
    assert abs(float(loss) - float(want_loss)) <= 1e-4 * abs(float(want_loss))
    assert float((got - want).abs().max()) <= 1e-3 * float(want.abs().max())
