"""The tensor-core GEMM (3xTF32 tcgen05) and the blocked Cholesky built on it,
against float64 (scipy) on the same inputs: predict.py:1224-1258's cho_factor /
cho_solve, which the reference leaves to cuSOLVER."""
import numpy as np
import pytest
import scipy.linalg as sla
import torch

pytestmark = pytest.mark.gpu


def _t(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


@pytest.mark.parametrize('m,n,k,alpha,beta', [(128, 128, 32, 1., 0.), (300, 130, 100, -1., 1.),
                                              (1000, 700, 515, 0.5, 2.), (7, 5, 3, 1., 0.)])
def test_gemm_tc_matches_float64(nt, m, n, k, alpha, beta):
    from nt_gb300 import _lib as L
    rng = np.random.default_rng(m + n + k)
    kp = (k + 3) // 4 * 4  # row pitch: a multiple of 4 floats
    a = np.zeros((m, kp), np.float32)
    b = np.zeros((n, kp), np.float32)
    a[:, :k] = rng.standard_normal((m, k))
    b[:, :k] = rng.standard_normal((n, k))
    c0 = rng.standard_normal((m, n)).astype(np.float32)
    ta, tb, tc = _t(a), _t(b), _t(c0)
    L.call('ntg_gemm_tc', L.stream(), ta.data_ptr(), kp, tb.data_ptr(), kp, tc.data_ptr(), n, m,
           n, k, alpha, beta, 0)
    got = tc.cpu().numpy().astype(np.float64)
    a64, b64 = a[:, :k].astype(np.float64), b[:, :k].astype(np.float64)
    want = alpha * a64 @ b64.T + beta * c0
    scale = abs(alpha) * np.abs(a64) @ np.abs(b64).T + abs(beta) * np.abs(c0)
    assert np.max(np.abs(got - want) / scale) < 2e-6


def test_gemm_tc_lower_triangle_only(nt):
    from nt_gb300 import _lib as L
    rng = np.random.default_rng(3)
    n, k = 260, 128
    p = rng.standard_normal((n, k)).astype(np.float32)
    c0 = rng.standard_normal((n, n)).astype(np.float32)
    tp, tc = _t(p), _t(c0)
    L.call('ntg_gemm_tc', L.stream(), tp.data_ptr(), k, tp.data_ptr(), k, tc.data_ptr(), n, n, n,
           k, -1., 1., 1)
    got = tc.cpu().numpy()
    p64 = p.astype(np.float64)
    want = c0 - p64 @ p64.T
    low = np.tril(np.ones((n, n), bool))
    scale = np.abs(p64) @ np.abs(p64).T + np.abs(c0)
    assert np.max(np.abs(got - want)[low] / scale[low]) < 2e-6
    np.testing.assert_array_equal(got[~low], c0[~low])  # the upper triangle is untouched


def _spd(n, seed, cond_reg=1e-3):
    rng = np.random.default_rng(seed)
    g = rng.standard_normal((n, n + 7))
    k = g @ g.T / n
    return k.astype(np.float32)


def _factor(nt, k, diag_reg):
    from nt_gb300 import predict
    return predict.CholeskySolver(_t(k), diag_reg, False)


@pytest.mark.parametrize('n', [64, 128, 300, 1000])
def test_factor_matches_float64(nt, n):
    k = _spd(n, n)
    s = _factor(nt, k, 1e-3)
    assert s.info == 0
    lf = s.L.cpu().numpy().astype(np.float64)
    assert np.all(np.triu(lf, 1) == 0)
    a = k.astype(np.float64) + 1e-3 * np.trace(k.astype(np.float64)) / n * np.eye(n)
    # backward error of the FP32 factorisation
    assert np.max(np.abs(lf @ lf.T - a)) / np.max(np.abs(a)) < 1e-5
    want = np.linalg.cholesky(a)
    assert np.max(np.abs(lf - want)) / np.max(np.abs(want)) < 1e-4


@pytest.mark.parametrize('n,m', [(300, 1), (1000, 10), (777, 16), (513, 40), (1000, 300)])
def test_solve_matches_float64(nt, n, m):
    k = _spd(n, n + m)
    s = _factor(nt, k, 1e-4)
    rng = np.random.default_rng(m)
    b = rng.standard_normal((n, m)).astype(np.float32)
    a = k.astype(np.float64) + 1e-4 * np.trace(k.astype(np.float64)) / n * np.eye(n)
    want = sla.cho_solve(sla.cho_factor(a), b.astype(np.float64))
    got = s.solve(_t(b)).cpu().numpy()
    assert np.max(np.abs(got - want)) / np.max(np.abs(want)) < 1e-6
    plain = s.solve(_t(b), refine_iters=0, residual=False).cpu().numpy()
    # the unrefined FP32 solve is within the conditioning of the problem (kappa ~ 4e4)
    assert np.max(np.abs(plain - want)) / np.max(np.abs(want)) < 5e-2
    assert float(s.residual.item()) < 1e-4 * np.max(np.abs(b))


def test_not_positive_definite_reports_the_pivot(nt):
    k = np.eye(200, dtype=np.float32)
    k[150, 150] = -1.
    with pytest.warns(UserWarning, match='not positive definite'):
        s = _factor(nt, k, 0.)
    assert s.info == 151


def test_logdet_matches_float64(nt):
    k = _spd(400, 9)
    s = _factor(nt, k, 1e-3)
    a = k.astype(np.float64) + 1e-3 * np.trace(k.astype(np.float64)) / 400 * np.eye(400)
    want = np.linalg.slogdet(a)[1]
    # each pivot carries the float32 factor's rounding (cond ~ 1e3 here)
    assert abs(float(s.logdet().item()) - want) < 5e-5 * abs(want)


def test_concurrent_factorisations_on_two_streams(nt):
    """Two host threads, each on its own stream, factorise different matrices at once: the
    library's per-device streams and events are taken by one factorisation at a time, so
    each factor is that of its own matrix."""
    import threading
    from nt_gb300 import predict
    ks = [_spd(700, 41 + i) for i in range(2)]
    out, errs = [None, None], []

    def work(i):
        try:
            st = torch.cuda.Stream()
            with torch.cuda.stream(st):
                for _ in range(3):
                    s = predict.CholeskySolver(_t(ks[i]), 1e-3, False)
                    out[i] = s.L.clone()
            st.synchronize()
        except Exception as e:  # reported below
            errs.append(e)
    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errs
    for i in range(2):
        a = ks[i].astype(np.float64)
        a = a + 1e-3 * np.trace(a) / 700 * np.eye(700)
        lf = out[i].cpu().numpy().astype(np.float64)
        assert np.max(np.abs(lf @ lf.T - a)) / np.max(np.abs(a)) < 1e-5


@pytest.mark.parametrize('n,m', [(1024, 65), (1030, 300), (777, 500), (2050, 65), (1500, 1500)])
def test_exact_residual(nt, n, m):
    """The tensor-core residual of many right-hand sides (from 2^26 products on) against
    float64: the largest residual of a returned solution, whose true size is 1e-9 to 1e-7 of
    the products it cancels. The digits carry 40 bits of each product, sums are exact, and
    float64's own sums are good to n 2^-53."""
    from nt_gb300 import predict
    g = torch.Generator(device='cuda').manual_seed(n + m)
    x = torch.randn((n, 64), generator=g, device='cuda', dtype=torch.float64)
    # a kernel with a large constant part and scales that differ from row to row
    s = torch.exp(torch.randn((n, 1), generator=g, device='cuda', dtype=torch.float64))
    k = ((x @ x.t() / 64 + 1.) ** 2 * s * s.t()).float()
    b = torch.randn((n, m), generator=g, device='cuda')
    b[:, 0] = 0.
    solver = predict.CholeskySolver(k, 1e-2, False)
    xs, x64 = solver.solve(b, refine_iters=1, want_x64=True)
    a = k.double() + float(solver.lam[0]) * torch.eye(n, device='cuda', dtype=torch.float64)
    r = b.double() - a @ x64
    size = (a.abs().amax(1, keepdim=True) * x64.abs().amax(0, keepdim=True)).max()
    assert abs(float(solver.residual) - float(r.abs().max())) < n ** .5 * 2. ** -38 * float(size)
    # and what the step made of it: the solution is that of float64 to float32 rounding
    want = torch.linalg.solve(a, b.double())
    assert float((x64 - want).norm() / want.norm()) < 1e-6
    assert float(xs[:, 0].abs().max()) == 0.
    # another solver's NaN row reaches every solution, as it does in float64
    bad = k.clone()
    bad[3, 5] = bad[5, 3] = float('nan')
    with pytest.warns(UserWarning, match='not positive definite'):
        out = predict.CholeskySolver(bad, 1e-2, False).solve(b, refine_iters=1)
    assert bool(torch.isnan(out).all())


def test_exact_residual_in_bands(nt):
    """A's digits are made 7296 rows at a time from there on: the largest residual once more,
    under the same bound, at two bands and a remainder of columns."""
    from nt_gb300 import predict
    n, m = 7300, 70
    g = torch.Generator(device='cuda').manual_seed(1)
    x = torch.randn((n, 64), generator=g, device='cuda')
    k = (x @ x.t() / 64 + 1.) ** 2
    k = (k + k.t()) / 2
    b = torch.randn((n, m), generator=g, device='cuda')
    # the large rows, and so the largest residual, in either band in turn
    for rows in (slice(0, 64), slice(n - 64, n)):
        b2 = b * 1e-4
        b2[rows] = b[rows]
        solver = predict.CholeskySolver(k, 1e-1, False)
        _, x64 = solver.solve(b2, refine_iters=1, want_x64=True)
        r = b2.double() - k.double() @ x64 - float(solver.lam[0]) * x64
        size = (k.abs().amax(1, keepdim=True) * x64.abs().amax(0, keepdim=True)).max()
        assert abs(float(solver.residual) - float(r.abs().max())) < n ** .5 * 2. ** -38 * float(size)


@pytest.mark.parametrize('n,m', [(1024, 65), (777, 500), (1500, 130)])
@pytest.mark.parametrize('kind', ['scales', 'decay'])
def test_exact_residual_of_wide_ranges(nt, kind, n, m):
    """Kernels whose samples differ in scale by 1e5, and kernels that decay to nothing: two
    refinement steps leave what the residual itself loses, 2^-46 of the largest products of the
    matrix scaled to a unit diagonal (twice 2^-48 for either operand and as much for the sums),
    times the root of their number and that matrix's condition."""
    from nt_gb300 import predict
    g = torch.Generator(device='cuda').manual_seed(n)
    r = lambda *s: torch.rand(s, generator=g, device='cuda', dtype=torch.float64)
    if kind == 'scales':
        x = torch.randn((n, 32), generator=g, device='cuda', dtype=torch.float64)
        x = x / x.norm(dim=1, keepdim=True)
        s = torch.exp(r(n, 1) * np.log(1e5))
        k = ((1. + x @ x.t()) ** 3 / 8 + 1e-2 * torch.eye(n, device='cuda')) * s * s.t()
    else:
        x = 30. * r(n, 2)
        k = torch.exp(-torch.cdist(x, x) ** 2) + 1e-2 * torch.eye(n, device='cuda')
    k = k.float()
    b = torch.randn((n, m), generator=g, device='cuda')
    _, x64 = predict.CholeskySolver(k, 0., True).solve(b, refine_iters=2, want_x64=True)
    a = k.double()
    root = a.diagonal().sqrt()[:, None]
    unit = torch.linalg.eigvalsh(a / root / root.t())
    want = torch.linalg.solve(a / root / root.t(), b.double() / root)
    err = float((x64 * root - want).norm() / want.norm())
    assert err < n ** .5 * 2. ** -46 * float(unit[-1] / unit[0])


@pytest.mark.parametrize('n,m', [(1, 17), (127, 17), (128, 130), (129, 40), (257, 17), (390, 300)])
def test_many_right_hand_sides_at_tile_edges(nt, n, m):
    """Products with the triangular inverses stop at the triangle, tile by tile: kappa <= 5, so
    one refinement step leaves the float32 rounding of the solution."""
    from nt_gb300 import predict
    rng = np.random.default_rng(n)
    q = rng.standard_normal((n, n))
    a = np.eye(n) + q @ q.T / n  # eigenvalues in [1, 5 + o(1)]
    b = rng.standard_normal((n, m)).astype(np.float32)
    x = predict.CholeskySolver(_t(a), 0., True).solve(_t(b), refine_iters=1)
    want = np.linalg.solve(a.astype(np.float32).astype(np.float64), b.astype(np.float64))
    assert np.max(np.abs(x.cpu().numpy() - want)) < 1e-6 * np.max(np.abs(want))


@pytest.mark.parametrize('n,m', [(1, 1), (15, 2), (16, 3), (17, 5), (129, 8), (300, 9), (513, 16),
                                 (4865, 4)])
def test_few_right_hand_sides_by_rows_and_columns(nt, n, m):
    """Conjugate-gradient solves at the edges of the row-and-column layout (a power of two of
    threads a row, 304 blocks): kappa <= 5 converges to the float32 rounding of the solution;
    one column zero, which stays zero."""
    from nt_gb300 import predict
    rng = np.random.default_rng(n)
    q = rng.standard_normal((n, min(n, 200)))
    a = (np.eye(n) + q @ q.T / max(n, 200)).astype(np.float32)
    b = rng.standard_normal((n, m)).astype(np.float32)
    b[:, -1] *= float(m == 1)
    solver = predict.CholeskySolver(_t(a), 0., True)
    x = solver.solve(_t(b)).cpu().numpy()
    want = np.linalg.solve(a.astype(np.float64), b.astype(np.float64))
    assert np.max(np.abs(x - want)) < 1e-6 * np.max(np.abs(want))
    assert m == 1 or np.max(np.abs(x[:, -1])) == 0.
    r = b - a.astype(np.float64) @ x
    # of the returned FP64 solution: below that of its float32 rounding, 2^-24 |A| |x|
    assert float(solver.residual) <= np.max(np.abs(r)) + 2. ** -24 * np.max(
        np.abs(a).astype(np.float64) @ np.abs(x))


@pytest.mark.parametrize('n', [128, 129, 143, 255, 256, 257, 385, 512, 900])
def test_factor_around_the_next_block(nt, n):
    """One to eight panels with remainders of 1 to 128 rows: the factor itself, |L L^T - A|
    within n products of 3xTF32 (2^-21) of the largest entry."""
    from nt_gb300 import predict
    rng = np.random.default_rng(n)
    q = rng.standard_normal((n, n))
    a = (np.eye(n) + q @ q.T / n).astype(np.float32)
    solver = predict.CholeskySolver(_t(a), 0., True)
    assert solver.info == 0
    l = np.tril(solver.L.cpu().numpy().astype(np.float64))
    assert np.max(np.abs(l @ l.T - a)) < n ** .5 * 2. ** -21 * np.max(np.abs(a))
