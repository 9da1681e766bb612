"""The block-Jacobi eigensolver (ntg_eigh) and the spectral-weight kernel behind the
finite-time predictions (predict.py:185-229, 1180-1294, where the reference calls eigh),
against float64 numpy on the same matrices."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _sym(n, seed, kind):
    rng = np.random.default_rng(seed)
    if kind == 'psd':  # a kernel-like matrix: fast-decaying spectrum, clustered tail
        g = rng.standard_normal((n, max(4, n // 4)))
        a = g @ g.T / g.shape[1] + 1e-3 * np.eye(n)
    else:  # indefinite
        g = rng.standard_normal((n, n))
        a = (g + g.T) / 2
    return a.astype(np.float32)


@pytest.mark.parametrize('n', [1, 5, 40, 64, 100, 257, 1000])
@pytest.mark.parametrize('kind', ['psd', 'indefinite'])
def test_eigh_matches_float64(nt, n, kind):
    from nt_gb300 import predict
    a = _sym(n, n, kind)
    evals, evecs = predict._eigh(torch.from_numpy(a).cuda(), 0.)
    w = evals.double().cpu().numpy()
    v = evecs.double().cpu().numpy()
    a64 = a.astype(np.float64)
    scale = np.linalg.norm(a64, 2)
    # residual of every pair, orthogonality, eigenvalues against numpy's
    assert np.max(np.abs(a64 @ v - v * w[None])) / scale < 2e-5
    assert np.max(np.abs(v.T @ v - np.eye(n))) < 2e-5
    want = np.linalg.eigvalsh(a64)
    assert np.max(np.abs(np.sort(w) - want)) / scale < 1e-5


def test_eigh_shift(nt):
    from nt_gb300 import predict
    a = _sym(80, 3, 'psd')
    e0, _ = predict._eigh(torch.from_numpy(a).cuda(), 0.)
    e1, _ = predict._eigh(torch.from_numpy(a).cuda(), 0.25)
    np.testing.assert_allclose(np.sort(e1.cpu().numpy()), np.sort(e0.cpu().numpy()) + 0.25,
                               atol=2e-5)


@pytest.mark.parametrize('kind', range(7))
def test_spectral_weights(nt, kind):
    from nt_gb300 import predict
    rng = np.random.default_rng(kind)
    lam = np.concatenate([rng.uniform(1e-3, 5., 30), [-1e-4, 2e-6]]).astype(np.float32)
    x = rng.standard_normal((32, 3)).astype(np.float32)
    ts = np.array([0.3, 2., 50.])
    got = predict._spectral(torch.from_numpy(lam).cuda(), torch.from_numpy(ts).cuda(), kind,
                            7., torch.from_numpy(x).cuda()).cpu().numpy()
    l64 = lam.astype(np.float64)[:, None]
    pos = np.maximum(l64, 0.)
    for j, t in enumerate(ts):
        e = pos * t / 7.
        w = [np.expm1(-e), np.expm1(-e) / np.abs(l64), pos * np.exp(-2 * e), np.exp(-e),
             -np.expm1(-2 * e) / np.abs(l64), -np.expm1(-e), -np.expm1(-e) / np.abs(l64)][kind]
        np.testing.assert_allclose(got[:, j, :], w * x, rtol=1e-6, atol=1e-30)


@pytest.mark.parametrize('n', [65, 96, 128, 129, 320])
def test_eigh_of_coupled_blocks(nt, n):
    """Two to ten blocks of 32, where the couplings inside a block are rotated once a sweep: a
    matrix whose couplings lie inside the blocks only, one whose couplings lie between them
    only, and both; the bounds of test_eigh_matches_float64."""
    from nt_gb300 import predict
    rng = np.random.default_rng(n)
    g = rng.standard_normal((n, n))
    g = (g + g.T) / 2
    inside = (np.arange(n)[:, None] // 32) == (np.arange(n)[None] // 32)
    for mask in (inside, ~inside | np.eye(n, dtype=bool), np.ones((n, n))):
        a = (g * mask).astype(np.float32)
        evals, evecs = predict._eigh(torch.from_numpy(a).cuda(), 0.)
        w, v = evals.double().cpu().numpy(), evecs.double().cpu().numpy()
        scale = np.linalg.norm(a.astype(np.float64), 2)
        assert np.max(np.abs(a @ v - v * w[None])) / scale < 2e-5
        assert np.max(np.abs(v.T @ v - np.eye(n))) < 2e-5
        assert np.max(np.abs(np.sort(w) - np.linalg.eigvalsh(a.astype(np.float64)))) < 1e-5 * scale


@pytest.mark.parametrize('n', [64, 100, 333])
def test_eigh_of_a_cluster(nt, n):
    """Half the spectrum at one eigenvalue, half 1e-5 apart: what the refinement cannot separate
    stays orthogonal; the bounds of test_eigh_matches_float64."""
    from nt_gb300 import predict
    g = torch.Generator(device='cuda').manual_seed(n)
    q = torch.linalg.qr(torch.randn((n, n), generator=g, device='cuda', dtype=torch.float64))[0]
    e = torch.ones(n, device='cuda', dtype=torch.float64)
    e[n // 2:] += 1e-5 * torch.arange(n - n // 2, device='cuda')
    a = ((q * e) @ q.t()).float()
    evals, evecs = predict._eigh(a, 0.)
    a, w, v = a.double(), evals.double(), evecs.double()
    assert float((a @ v - v * w).abs().max()) < 2e-5
    assert float((v.t() @ v - torch.eye(n, device='cuda')).abs().max()) < 2e-5
