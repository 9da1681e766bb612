"""The flat-input kernels at the edges of their tiles: the Gram and the variances against
float64 and against each other, a run of rules against one launch per layer."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

# one more and one less than the 32-, 64- and 128-wide tiles, on both sides of the rule that
# picks them (152 tiles), and depths off the slices of 16, 32 and 64
SIZES = [(1, 1, 1), (31, 33, 15), (32, 64, 32), (33, 95, 33), (65, 130, 70), (257, 300, 5),
         (385, 420, 129), (800, 801, 20), (801, 799, 17), (1600, 1607, 36), (1665, 1601, 33)]


def _data(n, d, seed):
    g = torch.Generator(device='cuda').manual_seed(seed)
    return torch.randn((n, d), generator=g, device='cuda')


@pytest.mark.parametrize('n1,n2,d', SIZES)
def test_gram_and_variances(nt, n1, n2, d):
    from nt_gb300 import _ops as O
    x1, x2 = _data(n1, d, 1), _data(n2, d, 2)
    x2[0] = x1[n1 - 1]
    q, c1, c2 = O.flat_input(x1, x2)
    want = x1.double() @ x2.double().t() / d
    # one fmaf chain of d products: at most (d + 1) u sum |x1 x2| / d
    bound = (d + 2) * 2. ** -24 * (x1.double().abs() @ x2.double().abs().t()) / d + 1e-30
    assert bool(((q.double() - want).abs() <= bound).all())
    # the same chain everywhere: a sample shared by both inputs meets its own variance
    assert float(q[n1 - 1, 0]) == float(c1[n1 - 1]) == float(c2[0])
    qs, cs, none = O.flat_input(x1, None)
    assert none is None and torch.equal(qs, qs.t()) and torch.equal(cs, O.cov_diag(x1))
    assert torch.equal(qs, O.gram(x1, x1.clone()))
    if d > 1:  # rows that do not start on 16 bytes
        wide = torch.zeros((n1 * d + 1,), device='cuda')
        wide[1:] = x1.reshape(-1)
        off = wide[1:].reshape(n1, d)
        assert torch.equal(O.gram(off, x2), q) and torch.equal(O.cov_diag(off), c1)


@pytest.mark.parametrize('precision', ['fp32', 'mixed'])
@pytest.mark.parametrize('n1,n2', [(1, 1), (31, 63), (32, 64), (33, 65), (70, 0), (200, 131)])
def test_run_of_rules_equals_layers(nt, n1, n2, precision):
    """A network's run of flat layers against its layers called one by one on Kernels."""
    s = nt.stax
    layers = [s.Dense(1, 1.4, 0.1), s.Relu(), s.Dense(1, 1.2, 0.2, parameterization='standard'),
              s.Erf(), s.Identity(), s.Dense(1, 0.9), s.LeakyRelu(0.1), s.Dense(1, 1.1, 0.3),
              s.Gelu(), s.Dense(1, 1.3, 0.1), s.Sin(1., 1.1, 0.2), s.Dense(1, 1.), s.Rbf(0.3)]
    x1 = _data(n1, 20, 3)
    x2 = _data(n2, 20, 4) if n2 else None
    whole = s.serial(*layers)[2](x1, x2, precision=precision)
    k = s.Identity()[2](x1, x2, precision=precision)
    for layer in layers:
        k = layer[2](k, precision=precision)
    for name in ('nngp', 'ntk', 'cov1', 'cov2'):
        a, b = getattr(whole, name), getattr(k, name)
        assert (a is None) == (b is None)
        if a is not None:
            assert torch.equal(a, b), name
    # the rules before they were fused: the same layers on kernels with one spatial position
    kp = s.Identity()[2](x1, x2, precision=precision)
    r = lambda t, nb: None if t is None else t.reshape(tuple(t.shape) + (1, 1))
    kp = kp.replace(nngp=r(kp.nngp, 2), cov1=r(kp.cov1, 1), cov2=r(kp.cov2, 1))
    kp = s.serial(*layers)[2](kp, precision=precision)
    for name in ('nngp', 'ntk', 'cov1', 'cov2'):
        a, b = getattr(whole, name), getattr(kp, name)
        if a is not None:
            assert torch.equal(a, b.reshape(a.shape)), name


def test_long_run_is_split(nt):
    """More layers than one launch takes; dropped and zero NTKs."""
    s = nt.stax
    layers = [v for _ in range(40) for v in (s.Dense(1, 1.4, 0.05), s.Relu())]
    x = _data(37, 12, 5)
    whole = s.serial(*layers)[2](x, None, ('nngp', 'ntk'))
    k = s.Identity()[2](x, None)
    for layer in layers:
        k = layer[2](k)
    assert torch.equal(whole.nngp, k.nngp) and torch.equal(whole.ntk, k.ntk)
    assert torch.equal(s.serial(*layers)[2](x, None, 'nngp'), whole.nngp)
    with pytest.raises(ValueError, match='must be Gaussian'):
        s.serial(s.Dense(1), s.Relu(), s.Relu())[2](x, None, 'nngp')
    y = np.asarray([[1., 2.], [3., 4.]], np.float32)
    assert s.Identity()[2](y, None).ntk.ndim == 0


@pytest.mark.parametrize('m,n,k', [(1, 1, 1), (31, 33, 15), (32, 32, 16), (33, 65, 17),
                                   (500, 60, 500), (640, 700, 100), (100, 4000, 33),
                                   (768, 832, 40)])
def test_small_products(nt, m, n, k):
    """Both sides of the rule (152 tiles of 64 x 64), plain and transposed, accumulating."""
    from nt_gb300 import _lib as L, predict
    a, b = _data(m, k, 6), _data(k, n, 7)
    want = a.double() @ b.double()
    # at most a chain of k products
    bound = (k + 3) * 2. ** -24 * (a.double().abs() @ b.double().abs())
    assert bool(((predict._gemm(a, b).double() - want).abs() <= bound).all())
    at = a.t().contiguous()
    assert bool(((predict._gemm_tn(at, b).double() - want).abs() <= bound).all())
    c = torch.ones((m, n), device='cuda')
    L.call('ntg_gemm_ex', L.stream(), L.ptr(a), L.ptr(b), L.ptr(c), m, n, k, 0, -2., 1)
    assert bool(((c.double() - (1. - 2. * want)).abs() <= 2 * bound + 2. ** -22
                 * (1. + 2. * want.abs())).all())


def test_dense_on_kernels_without_variances(nt):
    s = nt.stax
    k = s.Identity()[2](_data(5, 12, 8), _data(7, 12, 9))
    kf = s.serial(s.Dense(1, 1.3, .2), s.Dense(1, 1.1))[2]
    want = kf(k)
    for part in (k.replace(cov1=None, cov2=None), k.replace(cov2=None)):
        got = kf(part)
        assert torch.equal(got.nngp, want.nngp) and torch.equal(got.ntk, want.ntk)
        assert got.cov2 is None
