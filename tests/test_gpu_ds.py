"""The fused diagonal-spatial chain against the float64 oracle and against the layer rules, at
odd sizes, geometries and batch shapes."""
import numpy as np
import pytest
import torch

from oracle import nt_oracle as o

pytestmark = pytest.mark.gpu

NETS = {
    'relu3': lambda m: [m.Conv(1, (3, 3), padding='SAME', W_std=1.4, b_std=.1), m.Relu(),
                        m.Conv(1, (3, 3), padding='SAME', W_std=1.3), m.LeakyRelu(.1),
                        m.Flatten(), m.Dense(1, 1.2, .2), m.Relu(), m.Dense(1)],
    'valid5': lambda m: [m.Conv(1, (5, 3), padding='VALID', W_std=1.4, b_std=.1), m.Erf(),
                         m.Dense(1, 1.1, .1), m.Relu(), m.Conv(1, (2, 4), padding='SAME'),
                         m.Flatten(), m.Dense(1)],
    'rare': lambda m: [m.Conv(1, (3, 3), padding='SAME', W_std=1.2, b_std=.3), m.Gelu(),
                       m.Conv(1, (1, 1), padding='SAME', W_std=1.1), m.Sin(), m.Flatten()],
    'standard': lambda m: [m.Conv(1, (3, 3), padding='SAME', W_std=1.3, b_std=.1,
                                  parameterization='standard'), m.Relu(),
                           m.Conv(1, (3, 3), padding='VALID'), m.Flatten(), m.Dense(1)],
    # taken layer by layer: strides, wrap-around padding
    'strided': lambda m: [m.Conv(1, (3, 3), strides=(2, 1), padding='SAME'), m.Relu(),
                          m.Conv(1, (3, 3), padding='CIRCULAR'), m.Flatten()],
}


def _x(n, shape, seed):
    return np.random.default_rng(seed).standard_normal((n,) + shape).astype(np.float32)


@pytest.mark.parametrize('precision', ['fp32', 'mixed'])
@pytest.mark.parametrize('shape', [(8, 8, 3), (7, 9, 1), (31, 33, 2), (40, 6, 4), (6, 40, 3)])
@pytest.mark.parametrize('name', list(NETS))
def test_networks(nt, name, shape, precision):
    x1, x2 = _x(3, shape, 1), _x(5, shape, 2)
    x2[4] = x1[1]  # a self pair in a block
    layers = NETS[name](nt.stax)
    kf, ko = nt.stax.serial(*layers)[2], o.serial(*NETS[name](o))
    for b in (x2, None):
        get = ('nngp', 'ntk', 'cov1') + (() if b is None else ('cov2',))
        got, want = kf(x1, b, get, precision=precision), ko(x1, b, get)
        k = nt.stax.Identity()[2](x1, b, diagonal_spatial=True, precision=precision)
        for layer in layers:
            k = layer[2](k, precision=precision)
        for i, (g, w) in enumerate(zip(got, want)):
            scale = np.max(np.abs(w))
            assert np.max(np.abs(g.cpu().numpy() - w)) < 1e-5 * scale
            # the layer rules add the same windows in another order: a few u per layer
            assert np.max(np.abs((getattr(k, get[i]) - g).cpu().numpy())) < 1e-5 * scale
        if b is None:
            assert torch.equal(got.nngp, got.nngp.t()) and torch.equal(got.ntk, got.ntk.t())
        assert torch.equal(kf(x1, b, 'nngp', precision=precision), got.nngp)


@pytest.mark.parametrize('n1,n2', [(1, 1), (1, 300), (77, 16), (130, 130), (200, 0)])
def test_runs_of_samples(nt, n1, n2):
    """Pairs do not depend on the run of x2 samples a CTA takes."""
    x1 = torch.from_numpy(_x(n1, (9, 5, 1), 3)).cuda()
    x2 = torch.from_numpy(_x(n2, (9, 5, 1), 4)).cuda() if n2 else None
    kf = nt.stax.serial(*NETS['relu3'](nt.stax))[2]
    got = kf(x1, x2, ('nngp', 'ntk'))
    b = x1 if x2 is None else x2
    for i in {0, n1 // 2, n1 - 1}:
        one = kf(x1[i:i + 1], b[-3:], ('nngp', 'ntk'))
        for g, w in zip(one, got):
            assert torch.equal(g[0], w[i, -3:])


def test_one_spatial_dimension_and_global_pool(nt):
    x1, x2 = _x(4, (19, 3), 5), _x(3, (19, 3), 6)
    net = lambda m: [m.Conv(1, (3,), padding='SAME', W_std=1.3, b_std=.1), m.Relu(),
                     m.Conv(1, (2,), padding='VALID'), m.Relu(), m.Flatten(), m.Dense(1)]
    kf, ko = nt.stax.serial(*net(nt.stax))[2], o.serial(*net(o))
    for g, w in zip(kf(x1, x2, ('nngp', 'ntk')), ko(x1, x2, ('nngp', 'ntk'))):
        assert np.max(np.abs(g.cpu().numpy() - w)) < 1e-5 * np.max(np.abs(w))
    full = kf(x1, x2)
    assert not full.diagonal_spatial and full.shape1 == (4, 1) and not full.x1_is_x2
    z = kf(np.zeros((2, 19, 3), np.float32), None, ('nngp', 'ntk'))
    assert all(bool(torch.isfinite(v).all()) for v in z)


BANDS = {
    'one': lambda m: [m.Conv(1, (3, 3), padding='SAME', W_std=1.4, b_std=.1), m.Relu(),
                      m.Conv(1, (3, 3), padding='SAME', W_std=1.3, b_std=.2), m.Relu(),
                      m.AvgPool((2, 2), (2, 2)),
                      m.Conv(1, (3, 3), padding='SAME', W_std=1.2), m.Relu(), m.Flatten(),
                      m.Dense(1, 1.1, .1)],
    'two': lambda m: [m.Conv(1, (3, 2), padding='SAME', W_std=1.4, b_std=.1), m.Erf(),
                      m.AvgPool((2, 2), (2, 2)),
                      m.Conv(1, (3, 3), padding='SAME', W_std=1.2), m.LeakyRelu(.2),
                      m.AvgPool((2, 2), (2, 2)), m.Flatten(), m.Dense(1), m.Relu(), m.Dense(1)],
    # overlapping windows, strides that leave a gap, windows as large as the map
    'windows': lambda m: [m.Conv(1, (2, 2), padding='VALID', W_std=1.4, b_std=.1), m.Gelu(),
                          m.SumPool((3, 1), (2, 3)), m.Dense(1, 1.2, .1), m.Relu(),
                          m.AvgPool((1, 2), (1, 1)), m.Flatten()],
}


@pytest.mark.parametrize('precision', ['fp32', 'mixed'])
@pytest.mark.parametrize('shape', [(8, 8, 3), (7, 9, 1), (28, 28, 1), (15, 13, 2), (4, 33, 3)])
@pytest.mark.parametrize('name', list(BANDS))
def test_bands(nt, name, shape, precision):
    """Networks with poolings before a Flatten against the oracle and the layer rules, which
    carry the whole full-spatial kernel; the bound of test_networks."""
    from nt_gb300 import _chain, stax
    x1, x2 = _x(3, shape, 1), _x(4, shape, 2)
    x2[3] = x1[1]
    layers = BANDS[name](nt.stax)
    kf, ko = nt.stax.serial(*layers)[2], o.serial(*BANDS[name](o))
    assert _chain.plan_ds(kf.specs, x1.shape, stax._Ctx('fp32'), True) is not None
    for b in (x2, None):
        get = ('nngp', 'ntk', 'cov1') + (() if b is None else ('cov2',))
        got, want = kf(x1, b, get, precision=precision), ko(x1, b, get)
        k = nt.stax.Identity()[2](x1, b, diagonal_spatial=False, precision=precision)
        for layer in layers:
            k = layer[2](k, precision=precision)
        for i, (g, w) in enumerate(zip(got, want)):
            scale = np.max(np.abs(w))
            assert np.max(np.abs(g.cpu().numpy() - w)) < 1e-5 * scale
            assert np.max(np.abs((getattr(k, get[i]) - g).cpu().numpy())) < 1e-5 * scale
        if b is None:
            assert torch.equal(got.nngp, got.nngp.t()) and torch.equal(got.ntk, got.ntk.t())
        whole = kf(x1, b, precision=precision)
        for f in ('diagonal_spatial', 'is_gaussian', 'is_reversed', 'shape1', 'shape2', 'x1_is_x2'):
            assert getattr(whole, f) == getattr(k, f)


@pytest.mark.parametrize('shape,pool,padding,planned', [
    ((8, 8, 1), 2, 'VALID', True), ((8, 8, 1), 2, 'SAME', True), ((9, 8, 1), 2, 'SAME', False),
    ((8, 8, 1), 2, 'CIRCULAR', True), ((9, 9, 1), 3, 'CIRCULAR', True)])
def test_which_poolings_are_bands(nt, shape, pool, padding, planned):
    """Windows that reach past the map stay with the layer rules; both agree with the oracle."""
    from nt_gb300 import _chain, stax
    net = lambda m: [m.Conv(1, (3, 3), padding='SAME', W_std=1.3, b_std=.1), m.Relu(),
                     m.AvgPool((pool, pool), (pool, pool), padding), m.Flatten(), m.Dense(1)]
    kf, ko = nt.stax.serial(*net(nt.stax))[2], o.serial(*net(o))
    x1, x2 = _x(2, shape, 7), _x(3, shape, 8)
    assert (_chain.plan_ds(kf.specs, x1.shape, stax._Ctx('fp32'), True) is not None) == planned
    for g, w in zip(kf(x1, x2, ('nngp', 'ntk')), ko(x1, x2, ('nngp', 'ntk'))):
        assert np.max(np.abs(g.cpu().numpy() - w)) < 1e-5 * np.max(np.abs(w))
