"""Whole-network kernels where variances vanish: empty regions and empty images, with and without
a bias, in both parameterizations, against the float64 oracle. An entry with q = 0 and v1 v2 = 0
takes the angle pi / 2, and its ntk is 1 (not 0) in the standard parameterization with b_std = 0."""
import numpy as np
import pytest

from oracle import nt_oracle as o

pytestmark = pytest.mark.gpu


def _net(m, name, b, par):
    c = lambda: m.Conv(1, (3, 3), padding='SAME', W_std=1.3, b_std=b, parameterization=par)
    pool = lambda: m.AvgPool((2, 2), (2, 2))
    return {
        # the diagonal-spatial chain, the band behind a pooling, the 32 x 32 chain with three
        # segments (compiled for its shape), one segment, and a mix of rules
        'diagonal': lambda: [c(), m.Relu(), c(), m.LeakyRelu(.1), m.Flatten(), m.Dense(1)],
        'band': lambda: [c(), m.Relu(), pool(), c(), m.Relu(), m.Flatten(), m.Dense(1)],
        'chain5': lambda: [c(), m.Relu(), c(), m.Relu(), pool(), c(), m.Relu(), pool(), c(),
                           m.Relu(), m.GlobalAvgPool()],
        'chain1': lambda: [c(), m.Relu(), c(), m.Relu(), m.Flatten(), m.Dense(1)],
        'mixed_rules': lambda: [c(), m.Relu(), pool(), c(), m.Erf(), m.GlobalAvgPool()],
    }[name]()


def _images(n, shape, seed, empty):
    x = np.random.default_rng(seed).standard_normal((n,) + shape).astype(np.float32)
    if empty == 'border':
        x[:, :3] = x[:, -2:] = 0.
        x[:, :, :2] = x[:, :, -4:] = 0.
    elif empty == 'corner':
        x[:, :4, :5] = 0.
    elif empty == 'image':
        x[0] = 0.
    return x


SHAPES = {'diagonal': (10, 9, 2), 'band': (10, 9, 2), 'chain5': (32, 32, 3), 'chain1': (32, 32, 1),
          'mixed_rules': (32, 32, 1)}


@pytest.mark.parametrize('e1,e2', [('border', None), (None, 'corner'), ('border', 'border'),
                                   ('image', None), ('image', 'image')])
@pytest.mark.parametrize('b', [None, 0., .1])
@pytest.mark.parametrize('par', ['ntk', 'standard'])
@pytest.mark.parametrize('name', list(SHAPES))
def test_empty_regions(nt, name, par, b, e1, e2):
    """The bound of the dense-image tests, 1e-5 of the largest entry; also where nothing of the
    largest is left (both images empty: 0 is 0)."""
    x1, x2 = _images(2, SHAPES[name], 1, e1), _images(2, SHAPES[name], 2, e2)
    kf = nt.stax.serial(*_net(nt.stax, name, b, par))[2]
    ko = o.serial(*_net(o, name, b, par))
    for y in (x2, None):
        for g, w in zip(kf(x1, y, ('nngp', 'ntk')), ko(x1, y, ('nngp', 'ntk'))):
            assert np.max(np.abs(g.cpu().numpy() - w)) <= 1e-5 * np.max(np.abs(w))


# powers of two, so that float32 scales the images exactly; networks without a bias are homogeneous
@pytest.mark.parametrize('e1,e2', [(-12, -12), (-20, -20), (-27, -27), (-30, -30), (-32, -32),
                                   (-60, 0), (30, 30)])
@pytest.mark.parametrize('name', ['diagonal', 'band', 'chain5', 'chain1', 'layers'])
def test_scaled_images(nt, name, e1, e2):
    """Images far from unit size, against the same network on the unscaled images: one layer's
    v1 v2 - q^2 keeps 20 bits at 2^-128, the smallest product here (2^-149 is float32's step),
    and the angle is as good as its root; 1e-5 as for images of unit size. A variance's own
    covariances, products of 2^-240 at (-60, 0), are float32 zeros where poolings or layer rules
    take them from a whole per-sample kernel."""
    if e1 == -60 and name not in ('diagonal', 'chain1'):
        pytest.skip('the per-sample kernels underflow')
    shape = {'layers': (6, 6, 2)}.get(name, SHAPES.get(name))
    if name == 'layers':
        net = lambda m: [m.Conv(1, (3, 3), padding='SAME', W_std=1.3), m.Relu(),
                         m.Conv(1, (3, 3), padding='SAME', W_std=1.3), m.Relu(), m.GlobalAvgPool()]
    else:
        net = lambda m: _net(m, name, None, 'ntk')
    x1, x2 = _images(2, shape, 1, None), _images(2, shape, 2, None)
    kf, ko = nt.stax.serial(*net(nt.stax))[2], o.serial(*net(o))
    for precision in ('fp32', 'mixed'):
        got = kf(x1 * np.float32(2.) ** e1, x2 * np.float32(2.) ** e2, ('nngp', 'ntk'),
                 precision=precision)
        for g, w in zip(got, ko(x1, x2, ('nngp', 'ntk'))):
            g = g.cpu().numpy().astype(np.float64) * 2. ** -(e1 + e2)
            assert np.max(np.abs(g - w)) <= 1e-5 * np.max(np.abs(w))
