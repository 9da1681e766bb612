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
