"""The fused chain at the edges of its launch rule: few pairs are split over the lines of the
last segment, many share CTAs; self pairs; every segment count."""
import math

import numpy as np
import pytest
import torch

from oracle import nt_oracle as o

pytestmark = pytest.mark.gpu


def _net(m, name):
    c = lambda b=0.: m.Conv(1, (3, 3), padding='SAME', W_std=math.sqrt(2.), b_std=b)
    pool = lambda: m.AvgPool((2, 2), (2, 2))
    return {
        'myrtle5': lambda: [c(), m.Relu(), c(), m.Relu(), pool(), c(), m.Relu(), pool(), c(),
                            m.Relu(), pool(), pool(), pool(), m.Flatten(), m.Dense(1)],
        'one': lambda: [c(.1), m.Erf(), c(.1), m.Relu(), m.Flatten(), m.Dense(1), m.Relu(),
                        m.Dense(1)],
        'two': lambda: [c(.1), m.Relu(), pool(), c(.1), m.LeakyRelu(.2), c(.1), m.GlobalAvgPool(),
                        m.Dense(1)],
        'empty_segment': lambda: [c(), m.Relu(), pool(), pool(), c(), m.Relu(), m.GlobalAvgPool()],
        'rare': lambda: [c(.1), m.Gelu(), pool(), c(.1), m.Sin(), pool(), c(.1), m.Rbf(.3),
                         m.GlobalAvgPool()],
        'standard': lambda: [m.Conv(1, (3, 3), padding='SAME', W_std=1.3, b_std=.1,
                                    parameterization='standard'), m.Relu(), pool(), c(.1),
                             m.Relu(), pool(), c(.1), m.Relu(), m.GlobalAvgPool()],
    }[name]()


def _images(n, k, seed):
    return np.random.default_rng(seed).standard_normal((n, 32, 32, k)).astype(np.float32)


@pytest.mark.parametrize('name', ['myrtle5', 'one', 'two', 'empty_segment', 'rare', 'standard'])
@pytest.mark.parametrize('k', [1, 3])
def test_against_oracle(nt, name, k):
    x1, x2 = _images(1, k, 1), _images(2, k, 2)
    x2[1] = x1[0]  # a self pair in a block
    kf, ko = nt.stax.serial(*_net(nt.stax, name))[2], o.serial(*_net(o, name))
    for b in (x2, None):
        a = x1 if b is not None else x2
        got, want = kf(a, b, ('nngp', 'ntk', 'cov1')), ko(a, b, ('nngp', 'ntk', 'cov1'))
        for g, w in zip(got, want):
            assert np.max(np.abs(g.cpu().numpy() - w) / np.abs(w)) < 1e-5


@pytest.mark.parametrize('name', ['myrtle5', 'one', 'two', 'empty_segment'])
@pytest.mark.parametrize('n1,n2', [(1, 1), (1, 2), (2, 9), (1, 19), (4, 5), (6, 6), (1, 38),
                                   (5, 10), (3, 17), (1, 75), (2, 38), (7, 11)])
def test_split_pairs(nt, name, n1, n2):
    """The pairs of a small block (152 // pairs parts each, up to 8) against the same pairs in
    a launch of one part per pair: the same entries summed in another order, at most 2^20 of
    one sign in trees of depth < 100 (100 u < 1e-5; in practice a few u)."""
    x1, x2 = torch.from_numpy(_images(16, 3, 3)).cuda(), torch.from_numpy(_images(75, 3, 4)).cuda()
    kf = nt.stax.serial(*_net(nt.stax, name))[2]
    whole = kf(x1, x2, ('nngp', 'ntk'))
    part = kf(x1[:n1], x2[:n2], ('nngp', 'ntk'))
    for p, w in zip(part, whole):
        torch.testing.assert_close(p, w[:n1, :n2], rtol=1e-5, atol=0.)
    # and K(x, x), whose pairs are the triangle
    tri = kf(x2[:min(n2, 16)], None, ('nngp', 'ntk'))
    full = kf(x2[:20], None, ('nngp', 'ntk'))
    for p, w in zip(tri, full):
        m = p.shape[0]
        assert torch.equal(p, p.t())
        torch.testing.assert_close(p, w[:m, :m], rtol=1e-5, atol=0.)


def test_abi_without_a_workspace(nt):
    """ntg_chain_fwd and ntg_chain_fwd_sym bring their own scratch."""
    import ctypes
    from nt_gb300 import _chain, _lib as L, _ops as O
    from nt_gb300.stax import _Ctx
    kf = nt.stax.serial(*_net(nt.stax, 'myrtle5'))[2]
    x = torch.from_numpy(_images(6, 3, 5)).cuda()
    plan = _chain.plan_chain(kf.specs, tuple(x.shape), False)
    pg = _chain._program(plan, 3, _Ctx('fp32'))
    var = O.chain_vars(pg, x)
    want = [torch.empty((6, 6), device='cuda') for _ in range(2)]
    got = [torch.empty((6, 6), device='cuda') for _ in range(2)]
    O.chain_fwd(pg, x, x, 0, 6, 0, 6, var, var, want[0], want[1], 6)
    L.call('ntg_chain_fwd', L.stream(), ctypes.byref(pg), L.ptr(x), L.ptr(x), 0, 6, 0, 6,
           L.ptr(var), L.ptr(var), L.ptr(got[0]), L.ptr(got[1]), 6)
    assert all(torch.equal(g, w) for g, w in zip(got, want))
    O.chain_fwd_sym(pg, x, 0, 6, 0, 6, var, want[0], want[1], 6)
    L.call('ntg_chain_fwd_sym', L.stream(), ctypes.byref(pg), L.ptr(x), 0, 6, 0, 6, L.ptr(var),
           L.ptr(got[0]), L.ptr(got[1]), 6)
    assert all(torch.equal(g, w) for g, w in zip(got, want))
