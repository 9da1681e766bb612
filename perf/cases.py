"""The work that users of nt_gb300 have it do, as cases that can be timed and checked.

A case is a dict of plain values; `prepare` makes the inputs a program holds before the
call, `run` is one pass through the public entry points (``stax`` kernel functions,
``nt.batch``, ``nt.predict``), `exact` the same outputs from plain float64 torch.

Kinds
  fcn    kernel_fn of a fully connected network on flat inputs
  chain  nt.batch of a Myrtle conv network on 32 x 32 images (square K(x, x) or a block)
  cnn    kernel_fn of a pooled conv network on other image sizes (layer by layer)
  ds     kernel_fn of a conv network without pooling (diagonal-spatial kernels)
  krr    kernel-ridge loss of the Myrtle-5 NTK and its gradient in the support images
  nll    NNGP marginal likelihood of an FCN and its gradient in (W_std, b_std)
  inf    gradient_descent_mse predictions at infinite time (factorisation and solve)
  time   gradient_descent_mse predictions at finite times (eigenbasis)
"""
import math

import torch

import nt_gb300 as nt
from nt_gb300 import predict, stax

SQRT2 = math.sqrt(2.)


def listed():
    return [
        # a few flat samples against themselves: one active-learning or notebook step, where
        # the host path and the launches are all there is
        dict(name='fcn_small', kind='fcn', n1=24, n2=0, d=100, depth=2, act='relu', w=1.5,
             b=0.05, precision='fp32'),
        # the FCN of the first benchmark configuration: 256 x 256 MNIST-sized vectors
        dict(name='fcn_256', kind='fcn', n1=256, n2=256, d=784, depth=2, act='relu', w=1.5,
             b=0.05, precision='fp32'),
        # test-train block of flattened CIFAR images for an erf network, ragged, mixed form
        dict(name='fcn_large_mixed', kind='fcn', n1=4001, n2=1999, d=3072, depth=3, act='erf',
             w=1.3, b=0.2, precision='mixed'),
        # a handful of new images against a handful of anchors: the small call of a server
        dict(name='myrtle5_few', kind='chain', net='myrtle5', n1=5, n2=7, precision='fp32',
             batch=16),
        # the headline job's step: K(x, x) of CIFAR-sized images, plain FP32
        dict(name='myrtle5_square', kind='chain', net='myrtle5', n1=120, n2=0,
             precision='fp32', batch=100),
        # ragged test-train block of the deep network in the mixed form
        dict(name='myrtle10_block_mixed', kind='chain', net='myrtle10', n1=61, n2=97,
             precision='mixed', batch=96),
        # MNIST-sized images with a pooled conv network: full-spatial kernels layer by layer
        dict(name='cnn28', kind='cnn', size=28, chan=1, filt=3, act='relu', readout='flatten',
             n1=19, n2=24),
        # conv network with a flattening readout: only the spatial diagonal is carried
        dict(name='cnn_diagonal', kind='ds', size=32, chan=3, filt=3, act='relu', depth=3,
             n1=100, n2=90),
        # dataset distillation step: loss of a support set on targets, gradient in the images
        dict(name='krr_grad', kind='krr', n1=24, n2=40, precision='fp32'),
        # hyper-parameter step of a GP on 4096 flattened CIFAR images
        dict(name='nll_4096', kind='nll', n1=4096, d=3072, depth=3, m=10, precision='fp32'),
        # closed-form training on 5000 points, ten classes, predictions for 500
        dict(name='mse_inf_5000', kind='inf', n1=5000, n2=500, m=10),
        # learning curve: predictions along training time on 500 points
        dict(name='mse_time_500', kind='time', n1=500, n2=100, m=10, times=6),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['fcn', 'fcn', 'chain', 'chain', 'cnn', 'ds', 'krr', 'nll', 'inf', 'time'])
    if kind == 'fcn':
        return dict(kind=kind, n1=_log(rng, 8, 4001), n2=rng.choice([0, _log(rng, 8, 1999)]),
                    d=_log(rng, 16, 3072), depth=rng.randint(1, 4),
                    act=rng.choice(['relu', 'erf']), w=round(rng.uniform(1., 2.), 3),
                    b=round(rng.uniform(0., 0.2), 3), precision=rng.choice(['fp32', 'mixed']))
    if kind == 'chain':
        net = rng.choice(['myrtle5', 'myrtle7', 'myrtle10'])
        n1 = _log(rng, 1, 100)
        return dict(kind=kind, net=net, n1=n1, n2=rng.choice([0, _log(rng, 1, 5900 // n1)]),
                    precision=rng.choice(['fp32', 'mixed']), batch=rng.choice([16, 96, 100, 128]))
    if kind == 'cnn':
        size = rng.randint(8, 28)
        pairs = max(2, min(1600, int(19 * 24 * (28 / size) ** 4)))
        n1 = _log(rng, 1, min(pairs, 48))
        return dict(kind=kind, size=size, chan=rng.choice([1, 3]), filt=rng.choice([3, 3, 5]),
                    act=rng.choice(['relu', 'erf']), readout=rng.choice(['flatten', 'mean']),
                    n1=n1, n2=max(1, _log(rng, 1, max(1, pairs // n1))))
    if kind == 'ds':
        size = rng.randint(8, 40)
        pairs = int(9000 * (32 / size) ** 2)
        n1 = _log(rng, 4, 300)
        return dict(kind=kind, size=size, chan=rng.choice([1, 3]), filt=rng.choice([3, 3, 5]),
                    act=rng.choice(['relu', 'erf']), depth=rng.randint(1, 4), n1=n1,
                    n2=max(1, _log(rng, 4, max(4, min(300, pairs // n1)))))
    if kind == 'krr':
        return dict(kind=kind, n1=rng.randint(3, 24), n2=rng.randint(1, 40),
                    precision=rng.choice(['fp32', 'mixed']))
    if kind == 'nll':
        return dict(kind=kind, n1=_log(rng, 64, 4096), d=_log(rng, 32, 3072),
                    depth=rng.randint(1, 3), m=rng.randint(1, 10),
                    precision=rng.choice(['fp32', 'mixed']))
    if kind == 'inf':
        return dict(kind=kind, n1=_log(rng, 48, 5000), n2=_log(rng, 1, 500), m=rng.randint(1, 24))
    return dict(kind='time', n1=_log(rng, 16, 500), n2=_log(rng, 1, 100), m=rng.randint(1, 10),
                times=rng.randint(1, 6))


# ---------------------------------------------------------------------------
# Networks: one plain description, built from stax layers for the framework and
# walked by the float64 rules below.
# ---------------------------------------------------------------------------


def _layers(case):
    kind = case['kind']
    if kind in ('fcn', 'nll'):
        w, b = case.get('w', 1.5), case.get('b', 0.1)
        act = case.get('act', 'relu')
        out = []
        for _ in range(case['depth']):
            out += [('dense', w, b), (act,)]
        return out + [('dense', w, b)]
    if kind in ('chain', 'krr'):
        blocks, tail = {'myrtle5': ((2, 1, 1), 'pools'), 'myrtle7': ((2, 2, 2), 'pools'),
                        'myrtle10': ((3, 3, 3), 'mean')}[case.get('net', 'myrtle5')]
        out = []
        for i, n in enumerate(blocks):
            out += [('conv', 3, SQRT2, 0.), ('relu',)] * n
            if i < 2:
                out.append(('pool',))
        out += [('pool',)] * 3 + [('flatten',)] if tail == 'pools' else [('mean',)]
        return out + [('dense', SQRT2, 0.)]
    act = case['act']
    if kind == 'cnn':
        out = [('conv', case['filt'], SQRT2, 0.1), (act,), ('conv', case['filt'], SQRT2, 0.1),
               (act,), ('pool',), ('conv', case['filt'], SQRT2, 0.1), (act,),
               (case['readout'],)]
        return out + [('dense', SQRT2, 0.1)]
    return [('conv', case['filt'], SQRT2, 0.1), (act,)] * case['depth'] + [
        ('flatten',), ('dense', SQRT2, 0.1)]


def _network(layers):
    made = {'dense': lambda w, b: stax.Dense(1, W_std=w, b_std=b),
            'conv': lambda f, w, b: stax.Conv(1, (f, f), padding='SAME', W_std=w, b_std=b),
            'relu': stax.Relu, 'erf': stax.Erf, 'flatten': stax.Flatten,
            'mean': stax.GlobalAvgPool, 'pool': lambda: stax.AvgPool((2, 2), (2, 2))}
    return stax.serial(*[made[la[0]](*la[1:]) for la in layers])[2]


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device='cuda').manual_seed(seed)


def _images(gen, n, size, chan):
    """Images standardised per channel, as data loaders hand them over."""
    x = torch.randn((n, size, size, chan), generator=gen, device='cuda')
    return (x - x.mean((0, 1, 2))) / x.std((0, 1, 2))


def _one_hot(gen, n, m):
    y = torch.randint(0, m, (n,), generator=gen, device='cuda')
    return torch.nn.functional.one_hot(y, m).float()


def _regression(gen, n1, n2, m):
    """Train-train and test-train NTK of a one-hidden-layer ReLU network on random unit
    inputs in 64 dimensions (closed form), and m noisy targets that are smooth functions of
    the inputs, float32."""
    x = torch.randn((n1 + n2, 64), generator=gen, device='cuda', dtype=torch.float64)
    x = x / x.norm(dim=1, keepdim=True)
    c = (x @ x[:n1].t()).clamp(-1., 1.)
    c[:n1].fill_diagonal_(1.)
    th = torch.acos(c)
    dot = (math.pi - th) / math.pi
    k = (torch.sin(th) / math.pi + c * dot) + c * dot
    k = k.float()
    teacher = torch.randn((64, m), generator=gen, device='cuda', dtype=torch.float64)
    noise = torch.randn((n1, m), generator=gen, device='cuda', dtype=torch.float64)
    y = torch.tanh(x[:n1] @ teacher) + 0.05 * noise
    return k[:n1].contiguous(), k[n1:].contiguous(), y.float()


def _inputs(case, seed):
    gen = _gen(seed)
    kind = case['kind']
    s = {}
    if kind == 'fcn':
        s['x1'] = torch.randn((case['n1'], case['d']), generator=gen, device='cuda')
        if case['n2']:
            s['x2'] = torch.randn((case['n2'], case['d']), generator=gen, device='cuda')
    elif kind == 'chain':
        s['x1'] = _images(gen, case['n1'], 32, 3)
        if case['n2']:
            s['x2'] = _images(gen, case['n2'], 32, 3)
    elif kind in ('cnn', 'ds'):
        s['x1'] = _images(gen, case['n1'], case['size'], case['chan'])
        s['x2'] = _images(gen, case['n2'], case['size'], case['chan'])
    elif kind == 'krr':
        s['x1'] = _images(gen, case['n1'], 32, 3)
        s['x2'] = _images(gen, case['n2'], 32, 3)
        s['y1'], s['y2'] = _one_hot(gen, case['n1'], 10), _one_hot(gen, case['n2'], 10)
    elif kind == 'nll':
        s['x1'] = torch.randn((case['n1'], case['d']), generator=gen, device='cuda')
        s['y1'] = torch.randn((case['n1'], case['m']), generator=gen, device='cuda')
    else:
        s['k'], s['k_td'], s['y1'] = _regression(gen, case['n1'], case['n2'], case['m'])
        if kind == 'time':
            s['t'] = [10. ** (1. + 3. * i / max(1, case['times'] - 1))
                      for i in range(case['times'])]
    return s


KRR_REG = 1e-1   # relative ridge of the kernel-ridge step
NLL_REG = 1e-1   # relative noise variance of the marginal likelihood
MSE_REG = 1e-4


def prepare(case, seed):
    s = _inputs(case, seed)
    s['case'] = case
    kind = case['kind']
    if kind in ('fcn', 'chain', 'cnn', 'ds', 'krr'):
        s['kernel_fn'] = _network(_layers(case))
    if kind == 'chain':
        s['kernel_fn'] = nt.batch(s['kernel_fn'], batch_size=case['batch'])
    elif kind == 'krr':
        s['kernel_fn'] = nt.batch(s['kernel_fn'], batch_size=32, recompute_tile=32)
    elif kind == 'nll':
        s['w'] = torch.tensor(1.5, device='cuda', requires_grad=True)
        s['b'] = torch.tensor(0.1, device='cuda', requires_grad=True)
        s['kernel_fn'] = _network([(la[0], s['w'], s['b']) if la[0] == 'dense' else la
                                   for la in _layers(case)])
    return s


def run(s):
    case = s['case']
    kind = case['kind']
    if kind in ('fcn', 'chain', 'cnn', 'ds'):
        k = s['kernel_fn'](s['x1'], s.get('x2'), ('nngp', 'ntk'),
                           precision=case.get('precision', 'fp32'))
        return {'nngp': k.nngp, 'ntk': k.ntk}
    if kind == 'krr':
        x = s['x1'].detach().requires_grad_(True)
        kss = s['kernel_fn'](x, None, 'ntk', precision=case['precision'])
        kts = s['kernel_fn'](s['x2'], x, 'ntk', precision=case['precision'])
        pred = predict.kernel_ridge_predict(kts, kss, s['y1'], diag_reg=KRR_REG)
        loss = ((s['y2'] - pred) ** 2).sum()
        (g,) = torch.autograd.grad(loss, (x,))
        return {'loss': loss.detach(), 'prediction': pred.detach(), 'grad': g}
    if kind == 'nll':
        k = s['kernel_fn'](s['x1'], None, 'nngp', precision=case['precision'])
        nll = predict.negative_log_likelihood(k, s['y1'], diag_reg=NLL_REG)
        gw, gb = torch.autograd.grad(nll, (s['w'], s['b']))
        return {'nll': nll.detach(), 'grad_w': gw, 'grad_b': gb}
    fn = predict.gradient_descent_mse(s['k'], s['y1'], diag_reg=MSE_REG)
    if kind == 'inf':
        train, test = fn(None, 0., 0., s['k_td'])
    else:
        train, test = fn(s['t'], 0., 0., s['k_td'])
    return {'train': train, 'test': test}


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------

# operations of an activation rule per kernel entry (nngp and ntk)
ACT_FLOPS = 35.


def work(case):
    kind = case['kind']
    n1, n2 = case['n1'], case.get('n2', 0) or case['n1']
    if kind == 'fcn':
        pairs = n1 * (n1 + 1) / 2 if not case['n2'] else n1 * n2
        return {'bytes': 4. * (n1 + (case['n2'] or 0)) * case['d'] + 8. * n1 * n2,
                'flops': pairs * (2. * case['d'] + (ACT_FLOPS + 4.) * case['depth'])}
    if kind == 'chain':
        pairs = n1 * (n1 + 1) / 2 if not case['n2'] else n1 * n2
        per = _spatial_flops(_layers(case), 32, 3, False)
        return {'bytes': 4. * 3072 * (n1 + case['n2']) + 8. * n1 * n2, 'flops': pairs * per}
    if kind in ('cnn', 'ds'):
        per = _spatial_flops(_layers(case), case['size'], case['chan'], kind == 'ds')
        image = case['size'] ** 2 * case['chan']
        return {'bytes': 4. * image * (n1 + n2) + 8. * n1 * n2, 'flops': n1 * n2 * per}
    if kind == 'krr':
        pairs = n1 * (n1 + 1) / 2 + n1 * n2
        # the forward, its evaluation again tile by tile, and the adjoints (twice the forward)
        return {'bytes': 4. * 3072 * (2 * n1 + n2),
                'flops': 4. * pairs * _spatial_flops(_layers(case), 32, 3, False)}
    if kind == 'nll':
        # half the Gram, the rules and their adjoints, the factorisation and the inverse
        return {'bytes': 4. * n1 * case['d'],
                'flops': 1. * n1 * n1 * case['d'] + 3. * n1 * n1 * ACT_FLOPS * case['depth']
                + 1. * n1 ** 3}
    rows = case['n1'] + case['n2']
    if kind == 'inf':
        return {'bytes': 4. * rows * n1 + 8. * rows * case['m'],
                'flops': n1 ** 3 / 3. + 4. * n1 * n1 * case['m'] + 2. * case['n2'] * n1 * case['m']}
    return {'bytes': 4. * rows * n1 + 4. * rows * case['m'] * case['times'],
            'flops': 9. * n1 ** 3 + 2. * case['times'] * case['m'] * n1 * (n1 + rows)}


def _spatial_flops(layers, size, chan, diagonal):
    """Operations per pair: the input covariance, then each layer's entries once."""
    dim = 2 if diagonal else 4
    total, first = 2. * chan * size ** dim, True
    for la in layers:
        if la[0] == 'conv':
            total += size ** dim * (2. * la[1] * (1 if first else 2) + 4.)
            first = False
        elif la[0] in ('relu', 'erf'):
            total += size ** dim * ACT_FLOPS
        elif la[0] == 'pool':
            total += 2. * size ** dim
            size //= 2
        elif la[0] in ('flatten', 'mean'):
            total += 2. * (size ** dim if la[0] == 'mean' or diagonal else size ** 2)
            break
    return total


# ---------------------------------------------------------------------------
# The same outputs in float64 with plain torch
# ---------------------------------------------------------------------------


def _act(fn, q, t, v1, v2):
    """nngp, ntk after an activation, from the kernels and the variances before it. The
    square root's derivative is taken as zero where its argument vanishes."""
    if fn == 'relu':
        d = v1 * v2 - q * q
        ok = d > 1e-30
        s = torch.where(ok, d, torch.ones_like(d)).sqrt() * ok
        zero = (q == 0) & (s == 0)
        th = torch.atan2(s, torch.where(zero, torch.ones_like(q), q))
        dot = 0.5 - torch.where(zero, torch.full_like(q, math.pi / 2), th) / (2 * math.pi)
        return s / (2 * math.pi) + dot * q, None if t is None else t * dot
    s = ((1 + 2 * v1) * (1 + 2 * v2) - 4 * q * q).clamp(min=0.).sqrt()
    return 2 / math.pi * torch.atan2(2 * q, s), None if t is None else t * (4 / math.pi) / s


def _window(x, f, axes):
    """Sum over the f centred shifts of the given axes together, zero padded."""
    out = x
    for k in range(1, f // 2 + 1):
        for up in (True, False):
            y = x
            for a in axes:
                pad = torch.zeros_like(y.narrow(a, 0, k))
                part = y.narrow(a, 0 if up else k, y.shape[a] - k)
                y = torch.cat([pad, part] if up else [part, pad], dim=a)
            out = out + y
    return out


def _halve(x, axis):
    n = x.shape[axis] // 2
    x = x.narrow(axis, 0, 2 * n).unflatten(axis, (n, 2))
    return (x.select(axis + 1, 0) + x.select(axis + 1, 1)) / 2


def _spatial(layers, xa, xb, variances, diagonal):
    """Readout (nngp, ntk) of the pairs xa[p], xb[p], images [P, H, W, C]. `variances`: the
    pre-activation variance maps of both sides per activation as [P, H, W], or None for self
    pairs, whose own maps are then returned as well."""
    chan = xa.shape[-1]
    if diagonal:
        q = sum(xa[..., c] * xb[..., c] for c in range(chan)) / chan
        hw = ((1,), (2,))
    else:
        q = sum(xa[:, :, None, :, None, c] * xb[:, None, :, None, :, c]
                for c in range(chan)) / chan
        hw = ((1, 2), (3, 4))
    t, maps = None, []
    for la in layers:
        if la[0] in ('conv', 'dense'):
            if la[0] == 'conv':
                for axes in hw:
                    q = _window(q, la[1], axes)
                    t = None if t is None else _window(t, la[1], axes)
                q = q / la[1] ** 2
                t = None if t is None else t / la[1] ** 2
            w2, b2 = la[-2] ** 2, la[-1] ** 2
            q = w2 * q + b2
            t = q if t is None else w2 * t + q
        elif la[0] in ('relu', 'erf'):
            if variances is None:
                v = q if diagonal else q.diagonal(dim1=1, dim2=2).diagonal(dim1=1, dim2=2)
                va = vb = v
                maps.append(v)
            else:
                va, vb = variances[0][len(maps)], variances[1][len(maps)]
                maps.append(None)
            if not diagonal:
                va, vb = va[:, :, None, :, None], vb[:, None, :, None, :]
            q, t = _act(la[0], q, t, va, vb)
        elif la[0] == 'pool':
            for a in (1, 2, 3, 4):
                q, t = _halve(q, a), _halve(t, a)
        elif la[0] == 'mean' or diagonal:
            q, t = q.flatten(1).mean(1), t.flatten(1).mean(1)
        else:
            q, t = (z.diagonal(dim1=1, dim2=2).diagonal(dim1=1, dim2=2).flatten(1).mean(1)
                    for z in (q, t))
    return q, t, maps


def _self_maps(layers, x, diagonal, chunk):
    parts = [_spatial(layers, x[i:i + chunk], x[i:i + chunk], None, diagonal)[2]
             for i in range(0, x.shape[0], chunk)]
    return [torch.cat(p) for p in zip(*parts)]


def _pair_kernels(layers, x1, x2, maps1, maps2, i, j, diagonal):
    v = [m[i] for m in maps1], [m[j] for m in maps2]
    return _spatial(layers, x1[i], x2[j], v, diagonal)[:2]


def _grid(n1, n2, symmetric):
    i, j = torch.meshgrid(torch.arange(n1), torch.arange(n2), indexing='ij')
    keep = (i <= j) if symmetric else torch.ones_like(i, dtype=torch.bool)
    return i[keep].cuda(), j[keep].cuda()


def _conv_kernels(layers, x1, x2, diagonal):
    """K(x1, x2) (x2 None: K(x1, x1)) of a conv network, pair chunk by pair chunk."""
    symmetric = x2 is None
    xb = x1 if symmetric else x2
    entries = x1.shape[1] ** (2 if diagonal else 4)
    chunk = max(1, (1 << 26) // entries)
    m1 = _self_maps(layers, x1, diagonal, chunk)
    m2 = m1 if symmetric else _self_maps(layers, xb, diagonal, chunk)
    i, j = _grid(x1.shape[0], xb.shape[0], symmetric)
    out = torch.zeros((2, x1.shape[0], xb.shape[0]), dtype=torch.float64, device='cuda')
    for p in range(0, i.numel(), chunk):
        a, b = i[p:p + chunk], j[p:p + chunk]
        out[:, a, b] = torch.stack(_pair_kernels(layers, x1, xb, m1, m2, a, b, diagonal))
    if symmetric:
        out = torch.triu(out) + torch.triu(out, 1).transpose(1, 2)
    return out[0], out[1]


def _flat_kernels(layers, x1, x2):
    """nngp, ntk of an FCN; layers may hold tensors for W_std and b_std."""
    xb = x1 if x2 is None else x2
    d = x1.shape[1]
    q, t = x1 @ xb.t() / d, None
    v1 = q.diagonal() if x2 is None else (x1 * x1).sum(1) / d
    v2 = v1 if x2 is None else (x2 * x2).sum(1) / d
    for la in layers:
        if la[0] == 'dense':
            w2, b2 = la[1] ** 2, la[2] ** 2
            q, v1, v2 = w2 * q + b2, w2 * v1 + b2, w2 * v2 + b2
            t = q if t is None else w2 * t + q
        else:
            q, t = _act(la[0], q, t, v1[:, None], v2[None, :])
            if la[0] == 'relu':
                v1, v2 = v1 / 2, v2 / 2
            else:
                v1, v2 = (2 / math.pi * torch.asin(2 * v / (1 + 2 * v)) for v in (v1, v2))
    return q, t


def _ridge(k, reg):
    n = k.shape[0]
    return k + reg * k.diagonal().sum() / n * torch.eye(n, dtype=k.dtype, device=k.device)


def _exact_krr(case, s):
    layers = _layers(case)
    xs, xt = s['x1'].double(), s['x2'].double()
    kss, kts = (_conv_kernels(layers, a, b, False)[1].requires_grad_(True)
                for a, b in ((xs, None), (xt, xs)))
    pred = kts @ torch.linalg.solve(_ridge(kss, KRR_REG), s['y1'].double())
    loss = ((s['y2'].double() - pred) ** 2).sum()
    gss, gts = torch.autograd.grad(loss, (kss, kts))
    # one tile of pairs at a time: its kernels again with a graph, its share of the gradient
    grad = torch.zeros_like(xs)
    for g, rows in ((gss, xs), (gts, xt)):
        for r in range(0, rows.shape[0], 8):
            for c in range(0, xs.shape[0], 8):
                a = rows[r:r + 8].clone().requires_grad_(True)
                b = xs[c:c + 8].clone().requires_grad_(True)
                ma, mb = (_spatial(layers, x, x, None, False)[2] for x in (a, b))
                i, j = _grid(a.shape[0], b.shape[0], False)
                t = _pair_kernels(layers, a, b, ma, mb, i, j, False)[1]
                ga, gb = torch.autograd.grad((t * g[r:r + 8, c:c + 8].reshape(-1)).sum(), (a, b))
                if rows is xs:
                    grad[r:r + 8] += ga
                grad[c:c + 8] += gb
    return {'loss': loss.detach(), 'prediction': pred.detach(), 'grad': grad}


def exact(case, seed):
    s = _inputs(case, seed)
    kind = case['kind']
    if kind == 'fcn':
        with torch.no_grad():
            x2 = s['x2'].double() if 'x2' in s else None
            q, t = _flat_kernels(_layers(case), s['x1'].double(), x2)
        return {'nngp': q, 'ntk': t}
    if kind in ('chain', 'cnn', 'ds'):
        with torch.no_grad():
            x2 = s['x2'].double() if 'x2' in s else None
            q, t = _conv_kernels(_layers(case), s['x1'].double(), x2, kind == 'ds')
        return {'nngp': q, 'ntk': t}
    if kind == 'krr':
        return _exact_krr(case, s)
    if kind == 'nll':
        n, m = case['n1'], case['m']
        w = torch.tensor(1.5, device='cuda').double().requires_grad_(True)
        b = torch.tensor(0.1, device='cuda').double().requires_grad_(True)
        q, _ = _flat_kernels([(la[0], w, b) if la[0] == 'dense' else la
                              for la in _layers(case)], s['x1'].double(), None)
        y = s['y1'].double()
        chol = torch.linalg.cholesky(_ridge(q, NLL_REG))
        alpha = torch.cholesky_solve(y, chol)
        nll = (0.5 * (y * alpha).sum() + m * chol.diagonal().log().sum()
               + 0.5 * n * m * math.log(2 * math.pi))
        gw, gb = torch.autograd.grad(nll, (w, b))
        return {'nll': nll.detach(), 'grad_w': gw, 'grad_b': gb}
    k, ktd, y = s['k'].double(), s['k_td'].double(), s['y1'].double()
    a = _ridge(k, MSE_REG)
    if kind == 'inf':
        return {'train': y, 'test': ktd @ torch.linalg.solve(a, y)}
    ev, q = torch.linalg.eigh(a)
    t = torch.tensor(s['t'], dtype=torch.float64, device='cuda')[:, None, None]
    decay = -torch.expm1(-ev[None, :, None] * t / y.numel())
    proj = decay * (q.t() @ y)[None]
    return {'train': q @ proj, 'test': ktd @ (q @ (proj / ev[None, :, None]))}
