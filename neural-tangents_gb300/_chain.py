"""Planner and driver of the fused whole-network kernel (ntg_chain_fwd).

A ``serial`` network whose spatial part is a Myrtle-style chain

    [Conv(3x3, SAME, stride 1) + activation?] x n0, AvgPool(2, 2),
    [Conv + activation?] x n1, AvgPool(2, 2), ..., readout

on 32x32 inputs with at most 4 channels is evaluated per (x1[i], x2[j]) pair
in one CTA with nothing but the readout written to HBM. The readout is
GlobalAvgPool (after any number of AvgPool(2, 2)), AvgPool(2, 2) down to 1x1
followed by Flatten, or Flatten right after the last segment. The activation
rules need the per-sample pre-activation variances of every conv layer; those
come from a kernel of their own (ntg_chain_vars), one CTA per sample. Layers after the readout run through the
ordinary layer rules on [N1, N2] kernels. Anything else falls back to the
layer-by-layer path.
"""
from __future__ import annotations

import dataclasses
import math
from typing import Optional

import torch

from . import _lib as L
from . import _ops as O
from .kernel import Kernel
from .stax import Padding, _Ctx, _act_struct, _affine_struct, _conv_geometry, _pads

S0 = 32


@dataclasses.dataclass
class ChainPlan:
    nseg: int
    nconv: list          # conv layers per segment
    convs: list          # (conv params, act params | None, input channels)
    readout: int         # 0 = mean of all entries, 1 = mean of the spatial diagonal
    n_rpools: int        # AvgPools between the last segment and the readout
    readout_kind: str    # 'gpool' | 'flatten'
    post: list           # LayerSpecs after the readout
    spatial: list        # LayerSpecs up to and including the readout
    is_gaussian: bool


def _is_pool2(s) -> bool:
    p = s.params
    return (s.kind == 'pool' and p['pool'] == 'avg' and tuple(p['window_shape']) == (2, 2)
            and tuple(p['strides']) == (2, 2) and p['padding'] in (Padding.VALID, Padding.SAME))


def plan_chain(specs, x_shape, diagonal_spatial: bool) -> Optional[ChainPlan]:
    if diagonal_spatial or len(x_shape) != 4 or tuple(x_shape[1:3]) != (S0, S0):
        return None
    if not 1 <= x_shape[3] <= 4:
        return None
    specs = [s for s in specs if s.kind != 'identity']
    ridx = next((i for i, s in enumerate(specs) if s.kind in ('gpool', 'flatten')), None)
    if ridx is None:
        return None
    spatial, post = specs[:ridx], specs[ridx + 1:]
    readout_spec = specs[ridx]
    if any(s.kind not in ('dense', 'act') for s in post):
        return None
    last_conv = max((i for i, s in enumerate(spatial) if s.kind == 'conv'), default=None)
    if last_conv is None or spatial[0].kind != 'conv':
        return None
    nconv, convs = [0], []
    shape = tuple(x_shape)
    i = 0
    is_gaussian = False
    while i < len(spatial):
        s = spatial[i]
        if s.kind == 'conv':
            p = s.params
            if (tuple(p['filter_shape']) != (3, 3) or tuple(p['strides']) != (1, 1)
                    or p['padding'] != Padding.SAME or nconv[-1] == 3):
                return None
            act = None
            cin = shape[-1]
            shape = s.shape_fn(shape)
            is_gaussian = True
            if i + 1 < len(spatial) and spatial[i + 1].kind == 'act':
                act = spatial[i + 1].params
                if act.get('do_stabilize'):
                    return None  # the stabilised ABRelu rescales by the pre-activation maximum
                is_gaussian = False
                i += 1
            convs.append((p, act, cin))
            nconv[-1] += 1
        elif _is_pool2(s):
            if i < last_conv:
                nconv.append(0)
                if len(nconv) > 3:
                    return None
            else:
                break
            shape = s.shape_fn(shape)
        else:
            return None
        i += 1
    rpools = spatial[i:]
    if not all(_is_pool2(s) for s in rpools):
        return None
    nseg = len(nconv)
    s_last = S0 >> (nseg - 1)
    n_rp = len(rpools)
    if s_last >> n_rp < 1 or (s_last % (1 << n_rp)) != 0:
        return None
    if readout_spec.kind == 'gpool':
        if readout_spec.params['pool'] != 'avg':
            return None
        readout = 0
    else:
        if n_rp == 0:
            readout = 1
        elif s_last >> n_rp == 1:
            readout = 0
        else:
            return None
        is_gaussian = False
    return ChainPlan(nseg=nseg, nconv=nconv, convs=convs, readout=readout, n_rpools=n_rp,
                     readout_kind=readout_spec.kind, post=post, spatial=specs[:ridx + 1],
                     is_gaussian=is_gaussian)


def _program(plan: ChainPlan, channels: int, ctx: _Ctx) -> L.Chain:
    pg = L.Chain()
    pg.nseg = plan.nseg
    pg.s0 = S0
    pg.channels = channels
    pg.readout = plan.readout
    for sgi in range(plan.nseg):
        pg.nconv[sgi] = plan.nconv[sgi]
    off = 0
    li = 0
    for sgi in range(plan.nseg):
        S = S0 >> sgi
        for _ in range(plan.nconv[sgi]):
            p, act, cin = plan.convs[li]
            fan = cin * 9 / p['s'][0] if p['parameterization'] == 'standard' else None
            pg.aff[li] = _affine_struct(p['W_std'], p['b_std'], p['parameterization'], fan)
            pg.act[li] = O.NO_ACT if act is None else _act_struct(act, ctx)
            pg.var_off[li] = off
            off += S * S
            li += 1
    pg.var_stride = off
    return pg


def self_chain(x: torch.Tensor, plan: ChainPlan, ctx: _Ctx):
    """Per-sample kernels through the chain: (variance maps [N, total], readout cov [N])."""
    pg = _program(plan, x.shape[-1], ctx)
    x = x.contiguous()
    var = O.chain_vars(pg, x)
    return var, O.chain_fwd_self(pg, x, var)


def try_fused(kfn, x1: torch.Tensor, x2: Optional[torch.Tensor], diagonal_spatial: bool,
              compute_ntk: bool, ctx: _Ctx, whole: bool = True) -> Optional[Kernel]:
    """The fused chain's Kernel, or None for another network; whole: every field of it is
    wanted, x1_is_x2 (an element-wise comparison of x1 and x2) and the per-sample kernels
    too, else nngp and ntk are."""
    plan = plan_chain(kfn.specs, tuple(x1.shape), diagonal_spatial)
    if plan is None or (x2 is not None and tuple(x2.shape[1:]) != tuple(x1.shape[1:])):
        return None
    k = run_fused(plan, x1, x2, ctx, x1_is_x2=None if whole else x2 is None, covs=whole)
    k = kfn.apply_kernel(k, ctx, specs=plan.post)
    if not compute_ntk:
        k = k.replace(ntk=None)
    return k


def run_fused(plan: ChainPlan, x1: torch.Tensor, x2: Optional[torch.Tensor], ctx: _Ctx,
              out: Optional[tuple] = None, rows=None, cols=None, selfs=None,
              x1_is_x2: Optional[bool] = None, covs: bool = True) -> Kernel:
    """Readout Kernel of the chain for all pairs of x1 x x2 (x2 None: x1 x x1).

    ``x1_is_x2`` given skips the element-wise comparison of x1 and x2 (a host
    synchronisation, not allowed while a CUDA graph is being captured). covs=False: nobody
    reads cov1 and cov2, which take the self pairs of a block (x1, x2); the layers after the
    readout do when there is an activation among them."""
    pg = _program(plan, x1.shape[-1], ctx)
    covs = covs or any(s.kind == 'act' for s in plan.post)
    cov1 = cov2 = None
    if selfs is None:
        if x2 is None:
            var1 = var2 = O.chain_vars(pg, x1)
        else:
            var1, var2 = O.chain_vars(pg, x1, x2)
    else:
        var1, cov1, var2, cov2 = selfs
    xb = x1 if x2 is None else x2
    n1, n2 = x1.shape[0], xb.shape[0]
    if out is None:
        out_q = torch.empty((n1, n2), device=x1.device, dtype=torch.float32)
        out_t = torch.empty((n1, n2), device=x1.device, dtype=torch.float32)
    else:
        out_q, out_t = out
    if x2 is None:
        # K(x, x): the pairs i <= j once, mirrored (one launch over the triangle)
        O.chain_fwd_sym(pg, x1, 0, n1, 0, n1, var1, out_q, out_t, n2)
    else:
        O.chain_fwd(pg, x1, xb, 0, n1, 0, n2, var1, var2, out_q, out_t, n2)
    if cov1 is None:
        # the readout kernel of a sample with itself: out_q's diagonal, or its own self pairs
        # (nobody reads them: zeros keep the Kernel's shape)
        if x2 is None:
            cov1 = torch.diagonal(out_q) if plan.post else torch.diagonal(out_q).clone()
        elif covs:
            cov1, cov2 = O.chain_fwd_self(pg, x1, var1), O.chain_fwd_self(pg, xb, var2)
        else:
            none = out_q.new_zeros(max(n1, n2))
            cov1, cov2 = none[:n1], none[:n2]
    shape1 = tuple(x1.shape)
    shape2 = tuple(xb.shape)
    for s in plan.spatial:
        shape1, shape2 = s.shape_fn(shape1), s.shape_fn(shape2)
    return Kernel(nngp=out_q, ntk=out_t, cov1=cov1, cov2=cov2,
                  x1_is_x2=(x2 is None or bool(torch.equal(x1, x2))) if x1_is_x2 is None
                  else bool(x1_is_x2), is_gaussian=plan.is_gaussian,
                  is_reversed=False, is_input=False, diagonal_batch=True, diagonal_spatial=False,
                  shape1=shape1, shape2=shape2)


# ---------------------------------------------------------------------------
# Conv networks on diagonal-spatial kernels and on bands around them (ntg_ds_chain)
# ---------------------------------------------------------------------------

DS_MAX_SMEM = 100 * 1024  # two CTAs per SM; larger images go layer by layer
# One CTA walks all planes of a pair's band, 3 - 9 us a plane with the layers of its level, so
# that many planes take long for few pairs. 49 (two 2 x 2 poolings, one of 4 x 4): 0.36 - 0.49 ms
# from 1 to 256 pairs of 8 x 8 to 32 x 32 images, against 1.1 - 2.9 ms by the layer rules or the
# whole-kernel chain; 225 (three poolings): 1.3 - 1.9 ms against 1.3 - 1.4 ms up to 32 pairs.
BAND_MAX_PLANES = 49
# Many pairs of small images fill the GPU either way. A plane then takes the band 4 - 6 ns
# whatever its size, an entry of a whole pair the layer rules 14 - 58 ps, and a call by these no
# less than 0.8 ms. So the band is for pairs of 128 entries a plane, or for as many planes as it
# takes in that time. 10^4 pairs, two 2 x 2 poolings, band and layer rules: 4 x 4 images 3.1 and
# 0.9 ms, 8 x 8 3.2 and 2.4, 12 x 12 3.4 and 5.6; one pooling: 4 x 4 0.54 and 0.83, 8 x 8 0.54
# and 2.4. Past 2^29 entries, 8 GB in the layer rules' tensors, it is the band again, which holds
# none of them.
BAND_ENTRIES_PER_PLANE = 128
BAND_SMALL_CALL = 1 << 17
BAND_LARGE_CALL = 1 << 29


def _narrow_band(specs, size, pairs: int) -> bool:
    """Whether the poolings leave a Flatten no more than BAND_MAX_PLANES offsets to see, and few
    enough for `pairs` pairs of images of that size."""
    d = [0] * len(size)
    pools = [s.params for s in specs if s.kind == 'pool']
    for p in reversed(pools):
        if len(p['window_shape']) != len(size):
            return False
        d = [s * x + k - 1 for x, k, s in zip(d, p['window_shape'], p['strides'])]
    planes = 1
    for x, m in zip(d, size):
        planes *= 2 * min(x, m - 1) + 1
    if not pools or planes > BAND_MAX_PLANES:
        return False
    entries = math.prod(size) ** 2
    return (BAND_ENTRIES_PER_PLANE * planes <= entries or pairs * planes <= BAND_SMALL_CALL
            or pairs * entries > BAND_LARGE_CALL)


def plan_ds(specs, x_shape, ctx: _Ctx, pools: bool = False, pairs: int = 1):
    """(program, layers after the readout, is_gaussian) of a serial network whose layers up to a
    Flatten / GlobalAvgPool / GlobalSumPool readout are stride-1 zero-padded Conv, Dense and
    activations, on [N, A, K] or [N, A, C, K] inputs; None for another network. pools: a network
    with AvgPool / SumPool layers among these, their windows inside the maps, and a Flatten
    readout, which sees a band around the spatial diagonal; pairs: of the call."""
    if len(x_shape) not in (3, 4):
        return None
    specs = [s for s in specs if s.kind != 'identity']
    ridx = next((i for i, s in enumerate(specs) if s.kind in ('gpool', 'flatten')), None)
    if not ridx or ridx > 3 * L.DS_MAX_LAYERS or specs[0].kind == 'act':
        return None
    if pools and (specs[ridx].kind != 'flatten' or not _narrow_band(
            specs[:ridx], x_shape[1:-1], pairs)):
        return None
    a, c = x_shape[1], x_shape[2] if len(x_shape) == 4 else 1
    pg = L.DsChain()
    pg.a, pg.c, pg.channels = a, c, x_shape[-1]
    shape, n, off, gaussian, plane, pooled = tuple(x_shape), 0, 0, False, a * c, []
    for s in specs[:ridx]:
        p = s.params
        if s.kind == 'act':
            if not gaussian or p.get('do_stabilize'):
                return None
            pg.layer[n - 1].act = _act_struct(p, ctx)
            gaussian = False
            continue
        if s.kind == 'pool' and pools:
            if not n or pg.layer[n - 1].pool_h:
                return None
            (kh, sh), (kw, sw) = [
                (p['window_shape'][d], p['strides'][d]) if d < len(x_shape) - 2 else (1, 1)
                for d in (0, 1)]
            if len(p['window_shape']) != len(x_shape) - 2 or kh > a or kw > c or any(
                    _pads(m, f, st, p['padding']) != (0, (m - f) // st + 1)
                    for m, f, st in ((a, kh, sh), (c, kw, sw))):
                return None
            ly = pg.layer[n - 1]
            ly.pool_h, ly.pool_w, ly.pool_sh, ly.pool_sw = kh, kw, sh, sw
            ly.pool_scale = 1. / (kh * kw) ** 2 if p['pool'] == 'avg' else 1.
            pooled.append((kh, kw, sh, sw, a, c))
            a, c = (a - kh) // sh + 1, (c - kw) // sw + 1
            shape = s.shape_fn(shape)
            continue
        if s.kind not in ('conv', 'dense') or n == L.DS_MAX_LAYERS:
            return None
        fh = fw = 1
        ph, pw, ao, co = 0, 0, a, c
        if s.kind == 'conv':
            nsp = len(p['filter_shape'])
            if nsp != len(x_shape) - 2 or p['padding'] == Padding.CIRCULAR or \
                    any(st != 1 for st in p['strides']):
                return None
            fh, fw, _, _, ph, pw, ao, co = _conv_geometry(p, a, c, nsp == 2)
        fan = None
        if p['parameterization'] == 'standard':
            fan = shape[-1] * fh * fw / p['s'][0]
        if min(ao, co) < 1 or ph >= fh or pw >= fw:
            return None
        ly = pg.layer[n]
        ly.fh, ly.fw, ly.ph, ly.pw, ly.ao, ly.co, ly.var_off = fh, fw, ph, pw, ao, co, off
        ly.aff = _affine_struct(p['W_std'], p['b_std'], p['parameterization'], fan)
        ly.act = O.NO_ACT
        plane = max(plane, a * co)
        off += ao * co
        a, c, n, gaussian = ao, co, n + 1, True
        shape = s.shape_fn(shape)
    ro = specs[ridx]
    pg.nlayers, pg.var_stride = n, off
    flatten = ro.kind == 'flatten'
    average = flatten or ro.params['pool'] == 'avg'
    # linear.py:1771-1801 on diagonal kernels: the mean of the positions, divided by their
    # number once more for GlobalAvgPool
    pg.divisor = float(a * c) if average else 1.
    pg.scale = 1. / (a * c) if average and not flatten else 1.
    # the offsets of each level, from the readout back, and the entries of the pooled planes
    da = dc = entries = 0
    m, k = a, c
    for kh, kw, sh, sw, pa, pc in reversed(pooled):
        entries += (2 * da + 1) * (2 * dc + 1) * m * k
        da, dc = min(sh * da + kh - 1, pa - 1), min(sw * dc + kw - 1, pc - 1)
        m, k = pa, pc
    if 4 * (pg.channels * pg.a * pg.c + off + 4 * plane + 2 * entries) > DS_MAX_SMEM or \
            pg.c > 512 or pg.a > 4096:
        return None
    return pg, specs[:ridx + 1], specs[ridx + 1:], gaussian and not flatten


def try_ds(kfn, x1: torch.Tensor, x2: Optional[torch.Tensor], compute_ntk: bool, ctx: _Ctx,
           whole: bool, pools: bool = False) -> Optional[Kernel]:
    """The Kernel of a network plan_ds covers, on diagonal-spatial kernels or (pools) on a band
    around them; whole: see try_fused."""
    if x2 is not None and x2.shape[1:] != x1.shape[1:]:
        return None
    n = x1.shape[0]
    pairs = n * (n + 1) // 2 if x2 is None else n * x2.shape[0]
    plan = plan_ds(kfn.specs, tuple(x1.shape), ctx, pools, pairs)
    if plan is None:
        return None
    pg, spatial, post, gaussian = plan
    q, t, c1, c2 = O.ds_chain(pg, x1, x2, compute_ntk)
    shape1 = tuple(x1.shape)
    shape2 = shape1 if x2 is None else tuple(x2.shape)
    for s in spatial:
        shape1, shape2 = s.shape_fn(shape1), s.shape_fn(shape2)
    same = x2 is None or (whole and x1.shape == x2.shape and bool(torch.equal(x1, x2)))
    k = Kernel(nngp=q, ntk=t, cov1=c1, cov2=c2, x1_is_x2=same, is_gaussian=gaussian,
               is_reversed=False, is_input=False, diagonal_batch=True,
               diagonal_spatial=spatial[-1].kind != 'flatten', shape1=shape1, shape2=shape2)
    return kfn.apply_kernel(k, ctx, specs=post)
