"""Tensor-level wrappers over the C ABI (one function per entry point).

Each wrapper takes and returns contiguous float32 CUDA tensors, enqueues on
the current torch stream and raises NtgError when the library reports one.
"""
from __future__ import annotations

import math
from typing import Optional

import torch

from . import _lib as L


def affine(w2: float, b2: float, ntk_w2: float, ntk_nn: float = 1., ntk_c: float = 0.,
           nn_scaled: bool = True) -> L.Affine:
    return L.Affine(w2, b2, ntk_w2, ntk_nn, ntk_c, int(nn_scaled))


IDENTITY_AFFINE = affine(1., 0., 1., 0., 0., True)
NO_ACT = L.Act(L.NTG_ACT_NONE, 0., 0., 0., 0, 0.)
NO_VAR = L.Var(None, 0, 0, 0)


def var_view(cov: Optional[torch.Tensor], diag: bool) -> L.Var:
    """Strided view of the variances (diagonal) of a per-sample kernel."""
    if cov is None:
        return NO_VAR
    n = cov.shape[0]
    if cov.ndim == 1:
        return L.Var(L.ptr(cov), 1, 0, 0)
    if diag:
        a = cov.shape[1]
        c = cov.shape[2] if cov.ndim == 3 else 1
        return L.Var(L.ptr(cov), a * c, c, 1)
    a = cov.shape[1]
    c = cov.shape[3] if cov.ndim == 5 else 1
    del n
    return L.Var(L.ptr(cov), a * a * c * c, a * c * c + c * c, c + 1)


def spatial_ac(t: torch.Tensor, bnd: int, diag: bool) -> tuple[int, int]:
    """(A, C): spatial sizes of the first / second spatial axis (1 if absent)."""
    sp = t.shape[bnd:]
    if diag:
        if len(sp) == 0:
            return 1, 1
        if len(sp) == 1:
            return sp[0], 1
        if len(sp) == 2:
            return sp[0], sp[1]
    else:
        if len(sp) == 0:
            return 1, 1
        if len(sp) == 2:
            return sp[0], 1
        if len(sp) == 4:
            return sp[0], sp[2]
    raise NotImplementedError('nt_gb300 kernels support at most two spatial dimensions')


def gram(x1: torch.Tensor, x2: torch.Tensor, precision: int = 0) -> torch.Tensor:
    """x1 x2^T / D; precision 1 runs the split-BF16 tcgen05 tensor-core kernel."""
    n1, n2, d = x1.shape[0], x2.shape[0], x1.shape[1]
    out = torch.empty((n1, n2), device=x1.device, dtype=torch.float32)
    ws, nbytes = None, 0
    if precision == 1:
        nbytes = int(L.load().ntg_gram_workspace_bytes(n1, n2, d))
        ws = torch.empty((nbytes,), device=x1.device, dtype=torch.uint8)
    # a tensor-core pipeline wait that runs out raises the library's device error word,
    # which the public call around this one reads (L.boundary)
    L.call('ntg_gram', L.stream(), L.ptr(x1), L.ptr(x2), n1, n2, d, L.ptr(out), precision,
           None if ws is None else ws.data_ptr(), nbytes)
    return out


def flat_input(x1: torch.Tensor, x2: Optional[torch.Tensor], precision: int = 0):
    """nngp, cov1, cov2 of flat inputs in one call (x2 None: cov1 is nngp's diagonal, so that a
    self pair has var1 * var2 - nngp^2 == 0 exactly, and cov2 None)."""
    xb = x1 if x2 is None else x2
    n1, n2, d = x1.shape[0], xb.shape[0], x1.shape[1]
    out = torch.empty((n1, n2), device=x1.device, dtype=torch.float32)
    ws, nbytes = None, 0
    if precision == 1:
        nbytes = int(L.load().ntg_gram_workspace_bytes(n1, n2, d))
        ws = torch.empty((nbytes,), device=x1.device, dtype=torch.uint8)
    cov1 = cov2 = None
    if x2 is not None:
        cov1 = torch.empty((n1,), device=x1.device, dtype=torch.float32)
        cov2 = torch.empty((n2,), device=x1.device, dtype=torch.float32)
    L.call('ntg_flat_input', L.stream(), L.ptr(x1), L.ptr(xb), n1, n2, d, L.ptr(out), L.ptr(cov1),
           L.ptr(cov2), precision, None if ws is None else ws.data_ptr(), nbytes)
    return out, torch.diagonal(out) if x2 is None else cov1, cov2


def _strided(c: torch.Tensor, n: int) -> torch.Tensor:
    """c as n float32 device values with a positive stride."""
    if not c.is_cuda or c.dtype != torch.float32 or tuple(c.shape) != (n,):
        raise ValueError('nt_gb300 kernels take one float32 CUDA variance per sample')
    return c if c.stride(0) > 0 else c.contiguous()


def flat_rules(q, t, c1, c2, layers, want_t: bool):
    """A run of (affine | None, activation) layers on flat kernels q, t [N1, N2] (t None: zero)
    and c1 [N1], c2 [N2] or None, which may be strided: (q, t, c1, c2) after it."""
    n1, n2 = q.shape
    v1 = _strided(c1, n1)
    if c2 is None and n2 > n1:
        raise ValueError('a kernel of two inputs needs the variances of both')
    v2 = v1 if c2 is None else _strided(c2, n2)
    dev = q.device
    out_q = torch.empty((n1, n2), device=dev, dtype=torch.float32)
    out_t = torch.empty((n1, n2), device=dev, dtype=torch.float32) if want_t else None
    o1 = torch.empty((n1,), device=dev, dtype=torch.float32)
    o2 = None if c2 is None else torch.empty((n2,), device=dev, dtype=torch.float32)
    arr = (L.FlatLayer * len(layers))(*[
        L.FlatLayer(int(a is not None), IDENTITY_AFFINE if a is None else a, act)
        for a, act in layers])
    L.call('ntg_flat_rules', L.stream(), L.ptr(q), L.ptr(t), n1, n2, v1.data_ptr(),
           max(v1.stride(0), 1), v2.data_ptr(), max(v2.stride(0), 1), len(layers), arr,
           L.ptr(out_q), L.ptr(out_t), L.ptr(o1), L.ptr(o2))
    return out_q, out_t, o1, o2


def cov_diag(x: torch.Tensor) -> torch.Tensor:
    out = torch.empty((x.shape[0],), device=x.device, dtype=torch.float32)
    L.call('ntg_cov_diag', L.stream(), L.ptr(x), x.shape[0], x.shape[1], L.ptr(out))
    return out


def input_ds(x1: torch.Tensor, x2: Optional[torch.Tensor]) -> torch.Tensor:
    """x [N, *spatial, K] -> [N1, N2, *spatial] (pairs) or [N, *spatial] (x2 None): the
    diagonal-spatial input covariances."""
    sp = tuple(x1.shape[1:-1])
    p, k = int(math.prod(sp)), x1.shape[-1]
    x1 = x1.contiguous()
    if x2 is None:
        out = torch.empty((x1.shape[0],) + sp, device=x1.device, dtype=torch.float32)
        L.call('ntg_input_ds', L.stream(), L.ptr(x1), None, x1.shape[0], 0, p, k, L.ptr(out))
    else:
        x2 = x2.contiguous()
        out = torch.empty((x1.shape[0], x2.shape[0]) + sp, device=x1.device, dtype=torch.float32)
        L.call('ntg_input_ds', L.stream(), L.ptr(x1), L.ptr(x2), x1.shape[0], x2.shape[0], p, k,
               L.ptr(out))
    return out


def input_fs(x1: torch.Tensor, x2: Optional[torch.Tensor]) -> torch.Tensor:
    """x [N, A, C, K] -> [N1, N2, A, A, C, C] (pairs) or [N, A, A, C, C] (x2 None)."""
    n1, a, c, k = x1.shape
    if x2 is None:
        out = torch.empty((n1, a, a, c, c), device=x1.device, dtype=torch.float32)
        L.call('ntg_input_fs', L.stream(), L.ptr(x1), None, n1, 0, a, c, k, 0, L.ptr(out))
    else:
        n2 = x2.shape[0]
        out = torch.empty((n1, n2, a, a, c, c), device=x1.device, dtype=torch.float32)
        L.call('ntg_input_fs', L.stream(), L.ptr(x1), L.ptr(x2), n1, n2, a, c, k, 1, L.ptr(out))
    return out


def conv_fs(q, t, batch, n2, a, c, fh, fw, sh, sw, ph, pw, ao, co, circular, aff, act, var1,
            var2, want_t, lead):
    out_q = torch.empty(lead + (ao, ao, co, co), device=q.device, dtype=torch.float32)
    out_t = torch.empty_like(out_q) if want_t else None
    L.call('ntg_conv_fs', L.stream(), L.ptr(q), L.ptr(t), L.ptr(out_q), L.ptr(out_t), batch, n2,
           a, c, fh, fw, sh, sw, ph, pw, ao, co, int(circular), aff, act, var1, var2)
    return out_q, out_t


def conv_ds(q, t, batch, a, c, fh, fw, sh, sw, ph, pw, ao, co, circular, aff, want_t, lead,
            has_c):
    shape = lead + ((ao, co) if has_c else (ao,))
    out_q = torch.empty(shape, device=q.device, dtype=torch.float32)
    out_t = torch.empty_like(out_q) if want_t else None
    L.call('ntg_conv_ds', L.stream(), L.ptr(q), L.ptr(t), L.ptr(out_q), L.ptr(out_t), batch, a, c,
           fh, fw, sh, sw, ph, pw, ao, co, int(circular), aff)
    return out_q, out_t


def affine_act(q, t, batch, n2, a, c, diag, has_affine, aff, act, var1, var2, want_t):
    out_q = torch.empty_like(q)
    out_t = torch.empty_like(q) if want_t else None
    L.call('ntg_affine_act', L.stream(), L.ptr(q), L.ptr(t), L.ptr(out_q), L.ptr(out_t), batch,
           n2, a, c, int(diag), int(has_affine), aff, act, var1, var2)
    return out_q, out_t


def max_abs(x: torch.Tensor) -> float:
    out = torch.empty((1,), device=x.device, dtype=torch.float32)
    L.call('ntg_max_abs', L.stream(), L.ptr(x), x.numel(), L.ptr(out))
    return float(out.item())


def pool(x, batch, a, c, wa, wc, sa, sc, pa, pc, ao, co, circular, diag, average,
         normalize_edges, out_shape):
    out = torch.empty(out_shape, device=x.device, dtype=torch.float32)
    L.call('ntg_pool', L.stream(), L.ptr(x), L.ptr(out), batch, a, c, wa, wc, sa, sc, pa, pc, ao,
           co, int(circular), int(diag), int(average), int(normalize_edges))
    return out


def global_pool(x: torch.Tensor, bnd: int, average: bool, post_scale: float = 1.) -> torch.Tensor:
    lead = tuple(x.shape[:bnd])
    batch = 1
    for d in lead:
        batch *= d
    m = x.numel() // max(batch, 1)
    out = torch.empty(lead, device=x.device, dtype=torch.float32)
    L.call('ntg_global_pool', L.stream(), L.ptr(x), L.ptr(out), batch, m, int(average), post_scale)
    return out


def flatten_fs(x: torch.Tensor, bnd: int, a: int, c: int) -> torch.Tensor:
    lead = tuple(x.shape[:bnd])
    batch = 1
    for d in lead:
        batch *= d
    out = torch.empty(lead, device=x.device, dtype=torch.float32)
    L.call('ntg_flatten_fs', L.stream(), L.ptr(x), L.ptr(out), batch, a, c)
    return out


def ds_chain(prog: L.DsChain, x1, x2, want_t: bool):
    """nngp, ntk [N1, N2], cov1, cov2 after the readout of a conv network on diagonal-spatial
    kernels (x2 None: x1 with itself, cov2 None)."""
    import ctypes
    n1, n2 = x1.shape[0], (x1 if x2 is None else x2).shape[0]

    def new(*shape):
        return torch.empty(shape, device=x1.device, dtype=torch.float32)

    q, t = new(n1, n2), new(n1, n2) if want_t else None
    v1, c1 = new(n1, prog.var_stride), new(n1)
    v2, c2 = (None, None) if x2 is None else (new(n2, prog.var_stride), new(n2))
    L.call('ntg_ds_chain', L.stream(), ctypes.byref(prog), L.ptr(x1), L.ptr(x2), n1, n2, L.ptr(v1),
           L.ptr(v2), L.ptr(c1), L.ptr(c2), L.ptr(q), L.ptr(t))
    return q, t, c1, c2


def chain_vars(prog: L.Chain, x1, x2=None):
    """Pre-activation variance maps [N, var_stride] of every conv layer of the chain: of x1, or
    (of x1, of x2)."""
    import ctypes
    nbytes = int(L.load().ntg_chain_workspace_bytes())
    ws = torch.empty((nbytes,), device=x1.device, dtype=torch.uint8)
    var = [None if x is None else torch.empty((x.shape[0], prog.var_stride), device=x1.device,
                                              dtype=torch.float32) for x in (x1, x2)]
    L.call('ntg_chain_vars', L.stream(), ctypes.byref(prog), L.ptr(x1), x1.shape[0],
           L.ptr(var[0]), L.ptr(x2), 0 if x2 is None else x2.shape[0], L.ptr(var[1]),
           ws.data_ptr(), nbytes)
    return var[0] if x2 is None else tuple(var)


def _chain(prog, x1, x2, r0, n1, c0, n2, var1, var2, out_q, out_t, ld_out, mode):
    import ctypes
    nbytes = int(L.load().ntg_chain_workspace_bytes())
    ws = torch.empty((nbytes,), device=x1.device, dtype=torch.uint8)
    L.call('ntg_chain_fwd_ws', L.stream(), ctypes.byref(prog), L.ptr(x1), L.ptr(x2), r0, n1, c0,
           n2, L.ptr(var1), L.ptr(var2), out_q.data_ptr(),
           None if out_t is None else out_t.data_ptr(), ld_out, mode, ws.data_ptr(), nbytes)


def chain_fwd(prog: L.Chain, x1, x2, r0, n1, c0, n2, var1, var2, out_q, out_t, ld_out):
    _chain(prog, x1, x2, r0, n1, c0, n2, var1, var2, out_q, out_t, ld_out, 0)


def chain_fwd_sym(prog: L.Chain, x, r0, n1, c0, n2, var, out_q, out_t, ld_out):
    """Pairs (r0.., c0..) of x with itself, each written at (i, j) and (j, i) of the
    whole kernel out [., ld_out]; the tile is diagonal (only i <= j evaluated) or
    has disjoint row and column ranges."""
    _chain(prog, x, x, r0, n1, c0, n2, var, var, out_q, out_t, ld_out, 1)


def chain_fwd_self(prog: L.Chain, x, var):
    """nngp [N] of the pairs (x[i], x[i])."""
    out = torch.empty((x.shape[0],), device=x.device, dtype=torch.float32)
    _chain(prog, x, x, 0, x.shape[0], 0, 1, var, var, out, None, 1, 2)
    return out
