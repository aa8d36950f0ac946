"""Reverse-mode derivatives of hpsi and of the densities, as
torch.autograd.Functions over the library's kernels.

The reference gets these from JAX's reverse mode through hpsi01
(meanfield.py:41-159) and the density terms (densities.py:237-330).  Here
they follow from two exact properties of those discretisations:

* h is Hermitian, and the bilinear form <a|h[P]|b> is the integral of each
  potential field times the matching pair density of (a, b) -- upot: rho,
  bmass: tau, v_pair: 2 chi, aq: current, spot: sdens, wlspot: sodens --
  plus, for bmass, the Nyquist term of cderv02 (levels.py:314-330).  The
  pair densities come from the density kernel with two operands
  (hfb_pair_density).
* The densities are quadratic forms in psi, so their VJP is 2 w h[F_bar] psi
  (+ wu chi_bar psi) with the Nyquist term of the tau cotangent removed.

VJP of y = w h psi - wu v_pair psi:
    psi_bar = w h ybar - wu v_pair ybar,
    P_bar   = sum_s w_s F_s(ybar_s, psi_s) for each field (v_pair: -2 wu chi),
    bmass_bar additionally the Nyquist pair term (hfb_nyquist_pair).
VJP of the densities:
    psi_bar = hpsi with fields (rho_bar, tau_bar, chi_bar, current_bar,
              sdens_bar, sodens_bar), weights (2 w, -wu), minus the Nyquist
              term of tau_bar (hfb_nyquist_apply).

Complex gradients follow torch's convention, dL = Re sum conj(x.grad) dx.
States are [nst][2][nx][ny][nz], neutrons first (``nneut`` of them); fields
are per isospin, [2][...].
"""
from types import SimpleNamespace

import torch

from ._lib import aligned, call, ptr, stream_ptr, prec_of, HFB_F64, HFB_F32

_FIELDS = ("upot", "bmass", "v_pair", "aq", "spot", "wlspot")
_DENS = ("rho", "chi", "tau", "current", "sdens", "sodens")


def _vec(x, nst, dev):
    return torch.as_tensor(x, dtype=torch.float64, device=dev).reshape(-1).expand(nst).contiguous()


def _empty_densities(grids, dev):
    """The six density arrays, to be written by the library."""
    g = (grids.nx, grids.ny, grids.nz)
    return {k: torch.empty(((2,) if k in _DENS[:3] else (2, 3)) + g, dtype=torch.float64, device=dev) for k in _DENS}


def _densities(grids, psi, nneut, w, wu):
    """Densities of ``psi`` with occupation weights w and pairing weights wu."""
    nst = psi.shape[0]
    d = _empty_densities(grids, psi.device)
    one = torch.ones(nst, dtype=torch.float64, device=psi.device)
    call("hfb_add_density", grids.ctx.handle, prec_of(psi), nst, nneut, ptr(psi), ptr(w), ptr(wu), ptr(one), ptr(one),
         1.0, *(ptr(d[k]) for k in _DENS), None, None, stream_ptr())
    return d


def pair_densities(grids, a, b, nneut, w, wu):
    """sum_s w_s F(a_s, b_s) for rho, tau, current, sdens, sodens and
    sum_s wu_s chi(a_s, b_s), the pair densities Re(a^dagger O_F b)."""
    d = _empty_densities(grids, a.device)
    call("hfb_pair_density", grids.ctx.handle, prec_of(a), a.shape[0], nneut, ptr(a), ptr(b), ptr(w), ptr(wu),
         *(ptr(d[k]) for k in _DENS), stream_ptr())
    return d


def _pack(grids, fields, dtype):
    """The packed hpsi potentials (``.pot``, [2][12][n^3] in the precision of
    ``dtype``) of ``fields``; missing ones are zero."""
    g = (grids.nx, grids.ny, grids.nz)
    rd = torch.float64 if dtype == torch.complex128 else torch.float32
    pot = torch.empty((2, 12) + g, dtype=rd, device="cuda")
    src = []
    for k in _FIELDS:
        f = fields.get(k)
        if f is not None:
            shape = ((2,) if k in _FIELDS[:3] else (2, 3)) + g
            if f.dtype != torch.float64 or not f.is_cuda:
                f = f.detach().to(device="cuda", dtype=torch.float64)
            if f.shape != shape or not f.is_contiguous():
                f = torch.broadcast_to(f, shape).contiguous()
        src.append(f)
    call("hfb_pack_pot", grids.ctx.handle, HFB_F64 if rd == torch.float64 else HFB_F32, *(ptr(f) for f in src), ptr(pot),
         stream_ptr())
    return SimpleNamespace(pot=pot)


def _hpsi(grids, pot, x, nneut, w, wu):
    prec = prec_of(x)
    if prec == HFB_F32:
        x = aligned(x)
    out = torch.empty_like(x)
    call("hfb_hpsi", grids.ctx.handle, prec, ptr(pot), x.shape[0], nneut, ptr(x), ptr(w), ptr(wu), ptr(out),
         None, None, stream_ptr())
    return out


def hpsi_vjp(grids, pot, psi, nneut, w, wu, ybar):
    """(psi_bar, {field: cotangent}) for y = w h psi - wu v_pair psi."""
    nst = psi.shape[0]
    ybar = ybar.contiguous()
    psi_bar = _hpsi(grids, pot, ybar, nneut, w, wu)
    pd = pair_densities(grids, ybar, psi, nneut, w, -2.0 * wu)
    call("hfb_nyquist_pair", grids.ctx.handle, prec_of(psi), nst, nneut, ptr(ybar), ptr(psi), ptr(w), ptr(pd["tau"]),
         stream_ptr())
    bars = dict(upot=pd["rho"], bmass=pd["tau"], v_pair=pd["chi"], aq=pd["current"], spot=pd["sdens"],
                wlspot=pd["sodens"])
    return psi_bar, bars


def densities_vjp(grids, psi, nneut, w, wu, bars):
    """psi_bar for cotangents ``bars`` (dict over rho, chi, tau, current,
    sdens, sodens; missing ones zero) of the densities of psi."""
    f = dict(upot=bars.get("rho"), bmass=bars.get("tau"), v_pair=bars.get("chi"), aq=bars.get("current"),
             spot=bars.get("sdens"), wlspot=bars.get("sodens"))
    mf = _pack(grids, {k: v for k, v in f.items() if v is not None}, psi.dtype)
    w2 = (2.0 * w).contiguous()
    out = _hpsi(grids, mf.pot, psi, nneut, w2, (-wu).contiguous())
    tau = bars.get("tau")
    if tau is not None:
        call("hfb_nyquist_apply", grids.ctx.handle, prec_of(psi), psi.shape[0], nneut, ptr(tau.contiguous()), ptr(w2),
             ptr(psi), ptr(out), stream_ptr())
    return out


class HPsi(torch.autograd.Function):
    """y = w h[fields] psi - wu v_pair psi (meanfield.py:41-159, both
    isospins: states below ``nneut`` use the neutron fields), differentiable
    in psi and in the six potential fields (each [2][...], float64)."""

    @staticmethod
    def forward(ctx, psi, upot, bmass, v_pair, aq, spot, wlspot, grids, nneut, weight=1.0, weightuv=0.0):
        psi = psi.contiguous()
        nst = psi.shape[0]
        w, wu = _vec(weight, nst, psi.device), _vec(weightuv, nst, psi.device)
        fields = dict(upot=upot, bmass=bmass, v_pair=v_pair, aq=aq, spot=spot, wlspot=wlspot)
        mf = _pack(grids, fields, psi.dtype)
        ctx.save_for_backward(psi, mf.pot, w, wu)
        ctx.grids, ctx.nneut = grids, nneut
        return _hpsi(grids, mf.pot, psi, nneut, w, wu)

    @staticmethod
    def backward(ctx, ybar):
        psi, pot, w, wu = ctx.saved_tensors
        psi_bar, bars = hpsi_vjp(ctx.grids, pot, psi, ctx.nneut, w, wu, ybar.contiguous())
        return (psi_bar,) + tuple(bars[k] for k in _FIELDS) + (None, None, None, None)


class Densities(torch.autograd.Function):
    """(rho, chi, tau, current, sdens, sodens) of psi (densities.py:177-330)
    with per-state weights w = wocc * wstates and wu = wguv * pairwg *
    wstates, differentiable in psi."""

    @staticmethod
    def forward(ctx, psi, grids, nneut, weight=1.0, weightuv=0.0):
        psi = psi.contiguous()
        nst = psi.shape[0]
        w, wu = _vec(weight, nst, psi.device), _vec(weightuv, nst, psi.device)
        d = _densities(grids, psi, nneut, w, wu)
        ctx.save_for_backward(psi, w, wu)
        ctx.grids, ctx.nneut = grids, nneut
        return tuple(d[k] for k in _DENS)

    @staticmethod
    def backward(ctx, *grads):
        psi, w, wu = ctx.saved_tensors
        bars = {k: g.contiguous() for k, g in zip(_DENS, grads) if g is not None}
        return densities_vjp(ctx.grids, psi, ctx.nneut, w, wu, bars), None, None, None, None


def hpsi(psi, fields, grids, nneut, weight=1.0, weightuv=0.0):
    """Differentiable hpsi; ``fields`` a dict over upot, bmass, v_pair, aq,
    spot, wlspot (float64 tensors [2][...] / [2][3][...])."""
    return HPsi.apply(psi, *(fields[k] for k in _FIELDS), grids, nneut, weight, weightuv)


def densities(psi, grids, nneut, weight=1.0, weightuv=0.0):
    """Differentiable densities: dict over rho, chi, tau, current, sdens, sodens."""
    return dict(zip(_DENS, Densities.apply(psi, grids, nneut, weight, weightuv)))
