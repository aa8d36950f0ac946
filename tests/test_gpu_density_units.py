"""Densities, kinetic energies and pair densities (csrc/density.cu) over grids,
isospin splits and state counts whose runs of units start and end inside
tiles, isospins and axes, against the oracle.  Double precision: sums of at
most 30 states of n-point transforms, 1e-11 relative to the largest value;
single precision: the transforms round at 1e-7, 5e-6."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

D = (0.9, 1.0, 1.1)
FIELDS = ("rho", "chi", "tau", "current", "sdens", "sodens")


def _inputs(n, ns, seed):
    rng = np.random.default_rng(seed)
    x = [(np.arange(n) - (n - 1) / 2) * d for d in D]
    env = np.exp(-(x[0][:, None, None] ** 2 + x[1][None, :, None] ** 2 + x[2][None, None, :] ** 2) / (0.1 * n * n))
    psi = [(rng.standard_normal((ns, 2, n, n, n)) + 1j * rng.standard_normal((ns, 2, n, n, n))) * env for _ in range(2)]
    return psi, rng.uniform(0.1, 1.0, (4, ns))


def _sum(parts, nn):
    return [np.stack([p[:nn].sum(axis=0), p[nn:].sum(axis=0)]) for p in parts]


def _close(got, ref, tol):
    assert np.max(np.abs(got - ref)) <= tol * np.max(np.abs(ref))


@pytest.mark.parametrize("prec", ["f64", "f32"])
@pytest.mark.parametrize("n,ns,nn", [(8, 1, 1), (8, 1, 0), (8, 30, 11), (16, 7, 6), (24, 5, 5), (24, 3, 1), (32, 4, 1),
                                     (40, 3, 2), (48, 2, 1)])
def test_densities_against_oracle(n, ns, nn, prec):
    import hfb
    from hfb._lib import call, ptr, stream_ptr, prec_of
    from oracle import densities as od
    (psi, phi), (w, uv, pw, wst) = _inputs(n, ns, 100 * n + ns)
    dtype, tol = (torch.complex128, 1e-11) if prec == "f64" else (torch.complex64, 5e-6)
    g = hfb.grids.init_grids(hfb.params.init_params(), nx=n, ny=n, nz=n, dx=D[0], dy=D[1], dz=D[2])
    P, F = (torch.from_numpy(a).cuda().to(dtype).contiguous() for a in (psi, phi))
    psi, phi = (t.cpu().numpy().astype(np.complex128) for t in (P, F))
    W, U, PW, WS = (torch.from_numpy(a.copy()).cuda() for a in (w, uv, pw, wst))
    d = hfb.densities.init_densities(g)
    for k in ("rho", "tau", "chi"):
        getattr(d, k).fill_(0.5)
    kin = torch.zeros(ns, dtype=torch.float64, device="cuda")
    import ctypes as C
    h2m = (C.c_double * 2)(20.0, 21.0)
    args = [ptr(getattr(d, k)) for k in FIELDS]
    call("hfb_add_density", g.ctx.handle, prec_of(P), ns, nn, ptr(P), ptr(W), ptr(U), ptr(PW), ptr(WS), 0.2, *args, h2m,
         ptr(kin), stream_ptr())
    ref = dict(zip(FIELDS, _sum(od.state_contributions(w * wst, uv * pw * wst, psi, D), nn)))
    for k in ("rho", "tau", "chi"):
        ref[k] = 0.2 * ref[k] + 0.8 * 0.5
    for k in FIELDS:
        _close(getattr(d, k).cpu().numpy(), ref[k], tol)
    k2 = sum(np.reshape((2 * np.pi * np.minimum(np.arange(n), n - np.arange(n)) / (n * D[a])) ** 2,
                        [-1 if b == a else 1 for b in range(3)]) for a in range(3))
    f = np.fft.fftn(psi, axes=(2, 3, 4))
    e = D[0] * D[1] * D[2] * np.sum(np.abs(f) ** 2 * k2, axis=(1, 2, 3, 4)) / n ** 3
    ref_kin = e * np.where(np.arange(ns) < nn, 20.0, 21.0)
    _close(kin.cpu().numpy(), ref_kin, tol)
    kin.zero_()
    call("hfb_sp_kinetic", g.ctx.handle, prec_of(P), ns, nn, ptr(P), h2m, ptr(kin), stream_ptr())
    _close(kin.cpu().numpy(), ref_kin, tol)
    # pair densities: the polarisation of the quadratic ones
    call("hfb_pair_density", g.ctx.handle, prec_of(P), ns, nn, ptr(P), ptr(F), ptr(W), ptr(U), *args, stream_ptr())
    plus, minus = (od.state_contributions(w, uv, psi + s * phi, D) for s in (1.0, -1.0))
    scale = max(np.max(np.abs(x)) for x in _sum(plus, nn))
    for k, r in zip(FIELDS, _sum([(a - b) / 4.0 for a, b in zip(plus, minus)], nn)):
        assert np.max(np.abs(getattr(d, k).cpu().numpy() - r)) <= tol * max(scale, np.max(np.abs(r))), k
