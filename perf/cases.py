"""Performance cases: the work a user of this package has it do, through its
public entry points, with a plain 64-bit restatement of each result.

Kinds of case (``kind``), each on an n^3 grid of spacing ``d`` fm with
``npsi0`` + ``npsi1`` states for ``nneut`` neutrons and ``nprot`` protons:

* ``hpsi``     hfb.meanfield.hpsi01 on the neutron states;
* ``density``  hfb.densities.add_density, as in the loop (20 % mixing and the
               kinetic energies);
* ``fields``   hfb.meanfield.skyrme and hfb.energies.integ_energy;
* ``vjp_hpsi``, ``vjp_density``
               forward and backward through hfb.vjp;
* ``step``     hfb.static.grstep and diagstep: one orthonormalised gradient
               step of all states in a fixed mean field, without pairing;
* ``iterate``  hfb.static.iterate: one whole self-consistent iteration past
               the start-up phases, with the host's read of the energies and
               its step-size rule, with (``pairing``) or without BCS.

The states are oscillator states of the nucleus, deformed and spin-mixed by
smooth random factors (so that no symmetry leaves degenerate levels whose
basis would be arbitrary) and orthonormalised; the fields are the Skyrme
fields of those states.  Precision "f32" means complex64 states; results
that are computed from them are returned in single precision too.

With pairing the states of an iteration are eigenvectors, fixed up to a
phase: the iteration then returns what does not depend on the phase.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "jax-hfbfft_b200"))
import hfb  # noqa: E402
import hfb.vjp  # noqa: E402

DENS = ("rho", "chi", "tau", "current", "sdens", "sodens")
FIELDS = ("upot", "bmass", "v_pair", "aq", "spot", "wlspot")


def _case(name, kind, n, d, npsi, nucleus, prec, pairing=False):
    return dict(name=name, kind=kind, n=n, d=d, npsi0=npsi[0], npsi1=npsi[1], nneut=nucleus[0], nprot=nucleus[1],
                prec=prec, pairing=pairing)


def listed():
    return [
        # one spinor at a time, the way the reference's hpsi01 is called; the smallest call there is
        _case("hpsi_spinor_16_f64", "hpsi", 16, 1.0, (1, 1), (1, 1), "f64"),
        # the Hamiltonian on the neutron states of Pb208 in the single-precision bulk of a solve
        _case("hpsi_pb208_48_f32", "hpsi", 48, 0.8, (140, 96), (126, 82), "f32"),
        # densities of Sn132 as the sweep runs it
        _case("density_sn132_40_f32", "density", 40, 0.8, (90, 60), (82, 50), "f32"),
        # mean field and energy functional from densities; always double precision
        _case("fields_48", "fields", 48, 0.8, (140, 96), (126, 82), "f64"),
        # a loss on h psi differentiated to the states and the potentials
        _case("vjp_hpsi_ca48_32_f64", "vjp_hpsi", 32, 0.8, (40, 30), (28, 20), "f64"),
        # a loss on the densities differentiated to the states
        _case("vjp_density_o16_24_f64", "vjp_density", 24, 1.0, (10, 10), (8, 8), "f64"),
        # the wave-function half of a small nucleus's iteration: latency and launches
        _case("step_o16_24_f64", "step", 24, 1.0, (10, 10), (8, 8), "f64"),
        # the same for a medium nucleus in single precision, with state counts that fit no tile
        _case("step_zr90_40_f32", "step", 40, 0.8, (61, 47), (50, 40), "f32"),
        # whole iterations: the smallest preset, without pairing
        _case("iterate_o16_24_f64", "iterate", 24, 1.0, (10, 10), (8, 8), "f64"),
        # an open-shell nucleus with pairing, double precision
        _case("iterate_cr48_32_f64", "iterate", 32, 0.8, (32, 32), (24, 24), "f64", True),
        # the benchmark nucleus: the single-precision bulk of its solve, and the double-precision path
        _case("iterate_pb208_48_f32", "iterate", 48, 0.8, (140, 96), (126, 82), "f32", True),
        _case("iterate_pb208_48_f64", "iterate", 48, 0.8, (140, 96), (126, 82), "f64", True),
    ]


# largest number of states per isospin that a solve puts on each grid
_ROOM = {16: 20, 24: 30, 32: 60, 40: 100, 48: 140}


def draw(rng):
    kind = rng.choice(["hpsi", "density", "fields", "vjp_hpsi", "vjp_density", "step", "step", "iterate", "iterate",
                       "iterate"])
    n = rng.choice(sorted(_ROOM))
    room = _ROOM[n]
    if kind.startswith("vjp"):
        room = min(room, 60)
    lo = 1 if kind == "hpsi" else 6
    npsi0 = round(math.exp(rng.uniform(math.log(lo), math.log(room))))
    npsi1 = max(lo, round(npsi0 * rng.uniform(0.6, 1.0)))
    nneut = max(1, round(npsi0 * rng.uniform(0.7, 0.9)))
    nprot = max(1, round(npsi1 * rng.uniform(0.7, 0.9)))
    prec = "f64" if kind in ("fields", "vjp_hpsi", "vjp_density") else rng.choice(["f32", "f64"])
    d = round(rng.uniform(0.75, 1.0), 3) if n < 40 else round(rng.uniform(0.7, 0.85), 3)
    c = _case("", kind, n, d, (npsi0, npsi1), (nneut, nprot), prec, kind == "iterate" and rng.random() < 0.5)
    del c["name"]
    return c


# ------------------------------------------------------------------ inputs --
def _shell_order(count):
    """(i, j, k, spin) of the lowest oscillator states, two spins each."""
    out, shell = [], 0
    while len(out) < count:
        for k in range(shell + 1):
            for j in range(shell + 1 - k):
                out += [(shell - k - j, j, k, 0), (shell - k - j, j, k, 1)]
        shell += 1
    return out[:count]


def _coords(case):
    n = case["n"]
    return (torch.arange(n, dtype=torch.float64, device="cuda") - (n - 1) / 2.0) * case["d"]


def _radius(case):
    """The length r of the oscillator's Gaussian exp(-x^2 / r^2)."""
    a = case["nneut"] + case["nprot"]
    return 2.0 * math.sqrt(20.735530 * a ** (1.0 / 3.0) / 41.0)


def _dtype(case):
    return torch.complex64 if case["prec"] == "f32" else torch.complex128


def _blocks(case):
    n0, n1 = case["npsi0"], case["npsi1"]
    return (slice(0, n0), slice(n0, n0 + n1))


def _states(case, seed):
    """The states [nst][2][n][n][n], rounded to the case's precision and held
    in complex128."""
    n, x = case["n"], _coords(case)
    n0, n1 = case["npsi0"], case["npsi1"]
    g = np.random.default_rng([seed, 1])
    r = torch.from_numpy(g.standard_normal((n0 + n1, 8))).cuda()
    rad = _radius(case)
    e = torch.exp(-(x / rad) ** 2)
    psi = torch.zeros((n0 + n1, 2, n, n, n), dtype=torch.complex128, device="cuda")
    u = x / rad
    axes = (u[:, None, None], u[None, :, None], u[None, None, :])
    qn = _shell_order(n0) + _shell_order(n1)
    for s, (i, j, k, c) in enumerate(qn):
        fx, fy, fz = (e * u ** i), (e * u ** j), (e * u ** k)
        f = fx[:, None, None] * fy[None, :, None] * fz[None, None, :]
        f = f / torch.sqrt((f ** 2).sum())
        tilt = sum(a * (0.15 * r[s, m] + 0.15j * r[s, 3 + m]) for m, a in enumerate(axes))
        psi[s, c] = f * (1.0 + tilt)
        psi[s, 1 - c] = f * (0.2 * r[s, 6] + 0.2j * r[s, 7])
    for b in _blocks(case):
        p = psi[b].reshape(psi[b].shape[0], -1)
        p = p / torch.linalg.vector_norm(p, dim=1, keepdim=True)
        for _ in range(2):   # twice: the second pass removes what the first one's conditioning leaves
            low = torch.linalg.cholesky((p.conj() @ p.T).conj())
            p = torch.linalg.solve_triangular(low, p, upper=False)
        psi[b] = (p / case["d"] ** 1.5).reshape(psi[b].shape)
    return psi.to(_dtype(case)).to(torch.complex128)


def _weights(case):
    """Occupation and pairing weights of every state, smooth around the Fermi
    level as BCS leaves them."""
    out = []
    for ns, particles in ((case["npsi0"], case["nneut"]), (case["npsi1"], case["nprot"])):
        i = torch.arange(ns, dtype=torch.float64, device="cuda")
        v2 = 1.0 / (1.0 + torch.exp((i - particles + 0.5) / 2.0))
        out.append(torch.stack([v2, torch.sqrt(torch.clamp(v2 - v2 ** 2, min=1e-6))]))
    both = torch.cat(out, dim=1)
    return both[0].contiguous(), both[1].contiguous()


def _grids(case):
    n, d = case["n"], case["d"]
    return hfb.grids.init_grids(hfb.params.init_params(), nx=n, ny=n, nz=n, dx=d, dy=d, dz=d)


def _fields(case, psi):
    """The Skyrme fields of the states with the weights of _weights."""
    w, wu = _weights(case)
    dens = _x_density(case, psi, w, wu)
    return _x_skyrme(case, dens)


def _solver(case, seed):
    """A solver state in hand before an iteration: set up, the first mean
    field and gradient step done (hfb.static.prepare) and, with pairing, the
    loop's first iterations, whose constant gap gives the pairing field its
    start."""
    n, d = case["n"], case["d"]
    r = _radius(case)
    force = dict(name="SLy4", ipair=0, tbcs=False)
    if case["pairing"]:
        force = dict(name="SLy4", ipair=5, tbcs=True, pair_cutoff=[60.0, 60.0])
    st = hfb.config.setup(dict(
        grid=dict(nx=n, ny=n, nz=n, dx=d, dy=d, dz=d), force=force,
        levels=dict(nneut=case["nneut"], nprot=case["nprot"], npsi=[case["npsi0"], case["npsi1"]]),
        static=dict(maxiter=1000, serr=1e-20, x0dmp=0.2, e0dmp=100.0, tvaryx_0=True, radinx=r, radiny=r, radinz=r),
        mprint=1), dtype=_dtype(case))
    st["levels"].psi.copy_(_states(case, seed))
    del st["moment"]
    hfb.static.prepare(**st)
    for i in range(1, 1 + _START * case["pairing"]):
        hfb.static.iterate(i, **st)
    return st


_START = 3    # iterations with the constant gap before a case with pairing
_FIRST = 40   # first iteration of a pass: past the start-up phases of the loop


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("step", "iterate"):
        s = dict(kind=kind, pairing=case["pairing"], S=_solver(case, seed), i=_FIRST)
        s["S"]["params"].iteration = _FIRST
        return s
    g = _grids(case)
    psi = _states(case, seed)
    w, wu = _weights(case)
    s = dict(kind=kind, grids=g, nneut=case["npsi0"])
    if kind == "hpsi":
        mf = hfb.meanfield.init_meanfield(g, _dtype(case))
        for k, v in _fields(case, psi).items():
            if hasattr(mf, k):
                getattr(mf, k).copy_(v)
        mf.pack(_dtype(case))
        b = _blocks(case)[0]
        s.update(mf=mf, psi=psi[b].to(_dtype(case)).contiguous(), w=w[b].contiguous(), wu=wu[b].contiguous())
    elif kind == "density":
        p = hfb.params.init_params()
        lv = hfb.levels.init_levels(g, case["nneut"], case["nprot"], (case["npsi0"], case["npsi1"]),
                                    dtype=_dtype(case))
        lv.psi.copy_(psi)
        lv.wocc.copy_(w)
        lv.wguv.copy_(wu)
        s.update(levels=lv, dens=hfb.densities.init_densities(g), forces=hfb.forces.init_forces(p, name="SLy4"))
    elif kind == "fields":
        p = hfb.params.init_params()
        f = hfb.forces.init_forces(p, name="SLy4", ipair=5, tbcs=True, pair_cutoff=[60.0, 60.0])
        lv = hfb.levels.init_levels(g, case["nneut"], case["nprot"], (1, 1))
        _, st = hfb.static.init_static(f, lv, x0dmp=0.2, e0dmp=100.0)
        dens = hfb.densities.init_densities(g)
        for k, v in _x_density(case, psi, w, wu).items():
            if hasattr(dens, k):
                getattr(dens, k).copy_(v)
        s.update(params=p, forces=f, levels=lv, static=st, dens=dens, mf=hfb.meanfield.init_meanfield(g),
                 coulomb=hfb.coulomb.init_coulomb(g), energies=hfb.energies.init_energies(), pairs=hfb.pairs.Pairs())
    elif kind == "vjp_hpsi":
        f = _fields(case, psi)
        s.update(psi=psi.requires_grad_(), w=w, wu=wu, fields={k: f[k].requires_grad_() for k in FIELDS},
                 bar=_cotangent(case, seed, psi))
    elif kind == "vjp_density":
        s.update(psi=psi.requires_grad_(), w=w, wu=wu, bars=_density_bars(case, seed))
    return s


def _cotangent(case, seed, psi):
    g = np.random.default_rng([seed, 2])
    c = torch.from_numpy(g.standard_normal((psi.shape[0], 2, 2))).cuda()
    return (torch.roll(psi.detach(), 1, dims=0) * torch.complex(c[..., 0], c[..., 1])[..., None, None, None]).contiguous()


def _density_bars(case, seed):
    """Smooth cotangents of the six densities."""
    g = np.random.default_rng([seed, 3])
    x = _coords(case) / _radius(case)
    env = torch.exp(-(x[:, None, None] ** 2 + x[None, :, None] ** 2 + x[None, None, :] ** 2) / 2.0)
    out = {}
    for k in DENS:
        c = torch.from_numpy(g.standard_normal((2,) if k in DENS[:3] else (2, 3))).cuda()
        out[k] = (c[..., None, None, None] * env).contiguous()
    return out


# -------------------------------------------------------------------- runs --
def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_hpsi(s):
    return hfb.meanfield.hpsi01(s["grids"], s["mf"], 0, s["w"], s["wu"], s["psi"])


def _single(levels, out):
    """What was computed from single-precision states, in single precision."""
    if levels.psi.dtype == torch.complex128:
        return out
    to = {torch.float64: torch.float32, torch.complex128: torch.complex64}
    return {k: v.to(to.get(v.dtype, v.dtype)) for k, v in out.items()}


def _run_density(s):
    d, lv = s["dens"], s["levels"]
    hfb.densities.add_density(d, s["grids"], lv, mix=0.2, forces=s["forces"])
    return _single(lv, dict({k: getattr(d, k) for k in DENS}, sp_kinetic=lv.sp_kinetic))


def _run_fields(s):
    mf, co = hfb.meanfield.skyrme(s["coulomb"], s["dens"], s["forces"], s["grids"], s["mf"], s["params"], s["static"])
    hfb.energies.integ_energy(co, s["dens"], s["energies"], s["forces"], s["grids"], s["levels"], s["params"],
                              s["pairs"])
    return dict({k: getattr(mf, k) for k in FIELDS + ("divaq", "dbmass")}, wcoul=co.wcoul, energies=s["energies"].dev)


def _run_vjp_hpsi(s):
    y = hfb.vjp.hpsi(s["psi"], s["fields"], s["grids"], s["nneut"], s["w"], s["wu"])
    grads = torch.autograd.grad(y, [s["psi"]] + [s["fields"][k] for k in FIELDS], s["bar"])
    return dict(zip(("y", "psi") + FIELDS, (y.detach(),) + grads))


def _run_vjp_density(s):
    d = hfb.vjp.densities(s["psi"], s["grids"], s["nneut"], s["w"], s["wu"])
    grad, = torch.autograd.grad([d[k] for k in DENS], [s["psi"]], [s["bars"][k] for k in DENS])
    return dict({k: d[k].detach() for k in DENS}, psi=grad)


def _run_step(s):
    S = s["S"]
    lv, st = S["levels"], S["static"]
    hfb.static.grstep(S["forces"], S["grids"], lv, S["meanfield"], S["params"], st)
    hfb.static.diagstep(S["energies"], S["forces"], S["grids"], lv, st, False, True)
    return _single(lv, dict(psi=lv.psi, lagrange=lv.lagrange, hampsi=lv.hampsi, hmfpsi=lv.hmfpsi,
                            sp_energy=lv.sp_energy, sp_norm=lv.sp_norm, hmatrix=st.hmatrix, lam=st.lambda_save))


def _run_iterate(s):
    S = s["S"]
    hfb.static.iterate(s["i"], **S)
    s["i"] += 1
    lv, d, mf = S["levels"], S["densities"], S["meanfield"]
    out = dict({k: getattr(d, k) for k in DENS}, sp_energy=lv.sp_energy, sp_kinetic=lv.sp_kinetic, upot=mf.upot,
               bmass=mf.bmass, energies=S["energies"].dev)
    if s["pairing"]:
        out.update(wocc=lv.wocc, v_pair=mf.v_pair)
    else:
        out.update(psi=lv.psi, lagrange=lv.lagrange)
    return _single(lv, out)


# -------------------------------------------------------------------- work --
def work(case):
    n, kind = case["n"], case["kind"]
    n3 = n ** 3
    n0, n1 = case["npsi0"], case["npsi1"]
    ns = n0 + n1
    r = 4 if case["prec"] == "f32" else 8
    psi = 2 * n3 * 2 * r                      # bytes of one state
    fft = 2 * n3 * 5.0 * math.log2(n)         # flops of one set of line transforms of a state
    hpsi = 12 * fft + 300.0 * n3
    dens = 6 * fft + 150.0 * n3
    fields = 24 * n3 * 8
    skyrme = dict(bytes=fields + 32 * n3 * 8, flops=2 * 36 * 2.0 * n3 * n + 6 * 5.0 * 8 * n3 * math.log2(2 * n))
    if kind == "hpsi":
        return dict(bytes=4 * psi * n0 + 12 * n3 * r, flops=n0 * hpsi)
    if kind == "density":
        return dict(bytes=psi * ns + fields * 1.5, flops=ns * dens)
    if kind == "fields":
        return skyrme
    if kind == "vjp_hpsi":
        return dict(bytes=4 * psi * ns + 2 * fields, flops=ns * (2 * hpsi + 2 * dens))
    if kind == "vjp_density":
        return dict(bytes=2 * psi * ns + 2 * fields, flops=ns * (hpsi + dens))
    pair = 8.0 * 2 * n3 * (n0 * n0 + n1 * n1)   # one set of complex products of all pairs of states
    step = dict(bytes=(2 + 2 + 2) * psi * ns + 24 * n3 * r, flops=ns * (2 * hpsi + 2 * 3 * fft) + 3.0 * pair)
    if kind == "step":
        return step
    more = pair * 1.5 if case["pairing"] else 0.0
    return dict(bytes=step["bytes"] + skyrme["bytes"] + fields, flops=step["flops"] + more + skyrme["flops"] + ns * dens)


# ------------------------------------------------- the same in 64 bits -----
def _along(v, axis):
    s = [1, 1, 1]
    s[axis] = -1
    return v.reshape(s)


def _k(case):
    n, d = case["n"], case["d"]
    m = torch.arange(n, dtype=torch.float64, device="cuda")
    m = torch.where(m <= n // 2, m, m - n)
    return m * (2.0 * math.pi / (n * d))


def _x_diff(case, f, axis):
    """First derivative along one axis, the Nyquist mode left out."""
    k = _k(case).clone()
    k[case["n"] // 2] = 0.0
    return torch.fft.ifft(torch.fft.fft(f, dim=axis - 3) * _along(1j * k, axis), dim=axis - 3)


def _x_diff_b(case, d1, psi, b, axis):
    """d(B d psi) with the Nyquist mode of psi times the mean of B."""
    n, d = case["n"], case["d"]
    k = _k(case).clone()
    k[n // 2] = 0.0
    out = torch.fft.ifft(torch.fft.fft(b * d1, dim=axis - 3) * _along(1j * k, axis), dim=axis - 3)
    sign = _along(1.0 - 2.0 * (torch.arange(n, device="cuda") % 2).double(), axis)
    alt = (psi * sign).sum(dim=axis - 3, keepdim=True)
    return out - (math.pi / d) ** 2 / n * b.mean(dim=axis - 3, keepdim=True) * alt * sign


def _x_hpsi(case, f, iq, psi):
    """h psi of states of one isospin."""
    aq, sp, wl, b = f["aq"][iq], f["spot"][iq], f["wlspot"][iq], f["bmass"][iq]

    def lop(ax, a):
        p, q = a[:, 0], a[:, 1]
        if ax == 0:
            return torch.stack([-0.5j * (aq[0] - wl[1]) * p - 0.5 * wl[2] * q,
                                -0.5j * (aq[0] + wl[1]) * q + 0.5 * wl[2] * p], 1)
        if ax == 1:
            return torch.stack([-0.5j * (aq[1] + wl[0]) * p + 0.5j * wl[2] * q,
                                -0.5j * (aq[1] - wl[0]) * q + 0.5j * wl[2] * p], 1)
        return torch.stack([-0.5j * aq[2] * p + (0.5 * wl[0] - 0.5j * wl[1]) * q,
                            -0.5j * aq[2] * q + (-0.5 * wl[0] - 0.5j * wl[1]) * p], 1)

    p, q = psi[:, 0], psi[:, 1]
    u = f["upot"][iq]
    out = torch.stack([u * p + (sp[0] - 1j * sp[1]) * q + sp[2] * p, u * q + (sp[0] + 1j * sp[1]) * p - sp[2] * q], 1)
    for ax in range(3):
        d1 = _x_diff(case, psi, ax)
        out = out + lop(ax, d1) + _x_diff(case, lop(ax, psi), ax) - _x_diff_b(case, d1, psi, b, ax)
    return out


def _x_hpsi_all(case, f, psi):
    out = torch.empty_like(psi)
    for iq, b in enumerate(_blocks(case)):
        for s in range(b.start, b.stop, 16):
            e = min(s + 16, b.stop)
            out[s:e] = _x_hpsi(case, f, iq, psi[s:e])
    return out


def _col(v):
    return v[:, None, None, None, None]


def _x_density_block(case, psi, w, wu):
    a, b = psi[:, 0], psi[:, 1]
    ww = w[:, None, None, None]
    norm = (a * a.conj() + b * b.conj()).real
    rho = (ww * norm).sum(0)
    chi = (0.5 * wu[:, None, None, None] * norm).sum(0)
    ab = ww * a.conj() * b
    sdens = torch.stack([2.0 * ab.real.sum(0), 2.0 * ab.imag.sum(0), (ww * (a * a.conj() - b * b.conj()).real).sum(0)])
    tau, cur, j = 0.0, [], []
    for ax in range(3):
        q = _x_diff(case, psi, ax)
        tau = tau + (ww * (q * q.conj()).real.sum(1)).sum(0)
        uu, vv = ww * q[:, 0] * a.conj(), ww * q[:, 1] * b.conj()
        uv, vu = ww * q[:, 0] * b.conj(), ww * q[:, 1] * a.conj()
        cur.append((uu + vv).imag.sum(0))
        # Im(psi^+ sigma_s d psi) for s = x, y, z
        j.append([(vu + uv).imag.sum(0), (uv - vu).real.sum(0), (uu - vv).imag.sum(0)])
    so = torch.stack([j[1][2] - j[2][1], j[2][0] - j[0][2], j[0][1] - j[1][0]])
    return rho, chi, tau, torch.stack(cur), sdens, so


def _x_density(case, psi, w, wu):
    out = {k: [] for k in DENS}
    for b in _blocks(case):
        acc = None
        for s in range(b.start, b.stop, 16):
            e = min(s + 16, b.stop)
            part = _x_density_block(case, psi[s:e], w[s:e], wu[s:e])
            acc = part if acc is None else [x + y for x, y in zip(acc, part)]
        for k, v in zip(DENS, acc):
            out[k].append(v)
    return {k: torch.stack(v) for k, v in out.items()}


def _x_kinetic(case, psi, h2m):
    k = _k(case)
    k2 = _along(k ** 2, 0) + _along(k ** 2, 1) + _along(k ** 2, 2)
    out = torch.empty(psi.shape[0], dtype=torch.float64, device="cuda")
    for s in range(psi.shape[0]):
        f = torch.fft.fftn(psi[s], dim=(1, 2, 3))
        out[s] = h2m * case["d"] ** 3 * ((f * f.conj()).real * k2).sum() / case["n"] ** 3
    return out


_E2 = 1.4399784085965135


def _force():
    """SLy4 coefficients."""
    t0, t1, t2, t3, t4 = -2488.913, 486.818, -546.395, 13777.0, 123.0
    x0, x1, x2, x3, b4p, power = 0.834, -0.344, -1.0, 1.354, 61.5, 0.1666667
    f = dict(b0=t0 * (1 + 0.5 * x0), b0p=t0 * (0.5 + x0),
             b1=(t1 * (1 + 0.5 * x1) + t2 * (1 + 0.5 * x2)) / 4, b1p=(t1 * (0.5 + x1) - t2 * (0.5 + x2)) / 4,
             b2=(3 * t1 * (1 + 0.5 * x1) - t2 * (1 + 0.5 * x2)) / 8, b2p=(3 * t1 * (0.5 + x1) + t2 * (0.5 + x2)) / 8,
             b3=t3 * (1 + 0.5 * x3) / 4, b3p=t3 * (0.5 + x3) / 4, b4=t4 / 2, b4p=b4p, power=power,
             slate=(3 / math.pi) ** (1 / 3) * _E2, v0=(286.669, 295.369))
    return f


def _h2m(case):
    a = case["nneut"] + case["nprot"]
    return 20.735530 * (a - 1.0) / a


def _matrices(case):
    """Dense first and second derivative matrices of the fields (the Nyquist
    mode kept in the second)."""
    n, d = case["n"], case["d"]
    i = np.arange(n)
    diff = i[:, None] - i[None, :]
    kf = 2.0 * np.pi / (n * d)
    d1 = sum(-2.0 / n * k * kf * np.sin(2 * np.pi * k * diff / n) for k in range(1, n // 2))
    d2 = sum(-2.0 / n * (k * kf) ** 2 * np.cos(2 * np.pi * k * diff / n) for k in range(1, n // 2))
    d2 = d2 - (np.pi / d) ** 2 / n * np.cos(np.pi * diff)
    return torch.from_numpy(d1).cuda(), torch.from_numpy(d2).cuda()


def _apply(m, f, axis):
    return torch.movedim(torch.tensordot(f, m, dims=([f.dim() - 3 + axis], [1])), -1, f.dim() - 3 + axis)


def _curl(d1, v):
    d = lambda c, ax: _apply(d1, v[:, c], ax)  # noqa: E731
    return torch.stack([d(2, 1) - d(1, 2), d(0, 2) - d(2, 0), d(1, 0) - d(0, 1)], 1)


def _div(d1, v):
    return sum(_apply(d1, v[:, a], a) for a in range(3))


def _x_coulomb(case, rho):
    n, d = case["n"], case["d"]
    m = torch.arange(2 * n, dtype=torch.float64, device="cuda")
    m = (torch.where(m <= n, m, m - 2 * n) * d) ** 2
    r2 = _along(m, 0) + _along(m, 1) + _along(m, 2)
    r2[0, 0, 0] = 1.0
    q = 1.0 / torch.sqrt(r2)
    q[0, 0, 0] = 2.84 / d
    big = torch.zeros_like(q)
    big[:n, :n, :n] = rho
    w = torch.fft.ifftn(torch.fft.fftn(big) * torch.fft.fftn(q)).real * (_E2 * d ** 3)
    return w[:n, :n, :n].contiguous()


def _x_skyrme(case, dens):
    """Mean fields of the densities (volume pairing strengths in v_pair)."""
    f = _force()
    d1, d2 = _matrices(case)
    rho, tau = dens["rho"], dens["tau"]

    def mix(a, b, x):          # (a + b) x_q + a x_q'
        return (a + b) * x + a * x.flip(0)

    rt = rho.sum(0)
    p, b3, b3p = f["power"], f["b3"], f["b3p"]
    up = rt ** p * (b3 * (p + 2) / 3 * rt - 2 * b3p / 3 * rho
                    - b3p * p / 3 * (rho[0] ** 2 + rho[1] ** 2) / (rt + 1e-25))
    up = up - mix(f["b4"], f["b4p"], _div(d1, dens["sodens"]))
    wc = _x_coulomb(case, rho[1])
    up[1] = up[1] + wc - f["slate"] * rho[1] ** (1.0 / 3.0)
    lap = sum(_apply(d2, rho, a) for a in range(3))
    up = up + mix(f["b0"], -f["b0p"], rho) + mix(f["b1"], -f["b1p"], tau) - mix(f["b2"], -f["b2p"], lap)
    bm = _h2m(case) + mix(f["b1"], -f["b1p"], rho)
    wl = mix(f["b4"], f["b4p"], torch.stack([_apply(d1, rho, a) for a in range(3)], 1))
    aq = -2.0 * mix(f["b1"], -f["b1p"], dens["current"]) - mix(f["b4"], f["b4p"], _curl(d1, dens["sdens"]))
    sp = -mix(f["b4"], f["b4p"], _curl(d1, dens["current"]))
    v0 = torch.tensor(f["v0"], dtype=torch.float64, device="cuda")[:, None, None, None]
    return dict(upot=up, bmass=bm, v_pair=v0 * dens["chi"], aq=aq, spot=sp, wlspot=wl, divaq=_div(d1, aq),
                dbmass=torch.stack([_apply(d1, bm, a) for a in range(3)], 1), wcoul=wc)


def _x_energies(case, dens, wcoul, epair=0.0):
    """The 24 values of hfb.energies, without the sums over the states."""
    f = _force()
    d1, d2 = _matrices(case)
    w = case["d"] ** 3
    rho, tau, cur, sd = (dens[k] for k in ("rho", "tau", "current", "sdens"))
    lap = sum(_apply(d2, rho, a) for a in range(3))
    dj = _div(d1, dens["sodens"])
    cc = _curl(d1, cur)
    iso = lambda x: (x[0] + x[1], x[1] - x[0])  # noqa: E731
    (rt, r1), (t0, t1), (l0, l1), (j0, j1) = iso(rho), iso(tau), iso(lap), iso(dj)
    s = lambda x: float(w * x.sum())  # noqa: E731
    p = f["power"]
    e = dict.fromkeys(hfb._lib.ENERGY_KEYS, 0.0)
    e["ehft"] = s(_h2m(case) * t0)
    e["ehf0"] = s((f["b0"] * rt ** 2 - f["b0p"] * (rho ** 2).sum(0)) / 2)
    e["ehf1"] = s(f["b1"] * rt * t0 - f["b1p"] * (rho * tau).sum(0))
    e["ehf2"] = s((-f["b2"] * rt * l0 + f["b2p"] * (rho * lap).sum(0)) / 2)
    e["ehf3"] = s(rt ** p * (f["b3"] * rt ** 2 - f["b3p"] * (rho ** 2).sum(0)) / 3)
    e["ehflsodd"] = s(-f["b4"] * (sd.sum(0) * cc.sum(0)).sum(0) - f["b4p"] * (sd * cc).sum((0, 1)))
    e["ehfls"] = s(-f["b4"] * rt * j0 - f["b4p"] * (rho * dj).sum(0)) + e["ehflsodd"]
    sl = -0.75 * f["slate"] * rho[1] ** (4.0 / 3.0)
    e["ehfc"], e["ecorc"] = s(0.5 * rho[1] * wcoul + sl), s(sl / 3)
    e["e3corr"] = -p * e["ehf3"] / 2
    e["ehfCrho0"] = s((0.5 * f["b0"] - 0.25 * f["b0p"] + (f["b3"] / 3 - f["b3p"] / 6) * rt ** p) * rt ** 2)
    e["ehfCrho1"] = s((-0.25 * f["b0p"] - f["b3p"] / 6 * rt ** p) * r1 ** 2)
    e["ehfCdrho0"] = s((-0.5 * f["b2"] + 0.25 * f["b2p"]) * rt * l0)
    e["ehfCdrho1"] = s(0.25 * f["b2p"] * r1 * l1)
    c0, c1 = f["b1"] - 0.5 * f["b1p"], -0.5 * f["b1p"]
    e["ehfCtau0"], e["ehfCtau1"] = s(c0 * t0 * rt), s(c1 * t1 * r1)
    e["ehfCdJ0"], e["ehfCdJ1"] = s((-f["b4"] - 0.5 * f["b4p"]) * rt * j0), s(-0.5 * f["b4p"] * r1 * j1)
    # the reference indexes the last two axes of the current in these two
    e["ehfCj0"] = -w * c0 * float(sum(((cur[..., a, 0] + cur[..., a, 1]) ** 2).sum() for a in range(3)))
    e["ehfCj1"] = -w * c1 * float(sum(((cur[..., a, 1] - cur[..., a, 0]) ** 2).sum() for a in range(3)))
    e["ehfint"] = (e["ehft"] + e["ehf0"] + e["ehf1"] + e["ehf2"] + e["ehf3"] + e["ehfls"] + e["ehfc"]
                   - float(np.sum(epair)))
    return e


def _x_gradient(case, S, first):
    """One damped gradient step of S["psi"] in the fields S["f"]."""
    f, psi, w3, n = S["f"], S["psi"], case["d"] ** 3, case["n"]
    k = _k(case)
    k2 = _along(k ** 2, 0) + _along(k ** 2, 1) + _along(k ** 2, 2)
    bcs = case["pairing"]
    S["ham"] = _x_hpsi_all(case, f, psi)
    wocc = torch.ones_like(S["wocc"]) if bcs else S["wocc"]
    wguv = torch.zeros_like(S["wocc"]) if bcs else S["wguv"]
    vmax = [0.0 if bcs else float(f["v_pair"][q].max()) for q in (0, 1)]
    new = torch.empty_like(psi)
    for s in range(psi.shape[0]):
        iq = int(s >= case["npsi0"])
        w, wu = float(wocc[s]), float(wguv[s])
        g = w * S["ham"][s] - wu * f["v_pair"][iq] * psi[s]
        if first or bcs:
            g = g - w3 * (psi[s].conj() * g).sum().real * psi[s]
        else:
            g = g - S["lag"][s]
        den = max(w, 0.1) * (100.0 + 20.735530 * k2) + 0.5 * max(wu, 0.1) * vmax[iq]
        new[s] = psi[s] - S["x0"] * torch.fft.ifftn(torch.fft.fftn(g, dim=(1, 2, 3)) / den, dim=(1, 2, 3))
    S["psi"] = new
    S["hmf"] = _x_hpsi_all(case, f, new)


def _x_orthonormalise(case, S, eigen):
    w3, nmax = case["d"] ** 3, max(case["npsi0"], case["npsi1"])
    S["lag"] = torch.empty_like(S["psi"])
    S["h"] = torch.zeros((2, nmax, nmax), dtype=torch.complex128, device="cuda")
    S["lam"] = torch.zeros_like(S["h"])
    S["fluct"] = []
    for iq, b in enumerate(_blocks(case)):
        ns = b.stop - b.start
        p = S["psi"][b].reshape(ns, -1)
        prod = lambda x: w3 * (p.conj() @ x.reshape(ns, -1).T)  # noqa: E731
        ov = prod(p)
        S["norm"][b] = ov.diagonal().real
        val, vec = torch.linalg.eigh(ov)
        u = (vec / torch.sqrt(val)) @ vec.conj().T
        if eigen:
            u = u @ torch.linalg.eigh(prod(S["ham"][b]))[1]
        h = u.conj().T @ prod(S["hmf"][b]) @ u
        g = u.conj().T @ prod(S["f"]["v_pair"][iq] * S["psi"][b]) @ u
        if case["pairing"]:
            S["delta"][b] = g.diagonal().real * S["pairwg"][b]
            g = torch.diag(g.diagonal())
        else:
            g = torch.zeros_like(h)
        lam = S["wocc"][b][None, :] * h - (S["wguv"] * S["pairwg"])[b][None, :] * g
        off = (0.5 * (lam - lam.conj().T)).abs()
        S["fluct"].append((float(off.max()), float(torch.sqrt((off ** 2).sum())) / ns))
        lam = 0.5 * (lam + lam.conj().T)
        new = (p.T @ u).T
        S["e"][b] = h.diagonal().real
        S["h"][iq, :ns, :ns], S["lam"][iq, :ns, :ns] = h, lam
        S["psi"][b] = new.reshape(S["psi"][b].shape)
        S["lag"][b] = (new.T @ lam).T.reshape(S["psi"][b].shape)


def _x_bcs(case, S, const_gap):
    if const_gap:
        S["delta"].fill_(11.2 / math.sqrt(case["nneut"] + case["nprot"]))
    S["epair"] = []
    for iq, b in enumerate(_blocks(case)):
        e, gap = S["e"][b].cpu().numpy(), S["delta"][b].cpu().numpy()

        def occ(ef):
            return 0.5 * (1.0 - (e - ef) / np.maximum(np.sqrt((e - ef) ** 2 + gap ** 2), 1e-20))

        lo, hi = -100.0, 100.0
        for _ in range(200):
            mid = 0.5 * (lo + hi)
            lo, hi = ((mid, hi) if np.sum(np.clip(occ(mid), 1e-10, 1 - 1e-10)) < (case["nneut"], case["nprot"])[iq]
                      else (lo, mid))
        v2 = occ(0.5 * (lo + hi))
        uv = np.sqrt(np.maximum(v2 - v2 ** 2, 1e-6))
        S["pairwg"][b] = torch.from_numpy(1.0 / (1.0 + np.exp((e - 0.5 * (lo + hi) - 60.0) / 6.0))).cuda()
        S["wocc"][b] = torch.from_numpy(np.clip(v2, 1e-10, 1 - 1e-10)).cuda()
        S["wguv"][b] = torch.from_numpy(uv).cuda()
        S["epair"].append(float(np.sum(0.5 * uv * gap)))


def _x_solver(case, seed):
    """The state hfb.static.prepare leaves."""
    psi = _states(case, seed)
    ns = psi.shape[0]
    z = lambda v=0.0: torch.full((ns,), v, dtype=torch.float64, device="cuda")  # noqa: E731
    S = dict(psi=psi, wocc=z(), wguv=z(), pairwg=z(1.0), e=z(), delta=z(), norm=z(), x0=0.2, epair=[0.0, 0.0])
    for b, particles in zip(_blocks(case), (case["nneut"], case["nprot"])):
        S["wocc"][b.start:b.start + particles] = 1.0
        p = psi[b].reshape(b.stop - b.start, -1)
        val, vec = torch.linalg.eigh(case["d"] ** 3 * (p.conj() @ p.T))
        psi[b] = (p.T @ ((vec / torch.sqrt(val)) @ vec.conj().T)).T.reshape(psi[b].shape)
    S["dens"] = _x_density(case, psi, S["wocc"], S["wguv"] * S["pairwg"])
    S["f"] = _x_skyrme(case, S["dens"])
    if not case["pairing"]:
        S["f"]["v_pair"].zero_()
    _x_gradient(case, S, True)
    if case["pairing"]:
        # the gradient step leaves <h> of the states before it
        S["e"] = torch.stack([case["d"] ** 3 * (psi[s].conj() * S["ham"][s]).sum().real for s in range(ns)])
        _x_bcs(case, S, True)
    _x_orthonormalise(case, S, False)
    S["x0"] *= 3.0
    S["before"] = (0.0, 0.0, 0.0)
    for _ in range(_START * case["pairing"]):
        e = _x_iterate(case, S, True)["ehf"]
        f1, f2 = max(x[0] for x in S["fluct"]), 0.5 * sum(x[1] for x in S["fluct"])
        e0, p1, p2 = S["before"]
        better = (e < e0 and f1 < p1 * (1.0 - 1e-5)) or f2 < p2 * (1.0 - 1e-5)
        S["x0"] = min(max(S["x0"] * (1.005 if better else 0.8), 0.2), 1.0)
        S["before"] = (e, f1, f2)
    return S


def exact(case, seed):
    with torch.no_grad():
        return globals()["_exact_" + case["kind"]](case, seed)


def _exact_hpsi(case, seed):
    psi = _states(case, seed)
    b = _blocks(case)[0]
    w, wu = (x[b] for x in _weights(case))
    f = _fields(case, psi)
    if case["prec"] == "f32":   # the potentials are an input in the precision of the states
        f = {k: v.float().double() for k, v in f.items()}
    h = _x_hpsi_all(case, f, psi)[b]
    v = f["v_pair"][0] * psi[b]
    return _col(w) * h - _col(wu) * v, h, v


def _exact_density(case, seed):
    psi = _states(case, seed)
    w, wu = _weights(case)
    d = _x_density(case, psi, w, wu)
    mixed = {k: 0.2 * v if k in ("rho", "tau", "chi") else v for k, v in d.items()}
    return dict(mixed, sp_kinetic=_x_kinetic(case, psi, 20.735530))


def _exact_fields(case, seed):
    w, wu = _weights(case)
    dens = _x_density(case, _states(case, seed), w, wu)
    f = _x_skyrme(case, dens)
    e = _x_energies(case, dens, f["wcoul"])
    out = {k: f[k] for k in FIELDS + ("divaq", "dbmass", "wcoul")}
    return dict(out, energies=torch.tensor([e[k] for k in hfb._lib.ENERGY_KEYS], dtype=torch.float64))


def _exact_vjp_hpsi(case, seed):
    psi = _states(case, seed)
    f = _fields(case, psi)
    w, wu = _weights(case)
    bar = _cotangent(case, seed, psi)
    y, gp = torch.empty_like(psi), torch.empty_like(psi)
    gf = {k: torch.zeros_like(f[k]) for k in FIELDS}
    with torch.enable_grad():
        for iq, b in enumerate(_blocks(case)):
            for s in range(b.start, b.stop, 8):
                e = min(s + 8, b.stop)
                x = psi[s:e].clone().requires_grad_()
                leaf = {k: f[k].clone().requires_grad_() for k in FIELDS}
                out = _col(w[s:e]) * _x_hpsi(case, leaf, iq, x) - _col(wu[s:e]) * leaf["v_pair"][iq] * x
                g = torch.autograd.grad(out, [x] + [leaf[k] for k in FIELDS], bar[s:e])
                y[s:e], gp[s:e] = out.detach(), g[0]
                for k, v in zip(FIELDS, g[1:]):
                    gf[k] += v
    return dict(gf, y=y, psi=gp)


def _exact_vjp_density(case, seed):
    psi = _states(case, seed)
    w, wu = _weights(case)
    bars = _density_bars(case, seed)
    grad = torch.empty_like(psi)
    with torch.enable_grad():
        for iq, b in enumerate(_blocks(case)):
            for s in range(b.start, b.stop, 8):
                e = min(s + 8, b.stop)
                x = psi[s:e].clone().requires_grad_()
                out = _x_density_block(case, x, w[s:e], wu[s:e])
                grad[s:e], = torch.autograd.grad(out, [x], [bars[k][iq] for k in DENS])
    return dict(_x_density(case, psi, w, wu), psi=grad)


def _exact_step(case, seed):
    S = _x_solver(case, seed)
    _x_gradient(case, S, False)
    _x_orthonormalise(case, S, False)
    return dict(psi=S["psi"], lagrange=S["lag"], hampsi=S["ham"], hmfpsi=S["hmf"], sp_energy=S["e"],
                sp_norm=S["norm"], hmatrix=S["h"], lam=S["lam"])


def _x_iterate(case, S, const_gap):
    """One iteration of the loop; the energies as a dict."""
    _x_gradient(case, S, False)
    _x_orthonormalise(case, S, case["pairing"])
    if case["pairing"]:
        _x_bcs(case, S, const_gap)
    d = _x_density(case, S["psi"], S["wocc"], S["wguv"] * S["pairwg"])
    for k in ("rho", "tau", "chi"):
        d[k] = 0.2 * d[k] + 0.8 * S["dens"][k]
    S["dens"], S["f"] = d, _x_skyrme(case, d)
    S["kin"] = _x_kinetic(case, S["psi"], _h2m(case))
    e = _x_energies(case, d, S["f"]["wcoul"], S["epair"])
    e["tke"] = float((S["wocc"] * S["kin"]).sum())
    e["ehf"] = float((S["wocc"] * (S["kin"] + S["e"])).sum()) / 2 + e["e3corr"] + e["ecorc"] - float(np.sum(S["epair"]))
    return e


def _exact_iterate(case, seed):
    S = _x_solver(case, seed)
    e = _x_iterate(case, S, False)
    out = dict(S["dens"], sp_energy=S["e"], sp_kinetic=S["kin"], upot=S["f"]["upot"], bmass=S["f"]["bmass"],
               energies=torch.tensor([e[k] for k in hfb._lib.ENERGY_KEYS], dtype=torch.float64))
    if case["pairing"]:
        out.update(wocc=S["wocc"], v_pair=S["f"]["v_pair"])
    else:
        out.update(psi=S["psi"], lagrange=S["lag"])
    return out
