"""Mean fields, Coulomb potential and energies on every grid size with unequal
spacings, non-periodic and periodic, against the oracle.  Sums of at most
3 x 48 products in double precision: 1e-11 relative to the largest value
(the energies, sums over the grid with cancellation, 1e-10)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

D = (0.9, 1.0, 1.1)


def _densities(n, rng):
    x = [(np.arange(n) - (n - 1) / 2) * d for d in D]
    r2 = x[0][:, None, None] ** 2 + x[1][None, :, None] ** 2 + x[2][None, None, :] ** 2
    e = np.exp(-r2 / (0.08 * (n * 0.9) ** 2))
    wave = 1.0 + 0.1 * np.cos(x[0][:, None, None]) * np.sin(x[1][None, :, None] + 0.3 * x[2][None, None, :])
    s = {k: rng.uniform(0.02, 0.09, 2)[:, None, None, None] * e * wave for k in ("rho", "tau", "chi")}
    v = {k: rng.uniform(-0.02, 0.02, (2, 3))[:, :, None, None, None] * e * wave for k in ("current", "sdens", "sodens")}
    return {k: np.ascontiguousarray(a) for k, a in {**s, **v}.items()}


@pytest.mark.parametrize("periodic,ipair", [(False, 5), (True, 6)])
@pytest.mark.parametrize("n", [8, 16, 24, 32, 40, 48])
def test_fields_against_oracle(n, periodic, ipair):
    import hfb
    from oracle import model, densities as od, meanfield as omf, coulomb as oc, energies as oe, pairs as op
    rng = np.random.default_rng(n)
    dens = _densities(n, rng)
    grid = dict(nx=n, ny=n, nz=n, dx=D[0], dy=D[1], dz=D[2], periodic=periodic)
    force = dict(name="SLy4", ipair=ipair, v0prot=300.0, v0neut=290.0, rho0pr=0.16 if ipair == 6 else 0.0)
    # oracle
    go, fo = model.init_grids(**grid), model.init_forces(**force)
    do = od.Densities(**dens)
    mo, co = omf.skyrme(oc.init_coulomb(go), do, fo, go, omf.init_meanfield(go))
    lo = model.init_levels(go, 1, 1, (1, 1))
    eo = oe.integ_energy(co, do, oe.Energies(), fo, go, lo, op.Pairs())
    # device
    p = hfb.params.init_params()
    g, f = hfb.grids.init_grids(p, **grid), hfb.forces.init_forces(p, **force)
    d = hfb.densities.init_densities(g)
    for k, a in dens.items():
        getattr(d, k).copy_(torch.from_numpy(a))
    c, en, lv = hfb.coulomb.init_coulomb(g), hfb.energies.init_energies(), hfb.levels.init_levels(g, 1, 1, (1, 1))
    st = type("S", (), {"outertype": "N"})()
    for dtype in (torch.complex128, torch.complex64):
        mf = hfb.meanfield.init_meanfield(g, dtype)
        hfb.meanfield.skyrme(c, d, f, g, mf, p, st, dtype=dtype)
        for k in ("upot", "bmass", "divaq", "v_pair", "aq", "spot", "wlspot", "dbmass"):
            ref = getattr(mo, k)
            # div aq and grad bmass of the oracle carry the rounding of the terms that cancel in them
            scale = np.max(np.abs(ref)) + (np.max(np.abs(mo.aq)) + np.max(np.abs(mo.bmass)) if k in ("divaq", "dbmass") else 0)
            assert np.max(np.abs(getattr(mf, k).cpu().numpy() - ref)) <= 1e-11 * scale, k
        packed = mf.pot.clone()
        assert torch.equal(packed, mf.pack(dtype).pot)
        assert np.max(np.abs(c.wcoul.cpu().numpy() - co.wcoul)) <= 1e-11 * np.max(np.abs(co.wcoul))
        assert abs(mf.ecorrp - mo.ecorrp) <= 1e-10 * max(1.0, abs(mo.ecorrp))
    hfb.energies.integ_energy(c, d, en, f, g, lv, p, hfb.pairs.Pairs())
    en.sync()
    for k in ("ehft", "ehf0", "ehf1", "ehf2", "ehf3", "ehfls", "ehflsodd", "ehfc", "ecorc", "ehfint", "ehfCdrho0",
              "ehfCdrho1", "ehfCdJ0", "ehfCdJ1", "ehfCj0", "ehfCj1"):
        assert abs(getattr(en, k) - getattr(eo, k)) <= 1e-10 * max(1.0, abs(eo.ehf0)), k
