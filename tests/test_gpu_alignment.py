"""Single-precision states whose data is off a 16-byte boundary (a contiguous
view at an odd element offset): hpsi01 and the reverse mode copy them first, so
the results are those of aligned states to the bit.  (What the C entries do
with such an address is checked on the CPU: they refuse it.)"""
import pytest
import torch

pytestmark = pytest.mark.gpu

N = 24


def _off(x):
    """``x`` 8 bytes off a 16-byte boundary."""
    buf = torch.empty(x.numel() + 2, dtype=x.dtype, device=x.device)
    view = buf[1:1 + x.numel()].view(x.shape)
    view.copy_(x)
    assert view.data_ptr() % 16 == 8 and view.is_contiguous()
    return view


@pytest.fixture(scope="module")
def setup():
    import hfb
    g = hfb.grids.init_grids(hfb.params.init_params(), nx=N, ny=N, nz=N, dx=0.9, dy=0.9, dz=0.9)
    gen = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, dtype=torch.float64, device="cuda", generator=gen)  # noqa: E731
    psi = torch.complex(r(3, 2, N, N, N), r(3, 2, N, N, N)).to(torch.complex64)
    f = {k: r(2, N, N, N) for k in ("upot", "bmass", "v_pair")}
    f.update({k: r(2, 3, N, N, N) for k in ("aq", "spot", "wlspot")})
    return hfb, g, psi, f


def test_hpsi01_of_misaligned_states(setup):
    hfb, g, psi, f = setup
    mf = hfb.meanfield.init_meanfield(g, torch.complex64)
    for k, v in f.items():
        getattr(mf, k).copy_(v)
    mf.pack(torch.complex64)
    for a, b in zip(hfb.meanfield.hpsi01(g, mf, 0, 0.8, 0.3, psi), hfb.meanfield.hpsi01(g, mf, 0, 0.8, 0.3, _off(psi))):
        assert torch.equal(a, b)


def test_reverse_mode_of_misaligned_states(setup):
    _, g, psi, f = setup
    from hfb import vjp
    w, wu = (torch.linspace(a, b, 3, dtype=torch.float64, device="cuda") for a, b in ((0.3, 1.0), (0.1, 0.4)))
    yb = psi.flip(0).contiguous()
    pot = vjp._pack(g, f, torch.complex64).pot
    p0, b0 = vjp.hpsi_vjp(g, pot, psi, 2, w, wu, yb)
    p1, b1 = vjp.hpsi_vjp(g, pot, _off(psi), 2, w, wu, _off(yb))
    assert torch.equal(p0, p1) and all(torch.equal(b0[k], b1[k]) for k in b0)
    bars = dict(rho=f["upot"], chi=f["v_pair"], tau=f["bmass"], current=f["aq"], sdens=f["spot"], sodens=f["wlspot"])
    assert torch.equal(vjp.densities_vjp(g, psi, 2, w, wu, bars), vjp.densities_vjp(g, _off(psi), 2, w, wu, bars))
