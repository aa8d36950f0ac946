"""Packed potentials of hfb.vjp: missing, broadcast, strided, single-precision
and host fields, in both precisions, against plain tensor copies."""
import pytest
import torch

pytestmark = pytest.mark.gpu

FIELDS = ("upot", "bmass", "v_pair", "aq", "spot", "wlspot")


@pytest.mark.parametrize("n", [8, 24])
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
def test_pack_accepts_every_form(n, dtype):
    import hfb
    from hfb import vjp
    g = hfb.grids.init_grids(hfb.params.init_params(), nx=n, ny=n, nz=n, dx=0.9, dy=1.0, dz=1.1)
    torch.manual_seed(n)
    f = dict(upot=torch.randn(2, n, n, n, dtype=torch.float64, device="cuda"),
             bmass=torch.randn(1, n, n, n, dtype=torch.float64, device="cuda"),                    # broadcast
             v_pair=torch.randn(2, n, n, n, dtype=torch.float32, device="cuda"),                   # converted
             aq=torch.randn(2, n, n, n, 3, dtype=torch.float64, device="cuda").movedim(-1, 1),     # strided
             spot=torch.randn(2, 3, n, n, n, dtype=torch.float64))                                 # on the host
    rd = torch.float64 if dtype == torch.complex128 else torch.float32
    ref = torch.zeros((2, 12, n, n, n), dtype=rd, device="cuda")
    for k, sl in (("upot", 0), ("bmass", 1), ("v_pair", 2), ("aq", slice(3, 6)), ("spot", slice(6, 9))):
        ref[:, sl] = f[k].to(device="cuda", dtype=torch.float64).to(rd)
    assert torch.equal(vjp._pack(g, f, dtype).pot, ref)
    assert torch.equal(vjp._pack(g, {}, dtype).pot, torch.zeros_like(ref))
