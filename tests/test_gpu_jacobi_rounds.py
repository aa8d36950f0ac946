"""The Jacobi eigensolver where its rounds differ: one to three pairs (blocks
of several kinds coincide), 31 to 33 pairs (rotations in the round itself or in
the one before, one rotating warp or two), the folded triangle at odd and even
halves, and the largest size.  Degenerate pairs as time reversal gives them.
Bounds as for the solver's other sizes: 1e-11 of the largest eigenvalue, 1e-12
for orthogonality."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 8, 34, 61, 62, 63, 64, 66, 130, 167, 168])
def test_jacobi_rounds(n):
    import hfb
    from hfb._lib import call, ptr, stream_ptr
    g = hfb.grids.init_grids(hfb.params.init_params(), nx=8, ny=8, nz=8, dx=1.0, dy=1.0, dz=1.0)
    rng = np.random.default_rng(n)
    mats = []
    for scale in (0.02, 1.0):   # nearly diagonal (rounds without rotations), full
        d = np.repeat(np.sort(rng.uniform(-60.0, 40.0, (n + 1) // 2)), 2)[:n]
        h = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
        mats.append(np.diag(d) + scale * (h + h.conj().T))
    at = torch.from_numpy(np.ascontiguousarray(mats)).cuda()
    w = torch.empty((2, n), dtype=torch.float64, device="cuda")
    v = torch.empty((2, n, n), dtype=torch.complex128, device="cuda")
    call("hfb_eigh", g.ctx.handle, 2, n, n, ptr(at), ptr(w), ptr(v), None, stream_ptr())
    g.ctx.check("eigh")
    for b, m in enumerate(mats):
        ref, wn, vn = np.linalg.eigvalsh(m), w[b].cpu().numpy(), v[b].cpu().numpy()
        top = np.max(np.abs(ref))
        assert np.max(np.abs(wn - ref)) < 1e-11 * top
        assert np.max(np.abs(vn.conj().T @ vn - np.eye(n))) < 1e-12
        assert np.max(np.abs(vn.conj().T @ m @ vn - np.diag(wn))) < 1e-11 * top
