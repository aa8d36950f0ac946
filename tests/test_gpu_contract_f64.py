"""FP64 Gram and rotation (csrc/contract_f64.cu) at the edges of their tiles
(48, 32, 24 and 16 states; 8 to 48 output columns) against NumPy.  Sums of
K = 2 8^3 (or 2 16^3) terms of random data: rounding is below sqrt(K) eps
times the norms, so 1e-12 relative to the largest element."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _grid(n):
    import hfb
    return hfb.grids.init_grids(hfb.params.init_params(), nx=n, ny=n, nz=n, dx=0.8, dy=0.8, dz=0.8)


def _rand(rng, *s):
    return rng.standard_normal(s) + 1j * rng.standard_normal(s)


@pytest.mark.parametrize("n,ns", [(8, 1), (8, 8), (8, 16), (8, 17), (8, 24), (16, 25), (8, 32), (8, 33), (16, 48),
                                  (8, 49), (8, 64), (8, 96), (8, 97), (8, 145)])
def test_gram_tiles(n, ns):
    from hfb._lib import call, ptr, stream_ptr, HFB_F64
    rng = np.random.default_rng(ns)
    K = 2 * n ** 3
    g = _grid(n)
    psi, ham = _rand(rng, ns, K), _rand(rng, ns, K)
    f = rng.standard_normal((2, n ** 3))
    hmf = psi * np.tile(f[0], 2)
    out = torch.zeros((4, ns, ns), dtype=torch.complex128, device="cuda")
    P, H, M, V = (torch.from_numpy(a).cuda() for a in (psi, ham, hmf, f[1].copy()))
    for _ in range(2):   # twice: the tickets start over
        out.zero_()
        call("hfb_gram", g.ctx.handle, HFB_F64, 0, ns, 15, ptr(P), ptr(H), ptr(M), ptr(V), 0.7, ptr(out), stream_ptr())
        o = out.cpu().numpy()
        for a, x in enumerate((psi, ham, hmf, psi * np.tile(f[1], 2))):
            ref = 0.7 * psi.conj() @ x.T
            assert np.max(np.abs(o[a] - ref)) <= 1e-12 * np.max(np.abs(ref)), a


@pytest.mark.parametrize("npsi", [(1, 1), (4, 5), (8, 9), (12, 13), (16, 20), (24, 23), (33, 31), (70, 48)])
def test_rotation_tiles(npsi):
    """psi U and psi L through the diagonalisation step: U and U lambda from
    the overlap and H matrices of the same states."""
    from test_gpu_diag_chains import _run
    st, psi, ham, hmf, vpsi, w, uv, pw = _run(npsi, False, False, 0, seed=5)
    lv, dv = st["levels"], 0.9 ** 3
    new, lag = (t.cpu().numpy().reshape(psi.shape) for t in (lv.psi, lv.lagrange))
    lam = st["static"].lambda_save.cpu().numpy()
    for iq in range(2):
        b = slice(0, npsi[0]) if iq == 0 else slice(npsi[0], sum(npsi))
        p = psi[b]
        val, vec = np.linalg.eigh(dv * p.conj() @ p.T)
        ref = (p.T @ ((vec / np.sqrt(val)) @ vec.conj().T)).T
        assert np.max(np.abs(new[b] - ref)) <= 1e-11 * np.max(np.abs(ref))
        ref = (ref.T @ lam[iq, :npsi[iq], :npsi[iq]]).T
        assert np.max(np.abs(lag[b] - ref)) <= 1e-11 * np.max(np.abs(ref))
