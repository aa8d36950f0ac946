"""The k-space preconditioner (hfb_laplace) against numpy's FFT on every grid
size, out of place and in place: lines of 2, 4 and 8 lanes, exchange buffers in
the rows of the plane, threads past the last line (n = 8).  FP64: two
transforms of n^3 terms and a division, rounding of a few eps log2(n^3) in the
norm: 1e-13.  FP32: the same with 6e-8: 3e-6."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,tol", [(torch.complex128, 1e-13), (torch.complex64, 3e-6)])
@pytest.mark.parametrize("n", [8, 16, 24, 32, 40, 48])
def test_precond_every_grid(n, dtype, tol):
    import hfb
    from hfb._lib import call, ptr, stream_ptr, prec_of
    d = (0.8, 0.9, 1.0)
    g = hfb.grids.init_grids(hfb.params.init_params(), nx=n, ny=n, nz=n, dx=d[0], dy=d[1], dz=d[2])
    rng = np.random.default_rng(n)
    ns, e0, h2ma, vmax = 3, 100.0, 20.7, 3.5
    psi = rng.standard_normal((ns, 2, n, n, n)) + 1j * rng.standard_normal((ns, 2, n, n, n))
    psi = psi.astype(np.complex64).astype(np.complex128)
    wg, wu = np.array([0.05, 0.6, 1.0]), np.array([0.0, 0.3, 0.45])
    k2 = sum((2 * np.pi * np.fft.fftfreq(n, h).reshape([-1 if i == a else 1 for i in range(3)])) ** 2
             for a, h in enumerate(d))
    w = np.maximum(wg, 0.1)[:, None, None, None, None]
    den = w * (e0 + h2ma * k2) + 0.5 * np.maximum(wu, 0.1)[:, None, None, None, None] * vmax
    ref = np.fft.ifftn(np.fft.fftn(psi, axes=(2, 3, 4)) / den, axes=(2, 3, 4))
    x = torch.from_numpy(psi).cuda().to(dtype)
    twg, twu = torch.from_numpy(wg).cuda(), torch.from_numpy(wu).cuda()
    out = torch.empty_like(x)
    for dst in (out, x):
        call("hfb_laplace", g.ctx.handle, prec_of(x), ns, ptr(x), ptr(twg), ptr(twu), vmax, e0, h2ma, ptr(dst),
             stream_ptr())
        torch.cuda.synchronize()
        got = dst.cpu().numpy()
        assert np.linalg.norm(got - ref) <= tol * np.linalg.norm(ref)
