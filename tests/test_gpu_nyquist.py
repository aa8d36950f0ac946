"""The Nyquist-line terms of the reverse mode at every grid size (rows of up to 32
and of more points, odd shares of the states) against NumPy.

Sums of n signed terms in double, then at most three additions: 1e-13 relative
to the largest element in double; in single precision y is rounded at most
three times, 2^-23 relative to the largest element each."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

D = (0.9, 1.0, 1.1)


def _alt(n):
    return 1.0 - 2.0 * (np.arange(n) % 2)


@pytest.mark.parametrize("n,nst,nneut", [(n, *s) for n in (8, 16, 24, 32, 40, 48) for s in ((1, 1), (19, 17), (5, 0))]
                         + [(8, 150, 131)])   # more states than runs
@pytest.mark.parametrize("dtype", [torch.complex128, torch.complex64])
def test_nyquist_terms(n, nst, nneut, dtype):
    import hfb
    from hfb._lib import call, prec_of, ptr, stream_ptr
    g = hfb.grids.init_grids(hfb.params.init_params(), nx=n, ny=n, nz=n, dx=D[0], dy=D[1], dz=D[2])
    rng = np.random.default_rng(n + nst)
    put = lambda a, t: torch.from_numpy(np.ascontiguousarray(a)).cuda().to(t)  # noqa: E731
    c = lambda: rng.standard_normal((nst, 2, n, n, n)) + 1j * rng.standard_normal((nst, 2, n, n, n))  # noqa: E731
    x, y = put(c(), dtype), put(c(), dtype)
    b, w = rng.standard_normal((2, n, n, n)), rng.uniform(0.1, 1.0, nst)
    bt, wt = put(b, torch.float64), put(w, torch.float64)
    xs, ys = x.cpu().numpy().astype(complex), y.cpu().numpy().astype(complex)
    iso = (np.arange(nst) >= nneut).astype(int)
    pair, apply = b.copy(), ys.copy()
    for ax in range(3):
        e = _alt(n).reshape([n if k == ax else 1 for k in range(3)])
        k = (np.pi / D[ax]) ** 2
        xn, yn = ((e * v).sum(axis=ax + 2, keepdims=True) for v in (xs, ys))
        d = w[:, None, None, None] * (xn.conj() * yn).real.sum(axis=1)
        for iq in range(2):
            pair[iq] += k / n ** 2 * d[iso == iq].sum(axis=0)
        mean = b.mean(axis=ax + 1, keepdims=True)[iso][:, None]
        apply -= w[:, None, None, None, None] * (k / n) * mean * e * xn
    call("hfb_nyquist_pair", g.ctx.handle, prec_of(x), nst, nneut, ptr(x), ptr(y), ptr(wt), ptr(bt), stream_ptr())
    got = bt.cpu().numpy()
    assert np.max(np.abs(got - pair)) <= 1e-13 * np.max(np.abs(pair))
    bt = put(b, torch.float64)
    call("hfb_nyquist_apply", g.ctx.handle, prec_of(x), nst, nneut, ptr(bt), ptr(wt), ptr(x), ptr(y), stream_ptr())
    got = y.cpu().numpy()
    tol = 1e-13 if dtype == torch.complex128 else 3 * 2.0 ** -23
    assert np.max(np.abs(got - apply)) <= tol * np.max(np.abs(apply))
