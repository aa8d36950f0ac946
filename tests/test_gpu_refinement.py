"""That nearly diagonal matrices are solved by the refinement and not, unnoticed,
by the Jacobi solver behind it.

The perturbations have a Frobenius norm of about 1e-5 n, so the pairs that a
step leaves coupled (closer than twice that) are the multiplets alone; the
others, 0.3 and more apart, converge quadratically: three steps of the six.  The
tolerances are those of the other tests of these solvers."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _solve(a):
    import hfb
    from hfb._lib import call, ptr, stream_ptr
    g = hfb.grids.init_grids(hfb.params.init_params(), nx=8, ny=8, nz=8, dx=1.0, dy=1.0, dz=1.0)
    nb, n = a.shape[:2]
    w = torch.zeros((nb, n), dtype=torch.float64, device="cuda")
    v = torch.zeros((nb, n, n), dtype=torch.complex128, device="cuda")
    jacobi = torch.full((nb,), -1, dtype=torch.int32, device="cuda")
    call("hfb_eigh_near_diagonal_info", g.ctx.handle, nb, n, n, ptr(torch.from_numpy(a).cuda()), ptr(w), ptr(v),
         ptr(jacobi), stream_ptr())
    wv, vv = w.cpu().numpy(), v.cpu().numpy()
    for k in range(nb):
        amax = np.abs(a[k]).max()
        assert np.max(np.abs(wv[k] - np.linalg.eigvalsh(a[k]))) < 1e-12 * amax * n
        assert np.max(np.abs(a[k] @ vv[k] - vv[k] * wv[k][None, :])) < 1e-11 * amax
        assert np.max(np.abs(vv[k].conj().T @ vv[k] - np.eye(n))) < 1e-12
    return jacobi.cpu().tolist()


def _hermitian(rng, n):
    e = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    return (e + e.conj().T) / 2


def _near(rng, n, multiplet):
    levels = np.sort(rng.permutation(200)[:n // multiplet + 1] * 0.5 + rng.uniform(0.0, 0.2, n // multiplet + 1))
    return np.diag(np.repeat(levels, multiplet)[:n] - 60.0) + 1e-5 * _hermitian(rng, n)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 61, 80, 81, 97, 140])
@pytest.mark.parametrize("multiplet", [1, 2, 8])
def test_nearly_diagonal_matrices_are_refined(n, multiplet):
    rng = np.random.default_rng(100 * n + multiplet)
    for nb in (1, 2, 3):
        assert _solve(np.stack([_near(rng, n, multiplet) for _ in range(nb)])) == [0] * nb


@pytest.mark.parametrize("n", [17, 64, 97])
def test_other_matrices_go_to_the_jacobi_solver(n):
    """Far from diagonal, all pairs are coupled: one cluster of more than 16
    members.  Both matrices of a pair take the same way."""
    rng = np.random.default_rng(n)
    assert _solve(np.stack([_hermitian(rng, n), _near(rng, n, 1)])) == [1, 1]
    assert _solve(np.stack([_near(rng, n, 17), _near(rng, n, 1), _near(rng, n, 1)])) == [1, 1, 0]


def test_asymmetry_of_a_single_state():
    """A block of one state has a real lambda: no antisymmetric part."""
    from test_gpu_diag_chains import _run
    st = _run((1, 2), False, False, 5)[0]
    fl = st["energies"].efluct_dev.cpu().numpy()
    lam = st["static"].lambda_save[0, 0, 0].abs().item()
    assert lam > 0 and abs(fl[0]) <= 1e-11 * lam and abs(fl[2]) <= 1e-11 * lam
