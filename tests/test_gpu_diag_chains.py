"""The matrix chains of the diagonalisation step (S^-1/2, eigen refinement,
construct_hfb_matrices) at the edges of their 16 x 16 blocks and of the
cluster sizes, against NumPy.

States are an orthonormal set plus a 5 % perturbation (as a gradient step
leaves them), h and v_pair random real fields, so that every matrix is a
well-conditioned contraction of K = 2 8^3 terms: the products and the
Newton-Schulz iteration are rounding-level, n K eps times small factors, and
1e-11 relative is two orders above that for n <= 166."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

N, D = 8, 0.9


def _states(rng, ns):
    q, _ = np.linalg.qr(rng.standard_normal((2 * N ** 3, ns)) + 1j * rng.standard_normal((2 * N ** 3, ns)))
    e = rng.standard_normal(q.shape) + 1j * rng.standard_normal(q.shape)
    return ((q + 0.05 * e / np.linalg.norm(e, axis=0)) / D ** 1.5).T.copy()


def _run(npsi, diagonalize, tbcs, ipair, seed=3):
    import hfb
    from hfb import config
    case = config.case_dict("O16", grid=dict(nx=N, ny=N, nz=N, dx=D, dy=D, dz=D),
                            levels=dict(nneut=max(1, npsi[0] // 2), nprot=max(1, npsi[1] // 2), npsi=list(npsi)))
    case["force"].update(ipair=ipair, tbcs=tbcs)
    st = config.setup(case)
    rng = np.random.default_rng(seed)
    lv, s = st["levels"], st["static"]
    psi = np.concatenate([_states(rng, n) for n in npsi])
    fields = rng.uniform(-50.0, 20.0, (3, 2, N ** 3))
    iso = np.repeat([0, 1], npsi)
    two = lambda f: np.concatenate([f[iso], f[iso]], axis=1)  # noqa: E731
    ham, hmf, vpsi = (two(f) * psi for f in fields)
    w, uv, pw = (rng.uniform(0.1, 1.0, sum(npsi)) for _ in range(3))
    put = lambda t, a: t.copy_(torch.from_numpy(np.ascontiguousarray(a)).reshape(t.shape))  # noqa: E731
    for t, a in ((lv.psi, psi), (lv.hampsi, ham), (lv.hmfpsi, hmf), (lv.wocc, w), (lv.wguv, uv), (lv.pairwg, pw)):
        put(t, a)
    lv._v_pair = torch.from_numpy(fields[2].reshape(2, N, N, N).copy()).cuda()
    hfb.static.diagstep(st["energies"], st["forces"], st["grids"], lv, s, diagonalize, True)
    st["grids"].ctx.check("diagstep")
    return st, psi, ham, hmf, vpsi, w, uv, pw


def _close(got, ref, tol=1e-11):
    assert np.max(np.abs(got - ref)) <= tol * np.max(np.abs(ref))


@pytest.mark.parametrize("npsi", [(1, 2), (15, 16), (17, 33), (49, 64), (65, 97), (166, 140)])
@pytest.mark.parametrize("diagonalize,tbcs,ipair", [(False, False, 0), (False, False, 5), (True, True, 5)])
def test_diagstep_chains(npsi, diagonalize, tbcs, ipair):
    st, psi, ham, hmf, vpsi, w, uv, pw = _run(npsi, diagonalize, tbcs, ipair)
    lv, s, dv = st["levels"], st["static"], D ** 3
    get = lambda t: t.cpu().numpy()  # noqa: E731
    new, lag = get(lv.psi).reshape(psi.shape), get(lv.lagrange).reshape(psi.shape)
    for iq in range(2):
        b = slice(0, npsi[0]) if iq == 0 else slice(npsi[0], sum(npsi))
        n = npsi[iq]
        p = psi[b]
        gram = lambda x: dv * p.conj() @ x[b].T  # noqa: E731
        ov = gram(psi)
        _close(get(lv.sp_norm)[b], ov.diagonal().real)
        val, vec = np.linalg.eigh(ov)
        root = (vec / np.sqrt(val)) @ vec.conj().T
        if diagonalize:
            # U = S^-1/2 V: V is unitary and diagonalises lambda, values ascending
            u = np.linalg.solve(ov, dv * p.conj() @ new[b].T)
            v = np.linalg.solve(root, u)
            lam = gram(ham)
            dg = v.conj().T @ lam @ v
            assert np.max(np.abs(v.conj().T @ v - np.eye(n))) < 1e-11
            assert np.max(np.abs(dg - np.diag(dg.diagonal()))) < 1e-9 * np.abs(lam).max()
            assert np.all(np.diff(dg.diagonal().real) > -1e-9 * np.abs(lam).max())
        else:
            u = root
        _close(new[b], (p.T @ u).T)
        h = u.conj().T @ gram(hmf) @ u
        g = u.conj().T @ gram(vpsi) @ u if ipair else np.zeros_like(h)
        _close(get(s.hmatrix)[iq, :n, :n], h)
        _close(get(lv.sp_energy)[b], h.diagonal().real)
        if ipair:
            _close(get(lv.deltaf)[b], g.diagonal().real * pw[b])
        if tbcs:
            g = np.diag(g.diagonal())
        if ipair:
            _close(get(s.gapmatrix)[iq, :n, :n], g)
        lam = w[b][None, :] * h - (uv * pw)[b][None, :] * g
        sym, asym = 0.5 * (lam + lam.conj().T), 0.5 * (lam - lam.conj().T)
        _close(get(s.lambda_save)[iq, :n, :n], sym)
        assert np.max(np.abs(get(s.symcond)[iq, :n, :n] - asym)) <= 1e-11 * np.abs(lam).max()
        fl = get(st["energies"].efluct_dev)
        _close(np.array([fl[iq], fl[2 + iq]]), np.array([np.abs(asym).max(), np.sqrt((np.abs(asym) ** 2).sum()) / n]),
               1e-10 if n > 1 else np.inf)
        _close(lag[b], (new[b].T @ sym).T)


@pytest.mark.parametrize("n", [1, 15, 16, 17, 33, 61])
def test_refinement_block_edges(n):
    """hfb_eigh_near_diagonal on one and on two matrices (one cluster each)."""
    import hfb
    from hfb._lib import call, ptr, stream_ptr
    g = hfb.grids.init_grids(hfb.params.init_params(), nx=8, ny=8, nz=8, dx=1.0, dy=1.0, dz=1.0)
    rng = np.random.default_rng(n)
    for nb in (1, 2):
        e = rng.standard_normal((nb, n, n)) + 1j * rng.standard_normal((nb, n, n))
        a = np.stack([np.diag(np.sort(rng.uniform(-60.0, 40.0, n))) for _ in range(nb)])
        a = a + 1e-3 * (e + e.conj().transpose(0, 2, 1)) / 2
        w = torch.zeros((nb, n), dtype=torch.float64, device="cuda")
        v = torch.zeros((nb, n, n), dtype=torch.complex128, device="cuda")
        call("hfb_eigh_near_diagonal", g.ctx.handle, nb, n, n, ptr(torch.from_numpy(a).cuda()), ptr(w), ptr(v),
             stream_ptr())
        wv, vv = w.cpu().numpy(), v.cpu().numpy()
        for k in range(nb):
            amax = np.abs(a[k]).max()
            assert np.max(np.abs(wv[k] - np.linalg.eigvalsh(a[k]))) < 1e-12 * amax * n
            assert np.max(np.abs(a[k] @ vv[k] - vv[k] * wv[k][None, :])) < 1e-11 * amax
            assert np.max(np.abs(vv[k].conj().T @ vv[k] - np.eye(n))) < 1e-12
