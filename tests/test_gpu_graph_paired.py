"""Captured double-precision iterations that diagonalise lambda (pairing on): the
H, G Gram launch waits for the refinement's launch completion event, which a
capture turns into an edge of its own kind, alone and copied into the composite
of several instances.  The captured launches are those of the ordinary driver,
every sum in a fixed order, so the energies agree to rounding (1e-9 MeV)."""
import copy

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _case(n, npsi):
    from hfb import config
    return config.case_dict("Cr48", grid=dict(nx=n, ny=n, nz=n, dx=1.0, dy=1.0, dz=1.0),
                            levels=dict(nneut=12, nprot=12, npsi=npsi))


def _plain(case, iters):
    from hfb import config, static
    st = config.setup(copy.deepcopy(case))
    S = {k: st[k] for k in static._STATE_KEYS}
    static.prepare(**S)
    E = []
    for i in range(1, iters + 1):
        static.iterate(i, **S)
        E.append(st["energies"].ehf)
    assert st["static"].tdiag and st["forces"].ipair != 0
    return np.array(E)


@pytest.mark.parametrize("cases", [[(16, [20, 18])], [(16, [20, 18]), (24, [16, 20])]])
@pytest.mark.parametrize("keep", [False, True])
def test_captured_iterations_with_pairing(cases, keep, monkeypatch):
    """Each run's own graph, and (captures that keep their graph) the composite."""
    from hfb import config, graph
    if keep:
        real = torch.cuda.CUDAGraph
        monkeypatch.setattr(torch.cuda, "CUDAGraph", lambda: real(keep_graph=True))
    cases = [_case(*c) for c in cases]
    refs = [_plain(c, 42) for c in cases]
    runs = [graph.GraphRun(config.setup(copy.deepcopy(c))) for c in cases]
    for r in runs:
        r.start()
        r.plain(22)
    bg = graph.BatchGraph(runs, block=10).capture()
    assert (bg.comp is not None) == keep
    for _ in range(2):
        bg.replay()
    bg.release()
    for r, ref in zip(runs, refs):
        assert len(r.E) == 42
        assert np.max(np.abs(np.array(r.E) - ref)) < 1e-9
