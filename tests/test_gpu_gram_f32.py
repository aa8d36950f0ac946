"""Single-precision Gram on the tensor cores at the edges of its units: rows
of the stacked matrices in blocks of 128, columns in 16s up to 144, one or two
column parts, K slices of unequal length.  Against the FP64 product of the
same single-precision inputs, max error below 3e-6 of max |C| (three-term tf32
products, about 2^-21 each, summed with random signs); and every sum's order is
the same whichever matrices are computed together, so the bits are."""
import numpy as np
import pytest
import torch

from test_gpu_kernels import _gram_case, rel, T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,s0,ns", [(8, 0, 1), (8, 2, 15), (8, 0, 16), (16, 1, 17), (16, 0, 63), (16, 0, 64),
                                     (16, 2, 65), (24, 0, 128), (8, 0, 129), (16, 0, 144), (16, 3, 145), (8, 0, 160)])
def test_gram_units(n, s0, ns):
    from hfb._lib import call, ptr, stream_ptr, prec_of
    g, a, vp = _gram_case(n, s0, ns, 21)
    ta, vpt = [T(x, torch.complex64) for x in a], T(vp)

    def run(mask):
        out = torch.zeros((4, ns, ns), dtype=torch.complex128, device="cuda")
        call("hfb_gram", g.ctx.handle, prec_of(ta[0]), s0, ns, mask, ptr(ta[0]), ptr(ta[1]), ptr(ta[2]), ptr(vpt),
             0.5, ptr(out), stream_ptr())
        torch.cuda.synchronize()
        return out.cpu().numpy()

    every = run(15)
    sl = slice(s0, s0 + ns)
    refs = [0.5 * a[0][sl].conj() @ x.T for x in (a[0][sl], a[1][sl], a[2][sl], a[0][sl] * np.tile(vp, 2)[None])]
    for k in range(4):
        assert rel(every[k], refs[k]) < 3e-6, (k, rel(every[k], refs[k]))
    for mask in (3, 12, 1, 8):
        part = run(mask)
        for k in range(4):
            if mask >> k & 1:
                assert np.array_equal(part[k], every[k]), (mask, k)
