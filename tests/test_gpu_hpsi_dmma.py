"""FP64 hpsi on the FP64 tensor cores against the oracle, where the plain and
the persistent launches differ: one state of an isospin, half lines that are not a
multiple of the 8-point tile (n = 8, 24, 40), fewer planes than places, several
planes a CTA, and enough of them for the table of line means (40^3 from 30
states on).  1e-11 as for the FFT kernels: sums of n terms in FP64."""
import pytest
import torch

from test_gpu_kernels import _check_hpsi_batched

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,ns", [(8, 2), (8, 3), (16, 2), (24, 2), (32, 2), (32, 11), (40, 2), (40, 30), (48, 4)])
def test_hpsi_fp64_tensor_cores(n, ns):
    _check_hpsi_batched(n, torch.complex128, ns)
