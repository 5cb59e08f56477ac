"""The radix-2 split transforms (mc_fwd_dif.cu, sides 2 N with a two-level N)
where nothing is cropped: their columns then run in place."""
import numpy as np
import pytest

from motioncorr1exp_b200 import api

pytestmark = pytest.mark.gpu

# FP32 transforms of n <= 8192: every output is a chain of at most ~20 operations
# and one direct sum of 53 terms, rounding errors of 2^-24 adding like a random
# walk (the bound the mixed-radix lengths are tested with)
RTOL = 2e-6


@pytest.mark.parametrize("n", [7420, 8192, 3710, 4096])
@pytest.mark.parametrize("batch", [1, 300])
def test_rows_in_place(gpu, n, batch):
    """Every row overwritten by its own transform (one row, then more than one
    a multiprocessor): as the numpy transform, and as apart from its input."""
    import torch
    rng = np.random.default_rng(n + batch)
    x = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(np.complex64)
    d = torch.from_numpy(x.view(np.float32)).cuda()
    apart = torch.full_like(d, float("nan"))
    api.fft1d(d.data_ptr(), apart.data_ptr(), n, batch, False)
    api.fft1d(d.data_ptr(), d.data_ptr(), n, batch, False)
    torch.cuda.synchronize()
    got = d.cpu().numpy().view(np.complex64)
    ref = np.fft.fft(x.astype(np.complex128), axis=1)
    assert np.linalg.norm(got - ref) <= RTOL * np.linalg.norm(ref)
    np.testing.assert_array_equal(got, apart.cpu().numpy().view(np.complex64))
