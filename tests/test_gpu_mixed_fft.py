"""The mixed-radix engine (mixed_fft.cuh) at the lengths where it can go wrong:
every register radix alone and fused with a neighbour, radix 53, primes as a
direct sum from a table (first stage), a second such prime, a prime beyond the
tables, the largest side, and batches that leave the last CTA partly empty.
Against numpy's FP64 transform: every output is a sum of n terms whose FP32
rounding errors (2^-24 each, at most ~20 operations deep or a direct sum of
up to 131 terms) add like a random walk, below 2e-6 of the result."""
import numpy as np
import pytest

from motioncorr1exp_b200 import api

pytestmark = pytest.mark.gpu

RTOL = 2e-6


@pytest.mark.parametrize("n", [1, 6, 9, 10, 12, 14, 15, 22, 26, 34, 38, 46, 58, 62, 74, 118, 122, 226, 254, 262, 289,
                               323, 520, 646, 1500, 2540, 4092, 4050, 8190, 9216])
@pytest.mark.parametrize("batch", [1, 37])
def test_mixed_radix_lengths(gpu, n, batch):
    import torch
    rng = np.random.default_rng(n + batch)
    x = (rng.standard_normal((batch, n)) + 1j * rng.standard_normal((batch, n))).astype(np.complex64)
    d_in = torch.from_numpy(x.view(np.float32)).cuda()
    for inv in (False, True):
        d_out = torch.full_like(d_in, float("nan"))
        api.fft1d(d_in.data_ptr(), d_out.data_ptr(), n, batch, inv)
        torch.cuda.synchronize()
        got = d_out.cpu().numpy().view(np.complex64).astype(np.complex128)
        x64 = x.astype(np.complex128)
        ref = np.fft.ifft(x64, axis=1) * n if inv else np.fft.fft(x64, axis=1)
        err = np.linalg.norm(got - ref) / np.linalg.norm(ref)
        assert err <= RTOL, (n, batch, inv, err)
