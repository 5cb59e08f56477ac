"""The row pass of two-level sides with dark and gain (k_fwd_rows2l_refs): two
spectrum sets with references of one and of both sets, the one-output form of
binned movies, a side whose last CTA has only half its rows (3710 = 4 x 927 + 2),
missing references, odd crop offsets.  Spectra against FP64."""
import numpy as np
import pytest

from motioncorr1exp_b200 import api

pytestmark = pytest.mark.gpu

SPEC_RTOL = 1e-5  # as the parity tests'
DTYPE = {0: np.int8, 1: np.int16, 2: np.float32, 6: np.uint16, api.MODE_U8: np.uint8, api.MODE_F16: np.float16}


@pytest.mark.parametrize("side, bin_, mode, which", [
    (256, 1.0, 6, ("dark", "norm")),
    (256, 2.0, 0, ("dark", "norm")),
    (512, 1.0, api.MODE_F16, ("dark", "dark2", "norm", "norm2")),
    (512, 2.0, 1, ("dark", "dark2", "norm", "norm2")),
    (1024, 1.0, 2, ("dark",)),
    (1024, 2.0, 2, ("norm",)),
    (2048, 1.0, 1, ("norm", "norm2")),
    (3710, 1.0, api.MODE_U8, ("dark", "dark2", "norm", "norm2")),
    (3710, 1.5, 6, ("dark", "norm")),
    (4096, 2.0, api.MODE_U8, ("dark", "dark2", "norm")),
    (512, 1.0, 6, ()),
])
def test_reference_rows(gpu, side, bin_, mode, which):
    import torch
    nz, nx, ny, ox, oy = 3, side + 11, side + 5, 7, 3
    rng = np.random.default_rng(side + mode)
    frames = rng.poisson(6.0, (nz, ny, nx)).astype(DTYPE[mode])
    refs = {k: (rng.random((ny, nx), dtype=np.float32) if "dark" in k else
                1 + 0.2 * rng.random((ny, nx), dtype=np.float32)) for k in which}
    p = api.verify_params(api.Params(crop_nsam=side, crop_offsetx=ox, crop_offsety=oy, bin=bin_, FrameDistOffset=0,
                                     CCPeakSearchDim=64), nz)
    with api.Plan(p, nx, ny, nz, mode) as pl:
        assert pl.info["nsam_unbin"] == side
        n = pl.nsam
        if not refs:  # references set and taken away again: two equal sets
            pl.set_refs(dark=np.ones((ny, nx), np.float32))
        pl.set_refs(**refs)
        pl.load_frames(frames)
        pl.forward()
        for f in range(nz):
            for s, tail in enumerate(("", "2")):
                x = torch.from_numpy(frames[f].astype(np.float64)).cuda()
                if "dark" + tail in refs:
                    x = x - torch.from_numpy(refs["dark" + tail]).cuda()
                if "norm" + tail in refs:
                    x = x * torch.from_numpy(refs["norm" + tail]).cuda()
                F = torch.fft.rfft2(x[oy:oy + side, ox:ox + side])
                want = torch.cat([F[:n // 2, :n // 2 + 1], F[side - n // 2:, :n // 2 + 1]])
                err = torch.linalg.vector_norm(torch.from_numpy(pl.spectrum(f, s)).cuda() - want, dim=0)
                err = (err / torch.linalg.vector_norm(want, dim=0)).cpu().numpy()
                assert np.all(err <= SPEC_RTOL), (f, s, np.nonzero(~(err <= SPEC_RTOL))[0][:8], err.max())
