"""Whole sides of 7420 and 8192 (the radix-2 split transforms, mc_fwd_dif.cu)
that are not binned: every column of the half spectrum is kept, the one at
kx = n/2 among them, and the column pass runs in place."""
import numpy as np
import pytest

from motioncorr1exp_b200 import api

pytestmark = pytest.mark.gpu

SPEC_RTOL = 1e-5  # as the parity tests'


def _movie(n, nx, track, mean):
    """Frames (u8 counts) of a smooth random rate moving by whole pixels."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    pad, m = 8, (n + 16) // 10 + 2
    field = torch.randn((1, 1, m, m), generator=g, device="cuda")
    rate = torch.nn.functional.interpolate(field, size=(m * 10, m * 10), mode="bilinear")[0, 0]
    rate = mean * (1 + 0.5 * rate).clamp_(min=0.0)
    frames = []
    for dx, dy in track:
        r = rate[pad - dy:pad - dy + n, pad - dx:pad - dx + nx]
        frames.append(torch.poisson(r.contiguous(), generator=g).clamp_(max=255).to(torch.uint8).cpu().numpy())
    return np.stack(frames)


@pytest.mark.parametrize("n", [7420, 8192])
@pytest.mark.parametrize("refs", [False, True])
def test_unbinned_radix2_split(gpu, n, refs):
    import torch
    nx, track = n + 3, [(0, 0), (2, -1), (3, 1), (1, 3)]
    frames = _movie(n, nx, track, 8.0)
    p = api.verify_params(api.Params(FrameDistOffset=1), len(track))
    rng = np.random.default_rng(n)
    with api.Plan(p, nx, n, len(track), api.MODE_U8) as pl:
        assert (pl.nsam, pl.info["nsam_unbin"]) == (n, n)
        dark = gain = None
        if refs:
            dark = rng.random((n, nx), dtype=np.float32)
            gain = 1 + 0.1 * rng.random((n, nx), dtype=np.float32)
            pl.set_refs(dark=dark, norm=gain)
        pl.load_frames(frames)
        pl.forward()
        for f in (0, len(track) - 1):
            for s in range(2 if refs else 1):
                x = torch.from_numpy(frames[f]).cuda().double()
                if refs and s == 0:
                    x = (x - torch.from_numpy(dark).cuda().double()) * torch.from_numpy(gain).cuda().double()
                want = torch.fft.rfft2(x[:, :n])
                err = torch.linalg.vector_norm(torch.from_numpy(pl.spectrum(f, s)).cuda() - want, dim=0)
                err = (err / torch.linalg.vector_norm(want, dim=0)).cpu().numpy()
                assert np.all(err <= SPEC_RTOL), (f, s, np.nonzero(~(err <= SPEC_RTOL)), err.max())
                del x, want
        image = pl.run()
        assert np.isfinite(image).all()
        # whole-pixel drift with many counts: each pair's peak is exact to the 1/32-px grid
        assert np.abs(pl.frame_shifts() + np.array(track)).max() <= 0.05
