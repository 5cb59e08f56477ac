"""mc_plan_run_host on movies of several upload chunks (48 MiB each at least):
the pairs of a chunk's frames run when it has arrived, in another order than
the list, so windows, peaks, shifts and image must equal the run from device
memory bit for bit -- a last chunk smaller than the others, chunks of two frames
uploaded from both ends, of one frame, a compiled pair split and a generic one, references with two
spectrum sets, binning, and a plan re-targeted to another frame range."""
import numpy as np
import pytest

from motioncorr1exp_b200 import api, synth

pytestmark = pytest.mark.gpu


def _results(pl):
    return {"boxes": pl.boxes(), "shifts": pl.frame_shifts(), **pl.pair_results(), **pl.ki(), "means": pl.frame_means()}


def _same(a, b):
    for k in a:
        np.testing.assert_array_equal(a[k], b[k], err_msg=k)


@pytest.mark.parametrize("nx, ny, nz, kw, refs", [
    (1400, 1300, 13, dict(), False),                   # seven frames a chunk, the last holds six
    (2100, 2048, 5, dict(FrameDistOffset=0), False),   # three frames a chunk, compiled split 2048
    (2600, 2500, 6, dict(bin=2.0), False),             # two frames a chunk, binned
    (3700, 3600, 4, dict(FrameDistOffset=1), False),   # one frame a chunk
    (1400, 1300, 9, dict(FrameDistOffset=2), True),    # two spectrum sets
])
def test_chunked_host_run_equals_device_run(gpu, nx, ny, nz, kw, refs):
    base = synth.make_movie(700, 650, nz, mean=3.0, seed=nz, dtype="f32", speed=0.6, rw_sigma=0.4).frames
    frames = np.ascontiguousarray(np.tile(base, (1, 6, 6))[:, :ny, :nx])
    rng = np.random.default_rng(nz)
    p = api.verify_params(api.Params(CCPeakSearchDim=64, nEnd=nz - 1, **kw), nz)
    with api.Plan(p, nx, ny, nz, 2) as pl:
        assert pl.info["nx"] * pl.info["ny"] * 4 * nz > 48 << 20
        if refs:
            pl.set_refs(dark=rng.random((ny, nx), dtype=np.float32), norm=1 + 0.1 * rng.random((ny, nx), dtype=np.float32))
        img_h = pl.run_host(frames)
        host = _results(pl)
        pl.load_frames(frames)
        img_d = pl.run()
        _same(host, _results(pl))
        np.testing.assert_array_equal(img_h, img_d)
        # another range of the same plan: the chunk order follows
        q = api.verify_params(api.Params(CCPeakSearchDim=64, nStart=1, nEnd=nz - 1, **kw), nz)
        pl.reframe(q, nz)
        img_h = pl.run_host(frames[1:])
        host = _results(pl)
        pl.load_frames(frames[1:])
        img_d = pl.run()
        _same(host, _results(pl))
        np.testing.assert_array_equal(img_h, img_d)
