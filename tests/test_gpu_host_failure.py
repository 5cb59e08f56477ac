"""mc_plan_run_host when its upload cannot be queued: the call reports the error,
no frame counts as loaded afterwards, and the plan works on.  The failure is the
host's: the plan's stream is in a stream capture, in which the call may not wait
for it, and nothing of the capture ever runs."""
import ctypes as C

import numpy as np
import pytest

from motioncorr1exp_b200 import _lib, api, synth

pytestmark = pytest.mark.gpu


def test_failed_upload_leaves_no_frame_loaded(gpu):
    import torch
    torch.cuda.init()
    rt = C.CDLL("libcudart.so.12")  # the runtime libmc uses
    nz, ny, nx = 13, 1300, 1400
    base = synth.make_movie(700, 650, nz, mean=3.0, seed=5, dtype="f32", speed=0.6, rw_sigma=0.4).frames
    frames = np.ascontiguousarray(np.tile(base, (1, 2, 2))[:, :ny, :nx])
    p = api.verify_params(api.Params(CCPeakSearchDim=64), nz)
    with api.Plan(p, nx, ny, nz, 2) as pl:
        frames = np.ascontiguousarray(frames[pl.info["nstart"]: pl.info["nend"] + 1])
        assert frames.nbytes > 48 << 20  # several upload chunks
        graph = C.c_void_p()
        assert rt.cudaStreamBeginCapture(C.c_void_p(pl.stream), 2) == 0  # relaxed
        try:
            with pytest.raises(_lib.McError) as e:
                pl.run_host(frames)
            assert e.value.code == -2
        finally:
            rt.cudaStreamEndCapture(C.c_void_p(pl.stream), C.byref(graph))
            rt.cudaGetLastError()
        for stage in (pl.forward, pl.run):
            with pytest.raises(_lib.McError, match="not loaded"):
                stage()
        image = pl.run_host(frames)
        shifts = pl.frame_shifts()
        pl.load_frames(frames)
        np.testing.assert_array_equal(image, pl.run())
        np.testing.assert_array_equal(shifts, pl.frame_shifts())
