"""The device drift solve (k_solve_smem) against the host's (lsq.cpp, through
mc_plan_solve) on the same pair shifts: one step, step counts on both sides of
a warp and of the sixteen-column tiles, a threshold that every row passes (one
solve) and thresholds that drop rows (ranked, solved again).  Both run the
FP64 normal equations and a Cholesky factorisation of a matrix whose condition
grows with the square of the frame count (below 1e5 here), on shifts of a few
pixels: equal to 1e-9 px."""
import numpy as np
import pytest

from motioncorr1exp_b200 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz, fod", [(2, 0), (3, 0), (17, 3), (18, 4), (33, 5), (34, 2), (70, 4)])
@pytest.mark.parametrize("kith", [1e9, 0.2])
def test_device_solve_matches_host(gpu, nz, fod, kith):
    mv = synth.make_movie(100, 96, nz, mean=2.0, seed=nz, dtype="u8", speed=0.2, rw_sigma=0.2)
    p = api.Params(CCPeakSearchDim=32, FrameDistOffset=fod, kiThresh=kith, nEnd=nz - 1, nEndSum=nz - 1)
    with api.Plan(p, 100, 96, nz, 0) as pl:
        pl.load_frames(mv.frames)
        pl.run()
        dev, ki_d, shift_d = pl.frame_shifts(), pl.ki(), pl.pair_results()["shift"]
        pl.forward()
        pl.pairs()
        pl.solve()
        pl.iterate()
        host, ki_h, shift_h = pl.frame_shifts(), pl.ki(), pl.pair_results()["shift"]
    np.testing.assert_array_equal(shift_d, shift_h)
    np.testing.assert_array_equal(ki_d["kept"], ki_h["kept"])
    assert (len(ki_d["kept"]) == len(shift_d)) == (np.all(ki_d["ki1"] < kith) or nz <= 3)
    for k in ("ki1", "ki2"):
        np.testing.assert_allclose(ki_d[k], ki_h[k], rtol=0, atol=1e-9)
    np.testing.assert_allclose(dev, host, rtol=0, atol=1e-9)
