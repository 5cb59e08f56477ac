"""k_peak's integer and sub-pixel peaks (FindShift, cufunc.cu:396-497) against
the FP64 oracle on the plan's own CC windows, for pair counts on both sides of
the line where a pair's cluster goes from four CTAs to two, the smallest, an
odd and the largest box, and the noise-peak exclusion.  Both sides search the
same 512 x 512 grid in FP64 from the same float windows, so shifts and integer
peaks are equal; cc differs by its rounding to float (2^-24 relative)."""
import numpy as np
import pytest

from motioncorr1exp_b200 import api, synth
from oracle import mc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nz, fod, box, nps", [
    (2, 0, 16, 0),      # one pair, the smallest box
    (20, 2, 95, 3),     # 78 pairs, odd box, excluded centre
    (18, 3, 64, 0),     # 78 pairs
    (16, 3, 96, 1),     # 66 pairs: clusters of four
    (6, 1, 256, 5),     # the largest box
])
def test_peaks_match_oracle_on_the_same_windows(gpu, nz, fod, box, nps):
    n = 300 if box <= 128 else 260
    mv = synth.make_movie(n + 4, n, nz, mean=2.0, seed=nz + box, dtype="u8", speed=0.9, rw_sigma=0.6)
    p = api.Params(CCPeakSearchDim=box, FrameDistOffset=fod, NoisePeakSize=nps, nEnd=nz - 1, nEndSum=nz - 1)
    with api.Plan(p, n + 4, n, nz, 0) as pl:
        pl.load_frames(mv.frames)
        pl.forward()
        pl.pairs()
        boxes, got = pl.boxes(), pl.pair_results()
        assert pl.nsam == n
    for r in range(len(boxes)):
        sx, sy, cc, ix, iy = O.find_shift(boxes[r].astype(np.float64), n, nps)
        assert tuple(got["peak"][r]) == (ix, iy)
        assert tuple(got["shift"][r]) == (np.float32(sx), np.float32(sy))
        assert abs(got["cc"][r] - cc) <= 1e-6 * abs(cc)
