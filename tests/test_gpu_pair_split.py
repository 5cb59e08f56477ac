"""The pair stage of sizes without a compiled split (k_pair_cols_pruned,
k_pair_rows) where it can go wrong: one pair, pair counts that leave a CTA's
last group of units partly empty, register codelets with one to many units a
CTA, the mixed-radix engine with several units, with one and with the smallest
Q, the smallest, odd and largest boxes, and tile heights of 16 and 32 rows.
CC windows against the FP64 oracle's (cc_map + cc_box) of the plan's own
spectra, relative L2 <= 1e-5: products, weights and sums of at most ~4100 FP32
terms (2^-24 each) grow like their square root, below 4e-6."""
import numpy as np
import pytest

from motioncorr1exp_b200 import api, synth
from oracle import mc_oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n, box, nz, fod", [
    (16, 16, 2, 0),       # P = 1
    (256, 64, 9, 2),      # P = 4: every pair in one CTA
    (520, 95, 12, 3),     # P = 13, odd box
    (1500, 96, 6, 1),     # P = 25, five units a CTA
    (290, 256, 5, 1),     # the largest box
    (254, 64, 20, 6),     # 2 x 127: engine, sixteen units
    (998, 96, 4, 0),      # 2 x 499: Q = 2
    (1298, 128, 5, 1),    # 2 x 11 x 59
    (4092, 96, 3, 0),     # 4 x 3 x 11 x 31: one unit
])
def test_windows_match_oracle(gpu, n, box, nz, fod):
    mv = synth.make_movie(n + 3, n, nz, mean=2.0, seed=n + box, dtype="u8", speed=0.5, rw_sigma=0.4)
    p = api.Params(CCPeakSearchDim=box, FrameDistOffset=fod, nEnd=nz - 1, nEndSum=nz - 1)
    with api.Plan(p, n + 3, n, nz, 0) as pl:
        pl.load_frames(mv.frames)
        pl.forward()
        pl.pairs()
        boxes, pairs = pl.boxes(), pl.pair_results()["pairs"]
        F = [pl.spectrum(f).astype(np.complex128) for f in range(nz)]
    mask = O.bfactor_mask(n, p.bfactor)
    for r in sorted({0, len(pairs) // 2, len(pairs) - 1}):
        i, j = pairs[r]
        ref = O.cc_box(O.cc_map(F[i], F[j], mask, n), n, box)
        err = np.linalg.norm(boxes[r] - ref) / np.linalg.norm(ref)
        assert err <= 1e-5, (n, box, r, err)
