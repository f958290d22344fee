"""The LF prediction's 32-cell tiles (k_lf_tile<LfTile32>), which frames of 99
or more 512x512 groups take on 148 SMs: long thin frames, whose groups are
narrower than a tile, one tile and a part, and end in part groups, bit for bit
against the FP32 oracle. Half as many groups take the 16-cell tiles."""

import numpy as np
import pytest

from oracle import oraclepy
from pik_b200 import native, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(24, 50700), (50696, 40), (300, 50712),
                                  (40, 25000)])
def test_lf_large_frames_bitexact(size):
    frame = synthetic.make_frame(*size, seed=sum(size), have_ar=False,
                                 shares={"DCT32X32": 0.3, "DCT16X16": 0.3,
                                         "DCT": 0.2, "DCT2X2": 0.2})
    want = oraclepy.run(frame, precision=32, want=("dc", "idct"))
    ctx = native.Context(0)
    ctx.begin(frame)
    ctx.set_ac()
    ctx.reconstruct()
    np.testing.assert_array_equal(ctx.stage("dc"), want["dc"])
    np.testing.assert_array_equal(ctx.stage("idct"), want["idct"])
    ctx.close()
