"""The LF prediction's tiles and per-size lanes (k_lf_tile): frames whose
edges fall on, before and after the 16-cell tiles and the 64-cell groups,
with the 32x32 blocks' eight lanes, the 16x16 blocks' four and the one-lane
classes each alone and together, bit for bit against the FP32 oracle."""

import dataclasses

import numpy as np
import pytest

from oracle import oraclepy
from pik_b200 import native, synthetic

pytestmark = pytest.mark.gpu

MIXES = {
    "all32": {"DCT32X32": 1.0, "DCT": 1.0},
    "all16": {"DCT16X16": 1.0, "IDENTITY": 1.0},
    "mixed": {"DCT32X32": 0.3, "DCT16X16": 0.3, "DCT": 0.2, "DCT2X2": 0.2},
}


@pytest.mark.parametrize("mix", list(MIXES))
@pytest.mark.parametrize("size", [(32, 32), (128, 136), (120, 264),
                                  (513, 160), (544, 40)])
@pytest.mark.parametrize("lf,hf", [(1, 1), (1, 0), (0, 1)])
def test_lf_prediction_bitexact(size, mix, lf, hf):
    # The shares are of the free cells: the multi-block transforms take what
    # they can, the last type the rest.
    frame = dataclasses.replace(
        synthetic.make_frame(*size, seed=sum(size), shares=MIXES[mix]),
        predict_lf=lf, predict_hf=hf)
    want = oraclepy.run(frame, precision=32, want=("dc", "idct"))
    ctx = native.Context(0)
    ctx.begin(frame)
    ctx.set_ac()
    ctx.reconstruct()
    np.testing.assert_array_equal(ctx.stage("dc"), want["dc"])
    np.testing.assert_array_equal(ctx.stage("idct"), want["idct"])
    ctx.close()
