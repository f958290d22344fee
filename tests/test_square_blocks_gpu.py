"""The square transforms' inverse and clamp in the FP32 form
(k_square32_idct, k_square32_ar, k_square_ar_rows), bit for bit against the
FP32 oracle: from one block to several CTAs per SM, block counts that leave
the last warp or CTA part full, and dequantisation matrices at offsets that
rule out 16-byte loads."""

import dataclasses

import numpy as np
import pytest

from oracle import oraclepy
from pik_b200 import native, synthetic

pytestmark = pytest.mark.gpu


def check(frame):
    want = oraclepy.run(frame, precision=32, want=("idct", "ar", "linear"),
                        export_decisions=True)
    ctx = native.Context(0)
    ctx.begin(frame)
    ctx.set_ac()
    lin, _ = ctx.reconstruct()
    np.testing.assert_array_equal(ctx.stage("idct"), want["idct"])
    if frame.have_ar:
        # The clamp runs on filtered blocks only.
        assert (want["sigma"] >= 16).any()
        np.testing.assert_array_equal(ctx.stage("ar"), want["ar"])
    np.testing.assert_array_equal(lin, want["linear"])
    ctx.close()


@pytest.mark.parametrize("cls", ["DCT32X32", "DCT16X16", "DCT"])
@pytest.mark.parametrize("size", [(32, 32), (40, 72), (112, 48), (536, 520)])
@pytest.mark.parametrize("hf", [1, 0])
def test_square_blocks_bitexact(size, cls, hf):
    frame = synthetic.make_frame(*size, seed=size[0], shares={cls: 1.0,
                                                              "DCT": 1.0},
                                 qf_median=6.0)
    check(dataclasses.replace(frame, predict_hf=hf))


@pytest.mark.parametrize("shift", [1, 2, 4])
def test_unaligned_dequant_matrices(shift):
    frame = synthetic.make_frame(264, 136, seed=5, qf_median=6.0,
                                 shares={"DCT32X32": 0.4, "DCT16X16": 0.3,
                                         "DCT": 0.3})
    table = np.concatenate([np.ones(shift, np.float32), frame.dequant_table])
    check(dataclasses.replace(frame, dequant_table=table,
                              dequant_offsets=frame.dequant_offsets + shift))
