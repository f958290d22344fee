"""The tensor-core transforms and clamp at block counts that leave a batch
(eight 16x16 or four 32x32 blocks) part full, with one and several batches
per class, and with dequantisation matrices at offsets that rule out 16-byte
loads: against FP64 within the bounds of tests/test_split_bf16.py (2e-5 on
shared decisions), and the same bytes when the frame is repeated."""

import dataclasses

import numpy as np
import pytest

from pik_b200 import native, synthetic
from tests.test_split_bf16 import check_against_fp64

pytestmark = pytest.mark.gpu


def frame_of(size, cls, hf, shift=0):
    f = synthetic.make_frame(*size, seed=size[0] + 1,
                             shares={cls: 1.0, "DCT": 1.0}, qf_median=6.0)
    table = np.concatenate([np.ones(shift, np.float32), f.dequant_table])
    return dataclasses.replace(f, predict_hf=hf, dequant_table=table,
                               dequant_offsets=f.dequant_offsets + shift)


@pytest.mark.parametrize("hf", [1, 0])
@pytest.mark.parametrize("size,cls", [
    ((16, 16), "DCT16X16"), ((48, 48), "DCT16X16"), ((136, 72), "DCT16X16"),
    ((32, 32), "DCT32X32"), ((96, 64), "DCT32X32"), ((200, 136), "DCT32X32")])
def test_part_full_batches(size, cls, hf):
    for form in ("split_bf16", "split_bf16x3"):
        check_against_fp64(frame_of(size, cls, hf), form)


@pytest.mark.parametrize("cls", ["DCT16X16", "DCT32X32"])
def test_unaligned_dequant_matrices(cls):
    check_against_fp64(frame_of((104, 72), cls, 1, shift=1), "split_bf16")


def test_repeated_frames_are_identical():
    ctx = native.Context(0, form="split_bf16")
    f = synthetic.make_frame(520, 264, seed=2, qf_median=6.0)
    ctx.begin(f)
    ctx.set_ac()
    first, _ = ctx.reconstruct()
    for _ in range(4):
        again, _ = ctx.reconstruct()
        np.testing.assert_array_equal(again, first)
    ctx.close()
