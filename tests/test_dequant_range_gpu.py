"""AC dequantisation over the whole int16 range, bit for bit against the FP32
oracle through the inverse transform: magnitudes on both sides of the table of
biased values (0 .. 63), the largest ones of both signs, alone in a thread's
four coefficients and beside small ones, in frames whose width does not fill
the last CTA's cells."""

import numpy as np
import pytest

from oracle import oraclepy
from pik_b200 import native, synthetic

pytestmark = pytest.mark.gpu

VALUES = np.array([0, 1, -1, 2, -2, 31, -32, 62, 63, -63, 64, -64, 65, 127,
                   -128, 255, 4095, -4096, 32767, -32767, -32768], np.int16)


@pytest.mark.parametrize("size", [(8, 8), (136, 24), (200, 72)])
@pytest.mark.parametrize("share", [0.02, 1.0])
def test_dequant_int16_range(size, share):
    frame = synthetic.make_frame(*size, seed=size[1], have_ar=False,
                                 shares={"DCT": 0.7, "IDENTITY": 0.3})
    rng = np.random.default_rng(int(100 * share))
    q = frame.quantized_ac
    pick = rng.random(q.shape) < share
    q[pick] = rng.choice(VALUES, size=int(pick.sum()))
    want = oraclepy.run(frame, precision=32, want=("idct", "linear"))
    ctx = native.Context(0)
    ctx.begin(frame)
    ctx.set_ac()
    ctx.reconstruct()
    np.testing.assert_array_equal(ctx.stage("idct"), want["idct"])
    ctx.close()
