"""The EPF's work list: frames in which only some 64x32 regions hold filtered
blocks, so that the EPF leaves the others out and the final pass reads them
from the EPF's input, across region edges and the image border. Bit for bit
against the FP32 oracle, without and with the stage copies (which keep every
region), and the same bytes in both."""

import dataclasses

import numpy as np
import pytest

from oracle import oraclepy
from pik_b200 import layout, native, synthetic

pytestmark = pytest.mark.gpu


def patched(w, h, seed, pattern):
    f = synthetic.make_frame(w, h, seed=seed)
    by, bx = f.blocks
    y, x = np.indices((by, bx))
    low = {"none": np.zeros((by, bx), bool),
           "checker": ((y // 4) + (x // 8)) % 2 == 0,
           "one cell": (y == by // 2) & (x == bx // 2),
           "right": x >= bx // 2, "all": np.ones((by, bx), bool)}[pattern]
    qf = np.where(low, 6, 60).astype(np.int32)
    layout.broadcast_first_block(f.ac_strategy, qf)
    return dataclasses.replace(f, raw_quant_field=qf)


@pytest.mark.parametrize("pattern", ["none", "checker", "one cell", "right",
                                     "all"])
@pytest.mark.parametrize("size", [(64, 32), (72, 40), (203, 101), (600, 264),
                                  (1030, 300)])
def test_partly_filtered_frames_bitexact(size, pattern):
    frame = patched(*size, 7, pattern)
    want = oraclepy.run(frame, precision=32, want=("ar", "linear", "srgb8"),
                        export_decisions=True)
    for keep in (False, True):
        ctx = native.Context(0, keep_stages=keep)
        ctx.begin(frame)
        ctx.set_ac()
        for _ in range(3):  # direct launches, then graph replays
            lin, rgb = ctx.reconstruct(linear=True, srgb8=True)
            np.testing.assert_array_equal(lin, want["linear"])
            np.testing.assert_array_equal(rgb, want["srgb8"])
        np.testing.assert_array_equal(ctx.stage("ar"), want["ar"])
        np.testing.assert_array_equal(ctx.decisions()[1], want["sigma"])
        ctx.close()


def test_region_list_follows_the_frame():
    """A context's next frame of the same layout (the captured graph stays
    valid) filters other regions."""
    ctx = native.Context(0)
    for pattern in ("right", "right", "right", "checker", "none", "all"):
        frame = patched(328, 136, 3, pattern)
        ctx.begin(frame)
        ctx.set_ac()
        lin, _ = ctx.reconstruct()
        want = oraclepy.run(frame, precision=32, want=("linear",))
        np.testing.assert_array_equal(lin, want["linear"])
    ctx.close()


@pytest.mark.parametrize("gaborish,sharpened", [(2, 1), (0, 0), (4, 0)])
@pytest.mark.parametrize("size", [(8, 8), (13, 70), (139, 77), (1030, 300)])
def test_guide_sources_bitexact(size, gaborish, sharpened):
    """The guide from the staged tile, smoothed or not, beyond the border of
    images narrower than a tile's halo too."""
    frame = dataclasses.replace(patched(*size, 9, "all"), gaborish=gaborish,
                                epf_use_sharpened=sharpened)
    want = oraclepy.run(frame, precision=32, want=("linear",),
                        export_decisions=True)
    ctx = native.Context(0)
    ctx.begin(frame)
    ctx.set_ac()
    lin, _ = ctx.reconstruct()
    guide, sigma = ctx.decisions()
    np.testing.assert_array_equal(guide, want["guide"])
    np.testing.assert_array_equal(sigma, want["sigma"])
    np.testing.assert_array_equal(lin, want["linear"])
    ctx.close()
