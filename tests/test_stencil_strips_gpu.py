"""The stencil passes' strips of 120 columns (the guide's min/max and the
final pass): widths about a strip's and a region's edge, 8-bit rows at any
alignment, and a min/max over planes with NaNs."""

import dataclasses

import numpy as np
import pytest

from oracle import decisions, oraclepy
from pik_b200 import native, synthetic

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("epf,gaborish", [(1, 2), (0, 4), (1, 0), (0, 0)])
@pytest.mark.parametrize("size", [(1, 3), (8, 17), (119, 9), (120, 8),
                                  (121, 33), (125, 2), (128, 40), (241, 70)])
def test_strip_widths_bitexact(size, epf, gaborish):
    frame = dataclasses.replace(
        synthetic.make_frame(*size, seed=size[0], qf_median=6.0),
        have_ar=epf, gaborish=gaborish)
    want = oraclepy.run(frame, precision=32, want=("linear", "srgb8"),
                        export_decisions=bool(epf))
    ctx = native.Context(0)
    ctx.begin(frame)
    ctx.set_ac()
    lin, rgb = ctx.reconstruct(linear=True, srgb8=True)
    np.testing.assert_array_equal(lin, want["linear"])
    np.testing.assert_array_equal(rgb, want["srgb8"])
    if epf:
        guide, sigma = ctx.decisions()
        np.testing.assert_array_equal(guide, want["guide"])
        np.testing.assert_array_equal(sigma, want["sigma"])
    ctx.close()


@pytest.mark.parametrize("offset,pad", [(0, 0), (1, 0), (2, 3), (4, 4),
                                        (3, 1)])
def test_rgb8_alignment(offset, pad):
    import torch
    frame = synthetic.make_frame(134, 21, seed=3)
    w, h = frame.xsize, frame.ysize
    want = oraclepy.run(frame, precision=32, want=("srgb8",))["srgb8"]
    ctx = native.Context(0)
    ctx.begin(frame)
    ctx.set_ac()
    stride = 3 * w + pad
    buf = torch.full((offset + stride * h + 8,), 77, dtype=torch.uint8,
                     device="cuda")
    ctx.reconstruct_device(0, 0, buf.data_ptr() + offset, stride)
    got = buf.cpu().numpy()
    ctx.close()
    rows = got[offset:offset + stride * h].reshape(h, stride)
    np.testing.assert_array_equal(rows[:, :3 * w].reshape(h, w, 3), want)
    # Nothing beside the rows is written.
    assert (rows[:, 3 * w:] == 77).all()
    assert (got[:offset] == 77).all() and (got[offset + stride * h:] == 77).all()


@pytest.mark.parametrize("value", [np.nan, -np.nan, np.inf])
def test_minmax_of_planes_with_nan(value):
    """A channel whose plane holds NaNs: its minimum and maximum follow the
    values' bit order, and the frame's range ignores a channel whose extreme
    is NaN (fminf / fmaxf)."""
    frame = synthetic.make_frame(250, 72, seed=6, qf_median=6.0)
    table = frame.dequant_table.copy()
    # A coefficient of the 8x8 DCT in X alone.
    table[frame.dequant_offsets.reshape(-1, 7, 3)[0, 0, 0] + 9] = value
    frame = dataclasses.replace(frame, dequant_table=table)
    ctx = native.Context(0, keep_stages=True)
    ctx.begin(frame)
    ctx.set_ac()
    ctx.reconstruct()
    src = ctx.stage("smoothed")
    assert np.isnan(src[0]).any() and np.isfinite(src[1:]).all()
    _, sigma = ctx.decisions()
    ctx.close()
    lo, hi = [], []
    for p in src:
        bits = p.ravel().view(np.uint32)
        key = np.where(bits >> 31, ~bits, bits | np.uint32(1 << 31))
        lo.append(p.ravel()[key.argmin()])
        hi.append(p.ravel()[key.argmax()])
    amin, amax = np.fmin.reduce(lo), np.fmax.reduce(hi)
    with np.errstate(all="ignore"):
        stretch = np.float32(255) / np.float32(amax - amin)
    scale = np.ones(frame.ac_strategy.shape, np.float32)
    for t, s in decisions._AR_SCALE.items():
        scale[(frame.ac_strategy >> 4) == t] = s
    quant = frame.raw_quant_field.astype(np.float32) * scale * np.float32(
        0.039324273)
    want = decisions.sigma_from_quant(quant, stretch,
                                      frame.ar_sigma_lut_ids.astype(np.int64))
    np.testing.assert_array_equal(sigma, want)
