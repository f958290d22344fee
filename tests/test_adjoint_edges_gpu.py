"""The adjoint at the edges of its kernels' work split: frames narrower than a
64-pixel tile, one column beyond it and beyond the 256 columns a warp of the
loss takes, heights on and off the 16 rows of a tile, filtered and mostly
unfiltered blocks (quant medians 5 and 40), and each transform class nearly alone.
Against the FP64 reference gradient with the tolerances of
test_adjoint_gpu.py: relative L2 1e-3, entries within 1e-3 of the largest."""

import pytest

from pik_b200 import synthetic
from tests.test_adjoint_gpu import check_against_reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(16, 40), (64, 16), (72, 24), (257, 9),
                                  (129, 130)])
@pytest.mark.parametrize("qf_median", [5.0, 40.0])
def test_adjoint_tile_edges(size, qf_median):
    frame = synthetic.make_frame(*size, seed=31, qf_median=qf_median)
    check_against_reference(frame)


@pytest.mark.parametrize("name", ["DCT", "DCT_NOHF", "DCT16X16", "DCT32X32",
                                  "DCT4X4", "LINES"])
def test_adjoint_one_transform(name):
    frame = synthetic.make_frame(104, 72, seed=32, qf_median=6.0,
                                 shares={"DCT": 0.1, name: 0.9})
    check_against_reference(frame)
