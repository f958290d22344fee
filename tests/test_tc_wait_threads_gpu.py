"""A bounded wait of the tensor-core clamp that runs out in some of a CTA's
threads only, in its last batch: the call must report it. Every thread polls
for itself, so one may give up where the others see the completion; the
kernel's stores of that thread are then left out.

The library is built here with the wait of one thread per channel, in one of
the two inverse passes, limited to no polls at all (as if it had run out); the
pass is picked by the value of PIKGPU_OPT_TC_WAIT_POLLS, so that any other
value leaves the kernel as it is. As in test_tc_wait_timeout.py the thread then
drains the MMAs with its second wait: nothing hangs, nothing faults."""

import os
import shutil
import subprocess

import numpy as np
import pytest

from pik_b200 import build, native, synthetic

pytestmark = pytest.mark.gpu

THREAD = 64  # of a channel's 128, in another warp than the issuing thread 0
# Poll limits (far above what a wait takes) that select the pass.
PASS_POLLS = {"third": 1000003, "fourth": 1000004}
CALLS = {"third": "s.idct, 0, f.tc_polls)", "fourth": "s.idct, 1, f.tc_polls)"}


@pytest.fixture(scope="module")
def patched(tmp_path_factory):
    """The library with the waits above, in place of the in-tree one."""
    tmp = tmp_path_factory.mktemp("waits")
    src = tmp / "pik_b200" / "csrc"
    shutil.copytree(build.CSRC, src)
    shutil.copytree(os.path.join(build.ROOT, "include"), tmp / "include")
    path = src / "tc_kernels.cuh"
    text = path.read_text()
    for name, call in CALLS.items():
        assert text.count(call) == 1, call
        limit = (f"(t == {THREAD} && f.tc_polls == {PASS_POLLS[name]}u ? 0u : "
                 f"f.tc_polls))")
        text = text.replace(call, call.replace("f.tc_polls)", limit))
    path.write_text(text)
    out = tmp / "libpikgpu_waits.so"
    subprocess.run([build._nvcc(), *build.NVCC_FLAGS, "--split-compile=0",
                    "pikgpu.cu", "-o", str(out)], check=True, cwd=src)
    saved = native.LIB_PATH, native._lib
    native.LIB_PATH, native._lib = str(out), None
    yield
    native.LIB_PATH, native._lib = saved


def _run(ctx, frame):
    ctx.begin(frame)
    ctx.set_ac()
    return ctx.reconstruct(linear=True)[0]


@pytest.mark.parametrize("name", sorted(PASS_POLLS))
@pytest.mark.parametrize("form,cls", [("split_bf16", "DCT16X16"),
                                      ("split_bf16x3", "DCT16X16"),
                                      ("split_bf16", "DCT32X32")])
def test_one_threads_wait_is_reported(patched, form, cls, name):
    # A few blocks: every CTA of the clamp has one batch, its last.
    frame = synthetic.make_frame(104, 72, seed=5, qf_median=6.0,
                                 shares={cls: 1.0, "DCT": 1.0})
    ctx = native.Context(0, form=form)
    try:
        want = _run(ctx, frame)
        assert (ctx.decisions()[1] >= 16).all()  # every block is clamped
        ctx.set_option(native.OPT_TC_WAIT_POLLS, PASS_POLLS[name])
        with pytest.raises(native.PikGpuError, match="MMA.*timed out"):
            _run(ctx, frame)
        ctx.set_option(native.OPT_TC_WAIT_POLLS, -1)
        np.testing.assert_array_equal(_run(ctx, frame), want)
    finally:
        ctx.close()
