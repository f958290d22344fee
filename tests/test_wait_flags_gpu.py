"""The contexts' wait-timeout flags share one page of pinned memory: a wait
that runs out in one context (PIKGPU_OPT_TC_WAIT_POLLS = 0, see
test_tc_wait_timeout.py) is reported by that context alone, and a context that
takes over its word starts with a clear flag."""

import numpy as np
import pytest

from pik_b200 import native, synthetic

pytestmark = pytest.mark.gpu


def test_flags_of_contexts_are_apart():
    frame = synthetic.make_frame(264, 136, seed=3,
                                 shares={"DCT16X16": 0.6, "DCT": 0.4})

    def run(ctx):
        ctx.begin(frame)
        ctx.set_ac()
        return ctx.reconstruct(linear=True)[0]

    ctxs = [native.Context(0, form="split_bf16") for _ in range(3)]
    try:
        want = run(ctxs[0])
        ctxs[1].set_option(native.OPT_TC_WAIT_POLLS, 0)
        for _ in range(2):
            with pytest.raises(native.PikGpuError, match="timed out"):
                run(ctxs[1])
            for i in (0, 2):
                np.testing.assert_array_equal(run(ctxs[i]), want)
        ctxs.pop(1).close()
        ctxs.append(native.Context(0, form="split_bf16"))
        for ctx in ctxs:
            np.testing.assert_array_equal(run(ctx), want)
    finally:
        for ctx in ctxs:
            ctx.close()
