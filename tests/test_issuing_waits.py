"""Where a warp issues with no CTA-wide barrier between its waits, the lanes meet behind each wait: every lane polls for itself, and one
that fell two phases behind the elected lane would wait for a parity that comes back no more.  Checked in the source of the
kernels whose issuing warp runs ahead of the arithmetic."""

from __future__ import annotations

import os
import re

import pytest

from conftest import ROOT

CSRC = os.path.join(ROOT, "dilution-attention_b200", "csrc")

# kernel, file, where its issuing warpgroup (or warp) begins and where the compute warps' code begins
KERNELS = [
    ("forward_fused_kernel", "tc_fused_forward.cuh", "if (wg == G) {\n    // ---", "setmaxnreg.inc"),
    ("forward_main_async_kernel", "tc_kernels.cuh", "if (warp_u == 4 * NW) {", "// the checkpoint row this warpgroup starts from"),
    ("backward_main_kernel", "tc_kernels.cuh", "if (wg == 2) {\n    // ---", "setmaxnreg.inc"),
    ("wide_backward_main_kernel", "tc_wide_kernels.cuh", "setmaxnreg.dec", "setmaxnreg.inc"),
]


KERNELS += [
    ("backward_slices_kernel", "tc_kernels.cuh", "if (wg == 4) {\n    // ---", "setmaxnreg.inc"),
    ("rowpass_issuer_kernel", "tc_rowpass_kernels.cuh", "if (warp_u == 8 * NT) {", "drain_if_aborted"),
]


@pytest.mark.parametrize("kernel,name,begin,end", KERNELS, ids=[k[0] for k in KERNELS])
def test_lanes_meet_behind_every_wait(kernel, name, begin, end):
    text = open(os.path.join(CSRC, name)).read()
    text = text[re.search(r"\b" + kernel + r"\(\n", text).start():]
    part = text[text.index(begin):]
    part = part[:part.index(end)]
    waits = re.findall(r"(if \(lane == 0\) )?\b(mbar_wait\w*)\(", part)
    assert len(waits) >= 5
    for one_lane, wait in waits:
        assert wait == "mbar_wait_warp" or one_lane, (kernel, wait)


def test_the_wait_of_a_warp_meets():
    text = open(os.path.join(CSRC, "tc_common.cuh")).read()
    body = text[text.index("void mbar_wait_warp("):]
    body = body[:body.index("\n}\n")]
    assert body.index("mbar_wait(bar") < body.index("__syncwarp()")
