"""What the sources promise the hardware and no run need show.  tcgen05.ld fills its registers asynchronously, and a wait that
does not name them lets the compiler use them too early: every load is followed by a wait for the same registers.  The
.aligned cluster barrier wants whole warps, where the code in front of it has work for thread 0 alone."""

from __future__ import annotations

import glob
import os
import re

import pytest

from conftest import ROOT

SOURCES = sorted(glob.glob(os.path.join(ROOT, "dilution-attention_b200", "csrc", "tc_*.cuh")))
WAIT = {"1": "tmem_ld_wait1", "16": "tmem_ld_wait16", "32": "tmem_ld_wait"}


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_every_load_has_a_wait_that_names_its_registers(path):
    lines = open(path).read().split("\n")
    for at, line in enumerate(lines):
        assert "tmem_ld_wait()" not in line, (at + 1, line)
        load = re.search(r"^\s*tmem_ld(1|16|32)\((.*), ([&\w]+(?: \+ \d+)?)\);", line)
        if load:
            wait = f"{WAIT[load[1]]}({load[3]});"
            assert any(wait in after for after in lines[at + 1:at + 70]), (at + 1, line, wait)


def test_the_sources_are_found():
    assert sum("tmem_ld32(" in open(p).read() for p in SOURCES) >= 4


def test_cluster_barriers_do_not_take_whole_warps_for_granted():
    for path in glob.glob(os.path.join(ROOT, "dilution-attention_b200", "csrc", "*.cuh")):
        for line in open(path):
            assert not re.search(r'asm.*barrier\.cluster\..*\.aligned', line), (path, line)


@pytest.mark.parametrize("path", SOURCES, ids=os.path.basename)
def test_lanes_meet_between_a_poll_and_a_warp_wide_instruction(path):
    """Lanes may leave a polling loop in different turns; tcgen05.ld and .st and setmaxnreg want all 32 of them."""
    lines = open(path).read().split("\n")
    meets = re.compile(r"__sync(warp|threads)\(|mbar_wait_warp\(|wg_barrier\(|bar\.sync")
    wants = re.compile(r"\btmem_(ld|st)\d+\(|setmaxnreg|row_half_tile<|row_merge<")
    for at, line in enumerate(lines):
        if not re.search(r"\bmbar_wait\(", line) or "== 0) mbar_wait(" in line or "bool mbar_wait(" in line or path.endswith("tc_common.cuh"):
            continue
        for after in lines[at + 1:]:
            if meets.search(after) or after == "}":
                break
            assert not wants.search(after), (at + 1, line, after)
