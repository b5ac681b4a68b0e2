"""Bounded waits of whole warps: what must hold where none of them runs out, and so what no run on a GPU shows.

A wait of the tensor-core kernels ends after a limit, or when another role has given up, and lanes of a warp may see that in different polls.  Lanes
that part, one on its way to the CTA's last barrier and others at a __syncwarp() of the loop, would wait for each other for good.  So the kernels
whose warps wait as a whole let the lanes vote: by mbar_wait_warp, or in what follows the wait."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "clusternet_b200", "csrc")


def lines_of(name):
    with open(os.path.join(CSRC, name)) as f:
        return [re.sub(r"//.*", "", line) for line in f]


@pytest.mark.parametrize("name", ["cn_gemm_small.cu", "cn_gemm_planes.cu", "cn_gemm_outer.cu"])
def test_whole_warps_vote_on_their_waits(name):
    lines, waits = lines_of(name), 0
    for i, line in enumerate(lines):
        waits += "mbar_wait" in line
        if not re.search(r"\bmbar_wait\s*[<(]", line):
            continue
        # by one lane's own word: only where the lanes do not meet before the cluster's last barrier
        if "part_bar" in line:
            continue
        assert any("__all_sync" in f or "bar.red.and" in f for f in lines[i:i + 10]), f"{name}:{i + 1}: {line.strip()}"
    assert waits > 0


def test_the_vote():
    text = "".join(lines_of("cn_tc.cuh"))
    body = text[text.index("bool mbar_wait_warp("):text.index("void tma_load_2d(")]
    ends = re.findall(r"if \((.*)\)(?: return true;| \{)", body)
    assert "return false" in body and body.count("return") == 3
    assert body.count("if (__all_sync(0xffffffffu, mbar_try(bar, parity) != 0u)) return true;") == 2 and any(e.startswith("__any_sync(") for e in ends)


def test_workers_that_may_have_given_up_meet_at_bounded_barriers_only():
    """The weight-gradient kernel's workers may leave their loop one by one; the CTA's barriers stand before it and behind it."""
    text = "".join(lines_of("cn_gemm_outer.cu"))
    assert "bar.sync" not in text
    assert text.count("__syncthreads()") == 2
