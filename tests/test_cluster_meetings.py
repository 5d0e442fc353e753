"""Clusters whose CTAs read or write one another's shared memory, by the kernels' source: the last meeting before a CTA leaves is one
that releases and acquires, by whole warps.  A relaxed arrival says nothing of the accesses before it, so that a CTA's shared memory
could be gone while another CTA still reads it; that is nothing a run shows."""
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "unifur_b200", "csrc")


def _bodies(text):
    """The bodies of a source's kernels, by name, without comments."""
    text = re.sub(r"//[^\n]*", "", text)
    for m in re.finditer(r"__global__[^{;]*?(\w+_kernel)\s*\([^{;]*\)\s*\{", text):
        depth, at = 1, m.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        yield m.group(1), text[m.end():at]


def _kernels() -> list:
    found = []
    for name in sorted(os.listdir(CSRC)):
        if name.endswith(".cu"):
            with open(os.path.join(CSRC, name)) as f:
                for kernel, body in _bodies(f.read()):
                    if "map_shared_rank" in body:
                        found.append(pytest.param(body, id=kernel))
    return found


def test_the_kernels_are_found():
    assert {p.id for p in _kernels()} >= {"prepass_kernel", "prepass_f32_kernel", "prepass_tc_kernel", "gradient_kernel", "thin_product_kernel",
                                          "in_out_strip_kernel"}


@pytest.mark.parametrize("body", _kernels())
def test_last_meeting_releases_and_acquires(body):
    behind = body[body.rindex("map_shared_rank"):]
    assert "relaxed" not in behind
    meeting = re.search(r"cluster\.sync\(\)|cluster_sync_all\(\)|cluster\.barrier_arrive\(\);.*cluster\.barrier_wait\(\)", behind, re.S)
    assert meeting and "return" not in behind[:meeting.start()]


@pytest.mark.parametrize("body", _kernels())
def test_aligned_meetings_come_behind_a_converged_warp(body):
    last = list(re.finditer(r"cluster_sync_all\(\)|cluster\.barrier_(arrive|wait)\(\)", body[body.rindex("map_shared_rank"):]))
    for m in last:
        before = body[:body.rindex("map_shared_rank") + m.start()]
        assert re.search(r"(__syncwarp|__syncthreads)\(\);\s*(ptx::)?$", before)
