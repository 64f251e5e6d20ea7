"""The rounds of the coarsest level's 32x32 block factor exchange columns through
shared memory between the lanes of one warp. Lanes do not run in step: between a
read of a slot by other lanes and the next write to it, and between a write and
its read, there has to be a warp barrier, across the end of a round too."""

from __future__ import annotations

import re

import pytest

from conftest import ROOT


def _round_events(src: str):
    """Accesses to the shared columns S.col[k] and the warp barriers of one round, in program order."""
    body = src[src.index("__device__ __forceinline__ void chol_step"):]
    body = body[:body.index("\n}\n")]
    body = re.sub(r"//[^\n]*", "", body)
    ev = []
    for m in re.finditer(r"__syncwarp\(\)|S\.col\[(\d)\]\[(\w+)\]( = )?", body):
        if m.group(0).startswith("__syncwarp"):
            ev.append(("barrier", None))
        else:
            ev.append(("write" if m.group(3) else "read", int(m.group(1))))
    return ev


def _hazards(events):
    """(earlier, later, slot) pairs of a read and a write to one slot with no barrier between, over two rounds."""
    found = []
    ev = events + events
    for i, (a, ka) in enumerate(ev):
        if a == "barrier":
            continue
        for b, kb in ev[i + 1:]:
            if b == "barrier":
                break
            if ka == kb and {a, b} == {"read", "write"}:
                found.append((a, b, ka))
    return found


def test_rounds_of_the_block_factor_are_separated_by_warp_barriers():
    ev = _round_events((ROOT / "topogpu_b200" / "csrc" / "coarsest.cu").read_text())
    assert {k for a, k in ev if a == "write"} == {0, 1, 2}
    assert {k for a, k in ev if a == "read"} >= {0, 2}
    assert _hazards(ev) == []


@pytest.mark.parametrize("drop", [0, 1, 2])
def test_the_check_sees_a_missing_barrier(drop):
    ev = _round_events((ROOT / "topogpu_b200" / "csrc" / "coarsest.cu").read_text())
    at = [i for i, (a, _) in enumerate(ev) if a == "barrier"][drop]
    assert _hazards(ev[:at] + ev[at + 1:])
