"""Shared memory of another CTA of the cluster may be accessed only once that CTA has started: in every
kernel source, the first such access comes after a cluster barrier of a block that encloses it (so one
that is always passed on the way there)."""
from __future__ import annotations

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "dvr3d_b200" / "csrc"
REMOTE = re.compile(r"\b(map_shared_rank|st_async2?|bulk_to_cta|mbar_arrive_remote)\s*\(")
BARRIER = re.compile(r"(\.sync|\.barrier_wait)\s*\(\s*\)")


def _kernels(text: str):
    """(name, body) of every __global__ function, comments taken out."""
    text = re.sub(r"//[^\n]*", "", text)
    text = re.sub(r"__launch_bounds__\s*\((?:[^()]|\([^()]*\))*\)", "", text)
    for m in re.finditer(r"__global__[^;{]*?(\w+)\s*\((?=[^;{]*\)\s*\{)", text):
        start = text.index("{", m.end())
        depth = 0
        for end in range(start, len(text)):
            depth += (text[end] == "{") - (text[end] == "}")
            if depth == 0:
                break
        yield m.group(1), text[start:end + 1]


def _starts_first(body: str) -> bool:
    """A barrier whose enclosing block is still open at the first remote access."""
    at = REMOTE.search(body).start()
    for b in BARRIER.finditer(body, 0, at):
        depth = low = 0
        for ch in body[b.start():at]:
            depth += (ch == "{") - (ch == "}")
            low = min(low, depth)
        if low == 0:
            return True
    return False


def _remote_kernels():
    return [(f.name, name, body) for f in sorted(CSRC.glob("*.cu")) for name, body in _kernels(f.read_text())
            if REMOTE.search(body)]


def test_all_cluster_kernels_are_seen():
    assert {k for _, k, _ in _remote_kernels()} >= {"tridiag_kernel", "panel_qr_kernel", "vtx_kernel", "band_chase_kernel"}


@pytest.mark.parametrize("file,kernel,body", _remote_kernels(), ids=lambda v: v if len(v) < 40 else "")
def test_cluster_barrier_before_remote_access(file, kernel, body):
    assert _starts_first(body), f"{file}: {kernel} reaches into CTAs that may not have started"
