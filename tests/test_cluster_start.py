"""Kernels that write into the shared memory of the other blocks of their
cluster: a block's shared memory exists only once the block has started, so a
cluster barrier must have completed before the first such access.  Read from
the sources (no GPU): in every kernel that maps a peer's shared memory, the
first access through the mapping, by the kernel's text or by the first call of
a local lambda that makes it, comes after the first complete cluster barrier."""
import glob
import os
import re

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mbd_b200", "csrc")
BARRIER = r"cl\.sync\(|cl\.barrier_wait\(|cluster_wait\("


def _block_end(s, at):
    """Position behind the brace block that opens at or after `at`."""
    at = s.index("{", at)
    depth = 0
    for k in range(at, len(s)):
        depth += (s[k] == "{") - (s[k] == "}")
        if depth == 0:
            return k + 1
    raise ValueError("unbalanced braces")


def cluster_kernels():
    out = []
    for path in sorted(glob.glob(os.path.join(CSRC, "*.cu"))):
        with open(path) as fh:
            src = re.sub(r"//[^\n]*", "", fh.read())
        src = re.sub(r"/\*.*?\*/", "", src, flags=re.S)
        for m in re.finditer(r"__global__\s+void\s+(?:__launch_bounds__\((?:[^()]|\([^()]*\))*\)\s*)?(\w+)\(", src):
            body = src[src.index("{", m.end()):_block_end(src, m.end())]
            if "map_shared_rank" in body:
                out.append((m.group(1), body))
    return out


def first_access_and_barrier(body):
    """(first access to a peer's shared memory, first complete cluster barrier)"""
    lambdas = [(m.group(1), m.start(), _block_end(body, m.end()))
               for m in re.finditer(r"auto (\w+) = \[&\]", body)]
    inside = lambda k: next(((name, end) for name, start, end in lambdas if start <= k < end), None)
    uses = []
    for m in re.finditer(r"map_shared_rank", body):
        at = m.start()
        line = body[body.rindex("\n", 0, at) + 1:body.index(";", at) + 1]
        # an address kept in a variable (no access yet): its later uses count
        kept = re.match(r"\s*(?:\w+\s*\*\s*)?(\w+)(?:\[\w+\])? = cl\.map_shared_rank\([^;]*;$", line)
        if kept:
            later = [u.start() for u in re.finditer(r"\b%s\b" % kept.group(1), body) if u.start() > at]
            uses += later[:1]
        elif inside(at):
            name, end = inside(at)
            uses.append(min(u.start() for u in re.finditer(r"\b%s\(" % name, body) if u.start() >= end))
        else:
            uses.append(at)
    barriers = [m.start() for m in re.finditer(BARRIER, body) if not inside(m.start())]
    return min(uses), min(barriers)


def test_finds_the_cluster_kernels():
    names = {name for name, _ in cluster_kernels()}
    assert {"trsv_cluster_kernel", "cg_cluster_kernel", "qr_panel_kernel", "qr_panel2_kernel", "tsqr_panel_kernel",
            "sb2st_cluster_kernel"} <= names


@pytest.mark.parametrize("name,body", cluster_kernels(), ids=[k[0] for k in cluster_kernels()])
def test_peers_have_started_before_the_first_access(name, body):
    use, barrier = first_access_and_barrier(body)
    assert barrier < use
