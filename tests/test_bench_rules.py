"""bench.py names the kernel of a stage by the engine's size rules; where it
repeats one of their limits, it is the engine's."""
import os
import re

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_mixed_mode_limit():
    import bench
    with open(os.path.join(ROOT, "mbd_b200", "csrc", "context.h")) as fh:
        limit = int(re.search(r"constexpr int kMixedDirectMaxN = (\d+);", fh.read()).group(1))
    assert bench.MIXED_DIRECT_MAX_N == limit
