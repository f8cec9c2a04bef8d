"""Rules of the kernels' sources that no run shows."""
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "onyxia_b200", "csrc", "kernels")
ELECTING = [f for f in sorted(os.listdir(KERNELS)) if f.endswith(".cu") and "elect_one()" in open(os.path.join(KERNELS, f)).read()]


@pytest.mark.parametrize("name", ELECTING)
def test_all_lanes_come_to_an_election(name):
    """A bounded wait may run out for some lanes of a warp only. An election of one lane waits for all of them: nothing that a lane knows alone stands in front
    of it, and a loop with elections is not left by single lanes."""
    text = open(os.path.join(KERNELS, name)).read()
    assert not re.findall(r"&& elect_one\(\)", text)
    left = re.findall(r"if \(([^\n]*mbar_wait[^\n]*)\) \{\s*ok = false;\s*break;", text)
    assert all("__all_sync" in condition for condition in left), left
