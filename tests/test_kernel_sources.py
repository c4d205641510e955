"""What the kernels' sources promise and no run without a fault can show (no GPU needed)."""

import glob
import os
import re

import pytest

KERNELS = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "rust_llm_inference_server_b200", "csrc", "kernels")


def source(name):
    with open(os.path.join(KERNELS, name)) as f:
        return re.sub(r"//[^\n]*|/\*.*?\*/", "", f.read(), flags=re.S)


def role_of(text, at):
    """The innermost block around `at` that a warp's number opens."""
    depth = 0
    for i in range(at, -1, -1):
        if text[i] == "}":
            depth += 1
        elif text[i] == "{":
            depth -= 1
            if depth < 0:
                depth = 0
                if re.search(r"if \([^;{}]*\bwarp (==|<) [^;{}]*$", text[:i]):
                    end, level = i, 0
                    while True:
                        level += {"{": 1, "}": -1}.get(text[end], 0)
                        end += 1
                        if not level:
                            return text[i:end]
    raise AssertionError("no role")


ELECTING = sorted(os.path.basename(p) for p in glob.glob(os.path.join(KERNELS, "*.cu*")) if not p.endswith("tcgen05_utils.cuh") and "elect_one()" in open(p).read())


@pytest.mark.parametrize("name", ELECTING)
def test_a_warp_that_elects_a_lane_leaves_its_waits_together(name):
    """elect.sync names all 32 lanes, so no lane may have left the loop around it: what ends such a loop is voted on (bar_wait_warp), not a lane's own
    wait or its own look at the flag that another role sets."""
    text = source(name)
    places = [m.start() for m in re.finditer(r"elect_one\(\)", text)]
    assert places
    for at in places:
        role = role_of(text, at)
        assert "bar_wait_warp(" in role
        assert not re.search(r"\bbar_wait\(", role), name
        assert not re.search(r"(?<!&)ctrl->abort", role), name
