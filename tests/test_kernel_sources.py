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


def test_a_table_of_biases_reaches_every_distance_that_a_tile_reads():
    """All places of a tile against blocks of keys: the entries that its rows read, hidden keys included, lie in their head's copy of the table."""
    text = source("attention_prefill_tcgen05.cu")
    number = lambda name: int(re.search(rf"\b{name} = (\d+)\b", text).group(1))
    front, tq = number("BIAS_FRONT"), number("TQ")
    back = int(re.search(r"BIAS_PAD = BIAS_FRONT \+ (\w+)", text).group(1).replace("BIAS_BACK", str(number("BIAS_BACK")) if "BIAS_BACK" in text else ""))
    for tn in (64, 128):
        for n_dist in (1, 40, 129, 1024):
            for pos0 in range(0, 2 * n_dist + 3 * tn, 1 if n_dist < 1024 else 7):
                for tokens in {1, 2, tq - 1, tq}:
                    for key0 in range(0, pos0 + tokens, tn):
                        if pos0 - (key0 + tn - 1) >= n_dist - 1:
                            continue            # a block beyond the table's reach takes its last entry
                        first, last = pos0 - key0 - (tn - 1), pos0 + tq - 1 - key0          # (rows past the portion's end read, too)
                        assert -front <= first and last < n_dist + back, (tn, n_dist, pos0, tokens, key0)


@pytest.mark.parametrize("name,kernel", [("conv_recurrence.cuh", "delta_chunk_prepare"), ("conv_recurrence.cuh", "delta_chunk_walk"), ("conv_recurrence.cuh", "delta_chunk_outputs"),
                                         ("attention_prefill_tcgen05.cu", "attn_prefill_tc_kernel<HD, TN, false, true>"), ("gemm_f32_split.cu", "f32_split_many_kernel")])
def test_shared_memory_is_allowed_on_every_device(name, kernel):
    """What a launch asks for is set for each device that it meets (a flag for the process leaves the second device without), and its failure is told."""
    text = source(name)
    assert not re.search(r"cudaFuncSetAttribute\(" + re.escape(kernel) + r"\b", text)
    assert re.search(r"\be = rlis_allow_smem\(" + re.escape(kernel) + r"(?:<[^>]*>)?,", text)
