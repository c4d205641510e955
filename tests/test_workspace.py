"""A step's scratch buffers and the recorded graphs that point into them (no GPU needed)."""

import pytest
import torch


def runner():
    from rust_llm_inference_server_b200.engine.runner import ModelRunner
    r = ModelRunner.__new__(ModelRunner)
    r.device, r._ws, r._graphs, r._graph_pool, r._capturing, r._recorded = "cpu", {}, {}, None, False, set()
    return r


def test_only_a_buffer_that_a_graph_points_into_takes_the_graphs_along():
    from rust_llm_inference_server_b200.engine.runner import _CaptureAbort
    r = runner()
    decode, prompt = r.workspace("decode", (4, 8), torch.float32), r.workspace("prompt", (16,), torch.bfloat16)
    r._capturing = True
    assert r.workspace("decode", (2, 8), torch.float32).data_ptr() == decode.data_ptr()
    with pytest.raises(_CaptureAbort):
        r.workspace("decode", (5, 8), torch.float32)              # nothing grows while a graph is recorded
    r._capturing = False
    r._graphs["step"] = "recorded"
    grown = r.workspace("prompt", (17,), torch.bfloat16)           # a prompt's buffer: no graph has seen it
    assert grown.numel() == 17 and r._graphs == {"step": "recorded"}
    r.workspace("new", (3,), torch.float32)
    assert r._graphs == {"step": "recorded"}
    r.workspace("decode", (5, 8), torch.float32)
    assert not r._graphs
    r._graphs["step"] = "recorded anew"                             # what the dropped graphs pointed into is forgotten
    r.workspace("decode", (500, 8), torch.float32)
    assert r._graphs == {"step": "recorded anew"}


def test_a_buffer_that_grows_stays_near_what_is_asked_of_it():
    """Small ones double, so that few steps reallocate; large ones have at most the slack beyond the largest step."""
    r = runner()
    slack = r.WORKSPACE_SLACK // 4
    r.workspace("small", (1000,), torch.float32)
    r.workspace("small", (1001,), torch.float32)
    assert r._ws["small"].numel() == 2000
    r.workspace("large", (2 * slack,), torch.float32)
    r.workspace("large", (2 * slack + 1,), torch.float32)
    assert r._ws["large"].numel() == 3 * slack + 1
    assert r.workspace("large", (3 * slack,), torch.float32).data_ptr() == r._ws["large"].data_ptr()
    r.workspace("large", (8 * slack,), torch.float32)
    assert r._ws["large"].numel() == 8 * slack
    r.workspace("other", (5,), torch.bfloat16)
    r.workspace("other", (6,), torch.float32)           # of another type: nothing to go by
    assert r._ws["other"].numel() == 6
