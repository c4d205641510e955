"""The host-side rules that cut a decode step's contexts into pieces and choose between kernels (no GPU needed)."""

import pytest

from rust_llm_inference_server_b200 import ops


def test_decode_attention_pieces_by_batch_and_context():
    kv = 8
    sms = 148                      # the rule takes the device's count; the numbers below are a B200's
    splits = lambda n, kv, ctx: ops.decode_splits(n, kv, ctx, sms)
    for ctx in (1, 100, 512, 4096, 32768, 131072):
        # from 256 (request, kv head) pairs on the context stays whole
        assert splits(32, kv, ctx) == 1 and splits(200, kv, ctx) == 1
    for n in (1, 2, 4, 8, 12, 16, 24):
        last = 1
        for ctx in (64, 128, 500, 512, 1024, 2048, 4096, 8192, 32768):
            s = splits(n, kv, ctx)
            assert 1 <= s <= 32 and s >= last                    # never fewer pieces for a longer context
            assert s == 1 or ctx // s >= (512 if n * kv >= 64 else 128)    # no piece shorter than that
            if n * kv * min(s, 8) <= 4 * sms and s > 1:
                assert s & (s - 1) == 0                          # merged in a cluster: a power of two
            last = s
    assert splits(8, kv, 4096) == 4 and splits(1, kv, 4096) == 8 and splits(2, kv, 4096) == 8
    assert splits(16, kv, 4096) == 2 and splits(8, kv, 512) == 1
    # the rule is a function of the step's shape only: the same step, the same pieces
    assert splits(3, 2, 7000) == splits(3, 2, 7000)
    # a smaller part fills up with fewer pieces
    assert ops.decode_splits(8, kv, 4096, 32) <= splits(8, kv, 4096)


def test_float32_attention_counts_the_pieces_that_exist():
    class Step:
        def __init__(self, ctxs):
            self.decode_ctxs, self.n_decode, self.max_decode_ctx, self.carry = ctxs, len(ctxs), max(ctxs), {}

    piece, rows = ops.lib().rlis_attention_f32_piece(), ops.lib().rlis_attention_f32_split_rows()
    for ctxs in ([1], [piece], [piece + 1], [131072] + [200] * 63, [4096] * 8, [1, 255, 256, 257, 513, 5000]):
        for window in (0, 1, 255, 256, 257, 1000):
            exist = sum((c - 1) // piece - (max(0, c - window) // piece if window else 0) + 1 for c in ctxs)
            for _ in range(2):              # (the second time from the step)
                step = Step(ctxs)
                slots, folds = ops.attention_f32_split(step, window)
                assert exist <= slots < 2 * exist and slots & (slots - 1) == 0
                assert folds or exist == len(ctxs)
            step.decode_ctxs = None         # contexts known by the longest alone
            assert ops.attention_f32_split(step, window)[0] >= exist
    assert ops.attention_f32_split(Step([300] * (rows + 1)), 0) == (0, False)


def test_every_float32_product_kernel_is_reached_by_the_shapes_it_is_tested_with():
    from tests.test_float32_path_gpu import MANY_ROWS
    lib = ops.lib()
    chosen = {(lib.rlis_gemm_f32_shape(M, N, 1, int(K % 4 == 0), 148), K % 4 == 0) for (M, N, K), _ in MANY_ROWS}
    for (M, N, K), kernel in MANY_ROWS:
        assert lib.rlis_gemm_f32_shape(M, N, 1, int(K % 4 == 0), 148) == kernel
    # number 0 (few rows) has tests of its own; 1 and 2 exist for aligned rows only
    assert chosen == {(k, True) for k in range(1, lib.rlis_gemm_f32_shapes())} | {(k, False) for k in (3, 4, 5)}
    assert all(lib.rlis_gemm_f32_shape(M, N, 1, 1, 148) == 0 for M in (1, 32) for N in (16, 100000))
    assert lib.rlis_gemm_f32_shape(0, 4, 1, 1, 148) == -1


def test_formed_heads_by_step_and_memory():
    import torch

    class Step:
        n_decode, n_prefill_tiles = 0, 1

        def __init__(self, starts, lens):
            self.starts, self.q_lens = starts, lens

    takes = lambda step, window=0, heads=16, dtype=torch.bfloat16, dim=128: ops.latent_heads_takes(step, dtype, heads, dim, 64, 128, 512, window)
    assert takes(Step([0, 70], [130, 65]))
    assert not takes(Step([0], [64]), dtype=torch.float32) and not takes(Step([0], [64]), dim=96)
    long = Step([40000], [64])              # 328 MB of keys and values
    assert not takes(long) and takes(long, heads=8) and takes(long, window=1024)
    mixed = Step([0], [64])
    mixed.n_decode = 1
    assert not takes(mixed)


def test_long_portions_go_by_chunks_and_short_ones_token_by_token():
    from rust_llm_inference_server_b200.ops import _lightning_chunks_pay as pays
    assert pays(2048, 1, 2048, 2048, 148) and pays(2048, 4, 512, 2048, 148) and pays(898, 4, 700, 2048, 148)
    assert not pays(128, 1, 128, 2048, 148) and not pays(8, 8, 1, 2048, 148) and not pays(540, 41, 500, 2048, 148)
    # by the heads' key size and the rows' form: measured on both sides of the lines
    for d, form, faster, slower in [(128, "silu f32", (2048, 1, 2048, 2048), (4096, 16, 256, 2048)), (128, "plain", (256, 1, 256, 256), (128, 1, 128, 256)),
                                    (64, "plain", (256, 1, 256, 512), (128, 1, 128, 512)), (64, "silu bf16", (512, 1, 512, 1024), (192, 1, 192, 128)),
                                    (64, "silu f32", (512, 1, 512, 1024), (192, 1, 192, 128)), (128, "silu bf16", (2048, 4, 512, 2048), (8000, 8, 1000, 2048))]:
        assert pays(*faster, 148, d, form) and not pays(*slower, 148, d, form), (d, form)


# (heads, tokens of the portions, us token by token, 16 at a time, 64 at a time)
DELTA_RULE = [
    (8, [64], 20.2, 27.8, 58.6), (8, [100], 28.4, 35.5, 67.3), (8, [193], 49.0, 52.3, 75.0), (8, [256], 62.5, 62.1, 76.2), (8, [384], 92.5, 87.0, 85.4), (8, [512], 121.1, 110.2, 92.8),
    (8, [2048], 469.7, 396.1, 213.4), (8, [53, 140], 37.2, 42.5, 71.5), (8, [100, 100], 29.1, 36.9, 68.2), (8, [200, 56], 50.6, 54.0, 76.0), (8, [256, 256], 65.7, 68.0, 84.0),
    (8, [409, 1092], 258.1, 227.2, 151.0), (8, [60, 30, 100], 61.3, 48.8, 74.4), (8, [100] * 4, 66.2, 53.5, 82.4), (8, [512] * 4, 305.9, 198.4, 154.9), (8, [700] + [1] * 8, 261.4, 229.0, 154.8),
    (16, [64], 20.4, 28.1, 64.1), (16, [128], 35.3, 40.6, 70.4), (16, [193], 52.4, 57.1, 79.5), (16, [256], 66.1, 68.0, 85.3), (16, [512], 126.1, 119.3, 104.0), (16, [2048], 491.8, 435.4, 312.8),
    (16, [53, 140], 86.7, 62.6, 90.2), (16, [200, 56], 120.8, 83.0, 97.3), (16, [409, 1092], 633.2, 378.6, 272.8), (16, [200] * 4, 131.5, 198.5, 150.8), (16, [60, 30, 100], 65.7, 63.3, 87.8),
    (16, [700] + [1] * 8, 335.4, 304.6, 205.1), (16, [1500] + [1] * 30, 722.6, 660.5, 521.1),
    (32, [64], 42.9, 37.4, 70.6), (32, [128], 81.1, 61.1, 85.2), (32, [193], 122.0, 90.2, 101.3), (32, [512], 306.4, 197.4, 155.7), (32, [2048], 1229.4, 768.5, 576.9),
    (32, [53, 140], 91.7, 102.8, 107.2), (32, [409, 1092], 677.5, 700.7, 484.7), (32, [200] * 4, 228.6, 306.1, 279.4), (32, [700] + [1] * 8, 423.0, 361.7, 355.3), (32, [1500] + [1] * 30, 926.4, 814.2, 913.7)]


@pytest.mark.parametrize("heads,lens,single,sixteen,wide", DELTA_RULE)
def test_the_delta_rule_by_64_tokens_is_taken_where_it_is_faster(heads, lens, single, sixteen, wide):
    """Against what the three ways were measured to take: never slower than the way that a step would go otherwise, and never far from the faster one."""
    by_sixteen = sum(lens) >= ops.GATED_DELTA_CHUNKS_FROM * len(lens) and len(lens) * heads * 8 <= 3 * 148
    before = sixteen if by_sixteen else single
    took = wide if ops._gated_delta_wide_pays(sum(lens), len(lens), max(lens), heads * 128, 148, by_sixteen) else before
    assert took <= before and took <= 1.05 * min(before, wide)
