"""The float32 path's kernels at the edges of their tiles and of the rules that choose between them."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


def chained(a, w):
    """Every output as one chain of fused multiply-adds over k, for a few outputs: each step rounded once from float64
    (a float32 product is exact there, and so is the sum up to one rounding that ties cannot reach twice)."""
    acc = torch.zeros(a.shape[0], w.shape[0], dtype=torch.float32)
    for k in range(a.shape[1]):
        acc = (a[:, k:k + 1].double() * w[:, k].double() + acc.double()).float()
    return acc


# (rows, features, k): rows at the steps of the few-row kernels (1, 4, 8, 16, 32) and just over, features at the two
# lines between their shapes (16 and 64 an SM) and ragged, the tiles of 64 and 128 with remainders, k below a slice, no
# multiple of one, and no multiple of 4 (loads one by one)
@pytest.mark.parametrize("shape", [(1, 2368, 132), (1, 2369, 260), (1, 9473, 68), (3, 200, 20), (4, 9472, 64), (5, 9500, 96), (8, 16, 4), (8, 2400, 516),
                                   (9, 30, 128), (16, 2369, 200), (16, 9480, 40), (17, 2000, 300), (32, 9473, 36), (33, 300, 52), (64, 2048, 256),
                                   (65, 9500, 44), (129, 3000, 84), (200, 16390, 24), (700, 2048, 72), (130, 260, 257), (31, 77, 129)])
def test_every_float32_product_is_one_chain_over_k(shape):
    from rust_llm_inference_server_b200 import ops
    M, N, K = shape
    g = torch.Generator().manual_seed(M * 31 + N)
    a, w = torch.randn(M, K, generator=g), torch.randn(N, K, generator=g)
    ad, wd = a.cuda(), w.cuda()
    out = ops.gemm_f32(ad, wd)
    want = a.double() @ w.double().t()
    # a chain of K roundings of sums up to |a| |w|: K 2^-24 in the worst case, far less in practice
    bound = K * 2.0 ** -24 * (a.abs().double() @ w.abs().double().t())
    assert bool(((out.cpu().double() - want).abs() <= bound).all())
    rows, cols = sorted({0, M // 2, M - 1}), sorted({0, 1, N // 3, N - 1})
    assert torch.equal(out.cpu()[rows][:, cols], chained(a[rows], w[cols]))
    for m in rows:          # whatever else is in the batch
        assert torch.equal(ops.gemm_f32(ad[m:m + 1].contiguous(), wd)[0], out[m])


@pytest.mark.parametrize("M,B,K,N,pad", [(1, 3, 64, 48, 4), (7, 5, 128, 64, 8), (40, 2, 36, 96, 0), (9, 4, 30, 17, 3), (150, 3, 64, 130, 4)])
def test_products_of_a_batch_read_and_write_slices_of_wider_rows(M, B, K, N, pad):
    """The per-head maps: strides between rows and heads, aligned to 16 bytes or not."""
    from rust_llm_inference_server_b200 import ops
    g = torch.Generator().manual_seed(M + B)
    a, w = torch.randn(M, B, K + pad, generator=g).cuda(), torch.randn(B, N, K, generator=g).cuda()
    out = torch.full((M, B, N + pad), 7.0, device="cuda")
    ops.gemm_f32_batched(a[:, :, pad:], w, out[:, :, :N])
    for b in range(B):
        assert torch.equal(out[:, b, :N], ops.gemm_f32(a[:, b, pad:].contiguous(), w[b].contiguous()))
    assert pad == 0 or bool((out[:, :, N:] == 7.0).all())
