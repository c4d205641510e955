"""float32 products of long rows on the tensor cores: edges of tiles, segments and rings, the same bits in any step, and numbers that do not split."""

import pytest
import torch

pytestmark = pytest.mark.gpu


def operands(M, N, K, seed=0):
    g = torch.Generator(device="cuda").manual_seed(M * 31 + N + K + seed)
    return torch.randn(M, K, device="cuda", generator=g), torch.randn(N, K, device="cuda", generator=g)


def product(a, w):
    from rust_llm_inference_server_b200 import ops
    n0 = ops.launches_by_kernel.get("gemm_f32.split", 0)
    out = ops.gemm_f32(a, w)
    assert ops.launches_by_kernel["gemm_f32.split"] == n0 + 1
    return out


# rows at the ends of the kernels of few rows (16, 32) and of many, whose tiles have 16 to 160 rows in halves that are multiples of 16; features that end inside a
# tile of 128; k that ends with, inside and one float4 into a stage of 32 or 64 and a segment of 256; k cut over 1 to 12 CTAs
@pytest.mark.parametrize("M,N,K", [(1, 128, 2048), (3, 40, 2052), (8, 2048, 2048), (8, 20000, 2304), (16, 300, 8192), (17, 129, 2300), (31, 3000, 4096), (32, 16400, 2052),
                                   (33, 128, 2048), (50, 2048, 2084), (97, 300, 2560), (180, 2900, 2048), (193, 9500, 2052), (700, 2048, 2336), (800, 19000, 2048)])
def test_products_of_long_rows(M, N, K):
    from rust_llm_inference_server_b200 import ops
    a, w = operands(M, N, K)
    out = product(a, w)
    want, size = a.double() @ w.double().t(), a.abs().double() @ w.abs().double().t()
    # an accumulator truncates (a unit of 2^-23) 16 times a segment, the small products' 80 times at 2^-8 of it, the segments are added with
    # half a unit each, and three products of together 2^-24 at the most are left out
    assert bool(((out.double() - want).abs() <= (18 + K / 512) * 2.0 ** -23 * size).all())
    assert float((out.double() - want).norm() / want.norm()) <= 4e-7            # (a chain of 2,048 FMAs is 8e-7 off)
    for m in sorted({1, 8, 16, 17, 32, 33, 100, 200} & set(range(M))):          # whatever else is in the batch
        assert torch.equal(product(a[:m].contiguous(), w), out[:m])
    assert torch.equal(product(a[M // 2:].contiguous(), w), out[M // 2:])
    wide = torch.zeros(M, K + 12, device="cuda")
    wide[:, 8:8 + K] = a
    assert torch.equal(ops.linear(wide[:, 8:8 + K], w), out)                    # rows inside wider ones
    ops.check_device_errors()


@pytest.mark.parametrize("M", [4, 40])
def test_numbers_that_do_not_split_come_out_as_a_chain_gives_them(M):
    a, w = operands(M, 200, 2048)
    a[0, 5], a[1, 9], w[9, 100] = float("inf"), float("nan"), float("-inf")
    a[2, 0], a[2, 1:] = 3.4e38, 0.0                   # rounds to infinity in 8 bits; alone in its row
    a[3] *= 1e30
    w[30] *= 1e30
    got, chain = product(a, w), torch.zeros(M, 200, dtype=torch.float64, device="cuda")
    for k in range(a.shape[1]):         # the range of float32, step by step
        chain = (chain + a[:, k:k + 1].double() * w[:, k].double()).float().double()
    assert torch.equal(got.isnan(), chain.isnan()) and torch.equal(got.isinf(), chain.isinf()) and torch.equal(got[got.isinf()], chain[chain.isinf()].float())
    fine = chain.isfinite()
    size = a.abs().double() @ w.abs().double().t()
    assert bool(((got.double() - chain).abs()[fine] <= 2048 * 2.0 ** -23 * size[fine]).all()) and bool(fine.any())


def test_rows_beyond_the_scratch_go_in_portions(monkeypatch):
    from rust_llm_inference_server_b200 import ops
    a, w = operands(300, 200, 2048)
    out = product(a, w)
    monkeypatch.setattr(ops, "_SPLIT_PLANES", 100 * 6 * 2048)
    assert torch.equal(product(a, w), out)
    monkeypatch.setattr(ops, "_SPLIT_PLANES", 0)          # (33 rows at a time, the last portion of a few)
    assert torch.equal(product(a, w), out)


def test_the_rule_asks_for_the_matrix_and_the_alignment():
    from rust_llm_inference_server_b200 import ops
    a, w = operands(4, 64, 2052)
    assert ops._gemm_f32_splits(a, w) and ops._gemm_f32_splits(a[:1], w)
    assert not ops._gemm_f32_splits(a[:, :2044].contiguous(), w[:, :2044].contiguous())
    assert not ops._gemm_f32_splits(a[:, 1:2050], w[:, 1:2050])
    odd = torch.zeros(4 * 2052 + 1, device="cuda")[1:].view(4, 2052)
    assert not ops._gemm_f32_splits(odd, w)
    odd.copy_(a)
    assert torch.allclose(ops.gemm_f32(odd, w), ops.gemm_f32(a, w), rtol=0, atol=1e-3)


def test_weights_are_read_early_only_where_a_caller_says_so(monkeypatch):
    """A matrix that a kernel before may still be writing is safe in every product; the parts, whose weights are loaded, say that theirs may be read early."""
    from rust_llm_inference_server_b200 import ops
    asked = []
    real = ops._gemm_f32_split
    monkeypatch.setattr(ops, "_gemm_f32_split", lambda a, w, out, early=False: (asked.append(early), real(a, w, out, early))[1])
    a, w = operands(8, 3000, 2048)
    norm = torch.ones(2048, device="cuda")
    for _ in range(20):             # rows that are normed just before: a kernel that lets the next one start before it stores
        made = torch.zeros_like(w)
        ops.rmsnorm(w, norm, 1e-6, made)
        got = ops.linear(a, made)
        torch.cuda.synchronize()
        assert torch.equal(got, ops.gemm_f32(a, made))
    assert not any(asked)
    assert torch.equal(ops.linear(a, w, early=True), ops.gemm_f32(a, w)) and asked.count(True) == 1


@pytest.mark.parametrize("M,N,K", [(1, 300, 4100), (16, 200, 8192), (17, 300, 2052), (32, 500, 3072)])
def test_every_cut_of_k_has_the_same_bits(M, N, K):
    """k over 1 to 12 CTAs, as many as there are segments and shared memory has room for."""
    from rust_llm_inference_server_b200 import ops
    from rust_llm_inference_server_b200.ops.library import debug_set
    a, w = operands(M, N, K)
    want = product(a, w)
    try:
        for parts in range(1, 13):
            debug_set("f32_split_parts", parts)
            assert torch.equal(product(a, w), want), parts
    finally:
        debug_set("f32_split_parts", 0)
    ops.check_device_errors()


@pytest.mark.parametrize("M,N,K", [(33, 300, 2048), (170, 200, 4100)])
def test_every_height_of_a_tile_has_the_same_bits(M, N, K):
    from rust_llm_inference_server_b200 import ops
    from rust_llm_inference_server_b200.ops.library import debug_set
    a, w = operands(M, N, K)
    want = product(a, w)
    try:
        for rows in range(16, 161, 16):
            debug_set("f32_split_rows", rows)
            assert torch.equal(product(a, w), want), rows
    finally:
        debug_set("f32_split_rows", 0)
    ops.check_device_errors()


# powers of two that take a row's third part, its second and third, and all of it under the smallest bfloat16
@pytest.mark.parametrize("M,N,K", [(4, 200, 2048), (11, 300, 2304), (20, 300, 2304), (40, 200, 2048), (200, 3000, 2052), (8, 2048, 8192), (3, 20000, 2048)])
def test_small_numbers_are_as_exact_as_others(M, N, K):
    """Rows of tiny numbers against ordinary and against huge weights, tiny weights, rows of zeros: what a chain of K FMAs may be off by, and no more."""
    from rust_llm_inference_server_b200 import ops
    a, w = operands(M, N, K)
    for i in range(M):
        a[i] *= 2.0 ** (0, -90, -100, -110, -115, -120, -124, -126, -130)[i % 9]
    a[8:9] = 0.0
    w[5:60] *= 2.0 ** 100
    w[60:100] = 0.0
    w[100:130] *= 2.0 ** -110
    got = product(a, w)
    want, size = a.double() @ w.double().t(), a.abs().double() @ w.abs().double().t()
    # a rounding of half a unit at every step of the chain, and one of 2^-150 where a step's result is subnormal
    assert bool(((got.double() - want).abs() <= K * 2.0 ** -24 * size + K * 2.0 ** -150).all())
    assert not bool(got[:, 60:100].any()) and not bool(got[8:9].any())
    for m in sorted({0, 1, 4, 6, M - 1} & set(range(M))):               # whatever else is in the batch
        assert torch.equal(product(a[m:m + 1].contiguous(), w), got[m:m + 1])
    assert torch.equal(product(a[:17].contiguous(), w), got[:17])
    ops.check_device_errors()


def test_rows_that_overlap_and_rows_alone():
    """Rows that are one and the same, or a few numbers apart, go to the chains of FMAs as before; the stride of a single row is never used."""
    from rust_llm_inference_server_b200 import ops
    a, w = operands(5, 200, 2052)
    flat = torch.randn(2052 + 64, device="cuda")
    for M in (5, 40):
        same, near = a[:1].expand(M, 2052), flat.as_strided((M, 2052), (1 if M > 5 else 4, 1))
        for x in (same, near):
            assert not ops._gemm_f32_splits(x, w)
            assert torch.equal(ops.linear(x, w), chains(x, w))
    for stride in (0, 3, 2052, 5000):
        one = a.as_strided((1, 2052), (stride, 1))
        assert torch.equal(ops.linear(one, w), product(a[:1].contiguous(), w))


def chains(x, w):
    from rust_llm_inference_server_b200.ops.library import check, lib
    from rust_llm_inference_server_b200 import ops
    x, out = x.contiguous(), torch.empty(x.shape[0], w.shape[0], device="cuda")
    check(lib().rlis_gemm_f32_nt(x.data_ptr(), w.data_ptr(), out.data_ptr(), x.shape[0], w.shape[0], x.shape[1], ops._stream()), "gemm_f32")
    return out


def test_what_a_product_refuses():
    """Operands off the device, of other types and of other sizes are errors before anything is launched."""
    from rust_llm_inference_server_b200 import ops
    a, w = operands(4, 64, 2048)
    for bad in (w.cpu(), w.bfloat16(), w[:, :2044], w.t().contiguous().t(), w[:, None]):
        with pytest.raises(ops.KernelError):
            ops.linear(a, bad)
    with pytest.raises(ops.KernelError):
        ops.linear(a.cpu(), w)


@pytest.mark.parametrize("M", [4, 40])
def test_sums_that_cancel_are_not_small_numbers(M):
    """Terms that cancel exactly leave the zero that the segments' sums have, not the rounding of a chain."""
    a, w = operands(M, 200, 2048)
    w[:, 256:512], a[:, 256:512] = w[:, :256], -a[:, :256]              # a segment and its negative, term by term
    a[:, 512:] = 0.0
    assert not bool(product(a, w).any())
