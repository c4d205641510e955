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
    product_is_one_chain(*shape)


# what the shapes above leave out: the kernels of many rows in every form, whole and ragged, each with 16-byte and with single
# loads where it has both (the numbers are those of `rlis_gemm_f32_shape` on 148 SMs)
MANY_ROWS = [((250, 3070, 72), 4), ((256, 3072, 64), 4), ((250, 3070, 73), 4), ((256, 3072, 30), 4), ((1000, 4096, 36), 3), ((700, 2050, 33), 3),
             ((1030, 4000, 130), 3), ((40, 4001, 44), 1), ((64, 2048, 256), 2), ((33, 5001, 40), 5), ((33, 5001, 41), 5)]


@pytest.mark.parametrize("shape,kernel", MANY_ROWS)
def test_float32_products_of_many_rows_in_every_form(shape, kernel):
    from rust_llm_inference_server_b200 import ops
    product_is_one_chain(*shape)
    if ops.num_sms() == 148:
        assert ops.lib().rlis_gemm_f32_shape(shape[0], shape[1], 1, int(shape[2] % 4 == 0), 148) == kernel


def product_is_one_chain(M, N, K):
    from rust_llm_inference_server_b200 import ops
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


class Step:
    """The arrays of a step in which requests with `lens` cached tokens run their last `q_lens` tokens."""

    def __init__(self, lens, q_lens, tables, single):
        dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        self.positions = torch.cat([torch.arange(n - m, n, dtype=torch.int32) for n, m in zip(lens, q_lens)]).cuda()
        self.seq_of_token = torch.cat([torch.full((m,), b, dtype=torch.int32) for b, m in enumerate(q_lens)]).cuda()
        self.block_tables = [tables.cuda()]
        rows, dec, pf = 0, [], []
        for m in q_lens:
            (dec if single or m == 1 else pf).extend(range(rows, rows + m))
            rows += m
        self.n_decode, self.n_prefill_tokens = len(dec), len(pf)
        self.dec_rows, self.prefill_rows = dev(dec), dev(pf) if dec else None
        self.max_decode_ctx = max(lens)

    def buffer(self, name, shape, dtype):
        return torch.full(tuple(shape), float("nan"), dtype=dtype, device="cuda")


@pytest.mark.parametrize("nh,nkv,d,page,window", [(32, 8, 64, 16, 0), (6, 2, 128, 16, 0), (8, 1, 16, 8, 0), (5, 5, 48, 4, 0), (10, 2, 80, 32, 0),
                                                  (8, 2, 64, 16, 1), (8, 2, 64, 16, 33), (4, 2, 32, 16, 256), (3, 1, 64, 16, 400)])
def test_float32_attention_gives_a_token_the_same_bits_however_the_step_is_cut(nh, nkv, d, page, window):
    """Contexts around the edges of blocks (32) and pieces (256): against the kernel with a warp a head (the same up to the
    order of the sums), and every token as one of a prompt against itself as a single token."""
    from rust_llm_inference_server_b200 import ops
    lens, q_lens = [1, 32, 33, 255, 256, 257, 513, 800], [1, 32, 1, 255, 70, 257, 1, 800]
    g = torch.Generator().manual_seed(nh + window)
    pages = -(-max(lens) // page)
    tables = torch.randperm(len(lens) * pages, generator=g).to(torch.int32).view(len(lens), pages)
    kc, vc = (torch.randn(len(lens) * pages, nkv, page, d, generator=g).cuda() for _ in range(2))
    q = torch.randn(sum(q_lens), nh * d, generator=g).cuda()
    assert ops.attention_f32_takes(q.dtype, nh, nkv, d)
    args = (0, nh, nkv, d, page, 1 / math.sqrt(d), window)
    mixed, single = (ops.attention(q, kc, vc, torch.full_like(q, 7.0), Step(lens, q_lens, tables, s), *args) for s in (False, True))
    assert torch.equal(mixed, single)
    st = Step(lens, q_lens, tables, False)
    want = ops.attention_generic(q, kc, vc, torch.empty_like(q), st.seq_of_token, st.positions, st.block_tables[0], *args[1:])
    # sums of at most 800 terms of weights that add up to one and values around one
    assert (mixed - want).abs().max() <= 2e-5


def test_float32_attention_shows_a_page_that_is_not_there():
    from rust_llm_inference_server_b200 import ops
    tables = torch.arange(20, dtype=torch.int32).view(1, 20)
    tables[0, 17] = -1                      # keys 272 .. 287, in the second piece
    kc, vc, q = torch.randn(20, 1, 16, 64).cuda(), torch.randn(20, 1, 16, 64).cuda(), torch.randn(300, 64).cuda()
    for single in (False, True):
        out = ops.attention(q, kc, vc, torch.zeros_like(q), Step([300], [300], tables, single), 0, 1, 1, 64, 16, 0.125, 0)
        assert bool(torch.isfinite(out[:272]).all()) and bool(torch.isnan(out[272:]).all())


def test_pieces_cover_every_context():
    """Without a GPU's help: as many pieces as the longest context (or window) can touch, and a power of two."""
    from rust_llm_inference_server_b200 import ops
    piece = 256
    for ctx in (1, 255, 256, 257, 512, 513, 4095, 4097):
        for window in (0, 1, 255, 256, 257, 1000):
            touched = max(p // piece - (max(0, p - window + 1) if window else 0) // piece + 1 for p in range(ctx))
            n = ops.attention_f32_pieces(ctx, window)
            assert n >= touched and n & (n - 1) == 0 and n < 2 * touched + 2


@pytest.mark.parametrize("lo,hi", [(0, 32), (256, 288), (256, 512), (200, 300), (0, 512)])
def test_float32_attention_passes_by_keys_whose_scores_are_minus_infinity(lo, hi):
    """Whole blocks and pieces of such keys, at the start and behind others: what is left is the softmax over the other keys."""
    from rust_llm_inference_server_b200 import ops
    n = 600
    g = torch.Generator().manual_seed(lo + hi)
    tables = torch.arange(40, dtype=torch.int32).view(1, 40)
    kc, vc, q = torch.randn(40, 1, 16, 64, generator=g), torch.randn(40, 1, 16, 64, generator=g), torch.randn(n, 64, generator=g)
    q[:, 0] = 1.0
    kc.view(640, 64)[lo:hi, 0] = -torch.inf
    rows = list(range(hi, n))                                   # (the queries before them may see nothing else)
    outs = [ops.attention(q.cuda(), kc.cuda(), vc.cuda(), torch.zeros(n, 64, device="cuda"), Step([n], [n], tables, single), 0, 1, 1, 64, 16, 0.125, 0)
            for single in (False, True)]
    s = (q.double() @ kc.view(640, 64)[:n].double().t()) * 0.125
    s = s.masked_fill(torch.arange(n)[:, None] < torch.arange(n)[None], -torch.inf)
    want = torch.softmax(s[rows], dim=1) @ vc.view(640, 64)[:n].double()
    for out in outs:
        assert (out.cpu().double()[rows] - want).abs().max() <= 2e-5
    assert torch.equal(outs[0][rows], outs[1][rows])


def decode_step(lens, tables):
    """A step of one token for each of `lens` that knows every context, and what scratch memory it was asked for."""
    st = Step(lens, [1] * len(lens), tables, True)
    st.decode_ctxs, st.carry, st.asked = list(lens), {}, []
    def buffer(name, shape, dtype):
        st.asked.append(math.prod(shape))
        return torch.full(tuple(shape), float("nan"), dtype=dtype, device="cuda")
    st.buffer = buffer
    return st


@pytest.mark.parametrize("lens,nh,nkv,d,window", [([9000] + [20] * 40, 8, 2, 64, 0), ([300, 20000, 1, 256, 257], 4, 4, 32, 0), ([9000] * 3 + [5] * 90, 16, 2, 128, 700),
                                                  ([100] * 9, 8, 1, 64, 0), ([4097], 6, 2, 80, 0), ([513] * 300, 2, 2, 16, 0), ([600] + [3] * 1100, 4, 2, 16, 0)])
def test_float32_decode_asks_for_the_pieces_that_exist(lens, nh, nkv, d, window):
    """Ragged contexts: scratch memory by the sum of the pieces, not by the longest context for each; the bits of every request on its own."""
    from rust_llm_inference_server_b200 import ops
    page = 16
    g = torch.Generator().manual_seed(len(lens) + nh)
    used = [-(-n // page) for n in lens]
    tables = torch.full((len(lens), max(used)), -1, dtype=torch.int32)
    order = torch.randperm(sum(used), generator=g).to(torch.int32)
    for b, n in enumerate(used):
        tables[b, :n] = order[sum(used[:b]):sum(used[:b]) + n]
    kc, vc = (torch.randn(sum(used), nkv, page, d, generator=g).cuda() for _ in range(2))
    q = torch.randn(len(lens), nh * d, generator=g).cuda()
    args = (0, nh, nkv, d, page, 1 / math.sqrt(d), window)
    st = decode_step(lens, tables)
    out = ops.attention(q, kc, vc, torch.full_like(q, 7.0), st, *args)
    pieces = sum((n - 1) // 256 + 1 - (max(0, n - window) // 256 if window else 0) for n in lens)
    assert sum(st.asked) <= 2 * pieces * nh * (d + 2)
    for b in sorted({0, 1, len(lens) // 2, len(lens) - 1} & set(range(len(lens)))):
        one = Step([lens[b]], [1], tables[b:b + 1], True)
        assert torch.equal(ops.attention(q[b:b + 1].contiguous(), kc, vc, torch.zeros(1, nh * d, device="cuda"), one, *args)[0], out[b]), b
    want = ops.attention_generic(q, kc, vc, torch.empty_like(q), st.seq_of_token, st.positions, st.block_tables[0], *args[1:])
    # sums of weights that add up to one and values around one
    assert (out - want).abs().max() <= 2e-5


@pytest.mark.parametrize("interleave", [0, 4, 8])
def test_gates_four_at_a_time_are_the_gates_one_by_one(interleave):
    from rust_llm_inference_server_b200 import ops
    g = torch.Generator().manual_seed(interleave)
    T, I = 37, 200
    flat = torch.zeros(T * 2 * I + 1, device="cuda")
    gu, odd = (torch.randn(T, 2 * I, generator=g) * 3).cuda(), flat[1:].view(T, 2 * I)          # rows on a boundary of 16 bytes, and not
    odd.copy_(gu)
    outs = [ops.swiglu(x, torch.empty(T, I, device="cuda"), interleave) for x in (gu, odd)]
    assert torch.equal(*outs) and bool(outs[0].isfinite().all())
