"""The sort of the routed feed-forward, its router and its grouped products at the edges of their tiles."""

import math

import pytest
import torch

pytestmark = pytest.mark.gpu


class Step:
    def buffer(self, name, shape, dtype):
        return torch.full(tuple(shape), -7, dtype=dtype, device="cuda")


# pairs below, at and beyond what the sort's threads keep in registers (8,192); one set of counters a warp up to 256 experts
# and fewer beyond; router rows (with and without a shared gate's) one, two and four a warp, that fill
# the last warp's or do not; few pairs, with fewer sets
@pytest.mark.parametrize("T,W,E,top,shared,crowd", [(64, 64, 3, 2, True, False), (2048, 64, 32, 4, True, False), (2049, 68, 31, 4, False, False),
                                                    (5000, 36, 255, 6, False, False), (900, 40, 512, 10, False, False), (3000, 30, 5, 3, True, True), (300, 64, 16, 4, False, False),
                                                    (200, 36, 30, 5, True, False), (64, 32, 15, 3, False, False), (70, 32, 4096 // 16, 1, False, False),
                                                    (63, 32, 300, 2, False, False), (1, 64, 32, 4, True, False)])
def test_every_pair_has_a_slot_of_its_expert_and_every_tile_one_expert(T, W, E, top, shared, crowd):
    from rust_llm_inference_server_b200 import ops
    g = torch.Generator().manual_seed(T + E)
    x = torch.randn(T, W, generator=g).bfloat16()
    w = torch.randn(E + shared, W, generator=g) * 0.3
    corr = torch.zeros(E)
    if crowd:
        corr[:top] = 100.0          # everybody to the same experts
    plan = ops.moe_route(x.cuda(), w.cuda(), corr.cuda(), E, top, 2.5, shared, Step())
    z = x.double() @ w.double().t()
    scores = torch.sigmoid(z[:, :E])
    idx = plan.top_idx.view(T, top).cpu().long()
    assert bool(((idx >= 0) & (idx < E)).all()) and all(len(set(r)) == top for r in idx.tolist())
    # the chosen are the largest, up to what a float32 sum of W products can be off
    choice = scores + corr.double()
    chosen = torch.gather(choice, 1, idx)
    assert bool((chosen.min(1).values >= choice.sort(1, descending=True).values[:, top - 1] - 1e-5 * math.sqrt(W)).all())
    assert (plan.top_w.view(T, top).cpu().double() - 2.5 * torch.gather(scores, 1, idx)).abs().max() <= 1e-5 * math.sqrt(W)
    if shared:
        assert (plan.shared_gate.cpu().double() - torch.sigmoid(z[:, E])).abs().max() <= 1e-5 * math.sqrt(W)
    slots, pairs, tiles = plan.pair_slot.cpu().long(), plan.sorted_pair.cpu().long(), plan.tile_expert.cpu().long()
    n = int(tiles[plan.max_tiles])
    need = torch.bincount(idx.flatten(), minlength=E)
    assert n == int(((need + plan.tile - 1) // plan.tile).sum())
    assert bool((tiles[:n] >= 0).all()) and bool((tiles[n:plan.max_tiles] == -1).all())
    assert len(set(slots.tolist())) == T * top and bool((pairs[slots] == torch.arange(T * top)).all())
    assert int((pairs >= 0).sum()) == T * top
    assert bool((tiles[slots // plan.tile] == idx.flatten()).all())


@pytest.mark.parametrize("N,K,dtype", [(256, 64, torch.float32), (264, 72, torch.float32), (520, 200, torch.float32), (1032, 1032, torch.bfloat16),
                                       (2048, 1024, torch.float32)])
def test_grouped_products_store_ragged_columns(N, K, dtype):
    """float32 sums leave in turned blocks of 32 columns: N that ends inside a block, a tile left out, and its rows untouched."""
    from rust_llm_inference_server_b200 import ops
    E, tiles = 3, [2, 0, 0, -1, -1]
    g = torch.Generator().manual_seed(N)
    x = (torch.randn(128 * len(tiles), K, generator=g)).bfloat16()
    w = (torch.randn(E, N, K, generator=g) * 0.1).bfloat16()
    out = torch.full((x.shape[0], N), 7.0, dtype=dtype, device="cuda")
    ops.gemm_tcgen05_grouped(x.cuda(), w.cuda(), torch.tensor(tiles + [3], dtype=torch.int32).cuda(), out)
    ops.check_device_errors()
    for m, e in enumerate(tiles):
        got = out[m * 128:(m + 1) * 128].cpu()
        if e < 0:
            assert bool((got == 7.0).all())
            continue
        want = x[m * 128:(m + 1) * 128].double() @ w[e].double().t()
        # float32 sums of exact products; one rounding to bfloat16
        bound = 2.0 ** -24 * K * (x[m * 128:(m + 1) * 128].abs().double() @ w[e].abs().double().t()) + (2.0 ** -8 * want.abs() if dtype == torch.bfloat16 else 0)
        assert bool(((got.double() - want).abs() <= bound).all())


@pytest.mark.parametrize("M", [128, 300])
@pytest.mark.parametrize("glu", [(1.0, None, 0.0, 0.0), (1.702, 7.0, 1.0, 0.0), (float("inf"), None, 0.0, 0.0), (1.5957691, None, 0.0, 0.044715),
                                 (1.2, 3.0, 0.5, 0.05), (float("inf"), 2.0, 1.0, 0.0)])
def test_gates_in_the_epilogue_at_large_and_small_arguments(M, glu):
    """One rounding to bfloat16 of the gate's value: sums from far below to far above where the exponential saturates."""
    from rust_llm_inference_server_b200 import ops
    slope, limit, shift, cubic = glu
    I, K = 256, 64
    g = torch.Generator().manual_seed(M)
    x = (torch.randn(M, K, generator=g) * torch.logspace(-3, 2, M)[:, None]).bfloat16()
    w = (torch.randn(2 * I, K, generator=g) * 0.3).bfloat16()
    out = ops.gemm_tcgen05(x.cuda(), w.cuda(), "glu4", glu=glu).cpu().double()
    z = (x.double() @ w.double().t()).view(M, I // 4, 2, 4)
    gt, up = z[:, :, 0].reshape(M, I), z[:, :, 1].reshape(M, I)
    if limit is not None:
        gt, up = gt.clamp(max=limit), up.clamp(-limit, limit)
    gate = gt.clamp(min=0) if slope == float("inf") else gt * torch.sigmoid(slope * (gt + cubic * gt ** 3))
    want = gate * (up + shift)
    # half a unit of bfloat16, and what an error of the sums (2^-24 K |x| |w|) does to gate and linear branch (slopes below 1.2 and |u|)
    e = 2.0 ** -24 * K * (x.abs().double() @ w.abs().double().t()).view(M, I // 4, 2, 4).amax(2).reshape(M, I)
    bound = 2.0 ** -8 * want.abs() + 4 * e * (1 + (up + shift).abs() + gate.abs()) * (1 + 3 * cubic * gt ** 2) + 1e-30
    assert bool(((out - want).abs() <= bound).all())


@pytest.mark.parametrize("M,N,K", [(129, 264, 64), (300, 520, 72), (257, 1032, 200), (2000, 2056, 512)])
def test_float32_rows_of_a_pair_of_ctas_end_inside_a_block(M, N, K):
    """Rows and columns that end inside a turned block of 32 x 32 sums, several tiles a pair: the sums of one CTA a tile, bit for bit."""
    from rust_llm_inference_server_b200 import ops
    g = torch.Generator().manual_seed(M)
    x, w = (torch.randn(n, K, generator=g).bfloat16() for n in (M, N))
    out = ops.gemm_tcgen05(x.cuda(), w.cuda(), "float32")
    ops.debug_set("gemm_pair", 0)
    try:
        assert torch.equal(out, ops.gemm_tcgen05(x.cuda(), w.cuda(), "float32"))
    finally:
        ops.debug_set("gemm_pair", -1)
    ops.check_device_errors()
    bound = 2.0 ** -24 * K * (x.abs().double() @ w.abs().double().t())              # float32 sums of exact products
    assert bool(((out.cpu().double() - x.double() @ w.double().t()).abs() <= bound).all())
