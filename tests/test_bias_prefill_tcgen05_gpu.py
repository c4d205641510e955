"""Attention with a bias by distance, a gate and sinks over portions of prompts on tcgen05, against float64 and against the mma.sync kernel."""

import pytest
import torch

pytestmark = pytest.mark.gpu


class Step:
    """Portions of `lens` tokens behind `cached` ones, pages in a shuffled order."""

    def __init__(self, lens, cached, page, rng):
        dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        ctx = [n + c for n, c in zip(lens, cached)]
        need = [-(-c // page) for c in ctx]
        self.pages = sum(need) + 1
        order = (torch.randperm(self.pages - 1, generator=rng) + 1).tolist()
        tables = torch.zeros(len(lens), max(need), dtype=torch.int32)
        for b, n in enumerate(need):
            tables[b, :n] = torch.tensor([order.pop() for _ in range(n)], dtype=torch.int32)
        self.tables, self.block_tables = tables, [tables.cuda()]
        self.n_seqs, self.ctx = len(lens), ctx
        self.cu_seqlens, self.ctx_lens = dev([0] + torch.tensor(lens).cumsum(0).tolist()), dev(ctx)
        tiles = sorted(((b, t) for b, n in enumerate(lens) for t in range(0, n, 64)), key=lambda x: -(cached[x[0]] + x[1]))
        self.prefill_tiles, self.n_prefill_tiles, self.n_decode = dev(tiles), len(tiles), 0


# portions that end inside, at and one past a tile and a block of keys, with and without tokens before them; groups of 2, 3 and 4; tables of one entry, one that ends
# inside a block, and the longest; windows; pages of 8 to 64; tiles whose last token begins a block of 128 keys (64 behind 65)
@pytest.mark.parametrize("d,group,page,lens,cached,n_dist,window,gated,sunk", [
    (64, 4, 16, [130], [0], 129, 0, True, False), (64, 2, 8, [64, 1, 65], [0, 300, 127], 1, 0, True, True), (64, 3, 64, [200, 31], [70, 0], 1024, 0, False, True),
    (64, 4, 16, [257], [40], 0, 100, False, True), (128, 2, 32, [129, 70], [0, 513], 40, 0, True, True), (128, 4, 16, [300], [0], 129, 64, True, False),
    (64, 4, 16, [700], [0], 300, 0, True, True), (64, 4, 16, [64, 65, 63], [65, 193, 1], 129, 0, True, False), (64, 2, 8, [64, 200], [65, 449], 1024, 0, False, True)])
def test_portions_on_tcgen05(monkeypatch, d, group, page, lens, cached, n_dist, window, gated, sunk):
    from rust_llm_inference_server_b200 import ops
    rng = torch.Generator().manual_seed(sum(lens) + d)
    rnd = lambda *s: torch.randn(*s, generator=rng)
    nkv, nh, T = 2, 2 * group, sum(lens)
    st = Step(lens, cached, page, rng)
    q, kc, vc = (rnd(*s).bfloat16().cuda() for s in ((T, nh * d), (st.pages, nkv, page, d), (st.pages, nkv, page, d)))
    for b, n in enumerate(st.ctx):          # what lies behind the last token of a page is never seen
        if n % page:
            vc[st.tables[b, n // page].item(), :, n % page:] = float("nan")
    bias = (rnd(n_dist, nh) * 2).cuda() if n_dist else None
    gate = rnd(T, nh + 5).bfloat16().cuda()[:, 3:3 + nh] if gated else None
    sinks = (rnd(nh) * 3).cuda() if sunk else None
    run = lambda: ops.attention_biased(q, kc, vc, torch.full((T, nh * d), 7.0, dtype=torch.bfloat16, device="cuda"), bias, gate, st, 0, nh, nkv, d, d, page, d ** -0.5, window, sinks)
    key = "attention_bias.prefill.mma.tcgen05"
    n0 = ops.launches_by_kernel.get(key, 0)
    got = run()
    assert ops.launches_by_kernel.get(key, 0) == n0 + 1
    want, at = torch.empty(T, nh, d, dtype=torch.float64, device="cuda"), 0
    for b, (n, c) in enumerate(zip(lens, cached)):
        rows = st.block_tables[0][b, :-(-(n + c) // page)].long()
        k, v = (x[rows].transpose(1, 2).reshape(-1, nkv, d)[:n + c].double() for x in (kc, vc))
        back = (c + torch.arange(n, device="cuda"))[:, None] - torch.arange(n + c, device="cuda")[None]
        hidden = (back < 0) | (back >= (window or 1 << 30))
        for h in range(nh):
            s = q[at:at + n].view(n, nh, d)[:, h].double() @ k[:, h // group].T * d ** -0.5
            if bias is not None:
                s = s + bias.double()[back.clamp(0, n_dist - 1), h]
            s = s.masked_fill(hidden, float("-inf"))
            if sinks is not None:
                s = torch.cat([s, sinks[h].double().expand(n, 1)], 1)
            want[at:at + n, h] = torch.softmax(s, 1)[:, :n + c] @ v[:, h // group]
        if gate is not None:
            want[at:at + n] *= torch.sigmoid(gate[at:at + n].double())[:, :, None]
        at += n
    want = want.flatten(1)
    # weights and results are rounded to bfloat16: two errors of 2^-9 of what they are of, and float32 sums
    assert bool(((got.double() - want).abs() <= 2.0 ** -8 * (want.abs() + 3.0)).all())
    assert float((got.double() - want).norm() / want.norm()) <= 2.0 ** -8
    monkeypatch.setattr(ops, "_biased_prefill_tc", lambda *a: False)
    other = run()
    assert ops.launches_by_kernel.get(key, 0) == n0 + 1
    assert float((got.double() - want).norm()) <= 1.25 * float((other.double() - want).norm())
    ops.check_device_errors()


@pytest.mark.parametrize("d,n_dist,window,gated,sunk", [(64, 129, 0, True, False), (64, 0, 256, False, True), (128, 40, 0, True, True), (64, 300, 100, False, False)])
def test_both_kernels_have_the_same_bits(monkeypatch, d, n_dist, window, gated, sunk):
    """The tcgen05 kernel and the mma.sync one form and sum the same weights in the same order."""
    from rust_llm_inference_server_b200 import ops
    rng = torch.Generator().manual_seed(d + n_dist)
    rnd = lambda *s: torch.randn(*s, generator=rng)
    lens, cached, nkv, nh, page = [500, 333], [0, 100], 2, 8, 16
    st, T = Step(lens, cached, page, rng), sum(lens)
    q, kc, vc = (rnd(*s).bfloat16().cuda() for s in ((T, nh * d), (st.pages, nkv, page, d), (st.pages, nkv, page, d)))
    bias = (rnd(n_dist, nh) * 2).cuda() if n_dist else None
    gate = rnd(T, nh).bfloat16().cuda() if gated else None
    sinks = rnd(nh).cuda() if sunk else None
    outs = []
    for on in (True, False):
        monkeypatch.setattr(ops, "_biased_prefill_tc", lambda *a, on=on: on)
        outs.append(ops.attention_biased(q, kc, vc, torch.empty(T, nh * d, dtype=torch.bfloat16, device="cuda"), bias, gate, st, 0, nh, nkv, d, d, page, d ** -0.5, window, sinks))
    assert torch.equal(*outs)
    ops.check_device_errors()


@pytest.mark.parametrize("d", [64, 128])
def test_edges_come_out_as_with_the_other_kernel(monkeypatch, d):
    """Heads whose keys are all masked by the table, with -inf and with float32's lowest number; sinks at both ends; a scale below zero."""
    from rust_llm_inference_server_b200 import ops
    rng = torch.Generator().manual_seed(d)
    rnd = lambda *s: torch.randn(*s, generator=rng)
    lens, cached, nkv, nh, page = [140, 70], [0, 33], 2, 8, 16
    st, T = Step(lens, cached, page, rng), sum(lens)
    q, kc, vc = (rnd(*s).bfloat16().cuda() for s in ((T, nh * d), (st.pages, nkv, page, d), (st.pages, nkv, page, d)))
    bias = rnd(50, nh).cuda()
    bias[:, 0], bias[:, 1], bias[10:, 2], bias[0, 3] = float("-inf"), torch.finfo(torch.float32).min, float("-inf"), float("-inf")
    sinks = rnd(nh).cuda()
    sinks[0], sinks[4], sinks[5] = float("-inf"), float("inf"), -1e30
    for scale in (d ** -0.5, -2.0, 0.0):
        for at in (None, sinks):
            outs = []
            for on in (True, False):
                monkeypatch.setattr(ops, "_biased_prefill_tc", lambda *a, on=on: on)
                outs.append(ops.attention_biased(q, kc, vc, torch.empty(T, nh * d, dtype=torch.bfloat16, device="cuda"), bias, None, st, 0, nh, nkv, d, d, page, scale, 0, at))
            assert bool(outs[1].isfinite().all()) and not bool(outs[1][:, :2 * d].any())
            assert torch.equal(*outs)
    ops.check_device_errors()


def test_a_portion_has_its_bits_whatever_is_beside_it():
    """A short portion beside a long one and beside a single token of a long context: the bits that it has alone, and one launch for all portions, which
    the portions choose and not the single token."""
    from rust_llm_inference_server_b200 import ops
    rng = torch.Generator().manual_seed(3)
    rnd = lambda *s: torch.randn(*s, generator=rng)
    d, nkv, nh, page, keys = 64, 2, 8, 16, ("attention_bias.prefill.mma.tcgen05", "attention_bias.prefill.mma")
    lens, cached = [100, 500, 1], [20, 0, 900]
    st = Step(lens, cached, page, rng)
    q, kc, vc = (rnd(*s).bfloat16().cuda() for s in ((sum(lens), nh * d), (st.pages, nkv, page, d), (st.pages, nkv, page, d)))
    bias = rnd(129, nh).cuda()

    def run(rows):
        part = Step.__new__(Step)
        n, c = [lens[b] for b in rows], [cached[b] for b in rows]
        dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        part.n_seqs, part.block_tables, part.ctx_lens = len(rows), [st.block_tables[0][rows].contiguous()], dev([x + y for x, y in zip(n, c)])
        part.cu_seqlens = dev([0] + torch.tensor(n).cumsum(0).tolist())
        tiles = [(b, t) for b, x in enumerate(n) if x > 1 for t in range(0, x, 64)]
        part.prefill_tiles, part.n_prefill_tiles = dev(tiles), len(tiles)
        dec = [b for b, x in enumerate(n) if x == 1]
        part.n_decode, part.dec_rows, part.dec_seqs = len(dec), dev([sum(n[:b]) for b in dec]), dev(dec)
        part.max_ctx_len, part.max_decode_ctx = max(x + y for x, y in zip(n, c)), 901
        part.max_prefill_ctx = max(x + y for x, y in zip(n, c) if x > 1)
        part.buffer = lambda name, shape, dtype: torch.empty(shape, dtype=dtype, device="cuda")
        at = [sum(lens[:b]) for b in range(3)]
        x = torch.cat([q[at[b]:at[b] + lens[b]] for b in rows])
        n0 = [ops.launches_by_kernel.get(k, 0) for k in keys]
        out = ops.attention_biased(x, kc, vc, torch.full_like(x, 7.0), bias, None, part, 0, nh, nkv, d, d, page, d ** -0.5)
        tc, all_ = (ops.launches_by_kernel.get(k, 0) - m for k, m in zip(keys, n0))
        return out.split(n), (tc, all_ - tc)

    (short,), (long,) = (run([b])[0] for b in (0, 1))
    assert run([0])[1] == (0, 1) and run([1])[1] == (1, 0) and run([0, 2])[1] == (0, 1) and run([0, 1, 2])[1] == (1, 0)
    both = run([0, 1, 2])[0]
    assert torch.equal(both[0], short) and torch.equal(both[1], long) and torch.equal(run([0, 2])[0][0], short)
    ops.check_device_errors()


def test_what_goes_there():
    from rust_llm_inference_server_b200 import ops
    x, odd = torch.zeros(4, 128, dtype=torch.bfloat16, device="cuda"), torch.zeros(513, dtype=torch.bfloat16, device="cuda")[1:].view(4, 128)
    cache, table = torch.zeros(3, 1, 16, 64, dtype=torch.bfloat16, device="cuda"), torch.zeros(1025, 2, device="cuda")
    takes = lambda q=x, bias=table[:1024], gate=None, cols=1, slopes=None, dim=64, v_dim=64, ctx=400: ops._biased_prefill_tc(q, cache, cache, x, bias, gate, cols, slopes, 2, 1, dim, v_dim, 16, ctx)
    assert takes() and takes(bias=None) and takes(gate=x) and not takes(ctx=128) and takes(ctx=128, dim=128, v_dim=128)
    assert not takes(q=odd) and not takes(bias=table) and not takes(gate=x, cols=64) and not takes(slopes=x) and not takes(v_dim=32) and not takes(dim=96, v_dim=96)
