"""Attention over latents with every head's keys and values formed, against float64 and against attention on the rows."""

import pytest
import torch

pytestmark = pytest.mark.gpu


class Step:
    def __init__(self, starts, lens, page):
        dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        self.starts, self.q_lens, self.n_seqs = list(starts), list(lens), len(lens)
        ctx = [s + n for s, n in zip(starts, lens)]
        self.ctx_lens, self.cu_seqlens = dev(ctx), dev([0] + torch.tensor(lens).cumsum(0).tolist())
        width = max(-(-c // page) for c in ctx)
        perm = torch.randperm(len(lens) * width, generator=torch.Generator().manual_seed(sum(lens))).view(len(lens), width)
        self.pages, self.tables = len(lens) * width, perm
        self.block_tables = [dev(perm.tolist())]
        tiles = [(b, t) for b, n in enumerate(lens) for t in range(0, n, 64)]
        self.prefill_tiles, self.n_prefill_tiles, self.n_prefill_tokens = dev(tiles), len(tiles), sum(lens)
        self.n_decode = 0

    def buffer(self, name, shape, dtype):
        return torch.full(tuple(shape), float("nan"), dtype=dtype, device="cuda")


# portions at the edges of tiles of 64 tokens and keys, contexts before them, pages that do not divide a tile, windows inside one tile and over
# several; a latent of one vector and of 512
@pytest.mark.parametrize("starts,lens,page,window,rank,sink,gated", [([0], [64], 16, 0, 512, True, False), ([0, 70, 5], [130, 65, 2], 16, 0, 64, False, True),
                                                                     ([300], [193], 24, 40, 512, True, True), ([0, 1], [200, 63], 8, 1, 8, False, False),
                                                                     ([129, 0], [64, 257], 32, 128, 128, True, False)])
def test_heads_formed_from_latents(starts, lens, page, window, rank, sink, gated):
    from rust_llm_inference_server_b200 import ops
    H, dim, rot, dv, scale = 3, 128, 64, 128, 192 ** -0.5
    g = torch.Generator().manual_seed(rank + sum(lens))
    rnd = lambda *s: torch.randn(*s, generator=g)
    st, T = Step(starts, lens, page), sum(lens)
    cache = rnd(st.pages, 1, page, rank + rot).bfloat16().cuda()
    wide = rnd(T, H * (dim + rot) + 16).bfloat16().cuda()
    q, gate = wide[:, :H * (dim + rot)], wide[:, H * (dim + rot):H * (dim + rot) + H] if gated else None
    q_rot = rnd(T, H * rot).bfloat16().cuda()
    w = (rnd(H * (dim + dv), rank) * rank ** -0.5).bfloat16().cuda()
    sinks = rnd(H).cuda() if sink else None
    out = torch.full((T, H * dv), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.attention_latent_heads(q, q_rot, cache, w, out, st, 0, H, dim, rot, dv, rank, page, scale, sinks, window, gate=gate)
    # the kernel's inputs are the maps' results, rounded to bfloat16
    at = 0
    for b, (s, n) in enumerate(zip(starts, lens)):
        rows = cache[st.tables[b].cuda()].reshape(-1, rank + rot)[:s + n]
        kv = (rows[:, :rank] @ w.t()).double().view(s + n, -1)
        k, v = kv[:, :H * dim].view(-1, H, dim), kv[:, H * dim:].view(-1, H, dv)
        qp, qr = q[at:at + n].double().view(n, H, dim + rot)[..., :dim], q_rot[at:at + n].double().view(n, H, rot)
        sc = (torch.einsum("nhd,khd->hnk", qp, k) + torch.einsum("nhd,kd->hnk", qr, rows[:, rank:].double())) * scale
        back = (s + torch.arange(n, device="cuda"))[:, None] - torch.arange(s + n, device="cuda")[None]
        sc = sc.masked_fill((back < 0) | (back >= (window or 1 << 30)), -torch.inf)
        if sink:
            sc = torch.cat([sc, sinks.double()[:, None, None].expand(H, n, 1)], dim=2)
        p = torch.softmax(sc, dim=2)[:, :, :s + n]
        want, size = torch.einsum("hnk,khd->nhd", p, v), torch.einsum("hnk,khd->nhd", p, v.abs())
        if gated:
            f = torch.sigmoid(gate[at:at + n].double())[:, :, None]
            want, size = want * f, size * f
        # weights rounded to bfloat16 (2^-9 each), keys and values that another order of float32 sums rounds the other way (2^-8), the result's rounding
        got = out[at:at + n].double().view(n, H, dv)
        assert bool(((got - want).abs() <= 2.0 ** -6 * size + 1e-3).all()), b
        assert (got - want).norm() <= 2.0 ** -8 * 1.5 * want.norm() + 1e-6
        at += n


def test_prompts_form_heads_within_a_bound_of_memory():
    from rust_llm_inference_server_b200 import ops
    st = Step([0, 70], [130, 65], 16)
    takes = lambda s, **kw: ops.latent_heads_takes(s, kw.get("dtype", torch.bfloat16), kw.get("heads", 16), kw.get("dim", 128), 64, 128, 512)
    assert takes(st)
    assert not takes(st, dtype=torch.float32) and not takes(st, dim=96)
    st.n_decode = 1                                 # single tokens beside the portions
    assert not takes(st)
    st.n_decode, st.starts = 0, [0, 40000]          # 328 MB of keys and values
    assert not takes(st) and takes(st, heads=8)


@pytest.mark.parametrize("starts,lens,window,page", [([5000, 40, 0], [70, 3, 130], 100, 16), ([4096, 7000], [64, 2], 1, 32), ([3000], [200], 64, 24)])
def test_a_window_forms_only_the_keys_in_its_reach(starts, lens, window, page):
    """Long contexts behind a window, their early pages released: the scratch rows are those that some token of the step sees, and the outputs those
    of attention over the rows themselves with the maps behind it."""
    from rust_llm_inference_server_b200 import ops
    H, dim, rot, dv, rank, scale = 2, 128, 64, 128, 64, 192 ** -0.5
    g = torch.Generator().manual_seed(window)
    rnd = lambda *s: torch.randn(*s, generator=g)
    st, T = Step(starts, lens, page), sum(lens)
    cache = rnd(st.pages, 1, page, rank + rot).bfloat16().cuda()
    for b, s in enumerate(starts):
        released = max(0, s - window + 1) // page
        cache[st.tables[b][:released].cuda()] = float("nan")              # (another request's by now)
        st.block_tables[0][b, :released] = -1
    sizes = {}
    def buffer(name, shape, dtype):
        sizes[name] = tuple(shape)
        return torch.full(tuple(shape), float("nan"), dtype=dtype, device="cuda")
    st.buffer = buffer
    q, q_rot = rnd(T, H * (dim + rot)).bfloat16().cuda(), rnd(T, H * rot).bfloat16().cuda()
    w = (rnd(H * (dim + dv), rank) * rank ** -0.5).bfloat16().cuda()
    out = torch.full((T, H * dv), 7.0, dtype=torch.bfloat16, device="cuda")
    ops.attention_latent_heads(q, q_rot, cache, w, out, st, 0, H, dim, rot, dv, rank, page, scale, None, window)
    seen = sum(n + min(s, window - 1) for s, n in zip(starts, lens))
    assert sizes["latent_kv"][0] <= max(seen, 128) and sizes["latent_rows"][0] <= max(seen, 128)
    at = 0
    for b, (s, n) in enumerate(zip(starts, lens)):
        lo = max(0, s - window + 1)
        rows = cache[st.tables[b].cuda()].reshape(-1, rank + rot)[lo:s + n]
        kv = (rows[:, :rank] @ w.t()).double()
        k, v = kv[:, :H * dim].view(-1, H, dim), kv[:, H * dim:].view(-1, H, dv)
        qp, qr = q[at:at + n].double().view(n, H, dim + rot)[..., :dim], q_rot[at:at + n].double().view(n, H, rot)
        sc = (torch.einsum("nhd,khd->hnk", qp, k) + torch.einsum("nhd,kd->hnk", qr, rows[:, rank:].double())) * scale
        back = (s + torch.arange(n, device="cuda"))[:, None] - torch.arange(lo, s + n, device="cuda")[None]
        want = torch.einsum("hnk,khd->nhd", torch.softmax(sc.masked_fill((back < 0) | (back >= window), -torch.inf), dim=2), v)
        got = out[at:at + n].double().view(n, H, dv)
        assert bool(torch.isfinite(got).all()) and (got - want).norm() <= 2.0 ** -8 * 1.5 * want.norm() + 1e-6, b
        at += n


def test_a_window_bounds_the_memory_of_formed_heads():
    from rust_llm_inference_server_b200 import ops
    st = Step([32000, 70], [64, 65], 16)
    sizes = (torch.bfloat16, 32, 128, 64, 128, 512)
    assert not ops.latent_heads_takes(st, *sizes) and ops.latent_heads_takes(st, *sizes, window=1024)
