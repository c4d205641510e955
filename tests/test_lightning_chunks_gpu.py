"""The decayed recurrence 64 tokens at a time against the recurrence in float64, token by token."""

import pytest
import torch

pytestmark = pytest.mark.gpu


class Step:
    def __init__(self, lens, cached):
        dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        self.n_seqs, self.max_q_len = len(lens), max(lens)
        self.cu_seqlens = dev([0] + torch.tensor(lens).cumsum(0).tolist())
        self.ctx_lens = dev([n + c for n, c in zip(lens, cached)])
        self.state_slots = dev([(5 * b + 2) % (len(lens) + 2) for b in range(len(lens))])

    def buffer(self, name, shape, dtype):
        return torch.full(tuple(shape), float("nan"), dtype=dtype, device="cuda")


# portions that end inside, at and one past a chunk; requests that start here and that go on from a state; heads of 64 and 128,
# values of one and several blocks of 64 columns; columns of the projection further right
@pytest.mark.parametrize("lens,cached,H,d,dv,off", [([64], [0], 2, 128, 128, 0), ([65, 63, 1, 130], [0, 9, 0, 64], 3, 64, 192, 16), ([700], [5], 1, 128, 64, 8),
                                                    ([1, 257], [3, 0], 2, 64, 64, 0)])
@pytest.mark.parametrize("form", ["silu bf16", "silu f32", "plain"])
def test_chunks_are_the_recurrence(monkeypatch, lens, cached, H, d, dv, off, form):
    from rust_llm_inference_server_b200 import ops
    monkeypatch.setattr(ops, "_lightning_chunks_pay", lambda *a: True)
    g = torch.Generator().manual_seed(sum(lens) + d)
    T, st = sum(lens), Step(lens, cached)
    off = off if form != "plain" else 0
    rows = torch.randn(T, off + 2 * H * d + H * dv + (8 if form != "plain" else 0), generator=g)
    rows = (rows.bfloat16() if form == "silu bf16" else rows).cuda()
    decay = torch.tensor([1.0, 0.9, 0.5][:H], device="cuda")
    slots = len(lens) + 2
    before = torch.randn(slots, H, dv, d, generator=g).cuda()
    state, out = before.clone(), torch.full((T, H * dv), 7.0, device="cuda")
    n0 = dict(ops.launches_by_kernel)
    if form == "plain":
        ops.recurrence_scan(rows, out, state, decay, st, H, d, dv)
    else:
        ops.lightning_scan(rows, off, off + H * d, off + 2 * H * d, out, state, decay, st, H, d, dv)
    name = "recurrence_scan.chunks" if form == "plain" else "lightning_scan.chunks"
    assert ops.launches_by_kernel.get(name, 0) == n0.get(name, 0) + 1
    x = rows.double() if form == "plain" else torch.nn.functional.silu(rows.double())
    at, touched = 0, []
    for b, n in enumerate(lens):
        slot = (5 * b + 2) % slots
        touched.append(slot)
        q, k, v = (x[at:at + n, o:o + H * w].view(n, H, w) for o, w in ((off, d), (off + H * d, d), (off + 2 * H * d, dv)))
        S = before[slot].double() if cached[b] else torch.zeros_like(before[slot]).double()
        size = S.abs()                      # the same with every term positive: what rounding errors are measured by
        for t in range(n):
            S = decay.double()[:, None, None] * S + v[t, :, :, None] * k[t, :, None, :]
            size = decay.double()[:, None, None] * size + (v[t, :, :, None] * k[t, :, None, :]).abs()
            want, bound = (S @ q[t, :, :, None])[..., 0].flatten(), (size @ q[t, :, :, None].abs())[..., 0].flatten()
            # a few dozen roundings of half a unit each on any way from an input to an output
            assert bool(((out[at + t].double() - want).abs() <= 2.0 ** -24 * 64 * bound + 1e-12).all()), (b, t)
        assert bool(((state[slot].double() - S).abs() <= 2.0 ** -24 * 96 * size + 1e-12).all())
        at += n
    others = [s for s in range(slots) if s not in touched]
    assert torch.equal(state[others], before[others])


def test_long_portions_go_by_chunks_and_short_ones_token_by_token():
    from rust_llm_inference_server_b200.ops import _lightning_chunks_pay as pays
    assert pays(2048, 1, 2048, 2048, 148) and pays(2048, 4, 512, 2048, 148) and pays(898, 4, 700, 2048, 148)
    assert not pays(128, 1, 128, 2048, 148) and not pays(8, 8, 1, 2048, 148) and not pays(540, 41, 500, 2048, 148)


@pytest.mark.parametrize("at", [0, 5, 63, 64, 70])
@pytest.mark.parametrize("value", [float("inf"), float("nan")])
@pytest.mark.parametrize("part", ["q", "k", "v"])
def test_a_token_sees_nothing_of_what_comes_after_it(monkeypatch, at, value, part):
    """A number that is not finite in a token's query, key or value: the outputs before it are those without it, bit for bit."""
    from rust_llm_inference_server_b200 import ops
    monkeypatch.setattr(ops, "_lightning_chunks_pay", lambda *a: True)
    H, d, T = 2, 64, 100
    st, g = Step([T], [0]), torch.Generator().manual_seed(at)
    rows = torch.randn(T, 3 * H * d, generator=g).cuda()
    decay = torch.tensor([0.9, 0.5], device="cuda")
    outs = []
    for spoilt in (False, True):
        if spoilt:
            rows[at, {"q": 0, "k": H * d, "v": 2 * H * d}[part] + 3] = value              # (an entry of the first head)
        out, state = torch.zeros(T, H * d, device="cuda"), torch.zeros(3, H, d, d, device="cuda")
        ops.recurrence_scan(rows, out, state, decay, st, H, d, d)
        outs.append(out)
    clean, out = outs
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[:, d:], clean[:, d:])
    assert not bool(torch.isfinite(out[at, :d]).all())
    if part == "q":
        assert torch.equal(out[at + 1:], clean[at + 1:])
    elif part == "v":               # one column of the values
        others = [c for c in range(d) if c != 3]
        assert torch.equal(out[:, others], clean[:, others])
