"""The gated delta rule 64 tokens at a time against the rule in float64, token by token."""

import pytest
import torch

pytestmark = pytest.mark.gpu


class Step:
    def __init__(self, lens, cached):
        dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        self.n_seqs, self.max_q_len, self.n_tokens = len(lens), max(lens), sum(lens)
        self.cu_seqlens = dev([0] + torch.tensor(lens).cumsum(0).tolist())
        self.ctx_lens = dev([n + c for n, c in zip(lens, cached)])
        self.slots = [(5 * b + 2) % (len(lens) + 2) for b in range(len(lens))]
        self.state_slots = dev(self.slots)
        self.seq_of_token = dev([b for b, n in enumerate(lens) for _ in range(n)])

    def buffer(self, name, shape, dtype):
        return torch.full(tuple(shape), float("nan"), dtype=dtype, device="cuda")


class Case:
    def __init__(self, lens, cached, nh, nqk, dv, dtype, gate=0.0):
        from rust_llm_inference_server_b200 import ops
        self.lens, self.cached, self.nh, self.nqk, self.d, self.dv = lens, cached, nh, nqk, 128, dv
        g = torch.Generator().manual_seed(sum(lens) + nh)
        rnd = lambda *s: torch.randn(*s, generator=g)
        self.C = 2 * nqk * 128 + nh * dv
        self.proj = rnd(sum(lens), -(-(self.C + 2 * nh) // 8) * 8).to(dtype).cuda()
        self.taps, self.a_log, self.dt_bias = (rnd(self.C, 4) * 0.5).cuda(), (rnd(nh) * 0.1 + gate).cuda(), (rnd(nh) * 0.1).cuda()
        self.before = (rnd(len(lens) + 2, ops.conv_recurrence_state_floats(nh, nqk, 128, dv, 4)) * 0.3).cuda()

    def run(self):
        from rust_llm_inference_server_b200 import ops
        n0 = ops.launches_by_kernel.get("gated_delta.wide", 0)
        state, out, st = self.before.clone(), torch.full((sum(self.lens), self.nh * self.dv), 7.0, device="cuda"), Step(self.lens, self.cached)
        ops.gated_delta(self.proj, 0, self.C, self.C + self.nh, self.taps, self.a_log, self.dt_bias, state, out, st, self.nh, self.nqk, 128, self.dv, 4, 1e-6, 128 ** -0.5)
        return out, state, st.slots, ops.launches_by_kernel.get("gated_delta.wide", 0) - n0

    def plain(self, slots):
        nh, nqk, d, dv, C, S_size = self.nh, self.nqk, self.d, self.dv, self.C, self.nh * self.dv * self.d
        outs, states, at = [], {}, 0
        unit = lambda x: x / torch.sqrt((x * x).sum(-1, keepdim=True) + 1e-6)
        for b, n in enumerate(self.lens):
            old = self.before[slots[b]].double() if self.cached[b] else torch.zeros_like(self.before[0]).double()
            x = torch.cat([old[S_size:S_size + 3 * C].view(3, C), self.proj[at:at + n, :C].double()])
            y = torch.nn.functional.silu(sum(x[j:j + n] * self.taps.double()[:, j] for j in range(4)))
            q, k = (unit(y[:, o:o + nqk * d].view(n, nqk, d)).repeat_interleave(nh // nqk, 1) for o in (0, nqk * d))
            v = y[:, 2 * nqk * d:].view(n, nh, dv)
            beta = torch.sigmoid(self.proj[at:at + n, C:C + nh].double())
            g = torch.exp(-torch.exp(self.a_log.double()) * torch.nn.functional.softplus(self.proj[at:at + n, C + nh:C + 2 * nh].double() + self.dt_bias.double()))
            S, o = old[:S_size].view(nh, dv, d).clone(), torch.empty(n, nh, dv, dtype=torch.float64, device="cuda")
            for t in range(n):
                S = g[t][:, None, None] * S
                u = beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
                S = S + u[:, :, None] * k[t][:, None, :]
                o[t] = (S @ q[t][:, :, None])[..., 0] * d ** -0.5
            outs.append(o.flatten(1))
            states[slots[b]] = (S.flatten(), x[n:].flatten())
            at += n
        return torch.cat(outs), states


# portions that end inside, at and one past a chunk, single tokens beside them; requests that start here and that go on; query heads shared and not; 64,
# 128 and 192 columns a head; decays near 1 and near 0
@pytest.mark.parametrize("lens,cached,nh,nqk,dv,gate", [([64], [0], 2, 1, 128, 0.0), ([65, 63, 1, 130], [0, 9, 4, 64], 4, 2, 64, 0.0), ([700], [5], 2, 2, 192, -4.0),
                                                        ([1, 257], [3, 0], 4, 4, 128, 3.0)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_chunks_of_64_are_the_rule(monkeypatch, lens, cached, nh, nqk, dv, gate, dtype):
    from rust_llm_inference_server_b200 import ops
    monkeypatch.setattr(ops, "_gated_delta_wide_pays", lambda *a: True)
    c = Case(lens, cached, nh, nqk, dv, dtype, gate)
    out, state, slots, wide = c.run()
    assert wide == 1
    want, states = c.plain(slots)
    # unit keys and queries: a few dozen roundings of half a unit of what passes through the state
    assert float((out.double() - want).norm() / want.norm()) <= 2.0 ** -24 * 8
    assert float((out.double() - want).abs().max()) <= 2.0 ** -24 * 128 * float(want.abs().max())
    size = nh * dv * 128
    for slot, (S, tail) in states.items():
        assert float((state[slot, :size].double() - S).norm() / S.norm()) <= 2.0 ** -24 * 8
        assert torch.equal(state[slot, size:size + tail.numel()].double(), tail)
    others = [s for s in range(len(lens) + 2) if s not in slots]
    assert torch.equal(state[others], c.before[others])


@pytest.mark.parametrize("at", [0, 5, 16, 63, 64, 70])
@pytest.mark.parametrize("part", ["q", "k", "v", "b", "a"])
def test_a_token_sees_nothing_of_what_comes_after_it(monkeypatch, at, part):
    """A NaN in a token's projection: the outputs before it are those without it, bit for bit, and so are the other heads'."""
    from rust_llm_inference_server_b200 import ops
    monkeypatch.setattr(ops, "_gated_delta_wide_pays", lambda *a: True)
    c = Case([100], [0], 2, 2, 128, torch.float32)
    clean = c.run()[0]
    c.proj[at, {"q": 3, "k": 256 + 3, "v": 512 + 3, "b": c.C, "a": c.C + 2}[part]] = float("nan")
    out = c.run()[0]
    assert torch.equal(out[:at], clean[:at]) and torch.equal(out[:, 128:], clean[:, 128:])
    assert part == "a" or not bool(torch.isfinite(out[at, :128]).all())          # (a decay that is not a number counts as 0)


@pytest.mark.parametrize("logit", [300.0, 1e6, 1e12, 1e20, 1e30, float("inf")])
def test_tokens_behind_a_decay_of_nothing_keep_theirs(monkeypatch, logit):
    """A token whose decay is 0 (ln g far below float32's range of powers) empties the state; what comes after it decays as ever."""
    from rust_llm_inference_server_b200 import ops
    monkeypatch.setattr(ops, "_gated_delta_wide_pays", lambda *a: True)
    c = Case([130], [7], 2, 2, 128, torch.float32)
    for i, at in enumerate((0, 5, 9, 70, 71, 90)):          # (sums of them that have to be rounded)
        c.proj[at, c.C + c.nh] = logit * (1 + 0.37 * i)
    out, state, slots, wide = c.run()
    want, states = c.plain(slots)
    assert wide == 1 and float((out.double() - want).norm() / want.norm()) <= 2.0 ** -24 * 8
    S = states[slots[0]][0]
    assert float((state[slots[0], :S.numel()].double() - S).norm() / S.norm()) <= 2.0 ** -24 * 8


def test_long_portions_go_by_64(monkeypatch):
    from rust_llm_inference_server_b200 import ops
    pays = ops._gated_delta_wide_pays
    assert pays(2048, 1, 2048, 2048, 148, True) and pays(1501, 2, 1092, 2048, 148, True) and pays(2048, 4, 910, 2048, 148, False) and pays(512, 1, 512, 2048, 148, True)
    assert not pays(256, 1, 256, 2048, 148, True) and not pays(8, 8, 1, 2048, 148, False) and not pays(540, 41, 500, 2048, 148, False) and not pays(512, 4, 128, 2048, 148, False)
    monkeypatch.setattr(ops, "_gated_delta_wide_pays", lambda *a: True)
    monkeypatch.setattr(ops, "GATED_DELTA_WIDE_BYTES", 1 << 18)
    c = Case([64], [0], 2, 1, 128, torch.float32)
    assert c.run()[3] == 0          # too much scratch: the other kernels
