"""The inputs behind the short convolutions, four channels a lane, against one channel a lane: the same projection whose columns start on a boundary
of four entries or do not."""

import pytest
import torch

pytestmark = pytest.mark.gpu


class Step:
    def __init__(self, lens, cached):
        dev = lambda x: torch.tensor(x, dtype=torch.int32, device="cuda")
        self.n_seqs = len(lens)
        self.cu_seqlens = dev([0] + torch.tensor(lens).cumsum(0).tolist())
        self.ctx_lens = dev([n + c for n, c in zip(lens, cached)])
        self.state_slots = dev(list(reversed(range(len(lens)))))
        self.seq_of_token = dev([b for b, n in enumerate(lens) for _ in range(n)])

    def buffer(self, name, shape, dtype):
        return torch.full(tuple(shape), float("nan"), dtype=dtype, device="cuda")


# one token, fewer than four, a multiple of four tokens and not, short steps (a warp a token) and long ones (four), portions shorter than the taps that
# go on from a tail; heads of one quad a lane and of more, and of fewer than 32 quads
@pytest.mark.parametrize("lens,cached", [([1], [0]), ([1, 2, 3, 1], [9, 0, 5, 0]), ([63], [4]), ([64], [0]), ([30, 1, 2, 34], [3, 7, 0, 1]), ([257, 2], [0, 2])])
@pytest.mark.parametrize("nh,n_qk,d,dv", [(4, 2, 128, 128), (2, 2, 64, 192), (3, 1, 20, 36)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_quads_are_the_channels_one_by_one(lens, cached, nh, n_qk, d, dv, dtype):
    from rust_llm_inference_server_b200 import ops
    g = torch.Generator().manual_seed(sum(lens) + d)
    rnd = lambda *s: torch.randn(*s, generator=g)
    T, C = sum(lens), 2 * n_qk * d + nh * dv
    cols = rnd(T, C + 2 * nh).to(dtype).cuda()
    conv_w, a_log, dt_bias = (rnd(C, 4) * 0.5).cuda(), (rnd(nh) * 0.1).cuda(), (rnd(nh) * 0.1).cuda()
    state0 = (rnd(len(lens), ops.conv_recurrence_state_floats(nh, n_qk, d, dv, 4)) * 0.3).cuda()
    results = []
    for off in (4, 3):          # columns on a boundary of four, and between two
        proj = torch.zeros(T, -(-(C + 2 * nh + off) // 8) * 8, dtype=dtype, device="cuda")
        proj[:, off:off + C + 2 * nh] = cols
        state, out = state0.clone(), torch.full((T, nh * dv), 7.0, device="cuda")
        ops.gated_delta(proj, off, off + C, off + C + nh, conv_w, a_log, dt_bias, state, out, Step(lens, cached), nh, n_qk, d, dv, 4, 1e-6, d ** -0.5)
        results.append((out, state))
    # the sum of squares of a head is taken in another order: a few units of 2^-24, which the recurrence carries on
    for a, b in zip(*results):
        assert (a - b).abs().max() <= 2.0 ** -24 * 64 * b.abs().max()


@pytest.mark.parametrize("lens,cached", [([1, 2, 3, 1], [9, 0, 5, 0]), ([257, 2], [0, 2])])
@pytest.mark.parametrize("off", [4, 3])
def test_inputs_by_quads_and_by_channels_are_the_convolution(lens, cached, off):
    """Through the whole rule, against it written out in float64: convolution over the tail and the portion, silu, unit vectors, the recurrence."""
    from rust_llm_inference_server_b200 import ops
    nh, n_qk, d, dv, taps, eps = 4, 2, 64, 32, 4, 1e-6
    g = torch.Generator().manual_seed(sum(lens))
    rnd = lambda *s: torch.randn(*s, generator=g)
    T, C = sum(lens), 2 * n_qk * d + nh * dv
    proj = torch.zeros(T, -(-(C + 2 * nh + off) // 8) * 8)
    proj[:, off:off + C + 2 * nh] = rnd(T, C + 2 * nh)
    conv_w, a_log, dt_bias = rnd(C, taps) * 0.5, rnd(nh) * 0.1, rnd(nh) * 0.1
    state = rnd(len(lens), ops.conv_recurrence_state_floats(nh, n_qk, d, dv, taps)) * 0.3
    st, out = Step(lens, cached), torch.full((T, nh * dv), 7.0, device="cuda")
    ops.gated_delta(proj.cuda(), off, off + C, off + C + nh, conv_w.cuda(), a_log.cuda(), dt_bias.cuda(), state.cuda(), out, st, nh, n_qk, d, dv, taps, eps,
                    d ** -0.5)
    x, at = proj.double(), 0
    for b, n in enumerate(lens):
        slot = len(lens) - 1 - b
        S = state[slot, :nh * dv * d].double().view(nh, dv, d) if cached[b] else torch.zeros(nh, dv, d).double()
        tail = state[slot, nh * dv * d:nh * dv * d + (taps - 1) * C].double().view(taps - 1, C) if cached[b] else torch.zeros(taps - 1, C).double()
        rows = torch.cat([tail, x[at:at + n, off:off + C]])
        y = torch.nn.functional.silu(sum(conv_w[:, k].double() * rows[k:k + n] for k in range(taps)))
        q, k = (y[:, o:o + n_qk * d].reshape(n, n_qk, d) for o in (0, n_qk * d))
        q, k = (v / torch.sqrt((v * v).sum(2, keepdim=True) + eps) for v in (q, k))
        q, k = (v.repeat_interleave(nh // n_qk, dim=1) for v in (q * d ** -0.5, k))
        v = y[:, 2 * n_qk * d:].reshape(n, nh, dv)
        beta = torch.sigmoid(x[at:at + n, off + C:off + C + nh])
        decay = torch.exp(-torch.exp(a_log.double()) * torch.nn.functional.softplus(x[at:at + n, off + C + nh:off + C + 2 * nh] + dt_bias.double()))
        for t in range(n):
            S = decay[t][:, None, None] * S
            u = beta[t][:, None] * (v[t] - (S @ k[t][:, :, None])[..., 0])
            S = S + u[:, :, None] * k[t][:, None, :]
            want = (S @ q[t][:, :, None])[..., 0].flatten()
            # float32 sums over 64 entries, carried on by a recurrence that contracts
            assert (out[at + t].cpu().double() - want).abs().max() <= 2.0 ** -24 * 256 * max(1.0, S.abs().max().item()), (b, t)
        at += n
