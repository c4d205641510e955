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
