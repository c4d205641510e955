"""Where the filtered sampler's search for a threshold takes another turn: against its kernel that reads the row pass after pass."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def rows_of(V, rng):
    """Rows whose thresholds lie in the first bins with few and with many (ties) beside them, below the first bins' reach, among
    negative numbers, and rows with infinities and NaN."""
    x = (rng.normal(size=(16, V)) * 3).astype(np.float32)
    x[1] = np.round(x[1] * 4) / 4                                 # more ties than a list takes
    x[2] = 2.0
    x[3] = -100 - np.abs(x[3])
    x[4] *= 1e-20
    x[5] *= 1e4
    x[6] = 0.0
    x[6, V // 2] = 30.0                                           # one token in the top bin, everything else sixteen octaves further down
    x[7, ::3] = -np.inf
    x[8, V // 3] = np.inf
    x[9, V // 3] = np.nan
    x[10] = -x[10] * 0 - 3e38
    x[11] = rng.normal(size=V) * 1e-3 - 5
    x[12, -1] = 50.0
    x[13] = np.nan
    x[14, ::2] = -0.0
    x[15] = np.where(rng.random(V) < 0.5, x[15], -x[15] * 1e-3)
    return x


@pytest.mark.parametrize("V", [1, 7, 300, 4097, 32768, 65537, 131073, 262144])
def test_every_threshold_is_the_one_of_the_pass_after_pass_kernel(V):
    from rust_llm_inference_server_b200 import ops
    rng = np.random.default_rng(V)
    logits = torch.from_numpy(rows_of(V, rng)).cuda()
    bits = lambda f: int(np.float32(f).view(np.uint32))
    settings = [(1.0, 0, 0.9), (1.25, 50, 1.0), (1.0, 40, 0.95), (1.0, 0, 0.999999), (100.0, 0, 0.5), (0.3, max(1, V - 1), 0.99), (1.0, 1, 0.5),
                (1.0, 257, 0.9), (1.0, V // 2, 1.0), (1.0, 0, 0.0), (1.0, 0, 1.0)]
    for inv_t, k, p in settings:
        u = rng.integers(0, 1 << 53, size=16, dtype=np.uint64)
        params = np.stack([np.full(16, bits(inv_t), np.uint64), np.full(16, k, np.uint64), np.full(16, bits(p), np.uint64), u & 0xFFFFFFFF, u >> 32], axis=1)
        pt = torch.from_numpy(params.astype(np.uint32).view(np.int32)).cuda()
        got = ops.sample_filtered(logits, pt).tolist()
        ops.debug_set("filtered_cluster", 0)
        try:
            want = ops.sample_filtered(logits, pt).tolist()
        finally:
            ops.debug_set("filtered_cluster", 1)
        same = [r for r in range(16) if got[r] != want[r]]
        assert not same, (inv_t, k, p, same)
        assert all(0 <= t < V for t in got)


@pytest.mark.parametrize("V", [7, 300, 40000, 131073, 300000])
def test_logits_that_are_not_finite(V):
    """A NaN is never drawn and takes no place in a top-k set, infinite logits share the mass, a row without anything above -inf gives id 0; in
    vocabularies of either kernel, against the same draw among the other logits on the host."""
    from rust_llm_inference_server_b200 import ops
    rng = np.random.default_rng(V)
    x = np.round(rng.normal(size=(8, V)) * 8).astype(np.float32) / 4 - 3
    holes = rng.permutation(V)[:max(2, V // 3)]
    neg = np.array([0xFFC00000, 0xFFFFFFFF, 0x7F800001, 0x7FFFFFFF], np.uint32).view(np.float32)
    x[0, holes] = neg[np.arange(holes.size) % 4]                  # of both signs
    x[1, holes[0]] = np.nan
    x[1, holes[1]] = 90.0                                         # everything else weighs nothing
    x[2, holes[:2]] = np.inf
    x[3] = -np.inf
    x[4] = np.nan
    x[5, holes[0]], x[5, holes[1]] = np.inf, np.nan
    x[6] = np.nan
    x[6, holes[1]] = -5.0
    x[7, holes] = -np.inf
    bits = lambda f: int(np.float32(f).view(np.uint32))
    for k, p in [(0, 0.9), (5, 1.0), (40, 0.95), (0, 1.0), (V - 1, 0.99), (2, 0.3)]:
        u = rng.integers(0, 1 << 53, size=8, dtype=np.uint64)
        params = np.stack([np.full(8, bits(1.0), np.uint64), np.full(8, k, np.uint64), np.full(8, bits(p), np.uint64), u & 0xFFFFFFFF, u >> 32], axis=1)
        pt = torch.from_numpy(params.astype(np.uint32).view(np.int32)).cuda()
        got = ops.sample_filtered(torch.from_numpy(x).cuda(), pt).tolist()
        for r in range(8):
            live = np.flatnonzero(~np.isnan(x[r]))
            if live.size == 0 or x[r, live].max() == -np.inf:
                assert got[r] == 0
                continue
            top = x[r, live].max()
            with np.errstate(invalid="ignore"):
                w = np.where(x[r, live] == top, 1.0, np.exp(x[r, live].astype(np.float64) - top))
            order = np.lexsort((live, -x[r, live]))               # falling, ties by id
            kept = order[:k] if 0 < k < V else order
            if p < 1:
                share = np.cumsum(w[kept]) / w[kept].sum()
                kept = kept[:int(np.searchsorted(share, p - 1e-6)) + 1]
            assert got[r] in live[kept] or (p < 1 and got[r] in live[order[:kept.size + 1]]), (V, r, k, p)
            assert w[np.flatnonzero(live == got[r])[0]] > 0
