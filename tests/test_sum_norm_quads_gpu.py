"""Sums and norms by vectors of four against the definition: widths at the vectors' and the threads' edges, every combination of parts."""

import itertools

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H", [4, 260, 1024, 1028, 2048, 4096, 4100, 30])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_sum_norm_by_quads(H, dtype):
    from rust_llm_inference_server_b200 import ops
    g = torch.Generator().manual_seed(H)
    rnd = lambda *s: torch.randn(*s, generator=g).cuda()
    T = 3
    for n_branches, weighted, with_resid, with_out, normed in itertools.product((0, 1, 2), (False, True), (False, True), (False, True), (False, True)):
        if not (with_resid or with_out) or (n_branches == 0 and not with_resid):
            continue
        xs = [(rnd(T, H).to(dtype), rnd(H) if weighted else None, c) for c in (0.7, -0.4)][:n_branches]
        resid, w_out = rnd(T, H) if with_resid else None, rnd(H) if normed else None
        unit = lambda v, eps: v / torch.sqrt((v * v).mean(-1, keepdim=True) + eps)
        y = 1.5 * resid.double() if with_resid else torch.zeros(T, H, device="cuda", dtype=torch.float64)
        size = y.abs()
        for x, w, c in xs:
            term = c * (unit(x.double(), 1e-5) * w.double() if w is not None else x.double())
            y, size = y + term, size + term.abs()
        if normed:
            scale = w_out.double() / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-6)
            y, size = y * scale, size * scale.abs()
        out = torch.full((T, H), 7.0, dtype=dtype, device="cuda") if with_out else None
        ops.sum_norm(resid, 1.5, xs, w_out, 1e-6, out=out, eps_branch=1e-5)
        for got, ulp in ((resid, 2.0 ** -24), (out, 2.0 ** -24 if dtype == torch.float32 else 2.0 ** -9)):
            if got is not None:     # a norm's sum and root, and a dozen roundings
                assert bool(((got.double() - y).abs() <= (2.0 ** -24 * 32 + 2 * ulp) * size + 1e-9).all())


@pytest.mark.parametrize("dv,nh", [(128, 3), (64, 5), (36, 2), (132, 2), (30, 4)])
@pytest.mark.parametrize("gated,act", [(False, "sigmoid"), (True, "sigmoid"), (True, "silu")])
def test_head_norms_and_gates(dv, nh, gated, act):
    from rust_llm_inference_server_b200 import ops
    g = torch.Generator().manual_seed(dv)
    x, w = torch.randn(7, nh * dv, generator=g).cuda(), torch.randn(dv, generator=g).cuda()
    wide = torch.randn(7, nh * dv + 8, generator=g).bfloat16().cuda()
    gate = wide[:, 4:4 + nh * dv] if gated else None
    out = ops.head_norm_gate(x, w, 1e-5, torch.empty(7, nh * dv, dtype=torch.bfloat16, device="cuda"), nh, gate=gate, activation=act)
    v = x.double().view(7, nh, dv)
    want = (v / torch.sqrt((v * v).mean(-1, keepdim=True) + 1e-5) * w.double()).view(7, -1)
    if gated:
        z = gate.double()
        want = want * torch.sigmoid(z) * (z if act == "silu" else 1.0)
    assert bool(((out.double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-6).all())
