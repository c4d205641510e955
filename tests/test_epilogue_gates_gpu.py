"""Gates in the epilogues of the tcgen05 products: the same numbers as the gating kernels, and what is not a number stays so."""

import pytest
import torch

pytestmark = pytest.mark.gpu

INF = float("inf")


def selected(M, I, g):
    """x [M, K] with a one in each row, and w [2 I, K] in blocks of 4: every sum is an entry of w, exactly.  The gates cover the range in
    which their exponential is neither 0 nor infinite, in steps of a last place near zero."""
    K = 128
    x = torch.zeros(M, K)
    x[torch.arange(M), torch.arange(M) % K] = 1.0
    w = torch.randn(2 * I, K, generator=g) * torch.logspace(-3, 1.6, K)
    return x.bfloat16().cuda(), w.bfloat16().cuda()


# one CTA a tile and two; whole tiles and rows beyond them; the plain gate, and the general one in every form but gelu's without limits
@pytest.mark.parametrize("M", [128, 300])
@pytest.mark.parametrize("glu", [None, (1.702, 7.0, 1.0), (1.0, None, 0.0), (1.2, None, 0.5), (INF, 2.0, 0.0), (INF, None, 0.0), (1.2, 3.0, 0.5, 0.05)])
def test_a_gate_is_the_same_number_in_an_epilogue_and_in_the_gating_kernel(M, glu):
    from rust_llm_inference_server_b200 import ops
    I = 512
    x, w = selected(M, I, torch.Generator().manual_seed(M))
    sums = w.t()[torch.arange(M) % 128].contiguous()                    # [M, 2 I], blocks of 4 gates and 4 of the linear branch
    got, want = ops.gemm_tcgen05(x, w, "swiglu4" if glu is None else "glu4", glu=glu), torch.empty(M, I, dtype=torch.bfloat16, device="cuda")
    if glu is None:
        ops.swiglu(sums, want, interleave=4)
    else:
        slope, limit, shift, *cubic = glu
        ops.glu_act(sums, want, slope, limit, shift, 4, cubic=cubic[0] if cubic else 0.0)
    ops.check_device_errors()
    assert torch.equal(got, want)


def test_a_gate_is_the_same_number_in_the_grouped_product():
    from rust_llm_inference_server_b200 import ops
    I = 256
    x, w = selected(128, I, torch.Generator().manual_seed(1))
    got, want = (torch.empty(128, I, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    ops.gemm_tcgen05_grouped(x, w[None].contiguous(), torch.tensor([0, 1], dtype=torch.int32).cuda(), got, glu=(1.702, 7.0, 1.0))
    ops.glu_act(w.t().contiguous(), want, 1.702, 7.0, 1.0, 4)
    ops.check_device_errors()
    assert torch.equal(got, want)


@pytest.mark.parametrize("M", [128, 300])
@pytest.mark.parametrize("glu", [None, (1.0, None, 0.0), (1.2, None, 0.5), (1.5957691, None, 0.0, 0.044715)])
def test_what_is_not_a_number_stays_so_behind_a_gate_without_limits(M, glu):
    from rust_llm_inference_server_b200 import ops
    I = 256
    x, w = selected(M, I, torch.Generator().manual_seed(3))
    clean = ops.gemm_tcgen05(x, w, "swiglu4" if glu is None else "glu4", glu=glu)
    w[8 * 5 + 2] = float("nan")                                         # the gate of column 4 * 5 + 2
    w[8 * 9 + 4 + 1] = float("nan")                                     # the linear branch of column 4 * 9 + 1
    out = ops.gemm_tcgen05(x, w, "swiglu4" if glu is None else "glu4", glu=glu)
    ops.check_device_errors()
    lost = [22, 37]
    others = [c for c in range(I) if c not in lost]
    assert bool(torch.isnan(out[:, lost]).all())
    assert torch.equal(out[:, others], clean[:, others])
