"""What a latent attention layer keeps of its key and value maps (no GPU needed)."""

import pytest
import torch

from rust_llm_inference_server_b200.parts.latent_attention import LatentAttention
from rust_llm_inference_server_b200.parts.spec import LatentAttentionSpec


@pytest.mark.parametrize("dtype,dim,v_dim,formed", [(torch.bfloat16, 128, 128, True), (torch.float32, 128, 128, False), (torch.bfloat16, 96, 128, False),
                                                    (torch.bfloat16, 128, 64, False)])
def test_key_maps_are_kept_a_second_time_only_where_heads_are_formed(dtype, dim, v_dim, formed):
    H, rot, rank, hidden = 2, 64, 64, 32
    spec = LatentAttentionSpec(hidden=hidden, n_heads=H, dim=dim, rot_dim=rot, v_dim=v_dim, q_rank=None, kv_rank=rank, scale=0.1, eps=1e-6, q_down=None,
                               q_norm=None, q_up="q", kv_down="c", kv_norm="n", k_up="k", v_up="v", o_proj="o")
    part = LatentAttention(spec, dtype, torch.device("cpu"))
    g = torch.Generator().manual_seed(dim)
    maps = {name: torch.randn(shape, generator=g).to(dtype) for name, shape in part.tensors().items()}

    class Source:
        def get(self, name, kind=None):
            return maps[name]

    part.load(Source())
    assert torch.equal(part.w_v_up, maps["v"].view(H, v_dim, rank)) and part.w_v_up.is_contiguous()
    assert torch.equal(part.w_k_fold, maps["k"].view(H, dim, rank).transpose(1, 2))
    if formed:
        assert torch.equal(part.w_kv_up, torch.cat([maps["k"], maps["v"]]))
    else:
        held = {t.untyped_storage().data_ptr(): t.untyped_storage().nbytes() for t in vars(part).values() if isinstance(t, torch.Tensor)}
        assert part.w_kv_up is None and sum(held.values()) == sum(t.numel() * t.element_size() for t in maps.values())
