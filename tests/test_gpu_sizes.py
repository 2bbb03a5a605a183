"""Kernels at the sizes where their tiling can go wrong: edges of tiles, remainders, smallest and largest of a range."""

import pytest
import torch

from parity import assert_output_parity

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32], ids=["bf16", "f32"])
@pytest.mark.parametrize("key_dim,value_dim,steps", [(4, 4, 1), (36, 20, 3), (124, 36, 5), (128, 128, 4), (132, 44, 9), (256, 32, 2), (260, 8, 2)])
def test_linear_attention_strip_sizes(key_dim, value_dim, steps, dtype, cuda_device):
    """Row quads and column quads at and around the strip kernel's tiles (key_dim 260 is beyond it), step counts at and
    around its staging of four: the state bit-equal to the oracle's, the steps bit-equal to one-step calls."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import synthetic as syn
    from oracle import decode_oracle as oracle

    B, HK, HV = 2, 2, 4
    stream = list(syn.linear_step_stream(B, HK, HV, key_dim, value_dim, steps=steps, seed=key_dim + steps, dtype=dtype))
    dev = lambda name: torch.stack([s[name] for s in stream]).to(cuda_device)
    s_ref = syn.linear_state(B, HV, key_dim, value_dim, seed=3)
    s_one = s_ref.to(cuda_device)
    q, k, v, g, beta = (dev(n) for n in ("q", "k", "v", "g", "beta"))
    outs, final = mk.linear_attention_decode_steps(q, k, v, s_one, decay_per_step=g, beta_per_step=beta)
    for i, step in enumerate(stream):
        o_ref, s_ref = oracle.linear_attention_decode_per_head(step["q"], step["k"], step["v"], s_ref, step["g"], step["beta"])
        o_one, s_one = mk.linear_attention_decode_gated(q[i], k[i], v[i], s_one, decay_per_head=g[i], beta_per_head=beta[i])
        assert torch.equal(s_one.cpu(), s_ref)
        assert torch.equal(outs[i], o_one)
        assert_output_parity(o_one.cpu(), o_ref, what=f"strip {key_dim}x{value_dim} out {i}")
    assert torch.equal(final, s_one)
