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


@pytest.mark.parametrize("heads,position,capacity,stream", [((4, 2, 64), 0, 1, 1), ((4, 2, 64), 40, 64, 1), ((16, 2, 256), 97, 200, 0),
                                                            ((6, 2, 80), 70, 75, 1), ((24, 4, 256), 130, 131, 1)])
def test_attention_block_reads_caches_longer_than_the_context(heads, position, capacity, stream, cuda_device):
    """Three tokens, rotary embedding, caches with room behind the context: the streaming, the register-staged and the
    general attention kernel (head_dim 80) over a batch stride that is not the context length."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import cabi, synthetic as syn
    from oracle import decode_oracle as oracle

    (hq, hkv, d), B, H = heads, 3, 256
    qkv = syn.projection_tensors(H, (hq + 2 * hkv) * d, B, seed=position, norm=True, residual=False)
    outp = syn.projection_tensors(hq * d, H, B, seed=43, norm=False, residual=False)
    cache = syn.attention_tensors(B, hq, hkv, d, capacity, seed=44)
    ang = torch.arange(16, dtype=torch.float32) * 0.37 + 0.1
    cos, sin = ang.cos().repeat(2), ang.sin().repeat(2)
    dev = {n: t.to(cuda_device) for n, t in cache.items()}
    block = mk.AttentionBlockInputs(qkv["norm_weight"].to(cuda_device), qkv["weight"].to(cuda_device), outp["weight"].to(cuda_device), dev["k_cache"],
                                    dev["v_cache"], position, hq, hkv, d, cos=cos, sin=sin, rotary_dim=32)
    cabi.check(cabi.load().mk36_set_option(b"attn_stream", stream))
    try:
        out, attn = mk.attention_block_decode(qkv["x"].to(cuda_device), block)
    finally:
        cabi.check(cabi.load().mk36_set_option(b"attn_stream", 1))
    want, attn_ref, k_ref, v_ref = oracle.attention_block_decode(qkv["x"], qkv["norm_weight"], qkv["weight"], outp["weight"], cache["k_cache"],
                                                                 cache["v_cache"], position, hq, hkv, d, cos=cos, sin=sin, rotary_dim=32)
    assert_output_parity(attn.cpu(), attn_ref, what="block attention")
    assert_output_parity(out.cpu(), want, what="block output")
    assert_output_parity(dev["k_cache"][:, position].cpu(), k_ref[:, position], what="block key")
    assert_output_parity(dev["v_cache"][:, position].cpu(), v_ref[:, position], what="block value")
    rest = [i for i in range(capacity) if i != position]
    assert torch.equal(dev["k_cache"][:, rest].cpu(), cache["k_cache"][:, rest]) and torch.equal(dev["v_cache"][:, rest].cpu(), cache["v_cache"][:, rest])
