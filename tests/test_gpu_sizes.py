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


@pytest.mark.parametrize("kernel", ["dense_tiles", "projection_tiles", "projection_tiles_argmax", "projection_rows_argmax"])
def test_ring_fed_kernels_leave_together_when_their_waits_fail(kernel, cuda_device):
    """Behind a wait that has given up (made on the host side: a barrier that expects an arrival nobody makes) the status is
    still reported and nothing is stored; with the workspace initialised again the same call gives the operator's result."""
    import ctypes

    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import cabi, synthetic as syn

    lib, dev = cabi.load(), cuda_device
    nbytes = lib.mk36_workspace_bytes()
    ws = torch.empty(nbytes, dtype=torch.uint8, device=dev)
    stream = torch.cuda.current_stream().cuda_stream
    status = ctypes.c_int(-1)
    best = expect_best = None
    if kernel == "dense_tiles":
        t = {k: v.to(dev) for k, v in syn.dense_tensors(syn.DenseShape(2400, 1216), 5, seed=5).items()}
        out = torch.empty_like(t["x"])
        args = cabi.DenseFfnArgs(x=t["x"].data_ptr(), norm_weight=t["norm_weight"].data_ptr(), gate_weight=t["gate_weight"].data_ptr(),
                                 up_weight=t["up_weight"].data_ptr(), down_weight=t["down_weight"].data_ptr(), out=out.data_ptr(),
                                 partial_out=None, dtype=cabi.MK36_BF16, batch=5, hidden=2400, intermediate=1216, add_residual=1, eps=1e-6)
        call = lambda: lib.mk36_dense_ffn_decode(args, ws.data_ptr(), nbytes, stream)
        expect = mk.dense_ffn_decode(t["x"], mk.DenseFfnWeights(*[t[f] for f in syn.DENSE_WEIGHT_FIELDS]))
    else:  # 2304 = a whole stage of columns and a narrower one
        batch, argmax = (2 if "rows" in kernel else 4), "argmax" in kernel
        t = {k: v.to(dev) for k, v in syn.projection_tensors(2304, 5000, batch, seed=9, norm=True, residual=True).items()}
        out = torch.empty(batch, 5000, dtype=torch.bfloat16, device=dev)
        best = torch.empty(batch, dtype=torch.int64, device=dev) if argmax else None
        args = cabi.LinearArgs(x=t["x"].data_ptr(), norm_weight=t["norm_weight"].data_ptr(), weight=t["weight"].data_ptr(),
                               residual=t["residual"].data_ptr(), out=out.data_ptr(), argmax=best.data_ptr() if argmax else None,
                               dtype=cabi.MK36_BF16, batch=batch, in_features=2304, out_features=5000, eps=1e-6)
        call = lambda: lib.mk36_linear_decode(args, ws.data_ptr(), nbytes, stream)
        expect, expect_best = mk.linear_decode(t["x"], t["weight"], norm_weight=t["norm_weight"], residual=t["residual"], return_argmax=True)
    for spoilt in (True, False):
        cabi.check(lib.mk36_workspace_init(ws.data_ptr(), nbytes, stream))
        out.fill_(5.0)
        if best is not None:
            best.fill_(-7)
        if spoilt:
            cabi.check(lib.mk36_selftest_bounded_wait(ws.data_ptr(), nbytes, stream, 20))
        cabi.check(call())
        rc = lib.mk36_workspace_status(ws.data_ptr(), stream, ctypes.byref(status))
        if spoilt:
            assert rc == cabi.MK36_ERR_BARRIER_TIMEOUT and status.value == 901
            assert bool((out == 5.0).all()) and (best is None or bool((best == -7).all()))
        else:
            assert rc == 0 and status.value == 0
            assert torch.equal(out, expect) and (best is None or torch.equal(best, expect_best))


@pytest.mark.parametrize("shape,dtype", [((1, 4, 2, 128, 16), torch.bfloat16), ((1, 4, 2, 128, 16 * 33), torch.float16), ((1, 16, 2, 256, 16 * 64), torch.bfloat16),
                                         ((1, 4, 2, 128, 16 * 64 + 1), torch.bfloat16), ((5, 16, 2, 256, 611), torch.float16), ((4, 8, 2, 64, 300), torch.bfloat16)])
def test_attention_merges_at_the_split_counts_where_they_change(shape, dtype, cuda_device):
    """One split, 33 (a second round of the channel-wise merge), 64 (its last) and 65 (the merge over lanes); several batch
    items; head_dim 64, which the channel-wise merge does not take."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import synthetic as syn
    from oracle import decode_oracle as oracle

    t = syn.attention_tensors(*shape, seed=shape[4], dtype=dtype)
    got = mk.full_attention_decode(mk.FullAttentionInputs(*(t[n].to(cuda_device) for n in ("q", "k_cache", "v_cache")))).cpu()
    assert_output_parity(got, oracle.full_attention_decode(t["q"], t["k_cache"], t["v_cache"]), what=f"merge {shape}")


def _exactly_normalised(batch, hidden, dtype, gen, device):
    """x of +-1 and a norm weight: with eps 0 the normalised token is x * weight without any rounding."""
    x = (torch.randint(0, 2, (batch, hidden), generator=gen) * 2 - 1).to(dtype).to(device)
    return x, (torch.randn(hidden, generator=gen) * 0.6 + 1.0).to(dtype).to(device)


def _error(got, exact):
    return float((got.double() - exact).norm() / exact.norm())


@pytest.mark.parametrize("batch,intermediate,dtype", [(2, 2176, torch.float16), (8, 2176, torch.float16), (8, 2176, torch.bfloat16), (3, 4352, torch.bfloat16)],
                         ids=lambda v: str(v).replace("torch.", ""))
def test_dense_tiles_are_no_further_from_the_exact_sum_than_the_register_staged_kernel(batch, intermediate, dtype, cuda_device):
    """fp32 partial outputs of both kernels against 64-bit sums of the same inputs."""
    from mega_kernel_qwen36 import cabi, ops

    gen = torch.Generator().manual_seed(intermediate + batch)
    hidden = 5120
    x, norm = _exactly_normalised(batch, hidden, dtype, gen, cuda_device)
    gate, up, down = ((torch.randn(*s, generator=gen) * 0.02).to(dtype).to(cuda_device) for s in ((intermediate, hidden), (intermediate, hidden), (hidden, intermediate)))
    n = (x * norm).double()
    exact = (torch.nn.functional.silu(n @ gate.double().T) * (n @ up.double().T)) @ down.double().T
    errors = {}
    for tiles in (0, 1):
        cabi.check(cabi.load().mk36_set_option(b"dense_tiles", tiles))
        try:
            errors[tiles] = _error(ops._C.dense_ffn_decode_partial(x, norm, gate, up, down, 0.0), exact)
        finally:
            cabi.check(cabi.load().mk36_set_option(b"dense_tiles", 1))
    assert errors[1] <= errors[0], errors


@pytest.mark.parametrize("batch", [9, 32])
def test_moe_wide_kernel_is_as_close_to_the_exact_sum_as_the_batch_kernel(batch, cuda_device):
    """fp32 partial outputs of both kernels against 64-bit sums of the same inputs.  The two add in different orders, so
    that the ratio of their errors scatters by a few percent with the inputs (0.96 to 1.04 over 9 to 32 tokens): 1.1."""
    from mega_kernel_qwen36 import cabi, ops

    hidden, experts, k, width = 2048, 256, 8, 512
    gen = torch.Generator(device=cuda_device).manual_seed(batch)
    weight = lambda *s: (torch.randn(*s, generator=gen, device=cuda_device) * 0.02).bfloat16()
    router, gate, up, down = weight(experts, hidden), weight(experts, width, hidden), weight(experts, width, hidden), weight(experts, hidden, width)
    sgate, sup, sdown = weight(width, hidden), weight(width, hidden), weight(hidden, width)
    x, norm = _exactly_normalised(batch, hidden, torch.bfloat16, torch.Generator().manual_seed(batch), cuda_device)
    got = {}
    for wide in (0, 9):
        cabi.check(cabi.load().mk36_set_option(b"moe_wide", wide))
        try:
            got[wide], idx, _ = ops._C.moe_decode_partial(x, norm, router, gate, up, down, sgate, sup, sdown, 0.0, k, 0)
        finally:
            cabi.check(cabi.load().mk36_set_option(b"moe_wide", 9))
    n = (x * norm).double()
    silu = torch.nn.functional.silu
    mix = torch.softmax((n @ router.double().T).gather(1, idx), -1)
    exact = (silu(n @ sgate.double().T) * (n @ sup.double().T)) @ sdown.double().T
    for b in range(batch):
        for slot, e in enumerate(idx[b].tolist()):
            exact[b] += mix[b, slot] * ((silu(n[b] @ gate[e].double().T) * (n[b] @ up[e].double().T)) @ down[e].double().T)
    assert _error(got[9], exact) <= 1.1 * _error(got[0], exact)


def test_moe_wide_kernel_keeps_infinite_weights(cuda_device):
    """One infinite down weight in every other output row, at another channel in each: the output is an infinity of the
    activation's sign, as the batch kernel's is, also where a term that the activation is split into is zero."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import cabi, synthetic as syn

    t = {k: v.to(cuda_device) for k, v in syn.moe_tensors(syn.MOE_35B_A3B, 32, 3, torch.bfloat16).items()}
    rows = torch.arange(0, t["shared_down"].shape[0], 2, device=cuda_device)
    t["shared_down"][rows, (rows * 7) % t["shared_down"].shape[1]] = float("inf")
    weights = mk.MoeWeights(*[t[f] for f in syn.MOE_WEIGHT_FIELDS])
    got = mk.moe_decode(t["x"], weights)[0].float()
    cabi.check(cabi.load().mk36_set_option(b"moe_wide", 0))
    try:
        want = mk.moe_decode(t["x"], weights)[0].float()
    finally:
        cabi.check(cabi.load().mk36_set_option(b"moe_wide", 9))
    assert bool(want[:, rows].isinf().all())
    assert torch.equal(got[:, rows], want[:, rows])
    assert_output_parity(got[:, 1::2].cpu(), want[:, 1::2].cpu(), what="rows without an infinite weight")


def _graph_nodes(call):
    """How many nodes a call leaves in a CUDA graph: its launches."""
    import ctypes

    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        call()
    count = ctypes.c_size_t()
    assert ctypes.CDLL("libcudart.so.12").cudaGraphGetNodes(ctypes.c_void_p(graph.raw_cuda_graph()), None, ctypes.byref(count)) == 0
    return count.value


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16, torch.float32], ids=["bf16", "f16", "f32"])
@pytest.mark.parametrize("key_dim,value_dim,steps,offset", [(6, 8, 3, 0), (126, 36, 5, 0), (130, 32, 4, 1), (128, 128, 6, 1), (36, 20, 9, 3), (256, 32, 2, 1), (64, 64, 5, 2)])
def test_linear_attention_steps_keep_the_state_on_chip_for_odd_and_unaligned_inputs(key_dim, value_dim, steps, offset, dtype, cuda_device):
    """Key dimensions that are no multiple of four, and q, k, v that start `offset` elements off an aligned address: one
    launch for all steps, the state bit-equal to the oracle's, the outputs to those of one-step calls on aligned tensors."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import synthetic as syn
    from oracle import decode_oracle as oracle

    B, HK, HV = 2, 2, 4
    stream = list(syn.linear_step_stream(B, HK, HV, key_dim, value_dim, steps=steps, seed=key_dim + steps, dtype=dtype))

    def shifted(name):
        t = torch.stack([s[name] for s in stream])
        buf = torch.zeros(t.numel() + 8, dtype=dtype, device=cuda_device)
        buf[offset:offset + t.numel()] = t.flatten().to(cuda_device)
        return buf[offset:offset + t.numel()].view(t.shape)

    q, k, v = (shifted(n) for n in ("q", "k", "v"))
    g, beta = (torch.stack([s[n] for s in stream]).to(cuda_device) for n in ("g", "beta"))
    s_ref = syn.linear_state(B, HV, key_dim, value_dim, seed=3)
    state = s_ref.to(cuda_device)
    run = lambda: mk.linear_attention_decode_steps(q, k, v, state, decay_per_step=g, beta_per_step=beta)
    outs, final = run()
    s_one = state
    for i, step in enumerate(stream):
        o_ref, s_ref = oracle.linear_attention_decode_per_head(step["q"], step["k"], step["v"], s_ref, step["g"], step["beta"])
        o_one, s_one = mk.linear_attention_decode_gated(q[i].clone(), k[i].clone(), v[i].clone(), s_one, decay_per_head=g[i], beta_per_head=beta[i])
        o_off, _ = mk.linear_attention_decode_gated(q[i], k[i], v[i], state if i == 0 else s_prev, decay_per_head=g[i], beta_per_head=beta[i])
        s_prev = s_one
        assert torch.equal(s_one.cpu(), s_ref)
        assert torch.equal(outs[i], o_one) and torch.equal(o_off, o_one)
        assert_output_parity(outs[i].cpu(), o_ref, what=f"steps {key_dim}x{value_dim}+{offset} out {i}")
    assert torch.equal(final, s_one)
    assert _graph_nodes(run) == 1


@pytest.mark.parametrize("tiles", [1, 0], ids=["tiles", "register_staged"])
@pytest.mark.parametrize("what", ["f16_activation_beyond_f16", "infinite_weight"])
def test_dense_tensor_core_kernels_where_a_split_activation_is_not_finite(what, tiles, cuda_device):
    """The activations are multiplied as a high and a low half.  One that f16 cannot hold must still give the oracle's finite
    output, and an infinite down weight an infinity of the activation's sign, as with one token, where nothing is split."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import cabi, synthetic as syn
    from oracle import decode_oracle as oracle

    dtype = torch.float16 if what.startswith("f16") else torch.bfloat16
    t = syn.dense_tensors(syn.DenseShape(2400, 1216), 1, 5, dtype)
    t["x"] = t["x"].repeat(5, 1).contiguous()
    rows = torch.arange(0, 2400, 2)
    if what.startswith("f16"):
        for name in ("gate_weight", "up_weight"):
            t[name][7] = (t["x"][0].float().sign() * 2.0).to(dtype)  # about 3800 each, 1.5e7 as a product
        t["down_weight"][:, 7] = (t["down_weight"][:, 7].float() * 1e-3).to(dtype)
    else:
        t["down_weight"][rows, (rows * 7) % 1216] = float("inf")
    d = {k: v.to(cuda_device) for k, v in t.items()}
    weights = mk.DenseFfnWeights(*[d[f] for f in syn.DENSE_WEIGHT_FIELDS])
    cabi.check(cabi.load().mk36_set_option(b"dense_tiles", tiles))
    try:
        got = mk.dense_ffn_decode(d["x"], weights).cpu()
    finally:
        cabi.check(cabi.load().mk36_set_option(b"dense_tiles", 1))
    want = oracle.dense_ffn_decode(t["x"], *[t[f] for f in syn.DENSE_WEIGHT_FIELDS])
    if not what.startswith("f16"):
        assert bool(want[:, rows].isinf().all()) and torch.equal(got[:, rows], want[:, rows])
        got, want = got[:, 1::2], want[:, 1::2]
    assert_output_parity(got, want, what=f"{what} tiles={tiles}")


@pytest.mark.parametrize("form", ["strided", "expanded", "row_of_three_dimensions", "float64_on_the_host", "scalar"])
def test_attention_block_takes_cos_and_sin_as_tensor_operations_do(form, cuda_device):
    """cos and sin that are views with strides, leading dimensions, another type or device, or scalars give what their plain
    form gives, and the caches' version counters move as with any in-place operation."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import synthetic as syn

    hq, hkv, d, B, H, rotary = 4, 2, 64, 2, 256, 32
    qkv = syn.projection_tensors(H, (hq + 2 * hkv) * d, B, seed=1, norm=True, residual=False)
    outp = syn.projection_tensors(hq * d, H, B, seed=2, norm=False, residual=False)
    ang = torch.arange(rotary // 2, dtype=torch.float32) * 0.3 + 0.2
    cos, sin = ang.cos().repeat(2).to(cuda_device), ang.sin().repeat(2).to(cuda_device)
    if form in ("expanded", "scalar"):
        cos, sin = torch.full_like(cos, 0.6), torch.full_like(sin, 0.8)
    change = {"strided": lambda t: torch.stack((t, -t), dim=1)[:, 0], "expanded": lambda t: t[:1].expand(rotary),
              "row_of_three_dimensions": lambda t: t.view(1, 1, rotary), "float64_on_the_host": lambda t: t.double().cpu(), "scalar": lambda t: t[0]}[form]

    def run(c, s):
        cache = {n: t.to(cuda_device) for n, t in syn.attention_tensors(B, hq, hkv, d, 20, seed=3).items()}
        block = mk.AttentionBlockInputs(qkv["norm_weight"].to(cuda_device), qkv["weight"].to(cuda_device), outp["weight"].to(cuda_device), cache["k_cache"],
                                        cache["v_cache"], 11, hq, hkv, d, cos=c, sin=s, rotary_dim=rotary)
        before = cache["k_cache"]._version, cache["v_cache"]._version
        out, attn = mk.attention_block_decode(qkv["x"].to(cuda_device), block)
        assert cache["k_cache"]._version > before[0] and cache["v_cache"]._version > before[1]
        return out, attn, cache["k_cache"]

    for got, want in zip(run(change(cos), change(sin)), run(cos, sin)):
        assert_output_parity(got.cpu(), want.cpu(), what=f"cos and sin {form}")


@pytest.mark.parametrize("shape,batch", [((1024, 24, 4, 256, 512), 9), ((1024, 40, 8, 512, 0), 12), ((2048, 8, 1, 256, 256), 32)])
def test_moe_wide_kernel_at_other_shapes(shape, batch, cuda_device):
    """Hidden 1024, fewer experts than CTAs, top 4 and top 1 (every expert has several entries), a shared expert of another
    width than the routed ones, and none."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import mpk_graph, synthetic as syn
    from oracle import decode_oracle as oracle

    assert mpk_graph.moe_wide_kernel_fits(*shape)
    t = syn.moe_tensors(syn.MoeShape(*shape), batch, 60 + batch, torch.bfloat16)
    out, idx, w = mk.moe_decode(t["x"].to(cuda_device), mk.MoeWeights(*[t[f].to(cuda_device) for f in syn.MOE_WEIGHT_FIELDS]), top_k=shape[2])
    want, want_idx, want_w = oracle.moe_decode(t["x"], *[t[f] for f in syn.MOE_WEIGHT_FIELDS], top_k=shape[2])
    assert torch.equal(idx.cpu(), want_idx)
    torch.testing.assert_close(w.cpu(), want_w, atol=1e-5, rtol=1e-4)
    assert_output_parity(out.cpu(), want, what=f"wide {shape} b{batch}")


def test_moe_wide_kernel_on_slices_of_the_experts(cuda_device):
    """The fp32 partials of two expert-parallel slices add up to the whole layer."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import ops, parallel, synthetic as syn
    from oracle import decode_oracle as oracle

    t = syn.moe_tensors(syn.MoeShape(2048, 64, 8, 512, 512), 17, 6, torch.bfloat16)
    full = mk.MoeWeights(*[t[f].to(cuda_device) for f in syn.MOE_WEIGHT_FIELDS])
    x, total = t["x"].to(cuda_device), 0.0
    for rank in range(2):
        shard = parallel.shard_moe_weights(full, rank, 2)
        part, idx, _ = ops._C.moe_decode_partial(x, *[getattr(shard.weights, f) for f in syn.MOE_WEIGHT_FIELDS], 1e-6, 8, shard.expert_base)
        total = total + part
    want, want_idx, _ = oracle.moe_decode(t["x"], *[t[f] for f in syn.MOE_WEIGHT_FIELDS], top_k=8)
    assert torch.equal(idx.cpu(), want_idx)
    assert_output_parity((total + x.float()).bfloat16().cpu(), want, what="wide, two expert slices")


@pytest.mark.parametrize("batch,n_in,n_out,dtype", [(3, 2304, 5000, torch.bfloat16), (8, 5376, 700, torch.float16), (4, 256, 3, torch.bfloat16)],
                         ids=lambda v: str(v).replace("torch.", ""))
def test_projection_tiles_with_a_narrower_last_stage(batch, n_in, n_out, dtype, cuda_device):
    """Inner dimensions that are no multiple of a stage's columns, and fewer rows than CTAs."""
    import mega_kernel_qwen36 as mk
    from mega_kernel_qwen36 import synthetic as syn
    from oracle import decode_oracle as oracle

    t = syn.projection_tensors(n_in, n_out, batch, seed=n_in, dtype=dtype, norm=True, residual=True)
    d = {k: v.to(cuda_device) for k, v in t.items()}
    got = mk.linear_decode(d["x"], d["weight"], norm_weight=d["norm_weight"], residual=d["residual"]).cpu()
    want = oracle.linear_decode(t["x"], t["weight"], norm_weight=t["norm_weight"], residual=t["residual"])
    assert_output_parity(got, want, what=f"projection {n_in}->{n_out}")
