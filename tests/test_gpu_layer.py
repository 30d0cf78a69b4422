"""Whole-block parity on the GPU, through the C ABI, against the CPU oracle."""
import ctypes as C

import numpy as np
import pytest

import refcases as rc
from ffai_b200 import capi, synth
from ffai_b200.moe import MoELayer
from helpers import assert_parity, from_dev, parity, to_dev

pytestmark = pytest.mark.gpu


def run_and_check(oracle_mod, spec, T, seed=0, residual=False, max_tokens=None, layer=None, host=None,
                  token_mask=None, rel_rms_tol=5e-3, max_abs_norm_tol=2e-2, path=None, options=None):
    host = host or synth.make_layer(spec, seed)
    x = synth.make_tokens(T, spec.hidden, seed)
    res = synth.make_tokens(T, spec.hidden, seed + 17) if residual else None
    own = layer is None
    layer = layer or MoELayer(host, max_tokens or T)
    try:
        if path is not None:
            layer.set_option("path", path)
        for name, value in (options or {}).items():
            layer.set_option(name, value)
        out, dbg = layer.forward_host(x, residual=res, debug=True)
    finally:
        if own:
            layer.close()
    ref = oracle_mod.moe_forward(host, x, residual=res, token_mask=token_mask)
    # routing: bit-exact
    assert np.array_equal(dbg.logits, ref.logits), "router logits differ"
    assert np.array_equal(dbg.indices, ref.indices), "expert indices differ"
    assert np.array_equal(dbg.weights, ref.weights), "combine weights differ"
    assert np.array_equal(dbg.counts, ref.counts)
    assert np.array_equal(dbg.offsets, ref.offsets)
    assert np.array_equal(dbg.perm, ref.perm)
    assert np.array_equal(dbg.inv_perm, ref.inv_perm)
    if token_mask is not None:
        sel = np.nonzero(token_mask)[0]
        return assert_parity(out[sel], ref.out_f32[sel], rel_rms_tol, max_abs_norm_tol, what=spec.name)
    return assert_parity(out, ref.out_f32, rel_rms_tol, max_abs_norm_tol, what=spec.name)


def test_cfg1_tiny_layer(oracle_mod):
    run_and_check(oracle_mod, synth.cfg1_tiny(), 16)


@pytest.mark.parametrize("T", [1, 8, 32, 64])
def test_cfg2_gptoss_decode_batches(oracle_mod, T):
    run_and_check(oracle_mod, synth.cfg2_gptoss(), T)


def test_cfg2_with_expert_row_biases_and_residual(oracle_mod):
    run_and_check(oracle_mod, synth.cfg2_gptoss().with_(expert_row_bias=1), 5, residual=True)


def test_cfg3_qwen_small_prefill(oracle_mod):
    run_and_check(oracle_mod, synth.cfg3_qwen(), 96)


def test_cfg3_single_token(oracle_mod):
    run_and_check(oracle_mod, synth.cfg3_qwen(), 1)


def test_cfg4_shared_expert_small(oracle_mod):
    run_and_check(oracle_mod, synth.cfg4_shared(), 48)


def test_shared_expert_without_gate(oracle_mod):
    spec = synth.cfg1_tiny().with_(name="granite_style", shared_intermediate=256, shared_bits=4, shared_group_size=64)
    run_and_check(oracle_mod, spec, 7)


@pytest.mark.parametrize("bits", [3, 5, 6, 8])
def test_odd_bit_widths(oracle_mod, bits):
    spec = synth.LayerSpec(f"bits{bits}", 512, 256, 16, 4, expert_bits=bits)
    run_and_check(oracle_mod, spec, 40)


@pytest.mark.parametrize("gs", [32, 128])
def test_group_sizes(oracle_mod, gs):
    spec = synth.LayerSpec(f"gs{gs}", 512, 256, 8, 2, expert_group_size=gs)
    run_and_check(oracle_mod, spec, 9)


def test_softmax_without_renormalisation_and_expert_bias(oracle_mod):
    spec = synth.LayerSpec("raw_softmax", 256, 128, 16, 4, norm_topk_prob=0)
    run_and_check(oracle_mod, spec, 33)
    spec = synth.LayerSpec("lfm2_bias", 256, 128, 16, 4, router_expert_bias=1)
    run_and_check(oracle_mod, spec, 33)


def test_gelu_glu_activation(oracle_mod):
    spec = synth.LayerSpec("gelu", 256, 128, 8, 2, activation=capi.ACT_GELU_GLU, gating_mode=capi.GATING_TOPK_THEN_SOFTMAX)
    run_and_check(oracle_mod, spec, 12)


def test_skewed_routing_layer(oracle_mod):
    spec = synth.LayerSpec("skew", 512, 256, 64, 8, router_has_bias=1, zipf_s=1.1, zipf_strength=1.5)
    p = run_and_check(oracle_mod, spec, 200)
    assert p["ref_rms"] > 0


def test_ragged_token_counts_on_one_handle(oracle_mod):
    """One handle, many batch sizes (empty, 1, odd, max): no state leaks between calls."""
    spec = synth.LayerSpec("ragged", 256, 128, 8, 2)
    host = synth.make_layer(spec, 3)
    layer = MoELayer(host, 70)
    try:
        out, _ = layer.forward_host(np.zeros((0, spec.hidden), dtype=np.uint16))
        assert out.shape == (0, spec.hidden)
        for T in (70, 1, 13, 64, 2, 70):
            run_and_check(oracle_mod, spec, T, seed=T, layer=layer, host=host)
        with pytest.raises(capi.FFAICudaError) as ei:
            layer.forward_host(np.zeros((71, spec.hidden), dtype=np.uint16))
        assert ei.value.status == capi.FFAI_ERR_INVALID_ARG
    finally:
        layer.close()


def test_all_tokens_to_the_same_experts(oracle_mod):
    """Collision extreme: identical rows route every token to the same k experts."""
    spec = synth.LayerSpec("collide", 256, 128, 8, 2)
    host = synth.make_layer(spec, 4)
    x = np.repeat(synth.make_tokens(1, spec.hidden, 4), 50, axis=0)
    ref = oracle_mod.moe_forward(host, x)
    layer = MoELayer(host, 50)
    try:
        # path 1: CUDA-core GEMV (fp32 throughout).  path 2: tcgen05 GEMM, which rounds the
        # dequantised weights and the intermediate to bf16; on this single repeated row the output
        # is small against its intermediates (ref RMS 0.4), so that rounding shows: 2e-2 / 5e-2 there.
        for path, rel_tol, abs_tol in ((1, 5e-3, 2e-2), (2, 2e-2, 5e-2)):
            layer.set_option("path", path)
            out, dbg = layer.forward_host(x, debug=True)
            assert np.array_equal(dbg.indices, ref.indices) and np.array_equal(dbg.perm, ref.perm)
            assert (dbg.counts > 0).sum() == 2
            assert_parity(out, ref.out_f32, rel_tol, abs_tol, what=f"path {path}")
            assert np.all(out == out[0])  # identical rows give identical outputs: the reduction order is fixed
    finally:
        layer.close()


@pytest.mark.parametrize("with_shared", [False, True])
def test_reference_four_expert_layer(oracle_mod, with_shared):
    """MoELayerTests.swift:150-265 through the C ABI."""
    arrays, x, expected = rc.four_expert_layer(with_shared)
    spec = synth.LayerSpec("four_expert", 64, 64, 4, 2, router_kind=capi.LINEAR_F32, router_logits_bf16=0,
                           shared_intermediate=64 if with_shared else 0, shared_bits=4, shared_group_size=64)
    host = synth.HostLayer(spec, arrays)
    layer = MoELayer(host, 1)
    try:
        out, dbg = layer.forward_host(synth.f32_to_bf16(x)[None, :], debug=True)
    finally:
        layer.close()
    assert dbg.indices[0].tolist() == [1, 2]
    assert np.allclose(dbg.weights[0], [0.73107, 0.26893], atol=1e-4)
    got = float(synth.bf16_to_f32(out)[0, 0])
    assert abs(got - expected) <= abs(expected) * 2.0 ** -8 + 1e-3


def test_device_pointer_forward_matches_host_forward(oracle_mod):
    import torch
    spec = synth.cfg1_tiny()
    host = synth.make_layer(spec, 0)
    x = synth.make_tokens(16, spec.hidden, 0)
    layer = MoELayer(host, 16)
    try:
        out_h, _ = layer.forward_host(x)
        dx = to_dev(x)
        dout = torch.zeros(16 * spec.hidden, dtype=torch.int16, device="cuda")
        st = torch.cuda.Stream()
        with torch.cuda.stream(st):
            layer.forward_ptr(dx.data_ptr(), 16, dout.data_ptr(), stream=st.cuda_stream)
        st.synchronize()
        assert layer.launch_count() > 0
        assert np.array_equal(from_dev(dout, np.uint16).reshape(16, -1), out_h)
    finally:
        layer.close()


def test_forward_is_deterministic(oracle_mod):
    spec = synth.cfg2_gptoss()
    host = synth.make_layer(spec, 0)
    x = synth.make_tokens(32, spec.hidden, 0)
    layer = MoELayer(host, 32)
    try:
        a, _ = layer.forward_host(x)
        b, _ = layer.forward_host(x)
    finally:
        layer.close()
    assert np.array_equal(a, b)


def test_cfg3_full_prefill_sampled_tokens(oracle_mod):
    """Full 2048-token prefill: routing checked for every token, outputs for a token sample."""
    spec = synth.cfg3_qwen()
    mask = np.zeros(2048, dtype=np.uint8)
    mask[np.random.default_rng(0).choice(2048, size=64, replace=False)] = 1
    run_and_check(oracle_mod, spec, 2048, token_mask=mask)


# ── the tcgen05 grouped-GEMM path (forced), same oracle, same tolerances ──

TC = 2  # option "path": tensor-core grouped GEMM whenever possible


@pytest.mark.parametrize("T", [1, 16, 17, 300])
def test_tc_cfg1_shape(oracle_mod, T):
    run_and_check(oracle_mod, synth.cfg1_tiny(), T, path=TC)


@pytest.mark.parametrize("T", [8, 64])
def test_tc_cfg2_decode(oracle_mod, T):
    run_and_check(oracle_mod, synth.cfg2_gptoss(), T, path=TC)


def test_tc_cfg2_row_bias_residual(oracle_mod):
    run_and_check(oracle_mod, synth.cfg2_gptoss().with_(expert_row_bias=1), 40, residual=True, path=TC)


def test_tc_cfg3_small(oracle_mod):
    run_and_check(oracle_mod, synth.cfg3_qwen(), 200, path=TC)


def test_tc_cfg3_full_prefill_sampled(oracle_mod):
    mask = np.zeros(2048, dtype=np.uint8)
    mask[np.random.default_rng(1).choice(2048, size=64, replace=False)] = 1
    run_and_check(oracle_mod, synth.cfg3_qwen(), 2048, token_mask=mask, path=TC)


@pytest.mark.parametrize("tc_weights", [1, 2])
def test_tc_cfg3_full_prefill_one_weight_source(oracle_mod, tc_weights):
    """The same prefill with both grouped GEMMs dequantising the packed weights themselves (1) or both reading
    the bf16 weight cache (2); the automatic choice at this size is packed gate/up and cached down."""
    mask = np.zeros(2048, dtype=np.uint8)
    mask[np.random.default_rng(2).choice(2048, size=64, replace=False)] = 1
    run_and_check(oracle_mod, synth.cfg3_qwen(), 2048, token_mask=mask, path=TC, options={"tc_weights": tc_weights})


@pytest.mark.parametrize("bits", [3, 4, 5, 6, 8])
def test_tc_bf16_weight_cache_any_bit_width(oracle_mod, bits):
    """With the cache the tensor-core path takes every bit width: the experts are expanded once."""
    spec = synth.LayerSpec(f"cache_bits{bits}", 512, 256, 16, 4, expert_bits=bits, prefill_weight_cache=2)
    run_and_check(oracle_mod, spec, 300, path=TC)
    run_and_check(oracle_mod, spec, 300)          # automatic choice


def test_tc_weight_cache_with_ragged_row_blocks(oracle_mod):
    """2880 output rows are 22.5 blocks of 128: the tile-major cache pads the last block of gate/up with zero
    rows and gives down an even block count; both weight sources must still give the same bits."""
    spec = synth.cfg2_gptoss().with_(prefill_weight_cache=2, expert_row_bias=1)
    host = synth.make_layer(spec, 9)
    x = synth.make_tokens(600, spec.hidden, 9)
    layer = MoELayer(host, 600)
    try:
        layer.set_option("path", TC)
        layer.set_option("tc_weights", 2)
        cached, _ = layer.forward_host(x)
        layer.set_option("tc_weights", 1)
        packed, _ = layer.forward_host(x)
    finally:
        layer.close()
    assert np.array_equal(cached, packed)
    run_and_check(oracle_mod, spec, 600, seed=9, host=host, path=TC, options={"tc_weights": 2})


def test_tc_cache_and_packed_weights_agree(oracle_mod):
    spec = synth.LayerSpec("cache_vs_packed", 512, 256, 16, 4, prefill_weight_cache=2)
    host = synth.make_layer(spec, 3)
    x = synth.make_tokens(500, spec.hidden, 3)          # 125 rows per expert: between the limits of down (112) and gate/up (136)
    layer = MoELayer(host, 500)
    try:
        layer.set_option("path", TC)
        layer.set_option("tc_weights", 2)
        a, _ = layer.forward_host(x)
        layer.set_option("tc_weights", 1)
        b, _ = layer.forward_host(x)
        layer.set_option("tc_weights", 0)   # automatic: packed gate/up, cached down at this size
        c, _ = layer.forward_host(x)
    finally:
        layer.close()
    # both round fma(q, scale, bias) to bf16 once and run the same MMA sequence
    assert np.array_equal(a, b)
    assert np.array_equal(a, c)


def test_host_entry_in_chunks_gives_the_same_bits(oracle_mod):
    """A large batch through the host entry point is cut into chunks whose copies overlap the compute; tokens
    are independent, so the output equals the uncut call bit for bit (with a residual and the router's own rows
    too), and a sample of tokens agrees with the oracle."""
    spec = synth.LayerSpec("host_chunks", 512, 256, 16, 4, prefill_weight_cache=2)
    host = synth.make_layer(spec, 5)
    T = 4608 + 77                      # two chunks, the second one ragged
    x = synth.make_tokens(T, spec.hidden, 5)
    res = synth.make_tokens(T, spec.hidden, 6)
    layer = MoELayer(host, T)
    try:
        cut, _ = layer.forward_host(x, residual=res)
        cut_split, _ = layer.forward_host(x, residual=res, x_router=x)
        layer.set_option("host_chunks", 1)
        whole, _ = layer.forward_host(x, residual=res)
    finally:
        layer.close()
    assert np.array_equal(cut, whole)
    assert np.array_equal(cut_split, whole)
    mask = np.zeros(T, dtype=np.uint8)
    mask[np.random.default_rng(3).choice(T, size=48, replace=False)] = 1
    ref = oracle_mod.moe_forward(host, x, residual=res, token_mask=mask)
    sel = np.nonzero(mask)[0]
    assert_parity(cut[sel], ref.out_f32[sel], 5e-3, 2e-2, what=spec.name)


@pytest.mark.parametrize("gs", [32, 128])
def test_tc_group_sizes(oracle_mod, gs):
    run_and_check(oracle_mod, synth.LayerSpec(f"tc_gs{gs}", 512, 256, 8, 2, expert_group_size=gs), 150, path=TC)


def test_tc_skewed_many_token_tiles(oracle_mod):
    """One hot expert receives several 128-row token tiles; cold experts receive none."""
    spec = synth.LayerSpec("tc_skew", 512, 256, 64, 8, router_has_bias=1, zipf_s=1.1, zipf_strength=2.0)
    run_and_check(oracle_mod, spec, 700, path=TC)


def test_tc_shared_expert_4bit(oracle_mod):
    spec = synth.LayerSpec("tc_shared", 512, 256, 16, 4, shared_intermediate=256, shared_bits=4, shared_group_size=64,
                           shared_gate_kind=capi.LINEAR_BF16)
    run_and_check(oracle_mod, spec, 130, path=TC)
    run_and_check(oracle_mod, spec, 9, path=TC)


def test_tc_and_gemv_paths_agree_on_routing_and_nearly_on_values(oracle_mod):
    spec = synth.cfg3_qwen()
    host = synth.make_layer(spec, 0)
    x = synth.make_tokens(64, spec.hidden, 0)
    layer = MoELayer(host, 64)
    try:
        layer.set_option("path", 1)
        a, da = layer.forward_host(x, debug=True)
        layer.set_option("path", 2)
        b, db = layer.forward_host(x, debug=True)
        c, _ = layer.forward_host(x)
    finally:
        layer.close()
    assert np.array_equal(da.indices, db.indices) and np.array_equal(da.perm, db.perm)
    assert np.array_equal(b, c)                       # the tensor-core path is deterministic too
    fa, fb = synth.bf16_to_f32(a).astype(np.float64), synth.bf16_to_f32(b).astype(np.float64)
    assert np.sqrt(((fa - fb) ** 2).mean()) / np.sqrt((fa ** 2).mean()) < 5e-3


# ── the register-streaming decode kernels (forced), same oracle, same tolerances ──

MMA = 3  # option "path": per-warp streaming mma.sync kernels


@pytest.mark.parametrize("T", [1, 2, 8, 9, 32, 64])
def test_mma_cfg2_decode(oracle_mod, T):
    run_and_check(oracle_mod, synth.cfg2_gptoss(), T, path=MMA)


def test_mma_cfg2_row_bias_residual(oracle_mod):
    run_and_check(oracle_mod, synth.cfg2_gptoss().with_(expert_row_bias=1), 21, residual=True, path=MMA)


@pytest.mark.parametrize("T", [1, 16, 40])
def test_mma_cfg1_and_cfg3_shapes(oracle_mod, T):
    run_and_check(oracle_mod, synth.cfg1_tiny(), T, path=MMA)
    run_and_check(oracle_mod, synth.cfg3_qwen(), T, path=MMA)


def test_mma_group_size_128_and_many_rows_per_expert(oracle_mod):
    # 70 tokens over 8 experts: several passes of 8/16 activation rows per expert
    run_and_check(oracle_mod, synth.LayerSpec("mma_gs128", 512, 256, 8, 2, expert_group_size=128), 70, path=MMA)
    run_and_check(oracle_mod, synth.LayerSpec("mma_small", 64, 64, 4, 2), 5, path=MMA)


@pytest.mark.parametrize("T", [1, 4, 8, 20, 64])
def test_mma_group_size_32_gptoss_as_transcoded(oracle_mod, T):
    """GPT-OSS experts as the MXFP4 transcode leaves them: 4-bit, group 32, row biases; both pass widths."""
    spec = synth.cfg2_gptoss().with_(name="gptoss_gs32", expert_group_size=32, expert_row_bias=1)
    run_and_check(oracle_mod, spec, T, path=MMA)
    run_and_check(oracle_mod, spec, T)                      # the automatic choice: the same kernels from 9 tokens on


def test_mma_group_size_32_small_shapes(oracle_mod):
    run_and_check(oracle_mod, synth.LayerSpec("mma_gs32", 512, 256, 8, 2, expert_group_size=32), 70, path=MMA)
    run_and_check(oracle_mod, synth.LayerSpec("mma_gs32_small", 64, 64, 4, 2, expert_group_size=32), 5, path=MMA)
    run_and_check(oracle_mod, synth.LayerSpec("mma_gs32_odd_runs", 320, 192, 4, 2, expert_group_size=32), 11, path=MMA)


@pytest.mark.parametrize("ksplit", [1, 2, 4])
@pytest.mark.parametrize("gs", [32, 64])
def test_mma_every_reduction_split(oracle_mod, ksplit, gs):
    """The reduction axis cut into 1, 2 or 4 slices per 16-row block (the automatic choice only splits the
    smallest batches), for both scale layouts, with one and with several rows per expert."""
    spec = synth.cfg2_gptoss().with_(name=f"split{ksplit}_gs{gs}", expert_group_size=gs)
    for T in (1, 3, 24):
        run_and_check(oracle_mod, spec, T, path=MMA, options={"ksplit": ksplit})


def test_auto_path_is_deterministic_and_matches_forced_paths(oracle_mod):
    spec = synth.cfg2_gptoss()
    host = synth.make_layer(spec, 0)
    x = synth.make_tokens(9, spec.hidden, 0)
    layer = MoELayer(host, 9)
    try:
        a, _ = layer.forward_host(x)
        b, _ = layer.forward_host(x)
        small, _ = layer.forward_host(x[:8])
        again, _ = layer.forward_host(x[:8])
        assert layer.launch_count() == 1
        layer.set_option("path", MMA)
        c, _ = layer.forward_host(x)
        forced, _ = layer.forward_host(x[:8])
        assert layer.launch_count() > 1
    finally:
        layer.close()
    assert np.array_equal(a, b) and np.array_equal(a, c)   # small batches take the streaming kernels
    assert np.array_equal(small, again)
    # the smallest ones the one-launch kernel: fp32 sums in another order, about 1e-5 of the RMS, which turn few bf16 roundings (of
    # the activation's results, one in 1000, and of the outputs), each by at most 2**-7 of a value
    fa, fb = synth.bf16_to_f32(small).astype(np.float64), synth.bf16_to_f32(forced).astype(np.float64)
    assert 0 < np.sqrt(((fa - fb) ** 2).mean()) / np.sqrt((fb ** 2).mean()) < 1e-3


@pytest.mark.parametrize("option", [("decode", 1), ("decode", 2), ("path", MMA), ("nt2_cost", 8), ("tc_min_rows", 64), ("decode_team", 4)])
def test_options_of_other_kernels_keep_them_for_the_smallest_batches(oracle_mod, option):
    spec = synth.LayerSpec("other_kernels", 512, 256, 16, 4)
    host = synth.make_layer(spec, 61)
    layer = MoELayer(host, 8)
    try:
        run_and_check(oracle_mod, spec, 8, layer=layer, host=host)
        assert layer.launch_count() == 1
        for T in (1, 3, 8):
            run_and_check(oracle_mod, spec, T, layer=layer, host=host, options=dict([option]))
            assert layer.launch_count() > 1
    finally:
        layer.close()


@pytest.mark.parametrize("gs", [32, 64])
@pytest.mark.parametrize("T", [6, 7])
def test_one_launch_ends_where_the_token_rows_do_not_fit(oracle_mod, gs, T):
    """Rows of 7168 take 16 KB of shared memory each: six fit beside the rest, the seventh does not."""
    spec = synth.LayerSpec("long_rows", 7168, 64, 8, 2, expert_group_size=gs)
    host = synth.make_layer(spec, 71)
    layer = MoELayer(host, 8)
    try:
        run_and_check(oracle_mod, spec, T, layer=layer, host=host)
        assert (layer.launch_count() == 1) == (T == 6)
    finally:
        layer.close()


# ── Gemma-4-style routing: scaled logits, per-expert combine scale, GELU-GLU, the router's own input ──

@pytest.mark.parametrize("T,path", [(1, None), (6, None), (40, None), (150, None), (300, 2), (9, 1)])
def test_gemma4_style_block(oracle_mod, T, path):
    spec = synth.gemma4_style()
    host = synth.make_layer(spec, 4)
    x = synth.make_tokens(T, spec.hidden, 4)
    xr = synth.make_tokens(T, spec.hidden, 40)          # stands for rmsNorm(h, router.scale)
    layer = MoELayer(host, T)
    try:
        if path is not None:
            layer.set_option("path", path)
        out, dbg = layer.forward_host(x, debug=True, x_router=xr)
        same, _ = layer.forward_host(x, x_router=xr)
        plain, pdbg = layer.forward_host(x, debug=True)           # router reading x: a different routing
    finally:
        layer.close()
    ref = oracle_mod.moe_forward(host, x, x_router=xr)
    assert np.array_equal(dbg.indices, ref.indices) and np.array_equal(dbg.weights, ref.weights)
    assert np.array_equal(dbg.perm, ref.perm) and np.array_equal(out, same)
    assert_parity(out, ref.out_f32, what=spec.name)
    ref_plain = oracle_mod.moe_forward(host, x)
    assert np.array_equal(pdbg.indices, ref_plain.indices) and np.array_equal(pdbg.weights, ref_plain.weights)
    # the per-expert scale really is in the weights: they no longer sum to one
    assert np.abs(ref.weights.sum(axis=1) - 1.0).max() > 1e-2


# ── the remaining benchmark configurations at their full sizes (outputs on a token sample: the oracle is scalar) ──

def test_cfg4_full_prefill_sampled(oracle_mod):
    """256 experts, top-8, sigmoid-gated 8-bit shared expert, 8-bit router, 2048 tokens: routing and
    the plan for every token, outputs for 48 sampled tokens."""
    mask = np.zeros(2048, dtype=np.uint8)
    mask[np.random.default_rng(4).choice(2048, size=48, replace=False)] = 1
    run_and_check(oracle_mod, synth.cfg4_shared(), 2048, token_mask=mask)


@pytest.mark.parametrize("bits", [3, 4, 5, 6, 8])
def test_cfg5_skewed_routing_every_bit_width(oracle_mod, bits):
    """cfg3 shape with a Zipf(1.1) router bias (a few hot experts with many token tiles, most experts
    nearly empty) at every bit width; 1024 tokens, outputs for 32 sampled tokens."""
    mask = np.zeros(1024, dtype=np.uint8)
    mask[np.random.default_rng(bits).choice(1024, size=32, replace=False)] = 1
    run_and_check(oracle_mod, synth.cfg5_skewed(bits), 1024, token_mask=mask)


def test_cfg4_at_its_full_size(oracle_mod):
    """The 256-expert configuration at its 8192 tokens (65536 routed rows: the dispatch plan takes its
    count / scan / scatter form): routing and plan for every token, outputs for 32 sampled tokens."""
    mask = np.zeros(8192, dtype=np.uint8)
    mask[np.random.default_rng(44).choice(8192, size=32, replace=False)] = 1
    run_and_check(oracle_mod, synth.cfg4_shared(), 8192, token_mask=mask)


def test_cfg5_at_its_full_size_with_requantized_experts(oracle_mod):
    """The skewed configuration as it is described: the 4-bit layer of the cfg3 shape, its experts
    re-quantised at another width (5 bits here) from their dequantised values, Zipf router bias, 16384
    tokens (131072 routed rows); routing and plan for every token, outputs for 32 sampled tokens."""
    base = synth.make_layer(synth.cfg5_skewed(4), 0)
    host = synth.requantize_experts(base, 5)
    assert host.spec.expert_bits == 5
    mask = np.zeros(16384, dtype=np.uint8)
    mask[np.random.default_rng(55).choice(16384, size=32, replace=False)] = 1
    run_and_check(oracle_mod, host.spec, 16384, host=host, token_mask=mask)


# ── NemotronH-style block: sigmoid routing with selection bias and scaling factor, experts without a gate projection ──

@pytest.mark.parametrize("T", [1, 7, 64, 300])
def test_nemotronh_style_block(oracle_mod, T):
    spec = synth.nemotronh_style()
    run_and_check(oracle_mod, spec, T, seed=6, residual=(T == 7))


def test_nemotronh_style_block_other_widths(oracle_mod):
    run_and_check(oracle_mod, synth.nemotronh_style().with_(name="nemotronh_8bit", expert_bits=8, shared_bits=8, norm_topk_prob=0), 33)
    run_and_check(oracle_mod, synth.nemotronh_style().with_(name="nemotronh_no_shared", shared_intermediate=0, top_k=1), 20)


# ── the one-launch forward of the smallest batches ──

FUSED = [
    # name, T, spec changes.  H = 64 / I = 64 (one cell, ranges with fewer cells than warps), H = 1280 (whole rounds of down
    # items), H = 4672 (292 items: two rounds or a split axis), 64 routed rows (most) and 72 (one more token-slot row than
    # fits: the launch chain), every code width and group the kernel takes, one expert, shared experts of both widths
    ("smallest", 1, dict(hidden=64, intermediate=64, n_experts=1, top_k=1)),
    ("one_cell", 8, dict(hidden=64, intermediate=64, n_experts=8, top_k=8)),
    ("full_rows", 8, dict(hidden=512, intermediate=192, n_experts=40, top_k=8)),
    ("too_many_rows", 8, dict(hidden=512, intermediate=192, n_experts=40, top_k=9)),
    ("nine_tokens", 9, dict(hidden=512, intermediate=192, n_experts=40, top_k=4)),
    ("split_down", 7, dict(hidden=4672, intermediate=704, n_experts=12, top_k=5, expert_row_bias=1)),
    ("wide_router", 3, dict(hidden=256, intermediate=128, n_experts=300, top_k=20)),
    ("g128", 5, dict(hidden=1280, intermediate=384, n_experts=16, top_k=4, expert_group_size=128, expert_row_bias=1)),
    ("g32", 6, dict(hidden=1280, intermediate=320, n_experts=16, top_k=4, expert_group_size=32, expert_row_bias=1)),
    ("b8_g32", 2, dict(hidden=512, intermediate=320, n_experts=16, top_k=4, expert_bits=8, expert_group_size=32)),
    ("b8_g64_shared4", 4, dict(hidden=512, intermediate=320, n_experts=16, top_k=4, expert_bits=8, shared_intermediate=128, shared_bits=4,
                               shared_group_size=64, shared_gate_kind=capi.LINEAR_BF16)),
    ("b4_g32_shared8", 8, dict(hidden=512, intermediate=320, n_experts=16, top_k=2, expert_group_size=32, shared_intermediate=384, shared_bits=8,
                               shared_group_size=128, shared_gate_kind=capi.LINEAR_F32)),
    ("shared_ungated", 1, dict(hidden=2048, intermediate=64, n_experts=16, top_k=1, shared_intermediate=64, shared_bits=8, shared_group_size=64)),
]


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("name,T,kw", FUSED, ids=[f[0] for f in FUSED])
def test_one_launch_decode(oracle_mod, name, T, kw, residual):
    spec = synth.LayerSpec(name, **kw)
    host = synth.make_layer(spec, 11)
    layer = MoELayer(host, 12)
    try:
        for seed in (1, 2):     # the barrier word and the tickets come back to their start
            run_and_check(oracle_mod, spec, T, seed=seed, residual=residual, layer=layer, host=host)
        fused = T <= 8 and T * spec.top_k <= 64
        assert (layer.launch_count() == 1) == fused
    finally:
        layer.close()


# ── the wide router projection (128 tokens x 128 experts per block): ragged last tiles both ways, one chunk and three ──

@pytest.mark.parametrize("kind", [capi.LINEAR_F32, capi.LINEAR_BF16])
@pytest.mark.parametrize("T,E,H", [(1201, 1000, 192), (4800, 193, 64), (2500, 1000, 64)])     # the last: an odd count of rounds, narrow tiles
def test_wide_router_tiles(oracle_mod, kind, T, E, H):
    spec = synth.LayerSpec("wide_router_tiles", hidden=H, intermediate=64, n_experts=E, top_k=2, router_kind=kind, router_has_bias=1)
    mask = np.zeros(T, dtype=np.uint8)
    mask[:: 97] = 1     # routing is compared for every token, outputs for a sample
    run_and_check(oracle_mod, spec, T, token_mask=mask)


# ── groups of 32 on the tensor-core path: the re-tiled scale words, two per 64-k block ──

@pytest.mark.parametrize("H,I,T", [(320, 256, 130), (2880, 448, 45)])   # 5 / 45 and 4 / 7 blocks of 64: a last packed box of one, three and four blocks
def test_tc_group32_packed_words(oracle_mod, H, I, T):
    spec = synth.LayerSpec("tc_group32", H, I, 6, 3, expert_group_size=32, expert_row_bias=1, prefill_weight_cache=2)
    host = synth.make_layer(spec, 5)
    x = synth.make_tokens(T, H, 5)
    layer = MoELayer(host, T)
    try:
        layer.set_option("path", TC)
        layer.set_option("tc_weights", 2)
        cached, _ = layer.forward_host(x)
        layer.set_option("tc_weights", 1)
        packed, _ = layer.forward_host(x)
    finally:
        layer.close()
    assert np.array_equal(cached, packed)   # both round fma(q, scale, bias) to bf16 once and run the same MMA sequence
    run_and_check(oracle_mod, spec, T, seed=5, host=host, path=TC, options={"tc_weights": 1})


# ── precision of the one-launch forward: activation results of 8-bit experts and of the shared expert stay in fp32 ──

@pytest.mark.parametrize("gs,shared_bits,T", [(64, 0, 1), (32, 0, 8), (64, 8, 1), (128, 8, 8), (64, 4, 3)])
def test_one_launch_keeps_fp32_activation_results(oracle_mod, gs, shared_bits, T):
    """fp32 sums of these lengths are off by about 1e-5 of the output's RMS, a bf16 step is 2**-8 to 2**-7 of a value: about 0.3 % of
    the outputs may round the other way (0.05 % measured).  Activation results rounded to bf16 are off by 4e-4 and more: 2 to 10 %."""
    spec = synth.LayerSpec("fp32_inner", 1024, 768, 16, 4, expert_bits=8, expert_group_size=gs)
    if shared_bits:
        spec = spec.with_(shared_intermediate=512, shared_bits=shared_bits, shared_group_size=64, shared_gate_kind=capi.LINEAR_F32)
    host = synth.make_layer(spec, 21)
    x = synth.make_tokens(T, spec.hidden, 21)
    layer = MoELayer(host, 8)
    try:
        out, _ = layer.forward_host(x)
        assert layer.launch_count() == 1
    finally:
        layer.close()
    ref = oracle_mod.moe_forward(host, x)
    differ = float(np.mean(out != synth.f32_to_bf16(ref.out_f32)))
    assert differ <= 0.005, f"{100 * differ:.2f} % of the outputs differ from the rounded fp32 result"


@pytest.mark.parametrize("bits,gs", [(4, 64), (4, 32), (8, 64)])
@pytest.mark.parametrize("field,value", [("scales", np.inf), ("biases", np.nan)])
def test_one_launch_confines_non_finite_weights(oracle_mod, bits, gs, field, value):
    """An infinite or undefined scale of one expert reaches the tokens that selected it and no others."""
    spec = synth.LayerSpec("non_finite", 512, 256, 16, 4, expert_bits=bits, expert_group_size=gs)
    host = synth.make_layer(spec, 31)
    x = synth.make_tokens(8, spec.hidden, 31)
    ref = oracle_mod.moe_forward(host, x)
    share = np.array([(ref.indices == e).any(axis=1).mean() for e in range(16)])
    e = int(np.argmin(np.abs(share - 0.4)))             # some tokens select it, some do not
    has = (ref.indices == e).any(axis=1)
    assert has.any() and not has.all()
    host.arrays["experts.down_proj." + field][e] = 0x7F80 if value == np.inf else 0x7FC0
    layer = MoELayer(host, 8)
    try:
        out, dbg = layer.forward_host(x, debug=True)
        assert layer.launch_count() == 1
    finally:
        layer.close()
    assert np.array_equal(dbg.indices, ref.indices)
    assert_parity(out[~has], ref.out_f32[~has], what=spec.name)


# 4-bit experts of group 32 add re-tiled scale words (as large as scales and biases) for the decode kernels, 8-bit ones nothing
@pytest.mark.parametrize("bits,gs,extra", [(8, 64, 0.0), (8, 32, 0.0), (4, 32, 0.2)])
def test_loading_makes_no_further_copy_of_the_experts(bits, gs, extra):
    import torch
    spec = synth.LayerSpec("no_copy", 1024, 768, 24, 4, expert_bits=bits, expert_group_size=gs, shared_intermediate=1024, shared_bits=8,
                           shared_group_size=64)
    small = spec.with_(n_experts=4)
    warm = MoELayer(synth.make_layer(small, 1), 8)      # kernels are loaded on first use
    warm.forward_host(synth.make_tokens(3, spec.hidden, 1))
    host = synth.make_layer(spec, 1)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    layer = MoELayer(host, 8)
    try:
        used = before - torch.cuda.mem_get_info()[0]
        layer.forward_host(synth.make_tokens(3, spec.hidden, 1))
        assert layer.launch_count() == 1
    finally:
        layer.close()
        warm.close()
    shared_bf16 = 3 * 1024 * 1024 * 2                   # the shared expert's operand tiles of the prefill path
    # the rest: workspace of 8 tokens and the 2 MB granules of a few dozen small allocations
    assert used <= host.weight_bytes() * (1 + extra) + shared_bf16 + (24 << 20), f"{used / 2**20:.0f} MiB for {host.weight_bytes() / 2**20:.0f} MiB of weights"


def test_stream_with_a_part_of_the_sms_takes_the_launch_chain(oracle_mod):
    """A green context's stream may run on 64 SMs: one CTA per SM of the device cannot be resident there at once."""
    import torch
    cu = pytest.importorskip("cuda.bindings.driver")

    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1] if len(r) == 2 else r[1:]
    spec = synth.LayerSpec("part_of_sms", 512, 256, 16, 4)
    host = synth.make_layer(spec, 41)
    x = synth.make_tokens(3, spec.hidden, 41)
    ref = oracle_mod.moe_forward(host, x)
    layer = MoELayer(host, 8)
    try:
        xd = to_dev(x)
        out = torch.zeros_like(xd)
        torch.cuda.synchronize()
        dev = ok(cu.cuDeviceGet(torch.cuda.current_device()))
        sms = ok(cu.cuDeviceGetDevResource(dev, cu.CUdevResourceType.CU_DEV_RESOURCE_TYPE_SM))
        groups = ok(cu.cuDevSmResourceSplitByCount(1, sms, 0, 64))[0]
        desc = ok(cu.cuDevResourceGenerateDesc([groups[0]], 1))
        ctx = ok(cu.cuGreenCtxCreate(desc, dev, cu.CUgreenCtxCreate_flags.CU_GREEN_CTX_DEFAULT_STREAM))
        stream = ok(cu.cuGreenCtxStreamCreate(ctx, cu.CUstream_flags.CU_STREAM_NON_BLOCKING, 0))
        try:
            layer.forward_ptr(xd.data_ptr(), 3, out.data_ptr(), 0, int(stream))
            ok((cu.cuStreamSynchronize(stream)[0], None))
            layer.check_device_status()
            assert layer.launch_count() > 1
        finally:
            cu.cuStreamDestroy(stream)
            cu.cuGreenCtxDestroy(ctx)
        assert_parity(from_dev(out, np.uint16), ref.out_f32, what=spec.name)
        layer.forward_ptr(xd.data_ptr(), 3, out.data_ptr())      # the whole device again
        torch.cuda.synchronize()
        assert layer.launch_count() == 1
        assert_parity(from_dev(out, np.uint16), ref.out_f32, what=spec.name)
    finally:
        layer.close()


@pytest.mark.parametrize("polls", [0, 1])
def test_grid_barrier_that_is_given_up(oracle_mod, polls):
    """The wait runs out (no poll, or one right after arriving): the call and the calls queued behind it write no output, the status
    check reports it, and the next call is right again."""
    import torch
    spec = synth.LayerSpec("given_up", 1024, 512, 16, 4, expert_bits=8)
    host = synth.make_layer(spec, 51)
    x = synth.make_tokens(3, spec.hidden, 51)
    ref = oracle_mod.moe_forward(host, x)
    layer = MoELayer(host, 8)
    try:
        xd = to_dev(x)
        out = torch.full_like(xd, 77)

        def call():
            layer.forward_ptr(xd.data_ptr(), 3, out.data_ptr())
            assert layer.launch_count() == 1
            torch.cuda.synchronize()
        call()
        assert_parity(from_dev(out, np.uint16), ref.out_f32, what=spec.name)
        out.fill_(77)
        layer.set_option("decode_wait_polls", polls)
        call()
        assert bool((out == 77).all())
        layer.set_option("decode_wait_polls", 1 << 21)
        call()
        call()
        assert bool((out == 77).all())
        with pytest.raises(capi.FFAICudaError) as ei:
            layer.check_device_status()
        assert ei.value.status == capi.FFAI_ERR_DEVICE_CHECK
        layer.check_device_status()
        call()
        assert_parity(from_dev(out, np.uint16), ref.out_f32, what=spec.name)
        # the host entry checks by itself
        layer.set_option("decode_wait_polls", polls)
        with pytest.raises(capi.FFAICudaError):
            layer.forward_host(x)
        layer.set_option("decode_wait_polls", 1 << 21)
        assert_parity(layer.forward_host(x)[0], ref.out_f32, what=spec.name)
    finally:
        layer.close()


@pytest.mark.parametrize("E", [32, 100, 256, 300])
@pytest.mark.parametrize("gating", [capi.GATING_SOFTMAX_THEN_TOPK, capi.GATING_TOPK_THEN_SOFTMAX])
def test_an_undefined_logit_is_not_selected(oracle_mod, E, gating):
    """One expert's router row is NaN: every router kernel selects among the others, as comparing with `>` does (the expert is not
    the first one, which the oracle's scan starts from)."""
    spec = synth.LayerSpec("nan_logit", 256, 64, E, 4, gating_mode=gating, router_logits_bf16=0)
    host = synth.make_layer(spec, 81)
    host.arrays["gate.weight"][7] = 0x7FC0
    layer = MoELayer(host, 300)
    try:
        for T in (1, 8, 40, 300):
            x = synth.make_tokens(T, spec.hidden, T)
            out, dbg = layer.forward_host(x, debug=True)
            ref = oracle_mod.moe_forward(host, x)
            assert not (ref.indices == 7).any()
            assert np.array_equal(dbg.indices, ref.indices) and np.array_equal(dbg.weights, ref.weights)
            assert_parity(out, ref.out_f32, what=spec.name)
    finally:
        layer.close()


@pytest.mark.parametrize("bits,gs", [(4, 64), (4, 32), (8, 64)])
def test_one_launch_in_a_captured_graph(oracle_mod, bits, gs):
    import torch
    spec = synth.LayerSpec("captured", 512, 256, 16, 4, expert_bits=bits, expert_group_size=gs)
    host = synth.make_layer(spec, 91)
    layer = MoELayer(host, 8)
    try:
        x = torch.zeros(5, spec.hidden, dtype=torch.int16, device="cuda")
        out = torch.zeros_like(x)
        graph = torch.cuda.CUDAGraph()
        torch.cuda.synchronize()
        with torch.cuda.graph(graph):       # the handle's first call
            layer.forward_ptr(x.data_ptr(), 5, out.data_ptr(), 0, torch.cuda.current_stream().cuda_stream)
        assert layer.launch_count() == 1
        for seed in (1, 2, 3):
            rows = synth.make_tokens(5, spec.hidden, seed)
            x.copy_(to_dev(rows))
            graph.replay()
            torch.cuda.synchronize()
            assert_parity(from_dev(out, np.uint16), oracle_mod.moe_forward(host, rows).out_f32, what=spec.name)
        layer.check_device_status()
        del graph
    finally:
        layer.close()
