"""GPU parity of the KDA kernels (short conv, recurrence) through the C ABI, against the CPU oracle
and, when it was built, against the reference's own kernels compiled for sm_100a."""
import os
import subprocess
import sys
import tempfile

import numpy as np
import pytest
import torch

import hk_oracle as orc
import hk_ref as ref
from gpu_util import bf16_ulp_diff, bits, dev, dev_bf16, frob_rel, max_rel
import helios_glm53flash_b200 as hk
from helios_glm53flash_b200 import synth

pytestmark = pytest.mark.gpu


def _run_conv(x, st, w, bsz, dim, T, K=4, act=True, history=False, state_size=None, use_ref=False):
    state_size = state_size or K
    dx, dst, dw = dev_bf16(x), dev_bf16(st), dev_bf16(w)
    out = torch.empty(bsz, T, dim, dtype=torch.bfloat16, device="cuda")
    fn = ref.conv1d_update if use_ref else hk.cuda_causal_conv1d_update
    fn(dx, dst, None, dw, None, out, bsz, dim, T, state_size, K, act, history)
    torch.cuda.synchronize()
    return bits(out), bits(dst)


@pytest.mark.parametrize("dim,T", [(1536, 512), (1536, 1), (1536, 3), (1536, 37), (256, 200), (192, 4099), (12288, 128)])
def test_conv_vs_oracle_and_reference(dim, T):
    inp = synth.conv_inputs(T, dim, seed=dim + T)
    o_out, o_st = orc.conv1d_update(inp["x"], inp["state"], inp["weight"], None, 1, dim, T, 4, 4)
    g_out, g_st = _run_conv(inp["x"], inp["state"], inp["weight"], 1, dim, T)
    assert np.array_equal(g_st, o_st), "window state must match exactly"
    ulp = bf16_ulp_diff(g_out, o_out)
    assert ulp.max() <= 1 and (ulp > 0).mean() < 2e-3  # exp approximation may flip a rounding
    if ref.available():
        r_out, r_st = _run_conv(inp["x"], inp["state"], inp["weight"], 1, dim, T, use_ref=True)
        assert np.array_equal(g_st, r_st)
        assert np.array_equal(g_out, r_out), "same arithmetic as the reference kernel: bit-exact"


@pytest.mark.parametrize("bsz,T", [(1, 16), (2, 17), (1, 24), (1, 63), (3, 65), (2, 68), (1, 72), (2, 129), (1, 190)])
def test_conv_at_the_edges_of_its_tiles(bsz, T):
    """64-token tiles of 16-token groups: rows that start on 16 bytes, on an even and on an odd element, and several sequences"""
    dim = 192
    x = synth.f32_to_bf16_bits(synth.rng(T).standard_normal((bsz, dim, T), dtype=np.float32))
    st = synth.f32_to_bf16_bits(synth.rng(T + 1).standard_normal((bsz, dim, 4), dtype=np.float32))
    w = synth.f32_to_bf16_bits(synth.rng(T + 2).standard_normal((dim, 4), dtype=np.float32))
    o_out, o_st = orc.conv1d_update(x, st, w, None, bsz, dim, T, 4, 4)
    g_out, g_st = _run_conv(x, st, w, bsz, dim, T)
    assert np.array_equal(g_st.reshape(-1), o_st.reshape(-1))
    ulp = bf16_ulp_diff(g_out.reshape(-1), o_out.reshape(-1))
    assert ulp.max() <= 1 and (ulp > 0).mean() < 5e-3


@pytest.mark.parametrize("T", [16, 37, 40, 63, 64])
def test_conv_of_a_short_call_in_one_wave_and_in_several(T):
    """a tile per CTA (taps and window asked for ahead) against more tiles than CTAs: the same bits, with permuted slots, a wider window and a
    bias"""
    bsz, dim, S, piece = 2, 64 * 450, 6, 64 * 150
    g = torch.Generator(device="cuda").manual_seed(T)
    r = lambda *n: torch.randn(*n, generator=g, device="cuda").bfloat16()
    x, st, w, bias = r(bsz, dim, T), r(3, dim, S), r(dim, 4), r(dim)
    slots = torch.tensor([2, 0], dtype=torch.int32, device="cuda")
    whole, out = st.clone(), torch.empty(bsz, T, dim, dtype=torch.bfloat16, device="cuda")
    hk.cuda_causal_conv1d_update(x, whole, slots, w, bias, out, bsz, dim, T, S, 4, True, False)
    for c in range(0, dim, piece):
        part, o = st[:, c:c + piece].contiguous(), torch.empty(bsz, T, piece, dtype=torch.bfloat16, device="cuda")
        hk.cuda_causal_conv1d_update(x[:, c:c + piece].contiguous(), part, slots, w[c:c + piece].contiguous(), bias[c:c + piece].contiguous(), o, bsz,
                                     piece, T, S, 4, True, False)
        assert torch.equal(o, out[:, :, c:c + piece]) and torch.equal(part, whole[:, c:c + piece])


def test_conv_history_and_generic_k():
    dim, T, K, S = 96, 9, 3, 7
    inp = synth.conv_inputs(T, dim, K=K, seed=5)
    st = synth.f32_to_bf16_bits(synth.rng(9).standard_normal((1, dim, S), dtype=np.float32))
    for history in (False, True):
        o_out, o_st = orc.conv1d_update(inp["x"], st, inp["weight"], None, 1, dim, T, S, K, True, history)
        g_out, g_st = _run_conv(inp["x"], st, inp["weight"], 1, dim, T, K=K, history=history, state_size=S)
        assert np.array_equal(g_st, o_st)
        assert bf16_ulp_diff(g_out, o_out).max() <= 1


def _run_rec(inp, state, bsz, T, H, D, stride=1, cw=True, hist=False, use_ref=False, force_recurrent=True):
    q, g, b = dev_bf16(inp["mixed_qkv"]), dev(inp["g"]), dev_bf16(inp["beta"])
    st = dev(state)
    out = torch.empty(bsz, T, H, D, dtype=torch.bfloat16, device="cuda")
    o32 = torch.empty(bsz, T, H, D, dtype=torch.float32, device="cuda")
    if use_ref:
        ref.kda_recurrent(q, g, b, st, out, bsz, T, H, H, D, D, stride, None, cw, hist)
        o32 = None
    else:
        hk.cuda_recurrent_gated_delta_rule(q, g, b, st, out, bsz, T, H, H, D, D, stride, None, cw, hist,
                                           out_f32=o32, force_recurrent=force_recurrent)
    torch.cuda.synchronize()
    return bits(out), (None if o32 is None else o32.cpu().numpy()), st.cpu().numpy()


@pytest.mark.parametrize("T,H", [(1, 32), (16, 4), (70, 2), (1, 64)])
def test_recurrent_vs_oracle_and_reference(T, H):
    D = 128
    inp = synth.kda_inputs(T, H, D, seed=T)
    s0 = (0.1 * synth.rng(3).standard_normal((1, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    o_out, o_32, o_st = orc.kda_recurrent(inp["mixed_qkv"], inp["g"], inp["beta"], s0, 1, T, H, H, D, D)
    g_out, g_32, g_st = _run_rec(inp, s0, 1, T, H, D)
    assert max_rel(g_32, o_32) < 2e-3 and max_rel(g_32, o_32) < 1e-4
    assert frob_rel(g_st, o_st) < 1e-5
    assert bf16_ulp_diff(g_out, o_out).max() <= 1
    if ref.available():
        r_out, _, r_st = _run_rec(inp, s0, 1, T, H, D, use_ref=True)
        assert frob_rel(g_st, r_st) < 1e-5
        assert bf16_ulp_diff(g_out, r_out).max() <= 1
        assert frob_rel(o_st, r_st) < 1e-5, "oracle pinned to the reference kernel"


@pytest.mark.parametrize("dim,cw,hist,steps", [(64, False, False, 7), (64, False, True, 7), (128, False, True, 1),
                                               (128, True, True, 7), (128, True, False, 7), (128, False, False, 1)])
def test_recurrent_determinism_suite_shapes(dim, cw, hist, steps):
    """the 12-config grid of the reference's bit-repeatability test (test_deterministic_reductions.cu:19-49):
    same synthetic inputs, here also checked for VALUE against the oracle, then 4 repeats byte-equal."""
    heads, stride = 2, (steps + 1 if hist else 1)
    n = steps * 3 * heads * dim
    i = np.arange(n, dtype=np.float32)
    qkv = synth.f32_to_bf16_bits(np.sin(i * np.float32(0.019))).reshape(1, steps, 3 * heads * dim)
    bi = np.arange(steps * heads, dtype=np.float32)
    beta = synth.f32_to_bf16_bits((0.3 + np.cos(bi) * 0.1).astype(np.float32)).reshape(1, steps, heads)
    ng = steps * heads * (dim if cw else 1)
    g = (-0.01 - (np.arange(ng) % 7) * 0.003).astype(np.float32)
    s0 = (np.sin(np.arange(stride * heads * dim * dim, dtype=np.float32) * np.float32(0.017)) * 0.2).astype(np.float32)
    s0 = s0.reshape(1, stride, heads, dim, dim)
    inp = {"mixed_qkv": qkv, "g": g, "beta": beta}
    o_out, o_32, o_st = orc.kda_recurrent(qkv, g, beta, s0, 1, steps, heads, heads, dim, dim, stride,
                                          None, cw, hist)
    first = None
    for rep in range(4):
        g_out, g_32, g_st = _run_rec(inp, s0, 1, steps, heads, dim, stride, cw, hist)
        if first is None:
            first = (g_out.copy(), g_st.copy())
            assert max_rel(g_32, o_32) < 1e-4
            assert frob_rel(g_st, o_st) < 1e-5
        assert np.array_equal(g_out, first[0]) and np.array_equal(g_st.view(np.uint32), first[1].view(np.uint32))
    if ref.available():
        r_out, _, r_st = _run_rec(inp, s0, 1, steps, heads, dim, stride, cw, hist, use_ref=True)
        assert frob_rel(g_st, r_st) < 1e-5
        assert bf16_ulp_diff(g_out, r_out).max() <= 1


def test_recurrent_slots_and_batch():
    T, H, D, bsz = 3, 4, 128, 3
    inp = synth.kda_inputs(T, H, D, bsz=bsz, seed=11)
    slots = np.array([2, 0, 3], dtype=np.int32)
    s0 = (0.1 * synth.rng(4).standard_normal((4, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    o_out, o_32, o_st = orc.kda_recurrent(inp["mixed_qkv"], inp["g"], inp["beta"], s0, bsz, T, H, H, D, D, 1, slots)
    q, g, b, st = dev_bf16(inp["mixed_qkv"]), dev(inp["g"]), dev_bf16(inp["beta"]), dev(s0)
    out = torch.empty(bsz, T, H, D, dtype=torch.bfloat16, device="cuda")
    hk.cuda_recurrent_gated_delta_rule(q, g, b, st, out, bsz, T, H, H, D, D, 1, dev(slots), True, False)
    torch.cuda.synchronize()
    assert frob_rel(st.cpu().numpy(), o_st) < 1e-5
    assert np.array_equal(st.cpu().numpy()[1], s0[1]), "unused slot untouched"
    assert bf16_ulp_diff(bits(out), o_out).max() <= 1


def test_bad_arguments_are_rejected_before_launch():
    t = torch.zeros(16, device="cuda")
    with pytest.raises(hk.HeliosB200Error) as e:
        hk.cuda_recurrent_gated_delta_rule(t, t, t, t, t, 1, 1, 3, 4, 128, 128, 1, None, True, False)
    assert e.value.status == hk.HK_ERR_INVALID
    with pytest.raises(hk.HeliosB200Error) as e:
        hk.cuda_recurrent_gated_delta_rule(t, t, t, t, t, 1, 1, 4, 4, 96, 96, 1, None, False, False)
    assert e.value.status == hk.HK_ERR_UNSUPPORTED
    with pytest.raises(hk.HeliosB200Error):
        hk.cuda_causal_conv1d_update(t, t, None, t, None, t, 1, 64, 8, 2, 4, True, False)


# ------------------------------------------------------------------------------------------------
# chunked tensor-core prefill == the recurrence called with seqlen = T
# ------------------------------------------------------------------------------------------------
def _gate_like_reference(T, H, D, seed):
    """log-decay in the reference engine's range: lb * sigmoid(x), lb = -5 (src/engine/glue2.cu:347-360)"""
    x = synth.rng(seed).standard_normal((1, T, H, D), dtype=np.float32)
    return (-5.0 / (1.0 + np.exp(-x))).astype(np.float32)


@pytest.mark.parametrize("T,H,gate", [(64, 2, "config"), (65, 2, "config"), (127, 1, "config"), (128, 4, "config"),
                                      (200, 2, "config"), (512, 32, "config"), (256, 2, "reference"), (192, 2, "weak")])
def test_chunked_prefill_vs_oracle(T, H, gate):
    D = 128
    inp = synth.kda_inputs(T, H, D, seed=100 + T)
    if gate == "reference":
        inp["g"] = _gate_like_reference(T, H, D, 7)
    elif gate == "weak":
        inp["g"] = (inp["g"] * 0.02).astype(np.float32)      # long memory: state grows over many chunks
    s0 = (0.1 * synth.rng(3).standard_normal((1, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    o_out, o_32, o_st = orc.kda_recurrent(inp["mixed_qkv"], inp["g"], inp["beta"], s0, 1, T, H, H, D, D)
    q, g, b, st = dev_bf16(inp["mixed_qkv"]), dev(inp["g"]), dev_bf16(inp["beta"]), dev(s0)
    out = torch.empty(1, T, H, D, dtype=torch.bfloat16, device="cuda")
    o32 = torch.empty(1, T, H, D, dtype=torch.float32, device="cuda")
    path = hk.cuda_recurrent_gated_delta_rule(q, g, b, st, out, 1, T, H, H, D, D, 1, None, True, False, out_f32=o32)
    torch.cuda.synchronize()
    assert path == "chunked"
    assert hk.read_device_status() == 0
    e_out, e_st = max_rel(o32.cpu().numpy(), o_32), frob_rel(st.cpu().numpy(), o_st)
    print("chunked T=%d H=%d gate=%s: out max_rel %.2e, state frob %.2e" % (T, H, gate, e_out, e_st))
    assert e_out < 2e-3, "outputs within 2e-3 (max |a-b| / max |b|) of the recurrence"
    assert e_st < 1e-2, "state within 1e-2 relative Frobenius"
    # the rounded output is the round-toward-zero bf16 of the fp32 output
    want_bits = (o32.cpu().numpy().view(np.uint32) >> 16).astype(np.uint16)
    assert np.array_equal(bits(out), want_bits)


@pytest.mark.parametrize("gate,tol", [("resets", 2e-3), ("minus_inf", 2e-3), ("some", 2e-3), ("channels", 1.5e-2), ("strong", 1.5e-2)])
@pytest.mark.parametrize("gated", [False, True])
def test_chunked_prefill_of_gates_that_decay_a_block_below_fp32(gate, tol, gated):
    """a channel's decay over a 16-token block below e^-80: hard resets between mild gates (also e^-inf), a few strong gates in a block, every
    gate of some channels or of all of them stronger than e^-5.  The strongest of a block are weakened, at worst to e^-5 = 6.7e-3 of the
    state instead of less, which a token's output and update each see once: 1.5e-2; with room for e^-10 (5e-5) the usual bounds"""
    T, H, D = 200, 4, 128
    inp, r = synth.kda_inputs(T, H, D, seed=5), np.random.RandomState(5)
    f = np.abs(r.standard_normal((1, T, H, D))).astype(np.float32)
    hard = r.random((1, T, H, D)) < 0.08
    g = {"resets": np.where(hard, -100.0, -0.05 * f), "minus_inf": np.where(hard, -np.inf if not gated else -500.0, -0.05 * f),
         "some": np.where(r.random((1, T, H, D)) < 0.25, -30.0, -0.3 * f), "channels": np.where(np.arange(D) % 2, -8.0 - f, -0.05 * f),
         "strong": -5.5 - 5.0 * f}[gate].astype(np.float32)
    s0 = (0.1 * r.standard_normal((1, 1, H, D, D))).astype(np.float32)
    beta, st = inp["beta"], dev(s0)
    out, o32 = torch.empty(1, T, H, D, dtype=torch.bfloat16, device="cuda"), torch.empty(1, T, H, D, device="cuda")
    if gated:                                                # raw gates whose prepared values are g: a bound of -600, the sigmoid's inverse
        lb, fr = -600.0, np.log(np.maximum(-g, 1e-6) / (600.0 + g)).astype(np.float32)
        gd, bd = torch.empty(1, T, H, D, device="cuda"), torch.empty(1, T, H, dtype=torch.bfloat16, device="cuda")
        raw_b, zero, one = dev(r.standard_normal((1, T, H)).astype(np.float32)), torch.zeros(H, D, device="cuda"), torch.zeros(H, device="cuda")
        hk.kda_gate(raw_b, dev(fr), zero, one, lb, bd, gd, T, H, D)
        g, beta = gd.cpu().numpy(), bits(bd)
        hk.kda_chunked_prefill_gated(dev_bf16(inp["mixed_qkv"]), dev(fr), raw_b, zero, one, lb, st, out, 1, T, H, out_f32=o32)
    else:
        hk.cuda_recurrent_gated_delta_rule(dev_bf16(inp["mixed_qkv"]), dev(g), dev_bf16(beta), st, out, 1, T, H, H, D, D, 1, None, True, False,
                                           out_f32=o32)
    torch.cuda.synchronize()
    assert hk.read_device_status() == 0
    _, o_32, o_st = orc.kda_recurrent(inp["mixed_qkv"], g, beta, s0, 1, T, H, H, D, D)
    e_out, e_st = frob_rel(o32.cpu().numpy(), o_32), frob_rel(st.cpu().numpy(), o_st)
    print("gates %s: outputs %.2e, state %.2e" % (gate, e_out, e_st))
    assert e_out < tol and e_st < tol


def test_chunked_prefill_then_decode_continues_the_state():
    T, H, D, extra = 256, 4, 128, 16
    inp = synth.kda_inputs(T + extra, H, D, seed=9)
    s0 = np.zeros((1, 1, H, D, D), dtype=np.float32)
    _, o_32, o_st = orc.kda_recurrent(inp["mixed_qkv"], inp["g"], inp["beta"], s0, 1, T + extra, H, H, D, D)
    q, g, b, st = dev_bf16(inp["mixed_qkv"]), dev(inp["g"]), dev_bf16(inp["beta"]), dev(s0)
    out = torch.empty(1, T + extra, H, D, dtype=torch.bfloat16, device="cuda")
    o32 = torch.empty(1, T + extra, H, D, dtype=torch.float32, device="cuda")
    hk.cuda_recurrent_gated_delta_rule(q[:, :T], g[:, :T], b[:, :T], st, out[:, :T], 1, T, H, H, D, D, 1, None, True,
                                       False, out_f32=o32[:, :T])
    for s in range(T, T + extra):
        hk.cuda_recurrent_gated_delta_rule(q[:, s:s + 1], g[:, s:s + 1], b[:, s:s + 1], st, out[:, s:s + 1], 1, 1, H, H,
                                           D, D, 1, None, True, False, out_f32=o32[:, s:s + 1])
    torch.cuda.synchronize()
    assert max_rel(o32.cpu().numpy(), o_32) < 2e-3
    assert frob_rel(st.cpu().numpy(), o_st) < 1e-2


def test_chunked_matches_recurrent_kernel_and_reference_kernel():
    T, H, D = 320, 3, 128
    inp = synth.kda_inputs(T, H, D, seed=12)
    s0 = (0.05 * synth.rng(5).standard_normal((1, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    _, c32, c_st = _run_rec(inp, s0, 1, T, H, D, force_recurrent=False)
    _, r32, r_st = _run_rec(inp, s0, 1, T, H, D, force_recurrent=True)
    assert max_rel(c32, r32) < 2e-3 and frob_rel(c_st, r_st) < 1e-2
    if ref.available():
        _, _, ref_st = _run_rec(inp, s0, 1, T, H, D, use_ref=True)
        assert frob_rel(c_st, ref_st) < 1e-2, "state vs the reference's own kernel run with seqlen = T"


def test_chunked_batch_and_slots():
    T, H, D, bsz = 130, 2, 128, 2
    inp = synth.kda_inputs(T, H, D, bsz=bsz, seed=14)
    slots = np.array([1, 0], dtype=np.int32)
    s0 = (0.1 * synth.rng(6).standard_normal((2, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    _, o_32, o_st = orc.kda_recurrent(inp["mixed_qkv"], inp["g"], inp["beta"], s0, bsz, T, H, H, D, D, 1, slots)
    q, g, b, st = dev_bf16(inp["mixed_qkv"]), dev(inp["g"]), dev_bf16(inp["beta"]), dev(s0)
    out = torch.empty(bsz, T, H, D, dtype=torch.bfloat16, device="cuda")
    o32 = torch.empty(bsz, T, H, D, dtype=torch.float32, device="cuda")
    assert hk.cuda_recurrent_gated_delta_rule(q, g, b, st, out, bsz, T, H, H, D, D, 1, dev(slots), True, False,
                                              out_f32=o32) == "chunked"
    torch.cuda.synchronize()
    assert max_rel(o32.cpu().numpy(), o_32) < 2e-3 and frob_rel(st.cpu().numpy(), o_st) < 1e-2


@pytest.mark.parametrize("T,H,bsz", [(2100, 3, 1), (1500, 2, 2), (4096, 32, 1), (1200, 64, 1), (1100, 32, 3), (1100, 17, 3)])
def test_chunked_fused_launch_equals_two_kernel_form(T, H, bsz):
    """the persistent fused launch (chains + preparation workers through the L2 ring; T spans more chunks than the
    ring has slots, so slots are reused) against the two-kernel form on the same inputs: same bits; the short
    cases also against the oracle.  The last three cases have more than 48 chains: 32, 48 and 17 chain CTAs walk two,
    two and three chains each, one after the other."""
    D = 128
    inp = synth.kda_inputs(T, H, D, bsz=bsz, seed=200 + T)
    s0 = (0.1 * synth.rng(8).standard_normal((bsz, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    q, g, b = dev_bf16(inp["mixed_qkv"]), dev(inp["g"]), dev_bf16(inp["beta"])
    res = []
    try:
        for form in (1, 0):
            hk.kda_chunked_set_form(form)
            st = dev(s0)
            out = torch.empty(bsz, T, H, D, dtype=torch.bfloat16, device="cuda")
            o32 = torch.empty(bsz, T, H, D, dtype=torch.float32, device="cuda")
            ws_bytes = hk.kda_chunked_workspace_bytes(bsz, T, H)
            assert hk.cuda_recurrent_gated_delta_rule(q, g, b, st, out, bsz, T, H, H, D, D, 1, None, True, False,
                                                      out_f32=o32) == "chunked"
            # a second call on the same workspace-sized buffer: the ring flags are reset by every call
            st2 = dev(s0)
            ws = torch.empty(ws_bytes, dtype=torch.uint8, device="cuda")
            for _ in range(2):
                st2.copy_(dev(s0))
                hk.cuda_recurrent_gated_delta_rule(q, g, b, st2, out, bsz, T, H, H, D, D, 1, None, True, False,
                                                   out_f32=o32, workspace=ws)
            torch.cuda.synchronize()
            assert hk.read_device_status() == 0
            assert np.array_equal(st.cpu().numpy(), st2.cpu().numpy())
            res.append((ws_bytes, o32.cpu().numpy(), st.cpu().numpy(), bits(out)))
    finally:
        hk.kda_chunked_set_form(0)
    assert res[1][0] < res[0][0], "the fused form needs the ring only"
    assert np.array_equal(res[0][1], res[1][1]) and np.array_equal(res[0][2], res[1][2])
    assert np.array_equal(res[0][3], res[1][3])
    if T * H * bsz <= 8192:
        _, o_32, o_st = orc.kda_recurrent(inp["mixed_qkv"], inp["g"], inp["beta"], s0, bsz, T, H, H, D, D)
        assert max_rel(res[1][1], o_32) < 2e-3 and frob_rel(res[1][2], o_st) < 1e-2


@pytest.mark.parametrize("T,H,bsz,strong", [(4097, 1, 1, False), (4160, 16, 1, True), (1090, 23, 1, True), (1090, 24, 1, False),
                                            (600, 51, 1, False), (1040, 16, 3, True), (1030, 63, 1, False)])
def test_chunked_chain_shapes_and_ring_depths(T, H, bsz, strong):
    """One or two CTAs a chain, a slot of one to three chains, rings of 16 and 32 units, raw and formed gates, every token at the
    bound of the decay: the bits of the two-kernel form.  The deep ring (16 slots or fewer, 64 chunks or more) is asked for, not
    required: half its units are enough, with the same bits, and a workspace below them is refused."""
    D, unit = 128, 74240
    inp = synth.kda_inputs(T, H, D, bsz=bsz, seed=300 + T + H)
    q, b = dev_bf16(inp["mixed_qkv"]), dev_bf16(inp["beta"])
    g = dev(np.full_like(inp["g"], -5.0) if strong else inp["g"])
    gen = torch.Generator(device="cuda").manual_seed(T + H)
    f, bl = torch.randn(bsz, T, H, D, generator=gen, device="cuda"), torch.randn(bsz, T, H, generator=gen, device="cuda")
    dt, al = torch.randn(H, D, generator=gen, device="cuda"), torch.randn(H, generator=gen, device="cuda")
    s0 = 0.1 * torch.randn(bsz, 1, H, D, D, generator=gen, device="cuda")
    full = hk.kda_chunked_workspace_bytes(bsz, T, H)
    deep = H * bsz <= 16
    least = full - 16 * H * bsz * unit if deep else full

    def run(nbytes):
        ws = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
        got = []
        for gated in (False, True):
            st, out = s0.clone(), torch.empty(bsz, T, H, D, dtype=torch.bfloat16, device="cuda")
            o32 = torch.empty(bsz, T, H, D, device="cuda")
            if gated:
                hk.kda_chunked_prefill_gated(q, f, bl, dt, al, -5.0, st, out, bsz, T, H, out_f32=o32, workspace=ws)
            else:
                hk.cuda_recurrent_gated_delta_rule(q, g, b, st, out, bsz, T, H, H, D, D, 1, None, True, False, out_f32=o32,
                                                   workspace=ws)
            got += [st, out, o32]
        torch.cuda.synchronize()
        assert hk.read_device_status() == 0
        return got

    first = run(full)
    others = [run(least)] if deep else []
    with pytest.raises(hk.HeliosB200Error):
        run(least - 1)
    try:
        hk.kda_chunked_set_form(1)
        others.append(run(hk.kda_chunked_workspace_bytes(bsz, T, H)))
    finally:
        hk.kda_chunked_set_form(0)
    for got in others:
        assert all(torch.equal(x, y) for x, y in zip(first, got))


@pytest.mark.parametrize("H,bsz", [(32, 1), (4, 2), (64, 3), (64, 5)])
def test_decode_step_with_conv_inside_equals_the_two_launch_sequence(H, bsz):
    """hk_kda_decode_step (conv + recurrence of one decoded token in one launch, value slices of a head as a cluster)
    against cuda_causal_conv1d_update followed by cuda_recurrent_gated_delta_rule on the same buffers, 6 tokens in a
    row with carried window and state: same bits everywhere; the first token also against the oracle"""
    D, steps = 128, 6
    dim = 3 * H * D
    r = synth.rng(77 + H)
    x = synth.f32_to_bf16_bits(r.standard_normal((steps, bsz, dim), dtype=np.float32))
    w = synth.f32_to_bf16_bits((0.1 * r.standard_normal((dim, 4), dtype=np.float32)).astype(np.float32))
    bias = synth.f32_to_bf16_bits((0.05 * r.standard_normal((dim,), dtype=np.float32)).astype(np.float32))
    cst0 = synth.f32_to_bf16_bits(r.standard_normal((bsz, dim, 4), dtype=np.float32))
    gates = synth.kda_gates(steps, H, D, bsz=bsz, seed=3)
    g_all, beta_all = dev(np.ascontiguousarray(gates["g"].transpose(1, 0, 2, 3))), dev_bf16(np.ascontiguousarray(gates["beta"].transpose(1, 0, 2)))
    s0 = (0.1 * r.standard_normal((bsz, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    xd, wd, bd = dev_bf16(x), dev_bf16(w), dev_bf16(bias)
    # two-launch sequence
    cs_a, st_a = dev_bf16(cst0), dev(s0)
    qkv_a = torch.empty(steps, bsz, 1, dim, dtype=torch.bfloat16, device="cuda")
    out_a = torch.empty(steps, bsz, 1, H, D, dtype=torch.bfloat16, device="cuda")
    # fused
    cs_b, st_b = dev_bf16(cst0), dev(s0)
    qkv_b = torch.empty(steps, bsz, dim, dtype=torch.bfloat16, device="cuda")
    out_b = torch.empty(steps, bsz, H, D, dtype=torch.bfloat16, device="cuda")
    o32_b = torch.empty(steps, bsz, H, D, dtype=torch.float32, device="cuda")
    for s in range(steps):
        hk.cuda_causal_conv1d_update(xd[s].reshape(bsz, dim, 1), cs_a, None, wd, bd, qkv_a[s], bsz, dim, 1, 4, 4, True, False)
        hk.cuda_recurrent_gated_delta_rule(qkv_a[s], g_all[s], beta_all[s], st_a, out_a[s], bsz, 1, H, H, D, D, 1, None, True, False)
        hk.kda_decode_step(xd[s], cs_b, wd, bd, g_all[s], beta_all[s], st_b, out_b[s], bsz, H, out_f32=o32_b[s], conv_out=qkv_b[s])
    torch.cuda.synchronize()
    assert np.array_equal(bits(qkv_a.reshape(steps, bsz, dim)), bits(qkv_b)), "convolved q|k|v"
    assert np.array_equal(bits(cs_a), bits(cs_b)), "rolling window"
    assert np.array_equal(st_a.cpu().numpy(), st_b.cpu().numpy()), "recurrent state"
    assert np.array_equal(bits(out_a.reshape(steps, bsz, H, D)), bits(out_b)), "outputs"
    # first token against the oracle (conv, then recurrence)
    qkv0, _ = orc.conv1d_update(np.ascontiguousarray(x[0]).reshape(bsz, dim, 1), cst0, w, bias, bsz, dim, 1, 4, 4)
    assert np.array_equal(qkv0.reshape(bsz, dim), bits(qkv_b[0])) or \
        bf16_ulp_diff(qkv0.reshape(bsz, dim), bits(qkv_b[0])).max() <= 1
    _, o_32, _ = orc.kda_recurrent(bits(qkv_b[0]).reshape(bsz, 1, dim), np.ascontiguousarray(gates["g"][:, :1]),
                                   np.ascontiguousarray(gates["beta"][:, :1]), s0, bsz, 1, H, H, D, D)
    assert max_rel(o32_b[0].cpu().numpy().reshape(bsz, 1, H, D), o_32) < 2e-3


@pytest.mark.parametrize("H,bsz,w_bf16,g_bf16,y_f16", [(32, 1, True, False, True), (4, 3, False, True, False), (64, 2, True, True, True),
                                                        (37, 1, True, False, True), (19, 2, False, False, False)])
def test_decode_layer_in_one_launch_equals_the_five_call_sequence(H, bsz, w_bf16, g_bf16, y_f16):
    """hk_kda_decode_layer (cast, gate preparation, conv, recurrence, gated RMS norm of one decoded token in ONE launch)
    against kda_transpose_cast -> kda_gate -> cuda_causal_conv1d_update -> cuda_recurrent_gated_delta_rule ->
    gated_rms_norm on the same buffers, 5 tokens in a row with carried window and state: the same bits everywhere"""
    D, steps = 128, 5
    dim = 3 * H * D
    r = synth.rng(5 + H)
    x32 = dev(r.standard_normal((steps, bsz, dim), dtype=np.float32))
    raw = synth.kda_raw_gates(steps * bsz, H, D, seed=9)
    f = dev(raw["f"]).reshape(steps, bsz, H, D).contiguous()
    b = dev(raw["b"]).reshape(steps, bsz, H).contiguous()
    dtb, alog, lb = dev(raw["dt_bias"]), dev(raw["a_log"]), raw["lower_bound"]
    w = dev_bf16(synth.f32_to_bf16_bits((0.1 * r.standard_normal((dim, 4), dtype=np.float32)).astype(np.float32)))
    cst0 = synth.f32_to_bf16_bits(r.standard_normal((bsz, dim, 4), dtype=np.float32))
    s0 = (0.1 * r.standard_normal((bsz, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    nw = (1.0 + 0.1 * torch.randn(D, device="cuda"))
    nw = nw.to(torch.bfloat16) if w_bf16 else nw
    go = torch.randn(steps, bsz * H, D, device="cuda")
    go = go.to(torch.bfloat16) if g_bf16 else go
    ydt = torch.float16 if y_f16 else torch.float32
    cs_a, st_a, cs_b, st_b = dev_bf16(cst0), dev(s0), dev_bf16(cst0), dev(s0)
    x16 = torch.empty(bsz, dim, 1, dtype=torch.bfloat16, device="cuda")
    g = torch.empty(bsz, H, D, dtype=torch.float32, device="cuda")
    beta = torch.empty(bsz, H, dtype=torch.bfloat16, device="cuda")
    qkv = torch.empty(bsz, 1, dim, dtype=torch.bfloat16, device="cuda")
    out_a = torch.empty(steps, bsz, 1, H, D, dtype=torch.bfloat16, device="cuda")
    out_b = torch.empty(steps, bsz, H, D, dtype=torch.bfloat16, device="cuda")
    y_a = torch.empty(steps, bsz * H, D, dtype=ydt, device="cuda")
    y_b = torch.empty(steps, bsz * H, D, dtype=ydt, device="cuda")
    for s in range(steps):
        for q in range(bsz):
            hk.kda_transpose_cast(x16[q], x32[s, q:q + 1], 1, dim)
        hk.kda_gate(b[s], f[s], dtb, alog, lb, beta, g, bsz, H, D)
        hk.cuda_causal_conv1d_update(x16, cs_a, None, w, None, qkv, bsz, dim, 1, 4, 4, True, False)
        hk.cuda_recurrent_gated_delta_rule(qkv, g, beta, st_a, out_a[s], bsz, 1, H, H, D, D, 1, None, True, False)
        hk.gated_rms_norm(out_a[s], nw, y_a[s], go[s], bsz * H, D, 1e-6, gate_act=1)
        hk.kda_decode_layer(x32[s], cs_b, w, None, f[s], b[s], dtb, alog, lb, st_b, out_b[s], nw, go[s], y_b[s], bsz, H,
                            epsilon=1e-6, gate_act=1)
    torch.cuda.synchronize()
    assert np.array_equal(bits(cs_a), bits(cs_b)), "rolling window"
    assert np.array_equal(st_a.cpu().numpy(), st_b.cpu().numpy()), "recurrent state"
    assert np.array_equal(bits(out_a.reshape(steps, bsz, H, D)), bits(out_b)), "recurrence outputs"
    assert torch.equal(y_a, y_b), "normalised outputs"
    assert torch.isfinite(y_b.float()).all()


@pytest.mark.parametrize("H", [1, 32, 37, 38])
def test_decode_layer_beside_others_on_streams_gives_the_same_bits(H):
    """four streams at once, a CTA a head, against the call that is alone (four CTAs a head up to 37): outputs, windows and states, two tokens"""
    D, dim, n = 128, 3 * H * 128, 4
    gen = torch.Generator(device="cuda").manual_seed(H)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    w, dtb, alog, nw = (0.1 * r(dim, 4)).bfloat16(), r(H, D), 0.3 * r(H), (1 + 0.1 * r(D)).bfloat16()
    calls = [dict(x=r(2, dim), f=r(2, H, D), b=r(2, H), go=r(2, H, D), cs=r(1, dim, 4).bfloat16(), rs=0.1 * r(1, 1, H, D, D)) for _ in range(n)]

    def run(beside):
        streams = [torch.cuda.Stream() for _ in range(n)] if beside else [None] * n
        got = [(c["cs"].clone(), c["rs"].clone(), torch.empty(2, H, D, dtype=torch.bfloat16, device="cuda"),
                torch.empty(2, H, D, dtype=torch.float16, device="cuda")) for c in calls]
        torch.cuda.synchronize()
        for t in range(2):
            for c, (cs, rs, out, y), s in zip(calls, got, streams):
                hk.kda_decode_layer(c["x"][t], cs, w, None, c["f"][t], c["b"][t], dtb, alog, -5.0, rs, out[t], nw, c["go"][t], y[t], 1, H,
                                    stream=s, beside=beside)
        torch.cuda.synchronize()
        return got

    for alone, beside in zip(run(False), run(True)):
        assert all(torch.equal(a, b) for a, b in zip(alone, beside))
    assert hk.read_device_status() == 0


@pytest.mark.parametrize("H,bsz,slots", [(64, 5, False), (8, 41, True), (33, 9, True)])
def test_decode_of_many_heads_streams_the_same_bits(H, bsz, slots):
    """more heads than two per SM: the persistent form (heads stream through shared memory, ragged last round) against the
    per-sequence calls, which take the one-head-per-CTA form; carried window and state, slots out of order"""
    D, dim = 128, 3 * H * 128
    gen = torch.Generator(device="cuda").manual_seed(H)

    def rnd(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")
    raw = synth.kda_raw_gates(1, H, D, seed=9)
    dtb, alog, lb = dev(raw["dt_bias"]), dev(raw["a_log"]), raw["lower_bound"]
    w, nw = (0.1 * rnd(dim, 4)).to(torch.bfloat16), 1.0 + 0.1 * rnd(D)
    cs, st = rnd(bsz, dim, 4).to(torch.bfloat16), 0.1 * rnd(bsz, 1, H, D, D)
    order = torch.randperm(bsz, generator=torch.Generator().manual_seed(1)).to(torch.int32).cuda() if slots else None
    res = []
    for whole in (True, False):
        c, s = cs.clone(), st.clone()
        out, y = torch.empty(2, bsz, H, D, dtype=torch.bfloat16, device="cuda"), torch.empty(2, bsz, H * D, dtype=torch.float16, device="cuda")
        gen.manual_seed(7)
        for t in range(2):
            x, f, b, go = rnd(bsz, dim), rnd(bsz, H, D), rnd(bsz, H), rnd(bsz, H * D)
            if whole:
                hk.kda_decode_layer(x, c, w, None, f, b, dtb, alog, lb, s, out[t], nw, go, y[t], bsz, H, slots=order)
            else:
                for i in range(bsz):
                    j = int(order[i]) if slots else i
                    hk.kda_decode_layer(x[i], c[j], w, None, f[i], b[i], dtb, alog, lb, s[j], out[t, i], nw, go[i], y[t, i], 1, H)
        torch.cuda.synchronize()
        res.append((out, y, c, s))
    assert hk.read_device_status() == 0
    for whole, single in zip(*res):
        assert torch.equal(whole, single)


@pytest.mark.parametrize("T,Hk,Hv,bsz", [(1, 2, 4, 1), (7, 3, 3, 2), (8, 1, 2, 1), (9, 4, 4, 3), (63, 2, 2, 1), (1, 37, 74, 1), (1, 25, 75, 1),
                                            (1, 8, 16, 19), (2, 8, 40, 1), (3, 16, 32, 1), (4, 16, 32, 1)])
def test_per_token_kernel_around_its_batches_of_eight(T, Hk, Hv, bsz):
    """token counts either side of the 8 prepared at a time, single tokens either side of the head counts that are split over CTAs or
    streamed, two and three tokens of many chains, grouped key heads, against the oracle"""
    D = 128
    inp = synth.kda_inputs(T, Hv, D, bsz=bsz, seed=T)
    qkv = inp["mixed_qkv"].reshape(bsz, T, 3, Hv, D)
    qkv = np.concatenate([qkv[:, :, 0, :Hk].reshape(bsz, T, -1), qkv[:, :, 1, :Hk].reshape(bsz, T, -1), qkv[:, :, 2].reshape(bsz, T, -1)], axis=2)
    s0 = (0.1 * synth.rng(3).standard_normal((bsz, 1, Hv, D, D), dtype=np.float32)).astype(np.float32)
    _, o_32, o_st = orc.kda_recurrent(np.ascontiguousarray(qkv), inp["g"], inp["beta"], s0, bsz, T, Hk, Hv, D, D)
    q, g, b, st = dev_bf16(qkv), dev(inp["g"]), dev_bf16(inp["beta"]), dev(s0)
    out = torch.empty(bsz, T, Hv, D, dtype=torch.bfloat16, device="cuda")
    f32 = torch.empty(bsz, T, Hv, D, dtype=torch.float32, device="cuda")
    hk.cuda_recurrent_gated_delta_rule(q, g, b, st, out, bsz, T, Hk, Hv, D, D, 1, None, True, False, out_f32=f32)
    torch.cuda.synchronize()
    assert max_rel(f32.cpu().numpy(), o_32) < 1e-4 and frob_rel(st.cpu().numpy(), o_st) < 1e-5
    assert np.array_equal(bits(out), (f32.cpu().numpy().view(np.uint32) >> 16).astype(np.uint16)), "rounded toward zero"


@pytest.mark.parametrize("H,bsz", [(2, 1), (40, 1), (8, 3), (64, 17)])
def test_token_by_token_routes_agree_bit_for_bit(H, bsz):
    """tokens one at a time, several in a call, and calls on a state with room for a history, recording it or not: whichever
    kernel a call takes (2 chains narrow, 40 and 24 the per-token kernel or the older one by length, 1,088 streamed), the same bits"""
    D, T = 128, 7
    gen = torch.Generator(device="cuda").manual_seed(H)

    def rnd(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")
    qkv, g = rnd(bsz, T, 3 * H * D).to(torch.bfloat16), -5.0 * torch.sigmoid(rnd(bsz, T, H, D))
    beta, s0 = torch.sigmoid(rnd(bsz, T, H)).to(torch.bfloat16), 0.1 * rnd(bsz, 1, H, D, D)

    def call(t0, n, st, stride=1, history=False):
        q, gg, b = (x[:, t0:t0 + n].contiguous() for x in (qkv, g, beta))
        out, f32 = (torch.empty(bsz, n, H, D, dtype=d, device="cuda") for d in (torch.bfloat16, torch.float32))
        hk.cuda_recurrent_gated_delta_rule(q, gg, b, st, out, bsz, n, H, H, D, D, stride, None, True, history, out_f32=f32)
        assert torch.equal(out.view(torch.int16), (f32.view(torch.int32) >> 16).to(torch.int16)), "rounded toward zero"
        return f32
    st, outs, states = s0.clone(), [], []
    for t in range(T):
        outs.append(call(t, 1, st))
        states.append(st.clone())
    outs = torch.cat(outs, dim=1)
    for n in (2, 3, 6, 7):
        st = s0.clone()
        assert torch.equal(call(0, n, st), outs[:, :n]) and torch.equal(st, states[n - 1]), n
    for history in (False, True):
        st = torch.zeros(bsz, T, H, D, D, device="cuda")
        st[:, :1] = s0
        assert torch.equal(call(0, T, st, T, history), outs) and torch.equal(st[:, :1], states[-1])
        for t in range(T - 1 if history else 0):
            assert torch.equal(st[:, t + 1:t + 2], states[t])


@pytest.mark.parametrize("H", [4, 32])
def test_decode_steps_share_nothing(H):
    """heads split over CTAs, on several streams at a time and whatever `tickets` holds: windows, states and outputs of each as
    when it runs alone"""
    D, dim, steps = 128, 3 * H * 128, 6
    gen = torch.Generator(device="cuda").manual_seed(H)

    def rnd(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")
    x, w, cs0 = rnd(steps, dim).to(torch.bfloat16), (0.1 * rnd(dim, 4)).to(torch.bfloat16), rnd(1, dim, 4).to(torch.bfloat16)
    g, beta, s0 = -torch.rand(steps, H, D, generator=gen, device="cuda"), torch.sigmoid(rnd(steps, H)).to(torch.bfloat16), 0.1 * rnd(1, H, D, D)

    def run(stream, tickets, cs, st, out):
        for t in range(steps):
            hk.kda_decode_step(x[t], cs, w, None, g[t], beta[t], st, out[t], 1, H, stream=stream, tickets=tickets)
    junk = torch.full((H,), 3, dtype=torch.int32, device="cuda")
    jobs = [(torch.cuda.Stream(), junk if i == 3 else None, cs0.clone(), s0.clone(), torch.zeros(steps, H, D, dtype=torch.bfloat16, device="cuda"))
            for i in range(4)]
    run(None, torch.zeros(H, dtype=torch.int32, device="cuda"), *jobs[0][2:])
    torch.cuda.synchronize()
    for job in jobs[1:]:
        run(*job)
    torch.cuda.synchronize()
    for job in jobs[1:]:
        assert all(torch.equal(a, b) for a, b in zip(job[2:], jobs[0][2:]))
    assert (junk == 3).all()


@pytest.mark.parametrize("H,bsz", [(4, 2), (64, 5)])
def test_decode_layer_vs_oracle(H, bsz):
    """one token through the whole layer, a head per CTA (8 heads) and streamed (320, ragged last round), each stage from the
    stage before it: window and convolution, recurrence and state from the oracle; gates and norm in 64 bits"""
    D, dim = 128, 3 * H * 128
    r = synth.rng(40 + H)
    x32 = r.standard_normal((bsz, dim), dtype=np.float32)
    raw = synth.kda_raw_gates(bsz, H, D, seed=9)
    f, b = raw["f"].reshape(bsz, H, D), raw["b"].reshape(bsz, H)
    w = synth.f32_to_bf16_bits((0.1 * r.standard_normal((dim, 4))).astype(np.float32))
    cst0 = synth.f32_to_bf16_bits(r.standard_normal((bsz, dim, 4), dtype=np.float32))
    s0 = (0.1 * r.standard_normal((bsz, 1, H, D, D), dtype=np.float32)).astype(np.float32)
    nw, go = (1.0 + 0.1 * r.standard_normal(D)).astype(np.float32), r.standard_normal((bsz * H, D), dtype=np.float32)
    cs, st = dev_bf16(cst0), dev(s0)
    out, o32 = (torch.empty(bsz, H, D, dtype=d, device="cuda") for d in (torch.bfloat16, torch.float32))
    y = torch.empty(bsz * H, D, dtype=torch.float32, device="cuda")
    hk.kda_decode_layer(dev(x32), cs, dev_bf16(w), None, dev(f), dev(b), dev(raw["dt_bias"]), dev(raw["a_log"]), raw["lower_bound"], st, out,
                        dev(nw), dev(go), y, bsz, H, epsilon=1e-6, gate_act=1, out_f32=o32)
    torch.cuda.synchronize()
    assert hk.read_device_status() == 0
    x16 = synth.f32_to_bf16_bits(x32).reshape(bsz, dim, 1)
    qkv, o_cs = orc.conv1d_update(x16, cst0, w, None, bsz, dim, 1, 4, 4)
    assert np.array_equal(bits(cs).reshape(-1), o_cs.reshape(-1)), "rolling window"
    sig = lambda v: 1.0 / (1.0 + np.exp(-v.astype(np.float64)))
    g = (raw["lower_bound"] * sig(np.exp(raw["a_log"].astype(np.float64)).reshape(H, 1) * (f + raw["dt_bias"].reshape(H, D)))).astype(np.float32)
    beta = synth.f32_to_bf16_bits(sig(b).astype(np.float32))
    _, want, o_st = orc.kda_recurrent(qkv.reshape(bsz, 1, dim), g.reshape(bsz, 1, H, D), beta.reshape(bsz, 1, H), s0, bsz, 1, H, H, D, D)
    # the fast exponential may flip the last bit (2^-8) of a few of the convolution's and beta's bf16 values: 2e-3 as above
    assert max_rel(o32.cpu().numpy().reshape(want.shape), want) < 2e-3 and frob_rel(st.cpu().numpy(), o_st) < 2e-3
    assert np.array_equal(bits(out), (o32.cpu().numpy().view(np.uint32) >> 16).astype(np.uint16)), "rounded toward zero"
    o = synth.bf16_bits_to_f32(bits(out)).reshape(bsz * H, D).astype(np.float64)
    y64 = o * nw / np.sqrt((o * o).mean(axis=1, keepdims=True) + 1e-6) * sig(go)
    assert max_rel(y.cpu().numpy(), y64) < 1e-5


@pytest.mark.parametrize("Hk,Hv,bsz", [(8, 8, 1), (2, 18, 1), (19, 19, 1), (37, 37, 1), (19, 19, 2), (37, 74, 1)])
@pytest.mark.parametrize("T", [2, 9, 13, 16, 17, 63])
def test_few_chains_walk_to_the_same_bits(T, Hk, Hv, bsz):
    """eight, four and two CTAs a chain, either side of the batches of eight tokens and of the head counts where the split changes, a
    state of zeros among them, against the kernel that states off the 16-byte boundary take: same bits"""
    D = 128
    gen = torch.Generator(device="cuda").manual_seed(100 * T + Hv)
    qkv = torch.randn(bsz, T, (2 * Hk + Hv) * D, generator=gen, device="cuda").to(torch.bfloat16)
    qkv[:, ::3, :7] = 0
    g, beta = -5 * torch.rand(bsz, T, Hv, D, generator=gen, device="cuda"), torch.rand(bsz, T, Hv, generator=gen, device="cuda").to(torch.bfloat16)
    s0 = 0.1 * torch.randn(bsz, 1, Hv, D, D, generator=gen, device="cuda")
    s0[:, :, 0] = 0
    slots = torch.arange(bsz - 1, -1, -1, dtype=torch.int32, device="cuda")
    res = []
    for off in (0, 1):
        st = torch.empty(s0.numel() + 4, device="cuda")[off:off + s0.numel()].view(s0.shape)
        st.copy_(s0)
        out, o32 = torch.empty(bsz, T, Hv, D, dtype=torch.bfloat16, device="cuda"), torch.empty(bsz, T, Hv, D, device="cuda")
        hk.cuda_recurrent_gated_delta_rule(qkv, g, beta, st, out, bsz, T, Hk, Hv, D, D, 1, slots, True, False, out_f32=o32, force_recurrent=True)
        torch.cuda.synchronize()
        res.append([bits(out), o32.cpu().numpy().view(np.int32), st.cpu().numpy().view(np.int32)])
    for a, b in zip(*res):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("H,bsz", [(4, 1), (40, 2), (64, 5)])
def test_states_off_the_16_byte_boundary(H, bsz):
    """a state that starts on any fp32 element: the scalar forms (decode step and layer; 1, 3 and 9 tokens of the recurrence; no
    streaming) against the same call on an aligned copy, bit for bit"""
    D, dim, T = 128, 3 * H * 128, 9
    gen = torch.Generator(device="cuda").manual_seed(H)

    def rnd(*shape):
        return torch.randn(*shape, generator=gen, device="cuda")
    n = bsz * H * D * D
    buf, qkv, g = 0.1 * rnd(n + 1), rnd(bsz, T, dim).to(torch.bfloat16), -torch.rand(bsz, T, H, D, generator=gen, device="cuda")
    beta, cs0, w = torch.sigmoid(rnd(bsz, T, H)).to(torch.bfloat16), rnd(bsz, dim, 4).to(torch.bfloat16), (0.1 * rnd(dim, 4)).to(torch.bfloat16)
    x32, nw, go, a_log, dtb = rnd(bsz, dim), 1.0 + 0.1 * rnd(D), rnd(bsz * H, D), rnd(H) * 0.3, rnd(H, D)

    def run(st):
        res = []
        for t in (1, 3, 9):
            out = torch.empty(bsz, t, H, D, dtype=torch.bfloat16, device="cuda")
            hk.cuda_recurrent_gated_delta_rule(qkv[:, :t].contiguous(), g[:, :t].contiguous(), beta[:, :t].contiguous(), st, out, bsz, t, H, H,
                                               D, D, 1, None, True, False)
            res.append(out)
        cs, out, y = cs0.clone(), torch.empty(2, bsz, H, D, dtype=torch.bfloat16, device="cuda"), torch.empty(bsz * H, D, device="cuda")
        hk.kda_decode_step(qkv[:, 0].contiguous(), cs, w, None, g[:, 0].contiguous(), beta[:, 0].contiguous(), st, out[0], bsz, H)
        hk.kda_decode_layer(x32, cs, w, None, g[:, 1].contiguous(), rnd(bsz, H) * 0, dtb, a_log, -5.0, st, out[1], nw, go, y, bsz, H)
        torch.cuda.synchronize()
        return res + [cs, out, y, st.clone()]
    aligned, off = buf[1:].clone(), buf[1:]
    assert aligned.data_ptr() % 16 == 0 and off.data_ptr() % 16 == 4
    for a, b in zip(run(aligned), run(off)):
        assert torch.equal(a, b)


def test_an_explicit_stream_is_the_one_that_runs():
    """the binding's stream argument: a call given a side stream waits for that stream's earlier work, not for the current one's"""
    S, F = 64, 256
    src, dst, side = torch.zeros(S, F, device="cuda"), torch.zeros(F, S, dtype=torch.bfloat16, device="cuda"), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(side):
        torch.cuda._sleep(20_000_000)                          # about 10 ms
        src.fill_(3.0)
    hk.kda_transpose_cast(dst, src, S, F, stream=side)
    side.synchronize()
    assert (dst == 3.0).all()
    with pytest.raises(AttributeError):
        hk.kda_transpose_cast(dst, src, S, F, stream=1)
    with pytest.raises(TypeError):
        hk.gated_rms_norm(dst, src.int(), src, src, S, F, 1e-6)


@pytest.mark.parametrize("T,H,bsz", [(130, 4, 3), (3000, 1, 1)])
def test_chunked_prefill_without_the_tensor_map_encoder(T, H, bsz):
    """both chunked entry points are served token by token where the encoder is missing (here: switched off in a child process), with the
    bits of the gate kernel and the token-by-token recurrence; 3,000 tokens of one head are more gates than the workspace holds"""
    D, r = 128, synth.rng(T)
    raw = synth.kda_raw_gates(T, H, D, seed=T)
    case = {"qkv": r.standard_normal((bsz, T, 3 * H * D), dtype=np.float32), "s0": 0.1 * r.standard_normal((bsz, 1, H, D, D), dtype=np.float32),
            "f": np.broadcast_to(raw["f"], (bsz, T, H, D)).copy(), "b": r.standard_normal((bsz, T, H), dtype=np.float32),
            "dt": raw["dt_bias"], "al": raw["a_log"]}
    t = {k: dev(v.astype(np.float32)) for k, v in case.items()}
    qkv, g = t["qkv"].to(torch.bfloat16), torch.empty(bsz, T, H, D, device="cuda")
    beta, slots = torch.empty(bsz, T, H, dtype=torch.bfloat16, device="cuda"), torch.arange(bsz - 1, -1, -1, dtype=torch.int32, device="cuda")
    for i in range(bsz):
        hk.kda_gate(t["b"][i], t["f"][i], t["dt"], t["al"], -5.0, beta[i], g[i], T, H, D)
    want = []
    for sl in (None, slots):
        st, out, o32 = t["s0"].clone(), torch.empty(bsz, T, H, D, dtype=torch.bfloat16, device="cuda"), torch.empty(bsz, T, H, D, device="cuda")
        hk.cuda_recurrent_gated_delta_rule(qkv, g, beta, st, out, bsz, T, H, H, D, D, 1, sl, True, False, out_f32=o32, force_recurrent=True)
        torch.cuda.synchronize()
        want += [x.cpu() for x in (st, out, o32)]
    code = """
import sys, torch
import helios_glm53flash_b200 as hk
d = torch.load(sys.argv[1])
bsz, T, H, D = d["g"].shape
c = {k: v.cuda() for k, v in d.items()}
res = []
for gated in (False, True):
    for sl in (None, c["slots"]):
        st, out, o32 = c["s0"].clone(), torch.empty(bsz, T, H, D, dtype=torch.bfloat16, device="cuda"), torch.empty(bsz, T, H, D, device="cuda")
        if gated:
            hk.kda_chunked_prefill_gated(c["qkv"], c["f"], c["b"], c["dt"], c["al"], -5.0, st, out, bsz, T, H, slots=sl, out_f32=o32)
        else:
            hk.cuda_recurrent_gated_delta_rule(c["qkv"], c["g"], c["beta"], st, out, bsz, T, H, H, D, D, 1, sl, True, False, out_f32=o32)
        torch.cuda.synchronize()
        res += [x.cpu() for x in (st, out, o32)]
torch.save(res, sys.argv[2])
"""
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    with tempfile.TemporaryDirectory() as d:
        torch.save({"qkv": qkv.cpu(), "g": g.cpu(), "beta": beta.cpu(), "slots": slots.cpu(), **{k: t[k].cpu() for k in ("s0", "f", "b", "dt", "al")}},
                   os.path.join(d, "in.pt"))
        res = subprocess.run([sys.executable, "-c", code, os.path.join(d, "in.pt"), os.path.join(d, "out.pt")], cwd=root, capture_output=True,
                             text=True, timeout=300, env=dict(os.environ, HK_KDA_NO_TMA="1"))
        assert res.returncode == 0, res.stderr[-2000:]
        got = torch.load(os.path.join(d, "out.pt"))
    assert len(got) == 2 * len(want)
    for a, b in zip(got, want + want):
        assert torch.equal(a, b)
