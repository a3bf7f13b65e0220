"""Performance cases of the trunk-attention path: what a serving engine has this library do, layer by layer and token by token.

Every case goes through the public entry points of the package, as the engine's layer loop calls them, with the workspaces and
work buffers that such a program keeps.  Kinds of case:

  kda_decode     the KDA layer of one new token for each of `batch` sequences, from the projections' fp32 rows to the normalised
                 fp16 activations (one call)
  kda_prefill    the KDA layer over `tokens` tokens of `batch` sequences.  form "fused": cast + convolution, prefill that forms
                 its own gates, gated norm.  form "launchers": the call sequence of an engine that knows only the launchers
                 (transpose + cast, gate preparation, convolution, recurrence, gated norm)
  mla_layer      the sparse MLA layer over `rows` new tokens behind a context of `ctx` tokens: cache append, indexer keys, absorbed
                 query projection, selection of 512 pools, attention over the selected latents, absorbed output projection
  dsa            selection and attention alone, for a few decode rows, with bf16 or fp16 indexer keys
  dense_decode   dense MLA attention of `batch` sequences' new tokens over their concatenated caches
  dense_prefill  dense causal MLA attention of a chunk of `rows` tokens appended to a cache of `ctx` latents
  trunk_decode   one decode step of the whole trunk: 34 KDA and 11 MLA layers

Inputs are drawn on the GPU from the seed, with the distributions of the benchmark configurations.
"""
import math

import torch

import helios_glm53flash_b200 as hk
from helios_glm53flash_b200.trunk import TrunkAttention

D = 128                  # KDA head width, indexer head width
LAT = 512                # latent width
MLA_HEADS, NOPE, IDX_HEADS = 64, 256, 32
TOPK, KIDX = 512, 2052   # selected pools; their tokens and the 4 newest
IDX_BLOCK = 1024         # rows scored and selected at a time in a prefill chunk
N_KDA, N_MLA = 34, 11
LOWER_BOUND = -5.0
STEPS = 64               # decode positions that a state walks through before it starts over


def listed():
    return [
        # one user's next token through one KDA layer: the smallest call there is
        {"name": "kda_decode_1x32", "kind": "kda_decode", "batch": 1, "heads": 32},
        # a full decode batch at the 64 heads of an unsharded layer: 100 MB of state in and out
        {"name": "kda_decode_24x64", "kind": "kda_decode", "batch": 24, "heads": 64},
        # a short message, shorter than one 64-token chunk, in an engine that calls the launchers
        {"name": "kda_prefill_37x64", "kind": "kda_prefill", "batch": 1, "tokens": 37, "heads": 64, "form": "launchers"},
        # a page of prompt of no round length
        {"name": "kda_prefill_1003x32", "kind": "kda_prefill", "batch": 1, "tokens": 1003, "heads": 32, "form": "fused"},
        # the 32K-token prompt of the headline benchmark, through the launchers
        {"name": "kda_prefill_32768x32", "kind": "kda_prefill", "batch": 1, "tokens": 32768, "heads": 32, "form": "launchers"},
        # a 4,096-token chunk of eight sequences at a time
        {"name": "kda_prefill_8x4096x32", "kind": "kda_prefill", "batch": 8, "tokens": 4096, "heads": 32, "form": "fused"},
        # the next token of a chat of a few thousand tokens through one MLA layer
        {"name": "mla_layer_1_at_5001", "kind": "mla_layer", "rows": 1, "ctx": 5001},
        # a prefill chunk of a 32K-token prompt through one MLA layer
        {"name": "mla_layer_4096_at_28672", "kind": "mla_layer", "rows": 4096, "ctx": 28672},
        # a decode step's selection and sparse attention at 262,144 tokens of context, bf16 indexer keys
        {"name": "dsa_1_at_262144", "kind": "dsa", "rows": 1, "ctx": 262144, "keys": "bf16"},
        # dense decode of eight sequences of up to 32K tokens, each of its own length
        {"name": "dense_decode_8x32768", "kind": "dense_decode", "batch": 8, "ctx": 32768, "ragged": True},
        # a 4,096-token chunk appended to a 32K cache, dense
        {"name": "dense_prefill_4096_at_32768", "kind": "dense_prefill", "rows": 4096, "ctx": 32768},
        # the whole trunk's next token at the full context
        {"name": "trunk_decode_at_262144", "kind": "trunk_decode", "ctx": 262144},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["kda_decode", "kda_prefill", "kda_prefill", "mla_layer", "mla_layer", "dsa", "dense_decode", "dense_prefill",
                       "trunk_decode"])
    if kind == "kda_decode":
        heads = rng.choice([8, 16, 32, 64])          # 64 and 32: whole layers; 8 and 16: a layer sharded by heads
        return {"kind": kind, "batch": _log(rng, 1, 1536 // heads), "heads": heads}
    if kind == "kda_prefill":
        heads, batch = rng.choice([8, 16, 32, 64]), rng.choice([1, 1, 1, 2, 3, 4, 8])
        tokens = _log(rng, 2, 32768 * 32 // (max(heads, 32) * batch))
        form = "launchers" if tokens < 64 or rng.random() < 0.5 else "fused"
        return {"kind": kind, "batch": batch, "tokens": tokens, "heads": heads, "form": form}
    if kind == "mla_layer":
        rows = rng.choice([1, 1, _log(rng, 2, 8), _log(rng, 9, 4096), _log(rng, 9, 4096)])
        return {"kind": kind, "rows": rows, "ctx": _log(rng, 512, 262144)}
    if kind == "dsa":
        return {"kind": kind, "rows": _log(rng, 1, 8), "ctx": _log(rng, 512, 262144), "keys": rng.choice(["bf16", "fp16"])}
    if kind == "dense_decode":
        batch = _log(rng, 1, 16)
        return {"kind": kind, "batch": batch, "ctx": _log(rng, 100, 262144 // batch), "ragged": rng.random() < 0.7}
    if kind == "dense_prefill":
        return {"kind": kind, "rows": _log(rng, 2, 4096), "ctx": rng.choice([0, _log(rng, 16, 32768), _log(rng, 16, 32768)])}
    return {"kind": kind, "ctx": _log(rng, 2048, 262144)}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(gen, *shape, dtype=torch.float32, scale=1.0):
    t = torch.empty(shape, dtype=dtype, device="cuda").normal_(generator=gen)
    return t.mul_(scale) if scale != 1.0 else t


def _empty(*shape, dtype):
    return torch.empty(shape, dtype=dtype, device="cuda")


def _kda_weights(gen, s, heads):
    dim = 3 * heads * D
    s["conv_w"] = _randn(gen, dim, 4, scale=0.1).to(torch.bfloat16)
    s["dt_bias"] = _randn(gen, heads, D, scale=0.5)
    s["a_log"] = torch.empty(heads, device="cuda").uniform_(math.log(0.5), math.log(4.0), generator=gen)
    s["norm_w"] = (1.0 + _randn(gen, D, scale=0.05)).to(torch.bfloat16)


def _kda_state(gen, s, batch, heads):
    """windows and states of sequences that are under way"""
    s["conv_state"] = _randn(gen, batch, 3 * heads * D, 4, dtype=torch.bfloat16)
    s["rec_state"] = _randn(gen, batch, 1, heads, D, D, scale=0.1)


def _prepare_kda_decode(case, gen):
    B, H = case["batch"], case["heads"]
    s = {"B": B, "H": H, "x": _randn(gen, B, 3 * H * D), "f": _randn(gen, B, H, D), "b": _randn(gen, B, H),
         "gate_out": _randn(gen, B * H, D), "out": _empty(B, H, D, dtype=torch.bfloat16), "y": _empty(B * H, D, dtype=torch.float16),
         "tickets": torch.zeros(2 * B * H, dtype=torch.int32, device="cuda")}
    _kda_weights(gen, s, H)
    _kda_state(gen, s, B, H)
    return s


def _run_kda_decode(s):
    hk.kda_decode_layer(s["x"], s["conv_state"], s["conv_w"], None, s["f"], s["b"], s["dt_bias"], s["a_log"], LOWER_BOUND,
                        s["rec_state"], s["out"], s["norm_w"], s["gate_out"], s["y"], s["B"], s["H"], tickets=s["tickets"])
    return {"out": s["out"], "y": s["y"], "conv_state": s["conv_state"], "rec_state": s["rec_state"]}


def _prepare_kda_prefill(case, gen):
    B, T, H = case["batch"], case["tokens"], case["heads"]
    dim, bf = 3 * H * D, torch.bfloat16
    s = {"B": B, "T": T, "H": H, "dim": dim, "form": case["form"], "x": _randn(gen, B, T, dim), "f": _randn(gen, B, T, H, D),
         "b": _randn(gen, B, T, H), "gate_out": _randn(gen, B * T * H, D), "qkv": _empty(B, T, dim, dtype=bf),
         "out": _empty(B, T, H, D, dtype=bf), "y": _empty(B * T * H, D, dtype=torch.float16),
         "ws": _empty(max(256, hk.kda_chunked_workspace_bytes(B, T, H)), dtype=torch.uint8)}
    if case["form"] == "launchers":
        s["mixed"], s["g"], s["beta"] = _empty(B, dim, T, dtype=bf), _empty(B, T, H, D, dtype=torch.float32), _empty(B, T, H, dtype=bf)
    _kda_weights(gen, s, H)
    _kda_state(gen, s, B, H)
    return s


def _run_kda_prefill(s):
    B, T, H, dim = s["B"], s["T"], s["H"], s["dim"]
    if s["form"] == "fused":
        hk.kda_cast_conv(s["x"], s["conv_state"], None, s["conv_w"], None, s["qkv"], B, dim, T, True)
        hk.kda_chunked_prefill_gated(s["qkv"], s["f"], s["b"], s["dt_bias"], s["a_log"], LOWER_BOUND, s["rec_state"], s["out"], B, T, H,
                                     workspace=s["ws"])
    else:
        for i in range(B):
            hk.kda_transpose_cast(s["mixed"][i], s["x"][i], T, dim)
            hk.kda_gate(s["b"][i], s["f"][i], s["dt_bias"], s["a_log"], LOWER_BOUND, s["beta"][i], s["g"][i], T, H, D)
        hk.cuda_causal_conv1d_update(s["mixed"], s["conv_state"], None, s["conv_w"], None, s["qkv"], B, dim, T, 4, 4, True, False)
        hk.cuda_recurrent_gated_delta_rule(s["qkv"], s["g"], s["beta"], s["rec_state"], s["out"], B, T, H, H, D, D, 1, None, True, False,
                                           workspace=s["ws"])
    hk.gated_rms_norm(s["out"], s["norm_w"], s["y"], s["gate_out"], B * T * H, D, 1e-6, gate_act=1)
    return {"out": s["out"], "y": s["y"], "conv_state": s["conv_state"], "rec_state": s["rec_state"]}


def _prepare_mla_layer(case, gen):
    n, ctx, f16 = case["rows"], case["ctx"], torch.float16
    cap = (ctx + max(n, STEPS) + 7) // 4 * 4
    block = min(n, IDX_BLOCK)
    ns = hk.mla_auto_splits(n, KIDX)
    return {"n": n, "ctx": ctx, "step": 0,
            "ckv": _randn(gen, cap, LAT, dtype=f16), "pool": _randn(gen, cap // 4, D, dtype=f16), "ring": _randn(gen, n + 4, 2 * D, dtype=f16),
            "kv_pre": _randn(gen, n, LAT), "ln_w": 1.0 + _randn(gen, LAT, dtype=f16, scale=0.05), "idx_k": _randn(gen, n, D, dtype=f16),
            "idx_g": _randn(gen, n, D, dtype=f16), "knorm_w": 1.0 + _randn(gen, D, dtype=f16, scale=0.05),
            "knorm_b": _randn(gen, D, dtype=f16, scale=0.05), "ape": _randn(gen, 4, D, scale=0.1),
            "q_nope": _randn(gen, n, MLA_HEADS, NOPE, dtype=f16, scale=0.5), "q_idx": _randn(gen, n, IDX_HEADS, D, dtype=f16),
            "w": _randn(gen, n, IDX_HEADS, dtype=f16), "kv_b": _randn(gen, MLA_HEADS * 2 * NOPE, LAT, dtype=f16, scale=0.04),
            "q_pos": torch.arange(ctx, ctx + n, dtype=torch.int32, device="cuda"),
            "idx_kn": _empty(n, D, dtype=f16), "q_lat": _empty(n, MLA_HEADS, LAT, dtype=f16), "scores": _empty(block, cap // 4, dtype=f16),
            "topk": _empty(n, TOPK, dtype=torch.int32), "raw": _empty(n, KIDX, dtype=torch.int32),
            "lat": _empty(n, MLA_HEADS, LAT, dtype=f16), "o": _empty(n, MLA_HEADS, NOPE, dtype=f16),
            "ws": _empty(max(256, hk.mla_partial_bytes(ns, n * MLA_HEADS)), dtype=torch.uint8)}


def _run_mla_layer(s):
    n, pos = s["n"], s["ctx"]
    if n == 1:
        pos += s["step"]                             # a decoded token: the next position
        s["step"] = (s["step"] + 1) % STEPS
        hk.mla_decode_prologue(s["kv_pre"], s["ln_w"], s["ckv"], 1e-6, s["idx_k"], s["knorm_w"], s["knorm_b"], s["idx_kn"], 1e-5, s["idx_g"],
                               s["ring"], n + 4, s["pool"], s["ape"], pos, q_pos_out=s["q_pos"])
    else:
        hk.mla_cache_append(s["kv_pre"], s["ln_w"], s["ckv"], pos, n, 1e-6)
        hk.layernorm_f16(s["idx_k"], s["knorm_w"], s["knorm_b"], s["idx_kn"], n, D, 1e-5)
        hk.kpool_write(s["idx_kn"], s["idx_g"], s["ring"], n + 4, s["pool"], s["ape"], pos, n)
    hk.q_latent(s["q_nope"], s["kv_b"], s["q_lat"], n)
    npools = (pos + n) // 4
    k = min(TOPK, npools)
    if n <= 8:
        hk.indexer_select(s["q_idx"], s["pool"], s["w"], s["q_pos"], s["scores"], s["topk"], s["raw"], n, npools, k=k)
    else:
        for i in range(0, n, IDX_BLOCK):
            e = min(n, i + IDX_BLOCK)
            hk.indexer_score(s["q_idx"][i:e], s["pool"], s["w"][i:e], s["q_pos"][i:e], s["scores"], e - i, npools)
            hk.dsa_topk(s["scores"], npools, s["topk"][i:e], e - i, npools, k, TOPK)
        hk.pool_expand_row(s["topk"], s["q_pos"], s["raw"], n)
    hk.mla_sparse_decode(s["q_lat"], s["ckv"], s["raw"], KIDX, s["lat"], n, workspace=s["ws"])
    hk.o_absorb(s["lat"], s["kv_b"], s["o"], n)
    return {"o": s["o"], "lat": s["lat"], "topk": s["topk"], "raw": s["raw"], "ckv": s["ckv"], "pool": s["pool"], "ring": s["ring"]}


def _prepare_dsa(case, gen):
    m, ctx = case["rows"], case["ctx"]
    keys = torch.bfloat16 if case["keys"] == "bf16" else torch.float16
    ns = hk.mla_auto_splits(m, KIDX)
    return {"m": m, "npools": ctx // 4, "pool": _randn(gen, ctx // 4, D, dtype=keys), "q_idx": _randn(gen, m, IDX_HEADS, D, dtype=keys),
            "w": _randn(gen, m, IDX_HEADS, dtype=keys), "q_pos": torch.arange(ctx - m, ctx, dtype=torch.int32, device="cuda"),
            "ckv": _randn(gen, ctx, LAT, dtype=torch.float16), "q_lat": _randn(gen, m, MLA_HEADS, LAT, dtype=torch.float16),
            "scores": _empty(m, ctx // 4, dtype=torch.float16), "topk": _empty(m, TOPK, dtype=torch.int32),
            "raw": _empty(m, KIDX, dtype=torch.int32), "lat": _empty(m, MLA_HEADS, LAT, dtype=torch.float16),
            "ws": _empty(max(256, hk.mla_partial_bytes(ns, m * MLA_HEADS)), dtype=torch.uint8)}


def _run_dsa(s):
    hk.indexer_select(s["q_idx"], s["pool"], s["w"], s["q_pos"], s["scores"], s["topk"], s["raw"], s["m"], s["npools"],
                      k=min(TOPK, s["npools"]))
    hk.mla_sparse_decode(s["q_lat"], s["ckv"], s["raw"], KIDX, s["lat"], s["m"], scale=LAT ** -0.5, workspace=s["ws"])
    return {"lat": s["lat"], "topk": s["topk"], "raw": s["raw"]}


def _lengths(case):
    """cache lengths of a decode batch: all alike, or spread between half and the whole of ctx"""
    B, L = case["batch"], case["ctx"]
    return [L - (i * L) // (2 * B) if case["ragged"] else L for i in range(B)]


def _prepare_dense_decode(case, gen):
    lens = _lengths(case)
    B, base = len(lens), [sum(lens[:i]) for i in range(len(lens))]
    ns = hk.mla_auto_splits(B, max(lens))
    return {"B": B, "hint": max(lens), "ckv": _randn(gen, sum(lens), LAT, dtype=torch.float16),
            "q": _randn(gen, B, MLA_HEADS, LAT, dtype=torch.float16), "base": torch.tensor(base, dtype=torch.int64, device="cuda"),
            "len": torch.tensor(lens, dtype=torch.int32, device="cuda"), "lat": _empty(B, MLA_HEADS, LAT, dtype=torch.float16),
            "ws": _empty(max(256, hk.mla_partial_bytes(ns, B * MLA_HEADS)), dtype=torch.uint8)}


def _run_dense_decode(s):
    hk.mla_dense_prefill(s["q"], s["ckv"], s["lat"], s["B"], 0, scale=LAT ** -0.5, kv_base=s["base"], kv_len=s["len"], workspace=s["ws"],
                         n_keys_hint=s["hint"])
    return s["lat"]


def _prepare_dense_prefill(case, gen):
    n, ctx = case["rows"], case["ctx"]
    ns = hk.mla_auto_splits(n, ctx + n)
    return {"n": n, "ctx": ctx, "ckv": _randn(gen, ctx + n, LAT, dtype=torch.float16), "q": _randn(gen, n, MLA_HEADS, LAT, dtype=torch.float16),
            "lat": _empty(n, MLA_HEADS, LAT, dtype=torch.float16),
            "ws": _empty(max(256, hk.mla_partial_bytes(ns, n * MLA_HEADS)), dtype=torch.uint8)}


def _run_dense_prefill(s):
    hk.mla_dense_prefill(s["q"], s["ckv"], s["lat"], s["n"], s["ctx"], scale=LAT ** -0.5, workspace=s["ws"])
    return s["lat"]


def _prepare_trunk_decode(case, gen):
    ctx = case["ctx"]
    tr = TrunkAttention(n_kda=N_KDA, n_mla=N_MLA, heads=32, batch=1, max_ctx=(ctx + STEPS + 7) // 4 * 4, max_chunk=64, seed=gen.initial_seed())
    # one arena per kind of plane, filled with what a sequence under way has left there
    arenas = {"rec_state": _randn(gen, N_KDA, *tr.rec_state[0].shape, scale=0.1),
              "conv_state": _randn(gen, N_KDA, *tr.conv_state[0].shape, dtype=torch.bfloat16),
              "ckv": _randn(gen, N_MLA, *tr.ckv[0][0].shape, dtype=torch.float16), "pool": _randn(gen, N_MLA, *tr.pool[0][0].shape, dtype=torch.float16)}
    tr.rec_state, tr.conv_state = list(arenas["rec_state"]), list(arenas["conv_state"])
    tr.ckv, tr.pool = [list(arenas["ckv"])], [list(arenas["pool"])]
    return {"tr": tr, "ctx": ctx, "step": 0, **arenas}


def _run_trunk_decode(s):
    tr = s["tr"]
    tr.run_chunk(s["ctx"] + s["step"], 1)
    s["step"] = (s["step"] + 1) % STEPS
    return {"y": tr.kda_y[:tr.H], "o": tr.o_abs[:1], "topk": tr.topk[:1], "rec_state": s["rec_state"], "conv_state": s["conv_state"],
            "ckv": s["ckv"], "pool": s["pool"]}


_PREPARE = {"kda_decode": _prepare_kda_decode, "kda_prefill": _prepare_kda_prefill, "mla_layer": _prepare_mla_layer, "dsa": _prepare_dsa,
            "dense_decode": _prepare_dense_decode, "dense_prefill": _prepare_dense_prefill, "trunk_decode": _prepare_trunk_decode}
_RUN = {"kda_decode": _run_kda_decode, "kda_prefill": _run_kda_prefill, "mla_layer": _run_mla_layer, "dsa": _run_dsa,
        "dense_decode": _run_dense_decode, "dense_prefill": _run_dense_prefill, "trunk_decode": _run_trunk_decode}


def prepare(case, seed):
    return {**_PREPARE[case["kind"]](case, _gen(seed)), "run": _RUN[case["kind"]]}


def run(state):
    return state["run"](state)


# ---- what a pass cannot do without ----
def _kda_work(rows, batch, heads):
    """`rows` tokens of all sequences together: fp32 projections and gates in, bf16 recurrence outputs and fp16 activations out, the
    states in and out; 4 * 128 * 128 multiply-adds of the delta rule per token and head"""
    per_row = heads * (3 * D * 4 + D * 4 + 4 + D * 4 + D * 2 + D * 2)
    state = 2 * batch * heads * (D * D * 4 + 3 * D * 4 * 2)
    weights = heads * (3 * D * 4 * 2 + D * 4 + 4)
    return rows * per_row + state + weights, rows * heads * 2 * 4 * D * D


def _select_work(rows, npools, visible):
    """pooled keys and queries in, selected pools and tokens out; `visible` (row, pool) pairs are scored"""
    return npools * D * 2 + rows * IDX_HEADS * (D + 1) * 2 + rows * (TOPK + KIDX) * 4, visible * IDX_HEADS * D * 2


def _attend_work(rows, keys_read, pairs):
    """`keys_read` latents in, queries in, outputs out; `pairs` (row, key) pairs are attended by all heads"""
    return keys_read * LAT * 2 + 2 * rows * MLA_HEADS * LAT * 2, pairs * MLA_HEADS * LAT * 4


def _mla_layer_work(n, ctx):
    npools = (ctx + n) // 4
    visible = sum((ctx + i + 1) // 4 for i in range(n))
    attended = [min(KIDX, ctx + i + 1) for i in range(n)]
    sel = _select_work(n, npools, visible)
    att = _attend_work(n, min(ctx + n, sum(attended)), sum(attended))
    absorb_bytes = MLA_HEADS * 2 * NOPE * LAT * 2 + 2 * n * MLA_HEADS * NOPE * 2
    append = n * (LAT * 4 + LAT * 2 + 2 * D * 2 + 2 * D * 2)
    return sel[0] + att[0] + absorb_bytes + append, sel[1] + att[1] + 2 * n * MLA_HEADS * NOPE * LAT * 2


def work(case):
    kind = case["kind"]
    if kind == "kda_decode":
        nbytes, flops = _kda_work(case["batch"], case["batch"], case["heads"])
    elif kind == "kda_prefill":
        nbytes, flops = _kda_work(case["batch"] * case["tokens"], case["batch"], case["heads"])
    elif kind == "mla_layer":
        nbytes, flops = _mla_layer_work(case["rows"], case["ctx"])
    elif kind == "dsa":
        m, ctx = case["rows"], case["ctx"]
        sel = _select_work(m, ctx // 4, m * (ctx // 4))
        att = _attend_work(m, min(ctx, m * KIDX), m * min(KIDX, ctx))
        nbytes, flops = sel[0] + att[0], sel[1] + att[1]
    elif kind == "dense_decode":
        keys = sum(_lengths(case))
        nbytes, flops = _attend_work(case["batch"], keys, keys)
    elif kind == "dense_prefill":
        n, ctx = case["rows"], case["ctx"]
        nbytes, flops = _attend_work(n, ctx + n, n * ctx + n * (n + 1) // 2)
    else:
        kda, mla = _kda_work(1, 1, 32), _mla_layer_work(1, case["ctx"])
        shared = MLA_HEADS * 2 * NOPE * LAT * 2      # the layers of a kind share one set of synthetic weights
        nbytes = N_KDA * kda[0] + N_MLA * (mla[0] - shared) + shared
        flops = N_KDA * kda[1] + N_MLA * mla[1]
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """bf16 outputs (rounded toward zero) and fp16 tensor-core operands in the KDA prefill, bf16 outputs of fp32 arithmetic in its
    decode step, fp16 softmax weights and outputs in the attention.  Selections and positions are whole numbers and stay the same."""
    if case["kind"] == "kda_prefill":
        return {"rel": 1e-2}
    if case["kind"] in ("kda_decode", "trunk_decode"):
        return {"rel": 4e-3}
    return {"rel": 2e-3}
