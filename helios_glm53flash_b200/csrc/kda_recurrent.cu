// KDA / gated-delta-rule recurrence, one token at a time: the decode step, short sequences and the
// history (rewindable) mode.  Interface and arithmetic of
// helios::aux::cuda_recurrent_gated_delta_rule (reference: src/cuda/aux/gdn.cu:555-866).
//
// Kernels:
//   kda_decode_kernel, kda_decode_stream_kernel   one token per sequence (the decode step, the decode layer, the recurrence alone)
//   kda_recurrent_few_kernel, kda_recurrent_cols_kernel   several tokens, channelwise decay, no history: few chains; others
//   kda_recurrent_rows_kernel                     channelwise decay with a history, and a few tokens of many chains
//   kda_recurrent_kernel                          one decay per head, 128- and 64-wide heads
// The state lives in REGISTERS for the whole call (the reference re-reads and re-writes it from global memory on every token),
// so a call moves each state byte once in and once out, the HBM floor of 2*H*D*D*4 bytes.
//
// Channelwise decay: ONE arithmetic for all kernels, so that a token gives the same bits whichever kernel it takes - alone or
// with others in a call, with or without a history, by launcher, decode step or decode layer:
//   S_c = S_c d_c;  kv = sum k_c S_c;  u = (v - kv) beta;  S_c = fma(k_c, u, S_c);  o = sum q_c S_c
// (k_c d_c against the undecayed state, which is then rounded once per token, was no better: errors against 64 bits 2-6 % larger at
// the model's gates, short prompts 2 % longer).  A sum over the 128 state rows is taken in 16 groups, group rg = the 4-row chunks rg and
// rg + 16; a group runs over its even and its odd rows separately (the two halves of a packed fp32 pair), ascending; groups rg
// and rg + 8 are added first, then the 8 sums as a balanced tree.  Norms: inv_norm.
// One decay per head: 4 or 8 ascending row groups; for 128 x 32 slices that is the reference's 4 x 32 order (gdn.cu:683-705).
#include <algorithm>

#include "hk_common.cuh"
#include "kda_norm_common.cuh"
#include "tc05.cuh"

namespace hk {

__device__ __forceinline__ float tree8(float a0, float a1, float a2, float a3, float a4, float a5, float a6, float a7) {
  return __fadd_rn(__fadd_rn(__fadd_rn(a0, a1), __fadd_rn(a2, a3)), __fadd_rn(__fadd_rn(a4, a5), __fadd_rn(a6, a7)));
}
// 128 channels of one token in one warp, channel lane + 32 u in x[u]: 1 / |x|
__device__ __forceinline__ float inv_norm(const float (&x)[4]) {
  float s = 0.f;
#pragma unroll
  for (int u = 0; u < 4; u++) s = fmaf(x[u], x[u], s);
  return rsqrtf(warp_sum(s) + 1e-6f);
}

// ---------------------------------------------------------------------------------------------
// Channelwise decay, 128-wide heads: history mode, states with room for one, and a few tokens of many chains.  One CTA per
// (batch item, head, slice of NV value-columns); thread (kg, j) owns column j and the 16 / KG row groups of the shared order that
// make up kg's part of the balanced tree.  Three warps prepare a token (q with its norm; k with its norm; the decay).
// What bounds it: for few tokens the state in and out, in runs of 128 bytes; for many the three barriers of a token.  With the
// head-wide kernel's order below, every warp in the norms and four barriers: 3 tokens of 32 chains 5.0 us, now 4.2; 6 of 1,536
// 91 -> 69; 7 of 64 with history 13.1 -> 10.6; 63 of 8 with history 52 -> 36.
// ---------------------------------------------------------------------------------------------
template <int NV, bool HIST>
__global__ __launch_bounds__(128) void kda_recurrent_rows_kernel(
    const __nv_bfloat16* __restrict__ mixed_qkv, const float* __restrict__ g, const __nv_bfloat16* __restrict__ beta,
    float* __restrict__ state, __nv_bfloat16* __restrict__ out, float* __restrict__ out_f32, int seqlen, int Hk, int Hv, float scale,
    const int* __restrict__ slots, int history_stride) {
  constexpr int D = 128, KG = 128 / NV, PAIRS = 8 / KG, RPT = D / KG;    // thread groups; pairs of row groups and rows per thread
  const int b = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * NV;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, j = tid % NV, kg = tid / NV;
  const int k_head = head / (Hv / Hk);
  const size_t row = (size_t)2 * Hk * D + (size_t)Hv * D, state_size = (size_t)Hv * D * D;
  float* my_state = state + (size_t)(slots ? slots[b] : b) * history_stride * state_size + (size_t)head * D * D + v0 + j;
  const __nv_bfloat16* tok = mixed_qkv + (size_t)b * seqlen * row;
  const float* gp = g + ((size_t)b * seqlen * Hv + head) * D;
  const __nv_bfloat16* bp = beta + (size_t)b * seqlen * Hv + head;
  const size_t out_base = ((size_t)b * seqlen * Hv + head) * D + v0 + j;
  __shared__ __align__(16) float sh_q[D], sh_k[D], sh_d[D];
  __shared__ float sh_part[2][KG][NV];

  // row e of this thread's group i: groups PAIRS kg ... and the same 8 further on
  auto row_of = [&](int i, int e) { return 4 * (PAIRS * kg + i % PAIRS + 8 * (i / PAIRS) + 16 * (e >> 2)) + (e & 3); };
  float S[RPT];
#pragma unroll
  for (int r = 0; r < RPT; r++) S[r] = my_state[(size_t)row_of(r >> 3, r & 7) * D];
  // sums[i]: group i, even and odd rows
  auto group_sums = [&](float (&s)[2 * PAIRS][2], int r, float c, float x) { s[r >> 3][r & 1] = fmaf(c, x, s[r >> 3][r & 1]); };
  auto part_of = [&](const float (&s)[2 * PAIRS][2]) {
    float p[PAIRS];
#pragma unroll
    for (int i = 0; i < PAIRS; i++)
      p[i] = __fadd_rn(__fadd_rn(s[i][0], s[i][1]), __fadd_rn(s[i + PAIRS][0], s[i + PAIRS][1]));
    return PAIRS == 2 ? __fadd_rn(p[0], p[PAIRS - 1]) : p[0];
  };
  auto total_of = [&](const float (&p)[KG][NV]) {
    if constexpr (KG == 8) return tree8(p[0][j], p[1][j], p[2][j], p[3][j], p[4][j], p[5][j], p[6][j], p[7][j]);
    else return __fadd_rn(__fadd_rn(p[0][j], p[1][j]), __fadd_rn(p[2][j], p[3][j]));
  };

  // the next token's operands: channels lane + 32 u of q, k or g by warp 0, 1, 2; this column's v; beta
  __nv_bfloat16 nx[4], nv, nb;
  float ng[4];
  auto fetch = [&](int s) {
    const __nv_bfloat16* t = tok + (size_t)s * row;
#pragma unroll
    for (int u = 0; u < 4; u++) {
      if (warp < 2) nx[u] = t[(size_t)(warp * Hk + k_head) * D + lane + 32 * u];
      if (warp == 2) ng[u] = gp[(size_t)s * Hv * D + lane + 32 * u];
    }
    nv = t[(size_t)2 * Hk * D + (size_t)head * D + v0 + j];
    nb = bp[(size_t)s * Hv];
  };
  fetch(0);
  for (int s = 0; s < seqlen; s++) {
    const float v = __bfloat162float(nv), be = __bfloat162float(nb);
    if (warp < 2) {
      float x[4];
#pragma unroll
      for (int u = 0; u < 4; u++) x[u] = __bfloat162float(nx[u]);
      const float r = inv_norm(x);
#pragma unroll
      for (int u = 0; u < 4; u++) (warp == 0 ? sh_q : sh_k)[lane + 32 * u] = __fmul_rn(x[u], r);
    } else if (warp == 2) {
#pragma unroll
      for (int u = 0; u < 4; u++) sh_d[lane + 32 * u] = __expf(ng[u]);
    }
    if (s + 1 < seqlen) fetch(s + 1);
    __syncthreads();
    float a[2 * PAIRS][2] = {};
#pragma unroll
    for (int r = 0; r < RPT; r++) {
      const int c = row_of(r >> 3, r & 7);
      S[r] = __fmul_rn(S[r], sh_d[c]);
      group_sums(a, r, sh_k[c], S[r]);
    }
    sh_part[0][kg][j] = part_of(a);
    __syncthreads();
    const float un = __fmul_rn(__fsub_rn(v, total_of(sh_part[0])), be);
    float o[2 * PAIRS][2] = {};
#pragma unroll
    for (int r = 0; r < RPT; r++) {
      const int c = row_of(r >> 3, r & 7);
      S[r] = fmaf(sh_k[c], un, S[r]);
      group_sums(o, r, sh_q[c], S[r]);
    }
    sh_part[1][kg][j] = part_of(o);
    if (HIST) {
      // step s writes history slot s+1; the last step writes the final slot 0
      float* dst = s == seqlen - 1 ? my_state : my_state + (size_t)(s + 1) * state_size;
#pragma unroll
      for (int r = 0; r < RPT; r++) dst[(size_t)row_of(r >> 3, r & 7) * D] = S[r];
    }
    __syncthreads();
    if (kg == 0) {
      const float tot = total_of(sh_part[1]) * scale;
      const size_t oi = out_base + (size_t)s * Hv * D;
      out[oi] = __float2bfloat16_rz(tot);
      if (out_f32) out_f32[oi] = tot;
    }
  }
  if (!HIST) {
#pragma unroll
    for (int r = 0; r < RPT; r++) my_state[(size_t)row_of(r >> 3, r & 7) * D] = S[r];
  }
}

// ---------------------------------------------------------------------------------------------
// One decay per head: one CTA per (batch item, head, slice of NV value-columns); thread (kg, j) owns column j and the D/KG
// consecutive k-rows of group kg.
// ---------------------------------------------------------------------------------------------
template <int D, int NV, bool HIST>
__global__ __launch_bounds__(128) void kda_recurrent_kernel(
    const __nv_bfloat16* __restrict__ mixed_qkv, const float* __restrict__ g,
    const __nv_bfloat16* __restrict__ beta, float* __restrict__ state,
    __nv_bfloat16* __restrict__ out, float* __restrict__ out_f32, int seqlen, int Hk, int Hv,
    float scale, const int* __restrict__ slots, int history_stride) {
  constexpr int KG = 128 / NV;   // k-groups per CTA
  constexpr int RPT = D / KG;    // state rows per thread
  constexpr int NW = D / 32;     // warps that carry q/k channels
  const int b = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * NV;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int j = tid % NV, kg = tid / NV;
  const int group = Hv / Hk, k_head = head / group;
  const size_t row = (size_t)2 * Hk * D + (size_t)Hv * D;
  const size_t head_state = (size_t)D * D;
  const size_t state_size = (size_t)Hv * head_state;
  const int slot = slots ? slots[b] : b;
  float* slot_state = state + (size_t)slot * history_stride * state_size;
  float* my_state = slot_state + head * head_state + (size_t)(kg * RPT) * D + v0 + j;

  const __nv_bfloat16* tok = mixed_qkv + (size_t)b * seqlen * row;
  const float* gp = g + (size_t)b * seqlen * Hv + head;
  const __nv_bfloat16* bp = beta + (size_t)b * seqlen * Hv + head;
  const size_t out_base = ((size_t)b * seqlen * Hv + head) * D + v0 + j;

  __shared__ float sh_q[D], sh_k[D];
  __shared__ float sh_red[2][4];
  __shared__ float sh_part[2][KG][NV];

  float S[RPT];
#pragma unroll
  for (int i = 0; i < RPT; i++) S[i] = my_state[(size_t)i * D];

  // software prefetch of the next token's operands
  float nq = 0.f, nk = 0.f, ng, nv, nb;
  if (tid < D) {
    nq = __bfloat162float(tok[(size_t)k_head * D + tid]);
    nk = __bfloat162float(tok[(size_t)(Hk + k_head) * D + tid]);
  }
  ng = gp[0];
  nv = __bfloat162float(tok[(size_t)2 * Hk * D + (size_t)head * D + v0 + j]);
  nb = __bfloat162float(bp[0]);

  for (int s = 0; s < seqlen; s++) {
    float q = nq, k = nk, gv = ng, v = nv, beta_h = nb;
    if (s + 1 < seqlen) {
      const __nv_bfloat16* nt = tok + (size_t)(s + 1) * row;
      if (tid < D) {
        nq = __bfloat162float(nt[(size_t)k_head * D + tid]);
        nk = __bfloat162float(nt[(size_t)(Hk + k_head) * D + tid]);
      }
      ng = gp[(size_t)(s + 1) * Hv];
      nv = __bfloat162float(nt[(size_t)2 * Hk * D + (size_t)head * D + v0 + j]);
      nb = __bfloat162float(bp[(size_t)(s + 1) * Hv]);
    }
    // ---- L2 normalisation of q and k over the D channels ----
    float sq = warp_sum(q * q), sk = warp_sum(k * k);
    if (lane == 0 && warp < NW) {
      sh_red[0][warp] = sq;
      sh_red[1][warp] = sk;
    }
    __syncthreads();
    if (tid < D) {
      float tq = 0.f, tk = 0.f;
#pragma unroll
      for (int w = 0; w < NW; w++) {
        tq += sh_red[0][w];
        tk += sh_red[1][w];
      }
      sh_q[tid] = q * rsqrtf(tq + 1e-6f);
      sh_k[tid] = k * rsqrtf(tk + 1e-6f);
    }
    __syncthreads();
    // ---- kv_j = sum_c k_c S[c][j] ----
    const float g_h = __expf(gv);
    float sum = 0.f;
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      const int c = kg * RPT + i;
      sum = sum + sh_k[c] * S[i];
    }
    sh_part[0][kg][j] = sum;
    __syncthreads();
    float kv = 0.f;
#pragma unroll
    for (int p = 0; p < KG; p++) kv = __fadd_rn(kv, sh_part[0][p][j]);
    const float vp = v - kv * g_h;
    // ---- S <- S*decay + k v' beta ;  o_j = sum_c q_c S[c][j] ----
    float o = 0.f;
#pragma unroll
    for (int i = 0; i < RPT; i++) {
      const int c = kg * RPT + i;
      float st = S[i] * g_h + sh_k[c] * vp * beta_h;
      S[i] = st;
      o = o + sh_q[c] * st;
    }
    sh_part[1][kg][j] = o;
    if (HIST) {
      // step s writes history slot s+1; the last step writes the final slot 0
      float* dst = (s == seqlen - 1) ? my_state : my_state + (size_t)(s + 1) * state_size;
#pragma unroll
      for (int i = 0; i < RPT; i++) dst[(size_t)i * D] = S[i];
    }
    __syncthreads();
    if (kg == 0) {
      float tot = 0.f;
#pragma unroll
      for (int p = 0; p < KG; p++) tot = __fadd_rn(tot, sh_part[1][p][j]);
      tot *= scale;
      const size_t oi = out_base + (size_t)s * Hv * D;
      out[oi] = __float2bfloat16_rz(tot);
      if (out_f32) out_f32[oi] = tot;
    }
  }
  if (!HIST) {
#pragma unroll
    for (int i = 0; i < RPT; i++) my_state[(size_t)i * D] = S[i];
  }
}

// window and taps of one channel arrive as one 8-byte load each
__device__ __forceinline__ float conv4_silu_bf16(uint2 st, uint2 w, float bias, float cur) {
  // fp32 fma chain over the window [st1, st2, st3, x], taps ascending; SiLU as a / (1 + exp(-a)); rounded to bf16
  float acc = bias;
  acc = fmaf(bf16lo(w.x), bf16hi(st.x), acc);
  acc = fmaf(bf16hi(w.x), bf16lo(st.y), acc);
  acc = fmaf(bf16lo(w.y), bf16hi(st.y), acc);
  acc = fmaf(bf16hi(w.y), cur, acc);
  acc = acc * (1.0f / (1.0f + __expf(-acc)));
  return __bfloat162float(__float2bfloat16_rn(acc));
}
// new window [st1, st2, st3, x]
__device__ __forceinline__ uint2 conv4_rolled(uint2 st, __nv_bfloat16 cur) {
  uint2 r;
  r.x = (st.x >> 16) | (st.y << 16);
  r.y = (st.y >> 16) | ((uint32_t)__bfloat16_as_ushort(cur) << 16);
  return r;
}

// ---------------------------------------------------------------------------------------------
// Decode: the short convolution and the recurrence of ONE token per sequence in one launch, and (LAYER) everything else the
// KDA layer does with it - cast of the projected row, gate preparation in front, gated RMS norm behind.  The reference runs
// two launches here for the step and five for the layer (src/engine/runner.cpp:433-489); every value is formed by the same
// operations as in the separate kernels of this library, so results are bit-identical to calling them in turn.
//
// A CTA owns a whole head (64 KB of state): 8 warps hold the state (warp = row group, lane = 4 columns), three more prepare
// the token (q with its norm; k with its norm and the decay; v), and in the layer a twelfth warp asks for the norm's inputs at
// the start and finishes the output.  With the head in one CTA nothing crosses CTAs: a form of 4 or 8 value slices per head that handed the q / k window and the head's outputs
// over through two ticket counters, an atomic and an L2 round trip each (5.4 us per layer of 32 heads).
//
//   few heads: one head per CTA, or four CTAs a head where that leaves one on an SM (below), state straight between global memory and
//     registers (latency: one memory round trip, three barriers);
//   many heads (more than 2 per SM): persistent, one CTA per SM, heads stream through shared memory as 64 KB bulk copies: two
//     stages inwards, each asked for again as soon as its head sits in registers, and one outwards (stores straight from
//     registers held the SM to 26 B per cycle); the token of the next head is prepared meanwhile.  Layer, a head per CTA / streamed,
//     us: 144 heads 6.2 / 6.7, 200 9.8 / 9.4, 296 11.1 / 10.9, 320 13.8 / 12.6, 1,536 50.3 / 39.1; recurrence alone 200 heads 8.7 /
//     9.2, 296 9.9 / 10.0, 320 12.0 / 11.5.
// ---------------------------------------------------------------------------------------------
struct DecodeArgs {
  const void* x;                        // LAYER: fp32 projection row [dim], else bf16 [dim]
  __nv_bfloat16* conv_state;
  const __nv_bfloat16 *conv_w, *conv_bias;
  const float* g;                       // LAYER: raw gate projection f, else log decay
  const void* beta;                     // LAYER: fp32 logit, else bf16 beta
  const float *dt_bias, *a_log;
  float lower_bound;
  float* state;
  __nv_bfloat16* out;
  float* out_f32;
  __nv_bfloat16* conv_out;
  const void *norm_w, *gate_out;
  void* y;
  int w_bf16, g_bf16, y_f16, gate_act;
  float eps, cbias, scale;
  int H, n_heads;                       // heads of a sequence; batch * H
  int Hk;                               // key heads of a sequence (DEC_REC; else H)
  const int* slots;
  int* status;
};

struct alignas(16) DecodeToken {                    // one head's token, prepared
  float q[128], k[128], d[128], v[128];
  float beta;
};

enum { DEC_STEP, DEC_LAYER, DEC_REC };   // convolution + recurrence; the whole layer; recurrence of one token alone

constexpr int KD_STATE_WARPS = 8, KD_WARPS = 11, KD_THREADS = KD_WARPS * 32;

// role 0: q, 1: k and decay, 2: v; one warp each.  DEC_STEP leaves the rolled windows in `rolled` (decode_roll stores them)
template <int MODE>
__device__ __forceinline__ void decode_prepare(const DecodeArgs& a, DecodeToken& t, int bh, int role, int lane, uint2 (&rolled)[4]) {
  constexpr bool LAYER = MODE == DEC_LAYER;
  const int b = bh / a.H, head = bh - b * a.H, dim = (2 * a.Hk + a.H) * 128;
  const int slot = a.slots ? a.slots[b] : b;
  const int kh = MODE == DEC_REC ? head / (a.H / a.Hk) : head;
  const int c0 = (role * a.Hk + (role == 2 ? head : kh)) * 128 + lane;
  __nv_bfloat16* cs = a.conv_state + ((size_t)slot * dim + c0) * 4;
  __nv_bfloat16 x[4];
  uint2 st[4], w[4];
  float bias[4], gv[4];
  // (asked for up front; the layer's beta, a_log and dt_bias up front as well measured 0.1 us slower)
  const float beta = !LAYER && role == 2 ? __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(a.beta)[bh]) : 0.f;
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const size_t xi = (size_t)b * dim + c0 + 32 * u;
    if (LAYER) x[u] = __float2bfloat16(reinterpret_cast<const float*>(a.x)[xi]);
    else x[u] = reinterpret_cast<const __nv_bfloat16*>(a.x)[xi];
    if (MODE != DEC_REC) {
      st[u] = *reinterpret_cast<const uint2*>(cs + 128 * u);
      w[u] = *reinterpret_cast<const uint2*>(a.conv_w + (size_t)(c0 + 32 * u) * 4);
      bias[u] = a.conv_bias ? __bfloat162float(a.conv_bias[c0 + 32 * u]) : 0.f;
    }
    if (role == 1) gv[u] = a.g[(size_t)bh * 128 + lane + 32 * u];
  }
  float z[4];
#pragma unroll
  for (int u = 0; u < 4; u++) {
    if (MODE == DEC_REC) {
      z[u] = __bfloat162float(x[u]);
      continue;
    }
    z[u] = conv4_silu_bf16(st[u], w[u], bias[u], __bfloat162float(x[u]));
    rolled[u] = conv4_rolled(st[u], x[u]);
    if (!LAYER && a.conv_out) a.conv_out[(size_t)b * dim + c0 + 32 * u] = __float2bfloat16_rn(z[u]);
  }
  if (role == 2) {
#pragma unroll
    for (int u = 0; u < 4; u++) t.v[lane + 32 * u] = z[u];
    if (lane == 0)
      t.beta = LAYER ? __bfloat162float(__float2bfloat16(1.0f / (1.0f + __expf(-reinterpret_cast<const float*>(a.beta)[bh]))))
                     : beta;
    return;
  }
  const float r = inv_norm(z);
  float decay = 0.f;
  if (LAYER && role == 1) decay = __expf(a.a_log[head]);
#pragma unroll
  for (int u = 0; u < 4; u++) {
    const int c = lane + 32 * u;
    const float n = __fmul_rn(z[u], r);
    if (role == 0) {
      t.q[c] = n;
    } else {
      const float gl = LAYER ? gate_value(gv[u], a.dt_bias[head * 128 + c], decay, a.lower_bound) : gv[u];
      t.k[c] = n;
      t.d[c] = __expf(gl);
    }
  }
}

__device__ __forceinline__ void decode_roll(const DecodeArgs& a, int bh, int role, int lane, const uint2 (&rolled)[4]) {
  const int b = bh / a.H, head = bh - b * a.H;
  const int slot = a.slots ? a.slots[b] : b;
  __nv_bfloat16* cs = a.conv_state + ((size_t)slot * 3 * a.H * 128 + (role * a.H + head) * 128 + lane) * 4;
#pragma unroll
  for (int u = 0; u < 4; u++) *reinterpret_cast<uint2*>(cs + 128 * u) = rolled[u];
}

// state rows of warp w: groups w (i < 8) and w + 8; columns 4 lane .. 4 lane + 3
__device__ __forceinline__ int state_row(int w, int i) { return 4 * (w + 8 * (i >> 3) + 16 * ((i >> 2) & 1)) + (i & 3); }
struct GroupSums {                      // even and odd rows of the two groups
  float4 s[4];
  __device__ __forceinline__ void clear() {
#pragma unroll
    for (int u = 0; u < 4; u++) s[u] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __device__ __forceinline__ void add(int i, float c, float4 v) {
    float4& a = s[2 * (i >> 3) + (i & 1)];
    a.x = fmaf(c, v.x, a.x); a.y = fmaf(c, v.y, a.y); a.z = fmaf(c, v.z, a.z); a.w = fmaf(c, v.w, a.w);
  }
  __device__ __forceinline__ float4 total() const {
    return make_float4(__fadd_rn(__fadd_rn(s[0].x, s[1].x), __fadd_rn(s[2].x, s[3].x)), __fadd_rn(__fadd_rn(s[0].y, s[1].y), __fadd_rn(s[2].y, s[3].y)),
                       __fadd_rn(__fadd_rn(s[0].z, s[1].z), __fadd_rn(s[2].z, s[3].z)), __fadd_rn(__fadd_rn(s[0].w, s[1].w), __fadd_rn(s[2].w, s[3].w)));
  }
};

__device__ __forceinline__ void state_kv(float4 (&S)[16], const DecodeToken& t, int rg, int lane, float (*part)[128]) {
  GroupSums a;
  a.clear();
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const int c = state_row(rg, i);
    const float d = t.d[c];
    S[i] = make_float4(__fmul_rn(S[i].x, d), __fmul_rn(S[i].y, d), __fmul_rn(S[i].z, d), __fmul_rn(S[i].w, d));
    a.add(i, t.k[c], S[i]);
  }
  *reinterpret_cast<float4*>(&part[rg][4 * lane]) = a.total();
}
__device__ __forceinline__ float4 part_tree(const float (*part)[128], int lane) {
  float4 p[8];
#pragma unroll
  for (int i = 0; i < 8; i++) p[i] = *reinterpret_cast<const float4*>(&part[i][4 * lane]);
  return make_float4(tree8(p[0].x, p[1].x, p[2].x, p[3].x, p[4].x, p[5].x, p[6].x, p[7].x),
                     tree8(p[0].y, p[1].y, p[2].y, p[3].y, p[4].y, p[5].y, p[6].y, p[7].y),
                     tree8(p[0].z, p[1].z, p[2].z, p[3].z, p[4].z, p[5].z, p[6].z, p[7].z),
                     tree8(p[0].w, p[1].w, p[2].w, p[3].w, p[4].w, p[5].w, p[6].w, p[7].w));
}
__device__ __forceinline__ void state_update(float4 (&S)[16], const DecodeToken& t, int rg, int lane, const float (*part)[128],
                                             float (*opart)[128]) {
  const float4 kv = part_tree(part, lane);
  const float4 v = *reinterpret_cast<const float4*>(&t.v[4 * lane]);
  const float be = t.beta;
  const float4 un = make_float4(__fmul_rn(__fsub_rn(v.x, kv.x), be), __fmul_rn(__fsub_rn(v.y, kv.y), be),
                                __fmul_rn(__fsub_rn(v.z, kv.z), be), __fmul_rn(__fsub_rn(v.w, kv.w), be));
  GroupSums a;
  a.clear();
#pragma unroll
  for (int i = 0; i < 16; i++) {
    const int c = state_row(rg, i);
    const float k = t.k[c];
    S[i].x = fmaf(k, un.x, S[i].x);
    S[i].y = fmaf(k, un.y, S[i].y);
    S[i].z = fmaf(k, un.z, S[i].z);
    S[i].w = fmaf(k, un.w, S[i].w);
    a.add(i, t.q[c], S[i]);
  }
  *reinterpret_cast<float4*>(&opart[rg][4 * lane]) = a.total();
}

// one warp: the head's 128 outputs (lane = 4 columns), and LAYER: their gated RMS norm, as the one-warp-per-row norm kernel.
// load_finish is its loads, long before the outputs are there.
struct FinishIn {
  float4 gate, w;
};
template <int MODE>
__device__ __forceinline__ FinishIn load_finish(const DecodeArgs& a, int bh, int lane) {
  FinishIn f;
  if (MODE == DEC_LAYER) {
    const size_t o = (size_t)bh * 128 + 4 * lane;
    f.gate = a.g_bf16 ? load4(reinterpret_cast<const __nv_bfloat16*>(a.gate_out) + o) : load4(reinterpret_cast<const float*>(a.gate_out) + o);
    f.w = a.w_bf16 ? load4(reinterpret_cast<const __nv_bfloat16*>(a.norm_w) + 4 * lane) : load4(reinterpret_cast<const float*>(a.norm_w) + 4 * lane);
  }
  return f;
}
template <int MODE>
__device__ __forceinline__ void decode_finish(const DecodeArgs& a, const FinishIn& f, float4 tot, int bh, int lane) {
  constexpr bool LAYER = MODE == DEC_LAYER;
  const size_t o = (size_t)bh * 128 + 4 * lane;
  tot.x *= a.scale; tot.y *= a.scale; tot.z *= a.scale; tot.w *= a.scale;
  __nv_bfloat16 h[4] = {__float2bfloat16_rz(tot.x), __float2bfloat16_rz(tot.y), __float2bfloat16_rz(tot.z), __float2bfloat16_rz(tot.w)};
  if (LAYER) {
    uint2 r;
    r.x = __bfloat16_as_ushort(h[0]) | ((uint32_t)__bfloat16_as_ushort(h[1]) << 16);
    r.y = __bfloat16_as_ushort(h[2]) | ((uint32_t)__bfloat16_as_ushort(h[3]) << 16);
    *reinterpret_cast<uint2*>(a.out + o) = r;
  } else {
#pragma unroll
    for (int u = 0; u < 4; u++) a.out[o + u] = h[u];
  }
  if (a.out_f32) {
    a.out_f32[o] = tot.x; a.out_f32[o + 1] = tot.y; a.out_f32[o + 2] = tot.z; a.out_f32[o + 3] = tot.w;
  }
  if (LAYER) {
    const float4 xa = make_float4(__bfloat162float(h[0]), __bfloat162float(h[1]), __bfloat162float(h[2]), __bfloat162float(h[3]));
    const float s = warp_sum(sum_squares(0.f, xa));
    const float4 r = finish4(xa, f.w, f.gate, rsqrtf(s / 128.0f + a.eps), a.cbias, false, a.gate_act);
    if (a.y_f16) store4(reinterpret_cast<__half*>(a.y) + o, r);
    else store4(reinterpret_cast<float*>(a.y) + o, r);
  }
}

__device__ __forceinline__ float* head_state(const DecodeArgs& a, int bh) {
  const int b = bh / a.H, head = bh - b * a.H;
  const int slot = a.slots ? a.slots[b] : b;
  return a.state + ((size_t)slot * a.H + head) * 128 * 128;
}

// VEC: the state is 16-byte aligned.
// SLICES = 4, up to half a head per SM: a CTA owns 32 of the head's 128 columns (two state warps, a quarter warp per row group, the same sums in the
// same order).  One SM moves a head's 64 KB in and out in 0.6 us each, and a few heads leave the other SMs idle: one token's
// recurrence alone, whole / split: 32 heads 3.7 / 2.7 us, 74 4.2 / 3.5, 112 5.1 / 5.2; the step 32 heads 3.9 / 3.2, 64 4.4 / 4.1, 80
// 4.8 / 4.9.  In DEC_STEP and DEC_LAYER the
// four are a cluster: the windows are read by every slice and rolled by the first behind a cluster barrier that all have arrived at
// long before (32 heads 3.0 us per step; counting the slices through a word of global memory per head 3.13, at 8 heads 2.53 and
// 2.85, and calls on several streams needed counters of their own).  The layer's norm needs all columns of a head: the slices' outputs
// go to the first one's memory, 16 bytes a lane, which waits for all of them: up to a
// slice per SM, us a layer in a graph, whole / split: 8 heads 3.59 / 3.08, 32 3.59 / 3.25, 48 3.63 / 3.70, 74 3.73 / 6.2; 45-layer decode at
// 262,144 470 -> 459.
template <int MODE, bool VEC, int SLICES>
__global__ __launch_bounds__(KD_THREADS + 32) void kda_decode_kernel(const DecodeArgs a) {
  constexpr int SW = KD_STATE_WARPS / SLICES;                // state warps
  constexpr int FW = MODE == DEC_LAYER ? SW + 3 : SW;        // the warp that writes the outputs
  const int bh = blockIdx.x / SLICES, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rg = SLICES == 1 ? warp : 4 * warp + (lane >> 3);                                   // row group,
  const int cl = SLICES == 1 ? lane : (int)(blockIdx.x % SLICES) * (32 / SLICES) + (lane & 7);   // four columns
  __shared__ __align__(16) DecodeToken tok;
  __shared__ __align__(16) float part[8][128], opart[8][128];
  constexpr bool GATHER = MODE == DEC_LAYER && SLICES > 1;   // the first slice finishes the head
  __shared__ __align__(16) float4 outputs[32];
  __shared__ uint64_t here;
  __shared__ int abort_flag;
  const int slice = blockIdx.x % SLICES;
  if (GATHER && threadIdx.x == 0) {
    tc::mbar_init(&here, 1);
    tc::mbar_fence_init();
    abort_flag = 0;
    if (slice == 0) tc::mbar_arrive_expect_tx(&here, sizeof(outputs));
  }
  pdl_wait();
  float4 S[16];
  uint2 rolled[4];
  FinishIn fin;
  float* sp = nullptr;
  if (MODE == DEC_LAYER && warp == FW) {
    if (slice == 0) fin = load_finish<MODE>(a, bh, lane);                    // a warp of its own: 3 x 64 heads 7.46 -> 7.17 us, 1 x 32 3.92 -> 3.84
  } else if (warp < SW) {
    sp = head_state(a, bh) + 4 * cl;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      const float* p = sp + state_row(rg, i) * 128;
      S[i] = VEC ? *reinterpret_cast<const float4*>(p) : make_float4(p[0], p[1], p[2], p[3]);
    }
  } else {
    decode_prepare<MODE>(a, tok, bh, warp - SW, lane, rolled);
    if (MODE != DEC_REC && SLICES == 1) decode_roll(a, bh, warp - SW, lane, rolled);
  }
  __syncthreads();
  if (MODE != DEC_REC && SLICES > 1) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");   // windows read
  if (warp < SW) state_kv(S, tok, rg, cl, part);
  __syncthreads();
  if (warp < SW) {
    state_update(S, tok, rg, cl, part, opart);
#pragma unroll
    for (int i = 0; i < 16; i++) {
      float* p = sp + state_row(rg, i) * 128;
      if (VEC) *reinterpret_cast<float4*>(p) = S[i];
      else { p[0] = S[i].x; p[1] = S[i].y; p[2] = S[i].z; p[3] = S[i].w; }
    }
  }
  if (MODE != DEC_REC && SLICES > 1) {
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (warp >= SW && warp < SW + 3 && slice == 0) decode_roll(a, bh, warp - SW, lane, rolled);
  }
  __syncthreads();
  if (GATHER) {
    if (warp != FW) return;
    if (lane < 32 / SLICES) {
      const float4 tot = part_tree(opart, cl);
      uint32_t to, bar;
      asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"(tc::smem_u32(&outputs[cl])));
      asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(bar) : "r"(tc::smem_u32(&here)));
      asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to), "r"(__float_as_uint(tot.x)),
                   "r"(__float_as_uint(tot.y)), "r"(__float_as_uint(tot.z)), "r"(__float_as_uint(tot.w)), "r"(bar)
                   : "memory");
    }
    if (slice > 0) return;
    const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&here, 0, &abort_flag, 1)) != 0;   // (the norm is the whole warp's)
    if (ok) decode_finish<MODE>(a, fin, outputs[lane], bh, lane);
    else if (a.status) atomicExch(a.status, HK_ERR_TIMEOUT);
    return;
  }
  if (warp == FW && (SLICES == 1 || lane < 32 / SLICES)) decode_finish<MODE>(a, fin, part_tree(opart, SLICES == 1 ? lane : cl), bh, SLICES == 1 ? lane : cl);
}

// persistent form: CTA c takes heads c, c + gridDim.x, ...
constexpr int KD_STAGES = 2;
constexpr size_t KD_STREAM_SMEM = (size_t)(KD_STAGES + 1) * 65536;
constexpr int KD_STREAM_THREADS = KD_THREADS + 32;               // one more warp, which finishes the head before
template <int MODE>
__global__ __launch_bounds__(KD_STREAM_THREADS) void kda_decode_stream_kernel(const DecodeArgs a, int* __restrict__ status) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ __align__(16) DecodeToken tok[2];
  __shared__ __align__(16) float part[8][128], opart[2][8][128];
  __shared__ uint64_t full[KD_STAGES];
  __shared__ int abort_flag;
  const int step = gridDim.x, first = blockIdx.x;
  const int n = (a.n_heads - first + step - 1) / step;          // >= 1: the grid is no larger than the head count
  if (threadIdx.x == 0) {
    for (int s = 0; s < KD_STAGES; s++) tc::mbar_init(&full[s], 1);
    tc::mbar_fence_init();
    abort_flag = 0;
  }
  pdl_wait();
  auto fetch = [&](int i) {                                     // thread 0: head i of this CTA into its stage
    tc::mbar_arrive_expect_tx(&full[i % KD_STAGES], 65536);
    tc::bulk_g2s(smem + (i % KD_STAGES) * 65536, head_state(a, first + i * step), 65536, &full[i % KD_STAGES]);
  };
  if (threadIdx.x == 0)
    for (int i = 0; i < KD_STAGES && i < n; i++) fetch(i);
  uint2 rolled[4];
  auto prepare = [&](int i) {
    decode_prepare<MODE>(a, tok[i & 1], first + i * step, warp - KD_STATE_WARPS, lane, rolled);
    if (MODE != DEC_REC) decode_roll(a, first + i * step, warp - KD_STATE_WARPS, lane, rolled);
  };
  if (warp >= KD_STATE_WARPS && warp < KD_WARPS) prepare(0);
  __syncthreads();
  FinishIn fin;
  bool ok = true;
  for (int i = 0; i < n; i++) {
    const int bh = first + i * step;
    const float4* st = reinterpret_cast<const float4*>(smem + (i % KD_STAGES) * 65536) + lane;
    if (warp < KD_STATE_WARPS) {
      ok = tc::mbar_wait(&full[i % KD_STAGES], (i / KD_STAGES) & 1, &abort_flag, 1);
      float4 S[16];
#pragma unroll
      for (int r = 0; r < 16; r++) S[r] = st[state_row(warp, r) * 32];
      state_kv(S, tok[i & 1], warp, lane, part);
      if (threadIdx.x == 0) tc::bulk_wait_read<0>();
      asm volatile("bar.sync 1, 256;" ::: "memory");
      if (threadIdx.x == 0 && i + KD_STAGES < n) fetch(i + KD_STAGES);
      state_update(S, tok[i & 1], warp, lane, part, opart[i & 1]);
      // the outward stage is free: thread 0 has waited for its last reader, and passed the barrier above, since
      float4* so = reinterpret_cast<float4*>(smem + KD_STAGES * 65536) + lane;
#pragma unroll
      for (int r = 0; r < 16; r++) so[state_row(warp, r) * 32] = S[r];
      tc::fence_async_smem();
    } else {
      if (warp == KD_WARPS) {
        if (i > 0) decode_finish<MODE>(a, fin, part_tree(opart[(i - 1) & 1], lane), bh - step, lane);
        fin = load_finish<MODE>(a, bh, lane);
      }
      if (i + 1 < n && warp < KD_WARPS) prepare(i + 1);
    }
    __syncthreads();
    if (threadIdx.x == 0 && ok && !abort_flag) {
      tc::bulk_s2g(head_state(a, bh), smem + KD_STAGES * 65536, 65536);
      tc::bulk_commit();
    }
  }
  if (warp == KD_WARPS) decode_finish<MODE>(a, fin, part_tree(opart[(n - 1) & 1], lane), first + (n - 1) * step, lane);
  if (threadIdx.x == 0) {
    tc::bulk_wait_all<0>();
    if (abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
  }
}

template <int MODE>
static int launch_decode(DecodeArgs& a, cudaStream_t s, bool beside = false) {
  const bool vec = aligned(a.state, 16);
  // (asked for once, not four times: where the host bounds a call, one layer of 32 heads 3.81 -> 3.73 us; 3.72 with a CTA a head, 3.45 where the GPU does)
  const int dev = device_index(), sms = sm_count(dev);
  if (vec && a.n_heads > 2 * sms) {
    static bool attr_set[64] = {false};
    if (!attr_set[dev]) {
      if (cudaFuncSetAttribute(kda_decode_stream_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)KD_STREAM_SMEM) != cudaSuccess)
        return HK_ERR_CUDA;
      attr_set[dev] = true;
    }
    return pdl_launch(kda_decode_stream_kernel<MODE>, dim3(sms), dim3(KD_STREAM_THREADS), KD_STREAM_SMEM, s, a, device_status_ptr(dev)) == cudaSuccess ? HK_OK : HK_ERR_CUDA;
  }
  // The layer: a slice to an SM.  Not where the caller has such calls on other streams (`beside`): a slice's CTA prepares the whole token, and
  // two of them fill an SM.  30 layers of 32 heads on each of S streams, a CTA a head / four: S = 1 111 / 101 us, 2 117 / 117, 4 153 / 173, 6 188 /
  // 266, 8 221 / 354; of 16 heads 4 119 / 119, 8 160 / 176.
  if (vec && !beside && a.n_heads <= sms / (MODE == DEC_LAYER ? 4 : 2)) {
    if (MODE == DEC_LAYER) a.status = device_status_ptr(dev);
    return pdl_launch_cluster(MODE == DEC_REC ? 1 : 4, kda_decode_kernel<MODE, true, 4>, dim3(4 * a.n_heads), dim3((MODE == DEC_LAYER ? 6 : 5) * 32), 0, s,
                              a) == cudaSuccess
               ? HK_OK
               : HK_ERR_CUDA;
  }
  auto kern = vec ? kda_decode_kernel<MODE, true, 1> : kda_decode_kernel<MODE, false, 1>;
  return pdl_launch(kern, dim3(a.n_heads), dim3(KD_THREADS + (MODE == DEC_LAYER ? 32 : 0)), 0, s, a) == cudaSuccess ? HK_OK : HK_ERR_CUDA;
}

// ---------------------------------------------------------------------------------------------
// Token by token with channelwise decay, D = 128, no history: short prompts, and decode through the launchers.
//
// What bounds it is the chain from token to token.  The kernel above takes 1.07 us per token: every token is normalised inside
// the chain and crosses four block barriers.  Here a warp owns 2 CPL columns, lane (rg, c) the 8 rows of group rg of CPL
// columns, and the sums over the 16 groups are shuffles: no barrier inside the chain.  Everything that does not depend on the
// state (norms, decay) is prepared for 8 tokens at a time in the other half of a double buffer, a warp per token: one
// block barrier per 8 tokens.  The products run as packed fp32 pairs (two rows per instruction).
// Shared memory is the other limit: a warp reads a token's three prepared vectors (1.5 KB) whatever it does with them, as
// 6 reads of 4 wavefronts.  With 8 groups over 8 lanes (and k * d as a fourth vector) it was 16 reads (64 heads: 0.84 us per token with one column per lane,
// 0.57 with four).  The output sums of four tokens are taken together and exchange HALF of their values at each step (15
// shuffles for 16 values instead of 64).
// CPL 4 takes states on a 16-byte boundary, 1 any.
// ---------------------------------------------------------------------------------------------
// Sums of N values per lane over the L lanes that share their columns: of 16, lanes 8 apart first; then 1, 2, 4.  While a lane has more than one value it keeps one half and hands the
// other to its partner; a lane ends with the sum of value sum_index (the same in all lanes that agree in the bits used; sum_owner
// picks one of them).
template <int L>
__device__ __forceinline__ constexpr int sum_mask(int st) { return L == 16 ? (st == 0 ? 8 : 1 << (st - 1)) : 1 << st; }
template <int N, int L>
__device__ __forceinline__ int sum_index(int lane) {
  int idx = 0;
#pragma unroll
  for (int st = 0, n = N; n > 1; st++) {
    n >>= 1;
    if (lane & sum_mask<L>(st)) idx += n;
  }
  return idx;
}
template <int N, int L>
__device__ __forceinline__ bool sum_owner(int lane) {
  int left = L - 1;
#pragma unroll
  for (int st = 0, n = N; n > 1; st++, n >>= 1) left &= ~sum_mask<L>(st);
  return (lane & left) == 0;
}
template <int N, int L>
__device__ __forceinline__ float lane_sums(const float* v, int lane) {
  float x[N];
#pragma unroll
  for (int i = 0; i < N; i++) x[i] = v[i];
  int n = N;
#pragma unroll
  for (int st = 0; (1 << st) < L; st++) {
    const int m = sum_mask<L>(st);
    if (n > 1) {
      n >>= 1;
#pragma unroll
      for (int i = 0; i < N / 2; i++) {
        if (i < n) {
          const bool up = lane & m;
          const float keep = up ? x[i + n] : x[i], give = up ? x[i] : x[i + n];
          x[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, give, m));
        }
      }
    } else {
      x[0] = __fadd_rn(x[0], __shfl_xor_sync(0xffffffffu, x[0], m));
    }
  }
  return x[0];
}
constexpr int RC_TB = 8, RC_WARPS = 4;   // tokens of a batch; warps that prepare it, and that walk through it
template <int COLS>
struct alignas(16) RecBatch {           // 8 prepared tokens
  float q[RC_TB][128], k[RC_TB][128], d[RC_TB][128], v[RC_TB][COLS], beta[RC_TB];
};
// Tokens warp, warp + 4 of a batch on their way: channel lane + 32 u of q, k, g, columns lane, lane + 32 of v.  Kept as loaded: a
// conversion in fetch would wait for the loads.
template <int COLS>
struct RecTokens {
  static constexpr int TPW = RC_TB / RC_WARPS, NVL = (COLS + 31) / 32;
  __nv_bfloat16 q[TPW][4], k[TPW][4], v[TPW][NVL], be[TPW];
  float g[TPW][4];
  // tok, gp, bp: first token of the sequence; gp and bp of the head, v_at: first of the CTA's columns in a row
  __device__ __forceinline__ void fetch(int s0, int seqlen, int warp, int lane, const __nv_bfloat16* tok, size_t row, size_t q_at, size_t k_at,
                                        size_t v_at, const float* gp, const __nv_bfloat16* bp, int Hv) {
#pragma unroll
    for (int p = 0; p < TPW; p++) {
      const int s = s0 + warp + p * RC_WARPS;
      if (s >= seqlen) break;
      const __nv_bfloat16* t = tok + (size_t)s * row;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        q[p][u] = t[q_at + lane + 32 * u];
        k[p][u] = t[k_at + lane + 32 * u];
        g[p][u] = gp[(size_t)s * Hv * 128 + lane + 32 * u];
      }
#pragma unroll
      for (int u = 0; u < NVL; u++)
        if (lane + 32 * u < COLS) v[p][u] = t[v_at + lane + 32 * u];
      be[p] = bp[(size_t)s * Hv];
    }
  }
  __device__ __forceinline__ void prepare(RecBatch<COLS>& r, int s0, int seqlen, int warp, int lane) const {
#pragma unroll
    for (int p = 0; p < TPW; p++) {
      const int t = warp + p * RC_WARPS;
      if (s0 + t >= seqlen) break;
      float fq[4], fk[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        fq[u] = __bfloat162float(q[p][u]);
        fk[u] = __bfloat162float(k[p][u]);
      }
      const float iq = inv_norm(fq), ik = inv_norm(fk);
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int c = lane + 32 * u;
        r.q[t][c] = __fmul_rn(fq[u], iq);
        r.k[t][c] = __fmul_rn(fk[u], ik);
        r.d[t][c] = __expf(g[p][u]);
      }
#pragma unroll
      for (int u = 0; u < NVL; u++)
        if (lane + 32 * u < COLS) r.v[t][lane + 32 * u] = __bfloat162float(v[p][u]);
      if (lane == 0) r.beta[t] = __bfloat162float(be[p]);
    }
  }
};
// The CPL columns at p, a vector each way.
template <int CPL>
__device__ __forceinline__ void ld_cols(const float* p, float (&x)[CPL]) {
  if constexpr (CPL == 4) {
    const float4 v = *reinterpret_cast<const float4*>(p);
    x[0] = v.x; x[1] = v.y; x[2] = v.z; x[3] = v.w;
  } else if constexpr (CPL == 2) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    x[0] = v.x; x[1] = v.y;
  } else {
    x[0] = p[0];
  }
}
template <int CPL>
__device__ __forceinline__ void st_cols(float* p, const float (&x)[CPL]) {
  if constexpr (CPL == 4) *reinterpret_cast<float4*>(p) = make_float4(x[0], x[1], x[2], x[3]);
  else if constexpr (CPL == 2) *reinterpret_cast<float2*>(p) = make_float2(x[0], x[1]);
  else p[0] = x[0];
}

template <int CPL>
__global__ __launch_bounds__(RC_WARPS * 32) void kda_recurrent_cols_kernel(
    const __nv_bfloat16* __restrict__ mixed_qkv, const float* __restrict__ g, const __nv_bfloat16* __restrict__ beta,
    float* __restrict__ state, __nv_bfloat16* __restrict__ out, float* __restrict__ out_f32, int seqlen, int Hk, int Hv, float scale,
    const int* __restrict__ slots) {
  constexpr int COLS = RC_WARPS * 2 * CPL;                             // columns of the CTA
  __shared__ RecBatch<COLS> rb[2];
  __shared__ __align__(16) float s_o[2][RC_TB][COLS];
  const int b = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rg = lane & 15, col = (warp * 2 + (lane >> 4)) * CPL;       // first column of this lane
  const int k_head = head / (Hv / Hk);
  const size_t row = (size_t)2 * Hk * 128 + (size_t)Hv * 128;
  pdl_wait();
  const int slot = slots ? slots[b] : b;
  const __nv_bfloat16* tok = mixed_qkv + (size_t)b * seqlen * row;
  const float* gp = g + ((size_t)b * seqlen * Hv + head) * 128;
  const __nv_bfloat16* bp = beta + (size_t)b * seqlen * Hv + head;
  float* sp = state + ((size_t)slot * Hv + head) * 128 * 128 + v0 + col;

  RecTokens<COLS> ahead;
  auto fetch = [&](int s0) {
    ahead.fetch(s0, seqlen, warp, lane, tok, row, (size_t)k_head * 128, (size_t)(Hk + k_head) * 128, (size_t)2 * Hk * 128 + (size_t)head * 128 + v0, gp, bp,
                Hv);
  };
  fetch(0);
  // rows 4 (rg + 16 j) + e of the lane's columns, packed by row pairs
  uint64_t S[CPL][4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r0 = 4 * (rg + 16 * (i >> 1)) + 2 * (i & 1);
    float x0[CPL], x1[CPL];
    ld_cols(sp + (size_t)r0 * 128, x0);
    ld_cols(sp + (size_t)(r0 + 1) * 128, x1);
#pragma unroll
    for (int c = 0; c < CPL; c++) S[c][i] = pack2(x0[c], x1[c]);
  }
  ahead.prepare(rb[0], 0, seqlen, warp, lane);
  __syncthreads();
  int buf = 0;
  for (int s0 = 0; s0 < seqlen; s0 += RC_TB, buf ^= 1) {
    const int n = min(RC_TB, seqlen - s0);
    fetch(s0 + RC_TB);
    const RecBatch<COLS>& r = rb[buf];
    // A token's operands are read while the token before it is in its shuffles: read where they are used, they were a
    // third of the chain.
    struct Operands {
      uint64_t k[4], d[4], q[4];
      float v[CPL], be;
    };
    auto operands = [&](int t, Operands& o) {
      auto pieces = [&](const float (*p)[128], uint64_t (&x)[4]) {
#pragma unroll
        for (int j = 0; j < 2; j++) {
          const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(&p[t][4 * (rg + 16 * j)]);
          x[2 * j] = w.x;
          x[2 * j + 1] = w.y;
        }
      };
      pieces(r.d, o.d);
      pieces(r.k, o.k);
      pieces(r.q, o.q);
      o.be = r.beta[t];
#pragma unroll
      for (int c = 0; c < CPL; c++) o.v[c] = r.v[t][col + c];
    };
    auto token = [&](int t, Operands& o, float* ov) {
      auto group_sum = [&](const uint64_t (&x)[4], float* y) {
#pragma unroll
        for (int c = 0; c < CPL; c++) {
          uint64_t acc = 0;
#pragma unroll
          for (int i = 0; i < 4; i++) acc = fma2(x[i], S[c][i], acc);
          float lo, hi;
          unpack2(acc, lo, hi);
          y[c] = __fadd_rn(lo, hi);
        }
      };
      float y[CPL];
#pragma unroll
      for (int c = 0; c < CPL; c++)
#pragma unroll
        for (int i = 0; i < 4; i++) S[c][i] = mul2(S[c][i], o.d[i]);
      group_sum(o.k, y);
      Operands next;
      operands(min(t + 1, RC_TB - 1), next);
      // every lane needs the sums of all its columns: plain butterfly (halving the values and spreading them again takes
      // as many instructions and two more exchanges on the chain)
#pragma unroll
      for (int st = 0; st < 4; st++)
#pragma unroll
        for (int c = 0; c < CPL; c++) y[c] = __fadd_rn(y[c], __shfl_xor_sync(0xffffffffu, y[c], st == 0 ? 8 : 1 << (st - 1)));
#pragma unroll
      for (int c = 0; c < CPL; c++) {
        const float un = __fmul_rn(__fsub_rn(o.v[c], y[c]), o.be);
        const uint64_t u2 = pack2(un, un);
#pragma unroll
        for (int i = 0; i < 4; i++) S[c][i] = fma2(o.k[i], u2, S[c][i]);
      }
      group_sum(o.q, ov);
      o = next;
    };
    Operands ops;
    operands(0, ops);
    int t = 0;
#pragma unroll 1
    for (; t + 4 <= n; t += 4) {
      float ov[4 * CPL];                                 // group sums of the outputs of four tokens
#pragma unroll
      for (int tt = 0; tt < 4; tt++) token(t + tt, ops, ov + tt * CPL);
      const float o = lane_sums<4 * CPL, 16>(ov, lane);
      const int idx = sum_index<4 * CPL, 16>(lane);          // value (token t + idx / CPL, column col + idx % CPL)
      if (sum_owner<4 * CPL, 16>(lane)) s_o[buf][t + idx / CPL][col + idx % CPL] = o;
    }
#pragma unroll 1
    for (; t < n; t++) {
      float ov[CPL];
      token(t, ops, ov);
      const float o = lane_sums<CPL, 16>(ov, lane);
      if (sum_owner<CPL, 16>(lane)) s_o[buf][t][col + sum_index<CPL, 16>(lane)] = o;
    }
    ahead.prepare(rb[buf ^ 1], s0 + RC_TB, seqlen, warp, lane);
    __syncthreads();
    for (int i = tid; i < n * COLS; i += RC_WARPS * 32) {
      const float tot = s_o[buf][i / COLS][i % COLS] * scale;
      const size_t oi = (((size_t)b * seqlen + s0 + i / COLS) * Hv + head) * 128 + v0 + i % COLS;
      out[oi] = __float2bfloat16_rz(tot);
      if (out_f32) out_f32[oi] = tot;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int r0 = 4 * (rg + 16 * (i >> 1)) + 2 * (i & 1);
    float x0[CPL], x1[CPL];
#pragma unroll
    for (int c = 0; c < CPL; c++) unpack2(S[c][i], x0[c], x1[c]);
    st_cols(sp + (size_t)r0 * 128, x0);
    st_cols(sp + (size_t)(r0 + 1) * 128, x1);
  }
}

// ---------------------------------------------------------------------------------------------
// The same for few chains, a CTA to an SM at most.  What bounds it is a warp's chain from token to token: nothing else is there to fill an SM's
// slots.  So the CTA has a second half that takes everything off the chain that does not depend on the state (a batch of tokens prepared
// ahead, the outputs of the batch before written), handed over with named barriers; and a warp walks two halves of its columns, the
// second half a token behind by half: while the row sums of one are in their shuffles, the other has its products (both in one
// instruction stream, with two sets of operands that take turns).  L lanes share a column: with 8 a lane has two row groups (rg and
// rg + 8: the first of the four sums is a local one).  Sums in plain fp32: with one warp on a scheduler the packed form measured 107 cycles
// for 64 products of a sum, this one 82; updates packed (96, but half the issue slots), and the decay where a warp has 16 columns or 8 (two
// columns a lane: 2-4 % slower).  37 tokens x 64 chains 18.8 -> 15.8 us, x 32 16.5 -> 11.1, x 16 13.9 -> 9.5; without the halves 16.7 / 11.8 / 9.9.
// ---------------------------------------------------------------------------------------------
enum { RC_FULL = 1, RC_DONE = 3 };          // named barriers of the two batches: prepared; walked through
__device__ __forceinline__ void rc_sync(int bar) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(2 * RC_WARPS * 32) : "memory"); }
__device__ __forceinline__ void rc_arrive(int bar) { asm volatile("bar.arrive %0, %1;" ::"r"(bar), "n"(2 * RC_WARPS * 32) : "memory"); }

template <int CPL, int L>
__global__ __launch_bounds__(2 * RC_WARPS * 32, 1) void kda_recurrent_few_kernel(
    const __nv_bfloat16* __restrict__ mixed_qkv, const float* __restrict__ g, const __nv_bfloat16* __restrict__ beta,
    float* __restrict__ state, __nv_bfloat16* __restrict__ out, float* __restrict__ out_f32, int seqlen, int Hk, int Hv, float scale,
    const int* __restrict__ slots) {
  constexpr int COLS = RC_WARPS * (32 / L) * CPL, ROWS = 128 / L;       // columns of the CTA, rows of a lane
  __shared__ RecBatch<COLS> rb[2];
  __shared__ __align__(16) float s_o[2][RC_TB][COLS];
  const int b = blockIdx.x, head = blockIdx.y, v0 = blockIdx.z * COLS;
  const int tid = threadIdx.x, lane = tid & 31, warp = (tid >> 5) & (RC_WARPS - 1);
  pdl_wait();
  if (tid >= RC_WARPS * 32) {
    const int k_head = head / (Hv / Hk), n_batches = (seqlen + RC_TB - 1) / RC_TB;
    const size_t row = (size_t)2 * Hk * 128 + (size_t)Hv * 128;
    RecTokens<COLS> ahead;
    auto fetch = [&](int s0) {
      ahead.fetch(s0, seqlen, warp, lane, mixed_qkv + (size_t)b * seqlen * row, row, (size_t)k_head * 128, (size_t)(Hk + k_head) * 128,
                  (size_t)2 * Hk * 128 + (size_t)head * 128 + v0, g + ((size_t)b * seqlen * Hv + head) * 128, beta + (size_t)b * seqlen * Hv + head, Hv);
    };
    fetch(0);
    for (int j = 0; j < n_batches + 2; j++) {             // batch j prepared, batch j - 2 written out
      const int buf = j & 1;
      if (j >= 2) {
        rc_sync(RC_DONE + buf);
        const int s0 = (j - 2) * RC_TB, n = min(RC_TB, seqlen - s0);
        for (int i = tid - RC_WARPS * 32; i < n * COLS; i += RC_WARPS * 32) {
          const float tot = s_o[buf][i / COLS][i % COLS] * scale;
          const size_t oi = (((size_t)b * seqlen + s0 + i / COLS) * Hv + head) * 128 + v0 + i % COLS;
          out[oi] = __float2bfloat16_rz(tot);
          if (out_f32) out_f32[oi] = tot;
        }
      }
      if (j < n_batches) {
        ahead.prepare(rb[buf], j * RC_TB, seqlen, warp, lane);
        rc_arrive(RC_FULL + buf);
        if (j + 1 < n_batches) fetch((j + 1) * RC_TB);
      }
    }
    return;
  }
  const int rg = lane & (L - 1), col = (warp * (32 / L) + lane / L) * CPL;   // row groups from rg on; first column of this lane
  float* sp = state + ((size_t)(slots ? slots[b] : b) * Hv + head) * 128 * 128 + v0 + col;
  // row i of the lane: of group rg (i < 8) or rg + 8, of its first or second chunk of four
  auto row_of = [&](int i) { return 4 * (rg + 8 * (i >> 3) + 16 * ((i >> 2) & 1)) + (i & 3); };
  float S[CPL][ROWS];
#pragma unroll
  for (int i = 0; i < ROWS; i++) {
    float x[CPL];
    ld_cols(sp + (size_t)row_of(i) * 128, x);
#pragma unroll
    for (int c = 0; c < CPL; c++) S[c][i] = x[c];
  }
  struct Operands {
    float k[ROWS], d[ROWS], q[ROWS], v[CPL], be;
  };
  auto operands = [&](int s, Operands& o) {
    const RecBatch<COLS>& r = rb[(s / RC_TB) & 1];
    const int t = s % RC_TB;
    auto pieces = [&](const float (*p)[128], float (&x)[ROWS]) {
#pragma unroll
      for (int j = 0; j < ROWS / 4; j++) {
        const float4 w = *reinterpret_cast<const float4*>(&p[t][row_of(4 * j)]);
        x[4 * j] = w.x; x[4 * j + 1] = w.y; x[4 * j + 2] = w.z; x[4 * j + 3] = w.w;
      }
    };
    pieces(r.d, o.d);
    pieces(r.k, o.k);
    pieces(r.q, o.q);
    o.be = r.beta[t];
#pragma unroll
    for (int c = 0; c < CPL; c++) o.v[c] = r.v[t][col + c];
  };
  // sums over the lane's rows of half f of the columns: even and odd rows of a group by themselves
  constexpr int HC = CPL / 2;
  auto group_sum = [&](int f, const float (&x)[ROWS], float (&y)[HC]) {
    constexpr int P = ROWS / 4;
    float acc[HC][P];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int c = 0; c < HC; c++)
#pragma unroll
        for (int h = 0; h < P; h++) {
          const int r = 8 * (h >> 1) + 2 * i + (h & 1);
          acc[c][h] = __fmaf_rn(x[r], S[f * HC + c][r], i ? acc[c][h] : 0.f);
        }
#pragma unroll
    for (int c = 0; c < HC; c++) {
      y[c] = __fadd_rn(acc[c][0], acc[c][1]);
      if (P == 4) y[c] = __fadd_rn(y[c], __fadd_rn(acc[c][P - 2], acc[c][P - 1]));
    }
  };
  auto decay = [&](int f, const Operands& o, float (&y)[HC]) {           // S <- d S; the lane's part of k S
#pragma unroll
    for (int c = 0; c < HC; c++)
#pragma unroll
      for (int i = 0; i < ROWS; i += 2) {
        float &a = S[f * HC + c][i], &b = S[f * HC + c][i + 1];
        if (CPL == 4) {
          unpack2(mul2(pack2(a, b), pack2(o.d[i], o.d[i + 1])), a, b);
        } else {
          a = __fmul_rn(a, o.d[i]);
          b = __fmul_rn(b, o.d[i + 1]);
        }
      }
    group_sum(f, o.k, y);
  };
  auto across = [&](float (&y)[HC]) {                                     // summed over the lanes
#pragma unroll
    for (int st = 0; (1 << st) < L; st++)
#pragma unroll
      for (int c = 0; c < HC; c++) y[c] = __fadd_rn(y[c], __shfl_xor_sync(0xffffffffu, y[c], sum_mask<L>(st)));
  };
  auto update = [&](int f, const Operands& o, const float (&y)[HC], float (&ov)[HC]) {   // S <- S + k u; the lane's part of q S
#pragma unroll
    for (int c = 0; c < HC; c++) {
      const float un = __fmul_rn(__fsub_rn(o.v[f * HC + c], y[c]), o.be);
#pragma unroll
      for (int i = 0; i < ROWS; i += 2) {
        float &a = S[f * HC + c][i], &b = S[f * HC + c][i + 1];
        unpack2(fma2(pack2(o.k[i], o.k[i + 1]), pack2(un, un), pack2(a, b)), a, b);
      }
    }
    group_sum(f, o.q, ov);
  };
  float ya[HC], yb[HC], oa[HC];                            // half 0 runs half a token ahead of half 1
  auto emit = [&](int s, const float (&ob)[HC]) {          // output sums of token s
    float ov[CPL];
#pragma unroll
    for (int c = 0; c < HC; c++) {
      ov[c] = oa[c];
      ov[HC + c] = ob[c];
    }
    const float o = lane_sums<CPL, L>(ov, lane);
    if (sum_owner<CPL, L>(lane)) s_o[(s / RC_TB) & 1][s % RC_TB][col + sum_index<CPL, L>(lane)] = o;
    if (s % RC_TB == RC_TB - 1 || s == seqlen - 1) rc_arrive(RC_DONE + ((s / RC_TB) & 1));
  };
  auto step = [&](int s, Operands& now, Operands& before) {   // on return `before` holds token s + 1
    decay(0, now, ya);
    across(ya);
    float ob[HC];
    update(1, before, yb, ob);
    if ((s + 1) % RC_TB == 0 && s + 1 < seqlen) rc_sync(RC_FULL + (((s + 1) / RC_TB) & 1));
    operands(min(s + 1, seqlen - 1), before);
    decay(1, now, yb);
    emit(s - 1, ob);
    across(yb);
    update(0, now, ya, oa);
  };
  Operands o0, o1;
  rc_sync(RC_FULL);
  operands(0, o0);
  decay(0, o0, ya);
  across(ya);
  operands(min(1, seqlen - 1), o1);
  decay(1, o0, yb);
  across(yb);
  update(0, o0, ya, oa);
  int s = 1;
#pragma unroll 1
  for (; s + 2 <= seqlen; s += 2) {
    step(s, o1, o0);
    step(s + 1, o0, o1);
  }
  float ob[HC];
  if (s < seqlen) {
    step(s, o1, o0);
    update(1, o1, yb, ob);
  } else {
    update(1, o0, yb, ob);
  }
  emit(seqlen - 1, ob);
#pragma unroll
  for (int i = 0; i < ROWS; i++) {
    float x[CPL];
#pragma unroll
    for (int c = 0; c < CPL; c++) x[c] = S[c][i];
    st_cols(sp + (size_t)row_of(i) * 128, x);
  }
}

// narrower column slices when the (batch x head) count alone cannot cover the SMs
static bool narrow_slices(int bsz, int Hv) { return (long)bsz * Hv * 4 < sm_count(); }

static int launch_rows(const __nv_bfloat16* qkv, const float* g, const __nv_bfloat16* beta, float* state, __nv_bfloat16* out,
                       float* out_f32, int bsz, int seqlen, int Hk, int Hv, int history_stride, const int* slots, bool hist,
                       cudaStream_t s) {
  const bool narrow = narrow_slices(bsz, Hv);
  auto kern = narrow ? (hist ? kda_recurrent_rows_kernel<16, true> : kda_recurrent_rows_kernel<16, false>)
                     : (hist ? kda_recurrent_rows_kernel<32, true> : kda_recurrent_rows_kernel<32, false>);
  kern<<<dim3(bsz, Hv, narrow ? 8 : 4), 128, 0, s>>>(qkv, g, beta, state, out, out_f32, seqlen, Hk, Hv, 1.0f / sqrtf(128.0f), slots,
                                                     history_stride);
  return cudaPeekAtLastError() == cudaSuccess ? HK_OK : HK_ERR_CUDA;
}

template <int D, int NV>
static int launch_recurrent(const __nv_bfloat16* qkv, const float* g, const __nv_bfloat16* beta,
                            float* state, __nv_bfloat16* out, float* out_f32, int bsz, int seqlen,
                            int Hk, int Hv, int history_stride, const int* slots, bool hist, cudaStream_t s) {
  auto kern = hist ? kda_recurrent_kernel<D, NV, true> : kda_recurrent_kernel<D, NV, false>;
  kern<<<dim3(bsz, Hv, D / NV), 128, 0, s>>>(qkv, g, beta, state, out, out_f32, seqlen, Hk, Hv, 1.0f / sqrtf((float)D), slots,
                                             history_stride);
  return cudaPeekAtLastError() == cudaSuccess ? HK_OK : HK_ERR_CUDA;
}

}  // namespace hk

HK_API int hk_kda_recurrent(const void* mixed_qkv, const float* g, const void* beta, float* state,
                            void* out, float* out_f32, int bsz, int seqlen, int num_k_heads,
                            int num_v_heads, int k_head_dim, int v_head_dim, int history_stride,
                            const int* slots, int channelwise, int history, void* stream) {
  using namespace hk;
  HK_REQUIRE(mixed_qkv && g && beta && state && out);
  HK_REQUIRE(bsz > 0 && seqlen > 0 && num_k_heads > 0 && num_v_heads > 0 && history_stride >= 1);
  HK_REQUIRE(num_v_heads % num_k_heads == 0);
  if (history) HK_REQUIRE(history_stride >= seqlen);  // slots 1..seqlen-1 are written
  if (k_head_dim != v_head_dim) return HK_ERR_UNSUPPORTED;
  if (channelwise && k_head_dim != 128) return HK_ERR_INVALID;  // as the reference launcher
  auto q = (const __nv_bfloat16*)mixed_qkv;
  auto bt = (const __nv_bfloat16*)beta;
  auto o = (__nv_bfloat16*)out;
  cudaStream_t s = as_stream(stream);
  if (k_head_dim == 128 && channelwise && !history && history_stride == 1) {
    const int64_t chains = (int64_t)bsz * num_v_heads;
    if (seqlen == 1 && chains <= 1 << 28) {   // one token: the decode step's kernels without the convolution, the same bits
      DecodeArgs a{};
      a.x = q;
      a.g = g;
      a.beta = bt;
      a.state = state;
      a.out = o;
      a.out_f32 = out_f32;
      a.scale = 1.0f / sqrtf(128.0f);
      a.H = num_v_heads;
      a.Hk = num_k_heads;
      a.n_heads = (int)chains;
      a.slots = slots;
      return launch_decode<DEC_REC>(a, s);
    }
    // A few tokens of many chains are mostly the state in and out, which the rows kernel moves in longer runs; more tokens are the
    // chain from token to token, which is the columns kernel's.  Rows against columns, us: 8 chains 2 tokens 3.1 / 3.1; 16 chains 3
    // tokens 3.4 / 4.2, 4 tokens 4.2 / 4.1; 64 chains 5.3 / 5.7, 6.1 / 5.9; 256 chains 6 tokens 18.2 / 18.2, 8 tokens 22.0 / 19.8;
    // 512 chains 12 tokens 46.8 / 46.9, 16 tokens 58.8 / 55.0; 1,536 chains 16 tokens 152 / 158, 24 tokens 220 / 210.
    const int rows_up_to = chains >= 1024 ? 16 : (chains >= 384 ? 12 : (chains >= 128 ? 6 : (chains >= 16 ? 3 : 1)));
    if (seqlen > rows_up_to) {
      // As many CTAs to a chain as fit with one on an SM, 8 / 4 / 2: 18, 37 or 74 chains on 148 SMs.  The columns kernel / this one, us:
      // 8 chains 12 tokens 5.2 / 5.1 (8 tokens 4.4 / 4.7), 16 tokens 6.1 / 6.1, 37 tokens 11.5 / 9.4; 16 chains 8 tokens 5.2 / 4.9, 37 tokens
      // 13.9 / 9.5; 32 chains 4 tokens 5.5 / 4.9, 37 tokens 16.5 / 11.1, 63 tokens 25.0 / 16.5; 64 chains 4 tokens 5.6 / 5.8, 8 tokens 7.1 /
      // 7.2, 13 tokens 9.3 / 8.4, 37 tokens 18.8 / 15.8, 63 tokens 29.4 / 23.7.  More chains stay with the columns kernel, whose smaller CTAs
      // share an SM (this one with two CTAs a chain, 96 chains: 24.9 / 30.4, 256: 53.0 / 60.0), and states off the 16-byte boundary too.
      // Between those counts: 10, 12 and 15 chains 2 tokens 3.4 / 3.0-3.2, 4 tokens 3.7 / 3.5, 8 tokens 4.7 / 4.3, 12 tokens 5.9 / 5.0; 20, 24, 30
      // and 36 chains 4 tokens 4.5-5.4 / 3.6, 12 tokens 7.4-8.8 / 5.4; 38 to 63 chains 9 tokens 8.4-10.5 / 6.6, and their 4 to 8 tokens by the
      // columns kernel with four columns a lane 4.9-6.6, with two 6.2-9.6.
      const int per_chain = (int)std::min<int64_t>(sm_count() / chains, 8);
      const int more_than = per_chain < 4 ? 8 : (chains <= sm_count() / 16 ? 12 : 0);
      if (aligned(state, 16) && per_chain >= 2 && seqlen > more_than) {
        auto kern = per_chain == 8 ? kda_recurrent_few_kernel<2, 16> : (per_chain >= 4 ? kda_recurrent_few_kernel<4, 16> : kda_recurrent_few_kernel<4, 8>);
        return pdl_launch(kern, dim3(bsz, num_v_heads, per_chain == 8 ? 8 : (per_chain >= 4 ? 4 : 2)), dim3(2 * RC_WARPS * 32), 0, s, q, g, bt, state, o,
                          out_f32, seqlen, num_k_heads, num_v_heads, 1.0f / sqrtf(128.0f), slots) == cudaSuccess
                   ? HK_OK
                   : HK_ERR_CUDA;
      }
      const bool one = !aligned(state, 16) || chains < 16;
      return pdl_launch(one ? kda_recurrent_cols_kernel<1> : kda_recurrent_cols_kernel<4>, dim3(bsz, num_v_heads, one ? 16 : 4), dim3(RC_WARPS * 32), 0, s, q,
                        g, bt, state, o, out_f32, seqlen, num_k_heads, num_v_heads, 1.0f / sqrtf(128.0f), slots) == cudaSuccess
                 ? HK_OK
                 : HK_ERR_CUDA;
    }
  }
  if (channelwise)
    return launch_rows(q, g, bt, state, o, out_f32, bsz, seqlen, num_k_heads, num_v_heads, history_stride, slots, history, s);
  if (k_head_dim == 128)
    return narrow_slices(bsz, num_v_heads)
               ? launch_recurrent<128, 16>(q, g, bt, state, o, out_f32, bsz, seqlen, num_k_heads, num_v_heads, history_stride, slots, history, s)
               : launch_recurrent<128, 32>(q, g, bt, state, o, out_f32, bsz, seqlen, num_k_heads, num_v_heads, history_stride, slots, history, s);
  if (k_head_dim == 64)
    return launch_recurrent<64, 32>(q, g, bt, state, o, out_f32, bsz, seqlen, num_k_heads, num_v_heads, history_stride, slots, history, s);
  return HK_ERR_UNSUPPORTED;
}

HK_API int hk_kda_decode_step(const void* x, void* conv_state, const void* conv_weight, const void* conv_bias, const float* g,
                              const void* beta, float* rec_state, void* out, float* out_f32, void* conv_out, int bsz,
                              int num_heads, const int* slots, int* tickets, void* stream) {
  using namespace hk;
  HK_REQUIRE(x && conv_state && conv_weight && g && beta && rec_state && out);
  (void)tickets;
  HK_REQUIRE(bsz > 0 && bsz <= 65535 && num_heads > 0 && num_heads <= 65535);
  HK_REQUIRE(aligned(conv_state, 8) && aligned(conv_weight, 8));   // a channel's window and taps are one access each
  DecodeArgs a{};
  a.x = x;
  a.conv_state = (__nv_bfloat16*)conv_state;
  a.conv_w = (const __nv_bfloat16*)conv_weight;
  a.conv_bias = (const __nv_bfloat16*)conv_bias;
  a.g = g;
  a.beta = beta;
  a.state = rec_state;
  a.out = (__nv_bfloat16*)out;
  a.out_f32 = out_f32;
  a.conv_out = (__nv_bfloat16*)conv_out;
  a.scale = 1.0f / sqrtf(128.0f);
  a.H = a.Hk = num_heads;
  a.n_heads = bsz * num_heads;
  a.slots = slots;
  return launch_decode<DEC_STEP>(a, as_stream(stream));
}

namespace hk {
static int decode_layer(const float* x32, void* conv_state, const void* conv_weight, const void* conv_bias, const float* f, const float* b,
                        const float* dt_bias, const float* a_log, float lower_bound, float* rec_state, void* out, float* out_f32,
                        const void* norm_w, int w_type, const void* gate_out, int g_type, void* y, int y_type, float epsilon, float constant_bias,
                        int gate_act, int bsz, int num_heads, const int* slots, bool beside, void* stream) {
  HK_REQUIRE(x32 && conv_state && conv_weight && f && b && dt_bias && a_log && rec_state && out && norm_w && gate_out && y);
  HK_REQUIRE(bsz > 0 && bsz <= 65535 && num_heads > 0 && num_heads <= 65535);
  HK_REQUIRE(w_type == HK_F32 || w_type == HK_BF16);
  HK_REQUIRE(y_type == HK_F32 || y_type == HK_F16);
  HK_REQUIRE(g_type == HK_F32 || g_type == HK_BF16);
  HK_REQUIRE(gate_act == 0 || gate_act == 1);
  HK_REQUIRE(aligned(conv_state, 8) && aligned(conv_weight, 8));
  HK_REQUIRE(aligned(out, 8) && aligned(norm_w, w_type == HK_F32 ? 16 : 8) && aligned(y, y_type == HK_F32 ? 16 : 8) &&
             aligned(gate_out, g_type == HK_F32 ? 16 : 8));
  DecodeArgs a{};
  a.x = x32;
  a.conv_state = (__nv_bfloat16*)conv_state;
  a.conv_w = (const __nv_bfloat16*)conv_weight;
  a.conv_bias = (const __nv_bfloat16*)conv_bias;
  a.g = f;
  a.beta = b;
  a.dt_bias = dt_bias;
  a.a_log = a_log;
  a.lower_bound = lower_bound;
  a.state = rec_state;
  a.out = (__nv_bfloat16*)out;
  a.out_f32 = out_f32;
  a.norm_w = norm_w;
  a.gate_out = gate_out;
  a.y = y;
  a.w_bf16 = w_type == HK_BF16;
  a.g_bf16 = g_type == HK_BF16;
  a.y_f16 = y_type == HK_F16;
  a.gate_act = gate_act;
  a.eps = epsilon;
  a.cbias = constant_bias;
  a.scale = 1.0f / sqrtf(128.0f);
  a.H = a.Hk = num_heads;
  a.n_heads = bsz * num_heads;
  a.slots = slots;
  return launch_decode<DEC_LAYER>(a, as_stream(stream), beside);
}
}  // namespace hk

HK_API int hk_kda_decode_layer(const float* x32, void* conv_state, const void* conv_weight, const void* conv_bias, const float* f, const float* b,
                               const float* dt_bias, const float* a_log, float lower_bound, float* rec_state, void* out, float* out_f32,
                               const void* norm_w, int w_type, const void* gate_out, int g_type, void* y, int y_type, float epsilon,
                               float constant_bias, int gate_act, int bsz, int num_heads, const int* slots, int* /*tickets*/, void* stream) {
  return hk::decode_layer(x32, conv_state, conv_weight, conv_bias, f, b, dt_bias, a_log, lower_bound, rec_state, out, out_f32, norm_w, w_type,
                          gate_out, g_type, y, y_type, epsilon, constant_bias, gate_act, bsz, num_heads, slots, false, stream);
}
HK_API int hk_kda_decode_layer_beside(const float* x32, void* conv_state, const void* conv_weight, const void* conv_bias, const float* f,
                                      const float* b, const float* dt_bias, const float* a_log, float lower_bound, float* rec_state, void* out,
                                      float* out_f32, const void* norm_w, int w_type, const void* gate_out, int g_type, void* y, int y_type,
                                      float epsilon, float constant_bias, int gate_act, int bsz, int num_heads, const int* slots, int* /*tickets*/,
                                      void* stream) {
  return hk::decode_layer(x32, conv_state, conv_weight, conv_bias, f, b, dt_bias, a_log, lower_bound, rec_state, out, out_f32, norm_w, w_type,
                          gate_out, g_type, y, y_type, epsilon, constant_bias, gate_act, bsz, num_heads, slots, true, stream);
}
