// KDA short convolution: depthwise causal conv (window K) + SiLU over channel-major input, with a
// rolling window state.  Interface and arithmetic of helios::aux::cuda_causal_conv1d_update
// (reference: src/cuda/aux/gdn.cu:880-1023): fp32 fma chain k ascending, SiLU as a * 1/(1+exp(-a)),
// bf16 round-to-nearest output, state = last K inputs.
//
// Three kernels (the last one is the fused cast + convolution over token-major fp32 input, further below):
//   conv4_row_kernel    prefill (K = 4, no history, 16 tokens or more): persistent CTAs over [64 channel][64 token] tiles,
//                       asynchronous 16-byte copies into a three-stage ring, a lane computes 2 channels x 16 tokens
//                       (128-byte warp stores per output row).
//   conv_generic_kernel decode and every other case (any K <= 16, history, ragged shapes): one
//                       thread per channel; with seqlen = 1 its accesses are contiguous in channels.
#include <type_traits>

#include "hk_common.cuh"

namespace hk {

constexpr int CONV_MAX_K = 16;
constexpr int CT_CH = 64;       // channels per tile

__device__ __forceinline__ float silu_fast(float a) { return a * (1.0f / (1.0f + __expf(-a))); }

// Prefill.  2 B are read and 2 B written
// per channel-token; what a transposing access pattern reaches depends on the length of its runs, and the SiLU's exponential
// and reciprocal (230 us at 32,768 tokens x 12,288 channels on the special-function units alone) have to run under the copies.
// With 32 bytes per channel row and lane, straight into registers, that size took 362 us (4.45 TB/s; runs of 128 bytes copy in
// 268).  So the tile goes through shared memory, copied in asynchronously two tiles ahead: 324 us, and 16.8 -> 14.1 at 1,008
// tokens, 613 -> 331 at 32,760.  The 16-byte piece p of row r sits at p ^ (r / 2 % 8), which keeps the copies (8 lanes to a
// row) and the reads (32 lanes on rows 2 l and 2 l + 1) free of bank conflicts.  Small CTAs because one's barrier then stalls
// only four warps: 64-token tiles and six CTAs per SM 324 us, 128-token tiles and three or four 339, 353; five 345, eight 434
// (too many streams for the memory).
// RAGGED: the rows of a length that is no multiple of 8 start anywhere.  Then a row of the tile is the aligned 16-byte pieces
// that cover the 4 tokens before it and its own, up to ten, and is read word by word, rows that start on an odd element through
// a 16-bit funnel shift.  Rows lie 11 pieces apart, even ones first, so that the words of 32 lanes spread over all banks.  One
// element per load before: 690 -> 407 us at 32,763 tokens, 27.4 -> 17.1 at 1,003.
constexpr int CW_TOK = 64, CW_THREADS = CW_TOK * 2, CW_STAGES = 3, CW_CTAS = 6;
constexpr uint32_t CW_TILE = CT_CH * CW_TOK * 2, CW_PITCH = 11 * 16;
// 8 KB and the 4 tokens before each row, or 64 rows of up to ten pieces
__host__ __device__ constexpr uint32_t cw_stage(bool ragged) { return ragged ? CT_CH * CW_PITCH : CW_TILE + CT_CH * 8; }

// BRIEF: calls of at most 64 tokens and a tile per CTA, whose taps and window are asked for under the copies; one after the other they were a
// fifth of such a call (37 tokens x 24,576 channels 5.6 -> 4.6 us).  In the form for many tiles the registers for it cost more: 32,768 tokens
// 324 -> 336.
template <bool ACT, bool RAGGED, bool BRIEF>
__global__ __launch_bounds__(CW_THREADS, CW_CTAS) void conv4_row_kernel(
    const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ state,
    const int* __restrict__ slots, const __nv_bfloat16* __restrict__ weight,
    const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ out, int dim, int seqlen,
    int state_size, int tok_tiles, int total, size_t n_elem) {
  constexpr uint32_t CW_STAGE = cw_stage(RAGGED);
  extern __shared__ __align__(128) uint8_t smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const uint32_t sm0 = (uint32_t)__cvta_generic_to_shared(smem_raw);
  // tiles run over channels, tokens, batch: the CTAs at work write whole output rows.  A place in that order is moved on by the
  // grid without divisions.
  const int ch_tiles = dim / CT_CH, step_t = gridDim.x / ch_tiles, step_c = gridDim.x - step_t * ch_tiles;
  struct Place {
    int t, c, s, b;                                          // tile, channel tile, token tile, batch
  };
  auto advance = [&](Place& p) {
    p.t += gridDim.x;
    p.c += step_c;
    p.s += step_t;
    if (p.c >= ch_tiles) {
      p.c -= ch_tiles;
      p.s++;
    }
    while (p.s >= tok_tiles) {
      p.s -= tok_tiles;
      p.b++;
    }
  };
  const int cr = tid >> 3, cp = tid & 7;                     // copies: rows cr + 16 i, piece cp
  const uint32_t dst = sm0 + cr * 128 + ((cp ^ ((cr >> 1) & 7)) << 4);
  const size_t row16 = (size_t)seqlen * 16;
  auto copy_in = [&](const Place& p, int stage) {
    const __nv_bfloat16* xb = x + ((size_t)p.b * dim + p.c * CT_CH) * seqlen + p.s * CW_TOK;
    if (RAGGED) {
#pragma unroll
      for (int i = 0; i < 5; i++) {                          // pieces 0-7 with eight lanes to a row, then 8 and 9
        const int r = i < 4 ? cr + 16 * i : tid >> 1, pc = i < 4 ? cp : 8 + (tid & 1);
        const uintptr_t row = reinterpret_cast<uintptr_t>(xb + (size_t)r * seqlen);
        const uintptr_t src = ((row - 8) & ~(uintptr_t)15) + 16 * pc;
        if (src >= row + 2 * min(CW_TOK, seqlen - p.s * CW_TOK)) continue;
        const uint32_t to = stage * CW_STAGE + ((r >> 1) + 32 * (r & 1)) * CW_PITCH + 16 * pc;
        if (src >= reinterpret_cast<uintptr_t>(x) && src + 16 <= reinterpret_cast<uintptr_t>(x + n_elem)) {
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(sm0 + to), "l"(src) : "memory");
        } else {                                             // over an end of the whole input: element by element
#pragma unroll
          for (int e = 0; e < 8; e++) {
            const __nv_bfloat16* q = reinterpret_cast<const __nv_bfloat16*>(src) + e;
            if (q >= x && q < x + n_elem) reinterpret_cast<__nv_bfloat16*>(smem_raw + to)[e] = *q;
          }
        }
      }
      return;
    }
    if (p.s * CW_TOK + 8 * cp < seqlen) {
      const __nv_bfloat16* src = xb + (size_t)cr * seqlen + 8 * cp;
#pragma unroll
      for (int i = 0; i < 4; i++)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + stage * CW_STAGE + i * 2048), "l"(src + i * row16)
                     : "memory");
    }
    if (tid < CT_CH && p.s > 0)
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(sm0 + stage * CW_STAGE + CW_TILE + tid * 8),
                   "l"(xb + (size_t)tid * seqlen - 4)
                   : "memory");
  };
  Place in;
  in.t = blockIdx.x;
  in.s = in.t / ch_tiles;
  in.c = in.t - in.s * ch_tiles;
  in.b = in.s / tok_tiles;
  in.s -= in.b * tok_tiles;
  Place at = in;
  pdl_wait();
#pragma unroll
  for (int i = 0; i < CW_STAGES - 1; i++) {
    if (in.t < total) copy_in(in, i);
    advance(in);
    asm volatile("cp.async.commit_group;" ::: "memory");
  }
  int stage = 0;
  for (; at.t < total; advance(at)) {
    uint4 wv;
    uint16_t win[2][3], next[2][4];                          // BRIEF: the window's last three inputs, the window to come
    if (BRIEF) {
      const int c0 = at.c * CT_CH + lane * 2;
      wv = *reinterpret_cast<const uint4*>(weight + (size_t)c0 * 4);
      if (wid == 0) {
        const int slot = slots ? slots[at.b] : at.b;
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint16_t* u = reinterpret_cast<const uint16_t*>(state + ((size_t)slot * dim + c0 + h) * state_size);
          const uint16_t* r = reinterpret_cast<const uint16_t*>(x + ((size_t)at.b * dim + c0 + h + 1) * seqlen - 4);
#pragma unroll
          for (int k = 0; k < 3; k++) win[h][k] = u[k + 1];
#pragma unroll
          for (int k = 0; k < 4; k++) next[h][k] = r[k];
        }
      }
    }
    asm volatile("cp.async.wait_group %0;" ::"n"(CW_STAGES - 2) : "memory");
    __syncthreads();                                         // everyone's pieces are there, and the stage before is done with
    if (in.t < total) copy_in(in, stage == 0 ? CW_STAGES - 1 : stage - 1);
    advance(in);
    asm volatile("cp.async.commit_group;" ::: "memory");
    const int c0 = at.c * CT_CH + lane * 2, b = at.b;
    const uint8_t* rows = smem_raw + stage * CW_STAGE + lane * (RAGGED ? CW_PITCH : 256);   // channels c0 and c0 + 1
    const int t0 = at.s * CW_TOK + wid * 16;
    stage = stage == CW_STAGES - 1 ? 0 : stage + 1;
    if (t0 >= seqlen) continue;                              // warp-uniform
    uint2 pa, pe;                                            // tokens t0-4 .. t0-1 (the first is not used)
    if (t0 == 0) {
      // the first group takes its predecessors from the window state and rolls the state forward
      const int slot = slots ? slots[b] : b;
      __nv_bfloat16* st0 = state + ((size_t)slot * dim + c0) * state_size;
      __nv_bfloat16* st1 = st0 + state_size;
      if (BRIEF) {
        pa = make_uint2((uint32_t)win[0][0] << 16, (uint32_t)win[0][1] | ((uint32_t)win[0][2] << 16));
        pe = make_uint2((uint32_t)win[1][0] << 16, (uint32_t)win[1][1] | ((uint32_t)win[1][2] << 16));
#pragma unroll
        for (int k = 0; k < 4; k++) {
          reinterpret_cast<uint16_t*>(st0)[k] = next[0][k];
          reinterpret_cast<uint16_t*>(st1)[k] = next[1][k];
        }
      } else {
        const uint16_t* u0 = reinterpret_cast<const uint16_t*>(st0);
        const uint16_t* u1 = reinterpret_cast<const uint16_t*>(st1);
        pa = make_uint2((uint32_t)u0[1] << 16, (uint32_t)u0[2] | ((uint32_t)u0[3] << 16));
        pe = make_uint2((uint32_t)u1[1] << 16, (uint32_t)u1[2] | ((uint32_t)u1[3] << 16));
        const __nv_bfloat16* r0 = x + ((size_t)b * dim + c0) * seqlen;
#pragma unroll
        for (int k = 0; k < 4; k++) {                          // seqlen >= 16: the new window is the last 4 inputs
          st0[k] = r0[seqlen - 4 + k];
          st1[k] = r0[2 * (size_t)seqlen - 4 + k];
        }
      }
    } else if (!RAGGED) {
      if (wid == 0) {
        const uint4 h = *reinterpret_cast<const uint4*>(rows - lane * 256 + CW_TILE + lane * 16);
        pa = make_uint2(h.x, h.y);
        pe = make_uint2(h.z, h.w);
      } else {
        const int o = ((2 * wid - 1) ^ (lane & 7)) << 4;
        pa = *reinterpret_cast<const uint2*>(rows + o + 8);
        pe = *reinterpret_cast<const uint2*>(rows + 128 + o + 8);
      }
    }
    uint32_t wa[8], we[8];                                   // 16 tokens of either channel
    if (RAGGED) {
      uint32_t v[2][11];                                     // from token t0 - 4 (or the element before it) on
#pragma unroll
      for (int h = 0; h < 2; h++) {
        const uintptr_t row = reinterpret_cast<uintptr_t>(x + ((size_t)b * dim + c0 + h) * seqlen + at.s * CW_TOK) - 8;
        const int lead = (int)(row & 15) >> 1;
        const uint32_t* src = reinterpret_cast<const uint32_t*>(rows + h * 32 * CW_PITCH) + (lead >> 1) + wid * 8;
#pragma unroll
        for (int i = 0; i < 11; i++) v[h][i] = src[i];
        const uint32_t sh = 16 * (lead & 1);
#pragma unroll
        for (int i = 0; i < 10; i++) v[h][i] = __funnelshift_r(v[h][i], v[h][i + 1], sh);
      }
      if (t0 > 0) {
        pa = make_uint2(v[0][0], v[0][1]);
        pe = make_uint2(v[1][0], v[1][1]);
      }
#pragma unroll
      for (int i = 0; i < 8; i++) {
        wa[i] = v[0][2 + i];
        we[i] = v[1][2 + i];
      }
    } else {
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int o = ((2 * wid + j) ^ (lane & 7)) << 4;
        const uint4 ra = *reinterpret_cast<const uint4*>(rows + o), re = *reinterpret_cast<const uint4*>(rows + 128 + o);
        wa[4 * j] = ra.x; wa[4 * j + 1] = ra.y; wa[4 * j + 2] = ra.z; wa[4 * j + 3] = ra.w;
        we[4 * j] = re.x; we[4 * j + 1] = re.y; we[4 * j + 2] = re.z; we[4 * j + 3] = re.w;
      }
    }
    if (!BRIEF) wv = *reinterpret_cast<const uint4*>(weight + (size_t)c0 * 4);
    const uint64_t w0 = pack2(bf16lo(wv.x), bf16lo(wv.z)), w1 = pack2(bf16hi(wv.x), bf16hi(wv.z));
    const uint64_t w2 = pack2(bf16lo(wv.y), bf16lo(wv.w)), w3 = pack2(bf16hi(wv.y), bf16hi(wv.w));
    const uint64_t bs = bias ? pack2(__bfloat162float(bias[c0]), __bfloat162float(bias[c0 + 1])) : 0;
    uint64_t a0 = pack2(bf16hi(pa.x), bf16hi(pe.x)), a1 = pack2(bf16lo(pa.y), bf16lo(pe.y)), a2 = pack2(bf16hi(pa.y), bf16hi(pe.y));
    __nv_bfloat16* ob = out + ((size_t)b * seqlen + t0) * dim + c0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
      if ((RAGGED || i == 8) && t0 + i >= seqlen) break;
      const uint32_t a = wa[i >> 1], e = we[i >> 1];
      const uint64_t a3 = i & 1 ? pack2(bf16hi(a), bf16hi(e)) : pack2(bf16lo(a), bf16lo(e));
      float y0, y1;
      unpack2(fma2(w3, a3, fma2(w2, a2, fma2(w1, a1, fma2(w0, a0, bs)))), y0, y1);
      if (ACT) {
        y0 = silu_fast(y0);
        y1 = silu_fast(y1);
      }
      *reinterpret_cast<__nv_bfloat162*>(ob) = __floats2bfloat162_rn(y0, y1);
      ob += dim;
      a0 = a1; a1 = a2; a2 = a3;
    }
  }
}

template <bool ACT, bool HISTORY>
__global__ __launch_bounds__(256) void conv_generic_kernel(
    const __nv_bfloat16* __restrict__ x, __nv_bfloat16* __restrict__ state,
    const int* __restrict__ slots, const __nv_bfloat16* __restrict__ weight,
    const __nv_bfloat16* __restrict__ bias, __nv_bfloat16* __restrict__ out, int dim, int seqlen,
    int state_size, int K) {
  pdl_wait();
  const int d = blockIdx.x * 256 + threadIdx.x;
  if (d >= dim) return;
  const int b = blockIdx.y;
  const int slot = slots ? slots[b] : b;
  const __nv_bfloat16* x_d = x + ((size_t)b * dim + d) * seqlen;
  __nv_bfloat16* st = state + ((size_t)slot * dim + d) * state_size;
  float w[CONV_MAX_K], old[CONV_MAX_K], win[CONV_MAX_K];
#pragma unroll
  for (int k = 0; k < CONV_MAX_K; k++)
    if (k < K) {
      w[k] = __bfloat162float(weight[(size_t)d * K + k]);
      old[k] = __bfloat162float(st[k]);
    }
#pragma unroll
  for (int k = 0; k < CONV_MAX_K - 1; k++)
    if (k < K - 1) win[k] = old[k + 1];
  const float bias_d = bias ? __bfloat162float(bias[d]) : 0.0f;
  for (int s = 0; s < seqlen; s++) {
    float cur = __bfloat162float(x_d[s]);
    float acc = bias_d;
#pragma unroll
    for (int k = 0; k < CONV_MAX_K; k++)
      if (k < K) acc = fmaf(w[k], (k == K - 1) ? cur : win[k], acc);
    if (ACT) acc = silu_fast(acc);
    out[((size_t)b * seqlen + s) * dim + d] = __float2bfloat16_rn(acc);
#pragma unroll
    for (int k = 0; k < CONV_MAX_K - 1; k++)
      if (k < K - 1) win[k] = (k == K - 2) ? cur : win[k + 1];
  }
  if (!HISTORY) {
#pragma unroll
    for (int k = 0; k < CONV_MAX_K; k++)
      if (k < K) {
        int src_t = seqlen + k;
        float v = (src_t < K) ? old[src_t] : __bfloat162float(x_d[src_t - K]);
        st[k] = __float2bfloat16_rn(v);
      }
  } else {
    int total = K + seqlen;
    int write_size = state_size < total ? state_size : total;
    int dst_start = state_size - write_size, src_start = total - write_size;
    for (int j = 0; j < write_size; j++) {
      int src_t = src_start + j;
      float v = (src_t < K) ? old[src_t] : __bfloat162float(x_d[src_t - K]);
      st[dst_start + j] = __float2bfloat16_rn(v);
    }
  }
}


// Cast + convolution in one pass over TOKEN-major fp32 input (the projection's own output layout): the
// transposed bf16 copy that the channel-major kernels read is never made.  A thread owns 4 adjacent
// channels (one 16-byte load per token; a warp reads 512 contiguous bytes of a token row and writes 256)
// and walks CR_TOK consecutive tokens with the three previous inputs in registers.  Inputs are rounded
// to bf16 first, so the result equals transpose-cast followed by the channel-major convolution, bit for
// bit.  x [bsz][seqlen][dim] f32, out [bsz][seqlen][dim] bf16, state [slots][dim][4] bf16.
// 64 tokens per thread, 16 in short calls: 1,003 tokens x 12,288 channels gave 384 CTAs of 64, eight round trips to memory in a
// row each (22 us); while 64-token CTAs do not fill every slot of the GPU, more and shorter ones hide more of it.
// Channel pairs in packed instructions and six CTAs per SM: HBM-bound (6 B per element), but with scalar ones the instruction
// stream held it to 5.7 TB/s (8 x 4,096 tokens x 12,288 channels 426 -> 377 us, 1,003 tokens 18.6 -> 14.6).
constexpr int CR_TOK = 64, CR_TOK_SHORT = 16;

__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }

template <bool ACT, int TOK>
__global__ __launch_bounds__(128, 6) void conv4_cast_rows_kernel(
    const float* __restrict__ x, __nv_bfloat16* __restrict__ state, const int* __restrict__ slots,
    const __nv_bfloat16* __restrict__ weight, const __nv_bfloat16* __restrict__ bias,
    __nv_bfloat16* __restrict__ out, int dim, int seqlen) {
  pdl_wait();
  const int c = (blockIdx.x * 128 + threadIdx.x) * 4;
  if (c >= dim) return;
  const int s0 = blockIdx.y * TOK, b = blockIdx.z;
  const int s1 = min(s0 + TOK, seqlen);
  const float* xb = x + (size_t)b * seqlen * dim + c;
  float w[4][4], bs[4] = {0.f, 0.f, 0.f, 0.f};
  {
    const uint4 w01 = *reinterpret_cast<const uint4*>(weight + (size_t)c * 4);
    const uint4 w23 = *reinterpret_cast<const uint4*>(weight + (size_t)c * 4 + 8);
    const uint32_t ww[8] = {w01.x, w01.y, w01.z, w01.w, w23.x, w23.y, w23.z, w23.w};
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
      w[ch][0] = bf16lo(ww[2 * ch]); w[ch][1] = bf16hi(ww[2 * ch]);
      w[ch][2] = bf16lo(ww[2 * ch + 1]); w[ch][3] = bf16hi(ww[2 * ch + 1]);
    }
    if (bias) {
#pragma unroll
      for (int ch = 0; ch < 4; ch++) bs[ch] = __bfloat162float(bias[c + ch]);
    }
  }
  float h0[4], h1[4], h2[4];                                // inputs s-3, s-2, s-1 of the four channels
  if (s0 == 0) {
    // the first segment takes its predecessors from the window state and rolls the state forward
    const int slot = slots ? slots[b] : b;
    __nv_bfloat16* st = state + ((size_t)slot * dim + c) * 4;
    const uint4 o01 = *reinterpret_cast<const uint4*>(st), o23 = *reinterpret_cast<const uint4*>(st + 8);
    const uint32_t ow[8] = {o01.x, o01.y, o01.z, o01.w, o23.x, o23.y, o23.z, o23.w};
    uint32_t nw[8];
#pragma unroll
    for (int ch = 0; ch < 4; ch++) {
      const float old[4] = {bf16lo(ow[2 * ch]), bf16hi(ow[2 * ch]), bf16lo(ow[2 * ch + 1]), bf16hi(ow[2 * ch + 1])};
      h0[ch] = old[1]; h1[ch] = old[2]; h2[ch] = old[3];
      float nv[4];
#pragma unroll
      for (int k = 0; k < 4; k++) {                          // new window = last 4 of [old | x]
        const int src_t = seqlen + k;
        nv[k] = src_t < 4 ? old[src_t] : xb[(size_t)(src_t - 4) * dim + ch];
      }
      nw[2 * ch] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(nv[0])) |
                   ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(nv[1])) << 16);
      nw[2 * ch + 1] = (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(nv[2])) |
                       ((uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(nv[3])) << 16);
    }
    *reinterpret_cast<uint4*>(st) = make_uint4(nw[0], nw[1], nw[2], nw[3]);
    *reinterpret_cast<uint4*>(st + 8) = make_uint4(nw[4], nw[5], nw[6], nw[7]);
  } else {
    const float4 p0 = *reinterpret_cast<const float4*>(xb + (size_t)(s0 - 3) * dim);
    const float4 p1 = *reinterpret_cast<const float4*>(xb + (size_t)(s0 - 2) * dim);
    const float4 p2 = *reinterpret_cast<const float4*>(xb + (size_t)(s0 - 1) * dim);
    h0[0] = round_bf16(p0.x); h0[1] = round_bf16(p0.y); h0[2] = round_bf16(p0.z); h0[3] = round_bf16(p0.w);
    h1[0] = round_bf16(p1.x); h1[1] = round_bf16(p1.y); h1[2] = round_bf16(p1.z); h1[3] = round_bf16(p1.w);
    h2[0] = round_bf16(p2.x); h2[1] = round_bf16(p2.y); h2[2] = round_bf16(p2.z); h2[3] = round_bf16(p2.w);
  }
  __nv_bfloat16* ob = out + (size_t)b * seqlen * dim + c;
  uint64_t wp[2][4], bp[2], p0[2], p1[2], p2[2];             // channel pairs
#pragma unroll
  for (int c2 = 0; c2 < 2; c2++) {
#pragma unroll
    for (int k = 0; k < 4; k++) wp[c2][k] = pack2(w[2 * c2][k], w[2 * c2 + 1][k]);
    bp[c2] = pack2(bs[2 * c2], bs[2 * c2 + 1]);
    p0[c2] = pack2(h0[2 * c2], h0[2 * c2 + 1]);
    p1[c2] = pack2(h1[2 * c2], h1[2 * c2 + 1]);
    p2[c2] = pack2(h2[2 * c2], h2[2 * c2 + 1]);
  }
  for (int t0 = s0; t0 < s1; t0 += 8) {
    uint4 raw[8];
#pragma unroll
    for (int j = 0; j < 8; j++)
      raw[j] = t0 + j < s1 ? ld_stream16(xb + (size_t)(t0 + j) * dim) : make_uint4(0, 0, 0, 0);
#pragma unroll
    for (int j = 0; j < 8; j++) {
      if (t0 + j >= s1) break;
      const uint32_t rw[4] = {raw[j].x, raw[j].y, raw[j].z, raw[j].w};
      uint32_t pk[2];
#pragma unroll
      for (int c2 = 0; c2 < 2; c2++) {
        const __nv_bfloat162 xr = __floats2bfloat162_rn(__uint_as_float(rw[2 * c2]), __uint_as_float(rw[2 * c2 + 1]));
        const uint32_t xw = *reinterpret_cast<const uint32_t*>(&xr);
        const uint64_t cur = pack2(bf16lo(xw), bf16hi(xw));
        float y0, y1;
        unpack2(fma2(wp[c2][3], cur, fma2(wp[c2][2], p2[c2], fma2(wp[c2][1], p1[c2], fma2(wp[c2][0], p0[c2], bp[c2])))), y0, y1);
        if (ACT) {
          y0 = silu_fast(y0);
          y1 = silu_fast(y1);
        }
        p0[c2] = p1[c2]; p1[c2] = p2[c2]; p2[c2] = cur;
        const __nv_bfloat162 yr = __floats2bfloat162_rn(y0, y1);
        pk[c2] = *reinterpret_cast<const uint32_t*>(&yr);
      }
      *reinterpret_cast<uint2*>(ob + (size_t)(t0 + j) * dim) = make_uint2(pk[0], pk[1]);
    }
  }
}

}  // namespace hk

HK_API int hk_kda_cast_conv(const float* x, void* conv_state, const int* slots, const void* weight,
                            const void* bias, void* out, int bsz, int dim, int seqlen, int activation,
                            void* stream) {
  using namespace hk;
  HK_REQUIRE(x && conv_state && weight && out);
  HK_REQUIRE(bsz > 0 && bsz <= 65535 && dim > 0 && dim % 4 == 0 && seqlen > 0);
  HK_REQUIRE((seqlen + CR_TOK - 1) / CR_TOK <= 65535);
  HK_REQUIRE(aligned(x, 16) && aligned(conv_state, 16) && aligned(weight, 16) && aligned(out, 8));
  const int groups = (dim / 4 + 127) / 128;
  const bool brief = (int64_t)groups * ((seqlen + CR_TOK - 1) / CR_TOK) * bsz < (int64_t)sm_count() * 12;
  const int tok = brief ? CR_TOK_SHORT : CR_TOK;
  auto kern = activation ? (brief ? conv4_cast_rows_kernel<true, CR_TOK_SHORT> : conv4_cast_rows_kernel<true, CR_TOK>)
                         : (brief ? conv4_cast_rows_kernel<false, CR_TOK_SHORT> : conv4_cast_rows_kernel<false, CR_TOK>);
  return pdl_launch(kern, dim3(groups, (seqlen + tok - 1) / tok, bsz), dim3(128), 0, as_stream(stream), x, (__nv_bfloat16*)conv_state,
                    slots, (const __nv_bfloat16*)weight, (const __nv_bfloat16*)bias, (__nv_bfloat16*)out, dim, seqlen) == cudaSuccess
             ? HK_OK
             : HK_ERR_CUDA;
}

HK_API int hk_conv1d_update(const void* x, void* conv_state, const int* slots, const void* weight,
                            const void* bias, void* out, int bsz, int dim, int seqlen,
                            int state_size, int K, int activation, int history, void* stream) {
  using namespace hk;
  HK_REQUIRE(x && conv_state && weight && out);
  HK_REQUIRE(bsz > 0 && dim > 0 && seqlen > 0);
  HK_REQUIRE(K >= 1 && K <= CONV_MAX_K && state_size >= K);
  auto xs = (const __nv_bfloat16*)x;
  auto st = (__nv_bfloat16*)conv_state;
  auto w = (const __nv_bfloat16*)weight;
  auto bs = (const __nv_bfloat16*)bias;
  auto o = (__nv_bfloat16*)out;
  cudaStream_t s = as_stream(stream);

  const bool tile_ok = (K == 4) && !history && (dim % CT_CH == 0) && seqlen >= 16 &&
                       aligned(weight, 16) && aligned(out, 4);
  cudaError_t e;
  const int tok_tiles = (seqlen + CW_TOK - 1) / CW_TOK;
  const int64_t tiles = (int64_t)(dim / CT_CH) * tok_tiles * bsz;
  if (tile_ok && tiles < (1 << 30)) {
    const bool ragged = seqlen % 8 != 0 || !aligned(x, 16);
    const int64_t room = (int64_t)sm_count() * CW_CTAS;
    const bool brief = tok_tiles == 1 && tiles <= room;
    auto pick = [&](auto act, auto rag) {
      constexpr bool A = decltype(act)::value, R = decltype(rag)::value;
      return brief ? conv4_row_kernel<A, R, true> : conv4_row_kernel<A, R, false>;
    };
    const std::true_type yes;
    const std::false_type no;
    auto kern = activation ? (ragged ? pick(yes, yes) : pick(yes, no)) : (ragged ? pick(no, yes) : pick(no, no));
    const uint32_t smem = CW_STAGES * cw_stage(ragged);
    static bool attr_set[64][8] = {{false}};
    int dev = 0;
    cudaGetDevice(&dev);
    const int form = (brief ? 4 : 0) + (activation ? 2 : 0) + ragged;
    if (dev < 0 || dev >= 64 || !attr_set[dev][form]) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return HK_ERR_CUDA;
      if (dev >= 0 && dev < 64) attr_set[dev][form] = true;
    }
    e = pdl_launch(kern, dim3((unsigned)(tiles < room ? tiles : room)), dim3(CW_THREADS), smem, s, xs, st, slots, w, bs, o, dim, seqlen,
                   state_size, tok_tiles, (int)tiles, (size_t)bsz * dim * seqlen);
  } else {
    auto kern = activation ? (history ? conv_generic_kernel<true, true> : conv_generic_kernel<true, false>)
                           : (history ? conv_generic_kernel<false, true> : conv_generic_kernel<false, false>);
    e = pdl_launch(kern, dim3((dim + 255) / 256, bsz), dim3(256), 0, s, xs, st, slots, w, bs, o, dim, seqlen, state_size, K);
  }
  return e == cudaSuccess ? HK_OK : HK_ERR_CUDA;
}
