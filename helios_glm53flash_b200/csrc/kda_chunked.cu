// Chunked KDA prefill (gated delta rule with channelwise decay), chunk = 64 tokens, dk = dv = 128.
// The reference has no chunked kernel: its prefill runs the per-token recurrence with seqlen = n
// (src/engine/runner.cpp:468-471 -> src/cuda/aux/gdn.cu:555-749).  This file computes the same
// function: one persistent launch, or two kernels.
//
// Math, per head, for a chunk with incoming state S0 [128 k][128 v] (q^, k^ = L2-normalised rows,
// G_t = inclusive cumulative log-decay inside the chunk, all exponentials below have arguments <= 0
// except inside one 16-token sub-block):
//   A_ts = sum_c k^_t k^_s e^{G_t-G_s} (s<t),  B_ts = sum_c q^_t k^_s e^{G_t-G_s} (s<=t)
//   T = (I + A diag(beta))^-1                      K+ = k^ e^{G_t},  Q+ = q^ e^{G_t}
//   W = T K+,  Uloc = T V                           Kt = beta_t k^_t e^{G_last-G_t}
//   U = Uloc - W S0                                 (delta-rule residuals of the whole chunk)
//   O = scale (Q+ S0 + (B diag(beta)) U)            S' = diag(e^{G_last}) S0 + Kt^T U
//
// The preparation (prep_unit: kernel 1, or the workers of the fused launch) is parallel over every (batch, head, chunk).  It builds A
// and B on the warp-level tensor cores: 16-token blocks against earlier blocks in fp16 with exponents re-based at block starts (both
// operands at most 1), a block against itself in TF32 (e^{-x} needs the fp32 exponent range; the triangular tiles are smaller than a
// tcgen05 tile).  It inverts the unit-triangular system in fp32-class arithmetic and runs the dense W | Uloc = T [K+ | V] product on
// tcgen05 (weight-stationary M64 N128 K64, twice).  It writes, per chunk, operand tiles that are already in the shared-memory layout the
// scan needs (74,240 bytes).
//   Pairs of blocks were TF32 products of fp32 rows once.  fp16 has the same 11 bits and less range: values below 6e-5 lose bits, below
// 3e-8 they are 0.  What comes of the products, B beta and the inverse T, is stored as fp16 itself, with the same absolute spacing, so the
// operands' loss stays below that of the result.  Error against 64 bits, TF32 -> fp16, 16 seeds, outputs / state: the model's gates 4.19e-4
// -> 4.19e-4 / 2.94e-4 -> 2.94e-4; no decay 5.2 -> 5.1e-4 / 4.6 -> 4.4e-4; e^-8 and e^-12 a block, values in a chunk's first block only, beta
// 1e-6 behind it, keys nearly alike: every ratio within 0.993 and 1.003, the spread of the seeds.
//   What bounds it: latencies.  A unit crosses five barriers of its 256 threads and one product; two units share an SM (128 registers
//   a thread, 110 KB).  Inputs arrive by tensor copies issued as soon as their place is free (the log decays when half of the unit before
//   is over).  A worker's unit takes 20 thousand cycles with two workers on the SM.  It took 22.8 thousand while a warp's accesses met in
//   the same banks (log decays two channels a lane, q and k in 128-byte rows, operand tiles of 8-row pieces: 2,300 of the 7,650 passes of a
//   unit through shared memory and L1 were conflicts, now 700 of 6,100), W left as 16-byte halves of sectors, the flag was stored between
//   two barriers that all wait for, and log decays arrived 1,500 cycles into the unit.  32,768 tokens x 32 heads 0.90 -> 0.80 ms, 8 x 4,096 x
//   32 with gates formed inside 0.95 -> 0.88.
//   Registers decide: everything a thread keeps across stage 2 is the 32 packed left operands; a version that kept the fp32 rows (300
//   bytes of spills, whose reloads miss the L1 that shared memory leaves) took 30 thousand cycles.
// The scan walks the chunks of a chain in order; the fp32 state stays in registers.  Per chunk: D1 = [I ; 0] Uloc + [-W ; Q+] S0 (rows
// 0-63 are U), Kt^T U (state), [. ; B beta] U onto the Q+ S0 rows (outputs), all tcgen05 with TMEM accumulators.
#include <cuda.h>   // CUtensorMap (types only; the encoder is fetched through the runtime at first use)

#include <algorithm>
#include <climits>
#include <cstdlib>

#include "hk_common.cuh"
#include "tc05.cuh"

namespace hk {

constexpr int KC = 64;                    // chunk length
constexpr int KD = 128;                   // head dim (k and v)
// Fused form: ring slots (chunks) per chain slot, a power of two up to 32.  A worker's unit takes ten chunks of a chain from the moment
// its ring slot is free; few long chains are waited for by many workers and get the deeper ring where the workspace has the room (the
// query asks for it, a call runs without): 32,768 tokens x 8 heads 578 us, 627 with the ring of 16; x 16 heads 582 / 621; x 1 548 / 583.
// Many chains keep theirs within L2.
constexpr int RING = 16, DEEP_RING = 32;
// Flags: [0] launch-wide abort word, then a 128-byte line of ready flags per chain slot and one for the consumed count per chain CTA.  With all of
// them packed into a few lines of one page the polls of 232 workers held up the chains' own flags: 1.05 or 1.3-1.9 ms for 32,768
// tokens x 32 heads, by the die that the page's address falls to.
constexpr int F_FLAG_INTS = 32;
constexpr int F_LINE = 32;

// ---- per-chunk workspace unit (bytes); every tile is in its final shared-memory layout ----
// (the two operands that the preparation writes from its token rows are in 64-byte-swizzle atoms of 8 tokens x 32 channels: a warp's
// store is one atom, every quarter of it 128 contiguous bytes)
constexpr uint32_t U_WQ = 0;              // fp16 A operand, K-major, rows 0-63 -W, 64-127 Q+ ; K = 128 channels: [16 x 8 rows][4 x 32 channels] atoms
constexpr uint32_t U_UL = 32768;          // fp16 Uloc as B operand, MN-major [16 pieces of 8 columns][64 tokens], token t at t ^ 8
constexpr uint32_t U_BB = 49152;          // fp16 A operand rows (t), K = 64 (s): B_ts beta_s
constexpr uint32_t U_KT = 57344;          // fp16 A operand rows = 128 channels, K = 64 tokens: Kt^T, MN-major: [4 x 32 channels][8 atoms]
constexpr uint32_t U_DEC = 73728;         // f32 e^{G_last}[128]
constexpr uint32_t U_BYTES = 74240;

constexpr uint32_t ATOM = 512;            // bytes of an atom
constexpr uint32_t WQ_ROWS = 4 * ATOM, KT_BLK = 8 * ATOM;   // eight rows of WQ; 32 channels of Kt^T
__device__ __forceinline__ uint32_t atom_off(int r, int c) { return (uint32_t)(r & 7) * 64 + (uint32_t)((c ^ (r >> 1)) & 3) * 16; }   // chunk c of row r

// K-major tile with K = 64 (8 chunks) and no swizzle: LBO 128, SBO 1024
constexpr uint32_t LBO = 128;
constexpr uint32_t SBO_K64 = 1024;

__device__ __forceinline__ uint32_t f2tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// two values rounded toward zero to bf16
__device__ __forceinline__ uint32_t pack_bf2_rz(float lo, float hi) {
  uint32_t r;
  asm("cvt.rz.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}
__device__ __forceinline__ uint32_t pack_h2(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}

// ---- flags in global memory (fused form): release / acquire at GPU scope, bounded polls ----
__device__ __forceinline__ int ld_acquire_gpu(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ int ld_relaxed_gpu(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed_gpu(int* p, int v) {
  asm volatile("st.relaxed.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release_gpu(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
// orders this thread's generic-proxy accesses with its async-proxy accesses (bulk copies) in every state space
__device__ __forceinline__ void fence_proxy_async_all() { asm volatile("fence.proxy.async;" ::: "memory"); }

// Bounded poll of a flag in global memory until it is at least `want`.  Returns false once the CTA has given up
// (this wait or an earlier one) or another CTA has raised the launch-wide abort word.
__device__ __forceinline__ bool poll_flag_ge(const int* flag, int want, volatile int* abort_flag, int* g_abort, int code) {
  if (ld_acquire_gpu(flag) >= want) return true;
  const long long t0 = clock64();
  for (;;) {
    if (*abort_flag) return false;
    if (ld_acquire_gpu(flag) >= want) return true;
    __nanosleep(200);
    if (ld_relaxed_gpu(g_abort) != 0 || clock64() - t0 > tc::MBAR_WAIT_CYCLES) {
      *abort_flag = code;
      atomicExch(g_abort, code);
      return false;
    }
  }
}

// =================================================================================================
// kernel 1: per-chunk preparation.  256 threads, 110 KB of shared memory: two CTAs per SM, so the
// serial stages of one chunk overlap with another chunk's.
// =================================================================================================
// Warp w owns tokens 8 w .. 8 w + 7: lane 4 g8 + tig holds, of token 8 w + g8, the eight channels from 8 tig of every 32, of the
// k row and of the q row.  That is the fragment layout of the warp-level products in both places: as the left operand (rows
// 0-7 of a 16-row tile = k tokens, rows 8-15 = the q rows of the same tokens) and as the right operand (columns = tokens), so the
// product of a warp's tokens with themselves needs no shared memory, and one exponential serves k and q.
// Inputs arrive by tiled tensor copies: v and the log decays in the 128-byte-swizzle pattern (16-byte piece p of row r at p ^ (r % 8)), q and k
// in rows of 64 bytes without a swizzle.
constexpr uint32_t P1_PIECE = 1056;                      // bytes between the 8-channel pieces of K+ (1024 + 32: the four pieces that a
                                                         // quarter-warp writes start in different banks)
constexpr uint32_t P1_X = 0;                             // f32 log decays, then their sums x: four boxes [64 tokens][32 channels]; then the
                                                         // right operands of the even warps' tokens, then the next unit's log decays
constexpr uint32_t P1_V = 32768;                         // v: two boxes [64 tokens][64 channels], bf16 as loaded, fp16 in place: the B operand
constexpr uint32_t P1_RI = 49152;                        // fp16 right operands of the block pairs (i, j < i), 16 tokens x 256 B each;
                                                         // later the T operand (8 KB)
constexpr uint32_t P1_N = P1_RI + 6 * 4096;              // f32 N = A beta: rows 0-31 at a pitch of 36, rows 32-63 at 68
constexpr uint32_t P1_QK = P1_RI;                        // the next unit's q and k, [4 x 32 channels][64 tokens][64 B] each, over the two regions before
constexpr uint32_t P1_K = P1_N + 32 * (36 + 68) * 4;     // fp16 K+, B operand, MN-major, 16 pieces; behind its product W, as it leaves
constexpr uint32_t P1_TAB = P1_K + 16 * P1_PIECE;        // f32 tables [15][128 + 16], then the inverses of the diagonal blocks
constexpr int TAB_LD = KD + 16;                          // (blocks J and J + 1 start in different halves of the banks)
constexpr uint32_t P1_SMEM = (P1_TAB + 15 * TAB_LD * 4 + 1023) / 1024 * 1024;
constexpr int TAB_EP = 0, TAB_ETOT = 4, TAB_KE = 8, TAB_F = 12;   // rows: e^{P_J} | e^{tot_J} | e^{G_last - P_{J+1}} | (2,0), (3,1), (3,0)
static_assert(P1_SMEM % 1024 == 0 && P1_QK % 1024 == 0 && P1_QK + 32768 <= P1_K && P1_TAB % 16 == 0, "layout");
constexpr uint32_t P1_BOX = 8192;
constexpr int P1_LDX = 20;                               // pitch of a diagonal block's inverse

__device__ __forceinline__ int prep_n_row(int t) { return t < 32 ? t * 36 : 32 * 36 + (t - 32) * 68; }
__device__ __forceinline__ int prep_inv_at(int blk) { return blk * 16 * P1_LDX; }

// 16 x 16 left operand of a block product as TF32 heads and tails.  The contraction index is taken in the order in which an
// accumulator holds its columns (k slots tig and tig + 4 of step s are columns 8 s + 2 tig and 8 s + 2 tig + 1), so that the
// accumulator of one product is the left operand of the next without a detour.
struct Frag16 {
  uint32_t h[2][4], l[2][4];
  __device__ __forceinline__ void set(int ks, const float (&f)[4]) {   // f = (row g8: two columns, row g8 + 8: two columns)
    const float a[4] = {f[0], f[2], f[1], f[3]};
#pragma unroll
    for (int e = 0; e < 4; e++) {
      h[ks][e] = f2tf32(a[e]);
      l[ks][e] = f2tf32(a[e] - __uint_as_float(h[ks][e]));
    }
  }
  __device__ __forceinline__ void load(const float* __restrict__ p, int ld, int lane) {
    const int g8 = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int ks = 0; ks < 2; ks++) {
      const float2 u = *reinterpret_cast<const float2*>(p + g8 * ld + 8 * ks + 2 * tig);
      const float2 d = *reinterpret_cast<const float2*>(p + (g8 + 8) * ld + 8 * ks + 2 * tig);
      const float f[4] = {u.x, u.y, d.x, d.y};
      set(ks, f);
    }
  }
};
// two fp32 values of a register pair -> fp16 pair
__device__ __forceinline__ uint32_t pack_h2(uint64_t v) {
  float a, b;
  unpack2(v, a, b);
  return pack_h2(a, b);
}
// 4 register pairs = 8 channels of a token -> one 16-byte fp16 piece
__device__ __forceinline__ uint4 pack_piece(const uint64_t* v) { return make_uint4(pack_h2(v[0]), pack_h2(v[1]), pack_h2(v[2]), pack_h2(v[3])); }
// 8 floats of shared memory as 4 register pairs
__device__ __forceinline__ void load_pairs(const float* __restrict__ p, uint64_t (&v)[4]) {
  const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(p), b = *reinterpret_cast<const ulonglong2*>(p + 4);
  v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
__device__ __forceinline__ float ex2_approx(float x) {
  float r;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ void mma_f16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Right operand of a block product (16 x 16, fp32 in shared memory) as TF32 heads and tails
struct Right16 {
  uint32_t h[2][2][2], l[2][2][2];                         // [k step][column half][k slot]
  __device__ __forceinline__ void load(const float* __restrict__ R, int ld, int lane) {
    const int g8 = lane >> 2, tig = lane & 3;
#pragma unroll
    for (int ks = 0; ks < 2; ks++)
#pragma unroll
      for (int nt = 0; nt < 2; nt++)
#pragma unroll
        for (int u = 0; u < 2; u++) {
          const float b = R[(8 * ks + 2 * tig + u) * ld + 8 * nt + g8];
          h[ks][nt][u] = f2tf32(b);
          l[ks][nt][u] = f2tf32(b - __uint_as_float(h[ks][nt][u]));
        }
  }
};
// acc += L R: the three significant partial products, accumulated in fp32 (in sums of their own: shorter chains), which keeps the
// result at fp32-class accuracy
__device__ __forceinline__ void block16_mma(const Frag16& L, const Right16& R, float (&acc)[2][4]) {
  float lo[2][2][4];
#pragma unroll
  for (int e = 0; e < 16; e++) lo[e >> 3][(e >> 2) & 1][e & 3] = 0.f;
#pragma unroll
  for (int ks = 0; ks < 2; ks++)
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      mma_tf32(lo[0][nt], L.l[ks], R.h[ks][nt][0], R.h[ks][nt][1]);
      mma_tf32(lo[1][nt], L.h[ks], R.l[ks][nt][0], R.l[ks][nt][1]);
      mma_tf32(acc[nt], L.h[ks], R.h[ks][nt][0], R.h[ks][nt][1]);
    }
#pragma unroll
  for (int e = 0; e < 8; e++) acc[e >> 2][e & 3] += lo[0][e >> 2][e & 3] + lo[1][e >> 2][e & 3];
}

__device__ __forceinline__ void block16_mma(const Frag16& L, const float* __restrict__ R, int ld, float (&acc)[2][4], int lane) {
  Right16 r;
  r.load(R, ld, lane);
  block16_mma(L, r, acc);
}

// Row block i of the inverse, right to left: X_ij = - sum_{m = j+1}^{i} X_im P_mj, P_mj = N_mj X_jj (in place of N_mj), one warp,
// all blocks of the row in registers; each leaves as fp16 for the T operand.  Once X_im is known its products with all P_mj are
// formed together, so that only one product per block of the row stands behind another.
template <int I>
__device__ __forceinline__ void prep_inverse_row(const float* __restrict__ sN, const float* __restrict__ sX, uint8_t* __restrict__ sT, int lane) {
  const int g8 = lane >> 2, tig = lane & 3;
  float acc[I][2][4];
#pragma unroll
  for (int j = 0; j < I; j++)
#pragma unroll
    for (int e = 0; e < 8; e++) acc[j][e >> 2][e & 3] = 0.f;
  Frag16 X;
  X.load(sX + prep_inv_at(I), P1_LDX, lane);
#pragma unroll
  for (int m = I; m >= 1; m--) {
#pragma unroll
    for (int j = m - 1; j >= 0; j--) block16_mma(X, sN + prep_n_row(16 * m) + 16 * j, m < 2 ? 36 : 68, acc[j], lane);
    const int j = m - 1;                                   // X_ij is complete
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      const float f[4] = {-acc[j][nt][0], -acc[j][nt][1], -acc[j][nt][2], -acc[j][nt][3]};
      if (j > 0) X.set(nt, f);
      uint8_t* p = sT + (2 * I) * SBO_K64 + (2 * j + nt) * LBO + g8 * 16 + tig * 4;
      *reinterpret_cast<uint32_t*>(p) = pack_h2(f[0], f[1]);
      *reinterpret_cast<uint32_t*>(p + SBO_K64) = pack_h2(f[2], f[3]);
    }
  }
}

// The same with a warp a block: the blocks of the second diagonal need those of the first, X_30 needs X_31 as well.  What a block needs of
// the diagonal it forms ahead, and its other right operands are in registers before the left ones are there, so that one product stands
// behind each of the two barriers (six warps).  What a later block needs goes to shared memory as fp32, in place of N's diagonal
// blocks, which are inverted already; all go to T as fp16.  The shorter way with more instructions: the two-kernel form, whose CTAs are in
// step with one another, gains (1,003 tokens x 32 heads, all calls of the layer: 81.7 -> 76.9 us); where other units fill the gaps it loses
// (fused launch, 8 x 4,096 x 32: 1,455 -> 1,487).
__device__ __forceinline__ void prep_inverse_blocks(float* __restrict__ sN, const float* __restrict__ sX, uint8_t* __restrict__ sT, int warp, int lane, int bar) {
  const int g8 = lane >> 2, tig = lane & 3;
  auto P = [&](int m, int j) { return sN + prep_n_row(16 * m) + 16 * j; };
  auto ldn = [](int m) { return m < 2 ? 36 : 68; };
  // warp: 0 X_10, 1 X_21, 2 X_32, 3 X_20, 4 X_31, 5 X_30
  const int i = warp < 3 ? warp + 1 : warp == 3 ? 2 : 3, j = warp < 3 ? warp : warp == 4 ? 1 : 0;
  float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
  Frag16 L;
  Right16 R;
  auto put = [&](int keep) {                               // keep: the diagonal block whose place it takes, 0 = none
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      const float f[4] = {-acc[nt][0], -acc[nt][1], -acc[nt][2], -acc[nt][3]};
      if (keep) {
        float* x = sN + prep_n_row(16 * keep) + 16 * keep + 8 * nt + 2 * tig;
        *reinterpret_cast<float2*>(x + g8 * ldn(keep)) = make_float2(f[0], f[1]);
        *reinterpret_cast<float2*>(x + (g8 + 8) * ldn(keep)) = make_float2(f[2], f[3]);
      }
      uint8_t* p = sT + (2 * i) * SBO_K64 + (2 * j + nt) * LBO + g8 * 16 + tig * 4;
      *reinterpret_cast<uint32_t*>(p) = pack_h2(f[0], f[1]);
      *reinterpret_cast<uint32_t*>(p + SBO_K64) = pack_h2(f[2], f[3]);
    }
  };
  L.load(sX + prep_inv_at(i), P1_LDX, lane);
  R.load(P(i, j), ldn(i), lane);
  block16_mma(L, R, acc);                                  // X_ii P_ij
  if (warp < 3) put(warp == 0 ? 0 : warp + 1);             // X_21, X_32
  else if (warp == 4) R.load(P(2, 1), ldn(2), lane);
  else R.load(warp == 3 ? P(1, 0) : P(2, 0), ldn(warp == 3 ? 1 : 2), lane);
  asm volatile("bar.sync %0, 192;" ::"r"(bar) : "memory");
  if (warp >= 3) {
    L.load(P(warp == 3 ? 2 : 3, warp == 3 ? 2 : 3), 68, lane);   // X_21 P_10, X_32 P_21, X_32 P_20
    block16_mma(L, R, acc);
    if (warp == 5) R.load(P(1, 0), ldn(1), lane);
    else put(warp == 4 ? 1 : 0);                           // X_31
  }
  if (warp < 4) return;
  asm volatile("bar.sync %0, 64;" ::"r"(bar) : "memory");
  if (warp == 5) {
    L.load(P(1, 1), 36, lane);                             // X_31 P_10
    block16_mma(L, R, acc);
    put(0);
  }
}

// What a preparation worker (256 threads) keeps in static shared memory: its barriers and the units it has at hand (unit number `it`
// at it % 4; thread registers are too few to carry them through a unit).  SUB = false: the worker is a whole CTA with one unit
// (__syncthreads); SUB = true: it is one of the two workers of a CTA and uses the named barriers `bar_id` and `bar_id + 2` (behind a
// unit's last writes).
struct PrepDesc {
  int tok0;                                                // first token: batch * seqlen + 64 * chunk
  int b, t0;                                               // batch, first token in it
  int n_valid;                                             // its tokens, 0: no such unit
  int head;
  int unit;                                                // index of its place in the workspace or ring
  int slot, value;                                         // fused form: chain slot; running chunk number + 1 (the ready flag's value)
};
struct PrepShared {
  uint64_t mma_bar;                                        // the unit's tensor-core product is complete
  uint64_t g_bar;                                          // its gate rows have landed
  uint64_t qkv_bar;                                        // its q, k and v rows
  uint64_t pair_bar[4][4];                                 // right operands of the even warp of block I, channels 32 m .. 32 m + 31
  PrepDesc unit[4];
};
struct PrepCtx {
  uint8_t* smem;
  PrepShared* sh;
  volatile int* abort_flag;
  int tid;
  int bar_id;
};
template <bool SUB>
__device__ __forceinline__ void prep_sync(const PrepCtx& ctx) {
  if (SUB) asm volatile("bar.sync %0, 256;" ::"r"(ctx.bar_id) : "memory");
  else __syncthreads();
}
__device__ __forceinline__ void prep_init(PrepShared& sh) {  // one thread
  tc::mbar_init(&sh.mma_bar, 1);
  tc::mbar_init(&sh.g_bar, 1);
  tc::mbar_init(&sh.qkv_bar, 1);
  for (int i = 0; i < 16; i++) tc::mbar_init(&sh.pair_bar[i >> 2][i & 3], 1);
}
// a field of the unit `it`, read anew at every use
#define PREP_UNIT(field, it) (*const_cast<volatile int*>(&ctx.sh->unit[(it) & 3].field))

// Fused form: stores the ready flag of unit `it`.  Called by one warp, which meets the others behind the unit's last writes here; the
// release store is cumulative over them.  It waits until the CTA's stores are visible, 1,000 cycles: it is put off to a place in the next
// unit where its warp has nothing else to do, unless the worker has to wait for its ring slot.
constexpr int PUB_WARP = 7;
constexpr int FETCH_TID = 192;                            // works out the units and asks for q, k and v
__device__ __forceinline__ void prep_publish(const PrepCtx& ctx, int it, int* ready, int kr) {
  asm volatile("bar.sync %0, 256;" ::"r"(ctx.bar_id + 2) : "memory");
  if (ctx.tid == PUB_WARP * 32) {
    tc::bulk_wait_all<0>();                                // its copy of W, by this thread, is complete
    const int value = PREP_UNIT(value, it);
    st_release_gpu(ready + (size_t)PREP_UNIT(slot, it) * F_LINE + ((value - 1) & (kr - 1)), value);
  }
}

// Tensor maps of the inputs, tokens past the end read as zeros: qkv as [batch][token][3 H 128] bf16, box 64 tokens x 64 channels (v), and
// as [batch][32 channels of 3 H 128][token] with 64-byte rows, box 4 x 64 tokens (q and k: in 128-byte rows two of the eight tokens that a
// quarter-warp reads met in the same banks); g (or f) as [batch][token][H 128] f32, box 64 tokens x 32 channels.  128-byte swizzle for v and g.
__device__ __forceinline__ void prep_tma(uint8_t* dst, const CUtensorMap* map, int c, int t, int b, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(tc::smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c), "r"(t), "r"(b), "r"(tc::smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void prep_tma_rows(uint8_t* dst, const CUtensorMap* map, int c32, int t, int b, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(tc::smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(t), "r"(c32), "r"(b), "r"(tc::smem_u32(bar))
      : "memory");
}
// the next unit's inputs, each as soon as its place is free (one thread).  (q, k and v asked for in L2 earlier: 1,849 -> 1,861 us a layer.)
__device__ __forceinline__ void prep_fetch_g(const PrepCtx& ctx, int it, const CUtensorMap* map_g) {
  if (PREP_UNIT(n_valid, it) == 0) return;
  const int c = PREP_UNIT(head, it) * KD, t0 = PREP_UNIT(t0, it), b = PREP_UNIT(b, it);
  tc::mbar_arrive_expect_tx(&ctx.sh->g_bar, 4 * P1_BOX);
#pragma unroll
  for (int m = 0; m < 4; m++) prep_tma(ctx.smem + P1_X + m * P1_BOX, map_g, c + 32 * m, t0, b, &ctx.sh->g_bar);
}
__device__ __forceinline__ void prep_fetch_qkv(const PrepCtx& ctx, int it, const CUtensorMap* map_qkv, const CUtensorMap* map_qk, int H) {
  if (PREP_UNIT(n_valid, it) == 0) return;
  const int c = PREP_UNIT(head, it) * KD, t0 = PREP_UNIT(t0, it), b = PREP_UNIT(b, it);
  tc::mbar_arrive_expect_tx(&ctx.sh->qkv_bar, 6 * P1_BOX);
  prep_tma_rows(ctx.smem + P1_QK + 2 * P1_BOX, map_qk, (H * KD + c) / 32, t0, b, &ctx.sh->qkv_bar);
  prep_tma_rows(ctx.smem + P1_QK, map_qk, c / 32, t0, b, &ctx.sh->qkv_bar);
#pragma unroll
  for (int h = 0; h < 2; h++) prep_tma(ctx.smem + P1_V + h * P1_BOX, map_qkv, 2 * H * KD + c + 64 * h, t0, b, &ctx.sh->qkv_bar);
}

// Unit number `it` of a worker: (batch, head, chunk) of the preparation, into its place of `units`.
// GATED: `g` holds the raw gate projection f and `beta_in` the raw fp32 b; the kernel applies
//   g = lower_bound * sigmoid(exp(a_log[head]) * (f + dt_bias[head][channel])),  beta = bf16(sigmoid(b))
// itself (the arithmetic of the reference's separate gate kernel, src/engine/glue2.cu:347-360), so the
// fp32 gate tensor is never written to or read back from memory.
// The unit's inputs are on their way (prep_fetch_*); its end sends for those of the next.
// SLICES: chain CTAs of a slot in the fused form (SUB), 0 in the two-kernel form.  SUB: `ready` and `consumed` are the flags
// of the ring; on return the unit's last writes are on their way and its flag is still to be stored (prep_publish).
// `make_unit(it, desc)` works out a unit (one thread; two ahead, its divisions beside the inverse).
template <bool GATED, int SLICES, class MakeUnit>
__device__ __forceinline__ void prep_unit(
    const PrepCtx& ctx, const int it, const CUtensorMap* map_qkv, const CUtensorMap* map_qk, const CUtensorMap* map_g, const void* __restrict__ beta_in,
    uint8_t* __restrict__ units, int H, const float* __restrict__ dt_bias, const float* __restrict__ a_log, float lower_bound,
    const uint32_t tmem, int* ready, const int* consumed, int* g_abort, int kr, MakeUnit&& make_unit) {
  constexpr bool SUB = SLICES > 0;
  uint8_t* const smem = ctx.smem;
  uint8_t* const sK = smem + P1_K;
  float* const sX = reinterpret_cast<float*>(smem + P1_TAB);
  uint8_t* const sRI = smem + P1_RI;
  uint8_t* const sT = smem + P1_RI;
  float* const sN = reinterpret_cast<float*>(smem + P1_N);
  float* const sTab = reinterpret_cast<float*>(smem + P1_TAB);

  int tid = ctx.tid;
  asm volatile("" : "+r"(tid));                            // addresses are formed anew in every unit: hoisted out of the loop they would be spilled
  const int lane = tid & 31, warp = tid >> 5;
  const int g8 = lane >> 2, tig = lane & 3;
  const int I = warp >> 1;                                 // 16-token block of this warp
  const bool odd = warp & 1;
  const int t = 8 * warp + g8;                             // this lane's token
#define PREP_OUT (units + (size_t)PREP_UNIT(unit, it) * U_BYTES)

  // ---- stage 1: log-decay sums.  x_t = inclusive sum of the log decay (in units of log 2) INSIDE the 16-token block, in place.  Lane
  //      8 J + 4 b + p of warp w has channels 16 w + 4 p .. + 3 over tokens 8 b .. 8 b + 7 of block J, in the order 0-7 (b = 0) or
  //      4-7, 0-3: so the eight lanes of a block read and write all banks.  The block totals of a channel sit in eight lanes of one
  //      warp, which turn them into the tables, two channels each ----
  int seen = INT_MAX;                                      // publishing warp's first lanes: chunks that each CTA of the slot has consumed
  if (SUB && tid >= PUB_WARP * 32 && tid < PUB_WARP * 32 + SLICES)
    seen = ld_relaxed_gpu(consumed + (PREP_UNIT(slot, it) * SLICES + tid - PUB_WARP * 32) * F_LINE);
  float beta = 0.f;
  if (t < PREP_UNIT(n_valid, it)) {
    const size_t bi = (size_t)(PREP_UNIT(tok0, it) + t) * H + PREP_UNIT(head, it);
    if (GATED) beta = static_cast<const float*>(beta_in)[bi];
    else beta = __bfloat162float(static_cast<const __nv_bfloat16*>(beta_in)[bi]);
  }
  const int J = lane >> 3, half = (lane >> 2) & 1, g4 = 16 * warp + 4 * (lane & 3), gc = g4 + 2 * half;
  float2 dec;                                              // e^{G_last} of channels gc, gc + 1 (lanes with J = 3)
  {
    constexpr float LOG2E = 1.4426950408889634f;
    constexpr float FLOOR = -80.5f * LOG2E;                // keeps k^ e^{x} and k^ e^{-x} inside fp32's normal range (gates of -5: -80)
    float decay = 0.f;
    float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
    int n_valid = KC;
    if (GATED) {
      const int head = PREP_UNIT(head, it);
      n_valid = PREP_UNIT(n_valid, it);
      decay = __expf(__ldg(a_log + head));
      bias = __ldg(reinterpret_cast<const float4*>(dt_bias + (size_t)head * KD + g4));
    }
    uint8_t* const xb = smem + P1_X + (g4 >> 5) * P1_BOX + (16 * J + 8 * half) * 128;
    const int piece = (g4 >> 2) & 7, turn = 4 * half;      // slot i holds token i ^ turn of the half
    auto at = [&](int i) { return reinterpret_cast<float4*>(xb + (i ^ turn) * 128 + ((piece ^ i ^ turn) << 4)); };
    tc::mbar_wait(&ctx.sh->g_bar, it & 1, ctx.abort_flag, 12);
    float4 gr[8];
    auto load_gates = [&]() {
#pragma unroll
      for (int i = 0; i < 8; i++) gr[i] = *at(i);
      if (GATED) {
#pragma unroll
        for (int i = 0; i < 8; i++) {
          gr[i].x = lower_bound * (1.0f / (1.0f + __expf(-(decay * (gr[i].x + bias.x)))));
          gr[i].y = lower_bound * (1.0f / (1.0f + __expf(-(decay * (gr[i].y + bias.y)))));
          gr[i].z = lower_bound * (1.0f / (1.0f + __expf(-(decay * (gr[i].z + bias.z)))));
          gr[i].w = lower_bound * (1.0f / (1.0f + __expf(-(decay * (gr[i].w + bias.w)))));
        }
        if (n_valid < KC)                                  // the tokens past the end, whose f reads as zero, do not decay
#pragma unroll
          for (int i = 0; i < 8; i++)
            if (16 * J + 8 * half + (i ^ turn) >= n_valid) gr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      }
    };
    auto add4 = [](float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
    auto other = [&](float4 v) {                           // the same of the block's other half
      return make_float4(__shfl_xor_sync(0xffffffffu, v.x, 4), __shfl_xor_sync(0xffffffffu, v.y, 4), __shfl_xor_sync(0xffffffffu, v.z, 4),
                         __shfl_xor_sync(0xffffffffu, v.w, 4));
    };
    // gates -> sums inside slots 0-3 and inside slots 4-7
    auto run_sums = [&]() {
#pragma unroll
      for (int i = 0; i < 8; i++) {
        const float4 r = i & 3 ? gr[i - 1] : make_float4(0.f, 0.f, 0.f, 0.f);
        gr[i] = make_float4(fmaf(gr[i].x, LOG2E, r.x), fmaf(gr[i].y, LOG2E, r.y), fmaf(gr[i].z, LOG2E, r.z), fmaf(gr[i].w, LOG2E, r.w));
      }
    };
    load_gates();
    run_sums();
    float4 mine = add4(gr[3], gr[7]), theirs = other(mine), tot4 = add4(mine, theirs);
    if (__builtin_expect(__any_sync(0xffffffffu, fminf(fminf(tot4.x, tot4.y), fminf(tot4.z, tot4.w)) < FLOOR), 0)) {
      // Rare: a channel decays by more than e^-80 inside the block.  Sums that stop at a floor would take the tokens behind it as
      // not decaying at all, so the strongest of its gates are weakened instead: to e^-40, or to e^-20, e^-10 or e^-5, whichever is the
      // first that keeps the block's sum.
      load_gates();
      auto first_lo = [](float v) { return v < FLOOR ? -40.f : -INFINITY; };
      float4 lo = make_float4(first_lo(tot4.x), first_lo(tot4.y), first_lo(tot4.z), first_lo(tot4.w));
      auto at_least = [](float v, float l) { return v < l ? l : v; };   // (a NaN stays one)
      auto gate = [&](int i) {
        return make_float4(at_least(gr[i].x, lo.x), at_least(gr[i].y, lo.y), at_least(gr[i].z, lo.z), at_least(gr[i].w, lo.w));
      };
#pragma unroll 1
      for (int k = 0; k < 3; k++) {
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < 8; i++) sum = add4(sum, gate(i));
        sum = add4(sum, other(sum));
        if (sum.x < -80.f) lo.x *= 0.5f;
        if (sum.y < -80.f) lo.y *= 0.5f;
        if (sum.z < -80.f) lo.z *= 0.5f;
        if (sum.w < -80.f) lo.w *= 0.5f;
      }
#pragma unroll
      for (int i = 0; i < 8; i++) gr[i] = gate(i);
      run_sums();
      mine = add4(gr[3], gr[7]);
      theirs = other(mine);
      tot4 = add4(mine, theirs);
    }
    // what goes before the slots: the block's first half (b = 1), and this half's first four tokens, which are slots 4-7 where b = 1
    const float4 g3 = gr[3];
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float4 carry = i < 4 ? (half ? add4(theirs, gr[7]) : make_float4(0.f, 0.f, 0.f, 0.f)) : (half ? theirs : g3);
      *at(i) = add4(gr[i], carry);
    }
    const float2 tot = half ? make_float2(tot4.z, tot4.w) : make_float2(tot4.x, tot4.y);
    float2 before = make_float2(0.f, 0.f), after = make_float2(0.f, 0.f), next1 = before, next2 = before;
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const float qx = __shfl_sync(0xffffffffu, tot.x, 8 * q + (lane & 7)), qy = __shfl_sync(0xffffffffu, tot.y, 8 * q + (lane & 7));
      if (q < J) { before.x += qx; before.y += qy; }
      if (q > J) { after.x += qx; after.y += qy; }
      if (q == J + 1) next1 = make_float2(qx, qy);
      if (q == J + 2) next2 = make_float2(next1.x + qx, next1.y + qy);
    }
    auto put = [&](int r, float2 v) { *reinterpret_cast<float2*>(sTab + r * TAB_LD + gc) = make_float2(ex2_approx(v.x), ex2_approx(v.y)); };
    put(TAB_EP + J, before);
    // decay from a token to the end of ITS block is e^{tot - x} = e^{-x} e^{tot} (each factor within fp32 range for |x| <= 80.5),
    // the decay over the LATER blocks is e^{G_last - P_next} (may underflow: then Kt is 0)
    put(TAB_ETOT + J, tot);
    put(TAB_KE + J, after);
    if (J < 2) put(TAB_F + J, next1);                      // block pairs (2, 0), (3, 1)
    if (J == 0) put(TAB_F + 2, next2);                     // (3, 0)
    dec = make_float2(ex2_approx(before.x + tot.x), ex2_approx(before.y + tot.y));
  }
  if (GATED && t < PREP_UNIT(n_valid, it)) beta = __bfloat162float(__float2bfloat16(1.0f / (1.0f + __expf(-beta))));
  // q and k rows: piece 4 m + tig of a row (expanded when they are used)
  uint4 kraw[4], qraw[4];
  tc::mbar_wait(&ctx.sh->qkv_bar, it & 1, ctx.abort_flag, 13);
  float rk, rq;                                            // L2 normalisation of the rows
  {
    const uint8_t* qrow = smem + P1_QK + t * 64 + tig * 16;
#pragma unroll
    for (int m = 0; m < 4; m++) {
      qraw[m] = *reinterpret_cast<const uint4*>(qrow + m * 4096);
      kraw[m] = *reinterpret_cast<const uint4*>(qrow + 2 * P1_BOX + m * 4096);
    }
    float sk = 0.f, sq = 0.f;
#pragma unroll
    for (int m = 0; m < 4; m++) {
      const uint32_t kw[4] = {kraw[m].x, kraw[m].y, kraw[m].z, kraw[m].w}, qw[4] = {qraw[m].x, qraw[m].y, qraw[m].z, qraw[m].w};
#pragma unroll
      for (int e = 0; e < 4; e++) {
        sk = fmaf(bf16lo(kw[e]), bf16lo(kw[e]), fmaf(bf16hi(kw[e]), bf16hi(kw[e]), sk));
        sq = fmaf(bf16lo(qw[e]), bf16lo(qw[e]), fmaf(bf16hi(qw[e]), bf16hi(qw[e]), sq));
      }
    }
    sk += __shfl_xor_sync(0xffffffffu, sk, 1); sq += __shfl_xor_sync(0xffffffffu, sq, 1);
    sk += __shfl_xor_sync(0xffffffffu, sk, 2); sq += __shfl_xor_sync(0xffffffffu, sq, 2);
    rk = rsqrtf(sk + 1e-6f);
    rq = rsqrtf(sq + 1e-6f);
  }
  // fused form: the ring slot must have been drained before the first write to the unit (all of them follow)
  bool unpublished = SUB && it > 0;                        // the flag of the unit before this one
  if (SUB && it == 1 && warp == PUB_WARP) {                // the chains wait for a worker's first
    prep_publish(ctx, 0, ready, kr);
    unpublished = false;
  }
  if (SUB && warp == PUB_WARP) {
    const int want = PREP_UNIT(value, it) - kr;            // the slot held chunk value - 1 - kr
    if (__any_sync(0xffffffffu, seen < want)) {
      if (unpublished) prep_publish(ctx, it - 1, ready, kr);   // before a wait: the chains may need that unit to get on
      unpublished = false;
      if (lane < SLICES) poll_flag_ge(consumed + (PREP_UNIT(slot, it) * SLICES + lane) * F_LINE, want, ctx.abort_flag, g_abort, 20);
      __syncwarp();
    }
  }
  if (SUB && it > 0 && tid == PUB_WARP * 32) tc::bulk_wait_read<0>();   // the W of the unit before has left K+'s place
  prep_sync<SUB>(ctx);                                     // x and the tables are complete, q and k have been read

  // ---- stage 2: every operand that is a row of this warp's tokens times a decay, and the products of the warp's tokens with
  //      themselves and, odd warps, with the other eight of their block (TF32: e^{-x} needs the fp32 exponent range).  Left operands
  //      k^ e^{x}, q^ e^{x}; right operand R = beta k^ e^{-x}; R' = R e^{tot} <= 1 is moved on to the start of each later block (fp16,
  //      for the pairs of blocks) and to the end of the chunk (Kt) ----
  uint32_t ah[4][8];                                       // the left operands in fp16, both at most 1 in magnitude
  {
    uint8_t* const out = PREP_OUT;
    if (J == 3) *reinterpret_cast<float2*>(out + U_DEC + gc * 4) = dec;
    // tiles of B beta above the diagonal are never computed: zeros
    for (int i = lane; i < (7 - warp) * 8; i += 32)
      *reinterpret_cast<uint4*>(out + U_BB + warp * SBO_K64 + (warp + 1) * LBO + i * 16) = make_uint4(0, 0, 0, 0);
    float dg[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f};
    const float* tab = sTab + I * TAB_LD + 8 * tig;
    const uint64_t beta2 = pack2(beta, beta), rk2 = pack2(rk, rk), rq2 = pack2(rq, rq);
    uint8_t* ri = sRI + (t & 15) * 256;
    const int sw = (t & 1) << 2;                           // 16-byte pieces of odd rows are swapped in halves of 64 bytes: conflict-free reads
#pragma unroll
    for (int m = 0; m < 4; m++) {
      float4* const xp0 = reinterpret_cast<float4*>(smem + P1_X + m * P1_BOX + t * 128 + (((2 * tig) ^ g8) << 4));
      float4* const xp1 = reinterpret_cast<float4*>(smem + P1_X + m * P1_BOX + t * 128 + (((2 * tig + 1) ^ g8) << 4));
      const float4 x0 = *xp0, x1 = *xp1;
      const float xs[8] = {x0.x, x0.y, x0.z, x0.w, x1.x, x1.y, x1.z, x1.w};
      const uint32_t kw[4] = {kraw[m].x, kraw[m].y, kraw[m].z, kraw[m].w}, qw[4] = {qraw[m].x, qraw[m].y, qraw[m].z, qraw[m].w};
      uint64_t kl[4], ql[4], rb[4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        const uint64_t kn = mul2(pack2(bf16lo(kw[e]), bf16hi(kw[e])), rk2);
        const uint64_t up = pack2(ex2_approx(xs[2 * e]), ex2_approx(xs[2 * e + 1]));
        const uint64_t dn = pack2(ex2_approx(-xs[2 * e]), ex2_approx(-xs[2 * e + 1]));
        rb[e] = mul2(mul2(kn, beta2), dn);
        kl[e] = mul2(kn, up);
        ql[e] = mul2(mul2(pack2(bf16lo(qw[e]), bf16hi(qw[e])), rq2), up);
        ah[m][(e >> 1) * 4 + (e & 1) * 2] = pack_h2(kl[e]);
        ah[m][(e >> 1) * 4 + (e & 1) * 2 + 1] = pack_h2(ql[e]);
      }
      uint32_t rt[8], a[4][4];
#pragma unroll
      for (int e = 0; e < 4; e++) {
        float r0, r1, k0, k1, q0, q1;
        unpack2(rb[e], r0, r1);
        unpack2(kl[e], k0, k1);
        unpack2(ql[e], q0, q1);
        rt[2 * e] = f2tf32(r0);
        rt[2 * e + 1] = f2tf32(r1);
        a[e][0] = f2tf32(k0); a[e][1] = f2tf32(q0); a[e][2] = f2tf32(k1); a[e][3] = f2tf32(q1);
        mma_tf32(dg, a[e], rt[2 * e], rt[2 * e + 1]);
      }
      if (!odd) {                                          // for the odd warp of the block, in place of x
        *reinterpret_cast<uint4*>(xp0) = make_uint4(rt[0], rt[1], rt[2], rt[3]);
        *reinterpret_cast<uint4*>(xp1) = make_uint4(rt[4], rt[5], rt[6], rt[7]);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&ctx.sh->pair_bar[I][m]);
      } else {
        tc::mbar_wait(&ctx.sh->pair_bar[I][m], it & 1, ctx.abort_flag, 14);
        const uint4 r0 = *reinterpret_cast<const uint4*>(xp0 - 64), r1 = *reinterpret_cast<const uint4*>(xp1 - 64);   // eight rows up
        mma_tf32(sb, a[0], r0.x, r0.y);
        mma_tf32(sb, a[1], r0.z, r0.w);
        mma_tf32(sb, a[2], r1.x, r1.y);
        mma_tf32(sb, a[3], r1.z, r1.w);
      }
      uint64_t f[4], w[4];
      const int piece = 4 * m + tig;
      // K+ = k^ e^{G_t}: B operand; Q+ = q^ e^{G_t}: rows 64-127 of the unit's first tile (a chunk's first block: e^{x} is all of it)
      uint4 kp = make_uint4(ah[m][0], ah[m][2], ah[m][4], ah[m][6]), qp = make_uint4(ah[m][1], ah[m][3], ah[m][5], ah[m][7]);
      if (I > 0) {
        load_pairs(tab + TAB_EP * TAB_LD + 32 * m, f);
#pragma unroll
        for (int e = 0; e < 4; e++) w[e] = mul2(kl[e], f[e]);
        kp = pack_piece(w);
#pragma unroll
        for (int e = 0; e < 4; e++) w[e] = mul2(ql[e], f[e]);
        qp = pack_piece(w);
      }
      *reinterpret_cast<uint4*>(sK + piece * P1_PIECE + warp * 128 + g8 * 16) = kp;
      *reinterpret_cast<uint4*>(out + U_WQ + (8 + warp) * WQ_ROWS + m * ATOM + atom_off(g8, tig)) = qp;
      load_pairs(tab + TAB_ETOT * TAB_LD + 32 * m, f);
#pragma unroll
      for (int e = 0; e < 4; e++) rb[e] = mul2(rb[e], f[e]);
      const uint4 rp = pack_piece(rb);
      uint4 kt = rp;                                       // (the last block ends with the chunk)
      if (I < 3) {
        load_pairs(tab + TAB_KE * TAB_LD + 32 * m, f);
#pragma unroll
        for (int e = 0; e < 4; e++) w[e] = mul2(rb[e], f[e]);
        kt = pack_piece(w);
      }
      *reinterpret_cast<uint4*>(out + U_KT + m * KT_BLK + warp * ATOM + atom_off(g8, tig)) = kt;
      const int po = (piece ^ sw) << 4;
      if (I < 3) *reinterpret_cast<uint4*>(ri + ((I + 1) * I / 2 + I) * 4096 + po) = rp;
      if (I < 2) {
        load_pairs(sTab + (TAB_F + I) * TAB_LD + 8 * tig + 32 * m, f);
#pragma unroll
        for (int e = 0; e < 4; e++) w[e] = mul2(rb[e], f[e]);
        *reinterpret_cast<uint4*>(ri + ((I + 2) * (I + 1) / 2 + I) * 4096 + po) = pack_piece(w);
      }
      if (I < 1) {
        load_pairs(sTab + (TAB_F + 2) * TAB_LD + 8 * tig + 32 * m, f);
#pragma unroll
        for (int e = 0; e < 4; e++) w[e] = mul2(rb[e], f[e]);
        *reinterpret_cast<uint4*>(ri + 3 * 4096 + po) = pack_piece(w);
      }
    }
    // accumulator of a tile: N row t, columns s0, s0 + 1 (s0 = 8 * tile + 2 tig), then the same of B beta
    float* nrow = sN + prep_n_row(t) + 2 * tig;
    uint8_t* bbrow = out + U_BB + warp * SBO_K64 + g8 * 16 + tig * 4;
    const int s = 2 * tig;                                 // N strictly lower, B lower including the diagonal
    *reinterpret_cast<float2*>(nrow + 8 * warp) = make_float2(s < g8 ? dg[0] : 0.f, s + 1 < g8 ? dg[1] : 0.f);
    *reinterpret_cast<uint32_t*>(bbrow + warp * LBO) = pack_h2(s <= g8 ? dg[2] : 0.f, s + 1 <= g8 ? dg[3] : 0.f);
    if (odd) {
      *reinterpret_cast<float2*>(nrow + 8 * (warp - 1)) = make_float2(sb[0], sb[1]);
      *reinterpret_cast<uint32_t*>(bbrow + (warp - 1) * LBO) = pack_h2(sb[2], sb[3]);
    }
  }
  tc::fence_async_smem();
  prep_sync<SUB>(ctx);                                     // right operands and the diagonal blocks of N are complete

  // ---- stage 3: the products with earlier blocks (fp16), 2 I tiles a warp; the warps of the first block, which have none, invert the
  //      16 x 16 diagonal blocks of I + N, those of the second convert v as well ----
  if (tid == 0) prep_fetch_g(ctx, it + 1, map_g);          // x is free
  __syncwarp();
  {
    float* nrow = sN + prep_n_row(t) + 2 * tig;
    uint8_t* bbrow = PREP_OUT + U_BB + warp * SBO_K64 + g8 * 16 + tig * 4;
    const uint8_t* rbase = sRI + (I * (I - 1) / 2) * 4096 + g8 * 256;
    const int sw = (g8 & 1) << 2;
#pragma unroll 1
    for (int jb = 0; jb < I; jb++) {
      float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int m = 0; m < 4; m++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
          const uint4 r = *reinterpret_cast<const uint4*>(rbase + jb * 4096 + h * 2048 + (((4 * m + tig) ^ sw) << 4));
          mma_f16_16816(acc[h], ah[m][0], ah[m][1], ah[m][2], ah[m][3], r.x, r.y);
          mma_f16_16816(acc[h], ah[m][4], ah[m][5], ah[m][6], ah[m][7], r.z, r.w);
        }
#pragma unroll
      for (int h = 0; h < 2; h++) {
        *reinterpret_cast<float2*>(nrow + 16 * jb + 8 * h) = make_float2(acc[h][0], acc[h][1]);
        *reinterpret_cast<uint32_t*>(bbrow + (2 * jb + h) * LBO) = pack_h2(acc[h][2], acc[h][3]);
      }
    }
  }
  if (I == 0) {
    // inverse of a unit lower triangular 16 x 16 block, lane = column of one of two blocks: x_r = delta - sum_{s<r} N[r][s] x_s
    const int blk = 2 * warp + (lane >> 4), col = lane & 15;
    float x[16];
    const float* nd = sN + prep_n_row(16 * blk) + 16 * blk;
    const int ld = warp == 0 ? 36 : 68;
#pragma unroll
    for (int r = 0; r < 16; r++) {
      float a0 = (r == col) ? 1.f : 0.f, a1 = 0.f;
#pragma unroll
      for (int s = 0; s < r; s += 4) {
        const float4 n4 = *reinterpret_cast<const float4*>(nd + r * ld + s);
        const float nn[4] = {n4.x, n4.y, n4.z, n4.w};
#pragma unroll
        for (int u = 0; u < 4; u++) {
          if (s + u >= r) break;
          if (u & 1) a1 = fmaf(-nn[u], x[s + u], a1);
          else a0 = fmaf(-nn[u], x[s + u], a0);
        }
      }
      x[r] = a0 + a1;
    }
    float* xi = sX + prep_inv_at(blk) + col;
#pragma unroll
    for (int r = 0; r < 16; r++) xi[r * P1_LDX] = x[r];
  } else if (I == 1) {
    // bf16 -> fp16 in place.  (The product T V needs both operands in ONE 16-bit format: a kind::f16 product of an fp16 T with bf16
    // rows is rejected by the hardware as an illegal instruction.)
#pragma unroll
    for (int j = 0; j < 16; j++) {
      uint4* vp = reinterpret_cast<uint4*>(smem + P1_V) + tid - 64 + 64 * j;
      const uint4 vr = *vp;
      *vp = make_uint4(pack_h2(bf16lo(vr.x), bf16hi(vr.x)), pack_h2(bf16lo(vr.y), bf16hi(vr.y)), pack_h2(bf16lo(vr.z), bf16hi(vr.z)),
                       pack_h2(bf16lo(vr.w), bf16hi(vr.w)));
    }
  }
  prep_sync<SUB>(ctx);                                     // N and the diagonal inverses are complete, the right operands have been read

  // ---- stage 4: X = (I + N)^-1 below its diagonal blocks, and its fp16 copy T as the K-major A operand (K = 64).  First
  //      P_mj = N_mj X_jj in place of N_mj, one warp per block, while two warps write the diagonal of T and the zeros above it;
  //      then the blocks of X, while a warp publishes the unit before and one works out the unit after the next ----
  if (warp < 6) {
    const int m = warp < 1 ? 1 : (warp < 3 ? 2 : 3), j = warp - (m * (m - 1)) / 2, ld = m < 2 ? 36 : 68;
    float* nb = sN + prep_n_row(16 * m) + 16 * j;
    Frag16 L;
    L.load(nb, ld, lane);
    float acc[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
    block16_mma(L, sX + prep_inv_at(j), P1_LDX, acc, lane);
    __syncwarp();
#pragma unroll
    for (int nt = 0; nt < 2; nt++) {
      *reinterpret_cast<float2*>(nb + g8 * ld + 8 * nt + 2 * tig) = make_float2(acc[nt][0], acc[nt][1]);
      *reinterpret_cast<float2*>(nb + (g8 + 8) * ld + 8 * nt + 2 * tig) = make_float2(acc[nt][2], acc[nt][3]);
    }
  } else {
    const int e = tid - 192;
#pragma unroll
    for (int q = 0; q < 2; q++) {                          // 4 blocks x 16 rows x 2 pieces
      const int i = e + 64 * q, blk = i >> 5, r = (i & 7) + ((i >> 4) & 1) * 8, h = (i >> 3) & 1;
      const float* xi = sX + prep_inv_at(blk) + r * P1_LDX + 8 * h;
      const float4 v0 = *reinterpret_cast<const float4*>(xi), v1 = *reinterpret_cast<const float4*>(xi + 4);
      *reinterpret_cast<uint4*>(sT + (2 * blk + (r >> 3)) * SBO_K64 + (2 * blk + h) * LBO + (r & 7) * 16) =
          make_uint4(pack_h2(v0.x, v0.y), pack_h2(v0.z, v0.w), pack_h2(v1.x, v1.y), pack_h2(v1.z, v1.w));
    }
#pragma unroll
    for (int q = 0; q < 3; q++) {                          // 6 blocks x 16 rows x 2 pieces
      const int i = e + 64 * q, blk = i >> 5, zi = blk < 3 ? 0 : (blk < 5 ? 1 : 2), zj = blk < 3 ? blk + 1 : (blk < 5 ? blk - 1 : 3);
      *reinterpret_cast<uint4*>(sT + (2 * zi + ((i >> 4) & 1)) * SBO_K64 + (2 * zj + ((i >> 3) & 1)) * LBO + (i & 7) * 16) = make_uint4(0, 0, 0, 0);
    }
  }
  prep_sync<SUB>(ctx);
  if (!SUB) {
    if (warp < 6) prep_inverse_blocks(sN, sX, sT, warp, lane, ctx.bar_id + 4);
  } else if (warp == 1) prep_inverse_row<1>(sN, sX, sT, lane);
  else if (warp == 2) prep_inverse_row<2>(sN, sX, sT, lane);
  else if (warp == 3) prep_inverse_row<3>(sN, sX, sT, lane);
  else if (SUB && warp == PUB_WARP && unpublished) prep_publish(ctx, it - 1, ready, kr);
  else if (SUB && tid == FETCH_TID) make_unit(it + 2, ctx.sh->unit[(it + 2) & 3]);
  tc::fence_async_smem();
  tc::fence_before_sync();
  prep_sync<SUB>(ctx);
  tc::fence_after_sync();

  // ---- stage 5: W = T K+, Uloc = T V: tcgen05 weight-stationary M64 N128 K64, fp16 in, fp32 TMEM accumulators: columns 0-63 of the 64
  //      tokens in lanes 0-63, columns 64-127 in lanes 64-127, so that all eight warps read them ----
  if (tid == 0) {
    const uint32_t idesc = tc::make_idesc(64, KD, tc::FMT_F16, tc::FMT_F16, false, true);
    const uint32_t a_addr = tc::smem_u32(sT), k_addr = tc::smem_u32(sK);
    const uint64_t vd = tc::make_sdesc_sw128(tc::smem_u32(smem + P1_V), P1_BOX, 1024);
#pragma unroll
    for (int kk = 0; kk < KC / 16; kk++)
      tc::mma_ws_f16_if(1, tmem, tc::make_sdesc(a_addr + kk * 2 * LBO, LBO, SBO_K64), tc::make_sdesc(k_addr + kk * 2 * 128, 128, P1_PIECE), idesc, kk > 0);
#pragma unroll
    for (int kk = 0; kk < KC / 16; kk++)
      tc::mma_ws_f16_if(1, tmem + 64, tc::make_sdesc(a_addr + kk * 2 * LBO, LBO, SBO_K64), tc::sdesc_advance(vd, kk * 2048), idesc, kk > 0);
    tc::mma_commit(&ctx.sh->mma_bar);
  }
  const bool ok = __all_sync(0xffffffffu, tc::mbar_wait(&ctx.sh->mma_bar, it & 1, ctx.abort_flag, 1)) != 0;
  if (tid == FETCH_TID) prep_fetch_qkv(ctx, it + 1, map_qkv, map_qk, H);  // T, N, K+ and V are free
  __syncwarp();
  tc::fence_after_sync();
  // ---- stage 6: the accumulators leave: warps 0-3 take W, warps 4-7 Uloc, a token and 64 columns each thread.  A warp's piece of Uloc
  //      is 512 contiguous bytes; of W it would be 32 halves of 32-byte sectors, so W is put together where K+ was and copied out ----
  if (ok) {
    uint8_t* const out = PREP_OUT;
    const int et = (warp & 1) * 32 + lane, c0 = (warp & 2) * 32;
    const uint32_t acc = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (warp >> 2) * 64;
    auto piece = [](const uint32_t* r, uint32_t sign) {
      return make_uint4(pack_h2(__uint_as_float(r[0]), __uint_as_float(r[1])) ^ sign, pack_h2(__uint_as_float(r[2]), __uint_as_float(r[3])) ^ sign,
                        pack_h2(__uint_as_float(r[4]), __uint_as_float(r[5])) ^ sign, pack_h2(__uint_as_float(r[6]), __uint_as_float(r[7])) ^ sign);
    };
#pragma unroll
    for (int h = 0; h < 2; h++) {
      uint32_t r[32];
      tc::tmem_ld32(acc + 32 * h, r);
      tc::tmem_ld_wait();
      if (warp < 4) {                                      // stored negated
        uint8_t* const dst = sK + (et >> 3) * WQ_ROWS + ((c0 >> 5) + h) * ATOM;
#pragma unroll
        for (int u = 0; u < 4; u++) *reinterpret_cast<uint4*>(dst + atom_off(et, u)) = piece(r + 8 * u, 0x80008000u);
      } else {
        uint8_t* const dst = out + U_UL + (et ^ 8) * 16 + ((c0 >> 3) + 4 * h) * 1024;
#pragma unroll
        for (int u = 0; u < 4; u++) *reinterpret_cast<uint4*>(dst + u * 1024) = piece(r + 8 * u, 0u);
      }
    }
  }
  // (the warps meet whatever their waits said: behind one that gave up, the warps of this worker need not agree)
  if (warp < 4) {
    tc::fence_async_smem();
    asm volatile("bar.arrive %0, 160;" ::"r"(ctx.bar_id + 4) : "memory");
  } else if (warp == PUB_WARP) {
    asm volatile("bar.sync %0, 160;" ::"r"(ctx.bar_id + 4) : "memory");
    if (ok && tid == PUB_WARP * 32) {
      tc::bulk_s2g(PREP_OUT + U_WQ, sK, 8 * WQ_ROWS);
      tc::bulk_commit();
    }
  }
  tc::fence_before_sync();
  if (SUB && warp != PUB_WARP) asm volatile("bar.arrive %0, 256;" ::"r"(ctx.bar_id + 2) : "memory");
}

template <bool GATED>
__global__ __launch_bounds__(256, 2) void kda_chunk_prep_kernel(
    const __grid_constant__ CUtensorMap map_qkv, const __grid_constant__ CUtensorMap map_qk, const __grid_constant__ CUtensorMap map_g, const void* __restrict__ beta_in,
    uint8_t* __restrict__ ws, int seqlen, int H, int n_chunks, int* __restrict__ status,
    const float* __restrict__ dt_bias, const float* __restrict__ a_log, float lower_bound) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ PrepShared sh;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x;
  // heads are the fastest grid dimension: CTAs that run together read the same tokens, i.e. whole contiguous rows of the
  // activations.  Units are chunk-major: the CTAs that run together (same chunks, all heads) touch adjacent units, in
  // this kernel and in the scan, so their traffic spreads over all memory channels.
  PrepCtx ctx;
  ctx.smem = smem + ((1024u - (tc::smem_u32(smem) & 1023u)) & 1023u);
  ctx.sh = &sh; ctx.abort_flag = &abort_flag; ctx.tid = tid; ctx.bar_id = 0;
  if (tid == 0) {
    prep_init(sh);
    tc::mbar_fence_init();
    abort_flag = 0;
    PrepDesc& u = sh.unit[0];
    u.b = blockIdx.z;
    u.t0 = blockIdx.y * KC;
    u.tok0 = u.b * seqlen + u.t0;
    u.n_valid = min(KC, seqlen - u.t0);
    u.head = blockIdx.x;
    u.unit = (u.b * n_chunks + (int)blockIdx.y) * H + u.head;
    sh.unit[1].n_valid = 0;                                // a CTA has one unit
    pdl_wait();
    prep_fetch_g(ctx, 0, &map_g);
    prep_fetch_qkv(ctx, 0, &map_qkv, &map_qk, H);
  }
  if (tid < 32) tc::tmem_alloc(&tmem_slot, 128);
  pdl_wait();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  prep_unit<GATED, 0>(ctx, 0, &map_qkv, &map_qk, &map_g, beta_in, ws, H, dt_bias, a_log, lower_bound, tmem_slot, nullptr, nullptr, nullptr, 0,
                      [](int, PrepDesc&) {});
  if (tid == PUB_WARP * 32) tc::bulk_wait_all<0>();
  __syncthreads();
  if (tid < 32) tc::tmem_dealloc(tmem_slot, 128);
  if (tid == 0 && abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
}

// =================================================================================================
// The scan: one CTA of 512 threads walks the chunks of a chain in order, with NV of the head's 128 value columns (whose states, U and
// outputs do not depend on the other columns').  Shared by kernel 2 (units in a workspace) and the fused launch (units in a ring).
//
// Sixteen warps = four TMEM lane quarters (lq) x four groups, joined by mbarriers that complete once per chunk, never by the
// whole CTA; what is on the chunk-to-chunk chain is spread over many warps, the rest has warps of its own:
//   U         lq 0, 1 of all groups (token rows of D1), NV / 4 columns each
//   state     groups 0, 1: a k row and NV / 2 of its columns per thread, fp32 in registers
//   outputs   warps 10, 11: a token row each thread
//   issuer    warp 14: every product; it waits for operands only
//   producer  warp 15: ring protocol and operand copies
// A barrier's next phase cannot complete before its waiters have seen this one: U needs every U warp, the state operand every
// state warp; out_bar and d1_bar alternate by chunk, since the output warps may be a chunk behind or done with the one before.
//
// What bounds it: the products and hand-overs of a chunk in turn.  In cycles, NV = 128: state -> U 900 (eight products of 65, 350 until
// they are seen), U 500, Kt^T U 540, state 650, operand -> issuer 100: 2.7 thousand (2.1 with NV = 64, products of 49).  The form before, whose
// warps met at block barriers and emitted outputs in between, took 4.1 to 5.4.
// =================================================================================================
// fp16 A operand [I ; 0] (128 rows, K = 64) without storing it: its core matrix (i, j) depends on i - j only, so 23 core
// matrices, one of them the identity, serve all of them with 128 bytes as both strides.  The two core matrices of a K16 step then
// come in falling j, which is why Uloc keeps its 8-token blocks in swapped pairs.
constexpr uint32_t ID_BYTES = 23 * 128;
__device__ __forceinline__ void write_identity(uint8_t* dst, int tid, int nthreads) {
  for (int i = tid; i < (int)ID_BYTES / 16; i += nthreads) {
    const int r = i & 7;                                    // core matrix 7 is the identity, the others are zeros
    const uint32_t one = (i >> 3) == 7 ? 0x3C00u << (16 * (r & 1)) : 0u;
    reinterpret_cast<uint4*>(dst)[i] = make_uint4(r >> 1 == 0 ? one : 0u, r >> 1 == 1 ? one : 0u, r >> 1 == 2 ? one : 0u, r >> 1 == 3 ? one : 0u);
  }
}

// shared memory of a chain CTA: two operand stages (a unit with NV columns of Uloc), then the operands it makes itself
template <int NV>
struct Chain {
  static constexpr int SLICES = KD / NV;
  static constexpr uint32_t UL = U_UL, BB = UL + NV * 128, KT = BB + 8192, DEC = KT + 16384, STAGE = DEC + 512;
  static constexpr uint32_t S = 2 * STAGE;                  // fp16 B operand: state [128 k][NV], MN-major
  static constexpr uint32_t U = S + NV * 256;               // fp16 B operand: U [64 tokens][NV], MN-major
  static constexpr uint32_t O = U + NV * 128;               // bf16 output rows of one chunk: swizzled boxes of 64 tokens x 64 channels
  static constexpr uint32_t ID = O + NV * 128;              // [I ; 0]
  static constexpr uint32_t SMEM = ID + ID_BYTES + 1024;    // + slack to start the tiles at a 1 KB boundary
  static_assert(O % 1024 == 0 && STAGE % ATOM == 0 && KT % ATOM == 0 && BB >= 8192, "layout");
};
struct ChainBars {                  // two of most kinds by chunk parity, so that a warp that is held up may be a chunk behind
  uint64_t wu[2];                   // -W, Q+ and Uloc of a stage have landed
  uint64_t kb[2];                   // B beta, Kt^T and the decays
  uint64_t mma[2];                  // U and Q+ S0 are complete
  uint64_t mma2;                    // Kt^T U (state path) is complete
  uint64_t out[2];                  // (B beta) U is complete, and with it every product of the chunk
  uint64_t u;                       // the 256 token-row threads have written U
  uint64_t s[2];                    // the 256 state threads have written the state operand
  uint64_t d1[2];                   // the two output warps have read this half of D1
};
__device__ __forceinline__ void chain_init(ChainBars& bars) {   // one thread
  for (int i = 0; i < 2; i++) {
    tc::mbar_init(&bars.wu[i], 1);
    tc::mbar_init(&bars.kb[i], 1);
    tc::mbar_init(&bars.mma[i], 1);
    tc::mbar_init(&bars.out[i], 1);
    tc::mbar_init(&bars.s[i], 256);
    tc::mbar_init(&bars.d1[i], 2);
  }
  tc::mbar_init(&bars.mma2, 1);
  tc::mbar_init(&bars.u, 256);
}
// Chains job0, job0 + job_step, ... of n_chunks chunks each, n_virtual chunks in all; a job is (batch, head).  Chunk numbers run through
// all of them (`v`), and ring, flags and barrier parities go by v.  FLAGS (fused form, ring of kr units): `my_ready` and `my_consumed` are the slot's flags.
// `unit_of(v)`: the unit of a chunk.
template <int NV, bool FLAGS, class UnitOf>
__device__ __forceinline__ void chain_cta(uint8_t* smem, ChainBars& bars, const uint32_t tmem, int* abort_flag, UnitOf&& unit_of, const int* my_ready,
                                          int* my_consumed, int* g_abort, int kr, int job0, int job_step, int n_chunks, int n_virtual, int slice, int H,
                                          int seqlen, float* __restrict__ state, float* __restrict__ out_f32, const int* __restrict__ slots,
                                          float scale, const CUtensorMap* map_out) {
  using C = Chain<NV>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lq = warp & 3, grp = warp >> 2;
  const int rowi = lq * 32 + lane;                        // k row of the state / token row of U / output row + 64
  const int role = tc::warp_index_uniform();
  // D1 alternates between columns 0 .. NV - 1 and NV .. 2 NV - 1 by chunk parity, D2 follows
  write_identity(smem + C::ID, tid, 512);
  tc::fence_async_smem();
  __syncthreads();

  if (role == 14) {
    const uint32_t leader = tc::elect_one();
    const uint32_t idesc = tc::make_idesc(128, NV, tc::FMT_F16, tc::FMT_F16, false, true);
    const uint32_t idesc_kt = tc::make_idesc(128, NV, tc::FMT_F16, tc::FMT_F16, true, true);   // Kt^T: channels contiguous
    const uint32_t s_addr = tc::smem_u32(smem + C::S), u_addr = tc::smem_u32(smem + C::U), id_addr = tc::smem_u32(smem + C::ID);
    // D1 of chunk w = [I ; 0] Uloc, ahead of the state: the product with the identity is exact
    auto issue_uloc = [&](int w) {
      tc::fence_after_sync();
#pragma unroll
      for (int kk = 0; kk < KC / 16; kk++) {
        const uint64_t ad = tc::make_sdesc(id_addr + (6 - 2 * kk) * 128, 128, 128);
        const uint64_t bd = tc::make_sdesc(tc::smem_u32(smem + (w & 1) * C::STAGE) + C::UL + kk * 2 * 128, 128, 1024);
        tc::mma_f16_if(leader, tmem + (w & 1) * NV, ad, bd, idesc, kk > 0);
      }
    };
    int uloc = 0;                                          // chunks whose Uloc has been issued
    for (int v = 0; v < n_virtual; v++) {
      const uint32_t par = v & 1, ph = (v >> 1) & 1, stg_addr = tc::smem_u32(smem + par * C::STAGE);
      const uint32_t d1 = tmem + par * NV, d2 = tmem + 2 * NV;
      if (uloc == v) {
        tc::mbar_wait(&bars.wu[par], ph, abort_flag, 2);
        if (v >= 2) tc::mbar_wait(&bars.d1[par], ph ^ 1, abort_flag, 8);   // the output rows of chunk v - 2 have left this half of D1
        issue_uloc(v);
        uloc++;
      }
      // ---- D1 += [-W ; Q+] S0 ----
      tc::mbar_wait(&bars.s[par], ph, abort_flag, 6);
      tc::fence_after_sync();
#pragma unroll
      for (int kk = 0; kk < KD / 16; kk++) {
        const uint64_t ad = tc::make_sdesc_sw64(stg_addr + U_WQ + (kk >> 1) * ATOM + (kk & 1) * 32, 16, WQ_ROWS);
        const uint64_t bd = tc::make_sdesc(s_addr + kk * 2 * 128, 128, 2048);
        tc::mma_f16_if(leader, d1, ad, bd, idesc, true);
      }
      tc::mma_commit_if(leader, &bars.mma[par]);
      // the next chunk's Uloc while U leaves the tensor memory, if its operands and its half of D1 are there already (otherwise at
      // the chunk's start, where 260 cycles of products stand between the state and U)
      if (v + 1 < n_virtual) {
        const uint32_t nph = ((v + 1) >> 1) & 1;
        const bool here = tc::mbar_test_wait(&bars.wu[par ^ 1], nph) && (v == 0 || tc::mbar_test_wait(&bars.d1[par ^ 1], nph ^ 1));
        if (__all_sync(0xffffffffu, here)) {
          issue_uloc(v + 1);
          uloc++;
        }
      }
      // ---- D2 = Kt^T U (state path), then D1 rows 64-127 += (B beta) U (outputs) ----
      tc::mbar_wait(&bars.kb[par], ph, abort_flag, 11);
      tc::mbar_wait(&bars.u, par, abort_flag, 7);
      tc::fence_after_sync();
#pragma unroll
      for (int kk = 0; kk < KC / 16; kk++) {
        const uint64_t ad = tc::make_sdesc_sw64(stg_addr + C::KT + kk * 2 * ATOM, KT_BLK, ATOM);
        const uint64_t bd = tc::make_sdesc(u_addr + kk * 2 * 128, 128, 1024);
        tc::mma_f16_if(leader, d2, ad, bd, idesc_kt, kk > 0);
      }
      tc::mma_commit_if(leader, &bars.mma2);
      // rows 0-63 of this operand are whatever lies below B beta in the stage: they add to U's rows, which have been read
#pragma unroll
      for (int kk = 0; kk < KC / 16; kk++) {
        const uint64_t ad = tc::make_sdesc(stg_addr + C::BB - 8192 + kk * 2 * LBO, LBO, SBO_K64);
        const uint64_t bd = tc::make_sdesc(u_addr + kk * 2 * 128, 128, 1024);
        tc::mma_f16_if(leader, d1, ad, bd, idesc, true);
      }
      tc::mma_commit_if(leader, &bars.out[par]);
    }
  } else if (role == 15) {
    // a unit in two parts: a stage's first part is free as soon as the chunk's first product is complete, most of a chunk before
    // the rest.  74 KB take about as long as a chunk to arrive.
    auto load_wu = [&](int v) {
      if (lane == 0) {
        uint8_t* stg = smem + (v & 1) * C::STAGE;
        const uint8_t* u = unit_of(v);
        tc::mbar_arrive_expect_tx(&bars.wu[v & 1], C::BB);
        tc::bulk_g2s(stg, u, NV == KD ? C::BB : C::UL, &bars.wu[v & 1]);
        if (NV < KD) tc::bulk_g2s(stg + C::UL, u + U_UL + slice * (NV * 128), NV * 128, &bars.wu[v & 1]);
      }
      __syncwarp();
    };
    auto load_kb = [&](int v) {
      if (lane == 0) {
        tc::mbar_arrive_expect_tx(&bars.kb[v & 1], C::STAGE - C::BB);
        tc::bulk_g2s(smem + (v & 1) * C::STAGE + C::BB, unit_of(v) + U_BB, C::STAGE - C::BB, &bars.kb[v & 1]);
      }
      __syncwarp();
    };
    // Units are asked for a ring at a time: a flag takes a microsecond or more to read while the workers poll theirs, too long for
    // every chunk.
    int known = 0;                                         // units before this one are complete
    auto await_unit = [&](int v) {
      if (!FLAGS) return;
      const long long t0 = clock64();
      while (known <= v) {
        const bool here = lane < kr && ld_acquire_gpu(my_ready + ((known + lane) & (kr - 1))) > known + lane;
        const uint32_t missing = ~__ballot_sync(0xffffffffu, here);
        known += missing ? __ffs(missing) - 1 : 32;
        if (known > v) break;
        const bool give_up = *(volatile int*)abort_flag || ld_relaxed_gpu(g_abort) != 0 || clock64() - t0 > tc::MBAR_WAIT_CYCLES;
        if (__any_sync(0xffffffffu, give_up)) {
          if (lane == 0) {
            *(volatile int*)abort_flag = 21;
            atomicExch(g_abort, 21);
          }
          break;
        }
        __nanosleep(64);
      }
      __syncwarp();
      if (lane == 0) fence_proxy_async_all();
    };
    for (int v = 0; v < 2 && v < n_virtual; v++) {
      await_unit(v);
      load_wu(v);
      load_kb(v);
    }
    for (int v = 0; v < n_virtual; v++) {
      const uint32_t par = v & 1, ph = (v >> 1) & 1;
      // the unit of this chunk has landed in shared memory: its slot may be rewritten.  A relaxed store is enough:
      // the copy engine's reads are complete, nothing this thread wrote is handed over with the flag.
      tc::mbar_wait(&bars.wu[par], ph, abort_flag, 2);
      tc::mbar_wait(&bars.kb[par], ph, abort_flag, 2);
      if (FLAGS && lane == 0) st_relaxed_gpu(my_consumed, v + 1);
      if (v + 2 >= n_virtual) continue;
      await_unit(v + 2);
      tc::mbar_wait(&bars.mma[par], ph, abort_flag, 3);
      load_wu(v + 2);
      // all products of the chunk are complete and the state warps have read its decays
      tc::mbar_wait(&bars.out[par], ph, abort_flag, 5);
      tc::mbar_wait(&bars.s[par ^ 1], ((v + 1) >> 1) & 1, abort_flag, 9);
      load_kb(v + 2);
    }
  } else if (role == 10 || role == 11) {
    // Output rows: TMEM lanes 64-127 of a chunk's D1 half = tokens; a thread holds the columns of one token.  Stored directly,
    // a warp-wide 16-byte store would touch 32 different rows (32 L1 requests per instruction, over a thousand per chunk
    // on this one SM).  The bf16 rows are therefore assembled in shared memory and leave as tiled TMA stores (64 tokens x 64 channels
    // each, 128-byte-swizzle boxes; rows past the end of the sequence are clipped by the copy engine): the tile is written
    // conflict-free (16-byte piece p of row r at p ^ (r % 8)) and one thread hands it over.
    const int trow = rowi - 64;
    const bool issuer = role == 10 && lane == 0;
    bool valid = true;
    int c = 0, job = job0;                                 // chunk of the chain, chain
    for (int v = 0; v < n_virtual; v++) {
      const int b = job / H, head = job % H;
      const bool ok = tc::mbar_wait(&bars.out[v & 1], (v >> 1) & 1, abort_flag, 10);
      valid = valid && ok;
      tc::fence_after_sync();
      if (issuer) tc::bulk_wait_read<0>();                 // the previous chunk's tile has been read by the copy engine
      asm volatile("bar.sync 1, 64;" ::: "memory");
      const int tok = c * KC + trow;
#pragma unroll
      for (int q = 0; q < NV / 32; q++) {
        uint32_t r[32];
        tc::tmem_ld32(tmem + (v & 1) * NV + (uint32_t)(q * 32) + ((uint32_t)(lq * 32) << 16), r);
        tc::tmem_ld_wait();
#pragma unroll
        for (int u = 0; u < 4; u++) {
          uint32_t w[4];
#pragma unroll
          for (int e = 0; e < 4; e++) w[e] = pack_bf2_rz(__uint_as_float(r[8 * u + 2 * e]) * scale, __uint_as_float(r[8 * u + 2 * e + 1]) * scale);
          const int p = q * 4 + u;
          *reinterpret_cast<uint4*>(smem + C::O + (p >> 3) * 8192 + trow * 128 + (((p & 7) ^ (trow & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        if (out_f32 && tok < seqlen && valid) {
          float4* of = reinterpret_cast<float4*>(out_f32 + (((size_t)b * seqlen + tok) * H + head) * KD + slice * NV + q * 32);
#pragma unroll
          for (int u = 0; u < 8; u++)
            of[u] = make_float4(__uint_as_float(r[4 * u]) * scale, __uint_as_float(r[4 * u + 1]) * scale,
                                __uint_as_float(r[4 * u + 2]) * scale, __uint_as_float(r[4 * u + 3]) * scale);
        }
      }
      tc::fence_before_sync();
      if (lane == 0) tc::mbar_arrive(&bars.d1[v & 1]);     // chunk v + 2 may have this half of D1
      tc::fence_async_smem();
      asm volatile("bar.sync 1, 64;" ::: "memory");
      if (issuer && valid) {
#pragma unroll
        for (int hb = 0; hb < NV / 64; hb++)
          asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%1, %2, %3, %4}], [%5];" ::"l"(map_out),
                       "r"(slice * NV + hb * 64), "r"(head), "r"(c * KC), "r"(b), "r"(tc::smem_u32(smem + C::O + hb * 8192))
                       : "memory");
        tc::bulk_commit();
      }
      if (++c == n_chunks) { c = 0; job += job_step; }
    }
    if (issuer) tc::bulk_wait_all<0>();
  } else {
    constexpr int SC = NV / 2, UC = NV / 4;                // columns of a state thread, of a U thread
    const bool state_warp = grp < 2, u_warp = lq < 2;
    // chain number `ci`: its state row for this thread
    auto chain_state = [&](int ci) -> float* {
      const int job = job0 + job_step * ci, jb = job / H, jh = job % H;
      const int sl = slots ? slots[jb] : jb;
      return state + ((size_t)sl * H + jh) * KD * KD + (size_t)rowi * KD + slice * NV + grp * SC;
    };
    // B operand of the state, MN-major: off(k, n) = (n/8)*2048 + (k/8)*128 + (k%8)*16 + (n%8)*2
    uint8_t* sS_row = smem + C::S + (SC / 8 * grp) * 2048 + rowi * 16;
    float S[SC];
    auto load_state = [&](const float* st) {
#pragma unroll
      for (int u = 0; u < SC / 4; u++) {
        const float4 x = *reinterpret_cast<const float4*>(st + u * 4);
        S[4 * u] = x.x; S[4 * u + 1] = x.y; S[4 * u + 2] = x.z; S[4 * u + 3] = x.w;
      }
    };
    auto put_operand = [&](int u0, int n) {                // pieces u0 .. u0 + n - 1 of this row's columns as fp16
#pragma unroll
      for (int u = u0; u < u0 + n; u++)
        *reinterpret_cast<uint4*>(sS_row + u * 2048) = make_uint4(pack_h2(S[8 * u], S[8 * u + 1]), pack_h2(S[8 * u + 2], S[8 * u + 3]),
                                                                  pack_h2(S[8 * u + 4], S[8 * u + 5]), pack_h2(S[8 * u + 6], S[8 * u + 7]));
    };
    if (state_warp) {
      load_state(chain_state(0));
      put_operand(0, SC / 8);
      tc::fence_async_smem();
      tc::mbar_arrive(&bars.s[0]);
    }
    int in_chain = 0, chain = 0;                           // chunk of the chain, chain of the slot
    for (int v = 0; v < n_virtual; v++) {
      const uint32_t par = v & 1;
      const uint32_t d1 = tmem + par * NV, d2 = tmem + 2 * NV;
      // ---- U (token rows = TMEM lanes 0-63 of D1) as the next operand: off(t, n) = (n/8)*1024 + t*16 + (n%8)*2 ----
      if (u_warp) {
        tc::mbar_wait(&bars.mma[par], (v >> 1) & 1, abort_flag, 3);
        tc::fence_after_sync();
        uint32_t r[UC];
        if constexpr (UC == 32) tc::tmem_ld32(d1 + (uint32_t)(grp * UC) + ((uint32_t)(lq * 32) << 16), r);
        else tc::tmem_ld16(d1 + (uint32_t)(grp * UC) + ((uint32_t)(lq * 32) << 16), r);
        tc::tmem_ld_wait();
        uint8_t* urow = smem + C::U + (UC / 8 * grp) * 1024 + rowi * 16;
#pragma unroll
        for (int u = 0; u < UC / 8; u++)
          *reinterpret_cast<uint4*>(urow + u * 1024) =
              make_uint4(pack_h2(__uint_as_float(r[8 * u]), __uint_as_float(r[8 * u + 1])), pack_h2(__uint_as_float(r[8 * u + 2]), __uint_as_float(r[8 * u + 3])),
                         pack_h2(__uint_as_float(r[8 * u + 4]), __uint_as_float(r[8 * u + 5])), pack_h2(__uint_as_float(r[8 * u + 6]), __uint_as_float(r[8 * u + 7])));
        tc::fence_async_smem();
        tc::fence_before_sync();
        tc::mbar_arrive(&bars.u);
      }
      // ---- state: S <- S e^{G_last} + Kt^T U (lane = k row), refresh the fp16 operand copy ----
      if (state_warp) {
        tc::mbar_wait(&bars.kb[par], (v >> 1) & 1, abort_flag, 2);
        const float dec = reinterpret_cast<const float*>(smem + par * C::STAGE + C::DEC)[rowi];
        tc::mbar_wait(&bars.mma2, par, abort_flag, 4);
        tc::fence_after_sync();
        const bool last = in_chain == n_chunks - 1;
#pragma unroll
        for (int hf = 0; hf < SC / 32; hf++) {
          uint32_t r[32];
          tc::tmem_ld32(d2 + (uint32_t)(grp * SC + hf * 32) + ((uint32_t)(lq * 32) << 16), r);
          tc::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j++) S[hf * 32 + j] = fmaf(S[hf * 32 + j], dec, __uint_as_float(r[j]));
          if (!last) put_operand(4 * hf, 4);
        }
        if (last) {
          // last chunk of a chain: its final state goes back to memory and the slot's next chain begins
          float* st = chain_state(chain);
          if (!*(volatile int*)abort_flag) {
#pragma unroll
            for (int u = 0; u < SC / 4; u++)
              *reinterpret_cast<float4*>(st + u * 4) = make_float4(S[4 * u], S[4 * u + 1], S[4 * u + 2], S[4 * u + 3]);
          }
          if (v + 1 < n_virtual) {
            load_state(chain_state(chain + 1));
            put_operand(0, SC / 8);
          }
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        tc::mbar_arrive(&bars.s[par ^ 1]);
      }
      if (++in_chain == n_chunks) { in_chain = 0; chain++; }
    }
  }
}

// kernel 2: one chain's NV columns per CTA, units in the workspace
template <int NV>
__global__ __launch_bounds__(512, 1) void kda_chunk_scan_kernel(
    const uint8_t* __restrict__ ws, float* __restrict__ state, float* __restrict__ out_f32, int seqlen, int H, int n_chunks,
    const int* __restrict__ slots, float scale, int* __restrict__ status, const __grid_constant__ CUtensorMap map_out) {
  extern __shared__ __align__(128) uint8_t smem[];
  __shared__ ChainBars bars;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x;
  const int slice = blockIdx.x, job = blockIdx.z * H + blockIdx.y;
  if (tid == 0) {
    chain_init(bars);
    tc::mbar_fence_init();
    abort_flag = 0;
  }
  if (tid < 32) tc::tmem_alloc(&tmem_slot, 4 * NV);
  pdl_wait();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  // the unit of chunk v: heads are the fastest index (see kernel 1)
  const uint8_t* unit0 = ws + ((size_t)blockIdx.z * n_chunks * H + blockIdx.y) * U_BYTES;
  chain_cta<NV, false>(smem + ((1024u - (tc::smem_u32(smem) & 1023u)) & 1023u), bars, tmem, &abort_flag,
                       [&](int v) { return unit0 + (size_t)v * H * U_BYTES; }, nullptr, nullptr, nullptr, 0, job, 1, n_chunks, n_chunks, slice, H, seqlen,
                       state, out_f32, slots, scale, &map_out);
  tc::fence_before_sync();
  __syncthreads();
  if (tid < 32) tc::tmem_dealloc(tmem, 4 * NV);
  if (tid == 0 && abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
}

// =================================================================================================
// fused form: preparation and scan in ONE persistent launch
//
// One CTA of 512 threads per SM.  The first n_slots x (128 / NV) CTAs are chain CTAs: a slot is one (batch, head)
// chain - or, when the call has more than 48 chains, n_jobs / n_slots chains one after the other (the state is
// swapped at the chain boundary) - and has a CTA for every NV value columns.  Every other CTA
// hosts two preparation workers of 256 threads (its two halves, each with its own shared memory, TMEM columns and
// named barrier), which take the units round robin in the order the slots need them.  A unit travels through a ring
// of 16 or 32 chunk slots per chain slot in global memory - a few tens of MB that stay in L2 - instead of a per-chunk workspace in HBM:
//   ready[slot][v % depth] = v + 1 once the unit of that chunk is complete (release store after the worker's writes),
//   consumed[chain CTA]  = number of chunks whose unit has landed in the chain CTA's shared memory (the slot of chunk c
//                          may be rewritten once consumed > c for all CTAs of the slot).
// A worker that finds its slot still occupied, and a chain CTA that finds its unit not yet written, poll with a
// bound (about a second); on expiry they record HK_ERR_TIMEOUT, raise the launch-wide abort word and finish without
// waiting again.  All CTAs must be resident at once: the launch is cooperative and sized to the SM count.
// =================================================================================================
template <int NV>
constexpr uint32_t fused_smem() { return Chain<NV>::SMEM > 2 * P1_SMEM + 1024 ? Chain<NV>::SMEM : 2 * P1_SMEM + 1024; }

template <bool GATED, int NV>
__global__ __launch_bounds__(512, 1) void kda_fused_kernel(
    const __grid_constant__ CUtensorMap map_qkv, const __grid_constant__ CUtensorMap map_qk, const __grid_constant__ CUtensorMap map_g, const void* __restrict__ beta_in,
    uint8_t* __restrict__ ring, int* __restrict__ flags, float* __restrict__ state,
    float* __restrict__ out_f32, int seqlen, int H, int n_chunks, int n_jobs, int n_slots, int kr, const int* __restrict__ slots,
    float scale, int* __restrict__ status, const float* __restrict__ dt_bias, const float* __restrict__ a_log,
    float lower_bound, const __grid_constant__ CUtensorMap map_out) {
  extern __shared__ __align__(128) uint8_t smem_raw[];
  __shared__ ChainBars bars;
  __shared__ PrepShared prep[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;

  const int tid = threadIdx.x, warp = tid >> 5;
  constexpr int SLICES = Chain<NV>::SLICES;
  const int n_chain_ctas = n_slots * SLICES;
  int* g_abort = flags;
  int* ready = flags + F_FLAG_INTS;                        // [n_slots][ring depth], a line per slot
  int* consumed = ready + (size_t)n_slots * F_LINE;        // [n_chain_ctas], a line each
  const int n_virtual = (n_jobs / n_slots) * n_chunks;     // chunks a slot walks

  if (tid == 0) {
    chain_init(bars);
    prep_init(prep[0]);
    prep_init(prep[1]);
    tc::mbar_fence_init();
    abort_flag = 0;
  }
  if (warp == 0) tc::tmem_alloc(&tmem_slot, 512);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  // tiles start at a 1 KB boundary: the 128-byte-swizzle pattern is a function of the shared-memory address
  uint8_t* const smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);

  if ((int)blockIdx.x >= n_chain_ctas) {
    // =========================== two preparation workers ===========================
    const int sub = warp >> 3;
    // unit `it` of a worker, in the order the slots need them: running chunk v of every slot, then v + 1, ...
    auto make_unit = [&](int it, PrepDesc& u) {
      const long long n = ((int)blockIdx.x - n_chain_ctas) * 2 + sub + (long long)it * ((int)gridDim.x - n_chain_ctas) * 2;
      const int v = (int)min(n / n_slots, (long long)n_virtual), slot = (int)(n % n_slots);
      const int chunk = v % n_chunks, job = slot + n_slots * (v / n_chunks);
      u.b = job / H;
      u.t0 = chunk * KC;
      u.tok0 = u.b * seqlen + u.t0;
      u.n_valid = v < n_virtual ? min(KC, seqlen - chunk * KC) : 0;
      u.head = job % H;
      u.unit = (v & (kr - 1)) * n_slots + slot;
      u.slot = slot;
      u.value = v + 1;
    };
    PrepCtx ctx;
    ctx.smem = smem + sub * P1_SMEM; ctx.sh = &prep[sub]; ctx.abort_flag = &abort_flag; ctx.tid = tid & 255; ctx.bar_id = 1 + sub;
    if (ctx.tid < 2) make_unit(ctx.tid, prep[sub].unit[ctx.tid]);
    prep_sync<true>(ctx);
    if (ctx.tid == 0) {
      prep_fetch_g(ctx, 0, &map_g);
      prep_fetch_qkv(ctx, 0, &map_qkv, &map_qk, H);
    }
    int it = 0;
    for (; PREP_UNIT(n_valid, it) > 0; it++)
      prep_unit<GATED, SLICES>(ctx, it, &map_qkv, &map_qk, &map_g, beta_in, ring, H, dt_bias, a_log, lower_bound, tmem + sub * 256, ready, consumed,
                               g_abort, kr, make_unit);
    if (it > 0 && (ctx.tid >> 5) == PUB_WARP) prep_publish(ctx, it - 1, ready, kr);
  } else {
    const int cslot = blockIdx.x / SLICES;                  // this CTA's chain slot
    chain_cta<NV, true>(smem, bars, tmem, &abort_flag, [&](int v) { return ring + ((size_t)(v & (kr - 1)) * n_slots + cslot) * U_BYTES; },
                        ready + (size_t)cslot * F_LINE, consumed + (size_t)blockIdx.x * F_LINE, g_abort, kr, cslot, n_slots, n_chunks, n_virtual,
                        blockIdx.x % SLICES, H, seqlen, state, out_f32, slots, scale, &map_out);
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
  if (tid == 0 && abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
}

}  // namespace hk

namespace hk {
namespace {
// The fused launch serves calls with few (batch, head) chains: every chain occupies an SM or two, the rest prepare.
// hk_kda_chunked_set_form(1) keeps the two-kernel form for every call (cross-check of the two forms in the tests).
int g_chunked_form = 0;
// Chain slots of the fused launch and the value columns of a chain CTA for n_jobs (batch, head) chains; no slots = use the two-kernel
// form.  Chains share slots evenly (a slot walks its chains one after the other), and the preparation keeps 64 SMs or more.  Of the
// divisors of n_jobs from 16 to 48, or n_jobs itself, the one for which the longer of the two sides takes least per chunk of all
// chains.  The weights are tuned, not what the sides need: a chain CTA counts 1,380 a chunk with all 128 columns, 1,100 with 64, an SM of
// preparation workers 5,800 a unit (with 32 heads they need about 1,550 ns, 1,150 and 4,700, by which 3 x 8,192 x 32 would get 48 slots: 754 us,
// 664 with 32; a slot's start and the units' whole rounds are not in the sum).  What they choose was the fastest of all candidates at each of
// 18 shapes, among them 32,768 tokens x 8, 16, 32 heads, 16,384 x 64, 2 x 12,000 x 64, 4 x 3,000 x 16, 8 x 4,096 x 32, 6 x 4,000 x 24,
// 12 x 2,048 x 8, 3 x 5,000 x 16; us, chosen / next: 32,768 x 32 870 with a CTA a chain / 1,169 with two, x 16 573 with two / 686, x 8 561 / 686,
// 3 x 5,000 x 16 250 with 24 slots / 253 with 48, 5 x 4,096 x 32 562 with 32 / 593 with 40.
// Waits counted in a measuring build, 32,768 tokens x 32 heads: neither side is much the longer one, a worker waits 2,060 of a unit's 20,600
// cycles for a ring slot, a chain CTA 600 of a chunk's 3,000 for the 48 KB it needs first; with 16 and 8 heads the chains are the longer side.
// `room`: the slots that the workspace is sized for, the largest number that divides the chains: it covers calls of fewer sequences.
struct FusedShape { int slots, nv, room; };
FusedShape fused_shape(long long n_jobs) {
  FusedShape best{0, KD, 0};
  if (g_chunked_form != 0 || n_jobs <= 0) return best;
  const int sms = sm_count();
  long long best_cost = LLONG_MAX;
  for (int d = 48; d >= 1; d--) {
    if (n_jobs % d != 0 || (d != n_jobs && d < 16)) continue;
    for (int nv = KD; nv >= 64; nv /= 2) {
      const int workers = sms - d * (KD / nv);
      if (workers < 64) continue;
      if (!best.room) best.room = d;
      const long long chain = (nv == KD ? 1380000LL : 1100000LL) / d, prep = 5800000LL / workers, cost = chain > prep ? chain : prep;
      if (cost < best_cost) {
        best_cost = cost;
        best = {d, nv, best.room};
      }
    }
  }
  return best;
}
// Short calls run as two kernels although a fused form exists, in the ring's memory: the fused launch costs about 20 us before its first
// chunk is through (flags cleared, cooperative launch, ring start-up).  Fused / two kernels, us: 8 heads x 64 tokens 22.6 / 15.5, x 512 30.8 /
// 21.8, x 1,024 39.0 / 29.3; 32 heads x 256 31.7 / 18.8, x 1,003 61.4 / 46.3, x 1,024 60.6 / 46.6; 64 heads x 512 67.8 / 40.1.  The line
// is the memory: all units have to fit the ring's (16 chunks per slot).
bool short_call(long long n_jobs, int n_chunks, int n_slots) {
  return n_jobs * n_chunks <= (long long)RING * n_slots && (2 * n_jobs <= sm_count() || n_chunks <= 12);
}
typedef CUresult (*EncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                             const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeFn tensor_map_encoder() {
  static const EncodeFn fn = []() -> EncodeFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    return getenv("HK_KDA_NO_TMA") == nullptr &&             // debug switch: no copy engine, i.e. the token-by-token kernels
                   cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess && qres == cudaDriverEntryPointSuccess
               ? (EncodeFn)p
               : nullptr;
  }();
  return fn;
}
bool encode_rows(CUtensorMap* map, const void* base, CUtensorMapDataType type, int elem, int channels, int seqlen, int bsz, int box_channels) {
  const EncodeFn encode = tensor_map_encoder();
  const cuuint64_t dims[3] = {(cuuint64_t)channels, (cuuint64_t)seqlen, (cuuint64_t)bsz};
  const cuuint64_t strides[2] = {(cuuint64_t)channels * elem, (cuuint64_t)seqlen * channels * elem};
  const cuuint32_t box[3] = {(cuuint32_t)box_channels, (cuuint32_t)KC, 1}, estr[3] = {1, 1, 1};
  return encode(map, type, 3, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
bool deep_ring(int n_slots, long long n_virtual) { return n_slots <= 16 && n_virtual >= 64; }
size_t fused_flag_bytes(int n_slots) {
  return (((size_t)F_FLAG_INTS + (size_t)n_slots * 3 * F_LINE) * sizeof(int) + 255) / 256 * 256;
}
size_t ring_bytes(int n_slots, int depth) { return fused_flag_bytes(n_slots) + (size_t)depth * n_slots * U_BYTES; }
}  // namespace
}  // namespace hk

HK_API int hk_kda_dispatch_is_chunked(int seqlen, int num_k_heads, int num_v_heads, int k_head_dim, int v_head_dim,
                                      int history_stride, int channelwise, int history) {
  return (channelwise && !history && seqlen >= hk::KC && k_head_dim == hk::KD && v_head_dim == hk::KD &&
          num_k_heads == num_v_heads && history_stride == 1)
             ? 1
             : 0;
}

HK_API int hk_kda_chunked_set_form(int form) {
  if (form != 0 && form != 1) return HK_ERR_INVALID;
  hk::g_chunked_form = form;
  return HK_OK;
}

HK_API size_t hk_kda_chunked_workspace_bytes(int bsz, int seqlen, int num_heads) {
  if (bsz <= 0 || seqlen <= 0 || num_heads <= 0) return 0;
  const long long n_jobs = (long long)bsz * num_heads;
  const size_t n_chunks = ((size_t)seqlen + hk::KC - 1) / hk::KC;
  const hk::FusedShape shape = hk::fused_shape(n_jobs);
  if (shape.slots) {
    const size_t ring = hk::ring_bytes(shape.room, hk::RING);
    return hk::deep_ring(shape.slots, n_jobs / shape.slots * n_chunks) ? std::max(ring, hk::ring_bytes(shape.slots, hk::DEEP_RING)) : ring;
  }
  return (size_t)bsz * num_heads * n_chunks * hk::U_BYTES;
}

namespace hk {
namespace {
// Without the tensor-map encoder, which every input and output of the chunked kernels needs: the same recurrence token by token.  Gates
// that the call leaves to the preparation are formed by their own kernel, as many tokens at a time as the workspace holds.
int prefill_without_tensor_maps(const void* mixed_qkv, const float* g_or_f, const void* beta_or_b, const float* dt_bias, const float* a_log,
                                float lower_bound, bool gated, float* state, void* out, float* out_f32, int bsz, int seqlen, int H,
                                const int* slots, void* workspace, size_t workspace_bytes, void* stream) {
  if (!gated)
    return hk_kda_recurrent(mixed_qkv, g_or_f, beta_or_b, state, out, out_f32, bsz, seqlen, H, H, KD, KD, 1, slots, 1, 0, stream);
  const size_t row = (size_t)H * KD;
  const int piece = (int)std::min<size_t>(seqlen, workspace_bytes / (row * 4 + H * 2));
  if (piece < 1) return HK_ERR_WORKSPACE;
  float* g = (float*)workspace;
  void* beta = g + piece * row;
  for (int b = 0; b < bsz; b++)
    for (int t = 0; t < seqlen; t += piece) {
      const int n = std::min(piece, seqlen - t);
      const size_t at = (size_t)b * seqlen + t;
      int st = hk_kda_gate((const float*)beta_or_b + at * H, g_or_f + at * row, dt_bias, a_log, lower_bound, beta, g, n, H, KD, stream);
      if (st == HK_OK)
        st = hk_kda_recurrent((const __nv_bfloat16*)mixed_qkv + at * 3 * row, g, beta, slots ? state : state + (size_t)b * row * KD,
                              (__nv_bfloat16*)out + at * row, out_f32 ? out_f32 + at * row : nullptr, 1, n, H, H, KD, KD, 1,
                              slots ? slots + b : nullptr, 1, 0, stream);
      if (st != HK_OK) return st;
    }
  return HK_OK;
}
int chunked_prefill_launch(const void* mixed_qkv, const float* g_or_f, const void* beta_or_b, const float* dt_bias,
                           const float* a_log, float lower_bound, bool gated, float* state, void* out,
                           float* out_f32, int bsz, int seqlen, int num_heads, const int* slots,
                           void* workspace, size_t workspace_bytes, void* stream) {
  HK_REQUIRE(mixed_qkv && g_or_f && beta_or_b && state && out && workspace);
  HK_REQUIRE(!gated || (dt_bias && a_log && aligned(dt_bias, 16) && aligned(beta_or_b, 4)));
  HK_REQUIRE(bsz > 0 && seqlen > 0 && num_heads > 0);
  HK_REQUIRE(bsz <= 65535 && (seqlen + KC - 1) / KC <= 65535);   // grid limits
  HK_REQUIRE(aligned(mixed_qkv, 16) && aligned(g_or_f, 16) && aligned(state, 16) && aligned(out, 16) &&
             aligned(workspace, 256) && (!out_f32 || aligned(out_f32, 16)));
  const int n_chunks = (seqlen + KC - 1) / KC, n_jobs = bsz * num_heads;
  const FusedShape shape = fused_shape(n_jobs);
  const int n_slots = shape.slots;
  if (workspace_bytes < (n_slots ? ring_bytes(shape.room, RING) : hk_kda_chunked_workspace_bytes(bsz, seqlen, num_heads))) return HK_ERR_WORKSPACE;
  if (!tensor_map_encoder())
    return prefill_without_tensor_maps(mixed_qkv, g_or_f, beta_or_b, dt_bias, a_log, lower_bound, gated, state, out, out_f32, bsz, seqlen,
                                       num_heads, slots, workspace, workspace_bytes, stream);
  const bool deep = n_slots && deep_ring(n_slots, (long long)n_jobs / n_slots * n_chunks) && workspace_bytes >= ring_bytes(n_slots, DEEP_RING);
  const int kr = deep ? DEEP_RING : RING;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(kda_chunk_prep_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(P1_SMEM + 1024)) != cudaSuccess ||
        cudaFuncSetAttribute(kda_chunk_prep_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(P1_SMEM + 1024)) != cudaSuccess ||
        cudaFuncSetAttribute(kda_chunk_scan_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Chain<64>::SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(kda_chunk_scan_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Chain<128>::SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(kda_fused_kernel<false, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_smem<64>()) != cudaSuccess ||
        cudaFuncSetAttribute(kda_fused_kernel<true, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_smem<64>()) != cudaSuccess ||
        cudaFuncSetAttribute(kda_fused_kernel<false, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_smem<128>()) != cudaSuccess ||
        cudaFuncSetAttribute(kda_fused_kernel<true, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fused_smem<128>()) != cudaSuccess)
      return HK_ERR_CUDA;
    attr_set[dev] = true;
  }
  // tensor maps of the inputs, [batch][token][channels]: boxes of 64 tokens x 128 bytes, 128-byte swizzle, zeros past the last token;
  // and of the output [batch][token][head][128] bf16: 64 channels x 1 head x 64 tokens x 1 sequence
  alignas(64) CUtensorMap map_qkv, map_qk, map_g, map_out;
  if (!encode_rows(&map_qkv, mixed_qkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, 3 * num_heads * KD, seqlen, bsz, 64) ||
      !encode_rows(&map_g, g_or_f, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, num_heads * KD, seqlen, bsz, 32))
    return HK_ERR_CUDA;
  {
    const size_t row = (size_t)3 * num_heads * KD * 2;
    const cuuint64_t dims[4] = {32, (cuuint64_t)seqlen, (cuuint64_t)3 * num_heads * 4, (cuuint64_t)bsz};
    const cuuint64_t strides[3] = {row, 64, (cuuint64_t)seqlen * row};
    const cuuint32_t box[4] = {32, (cuuint32_t)KC, 4, 1}, estr[4] = {1, 1, 1, 1};
    if (tensor_map_encoder()(&map_qk, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(mixed_qkv), dims, strides, box, estr,
                             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return HK_ERR_CUDA;
  }
  {
    const cuuint64_t dims[4] = {(cuuint64_t)KD, (cuuint64_t)num_heads, (cuuint64_t)seqlen, (cuuint64_t)bsz};
    const cuuint64_t strides[3] = {(cuuint64_t)KD * 2, (cuuint64_t)num_heads * KD * 2, (cuuint64_t)seqlen * num_heads * KD * 2};
    const cuuint32_t box[4] = {64, 1, (cuuint32_t)KC, 1}, estr[4] = {1, 1, 1, 1};
    if (tensor_map_encoder()(&map_out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, out, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                             CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return HK_ERR_CUDA;
  }
  cudaStream_t s = as_stream(stream);
  int* st = device_status_ptr();
  const float scale = 1.0f / sqrtf((float)KD);
  if (!gated) {
    dt_bias = a_log = nullptr;
    lower_bound = 0.f;
  }
  if (n_slots && !short_call(n_jobs, n_chunks, n_slots)) {
    // one cooperative launch: chain CTAs first, preparation workers on all others
    const size_t flag_bytes = fused_flag_bytes(n_slots);
    if (cudaMemsetAsync(workspace, 0, flag_bytes, s) != cudaSuccess) return HK_ERR_CUDA;
    const bool split = shape.nv < KD;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(sm_count());
    cfg.blockDim = dim3(512);
    cfg.dynamicSmemBytes = split ? fused_smem<64>() : fused_smem<128>();
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    auto kern = gated ? (split ? kda_fused_kernel<true, 64> : kda_fused_kernel<true, 128>)
                      : (split ? kda_fused_kernel<false, 64> : kda_fused_kernel<false, 128>);
    return cudaLaunchKernelEx(&cfg, kern, map_qkv, map_qk, map_g, beta_or_b, (uint8_t*)workspace + flag_bytes, (int*)workspace, state, out_f32, seqlen,
                              num_heads, n_chunks, n_jobs, n_slots, kr, slots, scale, st, dt_bias, a_log, lower_bound, map_out) == cudaSuccess
               ? HK_OK
               : HK_ERR_CUDA;
  }
  const dim3 grid(num_heads, n_chunks, bsz);
  auto prep = gated ? kda_chunk_prep_kernel<true> : kda_chunk_prep_kernel<false>;
  if (pdl_launch(prep, grid, dim3(256), P1_SMEM + 1024, s, map_qkv, map_qk, map_g, beta_or_b, (uint8_t*)workspace, seqlen, num_heads, n_chunks, st,
                 dt_bias, a_log, lower_bound) != cudaSuccess)
    return HK_ERR_CUDA;
  // half a head per CTA while these are one wave
  const bool split = 2 * n_jobs <= sm_count();
  return pdl_launch(split ? kda_chunk_scan_kernel<64> : kda_chunk_scan_kernel<128>, dim3(split ? 2 : 1, num_heads, bsz), dim3(512),
                    split ? Chain<64>::SMEM : Chain<128>::SMEM, s, (const uint8_t*)workspace, state, out_f32, seqlen, num_heads, n_chunks, slots,
                    scale, st, map_out) == cudaSuccess
             ? HK_OK
             : HK_ERR_CUDA;
}
}  // namespace
}  // namespace hk

HK_API int hk_kda_chunked_prefill(const void* mixed_qkv, const float* g, const void* beta,
                                  float* state, void* out, float* out_f32, int bsz, int seqlen,
                                  int num_heads, const int* slots, void* workspace,
                                  size_t workspace_bytes, void* stream) {
  return hk::chunked_prefill_launch(mixed_qkv, g, beta, nullptr, nullptr, 0.f, false, state, out, out_f32, bsz,
                                    seqlen, num_heads, slots, workspace, workspace_bytes, stream);
}

HK_API int hk_kda_chunked_prefill_gated(const void* mixed_qkv, const float* f, const float* b,
                                        const float* dt_bias, const float* a_log, float lower_bound,
                                        float* state, void* out, float* out_f32, int bsz, int seqlen,
                                        int num_heads, const int* slots, void* workspace,
                                        size_t workspace_bytes, void* stream) {
  return hk::chunked_prefill_launch(mixed_qkv, f, b, dt_bias, a_log, lower_bound, true, state, out, out_f32, bsz,
                                    seqlen, num_heads, slots, workspace, workspace_bytes, stream);
}
