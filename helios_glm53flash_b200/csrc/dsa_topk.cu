// Exact top-k selection over fp16 score rows for the DSA indexer.
// Interface and output contract of helios::aux::dsa_topk (reference: src/cuda/aux/dsa_topk.cu:73-273,
// :668-732): on the order-preserving 16-bit key of the fp16 bit pattern (:21-24) find the k-th
// largest value v*; emit every entry above v* in ascending index order, then entries equal to v*
// in ascending index order until k are out; -inf (and anything below it) is never selected; if a
// row holds fewer than k selectable entries all of them are emitted; the rest of the k_pad-wide
// output row is -1.  Integer work: results are bit-exact by construction.
//
// Radix select: a histogram of the top 11 key bits, one of the low 5 bits inside the crossing bucket, then a single ordered
// compaction that places the "above" entries and the tie entries at once (the reference makes two histogram sweeps and two
// compaction sweeps of global memory).  Three kernels:
//   dsa_topk_cluster_kernel   at most 10 rows of 4,096 to 8,192 scores or 16 of up to 262,144, read once into the registers of a cluster of 8
//                             or 16 CTAs
//   dsa_topk_rows_kernel      other rows of up to 16,384 scores, read once into registers, a small CTA each
//   dsa_topk_kernel           every other call (many long rows, lengths known on the device only): one CTA of 1,024 threads per
//                             row, which sweeps the row three times; topk_row also selects among candidates in shared memory
#include <cooperative_groups.h>

#include <algorithm>

#include "hk_common.cuh"

namespace hk {

constexpr int TK_THREADS = 1024;
constexpr int TK_WARPS = TK_THREADS / 32;
constexpr uint32_t KEY_NEG_INF = 0x03ffu;  // key of fp16 -inf (0xfc00)

__device__ __forceinline__ uint32_t topk_key(uint32_t u16) {
  return (u16 & 0x8000u) ? (~u16 & 0xffffu) : (u16 | 0x8000u);
}

// Exclusive block scan of one int per thread; returns the exclusive prefix, *total = block sum.
// `scratch` holds TK_WARPS + 1 ints.  Contains two barriers.
__device__ __forceinline__ int block_exscan(int v, int* scratch, int* total) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int n = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += n;
  }
  if (lane == 31) scratch[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int wv = scratch[lane];
    int wi = wv;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int n = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += n;
    }
    scratch[lane] = wi - wv;
    if (lane == 31) scratch[TK_WARPS] = wi;
  }
  __syncthreads();
  *total = scratch[TK_WARPS];
  return scratch[warp] + incl - v;
}

// Rows are read as aligned 16-byte pieces whatever the row's start: piece i8 of a row that starts `lead` elements behind a
// 16-byte boundary holds elements 8 i8 - lead .. 8 i8 - lead + 7.  (Score rows follow one another with the caller's stride, the
// pool count, so seven of eight contexts have rows off the boundary; one 2-byte load per score made those sweeps 2-4 times
// longer.)  Pieces that reach over an end of the row are read element by element; what lies outside is key 0, never selected.
__device__ __forceinline__ int row_lead(const uint16_t* row) { return (int)((reinterpret_cast<uintptr_t>(row) & 15) >> 1); }
__device__ __forceinline__ uint4 load8_raw(const uint16_t* row, int lead, int i8, int T) {
  const int base = i8 * 8 - lead;
  if (base >= 0 && base + 8 <= T) return *reinterpret_cast<const uint4*>(row + base);
  uint32_t w[4] = {0, 0, 0, 0};   // 0xffff = key 0
#pragma unroll
  for (int j = 0; j < 8; j++) {
    const uint32_t u = base + j >= 0 && base + j < T ? row[base + j] : 0xffffu;
    w[j >> 1] |= u << (16 * (j & 1));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void keys8(uint4 v, uint32_t (&key)[8]) {
  const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
  for (int j = 0; j < 4; j++) {
    key[2 * j] = topk_key(w[j] & 0xffffu);
    key[2 * j + 1] = topk_key(w[j] >> 16);
  }
}

// Where a selected index goes: the index row and, optionally, the expanded token row of the same slot
// (helios::attn::pool_expand_row folded in: slot i -> tokens 4 idx .. 4 idx + 3, each kept if <= cur, else -1; the
// caller appends the four tail tokens in slot k_pad).
struct TopkSink {
  int* idx;          // [k_pad] (global or shared)
  int4* raw;         // [k_pad + 1] or nullptr
  int cur;
  __device__ __forceinline__ void put(int slot, int v) const {
    idx[slot] = v;
    if (raw) {
      const int tk = v * POOL;
      raw[slot] = v < 0 ? make_int4(-1, -1, -1, -1)
                        : make_int4(tk <= cur ? tk : -1, tk + 1 <= cur ? tk + 1 : -1, tk + 2 <= cur ? tk + 2 : -1,
                                    tk + 3 <= cur ? tk + 3 : -1);
    }
  }
  __device__ __forceinline__ void put_tail(int k_pad) const {
    if (raw)
      raw[k_pad] = make_int4(cur - 3 >= 0 ? cur - 3 : -1, cur - 2 >= 0 ? cur - 2 : -1, cur - 1 >= 0 ? cur - 1 : -1,
                             cur >= 0 ? cur : -1);
  }
};

// One row by one CTA of TK_THREADS threads; `row` and the sink's index row may point to global or shared memory.
__device__ __forceinline__ void topk_row(const uint16_t* row, const TopkSink row_o, int T, int k, int k_pad) {
  const int t = threadIdx.x;
  const int lead = row_lead(row), n_slots = (T + lead + 7) >> 3;

  __shared__ int hist[2048];
  __shared__ int scan_ws[TK_WARPS + 1];
  __shared__ int sh_sel[3];  // crossing bucket, count above it, (sweep 2) low bits

  // ---- sweep 1: histogram of key >> 5 over selectable entries (bucket >= 32 <=> key > -inf) ----
  for (int i = t; i < 2048; i += TK_THREADS) hist[i] = 0;
  __syncthreads();
  for (int i8 = t; i8 < n_slots; i8 += TK_THREADS) {
    uint32_t key[8];
    keys8(load8_raw(row, lead, i8, T), key);
#pragma unroll
    for (int j = 0; j < 8; j++)
      if (key[j] > KEY_NEG_INF) atomicAdd(&hist[key[j] >> 5], 1);
  }
  __syncthreads();
  // thread t owns buckets 2047-2t and 2046-2t (descending); find where the running count crosses k
  int h_hi = hist[2047 - 2 * t], h_lo = hist[2046 - 2 * t];
  int total_sel;
  int excl = block_exscan(h_hi + h_lo, scan_ws, &total_sel);
  if (t == 0) sh_sel[0] = -1;
  __syncthreads();
  if (total_sel >= k && k > 0) {
    if (excl < k && excl + h_hi >= k) { sh_sel[0] = 2047 - 2 * t; sh_sel[1] = excl; }
    else if (excl + h_hi < k && excl + h_hi + h_lo >= k) { sh_sel[0] = 2046 - 2 * t; sh_sel[1] = excl + h_hi; }
  }
  __syncthreads();
  const int b1 = sh_sel[0];
  uint32_t thresh;
  int cnt_gt, n_eq_take;
  if (b1 < 0) {
    // fewer than k selectable entries (or k == 0): take them all, no ties
    thresh = KEY_NEG_INF;
    cnt_gt = k > 0 ? total_sel : 0;
    n_eq_take = 0;
    if (k == 0) thresh = 0xffffu;
  } else {
    const int above1 = sh_sel[1];
    // ---- sweep 2: low 5 bits inside bucket b1 ----
    if (t < 32) hist[t] = 0;
    __syncthreads();
    for (int i8 = t; i8 < n_slots; i8 += TK_THREADS) {
      uint32_t key[8];
      keys8(load8_raw(row, lead, i8, T), key);
#pragma unroll
      for (int j = 0; j < 8; j++)
        if ((int)(key[j] >> 5) == b1) atomicAdd(&hist[key[j] & 31u], 1);
    }
    __syncthreads();
    if (t < 32) {
      // lane l owns low value 31-l (descending)
      const int hv = hist[31 - t];
      int incl = hv;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (t >= o) incl += n;
      }
      const int need = k - above1;
      if (incl - hv < need && incl >= need) { sh_sel[2] = 31 - t; sh_sel[1] = above1 + incl - hv; }
    }
    __syncthreads();
    thresh = ((uint32_t)b1 << 5) | (uint32_t)sh_sel[2];
    cnt_gt = sh_sel[1];
    n_eq_take = k - cnt_gt;
  }

  // ---- sweep 3: ordered compaction, 8 consecutive elements per thread per tile ----
  int base_gt = 0, base_eq = 0;
  const int n_tiles = (n_slots + TK_THREADS - 1) / TK_THREADS;
  for (int tile = 0; tile < n_tiles; tile++) {
    if (base_gt >= cnt_gt && base_eq >= n_eq_take) break;  // block-uniform
    const int i8 = tile * TK_THREADS + t;
    uint32_t m_gt = 0, m_eq = 0;
    if (i8 < n_slots) {
      uint32_t key[8];
      keys8(load8_raw(row, lead, i8, T), key);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        if (key[j] > thresh && key[j] > KEY_NEG_INF) m_gt |= 1u << j;
        if (key[j] == thresh && n_eq_take > 0) m_eq |= 1u << j;
      }
    }
    const int packed = __popc(m_gt) | (__popc(m_eq) << 16);
    int tot;
    const int ex = block_exscan(packed, scan_ws, &tot);
    int o_gt = base_gt + (ex & 0xffff);
    int o_eq = base_eq + (ex >> 16);
    const int ibase = i8 * 8 - lead;
    while (m_gt) {
      const int j = __ffs((int)m_gt) - 1;
      m_gt &= m_gt - 1;
      row_o.put(o_gt++, ibase + j);
    }
    while (m_eq) {
      const int j = __ffs((int)m_eq) - 1;
      m_eq &= m_eq - 1;
      if (o_eq < n_eq_take) row_o.put(cnt_gt + o_eq, ibase + j);
      o_eq++;
    }
    base_gt += tot & 0xffff;
    base_eq += tot >> 16;
  }
  const int emitted = cnt_gt + min(base_eq, n_eq_take);
  for (int j = emitted + t; j < k_pad; j += TK_THREADS) row_o.put(j, -1);
  if (t == 0) row_o.put_tail(k_pad);
}

// raw != nullptr: the expanded token rows [R][4 k_pad + 4] are written as well, row r clipped at q_pos[r]
__global__ __launch_bounds__(TK_THREADS) void dsa_topk_kernel(
    const uint16_t* scores, int* __restrict__ out, int T, int s_stride, int k,
    int k_pad, const int* __restrict__ t_ptr, int t_seq, int* __restrict__ raw, const int* __restrict__ q_pos) {
  pdl_wait();
  if (t_ptr) T = t_seq > 0 ? t_ptr[blockIdx.x / t_seq] : *t_ptr;
  TopkSink sink{out + (size_t)blockIdx.x * k_pad,
                raw ? reinterpret_cast<int4*>(raw + (size_t)blockIdx.x * (4 * k_pad + 4)) : nullptr,
                raw ? q_pos[blockIdx.x] : 0};
  topk_row(scores + (size_t)blockIdx.x * s_stride, sink, T, k, k_pad);
}

// ------------------------------------------------------------------------------------------------
// Rows of up to 16,384 scores, a CTA of 256 to 512 threads each: the row is read once, every thread keeps NP <= 4
// consecutive pieces (8 NP keys) in registers; histogram, threshold and compaction work from there.  What bounds the
// one-CTA kernel above on such rows is its 1,024-thread barriers and scans (13 of them, three sweeps); here there are six,
// and small CTAs share an SM and hide one another's.  1,024 rows x 1,250 scores 19.3 -> 8.4 us, 1,024 x 4,096 20.3 -> 11.1,
// 4,096 x 8,192 102 -> 66, 1,024 x 16,000 43.5 -> 36.4.  (More pieces per thread instead of more threads: 128 registers and
// spills, 1,024 x 8,191 40.7 us; 1,024 threads for 32,000 scores: 83 us against 74.)
// Up to a row per SM nothing is shared and the time is one CTA's: 1,024 threads with one or two pieces each, 140 x 8,000 scores
// 7.3 -> 5.0 us (few rows of more than 4,096 scores: clusters, below).
// ------------------------------------------------------------------------------------------------
constexpr int TKR_MAX_THREADS = 512, TKR_MAX_PIECES = 4 * TKR_MAX_THREADS;

// scores of a thread's pieces -> their keys, two a word
template <int NP>
__device__ __forceinline__ void to_keys(uint4 (&pc)[NP]) {
#pragma unroll
  for (int u = 0; u < NP; u++)
#pragma unroll
    for (int i = 0; i < 4; i++) {
      uint32_t& w = (&pc[u].x)[i];
      w ^= ((w >> 15) & 0x00010001u) * 0x7fffu + 0x80008000u;   // sign: all bits, else the top one
    }
}
// f(j, key) over the 8 NP keys of a thread's pieces, j ascending with the element index
template <int NP, class F>
__device__ __forceinline__ void for_keys(const uint4 (&pc)[NP], F f) {
#pragma unroll
  for (int u = 0; u < NP; u++) {
    const uint32_t w[4] = {pc[u].x, pc[u].y, pc[u].z, pc[u].w};
#pragma unroll
    for (int j = 0; j < 8; j++) f(8 * u + j, j & 1 ? w[j >> 1] >> 16 : w[j >> 1] & 0xffffu);
  }
}

template <int NP, int FIXED>   // FIXED: threads of the CTA, 0 = as launched
__global__ __launch_bounds__(FIXED ? FIXED : TKR_MAX_THREADS, FIXED == 256 ? 4 : FIXED ? 1 : 2) void dsa_topk_rows_kernel(const uint16_t* scores, int* __restrict__ out, int T, int s_stride,
                                                                    int k, int k_pad, int* __restrict__ raw,
                                                                    const int* __restrict__ q_pos) {
  constexpr int NB = 8;                                    // buckets of each of the first 256 threads
  __shared__ __align__(16) int hist[2048];
  __shared__ int low[32];
  __shared__ int wsum[2][32];
  __shared__ int sel[2];                                   // crossing bucket, count above it
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, threads = FIXED ? FIXED : blockDim.x, warps = threads >> 5;
  const uint16_t* row = scores + (size_t)blockIdx.x * s_stride;
  for (int i = t; i < 2048; i += threads) hist[i] = 0;
  if (t < 32) low[t] = 0;
  if (t == 0) sel[0] = -1;
  pdl_release();
  pdl_wait();
  const TopkSink sink{out + (size_t)blockIdx.x * k_pad,
                      raw ? reinterpret_cast<int4*>(raw + (size_t)blockIdx.x * (4 * k_pad + 4)) : nullptr, raw ? q_pos[blockIdx.x] : 0};
  const int lead = row_lead(row), i8 = t * NP;
  uint4 pc[NP];
#pragma unroll
  for (int u = 0; u < NP; u++) pc[u] = load8_raw(row, lead, i8 + u, T);
  to_keys<NP>(pc);
  __syncthreads();
  // exclusive prefix over the block; one barrier, `slot` alternates between calls
  auto exscan = [&](int v, int slot, int* total) {
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (lane == 31) wsum[slot][warp] = incl;
    __syncthreads();
    const int x = lane < warps ? wsum[slot][lane] : 0;
    const int before = (int)__reduce_add_sync(0xffffffffu, (unsigned)(lane < warp ? x : 0)), all = (int)__reduce_add_sync(0xffffffffu, (unsigned)x);
    *total = all;
    return before + incl - v;
  };
  for_keys<NP>(pc, [&](int, uint32_t key) {
    if (key > KEY_NEG_INF) atomicAdd(&hist[key >> 5], 1);
  });
  __syncthreads();
  // thread t owns the NB buckets from 2047 - NB t downwards; find where the running count crosses k
  int mine[NB], sum = 0;
#pragma unroll
  for (int i = 0; i < NB; i++) {
    mine[i] = t < 256 ? hist[2047 - NB * t - i] : 0;
    sum += mine[i];
  }
  int total_sel;
  int run = exscan(sum, 0, &total_sel);
  if (total_sel >= k && k > 0 && run < k && run + sum >= k) {
#pragma unroll
    for (int i = 0; i < NB; i++) {
      if (run < k && run + mine[i] >= k) {
        sel[0] = 2047 - NB * t - i;
        sel[1] = run;
      }
      run += mine[i];
    }
  }
  __syncthreads();
  const int b1 = sel[0];
  uint32_t thresh = k == 0 ? 0xffffu : KEY_NEG_INF;        // fewer than k selectable entries: all of them, no ties
  int cnt_gt = k > 0 ? total_sel : 0, n_eq = 0;
  if (b1 >= 0) {
    for_keys<NP>(pc, [&](int, uint32_t key) {
      if ((int)(key >> 5) == b1) atomicAdd(&low[key & 31u], 1);
    });
    __syncthreads();
    // every warp: lane l owns low value 31 - l (descending)
    const int hv = low[31 - lane];
    int incl = hv;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    const int need = k - sel[1];
    const int src = __ffs((int)__ballot_sync(0xffffffffu, incl - hv < need && incl >= need)) - 1;
    thresh = ((uint32_t)b1 << 5) | (uint32_t)(31 - src);
    cnt_gt = sel[1] + __shfl_sync(0xffffffffu, incl - hv, src);
    n_eq = k - cnt_gt;
  }
  // ---- ordered compaction ----
  int n_gt = 0, n_tie = 0;
  for_keys<NP>(pc, [&](int, uint32_t key) {
    n_gt += key > thresh && key > KEY_NEG_INF;
    n_tie += key == thresh && n_eq > 0;
  });
  int tot;
  const int ex = exscan(n_gt | (n_tie << 16), 1, &tot);
  int o_gt = ex & 0xffff, o_eq = (unsigned)ex >> 16;
  if (n_gt || (n_tie && o_eq < n_eq)) {
    const int ibase = i8 * 8 - lead;
    for_keys<NP>(pc, [&](int j, uint32_t key) {
      if (key > thresh && key > KEY_NEG_INF) sink.put(o_gt++, ibase + j);
      else if (key == thresh && n_eq > 0) {
        if (o_eq < n_eq) sink.put(cnt_gt + o_eq, ibase + j);
        o_eq++;
      }
    });
  }
  const int emitted = cnt_gt + n_eq;
  for (int j = emitted + t; j < k_pad; j += threads) sink.put(j, -1);
  if (t == 0) sink.put_tail(k_pad);
}

#ifdef HK_TOPK_TRACE
__device__ long long hk_topk_trace[16];
#define TK_TRACE(slot) do { if (threadIdx.x == 0 && blockIdx.x == 0) hk_topk_trace[slot] = clock64(); } while (0)
#else
#define TK_TRACE(slot) do { } while (0)
#endif
// ------------------------------------------------------------------------------------------------
// A few long rows (the decode case is ONE row): a thread-block cluster of 8 or 16 CTAs works on a row, every thread on NP consecutive
// pieces of 8 elements that stay in registers, so the row is read from global memory once and no sweep is longer than 8 NP keys per
// thread.  A CTA has as many threads as the row's pieces need in equal shares (256 to 1,024).  The CTAs meet through distributed shared
// memory: every CTA adds up the row's buckets by eights from all CTAs, then looks at the eight buckets of the crossing one; the
// low-bit count sets are read by every CTA, which finds the threshold and, from the per-CTA counts, the offset of its own
// ordered output - two cluster barriers that hand data over and one that is arrived at long before it is waited for.
// What bounds it: these steps one after the other (65,536 scores in eight CTAs: load and count 1.5 us, the crossing bucket 1.0, low bits 0.9,
// offsets 0.9, output 1.0).  With 1,024 threads whatever the row's length the first CTAs had all of it, and a row of 65,552 scores two
// pieces a thread in half of the CTAs.  One row, eight CTAs of 1,024 threads -> now, us: 5,000 scores 5.1 (one CTA) -> 4.5, 16,384 7.2 -> 4.2,
// 32,768 5.8 -> 4.6, 65,536 5.75 -> 5.1, 65,552 8.0 -> 5.4, 131,072 7.4 -> 6.2, 200,000 11.9 -> 7.5; 16 rows of 20,000 11.1 -> 5.2.
// (The launch bound names the CTA per SM: at the 32 registers taken without it the four-piece form spilled.)
// Eight CTAs with NP = 1, 2, 4 cover rows of 65,536, 131,072 and 262,144 scores (1M tokens of context), up to seven fewer where a row starts
// off a 16-byte boundary; sixteen with NP = 1, 2 the last two.
// ------------------------------------------------------------------------------------------------
constexpr int TKC_PIECES = 8 * TK_THREADS;                // pieces of 8 elements that eight CTAs hold with NP = 1
constexpr int TKC_MAX_NP = 4;

template <int NP, int CTAS>
__global__ __launch_bounds__(TK_THREADS, 1) void dsa_topk_cluster_kernel(
    const uint16_t* scores, int* __restrict__ out, int T, int s_stride, int k, int k_pad,
    int* __restrict__ raw, const int* __restrict__ q_pos) {
  __shared__ __align__(16) int hist[2048];   // this CTA's bucket counts
  __shared__ int coarse[256];      // the same by eight buckets
  __shared__ int low[33];          // this CTA: counts of the low 5 bits inside the crossing bucket; [32] = keys above it
  __shared__ int wsum[2][TK_WARPS];
  __shared__ int sh_sel[3];
  __shared__ int sh_off[6];        // threshold low bits, count above threshold, this CTA's bases, total ties
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5, threads = blockDim.x, warps = threads >> 5;
  for (int i = t; i < 2048; i += threads) hist[i] = 0;
  if (t < 33) low[t] = 0;
  if (t == 0) sh_sel[0] = -1;
  namespace cg = cooperative_groups;
  pdl_release();
  pdl_wait();
  cg::cluster_group cluster = cg::this_cluster();
  const int c = (int)cluster.block_rank();
  const int row_id = blockIdx.x / CTAS;
  const uint16_t* row = scores + (size_t)row_id * s_stride;
  const TopkSink row_o{out + (size_t)row_id * k_pad,
                       raw ? reinterpret_cast<int4*>(raw + (size_t)row_id * (4 * k_pad + 4)) : nullptr, raw ? q_pos[row_id] : 0};

  TK_TRACE(0);
  const int lead = row_lead(row), i8 = (c * threads + t) * NP;
  uint4 pc[NP];
#pragma unroll
  for (int u = 0; u < NP; u++) pc[u] = load8_raw(row, lead, i8 + u, T);
  to_keys<NP>(pc);
  __syncthreads();
  // exclusive prefix over the block; one barrier, `slot` alternates between calls
  auto exscan = [&](int v, int slot, int* total) {
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    if (lane == 31) wsum[slot][warp] = incl;
    __syncthreads();
    const int x = lane < warps ? wsum[slot][lane] : 0;
    const int before = (int)__reduce_add_sync(0xffffffffu, (unsigned)(lane < warp ? x : 0));
    *total = (int)__reduce_add_sync(0xffffffffu, (unsigned)x);
    return before + incl - v;
  };
  for_keys<NP>(pc, [&](int, uint32_t key) {
    if (key > KEY_NEG_INF) atomicAdd(&hist[key >> 5], 1);
  });
  __syncthreads();
  if (t < 256) {
    const int4 x = *reinterpret_cast<const int4*>(hist + 8 * t), y = *reinterpret_cast<const int4*>(hist + 8 * t + 4);
    coarse[t] = x.x + x.y + x.z + x.w + y.x + y.y + y.z + y.w;
  }
  cluster.sync();                  // (1) all local histograms are complete
  TK_TRACE(1);
  // Thread t < 256 sums eight buckets over the row (descending) and finds where the running count crosses k; a warp then looks at the
  // eight.  Every CTA does so for itself: 8 KB of remote counts each and one cluster barrier less than sharing out the sums.
  int sum = 0;
  if (t < 256) {
#pragma unroll
    for (int rk = 0; rk < CTAS; rk++) sum += cluster.map_shared_rank(coarse, rk)[255 - t];
  }
  int total_sel;
  const int excl = exscan(sum, 0, &total_sel);
  if (k > 0 && excl < k && excl + sum >= k) { sh_sel[0] = 255 - t; sh_sel[1] = excl; }
  __syncthreads();
  if (warp == 0 && sh_sel[0] >= 0) {
    // lane 8 r + j: bucket j from the top of the eight, CTAs r, r + 4, ...
    const int bin = 8 * sh_sel[0] + 7 - (lane & 7), above = sh_sel[1];
    int v = 0;
#pragma unroll
    for (int rk = 0; rk < CTAS; rk += 4) v += cluster.map_shared_rank(hist, (lane >> 3) + rk)[bin];
    v += __shfl_xor_sync(0xffffffffu, v, 8);
    v += __shfl_xor_sync(0xffffffffu, v, 16);
    int incl = v;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o, 8);
      if ((lane & 7) >= o) incl += n;
    }
    __syncwarp();
    if (lane < 8 && above + incl - v < k && above + incl >= k) { sh_sel[0] = bin; sh_sel[1] = above + incl - v; }
  }
  __syncthreads();
  const int b1 = sh_sel[0], above1 = sh_sel[1];
  TK_TRACE(2);
  // local counts: low 5 bits inside bucket b1, and the keys in buckets above it.  Without a crossing bucket
  // (fewer than k selectable entries, or k == 0) every selectable key counts as "above".
  const int b_eff = b1 < 0 ? 31 : b1;
  int n_above = 0;
  for_keys<NP>(pc, [&](int, uint32_t key) {
    const int bk = (int)(key >> 5);
    if (bk == b1) atomicAdd(&low[key & 31u], 1);
    n_above += bk > b_eff;
  });
  n_above = (int)__reduce_add_sync(0xffffffffu, (unsigned)n_above);
  if (lane == 0 && n_above) atomicAdd(&low[32], n_above);
  cluster.sync();                  // (2) all local low-bit counts complete
  TK_TRACE(3);
  if (warp == 0) {
    // lane l owns low value 31-l (descending): the row's count and that of the CTAs before this one; lane rk also keys above the bucket
    int g = 0, before = 0;
#pragma unroll
    for (int rk = 0; rk < CTAS; rk++) {
      const int mine = cluster.map_shared_rank(low, rk)[31 - lane];
      g += mine;
      if (rk < c) before += mine;
    }
    const int above_before = (int)__reduce_add_sync(0xffffffffu, (unsigned)(lane < c ? cluster.map_shared_rank(low, lane)[32] : 0));
    int lowbits = 0, cnt_gt_row = k > 0 ? total_sel : 0, need_eq = 0;
    if (b1 >= 0) {
      int incl = g;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        int n = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += n;
      }
      const int need = k - above1;
      const unsigned who = __ballot_sync(0xffffffffu, incl - g < need && incl >= need);
      const int src = __ffs((int)who) - 1;                  // lane of the crossing low value
      lowbits = 31 - src;
      cnt_gt_row = above1 + __shfl_sync(0xffffffffu, incl - g, src);
      need_eq = k - cnt_gt_row;
      // keys above the threshold = above the bucket + low values above lowbits (lanes < src); ties = lane src
      const int base_gt = above_before + (int)__reduce_add_sync(0xffffffffu, (unsigned)(lane < src ? before : 0));
      const int base_eq = __shfl_sync(0xffffffffu, before, src), all_eq = __shfl_sync(0xffffffffu, g, src);
      if (lane == 0) { sh_off[2] = base_gt; sh_off[3] = base_eq; sh_off[4] = all_eq; }
    } else if (lane == 0) {
      sh_off[2] = k > 0 ? above_before : 0; sh_off[3] = 0; sh_off[4] = 0;
    }
    if (lane == 0) { sh_off[0] = lowbits; sh_off[1] = cnt_gt_row; sh_off[5] = need_eq; }
  }
  __syncthreads();
  // no CTA leaves while a peer may still read its shared memory: this one has read the others'
  asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory");
  uint32_t thresh;
  const int cnt_gt = sh_off[1], n_eq_take = sh_off[5];
  if (b1 < 0) thresh = k == 0 ? 0xffffu : KEY_NEG_INF;
  else thresh = ((uint32_t)b1 << 5) | (uint32_t)sh_off[0];
  TK_TRACE(4);
  // ---- ordered compaction inside the CTA, offset by the counts of the CTAs before it ----
  uint32_t m_gt = 0, m_eq = 0;
  for_keys<NP>(pc, [&](int j, uint32_t key) {
    if (key > thresh && key > KEY_NEG_INF) m_gt |= 1u << j;
    if (key == thresh && n_eq_take > 0) m_eq |= 1u << j;
  });
  int tot;
  const int ex = exscan(__popc(m_gt) | (__popc(m_eq) << 16), 1, &tot);
  TK_TRACE(5);
  int o_gt = sh_off[2] + (ex & 0xffff);
  int o_eq = sh_off[3] + (ex >> 16);
  const int ibase = i8 * 8 - lead;
  while (m_gt) {
    const int j = __ffs((int)m_gt) - 1;
    m_gt &= m_gt - 1;
    row_o.put(o_gt++, ibase + j);
  }
  while (m_eq) {
    const int j = __ffs((int)m_eq) - 1;
    m_eq &= m_eq - 1;
    if (o_eq < n_eq_take) row_o.put(cnt_gt + o_eq, ibase + j);
    o_eq++;
  }
  if (c == 0) {
    const int emitted = cnt_gt + min(sh_off[4], n_eq_take);
    for (int j = emitted + t; j < k_pad; j += threads) row_o.put(j, -1);
    if (t == 0) row_o.put_tail(k_pad);
  }
  TK_TRACE(6);
  asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

}  // namespace hk

#ifdef HK_TOPK_TRACE
extern "C" __attribute__((visibility("default"))) int hk_debug_topk_trace(long long* host_out) {
  return cudaMemcpyFromSymbol(host_out, hk::hk_topk_trace, sizeof(long long) * 16) == cudaSuccess ? 0 : 3;
}
#endif

namespace hk {
// clusters of sixteen CTAs of 1,024 threads that run at once; 0 where such clusters cannot be had
static int wide_clusters() {
  static int room[64] = {0};                                // + 1
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
  if (!room[dev]) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 16;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(TK_THREADS);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(dsa_topk_cluster_kernel<1, 16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(dsa_topk_cluster_kernel<2, 16>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, dsa_topk_cluster_kernel<2, 16>, &cfg) != cudaSuccess) {
      cudaGetLastError();                                   // (no such clusters: not an error of the call)
      n = 0;
    }
    room[dev] = n + 1;
  }
  return room[dev] - 1;
}
// common launcher; raw != nullptr adds the expansion
static int topk_launch(const void* scores, int s_stride, int* indices, int R, int T, int k, int k_pad, const int* t_ptr,
                       int t_seq, int* raw, const int* q_pos, cudaStream_t s) {
  const uint16_t* sc = (const uint16_t*)scores;
  // pieces of the longest-reaching row: rows of a stride that is no multiple of 8 start at any offset
  const int lead = R == 1 || s_stride % 8 == 0 ? (int)(((uintptr_t)scores & 15) >> 1) : 7;
  const int64_t pieces = ((int64_t)T + lead + 7) / 8;
  auto rows = [&](auto kern, int threads) {
    return pdl_launch(kern, dim3(R), dim3(threads), 0, s, sc, indices, T, s_stride, k, k_pad, raw, q_pos);
  };
  auto cluster = [&](auto kern, int np, int ctas) {         // the pieces in equal shares for all threads
    const int threads = (int)((pieces + ctas * np * 32 - 1) / (ctas * np * 32)) * 32;
    return pdl_launch_cluster(ctas, kern, dim3(R * ctas), dim3(threads < 256 ? 256 : threads), 0, s, sc, indices, T, s_stride, k, k_pad, raw,
                              q_pos);
  };
  auto sweeps = [&]() {
    return pdl_launch(dsa_topk_kernel, dim3(R), dim3(TK_THREADS), 0, s, sc, indices, T, s_stride, k, k_pad, t_ptr, t_seq, raw, q_pos);
  };
  // (figures at the kernels.  With many rows the clusters queue for eight free SMs of one GPC each and the one-CTA kernel is 3 to 20
  // times faster, measured at 64 to 4,096 rows.  Up to 4,096 scores one CTA is faster than the cluster: 1 x 2,500 4.1 / 4.6 us, 1 x 5,000
  // 5.1 / 4.5; up to 8,192, a piece a thread of one CTA, from eleven rows on: 10 x 5,000 4.62 / 4.54, 11 4.62 / 4.73, 16 4.62 / 4.95, 16 x 8,192
  // 4.58 / 4.91, 16 x 8,193 6.36 / 4.94.  Sixteen CTAs a row: from 40,000 scores for up to 3 rows (1 x 33,000 4.8 with eight / 5.0, 1 x 50,000 5.3 / 5.1, 4 x 50,000
  // 5.4 / 5.8), beyond 65,536 scores, where eight take two pieces a thread, for as many rows as there is room for at once: 7 x 65,552
  // 6.7 / 5.5, 8 x 65,552 6.5 / 10.6)
  // With company clusters stay the better ones: 20 selections of 16,384 scores on each of 8 streams 132 -> 91 us, a decode step of 11 MLA
  // layers of 8 sequences at 32,768, one stream each, 986 with a CTA a row / 968, of 4 507 / 492.
  cudaError_t e;
  if (t_ptr) e = sweeps();
  else if (pieces <= 256) e = rows(dsa_topk_rows_kernel<1, 256>, 256);
  else if (pieces > 512 && pieces <= (int64_t)TKC_PIECES * TKC_MAX_NP && R <= (pieces <= 1024 ? 10 : 16)) {
    const bool wide = pieces > 5120 && R <= (pieces <= TKC_PIECES ? std::min(3, wide_clusters()) : wide_clusters());
    e = wide ? (pieces <= 2 * TKC_PIECES ? cluster(dsa_topk_cluster_kernel<1, 16>, 1, 16) : cluster(dsa_topk_cluster_kernel<2, 16>, 2, 16))
        : pieces <= TKC_PIECES     ? cluster(dsa_topk_cluster_kernel<1, 8>, 1, 8)
        : pieces <= 2 * TKC_PIECES ? cluster(dsa_topk_cluster_kernel<2, 8>, 2, 8)
                                   : cluster(dsa_topk_cluster_kernel<4, 8>, 4, 8);
  } else if (pieces <= TKR_MAX_PIECES && R <= sm_count())    // a row per SM: as many threads as there are pieces, up to 1,024
    e = pieces <= 512    ? rows(dsa_topk_rows_kernel<1, 512>, 512)
        : pieces <= 1024 ? rows(dsa_topk_rows_kernel<1, 1024>, 1024)
                         : rows(dsa_topk_rows_kernel<2, 1024>, 1024);
  else if (pieces <= TKR_MAX_PIECES)                         // rows share SMs: small CTAs of up to four pieces per thread
    e = pieces <= 512    ? rows(dsa_topk_rows_kernel<2, 256>, 256)
        : pieces <= 1024 ? rows(dsa_topk_rows_kernel<4, 256>, 256)
                         : rows(dsa_topk_rows_kernel<4, 0>, (int)((pieces + 127) / 128) * 32);
  else e = sweeps();
  return e == cudaSuccess && cudaPeekAtLastError() == cudaSuccess ? HK_OK : HK_ERR_CUDA;
}
}  // namespace hk

HK_API int hk_dsa_topk(const void* scores, int s_stride, int* indices, int R, int T, int k,
                       int k_pad, const int* t_ptr, int t_seq, void* stream) {
  using namespace hk;
  HK_REQUIRE(scores && indices && R >= 0 && T >= 0 && k >= 0 && k <= k_pad && s_stride >= 0);
  HK_REQUIRE(k <= 32767);  // packed 16-bit counters in the compaction scan
  if (R == 0) return HK_OK;
  return topk_launch(scores, s_stride, indices, R, T, k, k_pad, t_ptr, t_seq, nullptr, nullptr, as_stream(stream));
}

HK_API int hk_dsa_topk_expand(const void* scores, int s_stride, int* indices, int* raw_idx, const int* q_pos, int R, int T,
                              int k, int after_scorer, void* stream) {
  using namespace hk;
  HK_REQUIRE(scores && indices && raw_idx && q_pos && R >= 0 && T >= 0 && k >= 0 && k <= 512 && s_stride >= 0);
  HK_REQUIRE(aligned(raw_idx, 16));
  (void)after_scorer;   // every selection kernel is launched as a programmatic dependent
  if (R == 0) return HK_OK;
  return topk_launch(scores, s_stride, indices, R, T, k, 512, nullptr, 0, raw_idx, q_pos, as_stream(stream));
}

#include "dsa_select_splitkv.cuh"
