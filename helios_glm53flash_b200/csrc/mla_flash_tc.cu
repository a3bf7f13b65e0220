// Absorbed MLA flash attention over the 512-wide fp16 latent cache on the 5th-generation tensor
// cores: dense causal ranges and gathered (sparse) rows, decode and prefill rows, final output or
// split-KV partials.  One kernel serves helios::attn::mla_sparse_decode and
// helios::attn::mla_dense_prefill (reference: src/cuda/attn/attn.cu:394-699, scalar kernels, one
// block per (row, head) or head pair).
//
// Work item = (query row, key split) -> one CTA; all 64 heads of the row share every latent row that
// is staged, so the cache is read once per row (the reference re-reads it per head pair).
// Per tile of 64 keys (64 KB, three tiles in flight):
//   S [64 heads x 64 keys]     = Q K^T   32 x tcgen05.mma.ws M64 N64 K16
//   softmax: a thread owns one head and 32 keys -> max / exp2 / sum run inside the thread, its partner (the other
//            32 keys) is met once per tile for the maximum; the running reference max only moves when a tile exceeds
//            it by 2^8 (lazy rescale of O)
//   O [64 heads x 512 ch]     += P V     8 x tcgen05.mma.ws M64 N256 K16: the SAME tile read MN-major as B
//            (the latent row is both key and value)
//
// What bounds it (long runs) is shared-memory bandwidth, 128 B per cycle: every operand read of a product and every byte
// the copy engine lays down counts.  The first form of this kernel (48-key tiles, plain M64 N48 for S, O^T = V^T P^T as
// M128 N64) moved 240 KB per 48 keys: Q is 64 KB and was read for every tile, and P four times.  1,900 cycles, measured 1,950.
// Here, per 64 keys: tile in 64 KB, K 64 KB, V 64 KB, P 8 KB in and 16 KB out, and of Q only channels 0-127 (16 KB): channels
// 128-511 live in tensor memory.  232 KB per 64 keys = 1,856 cycles, 27 % less per key.  Tensor memory is full: O 256
// columns (the .ws form spreads M = 64 over all lanes), S 2 x 32, Q 192.  The .ws products themselves need 1,568 cycles.
//
// The key tile sits in the 128-byte-swizzle layout: 8 blocks of 64 channels, each block = 64 key rows of 128 bytes with
// 16-byte chunk c of row r stored at c ^ (r % 8); the same bytes are B of both products.  Whole tiles of a dense range arrive
// with ONE TMA tensor copy each (3-D box {64 channels, 64 keys, 8 blocks}); gathered rows, and the last tile of a ragged
// dense range, as gather4 copies (four cache rows x one 64-channel block each, 128 per tile; a negative row number reads as
// zeros, so nothing behind the range is read).
// All hand-offs are mbarriers with bounded waits, executed by every lane of the waiting warp.
#include <cuda.h>   // CUtensorMap (types only; the encoder is fetched through the runtime at first use)

#include <cstdlib>
#include <cstring>

#include "mla_args.cuh"
#include "tc05.cuh"

namespace hk {

constexpr int FT_KEYS = 64;                       // keys per tile
constexpr int FT_NBUF = 3;                        // key tiles in flight
constexpr int FT_HEADS = 64;
constexpr int FT_QS = 128;                        // channels of Q in shared memory; the other 384 are in tensor memory
constexpr uint32_t FT_BLK = FT_KEYS * 128;        // one block of 64 channels: one 128-byte row per key
constexpr uint32_t FT_TILE = 8 * FT_BLK;          // 65536
constexpr uint32_t FS_K = 0;                      // FT_NBUF tiles, 1 KB aligned
constexpr uint32_t FS_Q = FS_K + FT_NBUF * FT_TILE;        // [2 blocks][64 heads][128 B], swizzled
constexpr uint32_t FS_P = FS_Q + FT_QS * FT_HEADS * 2;     // 2 x [64 heads][64 keys], swizzled
constexpr uint32_t FP_BYTES = FT_HEADS * FT_KEYS * 2;
constexpr uint32_t FS_MISC = FS_P + 2 * FP_BYTES;
constexpr uint32_t FS_SMEM = FS_MISC + 2048 + 1024;        // + slack to align the base to 1 KB (swizzle atoms)
constexpr uint32_t FT_O = 0, FT_S = 256, FT_Q = 320;       // tensor-memory columns: O 2 x 128, S 2 x 32, Q 192
constexpr uint32_t FT_QPITCH = (LATENT - FT_QS) * 2 + 16;  // row pitch of the staged queries: conflict-free 16-byte rows
constexpr int FT_POLL_NS = 40;                    // poll back-off of the waiting warps
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_THRESHOLD = 8.0f;         // log2 units: P stays below 2^8, fine for fp16
// warps 0-3 softmax and epilogue (one TMEM lane quarter each), 4 issues S = Q K^T, 5 issues O += P V, the rest load tiles.
// A warp gets one gather4 copy out per about 90 cycles whichever lanes issue them: eight warps for gathered rows; dense
// ranges need them for the ragged last tile only.
template <bool G4>
struct FtRoles {
  static constexpr int LOAD_WARPS = G4 ? 8 : 4, THREADS = (6 + LOAD_WARPS) * 32, COPIES = 128 / LOAD_WARPS;
};

struct FtMisc {
  uint64_t k_full[FT_NBUF], t_done[FT_NBUF];      // per tile buffer: tile landed, its P V finished
  uint64_t s_full[2], s_free[2], p_full[2];       // per S / P buffer
  uint64_t q_ready;
  unsigned long long mask[FT_NBUF];               // valid key slots of the tile in the buffer
  float mx[2][128];                               // tile maxima, by softmax thread and tile parity
  float l[128];
  uint32_t tmem;
  int abort_flag;
};
static_assert(sizeof(FtMisc) <= 2048, "misc area");

__device__ __forceinline__ void tma_load_tile(void* smem_dst, const CUtensorMap* tmap, int row, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          tc::smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(0), "r"(row), "r"(0), "r"(tc::smem_u32(bar))
      : "memory");
}

// Four gathered cache rows x one 64-channel block (4 x 128 B) in one tensor copy: the 2-D map covers the cache as
// [row][512 channels] with a box of {64 channels, 1 row}; the instruction names four row coordinates, the copy engine
// lays the four 128-byte pieces down one after the other and applies the 128-byte swizzle by destination address, i.e.
// exactly key slots k .. k+3 of a block of the tile layout.  A negative row is outside the tensor: zero fill.
__device__ __forceinline__ void tma_gather4_rows(void* smem_dst, const CUtensorMap* tmap, int channel, int r0, int r1, int r2,
                                                 int r3, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(
          tc::smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(channel), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(tc::smem_u32(bar))
      : "memory");
}

// G4: gathered rows (raw_idx); otherwise dense ranges.  tmap_box: 3-D map of the cache, tmap_rows: 2-D map for gather4.
template <bool G4>
__global__ __launch_bounds__(FtRoles<G4>::THREADS, 1) void mla_flash_tc_kernel(MlaArgs a, int* __restrict__ status,
                                                                               const __grid_constant__ CUtensorMap tmap_box,
                                                                               const __grid_constant__ CUtensorMap tmap_rows) {
  using R = FtRoles<G4>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  FtMisc& ms = *reinterpret_cast<FtMisc*>(smem + FS_MISC);
  volatile int* abort_flag = &ms.abort_flag;

  const int tid = threadIdx.x, lane = tid & 31;
  // provably warp-uniform role index: the issuing warps' branches stay converged for the compiler
  const int warp = tc::warp_index_uniform();
  pdl_wait();
  // rows of a causal chunk grow with their number: the longest first, so that the last wave ends together
  const int sp = blockIdx.x, r = (!G4 && !a.kv_len) ? a.m - 1 - (int)blockIdx.y : (int)blockIdx.y;
  int n;
  int64_t base = 0;
  if (G4) {
    n = a.kidx;
  } else {
    n = a.kv_len ? a.kv_len[r] : a.pos_start + r + 1;
    base = a.kv_base ? a.kv_base[r] : 0;
    if (a.ckv_rows > 0) n = (int)max((int64_t)0, min((int64_t)n, a.ckv_rows - base));   // never past the end of the cache
  }
  // split boundaries on tile granularity
  const int tiles_total = (n + FT_KEYS - 1) / FT_KEYS;
  const int tiles_per = (tiles_total + a.n_split - 1) / a.n_split;
  const int k0 = min(n, sp * tiles_per * FT_KEYS), k1 = min(n, (sp + 1) * tiles_per * FT_KEYS);
  const int n_tiles = (k1 - k0 + FT_KEYS - 1) / FT_KEYS;
  auto tile_keys = [&](int t) { return min(FT_KEYS, k1 - k0 - t * FT_KEYS); };
  auto whole = [&](int t) { return !G4 && tile_keys(t) == FT_KEYS; };       // arrives as one box

  if (tid == 0) {
#pragma unroll
    for (int b = 0; b < FT_NBUF; b++) {
      tc::mbar_init(&ms.k_full[b], R::LOAD_WARPS);
      tc::mbar_init(&ms.t_done[b], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; b++) {
      tc::mbar_init(&ms.s_full[b], 1);
      tc::mbar_init(&ms.s_free[b], 128);
      tc::mbar_init(&ms.p_full[b], 128);
    }
    tc::mbar_init(&ms.q_ready, 128);
    tc::mbar_fence_init();
    ms.abort_flag = 0;
    // The boxes of the first two tiles leave at once and fly while the queries are staged (in the third buffer).  The
    // byte count is raised without an arrival; the loader warps arrive later like for every tile.
    for (int t = 0; t < FT_NBUF - 1 && t < n_tiles; t++)
      if (whole(t)) {
        tc::mbar_expect_tx(&ms.k_full[t], FT_TILE);
        tma_load_tile(smem + FS_K + t * FT_TILE, &tmap_box, (int)(base + k0 + t * FT_KEYS), &ms.k_full[t]);
      }
  }
  // (not ahead of the barrier set-up and the first copies: there it cost a many-wave launch 4 %)
  if (warp == 0) tc::tmem_alloc(&ms.tmem, 512);
  if (n_tiles > 0) {
    // Q: channels 0-127 -> the swizzled A operand, the rest -> rows in the third tile buffer, from where the softmax
    // threads carry them into tensor memory.  All warps, every load of a thread in flight at once.
    constexpr int NI = (FT_HEADS * 64 + R::THREADS - 1) / R::THREADS;      // 16-byte pieces per thread
    const uint4* q = reinterpret_cast<const uint4*>(a.q_lat + (size_t)r * FT_HEADS * LATENT);
    uint4 qs[NI];
#pragma unroll
    for (int u = 0; u < NI; u++) {
      const int i = tid + u * R::THREADS;
      if (i < FT_HEADS * 64) qs[u] = q[i];
    }
#pragma unroll
    for (int u = 0; u < NI; u++) {
      const int i = tid + u * R::THREADS, h = i >> 6, c = i & 63;
      if (i < FT_HEADS * 64) {
        uint8_t* dst = c < FT_QS / 8 ? smem + FS_Q + tc::sw128_off(h, c, FT_HEADS * 128)
                                     : smem + FS_K + (FT_NBUF - 1) * FT_TILE + h * FT_QPITCH + (c - FT_QS / 8) * 16;
        *reinterpret_cast<uint4*>(dst) = qs[u];
      }
    }
    tc::fence_async_smem();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = ms.tmem;
  bool ok = true;

  if (warp >= 6) {
    // =========================== loaders: the key tiles ===========================
    const int lw = warp - 6;
    // copy u of a tile: key quad u / 8, channel block u % 8
    const int u0 = lw * R::COPIES + lane;
    const bool issuer = lane < R::COPIES;
    auto row_of = [&](int tile, int slot) -> int {         // cache row of a key slot, -1 = hole
      const int p = k0 + tile * FT_KEYS + slot;
      if (tile >= n_tiles || p >= k1) return -1;
      if (!G4) return (int)(base + p);
      int v;
      asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(a.raw_idx + (size_t)r * a.kidx + p));
      return v;
    };
    // gathered row numbers beyond the cache are holes
    auto in_cache = [&](int v) -> int { return (v < 0 || (a.ckv_rows > 0 && (int64_t)v >= a.ckv_rows)) ? -1 : v; };
    // Row numbers are fetched TWO tiles ahead with volatile loads, so that they are issued where they stand and not moved
    // down to their first use (the row list of a query is read once, from HBM).
    int qa[4], qb[4], ma[2] = {-1, -1}, mb[2] = {-1, -1};
    if (G4) {
#pragma unroll
      for (int e = 0; e < 4; e++) {
        qa[e] = issuer ? row_of(0, (u0 >> 3) * 4 + e) : -1;
        qb[e] = issuer ? row_of(1, (u0 >> 3) * 4 + e) : -1;
      }
      if (lw == 0) {
#pragma unroll
        for (int e = 0; e < 2; e++) { ma[e] = row_of(0, 32 * e + lane); mb[e] = row_of(1, 32 * e + lane); }
      }
    }
    for (int tile = 0; tile < n_tiles; tile++) {
      const int buf = tile % FT_NBUF;
      uint8_t* dst = smem + FS_K + buf * FT_TILE;
      int rows[4];
      unsigned long long mask = 0;
      if (G4) {
#pragma unroll
        for (int e = 0; e < 4; e++) {
          rows[e] = in_cache(qa[e]);
          qa[e] = qb[e];
          qb[e] = issuer ? row_of(tile + 2, (u0 >> 3) * 4 + e) : -1;
        }
        if (lw == 0) {
#pragma unroll
          for (int e = 0; e < 2; e++) {
            mask |= (unsigned long long)__ballot_sync(0xffffffffu, in_cache(ma[e]) >= 0) << (32 * e);
            ma[e] = mb[e];
            mb[e] = row_of(tile + 2, 32 * e + lane);
          }
        }
      } else {
        mask = ~0ull >> (FT_KEYS - tile_keys(tile));
      }
      // the buffer is free: its last P V is done; the third buffer held the queries first
      if (tile >= FT_NBUF) ok = tc::mbar_wait<FT_POLL_NS>(&ms.t_done[buf], (tile / FT_NBUF - 1) & 1, abort_flag, 5) && ok;
      else if (tile == FT_NBUF - 1) ok = tc::mbar_wait<FT_POLL_NS>(&ms.q_ready, 0, abort_flag, 4) && ok;
      if (lw == 0 && lane == 0) ms.mask[buf] = mask;
      if (whole(tile)) {
        if (lane == 0) {
          if (lw == 0 && tile >= FT_NBUF - 1) {
            tc::mbar_arrive_expect_tx(&ms.k_full[buf], FT_TILE);
            tma_load_tile(dst, &tmap_box, (int)(base + k0 + tile * FT_KEYS), &ms.k_full[buf]);
          } else {
            tc::mbar_arrive(&ms.k_full[buf]);            // nothing to add, or the box left at kernel entry
          }
        }
      } else {
        if (lane == 0) tc::mbar_arrive_expect_tx(&ms.k_full[buf], R::COPIES * 512);
        __syncwarp();
        if (issuer) {
          const int kq = u0 >> 3, blk = u0 & 7;
          if (!G4) {
#pragma unroll
            for (int e = 0; e < 4; e++) rows[e] = row_of(tile, kq * 4 + e);
          }
          tma_gather4_rows(dst + blk * FT_BLK + kq * 512, &tmap_rows, blk * 64, rows[0], rows[1], rows[2], rows[3], &ms.k_full[buf]);
        }
      }
    }
  } else if (warp >= 4) {
    // =========================== tensor-core issue (whole warp, one elected lane) ===========================
    // Every lane runs the loop, polls the barriers and computes the (warp-uniform) descriptors; the elected lane alone
    // issues (tc05.cuh).  A leader-only wait would split the warp into two groups that run this loop at different times
    // while the compiler, which sees only warp-uniform branch conditions here, keeps loop state in per-warp registers.
    // The two products have issuing warps of their own: S of tile t + 1 goes out as soon as its keys have landed and the S
    // buffer is free, whatever the state of tile t's softmax; P V of tile t follows its P.
    const uint32_t leader = tc::elect_one();
    auto wait_u = [&](uint64_t* bar, uint32_t parity, int code) {
      const bool done = tc::mbar_wait<FT_POLL_NS>(bar, parity, abort_flag, code);
      ok = __all_sync(0xffffffffu, done) != 0 && ok;
    };
    if (warp == 4) {
      const uint32_t idesc = tc::make_idesc(64, FT_KEYS, tc::FMT_F16, tc::FMT_F16, false, false);
      const uint64_t qd = tc::make_sdesc_sw128(tc::smem_u32(smem + FS_Q), 16, 1024);
      if (n_tiles > 0) wait_u(&ms.q_ready, 0, 11);
      for (int tile = 0; tile < n_tiles; tile++) {
        const int b = tile & 1, kb = tile % FT_NBUF;
        wait_u(&ms.k_full[kb], (tile / FT_NBUF) & 1, 1);
        if (tile >= 2) wait_u(&ms.s_free[b], ((tile - 2) >> 1) & 1, 2);
        tc::fence_after_sync();
        // keys as N in 1 KB atoms; 16 channels = 32 B inside the 128-byte row, 64 channels per block
        const uint64_t kd = tc::make_sdesc_sw128(tc::smem_u32(smem + FS_K + kb * FT_TILE), 16, 1024);
#pragma unroll
        for (int kk = 0; kk < LATENT / 16; kk++) {
          const uint64_t bd = tc::sdesc_advance(kd, (kk >> 2) * FT_BLK + (kk & 3) * 32);
          if (kk < FT_QS / 16)
            tc::mma_ws_f16_if(leader, tmem + FT_S + b * 32, tc::sdesc_advance(qd, (kk >> 2) * (FT_HEADS * 128) + (kk & 3) * 32), bd, idesc, kk > 0);
          else
            tc::mma_ws_f16_tmem_a_if(leader, tmem + FT_S + b * 32, tmem + FT_Q + (kk - FT_QS / 16) * 8, bd, idesc, true);
        }
        tc::mma_commit_if(leader, &ms.s_full[b]);
      }
    } else {
      const uint32_t idesc = tc::make_idesc(64, 256, tc::FMT_F16, tc::FMT_F16, false, true);
      for (int tile = 0; tile < n_tiles; tile++) {
        const int b = tile & 1, kb = tile % FT_NBUF;
        wait_u(&ms.p_full[b], (tile >> 1) & 1, 3);
        tc::fence_after_sync();
        const uint64_t pd = tc::make_sdesc_sw128(tc::smem_u32(smem + FS_P + b * FP_BYTES), 16, 1024);
        // V: N = 256 channels = four 64-channel blocks (leading offset), K = keys in 8-row atoms of 1 KB
        const uint64_t vd = tc::make_sdesc_sw128(tc::smem_u32(smem + FS_K + kb * FT_TILE), FT_BLK, 1024);
        const int steps = (tile_keys(tile) + 15) >> 4;    // a ragged tile ends early
#pragma unroll
        for (int nh = 0; nh < 2; nh++)
#pragma unroll
          for (int kk = 0; kk < FT_KEYS / 16; kk++)
            if (kk < steps)
              tc::mma_ws_f16_if(leader, tmem + FT_O + nh * 128, tc::sdesc_advance(pd, kk * 32),
                                tc::sdesc_advance(vd, nh * 4 * FT_BLK + kk * 2048), idesc, tile > 0 || kk > 0);
        tc::mma_commit_if(leader, &ms.t_done[kb]);
      }
    }
  } else {
    // =========================== softmax warps ===========================
    // S: head h < 64 sits in lanes h (keys 0-31) and h + 64 (keys 32-63).
    const int head = tid & 63, half = tid >> 6;
    const uint32_t lanes = (uint32_t)(warp * 32) << 16;
    const float sc2 = a.scale * LOG2E;
    if (n_tiles > 0) {
      const uint8_t* row = smem + FS_K + (FT_NBUF - 1) * FT_TILE + head * FT_QPITCH;
#pragma unroll 1
      for (int c0 = 0; c0 < (LATENT - FT_QS) / 2; c0 += 32) {
        uint32_t v[32];
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint4 w = *reinterpret_cast<const uint4*>(row + c0 * 4 + u * 16);
          v[4 * u] = w.x; v[4 * u + 1] = w.y; v[4 * u + 2] = w.z; v[4 * u + 3] = w.w;
        }
        tc::tmem_st32(tmem + FT_Q + c0 + lanes, v);
      }
      tc::tmem_st_wait();
      tc::fence_before_sync();
      tc::mbar_arrive(&ms.q_ready);
    }
    float m = -INFINITY, l = 0.f;
    for (int tile = 0; tile < n_tiles; tile++) {
      const int b = tile & 1, kb = tile % FT_NBUF;
      ok = tc::mbar_wait<FT_POLL_NS>(&ms.k_full[kb], (tile / FT_NBUF) & 1, abort_flag, 6) && ok;   // makes the tile's mask visible
      ok = tc::mbar_wait<FT_POLL_NS>(&ms.s_full[b], (tile >> 1) & 1, abort_flag, 7) && ok;
      tc::fence_after_sync();
      uint32_t sv[32];
      tc::tmem_ld32(tmem + FT_S + b * 32 + lanes, sv);
      tc::tmem_ld_wait();
      tc::fence_before_sync();
      tc::mbar_arrive(&ms.s_free[b]);
      const uint32_t mask = (uint32_t)(ms.mask[kb] >> (32 * half));
      float tmax = -INFINITY;
#pragma unroll
      for (int j = 0; j < 32; j++) {
        const float v = (mask >> j) & 1u ? __uint_as_float(sv[j]) * sc2 : -INFINITY;
        sv[j] = __float_as_uint(v);
        tmax = fmaxf(tmax, v);
      }
      ms.mx[b][tid] = tmax;
      // the two warps of these heads: named barriers 1 (warps 0, 2) and 2 (warps 1, 3)
      asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 1)) : "memory");
      tmax = fmaxf(tmax, ms.mx[b][tid ^ 64]);
      const bool move = tmax > m + RESCALE_THRESHOLD || (m == -INFINITY && tmax > -INFINITY);
      float alpha = 1.f;
      if (move) {
        alpha = m == -INFINITY ? 0.f : exp2f(m - tmax);
        m = tmax;
        l *= alpha;
      }
      if (tile > 0 && __any_sync(0xffffffffu, move)) {
        // rare: a head's reference max moved.  O is rescaled after the previous tile's P V has completed and before this
        // tile's is issued (it waits for p_full below); both warps of these heads take the same decision.
        ok = tc::mbar_wait<FT_POLL_NS>(&ms.t_done[(tile - 1) % FT_NBUF], ((tile - 1) / FT_NBUF) & 1, abort_flag, 8) && ok;
        tc::fence_after_sync();
#pragma unroll 1
        for (int c0 = 0; c0 < 256; c0 += 32) {
          uint32_t o[32];
          tc::tmem_ld32(tmem + FT_O + c0 + lanes, o);
          tc::tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 32; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
          tc::tmem_st32(tmem + FT_O + c0 + lanes, o);
        }
        tc::tmem_st_wait();
      }
      // the P buffer of this parity was last read by the P V of tile - 2
      if (tile >= 2) ok = tc::mbar_wait<FT_POLL_NS>(&ms.t_done[(tile - 2) % FT_NBUF], ((tile - 2) / FT_NBUF) & 1, abort_flag, 9) && ok;
      uint8_t* prow = smem + FS_P + b * FP_BYTES;
      const float mref = m == -INFINITY ? 0.f : m;         // every key so far is a hole: exp2(-inf) = 0 below
      float sum = 0.f;
#pragma unroll
      for (int u = 0; u < 4; u++) {
        uint4 w;
        uint32_t* wp = &w.x;
#pragma unroll
        for (int e = 0; e < 4; e++) {
          const float p0 = exp2f(__uint_as_float(sv[8 * u + 2 * e]) - mref), p1 = exp2f(__uint_as_float(sv[8 * u + 2 * e + 1]) - mref);
          sum += p0 + p1;
          const __half2 hp = __floats2half2_rn(p0, p1);
          wp[e] = *reinterpret_cast<const uint32_t*>(&hp);
        }
        *reinterpret_cast<uint4*>(prow + tc::sw128_off(head, half * 4 + u, FT_BLK)) = w;
      }
      l += sum;
      tc::fence_async_smem();
      tc::fence_before_sync();
      tc::mbar_arrive(&ms.p_full[b]);
    }
    // ---- epilogue: wait for the last P V, lay the rows out in the (now idle) tile buffers, hand them to the copy engine ----
    ms.l[tid] = l;
    if (n_tiles > 0) ok = tc::mbar_wait<FT_POLL_NS>(&ms.t_done[(n_tiles - 1) % FT_NBUF], ((n_tiles - 1) / FT_NBUF) & 1, abort_flag, 10) && ok;
    tc::fence_after_sync();
    asm volatile("bar.sync 3, 128;" ::: "memory");
    l += ms.l[tid ^ 64];
    const bool final_out = a.out != nullptr;
    const float f = l > 0.f ? (final_out ? 1.f / l : 1.f) : 0.f;
    const uint32_t row_bytes = LATENT * (final_out ? 2 : 4), pitch = row_bytes + 16;
    uint8_t* orow = smem + FS_K + head * pitch;
#pragma unroll 1
    for (int c0 = 0; c0 < 256; c0 += 32) {
      uint32_t o[32];
      if (n_tiles > 0) {
        tc::tmem_ld32(tmem + FT_O + c0 + lanes, o);
        tc::tmem_ld_wait();
      } else {
#pragma unroll
        for (int j = 0; j < 32; j++) o[j] = 0u;
      }
#pragma unroll
      for (int j = 0; j < 32; j++) o[j] = l > 0.f ? __float_as_uint(__uint_as_float(o[j]) * f) : 0u;
      const int ch = (c0 >> 7) * 256 + half * 128 + (c0 & 127);
      if (final_out) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
          uint4 w;
          uint32_t* wp = &w.x;
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const __half2 h2 = __floats2half2_rn(__uint_as_float(o[8 * u + 2 * e]), __uint_as_float(o[8 * u + 2 * e + 1]));
            wp[e] = *reinterpret_cast<const uint32_t*>(&h2);
          }
          *reinterpret_cast<uint4*>(orow + ch * 2 + u * 16) = w;
        }
      } else {
#pragma unroll
        for (int u = 0; u < 8; u++)
          *reinterpret_cast<uint4*>(orow + ch * 4 + u * 16) = make_uint4(o[4 * u], o[4 * u + 1], o[4 * u + 2], o[4 * u + 3]);
      }
    }
    tc::fence_async_smem();
    asm volatile("bar.sync 3, 128;" ::: "memory");
    const size_t rows = (size_t)a.m * FT_HEADS, rh = (size_t)r * FT_HEADS + head;
    if (half == 0 && ok && !*abort_flag) {
      char* dst = final_out ? reinterpret_cast<char*>(a.out + rh * LATENT) : reinterpret_cast<char*>(a.part_acc + ((size_t)sp * rows + rh) * LATENT);
      tc::bulk_s2g(dst, orow, row_bytes);
      tc::bulk_commit();
      if (!final_out) {
        a.part_m[(size_t)sp * rows + rh] = (m == -INFINITY || !(l > 0.f)) ? -INFINITY : m / LOG2E;
        a.part_l[(size_t)sp * rows + rh] = l;
      }
      tc::bulk_wait_read<0>();
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
  if (tid == 0 && ms.abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
}

int mla_flash_tc_auto_splits(int m, int n_keys) {
  // at most one CTA per SM (a second wave would double the time), at least two tiles per split, splits of equal tile counts
  const int sms = sm_count();
  const int tiles = (n_keys + FT_KEYS - 1) / FT_KEYS;
  int want = sms / (m > 0 ? m : 1);
  if (want > 256) want = 256;
  if (want < 1) want = 1;
  int tiles_per = (tiles + want - 1) / want;
  if (tiles_per < 2) tiles_per = 2;
  int n_split = (tiles + tiles_per - 1) / tiles_per;
  return n_split < 1 ? 1 : n_split;
}

typedef CUresult (*FtEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                               const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static FtEncodeFn ft_encode_fn() {
  static const FtEncodeFn fn = []() -> FtEncodeFn {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (getenv("HK_MLA_NO_TMA") == nullptr &&   // debug switch: no copy engine, i.e. the CUDA-core kernel
        cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      return (FtEncodeFn)p;
    return nullptr;
  }();
  return fn;
}

int mla_flash_tc_launch(const MlaArgs& a, cudaStream_t s) {
  FtEncodeFn encode = ft_encode_fn();
  if (a.n_heads != FT_HEADS || !encode) return HK_ERR_UNSUPPORTED;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(mla_flash_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(mla_flash_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM) != cudaSuccess)
      return HK_ERR_CUDA;
    attr_set[dev] = true;
  }
  // Tensor maps over the latent cache.  The row extent is the cache's row count when the caller gave it (the copy engine
  // zero-fills anything past the end), else an upper bound.
  alignas(64) CUtensorMap box, rows;
  memset(&box, 0, sizeof(box));
  memset(&rows, 0, sizeof(rows));
  const cuuint64_t extent = a.ckv_rows > 0 ? (cuuint64_t)a.ckv_rows : (cuuint64_t)1 << 31;
  const cuuint32_t ones[3] = {1, 1, 1};
  {
    const cuuint64_t dims[2] = {LATENT, extent};
    const cuuint64_t strides[1] = {LATENT * 2};
    const cuuint32_t b[2] = {64, 1};
    if (encode(&rows, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, (void*)a.ckv, dims, strides, b, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return HK_ERR_UNSUPPORTED;
  }
  if (!a.raw_idx) {
    const cuuint64_t dims[3] = {64, extent, 8};
    const cuuint64_t strides[2] = {LATENT * 2, 128};
    const cuuint32_t b[3] = {64, FT_KEYS, 8};
    if (encode(&box, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, (void*)a.ckv, dims, strides, b, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return HK_ERR_UNSUPPORTED;
  }
  const dim3 grid(a.n_split, a.m);
  const cudaError_t e =
      a.raw_idx ? pdl_launch(mla_flash_tc_kernel<true>, grid, dim3(FtRoles<true>::THREADS), FS_SMEM, s, a, device_status_ptr(), box, rows)
                : pdl_launch(mla_flash_tc_kernel<false>, grid, dim3(FtRoles<false>::THREADS), FS_SMEM, s, a, device_status_ptr(), box, rows);
  return e == cudaSuccess && cudaPeekAtLastError() == cudaSuccess ? HK_OK : HK_ERR_CUDA;
}

}  // namespace hk
