// Absorbed MLA flash attention over the 512-wide fp16 latent cache on the 5th-generation tensor
// cores: dense causal ranges and gathered (sparse) rows, decode and prefill rows, final output or
// split-KV partials.  One kernel serves helios::attn::mla_sparse_decode and
// helios::attn::mla_dense_prefill (reference: src/cuda/attn/attn.cu:394-699, scalar kernels, one
// block per (row, head) or head pair).  Causal chunks of some length go to mla_pair_tc_kernel (mla_pair_tc.cuh), two rows at a time.
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
//
// Many gathered rows (prefill) run on a persistent grid, one CTA per SM that walks rows: a row's own costs - its first loads,
// Q into tensor memory, O out - were 14 K cycles of the 75 K of 2,052 keys.  Here the next row's Q and keys come through the
// ring while the current row is in its last tiles, Q is a pseudo-tile of the ring that the softmax warps move while
// the row's last P V runs, and O leaves through the P buffers.
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
constexpr int FT_POLL_NS = 40;                    // poll back-off of the waiting warps
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_THRESHOLD = 8.0f;         // log2 units: P stays below 2^8, fine for fp16
// warps 0-3 softmax, Q into tensor memory and epilogue (a TMEM lane quarter each), 4 issues S = Q K^T, 5 issues O += P V, the
// others load tiles (dense ranges need more than one only for the ragged last tile).
constexpr int FT_LOAD_WARPS = 4, FT_THREADS = (6 + FT_LOAD_WARPS) * 32, FT_SLOTS = FT_KEYS / FT_LOAD_WARPS;   // key slots per loader warp

constexpr int FT_PAIR_KEYS = 700;                 // keys of a row, on average, from which on two rows of a chunk go to a pair of CTAs
constexpr int FT_MINI = 16;                       // keys of a tile in Q's place
constexpr int FT_MAX_CL = 16;                     // CTAs of a cluster
// Parts that a row's output channels are shared out in, a cluster each.  Four: a quarter of the product, of the accumulator and of the
// shares for each CTA (11 MLA layers of a decode step 285 us, 303 with two).
constexpr int FT_CS = 4, FT_CS_CH = LATENT / FT_CS;
constexpr uint32_t FT_CL_ROW = FT_CS_CH * 4;                            // a head's share: its channels, and 8 bytes (m, l) behind all heads
constexpr uint32_t FT_CL_STAGE = FT_HEADS * (FT_CL_ROW + 8);            // outgoing shares behind the incoming ones, in the idle ring
static_assert(2 * FT_CL_STAGE <= FT_NBUF * FT_TILE && FT_CL_STAGE % 16 == 0 && (FT_HEADS / FT_MAX_CL) * (FT_CL_ROW + 8) % 16 == 0, "exchange area");
static_assert(FT_CS_CH == 128, "a part is one N = 128 product of two 64-channel blocks, a half of it 64 columns of the accumulator");
// all threads of all CTAs of the cluster.  Relaxed: the barriers only tell that memory is no longer in use, the data that crosses CTAs is
// announced by mbarriers (.release: 1,000 cycles more each)
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.relaxed;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// the address of a shared-memory word in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t cluster_addr(uint32_t addr, int rank) {
  uint32_t r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}

struct FtMisc {
  uint64_t full[FT_NBUF], free[FT_NBUF];          // ring slot (a key tile or a row's Q): landed, may be overwritten
  uint64_t s_full[2], s_free[2], p_full[2], pv_done[2];   // per tile parity
  uint64_t q_ready, o_free;                       // per row
  uint64_t full_mini;
  uint8_t mask[FT_NBUF + 1][FT_KEYS / 8];         // valid key slots of the tile in the ring slot; [FT_NBUF]: the ragged tile in Q's place
  float mx[2][128];                               // tile maxima, by softmax thread and tile parity
  float l[128];
  uint32_t tmem;
  int abort_flag;
};
static_assert(sizeof(FtMisc) <= 2048, "misc area");

// One work item: a row and a key split (cluster form: and a part of the output channels).
struct FtItem {
  int r, sp, cs, k0, k1, n_tiles;                 // cs: part of the output channels (cluster form)
  bool mini;                                      // cluster form: the ragged last tile comes first, from memory of its own
  int64_t base;
  __device__ __forceinline__ int keys(int t) const { return min(FT_KEYS, k1 - k0 - t * FT_KEYS); }
  __device__ __forceinline__ int nth(int i) const { return mini ? (i ? i - 1 : n_tiles - 1) : i; }   // the tile that is i-th in turn
};
template <bool G4, bool CL>
__device__ __forceinline__ FtItem ft_item(const MlaArgs& a, int idx) {
  FtItem it;
  it.sp = idx % a.n_split;
  it.r = idx / a.n_split;
  it.cs = 0;
  if (CL) {
    it.cs = it.r % FT_CS;
    it.r /= FT_CS;
  }
  // rows of a causal chunk grow with their number: the longest first, so that the CTAs end together
  if (!G4 && !a.kv_len) it.r = a.m - 1 - it.r;
  int n;
  it.base = 0;
  if (G4) {
    n = a.kidx;
  } else {
    n = a.kv_len ? a.kv_len[it.r] : a.pos_start + it.r + 1;
    it.base = a.kv_base ? a.kv_base[it.r] : 0;
    if (a.ckv_rows > 0) n = (int)max((int64_t)0, min((int64_t)n, a.ckv_rows - it.base));   // never past the end of the cache
  }
  // split boundaries on tile granularity
  const int tiles = (n + FT_KEYS - 1) / FT_KEYS, per = (tiles + a.n_split - 1) / a.n_split;
  // (cluster form: a fixed number of splits, so the tiles are shared out evenly)
  it.k0 = min(n, (CL ? tiles * it.sp / a.n_split : it.sp * per) * FT_KEYS);
  it.k1 = min(n, (CL ? tiles * (it.sp + 1) / a.n_split : (it.sp + 1) * per) * FT_KEYS);
  it.n_tiles = (it.k1 - it.k0 + FT_KEYS - 1) / FT_KEYS;
  // 2,052 keys are 32 tiles and 4 keys more.  A split with a third tile of up to 16 keys would have to wait for a ring slot: that
  // tile lies where Q's 128 channels are otherwise (16 key rows a block) and is attended to while the whole ones arrive.
  it.mini = CL && it.n_tiles > 2 && it.keys(it.n_tiles - 1) <= FT_MINI;
  return it;
}

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
// Executed by the whole warp with warp-uniform operands, issued by the lane with leader != 0: the eight copies of a key quad
// differ in two numbers.  Issued lane by lane (each lane its own copy) a copy cost about 90 cycles of operand moves, 1,440 per
// warp and tile, and the three-slot ring stood still for them: 2,110 cycles per tile of gathered rows against 1,760 dense.
__device__ __forceinline__ void tma_gather4_rows(uint32_t leader, uint32_t smem_dst, const CUtensorMap* tmap, int channel, int r0, int r1,
                                                 int r2, int r3, uint32_t bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %8, 0;\n\t"
      "@q cp.async.bulk.tensor.2d.shared::cluster.global.tile::gather4.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, %6}], [%7];\n\t}" ::"r"(
          smem_dst),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(channel), "r"(r0), "r"(r1), "r"(r2), "r"(r3), "r"(bar), "r"(leader)
      : "memory");
}

// G4: gathered rows (raw_idx); otherwise dense ranges.  tmap_box: 3-D map of the cache, tmap_rows: 2-D map of the cache for
// gather4, tmap_q: the queries as tmap_box, tmap_o: 2-D map of the final output.
// CL: cluster form for few rows of few keys (a decode step's gathered rows).  The splits of a row are the CTAs of a cluster, which merge
// their partials through distributed shared memory and write the final output: no partials in memory, no second kernel.  The row's
// output channels are shared out over FT_CS such clusters, each of which computes the scores for itself.
// What bounds it is latency, one thing after another on 64 SMs: row numbers 1,200 cycles, gathered keys 2,800, two tiles of S, softmax and
// P V 3,800, laying out and the barrier of the cluster 1,700, the shares 2,200, the merge 1,600.  2,052 gathered rows of one query 10.8 ->
// 9.2 us; MLA layer of one token at 5,001 32.1 -> 28.9, selection and attention at 262,144 23.8 -> 21.8.
template <bool G4, bool CL>
__global__ __launch_bounds__(FT_THREADS, 1) void mla_flash_tc_kernel(
    MlaArgs a, int* __restrict__ status, const __grid_constant__ CUtensorMap tmap_box, const __grid_constant__ CUtensorMap tmap_rows,
    const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_o) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  FtMisc& ms = *reinterpret_cast<FtMisc*>(smem + FS_MISC);
  volatile int* abort_flag = &ms.abort_flag;

  const int tid = threadIdx.x, lane = tid & 31;
  // provably warp-uniform role index: the issuing warps' branches stay converged for the compiler
  const int warp = tc::warp_index_uniform();
  const int n_items = CL ? gridDim.x : a.n_split * a.m, step = gridDim.x;
  // A CTA with one item of at most two tiles (a decode split) never needs Q's ring slot back: S reads Q from there, and the
  // 0.6 us of moving it are saved.  In the cluster form Q always stays and the other two slots serve all tiles.
  bool direct_q = CL;
  if (tid == 0) {
#pragma unroll
    for (int b = 0; b < FT_NBUF; b++) {
      tc::mbar_init(&ms.full[b], FT_LOAD_WARPS);
      tc::mbar_init(&ms.free[b], 1);
    }
#pragma unroll
    for (int b = 0; b < 2; b++) {
      tc::mbar_init(&ms.s_full[b], 1);
      tc::mbar_init(&ms.s_free[b], 128);
      tc::mbar_init(&ms.p_full[b], 128);
      tc::mbar_init(&ms.pv_done[b], 1);
    }
    if (CL) tc::mbar_init(&ms.full_mini, FT_LOAD_WARPS);
    tc::mbar_init(&ms.q_ready, CL ? 1 : 128);              // (cluster form: the shares of the other splits)
    tc::mbar_init(&ms.o_free, 128);
    tc::mbar_fence_init();
    if (CL) tc::mbar_arrive_expect_tx(&ms.q_ready, FT_CL_STAGE);
    ms.abort_flag = 0;
  }
  if (warp == 0) tc::tmem_alloc(&ms.tmem, 512);
  pdl_wait();
  if (!CL && step >= n_items) direct_q = ft_item<G4, CL>(a, blockIdx.x).n_tiles < FT_NBUF;
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = ms.tmem;
  bool ok = true;

  // Every role walks the same items and counts the same way: u = ring slots used so far, g = key tiles, q = rows with keys.
  // Ring slot of use u (the i-th tile of the item) and the earlier uses of that slot; cluster form: Q keeps slot 0.
  auto slot_of = [](const FtItem& it, uint32_t u, int i) -> int { return !CL ? u % FT_NBUF : it.mini && i == 0 ? FT_NBUF : 1 + ((i - it.mini) & 1); };
  auto turn_of = [](const FtItem& it, uint32_t u, int i) -> uint32_t { return !CL ? u / FT_NBUF : it.mini && i == 0 ? 0 : (i - it.mini) >> 1; };
  auto full_of = [&](int b) -> uint64_t* { return CL && b == FT_NBUF ? &ms.full_mini : &ms.full[b]; };
  auto tile_at = [](int b) -> uint32_t { return CL && b == FT_NBUF ? FS_Q : FS_K + b * FT_TILE; };
  auto blk_of = [](int b) -> uint32_t { return CL && b == FT_NBUF ? FT_MINI * 128 : FT_BLK; };   // bytes of a 64-channel block
  if (warp >= 6) {
    // =========================== loaders: per row its Q, then its key tiles ===========================
    const int lw = warp - 6;
    const uint32_t leader = tc::elect_one();
    // cache row of key slot lw * SLOTS + lane of a tile, -1 = hole; volatile, so that a look-ahead load is issued where it stands
    auto row_of = [&](const FtItem& it, int tile) -> int {
      const int p = it.k0 + tile * FT_KEYS + lw * FT_SLOTS + lane;
      if (lane >= FT_SLOTS || p >= it.k1) return -1;
      if (!G4) return (int)(it.base + p);
      int v;
      asm volatile("ld.global.nc.s32 %0, [%1];" : "=r"(v) : "l"(a.raw_idx + (size_t)it.r * a.kidx + p));
      return v;
    };
    // gathered row numbers beyond the cache are holes
    auto in_cache = [&](int v) -> int { return (v < 0 || (a.ckv_rows > 0 && (int64_t)v >= a.ckv_rows)) ? -1 : v; };
    // Gathered row numbers are fetched two tiles ahead (the row list of a query is read once, from HBM), across rows.
    int cur = -1, nxt = -1, ahead_item = blockIdx.x, ahead_tile = 0;
    FtItem ahead = ft_item<G4, CL>(a, ahead_item);
    auto fetch = [&]() -> int {
      if (!G4 || ahead_item >= n_items || ahead.n_tiles == 0) return -1;   // (gathered rows: every item has the same keys)
      const int v = row_of(ahead, ahead.nth(ahead_tile));
      if (++ahead_tile == ahead.n_tiles) {
        ahead_tile = 0;
        ahead_item += step;
        if (ahead_item < n_items) ahead = ft_item<G4, CL>(a, ahead_item);
      }
      return v;
    };
    if (G4) {
      cur = fetch();
      nxt = fetch();
    }
    uint32_t u = 0;
    auto next_slot = [&](const FtItem& it, int i) -> int { // waits until the slot may be overwritten (i < 0: for Q)
      const int b = CL && i < 0 ? 0 : slot_of(it, u, i);
      const uint32_t turn = CL && i < 0 ? 0 : turn_of(it, u, i);
      if (turn > 0) ok = tc::mbar_wait<FT_POLL_NS>(&ms.free[b], (turn - 1) & 1, abort_flag, 5) && ok;
      u++;
      return b;
    };
    for (int idx = blockIdx.x; idx < n_items; idx += step) {
      const FtItem it = ft_item<G4, CL>(a, idx);
      if (it.n_tiles == 0) continue;
      {
        const int b = next_slot(it, -1);
        if (lane == 0) {
          if (lw == 0) {
            tc::mbar_arrive_expect_tx(&ms.full[b], FT_TILE);
            tma_load_tile(smem + FS_K + b * FT_TILE, &tmap_q, it.r * FT_HEADS, &ms.full[b]);
          } else {
            tc::mbar_arrive(&ms.full[b]);
          }
        }
      }
      for (int i = 0; i < it.n_tiles; i++) {
        const int tile = it.nth(i);
        int row;
        if (G4) {
          row = in_cache(cur);
          cur = nxt;
          nxt = fetch();
        } else {
          row = row_of(it, tile);
        }
        const uint32_t valid = __ballot_sync(0xffffffffu, row >= 0);
        const int b = next_slot(it, i);
        if (lane < FT_SLOTS / 8) ms.mask[b][lw * (FT_SLOTS / 8) + lane] = (uint8_t)(valid >> (8 * lane));
        __syncwarp();
        if (!G4 && it.keys(tile) == FT_KEYS) {             // a whole tile of a dense range: one box
          if (lane == 0) {
            if (lw == 0) {
              tc::mbar_arrive_expect_tx(&ms.full[b], FT_TILE);
              tma_load_tile(smem + FS_K + b * FT_TILE, &tmap_box, (int)(it.base + it.k0 + tile * FT_KEYS), &ms.full[b]);
            } else {
              tc::mbar_arrive(&ms.full[b]);
            }
          }
        } else {
          const bool none = CL && b == FT_NBUF && lw > 0;  // a ragged tile in Q's place has the first warp's key slots only
          if (lane == 0) {
            if (none) tc::mbar_arrive(full_of(b));
            else tc::mbar_arrive_expect_tx(full_of(b), FT_SLOTS * LATENT * 2);
          }
          __syncwarp();
          if (none) continue;
          const uint32_t dst = tc::smem_u32(smem) + tile_at(b) + lw * FT_SLOTS * 128, bar = tc::smem_u32(full_of(b)), blk_bytes = blk_of(b);
#pragma unroll
          for (int j = 0; j < FT_SLOTS / 4; j++) {
            const int r0 = __shfl_sync(0xffffffffu, row, 4 * j), r1 = __shfl_sync(0xffffffffu, row, 4 * j + 1);
            const int r2 = __shfl_sync(0xffffffffu, row, 4 * j + 2), r3 = __shfl_sync(0xffffffffu, row, 4 * j + 3);
#pragma unroll
            for (int blk = 0; blk < 8; blk++)
              tma_gather4_rows(leader, dst + blk * blk_bytes + j * 512, &tmap_rows, blk * 64, r0, r1, r2, r3, bar);
          }
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
    uint32_t u = 0, g = 0, q = 0;
    if (warp == 4) {
      const uint32_t idesc = tc::make_idesc(64, FT_KEYS, tc::FMT_F16, tc::FMT_F16, false, false);
      // Addresses pass through an empty asm where their descriptors are built: the compiler would otherwise keep 32
      // loop-invariant descriptors per operand in registers and spill in the softmax loop.
      auto desc = [](const uint8_t* p) {
        uint32_t addr = tc::smem_u32(p);
        asm volatile("" : "+r"(addr));
        return tc::make_sdesc_sw128(addr, 16, 1024);
      };
      for (int idx = blockIdx.x; idx < n_items; idx += step) {
        const FtItem it = ft_item<G4, CL>(a, idx);
        const int n_tiles = it.n_tiles;
        if (n_tiles == 0) continue;
        if (direct_q) wait_u(&ms.full[0], 0, 15);
        else wait_u(&ms.q_ready, q & 1, 13);
        u++;                                               // the row's Q
        q++;
        for (int tile = 0; tile < n_tiles; tile++, u++, g++) {
          const int b = g & 1, kb = slot_of(it, u, tile);
          wait_u(full_of(kb), turn_of(it, u, tile) & 1, 1);
          if (g >= 2) wait_u(&ms.s_free[b], ((g - 2) >> 1) & 1, 2);
          tc::fence_after_sync();
          // keys as N in 1 KB atoms; 16 channels = 32 B inside the 128-byte row, 64 channels per block
          const uint64_t kd = desc(smem + tile_at(kb)), qd = desc(smem + (direct_q ? FS_K : FS_Q));
          const uint32_t kblk = blk_of(kb);
          if (direct_q) {
#pragma unroll
            for (int kk = 0; kk < LATENT / 16; kk++) {
              // (a ragged tile's columns past its keys are whatever lies there: masked)
              tc::mma_ws_f16_if(leader, tmem + FT_S + b * 32, tc::sdesc_advance(qd, (kk >> 2) * FT_BLK + (kk & 3) * 32),
                                tc::sdesc_advance(kd, (kk >> 2) * kblk + (kk & 3) * 32), idesc, kk > 0);
            }
          } else
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
      }
    } else {
      const uint32_t idesc = tc::make_idesc(64, 256, tc::FMT_F16, tc::FMT_F16, false, true);
      for (int idx = blockIdx.x; idx < n_items; idx += step) {
        const FtItem it = ft_item<G4, CL>(a, idx);
        if (it.n_tiles == 0) continue;
        u++;
        for (int tile = 0; tile < it.n_tiles; tile++, u++, g++) {
          const int b = g & 1, kb = slot_of(it, u, tile);
          wait_u(&ms.p_full[b], (g >> 1) & 1, 3);
          if (tile == 0 && q > 0) wait_u(&ms.o_free, (q - 1) & 1, 14);   // the row before has left the accumulator
          tc::fence_after_sync();
          const uint64_t pd = tc::make_sdesc_sw128(tc::smem_u32(smem + FS_P + b * FP_BYTES), 16, 1024);
          // V: N = 256 channels = four 64-channel blocks (leading offset), K = keys in 8-row atoms of 1 KB
          const uint64_t vd = tc::make_sdesc_sw128(tc::smem_u32(smem + tile_at(kb)), blk_of(kb), 1024);
          const int steps = (it.keys(it.nth(tile)) + 15) >> 4;   // a ragged tile ends early
          if (CL) {                                        // one product of this cluster's channels
            const uint32_t id = tc::make_idesc(64, FT_CS_CH, tc::FMT_F16, tc::FMT_F16, false, true);
            const uint64_t vc = tc::sdesc_advance(vd, it.cs * (FT_CS_CH / 64) * blk_of(kb));
#pragma unroll
            for (int kk = 0; kk < FT_KEYS / 16; kk++)
              if (kk < steps)
                tc::mma_ws_f16_if(leader, tmem + FT_O, tc::sdesc_advance(pd, kk * 32), tc::sdesc_advance(vc, kk * 2048), id, tile > 0 || kk > 0);
          } else
#pragma unroll
          for (int nh = 0; nh < 2; nh++)
#pragma unroll
            for (int kk = 0; kk < FT_KEYS / 16; kk++)
              if (kk < steps)
                tc::mma_ws_f16_if(leader, tmem + FT_O + nh * 128, tc::sdesc_advance(pd, kk * 32),
                                  tc::sdesc_advance(vd, nh * 4 * FT_BLK + kk * 2048), idesc, tile > 0 || kk > 0);
          tc::mma_commit_if(leader, &ms.pv_done[b]);
          if (!CL || kb < FT_NBUF) tc::mma_commit_if(leader, &ms.free[kb]);
        }
        q++;
      }
    }
  } else {
    // =========================== softmax warps ===========================
    // S: head h < 64 sits in lanes h (keys 0-31) and h + 64 (keys 32-63).
    const int head = tid & 63, half = tid >> 6;
    const uint32_t lanes = (uint32_t)(warp * 32) << 16;
    const float sc2 = a.scale * LOG2E;
    const bool final_out = a.out != nullptr;
    uint32_t u = 0, g = 0;
    auto wait_pv = [&](uint32_t tile_g, int code) { ok = tc::mbar_wait<FT_POLL_NS>(&ms.pv_done[tile_g & 1], (tile_g >> 1) & 1, abort_flag, code) && ok; };
    // The row's Q: ring slot -> shared-memory operand (channels 0-127, the same layout) and tensor memory.  The products that
    // read the row before have completed: these warps have seen its last S.
    auto move_q = [&]() {
      const int b = u % FT_NBUF;
      ok = tc::mbar_wait<FT_POLL_NS>(&ms.full[b], (u / FT_NBUF) & 1, abort_flag, 11) && ok;
      tc::fence_after_sync();
      const uint8_t* src = smem + FS_K + b * FT_TILE;
#pragma unroll
      for (int i = 0; i < (int)(FT_QS * FT_HEADS * 2 / 16 / 128); i++)
        reinterpret_cast<uint4*>(smem + FS_Q)[tid + 128 * i] = reinterpret_cast<const uint4*>(src)[tid + 128 * i];
#pragma unroll 1
      for (int j = FT_QS / 64; j < 8; j++) {
        uint32_t v[32];
#pragma unroll
        for (int c = 0; c < 8; c++) {
          const uint4 w = *reinterpret_cast<const uint4*>(src + j * FT_BLK + head * 128 + ((c ^ (head & 7)) << 4));
          v[4 * c] = w.x; v[4 * c + 1] = w.y; v[4 * c + 2] = w.z; v[4 * c + 3] = w.w;
        }
        tc::tmem_st32(tmem + FT_Q + (j - FT_QS / 64) * 32 + lanes, v);
      }
      tc::tmem_st_wait();
      tc::fence_async_smem();
      tc::fence_before_sync();
      tc::mbar_arrive(&ms.q_ready);
      asm volatile("bar.sync 3, 128;" ::: "memory");
      if (tid == 0) tc::mbar_arrive(&ms.free[b]);
      u++;
    };
    auto next_row = [&](int idx) {                         // the first item from idx on that has keys
      while (idx < n_items && ft_item<G4, CL>(a, idx).n_tiles == 0) idx += step;
      return idx;
    };
    int q_item = next_row(blockIdx.x);                     // the row whose Q is moved next
    if (direct_q) u = 1;
    else if (q_item < n_items) move_q();
    for (int idx = blockIdx.x; idx < n_items; idx += step) {
      const FtItem it = ft_item<G4, CL>(a, idx);
      float m = -INFINITY, l = 0.f;
      for (int tile = 0; tile < it.n_tiles; tile++, u++, g++) {
        const int b = g & 1, kb = slot_of(it, u, tile);
        ok = tc::mbar_wait<FT_POLL_NS>(full_of(kb), turn_of(it, u, tile) & 1, abort_flag, 6) && ok;   // makes the tile's mask visible
        ok = tc::mbar_wait<FT_POLL_NS>(&ms.s_full[b], (g >> 1) & 1, abort_flag, 7) && ok;
        tc::fence_after_sync();
        uint32_t sv[32];
        tc::tmem_ld32(tmem + FT_S + b * 32 + lanes, sv);
        tc::tmem_ld_wait();
        tc::fence_before_sync();
        tc::mbar_arrive(&ms.s_free[b]);
        const uint32_t mask = *reinterpret_cast<const uint32_t*>(&ms.mask[kb][4 * half]);
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
          wait_pv(g - 1, 8);
          tc::fence_after_sync();
#pragma unroll 1
          for (int c0 = 0; c0 < (CL ? FT_CS_CH / 2 : 256); c0 += 32) {
            uint32_t o[32];
            tc::tmem_ld32(tmem + FT_O + c0 + lanes, o);
            tc::tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 32; j++) o[j] = __float_as_uint(__uint_as_float(o[j]) * alpha);
            tc::tmem_st32(tmem + FT_O + c0 + lanes, o);
          }
          tc::tmem_st_wait();
        }
        // the P buffer of this parity was last read by the P V two tiles ago (a row's first two tiles: its predecessor's
        // epilogue has waited for all of them)
        if (tile >= 2) wait_pv(g - 2, 9);
        uint8_t* prow = smem + FS_P + b * FP_BYTES;
        const float mref = m == -INFINITY ? 0.f : m;       // every key so far is a hole: exp2(-inf) = 0 below
        float sum = 0.f;
#pragma unroll
        for (int v = 0; v < 4; v++) {
          uint4 w;
          uint32_t* wp = &w.x;
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float p0 = exp2f(__uint_as_float(sv[8 * v + 2 * e]) - mref), p1 = exp2f(__uint_as_float(sv[8 * v + 2 * e + 1]) - mref);
            sum += p0 + p1;
            const __half2 hp = __floats2half2_rn(p0, p1);
            wp[e] = *reinterpret_cast<const uint32_t*>(&hp);
          }
          *reinterpret_cast<uint4*>(prow + tc::sw128_off(head, half * 4 + v, FT_BLK)) = w;
        }
        l += sum;
        tc::fence_async_smem();
        tc::fence_before_sync();
        tc::mbar_arrive(&ms.p_full[b]);
      }
      // ---- epilogue of the row ----
      ms.l[tid] = l;
      if (it.n_tiles > 0) {
        q_item = next_row(q_item + step);
        if (q_item < n_items) move_q();
        wait_pv(g - 1, 10);
      }
      tc::fence_after_sync();
      asm volatile("bar.sync 3, 128;" ::: "memory");
      l += ms.l[tid ^ 64];
      const float f = l > 0.f ? (final_out && !CL ? 1.f / l : 1.f) : 0.f;
      if (CL) cluster_arrive();                            // this CTA's ring is idle
      auto load_o = [&](int c0, uint32_t (&o)[32]) {       // 32 of this thread's 256 channels, weighed
        if (it.n_tiles > 0) {
          tc::tmem_ld32(tmem + FT_O + c0 + lanes, o);
          tc::tmem_ld_wait();
        }
#pragma unroll
        for (int j = 0; j < 32; j++) o[j] = l > 0.f ? __float_as_uint(__uint_as_float(o[j]) * f) : 0u;
      };
      if (CL) {
        // The accumulator goes to the cluster's CTAs by heads: CTA j merges n_h of them.  It is laid out by destination in the idle
        // ring - n_h heads of the cluster's channels (16-byte chunk c of head h at c ^ (h % 8)), then their (m, l) - and leaves as one
        // bulk copy per CTA (16-byte remote stores: 3.6 us for 32 KB).
        const int n_h = FT_HEADS / a.n_split, row = FT_CL_ROW, share = n_h * (row + 8), j = head / n_h;
        uint8_t* const out = smem + FS_K + FT_CL_STAGE + j * share;
#pragma unroll 1
        for (int c0 = 0; c0 < FT_CS_CH / 2; c0 += 32) {
          uint32_t o[32];
          load_o(c0, o);
          const int lc = half * (FT_CS_CH / 2) + c0;       // channel within the cluster's part
#pragma unroll
          for (int v = 0; v < 8; v++)
            *reinterpret_cast<uint4*>(out + (head - j * n_h) * row + ((((lc >> 2) + v) ^ (head & 7)) << 4)) =
                make_uint4(o[4 * v], o[4 * v + 1], o[4 * v + 2], o[4 * v + 3]);
        }
        if (half == 0) *reinterpret_cast<float2*>(out + n_h * row + (head - j * n_h) * 8) = make_float2(l > 0.f ? m : -INFINITY, l);
        tc::fence_before_sync();
        tc::fence_async_smem();
        asm volatile("bar.sync 3, 128;" ::: "memory");
        cluster_wait();                                    // and so are the others'
        if (tid < a.n_split)
          asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                           cluster_addr(tc::smem_u32(smem + FS_K) + it.sp * share, tid)),
                       "r"(tc::smem_u32(smem + FS_K + FT_CL_STAGE) + tid * share), "r"(share), "r"(cluster_addr(tc::smem_u32(&ms.q_ready), tid))
                       : "memory");
      } else if (final_out) {
        // Four rounds of 2 x 64 channels through the P buffers: channels 256 (c0 / 128) + 128 half + c0 % 128 ... of all heads
        // as a swizzled box each.
#pragma unroll 1
        for (int c0 = 0; c0 < 256; c0 += 64) {
          uint8_t* box = smem + FS_P + half * FP_BYTES;
          if (tid == 0) tc::bulk_wait_read<0>();           // the boxes of the round before have left
          asm volatile("bar.sync 3, 128;" ::: "memory");
#pragma unroll
          for (int hc = 0; hc < 2; hc++) {
            uint32_t o[32];
            load_o(c0 + 32 * hc, o);
#pragma unroll
            for (int v = 0; v < 4; v++) {
              uint4 w;
              uint32_t* wp = &w.x;
#pragma unroll
              for (int e = 0; e < 4; e++) {
                const __half2 h2 = __floats2half2_rn(__uint_as_float(o[8 * v + 2 * e]), __uint_as_float(o[8 * v + 2 * e + 1]));
                wp[e] = *reinterpret_cast<const uint32_t*>(&h2);
              }
              *reinterpret_cast<uint4*>(box + tc::sw128_off(head, hc * 4 + v, FT_BLK)) = w;
            }
          }
          tc::fence_async_smem();
          asm volatile("bar.sync 3, 128;" ::: "memory");
          if (tid == 0 && ok && !*abort_flag) {
#pragma unroll
            for (int hf = 0; hf < 2; hf++)
              asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&tmap_o),
                           "r"((c0 >> 7) * 256 + hf * 128 + (c0 & 127)), "r"(it.r * FT_HEADS), "r"(tc::smem_u32(smem + FS_P + hf * FP_BYTES))
                           : "memory");
            tc::bulk_commit();
          }
        }
        tc::fence_before_sync();
        if (it.n_tiles > 0) tc::mbar_arrive(&ms.o_free);
        if (tid == 0) tc::bulk_wait_read<0>();
        asm volatile("bar.sync 3, 128;" ::: "memory");     // P may be written again
      } else {
        // a partial (the CTA's only item): fp32 rows in the idle ring, one bulk copy per head
        const uint32_t pitch = LATENT * 4 + 16;
        uint8_t* orow = smem + FS_K + head * pitch;
#pragma unroll 1
        for (int c0 = 0; c0 < 256; c0 += 32) {
          uint32_t o[32];
          load_o(c0, o);
          const int ch = (c0 >> 7) * 256 + half * 128 + (c0 & 127);
#pragma unroll
          for (int v = 0; v < 8; v++)
            *reinterpret_cast<uint4*>(orow + ch * 4 + v * 16) = make_uint4(o[4 * v], o[4 * v + 1], o[4 * v + 2], o[4 * v + 3]);
        }
        tc::fence_async_smem();
        asm volatile("bar.sync 3, 128;" ::: "memory");
        const size_t rows = (size_t)a.m * FT_HEADS, rh = (size_t)it.r * FT_HEADS + head;
        if (half == 0 && ok && !*abort_flag) {
          tc::bulk_s2g(a.part_acc + ((size_t)it.sp * rows + rh) * LATENT, orow, LATENT * 4);
          tc::bulk_commit();
          a.part_m[(size_t)it.sp * rows + rh] = (m == -INFINITY || !(l > 0.f)) ? -INFINITY : m / LOG2E;
          a.part_l[(size_t)it.sp * rows + rh] = l;
          tc::bulk_wait_read<0>();
        }
      }
    }
  }
  if (CL) {
    if (warp >= 4) {
      cluster_arrive();
      cluster_wait();
    }
    ok = tc::mbar_wait(&ms.q_ready, 0, abort_flag, 16) && ok;   // every split's share of this CTA's heads has arrived
    cluster_arrive();
    const FtItem it = ft_item<G4, CL>(a, blockIdx.x);
    const int n_h = FT_HEADS / a.n_split, row = FT_CL_ROW, share = n_h * (row + 8), chunks = row / 16;
    if (!*abort_flag) {
      for (int i = tid; i < n_h * chunks; i += FT_THREADS) {
        const int h = i / chunks, c = i - h * chunks, head = it.sp * n_h + h;
        const uint8_t* part = smem + FS_K;
        const uint8_t* ml = part + n_h * row + h * 8;
        float gm = -INFINITY, gl = 0.f;
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        // short loops: this code runs once, from a cold instruction cache (unrolled sixteen times 3,100 cycles)
#pragma unroll 4
        for (int sp = 0; sp < a.n_split; sp++) gm = fmaxf(gm, *reinterpret_cast<const float*>(ml + sp * share));
        if (gm == -INFINITY) gm = 0.f;
        const uint8_t* src = part + h * row + ((c ^ (head & 7)) << 4);
#pragma unroll 4
        for (int sp = 0; sp < a.n_split; sp++) {
          const float2 x = *reinterpret_cast<const float2*>(ml + sp * share);
          const float4 v = *reinterpret_cast<const float4*>(src + sp * share);
          const float w = exp2f(x.x - gm);                 // no keys: 0
          gl = fmaf(w, x.y, gl);
          o.x = fmaf(w, v.x, o.x); o.y = fmaf(w, v.y, o.y); o.z = fmaf(w, v.z, o.z); o.w = fmaf(w, v.w, o.w);
        }
        const float inv = gl > 0.f ? 1.f / gl : 0.f;
        const __half2 h0 = __floats2half2_rn(o.x * inv, o.y * inv), h1 = __floats2half2_rn(o.z * inv, o.w * inv);
        uint2 w;
        w.x = *reinterpret_cast<const uint32_t*>(&h0);
        w.y = *reinterpret_cast<const uint32_t*>(&h1);
        *reinterpret_cast<uint2*>(a.out + ((size_t)it.r * FT_HEADS + head) * LATENT + it.cs * FT_CS_CH + c * 4) = w;
      }
    }
    cluster_wait();                                        // nobody copies from this CTA's memory any more
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 0) tc::tmem_dealloc(tmem, 512);
  if (tid == 0 && ms.abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
}

}  // namespace hk
#include "mla_pair_tc.cuh"
namespace hk {

int mla_flash_tc_auto_splits(int m, int n_keys) {
  // At most one CTA per SM (a second wave would double the time), at least two tiles per split, splits of equal tile counts.  With
  // the merge, 1 / 2 / 3 tiles per split, us: 2,052 gathered rows of one query 12.1 / 11.3 / 12.7, of four 16.9 / 12.6 / 13.5 (more
  // partials to write and merge); dense, one row over 2,048 keys 11.8 / 11.2 / 12.7, over 8,192 15.4 / 13.6 / 14.9.
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

static int ft_prepare() {
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(mla_flash_tc_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(mla_flash_tc_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(mla_flash_tc_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(mla_flash_tc_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(mla_pair_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)FS_SMEM) != cudaSuccess ||
        cudaFuncSetAttribute(mla_flash_tc_kernel<false, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaFuncSetAttribute(mla_flash_tc_kernel<true, true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
      return HK_ERR_CUDA;
    attr_set[dev] = true;
  }
  return HK_OK;
}

// Cluster form: splits of a row for m rows of about `tiles` tiles, false where it is not the better one.
// One row, two tiles a split.  2,052 gathered rows 9.2 us against 10.8 with partials in memory; two rows
// find room for two parts each only (16 CTAs with a whole SM's memory in one GPC: seven clusters at once), whose shares of twice the size
// take longer to cross: 11.7 against 11.6, three 12.2 against 12.5, and from four rows on the partials' own kernel fills the GPU.
bool mla_flash_cluster_shape(int m, int tiles, int* n_split) {
  int c = 2;
  while (c < FT_MAX_CL && c * 2 < tiles) c *= 2;
  if (tiles < 2 || tiles > 2 * FT_MAX_CL + 1 || m != 1) return false;
  static int fit[64][5] = {{0}};                           // clusters of 2^i CTAs that run at once, + 1
  int dev = 0, lg = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || ft_prepare() != HK_OK) return false;
  while ((1 << lg) < c) lg++;
  if (fit[dev][lg] == 0) {
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = c;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(c);
    cfg.blockDim = dim3(FT_THREADS);
    cfg.dynamicSmemBytes = FS_SMEM;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, mla_flash_tc_kernel<true, true>, &cfg) != cudaSuccess) n = 0;
    fit[dev][lg] = n + 1;
  }
  const int room = fit[dev][lg] - 1;
  if (room < FT_CS) return false;
  *n_split = c;
  return true;
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

int mla_flash_tc_launch(const MlaArgs& a, cudaStream_t s, bool clusters) {
  FtEncodeFn encode = ft_encode_fn();
  if (a.n_heads != FT_HEADS || !encode) return HK_ERR_UNSUPPORTED;
  if (ft_prepare() != HK_OK) return HK_ERR_CUDA;
  // Tensor maps over the latent cache.  The row extent is the cache's row count when the caller gave it (the copy engine
  // zero-fills anything past the end), else an upper bound.
  alignas(64) CUtensorMap box, rows, qmap, omap;
  memset(&box, 0, sizeof(box));
  memset(&rows, 0, sizeof(rows));
  memset(&qmap, 0, sizeof(qmap));
  memset(&omap, 0, sizeof(omap));
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
  // 64 rows x 512 channels as one box: whole key tiles of a dense range, and a row's 64 heads of Q
  auto box_map = [&](CUtensorMap* m, const void* p, cuuint64_t n, cuuint32_t keys = 64, cuuint32_t blocks = 8) {
    const cuuint64_t dims[3] = {64, n, 8};
    const cuuint64_t strides[2] = {LATENT * 2, 128};
    const cuuint32_t b[3] = {64, keys, blocks};
    return encode(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(p), dims, strides, b, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  static_assert(FT_KEYS == 64 && FT_HEADS == 64, "one box shape for keys and queries");
  const cuuint64_t q_rows = (cuuint64_t)a.m * FT_HEADS;
  // Two rows of a causal chunk share their keys.  Below 700 keys a row on average the pair's own costs (a cluster to start, the later row's own
  // key as a tile) are more than it gains: us, a CTA a row / pairs, 148 rows at 300 15.3 / 15.4, at 600 19.7 / 19.5, at 1,000 25.5 / 24.2;
  // 500 at 300 65.7 / 67.8, at 700 89.7 / 86.5; 1,200 at 0 151 / 154, 1,500 209 / 208, 2,500 470 / 431.
  const bool pairs = !clusters && !a.raw_idx && !a.kv_len && !a.kv_base && a.out && a.n_split == 1 && a.m >= 2 && a.pos_start + a.m / 2 >= FT_PAIR_KEYS;
  if (!box_map(&qmap, a.q_lat, q_rows) || (!a.raw_idx && !pairs && !box_map(&box, a.ckv, extent))) return HK_ERR_UNSUPPORTED;
  if (a.out) {
    const cuuint64_t dims[2] = {LATENT, q_rows};
    const cuuint64_t strides[1] = {LATENT * 2};
    const cuuint32_t b[2] = {64, 64};
    if (encode(&omap, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, a.out, dims, strides, b, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
      return HK_ERR_UNSUPPORTED;
  }
  if (pairs) {
    alignas(64) CUtensorMap vbox;
    if (!box_map(&box, a.ckv, extent, 32, 8) || !box_map(&vbox, a.ckv, extent, 32, 4)) return HK_ERR_UNSUPPORTED;
    const cudaError_t e = pdl_launch_cluster(2, mla_pair_tc_kernel, dim3((unsigned)((a.m + 1) / 2 * 2)), dim3(PT_THREADS), FS_SMEM, s, a,
                                             device_status_ptr(), box, vbox, rows, qmap, omap);
    return e == cudaSuccess && cudaPeekAtLastError() == cudaSuccess ? HK_OK : HK_ERR_CUDA;
  }
  // Gathered rows: at most a CTA per SM (592 rows of 2,048 keys 180 -> 166 us).  Dense rows, whose loads start faster: a CTA
  // each (600 rows at 32,768 keys 2.72 ms, persistent 2.85).  Partials always: their rows leave through the idle ring.
  if (clusters) {
    const dim3 grid((unsigned)(a.m * FT_CS * a.n_split));
    const cudaError_t e = a.raw_idx ? pdl_launch_cluster(a.n_split, mla_flash_tc_kernel<true, true>, grid, dim3(FT_THREADS), FS_SMEM, s, a,
                                                         device_status_ptr(), box, rows, qmap, omap)
                                    : pdl_launch_cluster(a.n_split, mla_flash_tc_kernel<false, true>, grid, dim3(FT_THREADS), FS_SMEM, s, a,
                                                         device_status_ptr(), box, rows, qmap, omap);
    return e == cudaSuccess && cudaPeekAtLastError() == cudaSuccess ? HK_OK : HK_ERR_CUDA;
  }
  const int64_t items = (int64_t)a.n_split * a.m;
  const dim3 grid((unsigned)(a.raw_idx && a.out && items > sm_count() ? sm_count() : items));
  const cudaError_t e =
      a.raw_idx ? pdl_launch(mla_flash_tc_kernel<true, false>, grid, dim3(FT_THREADS), FS_SMEM, s, a, device_status_ptr(), box, rows, qmap, omap)
                : pdl_launch(mla_flash_tc_kernel<false, false>, grid, dim3(FT_THREADS), FS_SMEM, s, a, device_status_ptr(), box, rows, qmap, omap);
  return e == cudaSuccess && cudaPeekAtLastError() == cudaSuccess ? HK_OK : HK_ERR_CUDA;
}

}  // namespace hk
