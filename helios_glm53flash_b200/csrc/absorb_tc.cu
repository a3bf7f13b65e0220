// Absorbed MLA projections on the 5th-generation tensor cores: per head h
//   q_lat[r][h][0:512] = q_nope[r][h][0:256] . W_uk[h]        (helios::attn::q_latent / q_latent_t)
//   o[r][h][0:256]     = lat_out[r][h][0:512] . W_uv[h]^T     (helios::attn::o_absorb / o_absorb_t)
// with kv_b the raw [64*512][512] fp16 tensor (rows h*512 .. +255 = W_uk[h], +256 .. +511 = W_uv[h]);
// reference: src/cuda/attn/attn.cu:12-130 (one block per (row, head), the head's weights re-read per row).
//
// Three kernels: up to 8 rows with operands in registers (warp-level products), up to 32 with the weights as the M operand, more in
// 256 x 256 tiles.  In the last two operands arrive as TMA tensor copies in 128-byte-swizzle boxes (A [rows][64 k]; W either
// [64 k][64 n] with n contiguous - W_uk, transposed W_uv - or [n][64 k] with k contiguous - raw W_uv, so o_absorb needs no transposed
// copy of the weights).  Rows past the end of the batch are zero-filled by the copy engine and not stored.  All waits are bounded.
#include <cuda.h>   // CUtensorMap (types only; the encoder is fetched through the runtime at first use)

#include <cstdlib>
#include <cstring>

#include "hk_common.cuh"
#include "tc05.cuh"

namespace hk {

// Persistent CTAs over tiles of 256 rows x 256 columns x one head, K in chunks of 64 channels through a three-stage ring of
// 64 KB.  What bounds it is the traffic between L2 and the SMs, which needs some 190 KB in flight per SM to pass 34 B per cycle:
// 128-row tiles, two CTAs per SM and 96 KB each, moved 805 / 786 MB for the 403 MB that 4,096 rows cannot do without (113 us
// q_latent, 89 us o_absorb); a weight tile of 128 KB kept in shared memory left a ring of 64 KB and 20-24 B per cycle (87, 103).
// Here it is 524 MB: 86 and 80 us.  Tiles run over columns, heads, rows: the CTAs at work write one stretch of whole output rows
// and read all 16.8 MB of weights, which stay in L2.  At 512 rows 20.9 -> 14.8 and 16.6 -> 14.3 us, at 33 rows 8.7 -> 6.1 and
// 10.6 -> 6.6 (all copies of a tile fly at once).
// Warp 0 copies in, warp 1 issues the products (converged, elected lane) into 2 x 256 tensor-memory columns, warps 2-9 write
// out: a lane takes its whole row of the accumulator as fp16 into registers (the products of the next tile can start), then the
// warp sends it off in boxes of 32 rows x 64 columns through 4 KB of its own, with no barrier between warps.
constexpr int AB_BM = 128, AB_BN = 256, AB_BK = 64, AB_STAGES = 3;
constexpr uint32_t AB_A_BYTES = AB_BM * AB_BK * 2;            // 16 KB, two per stage
constexpr uint32_t AB_W_BYTES = AB_BN * AB_BK * 2;            // 32 KB
constexpr uint32_t AB_STAGE = 2 * AB_A_BYTES + AB_W_BYTES;
constexpr uint32_t AB_BOX = 32 * 128;                         // one output box
constexpr int AB_THREADS = 320;
constexpr uint32_t AB_SMEM = AB_STAGES * AB_STAGE + 8 * AB_BOX + 1024;   // + slack to align the base to 1 KB

__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* tmap, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          tc::smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(x), "r"(y), "r"(tc::smem_u32(bar))
      : "memory");
}

// W_MN: the weight tile has n contiguous ([k][n] in memory), else k contiguous ([n][k]).
template <bool W_MN, int K>
__global__ __launch_bounds__(AB_THREADS, 1) void absorb_gemm_tc_kernel(
    const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_o,
    int n_rows, int tile_rows, int n_tiles, int w_rows_per_head, int w_row_off, int* __restrict__ status) {
  constexpr int NK = K / AB_BK;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  __shared__ uint64_t full_bar[AB_STAGES], empty_bar[AB_STAGES], acc_full[2], acc_empty[2];
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = tc::warp_index_uniform();
  const int total = 64 * n_tiles * ((n_rows + tile_rows - 1) / tile_rows);

  if (tid == 0) {
    for (int i = 0; i < AB_STAGES; i++) {
      tc::mbar_init(&full_bar[i], 1);
      tc::mbar_init(&empty_bar[i], 1);
    }
    for (int i = 0; i < 2; i++) {
      tc::mbar_init(&acc_full[i], 1);
      tc::mbar_init(&acc_empty[i], 4);
    }
    tc::mbar_fence_init();
    abort_flag = 0;
  }
  if (warp == 2) tc::tmem_alloc(&tmem_slot, 512);
  pdl_wait();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  auto place = [&](int t, int& n0, int& h, int& row0) {
    n0 = (t % n_tiles) * AB_BN;
    h = (t / n_tiles) & 63;
    row0 = t / n_tiles / 64 * tile_rows;
  };

  if (warp == 0) {
    if (lane == 0) {
      uint32_t n = 0;                                        // chunks so far
      bool ok = true;
      for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
        int n0, h, row0;
        place(t, n0, h, row0);
        const bool two = tile_rows > AB_BM && row0 + AB_BM < n_rows;              // the second half has rows
        const int wy = h * w_rows_per_head + w_row_off;
        for (int kc = 0; kc < NK; kc++, n++) {
          const int s = n % AB_STAGES;
          if (n >= AB_STAGES && !tc::mbar_wait<32>(&empty_bar[s], (n / AB_STAGES - 1) & 1, &abort_flag, 1)) {
            ok = false;
            break;
          }
          uint8_t* sa = smem + s * AB_STAGE;
          uint8_t* sw = sa + 2 * AB_A_BYTES;
          tc::mbar_arrive_expect_tx(&full_bar[s], AB_W_BYTES + (two ? 2 : 1) * AB_A_BYTES);
          tma_load_2d(sa, &tmap_a, h * K + kc * AB_BK, row0, &full_bar[s]);
          if (two) tma_load_2d(sa + AB_A_BYTES, &tmap_a, h * K + kc * AB_BK, row0 + AB_BM, &full_bar[s]);
          if (W_MN) {                                        // boxes of 64 n x 64 k, each a stack of 8-row swizzle atoms
#pragma unroll
            for (int j = 0; j < AB_BN / 64; j++) tma_load_2d(sw + j * 8192, &tmap_w, n0 + j * 64, wy + kc * AB_BK, &full_bar[s]);
          } else {                                           // one box of 64 k x 256 n rows
            tma_load_2d(sw, &tmap_w, kc * AB_BK, wy + n0, &full_bar[s]);
          }
        }
      }
    }
  } else if (warp == 1) {
    const uint32_t leader = tc::elect_one();
    const uint32_t idesc = tc::make_idesc(AB_BM, AB_BN, tc::FMT_F16, tc::FMT_F16, false, W_MN);
    bool ok = true;
    auto wait_u = [&](uint64_t* bar, uint32_t parity, int code) {   // every lane waits (tc05.cuh)
      const bool done = tc::mbar_wait<32>(bar, parity, &abort_flag, code);
      ok = __all_sync(0xffffffffu, done) != 0 && ok;
    };
    uint32_t n = 0, used[2] = {0, 0};                        // chunks, and tiles of either half, so far
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int n0, h, row0;
      place(t, n0, h, row0);
      const bool two = tile_rows > AB_BM && row0 + AB_BM < n_rows;
      for (int kc = 0; kc < NK && ok; kc++, n++) {
        const int s = n % AB_STAGES;
        wait_u(&full_bar[s], (n / AB_STAGES) & 1, 2);
        tc::fence_after_sync();
        const uint32_t a_addr = tc::smem_u32(smem + s * AB_STAGE), w_addr = a_addr + 2 * AB_A_BYTES;
#pragma unroll
        for (int m = 0; m < 2; m++) {
          if (m == 1 && !two) break;
          if (kc == 0) {
            if (used[m] > 0) {
              wait_u(&acc_empty[m], (used[m] - 1) & 1, 3);
              tc::fence_after_sync();
            }
            used[m]++;
          }
          if (!ok) break;
#pragma unroll
          for (int k16 = 0; k16 < AB_BK / 16; k16++)
            tc::mma_f16_if(leader, tmem + m * AB_BN, tc::make_sdesc_sw128(a_addr + m * AB_A_BYTES + k16 * 32, 16, 1024),
                           W_MN ? tc::make_sdesc_sw128(w_addr + k16 * 2048, 8192, 1024) : tc::make_sdesc_sw128(w_addr + k16 * 32, 16, 1024),
                           idesc, kc > 0 || k16 > 0);
          if (m == (two ? 1 : 0)) tc::mma_commit_if(leader, &empty_bar[s]);
          if (kc == NK - 1) tc::mma_commit_if(leader, &acc_full[m]);
        }
      }
    }
  } else {
    // ---- epilogue: four warps per half; a warp may only touch the TMEM lane quarter warp % 4 ----
    const int q = warp & 3, m = (warp - 2) >> 2;
    uint8_t* box = smem + AB_STAGES * AB_STAGE + (warp - 2) * AB_BOX;
    uint32_t used = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int n0, h, row0;
      place(t, n0, h, row0);
      row0 += m * AB_BM;
      if (row0 >= n_rows || m * AB_BM >= tile_rows) break;                             // only the last row tile is short, and it comes last
      ok = __all_sync(0xffffffffu, tc::mbar_wait<64>(&acc_full[m], used & 1, &abort_flag, 4)) != 0;
      used++;
      if (!ok) break;
      tc::fence_after_sync();
      uint32_t pk[AB_BN / 2];                                // this lane's row: the accumulator is free again before the first store
#pragma unroll
      for (int c0 = 0; c0 < AB_BN; c0 += 32) {
        uint32_t v[32];
        tc::tmem_ld32(tmem + m * AB_BN + c0 + ((uint32_t)(q * 32) << 16), v);
        tc::tmem_ld_wait();
#pragma unroll
        for (int e = 0; e < 16; e++) {
          const __half2 h2 = __floats2half2_rn(__uint_as_float(v[2 * e]), __uint_as_float(v[2 * e + 1]));
          pk[c0 / 2 + e] = *reinterpret_cast<const uint32_t*>(&h2);
        }
      }
      tc::fence_before_sync();
      __syncwarp();
      if (lane == 0) tc::mbar_arrive(&acc_empty[m]);
#pragma unroll
      for (int c0 = 0; c0 < AB_BN; c0 += 64) {
        if (lane == 0) tc::bulk_wait_read<0>();              // the box before has left
        __syncwarp();
        // a lane lays its row into the box in the 128-byte-swizzle pattern: 16-byte piece u of row r at u ^ (r % 8)
#pragma unroll
        for (int u = 0; u < 8; u++) {
          const uint32_t* w = pk + c0 / 2 + 4 * u;
          *reinterpret_cast<uint4*>(box + lane * 128 + ((u ^ (lane & 7)) << 4)) = make_uint4(w[0], w[1], w[2], w[3]);
        }
        tc::fence_async_smem();
        __syncwarp();
        if (lane == 0 && row0 + q * 32 < n_rows) {           // rows past the end are clipped
          asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%1, %2, %3}], [%4];" ::"l"(&tmap_o),
                       "r"(n0 + c0), "r"(h), "r"(row0 + q * 32), "r"(tc::smem_u32(box))
                       : "memory");
          tc::bulk_commit();
        }
      }
    }
    if (lane == 0) tc::bulk_wait_read<0>();
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 2) tc::tmem_dealloc(tmem, 512);
  if (tid == 0 && abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
}

// ------------------------------------------------------------------------------------------------
// A few rows (at most 32): the 16.8 MB of weights are all there is to move.  As 128-row tiles such a call has 128
// tiles, on 128 SMs, of which a row uses 1/128: 7.8 (q) and 10.5 us (o).  Here the WEIGHTS are the M operand, 64 output
// columns per CTA (512 and 256 CTAs, all resident), the rows are N (8 to 32), and a CTA requests its whole K at once (32 /
// 64 KB, a barrier per 64-channel chunk): no ring, no empty barriers.
// ------------------------------------------------------------------------------------------------
constexpr int AF_BM = 64, AF_BK = 64, AF_MAX_ROWS = 32, AF_THREADS = 128;
constexpr uint32_t AF_A_CHUNK = AF_BM * AF_BK * 2;            // 8 KB

// W_MN: weights [k][n] with n contiguous, else [n][k].  nb = rows rounded up to 8 (box rows of tmap_x).
template <bool W_MN, int K>
__global__ __launch_bounds__(AF_THREADS) void absorb_few_rows_kernel(const __grid_constant__ CUtensorMap tmap_w,
                                                                     const __grid_constant__ CUtensorMap tmap_x,
                                                                     __half* __restrict__ out, int n_rows, int nb, int n_out,
                                                                     int w_rows_per_head, int w_row_off, int* __restrict__ status, bool release) {
  constexpr int NK = K / AF_BK;
  if (release) pdl_release();
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sW = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* sX = sW + NK * AF_A_CHUNK;
  __shared__ uint64_t full_bar[NK], done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = tc::warp_index_uniform();
  const int n0 = blockIdx.x * AF_BM, h = blockIdx.y;
  const uint32_t x_chunk = (uint32_t)nb * AF_BK * 2;
  const int wy = h * w_rows_per_head + w_row_off + (W_MN ? 0 : n0);
  if (tid == 0) {
    // the weights on their way into L2 while the kernel before this one may still run (34.2 -> 33.4 us for the MLA layer of one
    // token; 0.1 us lost where they are in L2 already)
    for (int kc = 0; kc < NK; kc++) {
      asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(reinterpret_cast<uint64_t>(&tmap_w)),
                   "r"(W_MN ? n0 : kc * AF_BK), "r"(wy + (W_MN ? kc * AF_BK : 0))
                   : "memory");
      tc::mbar_init(&full_bar[kc], 1);
    }
    tc::mbar_init(&done_bar, 1);
    tc::mbar_fence_init();
    abort_flag = 0;
    pdl_wait();
    for (int kc = 0; kc < NK; kc++) {
      tc::mbar_arrive_expect_tx(&full_bar[kc], AF_A_CHUNK + x_chunk);
      tma_load_2d(sW + kc * AF_A_CHUNK, &tmap_w, W_MN ? n0 : kc * AF_BK, wy + (W_MN ? kc * AF_BK : 0), &full_bar[kc]);
      tma_load_2d(sX + kc * x_chunk, &tmap_x, h * K + kc * AF_BK, 0, &full_bar[kc]);
    }
  }
  if (warp == 1) tc::tmem_alloc(&tmem_slot, 32);
  pdl_wait();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = tmem_slot;
  if (warp == 1) {
    // whole warp, one elected lane issues (tc05.cuh): M64 products leave every ~24 cycles
    const uint32_t leader = tc::elect_one();
    const uint32_t idesc = tc::make_idesc(AF_BM, nb, tc::FMT_F16, tc::FMT_F16, W_MN, false);
#pragma unroll 1
    for (int kc = 0; kc < NK; kc++) {
      const bool landed = tc::mbar_wait(&full_bar[kc], 0, &abort_flag, 1);
      if (!__all_sync(0xffffffffu, landed)) break;
      tc::fence_after_sync();
      const uint32_t w_addr = tc::smem_u32(sW + kc * AF_A_CHUNK), x_addr = tc::smem_u32(sX + kc * x_chunk);
#pragma unroll
      for (int k16 = 0; k16 < AF_BK / 16; k16++)
        tc::mma_f16_if(leader, tmem, tc::make_sdesc_sw128(w_addr + k16 * (W_MN ? 2048 : 32), W_MN ? 8192 : 16, 1024),
                       tc::make_sdesc_sw128(x_addr + k16 * 32, 16, 1024), idesc, kc > 0 || k16 > 0);
    }
    tc::mma_commit_if(leader, &done_bar);
  }
  const bool ok = tc::mbar_wait(&done_bar, 0, &abort_flag, 2);
  tc::fence_after_sync();
  // output column 16 w + i sits in TMEM lane 32 w + i, i < 16
  if (__all_sync(0xffffffffu, ok)) {
#pragma unroll 1
    for (int c0 = 0; c0 < nb; c0 += 16) {
      uint32_t v[16];
      tc::tmem_ld16(tmem + ((uint32_t)(warp * 32) << 16) + c0, v);
      tc::tmem_ld_wait();
      if (lane < 16) {
        __half* o = out + ((size_t)c0 * 64 + h) * n_out + n0 + warp * 16 + lane;
#pragma unroll
        for (int j = 0; j < 16; j++)
          if (c0 + j < n_rows) o[(size_t)j * 64 * n_out] = __float2half_rn(__uint_as_float(v[j]));
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 1) tc::tmem_dealloc(tmem, 32);
  if (tid == 0 && abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
}

// ------------------------------------------------------------------------------------------------
// Up to eight rows (a decode step).  What bounds it is latency: 16.8 MB over 148 SMs are 1 us from L2, and the tensor-map fetch, tensor
// memory, products behind barriers and the way back of the kernel above are more than that.  Here a lane loads its operand fragments of
// the warp-level product straight into registers, all of them at once (m16n8k16, the weights as the 16 rows and the batch as the 8
// columns, fp32 sums), the warps of a CTA share out K, and their sums meet once in shared memory.  The contraction index is taken in
// whatever order a lane's pieces hold it, the same for both operands.  1,024 CTAs of 16 KB, seven a SM (512 of 32 KB are 4 or 3: q 4.0).
// In a graph of 20 calls, weights in L2 / from HBM, 1 row: q 4.5 -> 3.7 / 4.8 -> 3.9 us, o 4.1 -> 3.1 / 5.2 -> 3.4; 8 rows: q 4.6 -> 4.5 /
// 5.0 -> 4.6, o 4.2 -> 3.4 / 5.4 -> 3.8.  MLA layer of one token at 5,001 29.3 -> 24.8 us.  From nine rows on, and for the transposed W_uv, whose
// CTAs hold twice the K here (8 rows 4.9 for 4.2), the kernel above is the better one.
// ------------------------------------------------------------------------------------------------
constexpr int A8_ROWS = 8;

__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
  asm(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void prefetch_l2_line(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// W_MN: weights [k][n] with n contiguous: a CTA has 32 columns, a warp 64 k of them, a lane four columns of 16 k, whose pairs along k it
// puts together itself.  Else [n][k]: a CTA has 16 columns, a warp 128 k, and a piece along k is what the product takes.
template <bool W_MN, int K>
__global__ __launch_bounds__(W_MN ? K / 2 : K / 4, W_MN ? 2048 / K : 8) void absorb_8_rows_kernel(const __half* __restrict__ w, const __half* x, __half* __restrict__ out,
                                                                        int n_rows, int n_out, int w_rows_per_head, int w_row_off) {
  // One row: the scorer's or the next layer's CTAs are placed as these end and ask for what they read (45-layer decode at 262,144 477 -> 470 us,
  // at 5,000 435 -> 429; with three rows 39.4 -> 40.4 for the layer).
  if (n_rows == 1) pdl_release();
  constexpr int WARPS = W_MN ? K / 64 : K / 128, BN = W_MN ? 32 : 16;
  __shared__ __align__(16) float red[WARPS][A8_ROWS][BN];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int n0 = blockIdx.x * BN, h = blockIdx.y;
  const bool row = g < n_rows;
  // 16-byte pieces of a row of sums change places by the row, so that a quarter-warp writes to all banks
  auto swap = [](int r) -> int { return W_MN ? (r >> 1) << 1 : 0; };
  if constexpr (W_MN) {
    // k = 64 warp + 16 s + 4 t + e; columns n0 + 4 g ..
    const __half* wp = w + (size_t)(h * w_rows_per_head + w_row_off + 64 * warp + 4 * t) * n_out + n0 + 4 * g;
    if (g == 0)
#pragma unroll
      for (int i = 0; i < 16; i++) prefetch_l2_line(wp + (size_t)((i >> 2) * 16 + (i & 3)) * n_out);
    pdl_wait();
    uint2 wr[16];
#pragma unroll
    for (int i = 0; i < 16; i++)
      asm volatile("ld.global.nc.L1::no_allocate.v2.u32 {%0,%1}, [%2];" : "=r"(wr[i].x), "=r"(wr[i].y) : "l"(wp + (size_t)((i >> 2) * 16 + (i & 3)) * n_out));
    uint2 xr[4];
#pragma unroll
    for (int s = 0; s < 4; s++)
      xr[s] = row ? __ldcg(reinterpret_cast<const uint2*>(x + ((size_t)g * 64 + h) * K + 64 * warp + 16 * s + 4 * t)) : make_uint2(0, 0);
    float c[4][4];
#pragma unroll
    for (int i = 0; i < 4; i++) c[i][0] = c[i][1] = c[i][2] = c[i][3] = 0.f;
#pragma unroll
    for (int s = 0; s < 4; s++) {
      const uint32_t* r0 = &wr[4 * s].x;
      const uint32_t* r1 = &wr[4 * s + 1].x;
      const uint32_t* r2 = &wr[4 * s + 2].x;
      const uint32_t* r3 = &wr[4 * s + 3].x;
#pragma unroll
      for (int i = 0; i < 4; i++) {                          // column 4 g + i: its four k as two pairs
        const uint32_t sel = i & 1 ? 0x7632 : 0x5410;
        mma_16816(c[i], __byte_perm(r0[i >> 1], r1[i >> 1], sel), 0, __byte_perm(r2[i >> 1], r3[i >> 1], sel), 0, xr[s].x, xr[s].y);
      }
    }
#pragma unroll
    for (int r = 0; r < 2; r++)
      if (2 * t + r < n_rows) {
        float4* p = reinterpret_cast<float4*>(red[warp][2 * t + r]);
        p[g ^ swap(2 * t)] = make_float4(c[0][r], c[1][r], c[2][r], c[3][r]);
      }
  } else {
    // k = 128 warp + 32 s + 8 t + e; columns n0 + g and n0 + g + 8
    const __half* wp = w + (size_t)(h * w_rows_per_head + w_row_off + n0 + g) * K + 128 * warp + 8 * t;
    if (t == 0)
#pragma unroll
      for (int i = 0; i < 4; i++) prefetch_l2_line(wp + (i >> 1) * 8 * K + (i & 1) * 64);
    pdl_wait();
    uint4 wr[4][2], xr[4];
#pragma unroll
    for (int s = 0; s < 4; s++)
#pragma unroll
      for (int u = 0; u < 2; u++) wr[s][u] = ld_stream16(wp + u * 8 * K + 32 * s);
#pragma unroll
    for (int s = 0; s < 4; s++)
      xr[s] = row ? __ldcg(reinterpret_cast<const uint4*>(x + ((size_t)g * 64 + h) * K + 128 * warp + 32 * s + 8 * t)) : make_uint4(0, 0, 0, 0);
    float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int s = 0; s < 4; s++) {
      mma_16816(c, wr[s][0].x, wr[s][1].x, wr[s][0].y, wr[s][1].y, xr[s].x, xr[s].y);
      mma_16816(c, wr[s][0].z, wr[s][1].z, wr[s][0].w, wr[s][1].w, xr[s].z, xr[s].w);
    }
#pragma unroll
    for (int e = 0; e < 4; e++)
      if (2 * t + (e & 1) < n_rows) red[warp][2 * t + (e & 1)][g + 8 * (e >> 1)] = c[e];
  }
  __syncthreads();
  const int n = tid % BN;
  for (int r = tid / BN; r < n_rows; r += WARPS * 32 / BN) {
    const int at = n ^ (swap(r) << 2);
    float sum = red[0][r][at];
#pragma unroll
    for (int i = 1; i < WARPS; i++) sum += red[i][r][at];
    out[((size_t)r * 64 + h) * n_out + n0 + n] = __float2half_rn(sum);
  }
}

template <bool W_MN, int K>
static int absorb_8_rows(const void* x, const void* w, void* out, int n_rows, int n_out, int w_rows_per_head, int w_row_off, cudaStream_t s) {
  return pdl_launch(absorb_8_rows_kernel<W_MN, K>, dim3(n_out / (W_MN ? 32 : 16), 64), dim3(W_MN ? K / 2 : K / 4), 0, s, (const __half*)w,
                    (const __half*)x, (__half*)out, n_rows, n_out, w_rows_per_head, w_row_off) == cudaSuccess
             ? HK_OK
             : HK_ERR_CUDA;
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  static bool looked_up = false;
  if (!looked_up) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qres) == cudaSuccess &&
        qres == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
    looked_up = true;
  }
  return fn;
}

// fp16 matrix [rows][cols] (cols contiguous), box [box_rows][box_cols], 128-byte swizzle, zero fill outside
static bool make_map_2d(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols, uint32_t box_rows, uint32_t box_cols) {
  EncodeTiledFn enc = encode_tiled_fn();
  if (!enc) return false;
  const cuuint64_t dims[2] = {cols, rows};
  const cuuint64_t strides[1] = {cols * 2};
  const cuuint32_t box[2] = {box_cols, box_rows};
  const cuuint32_t estr[2] = {1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <bool W_MN, int K>
static int absorb_few_rows(const void* x, const void* w, void* out, int n_rows, int n_out, uint64_t w_rows, uint64_t w_cols,
                           int w_rows_per_head, int w_row_off, bool release, cudaStream_t s) {
  const int nb = (n_rows + 7) & ~7;
  alignas(64) CUtensorMap mw, mx;
  memset(&mw, 0, sizeof(mw));
  memset(&mx, 0, sizeof(mx));
  if (!make_map_2d(&mw, w, w_rows, w_cols, AF_BM, AF_BK) || !make_map_2d(&mx, x, (uint64_t)n_rows, (uint64_t)64 * K, nb, AF_BK))
    return HK_ERR_UNSUPPORTED;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    const int most = K / AF_BK * (AF_A_CHUNK + AF_MAX_ROWS * AF_BK * 2) + 1024;
    if (cudaFuncSetAttribute(absorb_few_rows_kernel<W_MN, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess)
      return HK_ERR_CUDA;
    attr_set[dev] = true;
  }
  const size_t smem = (size_t)(K / AF_BK) * (AF_A_CHUNK + nb * AF_BK * 2) + 1024;
  return pdl_launch(absorb_few_rows_kernel<W_MN, K>, dim3(n_out / AF_BM, 64), dim3(AF_THREADS), smem, s, mw, mx, (__half*)out, n_rows,
                    nb, n_out, w_rows_per_head, w_row_off, device_status_ptr(), release) == cudaSuccess
             ? HK_OK
             : HK_ERR_CUDA;
}

template <bool W_MN, int K>
static int absorb_rows(const void* x, const void* w, void* out, int n_rows, int n_out, uint64_t w_rows, uint64_t w_cols,
                       int w_rows_per_head, int w_row_off, cudaStream_t s) {
  alignas(64) CUtensorMap mx, mw, mo;
  memset(&mx, 0, sizeof(mx));
  memset(&mw, 0, sizeof(mw));
  memset(&mo, 0, sizeof(mo));
  if (!make_map_2d(&mx, x, (uint64_t)n_rows, (uint64_t)64 * K, AB_BM, AB_BK) ||
      !make_map_2d(&mw, w, w_rows, w_cols, W_MN ? AB_BK : AB_BN, 64))
    return HK_ERR_UNSUPPORTED;
  // output as [row][head][n_out]: boxes of 64 columns x 1 head x 32 rows
  const cuuint64_t dims[3] = {(cuuint64_t)n_out, 64, (cuuint64_t)n_rows};
  const cuuint64_t strides[2] = {(cuuint64_t)n_out * 2, (cuuint64_t)64 * n_out * 2};
  const cuuint32_t box[3] = {64, 1, 32};
  const cuuint32_t estr[3] = {1, 1, 1};
  if (encode_tiled_fn()(&mo, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, out, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                        CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
    return HK_ERR_UNSUPPORTED;
  static bool attr_set[64] = {false};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr_set[dev]) {
    if (cudaFuncSetAttribute(absorb_gemm_tc_kernel<W_MN, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AB_SMEM) != cudaSuccess)
      return HK_ERR_CUDA;
    attr_set[dev] = true;
  }
  const int n_tiles = n_out / AB_BN;
  // one half at a time while that still is one wave (o_absorb of 256 rows 9.9 -> 9.2 us on 128 SMs instead of 64)
  const int tile_rows = (int64_t)64 * n_tiles * ((n_rows + AB_BM - 1) / AB_BM) <= sm_count() ? AB_BM : 2 * AB_BM;
  const int64_t total = (int64_t)64 * n_tiles * ((n_rows + tile_rows - 1) / tile_rows);
  if (total > 1 << 30) return HK_ERR_UNSUPPORTED;
  const int grid = (int)(total < sm_count() ? total : sm_count());
  return pdl_launch(absorb_gemm_tc_kernel<W_MN, K>, dim3(grid), dim3(AB_THREADS), AB_SMEM, s, mx, mw, mo, n_rows, tile_rows, n_tiles,
                    w_rows_per_head, w_row_off, device_status_ptr()) == cudaSuccess
             ? HK_OK
             : HK_ERR_CUDA;
}

// a [n_rows][64*K], weights as described above, out [n_rows][64*n_out]; returns HK_ERR_UNSUPPORTED when the
// tensor maps cannot be built (the caller then uses the CUDA-core kernels).
// `beside`: the caller has such calls on other streams.  Up to eight rows the kernel with operands in registers is the faster one alone and the
// slower one in company, whose 1,024 CTAs take every SM's registers while other streams' attention waits for whole SMs.  11 MLA layers of a
// decode step, one stream a sequence, that kernel / the one of few rows: at 5,000 tokens 2 sequences 363 / 357 us, 4 474 / 440, 8 731 / 689, at
// 32,768 381 / 372, 492 / 463, 970 / 908; one sequence 263 / 273.  (Without the early release of one row 367, 441, 684 and 382, 472, 932.)
int absorb_gemm_tc(const void* a, const void* b, void* out, int n_rows, int K, int n_out, bool b_mn,
                   uint64_t b_rows, uint64_t b_cols, int b_rows_per_head, int b_row_off, cudaStream_t s, bool beside) {
  if (!aligned(a, 16) || !aligned(b, 16) || !aligned(out, 16)) return HK_ERR_UNSUPPORTED;
  if (n_rows <= A8_ROWS && !beside) {
    if (K == 256 && b_mn) return absorb_8_rows<true, 256>(a, b, out, n_rows, n_out, b_rows_per_head, b_row_off, s);
    if (K == 512 && !b_mn) return absorb_8_rows<false, 512>(a, b, out, n_rows, n_out, b_rows_per_head, b_row_off, s);
  }
  if (n_rows <= AF_MAX_ROWS) {
    const bool release = beside && n_rows == 1;
    // q_latent (K 256, n contiguous), o_absorb (K 512, k contiguous), o_absorb_t (K 512, n contiguous)
    if (K == 256 && b_mn) return absorb_few_rows<true, 256>(a, b, out, n_rows, n_out, b_rows, b_cols, b_rows_per_head, b_row_off, release, s);
    if (K == 512 && !b_mn) return absorb_few_rows<false, 512>(a, b, out, n_rows, n_out, b_rows, b_cols, b_rows_per_head, b_row_off, release, s);
    if (K == 512 && b_mn) return absorb_few_rows<true, 512>(a, b, out, n_rows, n_out, b_rows, b_cols, b_rows_per_head, b_row_off, release, s);
  }
  if (K == 256 && b_mn) return absorb_rows<true, 256>(a, b, out, n_rows, n_out, b_rows, b_cols, b_rows_per_head, b_row_off, s);
  if (K == 512 && !b_mn) return absorb_rows<false, 512>(a, b, out, n_rows, n_out, b_rows, b_cols, b_rows_per_head, b_row_off, s);
  if (K == 512 && b_mn) return absorb_rows<true, 512>(a, b, out, n_rows, n_out, b_rows, b_cols, b_rows_per_head, b_row_off, s);
  return HK_ERR_UNSUPPORTED;
}

}  // namespace hk
