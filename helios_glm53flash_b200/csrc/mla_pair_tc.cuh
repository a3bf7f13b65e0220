// Dense causal attention of two neighbouring query rows by a pair of CTAs (tcgen05 cta_group::2).  Included by mla_flash_tc.cu.
//
// Two rows of a prefill chunk attend to the same keys but for the later row's own.  Their 2 x 64 heads are the 128 rows of one product:
// each CTA of the pair holds its row's queries, softmax weights and accumulator, and HALF of every B operand, which the tensor cores of
// both SMs read: for S = Q K^T 32 of a tile's 64 keys (all channels), for O += P V 256 of the 512 channels (all 64 keys).  What a CTA
// loads for a tile is 48 KB instead of 64 - 32 keys whole, and its channels of the other 32; its channels of its own keys are needed in
// both places and are copied inside the SM - and what its products read of K and V is 64 KB instead of 128.
// What bounds it: power.  A tile takes 1,230 cycles at the 1.32 GHz that the power limit leaves (a CTA a row: 1,900 at 1.6), most of it the
// softmax of 64 heads x 64 keys by one warp a scheduler (1,080).  4,096 rows at 32,768 keys 17.6 -> 14.8 ms (1.27 PFLOP/s; cuBLAS 1.40
// sustained; on another GPU 18.6 -> 15.7), 2,500 rows at 0 470 -> 431 us, 151 at 9,000 297 -> 228.  On the way: arrivals at the first CTA with
// cluster-scope release cost 700 cycles each (23.1 ms); K's part given back with V's left each load 1.5 tiles of time (16.4 ms; two
// loaders, each part given back by itself: 14.8); 64 KB from L2 a tile and CTA 16.5.
// Roles, buffers, softmax and tensor-memory plan are those of mla_flash_tc_kernel (O 256 columns, S 2 x 32, channels 128-511 of Q 192, the
// 64 rows of a CTA in lanes 0-63 and 64-127 with half of the columns each).  The first CTA of the pair issues every product for both;
// its barriers count the arrivals of both, and commits arrive at both.
// The later row's own key is a tile of its own, whose P V leaves the earlier row's accumulator alone (a mask of lanes): a weight of
// zero would not do where the cache row holds infinities or NaN.
#pragma once

namespace hk {

// ring slot, in blocks of 64 channels x 32 keys: K (8 blocks, this CTA's keys), V (4 blocks of the first CTA's keys, 4 of the second's)
constexpr uint32_t PT_BLK = 32 * 128, PT_V = 8 * PT_BLK, PT_V_HALF = 4 * PT_BLK;
static_assert(PT_V + 2 * PT_V_HALF == FT_TILE, "a slot");
constexpr int PT_THREADS = 8 * 32;                // softmax 0-3, S 4, P V 5, loads 6, copies inside the SM 7

struct PtMisc {
  uint64_t k_here[FT_NBUF], v_here[FT_NBUF];      // this CTA's part of K, of V
  uint64_t k_full[FT_NBUF];                       // the first CTA's: both parts of K
  uint64_t k_free[FT_NBUF], v_free[FT_NBUF];      // the products that read them are complete
  uint64_t s_full[2], s_free[2], p_full[2], pv_done[2];
  uint64_t q_full, q_moved, q_ready;
  float mx[2][128];
  float l[128];
  uint32_t tmem;
  int abort_flag;
};
static_assert(sizeof(PtMisc) <= 2048, "misc area");

__device__ __forceinline__ void pt_tma_box(void* smem_dst, const CUtensorMap* tmap, int row, int blk, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
          tc::smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(tmap)), "r"(0), "r"(row), "r"(blk), "r"(tc::smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void pt_mma(uint32_t leader, uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(ad), "l"(bd), "r"(idesc), "r"((uint32_t)acc), "r"(leader)
      : "memory");
}
__device__ __forceinline__ void pt_mma_tmem_a(uint32_t leader, uint32_t d, uint32_t a, uint64_t bd, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d),
      "r"(a), "l"(bd), "r"(idesc), "r"((uint32_t)acc), "r"(leader)
      : "memory");
}
// the second CTA's accumulator only: the first one's 128 lanes are left alone
__device__ __forceinline__ void pt_mma_second(uint32_t leader, uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, bool acc) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, {%6, %6, %6, %6, %7, %7, %7, %7}, p;\n\t}" ::"r"(d),
      "l"(ad), "l"(bd), "r"(idesc), "r"((uint32_t)acc), "r"(leader), "r"(0xffffffffu), "r"(0u)
      : "memory");
}
// Arrives at this barrier in both CTAs, some time after the products.  Each such arrival is waited for in both CTAs before either may leave (a
// slot that no tile takes over again is therefore not given back): behind its end a CTA's shared memory is another's.
__device__ __forceinline__ void pt_commit(uint32_t leader, uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %2;\n\t}" ::"r"(tc::smem_u32(bar)),
      "r"(leader), "h"((uint16_t)3)
      : "memory");
}
// Arrives at a barrier of either CTA; it releases, and pt_try_wait acquires, at the scope of a CTA.  What the first CTA's products then read of
// the other CTA is read by that SM's own tensor core, and all of it is ordered before the arrival where it was written: P by the writing
// threads' proxy fence, the accumulator and S by their tcgen05.wait and fence, K and V by the completed copies that the arriving thread has
// waited for.  No byte of it crosses to the waiting SM, only the arrival does.  (Two-SM kernels of CUTLASS arrive at the other CTA in this form.
// With the release at the scope of the cluster an arrival took 700 cycles: 23.1 ms for 14.8.)
__device__ __forceinline__ void pt_arrive(uint32_t cluster_bar) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_bar) : "memory");
}
__device__ __forceinline__ bool pt_try_wait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(tc::smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool pt_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, int code) {   // bounded as tc::mbar_wait
  if (pt_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    if (*abort_flag) return false;
    if (pt_try_wait(bar, parity)) return true;
    __nanosleep(FT_POLL_NS);
    if (clock64() - t0 > tc::MBAR_WAIT_CYCLES) {
      *abort_flag = code;
      return false;
    }
  }
}

// grid = 2 CTAs a pair of rows, cluster of 2.  tmap_k / tmap_v: boxes of 32 keys x 512 and x 256 channels; tmap_rows, tmap_q, tmap_o as in
// mla_flash_tc_kernel.
__global__ __launch_bounds__(PT_THREADS, 1) void mla_pair_tc_kernel(
    MlaArgs a, int* __restrict__ status, const __grid_constant__ CUtensorMap tmap_k, const __grid_constant__ CUtensorMap tmap_v,
    const __grid_constant__ CUtensorMap tmap_rows, const __grid_constant__ CUtensorMap tmap_q, const __grid_constant__ CUtensorMap tmap_o) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  PtMisc& ms = *reinterpret_cast<PtMisc*>(smem + FS_MISC);
  volatile int* abort_flag = &ms.abort_flag;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = tc::warp_index_uniform();
  const int rank = blockIdx.x & 1;                         // cluster of 2 along x
  // pairs from the last row on, the longest first; a chunk of an odd number of rows leaves row 0 alone, whose pair is a copy of it
  const int r1 = a.m - 1 - 2 * (int)(blockIdx.x >> 1), r0 = max(0, r1 - 1), row = rank == 0 ? r0 : r1;
  const bool lone = r1 == 0, mine = !(lone && rank == 1);
  const int n = a.pos_start + r0 + 1;                      // the keys of both rows
  const int whole = (n + FT_KEYS - 1) / FT_KEYS, n_tiles = whole + (lone ? 0 : 1);
  auto keys = [&](int t) -> int { return t < whole ? min(FT_KEYS, n - t * FT_KEYS) : 1; };
  auto key0 = [&](int t) -> int { return t < whole ? t * FT_KEYS : n; };

  if (tid == 0) {
    for (int b = 0; b < FT_NBUF; b++) {
      tc::mbar_init(&ms.k_here[b], 1);
      tc::mbar_init(&ms.v_here[b], 1);
      tc::mbar_init(&ms.k_full[b], 2);
      tc::mbar_init(&ms.k_free[b], 1);
      tc::mbar_init(&ms.v_free[b], 1);
    }
    for (int b = 0; b < 2; b++) {
      tc::mbar_init(&ms.s_full[b], 1);
      tc::mbar_init(&ms.s_free[b], 8);
      tc::mbar_init(&ms.p_full[b], 8);
      tc::mbar_init(&ms.pv_done[b], 1);
    }
    tc::mbar_init(&ms.q_full, 1);
    tc::mbar_init(&ms.q_moved, 4);
    tc::mbar_init(&ms.q_ready, 8);
    tc::mbar_fence_init();
    ms.abort_flag = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::smem_u32(&ms.tmem)), "r"(512) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  pdl_wait();
  tc::fence_before_sync();
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");   // both CTAs' barriers and tensor memory
  tc::fence_after_sync();
  const uint32_t tmem = ms.tmem;
  auto first = [&](uint64_t* bar) -> uint32_t { return cluster_addr(tc::smem_u32(bar), 0); };   // the first CTA's
  bool ok = true;

  auto slot = [&](int t) -> uint8_t* { return smem + FS_K + t % FT_NBUF * FT_TILE; };
  auto turn = [](int t) -> uint32_t { return t / FT_NBUF & 1; };
  const int other = 32 * (1 - rank);                       // the other CTA's keys of a tile
  // a ragged tile: four rows at a time, those past the end read as zeros
  auto gather = [&](uint32_t leader, int t, int k0, int blk0, int blocks, uint32_t dst, uint64_t* bar) {
    const int base = key0(t), valid = keys(t);
    auto at = [&](int k) -> int { return k < valid ? base + k : -1; };
#pragma unroll 1
    for (int q = 0; q < 8; q++)
#pragma unroll 1
      for (int blk = 0; blk < blocks; blk++)
        tma_gather4_rows(leader, dst + blk * PT_BLK + q * 512, &tmap_rows, (blk0 + blk) * 64, at(k0 + 4 * q), at(k0 + 4 * q + 1), at(k0 + 4 * q + 2),
                         at(k0 + 4 * q + 3), tc::smem_u32(bar));
  };
  if (warp == 6) {
    // =========================== loads: this row's Q, then this CTA's keys of every tile ===========================
    const uint32_t leader = tc::elect_one();
    if (lane == 0) {
      tc::mbar_arrive_expect_tx(&ms.q_full, FT_TILE);
      tma_load_tile(smem + FS_K + 2 * FT_TILE, &tmap_q, row * FT_HEADS, &ms.q_full);
    }
    __syncwarp();
    for (int t = 0; t < n_tiles; t++) {
      const int b = t % FT_NBUF;
      if (t == 2) ok = tc::mbar_wait<FT_POLL_NS>(&ms.q_moved, 0, abort_flag, 21) && ok;
      if (t >= FT_NBUF) {                                  // S has read the part, and the copy to V
        ok = tc::mbar_wait<FT_POLL_NS>(&ms.k_free[b], turn(t) ^ 1, abort_flag, 22) && ok;
        ok = tc::mbar_wait<FT_POLL_NS>(&ms.v_here[b], turn(t) ^ 1, abort_flag, 34) && ok;
      }
      if (lane == 0) tc::mbar_arrive_expect_tx(&ms.k_here[b], PT_V);
      __syncwarp();
      if (keys(t) < FT_KEYS) gather(leader, t, 32 * rank, 0, 8, tc::smem_u32(slot(t)), &ms.k_here[b]);
      else if (lane == 0) pt_tma_box(slot(t), &tmap_k, key0(t) + 32 * rank, 0, &ms.k_here[b]);
      __syncwarp();
    }
  } else if (warp == 7) {
    // =========================== V: the other CTA's keys of this CTA's channels from memory, its own from K's part ===========================
    const uint32_t leader = tc::elect_one();
    for (int t = 0; t < n_tiles; t++) {
      const int b = t % FT_NBUF;
      if (t == 2) ok = tc::mbar_wait<FT_POLL_NS>(&ms.q_moved, 0, abort_flag, 21) && ok;
      if (t >= FT_NBUF) ok = tc::mbar_wait<FT_POLL_NS>(&ms.v_free[b], turn(t) ^ 1, abort_flag, 35) && ok;
      if (lane == 0) tc::mbar_arrive_expect_tx(&ms.v_here[b], 2 * PT_V_HALF);
      __syncwarp();
      uint8_t* const dst = slot(t) + PT_V + (1 - rank) * PT_V_HALF;
      if (keys(t) < FT_KEYS) gather(leader, t, other, 4 * rank, 4, tc::smem_u32(dst), &ms.v_here[b]);
      else if (lane == 0) pt_tma_box(dst, &tmap_v, key0(t) + other, 4 * rank, &ms.v_here[b]);
      __syncwarp();
      ok = tc::mbar_wait<FT_POLL_NS>(&ms.k_here[b], turn(t), abort_flag, 32) && ok;
      if (lane == 0) {
        pt_arrive(first(&ms.k_full[b]));
        asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         tc::smem_u32(slot(t)) + PT_V + rank * PT_V_HALF),
                     "r"(tc::smem_u32(slot(t)) + 4 * rank * PT_BLK), "r"(PT_V_HALF), "r"(tc::smem_u32(&ms.v_here[b]))
                     : "memory");
      }
      __syncwarp();
    }
  } else if (warp >= 4) {
    // =========================== the first CTA issues for both (whole warp, one elected lane) ===========================
    const uint32_t leader = tc::elect_one();
    auto wait_u = [&](uint64_t* bar, uint32_t parity, int code) {
      const bool done = pt_wait(bar, parity, abort_flag, code);
      ok = __all_sync(0xffffffffu, done) != 0 && ok;
    };
    auto desc = [](const uint8_t* p, uint32_t lbo) {       // (formed anew: see mla_flash_tc_kernel)
      uint32_t addr = tc::smem_u32(p);
      asm volatile("" : "+r"(addr));
      return tc::make_sdesc_sw128(addr, lbo, 1024);
    };
    if (rank == 0 && warp == 4) {
      const uint32_t idesc = tc::make_idesc(128, FT_KEYS, tc::FMT_F16, tc::FMT_F16, false, false);
      wait_u(&ms.q_ready, 0, 23);
      for (int t = 0; t < n_tiles; t++) {
        const int b = t & 1, kb = t % FT_NBUF;
        wait_u(&ms.k_full[kb], (t / FT_NBUF) & 1, 24);
        if (t >= 2) wait_u(&ms.s_free[b], ((t - 2) >> 1) & 1, 25);
        tc::fence_after_sync();
        const uint64_t kd = desc(smem + FS_K + kb * FT_TILE, 16), qd = desc(smem + FS_Q, 16);
#pragma unroll
        for (int kk = 0; kk < LATENT / 16; kk++) {
          const uint64_t bd = tc::sdesc_advance(kd, (kk >> 2) * PT_BLK + (kk & 3) * 32);
          if (kk < FT_QS / 16)
            pt_mma(leader, tmem + FT_S + b * 32, tc::sdesc_advance(qd, (kk >> 2) * (FT_HEADS * 128) + (kk & 3) * 32), bd, idesc, kk > 0);
          else
            pt_mma_tmem_a(leader, tmem + FT_S + b * 32, tmem + FT_Q + (kk - FT_QS / 16) * 8, bd, idesc, true);
        }
        pt_commit(leader, &ms.s_full[b]);
        if (t + FT_NBUF < n_tiles) pt_commit(leader, &ms.k_free[kb]);
      }
    } else if (rank == 0) {
      const uint32_t idesc = tc::make_idesc(128, 256, tc::FMT_F16, tc::FMT_F16, false, true);
      for (int t = 0; t < n_tiles; t++) {
        const int b = t & 1, kb = t % FT_NBUF;
        wait_u(&ms.p_full[b], (t >> 1) & 1, 26);
        tc::fence_after_sync();
        const uint64_t pd = desc(smem + FS_P + b * FP_BYTES, 16), vd = desc(smem + FS_K + kb * FT_TILE + PT_V, PT_BLK);
        const int steps = (keys(t) + 15) >> 4;
        if (t < whole) {
#pragma unroll
          for (int nh = 0; nh < 2; nh++)
#pragma unroll
            for (int kk = 0; kk < FT_KEYS / 16; kk++)
              if (kk < steps)
                pt_mma(leader, tmem + FT_O + nh * 128, tc::sdesc_advance(pd, kk * 32), tc::sdesc_advance(vd, nh * 2 * PT_BLK + (kk >> 1) * PT_V_HALF + (kk & 1) * 2048), idesc,
                       t > 0 || kk > 0);
        } else {
#pragma unroll
          for (int nh = 0; nh < 2; nh++)
            pt_mma_second(leader, tmem + FT_O + nh * 128, pd, tc::sdesc_advance(vd, nh * 2 * PT_BLK), idesc, true);
        }
        pt_commit(leader, &ms.pv_done[b]);
        if (t + FT_NBUF < n_tiles) pt_commit(leader, &ms.v_free[kb]);
      }
    }
  } else {
    // =========================== softmax warps ===========================
    const int head = tid & 63, half = tid >> 6;
    const uint32_t lanes = (uint32_t)(warp * 32) << 16;
    const float sc2 = a.scale * LOG2E;
    auto wait_pv = [&](int t, int code) { ok = pt_wait(&ms.pv_done[t & 1], (t >> 1) & 1, abort_flag, code) && ok; };
    auto arrive_first = [&](uint64_t* bar) {               // one arrival a warp, at the first CTA's barrier
      __syncwarp();
      if (lane == 0) pt_arrive(first(bar));
    };
    {
      ok = tc::mbar_wait<FT_POLL_NS>(&ms.q_full, 0, abort_flag, 27) && ok;
      const uint8_t* src = smem + FS_K + 2 * FT_TILE;
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
      arrive_first(&ms.q_ready);
      if (lane == 0) tc::mbar_arrive(&ms.q_moved);
    }
    float m = -INFINITY, l = 0.f;
    for (int t = 0; t < n_tiles; t++) {
      const int b = t & 1;
      ok = pt_wait(&ms.s_full[b], (t >> 1) & 1, abort_flag, 28) && ok;
      tc::fence_after_sync();
      uint32_t sv[32];
      tc::tmem_ld32(tmem + FT_S + b * 32 + lanes, sv);
      tc::tmem_ld_wait();
      tc::fence_before_sync();
      arrive_first(&ms.s_free[b]);
      // keys of this thread: 32 half .. + 31 of the tile; the last tile is the second row's
      const int have = (t < whole || rank == 1 ? keys(t) : 0) - 32 * half;
      const uint32_t mask = have >= 32 ? 0xffffffffu : have <= 0 ? 0u : (1u << have) - 1u;
      float tmax = -INFINITY;
#pragma unroll
      for (int j = 0; j < 32; j++) {
        const float v = (mask >> j) & 1u ? __uint_as_float(sv[j]) * sc2 : -INFINITY;
        sv[j] = __float_as_uint(v);
        tmax = fmaxf(tmax, v);
      }
      ms.mx[b][tid] = tmax;
      asm volatile("bar.sync %0, 64;" ::"r"(1 + (warp & 1)) : "memory");
      tmax = fmaxf(tmax, ms.mx[b][tid ^ 64]);
      const bool move = tmax > m + RESCALE_THRESHOLD || (m == -INFINITY && tmax > -INFINITY);
      float alpha = 1.f;
      if (move) {
        alpha = m == -INFINITY ? 0.f : exp2f(m - tmax);
        m = tmax;
        l *= alpha;
      }
      if (t > 0 && __any_sync(0xffffffffu, move)) {
        wait_pv(t - 1, 29);
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
      if (t >= 2) wait_pv(t - 2, 30);                      // this parity's P has been read
      uint8_t* prow = smem + FS_P + b * FP_BYTES;
      const float mref = m == -INFINITY ? 0.f : m;
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
      ok = tc::mbar_wait<FT_POLL_NS>(&ms.v_here[t % FT_NBUF], (t / FT_NBUF) & 1, abort_flag, 33) && ok;   // this CTA's part of V
      tc::fence_async_smem();
      tc::fence_before_sync();
      arrive_first(&ms.p_full[b]);
    }
    // ---- the row's output: 2 x 64 channels at a time through the P buffers, thread half h has channels 256 h .. 256 h + 255 ----
    ms.l[tid] = l;
    if (n_tiles >= 2) wait_pv(n_tiles - 2, 36);
    wait_pv(n_tiles - 1, 31);
    tc::fence_after_sync();
    asm volatile("bar.sync 3, 128;" ::: "memory");
    l += ms.l[tid ^ 64];
    const float f = l > 0.f ? 1.f / l : 0.f;
#pragma unroll 1
    for (int c0 = 0; c0 < 256; c0 += 64) {
      uint8_t* box = smem + FS_P + half * FP_BYTES;
      if (tid == 0) tc::bulk_wait_read<0>();
      asm volatile("bar.sync 3, 128;" ::: "memory");
#pragma unroll
      for (int hc = 0; hc < 2; hc++) {
        uint32_t o[32];
        tc::tmem_ld32(tmem + FT_O + c0 + 32 * hc + lanes, o);
        tc::tmem_ld_wait();
#pragma unroll
        for (int v = 0; v < 4; v++) {
          uint4 w;
          uint32_t* wp = &w.x;
#pragma unroll
          for (int e = 0; e < 4; e++) {
            const float x0 = l > 0.f ? __uint_as_float(o[8 * v + 2 * e]) * f : 0.f, x1 = l > 0.f ? __uint_as_float(o[8 * v + 2 * e + 1]) * f : 0.f;
            const __half2 h2 = __floats2half2_rn(x0, x1);
            wp[e] = *reinterpret_cast<const uint32_t*>(&h2);
          }
          *reinterpret_cast<uint4*>(box + tc::sw128_off(head, hc * 4 + v, FT_BLK)) = w;
        }
      }
      tc::fence_async_smem();
      asm volatile("bar.sync 3, 128;" ::: "memory");
      if (tid == 0 && mine && ok && !*abort_flag) {
#pragma unroll
        for (int hf = 0; hf < 2; hf++)
          asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(&tmap_o), "r"(hf * 256 + c0),
                       "r"(row * FT_HEADS), "r"(tc::smem_u32(smem + FS_P + hf * FP_BYTES))
                       : "memory");
        tc::bulk_commit();
      }
    }
    if (tid == 0) tc::bulk_wait_read<0>();
  }
  // Behind a wait that gave up the loops above ran on: what they asked for ends first (far less than a millisecond).
  if (*abort_flag)
    for (const long long t0 = clock64(); clock64() - t0 < 4000000;) __nanosleep(1000);
  tc::fence_before_sync();
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");   // nothing of either CTA is in use any more
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  if (tid == 0 && ms.abort_flag && status) atomicExch(status, HK_ERR_TIMEOUT);
}

}  // namespace hk
