// Pooled indexer key of one pool, one thread per channel (helios::attn::kpool_write, reference: src/cuda/attn/attn.cu:332-390).
// A pool key is produced by the call that writes the pool's LAST member; members written by earlier calls are read back
// from the ring, members of this call straight from the inputs (and copied into the ring for later calls).
#pragma once
#include "hk_common.cuh"

namespace hk {

// ik / ig: the call's new key and gate rows [n_new][128] (any address space); p = pool, c = channel.  Everything is requested
// before anything is used or stored: the ring may be the same memory for all the compiler knows, and load after store after
// load is four round trips.  before_keys() runs between: after it ik may be read.
template <class F>
__device__ __forceinline__ void kpool_one(const __half* ik, const __half* ig, __half* __restrict__ ring, int raw_rows,
                                          __half* __restrict__ pk_nt, const float* __restrict__ ape, int pos_start, int n_new,
                                          int p, int c, F before_keys) {
  const int t0 = p * POOL;
  const int last = t0 + POOL - 1;
  const bool complete = last >= pos_start && last < pos_start + n_new;
  __half hk[POOL], hg[POOL];
  float kk[POOL], gg[POOL];
  float mx = -1e30f;
  int slot = t0 % raw_rows;
  const int slot0 = slot;
#pragma unroll
  for (int i = 0; i < POOL; i++) {
    const int src = t0 + i - pos_start;
    const __half* r = ring + (size_t)slot * 256;
    hk[i] = hg[i] = __float2half(0.f);
    if (src >= 0 && src < n_new) {
      hg[i] = ig[(size_t)src * 128 + c];
    } else if (complete && src < 0) {
      hk[i] = r[c];
      hg[i] = r[128 + c];
    }
    gg[i] = complete ? ape[i * 128 + c] : 0.f;
    slot = slot + 1 == raw_rows ? 0 : slot + 1;
  }
  before_keys();
#pragma unroll
  for (int i = 0; i < POOL; i++) {
    const int src = t0 + i - pos_start;
    if (src >= 0 && src < n_new) hk[i] = ik[(size_t)src * 128 + c];
  }
  slot = slot0;
#pragma unroll
  for (int i = 0; i < POOL; i++) {
    const int src = t0 + i - pos_start;
    if (src >= 0 && src < n_new) {
      __half* r = ring + (size_t)slot * 256;
      r[c] = hk[i];
      r[128 + c] = hg[i];
    }
    kk[i] = __half2float(hk[i]);
    gg[i] = __half2float(hg[i]) + gg[i];
    mx = fmaxf(mx, gg[i]);
    slot = slot + 1 == raw_rows ? 0 : slot + 1;
  }
  if (!complete) return;
  float sum = 0.f;
#pragma unroll
  for (int i = 0; i < POOL; i++) {
    gg[i] = __expf(gg[i] - mx);
    sum += gg[i];
  }
  float o = 0.f;
#pragma unroll
  for (int i = 0; i < POOL; i++) o += (gg[i] / sum) * kk[i];
  o *= 0.25f;
  pk_nt[(size_t)p * 128 + c] = __float2half_rn(o);
}

}  // namespace hk
