// Exclusive prefix sums of per-job arrays: what is scanned, and the work of one
// CTA (lc_scan.cu says how the sums are split over CTAs and launches).
#pragma once
#include <stdint.h>

#include "lc_device.cuh"
#include "lc_kernels.h"

namespace lc {
namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kTile = kScanThreads * kScanItems;
constexpr uint64_t kDirectMax = 131072;  // elements scanned without tile sums (lc_scan.cu)

template <int S>
struct ScanOf;
template <>
struct ScanOf<kScanBlkEnt> {
  using TI = uint32_t;
  using TO = uint64_t;
  static __device__ const TI* in(const JobDev& J) { return J.blk_nent; }
  static __device__ TO* out(const JobDev& J) { return J.blk_ent_base; }
  static __device__ uint64_t n(const JobDev& J) { return min(J.ctr->n_blocks_in, J.cap_blocks_in); }
  static __device__ uint64_t* total(const JobDev& J) { return &J.ctr->n_entries_in; }
};
template <>
struct ScanOf<kScanBcum> {
  using TI = uint32_t;
  using TO = uint64_t;
  static __device__ const TI* in(const JobDev& J) { return J.tmp32; }
  static __device__ TO* out(const JobDev& J) { return J.b_cum; }
  static __device__ uint64_t n(const JobDev& J) { return J.ctr->n_blocks_out; }
  static __device__ uint64_t* total(const JobDev&) { return nullptr; }
};
template <>
struct ScanOf<kScanGcum> {
  using TI = uint32_t;
  using TO = uint64_t;
  static __device__ const TI* in(const JobDev& J) { return J.b_gbytes; }
  static __device__ TO* out(const JobDev& J) { return J.b_gcum; }
  static __device__ uint64_t n(const JobDev& J) { return J.ctr->n_blocks_out; }
  static __device__ uint64_t* total(const JobDev&) { return nullptr; }
};
template <>
struct ScanOf<kScanIcum> {
  using TI = uint32_t;
  using TO = uint64_t;
  static __device__ const TI* in(const JobDev& J) { return J.b_isize; }
  static __device__ TO* out(const JobDev& J) { return J.b_icum; }
  static __device__ uint64_t n(const JobDev& J) { return J.ctr->n_blocks_out; }
  static __device__ uint64_t* total(const JobDev&) { return nullptr; }
};

template <>
struct ScanOf<kScanDecKey> {
  using TI = uint32_t;
  using TO = uint64_t;
  static __device__ const TI* in(const JobDev& J) { return J.k_klen; }
  static __device__ TO* out(const JobDev& J) { return J.dec_kcum; }  // null: job skipped
  static __device__ uint64_t n(const JobDev& J) { return J.ctr->n_kept; }
  static __device__ uint64_t* total(const JobDev&) { return nullptr; }
};

template <>
struct ScanOf<kScanKb> {
  using TI = uint32_t;
  using TO = uint64_t;
  static __device__ const TI* in(const JobDev& J) { return J.k_b; }
  static __device__ TO* out(const JobDev& J) { return J.k_pb; }
  static __device__ uint64_t n(const JobDev& J) { return J.ctr->n_kept; }
  static __device__ uint64_t* total(const JobDev&) { return nullptr; }
};

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Exclusive scan across the CTA; returns the exclusive prefix, *total = sum.
// The total has its own slot: with 32 warps every one of warp_sums[0..31]
// holds a warp's exclusive prefix.
template <typename T>
__device__ __forceinline__ T block_excl_scan(T v, T* total) {
  __shared__ T warp_sums[33];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nwarps = (blockDim.x + 31) >> 5;
  T incl = warp_incl_scan(v);
  if (lane == 31) warp_sums[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    T w = lane < nwarps ? warp_sums[lane] : T(0);
    T wi = warp_incl_scan(w);
    if (lane < nwarps) warp_sums[lane] = wi - w;
    if (lane == 31) warp_sums[32] = wi;  // lanes past nwarps add nothing
  }
  __syncthreads();
  T res = warp_sums[warp] + incl - v;
  *total = warp_sums[32];
  __syncthreads();
  return res;
}

// Eight consecutive elements from i (a multiple of 8) as 16-byte loads
// (every scanned array starts on a 256-byte boundary); elements at or past n
// read as zero.
template <typename TI, typename TO>
__device__ __forceinline__ void load8(const TI* in, uint64_t i, uint64_t n, TO (&v)[8]) {
  if (i + 8 <= n) {
    constexpr int kB = 8 * sizeof(TI);
    if constexpr (kB == 8) {
      const uint64_t w = *reinterpret_cast<const uint64_t*>(in + i);
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = (TO)((w >> (8 * k)) & 0xff);
    } else {
      alignas(16) TI x[8];
#pragma unroll
      for (int k = 0; k < kB / 16; k++)
        reinterpret_cast<uint4*>(x)[k] = reinterpret_cast<const uint4*>(in + i)[k];
#pragma unroll
      for (int k = 0; k < 8; k++) v[k] = (TO)x[k];
    }
  } else {
#pragma unroll
    for (int k = 0; k < 8; k++) v[k] = i + k < n ? (TO)in[i + k] : TO(0);
  }
}

// Sum of in[lo, hi) over the CTA (every thread gets it); lo a multiple of 8.
template <typename TO, typename TI>
__device__ __forceinline__ TO block_sum(const TI* in, uint64_t lo, uint64_t hi) {
  TO s = 0;
  for (uint64_t i = lo + 8 * threadIdx.x; i < hi; i += 8 * blockDim.x) {
    TO v[8];
    load8<TI, TO>(in, i, hi, v);
#pragma unroll
    for (int k = 0; k < 8; k++) s += v[k];
  }
  TO total;
  block_excl_scan<TO>(s, &total);
  return total;
}

// Sum over the CTA of the elements in tiles [t0, t1) of kT elements: from the
// elements (kDirect) or the tile sums.
template <typename TO, bool kDirect, typename TI>
__device__ __forceinline__ TO tiles_sum(const TI* in, const TO* tile_sums, uint64_t t0, uint64_t t1,
                                        uint64_t kT, uint64_t n) {
  if (t0 == t1) return 0;
  if constexpr (kDirect) return block_sum<TO>(in, t0 * kT, min(n, t1 * kT));
  TO x = 0, total;
  for (uint64_t i = t0 + threadIdx.x; i < t1; i += blockDim.x) x += tile_sums[i];
  block_excl_scan<TO>(x, &total);
  return total;
}

// CTA `cta` of `ctas` (of kThreads threads) of the scan of one job's array.
// kDirect: no tile sums; a CTA sums the elements before its tile itself.
template <int S, int kThreads, bool kDirect>
__device__ __forceinline__ void tile_scan(const JobDev& J, uint32_t cta, uint32_t ctas) {
  using SP = ScanOf<S>;
  using TO = typename SP::TO;
  constexpr uint64_t kT = (uint64_t)kThreads * kScanItems;
  const uint64_t n = SP::n(J);
  if (cta * kT > n) return;
  const TO* tile_sums = reinterpret_cast<const TO*>(J.scan_scratch);
  const typename SP::TI* in = SP::in(J);
  TO* out = SP::out(J);
  uint64_t* total_out = SP::total(J);
  // offset of this CTA's first tile; each step of the grid stride adds the
  // tiles it skips
  const auto before = [&](uint64_t t0, uint64_t t1) -> TO {
    return tiles_sum<TO, kDirect>(in, tile_sums, t0, t1, kT, n);
  };
  TO carry = before(0, cta);
  for (uint64_t t = cta; t * kT <= n; t += ctas) {
    const uint64_t tb = t * kT + (uint64_t)threadIdx.x * kScanItems;
    alignas(16) TO v[8];
    load8<typename SP::TI, TO>(in, tb, n, v);
    TO s = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) {
      const TO x = v[k];
      v[k] = s;
      s += x;
    }
    TO total;
    const TO ex = block_excl_scan<TO>(s, &total) + carry;
#pragma unroll
    for (int k = 0; k < kScanItems; k++) v[k] += ex;
    if (tb + kScanItems <= n) {
#pragma unroll
      for (int k = 0; k < (int)(kScanItems * sizeof(TO) / 16); k++)
        reinterpret_cast<uint4*>(out + tb)[k] = reinterpret_cast<const uint4*>(v)[k];
    } else {
#pragma unroll
      for (int k = 0; k < kScanItems; k++)
        if (tb + k < n) out[tb + k] = v[k];
    }
    if (tb <= n && n < tb + kScanItems) {  // the total after the last element
      TO all = ex + s;  // (elements past n are zero)
      out[n] = all;
      if (total_out) *total_out = (uint64_t)all;
    }
    if ((t + ctas) * kT <= n) {  // another tile of this CTA follows
      carry += before(t, t + ctas);
    }
  }
}

}  // namespace
}  // namespace lc
