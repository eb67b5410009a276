// Exclusive prefix sums of per-job arrays for a whole batch (grid y = job), in
// two launches: per-tile sums (scan_scratch; the scans of a job run one after
// another), then the scan of each tile from its offset, which every CTA sums
// from the tile sums before it.  Short arrays take the second launch alone,
// the offset summed from the elements.
//
// The array and its length are chosen by a selector from the job descriptor;
// the length lives in device memory, so a scan can be enqueued before the
// producing kernel's count is known on the host.  The grid is sized from a
// host-side estimate of the length; the kernels loop over the rest.  out has n+1
// entries: out[n] is the total, optionally also stored to a counter.
#include <cuda_runtime.h>
#include <algorithm>
#include <stdint.h>

#include "lc_device.cuh"
#include "lc_kernels.h"

namespace lc {

namespace {
thread_local uint32_t t_launches = 0;
}  // namespace

void note_launch(uint32_t n) { t_launches += n; }
uint32_t launches_on_this_thread() { return t_launches; }

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr int kTile = kScanThreads * kScanItems;

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
struct ScanOf<kScanBlkKey> {
  using TI = uint64_t;
  using TO = uint64_t;
  static __device__ const TI* in(const JobDev& J) { return J.blk_kbytes; }
  static __device__ TO* out(const JobDev& J) { return J.blk_key_base; }
  static __device__ uint64_t n(const JobDev& J) { return min(J.ctr->n_blocks_in, J.cap_blocks_in); }
  static __device__ uint64_t* total(const JobDev& J) { return &J.ctr->key_bytes_in; }
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

template <int S>
__global__ void k_tile_reduce(const JobDev* __restrict__ jobs) {
  pdl_begin();
  using SP = ScanOf<S>;
  using TO = typename SP::TO;
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error || SP::out(J) == nullptr;
  __syncthreads();
  if (s_failed) return;
  const uint64_t n = SP::n(J);
  TO* tile_sums = reinterpret_cast<TO*>(J.scan_scratch);
  for (uint64_t t = blockIdx.x; t * kTile <= n; t += gridDim.x) {
    const TO total = block_sum<TO>(SP::in(J), t * kTile, min(n, (t + 1) * kTile));
    if (threadIdx.x == 0) tile_sums[t] = total;
  }
}

// kDirect: no tile sums; a CTA sums the elements before its tile itself.
template <int S, int kThreads, bool kDirect>
__global__ void __launch_bounds__(kThreads) k_tile_scan(const JobDev* __restrict__ jobs) {
  pdl_begin();
  using SP = ScanOf<S>;
  using TO = typename SP::TO;
  constexpr uint64_t kT = (uint64_t)kThreads * kScanItems;
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error || SP::out(J) == nullptr;
  __syncthreads();
  if (s_failed) return;
  const uint64_t n = SP::n(J);
  if (blockIdx.x * kT > n) return;
  const TO* tile_sums = reinterpret_cast<const TO*>(J.scan_scratch);
  const typename SP::TI* in = SP::in(J);
  TO* out = SP::out(J);
  uint64_t* total_out = SP::total(J);
  // offset of this CTA's first tile; each step of the grid stride adds the
  // tiles it skips
  const auto before = [&](uint64_t t0, uint64_t t1) -> TO {  // tiles [t0, t1)
    if constexpr (kDirect) return block_sum<TO>(in, t0 * kT, min(n, t1 * kT));
    TO x = 0, total;
    for (uint64_t i = t0 + threadIdx.x; i < t1; i += blockDim.x) x += tile_sums[i];
    block_excl_scan<TO>(x, &total);
    return total;
  };
  TO carry = before(0, blockIdx.x);
  for (uint64_t t = blockIdx.x; t * kT <= n; t += gridDim.x) {
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
    if ((t + gridDim.x) * kT <= n) {  // another tile of this CTA follows
      carry += before(t, t + gridDim.x);
    }
  }
}

// Up to kDirectMax elements (by the caller's estimate; the kernel is right for
// any count): one launch with tiles of 8192, every CTA reading the elements
// before its tile, at most 16 tiles.  More: tile sums first.  At 80k elements
// one launch takes 4 us, two take 7.
constexpr uint64_t kDirectThreads = 1024;
constexpr uint64_t kDirectMax = 16 * kDirectThreads * kScanItems;

template <int S>
void scan_sel(const Batch& bt, uint64_t n_est, cudaStream_t st) {
  if (n_est <= kDirectMax) {
    launch(k_tile_scan<S, kDirectThreads, true>,
           dim3(grid_x(n_est + 1, kDirectThreads * kScanItems, 16), bt.B), kDirectThreads, 0, st, bt.d);
    return;
  }
  const unsigned tiles = grid_x(n_est + 1, kTile, bt.per_job(148 * 8));
  launch(k_tile_reduce<S>, dim3(tiles, bt.B), kScanThreads, 0, st, bt.d);
  launch(k_tile_scan<S, kScanThreads, false>, dim3(tiles, bt.B), kScanThreads, 0, st, bt.d);
}

}  // namespace

void scan_batch(ScanSel sel, const Batch& bt, uint64_t n_est, cudaStream_t st) {
  switch (sel) {
    case kScanBlkEnt: scan_sel<kScanBlkEnt>(bt, n_est, st); break;
    case kScanBlkKey: scan_sel<kScanBlkKey>(bt, n_est, st); break;
    case kScanBcum: scan_sel<kScanBcum>(bt, n_est, st); break;
    case kScanGcum: scan_sel<kScanGcum>(bt, n_est, st); break;
    case kScanIcum: scan_sel<kScanIcum>(bt, n_est, st); break;
    case kScanDecKey: scan_sel<kScanDecKey>(bt, n_est, st); break;
    case kScanKb: scan_sel<kScanKb>(bt, n_est, st); break;
  }
}

// tile sums for arrays of up to n_cap elements: 8 bytes for every kTile of them
// here, 4 bytes for every 512 in the drop rule's counts
uint64_t scan_scratch_elems(uint64_t n_cap) { return (n_cap + 1) / 1024 + 4; }
static_assert(kTile >= 1024, "scan_scratch_elems");

namespace {

// Small control transfers (descriptors, counters, per-file results) between
// device memory and mapped pinned host memory, done by SM loads and stores
// over PCIe rather than by a copy engine.  A copy engine serves the streams'
// copies in turn, so with other jobs' bulk uploads and downloads in flight a
// few-KB cudaMemcpyAsync waited behind megabytes of them and held up its
// job's next kernels.  16-byte words, then the last bytes.
__global__ void k_xfer(uint8_t* __restrict__ dst, const uint8_t* __restrict__ src, uint64_t n) {
  pdl_begin();
  const uint64_t n16 = n / 16;
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  for (uint64_t i = t; i < n16; i += stride)
    reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
  for (uint64_t i = n16 * 16 + t; i < n; i += stride) dst[i] = src[i];
}

}  // namespace

bool launch_xfer(void* dst, const void* src, uint64_t n, cudaStream_t st) {
  if (((uintptr_t)dst | (uintptr_t)src) & 15) return false;
  if (!n) return true;
  const uint64_t words = n / 16 + 1;
  const unsigned grid = (unsigned)std::min<uint64_t>((words + 255) / 256, 148);
  launch(k_xfer, dim3(grid), 256, 0, st, (uint8_t*)dst, (const uint8_t*)src, n);
  return true;
}

}  // namespace lc
