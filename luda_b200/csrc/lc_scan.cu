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
#include "lc_scan.cuh"

namespace lc {

namespace {
thread_local uint32_t t_launches = 0;
}  // namespace

void note_launch(uint32_t n) { t_launches += n; }
uint32_t launches_on_this_thread() { return t_launches; }

namespace {

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

template <int S, int kThreads, bool kDirect>
__global__ void __launch_bounds__(kThreads) k_tile_scan(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error || ScanOf<S>::out(J) == nullptr;
  __syncthreads();
  if (s_failed) return;
  tile_scan<S, kThreads, kDirect>(J, blockIdx.x, gridDim.x);
}

// Up to kDirectMax elements (by the caller's estimate; the kernel is right for
// any count): one launch with tiles of 8192, every CTA reading the elements
// before its tile, at most 16 tiles.  More: tile sums first.  At 80k elements
// one launch takes 4 us, two take 7.
constexpr uint64_t kDirectThreads = 1024;
static_assert(kDirectMax == 16 * kDirectThreads * kScanItems);

template <int S>
void launch_tile_sums(const Batch& bt, uint64_t n_est, cudaStream_t st) {
  launch(k_tile_reduce<S>, dim3(grid_x(n_est + 1, kTile, bt.per_job(148 * 8)), bt.B), kScanThreads, 0,
         st, bt.d);
}

template <int S>
void scan_sel(const Batch& bt, uint64_t n_est, cudaStream_t st) {
  if (n_est <= kDirectMax) {
    launch(k_tile_scan<S, kDirectThreads, true>,
           dim3(grid_x(n_est + 1, kDirectThreads * kScanItems, 16), bt.B), kDirectThreads, 0, st, bt.d);
    return;
  }
  const unsigned tiles = grid_x(n_est + 1, kTile, bt.per_job(148 * 8));
  launch_tile_sums<S>(bt, n_est, st);
  launch(k_tile_scan<S, kScanThreads, false>, dim3(tiles, bt.B), kScanThreads, 0, st, bt.d);
}

}  // namespace

void scan_batch(ScanSel sel, const Batch& bt, uint64_t n_est, cudaStream_t st) {
  switch (sel) {
    case kScanBlkEnt: scan_sel<kScanBlkEnt>(bt, n_est, st); break;
    case kScanBcum: scan_sel<kScanBcum>(bt, n_est, st); break;
    case kScanGcum: scan_sel<kScanGcum>(bt, n_est, st); break;
    case kScanIcum: scan_sel<kScanIcum>(bt, n_est, st); break;
    case kScanDecKey: scan_sel<kScanDecKey>(bt, n_est, st); break;
    case kScanKb: scan_sel<kScanKb>(bt, n_est, st); break;
  }
}

void tile_sums_kb(const Batch& bt, uint64_t n_est, cudaStream_t st) {
  launch_tile_sums<kScanKb>(bt, n_est, st);
}

// tile sums for arrays of up to n_cap elements: 8 bytes for every kTile of them
// here, 4 bytes for every 128 in the drop rule's counts
uint64_t scan_scratch_elems(uint64_t n_cap) { return (n_cap + 1) / 256 + 4; }
static_assert(kTile >= 256, "scan_scratch_elems");

namespace {

// Small control transfers (descriptors, counters, per-file results) between
// device memory and mapped pinned host memory, done by SM loads and stores
// over PCIe rather than by a copy engine.  A copy engine serves the streams'
// copies in turn, so with other jobs' bulk uploads and downloads in flight a
// few-KB cudaMemcpyAsync waited behind megabytes of them and held up its
// job's next kernels.  16-byte words, then the last bytes.
__global__ void k_xfer(uint8_t* dst, const uint8_t* src, uint64_t n) {
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
