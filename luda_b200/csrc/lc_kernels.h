// Host-callable launchers for the engine's kernels.
//
// Every kernel serves a batch of jobs in one launch: the grid's y dimension is
// the job index, and each kernel reads its job's descriptor from a device
// array (`jobs[blockIdx.y]`).  A plain compaction is a batch of one.  Launchers
// enqueue work on `st` and never synchronise; counts that are only known on
// the device are read by the kernels from each job's Counters, and grids are
// sized from host-side capacities (maxima over the batch).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "lc_job.h"

namespace lc {

// Sets the calling thread's lc_last_error() text.
void set_last_error(const std::string& msg);

// Kernel launches made by the calling thread (each batch runs on one thread).
void note_launch(uint32_t n = 1);
uint32_t launches_on_this_thread();

// Launches k so that it may be set up (its blocks placed, up to pdl_begin)
// while the kernel before it in the stream still runs: a job is a chain of
// some 20 to 35 kernels, most of a few microseconds, and a plain launch starts only
// when its predecessor has drained.  Every kernel launched so begins with
// pdl_begin(), and has no __restrict__ pointer to what its predecessor may still
// be writing (loads through one may be moved above the wait): the descriptors
// are one only where their upload cannot be the predecessor.  On B200, with chains
// of 49 kernels: an 800-entry job 288 -> 272 us a call, a 66 MiB job 756 -> 719 us.
// launch_clusters: the same, in thread-block clusters of `cluster` CTAs along x.
template <typename... P, typename... A>
inline void launch_clusters(unsigned cluster, void (*k)(P...), dim3 grid, unsigned threads,
                            size_t smem, cudaStream_t st, A... args) {
  cudaLaunchAttribute at[2] = {};
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = cluster;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cudaLaunchConfig_t c{};
  c.gridDim = grid;
  c.blockDim = dim3(threads);
  c.dynamicSmemBytes = smem;
  c.stream = st;
  c.attrs = at;
  c.numAttrs = cluster > 1 ? 2 : 1;
  cudaLaunchKernelEx(&c, k, P(args)...);
  note_launch();
}
template <typename... P, typename... A>
inline void launch(void (*k)(P...), dim3 grid, unsigned threads, size_t smem, cudaStream_t st,
                   A... args) {
  launch_clusters(1, k, grid, threads, smem, st, args...);
}

// Raise the dynamic shared-memory limits of the kernels that need more than
// 48 KiB; once per device, with that device current, before any launch or
// stream capture.
void decode_kernel_attributes();
void encode_kernel_attributes();
void merge_kernel_attributes();

// Survivors per chunk of the block chain (a CTA each): short chunks for batches
// too small to give every SM a long one, when blocks are expected (from the
// block size and the mean entry) to hold at most a quarter as many.  A job in
// which a block turns out longer than a short chunk goes by long ones
// (chain_chunk); blocks of more survivors than those are resolved one after
// the other.
constexpr uint32_t kChunk = 4096, kShortChunk = 1024;
// Chunks per group in the block-chain resolution.
constexpr uint32_t kChainGroup = 64;

// Block encoder (k_encode_blocks): a warp's shared-memory stage, the widest
// block assembled whole in it, and the windows of wider ones.  A block of z >
// kEncNarrow bytes has at most z / (kEncNarrow / 2) windows.
constexpr uint32_t kEncStage = 5120;
constexpr uint32_t kEncNarrow = kEncStage - 64;
constexpr uint32_t kEncWindow = 4608;  // whole 16-byte chunks, inside the stage

// Largest merge tile (threads x items) and the shared memory the tile takes
// per position.
constexpr uint32_t kMergeMaxTile = 4096;
constexpr uint32_t kMergeSmemPerPos = 14;

// Kernels that take a small job's steps in one launch: one cluster of CTAs per
// job (k_parse_blocks, k_partition).
constexpr uint32_t kPartThreads = 512, kPartMaxCtas = 8;
// Their CTAs: a power of two, a thread for every item or kPartMaxCtas.
inline unsigned part_ctas(uint64_t items) {
  unsigned c = 1;
  while ((uint64_t)c * kPartThreads < items && c < kPartMaxCtas) c *= 2;
  return c;
}

// k_scan_next: survivors after its tile that it keeps, and the largest entry
// and block size its 32-bit sums are for.
constexpr uint32_t kNextHalo = 512, kNextBig = 1u << 19;

struct Batch {
  const JobDev* d = nullptr;  // device array of B job descriptors
  uint32_t B = 0;
  // maxima over the batch, for grid sizes
  uint32_t max_tables = 0, max_gp = 0, max_cap_triggers = 0, max_cap_files = 0;
  uint64_t max_blocks_in = 0;  // data blocks, as the input's bytes suggest
  uint64_t max_entries = 0, max_cap_wide = 0;
  uint64_t max_blocks_out = 0;  // data blocks, as the bytes and the block size suggest
  uint64_t max_block_entries = 0;  // a block's entries, likewise (2^30: a block size past kNextBig)
  uint64_t max_dec_groups = 0, max_dec_units = 0;  // decode work units
  uint32_t merge_rounds = 0;
  uint32_t max_runs = 1;
  uint32_t chunk = kChunk;  // survivors per chunk of the block chain
  uint32_t chain_smem_words = 11 * 1024;
  bool any_verify = false;  // some job checks its input blocks' CRCs
  bool any_keep_decoded = false;  // some job keeps its outputs' decoded form
  // tunables (chosen by the autotuner in lc_engine.cu)
  uint32_t ctas_per_job = 0;  // grid x of the grid-stride kernels; 0 = from the sizes
  uint32_t merge_items = 8;   // outputs per thread in a merge round
  uint32_t merge_threads = 256;  // threads per merge CTA (tile = threads * items)
  // the batch's work in jobs of its largest one's size (>= 1)
  uint32_t jobs_of_largest = 1;
  // CTAs of one job for a kernel that `total` CTAs fill the device with: a job's
  // share by its size, were it the largest (the surplus of smaller ones exits
  // at once).  An equal share left the device to the largest jobs alone: a
  // batch of 32 jobs of 1-64 MiB 4223 -> 3119 us.
  unsigned per_job(unsigned total) const {
    if (ctas_per_job) return ctas_per_job;
    return total / jobs_of_largest ? total / jobs_of_largest : 1;
  }
};

// lc_scan.cu -- exclusive prefix sums over per-job arrays chosen by selector
enum ScanSel : int {
  kScanBlkEnt = 0,             // blk_nent -> blk_ent_base           (total: n_entries_in)
  kScanBcum,           // tmp32 -> b_cum
  kScanGcum,           // b_gbytes -> b_gcum
  kScanIcum,           // b_isize -> b_icum
  kScanDecKey,         // k_klen -> dec_kcum (jobs that keep their decoded form)
  kScanKb,             // k_b -> k_pb (block size estimates)
};
// n_est: about how many elements the longest job has (sizes the grid)
void scan_batch(ScanSel sel, const Batch& bt, uint64_t n_est, cudaStream_t st);
uint64_t scan_scratch_elems(uint64_t n_cap);
// the first of a long scan's two launches, for k_b (k_scan_next is the second)
void tile_sums_kb(const Batch& bt, uint64_t n_est, cudaStream_t st);

// lc_crc.cu -- masked CRC32C of one buffer; the kCrcScratchWords words of
// `scratch` must be zero at launch and are zero again when the kernel is done
void launch_crc32c_chunks(const uint8_t* data, uint64_t n, uint32_t* scratch, uint32_t* out,
                          cudaStream_t st);

// lc_decode.cu -- input tables -> decoded entries
void launch_table_index_count(const Batch& bt, cudaStream_t st);
void launch_table_index_entries(const Batch& bt, cudaStream_t st);
void launch_block_count(const Batch& bt, cudaStream_t st);     // exact key counts (full walk)
// entry counts from restart words and their sums, and what launch_parse_done does
void launch_parse_blocks(const Batch& bt, cudaStream_t st);
void launch_parse_done(const Batch& bt, cudaStream_t st);  // merge children's entries; counters out
// Checks the CRC32C trailer of every input data block of the jobs that ask
// for it (verify_checksums), after the block list is known.
void launch_verify_blocks(const Batch& bt, cudaStream_t st);
// Copies n bytes with a kernel (no copy engine); one side may be mapped
// pinned host memory given by its device alias.  False (nothing launched)
// unless both addresses are 16-byte aligned.
bool launch_xfer(void* dst, const void* src, uint64_t n, cudaStream_t st);
void launch_block_decode(const Batch& bt, cudaStream_t st);
void launch_entries_from_offsets(const Batch& bt, cudaStream_t st);

// lc_merge.cu -- merge, drop rule, grandparent cuts, survivors
// the keys' common bytes, entry prefixes after them, grandparent prefixes
void launch_key_skip(const Batch& bt, cudaStream_t st);
void launch_merge(const Batch& bt, cudaStream_t st);
void launch_drop(const Batch& bt, cudaStream_t st);
void launch_triggers(const Batch& bt, cudaStream_t st);
void launch_kept_compact(const Batch& bt, cudaStream_t st);  // survivors and their entry sizes

// lc_encode.cu -- survivors -> output tables
void launch_sizes(const Batch& bt, cudaStream_t st);       // flush encoder: entry sizes
// the survivors' blocks, files and index keys
void launch_partition(const Batch& bt, cudaStream_t st);
// data, filter and index blocks, metaindex, footer and file keys
void launch_encode_blocks(const Batch& bt, cudaStream_t st);
// the decoded form of the survivors, for jobs with keep_decoded
void launch_emit_decoded(const Batch& bt, cudaStream_t st);
// the trailers of the filter, metaindex and index blocks and of wide data blocks
void launch_encode_meta(const Batch& bt, cudaStream_t st);
// counters and per-file results to the jobs' host buffers (JobDev::res_*)
void launch_results(const Batch& bt, cudaStream_t st);

// grid x for a kernel over up to `items` items per job, `per` items per CTA,
// capped at `cap` CTAs (the kernel loops over the rest)
inline unsigned grid_x(uint64_t items, unsigned per, uint64_t cap) {
  uint64_t g = (items + per - 1) / per;
  if (g == 0) g = 1;
  if (g > cap) g = cap;
  return (unsigned)g;
}

}  // namespace lc
