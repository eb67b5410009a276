// Encode: survivors -> output tables, byte-identical to the reference's
// TableBuilder driven by DoCompactionWork.
//
// Reference behaviour reproduced here:
// * BlockBuilder (table/block_builder.cc:56-114): prefix compression against
//   the previous key of the block, a restart every `restart_interval` entries,
//   LUDA restart words (offset << 8) | run length, size estimate
//   buffer + 4 * restarts + 4.
// * TableBuilder::Add / Flush (table/table_builder.cc:94-140): a block is
//   flushed as soon as the estimate reaches block_size after an add.
// * DoCompactionWork's output split (db/db_impl.cc:1105-1111, 1174-1180): a
//   file ends once its flushed bytes (blocks + 5-byte trailers) reach
//   max_file_size, or before the first survivor at or after a grandparent cut.
// * Index block (table_builder.cc:101-108, 228-234): restart interval 1, one
//   entry per block keyed by FindShortestSeparator / FindShortSuccessor
//   (db/dbformat.cc:69-101, util/comparator.cc:29-64).
// * Filter block (table/filter_block.cc:21-76, util/bloom.cc:28-54): one
//   bloom filter per 2 KiB of data-block start offsets over the user keys of
//   the blocks that start there; empty filters for skipped indices.
// * Metaindex, footer (table_builder.cc:213-252, table/format.cc:31-40) and
//   masked CRC32C trailers (table_builder.cc:178-195).
//
// Block boundaries form a chain: where the next block starts depends on where
// this one started (restart positions and the prefix-compression reset).  Each
// survivor s gets next(s), the start of the following block if a block began
// at s.  The chain from survivor 0 is resolved in three steps: per chunk of
// survivors, a table of exits for every possible entry point (pointer chasing
// in shared memory), with the blocks started on the way; one thread composing
// the tables across chunks; and a per-chunk chase from the resolved entry
// point that writes the block starts.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "lc_device.cuh"
#include "lc_kernels.h"
#include "lc_scan.cuh"

namespace lc {

namespace {

constexpr uint32_t kNoSep = 0xffffffffu;
constexpr uint32_t kEncWarps = 16;
constexpr uint32_t kEncAhead = 32;  // entries of the next block copied ahead
constexpr uint32_t kEncLong = 33;   // values at least this long: by lane groups

__constant__ char kFilterName[] = "filter.leveldb.BuiltinBloomFilter2";
constexpr uint32_t kFilterNameLen = 34;

template <typename T>
__device__ __forceinline__ T warp_excl(T v, T* total) {
  const int lane = threadIdx.x & 31;
  T x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  *total = __shfl_sync(0xffffffffu, x, 31);
  return x - v;
}

__device__ __forceinline__ uint32_t bloom_bytes(uint64_t n, int bpk) {
  uint64_t bits = n * (uint64_t)bpk;
  if (bits < 64) bits = 64;
  return (uint32_t)((bits + 7) / 8);
}

__device__ __forceinline__ const uint8_t* kept_key(const JobDev& J, uint64_t k, uint32_t* len) {
  *len = J.k_klen[k];
  return J.keys + J.k_koff[k];
}

// The flush encoder's entry sizes: as a restart entry (k_a) and as a
// prefix-compressed entry (k_b), the shared prefix with the previous entry,
// byte totals.  (k_kept_compact computes a compaction's.)
__global__ void __launch_bounds__(256, 8) k_sizes(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // a failed job does no more work
  const uint64_t n = J.ctr->n_kept;
  unsigned long long kb = 0, vb = 0;
  for (uint64_t k0 = (uint64_t)blockIdx.x * blockDim.x; k0 < n; k0 += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t k = k0 + threadIdx.x;
    if (k >= n) continue;
    uint32_t kl;
    const uint8_t* key = kept_key(J, k, &kl);
    const uint32_t vl = J.k_vlen[k];
    uint32_t shared = 0;
    if (k > 0) {
      uint32_t pl;
      const uint8_t* pk = kept_key(J, k - 1, &pl);
      const uint32_t m = min(kl, pl);
      while (shared < m && pk[shared] == key[shared]) shared++;
    }
    J.k_a[k] = 1 + varint_len(kl) + varint_len(vl) + kl + vl;
    J.k_b[k] = varint_len(shared) + varint_len(kl - shared) + varint_len(vl) + (kl - shared) + vl;
    J.k_shared[k] = shared;
    kb += kl;
    vb += vl;
  }
  // survivor byte totals, one atomic per warp
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    kb += __shfl_xor_sync(0xffffffffu, kb, o);
    vb += __shfl_xor_sync(0xffffffffu, vb, o);
  }
  if ((threadIdx.x & 31) == 0 && (kb | vb)) {
    atomicAdd((unsigned long long*)&J.ctr->kept_key_bytes, kb);
    atomicAdd((unsigned long long*)&J.ctr->kept_value_bytes, vb);
  }
}

// TableBuilder's size estimate of a block [s, e] (buffer + 4 per restart +
// 4): the prefix-compressed sizes (k_pb, a prefix sum of k_b) plus, at every
// restart s + mR, the difference between the entry's restart size and its
// compressed size, plus the restart words.  `D` is that difference summed
// over the restarts up to segment m (the segment holding e).
struct BlockEst {
  const uint64_t* pb;
  const uint32_t *a, *b, *cuts;
  uint32_t R, ncuts;
  uint64_t bs;
  __device__ __forceinline__ explicit BlockEst(const JobDev& J)
      : pb(J.k_pb), a(J.k_a), b(J.k_b), cuts(J.t_kept), R(J.restart_interval),
        ncuts(J.ctr->n_triggers), bs(J.block_size) {}
  __device__ __forceinline__ uint64_t est(uint64_t s, uint64_t e, uint64_t D, uint64_t m) const {
    return pb[e + 1] - pb[s] + D + 4 * (m + 1) + 4;
  }
};

// next(s): the first survivor of the block after the one that starts at s.
// The block ends after the first e whose estimate reaches block_size
// (TableBuilder::Add, table/table_builder.cc:120-123), or before the first
// grandparent cut after s, or at the end.  Restart segments (R survivors)
// are stepped through, then the segment that reaches block_size is binary
// searched: O(block / R + log R) loads instead of a walk over the block.
__device__ __forceinline__ uint64_t next_of(const BlockEst& B, uint64_t s, uint64_t n) {
  const uint32_t R = B.R;
  uint32_t lo = 0, hi = B.ncuts;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (B.cuts[mid] <= s) lo = mid + 1;
    else hi = mid;
  }
  const uint64_t limit = lo < B.ncuts ? min(n, (uint64_t)B.cuts[lo]) : n;
  uint64_t D = 0;
  for (uint64_t m = 0;; m++) {
    const uint64_t a = s + m * R;
    if (a >= limit) return limit;
    D += B.a[a] - B.b[a];
    const uint64_t z = min(a + R, limit);  // segment [a, z)
    if (B.est(s, z - 1, D, m) >= B.bs) {
      uint64_t l = a, h = z - 1;
      while (l < h) {
        const uint64_t mid = (l + h) >> 1;
        if (B.est(s, mid, D, m) >= B.bs) h = mid;
        else l = mid + 1;
      }
      return l + 1;
    }
  }
}

__device__ __forceinline__ void next(const JobDev& J, uint32_t cta, uint32_t ctas) {
  const uint64_t n = J.ctr->n_kept;
  const BlockEst B(J);
  uint32_t* const out = J.k_next;
  const uint64_t stride = (uint64_t)ctas * blockDim.x;
  const uint64_t s0 = (uint64_t)cta * blockDim.x + threadIdx.x;
  const uint64_t w0 = s0 - (threadIdx.x & 31);
  const uint64_t trips = n > w0 ? (n - w0 + stride - 1) / stride : 0;
  uint32_t jump = 0;
  for (uint64_t it = 0, s = s0; it < trips; it++, s += stride) {
    if (s < n) {
      const uint64_t nxt = next_of(B, s, n);
      out[s] = (uint32_t)nxt;
      jump = max(jump, (uint32_t)(nxt - s));
    }
  }
  // the longest block, one atomic per warp
  jump = __reduce_max_sync(0xffffffffu, jump);
  if ((threadIdx.x & 31) == 0 && jump) atomicMax(&J.ctr->max_jump, jump);
}

__global__ void __launch_bounds__(256, 6) k_next(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // a failed job does no more work
  next(J, blockIdx.x, gridDim.x);
}

// k_pb and next() in one: a CTA scans a tile of k_b (the second launch of the
// long scan), keeps the sums of the tile and of the
// kNextHalo survivors after it in shared memory and finds next() from them.
// Blocks that reach beyond are followed a span at a time (next_beyond; walked
// entry by entry, 1M entries of which nine tenths were empty values in 32 KiB
// blocks of 2730 took 7319 us for the partition phase, so 510).
//
// The searches read k_pb (8 bytes a survivor) and k_a, k_b from memory before,
// about 14 dependent loads a survivor: 8M survivors in blocks of 66, the scan's
// second launch 33 and k_next 140 us, this kernel 76; 4M survivors in 32 jobs, 64
// and 38 us.  For up to kDirectMax survivors a scan of one launch and k_next
// take 13 us, a form of this kernel that summed the survivors before its tile
// itself 22.  Blocks of more than kNextHalo / 2 entries on average (many would
// reach past the halo) stay with k_next too.
constexpr uint32_t kNextSpan = kTile + kNextHalo;
static_assert((uint64_t)kNextSpan * kNextBig + 2 * kNextBig < 1ull << 31);

// The end of the range that a block from survivor s may cover: the first
// grandparent cut after s, or n.
__device__ __forceinline__ uint64_t next_limit(const uint32_t* cuts, uint32_t ncuts, uint64_t s, uint64_t n) {
  uint32_t lo = 0, hi = ncuts;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    if (cuts[mid] <= s) lo = mid + 1;
    else hi = mid;
  }
  return lo < ncuts ? min(n, (uint64_t)cuts[lo]) : n;
}

// next() of the survivors of the tile at t0 that have none yet (0), those whose
// block reaches past what k_scan_next holds.  The CTA takes the survivors from
// t0 on a span at a time and keeps where each search stands, the next restart
// (from t0) in tmp32 and the bytes still missing in b_size, both free until the
// blocks are sized.  Entries count as at most kNextBig bytes, which ends any
// block that reaches them (block sizes are at most that).
__device__ __forceinline__ void next_beyond(const JobDev& J, uint64_t t0, uint32_t* s_pb, uint32_t* s_d) {
  constexpr uint32_t kPer = kNextSpan / kScanThreads;
  const uint64_t n = J.ctr->n_kept;
  const uint32_t here = (uint32_t)min(n - t0, (uint64_t)kTile);
  const uint32_t R = J.restart_interval, ncuts = J.ctr->n_triggers;
  const uint32_t *const ka = J.k_a, *const kb = J.k_b, *const cuts = J.t_kept;
  uint32_t *const out = J.k_next, *const at = J.tmp32, *const rem = J.b_size;
  uint32_t jump = 0;
  bool left = false;
  for (uint32_t i = threadIdx.x; i < here; i += kScanThreads) left |= out[t0 + i] == 0;
  for (uint32_t w = 0; __syncthreads_or(left); w += kNextSpan) {
    const uint64_t w0 = t0 + w;
    const uint32_t len = (uint32_t)min(n - w0, (uint64_t)kNextSpan);
    uint32_t sum = 0, total;
    for (uint32_t k = kPer * threadIdx.x; k < kPer * (threadIdx.x + 1); k++) {
      const uint32_t b = k < len ? min(kb[w0 + k], kNextBig) : 0;
      s_d[k] = (k < len ? min(ka[w0 + k], kNextBig) : 0) - b;
      s_pb[k] = sum;
      sum += b;
    }
    const uint32_t ex = block_excl_scan<uint32_t>(sum, &total);
    for (uint32_t k = kPer * threadIdx.x; k < kPer * (threadIdx.x + 1); k++) s_pb[k] += ex;
    if (threadIdx.x == 0) s_pb[kNextSpan] = total;
    __syncthreads();
    left = false;
    for (uint32_t i = threadIdx.x; i < here; i += kScanThreads) {
      if (out[t0 + i]) continue;
      const uint64_t limit = next_limit(cuts, ncuts, t0 + i, n);
      const uint32_t end = (uint32_t)min(limit - t0, (uint64_t)w + len);  // searched up to here
      uint32_t cur = w ? w : i, x = w ? at[t0 + i] : i, nxt = 0;
      uint32_t need = (w ? rem[t0 + i] : (uint32_t)J.block_size - 4) + s_pb[cur - w];
      while (cur < end) {
        if (cur == x) {
          need -= s_d[cur - w] + 4;
          x += R;
        }
        const uint32_t z = min(x, end);
        if ((int32_t)(s_pb[z - w] - need) >= 0) {
          uint32_t l = cur, r = z - 1;
          while (l < r) {
            const uint32_t mid = (l + r) >> 1;
            if ((int32_t)(s_pb[mid + 1 - w] - need) >= 0) r = mid;
            else l = mid + 1;
          }
          nxt = l + 1;
          break;
        }
        cur = z;
      }
      if (!nxt && t0 + end == limit) nxt = end;
      if (nxt) {
        out[t0 + i] = (uint32_t)t0 + nxt;
        jump = max(jump, nxt - i);
      } else {
        at[t0 + i] = x;
        rem[t0 + i] = need - s_pb[end - w];
        left = true;
      }
    }
  }
  if (jump) atomicMax(&J.ctr->max_jump, jump);
}

__global__ void __launch_bounds__(kScanThreads, 5) k_scan_next(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  constexpr uint32_t kSpan = kNextSpan, kHaloItems = kNextHalo / kScanThreads;
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  // sums of k_b from the tile's first survivor (not used if an entry of the span
  // has more than kNextBig bytes), restarts' extra bytes
  __shared__ __align__(16) uint32_t s_pb[kSpan + 1], s_d[kSpan];
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  const uint64_t n = J.ctr->n_kept;
  if ((uint64_t)blockIdx.x * kTile > n) return;
  const uint64_t* tile_sums = reinterpret_cast<const uint64_t*>(J.scan_scratch);
  const uint32_t *const ka = J.k_a, *const kb = J.k_b, *const cuts = J.t_kept;
  uint64_t* const pb = J.k_pb;
  uint32_t* const out = J.k_next;
  const uint32_t R = J.restart_interval, ncuts = J.ctr->n_triggers;
  const uint32_t bs = (uint32_t)J.block_size;
  uint64_t carry = tiles_sum<uint64_t, false>(kb, tile_sums, 0, blockIdx.x, kTile, n);
  uint32_t jump = 0;
  bool left = false;
  for (uint64_t t = blockIdx.x; t * kTile <= n; t += gridDim.x) {
    const uint64_t t0 = t * kTile;
    const uint32_t avail = (uint32_t)min(n - t0, (uint64_t)kSpan);
    const uint32_t i0 = threadIdx.x * kScanItems;
    bool big = false;
    uint32_t v[kScanItems], h[kHaloItems], hs = 0;
    uint64_t s = 0;
    {
      uint32_t a[kScanItems];
      load8<uint32_t, uint32_t>(kb, t0 + i0, n, v);
      load8<uint32_t, uint32_t>(ka, t0 + i0, n, a);
#pragma unroll
      for (uint32_t k = 0; k < kHaloItems; k++) {
        const uint32_t i = kTile + threadIdx.x * kHaloItems + k;
        const uint32_t x = i < avail ? ka[t0 + i] : 0;
        h[k] = i < avail ? kb[t0 + i] : 0;
        s_d[i] = x - h[k];
        big |= x > kNextBig;
        hs += h[k];
      }
#pragma unroll
      for (int k = 0; k < kScanItems; k++) {
        s_d[i0 + k] = a[k] - v[k];
        big |= a[k] > kNextBig;
        s += v[k];
      }
    }
    uint64_t total;
    uint32_t htotal;
    uint64_t ex = block_excl_scan<uint64_t>(s, &total);
    uint32_t hx = block_excl_scan<uint32_t>(hs, &htotal) + (uint32_t)total;
#pragma unroll
    for (uint32_t k = 0; k < kHaloItems; k++) {
      s_pb[kTile + threadIdx.x * kHaloItems + k] = hx;
      hx += h[k];
    }
    if (threadIdx.x == 0) s_pb[kSpan] = (uint32_t)total + htotal;
    const uint64_t tb = t0 + i0;
    {
      uint32_t r = (uint32_t)ex;
#pragma unroll
      for (int k = 0; k < kScanItems; k++) {
        s_pb[i0 + k] = r;
        r += v[k];
      }
    }
    ex += carry;
    if (tb <= n && n < tb + kScanItems) pb[n] = ex + s;  // (survivors past n add nothing)
#pragma unroll
    for (int k = 0; k < kScanItems; k += 2) {
      const uint64_t e1 = ex + v[k];
      if (tb + k + 2 <= n)
        *reinterpret_cast<ulonglong2*>(pb + tb + k) = make_ulonglong2(ex, e1);
      else if (tb + k < n)
        pb[tb + k] = ex;
      ex = e1 + v[k + 1];
    }
    const bool over = __syncthreads_or(big);
    const uint32_t here = (uint32_t)min(n - t0, (uint64_t)kTile);
    for (uint32_t i = threadIdx.x; i < here; i += kScanThreads) {
      const uint64_t limit = next_limit(cuts, ncuts, t0 + i, n);
      const uint32_t last = over ? 0 : (uint32_t)min(limit - t0, (uint64_t)avail);  // searched up to here
      // as next_of: the restart segment that reaches the block size, then the entry
      uint32_t nxt = 0;                // from the tile's first survivor
      uint32_t need = bs + s_pb[i] - 4;  // less the restarts' extra bytes and words, and the count's
      for (uint32_t x = i; x < last; x += R) {
        need -= s_d[x] + 4;
        const uint32_t z = min(x + R, last);
        if ((int32_t)(s_pb[z] - need) >= 0) {
          uint32_t l = x, r = z - 1;
          while (l < r) {
            const uint32_t mid = (l + r) >> 1;
            if ((int32_t)(s_pb[mid + 1] - need) >= 0) r = mid;
            else l = mid + 1;
          }
          nxt = l + 1;
          break;
        }
      }
      if (!nxt && t0 + last == limit) nxt = last;
      out[t0 + i] = nxt ? (uint32_t)t0 + nxt : 0;
      if (nxt) jump = max(jump, nxt - i);
      else left = true;
    }
    __syncthreads();  // the tile's sums have been read
    if ((t + gridDim.x) * kTile <= n)
      carry += tiles_sum<uint64_t, false>(kb, tile_sums, t, t + gridDim.x, kTile, n);
  }
  if (__syncthreads_or(left))
    for (uint64_t t = blockIdx.x; t * kTile < n; t += gridDim.x) next_beyond(J, t * kTile, s_pb, s_d);
  // the longest block, one atomic per warp
  jump = __reduce_max_sync(0xffffffffu, jump);
  if ((threadIdx.x & 31) == 0 && jump) atomicMax(&J.ctr->max_jump, jump);
}

// Per chunk: exits of the chain for every entry point in the first `window`
// survivors of the chunk.  The chunk's next() values are staged in shared
// memory and cut into sub-chunks of kChainSub survivors: every (sub-chunk,
// entry point) pair is walked in parallel to the sub-chunk's exit, and the
// chunk's exits are composed from the sub-chunk exits (C / kChainSub steps
// per entry point instead of a walk over the whole chunk).  Windows wider
// than a sub-chunk walk the chunk directly.
constexpr uint32_t kChainSub = 256;

// The chunk the chain is followed by, from the longest block W.  Where it is
// longer than the one the job was launched for, next() is read from memory
// instead of a stage: room for a long chunk in every launch cost the kernel
// after k_chain_mark 7 us (k_partition of 80000 entries 21 -> 28.5 us).  60000
// entries of 250 bytes with 3000 empty values in a row, in 16 KiB blocks, block
// by block by one thread: 289 us for the partition phase, so 133.
__device__ __forceinline__ uint32_t chain_chunk(const JobDev& J, uint32_t W) {
  return W <= J.chunk ? J.chunk : kChunk;
}

// A chain table's word: how far past the (sub-)chunk's first survivor the
// chain leaves it (below 2^14: a chunk and a window), and above bit 16 the
// blocks started inside it.
__device__ __forceinline__ uint32_t chain_word(uint64_t exit_rel, uint32_t blocks) {
  return (uint32_t)exit_rel | (blocks << 16);
}

// The chain from survivor e of a chunk at c0 (s_next: its next() values) until it reaches `end`.
__device__ __forceinline__ uint32_t chain_walk(const uint32_t* s_next, uint64_t c0, uint64_t e,
                                               uint64_t end, uint64_t from) {
  uint32_t blocks = 0;
  while (e < end) {
    e = s_next[e - c0];
    blocks++;
  }
  return chain_word(e - from, blocks);
}

__device__ __forceinline__ void chain_tables(const JobDev& J, uint32_t cta, uint32_t ctas, uint32_t* s_next) {
  const uint32_t* const knext = J.k_next;
  uint32_t* const table = J.chunk_table;
  const uint64_t n = J.ctr->n_kept;
  const uint32_t W = J.ctr->max_jump;
  const uint32_t C = chain_chunk(J, W);
  if (W > C) return;  // resolved sequentially instead
  const bool sub = W <= kChainSub;
  uint32_t* s_sub = s_next + C;  // (C / kChainSub) x W
  for (uint64_t c = cta; c * C < n; c += ctas) {
    const uint64_t c0 = c * C;
    const uint64_t c1 = min(n, c0 + C);
    if (C != J.chunk) {
      for (uint32_t i = threadIdx.x; i < W; i += blockDim.x)
        table[c * C + i] = chain_walk(knext + c0, c0, c0 + i, c1, c0);
      continue;
    }
    __syncthreads();
    for (uint64_t i = threadIdx.x; i < c1 - c0; i += blockDim.x) s_next[i] = knext[c0 + i];
    __syncthreads();
    if (!sub) {
      for (uint32_t i = threadIdx.x; i < W; i += blockDim.x)
        table[c * C + i] = chain_walk(s_next, c0, c0 + i, c1, c0);
      continue;
    }
    const uint32_t nsub = (uint32_t)((c1 - c0 + kChainSub - 1) / kChainSub);
    for (uint32_t x = threadIdx.x; x < nsub * W; x += blockDim.x) {
      const uint32_t sb = x / W, i = x % W;
      const uint64_t s0 = c0 + (uint64_t)sb * kChainSub;
      s_sub[x] = chain_walk(s_next, c0, s0 + i, min(c1, s0 + kChainSub), s0);
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < W; i += blockDim.x) {
      uint64_t e = c0 + i;
      uint32_t blocks = 0;
      for (uint32_t sb = 0; sb < nsub && e < c1; sb++) {
        const uint64_t s0 = c0 + (uint64_t)sb * kChainSub;
        const uint32_t w = s_sub[sb * W + (uint32_t)(e - s0)];  // e: in the sub-chunk's first W
        e = s0 + (w & 0xffff);
        blocks += w >> 16;
      }
      table[c * C + i] = chain_word(e - c0, blocks);
    }
  }
}

__global__ void k_chain_tables(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  extern __shared__ __align__(16) uint32_t s_dyn[];
  chain_tables(J, blockIdx.x, gridDim.x, s_dyn);
}

// Exits (and blocks, in the high half) of groups of kChainGroup chunks for
// every entry point in the first `window` survivors of the group's first
// chunk, by following the chunk tables (one thread per entry point).  Only
// for more chunks than a group has whose tables do not fit the resolving
// CTA's shared memory (the host, which knows neither the survivors nor the
// window, launches this for every job that may have more than a group's).
__device__ __forceinline__ void chain_groups(const JobDev& J, uint32_t cta, uint32_t ctas) {
  const uint64_t n = J.ctr->n_kept;
  const uint32_t W = J.ctr->max_jump;
  const uint32_t C = chain_chunk(J, W);
  if (W > C || n == 0) return;
  const uint64_t M = (n + C - 1) / C;
  if (M <= kChainGroup || M * W <= J.chain_smem_words) return;  // resolved from the chunk tables
  const uint64_t G = (M + kChainGroup - 1) / kChainGroup;
  for (uint64_t x = (uint64_t)cta * blockDim.x + threadIdx.x; x < G * W;
       x += (uint64_t)ctas * blockDim.x) {
    const uint64_t g = x / W, i = x % W;
    const uint64_t c0 = g * kChainGroup, c1 = min(M, c0 + kChainGroup);
    uint64_t e = c0 * C + i, blocks = 0;
    for (uint64_t c = c0; c < c1 && e < n; c++) {
      const uint32_t w = J.chunk_table[c * C + (e - c * C)];
      e = c * C + (w & 0xffff);
      blocks += w >> 16;
    }
    J.group_table[g * C + i] = e | (blocks << 32);
  }
}

__global__ void k_chain_groups(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // a failed job does no more work
  chain_groups(J, blockIdx.x, gridDim.x);
}

// Entry point and first block of every chunk: the chain from survivor 0
// through the chunk tables.  Few chunks, or small tables: one thread walks
// the tables, over a shared-memory copy where they fit (else a dependent load
// a chunk, as a group's table would take to build).  Many: one thread walks
// the group tables (in shared memory when they fit), then one thread per group
// walks its chunks from the group's entry point.
__device__ __forceinline__ void chain_resolve(const JobDev& J, uint32_t* s_tab) {
  const uint64_t n = J.ctr->n_kept;
  const uint32_t W = J.ctr->max_jump;
  const uint32_t C = chain_chunk(J, W);
  const auto finish = [&](uint64_t blocks) {
    J.b_first[blocks] = (uint32_t)n;
    J.ctr->n_blocks_out = blocks;
  };
  if (n == 0) {
    if (threadIdx.x == 0) finish(0);
    return;
  }
  if (W > C) {
    // blocks longer than a chunk: walk the whole chain
    if (threadIdx.x != 0) return;
    uint64_t e = 0, b = 0;
    while (e < n) {
      J.b_first[b++] = (uint32_t)e;
      e = J.k_next[e];
    }
    finish(b);
    return;
  }
  const uint64_t M = (n + C - 1) / C;
  if (M * W <= J.chain_smem_words) {
    for (uint64_t i = threadIdx.x; i < M * W; i += blockDim.x)
      s_tab[i] = J.chunk_table[(i / W) * C + (i % W)];
    __syncthreads();
    if (threadIdx.x != 0) return;
    uint64_t e = 0, b = 0;
    for (uint64_t c = 0; c < M; c++) {
      J.chunk_entry[c] = make_uint2((uint32_t)e, (uint32_t)b);
      if (e < n) {
        const uint32_t w = s_tab[c * W + (e - c * C)];
        e = c * C + (w & 0xffff);
        b += w >> 16;
      }
    }
    finish(b);
    return;
  }
  if (M <= kChainGroup) {
    if (threadIdx.x != 0) return;
    const uint32_t* const table = J.chunk_table;
    uint32_t e = 0, b = 0;
    for (uint32_t c = 0; c < (uint32_t)M; c++) {
      J.chunk_entry[c] = make_uint2(e, b);
      if (e < n) {
        const uint32_t w = table[e];  // chunk c's table begins at its first survivor's place
        e = c * C + (w & 0xffff);
        b += w >> 16;
      }
    }
    finish(b);
    return;
  }
  const uint64_t G = (M + kChainGroup - 1) / kChainGroup;
  const bool staged = 2 * G * W <= J.chain_smem_words;
  uint64_t* s_grp = reinterpret_cast<uint64_t*>(s_tab);
  if (staged) {
    for (uint64_t i = threadIdx.x; i < G * W; i += blockDim.x)
      s_grp[i] = J.group_table[(i / W) * C + (i % W)];
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t e = 0, b = 0;
    for (uint64_t g = 0; g < G; g++) {
      const uint64_t c0 = g * kChainGroup;
      J.chunk_entry[c0] = make_uint2((uint32_t)e, (uint32_t)b);
      if (e < n) {
        const uint64_t w = staged ? s_grp[g * W + (e - c0 * C)] : J.group_table[g * C + (e - c0 * C)];
        e = w & 0xffffffffu;
        b += w >> 32;
      }
    }
    finish(b);
  }
  __syncthreads();
  for (uint64_t g = threadIdx.x; g < G; g += blockDim.x) {
    const uint64_t c0 = g * kChainGroup, c1 = min(M, c0 + kChainGroup);
    const uint2 at = J.chunk_entry[c0];
    uint64_t e = at.x;
    uint32_t b = at.y;
    for (uint64_t c = c0; c < c1; c++) {
      J.chunk_entry[c] = make_uint2((uint32_t)e, b);
      if (e < n) {
        const uint32_t w = J.chunk_table[c * C + (e - c * C)];
        e = c * C + (w & 0xffff);
        b += w >> 16;
      }
    }
  }
}

__global__ void k_chain_resolve(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  extern __shared__ __align__(16) uint32_t s_dyn[];
  chain_resolve(J, s_dyn);
}

// First survivor of every block: each chunk's chain from its resolved entry
// point.  With sub-chunks, one thread finds the sub-chunks' entry points from
// their words (recomputed as k_chain_tables does) and every sub-chunk is
// walked by its own thread.  (Block starts as flags that a scan over the
// survivors turns into block numbers: 8M survivors, 47 us more.)
__device__ __forceinline__ void chain_mark(const JobDev& J, uint32_t cta, uint32_t ctas, uint32_t* s_next) {
  const uint32_t* const knext = J.k_next;
  uint32_t* const first = J.b_first;
  const uint64_t n = J.ctr->n_kept;
  const uint32_t W = J.ctr->max_jump;
  const uint32_t C = chain_chunk(J, W);
  if (W > C) return;
  const bool sub = W <= kChainSub;
  uint32_t* s_sub = s_next + C;
  __shared__ uint2 s_entry[32];  // sub-chunk entry points and first blocks (C / kChainSub of them)
  for (uint64_t c = cta; c * C < n; c += ctas) {
    const uint64_t c0 = c * C;
    const uint64_t c1 = min(n, c0 + C);
    const uint2 at = J.chunk_entry[c];
    if (C != J.chunk) {
      if (threadIdx.x == 0) {
        uint32_t e = at.x, b = at.y;
        for (; e < c1; e = knext[e]) first[b++] = e;
      }
      continue;
    }
    __syncthreads();
    for (uint64_t i = threadIdx.x; i < c1 - c0; i += blockDim.x) s_next[i] = knext[c0 + i];
    __syncthreads();
    if (!sub) {
      if (threadIdx.x == 0) {
        uint64_t e = at.x;
        uint32_t b = at.y;
        while (e < c1) {
          first[b++] = (uint32_t)e;
          e = s_next[e - c0];
        }
      }
      continue;
    }
    const uint32_t nsub = (uint32_t)((c1 - c0 + kChainSub - 1) / kChainSub);
    for (uint32_t x = threadIdx.x; x < nsub * W; x += blockDim.x) {
      const uint32_t sb = x / W, i = x % W;
      const uint64_t s0 = c0 + (uint64_t)sb * kChainSub;
      s_sub[x] = chain_walk(s_next, c0, s0 + i, min(c1, s0 + kChainSub), s0);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      uint64_t e = at.x;
      uint32_t b = at.y;
      for (uint32_t sb = 0; sb < nsub; sb++) {
        s_entry[sb] = make_uint2((uint32_t)e, b);
        const uint64_t s0 = c0 + (uint64_t)sb * kChainSub;
        if (e < c1) {
          const uint32_t w = s_sub[sb * W + (uint32_t)(e - s0)];
          e = s0 + (w & 0xffff);
          b += w >> 16;
        }
      }
    }
    __syncthreads();
    for (uint32_t sb = threadIdx.x; sb < nsub; sb += blockDim.x) {
      const uint64_t s0 = c0 + (uint64_t)sb * kChainSub, send = min(c1, s0 + kChainSub);
      uint64_t e = s_entry[sb].x;
      uint32_t b = s_entry[sb].y;
      while (e < send) {
        first[b++] = (uint32_t)e;
        e = s_next[e - c0];
      }
    }
  }
}

__global__ void k_chain_mark(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  extern __shared__ __align__(16) uint32_t s_dyn[];
  chain_mark(J, blockIdx.x, gridDim.x, s_dyn);
}

// Sizes of the output blocks.
__device__ __forceinline__ void block_sizes(const JobDev& J, uint32_t cta, uint32_t ctas) {
  const uint32_t *const first = J.b_first, *const ka = J.k_a, *const kb = J.k_b;
  const uint64_t* const pb = J.k_pb;
  uint32_t *const sizes = J.b_size, *const flushed = J.tmp32;
  const uint64_t nb = J.ctr->n_blocks_out;
  const uint32_t R = J.restart_interval;
  for (uint64_t b = (uint64_t)cta * blockDim.x + threadIdx.x; b < nb;
       b += (uint64_t)ctas * blockDim.x) {
    const uint64_t k = first[b], e = first[b + 1];
    uint64_t D = 0;
    for (uint64_t a = k; a < e; a += R) D += ka[a] - kb[a];
    const uint64_t nrest = (e - k + R - 1) / R;
    const uint32_t size = (uint32_t)(pb[e] - pb[k] + D + 4 * nrest + 4);
    sizes[b] = size;
    flushed[b] = size + kTrailer;
  }
}

__global__ void k_block_sizes(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // a failed job does no more work
  block_sizes(J, blockIdx.x, gridDim.x);
}

// Like the block chain, a file's end depends on where it starts: every block
// b gets b_fnext[b], the first block of the next file if a file began at b (a
// binary search for the size cut, and the next forced block); one thread then
// walks the few file starts.

__device__ __forceinline__ void file_next(const JobDev& J, uint32_t cta, uint32_t ctas) {
  const uint64_t* const cum = J.b_cum;
  const uint32_t *const firsts = J.b_first, *const cuts = J.t_kept;
  uint32_t* const out = J.b_fnext;
  const uint64_t max_size = J.max_file_size;
  const uint64_t nb = J.ctr->n_blocks_out;
  const uint32_t nt = J.ctr->n_triggers;
  for (uint64_t b = (uint64_t)cta * blockDim.x + threadIdx.x; b < nb;
       b += (uint64_t)ctas * blockDim.x) {
    // first block end where the file's flushed bytes reach max_file_size
    const uint64_t cum0 = cum[b];
    const uint64_t target =
        max_size > ~0ull - cum0 ? ~0ull : cum0 + max_size;  // saturating
    uint64_t sc;
    if (cum[nb] < target) {
      sc = nb - 1;
    } else {
      uint64_t l = b, h = nb - 1;
      while (l < h) {
        const uint64_t mid = (l + h) >> 1;
        if (cum[mid + 1] >= target) h = mid;
        else l = mid + 1;
      }
      sc = l;
    }
    // or before the first grandparent cut after the block's start, which is a
    // block's start too: the block that starts at cut survivor kp
    uint32_t lo = 0, hi = nt;
    const uint32_t first = firsts[b];
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (cuts[mid] <= first) lo = mid + 1;
      else hi = mid;
    }
    if (lo < nt && cuts[lo] <= firsts[sc]) {
      const uint32_t kp = cuts[lo];
      uint64_t l = b + 1, h = sc;
      while (l < h) {
        const uint64_t mid = (l + h) >> 1;
        if (firsts[mid] >= kp) h = mid;
        else l = mid + 1;
      }
      sc = l - 1;
    }
    out[b] = (uint32_t)(sc + 1);
  }
}

__global__ void k_file_next(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // a failed job does no more work
  file_next(J, blockIdx.x, gridDim.x);
}

// The file starts are the orbit of block 0 under b_fnext, which only moves
// forward: the CTA loads a tile of b_fnext at the walk's position into shared
// memory, one 16-byte load per thread from the 16-byte boundary at or below
// it, and thread 0 walks inside it; a step that leaves the tile reloads.
// (b_fnext has N >= n_blocks_out words and 16 bytes of padding, so the last
// vector load stays inside its allocation.)
constexpr uint32_t kFileTile = 4096;
constexpr uint32_t kFileThreads = kFileTile / 4;
__device__ __forceinline__ void files(const JobDev& J) {
  __shared__ __align__(16) uint32_t tile[kFileTile];
  __shared__ uint64_t s_b;
  __shared__ uint32_t s_f;
  __shared__ bool s_stop;
  const uint64_t nb = J.ctr->n_blocks_out;
  if (threadIdx.x == 0) {
    s_b = 0;
    s_f = 0;
    s_stop = nb == 0;
  }
  __syncthreads();
  while (!s_stop) {
    const uint64_t t0 = s_b & ~uint64_t(3);
    for (uint64_t i = threadIdx.x; 4 * i < kFileTile && t0 + 4 * i < nb; i += blockDim.x)
      reinterpret_cast<uint4*>(tile)[i] = reinterpret_cast<const uint4*>(J.b_fnext + t0)[i];
    __syncthreads();
    if (threadIdx.x == 0) {
      uint64_t b = s_b;
      uint32_t f = s_f;
      while (b < nb && b < t0 + kFileTile) {
        const uint64_t end = tile[b - t0];
        if (f >= J.cap_files) {
          set_error(J.ctr, kErrLimit, 2);
          b = nb;
          break;
        }
        FileOut& F = J.files[f];  // first_kept / end_kept: k_block_layout
        F.first_block = (uint32_t)b;
        F.end_block = (uint32_t)end;
        f++;
        b = end;
      }
      s_b = b;
      s_f = f;
      s_stop = b >= nb;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) J.ctr->n_files = s_f;
}

__global__ void k_files(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  files(J);
}

__device__ __forceinline__ uint32_t file_of_block(const JobDev& J, uint64_t b) {
  uint32_t lo = 0, hi = J.ctr->n_files;
  while (hi - lo > 1) {
    uint32_t mid = (lo + hi) >> 1;
    if (J.files[mid].first_block <= b) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ void block_layout_one(const JobDev& J, uint64_t b);

__device__ __forceinline__ void block_layout(const JobDev& J, uint32_t cta, uint32_t ctas) {
  const uint64_t nb = J.ctr->n_blocks_out;
  for (uint64_t b = (uint64_t)cta * blockDim.x + threadIdx.x; b < nb;
       b += (uint64_t)ctas * blockDim.x)
    block_layout_one(J, b);
}

__global__ void __launch_bounds__(256, 5) k_block_layout(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // a failed job does no more work
  block_layout(J, blockIdx.x, gridDim.x);
}

__device__ void block_layout_one(const JobDev& J, uint64_t b) {
  // the loads that wait for nothing first
  const uint64_t cum = J.b_cum[b], cum1 = J.b_cum[b + 1], cum_before = b ? J.b_cum[b - 1] : 0;
  const uint32_t k0 = J.b_first[b], nx = J.b_first[b + 1], size = J.b_size[b];
  const uint32_t f = file_of_block(J, b);
  const uint32_t fb0 = J.files[f].first_block, fb1 = J.files[f].end_block;
  const bool last = b + 1 == fb1;
  const uint32_t llen = J.k_klen[nx - 1], ulen = llen - 8;
  const uint8_t* lkey = J.keys + J.k_koff[nx - 1];
  const uint32_t nlen = last ? 8 : J.k_klen[nx], shared = last ? 0 : J.k_shared[nx];
  const uint8_t* nkey = J.keys + (last ? 0 : J.k_koff[nx]);
  const uint64_t base = J.b_cum[fb0];
  const uint64_t off = cum - base;
  // filter group: blocks of this file whose start offsets share off >> 11
  uint32_t gbytes = 0, gkeys = 0;
  if (J.bits_per_key > 0) {
    const uint64_t j = off >> kFilterBaseLg;
    const bool start = b == fb0 || ((cum_before - base) >> kFilterBaseLg) != j;
    if (start) {
      uint64_t n = nx - k0;
      if (((cum1 - base) >> kFilterBaseLg) == j)
        for (uint64_t bb = b + 1; bb < fb1 && ((J.b_cum[bb] - base) >> kFilterBaseLg) == j; bb++)
          n += J.b_first[bb + 1] - J.b_first[bb];
      gkeys = (uint32_t)n;
      gbytes = bloom_bytes(n, J.bits_per_key) + 1;
    }
  }
  // index key for this block
  uint32_t sep = kNoSep, ilen = llen;
  if (!last) {
    // the prefix it shares with the next block's first key is known
    if (shared < ulen && shared < nlen - 8) {
      const uint32_t db = lkey[shared];
      if (db < 0xff && db + 1 < nkey[shared] && shared + 1 < ulen) {
        sep = shared;
        ilen = shared + 1 + 8;
      }
    }
  } else {
    uint32_t i = 0;
    while (i < ulen && lkey[i] == 0xff) i++;
    if (i < ulen && i + 1 < ulen) {
      sep = i;
      ilen = i + 1 + 8;
    }
  }
  const uint32_t hl = varint_len(off) + varint_len(size);
  if (b == fb0) J.files[f].first_kept = k0;
  if (last) J.files[f].end_kept = nx;
  J.b_file[b] = f;
  J.b_off[b] = off;
  J.b_gbytes[b] = gbytes;
  J.b_gkeys[b] = gkeys;
  J.b_sep[b] = sep;
  J.b_ilen[b] = ilen;
  J.b_isize[b] = 1 + varint_len(ilen) + varint_len(hl) + ilen + hl;
  if (size > kEncNarrow) {  // windows for the longest 16-byte phase
    const uint32_t n = (15 + size + 1 + kEncWindow - 1) / kEncWindow;
    const uint32_t at = atomicAdd(&J.ctr->n_wide, n);
    // (past the capacity: the files outgrow the output, an error of the file layout)
    for (uint32_t i = 0; i < n && at + i < J.cap_wide; i++) J.wide[at + i] = make_uint2((uint32_t)b, i);
    J.b_crc[b] = 0;
  }
}

// Pieces of a filter, metaindex or index block, a warp each in k_meta_crc.
constexpr uint32_t kMetaPiece = 4096;
__device__ __forceinline__ uint64_t meta_pieces(uint64_t len) { return (len + kMetaPiece - 1) / kMetaPiece; }

__device__ __forceinline__ void file_layout(const JobDev& J) {
  const uint32_t nf = J.ctr->n_files;
  uint32_t pieces = 0;
  for (uint32_t f = threadIdx.x; f < nf; f += blockDim.x) {
    FileOut& F = J.files[f];
    const uint32_t fb0 = F.first_block, fb1 = F.end_block;
    const uint64_t D = J.b_cum[fb1] - J.b_cum[fb0];
    F.data_bytes = D;
    uint64_t meta_off;
    if (J.bits_per_key > 0) {
      const uint64_t o_last = J.b_cum[fb1 - 1] - J.b_cum[fb0];
      const uint32_t nfl = (uint32_t)((D >> kFilterBaseLg) +
                                      ((D >> kFilterBaseLg) == (o_last >> kFilterBaseLg) ? 1 : 0));
      const uint64_t Ft = J.b_gcum[fb1] - J.b_gcum[fb0];
      const uint64_t fsize = Ft + 4ull * nfl + 4 + 1;
      F.filter_off = D;
      F.filter_size = fsize;
      F.n_filters = nfl;
      meta_off = D + fsize + kTrailer;
      F.meta_size = 3 + kFilterNameLen + varint_len(D) + varint_len(fsize) + 8;
    } else {
      F.filter_off = 0;
      F.filter_size = 0;
      F.n_filters = 0;
      meta_off = D;
      F.meta_size = 8;
    }
    F.meta_off = meta_off;
    F.crc_acc[0] = F.crc_acc[1] = F.crc_acc[2] = 0;
    F.index_off = meta_off + F.meta_size + kTrailer;
    F.index_size = (J.b_icum[fb1] - J.b_icum[fb0]) + 4ull * (fb1 - fb0) + 4;
    F.size = F.index_off + F.index_size + kTrailer + kFooter;
    pieces += (uint32_t)(meta_pieces(F.filter_size) + meta_pieces(F.meta_size) + meta_pieces(F.index_size));
  }
  pieces = __reduce_add_sync(0xffffffffu, pieces);
  if ((threadIdx.x & 31) == 0 && pieces) atomicAdd(&J.ctr->meta_pieces, pieces);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint64_t o = 0;
    for (uint32_t f = 0; f < nf; f++) {
      J.files[f].out_off = o;
      o += J.files[f].size;
    }
    J.ctr->bytes_out = o;
    // a single-pass job sized its output buffer from the input: rerun it
    // with exact counting instead of failing
    if (o > J.cap_out) set_error(J.ctr, J.reserve_keys ? kErrRetryExact : kErrLimit, 3);
  }
}

__global__ void k_file_layout(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  file_layout(J);
}

// All of the above (kAll: a job of few entries) or all from the block sizes on
// (a job of few blocks): one cluster of CTAs per job, a barrier where a launch
// would end.  Each of these kernels has microseconds of work in a small job;
// on B200 a launch of its own costs such a step about 3.5 us, a step in the
// cluster 1.2 to 2.8 us (what is left is the steps' chains of dependent loads).
// 512 threads a CTA: with 1024 the steps whose lanes each read a line of their
// own waited for the L1 of half as many SMs (block sizes of 2000 blocks 5.6
// instead of 4 us, block layout 14 instead of 5.6).
// Measured (a call): 800 entries 204 -> 191 us; 80000 entries in 2070 blocks
// 296 -> 283 us.  Above the limits below the kernels one by one are as fast or
// faster (2070 blocks and all 80000 entries in the cluster: no gain, 13600
// blocks: 20 us more), and many jobs at once fill the device with theirs.
constexpr uint64_t kPartEntries = 8192, kPartBlocks = 8192;
template <bool kAll>
__global__ void __launch_bounds__(kPartThreads, 1) k_partition(const JobDev* __restrict__ jobs) {
  pdl_begin();
  __shared__ JobDev s_job;
  extern __shared__ __align__(16) uint32_t s_dyn[];
  copy_job(jobs + blockIdx.y, &s_job);
  __syncthreads();
  const JobDev& J = s_job;
  const uint32_t cta = blockIdx.x, ctas = gridDim.x;  // the grid's x is one cluster
  if (*(volatile uint32_t*)&J.ctr->error) return;  // (the same in all CTAs: set before this kernel)
  if constexpr (kAll) {
    tile_scan<kScanKb, kPartThreads, true>(J, cta, ctas);
    cluster_sync();
    next(J, cta, ctas);
    cluster_sync();
    chain_tables(J, cta, ctas, s_dyn);
    cluster_sync();
    chain_groups(J, cta, ctas);
    cluster_sync();
    if (cta == 0) chain_resolve(J, s_dyn);
    cluster_sync();
    chain_mark(J, cta, ctas, s_dyn);
    cluster_sync();
  }
  block_sizes(J, cta, ctas);
  cluster_sync();
  tile_scan<kScanBcum, kPartThreads, true>(J, cta, ctas);
  cluster_sync();
  file_next(J, cta, ctas);
  cluster_sync();
  if (cta == 0) files(J);
  cluster_sync();
  if (*(volatile uint32_t*)&J.ctr->error) return;  // too many files (the next to set it is file_layout)
  block_layout(J, cta, ctas);
  cluster_sync();
  tile_scan<kScanIcum, kPartThreads, true>(J, cta, ctas);
  tile_scan<kScanGcum, kPartThreads, true>(J, ctas - 1 - cta, ctas);  // few tiles: another CTA's
  cluster_sync();
  if (cta == 0) file_layout(J);
}

// Data blocks, assembled in shared memory: one warp per block of at most
// kEncNarrow bytes, and one per window of kEncWindow bytes of a wider block
// (k_block_layout lists those).  The warp's stage has the block's own 16-byte
// phase in global memory: stage position p is global byte dst - ph + p0 + p,
// ph = dst & 15, p0 the window's first grid position (0 for a narrow block).
//  1. The stage is cleared, then the entries are taken in rounds of 32, one
//     lane per entry: sizes and places by a warp scan, entry headers and
//     restart words with byte stores, key deltas and short values (up to 32
//     bytes) lane by lane in words, longer values by groups of 8 or 32 lanes
//     in words (coalesced loads; source and destination alignments differ, so
//     every word is two source words and a funnel shift).  A word shared with
//     a neighbouring piece is ored into the cleared stage, all others are
//     stored, so no byte is stored twice and nothing is written bytewise but
//     headers.
//  2. The whole 16-byte chunks go out with one bulk copy from shared memory,
//     and meanwhile every lane folds a run of consecutive chunks into its last
//     32 bytes and looks those up (enc_out).  The grid bytes outside the message
//     are zero, so every chunk takes the same step; the initial all-ones
//     register enters at the end, as its register carried over the message's
//     length (crc_ones).
//  3. The lanes' registers combined, the trailer, and the partial chunks at
//     both ends with byte stores.  A window's register is moved over the
//     bytes after it and xored into its block's (k_meta_trailers finishes
//     wide blocks).
//
// Bound by issue, the integer pipe first (1 KiB values: ALU 62% of its cycles,
// issue 73%), at the warps an SM holds: 32 of them (64 registers, 5.8 KB of
// shared memory each) where 24 warps with a 6 KB stage took a third longer.
// Measured on B200, one launch, filters and index blocks included: 1 GiB of 1 KiB
// values 677 us, 512 MiB of 32-byte values 537, 66 MiB of lognormal values 88,
// 210 MiB in 16 KiB blocks 238, 280 MiB of 4-64 KiB values 225.  (The data blocks
// alone took 866, 712 and 224 us with values as 16-byte chunks straight from
// global to global memory through the row CRC and short pieces bytewise into the
// stage, and 2753 and 6759 us by a lane per entry, byte by byte, for any block
// beyond the stage.)
struct EncWarp {
  uint32_t ahead[5][kEncAhead];  // next block's entries: key length, shared, value length, key
                                 // offset, value offset
  __align__(16) uint8_t stage[kEncStage];
};
static_assert(kEncAhead % 32 == 0, "whole rounds of entries are copied ahead");
constexpr size_t kEncSmem = (size_t)kEncWarps * sizeof(EncWarp);

// Up to 4 kW bytes (len >= 1) from src (any alignment) to the cleared stage
// at p (any alignment), by one lane: all loads first; whole words stored,
// words shared with neighbours ored.  Only source words that hold a needed
// byte are loaded.
template <uint32_t kW>
__device__ __forceinline__ void enc_piece(uint8_t* p, const uint8_t* src, uint32_t len) {
  const uint32_t da = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3);
  const uintptr_t s = reinterpret_cast<uintptr_t>(src), s0 = s - da;  // stage word q: source s0 + 4q
  const uintptr_t b0 = s0 & ~uintptr_t(3);
  const uint32_t sh = 8 * (uint32_t)(s0 & 3);
  const uint32_t first = (uint32_t)(s - b0), end = first + len;  // needed bytes from b0
  const uint32_t* base = reinterpret_cast<const uint32_t*>(b0);
  uint32_t w[kW + 2];
#pragma unroll
  for (uint32_t i = 0; i < kW + 2; i++)
    w[i] = (4 * i + 4 > first && 4 * i < end) ? __ldg(base + i) : 0u;
  uint32_t* dw = reinterpret_cast<uint32_t*>(p - da);
  const uint32_t dend = da + len;
#pragma unroll
  for (uint32_t q = 0; q < kW + 1; q++) {
    if (4 * q >= dend) break;
    uint32_t v = __funnelshift_r(w[q], w[q + 1], sh);
    if (4 * q >= da && 4 * q + 4 <= dend) {
      dw[q] = v;
    } else {
      if (q == 0) v &= 0xffffffffu << (8 * da);
      if (4 * q + 4 > dend) v &= 0xffffffffu >> (8 * (4 * q + 4 - dend));
      smem_or(dw + q, v);
    }
  }
}

// The word at src (any alignment); bytes at or past end are zero.
__device__ __forceinline__ uint32_t enc_word(const uint8_t* src, const uint8_t* end) {
  const uintptr_t a = reinterpret_cast<uintptr_t>(src), q = a & ~uintptr_t(3);
  const uint32_t lo = __ldg(reinterpret_cast<const uint32_t*>(q));
  const uint32_t hi = ((a & 3) && q + 4 < reinterpret_cast<uintptr_t>(end))
                          ? __ldg(reinterpret_cast<const uint32_t*>(q + 4)) : 0u;
  const uint32_t v = __funnelshift_r(lo, hi, 8 * (uint32_t)(a & 3));
  const uint32_t n = (uint32_t)(end - src);
  return n >= 4 ? v : v & ((1u << (8 * n)) - 1u);
}

// x / R for the restart interval R: a shift when R is a power of two (the
// common 16), else a division.
struct RestartDiv {
  uint32_t R, sh;
  bool pow2;
  __device__ __forceinline__ explicit RestartDiv(uint32_t r) {
    R = r;
    pow2 = (r & (r - 1u)) == 0u;
    sh = (uint32_t)__popc(r - 1u);  // log2 r when r is a power of two
  }
  __device__ __forceinline__ uint32_t div(uint32_t x) const {
    uint32_t q;
    if (pow2)
      q = x >> sh;
    else
      q = x / R;
    return q;
  }
};

// A block's place and entry range, loaded one block ahead.
struct EncBlock {
  uint8_t* dst;
  uint32_t bsz, n, s;
  uint32_t off;  // in its file
};

// The block's first kEncAhead entries into the warp's `ahead` area, by cp.async
// (no registers held) while the block before it is still encoded; then
// enc_prefetch brings the lines that their keys and values lie in into L2.
__device__ __forceinline__ void enc_ahead_entries(const JobDev& J, EncWarp& W, const EncBlock& A,
                                                  uint32_t lane) {
#pragma unroll
  for (uint32_t j = lane; j < kEncAhead; j += 32) {
    if (j < A.n) {
      const uint32_t k = A.s + j;
      cp_async4(&W.ahead[0][j], J.k_klen + k);
      cp_async4(&W.ahead[1][j], J.k_shared + k);
      cp_async4(&W.ahead[2][j], J.k_vlen + k);
      cp_async4(&W.ahead[3][j], J.k_koff + k);
      cp_async4(&W.ahead[4][j], J.k_voff + k);
    }
  }
}
__device__ __forceinline__ void enc_prefetch(const JobDev& J, const EncWarp& W, uint32_t n,
                                             uint32_t lane) {
  for (uint32_t j = lane; j < min(n, kEncAhead); j += 32) {
    const uint32_t kl = W.ahead[0][j], vl = W.ahead[2][j];
    const uint32_t ko = W.ahead[3][j], vo = W.ahead[4][j];
    prefetch_l2(J.keys + ko);
    prefetch_l2(J.keys + ko + kl - 1);
    if (vl >= 256) {
      bulk_prefetch_l2(J.in + vo, vl);
    } else if (vl) {
      prefetch_l2(J.in + vo);
      prefetch_l2(J.in + vo + vl - 1);
    }
  }
}

// The entry that holds block byte `at`, and where in its block (bytes from the
// block's start) it starts: the prefix sums k_pb give an entry's place but for
// the restarts before it, whose extra bytes are summed here; first a lane per
// 32 entries, then a lane per entry.  (Rounds that started at a multiple of 32
// entries held the end of the window before too: 16 KiB blocks of 250-byte
// entries, two rounds a window instead of one; with the values' lines brought
// into L2 a round at a time the kernel took 239 instead of 283 us.)
__device__ __forceinline__ void enc_seek(const JobDev& J, const EncBlock& B, const RestartDiv& rd,
                                         uint32_t at, uint32_t lane, uint32_t* j0, uint32_t* pos) {
  const uint64_t pb0 = J.k_pb[B.s];
  uint32_t group = 0, extra = 0;  // extra bytes of the restarts before the group, before j0
  *j0 = 0;
  for (uint32_t g = 0; B.n > 32 && g < B.n; g += 1024) {
    const uint32_t a = g + 32 * lane, z = min(a + 32, B.n);  // the lane's entries
    uint32_t x = 0;
    for (uint32_t j = rd.div(a + rd.R - 1) * rd.R; j < z; j += rd.R) x += J.k_a[B.s + j] - J.k_b[B.s + j];
    uint32_t tot;
    const uint32_t before = warp_excl<uint32_t>(x, &tot) + group;
    group += tot;
    const uint32_t p = a < B.n ? (uint32_t)(J.k_pb[B.s + a] - pb0) + before : 0xffffffffu;
    const unsigned m = __ballot_sync(0xffffffffu, p <= at);
    if (!m) break;  // the group starts past `at`: among the last 32 of the one before
    const int l = 31 - __clz(m);
    *j0 = g + 32 * l;
    extra = __shfl_sync(0xffffffffu, before, l);
    if (l < 31) break;
  }
  const uint32_t j = *j0 + lane;
  const bool in = j < B.n;
  uint32_t tot;
  const uint32_t x = in && rd.div(j) * rd.R == j ? J.k_a[B.s + j] - J.k_b[B.s + j] : 0u;
  const uint32_t before = warp_excl<uint32_t>(x, &tot) + extra;
  const uint32_t p = in ? (uint32_t)(J.k_pb[B.s + j] - pb0) + before : 0xffffffffu;
  const int l = 31 - __clz(__ballot_sync(0xffffffffu, p <= at));
  *j0 += l;
  *pos = __shfl_sync(0xffffffffu, p, l);
}

// Grid positions [p0, p1) of the block into the warp's stage (kWide: a
// window; else the whole block, p0 = 0).
template <bool kWide>
__device__ __forceinline__ void enc_assemble(const JobDev& J, EncWarp& W, const EncBlock& B,
                                             const RestartDiv& rd, uint32_t ph, uint32_t p0,
                                             uint32_t p1, uint32_t lane) {
  uint8_t* st = W.stage;
  const uint32_t n = B.n, R = rd.R;
  const uint32_t nrest = rd.div(n + R - 1);
  const uint32_t rbase = ph + B.bsz - 4 * nrest - 4;  // grid position of the restart array
  for (uint32_t q = 16 * lane; q < p1 - p0; q += 512)
    *reinterpret_cast<uint4*>(st + q) = make_uint4(0u, 0u, 0u, 0u);
  __syncwarp();
  uint32_t carry = 0, j0 = 0;
  if (kWide) {
    if (p1 > rbase) {  // the window's restart words, a lane per run
      const uint64_t pb0 = J.k_pb[B.s];
      uint32_t extra = 0;
      for (uint32_t r0 = 0; r0 < nrest; r0 += 32) {
        const uint32_t r = r0 + lane, k = B.s + r * R;
        const bool on = r < nrest;
        uint32_t tot;
        const uint32_t before = warp_excl<uint32_t>(on ? J.k_a[k] - J.k_b[k] : 0u, &tot) + extra;
        extra += tot;
        if (on) {
          const uint32_t ex = (uint32_t)(J.k_pb[k] - pb0) + before;
          const uint32_t word = (ex << 8) | min(n - r * R, R), rp = rbase + 4 * r - p0;
#pragma unroll
          for (uint32_t i = 0; i < 4; i++)
            if (rp + i < p1 - p0) st[rp + i] = (uint8_t)(word >> (8 * i));
        }
      }
    }
    if (p0 && n > 1) enc_seek(J, B, rd, p0 - ph, lane, &j0, &carry);
  }
  for (; j0 < n; j0 += 32) {
    if (kWide && ph + carry >= p1) break;
    const uint32_t j = j0 + lane, k = B.s + j;
    const bool valid = j < n;
    uint32_t kd = 0, vl = 0, sh = 0, koff = 0, voff = 0, hl = 0, run = 0;
    bool restart = false;
    if (valid) {
      uint32_t kl;
      if (!kWide && j0 < kEncAhead) {
        kl = W.ahead[0][j], sh = W.ahead[1][j], vl = W.ahead[2][j];
        koff = W.ahead[3][j], voff = W.ahead[4][j];
      } else {
        kl = J.k_klen[k], sh = J.k_shared[k], vl = J.k_vlen[k];
        koff = J.k_koff[k], voff = J.k_voff[k];
      }
      run = rd.div(j);
      restart = run * R == j;
      if (restart) sh = 0;
      kd = kl - sh;
      hl = varint_len32(sh) + varint_len32(kd) + varint_len32(vl);
    }
    uint32_t tot;
    const uint32_t ex = warp_excl<uint32_t>(hl + kd + vl, &tot) + carry;
    const uint32_t hpos = ph + ex;
    const bool outside = kWide && (ph + carry + tot <= p0 || ph + carry >= p1);
    carry += tot;
    uint32_t kpos = hpos + hl, vpos = kpos + kd;
    if (valid) {
      // restart word and header bytes
      if (!kWide && restart) st_le32(st + rbase + 4 * run, (ex << 8) | min(n - j, R));
      if (!outside) {
        uint32_t q = hpos - p0;
        const auto put = [&](uint32_t v) {
          while (v >= 128) {
            if (!kWide || q < p1 - p0) st[q] = (uint8_t)(v | 128);
            q++;
            v >>= 7;
          }
          if (!kWide || q < p1 - p0) st[q] = (uint8_t)v;
          q++;
        };
        put(sh);
        put(kd);
        put(vl);
        // the value's place in its file, for the decoded form
        if (J.dec_vpos && (!kWide || (hpos >= p0 && hpos < p1)))
          J.dec_vpos[k] = B.off + ex + hl + kd;
      }
    }
    if (outside) continue;
    const uint8_t* key = J.keys + (koff + sh);
    const uint8_t* val = J.in + voff;
    if (kWide) {  // the pieces' parts inside the window
      const uint32_t ka = min(max(kpos, p0), p1), kz = min(max(vpos, p0), p1);
      const uint32_t ve = min(max(vpos + vl, p0), p1);
      key += ka - kpos, val += kz > vpos ? kz - vpos : 0;
      const uint32_t va = kz;
      kd = kz - ka, vl = ve - va;
      kpos = ka, vpos = va;
    }
    if (kWide && vl) {  // (a narrow block's were brought in before it was begun)
      if (vl >= 256) {
        bulk_prefetch_l2(val, vl);
      } else {
        prefetch_l2(val);
        prefetch_l2(val + vl - 1);
      }
    }
    kpos -= p0, vpos -= p0;  // stage positions
    __syncwarp();  // every header of the round is written: the words may be ored now
    const bool lng = vl >= kEncLong;
    const bool any_lng = __any_sync(0xffffffffu, lng);
    // a long value's partial words at both ends: loaded before the key's bytes
    // are, so that one wait covers both
    const uint32_t head = (0u - vpos) & 3, tail = (vpos + vl) & 3;
    uint32_t hw = 0, tw = 0;
    if (any_lng) {
      if (lng && head) hw = enc_word(val, val + head) << (8 * (4 - head));
      if (lng && tail) tw = enc_word(val + vl - tail, val + vl);
    }
    if (__any_sync(0xffffffffu, kd > 16)) {
      for (uint32_t t = 0; t < kd; t += 32) enc_piece<8>(st + kpos + t, key + t, min(32u, kd - t));
    } else if (kd) {
      enc_piece<4>(st + kpos, key, kd);
    }
    if (vl && !lng) enc_piece<8>(st + vpos, val, vl);
    if (any_lng) {
      if (lng) {
        if (head) smem_or(st + (vpos & ~3u), hw);
        if (tail) smem_or(st + ((vpos + vl) & ~3u), tw);
      }
      const uint32_t w0 = (vpos + head) >> 2;                   // first whole word,
      const uint32_t fw = lng ? ((vpos + vl) >> 2) - w0 : 0u;   // their count,
      const uint32_t so = (uint32_t)(val - J.in) + head;        // their source
      // the long values average 512 bytes or more: one after the other, all
      // lanes, 1 KiB in flight (a lane's higher source word is its neighbour's
      // lower one); else four at a time, 8 lanes each (a 100-byte value is
      // three steps)
      unsigned m = __ballot_sync(0xffffffffu, lng);
      if (__reduce_add_sync(0xffffffffu, lng ? vl : 0u) >= 512 * __popc(m)) {
        for (; m; m &= m - 1) {
          const int e = __ffs(m) - 1;
          const uint32_t efw = __shfl_sync(0xffffffffu, fw, e);
          const uintptr_t a = reinterpret_cast<uintptr_t>(J.in + __shfl_sync(0xffffffffu, so, e));
          const uint32_t* q = reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3)) + lane;
          const uint32_t fsh = 8 * (uint32_t)(a & 3);
          const uint32_t lim = efw + (fsh ? 1 : 0);  // source words
          uint32_t* d = reinterpret_cast<uint32_t*>(st) + __shfl_sync(0xffffffffu, w0, e) + lane;
          constexpr uint32_t kU = 8;
          for (uint32_t i = lane; i - lane < efw; i += 32 * kU, q += 32 * kU, d += 32 * kU) {
            uint32_t lo[kU + 1];
#pragma unroll
            for (uint32_t x = 0; x <= kU; x++)
              lo[x] = (i + 32 * x < lim && (x < kU || lane == 0)) ? __ldg(q + 32 * x) : 0u;
#pragma unroll
            for (uint32_t x = 0; x < kU; x++) {
              const uint32_t hi =
                  __shfl_sync(0xffffffffu, lane == 0 ? lo[x + 1] : lo[x], (lane + 1) & 31);
              if (i + 32 * x < efw) d[32 * x] = __funnelshift_r(lo[x], hi, fsh);
            }
          }
        }
      } else {
        constexpr uint32_t kU = 4;
        const uint32_t li = lane & 7;
        // words i, i + 8, .. (kU of them) of the value at d / q with efw words
        const auto step = [&](uint32_t* d, const uint32_t* q, uint32_t efw, uint32_t fsh, uint32_t i) {
          uint32_t lo[kU], hi[kU];
#pragma unroll
          for (uint32_t x = 0; x < kU; x++) {
            const bool on = i + x * 8 < efw;
            lo[x] = on ? __ldg(q + i + x * 8) : 0u;
            hi[x] = on && fsh ? __ldg(q + i + x * 8 + 1) : 0u;
          }
#pragma unroll
          for (uint32_t x = 0; x < kU; x++)
            if (i + x * 8 < efw) d[i + x * 8] = __funnelshift_r(lo[x], hi[x], fsh);
        };
        const auto value = [&](uint32_t e, uint32_t i) {
          const uint32_t ew0 = __shfl_sync(0xffffffffu, w0, e);
          const uint32_t efw = __shfl_sync(0xffffffffu, fw, e);
          const uint32_t eso = __shfl_sync(0xffffffffu, so, e);
          const uintptr_t a = reinterpret_cast<uintptr_t>(J.in + eso);
          step(reinterpret_cast<uint32_t*>(st) + ew0, reinterpret_cast<const uint32_t*>(a & ~uintptr_t(3)),
               efw, 8 * (uint32_t)(a & 3), i);
        };
        if (!__any_sync(0xffffffffu, fw > 8 * kU)) {  // one step each
          const uint32_t cnt = min(32u, n - j0);
          for (uint32_t e0 = 0; e0 < cnt; e0 += 4) value(e0 + (lane >> 3), li);
        } else {
          // the values' steps in one list, four at a time: of four values at a
          // time the shorter ones' lanes wait for the longest.  An entry has at
          // least one step, so that a step's entry is the number of entries that
          // start at or before it: those of the steps before, and those of a
          // mask of the starts among the next 32 steps.  (66 MiB of
          // lognormal values, median 128: the kernel 109 -> 93 us.)
          const uint32_t steps = valid ? max(1u, (fw + 8 * kU - 1) / (8 * kU)) : 0u;
          uint32_t all;
          const uint32_t at = warp_excl<uint32_t>(steps, &all);
          uint32_t before = 0;  // entries that start before step t0
          for (uint32_t t0 = 0; t0 < all; t0 += 32) {
            const unsigned starts =
                __reduce_or_sync(0xffffffffu, at - t0 < 32 ? 1u << (at - t0) : 0u);
            for (uint32_t t = t0; t < min(t0 + 32, all); t += 4) {
              const uint32_t r = t - t0 + (lane >> 3);  // this lane group's step
              const uint32_t e = before + __popc(starts & (0xffffffffu >> (31 - r))) - 1;
              const uint32_t first = __shfl_sync(0xffffffffu, at, e);
              value(e, (t0 + r - first) * 8 * kU + li);  // (past the last step: past the value's end)
            }
            before += __popc(starts);
          }
        }
      }
    }
    __syncwarp();  // the words are written before the next round's header bytes
  }
  if (lane == 0) {  // the restart count (and the type byte, 0: the stage is clear)
    const uint32_t rp = ph + B.bsz - 4 - p0;
#pragma unroll
    for (uint32_t i = 0; i < 4; i++)
      if (!kWide || rp + i < p1 - p0) st[rp + i] = (uint8_t)(nrest >> (8 * i));
  }
}

// The assembled stage out: the whole 16-byte chunks inside [m0, m1) with one
// bulk copy, every byte into the CRC.  Returns the raw register at m1 (from a
// zero register), the same in every lane.  The copy still reads the stage when
// this returns (enc_drain).
//
// The CRC: lane l takes q consecutive chunks (q odd, so the lanes' 16-byte
// reads, 16 q bytes apart, fall on different banks), and folds them into its
// last two with crc_fold_word, integer shifts and xors only; those 256 bits
// are looked up (crc_h8), and the register is moved to m1 by one product.  A
// lookup per 5 bits of every chunk, as in the row CRC, costs 26 lookups and 82
// integer instructions per chunk and lane; folding costs 40.
__device__ __forceinline__ uint32_t enc_out(const JobDev& J, const uint32_t* h8,
                                            const uint32_t* xinv, const uint32_t* tab8,
                                            uint8_t* gbase, const uint8_t* st, uint32_t m0,
                                            uint32_t m1, uint32_t lane) {
  const uint32_t nch = (m1 + 15) >> 4;
  const uint32_t q = max(((nch + 31) >> 5) | 1u, 3u);
  // the shift from the lane's last chunk's end to m1 (backwards for the lane
  // that holds m1, whose last chunks lie past it; lanes past that hold nothing)
  const int32_t n = (int32_t)m1 - (int32_t)(16 * q * (lane + 1));
  const uint32_t f = n >= 0 ? __ldg(J.crc_xpow + n)
                            : (n > -(int32_t)(16 * q) ? xinv[xinv_slot((uint32_t)-n)] : 0u);
  fence_proxy_async_smem();  // the lanes' stage writes, before the bulk copy's reads
  __syncwarp();
  const uint32_t c0 = (m0 + 15) >> 4, c1 = m1 >> 4;
  if (lane == 0 && c1 > c0) bulk_store(gbase + 16 * c0, st + 16 * c0, 16 * (c1 - c0));
  uint32_t c = lane * q;
  const uint32_t cz = c + q;
  const auto load = [&](uint32_t x) -> uint4 {
    return x < nch ? *reinterpret_cast<const uint4*>(st + 16 * x) : make_uint4(0u, 0u, 0u, 0u);
  };
  uint32_t v[8] = {};  // the folded words, a ring of the last eight
  {
    const uint4 x = load(c++);
    v[4] = x.x, v[5] = x.y, v[6] = x.z, v[7] = x.w;
    v[6] ^= v[4] << 1;
    v[7] ^= __funnelshift_l(v[4], v[5], 1);
  }
  for (; c + 2 < cz; c += 2) {
    const uint4 x = load(c), y = load(c + 1);
    const uint32_t m[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
    for (uint32_t i = 0; i < 8; i++) v[i] = m[i] ^ crc_fold_word<false>(v, i);
  }
  const uint4 x = load(c), y = load(c + 1);
  uint32_t r[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
#pragma unroll
  for (uint32_t i = 0; i < 8; i++) r[i] ^= crc_fold_word<true>(v, i);
  uint32_t u = gf2_mulmod_tab(tab8, crc_h8(h8, r), f);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) u ^= __shfl_xor_sync(0xffffffffu, u, o);
  return u;
}

// The partial chunks' bytes in [a, m1) at both ends (the message's first
// bytes, and those after its last whole chunk).
__device__ __forceinline__ void enc_ends(uint8_t* gbase, const uint8_t* st, uint32_t m0, uint32_t m1,
                                         uint32_t end, uint32_t lane) {
  const uint32_t cf0 = (m0 + 15) >> 4, cf1 = m1 >> 4;  // whole chunks [cf0, cf1) went out
  uint32_t h1 = 16 * cf0, t0 = 16 * cf1;
  if (cf1 < cf0) h1 = t0 = m0;  // the message lies inside one chunk
  const uint32_t nh = h1 - m0, nt = end - t0;
  for (uint32_t x = lane; x < nh + nt; x += 32) {
    const uint32_t q = x < nh ? m0 + x : t0 + (x - nh);
    gbase[q] = st[q];
  }
}

__device__ __forceinline__ void enc_drain(uint32_t lane) {
  if (lane == 0) bulk_wait_read();
  __syncwarp();
}

// Filter groups, each at its first block: a warp takes a run of up to 32
// blocks.  Its lanes first load everything about their own blocks' groups
// (one chain of dependent loads for all of them), write the groups' offsets
// and build those of a few keys in registers; the larger ones follow one at a
// time, lanes over the keys, whose hashes were kept when the keys were decoded
// (k_hash): the bits by shared-memory ors, then words out.  Filters beyond the
// warp's buffer are built in place with global atomics.
//
// Bound by latency: a warp per group that loaded its group's places and keys
// itself took 279 us for 8M keys in 126k groups on B200 (70 registers), and 54
// us for 1M keys in 256k groups; this form, as a kernel of its own, 86 and 19.
constexpr uint32_t kFilterSmem = 1024;
constexpr uint32_t kFilterFew = 8;    // keys, and at most 16 filter bytes: by one lane
__device__ __forceinline__ void encode_filters(const JobDev& J, uint32_t* sbuf, uint64_t warp,
                                               uint64_t warps, uint32_t lane) {
  if (J.bits_per_key <= 0) return;
  const uint64_t nb = J.ctr->n_blocks_out;
  const uint32_t K = J.bloom_k;
  const uint64_t run = min((uint64_t)32, (nb + warps - 1) / warps);  // blocks per warp and turn
  for (uint64_t b0 = warp * run; b0 < nb; b0 += warps * run) {
    const uint64_t b = b0 + lane;
    uint8_t* fdst = nullptr;
    uint32_t nbytes = 0, nk = 0, k0 = 0;
    uint64_t M = 0;
    bool big = false;
    if (lane < run && b < nb && J.b_gbytes[b]) {
      nbytes = J.b_gbytes[b] - 1;
      nk = J.b_gkeys[b];
      k0 = J.b_first[b];
      const FileOut& F = J.files[J.b_file[b]];
      const uint32_t fb0 = F.first_block, fb1 = F.end_block;
      uint8_t* fbase = J.out + F.out_off + F.filter_off;
      const uint64_t g0 = J.b_gcum[fb0], at = J.b_gcum[b] - g0, Ft = J.b_gcum[fb1] - g0;
      // filter offsets of the empty indices before this group and of the group
      const int64_t jb = (int64_t)(J.b_off[b] >> kFilterBaseLg);
      const int64_t jprev = (b == fb0) ? -1 : (int64_t)(J.b_off[b - 1] >> kFilterBaseLg);
      fdst = fbase + at;
      const FastMod mod(8 * nbytes);  // a group's filter is far below 2^29 bytes
      M = mod.M;
      for (int64_t jj = jprev + 1; jj <= jb; jj++) st_le32(fbase + Ft + 4 * jj, (uint32_t)at);
      fdst[nbytes] = (uint8_t)K;
      big = nk > kFilterFew || nbytes > 16;
      if (!big) {
        uint64_t lo = 0, hi = 0;
        for (uint32_t i = 0; i < nk; i++) {
          uint32_t h = J.k_hash[k0 + i];
          const uint32_t delta = (h >> 17) | (h << 15);
          for (uint32_t q = 0; q < K; q++) {
            const uint32_t bit = mod(h);  // byte bit / 8, bit bit % 8
            if (bit < 64) lo |= 1ull << bit;
            else hi |= 1ull << (bit - 64);
            h += delta;
          }
        }
        for (uint32_t i = 0; i < nbytes; i++) fdst[i] = (uint8_t)((i < 8 ? lo : hi) >> (8 * (i & 7)));
      }
    }
    for (unsigned m = __ballot_sync(0xffffffffu, big); m; m &= m - 1) {
      const int e = __ffs(m) - 1;
      uint8_t* d = reinterpret_cast<uint8_t*>(
          __shfl_sync(0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(fdst), e));
      const uint32_t eb = __shfl_sync(0xffffffffu, nbytes, e), en = __shfl_sync(0xffffffffu, nk, e);
      const uint32_t ek = __shfl_sync(0xffffffffu, k0, e);
      FastMod mod(__shfl_sync(0xffffffffu, (unsigned long long)M, e), 8 * eb);
      const bool in_smem = eb <= kFilterSmem;
      if (in_smem) {
        for (uint32_t i = lane; i <= eb / 4; i += 32) sbuf[i] = 0;
      } else {
        for (uint32_t i = lane; i < eb; i += 32) d[i] = 0;
      }
      __syncwarp();
      for (uint32_t i = lane; i < en; i += 32) {
        uint32_t h = J.k_hash[ek + i];
        const uint32_t delta = (h >> 17) | (h << 15);
        for (uint32_t q = 0; q < K; q++) {
          const uint32_t bit = mod(h);
          if (in_smem) {
            smem_or(sbuf + (bit >> 5), 1u << (bit & 31));
          } else {
            const uintptr_t a = reinterpret_cast<uintptr_t>(d + (bit >> 3));
            atomicOr(reinterpret_cast<unsigned int*>(a & ~uintptr_t(3)), 1u << ((a & 3) * 8 + (bit & 7)));
          }
          h += delta;
        }
      }
      __syncwarp();
      if (in_smem) {
        // the destination's whole words, and its bytes at both ends
        const uint32_t head = min((uint32_t)(-reinterpret_cast<uintptr_t>(d)) & 3, eb);
        const uint32_t words = (eb - head) / 4, tail = head + 4 * words;
        const uint8_t* sb = reinterpret_cast<const uint8_t*>(sbuf);
        for (uint32_t i = lane; i < words; i += 32)
          reinterpret_cast<uint32_t*>(d + head)[i] = __funnelshift_r(sbuf[i], sbuf[i + 1], 8 * head);
        if (lane < head) d[lane] = sb[lane];
        if (tail + lane < eb) d[tail + lane] = sb[tail + lane];
        __syncwarp();
      }
    }
  }
}

// Index entries: a warp takes a run of up to 32 blocks, a lane each; keys of
// more than kIndexLong bytes are copied by the warp, one after the other (by
// their lanes, 1500 keys of 9 KB took 15 ms on B200).
constexpr uint32_t kIndexLong = 64;
__device__ __forceinline__ void encode_index(const JobDev& J, uint64_t warp, uint64_t warps, uint32_t lane) {
  const uint64_t nb = J.ctr->n_blocks_out;
  const uint64_t run = min((uint64_t)32, (nb + warps - 1) / warps);  // blocks per warp and turn
  for (uint64_t b0 = warp * run; b0 < nb; b0 += warps * run) {
    const uint64_t b = b0 + lane;
    uint32_t from_key = 0;
    uint8_t* p = nullptr;
    const uint8_t* lkey = nullptr;
    if (lane < run && b < nb) {
      const FileOut& F = J.files[J.b_file[b]];
      const uint32_t fb0 = F.first_block, fb1 = F.end_block;
      uint8_t* ib = J.out + F.out_off + F.index_off;
      const uint64_t eoff = J.b_icum[b] - J.b_icum[fb0];
      p = ib + eoff;
      const uint32_t ilen = J.b_ilen[b], sep = J.b_sep[b];
      const uint64_t off = J.b_off[b];
      const uint32_t bsz = J.b_size[b];
      *p++ = 0;
      p = put_varint(p, ilen);
      p = put_varint(p, varint_len(off) + varint_len(bsz));
      uint32_t llen;
      lkey = kept_key(J, J.b_first[b + 1] - 1, &llen);
      // (copy_small loads a piece's bytes before it stores any)
      from_key = sep == kNoSep ? ilen : sep;
      if (from_key <= kIndexLong)
        for (uint32_t i = 0; i < from_key; i += 32) copy_small<32>(p + i, lkey + i, min(32u, from_key - i));
      if (sep != kNoSep) {
        p[sep] = (uint8_t)(lkey[sep] + 1);
        uint64_t t = kSeekTag;
        for (int i = 0; i < 8; i++) p[sep + 1 + i] = (uint8_t)(t >> (8 * i));
      }
      uint8_t* q = put_varint(p + ilen, off);
      put_varint(q, bsz);
      uint8_t* ra = ib + (J.b_icum[fb1] - J.b_icum[fb0]) + 4 * (b - fb0);
      st_le32(ra, ((uint32_t)eoff << 8) | 1u);
      if (b + 1 == fb1) st_le32(ra + 4, fb1 - fb0);
    }
    for (unsigned m = __ballot_sync(0xffffffffu, from_key > kIndexLong); m; m &= m - 1) {
      const int e = __ffs(m) - 1;
      const auto of = [&](const uint8_t* x) {
        return __shfl_sync(0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(x), e);
      };
      uint8_t* d = reinterpret_cast<uint8_t*>(of(p));
      const uint8_t* k = reinterpret_cast<const uint8_t*>(of(lkey));
      const uint32_t n = __shfl_sync(0xffffffffu, from_key, e);
      const uint32_t head = (uint32_t)(-reinterpret_cast<uintptr_t>(d)) & 3, words = (n - head) / 4;
      const uint32_t tail = head + 4 * words;
      if (lane < head) d[lane] = k[lane];
#pragma unroll 4
      for (uint32_t i = lane; i < words; i += 32)
        reinterpret_cast<uint32_t*>(d + head)[i] = enc_word(k + head + 4 * i, k + n);
      if (tail + lane < n) d[tail + lane] = k[tail + lane];
    }
  }
}

// File f's metaindex block, footer and the tail of its filter block's offset
// array (lane 0), and its smallest and largest keys, by one warp.
__device__ __forceinline__ void encode_meta_file(const JobDev& J, uint32_t f, uint32_t lane) {
  if (lane == 0) {
    const FileOut& F = J.files[f];
    uint8_t* base = J.out + F.out_off;
    if (J.bits_per_key > 0) {
      uint8_t* fb = base + F.filter_off;
      const uint64_t Ft = J.b_gcum[F.end_block] - J.b_gcum[F.first_block];
      const uint64_t jlast = J.b_off[F.end_block - 1] >> kFilterBaseLg;
      for (uint64_t jj = jlast + 1; jj < F.n_filters; jj++) st_le32(fb + Ft + 4 * jj, (uint32_t)Ft);
      st_le32(fb + Ft + 4ull * F.n_filters, (uint32_t)Ft);
      fb[Ft + 4ull * F.n_filters + 4] = (uint8_t)kFilterBaseLg;
      uint8_t* m = base + F.meta_off;
      m[0] = 0;
      m[1] = (uint8_t)kFilterNameLen;
      m[2] = (uint8_t)(varint_len(F.filter_off) + varint_len(F.filter_size));
      for (uint32_t i = 0; i < kFilterNameLen; i++) m[3 + i] = (uint8_t)kFilterName[i];
      uint8_t* p = m + 3 + kFilterNameLen;
      p = put_varint(p, F.filter_off);
      p = put_varint(p, F.filter_size);
      st_le32(p, 1u);  // restart word (0 << 8) | 1
      st_le32(p + 4, 1u);
    } else {
      uint8_t* m = base + F.meta_off;
      st_le32(m, 0u);
      st_le32(m + 4, 1u);
    }
    uint8_t* foot = base + F.size - kFooter;
    for (int i = 0; i < 40; i++) foot[i] = 0;
    uint8_t* p = foot;
    p = put_varint(p, F.meta_off);
    p = put_varint(p, F.meta_size);
    p = put_varint(p, F.index_off);
    p = put_varint(p, F.index_size);
    st_le32(foot + 40, 0x8b80fb57u);
    st_le32(foot + 44, 0xdb477524u);
  }
  const FileOut& F = J.files[f];
  // the file's smallest and largest internal keys (FileMetaData::smallest /
  // largest) into slots 2f and 2f + 1 of fkey_stride bytes, their lengths
  // into fkoff; every key fits a slot (a single-pass job with a longer key
  // was rerun with exact counting, whose stride is the longest key)
  for (uint32_t which = 0; which < 2; which++) {
    uint32_t l;
    const uint8_t* k = kept_key(J, which ? F.end_kept - 1 : F.first_kept, &l);
    uint8_t* d = J.fkeys + (2ull * f + which) * J.fkey_stride;
    for (uint32_t t = lane; t < l; t += 32) d[t] = k[t];
    if (lane == 0) J.fkoff[2 * f + which] = l;
  }
}

// Filter blocks, index blocks and the files' metadata need the layout only, not
// the data blocks: the first `side` CTAs of k_encode_blocks write them, beside
// the CTAs that encode (they finish early).  As three kernels after it they took
// another 24 us of an 80k-entry job, 121 us of 8M entries and 160 us of a
// 32-job batch on B200.
__device__ __forceinline__ void encode_side(const JobDev& J, uint32_t* sbuf, uint32_t cta,
                                            uint32_t ctas) {
  const uint32_t lane = threadIdx.x & 31;
  // Less than a full turn of blocks: consecutive warps on different CTAs, so that
  // a few large filters or long index keys spread over the SMs (side by side on
  // one they wait for its L1: 100000 entries in 64 KiB blocks at 20 bits a key, a
  // flush 1911 -> 886 us).  More: neighbours in one CTA (8M entries, 126k blocks:
  // the kernel 537 instead of 555 us).
  const uint32_t own = threadIdx.x >> 5, per = blockDim.x >> 5;
  const uint64_t warps = (uint64_t)ctas * per;
  const uint64_t warp = J.ctr->n_blocks_out < 32 * warps ? (uint64_t)own * ctas + cta : (uint64_t)cta * per + own;
  encode_filters(J, sbuf, warp, warps, lane);
  encode_index(J, warp, warps, lane);
  for (uint64_t f = warps - 1 - warp; f < J.ctr->n_files; f += warps) encode_meta_file(J, (uint32_t)f, lane);
}

__global__ void __launch_bounds__(kEncWarps * 32, 2) k_encode_blocks(const JobDev* __restrict__ jobs,
                                                                       uint32_t side) {
  pdl_begin();
  __shared__ uint32_t s_h8[kCrcH8Words];
  __shared__ uint32_t s_xinv[kCrcXinvSmem];
  __shared__ uint32_t s_tab8[256];
  __shared__ JobDev s_job;  // the job's descriptor, read from here in every step
  extern __shared__ __align__(16) uint8_t enc_smem[];
  const JobDev& G = jobs[blockIdx.y];
  if (G.ctr->error) return;
  if (blockIdx.x < side) {
    encode_side(G, reinterpret_cast<uint32_t*>(enc_smem) + (threadIdx.x >> 5) * (kFilterSmem / 4 + 1),
                blockIdx.x, side);
    return;
  }
  const uint32_t cta = blockIdx.x - side, ctas = gridDim.x - side;
  // the surplus CTAs of a small job leave before they load any table
  if (cta * kEncWarps >= max(G.ctr->n_blocks_out, (uint64_t)G.ctr->n_wide)) return;
  copy_job(jobs + blockIdx.y, &s_job);
  for (uint32_t i = threadIdx.x; i < kCrcH8Words; i += blockDim.x) s_h8[i] = G.crc_h8[i];
  for (uint32_t i = threadIdx.x; i < kCrcXinvN; i += blockDim.x) s_xinv[xinv_slot(i)] = G.crc_xinv[i];
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) s_tab8[i] = G.crc_byte[i];
  __syncthreads();
  const JobDev& J = s_job;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  EncWarp& W = reinterpret_cast<EncWarp*>(enc_smem)[warp];
  const uint32_t nb = (uint32_t)J.ctr->n_blocks_out;  // block and survivor indices fit 32 bits
  const RestartDiv rd(J.restart_interval);
  const uint32_t stride = ctas * kEncWarps;
  uint8_t* st = W.stage;
  uint32_t b = cta * kEncWarps + warp;
  EncBlock cur{};
  if (b < nb) {
    cur.off = (uint32_t)J.b_off[b];
    cur.dst = J.out + J.files[J.b_file[b]].out_off + J.b_off[b];
    cur.bsz = J.b_size[b];
    cur.s = J.b_first[b];
    cur.n = J.b_first[b + 1] - cur.s;
    enc_ahead_entries(J, W, cur, lane);
  }
  for (; b < nb; b += stride) {
    // the next block's place and range
    const uint32_t bn = b + stride;
    EncBlock nxt{};
    uint32_t n_file = 0;
    uint64_t n_off = 0;
    if (bn < nb) {
      n_file = J.b_file[bn];
      n_off = J.b_off[bn];
      nxt.bsz = J.b_size[bn];
      nxt.s = J.b_first[bn];
      nxt.n = J.b_first[bn + 1];  // (less nxt.s, below: not waited for here)
    }
    const bool narrow = cur.bsz <= kEncNarrow;  // wide blocks: by their windows, below
    const uint32_t ph = (uint32_t)(reinterpret_cast<uintptr_t>(cur.dst) & 15);
    const uint32_t m0 = ph, m1 = ph + cur.bsz + 1;  // the message: block and type byte
    cp_async_wait_all();  // this lane's entries of the block
    uint32_t ones = 0;
    if (narrow) {
      ones = __ldg(J.crc_ones + (m1 - m0));
      enc_drain(lane);
      enc_assemble<false>(J, W, cur, rd, ph, 0, m1, lane);
    }
    if (bn < nb) {  // the next block's place and entries, in flight meanwhile
      nxt.n -= nxt.s;
      nxt.off = (uint32_t)n_off;
      nxt.dst = J.out + J.files[n_file].out_off + n_off;
      enc_ahead_entries(J, W, nxt, lane);  // each lane's own slots
    }
    if (narrow) {
      uint8_t* gbase = cur.dst - ph;
      const uint32_t full =
          enc_out(J, s_h8, s_xinv, s_tab8, gbase, st, m0, m1, lane) ^ ones ^ 0xffffffffu;
      const uint32_t crc = ((full >> 15) | (full << 17)) + 0xa282ead8u;  // crc32c::Mask
      if (bn < nb && nxt.bsz <= kEncNarrow) {
        cp_async_wait_all();
        enc_prefetch(J, W, nxt.n, lane);
      }
      if (lane == 0) st_le32(st + m1, crc);
      __syncwarp();
      enc_ends(gbase, st, m0, m1, m1 + 4, lane);
      __syncwarp();
    }
    cur = nxt;
  }
  // windows of the wide blocks
  const uint32_t nw = min(J.ctr->n_wide, J.cap_wide);
  for (uint32_t x = cta * kEncWarps + warp; x < nw; x += stride) {
    const uint2 un = J.wide[x];  // block, window
    EncBlock B;
    B.off = (uint32_t)J.b_off[un.x];
    B.dst = J.out + J.files[J.b_file[un.x]].out_off + J.b_off[un.x];
    B.bsz = J.b_size[un.x];
    B.s = J.b_first[un.x];
    B.n = J.b_first[un.x + 1] - B.s;
    const uint32_t ph = (uint32_t)(reinterpret_cast<uintptr_t>(B.dst) & 15);
    const uint32_t end = ph + B.bsz + 1;  // the message's end
    const uint32_t p0 = un.y * kEncWindow, p1 = min(end, p0 + kEncWindow);
    if (p0 >= end) continue;  // the layout counted the longest phase
    enc_drain(lane);
    enc_assemble<true>(J, W, B, rd, ph, p0, p1, lane);
    uint8_t* gbase = B.dst - ph + p0;
    const uint32_t m0 = p0 ? 0 : ph, m1 = p1 - p0;
    const uint32_t raw = enc_out(J, s_h8, s_xinv, s_tab8, gbase, st, m0, m1, lane);
    if (lane == 0) atomicXor(J.b_crc + un.x, crc_shift_tab(J, s_tab8, raw, end - p1));
    enc_ends(gbase, st, m0, m1, m1, lane);
    __syncwarp();
  }
  cp_async_wait_all();
  enc_drain(lane);
}

// The survivors' decoded form for later jobs (keep_decoded): key bytes at
// dec_kcum (a scan of the key lengths), value lengths, prefixes and tags; the
// value places were written by k_encode_blocks.  One warp per 32 survivors,
// lanes over the group's key bytes.
__global__ void k_emit_decoded(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error || !J.dec_keys) return;
  const uint64_t n = J.ctr->n_kept;
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t warps = ((uint64_t)gridDim.x * blockDim.x) >> 5;
  for (uint64_t g = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; g * 32 < n; g += warps) {
    const uint64_t k = g * 32 + lane;
    if (k < n) {
      uint32_t kl;
      const uint8_t* key = kept_key(J, k, &kl);
      J.dec_vlen[k] = J.k_vlen[k];
      J.dec_pfx[k] = user_prefix(key, kl);
      J.dec_tag[k] = ld_le64(key + kl - 8);
    }
    const uint64_t k1 = min(n, g * 32 + 32);
    for (uint64_t j = g * 32; j < k1; j++) {
      uint32_t kl;
      const uint8_t* key = kept_key(J, j, &kl);
      uint8_t* d = J.dec_keys + J.dec_kcum[j];
      for (uint32_t t = lane; t < kl; t += 32) d[t] = key[t];
    }
  }
}

// The filter, metaindex and index blocks' trailers: each region is cut into
// kMetaPiece-byte pieces, one warp per piece (the row CRC, lanes over the
// piece's 16-byte chunks); a piece's raw register, moved to the region's end
// past its type byte, is xored into the file's accumulator (the xor of every
// byte's share is the register of the whole), and k_meta_trailers writes the
// finished CRCs.  As many CTAs work as there are pieces for (a grid of CTAs per
// file and file slot spent 446 us of a 32-job batch on CTAs that loaded their
// tables and had no file; one by the entries alone left the filter offsets of
// large values, 4 bytes per 2 KiB of data, to a few warps: 240 MiB of 4-64 KiB
// values 55 us, and 66 us for the trailers of their 61000 windows; now 12 and 5).

__device__ __forceinline__ void meta_region(const FileOut& F, uint32_t r, uint64_t* off,
                                            uint64_t* len) {
  if (r == 0) {
    *off = F.filter_off;
    *len = F.filter_size;
  } else if (r == 1) {
    *off = F.meta_off;
    *len = F.meta_size;
  } else {
    *off = F.index_off;
    *len = F.index_size;
  }
}

__global__ void __launch_bounds__(256) k_meta_crc(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_h5[kCrcH5Words];
  __shared__ uint32_t s_xinv[kCrcXinvSmem];
  __shared__ uint32_t s_tab8[256];
  if (J.ctr->error) return;
  const uint32_t ctas = min(gridDim.x, (J.ctr->meta_pieces + 7) / 8);  // at work: 8 warps each
  if (blockIdx.x >= ctas) return;
  for (uint32_t i = threadIdx.x; i < kCrcH5Words; i += blockDim.x) s_h5[i] = J.crc_h5[i];
  for (uint32_t i = threadIdx.x; i < kCrcXinvN; i += blockDim.x) s_xinv[xinv_slot(i)] = J.crc_xinv[i];
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) s_tab8[i] = J.crc_byte[i];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, nf = J.ctr->n_files;
  // the pieces of all files are dealt to the job's warps in turn; the lanes
  // look at 32 files at a time for the one that a turn falls into (one after
  // the other, a load chain each, took 23 us with 33 files)
  const uint64_t warps = (uint64_t)ctas * (blockDim.x / 32);
  uint64_t turn = (uint64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  const auto pieces = [&](const FileOut& F, uint64_t* off, uint64_t* len, uint64_t* np) -> uint64_t {
#pragma unroll
    for (uint32_t r = 0; r < 3; r++) {
      meta_region(F, r, &off[r], &len[r]);
      np[r] = meta_pieces(len[r]);  // (no filter: no bytes)
    }
    return np[0] + np[1] + np[2];
  };
  for (uint32_t f0 = 0; f0 < nf; f0 += 32) {
    uint64_t off[3], len[3], np[3];
    const uint64_t mine = f0 + lane < nf ? pieces(J.files[f0 + lane], off, len, np) : 0;
    uint64_t total;
    const uint64_t first = warp_excl<uint64_t>(mine, &total);
    for (; turn < total; turn += warps) {
      const int l = 31 - __clz(__ballot_sync(0xffffffffu, first <= turn && mine));
      const uint32_t f = f0 + l;
      const FileOut& F = J.files[f];
      const uint8_t* fbase = J.out + F.out_off;
      pieces(F, off, len, np);
      uint32_t r = 0;
      uint64_t q = turn - __shfl_sync(0xffffffffu, first, l);
      while (q >= np[r]) q -= np[r++];
      const uint64_t a = q * kMetaPiece, e = min(len[r], a + kMetaPiece);
      const uint8_t* pa = fbase + off[r] + a;
      const uint32_t m0 = (uint32_t)(reinterpret_cast<uintptr_t>(pa) & 15);
      const uint32_t m1 = m0 + (uint32_t)(e - a);
      const uint8_t* g = pa - m0;
      // the lane's chunks of the piece, all loaded before the CRC steps
      constexpr uint32_t kRows = (kMetaPiece + 15) / kCrcRowBytes + 1;
      uint4 v[kRows];
#pragma unroll
      for (uint32_t i = 0; i < kRows; i++) {
        const uint32_t x = 16 * lane + kCrcRowBytes * i;
        if (x < m1) v[i] = *reinterpret_cast<const uint4*>(g + x);
      }
      uint32_t u = 0, last = 0xffffffffu;
#pragma unroll
      for (uint32_t i = 0; i < kRows; i++) {
        const uint32_t x = 16 * lane + kCrcRowBytes * i;
        if (x < m1) {
          u = crc_chunk_step(s_h5, u, x, m0, m1, v[i].x, v[i].y, v[i].z, v[i].w, a == 0);
          last = x;
        }
      }
      const uint32_t raw = crc_rows_raw(s_xinv, s_tab8, u, last, m1);
      if (lane == 0)
        atomicXor(&J.files[f].crc_acc[r], crc_shift_tab(J, s_tab8, raw, len[r] + 1 - e));
    }
    turn -= total;
  }
}

// The register after n zero bytes from all ones.
__device__ __forceinline__ uint32_t crc_ones_after(const JobDev& J, uint64_t n) {
  const uint64_t N = J.crc_xpow_n;
  if (n < N) return J.crc_ones[n];
  if (n >= N * N) return crc_shift(J, 0xffffffffu, n);
  return gf2_mulmod(J.crc_ones[n % N], J.crc_xpow_hi[n / N]);
}

__device__ __forceinline__ void put_trailer(uint8_t* p, uint32_t raw) {
  const uint32_t full = raw ^ 0xffffffffu;
  p[0] = 0;  // kNoCompression
  st_le32(p + 1, ((full >> 15) | (full << 17)) + 0xa282ead8u);  // crc32c::Mask
}

// The trailers of the filter, metaindex and index blocks, and of the data
// blocks that were written in windows.
__global__ void k_meta_trailers(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;
  const uint32_t nf = J.ctr->n_files, nw = min(J.ctr->n_wide, J.cap_wide);
  const uint32_t t0 = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
  for (uint32_t x = t0; x < 3 * nf; x += stride) {
    const uint32_t f = x / 3, r = x % 3;
    if (r == 0 && J.bits_per_key <= 0) continue;
    const FileOut& F = J.files[f];
    uint64_t off, len;
    meta_region(F, r, &off, &len);
    put_trailer(J.out + F.out_off + off + len, F.crc_acc[r]);
  }
  for (uint32_t x = t0; x < nw; x += stride) {
    const uint2 un = J.wide[x];
    if (un.y != 0) continue;  // once per block
    const uint32_t b = un.x, size = J.b_size[b];
    put_trailer(J.out + J.files[J.b_file[b]].out_off + J.b_off[b] + size,
                J.b_crc[b] ^ crc_ones_after(J, (uint64_t)size + 1));
  }
}

// The job's counters and its files' descriptions and boundary keys straight
// into mapped pinned host memory, as many as there are: how many is known only
// here, and a copy of the arrays' capacity (hundreds of files a job) took the
// link 69 us and the host's reading of it 1.3 ms for a batch of 32 jobs.  One
// warp per file; the last kernel of a batch.
__global__ void __launch_bounds__(256) k_results(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (!J.res_ctr) return;
  const uint32_t lane = threadIdx.x & 31, w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const auto copy = [&](void* dst, const void* src, uint32_t n) {  // n: a multiple of 8
    for (uint32_t i = lane; i < n / 8; i += 32)
      reinterpret_cast<uint64_t*>(dst)[i] = reinterpret_cast<const uint64_t*>(src)[i];
  };
  if (w == 0) copy(J.res_ctr, J.ctr, sizeof(Counters));
  if (J.ctr->error) return;
  const uint32_t nf = J.ctr->n_files;
  for (uint32_t f = w; f < nf; f += (gridDim.x * blockDim.x) >> 5) {
    copy(J.res_files + f, J.files + f, sizeof(FileOut));
    const uint32_t l0 = (uint32_t)J.fkoff[2 * f], l1 = (uint32_t)J.fkoff[2 * f + 1];
    if (lane < 2) J.res_klen[2 * f + lane] = lane ? l1 : l0;
    const uint64_t at = 2ull * f * J.fkey_stride;
    for (uint32_t i = lane; i < l0; i += 32) J.res_keys[at + i] = J.fkeys[at + i];
    for (uint32_t i = lane; i < l1; i += 32)
      J.res_keys[at + J.fkey_stride + i] = J.fkeys[at + J.fkey_stride + i];
  }
}

}  // namespace

void launch_sizes(const Batch& bt, cudaStream_t st) {
  launch(k_sizes, dim3(grid_x(bt.max_entries, 256, bt.per_job(148 * 8)), bt.B), 256, 0, st, bt.d);
}

void launch_partition(const Batch& bt, cudaStream_t st) {
  const uint64_t chunks = (bt.max_entries + bt.chunk - 1) / bt.chunk + 1;
  // next() values, sub-chunk words (windows up to kChainSub)
  const size_t smem = ((size_t)bt.chunk + (bt.chunk / kChainSub) * kChainSub) * sizeof(uint32_t);
  const size_t resolve_smem = (size_t)bt.chain_smem_words * 4;
  const unsigned all_ctas = part_ctas(bt.max_entries), blk_ctas = part_ctas(bt.max_blocks_out);
  if (bt.max_entries <= kPartEntries && (uint64_t)all_ctas * bt.jobs_of_largest <= 148) {
    launch_clusters(all_ctas, k_partition<true>, dim3(all_ctas, bt.B), kPartThreads,
                    std::max(smem, resolve_smem), st, bt.d);
    return;
  }
  const auto grid = [&](uint64_t per) {
    return dim3(grid_x(bt.max_entries, (unsigned)per, bt.per_job(148 * 8)), bt.B);
  };
  if (bt.max_entries > kDirectMax && bt.max_block_entries <= kNextHalo / 2) {
    tile_sums_kb(bt, bt.max_entries, st);
    launch(k_scan_next, dim3(grid_x(bt.max_entries + 1, kTile, bt.per_job(148 * 5)), bt.B), kScanThreads,
           0, st, bt.d);
  } else {
    scan_batch(kScanKb, bt, bt.max_entries, st);
    launch(k_next, grid(256), 256, 0, st, bt.d);
  }
  const dim3 g((unsigned)std::min<uint64_t>(chunks, bt.per_job(148 * 4)), bt.B);
  launch(k_chain_tables, g, 256, smem, st, bt.d);
  if (chunks > kChainGroup)  // (one more than the survivors can have)
    launch(k_chain_groups, dim3(grid_x(chunks / kChainGroup * bt.chunk, 256, 148 * 4), bt.B), 256, 0, st, bt.d);
  launch(k_chain_resolve, dim3(1, bt.B), 1024, resolve_smem, st, bt.d);
  launch(k_chain_mark, g, 128, smem, st, bt.d);
  if (bt.max_blocks_out <= kPartBlocks && (uint64_t)blk_ctas * bt.jobs_of_largest <= 148) {
    launch_clusters(blk_ctas, k_partition<false>, dim3(blk_ctas, bt.B), kPartThreads, 0, st, bt.d);
    return;
  }
  launch(k_block_sizes, grid(1024), 256, 0, st, bt.d);
  scan_batch(kScanBcum, bt, bt.max_entries, st);
  launch(k_file_next, grid(256), 256, 0, st, bt.d);
  launch(k_files, dim3(1, bt.B), kFileThreads, 0, st, bt.d);
  launch(k_block_layout, grid(256), 256, 0, st, bt.d);
  scan_batch(kScanIcum, bt, bt.max_entries, st);
  scan_batch(kScanGcum, bt, bt.max_entries, st);
  launch(k_file_layout, dim3(1, bt.B), 256, 0, st, bt.d);
}
void encode_kernel_attributes() {
  cudaFuncSetAttribute(k_partition<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, 64 << 10);
  cudaFuncSetAttribute(k_encode_blocks, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kEncSmem);
}

void launch_encode_blocks(const Batch& bt, cudaStream_t st) {
  // grid-stride over the device-side counts of blocks and windows: 2 CTAs per
  // SM x 4 waves (a job of few entries may have as many windows as its output
  // bytes allow), after the CTAs for everything else: filters and index keys go by
  // the entries, filter offsets and long keys by the bytes
  const uint32_t side = grid_x(bt.max_entries + bt.max_cap_wide / 2, 2048, bt.per_job(148));
  const uint32_t enc =
      grid_x(std::max<uint64_t>(bt.max_entries, bt.max_cap_wide), kEncWarps, bt.per_job(148 * 2 * 4));
  launch(k_encode_blocks, dim3(side + enc, bt.B), kEncWarps * 32, kEncSmem, st, bt.d, side);
}
void launch_emit_decoded(const Batch& bt, cudaStream_t st) {
  if (!bt.any_keep_decoded) return;
  scan_batch(kScanDecKey, bt, bt.max_entries, st);
  launch(k_emit_decoded, dim3(grid_x(bt.max_entries, 256, bt.per_job(148 * 8)), bt.B), 256, 0, st, bt.d);
}
void launch_encode_meta(const Batch& bt, cudaStream_t st) {
  // a CTA for 32 KiB of filter and index: an entry has at most some 64 bytes of
  // them (when it is a block by itself), 16 MiB of data (6600 units of max_cap_wide)
  // have 32 KiB of filter offsets
  launch(k_meta_crc, dim3(grid_x(bt.max_entries + bt.max_cap_wide / 8, 512, bt.per_job(148 * 4)), bt.B),
         256, 0, st, bt.d);
  launch(k_meta_trailers,
         dim3(std::max((3 * bt.max_cap_files + 255) / 256, grid_x(bt.max_cap_wide, 512, bt.per_job(148 * 2))), bt.B),
         256, 0, st, bt.d);
}

void launch_results(const Batch& bt, cudaStream_t st) {
  launch(k_results, dim3(grid_x(bt.max_cap_files, 8, 16), bt.B), 256, 0, st, bt.d);
}

}  // namespace lc
