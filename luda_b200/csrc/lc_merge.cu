// Merge and drop: decoded runs -> survivors in output order.
//
// * Merge: the reference merges its children with MergingIterator
//   (table/merger.cc:148, linear FindSmallest; on equal keys the earlier child
//   wins).  Here the children are merged pairwise in rounds with merge path,
//   in tiles: two warps find the tile's cuts by search, then the CTA stages
//   its two stretches (entry ids and their 8-byte
//   user-key prefixes) in shared memory, merges them there (each thread its
//   own diagonal) and writes ids, prefixes and tags back coalesced, so that a
//   round reads and writes 20 bytes per entry and key bytes are read only for
//   equal prefixes.  Ties go to the left (earlier) group, which keeps child
//   order.  The drop rule then reads prefixes and tags in merged order.
// * Drop rule (db/db_impl.cc:1113-1147): an entry is hidden when the previous
//   entry has the same user key and a sequence number <= smallest_snapshot;
//   a deletion marker is dropped when its sequence number is <=
//   smallest_snapshot and no file at a level >= L+2 covers its user key
//   (Compaction::IsBaseLevelForKey, db/version_set.cc:1535-1554).  Keys whose
//   type byte is not 0/1 (ParseInternalKey fails) are kept and reset the state.
// * Grandparent cuts (Compaction::ShouldStopBefore, db/version_set.cc:
//   1556-1579): evaluated for every merged key, dropped or not.  The number of
//   grandparents whose largest key precedes each merged key is found by binary
//   search; the cut positions are then a chain of threshold searches over the
//   running overlap, which one thread resolves.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "lc_device.cuh"
#include "lc_kernels.h"

namespace lc {

namespace {

// The user-key bytes every input key of the job shares: the common prefix
// of the first and last keys of every merge child (each child is sorted, so
// its keys share what its two ends share) with the first key of child 0.
// Then, per grandparent, its prefix after those bytes, or where it sorts
// against every entry when it does not share them.  One CTA per job.
__global__ void k_key_skip(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed, s_skip;
  if (threadIdx.x == 0) {
    s_failed = J.ctr->error;
    s_skip = 0xffffffffu;
  }
  __syncthreads();
  if (s_failed) return;
  const uint64_t n = J.ctr->n_entries_in;
  uint32_t u0 = 0;
  const uint8_t* k0 = nullptr;
  if (n > 0) {
    k0 = J.keys + J.e_loc[0].x;
    u0 = J.e_loc[0].y - 8;
  }
  // boundary keys: 2 per child
  for (uint32_t x = threadIdx.x; x < 2 * J.n_runs && n > 0; x += blockDim.x) {
    const uint32_t r = x >> 1;
    const uint64_t a = J.run_entry_begin[r], z = J.run_entry_begin[r + 1];
    if (a == z) continue;
    const uint64_t e = (x & 1) ? z - 1 : a;
    const uint8_t* k = J.keys + J.e_loc[e].x;
    const uint32_t u = J.e_loc[e].y - 8, m = min(u, u0);
    uint32_t l = 0;
    while (l < m && k[l] == k0[l]) l++;
    atomicMin(&s_skip, l);
  }
  __syncthreads();
  const uint32_t L = n > 0 ? min(s_skip, u0) : 0;
  if (threadIdx.x == 0) J.ctr->key_skip = L;
  for (uint32_t g = threadIdx.x; g < J.n_gp; g += blockDim.x) {
    const uint64_t go = J.gp_key_off[g];
    const uint8_t* gk = J.gp_keys + go;
    const uint32_t gu = (uint32_t)(J.gp_key_off[g + 1] - go) - 8;
    uint32_t i = 0;
    const uint32_t m = min(gu, L);
    while (i < m && gk[i] == k0[i]) i++;
    uint8_t mode = 0;
    if (i < L) {
      // differs within the common bytes, or ends inside them: it sorts
      // before every entry (1) or after every entry (2)
      mode = (i == gu || gk[i] < k0[i]) ? 1 : 2;
    }
    J.gp_mode[g] = mode;
    J.gp_upfx[g] = mode ? 0 : user_prefix_after(gk, gu + 8, L);
  }
}

// True when entry e is the first of its merge child.
__device__ __forceinline__ bool run_first(const JobDev& J, uint64_t e) {
  // the last child whose first entry is at or before e
  uint32_t lo = 0, hi = J.n_runs;
  while (hi - lo > 1) {
    const uint32_t mid = (lo + hi) >> 1;
    if (J.run_entry_begin[mid] <= e) lo = mid;
    else hi = mid;
  }
  return J.run_entry_begin[lo] == e;
}

// e_pfx after the job's common bytes (the decode wrote the prefixes from the
// keys' first byte), and a check of the merge children's order: every key
// starts with the common bytes and sorts at or after the entry before it in
// its child.  table/merger.cc merges children it trusts to be sorted; a child
// out of order fails the job here (kErrUnsorted) rather than reaching the
// merge path, whose cuts assume sorted children.
__global__ void __launch_bounds__(256, 8) k_prefix(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;
  const uint32_t L = J.ctr->key_skip;
  const uint64_t n = J.ctr->n_entries_in;
  if (n == 0) return;
  const uint8_t* k0 = J.keys + J.e_loc[0].x;
  for (uint64_t e = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n;
       e += (uint64_t)gridDim.x * blockDim.x) {
    const uint8_t* k = J.keys + J.e_loc[e].x;
    const uint32_t kl = J.e_loc[e].y;  // >= 8: shorter keys failed the decode
    bool bad = false;
    uint64_t p;
    if (L) {
      if (kl - 8 < L) {
        bad = true;
      } else {
        for (uint32_t i = 0; i < L; i++) bad |= k[i] != k0[i];
      }
      p = user_prefix_after(k, kl, L);
      J.e_pfx[e] = p;  // neighbours recompute theirs from the key bytes
    } else {
      p = J.e_pfx[e];
    }
    if (!bad && e > 0 && !run_first(J, e)) {
      const uint8_t* kp = J.keys + J.e_loc[e - 1].x;
      const uint32_t klp = J.e_loc[e - 1].y;
      const uint64_t pp = L ? (klp - 8 < L ? 0 : user_prefix_after(kp, klp, L)) : J.e_pfx[e - 1];
      bad = pp > p || (pp == p && ikey_cmp(kp, klp, k, kl) > 0);
    }
    if (bad) set_error(J.ctr, kErrUnsorted, (uint32_t)e);
  }
}

// A single merge child (no round): the merged order is the input order.
__global__ void k_merge_single(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // a failed job does no more work
  const uint64_t n = J.ctr->n_entries_in;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    J.m_ids[i] = (uint32_t)i;
    J.m_pfx[i] = J.e_pfx[i];
    J.m_tag[i] = J.e_tag[i];
  }
}

// Round r of `rounds` merges groups of 2^r children pairwise: the output of
// pair p (groups 2p and 2p+1) is cut into tiles of `tile` positions.  Round 0
// reads the decoded entries in input order (ids are positions, prefixes and
// tags are e_pfx / e_tag); later rounds read the previous round's arrays.
// Jobs with fewer children copy through, so that every job of a batch ends
// with its merged order in m_ids / m_pfx / m_tag.
struct MergeRound {
  const uint32_t* src_ids;  // nullptr in round 0
  const uint64_t* src_pfx;
  const uint64_t* src_tag;
  uint32_t* dst_ids;
  uint64_t* dst_pfx;
  uint64_t* dst_tag;
};

__device__ __forceinline__ MergeRound merge_round(const JobDev& J, uint32_t r, uint32_t rounds) {
  const bool odd = ((rounds - r) & 1) != 0;
  MergeRound m;
  m.src_ids = r == 0 ? nullptr : (odd ? J.m_tmp : J.m_ids);
  m.src_pfx = r == 0 ? J.e_pfx : (odd ? J.m_pfx_tmp : J.m_pfx);
  m.src_tag = r == 0 ? J.e_tag : (odd ? J.m_tag_tmp : J.m_tag);
  m.dst_ids = odd ? J.m_ids : J.m_tmp;
  m.dst_pfx = odd ? J.m_pfx : J.m_pfx_tmp;
  m.dst_tag = odd ? J.m_tag : J.m_tag_tmp;
  return m;
}

// Pair and tile of the job's g-th merge tile in round r; false past the last.
struct MergeTile {
  uint64_t a0, na, nb;  // the pair's first group [a0, a0 + na), second [a0 + na, + nb)
  uint64_t d0, d1;      // the tile's output positions within the pair
  bool last;            // last tile of its pair
};

__device__ __forceinline__ bool merge_tile(const JobDev& J, uint32_t r, uint64_t g, uint32_t tile,
                                           MergeTile* t) {
  const uint32_t width = 1u << r;
  uint64_t acc = 0;
  for (uint32_t r0 = 0; r0 < J.n_runs; r0 += 2 * width) {
    const uint32_t r1 = min(r0 + width, J.n_runs), r2 = min(r0 + 2 * width, J.n_runs);
    const uint64_t a0 = J.run_entry_begin[r0], b0 = J.run_entry_begin[r1],
                   b1 = J.run_entry_begin[r2];
    const uint64_t len = b1 - a0, tiles = (len + tile - 1) / tile;
    if (g < acc + tiles) {
      const uint64_t k = g - acc;
      t->a0 = a0;
      t->na = b0 - a0;
      t->nb = b1 - b0;
      t->d0 = k * tile;
      t->d1 = min(len, t->d0 + tile);
      t->last = k + 1 == tiles;
      return true;
    }
    acc += tiles;
  }
  return false;
}

__device__ __forceinline__ uint32_t src_id(const MergeRound& m, uint64_t i) {
  return m.src_ids ? m.src_ids[i] : (uint32_t)i;
}

// Elements of the pair's first group before output position d (merge path:
// the first group wins ties, which keeps the children's order for equal
// internal keys, as MergingIterator does), by one warp: 32 places a step.
__device__ __forceinline__ uint64_t merge_split(const JobDev& J, const MergeRound& m,
                                                const MergeTile& t, uint64_t d) {
  const uint32_t lane = threadIdx.x & 31;
  const uint64_t a = t.a0, b = t.a0 + t.na;
  uint64_t lo = d > t.nb ? d - t.nb : 0, hi = d < t.na ? d : t.na;
  while (lo < hi) {
    const uint64_t step = (hi - lo + 31) / 32, mid = lo + lane * step;
    bool le = false;
    if (mid < hi) {
      const uint64_t ia = a + mid, ib = b + (d - 1 - mid);
      le = entry_le(J, src_id(m, ia), m.src_pfx[ia], src_id(m, ib), m.src_pfx[ib]);
    }
    const int c = __popc(__ballot_sync(0xffffffffu, le));  // true up to the split
    if (c == 0) break;
    hi = min(hi, lo + c * step);
    lo = lo + (c - 1) * step + 1;
  }
  return lo;
}

// One tile per CTA step: two warps find its cuts (a kernel of its own did, one
// thread per tile and 16 dependent steps: 21 us of an 80k-entry job's two
// rounds on B200), the tile's stretches of both groups (ids and prefixes) are
// loaded into shared memory with coalesced reads, every thread
// finds its own diagonal there and merges `items` outputs as source positions,
// and the tile is written back with coalesced stores, ids and prefixes from
// shared memory and the tags from memory by source position (two ascending
// streams).  Only equal prefixes read key bytes, word by word.  Bound by latency, the tile's
// loads and the barriers behind them before the serial merge in shared memory
// (of 2M entries 13.3, 7.6 and 2.2 cycles a warp and instruction issued; DRAM at
// 9%): 14 bytes of shared memory a position instead of 28 and 40 registers (the
// comparison's 48 bytes are spilled) give an SM 48 warps instead of 24 (8M entries on B200:
// 221 -> 166 us).
__global__ void __maxnreg__(40) k_merge_tile(const JobDev* __restrict__ jobs, uint32_t r,
                                                     uint32_t rounds, uint32_t items) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  __shared__ uint64_t s_cut[2];
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  const uint32_t tile = blockDim.x * items;
  extern __shared__ __align__(16) uint8_t merge_smem[];
  uint64_t* in_pfx = reinterpret_cast<uint64_t*>(merge_smem);
  uint32_t* in_ids = reinterpret_cast<uint32_t*>(in_pfx + tile);
  uint16_t* out_src = reinterpret_cast<uint16_t*>(in_ids + tile);  // source position (in the
                                                                   // tile) of each output
  const MergeRound m = merge_round(J, r, rounds);
  for (uint64_t g = blockIdx.x;; g += gridDim.x) {
    MergeTile t;
    if (!merge_tile(J, r, g, tile, &t)) break;
    __syncthreads();  // the previous tile's cuts have been read
    if (threadIdx.x < 64) {  // at least two warps (lc_set_tuning)
      const uint32_t w = threadIdx.x >> 5;
      const uint64_t cut = w && t.last ? t.na : merge_split(J, m, t, w ? t.d1 : t.d0);
      if ((threadIdx.x & 31) == 0) s_cut[w] = cut;
    }
    __syncthreads();
    const uint64_t i0 = s_cut[0], i1 = s_cut[1];
    if (i1 < i0 || i1 - i0 > t.d1 - t.d0) {
      // cuts out of order: only children out of order give these, and the
      // order check fails such a job first; the tile is skipped, never read
      if (threadIdx.x == 0) set_error(J.ctr, kErrUnsorted, (uint32_t)g);
      continue;
    }
    const uint64_t j0 = t.d0 - i0, j1 = t.d1 - i1;
    const uint32_t na = (uint32_t)(i1 - i0), nb = (uint32_t)(j1 - j0), len = na + nb;
    __syncthreads();  // the previous tile's stores have read the buffers
    for (uint32_t x = threadIdx.x; x < len; x += blockDim.x) {
      const uint64_t i = x < na ? t.a0 + i0 + x : t.a0 + t.na + j0 + (x - na);
      in_ids[x] = src_id(m, i);
      in_pfx[x] = m.src_pfx[i];
    }
    __syncthreads();
    const uint32_t k = threadIdx.x * items;
    if (k < len) {
      // this thread's diagonal within the tile
      uint32_t lo = k > nb ? k - nb : 0, hi = k < na ? k : na;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        const uint32_t jb = na + (k - 1 - mid);
        if (entry_le(J, in_ids[mid], in_pfx[mid], in_ids[jb], in_pfx[jb])) lo = mid + 1;
        else hi = mid;
      }
      uint32_t i = lo, j = k - lo;
      const uint32_t stop = min(len, k + items);
      for (uint32_t o = k; o < stop; o++) {
        const bool take_a =
            i < na && (j >= nb || entry_le(J, in_ids[i], in_pfx[i], in_ids[na + j], in_pfx[na + j]));
        out_src[o] = (uint16_t)(take_a ? i++ : na + j++);
      }
    }
    __syncthreads();
    const uint64_t o0 = t.a0 + t.d0;
    for (uint32_t x = threadIdx.x; x < len; x += blockDim.x) {
      const uint32_t y = out_src[x];
      m.dst_ids[o0 + x] = in_ids[y];
      m.dst_pfx[o0 + x] = in_pfx[y];
      m.dst_tag[o0 + x] = m.src_tag[y < na ? t.a0 + i0 + y : t.a0 + t.na + j0 + (y - na)];
    }
  }
}

__device__ __forceinline__ bool is_base_level(const JobDev& J, const uint8_t* ukey, uint32_t ulen) {
  for (uint32_t l = 0; l < J.n_base_levels; l++) {
    uint32_t lo = J.base_level_begin[l], hi = J.base_level_begin[l + 1];
    const uint32_t end = hi;
    // first file whose largest user key >= ukey
    while (lo < hi) {
      uint32_t mid = (lo + hi) >> 1;
      if (bytes_cmp(ukey, ulen, J.base_keys + J.base_large_off[mid], J.base_large_len[mid]) > 0)
        lo = mid + 1;
      else
        hi = mid;
    }
    if (lo < end &&
        bytes_cmp(ukey, ulen, J.base_keys + J.base_small_off[lo], J.base_small_len[lo]) >= 0)
      return false;
  }
  return true;
}

// Two entries of equal prefixes: the same user key?  (Lengths first: keys that
// are prefixes of one another would be walked to the shorter one's end.)
__device__ __forceinline__ bool same_user_key_rest(const JobDev& J, uint32_t a, uint32_t b) {
  return J.e_loc[a].y == J.e_loc[b].y && user_key_rest_cmp(J, a, b) == 0;
}

// The drop rule for merged position p (tag, prefix), after position p - 1
// (ptag, ppfx); `in`: there is such a position.  Every lane of the warp takes part:
// they meet again after each of the two rare searches.
__device__ __forceinline__ bool keep_entry(const JobDev& J, uint64_t p, bool in, uint64_t tag,
                                           uint64_t upfx, uint64_t ptag, uint64_t ppfx) {
  const uint32_t type = (uint32_t)(tag & 0xff);
  bool hidden = in && type <= 1 && p > 0 && ppfx == upfx && (ptag & 0xff) <= 1 &&
                (ptag >> 8) <= J.smallest_snapshot;
  if (__any_sync(0xffffffffu, hidden)) {
    if (hidden) hidden = same_user_key_rest(J, J.m_ids[p - 1], J.m_ids[p]);
    __syncwarp();
  }
  bool dead = in && !hidden && type == 0 && (tag >> 8) <= J.smallest_snapshot;
  if (__any_sync(0xffffffffu, dead)) {
    if (dead) {
      const uint32_t id = J.m_ids[p];
      dead = is_base_level(J, J.keys + J.e_loc[id].x, J.e_loc[id].y - 8);
    }
    __syncwarp();
  }
  return in && !hidden && !dead;
}

// Grandparents passed at merged position p: the count of g with key >
// largest[g] (internal-key order); the user-key prefixes decide unless equal.
__device__ __forceinline__ uint32_t grandparents_passed(const JobDev& J, uint64_t p, uint64_t upfx) {
  uint32_t lo = 0, hi = J.n_gp;
  while (lo < hi) {
    const uint32_t mid = (lo + hi) >> 1;
    const uint64_t gp = J.gp_upfx[mid];
    const uint32_t mode = J.gp_mode[mid];
    bool after;
    if (mode) {  // the grandparent lies outside the keys' common prefix
      after = mode == 1;
    } else if (gp != upfx) {
      after = upfx > gp;
    } else {
      const uint32_t id = J.m_ids[p];
      const uint64_t go = J.gp_key_off[mid];
      const uint32_t gl = (uint32_t)(J.gp_key_off[mid + 1] - go);
      after = ikey_cmp(J.keys + J.e_loc[id].x, J.e_loc[id].y, J.gp_keys + go, gl) > 0;
    }
    if (after) lo = mid + 1;
    else hi = mid;
  }
  return lo;
}

// Survivors are found and gathered in tiles of kKeepTile merged positions:
// k_drop marks them and counts each tile's, k_kept_compact gives every tile
// its place (the counts before it) and gathers.  A warp of k_drop loads its
// strips of 32 positions ahead (tag and prefix; the position before a lane's
// is its neighbour's, by shuffle); entry ids only where two prefixes are equal.
// Bound by latency: k_drop by its two streams' loads (40 registers for 48 warps an
// SM; the rare paths' 40 bytes are spilled), k_kept_compact by the gathers from
// the entry arrays (issue at 38%).  With the flags' scan and the gather as kernels
// of their own, 8M entries took 117 + 26 + 91 us on B200 and the entry sizes 108
// more; k_drop and k_kept_compact take 68 + 187.
// A tile is kStrips positions a thread: four, or one in jobs whose tiles of four
// would leave SMs with less than eight.  There the time is that of the rare paths'
// key comparisons in one warp, strip after strip: 232 deletions of keys with 40
// bytes in common, looked up in 60 files below, 238 us for both kernels with
// four, 90 with one; 80000 entries without long comparisons 18 and 16, 267000 55
// and 51.
constexpr uint32_t kKeepThreads = 128;
static_assert(kKeepThreads >= 128, "the counts fit scan_scratch (scan_scratch_elems)");

template <uint32_t kStrips>
__global__ void __launch_bounds__(kKeepThreads, 12) k_drop(const JobDev* __restrict__ jobs) {
  pdl_begin();
  constexpr uint32_t kKeepTile = kStrips * kKeepThreads;
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed, s_count;
  if (threadIdx.x == 0) {
    s_failed = J.ctr->error;
    s_count = 0;
  }
  __syncthreads();
  if (s_failed) return;
  const uint64_t n = J.ctr->n_entries_in;
  uint32_t* counts = reinterpret_cast<uint32_t*>(J.scan_scratch);
  const uint64_t* tags = J.m_tag;
  const uint64_t* pfx = J.m_pfx;
  const bool gps = J.n_gp != 0;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint64_t t = blockIdx.x; t * kKeepTile < n; t += gridDim.x) {
    const uint64_t w0 = t * kKeepTile + 32 * kStrips * warp;  // the warp's positions
    uint64_t tg[kStrips], px[kStrips];
#pragma unroll
    for (uint32_t i = 0; i < kStrips; i++) {
      const uint64_t p = w0 + 32 * i + lane;
      tg[i] = p < n ? tags[p] : 0xff;
      px[i] = p < n ? pfx[p] : 0;
    }
    uint64_t lt = w0 > 0 && w0 < n ? tags[w0 - 1] : 0, lp = w0 > 0 && w0 < n ? pfx[w0 - 1] : 0;
    uint32_t cnt = 0;
#pragma unroll
    for (uint32_t i = 0; i < kStrips; i++) {
      const uint64_t p = w0 + 32 * i + lane;
      const uint64_t ut = __shfl_up_sync(0xffffffffu, tg[i], 1);
      const uint64_t up = __shfl_up_sync(0xffffffffu, px[i], 1);
      const bool keep = keep_entry(J, p, p < n, tg[i], px[i], lane ? ut : lt, lane ? up : lp);
      if (p < n) {
        J.keep[p] = keep ? 1 : 0;
        if (gps) J.gp_idx[p] = grandparents_passed(J, p, px[i]);
      }
      lt = __shfl_sync(0xffffffffu, tg[i], 31);
      lp = __shfl_sync(0xffffffffu, px[i], 31);
      cnt += __popc(__ballot_sync(0xffffffffu, keep));
    }
    if (lane == 0 && cnt) atomicAdd(&s_count, cnt);
    __syncthreads();
    if (threadIdx.x == 0) {
      counts[t] = s_count;
      s_count = 0;
    }
    __syncthreads();
  }
}

// gp_first[g] = first merged position whose grandparent count reaches g
// (gp_idx is non-decreasing along the merge order).
__global__ void k_gp_first(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // a failed job does no more work
  uint32_t* gp_first = J.gp_first;
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g > J.n_gp) return;
  const uint64_t n = J.ctr->n_entries_in;
  uint64_t lo = 0, hi = n;
  while (lo < hi) {
    const uint64_t mid = (lo + hi) >> 1;
    if (J.gp_idx[mid] >= g) hi = mid;
    else lo = mid + 1;
  }
  gp_first[g] = (uint32_t)lo;
}

// The cut positions: after a cut at t (or from the first key), the next cut
// is the first key whose running overlap exceeds the limit, i.e. the first
// position whose grandparent count reaches the smallest g with
// prefix[g] - prefix[gp_idx[t]] > limit.  Few cuts; one thread walks them
// over shared-memory copies of the prefix and first-position arrays.
__global__ void k_triggers(const JobDev* __restrict__ jobs, bool in_smem) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed;  // read once per CTA: the CTA's barriers stay uniform
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  const uint32_t* gp_first = J.gp_first;
  extern __shared__ uint64_t s_tr[];
  const uint64_t n = J.ctr->n_entries_in;
  const uint32_t G = J.n_gp;
  const uint64_t* pre = J.gp_prefix;
  const uint32_t* first = gp_first;
  if (in_smem) {  // G + 1 prefixes, then G + 1 first positions
    uint32_t* s_first = reinterpret_cast<uint32_t*>(s_tr + G + 1);
    for (uint32_t g = threadIdx.x; g <= G; g += blockDim.x) {
      s_tr[g] = J.gp_prefix[g];
      s_first[g] = gp_first[g];
    }
    pre = s_tr;
    first = s_first;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  uint32_t cnt = 0;
  if (n > 0 && G > 0) {
    const uint64_t limit = (uint64_t)J.max_gp_overlap;
    uint32_t gb = J.gp_idx[0];
    while (true) {
      const uint64_t target = pre[gb] + limit;  // need prefix > target
      uint32_t lo = gb + 1, hi = G + 1;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (pre[mid] > target) hi = mid;
        else lo = mid + 1;
      }
      if (lo > G) break;
      const uint64_t t = first[lo];
      if (t >= n) break;
      if (cnt >= J.cap_triggers) {
        set_error(J.ctr, kErrLimit, 1);
        break;
      }
      J.triggers[cnt++] = (uint32_t)t;
      gb = J.gp_idx[t];
    }
  }
  J.ctr->n_triggers = cnt;
}

// Sum of v over the CTA (kKeepThreads threads); every thread gets it, and *before
// the sum over the threads before it.
__device__ __forceinline__ uint32_t keep_scan(uint32_t v, uint32_t* s_warp, uint32_t* before) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t u = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += u;
  }
  __syncthreads();  // the last call's sums have been read
  if (lane == 31) s_warp[warp] = x;
  __syncthreads();
  uint32_t all = 0, b = 0;
#pragma unroll
  for (uint32_t w = 0; w < kKeepThreads / 32; w++) {
    const uint32_t y = s_warp[w];
    if (w < warp) b += y;
    all += y;
  }
  *before = b + x - v;
  return all;
}

// The last survivor before tile t (which has some before it), by one warp.
template <uint32_t kKeepTile>
__device__ __forceinline__ uint64_t last_kept_before(const JobDev& J, const uint32_t* counts,
                                                     uint64_t t) {
  const uint32_t lane = threadIdx.x & 31;
  uint64_t hi = t;  // the tile, from 32 at a time
  while (true) {
    const bool any = hi > lane && counts[hi - 1 - lane] != 0;
    const unsigned m = __ballot_sync(0xffffffffu, any);
    if (m) {
      hi = hi - 1 - (__ffs(m) - 1);
      break;
    }
    hi -= 32;
  }
  for (int32_t w = kKeepTile / 32 - 1; w >= 0; w--) {
    const uint64_t p = hi * kKeepTile + 32 * w + lane;
    const unsigned m = __ballot_sync(0xffffffffu, J.keep[p] != 0);
    if (m) return p - lane + (31 - __clz(m));
  }
  return 0;  // not reached
}

// The tile's survivors gather their entries and get their sizes: as a restart
// entry (k_a), as a prefix-compressed entry (k_b), and the prefix each shares
// with the survivor before it (its neighbour's id, key length and prefix come by
// shuffle).  The two prefixes (the 8 user-key bytes after the job's common
// ones) give the shared length when they differ inside both user keys; key
// bytes are read only otherwise.  kPer survivors per thread at a time, so that
// their loads overlap.
template <uint32_t kPer>
__device__ __forceinline__ void gather_kept(const JobDev& J, const uint16_t* s_list, uint32_t total,
                                            uint64_t t0, uint32_t base, uint64_t prev,
                                            unsigned long long* kb, unsigned long long* vb) {
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t L = J.ctr->key_skip;
  for (uint32_t j0 = 32 * kPer * warp; j0 < total; j0 += kPer * kKeepThreads) {
    uint32_t id[kPer], koff[kPer], kl[kPer], voff[kPer], vl[kPer], hash[kPer];
    uint64_t px[kPer];
#pragma unroll
    for (uint32_t i = 0; i < kPer; i++) {
      const uint32_t j = j0 + 32 * i + lane;
      const uint64_t p = t0 + s_list[j < total ? j : 0];
      id[i] = J.m_ids[p];
      px[i] = J.m_pfx[p];
    }
    // the survivor before the warp's first
    const bool any_prev = base + j0 != 0;
    const uint64_t pp = j0 ? t0 + s_list[j0 - 1] : prev;
    uint32_t lid = any_prev ? J.m_ids[pp] : 0u, lkl = any_prev ? J.e_loc[lid].y : 8u;
    uint64_t lpx = any_prev ? J.m_pfx[pp] : 0u;
#pragma unroll
    for (uint32_t i = 0; i < kPer; i++) {
      const uint4 loc = J.e_loc[id[i]];
      koff[i] = loc.x, kl[i] = loc.y, voff[i] = loc.z, vl[i] = loc.w;
      hash[i] = J.bits_per_key > 0 ? J.e_hash[id[i]] : 0u;
    }
#pragma unroll
    for (uint32_t i = 0; i < kPer; i++) {
      const uint32_t j = j0 + 32 * i + lane;
      uint32_t pid = __shfl_up_sync(0xffffffffu, id[i], 1);
      uint32_t pl = __shfl_up_sync(0xffffffffu, kl[i], 1);
      uint64_t ppx = __shfl_up_sync(0xffffffffu, px[i], 1);
      if (lane == 0) pid = lid, pl = lkl, ppx = lpx;
      lid = __shfl_sync(0xffffffffu, id[i], 31);
      lkl = __shfl_sync(0xffffffffu, kl[i], 31);
      lpx = __shfl_sync(0xffffffffu, px[i], 31);
      if (j >= total) continue;
      const uint32_t k = base + j;
      uint32_t shared = 0;
      if (k) {
        const uint32_t m = min(kl[i], pl), mu = m - 8;
        const uint64_t d = px[i] ^ ppx;
        shared = min(L + (d ? (uint32_t)__clzll(d) >> 3 : 8u), mu);
        if (!d || shared == mu) {
          const uint8_t *x = J.keys + koff[i], *y = J.keys + J.e_loc[pid].x;
          while (shared < m && x[shared] == y[shared]) shared++;
        }
      }
      J.k_koff[k] = koff[i];
      J.k_klen[k] = kl[i];
      J.k_voff[k] = voff[i];
      J.k_vlen[k] = vl[i];
      if (J.bits_per_key > 0) J.k_hash[k] = hash[i];
      J.k_a[k] = 1 + varint_len32(kl[i]) + varint_len32(vl[i]) + kl[i] + vl[i];
      J.k_b[k] = varint_len32(shared) + varint_len32(kl[i] - shared) + varint_len32(vl[i]) +
                 (kl[i] - shared) + vl[i];
      J.k_shared[k] = shared;
      *kb += kl[i];
      *vb += vl[i];
    }
  }
}

template <uint32_t kStrips>
__global__ void __launch_bounds__(kKeepThreads, 8) k_kept_compact(const JobDev* __restrict__ jobs) {
  pdl_begin();
  constexpr uint32_t kKeepTile = kStrips * kKeepThreads;
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_failed, s_warp[kKeepThreads / 32];
  __shared__ uint16_t s_list[kKeepTile];  // the tile's survivors
  __shared__ uint64_t s_prev;
  if (threadIdx.x == 0) s_failed = J.ctr->error;
  __syncthreads();
  if (s_failed) return;
  const uint64_t n = J.ctr->n_entries_in;
  if (blockIdx.x * (uint64_t)kKeepTile >= n) return;
  const uint32_t* counts = reinterpret_cast<const uint32_t*>(J.scan_scratch);
  const uint32_t nt = J.ctr->n_triggers;
  const auto before = [&](uint64_t a, uint64_t z) -> uint32_t {  // survivors of tiles [a, z)
    uint32_t x = 0, ex;
    for (uint64_t i = a + threadIdx.x; i < z; i += kKeepThreads) x += counts[i];
    return keep_scan(x, s_warp, &ex);
  };
  uint32_t base = before(0, blockIdx.x);
  unsigned long long kb = 0, vb = 0;
  for (uint64_t t = blockIdx.x; t * kKeepTile < n; t += gridDim.x) {
    const uint64_t t0 = t * kKeepTile, tb = t0 + kStrips * threadIdx.x;
    uint32_t w = 0;  // the thread's flags
    if constexpr (kStrips == 4) {
      w = tb < n ? *reinterpret_cast<const uint32_t*>(J.keep + tb) : 0;
      if (tb < n && n - tb < 4) w &= (1u << (8 * (uint32_t)(n - tb))) - 1;
    } else {
      static_assert(kStrips == 1);
      w = tb < n ? J.keep[tb] : 0;
    }
    uint32_t at;
    const uint32_t total = keep_scan((uint32_t)__popc(w), s_warp, &at);
    for (uint32_t m = w; m; m &= m - 1) s_list[at++] = (uint16_t)(kStrips * threadIdx.x + ((__ffs(m) - 1) >> 3));
    if (base && threadIdx.x < 32) {
      const uint64_t x = last_kept_before<kKeepTile>(J, counts, t);
      if (threadIdx.x == 0) s_prev = x;
    }
    __syncthreads();
    gather_kept<kStrips == 1 ? 1 : 2>(J, s_list, total, t0, base, s_prev, &kb, &vb);
    // the survivors before each grandparent cut in the tile
    if (nt) {
      uint32_t lo = 0, hi = nt;
      while (lo < hi) {
        const uint32_t mid = (lo + hi) >> 1;
        if (J.triggers[mid] < t0) lo = mid + 1;
        else hi = mid;
      }
      for (uint32_t i = lo + threadIdx.x; i < nt && J.triggers[i] < t0 + kKeepTile; i += kKeepThreads) {
        const uint32_t off = (uint32_t)(J.triggers[i] - t0);
        uint32_t a = 0, z = total;
        while (a < z) {
          const uint32_t mid = (a + z) >> 1;
          if (s_list[mid] < off) a = mid + 1;
          else z = mid;
        }
        J.t_kept[i] = base + a;
      }
    }
    if (t0 + kKeepTile >= n && threadIdx.x == 0) J.ctr->n_kept = base + total;
    if ((t + gridDim.x) * kKeepTile < n) base += total + before(t + 1, t + gridDim.x);
    __syncthreads();  // the list is rewritten
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

}  // namespace

static unsigned flat_ctas(const Batch& bt, uint64_t items, unsigned per) {
  return grid_x(items, per, bt.per_job(148 * 8));
}

// Merge tile: threads x items, at most kMergeMaxTile (a source position in
// the tile fits 16 bits), and no more items than leave every SM two tiles: a
// small job is bound by one tile's serial merge, so it takes more, shorter ones
// (80k entries in
// two rounds on B200: 44 us with 2048-position tiles, 20 us with 512).
static uint32_t merge_items_of(const Batch& bt) {
  uint32_t items = std::max<uint32_t>(1, bt.merge_items);
  while ((uint64_t)bt.merge_threads * items > kMergeMaxTile && items > 1) items >>= 1;
  while (items > 1 && bt.max_entries * bt.jobs_of_largest < 2ull * 148 * bt.merge_threads * items)
    items >>= 1;
  return items;
}

void merge_kernel_attributes() {
  cudaFuncSetAttribute(k_merge_tile, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)(kMergeSmemPerPos * kMergeMaxTile));
}

void launch_key_skip(const Batch& bt, cudaStream_t st) {
  launch(k_key_skip, dim3(1, bt.B), 256, 0, st, bt.d);
  launch(k_prefix, dim3(flat_ctas(bt, bt.max_entries, 256), bt.B), 256, 0, st, bt.d);
}

void launch_merge(const Batch& bt, cudaStream_t st) {
  if (bt.merge_rounds == 0) {
    launch(k_merge_single, dim3(flat_ctas(bt, bt.max_entries, 256), bt.B), 256, 0, st, bt.d);
    return;
  }
  const uint32_t items = merge_items_of(bt);
  const uint32_t threads = bt.merge_threads;
  const uint32_t tile = threads * items;
  const uint64_t tiles = bt.max_entries / tile + bt.max_runs + 1;
  for (uint32_t r = 0; r < bt.merge_rounds; r++) {
    launch(k_merge_tile, dim3(flat_ctas(bt, tiles, 1), bt.B), threads, kMergeSmemPerPos * (size_t)tile, st, bt.d, r, bt.merge_rounds, items);
  }
}

// Positions a thread of k_drop and k_kept_compact: four when the batch has eight
// tiles of four for every SM.
static uint32_t keep_strips(const Batch& bt) {
  return bt.max_entries * bt.jobs_of_largest < 148ull * 8 * 4 * kKeepThreads ? 1 : 4;
}

void launch_drop(const Batch& bt, cudaStream_t st) {
  const uint32_t strips = keep_strips(bt);
  const dim3 g(grid_x(bt.max_entries, strips * kKeepThreads, bt.per_job(148 * 12)), bt.B);
  launch(strips == 1 ? k_drop<1> : k_drop<4>, g, kKeepThreads, 0, st, bt.d);
}

void launch_triggers(const Batch& bt, cudaStream_t st) {
  if (!bt.max_gp) return;  // no job has grandparents: no cuts (the counters start at zero)
  launch(k_gp_first, dim3((bt.max_gp + 1 + 255) / 256, bt.B), 256, 0, st, bt.d);
  const size_t smem = (size_t)(bt.max_gp + 1) * 12;
  const bool in_smem = smem + 64 <= 48 * 1024;  // with the kernel's static shared memory
  launch(k_triggers, dim3(1, bt.B), 256, in_smem ? smem : 0, st, bt.d, in_smem);
}

void launch_kept_compact(const Batch& bt, cudaStream_t st) {
  const uint32_t strips = keep_strips(bt);
  const dim3 g(grid_x(bt.max_entries, strips * kKeepThreads, bt.per_job(148 * 12)), bt.B);
  launch(strips == 1 ? k_kept_compact<1> : k_kept_compact<4>, g, kKeepThreads, 0, st, bt.d);
}

}  // namespace lc
