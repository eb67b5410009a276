// Decode: input tables -> entries (keys reconstructed into a key arena, values
// left in place).
//
// Follows the reference's table reader: Footer::DecodeFrom
// (table/format.cc:42-62), the index block's block handles
// (table/table.cc:38-111), and Block::Iter's entry parse (table/block.cc:
// 170-190, 340-367).  The LUDA restart word (table/block_builder.cc:62-66,
// 90-96) is (offset << 8) | entries in that restart run, so every restart run
// is decoded independently: the run's first entry has no shared prefix, and
// the run's entry count is known from the word before any entry is parsed.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "lc_device.cuh"
#include "lc_kernels.h"
#include "lc_scan.cuh"

namespace lc {

namespace {

constexpr uint32_t kMagicLo = 0x8b80fb57u;  // kTableMagicNumber (table/format.h:77)
constexpr uint32_t kMagicHi = 0xdb477524u;

template <typename T>
__device__ __forceinline__ T warp_sum(T v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

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

// Locates the index block of a table; false if the footer is invalid.
__device__ bool parse_footer(const uint8_t* t, uint64_t n, uint64_t* i_off, uint64_t* i_size) {
  if (n < kFooter) return false;
  const uint8_t* f = t + n - kFooter;
  if (ld_le32(f + 40) != kMagicLo || ld_le32(f + 44) != kMagicHi) return false;
  uint64_t m_off, m_size;
  const uint8_t* p = f;
  const uint8_t* lim = f + 40;
  if (!(p = get_varint64(p, lim, &m_off))) return false;
  if (!(p = get_varint64(p, lim, &m_size))) return false;
  if (!(p = get_varint64(p, lim, i_off))) return false;
  if (!(p = get_varint64(p, lim, i_size))) return false;
  if (*i_off > n || *i_size < 4 || *i_size + kTrailer > n - *i_off) return false;
  return true;
}

// Parses one entry header at p (bounded by lim).  Returns the key-delta
// pointer or nullptr.
__device__ __forceinline__ const uint8_t* entry_header(const uint8_t* p, const uint8_t* lim,
                                                       uint32_t* shared, uint32_t* non_shared,
                                                       uint32_t* vlen) {
  if (lim - p < 3) return nullptr;
  uint32_t a = p[0], b = p[1], c = p[2];
  if ((a | b | c) < 128) {
    *shared = a;
    *non_shared = b;
    *vlen = c;
    p += 3;
  } else {
    if (!(p = get_varint32(p, lim, shared))) return nullptr;
    if (!(p = get_varint32(p, lim, non_shared))) return nullptr;
    if (!(p = get_varint32(p, lim, vlen))) return nullptr;
  }
  if ((uint64_t)(lim - p) < (uint64_t)*non_shared + *vlen) return nullptr;
  return p;
}

__global__ void k_table_index_count(const JobDev* jobs) {  // may follow the upload
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  const uint32_t t = blockIdx.x;
  if (t >= J.n_tables) return;
  const TableDesc T = J.tables[t];
  if (T.cached) {  // read from its decoded form: pseudo blocks of kDecRunBlock entries
    if (threadIdx.x == 0) {
      J.tbl_nblocks[t] = (uint32_t)((J.dec_runs[t].n + kDecRunBlock - 1) / kDecRunBlock);
      J.tbl_unit[t] = 0;
    }
    return;
  }
  const uint8_t* base = J.in + T.off;
  __shared__ uint64_t s_ioff, s_isize;
  __shared__ uint32_t s_nr, s_ok;
  __shared__ uint32_t s_part[32], s_other[32];
  if (threadIdx.x == 0) {
    uint64_t io = 0, is = 0;
    bool ok = parse_footer(base, T.size, &io, &is);
    uint32_t nr = 0;
    if (ok) {
      nr = ld_le32(base + io + is - 4);
      if ((uint64_t)nr * 4 + 4 > is) ok = false;
    }
    if (!ok) set_error(J.ctr, kErrBadFooter, t);
    s_ioff = io;
    s_isize = is;
    s_nr = nr;
    s_ok = ok;
  }
  __syncthreads();
  if (!s_ok) {
    if (threadIdx.x == 0) {
      J.tbl_nblocks[t] = 0;
      J.tbl_unit[t] = 0;
    }
    return;
  }
  const uint8_t* ra = base + s_ioff + s_isize - 4 - 4ull * s_nr;
  uint32_t sum = 0, other = 0;  // entries; restart runs of other than one entry
  for (uint32_t r = threadIdx.x; r < s_nr; r += blockDim.x) {
    const uint32_t c = ld_le32(ra + 4ull * r) & 0xff;
    sum += c;
    other += c != 1;
  }
  sum = warp_sum(sum);
  other = warp_sum(other);
  if ((threadIdx.x & 31) == 0) {
    s_part[threadIdx.x >> 5] = sum;
    s_other[threadIdx.x >> 5] = other;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t s = 0, o = 0;
    for (uint32_t w = 0; w < (blockDim.x + 31) / 32; w++) s += s_part[w], o += s_other[w];
    J.tbl_nblocks[t] = s;
    J.tbl_unit[t] = o == 0;
  }
}

// Data block handles from the index blocks.  An index block whose restart
// runs each hold one entry (the table builder writes index blocks with a
// restart interval of 1) is cut into kIdxSplit parts, one CTA each, every
// thread parsing its own entries; any other is parsed by one CTA, the
// entries' places from a block-wide scan of the run counts.
constexpr uint32_t kIdxSplit = 16;

__global__ void k_table_index_entries(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  const uint32_t t = blockIdx.x / kIdxSplit, part = blockIdx.x % kIdxSplit;
  if (t >= J.n_tables) return;
  const TableDesc T = J.tables[t];
  const bool unit = J.tbl_unit[t] != 0;
  if (part != 0 && (T.cached || !unit)) return;
  // the blocks of the tables before this one; kept for the kernels after (the
  // total by the last table's CTA)
  __shared__ unsigned long long s_base;
  if (threadIdx.x == 0) s_base = 0;
  __syncthreads();
  uint32_t before = 0;
  for (uint32_t x = threadIdx.x; x < t; x += blockDim.x) before += J.tbl_nblocks[x];
  if (before) atomicAdd(&s_base, (unsigned long long)before);
  __syncthreads();
  const uint64_t out_base = s_base, out_end = out_base + J.tbl_nblocks[t];
  if (part == 0 && threadIdx.x == 0) {
    J.tbl_block_base[t] = out_base;
    if (t + 1 == J.n_tables) {
      J.tbl_block_base[t + 1] = out_end;
      J.ctr->n_blocks_in = out_end;
    }
  }
  if (T.cached) {
    for (uint64_t o = out_base + threadIdx.x; o < out_end && o < J.cap_blocks_in; o += blockDim.x) {
      J.blk_off[o] = ((uint64_t)t << 32) | ((o - out_base) * kDecRunBlock);
      J.blk_size[o] = kPseudoBlock;
      J.blk_run[o] = T.run;
    }
    return;
  }
  const uint8_t* base = J.in + T.off;
  uint64_t io, is;
  if (!parse_footer(base, T.size, &io, &is)) return;  // error already recorded
  const uint32_t nr = ld_le32(base + io + is - 4);
  if ((uint64_t)nr * 4 + 4 > is) return;
  const uint8_t* idx = base + io;
  const uint64_t ra_off = is - 4 - 4ull * nr;
  const uint8_t* ra = idx + ra_off;
  if (unit) {
    const uint32_t r0 = (uint32_t)((uint64_t)nr * part / kIdxSplit);
    const uint32_t r1 = (uint32_t)((uint64_t)nr * (part + 1) / kIdxSplit);
    for (uint32_t r = r0 + threadIdx.x; r < r1; r += blockDim.x) {
      const uint64_t start = ld_le32(ra + 4ull * r) >> 8;
      const uint64_t end = (r + 1 < nr) ? (ld_le32(ra + 4ull * (r + 1)) >> 8) : ra_off;
      bool ok = start <= end && end <= ra_off;
      const uint8_t* p = idx + start;
      const uint8_t* lim = idx + end;
      uint32_t sh, ns, vl;
      const uint8_t* q = ok ? entry_header(p, lim, &sh, &ns, &vl) : nullptr;
      uint64_t b_off = 0, b_size = 0;
      const uint8_t* h = nullptr;
      if (q) {
        q += ns;
        h = get_varint64(q, q + vl, &b_off);
        if (h) h = get_varint64(h, q + vl, &b_size);
      }
      const uint64_t o = out_base + r;
      ok = h && b_off <= T.size && b_size + kTrailer <= T.size - b_off && o < out_end &&
           o < J.cap_blocks_in && q + vl == lim;
      if (ok) {
        J.blk_off[o] = T.off + b_off;
        J.blk_size[o] = (uint32_t)b_size;
        J.blk_run[o] = T.run;
      } else {
        set_error(J.ctr, kErrBadIndex, t);
      }
    }
    return;
  }
  __shared__ uint32_t s_warp[32];
  __shared__ uint32_t s_carry;
  if (threadIdx.x == 0) s_carry = 0;
  __syncthreads();
  for (uint32_t base_r = 0; base_r < nr; base_r += blockDim.x) {
    const uint32_t r = base_r + threadIdx.x;
    uint32_t w = r < nr ? ld_le32(ra + 4ull * r) : 0;
    uint32_t cnt = w & 0xff;
    // block-wide exclusive scan of cnt
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    uint32_t tot;
    uint32_t ex = warp_excl(cnt, &tot);
    if (lane == 0) s_warp[wid] = tot;
    __syncthreads();
    uint32_t before = s_carry;
    for (int k = 0; k < wid; k++) before += s_warp[k];
    uint32_t all = 0;
    for (int k = 0; k < (int)((blockDim.x + 31) / 32); k++) all += s_warp[k];
    ex += before;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += all;
    if (r < nr) {
      uint64_t start = w >> 8;
      uint64_t end = (r + 1 < nr) ? (ld_le32(ra + 4ull * (r + 1)) >> 8) : ra_off;
      bool ok = start <= end && end <= ra_off;
      const uint8_t* p = idx + start;
      const uint8_t* lim = idx + end;
      for (uint32_t k = 0; ok && k < cnt; k++) {
        uint32_t sh, ns, vl;
        const uint8_t* q = entry_header(p, lim, &sh, &ns, &vl);
        if (!q) {
          ok = false;
          break;
        }
        q += ns;
        uint64_t b_off, b_size;
        const uint8_t* h = q;
        if (!(h = get_varint64(h, q + vl, &b_off)) || !(h = get_varint64(h, q + vl, &b_size))) {
          ok = false;
          break;
        }
        if (b_off > T.size || b_size + kTrailer > T.size - b_off) {
          ok = false;
          break;
        }
        const uint64_t o = out_base + ex + k;
        if (o >= out_end || o >= J.cap_blocks_in) {
          ok = false;
          break;
        }
        J.blk_off[o] = T.off + b_off;
        J.blk_size[o] = (uint32_t)b_size;
        J.blk_run[o] = T.run;
        p = q + vl;
      }
      if (ok && p != lim) ok = false;
      if (!ok) set_error(J.ctr, kErrBadIndex, t);
    }
    __syncthreads();
  }
}

// A pseudo block: entries [*j0, *j1) of the decoded run of table *t.
__device__ __forceinline__ const DecRun& pseudo_block(const JobDev& J, uint64_t b, uint32_t* t,
                                                      uint64_t* j0, uint64_t* j1) {
  const uint64_t o = J.blk_off[b];
  *t = (uint32_t)(o >> 32);
  const DecRun& R = J.dec_runs[*t];
  *j0 = o & 0xffffffffull;
  *j1 = min(R.n, *j0 + kDecRunBlock);
  return R;
}

// Walks the entries of one restart run without writing them: counts key bytes
// and validates every header against the run's bounds.
__device__ __forceinline__ bool walk_run(const uint8_t* p, const uint8_t* lim, uint32_t cnt,
                                         uint64_t* kbytes, uint32_t* maxk, bool* short_key) {
  uint32_t prev = 0;
  uint64_t kb = 0;
  for (uint32_t k = 0; k < cnt; k++) {
    uint32_t sh, ns, vl;
    const uint8_t* q = entry_header(p, lim, &sh, &ns, &vl);
    if (!q) return false;
    if ((k == 0 && sh != 0) || sh > prev) return false;
    uint32_t kl = sh + ns;
    if (kl < 8) *short_key = true;
    kb += kl;
    *maxk = max(*maxk, kl);
    prev = kl;
    p = q + ns + vl;
  }
  *kbytes = kb;
  return p == lim;
}

struct BlockView {
  const uint8_t* p;
  uint64_t ra;  // offset of the restart array (end of entries)
  uint32_t nr;
  bool ok;
};

// View of data block b whose bytes are at `base` (a shared-memory stage or
// the block in global memory).
__device__ __forceinline__ BlockView block_view(const JobDev& J, uint64_t b, const uint8_t* base) {
  BlockView v;
  v.p = base;
  const uint32_t size = J.blk_size[b];
  v.ok = size >= 4;
  v.nr = v.ok ? ld_le32(v.p + size - 4) : 0;
  if (v.ok && (uint64_t)v.nr * 4 + 4 > size) v.ok = false;
  v.ra = v.ok ? size - 4 - 4ull * v.nr : 0;
  return v;
}

__device__ __forceinline__ void run_bounds(const BlockView& v, uint32_t r, uint64_t* start,
                                           uint64_t* end, uint32_t* cnt) {
  const uint32_t w = ld_le32(v.p + v.ra + 4ull * r);
  *cnt = w & 0xff;
  *start = w >> 8;
  *end = (r + 1 < v.nr) ? (ld_le32(v.p + v.ra + 4ull * (r + 1)) >> 8) : v.ra;
}

// Per-warp shared memory of the counting walk (k_block_count), and the key
// buffers of the decode.
constexpr uint32_t kDecWarps = 4;
constexpr uint32_t kDecStage = 8448;    // data block bytes + 16-byte phase
constexpr uint32_t kDecKeyBuf = 4096 + 32;  // a round's keys + phase
constexpr uint32_t kDecLastKey = 256;   // longest key the decode's buffers carry
struct DecWarpSmem {
  uint8_t stage[kDecStage];
};

// Copies data block b into this warp's stage at the block's own 16-byte phase
// with 16-byte loads; returns the staged pointer, or nullptr if it is too big.
__device__ __forceinline__ const uint8_t* stage_block(const JobDev& J, uint64_t b, uint8_t* stage,
                                                      uint32_t lane) {
  const uint8_t* src = J.in + J.blk_off[b];
  const uint32_t size = J.blk_size[b];
  const uintptr_t a = reinterpret_cast<uintptr_t>(src);
  const uint32_t phase = (uint32_t)(a & 15);
  if (size + phase + 16 > kDecStage) return nullptr;
  const uintptr_t base = a - phase;
  const uint32_t nch = (phase + size + 15) >> 4;
  const uintptr_t lo = reinterpret_cast<uintptr_t>(J.in), hi = reinterpret_cast<uintptr_t>(J.in_end);
  for (uint32_t c = lane; c < nch; c += 32) {
    const uintptr_t q = base + 16ull * c;
    if (q >= lo && q + 16 <= hi) {
      cp_async16(stage + 16 * c, reinterpret_cast<const void*>(q));
    } else {
      uint32_t w[4] = {0, 0, 0, 0};
      for (int i = 0; i < 16; i++) {
        const uintptr_t x = q + i;
        if (x >= a && x < a + size) w[i >> 2] |= (uint32_t)(*reinterpret_cast<const uint8_t*>(x)) << (8 * (i & 3));
      }
      *reinterpret_cast<uint4*>(stage + 16 * c) = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
  cp_async_wait_all();
  __syncwarp();
  return stage + phase;
}

__device__ void block_count_one(const JobDev& J, uint64_t b, uint32_t lane, const uint8_t* base) {
  BlockView v = block_view(J, b, base);
  uint64_t ent = 0, kb = 0;
  uint32_t maxk = 0;
  bool ok = v.ok, short_key = false;
  for (uint32_t r = lane; ok && r < v.nr; r += 32) {
    uint64_t s, e;
    uint32_t cnt;
    run_bounds(v, r, &s, &e, &cnt);
    if (s > e || e > v.ra) {
      ok = false;
      break;
    }
    uint64_t rk = 0;
    if (!walk_run(v.p + s, v.p + e, cnt, &rk, &maxk, &short_key)) {
      ok = false;
      break;
    }
    ent += cnt;
    kb += rk;
  }
  const bool all_ok = __all_sync(0xffffffffu, ok);
  const bool any_short = __any_sync(0xffffffffu, short_key);
  ent = warp_sum(ent);
  kb = warp_sum(kb);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) maxk = max(maxk, __shfl_xor_sync(0xffffffffu, maxk, o));
  if (lane == 0) {
    if (!all_ok) set_error(J.ctr, kErrBadBlock, (uint32_t)b);
    else if (any_short) set_error(J.ctr, kErrShortKey, (uint32_t)b);
    J.blk_nent[b] = all_ok ? (uint32_t)ent : 0;
    if (all_ok) atomicAdd((unsigned long long*)&J.ctr->key_bytes_in, (unsigned long long)kb);
    atomicMax(&J.ctr->max_klen, maxk);
  }
}

__global__ void __launch_bounds__(kDecWarps * 32) k_block_count(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  extern __shared__ __align__(16) uint8_t dec_smem[];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  DecWarpSmem& W = reinterpret_cast<DecWarpSmem*>(dec_smem)[warp];
  // after a footer or index error some block handles were never written
  if (J.ctr->error) return;
  const uint64_t nblk = min(J.ctr->n_blocks_in, J.cap_blocks_in);
  for (uint64_t b = (uint64_t)blockIdx.x * kDecWarps + warp; b < nblk;
       b += (uint64_t)gridDim.x * kDecWarps) {
    if (J.blk_size[b] == kPseudoBlock) {
      uint32_t t;
      uint64_t j0, j1;
      const DecRun& R = pseudo_block(J, b, &t, &j0, &j1);
      uint32_t mk = 0;
      for (uint64_t j = j0 + lane; j < j1; j += 32) mk = max(mk, (uint32_t)(R.kcum[j + 1] - R.kcum[j]));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) mk = max(mk, __shfl_xor_sync(0xffffffffu, mk, o));
      if (lane == 0) {
        J.blk_nent[b] = (uint32_t)(j1 - j0);
        atomicAdd((unsigned long long*)&J.ctr->key_bytes_in, (unsigned long long)(R.kcum[j1] - R.kcum[j0]));
        atomicMax(&J.ctr->max_klen, mk);
      }
      continue;
    }
    const uint8_t* st = stage_block(J, b, W.stage, lane);
    block_count_one(J, b, lane, st ? st : J.in + J.blk_off[b]);
    __syncwarp();
  }
}

// Entries per data block from its restart array alone (the LUDA restart word
// holds the entry count of its run): one thread per block.  The run byte
// ranges are checked here; the entries themselves when they are decoded.
__device__ __forceinline__ void block_restarts(const JobDev& J, uint32_t cta, uint32_t ctas) {
  const uint64_t nblk = min(J.ctr->n_blocks_in, J.cap_blocks_in);
  for (uint64_t b = (uint64_t)cta * blockDim.x + threadIdx.x; b < nblk;
       b += (uint64_t)ctas * blockDim.x) {
    const uint32_t size = J.blk_size[b];
    if (size == kPseudoBlock) {
      uint32_t t;
      uint64_t j0, j1;
      pseudo_block(J, b, &t, &j0, &j1);
      J.blk_nent[b] = (uint32_t)(j1 - j0);
      continue;
    }
    const uint8_t* p = J.in + J.blk_off[b];
    bool ok = size >= 4;
    const uint32_t nr = ok ? ld_le32(p + size - 4) : 0;
    if (ok && (uint64_t)nr * 4 + 4 > size) ok = false;
    const uint64_t ra = ok ? size - 4 - 4ull * nr : 0;
    uint64_t ent = 0, prev_end = 0;
    for (uint32_t r = 0; ok && r < nr; r++) {
      const uint32_t w = ld_le32(p + ra + 4ull * r);
      const uint64_t s0 = w >> 8;
      const uint64_t e0 = (r + 1 < nr) ? (ld_le32(p + ra + 4ull * (r + 1)) >> 8) : ra;
      if (s0 > e0 || e0 > ra || s0 < prev_end) ok = false;
      prev_end = e0;
      ent += w & 0xff;
    }
    if (!ok) set_error(J.ctr, kErrBadBlock, (uint32_t)b);
    J.blk_nent[b] = ok ? (uint32_t)ent : 0;
  }
}

__global__ void k_block_restarts(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  if (J.ctr->error) return;  // after a footer or index error some handles are unset
  block_restarts(J, blockIdx.x, gridDim.x);
}

// Input block checksums, for jobs that ask for them: the check ReadBlock
// makes when ReadOptions::verify_checksums is set (table/format.cc:86-95; the
// reference build has it switched off with `&& 0`, and LevelDB sets it for a
// compaction's inputs from Options::paranoid_checks, db/version_set.cc:1239):
// the fixed32 after the type byte must be Mask(crc32c(contents + type)).  One
// warp per data block; runs before the blocks are parsed, so that a damaged
// block reports the checksum rather than whatever its bytes break.
//
// Row CRC (lc_device.cuh): each lane loads up to four 16-byte chunks of the
// block ahead of their CRC steps.  10 MiB in 4 KiB blocks on B200: 23.0 us
// with one byte run per lane (a table lookup and a byte load per byte), 12.2
// us so.
__global__ void __launch_bounds__(256) k_verify_blocks(const JobDev* __restrict__ jobs) {
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  __shared__ uint32_t s_h5[kCrcH5Words];
  __shared__ uint32_t s_xinv[kCrcXinvSmem];
  __shared__ uint32_t s_tab8[256];
  __shared__ uint32_t s_skip;
  if (threadIdx.x == 0) s_skip = (!J.verify_checksums || J.ctr->error) ? 1u : 0u;
  __syncthreads();
  if (s_skip) return;
  for (uint32_t i = threadIdx.x; i < kCrcH5Words; i += blockDim.x) s_h5[i] = J.crc_h5[i];
  for (uint32_t i = threadIdx.x; i < kCrcXinvN; i += blockDim.x) s_xinv[xinv_slot(i)] = J.crc_xinv[i];
  for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) s_tab8[i] = J.crc_byte[i];
  __syncthreads();
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  const uint64_t nblk = min(J.ctr->n_blocks_in, J.cap_blocks_in);
  for (uint64_t b = (uint64_t)blockIdx.x * nw + warp; b < nblk; b += (uint64_t)gridDim.x * nw) {
    // the index parse checked that the block and its 5-byte trailer lie in the table
    const uint32_t size = J.blk_size[b];
    if (size == kPseudoBlock) continue;  // a decoded form: no block bytes to check
    const uint8_t* p = J.in + J.blk_off[b];
    const uint32_t m0 = (uint32_t)(reinterpret_cast<uintptr_t>(p) & 15);
    const uint32_t m1 = m0 + size + 1;  // the message: contents and the stored type byte
    const uint8_t* g = p - m0;
    uint32_t u = 0, last = 0xffffffffu;
    constexpr uint32_t kAhead = 4;
    for (uint32_t q0 = 16 * lane; q0 < m1; q0 += kAhead * kCrcRowBytes) {
      uint4 v[kAhead];
#pragma unroll
      for (uint32_t i = 0; i < kAhead; i++) {
        const uint32_t q = q0 + i * kCrcRowBytes;
        if (q >= m1) break;
        if (g + q >= J.in) {  // a block is followed by its CRC and a footer: the chunk's end is inside
          v[i] = __ldg(reinterpret_cast<const uint4*>(g + q));
        } else {  // the first chunk starts before the input's memory: its own bytes only
          uint32_t w[4] = {0, 0, 0, 0};
          for (uint32_t k = m0; k < 16 && k < m1; k++) w[k >> 2] |= (uint32_t)g[k] << (8 * (k & 3));
          v[i] = make_uint4(w[0], w[1], w[2], w[3]);
        }
      }
#pragma unroll
      for (uint32_t i = 0; i < kAhead; i++) {
        const uint32_t q = q0 + i * kCrcRowBytes;
        if (q >= m1) break;
        u = crc_chunk_step(s_h5, u, q, m0, m1, v[i].x, v[i].y, v[i].z, v[i].w);
        last = q;
      }
    }
    const uint32_t crc = crc_rows_finish(s_xinv, s_tab8, u, last, m1);
    if (lane == 0 && crc != ld_le32(p + size + 1)) set_error(J.ctr, kErrChecksum, (uint32_t)b);
  }
}

// The parse's last kernel.  Entries of merge child r start at the first block
// of its first table: one thread per table, the first table of each run writes
// the run's start.  Then the counters, final now, to the host (res_ctr: mapped
// pinned memory).
__device__ __forceinline__ void parse_done(const JobDev& J, uint32_t cta, uint32_t ctas) {
  const bool bad = J.ctr->error != 0;  // the job fails; keep every read in bounds
  for (uint32_t t = cta * blockDim.x + threadIdx.x; t < J.n_tables;
       t += ctas * blockDim.x) {
    const uint32_t run = J.tables[t].run;
    if (t == 0 || J.tables[t - 1].run != run)
      J.run_entry_begin_w[run] =
          bad ? 0 : J.blk_ent_base[min(J.tbl_block_base[t], J.cap_blocks_in)];
  }
  if (cta != 0) return;
  if (threadIdx.x == 0) J.run_entry_begin_w[J.n_runs] = J.ctr->n_entries_in;
  if (J.res_ctr)
    for (uint32_t i = threadIdx.x; i < sizeof(Counters) / 8; i += blockDim.x)
      reinterpret_cast<uint64_t*>(J.res_ctr)[i] = reinterpret_cast<const uint64_t*>(J.ctr)[i];
}

__global__ void k_parse_done(const JobDev* jobs) {  // may follow the upload
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  parse_done(J, blockIdx.x, gridDim.x);
}

// A small job's last three steps of the parse in one cluster: an 800-entry job
// 192 -> 186 us against a launch each, jobs of 8 to 66 MiB the same
// within noise.
constexpr uint64_t kParseBlocks = 8192;
__global__ void __launch_bounds__(kPartThreads, 1) k_parse_blocks(const JobDev* __restrict__ jobs) {
  pdl_begin();
  __shared__ JobDev s_job;
  copy_job(jobs + blockIdx.y, &s_job);
  __syncthreads();
  const JobDev& J = s_job;
  const uint32_t cta = blockIdx.x, ctas = gridDim.x;  // the grid's x is one cluster
  const volatile uint32_t* const error = &J.ctr->error;
  if (!*error) block_restarts(J, cta, ctas);  // (an error of the kernels before)
  cluster_sync();
  if (!*error) tile_scan<kScanBlkEnt, kPartThreads, true>(J, cta, ctas);  // the same in all CTAs
  cluster_sync();
  if (cta == 0) parse_done(J, 0, 1);
}

// ---------------------------------------------------------------------------
// Decode of the data blocks into the entry arrays, in two passes.
//
// Pass 1 (k_decode_walk): one warp per group of dec_group consecutive data
// blocks (as many as have 32 restart runs, at most 32).  The group's restart runs,
// one lane per run in rounds of 32, walk their entry headers straight from
// global memory (the lines a run's headers lie in are read once, through L1)
// with the checks of the counting walk, and write one 16-byte record per
// entry -- where its key delta lies, its shared and key lengths, its value's
// length and place -- and its key length.  A pseudo block (a decoded run,
// from the decoded form of an earlier output) is cut into runs of
// kDecRunSlice entries whose records come from that form.
//
// Pass 2 (k_decode_keys): one warp per unit of about dec_unit entries, cut
// at entries without a shared prefix (every restart has none).  A unit takes
// its part of the key arena with one atomic add (each key's slot is its length
// rounded up to a multiple of 8; where in the arena a unit lies does not
// matter; a scan of all lengths before this kernel cost 7-10 us of a small job
// and 2170 instead of 2064 us of a call on 64 MiB of 32-byte values).  Rounds
// of 32, one lane per entry.  A round whose keys have at most 32 bytes is decoded
// in registers: a lane loads its key delta at the key's own byte positions,
// and the shared prefixes come by a scan over the lanes (a key is a head of
// the key before it and its own bytes; two such steps compose into one).
// Rounds with longer keys go through the warp's key buffer in shared memory:
// key deltas at the keys' places, then the shared prefixes in entry order, then
// 16-byte stores to the arena; keys beyond that buffer are built in the arena.
// The round's last key carries into the next round.
//
// Pass 1 is bound by its chain of loads (a header names the next one's place):
// of 2M entries of 32-byte keys its warps wait for one 46 cycles per instruction
// issued, DRAM at 34% of its rate.  Pass 2 by L1 (69% of its rate; the lanes read
// a line each) and the latency of its loads, issue at 38%, DRAM at 48%.  8M such
// entries on B200: pass 1 193 us, pass 2 235 us with the filters' hashes (452 with
// every round through the buffer, whose bytewise steps met 8-way bank conflicts
// at this key length).
constexpr uint32_t kDecGroupMax = 32;   // data blocks per warp in pass 1
constexpr uint32_t kDecRunSlice = 16;   // pseudo-block entries per lane
constexpr uint32_t kDecPseudo = 0xffffu;  // shared length of a pseudo entry's record

// Record of entry e: x key delta offset in `in` (a pseudo entry: its block),
// y shared length | key length << 16, z value length, w value offset in `in`.
__device__ __forceinline__ uint4 dec_record(uint32_t src, uint32_t sh, uint32_t kl, uint32_t vl,
                                            uint32_t voff) {
  return make_uint4(src, sh | (kl << 16), vl, voff);
}

__global__ void __launch_bounds__(256, 5) k_decode_walk(const JobDev* jobs) {  // may follow the upload
  pdl_begin();
  __shared__ JobDev s_job;
  {  // the surplus CTAs of a small job leave at once
    const JobDev& G = jobs[blockIdx.y];
    if (blockIdx.x * 8ull * G.dec_group >= G.ctr->n_blocks_in) return;
  }
  copy_job(jobs + blockIdx.y, &s_job);
  __syncthreads();
  const JobDev& J = s_job;
  __shared__ uint32_t s_rb[8][kDecGroupMax + 1];  // per warp: first run of each block of its group
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (J.ctr->error) return;
  const uint64_t nblk = min(J.ctr->n_blocks_in, J.cap_blocks_in);
  const uint32_t G = J.dec_group;
  const uint64_t ngrp = (nblk + G - 1) / G;
  for (uint64_t g = (uint64_t)blockIdx.x * 8 + warp; g < ngrp; g += (uint64_t)gridDim.x * 8) {
    const uint64_t g0 = g * G;
    // runs of the lane's block (a pseudo block: slices of its entries)
    uint32_t nr = 0;
    if (lane < G && g0 + lane < nblk) {
      const uint64_t b = g0 + lane;
      const uint32_t size = J.blk_size[b];
      if (size == kPseudoBlock) {
        nr = (J.blk_nent[b] + kDecRunSlice - 1) / kDecRunSlice;
      } else {
        nr = ld_le32(J.in + J.blk_off[b] + size - 4);  // checked by k_block_restarts
      }
    }
    uint32_t nrt;
    s_rb[warp][lane] = warp_excl<uint32_t>(nr, &nrt);
    if (lane == 0) s_rb[warp][kDecGroupMax] = nrt;
    __syncwarp();
    const uint32_t pad = J.key_pad;
    uint64_t kb = 0, kr = 0;
    uint32_t maxk = 0;
    bool bad = false, short_key = false, long_key = false;
    for (uint32_t q0 = 0; q0 < nrt; q0 += 32) {
      const uint32_t q = q0 + lane;
      if (q >= nrt) continue;
      // the block of run q: the last with its first run at or before q
      uint32_t lo = 0, hi = G;
      while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (s_rb[warp][mid] <= q) lo = mid;
        else hi = mid;
      }
      const uint64_t b = g0 + lo;
      const uint32_t r = q - s_rb[warp][lo];
      const uint64_t ebase = J.blk_ent_base[b];
      const uint32_t size = J.blk_size[b];
      if (size == kPseudoBlock) {
        uint32_t t;
        uint64_t j0, j1;
        const DecRun& R = pseudo_block(J, b, &t, &j0, &j1);
        const TableDesc& T = J.tables[t];
        const uint64_t ja = j0 + (uint64_t)r * kDecRunSlice, jz = min(j1, ja + kDecRunSlice);
        for (uint64_t j = ja; j < jz; j++) {
          const uint32_t kl = (uint32_t)(R.kcum[j + 1] - R.kcum[j]);
          const uint32_t vl = R.vlen[j], vp = R.vpos[j];
          if (kl < 8) short_key = true;
          if (kl > 0xffff) long_key = true;
          if ((uint64_t)vp + vl > T.size) bad = true;
          const uint64_t e = ebase + (j - j0);
          J.e_rec[e] = dec_record((uint32_t)b, kDecPseudo, kl, vl, (uint32_t)(T.off + vp));
          kb += kl;
          kr += (kl + pad) & ~pad;
          maxk = max(maxk, kl);
        }
        continue;
      }
      const uint8_t* p = J.in + J.blk_off[b];
      const uint32_t nrb = ld_le32(p + size - 4);
      const uint32_t ra = size - 4 - 4 * nrb;
      const uint32_t w = ld_le32(p + ra + 4 * r);
      const uint32_t cnt = w & 0xff;
      const uint32_t s = w >> 8, e = (r + 1 < nrb) ? (ld_le32(p + ra + 4 * (r + 1)) >> 8) : ra;
      uint32_t before = 0;  // entries of the block's earlier runs
      for (uint32_t x = 0; x < r; x++) before += ld_le32(p + ra + 4 * x) & 0xff;
      const uint8_t* qp = p + s;
      const uint8_t* lim = p + e;  // run ranges checked by k_block_restarts
      const uint32_t boff = (uint32_t)J.blk_off[b];
      // the record array in a register: the stores below cannot then make the
      // compiler reload it from the job descriptor
      uint4* const rec = J.e_rec + ebase + before;
      uint32_t prev = 0;
      for (uint32_t k = 0; k < cnt; k++) {
        uint32_t sh, ns, vl;
        const uint8_t* d = entry_header(qp, lim, &sh, &ns, &vl);
        if (!d || (k == 0 && sh != 0) || sh > prev) {
          bad = true;
          break;
        }
        const uint32_t kl = sh + ns;
        if (kl < 8) short_key = true;
        if (kl > 0xffff || sh >= kDecPseudo) long_key = true;
        const uint32_t doff = boff + (uint32_t)(d - p);
        rec[k] = dec_record(doff, sh, kl, vl, doff + ns);
        kb += kl;
        kr += (kl + pad) & ~pad;
        maxk = max(maxk, kl);
        prev = kl;
        qp = d + ns + vl;
      }
      if (!bad && qp != lim) bad = true;
    }
    const bool any_bad = __any_sync(0xffffffffu, bad);
    const bool any_short = __any_sync(0xffffffffu, short_key);
    const bool any_long = __any_sync(0xffffffffu, long_key);
    kb = warp_sum(kb);
    kr = warp_sum(kr);
    maxk = __reduce_max_sync(0xffffffffu, maxk);
    if (lane == 0) {
      atomicMax(&J.ctr->max_klen, maxk);
      atomicAdd((unsigned long long*)&J.ctr->key_total, (unsigned long long)kb);
      atomicAdd((unsigned long long*)&J.ctr->key_round, (unsigned long long)kr);
      if (any_bad) set_error(J.ctr, kErrBadBlock, (uint32_t)g0);
      else if (any_short) set_error(J.ctr, kErrShortKey, (uint32_t)g0);
      else if (any_long) set_error(J.ctr, kErrLimit, 4);
      else if (J.reserve_keys && maxk > J.max_key_len) set_error(J.ctr, kErrRetryExact, (uint32_t)g0);
    }
    __syncwarp();
  }
}

struct DecKeysSmem {
  uint8_t buf[kDecKeyBuf];    // the round's keys, at the arena's 16-byte phase
  __align__(16) uint8_t last[kDecLastKey];  // the previous round's last key
};

// The key bytes a record points at: the key delta in `in`, or a pseudo
// entry's whole key in its decoded run.
__device__ __forceinline__ const uint8_t* dec_delta(const JobDev& J, uint64_t e, uint4 rec) {
  if ((rec.y & 0xffff) == kDecPseudo) {
    uint32_t t;
    uint64_t j0, j1;
    const uint64_t b = rec.x;
    const DecRun& R = pseudo_block(J, b, &t, &j0, &j1);
    return R.keys + R.kcum[j0 + (e - J.blk_ent_base[b])];
  }
  return J.in + rec.x;
}

// First entry at or after e (below n) without a shared prefix, else n.
__device__ __forceinline__ uint64_t dec_unit_start(const JobDev& J, uint64_t e, uint64_t n,
                                                   uint32_t lane) {
  for (; e < n; e += 32) {
    const uint64_t x = e + lane;
    const uint32_t sh = x < n ? (J.e_rec[x].y & 0xffff) : 1u;
    const unsigned m = __ballot_sync(0xffffffffu, x < n && (sh == 0 || sh == kDecPseudo));
    if (m) return e + (__ffs(m) - 1);
  }
  return n;
}

constexpr uint32_t kDecRegWords = 8;  // key words a lane decodes in registers

// Bytes of key word q below byte s of the key.
__device__ __forceinline__ uint32_t dec_below(uint32_t s, uint32_t q) {
  const int32_t n = (int32_t)s - 4 * (int32_t)q;
  return n >= 4 ? 0xffffffffu : (n <= 0 ? 0u : (1u << (8 * n)) - 1u);
}

// The shared prefixes of a round's keys w (at most 4 N bytes each, s of them
// the lane's own): key l takes its bytes below s from the key o before it, s
// becoming the least shared length over those o keys, until s is 0 or reaches
// before the round (`last`).
template <uint32_t N>
__device__ __forceinline__ void dec_share(uint32_t (&w)[kDecRegWords], uint32_t s, const uint8_t* last,
                                          uint32_t lane) {
#pragma unroll
  for (uint32_t k = 0; k < 5; k++) {
    const uint32_t o = 1u << k;
    const uint32_t ps = __shfl_up_sync(0xffffffffu, s, o);
    const uint32_t take = lane >= o ? s : 0u;
#pragma unroll
    for (uint32_t q = 0; q < N; q++) {
      const uint32_t pw = __shfl_up_sync(0xffffffffu, w[q], o), m = dec_below(take, q);
      w[q] = (w[q] & ~m) | (pw & m);
    }
    if (lane >= o) s = min(s, ps);
  }
  if (!s) return;
#pragma unroll
  for (uint32_t q = 0; q < N; q++) {
    const uint32_t m = dec_below(s, q);
    w[q] = (w[q] & ~m) | (*reinterpret_cast<const uint32_t*>(last + 4 * q) & m);
  }
}

// A round of keys of at most 4 kDecRegWords bytes, lane l's key delta at src
// (key bytes [sh, kl)); `last`: the key before the round's first (read only
// when that one shares a prefix), then the round's last key.
__device__ __forceinline__ void decode_round_regs(const JobDev& J, uint8_t* last, uint64_t e,
                                                  bool valid, uint4 rec, const uint8_t* src,
                                                  uint32_t koff, uint32_t kl, uint32_t sh,
                                                  uint32_t cnt, uint32_t lane) {
  uint32_t w[kDecRegWords];
#pragma unroll
  for (uint32_t q = 0; q < kDecRegWords; q++) w[q] = 0u;
  if (valid) {
    const uintptr_t s = reinterpret_cast<uintptr_t>(src), s0 = s - sh;  // s0: the key's byte 0
    const uintptr_t b0 = s0 & ~uintptr_t(3);
    const uint32_t fsh = 8 * (uint32_t)(s0 & 3);
    const uint32_t first = (uint32_t)(s - b0), end = first + (kl - sh);  // needed bytes from b0
    uint32_t x[kDecRegWords + 1];
#pragma unroll
    for (uint32_t i = 0; i <= kDecRegWords; i++)
      x[i] = (4 * i + 4 > first && 4 * i < end) ? __ldg(reinterpret_cast<const uint32_t*>(b0) + i) : 0u;
#pragma unroll
    for (uint32_t q = 0; q < kDecRegWords; q++) w[q] = __funnelshift_r(x[q], x[q + 1], fsh);
  }
  const uint32_t s = valid ? sh : 0;
  const uint32_t smax = __reduce_max_sync(0xffffffffu, s);
  if (smax > 16) dec_share<kDecRegWords>(w, s, last, lane);
  else if (smax > 4) dec_share<4>(w, s, last, lane);
  else if (smax) dec_share<1>(w, s, last, lane);
  __syncwarp();  // the previous key has been read
  if (lane == cnt - 1) {
#pragma unroll
    for (uint32_t q = 0; q < kDecRegWords; q += 4)
      *reinterpret_cast<uint4*>(last + 4 * q) = make_uint4(w[q], w[q + 1], w[q + 2], w[q + 3]);
  }
  if (!valid) return;
  uint64_t* d = reinterpret_cast<uint64_t*>(J.keys + koff);  // the slot: 8-byte aligned
#pragma unroll
  for (uint32_t q = 0; q < kDecRegWords; q += 2)
    if (4 * q < kl) d[q / 2] = (uint64_t)w[q] | ((uint64_t)w[q + 1] << 32);
  const uint32_t u = kl - 8;  // user key bytes
  // the first 8 user-key bytes, big endian, zero padded
  uint64_t p = ((uint64_t)__byte_perm(w[0], 0, 0x0123) << 32) | __byte_perm(w[1], 0, 0x0123);
  if (u < 8) p = u ? p & (~0ull << (64 - 8 * u)) : 0;
  // the last 8 bytes
  const uint32_t t = u >> 2;  // words t.. of the key, moved down by t's bits
  uint32_t y[6], z[4];
#pragma unroll
  for (uint32_t q = 0; q < 6; q++) y[q] = (t & 4) ? (q + 4 < kDecRegWords ? w[(q + 4) & 7] : 0u) : w[q];
#pragma unroll
  for (uint32_t q = 0; q < 4; q++) z[q] = (t & 2) ? y[q + 2] : y[q];
  const uint32_t t0 = (t & 1) ? z[1] : z[0], t1 = (t & 1) ? z[2] : z[1], t2 = (t & 1) ? z[3] : z[2];
  const uint32_t ts = 8 * (u & 3);
  const uint64_t tag = (uint64_t)__funnelshift_r(t0, t1, ts) | ((uint64_t)__funnelshift_r(t1, t2, ts) << 32);
  J.e_pfx[e] = p;
  J.e_tag[e] = tag;
  if (J.bits_per_key > 0) {  // bloom_hash
    const uint32_t m = 0xc6a4a793u;
    uint32_t h = 0xbc9f1d34u ^ (u * m);
#pragma unroll
    for (uint32_t q = 0; q + 2 < kDecRegWords; q++) {
      if (4 * q + 4 <= u) {
        h += w[q];
        h *= m;
        h ^= h >> 16;
      } else if (4 * q < u) {
        h += w[q] & ((1u << (8 * (u - 4 * q))) - 1u);
        h *= m;
        h ^= h >> 24;
      }
    }
    J.e_hash[e] = h;
  }
}

__global__ void __launch_bounds__(256, 4) k_decode_keys(const JobDev* __restrict__ jobs) {
  pdl_begin();
  __shared__ JobDev s_job;
  {
    const JobDev& G = jobs[blockIdx.y];
    if (blockIdx.x * 8ull * G.dec_unit >= G.ctr->n_entries_in) return;
  }
  copy_job(jobs + blockIdx.y, &s_job);
  __syncthreads();
  const JobDev& J = s_job;
  __shared__ __align__(16) DecKeysSmem s_w[8];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  DecKeysSmem& W = s_w[warp];
  if (J.ctr->error) return;
  if (J.ctr->key_round > J.cap_key_bytes) {  // the arena does not hold the keys
    set_error(J.ctr, J.reserve_keys ? kErrRetryExact : kErrArenaOverflow, 5);
    return;
  }
  const uint32_t pad = J.key_pad;
  const uint64_t n = J.ctr->n_entries_in;
  const uint64_t unit = J.dec_unit, nunits = (n + unit - 1) / unit;
  for (uint64_t u = (uint64_t)blockIdx.x * 8 + warp; u < nunits; u += (uint64_t)gridDim.x * 8) {
    const uint64_t e0 = u == 0 ? 0 : dec_unit_start(J, u * unit, n, lane);
    const uint64_t e1 = dec_unit_start(J, (u + 1) * unit, n, lane);
    uint64_t room = 0;  // the unit's part of the arena
    for (uint64_t e = e0 + lane; e < e1; e += 32) room += ((J.e_rec[e].y >> 16) + pad) & ~pad;
    room = warp_sum(room);
    uint64_t kpos = 0;  // arena offset of the round's first key
    if (lane == 0) kpos = atomicAdd((unsigned long long*)&J.ctr->key_cursor, (unsigned long long)room);
    kpos = __shfl_sync(0xffffffffu, kpos, 0);
    bool last_staged = true;  // the previous key is in W.last (not needed at a unit start)
    uint64_t last_at = 0;     // else its arena offset
    for (uint64_t r0 = e0; r0 < e1; r0 += 32) {
      const uint64_t e = r0 + lane;
      const bool valid = e < e1;
      const uint32_t cnt = (uint32_t)min(32ull, (unsigned long long)(e1 - r0));
      const uint4 rec = valid ? J.e_rec[e] : make_uint4(0, 0, 0, 0);
      const uint32_t kl = rec.y >> 16;
      const uint32_t sh = (rec.y & 0xffff) == kDecPseudo ? 0 : (rec.y & 0xffff);
      const uint8_t* src = valid ? dec_delta(J, e, rec) : nullptr;
      const uint32_t mk = __reduce_max_sync(0xffffffffu, kl);
      const uint32_t sh0 = __shfl_sync(0xffffffffu, sh, 0);
      uint32_t tot;
      const uint32_t ko = warp_excl<uint32_t>((kl + pad) & ~pad, &tot);  // offset within the round
      if (valid) {
        J.e_loc[e] = make_uint4((uint32_t)(kpos + ko), kl, rec.w, rec.z);
      }
      if (mk <= 4 * kDecRegWords && pad && (sh0 == 0 || last_staged)) {
        decode_round_regs(J, W.last, e, valid, rec, src, (uint32_t)(kpos + ko), kl, sh, cnt, lane);
        last_staged = true;
        kpos += tot;
        __syncwarp();
        continue;
      }
      uint8_t* gdst = J.keys + kpos;
      const uint32_t kph = (uint32_t)(reinterpret_cast<uintptr_t>(gdst) & 15);
      const uint32_t lkl = __shfl_sync(0xffffffffu, kl, cnt - 1);
      const uint32_t lko = __shfl_sync(0xffffffffu, ko, cnt - 1);
      if (tot + kph + 16 <= kDecKeyBuf && mk <= kDecLastKey && (sh0 == 0 || last_staged)) {
        uint8_t* kb = W.buf + kph;
        // deltas, every lane at once
        if (valid) {
          const uint32_t dl = kl - sh;
          for (uint32_t t = 0; t < dl; t += 32) copy_small_w(kb + ko + sh + t, src + t, min(32u, dl - t));
        }
        __syncwarp();
        // shared prefixes.  Within the round, an entry z without a shared
        // prefix holds its whole key as its delta; for the entries after it
        // (up to the next such entry), the bytes below the least shared
        // length since z are z's bytes -- every entry in between shares them.
        // Before the round's first such entry the same holds with the
        // previous round's last key.  Each other prefix byte is the own
        // (delta) byte of the nearest earlier entry whose shared length lies
        // below it (the entries in between share it), found by a walk back
        // that ends at the entry with that least shared length.
        const unsigned zmask = __ballot_sync(0xffffffffu, valid && sh == 0);
        const unsigned zbelow = zmask & (0xffffffffu >> (31 - lane));
        const int z = zbelow ? 31 - __clz(zbelow) : -1;
        const uint32_t koz = __shfl_sync(0xffffffffu, ko, z < 0 ? 0 : z);
        // segmented running minimum of the shared lengths since z (z excluded)
        uint32_t m = (valid && sh != 0) ? sh : 0xffffffffu;
        bool seg = valid && sh == 0;  // this lane's range reaches a segment head
#pragma unroll
        for (uint32_t o = 1; o < 32; o <<= 1) {
          const uint32_t y = __shfl_up_sync(0xffffffffu, m, o);
          const bool ys = __shfl_up_sync(0xffffffffu, seg, o);
          if (lane >= o && !seg) {
            m = min(m, y);
            seg = ys;
          }
        }
        if (!valid || sh == 0) m = 0;
        if (valid && m) {
          const uint8_t* from = z >= 0 ? kb + koz : W.last;
          for (uint32_t t = 0; t < m; t++) kb[ko + t] = from[t];
        }
        uint32_t lim = valid ? sh : 0;
        for (uint32_t d = 1; d < 32 && __any_sync(0xffffffffu, lim > m); d++) {
          const uint32_t j = lane >= d ? lane - d : lane;
          const uint32_t shj = __shfl_sync(0xffffffffu, sh, j);
          const uint32_t koj = __shfl_sync(0xffffffffu, ko, j);
          if (lim > m && lane >= d && shj < lim) {
            const uint32_t a = max(shj, m);
            for (uint32_t t = a; t < lim; t++) kb[ko + t] = kb[koj + t];
            lim = a;
          }
        }
        __syncwarp();
        // the round's last key for the next round; keys out: head bytes,
        // 16-byte body, tail bytes
        for (uint32_t t = lane; t < lkl; t += 32) W.last[t] = kb[lko + t];
        last_staged = true;
        const uint32_t head = (16 - kph) & 15;
        const uint32_t h = head < tot ? head : tot;
        if (lane < h) gdst[lane] = kb[lane];
        const uint32_t body = (tot - h) & ~15u;
        const uint4* sv = reinterpret_cast<const uint4*>(kb + h);
        uint4* dv = reinterpret_cast<uint4*>(gdst + h);
        for (uint32_t c = lane; c < body / 16; c += 32) dv[c] = sv[c];
        const uint32_t t0 = h + body;
        if (t0 + lane < tot) gdst[t0 + lane] = kb[t0 + lane];
        if (valid) {
          J.e_pfx[e] = user_prefix(kb + ko, kl);
          J.e_tag[e] = ld_le64(kb + ko + kl - 8);
          if (J.bits_per_key > 0) J.e_hash[e] = bloom_hash(kb + ko, kl);
        }
      } else {
        // long keys: built in the arena, one key at a time, the lanes over
        // its bytes
        for (uint32_t i = 0; i < cnt; i++) {
          const uint32_t shi = __shfl_sync(0xffffffffu, sh, i);
          const uint32_t kli = __shfl_sync(0xffffffffu, kl, i);
          const uint32_t koi = __shfl_sync(0xffffffffu, ko, i);
          const uint32_t kpi = __shfl_sync(0xffffffffu, ko, (i + 31) & 31);
          const uint8_t* srci = reinterpret_cast<const uint8_t*>(__shfl_sync(
              0xffffffffu, (unsigned long long)reinterpret_cast<uintptr_t>(src), i));
          const uint8_t* prev = i ? gdst + kpi : (last_staged ? W.last : J.keys + last_at);
          uint8_t* d = gdst + koi;
          for (uint32_t t = lane; t < kli; t += 32) d[t] = t < shi ? prev[t] : srci[t - shi];
          __syncwarp();
        }
        last_at = kpos + lko;
        last_staged = lkl <= kDecLastKey;
        if (last_staged)
          for (uint32_t t = lane; t < lkl; t += 32) W.last[t] = gdst[lko + t];
        if (valid) {
          J.e_pfx[e] = user_prefix(gdst + ko, kl);
          J.e_tag[e] = ld_le64(gdst + ko + kl - 8);
          if (J.bits_per_key > 0) J.e_hash[e] = bloom_hash(gdst + ko, kl);
        }
      }
      kpos += tot;
      __syncwarp();
    }
  }
}

__global__ void k_entries_from_offsets(const JobDev* jobs) {  // may follow the upload
  pdl_begin();
  const JobDev& J = jobs[blockIdx.y];
  const uint64_t n = J.cap_entries;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t ko = J.src_koffs[i], kl = J.src_koffs[i + 1] - ko;
    if (kl < 8) {
      set_error(J.ctr, kErrShortKey, (uint32_t)i);
      continue;
    }
    J.k_koff[i] = (uint32_t)ko;
    J.k_klen[i] = (uint32_t)kl;
    J.k_voff[i] = (uint32_t)J.src_voffs[i];
    J.k_vlen[i] = (uint32_t)(J.src_voffs[i + 1] - J.src_voffs[i]);
    if (J.bits_per_key > 0) J.k_hash[i] = bloom_hash(J.keys + ko, (uint32_t)kl);
  }
}

}  // namespace

void launch_table_index_count(const Batch& bt, cudaStream_t st) {
  launch(k_table_index_count, dim3(bt.max_tables, bt.B), 1024, 0, st, bt.d);
}
void launch_table_index_entries(const Batch& bt, cudaStream_t st) {
  launch(k_table_index_entries, dim3(bt.max_tables * kIdxSplit, bt.B), 256, 0, st, bt.d);
}

static void dec_smem_attr(const void* fn) {
  cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                       (int)(kDecWarps * sizeof(DecWarpSmem)));
}

static unsigned dec_ctas(const Batch& bt) {
  // grid-stride over the device-side block count: 3 CTAs per SM x 8 waves in
  // total, shared out among the jobs of the batch
  return grid_x(bt.max_blocks_in, kDecWarps, bt.per_job(148 * 3 * 8));
}

void decode_kernel_attributes() { dec_smem_attr((const void*)k_block_count); }

void launch_block_count(const Batch& bt, cudaStream_t st) {
  launch(k_block_count, dim3(dec_ctas(bt), bt.B), kDecWarps * 32, kDecWarps * sizeof(DecWarpSmem), st, bt.d);
}
void launch_parse_blocks(const Batch& bt, cudaStream_t st) {
  const unsigned ctas = part_ctas(bt.max_blocks_in);
  if (bt.max_blocks_in <= kParseBlocks && (uint64_t)ctas * bt.jobs_of_largest <= 148) {
    launch_clusters(ctas, k_parse_blocks, dim3(ctas, bt.B), kPartThreads, 0, st, bt.d);
    return;
  }
  launch(k_block_restarts, dim3(grid_x(bt.max_blocks_in, 256, bt.per_job(148 * 8)), bt.B), 256, 0, st, bt.d);
  scan_batch(kScanBlkEnt, bt, bt.max_blocks_in, st);
  launch_parse_done(bt, st);
}
void launch_verify_blocks(const Batch& bt, cudaStream_t st) {
  if (!bt.any_verify) return;
  launch(k_verify_blocks, dim3(grid_x(bt.max_blocks_in, 8, bt.per_job(148 * 4)), bt.B), 256, 0, st, bt.d);
}
void launch_parse_done(const Batch& bt, cudaStream_t st) {
  launch(k_parse_done, dim3((bt.max_tables + 127) / 128 + 1, bt.B), 128, 0, st, bt.d);
}
void launch_block_decode(const Batch& bt, cudaStream_t st) {
  // pass 1: one warp per group of blocks; pass 2: one warp per unit of
  // entries, as many CTAs as the SMs hold at once (5 and 4 each); 8 warps per
  // CTA
  launch(k_decode_walk, dim3(grid_x(bt.max_dec_groups, 8, bt.per_job(148 * 5)), bt.B), 256, 0, st, bt.d);
  launch(k_decode_keys, dim3(grid_x(bt.max_dec_units, 8, bt.per_job(148 * 4)), bt.B), 256, 0, st, bt.d);
}
void launch_entries_from_offsets(const Batch& bt, cudaStream_t st) {
  launch(k_entries_from_offsets, dim3(grid_x(bt.max_entries, 256, 148 * 8), bt.B), 256, 0, st, bt.d);
}

}  // namespace lc
