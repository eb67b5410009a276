// Masked CRC32C of one large buffer, split over many CTAs.
//
// The buffer's 16-byte chunks (of the 16-byte grid it lies on) are put in
// rows of 32, the last row ending with the last chunk; a CTA takes a run of
// consecutive rows, warp w of its 16 every 16th of them, lane l a row's chunk
// l, and carries the interleaved raw register of lc_device.cuh (crc_h5: 26
// conflict-free table lookups per chunk) with tables for that distance.  Rows
// and chunks before the run or the buffer count as zeros, which a zero
// register ignores.  At the end each thread's register is moved back by its
// place (one product), the CTA's xor of them is moved over the rows after the
// CTA's run (the powers of the shift's bits multiplied across one warp's
// lanes) and xored into one accumulator, to which CTA 0 adds the initial
// register carried over the message.  The CTA that finishes last (an atomic
// ticket, no waiting) moves the sum back over the last chunk's bytes past the
// buffer and stores crc32c::Mask(crc) (util/crc32c.h:29-32), what LevelDB
// writes in a block trailer.
//
// Bound by the L1/shared and integer pipes (26 lookups, 70 integer
// instructions and one 16-byte load per chunk and lane); four rows' loads are
// in flight while the four before them are looked up.  64 MiB in device
// memory on B200: the bytewise form this replaces took 290 us (0.23 TB/s, one
// 256-byte run per thread, uncoalesced byte loads); warps with runs of their
// own 42 us (seven serial products per warp at the end); this form
// 32 us (2.1 TB/s).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "lc_device.cuh"

namespace lc {

constexpr uint32_t kCrcChunkThreads = 512;
constexpr uint32_t kCrcChunkWarps = kCrcChunkThreads / 32;
// scratch words: [0] the accumulator, [1] the ticket counter; both zero at
// launch, and zero again when the kernel has finished
constexpr uint32_t kCrcScratchWords = 2;

// Powers of x mod P in the reflected representation (bit 31 = x^0).
constexpr uint32_t crcc_mul_c(uint32_t a, uint32_t b) {
  uint32_t p = 0;
  for (int i = 0; i < 32; i++) {
    if (a & 0x80000000u) p ^= b;
    a <<= 1;
    b = (b & 1) ? (b >> 1) ^ kCrcPoly : (b >> 1);
  }
  return p;
}
constexpr uint32_t crcc_back_bit(uint32_t c) {  // c x^-1
  return (c >> 31) ? ((c ^ kCrcPoly) << 1) | 1u : c << 1;
}
struct CrcPowers {
  uint32_t up[64];                  // x^(8 2^k)
  uint32_t back[kCrcChunkThreads];  // x^(-8 (512 w + 16 l)), thread 32 w + l
  uint32_t tail[16];                // x^(-8 t)
  uint32_t row;  // register left by the last bit of a chunk and the run of zeros after it
};
constexpr CrcPowers crcc_powers() {
  CrcPowers t{};
  uint32_t c = 0x80000000u;
  for (int i = 0; i < 8; i++) c = (c & 1) ? (c >> 1) ^ kCrcPoly : (c >> 1);
  for (int k = 0; k < 64; k++) {
    t.up[k] = c;
    c = crcc_mul_c(c, c);
  }
  c = 0x80000000u;
  for (int i = 0; i < 16; i++) {
    t.tail[i] = c;
    for (int k = 0; k < 8; k++) c = crcc_back_bit(c);
  }
  const uint32_t back16 = c;
  c = 0x80000000u;
  for (uint32_t i = 0; i < kCrcChunkThreads; i++) {
    t.back[i] = c;
    c = crcc_mul_c(c, back16);
  }
  // x^32 (the register's width), then the zero bytes up to the warp's next row
  t.row = t.up[2];
  for (uint32_t n = kCrcChunkWarps * kCrcRowBytes - 16, k = 0; n; n >>= 1, k++)
    if (n & 1) t.row = crcc_mul_c(t.row, t.up[k]);
  return t;
}
static __device__ const CrcPowers g_crc_pow = crcc_powers();

// x^(8m) mod P, the same in every lane: lane k's factor is that of the bits k
// and k + 32 of m, multiplied across the warp.
__device__ __forceinline__ uint32_t crcc_xpow_warp(uint64_t m) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t f = ((m >> lane) & 1) ? g_crc_pow.up[lane] : 0x80000000u;
  if ((m >> (lane + 32)) & 1) f = gf2_mulmod(f, g_crc_pow.up[lane + 32]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) f = gf2_mulmod(f, __shfl_xor_sync(0xffffffffu, f, o));
  return f;
}

// The row tables (crc_h5's layout) into shared memory, computed by the CTA:
// bit i of a chunk followed by zero bytes up to the warp's next row leaves the
// register x^(127 - i) times that of the chunk's last bit.
__device__ __forceinline__ void crcc_row_tables(uint32_t* h5, uint32_t* basis) {
  if (threadIdx.x < 128) {
    uint32_t c = g_crc_pow.row;
    for (uint32_t k = threadIdx.x; k < 127; k++) c = (c & 1) ? (c >> 1) ^ kCrcPoly : (c >> 1);
    basis[threadIdx.x] = c;
  }
  __syncthreads();
  for (uint32_t x = threadIdx.x; x < kCrcH5Words; x += blockDim.x) {
    const uint32_t b0 = kCrcFieldBits * (x / kCrcFieldEntries), v = x % kCrcFieldEntries;
    uint32_t r = 0;
#pragma unroll
    for (uint32_t k = 0; k < kCrcFieldBits; k++)
      if (((v >> k) & 1) && b0 + k < 128) r ^= basis[b0 + k];
    h5[x] = r;
  }
  __syncthreads();
}

// Chunk c of the grid that starts at g, zero outside the buffer [a, a + n);
// only the buffer's own bytes are read.
__device__ __forceinline__ uint4 crcc_edge_chunk(const uint8_t* g, const uint8_t* a, uint64_t n,
                                                 int64_t c) {
  uint32_t w[4] = {0, 0, 0, 0};
  for (uint32_t i = 0; i < 16; i++) {
    const int64_t q = 16 * c + i - (a - g);  // byte of the buffer
    if (q >= 0 && (uint64_t)q < n) w[i >> 2] |= (uint32_t)a[q] << (8 * (i & 3));
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// Body shared by every kernel that computes a chunked CRC: grid x any number
// of CTAs of kCrcChunkThreads.
__device__ __forceinline__ void crc32c_chunks_body(const uint8_t* data, uint64_t n,
                                                   uint32_t* scratch, uint32_t* out) {
  __shared__ uint32_t s_h5[kCrcH5Words];
  __shared__ uint32_t s_basis[128];
  __shared__ uint32_t s_acc;
  if (threadIdx.x == 0) s_acc = 0;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t ph = (uint32_t)(reinterpret_cast<uintptr_t>(data) & 15);
  const uint8_t* g = data - ph;
  const int64_t C = n ? (int64_t)((ph + n + 15) / 16) : 0;
  const uint32_t over = (uint32_t)(16 * C - (n ? ph + n : 0));  // the last chunk's bytes past the buffer
  const int64_t R = (C + 31) / 32;
  const int64_t S = (R + gridDim.x - 1) / gridDim.x;
  const int64_t r0 = min(R, (int64_t)blockIdx.x * S), r1 = min(R, r0 + S);
  constexpr int kW = (int)kCrcChunkWarps, kAhead = 4;  // the warp's rows loaded at once
  // the warp's rows: r, r + kW, ..., the last in the run's last kW rows
  int64_t r = r1 - kW * ((r1 - r0 + kW - 1) / kW) + warp;
  const auto load = [&](int64_t row) -> uint4 {
    const int64_t c = C - 32 * (R - row) + lane;
    if (row < r0 || row >= r1 || c < 0) return make_uint4(0, 0, 0, 0);
    if (c == 0 || c + 1 == C) return crcc_edge_chunk(g, data, n, c);
    return __ldcs(reinterpret_cast<const uint4*>(g) + c);
  };
  uint4 v[kAhead];
#pragma unroll
  for (int k = 0; k < kAhead; k++) v[k] = load(r + kW * k);
  crcc_row_tables(s_h5, s_basis);
  uint32_t u = 0;
  for (; r < r1; r += kW * kAhead) {
    uint4 w[kAhead];
    const int64_t nx = r + kW * kAhead, last = nx + kW * (kAhead - 1);
    if (C - 32 * (R - last) + 32 < C && last < r1) {  // rows within the run, the last chunk not among them
      const uint4* p = reinterpret_cast<const uint4*>(g) + (C - 32 * (R - nx) + lane);
#pragma unroll
      for (int k = 0; k < kAhead; k++) w[k] = __ldcs(p + 32 * kW * k);
    } else {
#pragma unroll
      for (int k = 0; k < kAhead; k++) w[k] = load(nx + kW * k);
    }
#pragma unroll
    for (int k = 0; k < kAhead; k++)
      if (r + kW * k < r1) u = crc_h5(s_h5, v[k].x ^ u, v[k].y, v[k].z, v[k].w);
#pragma unroll
    for (int k = 0; k < kAhead; k++) v[k] = w[k];
  }
  u = gf2_mulmod(u, g_crc_pow.back[threadIdx.x]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) u ^= __shfl_xor_sync(0xffffffffu, u, o);
  if (lane == 0) atomicXor(&s_acc, u);
  __syncthreads();
  if (warp == 0) {
    const uint32_t x = gf2_mulmod(s_acc, crcc_xpow_warp((uint64_t)(R - r1) * kCrcRowBytes));
    if (lane == 0) atomicXor(scratch, x);
  } else if (warp == 1 && blockIdx.x == 0) {
    const uint32_t x = gf2_mulmod(0xffffffffu, crcc_xpow_warp(n + over));
    if (lane == 0) atomicXor(scratch, x);
  }
  __threadfence();
  __syncthreads();
  if (threadIdx.x != 0) return;
  if (atomicAdd(scratch + 1, 1u) != gridDim.x - 1) return;
  __threadfence();
  const uint32_t full = gf2_mulmod(atomicExch(scratch, 0u), g_crc_pow.tail[over]) ^ 0xffffffffu;
  scratch[1] = 0;
  *out = ((full >> 15) | (full << 17)) + 0xa282ead8u;
}

// CTAs for a buffer of n bytes: two rows per warp (a CTA's fixed cost, the
// tables and the products, is that of a dozen rows, but small buffers are bound
// by their latency), at most two CTAs (32 warps) on each of the 148 SMs.
inline uint32_t crc32c_chunk_ctas(uint64_t n) {
  const uint64_t rows = n / kCrcRowBytes + 2;
  const uint64_t c = (rows + 2 * kCrcChunkWarps - 1) / (2 * kCrcChunkWarps);
  return (uint32_t)(c < 296 ? c : 296);
}

}  // namespace lc
