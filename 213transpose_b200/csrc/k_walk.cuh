// Segment cycles over rows with a remainder: the movers of the ragged band
// plans.
//
// A slice is rows of `pitch` bytes that hold q segments of seg_bytes each and
// a few elements more (the remainder, saved and written by the tail kernels
// below).  Segment s lies at (s / q) * pitch + (s % q) * seg_bytes, so the
// segments of different rows start at different bytes of a 16-byte block
// unless the pitch is a multiple of 16.
//
// k_seg_walk moves the segments along the chunks of a cycle table (k_cycles.cuh
// describes chunks and carries).  A CTA walks one piece of one chunk: a ring
// of kWalkRing pieces is loaded ahead by 16-byte asynchronous copies of the
// blocks that cover a piece, and a piece is written to the next position, in
// 16-byte words where both have the same offset in a block, else in 4-byte
// words (funnel-shifted for 1- and 2-byte elements at odd distances).  One
// barrier per step orders the landing of a position's old value before its
// overwriting and the last read of a buffer before its reload.
//
// Bound by memory, in practice by the loads in flight (three pieces of 16 KB
// a CTA, three CTAs an SM) and by the step barrier where segments are short.
// The whole ragged transpose of fp32 (1000003, 37, 1), 148 MB, takes 136 us
// against 587 us of the gathers through a scratch copy that it replaced; fp64
// (101, 100003, 2) 160 against 318, bf16 (31424, 3160, 1) 204 against 1091.
#pragma once

#include "common.cuh"
#include "functors.cuh"
#include "k_cycles.cuh"
#include "tma.cuh"

namespace t213 {

constexpr int kWalkThreads = 256;
constexpr int kWalkRing = 4;
constexpr int kWalkPiece = 16 * 1024;

struct SegRows {
  FastDiv<uint32_t> q;
  int64_t pitch, seg_bytes;
  __device__ __forceinline__ int64_t at(uint32_t s) const {
    const uint32_t r = q.div(s);
    return (int64_t)r * pitch + (int64_t)(s - r * q.get()) * seg_bytes;
  }
};

template <int N>
__device__ __forceinline__ void walk_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void walk_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

// Copies pb bytes at g into buf, at their offset in a 16-byte block.
__device__ __forceinline__ void walk_load(unsigned char *buf, const char *g, uint32_t pb) {
  const uint32_t sh = (uint32_t)(uintptr_t)g & 15u;
  const char *ga = g - sh;
  const uint32_t nc = (sh + pb + 15) >> 4;
  for (uint32_t c = threadIdx.x; c < nc; c += kWalkThreads) cp_async<16>(buf + c * 16, ga + (size_t)c * 16);
}

// Writes the pb bytes at buf + sh to d.
template <int EB>
__device__ __forceinline__ void walk_store(char *d, const unsigned char *buf, uint32_t sh, uint32_t pb) {
  const uint32_t dd = (uint32_t)(uintptr_t)d;
  if (((dd ^ sh) & 15u) == 0) {
    const uint32_t head = min((16u - sh) & 15u, pb), body = (pb - head) >> 4;
    const unsigned char *b = buf + sh + head;
    char *o = d + head;
#pragma unroll 4
    for (uint32_t c = threadIdx.x; c < body; c += kWalkThreads)
      *reinterpret_cast<uint4 *>(o + (size_t)c * 16) = *reinterpret_cast<const uint4 *>(b + c * 16);
    // the ends, in elements (of at most 16 bytes) or single bytes
    constexpr uint32_t T = EB < 16 ? EB : 16;
    const uint32_t tail = pb - head - body * 16;
    for (uint32_t x = threadIdx.x * T; x < head + tail; x += kWalkThreads * T) {
      const uint32_t off = x < head ? x : x + body * 16;
      using E = typename ElemT<EB>::type;
      *reinterpret_cast<E *>(d + off) = *reinterpret_cast<const E *>(buf + sh + off);
    }
    return;
  }
  if constexpr (EB >= 8) {
    using E = typename ElemT<8>::type;
    const uint32_t nw = pb >> 3;
#pragma unroll 4
    for (uint32_t w = threadIdx.x; w < nw; w += kWalkThreads)
      *reinterpret_cast<E *>(d + (size_t)w * 8) = *reinterpret_cast<const E *>(buf + sh + w * 8);
  } else if constexpr (EB == 4) {
    const uint32_t nw = pb >> 2;
#pragma unroll 4
    for (uint32_t w = threadIdx.x; w < nw; w += kWalkThreads)
      *reinterpret_cast<uint32_t *>(d + (size_t)w * 4) = *reinterpret_cast<const uint32_t *>(buf + sh + w * 4);
  } else {
    using E = typename ElemT<EB>::type;
    const uint32_t head = min((4u - (dd & 3u)) & 3u, pb), body = (pb - head) >> 2;
    const uint32_t so = sh + head, f = (so & 3u) * 8;
    const uint32_t *b = reinterpret_cast<const uint32_t *>(buf + (so & ~3u));
    char *o = d + head;
#pragma unroll 4
    for (uint32_t w = threadIdx.x; w < body; w += kWalkThreads)
      *reinterpret_cast<uint32_t *>(o + (size_t)w * 4) = __funnelshift_r(b[w], b[w + 1], f);
    const uint32_t tail = pb - head - body * 4;
    for (uint32_t x = threadIdx.x * EB; x < head + tail; x += kWalkThreads * EB) {
      const uint32_t off = x < head ? x : x + body * 4;
      *reinterpret_cast<E *>(d + off) = *reinterpret_cast<const E *>(buf + sh + off);
    }
  }
}

template <int EB, typename P>
__global__ void __launch_bounds__(kWalkThreads)
    k_seg_walk(char *__restrict__ data, int64_t slice_bytes, int64_t d3, SegRows rows, uint32_t piece_bytes,
               uint32_t pieces, const Chunk *__restrict__ chunks, int64_t n_chunks, const char *__restrict__ carry,
               int64_t carry_pitch, P dst) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const uint32_t bufsz = (piece_bytes + 15) / 16 * 16 + 32;  // the covering blocks, a word more for the funnel
  const int64_t per_chunk = (int64_t)pieces * d3;
  const int64_t items = n_chunks * per_chunk;
  for (int64_t it = blockIdx.x; it < items; it += gridDim.x) {
    const int64_t c = it / per_chunk;
    const int64_t rest = it - c * per_chunk;
    const int64_t k = rest / pieces;
    const int64_t off = (rest - k * pieces) * piece_bytes;
    const Chunk ch = chunks[c];
    const uint32_t pb = (uint32_t)min((int64_t)piece_bytes, rows.seg_bytes - off);
    char *base = data + k * slice_bytes + off;
    const int64_t L = ch.len;
    // position 0 comes from its carry slot or from its place
    uint32_t xl = (uint32_t)ch.start;  // newest position loaded
    const char *g0 = ch.carry >= 0 ? carry + (ch.carry * d3 + k) * carry_pitch + off : base + rows.at(xl);
    __syncthreads();  // the previous item's buffers have been read
    walk_load(smem_raw, g0, pb);
    walk_commit();
    // kWalkRing - 2 positions ahead; an empty group keeps the count where
    // there is nothing left to load
#pragma unroll
    for (int j = 1; j <= kWalkRing - 2; j++) {
      if (j < L) {
        xl = dst(xl);
        walk_load(smem_raw + (size_t)j * bufsz, base + rows.at(xl), pb);
      }
      walk_commit();
    }
    uint32_t sh = (uint32_t)(uintptr_t)g0 & 15u;  // offset of the piece in the previous buffer
    uint32_t x = (uint32_t)ch.start;
    int bp = 0;  // buffer of position s - 1
    for (int64_t s = 1; s <= L; s++) {
      // positions up to s have landed (groups up to s + kWalkRing - 3 exist)
      walk_wait<kWalkRing - 3>();
      __syncthreads();
      x = dst(x);
      char *d = base + rows.at(x);
      walk_store<EB>(d, smem_raw + (size_t)bp * bufsz, sh, pb);
      // buffer of position s - 2, read in the previous step by every thread
      int bl = bp - 1;
      if (bl < 0) bl += kWalkRing;
      if (s + kWalkRing - 2 < L) {
        xl = dst(xl);
        walk_load(smem_raw + (size_t)bl * bufsz, base + rows.at(xl), pb);
      }
      walk_commit();
      sh = (uint32_t)(uintptr_t)d & 15u;
      if (++bp == kWalkRing) bp = 0;
    }
    walk_wait<0>();
  }
}

// Saves the old value of every split chunk's start.  EB bytes a thread.
template <int EB>
__global__ void __launch_bounds__(kWalkThreads)
    k_walk_carry(const char *__restrict__ data, int64_t slice_bytes, int64_t d3, SegRows rows,
                 const CarryItem *__restrict__ items, int64_t n_items, char *__restrict__ carry,
                 int64_t carry_pitch) {
  using E = typename ElemT<EB>::type;
  const int64_t per = rows.seg_bytes / EB, blocks = (per + 4 * kWalkThreads - 1) / (4 * kWalkThreads);
  const int64_t total = n_items * d3 * blocks;
  for (int64_t t = blockIdx.x; t < total; t += gridDim.x) {
    const int64_t r = t / blocks, b = t - r * blocks;
    const int64_t ii = r / d3, k = r - ii * d3;
    const CarryItem ci = items[ii];
    const E *g = reinterpret_cast<const E *>(data + k * slice_bytes + rows.at((uint32_t)ci.pos));
    E *o = reinterpret_cast<E *>(carry + (ci.slot * d3 + k) * carry_pitch);
    E v[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int64_t w = b * 4 * kWalkThreads + q * kWalkThreads + threadIdx.x;
      if (w < per) v[q] = __ldcg(g + w);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const int64_t w = b * 4 * kWalkThreads + q * kWalkThreads + threadIdx.x;
      if (w < per) o[w] = v[q];
    }
  }
}

// The remainder of rows x cols elements per slice: element (i, j) at
// in + i * is + j * js goes to out + i * os + j * ot (strides in elements),
// j fastest over the threads.
template <int EB>
__global__ void __launch_bounds__(kWalkThreads)
    k_walk_tail(const char *__restrict__ in, int64_t in_slice, int64_t is, int64_t js, char *__restrict__ out,
                int64_t out_slice, int64_t os, int64_t ot, int64_t rows, int64_t cols, int64_t d3) {
  using E = typename ElemT<EB>::type;
  const int64_t per = rows * cols, total = per * d3;
  for (int64_t t = (int64_t)blockIdx.x * kWalkThreads + threadIdx.x; t < total; t += (int64_t)gridDim.x * kWalkThreads) {
    const int64_t k = t / per, e = t - k * per, i = e / cols, j = e - i * cols;
    reinterpret_cast<E *>(out + k * out_slice)[i * os + j * ot] =
        __ldcg(reinterpret_cast<const E *>(in + k * in_slice) + i * is + j * js);
  }
}

}  // namespace t213
