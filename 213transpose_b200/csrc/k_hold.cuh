// One-pass 213 transpose of slices that fit the shared memory of a team of
// CTAs: one CTA, a thread-block cluster (up to 16 CTAs), or up to the whole
// chip (slices of up to about 30 MB).
//
// A slice (m = d2 rows of n = d1 elements) is cut into TR x TC tiles of
// tm x tn elements.  Every CTA of the team loads its tiles into its own shared
// memory; one team barrier orders every load of the slice before any store;
// then every CTA writes its own tiles transposed.  A tile is read and written
// by the same CTA, so nothing is exchanged between CTAs but the barrier, and
// every element crosses memory once in each direction: one sweep, for any m
// and n, coprime ones included, against the two or three of the other plans.
//
// Bound by memory once the slices of a launch fill the chip; below that by
// one load latency, one barrier and one store latency.  Row pieces are read
// tn elements long and written tm elements long, so tiles are kept as square
// as the shared memory allows (pieces of 600-900 bytes for the largest
// slices); a launch runs two CTAs of 512 threads per SM with about 113 KB
// each, so one CTA's loads are in flight while the other writes.
//
// Forms: scalar (any pitch and base: the 16-byte blocks that cover a row piece
// come in, a few bytes of its neighbours among them that are never used;
// elements leave one by one, those of 1 and 2 bytes in 4-byte words), vector (2- and
// 4-byte elements on 16-byte pitches both ways: 16-byte copies into a
// swizzled tile, Q x Q register transposes, 16-byte stores), wide (elements
// of several 16-byte words, the rank-N permutations' merged leading axes).
#pragma once

#include "common.cuh"
#include "internal.h"
#include "tma.cuh"

namespace t213 {

constexpr int kHoldThreads = 512;
constexpr int kHoldSlots = 4096;  // barrier slots: one per stream, one per captured launch
constexpr int kHoldTeams = 20;    // grid teams of a launch (17 CTAs or more each)

// RAG_DST / RAG_SRC: scalar tiles of one band of a ragged band plan, whose
// output columns / source rows lie as the segments of rows with a remainder.
enum HoldForm { HOLD_SCALAR = 0, HOLD_VEC = 1, HOLD_WIDE = 2, HOLD_RAG_DST = 3, HOLD_RAG_SRC = 4 };

struct HoldArgs {
  int64_t d3, slice_bytes;
  uint32_t m, n;            // slice rows and columns (elements)
  uint32_t tm, tn, TC, T;   // tile sides, tiles per slice row, tiles per slice
  uint32_t ctas, teams, S;  // CTAs per team, teams, tiles per CTA (at most)
  uint32_t P, H, tile_bytes;  // shared-memory row pitch, region and tile size
  int32_t packed;             // narrow rows, one contiguous piece per tile
  int32_t mode, slot;
  int32_t lgs;  // log2 of the lanes that share an output column
  uint32_t we;       // wide form: 16-byte words per element
  FastDiv<uint32_t> wediv, tcdiv, rbdiv;
  // ragged bands: m x n is a band, nb bands per slice; segment s of a slice
  // (seg_bytes long, q to a row of rag_pitch bytes) at
  // (s / q) * rag_pitch + (s % q) * seg_bytes
  FastDiv<uint32_t> qdiv;
  uint32_t nb, seg_bytes;
  int64_t rag_pitch;
  __device__ __forceinline__ uint64_t seg_at(uint32_t s) const {
    const uint32_t r = qdiv.div(s);
    return (uint64_t)r * (uint64_t)rag_pitch + (uint64_t)(s - r * qdiv.get()) * seg_bytes;
  }
};

// ---- tiles -------------------------------------------------------------------
// Shared-memory layout of a scalar tile: a row piece lies in the 16-byte
// blocks that cover it, at its own offset in the first block.  The N = 4 / EB
// rows that share an output word (N = 1 from 4 bytes on) lie in N regions of
// H bytes; row i is the (i / N)-th of region i % N, at pitch P (an odd number
// of blocks) plus one block per 8 rows.  A column of odd-pitched 4-byte rows
// then falls into 32 different banks: 8 rows take the 8 block positions of a
// bank line, the offset rotates over the 4 words of a block from row to row,
// and the extra block separates rows 8 apart.  A packed tile (all columns of
// narrow rows) is one contiguous piece.
template <int EB, int FORM>
__device__ __forceinline__ uint32_t hold_row(const HoldArgs &a, uint32_t i, uint32_t lo, uint32_t pitch_lo,
                                             uint32_t s0) {
  constexpr uint32_t N = EB < 4 ? 4 / EB : 1;
  const uint32_t l = i / N, b = i % N;
  if constexpr (FORM == HOLD_RAG_SRC) {
    return b * a.H + l * a.P + (l >> 3) * 16 + ((lo + (uint32_t)a.seg_at(s0 + i)) & 15u);
  } else {
    if (a.packed) return (lo & 15u) + i * (a.n * EB);
    return b * a.H + l * a.P + (l >> 3) * 16 + ((lo + i * pitch_lo) & 15u);
  }
}

// `slice` is the slice, or the band's rows (RAG_DST), or the start of the
// slice that the band belongs to (RAG_SRC, with s0 the band's first segment).
template <int EB, int FORM>
__device__ __forceinline__ void hold_load(const char *slice, const HoldArgs &a, uint32_t r0, uint32_t c0,
                                          unsigned char *s, uint32_t s0) {
  uint32_t rows = min(a.tm, a.m - r0), cols = min(a.tn, a.n - c0);
  const uint32_t E = EB * (FORM == HOLD_WIDE ? a.we : 1);
  const uint32_t pitch = a.n * E;  // a slice is far below 4 GB
  const char *g0 = slice + (FORM == HOLD_RAG_SRC ? 0 : (size_t)r0 * pitch) + (size_t)c0 * E;
  if ((FORM == HOLD_SCALAR || FORM == HOLD_RAG_DST) && a.packed) {
    const uint32_t sh = (uint32_t)(uintptr_t)g0 & 15u;
    const char *g = g0 - sh;
    const uint32_t nc = (sh + rows * pitch + 15) >> 4;
#pragma unroll 4
    for (uint32_t c = threadIdx.x; c < nc; c += kHoldThreads) cp_async<16>(s + c * 16, g + c * 16);
    return;
  }
  // thread t takes blocks t, t + 512, ... of the tile's rows x nc blocks and
  // carries (row, block) along: no lane idles at a row's end
  const uint32_t nc = FORM == HOLD_VEC ? cols * EB / 16 : FORM == HOLD_WIDE ? cols * a.we : (cols * EB + 31 - EB) / 16;
  const uint32_t di = kHoldThreads / nc, dc = kHoldThreads - di * nc;
  uint32_t i = threadIdx.x / nc, c = threadIdx.x - i * nc;
#pragma unroll 4
  for (; i < rows;) {
    const char *g = g0 + (FORM == HOLD_RAG_SRC ? (size_t)a.seg_at(s0 + r0 + i) : (size_t)(i * pitch));
    if constexpr (FORM == HOLD_VEC) {
      constexpr uint32_t Q = 16 / EB;
      cp_async<16>(s + i * a.P + ((c ^ ((i / Q) & 7u)) << 4), g + c * 16);
    } else if constexpr (FORM == HOLD_WIDE) {
      cp_async<16>(s + i * a.P + c * 16, g + c * 16);
    } else {
      constexpr uint32_t N = EB < 4 ? 4 / EB : 1;
      const uint32_t sh = (uint32_t)(uintptr_t)g & 15u, l = i / N, b = i % N;
      // a piece that starts early in its first block may need one block less
      if (c * 16 < sh + cols * EB) cp_async<16>(s + b * a.H + l * a.P + (l >> 3) * 16 + c * 16, g - sh + c * 16);
    }
    i += di;
    c += dc;
    if (c >= nc) {
      c -= nc;
      i++;
    }
  }
}

// `slice` is where the columns go, `from` where the rows came from (hold_load's
// `slice`), s0 the band's first segment.
template <int EB, int FORM>
__device__ __forceinline__ void hold_store(char *slice, const char *from, const HoldArgs &a, uint32_t r0, uint32_t c0,
                                           const unsigned char *s, uint32_t s0) {
  using E = typename ElemT<EB>::type;
  const uint32_t rows = min(a.tm, a.m - r0), cols = min(a.tn, a.n - c0);
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if constexpr (FORM == HOLD_VEC) {
    // a warp takes 8 row blocks by 4 column chunks: its 8-lane phases read 8
    // different chunks of the swizzle, and it writes 4 x 128 bytes at a time
    constexpr uint32_t Q = 16 / EB;
    union V {
      uint4 v;
      E e[Q];
    };
    const uint32_t RB = rows / Q, CB = cols / Q;
    const uint32_t ra = lane & 7, ca = lane >> 3;
    const uint32_t ntr = (RB + 7) / 8, ntc = (CB + 3) / 4;
    const bool full = rows == a.tm;
    for (uint32_t t = warp; t < ntr * ntc; t += nw) {
      const uint32_t tc = full ? a.rbdiv.div(t) : t / ntr;
      const uint32_t rb = (t - tc * ntr) * 8 + ra, cb = tc * 4 + ca;
      if (rb >= RB || cb >= CB) continue;
      V in[Q];
      const unsigned char *p = s + (rb * Q) * a.P + ((cb ^ (rb & 7u)) << 4);
#pragma unroll
      for (uint32_t i = 0; i < Q; i++) in[i].v = *reinterpret_cast<const uint4 *>(p + i * a.P);
      char *g = slice + (size_t)(((c0 + cb * Q) * a.m + r0 + rb * Q) * EB);
#pragma unroll
      for (uint32_t j = 0; j < Q; j++) {
        V o;
#pragma unroll
        for (uint32_t i = 0; i < Q; i++) o.e[i] = in[i].e[j];
        *reinterpret_cast<uint4 *>(g + (size_t)(j * a.m * EB)) = o.v;
      }
    }
  } else if constexpr (FORM == HOLD_WIDE) {
    const uint32_t L = 1u << a.lgs, li = lane & (L - 1), sub = lane >> a.lgs;
    const uint32_t jstep = nw << (5 - a.lgs);
    const uint32_t total = rows * a.we;
    for (uint32_t j = (warp << (5 - a.lgs)) + sub; j < cols; j += jstep) {
      char *g = slice + (size_t)(((c0 + j) * a.m + r0) * a.we) * 16;
#pragma unroll 4
      for (uint32_t w = li; w < total; w += L) {
        const uint32_t i = a.wediv.div(w), q = w - i * a.we;
        *reinterpret_cast<uint4 *>(g + w * 16) =
            *reinterpret_cast<const uint4 *>(s + i * a.P + (j * a.we + q) * 16);
      }
    }
  } else {
    // A unit: the 32 lanes take L output words of a column (a word is N rows
    // of it) by 32 / L columns, U column steps one after the other: U reads
    // at fixed offsets, then U stores.  Steps are N columns apart, so that the
    // output rows of a unit start at the same byte of a 4-byte word.
    constexpr uint32_t N = EB < 4 ? 4 / EB : 1;
    constexpr uint32_t U = EB == 16 ? 4 : EB == 4 ? 16 : 8;
    const uint32_t L = 1u << a.lgs, G = 32u >> a.lgs, li = lane & (L - 1), sub = lane >> a.lgs;
    const uint32_t plo = a.n * EB;
    const uint32_t lo = (uint32_t)(uintptr_t)from + (FORM == HOLD_RAG_SRC ? c0 * EB : (r0 * a.n + c0) * EB);
    const uint32_t sr = s0 + r0;  // RAG_SRC: the segment of the tile's first row
    const uint32_t words = N == 1 ? rows : (rows + 2 * N - 2) / N;  // one more covers every offset
    const uint32_t nrb = (words + L - 1) >> a.lgs, ncg = (cols + U * G * N - 1) / (U * G * N) * N;
    const bool full = rows == a.tm;
    for (uint32_t u = warp; u < nrb * ncg; u += nw) {
      const uint32_t cg = full ? a.rbdiv.div(u) : u / nrb;
      const uint32_t w = ((u - cg * nrb) << a.lgs) + li;
      const uint32_t j0 = cg / N * (U * G * N) + cg % N * G + sub;
      if (w >= words || j0 >= cols) continue;
      const uint32_t o = ((c0 + j0) * a.m + r0) * EB;
      const uint32_t gs = G * N * a.m * EB;
      const uint32_t ps = G * N * EB;
      const uint32_t left = (cols - 1 - j0) / (G * N) + 1;  // column steps of this lane
      if constexpr (N == 1) {
        const unsigned char *p = s + hold_row<EB, FORM>(a, w, lo, plo, sr) + j0 * EB;
        E v[U];
        if constexpr (FORM == HOLD_RAG_DST) {
          char *g = slice + (size_t)((r0 + w) * EB);
          const uint32_t sj = s0 + c0 + j0;
#pragma unroll
          for (uint32_t q = 0; q < U; q++)
            if (q < left) v[q] = *reinterpret_cast<const E *>(p + q * ps);
#pragma unroll
          for (uint32_t q = 0; q < U; q++)
            if (q < left) *reinterpret_cast<E *>(g + a.seg_at(sj + q * G)) = v[q];
          continue;
        }
        char *g = slice + (size_t)(o + w * EB);
        if (left >= U) {
#pragma unroll
          for (uint32_t q = 0; q < U; q++) v[q] = *reinterpret_cast<const E *>(p + q * ps);
#pragma unroll
          for (uint32_t q = 0; q < U; q++, g += gs) *reinterpret_cast<E *>(g) = v[q];
        } else {
#pragma unroll
          for (uint32_t q = 0; q < U; q++)
            if (q < left) *reinterpret_cast<E *>(g + (size_t)(q * gs)) = *reinterpret_cast<const E *>(p + q * ps);
        }
      } else if constexpr (FORM == HOLD_RAG_DST) {
        // the offset of an output row is its own: column by column
        for (uint32_t q = 0; q < min(left, U); q++) {
          char *g = slice + a.seg_at(s0 + c0 + j0 + q * (G * N)) + (size_t)(r0 * EB);
          const uint32_t h = ((uint32_t)(uintptr_t)g & 3u) / EB;
          const int32_t e0 = (int32_t)(w * N) - (int32_t)h;
          uint32_t v = 0;
#pragma unroll
          for (uint32_t b = 0; b < N; b++)
            v |= (uint32_t) * reinterpret_cast<const E *>(
                     s + hold_row<EB, FORM>(a, min((uint32_t)max(e0 + (int32_t)b, 0), rows - 1), lo, plo, sr) +
                     j0 * EB + q * ps)
                 << (8 * EB * b);
          g += (int64_t)e0 * EB;
          if (e0 >= 0 && e0 + (int32_t)N <= (int32_t)rows) {
            *reinterpret_cast<uint32_t *>(g) = v;
          } else {
#pragma unroll
            for (uint32_t b = 0; b < N; b++)
              if ((uint32_t)(e0 + (int32_t)b) < rows) *reinterpret_cast<E *>(g + b * EB) = (E)(v >> (8 * EB * b));
          }
        }
      } else {
        const uint32_t h = (((uint32_t)(uintptr_t)slice + o) & 3u) / EB;
        const int32_t e0 = (int32_t)(w * N) - (int32_t)h;
        const unsigned char *p[N];
#pragma unroll
        for (uint32_t b = 0; b < N; b++)
          p[b] = s + hold_row<EB, FORM>(a, min((uint32_t)max(e0 + (int32_t)b, 0), rows - 1), lo, plo, sr) + j0 * EB;
        uint32_t v[U];
#pragma unroll
        for (uint32_t q = 0; q < U; q++) {
          v[q] = 0;
          if (q < left) {
#pragma unroll
            for (uint32_t b = 0; b < N; b++)
              v[q] |= (uint32_t) * reinterpret_cast<const E *>(p[b] + q * ps) << (8 * EB * b);
          }
        }
        char *g = slice + (size_t)o + (int64_t)e0 * EB;
        if (e0 >= 0 && e0 + (int32_t)N <= (int32_t)rows) {
#pragma unroll
          for (uint32_t q = 0; q < U; q++, g += gs)
            if (q < left) *reinterpret_cast<uint32_t *>(g) = v[q];
        } else {
          // a word across the end of the column's piece: its elements one by one
#pragma unroll
          for (uint32_t b = 0; b < N; b++)
            if ((uint32_t)(e0 + (int32_t)b) < rows) {
#pragma unroll
              for (uint32_t q = 0; q < U; q++)
                if (q < left) *reinterpret_cast<E *>(g + (size_t)(q * gs) + b * EB) = (E)(v[q] >> (8 * EB * b));
            }
        }
      }
    }
  }
}

// ---- team barrier ---------------------------------------------------------------
// Grid teams: an arrival counter and a generation word per (slot, team).  The
// last arrival resets the counter and raises the generation, so the words
// need no clearing between launches.  The launch is cooperative (all CTAs
// resident); the wait is bounded all the same.
__device__ __forceinline__ uint32_t ld_relaxed_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ bool hold_grid_arrive_wait(uint32_t *bar, uint32_t ctas, uint32_t gen) {
  uint32_t old;
  asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(bar) : "memory");
  if (old == ctas - 1) {
    asm volatile("st.relaxed.gpu.global.u32 [%0], 0;" ::"l"(bar) : "memory");
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(bar + 1), "r"(gen + 1) : "memory");
    return true;
  }
  const uint64_t t0 = global_ns();
  uint32_t spins = 0;
  while (ld_acquire_u32(bar + 1) == gen) {
    if ((++spins & 1023u) == 0 && global_ns() - t0 > kWaitNs) {
      // withdraw the arrival, so that the words are clear for later launches,
      // unless the barrier completed meanwhile
      uint32_t c = ld_relaxed_u32(bar);
      while (c != 0 && c < ctas) {
        const uint32_t was = atomicCAS(bar, c, c - 1);
        if (was == c) return false;
        c = was;
      }
      for (int i = 0; i < 1 << 20; i++)
        if (ld_acquire_u32(bar + 1) != gen) return true;
      return false;
    }
  }
  return true;
}

template <int EB, int FORM>
__global__ void __launch_bounds__(kHoldThreads, 2)
    k_hold(char *__restrict__ data, const __grid_constant__ HoldArgs a, uint32_t *bars, int *status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int ok_s;
  const uint32_t team = blockIdx.x / a.ctas, rank = blockIdx.x - team * a.ctas;
  int64_t k = team;
  if (k >= a.d3) return;
  uint32_t *bar = bars ? bars + ((size_t)a.slot * kHoldTeams + team) * 8 : nullptr;
  uint32_t gen = 0;
  if (a.mode == HOLD_GRID && threadIdx.x == 0) gen = ld_relaxed_u32(bar + 1);
  auto tile_pos = [&](uint32_t t, uint32_t &r0, uint32_t &c0) {
    const uint32_t tr = a.tcdiv.div(t);
    r0 = tr * a.tm;
    c0 = (t - tr * a.TC) * a.tn;
  };
  // item k: a slice, or a band of one.  RAG_DST takes a slice's bands from the
  // last to the first, because a band's columns reach past the end of its
  // rows into those of the band after it, which the barrier of the item
  // before has seen loaded; RAG_SRC takes them from the first to the last.
  // The next item's rows never overlap this item's columns, so they are
  // loaded while those are written.
  auto item = [&](int64_t kk, char *&slice, char *&from, uint32_t &s0) {
    if constexpr (FORM == HOLD_RAG_DST || FORM == HOLD_RAG_SRC) {
      const int64_t sl = kk / a.nb;
      const uint32_t b = FORM == HOLD_RAG_DST ? a.nb - 1 - (uint32_t)(kk - sl * a.nb) : (uint32_t)(kk - sl * a.nb);
      const size_t band = (size_t)b * a.m * a.n * EB;
      char *base = data + sl * a.slice_bytes;
      slice = FORM == HOLD_RAG_DST ? base : base + band;
      from = FORM == HOLD_RAG_DST ? base + band : base;
      s0 = b * (FORM == HOLD_RAG_DST ? a.n : a.m);
    } else {
      slice = from = data + kk * a.slice_bytes;
      s0 = 0;
    }
  };
  char *slice, *from;
  uint32_t s0;
  item(k, slice, from, s0);
  {
    uint32_t q = 0;
    for (uint32_t t = rank; t < a.T; t += a.ctas, q++) {
      uint32_t r0, c0;
      tile_pos(t, r0, c0);
      hold_load<EB, FORM>(from, a, r0, c0, smem_raw + (size_t)q * a.tile_bytes, s0);
    }
  }
  for (;;) {
    cp_async_wait_all();
    __syncthreads();  // the CTA's tiles have landed
    if (a.mode == HOLD_CLUSTER) {
      // execution order only: every thread has waited for its own copies
      asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    } else if (a.mode == HOLD_GRID) {
      if (threadIdx.x == 0) {
        ok_s = hold_grid_arrive_wait(bar, a.ctas, gen);
        gen++;
      }
      __syncthreads();
      if (!ok_s) {
        if (threadIdx.x == 0) atomicExch(status, 5 /* T213_ERR_TIMEOUT */);
        return;
      }
    }
    const int64_t next = k + a.teams;
    char *nslice = slice, *nfrom = from;
    uint32_t ns0 = s0;
    if (next < a.d3) item(next, nslice, nfrom, ns0);
    uint32_t q = 0;
    for (uint32_t t = rank; t < a.T; t += a.ctas, q++) {
      uint32_t r0, c0;
      tile_pos(t, r0, c0);
      unsigned char *buf = smem_raw + (size_t)q * a.tile_bytes;
      hold_store<EB, FORM>(slice, from, a, r0, c0, buf, s0);
      if (next < a.d3) {
        __syncthreads();  // every thread has read the tile: the next item's may land
        hold_load<EB, FORM>(nfrom, a, r0, c0, buf, ns0);
      }
    }
    if (next >= a.d3) break;
    k = next;
    slice = nslice;
    from = nfrom;
    s0 = ns0;
  }
}

// ---- many tensors in rounds -------------------------------------------------------
// The batched form: the slices of many tensors, cut into tiles, are dealt to
// the resident CTAs in rounds.  All tiles of a slice are in one round; a CTA
// has some tiles of every round, as many bytes as any other, in one of two
// buffers.  One grid barrier per round (every load of the round before any of
// its stores) is overlapped with the loads of the next round, which is in
// other slices: the barrier's latency costs nothing while rounds are large.
struct RoundTensor {
  HoldArgs a;
  char *data;
  int32_t kind;  // element bytes, negative for the vector form
};
struct RoundTile {
  uint32_t tensor, slice, tile, off;  // tile of the slice, byte offset in the buffer
};

template <int EB, int FORM>
__device__ __noinline__ void round_load(const RoundTensor &t, const RoundTile &ti, unsigned char *buf) {
  const HoldArgs a = t.a;  // a copy: the tile's stores must not make the compiler read it again
  const uint32_t tr = a.tcdiv.div(ti.tile);
  hold_load<EB, FORM>(t.data + (int64_t)ti.slice * a.slice_bytes, a, tr * a.tm, (ti.tile - tr * a.TC) * a.tn,
                      buf + ti.off, 0);
}
template <int EB, int FORM>
__device__ __noinline__ void round_store(const RoundTensor &t, const RoundTile &ti, const unsigned char *buf) {
  const HoldArgs a = t.a;
  const uint32_t tr = a.tcdiv.div(ti.tile);
  char *slice = t.data + (int64_t)ti.slice * a.slice_bytes;
  hold_store<EB, FORM>(slice, slice, a, tr * a.tm, (ti.tile - tr * a.TC) * a.tn, buf + ti.off, 0);
}

__global__ void __launch_bounds__(kHoldThreads, 2)
    k_hold_rounds(const RoundTensor *__restrict__ tensors, const RoundTile *__restrict__ tiles,
                  const uint32_t *__restrict__ first, uint32_t rounds, uint32_t buf_bytes, uint32_t *counter,
                  int *status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int ok_s;
  const uint32_t G = gridDim.x;
  auto load = [&](uint32_t r) {
    unsigned char *buf = smem_raw + (size_t)(r & 1) * buf_bytes;
    const uint32_t q0 = first[(size_t)r * G + blockIdx.x], q1 = first[(size_t)r * G + blockIdx.x + 1];
    for (uint32_t q = q0; q < q1; q++) {
      const RoundTile ti = tiles[q];
      const RoundTensor &t = tensors[ti.tensor];
      switch (t.kind) {
        case 1: round_load<1, HOLD_SCALAR>(t, ti, buf); break;
        case 2: round_load<2, HOLD_SCALAR>(t, ti, buf); break;
        case 4: round_load<4, HOLD_SCALAR>(t, ti, buf); break;
        case 8: round_load<8, HOLD_SCALAR>(t, ti, buf); break;
        case 16: round_load<16, HOLD_SCALAR>(t, ti, buf); break;
        case -2: round_load<2, HOLD_VEC>(t, ti, buf); break;
        default: round_load<4, HOLD_VEC>(t, ti, buf); break;
      }
    }
  };
  load(0);
  for (uint32_t r = 0; r < rounds; r++) {
    cp_async_wait_all();
    __syncthreads();  // this CTA's loads of round r have landed, its stores of round r - 1 are issued
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    if (r + 1 < rounds) load(r + 1);
    if (threadIdx.x == 0) {
      const uint32_t target = (r + 1) * G;
      const uint64_t t0 = global_ns();
      uint32_t spins = 0;
      int ok = 1;
      while (ld_acquire_u32(counter) < target) {
        if ((++spins & 1023u) == 0 && global_ns() - t0 > kWaitNs) {
          ok = 0;
          break;
        }
      }
      ok_s = ok;
    }
    __syncthreads();
    if (!ok_s) {
      cp_async_wait_all();
      if (threadIdx.x == 0) atomicExch(status, 5 /* T213_ERR_TIMEOUT */);
      return;
    }
    const unsigned char *buf = smem_raw + (size_t)(r & 1) * buf_bytes;
    const uint32_t q0 = first[(size_t)r * G + blockIdx.x], q1 = first[(size_t)r * G + blockIdx.x + 1];
    for (uint32_t q = q0; q < q1; q++) {
      const RoundTile ti = tiles[q];
      const RoundTensor &t = tensors[ti.tensor];
      switch (t.kind) {
        case 1: round_store<1, HOLD_SCALAR>(t, ti, buf); break;
        case 2: round_store<2, HOLD_SCALAR>(t, ti, buf); break;
        case 4: round_store<4, HOLD_SCALAR>(t, ti, buf); break;
        case 8: round_store<8, HOLD_SCALAR>(t, ti, buf); break;
        case 16: round_store<16, HOLD_SCALAR>(t, ti, buf); break;
        case -2: round_store<2, HOLD_VEC>(t, ti, buf); break;
        default: round_store<4, HOLD_VEC>(t, ti, buf); break;
      }
    }
  }
}

}  // namespace t213
