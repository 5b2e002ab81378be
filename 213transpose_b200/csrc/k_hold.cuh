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
#include "team_barrier.cuh"
#include "tma.cuh"

namespace t213 {

constexpr int kHoldThreads = 512;
constexpr int kHoldSlots = 4096;  // barrier slots: one per stream, one per captured launch
constexpr int kHoldTeams = 20;    // grid teams of a launch (17 CTAs or more each)

// RAG_DST / RAG_SRC: scalar tiles of one band of a ragged band plan, whose
// output columns / source rows lie as the segments of rows with a remainder.
// RAG_SRC also takes slices whose rows come in swapped order (two steps of a
// rank-N permutation in one pass): row b * q + a of the output order is row
// a * h + b of the slice, which the same two constants say, with a negative
// remainder.
enum HoldForm { HOLD_SCALAR = 0, HOLD_VEC = 1, HOLD_WIDE = 2, HOLD_RAG_DST = 3, HOLD_RAG_SRC = 4 };

struct HoldArgs {
  int64_t d3, slice_bytes;
  uint32_t m, n;            // slice rows and columns (elements)
  uint32_t tm, tn, TC, T;   // tile sides, tiles per slice row, tiles per slice
  uint32_t ctas, teams, S;  // CTAs per team, teams, tiles per CTA (at most)
  uint32_t P, H, tile_bytes;  // shared-memory row pitch, region and tile size
  int32_t packed;             // narrow rows, one contiguous piece per tile
  int32_t bulk;               // row pieces come by bulk copies
  int32_t mode, slot;
  int32_t lgs;  // log2 of the lanes that share an output column
  uint32_t we;       // wide form: 16-byte words per element
  FastDiv<uint32_t> wediv, tcdiv, rbdiv;
  // ragged bands: m x n is a band, nb bands per slice; segment s of a slice is
  // seg_bytes long, and rest_bytes lie between the q-th segment of a row and
  // the next row
  FastDiv<uint32_t> qdiv;
  uint32_t nb, seg_bytes;
  int32_t rest_bytes;
  uint32_t need;     // arrivals that end a team barrier: ctas (one more in a test of the limit)
  uint64_t wait_ns;  // limit of a wait there
  __device__ __forceinline__ uint64_t seg_at(uint32_t s) const {
    return (uint64_t)((int64_t)s * seg_bytes + (int64_t)qdiv.div(s) * rest_bytes);
  }
};

// The warp's index, broadcast so that the compiler keeps what follows from it
// (unit, column, output row) in uniform registers.
__device__ __forceinline__ uint32_t warp_index() { return __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0); }

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

// Adds bytes that bulk copies will bring to what the barrier waits for.
__device__ __forceinline__ void mbar_expect(uint64_t *mb, uint32_t bytes) {
  asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(mb)), "r"(bytes) : "memory");
}
// After a warp's last load of an item: the barrier's phase ends when every
// warp has come here and every announced byte has landed.
__device__ __forceinline__ void hold_loaded(uint64_t *mb) {
  __syncwarp();
  if ((threadIdx.x & 31) == 0) mbar_arrive(mb);
}
// Waits, bounded, for an item's loads of either kind.
__device__ __forceinline__ bool hold_landed(uint64_t *mb, uint32_t &phase) {
  cp_async_wait_all();
  const bool ok = mbar_wait(mb, phase);
  phase ^= 1u;
  return __syncthreads_and(ok);
}

// `slice` is the slice, or the band's rows (RAG_DST), or the start of the
// slice that the band belongs to (RAG_SRC, with s0 the band's first segment).
template <int EB, int FORM, uint32_t THREADS = kHoldThreads>
__device__ __forceinline__ void hold_load(const char *slice, const HoldArgs &a, uint32_t r0, uint32_t c0,
                                          unsigned char *s, uint32_t s0, uint64_t *mb) {
  uint32_t rows = min(a.tm, a.m - r0), cols = min(a.tn, a.n - c0);
  const uint32_t E = EB * (FORM == HOLD_WIDE ? a.we : 1);
  const uint32_t pitch = a.n * E;  // a slice is far below 4 GB
  const char *g0 = slice + (FORM == HOLD_RAG_SRC ? 0 : (size_t)r0 * pitch) + (size_t)c0 * E;
  if ((FORM == HOLD_SCALAR || FORM == HOLD_RAG_DST) && a.packed) {
    const uint32_t sh = (uint32_t)(uintptr_t)g0 & 15u;
    const char *g = g0 - sh;
    const uint32_t nc = (sh + rows * pitch + 15) >> 4;
#pragma unroll 4
    for (uint32_t c = threadIdx.x; c < nc; c += THREADS) cp_async<16>(s + c * 16, g + c * 16);
    return;
  }
  if (FORM != HOLD_VEC && FORM != HOLD_WIDE && a.bulk) {
    // row pieces long enough for a bulk copy each: one thread a row
    constexpr uint32_t N = EB < 4 ? 4 / EB : 1;
    for (uint32_t base = threadIdx.x & ~31u; base < rows; base += THREADS) {
      const uint32_t i = base + (threadIdx.x & 31);
      const char *g = g0 + (FORM == HOLD_RAG_SRC ? (size_t)a.seg_at(s0 + r0 + min(i, rows - 1)) : (size_t)(i * pitch));
      const uint32_t sh = (uint32_t)(uintptr_t)g & 15u, l = i / N, b = i % N;
      const uint32_t bytes = i < rows ? (sh + cols * EB + 15) & ~15u : 0;
      const uint32_t sum = __reduce_add_sync(0xffffffffu, bytes);
      if ((threadIdx.x & 31) == 0) mbar_expect(mb, sum);
      __syncwarp();
      if (bytes) bulk_g2s(s + b * a.H + l * a.P + (l >> 3) * 16, g - sh, bytes, mb);
    }
    return;
  }
  // thread t takes blocks t, t + THREADS, ... of the tile's rows x nc blocks and
  // carries (row, block) along: no lane idles at a row's end
  const uint32_t nc = FORM == HOLD_VEC ? cols * EB / 16 : FORM == HOLD_WIDE ? cols * a.we : (cols * EB + 31 - EB) / 16;
  const uint32_t di = THREADS / nc, dc = THREADS - di * nc;
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
template <int EB, int FORM, bool ROUNDS = false>
__device__ __forceinline__ void hold_store(char *slice, const char *from, const HoldArgs &a, uint32_t r0, uint32_t c0,
                                           const unsigned char *s, uint32_t s0) {
  using E = typename ElemT<EB>::type;
  const uint32_t rows = min(a.tm, a.m - r0), cols = min(a.tn, a.n - c0);
  const uint32_t lane = threadIdx.x & 31, warp = warp_index();
  constexpr uint32_t nw = kHoldThreads / 32;
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
    // ROUNDS: the arguments take registers there, and 16 reads spill (a batch of
    // 64 tensors, 630 MB, 431 us with 16, 426 with 8)
    constexpr uint32_t U = EB == 16 ? 4 : EB == 4 && !ROUNDS ? 16 : 8;
    auto units = [&](auto whole) {
      // `whole`: the 32 lanes share a column
      constexpr bool W32 = decltype(whole)::value;
      const uint32_t lgs = W32 ? 5u : (uint32_t)a.lgs;
      const uint32_t L = 1u << lgs, G = W32 ? 1u : 32u >> lgs, li = W32 ? lane : lane & (L - 1), sub = W32 ? 0u : lane >> lgs;
      const uint32_t plo = a.n * EB;
      const uint32_t lo = (uint32_t)(uintptr_t)from + (FORM == HOLD_RAG_SRC ? c0 * EB : (r0 * a.n + c0) * EB);
      const uint32_t sr = s0 + r0;  // RAG_SRC: the segment of the tile's first row
      const uint32_t words = N == 1 ? rows : (rows + 2 * N - 2) / N;  // one more covers every offset
      const uint32_t nrb = (words + L - 1) >> lgs, ncg = (cols + U * G * N - 1) / (U * G * N) * N;
      const bool full = rows == a.tm;
      for (uint32_t u = warp; u < nrb * ncg; u += nw) {
        const uint32_t cg = full ? a.rbdiv.div(u) : u / nrb;
        const uint32_t w = ((u - cg * nrb) << lgs) + li;
        const uint32_t j0 = cg / N * (U * G * N) + cg % N * G + sub;
        if (w >= words || j0 >= cols) continue;
        [[maybe_unused]] const uint32_t o = ((c0 + j0) * a.m + r0) * EB;
        [[maybe_unused]] const uint32_t gs = G * N * a.m * EB;
        const uint32_t ps = G * N * EB;
        const uint32_t left = (cols - 1 - j0) / (G * N) + 1;  // column steps of this lane
        if constexpr (N == 1) {
          const unsigned char *p = s + hold_row<EB, FORM>(a, w, lo, plo, sr) + j0 * EB;
          E v[U];
          if constexpr (FORM == HOLD_RAG_DST) {
            const uint32_t sj = s0 + c0 + j0;
            char *g = slice + (size_t)((r0 + w) * EB) + a.seg_at(sj);
            uint32_t col = sj - a.qdiv.div(sj) * a.qdiv.get();  // the segment's place in its row
  #pragma unroll
            for (uint32_t q = 0; q < U; q++)
              if (q < left) v[q] = *reinterpret_cast<const E *>(p + q * ps);
  #pragma unroll
            for (uint32_t q = 0; q < U; q++) {
              if (q < left) *reinterpret_cast<E *>(g) = v[q];
              if constexpr (W32) {
                const bool wrap = ++col == a.qdiv.get();
                g += (size_t)a.seg_bytes + (wrap ? (uint32_t)a.rest_bytes : 0u);
                if (wrap) col = 0;
              } else {
                g = slice + (size_t)((r0 + w) * EB) + a.seg_at(sj + (q + 1) * G);
              }
            }
            continue;
          }
          char *g = slice + (size_t)(o + w * EB);
          if (left >= U) {
            if constexpr (W32) {  // consecutive columns: reads at constant offsets
  #pragma unroll
              for (uint32_t q = 0; q < U; q++) v[q] = *reinterpret_cast<const E *>(p + q * EB);
            } else {
  #pragma unroll
              for (uint32_t q = 0; q < U; q++) v[q] = *reinterpret_cast<const E *>(p + q * ps);
            }
  #pragma unroll
            for (uint32_t q = 0; q < U; q++, g += gs) *reinterpret_cast<E *>(g) = v[q];
          } else {
  #pragma unroll
            for (uint32_t q = 0; q < U; q++)
              if (q < left) *reinterpret_cast<E *>(g + (size_t)(q * gs)) = *reinterpret_cast<const E *>(p + q * ps);
          }
        } else if constexpr (FORM == HOLD_RAG_DST) {
          // the offset of an output row in its first word is the column's own:
          // the N rows of the word are picked out of the 2 N - 1 that they can be
          uint32_t ro[2 * N - 1];
  #pragma unroll
          for (uint32_t b = 0; b < 2 * N - 1; b++)
            ro[b] = hold_row<EB, FORM>(a, min((uint32_t)max((int32_t)(w * N + b) - (int32_t)(N - 1), 0), rows - 1), lo, plo, sr);
          const uint32_t sj = s0 + c0 + j0;
          char *g0 = slice + (size_t)(r0 * EB);
  #pragma unroll 4
          for (uint32_t q = 0; q < min(left, U); q++) {
            char *g = g0 + a.seg_at(sj + q * (G * N));
            const uint32_t h = ((uint32_t)(uintptr_t)g & 3u) / EB, at = N - 1 - h;
            uint32_t x[2 * N - 1];
  #pragma unroll
            for (uint32_t b = 0; b < 2 * N - 1; b++) x[b] = ro[b];
  #pragma unroll
            for (uint32_t k = 1; k < N; k *= 2) {
  #pragma unroll
              for (uint32_t b = 0; b + k < 2 * N - 1; b++) x[b] = at & k ? x[b + k] : x[b];
            }
            const unsigned char *p = s + j0 * EB + q * ps;
            uint32_t v = 0;
  #pragma unroll
            for (uint32_t b = 0; b < N; b++) v |= (uint32_t) * reinterpret_cast<const E *>(p + x[b]) << (8 * EB * b);
            const int32_t e0 = (int32_t)(w * N) - (int32_t)h;
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
    };
    if (a.lgs == 5)
      units(std::true_type{});
    else
      units(std::false_type{});
  }
}

// ---- team barrier (team_barrier.cuh) ----------------------------------------------
__device__ __forceinline__ uint32_t ld_acquire_u32(const uint32_t *p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
struct TeamWord {
  uint32_t *p;
  __device__ __forceinline__ uint32_t load() const { return ld_acquire_u32(p); }
  __device__ __forceinline__ uint32_t add1() const {
    uint32_t old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], 1;" : "=r"(old) : "l"(p) : "memory");
    return old;
  }
  __device__ __forceinline__ void store(uint32_t v) const {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
  }
  __device__ __forceinline__ uint32_t cas(uint32_t old, uint32_t v) const { return atomicCAS(p, old, v); }
};

__device__ __forceinline__ bool hold_grid_wait(uint32_t *bar, const HoldArgs &a, uint32_t gen) {
  const TeamWord w{bar};
  const uint64_t t0 = global_ns();
  uint32_t spins = 0;
  while (team_gen(w.load()) == gen)
    if ((++spins & 1023u) == 0 && global_ns() - t0 > a.wait_ns) return !team_withdraw(w, a.need, gen);
  return true;
}

// Arrives; true when this was the last arrival, which also ends the barrier.
__device__ __forceinline__ bool hold_grid_arrive(uint32_t *bar, const HoldArgs &a, uint32_t gen) {
  return team_arrive(TeamWord{bar}, a.need, gen);
}

template <int EB, int FORM>
__global__ void __launch_bounds__(kHoldThreads, 2)
    k_hold(char *__restrict__ data, const __grid_constant__ HoldArgs a, uint32_t *bars, int *status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int ok_s;
  __shared__ uint64_t mb;
  const uint32_t team = blockIdx.x / a.ctas, rank = blockIdx.x - team * a.ctas;
  int64_t k = team;
  if (k >= a.d3) return;
  if (threadIdx.x == 0) {
    mbar_init(&mb, kHoldThreads / 32);
    fence_barrier_init();
  }
  __syncthreads();
  uint32_t phase = 0;
  uint32_t *bar = bars ? bars + ((size_t)a.slot * kHoldTeams + team) * 8 : nullptr;
  uint32_t gen = 0;
  if (a.mode == HOLD_GRID && threadIdx.x == 0) gen = team_gen(TeamWord{bar}.load());
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
      hold_load<EB, FORM>(from, a, r0, c0, smem_raw + (size_t)q * a.tile_bytes, s0, &mb);
    }
    hold_loaded(&mb);
  }
  for (;;) {
    // the CTA's tiles have landed; a copy that never does is reported, and
    // the team's other CTAs run out of the same patience at their barrier
    if (!hold_landed(&mb, phase)) {
      if (threadIdx.x == 0) atomicExch(status, 5 /* T213_ERR_TIMEOUT */);
      return;
    }
    if (a.mode == HOLD_CLUSTER) {
      // execution order only: every thread has waited for its own copies
      asm volatile("barrier.cluster.arrive.relaxed.aligned;\n\tbarrier.cluster.wait.aligned;" ::: "memory");
    } else if (a.mode == HOLD_GRID) {
      if (threadIdx.x == 0) {
        ok_s = hold_grid_arrive(bar, a, gen) || hold_grid_wait(bar, a, gen);
        gen += kTeamGen;
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
        fence_proxy_async();
        hold_load<EB, FORM>(nfrom, a, r0, c0, buf, ns0, &mb);
      }
    }
    if (next < a.d3) hold_loaded(&mb);
    if (next >= a.d3) break;
    k = next;
    slice = nslice;
    from = nfrom;
    s0 = ns0;
  }
}

// ---- several slices per team: tensor memory as the second buffer -----------------
// A team that takes one slice after the other would have to wait for the
// barrier with nothing in flight once its tile fills the shared memory.  Here
// a landed tile moves on to the SM's tensor memory (TMEM, 256 KB beside the
// shared memory) before the barrier, in the order in which it will be written:
// lane l of a warp's quarter holds output word l of a column, successive TMEM
// columns successive matrix columns, so that a 32x32b load hands every lane
// the words it writes and the transposition costs no second pass.  The shared
// memory is free at once: the next slice's loads are in flight during the
// barrier and the stores.  TMEM is used as memory only; a warp reads back what
// it wrote itself.
//
// One CTA of 1024 threads per SM: a kernel that allocates tensor memory is
// resident once per SM, whatever its size.
constexpr int kTmemThreads = 1024;
constexpr int kTmemCols = 512;
constexpr int kTmemUnitCols = 16;  // one unit: 16 words per lane
constexpr int kTmemWarpCols = kTmemCols / (kTmemThreads / 128);  // 8 warps share a quarter's lanes
constexpr int kTmemUnits = kTmemWarpCols / kTmemUnitCols;        // per warp

__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
      "%16};" ::"r"(addr),
      "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
      "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
      : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];\n\ttcgen05.wait::ld.sync.aligned;"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(addr)
      : "memory");
}

// The units of hold_store's scalar form with 16 words per lane.  W32: the 32
// lanes share a column, and all but the lane's word is uniform in the warp.
template <int EB, bool W32>
struct TmemUnit {
  static constexpr uint32_t N = EB < 4 ? 4 / EB : 1;
  static constexpr uint32_t W = EB < 4 ? 1 : EB / 4;  // words per element
  static constexpr uint32_t U = kTmemUnitCols / W;    // column steps
  uint32_t w, j0, left, gn;  // word, first column, column steps left, columns per step
  bool in;                   // the lane has a word
  __device__ __forceinline__ TmemUnit(const HoldArgs &a, uint32_t u, uint32_t rows, uint32_t cols, uint32_t lane) {
    const uint32_t lgs = W32 ? 5u : (uint32_t)a.lgs;
    const uint32_t L = 1u << lgs, G = W32 ? 1u : 32u >> lgs;
    const uint32_t li = W32 ? lane : lane & (L - 1), sub = W32 ? 0u : lane >> lgs;
    const uint32_t words = N == 1 ? rows : (rows + 2 * N - 2) / N;
    const uint32_t nrb = (words + L - 1) >> lgs;
    const uint32_t cg = rows == a.tm ? a.rbdiv.div(u) : u / nrb;
    w = ((u - cg * nrb) << lgs) + li;
    gn = G * N;
    j0 = cg / N * (U * gn) + cg % N * G + sub;
    left = j0 < cols ? min((cols - 1 - j0) / gn + 1, U) : 0;
    in = w < words;
  }
  __device__ static __forceinline__ uint32_t count(const HoldArgs &a, uint32_t rows, uint32_t cols) {
    const uint32_t L = 1u << a.lgs, G = 32u >> a.lgs;
    const uint32_t words = N == 1 ? rows : (rows + 2 * N - 2) / N;
    return ((words + L - 1) >> a.lgs) * ((cols + U * G * N - 1) / (U * G * N) * N);
  }
};

template <int EB, int FORM, bool W32>
__device__ __forceinline__ void tmem_fill(const char *slice, const char *from, const HoldArgs &a, uint32_t r0,
                                          uint32_t c0, const unsigned char *s, uint32_t s0, uint32_t taddr) {
  using E = typename ElemT<EB>::type;
  using TU = TmemUnit<EB, W32>;
  constexpr uint32_t N = TU::N;
  const uint32_t rows = min(a.tm, a.m - r0), cols = min(a.tn, a.n - c0);
  const uint32_t lane = threadIdx.x & 31, warp = warp_index();
  const uint32_t plo = a.n * EB;
  const uint32_t lo = (uint32_t)(uintptr_t)from + (FORM == HOLD_RAG_SRC ? c0 * EB : (r0 * a.n + c0) * EB);
  const uint32_t sr = s0 + r0;
  const uint32_t units = TU::count(a, rows, cols);
  for (uint32_t u = warp; u < units; u += kTmemThreads / 32, taddr += kTmemUnitCols) {
    const TU t(a, u, rows, cols, lane);
    const uint32_t j0 = min(t.j0, cols - 1);
    union {
      uint32_t w[16];
      E e[TU::U];
    } v;
    const unsigned char *p[N];
    if constexpr (N == 1) {
      // lanes without a word read the last row's, and write nothing later
      p[0] = s + hold_row<EB, FORM>(a, min(t.w, rows - 1), lo, plo, sr) + j0 * EB;
    } else {
      const uint32_t h = (((uint32_t)(uintptr_t)slice + ((c0 + t.j0) * a.m + r0) * EB) & 3u) / EB;
      const int32_t e0 = (int32_t)(t.w * N) - (int32_t)h;
#pragma unroll
      for (uint32_t b = 0; b < N; b++)
        p[b] = s + hold_row<EB, FORM>(a, min((uint32_t)max(e0 + (int32_t)b, 0), rows - 1), lo, plo, sr) + j0 * EB;
    }
    auto read = [&](uint32_t q, uint32_t off) {
      if constexpr (N == 1) {
        v.e[q] = *reinterpret_cast<const E *>(p[0] + off);
      } else {
        v.w[q] = 0;
#pragma unroll
        for (uint32_t b = 0; b < N; b++)
          v.w[q] |= (uint32_t) * reinterpret_cast<const E *>(p[b] + off) << (8 * EB * b);
      }
    };
    if (W32 && t.left == TU::U) {
#pragma unroll
      for (uint32_t q = 0; q < TU::U; q++) read(q, q * N * EB);
    } else {
#pragma unroll
      for (uint32_t q = 0; q < TU::U; q++)
        if (q < t.left) read(q, q * t.gn * EB);
    }
    __syncwarp();
    tmem_st16(taddr, v.w);
  }
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

template <int EB, int FORM, bool W32>
__device__ __forceinline__ void tmem_drain(char *slice, const HoldArgs &a, uint32_t r0, uint32_t c0, uint32_t s0,
                                           uint32_t taddr) {
  using E = typename ElemT<EB>::type;
  using TU = TmemUnit<EB, W32>;
  constexpr uint32_t N = TU::N;
  const uint32_t rows = min(a.tm, a.m - r0), cols = min(a.tn, a.n - c0);
  const uint32_t lane = threadIdx.x & 31, warp = warp_index();
  const uint32_t units = TU::count(a, rows, cols);
  for (uint32_t u = warp; u < units; u += kTmemThreads / 32, taddr += kTmemUnitCols) {
    const TU t(a, u, rows, cols, lane);
    union {
      uint32_t w[16];
      E e[TU::U];
    } v;
    __syncwarp();
    tmem_ld16(taddr, v.w);
    if (!t.in) continue;
    if constexpr (FORM == HOLD_RAG_DST) {
      static_assert(N == 1, "the byte offset of an output row is its own");
      const uint32_t sj = s0 + c0 + t.j0;
      char *g = slice + (size_t)((r0 + t.w) * EB) + a.seg_at(sj);
      uint32_t col = sj - a.qdiv.div(sj) * a.qdiv.get();  // the segment's place in its row
#pragma unroll
      for (uint32_t q = 0; q < TU::U; q++) {
        if (q < t.left) *reinterpret_cast<E *>(g) = v.e[q];
        if constexpr (W32) {
          const bool wrap = ++col == a.qdiv.get();
          g += (size_t)a.seg_bytes + (wrap ? (uint32_t)a.rest_bytes : 0u);
          if (wrap) col = 0;
        } else {
          g = slice + (size_t)((r0 + t.w) * EB) + a.seg_at(sj + (q + 1) * t.gn);
        }
      }
    } else {
      const uint32_t o = ((c0 + t.j0) * a.m + r0) * EB, gs = t.gn * a.m * EB;
      if constexpr (N == 1) {
        char *g = slice + (size_t)(o + t.w * EB);
        if (W32 && t.left == TU::U) {
#pragma unroll
          for (uint32_t q = 0; q < TU::U; q++, g += gs) *reinterpret_cast<E *>(g) = v.e[q];
        } else {
#pragma unroll
          for (uint32_t q = 0; q < TU::U; q++, g += gs)
            if (q < t.left) *reinterpret_cast<E *>(g) = v.e[q];
        }
      } else {
        const uint32_t h = (((uint32_t)(uintptr_t)slice + o) & 3u) / EB;
        const int32_t e0 = (int32_t)(t.w * N) - (int32_t)h;
        char *g = slice + (size_t)o + (int64_t)e0 * EB;
        if (e0 >= 0 && e0 + (int32_t)N <= (int32_t)rows) {
          if (W32 && t.left == TU::U) {
#pragma unroll
            for (uint32_t q = 0; q < 16; q++, g += gs) *reinterpret_cast<uint32_t *>(g) = v.w[q];
          } else {
#pragma unroll
            for (uint32_t q = 0; q < 16; q++, g += gs)
              if (q < t.left) *reinterpret_cast<uint32_t *>(g) = v.w[q];
          }
        } else {
#pragma unroll
          for (uint32_t b = 0; b < N; b++)
            if ((uint32_t)(e0 + (int32_t)b) < rows) {
#pragma unroll
              for (uint32_t q = 0; q < 16; q++)
                if (q < t.left) *reinterpret_cast<E *>(g + (size_t)(q * gs) + b * EB) = (E)(v.w[q] >> (8 * EB * b));
            }
        }
      }
    }
  }
}

template <int EB, int FORM>
__global__ void __launch_bounds__(kTmemThreads, 1)
    k_hold_tmem(char *__restrict__ data, const __grid_constant__ HoldArgs a, uint32_t *bars, int *status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int ok_s;
  __shared__ uint32_t tbase_s;
  __shared__ uint64_t mb;
  if (threadIdx.x == 0) {
    mbar_init(&mb, kTmemThreads / 32);
    fence_barrier_init();
  }
  uint32_t phase = 0;
  const uint32_t team = blockIdx.x / a.ctas, rank = blockIdx.x - team * a.ctas;
  int64_t k = team;
  const uint32_t warp = threadIdx.x >> 5;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tbase_s)),
                 "n"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  uint32_t *bar = bars + ((size_t)a.slot * kHoldTeams + team) * 8;
  uint32_t gen = 0;
  if (threadIdx.x == 0) gen = team_gen(TeamWord{bar}.load());
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tbase = tbase_s;
  // a warp reaches the 32 lanes of its quarter; the 8 warps of a quarter have
  // an eighth of the columns each
  const uint32_t taddr = tbase + ((warp & 3u) << 21) + (warp >> 2) * kTmemWarpCols;
  const bool mine = rank < a.T;
  const uint32_t tr = a.tcdiv.div(rank), r0 = tr * a.tm, c0 = (rank - tr * a.TC) * a.tn;
  auto item = [&](int64_t kk, char *&slice, char *&from, uint32_t &s0) {
    if constexpr (FORM == HOLD_RAG_DST || FORM == HOLD_RAG_SRC) {  // as in k_hold
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
  char *slice = nullptr, *from = nullptr;
  uint32_t s0 = 0;
  if (k < a.d3) {
    item(k, slice, from, s0);
    if (mine) hold_load<EB, FORM, kTmemThreads>(from, a, r0, c0, smem_raw, s0, &mb);
    hold_loaded(&mb);
  }
  while (k < a.d3) {
    if (!hold_landed(&mb, phase)) {  // as in k_hold
      if (threadIdx.x == 0) atomicExch(status, 5 /* T213_ERR_TIMEOUT */);
      break;
    }
    bool last = false;
    if (threadIdx.x == 0) last = hold_grid_arrive(bar, a, gen);
    if (mine) {
      if (a.lgs == 5)
        tmem_fill<EB, FORM, true>(slice, from, a, r0, c0, smem_raw, s0, taddr);
      else
        tmem_fill<EB, FORM, false>(slice, from, a, r0, c0, smem_raw, s0, taddr);
    }
    __syncthreads();  // every warp has read the tile: the next slice's may land
    const int64_t next = k + a.teams;
    char *nslice = slice, *nfrom = from;
    uint32_t ns0 = s0;
    if (next < a.d3) {
      item(next, nslice, nfrom, ns0);
      fence_proxy_async();
      if (mine) hold_load<EB, FORM, kTmemThreads>(nfrom, a, r0, c0, smem_raw, ns0, &mb);
      hold_loaded(&mb);
    }
    if (threadIdx.x == 0) {
      ok_s = last || hold_grid_wait(bar, a, gen);
      gen += kTeamGen;
    }
    __syncthreads();
    if (!ok_s) {
      if (next < a.d3) hold_landed(&mb, phase);  // nothing may land after the CTA has gone
      if (threadIdx.x == 0) atomicExch(status, 5 /* T213_ERR_TIMEOUT */);
      break;
    }
    if (mine) {
      if (a.lgs == 5)
        tmem_drain<EB, FORM, true>(slice, a, r0, c0, s0, taddr);
      else
        tmem_drain<EB, FORM, false>(slice, a, r0, c0, s0, taddr);
    }
    k = next;
    slice = nslice;
    from = nfrom;
    s0 = ns0;
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "n"(kTmemCols) : "memory");
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
__device__ __noinline__ void round_load(const RoundTensor &t, const RoundTile &ti, unsigned char *buf, uint64_t *mb) {
  const HoldArgs a = t.a;  // a copy: the tile's stores must not make the compiler read it again
  const uint32_t tr = a.tcdiv.div(ti.tile);
  hold_load<EB, FORM>(t.data + (int64_t)ti.slice * a.slice_bytes, a, tr * a.tm, (ti.tile - tr * a.TC) * a.tn,
                      buf + ti.off, 0, mb);
}
template <int EB, int FORM>
__device__ __noinline__ void round_store(const RoundTensor &t, const RoundTile &ti, const unsigned char *buf) {
  const HoldArgs a = t.a;
  const uint32_t tr = a.tcdiv.div(ti.tile);
  char *slice = t.data + (int64_t)ti.slice * a.slice_bytes;
  hold_store<EB, FORM, true>(slice, slice, a, tr * a.tm, (ti.tile - tr * a.TC) * a.tn, buf + ti.off, 0);
}

__global__ void __launch_bounds__(kHoldThreads, 2)
    k_hold_rounds(const RoundTensor *__restrict__ tensors, const RoundTile *__restrict__ tiles,
                  const uint32_t *__restrict__ first, uint32_t rounds, uint32_t buf_bytes, uint32_t *counter,
                  uint32_t extra, uint64_t wait_ns, int *status) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  __shared__ int ok_s;
  __shared__ uint64_t mb;
  if (threadIdx.x == 0) {
    mbar_init(&mb, kHoldThreads / 32);
    fence_barrier_init();
  }
  __syncthreads();
  uint32_t phase = 0;
  const uint32_t G = gridDim.x;
  auto load = [&](uint32_t r) {
    unsigned char *buf = smem_raw + (size_t)(r & 1) * buf_bytes;
    const uint32_t q0 = first[(size_t)r * G + blockIdx.x], q1 = first[(size_t)r * G + blockIdx.x + 1];
    for (uint32_t q = q0; q < q1; q++) {
      const RoundTile ti = tiles[q];
      const RoundTensor &t = tensors[ti.tensor];
      switch (t.kind) {
        case 1: round_load<1, HOLD_SCALAR>(t, ti, buf, &mb); break;
        case 2: round_load<2, HOLD_SCALAR>(t, ti, buf, &mb); break;
        case 4: round_load<4, HOLD_SCALAR>(t, ti, buf, &mb); break;
        case 8: round_load<8, HOLD_SCALAR>(t, ti, buf, &mb); break;
        case 16: round_load<16, HOLD_SCALAR>(t, ti, buf, &mb); break;
        case -2: round_load<2, HOLD_VEC>(t, ti, buf, &mb); break;
        default: round_load<4, HOLD_VEC>(t, ti, buf, &mb); break;
      }
    }
    hold_loaded(&mb);
  };
  load(0);
  for (uint32_t r = 0; r < rounds; r++) {
    // this CTA's loads of round r have landed, its stores of round r - 1 are issued
    if (!hold_landed(&mb, phase)) {
      if (threadIdx.x == 0) atomicExch(status, 5 /* T213_ERR_TIMEOUT */);
      return;
    }
    fence_proxy_async();
    if (threadIdx.x == 0) asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(counter) : "memory");
    if (r + 1 < rounds) load(r + 1);
    if (threadIdx.x == 0) {
      const uint32_t target = (r + 1) * G + extra;
      const uint64_t t0 = global_ns();
      uint32_t spins = 0;
      int ok = 1;
      while (ld_acquire_u32(counter) < target) {
        if ((++spins & 1023u) == 0 && global_ns() - t0 > wait_ns) {
          ok = 0;
          break;
        }
      }
      ok_s = ok;
    }
    __syncthreads();
    if (!ok_s) {
      if (r + 1 < rounds) hold_landed(&mb, phase);  // nothing may land after the CTA has gone
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
