// Many slices of at most a few KB: matrices of a handful of elements, such as
// (d3, 3, 3) or (d3, 4, 4).
//
// A CTA takes a run of whole slices, about 16 KB and contiguous, into shared
// memory by the 16-byte blocks that cover it, and writes the run back in
// order, each output element picked from its place: reads and writes of memory
// are whole lines whatever the sides, and nothing is exchanged between CTAs.
// (The blocks at a run's ends hold bytes of its neighbours, never used.)
//
// Bound by memory for elements of 4 bytes and more (fp32 (3, 3, 3333333), 120
// MB, 39 us, 0.95 of the copy rate), for 1- and 2-byte elements by the index
// arithmetic (a word of 4 bytes is put together from 4 or 2 elements, one
// division for the first; 84 and 62 us).  Eight CTAs per SM keep 128 KB in
// flight.
#pragma once

#include "common.cuh"
#include "internal.h"
#include "tma.cuh"

namespace t213 {

constexpr int kCrumbThreads = 256;
constexpr int kCrumbRun = 16 * 1024;  // bytes of a run

struct CrumbArgs {
  int64_t d3;
  uint32_t m, n, V, per;  // rows, columns, elements of a slice, slices of a run
  uint32_t h1, h2;        // h2: row b * h2 + a of the output order is row a * h1 + b; 0: in order
  FastDiv<uint32_t> vdiv, mdiv, h2div;
  __device__ __forceinline__ uint32_t row(uint32_t i) const {
    if (h2 == 0) return i;
    const uint32_t b = h2div.div(i);
    return (i - b * h2) * h1 + b;
  }
};

template <int EB>
__global__ void __launch_bounds__(kCrumbThreads, 8) k_crumbs(char *__restrict__ data, const __grid_constant__ CrumbArgs a) {
  using E = typename ElemT<EB>::type;
  __shared__ __align__(16) unsigned char s[kCrumbRun + 32];
  for (int64_t r0 = (int64_t)blockIdx.x * a.per; r0 < a.d3; r0 += (int64_t)gridDim.x * a.per) {
    char *base = data + r0 * a.V * EB;
    const uint32_t total = (uint32_t)min((int64_t)a.per, a.d3 - r0) * a.V;
    const uint32_t sh = (uint32_t)(uintptr_t)base & 15u, nc = (sh + total * EB + 15) >> 4;
    for (uint32_t c = threadIdx.x; c < nc; c += kCrumbThreads) cp_async<16>(s + c * 16, base - sh + c * 16);
    cp_async_wait_all();
    __syncthreads();
    const unsigned char *p = s + sh;
    auto pick = [&](uint32_t sl, uint32_t j, uint32_t i) {
      return *reinterpret_cast<const E *>(p + (sl * a.V + a.row(i) * a.n + j) * EB);
    };
    auto element = [&](uint32_t e) {
      const uint32_t sl = a.vdiv.div(e), r = e - sl * a.V, j = a.mdiv.div(r);
      return pick(sl, j, r - j * a.m);
    };
    if constexpr (EB >= 4) {
#pragma unroll 4
      for (uint32_t e = threadIdx.x; e < total; e += kCrumbThreads) reinterpret_cast<E *>(base)[e] = element(e);
    } else {
      constexpr uint32_t N = 4 / EB;
      const uint32_t head = min(((4u - ((uint32_t)(uintptr_t)base & 3u)) & 3u) / EB, total);
      const uint32_t words = (total - head) / N, tail = total - head - words * N;
      uint32_t *o = reinterpret_cast<uint32_t *>(base + head * EB);
#pragma unroll 2
      for (uint32_t w = threadIdx.x; w < words; w += kCrumbThreads) {
        const uint32_t e = head + w * N;
        uint32_t sl = a.vdiv.div(e), r = e - sl * a.V, j = a.mdiv.div(r), i = r - j * a.m, v = 0;
#pragma unroll
        for (uint32_t b = 0; b < N; b++) {
          v |= (uint32_t)pick(sl, j, i) << (8 * EB * b);
          if (++i == a.m) {
            i = 0;
            if (++j == a.n) {
              j = 0;
              sl++;
            }
          }
        }
        o[w] = v;
      }
      if (threadIdx.x < head + tail) {
        const uint32_t e = threadIdx.x < head ? threadIdx.x : threadIdx.x + words * N;
        reinterpret_cast<E *>(base)[e] = element(e);
      }
    }
    __syncthreads();  // the run has been read: the next may land
  }
}

}  // namespace t213
