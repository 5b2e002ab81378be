// Launch of the kernel for many small slices (k_crumbs.cuh).
#include <algorithm>

#include "k_crumbs.cuh"

namespace t213 {

namespace {
template <int EB>
void launch(char *data, const CrumbArgs &a, int64_t grid, cudaStream_t st) {
  k_crumbs<EB><<<(unsigned)grid, kCrumbThreads, 0, st>>>(data, a);
}
}  // namespace

// Slices of up to 1 KB; up to 4 KB where lanes that read down a column fall
// into different banks (the power of two in their distance is at most 32
// bytes; a lane of 1- and 2-byte elements takes 4 or 2 rows).  More slices
// than two a SM: fewer leave SMs idle, which the one-pass slice kernel's small
// teams do not.  Measured on 120 MB (B200, us, floor 37), here / the best of
// blocks, bands and slice: fp32 (4, 4) 39 / far above 1000, (8, 8) 39 / 408,
// (16, 16) 45 / 105, (24, 24) 39 / 52, (31, 31) 39 / 80, bytes (16, 16) 84 /
// 386, bf16 (45, 45) 62 / 122; kept out: fp32 (16, 32) 71 / 54, (32, 32) 121 /
// 44, fp64 (16, 16) 74 / 53, bf16 (32, 32) 117 / 73.
bool crumbs_fit(int64_t m, int64_t n, int eb, int64_t d3) {
  if (m < 2 || n < 2 || m > kCrumbRun || n > kCrumbRun || d3 <= 2 * dev_info().sms) return false;
  const int64_t step = n * eb * std::max(1, 4 / eb), pow2 = step & -step;
  return m * n * eb <= 1024 || (m * n * eb <= kCrumbMax && pow2 <= 32);
}

int launch_crumbs(char *data, int64_t d3, int64_t m, int64_t n, int eb, cudaStream_t st, LaunchStats *ls, int64_t h2) {
  if (d3 <= 0) return T213_OK;
  CrumbArgs a{};
  a.d3 = d3;
  a.m = (uint32_t)m;
  a.n = (uint32_t)n;
  a.V = a.m * a.n;
  a.per = (uint32_t)(kCrumbRun / (m * n * eb));
  if (a.per >= 32) a.per -= a.per % 32;  // runs of whole sectors
  a.h2 = (uint32_t)h2;
  a.h1 = h2 ? (uint32_t)(m / h2) : 0;
  a.vdiv = FastDiv<uint32_t>((uint64_t)a.V);
  a.mdiv = FastDiv<uint32_t>((uint64_t)m);
  a.h2div = FastDiv<uint32_t>((uint64_t)std::max<int64_t>(h2, 1));
  const int64_t grid = std::min<int64_t>((d3 + a.per - 1) / a.per, 1 << 30);
  switch (eb) {
    case 1: launch<1>(data, a, grid, st); break;
    case 2: launch<2>(data, a, grid, st); break;
    case 4: launch<4>(data, a, grid, st); break;
    case 8: launch<8>(data, a, grid, st); break;
    case 16: launch<16>(data, a, grid, st); break;
    default: set_error("unsupported element size"); return T213_ERR_UNSUPPORTED;
  }
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e, "k_crumbs launch");
  if (ls) ls->launches++;
  return T213_OK;
}

}  // namespace t213
