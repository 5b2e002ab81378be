// Geometry and launch of the one-pass slice kernel (k_hold.cuh).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <deque>
#include <map>
#include <thread>
#include <tuple>
#include <vector>

#include "internal.h"
#include "k_hold.cuh"

namespace t213 {

struct HoldReady {
  std::mutex mu;
  struct Form {
    std::atomic<bool> ready{false};
    HoldArgs args{};
    const void *kern = nullptr;
    int64_t smem = 0;
    int resident = 1;  // teams resident at once (grid teams: on all SMs of the device)
    int per_sm = 1;    // grid teams: CTAs resident on an SM
    uint32_t *bars = nullptr;
    int *status = nullptr;
  } any, vec;
};

namespace {

__device__ uint32_t g_hold_bars[(size_t)kHoldSlots * kHoldTeams * 8];

// Shared memory of one CTA when two are resident on an SM.
int64_t hold_budget() {
  const DevInfo &d = dev_info();
  const int64_t half = d.smem_per_sm / 2 - 1024 - 320;  // 1 KB reserved per CTA, the barrier flag, rounding
  return std::min<int64_t>(half, d.smem_optin - 64) / 128 * 128;
}

int64_t up(int64_t x, int64_t u) { return (x + u - 1) / u * u; }

// Row pitch in shared memory (see the layout in k_hold.cuh): an odd number of
// 16-byte blocks; whole 128-byte groups for the swizzled vector form.
int64_t hold_pitch(int64_t tn, int eb, int64_t we, int form) {
  if (form == HOLD_VEC) return up(tn * eb, 128);
  if (form == HOLD_WIDE) return ((tn * we) | 1) * 16;
  if (eb == 16) return (tn | 1) * 16;
  return (((tn * eb + 15 - eb) / 16 + 1) | 1) * 16;  // the blocks that cover a piece at any offset
}

// Bytes of one region of a tile (the tile itself unless the elements are
// smaller than 4 bytes).
int64_t hold_region(int64_t tm, int64_t P, int eb, int form) {
  if (form == HOLD_VEC || form == HOLD_WIDE) return tm * P;
  const int64_t N = eb < 4 ? 4 / eb : 1, l = (tm + N - 1) / N;
  return l * P + l / 8 * 16;
}

int64_t hold_tile_bytes(int64_t tm, int64_t tn, int64_t P, int eb, int form, bool packed) {
  if (packed) return up(tm * tn * eb + 30, 128);
  const int64_t N = form != HOLD_VEC && form != HOLD_WIDE && eb < 4 ? 4 / eb : 1;
  return up(N * hold_region(tm, P, eb, form), 128);
}

// Narrow rows whose whole width is in the tile are kept packed: nothing is
// lost to the 16-byte blocks of every row, and at strides with few common
// factors with the 32 banks a column costs few conflicts.
bool hold_packed(int64_t n, int eb, int form) {
  if ((form != HOLD_SCALAR && form != HOLD_RAG_DST) || n * eb > 256) return false;
  const int64_t stride = eb < 4 ? n : n * eb / 4;  // words from lane to lane
  int64_t g = 1;
  while (g < 32 && stride % (g * 2) == 0) g *= 2;
  return n * eb < 32 || g <= std::max(1, eb / 4) * 2;
}

int lanes_log2(int64_t x) {
  int l = 0;
  while (l < 5 && (1 << l) < x) l++;
  return l;
}

// The tiling of m x n slices of eb-byte elements (we 16-byte words each in the
// wide form): tile sides, team size and mode with the smallest modelled time.
//
// Model (B200): an SM moves its CTAs' shares at most at 60 GB/s and all SMs
// together at 6.4 TB/s; a slice costs a load and a store latency of
// 1 us each and a barrier with its costlier launch (cluster 1.2 us, grid 2.5 us);
// a slice of one CTA waits for no other; short row pieces cost
// a 32-byte sector more per piece.
// `tmem`: tilings of the form that keeps a team's next slice in flight
// (k_hold_tmem): one tile per CTA, its words in the SM's tensor
// memory; the barrier and the latencies are then hidden from the second slice
// on, and 1 us a slice is left.
// `bands`: the items of a slice are its bands, taken in order by one team.
bool hold_search(HoldGeom &g, int64_t m, int64_t n, int eb, int64_t we, int64_t d3, int form, bool tmem = false,
                 bool bands = true) {
  const DevInfo &d = dev_info();
  const int64_t E = eb * we;
  const int64_t budget = tmem ? (d.smem_optin - 128) / 128 * 128 : hold_budget();
  const int64_t slots = tmem ? d.sms : 2ll * d.sms;
  const int64_t Q = form == HOLD_VEC ? 16 / eb : 1;
  // tile sides in whole 32-byte sectors where the rows are
  const int64_t un = std::max<int64_t>(Q, (n * E) % 32 == 0 && E < 32 ? 32 / E : 1);
  const int64_t um = std::max<int64_t>(Q, (m * E) % 32 == 0 && E < 32 ? 32 / E : 1);
  const bool rag = bands && (form == HOLD_RAG_DST || form == HOLD_RAG_SRC);
  double best = 1e30;
  g.ok = false;
  const int64_t N4 = eb < 4 ? 4 / eb : 1;
  auto tmem_fits = [&](int64_t tm, int64_t tn) {
    const int64_t words = N4 == 1 ? tm : (tm + 2 * N4 - 2) / N4, U = kTmemUnitCols / std::max(1, eb / 4);
    const int lg = lanes_log2(words);
    const int64_t step = U * (32 >> lg) * N4;
    return ((words + (1 << lg) - 1) >> lg) * ((tn + step - 1) / step * N4) <= kTmemUnits * (kTmemThreads / 32);
  };
  for (int S = 1; S <= (tmem ? 1 : 2); S++) {
    const int64_t tile_cap = budget / S;
    const int64_t max_tiles = slots * S;
    for (int64_t TC = 1; TC <= std::min<int64_t>(max_tiles, n); TC = TC < 48 ? TC + 1 : TC + TC / 16) {
      const int64_t tn = std::min(n, up((n + TC - 1) / TC, un));
      const int64_t tcs = (n + tn - 1) / tn;
      const bool packed = tcs == 1 && hold_packed(n, eb, form);
      const int64_t P = packed ? n * eb : hold_pitch(tn, eb, we, form);
      auto fits = [&](int64_t tm) { return hold_tile_bytes(tm, tn, P, eb, form, packed) <= tile_cap; };
      if (!fits(1)) continue;
      int64_t tm_max = std::max<int64_t>(1, tile_cap / P);
      if (tm_max > um) tm_max = tm_max / um * um;
      while (tm_max > 1 && !fits(tm_max)) tm_max -= tm_max > 2 * um ? um : 1;
      tm_max = tm_max / Q * Q;
      if (tm_max < 1) continue;
      tm_max = std::min(tm_max, m);
      const int64_t trmin = (m + tm_max - 1) / tm_max;
      for (int64_t tr = trmin; tr <= m; tr += tr < trmin + 6 ? 1 : std::max<int64_t>(1, tr / 4)) {
        int64_t tm = std::min(m, up((m + tr - 1) / tr, um));
        if (tm > tm_max) tm = tm_max;
        const int64_t trs = (m + tm - 1) / tm;
        const int64_t T = trs * tcs;
        if (T > max_tiles) break;
        const int64_t ctas = (T + S - 1) / S;
        const int mode = ctas == 1 ? HOLD_CTA : ctas <= 16 ? HOLD_CLUSTER : HOLD_GRID;
        if (S > 1 && mode != HOLD_GRID) continue;
        if ((rag || tmem) && mode != HOLD_GRID) continue;
        if (tmem && !tmem_fits(tm, tn)) continue;
        const int64_t teams = rag ? 1 : std::min<int64_t>(d3, slots / ctas);
        if (mode == HOLD_GRID && teams > kHoldTeams) continue;
        const int64_t waves = (d3 + teams - 1) / teams;
        const int64_t conc = teams * ctas, per_sm = (conc + d.sms - 1) / d.sms;
        const double bw = std::min(tmem ? 40e9 : 60e9, 6.4e12 / (double)std::min<int64_t>(conc, d.sms)) / (double)per_sm;
        const double share = (double)S * tm * tn * E;
        // lanes left idle by tiles of a few rows more than a multiple of 32
        const int64_t N = eb < 4 ? 4 / eb : 1, wd = form != HOLD_VEC && form != HOLD_WIDE ? (tm + N - 1) / N : 32;
        const double idle = wd >= 32 ? 0.5 * (double)(up(wd, 32) - wd) / (double)wd : 0.0;
        const double ineff = idle + 2.0 + 32.0 / (double)(tn * E) + 32.0 / (double)(tm * E);
        const double bar = mode == HOLD_CTA ? 0.2e-6 : mode == HOLD_CLUSTER ? 1.2e-6 : 2.5e-6;
        const double lat = waves > 1 && S > 1 ? 1.5e-6 : 2e-6;
        const double t = tmem ? 4e-6 + waves * (1e-6 + share * ineff / bw) : waves * (lat + bar + share * ineff / bw);
        if (t < best * 0.999) {
          best = t;
          g.ok = true;
          g.tm = (uint32_t)tm;
          g.tn = (uint32_t)tn;
          g.TC = (uint32_t)tcs;
          g.T = (uint32_t)T;
          g.ctas = (uint32_t)ctas;
          g.teams = (uint32_t)teams;
          g.S = (uint32_t)S;
          g.P = (uint32_t)P;
          g.packed = packed;
          g.mode = mode;
          g.form = form;
          g.tmem = tmem;
          g.est_us = t * 1e6;
        }
      }
    }
  }
  return g.ok;
}

// Barrier slots of grid launches.  Launches on one stream run one after the
// other and share a slot.  A captured launch may be replayed on any stream and
// gets a slot of its own, given back when the graph and everything
// instantiated from it are gone.
struct HoldSlots {
  std::mutex mu;
  // by handle, with the stream's own id: a handle comes back for another
  // stream after its first one was destroyed, whose last launch may still run
  std::map<std::tuple<cudaStream_t, std::thread::id>, std::pair<unsigned long long, int>> of_stream;
  std::deque<int> free_list;     // of captured launches whose graph is gone
  std::deque<int> retired_list;  // of destroyed streams, the oldest first
  int next = 0;
  int take() {
    if (!free_list.empty()) {
      const int s = free_list.front();
      free_list.pop_front();
      return s;
    }
    if (next < kHoldSlots) return next++;
    if (retired_list.size() > kHoldSlots / 4) {  // a thousand streams have come and gone since
      const int s = retired_list.front();
      retired_list.pop_front();
      return s;
    }
    return -1;
  }
};

HoldSlots &hold_slots(int dev) {
  static std::mutex mu;
  static auto &all = *new std::map<int, HoldSlots>;  // never destroyed: graphs may outlive statics
  std::lock_guard<std::mutex> lk(mu);
  return all[dev];
}

struct HoldSlotLease {
  int dev, slot;
};

void CUDART_CB hold_slot_return(void *p) {
  auto *l = (HoldSlotLease *)p;
  HoldSlots &hs = hold_slots(l->dev);
  {
    std::lock_guard<std::mutex> lk(hs.mu);
    hs.free_list.push_back(l->slot);
  }
  delete l;
}

// -1 when no slot is left.
int hold_slot(cudaStream_t st) {
  const int dev = dev_info().id;
  HoldSlots &hs = hold_slots(dev);
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaGraph_t graph = nullptr;
  if (cudaStreamGetCaptureInfo_v2(st, &cs, nullptr, &graph, nullptr, nullptr) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  if (cs == cudaStreamCaptureStatusActive) {
    int slot;
    {
      std::lock_guard<std::mutex> lk(hs.mu);
      slot = hs.take();
    }
    if (slot < 0) return -1;
    auto *l = new HoldSlotLease{dev, slot};
    cudaUserObject_t obj = nullptr;
    if (cudaUserObjectCreate(&obj, l, hold_slot_return, 1, cudaUserObjectNoDestructorSync) != cudaSuccess) {
      cudaGetLastError();
      hold_slot_return(l);
      return -1;
    }
    if (cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove) != cudaSuccess) {
      cudaGetLastError();
      cudaUserObjectRelease(obj, 1);  // runs hold_slot_return
      return -1;
    }
    return slot;
  }
  unsigned long long id = 0;
  if (cudaStreamGetId(st, &id) != cudaSuccess) {
    cudaGetLastError();
    return -1;
  }
  std::lock_guard<std::mutex> lk(hs.mu);
  // the per-thread default stream is one handle for a stream of every thread
  const auto key = std::make_tuple(st, st == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id());
  auto it = hs.of_stream.find(key);
  if (it != hs.of_stream.end() && it->second.first == id) return it->second.second;
  const int slot = hs.take();
  if (slot < 0) return -1;
  if (it != hs.of_stream.end()) hs.retired_list.push_back(it->second.second);
  hs.of_stream[key] = {id, slot};
  return slot;
}

uint32_t *hold_bars(int *status) {
  static std::mutex mu;
  static std::map<int, uint32_t *> ptr;
  const int dev = dev_info().id;
  std::lock_guard<std::mutex> lk(mu);
  auto it = ptr.find(dev);
  if (it != ptr.end()) return it->second;
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_hold_bars);
  if (e != cudaSuccess) {
    *status = cuda_status(e, "slice barrier words");
    return nullptr;
  }
  return ptr[dev] = (uint32_t *)p;
}

}  // namespace

// Tensor memory as the second buffer, where one team takes slices that fill
// more than half of the chip one after the other.  Measured on B200, with and
// without, us: bf16 (4099, 2053, 8) 88.5 / 89.0, fp32 (3001, 2000, 4) 48.2 /
// 49.4, fp64 (2408, 1432, 4) 52.1 / 53.5, ragged fp32 (561, 62490, 2) 260 / 267
// and (7402, 10752, 1) 308 / 317.  Several teams beside each other
// already overlap, and two CTAs per SM serve them better: fp32 (1500, 1301, 8)
// 37.8 / 34.1.
void hold_try_tmem(HoldGeom &g, int64_t m, int64_t n, int eb, int64_t d3, int form, bool bands = true) {
  if (!g.ok || g.mode != HOLD_GRID || g.teams > 1 || d3 <= 1) return;
  HoldGeom t;
  if (hold_search(t, m, n, eb, 1, d3, form, true, bands) && t.tm * 4 >= std::min<uint32_t>(t.tn, 128)) g = t;
}

void hold_plan(HoldPlan &hp, int64_t m, int64_t n, int eb, int64_t we, int64_t d3) {
  hp.ready = std::make_shared<HoldReady>();
  if (we > 1) {
    hold_search(hp.any, m, n, 16, we, d3, HOLD_WIDE);
    return;
  }
  hold_search(hp.any, m, n, eb, 1, d3, HOLD_SCALAR);
  hold_try_tmem(hp.any, m, n, eb, d3, HOLD_SCALAR);
  if ((eb == 2 || eb == 4) && (n * eb) % 16 == 0 && (m * eb) % 16 == 0)
    hold_search(hp.vec, m, n, eb, 1, d3, HOLD_VEC);
}

void hold_plan_swapped(HoldPlan &hp, int64_t m, int64_t n, int eb, int64_t d3) {
  hp.ready = std::make_shared<HoldReady>();
  hold_search(hp.any, m, n, eb, 1, d3, HOLD_RAG_SRC, false, false);
  hold_try_tmem(hp.any, m, n, eb, d3, HOLD_RAG_SRC, false);
}

int64_t hold_cluster_bytes() { return 16 * hold_budget(); }

std::string describe_slice(const HoldPlan &hp) {
  const HoldGeom &g = hp.vec.ok ? hp.vec : hp.any;
  char buf[160];
  snprintf(buf, sizeof buf, "slice(%s tiles=%u of %ux%u per cta=%u ctas=%u teams=%u%s)",
           g.mode == HOLD_CTA ? "cta" : g.mode == HOLD_CLUSTER ? "cluster" : "grid", g.T, g.tm, g.tn, g.S, g.ctas,
           g.teams, g.form == HOLD_VEC ? " vec" : g.tmem ? " tmem" : "");
  return buf;
}

namespace {

void hold_args(HoldArgs &a, const HoldGeom &g, int64_t m, int64_t n, int eb, int64_t we) {
  a.slice_bytes = m * n * eb * we;
  a.m = (uint32_t)m;
  a.n = (uint32_t)n;
  a.tm = g.tm;
  a.tn = g.tn;
  a.TC = g.TC;
  a.T = g.T;
  a.ctas = g.ctas;
  a.teams = g.teams;
  a.S = g.S;
  a.P = g.P;
  a.H = (uint32_t)hold_region(g.tm, g.P, eb, g.form);
  a.packed = g.packed;
  // bulk copies from 256 bytes a row piece: one instruction a row instead of
  // one a 512 bytes (without / with, us: fp32 (3001, 2000, 4) 54.1 / 48.2, ragged
  // fp32 (1000003, 37, 1) 144 / 136); shorter pieces are many small copies
  a.bulk = !g.packed && (g.form == HOLD_SCALAR || g.form == HOLD_RAG_DST || g.form == HOLD_RAG_SRC) &&
           (int64_t)g.tn * eb >= 256;
  a.tile_bytes = (uint32_t)hold_tile_bytes(g.tm, g.tn, g.P, eb, g.form, g.packed);
  a.mode = g.mode;
  a.wait_ns = kWaitNs;
  a.need = g.ctas;
  a.we = (uint32_t)we;
  a.wediv = FastDiv<uint32_t>((uint64_t)we);
  a.tcdiv = FastDiv<uint32_t>(g.TC);
  if (g.form == HOLD_VEC) {
    a.rbdiv = FastDiv<uint32_t>((uint64_t)(g.tm / (16 / eb) + 7) / 8);
  } else if (g.form == HOLD_WIDE) {
    a.lgs = lanes_log2(g.tm * we);
  } else {
    const int N = eb < 4 ? 4 / eb : 1;
    const int64_t words = N == 1 ? g.tm : ((int64_t)g.tm + 2 * N - 2) / N;
    a.lgs = lanes_log2(words);
    a.rbdiv = FastDiv<uint32_t>((uint64_t)(words + (1 << a.lgs) - 1) >> a.lgs);
  }
}

template <int EB>
const void *hold_kernel_of(const HoldGeom &g) {
  if constexpr (EB == 2 || EB == 4)
    if (g.form == HOLD_VEC) return (const void *)k_hold<EB, HOLD_VEC>;
  if constexpr (EB == 16)
    if (g.form == HOLD_WIDE) return (const void *)k_hold<16, HOLD_WIDE>;
  switch (g.form) {
    case HOLD_SCALAR:
      return g.tmem ? (const void *)k_hold_tmem<EB, HOLD_SCALAR> : (const void *)k_hold<EB, HOLD_SCALAR>;
    case HOLD_RAG_SRC:
      return g.tmem ? (const void *)k_hold_tmem<EB, HOLD_RAG_SRC> : (const void *)k_hold<EB, HOLD_RAG_SRC>;
    case HOLD_RAG_DST:
      if constexpr (EB >= 4)
        if (g.tmem) return (const void *)k_hold_tmem<EB, HOLD_RAG_DST>;
      return (const void *)k_hold<EB, HOLD_RAG_DST>;
  }
  return nullptr;
}

const void *hold_kernel(const HoldGeom &g, int eb) {
  switch (eb) {
    case 1:
      return hold_kernel_of<1>(g);
    case 2:
      return hold_kernel_of<2>(g);
    case 4:
      return hold_kernel_of<4>(g);
    case 8:
      return hold_kernel_of<8>(g);
    case 16:
      return hold_kernel_of<16>(g);
  }
  return nullptr;
}

int hold_prepare(HoldReady::Form &f, const HoldGeom &g, int64_t m, int64_t n, int eb, int64_t we) {
  int status = T213_OK;
  f.status = device_status_word(&status);
  if (!f.status) return status;
  hold_args(f.args, g, m, n, eb, we);
  f.smem = (int64_t)g.S * f.args.tile_bytes;
  f.kern = hold_kernel(g, eb);
  if (!f.kern) {
    set_error("unsupported element size");
    return T213_ERR_UNSUPPORTED;
  }
  if (!kernel_attr_once(f.kern, f.smem, g.mode == HOLD_CLUSTER ? (int)g.ctas : 1))
    return cuda_status(cudaGetLastError(), "cudaFuncSetAttribute(slice)");
  if (g.mode == HOLD_GRID) {
    f.bars = hold_bars(&status);
    if (!f.bars) return status;
    occupancy_cached(f.kern, g.tmem ? kTmemThreads : kHoldThreads, f.smem, 1, &f.per_sm);
    f.resident = (int)g.teams;
  } else {
    occupancy_cached(f.kern, kHoldThreads, f.smem, (int)g.ctas, &f.resident);
    if (g.mode == HOLD_CTA) f.resident *= dev_info().sms;
    f.resident = std::max(1, f.resident);
  }
  return T213_OK;
}

// Teams resident at once on the SMs that the stream has.  Clusters of more
// than the portable 8 CTAs are kept to streams that have them all.
int hold_resident(const HoldReady::Form &f, const HoldGeom &g, cudaStream_t st) {
  if (g.mode == HOLD_CLUSTER && g.ctas > 8 && stream_sms(st) < dev_info().sms) return 0;
  if (g.mode != HOLD_GRID) return f.resident;
  return (int)std::min<int64_t>(f.resident, (int64_t)f.per_sm * stream_sms(st) / g.ctas);
}

int hold_enqueue(const HoldReady::Form &f, const HoldGeom &g, HoldArgs &a, char *data, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(a.teams * a.ctas, 1, 1);
  cfg.blockDim = dim3(g.tmem ? kTmemThreads : kHoldThreads, 1, 1);
  cfg.dynamicSmemBytes = (size_t)f.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  if (g.mode == HOLD_CLUSTER) {
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = g.ctas;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.numAttrs = 1;
  } else if (g.mode == HOLD_GRID) {
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.numAttrs = 1;
  }
  cfg.attrs = attr;
  uint32_t *bars = f.bars;
  int *status = f.status;
  void *args[] = {&data, &a, &bars, &status};
  const cudaError_t e = cfg.numAttrs ? cudaLaunchKernelExC(&cfg, f.kern, args)
                                     : cudaLaunchKernel(f.kern, cfg.gridDim, cfg.blockDim, args, cfg.dynamicSmemBytes, st);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return kHoldNoSlot;
  }
  return e == cudaSuccess ? T213_OK : cuda_status(e, "k_hold launch");
}

int hold_form_ready(HoldReady &r, HoldReady::Form &f, const HoldGeom &g, int64_t m, int64_t n, int eb, int64_t we) {
  if (f.ready.load(std::memory_order_acquire)) return T213_OK;
  std::lock_guard<std::mutex> lk(r.mu);
  if (f.ready.load(std::memory_order_relaxed)) return T213_OK;
  const int rc = hold_prepare(f, g, m, n, eb, we);
  if (rc == T213_OK) f.ready.store(true, std::memory_order_release);
  return rc;
}

}  // namespace

bool ragged_geometry(RaggedPlan &rp, int64_t m, int64_t n, int eb, int64_t d3) {
  rp.ok = false;
  const int64_t u = std::max(1, 16 / eb);
  const double chip = 2.0 * dev_info().sms * (double)hold_budget();
  const int64_t q0 = std::max<int64_t>(2, (int64_t)std::ceil((double)m * (double)n * eb / chip));
  // The longer side is cut; 1- and 2-byte elements, whose output words are
  // put together column by column in the row form, prefer the column form
  // while its segments are long enough for the walker (f16 (3712, 5208, 8) 391
  // us by columns, 411 by rows).
  rp.cols = n >= m || (eb < 4 && n / q0 * eb >= 3000);
  const int64_t big = rp.cols ? n : m, small = rp.cols ? m : n;
  for (int64_t q = q0; q <= q0 + q0 / 4 + 4; q++) {
    int64_t t = big / q;
    if (t >= 4 * u) t = t / u * u;  // segments of whole 16-byte blocks
    if (t * eb < 256 || (double)q * small > 4.0e6) return false;
    const int64_t r = big - q * t;
    rp.hold = HoldPlan{};
    rp.hold.ready = std::make_shared<HoldReady>();
    const int form = rp.cols ? HOLD_RAG_SRC : HOLD_RAG_DST;
    if (!hold_search(rp.hold.any, rp.cols ? m : t, rp.cols ? t : n, eb, 1, d3 * q, form)) continue;
    if (rp.cols || eb >= 4) hold_try_tmem(rp.hold.any, rp.cols ? m : t, rp.cols ? t : n, eb, d3 * q, form);
    rp.t = t;
    rp.q = q;
    rp.r = r;
    rp.small = small;
    PermSpec ps;
    ps.kind = 0;
    ps.A = rp.cols ? m : q;
    ps.Mid = 1;
    ps.C = rp.cols ? q : n;
    ps.S = q * small;
    rp.perm = ps;
    rp.ok = true;
    return true;
  }
  return false;
}

int hold_rag_ready(const RaggedPlan &rp, int eb, cudaStream_t st, int *slot) {
  HoldReady &r = *rp.hold.ready;
  const int64_t m = rp.cols ? rp.small : rp.t, n = rp.cols ? rp.t : rp.small;
  const int rc = hold_form_ready(r, r.any, rp.hold.any, m, n, eb, 1);
  if (rc) return rc;
  if (hold_resident(r.any, rp.hold.any, st) == 0) return kHoldNoSlot;
  *slot = hold_slot(st);
  return *slot < 0 ? kHoldNoSlot : T213_OK;
}

int launch_hold_rag(const RaggedPlan &rp, char *data, int64_t d3, int64_t slice_bytes, int eb, int slot,
                    cudaStream_t st) {
  const HoldReady::Form &f = rp.hold.ready->any;
  HoldArgs a = f.args;
  a.d3 = d3 * rp.q;
  a.slice_bytes = slice_bytes;
  a.teams = 1;
  a.slot = slot;
  a.nb = (uint32_t)rp.q;
  a.qdiv = FastDiv<uint32_t>((uint64_t)rp.q);
  a.seg_bytes = (uint32_t)(rp.t * eb);
  a.rest_bytes = (int32_t)(rp.r * eb);
  return hold_enqueue(f, rp.hold.any, a, data, st);
}

int launch_slice(const HoldPlan &hp, char *data, int64_t d3, int64_t m, int64_t n, int eb, int64_t we,
                 cudaStream_t st, LaunchStats *ls, int64_t h2, uint64_t stall_ns) {
  if (d3 <= 0 || m <= 0 || n <= 0) return T213_OK;
  const bool vec = hp.vec.ok && (uintptr_t)data % 16 == 0;
  const HoldGeom &g = vec ? hp.vec : hp.any;
  if (!g.ok) {
    set_error("slice does not fit the chip's shared memory");
    return T213_ERR_UNSUPPORTED;
  }
  HoldReady::Form &f = vec ? hp.ready->vec : hp.ready->any;
  {
    const int rc = hold_form_ready(*hp.ready, f, g, m, n, eb, we);
    if (rc) return rc;
  }
  HoldArgs a = f.args;
  a.d3 = d3;
  if (h2) {  // row b * h2 + a of the output order is row a * (m / h2) + b
    a.nb = 1;
    a.qdiv = FastDiv<uint32_t>((uint64_t)h2);
    a.seg_bytes = (uint32_t)(m / h2 * n * eb);
    a.rest_bytes = (int32_t)(n * eb - m * n * eb);
  }
  // persistent: as many teams as are resident at once
  a.teams = (uint32_t)std::min<int64_t>(hold_resident(f, g, st), d3);
  if (a.teams == 0) return kHoldNoSlot;  // a stream of a few of the device's SMs
  if (g.mode == HOLD_GRID) {
    a.slot = hold_slot(st);
    if (a.slot < 0) return kHoldNoSlot;
  }
  if (stall_ns) {
    if (g.mode != HOLD_GRID) {
      set_error("the slice's team has no barrier in memory");
      return T213_ERR_UNSUPPORTED;
    }
    a.wait_ns = stall_ns;
    a.need++;
  }
  const int rc = hold_enqueue(f, g, a, data, st);
  if (rc) return rc;
  if (ls) ls->launches++;
  return T213_OK;
}

// ---- rounds ------------------------------------------------------------------------
struct HoldRounds {
  RoundTensor *d_tensors = nullptr;
  RoundTile *d_tiles = nullptr;
  uint32_t *d_first = nullptr, *d_counter = nullptr;
  uint32_t rounds = 0, buf_bytes = 0, ctas = 0;
  uint32_t extra = 0;          // arrivals that no CTA makes
  uint64_t wait_ns = kWaitNs;  // limit of a wait at a round's barrier
};

namespace {

// Slices of more than this share of a round run their own plan, which has
// twice the room.  Measured on B200, shares of 0.35 / 0.5 / 0.75, us: batches
// of 64 tensors 400 / 408 / 441 (630 MB) and 749 / 752 / 752, of 512 tensors
// 6372 / 6346 / 6458.
constexpr double kRoundShare = 0.5;

// Tiles of at most `cap` bytes with the least work: bytes with their padding,
// a sector more per row piece, and idle lanes.
bool round_tiling(HoldGeom &g, int64_t m, int64_t n, int eb, int form, int64_t cap) {
  const int64_t Q = form == HOLD_VEC ? 16 / eb : 1;
  const int64_t un = std::max<int64_t>(Q, (n * eb) % 32 == 0 ? 32 / std::min(eb, 32) : 1);
  const int64_t um = std::max<int64_t>(Q, (m * eb) % 32 == 0 ? 32 / std::min(eb, 32) : 1);
  double best = 1e30;
  g.ok = false;
  for (int64_t TC = 1; TC <= n; TC = TC < 64 ? TC + 1 : TC + TC / 16) {
    const int64_t tn = std::min(n, up((n + TC - 1) / TC, un)), tcs = (n + tn - 1) / tn;
    if (tn * eb < 64 && tn < n) break;
    const bool packed = tcs == 1 && hold_packed(n, eb, form);
    const int64_t P = packed ? n * eb : hold_pitch(tn, eb, 1, form);
    auto fits = [&](int64_t tm) { return hold_tile_bytes(tm, tn, P, eb, form, packed) <= cap; };
    int64_t tm = std::min(m, std::max<int64_t>(1, cap / P));
    while (tm > 1 && !fits(tm)) tm--;
    if (!fits(tm)) continue;
    if (tm < m && tm > um) tm = tm / um * um;
    tm = tm / Q * Q;
    if (tm < 1) continue;
    const int64_t trs = (m + tm - 1) / tm;
    tm = std::min(tm, up((m + trs - 1) / trs, um));
    const int64_t N = eb < 4 ? 4 / eb : 1, wd = form == HOLD_VEC ? 32 : (tm + N - 1) / N;
    const double idle = wd >= 32 ? 0.5 * (double)(up(wd, 32) - wd) / (double)wd : 0.0;
    const double c = (double)trs * tm * tcs * tn * eb * (idle + 2.0 + 32.0 / (tn * eb) + 32.0 / (tm * eb)) +
                     (double)trs * tcs * 2048;  // a tile costs about as much as 2 KB more
    if (c < best) {
      best = c;
      g.ok = true;
      g.tm = (uint32_t)tm;
      g.tn = (uint32_t)tn;
      g.TC = (uint32_t)tcs;
      g.T = (uint32_t)(trs * tcs);
      g.ctas = g.teams = g.S = 1;
      g.P = (uint32_t)P;
      g.packed = packed;
      g.mode = HOLD_GRID;
      g.form = form;
    }
  }
  return g.ok;
}

}  // namespace

void hold_rounds_destroy(HoldRounds *r) {
  if (!r) return;
  cudaFree(r->d_tensors);
  cudaFree(r->d_tiles);
  cudaFree(r->d_first);
  cudaFree(r->d_counter);
  delete r;
}

HoldRounds *hold_rounds_create(const t213_tensor_desc *tensors, const std::vector<int> &which,
                               std::vector<int> &taken, int *status) {
  *status = T213_OK;
  taken.clear();
  const int64_t buf = hold_budget() / 2 / 128 * 128;
  const int sms = dev_info().sms;
  const uint32_t G = (uint32_t)(2 * sms);
  const int64_t smem = 2 * buf;
  if (!kernel_attr_once((const void *)k_hold_rounds, smem, 1)) {
    *status = cuda_status(cudaGetLastError(), "cudaFuncSetAttribute(rounds)");
    return nullptr;
  }
  int per_sm = 0;
  occupancy_cached((const void *)k_hold_rounds, kHoldThreads, smem, 1, &per_sm);
  if (per_sm < 2) return nullptr;
  struct Slice {
    uint32_t tensor, slice, T;
    int64_t bytes;  // of one tile's buffer space
    int64_t total;
  };
  std::vector<RoundTensor> ts;
  std::vector<Slice> slices;
  for (int i : which) {
    const t213_tensor_desc &d = tensors[i];
    const int eb = d.elem_bytes;
    const bool vec = (eb == 2 || eb == 4) && (d.d1 * eb) % 16 == 0 && (d.d2 * eb) % 16 == 0 && (uintptr_t)d.data % 16 == 0;
    const int64_t sb = d.d1 * d.d2 * eb;
    HoldGeom g;
    if (crumbs_fit(d.d2, d.d1, eb, d.d3)) continue;  // a tile each would be far too many
    // small slices take tiles of half a buffer, so that tiles of several fit
    if (d.d1 > (1 << 30) || d.d2 > (1 << 30) ||
        !round_tiling(g, d.d2, d.d1, eb, vec ? HOLD_VEC : HOLD_SCALAR, sb < (2 << 20) ? buf / 2 : buf))
      continue;
    RoundTensor t{};
    hold_args(t.a, g, d.d2, d.d1, eb, 1);
    if ((int64_t)g.T > (int64_t)G * (buf / t.a.tile_bytes)) continue;  // more tiles than a round has places
    if (sb > (int64_t)(kRoundShare * (double)G * (double)buf)) continue;
    t.data = (char *)d.data;
    t.kind = vec ? -eb : eb;
    for (int64_t k = 0; k < d.d3; k++)
      slices.push_back(Slice{(uint32_t)ts.size(), (uint32_t)k, g.T, (int64_t)t.a.tile_bytes, (int64_t)g.T * t.a.tile_bytes});
    ts.push_back(t);
    taken.push_back(i);
  }
  if (ts.empty()) return nullptr;
  // Rounds: the largest slice left opens one, smaller ones fill it; every tile
  // goes to the CTA with the least in its buffer.
  std::stable_sort(slices.begin(), slices.end(), [](const Slice &a, const Slice &b) { return a.total > b.total; });
  std::vector<RoundTile> tiles;
  std::vector<uint32_t> first;
  std::vector<std::vector<RoundTile>> mine(G);
  std::vector<int64_t> used(G);
  std::vector<char> done(slices.size(), 0);
  size_t lo = 0;
  const int64_t capacity = (int64_t)G * buf;
  while (lo < slices.size()) {
    for (uint32_t c = 0; c < G; c++) {
      mine[c].clear();
      used[c] = 0;
    }
    std::vector<std::pair<int64_t, uint32_t>> heap;  // (bytes used, CTA), least first
    for (uint32_t c = 0; c < G; c++) heap.push_back({0, c});
    auto gt = [](const std::pair<int64_t, uint32_t> &a, const std::pair<int64_t, uint32_t> &b) { return a > b; };
    std::make_heap(heap.begin(), heap.end(), gt);
    int64_t filled = 0;
    int misses = 0;
    for (size_t i = lo; i < slices.size() && misses < 16; i++) {
      if (done[i]) continue;
      const Slice &s = slices[i];
      if (filled + s.total > capacity) {
        misses++;
        continue;
      }
      // all tiles or none: the least full CTA has room for one more as long as
      // any has, so they all fit when the free places are enough
      int64_t places = 0;
      for (uint32_t c = 0; c < G && places < s.T; c++) places += (buf - used[c]) / s.bytes;
      if (places < s.T) {
        misses++;
        continue;
      }
      for (uint32_t t = 0; t < s.T; t++) {
        std::pop_heap(heap.begin(), heap.end(), gt);
        auto &top = heap.back();
        mine[top.second].push_back(RoundTile{s.tensor, s.slice, t, (uint32_t)top.first});
        top.first += s.bytes;
        used[top.second] = top.first;
        std::push_heap(heap.begin(), heap.end(), gt);
      }
      filled += s.total;
      done[i] = 1;
    }
    for (uint32_t c = 0; c < G; c++) {
      first.push_back((uint32_t)tiles.size());
      tiles.insert(tiles.end(), mine[c].begin(), mine[c].end());
    }
    const size_t was = lo;
    while (lo < slices.size() && done[lo]) lo++;
    if (lo == was) {  // cannot happen: an empty round takes every slice that was admitted
      set_error("batch rounds: a slice fits no round");
      *status = T213_ERR_UNSUPPORTED;
      return nullptr;
    }
  }
  first.push_back((uint32_t)tiles.size());
  auto *r = new HoldRounds();
  r->rounds = (uint32_t)((first.size() - 1) / G);
  r->buf_bytes = (uint32_t)buf;
  r->ctas = G;
  cudaError_t e = cudaMalloc(&r->d_tensors, ts.size() * sizeof(RoundTensor));
  if (!e) e = cudaMalloc(&r->d_tiles, tiles.size() * sizeof(RoundTile));
  if (!e) e = cudaMalloc(&r->d_first, first.size() * sizeof(uint32_t));
  if (!e) e = cudaMalloc(&r->d_counter, 256);
  if (!e) e = cudaMemcpy(r->d_tensors, ts.data(), ts.size() * sizeof(RoundTensor), cudaMemcpyHostToDevice);
  if (!e) e = cudaMemcpy(r->d_tiles, tiles.data(), tiles.size() * sizeof(RoundTile), cudaMemcpyHostToDevice);
  if (!e) e = cudaMemcpy(r->d_first, first.data(), first.size() * sizeof(uint32_t), cudaMemcpyHostToDevice);
  if (!e) e = cudaStreamSynchronize(0);  // the copies landed before any stream's launch
  if (e) {
    *status = cuda_status(e, "batch rounds");
    hold_rounds_destroy(r);
    return nullptr;
  }
  return r;
}

void hold_rounds_debug_stall(HoldRounds *r, uint64_t wait_ns) {
  r->extra = 1;
  r->wait_ns = wait_ns;
}

int hold_rounds_count(const HoldRounds *r) { return (int)r->rounds; }

int hold_rounds_launch(HoldRounds *r, int *status_word, cudaStream_t st) {
  if (2 * stream_sms(st) < (int)r->ctas) return kHoldNoSlot;  // two CTAs an SM
  cudaError_t e = cudaMemsetAsync(r->d_counter, 0, sizeof(uint32_t), st);
  if (e != cudaSuccess) return cuda_status(e, "batch rounds counter");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(r->ctas, 1, 1);
  cfg.blockDim = dim3(kHoldThreads, 1, 1);
  cfg.dynamicSmemBytes = 2 * (size_t)r->buf_bytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  e = cudaLaunchKernelEx(&cfg, k_hold_rounds, (const RoundTensor *)r->d_tensors, (const RoundTile *)r->d_tiles,
                         (const uint32_t *)r->d_first, r->rounds, r->buf_bytes, r->d_counter, r->extra, r->wait_ns,
                         status_word);
  if (e == cudaErrorCooperativeLaunchTooLarge) {
    cudaGetLastError();
    return kHoldNoSlot;
  }
  return e == cudaSuccess ? T213_OK : cuda_status(e, "k_hold_rounds launch");
}

}  // namespace t213
