// Host runtime of the in-place 213 transpose: error reporting, device
// properties, per-stream workspaces, per-pass timing, the planner, and the
// C ABI declared in include/t213.h.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <list>
#include <map>
#include <thread>
#include <tuple>

#include <cudaTypedefs.h>

#include "plan.h"

namespace t213 {

// ------------------------------------------------------------------ errors --
namespace {
thread_local std::string tl_error;
}
void set_error(const std::string &msg) { tl_error = msg; }
const std::string &last_error() { return tl_error; }
int cuda_status(cudaError_t e, const char *where) {
  set_error(std::string(where) + ": " + cudaGetErrorString(e));
  cudaGetLastError();
  return e == cudaErrorMemoryAllocation ? T213_ERR_OUT_OF_MEMORY : T213_ERR_CUDA;
}

// ------------------------------------------------------------------ device --
const DevInfo &dev_info() {
  static std::mutex mu;
  static std::map<int, DevInfo> cache;
  // asked several times by every call: the thread's last answer, which stays
  // where it is in the map, needs no lock
  thread_local const DevInfo *last = nullptr;
  int dev = 0;
  cudaGetDevice(&dev);
  if (last && last->id == dev) return *last;
  std::lock_guard<std::mutex> lk(mu);
  auto it = cache.find(dev);
  if (it != cache.end()) return *(last = &it->second);
  DevInfo d;
  d.id = dev;
  int v = 0;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess) d.sms = v;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) == cudaSuccess) d.smem_optin = v;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) == cudaSuccess) d.smem_per_sm = v;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxThreadsPerMultiProcessor, dev) == cudaSuccess) d.max_threads_sm = v;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrComputeCapabilityMajor, dev) == cudaSuccess) d.cc_major = v;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrComputeCapabilityMinor, dev) == cudaSuccess) d.cc_minor = v;
  if (cudaDeviceGetAttribute(&v, cudaDevAttrL2CacheSize, dev) == cudaSuccess) d.l2_bytes = v;
  cudaGetLastError();
  return cache.emplace(dev, d).first->second;
}

// Through the runtime's driver entry point (no link against libcuda).
int stream_sms(cudaStream_t st) {
  struct Entry {
    PFN_cuStreamGetCtx_v12050 ctx = nullptr;
    PFN_cuGreenCtxGetDevResource_v12040 resource = nullptr;
  };
  static const Entry fn = [] {
    Entry e;
    cudaDriverEntryPointQueryResult q = cudaDriverEntryPointSymbolNotFound;
    void *p = nullptr, *r = nullptr;
    if (cudaGetDriverEntryPointByVersion("cuStreamGetCtx", &p, 12050, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess &&
        cudaGetDriverEntryPointByVersion("cuGreenCtxGetDevResource", &r, 12040, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess) {
      e.ctx = (PFN_cuStreamGetCtx_v12050)p;
      e.resource = (PFN_cuGreenCtxGetDevResource_v12040)r;
    }
    cudaGetLastError();
    return e;
  }();
  if (!fn.ctx) return dev_info().sms;  // a driver without green contexts
  CUcontext c = nullptr;
  CUgreenCtx g = nullptr;
  if (fn.ctx((CUstream)st, &c, &g) != CUDA_SUCCESS) return 0;
  if (!g) return dev_info().sms;
  CUdevResource r = {};
  return fn.resource(g, &r, CU_DEV_RESOURCE_TYPE_SM) == CUDA_SUCCESS ? (int)r.sm.smCount : 0;
}

// --------------------------------------------------------------- workspace --
namespace {
std::mutex g_ws_mu;
// Streams by device and handle, the per-thread default stream also by thread.
using StreamKey = std::tuple<int, cudaStream_t, std::thread::id>;
StreamKey stream_key(int dev, cudaStream_t st) {
  return {dev, st, st == cudaStreamPerThread ? std::this_thread::get_id() : std::thread::id()};
}
}  // namespace

struct Workspace {
  char *p = nullptr;
  size_t bytes = 0;
  // A handle, or a thread's id, comes back for another stream after its first
  // one was destroyed, whose last use of the buffer may still run: the new
  // stream then waits for `last`.
  unsigned long long id = 0;
  cudaEvent_t last = nullptr;
};

namespace {
std::map<StreamKey, Workspace> g_ws;

void free_workspace(Workspace &w) {
  if (w.last) {
    cudaEventSynchronize(w.last);
    cudaEventDestroy(w.last);
  }
  if (w.p) cudaFree(w.p);
}
}  // namespace

CaptureRelaxed::CaptureRelaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }
CaptureRelaxed::~CaptureRelaxed() { cudaThreadExchangeStreamCaptureMode(&mode); }

bool capturing(cudaStream_t st, cudaGraph_t *graph, unsigned long long *id) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamGetCaptureInfo_v2(st, &cs, id, graph, nullptr, nullptr) != cudaSuccess) {
    cudaGetLastError();  // the legacy stream while another one captures
    return false;
  }
  return cs == cudaStreamCaptureStatusActive;
}

namespace {
// What graphs that are gone have kept.  Their callbacks may make no CUDA call,
// so it is let go by a later call outside a capture, or a buffer is taken by
// a later capture.
struct Graveyard {
  std::mutex mu;
  std::vector<std::shared_ptr<void>> kept;
  std::vector<std::shared_ptr<GraphBuffer>> buffers;
  std::atomic<bool> any{false};
};
Graveyard &graveyard() {
  static auto &g = *new Graveyard;  // never destroyed: graphs may outlive statics
  return g;
}

struct Kept {
  std::shared_ptr<void> what;
  std::shared_ptr<GraphBuffer> buffer;
};

void CUDART_CB graph_gone(void *p) {
  auto *k = (Kept *)p;
  Graveyard &g = graveyard();
  {
    std::lock_guard<std::mutex> lk(g.mu);
    if (k->what) g.kept.push_back(std::move(k->what));
    if (k->buffer) g.buffers.push_back(std::move(k->buffer));
    g.any.store(true, std::memory_order_release);
  }
  delete k;
}

int keep(cudaGraph_t graph, Kept what) {
  auto *k = new Kept(std::move(what));
  cudaUserObject_t obj = nullptr;
  cudaError_t e = cudaUserObjectCreate(&obj, k, graph_gone, 1, cudaUserObjectNoDestructorSync);
  if (e != cudaSuccess) {
    graph_gone(k);
    return cuda_status(e, "cudaUserObjectCreate");
  }
  e = cudaGraphRetainUserObject(graph, obj, 1, cudaGraphUserObjectMove);
  if (e != cudaSuccess) {
    cudaUserObjectRelease(obj, 1);  // runs graph_gone
    return cuda_status(e, "cudaGraphRetainUserObject");
  }
  return T213_OK;
}

// Buffers of captures in progress: of a stream's newest capture, by its id.
struct CapturedBuffer {
  unsigned long long id;
  char *p;
  size_t bytes;
};
std::map<StreamKey, CapturedBuffer> g_captured;

// A captured call's scratch belongs to the graph: a replay may run beside the
// stream's own calls, and long after the stream's workspace has moved.  The
// calls captured on one stream run in order and share one.
char *captured_workspace(cudaStream_t st, cudaGraph_t graph, unsigned long long id, size_t bytes, int *status) {
  const int dev = dev_info().id;
  std::lock_guard<std::mutex> lk(g_ws_mu);
  auto it = g_captured.find(stream_key(dev, st));
  if (it != g_captured.end() && it->second.id == id && it->second.bytes >= bytes) return it->second.p;
  std::shared_ptr<GraphBuffer> b;
  {
    Graveyard &g = graveyard();
    std::lock_guard<std::mutex> lk2(g.mu);
    for (auto &old : g.buffers)
      if (old->dev == dev && old->bytes >= bytes) {
        b = std::move(old);
        old = std::move(g.buffers.back());
        g.buffers.pop_back();
        break;
      }
  }
  if (!b) {
    b = std::make_shared<GraphBuffer>();
    b->dev = dev;
    b->bytes = (bytes + 255) & ~(size_t)255;
    CaptureRelaxed relaxed;
    cudaError_t e = cudaMalloc(&b->p, b->bytes);
    if (e != cudaSuccess) {
      *status = cuda_status(e, "workspace cudaMalloc");
      return nullptr;
    }
  }
  const CapturedBuffer c{id, b->p, b->bytes};
  if ((*status = keep(graph, Kept{nullptr, std::move(b)}))) return nullptr;
  g_captured[stream_key(dev, st)] = c;
  return c.p;
}
}  // namespace

GraphBuffer::~GraphBuffer() {
  if (p) cudaFree(p);  // its graph and every launch of it are gone
}

int keep_with_graph(cudaGraph_t graph, std::shared_ptr<void> what) { return keep(graph, Kept{std::move(what), nullptr}); }

void release_kept() {
  Graveyard &g = graveyard();
  if (!g.any.load(std::memory_order_acquire)) return;
  // another thread may be capturing: a free in this one's default mode would
  // invalidate its capture
  CaptureRelaxed relaxed;
  std::vector<std::shared_ptr<void>> kept;
  std::vector<std::shared_ptr<GraphBuffer>> buffers;
  {
    std::lock_guard<std::mutex> lk(g.mu);
    kept.swap(g.kept);
    buffers.swap(g.buffers);
    g.any.store(false, std::memory_order_release);
  }
}

static std::mutex &g_enqueue_mu = *new std::mutex;  // never destroyed: threads may outlive statics

WorkspaceUse::WorkspaceUse() : lk(g_enqueue_mu) {}

WorkspaceUse::~WorkspaceUse() {
  if (w && cudaEventRecord(w->last, st) != cudaSuccess) cudaGetLastError();  // the launches before it report
}

char *workspace(WorkspaceUse &use, cudaStream_t st, size_t bytes, int *status) {
  const int dev = dev_info().id;
  cudaGraph_t graph = nullptr;
  unsigned long long id = 0;
  if (capturing(st, &graph, &id)) return captured_workspace(st, graph, id, bytes, status);
  release_kept();
  std::lock_guard<std::mutex> lk(g_ws_mu);
  auto &w = g_ws[stream_key(dev, st)];
  cudaError_t e = cudaStreamGetId(st, &id);
  if (e == cudaSuccess && !w.last) e = cudaEventCreateWithFlags(&w.last, cudaEventDisableTiming);
  if (e == cudaSuccess && w.p && w.id != id) e = cudaStreamWaitEvent(st, w.last, 0);
  if (e != cudaSuccess) {
    *status = cuda_status(e, "workspace");
    return nullptr;
  }
  w.id = id;
  use.w = &w;
  use.st = st;
  if (w.p && w.bytes >= bytes) return w.p;
  if (w.p) {
    // cudaFree does not promise to wait for kernels in flight: finish the
    // buffer's last use first
    cudaEventSynchronize(w.last);
    cudaFree(w.p);
    w.p = nullptr;
    w.bytes = 0;
  }
  size_t want = std::max<size_t>(bytes, (size_t)1 << 20);
  want = (want + ((size_t)1 << 20) - 1) & ~(((size_t)1 << 20) - 1);
  e = cudaMalloc(&w.p, want);
  if (e != cudaSuccess) {
    w.p = nullptr;
    *status = cuda_status(e, "workspace cudaMalloc");
    return nullptr;
  }
  w.bytes = want;
  return w.p;
}

// A variable of the module rather than an allocation: it is zero from the
// start, and a first call inside a stream capture may take its address.
__device__ int g_status_word[64];

int *device_status_word(int *status) {
  static std::mutex mu;
  static std::map<int, int *> words;
  const int dev = dev_info().id;
  std::lock_guard<std::mutex> lk(mu);
  auto it = words.find(dev);
  if (it != words.end()) return it->second;
  void *p = nullptr;
  cudaError_t e = cudaGetSymbolAddress(&p, g_status_word);
  if (e != cudaSuccess) {
    *status = cuda_status(e, "status word");
    return nullptr;
  }
  return words[dev] = (int *)p;
}

void release_stream_workspace(cudaStream_t st) {
  const int dev = dev_info().id;
  std::lock_guard<std::mutex> users(g_enqueue_mu), lk(g_ws_mu);
  g_captured.erase(stream_key(dev, st));
  auto it = g_ws.find(stream_key(dev, st));
  if (it == g_ws.end()) return;
  free_workspace(it->second);
  g_ws.erase(it);
}

static void release_workspaces() {
  const int dev = dev_info().id;
  std::lock_guard<std::mutex> users(g_enqueue_mu), lk(g_ws_mu);
  for (auto it = g_ws.begin(); it != g_ws.end();) {
    if (std::get<0>(it->first) == dev) {
      free_workspace(it->second);
      it = g_ws.erase(it);
    } else {
      ++it;
    }
  }
}

// ----------------------------------------------------------- launch cache --
namespace {
std::mutex g_lc_mu;
std::map<std::tuple<const void *, int64_t, int, int>, int> g_attr_done;
std::map<std::tuple<const void *, int, int64_t, int, int>, int> g_occ;
}  // namespace

bool kernel_attr_once(const void *kern, int64_t smem, int cluster) {
  // The dynamic shared-memory attribute is an upper bound: raise it when a
  // launch needs more than any earlier one, never lower it.
  const int dev = dev_info().id;
  std::lock_guard<std::mutex> lk(g_lc_mu);
  auto key = std::make_tuple(kern, (int64_t)0, 0, dev);
  auto it = g_attr_done.find(key);
  const int64_t have = it == g_attr_done.end() ? -1 : it->second;
  if (smem > have) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return false;
    g_attr_done[key] = (int)smem;
  }
  if (cluster > 8) {
    auto ck = std::make_tuple(kern, (int64_t)1, 1, dev);
    if (!g_attr_done.count(ck)) {
      if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) return false;
      g_attr_done[ck] = 1;
    }
  }
  return true;
}

int occupancy_cached(const void *kern, int threads, int64_t smem, int cluster, int *out) {
  const int dev = dev_info().id;
  {
    std::lock_guard<std::mutex> lk(g_lc_mu);
    auto it = g_occ.find(std::make_tuple(kern, threads, smem, cluster, dev));
    if (it != g_occ.end()) {
      *out = it->second;
      return T213_OK;
    }
  }
  int v = 0;
  if (cluster <= 1) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&v, kern, threads, (size_t)smem) != cudaSuccess || v < 1) {
      cudaGetLastError();
      v = 1;
    }
  } else {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(cluster * 8), 1, 1);
    cfg.blockDim = dim3(threads, 1, 1);
    cfg.dynamicSmemBytes = (size_t)smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&v, kern, &cfg) != cudaSuccess || v < 1) {
      cudaGetLastError();
      v = std::max(1, dev_info().sms / cluster);
    }
  }
  std::lock_guard<std::mutex> lk(g_lc_mu);
  g_occ[std::make_tuple(kern, threads, smem, cluster, dev)] = v;
  *out = v;
  return T213_OK;
}

// ------------------------------------------------------------------ timing --
namespace {
std::atomic<bool> g_timing{false};
std::mutex g_tmu;
struct TimingRec {
  std::vector<std::pair<cudaEvent_t, cudaEvent_t>> pending;
  double total_ms = 0;
  int64_t launches = 0;
};
std::map<std::string, TimingRec> g_trec;
}  // namespace

bool pass_timing_on() { return g_timing.load(); }

PassTimer::PassTimer(const char *n, cudaStream_t s) : name(n), st(s) {
  if (!g_timing.load()) return;
  if (cudaEventCreate(&a) != cudaSuccess || cudaEventCreate(&b) != cudaSuccess) {
    a = b = nullptr;
    cudaGetLastError();
    return;
  }
  cudaEventRecord(a, st);
}

PassTimer::~PassTimer() {
  if (!a) return;
  cudaEventRecord(b, st);
  std::lock_guard<std::mutex> lk(g_tmu);
  g_trec[name].pending.push_back({a, b});
}

// ---------------------------------------------------------------- planning --
int64_t ext_gcd(int64_t a, int64_t b, int64_t *mmi) {
  // gcd and the inverse of a modulo b (0 if gcd != 1), extended Euclid
  int64_t x = 0, lastx = 1, origb = b;
  while (b != 0) {
    int64_t q = a / b, nb = a % b;
    a = b;
    b = nb;
    int64_t nx = lastx - q * x;
    lastx = x;
    x = nx;
  }
  if (mmi) *mmi = (a == 1) ? (lastx < 0 ? lastx + origb : lastx) : 0;
  return a;
}

const char *PassDesc::name() const {
  switch (type) {
    case PT_COL:
      return "col_gather";
    case PT_ROW:
      return "row_gather";
    case PT_SEG:
      return "segment_cycles";
    case PT_TILE:
      return "tile_swap";
    case PT_BAND:
      return "band_transpose";
    case PT_SLICE:
      return "slice";
    case PT_RAGGED:
      return "ragged";
    case PT_CRUMBS:
      return "crumbs";
  }
  return "?";
}

namespace {

PassDesc col_pass(int kind, std::initializer_list<int64_t> prm, int64_t m, int64_t n) {
  PassDesc p;
  p.type = PT_COL;
  p.fn.kind = kind;
  int q = 0;
  for (int64_t v : prm) p.fn.p[q++] = v;
  p.m = m;
  p.n = n;
  return p;
}

PassDesc row_pass(int kind, std::initializer_list<int64_t> prm, int64_t m, int64_t n) {
  PassDesc p = col_pass(kind, prm, m, n);
  p.type = PT_ROW;
  return p;
}

// Items per chunk for the walker: pieces of a segment (16-byte words, team of
// up to 256 threads) times slices.
int64_t items_per_chunk(int64_t seg_bytes, int64_t d3) {
  int team = seg_cycles_team(seg_bytes, 16);
  int64_t words = std::max<int64_t>(1, seg_bytes / 16);
  return std::max<int64_t>(1, (words + team - 1) / team) * std::max<int64_t>(1, d3);
}

int add_seg_pass(Plan &P, const PermSpec &ps, int64_t seg_bytes, bool skip_identity) {
  int st = T213_OK;
  PassDesc p;
  p.type = PT_SEG;
  p.perm = ps;
  p.seg_bytes = seg_bytes;
  p.table = get_cycle_table(ps, items_per_chunk(seg_bytes, P.d3), &st);
  if (!p.table) return st;
  if (skip_identity && p.table->n_chunks == 0) return T213_OK;
  P.passes.push_back(p);
  return T213_OK;
}

// Fraction of the copy bandwidth a segment-cycle pass reaches, by segment
// size (bulk-copy walker from 1 KB up, register walker below).
double seg_eff(int64_t seg_bytes) {
  if (seg_bytes >= 4096) return 0.88;
  if (seg_bytes >= 1024) return 0.8;
  if (seg_bytes >= 512) return 0.65;  // bulk walker when 16-byte aligned: 0.72 at 704 B
  if (seg_bytes >= 256) return 0.5;   // 0.61 at 480 B
  if (seg_bytes >= 128) return 0.3;
  if (seg_bytes >= 64) return 0.18;
  return 0.08;
}

std::string fmt_plan(const Plan &P) {
  VariantScope vs(P.var);  // the pass descriptions show the kernels this plan's variant picks
  static const char *kn[] = {"auto", "c2r", "r2c", "skinny", "blocks", "bands", "bands_t", "identity", "slice", "ragged", "crumbs"};
  std::string s = kn[P.kind >= 0 && P.kind <= kPlanCrumbs ? P.kind : 0];
  char buf[256];
  if (P.t) {
    snprintf(buf, sizeof buf, " t=%lld", (long long)P.t);
    s += buf;
  }
  s += ":";
  for (const PassDesc &p : P.passes) {
    s += " ";
    switch (p.type) {
      case PT_COL:
        {
          const std::string d = describe_col_gather_fn(p.fn, p.m, p.n, P.eb, nullptr);
          snprintf(buf, sizeof buf, "%s(fn=%d)%s", d.substr(0, d.find('[')).c_str(), p.fn.kind,
                   d.substr(d.find('[')).c_str());
        }
        break;
      case PT_ROW:
        snprintf(buf, sizeof buf, "row_gather(fn=%d)%s", p.fn.kind, describe_row_gather(p.m, p.n, P.eb, nullptr).substr(10).c_str());
        break;
      case PT_SLICE:
        snprintf(buf, sizeof buf, "%s", describe_slice(p.hold).c_str());
        break;
      case PT_CRUMBS:
        snprintf(buf, sizeof buf, "crumbs(%lldB)", (long long)(p.m * p.n * P.eb));
        break;
      case PT_RAGGED:
        snprintf(buf, sizeof buf, "%s(q=%lld r=%lld seg=%lldB chunks=%lld carry=%lld) %s", p.ragged.cols ? "cols" : "rows",
                 (long long)p.ragged.q, (long long)p.ragged.r, (long long)(p.ragged.t * P.eb),
                 (long long)p.ragged.table->n_chunks, (long long)p.ragged.table->n_carry,
                 describe_slice(p.ragged.hold).c_str());
        break;
      case PT_SEG:
        snprintf(buf, sizeof buf, "segment_cycles(S=%lld seg=%lldB cycles=%lld chunks=%lld carry=%lld maxlen=%lld)",
                 (long long)p.perm.S, (long long)p.seg_bytes, (long long)p.table->n_cycles,
                 (long long)p.table->n_chunks, (long long)p.table->n_carry, (long long)p.table->max_len);
        break;
      case PT_TILE:
        snprintf(buf, sizeof buf, "tile_swap(t=%lld)", (long long)p.t);
        break;
      case PT_BAND:
        snprintf(buf, sizeof buf, "band_transpose(%lldx%lld)", (long long)p.R, (long long)p.C);
        break;
    }
    s += buf;
  }
  return s;
}

// C2R on an m x n slice (m = d2 rows, n = d1 columns): src/transpose.cu:30-47
// and src/skinny.cu:313-333.  The column op is always the fused column
// shuffle: on B200 a 32-column strip of any realistic height fits a thread-
// block cluster's shared memory, which replaces the reference's 48 KB switch
// to post-rotation + row scatter.
void c2r_passes(Plan &P, int64_t m, int64_t n, bool skinny) {
  int64_t t, c = ext_gcd(m, n, &t), k;
  if (c > 1)
    ext_gcd(m / c, n / c, &k);
  else
    k = t;
  if (c > 1) {
    if (skinny)
      P.passes.push_back(col_pass(T213_FN_C2R_FUSED_PREOP, {m, n / c}, m, n));
    else
      P.passes.push_back(col_pass(T213_FN_C2R_PREROTATOR, {n / c}, m, n));
  }
  P.passes.push_back(row_pass(skinny ? T213_FN_C2R_LONG_SHUFFLE : T213_FN_C2R_SHUFFLE, {m, n, c, k}, m, n));
  P.passes.push_back(col_pass(T213_FN_C2R_FUSED_POSTOP, {m, n, c}, m, n));
}

// R2C with the passes on the m x n output view: src/transpose.cu:58-89,
// src/skinny.cu:344-363.
void r2c_passes(Plan &P, int64_t m, int64_t n, bool skinny) {
  int64_t t, c = ext_gcd(n, m, &t), q;
  if (c > 1)
    ext_gcd(n / c, m / c, &q);
  else
    q = t;
  P.passes.push_back(col_pass(T213_FN_R2C_FUSED_PREOP, {m / c, c, m, q}, m, n));
  P.passes.push_back(row_pass(T213_FN_R2C_SHUFFLE, {m, n, c, 0}, m, n));
  if (c > 1) {
    if (skinny)
      P.passes.push_back(col_pass(T213_FN_R2C_FUSED_POSTOP, {m, n / c}, m, n));
    else
      P.passes.push_back(col_pass(T213_FN_R2C_POSTROTATOR, {n / c, m}, m, n));
  }
}

// Fraction of the copy rate a gather pass reaches, by variant, from B200
// measurements: cluster-local column strips 0.5-0.64, staged column strips
// 0.3-0.45, DSMEM-clustered columns about 0.25; staged rows 0.6-0.8.  Rows
// longer than shared memory, gathered from a global scratch copy, about 0.17
// (DSMEM-clustered rows 0.06); columns taller than a 16-CTA cluster, from a
// scratch copy, about 0.06 (C2R on (344, 359054, 4) fp32).
double gather_cost(const PassDesc &p, int eb) {
  if (p.type == PT_COL) {
    std::string d = describe_col_gather_fn(p.fn, p.m, p.n, eb, nullptr);
    if (d.find("[local") != std::string::npos) return 1 / 0.6;
    if (d.find("scratch") != std::string::npos) return 1 / 0.06;
    if (d.find("cluster=1 ") != std::string::npos) return 1 / 0.4;
    return 1 / 0.25;
  }
  std::string d = describe_row_gather(p.m, p.n, eb, nullptr);
  if (d.find("scratch") != std::string::npos) return 1 / 0.17;
  if (d.find("cluster") != std::string::npos) return 1 / 0.06;
  return 1 / 0.65;
}

int64_t largest_divisor_le(int64_t x, int64_t limit) {
  // largest divisor of x that is <= limit
  int64_t best = 1;
  for (int64_t f = 1; f * f <= x; f++) {
    if (x % f) continue;
    if (f <= limit) best = std::max(best, f);
    if (x / f <= limit) best = std::max(best, x / f);
  }
  return best;
}

// Candidate block / band sizes.
int64_t pick_block_t(int64_t m, int64_t n) { return ext_gcd(m, n, nullptr); }
int64_t pick_band_t(int64_t m, int64_t n, int eb) {
  // t | m, band t x n fits shared memory; a whole slice up to 96 KB is one band
  if (band_smem_bytes(m, n, eb) <= 96 * 1024) return m;
  int64_t per_row = band_smem_bytes(1, n, eb);
  if (per_row > band_smem_limit()) return 0;
  return largest_divisor_le(m, band_smem_limit() / per_row);
}
int64_t pick_band_t_t(int64_t m, int64_t n, int eb) {
  // t | n, band m x t fits shared memory
  int64_t lim = band_smem_limit() / std::max<int64_t>(1, m * eb);
  if (lim < 1) return 0;
  return largest_divisor_le(n, lim);
}

// Fraction of the copy bandwidth the square-block tile pass reaches (measured
// on (8192, 6144, d3) blocks of t = 2048): the TMA kernel's 64-wide fp32
// tiles 0.91, the register kernel's 32-wide tiles 0.90 (8-byte) and 0.93
// (16-byte) but 0.72 for 4-byte elements, whose 32-wide rows are only 128
// bytes; the element-wise kernel about 0.35.
double tile_eff(int64_t t, int eb) {
  if (eb == 4 && t % 64 == 0) return 0.91;
  if ((eb == 8 || eb == 16) && t % 32 == 0) return 0.9;
  if (eb == 4 && t % 32 == 0) return 0.72;
  return 0.35;
}

int build_plan(Plan &P, int kind, int64_t t) {
  const int64_t d1 = P.d1, d2 = P.d2, d3 = P.d3;
  const int eb = P.eb;
  const int64_t m = d2, n = d1;
  P.kind = kind;
  P.t = 0;
  P.passes.clear();
  switch (kind) {
    case T213_PLAN_IDENTITY:
      if (d1 != 1 && d2 != 1) {
        set_error("identity plan needs d1 == 1 or d2 == 1");
        return T213_ERR_UNSUPPORTED;
      }
      return T213_OK;
    case T213_PLAN_C2R:
      c2r_passes(P, m, n, false);
      return T213_OK;
    case T213_PLAN_R2C:
      r2c_passes(P, d1, d2, false);  // output view: d1 rows x d2 columns
      return T213_OK;
    case T213_PLAN_SKINNY:
      if (d2 <= 32 && d2 < d1) {
        c2r_passes(P, m, n, true);
        return T213_OK;
      }
      if (d1 <= 32) {
        r2c_passes(P, d1, d2, true);
        return T213_OK;
      }
      set_error("skinny plan needs min(d1,d2) <= 32");
      return T213_ERR_UNSUPPORTED;
    case T213_PLAN_BLOCKS: {
      if (t <= 0) t = pick_block_t(m, n);
      if (m % t || n % t) {
        set_error("block size must divide gcd(d1,d2)");
        return T213_ERR_UNSUPPORTED;
      }
      P.t = t;
      PassDesc tp;
      tp.type = PT_TILE;
      tp.t = t;
      tp.m = m;
      tp.n = n;
      P.passes.push_back(tp);
      PermSpec ps;
      ps.kind = 0;
      ps.A = m / t;
      ps.Mid = t;
      ps.C = n / t;
      ps.S = m * n / t;
      if (ps.A == 1 && ps.C == 1) return T213_OK;
      return add_seg_pass(P, ps, t * eb, true);
    }
    case T213_PLAN_BANDS: {
      if (t <= 0) t = pick_band_t(m, n, eb);
      if (t <= 0 || m % t || !band_fits(t, n, eb)) {
        set_error("band size must divide d2 and a t x d1 band must fit shared memory");
        return T213_ERR_UNSUPPORTED;
      }
      P.t = t;
      PassDesc bp;
      bp.type = PT_BAND;
      bp.R = t;
      bp.C = n;
      bp.bands = m / t;
      P.passes.push_back(bp);
      PermSpec ps;
      ps.kind = 0;
      ps.A = m / t;
      ps.Mid = 1;
      ps.C = n;
      ps.S = (m / t) * n;
      return add_seg_pass(P, ps, t * eb, true);
    }
    case T213_PLAN_SLICE: {
      PassDesc sp;
      sp.type = PT_SLICE;
      sp.m = m;
      sp.n = n;
      if (m >= 2 && n >= 2 && m <= (1 << 30) && n <= (1 << 30)) hold_plan(sp.hold, m, n, eb, 1, d3);
      if (!sp.hold.any.ok) {
        set_error("slice plan needs a slice that fits the chip's shared memory");
        return T213_ERR_UNSUPPORTED;
      }
      P.passes.push_back(sp);
      return T213_OK;
    }
    case kPlanCrumbs: {
      if (!crumbs_fit(m, n, eb, d3)) return T213_ERR_UNSUPPORTED;
      PassDesc cp;
      cp.type = PT_CRUMBS;
      cp.m = m;
      cp.n = n;
      P.passes.push_back(cp);
      return T213_OK;
    }
    case kPlanRagged: {
      PassDesc rp;
      rp.type = PT_RAGGED;
      rp.m = m;
      rp.n = n;
      if (!ragged_geometry(rp.ragged, m, n, eb, d3)) {
        set_error("no bands of this slice fit the chip");
        return T213_ERR_UNSUPPORTED;
      }
      const int st = ragged_table(rp.ragged, eb, d3);
      if (st) return st;
      P.t = rp.ragged.t;
      P.passes.push_back(rp);
      return T213_OK;
    }
    case T213_PLAN_BANDS_T: {
      if (t <= 0) t = pick_band_t_t(m, n, eb);
      if (t <= 0 || n % t || !band_fits(m, t, eb)) {
        set_error("band size must divide d1 and a d2 x t band must fit shared memory");
        return T213_ERR_UNSUPPORTED;
      }
      P.t = t;
      PermSpec ps;
      ps.kind = 0;
      ps.A = m;
      ps.Mid = 1;
      ps.C = n / t;
      ps.S = m * (n / t);
      int st = add_seg_pass(P, ps, t * eb, true);
      if (st) return st;
      PassDesc bp;
      bp.type = PT_BAND;
      bp.R = m;
      bp.C = t;
      bp.bands = n / t;
      P.passes.push_back(bp);
      return T213_OK;
    }
  }
  set_error("unknown plan kind");
  return T213_ERR_INVALID_ARGUMENT;
}

// Bytes of the column strips that a plan gathers.
int64_t col_strip_bytes(const Plan &P) {
  int64_t w = 1 << 20;
  for (const PassDesc &p : P.passes)
    if (p.type == PT_COL) w = std::min(w, col_strip_width(p.fn, p.m, p.n, P.eb) * P.eb);
  return w;
}

// The ragged bands, in the units of the other estimates.  Measured on slices
// larger than the chip (B200, times over that of one copy of the tensor, the
// other plan / ragged, fp32 unless said): two gathers over 128-byte strips
// 2.5-3.2 / 2.6-3.5, three gathers 4.0-5.6 / 2.8-3.8, narrower strips 5.5-8 /
// 3.1-3.6, 1- and 2-byte gathers 6-40 / 3.5-5.9, rows or columns through
// scratch 12-28 / 2.5-3.6; bands of aligned segments from 448 bytes 1.9-2.8 /
// 2.6-4.8, unaligned ones 7.4 / 3.5 (8-byte elements 3.4 / 4.0), blocks of odd
// sides 5.8 / 2.6.
constexpr double kRaggedCost = 3.6;

double plan_cost(const Plan &P) {
  double c = 0;
  for (const PassDesc &p : P.passes) {
    switch (p.type) {
      case PT_COL:
      case PT_ROW:
        c += gather_cost(p, P.eb);
        break;
      case PT_SEG: {
        c += 1.0 / seg_eff(p.seg_bytes) * (double)p.table->moved / std::max<int64_t>(1, p.perm.S);
        break;
      }
      case PT_TILE:
        c += 1 / tile_eff(p.t, P.eb);
        break;
      case PT_BAND:
        c += 1 / 0.5;
        break;
      case PT_SLICE:
      case PT_CRUMBS:
        c += 1 / 0.6;
        break;
      case PT_RAGGED:
        c += kRaggedCost;
        break;
    }
  }
  return c;
}

// The cost of a C2R, R2C or skinny plan where the ragged bands are the
// alternative: 1- and 2-byte elements and narrow strips count double.
double gather_plan_cost(const Plan &P) {
  const double c = plan_cost(P);
  return P.eb < 4 || col_strip_bytes(P) < 128 ? 2 * c : c;
}

// Cheap estimate used to rank candidates before any cycle table is built.
double estimate_cost(int kind, int64_t m, int64_t n, int64_t t, int eb, int64_t d3) {
  (void)d3;
  const double S_limit = 4.0e6;  // first-call host cycle walk stays around 20 ms
  switch (kind) {
    case T213_PLAN_BLOCKS: {
      if (t <= 0 || t * eb < 16) return 1e9;
      const double tile = 1 / tile_eff(t, eb);
      if (m == n && m == t) return tile;
      double S = (double)m * (double)n / (double)t;
      if (S > S_limit) return 1e9;
      return tile + 1 / seg_eff(t * eb);
    }
    case T213_PLAN_BANDS:
    case T213_PLAN_BANDS_T: {
      if (t <= 0 || t * eb < 32) return 1e9;
      double S = (double)m * (double)n / (double)t;
      if (S > S_limit) return 1e9;
      if ((kind == T213_PLAN_BANDS && t == m) || (kind == T213_PLAN_BANDS_T && t == n)) return 1 / 0.5;
      return 1 / 0.5 + 1 / seg_eff(t * eb);
    }
  }
  return 1e9;
}

struct PlanKey {
  int64_t d1, d2, d3;
  int eb, kind;
  int64_t t;
  int dev;
  int var = 0;  // Variant::packed()
  bool operator<(const PlanKey &o) const {
    return std::tie(d1, d2, d3, eb, kind, t, dev, var) < std::tie(o.d1, o.d2, o.d3, o.eb, o.kind, o.t, o.dev, o.var);
  }
};

// LRU cache of plans (front = most recently used).  Evicting a plan can drop
// the last reference to its cycle tables; their device memory is then freed
// only after a device-wide synchronisation (see CycleTable).
// Heap objects that are never destroyed: at process exit the plans (and the
// CUDA resources of their cycle tables) are left to the driver's teardown
// instead of being released by static destructors in an unspecified order.
std::mutex &g_plan_mu = *new std::mutex;
auto &g_plan_lru = *new std::list<std::pair<PlanKey, std::shared_ptr<Plan>>>;
auto &g_plans = *new std::map<PlanKey, std::list<std::pair<PlanKey, std::shared_ptr<Plan>>>::iterator>;
constexpr size_t kPlanCacheMax = 1024;

std::shared_ptr<Plan> new_plan(int64_t d1, int64_t d2, int64_t d3, int eb) {
  auto P = std::make_shared<Plan>();
  P->d1 = d1;
  P->d2 = d2;
  P->d3 = d3;
  P->eb = eb;
  return P;
}

}  // namespace

int tuner_lookup_internal(int64_t d1, int64_t d2, int64_t d3, int eb, int *kind, int64_t *t, Variant *v);

std::shared_ptr<Plan> get_plan_variant(int64_t d1, int64_t d2, int64_t d3, int eb, int kind, int64_t t,
                                       const Variant &v, int *status) {
  std::shared_ptr<Plan> base = get_plan(d1, d2, d3, eb, kind, t, status);
  if (!base || !v.any()) return base;
  PlanKey key{d1, d2, d3, eb, kind, t, dev_info().id, v.packed()};
  std::lock_guard<std::mutex> lk(g_plan_mu);
  auto it = g_plans.find(key);
  if (it != g_plans.end()) {
    g_plan_lru.splice(g_plan_lru.begin(), g_plan_lru, it->second);
    return it->second->second;
  }
  auto P = std::make_shared<Plan>(*base);
  P->var = v;
  P->desc = fmt_plan(*P);  // the pass descriptions under this variant
  char buf[64];
  snprintf(buf, sizeof buf, " [variant col=%d row=%d tile=%d seg=%d]", v.col, v.row, v.tile, v.seg);
  P->desc += buf;
  g_plan_lru.emplace_front(key, P);
  g_plans[key] = g_plan_lru.begin();
  while (g_plan_lru.size() > kPlanCacheMax) {
    g_plans.erase(g_plan_lru.back().first);
    g_plan_lru.pop_back();
  }
  return P;
}

bool plan_cached(int64_t d1, int64_t d2, int64_t d3, int eb, int kind, int64_t t) {
  PlanKey key{d1, d2, d3, eb, kind, t, dev_info().id};
  std::lock_guard<std::mutex> lk(g_plan_mu);
  return g_plans.find(key) != g_plans.end();
}

std::shared_ptr<Plan> get_plan(int64_t d1, int64_t d2, int64_t d3, int eb, int kind, int64_t t, int *status) {
  *status = T213_OK;
  const int dev = dev_info().id;
  const bool untuned = kind == kPlanUntuned;
  if (untuned) kind = T213_PLAN_AUTO;
  if (kind == T213_PLAN_AUTO && !untuned) {
    int tk = 0;
    int64_t tt = 0;
    Variant tv;
    if (tuner_lookup_internal(d1, d2, d3, eb, &tk, &tt, &tv) == T213_OK && tk != T213_PLAN_AUTO) {
      auto p = get_plan_variant(d1, d2, d3, eb, tk, tt, tv, status);
      if (!p && tt) p = get_plan_variant(d1, d2, d3, eb, tk, 0, tv, status);  // block size of another shape
      if (p) return p;
      *status = T213_OK;
    }
  }
  PlanKey key{d1, d2, d3, eb, kind, t, dev};
  {
    std::lock_guard<std::mutex> lk(g_plan_mu);
    auto it = g_plans.find(key);
    if (it != g_plans.end()) {
      g_plan_lru.splice(g_plan_lru.begin(), g_plan_lru, it->second);
      return it->second->second;
    }
  }
  std::shared_ptr<Plan> best;
  if (kind == kPlanWideSlice || kind == kPlanSwappedSlice) {
    // no passes: a slice of these elements does not fit the chip
    best = new_plan(d1, d2, d3, eb);
    best->kind = T213_PLAN_SLICE;
    PassDesc sp;
    sp.type = PT_SLICE;
    sp.m = d2;
    sp.n = d1;
    if (d1 * d2 * eb < (64 << 20)) {
      if (kind == kPlanWideSlice)
        hold_plan(sp.hold, d2, d1, 16, eb / 16, d3);
      else
        hold_plan_swapped(sp.hold, d2, d1, eb, d3);
    }
    if (sp.hold.any.ok) best->passes.push_back(sp);
  } else if (kind != T213_PLAN_AUTO && kind != kPlanSweeps) {
    best = new_plan(d1, d2, d3, eb);
    int st = T213_ERR_UNSUPPORTED;
    if (kind <= kPlanOnePassOr) {
      if (d1 == 1 || d2 == 1)
        st = build_plan(*best, T213_PLAN_IDENTITY, 0);
      else if (crumbs_fit(d2, d1, eb, d3))
        st = build_plan(*best, kPlanCrumbs, 0);
      else if (d1 * d2 * eb < (64 << 20))  // above the shared memory of any chip
        st = build_plan(*best, T213_PLAN_SLICE, 0);
    }
    if (st && kind <= kPlanOnePassOr) {
      const int family = kPlanOnePassOr - kind;
      st = build_plan(*best, family, 0);
      if (st == T213_OK && gather_plan_cost(*best) > kRaggedCost) {
        auto R = new_plan(d1, d2, d3, eb);
        if (build_plan(*R, kPlanRagged, 0) == T213_OK) {
          R->fallback = family;
          best = R;
        }
      }
    } else if (st) {
      st = build_plan(*best, kind, t);
    }
    if (st) {
      *status = st;
      return nullptr;
    }
    best->est_cost = plan_cost(*best);
  } else {
    const int64_t m = d2, n = d1;
    if (d1 == 1 || d2 == 1 || d1 == 0 || d2 == 0 || d3 == 0) {
      best = new_plan(d1, d2, d3, eb);
      best->kind = T213_PLAN_IDENTITY;
    } else {
      // rank the cheap estimates first; build only the winners
      struct Cand {
        int kind;
        int64_t t;
        double est;
      };
      std::vector<Cand> cands;
      int64_t tb = pick_block_t(m, n);
      cands.push_back({T213_PLAN_BLOCKS, tb, estimate_cost(T213_PLAN_BLOCKS, m, n, tb, eb, d3)});
      int64_t tr = pick_band_t(m, n, eb);
      cands.push_back({T213_PLAN_BANDS, tr, estimate_cost(T213_PLAN_BANDS, m, n, tr, eb, d3)});
      int64_t tc = pick_band_t_t(m, n, eb);
      cands.push_back({T213_PLAN_BANDS_T, tc, estimate_cost(T213_PLAN_BANDS_T, m, n, tc, eb, d3)});
      // The one-pass plan (T213_PLAN_SLICE) is the fastest wherever a slice
      // fits the chip, but for four classes (B200, us).  Many slices of a few KB
      // at most are k_crumbs's (crumbs_fit).  Square slices of whole tiles are
      // one sweep of tile swaps without a barrier: 16-byte (1024, 1024, 4) 24.8
      // against 31.1, fp32 (2048, 2048, 8) 51.2 against 58.2; at 8 MB and below
      // they tie or lose.  Many slices of less than
      // 32 KB are one sweep of bands or tiles that takes the next slice's load
      // ahead: fp32 (48, 60, 12000) 51 against 81, (16, 16, 20000) 20 against
      // 86, (100, 100, 1000), 40 KB, 21 either way.  A small slice that needs
      // a cooperative launch (more than 16 CTAs' memory) and has a block or
      // band plan of aligned segments of 256 bytes or more keeps that plan up
      // to 4 MB: such a launch starts only when the whole chip is free of
      // other streams' kernels, for a gain of a few us.
      bool one_pass = false;  // a slice fits the chip
      if (kind == T213_PLAN_AUTO && crumbs_fit(m, n, eb, d3)) {
        best = new_plan(d1, d2, d3, eb);
        build_plan(*best, kPlanCrumbs, 0);
        best->est_cost = plan_cost(*best);
      } else if (kind == T213_PLAN_AUTO) {
        auto P = new_plan(d1, d2, d3, eb);
        if (build_plan(*P, T213_PLAN_SLICE, 0) == T213_OK) {
          one_pass = true;
          const HoldPlan &hp = P->passes[0].hold;
          const bool coop = hp.any.mode == HOLD_GRID && d1 * d2 * eb > hold_cluster_bytes();
          const double total = (double)d1 * d2 * d3 * eb;
          bool seg = false;
          for (const Cand &c : cands) seg = seg || (eb >= 4 && c.est < 1e8 && c.t * eb >= 256 && c.t * eb % 16 == 0);
          const bool square = m == n && tb == m && tile_eff(tb, eb) >= 0.9 && total > (8 << 20);
          const bool crumbs = d3 > 2 * dev_info().sms && d1 * d2 * eb < (32 << 10);
          if (!square && !crumbs && !(coop && seg && total <= (4 << 20))) {
            P->est_cost = plan_cost(*P);
            best = P;
          }
        }
      }
      if (!best) {
        // The Catanzaro decomposition both ways: the reference's dispatcher
        // takes C2R when d1 >= d2, else R2C (src/transpose.cu:117-123); here
        // both are costed, since which one keeps its rows inside shared
        // memory decides the faster one for tall or wide slices.
        for (int k : {T213_PLAN_C2R, T213_PLAN_R2C}) {
          Plan tmp;
          tmp.d1 = d1;
          tmp.d2 = d2;
          tmp.d3 = d3;
          tmp.eb = eb;
          build_plan(tmp, k, 0);
          // ties go to the reference's choice
          const bool ref_choice = (k == T213_PLAN_C2R) == (d1 >= d2);
          cands.push_back({k, 0, plan_cost(tmp) * (ref_choice ? 1.0 : 1.0001)});
        }
        if (kind == T213_PLAN_AUTO && !one_pass) {
          // The ragged bands against the others: the estimates of the classes
          // that lose to them, or win, are set right here, where they are the
          // alternative (kRaggedCost has the measurements).
          for (Cand &c : cands) {
            if (c.est >= 1e8) continue;
            if (c.kind == T213_PLAN_C2R || c.kind == T213_PLAN_R2C) {
              Plan tmp;
              tmp.d1 = d1;
              tmp.d2 = d2;
              tmp.d3 = d3;
              tmp.eb = eb;
              build_plan(tmp, c.kind, 0);
              if (gather_plan_cost(tmp) > plan_cost(tmp)) c.est *= 2;
            } else if (!(m == n && c.t == m)) {
              const bool bands = c.kind != T213_PLAN_BLOCKS;
              if (c.t * eb % 16 == 0 && c.t * eb >= 448)
                c.est = bands ? std::min(c.est, kRaggedCost - 0.1) : c.est;
              else if (!(bands && eb >= 8 && c.t * eb >= 1024))
                c.est += 4;
            }
          }
          cands.push_back({kPlanRagged, 0, kRaggedCost});
        }
        std::sort(cands.begin(), cands.end(), [](const Cand &a, const Cand &b) { return a.est < b.est; });
        for (const Cand &c : cands) {
          if (c.est >= 1e8) continue;
          auto P = new_plan(d1, d2, d3, eb);
          if (build_plan(*P, c.kind, c.t) == T213_OK) {
            P->est_cost = plan_cost(*P);
            best = P;
            break;
          }
        }
      }
      if (!best) {
        *status = T213_ERR_UNSUPPORTED;
        set_error("no plan applies to this shape");
        return nullptr;
      }
    }
  }
  best->desc = fmt_plan(*best);
  {
    std::lock_guard<std::mutex> lk(g_plan_mu);
    auto it = g_plans.find(key);
    if (it == g_plans.end()) {
      g_plan_lru.push_front({key, best});
      g_plans[key] = g_plan_lru.begin();
      while (g_plan_lru.size() > kPlanCacheMax) {
        g_plans.erase(g_plan_lru.back().first);
        g_plan_lru.pop_back();
      }
    }
  }
  return best;
}

size_t plan_workspace_bytes(const Plan &p) {
  size_t w = 0;
  for (const PassDesc &q : p.passes)
    if (q.type == PT_RAGGED)
      w = std::max(w, ragged_workspace(q.ragged, p.eb, p.d3));
    else if (q.type == PT_SEG && q.table) w = std::max(w, seg_cycles_carry_bytes(*q.table, p.d3, q.seg_bytes));
  return w;
}

namespace {
thread_local Variant t_variant;
}  // namespace

const Variant &current_variant() { return t_variant; }
VariantScope::VariantScope(const Variant &v) : saved(t_variant) { t_variant = v; }
VariantScope::~VariantScope() { t_variant = saved; }

// Slices per group when a plan runs its passes group by group
// (T213_SLICE_GROUP_MB: the group's size in MB; unset or 0: all slices in
// one group).  Every pass of a group runs before the next group starts, so a
// pass finds part of what the previous pass wrote still in L2.
int64_t slice_group(const Plan &P) {
  static const int64_t mb = [] {
    const char *v = std::getenv("T213_SLICE_GROUP_MB");
    return v ? (int64_t)std::atoll(v) : 0;
  }();
  const int64_t slice_bytes = P.d1 * P.d2 * P.eb;
  if (mb <= 0 || slice_bytes <= 0 || P.d3 <= 1) return std::max<int64_t>(1, P.d3);
  return std::max<int64_t>(1, std::min<int64_t>(P.d3, (mb << 20) / slice_bytes));
}

int run_plan(const Plan &P, char *data, cudaStream_t st, LaunchStats *ls) {
  const int64_t slice_bytes = P.d1 * P.d2 * P.eb;
  VariantScope vs(P.var);
  const int64_t group = slice_group(P);
  for (int64_t k0 = 0; k0 < P.d3; k0 += group) {
    const int64_t g = std::min<int64_t>(group, P.d3 - k0);
    char *gd = data + k0 * slice_bytes;
    for (const PassDesc &p : P.passes) {
      PassTimer tm(p.name(), st);
      int rc = T213_OK;
      switch (p.type) {
        case PT_COL:
          rc = launch_col_gather(p.fn, gd, g, p.m, p.n, P.eb, st, ls);
          break;
        case PT_ROW:
          rc = launch_row_gather(p.fn, gd, g, p.m, p.n, P.eb, st, ls);
          break;
        case PT_TILE:
          rc = launch_tile_swap(gd, g, p.m, p.n, p.t, P.eb, st, ls);
          break;
        case PT_BAND:
          rc = launch_band_transpose(gd, g * p.bands, p.R, p.C, P.eb, st, ls);
          break;
        case PT_SEG:
          rc = launch_seg_cycles(*p.table, gd, g, slice_bytes, p.seg_bytes, st, ls, nullptr, 0);
          break;
        case PT_RAGGED:
          rc = launch_ragged(p.ragged, gd, g, p.m, p.n, P.eb, st, ls);
          if (rc == kHoldNoSlot) {
            auto alt = get_plan(P.d1, P.d2, g, P.eb, P.fallback, 0, &rc);
            if (alt) rc = run_plan(*alt, gd, st, ls);
          }
          break;
        case PT_CRUMBS:
          rc = launch_crumbs(gd, g, p.m, p.n, P.eb, st, ls);
          break;
        case PT_SLICE:
          rc = launch_slice(p.hold, gd, g, p.m, p.n, P.eb, 1, st, ls);
          if (rc == kHoldNoSlot) {
            // the slices' CTAs cannot all be resident here: another plan
            auto alt = get_plan(P.d1, P.d2, g, P.eb, kPlanSweeps, 0, &rc);
            if (alt) rc = run_plan(*alt, gd, st, ls);
          }
          break;
      }
      if (rc) return rc;
    }
  }
  return T213_OK;
}

int check_plan_kind(int32_t plan_kind) {
  if (plan_kind >= T213_PLAN_AUTO && plan_kind <= T213_PLAN_SLICE) return T213_OK;
  set_error("unknown plan kind");
  return T213_ERR_INVALID_ARGUMENT;
}

int check_args(const void *data, int64_t d1, int64_t d2, int64_t d3, int32_t eb) {
  if (d1 < 0 || d2 < 0 || d3 < 0) {
    set_error("negative dimension");
    return T213_ERR_INVALID_ARGUMENT;
  }
  if (eb != 1 && eb != 2 && eb != 4 && eb != 8 && eb != 16) {
    set_error("element size must be 1, 2, 4, 8 or 16 bytes");
    return T213_ERR_UNSUPPORTED;
  }
  const double vol = (double)d1 * (double)d2 * (double)d3 * (double)eb;
  if (vol >= 9.0e18) {
    set_error("tensor too large");
    return T213_ERR_INVALID_ARGUMENT;
  }
  if (vol > 0 && !data) {
    set_error("data is NULL");
    return T213_ERR_INVALID_ARGUMENT;
  }
  if (((uintptr_t)data) % (uintptr_t)std::min(eb, 16)) {
    set_error("data is not aligned to its element size");
    return T213_ERR_INVALID_ARGUMENT;
  }
  return T213_OK;
}

}  // namespace t213

// =========================================================================
// C ABI
// =========================================================================
using namespace t213;

namespace {

int prefetch_if_managed(void *data, size_t bytes, cudaStream_t st) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, data) != cudaSuccess) {
    cudaGetLastError();
    set_error("data is not a CUDA device or managed pointer");
    return T213_ERR_INVALID_ARGUMENT;
  }
  if (at.type == cudaMemoryTypeManaged) {
    cudaError_t e = cudaMemPrefetchAsync(data, bytes, dev_info().id, st);
    if (e != cudaSuccess) return cuda_status(e, "cudaMemPrefetchAsync");
  } else if (at.type != cudaMemoryTypeDevice) {
    set_error("data must be device or managed memory (use t213_transpose_host for host buffers)");
    return T213_ERR_INVALID_ARGUMENT;
  }
  return T213_OK;
}

int run_shape(void *data, int64_t d1, int64_t d2, int64_t d3, int32_t eb, int kind, int64_t t,
              cudaStream_t st, int which /*0 auto/with_plan, 1 c2r, 2 r2c, 3 skinny c2r, 4 skinny r2c*/) {
  int rc = check_args(data, d1, d2, d3, eb);
  if (rc) return rc;
  if (d1 == 0 || d2 == 0 || d3 == 0) return T213_OK;
  rc = prefetch_if_managed(data, (size_t)(d1 * d2 * d3 * eb), st);
  if (rc) return rc;
  std::shared_ptr<Plan> P;
  // The decomposition's entry points are transposes too: C2R and skinny C2R
  // of (d1, d2), R2C and skinny R2C of the shape they make, (d2, d1).  They
  // take the one-pass plan where a slice fits the chip (fp32 r2c to
  // (2000, 3001, 4): 78 us by its gathers, 51 us in one pass), the ragged
  // bands where those are the better ones, else their own passes, all from
  // the plan cache (building a plan cost 20 us a call).
  if ((which == 3 || which == 4) && d2 > 32) {
    set_error(which == 3 ? "skinny C2R needs d2 <= 32" : "skinny R2C needs d2 <= 32");
    return T213_ERR_INVALID_ARGUMENT;
  }
  if (which == 2 || which == 4) std::swap(d1, d2);
  if (which == 1) kind = kPlanOnePassOr - T213_PLAN_C2R;
  if (which == 2) kind = kPlanOnePassOr - T213_PLAN_R2C;
  if (which >= 3) kind = kPlanOnePassOr - T213_PLAN_SKINNY;
  P = get_plan(d1, d2, d3, eb, kind, t, &rc);
  if (!P) return rc ? rc : T213_ERR_UNSUPPORTED;
  return run_plan(*P, (char *)data, st, nullptr);
}

int run_single_pass(int type, int32_t fn_kind, const int64_t *prm, int32_t np, void *data, int64_t d3,
                    int64_t d2, int64_t d1, int32_t eb, cudaStream_t st) {
  int rc = check_args(data, d1, d2, d3, eb);
  if (rc) return rc;
  if (np < 0 || np > 4 || (np > 0 && !prm)) {
    set_error("functor parameters: 0..4 values");
    return T213_ERR_INVALID_ARGUMENT;
  }
  FnSpec f;
  f.kind = fn_kind;
  for (int q = 0; q < np; q++) f.p[q] = prm[q];
  for (int q = 0; q < np; q++)
    if (f.p[q] < 0) {
      set_error("functor parameters must be non-negative");
      return T213_ERR_INVALID_ARGUMENT;
    }
  if (d1 == 0 || d2 == 0 || d3 == 0) return T213_OK;
  rc = prefetch_if_managed(data, (size_t)(d1 * d2 * d3 * eb), st);
  if (rc) return rc;
  const int64_t m = d2, n = d1;
  // divisor-type parameters must be positive
  auto need_pos = [&](std::initializer_list<int> idx) -> bool {
    for (int q : idx)
      if (f.p[q] <= 0) return false;
    return true;
  };
  switch (type) {
    case PT_COL: {
      bool ok = true;
      switch (fn_kind) {
        case T213_FN_C2R_PREROTATOR:
        case T213_FN_C2R_POSTROTATOR:
        case T213_FN_R2C_PREROTATOR:
          ok = need_pos({0});
          break;
        case T213_FN_R2C_POSTROTATOR:
          ok = need_pos({0});
          break;
        case T213_FN_C2R_FUSED_PREOP:
        case T213_FN_R2C_FUSED_POSTOP:
          ok = need_pos({0, 1}) && f.p[0] == m;
          break;
        case T213_FN_C2R_FUSED_POSTOP:
          ok = need_pos({0}) && f.p[0] == m;
          break;
        case T213_FN_R2C_FUSED_PREOP:
          ok = need_pos({0, 1, 2}) && f.p[2] == m;
          break;
        default:
          set_error("functor kind is not a rotator or column shuffler");
          return T213_ERR_INVALID_ARGUMENT;
      }
      if (!ok) {
        set_error("functor parameters do not match the slice (m must equal d2, divisors positive)");
        return T213_ERR_INVALID_ARGUMENT;
      }
      PassTimer tm("col_gather", st);
      return launch_col_gather(f, (char *)data, d3, m, n, eb, st, nullptr);
    }
    case PT_ROW: {
      if (fn_kind != T213_FN_C2R_SHUFFLE && fn_kind != T213_FN_C2R_LONG_SHUFFLE && fn_kind != T213_FN_R2C_SHUFFLE) {
        set_error("functor kind is not a row shuffler");
        return T213_ERR_INVALID_ARGUMENT;
      }
      if (!need_pos({0, 1, 2}) || f.p[0] != m || f.p[1] != n) {
        set_error("row shuffler parameters must be (m=d2, n=d1, c>0, k)");
        return T213_ERR_INVALID_ARGUMENT;
      }
      PassTimer tm("row_gather", st);
      return launch_row_gather(f, (char *)data, d3, m, n, eb, st, nullptr);
    }
    case PT_SEG: {
      if (fn_kind != T213_FN_C2R_POSTPERMUTER && fn_kind != T213_FN_R2C_PREPERMUTER) {
        set_error("functor kind is not a row permuter");
        return T213_ERR_INVALID_ARGUMENT;
      }
      if (!need_pos({0, 1, 2}) || f.p[0] != m || f.p[1] != n || m % f.p[2] || n % f.p[2]) {
        set_error("row permuter parameters must be (m=d2, n=d1, c) with c dividing both");
        return T213_ERR_INVALID_ARGUMENT;
      }
      PermSpec ps;
      ps.kind = fn_kind;
      ps.fn = f;
      ps.S = m;
      const int64_t seg = n * eb;
      std::shared_ptr<CycleTable> ct = get_cycle_table(ps, items_per_chunk(seg, d3), &rc);
      if (!ct) return rc;
      PassTimer tm("segment_cycles", st);
      return launch_seg_cycles(*ct, (char *)data, d3, m * n * eb, seg, st, nullptr, nullptr, 0);
    }
  }
  return T213_ERR_INVALID_ARGUMENT;
}

}  // namespace

extern "C" {

const char *t213_status_string(int status) {
  switch (status) {
    case T213_OK:
      return "ok";
    case T213_ERR_INVALID_ARGUMENT:
      return "invalid argument";
    case T213_ERR_UNSUPPORTED:
      return "unsupported";
    case T213_ERR_CUDA:
      return "CUDA error";
    case T213_ERR_OUT_OF_MEMORY:
      return "out of device memory";
    case T213_ERR_TIMEOUT:
      return "device-side wait timed out";
    case T213_ERR_BUDGET:
      return "request exceeds the HBM budget";
    case T213_ERR_NOT_READY:
      return "not ready";
  }
  return "unknown status";
}

const char *t213_last_error(void) { return last_error().c_str(); }

const char *t213_version(void) { return "213transpose_b200 1.0 (sm_100a)"; }

int t213_transpose(void *data, int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes, t213_stream_t stream) {
  return run_shape(data, d1, d2, d3, elem_bytes, T213_PLAN_AUTO, 0, (cudaStream_t)stream, 0);
}

int t213_transpose_with_plan(void *data, int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes, int32_t plan_kind,
                             int64_t t, t213_stream_t stream) {
  if (plan_kind < T213_PLAN_AUTO || plan_kind > T213_PLAN_SLICE || t < 0) {
    set_error("bad plan kind or block size");
    return T213_ERR_INVALID_ARGUMENT;
  }
  return run_shape(data, d1, d2, d3, elem_bytes, plan_kind, t, (cudaStream_t)stream, 0);
}

// Two permutation steps in one pass with the rows loaded in swapped order:
// bound by memory where the slices fill the chip, like the transposes that it
// joins, at one sweep for two.  Over 130 random (g1, h1, h2, slices) of 0.2 to
// 300 MB one pass took less than the two in all but a few that are kept out
// here: many slices whose rows are below 24 bytes, a copy instruction each
// (fp32 (4, 31, 34, 1727) 29.8 us against 27.0), or which are small, a CTA's
// round trip each: below 4 KB (16-byte (3, 11, 6, 3722) 27.0 against 18.8),
// below 12 KB where the second step is k_crumbs's (fp32 (40, 24, 2, 14855) 134
// against 80).  Ten slices an SM are many.  B200, us, one / two: fp32 (102, 30,
// 1134, 16) 112 / 192, f16 (104, 8, 96, 1575) 134 / 343, fp64 (30, 5, 3, 299)
// 8.1 / 11.7; fp32 (48, 60, 100, 120) reversed, three steps of which two join,
// 228 -> 178.
static bool swapped_in_one_pass(int64_t row_bytes, int64_t slice_bytes, int64_t slices, bool second_crumbs) {
  return slices <= 10ll * dev_info().sms || (row_bytes >= 24 && slice_bytes >= (second_crumbs ? 12 << 10 : 4 << 10));
}

int t213_permute(void *data, int32_t rank, const int64_t *dims, const int32_t *perm, int32_t elem_bytes,
                 t213_stream_t stream) {
  if (rank < 0 || rank > 32 || (rank > 0 && (!dims || !perm))) {
    set_error("t213_permute: rank must be 0..32 with dims and perm given");
    return T213_ERR_INVALID_ARGUMENT;
  }
  std::vector<int> seen(rank, 0);
  double vol = 1;
  for (int i = 0; i < rank; i++) {
    if (dims[i] < 0 || perm[i] < 0 || perm[i] >= rank || seen[perm[i]]++) {
      set_error("t213_permute: dims must be >= 0 and perm a permutation of 0..rank-1");
      return T213_ERR_INVALID_ARGUMENT;
    }
    vol *= (double)dims[i];
  }
  if (vol * elem_bytes >= 9.0e18) {
    set_error("tensor too large");
    return T213_ERR_INVALID_ARGUMENT;
  }
  const int rc0 = check_args(data, vol > 0 ? 1 : 0, 1, 1, elem_bytes);  // element size, NULL, alignment
  if (rc0) return rc0;
  if (vol == 0 || rank < 2) return T213_OK;
  // Leading axes the permutation keeps in place become part of the element:
  // up to 16 bytes the 213 plans move it as one element; from 64 bytes on,
  // a 213 step of such elements is a single segment-cycle pass (one read and
  // one write of the tensor) as long as its cycle table stays small.
  const double total_bytes = vol * elem_bytes;
  int64_t E = elem_bytes;
  int q0 = 0;
  while (q0 < rank - 1 && perm[q0] == q0) {
    const int64_t E2 = E * dims[q0];
    const bool small = E2 <= 16 && (E2 & (E2 - 1)) == 0;
    const bool seg = E2 >= 64 && total_bytes / (double)E2 <= 4.0e6;
    if (!small && !seg) break;
    E = E2;
    q0++;
  }
  // cur[q]: the input axis now at position q (fastest first) among axes
  // q0..rank-1.  For k from the slowest position down, bring perm[k] to
  // position k by rotating the prefix [q0, k]: the group [q0, p] (ending with
  // that axis) moves behind the group [p+1, k], which is one 213 transpose
  // with d1 = the first group's volume, d2 = the second's and d3 = everything
  // slower.
  std::vector<int> cur(rank);
  for (int i = 0; i < rank; i++) cur[i] = i;
  for (int k = rank - 1; k > q0; k--) {
    int p = q0;
    while (cur[p] != perm[k]) p++;
    if (p == k) continue;
    int64_t g1 = 1, g2 = 1, g3 = 1;
    for (int q = q0; q <= p; q++) g1 *= dims[cur[q]];
    for (int q = p + 1; q <= k; q++) g2 *= dims[cur[q]];
    for (int q = k + 1; q < rank; q++) g3 *= dims[cur[q]];
    int rc;
    if (E <= 16) {
      // The next step that moves anything, when it permutes just the g2
      // elements that now come first: [h2][h1][g1] -> [g1][h2 x h1 swapped].
      // Where a slice fits the chip both are one pass, its rows loaded in the
      // order in which the columns are written.
      std::vector<int> nxt = cur;
      std::rotate(nxt.begin() + q0, nxt.begin() + p + 1, nxt.begin() + k + 1);
      int k2 = k - 1, p2 = q0;
      for (; k2 > q0; k2--) {
        p2 = q0;
        while (nxt[p2] != perm[k2]) p2++;
        if (p2 != k2) break;
      }
      int64_t h1 = 1, h2 = 1;
      if (k2 > q0) {
        for (int q = q0; q <= p2; q++) h1 *= dims[nxt[q]];
        for (int q = p2 + 1; q <= k2; q++) h2 *= dims[nxt[q]];
      }
      const bool joined = g1 > 1 && h1 > 1 && h2 > 1 && h1 * h2 == g2;
      // the rows of a column lie h1 rows apart there
      const bool crumbs = joined && crumbs_fit(h2, h1 * g1, (int)E, g3);
      if (crumbs || (joined && swapped_in_one_pass(g1 * E, g1 * g2 * E, g3, crumbs_fit(h2, h1, (int)E, g3 * g1)))) {
        rc = check_args(data, g1, g2, g3, (int32_t)E);
        if (!rc) rc = prefetch_if_managed(data, (size_t)(g1 * g2 * g3 * E), (cudaStream_t)stream);
        if (rc) return rc;
        std::shared_ptr<Plan> P;
        if (!crumbs && !(P = get_plan(g1, g2, g3, (int)E, kPlanSwappedSlice, 0, &rc))) return rc;
        rc = kHoldNoSlot;
        if (crumbs) {
          PassTimer tm("crumbs", (cudaStream_t)stream);
          rc = launch_crumbs((char *)data, g3, g2, g1, (int)E, (cudaStream_t)stream, nullptr, h2);
        } else if (!P->passes.empty()) {
          PassTimer tm("slice", (cudaStream_t)stream);
          rc = launch_slice(P->passes[0].hold, (char *)data, g3, g2, g1, (int)E, 1, (cudaStream_t)stream, nullptr, h2);
        }
        if (rc == T213_OK) {
          cur = nxt;
          std::rotate(cur.begin() + q0, cur.begin() + p2 + 1, cur.begin() + k2 + 1);
          k = k2;
          continue;
        }
        if (rc != kHoldNoSlot) return rc;
      }
      rc = run_shape(data, g1, g2, g3, (int32_t)E, T213_PLAN_AUTO, 0, (cudaStream_t)stream, 0);
    } else if (g1 == 1 || g2 == 1) {
      rc = T213_OK;  // the memory layout does not change
    } else {
      // segments of E bytes: [g2][g1] -> [g1][g2] in each of the g3 slices.
      // Below 512 bytes in the one-pass form where a slice fits the chip,
      // from there on by the cycle walkers, whose bulk copies then reach 5
      // TB/s (B200, one-pass against cycles, us): 64 B (512, 64, 32) 26 / 225,
      // 128 B (64, 512, 16) 29 / 133, 256 B (8, 2048, 32) 60 / 84, 512 B
      // (4, 2048, 16) 31 / 27, 1 KB (4, 2048, 16) 61 / 53.
      rc = kHoldNoSlot;
      if (E % 16 == 0 && E < 512 && (uintptr_t)data % 16 == 0) {
        auto P = get_plan(g1, g2, g3, (int)E, kPlanWideSlice, 0, &rc);
        if (!P) return rc;
        rc = kHoldNoSlot;
        if (!P->passes.empty()) {
          PassTimer tm("slice", (cudaStream_t)stream);
          rc = launch_slice(P->passes[0].hold, (char *)data, g3, g2, g1, 16, E / 16, (cudaStream_t)stream, nullptr);
        }
      }
      if (rc != kHoldNoSlot) {
        if (rc) return rc;
        std::rotate(cur.begin() + q0, cur.begin() + p + 1, cur.begin() + k + 1);
        continue;
      }
      PermSpec ps;
      ps.kind = 0;
      ps.A = g2;
      ps.Mid = 1;
      ps.C = g1;
      ps.S = g1 * g2;
      rc = T213_OK;
      auto ct = get_cycle_table(ps, items_per_chunk(E, g3), &rc);
      if (!ct) return rc;
      if (ct->n_chunks > 0)
        rc = launch_seg_cycles(*ct, (char *)data, g3, g1 * g2 * E, E, (cudaStream_t)stream, nullptr, nullptr, 0);
    }
    if (rc) return rc;
    std::rotate(cur.begin() + q0, cur.begin() + p + 1, cur.begin() + k + 1);
  }
  return T213_OK;
}

int t213_c2r_transpose(void *data, int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes, t213_stream_t stream) {
  return run_shape(data, d1, d2, d3, elem_bytes, 0, 0, (cudaStream_t)stream, 1);
}

int t213_r2c_transpose(void *data, int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes, t213_stream_t stream) {
  return run_shape(data, d1, d2, d3, elem_bytes, 0, 0, (cudaStream_t)stream, 2);
}

int t213_skinny_c2r_transpose(void *data, int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes,
                              t213_stream_t stream) {
  return run_shape(data, d1, d2, d3, elem_bytes, 0, 0, (cudaStream_t)stream, 3);
}

int t213_skinny_r2c_transpose(void *data, int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes,
                              t213_stream_t stream) {
  return run_shape(data, d1, d2, d3, elem_bytes, 0, 0, (cudaStream_t)stream, 4);
}

int t213_rotate(int32_t fn_kind, const int64_t *fn_params, int32_t n_params, void *data, int64_t d3, int64_t d2,
                int64_t d1, int32_t elem_bytes, t213_stream_t stream) {
  if (fn_kind < T213_FN_C2R_PREROTATOR || fn_kind > T213_FN_R2C_POSTROTATOR) {
    set_error("functor kind is not a rotator");
    return T213_ERR_INVALID_ARGUMENT;
  }
  return run_single_pass(PT_COL, fn_kind, fn_params, n_params, data, d3, d2, d1, elem_bytes, (cudaStream_t)stream);
}

int t213_row_shuffle(int32_t fn_kind, const int64_t *fn_params, int32_t n_params, void *data, int64_t d3,
                     int64_t d2, int64_t d1, int32_t elem_bytes, t213_stream_t stream) {
  return run_single_pass(PT_ROW, fn_kind, fn_params, n_params, data, d3, d2, d1, elem_bytes, (cudaStream_t)stream);
}

int t213_col_shuffle(int32_t fn_kind, const int64_t *fn_params, int32_t n_params, void *data, int64_t d3,
                     int64_t d2, int64_t d1, int32_t elem_bytes, t213_stream_t stream) {
  if (fn_kind < T213_FN_C2R_FUSED_PREOP || fn_kind > T213_FN_R2C_FUSED_POSTOP) {
    set_error("functor kind is not a column shuffler");
    return T213_ERR_INVALID_ARGUMENT;
  }
  return run_single_pass(PT_COL, fn_kind, fn_params, n_params, data, d3, d2, d1, elem_bytes, (cudaStream_t)stream);
}

int t213_scatter_permute(int32_t fn_kind, const int64_t *fn_params, int32_t n_params, void *data, int64_t d3,
                         int64_t d2, int64_t d1, int32_t elem_bytes, t213_stream_t stream) {
  return run_single_pass(PT_SEG, fn_kind, fn_params, n_params, data, d3, d2, d1, elem_bytes, (cudaStream_t)stream);
}

int t213_plan_describe(int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes, int32_t plan_kind, int64_t t,
                       char *buf, size_t buflen) {
  int rc = check_args((void *)16, d1, d2, d3, elem_bytes);
  if (rc || (rc = check_plan_kind(plan_kind))) return rc;
  if (!buf || buflen == 0) {
    set_error("buffer is NULL");
    return T213_ERR_INVALID_ARGUMENT;
  }
  std::shared_ptr<Plan> P = get_plan(d1, d2, d3, elem_bytes, plan_kind, t, &rc);
  if (!P) return rc;
  snprintf(buf, buflen, "%s", P->desc.c_str());
  return T213_OK;
}

int t213_plan_launches(int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes, int32_t plan_kind, int64_t t,
                       int32_t *launches) {
  int rc = check_args((void *)16, d1, d2, d3, elem_bytes);
  if (rc || (rc = check_plan_kind(plan_kind))) return rc;
  if (!launches) return T213_ERR_INVALID_ARGUMENT;
  std::shared_ptr<Plan> P = get_plan(d1, d2, d3, elem_bytes, plan_kind, t, &rc);
  if (!P) return rc;
  int n = 0;
  const int64_t group = slice_group(*P);
  for (int64_t k0 = 0; k0 < d3; k0 += group) {
    const int64_t g = std::min<int64_t>(group, d3 - k0);
    for (const PassDesc &p : P->passes) {
      switch (p.type) {
        case PT_COL:
          n += count_col_gather(g, p.m, p.n, elem_bytes);
          break;
        case PT_ROW:
          n += count_row_gather(g, p.m, p.n, elem_bytes);
          break;
        case PT_SEG:
          n += (p.table->n_chunks > 0) + (p.table->n_carry > 0);
          break;
        case PT_RAGGED:
          n += ragged_launches(p.ragged);
          break;
        default:
          n += 1;
      }
    }
  }
  *launches = n;
  return T213_OK;
}

int t213_slice_debug_stall(void *data, int64_t d1, int64_t d2, int64_t d3, int32_t elem_bytes, int64_t wait_ns,
                           t213_stream_t stream) {
  int rc = check_args(data, d1, d2, d3, elem_bytes);
  if (rc) return rc;
  if (wait_ns <= 0 || d1 < 2 || d2 < 2 || d3 < 1) {
    set_error("t213_slice_debug_stall: bad arguments");
    return T213_ERR_INVALID_ARGUMENT;
  }
  std::shared_ptr<Plan> P = get_plan(d1, d2, d3, elem_bytes, T213_PLAN_SLICE, 0, &rc);
  if (!P) return rc;
  rc = launch_slice(P->passes[0].hold, (char *)data, d3, d2, d1, elem_bytes, 1, (cudaStream_t)stream, nullptr, 0,
                    (uint64_t)wait_ns);
  if (rc != kHoldNoSlot) return rc;
  set_error("the slice's CTAs cannot all be resident");
  return T213_ERR_UNSUPPORTED;
}

int t213_device_status(t213_stream_t stream, int32_t *device_status) {
  if (!device_status) return T213_ERR_INVALID_ARGUMENT;
  int rc = T213_OK;
  int *w = device_status_word(&rc);
  if (!w) return rc;
  cudaError_t e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_status(e, "cudaStreamSynchronize");
  int v = 0;
  if ((e = cudaMemcpy(&v, w, sizeof(int), cudaMemcpyDeviceToHost)) != cudaSuccess) return cuda_status(e, "status read");
  if (v && (e = cudaMemsetAsync(w, 0, sizeof(int), (cudaStream_t)stream)) == cudaSuccess)
    e = cudaStreamSynchronize((cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_status(e, "status reset");
  *device_status = v;
  return T213_OK;
}

int t213_pass_timing_enable(int32_t enable) {
  g_timing.store(enable != 0);
  return T213_OK;
}

int t213_pass_timing_read(const char *pass_name, double *total_ms, int64_t *launches) {
  if (!pass_name || !total_ms || !launches) return T213_ERR_INVALID_ARGUMENT;
  std::lock_guard<std::mutex> lk(g_tmu);
  TimingRec &r = g_trec[pass_name];
  for (auto &pr : r.pending) {
    cudaEventSynchronize(pr.second);
    float ms = 0;
    if (cudaEventElapsedTime(&ms, pr.first, pr.second) == cudaSuccess) r.total_ms += ms;
    cudaEventDestroy(pr.first);
    cudaEventDestroy(pr.second);
    r.launches++;
  }
  r.pending.clear();
  cudaGetLastError();
  *total_ms = r.total_ms;
  *launches = r.launches;
  return T213_OK;
}

int t213_pass_timing_reset(void) {
  std::lock_guard<std::mutex> lk(g_tmu);
  for (auto &kv : g_trec)
    for (auto &pr : kv.second.pending) {
      cudaEventSynchronize(pr.second);
      cudaEventDestroy(pr.first);
      cudaEventDestroy(pr.second);
    }
  g_trec.clear();
  cudaGetLastError();
  return T213_OK;
}

int t213_release_cache(void) {
  cudaDeviceSynchronize();
  {
    std::lock_guard<std::mutex> lk(g_plan_mu);
    g_plans.clear();
    g_plan_lru.clear();
  }
  release_workspaces();
  release_kept();
  flush_deferred_frees();
  return T213_OK;
}

}  // extern "C"
