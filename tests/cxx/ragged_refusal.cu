// launch_ragged on the host with its neighbours stubbed: the bands' launch
// answers that its CTAs cannot all be resident.  Where the segments have been
// walked by then (columns cut) that must be an error; where the tensor is
// untouched (rows cut) the caller may take another plan.  A plan whose launch
// is refused beforehand asks for neither table nor workspace.
#include <cstdio>

#include "launch_ragged.cu"

namespace t213 {
static int launches = 0, uploads = 0, workspaces = 0, ready_answer = T213_OK;
static std::string message;
void set_error(const std::string &m) { message = m; }
int cuda_status(cudaError_t, const char *) { return T213_ERR_CUDA; }
const DevInfo &dev_info() {
  static DevInfo d;
  return d;
}
WorkspaceUse::WorkspaceUse() {}
WorkspaceUse::~WorkspaceUse() {}
char *workspace(WorkspaceUse &, cudaStream_t, size_t, int *) {
  static char b[256];
  workspaces++;
  return b;
}
bool kernel_attr_once(const void *, int64_t, int) { return true; }
int occupancy_cached(const void *, int, int64_t, int, int *v) { return *v = 1, T213_OK; }
std::shared_ptr<CycleTable> get_cycle_table(const PermSpec &, int64_t, int *) { return std::make_shared<CycleTable>(); }
int CycleTable::ensure_uploaded(cudaStream_t) { return uploads++, T213_OK; }
int CycleTable::wait_uploaded() { return T213_OK; }
CycleTable::~CycleTable() {}
int hold_rag_ready(const RaggedPlan &, int, cudaStream_t, int *slot) { return *slot = 0, ready_answer; }
int launch_hold_rag(const RaggedPlan &, char *, int64_t, int64_t, int, int, cudaStream_t) { return launches++, kHoldNoSlot; }
}  // namespace t213

using namespace t213;

int main() {
  int bad = 0;
  auto check = [&](bool ok, const char *what) {
    if (!ok) bad++, printf("wrong: %s\n", what);
  };
  for (bool cols : {true, false}) {
    RaggedPlan rp;
    rp.ok = true;
    rp.cols = cols;
    rp.t = 128;
    rp.q = 2;
    rp.r = 0;  // no remainder and an empty table: nothing is launched before the bands
    rp.small = 3;
    int rc = ragged_table(rp, 4, 1);
    check(rc == T213_OK, "table");
    launches = 0;
    message.clear();
    rc = launch_ragged(rp, nullptr, 1, cols ? 3 : 256, cols ? 256 : 3, 4, nullptr, nullptr);
    check(launches == 1, "the bands are launched once");
    check(cols ? rc == T213_ERR_CUDA && !message.empty() : rc == kHoldNoSlot, cols ? "refused after the walk" : "refused before");
    launches = uploads = workspaces = 0;
    rp.table->n_chunks = 1;
    ready_answer = kHoldNoSlot;
    rc = launch_ragged(rp, nullptr, 1, cols ? 3 : 256, cols ? 256 : 3, 4, nullptr, nullptr);
    check(rc == kHoldNoSlot && !launches && !uploads && !workspaces, "refused before anything is asked for");
    ready_answer = T213_OK;
  }
  printf(bad ? "%d wrong\n" : "ok\n", bad);
  return bad;
}
