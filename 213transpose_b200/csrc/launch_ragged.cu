// Launches of the ragged band plan: the remainder, the segment cycles and the
// bands (see RaggedPlan).
#include <algorithm>
#include <optional>

#include "internal.h"
#include "k_walk.cuh"

namespace t213 {

namespace {

int64_t up16(int64_t x) { return (x + 15) / 16 * 16; }

int64_t tail_bytes(const RaggedPlan &rp, int eb, int64_t d3) { return up16(rp.r * rp.small * eb * d3); }
int64_t carry_pitch(const RaggedPlan &rp, int eb) { return up16(rp.t * eb); }

// Pieces of 16 KB, halved down to 4 KB while chunks of 16 steps would leave
// resident CTAs without a piece.
int64_t walk_piece(const RaggedPlan &rp, int eb, int64_t d3) {
  int64_t piece = kWalkPiece;
  const int64_t seg = rp.t * eb;
  while (piece > 4096 && (seg + piece - 1) / piece * rp.perm.S * d3 < 16 * 6 * (int64_t)dev_info().sms) piece /= 2;
  return std::min(piece, seg);
}
int64_t walk_pieces(const RaggedPlan &rp, int eb, int64_t d3) {
  const int64_t piece = walk_piece(rp, eb, d3);
  return (rp.t * eb + piece - 1) / piece;
}

template <typename Fn>
int by_eb(int eb, Fn &&fn) {
  switch (eb) {
    case 1:
      return fn(IC<1>{});
    case 2:
      return fn(IC<2>{});
    case 4:
      return fn(IC<4>{});
    case 8:
      return fn(IC<8>{});
    case 16:
      return fn(IC<16>{});
  }
  set_error("unsupported element size");
  return T213_ERR_UNSUPPORTED;
}

int launched(const char *what, LaunchStats *ls) {
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_status(e, what);
  if (ls) ls->launches++;
  return T213_OK;
}

// The remainder to the workspace (save) or from there to its place.
int tail(const RaggedPlan &rp, bool save, char *data, char *ws, int64_t d3, int64_t m, int64_t n, int eb,
         cudaStream_t st, LaunchStats *ls) {
  const int64_t slice = m * n, head = rp.q * rp.t, per = rp.r * rp.small;
  const int64_t grid = std::min<int64_t>((int64_t)dev_info().sms * 8, (per * d3 + kWalkThreads - 1) / kWalkThreads);
  return by_eb(eb, [&](auto EBc) -> int {
    constexpr int EB = decltype(EBc)::value;
    const dim3 g((unsigned)std::max<int64_t>(1, grid));
    if (rp.cols) {
      if (save)  // column head + j of row i -> saved[j][i]
        k_walk_tail<EB><<<g, kWalkThreads, 0, st>>>(data + head * EB, slice * EB, n, 1, ws, per * EB, 1, m, m, rp.r, d3);
      else  // saved, in order, -> the last r output rows
        k_walk_tail<EB><<<g, kWalkThreads, 0, st>>>(ws, per * EB, m, 1, data + head * m * EB, slice * EB, m, 1, rp.r, m,
                                                    d3);
    } else {
      if (save)  // the last r rows, in order
        k_walk_tail<EB><<<g, kWalkThreads, 0, st>>>(data + head * n * EB, slice * EB, n, 1, ws, per * EB, n, 1, rp.r, n,
                                                    d3);
      else  // saved[j][i] -> column head + j of output row i
        k_walk_tail<EB><<<g, kWalkThreads, 0, st>>>(ws, per * EB, 1, n, data + head * EB, slice * EB, m, 1, n, rp.r, d3);
    }
    return launched("k_walk_tail launch", ls);
  });
}

int walk(const RaggedPlan &rp, char *data, char *carry, int64_t d3, int64_t m, int64_t n, int eb, cudaStream_t st,
         LaunchStats *ls) {
  const CycleTable &ct = *rp.table;
  if (ct.n_chunks == 0) return T213_OK;
  SegRows rows;
  rows.q = FastDiv<uint32_t>((uint64_t)rp.q);
  rows.pitch = (rp.q * rp.t + rp.r) * eb;
  rows.seg_bytes = rp.t * eb;
  const int64_t slice_bytes = m * n * eb, cp = carry_pitch(rp, eb);
  const uint32_t piece = (uint32_t)walk_piece(rp, eb, d3);
  const int64_t pieces = walk_pieces(rp, eb, d3);
  const int64_t smem = (int64_t)kWalkRing * ((piece + 15) / 16 * 16 + 32);
  const SegPerm3<uint32_t> dst(rp.perm.A, rp.perm.Mid, rp.perm.C);
  return by_eb(eb, [&](auto EBc) -> int {
    constexpr int EB = decltype(EBc)::value;
    if (ct.n_carry > 0) {
      const int64_t blocks = (rows.seg_bytes / EB + 4 * kWalkThreads - 1) / (4 * kWalkThreads) * ct.n_carry * d3;
      k_walk_carry<EB><<<(unsigned)std::min<int64_t>((int64_t)dev_info().sms * 8, blocks), kWalkThreads, 0, st>>>(
          data, slice_bytes, d3, rows, (const CarryItem *)ct.d_carry_items, ct.n_carry, carry, cp);
      const int rc = launched("k_walk_carry launch", ls);
      if (rc) return rc;
    }
    auto kern = k_seg_walk<EB, SegPerm3<uint32_t>>;
    if (!kernel_attr_once((const void *)kern, smem, 1))
      return cuda_status(cudaGetLastError(), "cudaFuncSetAttribute(k_seg_walk)");
    int per_sm = 1;
    occupancy_cached((const void *)kern, kWalkThreads, smem, 1, &per_sm);
    const int64_t items = ct.n_chunks * pieces * d3;
    const int64_t grid = std::min<int64_t>((int64_t)per_sm * dev_info().sms, items);
    kern<<<(unsigned)grid, kWalkThreads, (size_t)smem, st>>>(data, slice_bytes, d3, rows, piece, (uint32_t)pieces,
                                                           (const Chunk *)ct.d_chunks, ct.n_chunks, carry, cp, dst);
    return launched("k_seg_walk launch", ls);
  });
}

}  // namespace

int ragged_table(RaggedPlan &rp, int eb, int64_t d3) {
  int st = T213_OK;
  rp.table = get_cycle_table(rp.perm, 2 * walk_pieces(rp, eb, d3) * d3, &st);
  return rp.table ? T213_OK : st;
}

size_t ragged_workspace(const RaggedPlan &rp, int eb, int64_t d3) {
  return (size_t)(tail_bytes(rp, eb, d3) + rp.table->n_carry * d3 * carry_pitch(rp, eb));
}

int ragged_launches(const RaggedPlan &rp) {
  return (rp.r > 0 ? 2 : 0) + (rp.table->n_carry > 0) + (rp.table->n_chunks > 0) + 1;
}

int launch_ragged(const RaggedPlan &rp, char *data, int64_t d3, int64_t m, int64_t n, int eb, cudaStream_t st,
                  LaunchStats *ls) {
  if (d3 <= 0) return T213_OK;
  // Everything that can fail is asked for before the first kernel touches the
  // tensor.
  const size_t need = ragged_workspace(rp, eb, d3);
  CycleTable &ct = *rp.table;
  int slot = -1;
  int rc = hold_rag_ready(rp, eb, st, &slot);
  if (rc) return rc;
  if (ct.n_chunks > 0 && (rc = ct.ensure_uploaded(st))) return rc;
  char *ws = nullptr;
  std::optional<WorkspaceUse> use;  // to the end of the call
  if (need && !(ws = workspace(use.emplace(), st, need, &rc))) return rc;
  char *carry = ws + tail_bytes(rp, eb, d3);
  if (rp.r > 0 && (rc = tail(rp, true, data, ws, d3, m, n, eb, st, ls))) return rc;
  if (rp.cols && (rc = walk(rp, data, carry, d3, m, n, eb, st, ls))) return rc;
  rc = launch_hold_rag(rp, data, d3, m * n * eb, eb, slot, st);
  if (rc == kHoldNoSlot && rp.cols) {  // no other plan may run on the walked segments
    set_error("the bands' cooperative launch was refused after the segments had moved");
    return T213_ERR_CUDA;
  }
  if (rc) return rc;
  if (ls) ls->launches++;
  if (!rp.cols && (rc = walk(rp, data, carry, d3, m, n, eb, st, ls))) return rc;
  if (rp.r > 0) return tail(rp, false, data, ws, d3, m, n, eb, st, ls);
  return T213_OK;
}

}  // namespace t213
