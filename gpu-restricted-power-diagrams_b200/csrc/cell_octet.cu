// Cell launches that clip with eight lanes per cell (device code in
// clip_octet.cuh): the clipping kernel, the finish kernel for the cells that
// need a warp, and the cone kernels.
#include "clip_octet.cuh"

namespace rpd {

bool octet_applies(const CellLaunch &a) {
  return a.precision <= 1 && !a.safe_radius && !a.counters && !a.trace && a.border_d == 0 && a.only_status < 0 &&
         a.K <= 256;
}

namespace {

template <int MW, bool GRID, bool AHEAD>
cudaError_t launch_clip_ahead(const CellLaunch &a, cudaStream_t st) {
  const OctLayout O = oct_layout<MW>(a.P, a.V, AHEAD);
  const int threads = 128, cells = threads / kOct;
  const size_t smem = size_t(O.total) * cells;
  cudaError_t e = allow_smem(reinterpret_cast<const void *>(k_clip<MW, GRID, AHEAD>), smem);
  if (e != cudaSuccess) return e;
  k_clip<MW, GRID, AHEAD><<<(a.num + cells - 1) / cells, threads, smem, st>>>(a, O);
  return cudaGetLastError();
}

template <int MW, bool GRID>
cudaError_t launch_clip(const CellLaunch &a, cudaStream_t st) {
  return a.ahead && a.ahead_first ? launch_clip_ahead<MW, GRID, true>(a, st) : launch_clip_ahead<MW, GRID, false>(a, st);
}

template <int VS, bool GRID, bool INL>
cudaError_t launch_finish(const CellLaunch &a, const Layout &L, cudaStream_t st, int sm_count) {
  const int wpb = warps_per_block_for(L);
  if (wpb == 0) return cudaErrorInvalidValue;
  const size_t smem = size_t(L.total) * wpb;
  cudaError_t e = allow_smem(reinterpret_cast<const void *>(k_finish<VS, GRID, INL>), smem);
  if (e != cudaSuccess) return e;
  const int blocks = std::min(sm_count * 5, (a.num + wpb - 1) / wpb);
  k_finish<VS, GRID, INL><<<blocks, wpb * 32, smem, st>>>(a, L);
  return cudaGetLastError();
}

template <int VS>
cudaError_t launch_octet_vs(const CellLaunch &a, const Layout &L, cudaStream_t st, int sm_count, int *launches) {
  cudaError_t e;
  if (a.grid.size > 0) e = a.P <= 32 ? launch_clip<1, true>(a, st) : launch_clip<2, true>(a, st);
  else e = a.P <= 32 ? launch_clip<1, false>(a, st) : launch_clip<2, false>(a, st);
  if (e != cudaSuccess) return e;
  if (launches) ++*launches;
  if (a.grid.size > 0 && a.defer.slots) {
    if ((e = launch_finish<VS, true, false>(a, L, st, sm_count)) != cudaSuccess) return e;
    if (a.after_cell) cudaEventRecord(a.after_cell, st);
    if (launches) ++*launches;
    return launch_cones<VS>(a, L, st, sm_count, launches);
  }
  if (a.grid.size > 0) e = launch_finish<VS, true, true>(a, L, st, sm_count);
  else if (a.hess) e = launch_finish<VS, false, true>(a, L, st, sm_count);
  if (e != cudaSuccess) return e;
  if (a.after_cell) cudaEventRecord(a.after_cell, st);
  if (launches && (a.grid.size > 0 || a.hess)) ++*launches;
  return cudaGetLastError();
}

template <int MW, bool GRID, bool AHEAD>
cudaError_t batch_clip_ahead(const CellBatch &b, const CellLaunch *descs, const int *start, long rows, cudaStream_t st,
                             int sm_count) {
  const OctLayout O = oct_layout<MW>(b.P, b.V, AHEAD);
  const int threads = 128, cells = threads / kOct;
  const size_t smem = size_t(O.total) * cells;
  auto k = k_clip_batch<MW, GRID, AHEAD>;
  cudaError_t e = allow_smem(reinterpret_cast<const void *>(k), smem);
  if (e != cudaSuccess) return e;
  int blocks;
  int *work = nullptr;
  if (rows >= 0) {
    blocks = int(std::max<long>(1, (rows + cells - 1) / cells));
  } else {
    blocks = resident_blocks(k, threads, smem, sm_count);
    work = b.work;
    if ((e = cudaMemsetAsync(work, 0, sizeof(int), st)) != cudaSuccess) return e;
  }
  k<<<blocks, threads, smem, st>>>(descs, start, b.ndiag, O, rows >= 0 ? 0 : kOctetMinRows, work);
  return cudaGetLastError();
}

template <int MW, bool GRID>
cudaError_t batch_clip(const CellBatch &b, const CellLaunch *descs, const int *start, long rows, cudaStream_t st,
                       int sm_count) {
  return b.ahead ? batch_clip_ahead<MW, GRID, true>(b, descs, start, rows, st, sm_count)
                 : batch_clip_ahead<MW, GRID, false>(b, descs, start, rows, st, sm_count);
}

template <int VS, bool GRID, bool INL>
cudaError_t batch_finish(const CellBatch &b, const CellLaunch *descs, const Layout &L, cudaStream_t st, int sm_count) {
  const int wpb = warps_per_block_for(L);
  if (wpb == 0) return cudaErrorInvalidValue;
  const size_t smem = size_t(L.total) * wpb;
  auto k = k_finish_batch<VS, GRID, INL>;
  cudaError_t e = allow_smem(reinterpret_cast<const void *>(k), smem);
  if (e != cudaSuccess) return e;
  k<<<resident_blocks(k, wpb * 32, smem, sm_count), wpb * 32, smem, st>>>(descs, b.hand, L);
  return cudaGetLastError();
}

// The cells of a launch: with eight lanes each (their records are left), or
// of few rows with a warp each.  Where only the device knows the rows
// (rows < 0) both kernels are launched and one of them does nothing.
template <int VS, bool GRID, bool INL>
cudaError_t batch_rows(const CellBatch &b, const CellLaunch *descs, const int *start, long rows, const Layout &L,
                       cudaStream_t st, int sm_count, int &n) {
  cudaError_t e;
  const bool some = rows < 0;
  if (some || rows >= kOctetMinRows) {
    e = b.P <= 32 ? batch_clip<1, GRID>(b, descs, start, rows, st, sm_count)
                  : batch_clip<2, GRID>(b, descs, start, rows, st, sm_count);
    if (e != cudaSuccess) return e;
    ++n;
  }
  if (some || rows < kOctetMinRows) {
    if ((e = batch_cells<VS, GRID, INL>(descs, start, b.ndiag, L, -1, nullptr, 0, rows, b.work, st, sm_count, nullptr,
                                        kOctetMinRows, some)) != cudaSuccess)
      return e;
    ++n;
  }
  return cudaSuccess;
}

// The plain diagrams' cells (no domain), then those with one; the records of
// each are finished, and the cells left over re-run with a warp each, before
// the next use of the counters.
template <int VS>
cudaError_t launch_batch_octet_vs(const CellBatch &b, const Layout &Lg, const Layout &Lp, cudaStream_t st, int sm_count,
                                  int *launches) {
  cudaError_t e;
  const size_t ctr_bytes = sizeof(int) * kClipCounters;
  int n = 0;
  if (b.start_plain) {
    if ((e = cudaMemsetAsync(b.hand.ctr, 0, ctr_bytes, st)) != cudaSuccess) return e;
    if ((e = batch_rows<VS, false, true>(b, b.descs_inline, b.start_plain, b.rows_plain, Lp, st, sm_count, n)) !=
        cudaSuccess)
      return e;
    if (b.HC && (e = batch_finish<VS, false, true>(b, b.descs_inline, Lp, st, sm_count)) != cudaSuccess) return e;
    if ((e = batch_cells<VS, false, true>(b.descs_inline, b.start_plain, b.ndiag, Lp, kParkOverflow, nullptr, 0, -1,
                                          b.work, st, sm_count, b.hand.ctr + 2)) != cudaSuccess)
      return e;
    n += 1 + (b.HC ? 1 : 0);
  }
  if (b.start_grid) {
    const bool park = b.defer.slots != nullptr;
    const CellLaunch *descs = park ? b.descs : b.descs_inline;
    if ((e = cudaMemsetAsync(b.hand.ctr, 0, ctr_bytes, st)) != cudaSuccess) return e;
    e = park ? batch_rows<VS, true, false>(b, descs, b.start_grid, b.rows_grid, Lg, st, sm_count, n)
             : batch_rows<VS, true, true>(b, descs, b.start_grid, b.rows_grid, Lg, st, sm_count, n);
    if (e != cudaSuccess) return e;
    e = park ? batch_finish<VS, true, false>(b, descs, Lg, st, sm_count)
             : batch_finish<VS, true, true>(b, descs, Lg, st, sm_count);
    if (e != cudaSuccess) return e;
    ++n;
    if ((e = record_after_cell(b, st)) != cudaSuccess) return e;
    if (park) {
      if ((e = launch_cones_batch<VS>(b, Lg, st, sm_count)) != cudaSuccess) return e;
      n += 3;
    }
    if ((e = batch_cells<VS, true, true>(b.descs_inline, b.start_grid, b.ndiag, Lg, kParkOverflow,
                                         park ? b.defer.counters : nullptr, b.defer.capacity, -1, b.work, st, sm_count,
                                         b.hand.ctr + 2)) != cudaSuccess)
      return e;
    ++n;
  } else if ((e = record_after_cell(b, st)) != cudaSuccess) {
    return e;
  }
  if (launches) *launches += n;
  return cudaGetLastError();
}

}  // namespace

cudaError_t cell_batch_launch_octet(const CellBatch &b, cudaStream_t st, int sm_count, int *launches) {
  if (b.P > kMaxP || b.V > kMaxV || b.T > kMaxT || b.P < 7 || b.V < 8) return cudaErrorInvalidValue;
  if (b.HC && b.defer.slots) return cudaErrorInvalidValue;  // Hessian rows are summed inline
  const Layout Lg = make_layout(b.P, b.V, b.T, true, b.HC, b.T_slot, 0, b.disjoint),
               Lp = make_layout(b.P, b.V, b.T, false, b.HC);
  if (b.defer.slots && (b.defer.slot_bytes < slot_bytes_for(Lg, Lg.T) || b.defer.items < 1))
    return cudaErrorInvalidValue;
  const int vs = Lg.Vc / 32;
  if (vs <= 2) return launch_batch_octet_vs<2>(b, Lg, Lp, st, sm_count, launches);
  if (vs <= 3) return launch_batch_octet_vs<3>(b, Lg, Lp, st, sm_count, launches);
  if (vs <= 4) return launch_batch_octet_vs<4>(b, Lg, Lp, st, sm_count, launches);
  if (vs <= 6) return launch_batch_octet_vs<6>(b, Lg, Lp, st, sm_count, launches);
  return launch_batch_octet_vs<8>(b, Lg, Lp, st, sm_count, launches);
}

cudaError_t cell_launch_octet(const CellLaunch &a, cudaStream_t st, int sm_count, int *launches) {
  if (a.P > kMaxP || a.V > kMaxV || a.T > kMaxT || a.P < 7 || a.V < 8) return cudaErrorInvalidValue;
  if (a.hess && (a.defer.slots || a.H < 1 || (a.HC != 1 && a.HC != 4))) return cudaErrorInvalidValue;
  if (a.T_ahead > kMaxT || (a.T_ahead > a.T && (!a.defer.slots || a.hess))) return cudaErrorInvalidValue;
  const Layout L = make_layout(a.P, a.V, a.T, a.grid.size > 0, a.hess ? a.HC : 0, a.T_ahead, 0,
                               a.grid.lists_disjoint != 0);
  if (a.defer.slots && (a.defer.slot_bytes < slot_bytes_for(L, L.T) || a.defer.items < 1))
    return cudaErrorInvalidValue;
  const int vs = L.Vc / 32;
  if (vs <= 2) return launch_octet_vs<2>(a, L, st, sm_count, launches);
  if (vs <= 3) return launch_octet_vs<3>(a, L, st, sm_count, launches);
  if (vs <= 4) return launch_octet_vs<4>(a, L, st, sm_count, launches);
  if (vs <= 6) return launch_octet_vs<6>(a, L, st, sm_count, launches);
  return launch_octet_vs<8>(a, L, st, sm_count, launches);
}

}  // namespace rpd
