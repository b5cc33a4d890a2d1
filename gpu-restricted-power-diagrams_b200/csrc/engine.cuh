// Engine state behind the C ABI: device context, resident seed sets.
#pragma once
#include <cstring>
#include <string>
#include <vector>

#include "../../include/rpd.h"
#include "bins.cuh"
#include "cell.cuh"
#include "grid_host.h"
#include "knn.cuh"

namespace rpd {

// Owning device allocation that only grows.
// Device memory comes from the stream-ordered pool of the current device,
// through one allocation stream per device: allocating and freeing never
// synchronize the device, so solvers on other streams keep running (the
// serving loop depends on it).  A buffer is grown or released only when no
// work that uses it is pending: every entry point of the engine ends with a
// synchronization of its stream.
//
// Freed blocks of up to 4 GB are kept and handed out again without a call
// into the driver: the smallest one that holds the bytes, if it is at most
// twice as large; up to 1/16 of the device's memory while a context of the
// device exists.  The serving loop gives back what its budget does not hold
// (pool_trim).  The driver's pool puts a large block together from fragments
// where freed blocks of other sizes lie in between, or maps new memory; that
// takes 10 ms to a second and stops all streams.  600 served requests of 10K
// to 2M seeds on four streams, four runs each: with blocks kept by exact size
// class 1,900 calls into the driver, 6 to 14 s in the slow ones, 27 to 28M
// cells/s; now 900, 0.2 to 0.4 s, 33.5M; with blocks of up to 1.5 times 680
// (1/8 of the memory), 2 s.  Half that load, p50 / p99: 13 / 110 to 570 ms ->
// 13 / 55.  Everything to the driver's pool, the kernels before: 19M cells/s,
// 24 / 114 ms.
cudaError_t pool_alloc(void **p, size_t bytes, size_t *block, int *device);
void pool_free(void *p, size_t block, int device);
void pool_context(int device, int change, size_t device_bytes = 0);  // a context made (1) or destroyed (-1)
// Gives kept blocks back to the driver's pool until at most `most` bytes are kept.
void pool_trim(int device, size_t most);

struct DevBuf {
  void *ptr = nullptr;
  size_t bytes = 0;
  size_t block = 0;  // the size of the block that holds them
  int device = 0;    // the block's
  DevBuf() = default;
  DevBuf(const DevBuf &) = delete;
  DevBuf &operator=(const DevBuf &) = delete;
  ~DevBuf() { release(); }
  void release() {
    if (ptr) pool_free(ptr, block, device);
    ptr = nullptr;
    bytes = block = 0;
  }
  cudaError_t ensure(size_t want) {
    if (want <= bytes && ptr) return cudaSuccess;
    release();
    cudaError_t e = pool_alloc(&ptr, want ? want : 16, &block, &device);
    if (e == cudaSuccess) bytes = want ? want : 16;
    else ptr = nullptr;
    return e;
  }
  template <class T>
  T *as() const {
    return static_cast<T *>(ptr);
  }
};

void set_error(rpd_context *ctx, const std::string &msg);
int map_cuda(rpd_context *ctx, cudaError_t e, const char *what);
const HostGrid *host_grid(const rpd_grid *g);
rpd_grid *grid_handle(HostGrid &&g);

}  // namespace rpd

struct rpd_context {
  int device = 0;
  int sm_count = 0;
  cudaStream_t stream = nullptr;
  std::string error;
  // neighbour-search variants (rpd::KnnVariant, -1 none): pinned per K, the
  // last one used for K, and per K and power of two of the rows the one picked
  // by a timed trial on this device
  signed char knn_pin[257], knn_last[257], knn_choice[rpd::kKnnTrialMaxK + 1][31];
  rpd_context() {
    std::memset(knn_pin, -1, sizeof(knn_pin));
    std::memset(knn_last, -1, sizeof(knn_last));
    std::memset(knn_choice, -1, sizeof(knn_choice));
  }
};

struct rpd_solver {
  rpd_context *ctx = nullptr;
  int n = 0;
  int dim = 0;
  rpd::DevBuf user;            // float4[n] as given
  rpd::DevBuf stored;          // float4[n] stored (binned) order
  rpd::DevBuf perm;            // int[n] stored -> user
  rpd::DevBuf user_to_stored;  // int[n]
  rpd::DevBuf weights;         // float[n]: staging for rpd_solver_set_weights
  rpd::DevBuf wmin;            // int[2]: the smallest weight of the seeds that are not walls
                               // (float_to_ordered); a flag of rpd_solver_set_weights
  rpd::DevBuf counters;        // int[dim^3+1]
  rpd::DevBuf bin_ws;
  rpd::DevBuf ring_bound;      // float[dim+2]
  rpd::DevBuf knn;             // unsigned[n*K]: every cell's neighbours (stored ids)
  int knn_full_K = 0;          // K of the table in knn for all n cells (0: none)
  int knn_full_Kx = 0;         // neighbours per row of that table
  int launches_since_points = 0;  // launches since the seeds were set (the outside probe runs on the first)
  long long grid_nonplain = -1;   // voxels of the grid that are not plainly outside (-1: not read yet)
  rpd::DevBuf knn_part;        // unsigned[num*K]: rows of a retry pass or a trace
  rpd::DevBuf knn_user;        // int[n*K]
  rpd::DevBuf counter64;       // unsigned long long[RPD_CTR_NUM + 1]
  // domain on the device
  rpd::DevBuf g_flags, g_points, g_tris, g_list, g_offsets, g_sat, g_tsat;
  rpd::DevGrid grid;           // grid.size == 0: no domain
  int grid_points = 0, grid_triangles = 0;  // of the domain's surface
  // results (stored order) and pass bookkeeping
  rpd::DevBuf out;             // double4[n]
  rpd::DevBuf status;          // int[n]
  rpd::DevBuf ids_a, ids_b, ids_c;  // int[n] failing-id lists
  rpd::DevBuf ids_range;       // int[count]: a part's stored ids (rpd_solver_launch_part)
  rpd::DevBuf tri_count;       // int[n]: triangle counts of the triangle overflows (CellLaunch::tri_count)
  rpd::DevBuf fail_ws;         // flags + scans
  rpd::DevBuf hist;            // int[16]: status histogram + counts
  rpd::DevBuf gather;          // user-order staging for outputs
  rpd::DevBuf defer_slots, defer_part, defer_fail, defer_ctr, defer_chunk_slot;  // parked boundary cells
  rpd::DevBuf hand_recs, hand_ctr;  // cells handed from the octet clipping to a warp
  rpd::DevBuf ahead;           // AheadRecord[n]: cells clipped past the first pass's caps
  bool ahead_on = false;       // in the current launch
  int level_P = 0, level_V = 0;                                  // growths of P and V so far
  int lad_P[rpd::kAheadLevels] = {}, lad_V[rpd::kAheadLevels] = {};  // the caps after each
  int ahead_max = 0;           // the largest triangle count the first pass parked ahead
  bool have_results = false;
  bool use_defer = true;       // park heavy boundary cells for the chunked kernel
  bool inner_apex = true;      // cone apex at a grid corner inside the cell
  bool fresh_knn = false;      // recompute the neighbour table at this launch
  int precision = 0;           // RPD_PRECISION_* of the clipping loop
  unsigned launch_flags = 0;   // RPD_FLAG_* of the current launch
  // used cells (keep_distance >= 0 with a domain)
  rpd::DevBuf used;            // unsigned char[n], stored order: 0 or the ring distance
  bool used_on = false;
  int keep_distance = -1;
  double keep_volume = 0.0;
  int used_count = -1;         // of the last launch, -1: none
  // --hessian rows (stored order) of the last launch with hessian_h > 0
  rpd::DevBuf hess;            // double[n*H*HC]
  rpd::DevBuf hessid;          // int[n*H]: stored ids, -1 after a row's last facet
  int hess_h = 0, hess_hc = 1; // of the last launch (0: no rows)
  rpd_stats stats{};
};

namespace rpd {
// Hooks of the serving loop (csrc/server.cu).
void solver_rebind(rpd_solver *s, rpd_context *ctx);
void solver_share_grid(rpd_solver *dst, const rpd_solver *src);
size_t solver_device_bytes(const rpd_solver *s);
void solver_trim(rpd_solver *s);
// Records for the clipped cells of a launch that need a warp: its boundary
// cells, whose share falls as the cell count grows.  (Launches with Hessian
// rows or used cells hand over all of their cells.)
int clip_hand_capacity(int num);

}  // namespace rpd
