// Per-seed restricted power cell: clipping, domain restriction, integration.
#pragma once
#include "common.cuh"

namespace rpd {

// Domain grid on the device (the reference Grid, Grid.h:14-70).
struct DevGrid {
  int size = 0;                       // voxels per axis
  float voxel = 0.f;                  // 1000 / size
  const signed char *flags = nullptr; // size^3 corner flags: 0 out, 1 border, 2 in
  const float4 *points = nullptr;     // triangle vertices (w unused)
  const int *tris = nullptr;          // 3 ids per triangle
  const int *list = nullptr;          // per-voxel sorted triangle ids
  const int *offsets = nullptr;       // size^3 + 1
  int has_border_corners = 0;         // any flag == 1
  // Summed-volume table, (size+1)^3, of voxels that are not plainly outside
  // (first-corner flag != 0 or a non-empty triangle list); null: unused.
  const int *sat = nullptr;
  // No triangle id appears in two voxel lists: the union of the lists of a
  // voxel range is their concatenation (no sort needed).
  int lists_disjoint = 0;
  // With disjoint lists: summed triangle counts, (size+1)^3, so a voxel
  // range's triangle count is 8 reads; null: unused.
  const int *tsat = nullptr;
};

// Counters of one launch (optional): cells by outcome and work done.
enum CellCounter {
  kCtrPlanesTested = 0,   // neighbour planes tested against the cell
  kCtrClips,              // clips that removed vertices
  kCtrVertexTests,        // vertex half-space tests
  kCtrVerticesMade,       // vertices created
  kCtrBoundaryCells,      // cells with at least one boundary triangle
  kCtrTriangles,          // boundary triangles processed
  kCtrExports,            // integrations (cell or cone pieces)
  kCtrExportVertices,     // vertices integrated
  kCtrOutside,            // cells proven outside the domain before the end of clipping
  kCtrConeEmpty,          // boundary triangles whose cone misses the cell
  kCtrConesSkipped,       // boundary triangles dropped: they miss the cell (apex inside it)
  kCtrEscTests,           // FP32 clipping: sign tests escalated to FP64
  kCtrEscVertices,        // FP32 clipping: vertices made in FP64 (near-degenerate)
  kCtrEscRadii,           // FP32 clipping: radius tests escalated to the exact FP64 radius
  kCtrStartCorner,        // boundary cells with cones from the reference's start corner
  kCtrNum
};

// Triangles of one work item of the cone kernels; a cell's sum adds its
// chunks' sums in order, also where a cell's own warp takes them all.  A warp
// takes four triangles at a time, about 30 us each time: a pass of few cells
// lasts as long as one item.  16 -> 8: 1K seeds 0.82 -> 0.65 ms, 100K in a
// blob 3.65 -> 3.39, 50K in a field 3.08 -> 2.84, 1M 11.8 -> 11.7; 48 uneven
// diagrams 60.6 -> 61.2 (more items load and prepare their cell).
constexpr int kConeChunk = 8;

// Boundary cells with many triangles park their clipped cell here; a second
// kernel spreads their triangles over all warps in chunks.
struct DeferQueue {
  unsigned char *slots = nullptr;  // capacity slots of slot_bytes
  int capacity = 0;
  size_t slot_bytes = 0;
  // [0] cells parked, [1] next work item (cells with an inner apex), [2]
  // chunks taken, [3] the largest triangle count parked ahead
  // (CellLaunch::T_ahead), [4] next work item (cells with the reference's
  // start corner), [5] cells that found a slot but no work items left, to be
  // solved again (kParkOverflow); zeroed before a pass
  int *counters = nullptr;
  // Work items are chunks, numbered compactly: a parked cell takes its
  // chunks' range from counters[2] and writes its slot for each of them
  int items = 0;                   // work items the arrays below hold (defer_items)
  int *chunk_slot = nullptr;       // items
  double *part = nullptr;          // items * 4 partial moments
  int *fail = nullptr;             // items: (triangle << 4) | status, or INT_MAX
  int chunk = kConeChunk;          // triangles per work item
  int inline_max = 16;             // cells with at most this many triangles stay inline
};

// Cells clipped with eight lanes each (clip_octet.cuh) that need a whole
// warp from there on, as records for the launch's finish kernel.
constexpr int kClipRecordBytes = 320;
constexpr int kClipCounters = 3;
struct ClipHand {
  unsigned char *recs = nullptr;  // capacity records
  int capacity = 0;
  // [0] cells handed over, [1] next record to finish, [2] cells left with
  // status kParkOverflow (no record free, or larger than the octet's caps) to
  // be solved by the warp-per-cell kernel; zeroed before a launch
  int *ctr = nullptr;
};

// Launches of fewer rows clip with a warp per cell: an octet's cell takes
// longer than a warp's, which only more cells at a time repay (uniform seeds,
// K 50, octet / warp: 2,000 rows 0.102 / 0.076 ms in the box and 0.145 /
// 0.122 in a cube domain, 4,000 rows 0.109 / 0.127 and 0.156 / 0.189, 16,000
// rows 0.205 / 0.377 and 0.295 / 0.547).  Batched launches whose rows only
// the device knows hold both kernels, one of which returns at once (four
// diagrams of 1K seeds in the box, every pass with eight lanes 1.23 ms, now
// 0.96; eight of 2K 1.83 -> 1.54).
constexpr int kOctetMinRows = 4096;

// What a cell that failed a cap of the first pass needs, known since the
// clipping went on past it (CellLaunch::ahead): the retry passes settle the
// cell from this record instead of clipping it again.
constexpr int kMaxT = 4096;
constexpr int kAheadLevels = 6;  // caps of the schedule: the first pass's, grown x1.5 one to five times
constexpr int kNoStop = 255;     // a level that stops the clipping nowhere (first passes record lists of up to 200)
struct AheadRecord {
  unsigned short need;  // neighbours it takes to the security radius (0: no record)
  // the neighbour at which the cap of each level stops the clipping (kNoStop:
  // none): before its plane test, and at its cut
  unsigned char jP[kAheadLevels], jV[kAheadLevels];
  unsigned short ntri;  // triangles its restriction needs, when more than the T of the recording pass (else 0)
};
static_assert(sizeof(AheadRecord) == 16, "ahead record size");

// The status of a recorded cell in a pass of K neighbours, T triangles and
// cap levels lP and lV: the first cap that stops it decides.
__host__ __device__ inline int ahead_status(const AheadRecord &r, int K, int T, int lP, int lV) {
  const int never = 1 << 16;
  const int p = lP < kAheadLevels && r.jP[lP] != kNoStop ? r.jP[lP] : never;
  const int v = lV < kAheadLevels && r.jV[lV] != kNoStop ? r.jV[lV] : never;
  const int first = p < v ? p : v, end = K < r.need ? K : r.need;
  if (first < end) return p <= v ? kPlaneOverflow : kVertexOverflow;
  if (r.need > K) return kSecurityRadiusNotReached;
  return r.ntri > T ? kTriangleOverflow : kSuccess;
}

// Whether a first pass of these caps clips past them, and the neighbours its
// rows hold then.  Measured: with tight caps 30 to 95% of the cells fail it,
// and the two passes that clip them again cost more than larger shared memory
// and neighbour rows -- 2M blue-noise seeds (K 20, P 25, V 30, 94% failing)
// 53.3 -> 37.4 ms on the device.  At K 50 .. 70, P 30, V 40 a few percent
// fail, and clipping past the caps loses: 1M weighted seeds 11.7 -> 12.7 ms,
// 100K 4.20 -> 4.42 ms.
__host__ __device__ inline bool ahead_pays(int K, int V) { return K <= 24 || (V <= 32 && K <= 200); }
__host__ __device__ inline int ahead_columns(int K) { return K <= 24 ? 48 : K; }

struct CellLaunch {
  const float4 *stored = nullptr;  // n seeds in stored order (reference frame)
  int n = 0;
  const unsigned *knn = nullptr;   // num rows of K stored neighbour ids
  int K = 0;
  int Kx = 0;                      // neighbours per row of knn (K, or more with ahead)
  const int *ids = nullptr;        // stored ids of the rows (null: row i = seed i)
  int num = 0;
  int P = 0, V = 0, T = 0;         // caps of this pass
  // clipping precision: 0 FP64; 1 mixed (FP32 with FP64 escalation, the FP64
  // clipping's decisions); 2 plain FP32 (float planes, no escalation)
  int precision = 0;
  // a cell whose clip succeeded and whose range holds more than T but at most
  // T_ahead triangles (with disjoint lists, counted by grid.tsat)
  // is parked now with all of them -- the result the retry passes would give
  // it -- its start corner found as they would (out_domain_ahead); 0: off
  int T_ahead = 0;
  int out_domain_ahead = 0;
  int *ahead_max = nullptr;  // the largest count parked ahead (atomicMax; null: defer.counters[3])
  float cube_eps = 0.f;            // box [-eps, 1000+eps]^3
  int out_domain = 0;              // GRID_OUT_DOMAIN fallback for the start corner
  int early_out = 1;               // stop clipping cells proven outside the domain (needs grid.sat)
  // Triangle counts of the cells that failed with triangle_overflow (n ints,
  // stored order; optional, with disjoint lists): the first pass of a launch
  // (tri_first) writes every row's (0: none); a later pass settles a row whose
  // count is above its T at once -- the clip would give the same cell and
  // the same overflow
  int *tri_count = nullptr;
  int tri_first = 0;
  const int *wmin = nullptr;       // the smallest weight of the seeds that are not walls
                                   // (float_to_ordered); null: no early exit
  int inner_apex = 1;              // cone apex at a grid corner inside the cell when there is one
  int safe_radius = 0;             // the weighted security-radius guard instead of the reference's test
  DevGrid grid;                    // grid.size == 0: no domain
  int *status = nullptr;           // n, stored order
  double4 *out = nullptr;          // n, stored order: (m*x, m*y, m*z, m)
  unsigned long long *counters = nullptr;  // kCtrNum, optional
  // Trace of one cell (debugging): every clip and integration of stored seed
  // `trace_seed` appended to `trace` as records of kTraceRecord doubles;
  // trace[0] counts the records.
  int trace_seed = -1;
  double *trace = nullptr;
  int trace_cap = 0;  // records
  DeferQueue defer;   // slots == null: every boundary cell inline
  int only_status = -1;  // >= 0: process only the rows whose status equals it
  cudaEvent_t after_cell = nullptr;  // recorded after the cell kernel, before the cone kernels
  // used cells (a domain only): a successful cell with mass >= keep_volume
  // sets used[sid] = 1 and, with mark_dist >= 1, marks its face neighbours;
  // border_d > 0: bordering pass, clip only and mark the neighbours border_d
  unsigned char *used = nullptr;
  double keep_volume = 0.0;
  int mark_dist = 0;
  int border_d = 0;
  int diag = 0;  // index of this diagram in a batched launch (parked cells record it)
  // --hessian (no defer queue): per cell a row of H facets, HC values each,
  // and their neighbours (stored ids, -1 after the last), stored order
  double *hess = nullptr;
  int *hessid = nullptr;
  int H = 0, HC = 1;
  ClipHand hand;  // recs == null: clip with a warp per cell
  // Records of the cells clipped past the first pass's caps (n, stored order;
  // null: off).  The first pass (ahead_first) writes every row's; the later
  // ones settle the rows that have one.  Not with counters, used cells,
  // Hessian rows or launches of one pass.
  AheadRecord *ahead = nullptr;
  int ahead_first = 0;
  int lP = 0, lV = 0;              // levels of P and V
  int ladP[kAheadLevels] = {}, ladV[kAheadLevels] = {};
  // A retry pass of few cells (retry) takes Kx neighbours where a cell does
  // not reach its radius with K, and parks cells of up to T_ahead triangles;
  // a cell that needs more than K, or more than T_sure, gets a record and its
  // status (kSuccess when all went well) is that of a later pass
  // (k_retry_status puts this one's).
  int retry = 0;
  int T_sure = kMaxT;
};
constexpr int kParkOverflow = 101;  // internal status: the queue was full
constexpr int kProbeMiss = 102;     // internal status: the outside probe proved nothing
constexpr int kDeferCounters = 6;   // ints of DeferQueue::counters
constexpr int kTraceRecord = 12;

// Largest caps of one build: P <= 255 (uchar plane ids in the reference,
// voronoi.cpp:867), V <= 256, T <= kMaxT.
constexpr int kMaxP = 255;
constexpr int kMaxV = 256;

// The T of the last retry pass that surely runs after a cell's triangle
// overflow in a pass of these caps: passes grow T x1.5 while the cell fails,
// up to max_extra more, and stop once P or K (assumed to grow in every pass)
// outgrow their limits (voronoi.cpp:867); 0 when no retry surely runs.
__host__ __device__ inline int t_ahead_cap(int P, int K, int T, int max_extra) {
  int ahead = 0;
  for (int j = 0; j < max_extra; ++j) {
    P = int(P * 1.5);
    K = int(K * 1.5);
    if (P > kMaxP || K > 256) break;
    T = int(T * 1.5) < kMaxT ? int(T * 1.5) : kMaxT;
    ahead = T;
  }
  return ahead;
}

// Work items for `capacity` parked cells of up to T triangles: what all of
// them could need, but at most the larger of one item per 32 triangles and of
// one per cell and surface triangle.  A triangle lies in a few cells, so with
// an apex inside, whose cells keep the triangles they meet, the last holds
// them all; cells that find none run again with their cones in their own
// warp.  40 bytes each: worst-case arrays of items of 8 triangles took 3.2 GB
// for 10M seeds at T 100 and 25.6 GB at T 1000, these 0.8 and 6.4.
inline int defer_items(size_t capacity, int T, size_t surface) {
  auto of = [&](int chunk) { return capacity * size_t(T > chunk ? (T + chunk - 1) / chunk : 1); };
  const size_t most = of(kConeChunk), usual = of(32), near = capacity + surface;
  const size_t items = usual > near ? usual : near;
  const size_t limit = 0x7fffffff;
  return int(most < items ? (most < limit ? most : limit) : (items < limit ? items : limit));
}

// Shared memory bytes one warp needs for these caps.
size_t cell_warp_smem(int P, int V, int T, bool grid);
// Bytes of one parked boundary cell for these caps.
size_t defer_slot_bytes(int P, int V, int T);
// k_cell over the rows; with a domain and a defer queue, also the chunked
// boundary-triangle kernel and the per-cell reduction (3 launches).
cudaError_t cell_launch(const CellLaunch &a, cudaStream_t st, int sm_count = 148, int *launches = nullptr);
// The same with eight lanes per cell (a.hand.recs; cell_octet.cu), and whether
// a launch's cells can be clipped so.
cudaError_t cell_launch_octet(const CellLaunch &a, cudaStream_t st, int sm_count, int *launches);
bool octet_applies(const CellLaunch &a);
// The same for a.precision > 0 (cell_prec.cu), and for FP64 clipping with
// the weighted security-radius guard (a.safe_radius; cell_safe.cu).
cudaError_t cell_launch_prec(const CellLaunch &a, cudaStream_t st, int sm_count, int *launches);
cudaError_t cell_launch_safe(const CellLaunch &a, cudaStream_t st, int sm_count, int *launches);

// Outside probe of a first pass with a domain.  The seeds of the 3x3x3 bins
// around a seed's own are a subset of all seeds, so their bisectors bound a
// region that contains the seed's power cell.  When that region fits the
// ball of plainly-outside voxels (flag 0, no triangle) around the seed, the
// cell is the domain's empty cell: status success and mass 0, as the full
// solve gives it.  Shown by a closed-form bound over 26 directions (balls of
// at least min_plain_cage) or by clipping with the 32 nearest of them
// (balls of at least min_plain).  Every other row gets kProbeMiss and is
// solved by the full pass.
struct ProbeLaunch {
  const float4 *stored = nullptr;  // n seeds in stored (bin) order
  int n = 0;                       // rows: the stored seeds first .. first + n - 1
  int first = 0;
  const int *bins = nullptr;       // dim^3 + 1 bin starts of the stored order
  int dim = 0;
  DevGrid grid;                    // with its summed-volume table (grid.sat)
  int P = 0, V = 0;                // caps of the first pass
  float cube_eps = 0.f;
  double min_plain_cage = 0.0;     // the cage test for balls at least this wide (reference frame)
  double min_plain = 0.0;          // clipping for balls at least this wide
  const int *wmin = nullptr;       // the smallest weight of the seeds that are not walls (float_to_ordered)
  int *status = nullptr;           // n, stored order
  double4 *out = nullptr;          // n, stored order
};
cudaError_t probe_launch(const ProbeLaunch &p, cudaStream_t st);
// The probe over every seed of many diagrams (batched solves): diagram d's
// record probes[d] (device) and rows start[d] .. start[d+1] (device; `rows`
// of them in all, known when the launch is made); P and V at least every
// diagram's first-pass caps.
cudaError_t probe_batch_launch(const ProbeLaunch *probes, const int *start, int ndiag, long rows, int P, int V,
                               cudaStream_t st);

// Whether one warp's layout for these caps fits a block's shared memory.
bool cell_caps_fit(int P, int V, int T, bool grid, int hc = 0);

// The cells of many diagrams in shared persistent launches (batched
// solves).  Row prefixes and launch records live on the device, written by
// earlier kernels of the same stream, so the launches can be captured in a
// graph before their row counts are known.
struct CellBatch {
  const CellLaunch *descs = nullptr;         // ndiag records; defer = the shared queue
  const CellLaunch *descs_inline = nullptr;  // the same records without the queue
  const int *start_grid = nullptr;   // ndiag+1 row prefixes of the diagrams with a domain (null: none)
  const int *start_plain = nullptr;  // ndiag+1 row prefixes of the diagrams without one (null: none)
  int ndiag = 0;
  DeferQueue defer;                  // slots == null: every boundary cell inline
  int P = 0, V = 0, T = 0;           // layout caps: at least every diagram's caps of this pass
  int T_slot = 0;                    // ids a parked cell's slot holds, when more than T (T_ahead)
  cudaEvent_t after_cell = nullptr;  // recorded (as a graph node when capturing) after the cell kernel
  // rows of the diagrams with / without a domain when known when the launch
  // is made (one warp per row), else -1 (persistent launches)
  long rows_grid = -1, rows_plain = -1;
  int *work = nullptr;  // one device int: the row counter of persistent launches (optional)
  bool safe = false;    // a diagram uses the weighted security-radius guard (its launch record decides)
  int HC = 0;           // Hessian rows' components (a diagram with rows; then no defer queue), else 0
  bool disjoint = false;  // every diagram's grid lists each triangle in one voxel (a smaller id buffer)
  ClipHand hand;          // recs != null: clip with eight lanes per cell (the records' hand too)
  bool ahead = false;     // a first pass with diagrams that clip past their caps (CellLaunch::ahead)
};
cudaError_t cell_batch_launch(const CellBatch &b, cudaStream_t st, int sm_count, int *launches = nullptr);
// The same with eight lanes per cell where the rows are many (b.hand.recs;
// cell_octet.cu), and with the guard compiled in (cell_safe.cu).
cudaError_t cell_batch_launch_octet(const CellBatch &b, cudaStream_t st, int sm_count, int *launches);
cudaError_t cell_batch_launch_safe(const CellBatch &b, cudaStream_t st, int sm_count, int *launches);

}  // namespace rpd
