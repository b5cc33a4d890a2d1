// Clipping with eight lanes per cell (an octet), four cells per warp: the
// launches' first kernel where it applies (octet_applies), followed by
// k_finish for the cells that need a whole warp (boundary cells, Hessian
// rows, used cells).
//
// Why: the warp-per-cell kernel (cell_row) is bound by instruction issue,
// not by memory or FP64 throughput: ~430 warp instructions per clip, of
// which most lanes take no part (8 to 30 vertices are tested, 3 to 8 new ones
// made, the cavity has 3 to 10 triangles).  With eight lanes per cell the
// same instructions serve four cells: 4.6K warp instructions per cell instead
// of 8.8K on 1M weighted lattice seeds in a blob (K 50), first pass 15.8 ->
// 7.1 ms with the finish kernel (6.1 + 1.0); 2M blue-noise seeds (K 20, P 25,
// V 30) 32.5 -> 10.0 ms.  What bounds it: instruction issue (2.67 of 4 per
// cycle) and instruction fetch -- the loop's code is kept small (seldom taken loops
// rolled, the end of a cell out of line): 8.4 -> 6.8 ms by that alone.
// Five or six blocks per SM, by registers (96 / 80) and shared memory (2.2 KB
// per cell at P 30, V 40); sixteen lanes would serve two cells only, four
// lanes need twice the shared memory per warp.
//
// Decisions are the FP64 clipping's, bit for bit.  A vertex is kept as its
// position rounded from the FP64 cofactor (float3, 16 bytes with its plane
// triple); a half-space test, a radius test or a voxel index decides in float
// where its value is farther than a bound of the rounding from the
// threshold, and otherwise recomputes the FP64 value from the FP64 planes
// with the FP64 clipping's own functions (vertices made in FP64 too).  The
// bound needs no per-vertex majorants since the positions come from FP64
// cofactors: with u = 2^-24 a position is within 4u |p_i| of the FP64 one per
// coordinate (cofactor, reciprocal and product rounded), the plane (n, d)
// within u, so the value n.p + d moves by at most 5u |p|_1 + u |d| and its
// evaluation adds 3u (|p|_1 + |d|); kTestErr takes 16u (sqrt(3) R + |d|), R
// the cell's radius.
//
// AHEAD (CellLaunch::ahead, where ahead_pays): a first pass with tight caps
// goes on past them and writes what the cell needs, so that the retry passes
// need not clip it again: 2M blue-noise seeds' pass 1 10.3 -> 20.4 ms, passes
// 2 to 5 29.2 -> 4.4 ms.
//
// Vertices keep the warp kernel's positions (holes filled by survivors in
// order, then by the new vertices in boundary order), so that the cell's
// later sums add the same terms in the same order.
#pragma once
#include "cell_kernels.cuh"

namespace rpd {

namespace {

constexpr int kOct = 8;           // lanes per cell
constexpr int kOctV = 64;         // most vertices of a cell here (64-bit masks)
constexpr int kOctP = 48;         // most planes (a Voronoi cell has about 15)
constexpr float kTestErr = 16.0f * kU32;
constexpr float kR2Err = 32.0f * kU32;  // relative bound of the float |p|^2 against the FP64 one

// A clipped cell handed to a warp: its planes as neighbour row positions
// (planes 0..5 are the box) and its vertices' plane triples.
struct ClipRecord {
  int row, diag;
  int np, nv;
  unsigned char nb[kOctP];
  unsigned tri[kOctV];
};
static_assert(sizeof(ClipRecord) == kClipRecordBytes, "clip record size");

// Shared memory of one cell.
struct OctLayout {
  int Pc, Vc;
  int mask4;  // 16-byte words of the edge masks, per lane
  unsigned o_vert, o_cand, o_mask, o_edge, o_next, o_nb, total;
};

// Fixed part of a cell's shared memory: the seed and the chunk of neighbours
// at hand (planes in FP64 and float).  Kept out of
// registers: the clipping loop spills without it.
struct OctCell {
  float4 s;
  Plane pl[kOct];
  float4 cand[kOct];
  // clipping past the caps (CellLaunch::ahead): the status under the caps (-1:
  // none of them reached), the last neighbour, and the record's levels
  int vst, last;
  unsigned char jP[kAheadLevels], jV[kAheadLevels], lP, lV;
  unsigned char pad[2];
};

// ahead: room to clip past caps P and V.
template <int MW>
__host__ __device__ inline OctLayout oct_layout(int P, int V, bool ahead = false) {
  OctLayout L;
  if (ahead) {
    P = P < 32 * MW ? 32 * MW : P;
    V += 8;
  }
  L.Pc = P < kOctP ? P : kOctP;
  L.Vc = V < kOctV ? (V + (ahead ? 15 : 7)) & (ahead ? ~15 : ~7) : kOctV;
  unsigned o = 32u * L.Pc;
  L.o_vert = o; o += 16u * L.Vc;
  L.o_cand = o; o += align16(unsigned(sizeof(OctCell)));
  L.mask4 = (L.Pc * MW + 31) / 32;
  L.o_mask = o; o += 128u * L.mask4;
  L.o_edge = o; o += align16(2u * 32 * MW);  // a manifold boundary has at most one edge per plane
  L.o_next = o; o += align16(L.Pc);
  L.o_nb = o; o += align16(L.Pc);
  L.total = o;
  return L;
}

// A condition that seldom holds: its code moves out of the hot path, which
// the instruction cache holds then.
__device__ __forceinline__ bool rare(bool c) { return __builtin_expect(c, 0); }

// Vertex from three planes as its rounded position and triple (x = NaN when
// the cofactor's sign is not the usual one: every test of it is then decided
// in FP64); false when degenerate, as make_vertex.
__device__ __forceinline__ bool oct_vertex(const Plane *pl, unsigned a, unsigned b, unsigned c, float4 &q) {
  double cx, cy, cz, cw;
  cofactor(pl[a], pl[b], pl[c], cx, cy, cz, cw);
  const float inv = __frcp_rn(float(cw));
  const float px = float(cx) * inv, py = float(cy) * inv, pz = float(cz) * inv;
  q = make_float4(cw < 0.0 ? px : __int_as_float(0x7fffffff), py, pz, __uint_as_float(a | (b << 8) | (c << 16)));
  // finite in float: far below make_vertex's limit
  return !rare(!(fabsf(px) + fabsf(py) + fabsf(pz) < 1e38f)) || vertex_d2(cx, cy, cz, cw) < 1e300;
}

// The FP64 clipping's half-space test of the vertex with triple t.
__device__ __noinline__ bool oct_cut_exact(const Plane *pl, unsigned t, const Plane &e) {
  double cx, cy, cz, cw;
  cofactor(pl[t & 0xff], pl[(t >> 8) & 0xff], pl[(t >> 16) & 0xff], cx, cy, cz, cw);
  return plane_side(cx, cy, cz, cw, e) > kTieEps * fabs(cw);
}

// The FP64 clipping's squared radius of the octet's cell.
__device__ __noinline__ double oct_radius2_exact(const Plane *pl, const float4 *vert, int nv, int l8) {
  double r = 0.0;
#pragma unroll 1
  for (int v = l8; v < nv; v += kOct) {
    const unsigned t = __float_as_uint(vert[v].w);
    double cx, cy, cz, cw;
    cofactor(pl[t & 0xff], pl[(t >> 8) & 0xff], pl[(t >> 16) & 0xff], cx, cy, cz, cw);
    r = fmax(r, vertex_d2(cx, cy, cz, cw));
  }
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) r = fmax(r, __shfl_xor_sync(kFull, r, o));
  return r;
}

// Integration of the octet's cell: integrate()'s terms and its sum tree over
// 32 lanes, lane l here holding that tree's leaves l, l+8, l+16, l+24.
__device__ __noinline__ void oct_integrate(const Plane *pl, const float4 *vert, int nv, int l8, double acc[4]) {
  double h[2][4];
#pragma unroll 1
  for (int b = 0; b < 2; ++b) {
    double p[4] = {0, 0, 0, 0};
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      double sx = 0, sy = 0, sz = 0, sw = 0;
#pragma unroll 1
      for (int v = l8 + kOct * (b + 2 * k); v < nv; v += 32) {
        const unsigned t = __float_as_uint(vert[v].w);
        double cx, cy, cz, cw;
        cofactor(pl[t & 0xff], pl[(t >> 8) & 0xff], pl[(t >> 16) & 0xff], cx, cy, cz, cw);
        integrate_vertex(pl, t, cx, cy, cz, cw, sx, sy, sz, sw);
      }
      p[0] += sx;
      p[1] += sy;
      p[2] += sz;
      p[3] += sw;
    }
    if (b == 0) {
      for (int d = 0; d < 4; ++d) h[0][d] = p[d];
    } else {
      for (int d = 0; d < 4; ++d) h[1][d] = p[d];
    }
  }
#pragma unroll
  for (int d = 0; d < 4; ++d) {
    double x = h[0][d] + h[1][d];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    acc[d] = __dmul_rn(x, 1.0 / 6.0);
  }
}

// plain_radius2 with the octet's lanes on the corners of one cube at a time:
// the first cube with a voxel that is not plainly outside, by bisection (the
// cubes grow).  chk: the octet takes part.
__device__ double oct_plain_radius2(const DevGrid &g, float4 s, bool chk, int l8) {
  const int S = g.size, S1 = S + 1;
  const double h = double(g.voxel);
  const double c[3] = {s.x, s.y, s.z};
  int v[3] = {0, 0, 0};
  if (chk) {
#pragma unroll
    for (int d = 0; d < 3; ++d) v[d] = min(S - 1, max(0, int(c[d] / h)));
  }
  // whether the cube of half-size k holds a voxel that is not plain
  auto hit = [&](int k) {
    int cnt = 0;
    if (chk) {
      const int x = (l8 & 1) ? min(S - 1, v[0] + k) + 1 : max(0, v[0] - k);
      const int y = (l8 & 2) ? min(S - 1, v[1] + k) + 1 : max(0, v[1] - k);
      const int z = (l8 & 4) ? min(S - 1, v[2] + k) + 1 : max(0, v[2] - k);
      const int t = __ldg(&g.sat[x + S1 * (y + S1 * z)]);
      cnt = ((l8 & 1) ^ ((l8 >> 1) & 1) ^ ((l8 >> 2) & 1)) ? t : -t;
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) cnt += __shfl_xor_sync(kFull, cnt, o);
    return cnt != 0;
  };
  const bool own = hit(0);
  if (!__any_sync(kFull, chk && !own)) return -1.0;
  int lo = 0, hi = 32;
#pragma unroll 1
  for (int it = 0; it < 5; ++it) {
    const int mid = (lo + hi) >> 1;
    if (hit(mid)) hi = mid;
    else lo = mid;
  }
  if (!chk || own) return -1.0;
  const int k = hi;
  double r = 1e300;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    if (v[d] - (k - 1) > 0) r = fmin(r, c[d] - (v[d] - (k - 1)) * h);
    if (v[d] + (k - 1) < S - 1) r = fmin(r, (v[d] + k) * h - c[d]);
  }
  r -= 1e-6 * h;
  return r > 0.0 ? (r >= 1e150 ? 1e300 : r * r) : -1.0;
}

// Position of set bit number k (0..7) of m, -1 when it has fewer.
__device__ __forceinline__ int nth_bit(unsigned long long m, int k) {
  const unsigned l = unsigned(m), h = unsigned(m >> 32);
  const int c = __popc(l);
  const bool up = k >= c;
  unsigned w = up ? h : l;
  k -= up ? c : 0;
  if (k & 4) {
    w &= w - 1;
    w &= w - 1;
    w &= w - 1;
    w &= w - 1;
  }
  if (k & 2) {
    w &= w - 1;
    w &= w - 1;
  }
  if (k & 1) w &= w - 1;
  return w ? __ffs(w) - 1 + (up ? 32 : 0) : -1;
}

// m with its k lowest set bits cleared.
__device__ __forceinline__ unsigned long long drop_bits(unsigned long long m, int k) {
#pragma unroll 1
  for (int i = 0; i < k; ++i) m &= m - 1;
  return m;
}

// Whether neighbour i of the row lies past twice the radius (the FP64
// clipping's own test, radius_reached).
__device__ __noinline__ bool oct_past(const CellLaunch &a, int row, int i, float4 s, double R2) {
  if (i < 0 || i >= a.Kx) return false;
  const unsigned z = __ldg(&a.knn[size_t(row) * a.Kx + i]);
  return z != kNone && seed_dist2(__ldg(&a.stored[z]), s) > 4.0 * R2;
}

// sqrt to within 2^-23.
__device__ __forceinline__ float approx_sqrt(float x) {
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

constexpr unsigned kFinWork = 1, kFinReclip = 2, kFinOdd = 4, kFinInside = 8;

// The end of a warp's four cells: the cells without boundary triangles are
// restricted, integrated and written, the others handed to a warp.  Out of
// line, so that the clipping loop has the registers to itself.
template <bool GRID>
__device__ __noinline__ void oct_finish(const CellLaunch &a, const OctLayout &L, unsigned char *osm, int row,
                                        unsigned flags, int status, int np, int nv, float m2, int lane) {
  const int l8 = lane & 7;
  const unsigned osh = lane & 24;
  Plane *plane = reinterpret_cast<Plane *>(osm);
  float4 *vert = reinterpret_cast<float4 *>(osm + L.o_vert);
  const unsigned char *pnb = osm + L.o_nb;
  auto oct_bits = [&](bool p) { return (__ballot_sync(kFull, p) >> osh) & 0xffu; };
  const bool work = flags & kFinWork, reclip = flags & kFinReclip, odd = flags & kFinOdd, inside = flags & kFinInside;
  const int sid = work ? (a.ids ? a.ids[row] : row) : 0;
  const OctCell &oc = *reinterpret_cast<const OctCell *>(osm + L.o_cand);
  const float4 s = oc.s;
  const int vst = oc.vst;  // >= 0: the cell passed a cap, its status for now
  bool ok = work && !reclip && status == kSuccess;
  bool hand = false, zero = false;  // goes on in a warp; mass 0
  if constexpr (GRID) {
    const DevGrid &g = a.grid;
    // proven outside the domain: the clipped cell fits the plainly-outside
    // ball around its seed (plain_radius2)
    const bool chk = ok && a.early_out && g.sat && inside;
    if (__any_sync(kFull, chk)) {
      const double plain2 = oct_plain_radius2(g, s, chk, l8);
      const double r2 = double(m2);
      zero = chk && !odd && r2 * (1.0 + kR2Err) <= plain2;
      const bool near = chk && !zero && plain2 >= 0.0 && (odd || r2 * (1.0 - kR2Err) <= plain2);
      if (__any_sync(kFull, near)) {
        const double R2 = oct_radius2_exact(plane, vert, nv, l8);
        if (near) zero = R2 <= plain2;
      }
    }
    bool open = ok && !zero;  // to be restricted
    if (open && (a.used || a.hess)) hand = true;
    open = open && !hand;
    if (__any_sync(kFull, open)) {
      // bounding box -> voxel range (restrict_to_domain), each index from
      // float positions where the rounding cannot change it
      float lo[3] = {3e38f, 3e38f, 3e38f}, hi[3] = {-3e38f, -3e38f, -3e38f};
      for (int v = l8; v < nv; v += kOct) {
        const float4 q = vert[v];
        lo[0] = fminf(lo[0], q.x);
        hi[0] = fmaxf(hi[0], q.x);
        lo[1] = fminf(lo[1], q.y);
        hi[1] = fmaxf(hi[1], q.y);
        lo[2] = fminf(lo[2], q.z);
        hi[2] = fmaxf(hi[2], q.z);
      }
#pragma unroll
      for (int d = 0; d < 3; ++d)
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) {
          lo[d] = fminf(lo[d], __shfl_xor_sync(kFull, lo[d], o));
          hi[d] = fmaxf(hi[d], __shfl_xor_sync(kFull, hi[d], o));
        }
      int vmin[3] = {0, 0, 0}, vmax[3] = {-1, -1, -1};
      if (open) {
        const int S = g.size;
        const double ih = 1.0 / double(g.voxel);
        const double mar = 8.0 * kU32 * sqrt(double(m2)) + 1e-9;
        const double c[3] = {s.x, s.y, s.z};
        bool same = !odd;
#pragma unroll
        for (int d = 0; d < 3; ++d) {
          const double l = double(lo[d]) + c[d], h = double(hi[d]) + c[d];
          vmin[d] = int(fmin(1000.0, l - mar) * ih - 1e-9);
          vmax[d] = int(fmax(0.0, h - mar) * ih - 1e-9);
          same &= vmin[d] == int(fmin(1000.0, l + mar) * ih + 1e-9) && vmax[d] == int(fmax(0.0, h + mar) * ih + 1e-9);
          vmin[d] = max(0, vmin[d]);
          vmax[d] = min(S - 1, vmax[d]);
        }
        if (!same || vmin[0] > vmax[0] || vmin[1] > vmax[1] || vmin[2] > vmax[2]) {
          hand = true;
          open = false;
        }
      }
      const int S = open ? g.size : 1;
      const int ex = vmax[0] - vmin[0] + 1, ey = vmax[1] - vmin[1] + 1, ez = vmax[2] - vmin[2] + 1;
      const int nvox = open ? ex * ey * ez : 0;
      int ntri = 0;
      if (open && g.tsat) {
        const int S1 = S + 1;
        const int x = (l8 & 1) ? vmax[0] + 1 : vmin[0], y = (l8 & 2) ? vmax[1] + 1 : vmin[1],
                  z = (l8 & 4) ? vmax[2] + 1 : vmin[2];
        const int t = __ldg(&g.tsat[x + S1 * (y + S1 * z)]);
        ntri = ((l8 & 1) ^ ((l8 >> 1) & 1) ^ ((l8 >> 2) & 1)) ? t : -t;
      } else if (open) {
        for (int q = l8; q < nvox; q += kOct) {
          const int vid = (vmin[0] + q % ex) + S * ((vmin[1] + (q / ex) % ey) + S * (vmin[2] + q / (ex * ey)));
          ntri += __ldg(&g.offsets[vid + 1]) - __ldg(&g.offsets[vid]);
        }
      }
#pragma unroll
      for (int o = 4; o > 0; o >>= 1) ntri += __shfl_xor_sync(kFull, ntri, o);
      if (open && ntri > 0) {
        if (g.tsat && ntri > a.T && (ntri > a.T_ahead || !a.defer.slots) && vst < 0) {
          if (a.tri_count && l8 == 0) a.tri_count[sid] = ntri;
          status = kTriangleOverflow;
          ok = false;
        } else {
          hand = true;
        }
        open = false;
      }
      // no triangle: the first corner with flag != 1 in (z, y, x) scan order
      // decides
      int f = 1;
      for (int b0 = 0; __any_sync(kFull, open && f == 1 && b0 < nvox); b0 += kOct) {
        const int q = b0 + l8;
        int fl = 1;
        if (open && f == 1 && q < nvox)
          fl = g.flags[(vmin[0] + q % ex) + S * ((vmin[1] + (q / ex) % ey) + S * (vmin[2] + q / (ex * ey)))];
        const unsigned fm = oct_bits(fl != 1);
        const int ff = __shfl_sync(kFull, fl, fm ? int(osh) + __ffs(fm) - 1 : int(osh));
        if (fm) f = ff;
      }
      if (open) {
        if (f == 0) zero = true;
        else if (f != 2) hand = true;  // no start corner yet: the warp kernel's fallback
      }
    }
  } else {
    if (ok && a.hess) hand = true;
  }
  if (vst >= 0 && hand) {
    // past a cap and with boundary triangles: left to the retry passes
    status = vst;
    ok = hand = false;
  }
  const bool sum = ok && !hand && !zero;
  double acc[4] = {0, 0, 0, 0};
  if (__any_sync(kFull, sum)) {
    double t[4];
    oct_integrate(plane, vert, sum ? nv : 0, l8, t);
    if (sum)
      for (int d = 0; d < 4; ++d) acc[d] = t[d];
  }
  if (!work) return;
  if (hand) {
    int k = 0;
    if (l8 == 0) k = atomicAdd(&a.hand.ctr[0], 1);
    k = __shfl_sync(0xffu << osh, k, int(osh));
    if (k < a.hand.capacity) {
      ClipRecord *r = reinterpret_cast<ClipRecord *>(a.hand.recs) + k;
      if (l8 == 0) {
        r->row = row;
        r->diag = a.diag;
        r->np = np;
        r->nv = nv;
      }
      for (int i = l8; i < np; i += kOct) r->nb[i] = pnb[i];
      for (int v = l8; v < nv; v += kOct) r->tri[v] = __float_as_uint(vert[v].w);
    } else if (l8 == 0) {
      a.status[sid] = kParkOverflow;
      atomicAdd(&a.hand.ctr[2], 1);
    }
    return;
  }
  if (l8 == 0) {
    if (reclip) {
      a.status[sid] = kParkOverflow;
      atomicAdd(&a.hand.ctr[2], 1);
      return;
    }
    a.status[sid] = ok && vst >= 0 ? vst : status;
    a.out[sid] = ok ? global_moments(acc, s) : make_double4(0.0, 0.0, 0.0, 0.0);
    if (ok && vst >= 0) {
      // a list that ended at `last` has no neighbour there whose plane test a
      // cap could stop
      const bool ended = __ldg(&a.knn[size_t(row) * a.Kx + oc.last]) == kNone;
      AheadRecord r;
      r.need = (unsigned short)(oc.last + 1);
      for (int k = 0; k < kAheadLevels; ++k) {
        r.jP[k] = ended && oc.jP[k] == oc.last ? kNoStop : oc.jP[k];
        r.jV[k] = oc.jV[k];
      }
      r.ntri = 0;
      a.ahead[sid] = r;
    }
  }
}

// One cell per octet: clip, and where the cell needs no boundary triangles,
// restrict, integrate and write.  act: the octet has row `row` of a.
// AHEAD: launches with a first pass that clips past its caps (a.ahead).
template <int MW, bool GRID, bool AHEAD>
__device__ __forceinline__ void clip_octet(const CellLaunch &a, const OctLayout &L, unsigned char *osm, int row,
                                           bool act, int lane) {
  const int l8 = lane & 7;
  const unsigned osh = lane & 24;  // the octet's first lane
  const unsigned lt8 = (1u << l8) - 1u;
  Plane *plane = reinterpret_cast<Plane *>(osm);
  float4 *vert = reinterpret_cast<float4 *>(osm + L.o_vert);
  OctCell &oc = *reinterpret_cast<OctCell *>(osm + L.o_cand);
  unsigned *mask = reinterpret_cast<unsigned *>(osm + L.o_mask);
  unsigned short *edge = reinterpret_cast<unsigned short *>(osm + L.o_edge);
  unsigned char *next = osm + L.o_next;
  unsigned char *pnb = osm + L.o_nb;
  auto oct_bits = [&](bool p) { return (__ballot_sync(kFull, p) >> osh) & 0xffu; };

  int status = kSuccess;
  bool run = act;
  float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
  if (act) {
    const int sid = a.ids ? a.ids[row] : row;
    s = __ldg(&a.stored[sid]);
    if (a.ahead && settle_ahead(a, sid, l8 == 0)) run = false;
    if (a.hess && l8 == 0) a.hessid[size_t(sid) * a.H] = -1;  // an empty row until the cell succeeds
    if (GRID && run && a.tri_count) {
      if (a.tri_first) {
        if (l8 == 0) a.tri_count[sid] = 0;
      } else if (a.tri_count[sid] > max(a.T, a.T_ahead)) {
        // clipped again it would be the same cell, past T again
        if (l8 == 0) {
          a.status[sid] = kTriangleOverflow;
          a.out[sid] = make_double4(0.0, 0.0, 0.0, 0.0);
        }
        run = false;
      }
    }
    if (run && s.w <= kNoCellLimits) {
      if (l8 == 0) {
        a.status[sid] = kSuccess;
        a.out[sid] = make_double4(s.x, s.y, s.z, s.w);
      }
      run = false;
    }
  }
  const bool work = run;  // the octet has a cell to clip
  bool reclip = false;    // left to the warp kernel: the caps here do not hold the cell, or its seed
  // the neighbours' ids, a chunk ahead of their use
  unsigned zn = kNone;
  const bool ahead = AHEAD && work && a.ahead && a.ahead_first;
  const int Kend = ahead ? a.Kx : a.K;  // neighbours at hand
  auto fetch = [&](int i) { zn = run && i < Kend ? __ldg(&a.knn[size_t(row) * a.Kx + i]) : kNone; };
  fetch(l8);
  if (l8 == 0) {
    oc.s = s;
    oc.vst = -1;
    if (ahead) {
      for (int k = 0; k < kAheadLevels; ++k) oc.jP[k] = oc.jV[k] = kNoStop;
      oc.lP = oc.lV = 0;
    }
  }
  int vst = -1;  // the status under the caps, once one of them is passed
  // the domain box
  {
    bool out = false;
    if (l8 < 6) {
      const Plane p = box_plane(s, work ? a.cube_eps : 0.f, l8);
      plane[l8] = p;
      out = p.w < 0.0;
    }
    // a seed outside the box: clipped to its end its cell may be empty, where
    // the warp kernel has proven it outside the domain before (a success)
    if (GRID && oct_bits(out) && run) {
      reclip = true;
      run = false;
    }
  }
  __syncwarp();
  {
    // its corners: exact, the planes being axis-parallel
    const unsigned t = box_vertex(l8);
    const unsigned has = 1u << (t & 0xff) | 1u << ((t >> 8) & 0xff) | 1u << ((t >> 16) & 0xff);
    vert[l8] = make_float4(has & 1u ? -float(plane[0].w) : float(plane[1].w),
                           has & 4u ? -float(plane[2].w) : float(plane[3].w),
                           has & 16u ? -float(plane[4].w) : float(plane[5].w), __uint_as_float(t));
  }
  __syncwarp();
  int np = 6, nv = 8;
  const int Pm = !work ? 0 : (ahead ? L.Pc : min(a.P, kOctP));
  const int Vm = ahead ? L.Vc : min(a.V, kOctV);
  bool inside = false;    // the seed surely lies in its own cell (nonempty_cell)
  bool cut = false;
  int i0 = -kOct, jj = kOct;  // neighbour i0 + jj comes next (jj == kOct: the next chunk's first)
  float nd2 = 0.f;        // squared distance of this lane's neighbour of the chunk
  float m2 = 0.f;         // the largest vertex |p|^2, float
  float rb = 0.f;         // the test bound's part for the cell's radius
  bool odd = false;       // a vertex of unusual sign: tests and radii in FP64
  unsigned vbits = 0, stop = 0;  // the chunk's neighbours: there; past twice the cell's radius
  unsigned long long rm = 0;
  auto radius = [&](int nvmax) {
    float m = 0.f;
#pragma unroll
    for (int v0 = 0; v0 < kOctV; v0 += kOct) {
      if (v0 >= nvmax) break;
      if (v0 + l8 < nv) {
        const float4 q = vert[v0 + l8];
        m = fmaxf(m, fmaf(q.x, q.x, fmaf(q.y, q.y, q.z * q.z)));
      }
    }
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(kFull, m, o));
    if (run) {  // a finished cell keeps its radius
      m2 = m;
      rb = kTestErr * 1.7321f * 1.0001f * approx_sqrt(m) + 1e-9f;
    }
  };
  // the reference's security radius (radius_reached) for the chunk
  auto stops = [&]() {
    const float r4 = 4.0f * m2;
    const bool valid = (vbits >> l8) & 1u;
    bool st = valid && !odd && nd2 > r4 * (1.0f + 2.0f * kR2Err);
    const bool near = valid && !st && (odd || nd2 > r4 * (1.0f - 2.0f * kR2Err));
    if (rare(__any_sync(kFull, near))) {
      // too close to call in float: the FP64 clipping's own test
      const double R2 = oct_radius2_exact(plane, vert, nv, l8);
      if (near) st = oct_past(a, row, i0 + l8, oc.s, R2);
    }
    stop = oct_bits(st);
  };
  radius(kOct);
  // the chunk's first neighbour that needs more than a test: past the chunk,
  // past the row, or with the planes used up (0 before the first chunk)
  int lim = 0;
  int smax = kOct;  // at least every octet's vertex count
  for (;;) {
    // ---- the next neighbour that cuts, for every octet ----
    for (;;) {
      bool need = run && !cut;
      if (!__any_sync(kFull, need)) break;
      if (__any_sync(kFull, need && jj >= lim)) {
        bool valid = (vbits >> l8) & 1u;
        if (need && jj == kOct) {
          i0 += kOct;
          jj = 0;
          valid = zn != kNone;
          double d = 0.0;
          if (valid) {
            const Plane pl = bisector(__ldg(&a.stored[zn]), oc.s, d);
            oc.pl[l8] = pl;
            oc.cand[l8] = plane_f(pl);
          }
          nd2 = float(d);
          fetch(i0 + kOct + l8);
          if (GRID && i0 == 0 && a.wmin) {
            const double d0 = __shfl_sync(0xffu << osh, d, int(osh));
            inside = nonempty_cell(oc.s, __ballot_sync(0xffu << osh, valid) >> osh, d0, a.wmin);
          }
        }
        __syncwarp();
        vbits = oct_bits(valid);
        stops();
        auto limit = [&]() {
          lim = np >= Pm || (AHEAD && ahead && vst < 0 && np >= a.P) ? 0 : (vbits == 0xffu ? kOct : __ffs(~vbits) - 1);
          if (AHEAD && ahead && vst < 0) lim = min(lim, max(a.K - i0, 0));
        };
        limit();
        if (need && jj >= lim) {
          const int i = i0 + jj;
          const bool there = i < Kend && ((vbits >> jj) & 1u);
          if (AHEAD && ahead && vst < 0) {
            if (i >= a.K) vst = kSecurityRadiusNotReached;
            else if (there && np >= a.P) vst = kPlaneOverflow;
          }
          bool on = false;
          if (i >= Kend) {
            status = AHEAD && vst >= 0 ? vst : kSecurityRadiusNotReached;
          } else if (there) {
            if (np < Pm) on = AHEAD;  // past a cap only
            else if (AHEAD && vst >= 0) status = vst;
            else if (np >= a.P) status = kPlaneOverflow;
            else reclip = true;
          }  // else fewer than K other seeds: all have been clipped
          if (AHEAD && on) limit();
          else run = need = false;
        }
      }
      const float4 e = oc.cand[jj & 7];
      const int nvt = need ? nv : 0;
      unsigned rl = 0, rh = 0;
      float nearest = 3e38f;
#pragma unroll
      for (int v0 = 0; v0 < kOctV; v0 += kOct) {
        if (v0 >= smax) break;
        float t = 3e38f;
        if (v0 + l8 < nvt) {
          const float4 q = vert[v0 + l8];
          t = fmaf(q.x, e.x, fmaf(q.y, e.y, fmaf(q.z, e.z, e.w)));
        }
        nearest = fminf(nearest, fabsf(t));
        const unsigned c = oct_bits(t < 0.f);
        if (v0 < 32) rl |= c << v0;
        else rh |= c << (v0 - 32);
      }
      unsigned long long rt = rl | (static_cast<unsigned long long>(rh) << 32);
      const float bound = fmaf(kTestErr, fabsf(e.w), rb);
      if (rare(__any_sync(kFull, need && (odd || !(nearest > bound))))) {
        // too close to call in float: the FP64 clipping's own test
        rt = 0;
#pragma unroll 1
        for (int v0 = 0; v0 < smax; v0 += kOct) {
          const int v = v0 + l8;
          bool c = false;
          if (v < nvt) {
            const float4 q = vert[v];
            const float t = fmaf(q.x, e.x, fmaf(q.y, e.y, fmaf(q.z, e.z, e.w)));
            c = fabsf(t) > bound ? t < 0.f : oct_cut_exact(plane, __float_as_uint(q.w), oc.pl[jj & 7]);
          }
          rt |= static_cast<unsigned long long>(oct_bits(c)) << v0;
        }
      }
      const bool past = (stop >> jj) & 1u;
      if (need) rm = rt;
      cut |= need && rt != 0;
      run = run && !(need && rt == 0 && past);  // reached
      jj += need && rt == 0 && !past ? 1 : 0;
    }
    if (!__any_sync(kFull, cut)) break;
    // ---- the cut ----
    const int pid = np;
    if (cut) {
      reinterpret_cast<float *>(&plane[pid])[l8] = reinterpret_cast<const float *>(&oc.pl[jj])[l8];
      if (l8 == 0) pnb[pid] = (unsigned char)(i0 + jj);
    }
    const unsigned long long live = nv >= 64 ? ~0ull : (1ull << nv) - 1ull;
    const int nrem = __popcll(rm), nkeep = nv - nrem;
    // the cavity boundary is found from the smaller side, in the warp
    // kernel's order (clip): its directed edges whose twin is not in it
    const bool from_kept = min(nrem, nkeep) <= 10 && nkeep < nrem;
    if (cut && nkeep == 0) {
      status = AHEAD && vst >= 0 ? vst : kEmptyCell;
      run = cut = false;
    }
    const unsigned long long side = cut ? (from_kept ? ~rm & live : rm) : 0ull;
    const int nside = __popcll(side);
    for (int k = 0; k < (MW == 1 ? 1 : L.mask4); ++k)
      reinterpret_cast<uint4 *>(mask)[l8 + kOct * k] = make_uint4(0, 0, 0, 0);
    const bool more = __any_sync(kFull, nside > kOct);  // a second round of eight
    const int pos0 = nth_bit(side, l8);  // the l8-th vertex of the side
    const unsigned long long m0 = pos0 >= 0 ? side >> pos0 << pos0 : 0ull;
    const unsigned t0 = pos0 >= 0 ? __float_as_uint(vert[pos0].w) : 0u;
    __syncwarp();
    {
      unsigned long long m = m0;
      unsigned t = t0;
#pragma unroll 1
      for (;;) {
        if (m) {
          const unsigned ta = t & 0xff, tb = (t >> 8) & 0xff, tc = (t >> 16) & 0xff;
          atomicOr(&mask[ta * MW + (MW > 1 ? tb >> 5 : 0)], 1u << (tb & 31));
          atomicOr(&mask[tb * MW + (MW > 1 ? tc >> 5 : 0)], 1u << (tc & 31));
          atomicOr(&mask[tc * MW + (MW > 1 ? ta >> 5 : 0)], 1u << (ta & 31));
        }
        if (!more) break;
        m = drop_bits(m, kOct);
        if (!__any_sync(kFull, m != 0)) break;
        t = m ? __float_as_uint(vert[__ffsll(m) - 1].w) : 0u;
      }
    }
    __syncwarp();
    int nb = 0;
    {
      unsigned long long m = m0;
      unsigned t = t0;
#pragma unroll 1
      for (;;) {
        bool b[3] = {false, false, false};
        if (m) {
#pragma unroll
          for (int k = 0; k < 3; ++k) {
            const unsigned u = (t >> (8 * k)) & 0xff, v = (t >> (8 * ((k + 1) % 3))) & 0xff;
            b[k] = !((mask[v * MW + (MW > 1 ? u >> 5 : 0)] >> (u & 31)) & 1u);
          }
        }
        const unsigned B0 = oct_bits(b[0]), B1 = oct_bits(b[1]), B2 = oct_bits(b[2]);
        int q = nb + __popc(B0 & lt8) + __popc(B1 & lt8) + __popc(B2 & lt8);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          if (!b[k]) continue;
          unsigned u = (t >> (8 * k)) & 0xff, v = (t >> (8 * ((k + 1) % 3))) & 0xff;
          if (from_kept) {
            const unsigned x = u;
            u = v;
            v = x;
          }
          if (q < 32 * MW) {
            edge[q] = (unsigned short)(u | (v << 8));
            next[u] = (unsigned char)q;
          }
          ++q;
        }
        nb += __popc(B0) + __popc(B1) + __popc(B2);
        if (!more) break;
        m = drop_bits(m, kOct);
        if (!__any_sync(kFull, m != 0)) break;
        t = m ? __float_as_uint(vert[__ffsll(m) - 1].w) : 0u;
      }
    }
    __syncwarp();
    // one cycle through all boundary edges, every plane starting one edge
    const bool many = __any_sync(kFull, cut && nb > kOct);
    bool bad = cut && (nb < 3 || nb > 32 * MW);
    const unsigned e0 = l8 < nb && cut ? edge[l8] : 0u;  // the octet's l8-th edge
    const unsigned eu = e0 & 0xff, ev = e0 >> 8;
    {
      const bool on = cut && !bad && l8 < nb;
      int succ = l8;
      if (on) {
        bad |= next[eu] != l8;
        succ = next[ev];
        if (succ >= nb || (edge[succ] & 0xff) != ev) {
          bad = true;
          succ = l8;
        }
      }
      if (!rare(many)) {
        int mn = l8;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const int om = __shfl_sync(kFull, mn, succ & 7, kOct);
          succ = __shfl_sync(kFull, succ, succ & 7, kOct);
          mn = min(mn, om);
        }
        const unsigned leaders = oct_bits(on && mn == l8);
        bad |= cut && __popc(leaders) != 1;
      } else {
#pragma unroll 1
        for (int q = l8 + kOct; q < nb && cut && !bad; q += kOct) bad |= next[edge[q] & 0xff] != q;
        if (cut && !bad && l8 == 0) {
          int q = 0, steps = 0;
#pragma unroll 1
          do {
            const unsigned v = edge[q] >> 8;
            q = next[v];
            if (q >= nb || (edge[q] & 0xff) != v) break;
            ++steps;
          } while (q != 0 && steps <= nb);
          bad |= q != 0 || steps != nb;
        }
      }
    }
    bad = oct_bits(bad) != 0;
    const int F = nkeep + nb;
    if (cut && bad) {
      status = AHEAD && vst >= 0 ? vst : kInconsistentBoundary;
      run = cut = false;
    }
    if (AHEAD && ahead && cut) {
      // the levels that this cut passes
      if (F > a.V && vst < 0) vst = kVertexOverflow;
      if (l8 == 0) {
        while (oc.lV < kAheadLevels && F > a.ladV[oc.lV]) oc.jV[oc.lV++] = (unsigned char)(i0 + jj);
        while (oc.lP < kAheadLevels && pid + 1 >= a.ladP[oc.lP]) oc.jP[oc.lP++] = (unsigned char)(i0 + jj + 1);
      }
    }
    if (cut && F > Vm) {
      if (AHEAD && vst >= 0) status = vst;
      else if (F > a.V) status = kVertexOverflow;
      else reclip = true;
      run = cut = false;
    }
    // the new vertices fill the removed positions in order and go on past
    // the last one; with fewer new vertices than removed ones the survivors
    // past the new count move into the first holes
    int dst0 = pos0;
    if (rare(__any_sync(kFull, cut && from_kept))) {
      if (from_kept) dst0 = nth_bit(rm, l8);
    }
    if (l8 >= nrem) dst0 = nv + (l8 - nrem);
    unsigned long long holes = rm;
    int nmov = 0, in_holes = nrem;
    if (rare(__any_sync(kFull, cut && nb < nrem))) {
      if (cut && nb < nrem) {
        const unsigned long long low = F >= 64 ? ~0ull : (1ull << F) - 1ull;
        const unsigned long long movers = ~rm & live & ~low;
        holes = rm & low;
        nmov = __popcll(movers);
        in_holes = __popcll(holes) - nmov;
#pragma unroll 1
        for (int k = l8; k < nmov; k += kOct)
          vert[__ffsll(drop_bits(holes, k)) - 1] = vert[__ffsll(drop_bits(movers, k)) - 1];
        dst0 = l8 < in_holes ? __ffsll(drop_bits(holes, nmov + l8)) - 1 : nv + (l8 - in_holes);
      }
    }
    bool degenerate = false, od = false;
#pragma unroll 1
    for (int q = l8; q < nb && cut; q += kOct) {
      const unsigned ed = q < kOct ? e0 : edge[q];
      const int dst = q < kOct ? dst0 : (q < in_holes ? __ffsll(drop_bits(holes, nmov + q)) - 1 : nv + (q - in_holes));
      float4 x;
      degenerate |= !oct_vertex(plane, unsigned(pid), ed & 0xff, ed >> 8, x);
      od |= !(x.x == x.x);
      vert[dst] = x;
    }
    __syncwarp();
    if (rare(__any_sync(kFull, degenerate || od))) {
      odd |= oct_bits(od) != 0;
      if (oct_bits(degenerate) != 0 && cut) {
        status = AHEAD && vst >= 0 ? vst : kInconsistentBoundary;
        run = cut = false;
      }
    }
    if (cut) {
      nv = F;
      np = pid + 1;
    }
    if (np >= Pm || (AHEAD && ahead && np >= a.P)) lim = 0;
    smax = __reduce_max_sync(kFull, run ? nv : 0);
    radius(smax);
    stops();
    if (cut) {
      if ((stop >> jj) & 1u) run = false;  // reached
      else ++jj;
    }
    cut = false;
  }

  const unsigned flags = (work ? kFinWork : 0u) | (reclip ? kFinReclip : 0u) | (odd ? kFinOdd : 0u) |
                         (inside ? kFinInside : 0u);
  if (AHEAD && ahead && l8 == 0) {
    oc.vst = vst;
    oc.last = i0 + jj;
  }
  __syncwarp();
  oct_finish<GRID>(a, L, osm, row, flags, status, np, nv, m2, lane);
}

template <int MW, bool GRID, bool AHEAD>
__global__ void __launch_bounds__(128, MW == 1 && !AHEAD ? 6 : 5)
    k_clip(const __grid_constant__ CellLaunch a, const __grid_constant__ OctLayout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  const int row = (blockIdx.x * blockDim.x + threadIdx.x) / kOct;
  if ((row & ~3) >= a.num) return;  // the whole warp
  clip_octet<MW, GRID, AHEAD>(a, L, smem + size_t(threadIdx.x / kOct) * L.total, row, row < a.num, lane);
}

// The rows of many diagrams (k_cell_batch's scheme): diagram d owns rows
// start[d] .. start[d+1].  work (optional, zeroed before the launch): warps
// take four rows at a time from it; null: one octet per row.  from: launches
// of fewer rows are another kernel's.
template <int MW, bool GRID, bool AHEAD>
__global__ void __launch_bounds__(128, 5)
    k_clip_batch(const CellLaunch *__restrict__ descs, const int *__restrict__ start, int ndiag,
                 const __grid_constant__ OctLayout L, int from, int *__restrict__ work) {
  extern __shared__ __align__(16) unsigned char smem[];
  const int lane = threadIdx.x & 31;
  unsigned char *osm = smem + size_t(threadIdx.x / kOct) * L.total;
  const int total = start[ndiag];
  if (total < from) return;
  int r0 = (blockIdx.x * blockDim.x + threadIdx.x) / 32 * 4;
  for (;;) {
    if (work) {
      r0 = lane == 0 ? atomicAdd(work, 4) : 0;
      r0 = __shfl_sync(kFull, r0, 0);
    }
    if (r0 >= total) break;
    const int r = r0 + lane / kOct;
    const bool act = r < total;
    const int d = owner_of_row(start, ndiag, act ? r : r0);
    clip_octet<MW, GRID, AHEAD>(descs[d], L, osm, r - start[d], act, lane);
    if (!work) break;
    __syncwarp();
  }
}

// The clipped cells handed over by k_clip, one warp each, taken from a
// counter: the warp kernel's state is rebuilt from the record (planes from
// the neighbours, vertices from their triples, as the clipping made them).
template <int VS, bool GRID, bool INL, class Desc>
__device__ __forceinline__ void finish_records(const ClipHand &hd, const Layout &L, Desc desc, unsigned char *wsmem,
                                               int lane) {
  const int count = min(*(volatile int *)&hd.ctr[0], hd.capacity);
  for (;;) {
    int k = 0;
    if (lane == 0) k = atomicAdd(&hd.ctr[1], 1);
    k = __shfl_sync(kFull, k, 0);
    if (k >= count) break;
    const ClipRecord *r = reinterpret_cast<const ClipRecord *>(hd.recs) + k;
    const CellLaunch &a = desc(r->diag);
    WarpCell w = bind(wsmem, L);
    if constexpr (Desc::kBatch) w.vc = vertex_capacity(a, L);
    const int row = r->row, np = r->np, nv = r->nv;
    const int sid = a.ids ? a.ids[row] : row;
    const float4 s = a.stored[sid];
    const unsigned *nrow = a.knn + size_t(row) * a.Kx;
    const bool track = (GRID && a.used) || (INL && a.hess);
    for (int i = lane; i < np; i += 32) {
      int z = -1;
      if (i < 6) {
        w.plane[i] = box_plane(s, a.cube_eps, i);
      } else {
        z = int(__ldg(&nrow[r->nb[i]]));
        double d2;
        w.plane[i] = bisector(__ldg(&a.stored[z]), s, d2);
      }
      if (track) w.pnb[i] = z;
    }
    if constexpr (INL) {
      if (w.harea)
        for (int i = lane; i < w.hc * (L.Pc + 4); i += 32) w.harea[i] = 0.0;
    }
    __syncwarp();
    for (int v = lane; v < nv; v += 32) {
      const unsigned t = r->tri[v];
      make_vertex(w, v, t & 0xff, (t >> 8) & 0xff, (t >> 16) & 0xff);
    }
    __syncwarp();
    w.np = np;
    w.nv = nv;
    finish_cell<VS, GRID, INL>(w, a, L, s, sid, kSuccess, false, lane, nullptr, 0);
    __syncwarp();  // the warp's shared memory is reused by its next cell
  }
}

template <int VS, bool GRID, bool INL>
__global__ void __launch_bounds__(128, 5) k_finish(const __grid_constant__ CellLaunch a, const __grid_constant__ Layout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  finish_records<VS, GRID, INL>(a.hand, L, SingleDesc{&a}, smem + size_t(threadIdx.x >> 5) * L.total,
                                threadIdx.x & 31);
}

template <int VS, bool GRID, bool INL>
__global__ void __launch_bounds__(128, 5)
    k_finish_batch(const CellLaunch *__restrict__ descs, const __grid_constant__ ClipHand hd,
                   const __grid_constant__ Layout L) {
  extern __shared__ __align__(16) unsigned char smem[];
  finish_records<VS, GRID, INL>(hd, L, BatchDesc{descs}, smem + size_t(threadIdx.x >> 5) * L.total, threadIdx.x & 31);
}

}  // namespace

}  // namespace rpd
