// walk.cu -- face-adjacency tet walk (MeshManager::next_element /
// walk_elements, mesh_manager_interface.cpp:106-200) on the GPU.
//
// One thread walks one track.  Each step tests the four faces of the current
// tet for an exiting Plucker hit (orientation +1, plucker.h:64-161), takes
// the nearest (strict <, lowest face index on ties, :186-196), emits
// (element id, min(exit, remaining)) -- zero-length segments included -- and
// moves r += len * u in FP64, exactly like :117-133.
//
// The FP64 variant evaluates the tet's six edge coordinates in FP64 and takes
// the distance to the faces their signs leave.  The mixed
// variant first evaluates the six edge coordinates of the tet once in FP32
// (each face uses three of them, with a sign flip when it runs an edge
// backwards -- the exact coordinates of opposite directions are exact
// negatives) and skips a face only when some coordinate is certainly
// positive, which makes the FP64 test exit early (plucker.h:83-113).  The
// remaining faces -- normally just the exit face -- are evaluated in FP64
// with the reference's operations, so lengths and element sequences are
// bit-identical.
//
// What bounds it: the FP64 unit, 39 ns a warp instruction.  The exact test of
// the exit face is some 75 FP64 operations a step; the products among them
// run on the integer pipes instead (imul64.cuh), beside the sums.
//
// FP32 bound for a tet (u = 2^-24, D = |u|_inf, W = max |v_k - r|_inf,
// Av = max |v_k|_inf, A = Av + |r|_inf; vertices and r rounded to FP32
// individually, edges e = v_b - v_a so |e| <= 2W):
//    |pip32 - pip| <= u D W (97 W + 13 Av + 13 A)
// (gamma_5 rounding of the triple product plus the input perturbations; the
// FP64 evaluation error and the 20*DBL_EPSILON snap are added as in geom.cuh).
#include "walk.h"

#include <algorithm>
#include <atomic>

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>

#include "imul64.cuh"
#include "internal.cuh"
#include "sample.cuh"

namespace xdgcu {

namespace {

constexpr int kBlock = 128;
constexpr float kU32 = 5.9604645e-08f;

// MOAB canonical face order (moab/direct_access.h:181-183)
__device__ __forceinline__ constexpr int moab_face(int f, int j) {
  return (f == 0) ? (j == 0 ? 0 : (j == 1 ? 1 : 3))
         : (f == 1) ? (j == 0 ? 1 : (j == 1 ? 2 : 3))
         : (f == 2) ? (j == 0 ? 2 : (j == 1 ? 0 : 3))
                    : (j == 0 ? 0 : (j == 1 ? 2 : 1));
}

template <int FO>
__device__ __forceinline__ int face_local(const WalkArgs& a, int f, int j) {
  if (FO == 0) return moab_face(f, j);
  return a.face[3 * f + j];
}

template <typename T>
__device__ __forceinline__ T sel4(const T* v, int k) {
  return k == 0 ? v[0] : (k == 1 ? v[1] : (k == 2 ? v[2] : v[3]));
}

template <typename T>
__device__ __forceinline__ T sel6(const T* v, int k) {
  return k == 0 ? v[0]
                : (k == 1 ? v[1] : (k == 2 ? v[2] : (k == 3 ? v[3] : (k == 4 ? v[4] : v[5]))));
}

__device__ __forceinline__ float triple32(float dx, float dy, float dz, float ex, float ey,
                                          float ez, float wx, float wy, float wz) {
  const float cx = ey * wz - ez * wy;
  const float cy = ez * wx - ex * wz;
  const float cz = ex * wy - ey * wx;
  return dx * cx + dy * cy + dz * cz;
}

// index of the unordered vertex pair (i, j), i != j, in
// (0,1),(0,2),(0,3),(1,2),(1,3),(2,3)
__device__ __forceinline__ int pair_index(int i, int j) {
  const int a = i < j ? i : j, b = i < j ? j : i;
  return a == 0 ? b - 1 : (a == 1 ? b + 1 : 5);
}

// (32-bit: a thread's share of one launch stays far below 2^32)
struct StepCnt {
  uint32_t steps, esc;
};

// A tet's record (WalkArgs::rec): its vertices, neighbours, edge references and
// mesh id, 64 bytes in one line, so that a step fetches all it needs of the
// tet at once instead of from four arrays.
struct TetRec {
  int32_t v[4], adj[4], edge[6], id;
};

__device__ __forceinline__ TetRec load_rec(const WalkArgs& a, int32_t elem) {
  const int4* p = a.rec + 4 * (int64_t)elem;
  const int4 v = __ldg(p), n = __ldg(p + 1), e = __ldg(p + 2), f = __ldg(p + 3);
  return {{v.x, v.y, v.z, v.w}, {n.x, n.y, n.z, n.w}, {e.x, e.y, e.z, e.w, f.x, f.y}, f.z};
}

// The edge from local vertex la to lb of a tet (its six edge references at
// te): the edge's index, bit 31 set when the test runs it against first()
// order (the reference negates the coordinate then, plucker.h:48).
__device__ __forceinline__ int32_t edge_ref(const int32_t te[6], int la, int lb) {
  const int32_t ref = sel6(te, pair_index(la, lb));
  const bool second_is_lo = ref < 0;
  const bool la_is_lo = second_is_lo == (la > lb);
  return (ref & 0x7fffffff) | (la_is_lo ? 0 : (int32_t)0x80000000);
}

// plucker64 for the face (l0, l1, l2) of tet `tet` (vertex indices ci), its
// three edge coordinates taken from the mesh's edge table: the same values
// plucker_edge64 computes from the vertices, for a third of the FP64
// operations.  Only component plucker_axis(u) of the vertices is read.
__device__ __forceinline__ bool plucker64_face_pre(const WalkArgs& a, int32_t tet,
                                                   const int32_t ci[4], int l0, int l1, int l2,
                                                   d3 r, d3 u, d3 rn, double* t) {
  const TetRec T = load_rec(a, tet);
  const int32_t* te = T.edge;
  auto coord = [&](int la, int lb) {
    const int32_t ref = edge_ref(te, la, lb);
    return plucker_edge_pre(a.edge + 6 * (int64_t)(ref & 0x7fffffff), ref < 0, u, rn);
  };
  const double c0 = coord(l0, l1), c1 = coord(l1, l2), c2 = coord(l2, l0);
  const int idx = plucker_axis(u);
  const double v0i = __ldg(&a.xyz[3 * (int64_t)sel4(ci, l0) + idx]);
  const double v1i = __ldg(&a.xyz[3 * (int64_t)sel4(ci, l1) + idx]);
  const double v2i = __ldg(&a.xyz[3 * (int64_t)sel4(ci, l2) + idx]);
  return plucker64_coords(c0, c1, c2, v0i, v1i, v2i, comp3(r, idx), comp3(u, idx), INFTY, 0.0,
                          true, 1, t);
}

// ---------------------------------------------------------------------------
// The step's exact arithmetic with its products on the integer pipes
// (imul64.cuh).  A step takes this path when the mesh's coordinates
// (WalkArgs::int_ok), the track's direction and its position are in range;
// any other step takes the *_hw functions, whose products run on the FP64
// unit.  Those are not inlined: a predicated-off FP64 instruction holds the
// FP64 unit like one that runs, so the path not taken has to stay behind a
// real branch.  FP64 unit instructions a step: mixed 81 -> 43, FP64 396 -> 57
// (r += len * u stays there: its three products made no difference).
// ---------------------------------------------------------------------------

__device__ __forceinline__ bool in_range3(d3 v) {
  return in_range(v.x) && in_range(v.y) && in_range(v.z);
}

// a * b on the integer pipes (INT) or the FP64 unit
template <bool INT>
__device__ __forceinline__ double mul_p(double a, double b) {
  return INT ? mul_int(a, b) : a * b;
}

template <bool INT>
__device__ __forceinline__ double dot3_p(d3 a, d3 b) {
  return mul_p<INT>(a.x, b.x) + mul_p<INT>(a.y, b.y) + mul_p<INT>(a.z, b.z);
}

template <bool INT>
__device__ __forceinline__ d3 cross3_p(d3 a, d3 b) {
  return mk3(mul_p<INT>(a.y, b.z) - mul_p<INT>(a.z, b.y),
             mul_p<INT>(a.z, b.x) - mul_p<INT>(a.x, b.z),
             mul_p<INT>(a.x, b.y) - mul_p<INT>(a.y, b.x));
}

// plucker_edge_pre for a reference of edge_ref()
template <bool INT>
__device__ __forceinline__ double edge_coord_p(const double* edge, int32_t ref, d3 u, d3 rn) {
  const double* E = edge + 6 * (int64_t)(ref & 0x7fffffff);
  const double2 a = __ldg(reinterpret_cast<const double2*>(E));
  const double2 b = __ldg(reinterpret_cast<const double2*>(E + 2));
  const double2 c = __ldg(reinterpret_cast<const double2*>(E + 4));
  double pip = dot3_p<INT>(u, mk3(b.y, c.x, c.y)) + dot3_p<INT>(rn, mk3(a.x, a.y, b.x));
  pip = __longlong_as_double(__double_as_longlong(pip) ^ ((long long)(ref & 0x80000000) << 32));
  if (absbits(pip) < absbits(ZERO_TOL)) pip = 0.0;
  return pip;
}

__device__ __noinline__ bool sum_above_one(double a, double b) { return dlt(1.0, a + b); }

// The exit distance through one face, as face_distance_p, from the edge
// table with the products on the FP64 unit: edge references e0..e2 of
// edge_ref(), vertex indices i0..i2.
__device__ __noinline__ double face_exit_hw(const double* edge, const double* xyz, int32_t e0,
                                            int32_t e1, int32_t e2, int32_t i0, int32_t i1,
                                            int32_t i2, d3 r, d3 u) {
  const d3 rn = cross3(u, r);
  const double c0 = plucker_edge_pre(edge + 6 * (int64_t)(e0 & 0x7fffffff), e0 < 0, u, rn);
  const double c1 = plucker_edge_pre(edge + 6 * (int64_t)(e1 & 0x7fffffff), e1 < 0, u, rn);
  const double c2 = plucker_edge_pre(edge + 6 * (int64_t)(e2 & 0x7fffffff), e2 < 0, u, rn);
  const int idx = plucker_axis(u);
  double t;
  const bool hit =
      plucker64_coords(c0, c1, c2, __ldg(&xyz[3 * (int64_t)i0 + idx]),
                       __ldg(&xyz[3 * (int64_t)i1 + idx]), __ldg(&xyz[3 * (int64_t)i2 + idx]),
                       comp3(r, idx), comp3(u, idx), INFTY, 0.0, true, 1, &t);
  return hit ? (gt0(t) ? t : 0.0) : INFTY;
}

// the same from the vertices (a mesh without an edge table)
__device__ __noinline__ double face_exit_xyz(const double* xyz, int32_t i0, int32_t i1, int32_t i2,
                                             d3 r, d3 u) {
  double t;
  const bool hit = plucker64(load3(xyz, i0), load3(xyz, i1), load3(xyz, i2), r, u, cross3(u, r),
                             INFTY, 0.0, true, 1, &t);
  return hit ? (gt0(t) ? t : 0.0) : INFTY;
}

// FP32 value nearest to x (to even), by integer operations: a conversion
// instruction holds the FP64 unit for 33 ns a warp.  Magnitudes below FLT_MIN
// give 0 (an error below 2^-126: of a position far inside the filter's
// absolute term, of a direction see step_dir).
__device__ __forceinline__ float f32_near(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned long long q = b + 0x0fffffffull + ((b >> 29) & 1ull);
  const unsigned hi = (unsigned)(q >> 32);
  const unsigned e = (hi >> 20) & 0x7ffu;
  const unsigned sign = (unsigned)(b >> 32) & 0x80000000u;
  if (e <= 896u) return __uint_as_float(sign);
  if (e >= 1151u) return __uint_as_float(sign | 0x7f800000u);
  return __uint_as_float(sign | ((unsigned)(q >> 29) - (896u << 23)) & 0x7fffffffu);
}

// What a step needs of the track's direction, set when it changes.
struct StepDir {
  float x, y, z;  // FP32, nearest (x is NaN where FP32 may not decide)
  int axis;       // plucker_axis
  bool safe;      // the mesh and the direction are in range (imul64.cuh)
};

__device__ __forceinline__ StepDir step_dir(const WalkArgs& a, d3 u) {
  StepDir s;
  s.x = f32_near(u.x);
  s.y = f32_near(u.y);
  s.z = f32_near(u.z);
  // The filter's bound has a term u D W^2 for the direction's rounding, which
  // covers a component flushed to zero (2^-126 W^2) only for a longer D; with
  // NaN no FP32 coordinate is above the bound and every face is tested.
  if (!(fmaxf(fabsf(s.x), fmaxf(fabsf(s.y), fabsf(s.z))) >= 0x1p-100f)) s.x = NAN;
  s.axis = plucker_axis(u);
  s.safe = a.edge && a.int_ok && in_range3(u);
  return s;
}

// Lanes of a track.  G = 4: four neighbouring lanes hold the same track and go
// the same way; in a safe step they share its independent values (a component
// of u x r, an edge's coordinate, a weight) and hand them round.  A step of a
// lone warp is a chain of some 1,900 instructions and 43 FP64 ones, 32 lanes
// wide or one; shared it is two thirds of that, for a quarter of the tracks a
// warp, so small batches walk this way (kTeamWarps).  1,000 tracks located and
// walked: mixed 1.34 -> 1.10 ms, all-FP64 1.85 -> 1.35; 1,000 particles of the
// walk_elements loop 6.0 -> 5.1 ms.
template <int G>
struct Team {
  unsigned mask;
  int q;  // the lane's place in its team
  __device__ __forceinline__ Team() {
    const int lane = threadIdx.x & 31;
    q = G > 1 ? lane & (G - 1) : 0;
    mask = G > 1 ? ((1u << G) - 1u) << (lane & ~(G - 1)) : 0u;
  }
  __device__ __forceinline__ double from(double v, int place) const {
    return G > 1 ? __shfl_sync(mask, v, place, G) : v;
  }
  __device__ __forceinline__ d3 gather(double v) const {
    return mk3(from(v, 0), from(v, 1), from(v, 2));
  }
};

// plucker64_coords for the walk's call (orientation +1, distances 0 ..
// INFTY), for coordinates that are all <= 0 and not all 0: max(0, distance),
// or INFTY for no hit.  The weights are >= 0, and their sum is tested only
// where it can exceed 1: w1 >= 2^-48 keeps w0 + w2 below 1, since the
// weights' sum is within 6 eps of 1.
template <bool INT, int G>
__device__ __forceinline__ double face_distance_p(const Team<G>& team, double c0, double c1,
                                                  double c2, const double* xyz, int32_t i0,
                                                  int32_t i1, int32_t i2, double oi, double di) {
  // (xyz: the vertices' components along plucker_axis)
  auto comp = [&](int32_t i) { return __ldg(&xyz[3 * (int64_t)i]); };
  const double inv = 1.0 / (c0 + c1 + c2);
  double w0, w1, w2, hit;
  if (G == 1) {
    w0 = mul_p<INT>(c0, inv);
    w1 = mul_p<INT>(c1, inv);
    w2 = mul_p<INT>(c2, inv);
    hit = (mul_p<INT>(w0, comp(i2)) + mul_p<INT>(w1, comp(i0))) + mul_p<INT>(w2, comp(i1));
  } else {
    const int k = team.q == 3 ? 0 : team.q;
    const double w = mul_p<INT>(k == 0 ? c0 : (k == 1 ? c1 : c2), inv);
    const d3 p = team.gather(mul_p<INT>(w, comp(k == 0 ? i2 : (k == 1 ? i0 : i1))));
    w0 = team.from(w, 0);
    w1 = team.from(w, 1);
    w2 = team.from(w, 2);
    hit = (p.x + p.y) + p.z;
  }
  double t = (hit - oi) / di;
  if (absbits(w1) < 0x3cf0000000000000ull && sum_above_one(w2, w0)) t = -1.0;
  if (lt0(t) || dlt(INFTY, t)) return INFTY;
  return gt0(t) ? t : 0.0;
}

template <int G>
__device__ __forceinline__ d3 walk_move(const Team<G>& team, d3 r, double len, d3 u) {
  if (G == 1) return add3(r, scl3(len, u));
  const int k = team.q == 3 ? 0 : team.q;
  return team.gather(comp3(r, k) + len * comp3(u, k));
}

// MeshManager::next_element for the tet of record T at r along u.  Returns the face
// index (or -1) and writes the exit distance.
// INT: the products of a safe step run on the integer pipes.
template <int FO, bool MIXED, bool INT = true, int G = 1>
__device__ __forceinline__ int next_face(const WalkArgs& a, const TetRec& T, d3 r, d3 u,
                                         const StepDir& sd, bool safe, double* exit_dist,
                                         StepCnt& cnt, const Team<G>& team = Team<G>()) {
  const int32_t* ci = T.v;
  const int32_t* te = T.edge;
  const int tq = team.q == 3 ? 0 : team.q;  // the value of three that this lane evaluates
  // the faces that may be the exit face: only these take the distance below
  unsigned escm = 0u;
  d3 rn = mk3(0.0, 0.0, 0.0);
  double pe[6];  // FP64 path: the six coordinates, pair (i, j), i < j, run i -> j
  if (safe) {  // plucker.h:75
    if (G == 1) {
      rn = cross3_p<INT>(u, r);
    } else {
      const int k1 = tq == 2 ? 0 : tq + 1, k2 = tq == 0 ? 2 : tq - 1;
      rn = team.gather(mul_p<INT>(comp3(u, k1), comp3(r, k2)) -
                       mul_p<INT>(comp3(u, k2), comp3(r, k1)));
    }
  }
  if (!MIXED) {
    escm = 0xfu;
    if (safe) {
      escm = 0u;
      // (a record's own references run their pairs i -> j)
      if (G == 1) {
#pragma unroll
        for (int k = 0; k < 6; ++k) pe[k] = edge_coord_p<INT>(a.edge, te[k], u, rn);
      } else {
        const double p = edge_coord_p<INT>(a.edge, sel4(te, team.q), u, rn);
        const double p4 = edge_coord_p<INT>(a.edge, (team.q & 1) ? te[5] : te[4], u, rn);
#pragma unroll
        for (int k = 0; k < 4; ++k) pe[k] = team.from(p, k);
        pe[4] = team.from(p4, 0);
        pe[5] = team.from(p4, 1);
      }
#pragma unroll
      for (int f = 0; f < 4; ++f) {
        const int l[3] = {face_local<FO>(a, f, 0), face_local<FO>(a, f, 1),
                          face_local<FO>(a, f, 2)};
        bool out = false, zero = true;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          const int la = l[q], lb = l[(q + 1) % 3];
          const double p = sel6(pe, pair_index(la, lb));
          out |= la < lb ? gt0(p) : lt0(p);  // a positive coordinate rejects (plucker.h:83-113)
          zero &= is0(p);
        }
        if (!out && !zero) escm |= 1u << f;
      }
    }
    if (team.q == 0) cnt.esc += 4;  // (a team's lanes share one step)
  } else {
    float4 P[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) P[k] = __ldg(&a.xyz32[ci[k]]);
    const float rx = f32_near(r.x), ry = f32_near(r.y), rz = f32_near(r.z);
    const float ux = sd.x, uy = sd.y, uz = sd.z;
    float wx[4], wy[4], wz[4];
    float W = 0.0f, Av = 0.0f;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      wx[k] = P[k].x - rx;
      wy[k] = P[k].y - ry;
      wz[k] = P[k].z - rz;
      W = fmaxf(W, fmaxf(fabsf(wx[k]), fmaxf(fabsf(wy[k]), fabsf(wz[k]))));
      Av = fmaxf(Av, P[k].w);
    }
    const float D = fmaxf(fabsf(ux), fmaxf(fabsf(uy), fabsf(uz)));
    const float A = Av + fmaxf(fabsf(rx), fmaxf(fabsf(ry), fabsf(rz)));
    const float thr =
        kU32 * 1.000001f * D * W * (97.0f * W + 13.0f * Av + 13.0f * A) * 1.0001f + 4.5e-15f;
    // pip(i -> j) = u . ((v_j - v_i) x (v_i - r)) for the six pairs i < j
    float pf[6];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = i + 1; j < 4; ++j)
        pf[pair_index(i, j)] = triple32(ux, uy, uz, P[j].x - P[i].x, P[j].y - P[i].y,
                                        P[j].z - P[i].z, wx[i], wy[i], wz[i]);
    // faces whose FP32 coordinates do not certify an early exit
#pragma unroll
    for (int f = 0; f < 4; ++f) {
      const int l0 = face_local<FO>(a, f, 0), l1 = face_local<FO>(a, f, 1),
                l2 = face_local<FO>(a, f, 2);
      const int e0 = pair_index(l0, l1), e1 = pair_index(l1, l2), e2 = pair_index(l2, l0);
      const float p0 = l0 < l1 ? sel6(pf, e0) : -sel6(pf, e0);
      const float p1 = l1 < l2 ? sel6(pf, e1) : -sel6(pf, e1);
      const float p2 = l2 < l0 ? sel6(pf, e2) : -sel6(pf, e2);
      if (!(p0 > thr || p1 > thr || p2 > thr)) escm |= 1u << f;
    }
  }
  // the neighbour behind the (normally only) remaining face is the next step's
  // tet: its record comes in while this step's arithmetic runs
  if (escm) {
    const int32_t nx = sel4(T.adj, __ffs(escm) - 1);
    if (nx >= 0 && nx < a.n_tets)
      asm volatile("prefetch.global.L1 [%0];" ::"l"(a.rec + 4 * (int64_t)nx));
  }
  // The distance to the remaining faces, in increasing face order (the
  // strict-< argmin is then the reference's, :191-196).  Every lane runs its
  // first remaining face in the same iteration, so the FP64 work of a warp is
  // issued once for all lanes.
  int idx = -1;
  double best = INFTY;
  while (escm) {
    const int f = __ffs(escm) - 1;
    escm &= escm - 1u;
    if (MIXED && team.q == 0) cnt.esc++;
    const int l0 = face_local<FO>(a, f, 0), l1 = face_local<FO>(a, f, 1),
              l2 = face_local<FO>(a, f, 2);
    const int32_t i0 = sel4(ci, l0), i1 = sel4(ci, l1), i2 = sel4(ci, l2);
    double df = INFTY;
    if (safe) {
      double c0, c1, c2;
      if (MIXED && G > 1) {
        const int la = tq == 0 ? l0 : (tq == 1 ? l1 : l2), lb = tq == 0 ? l1 : (tq == 1 ? l2 : l0);
        const d3 c = team.gather(edge_coord_p<INT>(a.edge, edge_ref(te, la, lb), u, rn));
        c0 = c.x;
        c1 = c.y;
        c2 = c.z;
      } else if (MIXED) {
        c0 = edge_coord_p<INT>(a.edge, edge_ref(te, l0, l1), u, rn);
        c1 = edge_coord_p<INT>(a.edge, edge_ref(te, l1, l2), u, rn);
        c2 = edge_coord_p<INT>(a.edge, edge_ref(te, l2, l0), u, rn);
      } else {
        // (negated where the face runs the pair backwards; 0 stays +0)
        auto coord = [&](int la, int lb) {
          const double p = sel6(pe, pair_index(la, lb));
          return la < lb || is0(p) ? p : -p;
        };
        c0 = coord(l0, l1);
        c1 = coord(l1, l2);
        c2 = coord(l2, l0);
      }
      if (!(gt0(c0) || gt0(c1) || gt0(c2)) && !(is0(c0) && is0(c1) && is0(c2)))
        df = face_distance_p<INT, G>(team, c0, c1, c2, a.xyz + sd.axis, i0, i1, i2,
                                     comp3(r, sd.axis), comp3(u, sd.axis));
    } else if (a.edge) {
      df = face_exit_hw(a.edge, a.xyz, edge_ref(te, l0, l1), edge_ref(te, l1, l2),
                        edge_ref(te, l2, l0), i0, i1, i2, r, u);
    } else {
      df = face_exit_xyz(a.xyz, i0, i1, i2, r, u);
    }
    if (dlt(df, best)) {
      best = df;
      idx = f;
    }
  }
  *exit_dist = best;
  return idx;
}

__device__ __forceinline__ void flush(unsigned long long* g, const StepCnt& c, unsigned long long rays) {
  unsigned long long v[3] = {c.steps, c.esc, rays};
  for (int k = 0; k < 3; ++k) {
    unsigned long long x = v[k];
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(__activemask(), x, off);
    v[k] = x;
  }
  if ((threadIdx.x & 31) == __ffs(__activemask()) - 1) {
    atomicAdd(&g[CNT_STEPS], v[0]);
    atomicAdd(&g[CNT_ESCALATE], v[1]);
    atomicAdd(&g[CNT_RAYS], v[2]);
  }
}

// The optional end state of track i's walk (WalkArgs::sum_out, end_r,
// end_dist): the running length sum, the position and the distance left.
__device__ __forceinline__ void walk_end_state(const WalkArgs& a, int64_t i, d3 r, double dist,
                                               double sum) {
  if (a.sum_out) a.sum_out[i] = sum;
  if (a.end_r) {
    a.end_r[3 * i] = r.x;
    a.end_r[3 * i + 1] = r.y;
    a.end_r[3 * i + 2] = r.z;
  }
  if (a.end_dist) a.end_dist[i] = dist;
}

// Where a warp's tracks come from: positions cursor .. end - 1 of the batch,
// or of the length order.  Without an order, one contiguous chunk.  With one,
// the warp takes 32 (of four-lane teams, 8) consecutive positions at a time,
// longest first, from the launch's work counter.  The lanes of a warp then hold tracks of about the
// same length and end together, so the FP64 unit, which takes as long for one
// lane as for 32, sees full warps (dealt one by one, every warp held one of
// the longest tracks and stepped on for it alone), and the warps end together
// too (dealt in fixed shares, the SMs were idle a fifth of the launch on
// 3e5 tracks).
template <int G = 1>
struct WarpTracks {
  static constexpr int kTake = 32 / G;  // tracks a warp holds
  int64_t cursor, end, last;  // `last`: the end of its part of the order
  unsigned long long* work;   // that part's work counter, from its first position `first`
  int64_t first;
  bool open;                  // the order may hold more
  __device__ __forceinline__ WarpTracks(const WalkArgs& a, int64_t gwarp, int64_t chunk) {
    cursor = a.order ? 0 : gwarp * chunk;
    end = a.order ? 0 : min(a.n, cursor + chunk);
    part(a, 0, a.n, 0);
  }
  // positions first_ .. last_ - 1 of the order, by work counter k
  __device__ __forceinline__ void part(const WalkArgs& a, int64_t first_, int64_t last_, int k) {
    first = first_;
    last = last_;
    work = a.order ? a.work + k : nullptr;
    open = a.order != nullptr;
  }
  __device__ __forceinline__ bool more() const { return cursor < end || open; }
  // the track of the `rank`-th of `want` lanes, or -1 (warp-uniform but for
  // rank; all lanes of the warp call it)
  __device__ __forceinline__ int64_t take(const WalkArgs& a, int rank, int want) {
    if (cursor >= end && open) {
      unsigned long long base = 0ull;
      if ((threadIdx.x & 31) == 0) base = atomicAdd(work, (unsigned long long)kTake);
      base = __shfl_sync(0xffffffffu, base, 0);
      cursor = first + (int64_t)base;
      end = min(last, cursor + kTake);
      open = end > cursor;
      if (!open) cursor = end = 0;
    }
    const int64_t pos = cursor + rank;
    cursor = min(end, cursor + want);
    if (pos >= end) return -1;
    if (!a.order) return pos;
    const int64_t i = __ldg(&a.order[pos]);
    return i >= 0 && i < a.n ? i : -1;  // (an entry out of range names no track)
  }
};

// Persistent walk: a lane whose track has ended takes the warp's next one, so
// a warp keeps all 32 lanes stepping until its tracks are used up (track
// lengths are exponentially distributed, so one-track-per-lane would leave
// most lanes idle behind the longest track of the warp).
// SUM: the running length sum is wanted (WalkArgs::sum_out).  INT: products on
// the integer pipes (next_face).  G: lanes of a track (Team).
template <int FO, bool MIXED, bool SUM, bool INT, int G>
__device__ __forceinline__ void walk_tracks(const WalkArgs& a, WarpTracks<G> list, StepCnt& cnt,
                                            unsigned long long& tracks) {
  const Team<G> team;
  bool has = false;
  int64_t i = 0;
  d3 r = mk3(0, 0, 0), u = mk3(0, 0, 0);
  double dist = 0.0, sum = 0.0;
  int32_t elem = -1, k = 0, st = RAY_OK;
  StepDir sd = {};
  int32_t* oe = nullptr;
  double* ol = nullptr;
  while (true) {
    const unsigned need = __ballot_sync(0xffffffffu, !has);
    if (need != 0u) {
      unsigned lt;
      asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
      if (G > 1) lt = (1u << (threadIdx.x & 31 & ~(G - 1))) - 1u;
      const int64_t cand = list.take(a, __popc(need & lt) / G, __popc(need) / G);
      if (!has) {
        if (cand >= 0) {
          i = cand;
          has = true;
          r = load3(a.org, i);
          u = load3(a.dir, i);
          sd = step_dir(a, u);
          dist = a.dist[i];
          sum = SUM && a.sum_in ? a.sum_in[i] : 0.0;
          elem = a.start[i];
          k = 0;
          st = RAY_OK;
          if (a.out_mode == WALK_STRIDED) {
            oe = a.seg_elem + i * (int64_t)a.max_segs;
            ol = a.seg_len + i * (int64_t)a.max_segs;
          } else if (a.out_mode == WALK_PACKED) {
            const int64_t off = a.offsets[i];
            const int64_t cnt_i = a.offsets[i + 1] - off;
            if (off + cnt_i <= a.capacity) {
              oe = a.seg_elem + off;
              ol = a.seg_len + off;
            } else {
              oe = nullptr;  // does not fit: the track is walked, nothing is written
              ol = nullptr;
            }
          } else {
            oe = nullptr;
            ol = nullptr;
          }
          if (elem < 0 || elem >= a.n_tets || !finite3(r) || !finite3(u) || nan_bits(dist)) {
            st = RAY_INVALID;
            dist = 0.0;  // finishes below without a step
          }
        }
      }
    }
    if (__ballot_sync(0xffffffffu, has) == 0u) {
      if (list.more()) continue;
      break;
    }
    if (has) {
      bool done = !gt0(dist);  // while (distance > 0), mesh_manager_interface.cpp:117
      if (!done && k >= a.max_segs) {
        st = RAY_WALK_LIMIT;
        done = true;
      }
      if (!done) {
        if (team.q == 0) cnt.steps++;
        double ex;
        const TetRec T = load_rec(a, elem);
        const bool safe = sd.safe && in_range3(r);
        const int f = next_face<FO, MIXED, INT, G>(a, T, r, u, sd, safe, &ex, cnt, team);
        int32_t nxt = -1;
        if (f < 0) {
          st = RAY_NO_EXIT_FACE;  // the reference would index adjacency with -1
        } else {
          nxt = sel4(T.adj, f);
        }
        ex = dlt(dist, ex) ? dist : ex;  // std::min(exit, distance)
        dist -= ex;
        if (SUM) sum = sum + ex;
        if (oe && team.q == 0) {
          oe[k] = T.id;
          ol[k] = ex;
        }
        ++k;
        r = walk_move(team, r, ex, u);  // r += exit.second * u
        if (nxt < -1 || nxt >= a.n_tets) {
          st = RAY_INVALID;  // corrupt adjacency: stop instead of reading out of range
          done = true;
        } else {
          elem = nxt;
          if (elem == -1) done = true;
        }
      }
      if (done) has = false;
      if (done && team.q == 0) {
        if (a.out_mode == WALK_COUNT) {
          a.offsets[i] = k;
        } else {
          if (a.seg_count) a.seg_count[i] = k;
          if (a.out_mode == WALK_PACKED && !oe && k > 0 && st == RAY_OK) st = RAY_OUTPUT_FULL;
        }
        if (a.status) a.status[i] = st;
        if (a.stop_elem) a.stop_elem[i] = elem;  // where a capped walk resumes
        walk_end_state(a, i, r, dist, sum);
        tracks++;
      }
    }
  }
}

template <int FO, bool MIXED, bool SUM, bool INT, int G>
__global__ void __launch_bounds__(kBlock, 4) k_walk(WalkArgs a, int64_t chunk) {
  const int64_t gwarp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  StepCnt cnt = {0, 0};
  unsigned long long tracks = 0;
  walk_tracks<FO, MIXED, SUM, INT, G>(a, WarpTracks<G>(a, gwarp, chunk), cnt, tracks);
  if (a.counters) flush(a.counters, cnt, tracks);
}

// A walk in length order that lasts as long as its longest tracks: the first
// `team_blocks` blocks walk the first n_team of the order four lanes to a
// track (Team), the others the rest, and then they help.
template <int FO, bool MIXED>
__global__ void __launch_bounds__(kBlock, 4) k_walk_mix(WalkArgs a, int64_t n_team,
                                                        unsigned team_blocks) {
  StepCnt cnt = {0, 0};
  unsigned long long tracks = 0;
  if (blockIdx.x < team_blocks) {
    WarpTracks<4> list(a, 0, 0);
    list.part(a, 0, n_team, 0);
    walk_tracks<FO, MIXED, false, MIXED, 4>(a, list, cnt, tracks);
  }
  WarpTracks<1> list(a, 0, 0);
  list.part(a, n_team, a.n, 1);
  walk_tracks<FO, MIXED, false, true, 1>(a, list, cnt, tracks);
  if (a.counters) flush(a.counters, cnt, tracks);
}


template <int FO, bool MIXED>
__global__ void __launch_bounds__(kBlock) k_next(WalkArgs a) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  StepCnt cnt = {0, 0};
  if (i < a.n) {
    const d3 r = load3(a.org, i);
    const d3 u = load3(a.dir, i);
    const int32_t elem = a.start[i];
    int32_t st = RAY_OK, nxt = -1;
    double ex = INFTY;
    if (elem < 0 || elem >= a.n_tets || !finite3(r) || !finite3(u)) {
      st = RAY_INVALID;
    } else {
      cnt.steps++;
      const TetRec T = load_rec(a, elem);
      const StepDir sd = step_dir(a, u);
      const int f = next_face<FO, MIXED>(a, T, r, u, sd, sd.safe && in_range3(r), &ex, cnt);
      if (f < 0) {
        st = RAY_NO_EXIT_FACE;
      } else {
        nxt = sel4(T.adj, f);
      }
    }
    a.next_out[i] = nxt;
    a.dist_out[i] = ex;
    if (a.status) a.status[i] = st;
  }
  if (a.counters) flush(a.counters, cnt, i < a.n ? 1ull : 0ull);
}

// ---------------------------------------------------------------------------
// Mixed-precision walk with a per-warp FP64 queue.
//
// Each step of a track runs the FP32 edge filter for its tet (six edge
// coordinates, truncated FP32 inputs, bound below) and queues every face the
// filter cannot reject as a (lane, face) task.  When 32 tasks are queued, or
// lanes wait on the queue, the whole warp runs 32 tasks at once -- each lane
// evaluates one face of some lane's tet with the FP64 Plucker test -- and each
// owner keeps the smallest (distance, face index) of its results, which is
// the reference's strict-< scan over faces 0..3 (:186-196) in any order.  A
// lane whose tasks are all done completes its step (segment, r += len * u)
// and starts the next one, so FP64 instructions run with (nearly) all 32
// lanes busy however many faces each step escalates.
//
// FP32 bound with truncated inputs (u = 2^-24; r and the direction truncated,
// relative error 2u; stored vertices rounded, u; W = max |v_k - r|_inf over
// the FP32 differences; Wb = W (1 + 2^-20) + 1.01 u (Av + 2 R) bounds the
// exact |v_k - r|_inf; edges |e| <= 2 Wb; D = |u|_inf, Av = max |v_k|_inf,
// R = |r|_inf):
//   rounding of the triple product (gamma_5, six terms)   <= 60 u D Wb^2
//   input perturbation (direction 2u, edges, differences) <= u D Wb (48 Wb + 24 Av + 24 R)
// so |pip32 - pip| <= u D Wb (108 Wb + 24 Av + 24 R); the threshold uses
// 110 / 26 / 26 and a factor 1.01 for second-order terms, the FP64
// evaluation error and the rounding of the threshold itself, plus the
// 20*DBL_EPSILON snap.
// ---------------------------------------------------------------------------

constexpr int kWQ = 256;  // ring entries per warp: < 32 left over + 4 per lane

struct WalkQueue {
  uint32_t ent[kWQ];  // (owner lane << 2) | face
  double rd[32];
  int32_t rf[32];
  uint32_t head, tail;
};

template <int FO>
__device__ __forceinline__ unsigned walk_filter32(const WalkArgs& a, const int32_t ci[4], float rx,
                                                  float ry, float rz, float ux, float uy, float uz,
                                                  float D, float R) {
  float4 P[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) P[k] = __ldg(&a.xyz32[ci[k]]);
  float wx[4], wy[4], wz[4];
  float W = 0.0f, Av = 0.0f;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    wx[k] = P[k].x - rx;
    wy[k] = P[k].y - ry;
    wz[k] = P[k].z - rz;
    W = fmaxf(W, fmaxf(fabsf(wx[k]), fmaxf(fabsf(wy[k]), fabsf(wz[k]))));
    Av = fmaxf(Av, P[k].w);
  }
  const float Wb = W * 1.000001f + kU32 * 1.01f * (Av + 2.0f * R);
  const float thr = kU32 * D * Wb * (110.0f * Wb + 26.0f * Av + 26.0f * R) * 1.01f + 4.5e-15f;
  float pe[6];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = i + 1; j < 4; ++j)
      pe[pair_index(i, j)] = triple32(ux, uy, uz, P[j].x - P[i].x, P[j].y - P[i].y,
                                      P[j].z - P[i].z, wx[i], wy[i], wz[i]);
  unsigned escm = 0u;
#pragma unroll
  for (int f = 0; f < 4; ++f) {
    const int l0 = face_local<FO>(a, f, 0), l1 = face_local<FO>(a, f, 1),
              l2 = face_local<FO>(a, f, 2);
    const int e0 = pair_index(l0, l1), e1 = pair_index(l1, l2), e2 = pair_index(l2, l0);
    const float p0 = l0 < l1 ? sel6(pe, e0) : -sel6(pe, e0);
    const float p1 = l1 < l2 ? sel6(pe, e1) : -sel6(pe, e1);
    const float p2 = l2 < l0 ? sel6(pe, e2) : -sel6(pe, e2);
    if (!(p0 > thr || p1 > thr || p2 > thr)) escm |= 1u << f;
  }
  return escm;
}

template <int FO>
__global__ void __launch_bounds__(kBlock) k_walk_q(WalkArgs a, int64_t chunk) {
  __shared__ WalkQueue qs[kBlock / 32];
  WalkQueue& Q = qs[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const int64_t gwarp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  WarpTracks<> list(a, gwarp, chunk);
  if (lane == 0) {
    Q.head = 0u;
    Q.tail = 0u;
  }
  __syncwarp();
  StepCnt cnt = {0, 0};
  unsigned long long tracks = 0;
  // track state
  bool has = false;
  int64_t i = 0;
  d3 r = mk3(0, 0, 0), u = mk3(0, 0, 0);
  double dist = 0.0, sum = 0.0;
  int32_t elem = -1, k = 0, st = RAY_OK;
  int32_t* oe = nullptr;
  double* ol = nullptr;
  float ux = 0.f, uy = 0.f, uz = 0.f, D = 0.f;
  // step state
  bool in_step = false;
  int npend = 0;
  double bd = INFTY;
  int32_t bf = -1;
  d3 rn = mk3(0, 0, 0);
  int32_t ci[4] = {0, 0, 0, 0};

  while (true) {
    // ---- refill lanes without a track from the warp's chunk ----
    const unsigned need = __ballot_sync(0xffffffffu, !has);
    if (need != 0u) {
      unsigned lt;
      asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
      const int64_t cand = list.take(a, __popc(need & lt), __popc(need));
      if (!has) {
        if (cand >= 0) {
          i = cand;
          has = true;
          in_step = false;
          r = load3(a.org, i);
          u = load3(a.dir, i);
          dist = a.dist[i];
          sum = a.sum_in ? a.sum_in[i] : 0.0;
          elem = a.start[i];
          k = 0;
          st = RAY_OK;
          ux = f32_trunc(u.x);
          uy = f32_trunc(u.y);
          uz = f32_trunc(u.z);
          D = fmaxf(fabsf(ux), fmaxf(fabsf(uy), fabsf(uz))) * 1.0000002f;
          if (a.out_mode == WALK_STRIDED) {
            oe = a.seg_elem + i * (int64_t)a.max_segs;
            ol = a.seg_len + i * (int64_t)a.max_segs;
          } else if (a.out_mode == WALK_PACKED) {
            const int64_t off = a.offsets[i];
            const int64_t cnt_i = a.offsets[i + 1] - off;
            if (off + cnt_i <= a.capacity) {
              oe = a.seg_elem + off;
              ol = a.seg_len + off;
            } else {
              oe = nullptr;  // does not fit: the track is walked, nothing is written
              ol = nullptr;
            }
          } else {
            oe = nullptr;
            ol = nullptr;
          }
          if (elem < 0 || elem >= a.n_tets || !finite3(r) || !finite3(u) || nan_bits(dist)) {
            st = RAY_INVALID;
            dist = 0.0;  // finishes below without a step
          }
        }
      }
    }
    if (__ballot_sync(0xffffffffu, has) == 0u) {
      if (list.more()) continue;
      break;
    }

    // ---- start a step: FP32 filter, queue the faces it cannot reject ----
    unsigned escm = 0u;
    if (has && !in_step) {
      bool done = !gt0(dist);  // while (distance > 0), mesh_manager_interface.cpp:117
      if (!done && k >= a.max_segs) {
        st = RAY_WALK_LIMIT;
        done = true;
      }
      if (done) {
        if (a.out_mode == WALK_COUNT) {
          a.offsets[i] = k;
        } else {
          if (a.seg_count) a.seg_count[i] = k;
          if (a.out_mode == WALK_PACKED && !oe && k > 0 && st == RAY_OK) st = RAY_OUTPUT_FULL;
        }
        if (a.status) a.status[i] = st;
        if (a.stop_elem) a.stop_elem[i] = elem;  // where a capped walk resumes
        walk_end_state(a, i, r, dist, sum);
        has = false;
        tracks++;
      } else {
        cnt.steps++;
        in_step = true;
        const int4 c = __ldg(a.rec + 4 * (int64_t)elem);
        ci[0] = c.x;
        ci[1] = c.y;
        ci[2] = c.z;
        ci[3] = c.w;
        const float rx = f32_trunc(r.x), ry = f32_trunc(r.y), rz = f32_trunc(r.z);
        const float R = fmaxf(fabsf(rx), fmaxf(fabsf(ry), fabsf(rz))) * 1.0000002f;
        escm = walk_filter32<FO>(a, ci, rx, ry, rz, ux, uy, uz, D, R);
        rn = cross3(u, r);  // plucker.h:75
        bd = INFTY;
        bf = -1;
        npend = __popc(escm);
        cnt.esc += npend;
      }
    }
    {
      const int c = __popc(escm);
      int incl = c;
#pragma unroll
      for (int off = 1; off < 32; off <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += y;
      }
      const int total = __shfl_sync(0xffffffffu, incl, 31);
      if (total > 0) {
        const uint32_t tail = Q.tail;
        __syncwarp();
        uint32_t pos = tail + (uint32_t)(incl - c);
        unsigned m = escm;
        while (m) {
          const int f = __ffs(m) - 1;
          m &= m - 1u;
          Q.ent[pos & (kWQ - 1)] = ((uint32_t)lane << 2) | (uint32_t)f;
          ++pos;
        }
        __syncwarp();
        if (lane == 0) Q.tail = tail + (uint32_t)total;
      }
      __syncwarp();
    }

    // ---- run queued FP64 face tests with the whole warp ----
    while (true) {
      const uint32_t head = Q.head;
      const int qn = (int)(Q.tail - head);
      const unsigned waiting = __ballot_sync(0xffffffffu, in_step && npend > 0);
      const unsigned progress = __ballot_sync(0xffffffffu, has && !(in_step && npend > 0));
      if (!(qn >= 32 || (qn > 0 && (progress == 0u || __popc(waiting) >= a.flush_wait)))) break;
      const int nq = min(qn, 32);
      const bool mine = lane < nq;
      const uint32_t ent = mine ? Q.ent[(head + lane) & (kWQ - 1)] : ((uint32_t)lane << 2);
      const int owner = (int)(ent >> 2);
      const int f = (int)(ent & 3u);
      d3 orr, ou, orn;
      orr.x = __shfl_sync(0xffffffffu, r.x, owner);
      orr.y = __shfl_sync(0xffffffffu, r.y, owner);
      orr.z = __shfl_sync(0xffffffffu, r.z, owner);
      ou.x = __shfl_sync(0xffffffffu, u.x, owner);
      ou.y = __shfl_sync(0xffffffffu, u.y, owner);
      ou.z = __shfl_sync(0xffffffffu, u.z, owner);
      orn.x = __shfl_sync(0xffffffffu, rn.x, owner);
      orn.y = __shfl_sync(0xffffffffu, rn.y, owner);
      orn.z = __shfl_sync(0xffffffffu, rn.z, owner);
      int32_t oc[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) oc[q] = __shfl_sync(0xffffffffu, ci[q], owner);
      const int32_t oel = __shfl_sync(0xffffffffu, elem, owner);
      double df = INFTY;
      if (mine) {
        const int l0 = face_local<FO>(a, f, 0), l1 = face_local<FO>(a, f, 1),
                  l2 = face_local<FO>(a, f, 2);
        double t;
        bool hit;
        if (a.edge) {
          hit = plucker64_face_pre(a, oel, oc, l0, l1, l2, orr, ou, orn, &t);
        } else {
          const d3 f0 = load3(a.xyz, sel4(oc, l0));
          const d3 f1 = load3(a.xyz, sel4(oc, l1));
          const d3 f2 = load3(a.xyz, sel4(oc, l2));
          hit = plucker64(f0, f1, f2, orr, ou, orn, INFTY, 0.0, true, 1, &t);
        }
        df = hit ? (gt0(t) ? t : 0.0) : INFTY;  // std::max(0.0, t)
      }
      Q.rd[lane] = df;
      Q.rf[lane] = f;
      __syncwarp();
      for (int j = 0; j < nq; ++j) {
        if (__shfl_sync(0xffffffffu, owner, j) != lane) continue;
        npend--;
        const double dj = Q.rd[j];
        const int32_t fj = Q.rf[j];
        // first minimum over faces 0..3 with strict < (:186-196)
        if (dlt(dj, bd) || (bf >= 0 && okey(dj) == okey(bd) && fj < bf)) {
          bd = dj;
          bf = fj;
        }
      }
      __syncwarp();
      if (lane == 0) Q.head = head + (uint32_t)nq;
      __syncwarp();
    }

    // ---- complete the steps whose faces are all evaluated ----
    if (has && in_step && npend == 0) {
      in_step = false;
      int32_t nxt = -1;
      double ex = bd;
      if (bf < 0) {
        st = RAY_NO_EXIT_FACE;  // the reference would index adjacency with -1
      } else {
        const int4 ad = __ldg(a.rec + 4 * (int64_t)elem + 1);
        nxt = bf == 0 ? ad.x : (bf == 1 ? ad.y : (bf == 2 ? ad.z : ad.w));
      }
      ex = dlt(dist, ex) ? dist : ex;  // std::min(exit, distance)
      dist -= ex;
      if (a.sum_out) sum = sum + ex;
      if (oe) {
        oe[k] = __ldg(a.rec + 4 * (int64_t)elem + 3).z;
        ol[k] = ex;
      }
      ++k;
      r = add3(r, scl3(ex, u));  // r += exit.second * u
      bool done = false;
      if (nxt < -1 || nxt >= a.n_tets) {
        st = RAY_INVALID;  // corrupt adjacency: stop instead of reading out of range
        done = true;
      } else {
        elem = nxt;
        if (elem == -1) done = true;
      }
      if (done) {
        if (a.out_mode == WALK_COUNT) {
          a.offsets[i] = k;
        } else {
          if (a.seg_count) a.seg_count[i] = k;
          if (a.out_mode == WALK_PACKED && !oe && k > 0 && st == RAY_OK) st = RAY_OUTPUT_FULL;
        }
        if (a.status) a.status[i] = st;
        if (a.stop_elem) a.stop_elem[i] = elem;  // where a capped walk resumes
        walk_end_state(a, i, r, dist, sum);
        has = false;
        tracks++;
      }
    }
  }
  if (a.counters) flush(a.counters, cnt, tracks);
}

constexpr int kScanBlock = 1024;

// sum of each block of kScanBlock counts
__global__ void __launch_bounds__(kScanBlock) k_block_sums(const int64_t* __restrict__ v, int64_t n,
                                                           int64_t* __restrict__ sums) {
  __shared__ int64_t ws[kScanBlock / 32];
  const int64_t i = blockIdx.x * (int64_t)kScanBlock + threadIdx.x;
  int64_t x = i < n ? v[i] : 0;
  for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x < 32) {
    int64_t y = ws[threadIdx.x];
    for (int off = 16; off > 0; off >>= 1) y += __shfl_xor_sync(0xffffffffu, y, off);
    if (threadIdx.x == 0) sums[blockIdx.x] = y;
  }
}

// exclusive scan of the block sums by one block; sums[nb] = total
__global__ void __launch_bounds__(kScanBlock) k_scan_sums(int64_t* __restrict__ sums, int64_t nb) {
  __shared__ int64_t ws[kScanBlock / 32];
  __shared__ int64_t carry;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int64_t base = 0; base < nb; base += kScanBlock) {
    const int64_t i = base + threadIdx.x;
    const int64_t x = i < nb ? sums[i] : 0;
    int64_t incl = x;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int off = 1; off < 32; off <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, incl, off);
      if (lane >= off) incl += y;
    }
    if (lane == 31) ws[w] = incl;
    __syncthreads();
    if (w == 0) {
      int64_t s = ws[lane];
      for (int off = 1; off < 32; off <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, s, off);
        if (lane >= off) s += y;
      }
      ws[lane] = s;
    }
    __syncthreads();
    const int64_t before = carry + (w > 0 ? ws[w - 1] : 0) + incl - x;
    if (i < nb) sums[i] = before;
    __syncthreads();
    if (threadIdx.x == kScanBlock - 1) carry = before + x;
    __syncthreads();
  }
  if (threadIdx.x == 0) sums[nb] = carry;
}

// in-place exclusive scan of each block plus its block offset
__global__ void __launch_bounds__(kScanBlock) k_scan_apply(int64_t* __restrict__ v, int64_t n,
                                                           const int64_t* __restrict__ sums,
                                                           int64_t nb) {
  __shared__ int64_t ws[kScanBlock / 32];
  const int64_t i = blockIdx.x * (int64_t)kScanBlock + threadIdx.x;
  const int64_t x = i < n ? v[i] : 0;
  int64_t incl = x;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  for (int off = 1; off < 32; off <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, incl, off);
    if (lane >= off) incl += y;
  }
  if (lane == 31) ws[w] = incl;
  __syncthreads();
  if (w == 0) {
    int64_t s = ws[lane];
    for (int off = 1; off < 32; off <<= 1) {
      const int64_t y = __shfl_up_sync(0xffffffffu, s, off);
      if (lane >= off) s += y;
    }
    ws[lane] = s;
  }
  __syncthreads();
  const int64_t excl = sums[blockIdx.x] + (w > 0 ? ws[w - 1] : 0) + incl - x;
  if (i < n) v[i] = excl;
  if (blockIdx.x == 0 && threadIdx.x == 0) v[n] = sums[nb];
}

template <int FO, bool MIXED, bool QUEUE, bool SUM, bool INT = true, int G = 1>
cudaError_t launch_walk_s(const WalkArgs& a, cudaStream_t st) {
  static std::atomic<int> cached[kMaxDevices];  // resident blocks per SM, per device
  auto kern = QUEUE ? k_walk_q<FO> : k_walk<FO, MIXED, SUM, INT, G>;
  int per_sm = 0;
  const cudaError_t e = occupancy_cached(cached, kern, kBlock, 0, per_sm);
  if (e != cudaSuccess) return e;
  int64_t blocks = (int64_t)device_sm_count() * per_sm;
  const int lanes = a.order ? 32 / G : std::min(32 / G, lanes_per_warp(a.n, kFp64Warps));
  const int64_t max_blocks = ((a.n + lanes - 1) / lanes + kBlock / 32 - 1) / (kBlock / 32);
  if (blocks > max_blocks) blocks = max_blocks;
  if (blocks < 1) blocks = 1;
  const int64_t warps = blocks * (kBlock / 32);
  const int64_t chunk = (a.n + warps - 1) / warps;
  if (a.order) {
    const cudaError_t m = cudaMemsetAsync(a.work, 0, sizeof(*a.work), st);
    if (m != cudaSuccess) return m;
  }
  kern<<<(unsigned)blocks, kBlock, 0, st>>>(a, chunk);
  return cudaGetLastError();
}

// Warps of eight four-lane tracks per SM up to which a batch walks that way
// (24,320 tracks): ms at 14 / 20 / 28, mixed: tally of 22,000 tracks 1.93 / 1.62 /
// 1.61, 34,000 1.94 / 1.92 / 1.64; global tracks, whose rounds shrink, 22,000
// 3.44 / 3.30 / 3.32, 60,000 4.07 / 4.07 / 4.24.
constexpr int kTeamWarps = 20;

// k_walk_mix: one in kMixPart of the tracks, the longest, in teams, on at most
// a third of the resident blocks, for batches of up to kMixWarps * 32 tracks
// per SM (107,008).  Located and walked, without / with, ms: 28,000 tracks
// 1.91 / 1.54 mixed, 2.57 / 2.06 all-FP64; 50,000 2.16 / 1.71 and 3.46 / 2.30;
// 100,000 2.42 / 2.07 and 3.95 / 2.81 (an eighth in teams 2.26 and 3.18, a quarter
// 2.65 and 3.58); 200,000, an eighth, 2.75 / 3.59 and 4.44 / 4.87.  Not for the
// global loop's walks, whose order is by the track's length and not the walk's:
// 50,000 tracks 4.00 / 4.17.
constexpr int kMixPart = 14, kMixWarps = 22;

template <int FO, bool MIXED>
cudaError_t launch_walk_mix(const WalkArgs& a, cudaStream_t st) {
  static std::atomic<int> cached[kMaxDevices];
  auto kern = k_walk_mix<FO, MIXED>;
  int per_sm = 0;
  cudaError_t e = occupancy_cached(cached, kern, kBlock, 0, per_sm);
  if (e == cudaSuccess) e = cudaMemsetAsync(a.work, 0, 2 * sizeof(*a.work), st);
  if (e != cudaSuccess) return e;
  const int64_t resident = (int64_t)device_sm_count() * per_sm;
  const int64_t n_team = a.n / kMixPart / 8 * 8;
  const int64_t team_blocks = std::min((n_team + 31) / 32, std::max<int64_t>(1, resident / 3));
  const int64_t rest = std::min((a.n - n_team + kBlock - 1) / kBlock,
                                std::max<int64_t>(1, resident - team_blocks));
  kern<<<(unsigned)(team_blocks + rest), kBlock, 0, st>>>(a, n_team, (unsigned)team_blocks);
  return cudaGetLastError();
}

template <int FO, bool MIXED, bool QUEUE>
cudaError_t launch_walk_t(const WalkArgs& a, cudaStream_t st) {
  // With at most about one warp a scheduler a step is a chain, and in the
  // all-FP64 step, with 45 products, the FP64 unit's are the shorter links
  // (1,000 tracks located and walked 2.11 ms with the integer products, 1.84
  // without; 20,000 3.25 and 2.49; 60,000 3.71 and 4.27)
  const int64_t team_max = (int64_t)device_sm_count() * kTeamWarps * 8;
  if constexpr (FO == 0 && !QUEUE) {
    if (a.n <= team_max)
      return a.sum_out ? launch_walk_s<FO, MIXED, false, true, MIXED, 4>(a, st)
                       : launch_walk_s<FO, MIXED, false, false, MIXED, 4>(a, st);
    if (a.order && !a.sum_out && a.n <= (int64_t)device_sm_count() * kMixWarps * 32)
      return launch_walk_mix<FO, MIXED>(a, st);
  }
  if (!MIXED && a.n <= (int64_t)device_sm_count() * kFp64Warps * 32)
    return a.sum_out ? launch_walk_s<FO, MIXED, QUEUE, true, MIXED>(a, st)
                     : launch_walk_s<FO, MIXED, QUEUE, false, MIXED>(a, st);
  return a.sum_out ? launch_walk_s<FO, MIXED, QUEUE, true>(a, st)
                   : launch_walk_s<FO, MIXED, QUEUE, false>(a, st);
}

}  // namespace

cudaError_t launch_walk(bool mixed, int face_order, const WalkArgs& a, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  const int sel = (face_order == 0 ? 0 : 2) + (mixed ? 1 : 0);
  const bool q = mixed && a.walk_queue;
  switch (sel) {
    case 0: return launch_walk_t<0, false, false>(a, st);
    case 1: return q ? launch_walk_t<0, true, true>(a, st) : launch_walk_t<0, true, false>(a, st);
    case 2: return launch_walk_t<1, false, false>(a, st);
    default: return q ? launch_walk_t<1, true, true>(a, st) : launch_walk_t<1, true, false>(a, st);
  }
}

namespace {

// ---------------------------------------------------------------------------
// Device particle loop over the tet mesh: the body of the walk_elements tool
// (tools/walk_elements.h:73-95) for particles inside the mesh.  Per event:
//   (next, exit) = next_element(elem, r, u)             (next_face above)
//   c = -log(1 - U) * mfp                                (sample.cuh)
//   c < exit: r += u c, distance += c, u = new isotropic direction
//   else:     r += u exit, distance += exit, elem = next
//   events++
// until the particle leaves the mesh (elem = -1, status OK: the caller
// decides on re-entry, which the tool does by ray_fire in the implicit
// complement and find_element, :88-94) or reaches max_events
// (RAY_EVENT_LIMIT).  With `tally`, each event adds its path length to the
// tet it was made in (atomicAdd, so the sums' rounding depends on the order).
// Warps own contiguous chunks of particles and refill lanes as particles
// finish, as in k_walk.  The collision sample's FP64 logarithm and the new
// direction are only computed where needed (see the FP32 test below) and for
// many lanes at once.
// ---------------------------------------------------------------------------

// G: lanes of a particle (Team).
template <int FO, bool MIXED, int G>
__global__ void __launch_bounds__(kBlock, 4) k_transport(TransportArgs t, int64_t chunk) {
  const WalkArgs& a = t.mesh;
  const Team<G> team;
  const int64_t gwarp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int64_t cursor = gwarp * chunk;
  const int64_t end = min(t.n, cursor + chunk);
  StepCnt cnt = {0, 0};
  unsigned long long parts = 0;
  bool has = false;
  int64_t i = 0;
  d3 r = mk3(0, 0, 0), u = mk3(0, 0, 0);
  double dist = 0.0;
  int32_t elem = -1, ev = 0, st = RAY_OK;
  unsigned long long rs = 0;
  // an event whose FP64 part waits for the warp's batch: its uniform draw,
  // exit distance and exit face
  bool pend = false;
  unsigned long long pu = 0ull;
  double pex = 0.0;
  int pf = -1;
  StepDir sd = {};
  const float mfp32 = (float)t.mfp;
  const bool quick = t.mfp < 1e30;

  // moves the particle to the exit face and into the neighbour (:86-90);
  // returns true when it stops
  auto exit_step = [&](double ex, int f, const int32_t adj[4]) -> bool {
    if (f < 0) {
      st = RAY_NO_EXIT_FACE;  // exit = INFTY and c >= INFTY: no finite step exists
      return true;
    }
    const int32_t nxt = sel4(adj, f);
    r = walk_move(team, r, ex, u);
    dist += ex;
    if (t.tally && team.q == 0) atomicAdd(&t.tally[elem], ex);
    if (nxt < -1 || nxt >= a.n_tets) {
      st = RAY_INVALID;  // corrupt adjacency
      return true;
    }
    elem = nxt;
    ++ev;
    return elem < 0;
  };

  while (true) {
    const unsigned need = __ballot_sync(0xffffffffu, !has);
    if (need != 0u && cursor < end) {
      if (!has) {
        unsigned lt;
        asm("mov.u32 %0, %%lanemask_lt;" : "=r"(lt));
        if (G > 1) lt = (1u << (threadIdx.x & 31 & ~(G - 1))) - 1u;
        const int64_t kk = cursor + __popc(need & lt) / G;
        if (kk < end) {
          i = kk;
          has = true;
          pend = false;
          elem = t.elem[i];
          r = load3(t.pos, i);
          u = load3(t.dir, i);
          sd = step_dir(a, u);
          rs = t.rng[i];
          dist = t.distance[i];
          ev = t.events[i];
          st = RAY_OK;
          if (elem >= a.n_tets || !finite3(r) || !finite3(u) || nan_bits(dist)) st = RAY_INVALID;
        }
      }
      cursor += __popc(need) / G;
    }
    if (__ballot_sync(0xffffffffu, has) == 0u) break;
    bool done = false;
    if (has && !pend) {
      done = st != RAY_OK || elem < 0;  // nothing to do outside the mesh
      if (!done && ev >= t.max_events) {
        st = RAY_EVENT_LIMIT;
        done = true;
      }
      if (!done) {
        if (team.q == 0) cnt.steps++;
        double ex;
        const TetRec T = load_rec(a, elem);
        const int f = next_face<FO, MIXED, true, G>(a, T, r, u, sd, sd.safe && in_range3(r), &ex, cnt,
                                                 team);
        // 1 - U of U = k 2^-53 is (2^53 - k) 2^-53, exactly
        const unsigned long long U = (1ull << 53) - uniform_bits(rs);
        // Most events leave the tet: an FP32 logarithm with a certified
        // margin decides c >= exit without the FP64 series.  |c32 - c| <=
        // 6.1e-8 mfp + 3.7e-7 c (rounding 1 - U to FP32, logf within 2 ulp,
        // two FP32 products); the margin below is 1.1e-6 (c32 + mfp).
        bool leaves = false;
        if (quick) {
          const float c32 = -logf(__ull2float_rn(U) * 1.1102230246251565e-16f) * mfp32;
          const float lo = c32 - 1.1e-6f * (c32 + mfp32);
          leaves = f32_up(ex) < lo;  // c >= lo > exit
        }
        if (leaves) {
          done = exit_step(ex, f, T.adj);
        } else {
          pend = true;  // the exact sample and the event run with the warp's batch
          pu = U;
          pex = ex;
          pf = f;
        }
      }
    }
    // Events that need the FP64 sample (collisions, and exits the FP32 test
    // could not certify) run together once event_wait lanes wait or no lane
    // can step: FP64 instructions cost the same issue time for 1 or 32 lanes.
    const unsigned pm = __ballot_sync(0xffffffffu, has && pend);
    if (pm != 0u) {
      const unsigned run = __ballot_sync(0xffffffffu, has && !pend && !done);
      if (__popc(pm) >= t.event_wait || run == 0u) {
        if (has && pend) {
          pend = false;
          // the collision distance
          const double c = -series_log(unit_scaled(pu, -53)) * t.mfp;
          if (dlt(c, pex)) {
            // collision inside the tet (:81-85)
            r = walk_move(team, r, c, u);
            dist += c;
            if (t.tally && team.q == 0) atomicAdd(&t.tally[elem], c);
            u = sample_direction(rs);
            sd = step_dir(a, u);
            ++ev;
          } else {
            const int4 ad = __ldg(a.rec + 4 * (int64_t)elem + 1);
            const int32_t adj[4] = {ad.x, ad.y, ad.z, ad.w};
            done = exit_step(pex, pf, adj);
          }
        }
      }
    }
    if (has && done) {
      has = false;
      if (team.q != 0) continue;
      t.elem[i] = elem;
      t.pos[3 * i] = r.x;
      t.pos[3 * i + 1] = r.y;
      t.pos[3 * i + 2] = r.z;
      t.dir[3 * i] = u.x;
      t.dir[3 * i + 1] = u.y;
      t.dir[3 * i + 2] = u.z;
      t.rng[i] = rs;
      t.distance[i] = dist;
      t.events[i] = ev;
      if (t.status) t.status[i] = st;
      parts++;
    }
  }
  if (t.counters) flush(t.counters, cnt, parts);
}

template <int FO, bool MIXED, int G = 1>
cudaError_t launch_transport_t(const TransportArgs& a, cudaStream_t st) {
  static std::atomic<int> cached[kMaxDevices];  // resident blocks per SM, per device
  auto kern = k_transport<FO, MIXED, G>;
  int per_sm = 0;
  const cudaError_t e = occupancy_cached(cached, kern, kBlock, 0, per_sm);
  if (e != cudaSuccess) return e;
  int64_t blocks = (int64_t)device_sm_count() * per_sm;
  const int lanes = std::min(32 / G, lanes_per_warp(a.n, kFp64Warps));
  const int64_t max_blocks = ((a.n + lanes - 1) / lanes + kBlock / 32 - 1) / (kBlock / 32);
  if (blocks > max_blocks) blocks = max_blocks;
  if (blocks < 1) blocks = 1;
  const int64_t warps = blocks * (kBlock / 32);
  const int64_t chunk = (a.n + warps - 1) / warps;
  kern<<<(unsigned)blocks, kBlock, 0, st>>>(a, chunk);
  return cudaGetLastError();
}

}  // namespace

cudaError_t launch_transport(bool mixed, int face_order, const TransportArgs& a, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  if (face_order == 0 && a.n <= (int64_t)device_sm_count() * kTeamWarps * 8)
    return mixed ? launch_transport_t<0, true, 4>(a, st) : launch_transport_t<0, false, 4>(a, st);
  switch ((face_order == 0 ? 0 : 2) + (mixed ? 1 : 0)) {
    case 0: return launch_transport_t<0, false>(a, st);
    case 1: return launch_transport_t<0, true>(a, st);
    case 2: return launch_transport_t<1, false>(a, st);
    default: return launch_transport_t<1, true>(a, st);
  }
}

int64_t scan_scratch_entries(int64_t n) { return (n + kScanBlock - 1) / kScanBlock + 1; }

namespace {

// local vertex pairs of a tet in pair_index order
__device__ __forceinline__ void pair_of(int p, int& i, int& j) {
  i = p < 3 ? 0 : (p < 5 ? 1 : 2);
  j = p < 3 ? p + 1 : (p < 5 ? p - 1 : 3);
}

__device__ __forceinline__ int32_t conn_at(int4 c, int k) {
  return k == 0 ? c.x : (k == 1 ? c.y : (k == 2 ? c.z : c.w));
}

__global__ void k_edge_keys(const int4* __restrict__ conn, int64_t n_tets,
                            unsigned long long* __restrict__ keys, int32_t* __restrict__ slots) {
  const int64_t s = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (s >= 6 * n_tets) return;
  const int4 c = conn[s / 6];
  int i, j;
  pair_of((int)(s % 6), i, j);
  const unsigned a = (unsigned)conn_at(c, i), b = (unsigned)conn_at(c, j);
  const unsigned lo = a < b ? a : b, hi = a < b ? b : a;
  keys[s] = ((unsigned long long)lo << 32) | hi;
  slots[s] = (int32_t)s;
}

__global__ void k_edge_heads(const unsigned long long* __restrict__ keys, int64_t n,
                             int32_t* __restrict__ head) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  head[k] = (k == 0 || keys[k] != keys[k - 1]) ? 1 : 0;
}

// e = hi - lo and en = e x lo of each unique edge (plucker.h:45-62 with
// first() ordering the two vertices); lo_vertex = the vertex index of lo
__global__ void k_edge_data(const unsigned long long* __restrict__ keys,
                            const int32_t* __restrict__ head, const int32_t* __restrict__ id,
                            int64_t n, const double* __restrict__ xyz, double* __restrict__ edge,
                            int32_t* __restrict__ lo_vertex) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n || !head[k]) return;
  const int64_t e = id[k] - 1;
  const int32_t ga = (int32_t)(keys[k] >> 32), gb = (int32_t)(keys[k] & 0xffffffffull);
  const d3 va = load3(xyz, ga), vb = load3(xyz, gb);
  const bool f = first_lower(va, vb);
  const d3 lo = f ? va : vb;
  const d3 hi = f ? vb : va;
  const d3 ev = sub3(hi, lo);
  const d3 en = cross3(ev, lo);
  double* E = edge + 6 * e;
  E[0] = ev.x;
  E[1] = ev.y;
  E[2] = ev.z;
  E[3] = en.x;
  E[4] = en.y;
  E[5] = en.z;
  lo_vertex[e] = f ? ga : gb;
}

__global__ void k_edge_scatter(const int32_t* __restrict__ slots, const int32_t* __restrict__ id,
                               int64_t n, const int4* __restrict__ conn,
                               const int32_t* __restrict__ lo_vertex,
                               int32_t* __restrict__ tet_edge) {
  const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (k >= n) return;
  const int32_t s = slots[k];
  const int32_t e = id[k] - 1;
  int i, j;
  pair_of(s % 6, i, j);
  const bool second_is_lo = conn_at(conn[s / 6], j) == lo_vertex[e];
  tet_edge[s] = e | (second_is_lo ? (int32_t)0x80000000u : 0);
}

}  // namespace

cudaError_t build_edge_table(const double* xyz, const int4* conn, int64_t n_tets, double** edge,
                             int32_t** tet_edge, int64_t* n_edges, cudaStream_t st) {
  *edge = nullptr;
  *tet_edge = nullptr;
  *n_edges = 0;
  const int64_t n = 6 * n_tets;
  if (n_tets <= 0 || n >= (1ll << 31)) return cudaErrorInvalidValue;
  const unsigned g = (unsigned)((n + 255) / 256);
  unsigned long long *keys = nullptr, *keys2 = nullptr;
  int32_t *slots = nullptr, *slots2 = nullptr, *head = nullptr, *id = nullptr, *lo = nullptr;
  void* tmp = nullptr;
  size_t tb_sort = 0, tb_scan = 0;
  cudaError_t e = cub::DeviceRadixSort::SortPairs(nullptr, tb_sort, keys, keys2, slots, slots2,
                                                  (int)n, 0, 64, st);
  if (e == cudaSuccess) e = cub::DeviceScan::InclusiveSum(nullptr, tb_scan, head, id, (int)n, st);
  const size_t tb = tb_sort > tb_scan ? tb_sort : tb_scan;
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&keys, sizeof(*keys) * n, st);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&keys2, sizeof(*keys2) * n, st);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&slots, sizeof(*slots) * n, st);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&slots2, sizeof(*slots2) * n, st);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&head, sizeof(*head) * n, st);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&id, sizeof(*id) * n, st);
  if (e == cudaSuccess) e = cudaMallocAsync(&tmp, tb, st);
  if (e == cudaSuccess) {
    k_edge_keys<<<g, 256, 0, st>>>(conn, n_tets, keys, slots);
    e = cudaGetLastError();
  }
  size_t t1 = tb;
  if (e == cudaSuccess)
    e = cub::DeviceRadixSort::SortPairs(tmp, t1, keys, keys2, slots, slots2, (int)n, 0, 64, st);
  if (e == cudaSuccess) {
    k_edge_heads<<<g, 256, 0, st>>>(keys2, n, head);
    e = cudaGetLastError();
  }
  size_t t2 = tb;
  if (e == cudaSuccess) e = cub::DeviceScan::InclusiveSum(tmp, t2, head, id, (int)n, st);
  int32_t ne = 0;
  if (e == cudaSuccess) e = cudaMemcpyAsync(&ne, id + (n - 1), sizeof(ne), cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e == cudaSuccess) e = cudaMalloc((void**)edge, sizeof(double) * 6 * (size_t)ne);
  if (e == cudaSuccess) e = cudaMalloc((void**)tet_edge, sizeof(int32_t) * (size_t)n);
  if (e == cudaSuccess) e = cudaMallocAsync((void**)&lo, sizeof(int32_t) * (size_t)ne, st);
  if (e == cudaSuccess) {
    k_edge_data<<<g, 256, 0, st>>>(keys2, head, id, n, xyz, *edge, lo);
    k_edge_scatter<<<g, 256, 0, st>>>(slots2, id, n, conn, lo, *tet_edge);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  for (void* p : {(void*)keys, (void*)keys2, (void*)slots, (void*)slots2, (void*)head, (void*)id,
                  tmp, (void*)lo})
    if (p) cudaFreeAsync(p, st);
  cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    if (*edge) cudaFree(*edge);
    if (*tet_edge) cudaFree(*tet_edge);
    *edge = nullptr;
    *tet_edge = nullptr;
    return e;
  }
  *n_edges = ne;
  return cudaSuccess;
}

namespace {
__global__ void k_tet_records(const int4* __restrict__ conn, const int4* __restrict__ adj,
                              const int32_t* __restrict__ tet_edge,
                              const int32_t* __restrict__ ids, int64_t n, int4* __restrict__ rec) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  int32_t e[6] = {0, 0, 0, 0, 0, 0};
  if (tet_edge)
    for (int k = 0; k < 6; ++k) e[k] = tet_edge[6 * i + k];
  rec[4 * i] = conn[i];
  rec[4 * i + 1] = adj[i];
  rec[4 * i + 2] = make_int4(e[0], e[1], e[2], e[3]);
  rec[4 * i + 3] = make_int4(e[4], e[5], ids[i], 0);
}
}  // namespace

cudaError_t build_tet_records(const int4* conn, const int4* adj, const int32_t* tet_edge,
                              const int32_t* ids, int64_t n_tets, int4* rec, cudaStream_t st) {
  if (n_tets <= 0) return cudaSuccess;
  k_tet_records<<<(unsigned)((n_tets + 255) / 256), 256, 0, st>>>(conn, adj, tet_edge, ids, n_tets,
                                                                  rec);
  return cudaGetLastError();
}

namespace {
// Sort keys of the length order: the length's FP32 exponent and leading 8
// mantissa bits.  The order only groups tracks of about the same length, and
// 16 bits take two radix passes where the 64 of the length took eight (1e6
// tracks, two rounds: 215 -> 60 us).
__global__ void k_length_keys(const double* __restrict__ dist, int64_t n,
                              uint32_t* __restrict__ keys, int32_t* __restrict__ idx) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double d = dist[i];
  keys[i] = gt0(d) && !nan_bits(d) ? __float_as_uint(f32_trunc(d)) >> 15 : 0u;
  idx[i] = (int32_t)i;
}
constexpr int kLengthBits = 16;

size_t length_sort_bytes(int64_t n) {
  size_t tmp = 0;
  cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, (const uint32_t*)nullptr,
                                            (uint32_t*)nullptr, (const int32_t*)nullptr,
                                            (int32_t*)nullptr, (int)n, 0, kLengthBits);
  return (tmp + 255) & ~(size_t)255;
}
}  // namespace

size_t walk_order_scratch_bytes(int64_t n) {
  return length_sort_bytes(n) + 3 * ((sizeof(uint32_t) * n + 255) & ~(size_t)255);
}

cudaError_t walk_order(const double* dist, int64_t n, int32_t* order, void* scratch,
                       size_t scratch_bytes, cudaStream_t st) {
  if (walk_order_scratch_bytes(n) > scratch_bytes) return cudaErrorInvalidValue;
  size_t tmp = length_sort_bytes(n);
  const size_t arr = (sizeof(uint32_t) * n + 255) & ~(size_t)255;
  char* p = (char*)scratch;
  uint32_t* keys = (uint32_t*)(p + tmp);
  uint32_t* keys_out = (uint32_t*)(p + tmp + arr);
  int32_t* idx = (int32_t*)(p + tmp + 2 * arr);
  k_length_keys<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(dist, n, keys, idx);
  return cub::DeviceRadixSort::SortPairsDescending(p, tmp, keys, keys_out, idx, order, (int)n, 0,
                                                   kLengthBits, st);
}

cudaError_t scan_offsets(int64_t* offsets, int64_t n, int64_t* block_sums, cudaStream_t st) {
  if (n <= 0) return cudaMemsetAsync(offsets, 0, sizeof(int64_t), st);
  const int64_t nb = (n + kScanBlock - 1) / kScanBlock;
  k_block_sums<<<(unsigned)nb, kScanBlock, 0, st>>>(offsets, n, block_sums);
  k_scan_sums<<<1, kScanBlock, 0, st>>>(block_sums, nb);
  k_scan_apply<<<(unsigned)nb, kScanBlock, 0, st>>>(offsets, n, block_sums, nb);
  return cudaGetLastError();
}

cudaError_t launch_next_element(bool mixed, int face_order, const WalkArgs& a, cudaStream_t st) {
  if (a.n <= 0) return cudaSuccess;
  const unsigned g = (unsigned)((a.n + kBlock - 1) / kBlock);
  const int sel = (face_order == 0 ? 0 : 2) + (mixed ? 1 : 0);
  switch (sel) {
    case 0: k_next<0, false><<<g, kBlock, 0, st>>>(a); break;
    case 1: k_next<0, true><<<g, kBlock, 0, st>>>(a); break;
    case 2: k_next<1, false><<<g, kBlock, 0, st>>>(a); break;
    default: k_next<1, true><<<g, kBlock, 0, st>>>(a); break;
  }
  return cudaGetLastError();
}

}  // namespace xdgcu
