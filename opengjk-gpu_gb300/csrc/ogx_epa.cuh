// ogx_epa.cuh -- EPA penetration depth for one colliding pair, run by a team of L lanes.
//
// Semantics follow the reference's computeCollisionInformation (GJK/cpu/EPA.c:362-863,
// GJK/gpu/openGJK.cu:1836-2726): a separated pair only gets its contact normal
// (normalised w1 - w0); a contact whose GJK simplex has fewer than four points is grown
// by supports along fixed directions (point, edge-perpendicular, triangle normal and its
// opposite) and reported with depth 0 when no new point appears; otherwise the simplex
// seeds a polytope that is expanded towards its closest face until the support point
// along that face's normal does not improve on it.  The result is depth = -distance of
// the closest face, its normal, and witnesses from the origin's barycentric position on
// that face (clamped to the triangle as in EPA.c:238-304).
//
// Design (not the reference's):
//  * The polytope keeps face adjacency.  The faces visible from the new point are found
//    in parallel (faces are split over the lanes), the horizon is every edge of a visible
//    face whose neighbour is not visible, and new faces are linked to each other through
//    two per-vertex tables -- O(F) per step instead of the reference's O(F^2) edge
//    de-duplication.  Winding is inherited from the horizon edge, so no centroid test.
//  * Face normals are computed once when the face is created (the reference recomputes
//    all of them every step) in FP32, in FP64 from the exact points for sliver faces.
//  * Polytope capacity is 68 vertices / 132 faces, enough for the 64-step cap (the
//    reference's 128-face list can overflow in its last steps).
//  * Duplicate detection compares the support pair's vertex indices.
//  * The chosen face can be re-solved in FP64 afterwards (same pass as the GJK polish).
#pragma once

#include "ogx_common.cuh"
#include "ogx_gjk.cuh"

namespace ogx {

// A set of faces: one bit per slot, in registers.  put() takes the bits of slots f0..f0+31
// (f0 a multiple of the team's width, so they lie in one word).
template <int W>
struct FaceSet {
  uint64_t w[W];
  OGX_HD void clear() {
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = 0u;
  }
  OGX_HD void put(int f0, uint32_t bits) {
#pragma unroll
    for (int i = 0; i < W; ++i)
      if (W == 1 || i == (f0 >> 6)) w[i] |= (uint64_t)bits << (f0 & 63);
  }
  OGX_HD bool has(int f) const {
    uint64_t x = w[0];
#pragma unroll
    for (int i = 1; i < W; ++i)
      if (i == (f >> 6)) x = w[i];
    return (x >> (f & 63) & 1u) != 0u;
  }
  OGX_HD int count() const {
    int n = 0;
#pragma unroll
    for (int i = 0; i < W; ++i) n += popc64(w[i]);
    return n;
  }
  OGX_HD void save(uint32_t* m) const {
#pragma unroll
    for (int i = 0; i < W; ++i) {
      m[2 * i] = (uint32_t)w[i];
      m[2 * i + 1] = (uint32_t)(w[i] >> 32);
    }
  }
  OGX_HD void load(const uint32_t* m) {
#pragma unroll
    for (int i = 0; i < W; ++i) w[i] = (uint64_t)m[2 * i] | (uint64_t)m[2 * i + 1] << 32;
  }
  // the k-th face of the set (k < count())
  OGX_HD int nth(int k) const {
    uint64_t m = w[0];
    int base = 0;
#pragma unroll
    for (int i = 1; i < W; ++i) {
      const int c = popc64(m);
      if (base == 64 * (i - 1) && k >= c) {
        k -= c;
        m = w[i];
        base = 64 * i;
      }
    }
#pragma unroll 1
    for (; k > 0; --k) m &= m - 1u;
    return base + lowest64(m);
  }
};

// Shared-memory working set of one pair, for at most VMAX polytope vertices and FMAX faces.
// A retired face keeps no flag: its plane is at infinity (never visible, never the closest).
template <int VMAX, int FMAX>
struct EpaMemT {
  static constexpr int kV = VMAX;
  static constexpr int kF = FMAX;
  typedef FaceSet<(FMAX + 63) / 64> Faces;
  float4 fn[FMAX];       // unit outward normal, w = plane distance from origin
  float4 vp[VMAX];       // polytope vertices (Minkowski points)
  int2 vid[VMAX];        // (index in body 1, index in body 2)
  uint32_t fv[FMAX];     // face vertices a | b << 8 | c << 16
  uint16_t fa[FMAX][4];  // across edge e = (v_e, v_{e+1 mod 3}): face | its edge << 8
  uint32_t hz[FMAX];     // horizon edges (this step): a | b << 8 | face beyond << 16 | its edge << 24
  uint8_t hstart[VMAX];  // new face whose horizon edge starts at vertex
  uint8_t hend[VMAX];    // new face whose horizon edge ends at vertex
  OGX_HD int vertex(int f, int k) const { return (int)((fv[f] >> (8 * k)) & 0xffu); }
  OGX_HD int beyond(int f, int e) const { return fa[f][e] & 0xff; }
  OGX_HD bool alive(int f) const { return fn[f].w < INFINITY; }
};
// small capacity: 24 expansions (2.4 KB); a pair that needs more is handed to a
// full-capacity pass
constexpr int kEpaSmallIters = 24;
struct EpaMemSmall : EpaMemT<4 + kEpaSmallIters, 4 + 2 * kEpaSmallIters> {
  static constexpr bool kFull = false;
};
// full capacity: every pair within the 64-expansion cap (68 vertices, 132 faces); for the
// certified run every face's plane and every vertex are also kept in FP64
struct EpaMemCert : EpaMemT<kEpaVmax, kEpaFmax> {
  static constexpr bool kFull = true;
  double4 fn64[kEpaFmax];  // unit outward normal and plane distance, from exact points
  dv3 vp64[kEpaVmax];      // exact Minkowski points
};

// A small-capacity expansion that ran out of room, kept for the full-capacity pass to
// continue from instead of starting again: the polytope and the loop state at the top of
// the iteration that overflowed.  The full pass makes the same decisions up to there (the
// face slots do not depend on the capacity), so the result is the same as a restart.
struct EpaResume {
  int pair, nv, fend, it, st, status;
  float scale2;
  float4 fn[EpaMemSmall::kF];
  float4 vp[EpaMemSmall::kV];
  int2 vid[EpaMemSmall::kV];
  uint32_t fv[EpaMemSmall::kF];
  uint16_t fa[EpaMemSmall::kF][4];
};
// where a spilling expansion saves itself: cap records in buf, *count the next free one
// (buf null or full: the full pass restarts the contact)
struct EpaResumeSink {
  EpaResume* buf;
  int* count;
  int cap;
};
// The certified re-run.  An FP32 expansion that stops with the support still above the
// closest face by more than rounding (kEpaCertGain * scale; the FP32 test accepts up to
// epa_rel * scale), or whose support repeats a vertex before converging, is run again at
// full capacity with every face plane in FP64 from the exact points, visibility decided
// on those planes, exact (FP64) supports, and convergence when the support improves on
// the closest face by at most kEpaCertTol * max(1, scale).
constexpr float kEpaCertGain = 2.5e-7f;
constexpr double kEpaCertTol = 1e-10;
// Thin contacts: the closest face within kEpaThin * scale of the origin (thin bodies such
// as 1e-4-thick disks, or barely overlapping ones).  Their long, flat faces carry FP32
// normals whose rounding (~1e-6) can hide a support that improves on the face by more
// than the FP32 convergence tolerance; at FP32 convergence such a contact is checked with
// exact supports along its face's FP64 plane and run again certified if they improve on
// the face by more than that tolerance.
constexpr float kEpaThin = 1e-3f;
// Largest squared sine of the angle between the closest face and a neighbour the
// origin's projection moves to, for the FP32 pass to accept the neighbour's result.
constexpr float kEpaHopSin2 = 1e-10f;
constexpr double kEpaCertVis = 1e-12;
// Certified runs decide visibility on FP64 heights; the FP32 height of the rounded point
// over the rounded plane differs from it by less than 8 x 2^-24 x (|q|_1 + |w|) < 1.5e-6 scale
// (q and w at most scale), so farther from zero than this its sign is enough.
constexpr float kEpaVisBand = 4e-6f;

struct EpaOut {
  float dist;   // -depth for contacts, the GJK distance otherwise
  fv3 w0, w1;   // witnesses
  fv3 nrm;      // contact normal, body 1 -> body 2
  int status;
  int iters;
  int face[3][2];  // vertex index pairs of the final face (FP64 re-solve)
  bool polish;
  bool spill;      // ran out of (small) capacity: nothing written, run again at full capacity
  bool spill64;    // ... because the FP32 expansion met an inconsistent horizon: the re-run
                   // solves every face plane in FP64
  int resume;      // a capacity spill saved to this EpaResume record (-1: none)
  bool kept;       // no face was found: the GJK distance and witnesses stay (not set here)
};

OGX_HD fv3 unit_or_x(fv3 d) {
  const float n = sqrtf(dot(d, d));
  if (n > FLT_EPSILON) return d * (1.0f / n) ;
  return v3<float>(1.0f, 0.0f, 0.0f);
}

// Normal of a separated pair: the reference's normalize(w1 - w0) with (1,0,0) when the
// witnesses coincide (GJK/cpu/EPA.c:350-360).  In exact arithmetic w1 - w0 = -v, v the
// closest point of the Minkowski difference to the origin, and the normal is computed
// from -v: v carries the accuracy of the distance (each component rounded relative to
// itself), while the difference of two FP32 witnesses keeps their absolute rounding, a
// few 1e-7 of the coordinates, which is more than 1e-4 of a distance below ~1e-3.
OGX_HD fv3 sep_normal(const GjkState& g) { return unit_or_x(-g.v); }

// The same normal from a GJK simplex given by a caller (EPA-only calls): v is re-solved
// from the simplex's points of the two bodies (exact Minkowski differences, closest point
// in double-float, as the certified re-solve of the GJK pass does); where the simplex's
// vertex indices do not address the bodies, the reference's rule on the given witnesses.
OGX_HD fv3 simplex_sep_normal(const MemBodies& B, const gkSimplex& s) {
  const int n = s.nvrtx;
  bool ok = n >= 1 && n <= 3;
  xv3 P[3];
  for (int j = 0; j < 3; ++j) {
    if (!ok || j >= n) break;
    const int ia = s.vrtx_idx[j][0], ib = s.vrtx_idx[j][1];
    ok = ia >= 0 && ia < B.n[0] && ib >= 0 && ib < B.n[1];
    if (ok) P[j] = xdiff(B.point(0, ia), B.point(1, ib));
  }
  if (ok) {
    df lam[4];
    xv3 v;
    closest_on_simplex_t<df>(n, P, lam, v);
    return unit_or_x(v3<float>(-to_float(v.x), -to_float(v.y), -to_float(v.z)));
  }
  const fv3 w0 = v3<float>(s.witnesses[0][0], s.witnesses[0][1], s.witnesses[0][2]);
  const fv3 w1 = v3<float>(s.witnesses[1][0], s.witnesses[1][1], s.witnesses[1][2]);
  return unit_or_x(w1 - w0);
}

// A scan whose values are all NaN or -infinity (coordinates whose products overflow) finds no
// point: any one then, for the index is read with.
OGX_HD int found(int i) { return i == 0x7fffffff ? 0 : i; }

// support of the Minkowski difference along d (first maximum wins, EPA.c:307-344)
template <class Team, class Bodies>
OGX_HD fv3 msupport(const Team& t, const Bodies& B, fv3 d, int& ia, int& ib) {
  float ba, bb;
  B.scan(t, 0, d, ba, ia);
  B.scan(t, 1, -d, bb, ib);
  t.argmax_pair(ba, ia, bb, ib);
  ia = found(ia);
  ib = found(ib);
  return B.point(0, ia) - B.point(1, ib);
}

// FP64 plane (unit normal, offset) of the triangle q0, q1, q2; w = INFINITY when degenerate
OGX_LEAF double4 plane64(dv3 q0, dv3 q1, dv3 q2) {
  const dv3 m = cross(q1 - q0, q2 - q0);
  const double mm = dot(m, m);
  if (!(mm > 0.0)) return make_double4_(0.0, 0.0, 0.0, (double)INFINITY);
  const double inv = 1.0 / sqrt(mm);
  return make_double4_(m.x * inv, m.y * inv, m.z * inv, dot(m, q0) * inv);
}
// the same of polytope vertices a, b, c, from their exact points
template <class Mem, class Bodies>
OGX_HD double4 face_plane64(const Mem& M, const Bodies& B, int a, int b, int c) {
  return plane64(B.dpoint(0, M.vid[a].x) - B.dpoint(1, M.vid[a].y), B.dpoint(0, M.vid[b].x) - B.dpoint(1, M.vid[b].y),
                 B.dpoint(0, M.vid[c].x) - B.dpoint(1, M.vid[c].y));
}

// (degenerate: w infinite, never the closest face, never visible)
OGX_HD float4 rounded(double4 p) { return make_float4_((float)p.x, (float)p.y, (float)p.z, (float)p.w); }

// Thin-contact check at FP32 convergence: true when exact supports along face f's FP64
// plane improve on the face by more than tol.
template <class Team, class Bodies, class Mem>
OGX_HD bool thin_gain_exceeds(const Team& t, const Bodies& B, const Mem& M, int f, float tol) {
  const double4 p = face_plane64(M, B, M.vertex(f, 0), M.vertex(f, 1), M.vertex(f, 2));
  if (!(p.w < (double)INFINITY)) return false;
  const dv3 n64 = v3<double>(p.x, p.y, p.z);
  double ha, hb;
  float ma = -1.0f, mb = -1.0f;
  const fv3 n = floats(n64);
  exact_support(t, B, 0, n64, n, ma, &ha);
  exact_support(t, B, 1, -n64, -n, mb, &hb);
  return ha + hb - p.w > (double)tol;
}

// plane of face (a, b, c): FP32, FP64 from exact points for slivers
template <class Mem, class Bodies>
OGX_HD float4 face_plane(const Mem& M, const Bodies& B, int a, int b, int c, bool escalate, bool all64,
                         int& status) {
  const float4 P0 = M.vp[a], P1 = M.vp[b], P2 = M.vp[c];
  const fv3 p0 = v3<float>(P0.x, P0.y, P0.z);
  const fv3 e0 = v3<float>(P1.x, P1.y, P1.z) - p0;
  const fv3 e1 = v3<float>(P2.x, P2.y, P2.z) - p0;
  const fv3 n = cross(e0, e1);
  const float nn = dot(n, n);
  const float s = l1(e0) * l1(e1);
  float4 r;
  if (all64 || (escalate && nn < 1e-6f * s * s)) {
    // sine of the face angle below ~1e-3: FP32 normal unreliable
    status |= OGX_S_EPA_ESCALATED;
    return rounded(face_plane64(M, B, a, b, c));
  }
  if (nn > 0.0f) {
    const float inv = 1.0f / sqrtf(nn);
    r.x = n.x * inv;
    r.y = n.y * inv;
    r.z = n.z * inv;
    r.w = r.x * p0.x + r.y * p0.y + r.z * p0.z;
  } else {
    r.x = r.y = r.z = 0.0f;
    r.w = INFINITY;
  }
  return r;
}

// barycentric weights of the origin's projection on triangle (p0, p1, p2), clamped to
// the triangle's edges as EPA.c:238-304 does
OGX_HD int tri_weights(fv3 p0, fv3 p1, fv3 p2, float* l) {
  const fv3 e0 = p1 - p0, e1 = p2 - p0;
  const float d00 = dot(e0, e0), d01 = dot(e0, e1), d11 = dot(e1, e1);
  const float d20 = -dot(p0, e0), d21 = -dot(p0, e1);
  const float den = d00 * d11 - d01 * d01;
  if (fabsf(den) < FLT_EPSILON) {
    l[0] = l[1] = l[2] = 1.0f / 3.0f;
    return -1;
  }
  const float inv = 1.0f / den;
  const float u = (d11 * d20 - d01 * d21) * inv;
  const float v = (d00 * d21 - d01 * d20) * inv;
  const float w = 1.0f - u - v;
  if (w < 0.0f) {
    const fv3 e12 = p2 - p1;
    float tt = -dot(p1, e12) / dot(e12, e12);
    tt = fmaxf(0.0f, fminf(1.0f, tt));
    l[0] = 0.0f;
    l[1] = 1.0f - tt;
    l[2] = tt;
    return 1;  // beyond edge p1-p2 (edge 1 of the face)
  } else if (u < 0.0f) {
    float tt = -dot(p0, e1) / dot(e1, e1);
    tt = fmaxf(0.0f, fminf(1.0f, tt));
    l[0] = 1.0f - tt;
    l[1] = 0.0f;
    l[2] = tt;
    return 2;  // beyond edge p2-p0
  } else if (v < 0.0f) {
    float tt = -dot(p0, e0) / dot(e0, e0);
    tt = fmaxf(0.0f, fminf(1.0f, tt));
    l[0] = 1.0f - tt;
    l[1] = tt;
    l[2] = 0.0f;
    return 0;  // beyond edge p0-p1
  }
  l[0] = w;
  l[1] = u;
  l[2] = v;
  return -1;
}

// Result from face f.  When the origin's projection falls outside f and the face across
// that edge lies in the same plane (the Minkowski face of an edge-edge or face-face
// contact is split into coplanar triangles), the neighbour that holds the projection is
// used, so that w0 - w1 = depth * normal holds.
template <class Mem, class Bodies>
// With rerun_ok, returns true when the origin's projection leaves the closest face
// towards a neighbour more than 1e-5 rad off its plane (sine from the cross product of the
// two FP32 normals, kEpaHopSin2): nothing is emitted then and the caller runs the contact
// again with FP64 planes.  Without (the FP64-plane pass
// itself, whose closest face is picked on the planes rounded to float, so two faces a
// rounding apart can swap), the result comes from that near-coplanar neighbour, which
// holds the projection.
// dead: faces retired by a step that was not completed.
OGX_HD bool epa_emit(const Mem& M, const Bodies& B, int f, float tie, EpaOut& o, bool rerun_ok,
                     const typename Mem::Faces dead) {
  int a = M.vertex(f, 0), b = M.vertex(f, 1), c = M.vertex(f, 2);
  float l[3];
#pragma unroll 1
  for (int hop = 0; hop < 4; ++hop) {
    a = M.vertex(f, 0);
    b = M.vertex(f, 1);
    c = M.vertex(f, 2);
    const float4 P0 = M.vp[a], P1 = M.vp[b], P2 = M.vp[c];
    const int out = tri_weights(v3<float>(P0.x, P0.y, P0.z), v3<float>(P1.x, P1.y, P1.z),
                                v3<float>(P2.x, P2.y, P2.z), l);
    if (out < 0) break;
    const int g2 = M.beyond(f, out);
    const float4 nf = M.fn[f], ng = M.fn[g2];
    const bool near = M.alive(g2) && !dead.has(g2) && fabsf(ng.w - nf.w) <= tie &&
                      (nf.x * ng.x + nf.y * ng.y + nf.z * ng.z) > 1.0f - 1e-5f;
    if (!near) break;
    // In exact arithmetic the origin projects into the closest face of the convex
    // polytope, so a neighbour it leaves through is coplanar with it (a flat patch split
    // into triangles -- two points of one body against two of the other make an exact
    // parallelogram: the witnesses come from the neighbour).  A neighbour more than 1e-5
    // rad off -- FP32 planes made the polytope a little non-convex or ranked the faces
    // wrongly, on dense flat patches -- would give a normal up to a few 1e-4 off and
    // witnesses off the normal: the FP32 pass runs the contact again on FP64 planes.
    const float sx = nf.y * ng.z - nf.z * ng.y, sy = nf.z * ng.x - nf.x * ng.z, sz = nf.x * ng.y - nf.y * ng.x;
    if (sx * sx + sy * sy + sz * sz > kEpaHopSin2 && rerun_ok) return true;
    f = g2;
  }
  const int2 ia = M.vid[a], ib = M.vid[b], ic = M.vid[c];
  o.w0 = B.point(0, ia.x) * l[0] + B.point(0, ib.x) * l[1] + B.point(0, ic.x) * l[2];
  o.w1 = B.point(1, ia.y) * l[0] + B.point(1, ib.y) * l[1] + B.point(1, ic.y) * l[2];
  const float4 n = M.fn[f];
  o.kept = false;
  o.nrm = v3<float>(n.x, n.y, n.z);
  o.dist = -n.w;
  o.face[0][0] = ia.x;
  o.face[0][1] = ia.y;
  o.face[1][0] = ib.x;
  o.face[1][1] = ib.y;
  o.face[2][0] = ic.x;
  o.face[2][1] = ic.y;
  return false;
}

OGX_HD void epa_touch(fv3 a, fv3 b, EpaOut& o) {
  o.kept = false;
  o.dist = 0.0f;
  o.w0 = a;
  o.w1 = b;
  o.nrm = unit_or_x(b - a);
  o.status |= OGX_S_EPA_TOUCH;
}

// exact FP64 re-solve of the final face (plane, depth, witnesses)
template <class Bodies>
OGX_HD void epa_polish(const Bodies& B, EpaOut& o) {
  // double-float arithmetic (about 48 bits) on the FP32 pipes: FP64 issues at 1/64 of
  // the FP32 rate on this part, and the results are rounded to float
  fv3 A[3], Bq[3];
  xv3 Q[3];
  for (int k = 0; k < 3; ++k) {
    A[k] = B.point(0, o.face[k][0]);
    Bq[k] = B.point(1, o.face[k][1]);
    Q[k] = xdiff(A[k], Bq[k]);
  }
  const df zero = sc<df>(0.0f), one = sc<df>(1.0f);
  const xv3 m = cross(Q[1] - Q[0], Q[2] - Q[0]);
  const df mm = dot(m, m);
  if (!(mm > zero)) return;
  const df inv = one / df_sqrt(mm);
  xv3 n = m * inv;
  df d = dot(n, Q[0]);
  // keep the orientation chosen during the expansion
  if (n.x * sc<df>(o.nrm.x) + n.y * sc<df>(o.nrm.y) + n.z * sc<df>(o.nrm.z) < zero) {
    n = -n;
    d = -d;
  }
  // barycentric weights of the projection of the origin, clamped like tri_weights
  const xv3 e0 = Q[1] - Q[0], e1 = Q[2] - Q[0];
  const df d00 = dot(e0, e0), d01 = dot(e0, e1), d11 = dot(e1, e1);
  const df d20 = -dot(Q[0], e0), d21 = -dot(Q[0], e1);
  const df den = d00 * d11 - d01 * d01;
  const df third = one / sc<df>(3.0f);
  df l[3] = {third, third, third};
  if (den.hi != 0.0f) {
    const df u = (d11 * d20 - d01 * d21) / den;
    const df v = (d00 * d21 - d01 * d20) / den;
    const df w = one - u - v;
    if (w < zero) {
      const xv3 e12 = Q[2] - Q[1];
      df tt = -dot(Q[1], e12) / dot(e12, e12);
      tt = tt < zero ? zero : (tt > one ? one : tt);
      l[0] = zero; l[1] = one - tt; l[2] = tt;
    } else if (u < zero) {
      df tt = -dot(Q[0], e1) / dot(e1, e1);
      tt = tt < zero ? zero : (tt > one ? one : tt);
      l[0] = one - tt; l[1] = zero; l[2] = tt;
    } else if (v < zero) {
      df tt = -dot(Q[0], e0) / dot(e0, e0);
      tt = tt < zero ? zero : (tt > one ? one : tt);
      l[0] = one - tt; l[1] = tt; l[2] = zero;
    } else {
      l[0] = w; l[1] = u; l[2] = v;
    }
  }
  auto lift = [](fv3 p) { return v3<df>(sc<df>(p.x), sc<df>(p.y), sc<df>(p.z)); };
  const xv3 w0 = lift(A[0]) * l[0] + lift(A[1]) * l[1] + lift(A[2]) * l[2];
  const xv3 w1 = lift(Bq[0]) * l[0] + lift(Bq[1]) * l[1] + lift(Bq[2]) * l[2];
  o.w0 = v3<float>(to_float(w0.x), to_float(w0.y), to_float(w0.z));
  o.w1 = v3<float>(to_float(w1.x), to_float(w1.y), to_float(w1.z));
  o.nrm = v3<float>(to_float(n.x), to_float(n.y), to_float(n.z));
  o.dist = to_float(-d);
  o.status |= OGX_S_POLISHED;
}

// saves a small expansion for the full pass
template <class Team, class Mem>
OGX_HD void epa_save(const Team& t, const Mem& M, const EpaResumeSink& sink, EpaOut& o, int nv, int fend, int it,
                     int st, float scale2) {
  if (!sink.buf) return;
  int slot = -1;
  if (t.lane() == 0) {
#if defined(__CUDA_ARCH__)
    slot = atomicAdd(sink.count, 1);
#else
    slot = (*sink.count)++;
#endif
  }
  slot = t.imax(slot);
  if (slot >= sink.cap) return;
  EpaResume& R = sink.buf[slot];
#pragma unroll 1
  for (int j = t.lane(); j < nv; j += Team::L) {
    R.vp[j] = M.vp[j];
    R.vid[j] = M.vid[j];
  }
#pragma unroll 1
  for (int f = t.lane(); f < fend; f += Team::L) {
    R.fn[f] = M.fn[f];
    R.fv[f] = M.fv[f];
    for (int k = 0; k < 3; ++k) R.fa[f][k] = M.fa[f][k];
  }
  if (t.lane() == 0) {
    R.nv = nv;
    R.fend = fend;
    R.it = it;
    R.st = st;
    R.status = o.status;
    R.scale2 = scale2;
  }
  o.resume = slot;
}

// What both capacities start with: the output's flags, and the GJK simplex grown to a
// tetrahedron (EPA.c:369-583).  False: the pair is finished (separated, or only touching).
template <class Team, class Bodies>
OGX_HD bool epa_begin(const Team& t, const Bodies& B, const GjkState& g, EpaOut& o) {
  o.status = 0;
  o.iters = 0;
  o.polish = false;
  o.spill = false;
  o.spill64 = false;
  o.resume = -1;
  o.kept = true;
  if (g.n != 4 && g.dist > FLT_EPSILON) return false;  // separated (EPA.c:369-373)
  o.status |= OGX_S_EPA_RUN;
  return true;
}
template <class Team, class Bodies>
OGX_HD bool epa_grow(const Team& t, const Bodies& B, const GjkState& g, EpaOut& o, fv3* P, int* IA, int* IB) {
  int n = g.n;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    P[j] = g.P[j];
    IA[j] = g.ia[j];
    IB[j] = g.ib[j];
  }
  const float e2 = FLT_EPSILON * FLT_EPSILON;
  auto is_new = [&](fv3 q, int qa, int qb) {
    bool fresh = true;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const fv3 d = q - P[j];
      if (j < n && (dot(d, d) < e2 || (IA[j] == qa && IB[j] == qb))) fresh = false;
    }
    return fresh;
  };
  auto append = [&](fv3 q, int qa, int qb) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j == n) {
        P[j] = q;
        IA[j] = qa;
        IB[j] = qb;
      }
    ++n;
  };
  bool flip = false;  // the triangle's second direction
#pragma unroll 1
  while (n < 4) {
    fv3 d = P[0];
    if (n == 2) {
      const fv3 e = P[1] - P[0];
      fv3 axis = v3<float>(1.0f, 0.0f, 0.0f);
      const float el = sqrtf(dot(e, e));
      if (el > FLT_EPSILON && fabsf(e.x) > 0.9f * el) axis = v3<float>(0.0f, 1.0f, 0.0f);
      d = cross(e, axis);
      if (dot(d, d) < FLT_EPSILON) d = cross(e, v3<float>(0.0f, 0.0f, 1.0f));
    } else if (n == 3) {
      d = cross(P[1] - P[0], P[2] - P[0]);
      if (flip) d = -d;
    }
    int qa, qb;
    const fv3 q = msupport(t, B, d, qa, qb);
    if (is_new(q, qa, qb)) {
      append(q, qa, qb);
    } else if (n == 3 && !flip) {
      flip = true;
    } else {
      epa_touch(B.point(0, qa), B.point(1, qb), o);
      return false;
    }
  }
  return true;
}

// the plane of face (a, b, c) into slot s
template <bool kCert, class Mem, class Bodies>
OGX_HD float4 set_plane(Mem& M, const Bodies& B, int s, int a, int b, int c, bool escalate, bool all64, bool cert,
                        int& st) {
  float4 pl;
  if constexpr (kCert) {
    if (cert) {
      st |= OGX_S_EPA_ESCALATED;
      const double4 p = plane64(M.vp64[a], M.vp64[b], M.vp64[c]);
      M.fn64[s] = p;
      pl = rounded(p);
      M.fn[s] = pl;
      return pl;
    }
  }
  pl = face_plane(M, B, a, b, c, escalate, all64, st);
  M.fn[s] = pl;
  return pl;
}

#if defined(__CUDACC__)
// The certified run's planes of n faces (face(k, s, a, b, c): slot and vertices), three lanes
// per face, each with one component of every vector: plane64's operations, bit for bit, and
// set_plane's stores.  An FP64 instruction takes its quadrant's unit for about 65 cycles
// however many lanes are active, so the components side by side take 13 of them beside the
// square root and the reciprocal (~600 cycles each) where one lane per face took 29.  The
// full-capacity pass of 30k stress pairs 303 -> 289 us, of 5,003 ellipsoid pairs (3 contacts,
// one chain each) 74 -> 68.
template <class Mem, class Face>
__device__ __forceinline__ void planes64_by_component(Mem& M, int n, Face face, float& cbd, int& cbest) {
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int c = lane % 3, first = lane - c;
  const int li = first + (c + 1) % 3, lj = first + (c + 2) % 3;  // (lanes 30 and 31 take no face)
  for (int k0 = 0; k0 < n; k0 += 10) {
    const int k = k0 + lane / 3;
    const bool mine = lane < 30 && k < n;
    int s, va, vb, vc;
    face(mine ? k : 0, s, va, vb, vc);
    const double q0 = (&M.vp64[va].x)[c];
    const double e1 = (&M.vp64[vb].x)[c] - q0, e2 = (&M.vp64[vc].x)[c] - q0;
    const double e1i = __shfl_sync(full, e1, li), e1j = __shfl_sync(full, e1, lj);
    const double e2i = __shfl_sync(full, e2, li), e2j = __shfl_sync(full, e2, lj);
    const double m = e1i * e2j - e1j * e2i;
    const double m2 = m * m, mq = m * q0;
    auto sum = [&](double x) {
      return __shfl_sync(full, x, first) + __shfl_sync(full, x, first + 1) + __shfl_sync(full, x, first + 2);
    };
    const double mm = sum(m2), mq3 = sum(mq);
    double x = 0.0, w = (double)INFINITY;
    if (mm > 0.0) {
      const double inv = 1.0 / sqrt(mm);
      x = m * inv;
      w = mq3 * inv;
    }
    if (mine) {
      const float fw = (float)w;
      (&M.fn64[s].x)[c] = x;
      (&M.fn[s].x)[c] = (float)x;
      if (c == 0) {
        M.fn64[s].w = w;
        M.fn[s].w = fw;
        if (fw < cbd || (fw == cbd && s < cbest)) {
          cbd = fw;
          cbest = s;
        }
      }
    }
  }
}
#endif

// EPA for one pair whose GJK result is g.  `M` is this pair's shared working set.
//
// One expansion step, with the faces of the polytope split over the team's lanes
// (face f on lane f mod L):
//   1. every lane tests its live faces for visibility from the new point q and keeps the
//      closest face that stays (not visible);
//   2. visible faces are ranked in increasing slot order and horizon edges in increasing
//      (face, edge) order with ballots, so slot assignment does not depend on L; new face
//      k takes the k-th visible slot, then fresh slots at the end of the used range;
//   3. faces beyond the horizon are relinked to the new faces, the visible faces retired;
//   4. new faces are linked to each other through the per-vertex tables and their planes
//      computed; the closest new face joins the lane's candidate.
// The next step's closest face is the team's minimum over the candidates.
//
// The steps are arranged for the length of the dependent chain, which is what bounds a
// contact (an expansion by one warp took ~11,000 cycles as byte flags, per-face lists and
// searched links in shared memory, ~4,000 now): the visible set is a bit set in registers,
// the horizon one ballot over the visible faces' edges, the relinking one store per edge (a
// link carries the neighbour's edge), and the scale's square root is taken only when the
// scale grows.
//
// EpaMemSmall: can_spill (always set in the pipelines) lets a contact that needs the full
// capacity or the certified run leave with o.spill set; sink: where a capacity spill saves
// itself (FP32 planes only).  EpaMemCert: no larger capacity; rs: a saved expansion to continue
// instead of starting from the GJK simplex.  kCert (full capacity only): with FP64 face planes on, run
// the certified expansion described at kEpaCertGain.
// The loop state of one expansion (registers that live through the loop: kept few).
template <class Mem>
struct EpaRun {
  int nv, fend, it, st;
  float scale2, root;  // largest |vertex|^2, and its square root (at convergence: of the last scale)
  // per-lane closest candidate (slot, plane distance); -1 = none
  float cbd;
  int cbest;
  int best;        // the step's closest face
  uint32_t flags;  // kRun*: how the loop ended
  float amax0, amax1;  // the bodies' largest |coordinate| (certified run)
};
constexpr uint32_t kRunDone = 1;    // ended, not by the iteration cap
constexpr uint32_t kRunAgain = 2;   // leaves for the certified run
constexpr uint32_t kRunThin = 4;    // a thin contact, to be checked
constexpr uint32_t kRunHalted = 8;  // stopped half way through a step: the faces it retired are in M.hz
constexpr uint32_t kRunLate = 16;   // capacity spill found after the vertex was added

// The polytope's first faces.  False: the pair is finished already, its result in o.
template <bool kCert = false, class Team, class Bodies, class Mem>
OGX_HD bool epa_start(const Team& t, const Bodies& B, const Config& cfg, const GjkState& g, Mem& M, EpaOut& o,
                      EpaRun<Mem>& r, const EpaResume* rs = nullptr) {
  const int L = Team::L;
  const int lane = t.lane();
  const bool escalate = (cfg.flags & OGX_F_FP64_ESCALATE) != 0;
  const bool all64 = (cfg.flags & OGX_F_EPA_FP64_PLANES) != 0;
  const bool cert = kCert && all64;
  if (!epa_begin(t, B, g, o)) return false;
  float& scale2 = r.scale2;
  float& cbd = r.cbd;
  int& cbest = r.cbest;
  int& st = r.st;
  scale2 = 0.0f;
  st = 0;
  cbd = INFINITY;
  cbest = -1;
  int nv = 4, fend = 4;
  int it = 0;
  if (Mem::kFull && rs) {
    nv = rs->nv;
    fend = rs->fend;
    it = rs->it;
    st = rs->st;
    scale2 = rs->scale2;
    o.status = rs->status;
#pragma unroll 1
    for (int j = lane; j < nv; j += L) {
      M.vp[j] = rs->vp[j];
      M.vid[j] = rs->vid[j];
    }
#pragma unroll 1
    for (int f = lane; f < fend; f += L) {
      const float4 pl = rs->fn[f];
      M.fn[f] = pl;
      M.fv[f] = rs->fv[f];
      for (int k = 0; k < 3; ++k) M.fa[f][k] = rs->fa[f][k];
      if (pl.w < cbd) {
        cbd = pl.w;
        cbest = f;
      }
    }
    t.sync();
  } else {
    fv3 P[4];
    int IA[4], IB[4];
    if (!epa_grow(t, B, g, o, P, IA, IB)) return false;
    // outward faces of a positively oriented tetrahedron (0,1,2,3); swap 1 and 2 otherwise:
    // (0, i2, i1), (0, i1, 3), (i1, i2, 3), (i2, 0, 3).  The face across edge k of face f
    // (edge k = vertices k, k+1 mod 3) and its edge are the same for both orientations:
    // {3,2,1}, {0,2,3}, {0,3,1}, {0,1,2} across edges {0,0,0}, {2,2,1}, {1,2,1}, {0,2,1}.
    const float vol = dot(P[1] - P[0], cross(P[2] - P[0], P[3] - P[0]));
    const int i1 = vol >= 0.0f ? 1 : 2, i2 = vol >= 0.0f ? 2 : 1;
    if (lane == 0) {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        M.vp[j] = make_float4_(P[j].x, P[j].y, P[j].z, 0.0f);
        M.vid[j] = make_int2_(IA[j], IB[j]);
        if constexpr (kCert)
          if (cert) M.vp64[j] = B.dpoint(0, IA[j]) - B.dpoint(1, IB[j]);
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) scale2 = fmaxf(scale2, dot(P[j], P[j]));
    t.sync();
#pragma unroll 1
    for (int f = lane; f < 4; f += L) {
      const int va = f == 2 ? i1 : (f == 3 ? i2 : 0);
      const int vb = f == 0 ? i2 : (f == 1 ? i1 : (f == 2 ? i2 : 0));
      const int vc = f == 0 ? i1 : 3;
      M.fv[f] = (uint32_t)(va | vb << 8 | vc << 16);
      M.fa[f][0] = (uint16_t)(f == 0 ? 3 : (f == 1 ? 0 | 2 << 8 : (f == 2 ? 0 | 1 << 8 : 0)));
      M.fa[f][1] = (uint16_t)(f == 0 ? 2 : (f == 1 ? 2 | 2 << 8 : (f == 2 ? 3 | 2 << 8 : 1 | 2 << 8)));
      M.fa[f][2] = (uint16_t)(f == 0 ? 1 : (f == 1 ? 3 | 1 << 8 : (f == 2 ? 1 | 1 << 8 : 2 | 1 << 8)));
      const float4 pl = set_plane<kCert>(M, B, f, va, vb, vc, escalate, all64, cert, st);
      if (pl.w < cbd) {
        cbd = pl.w;
        cbest = f;
      }
    }
    t.sync();
  }
  r.nv = nv;
  r.fend = fend;
  r.it = it;
  r.root = sqrtf(scale2);
  r.best = -1;
  r.flags = 0u;
  r.amax0 = r.amax1 = -1.0f;
  return true;
}

// One expansion (r.it < the cap).  False: the loop has ended.  live = false: a team that only
// takes part in the operations of its warp's other teams.
template <bool kCert = false, class Team, class Bodies, class Mem>
OGX_HD bool epa_step(const Team& t, const Bodies& B, const Config& cfg, Mem& M, EpaOut& o, EpaRun<Mem>& r,
                     bool can_spill, bool live = true) {
  static_assert(Mem::kFull || !kCert, "certified runs need the full capacity");
  const int L = Team::L;
  const int lane = t.lane();
  const bool escalate = (cfg.flags & OGX_F_FP64_ESCALATE) != 0;
  const bool all64 = (cfg.flags & OGX_F_EPA_FP64_PLANES) != 0;
  const bool cert = kCert && all64;
#if defined(__CUDA_ARCH__)
  const bool by_component = cert && L == 32;
#else
  const bool by_component = false;
#endif
  // may the contact be run again with FP64 planes?
  const bool rerun = !Mem::kFull && can_spill && escalate;
  // closest live face
  float bd = live ? r.cbd : INFINITY;
  int best = live ? r.cbest : -1;
  t.argmin(bd, best);
  if (live) {
    ++r.it;
    r.best = best;
    if (best < 0 || !(bd < INFINITY)) {
      o.status |= OGX_S_EPA_TOPOLOGY;
      r.best = -1;
      r.flags = kRunDone;
      live = false;
    }
  }
  int qa = 0, qb = 0;
  fv3 q = v3<float>(0.0f, 0.0f, 0.0f);
  dv3 q64 = v3<double>(0.0, 0.0, 0.0);
  float ac = 0.0f, bc = 0.0f;  // this lane's coordinate of q's points (by_component)
  float qq = 0.0f, scale = 0.0f;  // |q|^2, sqrt(max(scale2, |q|^2))
  bool conv = false;
  float gain = 0.0f, tol = 0.0f;
  if (kCert && cert) {
    if constexpr (kCert) {
      if (live) {
        // exact supports along the closest face's FP64 normal
        const double4 pl = M.fn64[best];
        const dv3 n64 = v3<double>(pl.x, pl.y, pl.z);
        const float4 nf = M.fn[best];  // rounded(pl)
        const fv3 n = v3<float>(nf.x, nf.y, nf.z);
        float ea, eb;
        qa = exact_support<Team, Bodies, double>(t, B, 0, n64, n, r.amax0, nullptr, &ea);
        qb = exact_support<Team, Bodies, double>(t, B, 1, -n64, -n, r.amax1, nullptr, &eb);
        const fv3 pa = B.point(0, qa), pb = B.point(1, qb);
        q = pa - pb;
        if (by_component) {
          static_assert(!kCert || !Bodies::kExact64, "the points are floats");
          ac = lane == 0 ? pa.x : (lane == 1 ? pa.y : pa.z);
          bc = lane == 0 ? pb.x : (lane == 1 ? pb.y : pb.z);
        } else {
          q64 = B.dpoint(0, qa) - B.dpoint(1, qb);
        }
        qq = dot(q, q);
        scale = qq > r.scale2 ? sqrtf(qq) : r.root;
        // The support's gain over the face.  Its FP32 value is within ea + eb (the supports'
        // bounds) and a few roundings of the terms; only a gain nearer the tolerance than that
        // is evaluated in FP64.
        const float fa = sdot(pa, n);
        const float fb = sdot(pb, -n);
        const float fw = nf.w;
        const float slack = 2.0f * (ea + eb) + 4.0f * FLT_EPSILON * (fabsf(fa) + fabsf(fb) + fabsf(fw)) +
                            2e-10f * fmaxf(1.0f, scale);
        conv = !(fa + fb - fw > slack);
        if (conv) {
          const dv3 xa = B.dpoint(0, qa), xb = B.dpoint(1, qb);
          const double ha = xa.x * n64.x + xa.y * n64.y + xa.z * n64.z;
          const double hb = xb.x * -n64.x + xb.y * -n64.y + xb.z * -n64.z;
          conv = !(ha + hb - pl.w > kEpaCertTol * fmax(1.0, (double)scale));
        }
      }
    }
  } else {
    fv3 n = v3<float>(0.0f, 0.0f, 0.0f);
    float ba = -INFINITY, bb = -INFINITY;
    if (live) {
      const float4 nf = M.fn[best];
      n = v3<float>(nf.x, nf.y, nf.z);
      B.scan(t, 0, n, ba, qa);
      B.scan(t, 1, -n, bb, qb);
    }
    t.argmax_pair(ba, qa, bb, qb);
    if (live) {
      qa = found(qa);
      qb = found(qb);
      q = B.point(0, qa) - B.point(1, qb);
      qq = dot(q, q);
      scale = qq > r.scale2 ? sqrtf(qq) : r.root;
      tol = fmaxf(cfg.epa_tol, cfg.epa_rel * scale);
      gain = dot(n, q) - bd;
      conv = gain < tol;
    }
  }
  if (live && conv) {
    // with room left for an improvement, the certified run decides
    const bool room = rerun && !all64 && gain > kEpaCertGain * scale;
    // a thin contact: the FP32 test may have been fooled by the face normal's rounding;
    // checked after the loop (its FP64 scans would weigh on the loop's registers)
    const bool thin = rerun && !all64 && !(gain > kEpaCertGain * scale) && bd < kEpaThin * scale;
    r.flags = kRunDone | (room ? kRunAgain : 0u) | (thin ? kRunThin : 0u);
    r.root = scale;
    o.status |= OGX_S_EPA_CONVERGED;
    live = false;
  }
  bool dup = false;
  if (live) {
#pragma unroll 1
    for (int j = lane; j < r.nv; j += L) {
      const int2 id = M.vid[j];
      dup |= (id.x == qa && id.y == qb);
    }
  }
  if (t.any(dup)) {
    // the support is already a vertex although the closest face is not converged:
    // FP32 planes put a vertex in front of a face; re-run certified
    r.flags = kRunDone | (rerun && !all64 ? kRunAgain : 0u);
    o.status |= OGX_S_EPA_DUPLICATE;
    live = false;
  }
  if (live && r.nv >= Mem::kV) {
    r.flags = kRunDone;
    if (!Mem::kFull && can_spill)
      o.spill = true;
    else
      o.status |= OGX_S_EPA_CAPACITY;
    live = false;
  }
  const int p = r.nv;
  float vis_eps = 0.0f;
  float cbd = INFINITY;
  int cbest = -1;
  if (live) {
    if (lane == 0) {
      M.vp[p] = make_float4_(q.x, q.y, q.z, 0.0f);
      M.vid[p] = make_int2_(qa, qb);
      if constexpr (kCert)
        if (cert && !by_component) M.vp64[p] = q64;
    }
#if defined(__CUDA_ARCH__)
    if constexpr (kCert) {
      if (by_component) {
        // a component per lane (planes64_by_component)
        if (lane < 3) (&M.vp64[p].x)[lane] = (double)ac - (double)bc;
        t.sync();
        q64 = M.vp64[p];
      }
    }
#endif
    ++r.nv;
    r.scale2 = fmaxf(r.scale2, qq);
    r.root = scale;
    vis_eps = cfg.epa_vis * scale;
  }

  // 1. faces seen from q; the closest face that stays
  typename Mem::Faces vis;
  vis.clear();
  const int rounds = t.warp_max(live ? r.fend : 0);
#pragma unroll 1
  for (int f0 = 0; f0 < rounds; f0 += L) {
    const int f = f0 + lane;
    float4 fp = make_float4_(0.0f, 0.0f, 0.0f, INFINITY);
    if (live && f < r.fend) fp = M.fn[f];
    const float h = (fp.x * q.x + fp.y * q.y + fp.z * q.z) - fp.w;
    bool s = h > vis_eps;
    if constexpr (kCert) {
      if (cert) {
        // the rounded plane and point are within 2e-6 scale of the FP64 height: only
        // heights nearer zero than that need it
        s = h > 0.0f;
        if (f < r.fend && fabsf(h) <= kEpaVisBand * scale) {
          const double4 pl = M.fn64[f];
          s = (pl.x * q64.x + pl.y * q64.y + pl.z * q64.z) - pl.w > kEpaCertVis * (double)scale;
        }
      }
    }
    if (!s && fp.w < cbd) {
      cbd = fp.w;
      cbest = f;
    }
    vis.put(f0, t.ballot(s));
  }
  // 2. horizon edges: edge e of a visible face whose neighbour is not visible
  const int nvis = vis.count();
  int htot = 0;
  const int edges = t.warp_max(3 * nvis);
#pragma unroll 1
  for (int i0 = 0; i0 < edges; i0 += L) {
    const int i = i0 + lane;
    bool h = false;
    uint32_t edge = 0u;
    if (i < 3 * nvis) {
      const int k = (int)(((uint32_t)i * 43691u) >> 17);  // i / 3
      const int e = i - 3 * k;
      const int f = vis.nth(k);
      const uint32_t nb = M.fa[f][e], v = M.fv[f];
      h = !vis.has((int)(nb & 0xffu));
      edge = ((v >> (8 * e)) & 0xffu) | ((v >> (e == 2 ? 0 : 8 * e + 8)) & 0xffu) << 8 | (nb & 0xffu) << 16 |
             (nb >> 8) << 24;
    }
    const uint32_t m = t.ballot(h);
    const int k = htot + popc32(m & t.below());
    if (h && k < Mem::kF) M.hz[k] = edge;
    htot += popc32(m);
  }
  // new face k goes to the k-th visible slot, else to fresh slot fend + k - nvis
  const int fresh = htot > nvis ? htot - nvis : 0;
  if (live) {
    if (!vis.has(best) || htot < 3) {
      // the closest face must be seen (gain >= tol > vis threshold) and have a horizon;
      // otherwise stop, or start again with FP64 planes in the full pass
      r.flags = kRunDone | (rerun ? kRunAgain : 0u);
      o.status |= OGX_S_EPA_TOPOLOGY;
      live = false;
    } else if (r.fend + fresh > Mem::kF) {
      r.flags = kRunDone | kRunLate;
      if (!Mem::kFull && can_spill)
        o.spill = true;
      else
        o.status |= OGX_S_EPA_CAPACITY;
      live = false;
    }
  }
  if (!live) htot = 0;
  t.sync();
  // 3. relink the faces outside the horizon, index the horizon by its vertices.  The lane's
  // first edge stays in registers; only a horizon longer than the team is wide loops.
  auto slot_of = [&](int k) { return k < nvis ? vis.nth(k) : r.fend + k - nvis; };
  auto relink = [&](uint32_t h, int s) {
    M.fa[(h >> 16) & 0xffu][h >> 24] = (uint16_t)s;
    M.hstart[h & 0xffu] = (uint8_t)s;
    M.hend[(h >> 8) & 0xffu] = (uint8_t)s;
  };
  uint32_t h0 = 0u;
  int s0 = 0;
  if (lane < htot) {
    h0 = M.hz[lane];
    s0 = slot_of(lane);
    relink(h0, s0);
  }
#pragma unroll 1
  for (int k = lane + L; k < htot; k += L) relink(M.hz[k], slot_of(k));
  t.sync();
  // a vertex that starts (or ends) two horizon edges means the horizon is not one
  // simple loop; keep the closest face found this step and stop
  const int a0 = (int)(h0 & 0xffu), b0 = (int)((h0 >> 8) & 0xffu);
  bool bad = false;
  int link1 = 0, link2 = 0;  // the new faces across the new face's edges b-p and p-a
  if (lane < htot) {
    bad = M.hstart[a0] != s0 || M.hend[b0] != s0;
    link1 = M.hstart[b0];
    link2 = M.hend[a0];
  }
#pragma unroll 1
  for (int k = lane + L; k < htot; k += L) {
    const int s = slot_of(k);
    const uint32_t h = M.hz[k];
    bad |= (M.hstart[h & 0xffu] != s) || (M.hend[(h >> 8) & 0xffu] != s);
  }
  if (t.any(bad)) {
    r.flags = kRunDone | kRunHalted | (rerun ? kRunAgain : 0u);
    o.status |= OGX_S_EPA_TOPOLOGY;
    if (lane == 0) vis.save(M.hz);
    live = false;
    htot = 0;
  }
  // 4. new face (a, b, p) across each horizon edge a->b
#pragma unroll 1
  for (int k = lane; k < htot; k += L) {
    if (k >= L) {
      s0 = slot_of(k);
      h0 = M.hz[k];
      link1 = M.hstart[(h0 >> 8) & 0xffu];
      link2 = M.hend[h0 & 0xffu];
    }
    M.fv[s0] = (h0 & 0xffffu) | (uint32_t)p << 16;
    M.fa[s0][0] = (uint16_t)((h0 >> 16 & 0xffu) | (h0 >> 24) << 8);
    M.fa[s0][1] = (uint16_t)(link1 | 2u << 8);
    M.fa[s0][2] = (uint16_t)(link2 | 1u << 8);
    if (by_component) continue;
    const float4 pl = set_plane<kCert>(M, B, s0, (int)(h0 & 0xffu), (int)((h0 >> 8) & 0xffu), p, escalate, all64,
                                       cert, r.st);
    if (pl.w < cbd || (pl.w == cbd && s0 < cbest)) {
      cbd = pl.w;
      cbest = s0;
    }
  }
#if defined(__CUDA_ARCH__)
  if constexpr (kCert && Team::L == 32) {
    if (by_component) {
      r.st |= OGX_S_EPA_ESCALATED;
      planes64_by_component(
          M, htot,
          [&](int k, int& s, int& va, int& vb, int& vc) {
            const uint32_t h = M.hz[k];
            s = slot_of(k);
            va = (int)(h & 0xffu);
            vb = (int)((h >> 8) & 0xffu);
            vc = p;
          },
          cbd, cbest);
    }
  }
#endif
  if (live) {
#pragma unroll 1
    for (int k = htot + lane; k < nvis; k += L) M.fn[vis.nth(k)] = make_float4_(0.0f, 0.0f, 0.0f, INFINITY);
    r.fend += fresh;
    r.cbd = cbd;
    r.cbest = cbest;
  }
  t.sync();
  return live;
}

// Keeps an expansion that outgrew the small capacity: the polytope as it was at the top of the
// last step.  With FP64 planes the full pass is a certified run, whose FP64 planes and points a
// record does not hold: that one starts again.
template <class Team, class Mem>
OGX_HD void epa_save_run(const Team& t, const Config& cfg, const Mem& M, const EpaResumeSink& sink, EpaOut& o,
                         const EpaRun<Mem>& r) {
  if (!(cfg.flags & OGX_F_EPA_FP64_PLANES))
    epa_save(t, M, sink, o, r.flags & kRunLate ? r.nv - 1 : r.nv, r.fend, r.it - 1, r.st, r.scale2);
}

// The result once the loop has ended; a capacity spill (o.spill, at the top of its last
// expansion) saves itself.
template <bool kCert = false, class Team, class Bodies, class Mem>
OGX_HD void epa_finish(const Team& t, const Bodies& B, const Config& cfg, Mem& M, EpaOut& o, const EpaRun<Mem>& r,
                       bool can_spill, const EpaResumeSink& sink) {
  if (o.spill) {
    if constexpr (!Mem::kFull) epa_save_run(t, cfg, M, sink, o, r);
    return;
  }
  const bool escalate = (cfg.flags & OGX_F_FP64_ESCALATE) != 0;
  const bool all64 = (cfg.flags & OGX_F_EPA_FP64_PLANES) != 0;
  const bool cert = kCert && all64;
  const bool rerun = !Mem::kFull && can_spill && escalate;
  bool again = (r.flags & kRunAgain) != 0u;
  if (!again) {
    o.iters = r.it;
    o.status |= r.st ? OGX_S_EPA_ESCALATED : 0;
    o.status |= cert ? OGX_S_EPA_CERTIFIED : 0;
    int best = r.best;
    if (!(r.flags & kRunDone)) {
      // iteration cap: closest current face
      float bd = r.cbd;
      best = r.cbest;
      t.argmin(bd, best);
      o.status |= OGX_S_EPA_CAP;
    }
    if (!Mem::kFull && (r.flags & kRunThin) && best >= 0)
      again = thin_gain_exceeds(t, B, M, best, fmaxf(cfg.epa_tol, cfg.epa_rel * r.root));
    if (!again && best >= 0) {
      typename Mem::Faces dead;
      dead.clear();
      if (r.flags & kRunHalted) dead.load(M.hz);
      again = epa_emit(M, B, best, fmaxf(cfg.epa_tol, cfg.epa_rel * sqrtf(r.scale2)), o, rerun && !all64, dead);
      o.polish = !again && (cfg.flags & OGX_F_FP64_POLISH) != 0;
    }
  }
  o.spill = o.spill64 = again;
}

// r: the loop's state when it ended
template <bool kCert = false, class Team, class Bodies, class Mem>
OGX_HD void epa_pair(const Team& t, const Bodies& B, const Config& cfg, const GjkState& g, Mem& M, EpaOut& o,
                     bool can_spill, EpaResumeSink sink, const EpaResume* rs, EpaRun<Mem>& r) {
  if (epa_start<kCert>(t, B, cfg, g, M, o, r, rs)) {
#pragma unroll 1
    while (r.it < cfg.epa_max_iter && epa_step<kCert>(t, B, cfg, M, o, r, can_spill)) {
    }
    epa_finish<kCert>(t, B, cfg, M, o, r, can_spill, sink);
  }
  if (o.kept) {
    o.dist = g.dist;
    o.w0 = g.w0;
    o.w1 = g.w1;
    o.nrm = unit_or_x(g.w1 - g.w0);
  }
}

template <bool kCert = false, class Team, class Bodies, class Mem>
OGX_HD void epa_pair(const Team& t, const Bodies& B, const Config& cfg, const GjkState& g, Mem& M, EpaOut& o,
                     bool can_spill, EpaResumeSink sink = EpaResumeSink{nullptr, nullptr, 0},
                     const EpaResume* rs = nullptr) {
  EpaRun<Mem> r;
  epa_pair<kCert>(t, B, cfg, g, M, o, can_spill, sink, rs, r);
}

}  // namespace ogx
