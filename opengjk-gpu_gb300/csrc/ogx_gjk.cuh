// ogx_gjk.cuh -- GJK distance for one pair, run by a team of L lanes.
//
// Algorithm (the reference's GJK, GJK/cpu/openGJK.c:952-1056 and
// GJK/gpu/openGJK.cu:1253-1425): start from v = A[0] - B[0]; each iteration takes the
// support points s_A(-v), s_B(v), stops when the new point cannot reduce |v| (relative
// gap test), otherwise appends w = s_A - s_B to the simplex and runs the signed-volume
// sub-distance algorithm (Montanari's hff tests, openGJK.c:219-613), which returns the
// point of the simplex closest to the origin and drops the vertices it does not need.
//
// What differs from the reference, and why:
//  * The support scans are split over the team's lanes and combined with a shuffle
//    argmax; the tie rule (keep the previous support unless strictly beaten, then the
//    lowest index) is the reference CPU's rule (openGJK.c:615-639).
//  * Every lane runs the sub-distance redundantly, so nothing is broadcast.
//  * The sub-distance runs in FP32.  Each sign decision carries a forward error bound;
//    if any decision of a step falls inside its bound, the whole step is re-run in FP64
//    on the exact Minkowski points re-read from the pool (OGX_F_FP64_ESCALATE).
//  * Termination also stops when the support pair is already in the simplex (no
//    progress is possible) and when the gap is below FP32 rounding of |v| |w|.
//  * The final simplex of a separated pair is re-solved in FP64 (exact closest point of
//    the final feature, certified by an exact support check, else GJK continues in FP64;
//    OGX_F_FP64_POLISH); on the device that runs as a separate pass.
#pragma once

#include "ogx_common.cuh"
#include "ogx_subdist.cuh"

namespace ogx {

template <class T>
struct Vx {
  vec3<T> p;
  int k;  // slot of this vertex in the caller's simplex
};

template <class T>
struct Sx {
  int n;
  Vx<T> v[4];
};

// The predicates and projections of the signed-volume step on exact points.  Each is one
// out-of-line function, evaluated only where the decision asks for it.

// (p - q) . p > 0 : the origin projects beyond p towards q (openGJK.c:219-230)
template <class T>
OGX_LEAF bool edge_keeps(vec3<T> p, vec3<T> q) {
  T acc = T(0);
  acc += (p.x * p.x - p.x * q.x);
  acc += (p.y * p.y - p.y * q.y);
  acc += (p.z * p.z - p.z * q.z);
  return acc > T(0);
}

// origin beyond edge pq, away from r, in the plane pqr (openGJK.c:232-248)
template <class T>
OGX_LEAF bool edge_drops(vec3<T> p, vec3<T> q, vec3<T> r) {
  const vec3<T> e1 = q - p, e2 = r - p;
  const vec3<T> nrm = cross(e1, cross(e1, e2));
  return dot(p, nrm) < T(0);
}

// p . (q x r) <= 0 (openGJK.c:250-255); also the sign of the tetrahedron's volume
template <class T>
OGX_LEAF bool face_drops(vec3<T> p, vec3<T> q, vec3<T> r) {
  return dot(p, cross(q, r)) <= T(0);
}

template <class T>
OGX_LEAF vec3<T> onto_line(vec3<T> p, vec3<T> q) {
  const vec3<T> d = p - q;
  const T t = dot(p, d) / dot(d, d);
  return p - d * t;
}

template <class T>
OGX_LEAF vec3<T> onto_plane(vec3<T> p, vec3<T> q, vec3<T> r) {
  const vec3<T> nrm = cross(p - q, p - r);
  return nrm * (dot(nrm, p) / dot(nrm, nrm));
}

// predicate `m` (one PB_* bit) of the step on s (n points, newest last), on exact points
template <class T>
OGX_LEAF bool exact_bit(const Vx<T>* s, int n, uint32_t m) {
  const vec3<T> q1 = s[n - 1].p;
  if (m < PB_NEG) return edge_keeps(q1, s[m >> 1].p);  // 1, 2, 4: slots 0, 1, 2
  if (m < (1u << PB_D)) {
    if (m == PB_NEG) return face_drops(s[1].p - q1, s[0].p - q1, s[2].p - q1);
    const int j = m == PB_F2 ? 1 : (m == PB_F3 ? 0 : 2), k = m == PB_F2 ? 0 : (m == PB_F3 ? 2 : 1);
    return face_drops(q1, s[j].p, s[k].p);
  }
  // hff2 pairs in dpair() order: (0,1) (1,0) (0,2) (2,0) (1,2) (2,1)
  const int d = m < (4u << PB_D) ? (m < (2u << PB_D) ? 0 : 1)
                                 : (m < (16u << PB_D) ? (m < (8u << PB_D) ? 2 : 3) : (m < (32u << PB_D) ? 4 : 5));
  const int lo = d < 4 ? 0 : 1, hi = d < 2 ? 1 : 2;
  return edge_drops(q1, s[(d & 1) ? hi : lo].p, s[(d & 1) ? lo : hi].p);
}

// Signed-volume step (openGJK.c:257-613) on exact points: reduces s (2 to 4 points, newest
// last) to the vertices it needs and sets dir to its closest point to the origin.  The
// decision is the FP32 step's, on exactly evaluated bits: `bits` are its predicates, those
// in `known` already right (step_known); the others are evaluated when the decision comes to
// depend on them, each once.
template <class T>
OGX_LEAF void subdistance(Sx<T>& s, vec3<T>& dir, const uint32_t* subtab, uint32_t bits, uint32_t known) {
  const int n = s.n;
  if (n < 2) return;
  SubOut o;
#pragma unroll 1
  for (;;) {
    o = step_decide(n, bits, subtab);
    uint32_t need = o.used & ~known;
    if (need == 0u) break;
    need &= 0u - need;  // the lowest one first: the edge tests, then the faces, then the rest
    known |= need;
    bits = exact_bit(s.v, n, need) ? bits | need : bits & ~need;
  }
  const vec3<T> q1 = s.v[n - 1].p;
  switch (o.kind) {
    case SO_VERTEX: dir = q1; break;
    case SO_LINE: dir = onto_line(q1, s.v[o.a].p); break;
    case SO_PLANE: dir = onto_plane(q1, s.v[o.a].p, s.v[o.b].p); break;
    case SO_ZERO: dir = v3<T>(T(0), T(0), T(0)); break;
    default: break;  // undecided: unchanged
  }
  if (o.n == 4) return;
  // (slots are numbered for the tetrahedron, newest = 3)
  const Vx<T> r0 = s.v[o.s[0] == 3 ? n - 1 : o.s[0]], r1 = s.v[o.s[1] == 3 ? n - 1 : o.s[1]],
              r2 = s.v[o.s[2] == 3 ? n - 1 : o.s[2]];
  s.n = o.n;
  s.v[0] = r0;
  if (o.n > 1) s.v[1] = r1;
  if (o.n > 2) s.v[2] = r2;
}

// --------------------------------------------------------------------------------
// exact closest point of a simplex with <= 3 vertices to the origin, FP64
// (region tests of Ericson, Real-Time Collision Detection, sec. 5.1.5, restated)

template <class T>
OGX_LEAF void closest_on_simplex_t(int n, const vec3<T>* P, T* lam, vec3<T>& v) {
  const T zero = sc<T>(0.0f), one = sc<T>(1.0f);
  lam[0] = one;
  lam[1] = lam[2] = lam[3] = zero;
  if (n == 1) {
    v = P[0];
    return;
  }
  if (n == 2) {
    const vec3<T> e = P[1] - P[0];
    const T ee = dot(e, e);
    T t = ee > zero ? -dot(P[0], e) / ee : zero;
    t = t < zero ? zero : (t > one ? one : t);
    lam[0] = one - t;
    lam[1] = t;
    v = P[0] + e * t;
    return;
  }
  const vec3<T> a = P[0], b = P[1], c = P[2];
  const vec3<T> ab = b - a, ac = c - a;
  const T d1 = -dot(ab, a), d2 = -dot(ac, a);
  if (d1 <= zero && d2 <= zero) {
    v = a;
    return;
  }
  const T d3 = -dot(ab, b), d4 = -dot(ac, b);
  if (d3 >= zero && d4 <= d3) {
    lam[0] = zero;
    lam[1] = one;
    v = b;
    return;
  }
  const T vc = d1 * d4 - d3 * d2;
  if (vc <= zero && d1 >= zero && d3 <= zero) {
    const T t = d1 / (d1 - d3);
    lam[0] = one - t;
    lam[1] = t;
    v = a + ab * t;
    return;
  }
  const T d5 = -dot(ab, c), d6 = -dot(ac, c);
  if (d6 >= zero && d5 <= d6) {
    lam[0] = zero;
    lam[2] = one;
    v = c;
    return;
  }
  const T vb = d5 * d2 - d1 * d6;
  if (vb <= zero && d2 >= zero && d6 <= zero) {
    const T t = d2 / (d2 - d6);
    lam[0] = one - t;
    lam[2] = t;
    v = a + ac * t;
    return;
  }
  const T va = d3 * d6 - d5 * d4;
  if (va <= zero && (d4 - d3) >= zero && (d5 - d6) >= zero) {
    const T t = (d4 - d3) / ((d4 - d3) + (d5 - d6));
    lam[0] = zero;
    lam[1] = one - t;
    lam[2] = t;
    v = b + (c - b) * t;
    return;
  }
  const T den = one / (va + vb + vc);
  const T s1 = vb * den, s2 = vc * den;
  lam[0] = one - s1 - s2;
  lam[1] = s1;
  lam[2] = s2;
  v = a + ab * s1 + ac * s2;
}

// --------------------------------------------------------------------------------
// per-pair GJK

struct GjkState {
  int n;        // simplex size (4 = origin enclosed)
  fv3 P[4];     // simplex Minkowski points, newest last
  int ia[4], ib[4];
  fv3 v;        // closest point of the simplex to the origin
  float dist;
  float wmax2;  // max |P|^2 seen (scale of the problem)
  fv3 w0, w1;   // witnesses on body 1 and body 2
  int iters;
  int status;
  int exit;     // why the loop ended (GJK_EXIT_*)
  bool polish;  // separated: certify and re-solve (or continue) in FP64
  bool certain; // the final support is the exact (FP64) one along the exact direction
};

// loop exit reasons (reported in status bits 16..18)
enum {
  GJK_EXIT_GAP_REL = 1,   // |v|^2 - v.w <= eps_rel |v|^2
  GJK_EXIT_GAP_NOISE = 2, // gap below the FP32 rounding floor (or eps_tot)
  GJK_EXIT_NULL_V = 3,    // |v| < eps_rel
  GJK_EXIT_DUPLICATE = 4, // support pair already in the simplex
  GJK_EXIT_CONTACT = 5,   // |v| negligible against the simplex scale
  GJK_EXIT_ENCLOSED = 6,  // origin inside the tetrahedron
  GJK_EXIT_CAP = 7,       // iteration cap
};

// The pair is in contact (EPA runs) when GJK enclosed the origin or the distance is
// below FLT_EPSILON -- the reference's FP32 test (GJK/cpu/EPA.c:370).
OGX_HD bool gjk_contact(const GjkState& g) { return g.n == 4 || !(g.dist > FLT_EPSILON); }

// barycentric weights of the closest point v of the final simplex, FP32
OGX_HD void simplex_weights(const GjkState& g, float* lam) {
  lam[0] = 1.0f;
  lam[1] = lam[2] = lam[3] = 0.0f;
  if (g.n == 2) {
    const fv3 e = g.P[1] - g.P[0];
    const float ee = dot(e, e);
    float t = ee > 0.0f ? -dot(g.P[0], e) / ee : 0.0f;
    t = fminf(fmaxf(t, 0.0f), 1.0f);
    lam[0] = 1.0f - t;
    lam[1] = t;
  } else if (g.n == 3) {
    const fv3 e1 = g.P[1] - g.P[0], e2 = g.P[2] - g.P[0];
    const float g11 = dot(e1, e1), g12 = dot(e1, e2), g22 = dot(e2, e2);
    const float r1 = -dot(g.P[0], e1), r2 = -dot(g.P[0], e2);
    const float det = g11 * g22 - g12 * g12;
    if (det != 0.0f) {
      const float a1 = (g22 * r1 - g12 * r2) / det;
      const float a2 = (g11 * r2 - g12 * r1) / det;
      lam[0] = 1.0f - a1 - a2;
      lam[1] = a1;
      lam[2] = a2;
    }
  } else if (g.n == 4) {
    const fv3 e1 = g.P[1] - g.P[0], e2 = g.P[2] - g.P[0], e3 = g.P[3] - g.P[0];
    const fv3 c23 = cross(e2, e3), c31 = cross(e3, e1), c12 = cross(e1, e2);
    const float det = dot(e1, c23);
    if (det != 0.0f) {
      const fv3 o = -g.P[0];
      const float a1 = dot(o, c23) / det, a2 = dot(o, c31) / det, a3 = dot(o, c12) / det;
      lam[0] = 1.0f - a1 - a2 - a3;
      lam[1] = a1;
      lam[2] = a2;
      lam[3] = a3;
    }
  }
}

// FP64 re-run of one sub-distance step on the exact Minkowski points (cold path: taken
// when an FP32 decision of the step falls inside its rounding bound).  Returns the new
// slot order in `order` and the new direction.
template <class Mem>
#if defined(__CUDACC__)
__noinline__
#endif
OGX_HD int escalate_step(const Mem B, int n, const int* ia, const int* ib, fv3 vold, int* order, fv3* vout,
                         const uint32_t* subtab, uint32_t bits, uint32_t known) {
  Sx<double> sd;
  sd.n = n;
  for (int j = 0; j < n; ++j) {
    sd.v[j].p = B.dpoint(0, ia[j]) - B.dpoint(1, ib[j]);
    sd.v[j].k = j;
  }
  dv3 vd = cvt<double>(vold);
  subdistance(sd, vd, subtab, bits, known);
  for (int j = 0; j < sd.n; ++j) order[j] = sd.v[j].k;
  *vout = cvt<float>(vd);
  return sd.n;
}

// GJK as a loop of iterations: gjk_start sets the state up, each gjk_iterate runs one
// iteration (support, termination tests, sub-distance step) until r.done, gjk_end
// finishes (witnesses, certification).  gjk_pair chains them.  live = false: a team that only
// takes part in the operations of its warp's other teams.
struct GjkRun {
  fv3 v;
  float vv;  // dot(v, v)
  fv3 P[4];  // simplex in registers: slots 0..3, newest last; every index is unrolled
  int IA[4], IB[4];
  int n;
  float wmax2;
  fv3 sa, sb;
  int ia, ib;
  int k;
  int status, exit;
  bool done;
};

template <class Bodies>
OGX_HD void gjk_start(const Bodies& B, GjkRun& r, int start_a = 0, int start_b = 0) {
  // first point of the Minkowski difference: point 0 of each body (the reference's
  // start), or a warm-start pair of vertex indices (e.g. the previous frame's simplex)
  const fv3 a0 = B.point(0, start_a), b0 = B.point(1, start_b);
  r.v = a0 - b0;
  r.vv = dot(r.v, r.v);
  r.P[0] = r.v;
  r.P[1] = r.P[2] = r.P[3] = r.v;
  r.IA[0] = start_a;
  r.IB[0] = start_b;
  r.IA[1] = r.IA[2] = r.IA[3] = r.IB[1] = r.IB[2] = r.IB[3] = -1;
  r.n = 1;
  r.wmax2 = 0.0f;
  r.sa = a0;
  r.sb = b0;
  r.ia = start_a;
  r.ib = start_b;
  r.k = 0;
  r.status = 0;
  r.exit = 0;
  r.done = false;
}

// The gap below which FP32 rounding of |v| |w| hides any progress.
OGX_COLD float gap_floor(const Config cfg, float vv, float ww) {
  const float nv = sqrtf(vv);
  return fmaxf(cfg.gjk_eps_tot, cfg.gjk_noise * FLT_EPSILON * nv * (nv + sqrtf(ww)));
}

// One iteration is a chain of dependent steps (scan, team reduction, support points, gap,
// predicates, table, projection) that a pair cannot overlap with anything of its own, so
// what bounds it is the chain's length and, over a full GPU, its instruction count.  Hence:
// both bodies' reductions side by side and both candidate points loaded at once; the
// noise floor's square roots only where an upper bound says they can matter; one division
// for whichever projection the step takes; |w|^2 of the new point alone for the scale (the
// older points were counted when they joined); one branch for all the exit tests.
template <class Team, class Bodies>
OGX_HD void gjk_iterate(const Team& t, const Bodies& B, const Config& cfg, GjkRun& r,
                        const uint32_t* subtab = nullptr, bool live = true) {
  const bool reftol = (cfg.flags & OGX_F_REFERENCE_TOL) != 0;
  const bool escalate = (cfg.flags & OGX_F_FP64_ESCALATE) != 0;
  // |v| this small against the simplex points is below FP32 resolution: stop
  const float contact = reftol ? cfg.gjk_eps_tot : 0.5f * FLT_EPSILON;
  fv3& v = r.v;
  fv3* P = r.P;
  int* IA = r.IA;
  int* IB = r.IB;
  const fv3 mv = -v;
  float ba = -INFINITY, bb = -INFINITY;
  int xa = 0, xb = 0;
  if (live) {
    B.scan(t, 0, mv, ba, xa);
    B.scan(t, 1, v, bb, xb);
  }
  t.argmax_pair(ba, xa, bb, xb);
  if (!live) return;
  ++r.k;
  // the candidates (a scan that no value won has no index: the last support then)
  const fv3 pa = B.point(0, ba > -INFINITY ? xa : r.ia), pb = B.point(1, bb > -INFINITY ? xb : r.ib);
  if (ba > sdot(r.sa, mv)) {
    r.ia = xa;
    r.sa = pa;
  }
  if (bb > sdot(r.sb, v)) {
    r.ib = xb;
    r.sb = pb;
  }
  const int ia = r.ia, ib = r.ib;
  const fv3 w = r.sa - r.sb;
  const float vv = r.vv, ww = dot(w, w);
  const float gap = vv - dot(v, w);
  float floor_ = cfg.gjk_eps_tot;
  // gap_floor <= noise eps (vv + (vv + ww) / 2), up to rounding that the last factor covers
  // (where vv is far from the subnormals)
  const float bound = cfg.gjk_noise * FLT_EPSILON * (1.5f * vv + 0.5f * ww) * 1.0001f;
  if (!reftol && (gap < bound || vv < 1e-30f)) floor_ = gap_floor(cfg, vv, ww);
  bool dup = false;
#pragma unroll
  for (int j = 0; j < 4; ++j) dup |= (j < r.n) && IA[j] == ia && IB[j] == ib;
  const int stop = gap <= cfg.gjk_eps_rel * vv                ? GJK_EXIT_GAP_REL
                   : gap < floor_                             ? GJK_EXIT_GAP_NOISE
                   : vv < cfg.gjk_eps_rel * cfg.gjk_eps_rel   ? GJK_EXIT_NULL_V
                   : (dup && !reftol)                         ? GJK_EXIT_DUPLICATE
                                                              : 0;
  if (stop) {
    r.exit = stop;
    r.done = true;
    return;
  }
  const int n = r.n + 1;  // w joins in slot n - 1
#pragma unroll
  for (int j = 1; j < 3; ++j)
    if (j == n - 1) {
      P[j] = w;
      IA[j] = ia;
      IB[j] = ib;
    }

  StepIn S;
  uint32_t bits, unc;
  step_predicates(n, P, w, S, bits, unc);
  const SubOut o = step_decide(n, bits, subtab);
  // the line through w and slot a, or the plane through w and slots a, b
  const StepSpan span = step_span(S, o);
  // degenerate spans make the projection itself unreliable
  if (span.degenerate) unc |= o.used | 1u;
  int nn;
  int slot[3];
  if ((unc & o.used) != 0u && escalate) {
    int ias[4], ibs[4];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      ias[j] = IA[j];
      ibs[j] = IB[j];
    }
    if (n == 4) {
      ias[3] = ia;
      ibs[3] = ib;
    }
    int order[4] = {0, 1, 2, 3};
    fv3 vd;
    nn = escalate_step(B.mem_view(), n, ias, ibs, v, order, &vd, subtab, bits, step_known(n, S, unc));
    v = vd;
    r.status |= OGX_S_GJK_ESCALATED;
#pragma unroll
    for (int j = 0; j < 3; ++j) slot[j] = order[j];
  } else {
    v = step_direction(w, span, o, v);
    nn = o.n;
#pragma unroll
    for (int j = 0; j < 3; ++j) slot[j] = o.s[j];
  }
  // does w stay?  (an undecided step keeps the older three)
  const bool kept = nn == 4 || slot[0] == n - 1 || (nn > 1 && slot[1] == n - 1) || (nn > 2 && slot[2] == n - 1);
  if (kept) r.wmax2 = fmaxf(r.wmax2, ww);
  if (r.k == 1 && nn == 2) r.wmax2 = fmaxf(r.wmax2, dot(P[0], P[0]));  // the starting point stays
  if (nn < 4) {
    fv3 P2[3];
    int A2[3], B2[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      P2[j] = sel3(slot[j], P[0], P[1], P[2], w);
      A2[j] = seli(slot[j], IA[0], IA[1], IA[2], ia);
      B2[j] = seli(slot[j], IB[0], IB[1], IB[2], ib);
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      P[j] = P2[j];
      IA[j] = A2[j];
      IB[j] = B2[j];
    }
  } else {
    P[3] = w;
    IA[3] = ia;
    IB[3] = ib;
  }
  r.n = nn;
  r.vv = dot(v, v);
  r.exit = r.vv <= contact * contact * r.wmax2 ? GJK_EXIT_CONTACT
           : nn == 4                           ? GJK_EXIT_ENCLOSED
           : r.k == cfg.gjk_max_iter           ? GJK_EXIT_CAP
                                               : 0;
  r.done = r.exit != 0;
}

template <class Team, class Bodies>
OGX_HD void gjk_end(const Team& t, const Bodies& B, const Config& cfg, const GjkRun& r, GjkState& g) {
  const fv3 v = r.v;
  const fv3* P = r.P;
  const int* IA = r.IA;
  const int* IB = r.IB;
  const int n = r.n;
  const float wmax2 = r.wmax2;
  const int k = r.k;
  g.status = r.status;
  g.exit = r.exit;
  g.n = n;
  g.wmax2 = wmax2;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    g.P[j] = P[j];
    g.ia[j] = IA[j];
    g.ib[j] = IB[j];
  }
  if (k == cfg.gjk_max_iter && g.n != 4) g.status |= OGX_S_GJK_CAP;
  g.status |= g.exit << 16;
  g.iters = k;
  g.v = v;
  g.dist = sqrtf(dot(v, v));

  float lam[4];
  simplex_weights(g, lam);
  fv3 w0 = v3<float>(0.f, 0.f, 0.f), w1 = w0;
#pragma unroll
  for (int j = 0; j < 4; ++j)
    if (j < n) {
      w0 = w0 + B.point(0, IA[j]) * lam[j];
      w1 = w1 + B.point(1, IB[j]) * lam[j];
    }
  g.w0 = w0;
  g.w1 = w1;

  // FP32 error of |v| is a few ulp of the simplex scale; ask for an FP64 re-solve when
  // that is not small against the distance.
  g.polish = false;
  g.certain = false;
  if ((cfg.flags & OGX_F_FP64_POLISH) && g.n >= 1 && g.n <= 3 && !gjk_contact(g)) {
    // Every separated pair is certified or continued in FP64: a stop on the FP32 gap
    // bounds the distance (about 1e-7 relative) but not its direction, which on flat
    // closest features can stay ~1e-4 off until the exact feature is found; a pair that
    // ran into the iteration cap has not converged at all (the region decisions can cycle).
    g.polish = true;
  }
  if (g.polish) {
    // Is the exact support along the exact closest point v64 one of the final simplex's
    // own points?  Then GJK's stop is exact and the FP64 closest point of the simplex is
    // the answer.  Each body's points outside the simplex must trail its best point by
    // more than twice the error of an FP32 support value against the exact value along
    // v64: FP32 dot rounding (4 eps amax |v|_1) plus the FP32 projection error of v
    // (16 eps |W| per component).
    int exa[3], exb[3];
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      exa[j] = j < n ? IA[j] : -1;
      exb[j] = j < n ? IB[j] : -1;
    }
    float a1, ao, am, b1, bo, bm;
    B.scan_excl(t, 0, -v, exa, a1, ao, am);
    B.scan_excl(t, 1, v, exb, b1, bo, bm);
    a1 = t.fmax_(a1);
    ao = t.fmax_(ao);
    am = t.fmax_(am);
    b1 = t.fmax_(b1);
    bo = t.fmax_(bo);
    bm = t.fmax_(bm);
    const float dv = 16.0f * FLT_EPSILON * sqrtf(g.wmax2) * 3.0f;
    const float l1v = fabsf(v.x) + fabsf(v.y) + fabsf(v.z);
    const float ea = 4.0f * FLT_EPSILON * am * l1v + am * dv;
    const float eb = 4.0f * FLT_EPSILON * bm * l1v + bm * dv;
    g.certain = (a1 - ao > 2.0f * ea) && (b1 - bo > 2.0f * eb);
  }
}

template <class Team, class Bodies>
OGX_HD void gjk_pair(const Team& t, const Bodies& B, const Config& cfg, GjkState& g, int start_a = 0,
                     int start_b = 0, const uint32_t* subtab = nullptr) {
  GjkRun r;
  gjk_start(B, r, start_a, start_b);
  while (!r.done) gjk_iterate(t, B, cfg, r, subtab);
  gjk_end(t, B, cfg, r, g);
}

// Exact (FP64) support index of body w along d.  An FP32 scan finds the maximum m of
// fl(x . d32); every point whose exact value could exceed the true maximum satisfies
// fl(x . d32) >= m - 2e with e >= |fl(x . d32) - x . d| <= 2 FLT_EPSILON |x|_max |d|_1
// (rounding of d to FP32 plus the FP32 dot product).  Almost always the maximum is alone in
// that band (the scan keeps the runner-up) and is the support with no FP64 work -- an FP64
// instruction, a conversion or comparison too, costs 65 cycles on this part.  Otherwise the
// band's points are evaluated in FP64, ties to the lowest index: each lane's best, at once, as
// long as no lane holds two of them, else by a second pass over the body; the values are
// compared as integers.  Where a product or a sum of the scan may overflow, the scan says
// nothing and the second pass takes every point.  (Always the second pass, doubles compared in
// the reduction: 1,000 pairs of 1,000-point shells 75 us, now 65; 30k stress pairs 833 -> 771.)
// amax: the body's largest |coordinate|, or negative to have it found (and returned there).
// fd: d rounded to FP32; val (may be null): the exact value; err (may be null): e.
template <class Team, class Bodies, class T>
OGX_LEAF int exact_support_of(const Team t, const Bodies B, int w, vec3<T> d, fv3 fd, float* amax, T* val,
                              float* err) {
  const int n = B.n[w];
  float am = *amax;
  float best, second;
  int bi;
  if (am < 0.0f) {
    B.template scan_top<true>(t, w, fd, best, bi, second, am);
    *amax = am = t.fmax_(am);
  } else {
    float unused;
    B.template scan_top<false>(t, w, fd, best, bi, second, unused);
  }
  float m = best;
  int mi = bi;
  t.argmax(m, mi);
  // bodies given in double: the float points are the inputs rounded (half an ulp each),
  // one more FLT_EPSILON * amax * |d|_1 of difference to cover
  const float ef = Bodies::kExact64 ? 5.0f : 4.0f;
  const float l1d = fabsf(fd.x) + fabsf(fd.y) + fabsf(fd.z);
  const float e = ef * FLT_EPSILON * am * l1d + FLT_MIN;
  if (err) *err = e;
  const float lo = am * l1d < 1e38f ? m - 2.0f * e : -INFINITY;
  auto exact = [&](int i) -> T {
    if constexpr (Bodies::kExact64) {
      const dv3 p = B.dpoint(w, i);
      return p.x * d.x + p.y * d.y + p.z * d.z;
    } else {
      const fv3 p = B.point(w, i);
      return sc<T>(p.x) * d.x + sc<T>(p.y) * d.y + sc<T>(p.z) * d.z;
    }
  };
  int64_t k1 = order_key64(-INFINITY);
  int i1 = 0x7fffffff;
  if (m > -INFINITY && !t.any(second >= lo)) {
    // each lane's best is its only point in the band
    if (!t.any(best >= lo && bi != mi)) {
      if (val) *val = exact(mi);
      return mi;
    }
    if (best >= lo) {
      k1 = order_key64(exact(bi));
      i1 = bi;
    }
  } else {
#pragma unroll 1
    for (int i = t.lane(); i < n; i += Team::L) {
      if (sdot(B.point(w, i), fd) < lo) continue;
      const int64_t k = order_key64(exact(i));
      if (k > k1 || (k == k1 && i < i1)) {
        k1 = k;
        i1 = i;
      }
    }
  }
  t.argmax_key(k1, i1);
  if (val) *val = order_value64(k1);
  return i1 == 0x7fffffff ? 0 : i1;  // (every value NaN: d is)
}
// (on copies of the team and of the points-by-index view, so that the caller's body source
// keeps its registers)
template <class Team, class Bodies, class T>
OGX_HD int exact_support(const Team& t, const Bodies& B, int w, vec3<T> d, fv3 fd, float& amax, T* val = nullptr,
                         float* err = nullptr) {
  float am = amax;
  int i;
  if constexpr (Bodies::kExact64)
    i = exact_support_of(t, B, w, d, fd, &am, val, err);
  else
    i = exact_support_of(t, B.mem_view(), w, d, fd, &am, val, err);
  amax = am;
  return i;
}
template <class T>
OGX_HD fv3 floats(vec3<T> d) {
  return v3<float>(to_float(d.x), to_float(d.y), to_float(d.z));
}

// the Minkowski point a_i - b_j exactly (double), or as double-float components
template <class T>
struct Tag {};
template <class Bodies>
OGX_HD dv3 mpoint(Tag<double>, const Bodies& B, int i, int j) { return B.dpoint(0, i) - B.dpoint(1, j); }
template <class Bodies>
OGX_HD xv3 mpoint(Tag<df>, const Bodies& B, int i, int j) { return xdiff(B.point(0, i), B.point(1, j)); }

// FP64 continuation of GJK from the FP32 result: exact supports, FP64 sub-distance,
// stop when the FP64 gap |v|^2 - v.w <= 1e-12 |v|^2 or the support repeats.  Certifies
// (or corrects) the FP32 answer; sets g.n = 4 if the origin turns out to be enclosed.
// Split in three so that a warp can run the supports of 32 pairs cooperatively while
// each lane keeps its own pair's state (refine_begin, then refine_step with the exact
// supports along -v / v until done, then refine_end).
// written for double and double-float; the continuation runs in FP64: its progress
// and gap tests need |v|^2 to about 1e-12 relative, and near-coplanar thin bodies put the
// origin 1e-5 of the coordinates' scale from the simplex, where the 48 bits of
// double-float leave |v|^2 with ~1e-10 relative noise (it stopped a step early on some
// 1e-4-thick disks).  The one-shot re-solves (refine_certain, epa_polish) have no such
// decision and run in double-float.
template <class T>
struct RefineStateT {
  Sx<T> s;
  int ia[4], ib[4];
  vec3<T> v;
  T lam[4];   // barycentric weights of v on s (valid while no step changed s)
  bool lam_valid;
  T vv;       // dot(v, v)
  T wmax2;
  int it, max_iter;
  bool done, enclosed;
};
typedef RefineStateT<double> RefineState;

template <class Bodies, class T>
OGX_HD void refine_begin(const Bodies& B, const GjkState& g, int max_iter, RefineStateT<T>& r) {
  Sx<T>& s = r.s;
  const T zero = sc<T>(0.0f);
  s.n = g.n > 3 ? 3 : g.n;
  for (int j = 0; j < s.n; ++j) {
    r.ia[j] = g.ia[j];
    r.ib[j] = g.ib[j];
    s.v[j].p = mpoint(Tag<T>(), B, r.ia[j], r.ib[j]);
    s.v[j].k = j;
  }
  // exact closest point of the FP32 result's simplex; keep only the vertices it uses
  vec3<T> P[3];
  for (int j = 0; j < s.n; ++j) P[j] = s.v[j].p;
  T lam[4];
  closest_on_simplex_t<T>(s.n, P, lam, r.v);
  {
    Sx<T> q;
    q.n = 0;
    int qa[4], qb[4];
    for (int j = 0; j < s.n; ++j)
      if (lam[j] > zero || (s.n == 1)) {
        q.v[q.n] = s.v[j];
        qa[q.n] = r.ia[j];
        qb[q.n] = r.ib[j];
        q.n++;
      }
    T ql[4] = {sc<T>(1.0f), zero, zero, zero};
    int m = 0;
    for (int j = 0; j < s.n; ++j)
      if (lam[j] > zero || (s.n == 1)) ql[m++] = lam[j];
    r.lam_valid = q.n > 0;
    if (q.n == 0) {
      q.v[0] = s.v[0];
      qa[0] = r.ia[0];
      qb[0] = r.ib[0];
      q.n = 1;
    }
    s = q;
    for (int j = 0; j < s.n; ++j) {
      r.ia[j] = qa[j];
      r.ib[j] = qb[j];
      s.v[j].k = j;
      r.lam[j] = ql[j];
    }
  }
  r.wmax2 = zero;
  for (int j = 0; j < s.n; ++j) r.wmax2 = tmax(r.wmax2, dot(s.v[j].p, s.v[j].p));
  r.vv = dot(r.v, r.v);
  r.max_iter = max_iter;
  r.enclosed = false;
  r.it = g.certain ? max_iter + 1 : 0;  // the FP32 pass proved the simplex final
  r.done = r.it >= max_iter;
}

// Closest point of a simplex to the origin by exhaustive search (Johnson's method without
// the region tests): every sub-simplex that holds the newest vertex s.v[s.n-1] is solved
// on its affine hull (Gram system), those whose barycentric weights are all >= 0 are
// feasible, and the feasible one nearest the origin wins (fewer vertices on ties).  In
// exact arithmetic the closest point after a GJK step lies on such a sub-simplex.  Cold
// path: taken when the signed-volume region decisions made no progress -- on some
// configurations the hff tests of the reference's sub-distance (GJK/cpu/openGJK.c:315-613)
// pick a region whose point is farther than the last one, and GJK then cycles until its
// iteration cap (the reference's own FP64 code does so on a pair of the 1M-pair power-law
// batch and returns a distance 1.3% too large).  Returns the reduced simplex in s (slots
// keep their .k) and its closest point in v; s.n == 4 means the origin is enclosed.
template <class T>
OGX_COLD void closest_exhaustive(Sx<T>& s, vec3<T>& v) {
  const int n = s.n;
  const int nw = n - 1;
  const T zero = T(0);
  T best = T(INFINITY);
  int best_mask = 1 << nw, best_k = 5;
  vec3<T> best_v = s.v[nw].p;
#pragma unroll 1
  for (int mask = 1; mask < (1 << n); ++mask) {
    if (!(mask & (1 << nw))) continue;
    int idx[4], k = 0;
    idx[k++] = nw;  // the newest vertex first
    for (int j = 0; j < n; ++j)
      if (j != nw && (mask & (1 << j))) idx[k++] = j;
    const vec3<T> p0 = s.v[idx[0]].p;
    T lam[4] = {T(1), zero, zero, zero};
    bool ok = true;
    if (k >= 2) {
      vec3<T> e[3];
      for (int a = 1; a < k; ++a) e[a - 1] = s.v[idx[a]].p - p0;
      const int m = k - 1;
      T G[3][3], r[3];
      for (int a = 0; a < m; ++a) {
        r[a] = -dot(p0, e[a]);
        for (int c = 0; c < m; ++c) G[a][c] = dot(e[a], e[c]);
      }
      T x[3] = {zero, zero, zero};
      if (m == 1) {
        ok = G[0][0] > zero;
        if (ok) x[0] = r[0] / G[0][0];
      } else if (m == 2) {
        const T det = G[0][0] * G[1][1] - G[0][1] * G[1][0];
        ok = det > zero;
        if (ok) {
          x[0] = (r[0] * G[1][1] - G[0][1] * r[1]) / det;
          x[1] = (G[0][0] * r[1] - r[0] * G[1][0]) / det;
        }
      } else {
        // x = adj(G) r / det(G), adj(G)[i][j] = C[j][i] with C the cofactor matrix
        T C[3][3];
        C[0][0] = G[1][1] * G[2][2] - G[1][2] * G[2][1];
        C[0][1] = G[1][2] * G[2][0] - G[1][0] * G[2][2];
        C[0][2] = G[1][0] * G[2][1] - G[1][1] * G[2][0];
        C[1][0] = G[0][2] * G[2][1] - G[0][1] * G[2][2];
        C[1][1] = G[0][0] * G[2][2] - G[0][2] * G[2][0];
        C[1][2] = G[0][1] * G[2][0] - G[0][0] * G[2][1];
        C[2][0] = G[0][1] * G[1][2] - G[0][2] * G[1][1];
        C[2][1] = G[0][2] * G[1][0] - G[0][0] * G[1][2];
        C[2][2] = G[0][0] * G[1][1] - G[0][1] * G[1][0];
        const T det = G[0][0] * C[0][0] + G[0][1] * C[0][1] + G[0][2] * C[0][2];
        ok = det > zero;
        if (ok)
          for (int a = 0; a < 3; ++a) x[a] = (C[0][a] * r[0] + C[1][a] * r[1] + C[2][a] * r[2]) / det;
      }
      T sum = zero;
      for (int a = 0; a < m; ++a) {
        lam[a + 1] = x[a];
        sum = sum + x[a];
      }
      lam[0] = T(1) - sum;
    }
    if (!ok) continue;
    bool feasible = true;
    for (int a = 0; a < k; ++a) feasible = feasible && !(lam[a] < zero);
    if (!feasible) continue;
    vec3<T> p = p0 * lam[0];
    for (int a = 1; a < k; ++a) p = p + s.v[idx[a]].p * lam[a];
    const T d2 = k == 4 ? zero : dot(p, p);  // a feasible tetrahedron holds the origin
    if (d2 < best || (d2 == best && k < best_k)) {
      best = d2;
      best_mask = mask;
      best_k = k;
      best_v = k == 4 ? vec3<T>{zero, zero, zero} : p;
    }
  }
  Sx<T> q;
  q.n = 0;
  for (int j = 0; j < n; ++j)
    if (best_mask & (1 << j)) q.v[q.n++] = s.v[j];
  s = q;
  v = best_v;
}

// One iteration with the exact supports xa (body 1 along -v) and xb (body 2 along v).  FP64 is
// spent on the point, the gap, the projection and the predicates FP32 cannot decide; what
// only guards against rounding is bounded in FP32 first.
template <class Bodies, class T>
OGX_HD void refine_step(const Bodies& B, RefineStateT<T>& r, int xa, int xb, const uint32_t* subtab) {
  Sx<T>& s = r.s;
  const vec3<T> w = mpoint(Tag<T>(), B, xa, xb);
  // The points rounded to FP32.  Of float inputs that is their FP32 difference (the difference
  // rounded to 53 bits first rounds to the same 24), without conversions: each costs as much
  // as an FP64 instruction.
  auto point32 = [&](const vec3<T>& p, int i, int j) {
    return Bodies::kExact64 ? floats(p) : B.point(0, i) - B.point(1, j);
  };
  const fv3 wf = point32(w, xa, xb);
  fv3 Pf[3];
  const T vv = r.vv;
  // FP64 gap test.  In exact arithmetic v.p_j = |v|^2 for every vertex p_j of the
  // current feature, so the gap |v|^2 - v.w equals v.(p_j - w); that form rounds in
  // proportion to |p_j - w| (small near convergence) instead of |w|^2.  Relative
  // tolerance of the FP64 oracle (eps * 1e4) and a rounding floor.
  T gap = sc<T>(INFINITY);
  float dmaxf = 0.0f;
#pragma unroll
  for (int j = 0; j < 3; ++j) {
    if (j < s.n) {
      gap = tmin(gap, dot(r.v, s.v[j].p - w));
      Pf[j] = point32(s.v[j].p, r.ia[j], r.ib[j]);
      const fv3 e = Pf[j] - wf;
      dmaxf = fmaxf(dmaxf, dot(e, e));
    } else {
      Pf[j] = wf;
    }
  }
  if (gap <= T(1e-12) * vv) {
    r.done = true;
    return;
  }
  // The rounding floor 4 eps max|p| max|p - w|, bounded in FP32 (the rounded points' difference
  // is within 2^-22 max(|p|, |w|) of the exact one).
  const float wm = fmaxf(to_float(r.wmax2), dot(wf, wf));
  const float bound = (float)(4.2 * prec_eps<T>()) * sqrtf(wm) * (sqrtf(dmaxf) + 5e-7f * sqrtf(wm)) + FLT_MIN;
  if (!(to_float(gap) > bound)) {
    T dmax = sc<T>(0.0f);
    for (int j = 0; j < s.n; ++j) {
      const vec3<T> e = s.v[j].p - w;
      dmax = tmax(dmax, dot(e, e));
    }
    if (gap <= T(4.0 * prec_eps<T>()) * tsqrt(r.wmax2) * tsqrt(dmax)) {
      r.done = true;
      return;
    }
  }
  bool dup = false;
  for (int j = 0; j < s.n; ++j) dup |= (r.ia[j] == xa && r.ib[j] == xb);
  if (dup) {
    r.done = true;
    return;
  }
  const Sx<T> prev = s;
  int pa[4], pb[4];
  for (int j = 0; j < s.n; ++j) {
    pa[j] = r.ia[j];
    pb[j] = r.ib[j];
  }
  const vec3<T> vprev = r.v;
  const int nw = s.n;  // the new point's slot
  s.v[nw].p = w;
  s.v[nw].k = nw;
  r.ia[nw] = xa;
  r.ib[nw] = xb;
  s.n++;
  // predicates whose FP32 value on the rounded points has the exact sign are decided there
  StepIn S;
  uint32_t bits, unc;
  step_predicates(s.n, Pf, wf, S, bits, unc);
  subdistance(s, r.v, subtab, bits, step_known(s.n, S, unc));
  T vnew = dot(r.v, r.v);
  r.lam_valid = false;
  if (s.n != 4 && !(vnew < vv * T(1.0 - 1e-12))) {
    // the region decisions made no progress although the gap says progress is possible:
    // solve the step again by exhaustive search on the grown simplex
    Sx<T> t = prev;
    t.v[t.n].p = w;
    t.v[t.n].k = t.n;
    t.n++;
    vec3<T> vt;
    closest_exhaustive(t, vt);
    if (t.n == 4 || dot(vt, vt) < vv * T(1.0 - 1e-12)) {
      s = t;
      r.v = vt;
      vnew = dot(vt, vt);
    }
  }
  if (s.n != 4 && !(vnew < vv * T(1.0 - 1e-12))) {
    // still none: a tie support spanning a degenerate simplex -- keep the last answer
    s = prev;
    r.v = vprev;
    for (int j = 0; j < s.n; ++j) {
      r.ia[j] = pa[j];
      r.ib[j] = pb[j];
    }
    r.done = true;
    return;
  }
  r.vv = vnew;
  // (the older vertices are in wmax2 already)
  bool kept = false;
  int na[4], nb[4];
  for (int j = 0; j < s.n; ++j) {
    kept = kept || s.v[j].k == nw;
    na[j] = r.ia[s.v[j].k];
    nb[j] = r.ib[s.v[j].k];
  }
  for (int j = 0; j < s.n; ++j) {
    r.ia[j] = na[j];
    r.ib[j] = nb[j];
    s.v[j].k = j;
  }
  if (kept && dot(wf, wf) * 1.00001f >= to_float(r.wmax2)) r.wmax2 = tmax(r.wmax2, dot(w, w));
  if (s.n == 4) {
    r.enclosed = true;
    r.done = true;
    return;
  }
  ++r.it;
  if (r.it >= r.max_iter) r.done = true;
}

template <class Bodies, class T>
OGX_HD void refine_end(const Bodies& B, const RefineStateT<T>& r, GjkState& g) {
  const Sx<T>& s = r.s;
  g.n = s.n;
  for (int j = 0; j < s.n; ++j) {
    g.ia[j] = r.ia[j];
    g.ib[j] = r.ib[j];
    g.P[j] = v3<float>(to_float(s.v[j].p.x), to_float(s.v[j].p.y), to_float(s.v[j].p.z));
  }
  g.status |= (r.it == r.max_iter + 1) ? OGX_S_POLISHED : (OGX_S_POLISHED | OGX_S_GJK_ESCALATED);
  if (r.it == r.max_iter) g.status |= OGX_S_GJK_CAP;
  if (r.enclosed) {
    g.v = v3<float>(0.f, 0.f, 0.f);
    g.dist = 0.0f;
    return;
  }
  T lam[4];
  vec3<T> v;
  if (r.lam_valid) {
    // the simplex is the one refine_begin solved: reuse its closest point
    v = r.v;
    for (int j = 0; j < 4; ++j) lam[j] = r.lam[j];
  } else {
    vec3<T> P[3];
    for (int j = 0; j < s.n; ++j) P[j] = s.v[j].p;
    closest_on_simplex_t<T>(s.n, P, lam, v);
  }
  // The distance needs the FP64 closest point; its square root and the witnesses do
  // not: FP32 from here on (|v|^2 rounded once, then a correctly rounded sqrtf: 1 ulp;
  // witnesses to a few ulp of the coordinates, the 1e-4 witness tolerance being far
  // above).  FP64 issues at 1/64 of the FP32 rate here.
  fv3 w0 = v3<float>(0.f, 0.f, 0.f), w1 = w0;
  for (int j = 0; j < s.n; ++j) {
    const float l = to_float(lam[j]);
    w0 = w0 + B.point(0, r.ia[j]) * l;
    w1 = w1 + B.point(1, r.ib[j]) * l;
  }
  g.v = v3<float>(to_float(v.x), to_float(v.y), to_float(v.z));
  g.dist = sqrtf(to_float(dot(v, v)));
  g.w0 = w0;
  g.w1 = w1;
}

// The re-solve of a pair whose final simplex the FP32 pass proved final (its support is
// certified), in double-float arithmetic on the FP32 pipes instead of FP64: the exact
// Minkowski points a - b, the closest point of their simplex to about 48 bits, the
// vertices it uses; then, as refine_end, FP32 witnesses and a correctly rounded distance.
template <class Bodies>
OGX_HD void refine_certain(const Bodies& B, GjkState& g) {
  const int n0 = g.n > 3 ? 3 : g.n;
  xv3 P[3];
  int ia[3], ib[3];
  for (int j = 0; j < n0; ++j) {
    ia[j] = g.ia[j];
    ib[j] = g.ib[j];
    P[j] = xdiff(B.point(0, ia[j]), B.point(1, ib[j]));
  }
  df lam[4];
  xv3 v;
  closest_on_simplex_t<df>(n0, P, lam, v);
  // keep the vertices the closest point uses (the single vertex of a point simplex)
  int m = 0;
  float ql[3] = {1.0f, 0.0f, 0.0f};
  int qa[3] = {ia[0], 0, 0}, qb[3] = {ib[0], 0, 0};
  xv3 Q[3];
  Q[0] = P[0];
  for (int j = 0; j < n0; ++j)
    if (lam[j] > sc<df>(0.0f) || n0 == 1) {
      Q[m] = P[j];
      qa[m] = ia[j];
      qb[m] = ib[j];
      ql[m] = to_float(lam[j]);
      ++m;
    }
  if (m == 0) {  // as the FP64 path: the first vertex alone
    m = 1;
    ql[0] = 1.0f;
    v = P[0];
  }
  g.n = m;
  for (int j = 0; j < m; ++j) {
    g.ia[j] = qa[j];
    g.ib[j] = qb[j];
    g.P[j] = v3<float>(Q[j].x.hi, Q[j].y.hi, Q[j].z.hi);
  }
  g.status |= OGX_S_POLISHED;
  fv3 w0 = v3<float>(0.f, 0.f, 0.f), w1 = w0;
  for (int j = 0; j < m; ++j) {
    w0 = w0 + B.point(0, qa[j]) * ql[j];
    w1 = w1 + B.point(1, qb[j]) * ql[j];
  }
  g.v = v3<float>(to_float(v.x), to_float(v.y), to_float(v.z));
  g.dist = sqrtf(to_float(dot(v, v)));
  g.w0 = w0;
  g.w1 = w1;
}

template <class Team, class Bodies>
OGX_HD void gjk_refine(const Team& t, const Bodies& B, GjkState& g, int max_iter,
                       const uint32_t* subtab = nullptr) {
  if (g.certain) {
    refine_certain(B, g);
    return;
  }
  RefineState r;
  refine_begin(B, g, max_iter, r);
  float ma = -1.0f, mb = -1.0f;
  while (!r.done) {
    const fv3 fv = floats(r.v);
    const int xa = exact_support(t, B, 0, -r.v, -fv, ma);
    const int xb = exact_support(t, B, 1, r.v, fv, mb);
    refine_step(B, r, xa, xb, subtab);
  }
  refine_end(B, r, g);
}

}  // namespace ogx
