// ogx_twin.cpp -- TEST BUILD ONLY.  Runs the engine's per-pair GJK/EPA code (the same
// __host__ __device__ source the CUDA kernels instantiate) on the CPU with a one-lane
// team, so the algorithm can be checked against the oracle on a machine without a GPU
// and GPU results can be compared with the identical arithmetic on the host.  The
// product library never contains this file.
#include <pthread.h>
#include <string.h>

#include <vector>

#include "ogx_bodies.cuh"
#include "ogx_epa.cuh"
#include "ogx_gjk.cuh"

using namespace ogx;

namespace {

struct Job {
  int lo, hi, mode;
  const float* pool;
  const uint32_t* quad;
  const int32_t* counts;
  const int32_t* pairs;
  const ogx_config* cfg;
  float* dist;
  gkSimplex* smp;
  float* nrm;
  int32_t* status;
  int32_t* iters;
  const float* xf;  // poses (12 floats per body) for the posed pipeline, or null
};

struct Work {
  EpaMemSmall small;
  EpaMemCert full;
  EpaResume saved;
};

void bind(MemBodies& B, const Job& J, int b1, int b2, BodyRef A, BodyRef Bb) { B.bind(J.pool, A, Bb); }
void bind(Posed<MemBodies>& B, const Job& J, int b1, int b2, BodyRef A, BodyRef Bb) {
  B.bind_posed(J.pool, A, Bb, J.xf + 12 * (size_t)b1, J.xf + 12 * (size_t)b2);
}

template <class Bodies>
void one(const Job& J, int i, Work& M) {
  const int b1 = J.pairs[2 * i], b2 = J.pairs[2 * i + 1];
  BodyRef A{J.quad[b1], J.counts[b1]}, Bb{J.quad[b2], J.counts[b2]};
  Bodies B;
  bind(B, J, b1, b2, A, Bb);
  SerialTeam t;
  GjkState g;
  gjk_pair(t, B, *J.cfg, g);
  // same order as the device pipeline: the contact decision is taken on the FP32 GJK
  // result, separated pairs are then re-solved in FP64, contacts go through EPA
  bool contact = gjk_contact(g);
  bool late = false;  // a contact only the FP64 refinement found
  if (g.polish) {
    gjk_refine(t, B, g, 16);
    contact = gjk_contact(g);
    late = contact;
  }
  gkSimplex& s = J.smp[i];
  s.nvrtx = g.n;
  for (int k = 0; k < 4; ++k) {
    const bool live = k < g.n;
    s.vrtx[k][0] = live ? g.P[k].x : 0.f;
    s.vrtx[k][1] = live ? g.P[k].y : 0.f;
    s.vrtx[k][2] = live ? g.P[k].z : 0.f;
    s.vrtx_idx[k][0] = live ? g.ia[k] : 0;
    s.vrtx_idx[k][1] = live ? g.ib[k] : 0;
  }
  float d = g.dist;
  fv3 w0 = g.w0, w1 = g.w1, n = v3<float>(0.f, 0.f, 0.f);
  int st = g.status, ei = 0;
  if (J.mode >= 2) {
    if (contact) {
      // as on the device: the small working set first, full capacity when it runs out;
      // contacts found by the refinement go straight to the certified full pass.  Mode 3: a
      // contact that outgrew the small capacity is saved and continued, as the bucket kernels do
      EpaOut o;
      int nsaved = 0;
      EpaResumeSink sink{J.mode == 3 ? &M.saved : nullptr, &nsaved, 1};
      if (late) {
        o.spill = true;
        o.spill64 = true;
      } else {
        epa_pair(t, B, *J.cfg, g, M.small, o, true, sink);
      }
      if (o.spill) {
        ogx_config c = *J.cfg;
        if (o.spill64) c.flags |= OGX_F_EPA_FP64_PLANES;
        const EpaResume* rs = !late && o.resume == 0 ? &M.saved : nullptr;
        memset(&M.full, 0xff, sizeof M.full);  // (a pass that reads what it did not write shows)
        epa_pair<true>(t, B, c, g, M.full, o, false, EpaResumeSink{nullptr, nullptr, 0}, rs);
      }
      if (o.polish) epa_polish(B, o);
      d = o.dist;
      w0 = o.w0;
      w1 = o.w1;
      n = o.nrm;
      st |= o.status;
      ei = o.iters;
    } else {
      n = sep_normal(g);
    }
  }
  J.dist[i] = d;
  s.witnesses[0][0] = w0.x;
  s.witnesses[0][1] = w0.y;
  s.witnesses[0][2] = w0.z;
  s.witnesses[1][0] = w1.x;
  s.witnesses[1][1] = w1.y;
  s.witnesses[1][2] = w1.z;
  if (J.nrm) {
    J.nrm[3 * i] = n.x;
    J.nrm[3 * i + 1] = n.y;
    J.nrm[3 * i + 2] = n.z;
  }
  if (J.status) J.status[i] = st;
  if (J.iters) {
    J.iters[2 * i] = g.iters;
    J.iters[2 * i + 1] = ei;
  }
}

void* worker(void* arg) {
  const Job& J = *static_cast<const Job*>(arg);
  Work* M = new Work;
  for (int i = J.lo; i < J.hi; ++i) {
    if (J.xf)
      one<Posed<MemBodies>>(J, i, *M);
    else
      one<MemBodies>(J, i, *M);
  }
  delete M;
  return nullptr;
}

}  // namespace

extern "C" {

int twin_config(int reference, ogx_config* out) {
  *out = reference ? reference_config() : default_config();
  return 0;
}

// posed points of every body (the fused-transform pipeline's world points): out and
// local are xyz of all bodies concatenated, xf 12 floats per body
int twin_pose_points(int nbodies, const int32_t* counts, const float* local, const float* xf, float* out) {
  size_t k = 0;
  for (int b = 0; b < nbodies; ++b)
    for (int i = 0; i < counts[b]; ++i, ++k) {
      const fv3 p = pose_point(xf + 12 * (size_t)b, v3<float>(local[3 * k], local[3 * k + 1], local[3 * k + 2]));
      out[3 * k] = p.x;
      out[3 * k + 1] = p.y;
      out[3 * k + 2] = p.z;
    }
  return 0;
}

// order_key64 element by element, and the keys' values back
int twin_order_key64(int64_t n, const double* x, int64_t* key, double* back) {
  for (int64_t i = 0; i < n; ++i) {
    key[i] = order_key64(x[i]);
    back[i] = order_value64(key[i]);
  }
  return 0;
}

// Predicates of n-point steps (count of them; p: 4 points each as 2 x 3 floats a, b, the point
// being a - b, newest at n - 1): the FP32 bits on the rounded points, those that an exact
// evaluation takes over, and the bits evaluated in FP64
int twin_step_bits(int count, int n, const float* p, uint32_t* bits, uint32_t* known, uint32_t* exact) {
  for (int i = 0; i < count; ++i) {
    fv3 P[3], q = v3<float>(0.f, 0.f, 0.f);
    Vx<double> s[4];
    for (int j = 0; j < n; ++j) {
      const float *a = p + 24 * (size_t)i + 6 * j, *b = a + 3;
      const fv3 w = v3<float>(a[0], a[1], a[2]) - v3<float>(b[0], b[1], b[2]);
      if (j == n - 1)
        q = w;
      else
        P[j] = w;
      s[j].p = v3<double>((double)a[0] - b[0], (double)a[1] - b[1], (double)a[2] - b[2]);
    }
    for (int j = n - 1; j < 3; ++j) P[j] = q;
    StepIn S;
    uint32_t unc;
    step_predicates(n, P, q, S, bits[i], unc);
    known[i] = step_known(n, S, unc);
    exact[i] = 0u;
    for (int k = 0; k < 13; ++k) {
      const bool needs4 = k >= 3 && k < 7;
      const int slot = k < 3 ? k : (k < (int)PB_D + 2 ? 1 : 2);
      if (needs4 ? n == 4 : slot < n - 1) exact[i] |= exact_bit(s, n, 1u << k) ? 1u << k : 0u;
    }
  }
  return 0;
}

// The sub-distance step on exact 3-point simplices (newest last): the points that stay, and the
// closest point to the origin
int twin_triangle_step(int count, const double* p, int32_t* left, double* dir) {
  for (int i = 0; i < count; ++i) {
    Sx<double> s;
    s.n = 3;
    for (int j = 0; j < 3; ++j) {
      const double* q = p + 9 * (size_t)i + 3 * j;
      s.v[j].p = v3<double>(q[0], q[1], q[2]);
      s.v[j].k = j;
    }
    dv3 v = v3<double>(0.0, 0.0, 0.0);
    subdistance(s, v, nullptr, 0u, 0u);
    left[i] = s.n;
    dir[3 * i] = v.x;
    dir[3 * i + 1] = v.y;
    dir[3 * i + 2] = v.z;
  }
  return 0;
}

// exact support index and value of one body (SoA pool at quad 0, n points) along count directions
int twin_exact_support(const float* pool, int n, int count, const double* d, int32_t* index, double* value) {
  MemBodies B;
  B.bind(pool, BodyRef{0u, n}, BodyRef{0u, n});
  SerialTeam t;
  float amax = -1.0f;
  for (int i = 0; i < count; ++i) {
    const dv3 v = v3<double>(d[3 * i], d[3 * i + 1], d[3 * i + 2]);
    index[i] = exact_support(t, B, 0, v, floats(v), amax, value + i);
  }
  return 0;
}

// world points of the transform kernel (world_point); settled[i]: all of point i's coordinates
// came from the FP32 instructions
int twin_world_points(int n, const float* xf, const float* local, float* out, uint8_t* settled) {
  for (int i = 0; i < n; ++i) {
    const float* m = xf + 12 * (size_t)i;
    const fv3 p = v3<float>(local[3 * i], local[3 * i + 1], local[3 * i + 2]);
    const fv3 w = world_point(m, p);
    out[3 * i] = w.x;
    out[3 * i + 1] = w.y;
    out[3 * i + 2] = w.z;
    bool s[3];
    for (int k = 0; k < 3; ++k) world_coord(m[3 * k], m[3 * k + 1], m[3 * k + 2], m[9 + k], p, s[k]);
    settled[i] = s[0] && s[1] && s[2];
  }
  return 0;
}

// xf: null, or poses (12 floats per body) to run the posed pipeline on the pool's bodies
int twin_run_posed(int npairs, const float* pool, const uint32_t* quad, const int32_t* counts,
                   const int32_t* pairs, int mode, const ogx_config* cfg, float* dist, gkSimplex* smp,
                   float* nrm, int32_t* status, int32_t* iters, int nthreads, const float* xf) {
  if (npairs < 0 || mode < 1 || mode > 3) return -1;
  Job base{0, npairs, mode, pool, quad, counts, pairs, cfg, dist, smp, nrm, status, iters, xf};
  if (nthreads <= 1 || npairs < 64) {
    worker(&base);
    return 0;
  }
  if (nthreads > 64) nthreads = 64;
  std::vector<pthread_t> th(nthreads);
  std::vector<Job> jobs(nthreads, base);
  for (int k = 0; k < nthreads; ++k) {
    jobs[k].lo = (int)((int64_t)npairs * k / nthreads);
    jobs[k].hi = (int)((int64_t)npairs * (k + 1) / nthreads);
    pthread_create(&th[k], nullptr, worker, &jobs[k]);
  }
  for (int k = 0; k < nthreads; ++k) pthread_join(th[k], nullptr);
  return 0;
}

int twin_run(int npairs, const float* pool, const uint32_t* quad, const int32_t* counts,
             const int32_t* pairs, int mode, const ogx_config* cfg, float* dist, gkSimplex* smp,
             float* nrm, int32_t* status, int32_t* iters, int nthreads) {
  return twin_run_posed(npairs, pool, quad, counts, pairs, mode, cfg, dist, smp, nrm, status, iters, nthreads,
                        nullptr);
}
}
