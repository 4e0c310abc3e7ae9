// ogx_k_warp.cu -- the whole pipeline of a pair in one warp, for batches too small to fill
// the GPU with the bucket kernels' teams.
//
// A small batch is bound by latency: the slowest pair of each stage, the launches and the
// stream joins between ~20 kernels.  Here a block of one warp runs one pair from its
// check to its stored result -- GJK, the FP64 continuation or re-solve of a separated
// pair, EPA with its certified re-run, the face polish -- with the state kept in
// registers between the stages, so a call is a counter reset and one launch.  All 32
// lanes scan the bodies (each lane keeps its first block of 4 points of both bodies in
// registers) and split the EPA faces; the reductions are the warp's integer ones
// (order_key).  The stages are the bucket kernels' own functions and the results do not
// depend on the team width, so they are the pipeline's bit for bit.
#include "ogx_kernels.cuh"

namespace ogx {

// Bodies of a full-warp team: block `lane` of each body (the first 128 points) in
// registers, later blocks re-read from memory, four in flight.
struct WarpBodies {
  static constexpr bool kExact64 = false;
  float4 x[2], y[2], z[2];
  MemBodies mem;

  __device__ void bind(const float* pool, BodyRef a, BodyRef b, int lane) {
    mem.bind(pool, a, b);
#pragma unroll
    for (int w = 0; w < 2; ++w) {
      const int nb = mem.n4[w] >> 2;
      const float4* X = reinterpret_cast<const float4*>(mem.base[w]);
      const int q = lane < nb ? lane : 0;  // beyond the body: repeat block 0 (never wins)
      x[w] = __ldg(X + q);
      y[w] = __ldg(X + nb + q);
      z[w] = __ldg(X + 2 * nb + q);
    }
  }
  __device__ fv3 point(int w, int i) const { return mem.point(w, i); }
  __device__ dv3 dpoint(int w, int i) const { return mem.dpoint(w, i); }
  __device__ const MemBodies& mem_view() const { return mem; }
  template <class Team>
  __device__ void scan_excl(const Team& t, int w, fv3 d, const int* ex, float& b1, float& bo,
                            float& amax) const {
    mem.scan_excl(t, w, d, ex, b1, bo, amax);
  }
  template <class Team>
  __device__ void scan(const Team& t, int w, fv3 d, float& best, int& bi) const {
    best = -INFINITY;
    bi = 0x7fffffff;
    float v[4];
    sdot4(x[w], y[w], z[w], d, v);
    block_best(v, 4 * t.lane(), best, bi);
    const int nb = mem.n4[w] >> 2;
    if (nb <= 32) return;
    const float4* X4 = reinterpret_cast<const float4*>(mem.base[w]);
    int q = t.lane() + 32;
    for (; q + 96 < nb; q += 128) {
      float4 bx[4], by[4], bz[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        bx[u] = __ldg(X4 + q + 32 * u);
        by[u] = __ldg(X4 + nb + q + 32 * u);
        bz[u] = __ldg(X4 + 2 * nb + q + 32 * u);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        sdot4(bx[u], by[u], bz[u], d, v);
        block_best(v, 4 * (q + 32 * u), best, bi);
      }
    }
    for (; q < nb; q += 32) {
      const float4 bx = __ldg(X4 + q), by = __ldg(X4 + nb + q), bz = __ldg(X4 + 2 * nb + q);
      sdot4(bx, by, bz, d, v);
      block_best(v, 4 * q, best, bi);
    }
  }
};

// The rare and FP64-heavy stages, out of line on copies of the pair's state so that
// neither their registers nor its address weigh on the GJK and EPA loops.
__device__ __noinline__ void warp_refine(const WarpTeam<32> t, const MemBodies B, GjkState* g,
                                         const uint32_t* subtab) {
  GjkState s = *g;
  gjk_refine(t, B, s, kRefineIters, subtab);
  *g = s;
}

// full capacity: certified, from the start, or (a contact that only outgrew the small
// capacity) with FP32 planes, on from the polytope that the small pass left in smem, which is
// kept in a record of the batch's meanwhile
__device__ __noinline__ void warp_epa_full(const WarpTeam<32> t, const MemBodies B, const Config* cfg, bool certified,
                                           const GjkState* g, unsigned char* smem, const EpaResumeSink sink,
                                           const EpaRun<EpaMemSmall>* run, int status, EpaOut* out) {
  Config c = *cfg;
  EpaOut o;
  o.status = status;
  o.resume = -1;
  if (certified)
    c.flags |= OGX_F_EPA_FP64_PLANES;
  else
    epa_save_run(t, c, *reinterpret_cast<EpaMemSmall*>(smem), sink, o, *run);
  t.sync();
  const EpaResume* rs = o.resume >= 0 ? sink.buf + o.resume : nullptr;
  epa_pair<true>(t, B, c, *g, *reinterpret_cast<EpaMemCert*>(smem), o, false, EpaResumeSink{nullptr, nullptr, 0}, rs);
  *out = o;
}

__device__ __forceinline__ void count(const DevBatch& B, int slot, bool lead) {
  if (lead) atomicAdd(B.counts + slot, 1);
}

template <int kMode>
__global__ void __launch_bounds__(32, kMode == kModeGjk ? 20 : 16) k_warp_pair(DevBatch B) {
  extern __shared__ __align__(16) unsigned char smem_raw[];  // EPA modes: one EpaMemCert
  const WarpTeam<32> t;
  const int p = blockIdx.x;
  const bool lead = t.lane() == 0;
  const int2 pr = B.pairs[p];
  bool bad = pr.x < 0 || pr.x >= B.nbodies || pr.y < 0 || pr.y >= B.nbodies;
  BodyRef ra{0u, 0}, rb{0u, 0};
  if (!bad) {
    ra = B.bodies[pr.x];
    rb = B.bodies[pr.y];
    bad = ra.n < 1 || rb.n < 1;
  }
  if (bad) {
    if (lead) mark_bad(B, p);
    return;
  }
  const int bucket = bucket_of(ra.n > rb.n ? ra.n : rb.n);
  WarpBodies src;
  src.bind(B.pool, ra, rb, t.lane());
  GjkState g;
  int status = 0;
  bool late = false;  // a contact that the FP64 continuation found: certified EPA at once
  if constexpr (kMode != kModeEpa) {
    count(B, kCntGjk + bucket, lead);
    int2 ws = make_int2(0, 0);
    if (B.warm) {
      ws = B.warm[p];
      if (ws.x < 0 || ws.x >= ra.n || ws.y < 0 || ws.y >= rb.n) ws = make_int2(0, 0);
    }
    gjk_pair(t, src, B.cfg, g, ws.x, ws.y, B.subtab);
    status = g.status;
    if (g.polish) {
      count(B, g.certain ? kCntRefine : bucket_max(bucket) <= kRefineLaneMax ? kCntRefineFull : kCntRefineBig, lead);
      GjkState r = g;
      r.status = 0;
      warp_refine(t, src.mem, &r, B.subtab);
      status |= r.status;
      late = kMode == kModeGjkEpa && gjk_contact(r);
      g = r;
    }
    if (kMode == kModeGjk || !gjk_contact(g)) {
      if (lead) {
        store_simplex(B.smp + p, g);
        B.dist[p] = g.dist;
        if (B.status) B.status[p] = status;
        if (kMode == kModeGjkEpa) store3(B.nrm + 3 * (size_t)p, sep_normal(g));
      }
      return;
    }
    if (lead) store_simplex(B.smp + p, g);
  } else {
    const gkSimplex& s = B.smp[p];
    const float d = B.dist[p];
    if (!(s.nvrtx == 4 || !(d > FLT_EPSILON))) {  // separated: only a normal
      const fv3 n = simplex_sep_normal(src.mem, s);
      if (lead) {
        store3(B.nrm + 3 * (size_t)p, n);
        if (B.status) B.status[p] = 0;
      }
      return;
    }
    load_simplex(&s, d, g);
    t.sync();  // every lane has read the simplex before lane 0 replaces its witnesses
  }
  if constexpr (kMode != kModeGjk) {
    EpaOut o;
    EpaRun<EpaMemSmall> run;
    if (!late) {
      count(B, kCntEpa + bucket, lead);
      epa_pair(t, src, B.cfg, g, *reinterpret_cast<EpaMemSmall*>(smem_raw), o, true,
               EpaResumeSink{nullptr, nullptr, 0}, nullptr, run);
      if (!o.spill && o.polish) count(B, kCntPolish, lead);
    } else {
      o.spill = o.spill64 = true;
    }
    if (o.spill) {
      count(B, late ? kCntSpillLate : kCntSpill, lead);
      t.sync();
      const GjkState g2 = g;
      EpaOut o2;
      const EpaRun<EpaMemSmall> run2 = run;
      const EpaResumeSink sink{B.resume, B.counts + kCntResume, B.resume_cap};
      warp_epa_full(t, src.mem, &B.cfg, o.spill64, &g2, smem_raw, sink, &run2, o.status, &o2);
      o = o2;
    }
    if (o.polish) epa_polish(src, o);
    if (lead) {
      B.dist[p] = o.dist;
      gkSimplex* s = B.smp + p;
      s->witnesses[0][0] = o.w0.x;
      s->witnesses[0][1] = o.w0.y;
      s->witnesses[0][2] = o.w0.z;
      s->witnesses[1][0] = o.w1.x;
      s->witnesses[1][1] = o.w1.y;
      s->witnesses[1][2] = o.w1.z;
      store3(B.nrm + 3 * (size_t)p, o.nrm);
      if (B.status) B.status[p] = status | o.status;
    }
  }
}

cudaError_t launch_warp_pairs(const DevBatch& B, cudaStream_t st) {
  if (B.mode == kModeGjk)
    k_warp_pair<kModeGjk><<<B.npairs, 32, 0, st>>>(B);
  else if (B.mode == kModeGjkEpa)
    k_warp_pair<kModeGjkEpa><<<B.npairs, 32, sizeof(EpaMemCert), st>>>(B);
  else
    k_warp_pair<kModeEpa><<<B.npairs, 32, sizeof(EpaMemCert), st>>>(B);
  return cudaGetLastError();
}

}  // namespace ogx
