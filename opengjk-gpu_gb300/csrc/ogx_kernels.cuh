// ogx_kernels.cuh -- device kernels of the batched pipeline.
//
//   k_pack    AoS points (bodies concatenated) -> padded SoA pool, one warp per body
//   k_bin     validate each pair and append it to the work list of its size bucket
//             (bucket = larger point count: <=16, 32, 64, 128, 256, 512, more)
//   k_gjk     persistent GJK over one bucket: a team of L lanes per pair, both bodies
//             in registers (K float4 blocks of x, y, z per lane and body); contacts are
//             appended to the bucket's EPA list, separated pairs to the refinement's: those
//             whose support is proved exact, and those to be continued in FP64
//   k_refine, k_refine_cont
//             exact closest points of the former, FP64 continuations of the latter
//   k_epa     persistent EPA over one bucket's contacts, polytope in shared memory (k_epa_few:
//             the same for small and medium batches)
//   k_epa_spill
//             EPA at full capacity, and the certified runs, one warp per contact
//   k_polish  FP64 re-solve of the bucket kernels' final faces, one thread per contact
//   k_warp_pair
//             all of it with one warp per pair, for small batches
// All work lists are filled with warp-aggregated atomics (a contact's face is kept at its
// pair's index); kernels stride over them, so the grid size is independent of the batch (persistent launch, graph-capturable).
#pragma once

#include "ogx_bodies.cuh"
#include "ogx_epa.cuh"
#include "ogx_gjk.cuh"

namespace ogx {

constexpr int kBuckets = 7;
constexpr int kBucketMax[kBuckets] = {16, 32, 64, 128, 256, 512, 0x7fffffff};

OGX_HD int bucket_of(int m) {
  return m <= 16 ? 0 : m <= 32 ? 1 : m <= 64 ? 2 : m <= 128 ? 3 : m <= 256 ? 4 : m <= 512 ? 5 : 6;
}

OGX_HD int bucket_max(int b) { return b == kBuckets - 1 ? 0x7fffffff : 16 << b; }

// re-solve request of a contact, at its pair's index: none (kind 0), or the final EPA face
// (kind 1)
struct PolishRec {
  int pair;
  int kind;
  int face[3][2];
};

enum { kModeGjk = 1, kModeGjkEpa = 2, kModeEpa = 3 };

// counter slots in DevBatch::counts
constexpr int kCntGjk = 0;                  // [0, kBuckets)
constexpr int kCntEpa = kBuckets;           // [kBuckets, 2 kBuckets)
constexpr int kCntPolish = 2 * kBuckets;    // EPA faces to re-solve in FP64
constexpr int kCntRefine = 2 * kBuckets + 1;  // separated pairs to re-solve (support certified)
constexpr int kCntRefineFull = 2 * kBuckets + 2;  // separated pairs to continue in FP64, bodies <= 128 points
constexpr int kCntSpill = 2 * kBuckets + 3;  // contacts that outgrew the small EPA capacity
constexpr int kCntRefineBig = 2 * kBuckets + 4;  // the same, larger bodies
constexpr int kCntSpillLate = 2 * kBuckets + 5;  // contacts found by the FP64 refinement
constexpr int kCntResume = 2 * kBuckets + 6;  // capacity spills saved for the full pass to resume
constexpr int kCntSlots = 2 * kBuckets + 7;
// FP64 continuations of pairs whose bodies have at most this many points are scanned by
// teams of 8 lanes, larger ones by whole warps
constexpr int kRefineLaneMax = 128;
constexpr int kRefineIters = 16;

struct DevBatch {
  const float* pool;
  const BodyRef* bodies;
  int nbodies;
  const int2* pairs;  // gkCollisionPair
  int npairs;
  gkSimplex* smp;
  float* dist;
  float* nrm;       // may be null in GJK mode
  int32_t* status;  // may be null
  int* lists;       // kBuckets regions of npairs entries
  int* elists;      // kBuckets regions of npairs entries
  int* counts;      // kCntSlots
  PolishRec* polish;
  int* refine;        // npairs entries: separated pairs whose FP32 support was proved exact
  int* refine_full;   // npairs entries: the others (small bodies from the front, large ones
                      // from the back)
  int* spill;         // npairs entries: contacts to re-run at full EPA capacity
  EpaResume* resume;  // resume_cap saved small-capacity expansions (null: none)
  int resume_cap;
  const int2* warm;   // optional: GJK start vertex indices per pair (out of range: ignored)
  const uint32_t* subtab;  // sub-distance decision table (fill_subtab); null: the tree
  const float* xf;    // posed kernels only: 12 floats per body (R row-major, t), the pool
                      // then holds the bodies in their own frame
  ogx_config cfg;
  int mode;
  int wide_contacts = 0;  // k_epa_few: a warp per contact up to this many
  int epa_min = 0, epa_max = 0x7fffffff;  // k_epa: runs for this many contacts of the bucket only
};

// Append `want` lanes' items to a list guarded by counter *ctr; returns the slot of this
// lane (valid where want).  One atomic per converged group of lanes.
__device__ __forceinline__ int warp_append(int* ctr, bool want) {
  const unsigned act = __activemask();
  const unsigned m = __ballot_sync(act, want);
  if (m == 0u) return -1;
  const int wl = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  int base = 0;
  if (wl == leader) base = atomicAdd(ctr, __popc(m));
  base = __shfl_sync(act, base, leader);
  return base + __popc(m & ((1u << wl) - 1u));
}

__device__ __forceinline__ void store_simplex(gkSimplex* s, const GjkState& g) {
  s->nvrtx = g.n;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const bool live = k < g.n;
    s->vrtx[k][0] = live ? g.P[k].x : 0.f;
    s->vrtx[k][1] = live ? g.P[k].y : 0.f;
    s->vrtx[k][2] = live ? g.P[k].z : 0.f;
    s->vrtx_idx[k][0] = live ? g.ia[k] : 0;
    s->vrtx_idx[k][1] = live ? g.ib[k] : 0;
  }
  s->witnesses[0][0] = g.w0.x;
  s->witnesses[0][1] = g.w0.y;
  s->witnesses[0][2] = g.w0.z;
  s->witnesses[1][0] = g.w1.x;
  s->witnesses[1][1] = g.w1.y;
  s->witnesses[1][2] = g.w1.z;
}

__device__ __forceinline__ void load_simplex(const gkSimplex* s, float dist, GjkState& g) {
  g.n = s->nvrtx;
  if (g.n < 1 || g.n > 4) g.n = 1;
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    g.P[k] = v3<float>(s->vrtx[k][0], s->vrtx[k][1], s->vrtx[k][2]);
    g.ia[k] = s->vrtx_idx[k][0];
    g.ib[k] = s->vrtx_idx[k][1];
  }
  g.w0 = v3<float>(s->witnesses[0][0], s->witnesses[0][1], s->witnesses[0][2]);
  g.w1 = v3<float>(s->witnesses[1][0], s->witnesses[1][1], s->witnesses[1][2]);
  g.dist = dist;
  g.status = 0;
  g.polish = false;
}

__device__ __forceinline__ void store3(float* p, fv3 v) {
  p[0] = v.x;
  p[1] = v.y;
  p[2] = v.z;
}

// a pair that cannot be run: status OGX_PAIR_BAD_INPUT, distance NaN, normal (1, 0, 0)
__device__ __forceinline__ void mark_bad(const DevBatch& B, int p) {
  B.dist[p] = __int_as_float(0x7fc00000);
  if (B.status) B.status[p] = OGX_S_BAD_INPUT;
  if (B.nrm) store3(B.nrm + 3 * (size_t)p, v3<float>(1.f, 0.f, 0.f));
  if (B.mode != kModeEpa) B.smp[p].nvrtx = 0;
}

// ---------------------------------------------------------------------------------
// source of body points for bucket kernels: registers (K > 0), memory (K == 0), or
// memory staged through D shared-memory slots per lane (K == 0, D > 0)
template <int L, int K, int D = 0>
struct SrcOf {
  typedef RegBodies<L, K> type;
};
template <int L>
struct SrcOf<L, 0, 0> {
  typedef MemBodies type;
};
template <int L, int D>
struct SrcOf<L, 0, D> {
  typedef StagedBodies<L, D> type;
};

// the GJK kernels' memory scans keep four blocks per lane in flight
template <int L, int K, int D = 0>
struct GjkSrcOf {
  typedef typename SrcOf<L, K, D>::type type;
};
template <int L>
struct GjkSrcOf<L, 0, 0> {
  typedef WideMemBodies type;
};
// posed kernel variants (memory scans only): the source of the plain variant with the
// poses applied on the fly
template <bool kPosed, class Src>
struct PoseOf {
  typedef Src type;
};
template <class Src>
struct PoseOf<true, Src> {
  typedef Posed<Src> type;
};

// shared memory of the staging slots of a block of kStageStride threads
OGX_HD constexpr size_t staging_bytes(int D) { return D > 0 ? (size_t)(D + 1) * 3 * sizeof(float4) * kStageStride : 0; }

// xa, xb: the poses of the pair's bodies (read by posed sources only)
template <int L, int K>
__device__ __forceinline__ void bind_src(RegBodies<L, K>& s, const float* pool, BodyRef a,
                                         BodyRef b, int lane, float4*, const float*, const float*) {
  s.bind(pool, a, b, lane);
}
template <int L>
__device__ __forceinline__ void bind_src(MemBodies& s, const float* pool, BodyRef a, BodyRef b,
                                         int, float4*, const float*, const float*) {
  s.bind(pool, a, b);
}
template <int L, int D>
__device__ __forceinline__ void bind_src(StagedBodies<L, D>& s, const float* pool, BodyRef a,
                                         BodyRef b, int lane, float4* slots, const float*, const float*) {
  s.bind(pool, a, b, lane, slots);
}
template <int L, class Base>
__device__ __forceinline__ void bind_src(Posed<Base>& s, const float* pool, BodyRef a, BodyRef b,
                                         int, float4*, const float* xa, const float* xb) {
  s.bind_posed(pool, a, b, xa, xb);
}
// the pose of body i (posed kernels), or null
template <bool kPosed>
__device__ __forceinline__ const float* pose_of(const DevBatch& B, int i) {
  return kPosed ? B.xf + 12 * (size_t)i : nullptr;
}

// A team's next pair, loaded one pair ahead: the chain list -> pair -> bodies is three
// dependent loads, which otherwise start every pair.
struct NextPair {
  int p;
  int2 pr;
  BodyRef ra, rb;
  __device__ __forceinline__ void load(const DevBatch& B, const int* list, int j, int cnt) {
    p = -1;
    if (j < cnt) {
      p = list[j];
      pr = B.pairs[p];
      ra = B.bodies[pr.x];
      rb = B.bodies[pr.y];
    }
  }
};

// Store one finished pair's GJK result and route it (EPA list, FP64 refinement list).
__device__ __forceinline__ void gjk_store(const DevBatch& B, int bucket, int p, const GjkState& g, bool lead) {
  const bool contact = gjk_contact(g);
  if (lead) {
    store_simplex(B.smp + p, g);
    B.dist[p] = g.dist;
    if (B.status) B.status[p] = g.status;
    if (B.mode == kModeGjkEpa && !contact && !g.polish) store3(B.nrm + 3 * (size_t)p, sep_normal(g));
    // pairs sent to the FP64 refinement get their normal there
  }
  // The lists' slots: one atomic per list for the converged lanes, all three on their way
  // before the first is waited for.  Certified pairs are re-solved; the uncertain ones go to
  // the FP64 continuation's lists.
  const bool to_epa = lead && B.mode == kModeGjkEpa && contact;
  const bool certain = lead && g.polish && g.certain, uncertain = lead && g.polish && !g.certain;
  const bool small = bucket_max(bucket) <= kRefineLaneMax;
  const unsigned act = __activemask();
  const unsigned me = __ballot_sync(act, to_epa), mc = __ballot_sync(act, certain), mu = __ballot_sync(act, uncertain);
  const int wl = threadIdx.x & 31;
  const unsigned below = (1u << wl) - 1u;
  int be = 0, bc = 0, bu = 0;
  if (me && wl == __ffs(me) - 1) be = atomicAdd(B.counts + kCntEpa + bucket, __popc(me));
  if (mc && wl == __ffs(mc) - 1) bc = atomicAdd(B.counts + kCntRefine, __popc(mc));
  if (mu && wl == __ffs(mu) - 1) bu = atomicAdd(B.counts + (small ? kCntRefineFull : kCntRefineBig), __popc(mu));
  if (me) {
    be = __shfl_sync(act, be, __ffs(me) - 1);
    if (to_epa) B.elists[(size_t)bucket * B.npairs + be + __popc(me & below)] = p;
  }
  if (mc) {
    bc = __shfl_sync(act, bc, __ffs(mc) - 1);
    if (certain) B.refine[bc + __popc(mc & below)] = p;
  }
  if (mu) {
    bu = __shfl_sync(act, bu, __ffs(mu) - 1);
    const int u = bu + __popc(mu & below);
    if (uncertain) B.refine_full[small ? u : B.npairs - 1 - u] = p;
  }
}

template <int L, int K, int OCC = 1, int D = 0, bool kPosed = false>
__global__ void __launch_bounds__(kStageStride, OCC) k_gjk(DevBatch B, int bucket) {
  extern __shared__ __align__(16) unsigned char smem_raw[];  // staging slots (D > 0)
  float4* slots = reinterpret_cast<float4*>(smem_raw) + threadIdx.x;
  const WarpTeam<L> t;
  const WarpTeam<L, true> all;  // the iterations, by all teams of the warp together
  const int team = (blockIdx.x * blockDim.x + threadIdx.x) / L;
  const int nteams = (gridDim.x * blockDim.x) / L;
  const int cnt = B.counts[kCntGjk + bucket];
  const int* list = B.lists + (size_t)bucket * B.npairs;
  NextPair next;
  next.load(B, list, team, cnt);
#pragma unroll 1
  for (int j = team; all.warp_any(j < cnt); j += nteams) {
    const bool have = j < cnt;
    typename PoseOf<kPosed, typename GjkSrcOf<L, K, D>::type>::type src;
    GjkRun r;
    const int p = next.p;
    r.done = true;
    if (have) {
      bind_src<L>(src, B.pool, next.ra, next.rb, t.lane(), slots, pose_of<kPosed>(B, next.pr.x),
                  pose_of<kPosed>(B, next.pr.y));
      int2 ws = make_int2(0, 0);
      if (B.warm) {
        ws = B.warm[p];
        if (ws.x < 0 || ws.x >= next.ra.n || ws.y < 0 || ws.y >= next.rb.n) ws = make_int2(0, 0);
      }
      gjk_start(src, r, ws.x, ws.y);
    }
#pragma unroll 1
    while (all.warp_any(!r.done)) gjk_iterate(all, src, B.cfg, r, B.subtab, !r.done);
    next.load(B, list, j + nteams, cnt);  // on its way while this pair is finished
    if (have) {
      GjkState g;
      gjk_end(t, src, B.cfg, r, g);
      gjk_store(B, bucket, p, g, t.lane() == 0);
    }
  }
  if constexpr (D > 0) cp_async_wait<0>();  // no copy outlives the block
}


// kFull: the full-capacity pass over the spill list -- certified re-runs where the entry
// asks for FP64 planes, and the FP64 polish of the result done here by lane 0 instead of
// through the polish list, so that the polish pass need not wait for this one
// spill list entry codes: a pair index, or a saved expansion to resume
constexpr int kSpill64 = 1 << 30;      // the re-run solves every face plane in FP64
constexpr int kSpillResume = 1 << 29;  // low bits: the EpaResume record to continue

__device__ __forceinline__ int status_so_far(const DevBatch& B, int p) {
  return B.status && B.mode != kModeEpa ? B.status[p] : 0;
}

// Stores a contact's result, or (false) its spill list code.
// before: the pair's status so far (0 for EPA-only calls)
template <bool kFull, class Team, class Src>
__device__ __forceinline__ bool epa_store(const Team& t, const DevBatch& B, int p, int before, const Src& src,
                                          EpaOut& o, int* spill_code) {
  const bool lead = t.lane() == 0;
  if (o.spill) {
    if (o.resume >= 0 && lead) B.resume[o.resume].pair = p;
    if (lead && !kFull) B.polish[p].kind = 0;  // the full pass polishes its own
    if (spill_code) *spill_code = o.resume >= 0 ? (kSpillResume | o.resume) : (p | (o.spill64 ? kSpill64 : 0));
    return false;
  }
  if (kFull && lead && o.polish) {
    epa_polish(src, o);
    o.polish = false;
  }
  if (lead && o.kept) {
    const gkSimplex& s = B.smp[p];
    store3(B.nrm + 3 * (size_t)p, unit_or_x(v3<float>(s.witnesses[1][0] - s.witnesses[0][0],
                                                      s.witnesses[1][1] - s.witnesses[0][1],
                                                      s.witnesses[1][2] - s.witnesses[0][2])));
    if (B.status) B.status[p] = before | o.status;
  } else if (lead) {
    B.dist[p] = o.dist;
    gkSimplex* s = B.smp + p;
    s->witnesses[0][0] = o.w0.x;
    s->witnesses[0][1] = o.w0.y;
    s->witnesses[0][2] = o.w0.z;
    s->witnesses[1][0] = o.w1.x;
    s->witnesses[1][1] = o.w1.y;
    s->witnesses[1][2] = o.w1.z;
    store3(B.nrm + 3 * (size_t)p, o.nrm);
    if (B.status) B.status[p] = before | o.status;
  }
  if (lead && o.polish) {
    PolishRec r;
    r.pair = p;
    r.kind = 1;
    for (int k = 0; k < 3; ++k) {
      r.face[k][0] = o.face[k][0];
      r.face[k][1] = o.face[k][1];
    }
    B.polish[p] = r;
    atomicAdd(B.counts + kCntPolish, 1);  // (a count only: nothing waits for its value)
  } else if (lead && !kFull) {
    B.polish[p].kind = 0;
  }
  return true;
}

template <int L, int K, bool kFull = false, int D = 0, bool kPosed = false, class Mem>
__device__ __forceinline__ bool epa_item(const WarpTeam<L>& t, const DevBatch& B, const Config& cfg, int p,
                                         Mem& M, bool can_spill, int* spill_code = nullptr,
                                         const EpaResume* rs = nullptr, float4* slots = nullptr) {
  const int2 pr = B.pairs[p];
  typename PoseOf<kPosed, typename SrcOf<L, K, D>::type>::type src;
  bind_src<L>(src, B.pool, B.bodies[pr.x], B.bodies[pr.y], t.lane(), slots, pose_of<kPosed>(B, pr.x),
              pose_of<kPosed>(B, pr.y));
  GjkState g;
  load_simplex(B.smp + p, B.dist[p], g);
  EpaOut o;
  const int before = status_so_far(B, p);
  const EpaResumeSink sink{can_spill ? B.resume : nullptr, B.counts + kCntResume, B.resume_cap};
  epa_pair<kFull>(t, src, cfg, g, M, o, can_spill, sink, rs);
  return epa_store<kFull>(t, B, p, before, src, o, spill_code);
}

// EPA over one bucket's contacts with the small working set (EpaMemSmall per team in
// shared memory); contacts that need more than kEpaSmallIters expansions, or whose FP32
// expansion met an inconsistent horizon, go to the spill list
// Byte stride between the teams' working sets in shared memory: whole 128-byte lines
// plus 4 L bytes, so that the teams of a warp start L banks apart and their lanes' 4-byte
// and 1-byte accesses to the same field of their own working sets fall in different banks
// (the unpadded 2288-byte sets started 28 banks apart, and lanes of neighbouring teams
// met in the same banks: 466k conflicts in one 16-point EPA launch).
OGX_HD constexpr size_t epa_team_stride(int L) {
  return (sizeof(EpaMemSmall) + 127) / 128 * 128 + (L >= 4 ? (4 * (size_t)L) % 128 : 16);
}

// shared memory of k_epa: the teams' working sets, then the staging slots (D > 0)
template <int L>
OGX_HD constexpr size_t epa_mem_bytes() { return (kStageStride / L) * epa_team_stride(L); }

template <int L, int K, int D = 0, bool kPosed = false>
__device__ __forceinline__ void epa_bucket(const DevBatch& B, int bucket, int cnt) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  float4* slots = reinterpret_cast<float4*>(smem_raw + epa_mem_bytes<L>()) + threadIdx.x;
  const WarpTeam<L> t;
  EpaMemSmall& M = *reinterpret_cast<EpaMemSmall*>(smem_raw + (threadIdx.x / L) * epa_team_stride(L));
  const int team = (blockIdx.x * blockDim.x + threadIdx.x) / L;
  const int nteams = (gridDim.x * blockDim.x) / L;
  const int* list = B.elists + (size_t)bucket * B.npairs;
  const WarpTeam<L, true> all;  // the expansions, by all teams of the warp together
  const EpaResumeSink sink{B.resume, B.counts + kCntResume, B.resume_cap};
  NextPair next;
  next.load(B, list, team, cnt);
#pragma unroll 1
  for (int j = team; all.warp_any(j < cnt); j += nteams) {
    typename PoseOf<kPosed, typename SrcOf<L, K, D>::type>::type src;
    EpaRun<EpaMemSmall> r;
    EpaOut o;
    const int p = next.p;
    bool run = false;
    if (j < cnt) {
      bind_src<L>(src, B.pool, next.ra, next.rb, t.lane(), slots, pose_of<kPosed>(B, next.pr.x),
                  pose_of<kPosed>(B, next.pr.y));
      GjkState g;
      load_simplex(B.smp + p, B.dist[p], g);
      run = epa_start(t, src, B.cfg, g, M, o, r);
      if (!run) epa_store<false>(t, B, p, status_so_far(B, p), src, o, nullptr);  // touching
    }
    const bool loop = run;
#pragma unroll 1
    while (all.warp_any(run)) {
      run = epa_step(all, src, B.cfg, M, o, r, true, run);
      run = run && r.it < B.cfg.epa_max_iter;
    }
    // (on their way while this contact's face is worked out; not through the loop, whose
    // registers they would take)
    next.load(B, list, j + nteams, cnt);
    if (loop) {
      const int before = status_so_far(B, p);
      epa_finish(t, src, B.cfg, M, o, r, true, sink);
      int code = 0;
      const bool ok = epa_store<false>(t, B, p, before, src, o, &code);
      const bool lead = t.lane() == 0;
      const int q = warp_append(B.counts + kCntSpill, lead && !ok);
      if (lead && !ok) B.spill[q] = code;
    }
    all.sync();  // the next contact reuses M
  }
  if constexpr (D > 0) cp_async_wait<0>();  // no copy outlives the block
}

template <int L, int K, int OCC = 1, int D = 0, bool kPosed = false>
__global__ void __launch_bounds__(kStageStride, OCC) k_epa(DevBatch B, int bucket) {
  const int cnt = B.counts[kCntEpa + bucket];
  epa_bucket<L, K, D, kPosed>(B, bucket, cnt >= B.epa_min && cnt <= B.epa_max ? cnt : 0);
}

// EPA over one bucket's contacts in a batch of at most 24,576 pairs.  A contact is bound by its
// chain of expansions, which a whole warp ends soonest, as long as the contacts do not queue for
// warps; a bucket with more of them than about a wave (4 blocks of 4 warps on 152 SMs are 2,432;
// the buckets of small bodies run beside one another) is done sooner by narrow teams.  How many
// there are only the device knows, so both are in one kernel.  (A warp per contact whatever their
// number, by the batch's pairs alone: 16,000 contacts of 16-point bodies 418 us, now 286, 16,000
// of 64-point ones 1,213 and 1,025, 20,000 power-law pairs 370 and 333.  Limits of 1,000, 1,500,
// 2,000 and 2,432 contacts in every bucket: 20,000 power-law pairs 333, 333, 342, 344; but with
// 1,000 for large bodies too 6,500 ellipsoid pairs took 279 us, now 244, 20,000 scene pairs 381
// and 330.)
constexpr int kWideContacts[kBuckets] = {1000, 1000, 1000, 1000, 2000, 3000, 2000};
template <int LN>
__global__ void __launch_bounds__(kStageStride, 4) k_epa_few(DevBatch B, int bucket) {
  const int cnt = B.counts[kCntEpa + bucket];
  if (cnt <= B.wide_contacts)
    epa_bucket<32, 0>(B, bucket, cnt);
  else
    epa_bucket<LN, 0>(B, bucket, cnt);
}

// ---------------------------------------------------------------------------------
// launch table (one translation unit per kernel family, see ogx_k_*.cu)

typedef void (*BucketKernel)(DevBatch, int);

struct KernelInfo {
  BucketKernel fn;
  int L;  // lanes per pair
  int K;  // float4 blocks per lane and body kept in registers (0: read from memory);
          // + 256 * m for a variant compiled for at least m resident blocks per SM
          // (fewer registers per thread, more warps)
          // + 65536 * D for a memory variant that stages D blocks per lane through
          // shared memory
};
constexpr int kOccShift = 8;
constexpr int kStageShift = 16;
OGX_HD int variant_blocks(int K) { return K & ((1 << kOccShift) - 1); }
OGX_HD int variant_stages(int K) { return (K >> kStageShift) & 0xff; }

// Compiled variants of the bucket kernels (ogx_k_gjk_*.cu / ogx_k_epa_*.cu).  A variant
// (L, K) can serve a bucket whose bodies have at most 4 L K points (K = 0: any size, the
// points are re-read from memory).  The engine picks one per bucket (autotuned).
int gjk_variants(const KernelInfo** out);
int epa_variants(const KernelInfo** out);
int gjk_variants_a(const KernelInfo** out);
int gjk_variants_b(const KernelInfo** out);
int gjk_variants_c(const KernelInfo** out);
int gjk_variants_d(const KernelInfo** out);
int gjk_variants_e(const KernelInfo** out);
int epa_variants_a(const KernelInfo** out);
int epa_variants_b(const KernelInfo** out);
int epa_variants_c(const KernelInfo** out);
int epa_variants_d(const KernelInfo** out);
// the posed kernels (ogx_k_posed.cu): one GJK and one EPA variant per bucket
void posed_variants(const KernelInfo** gjk, const KernelInfo** epa);
// EPA of small and medium batches, one kernel per bucket (ogx_k_epa_few.cu)
void few_variants(const KernelInfo** epa);

// non-template kernels (ogx_k_misc.cu, ogx_k_bin.cu, ogx_k_spill.cu)
cudaError_t launch_refine(const DevBatch& B, int grid, int grid_cont, cudaStream_t st, cudaStream_t st2,
                          cudaEvent_t ready);
cudaError_t continue_occupancy(int block, int* per_sm);
cudaError_t launch_epa_spill(const DevBatch& B, int grid, cudaStream_t st, bool late = false);
cudaError_t epa_spill_occupancy(int block, int* per_sm);
cudaError_t refine_occupancy(int block, int* per_sm);
cudaError_t launch_pack(const float* aos, const int64_t* voff, BodyRef* bodies, int nbodies,
                        float* pool, int grid, cudaStream_t st);
// packs bodies whose points the device reads where the caller keeps them (src[b]: xyz of
// body b, host memory of a device that reads pageable memory); bodies[] already holds
// each body's count and pool offset
cudaError_t launch_pack_ptrs(const float* const* src, int nbodies, BodyRef* bodies, float* pool, int grid,
                             cudaStream_t st);
cudaError_t launch_pack_ptrs64(const double* const* src, int nbodies, const int64_t* voff, BodyRef* bodies,
                               float* pool, double* c64, int grid, cudaStream_t st);
cudaError_t launch_bin(const DevBatch& B, int grid, cudaStream_t st);
// the whole pipeline with one warp per pair (ogx_k_warp.cu), any mode; not posed
cudaError_t launch_warp_pairs(const DevBatch& B, cudaStream_t st);
cudaError_t launch_polish(const DevBatch& B, int grid, cudaStream_t st);
cudaError_t polish_occupancy(int block, int* per_sm);

}  // namespace ogx
