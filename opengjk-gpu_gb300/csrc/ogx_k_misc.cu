// ogx_k_misc.cu -- pool packing, the FP64 refinement and polish passes.
#include "ogx_kernels.cuh"
#include "ogx_continue.cuh"

namespace ogx {

// ---------------------------------------------------------------------------------
// Packs every body and marks the ones with a NaN or infinite coordinate in the body
// table (point count stored negated, see body_points), which the binning turns into
// OGX_PAIR_BAD_INPUT for their pairs; a later upload of finite points clears the mark.
__global__ void k_pack(const float* __restrict__ aos, const int64_t* __restrict__ voff,
                       BodyRef* __restrict__ bodies, int nbodies, float* __restrict__ pool) {
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int b = warp; b < nbodies; b += nwarps) {
    const BodyRef r = bodies[b];
    const int n = body_points(r);
    const int n4 = round4(n);
    const float* src = aos + 3 * voff[b];
    float* dst = pool + 4 * (size_t)r.quad;
    bool finite = true;
    for (int i = lane; i < n4; i += 32) {
      const int s = i < n ? i : 0;
      const float x = src[3 * s], y = src[3 * s + 1], z = src[3 * s + 2];
      finite = finite && is_finite(x) && is_finite(y) && is_finite(z);
      dst[i] = x;
      dst[n4 + i] = y;
      dst[2 * n4 + i] = z;
    }
    finite = __all_sync(0xffffffffu, finite);
    if (lane == 0) bodies[b].n = finite ? n : -n;
  }
}

// After FP64 refinement: contacts join their bucket's EPA list, separated pairs get their
// normal from the refined witnesses.
__device__ void refine_store(const DevBatch& B, int p, const GjkState& g) {
  store_simplex(B.smp + p, g);
  B.dist[p] = g.dist;
  if (B.status) B.status[p] |= g.status;
  if (B.mode == kModeGjkEpa) {
    if (gjk_contact(g)) {
      // the FP32 pass called it separated: a contact within rounding of the boundary,
      // for the certified full-capacity pass over the late list (filled from the end of
      // the spill array: these pairs are not contacts of the FP32 pass, so both lists
      // together hold at most npairs entries)
      const int q = atomicAdd(B.counts + kCntSpillLate, 1);
      B.spill[B.npairs - 1 - q] = p | kSpill64;
    } else {
      store3(B.nrm + 3 * (size_t)p, sep_normal(g));
    }
  }
}

// The pair's bodies for the FP64 passes: as stored, or posed (the posed pipeline)
__device__ __forceinline__ void bind_mem(MemBodies& mb, const DevBatch& B, int2, BodyRef ra, BodyRef rb) {
  mb.bind(B.pool, ra, rb);
}
__device__ __forceinline__ void bind_mem(Posed<MemBodies>& mb, const DevBatch& B, int2 pr, BodyRef ra,
                                         BodyRef rb) {
  mb.bind_posed(B.pool, ra, rb, B.xf + 12 * (size_t)pr.x, B.xf + 12 * (size_t)pr.y);
}
// Re-solve of the separated pairs whose final support the GJK kernel proved exact (one
// thread per pair): the exact closest point of their simplex in double-float arithmetic.
template <bool kPosed>
__global__ void __launch_bounds__(128) k_refine(DevBatch B) {
  const int cnt = B.counts[kCntRefine];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += gridDim.x * blockDim.x) {
    const int p = B.refine[k];
    const int2 pr = B.pairs[p];
    const BodyRef ra = B.bodies[pr.x], rb = B.bodies[pr.y];
    typename PoseOf<kPosed, MemBodies>::type mb;
    bind_mem(mb, B, pr, ra, rb);
    GjkState g;
    load_simplex(B.smp + p, B.dist[p], g);
    refine_certain(mb, g);
    refine_store(B, p, g);
  }
}

// A continuation list of the batch (dir = -1: filled from the end of its array)
template <bool kPosed>
struct ListWork {
  typedef typename PoseOf<kPosed, MemBodies>::type Bodies;
  const DevBatch& B;
  const int* list;
  int dir;
  __device__ void idle(Bodies& mb) const { bind_mem(mb, B, make_int2(0, 0), BodyRef{0u, 1}, BodyRef{0u, 1}); }
  __device__ int load(int k, Bodies& mb, GjkState& g) const {
    const int p = list[dir * k];
    const int2 pr = B.pairs[p];
    bind_mem(mb, B, pr, B.bodies[pr.x], B.bodies[pr.y]);
    load_simplex(B.smp + p, B.dist[p], g);
    return p;
  }
  __device__ void store(int p, const GjkState& g) const { refine_store(B, p, g); }
};

// Each list gets a share of the warps by its work: a larger body's continuation (refine_full
// filled from its end, a whole warp scans) counts as kBigCost small ones (four scanned at a
// time).  Both halves of the split at 1:1, 2 blocks per SM -> this split, 3 blocks per SM (what
// 168 registers allow): 30k stress pairs (3,289 large and 13,814 small) 930 -> 852 us, 200k
// scene pairs (14,680 and 3,128) 1,018 -> 1,010, 1M power-law pairs 5,225 -> 5,190; weighted 8,
// 915 / 1,065 / 5,255.  More blocks at fewer registers spill and gain nothing more.
constexpr int kBigCost = 2;
template <bool kPosed>
__global__ void __launch_bounds__(128, 3) k_refine_cont(DevBatch B) {
  const int big = B.counts[kCntRefineBig], small = B.counts[kCntRefineFull];
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  const int64_t cost = (int64_t)kBigCost * big;
  int split = big == 0 ? 0 : (int)(nwarps * cost / (cost + small));
  if (big > 0 && small > 0) split = min(max(split, 1), nwarps - 1);
  if (warp < split)
    continue_pairs<32>(ListWork<kPosed>{B, B.refine_full + (B.npairs - 1), -1}, big, warp, split, B.subtab);
  else
    continue_pairs<8>(ListWork<kPosed>{B, B.refine_full, 1}, small, warp - split, nwarps - split, B.subtab);
}

// The bucket kernels' contacts, list after list, each with the record at its pair's index
template <bool kPosed>
__global__ void __launch_bounds__(128) k_polish(DevBatch B) {
  int first[kBuckets + 1];
  first[0] = 0;
#pragma unroll
  for (int b = 0; b < kBuckets; ++b) first[b + 1] = first[b] + B.counts[kCntEpa + b];
  const int cnt = first[kBuckets];
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < cnt; k += gridDim.x * blockDim.x) {
    int b = 0, f = 0;
#pragma unroll
    for (int q = 1; q < kBuckets; ++q)
      if (k >= first[q]) {
        b = q;
        f = first[q];
      }
    const int p = B.elists[(size_t)b * B.npairs + (k - f)];
    const PolishRec r = B.polish[p];
    if (r.kind != 1) continue;
    const int2 pr = B.pairs[p];
    typename PoseOf<kPosed, MemBodies>::type mb;
    bind_mem(mb, B, pr, B.bodies[pr.x], B.bodies[pr.y]);
    gkSimplex* s = B.smp + p;
    {
      EpaOut o;
      for (int m = 0; m < 3; ++m) {
        o.face[m][0] = r.face[m][0];
        o.face[m][1] = r.face[m][1];
      }
      const float* n = B.nrm + 3 * (size_t)p;
      o.nrm = v3<float>(n[0], n[1], n[2]);
      o.dist = B.dist[p];
      o.status = 0;
      epa_polish(mb, o);
      if (!(o.status & OGX_S_POLISHED)) continue;
      B.dist[p] = o.dist;
      s->witnesses[0][0] = o.w0.x;
      s->witnesses[0][1] = o.w0.y;
      s->witnesses[0][2] = o.w0.z;
      s->witnesses[1][0] = o.w1.x;
      s->witnesses[1][1] = o.w1.y;
      s->witnesses[1][2] = o.w1.z;
      store3(B.nrm + 3 * (size_t)p, o.nrm);
    }
    if (B.status) B.status[p] |= OGX_S_POLISHED;
  }
}


// Pack from a table of coordinate pointers (one per body, xyz interleaved) that address
// the caller's host arrays: on a device that reads pageable host memory through the host's
// page tables (cudaDevAttrPageableMemoryAccess, the GPU of a Grace system over NVLink-C2C)
// the kernel loads the points where the caller keeps them, so the host gathers nothing.
// Bodies with a NaN or infinite coordinate are marked as k_pack does.  From doubles, the pool
// takes each rounded to float and c64 the doubles themselves (point i of body b at
// 3 (voff[b] + i)).  One warp per body; the reads' latency over the link bounds it, so a lane
// has kDeep points on their way before it stores any (one: 31 us for the 2,000 bodies of
// 1,000 power-law pairs, now 13).
template <class T>
__global__ void __launch_bounds__(256) k_pack_ptrs(const T* const* __restrict__ src, int nb,
                                                   BodyRef* __restrict__ bodies, float* __restrict__ pool,
                                                   const int64_t* __restrict__ voff, double* __restrict__ c64) {
  constexpr int kDeep = sizeof(T) == sizeof(double) ? 8 : 16;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int nwarps = (gridDim.x * blockDim.x) >> 5;
  for (int b = warp; b < nb; b += nwarps) {
    const BodyRef r = bodies[b];
    const T* c = src[b];
    const int n4 = round4(r.n);
    float* dst = pool + 4 * (size_t)r.quad;
    bool finite = true;
    for (int i0 = lane; i0 < n4; i0 += 32 * kDeep) {
      T v[kDeep][3];
#pragma unroll
      for (int u = 0; u < kDeep; ++u) {
        const int i = i0 + 32 * u, s = i < r.n ? i : 0;  // (the padding repeats point 0)
        if (i < n4) {
          v[u][0] = c[3 * s];
          v[u][1] = c[3 * s + 1];
          v[u][2] = c[3 * s + 2];
        }
      }
#pragma unroll
      for (int u = 0; u < kDeep; ++u) {
        const int i = i0 + 32 * u;
        if (i >= n4) continue;
        if constexpr (sizeof(T) == sizeof(double)) {
          if (i < r.n) {
            double* d = c64 + 3 * (voff[b] + i);
            d[0] = v[u][0];
            d[1] = v[u][1];
            d[2] = v[u][2];
          }
        }
        const float x = (float)v[u][0], y = (float)v[u][1], z = (float)v[u][2];
        finite = finite && is_finite(x) && is_finite(y) && is_finite(z);
        dst[i] = x;
        dst[n4 + i] = y;
        dst[2 * n4 + i] = z;
      }
    }
    finite = __all_sync(0xffffffffu, finite);
    if (lane == 0 && !finite) bodies[b].n = -r.n;
  }
}

cudaError_t launch_pack_ptrs(const float* const* src, int nbodies, BodyRef* bodies, float* pool, int grid,
                             cudaStream_t st) {
  if (nbodies <= 0) return cudaSuccess;
  k_pack_ptrs<float><<<grid, 256, 0, st>>>(src, nbodies, bodies, pool, nullptr, nullptr);
  return cudaGetLastError();
}

cudaError_t launch_pack_ptrs64(const double* const* src, int nbodies, const int64_t* voff, BodyRef* bodies,
                               float* pool, double* c64, int grid, cudaStream_t st) {
  if (nbodies <= 0) return cudaSuccess;
  k_pack_ptrs<double><<<grid, 256, 0, st>>>(src, nbodies, bodies, pool, voff, c64);
  return cudaGetLastError();
}

cudaError_t launch_pack(const float* aos, const int64_t* voff, BodyRef* bodies, int nbodies,
                        float* pool, int grid, cudaStream_t st) {
  k_pack<<<grid, 256, 0, st>>>(aos, voff, bodies, nbodies, pool);
  return cudaGetLastError();
}

// the launchers run the posed kernels when the batch carries poses (B.xf)
cudaError_t launch_polish(const DevBatch& B, int grid, cudaStream_t st) {
  if (B.xf)
    k_polish<true><<<grid, 128, 0, st>>>(B);
  else
    k_polish<false><<<grid, 128, 0, st>>>(B);
  return cudaGetLastError();
}

// k_refine and the FP64 continuations touch disjoint pairs and run on st and st2, beside one
// another when the streams differ (st2 then starts behind `ready`, recorded here; the caller
// joins it back)
cudaError_t launch_refine(const DevBatch& B, int grid, int grid_cont, cudaStream_t st, cudaStream_t st2,
                          cudaEvent_t ready) {
  cudaError_t e = cudaSuccess;
  if (st2 != st) {
    e = cudaEventRecord(ready, st);
    if (e == cudaSuccess) e = cudaStreamWaitEvent(st2, ready, 0);
  }
  if (e != cudaSuccess) return e;
  if (B.xf) {
    k_refine_cont<true><<<grid_cont, 128, 0, st2>>>(B);
    k_refine<true><<<grid, 128, 0, st>>>(B);
  } else {
    k_refine_cont<false><<<grid_cont, 128, 0, st2>>>(B);
    k_refine<false><<<grid, 128, 0, st>>>(B);
  }
  return cudaGetLastError();
}

cudaError_t continue_occupancy(int block, int* per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_refine_cont<false>, block, 0);
}

cudaError_t refine_occupancy(int block, int* per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_refine<false>, block, 0);
}

cudaError_t polish_occupancy(int block, int* per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_polish<false>, block, 0);
}

}  // namespace ogx
