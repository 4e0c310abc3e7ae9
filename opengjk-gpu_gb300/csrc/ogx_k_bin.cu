// ogx_k_bin.cu -- pair binning.  A translation unit of its own for the double-float arithmetic of
// EPA-only calls' normals: inline here, where it is one chain per thread (300,000 separated pairs
// 71 us, with calls 87), out of line in the kernels whose code it would swell.
#define OGX_INLINE_LEAVES
#include "ogx_kernels.cuh"

namespace ogx {

__device__ __forceinline__ bool pair_ok(const DevBatch& B, int2 pr) {
  return pr.x >= 0 && pr.x < B.nbodies && pr.y >= 0 && pr.y < B.nbodies;
}

__global__ void k_bin(DevBatch B) {
  const int stride = gridDim.x * blockDim.x;
  const int n32 = (B.npairs + 31) & ~31;
  for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n32; p += stride) {
    const bool in = p < B.npairs;
    int b = -1;
    bool bad = false;
    bool work = false;
    if (in) {
      const int2 pr = B.pairs[p];
      bad = !pair_ok(B, pr);
      if (!bad) {
        const int na = B.bodies[pr.x].n, nb = B.bodies[pr.y].n;
        bad = na < 1 || nb < 1;
        b = bucket_of(na > nb ? na : nb);
      }
      if (bad) {
        mark_bad(B, p);
      } else if (B.mode == kModeEpa) {
        // EPA only: contacts go to the EPA lists, separated pairs only get a normal
        const gkSimplex& s = B.smp[p];
        work = s.nvrtx == 4 || !(B.dist[p] > FLT_EPSILON);
        if (!work) {
          MemBodies mb;
          mb.bind(B.pool, B.bodies[pr.x], B.bodies[pr.y]);
          store3(B.nrm + 3 * (size_t)p, simplex_sep_normal(mb, s));
          if (B.status) B.status[p] = 0;
        }
      } else {
        work = true;
      }
    }
    // warp-aggregated append per bucket
    const int key = work ? b : -1;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int wl = threadIdx.x & 31;
    const int leader = __ffs(peers) - 1;
    if (key >= 0) {
      int* ctr = B.counts + (B.mode == kModeEpa ? kCntEpa : kCntGjk) + key;
      int* list = (B.mode == kModeEpa ? B.elists : B.lists) + (size_t)key * B.npairs;
      int base = 0;
      if (wl == leader) base = atomicAdd(ctr, __popc(peers));
      base = __shfl_sync(peers, base, leader);
      list[base + __popc(peers & ((1u << wl) - 1u))] = p;
    }
  }
}

cudaError_t launch_bin(const DevBatch& B, int grid, cudaStream_t st) {
  k_bin<<<grid, 256, 0, st>>>(B);
  return cudaGetLastError();
}

}  // namespace ogx
