// ogx_continue.cuh -- FP64 continuations of GJK by warps that share the supports' scans: the
// refinement's lists, and the separated pairs of bodies given in double.
#pragma once

#include "ogx_kernels.cuh"

namespace ogx {

// the bodies of lane j's pair (j may differ from lane to lane)
__device__ __forceinline__ void shfl_bodies(MemBodies& to, const MemBodies& from, int j) {
#pragma unroll
  for (int w = 0; w < 2; ++w) {
    to.base[w] = reinterpret_cast<const float*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<long long>(from.base[w]), j));
    to.n[w] = __shfl_sync(0xffffffffu, from.n[w], j);
    to.n4[w] = round4(to.n[w]);
  }
}
__device__ __forceinline__ void shfl_bodies(Posed<MemBodies>& to, const Posed<MemBodies>& from, int j) {
  shfl_bodies(static_cast<MemBodies&>(to), static_cast<const MemBodies&>(from), j);
#pragma unroll
  for (int w = 0; w < 2; ++w)
    to.xf[w] = reinterpret_cast<const float*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<long long>(from.xf[w]), j));
}
__device__ __forceinline__ void shfl_bodies(D64Bodies& to, const D64Bodies& from, int j) {
  shfl_bodies(static_cast<MemBodies&>(to), static_cast<const MemBodies&>(from), j);
#pragma unroll
  for (int w = 0; w < 2; ++w)
    to.aos[w] = reinterpret_cast<const double*>(
        __shfl_sync(0xffffffffu, reinterpret_cast<long long>(from.aos[w]), j));
}

// FP64 continuation of GJK for the pairs whose FP32 support was not certain.  An FP64
// instruction holds its SM quadrant's FP64 unit for about 65 cycles however many lanes are
// active (measured, GB300), and a pair's continuation is a chain of a few hundred of them,
// so what counts is that every quadrant has a warp of its own and that a warp's
// instructions serve several pairs only once there are more pairs than that: a warp takes
// ceil(pairs / warps) pairs (1 to 32), one per lane.  Each FP64 iteration scans the warp's
// unfinished pairs for their exact supports, 32 / TL at a time with teams of TL lanes, then
// every lane takes its own pair's FP64 sub-distance step.  (32 pairs per warp always, and
// one thread's serial scans for bodies of at most 128 points, left most SMs idle: 92 + 265
// us for the 6,600 continuations of 200k power-law pairs.)
//
// The work of warp `warp` of `nwarps` over cnt entries.  W.load binds entry k's bodies, loads
// its simplex and returns its pair (negative: nothing to do); W.idle binds a lane that has none
// (never scanned: its r.done stays set); W.store takes the result.
template <int TL, class Work>
__device__ __forceinline__ void continue_pairs(const Work& W, int cnt, int warp, int nwarps,
                                               const uint32_t* subtab) {
  const WarpTeam<TL> t;
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  constexpr int kTeams = 32 / TL;
  const int per = min(32, max(1, (cnt + nwarps - 1) / nwarps));
#pragma unroll 1
  for (int base = per * warp; base < cnt; base += per * nwarps) {
    const int k = base + lane;
    int p = -1;
    typename Work::Bodies mb;
    W.idle(mb);
    GjkState g;
    RefineState r;
    r.done = true;
    if (lane < per && k < cnt) p = W.load(k, mb, g);
    if (p >= 0) {
      g.certain = false;
      refine_begin(mb, g, kRefineIters, r);
    }
#pragma unroll 1
    for (;;) {
      const unsigned m = __ballot_sync(full, !r.done);
      if (m == 0u) break;
      int my_xa = 0, my_xb = 0;
#pragma unroll 1
      for (int j0 = 0; j0 < per; j0 += kTeams) {
        if (((m >> j0) & ((kTeams == 32 ? 0u : (1u << kTeams)) - 1u)) == 0u) continue;
        const int j = j0 + lane / TL;  // this team's pair (lane j & 31's)
        typename Work::Bodies bj;
        shfl_bodies(bj, mb, j & 31);
        const dv3 vj = v3<double>(__shfl_sync(full, r.v.x, j & 31), __shfl_sync(full, r.v.y, j & 31),
                                  __shfl_sync(full, r.v.z, j & 31));
        int xa = 0, xb = 0;
        if (j < 32 && ((m >> j) & 1u)) {
          float ma = -1.0f, mb2 = -1.0f;
          const fv3 fj = floats(vj);
          xa = exact_support(t, bj, 0, -vj, -fj, ma);
          xb = exact_support(t, bj, 1, vj, fj, mb2);
        }
        __syncwarp();
        const int src = ((lane - j0) * TL) & 31;  // the first lane of the team that scanned this lane's pair
        xa = __shfl_sync(full, xa, src);
        xb = __shfl_sync(full, xb, src);
        if (lane >= j0 && lane < j0 + kTeams) {
          my_xa = xa;
          my_xb = xb;
        }
      }
      if (!r.done) refine_step(mb, r, my_xa, my_xb, subtab);
      __syncwarp();
    }
    if (p >= 0) {
      refine_end(mb, r, g);
      W.store(p, g);
    }
    __syncwarp();
  }
}

}  // namespace ogx
