// ogx_k_spill.cu -- EPA at full capacity.  A translation unit of its own for the long arithmetic
// inline: with calls (OGX_LEAF) the kernel held 168 registers, three blocks per SM, and spilled at
// 128; inline it takes 128 and spills nothing.  Where many contacts come here their number per SM
// is what counts: 60,000 contacts of 1,000-point bodies 10,910 us, now 8,930; of 100 points 3,750 and
// 3,390; the contacts that the refinement finds among 30k stress pairs, the whole call 811 and 749.
#define OGX_INLINE_LEAVES
#include "ogx_kernels.cuh"

namespace ogx {

// EPA at full capacity over the spill list: contacts that ran out of the small working
// set, and -- certified, every face plane from FP64, exact supports -- contacts whose FP32
// expansion met an inconsistent horizon or stopped short of the FP32 rounding level; or
// (late != 0) over the contacts the FP64 refinement found, all certified.  One warp per
// contact, points read from memory (any body size).
template <bool kPosed>
__global__ void __launch_bounds__(128, 4) k_epa_spill(DevBatch B, int late) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  EpaMemCert* mem = reinterpret_cast<EpaMemCert*>(smem_raw);
  const WarpTeam<32> t;
  EpaMemCert& M = mem[threadIdx.x / 32];
  const int team = (blockIdx.x * blockDim.x + threadIdx.x) / 32;
  const int nteams = (gridDim.x * blockDim.x) / 32;
  const int cnt = B.counts[late ? kCntSpillLate : kCntSpill];
  Config cfg64 = B.cfg;
  cfg64.flags |= OGX_F_EPA_FP64_PLANES;
  for (int j = team; j < cnt; j += nteams) {
    const int e = late ? B.spill[B.npairs - 1 - j] : B.spill[j];
    if (e & kSpillResume) {  // continue the small pass's saved expansion
      const EpaResume* rs = B.resume + (e & (kSpillResume - 1));
      epa_item<32, 0, true, 0, kPosed>(t, B, B.cfg, rs->pair, M, false, nullptr, rs);
    } else {
      epa_item<32, 0, true, 0, kPosed>(t, B, (e & kSpill64) ? cfg64 : B.cfg, e & ~kSpill64, M, false);
    }
    t.sync();
  }
}

cudaError_t launch_epa_spill(const DevBatch& B, int grid, cudaStream_t st, bool late) {
  if (B.xf)
    k_epa_spill<true><<<grid, 128, 4 * sizeof(EpaMemCert), st>>>(B, late ? 1 : 0);
  else
    k_epa_spill<false><<<grid, 128, 4 * sizeof(EpaMemCert), st>>>(B, late ? 1 : 0);
  return cudaGetLastError();
}

cudaError_t epa_spill_occupancy(int block, int* per_sm) {
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, k_epa_spill<false>, block,
                                                       (block / 32) * sizeof(EpaMemCert));
}

}  // namespace ogx
