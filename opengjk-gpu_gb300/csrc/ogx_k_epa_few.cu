// ogx_k_epa_few.cu -- EPA bucket kernels of small and medium batches, one per bucket: a warp per
// contact where the bucket has few of them, teams of 8 (bodies above 512 points: 16) lanes
// where it has many.  Both read the bodies from memory on every support scan.
#include "ogx_kernels.cuh"

namespace ogx {

static const KernelInfo kVar[kBuckets] = {
    {k_epa_few<8>, 8, 4 << kOccShift}, {k_epa_few<8>, 8, 4 << kOccShift},  {k_epa_few<8>, 8, 4 << kOccShift},
    {k_epa_few<8>, 8, 4 << kOccShift}, {k_epa_few<8>, 8, 4 << kOccShift},  {k_epa_few<8>, 8, 4 << kOccShift},
    {k_epa_few<16>, 16, 4 << kOccShift},
};

void few_variants(const KernelInfo** epa) { *epa = kVar; }

}  // namespace ogx
