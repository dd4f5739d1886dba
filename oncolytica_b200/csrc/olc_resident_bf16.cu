// The resident field kernel on OLC_FIELD_BF16 storage.
#include "olc_resident16.cuh"

namespace olc {
template cudaError_t launch_resident16<OLC_FIELD_BF16>(int, const ResidentArgs&, const ResidentPlan&, cudaStream_t);
}  // namespace olc
