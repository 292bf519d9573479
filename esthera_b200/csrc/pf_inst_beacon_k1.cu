// Kernel instantiations: the fused sample+weight+sort kernel for the beacon (range-only unicycle) model.
#define PF_PART_K1
#include "pf_launch_impl.cuh"
#include "pf_host.cuh"
namespace pfdev {
template cudaError_t Launch<Beacon>::sample_sort(int, int, int, bool, int, cudaStream_t, const FilterDesc*, const int2*, InputRef, bool);
}  // namespace pfdev
// the model registers itself here (once for the library)
PF_REGISTER_MODEL(pfdev::Beacon, PF_MODEL_BEACON, pf_beacon_params, "beacon");
