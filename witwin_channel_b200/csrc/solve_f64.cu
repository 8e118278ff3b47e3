// The per-cell kernels in FP64.
#include "launch_components.cuh"

namespace wcb {

template void launch_components<double>(const MainParams&, int, unsigned, int, size_t, cudaStream_t, cudaStream_t,
                                    ComponentEvents*, const DiffractionPlan&);

}  // namespace wcb
