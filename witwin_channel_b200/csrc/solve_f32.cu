// The per-cell kernels in mixed precision (FP32 traversal and fields).
#include "launch_components.cuh"

namespace wcb {

template void launch_components<float>(const MainParams&, int, unsigned, int, size_t, cudaStream_t, cudaStream_t,
                                    ComponentEvents*, const DiffractionPlan&);

}  // namespace wcb
