// The transmission records' VJP kernel (dual lanes through the layer stack), in
// its own translation unit: it takes most of the derivative kernels' compile
// time.
#include "adjoint.cuh"

namespace wcb {
namespace adj {

void launch_vjp_transmission(const AdjParams& p, cudaStream_t s) {
    if (p.order_count <= 0) return;
    k_vjp_rows<kLanes, 5><<<unsigned((p.order_count + kBlock - 1) / kBlock), kBlock, 0, s>>>(p);
}

}  // namespace adj
}  // namespace wcb
