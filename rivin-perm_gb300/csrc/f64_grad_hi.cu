// Instantiations of glynn_gradient_kernel: orders 25..32.
#include "f64_gradient.cuh"

namespace pg {

cudaError_t launch_gradient_hi(int n, const GradArgs &a, cudaStream_t s) {
    switch (n) {
    case 25: return launch_glynn_gradient<25>(a, s);
    case 26: return launch_glynn_gradient<26>(a, s);
    case 27: return launch_glynn_gradient<27>(a, s);
    case 28: return launch_glynn_gradient<28>(a, s);
    case 29: return launch_glynn_gradient<29>(a, s);
    case 30: return launch_glynn_gradient<30>(a, s);
    case 31: return launch_glynn_gradient<31>(a, s);
    case 32: return launch_glynn_gradient<32>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
