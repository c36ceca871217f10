// Instantiations of glynn_gradient_kernel: orders 17..24.
#include "f64_gradient.cuh"

namespace pg {

cudaError_t launch_gradient_mid(int n, const GradArgs &a, cudaStream_t s) {
    switch (n) {
    case 17: return launch_glynn_gradient<17>(a, s);
    case 18: return launch_glynn_gradient<18>(a, s);
    case 19: return launch_glynn_gradient<19>(a, s);
    case 20: return launch_glynn_gradient<20>(a, s);
    case 21: return launch_glynn_gradient<21>(a, s);
    case 22: return launch_glynn_gradient<22>(a, s);
    case 23: return launch_glynn_gradient<23>(a, s);
    case 24: return launch_glynn_gradient<24>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
