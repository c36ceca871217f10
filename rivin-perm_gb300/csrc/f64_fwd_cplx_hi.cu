// Instantiations of glynn_forward_kernel: complex matrices, orders 23..32.
#include "f64_forward.cuh"

namespace pg {

cudaError_t launch_forward_cplx_hi(int n, const FwdArgs &a, cudaStream_t s) {
    switch (n) {
    case 23: return launch_glynn_forward<23, true>(a, s);
    case 24: return launch_glynn_forward<24, true>(a, s);
    case 25: return launch_glynn_forward<25, true>(a, s);
    case 26: return launch_glynn_forward<26, true>(a, s);
    case 27: return launch_glynn_forward<27, true>(a, s);
    case 28: return launch_glynn_forward<28, true>(a, s);
    case 29: return launch_glynn_forward<29, true>(a, s);
    case 30: return launch_glynn_forward<30, true>(a, s);
    case 31: return launch_glynn_forward<31, true>(a, s);
    case 32: return launch_glynn_forward<32, true>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
