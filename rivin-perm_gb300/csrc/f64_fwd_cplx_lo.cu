// Instantiations of glynn_forward_kernel: complex matrices, orders 2..22.
#include "f64_forward.cuh"

namespace pg {

cudaError_t launch_forward_cplx_lo(int n, const FwdArgs &a, cudaStream_t s) {
    switch (n) {
    case 2: return launch_glynn_forward<2, true>(a, s);
    case 3: return launch_glynn_forward<3, true>(a, s);
    case 4: return launch_glynn_forward<4, true>(a, s);
    case 5: return launch_glynn_forward<5, true>(a, s);
    case 6: return launch_glynn_forward<6, true>(a, s);
    case 7: return launch_glynn_forward<7, true>(a, s);
    case 8: return launch_glynn_forward<8, true>(a, s);
    case 9: return launch_glynn_forward<9, true>(a, s);
    case 10: return launch_glynn_forward<10, true>(a, s);
    case 11: return launch_glynn_forward<11, true>(a, s);
    case 12: return launch_glynn_forward<12, true>(a, s);
    case 13: return launch_glynn_forward<13, true>(a, s);
    case 14: return launch_glynn_forward<14, true>(a, s);
    case 15: return launch_glynn_forward<15, true>(a, s);
    case 16: return launch_glynn_forward<16, true>(a, s);
    case 17: return launch_glynn_forward<17, true>(a, s);
    case 18: return launch_glynn_forward<18, true>(a, s);
    case 19: return launch_glynn_forward<19, true>(a, s);
    case 20: return launch_glynn_forward<20, true>(a, s);
    case 21: return launch_glynn_forward<21, true>(a, s);
    case 22: return launch_glynn_forward<22, true>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
