// Instantiations of glynn_gradient_kernel: orders 2..16.
#include "f64_gradient.cuh"

namespace pg {

template <int N>
static void shape_of(int n, int *lw, int *rmax) {
    if (n == N) {
        *lw = GradShape<N>::LW;
        *rmax = GradShape<N>::RMAX;
    } else if constexpr (N < 32) {
        shape_of<N + 1>(n, lw, rmax);
    }
}
void gradient_shape(int n, int *log_walkers, int *log_range_max) {
    shape_of<2>(n, log_walkers, log_range_max);
}

cudaError_t launch_gradient_lo(int n, const GradArgs &a, cudaStream_t s) {
    switch (n) {
    case 2: return launch_glynn_gradient<2>(a, s);
    case 3: return launch_glynn_gradient<3>(a, s);
    case 4: return launch_glynn_gradient<4>(a, s);
    case 5: return launch_glynn_gradient<5>(a, s);
    case 6: return launch_glynn_gradient<6>(a, s);
    case 7: return launch_glynn_gradient<7>(a, s);
    case 8: return launch_glynn_gradient<8>(a, s);
    case 9: return launch_glynn_gradient<9>(a, s);
    case 10: return launch_glynn_gradient<10>(a, s);
    case 11: return launch_glynn_gradient<11>(a, s);
    case 12: return launch_glynn_gradient<12>(a, s);
    case 13: return launch_glynn_gradient<13>(a, s);
    case 14: return launch_glynn_gradient<14>(a, s);
    case 15: return launch_glynn_gradient<15>(a, s);
    case 16: return launch_glynn_gradient<16>(a, s);
    default: return cudaErrorInvalidValue;
    }
}

}  // namespace pg
