// Instantiations of poly_esym_kernel for row sums up to 15.
#include "poly_esym.cuh"

namespace pg {

template <int N>
static bool entry(int n, EsymEntry *out) {
    if (n > N) return false;
    out->layout = esym_layout<N, 15>();
    out->launch = launch_esym<N, 15>;
    return true;
}

bool esym_entry_15(int n, EsymEntry *out) {
    return entry<16>(n, out) || entry<20>(n, out) || entry<25>(n, out) || entry<28>(n, out) ||
           entry<31>(n, out);
}

}  // namespace pg
