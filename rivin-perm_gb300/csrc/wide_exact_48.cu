// Instantiations of wide_exact_kernel for row sums below 2^48.
#include "wide_exact.cuh"

namespace pg {

bool wide_entry_48(int n, WideEntry *out) {
    return wide_entry<12, 48>(n, out) || wide_entry<16, 48>(n, out) ||
           wide_entry<18, 48>(n, out) || wide_entry<20, 48>(n, out) ||
           wide_entry<22, 48>(n, out) || wide_entry<24, 48>(n, out) ||
           wide_entry<25, 48>(n, out) || wide_entry<26, 48>(n, out) ||
           wide_entry<28, 48>(n, out) || wide_entry<30, 48>(n, out) ||
           wide_entry<32, 48>(n, out);
}

}  // namespace pg
