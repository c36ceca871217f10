// Instantiations of wide_exact_kernel for row sums below 2^40.
#include "wide_exact.cuh"

namespace pg {

bool wide_entry_40(int n, WideEntry *out) {
    return wide_entry<12, 40>(n, out) || wide_entry<16, 40>(n, out) ||
           wide_entry<18, 40>(n, out) || wide_entry<20, 40>(n, out) ||
           wide_entry<22, 40>(n, out) || wide_entry<24, 40>(n, out) ||
           wide_entry<25, 40>(n, out) || wide_entry<26, 40>(n, out) ||
           wide_entry<28, 40>(n, out) || wide_entry<30, 40>(n, out) ||
           wide_entry<32, 40>(n, out);
}

}  // namespace pg
