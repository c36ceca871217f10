// Instantiations of wide_exact_kernel for row sums below 2^36.
#include "wide_exact.cuh"

namespace pg {

bool wide_entry_36(int n, WideEntry *out) {
    return wide_entry<12, 36>(n, out) || wide_entry<16, 36>(n, out) ||
           wide_entry<18, 36>(n, out) || wide_entry<20, 36>(n, out) ||
           wide_entry<22, 36>(n, out) || wide_entry<24, 36>(n, out) ||
           wide_entry<25, 36>(n, out) || wide_entry<26, 36>(n, out) ||
           wide_entry<28, 36>(n, out) || wide_entry<30, 36>(n, out) ||
           wide_entry<32, 36>(n, out);
}

}  // namespace pg
