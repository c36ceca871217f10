// Instantiations of wide_exact_kernel for row sums below 2^44.
#include "wide_exact.cuh"

namespace pg {

bool wide_entry_44(int n, WideEntry *out) {
    return wide_entry<12, 44>(n, out) || wide_entry<16, 44>(n, out) ||
           wide_entry<18, 44>(n, out) || wide_entry<20, 44>(n, out) ||
           wide_entry<22, 44>(n, out) || wide_entry<24, 44>(n, out) ||
           wide_entry<25, 44>(n, out) || wide_entry<26, 44>(n, out) ||
           wide_entry<28, 44>(n, out) || wide_entry<30, 44>(n, out) ||
           wide_entry<32, 44>(n, out);
}

}  // namespace pg
