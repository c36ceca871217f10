// Instantiations of wide_exact_kernel for row sums below 2^36.
#include "wide_exact.cuh"

namespace pg {

// Every order from 16 on (and 12, for short walks): a padded row is one more
// factor of the product tree and often one more word of its products.  Odd
// orders against the next even one's shape: 17..29 2 to 10 % faster (27 x 27 of
// 38 bits 7.13 -> 6.65 ms), but 29 below 2^44 31.6 ms against 30.5 and left out.
bool wide_entry_36(int n, WideEntry *out) {
    return wide_entry<12, 36>(n, out) || wide_entry<16, 36>(n, out) || wide_entry<17, 36>(n, out) ||
           wide_entry<18, 36>(n, out) || wide_entry<19, 36>(n, out) || wide_entry<20, 36>(n, out) ||
           wide_entry<21, 36>(n, out) || wide_entry<22, 36>(n, out) || wide_entry<23, 36>(n, out) ||
           wide_entry<24, 36>(n, out) || wide_entry<25, 36>(n, out) || wide_entry<26, 36>(n, out) ||
           wide_entry<27, 36>(n, out) || wide_entry<28, 36>(n, out) || wide_entry<29, 36>(n, out) ||
           wide_entry<30, 36>(n, out) || wide_entry<31, 36>(n, out) || wide_entry<32, 36>(n, out);
}

}  // namespace pg
