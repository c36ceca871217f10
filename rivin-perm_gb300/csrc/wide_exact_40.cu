// Instantiations of wide_exact_kernel for row sums below 2^40.
#include "wide_exact.cuh"

namespace pg {

// Every order from 16 on (and 12, for short walks): a padded row is one more
// factor of the product tree and often one more word of its products.  Odd
// orders against the next even one's shape: 17..29 2 to 10 % faster (27 x 27 of
// 38 bits 7.13 -> 6.65 ms), but 29 below 2^44 31.6 ms against 30.5 and left out.
bool wide_entry_40(int n, WideEntry *out) {
    return wide_entry<12, 40>(n, out) || wide_entry<16, 40>(n, out) || wide_entry<17, 40>(n, out) ||
           wide_entry<18, 40>(n, out) || wide_entry<19, 40>(n, out) || wide_entry<20, 40>(n, out) ||
           wide_entry<21, 40>(n, out) || wide_entry<22, 40>(n, out) || wide_entry<23, 40>(n, out) ||
           wide_entry<24, 40>(n, out) || wide_entry<25, 40>(n, out) || wide_entry<26, 40>(n, out) ||
           wide_entry<27, 40>(n, out) || wide_entry<28, 40>(n, out) || wide_entry<29, 40>(n, out) ||
           wide_entry<30, 40>(n, out) || wide_entry<31, 40>(n, out) || wide_entry<32, 40>(n, out);
}

}  // namespace pg
