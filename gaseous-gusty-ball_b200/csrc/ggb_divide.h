// ggb_divide.h — division of a cell or row index by the grid edge N as one
// multiplication.  Plain C++, so that it can be checked on the host.
#pragma once

namespace ggb {

// ceil(2^46 / N): c / N = (c * factor) >> 46 exactly for every index c < 6 N^2 of
// every grid that cs_init takes (N <= 16384).  The factor is too large by less than
// N / 2^46 of itself, which moves the quotient by less than c / 2^46 < 1 / N while
// c N < 6 N^3 < 2^46; c * factor < 6 N 2^46 < 2^63.  (With 2^40 that ends at N = 5680.)
constexpr int kDivShift = 46;
constexpr unsigned long long div_factor(int N) { return ((1ull << kDivShift) + N - 1) / N; }
constexpr int div_by(unsigned c, unsigned long long factor) { return (int)((c * factor) >> kDivShift); }

}  // namespace ggb
