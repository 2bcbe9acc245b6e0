// FFT pass kernels of the lengths L with L % 8 == 1.
#include "tr_lines_part.cuh"

namespace tr {
void lp_fill_1(LineKernels* table) { lp_fill_part<1>(table); }
}  // namespace tr
