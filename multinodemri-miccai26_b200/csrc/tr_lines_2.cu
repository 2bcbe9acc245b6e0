// FFT pass kernels of the lengths L with L % 8 == 2.
#include "tr_lines_part.cuh"

namespace tr {
void lp_fill_2(LineKernels* table) { lp_fill_part<2>(table); }
}  // namespace tr
