// FFT pass kernels of the lengths L with L % 8 == 0.
#include "tr_lines_part.cuh"

namespace tr {
void lp_fill_0(LineKernels* table) { lp_fill_part<0>(table); }
}  // namespace tr
