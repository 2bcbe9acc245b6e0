// FFT pass kernels of the lengths L with L % 8 == 3.
#include "tr_lines_part.cuh"

namespace tr {
void lp_fill_3(LineKernels* table) { lp_fill_part<3>(table); }
}  // namespace tr
