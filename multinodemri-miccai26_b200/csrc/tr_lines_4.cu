// FFT pass kernels of the lengths L with L % 8 == 4.
#include "tr_lines_part.cuh"

namespace tr {
void lp_fill_4(LineKernels* table) { lp_fill_part<4>(table); }
}  // namespace tr
