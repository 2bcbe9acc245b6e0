// FFT pass kernels of the lengths L with L % 8 == 7.
#include "tr_lines_part.cuh"

namespace tr {
void lp_fill_7(LineKernels* table) { lp_fill_part<7>(table); }
}  // namespace tr
