// FFT pass kernels of the lengths L with L % 8 == 5.
#include "tr_lines_part.cuh"

namespace tr {
void lp_fill_5(LineKernels* table) { lp_fill_part<5>(table); }
}  // namespace tr
