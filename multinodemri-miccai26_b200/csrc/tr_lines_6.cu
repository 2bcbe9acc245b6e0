// FFT pass kernels of the lengths L with L % 8 == 6.
#include "tr_lines_part.cuh"

namespace tr {
void lp_fill_6(LineKernels* table) { lp_fill_part<6>(table); }
}  // namespace tr
