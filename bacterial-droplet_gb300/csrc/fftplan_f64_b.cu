// fftplan_f64_b.cu — the per-size FFT kernels (fftplan_impl.cuh) of a third of the sizes, for double.
#define TTSH_FFTPLAN_T double
#include "fftplan_impl.cuh"

namespace ttsh {
TTSH_FFTPLAN_UNIT(fftplan_f64_b, double, TTSH_FFTPLAN_B)
}  // namespace ttsh
