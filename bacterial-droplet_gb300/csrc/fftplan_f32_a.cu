// fftplan_f32_a.cu — the per-size FFT kernels (fftplan_impl.cuh) of a third of the sizes, for float.
#define TTSH_FFTPLAN_T float
#include "fftplan_impl.cuh"

namespace ttsh {
TTSH_FFTPLAN_UNIT(fftplan_f32_a, float, TTSH_FFTPLAN_A)
}  // namespace ttsh
