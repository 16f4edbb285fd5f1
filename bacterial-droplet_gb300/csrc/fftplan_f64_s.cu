// fftplan_f64_s.cu — the FFT kernels (fftplan_impl.cuh) of the register kernels' small sizes in FP64.
#define TTSH_FFTPLAN_T double
#define TTSH_FFTPLAN_SMALL true
#include "fftplan_impl.cuh"

namespace ttsh {
TTSH_FFTPLAN_UNIT(fftplan_f64_s, double, TTSH_FFTPLAN_S)
}  // namespace ttsh
