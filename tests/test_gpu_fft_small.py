"""The FP64 FFT kernels of the small sizes 24, 32, 48 against cuFFT, alone and in a batch whose last wave is
partial, and against the register kernels (one launch per axis): the same steps, so the same bits.
Tolerance: that of test_gpu_cufft.py, FP64 1e-12 (relative L2)."""
import numpy as np
import pytest

from conftest import random_state
from test_gpu_cufft import cufft_projection, relerr

pytestmark = pytest.mark.gpu


def step(N, n, kind=2):
    import ttsh
    inp = ttsh.default_input(Nx=N, Ny=N, Nz=N)
    ext = ttsh.default_ext(precision=64, quirks=0, zeta=0.02)
    with ttsh.Sim([inp] * n, [ext] * n) as s:
        s.set_tuning(0, dict(s.tuning()[0], fft_kind=kind))
        for i in range(n):
            st = random_state(N, seed=N + i)
            s.set_state(i, st["phi"], st["P"], st["u"], st["us"], st["ps"])
        s.step(2)
        return [(s.get_state(i), s.get_provisional(i)) for i in range(n)], inp


@pytest.mark.parametrize("n", [1, 5])
@pytest.mark.parametrize("N", [24, 32, 48])
def test_small_sizes(N, n):
    got, inp = step(N, n)
    axes, _ = step(N, n, 0)
    for (g, (us, ps)), (a, _) in zip(got, axes):
        pv, pp = cufft_projection(us, ps, inp.h, inp.dt0)
        assert relerr(g["pv"], pv) <= 1e-12 and relerr(g["pp"], pp) <= 1e-12
        for f in ("phi", "P", "u", "pv", "pp"):
            assert np.array_equal(g[f], a[f]), f
