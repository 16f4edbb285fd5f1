"""The FP32 plain form's marching kernels at boxes smaller than a tile (8, 10), with partial tiles and a
last chunk of planes shorter than the others (18, 50, 54, 100), several droplets per launch and every
switch, against the FP64 form after 3 steps: 1e-5 relative L2 (a few tens of roundings of 6e-8 per field
value; the source of the pressures is not nearly solenoidal here). A batch gives the bits of single
droplets."""
import numpy as np
import pytest

from conftest import random_state
from test_gpu_parity import relerr, run_gpu

pytestmark = pytest.mark.gpu



@pytest.mark.parametrize("N", [8, 10, 18, 50, 54, 100])
@pytest.mark.parametrize("stale,zeta,A", [(1, 0.0, 0.0), (0, 0.02, 0.3)])
def test_fp32_matches_fp64(N, stale, zeta, A):
    st = random_state(N, seed=N)
    a = run_gpu(st, 3, 64, 0, stale, zeta, A=A)
    b = run_gpu(st, 3, 32, 0, stale, zeta, A=A)
    errs = {k: relerr(b[k], a[k]) for k in ("phi", "P", "u", "pv", "pp", "us", "ps")}
    assert max(errs.values()) <= 1e-5, errs


def test_fp32_batch_equals_single():
    import ttsh
    out = []
    for sizes in ((54, 90, 54, 10), (54,), (90,)):
        with ttsh.Sim([ttsh.default_input(Nx=N, Ny=N, Nz=N) for N in sizes],
                      [ttsh.default_ext(precision=32, zeta=0.02) for _ in sizes]) as s:
            for k, N in enumerate(sizes):
                st = random_state(N, seed=N)
                s.set_state(k, st["phi"], st["P"], st["u"], st["us"], st["ps"])
            s.step(3)
            out.append([s.get_state(k) for k in range(len(sizes))])
    for f in ("phi", "P", "u", "pv", "pp"):
        assert np.array_equal(out[0][0][f], out[1][0][f]) and np.array_equal(out[0][2][f], out[1][0][f]), f
        assert np.array_equal(out[0][1][f], out[2][0][f]), f
