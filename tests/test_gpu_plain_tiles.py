"""The FP64 form's tiled kernels at the sizes where a tile, its halo or the last row of tiles can go
wrong: boxes smaller than a tile (8, 10, 12), tile widths that are no multiple of a warp (18, 30, 50,
54), boxes cut into partial last tiles, several instances per launch, and the terms behind a switch
(active stress, A, the stale halo). FP64 against the CPU oracle: 1e-11 relative L2, the tolerance of
the other FP64 tests (a few hundred roundings of 1.1e-16 and the 1/dt of the pressure source). A batch
gives the bits of single droplets."""
import numpy as np
import pytest

from conftest import random_state
from test_gpu_parity import FP64_TOL, relerr, run_gpu, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [8, 10, 12, 18, 30, 36, 50, 54])
@pytest.mark.parametrize("stale,zeta,A", [(1, 0.0, 0.0), (0, 0.02, 0.3)])
def test_fp64_tiles_match_oracle(oracle_mod, N, stale, zeta, A):
    st = random_state(N, seed=N)
    g = run_gpu(st, 3, 64, 0, stale, zeta, A=A)
    o = run_oracle(oracle_mod, st, 3, 0, stale, zeta, A=A)
    errs = {k: relerr(g[k], o[k]) for k in ("phi", "P", "u", "pv", "pp", "us", "ps")}
    assert max(errs.values()) <= FP64_TOL, errs


def test_fp64_batch_equals_single():
    import ttsh
    sizes = (54, 90, 54, 10)
    st = [random_state(N, seed=N + k) for k, N in enumerate(sizes)]

    def run(which):
        with ttsh.Sim([ttsh.default_input(Nx=sizes[k], Ny=sizes[k], Nz=sizes[k]) for k in which],
                      [ttsh.default_ext(precision=64, zeta=0.02) for _ in which]) as s:
            for i, k in enumerate(which):
                s.set_state(i, st[k]["phi"], st[k]["P"], st[k]["u"], st[k]["us"], st[k]["ps"])
            s.step(3)
            return [s.get_state(i) for i in range(len(which))]

    batch = run(range(len(sizes)))
    for k, b in enumerate(batch):
        a = run([k])[0]
        for f in ("phi", "P", "u", "pv", "pp"):
            assert np.array_equal(a[f], b[f]), (sizes[k], f)
