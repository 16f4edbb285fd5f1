"""The diagnostics' velocity kernels (max |D.u|, max |u|, non-finite count) at boxes smaller than a tile,
with partial tiles and several droplets, against numpy on the state read back. D.u is compared at
its own rounding: FP64 1e-12, FP32 1e-5 of max |u| / h (27 terms of relative 6e-8). A NaN or an infinity
anywhere in u or P is counted and leaves the other droplets' diagnostics alone."""
import numpy as np
import pytest

from conftest import random_state

pytestmark = pytest.mark.gpu


def max_div(u, h):
    def s(f, a):
        return np.roll(f, 1, a) + 4 * f + np.roll(f, -1, a)
    d = 0
    for c, ax in enumerate((2, 1, 0)):
        f = np.roll(u[c], -1, ax) - np.roll(u[c], 1, ax)
        for a in range(3):
            f = s(f, a) if a != ax else f
        d = d + f / (72 * h)
    return np.abs(d).max()


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 1e-5)])
@pytest.mark.parametrize("sizes", [(8,), (10, 10, 10), (54, 54), (64,), (100,), (96, 40, 96)])
def test_full_diagnostics(sizes, precision, tol):
    import ttsh
    with ttsh.Sim([ttsh.default_input(Nx=N, Ny=N, Nz=N) for N in sizes],
                  [ttsh.default_ext(precision=precision, zeta=0.02) for _ in sizes]) as s:
        for k, N in enumerate(sizes):
            st = random_state(N, seed=N + k)
            s.set_state(k, st["phi"], st["P"], st["u"], st["us"], st["ps"])
        s.step(1)
        got = s.reduce_all()
        for k, g in enumerate(got):
            u = s.get_state(k)["u"]
            assert abs(g["max_abs_u"] - np.abs(u).max()) <= 1e-7 * np.abs(u).max()
            assert abs(g["max_div_u"] - max_div(u, 1.0)) <= tol * np.abs(u).max()
            assert g["nonfinite"] == 0


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("field,value", [("u", np.nan), ("P", np.inf), ("u", -np.inf)])
def test_nonfinite_is_counted(precision, field, value):
    import ttsh
    N = 36
    with ttsh.Sim([ttsh.default_input(Nx=N, Ny=N, Nz=N)] * 2, [ttsh.default_ext(precision=precision)] * 2) as s:
        for k in range(2):
            st = random_state(N, seed=k)
            if k:
                st[field] = st[field].copy()
                st[field][2, N - 1, 0, N - 1] = value
            s.set_state(k, st["phi"], st["P"], st["u"])
        a, b = s.reduce_all(check=False)
    assert a["nonfinite"] == 0 and b["nonfinite"] == 1
    assert np.isfinite(a["max_div_u"]) and not np.isnan(b["max_div_u"]) and not np.isnan(b["max_abs_u"])
