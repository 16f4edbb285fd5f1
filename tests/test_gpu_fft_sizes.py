"""The FFT for any size (fft.cu) against cuFFT at sizes that take one step (9, 10, 15), two (18 .. 250:
every radix of dft.cuh, every stage pair of the FP32 form) and three (270, 320), with lines per CTA that
fill partial warps; and its launch forms (x and y of a plane in one launch, one launch per axis,
explicit lines per CTA), which give the same bits. Tolerances: those of test_gpu_cufft.py, FP64 1e-12,
FP32 2e-5 (relative L2)."""
import numpy as np
import pytest

from conftest import random_state
from test_gpu_cufft import cufft_projection, relerr

pytestmark = pytest.mark.gpu


def _factors(n):
    return [p for p in range(2, n + 1) if n % p == 0 and all(p % q for q in range(2, p))]


def projection(N, precision, steps=1, cfg=None):
    import ttsh
    st = random_state(N, seed=N + 3)
    inp = ttsh.default_input(Nx=N, Ny=N, Nz=N)
    ext = ttsh.default_ext(precision=precision, quirks=0, zeta=0.02, form=ttsh.FORM_PLAIN)
    with ttsh.Sim(inp, ext) as s:
        if cfg:
            s.set_tuning(0, dict(s.tuning()[0], **cfg))
        s.set_state(0, st["phi"], st["P"], st["u"], st["us"], st["ps"])
        s.step(steps)
        return s.get_state(0), s.get_provisional(0), inp


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-5)])
@pytest.mark.parametrize("N", [9, 10, 15, 18, 20, 25, 27, 30, 36, 45, 54, 60, 72, 75, 80, 81, 90, 100, 108, 120, 135, 144, 150,
                               162, 200, 225, 240, 250, 270, 320])
def test_any_size_matches_cufft(N, precision, tol):
    if N % 2 and precision == 32:
        pytest.skip("odd N: the reference's wavenumbers are not symmetric, so the scaling of the packed source shows")
    g, (us, ps), inp = projection(N, precision)
    pv, pp = cufft_projection(us, ps, inp.h, inp.dt0)
    assert relerr(g["pv"], pv) <= tol, relerr(g["pv"], pv)
    assert relerr(g["pp"], pp) <= tol, relerr(g["pp"], pp)


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N", [10, 50, 90, 100, 120, 144])
def test_launch_forms_give_the_same_bits(N, precision):
    lb = next(b for b in (16, 8, 4, 2, 1) if N % b == 0)
    want = projection(N, precision, 2)[0]
    for cfg in ({"fft_kind": 0}, {"fft_kind": 1}, {"fft_kind": 1, "fft_lb": lb}, {"fft_kind": 2, "fft_lb": 1}):
        got = projection(N, precision, 2, cfg)[0]
        for f in ("phi", "P", "u", "pv", "pp"):
            assert np.array_equal(got[f], want[f]), (cfg, f)


# every size with kernels of its own (the products of 2, 3 and 5 up to 270 without a register kernel)
PLAN_SIZES = [n for n in range(9, 271) if n not in (8, 16, 24, 32, 48, 64, 96, 128, 160, 192, 256)
              and all(p in (2, 3, 5) for p in _factors(n))]


@pytest.mark.parametrize("precision", [64, 32])
def test_per_size_kernels_equal_the_any_size_kernel(precision):
    """One solve of a random source by the kernels built for a size and by the kernel for any size (one
    launch per axis): the same bits."""
    import ttsh
    rng = np.random.default_rng(0)
    for N in PLAN_SIZES:
        u, P = rng.standard_normal((2, 3, N, N, N)) * 0.01
        phi = rng.random((N, N, N))
        out = []
        for kind in (2, 1):
            with ttsh.Sim(ttsh.default_input(Nx=N, Ny=N, Nz=N), ttsh.default_ext(precision=precision, form=ttsh.FORM_PLAIN)) as s:
                s.set_tuning(0, dict(s.tuning()[0], fft_kind=kind))
                s.set_state(0, phi, P, u)
                s.step(1)
                out.append(s.get_state(0))
        for f in ("pv", "pp", "u", "P"):
            assert np.array_equal(out[0][f], out[1][f]), (N, f)


@pytest.mark.parametrize("N,n", [(8, 100), (18, 5), (25, 2), (27, 2), (48, 6), (64, 3)])
def test_few_and_many_line_groups_give_the_same_bits(N, n):
    """FP32, one launch per axis: a single droplet's few line groups go through shared memory stage by stage, those of a
    batch of n as every size's; with the default lines per CTA, one line, and the reverse plan."""
    import ttsh
    st = random_state(N, seed=N)

    def run(n, cfg):
        with ttsh.Sim([ttsh.default_input(Nx=N, Ny=N, Nz=N)] * n, [ttsh.default_ext(precision=32, zeta=0.02, form=ttsh.FORM_PLAIN)] * n) as s:
            t = s.tuning()[0]
            s.set_tuning(0, dict(t, fft_kind=1, **({"radix": t["radix"][::-1]} if cfg == "reverse" else {"fft_lb": cfg})))
            for k in range(n):
                s.set_state(k, st["phi"], st["P"], st["u"], st["us"], st["ps"])
            s.step(2)
            return s.get_state(n - 1)

    for cfg in (0, 1, "reverse"):
        a, b = run(1, cfg), run(n, cfg)
        for f in ("phi", "P", "u", "pv", "pp"):
            assert np.array_equal(a[f], b[f]), (cfg, f)


@pytest.mark.parametrize("precision,N,cfg,launches", [(32, 50, {}, 7), (32, 50, {"fft_lb": 2}, 9), (32, 50, {"radix": [5, 5, 2]}, 9),
                                                      (64, 50, {}, 7), (64, 50, {"fft_lb": 2}, 9), (64, 50, {"radix": [5, 5, 2]}, 7),
                                                      (32, 64, {"fft_lb": 2}, 7), (64, 64, {"fft_lb": 2}, 7)])
def test_explicit_choices_go_per_axis(precision, N, cfg, launches):
    """fft_kind 2: an explicit choice of lines (and in FP32 of the plan) is run one launch per axis at the sizes without
    register kernels, the defaults by plane; the same bits."""
    import ttsh
    inp, ext = ttsh.default_input(Nx=N, Ny=N, Nz=N), ttsh.default_ext(precision=precision, form=ttsh.FORM_PLAIN)
    with ttsh.Sim(inp, ext) as s:
        s.set_tuning(0, dict(s.tuning()[0], **cfg))
        assert s.launches_per_step() == launches
    if "radix" not in cfg:
        got, want = projection(N, precision, 2, cfg)[0], projection(N, precision, 2)[0]
        for f in ("phi", "P", "u", "pv", "pp"):
            assert np.array_equal(got[f], want[f]), f


# ---- large boxes: one step from white noise, made on the GPU and handed over in page-locked arrays ----
LARGE = 576  # the largest box below


@pytest.fixture(scope="module")
def noise():
    import torch
    g = torch.Generator(device="cuda").manual_seed(1)
    host = torch.empty(4 * LARGE ** 3, dtype=torch.float64, pin_memory=True)
    for part in host.split(LARGE ** 3):
        part.copy_(torch.rand(part.numel(), generator=g, device="cuda", dtype=torch.float64).sub_(0.5).mul_(0.02))
    torch.cuda.empty_cache()
    return host.numpy()


def solve(noise, N, precision, cfg, provisional=False):
    """Pressures (and u*, P*) of one step."""
    import torch
    import ttsh
    n = N ** 3
    pinned = lambda *shape: torch.empty(shape, dtype=torch.float64, pin_memory=True).numpy()
    with ttsh.Sim(ttsh.default_input(Nx=N, Ny=N, Nz=N), ttsh.default_ext(precision=precision, quirks=0, form=ttsh.FORM_PLAIN)) as s:
        s.set_tuning(0, dict(s.tuning()[0], **cfg))
        s.set_state(0, noise[:n].reshape(N, N, N), noise[n:].reshape(-1)[:3 * n].reshape(3, N, N, N), noise[:3 * n].reshape(3, N, N, N))
        s.step(1)
        out = [pinned(N, N, N), pinned(N, N, N)]
        ttsh._check(ttsh.lib().ttsh_get_state(s.handle, 0, None, None, None, ttsh._p(out[0]), ttsh._p(out[1])))
        if provisional:
            out += [pinned(3, N, N, N), pinned(3, N, N, N)]
            ttsh._check(ttsh.lib().ttsh_get_provisional(s.handle, 0, ttsh._p(out[2]), ttsh._p(out[3])))
        return out


def against_cufft(out, tol):
    import torch
    import ttsh
    inp = ttsh.default_input()
    for got, want in zip(out, cufft_projection(out[2], out[3], inp.h, inp.dt0)):
        assert relerr(got, want) <= tol, relerr(got, want)
    torch.cuda.empty_cache()


@pytest.mark.parametrize("precision", [64, 32])
@pytest.mark.parametrize("N", [n for n in range(271, 501) if all(p in (2, 3, 5) for p in _factors(n))])
def test_large_per_size_kernels_equal_the_any_size_kernel(noise, N, precision):
    """The sizes above 270 with kernels of their own: the bits of the kernel for any size."""
    for a, b in zip(*(solve(noise, N, precision, {"fft_kind": kind}) for kind in (2, 1))):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("precision,tol", [(64, 1e-12), (32, 2e-5)])
@pytest.mark.parametrize("N", [540, 576])
def test_any_size_kernel_above_500(noise, N, precision, tol):
    """Sizes without kernels of their own: the plane launches with the default lines per CTA against cuFFT, one launch
    per axis and one line per CTA the same bits."""
    want = solve(noise, N, precision, {}, True)
    against_cufft(want, tol)
    for cfg in ({"fft_kind": 1}, {"fft_lb": 1}):
        for a, b in zip(solve(noise, N, precision, cfg), want):
            assert np.array_equal(a, b), cfg


@pytest.mark.parametrize("N", [64, 96, 128, 160, 192, 256, 512])
def test_fp64_register_kernels_match_cufft(noise, N):
    """The FP64 register kernels, x and y of a plane in one launch, against cuFFT; per axis the same bits."""
    want = solve(noise, N, 64, {}, True)
    against_cufft(want, 1e-12)
    for a, b in zip(solve(noise, N, 64, {"fft_kind": 0}), want):
        assert np.array_equal(a, b)
