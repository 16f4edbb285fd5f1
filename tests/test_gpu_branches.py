"""A batch of several sizes runs its size groups as parallel branches of the step graph: the bits of
single-droplet runs, over steps of both parities, with a caller's stream and after a re-capture."""
import numpy as np
import pytest

from conftest import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision,sizes", [(32, (64, 32, 50, 64, 96)), (64, (16, 24, 20, 24))])
def test_branches_equal_single_runs(precision, sizes):
    import torch
    import ttsh
    st = [random_state(N, seed=N + k) for k, N in enumerate(sizes)]

    def run(which, stream=None):
        with ttsh.Sim([ttsh.default_input(Nx=sizes[k], Ny=sizes[k], Nz=sizes[k]) for k in which],
                      [ttsh.default_ext(precision=precision, zeta=0.02, form=ttsh.FORM_PLAIN) for _ in which]) as s:
            if stream is not None:
                s.set_stream(stream.cuda_stream)
            for i, k in enumerate(which):
                s.set_state(i, st[k]["phi"], st[k]["P"], st[k]["u"], st[k]["us"], st[k]["ps"])
            s.step(3)
            s.set_tuning(0, s.tuning()[0])  # captures the graphs again
            s.step(4)
            return [s.get_state(i) for i in range(len(which))]

    batch = run(range(len(sizes)), torch.cuda.Stream())
    for k in range(len(sizes)):
        a = run([k])[0]
        for f in ("phi", "P", "u", "pv", "pp"):
            assert np.array_equal(a[f], batch[k][f]), (sizes[k], f)


@pytest.mark.parametrize("k2_mode", [0, 1])
@pytest.mark.parametrize("precision,form,N", [(64, "PLAIN", 20), (64, "PLAIN", 32), (64, "PLAIN", 64), (32, "PLAIN", 20),
                                              (32, "PLAIN", 32), (32, "FUSED", 32)])
def test_droplets_of_one_size_with_their_own_h(precision, form, N, k2_mode):
    """Droplets of one size that differ in the lattice constant (and the time step) have the bits of
    single-droplet runs: each has the wavenumbers of its own h."""
    import ttsh
    consts = [dict(h=1.0), dict(h=0.7, dt0=0.005), dict(h=1.0), dict(h=1.3)]
    st = random_state(N, seed=N)

    def run(which):
        with ttsh.Sim([ttsh.default_input(Nx=N, Ny=N, Nz=N, **consts[k]) for k in which],
                      [ttsh.default_ext(precision=precision, zeta=0.02, k2_mode=k2_mode, form=getattr(ttsh, "FORM_" + form))
                       for _ in which]) as s:
            for i in range(len(which)):
                s.set_state(i, st["phi"], st["P"], st["u"], st["us"], st["ps"])
            s.step(3)
            return [s.get_state(i) for i in range(len(which))]

    batch = run(range(len(consts)))
    for k in range(len(consts)):
        a = run([k])[0]
        for f in ("phi", "P", "u", "pv", "pp"):
            assert np.array_equal(a[f], batch[k][f]), (k, f)
