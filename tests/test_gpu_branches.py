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
