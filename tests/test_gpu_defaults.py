"""The schedules a group starts with (fused_default_zc) change nothing: the same bits as one chunk
per tile column, at sizes whose default chunk is a single plane (32), a few planes (32 x 8, 64), does
not divide N (160: the last chunk is shorter) and is at its cap."""
import numpy as np
import pytest

from conftest import random_state

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sizes", [(32,), (32,) * 8, (64,), (160,), (96,) * 9])
def test_default_schedule_is_bit_exact(sizes):
    import ttsh
    N = sizes[0]
    out = []
    for one_chunk in (False, True):
        with ttsh.Sim([ttsh.default_input(Nx=N, Ny=N, Nz=N)] * len(sizes),
                      [ttsh.default_ext(precision=32, zeta=0.02)] * len(sizes)) as s:
            if one_chunk:
                s.set_tuning(0, dict(s.tuning()[0], zc=[0, N, N]))
            else:
                assert all(0 < z <= N for z in s.tuning()[0]["zc"][1:])
            for k in range(len(sizes)):
                st = random_state(N, seed=3 + k % 2)
                s.set_state(k, st["phi"], st["P"], st["u"], st["us"], st["ps"])
            s.step(3)
            out.append([s.get_state(k) for k in (0, len(sizes) - 1)])
    for a, b in zip(*out):
        for f in ("phi", "P", "u", "pv", "pp"):
            assert np.array_equal(a[f], b[f]), f


@pytest.mark.parametrize("sizes,chunked", [((32,) * 3, True), ((32,) * 8, True), ((64,), True), ((160,), True), ((128,), False),
                                           ((64,) * 20, False), ((64, 32), False)])
def test_fused_rhs_default_follows_the_chunk_length(sizes, chunked):
    """fused_rhs starts in one wave of chunks wherever these are at most three planes longer than the
    persistent grid's shares, whatever the share; a batch of several sizes keeps the persistent grid."""
    import torch
    import ttsh
    if torch.cuda.get_device_properties(0).multi_processor_count != 152:
        pytest.skip("the lengths are those of 152 SMs")
    with ttsh.Sim([ttsh.default_input(Nx=N, Ny=N, Nz=N) for N in sizes], [ttsh.default_ext(precision=32) for _ in sizes]) as s:
        assert (s.tuning()[0]["zc"][0] > 0) == chunked, s.tuning()[0]["zc"]
