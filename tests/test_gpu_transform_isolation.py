"""Fields transformed in one call do not reach one another: odd row counts,
neighbours of very different size, infinities and NaN next door."""
import ctypes

import numpy as np
import pytest

from oracle.tarang_oracle import forward_2d, rel_l2

pytestmark = pytest.mark.gpu


def forward(tb, plan, grid):
    import torch

    nf, Nz, Nx = grid.shape
    dg = torch.as_tensor(grid, device="cuda")
    dc = torch.empty((nf, Nz, Nx // 2 + 1), dtype=torch.complex128, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert tb.lib.tb_transform_forward(plan.ptr, ptr(dg), ptr(dc), nf) == 0
    return dc.cpu().numpy()


@pytest.mark.parametrize("Nx,Nz", [(12, 9), (64, 33), (512, 129), (48, 16)])
@pytest.mark.parametrize("nf", [2, 7])
def test_fields_of_very_different_size(tb, Nx, Nz, nf):
    plan = tb.ChannelDomain(Nx, Nz, Lx=4.0, Lz=1.0).transform_plan()
    grid = np.random.default_rng(Nx).standard_normal((nf, Nz, Nx))
    grid[::2] *= 1e12
    for got, g in zip(forward(tb, plan, grid), grid):
        # FP64 rounding of each field alone, as tests of equal fields
        assert rel_l2(got, forward_2d(g)) < 1e-13


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("Nx,Nz", [(12, 9), (64, 33), (48, 16)])
def test_nan_and_inf_stay_in_their_field(tb, Nx, Nz, bad):
    plan = tb.ChannelDomain(Nx, Nz, Lx=4.0, Lz=1.0).transform_plan()
    grid = np.random.default_rng(Nz).standard_normal((3, Nz, Nx))
    want = forward(tb, plan, grid)
    grid[0, -1, 3] = grid[2, 0, 5] = bad  # the rows next to field 1
    assert np.array_equal(forward(tb, plan, grid)[1], want[1])


def test_checkpoint_load_keeps_fields_apart(tb):
    Nx, Nz = 64, 33
    plan = tb.Plan(tb.ChannelDomain(Nx, Nz, Lx=4.0, Lz=1.0), 1e-3, 1e-3, 1.0, 0.0, tb._lib.TB_RK222)
    grid = np.random.default_rng(3).standard_normal((4, Nz, Nx)) * np.array([1e12, 1.0, 1e12, 1.0])[:, None, None]
    data = np.ascontiguousarray(grid)
    clock = (ctypes.c_double * 3)(0.0, 0.0, 0.0)
    tb._lib.check(tb.lib.tb_checkpoint_load(plan.ptr, data.ctypes.data_as(ctypes.c_void_p), tb._lib.TB_HOST, clock),
                  plan.ctx)
    for f in range(4):
        assert rel_l2(plan.get_state(f), forward_2d(grid[f])) < 1e-13
