"""Kernels launched before their predecessor has finished (grids of up to 444
blocks) read nothing early: runs of many steps, queued without a wait between
them, give the bits of the same steps with an event between any two kernels."""
import ctypes

import numpy as np
import pytest

from oracle.tarang_oracle import backward_2d, forward_2d, rel_l2

pytestmark = pytest.mark.gpu


# smallest grids; one with grids on both sides of 444 blocks; beyond it throughout
@pytest.mark.parametrize("Nx,Nz", [(8, 8), (64, 32), (256, 112), (512, 200)])
@pytest.mark.parametrize("ts", [0, 1, 2, 3])
@pytest.mark.parametrize("precision", ["f64", "mixed"])
def test_chained_steps_match_separated_kernels(tb, Nx, Nz, ts, precision):
    rng = np.random.default_rng(Nx + ts)
    b0 = forward_2d(1e-2 * rng.standard_normal((Nz, Nx)))
    got = []
    for separated in (True, False):
        plan = tb.Plan(tb.ChannelDomain(Nx, Nz, Lx=4.0, Lz=1.0), 1e-3, 1e-3, 1.0, 0.0, ts,
                       precision=tb._lib.TB_PREC_MIXED if precision == "mixed" else tb._lib.TB_PREC_F64)
        plan.set_state(0, b0)
        if separated:  # profiled steps record an event on either side of every kernel
            plan.set_profiling(True)
        plan.step(0.005, 12)
        got.append([plan.get_state(f) for f in (0, 1, 2)])
    for a, b in zip(*got):
        assert np.isfinite(a).all() and np.array_equal(a, b)


# 444 and 448 blocks of the row transforms (two rows of a field a block, four fields)
@pytest.mark.parametrize("Nz", [221, 222, 223])
def test_field_transforms_around_the_limit(tb, Nz):
    import torch

    nf, Nx = 4, 12
    plan = tb.ChannelDomain(Nx, Nz, Lx=4.0, Lz=1.0).transform_plan()
    grid = np.random.default_rng(Nz).standard_normal((nf, Nz, Nx))
    dg = torch.as_tensor(grid, device="cuda")
    dc = torch.empty((nf, Nz, Nx // 2 + 1), dtype=torch.complex128, device="cuda")
    back = torch.empty_like(dg)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    for _ in range(3):
        assert tb.lib.tb_transform_forward(plan.ptr, ptr(dg), ptr(dc), nf) == 0
        assert tb.lib.tb_transform_backward(plan.ptr, ptr(dc), ptr(back), nf) == 0
    for f in range(nf):
        # FP64 transforms: rounding times the growth of a 223-point Chebyshev sum
        assert rel_l2(dc[f].cpu().numpy(), forward_2d(grid[f])) < 1e-13
        assert rel_l2(back[f].cpu().numpy(), backward_2d(forward_2d(grid[f]), Nx)) < 1e-13
