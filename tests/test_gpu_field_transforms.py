"""Field transforms through the device-pointer calls: several fields a launch
(chunks of six), rows in pairs (odd row counts, the mid-plane row of odd Nz)."""
import ctypes

import numpy as np
import pytest

from oracle.tarang_oracle import backward_2d, forward_2d, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Nz", [(8, 8), (12, 9), (48, 17), (64, 33), (512, 129)])
@pytest.mark.parametrize("nf", [1, 2, 6, 7, 13])
def test_fields_match_oracle(tb, Nx, Nz, nf):
    import torch

    if nf > 7 and Nx > 64:
        pytest.skip("one large size per chunk count is enough")
    plan = tb.ChannelDomain(Nx, Nz, Lx=4.0, Lz=1.0).transform_plan()
    rng = np.random.default_rng(nf)
    grid = rng.standard_normal((nf, Nz, Nx))
    want = np.stack([forward_2d(g) for g in grid])
    dg = torch.as_tensor(grid, device="cuda")
    dc = torch.empty((nf, Nz, Nx // 2 + 1), dtype=torch.complex128, device="cuda")
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    assert tb.lib.tb_transform_forward(plan.ptr, ptr(dg), ptr(dc), nf) == 0
    got = dc.cpu().numpy()
    for g, w in zip(got, want):
        assert rel_l2(g, w) < 1e-13
    # coefficients with Im at DC and Nyquist, which the backward transform ignores
    coeff = want + 1j * rng.standard_normal(want.shape)
    dc.copy_(torch.as_tensor(coeff))
    back = torch.empty_like(dg)
    assert tb.lib.tb_transform_backward(plan.ptr, ptr(dc), ptr(back), nf) == 0
    for g, c in zip(back.cpu().numpy(), coeff):
        assert rel_l2(g, backward_2d(c, Nx)) < 1e-13
