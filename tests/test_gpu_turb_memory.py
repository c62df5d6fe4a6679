"""Turbulence plans hold the spectra that a server charges a request for."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_spectra_held_as_charged(tb):
    import torch

    L = tb._lib
    N = 1024
    q0 = np.zeros((N, N // 2 + 1), complex)
    spec = (N // 2 + 1) * N * 8
    grain = 2 << 20  # cudaMalloc's unit for buffers of this size
    held, charged = {}, {}
    for ts in (L.TB_SBDF2, L.TB_RK222, L.TB_RK443):
        server = tb.Server(1 << 30)
        server.submit(tb.turb_desc(N, N, 1e-3, timestepper=ts), 1e-3, 1, q0)
        server.wait_all()
        charged[ts] = server.stats()["peak_bytes"]
        server.close()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        plan = tb.Turb2D(N, N, 1e-3, q0, timestepper=ts)
        held[ts] = before - torch.cuda.mem_get_info()[0]
        del plan
    unit = (spec + grain - 1) // grain * grain
    for ts in (L.TB_RK222, L.TB_RK443):
        assert round((held[ts] - held[L.TB_SBDF2]) / unit) == round((charged[ts] - charged[L.TB_SBDF2]) / spec)
