"""The fused stage kernels of the 2D steppers where a grid round trip drops part
of the state: Im of the DC and Nyquist columns is nonzero, so L X carries the
correction of every equation plane (continuity rows included) and the multistep
M X its projection."""
import numpy as np
import pytest

from oracle.tarang_oracle import RBC2D, RBCParams, forward_2d, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme,ts", [("RK222", 0), ("RK443", 1), ("SBDF1", 2), ("SBDF2", 3)])
# (8, 801): the final update's columns pass the default shared-memory limit
@pytest.mark.parametrize("Nx,Nz", [(8, 8), (24, 17), (256, 9), (288, 8), (8, 801)])
def test_complex_edge_columns_match_oracle(tb, scheme, ts, Nx, Nz):
    p = RBCParams(Nx=Nx, Nz=Nz, Ra=1e4)
    rng = np.random.default_rng(Nx + Nz)
    decay = np.exp(-0.3 * np.arange(Nz))[:, None]
    # smooth in z, white along x, complex everywhere (DC and Nyquist too)
    fields = [decay * (rng.standard_normal((Nz, Nx // 2 + 1)) + 1j * rng.standard_normal((Nz, Nx // 2 + 1)))
              for _ in range(3)]
    fields[0] += forward_2d(np.broadcast_to(1.0 - 0.5 * (1 - np.cos(np.pi * np.arange(Nz) / (Nz - 1)))[:, None], (Nz, Nx)))
    sim = RBC2D(p)
    sim.b[:], sim.ux[:], sim.uz[:] = fields
    plan = tb.Plan(tb.ChannelDomain(Nx, Nz, Lx=p.Lx, Lz=p.Lz), p.kappa, p.nu, p.Lz, 0.0, ts)
    for f, a in enumerate(fields):
        plan.set_state(f, a)
    for _ in range(3):
        sim.step(0.005, scheme)
    plan.step(0.005, 3)
    for f, want in ((0, sim.b), (1, sim.ux), (2, sim.uz)):
        # FP64 solves of systems with condition below 1e5: 1e-10 as the step parity tests
        assert rel_l2(plan.get_state(f), want) < 1e-10
    if scheme.startswith("SBDF"):
        assert rel_l2(plan.get_state(3), sim.pr) < 1e-10
    else:
        assert not plan.get_state(3).any() and not plan.get_state(4).any()
