"""Tau solves of small systems by their dense inverses: at the edges of the lane
blocks (n + 4 = 32, 64, 96, 128, 160 with n = 2 Nz band rows), the largest
system that takes them and the first that does not, against the oracle and the
banded solve of the same plan."""
import numpy as np
import pytest

from oracle.tarang_oracle import RBCParams, forward_2d, rbc_initial_b, rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nz", [8, 13, 14, 15, 30, 31, 46, 47, 62, 63, 76, 77, 78, 79])
@pytest.mark.parametrize("scheme,ts", [("RK222", 0), ("SBDF2", 3)])
def test_dense_and_banded_solves_match_oracle(tb, scheme, ts, Nz):
    p = RBCParams(Nx=12, Nz=Nz, Ra=1e6)
    b0 = forward_2d(rbc_initial_b(p, 42, amp=1e-2))
    sim = run_rbc_amp(p, scheme, 0.02, 3)
    got = {}
    for parts in (0, 1):  # 0: the plan's own choice, 1: one warp per mode group
        plan = tb.Plan(tb.ChannelDomain(12, Nz, Lx=p.Lx, Lz=p.Lz), p.kappa, p.nu, p.Lz, 0.0, ts)
        if parts:
            plan.set_variant(tau_parts=parts)
        plan.set_state(0, b0)
        plan.step(0.02, 3)
        got[parts] = [plan.get_state(f) for f in (0, 1, 2)]
        for g, want in zip(got[parts], (sim.b, sim.ux, sim.uz)):
            # FP64 direct solves: rounding times a condition below 1e5
            assert rel_l2(g, want) < 1e-10
    for g, w in zip(got[0], got[1]):
        assert rel_l2(g, w) < 1e-11


def run_rbc_amp(p, scheme, dt, n):
    from oracle.tarang_oracle import RBC2D

    sim = RBC2D(p)
    sim.set_b_grid(rbc_initial_b(p, 42, amp=1e-2))
    for _ in range(n):
        sim.step(dt, scheme)
    return sim
