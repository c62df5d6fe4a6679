"""A step at a new time step (factors, partition responses, step graph) on the
default plan of a large grid costs no more than with one-warp solves, which need
no responses."""
import time

import numpy as np
import pytest

from oracle.tarang_oracle import RBCParams, forward_2d, rbc_initial_b

pytestmark = pytest.mark.gpu


def new_dt_seconds(tb, parts):
    import torch

    p = RBCParams(Nx=1536, Nz=384, Ra=1e8)
    plan = tb.Plan(tb.ChannelDomain(1536, 384, Lx=p.Lx, Lz=p.Lz), p.kappa, p.nu, p.Lz, 0.0, tb._lib.TB_RK222)
    if parts:
        plan.set_variant(tau_parts=parts)
    plan.set_state(0, forward_2d(rbc_initial_b(p, 42, amp=1e-2)))
    best = np.inf
    for i in range(12):
        torch.cuda.synchronize()
        t = time.perf_counter()
        plan.step(1e-3 * (1 + 1e-3 * i), 1)
        torch.cuda.synchronize()
        best = min(best, time.perf_counter() - t) if i >= 3 else best
    return best, plan.variant()[0]


def test_first_step_at_a_new_dt(tb):
    t, parts = new_dt_seconds(tb, 0)
    assert parts > 1
    one, _ = new_dt_seconds(tb, 1)
    # measured 1.02 (2.34 ms against 2.30); 1.24 while the responses took 0.78 ms
    assert t < 1.12 * one, (t, one)
