"""3D plans: the partitions a new plan starts with can be set and are among the
tuner's (its decoupled velocity component, with half the rows, is not
partitioned and sets no limit)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("Nx,Nz", [(24, 64), (24, 80), (24, 96), (12, 100)])
def test_reported_variant_is_accepted(tb, Nx, Nz):
    plan = tb.Plan3D(Nx, Nx, Nz, 1e-3, 1e-3, 0, 4.0, 4.0, 1.0)
    parts, rows = plan.variant()
    assert parts == 8
    plan.set_variant(tau_parts=4)
    plan.set_variant(parts, rows)
    assert plan.variant() == (parts, rows)
    if Nz >= 80:  # 16 windows of 12 padded rows
        plan.set_variant(tau_parts=16)
    else:
        with pytest.raises(tb.TarangError):
            plan.set_variant(tau_parts=16)


def test_partitions_agree(tb):
    rng = np.random.default_rng(2)
    b = 0.1 * rng.standard_normal((64, 24, 24))
    out = []
    for parts in (8, 4, 1):
        plan = tb.Plan3D(24, 24, 64, 1e-3, 1e-3, 0, 4.0, 4.0, 1.0)
        plan.set_variant(tau_parts=parts)
        plan.set_state(0, plan.forward(b))
        plan.step(0.01, 2)
        out.append([plan.get_state(f) for f in (0, 1, 2)])
    for o in out[1:]:
        for x, y in zip(o, out[0]):
            # partitions change the rounding of the sweeps, not the solution
            assert np.linalg.norm(x - y) <= 1e-11 * np.linalg.norm(y)
