"""The dense form of small tau systems as a setting: reported, settable, kept by a
plan's own variant and by the tuners, with dynamic walls and in stacked plans."""
import numpy as np
import pytest

from oracle.tarang_oracle import RBCParams, forward_2d, rbc_initial_b, rel_l2, run_rbc

pytestmark = pytest.mark.gpu


def make(tb, Nx, Nz, ts=0, kappa=1e-3, nu=1e-3, seed=42):
    plan = tb.Plan(tb.ChannelDomain(Nx, Nz, Lx=4.0, Lz=1.0), kappa, nu, 1.0, 0.0, ts)
    plan.set_state(0, forward_2d(rbc_initial_b(RBCParams(Nx=Nx, Nz=Nz), seed, amp=1e-1)))
    return plan


def state(plan):
    return [plan.get_state(f) for f in (0, 1, 2)]


# band rows 2 Nz up to 156, inverses of all modes up to 40 MiB
@pytest.mark.parametrize("Nx,Nz,dense", [(12, 8, True), (12, 78, True), (12, 79, False), (192, 76, True), (216, 76, False),
                                         (512, 48, True), (576, 48, False)])
def test_default_form(tb, Nx, Nz, dense):
    plan = make(tb, Nx, Nz)
    nk = Nx // 2 + 1
    n = 2 * Nz
    assert dense == (n + 4 <= 160 and nk * 2 * (n + 4) * ((n + 7) // 4 * 4) * 8 <= 40 << 20)
    assert plan.solve_form() == dense
    if n + 4 > 160:
        with pytest.raises(tb.TarangError):
            plan.set_solve_form(True)
    else:
        plan.set_solve_form(not dense)
        assert plan.solve_form() != dense


@pytest.mark.parametrize("Nx,Nz", [(12, 8), (64, 32), (64, 64), (1536, 8)])
def test_own_variant_changes_nothing(tb, Nx, Nz):
    want = make(tb, Nx, Nz)
    want.step(0.01, 2)
    plan = make(tb, Nx, Nz)
    plan.set_variant(*plan.variant())
    assert plan.solve_form()
    plan.step(0.01, 2)
    for a, b in zip(state(plan), state(want)):
        assert np.array_equal(a, b)
    # another value: partitioned; back again only by the form
    parts = plan.variant()[0]
    plan.set_variant(tau_parts=1 if parts != 1 else 4)
    assert not plan.solve_form()
    plan.set_variant(tau_parts=parts)
    assert not plan.solve_form() and plan.variant()[0] == parts
    plan.set_solve_form(True)
    assert plan.solve_form() and plan.variant()[0] == parts


@pytest.mark.parametrize("Nz,parts", [(24, 4), (64, 8), (64, 4), (64, 1), (76, 16)])
@pytest.mark.parametrize("scheme,ts", [("RK443", 1), ("SBDF2", 3)])
def test_forms_match_oracle(tb, scheme, ts, Nz, parts):
    p = RBCParams(Nx=48, Nz=Nz, Lx=4.0, Lz=1.0, Ra=1e8)
    sim = run_rbc(p, scheme, 0.01, 5, seed=42)
    for dense in (True, False):
        plan = tb.Plan(tb.ChannelDomain(48, Nz, Lx=4.0, Lz=1.0), p.kappa, p.nu, 1.0, 0.0, ts)
        plan.set_variant(tau_parts=parts)
        plan.set_solve_form(dense)
        assert plan.solve_form() == dense and plan.variant()[0] == parts
        plan.set_state(0, forward_2d(rbc_initial_b(p, 42)))
        plan.step(0.01, 5)
        for got, want in zip(state(plan), (sim.b, sim.ux, sim.uz)):
            # FP64 direct solves: rounding times a condition below 1e5
            assert rel_l2(got, want) < 1e-10


def test_tuned_variant_on_a_fresh_plan(tb):
    plan = make(tb, 64, 32)
    chosen = plan.tune(0.01, trial_steps=2)
    assert plan.solve_form() and chosen == plan.variant()
    other = make(tb, 64, 32)
    other.set_variant(*chosen)
    assert other.solve_form()
    plan.step(0.01, 3)
    other.step(0.01, 3)
    for a, b in zip(state(plan), state(other)):
        assert np.array_equal(a, b)


def test_dynamic_walls(tb):
    Nx, Nz = 32, 16
    rng = np.random.default_rng(1)
    nk = Nx // 2 + 1
    walls = [rng.standard_normal((2, nk)) + 1j * rng.standard_normal((2, nk)) for _ in range(2)]
    out = []
    for dense in (True, False):
        plan = make(tb, Nx, Nz)
        plan.set_solve_form(dense)
        plan.set_wall_values(0, *walls[0])
        plan.set_wall_values(1, *walls[1])
        plan.step(0.01, 3)
        out.append(state(plan))
    for a, b in zip(*out):
        assert rel_l2(a, b) < 1e-11  # two direct solves of one system


def test_stacked_plans(tb):
    # equal shapes, own diffusivities: one stacked plan, one inverse a member and mode
    sizes = [(64, 32, 1e-3, 2e-3), (64, 32, 5e-3, 1e-3), (64, 32, 2e-4, 4e-3)]
    plans = [make(tb, Nx, Nz, kappa=k, nu=v, seed=i) for i, (Nx, Nz, k, v) in enumerate(sizes)]
    ens = tb.Ensemble(plans)
    ens.set_form(True)
    ens.run(0.01, 3)
    assert ens.form() == (True, 1)
    for i, (Nx, Nz, k, v) in enumerate(sizes):
        alone = make(tb, Nx, Nz, kappa=k, nu=v, seed=i)
        alone.set_solve_form(False)
        alone.step(0.01, 3)
        for a, b in zip(state(plans[i]), state(alone)):
            assert rel_l2(a, b) < 1e-11


def test_ensemble_tune_weighs_the_dense_form(tb):
    plans = [make(tb, 64, 32, seed=i) for i in range(3)] + [make(tb, 64, 96)]
    before = [state(p) for p in plans]
    ens = tb.Ensemble(plans)
    ens.tune(0.01, trial_steps=2)
    assert len({p.variant()[0] for p in plans}) == 1
    assert not plans[3].solve_form() and len({p.solve_form() for p in plans[:3]}) == 1
    for p, want in zip(plans, before):
        for a, b in zip(state(p), want):
            assert np.array_equal(a, b)
    # a lone small member: the inverses take half the time of the sweeps
    lone = make(tb, 256, 64)
    tb.Ensemble([lone]).tune(0.01, trial_steps=8)
    assert lone.solve_form()
