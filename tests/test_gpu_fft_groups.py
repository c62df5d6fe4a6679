"""The column-group and row-pair transforms of the turbulence and 3D programs at
the sizes where their dispatch changes: every group width (kx columns a block),
partial last groups, the shortest and longest rows, radix-3 lengths."""
import numpy as np
import pytest

from oracle.tarang_oracle import (RBC3D, TABLEAUS, RBC3Params, rbc3_initial_b, rel_l2, run_turb, run_turb_rk, turb_forward,
                                  turb_initial_spec)

pytestmark = pytest.mark.gpu


# kx columns 5 .. 1025 against 1, 2 and 4 a block; padded lengths 12 .. 3072; the
# last two exceed three blocks an SM in the y and in the x transforms
@pytest.mark.parametrize("Nx,Ny", [(8, 8), (8, 64), (12, 16), (108, 72), (256, 48), (512, 32), (1024, 16), (2048, 8),
                                   (16, 2048), (972, 12), (2048, 256), (512, 1152)])
@pytest.mark.parametrize("scheme", ["SBDF2", "RK222", "RK443"])
def test_turbulence_sizes_match_oracle(tb, scheme, Nx, Ny):
    ts = {"RK222": tb._lib.TB_RK222, "RK443": tb._lib.TB_RK443, "SBDF2": tb._lib.TB_SBDF2}[scheme]
    rng = np.random.default_rng(Nx + Ny)
    # white noise (Nyquist rows and columns too), of unit size
    q0 = turb_forward(rng.standard_normal((Ny, Nx)))
    nu, dt, n = 1e-3, 0.05 / max(Nx, Ny), 2
    run = (lambda: run_turb(q0, Nx, 2 * np.pi, 2 * np.pi, nu, dt, n)) if scheme == "SBDF2" else (
        lambda: run_turb_rk(q0, Nx, 2 * np.pi, 2 * np.pi, nu, dt, n, scheme))
    t = tb.Turb2D(Nx, Ny, nu, q0, timestepper=ts)
    t.step(dt, n)
    # FP32 state: 6e-8 a rounding, a few tens of them a step
    assert rel_l2(t.vorticity(), run()) < 1e-5


def test_turbulence_state_round_trip(tb):
    # the state copies transpose and convert on the device: exactly the FP32 rounding
    for Nx, Ny in ((8, 12), (64, 36), (96, 256)):
        q = turb_initial_spec(Nx, Ny, seed=3)
        t = tb.Turb2D(Nx, Ny, 1e-3, q)
        want = q.astype(np.complex64).astype(np.complex128)
        assert np.array_equal(t.vorticity(), want)
        t.set_vorticity(2.0 * q)
        assert np.array_equal(t.vorticity(), (2.0 * q).astype(np.complex64).astype(np.complex128))


# (Nx, Ny, Nz): kx groups with remainders, x rows of 12 .. 768 points, y columns
# long enough that fewer columns fit a block
@pytest.mark.parametrize("Nx,Ny,Nz", [(8, 8, 8), (8, 16, 10), (24, 12, 8), (36, 8, 8), (512, 8, 8), (8, 512, 8)])
@pytest.mark.parametrize("rows", [1, 2, 4])
def test_rbc3d_mixed_groups_match_oracle(tb, rows, Nx, Ny, Nz):
    _rbc3d(tb, Nx, Ny, Nz, rows, tb._lib.TB_PREC_MIXED, 1e-6)


@pytest.mark.parametrize("Nx,Ny,Nz", [(8, 8, 8), (24, 12, 8), (36, 8, 8), (256, 8, 8), (8, 256, 8)])
@pytest.mark.parametrize("rows", [1, 2])
def test_rbc3d_f64_groups_match_oracle(tb, rows, Nx, Ny, Nz):
    _rbc3d(tb, Nx, Ny, Nz, rows, tb._lib.TB_PREC_F64, 1e-10)


def _rbc3d(tb, Nx, Ny, Nz, rows, precision, bar):
    p = RBC3Params(Nx=Nx, Ny=Ny, Nz=Nz, Ra=1e5)
    plan = tb.Plan3D(Nx, Ny, Nz, p.kappa, p.nu, 0, p.Lx, p.Ly, 1.0, precision=precision)
    try:
        plan.set_variant(0, rows)
    except tb.TarangError:
        pytest.skip("rows do not divide or fit at this size")
    plan.set_state(tb._lib.TB_FIELD_B, plan.forward(rbc3_initial_b(p, 7, amp=1e-2)))
    plan.step(0.01, 2)
    sim = RBC3D(p)
    sim.set_b_grid(rbc3_initial_b(p, 7, amp=1e-2))
    for _ in range(2):
        sim.step_rk(0.01, TABLEAUS["RK222"])
    for f, want in ((0, sim.b), (1, sim.ux), (5, sim.uy), (2, sim.uz)):
        assert rel_l2(plan.get_state(f), want) < bar
