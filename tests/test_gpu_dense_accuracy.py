"""The dense inverses of small systems give the solution to within the rounding
of its right-hand side: one SBDF1 step from rest against the tau systems solved
in 40 digits."""
import numpy as np
import pytest

from oracle.tarang_oracle import RBC2D, RBCParams, forward_2d, rbc_initial_b, rel_l2

pytestmark = pytest.mark.gpu


def solve_mp(A, b):
    """A x = b by elimination with row pivoting in 40 digits (A, b of FP64 numbers and their sums)."""
    import mpmath

    n = len(b)
    rows = [[A[i][j] for j in range(n)] + [b[i]] for i in range(n)]
    for j in range(n):
        p = max(range(j, n), key=lambda i: abs(rows[i][j]))
        rows[j], rows[p] = rows[p], rows[j]
        top = rows[j]
        nz = [c for c in range(j + 1, n + 1) if top[c] != 0]
        for i in range(j + 1, n):
            if rows[i][j] != 0:
                f = rows[i][j] / top[j]
                for c in nz:
                    rows[i][c] -= f * top[c]
    x = [mpmath.mpc(0)] * n
    for i in range(n - 1, -1, -1):
        x[i] = (rows[i][n] - sum(rows[i][c] * x[c] for c in range(i + 1, n))) / rows[i][i]
    return np.array([complex(v) for v in x])


@pytest.mark.parametrize("Nz,Ra,dt", [(9, 1e7, 0.02), (16, 1e8, 0.01)])
def test_solution_within_rounding(tb, Nz, Ra, dt):
    import mpmath

    mpmath.mp.dps = 40
    p = RBCParams(Nx=12, Nz=Nz, Lx=4.0, Lz=1.0, Ra=Ra)
    b0 = forward_2d(rbc_initial_b(p, 42, amp=1e-1))
    plan = tb.Plan(tb.ChannelDomain(12, Nz, Lx=4.0, Lz=1.0), p.kappa, p.nu, 1.0, 0.0, tb._lib.TB_SBDF1)
    plan.set_state(0, b0)
    plan.step(dt, 1)  # u = 0: no advection, so the step is one solve of (M / dt + L) x = M b / dt
    got = [plan.get_state(f) for f in (3, 0, 1, 2)]  # p, b, u_x, u_z
    sim = RBC2D(p)
    want = [np.zeros_like(b0) for _ in range(4)]
    for m in (0, 1, 4):
        M, L, _, algf = sim.dense_mode_matrices(m)
        n = len(M)
        a = mpmath.mpf(1.0 / dt)
        mp = lambda z: mpmath.mpc(z.real, z.imag)  # noqa: E731
        A = [[a * mp(complex(M[i, j])) + mp(complex(L[i, j])) for j in range(n)] for i in range(n)]
        rhs = [a * sum((mp(complex(M[i, Nz + k])) * mp(complex(b0[k, m])) for k in range(Nz) if M[i, Nz + k] != 0),
                       mpmath.mpc(0)) + mp(complex(algf[i])) for i in range(n)]
        x = solve_mp(A, rhs)
        for f in range(4):
            want[f][:, m] = x[f * Nz:(f + 1) * Nz]
    for g, w in zip(got, want):
        # the right-hand side (three products a row), the inverse's entries and the
        # product with it are each within a few roundings of 1.1e-16
        assert rel_l2(g[:, [0, 1, 4]], w[:, [0, 1, 4]]) < 1e-15
