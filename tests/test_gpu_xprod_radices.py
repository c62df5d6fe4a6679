"""Row products of the advection right-hand side at every kind of transform
plan the in-place form (x-products form 3) takes: one to four passes, each
radix from 2 to 16, last passes of 2, 3, 4, 6 and 8, both CTA sizes, the
longest row, odd Nz (the mid-plane row is its own mirror)."""
import numpy as np
import pytest

from oracle.tarang_oracle import RBC2D, RBCParams, forward_2d, rel_l2

pytestmark = pytest.mark.gpu

SIZES = [(8, 9), (12, 8), (16, 8), (24, 8), (36, 9), (48, 8), (96, 8), (108, 8), (128, 8), (216, 9), (256, 8),
         (324, 8), (384, 8), (512, 9), (648, 8), (768, 8), (972, 8), (1024, 8), (1152, 8), (1536, 8), (1944, 8),
         (2048, 8)]


@pytest.mark.parametrize("mixed", [False, True])
@pytest.mark.parametrize("Nx,Nz", SIZES)
def test_products_match_oracle(tb, Nx, Nz, mixed):
    L = tb._lib
    p = RBCParams(Nx=Nx, Nz=Nz, Ra=1e5)
    dom = tb.ChannelDomain(Nx, Nz, Lx=p.Lx, Lz=p.Lz)
    plan = tb.Plan(dom, p.kappa, p.nu, p.Lz, 0.0, L.TB_RK222,
                   precision=L.TB_PREC_MIXED if mixed else L.TB_PREC_F64)
    plan.set_variant(0, 3)
    rng = np.random.default_rng(Nx + Nz)
    # white noise reaches every bin, the Nyquist fold and split among them
    c = [forward_2d(rng.standard_normal((Nz, Nx))) for _ in range(3)]
    want = RBC2D(p).rhs(*c)
    got = plan.rhs_advection(*c)
    for g, w in zip(got, want):
        # FP64: rounding of log2(M) butterfly levels and an Nz-term product sum,
        # well under 1e-13; FP32 the same in units of 6e-8
        assert rel_l2(g, w) < (2e-6 if mixed else 1e-13)


@pytest.mark.parametrize("mixed", [False, True])
def test_forms_agree(tb, mixed):
    """The three x-products forms on one grid (stacked passes, ping-pong, in place)."""
    L = tb._lib
    Nx, Nz = 288, 17
    dom = tb.ChannelDomain(Nx, Nz, Lx=4.0, Lz=1.0)
    plan = tb.Plan(dom, 1e-3, 1e-3, 1.0, 0.0, L.TB_RK222, precision=L.TB_PREC_MIXED if mixed else L.TB_PREC_F64)
    rng = np.random.default_rng(5)
    c = [forward_2d(rng.standard_normal((Nz, Nx))) for _ in range(3)]
    out = []
    for form in (1, 2, 3):
        plan.set_variant(0, form)
        out.append(plan.rhs_advection(*c))
    for other in out[:2]:
        for g, w in zip(out[2], other):
            assert rel_l2(g, w) < (2e-6 if mixed else 1e-13)
