"""Timed cases of the library's paths, each called as a user's program calls it.

A case is a dict of plain values; `kind` selects the path:

  channel    2D Rayleigh-Benard steps: state in (device), n steps, state out
  channel3d  the same in 3D
  turbulence FP32 doubly periodic vorticity: n steps, vorticity out (host)
  transform  grid <-> coefficient transforms of whole fields (device buffers)
  ensemble   uneven channel members stepped together

`exact` restates each path in 64 bits with dense per-mode solves and plain
FFTs, and shares no code with the library.
"""
from __future__ import annotations

import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

DEVICE = "cuda" if torch.cuda.is_available() else "cpu"
LX, LZ = 4.0, 1.0  # box of the channel problems (ChannelDomain(Nx, Nz; Lx=4.0, Lz=1.0))


def _package():
    """The package directory's name holds a dot, so it is loaded by path."""
    if "tarang_b200" not in sys.modules:
        root = os.path.join(os.getcwd(), "tarang.jl_b200")
        spec = importlib.util.spec_from_file_location("tarang_b200", os.path.join(root, "__init__.py"),
                                                      submodule_search_locations=[root])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["tarang_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["tarang_b200"]


# ---------------------------------------------------------------------------
# The cases
# ---------------------------------------------------------------------------


def _channel(name, Nx, Nz, scheme, steps, mixed=False, tuned=False, Ra=1e7):
    return dict(name=name, kind="channel", Nx=Nx, Nz=Nz, scheme=scheme, steps=steps, mixed=mixed, tuned=tuned, Ra=Ra)


def _channel3d(name, Nx, Ny, Nz, scheme, steps, mixed, Ra=1e7):
    return dict(name=name, kind="channel3d", Nx=Nx, Ny=Ny, Nz=Nz, scheme=scheme, steps=steps, mixed=mixed, Ra=Ra)


def _turbulence(name, Nx, Ny, scheme, steps):
    return dict(name=name, kind="turbulence", Nx=Nx, Ny=Ny, scheme=scheme, steps=steps)


def listed():
    return [
        # a solver coupled to a host program that owns the fields (the Julia
        # extension): one small step per call, all latency
        _channel("channel_128x32_rk222", 128, 32, "RK222", 1, Ra=1e6),
        # the quick-start script: ChannelDomain(256, 64), run! between callbacks
        _channel("channel_256x64_rk222_run", 256, 64, "RK222", 20, Ra=2e6),
        # the headline benchmark's step, on a plan tuned as its loop tunes it
        _channel("channel_1024x256_rk443", 1024, 256, "RK443", 1, tuned=True, Ra=1e8),
        # the same step in mixed precision
        _channel("channel_1024x256_rk443_mixed", 1024, 256, "RK443", 1, mixed=True, tuned=True, Ra=1e8),
        # a multistep run on a grid of odd Nz and a radix-3 length
        _channel("channel_768x193_sbdf2_run", 768, 193, "SBDF2", 10),
        # a large production channel on the plan a script gets by default
        _channel("channel_1536x384_rk222", 1536, 384, "RK222", 1, Ra=1e9),
        # a small 3D box, as a convergence study or a test runs it
        _channel3d("channel3d_64x64x32_rk222", 64, 64, 32, "RK222", 1, False),
        # the 3D benchmark's step
        _channel3d("channel3d_256x256x128_mixed", 256, 256, 128, "RK222", 1, True),
        # decaying turbulence between two outputs: small and launch-bound, and
        # large with the costlier stepper
        _turbulence("turbulence_256_sbdf2_run", 256, 256, "SBDF2", 100),
        _turbulence("turbulence_1024_rk443_run", 1024, 1024, "RK443", 10),
        # field["g"] / field["c"] of four fields (analysis, checkpoints), odd Nz
        dict(name="transform_512x129", kind="transform", Nx=512, Nz=129, fields=4),
        # an ensemble of uneven members (sizes 128x32 to 512x128), fused form
        dict(name="ensemble_12", kind="ensemble", members=12, steps=10),
    ]


def _smooth(rng, lo, hi):
    """A 2^a 3^b whose 3/2 multiple is even (the lengths the transforms take) near a log-uniform draw."""
    x = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    sizes = [2 ** a * 3 ** b for a in range(2, 12) for b in range(0, 7) if lo <= 2 ** a * 3 ** b <= hi]
    return min(sizes, key=lambda n: (abs(math.log(n / x)), n))


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channel"] * 5 + ["channel3d"] * 2 + ["turbulence"] * 2 + ["transform", "ensemble"])
    Ra = 10.0 ** rng.uniform(6.0, 8.0)
    if kind == "channel":
        Nx, Nz = _smooth(rng, 96, 1536), _logint(rng, 24, 384)
        scheme = rng.choice(["RK222", "RK443", "SBDF1", "SBDF2"])
        return dict(kind=kind, Nx=Nx, Nz=Nz, scheme=scheme, steps=_logint(rng, 1, 20), mixed=rng.random() < 0.35,
                    tuned=rng.random() < 0.25, Ra=Ra)
    if kind == "channel3d":
        return dict(kind=kind, Nx=_smooth(rng, 24, 128), Ny=_smooth(rng, 24, 128), Nz=2 * _logint(rng, 8, 48),
                    scheme=rng.choice(["RK222", "RK443", "SBDF2"]), steps=rng.randint(1, 3), mixed=rng.random() < 0.5,
                    Ra=Ra)
    if kind == "turbulence":
        return dict(kind=kind, Nx=_smooth(rng, 96, 1024), Ny=_smooth(rng, 96, 1024),
                    scheme=rng.choice(["SBDF2", "RK222", "RK443"]), steps=_logint(rng, 5, 40))
    if kind == "transform":
        return dict(kind=kind, Nx=_smooth(rng, 96, 1536), Nz=_logint(rng, 24, 384), fields=rng.randint(1, 4))
    return dict(kind=kind, members=rng.randint(4, 12), steps=rng.randint(2, 10))


def _members(case):
    """(Nx, Nz, Ra, Pr) of an ensemble: the four sizes of the ensemble benchmark in turn."""
    sizes = ((128, 32), (256, 64), (384, 96), (512, 128))
    return [(*sizes[i % 4], 10.0 ** (5.0 + 3.0 * ((7 * i) % 12) / 11.0), 0.7 + 6.3 * ((5 * i) % 12) / 11.0)
            for i in range(case["members"])]


def _dt(case):
    if case["kind"] == "turbulence":
        return 0.4 / max(case["Nx"], case["Ny"])
    if case["kind"] == "ensemble":
        return 0.01
    return min(0.02, 4.0 / max(case["Nx"], case.get("Ny", 0)))


_TS = {"RK222": 0, "RK443": 1, "SBDF1": 2, "SBDF2": 3}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _cheb(N):
    """(forward, backward) Chebyshev matrices on z_j = (1 - cos(pi j/(N-1)))/2."""
    n = torch.arange(N, dtype=torch.float64, device=DEVICE)
    c = torch.cos(torch.remainder(torch.outer(n, n), 2 * (N - 1)) * (math.pi / (N - 1)))
    sign = 1.0 - 2.0 * torch.remainder(n, 2)
    end = torch.ones_like(n)
    end[0] = end[-1] = 0.5
    fwd = (2.0 / (N - 1)) * (end * sign)[:, None] * c * end[None, :]
    return fwd, c.T * sign[None, :]


def _to_coeff(g):
    """Grid (..., Nz, Ny, Nx) -> coefficients: rfft along x, fft along y, Chebyshev along z."""
    c = torch.fft.rfft(g, dim=-1)
    if g.shape[-2] > 1:
        c = torch.fft.fft(c, dim=-2)
    fwd, _ = _cheb(g.shape[-3])
    return torch.einsum("nz,...zyk->...nyk", fwd.to(c.dtype), c)


def _to_grid(c, Nx):
    _, bwd = _cheb(c.shape[-3])
    g = torch.einsum("zn,...nyk->...zyk", bwd.to(c.dtype), c)
    if c.shape[-2] > 1:
        g = torch.fft.ifft(g, dim=-2)
    g = g.clone()
    g[..., 0].imag.zero_()
    g[..., Nx // 2].imag.zero_()
    return torch.fft.irfft(g, n=Nx, dim=-1)


def _wavenumbers(Nx, Ny, Lx, Ly):
    kx = (2 * math.pi / Lx) * torch.arange(Nx // 2 + 1, dtype=torch.float64, device=DEVICE)
    iy = torch.arange(Ny, dtype=torch.float64, device=DEVICE)
    ky = (2 * math.pi / Ly) * torch.where(iy < Ny / 2, iy, iy - Ny) if Ny > 1 else torch.zeros_like(iy)
    return kx, ky


def _planform(gen, count, Nx, Ny, Lx, Ly):
    """Random horizontal functions with a decaying spectrum (unit RMS) and their
    x and y derivatives, (count, Ny, Nx) each."""
    kx, ky = _wavenumbers(Nx, Ny, Lx, Ly)
    re, im = torch.randn((2, count, Ny, Nx // 2 + 1), generator=gen, dtype=torch.float64).to(DEVICE)
    k = torch.sqrt(kx[None, :] ** 2 + ky[:, None] ** 2)
    top = (2 * math.pi / Lx) * Nx / 3
    a = torch.complex(re, im) * torch.where((k > 0) & (k <= top), (1.0 + (k / 6.0) ** 2) ** -1.5, torch.zeros_like(k))
    a[..., 0] = 0.0
    grid = lambda s: torch.fft.irfft(torch.fft.ifft(s, dim=-2) if Ny > 1 else s, n=Nx, dim=-1)  # noqa: E731
    f = grid(a)
    scale = 1.0 / f.square().mean(dim=(-2, -1), keepdim=True).sqrt()
    return f * scale, grid(1j * kx[None, :] * a) * scale, grid(1j * ky[:, None] * a) * scale


def _channel_fields(seed, Nx, Ny, Nz, ndim):
    """Coefficients (fields, Nz, Ny, Nx/2+1) of b, the velocity and p: a
    conductive profile with thermal plumes, and a solenoidal no-slip velocity
    with several vertical scales."""
    gen = torch.Generator().manual_seed(seed)
    terms = 4
    f, fx, fy = _planform(gen, 3 * terms, Nx, Ny, LX, LX)
    z = 0.5 * (1.0 - torch.cos(math.pi * torch.arange(Nz, dtype=torch.float64, device=DEVICE) / (Nz - 1)))
    col = lambda v: v[:, None, None]  # noqa: E731
    b = col(LZ - z) * torch.ones((1, Ny, Nx), dtype=torch.float64, device=DEVICE)
    u = torch.zeros((3, Nz, Ny, Nx), dtype=torch.float64, device=DEVICE)
    for m in range(terms):
        w = (m + 1) * math.pi
        s, c = torch.sin(w * z), torch.cos(w * z)
        hat = 16.0 * (z * (1 - z)) ** 2
        phi, dphi = 0.05 / (m + 1) * hat * c, 0.05 / (m + 1) * (32.0 * z * (1 - z) * (1 - 2 * z) * c - w * hat * s)
        i, j, k = 3 * m, 3 * m + 1, 3 * m + 2
        b = b + col(0.1 / (m + 1) * s) * f[i]
        # u = curl(phi S1, phi S2, 0): the S2 part alone is the 2D stream function
        u[0] -= col(dphi) * f[j]
        u[2] += col(phi) * fx[j]
        if ndim == 3:
            u[1] += col(dphi) * f[k]
            u[2] -= col(phi) * fy[k]
    comps = [b, u[0], u[1], u[2]] if ndim == 3 else [b, u[0], u[2]]
    return _to_coeff(torch.stack(comps + [torch.zeros_like(b)]))


def _turbulence_spec(seed, Nx, Ny):
    """Vorticity coefficients (Ny, Nx/2+1) with a k^-3 energy spectrum, max |q| = 10 on the grid."""
    rng = np.random.default_rng(seed)
    kx = np.arange(Nx // 2 + 1)[None, :]
    ky = np.concatenate([np.arange(Ny // 2), np.arange(-(Ny // 2), 0)])[:, None]
    k = np.sqrt(kx ** 2 + ky ** 2)
    mag = np.where((k >= 1.0) & (k <= min(Nx, Ny) / 3.0), 1.0 / np.maximum(k, 1e-30), 0.0)
    g = np.fft.irfft(np.fft.ifft(mag * np.exp(2j * np.pi * rng.uniform(size=mag.shape)), axis=0), n=Nx, axis=1)
    return np.fft.fft(np.fft.rfft(g * (10.0 / np.abs(g).max()), axis=1), axis=0)


class _Channel:
    """A 2D plan and the device buffers of the program that owns its fields."""

    def __init__(self, seed, Nx, Nz, scheme, mixed, Ra, Pr=1.0):
        tb = _package()
        self.kappa, self.nu = (Ra * Pr) ** -0.5, (Ra / Pr) ** -0.5
        domain = tb.ChannelDomain(Nx, Nz, Lx=LX, Lz=LZ)
        self.plan = tb.Plan(domain, self.kappa, self.nu, LZ, 0.0, _TS[scheme],
                            precision=tb._lib.TB_PREC_MIXED if mixed else tb._lib.TB_PREC_F64)
        self.init = _channel_fields(seed, Nx, 1, Nz, 2).reshape(4, Nz, Nx // 2 + 1).contiguous()
        self.out = torch.empty_like(self.init)
        L = tb._lib
        self.lib, self.check = L.lib, L.check
        self.sel = (ctypes.c_int * 4)(L.TB_FIELD_B, L.TB_FIELD_UX, L.TB_FIELD_UZ, L.TB_FIELD_P)
        ptrs = lambda t: (ctypes.c_void_p * 4)(*[t[i].data_ptr() for i in range(4)])  # noqa: E731
        self.pin, self.pout = ptrs(self.init), ptrs(self.out)
        self.where_in, self.where_out = L.TB_DEVICE | L.TB_NO_WAIT, L.TB_DEVICE
        self.multistep = scheme.startswith("SBDF")
        torch.cuda.synchronize()
        if self.multistep:
            self.write()

    def write(self):
        self.check(self.lib.tb_set_states(self.plan.ptr, 4, self.sel, self.pin, self.where_in), self.plan.ctx)

    def read(self):
        self.check(self.lib.tb_get_states(self.plan.ptr, 4, self.sel, self.pout, self.where_out), self.plan.ctx)
        return dict(zip(("b", "ux", "uz", "p"), self.out))


class _Channel3D:
    def __init__(self, case, seed):
        tb = _package()
        L = tb._lib
        kappa = case["Ra"] ** -0.5
        self.plan = tb.Plan3D(case["Nx"], case["Ny"], case["Nz"], kappa, kappa, _TS[case["scheme"]], LX, LX, LZ,
                              precision=L.TB_PREC_MIXED if case["mixed"] else L.TB_PREC_F64)
        self.lib, self.check, self.dev = L.lib, L.check, L.TB_DEVICE
        self.init = _channel_fields(seed, case["Nx"], case["Ny"], case["Nz"], 3).contiguous()
        self.out = torch.empty_like(self.init)
        self.sel = (L.TB_FIELD_B, L.TB_FIELD_UX, L.TB_FIELD_UY, L.TB_FIELD_UZ, L.TB_FIELD_P)
        self.multistep = case["scheme"].startswith("SBDF")
        torch.cuda.synchronize()
        if self.multistep:
            self.write()

    def write(self):
        for f, t in zip(self.sel, self.init):
            self.check(self.lib.tb_set_state(self.plan.ptr, f, t.data_ptr(), self.dev), self.plan.ctx)

    def read(self):
        for f, t in zip(self.sel, self.out):
            self.check(self.lib.tb_get_state(self.plan.ptr, f, t.data_ptr(), self.dev), self.plan.ctx)
        return dict(zip(("b", "ux", "uy", "uz", "p"), self.out))


def prepare(case, seed):
    tb = _package()
    kind, state = case["kind"], dict(case=case, dt=_dt(case))
    if kind == "channel":
        sim = _Channel(seed, case["Nx"], case["Nz"], case["scheme"], case["mixed"], case["Ra"])
        if case["tuned"]:
            sim.write()
            sim.plan.tune(state["dt"], 3)  # leaves the state as it was
        state["sim"] = sim
    elif kind == "channel3d":
        state["sim"] = _Channel3D(case, seed)
    elif kind == "turbulence":
        q = _turbulence_spec(seed, case["Nx"], case["Ny"])
        state["sim"] = tb.Turb2D(case["Nx"], case["Ny"], 1e-4, q, timestepper=_TS[case["scheme"]])
    elif kind == "transform":
        Nx, Nz, n = case["Nx"], case["Nz"], case["fields"]
        state["plan"] = tb.ChannelDomain(Nx, Nz, Lx=LX, Lz=LZ).transform_plan()
        coeff = torch.cat([_channel_fields(seed + 7919 * i, Nx, 1, Nz, 2)[:1] for i in range(n)])
        grid = _to_grid(torch.cat([_channel_fields(seed + 7919 * i + 1, Nx, 1, Nz, 2)[1:2] for i in range(n)]), Nx)
        state["coeff"] = coeff.reshape(n, Nz, Nx // 2 + 1).contiguous()
        state["grid"] = grid.reshape(n, Nz, Nx).contiguous()
        state["coeff_out"], state["grid_out"] = torch.empty_like(state["coeff"]), torch.empty_like(state["grid"])
    else:
        sims = [_Channel(seed + 101 * i, Nx, Nz, "RK222", False, Ra, Pr)
                for i, (Nx, Nz, Ra, Pr) in enumerate(_members(case))]
        state["sims"] = sims
        state["ensemble"] = tb.Ensemble([s.plan for s in sims])
        state["ensemble"].set_form(True)
    return state


def run(state):
    case, dt = state["case"], state["dt"]
    kind = case["kind"]
    if kind in ("channel", "channel3d"):
        sim = state["sim"]
        # the owner of the fields writes them before a one-step method's steps;
        # a multistep run continues on the plan's own history
        if not sim.multistep:
            sim.write()
        sim.plan.step_async(dt, case["steps"])
        return sim.read()
    if kind == "turbulence":
        state["sim"].step(dt, case["steps"])
        return state["sim"].vorticity()
    if kind == "transform":
        tb, p = _package(), state["plan"]
        ptr = lambda k: state[k].data_ptr()  # noqa: E731
        tb._lib.check(tb.lib.tb_transform_forward(p.ptr, ptr("grid"), ptr("coeff_out"), case["fields"]), p.ctx)
        tb._lib.check(tb.lib.tb_transform_backward(p.ptr, ptr("coeff"), ptr("grid_out"), case["fields"]), p.ctx)
        return dict(coeff=state["coeff_out"], grid=state["grid_out"])
    for s in state["sims"]:
        s.write()
    state["ensemble"].run(dt, case["steps"])
    return [s.read() for s in state["sims"]]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------


def _channel_work(Nx, Ny, Nz, scheme, steps, ndim):
    """Bytes: the state in and out, and per implicit solve the real banded
    factors of every mode (4 + 1 + 8 numbers a row).  FLOPs: per right-hand
    side the fast transforms of the values and gradients and of the products on
    the 3/2 grid, and the banded solves."""
    solves = {"RK222": 2, "RK443": 3}.get(scheme, 1) * steps
    rhss = {"RK222": 3, "RK443": 4}.get(scheme, 1) * steps
    modes = (Nx // 2 + 1) * Ny
    rows = modes * (ndim + 2) * Nz
    padded = 1.5 ** (ndim - 1) * Nx * Ny * Nz
    inverse, forward = (ndim + 1) * (ndim + 1), ndim + 1
    fft = 2.5 * padded * math.log2(padded / Nz) + 2.5 * Nx * Ny * Nz * math.log2(Nz)
    return dict(bytes=2 * rows * 16.0 + solves * rows * 13 * 8.0,
                flops=rhss * (inverse + forward) * fft + solves * rows * 2 * 2 * 13.0)


def work(case):
    kind = case["kind"]
    if kind in ("channel", "channel3d"):
        ndim = 2 if kind == "channel" else 3
        return _channel_work(case["Nx"], case.get("Ny", 1), case["Nz"], case["scheme"], case["steps"], ndim)
    if kind == "turbulence":
        Nx, Ny = case["Nx"], case["Ny"]
        rhss = {"SBDF2": 1, "RK222": 2, "RK443": 3}[case["scheme"]] * case["steps"]
        coeff, padded = (Nx // 2 + 1) * Ny, 2.25 * Nx * Ny
        # the coefficients in and out of each right-hand side in FP32; 4 inverse and 1 forward transforms
        return dict(bytes=rhss * 2 * coeff * 8.0 + coeff * 16.0, flops=rhss * 5 * 2.5 * padded * math.log2(padded))
    if kind == "transform":
        pts = case["Nx"] * case["Nz"]
        coeff = (case["Nx"] // 2 + 1) * case["Nz"]
        return dict(bytes=2.0 * case["fields"] * (8 * pts + 16 * coeff),
                    flops=2.0 * case["fields"] * 2.5 * pts * math.log2(pts))
    parts = [_channel_work(Nx, 1, Nz, "RK222", case["steps"], 2) for Nx, Nz, _, _ in _members(case)]
    return dict(bytes=sum(p["bytes"] for p in parts), flops=sum(p["flops"] for p in parts))


def tolerance(case):
    """The relative 2-norm error another correct implementation may show."""
    kind = case["kind"]
    if kind == "turbulence":
        return {"rel": 4e-5, "max": 4e-3}
    if kind == "transform":
        return {"rel": 1e-13, "max": 1e-11}
    if case.get("mixed"):
        return {"rel": 1e-5, "max": 1e-3}
    return {"rel": 1e-10, "max": 1e-8}


# ---------------------------------------------------------------------------
# The same passes in 64 bits, written out
# ---------------------------------------------------------------------------

_G = 1.0 - 1.0 / math.sqrt(2.0)
_H = 0.4358665215084590
_TABLEAUS = {  # (explicit, implicit, weights): stage rows first, the update's row last
    "RK222": ([[0, 0, 0], [_G, 0, 0], [_G, 1 - _G, 0]], [[0, 0, 0], [0, _G, 0], [0, 1 - _G, _G]], [0, 1 - _G, _G]),
    "RK443": ([[0, 0, 0, 0], [_H, 0, 0, 0], [0.3212788860285571, 0.3966543747256624, 0, 0],
               [-0.105858296071263, 0.5529291479590279, 0.5529291481122351, 0]],
              [[0, 0, 0, 0], [0, _H, 0, 0], [0, 0.2820667392457805, _H, 0],
               [0, 1.208496649176010, -0.6443631706844688, _H]],
              [0, 1.208496649176010, -0.6443631706844688, _H]),
}


def _dealiased(a, b, dims):
    """3/2-padded product of real grids along dims, the Nyquist bin split on the way up and folded on the way down."""
    def pad(g):
        g = g.to(torch.complex128)
        for d in dims:
            N = g.shape[d]
            M, h = 3 * N // 2, N // 2
            s = torch.fft.fft(g, dim=d).movedim(d, -1)
            p = torch.zeros(s.shape[:-1] + (M,), dtype=s.dtype, device=s.device)
            p[..., :h], p[..., M - h + 1:] = s[..., :h], s[..., h + 1:]
            p[..., h] = p[..., M - h] = 0.5 * s[..., h]
            g = torch.fft.ifft(p.movedim(-1, d), dim=d)
        return g

    r = pad(a) * pad(b)
    for d in dims:
        M = r.shape[d]
        N, h = 2 * M // 3, M // 3
        p = torch.fft.fft(r, dim=d).movedim(d, -1)
        s = torch.cat([p[..., :h], p[..., h:h + 1] + p[..., M - h:M - h + 1], p[..., M - h + 1:]], dim=-1)
        r = torch.fft.ifft(s.movedim(-1, d), dim=d) * (M / N)
    return r.real


class _Boussinesq:
    """The tau-method Boussinesq system with one dense matrix per Fourier mode.

    Unknowns of a mode: b, the velocity, p (Nz each), tau_p, tau_b1, tau_b2,
    tau_u1, tau_u2; equations: continuity, b, momentum (Nz rows each), the
    walls of b and u at z = 0 and Lz, and integ(p) = 0 (tau_p = 0 away from
    the mean mode)."""

    def __init__(self, Nx, Ny, Nz, ndim, kappa, nu):
        self.Nx, self.Ny, self.Nz, self.ndim, self.kappa, self.nu = Nx, Ny, Nz, ndim, kappa, nu
        self.kx, self.ky = _wavenumbers(Nx, Ny, LX, LX)
        j = torch.arange(Nz, dtype=torch.float64, device=DEVICE)
        D = torch.where((j[None, :] > j[:, None]) & (torch.remainder(j[None, :] - j[:, None], 2) == 1), 2 * j[None, :],
                        torch.zeros((), dtype=torch.float64, device=DEVICE))
        D[0] *= 0.5
        self.D = D * (2.0 / LZ)
        self.n = (ndim + 2) * Nz + 1 + 2 * (ndim + 1)
        self.modes = torch.cartesian_prod(torch.arange(Ny, device=DEVICE), torch.arange(Nx // 2 + 1, device=DEVICE))
        self.chunk = max(1, int(2e9 / (16.0 * self.n * self.n)))
        self.lu = {}

    def memory(self):
        return 16.0 * self.n * self.n * len(self.modes)

    def matrix(self, modes, alpha, beta):
        """alpha M + beta L of the given modes, with the wall rows scaled by beta."""
        N, nd, n = self.Nz, self.ndim, self.n
        kx, ky = self.kx[modes[:, 1]], self.ky[modes[:, 0]]
        A = torch.zeros((len(modes), n, n), dtype=torch.complex128, device=DEVICE)
        eye = torch.eye(N, dtype=torch.float64, device=DEVICE)
        col = {f: i * N for i, f in enumerate(["b"] + list("xyz" if nd == 3 else "xz") + ["p"])}
        t0 = (nd + 2) * N
        tau_p, comps = t0, ["b"] + list("xyz" if nd == 3 else "xz")
        tau1 = {f: t0 + 1 + (0 if f == "b" else 2 + "xyz"[:3].index(f) if nd == 3 else 2 + "xz".index(f)) for f in comps}
        tau2 = {f: (t0 + 2 if f == "b" else tau1[f] + nd) for f in comps}
        row = {f: (1 + i) * N for i, f in enumerate(comps)}
        lift = N - 1
        grad = {"x": 1j * kx, "y": 1j * ky}
        for f in comps[1:]:  # continuity
            if f == "z":
                A[:, :N, col[f]:col[f] + N] += beta * self.D
                A[:, lift, tau1[f]] += beta
            else:
                A[:, :N, col[f]:col[f] + N] += beta * grad[f][:, None, None] * eye
        lap = (self.D @ self.D)[None] - (kx * kx + ky * ky)[:, None, None] * eye
        for f in comps:
            r, c, nu = row[f], col[f], self.kappa if f == "b" else self.nu
            A[:, r:r + N, c:c + N] += alpha * eye - beta * nu * lap
            A[:, r:r + N, tau1[f]] -= beta * nu * self.D[:, lift]
            A[:, r + lift, tau2[f]] += beta
            if f == "z":
                A[:, r:r + N, col["p"]:col["p"] + N] += beta * self.D
                A[:, r:r + N, col["b"]:col["b"] + N] -= beta * eye
            elif f != "b":
                A[:, r:r + N, col["p"]:col["p"] + N] += beta * grad[f][:, None, None] * eye
        deg = torch.arange(N, device=DEVICE)
        for i, f in enumerate(comps):
            A[:, t0 + i, col[f]:col[f] + N] = beta * (1.0 - 2.0 * (deg % 2)).to(torch.complex128)
            A[:, t0 + nd + 1 + i, col[f]:col[f] + N] = beta
        mean = (modes[:, 0] == 0) & (modes[:, 1] == 0)
        A[mean, 0, tau_p] += beta
        w = torch.where(deg % 2 == 0, LZ / (1.0 - deg.to(torch.float64) ** 2), torch.zeros_like(self.D[0]))
        A[mean, n - 1, col["p"]:col["p"] + N] = beta * w.to(torch.complex128)
        A[~mean, n - 1, tau_p] = beta
        return A

    def vectors(self, fields):
        """(fields, Nz, Ny, Kx) -> (modes, fields * Nz)."""
        return fields.permute(2, 3, 0, 1).reshape(len(self.modes), -1)

    def fields(self, v):
        nf = self.ndim + 2
        return v[:, :nf * self.Nz].reshape(self.Ny, self.Nx // 2 + 1, nf, self.Nz).permute(2, 3, 0, 1)

    def solve(self, rhs, alpha, beta):
        """rhs: (modes, n) with the PDE rows set; the wall rows are filled here."""
        t0 = (self.ndim + 2) * self.Nz
        rhs = rhs.clone()
        rhs[:, t0:] = 0.0
        rhs[0, t0] = beta * LZ * self.Nx * self.Ny  # b(z=0) = Lz, b(z=Lz) = 0
        out = torch.empty_like(rhs)
        for a in range(0, len(rhs), self.chunk):
            key = (a, alpha, beta)
            if key not in self.lu:
                self.lu[key] = torch.linalg.lu_factor(self.matrix(self.modes[a:a + self.chunk], alpha, beta))
            out[a:a + self.chunk] = torch.linalg.lu_solve(*self.lu[key], rhs[a:a + self.chunk, :, None])[..., 0]
        return out

    def apply_L(self, v):
        out = torch.empty_like(v)
        for a in range(0, len(v), self.chunk):
            L = self.matrix(self.modes[a:a + self.chunk], 0.0, 1.0)
            out[a:a + self.chunk] = (L @ v[a:a + self.chunk, :, None])[..., 0]
        return out

    def rows(self, fields):
        """Right-hand-side vectors with the given b and velocity rows."""
        v = torch.zeros((len(self.modes), self.n), dtype=torch.complex128, device=DEVICE)
        v[:, self.Nz:(self.ndim + 2) * self.Nz] = self.vectors(fields)
        return v

    def projected(self, c):
        return _to_coeff(_to_grid(c, self.Nx))

    def advection(self, c):
        """-(u . grad) f of b and the velocity."""
        dims = (-1, -2) if self.ndim == 3 else (-1,)
        g = _to_grid(c, self.Nx)
        c = _to_coeff(g)
        D = self.D.to(torch.complex128)
        grads = [1j * self.kx * c, 1j * self.ky[:, None] * c, torch.einsum("zn,fnyk->fzyk", D, c)]
        if self.ndim == 2:
            del grads[1]
        out = torch.zeros_like(g)
        for i, d in enumerate(grads):
            dg = _to_grid(d, self.Nx)
            for f in range(len(g)):
                out[f] -= _dealiased(g[1 + i], dg[f], dims)
        return _to_coeff(out)

    def run_rk(self, c, dt, steps, scheme):
        AE, AI, w = _TABLEAUS[scheme]
        nv = self.ndim + 1
        for _ in range(steps):
            MX, F, LX, cur = self.rows(c[:nv]), [], [], c[:nv]
            for i in range(len(w)):
                taus = None
                if i > 0:
                    rhs = MX.clone()
                    for j in range(i):
                        rhs += dt * AE[i][j] * F[j]
                        if AI[i][j]:
                            rhs -= dt * AI[i][j] * LX[j]
                    x = self.solve(rhs, 1.0, dt * AI[i][i])
                    cur, taus = self.fields(x)[:nv], x
                F.append(self.rows(self.advection(cur)))
                if taus is None:
                    LX.append(None)  # no stage or update weighs it
                else:
                    v = taus.clone()
                    v[:, :nv * self.Nz] = self.vectors(self.projected(cur))
                    LX.append(self.apply_L(v))
            x = MX
            for i in range(1, len(w)):
                x = x + dt * w[i] * (F[i] - LX[i])
            new = x[:, self.Nz:(self.ndim + 2) * self.Nz].reshape(self.Ny, self.Nx // 2 + 1, nv, self.Nz)
            c = torch.cat([new.permute(2, 3, 0, 1), torch.zeros_like(c[:1])])
        return c

    def run_sbdf(self, c, dt, steps, order):
        nv, old = self.ndim + 1, None
        for _ in range(steps):
            F, MX = self.rows(self.advection(c[:nv])), self.rows(self.projected(c[:nv]))
            if old is None or order == 1:
                x = self.solve(F + MX / dt, 1.0 / dt, 1.0)
            else:
                x = self.solve(2 * F - old[0] + (2 * MX - 0.5 * old[1]) / dt, 1.5 / dt, 1.0)
            old = (F, MX)
            c = self.fields(x).clone()
        return c

    def run(self, c, dt, steps, scheme):
        return self.run_rk(c, dt, steps, scheme) if scheme[0] == "R" else self.run_sbdf(c, dt, steps, int(scheme[-1]))


def _turbulence_exact(q, Nx, Ny, dt, steps, scheme, nu=1e-4):
    q = torch.from_numpy(q).to(DEVICE)
    kx, ky = _wavenumbers(Nx, Ny, 2 * math.pi, 2 * math.pi)
    ky = ky[:, None]
    k2 = kx ** 2 + ky ** 2
    inv = torch.where(k2 > 0, 1.0 / torch.where(k2 > 0, k2, torch.ones_like(k2)), torch.zeros_like(k2))
    lam = nu * k2

    def grid(c):
        c = torch.fft.ifft(c, dim=0)
        c[:, 0].imag.zero_()
        c[:, Nx // 2].imag.zero_()
        return torch.fft.irfft(c, n=Nx, dim=1)

    def rhs(c):
        psi = -c * inv
        dims = (-1, -2)
        f = _dealiased(grid(-1j * ky * psi), grid(1j * kx * c), dims)
        f = f + _dealiased(grid(1j * kx * psi), grid(1j * ky * c), dims)
        return -torch.fft.fft(torch.fft.rfft(f, dim=1), dim=0)

    old = None
    for _ in range(steps):
        if scheme == "SBDF2":
            F = rhs(q)
            if old is None:
                new = (q + dt * F) / (1.0 + dt * lam)
            else:
                new = (2.0 * q - 0.5 * old[0] + dt * (2.0 * F - old[1])) / (1.5 + dt * lam)
            old, q = (q, F), new
            continue
        AE, AI, w = _TABLEAUS[scheme]
        Y, F = [], []
        for i in range(len(w)):
            y = q.clone()
            for j in range(i):
                y = y + dt * AE[i][j] * F[j] - dt * AI[i][j] * lam * Y[j]
            Y.append(y / (1.0 + dt * AI[i][i] * lam))
            F.append(rhs(Y[-1]))
        for i in range(len(w)):
            q = q + dt * w[i] * (F[i] - lam * Y[i])
    return q.cpu().numpy()


def _channel_exact(seed, Nx, Ny, Nz, ndim, scheme, steps, dt, kappa, nu):
    eq = _Boussinesq(Nx, Ny, Nz, ndim, kappa, nu)
    # the matrices of SBDF2 are two sets (its first step is SBDF1)
    if eq.memory() * (2 if scheme == "SBDF2" else 1) > 5e10 or eq.memory() * eq.n > 6e13:
        return None
    c = eq.run(_channel_fields(seed, Nx, Ny, Nz, ndim), dt, steps, scheme)
    if ndim == 2:
        return dict(zip(("b", "ux", "uz", "p"), c.reshape(4, Nz, Nx // 2 + 1)))
    return dict(zip(("b", "ux", "uy", "uz", "p"), c))


def exact(case, seed):
    kind, dt = case["kind"], _dt(case)
    if kind in ("channel", "channel3d"):
        kappa = case["Ra"] ** -0.5
        return _channel_exact(seed, case["Nx"], case.get("Ny", 1), case["Nz"], 2 if kind == "channel" else 3,
                              case["scheme"], case["steps"], dt, kappa, kappa)
    if kind == "turbulence":
        q = _turbulence_spec(seed, case["Nx"], case["Ny"])
        return _turbulence_exact(q, case["Nx"], case["Ny"], dt, case["steps"], case["scheme"])
    if kind == "transform":
        Nx, Nz, n = case["Nx"], case["Nz"], case["fields"]
        coeff = torch.cat([_channel_fields(seed + 7919 * i, Nx, 1, Nz, 2)[:1] for i in range(n)])
        grid = _to_grid(torch.cat([_channel_fields(seed + 7919 * i + 1, Nx, 1, Nz, 2)[1:2] for i in range(n)]), Nx)
        return dict(coeff=_to_coeff(grid).reshape(n, Nz, Nx // 2 + 1), grid=_to_grid(coeff, Nx).reshape(n, Nz, Nx))
    return [_channel_exact(seed + 101 * i, Nx, 1, Nz, 2, "RK222", case["steps"], dt, (Ra * Pr) ** -0.5, (Ra / Pr) ** -0.5)
            for i, (Nx, Nz, Ra, Pr) in enumerate(_members(case))]
