"""Performance cases of nsrno_b200: the calls a user's program makes, with their inputs.

``listed()`` names the cases, ``draw(rng)`` gives another case of the same
ranges, ``prepare`` makes what a program has in hand before the call, ``run``
makes one call through the package's public entry points, ``work`` counts the
bytes and operations the call cannot do without, and ``exact`` evaluates the
same quantity in 64 bits with plain torch.

Grids, bands, angle counts and media are those of the package's own records
(``nsrno_b200.media``), tests and benchmark: 256 x 256 blob records at 0.1 mm,
256 x 384 training media and 768 x 1024 breast records at 0.05 mm, the
1024 x 1536 Gauss-Newton grid at 0.04 mm, odd grids (243 x 729), and the dense
operator's 961 x 1121 medium with its 1056 x 1216 padding.
"""
import cmath
import math

import numpy as np
import torch

from nsrno_b200 import api, dense, learned, media, solver

DEVICE = "cuda"
SHIFT = 0.15
BINS = media.breast_bins()


def listed():
    return [
        # One operator application on one small field: the smallest call there
        # is, made inside a user's own Krylov loop or residual check.
        dict(name="apply_small", kind="apply", nz=256, nx=256, systems=1, fp64=False, adjoint=False),
        # FP64 adjoint operator on an odd grid: adjoint identities and residuals
        # of a record whose size is not a power of two.
        dict(name="apply_fp64_ragged", kind="apply", nz=243, nx=729, systems=6, fp64=True, adjoint=True),
        # The fixed shifted-Laplace preconditioner for the 11 angles of one
        # bin of the benchmark record.
        dict(name="precondition_bin", kind="precondition", nz=768, nx=1024, systems=11, adjoint=False),
        # Adjoint of the learned preconditioner for one training batch.
        dict(name="learned_adjoint_batch", kind="learned_precondition", nz=256, nx=384, systems=4, adjoint=True),
        # Network set-up of the four bins of one benchmark step.
        dict(name="learned_setup_step", kind="learned_setup", nz=768, nx=1024, frequencies=4),
        # Channels of three angles and their implicit gradient: one inner step
        # of an inversion on the 256 x 256 record.
        dict(name="implicit_gradient", kind="implicit", nz=256, nx=256, angles=3, frequency=1.5e6),
        # One step of the benchmark: 4 bins x 11 angles of the breast record to
        # 1e-6 through 22 resident systems, learned set-up included.
        dict(name="record_step", kind="record", nz=768, nx=1024, bins=4, angles=11, slots=22, learned=True,
             adjoint=False),
        # The 8-step GMRES warm start of one bin (solve_system's first phase).
        dict(name="warm_start_bin", kind="warm_start", nz=768, nx=1024, systems=11, steps=8),
        # Material gradient of two bins on the Gauss-Newton grid.
        dict(name="gradient_gauss_newton", kind="gradient", nz=1024, nx=1536, systems=22, fp64=False),
        # The dense operator on the 11 angles of one bin of its native medium.
        dict(name="dense_apply_bin", kind="dense_apply", h=961, w=1121, fields=11, fp64=False, adjoint=False),
        # Its preconditioner on the 1056 x 1216 padding.
        dict(name="dense_precondition_bin", kind="dense_precondition", h=961, w=1121, fields=11, adjoint=False),
        # A converged dense solve of five angles on a small medium.
        dict(name="dense_solve", kind="dense_solve", h=96, w=128, fields=5, frequency=4.2e6, adjoint=False),
    ]


# Grids the transforms take: the records' own, odd ones and prime-factor ones.
FFT_GRIDS = ((81, 81), (96, 54), (110, 140), (128, 192), (243, 729), (256, 256), (256, 384), (384, 512), (486, 640),
             (512, 768), (640, 840), (768, 1024), (1024, 1536))


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("apply", "apply", "precondition", "precondition", "learned_precondition", "learned_setup",
                       "implicit", "record", "record", "warm_start", "gradient", "dense_apply", "dense_precondition",
                       "dense_solve"))
    flag = lambda: rng.random() < 0.5  # noqa: E731
    if kind == "apply":
        nz, nx = _log_int(rng, 64, 1024), _log_int(rng, 64, 1536)
        return dict(kind=kind, nz=nz, nx=nx, systems=rng.randint(1, 22), fp64=flag(), adjoint=flag())
    if kind in ("precondition", "learned_precondition"):
        nz, nx = rng.choice(FFT_GRIDS)
        return dict(kind=kind, nz=nz, nx=nx, systems=rng.randint(1, 22), adjoint=flag())
    if kind == "learned_setup":
        return dict(kind=kind, nz=_log_int(rng, 96, 1024), nx=_log_int(rng, 96, 1536), frequencies=rng.randint(1, 8))
    if kind == "implicit":
        nz, nx = rng.choice(((128, 128), (128, 192), (192, 243), (243, 256), (256, 256), (256, 384)))
        return dict(kind=kind, nz=nz, nx=nx, angles=rng.randint(1, 8), frequency=rng.uniform(0.8e6, 1.6e6))
    if kind == "record":
        nz, nx = rng.choice(((110, 140), (128, 192), (243, 729), (256, 384), (384, 512), (512, 768), (768, 1024)))
        small = nz * nx <= 256 * 384
        return dict(kind=kind, nz=nz, nx=nx, bins=rng.randint(1, 4 if small else 2), angles=rng.randint(1, 11),
                    slots=rng.randint(1, 22), learned=flag() or not small, adjoint=flag())
    if kind == "warm_start":
        nz, nx = rng.choice(FFT_GRIDS)
        return dict(kind=kind, nz=nz, nx=nx, systems=rng.randint(1, 11), steps=rng.randint(4, 12))
    if kind == "gradient":
        return dict(kind=kind, nz=_log_int(rng, 64, 1024), nx=_log_int(rng, 64, 1536), systems=rng.randint(1, 22),
                    fp64=flag())
    if kind == "dense_solve":
        return dict(kind=kind, h=rng.randint(32, 96), w=rng.randint(40, 128), fields=rng.randint(1, 6),
                    frequency=rng.uniform(4.0e6, 4.6e6), adjoint=flag())
    case = dict(kind=kind, h=_log_int(rng, 64, 961), w=_log_int(rng, 64, 1121), fields=rng.randint(1, 11),
                adjoint=flag())
    if kind == "dense_apply":
        case["fp64"] = flag()
    return case


# ---------------------------------------------------------------------------
# What a program has in hand before the call
# ---------------------------------------------------------------------------
def _breast(nz, nx, seed, **more):
    """A breast-like record of the benchmark family (PML and array scaled to the grid)."""
    small = min(nz, nx)
    n_pml = 24 if small >= 256 else max(4, small // 12)
    h = 4e-5 if nx > 1024 or nz > 768 else 5e-5
    pitch = 4 if nx >= 64 else 2
    return media.breast_record(seed=seed, nz=nz, nx=nx, h=h, n_pml=n_pml, rx_pitch=pitch,
                               n_rx=max(8, min(192, nx // pitch - 8)), **more)


def _medium(rec):
    return solver.Medium(solver.Geometry.from_record(rec), rec.c, rec.rho, rec.alpha, device=DEVICE)


def _plain_medium(nz, nx, seed, h=5e-5):
    """A smooth random medium of any size with a PML (grids the record family does not fit)."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    low = torch.randn((1, 3, 9, 9), generator=gen, device=DEVICE)
    c, rho, alpha = torch.nn.functional.interpolate(low, size=(nz, nx), mode="bicubic", align_corners=True)[0]
    geo = solver.Geometry(nz=nz, nx=nx, h=h, n_pml=max(4, min(24, min(nz, nx) // 10)), face=6,
                          rx_cols=np.arange(8, nx - 8, 4), aperture_half_width=0.4 * nx * h)
    return solver.Medium(geo, 1500 + 40 * c, 1000 + 40 * rho, (0.5 + 0.2 * alpha).clamp_min(0.0), device=DEVICE)


def _frequencies(count, seed):
    return np.random.default_rng(seed).choice(BINS, size=count, replace=count > len(BINS))


def _fields(count, nz, nx, h, freqs, seed, dtype=torch.complex64):
    """Wavefield-like fields: a few plane waves of each frequency and 5% noise."""
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    z = torch.arange(nz, device=DEVICE, dtype=torch.float64)[:, None] * h
    x = torch.arange(nx, device=DEVICE, dtype=torch.float64)[None, :] * h
    out = torch.empty((count, nz, nx), dtype=dtype, device=DEVICE)
    for s in range(count):
        k0 = 2 * math.pi * float(freqs[s]) / 1500.0
        th = torch.rand(3, generator=gen, device=DEVICE, dtype=torch.float64) * 2 * math.pi
        w = torch.randn(3, generator=gen, device=DEVICE, dtype=torch.float64)
        noise = torch.randn((2, nz, nx), generator=gen, device=DEVICE, dtype=torch.float32)
        u = 0.05 * torch.complex(noise[0], noise[1]).to(torch.complex128)
        for q in range(3):
            u += w[q] * torch.exp(1j * k0 * (x * th[q].cos() + z * th[q].sin()))
        out[s] = u.to(dtype)
    return out


def _dense_spec(h, w, frequency=None):
    half = 0.5 * (w - 1) * 5e-5
    count = max(4, min(192, w // 4 - 4))
    return {"medium_shape": [h, w], "dx_m": 5e-5, "x0_m": -half, "z0_m": -0.0002, "native_dt_s": 2.5e-9,
            "pml": 24 if min(h, w) >= 256 else 12 if min(h, w) >= 64 else 6, "eta_per_unit_alpha": [0.012, 0.021],
            "taus_s": [2.0e-8, 1.5e-7], "source_c_lookup_zx": [10, 20], "rx_count": count, "rx_pitch_m": 0.0002,
            "rx_first_m": -0.0001 * (count - 1)}


def _dense_medium(h, w, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    low = torch.randn((1, 3, 9, 9), generator=gen, device=DEVICE, dtype=torch.float64)
    c, rho, alpha = torch.nn.functional.interpolate(low, size=(h, w), mode="bicubic", align_corners=True)[0]
    return torch.stack((1540 + 30 * c, 1000 + 30 * rho)), (0.6 + 0.2 * alpha).clamp_min(0.0)


def _dense_frequency(case, seed):
    return float(case.get("frequency") or _frequencies(1, seed)[0])


def prepare(case, seed):
    kind = case["kind"]
    if kind.startswith("dense"):
        return _prepare_dense(case, seed)
    nz, nx = case["nz"], case["nx"]
    if kind == "implicit":
        rec = media.blob_record(seed=seed, nz=nz, nx=nx, n_pml=20 if min(nz, nx) >= 192 else 12,
                                n_rx=min(192, nx - 48))
        angles = np.linspace(-15.0, 15.0, case["angles"]) if case["angles"] > 1 else [0.0]
        data = api.AcquisitionData(solver.Geometry.from_record(rec), angles, response=False)
        medium = torch.as_tensor(np.stack((rec.c, rec.rho)), device=DEVICE).requires_grad_(True)
        gen = torch.Generator(device=DEVICE).manual_seed(seed)
        cot = torch.randn((2, case["angles"], len(rec.rx_cols)), generator=gen, device=DEVICE, dtype=torch.float64)
        return dict(case=case, medium=medium, alpha=torch.as_tensor(rec.alpha, device=DEVICE), data=data,
                    cotangent=torch.complex(cot[0], cot[1]))
    if kind == "record":
        rec = _breast(nz, nx, seed, n_angles=case["angles"], bins=np.sort(_frequencies(case["bins"], seed)))
        f, a = rec.systems()
        st = dict(case=case, medium=_medium(rec), freqs=f, angles=a, bins=rec.frequencies)
        if case["learned"]:
            st["net"] = learned.LearnedPreconditioner.load(device=DEVICE)
        if case["adjoint"]:
            gen = torch.Generator(device=DEVICE).manual_seed(seed)
            val = torch.randn((2, len(f), len(rec.rx_cols)), generator=gen, device=DEVICE)
            st["rhs"] = torch.zeros((len(f), nz, nx), dtype=torch.complex64, device=DEVICE)
            st["rhs"][:, rec.face, torch.as_tensor(rec.rx_cols, device=DEVICE)] = torch.complex(val[0], val[1])
        return st
    if kind in ("learned_precondition", "warm_start"):
        med = _medium(_breast(nz, nx, seed))
        net = learned.LearnedPreconditioner.load(device=DEVICE)
        rng = np.random.default_rng(seed)
        if kind == "warm_start":      # the angles of one bin share its frequency
            f = np.repeat(_frequencies(1, seed), case["systems"])
            angles = np.deg2rad(np.linspace(-25.0, 25.0, case["systems"])) if case["systems"] > 1 else np.zeros(1)
            return dict(case=case, medium=med, net=net, setup=net.setup(med, f[:1]), freqs=f, angles=angles)
        f = rng.choice(BINS, size=case["systems"], replace=False)
        x = _fields(case["systems"], nz, nx, med.geometry.h, f, seed)
        return dict(case=case, medium=med, net=net, setup=net.setup(med, f), freqs=f, x=x,
                    index=torch.arange(case["systems"], dtype=torch.int32, device=DEVICE))
    if kind == "learned_setup":
        med = _plain_medium(nz, nx, seed)
        return dict(case=case, medium=med, net=learned.LearnedPreconditioner.load(device=DEVICE),
                    freqs=torch.as_tensor(_frequencies(case["frequencies"], seed), device=DEVICE))
    # operators on fields: apply, precondition, gradient
    med = _plain_medium(nz, nx, seed)
    S = case["systems"]
    f = np.repeat(_frequencies((S + 10) // 11, seed), 11)[:S]
    dtype = torch.complex128 if case.get("fp64") else torch.complex64
    st = dict(case=case, medium=med, freqs=torch.as_tensor(f, device=DEVICE),
              x=_fields(S, nz, nx, med.geometry.h, f, seed, dtype))
    if kind == "gradient":
        st["lam"] = _fields(S, nz, nx, med.geometry.h, f, seed + 1, dtype)
    return st


def _prepare_dense(case, seed):
    geo = dense.DenseGeometry(_dense_spec(case["h"], case["w"]))
    medium, alpha = _dense_medium(case["h"], case["w"], seed)
    f = _dense_frequency(case, seed)
    system = dense.DenseSystem(geo, medium, alpha, f, device=DEVICE)
    st = dict(case=case, system=system)
    if case["kind"] == "dense_solve":
        # plane-wave lines on the array row, as complex64 right-hand sides
        x = (torch.arange(geo.w, device=DEVICE, dtype=torch.float64) - 0.5 * (geo.w - 1)) * geo.dx
        th = torch.linspace(-0.4, 0.4, case["fields"], device=DEVICE, dtype=torch.float64)[:, None]
        taper = torch.cos(0.5 * math.pi * x / (0.5 * geo.w * geo.dx)) ** 2
        line = taper * torch.exp(2j * math.pi * f / 1540.0 * x * torch.sin(th))
        st["rhs"] = system.source(line).to(torch.complex64)
    else:
        dtype = torch.complex128 if case.get("fp64") else torch.complex64
        st["x"] = _fields(case["fields"], geo.H, geo.W, geo.dx, [f] * case["fields"], seed, dtype)
    return st


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "apply":
        return solver.apply(state["medium"], state["x"], state["freqs"], adjoint=case["adjoint"])
    if kind == "precondition":
        return solver.precondition(state["medium"], state["x"], state["freqs"], adjoint=case["adjoint"])
    if kind == "learned_precondition":
        return learned.learned_precondition(state["medium"], state["setup"], state["x"], state["freqs"],
                                            adjoint=case["adjoint"], gain_index=state["index"])
    if kind == "learned_setup":
        return state["net"].setup(state["medium"], state["freqs"]).gains
    if kind == "implicit":
        ch = api.implicit_channels(state["medium"], state["alpha"], state["data"], case["frequency"],
                                   range(case["angles"]), tolerance=1e-8)
        grad, = torch.autograd.grad(ch, state["medium"], state["cotangent"])
        # the field is good to the solve's tolerance: the channels are handed on
        # in complex64, as solve_frequency hands them on
        return {"channels": ch.detach().to(torch.complex64), "gradient": grad}
    if kind == "record":
        setup = state["net"].setup(state["medium"], state["bins"]) if case["learned"] else None
        rhs = state.get("rhs")
        res = solver.solve_batched(state["medium"], state["freqs"], None if rhs is not None else state["angles"],
                                   rhs=rhs, adjoint=case["adjoint"], learned=setup, tolerance=1e-6,
                                   max_iterations=4000, n_slots=case["slots"], return_fields=True)
        # fields and receiver values to 1e-6 (complex64 as above) and each system's status
        return {"fields": res.fields, "receivers": res.iq.to(torch.complex64), "status": res.status}
    if kind == "warm_start":
        x0, _ = learned.warm_start(state["medium"], state["setup"], state["freqs"], state["angles"],
                                   steps=case["steps"], n_slots=case["systems"])
        return x0
    if kind == "gradient":
        return solver.grad_accum(state["medium"], state["freqs"], state["x"], state["lam"])
    if kind == "dense_apply":
        return (state["system"].adjoint if case["adjoint"] else state["system"].apply)(state["x"])
    if kind == "dense_precondition":
        return state["system"].fixed_preconditioner(adjoint=case["adjoint"])(state["x"])
    x, _ = dense.solve(state["system"], state["rhs"], adjoint=case["adjoint"], tolerance=1e-6, max_cycles=400)
    return x


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _fft_flops(nz, nx):
    return 5.0 * nz * nx * math.log2(nz * nx)


def work(case):
    kind = case["kind"]
    if kind.startswith("dense"):
        H, W = (math.ceil((v + 64) / 32) * 32 for v in (case["h"], case["w"]))
        n, S = H * W, case["fields"]
        b = 16 if case.get("fp64") else 8
        if kind == "dense_apply":          # field in and out, ax, az and the mass term
            return dict(bytes=n * (2 * b * S + 32), flops=n * S * 120)
        pre = 2 * _fft_flops(H, W) + 16 * n
        if kind == "dense_precondition":
            return dict(bytes=16 * n * S, flops=pre * S)
        # about 72 Arnoldi steps of restart 24: the preconditioned vector and the
        # operator in and out, the basis (12 vectors on average) read twice
        steps = 72
        return dict(bytes=steps * n * S * 8 * (4 + 24), flops=steps * S * (pre + n * (120 + 16 * 24)))
    n = case["nz"] * case["nx"]
    if kind == "learned_setup":
        F = case["frequencies"]
        return dict(bytes=n * (12 + 16 * F), flops=F * (2 * 3600 * n / 64 + 80 * n))
    if kind == "implicit":
        # about 60 iterations forward and 60 back: the six Krylov vectors of an
        # iteration once each (88 B per node), four transforms and two stencils
        it = 120 * case["angles"]
        return dict(bytes=it * n * 88, flops=it * (4 * _fft_flops(case["nz"], case["nx"]) + n * 150))
    if kind == "record":
        it = (50 if case["learned"] else 160) * case["bins"] * case["angles"]
        return dict(bytes=it * n * 88, flops=it * (4 * _fft_flops(case["nz"], case["nx"]) + n * 150))
    S = case["systems"]
    if kind == "apply":
        b = 2 if case["fp64"] else 1
        return dict(bytes=n * (16 * b * S + 12 * b), flops=n * S * 45)
    if kind in ("precondition", "learned_precondition"):
        gains = 16 if kind == "learned_precondition" else 0
        return dict(bytes=n * (16 + gains) * S, flops=S * (2 * _fft_flops(case["nz"], case["nx"]) + 16 * n))
    if kind == "gradient":
        return dict(bytes=n * ((32 if case["fp64"] else 16) * S + 24 + 16), flops=n * S * 150)
    m = case["steps"]                       # warm start: basis vectors read twice, fields written
    return dict(bytes=S * n * (8 * (m * (m + 1) + 6 * m) + 16),
                flops=S * ((m + 1) * 2 * _fft_flops(case["nz"], case["nx"]) + n * (45 * m + 16 * m * m)))


# ---------------------------------------------------------------------------
# The same quantities in 64 bits, with plain torch
# ---------------------------------------------------------------------------
def _stretch(pos, n, n_pml):
    f = torch.maximum(n_pml - pos, pos - (n - 1 - n_pml)) / n_pml if n_pml > 0 else torch.zeros_like(pos)
    return f.clamp(0.0, 1.0) ** 2


class _Operator:
    """The h^2-scaled 5-point operator of one medium at one frequency (complex128)."""

    def __init__(self, med, f):
        g = med.geometry
        c, rho, alpha = (v.double() for v in (med.c, med.rho, med.alpha))
        self.g, self.f = g, float(f)
        omega = 2 * math.pi * self.f
        sig = g.pml_strength * g.c0 / (g.n_pml * g.h) / omega if g.n_pml > 0 else 0.0
        self.kh2 = (omega / g.c0 * g.h) ** 2
        self.k0 = omega / g.c0
        z = torch.arange(g.nz, device=c.device, dtype=torch.float64)[:, None]
        x = torch.arange(g.nx, device=c.device, dtype=torch.float64)[None, :]
        s = lambda pos, n: 1 + 1j * sig * _stretch(pos, n, g.n_pml)  # noqa: E731
        sx, sz = s(x, g.nx), s(z, g.nz)
        self.a = g.rho0 / rho
        ap = torch.nn.functional.pad(self.a[None, None], (1, 1, 1, 1), value=1.0)[0, 0]
        self.w = [sz / s(x + 0.5, g.nx), sz / s(x - 0.5, g.nx), sx / s(z + 0.5, g.nz), sx / s(z - 0.5, g.nz)]
        nb = [ap[1:-1, 2:], ap[1:-1, :-2], ap[2:, 1:-1], ap[:-2, 1:-1]]
        self.flux = [0.5 * (self.a + q) * w for q, w in zip(nb, self.w)]
        b = g.rho0 * g.c0 ** 2 / (rho * c * c)
        neper = 100.0 * math.log(10.0) / 20.0
        self.onepie = 1 + 1j * alpha * neper * c / (2 * math.pi * 1e6) * (self.f / 1e6) ** (g.alpha_power - 1.0)
        self.cell = self.kh2 * b * sx * sz
        self.mass = self.cell * self.onepie ** 2

    @staticmethod
    def neighbours(u):
        p = torch.nn.functional.pad(u, (1, 1, 1, 1))
        return p[..., 1:-1, 2:], p[..., 1:-1, :-2], p[..., 2:, 1:-1], p[..., :-2, 1:-1]

    def apply(self, u, adjoint=False):
        cj = torch.conj if adjoint else (lambda v: v)
        y = cj(self.mass) * u
        for fl, q in zip(self.flux, self.neighbours(u)):
            y = y + cj(fl) * (q - u)
        return y

    def source(self, angle):
        """h^2-scaled plane-wave source of the array row."""
        g = self.g
        x = (torch.arange(g.nx, device=self.a.device, dtype=torch.float64) - 0.5 * (g.nx - 1)) * g.h
        taper = torch.where(x.abs() > g.aperture_half_width, 0.0 * x,
                            0.5 * (1 + torch.cos(math.pi * x / g.aperture_half_width)))
        b = torch.zeros((g.nz, g.nx), dtype=torch.complex128, device=x.device)
        b[g.face] = -taper * torch.exp(-1j * self.k0 * x * math.sin(angle))
        return b

    def gradient(self, u, lam):
        """-Re(lam^H dA/dm u) for m = log c, log rho."""
        lu = lam.conj() * u
        gc = -(lu * (-2 * self.cell * self.onepie)).real
        edge = 0
        for w, uq, lq in zip(self.w, self.neighbours(u), self.neighbours(lam)):
            edge = edge + 0.5 * w * (lq - lam).conj() * (uq - u)
        gr = -(lu * (-self.mass)).real - self.a * edge.real
        return gc / self.g.h ** 2, gr / self.g.h ** 2

    def factor(self):
        """Inverse Schur blocks of the block-tridiagonal elimination along z."""
        g = self.g
        fe, fw, fs, fn = self.flux
        diag = self.mass - fe - fw - fs - fn
        inv = torch.empty((g.nz, g.nx, g.nx), dtype=torch.complex128, device=self.a.device)
        for i in range(g.nz):
            d = torch.diag(diag[i]) + torch.diag(fe[i, :-1], 1) + torch.diag(fw[i, 1:], -1)
            if i:
                d = d - fn[i][:, None] * inv[i - 1] * fs[i - 1][None, :]
            inv[i] = torch.linalg.inv(d)
        self.inv = inv

    def solve(self, b):
        """``A u = b`` for b [S, nz, nx] (after :meth:`factor`)."""
        g, fs, fn = self.g, self.flux[2], self.flux[3]
        y = b.clone()
        for i in range(1, g.nz):
            y[:, i] -= fn[i] * (y[:, i - 1] @ self.inv[i - 1].T)
        u = torch.empty_like(y)
        for i in range(g.nz - 1, -1, -1):
            r = y[:, i] - (fs[i] * u[:, i + 1] if i + 1 < g.nz else 0)
            u[:, i] = r @ self.inv[i].T
        return u


def _sin2(n):
    return torch.sin(math.pi * torch.arange(n, device=DEVICE, dtype=torch.float64) / n) ** 2


def _gains(net, med, f):
    """Inner and outer gain planes of the learned preconditioner, complex128."""
    F = torch.nn.functional
    p = net.params.double()
    w1, b1 = p[9:729].reshape(16, 5, 3, 3), p[729:745]
    w2, b2 = p[745:3049].reshape(16, 16, 3, 3), p[3049:3065]
    w3, b3 = p[3065:3641].reshape(4, 16, 3, 3), p[3641:3645]
    c, rho, alpha = (v.double() for v in (med.c, med.rho, med.alpha))
    ctx = torch.stack(((c / 1540).log() / 0.06, (rho / 1000).log() / 0.08, torch.log1p(alpha),
                       torch.full_like(c, float(f) / 6e6 - 1), torch.ones_like(c)))[None]
    conv = lambda v, w, b: F.conv2d(v, w, b, padding=1)  # noqa: E731
    m = conv(torch.tanh(conv(torch.tanh(conv(F.avg_pool2d(ctx, 8), w1, b1)), w2, b2)), w3, b3)
    t = torch.tanh(F.interpolate(m, size=tuple(c.shape), mode="bilinear", align_corners=False)[0])
    return (1 + 0.5 * t[0]) * torch.exp(-0.5j * t[1]), (1 + 0.5 * t[2]) * torch.exp(-0.5j * t[3])


def _spectral(net, g, f):
    """Learned multiplier [nz, nx] of the 5-point path."""
    p = net.params.double()
    kh2 = (2 * math.pi * float(f) / g.c0 * g.h) ** 2
    s2z, s2x = _sin2(g.nz)[:, None], _sin2(g.nx)[None, :]
    q2 = 4 * (s2z + s2x) / kh2
    rq = q2 / (1 + q2)
    ang = 4 * s2x / (4 * (s2x + s2z) + g.h ** 2)
    mod = [p[4 * k] + p[4 * k + 1] * rq + (p[4 * k + 2] + p[4 * k + 3] * rq) * ang for k in range(2)]
    shift = p[8].exp().clamp(0.01, 1.0)
    return torch.exp(0.5 * torch.tanh(mod[0]) - 0.5j * torch.tanh(mod[1])) / (kh2 - kh2 * q2 + 1j * kh2 * shift)


def _learned_map(net, med, f):
    inner, outer = _gains(net, med, f)
    mul = _spectral(net, med.geometry, f)

    def m(r, adjoint=False):
        if adjoint:
            return inner.conj() * torch.fft.ifft2(mul.conj() * torch.fft.fft2(outer.conj() * r))
        return outer * torch.fft.ifft2(mul * torch.fft.fft2(inner * r))
    return m


def _gmres_cycle(a, m, b, steps):
    """argmin ||b - A M y|| over the Krylov space of ``steps`` vectors from zero; returns M y."""
    beta = torch.linalg.vector_norm(b)
    V = [b / beta]
    H = torch.zeros((steps + 1, steps), dtype=torch.complex128, device=b.device)
    for j in range(steps):
        w = a(m(V[j]))
        for _ in range(2):
            for i in range(j + 1):
                h = torch.vdot(V[i].flatten(), w.flatten())
                H[i, j] += h
                w = w - h * V[i]
        H[j + 1, j] = torch.linalg.vector_norm(w)
        V.append(w / H[j + 1, j])
    e = torch.zeros((steps + 1, 1), dtype=torch.complex128, device=b.device)
    e[0] = beta
    y = torch.linalg.lstsq(H, e).solution[:, 0]
    return m(sum(y[i] * V[i] for i in range(steps)))


class _Dense:
    """The 8th-order operator of one medium at one frequency (complex128, periodic shifts)."""

    COEF = (1225 / 1024, -245 / 3072, 49 / 5120, -5 / 7168)

    def __init__(self, geo, medium, alpha, f):
        self.g = g = geo
        pad = geo.pad_material_t
        c, rho = pad(medium)
        al = pad(alpha[None])[0]
        dt, c0 = g.dt, 1540.0
        D = cmath.exp(2j * math.pi * f * dt)
        q = 1 / D
        self.k0 = 2 * math.sin(math.pi * f * dt) / (dt * c0)
        self.scal = (D - 1) / D / self.k0 ** 2
        self.mask = torch.zeros_like(c)
        self.mask[g.pz:g.pz + g.h, g.px:g.px + g.w] = 1.0
        a = 1000.0 / rho
        mean = lambda d: 2 * a * torch.roll(a, -1, d) / (a + torch.roll(a, -1, d)) * self.mask  # noqa: E731
        eta = [al * c / c0 * v for v in g.spec["eta_per_unit_alpha"]]
        amp = (1 + 0.5 * (eta[0] + eta[1])) ** 2
        r = sum(e / (amp * (1 + t * (D - 1) / dt)) for e, t in zip(eta, g.spec["taus_s"]))
        self.mass = a * (c0 / c) ** 2 / (amp * (1 - r) / (1 - (1 - q) * r))
        self.axis = []
        for d, n, n0, first in ((1, g.W, g.w, g.px), (0, g.H, g.h, g.pz)):
            pos = torch.arange(n, device=c.device, dtype=torch.float64) - first

            def damping(stagger):
                lo = torch.where(pos < g.pml, (1 - (pos + stagger) / g.pml) ** 4, 0.0 * pos)
                hi = torch.where(pos >= n0 - g.pml, (1 - (n0 - 1 - pos - stagger) / g.pml) ** 4, 0.0 * pos)
                return 1 - dt * (lo + hi) * 2 * c0 / g.dx
            ar, av = damping(0.0), damping(0.5)
            m = (ar != 1.0).double()
            prof = [(D - 1) / (D - av), 1 + (1 - av) * q, m / (D - ar), 1 + (1 - m) / (D - ar)]
            shape = (1, n) if d == 1 else (n, 1)
            self.axis.append((d - 2, mean(d), *[v.reshape(shape) for v in prof]))

    def grad(self, p, d):
        return sum(a * (torch.roll(p, -1 - k, d) - torch.roll(p, k, d)) for k, a in enumerate(self.COEF)) / self.g.dx

    def div(self, p, d):
        return sum(a * (torch.roll(p, -k, d) - torch.roll(p, 1 + k, d)) for k, a in enumerate(self.COEF)) / self.g.dx

    def apply(self, p, adjoint=False):
        u = self.mask * p
        if not adjoint:
            acc = 0
            for d, ax, sv, gv, left, right in self.axis:
                x = ax * sv * self.grad(u, d)
                acc = acc + left * self.div(x, d) + right * self.div(gv * x, d)
            return self.mask * (self.scal * acc + self.mass * u) + (1 - self.mask) * p
        w = self.scal.conjugate() * u
        acc = self.mass.conj() * u
        for d, ax, sv, gv, left, right in self.axis:
            flux = (ax * sv).conj() * -(self.grad(left.conj() * w, d) + gv.conj() * self.grad(right.conj() * w, d))
            acc = acc - self.div(flux, d)
        return self.mask * acc + (1 - self.mask) * p

    def precondition(self, r, adjoint):
        sym = []
        for n in (self.g.H, self.g.W):
            q = 2 * math.pi * torch.arange(n, device=r.device, dtype=torch.float64) / n
            sym.append((2 * sum(a * torch.sin((k + 0.5) * q) for k, a in enumerate(self.COEF)) / self.g.dx) ** 2)
        m = 1 / (1 - (sym[0][:, None] + sym[1][None, :]) / self.k0 ** 2 - 1j * SHIFT)
        return self.mask * torch.fft.ifft2((m.conj() if adjoint else m) * torch.fft.fft2(r))


def exact(case, seed):
    kind = case["kind"]
    if kind in ("record", "dense_solve"):
        return None      # a direct solve of these grids takes minutes
    st = prepare(case, seed)
    if kind.startswith("dense"):
        medium, alpha = _dense_medium(case["h"], case["w"], seed)
        op = _Dense(st["system"].g, medium, alpha, _dense_frequency(case, seed))
        f = op.apply if kind == "dense_apply" else op.precondition
        return torch.stack([f(v.to(torch.complex128), case["adjoint"]) for v in st["x"]])
    med = st["medium"]
    if kind == "implicit":
        g = st["data"].geometry
        md = st["medium"].detach()
        op = _Operator(solver.Medium(g, md[0], md[1], st["alpha"], device=DEVICE), case["frequency"])
        op.factor()
        u = op.solve(torch.stack([op.source(t) for t in st["data"].angles]))
        rx = torch.as_tensor(np.asarray(g.rx_cols), device=DEVICE)
        rhs = torch.zeros_like(u)
        rhs[:, g.face, rx] = st["cotangent"] * g.h ** 2
        lam = op.solve(rhs.conj()).conj()
        gc, gr = (sum(v) for v in zip(*[op.gradient(a, b) for a, b in zip(u, lam)]))
        return {"channels": u[:, g.face, rx], "gradient": torch.stack((gc / md[0].double(), gr / md[1].double()))}
    g = med.geometry
    if kind == "learned_setup":
        return torch.stack([torch.stack(_gains(st["net"], med, f)) for f in st["freqs"].tolist()])
    if kind == "learned_precondition":
        return torch.stack([_learned_map(st["net"], med, f)(v.to(torch.complex128), case["adjoint"])
                            for v, f in zip(st["x"], st["freqs"])])
    if kind == "warm_start":
        op, m = _Operator(med, st["freqs"][0]), _learned_map(st["net"], med, st["freqs"][0])
        return torch.stack([_gmres_cycle(op.apply, m, op.source(t), case["steps"]) for t in st["angles"]])
    freqs = st["freqs"].tolist()
    if kind == "apply":
        return torch.stack([_Operator(med, f).apply(v.to(torch.complex128), case["adjoint"])
                            for v, f in zip(st["x"], freqs)])
    if kind == "precondition":
        out = []
        lap = 4 * (_sin2(g.nz)[:, None] + _sin2(g.nx)[None, :])
        for v, f in zip(st["x"], freqs):
            m = 1 / ((2 * math.pi * f / g.c0 * g.h) ** 2 * (1 + 1j * SHIFT) - lap)
            out.append(torch.fft.ifft2((m.conj() if case["adjoint"] else m) * torch.fft.fft2(v.to(torch.complex128))))
        return torch.stack(out)
    parts = [_Operator(med, f).gradient(u.to(torch.complex128), v.to(torch.complex128))
             for u, v, f in zip(st["x"], st["lam"], freqs)]
    return sum(p[0] for p in parts), sum(p[1] for p in parts)
