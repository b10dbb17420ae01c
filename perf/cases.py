"""The calls a user of this framework makes, as measurable cases.

A case is one pass through a public entry point: the mobility solve on device
or host arrays, the fixed-position operator, the resistance solve, the
objective gradient and the batched form. Sizes are those of the benchmark
workloads, of the reference's published GPU record (N = 186,510, L = 250,
256^3, M_G = 10, R_c = 5.642) and generic ones (grids with factors 3, 5, 7;
stencils of 6 to 12 points; both precisions).

Keys of a case:
  call    mobility | host | operator | resistance | gradient | batch
  f64     working precision Float64 instead of Float32
  N       particles (batch: of the largest system; the smallest holds N_min)
  mx, my, mz, h   grid points per axis and the grid spacing (box = M h)
  M_G, R_c        stencil width and pair cutoff
  layout  suspension (non-overlapping, disordered lattice) | uniform | clustered
  iters   conjugate-gradient iterations of a resistance solve
  systems, nrhs   systems and right-hand sides of a batch
"""
import importlib.util
import math
import sys
from pathlib import Path

import numpy as np
import torch

RATIO = 2.0          # kernel widths ratio Sigma / sigma
SIGMA = 1.0 / math.sqrt(math.pi)
WIDE = RATIO * SIGMA
MU = 1.0


def _package():
    """`ffcm.jl_b200/` of the working folder, under its import name."""
    if "ffcm_b200" not in sys.modules:
        pkg = Path.cwd() / "ffcm.jl_b200"
        spec = importlib.util.spec_from_file_location("ffcm_b200", pkg / "__init__.py",
                                                      submodule_search_locations=[str(pkg)])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["ffcm_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["ffcm_b200"]


def _case(name, call, N, grid, h, M_G=8, R_c=3.0, f64=False, layout="suspension", **more):
    mx, my, mz = grid if isinstance(grid, tuple) else (grid,) * 3
    c = dict(call=call, N=N, mx=mx, my=my, mz=mz, h=h, M_G=M_G, R_c=R_c, f64=f64, layout=layout, **more)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # a small suspension stepped by a device-resident program: launches count
        _case("small", "mobility", 2_000, 64, 40.0 / 64),
        # the same from host arrays, as a script calls it: copies and latency
        _case("small_host", "host", 2_000, 64, 40.0 / 64),
        # a mid-size suspension in double precision
        _case("mid_f64", "mobility", 62_500, 256, 139.0 / 256, f64=True),
        # the configuration of the reference's published GPU record, both precisions
        _case("record_f32", "mobility", 186_510, 256, 250.0 / 256, M_G=10, R_c=5.642, layout="uniform"),
        _case("record_f64", "mobility", 186_510, 256, 250.0 / 256, M_G=10, R_c=5.642, layout="uniform", f64=True),
        # a non-cubic box on a grid that is no power of two
        _case("ragged", "mobility", 29_000, (240, 200, 160), 0.54),
        # odd factors, a wide stencil and double precision together
        _case("ragged_wide", "mobility", 9_000, (120, 108, 105), 0.7, M_G=12, R_c=4.0, f64=True),
        # a fixed number of Krylov iterations of the resistance problem, as a time step takes them
        _case("resistance", "resistance", 2_000, 64, 40.0 / 64, iters=30),
        # forward and backward: an objective with its gradients
        _case("gradient", "gradient", 100_000, 256, 161.0 / 256),
        # several suspensions of different sizes with several force sets each
        _case("batch", "batch", 64_000, 256, 0.54, systems=6, nrhs=4, N_min=2_000),
        # the benchmark's headline solve
        _case("large", "mobility", 500_000, 512, 275.6 / 512),
        # the largest: the fixed-position operator on a dense clustered suspension
        _case("clustered", "operator", 2_000_000, 1024, 300.0 / 1024, layout="clustered"),
    ]


# FFT-friendly lengths (factors up to 13), as users choose them for boxes that no power of two fits
_LENGTHS = [24, 27, 28, 30, 35, 36, 40, 42, 45, 48, 50, 54, 56, 60, 63, 66, 70, 72, 75, 78, 80, 81, 84, 88, 90, 96, 98,
            100, 105, 108, 110, 112, 117, 120, 125, 126, 135, 140, 144, 150, 160, 162, 168, 175, 180, 189, 192, 200,
            210, 216, 225, 240, 250, 264, 270, 280, 288, 300, 312, 320]
_POWERS = [32, 64, 128, 256]


def draw(rng):
    call = rng.choice(["mobility"] * 5 + ["host", "operator", "gradient", "resistance", "batch"])
    f64 = rng.random() < 0.4
    M_G = rng.choice([6, 7, 8, 8, 8, 9, 10, 11, 12])
    # the stencil reaches 1.9 to 4.3 standard deviations of the wide kernel
    h = round(WIDE * rng.uniform(3.8, 8.6) / M_G, 4)
    top = 128 if call == "resistance" else 320
    if call == "batch":
        return _case(None, "batch", rng.randint(8_000, 64_000), 256, 0.54, M_G=8, f64=f64, systems=rng.randint(3, 8),
                     nrhs=rng.randint(1, 6), N_min=rng.randint(1_000, 4_000))
    base = math.exp(rng.uniform(math.log(24), math.log(top)))
    lengths = [m for m in (_POWERS if rng.random() < 0.35 else _LENGTHS) if m <= top]

    def near(x):
        return min(lengths, key=lambda m: abs(math.log(m / x)))

    if rng.random() < 0.4:
        grid = (near(base),) * 3
    else:
        grid = tuple(near(min(top, max(24.0, base * rng.uniform(0.6, 1.6)))) for _ in range(3))
    box = [m * h for m in grid]
    phi = math.exp(rng.uniform(math.log(0.02), math.log(0.2)))
    N = int(phi * box[0] * box[1] * box[2] / (4.0 / 3.0 * math.pi))
    N = max(20, min(N, 100_000 if call == "gradient" else 200_000))
    R_c = min(rng.choice([3.0, 3.0, 4.0, 5.6]), 0.45 * min(box))
    more = dict(iters=rng.randint(8, 30)) if call == "resistance" else {}
    return _case(None, call, N, grid, h, M_G=M_G, R_c=round(R_c, 3), f64=f64,
                 layout=rng.choice(["suspension", "suspension", "uniform"]), **more)


# ---- inputs -----------------------------------------------------------------

def _types(case):
    return (np.float64, torch.float64) if case["f64"] else (np.float32, torch.float32)


def _systems(case):
    """The systems of a case: dicts with L, R_c, N, num_grid_points."""
    if case["call"] != "batch":
        M = (case["mx"], case["my"], case["mz"])
        return [dict(L=tuple(m * case["h"] for m in M), R_c=case["R_c"], N=case["N"], num_grid_points=M)]
    out = []
    for i in range(case["systems"]):
        # N geometric from N_min to N; 10% by volume; the power of two nearest to L / h
        t = i / (case["systems"] - 1)
        N = int(round(case["N_min"] ** (1 - t) * case["N"] ** t))
        L = (N * 4.0 / 3.0 * math.pi / 0.1) ** (1.0 / 3.0)
        M = min(case["mx"], max(64, 2 ** round(math.log2(L / case["h"]))))
        out.append(dict(L=(L,) * 3, R_c=case["R_c"], N=N, num_grid_points=(M,) * 3))
    return out


def _positions(N, L, layout, gen):
    """(N, 3) float64 positions in the box on the GPU, in random caller order."""
    box = torch.tensor(L, dtype=torch.float64, device="cuda")

    def uniform(*shape):
        return torch.rand(*shape, generator=gen, device="cuda", dtype=torch.float64)

    if layout == "uniform":
        return uniform(N, 3) * box
    if layout == "clustered":
        # 1000 spheres a cluster, log-normal widths (median 3 radii)
        k = max(1, N // 1000)
        centres = uniform(k, 3) * box
        widths = torch.exp(math.log(3.0) + 0.5 * torch.randn(k, generator=gen, device="cuda", dtype=torch.float64))
        c = torch.randint(k, (N,), generator=gen, device="cuda")
        away = torch.randn(N, 3, generator=gen, device="cuda", dtype=torch.float64)
        return torch.remainder(centres[c] + away * widths[c, None], box)
    # spheres of radius 1 on randomly filled lattice sites, each displaced as
    # far as it can be without touching a neighbour
    s = (L[0] * L[1] * L[2] / N) ** (1.0 / 3.0)
    n = [math.ceil(x / s) for x in L]
    site = torch.randperm(n[0] * n[1] * n[2], generator=gen, device="cuda")[:N]
    at = torch.stack((site % n[0], (site // n[0]) % n[1], site // (n[0] * n[1])), 1).to(torch.float64)
    step = box / torch.tensor(n, dtype=torch.float64, device="cuda")
    free = torch.clamp((step - 2.0) / 2.0, min=0.0)
    return torch.remainder((at + 0.5) * step + (2.0 * uniform(N, 3) - 1.0) * free, box)


def _inputs(case, seed):
    """Per system (Y, [F of each right-hand side]) of the case's type on the GPU."""
    gen = torch.Generator("cuda")
    gen.manual_seed(int(seed) * 7919 + 17)
    dt = _types(case)[1]
    out = []
    for s in _systems(case):
        Y = _positions(s["N"], s["L"], case["layout"], gen).to(dt)
        Fs = [torch.randn(s["N"], 3, generator=gen, device="cuda", dtype=torch.float64).to(dt)
              for _ in range(case.get("nrhs", 1))]
        out.append((Y, Fs))
    return out


def prepare(case, seed):
    ffcm = _package()
    T = _types(case)[0]
    systems = _systems(case)
    data = _inputs(case, seed)
    call = case["call"]
    if call == "batch":
        b = ffcm.FFCMBatch(T, systems=systems, kernel_widths_ratio=RATIO, M_G=case["M_G"], viscosity=MU,
                           nrhs=case["nrhs"])
        Y = torch.cat([y for y, _ in data])
        F = torch.cat([f for _, fs in data for f in fs])
        return dict(call=call, batch=b, Y=Y, F=F, V=torch.empty_like(F))
    cfg = ffcm.FFCMConfig(T, kernel_widths_ratio=RATIO, M_G=case["M_G"], viscosity=MU, **systems[0])
    Y, (F,) = data[0]
    state = dict(call=call, cfg=cfg, Y=Y, F=F)
    if call == "host":
        state.update(Y=Y.cpu().numpy(), F=F.cpu().numpy(), V=np.empty((case["N"], 3), T))
    elif call == "mobility":
        state.update(V=torch.empty_like(F))
    elif call in ("operator", "resistance"):
        state.update(M=ffcm.FFCMMobility(cfg, Y), iters=case.get("iters"))
    else:
        # the target: the velocities of isolated spheres
        state.update(target=F / (6.0 * math.pi * MU))
    return state


def run(state):
    ffcm = _package()
    call = state["call"]
    if call == "batch":
        return state["batch"].mobility(state["V"], state["Y"], state["F"])
    if call in ("mobility", "host"):
        return ffcm.mobility(state["V"], state["cfg"], state["Y"], state["F"])
    if call == "operator":
        return state["M"] @ state["F"]
    if call == "resistance":
        # F holds prescribed velocities here
        return ffcm.cg(state["M"], state["F"], reltol=0.0, maxiter=state["iters"])
    J, dY, dF, V = ffcm.objective_gradient(state["cfg"], state["Y"], state["F"], state["target"])
    # the loss in single precision, as an optimiser logs it
    return J.to(torch.float32), dY, dF, V


def work(case):
    """Bytes: particles in and out, and the grid's three components written by
    the spread, read and written by the Stokes solve, read by the
    interpolation. Operations: the transforms (2.5 n log2 n a real component
    and direction), the projector and 10 per stencil point of spread and
    interpolation."""
    w = 8 if case["f64"] else 4
    solves = {"resistance": case.get("iters", 0), "gradient": 2, "batch": case.get("nrhs", 0)}.get(case["call"], 1)
    nbytes = flops = 0.0
    for s in _systems(case):
        M = s["num_grid_points"]
        n = float(M[0] * M[1] * M[2])
        stencil = float(s["N"]) * case["M_G"] ** 3
        nbytes += solves * (9.0 * s["N"] * w + 4 * 3 * n * w)
        flops += solves * (2 * 3 * 2.5 * n * math.log2(n) + 12.0 * n + 2 * 10.0 * stencil)
        if case["call"] == "gradient":
            nbytes += 6.0 * n * w     # u and psi read by the gather
            flops += 22.0 * stencil
    return dict(bytes=nbytes, flops=flops)


# ---- the same in 64 bits ----------------------------------------------------

class _Exact:
    """One system in Float64 torch. The integer choice of each stencil's
    anchor, round(Y / h), is made in the working precision, as the method
    defines it; everything else is 64 bits."""

    def __init__(self, case, system, Y):
        self.dt = Y.dtype
        np_t = _types(case)[0]
        self.M, self.MG, self.N = system["num_grid_points"], case["M_G"], system["N"]
        self.L = [float(np_t(x)) for x in system["L"]]
        self.Rc = float(np_t(system["R_c"]))
        self.h = self.L[0] / self.M[0]
        box_t = torch.tensor(self.L, dtype=torch.float64, device="cuda").to(self.dt)
        inv_h = np_t(1) / (np_t(self.L[0]) / np_t(self.M[0]))
        Yw = torch.remainder(Y, box_t)
        self.anchor = torch.round(Yw * torch.tensor(inv_h, dtype=self.dt, device="cuda")).to(torch.int64)
        self.Y = Yw.to(torch.float64)
        self.box = torch.tensor(self.L, dtype=torch.float64, device="cuda")
        d = SIGMA ** 2 - WIDE ** 2
        self.d = d
        self.a0 = 1.0 - 3.0 * d / (2.0 * WIDE ** 2)
        self.a2 = d / (2.0 * WIDE ** 4)
        wide_a = WIDE * math.sqrt(math.pi)
        self.self_term = (1 / (6 * math.pi * MU) - 1 / (6 * math.pi * MU * wide_a) + d / (12 * MU * wide_a ** 3)
                          - d * d / (32 * MU * WIDE ** 5 * math.sqrt(math.pi ** 3)))
        self._cells()

    # grid part
    def _chunks(self):
        step = max(1, (1 << 25) // self.MG ** 3)
        return [(a, min(self.N, a + step)) for a in range(0, self.N, step)]

    def _stencil(self, a, b, Y):
        """Weights (n, MG^3) and flat grid indices of particles [a, b)."""
        k = torch.arange(self.MG, device="cuda") - self.MG // 2
        g = self.anchor[a:b, :, None] + k                     # (n, 3, MG)
        x2 = (g.to(torch.float64) * self.h - Y[:, :, None]) ** 2
        w = torch.exp(-x2 / (2 * WIDE ** 2)) / math.sqrt(2 * math.pi * WIDE ** 2)
        n = b - a
        r2 = x2[:, 2, :, None, None] + x2[:, 1, None, :, None] + x2[:, 0, None, None, :]
        gw = w[:, 2, :, None, None] * w[:, 1, None, :, None] * w[:, 0, None, None, :]
        gw = (self.a0 + self.a2 * r2) * gw
        i = [torch.remainder(g[:, q], self.M[q]) for q in range(3)]
        at = (i[2][:, :, None, None] * self.M[1] + i[1][:, None, :, None]) * self.M[0] + i[0][:, None, None, :]
        return gw.reshape(n, -1), at.reshape(n, -1)

    def flow(self, F):
        """Velocity grid (3, cells) of the forces F."""
        cells = self.M[0] * self.M[1] * self.M[2]
        f = torch.zeros(3, cells, dtype=torch.float64, device="cuda")
        for a, b in self._chunks():
            w, at = self._stencil(a, b, self.Y[a:b])
            for c in range(3):
                f[c].index_add_(0, at.reshape(-1), (w * F[a:b, c, None]).reshape(-1))
        shape = (self.M[2], self.M[1], self.M[0])
        spec = [torch.fft.rfftn(f[c].view(shape)) for c in range(3)]
        del f

        def waves(m, L, half=False):
            j = torch.arange(m // 2 + 1 if half else m, device="cuda", dtype=torch.float64)
            return 2 * math.pi * (j if half else torch.where(j <= m // 2, j, j - m)) / L

        kx = waves(self.M[0], self.L[0], True)[None, None, :]
        ky = waves(self.M[1], self.L[1])[None, :, None]
        kz = waves(self.M[2], self.L[2])[:, None, None]
        k2 = kx * kx + ky * ky + kz * kz
        k2[0, 0, 0] = 1.0
        along = (kx * spec[0] + ky * spec[1] + kz * spec[2]) / k2
        out = torch.empty(3, cells, dtype=torch.float64, device="cuda")
        for c, k in enumerate((kx, ky, kz)):
            s = (spec[c] - k * along) / (MU * k2)
            spec[c] = None
            s[0, 0, 0] = 0.0
            s = torch.fft.ifft(torch.fft.ifft(s, dim=0), dim=1)
            s[..., 0].imag.zero_()
            if self.M[0] % 2 == 0:
                s[..., -1].imag.zero_()
            out[c] = torch.fft.irfft(s, n=self.M[0], dim=2).reshape(-1)
            del s
        return out

    def gather(self, u):
        v = torch.empty(self.N, 3, dtype=torch.float64, device="cuda")
        for a, b in self._chunks():
            w, at = self._stencil(a, b, self.Y[a:b])
            for c in range(3):
                v[a:b, c] = self.h ** 3 * (w * u[c][at]).sum(1)
        return v

    def gather_gradient(self, u, psi, F, lam):
        g = torch.empty(self.N, 3, dtype=torch.float64, device="cuda")
        for a, b in self._chunks():
            y = self.Y[a:b].clone().requires_grad_(True)
            w, at = self._stencil(a, b, y)
            s = sum(lam[a:b, c, None] * u[c][at] + F[a:b, c, None] * psi[c][at] for c in range(3))
            (g[a:b],) = torch.autograd.grad(self.h ** 3 * (w * s).sum(), y)
        return g

    # pair part: every ordered pair closer than R_c
    def _cells(self):
        m = [max(3, int(x // self.Rc)) for x in self.L]
        c = torch.minimum((self.Y / self.box * torch.tensor(m, device="cuda")).to(torch.int64),
                          torch.tensor(m, device="cuda") - 1)
        key = c[:, 0] + m[0] * (c[:, 1] + m[1] * c[:, 2])
        self.order = torch.argsort(key)
        self.cell, self.m = c[self.order], m
        self.count = torch.bincount(key, minlength=m[0] * m[1] * m[2])
        self.start = torch.cumsum(self.count, 0) - self.count

    def _pairs(self):
        """Chunks (i, j, x) of close pairs, x = Y_i - Y_j (nearest image)."""
        for q in range(27):
            n = [torch.remainder(self.cell[:, k] + (q // 3 ** k) % 3 - 1, self.m[k]) for k in range(3)]
            nb = n[0] + self.m[0] * (n[1] + self.m[1] * n[2])
            cnt, first = self.count[nb], self.start[nb]
            ends = torch.cumsum(cnt, 0).cpu()
            a = 0
            while a < self.N:
                before = int(ends[a - 1]) if a else 0
                b = max(a + 1, int(torch.searchsorted(ends, before + (1 << 25), right=True)))
                c = cnt[a:b]
                i = torch.repeat_interleave(torch.arange(a, b, device="cuda"), c)
                back = torch.cumsum(c, 0) - c
                j = first[i] + torch.arange(i.numel(), device="cuda") - back[i - a]
                i, j = self.order[i], self.order[j]
                x = self.Y[i] - self.Y[j]
                x = x - self.box * torch.round(x / self.box)
                near = ((x * x).sum(1) < self.Rc ** 2) & (i != j)
                yield i[near], j[near], x[near]
                a = b

    def _scalars(self, r2):
        r = torch.sqrt(r2)
        s2, S2, pi, d = SIGMA ** 2, WIDE ** 2, math.pi, self.d
        e = torch.erf(r / (2 * SIGMA)) - torch.erf(r / (2 * WIDE))
        Ds = (4 * pi * s2) ** -1.5 * torch.exp(-r2 / (4 * s2))
        DS = (4 * pi * S2) ** -1.5 * torch.exp(-r2 / (4 * S2))
        q = d * d / 4
        A = (e * (1 / (8 * pi * MU * r) + s2 / (4 * pi * MU * r ** 3)) - 2 * s2 ** 2 / (MU * r2) * Ds
             + (2 * S2 ** 2 / (MU * r2) + d / MU * (1 + 2 * S2 / r2) - q * (2 - r2 / (2 * S2)) / (2 * MU * S2)) * DS)
        B = (e * (1 / (8 * pi * MU * r ** 3) - 3 * s2 / (4 * pi * MU * r ** 5)) + 6 * s2 ** 2 / (MU * r2 ** 2) * Ds
             + (-6 * S2 ** 2 / (MU * r2 ** 2) - d / (MU * r2) * (1 + 6 * S2 / r2) - q / (4 * MU * S2 ** 2)) * DS)
        return A, B

    def correct(self, F):
        v = self.self_term * F
        for i, j, x in self._pairs():
            A, B = self._scalars((x * x).sum(1))
            f = F[j]
            v.index_add_(0, i, A[:, None] * f + (B * (x * f).sum(1))[:, None] * x)
        return v

    def correct_gradient(self, F, lam):
        g = torch.zeros(self.N, 3, dtype=torch.float64, device="cuda")
        for i, j, x in self._pairs():
            x.requires_grad_(True)
            A, B = self._scalars((x * x).sum(1))
            s = (A * (lam[i] * F[j]).sum(1) + B * (x * lam[i]).sum(1) * (x * F[j]).sum(1)).sum()
            (dx,) = torch.autograd.grad(s, x)
            g.index_add_(0, i, dx)
            g.index_add_(0, j, -dx)
        return g

    def apply(self, F):
        return self.gather(self.flow(F)) + self.correct(F)


def exact(case, seed):
    out = []
    for system, (Y, Fs) in zip(_systems(case), _inputs(case, seed)):
        e = _Exact(case, system, Y)
        Fs = [f.to(torch.float64) for f in Fs]
        if case["call"] == "gradient":
            F = Fs[0]
            target = (Fs[0].to(Y.dtype) / (6.0 * math.pi * MU)).to(torch.float64)
            u = e.flow(F)
            V = e.gather(u) + e.correct(F)
            lam = V - target
            psi = e.flow(lam)
            dF = e.gather(psi) + e.correct(lam)
            dY = e.gather_gradient(u, psi, F, lam) + e.correct_gradient(F, lam)
            return 0.5 * (lam * lam).sum().reshape(1), dY, dF, V
        if case["call"] == "resistance":
            # Hestenes-Stiefel from zero
            x, r = torch.zeros_like(Fs[0]), Fs[0].clone()
            p, rr = r.clone(), (r * r).sum()
            for _ in range(case["iters"]):
                q = e.apply(p)
                alpha = rr / (p * q).sum()
                x, r = x + alpha * p, r - alpha * q
                new = (r * r).sum()
                p, rr = r + new / rr * p, new
            return x
        out += [e.apply(f) for f in Fs]
    return torch.cat(out)
