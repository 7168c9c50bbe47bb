"""What this framework is measured on: the work that a program which uses it
has it do, through its public entry points, on arrays that live on the GPU.

A case is one call or a stretch of a run between two outputs:

  helm      pq_helm: one Helmholtz problem in a caller's device array
  pv        pq_pv_inversion: potential vorticity to streamfunction
  batch     pq_batch_helm: many Helmholtz problems of mixed sizes
  basin     Model: CABARET steps of a closed double gyre, psi read back
  channel   the same periodic in j (momentum-corrected inversion)
  leapfrog  the leapfrog scheme of the closed basin
  ensemble  Ensemble: several runs of one configuration, psi of each read

Grids have ii = 2^p + 1 nodes (the row transform's lengths) and any jj; the
basin, the physics and the 1e-7 smoothed-noise initial PV are those of
pequod_b200.workloads.  A mixed-precision run holds its state in 32 bits and
hands its psi on in 32 bits; everything else is FP64.
"""
import ctypes
import math

import numpy as np
import torch

import pequod_b200 as pq
from pequod_b200.workloads import BASIN_CM, LAYERS

SIZES = (65, 129, 257, 513, 1025, 2049)


def listed():
    return [
        # The smallest call: a one-layer elliptic solve inside a host program's own loop.
        dict(name="helm 65x65x1", kind="helm", ii=65, jj=65, layers=1, mixed=False, steps=1),
        # One inversion at a time, on a basin that is not square and odd in j.
        dict(name="pv 513x385x3", kind="pv", ii=513, jj=385, layers=3, mixed=False, steps=1),
        # Independent elliptic problems of one program solved together (the batched workload's sizes).
        dict(name="batch 48", kind="batch", ii=1025, jj=1025, layers=5, mixed=False, steps=48),
        # The default three-layer gyre at 30 km: every launch counts.
        dict(name="basin 129x129x3 f64", kind="basin", ii=129, jj=129, layers=3, mixed=False, steps=40),
        # An adaptive time step on a ragged grid of four layers, mixed precision.
        dict(name="basin 257x161x4 mixed adapt", kind="basin", ii=257, jj=161, layers=4, mixed=True, steps=30,
             adapt=True),
        # A medium run in full precision.
        dict(name="basin 513x513x3 f64", kind="basin", ii=513, jj=513, layers=3, mixed=False, steps=20),
        # The benchmark configuration in both forms.
        dict(name="basin 1025x1025x3 mixed", kind="basin", ii=1025, jj=1025, layers=3, mixed=True, steps=12),
        dict(name="basin 1025x1025x3 f64", kind="basin", ii=1025, jj=1025, layers=3, mixed=False, steps=12),
        # The largest configuration, with the energy diagnostics of its output interval.
        dict(name="basin 2049x2049x5 mixed", kind="basin", ii=2049, jj=2049, layers=5, mixed=True, steps=5,
             energy=True),
        # A zonal channel.
        dict(name="channel 513x320x3 f64", kind="channel", ii=513, jj=320, layers=3, mixed=False, steps=12),
        # The other time scheme.
        dict(name="leapfrog 257x257x3 f64", kind="leapfrog", ii=257, jj=257, layers=3, mixed=False, steps=20),
        # Perturbed copies of one small run.
        dict(name="ensemble 8x129x129x3 mixed", kind="ensemble", ii=129, jj=129, layers=3, mixed=True, steps=100,
             members=8),
    ]


def draw(rng):
    kind = rng.choice(["helm", "pv", "batch", "channel", "leapfrog", "ensemble"] + ["basin"] * 6)
    if kind == "batch":
        return dict(kind=kind, ii=1025, jj=1025, layers=5, mixed=rng.random() < 0.3, steps=rng.randint(8, 60))
    sizes = SIZES[:3] if kind == "ensemble" else SIZES[:5] if kind in ("channel", "leapfrog") else SIZES
    ii = rng.choice(sizes)
    layers = rng.choice([2, 3, 3, 4, 5] if kind == "channel" else [1, 2, 3, 3, 4, 5])
    if rng.random() < 0.3:
        jj = ii
    else:
        jj = int(round(math.exp(rng.uniform(math.log(max(40, ii // 3)), math.log(min(2049, 2 * ii))))))
    c = dict(kind=kind, ii=ii, jj=jj, layers=layers, mixed=False, steps=1)
    if kind in ("helm", "pv"):
        return c
    if kind == "ensemble":
        c.update(mixed=rng.random() < 0.6, members=rng.randint(2, 10))
    elif kind != "leapfrog":
        c.update(mixed=rng.random() < 0.5, adapt=rng.random() < 0.25, energy=rng.random() < 0.3)
    nodes = ii * jj * layers * c.get("members", 1)
    most = 80_000_000 // nodes if kind in ("basin", "ensemble") else 24_000_000 // nodes
    c["steps"] = max(1, min(most, rng.randint(5, 60)))
    return c


def dt_seconds(ii):
    return 1800.0 if ii <= 257 else 900.0 if ii <= 1025 else 300.0


def physical(case):
    H, gp = LAYERS[case["layers"]]
    return dict(layers=case["layers"], dt=dt_seconds(case["ii"]), dx=BASIN_CM / (case["ii"] - 1), H=H, gprime=gp,
                adapt_dt=int(bool(case.get("adapt"))), max_dt=7200.0)


def config(case):
    cfg = pq.Config.from_physical(pq.double_gyre_physical(
        case["ii"], case["jj"], precision=pq.PREC_MIXED if case["mixed"] else pq.PREC_FP64,
        scheme=pq.SCHEME_LEAPFROG if case["kind"] == "leapfrog" else pq.SCHEME_CABARET, **physical(case)))
    cfg.desc.periodic_j = int(case["kind"] == "channel")
    return cfg


def gpu():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def smooth_noise(gen, shape, sigma=3.0):
    """N(0, 1) noise smoothed by a Gaussian of sigma cells, (..., jj, ii)."""
    x = torch.randn(shape, generator=gen, dtype=torch.float64, device=gen.device)
    kj = torch.fft.fftfreq(shape[-2], device=gen.device, dtype=torch.float64)[:, None]
    ki = torch.fft.rfftfreq(shape[-1], device=gen.device, dtype=torch.float64)[None, :]
    ker = torch.exp(-2.0 * (math.pi * sigma) ** 2 * (ki * ki + kj * kj))
    return torch.fft.irfft2(torch.fft.rfft2(x) * ker, s=shape[-2:])


def generator(seed):
    g = torch.Generator(device=gpu())
    g.manual_seed(seed)
    return g


def initial_pv(case, seed):
    """Members' (or leapfrog levels') initial PV, (n, L, jj, ii)."""
    n = 2 if case["kind"] == "leapfrog" else case.get("members", 1)
    t_scale = BASIN_CM / (case["ii"] - 1)
    return 1e-7 * t_scale * smooth_noise(generator(seed), (n, case["layers"], case["jj"], case["ii"]))


def batch_problems(case, seed):
    """Shapes and Helmholtz constants of the batch (those of the problem set,
    not of the seed) and each member's right-hand side: k^-3 random fields."""
    r = np.random.default_rng(case["steps"])
    gen, probs = generator(seed), []
    for _ in range(case["steps"]):
        ii, jj = (int(v) for v in r.choice((65, 129, 257, 513, 1025), 2))
        L = int(r.integers(1, case["layers"] + 1))
        H = tuple(float(h) for h in r.uniform(2.0e4, 4.0e5, L))
        ss = stratification(H, [1.5 * 2.0 ** -k for k in range(L - 1)], BASIN_CM / (ii - 1))["ss"]
        x = torch.randn((L, jj, ii), generator=gen, dtype=torch.float64, device=gen.device)
        kj = torch.fft.fftfreq(jj, device=gen.device, dtype=torch.float64)[:, None]
        ki = torch.fft.rfftfreq(ii, device=gen.device, dtype=torch.float64)[None, :]
        k = torch.sqrt(ki * ki + kj * kj)
        k[0, 0] = math.inf
        f = torch.fft.irfft2(torch.fft.rfft2(x) * k ** -1.5, s=(jj, ii))
        probs.append(((ii, jj, L), ss, f / f.square().mean((1, 2), keepdim=True).sqrt()))
    return probs


def ptr(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def stream_of(handle):
    return torch.cuda.ExternalStream(int(handle))


def prepare(case, seed):
    if case["kind"] == "batch":
        probs = batch_problems(case, seed)
        b = pq.Batch([p[0] for p in probs], [p[1] for p in probs],
                     precision=pq.PREC_MIXED if case["mixed"] else pq.PREC_FP64)
        rhs = [p[2] for p in probs]
        z = [torch.empty_like(r) for r in rhs]
        ptrs = (ctypes.POINTER(ctypes.c_double) * len(z))(*[ptr(t) for t in z])
        return dict(case=case, batch=b, rhs=rhs, z=z, ptrs=ptrs, stream=stream_of(b.stream))
    cfg, ic = config(case), initial_pv(case, seed)
    if case["kind"] == "ensemble":
        e = pq.Ensemble(cfg, case["members"])
        for k in range(case["members"]):
            e.init(k, ic[k].cpu().numpy().transpose(2, 1, 0))
        return dict(case=case, ensemble=e)
    m = pq.Model(cfg)
    out = torch.zeros(ic.shape[1:], dtype=torch.float64, device=ic.device)
    s = dict(case=case, model=m, psi=out)
    if case["kind"] in ("helm", "pv"):
        s.update(rhs=ic[0].contiguous(), stream=stream_of(m.stream))
    else:
        check(pq.lib().pq_init_perturb(m.ctx, ptr(ic.contiguous()), pq.PTR_DEVICE))
    return s


def check(rc):
    if rc != pq.PQ_OK:
        raise RuntimeError(f"pequod_b200 error {rc}")


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "batch":  # each right-hand side into its in/out array, then one call
        with torch.cuda.stream(state["stream"]):
            torch._foreach_copy_(state["z"], state["rhs"])
        check(pq.lib().pq_batch_helm(state["batch"].ctx, state["ptrs"], pq.PTR_DEVICE))
        return state["z"]
    if kind == "ensemble":
        e = state["ensemble"]
        e.step(case["steps"])
        psi = [m.sdata("psi") for m in e.members]
        return [p.astype(np.float32) for p in psi] if case["mixed"] else psi
    m, psi = state["model"], state["psi"]
    if kind == "helm":
        with torch.cuda.stream(state["stream"]):
            psi.copy_(state["rhs"])
        check(pq.lib().pq_helm(m.ctx, ptr(psi), pq.PTR_DEVICE))
        return psi
    if kind == "pv":
        check(pq.lib().pq_pv_inversion(m.ctx, ptr(state["rhs"]), ptr(psi), pq.PTR_DEVICE))
        return psi
    # A run's stretch between two outputs: steps, psi to a device array, the
    # NaN check that also waits, the diagnostics where they are asked for.
    m.step_async(case["steps"] - 1)
    m.step_exchange(None, psi.data_ptr(), pq.PTR_DEVICE)
    m.check()
    out = [psi.float() if case["mixed"] else psi]
    if case.get("energy"):
        ekin, epot = m.energy()
        out += [ekin, epot, m.cfl()]
    return out


def work(case):
    """Bytes and flops of a pass.  A step reads and writes the prognostic
    fields once (22 + 1/L values per cell-layer FP64, 20 + 1/L in 32 bits and
    psi's two in the mixed form) and does two row transforms, a tridiagonal
    solve, the modal products and about 150 operations of advection; a
    leapfrog sub-step holds 14 fields; a solve reads its input and writes
    its result."""
    def elliptic(ii, jj, L):
        return ii * jj * L * (2 * (2.5 * math.log2(ii) + 10) + 14 + 4 * L)

    if case["kind"] == "batch":
        r = np.random.default_rng(case["steps"])
        nbytes = flops = 0
        for _ in range(case["steps"]):
            ii, jj = (int(v) for v in r.choice((65, 129, 257, 513, 1025), 2))
            L = int(r.integers(1, case["layers"] + 1))
            r.uniform(2.0e4, 4.0e5, L)
            nbytes += 16 * ii * jj * L
            flops += elliptic(ii, jj, L)
        return dict(bytes=nbytes, flops=flops)
    ii, jj, L = case["ii"], case["jj"], case["layers"]
    nodes = ii * jj * L
    if case["kind"] in ("helm", "pv"):
        return dict(bytes=16 * nodes, flops=elliptic(ii, jj, L))
    n = case["steps"] * case.get("members", 1)
    if case["kind"] == "leapfrog":
        per = 8 * 14
    else:
        per = 4 * (20 + 1 / L) + 16 if case["mixed"] else 8 * (22 + 1 / L)
    return dict(bytes=n * nodes * per, flops=n * (elliptic(ii, jj, L) + 150 * nodes))


# ---------------------------------------------------------------------------
# The same in 64 bits with plain torch: fields (L, jj, ii), the equations of
# the reference (qg3p_helmholtz.F90, qg3p_aux.F90, qg3p_diagnostics.F90).


def stratification(H, gprime, l_scale, f0=9.4e-5):
    L = len(H)
    S, s1, s2 = np.zeros((L, L)), np.zeros(L), np.zeros(L)
    for k in range(L - 1):
        f2g = f0 * f0 / gprime[k] * l_scale ** 2
        s2[k], s1[k + 1] = f2g / H[k], f2g / H[k + 1]
    for k in range(L):
        S[k, k] = -s1[k] - s2[k]
        if k + 1 < L:
            S[k, k + 1], S[k + 1, k] = s2[k], s1[k + 1]
    w = np.ones(L)
    for k in range(L - 1):
        w[k + 1] = w[k] * math.sqrt(S[k, k + 1] / S[k + 1, k])
    val, vec = np.linalg.eigh(w[:, None] * S / w[None, :])
    order = np.argsort(-val)
    m2z, ss = vec[:, order] / w[:, None], -val[order]
    m2z[:, 0], ss[0] = 1.0, 0.0
    return dict(s1=s1, s2=s2, ss=ss, m2z=m2z, z2m=np.linalg.inv(m2z))


class Equations:
    """The non-dimensional problem of a case."""

    def __init__(self, case):
        p = physical(case)
        self.case, self.dev = case, gpu()
        self.ii, self.jj, self.L = case["ii"], case["jj"], case["layers"]
        self.per = case["kind"] == "channel"
        ii, jj, L = self.ii, self.jj, self.L
        ls = p["dx"]
        for k, v in stratification(p["H"], p["gprime"], ls).items():
            setattr(self, k, torch.tensor(v, dtype=torch.float64, device=self.dev))
        self.h = torch.tensor(p["H"], dtype=torch.float64, device=self.dev) / ls
        self.dt, self.max_dt, self.cfl, self.grow = p["dt"] / ls, p["max_dt"] / ls, 0.1, 1.5
        self.beta, self.nu, self.vb = 1.8e-13 * ls * ls, 1.0e6 / ls, 1.0e-7 * ls
        alpha = ls / 120.0e5
        self.slip = alpha / (alpha + 3.0)
        i = torch.arange(ii, device=self.dev)
        j = torch.arange(jj, device=self.dev)[:, None]
        y = 0.5 - i.double() / (ii - 1)
        f = torch.where(y < 0, -torch.sin(math.pi * (0.5 + y) / 0.5), torch.sin(math.pi * y / 0.5))
        self.wind = torch.zeros((L, jj, ii), dtype=torch.float64, device=self.dev)
        self.wind[0] = 0.8 / (ii - 1) / self.h[0] * 2.0 * math.pi * f
        self.i, self.j = i, j
        every = torch.ones((jj, 1), dtype=torch.bool, device=self.dev)
        in_j = every if self.per else (j >= 1) & (j <= jj - 2)
        self.inner = (i >= 1) & (i <= ii - 2) & in_j
        self.iface = (i >= 1) & in_j
        self.jface = (i >= 1) & (i <= ii - 2) & (every if self.per else j >= 1)


    def helm(self, f, ss):
        """(d_xx + d_yy - ss) phi = f on the interior, zero walls; (n, jj, ii)."""
        return solve_helm(f, ss, self.per)

    def correction(self):
        one = self.inner.double().expand(self.L, -1, -1)
        ss = self.ss[:, None, None]
        if not self.per:
            p = self.helm(one, self.ss)
            mean = p.sum((1, 2), keepdim=True) / ((self.ii - 1) * (self.jj - 1))
            return ((1 + ss * p) / (1 + ss * mean),)
        fs = []
        for wall in (0, self.ii - 1):
            rhs = torch.zeros((self.L, self.jj, self.ii), dtype=torch.float64, device=self.dev)
            rhs[:, :, 1 if wall == 0 else self.ii - 2] -= 1.0
            p = self.helm(rhs, self.ss)
            p[:, :, wall] = 1.0
            fs.append(p)
        return tuple(fs)

    def wall_pv(self, p):
        """Mean PV of the two channel walls of each mode, (L, 2)."""
        w = []
        for a, b, c in ((0, 1, 2), (-1, -2, -3)):
            v = self.slip * (-3.5 * p[:, :, a] + 4.0 * p[:, :, b] - 0.5 * p[:, :, c])
            w.append((v - self.ss[:, None] * p[:, :, a]).mean(1))
        return torch.stack(w, 1)

    def invert(self, z):
        if not hasattr(self, "corr"):
            self.corr = self.correction()
        z = torch.where(self.inner, z, 0.0)
        phi = self.helm(torch.einsum("ml,lji->mji", self.z2m, z), self.ss)
        if self.per:
            zb = self.wall_pv(phi)
            a = torch.stack([self.wall_pv(c) for c in self.corr], 2)
            for m in range(1, self.L):
                q = torch.linalg.solve(a[m], zb[m])
                phi[m] -= q[0] * self.corr[0][m] + q[1] * self.corr[1][m]
            return torch.einsum("lm,mji->lji", self.m2z, phi)
        c = phi.sum((1, 2)) / ((self.ii - 1) * (self.jj - 1))
        phi[1:] -= c[1:, None, None] * self.corr[0][1:]
        return phi[0] - c[0] + torch.einsum("lm,mji->lji", self.m2z[:, 1:], phi[1:])

    def couple(self, p):
        out = torch.zeros_like(p)
        if self.L > 1:
            out[1:] += self.s1[1:, None, None] * (p[1:] - p[:-1])
            out[:-1] += self.s2[:-1, None, None] * (p[:-1] - p[1:])
        return out

    def rel(self, z, p):
        r = torch.where(self.inner, z + self.couple(p), 0.0)
        lap = lambda a, b, c: self.slip * (-3.5 * a + 4.0 * b - 0.5 * c)  # noqa: E731
        r[:, :, 0] = lap(p[:, :, 0], p[:, :, 1], p[:, :, 2])
        r[:, :, -1] = lap(p[:, :, -1], p[:, :, -2], p[:, :, -3])
        if not self.per:
            r[:, 0] = lap(p[:, 0], p[:, 1], p[:, 2])
            r[:, -1] = lap(p[:, -1], p[:, -2], p[:, -3])
        return r

    def with_wall_pv(self, z, r, p):
        return torch.where(self.inner, z, r - self.couple(p))

    def laplacian(self, r):
        return -4 * r + E(r) + W(r) + N(r) + S(r)

    # ---- CABARET ----------------------------------------------------------

    def start(self, ic):
        z = torch.where(self.i * (self.ii - 1 - self.i) > 0, ic, 0.0)
        if not self.per:
            z[:, 0] = z[:, -1] = 0.0
        self.psi = self.invert(z)
        zero = torch.zeros_like(z)
        self.z = self.with_wall_pv(z, self.rel(z, self.psi), self.psi)
        self.res = self.rb = self.ui = self.uim = self.ujm = self.fi = self.fj = zero
        self.ta = self.tu = 0.5

    def extrapolate(self, u, f, z, zo, back, ahead, first, last):
        """Face values by the limited upwind extrapolation; back(x) is x one
        node or face behind, `first` / `last` the faces next to a wall."""
        pos = u >= 0
        u2 = torch.where(pos, back(u), ahead(u))
        f2 = torch.where(pos, back(f), ahead(f))
        n, o = torch.where(pos, back(z), z), torch.where(pos, back(zo), zo)
        wall = torch.where(pos, first, last)
        f2 = torch.where(wall, n, f2)
        sign = torch.where(pos, 1.0, -1.0)
        d = -2 * (n - o) - self.dt * 0.5 * (u + u2) * sign * (f - f2)
        d = torch.where(wall, -(n - o), d)
        hi = torch.maximum(torch.maximum(f, f2), n) - d
        lo = torch.minimum(torch.minimum(f, f2), n) - d
        return torch.maximum(torch.minimum(2 * n - f2, hi), lo)

    def step(self):
        dt, ta, tu = self.dt, self.ta, self.tu
        rb = torch.where(self.inner, dt * 0.5 * (E(self.ui) + self.ui) * self.beta, 0.0)
        zo = self.z
        z = torch.where(self.inner, zo + 0.5 * dt * self.res + (1 + ta) * rb - ta * self.rb, 0.0)
        self.rb = rb
        p = self.psi = self.invert(z)
        r = self.rel(z, p)
        f = self.wind + self.nu * self.laplacian(r)
        f[-1] -= self.vb * r[-1]
        z = torch.where(self.inner, z + dt * f, r - self.couple(p))
        pe = 0.25 * (p + S(p) + W(p) + S(W(p)))
        uim = torch.where(self.iface, pe - N(pe), 0.0)
        ujm = torch.where(self.jface, E(pe) - pe, 0.0)
        ui = torch.where(self.iface, (1 + tu) * uim - tu * self.uim, 0.0)
        uj = torch.where(self.jface, (1 + tu) * ujm - tu * self.ujm, 0.0)
        i, j, never = self.i, self.j, torch.zeros_like(self.j, dtype=torch.bool)
        fi = self.extrapolate(ui, self.fi, z, zo, W, E, i == 1, i == self.ii - 1)
        fj = self.extrapolate(uj, self.fj, z, zo, S, N, never if self.per else j == 1,
                              never if self.per else j == self.jj - 1)
        self.fi, self.fj = torch.where(self.iface, fi, 0.0), torch.where(self.jface, fj, 0.0)
        a, b = ui * self.fi, uj * self.fj
        self.res = torch.where(self.inner, -(E(a) - a + N(b) - b), 0.0)
        self.z = z + 0.5 * dt * self.res
        self.ui, self.uim, self.ujm = ui, uim, ujm
        top = max(float(ui.abs().max()), float(uj.abs().max()))
        self.cfl_now = top * dt
        if self.case.get("adapt"):
            self.dt = min(self.cfl / top, dt * self.grow, self.max_dt)
            self.ta, self.tu = 0.5 * self.dt / dt, self.dt / (dt + self.dt)

    def energy(self):
        p, htot = self.psi, self.h.sum()
        scale = 1.0 / ((self.ii - 1) * (self.jj if self.per else self.jj - 1))
        back = S(p)
        ek = 0.25 * ((W(p) + p - S(W(p)) - back) ** 2 + (back + p - S(W(p)) - W(p)) ** 2)
        ek = ek[:, :, 1:] if self.per else ek[:, 1:, 1:]
        ekin = 0.5 * scale * self.h / htot * ek.sum((1, 2))
        w = torch.where((self.i == 0) | (self.i == self.ii - 1), 0.5, 1.0).double()
        wj = torch.ones((self.jj, 1), dtype=torch.float64, device=self.dev)
        if not self.per:
            wj[0] = wj[-1] = 0.5
        d = (p[:-1] - p[1:]).square() * w * wj
        epot = scale * (0.5 * self.s2[:-1] * self.h[:-1] / htot * d.sum((1, 2))).sum()
        return [ekin, float(epot), self.cfl_now]

    # ---- leapfrog ---------------------------------------------------------

    def tendency(self, p, r, rp):
        q = self.beta * (0.5 * (self.ii - 3) - self.i.double()) + r
        if self.L > 1:
            q = q.clone()
            q[1:] += self.s1[1:, None, None] * p[:-1]
            q[:-1] += self.s2[:-1, None, None] * p[1:]
        ne, nw, se, sw = N(E(p)), N(W(p)), S(E(p)), S(W(p))
        jac = 0.25 * (N(q) * (nw - ne) - S(q) * (sw - se) - W(q) * (nw - sw) + E(q) * (ne - se))
        lap = self.laplacian(rp)
        if self.L == 1:
            return jac + self.wind + self.nu * (lap - self.vb * rp)
        out = jac + self.wind + self.nu * lap
        out[-1] -= self.vb * rp[-1]
        return out

    def leapfrog(self, ic, steps):
        zs, ps, rs, olds = [], [], [], []
        for lv in range(2):
            z = torch.where(self.inner, ic[lv], 0.0)
            p = self.invert(z)
            r = self.rel(z, p)
            z = self.with_wall_pv(z, r, p)
            zs.append(z), ps.append(p), rs.append(r), olds.append(z)

        def settle(lv, keep):
            ps[lv] = self.invert(zs[lv])
            rs[lv] = self.rel(zs[lv], ps[lv])
            zs[lv] = self.with_wall_pv(zs[lv], rs[lv], ps[lv])
            if keep:
                olds[lv] = zs[lv]

        zs[1] = torch.where(self.inner, zs[0] + self.dt * self.tendency(ps[0], rs[0], rs[0]), zs[1])
        settle(1, True)
        nu, al = 0.02, 0.5
        w21, w11 = 0.5 * nu * al, -0.5 * nu * (1 - al)
        for k in range(steps):
            lv, m = k % 2, 1 - k % 2
            new = zs[lv] + torch.where(self.inner, 2 * self.dt * self.tendency(ps[m], rs[m], rs[lv]), 0.0)
            zl = w11 * olds[lv] - 2 * w11 * zs[m] + (1 + w11) * new
            zs[m] = olds[m] = w21 * (olds[lv] + new) + (1 - 2 * w21) * zs[m]
            zs[lv] = zl
            settle(lv, False)
        return ps[0]


def E(x):
    return torch.roll(x, -1, -1)


def W(x):
    return torch.roll(x, 1, -1)


def N(x):
    return torch.roll(x, -1, -2)


def S(x):
    return torch.roll(x, 1, -2)


def sine(x, dim):
    """DST-I over the interior of `dim`."""
    n = x.shape[dim]
    zero = torch.zeros_like(x.narrow(dim, 0, 1))
    y = torch.fft.rfft(torch.cat([zero, x, zero, -x.flip(dim)], dim), dim=dim).imag
    return -0.5 * y.narrow(dim, 1, n)


def solve_helm(f, ss, periodic):
    L, jj, ii = f.shape
    k = torch.arange(1, ii - 1, device=f.device, dtype=torch.float64)
    lam = -4 * torch.sin(k * math.pi / (2 * (ii - 1))) ** 2 - ss[:, None, None]
    out = torch.zeros_like(f)
    if periodic:
        x = torch.fft.fft(sine(f[:, :, 1:-1], 2), dim=1)
        q = torch.arange(jj, device=f.device, dtype=torch.float64)[:, None]
        x = x / (lam - 4 * torch.sin(q * math.pi / jj) ** 2)
        out[:, :, 1:-1] = sine(torch.fft.ifft(x, dim=1).real, 2) * 2.0 / (ii - 1)
        return out
    x = sine(sine(f[:, 1:-1, 1:-1], 2), 1)
    q = torch.arange(1, jj - 1, device=f.device, dtype=torch.float64)[:, None]
    x = x / (lam - 4 * torch.sin(q * math.pi / (2 * (jj - 1))) ** 2)
    out[:, 1:-1, 1:-1] = sine(sine(x, 1), 2) * 4.0 / ((ii - 1) * (jj - 1))
    return out


def helm_result(f, ss):
    """helm's in-place semantics: the interior solved, row ii of the interior
    rows and column 1's interior zeroed, the other boundary values kept."""
    out = f.clone()
    out[:, 1:-1, 1:-1] = solve_helm(f, ss, False)[:, 1:-1, 1:-1]
    out[:, 1:-1, -1] = 0.0
    out[:, 0, 1:-1] = 0.0
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return [helm_result(f, torch.tensor(ss, dtype=torch.float64, device=f.device))
                for _, ss, f in batch_problems(case, seed)]
    ic = initial_pv(case, seed)
    q = Equations(case)
    if kind == "helm":
        return helm_result(ic[0], q.ss)
    if kind == "pv":
        return q.invert(ic[0])
    if kind == "leapfrog":
        return [q.leapfrog(ic, case["steps"])]
    runs = []
    for k in range(case.get("members", 1)):
        q.start(ic[k])
        for _ in range(case["steps"]):
            q.step()
        runs.append(q.psi)
    if kind == "ensemble":
        return [p.permute(2, 1, 0) for p in runs]
    return runs + (q.energy() if case.get("energy") else [])
