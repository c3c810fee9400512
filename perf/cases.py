"""The work that users of fasttools2d_gb300 have it do, as cases that can be timed.

Each case is one call (or one call and its backward pass) through the public
entry points: the drivers on host arrays, the composites on CUDA tensors, the
MEX gateways, the autograd binding and the many-density ``Geometry``.  Sizes
are those of the repository's workloads and tests: xi rc near 4.8 and
M / xi near 3.15 with P = 24 (tolerance about 1e-10), xi rc near 3.6 and
M / xi near 2.4 with P = 12 for the FP32-grid form (tolerance about 1e-6).
"""
import functools
import math

import numpy as np
import torch

import fasttools2d_gb300 as ft
from fasttools2d_gb300.autograd import stokes_ewald_torch

DEV = "cuda:0"


def listed():
    def case(name, op, ns, nt, xi, nside, M, P=24, Ly=1, pts="uniform", **more):
        return dict({"name": name, "op": op, "pts": pts, "ns": ns, "nt": nt, "xi": float(xi),
                     "nside": nside, "M": M, "P": P, "Ly": Ly, "precision": "fp64", "nrhs": 1},
                    **more)

    return [
        # the smallest call: a Stokeslet sum of a thousand particles on themselves
        case("slp_1k_self", "slp", 1000, 0, 19.2, 4, 64),
        # the smallest differentiated call: one gradient step of an optimisation
        case("grad_1500", "grad", 1500, 1500, 36.0, 6, 96),
        # the MATLAB driver on host arrays; it chooses xi, the boxes and the grid itself
        case("driver_host_20k", "driver", 20000, 20011, 0.0, 0, 0),
        # an ordinary sum on ragged point sets, both kernels
        case("stokes_50k_ragged", "stokes", 50021, 20003, 200.0, 45, 640),
        # one application inside a solver: droplet boundaries on themselves, one density
        case("solver_dlp_32k", "geometry", 32768, 0, 120.0, 25, 384, pts="circles", kinds="dlp"),
        # a double-layer potential evaluated away from the boundaries that carry it
        case("dlp_circles_64k", "dlp", 65536, 65536, 60.0, 12, 192, pts="circles"),
        # the four gateways' Stokeslet pair on a non-square box, as existing MEX callers use it
        case("mex_slp_rect_131k", "mex_slp", 131071, 131071, 215.0, 45, 676, Ly=2),
        # forward and backward at the size of a differentiable simulation
        case("grad_262k", "grad", 262144, 262144, 430.0, 90, 1344),
        # several densities at once on one geometry (a block solver)
        case("geometry_4rhs_262k", "geometry", 262144, 262144, 430.0, 90, 1344, kinds="both",
             nrhs=4),
        # a million points on a million, in full precision and in the FP32-grid form
        case("stokes_1m", "stokes", 1 << 20, 1 << 20, 860.0, 178, 2688),
        case("stokes_1m_fp32grid", "stokes", 1 << 20, 1 << 20, 860.0, 238, 2048, P=12,
             precision="fp32_grid"),
    ]


def draw(rng):
    op = rng.choice(["slp", "dlp", "stokes", "stokes", "grad", "geometry", "mex_slp", "driver"])
    most = {"grad": 2 ** 18, "geometry": 2 ** 18, "driver": 2 ** 16}.get(op, 700000)
    low = op == "stokes" and rng.random() < 0.35
    pts = "circles" if op in ("dlp", "geometry") and rng.random() < 0.6 else "uniform"
    if pts == "circles":
        most = 65536
    ns = int(math.exp(rng.uniform(math.log(1000), math.log(most))))
    nt = 0 if op in ("slp", "geometry") and rng.random() < 0.5 else \
        max(1, min(most, int(ns * math.exp(rng.uniform(-1.2, 1.2)))))
    Ly = 2 if rng.random() < 0.2 and pts == "uniform" else 1
    # points per box as a user chooses them, boxes larger along boundaries
    nb = rng.uniform(20, 45) if pts == "uniform" else rng.uniform(60, 200)
    nside = max(3, round(math.sqrt(ns / nb / Ly)))
    xi = round((rng.uniform(3.5, 3.7) if low else rng.uniform(4.6, 5.0)) * nside, 2)
    # half of the grids as rounded up to a good length, half as the estimates give them
    M = int(xi * (rng.uniform(2.3, 2.5) if low else rng.uniform(3.1, 3.4)))
    M = max(48, (M + 31) // 32 * 32 if rng.random() < 0.5 else 2 * (M // 2))
    case = {"op": op, "pts": pts, "ns": ns, "nt": nt, "xi": xi, "nside": nside, "M": M,
            "P": rng.choice([10, 12, 14]) if low else rng.choice([20, 24, 24, 26]), "Ly": Ly,
            "precision": "fp32_grid" if low else "fp64", "nrhs": 1}
    if op == "geometry":
        case["kinds"] = rng.choice(["slp", "dlp", "both"])
        case["nrhs"] = rng.choice([1, 1, 2, 4])
    if op == "driver":
        case.update(xi=0.0, nside=0, M=0, P=24, Ly=1, nt=max(nt, 1))
    return case


# ----------------------------------------------------------------------------
# inputs
# ----------------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _plan(precision):
    """One plan per precision form, as a program keeps it."""
    if precision == "fp64":
        return ft.default_plan(0)
    plan = ft.Plan(0)
    plan.set_precision(precision)
    return plan


def _circles(gen, n):
    """8 non-overlapping circles of radii U(0.05, 0.1): n boundary points with
    normals and a density of low Fourier modes times the quadrature weight."""
    rnd = lambda *s: torch.rand(*s, generator=gen, device="cpu", dtype=torch.float64)
    rows = []
    while len(rows) < 8:
        r, x, y = 0.05 + 0.05 * rnd(1).item(), rnd(1).item(), rnd(1).item()
        apart = lambda d: abs((d + 0.5) % 1.0 - 0.5)
        if all(math.hypot(apart(x - a), apart(y - b)) > r + q for a, b, q in rows):
            rows.append((x, y, r))
    circ = torch.tensor(rows, dtype=torch.float64)
    amp = torch.randn(8, 9, 2, 2, generator=gen, dtype=torch.float64)
    which = torch.arange(n) * 8 // n
    first = torch.searchsorted(which, torch.arange(8))
    count = torch.bincount(which, minlength=8)
    th = 2 * math.pi * (torch.arange(n) - first[which]).double() / count[which]
    c = circ.to(DEV)[which.to(DEV)]
    th, amp = th.to(DEV), amp.to(DEV)[which.to(DEV)]
    nrm = torch.stack([torch.cos(th), torch.sin(th)], 1)
    modes = torch.arange(9, device=DEV, dtype=torch.float64)[None, :] * th[:, None]
    f = (amp[:, :, 0] * torch.cos(modes)[..., None] + amp[:, :, 1] * torch.sin(modes)[..., None])
    wq = 2 * math.pi * c[:, 2:] / count.to(DEV)[which.to(DEV)].double()[:, None]
    return c[:, :2] + c[:, 2:] * nrm, f.sum(1) * wq, nrm, circ


def _outside(gen, n, circ):
    got, have = [], 0
    c = circ.to(DEV)
    while have < n:
        p = torch.rand(2 * n + 64, 2, generator=gen, device=DEV, dtype=torch.float64)
        d = torch.remainder(p[:, None, :] - c[None, :, :2] + 0.5, 1.0) - 0.5
        p = p[(d.square().sum(2) > c[None, :, 2] ** 2).all(1)]
        got.append(p)
        have += len(p)
    return torch.cat(got)[:n].contiguous()


@functools.lru_cache(maxsize=1)
def _inputs_of(key, seed):
    case = dict(key)
    gen = torch.Generator(DEV).manual_seed(seed)
    box = torch.tensor([1.0, float(case["Ly"])], device=DEV, dtype=torch.float64)
    ns, nt, nrhs = case["ns"], case["nt"], case["nrhs"]
    randn = lambda *s: torch.randn(*s, generator=gen, device=DEV, dtype=torch.float64)
    rand = lambda n: torch.rand(n, 2, generator=gen, device=DEV, dtype=torch.float64) * box
    if case["pts"] == "circles":
        ps, fd, nrm, circ = _circles(torch.Generator().manual_seed(seed), ns)
        pt = _outside(gen, nt, circ) if nt else ps
        scale = fd.square().mean().sqrt()
        fs = randn(nrhs, ns, 2) * scale
        fd = torch.stack([fd] + [randn(ns, 2) * scale for _ in range(nrhs - 1)])
    else:
        ps = rand(ns)
        pt = rand(nt) if nt else ps
        fs, fd = randn(nrhs, ns, 2), randn(nrhs, ns, 2)
        th = 2 * math.pi * torch.rand(ns, generator=gen, device=DEV, dtype=torch.float64)
        nrm = torch.stack([torch.cos(th), torch.sin(th)], 1)
    out = {"ps": ps, "pt": pt, "fs": fs, "fd": fd, "n": nrm}
    if case["op"] == "grad":
        out["ws"], out["wd"] = randn(nt, 2), randn(nt, 2)
    if case["op"] == "mex_slp":           # the gateways take wrapped points
        out["ps"], out["pt"] = _wrap(ps, case["Ly"]), _wrap(pt, case["Ly"])
    return out


def _inputs(case, seed):
    return dict(_inputs_of(tuple(sorted((k, v) for k, v in case.items() if k != "name")), seed))


def _params(case):
    return ft.EwaldParams.derived(case["xi"], case["nside"], case["nside"] * case["Ly"],
                                  case["M"], case["M"] * case["Ly"], case["P"], 1.0,
                                  float(case["Ly"]))


def prepare(case, seed):
    s = _inputs(case, seed)
    _inputs_of.cache_clear()
    s["op"], s["plan"] = case["op"], _plan(case["precision"])
    s["fs1"], s["fd1"] = s["fs"][0].contiguous(), s["fd"][0].contiguous()
    if case["op"] == "driver":
        host = lambda a: tuple(np.ascontiguousarray(c) for c in a.T.cpu().numpy())
        s.update(hs=host(s["ps"]), ht=host(s["pt"]), hf=host(s["fs1"]))
        return s
    s["prm"] = _params(case)
    if case["op"] == "grad":
        for k in ("ps", "fs1", "fd1", "n"):
            s[k].requires_grad_(True)
    if case["op"] == "geometry":
        s["geom"] = ft.Geometry(s["ps"], s["pt"], s["prm"], n=s["n"], kinds=case["kinds"],
                                plan=s["plan"])
    return s


def run(s):
    op, plan = s["op"], s["plan"]
    if op == "slp":
        return ft.slp_ewald(s["ps"], s["pt"], s["fs1"], s["prm"], plan=plan)
    if op == "dlp":
        return ft.dlp_ewald(s["ps"], s["pt"], s["fd1"], s["n"], s["prm"], plan=plan)
    if op == "stokes":
        return ft.stokes_ewald(s["ps"], s["pt"], s["fs1"], s["fd1"], s["n"], s["prm"], plan=plan)
    if op == "grad":
        u = stokes_ewald_torch(s["ps"], s["pt"], s["fs1"], s["fd1"], s["n"], s["prm"], plan)
        g = torch.autograd.grad(u, (s["ps"], s["fs1"], s["fd1"], s["n"]), (s["ws"], s["wd"]))
        return [x.detach() for x in u] + list(g)
    if op == "geometry":
        return [u for u in s["geom"].apply(s["fs"], s["fd"]) if u is not None]
    if op == "mex_slp":
        p = s["prm"]
        return (ft.mex_stokes_slp_real(s["ps"], s["pt"], s["fs1"], p.xi, p.nside_x, p.nside_y,
                                       p.Lx, p.Ly, plan=plan),
                ft.mex_stokes_slp_kspace(s["ps"], s["pt"], p.xi, p.eta, s["fs1"], p.Mx, p.My,
                                         p.Lx, p.Ly, p.w, p.P, plan=plan))
    return ft.StokesSLP_ewald_2p(*s["hs"], *s["ht"], *s["hf"], 1.0, 1.0, plan=plan)


# ----------------------------------------------------------------------------
# what a pass cannot do without
# ----------------------------------------------------------------------------
def work(case):
    ns, op, nrhs = case["ns"], case["op"], case["nrhs"]
    nt = case["nt"] or ns
    kind = {"slp": "slp", "mex_slp": "slp", "driver": "slp", "dlp": "dlp"}.get(
        op, case.get("kinds", "both"))
    nin, nout = {"slp": (2, 2), "dlp": (3, 2), "both": (5, 4)}[kind]
    if op == "driver":                    # about what the driver chooses at tolerance 1e-16
        nside = math.ceil(math.sqrt((ns + nt) / (24 * round(math.log2(ns + nt)))))
        M, P, xi = 24 * nside, 24, 6.0 * nside
    else:
        nside, M, P, xi = case["nside"], case["M"], case["P"], case["xi"]
    vectors = ns * (1 + (kind != "dlp") * nrhs + (kind != "slp") * (nrhs + 1)) + \
        nt * (1 + (nout // 2) * nrhs)
    # pairs in the cutoff disc; about 40 operations for exp, E1 and 1/r^2 and
    # 20 for each kernel's contraction
    pairs = math.pi * ns * nt / (nside * nside * case["Ly"])
    if case["pts"] == "circles":          # points near boundaries see the boundary's own
        pairs *= 3.0
    G = M * M * case["Ly"]
    stencil = (P + 1) ** 2
    flops = nrhs * (pairs * (40 + 10 * nout) + 2 * stencil * (ns * nin + nt * nout) +
                    2.5 * G * math.log2(G) * (nin + nout) + 20 * G)
    if op == "grad":                      # the backward pass: the transposed sums and gradients
        vectors += ns * 4 + nt * 2 + ns * 4
        flops += pairs * 120 + 2 * stencil * (nt * 4 + ns * 15) + \
            2.5 * G * math.log2(G) * (4 + 5) + 20 * G
    return {"bytes": 16.0 * vectors, "flops": float(flops)}


# ----------------------------------------------------------------------------
# the same sums in plain 64-bit torch
# ----------------------------------------------------------------------------
def _wrap(p, Ly):
    L = torch.tensor([1.0, float(Ly)], device=p.device, dtype=torch.float64)
    return torch.remainder(p + L / 2, L) - L / 2


class _E1(torch.autograd.Function):
    """E1(x) for x > 0: the power series below 1.5, the continued fraction above."""

    @staticmethod
    def forward(ctx, x):
        ctx.save_for_backward(x)
        a = x.clamp(max=1.5)
        s, t = torch.zeros_like(a), torch.ones_like(a)
        for k in range(1, 26):
            t = -t * a / k
            s = s - t / k
        small = s - torch.log(a) - 0.57721566490153286061
        b = x.clamp(min=1.5)
        f = torch.zeros_like(b)
        for k in range(64, 0, -1):
            f = k * k / (b + (2 * k + 1) - f)
        return torch.where(x < 1.5, small, torch.exp(-b) / (b + 1 - f))

    @staticmethod
    def backward(ctx, g):
        x, = ctx.saved_tensors
        return -g * torch.exp(-x) / x


def _pairs(ps, pt, nx, ny, Ly, most=1 << 25):
    """Pairs of the real-space sum, (target, source, offset s - t) a chunk at a
    time: every pair of a box, and neighbour boxes' within the box's size."""
    L, n = (1.0, float(Ly)), (nx, ny)
    cell = lambda p: [torch.floor(n[c] * (p[:, c] / L[c] + 0.5)).long().clamp(0, n[c] - 1)
                      for c in (0, 1)]
    sx, sy = cell(ps)
    tx, ty = cell(pt)
    sbox = sy * nx + sx
    order = torch.argsort(sbox)
    count = torch.bincount(sbox, minlength=nx * ny)
    start = torch.cumsum(count, 0) - count
    torder = torch.argsort(ty * nx + tx)
    per = max(1, int(most / max(1, 4 * int(count.max()))))
    cut2 = 1.0 * Ly / nx / ny
    for t0 in range(0, len(pt), per):
        t = torder[t0:t0 + per]
        for ox in (-1, 0, 1):
            for oy in (-1, 0, 1):
                ux, uy = tx[t] + ox, ty[t] + oy
                wx, wy = torch.remainder(ux, nx), torch.remainder(uy, ny)
                b = wy * nx + wx
                m = count[b]
                ti = torch.repeat_interleave(t, m)
                if not len(ti):
                    continue
                lead = torch.repeat_interleave(start[b] - (torch.cumsum(m, 0) - m), m)
                si = order[torch.arange(len(ti), device=ti.device) + lead]
                z = torch.stack([L[0] * (ux - wx) / nx, L[1] * (uy - wy) / ny], 1)
                d = ps[si] - (pt[ti] - torch.repeat_interleave(z, m, 0))
                if ox or oy:
                    near = d.square().sum(1) < cut2
                    ti, si, d = ti[near], si[near], d[near]
                yield ti, si, d


def _slp_pair(d, f, xi):
    r2 = d.square().sum(1)
    hit = r2 == 0
    r2 = torch.where(hit, torch.ones_like(r2), r2)
    x = xi * xi * r2
    e = torch.exp(-x)
    u = (0.5 * _E1.apply(x) - e)[:, None] * f + (e * (d * f).sum(1) / r2)[:, None] * d
    own = -1.288607832450766155 - math.log(xi)     # -(gamma/2 + 1) - log xi
    return torch.where(hit[:, None], own * f, u) / (4 * math.pi)


def _dlp_pair(d, f, n, xi):
    r2 = d.square().sum(1)
    hit = r2 == 0
    r2 = torch.where(hit, torch.ones_like(r2), r2)
    x = xi * xi * r2
    e = torch.exp(-x)
    df, dn, fn = (d * f).sum(1), (d * n).sum(1), (f * n).sum(1)
    u = (-4 * (1 + x) / (r2 * r2) * df * dn)[:, None] * d + \
        2 * xi * xi * (fn[:, None] * d + df[:, None] * n + dn[:, None] * f)
    return torch.where(hit[:, None], torch.zeros_like(u), e[:, None] * u) / (4 * math.pi)


class _Grid:
    """The k-space part on an M x (M Ly) grid: Gaussian weights, spread, filter, gather."""

    def __init__(self, xi, M, P, Ly):
        self.xi, self.P, self.Mx, self.My = xi, P, M, M * Ly
        self.h = 1.0 / M
        self.L = (1.0, float(Ly))
        w = P * self.h / 2
        self.eta = (2 * xi * w / (0.95 * math.sqrt(math.pi * P))) ** 2
        self.a = -2 * xi * xi / self.eta
        self.scale = (4 * xi * xi / self.eta) ** 2 * self.h ** 2 / math.pi / (4 * math.pi)
        kx = 2 * math.pi / self.L[0] * self._freq(self.Mx)[:, None]
        ky = 2 * math.pi / self.L[1] * self._freq(self.My)[None, :]
        K2 = kx * kx + ky * ky
        K2[0, 0] = 1.0
        damp = torch.exp(-0.25 * (1 - self.eta) / xi ** 2 * K2)
        live = torch.ones_like(K2)
        live[0, 0] = 0.0
        self.kx, self.ky, self.K2 = kx, ky, K2
        self.cs = live * (1 / K2 ** 2 + 0.25 / (K2 * xi * xi)) * damp
        self.cd = live * damp / K2 / K2 * (1 + 0.25 * K2 / xi / xi)

    @staticmethod
    def _freq(M):
        j = torch.arange(M, device=DEV, dtype=torch.float64)
        return torch.where(j <= M // 2, j, j - M)

    def weights(self, p):
        """Node numbers and Gaussian factors of the (P + 1)^2 nodes about each point."""
        j = torch.arange(self.P + 1, device=DEV)
        off = (j - self.P // 2).double() * self.h
        out = []
        for c, M in ((0, self.Mx), (1, self.My)):
            x = p[:, c]
            m = torch.floor((x.detach() + self.L[c] / 2) / self.h).long() - self.P // 2
            rest = x - self.h * torch.floor(x.detach() / self.h)
            out.append((torch.remainder(m[:, None] + j, M),
                        torch.exp(self.a * (rest[:, None] - off).square())))
        return out

    def _chunks(self, p, step=1 << 16):
        for i in range(0, len(p), step):
            (ix, X), (iy, Y) = self.weights(p[i:i + step])
            yield slice(i, i + step), (ix[:, :, None] * self.My + iy[:, None, :]).flatten(), X, Y

    def spread(self, p, c):
        g = torch.zeros(c.shape[1], self.Mx * self.My, device=DEV, dtype=torch.float64)
        for at, idx, X, Y in self._chunks(p):
            W = X[:, :, None] * Y[:, None, :]
            for k in range(c.shape[1]):
                g[k].index_add_(0, idx, (c[at, k][:, None, None] * W).flatten())
        return g.view(-1, self.Mx, self.My)

    def gather(self, p, g):
        u = torch.empty(len(p), len(g), device=DEV, dtype=torch.float64)
        for at, idx, X, Y in self._chunks(p):
            for k in range(len(g)):
                v = g[k].reshape(-1)[idx].view(len(X), self.P + 1, self.P + 1)
                u[at, k] = ((v * Y[:, None, :]).sum(2) * X).sum(1)
        return u * self.scale

    def slp(self, g):
        h = torch.fft.fft2(g)
        q = self.cs * (self.ky * h[0] - self.kx * h[1])
        return torch.fft.ifft2(torch.stack([self.ky * q, -self.kx * q])).real

    def dlp(self, g):
        h = torch.fft.fft2(g)
        kx, ky, K2 = self.kx, self.ky, self.K2
        tr = h[0] + h[2]
        kS = kx * kx * h[0] + kx * ky * h[1] + ky * ky * h[2]
        o1 = K2 * (kx * tr + 2 * kx * h[0] + ky * h[1]) - 2 * kx * kS
        o2 = K2 * (ky * tr + 2 * ky * h[2] + kx * h[1]) - 2 * ky * kS
        return torch.fft.ifft2(self.cd * torch.stack([o1, o2])).imag


def _tensor_S(f, n):
    return torch.stack([f[:, 0] * n[:, 0], f[:, 0] * n[:, 1] + f[:, 1] * n[:, 0],
                        f[:, 1] * n[:, 1]], 1)


def _forward(kind, ps, pt, f, n, xi, nside, M, P, Ly):
    """(real part, k part) of the SLP or DLP sum; points wrapped already."""
    ur = torch.zeros(len(pt), 2, device=DEV, dtype=torch.float64)
    for ti, si, d in _pairs(ps, pt, nside, nside * Ly, Ly):
        ur.index_add_(0, ti, _slp_pair(d, f[si], xi) if kind == "slp"
                      else _dlp_pair(d, f[si], n[si], xi))
    G = _Grid(xi, M, P, Ly)
    g = G.slp(G.spread(ps, f)) if kind == "slp" else G.dlp(G.spread(ps, _tensor_S(f, n)))
    return ur, G.gather(pt, g)


def _potential(kind, case, raw, ps, pt, f, n):
    ur, uk = _forward(kind, ps, pt, f, n, case["xi"], case["nside"], case["M"], case["P"],
                      case["Ly"])
    if kind == "slp":
        return ur + uk
    zero = ((f * n).sum(1)[:, None] * raw).sum(0) / case["Ly"]
    return -(ur + uk - zero)


def _gradients(case, s, ps, pt):
    """d/d(positions, forces, densities, normals) of sum w_slp.u_slp + w_dlp.u_dlp."""
    xi, Ly = case["xi"], case["Ly"]
    f, g, n = s["fs"][0], s["fd"][0], s["n"]
    out = [torch.zeros_like(ps) for _ in range(4)]
    for ti, si, d in _pairs(ps, pt, case["nside"], case["nside"] * Ly, Ly, most=1 << 24):
        v = [x.clone().requires_grad_(True) for x in (d, f[si], g[si], n[si])]
        with torch.enable_grad():
            J = (s["ws"][ti] * _slp_pair(v[0], v[1], xi)).sum() - \
                (s["wd"][ti] * _dlp_pair(v[0], v[2], v[3], xi)).sum()
            for o, q in zip(out, torch.autograd.grad(J, v)):
                o.index_add_(0, si, q)
    G = _Grid(xi, case["M"], case["P"], Ly)
    back = []
    for kind, w, nc in (("slp", s["ws"], 2), ("dlp", -s["wd"], 3)):
        src = torch.zeros(nc, G.Mx, G.My, device=DEV, dtype=torch.float64, requires_grad=True)
        with torch.enable_grad():          # the filter is linear: its transpose at any grid
            J = (getattr(G, kind)(src) * G.spread(pt, w)).sum() * G.scale
            back.append(torch.autograd.grad(J, src)[0].reshape(nc, -1))
    step = 1 << 15
    for i in range(0, len(ps), step):
        at = slice(i, i + step)
        v = [x[at].clone().requires_grad_(True) for x in (ps, f, g, n)]
        with torch.enable_grad():
            (ix, X), (iy, Y) = G.weights(v[0])
            idx = (ix[:, :, None] * G.My + iy[:, None, :]).flatten()
            J = 0
            for c, grid in ((v[1], back[0]), (_tensor_S(v[2], v[3]), back[1])):
                for k in range(len(grid)):
                    q = grid[k][idx].view(len(X), G.P + 1, G.P + 1)
                    J = J + (((q * Y[:, None, :]).sum(2) * X).sum(1) * c[:, k]).sum()
            for o, q in zip(out, torch.autograd.grad(J, v)):
                o[at] += q
    # the k = 0 term of the DLP, sum (g.n) x / area
    wsum = s["wd"].sum(0) / Ly
    gn, wx = (g * n).sum(1, keepdim=True), (s["ps"] * wsum).sum(1, keepdim=True)
    out[0] += gn * wsum
    out[2] += n * wx
    out[3] += g * wx
    return out


@torch.no_grad()
def exact(case, seed):
    s = _inputs(case, seed)
    _inputs_of.cache_clear()
    op = case["op"]
    ps, pt = _wrap(s["ps"], case["Ly"]), _wrap(s["pt"], case["Ly"])
    if op == "mex_slp":
        return _forward("slp", s["ps"], s["pt"], s["fs"][0], None, case["xi"], case["nside"],
                        case["M"], case["P"], case["Ly"])
    if op == "driver":
        # the sum itself does not depend on how it is split: a split of its
        # own, fine enough for 64 bits
        nside = max(3, round(math.sqrt(len(ps) / 60)))
        xi = 6.0 * nside
        u = sum(_forward("slp", ps, pt, s["fs"][0], None, xi, nside, 2 * int(2.2 * xi), 34, 1))
        u = u.cpu().numpy()
        return u[:, 0].copy(), u[:, 1].copy(), None, None, None
    pot = lambda kind, r: _potential(kind, case, s["ps"], ps, pt,
                                     s["fs" if kind == "slp" else "fd"][r], s["n"])
    if op in ("slp", "dlp"):
        return pot(op, 0)
    if op == "geometry":
        kinds = ("slp", "dlp") if case["kinds"] == "both" else (case["kinds"],)
        return [torch.stack([pot(k, r) for r in range(case["nrhs"])]) for k in kinds]
    u = [pot("slp", 0), pot("dlp", 0)]
    return u + _gradients(case, s, ps, pt) if op == "grad" else u
