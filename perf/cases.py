"""Performance cases of the Neumann-series RTE solver: what its users run, through the public entry points.

Each case is one call pattern of a program that holds a solver context (grid, order, model) and brings new
media, sources or data to it.  `prepare` makes the context and the inputs, `run` is one pass, `work` the
bytes and operations the pass cannot do without, `exact` the same result from plain torch in 64 bits.

Mixed-precision solves sum in FP32, in an order that the launch tuner picks per process: their results are
single-precision numbers, and the program keeps them as such.  FP64 solves keep theirs in double."""
import math

import numpy as np
import torch

import doi_b200 as R

DX = 0.1      # voxel edge, cm
TERMS = 20    # Neumann terms of the fixed-length solves


# ---------------------------------------------------------------------------------------- cases
def listed():
    return [
        # The drop-in path of the reference's forward main at its shipped size: tissue map, beam, Neumann()
        # to its own stop rule, both images.  The smallest call: launches and host work count.
        dict(name="neumann_10x10x20_L2", kind="neumann", nx=10, ny=10, nz=20, L=2),
        # The CPU package's workload: one uniform 11^3 medium, L=3, until the terms change it by < 1e-7.
        dict(name="uniform_11_L3", kind="forward", nx=11, ny=11, nz=11, L=3, prec="fp64", medium="uniform",
             stop="rel"),
        # A forward solve in plain FP64 (the default precision) on a phantom of ordinary size.
        dict(name="forward_21_L5_fp64", kind="forward", nx=21, ny=21, nz=21, L=5, prec="fp64", medium="spheres",
             stop="fixed"),
        # One source on a new 33^3 phantom, mixed precision.
        dict(name="forward_33_L5", kind="forward", nx=33, ny=33, nz=33, L=5, prec="mixed", medium="spheres",
             stop="fixed"),
        # The benchmark's step: four sources on a new 33^3 phantom.
        dict(name="batch4_33_L5", kind="batch", nx=33, ny=33, nz=33, L=5, nsrc=4),
        # Requests of mixed shapes that arrive at the server together.
        dict(name="serve_8", kind="serve", count=8, grids="17,25", orders="3,5"),
        # High order: FP64 angular recurrence; an isotropic point on a side face.
        dict(name="forward_25_L7_point", kind="forward", nx=25, ny=25, nz=25, L=7, prec="mixed", medium="spheres",
             stop="fixed", source="point", face=4),
        # The largest served grid at low order.
        dict(name="forward_41_L3", kind="forward", nx=41, ny=41, nz=41, L=3, prec="mixed", medium="spheres",
             stop="fixed"),
        # The adjoint gradient of a reconstruction step: 4 sources, 8 x 8 bins on six faces.
        dict(name="gradient_33_L5", kind="gradient", nx=33, ny=33, nz=33, L=5, prec="mixed", nsrc=4, nbins=8),
        # The same in plain FP64 on a small problem.
        dict(name="gradient_15_L3_fp64", kind="gradient", nx=15, ny=15, nz=15, L=3, prec="fp64", nsrc=2, nbins=8),
        # Fisher information of one inclusion, path integrals recomputed in every term.
        dict(name="fisher_17_L5", kind="fisher", nx=17, ny=17, nz=17, L=5, nsrc=2, nbins=8),
        # A frequency-domain solve (complex mu_t).
        dict(name="modulated_17_L3_fp64", kind="modulated", nx=17, ny=17, nz=17, L=3, prec="fp64"),
    ]


def _shape(rng, lo, hi, even=False):
    """A grid of lo..hi voxels (log-uniform), its edges within a factor of about two of one another."""
    side = math.exp(rng.uniform(math.log(lo), math.log(hi))) ** (1.0 / 3.0)
    f = [math.exp(rng.uniform(-0.3, 0.3)) for _ in range(3)]
    g = (f[0] * f[1] * f[2]) ** (1.0 / 3.0)
    n = [max(4, int(round(side * x / g))) for x in f]
    if even:
        n[0] += n[0] % 2
        n[1] += n[1] % 2
    while n[0] * n[1] * n[2] > hi:
        q = max(range(3), key=lambda a: n[a])
        n[q] -= 2 if even else 1
    return dict(nx=n[0], ny=n[1], nz=n[2])


def draw(rng):
    kind = rng.choice(["forward", "forward", "forward", "batch", "neumann", "serve", "gradient", "fisher", "modulated"])
    if kind == "neumann":
        return dict(kind=kind, **_shape(rng, 300, 5000, even=True), L=rng.randint(1, 4))
    if kind == "serve":
        return dict(kind=kind, count=rng.randint(2, 10), grids=rng.choice(["17", "17,25", "25"]),
                    orders=rng.choice(["3", "3,5", "5", "7"]))
    if kind == "gradient":
        prec = rng.choice(["mixed", "fp64"])
        return dict(kind=kind, **_shape(rng, 300, 8000 if prec == "mixed" else 3400), L=rng.randint(2, 5), prec=prec,
                    nsrc=rng.randint(1, 3), nbins=rng.choice([4, 8]))
    if kind == "fisher":
        return dict(kind=kind, **_shape(rng, 300, 3500), L=rng.randint(2, 5), nsrc=rng.randint(1, 2), nbins=8)
    if kind == "modulated":
        return dict(kind=kind, **_shape(rng, 300, 5000), L=rng.randint(1, 5), prec=rng.choice(["mixed", "fp64"]))
    L = rng.choice([1, 2, 3, 3, 4, 5, 5, 6, 7])
    if kind == "batch":
        return dict(kind=kind, **_shape(rng, 700, 30000 if L <= 5 else 14000), L=L, nsrc=rng.randint(2, 4))
    prec = rng.choice(["mixed", "mixed", "fp64"])
    top = (40000 if L <= 3 else 33000 if L <= 5 else 15000) if prec == "mixed" else (9000 if L <= 5 else 4500)
    c = dict(kind=kind, **_shape(rng, 300, top), L=L, prec=prec,
             medium=rng.choice(["spheres", "spheres", "spheres", "uniform"]), stop=rng.choice(["fixed", "fixed", "rel"]))
    if rng.random() < 0.4:
        c["source"] = rng.choice(["beam", "point"])
        c["face"] = rng.randint(0, 5)
    if rng.random() < 0.2:  # coupling limited to a distance (propThresh)
        c["thresh"] = round(rng.uniform(0.5, 0.9), 3)
    return c


# ---------------------------------------------------------------------------------------- inputs
def _centres(c):
    x = (np.arange(c["nx"]) + 0.5) * DX - c["nx"] * DX / 2
    y = (np.arange(c["ny"]) + 0.5) * DX - c["ny"] * DX / 2
    z = (np.arange(c["nz"]) + 0.5) * DX
    Z, Y, X = np.meshgrid(z, y, x, indexing="ij")
    return X.ravel(), Y.ravel(), Z.ravel()


def _spheres(c, rng, count=3):
    """Three spherical inclusions: radius 0.2-0.6 cm (within the box), mu_a x [2, 10], mu_s x [0.5, 2]."""
    hi = np.array([c["nx"], c["ny"], c["nz"]]) * DX
    out = []
    for _ in range(count):
        r = min(rng.uniform(0.2, 0.6), 0.4 * hi.min())
        ctr = rng.uniform(r, hi - r) - np.array([hi[0] / 2, hi[1] / 2, 0.0])
        out.append((r, ctr, rng.uniform(2, 10), rng.uniform(0.5, 2)))
    return out


def _phantom(c, rng, count=3):
    X, Y, Z = _centres(c)
    mua, mus = np.full(X.size, 0.01), np.full(X.size, 1.0)
    for r, ctr, ka, ks in _spheres(c, rng, count):
        inside = (X - ctr[0]) ** 2 + (Y - ctr[1]) ** 2 + (Z - ctr[2]) ** 2 <= r * r
        mua[inside] = 0.01 * ka
        mus[inside] = ks
    return mua, mus


def _face_source(c, kind, face, rng):
    a = rng.uniform(-0.4, 0.4, 2) * np.array([c["nx"], c["ny"]]) * DX
    return R.Source(pos_x=float(a[0]), pos_y=float(a[1]), pos_z=float(rng.uniform(0.1, 0.9) * c["nz"] * DX),
                    kind=R.SRC_POINT if kind == "point" else R.SRC_BEAM, face=face)


def _column_sources(c, count):
    """Collimated z = 0 beams at a quarter of the face, one beam in the middle."""
    if count == 1:
        return [R.Source(kind=R.SRC_COLUMN)]
    h, v = 0.25 * c["nx"] * DX, 0.25 * c["ny"] * DX
    return [R.Source(pos_x=sx * h, pos_y=sy * v, kind=R.SRC_COLUMN)
            for sx, sy in ((-1, -1), (1, -1), (-1, 1), (1, 1))][:count]


def _stop(c):
    return R.Stop(R.STOP_REL_L2, 30, 1e-7) if c.get("stop") == "rel" else R.Stop(R.STOP_FIXED, TERMS)


def _inputs(c, seed):
    """The case's inputs from the seed alone (no context)."""
    rng = np.random.default_rng([seed, 17])
    k = c["kind"]
    s = dict(case=c, stop=_stop(c))
    if k == "neumann":  # a map of three tissues with a table of coefficients
        mua_tab = np.array([0.01, 0.03, 0.1]) * rng.uniform(0.8, 1.2, 3)
        mus_tab = np.array([1.0, 1.5, 0.6]) * rng.uniform(0.8, 1.2, 3)
        X, Y, Z = _centres(c)
        tiss = np.zeros(X.size, np.uint8)
        for t, (r, ctr, _, _) in enumerate(_spheres(c, rng, 2)):
            tiss[(X - ctr[0]) ** 2 + (Y - ctr[1]) ** 2 + (Z - ctr[2]) ** 2 <= r * r] = t + 1
        s.update(tiss=tiss, mua_tab=mua_tab, mus_tab=mus_tab, src=R.Source(kind=R.SRC_FIM),
                 stop=R.Stop(R.STOP_REFERENCE))
    elif k == "serve":
        s["requests"] = []
        grids, orders = c["grids"].split(","), c["orders"].split(",")
        for q in range(c["count"]):
            n, L = int(grids[q % len(grids)]), int(orders[(q // len(grids)) % len(orders)])
            box = dict(nx=n, ny=n, nz=n, L=L)
            mua, mus = _phantom(box, rng, 1 + q % 3)
            src = _face_source(box, "point" if q % 2 else "beam", int(rng.integers(0, 6)), rng)
            s["requests"].append((box, mua, mus, src))
    elif k == "fisher":  # one inclusion with a one-voxel partial-volume ramp: d/d(x, y, z, contrast)
        r, ctr, ka, _ = _spheres(c, rng, 1)[0]
        X, Y, Z = _centres(c)
        rel = np.stack([X, Y, Z], 1) - ctr
        rho = np.linalg.norm(rel, axis=1)
        u = 0.5 + (r - rho) / DX
        f, ramp = np.clip(u, 0, 1), (u > 0) & (u < 1)
        s["mua"], s["mus"] = 0.02 * (1 + (ka - 1) * f), np.full(X.size, 2.0)
        d = np.where(ramp[:, None], rel / (DX * np.maximum(rho, 1e-300))[:, None], 0.0)
        s["dmua"] = np.stack([0.02 * (ka - 1) * d[:, a] for a in range(3)] + [0.02 * f])
        s["dmus"] = np.zeros_like(s["dmua"])
        h = c["nz"] * DX / 2
        s["srcs"] = [R.Source(kind=R.SRC_BEAM, face=0), R.Source(kind=R.SRC_BEAM, face=4, pos_z=h)][:c["nsrc"]]
        s["det"] = R.Detector(nbins=c["nbins"], faces=63)
    else:
        if c.get("medium") == "uniform":
            n = c["nx"] * c["ny"] * c["nz"]
            s["mua"], s["mus"] = np.full(n, 0.01 * rng.uniform(0.8, 1.2)), np.full(n, 1.0 * rng.uniform(0.8, 1.2))
        else:
            s["mua"], s["mus"] = _phantom(c, rng)
        if k == "batch":
            s["srcs"] = _column_sources(c, c["nsrc"])
        elif k == "gradient":
            s["srcs"] = _column_sources(c, c["nsrc"])
            s["det"] = R.Detector(nbins=c["nbins"], faces=63)
            s["target"] = rng.lognormal(-7.0, 1.0, (c["nsrc"], 6, c["nbins"], c["nbins"]))
        elif k == "modulated":
            s["src"] = R.Source(kind=R.SRC_COLUMN, modulation=float(rng.uniform(0.3, 0.8)))
        elif c.get("source"):
            s["src"] = _face_source(c, c["source"], c["face"], rng)
        else:
            s["src"] = R.Source(kind=R.SRC_COLUMN)
    return s


def _thresh(c):
    return c["thresh"] * DX * math.sqrt(c["nx"] ** 2 + c["ny"] ** 2 + c["nz"] ** 2) if "thresh" in c else None


def prepare(case, seed):
    s = _inputs(case, seed)
    if case["kind"] == "serve":
        s["server"] = R.Server(hbm_budget_gb=24.0, workers=4)
        return s
    fim = case["kind"] == "neumann"
    fisher = case["kind"] == "fisher"
    prec = R.PREC_FP64 if fim or case.get("prec") == "fp64" else R.PREC_MIXED
    s["ctx"] = R.Context(case["nx"], case["ny"], case["nz"], dx=DX, nL=case["L"], g=0.9 if fisher else 0.8,
                         model=R.MODEL_FIM if fim else R.MODEL_EXACT, precision=prec, prop_thresh=_thresh(case),
                         kernel_mode=R.KERNEL_RECOMPUTE if fisher else R.KERNEL_AUTO)
    return s


def _kept(s, arrays):
    """Mixed results are kept in single precision, FP64 results in double."""
    c = s["case"]
    if c["kind"] == "neumann" or c.get("prec") == "fp64":
        return arrays
    return {k: v.astype(np.complex64 if v.dtype.kind == "c" else np.float32) for k, v in arrays.items()}


def run(s):
    c, k = s["case"], s["case"]["kind"]
    if k == "serve":
        srv = s["server"]
        tickets = [srv.submit(mua, mus, [src], b["nx"], dx=DX, nL=b["L"], g=0.8, terms=TERMS)
                   for b, mua, mus, src in s["requests"]]
        res = {}
        for q, t in enumerate(tickets):
            tr, rf, _ = srv.wait(t)
            res["trans%d" % q], res["ref%d" % q] = tr, rf
        return _kept(s, res)
    ctx = s["ctx"]
    if k == "neumann":
        ctx.set_medium_tissue(s["tiss"], s["mua_tab"], s["mus_tab"])
        xi = ctx.source_beam(s["src"])
        out, _ = ctx.neumann(xi, xi, 1, s["stop"])
        tr, rf = ctx.images(out, s["src"])
        return dict(W=out, trans=tr, ref=rf)
    ctx.set_medium_voxel(s["mua"], s["mus"])
    if k == "gradient":
        loss, ga, gs = ctx.gradient(s["srcs"], s["stop"], s["det"], s["target"])
        return _kept(s, dict(loss=np.array([loss]), g_mua=ga, g_mus=gs))
    if k == "fisher":
        F, J = ctx.fisher(s["srcs"], s["stop"], s["det"], s["dmua"], s["dmus"], want_J=True)
        return _kept(s, dict(F=F, J=J))
    if k == "batch":
        r = ctx.forward_batch(s["srcs"], s["stop"], want_W=False)
        return _kept(s, dict(trans=r["trans"], ref=r["ref"]))
    fp64 = c.get("prec") == "fp64"
    r = ctx.forward(s["src"], s["stop"], want_W=fp64)
    return _kept(s, {q: r[q] for q in ("W", "trans", "ref") if q in r})


# ---------------------------------------------------------------------------------------- floors
def work(c):
    """Operations: along one line of sight column a field of order L has 2L+1 angular terms, read in and
    written out once per pair, application and right-hand side (two operations each); the path integral of
    every unordered pair, two operations per voxel crossed; uniform media by convolution.  Bytes: the
    medium in, the results out."""
    if c["kind"] == "serve":
        grids, orders = c["grids"].split(","), c["orders"].split(",")
        b = f = 0.0
        for q in range(c["count"]):
            n, L = int(grids[q % len(grids)]), int(orders[(q // len(grids)) % len(orders)])
            w = work(dict(kind="forward", nx=n, ny=n, nz=n, L=L, prec="mixed"))
            b, f = b + w["bytes"], f + w["flops"]
        return dict(bytes=b, flops=f)
    nx, ny, nz, L = c["nx"], c["ny"], c["nz"], c["L"]
    N, C, k = nx * ny * nz, (L + 1) ** 2, c["kind"]
    pairs = float(N) * (N - 1)
    steps = (nx + ny + nz) / 3.0
    apps, rhs = TERMS + 1, c.get("nsrc", 1)
    image = 2 * 16.0 * nx * ny
    out = image * rhs + (16.0 * N * C if c.get("prec") == "fp64" or k == "neumann" else 0.0)
    walks = 1
    if k == "neumann":
        apps = 8
    elif k == "gradient":
        apps, out = 2 * apps, 16.0 * N
        walks = 2
    elif k == "fisher":
        apps, rhs, out = apps, 5 * rhs, 8.0 * 6 * c["nbins"] ** 2 * 4 * rhs
    elif k == "modulated":
        rhs = 2
    if c.get("medium") == "uniform":
        M = 8.0 * N
        flops = apps * (2 * C * 2.5 * M * math.log2(M) + 2.0 * C * C * M / 2)
    else:
        flops = apps * rhs * pairs * 4.0 * (2 * L + 1) + walks * pairs / 2 * steps * 2
    return dict(bytes=16.0 * N + out, flops=flops)


# ---------------------------------------------------------------------------------------- exact values
_DEV = "cuda" if torch.cuda.is_available() else "cpu"
_T = dict(dtype=torch.float64, device=_DEV)


def _real_sh(L, x, y, z):
    """Real orthonormal spherical harmonics (Condon-Shortley phase) at unit vectors, [..., (L+1)^2]."""
    out = np.zeros(x.shape + ((L + 1) ** 2,))
    e = x + 1j * y  # sin(theta) e^(i phi)
    for m in range(L + 1):
        p = np.full(x.shape, (-1.0) ** m * float(np.prod(np.arange(1, 2 * m, 2))))  # P_m^m / sin^m
        prev = np.zeros_like(p)
        az = e ** m
        for l in range(m, L + 1):
            if l > m:
                p, prev = ((2 * l - 1) * z * p - (l + m - 1) * prev) / (l - m), p
            nrm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - m) / math.factorial(l + m))
            if m == 0:
                out[..., l * l + l] = nrm * p
            else:
                out[..., l * l + l + m] = math.sqrt(2) * nrm * p * az.real
                out[..., l * l + l - m] = math.sqrt(2) * nrm * p * az.imag
    return out


def _table_directions(dx, dy, dz, dist):
    """Nearest cell of the reference's 100 x 100 direction table, its azimuth not wrapped."""
    with np.errstate(invalid="ignore", divide="ignore"):
        ti = np.rint((99 * np.arccos(np.nan_to_num(dz / dist)) / np.pi).astype(np.float32)).astype(int)
    pj = np.rint((99 * np.arctan2(dy, dx) / (2 * np.pi)).astype(np.float32)).astype(int)
    off = np.maximum(ti * 100 + pj, 0)
    th, ph = (off // 100) * np.pi / 99, (off % 100) * 2 * np.pi / 99
    return np.sin(th) * np.cos(ph), np.sin(th) * np.sin(ph), np.cos(th)


def _leg(l, u):
    return np.polynomial.legendre.Legendre.basis(l)(u)


class _Model:
    """The discrete model of one case in plain torch, 64 bits."""

    def __init__(self, c, fim=False, g=0.8):
        self.c, self.fim, self.g, self.L = c, fim, g, c["L"]
        self.n = nx, ny, nz = c["nx"], c["ny"], c["nz"]
        self.N, self.C = nx * ny * nz, (self.L + 1) ** 2
        if fim:  # float extents, as the reference keeps them
            f = np.float32
            self.d = [float(f(nn * DX / 2) - f(-nn * DX / 2)) / nn for nn in (nx, ny)] + [float(f(nz * DX)) / nz]
        else:
            self.d = [(nn * DX / 2 + nn * DX / 2) / nn for nn in (nx, ny)] + [nz * DX / nz]
        self.dV = self.d[0] * self.d[1] * self.d[2]
        self.thresh = _thresh(c) or 2.0 * math.sqrt((nx * DX) ** 2 + (ny * DX) ** 2 + (nz * DX) ** 2)
        iz, iy, ix = np.meshgrid(np.arange(1 - nz, nz), np.arange(1 - ny, ny), np.arange(1 - nx, nx), indexing="ij")
        X, Y, Z = ix * self.d[0], iy * self.d[1], iz * self.d[2]
        dist = np.sqrt(X * X + Y * Y + Z * Z)
        if fim:
            u = _table_directions(X, Y, Z, dist)
        else:
            safe = np.where(dist > 0, dist, 1.0)
            u = (X / safe, Y / safe, Z / safe)
        rt = _real_sh(self.L, *u)
        rt[nz - 1, ny - 1, nx - 1] = 0.0
        # flipped, so that the sources of one destination are an ascending sub-box
        self.R = torch.tensor(np.ascontiguousarray(rt[::-1, ::-1, ::-1]), **_T)
        ls = np.array([l for l in range(self.L + 1) for _ in range(2 * l + 1)])
        gl = float(int(g)) ** ls if fim else g ** ls.astype(float)
        self.scat = torch.tensor(gl, **_T)
        self._quadrature()

    def _quadrature(self):
        """Self-voxel quadrature: directions, weights, distance from the voxel centre to its surface."""
        ang = 100 if self.fim else 200
        th, ph = [v.ravel() for v in np.meshgrid(np.arange(ang) * np.pi / ang, np.arange(ang) * 2 * np.pi / ang,
                                                 indexing="ij")]
        s = [np.cos(ph) * np.sin(th), np.sin(ph) * np.sin(th), np.cos(th)]
        R = _real_sh(self.L, *s)
        self.qw = torch.tensor(np.sin(th) * (np.pi / ang) * (2 * np.pi / ang), **_T)
        if not self.fim:
            s = [v.astype(np.float32).astype(np.float64) for v in s]
        best = np.zeros((3, th.size))
        for a in range(3):
            for sign in (1.0, -1.0):
                with np.errstate(divide="ignore", invalid="ignore"):
                    p = [np.full(th.size, sign) if b == a else sign * s[b] / s[a] for b in range(3)]
                    if not self.fim:  # face points are floats there
                        p = [v.astype(np.float32).astype(np.float64) for v in p]
                    hit = (s[a] != 0) & (s[a] * sign >= 0)
                    for v in p:
                        hit &= np.abs(v) <= 1.0
                for b in range(3):
                    best[b][hit] = p[b][hit]
        best = best.astype(np.float32).astype(np.float64)
        half = [self.d[0] / 2] * 3 if self.fim else [v / 2 for v in self.d]
        self.beta = torch.tensor(np.sqrt(sum((best[b] * half[b]) ** 2 for b in range(3))), **_T)
        self.qR = torch.tensor(R, **_T)

    def self_matrices(self, mut):
        """D(mu_t) per distinct value; returns (matrices, voxel -> row).  mut may carry gradients."""
        vals, idx = np.unique(mut.detach().cpu().numpy(), return_inverse=True)
        first = np.zeros(len(vals), int)
        first[idx.ravel()[::-1]] = np.arange(idx.size)[::-1]
        mu = mut[torch.tensor(first, device=_DEV)][:, None]
        mats = self.contract((1 - torch.exp(-mu * self.beta)) / mu)
        return mats, torch.tensor(idx.ravel(), device=_DEV)

    def contract(self, f):
        """sum_w f[v][w] weight R_a R_b: [v, C, C]."""
        if not hasattr(self, "RR"):
            self.RR = (self.qw[:, None, None] * self.qR[:, :, None] * self.qR[:, None, :]).reshape(len(self.qw), -1)
        m = torch.complex(f.real @ self.RR, f.imag @ self.RR) if f.is_complex() else f @ self.RR
        return m.reshape(-1, self.C, self.C)

    def _walk(self, lo, hi, visit):
        """Siddon walk between the centres of every pair (destination in lo..hi, source < hi): visit(voxel,
        segment) per step, lengths scaled by Q / distance; returns (distance, Q)."""
        nx, ny, nz = self.n
        dv = torch.arange(lo, hi, device=_DEV, dtype=torch.int32)[:, None]
        sv = torch.arange(0, hi, device=_DEV, dtype=torch.int32)[None, :]
        co = lambda v: (v % nx, (v // nx) % ny, v // (nx * ny))  # noqa: E731
        a, b = co(dv), co(sv)
        D = [(p - q).abs() for p, q in zip(a, b)]
        m = [torch.clamp(v, min=1) for v in D]
        Q = 2 * m[0] * m[1] * m[2]
        big = torch.tensor(1 << 30, device=_DEV, dtype=torch.int32)
        h = [m[1] * m[2], m[0] * m[2], m[0] * m[1]]
        A = [torch.where(D[q] > 0, h[q], big).contiguous() for q in range(3)]
        stride = (1, nx, nx * ny)
        st = [torch.where(b[q] > a[q], stride[q], -stride[q]).to(torch.int32) for q in range(3)]
        v = dv.expand(Q.shape).contiguous()
        prev = torch.zeros_like(Q)
        steps = int((D[0] + D[1] + D[2]).max()) + 1
        for _ in range(steps):
            t = torch.minimum(torch.minimum(A[0], A[1]), torch.minimum(A[2], Q))
            visit(v, t - prev)
            prev = t
            bz = A[2] == t
            by = (A[1] == t) & ~bz
            bx = (A[0] == t) & ~bz & ~by
            for q, hit in ((0, bx), (1, by), (2, bz)):
                v = v + torch.where(hit, st[q], 0)
                A[q] = A[q] + torch.where(hit, 2 * h[q], 0)
        dist = torch.sqrt(sum((D[q].double() * self.d[q]) ** 2 for q in range(3)))
        return dist, Q

    def _blocks(self):
        lo = 0
        while lo < self.N:
            hi = min(self.N, lo + max(1, int(2.0e7 // self.N)))
            yield lo, hi
            lo = hi

    def kernel(self, mut, kappa=0.0):
        """exp(-tau) dV / r^2 of every pair, [N, N]."""
        K = torch.zeros((self.N, self.N), dtype=torch.complex128 if kappa else mut.dtype, device=_DEV)
        for lo, hi in self._blocks():
            acc = torch.zeros((hi - lo, hi), dtype=mut.dtype, device=_DEV)

            def visit(v, seg):
                acc.add_(mut[v.long()] * seg)

            dist, Q = self._walk(lo, hi, visit)
            tau = acc * dist / Q
            if kappa:
                tau = tau + 1j * kappa * dist
            k = torch.exp(-tau) * self.dV / torch.where(dist > 0, dist, 1.0) ** 2
            k = torch.where((dist > 0) & (dist < self.thresh), k, 0.0)
            K[lo:hi, :hi] = k
            K[:hi, lo:hi] = k.T
        return K

    def kernel_gradient(self, K, gK):
        """dL/dmu_t from dL/dK through the path integrals."""
        g = torch.zeros(self.N, **_T)
        G = -(gK * K)
        for lo, hi in self._blocks():
            w = G[lo:hi, :hi] + G[:hi, lo:hi].T
            w[:, lo:] = torch.tril(w[:, lo:], -1)
            dist, Q = self._walk(lo, hi, lambda v, s: None)
            w = w * dist / Q
            self._walk(lo, hi, lambda v, s: g.index_add_(0, v.reshape(-1).long(), (w * s).reshape(-1)))
        return g

    def _rows(self):
        nx, ny, nz = self.n
        for i in range(nz):
            for j in range(ny):
                box = self.R[nz - 1 - i:2 * nz - 1 - i, ny - 1 - j:2 * ny - 1 - j]      # [nz, ny, 2nx-1, C]
                win = box.unfold(2, nx, 1).flip(2)                                       # window k: offset nx-1-k
                yield (i * ny + j) * nx, win.permute(2, 0, 1, 4, 3).reshape(nx, self.N, self.C)

    def off_diagonal(self, K, W):
        """sum_r' R(w) K R(w) . W[r'] for W [N, C, B]."""
        if not hasattr(self, "Rall") and self.N * self.N * self.C * 8.0 < 12e9:
            self.Rall = torch.cat([r for _, r in self._rows()])
        rows = [(0, self.Rall)] if hasattr(self, "Rall") else self._rows()
        out = []
        for r0, Rw in rows:
            Rw = Rw.to(W.dtype)
            S = torch.bmm(Rw.transpose(0, 1), W).transpose(0, 1)            # [d, s, B]
            T = K[r0:r0 + Rw.shape[0], :, None] * S
            out.append(torch.bmm(Rw.transpose(1, 2), T))
        return torch.cat(out)

    def apply(self, K, D, W, mus=None):
        out = self.off_diagonal(K, W)
        mats, idx = D
        out = out + torch.bmm(mats.to(W.dtype)[idx], W)
        if mus is not None:
            out = out * (self.scat[None, :, None] * mus[:, None, None])
        return out

    def column(self, src):
        """Face pixel, voxels along the beam, inward direction of a source."""
        nx, ny, nz = self.n
        ext = ((src.pos_x + nx * DX / 2) / self.d[0], (src.pos_y + ny * DX / 2) / self.d[1], src.pos_z / self.d[2])
        k, j, i = [min(max(int(math.floor(e)), 0), nn - 1) for e, nn in zip(ext, self.n)]
        if src.kind == R.SRC_FIM:
            k, j = nx // 2, ny // 2
        f = src.face if src.kind in (R.SRC_BEAM, R.SRC_POINT) else 0
        ax = (2, 2, 1, 1, 0, 0)[f]
        t = np.arange(self.n[ax]) if f % 2 == 0 else np.arange(self.n[ax])[::-1]
        pix = (j * nx + k, i * nx + k, i * ny + j)[f // 2]
        vox = {2: t * nx * ny + j * nx + k, 1: i * nx * ny + t * nx + k, 0: i * nx * ny + j * nx + t}[ax]
        way = [0.0, 0.0, 0.0]
        way[ax] = 1.0 if f % 2 == 0 else -1.0
        return f, pix, torch.tensor(np.ascontiguousarray(vox), device=_DEV), way, self.d[ax]

    def beam(self, src, mut, mus, kappa=0.0):
        """Scattered first-order source and the ballistic flux at the exit pixel."""
        f, pix, vox, way, step = self.column(src)
        mt = mut[vox] + (1j * kappa if kappa else 0.0)
        e = torch.exp(-mt * step)
        att = torch.cat([torch.ones(1, dtype=e.dtype, device=_DEV), torch.cumprod(e, 0)])
        amp = mus[vox] / mt * att[:-1] * (1 - e) / self.dV
        dirs = _real_sh(self.L, *[np.array([w]) for w in way])[0]
        ls = np.array([l for l in range(self.L + 1) for _ in range(2 * l + 1)])
        coef = torch.tensor(src.mag * self.g ** ls.astype(float) * dirs, **_T)
        xi = torch.zeros((self.N, self.C), dtype=amp.dtype, device=_DEV).index_add(0, vox, amp[:, None] * coef)
        return xi, src.mag * att[-1], f ^ 1, pix

    def series(self, K, mut, mus, srcs, stop, kappa=0.0):
        """A sum_k (DA)^k xi for each source, [N, C, B], and the ballistic exits."""
        D = self.self_matrices(mut + 1j * kappa if kappa else mut)
        xs, qs, balls = [], [], []
        for s in srcs:
            if s.kind == R.SRC_POINT:
                _, _, vox, _, _ = self.column(s)
                q = torch.zeros((self.N, self.C), **_T)
                q[vox[0], 0] = s.mag / (math.sqrt(4 * math.pi) * self.dV)
                xs.append(torch.zeros_like(q))
                qs.append(q)
                balls.append(None)
            else:
                xi, b, f, p = self.beam(s, mut, mus, kappa)
                xs.append(xi)
                qs.append(torch.zeros_like(xi))
                balls.append((b, f, p))
        W, q = torch.stack(xs, 2), torch.stack(qs, 2)
        total = W
        if any(s.kind == R.SRC_POINT for s in srcs):
            W = W + self.apply(K, D, q, mus)
            total = W + q
        fi, terms = 1.0, 0
        while terms < (10000 if stop.rule == R.STOP_REFERENCE else stop.max_terms):
            if stop.rule == R.STOP_REFERENCE and self._stops(W, total, fi):
                break
            if stop.rule == R.STOP_REFERENCE:
                fi = self._ratio(W, total)
            W = self.apply(K, D, W, mus)
            total = total + W
            terms += 1
            if stop.rule == R.STOP_REL_L2 and float(torch.linalg.norm(W.abs()) / torch.linalg.norm(total.abs())) < stop.tol:
                break
        return self.apply(K, D, total), balls

    def _ratio(self, W, total):
        """Last layer's sum over m of the complex-basis coefficients, of the term over the running sum."""
        plane = self.n[0] * self.n[1]
        w = np.zeros(self.C)
        for l in range(self.L + 1):
            w[l * l + l] = 1.0
            for m in range(2, l + 1, 2):
                w[l * l + l + m] = math.sqrt(2)
        w = torch.tensor(w, **_T)[None, :, None]
        return float((W[-plane:] * w).sum()) / float((total[-plane:] * w).sum())

    def _stops(self, W, total, fi):
        s = self._ratio(W, total)
        if s == fi:  # the first term: 1 / 0, no stop
            return False
        hi = 1.0 - s * (1.0 / (1.0 - s / fi))
        return 0.9999 < hi <= 1.0

    def images(self, out, ball, mag=1.0):
        """Transmission and reflection images [ny, nx] of one right-hand side."""
        nx, ny, nz = self.n
        if self.fim:
            u, w = np.arange(100) / 99.0, np.full(100, 1 / 99.0)
        else:
            u, w = np.polynomial.legendre.leggauss(24)
            u, w = (u + 1) / 2, w / 2
        fac = 2 * math.pi * self.d[0] * self.d[1] / math.sqrt(4 * math.pi)
        tr = torch.zeros(nx * ny, dtype=out.dtype, device=_DEV)
        rf = torch.zeros_like(tr)
        for l in range(self.L + 1):
            wt = fac * math.sqrt(2 * l + 1) * float(np.sum(_leg(l, u) * u * w))
            wr = wt if self.fim else fac * math.sqrt(2 * l + 1) * float(np.sum(_leg(l, -u) * u * w))
            tr = tr + wt * out[-nx * ny:, l * l + l]
            rf = rf + wr * out[:nx * ny, l * l + l]
        if ball is not None:
            b, f, p = ball
            if f == 1:
                tr[p] += b
            elif f == 0:
                rf[p] += b
        return tr.reshape(ny, nx), rf.reshape(ny, nx)

    def to_complex(self, u):
        """Real-basis coefficients (of a real or complex function) -> complex spherical-harmonic basis."""
        out = u.to(torch.complex128).clone()
        for l in range(1, self.L + 1):
            for m in range(1, l + 1):
                a, b = u[:, l * l + l + m], u[:, l * l + l - m]
                out[:, l * l + l + m] = (a - 1j * b) / math.sqrt(2)
                out[:, l * l + l - m] = (-1) ** m * (a + 1j * b) / math.sqrt(2)
        return out

    def flux_bins(self, out, ball, nbins):
        """Exitant flux of one right-hand side through the six faces, binned: [6, nbins, nbins]."""
        nx, ny, nz = self.n
        u, w = np.polynomial.legendre.leggauss(24)
        u, w = (u + 1) / 2, w / 2
        az = 2 * np.pi * (np.arange(64) + 0.5) / 64
        grid = out.reshape(nz, ny, nx, self.C)
        bins = []
        for f in range(6):
            ax, sign = (2, 2, 1, 1, 0, 0)[f], (-1.0 if f % 2 == 0 else 1.0)
            s = np.sqrt(1 - u * u)[:, None]
            v = [s * np.cos(az), s * np.sin(az)]
            dirs = [None] * 3
            dirs[ax] = sign * np.repeat(u[:, None], 64, 1)
            for b, q in zip([b for b in range(3) if b != ax], v):
                dirs[b] = q
            area = self.dV / self.d[ax]
            h = area * np.einsum("a,abc->c", w * u * 2 * np.pi / 64, _real_sh(self.L, *dirs))
            face = grid.select(2 - ax, 0 if f % 2 == 0 else self.n[ax] - 1)
            J = face @ torch.tensor(h, **_T).to(out.dtype)
            if ball is not None and ball[1] == f:
                e = torch.zeros(J.numel(), **_T)
                e[ball[2]] = 1.0
                J = J + ball[0] * e.reshape(J.shape)
            ov = []
            for P in J.shape:
                p, a = np.arange(P)[:, None], np.arange(nbins)[None, :]
                lo, hi = np.maximum(p / P, a / nbins), np.minimum((p + 1) / P, (a + 1) / nbins)
                ov.append(torch.tensor(np.maximum(hi - lo, 0) * P, **_T).to(out.dtype))
            bins.append(ov[0].T @ J @ ov[1])
        return torch.stack(bins)


def _np(t):
    return t.detach().cpu().numpy()


def _exact_forward(c, mua, mus, srcs, stop, kappa=0.0, want_W=False):
    M = _Model(c)
    mua, mus = torch.tensor(mua, **_T), torch.tensor(mus, **_T)
    out, balls = M.series(M.kernel(mua + mus, kappa), mua + mus, mus, srcs, stop, kappa)
    pics = [M.images(out[:, :, b], balls[b]) for b in range(len(srcs))]
    res = dict(trans=[_np(p[0].to(torch.complex128)) for p in pics], ref=[_np(p[1].to(torch.complex128)) for p in pics])
    if want_W:
        res["W"] = _np(M.to_complex(out[:, :, 0]))
    return res


def exact(case, seed):
    c, k = case, case["kind"]
    if k != "serve":
        n = c["nx"] * c["ny"] * c["nz"]
        per_app = 1.0 * n * n * (c["L"] + 1) ** 2
        if per_app > (5e10 if k not in ("gradient", "fisher") else 1e9):
            return None  # over about 20 seconds
    with torch.no_grad():
        return _exact(c, k, _inputs(c, seed))


def _exact(c, k, s):
    if k == "serve":
        res = {}
        for q, (box, mua, mus, src) in enumerate(s["requests"]):
            r = _exact_forward(box, mua, mus, [src], s["stop"])
            res["trans%d" % q], res["ref%d" % q] = np.stack(r["trans"]), np.stack(r["ref"])
        return _kept(s, res)
    if k == "neumann":
        M = _Model(c, fim=True)
        mua, mus = (torch.tensor(t[s["tiss"]], **_T) for t in (s["mua_tab"], s["mus_tab"]))
        out, balls = M.series(M.kernel(mua + mus), mua + mus, mus, [s["src"]], s["stop"])
        tr, rf = M.images(out[:, :, 0], balls[0])
        return dict(W=_np(M.to_complex(out[:, :, 0])), trans=_np(tr.to(torch.complex128)),
                    ref=_np(rf.to(torch.complex128)))
    if k == "gradient":
        return _kept(s, _exact_gradient(c, s))
    if k == "fisher":
        return _kept(s, _exact_fisher(c, s))
    fp64 = c.get("prec") == "fp64"
    srcs = s["srcs"] if k == "batch" else [s["src"]]
    kappa = s["src"].modulation if k == "modulated" else 0.0
    r = _exact_forward(c, s["mua"], s["mus"], srcs, s["stop"], kappa, want_W=fp64)
    if k == "batch":
        return _kept(s, dict(trans=np.stack(r["trans"]), ref=np.stack(r["ref"])))
    return _kept(s, {q: (v if q == "W" else v[0]) for q, v in r.items()})


def _exact_gradient(c, s):
    M = _Model(c)
    mus = torch.tensor(s["mus"], **_T)
    mut0 = torch.tensor(s["mua"] + s["mus"], **_T)
    K0 = M.kernel(mut0)
    loss, g_mut, g_mus, gK = 0.0, torch.zeros(M.N, **_T), torch.zeros(M.N, **_T), torch.zeros_like(K0)
    for q, src in enumerate(s["srcs"]):
        with torch.enable_grad():
            K, mut, ms = (t.clone().requires_grad_() for t in (K0, mut0, mus))
            out, balls = _series_by_voxel(M, K, mut, ms, src, s["stop"])
            bins = M.flux_bins(out[:, :, 0], balls[0], c["nbins"])
            e = ((bins - torch.tensor(s["target"][q], **_T)) ** 2).sum()
            a, b, d = torch.autograd.grad(e, (K, mut, ms))
        loss += float(e)
        gK, g_mut, g_mus = gK + a, g_mut + b, g_mus + d
    g_mut = g_mut + M.kernel_gradient(K0, gK)
    return dict(loss=np.array([loss]), g_mua=_np(g_mut), g_mus=_np(g_mut + g_mus))


class _SelfTerm(torch.autograd.Function):
    """D(mu_t(r)) W[r] with the derivative in every voxel's mu_t."""

    @staticmethod
    def forward(ctx, mats, dmats, idx, mut, W):
        ctx.save_for_backward(mats, dmats, idx, W)
        return torch.bmm(mats[idx], W)

    @staticmethod
    def backward(ctx, g):
        mats, dmats, idx, W = ctx.saved_tensors
        return None, None, None, (g * torch.bmm(dmats[idx], W)).sum((1, 2)), torch.bmm(mats[idx].transpose(1, 2), g)


def _series_by_voxel(M, K, mut, mus, src, stop):
    vals, idx = np.unique(_np(mut), return_inverse=True)
    idx = torch.tensor(idx.ravel(), device=_DEV)
    with torch.no_grad():
        v = torch.tensor(vals, **_T)[:, None]
        f = (1 - torch.exp(-v * M.beta)) / v
        mats, dmats = M.contract(f), M.contract((M.beta * torch.exp(-v * M.beta) - f) / v)

    def apply(W, scatter):
        out = M.off_diagonal(K, W) + _SelfTerm.apply(mats, dmats, idx, mut, W)
        return out * (M.scat[None, :, None] * mus[:, None, None]) if scatter else out

    xi, b, f, p = M.beam(src, mut, mus)
    W = total = xi[:, :, None]
    for _ in range(stop.max_terms):
        W = apply(W, True)
        total = total + W
    return apply(total, False), [(b, f, p)]


def _exact_fisher(c, s):
    """Each parameter's derivative by a complex step (the model is analytic in the medium)."""
    M = _Model(c, g=0.9)
    P, h = len(s["dmua"]), 1e-20
    nb = c["nbins"]
    J = np.zeros((len(s["srcs"]), 6, nb, nb, P))
    F = np.zeros((P, P))
    y = None
    for p in range(P):
        mus = torch.tensor(s["mus"] + 1j * h * s["dmus"][p], device=_DEV)
        mut = torch.tensor(s["mua"] + s["mus"] + 1j * h * (s["dmua"][p] + s["dmus"][p]), device=_DEV)
        out, balls = M.series(M.kernel(mut), mut, mus, s["srcs"], s["stop"])
        bins = [_np(M.flux_bins(out[:, :, q], balls[q], nb)) for q in range(len(s["srcs"]))]
        for q, b in enumerate(bins):
            J[q, ..., p] = b.imag / h
        y = np.stack(bins).real
    w = np.where(y > 0, 1.0 / np.where(y > 0, y, 1.0), 0.0)
    F = np.einsum("sfabp,sfabq,sfab->pq", J, J, w)
    return dict(F=F, J=J)
