"""Workloads of this framework, for measurement: the calls a user's program makes,
over the sizes it makes them at.

The systems are diamond-silicon supercells as in libisdf_b200/synth.py (random s/p
Gaussians on the diamond sites, orthonormalised over grid points), at 16 to 40 grid
points per cubic cell, with 32 states and 320 interpolation points per 8 atoms or fewer.

Kinds of case:
  solve    ISDF(): selection and fit of one system (selector Kmeans or QRCP, FP64 or
           mixed precision), the whole call of a GW / RPA / TDDFT / hybrid-functional code
  fit      fit(): theta for pivots that the program already has (an MD or SCF program
           that keeps its pivots while the orbitals move)
  select   kmeans_weight() and kmeans_select(): the points alone
  batch    kmeans_select_batch(): the points of several small systems at once, as the
           server's batcher runs them
  coulomb  coulomb_matrix(): the operator built from theta, its first consumer
"""
import math

import numpy as np
import torch

import libisdf_b200 as isdf
from libisdf_b200 import synth

_DEV = "cuda"
_user_stream = None


def _case(kind, name=None, grid=(16, 16, 16), cells=(1, 1, 1), nstate=32, window="all", mu=320,
          iters=100, selector="Kmeans", precision="fp64", factor=1.5, count=1):
    c = {} if name is None else {"name": name}
    c.update(kind=kind, nx=grid[0], ny=grid[1], nz=grid[2], cx=cells[0], cy=cells[1],
             cz=cells[2], nstate=nstate, window=window, mu=mu, iters=iters, selector=selector,
             precision=precision, factor=factor, count=count)
    return c


def listed():
    return [
        # the smallest whole solve: the reference's own Si8 example (16^3 grid, 16 valence
        # states, 192 points), where launches and latency are what a call costs
        _case("solve", "solve_si8_16", (16, 16, 16), (1, 1, 1), 32, "valence", 192, 500),
        # one 8-atom cell on the benchmark's 40^3 grid: the small request of the serving mix
        _case("solve", "solve_si8_40", (40, 40, 40), (1, 1, 1), 32, "all", 320),
        # 64 atoms, plain FP64: the medium request and the ordinary production size
        _case("solve", "solve_si64_80", (80, 80, 80), (2, 2, 2), 256, "all", 2048),
        # 216 atoms in the mixed-precision form: the largest (72^3 grid: 24 points per cell
        # edge, so that several states fit the card at once)
        _case("solve", "solve_si216_mixed", (72, 72, 72), (3, 3, 3), 864, "all", 4320, 100,
              "Kmeans", "mixed"),
        # valence x conduction pairs (GW / BSE) on an odd grid, two different factors
        _case("solve", "solve_window_odd", (45, 45, 75), (1, 1, 2), 128, "vc", 507),
        # the QRCP selector at the reference's oversampling
        _case("solve", "solve_qrcp", (48, 48, 48), (1, 2, 2), 128, "all", 640, 100, "QRCP",
              "fp64", 1.5),
        # a fit for known pivots, an odd number of points (K-means drops duplicates)
        _case("fit", "fit_fp64_1201", (64, 64, 60), (2, 2, 1), 160, "all", 1201),
        # the same in the mixed-precision form
        _case("fit", "fit_mixed_1600", (60, 60, 60), (2, 2, 2), 224, "all", 1600, 100, "Kmeans",
              "mixed"),
        # the points of a large system alone
        _case("select", "select_96", (96, 96, 96), (3, 3, 3), 96, "all", 3000),
        # eight small systems' points at once (serving)
        _case("batch", "batch_8x36", (36, 36, 36), (1, 1, 1), 32, "all", 256, 100, count=8),
        # the Coulomb operator of one cell and of a larger system
        _case("coulomb", "coulomb_si8", (40, 40, 40), (1, 1, 1), 32, "all", 320),
        _case("coulomb", "coulomb_1024", (60, 54, 64), (2, 2, 2), 192, "all", 1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "solve", "qrcp", "fit", "fit", "select", "batch",
                       "coulomb"])
    small = kind == "batch" or rng.random() < 0.4
    cells = (1, 1, 1) if small else tuple(rng.randint(1, 3) for _ in range(3))
    ncell = cells[0] * cells[1] * cells[2]
    # grid points per cell edge, the same along each direction up to a point or two (odd
    # extents among them); the larger the supercell, the coarser
    per = rng.uniform(16, 40 if ncell <= 8 else 26)
    grid = tuple(max(12, int(round(per * c)) + rng.randint(-1, 2)) for c in cells)
    ng = grid[0] * grid[1] * grid[2]
    nstate = max(16, int(32 * ncell * rng.uniform(0.6, 1.0)))
    window = rng.choice(["all", "all", "valence", "vc"])
    width = nstate if window == "all" else nstate // 2
    mu = max(48, min(4320, ng // 20, int(width * rng.uniform(5.0, 10.0))))
    precision = rng.choice(["fp64", "fp64", "mixed"])
    if kind in ("solve", "fit"):  # no dearer than the largest listed ones
        lim = 1.9e12 if precision == "fp64" else 6.5e12
        mu = min(mu, int(math.sqrt(lim / ng)))
    iters = rng.choice([50, 100, 100, 200])
    if kind == "qrcp":
        nstate, window = max(nstate, 24), "all"
        factor = rng.choice([1.5, 1.5, 2.0, 2.5])
        mu = min(mu, 800, int((nstate - 1) ** 2 / factor))
        return _case("solve", None, grid, cells, nstate, window, mu, iters, "QRCP", "fp64", factor)
    if kind == "batch":
        return _case("batch", None, grid, cells, nstate, window, min(mu, 512), iters,
                     count=_log_int(rng, 2, 24))
    if kind == "coulomb":
        return _case("coulomb", None, grid, cells, nstate, "all", min(mu, int(2.1e8 / ng), 1024),
                     iters)
    return _case(kind, None, grid, cells, nstate, window, mu, iters, "Kmeans", precision)


# ------------------------------------------------------------------ inputs
def _windows(c):
    """(nocc, nv1, nc1, nv2, nc2)"""
    n, occ = c["nstate"], c["nstate"] // 2
    if c["window"] == "all":
        return occ, occ, n - occ, occ, n - occ
    if c["window"] == "valence":
        return occ, occ, 0, occ, 0
    return occ, occ, 0, 0, n - occ  # "vc": valence x conduction pairs


def _grid(c):
    return c["nx"], c["ny"], c["nz"]


def _domain(c):
    return isdf.Domain(length=tuple(synth.A_SI * c[k] for k in ("cx", "cy", "cz")),
                       num_grid=_grid(c))


def _orbitals(c, seed):
    """(nstate, Ng) on the GPU: column-major psi."""
    rng = np.random.default_rng(seed)
    cells, n = (c["cx"], c["cy"], c["cz"]), _grid(c)
    frac = synth.diamond_sites(1)
    sites = np.concatenate([frac + synth.A_SI * np.array([i, j, k]) for i in range(cells[0])
                            for j in range(cells[1]) for k in range(cells[2])])
    per = 4 * synth.NEXP
    alpha = torch.from_numpy(rng.uniform(0.3, 1.5, size=(len(sites), per))).to(_DEV)
    coef = torch.from_numpy(rng.standard_normal((c["nstate"], len(sites) * per))).to(_DEV)
    length = [synth.A_SI * x for x in cells]
    axes = [torch.arange(n[d], dtype=torch.float64, device=_DEV) * (length[d] / n[d])
            for d in range(3)]
    ng = n[0] * n[1] * n[2]
    psi = torch.zeros((c["nstate"], ng), dtype=torch.float64, device=_DEV)
    for s, site in enumerate(sites):
        # minimum-image displacements; a Gaussian is a product over the directions
        d = [a - float(site[i]) for i, a in enumerate(axes)]
        d = [x - length[i] * torch.round(x / length[i]) for i, x in enumerate(d)]
        e = [torch.exp(-alpha[s][:, None] * x * x) for x in d]  # (per, n_i)
        for k in range(3):  # kinds s, px, py, pz in turn
            e[k][k + 1::4] *= d[k]
        g = (e[2][:, :, None] * e[1][:, None, :]).reshape(per, -1)  # (per, nz * ny)
        g = (g[:, :, None] * e[0][:, None, :]).reshape(per, ng)
        psi.addmm_(coef[:, s * per:(s + 1) * per], g)
    chol = torch.linalg.cholesky(psi @ psi.T)
    return torch.linalg.solve_triangular(chol, psi, upper=False).contiguous()


def _stream():
    """The program's stream for the calls that take one (the library's own otherwise)."""
    global _user_stream
    if _user_stream is None:
        _user_stream = torch.cuda.Stream()
    return _user_stream.cuda_stream


def _pivots(c, psi, dom, iters):
    """mu pivots: the selection drops duplicates, so it is asked for more and thinned."""
    w = torch.empty(dom.NumGridTotal(), dtype=torch.float64, device=_DEV)
    torch.cuda.synchronize()
    isdf.kmeans_weight(psi, w.numel(), c["nstate"], *_windows(c), w, stream=_stream())
    piv, rk, _, _ = isdf.kmeans_select(dom, w, int(1.3 * c["mu"]) + 16, iters, stream=_stream())
    assert rk >= c["mu"], "too few distinct points"
    return piv[np.linspace(0, rk - 1, c["mu"]).round().astype(np.int64)].copy()


def prepare(case, seed):
    c, dom = case, _domain(case)
    ng, s = dom.NumGridTotal(), {"case": case, "dom": dom}
    if c["kind"] == "batch":
        s["psi"] = [_orbitals(c, seed * 100 + i) for i in range(c["count"])]
        s["w"] = [torch.empty(ng, dtype=torch.float64, device=_DEV) for _ in s["psi"]]
    elif c["kind"] == "select":
        s["psi"] = _orbitals(c, seed)
        s["w"] = torch.empty(ng, dtype=torch.float64, device=_DEV)
    else:
        psi = _orbitals(c, seed)
        theta = torch.zeros((c["mu"], ng), dtype=torch.float64, device=_DEV)
        if c["kind"] == "solve":
            s.update(psi=psi, theta=theta, piv=np.zeros(ng, dtype=np.int32))
        elif c["kind"] == "fit":
            s.update(psi=psi, theta=theta, piv=_pivots(c, psi, dom, 30))
        else:
            piv = _pivots(c, psi, dom, 30)
            isdf.fit(psi, ng, c["nstate"], *_windows(c), c["mu"], piv, theta)
            s.update(theta=theta, A=torch.empty((c["mu"], c["mu"]), dtype=torch.float64,
                                                device=_DEV))
    torch.cuda.synchronize()
    return s


def run(s):
    c, dom = s["case"], s["dom"]
    ng = dom.NumGridTotal()
    win = _windows(c)
    if c["kind"] == "solve":
        opt = isdf.Options(precision=isdf.PRECISION_MIXED if c["precision"] == "mixed"
                           else isdf.PRECISION_FP64, qrcp_oversample=c["factor"])
        r = isdf.ISDF(s["psi"], dom, win[0], c["nstate"], *win[1:], c["mu"], s["theta"], s["piv"],
                      c["iters"], c["selector"], options=opt)
        return {"theta": s["theta"], "piv": s["piv"], "rk": r.rk_eff, "iters": r.kmeans_iters}
    if c["kind"] == "fit":
        isdf.fit(s["psi"], ng, c["nstate"], *win, c["mu"], s["piv"], s["theta"],
                 precision=isdf.PRECISION_MIXED if c["precision"] == "mixed"
                 else isdf.PRECISION_FP64)
        return {"theta": s["theta"]}
    stream = _stream()
    if c["kind"] == "select":
        isdf.kmeans_weight(s["psi"], ng, c["nstate"], *win, s["w"], stream=stream)
        piv, rk, iters, npt = isdf.kmeans_select(dom, s["w"], c["mu"], c["iters"], stream=stream)
        return {"w": s["w"], "piv": piv, "rk": rk, "iters": iters, "npt": npt}
    if c["kind"] == "batch":
        for psi, w in zip(s["psi"], s["w"]):
            isdf.kmeans_weight(psi, ng, c["nstate"], *win, w, stream=stream)
        got = isdf.kmeans_select_batch([dom] * c["count"], s["w"], [c["mu"]] * c["count"],
                                       [c["iters"]] * c["count"], stream=stream)
        return {"piv": np.stack([g[0] for g in got]),
                "rk_iters_npt": np.array([g[1:] for g in got], dtype=np.int64)}
    isdf.coulomb_matrix(dom, s["theta"], c["mu"], s["A"], stream=stream)
    return {"A": s["A"]}


# ------------------------------------------------------------------ cost
def work(case):
    """Selections count the orbitals (or their weight) in and the pivots out, one distance
    per point, and for QRCP the sketch; fits their products; the Coulomb matrix its
    transforms and one symmetric product."""
    c = case
    ng, mu, n = c["nx"] * c["ny"] * c["nz"], c["mu"], c["count"]
    _, nv1, nc1, nv2, nc2 = _windows(c)
    k1, k2 = nv1 + nc1, nv2 + nc2
    used = k1 if c["window"] != "vc" else k1 + k2
    kind = c["kind"]
    if kind in ("select", "batch"):
        return {"bytes": n * (8.0 * ng * used + 8.0 * ng + 4.0 * ng),
                "flops": n * (2.0 * ng * used + 8.0 * ng)}
    if kind == "coulomb":
        nh = (c["nx"] // 2 + 1) * c["ny"] * c["nz"]
        return {"bytes": 8.0 * ng * mu + 8.0 * mu * mu,
                "flops": mu * 2.5 * ng * math.log2(ng) + 2.0 * mu * (mu + 1) / 2 * 2 * nh}
    flops = 2.0 * ng * mu * (k1 if c["window"] != "vc" else k1 + k2)  # Z C^T
    flops += 2.0 * ng * mu * mu + mu ** 3 / 3.0  # triangular solves, Cholesky
    if c["selector"] == "QRCP":
        p = round(math.sqrt(mu * c["factor"]))
        flops += 2.0 * ng * p * (k1 + k2)
    return {"bytes": 8.0 * ng * used + 8.0 * ng * mu, "flops": flops}


# ------------------------------------------------------------------ 64-bit results
def exact(case, seed):
    """In torch, double precision throughout. Whole solves have none (their pivots decide
    theta), nor have the selections, whose results are whole numbers."""
    c = case
    if c["kind"] == "select":
        psi = _orbitals(c, seed)
        occ, nv1, nc1, nv2, nc2 = _windows(c)
        s1, s2 = psi[occ - nv1:occ + nc1], psi[occ - nv2:occ + nc2]
        return {"w": (s1 * s1).sum(0) * (s2 * s2).sum(0), "piv": None, "rk": None, "iters": None,
                "npt": None}
    if c["kind"] not in ("fit", "coulomb"):
        return None
    s = prepare(case, seed)
    dom = s["dom"]
    ng, mu = dom.NumGridTotal(), c["mu"]
    if c["kind"] == "fit":
        occ, nv1, nc1, nv2, nc2 = _windows(c)
        psi, piv = s["psi"], torch.from_numpy(s["piv"].astype(np.int64)).to(_DEV)
        s1, s2 = psi[occ - nv1:occ + nc1], psi[occ - nv2:occ + nc2]
        z = (s1[:, piv].T @ s1) * (s2[:, piv].T @ s2)  # (mu, Ng): Z C^T transposed
        cct = z[:, piv]
        eps = 1e-10 * (torch.diagonal(cct).sum() / mu)
        chol = torch.linalg.cholesky(cct + eps * torch.eye(mu, dtype=torch.float64, device=_DEV))
        return {"theta": torch.cholesky_solve(z, chol)}
    nx, ny, nz = _grid(c)
    lx, ly, lz = dom.length
    k = [2 * math.pi * n * torch.fft.fftfreq(n, d=1.0, dtype=torch.float64, device=_DEV) / ln
         for n, ln in ((nz, lz), (ny, ly), (nx, lx))]
    g2 = k[0][:, None, None] ** 2 + k[1][None, :, None] ** 2 + k[2][None, None, :] ** 2
    radius = 5.0
    v = torch.where(g2 < 2e-8, torch.full_like(g2, 4 * math.pi * radius * radius),
                    8 * math.pi / g2.clamp_min(1e-30) * (1 - torch.cos(g2.sqrt() * radius)))
    sv = (v.sqrt() * (lx * ly * lz / ng)).reshape(-1)
    step = max(1, int(2.5e8) // ng)
    zeta = [(torch.fft.fftn(s["theta"][i:i + step].reshape(-1, nz, ny, nx), dim=(1, 2, 3))
             .reshape(-1, ng) * sv) for i in range(0, mu, step)]
    zeta = torch.cat(zeta)
    return {"A": zeta.real @ zeta.real.T + zeta.imag @ zeta.imag.T}
