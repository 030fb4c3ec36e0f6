"""The workloads whose speed is followed from change to change.

Each case is one call that a program built on this package makes, through the public entry
points, on inputs made from a seed: the pressure solves, the 1-D boiling columns, the 2-D film
step, the level-set transport, the bubble statistics and the learned guess.  Sizes are those of
the package's benchmark, tests and training configurations, and the range around them.

  listed()            the followed cases
  draw(rng)           one more case of the same ranges
  prepare(case, seed) what a program holds before the call
  run(state)          one pass, its outputs
  work(case)          bytes and operations one pass cannot do without
  exact(case, seed)   the outputs by plain torch in 64 bits, where that is practical
"""
import math
import os
import tempfile

import numpy as np
import torch

from lica_boiling1d_b200 import autotune, bubbles, film2d, levelset, poisson, train_guess
from lica_boiling1d_b200.column import ColumnBatch, ColumnGeometry, ColumnProps, Columns, uneven_batch
from lica_boiling1d_b200.grid import Section, section
from lica_boiling1d_b200.unet import LearnedGuess

DEV = "cuda"

# launch shapes are tuned on this machine by this build, not read from another run's cache
os.environ["LICA_TUNE_CACHE"] = os.path.join(tempfile.mkdtemp(prefix="lica_tune_"), "column_tune.json")

# U-Net layers: inputs from below, inputs from the skip, outputs, level (half sizes per level)
UNET = ((16, 0, 32, 0), (32, 0, 32, 0), (32, 0, 64, 1), (64, 0, 64, 1), (64, 0, 128, 2), (128, 0, 128, 2),
        (128, 64, 64, 1), (64, 0, 64, 1), (64, 32, 32, 0), (32, 0, 32, 0))


def listed():
    return [
        # a small pressure solve on the host's critical path: launches and waits count
        dict(name="poisson_64", kind="poisson", nx=64, ny=64, precision="fp64", smoother="rb"),
        # the benchmark's pressure solve
        dict(name="poisson_1024", kind="poisson", nx=1024, ny=1024, precision="fp64", smoother="rb"),
        # the mixed-precision configuration's large grid
        dict(name="poisson_2048_mixed", kind="poisson", nx=2048, ny=2048, precision="mixed", smoother="rb"),
        # a wall-clustered grid, cells much finer in y: line relaxation
        dict(name="poisson_yline_256", kind="poisson", nx=256, ny=256, precision="fp64", smoother="yline"),
        # a short column stepped from a host program's own arrays, one step per call
        dict(name="column_host_128", kind="columns", ncol=1, n=128, steps=1, path="host", grid="uniform"),
        # the benchmark's single column, some steps of one launch
        dict(name="column_512", kind="columns", ncol=1, n=512, steps=20, path="device", grid="uniform"),
        # the benchmark's batch of thousands of uneven columns
        dict(name="columns_uneven_4096", kind="uneven", ncol=4096, nmin=128, nmax=2048, steps=3),
        # the 2-D film-boiling benchmark's steps
        dict(name="film_512x1536", kind="film", nx=512, ny=1536, precision="fp64", steps=2),
        # level-set transport of many columns (the per-substep call of a host time loop)
        dict(name="transport_1024x256", kind="transport", ncol=1024, n=256),
        # bubble statistics of several level sets on a 3-D grid
        dict(name="bubbles_4x256", kind="bubbles", nlvs=4, n1=256, n2=256, n3=256),
        # the learned initial guess of the benchmark's pressure solve
        dict(name="guess_1024", kind="guess", images=1, h=1024, w=1024),
        # the gradient of a training batch
        dict(name="guess_grad_4x256", kind="grad", images=4, h=256, w=256),
    ]


def _levels(nx, ny):
    return max(2, film2d.levels_for(nx, ny))


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["poisson", "poisson", "poisson", "yline", "columns", "columns", "uneven", "film", "transport",
                       "bubbles", "guess", "grad"])
    if kind in ("poisson", "yline"):
        while True:
            nx, ny = (rng.choice([16, 32, 48]) << rng.randint(1, 3 if kind == "yline" else 6) for _ in range(2))
            coarsest = nx * ny >> 2 * (_levels(nx, ny) - 1)
            if 64 <= min(nx, ny) and nx * ny <= 2048 * 2048 and max(nx, ny) <= 4 * min(nx, ny) and coarsest <= 2304:
                break
        return dict(kind="poisson", nx=nx, ny=ny, precision="fp64" if kind == "yline" else rng.choice(["fp64", "mixed"]),
                    smoother="rb" if kind == "poisson" else "yline")
    if kind == "columns":
        n = _log(rng, 64, 1024)
        path = rng.choice(["device", "device", "host"])
        return dict(kind="columns", ncol=_log(rng, 1, 256), n=n, steps=1 if path == "host" else rng.randint(2, 20),
                    path=path, grid=rng.choice(["uniform", "uniform", "tanh"]))
    if kind == "uneven":
        nmax = _log(rng, 256, 2048)
        return dict(kind="uneven", ncol=_log(rng, 64, 4096), nmin=max(64, nmax // rng.randint(2, 16)), nmax=nmax,
                    steps=3)
    if kind == "film":
        nx = 64 << rng.randint(0, 3)
        return dict(kind="film", nx=nx, ny=nx * rng.randint(1, 3), precision=rng.choice(["fp64", "mixed"]),
                    steps=rng.choice([1, 3]))
    if kind == "transport":
        return dict(kind="transport", ncol=_log(rng, 1, 4096), n=_log(rng, 64, 1024))
    if kind == "bubbles":
        while True:
            n1, n2, n3 = (_log(rng, 24, 300) for _ in range(3))
            nlvs = rng.randint(1, 8)
            if nlvs * n1 * n2 * n3 <= 4 * 256 ** 3:
                return dict(kind="bubbles", nlvs=nlvs, n1=n1, n2=n2, n3=n3)
    if kind == "guess":
        return dict(kind="guess", images=rng.randint(1, 4), h=64 * rng.randint(1, 8), w=64 * rng.randint(1, 8))
    return dict(kind="grad", images=rng.randint(1, 4), h=64 * rng.randint(1, 4), w=64 * rng.randint(1, 4))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _faces(rho):
    """1/rho on the faces of (..., ny, nx) cell densities (periodic in x, walls in y)."""
    bx = 2.0 / (rho + torch.roll(rho, 1, dims=-1))
    by = torch.empty(rho.shape[:-2] + (rho.shape[-2] + 1, rho.shape[-1]), dtype=torch.float64, device=DEV)
    by[..., 1:-1, :] = 2.0 / (rho[..., 1:, :] + rho[..., :-1, :])
    by[..., 0, :] = 1.0 / rho[..., 0, :]
    by[..., -1, :] = 1.0 / rho[..., -1, :]
    return bx.contiguous(), by


def _bubble_density(rng, nx, ny):
    """Density 1000 inside circles (64 per square, radii 8-48 cells at 1024 across), 1 outside."""
    scale = nx / 1024.0
    count = max(4, 64 * ny // nx)
    x = torch.arange(nx, device=DEV, dtype=torch.float64) + 0.5
    y = torch.arange(ny, device=DEV, dtype=torch.float64) + 0.5
    rho = torch.ones((ny, nx), dtype=torch.float64, device=DEV)
    for cx, cy, r in zip(rng.uniform(0, nx, count), rng.uniform(0, ny, count), rng.uniform(8, 48, count)):
        dx = (x - cx).abs()
        dx = torch.minimum(dx, nx - dx)
        rho[((y - cy) ** 2)[:, None] + (dx ** 2)[None, :] <= (max(2.0, r * scale)) ** 2] = 1000.0
    return rho


def _poisson_inputs(case, seed):
    """f, bx, by, hx, hy of the case's system (CUDA tensors)."""
    nx, ny = case["nx"], case["ny"]
    rng = np.random.default_rng(seed)
    f = torch.randn((ny, nx), generator=_gen(seed), dtype=torch.float64, device=DEV)
    if case["smoother"] == "rb":
        f -= f.mean()
        bx, by = _faces(_bubble_density(rng, nx, ny))
        return f, bx, by, 1.0 / nx, 1.0 / nx
    # wall-clustered faces (hyperbolic tangent), liquid with scattered vapour cells, density ratio 40
    y = np.zeros(ny + 1)
    section(Section(3, 0.0, 1.0, 1, ny + 1, 3, 3.0, 1.0), y)
    rho = torch.where(torch.rand((ny, nx), generator=_gen(seed + 1), device=DEV, dtype=torch.float64) < 0.2, 1.0, 40.0)
    bx, by = _faces(rho)
    bxs, bys, fs = poisson.stretched_system(y, bx.cpu().numpy(), by.cpu().numpy(), f.cpu().numpy())
    return tuple(torch.from_numpy(a).to(DEV) for a in (fs, bxs, bys)) + (1.0 / nx, 1.0)


def _props(seed):
    """A water-like column of the shipped range: 2-20 K of superheat, density ratio 100-1600."""
    rng = np.random.default_rng(seed)
    return ColumnProps(denr=float(rng.uniform(100.0, 1600.0)), visr=20.0, tcr=25.0,
                       jakob=0.009 * float(rng.uniform(0.2, 2.0)), cflmax=0.3), rng


def _columns(case, seed):
    props, rng = _props(seed)
    geo = ColumnGeometry.tanh(case["n"], 1.0, 1.5) if case["grid"] == "tanh" else None
    z0 = rng.uniform(0.08, 0.4, case["ncol"])
    return Columns.film(case["n"], 1.0, z0, props, geo), props


def _unet_inputs(case, seed):
    rng = np.random.default_rng(seed)
    h, w = case["h"], case["w"]
    rho = torch.stack([_bubble_density(rng, w, h) for _ in range(case["images"])])
    f = torch.randn((case["images"], h, w), generator=_gen(seed), dtype=torch.float64, device=DEV)
    f -= f.mean(dim=(1, 2), keepdim=True)
    yy = torch.arange(h, device=DEV, dtype=torch.float64)[:, None] / h
    xx = torch.arange(w, device=DEV, dtype=torch.float64)[None, :] / w
    gx0 = 1e3 * (1.0 + 0.5 * torch.sin(2 * math.pi * xx + seed % 7) * torch.cos(2 * math.pi * yy)) / rho
    return rho, f, gx0.contiguous(), 1.0 / w ** 2


def _bubble_inputs(case, seed):
    """Two rotated smeared ellipsoids per level set in a box of unit-sized cells, velocity noise."""
    rng = np.random.default_rng(seed)
    n1, n2, n3 = case["n1"], case["n2"], case["n3"]
    nm = max(n1, n2, n3)
    grid = bubbles.BubbleGrid.uniform(n1, n2, n3, n1 / nm, n2 / nm, n3 / nm)
    z, y, x = (torch.from_numpy(a).to(DEV) for a in (grid.zp, grid.yp, grid.xp))
    psi = torch.ones((case["nlvs"],) + grid.field_shape, dtype=torch.float64, device=DEV)
    box, small = np.array([n1, n2, n3]) / nm, min(n1, n2, n3) / nm
    for lv in range(case["nlvs"]):
        for _ in range(2):
            c = rng.uniform(0.3, 0.7, 3) * box
            ax = small * np.sort(rng.uniform(0.08, 0.28, 3))[::-1] * np.array([1.2, 1.0, 0.8])
            rot = np.linalg.qr(rng.standard_normal((3, 3)))[0]
            r2 = 0.0
            for a in range(3):
                d = (x - c[0])[None, None, :] * rot[0, a] + (y - c[1])[None, :, None] * rot[1, a] + \
                    (z - c[2])[:, None, None] * rot[2, a]
                r2 = r2 + (d / ax[a]) ** 2
            phi = (r2.sqrt_() - 1.0) * min(ax)
            torch.minimum(psi[lv], (0.5 + phi * (nm / 1.5)).clamp_(0.0, 1.0), out=psi[lv])
    for d in (1, 2, 3):
        psi.select(d, 0).fill_(1.0)
        psi.select(d, psi.shape[d] - 1).fill_(1.0)
    g = _gen(seed)
    u, v, w = (torch.randn(grid.field_shape, generator=g, dtype=torch.float64, device=DEV) for _ in range(3))
    return grid, psi, u, v, w


class _Kept:
    """A copy of a state's arrays, put back by a few copies (one per data type)."""

    def __init__(self, arrays):
        self.host = isinstance(next(iter(arrays.values())), np.ndarray)
        self.pairs = {}
        for a in arrays.values():
            to, kept = self.pairs.setdefault(a.dtype, ([], []))
            to.append(a)
            kept.append(a.copy() if self.host else a.clone())

    def restore(self):
        for to, kept in self.pairs.values():
            if self.host:
                for a, b in zip(to, kept):
                    a[...] = b
            else:
                torch._foreach_copy_(to, kept)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        f, bx, by, hx, hy = _poisson_inputs(case, seed)
        nx, ny = case["nx"], case["ny"]
        solver = poisson.MultigridPoisson(nx, ny, hx, hy, nlevels=_levels(nx, ny), ncoarse=1,
                                          precision=case["precision"], smoother=case["smoother"])
        return dict(kind=kind, solver=solver, p=torch.zeros_like(f), f=f, bx=bx, by=by)
    if kind == "columns":
        cols, props = _columns(case, seed)
        cols = cols if case["path"] == "host" else cols.to(DEV)
        return dict(kind=kind, start=_Kept(cols.arrays), cols=cols, props=props, steps=case["steps"])
    if kind == "uneven":
        # the sizes belong to the case, films and properties to the seed
        n, length, z0, _ = uneven_batch(case["ncol"], 0, case["nmin"], case["nmax"])
        props = uneven_batch(case["ncol"], seed, case["nmin"], case["nmax"])[3]
        z0 = z0 * np.random.default_rng(seed).uniform(0.8, 1.4, case["ncol"])
        batch = ColumnBatch.films(n, length, z0, props).to(DEV)
        autotune.tune(batch)   # the launch shape is chosen once per batch and kept
        return dict(kind=kind, start=_Kept(batch.arrays), batch=batch, steps=case["steps"])
    if kind == "film":
        rng = np.random.default_rng(seed)
        nx, ny = case["nx"], case["ny"]
        props = film2d.default_props()
        y0, amp = nx / 8.0 * rng.uniform(0.9, 1.3), nx / 128.0 * rng.uniform(0.6, 1.2)
        state = film2d.to_device(film2d.initial_state(nx, ny, y0, amp, props=props))
        film = film2d.Film2D(nx, ny, props, precision=case["precision"])
        return dict(kind=kind, film=film, start=_Kept(state), fields=state, dt=film2d.stable_dt(nx, props), steps=case["steps"])
    if kind == "transport":
        cols, props = _columns(dict(case, grid="uniform"), seed)
        rng = np.random.default_rng(seed + 1)
        n, nc, a = case["n"], case["ncol"], cols.arrays
        zz = np.arange(n + 2)[None, :] / n
        w = 3.0 * (rng.uniform(0.3, 1.0, (nc, 1)) +
                   0.3 * np.sin(2 * np.pi * (zz * rng.integers(1, 4, (nc, 1)) + rng.uniform(0, 1, (nc, 1)))))
        w[:, :2] = 0.0
        mf = np.where(a["layer"] > 0, 0.05 * rng.uniform(0.5, 1.0, a["phi"].shape), 0.0)
        vol = a["scal"][:, 3].copy()
        batch = levelset.ColumnBatch.from_arrays(n, 1.0, phi=a["phi"], layer=a["layer"], psif=a["psif"], wo=a["wo"],
                                                 vol_tot_ori=vol, psi_cn=a["psi_cn"], psi_zn=a["psi_zn"]).to(DEV)
        t = lambda v: torch.from_numpy(np.ascontiguousarray(v)).to(DEV)  # noqa: E731
        fields = {k: getattr(batch, k) for k in levelset.FIELDS}
        return dict(kind=kind, start=_Kept(fields), batch=batch, fields=fields, w=t(w), mf=t(mf), vi=t(vol * (1.0 + rng.uniform(0, 2e-4, nc))),
                    denr=props.denr)
    if kind == "bubbles":
        grid, psi, u, v, w = _bubble_inputs(case, seed)
        return dict(kind=kind, tracker=bubbles.BubbleTracker(grid, case["nlvs"]), fields=(psi, u, v, w))
    rho, f, gx0, hsq = _unet_inputs(case, seed)
    net = LearnedGuess(case["images"], case["h"], case["w"])
    train_guess.load(net)
    return dict(kind=kind, net=net, rho=rho, f=f, gx0=gx0, hsq=hsq)


# ------------------------------------------------------------------ one pass
def run(state):
    s, kind = state, state["kind"]
    if kind == "poisson":
        s["p"].zero_()
        s["solver"].solve(s["p"], s["f"], s["bx"], s["by"], rtol=1e-10, max_iters=200)
        return s["p"]
    if "start" in s:
        s["start"].restore()     # a run from a kept state
    if kind == "columns":
        status = s["cols"].steps(s["steps"], s["props"])
        return dict(s["cols"].arrays, status=status)
    if kind == "uneven":
        status = s["batch"].steps(s["steps"])
        return dict(s["batch"].arrays, status=status)
    if kind == "film":
        for _ in range(s["steps"]):
            s["film"].step(s["fields"], s["dt"])
        return s["fields"]
    if kind == "transport":
        status, stats = levelset.transport(s["batch"], s["w"], s["mf"], s["vi"], iphs=1, denr=s["denr"], dtconst=1e-3,
                                           first=0, m_step=50)
        return dict(s["fields"], status=status, stats=stats)
    if kind == "bubbles":
        rec = bubbles.records(s["tracker"].track(*s["fields"]))
        return {k: np.ascontiguousarray(rec[k]) for k in ("col", "vel", "vol")} | {"ami": np.sort(rec["ami"], axis=1)}
    if kind == "guess":
        return s["net"].guess(s["rho"], s["f"], s["hsq"])
    return s["net"].grad(s["rho"], s["f"], s["hsq"], s["gx0"])


# ------------------------------------------------------------------ necessary work
def _unet_flops(images, h, w):
    return images * sum(2.0 * 9 * (a + b) * co * (h >> lv) * (w >> lv) for a, b, co, lv in UNET)


def work(case):
    kind = case["kind"]
    if kind == "poisson":
        # p, f, bx, by once, and about a dozen V(2,2)-preconditioned CG iterations of 4/3 * 40 + 25 operations
        # per cell
        n = case["nx"] * case["ny"]
        return {"bytes": 8.0 * (4 * n + n + case["nx"]), "flops": 12 * 78.0 * n}
    if kind in ("columns", "uneven"):
        n = case["n"] if kind == "columns" else 0.5 * (case["nmin"] + case["nmax"])
        cells = case["ncol"] * n
        # 14 flow-sized state arrays' worth, read once and written once; three substeps of about 400 operations
        return {"bytes": 2 * 8.0 * 15 * cells, "flops": 3 * 400.0 * cells * case["steps"]}
    if kind == "film":
        n = case["nx"] * case["ny"]
        # u, v, p, theta and four phi per cell, in and out; per substep a dozen solver iterations and about 600
        # operations per cell
        return {"bytes": 2 * 8.0 * 8 * n, "flops": case["steps"] * 3 * (12 * 78.0 + 600.0) * n}
    if kind == "transport":
        # phi, layer, psif and the flow arrays in; all but w, mflvs out; the band's arithmetic
        return {"bytes": case["ncol"] * case["n"] * 8.0 * (2 + 1 + 2 + 1 + 2 + 1 + 2 + 2 + 1 + 2 + 1),
                "flops": case["ncol"] * 22 * 3 * 300.0}
    if kind == "bubbles":
        cells = case["n1"] * case["n2"] * case["n3"]
        return {"bytes": 8.0 * case["nlvs"] * cells * 1.03, "flops": 2.0 * case["nlvs"] * cells}
    hw = case["images"] * case["h"] * case["w"]
    if kind == "guess":
        return {"bytes": 3 * 8.0 * hw + 2 * 470593, "flops": _unet_flops(case["images"], case["h"], case["w"])}
    return {"bytes": 3 * 8.0 * hw + 6 * 470593, "flops": 3 * _unet_flops(case["images"], case["h"], case["w"])}


# ------------------------------------------------------------------ the outputs in 64 bits
def _exact_poisson(case, seed):
    """Conjugate gradients with a diagonal preconditioner, restarted from the true residual."""
    f, bx, by, hx, hy = _poisson_inputs(case, seed)
    cx, cy = 1.0 / hx ** 2, 1.0 / hy ** 2
    w, e = cx * bx, cx * torch.roll(bx, -1, dims=1)
    s, n = cy * by[:-1].clone(), cy * by[1:].clone()
    s[0] = 0.0
    n[-1] *= 2.0
    diag = w + e + s + n

    def a(p):   # -A p
        up, dn = torch.zeros_like(p), torch.zeros_like(p)
        up[:-1], dn[1:] = p[1:], p[:-1]
        return diag * p - w * torch.roll(p, 1, dims=1) - e * torch.roll(p, -1, dims=1) - n * up - s * dn
    p, best, best_p = torch.zeros_like(f), math.inf, None
    fn = float(f.norm())
    for _ in range(12):
        r = -f - a(p)
        rn = float(r.norm()) / fn
        if rn < best:
            gained, best, best_p = best / rn, rn, p.clone()
        else:
            gained = 1.0
        if best < 1e-15 or gained < 1.5:
            break
        z = r / diag
        d, x, rz = z.clone(), torch.zeros_like(p), (r * z).sum()
        r0 = float(r.norm())
        for it in range(12000):
            q = a(d)
            al = rz / (d * q).sum()
            x.add_(al * d)
            r.sub_(al * q)
            torch.div(r, diag, out=z)
            rzn = (r * z).sum()
            d.mul_(rzn / rz).add_(z)
            rz = rzn
            if it % 100 == 99 and float(r.norm()) < 1e-9 * r0:
                break
        p = p + x
    return best_p


def _exact_bubbles(case, seed):
    grid, psi, u, v, w = _bubble_inputs(case, seed)
    n1, n2, n3 = case["n1"], case["n2"], case["n3"]
    x, y, z = (torch.from_numpy(a[1:-1]).to(DEV) for a in (grid.xp, grid.yp, grid.zp))
    cell = float(grid.sdx[1] * grid.sdy[1] * grid.sdz[1])
    inner = (slice(1, n3 + 1), slice(1, n2 + 1), slice(1, n1 + 1))
    ip = torch.arange(2, n1 + 2, device=DEV)
    jp = torch.arange(2, n2 + 2, device=DEV)
    kp = torch.arange(2, n3 + 2, device=DEV)
    ip[-1], jp[-1] = 1, 1
    uc = 0.5 * (u[inner] + u[1:n3 + 1, 1:n2 + 1][:, :, ip])
    vc = 0.5 * (v[inner] + v[1:n3 + 1][:, :, 1:n1 + 1][:, jp])
    wc = 0.5 * (w[inner] + w[:, 1:n2 + 1, 1:n1 + 1][kp])
    vels, vols, amis = [], [], []
    for lv in range(case["nlvs"]):
        p = psi[lv][inner]
        g = (1.0 - p) * cell
        vol = g.sum()
        cx, cy, cz = ((g * q).sum() / vol for q in (x[None, None, :], y[None, :, None], z[:, None, None]))
        d = ((x - cx)[None, None, :], (y - cy)[None, :, None], (z - cz)[:, None, None])
        m = torch.stack([torch.stack([(g * d[i] * d[j]).sum() for j in range(3)]) for i in range(3)]) / vol
        vols.append(vol)
        vels.append(torch.stack([(g * q).sum() / vol for q in (uc, vc, wc)]))
        amis.append(torch.linalg.eigvalsh(m))
    return {"col": None, "vel": torch.stack(vels).cpu().numpy(), "vol": torch.stack(vols).cpu().numpy(),
            "ami": torch.stack(amis).cpu().numpy()}


def _unet64(params, rho, f, hsq):
    """The network in plain FP64 (no rounding between the layers)."""
    F = torch.nn.functional
    ws, o = [], 0
    for a, b, co, _ in UNET:
        k = co * 9 * (a + b)
        ws.append((params[o:o + k].view(co, 3, 3, a + b).permute(0, 3, 1, 2), params[o + k:o + k + co]))
        o += k + co
    wh, bh = params[o:o + 32], params[o + 32]
    sigma = f.square().mean(dim=(1, 2)).sqrt()[:, None, None]
    x = torch.zeros((f.shape[0], 16) + f.shape[1:], dtype=torch.float64, device=DEV)
    x[:, 0], x[:, 1] = torch.log10(rho) / 3.0, f / sigma

    def conv(k, t):
        # as nine matrix products: the direct 64-bit convolution is slow
        wt, b = ws[k]
        h, w = t.shape[2:]
        tp = F.pad(t, (1, 1, 1, 1))
        out = b[None, :, None].expand(t.shape[0], -1, h * w)
        for dy in range(3):
            for dx in range(3):
                out = out + wt[:, :, dy, dx] @ tp[:, :, dy:dy + h, dx:dx + w].reshape(t.shape[0], t.shape[1], h * w)
        return torch.relu(out).view(t.shape[0], -1, h, w)

    def up(t):
        return t.repeat_interleave(2, dim=2).repeat_interleave(2, dim=3)
    e1 = conv(1, conv(0, x))
    e2 = conv(3, conv(2, F.avg_pool2d(e1, 2)))
    m = conv(5, conv(4, F.avg_pool2d(e2, 2)))
    d2 = conv(7, conv(6, torch.cat([up(m), e2], dim=1)))
    d1 = conv(9, conv(8, torch.cat([up(d2), e1], dim=1)))
    return ((d1 * wh[None, :, None, None]).sum(dim=1) + bh) * sigma * hsq * rho


def exact(case, seed):
    kind = case["kind"]
    if kind == "poisson":
        return _exact_poisson(case, seed)
    if kind == "bubbles":
        return _exact_bubbles(case, seed)
    if kind in ("guess", "grad"):
        rho, f, gx0, hsq = _unet_inputs(case, seed)
        params = torch.from_numpy(np.load(train_guess.WEIGHTS).astype(np.float64)).to(DEV)
        if kind == "guess":
            return _unet64(params, rho, f, hsq)
        params.requires_grad_(True)
        (_unet64(params, rho, f, hsq) * gx0).sum().backward()
        return params.grad
    return None     # the column and film steps: some thousand lines of arithmetic, whose oracle is the test suite's
