"""The work that users of this framework have it do, as timed cases.

A pass is what a program calls for one simulation on a handle that it keeps:
``reset(); run(steps)`` and the receiver traces (with the final fields where
the domain is small enough for a program to look at them), or one iteration
of a permittivity inversion: a new model into the handle, the recorded
forward run, the misfit and its gradient.

Families
  fdtd   Yee grid, FP64 (the reference's own arithmetic) or FP32, PEC box or
         CPML, uniform or per-cell eps and sigma.
  hex    hexahedral edge elements of order 1 or 2 (the reference's fem_v2,
         symplectic_2 and symplectic_4 programs), FP64 or FP32.
  tet    tetrahedral Nedelec elements of order 1 or 2, one mesh or a batch of
         shots on cubes of uneven size, forward runs and gradients.

Every source, material, receiver and observed trace comes from the seed.
``exact`` restates each scheme in 64 bits with plain torch operations."""
import math
import os

import numpy as np
import torch

import emsolvers_gb300 as ems

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
KMAT = os.path.join(ROOT, "tests", "golden", "kmat")
EPS0, MU0, C0 = 8.854187817e-12, 1.25663706212e-6, 299792458.0
H = 1e-3                       # cell size [m]
TS = H / C0                    # seconds per normalised time unit of the tetrahedral solvers
X1 = 1.0 / (2.0 - 2.0 ** (1.0 / 3.0))
SUB = {"symp2": (1.0,), "symp4": (X1, 1.0 - 2.0 * X1, X1)}   # substeps of the symplectic integrators
INTEG = {"leapfrog": ems.LEAPFROG, "symp2": ems.SYMP2, "symp4": ems.SYMP4}


def _fdtd(name, nx, ny, nz, steps, prec, pml, blocks, nrec, fields):
    return {"name": name, "family": "fdtd", "nx": nx, "ny": ny, "nz": nz, "steps": steps, "prec": prec, "pml": pml,
            "blocks": blocks, "nrec": nrec, "fields": fields}


def _hex(name, order, nx, ny, nz, steps, prec, integ, nrec):
    return {"name": name, "family": "hex", "order": order, "nx": nx, "ny": ny, "nz": nz, "steps": steps, "prec": prec,
            "integ": integ, "nrec": nrec}


def _tet(name, order, shots, steps, prec, integ, nrec, grad=False, sigma=False):
    return {"name": name, "family": "tet", "order": order, "shots": shots, "steps": steps, "prec": prec, "integ": integ,
            "nrec": nrec, "grad": grad, "sigma": sigma}


def listed():
    return [
        # the smallest call: a quick look at a tiny box, where launches and call overhead are all there is
        _fdtd("fdtd_small_fp64", 24, 20, 16, 60, 64, 0, 0, 2, True),
        # the reference-sized FP64 run: a dielectric obstacle in a 64^3 PEC box, 1000 steps, 8 receivers
        _fdtd("fdtd_64_fp64", 64, 64, 64, 1000, 64, 0, 16, 8, True),
        # an ordinary open-boundary study on an odd grid: FP32, 10-cell CPML, lossy dielectric blocks
        _fdtd("fdtd_cpml_fp32", 141, 117, 93, 200, 32, 10, 16, 8, True),
        # a large open domain: the traces of 64 receivers
        _fdtd("fdtd_large_fp32", 400, 384, 368, 60, 32, 10, 16, 64, False),
        # the reference's leapfrog program on order-1 hexahedra, FP64, odd sizes
        _hex("hex1_leapfrog_fp64", 1, 37, 33, 41, 300, 64, "leapfrog", 3),
        # order-2 hexahedra under the 4th-order symplectic step, FP32
        _hex("hex2_symp4_fp32", 2, 72, 72, 72, 100, 32, "symp4", 4),
        # one order-1 tetrahedral solve, 32^3 cubes x 6, 2000 steps
        _tet("tet1_32_symp4_fp32", 1, "32x32x32", 2000, 32, "symp4", 8),
        # a batch of order-1 shots of uneven size
        _tet("tet1_batch_fp32", 1, "12x12x12,40x40x40,27x27x27,33x33x33,19x19x19,36x36x36,23x23x23,38x38x38,15x15x15,29x29x29",
             300, 32, "symp4", 2),
        # one inversion iteration on order-1 tetrahedra: four shots, lossy start model
        _tet("tet1_gradient_fp32", 1, "28x28x28,28x28x28,28x28x28,28x28x28", 300, 32, "symp4", 16, grad=True, sigma=True),
        # one order-2 forward model at the size of the inversion mesh
        _tet("tet2_48_fp32", 2, "48x48x48", 20, 32, "symp4", 8),
        # a batch of order-2 shots of uneven size
        _tet("tet2_batch_fp32", 2, "21x21x21,35x35x35,12x12x12,40x40x40,30x30x30", 12, 32, "symp4", 2),
        # one inversion iteration on order-2 tetrahedra
        _tet("tet2_gradient_fp32", 2, "24x22x23", 30, 32, "symp4", 16, grad=True),
    ]


def draw(rng):
    def ilog(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["fdtd", "fdtd", "hex", "tet1", "tet2", "tet1g", "tet2g"])
    if kind == "fdtd":
        prec = rng.choice([64, 32, 32])
        n = [ilog(16, 112 if prec == 64 else 288) for _ in range(3)]
        pml = rng.choice([0, 6, 10]) if min(n) > 24 else 0
        cells = n[0] * n[1] * n[2]
        return {k: v for k, v in _fdtd("", *n, min(ilog(60, 1000), max(30, int(2e9 / cells))), prec, pml,
                                       rng.choice([0, 16, 8]), ilog(1, 64), cells < 3e6).items() if k != "name"}
    if kind == "hex":
        order = rng.choice([1, 2])
        integ = rng.choice(["leapfrog", "symp2", "symp4"])
        n = [order * ilog(6, 72 // order) for _ in range(3)]
        cost = n[0] * n[1] * n[2] * order ** 2 * (3 if integ == "symp4" else 1)
        return {k: v for k, v in _hex("", order, *n, min(ilog(30, 300), max(10, int(2e8 / cost))), rng.choice([64, 32]), integ,
                                      rng.randint(1, 4)).items() if k != "name"}
    order, grad = int(kind[3]), kind.endswith("g")
    if grad or rng.random() < 0.4:
        n = [ilog(8, 36 if order == 1 else 24) for _ in range(3)]
        shots = ["%dx%dx%d" % tuple(n)] * (rng.choice([1, 2, 4]) if order == 1 else 1)
    else:
        shots = ["%dx%dx%d" % (n, n, n) for n in (rng.randint(12, 40) for _ in range(rng.randint(1, 8 if order == 1 else 4)))]
    nodes = sum((a + 1) * (b + 1) * (c + 1) for a, b, c in _cells(",".join(shots)))
    prec = rng.choice([32, 32, 64]) if nodes < (60000 if order == 1 else 8000) else 32
    if order == 1:
        steps = min(ilog(100, 2000), max(60, int((4e7 if grad else 1.2e8) / nodes)))
    else:
        steps = min(ilog(8, 60), max(4, int((5e5 if grad else 2e6) / nodes)))
    integ = rng.choice(["symp4", "symp2"] if grad else ["symp4", "symp4", "symp2", "leapfrog"])
    return {k: v for k, v in _tet("", order, ",".join(shots), steps, prec, integ, rng.randint(1, 16), grad,
                                  grad and order == 1 and rng.random() < 0.5).items() if k != "name"}


def _cells(shots):
    return [tuple(int(v) for v in s.split("x")) for s in shots.split(",")]


# ------------------------------------------------------------------- inputs
def _fdtd_inputs(c, seed):
    r = np.random.default_rng(seed)
    n = np.array([c["nx"], c["ny"], c["nz"]])
    dt = 0.99 * H / (2.998e8 * math.sqrt(3.0))
    eps = sig = None
    if c["blocks"]:
        b = c["blocks"]
        m = [-(-int(v) // b) for v in n]
        idx = [torch.arange(int(v)) // b for v in n]
        pick = (idx[0][None, None, :] + m[0] * (idx[1][None, :, None] + m[1] * idx[2][:, None, None])).reshape(-1)
        eps = torch.from_numpy(10 ** r.uniform(0, 1, m[0] * m[1] * m[2]) * EPS0)[pick].numpy()
        sig = torch.from_numpy(r.uniform(0, 0.05, m[0] * m[1] * m[2]))[pick].numpy()
    lo = np.minimum(c["pml"] + 2, n // 3)
    # every component is driven: with one alone its H component stays at the rounding of zero
    srcs = [(q % 3, tuple(int(v) for v in r.integers(lo, n - lo)), float(r.uniform(5e9, 15e9)), float(r.uniform(0.5, 2)))
            for q in range(4)]
    recs = []
    for q in range(c["nrec"]):   # near a source: within the reach of the wave
        at = np.array(srcs[q % 4][1]) + r.integers(-12, 13, 3)
        recs.append(tuple(int(v) for v in np.clip(at, 1, n - 1)))
    return dt, eps, sig, srcs, recs


def _hex_inputs(c, seed):
    r = np.random.default_rng(seed)
    n = np.array([c["nx"], c["ny"], c["nz"]])
    h = 0.05
    dt = float(r.uniform(0.9, 1.0)) * h / (2.998e8 * math.sqrt(3.0)) / 2.0
    srcs = [(q, tuple(int(v) for v in r.integers(n // 3, n - n // 3))) for q in range(3)]
    recs = [tuple(int(v) for v in np.clip(np.array(srcs[q % 3][1]) + r.integers(-3, 4, 3), 1, n - 1)) for q in range(c["nrec"])]
    return h, dt, srcs, recs


# time step in units of H / c0: inside the stability limit for eps_r >= 1
_DT = {1: {"symp4": 0.15, "symp2": 0.17, "leapfrog": 0.17}, 2: {"symp4": 0.055, "symp2": 0.062, "leapfrog": 0.062}}


def _blobs(cells, r):
    """eps_r of one shot: 2 plus three Gaussian blobs, at the tetrahedron centroids."""
    off = np.zeros((6, 3))
    for p, (a, b, c) in enumerate(_PERM):
        off[p, a], off[p, b], off[p, c] = 0.75, 0.5, 0.25
    k, j, i = np.meshgrid(*[np.arange(v) for v in cells[::-1]], indexing="ij")
    x = (np.stack([i.ravel(), j.ravel(), k.ravel()], 1)[:, None, :] + off).reshape(-1, 3)
    e = np.full(x.shape[0], 2.0)
    for _ in range(3):
        c, amp, w = r.uniform(0.25, 0.75, 3) * np.array(cells), r.uniform(1, 3), r.uniform(0.1, 0.2) * max(cells)
        e += amp * np.exp(-((x - c) ** 2).sum(1) / (2 * w * w))
    return e


def _tet_inputs(c, seed):
    r = np.random.default_rng(seed)
    cells = _cells(c["shots"])
    eps = [_blobs(s, r) if c["grad"] else r.uniform(1.0, 4.0, 6 * s[0] * s[1] * s[2]) for s in cells]
    sig = [r.uniform(0, 0.02, e.size) for e in eps] if c["sigma"] else None
    src = [r.uniform(0.35, 0.65, 3) * np.array(s) for s in cells]
    # within a few cells of the source: reached by the wave in a short run
    rec = [[np.clip(src[k] + r.uniform(-4, 4, 3), 0.3, np.array(s) - 0.3) for _ in range(c["nrec"])] for k, s in enumerate(cells)]
    dt = _DT[c["order"]][c["integ"]] * float(r.uniform(0.97, 1.0))
    f0 = 0.1 / math.sqrt(2.5)   # 10 cells per wavelength
    obs = None
    if c["grad"]:   # observed traces: the size of the signal, from the seed
        nrec = c["nrec"] * len(cells)
        t = np.arange(c["steps"]) * dt
        obs = np.zeros((nrec, c["steps"], 4))
        obs[..., 0] = t * TS
        obs[..., 1:] = r.normal(0, 0.02, (nrec, 1, 3)) * np.sin(2 * np.pi * f0 * t)[None, :, None]
    return cells, eps, sig, src, rec, dt, f0, obs


# ------------------------------------------------------------- entry points
def prepare(case, seed):
    c = case
    prec = ems.FP64 if c["prec"] == 64 else ems.FP32
    if c["family"] == "fdtd":
        dt, eps, sig, srcs, recs = _fdtd_inputs(c, seed)
        s = ems.FdtdSimulation((c["nx"], c["ny"], c["nz"]), H, dt, EPS0, MU0, 1, precision=prec, pml_cells=c["pml"])
        if eps is not None:
            s.set_material(eps, sig)
        for comp, at, f0, amp in srcs:
            (s.setSource_x, s.setSource_y, s.setSource_z)[comp](at, waveform=ems.WAVE_RICKER, f0=f0, amplitude=amp)
        for q in recs:
            s.setObservationPoint(([q], [q], [q]))
        return {"case": c, "sim": s}
    if c["family"] == "hex":
        h, dt, srcs, recs = _hex_inputs(c, seed)
        s = ems.HexFemSimulation(c["order"], (c["nx"], c["ny"], c["nz"]), h, dt, EPS0, MU0, 1, 1, integrator=INTEG[c["integ"]],
                                 precision=prec, kmat_dir=KMAT)
        for comp, at in srcs:
            (s.setSource_x, s.setSource_y, s.setSource_z)[comp](at)
        for q in recs:
            s.setObservationPoint(q)
        return {"case": c, "sim": s}
    cells, eps, sig, src, rec, dt, f0, obs = _tet_inputs(c, seed)
    batch = len(cells) > 1
    kw = dict(order=c["order"], integrator=INTEG[c["integ"]], precision=prec, dt=dt * TS)
    s = ems.TetFemBatch(cells, H, **kw) if batch else ems.TetFemSimulation(cells[0], H, **kw)
    eps, sig = np.concatenate(eps), None if sig is None else np.concatenate(sig)
    s.set_material(eps, sig)
    for k in range(len(cells)):
        shot = (k,) if batch else ()
        s.add_dipole(*shot, src[k] * H, (0.0, 0.6, 0.8), ems.WAVE_RICKER, f0 / TS, 1.0)
        for q in rec[k]:
            s.add_receiver(*shot, q * H)
    s.time_step()   # a program looks at the time step and its limit before it runs
    return {"case": c, "sim": s, "eps": eps, "sig": sig, "obs": obs}


def run(state):
    c, s = state["case"], state["sim"]
    if c["family"] == "tet" and c["grad"]:   # one inversion iteration: the model enters on every pass
        s.set_material(state["eps"], state["sig"])
        out = s.gradient(c["steps"], state["obs"], kind=0, nsnap=8, sigma=c["sigma"])
        return {"misfit": out[0], "grad": out[1:], "traces": s.traces()[..., 1:]}
    s.reset()
    s.run(c["steps"])
    if c["family"] == "fdtd":
        return {"traces": s.traces(), "fields": [s.get_field(q) for q in range(6)] if c["fields"] else []}
    if c["family"] == "hex":
        return {"traces": s.traces()[..., 1:], "fields": s.levels()}
    return {"traces": s.traces()[..., 1:], "fields": [s.get_field(0)]}


def work(case):
    """The bytes and operations of one pass that the scheme itself asks for."""
    c, w = case, case["prec"] // 8
    if c["family"] == "fdtd":
        n = c["nx"] * c["ny"] * c["nz"]
        inner = (c["nx"] - 2 * c["pml"]) * (c["ny"] - 2 * c["pml"]) * (c["nz"] - 2 * c["pml"])
        # per step E and H read and written once, the material's 2-byte id, the layer's auxiliary values
        return {"bytes": c["steps"] * (12 * w * n + (2 * n if c["blocks"] else 0) + 16 * w * (n - inner)),
                "flops": c["steps"] * (36 * n + 24 * (n - inner))}
    if c["family"] == "hex":
        o = c["order"]
        ne, t = (c["nx"] // o) * (c["ny"] // o) * (c["nz"] // o), 3 * o * (o + 1) ** 2
        nd = 3 * c["nx"] * c["ny"] * c["nz"]
        kicks = 1 if c["integ"] == "leapfrog" else len(SUB[c["integ"]])
        return {"bytes": c["steps"] * kicks * nd * w * (3 if c["integ"] == "leapfrog" else 4), "flops": c["steps"] * kicks * 2 * t * t * ne}
    nodes = sum((a + 1) * (b + 1) * (d + 1) for a, b, d in _cells(c["shots"]))
    subs = 1 if c["integ"] == "leapfrog" else len(SUB[c["integ"]])
    runs = 3 if c["grad"] else 1   # forward, recomputed forward, adjoint
    if c["order"] == 1:   # U and P read and written, the node's mass block read
        return {"bytes": runs * c["steps"] * subs * nodes * w * 56, "flops": runs * c["steps"] * subs * nodes * 500}
    # every substep: 28 iterations (right-hand side, iterate and step of the 38 values of a node), one stiffness apply
    return {"bytes": runs * c["steps"] * subs * nodes * w * (28 * 38 * 5 + 38 * 6), "flops": runs * c["steps"] * subs * nodes * 6 * (28 * 800 + 960)}


# -------------------------------------------------- the schemes in 64 bits
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def exact(case, seed):
    c = case
    if c["family"] == "fdtd":
        return _exact_fdtd(c, seed)
    if c["family"] == "hex":
        return _exact_hex(c, seed)
    return _exact_tet(c, seed, _Tet1 if c["order"] == 1 else _Tet2)


def _exact_fdtd(c, seed):
    """Yee leapfrog with per-cell materials and a convolutional PML (Roden and Gedney 2000)."""
    dt, eps, sig, srcs, recs = _fdtd_inputs(c, seed)
    nx, ny, nz = n = (c["nx"], c["ny"], c["nz"])
    f8, dev = torch.float64, _dev()
    se = [(nz + 2, ny + 2, nx + 1), (nz + 2, ny + 1, nx + 2), (nz + 1, ny + 2, nx + 2)]
    sh = [(nz + 1, ny + 1, nx), (nz + 1, ny, nx + 1), (nz, ny + 1, nx + 1)]
    E = [torch.zeros(s, dtype=f8, device=dev) for s in se]
    Hf = [torch.zeros(s, dtype=f8, device=dev) for s in sh]
    ch, ce = dt / MU0 / H, dt / EPS0 / H
    if eps is not None:
        e = torch.from_numpy(eps).to(dev).reshape(nz, ny, nx)
        s = torch.from_numpy(sig).to(dev).reshape(nz, ny, nx) * dt / (2 * e)
        div, A, B = 1 + s, (1 - s) / (1 + s), dt / e / H / (1 + s)

        def edge(v, d):   # Ex along x has one value more than cells: the last cell's again (Ey, Ez alike)
            last = v.narrow(2 - d, v.shape[2 - d] - 1, 1)
            return torch.cat([v, last], 2 - d)

        ca, cb = [edge(A, d) for d in range(3)], [edge(B, d) for d in range(3)]
    L = c["pml"]

    def prof(m, shift):
        x = np.arange(m + 2) + shift
        d = np.clip(np.maximum(L - x, x - (m - L)), 0, L) / L
        smax = -4.0 * math.log(1e-6) / (2.0 * math.sqrt(MU0 / EPS0) * L * H)
        sg = smax * d ** 3
        b = np.where(d > 0, np.exp(-sg * dt / EPS0), 0.0)
        a = np.where(d > 0, b - 1.0, 0.0)
        return torch.from_numpy(b).to(dev), torch.from_numpy(a).to(dev)

    if L:
        pe, ph = [prof(m, -0.5) for m in n], [prof(m, 0.0) for m in n]
    psi = {}

    def stretch(key, d, axis, p, lo):
        """d plus its auxiliary value along one axis (grid index lo upward)."""
        if not L:
            return d
        shape = [1, 1, 1]
        shape[2 - axis] = -1
        m = d.shape[2 - axis]
        b, a = p[axis][0][lo:lo + m].reshape(shape), p[axis][1][lo:lo + m].reshape(shape)
        if key not in psi:
            psi[key] = torch.zeros_like(d)
        psi[key].mul_(b).addcmul_(d, a.expand_as(d))
        return d + psi[key]

    ns = len(srcs)
    tr = torch.zeros((len(recs), c["steps"] + 1, 3), dtype=f8, device=dev)
    ridx = [tuple(torch.tensor([q[2 - a] for q in recs], device=dev) for a in range(3)) for _ in range(3)]
    t = 0.0
    for step in range(1, c["steps"] + 1):
        Ex, Ey, Ez = E
        Hx, Hy, Hz = Hf
        # H on its whole array: index (k, j, i)
        dzy, dyz = Ez[:, 1:, 1:] - Ez[:, :-1, 1:], Ey[1:, :, 1:] - Ey[:-1, :, 1:]
        Hx.sub_(stretch("h0", dzy[:, :, :nx], 1, ph if L else None, 0) - stretch("h1", dyz[:, :, :nx], 2, ph if L else None, 0), alpha=ch)
        dxz, dzx = Ex[1:, 1:, :] - Ex[:-1, 1:, :], Ez[:, 1:, 1:] - Ez[:, 1:, :-1]
        Hy.sub_(stretch("h2", dxz[:, :ny, :], 2, ph if L else None, 0) - stretch("h3", dzx[:, :ny, :], 0, ph if L else None, 0), alpha=ch)
        dyx, dxy = Ey[1:, :, 1:] - Ey[1:, :, :-1], Ex[1:, 1:, :] - Ex[1:, :-1, :]
        Hz.sub_(stretch("h4", dyx[:nz], 0, ph if L else None, 0) - stretch("h5", dxy[:nz], 1, ph if L else None, 0), alpha=ch)
        # E inside (indices from 1 in the two directions across the component)
        cur = [stretch("e0", Hz[:, 1:] - Hz[:, :-1], 1, pe if L else None, 1) - stretch("e1", Hy[1:] - Hy[:-1], 2, pe if L else None, 1),
               stretch("e2", Hx[1:] - Hx[:-1], 2, pe if L else None, 1) - stretch("e3", Hz[:, :, 1:] - Hz[:, :, :-1], 0, pe if L else None, 1),
               stretch("e4", Hy[:, :, 1:] - Hy[:, :, :-1], 0, pe if L else None, 1) - stretch("e5", Hx[:, 1:] - Hx[:, :-1], 1, pe if L else None, 1)]
        inner = [Ex[1:nz + 1, 1:ny + 1, :], Ey[1:nz + 1, :, 1:nx + 1], Ez[:, 1:ny + 1, 1:nx + 1]]
        for d in range(3):
            if eps is None:
                inner[d].add_(cur[d], alpha=ce)
            else:
                inner[d].mul_(ca[d]).addcmul_(cb[d], cur[d])
        for s in range(ns):
            comp, at, f0, amp = srcs[s]
            tau = t - math.sqrt(2.0) / f0
            g = (1 - 2 * math.pi ** 2 * f0 ** 2 * tau ** 2) * math.exp(-math.pi ** 2 * f0 ** 2 * tau ** 2) / H ** 3 * 0.001
            ep, dv = EPS0, 1.0
            if eps is not None:
                cell = [at[d] - 1 if d != comp else min(at[d], n[d] - 1) for d in range(3)]
                if step == 1:
                    psi["s%d" % s] = (float(e[cell[2], cell[1], cell[0]]), float(div[cell[2], cell[1], cell[0]]))
                ep, dv = psi["s%d" % s]
            E[comp][at[2], at[1], at[0]] -= g * amp * dt / ep / dv
        for d in range(3):
            tr[:, step, d] = E[d][ridx[d]]
        t += dt
    return {"traces": tr.cpu().numpy(), "fields": [v.reshape(-1).cpu().numpy() for v in E + Hf] if c["fields"] else []}


def _kmat(order):
    def val(s):
        p = s.strip().strip('"').split("/")
        return float(p[0]) / float(p[1]) if len(p) == 2 else float(p[0])

    with open(os.path.join(KMAT, "%d.csv" % order)) as f:
        return np.array([[val(v) for v in line.split(",") if v.strip()] for line in f if line.strip()])


def _exact_hex(c, seed):
    """K of every element applied to its edge values, summed; leapfrog or symplectic steps."""
    h, dt, srcs, recs = _hex_inputs(c, seed)
    o, dev, f8 = c["order"], _dev(), torch.float64
    n = (c["nx"], c["ny"], c["nz"])
    ne = [v // o for v in n]
    shape = [tuple(n[a] + (0 if a == d else 1) for a in (2, 1, 0)) for d in range(3)]
    size = [int(np.prod(s)) for s in shape]
    base = np.concatenate([[0], np.cumsum(size)])
    ek, ej, ei = np.meshgrid(*[np.arange(v) for v in ne[::-1]], indexing="ij")
    cols, pec = [], []
    for d in range(3):
        ext = [o + (0 if a == d else 1) for a in range(3)]
        for z in range(ext[2]):
            for y in range(ext[1]):
                for x in range(ext[0]):
                    cols.append((base[d] + (o * ei + x) + shape[d][2] * ((o * ej + y) + shape[d][1] * (o * ek + z))).reshape(-1))
        k, j, i = np.meshgrid(*[np.arange(v) for v in shape[d]], indexing="ij")
        pos = (i, j, k)
        pec.append(np.any([(pos[a] == 0) | (pos[a] == n[a]) for a in range(3) if a != d], axis=0).reshape(-1))
    dof = torch.from_numpy(np.stack(cols)).to(dev)
    live = torch.from_numpy((~np.concatenate(pec)).astype(np.float64)).to(dev)
    leap = c["integ"] == "leapfrog"
    scale = 4.0 / (h * o) ** 2 / MU0 / EPS0 * (dt * dt / (8.0 / o ** 3) if leap else 1.0)
    K = torch.from_numpy(_kmat(o) * scale).to(dev)
    flat = lambda d, q: int(base[d] + q[0] + shape[d][2] * (q[1] + shape[d][1] * q[2]))  # noqa: E731
    src = torch.tensor([flat(d, q) for d, q in srcs], device=dev)

    def force(u):
        return torch.zeros_like(u).index_add_(0, dof.reshape(-1), (K @ u[dof]).reshape(-1))

    def wave(t):
        zeta, dl = 2.0 * math.pi ** 2 * 1e18, t - 1e-9
        return 2.0 * zeta * (2.0 * zeta * dl * dl - 1.0) * math.exp(-zeta * dl * dl) * 0.001

    gx, gy = n[0], n[1]
    ri = []
    for q in recs:
        x, y = flat(0, q), flat(1, q)
        px, py = gx * (gy + 1), (gx + 1) * gy
        ri.append([[x - 1, x, x + px - 1, x + px], [y - (gx + 1), y, y + py - (gx + 1), y + py], [flat(2, q)] * 4])
    ri = torch.tensor(ri, device=dev)
    tr = torch.zeros((len(recs), c["steps"], 3), dtype=f8, device=dev)
    lev = [torch.zeros(int(base[3]), dtype=f8, device=dev) for _ in range(3)]
    m = 8.0 / o ** 3
    t = 0.0
    for step in range(c["steps"]):
        if leap:
            e0, e1, e2 = (lev[(step + q) % 3] for q in range(3))
            tr[:, step] = e1[ri].mean(-1)
            e2.copy_(2 * e1 - e0 - force(e1) * live)
            e2.index_add_(0, src, torch.full((3,), -wave(t) * dt * dt / EPS0 / h ** 3, dtype=f8, device=dev))
            e2.mul_(live)
        else:
            U, P, F = lev
            tr[:, step] = U[ri].mean(-1)
            off = 0.0
            for a in SUB[c["integ"]]:
                a = a * dt
                U.add_(P, alpha=0.5 * a / m)
                F.copy_(force(U))
                F.index_add_(0, src, torch.full((3,), wave(t + off + 0.5 * a) * 8.0 / EPS0 / (h * o) ** 3, dtype=f8, device=dev))
                F.mul_(live)
                P.sub_(F, alpha=a)
                U.add_(P, alpha=0.5 * a / m)
                U.mul_(live)
                P.mul_(live)
                off += a
        t += dt
    # each component's three levels behind one another
    return {"traces": tr.cpu().numpy(), "fields": [torch.cat([v[base[d]:base[d + 1]] for v in lev]).cpu().numpy() for d in range(3)]}


# Kuhn tetrahedra: vertices c, +e_a, +e_b, +e_c for the six permutations (a, b, c)
_PERM = [(0, 1, 2), (0, 2, 1), (1, 0, 2), (1, 2, 0), (2, 0, 1), (2, 1, 0)]
_LOC = [(0, 1), (0, 2), (0, 3), (1, 2), (1, 3), (2, 3)]
_FACE = [(0, 1, 2), (0, 1, 3), (0, 2, 3), (1, 2, 3)]
_DIR = [(1, 0, 0), (0, 1, 0), (0, 0, 1), (1, 1, 0), (1, 0, 1), (0, 1, 1), (1, 1, 1)]


def _shape(p):
    a, b, c = _PERM[p]
    g, v = np.zeros((4, 3)), np.zeros((4, 3), int)
    g[0, a], g[1, a], g[1, b], g[2, b], g[2, c], g[3, c] = -1, 1, -1, 1, -1, 1
    v[1, a] = v[2, a] = v[2, b] = 1
    v[3] = 1
    return g, v


def _find(cells, x):
    """Cell, type and barycentric coordinates of a point."""
    cell = np.clip(np.floor(x).astype(int), 0, np.array(cells) - 1)
    s = x - cell
    ax = tuple(int(v) for v in np.argsort(-s, kind="stable"))
    lam = np.array([1 - s[ax[0]], s[ax[0]] - s[ax[1]], s[ax[1]] - s[ax[2]], s[ax[2]]])
    return cell, _PERM.index(ax), lam


class _Mesh:
    def __init__(self, cells):
        self.cells, self.dev = cells, _dev()
        self.n1 = [v + 1 for v in cells]
        self.nnode = int(np.prod(self.n1))
        self.ncube = int(np.prod(cells))
        k, j, i = np.meshgrid(*[np.arange(v) for v in cells[::-1]], indexing="ij")
        self.v0 = (i + self.n1[0] * (j + self.n1[1] * k)).reshape(-1)
        k, j, i = np.meshgrid(*[np.arange(v) for v in self.n1[::-1]], indexing="ij")
        self.pos = [i.reshape(-1), j.reshape(-1), k.reshape(-1)]

    def node(self, v):
        return int(v[0] + self.n1[0] * (v[1] + self.n1[1] * v[2]))

    def dead(self, axes):
        """Entities leaving the grid, or in a boundary face, by their lowest node."""
        bad = np.zeros(self.nnode, bool)
        for q in range(3):
            bad |= (self.pos[q] + axes[q] > self.cells[q]) if axes[q] else ((self.pos[q] == 0) | (self.pos[q] == self.cells[q]))
        return bad

    def add(self, out, vals):
        return out.index_add_(0, self.dof.reshape(-1), vals.reshape(-1))


class _Tet1(_Mesh):
    """Whitney elements with the mass lumped into one block per node."""

    def __init__(self, cells, eps, sig, dt):
        super().__init__(cells)
        dev, nn = self.dev, self.nnode
        eps6 = torch.from_numpy(eps).to(dev).reshape(self.ncube, 6).T
        dof = np.zeros((6, 6, self.ncube), np.int64)
        curl, wint, wsq = np.zeros((6, 6, 3)), np.zeros((6, 6, 3)), np.zeros((6, 6))
        for p in range(6):
            g, v = _shape(p)
            for e, (a, b) in enumerate(_LOC):
                dof[p, e] = 7 * (self.v0 + self.node(v[a])) + _DIR.index(tuple(v[b] - v[a]))
                curl[p, e] = 2 * np.cross(g[a], g[b])
                wint[p, e] = (g[b] - g[a]) / 24.0
                wsq[p, e] = (g[b] @ g[b] - g[a] @ g[b] + g[a] @ g[a]) / 60.0
        self.dof = torch.from_numpy(dof).to(dev)
        self.curl = torch.from_numpy(curl).to(dev)
        dead = np.stack([self.dead(d) for d in _DIR], 1)
        self.live = torch.from_numpy((~dead).reshape(-1).astype(float)).to(dev)
        lv = self.live.reshape(nn, 7)
        D = torch.tensor(_DIR, dtype=torch.float64, device=dev)[None] * lv[..., None]
        W = torch.stack([self.add(torch.zeros(7 * nn, dtype=torch.float64, device=dev),
                                  torch.from_numpy(wint[:, :, q]).to(dev)[:, :, None] * eps6[:, None, :]) for q in range(3)], 1)
        W = W.reshape(nn, 7, 3) * lv[..., None]
        w2 = torch.from_numpy(wsq).to(dev)[:, :, None]
        den = (self.add(torch.zeros(7 * nn, dtype=torch.float64, device=dev), w2 * eps6[:, None, :]).reshape(nn, 7) * lv).sum(1)
        alpha = den / lv.sum(1).clamp(min=1)

        def pinv(S):
            w, V = (torch.cat(x) for x in zip(*[torch.linalg.eigh(part) for part in S.split(16384)]))
            ok = w > 1e-10 * w.abs().amax(1, keepdim=True)
            return (V * torch.where(ok, 1.0 / torch.where(ok, w, torch.ones_like(w)), torch.zeros_like(w))[:, None, :]) @ V.mT

        S = D.mT @ W
        M = W @ pinv(0.5 * (S + S.mT)) @ W.mT
        M = M + alpha[:, None, None] * (torch.diag_embed(lv) - D @ pinv(D.mT @ D) @ D.mT) + torch.diag_embed(1.0 - lv)
        self.minv = torch.linalg.inv(M) * lv[:, :, None] * lv[:, None, :]
        self.size = 7 * nn
        self.loss = None
        if sig is not None:
            s6 = torch.from_numpy(sig * TS / EPS0).to(dev).reshape(self.ncube, 6).T
            num = (self.add(torch.zeros(7 * nn, dtype=torch.float64, device=dev), w2 * s6[:, None, :]).reshape(nn, 7) * lv).sum(1)
            self.loss = torch.where(den > 0, num / den.clamp(min=1e-300), torch.zeros_like(den)).repeat_interleave(7)

    def K(self, u):
        c = torch.einsum("pen,pec->pnc", u[self.dof], self.curl) / 6.0
        return self.add(torch.zeros_like(u), torch.einsum("pnc,pec->pen", c, self.curl)) * self.live

    def solve(self, b):
        return torch.bmm(self.minv, b.reshape(self.nnode, 7, 1)).reshape(-1)

    def at(self, x):
        cell, p, lam = _find(self.cells, x)
        g, v = _shape(p)
        w = np.array([lam[a] * g[b] - lam[b] * g[a] for a, b in _LOC])
        d = [7 * self.node(cell + v[a]) + _DIR.index(tuple(v[b] - v[a])) for a, b in _LOC]
        return torch.tensor(d, device=self.dev), torch.from_numpy(w).to(self.dev)


class _Tet2(_Mesh):
    """Complete second-order Nedelec elements; the consistent mass inverted by
    the degree-28 Chebyshev polynomial of its block-preconditioned form."""
    ENT = [d for d in _DIR] + [tuple((s1 | s2) >> q & 1 for q in range(3)) for s1 in range(1, 8) for s2 in range(1, 8) if not s1 & s2]
    FACES = [(s1, s2) for s1 in range(1, 8) for s2 in range(1, 8) if not s1 & s2]
    loss = None

    @staticmethod
    def funs():
        """Function a as (coefficients of the linear factor, i, j) of w_ij."""
        out = []
        for side in (0, 1):
            for e in _LOC:
                co = np.full(4, -0.625)
                co[list(e)] = 0.0
                co[e[side]] = 1.0
                out.append((co, *e))
        for i, j, k in _FACE:
            out += [(np.eye(4)[k], i, j), (np.eye(4)[i], j, k)]
        return out

    @classmethod
    def values(cls, p, lam):
        g, _ = _shape(p)
        return np.array([(co @ lam) * (lam[i] * g[j] - lam[j] * g[i]) for co, i, j in cls.funs()])

    @classmethod
    def matrices(cls, p):
        g, _ = _shape(p)
        M = np.zeros((20, 20))
        x, w = np.polynomial.legendre.leggauss(5)
        x, w = 0.5 * (x + 1), 0.5 * w
        for a in range(5):
            for b in range(5):
                for c in range(5):
                    X, Y = x[a], x[b] * (1 - x[a])
                    Z = x[c] * (1 - x[a]) * (1 - x[b])
                    v = cls.values(p, np.array([1 - X - Y - Z, X, Y, Z]))
                    M += w[a] * w[b] * w[c] * (1 - x[a]) ** 2 * (1 - x[b]) * (v @ v.T)
        C = np.zeros((20, 4, 3))
        for f, (co, i, j) in enumerate(cls.funs()):
            G = co @ g   # the gradient of the linear factor
            for v in range(4):
                C[f, v] = 2 * co[v] * np.cross(g[i], g[j]) + (v == i) * np.cross(G, g[j]) - (v == j) * np.cross(G, g[i])
        P1 = (np.ones((4, 4)) + np.eye(4)) / 120.0
        return M, np.einsum("avq,vw,bwq->ab", C, P1, C)

    def __init__(self, cells, eps, sig, dt):
        super().__init__(cells)
        dev, nn = self.dev, self.nnode
        self.size = 38 * nn
        self.eps6 = torch.from_numpy(eps).to(dev).reshape(self.ncube, 6).T
        self.map = [self.places(p) for p in range(6)]
        dof = np.zeros((6, 20, self.ncube), np.int64)
        Ms, Ks = [], []
        for p in range(6):
            for a, (plane, v) in enumerate(self.map[p]):
                dof[p, a] = plane * nn + self.v0 + self.node(v)
            M, K = self.matrices(p)
            Ms.append(M)
            Ks.append(K)
        self.dof = torch.from_numpy(dof).to(dev)
        self.Me, self.Ke = torch.from_numpy(np.stack(Ms)).to(dev), torch.from_numpy(np.stack(Ks)).to(dev)
        dead = np.zeros((38, nn), bool)
        for e, ax in enumerate(self.ENT):
            for pl in ((e, e + 7) if e < 7 else (14 + 2 * (e - 7), 15 + 2 * (e - 7))):
                dead[pl] = self.dead(ax)
        self.live = torch.from_numpy((~dead).reshape(-1).astype(float)).to(dev)
        # 2 x 2 blocks of an edge or face, and the bounds of the preconditioned element masses
        pair = [(l, l + 6) for l in range(6)] + [(12 + 2 * f, 13 + 2 * f) for f in range(4)]
        mate = np.zeros(20, int)
        for a, b in pair:
            mate[a], mate[b] = b, a
        lo, hi = [], []
        for M in Ms:
            R = np.zeros((20, 20))
            for a, b in pair:
                R[np.ix_((a, b), (a, b))] = np.linalg.inv(np.linalg.cholesky(M[np.ix_((a, b), (a, b))]))
            w = np.linalg.eigvalsh(R @ M @ R.T)
            lo.append(w[0])
            hi.append(w[-1])
        self.lo, self.hi = min(lo), max(hi)
        z = lambda: torch.zeros(self.size, dtype=torch.float64, device=dev)  # noqa: E731
        ar = torch.arange(20, device=dev)
        mt = torch.from_numpy(mate).to(dev)
        self.mdiag = self.add(z(), self.Me[:, ar, ar][:, :, None] * self.eps6[:, None, :])
        self.moff = self.add(z(), self.Me[:, ar, mt][:, :, None] * self.eps6[:, None, :])
        other = np.concatenate([np.arange(7, 14), np.arange(0, 7), np.arange(14, 38) ^ 1])
        self.other = torch.from_numpy((other[:, None] * nn + np.arange(nn)[None]).reshape(-1)).to(dev)
        det = self.mdiag * self.mdiag[self.other] - self.moff ** 2
        ok = (self.live > 0) & (det > 0)
        det = torch.where(ok, det, torch.ones_like(det))
        self.p0 = torch.where(ok, self.mdiag[self.other] / det, torch.zeros_like(det))
        self.p1 = torch.where(ok, -self.moff / det, torch.zeros_like(det))

    def places(self, p):
        _, v = _shape(p)
        out = []
        for a in range(20):
            if a < 12:
                i, j = _LOC[a % 6]
                out.append((_DIR.index(tuple(v[j] - v[i])) + 7 * (a >= 6), v[i]))
            else:
                i, j, k = _FACE[(a - 12) // 2]
                s = tuple(int(((v[y] - v[x]) * (1, 2, 4)).sum()) for x, y in ((i, j), (j, k)))
                out.append((14 + 2 * self.FACES.index(s) + (a - 12) % 2, v[i]))
        return out

    def elem(self, A, u, e=None):
        y = torch.bmm(A, u[self.dof])
        return y if e is None else y * e[:, None, :]

    def K(self, u):
        return self.add(torch.zeros_like(u), self.elem(self.Ke, u)) * self.live

    def M(self, u):
        return self.add(torch.zeros_like(u), self.elem(self.Me, u, self.eps6)) * self.live

    def pre(self, r):
        return self.p0 * r + self.p1 * r[self.other]

    def solve(self, b):
        b = b * self.live
        th, de = 0.5 * (self.hi + self.lo), 0.5 * (self.hi - self.lo)
        sg = th / de
        rho = 1.0 / sg
        d = self.pre(b) / th
        x = d.clone()
        for _ in range(27):
            rn = 1.0 / (2.0 * sg - rho)
            d = rn * rho * d + 2.0 * rn / de * self.pre(b - self.M(x))
            x = x + d
            rho = rn
        return x

    def at(self, x):
        cell, p, lam = _find(self.cells, x)
        d = [pl * self.nnode + self.node(cell + v) for pl, v in self.map[p]]
        return torch.tensor(d, device=self.dev), torch.from_numpy(self.values(p, lam)).to(self.dev)

    def api(self, u):
        return u.reshape(38, self.nnode).T.reshape(-1)


def _exact_tet(c, seed, kind):
    cells, eps, sig, src, rec, dt, f0, obs = _tet_inputs(c, seed)
    if kind is _Tet2 and sum(int(np.prod(s)) for s in cells) * c["steps"] * (3 if c["grad"] else 1) > 3e6:
        return None   # over 20 seconds
    traces, fields, J, grads = [], [], 0.0, []
    for k, s in enumerate(cells):
        m = kind(s, eps[k], sig[k] if sig else None, dt)
        sd, sw = m.at(src[k])
        sw = sw @ torch.tensor([0.0, 0.6, 0.8], dtype=torch.float64, device=m.dev)
        sw = sw * m.live[sd]
        rd, rw = zip(*[m.at(q) for q in rec[k]])
        rd, rw = torch.stack(rd), torch.stack(rw)
        sub = SUB.get(c["integ"])

        def wave(t):
            tau = t - math.sqrt(2.0) / f0
            return (1 - 2 * math.pi ** 2 * f0 ** 2 * tau ** 2) * math.exp(-math.pi ** 2 * f0 ** 2 * tau ** 2)

        U = torch.zeros(m.size, dtype=torch.float64, device=m.dev)
        P = torch.zeros_like(U)
        tr = torch.zeros((len(rec[k]), c["steps"], 3), dtype=torch.float64, device=m.dev)
        keep = []
        if sub:
            damp = torch.exp(-0.5 * dt * m.loss) if m.loss is not None else None
            Y = m.solve(P)
        elif m.loss is not None:
            r = 0.5 * dt * m.loss
        t = 0.0
        for n in range(c["steps"]):
            tr[:, n] = torch.einsum("ra,raq->rq", U[rd], rw)
            if sub is None:
                F = m.K(U).index_add_(0, sd, -sw * wave(t))
                Z = dt * dt * m.solve(F)
                U, P = (2 * U - P - Z, U) if m.loss is None else ((2 * U - (1 - r) * P - Z) / (1 + r), U)
            else:
                off = 0.0
                for q, a in enumerate(sub):
                    a *= dt
                    U = U + 0.5 * a * Y
                    F = m.K(U).index_add_(0, sd, -sw * wave(t + off + 0.5 * a))
                    if damp is not None and q == len(sub) // 2:
                        P = damp * (damp * P - a * F)
                    else:
                        P = P - a * F
                    if c["grad"] and kind is _Tet2:
                        keep += [Y, m.solve(P)]
                        Y = keep[-1]
                    else:
                        Y = m.solve(P)
                    U = U + 0.5 * a * Y
                    off += a
            t += dt
        traces.append(tr.cpu().numpy())
        fields.append((m.api(U) if kind is _Tet2 else U).cpu().numpy())
        if not c["grad"]:
            continue
        # the steps reversed: drift and kick transposed, dM/deps in every drift
        res = tr - torch.from_numpy(obs[k * c["nrec"]:(k + 1) * c["nrec"], :, 1:]).to(m.dev)
        J += 0.5 * float((res ** 2).sum())
        if kind is _Tet1:   # no closed form here for the derivative of its blocks
            continue
        Ub, Pb = torch.zeros_like(U), torch.zeros_like(U)
        g = torch.zeros_like(m.eps6)
        for n in range(c["steps"] - 1, -1, -1):
            for q in range(len(sub) - 1, -1, -1):
                a = sub[q] * dt
                for half in (1, 0):
                    Z = m.solve(Ub)
                    Pb = Pb + 0.5 * a * Z
                    yk = keep[2 * (n * len(sub) + q) + half]
                    g -= 0.5 * a * (Z[m.dof] * m.elem(m.Me, yk)).sum(1)
                    if half:
                        Ub = Ub - a * m.K(Pb)
            Ub.index_add_(0, rd.reshape(-1), torch.einsum("rq,raq->ra", res[:, n], rw).reshape(-1))
            Ub = Ub * m.live
        grads.append(g.T.reshape(-1).cpu().numpy())
    out = {"traces": np.concatenate(traces)}
    if c["grad"]:
        return {**out, "misfit": J, "grad": [np.concatenate(grads) if grads else None]}
    return {**out, "fields": [np.concatenate(fields)]}
