"""Workloads of the SPH + FMM planetary-impact step, from single passes to whole
steps, as a program that uses the library calls them.

A case names what is called (`call`) and on what:

  cells     sph_sort_cells_noalloc: the cell sort on a caller's own positions
  sort      Compute.sort(): cell hash, radix sort and cell ranges
  gravity   Compute.updateOctreeBuffer() + gravitationalPass()
  density   Compute.densityPass()
  accel     Compute.accelerationPass()
  step      Compute.step_all(): whole steps with the state on the device
  host      Compute.step_host(): a whole step with the state in pinned memory
  ensemble  Ensemble.step(): several impacts advanced together

The particles are the seeded two-body impacts, Plummer spheres and cubes of the
package's `ic` module.  An impact also gets what a running simulation has by
then: velocity gradients inside the bodies, energies that are not uniform, and
the gravity field of the previous step (the reference form's acceptance test
reads it).  All of it comes from the seed alone, not from earlier passes of the
code, so every version of the library starts from the same bits.

A pass first puts back what it changes (the smoothing lengths before a density
pass, the state before a step) by device copies into the library's own buffers,
so that each pass does the same work.
"""
import ctypes
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("real-time-planetary-impacts-mps_b200")

G = 6.67e-5
SOFTENING = 0.04
CELL = np.float32(0.18)
ETA_RES = 1.2348       # h = ETA_RES (m / rho)^(1/3) at the fixed point
ETA_TOL = 0.005        # relative change at which the h iteration stops
H_MAX = 1.0
TICK = 32.0 / 65536.0  # seconds
EXACT_MOST = 65536     # particles up to which exact() sums over all pairs


# ---- what is measured --------------------------------------------------------

def listed():
    return [
        # the smallest call: the tests' 16384 + 4096 particles, sorted on
        # positions that the caller owns, without an allocation
        dict(name="cells_20k", call="cells", bodies="impact", n=20480),
        # the cell sort of a production-size impact, an odd particle count
        dict(name="sort_1m", call="sort", bodies="impact", n=1000003),
        # the reference's gravity at the size of its published frame rate and
        # its own leaf capacity
        dict(name="gravity_ref_100k_leaf4", call="gravity", bodies="impact", n=100003, leaf=4, gravity="reference"),
        # the reference's gravity at the benchmark's size and leaf capacity
        dict(name="gravity_ref_1m", call="gravity", bodies="impact", n=1000000, leaf=32, gravity="reference"),
        # the opening-angle form on the gravity-only check's Plummer sphere,
        # whose far outliers need the deepest tree
        dict(name="gravity_theta_plummer_1m", call="gravity", bodies="plummer", n=1 << 20, leaf=32, depth=10,
             gravity="theta", theta=0.5),
        # a small impact, whose h spans several cells: the coarse tiles take it all
        dict(name="density_20k", call="density", bodies="impact", n=20480),
        # the largest pass of a production step
        dict(name="density_1m", call="density", bodies="impact", n=1000000),
        # its second largest, at the reference's precision
        dict(name="accel_1m", call="accel", bodies="impact", n=1000000, precision="reference"),
        # real time: the reference's demo size at its defaults, two steps a frame
        dict(name="step_demo_11k", call="step", bodies="impact", n=10766, leaf=4, gravity="reference",
             precision="reference", steps=2),
        # real time at the size of the reference's published frame rate
        dict(name="step_100k", call="step", bodies="impact", n=100000, leaf=32, gravity="theta", theta=0.6,
             precision="mixed", steps=2),
        # the benchmark's end-to-end step: opening-angle gravity, FP64
        # positions, learned smoothing-length seed refreshed every step
        dict(name="host_learned_1m", call="host", bodies="impact", n=1000000, leaf=32, gravity="theta", theta=0.6,
             precision="mixed", learned=True),
        # a batch of small impacts of uneven size
        dict(name="ensemble_4", call="ensemble", bodies="impact", n=30011, n2=100003, members=4, leaf=32,
             gravity="theta", theta=0.6, precision="mixed"),
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n | 1 if rng.random() < 0.5 else n

    call = rng.choice(["cells", "sort", "gravity", "gravity", "density", "density", "accel", "accel", "step", "step",
                       "host", "ensemble"])
    c = dict(call=call, bodies="impact")
    leaf = rng.choice([4, 16, 32])
    if call == "cells":
        c.update(n=size(1e4, 262144))
    elif call in ("sort", "density"):
        c.update(n=size(1e4, 1e6))
    elif call == "gravity":
        c["gravity"] = rng.choice(["reference", "theta"])
        if c["gravity"] == "theta":
            c["bodies"] = rng.choice(["impact", "plummer", "cube"])
            c["theta"] = rng.choice([0.5, 0.6, 0.7])
            if c["bodies"] == "plummer":
                c["depth"] = 10
        c.update(n=size(1e4, 2e5 if leaf == 4 else 1e6), leaf=leaf)
    elif call == "accel":
        c.update(n=size(1e4, 1e6), precision=rng.choice(["reference", "mixed"]))
    elif call in ("step", "host"):
        c.update(n=size(1e4, 2e5 if leaf == 4 else 8e5), leaf=leaf, gravity=rng.choice(["reference", "theta"]),
                 precision=rng.choice(["reference", "mixed"]))
        if c["gravity"] == "theta":
            c["theta"] = rng.choice([0.5, 0.6])
        if call == "step":
            c["steps"] = 1
        else:
            c["learned"] = c["gravity"] == "theta" and c["precision"] == "mixed"
    else:
        c.update(n=size(2e4, 6e4), n2=size(6e4, 1.2e5), members=rng.choice([2, 3, 4]), leaf=32,
                 gravity="theta", theta=0.6, precision="mixed")
    return c


def _sizes(case):
    """Particle counts of an ensemble's members, geometrically between n and n2."""
    k = case["members"]
    return [int(round(case["n"] * (case["n2"] / case["n"]) ** (i / max(k - 1, 1)))) for i in range(k)]


# ---- inputs ------------------------------------------------------------------

def _initial(bodies, n, seed):
    """Initial conditions in the layout Compute takes, plus "grav": the field
    acceleration per unit G of each particle (n, 3), from the enclosed masses."""
    if bodies == "plummer":
        ic = pkg.ic.make_plummer(n, seed=seed)
        split = n
    elif bodies == "cube":
        ic = pkg.ic.make_cube(n, seed=seed)
        split = n
    else:
        split = n - n // 5
        ic = pkg.ic.make_impact(split, n - split, seed=seed)
        for body in (slice(0, split), slice(split, n)):
            _settle(ic, body, seed)
        _flow(ic, split, seed)
    pos = ic["pos"].astype(np.float64)
    m = ic["mass"].astype(np.float64)
    g = np.zeros_like(pos)
    parts = [slice(0, split)] + ([slice(split, n)] if split < n else [])
    for p in parts:
        c = np.average(pos[p], axis=0, weights=m[p])
        d = pos[p] - c
        r = np.sqrt((d * d).sum(axis=1))
        order = np.argsort(r, kind="stable")
        inside = np.empty_like(r)
        inside[order] = np.cumsum(m[p][order])
        g[p] -= (inside / np.maximum(r, 0.1) ** 3)[:, None] * d
        for q in parts:
            if q != p:  # the other body as a point mass
                e = pos[q] - c
                g[q] -= (m[p].sum() / ((e * e).sum(axis=1) + 1.0) ** 1.5)[:, None] * e
    ic["grav"] = g
    return ic


def _settle(ic, body, seed):
    """Densities and smoothing lengths of a body as its first steps leave them:
    the layers' densities smoothed over the kernel, so lower at the surface and
    between at the core's edge (the surfaces taken as planes), and h = ETA_RES
    (m / rho)^(1/3) up to what a step's motion leaves for the iteration to find:
    a smooth change of up to 7 % and one of up to 2 % from particle to particle,
    for which it takes three to four sweeps, as in a running simulation."""
    z = np.linspace(-2.0, 2.0, 401)
    # the part of the cubic spline's weight below the plane at offset z
    q = np.abs(z)
    plane = np.where(q > 1, (2 - q) ** 4 * (1 + 2 * q) / 40, 0.35 - q * q * (0.5 - q * q * (0.375 - 0.15 * q)))
    below = np.concatenate([[0.0], np.cumsum(0.5 * (plane[1:] + plane[:-1]))])
    below /= below[-1]
    x = ic["pos"][body].astype(np.float64)
    r = np.sqrt(((x - x.mean(axis=0)) ** 2).sum(axis=1))
    m = ic["mass"][body].astype(np.float64)
    core = ic["material"][body] == pkg.ic.MAT_FE85SI15
    r_core = (3.0 * m[core].sum() / (4.0 * math.pi * pkg.ic.RHO_CORE)) ** (1 / 3)
    r_out = (r_core ** 3 + 3.0 * m[~core].sum() / (4.0 * math.pi * pkg.ic.RHO_MANTLE)) ** (1 / 3)
    h = ic["h"][body].astype(np.float64)
    for _ in range(12):
        f_out = np.interp((r_out - r) / h, z, below)
        f_core = np.interp((r_core - r) / h, z, below)
        rho = pkg.ic.RHO_MANTLE * np.maximum(f_out, 0.05) + (pkg.ic.RHO_CORE - pkg.ic.RHO_MANTLE) * f_core
        h = 0.5 * h + 0.5 * np.minimum(ETA_RES * (m / rho) ** (1 / 3), 0.99 * H_MAX)
    rng = np.random.default_rng(seed + 104729 + body.start)
    k = rng.normal(size=3)
    k *= 1.2 / np.linalg.norm(k)
    h *= 1.0 + 0.07 * np.sin(x @ k + rng.uniform(0.0, 2.0 * math.pi)) + rng.uniform(-0.02, 0.02, size=h.size)
    ic["rho"][body], ic["h"][body] = rho, np.minimum(h, 0.99 * H_MAX)


def _flow(ic, split, seed):
    """A smooth velocity field (three modes of the body's size, about a tenth
    of the escape speed) and a smooth change of the energies on top of the two
    bodies' uniform ones, as a simulation has them once the bodies feel each
    other: without them every viscosity and divergence term is zero."""
    rng = np.random.default_rng(seed + 7919)
    pos = ic["pos"].astype(np.float64)
    vel = ic["vel"].astype(np.float64)
    x = pos - pos[:split].mean(axis=0)
    for _ in range(3):
        k = rng.normal(size=3)
        k *= rng.uniform(0.3, 0.9) / np.linalg.norm(k)
        amp = rng.normal(size=3) * 4e-4
        vel += np.sin(x @ k + rng.uniform(0.0, 2.0 * math.pi))[:, None] * amp
    k = rng.normal(size=3)
    k *= 0.5 / np.linalg.norm(k)
    ic["u"] = (ic["u"] * (1.0 + 0.1 * np.sin(x @ k))).astype(np.float32)
    ic["vel"] = np.ascontiguousarray(vel, dtype=np.float32)


class _Borrowed:
    """One of the library's device buffers, for torch.as_tensor; the tensor
    keeps `owner`, whose end would free the buffer."""

    def __init__(self, owner, ptr, shape, strides, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(shape=shape, strides=strides, typestr=typestr, data=(ptr, False),
                                             version=3)


_INT = ("material", "next_active_time", "global_time", "dt", "cell_key", "cell_index")


def _view(c, field, owner=None):
    """A field's device buffer as a tensor (no copy).  `owner`: what the buffer
    belongs to, where that is not `c` (an ensemble's instances are its own)."""
    owner = owner or c
    ptr, size, stride = c.device_buffer(field)
    if field in ("pos", "vel", "acc"):
        return torch.as_tensor(_Borrowed(owner, ptr, (c.nParticles, 3), (stride, 4), "<f4"), device="cuda")
    if field == "pos64":
        return torch.as_tensor(_Borrowed(owner, ptr, (c.nParticles, 3), (stride, 8), "<f8"), device="cuda")
    kind = "<i4" if field in _INT else "<f4"
    return torch.as_tensor(_Borrowed(owner, ptr, (size // stride,), None, kind), device="cuda")


def _form(case):
    return dict(gravity=case.get("gravity", "reference"), theta=case.get("theta", 0.5),
                precision=case.get("precision", "reference"))


def _compute(case, ic):
    c = pkg.Compute(ic, max_children_in_leaf=case.get("leaf", 32), max_tree_depth=case.get("depth", 7))
    c.set_form(**_form(case))
    c.upload("grav_norm", np.sqrt((ic["grav"] ** 2).sum(axis=1)))
    c.upload("acc", G * ic["grav"])
    return c


def _keep(c, fields, owner=None):
    """(buffer, copy of its present contents) of each field."""
    return [(v, v.clone()) for v in (_view(c, f, owner) for f in fields)]


def _state_fields(case):
    mixed = case.get("precision") == "mixed"
    return (["pos64"] if mixed else []) + ["pos", "vel", "u", "h", "rho"]


def prepare(case, seed):
    call, n = case["call"], case["n"]
    st = dict(call=call, restore=[], out={})
    if call == "cells":
        ic = _initial(case["bodies"], n, seed)
        st["lib"] = pkg._lib.load()
        st["n"] = n
        st["pos"] = torch.from_numpy(ic["pos"]).cuda()
        st["out"] = {k: torch.empty(n, dtype=torch.int32, device="cuda") for k in ("cell_key", "cell_index")}
        return st
    if call == "ensemble":
        ics = [_initial(case["bodies"], k, seed + 31 * i) for i, k in enumerate(_sizes(case))]
        e = pkg.Ensemble(ics, [_form(case)] * len(ics), max_children_in_leaf=case["leaf"])
        st["e"] = e
        fields = _state_fields(case)
        outs = []
        for c, ic in zip(e.instances, ics):
            c.upload("acc", G * ic["grav"])
            st["restore"] += _keep(c, fields, e)
            outs.append({f: _view(c, f, e) for f in fields if f != "pos" or "pos64" not in fields})
        st["out"] = outs
        return st
    ic = _initial(case["bodies"], n, seed)
    c = _compute(case, ic)
    st["c"] = c
    if call == "sort":
        st["out"] = {f: _view(c, f) for f in ("cell_key", "cell_index")}
    elif call == "gravity":
        fields = ["acc", "grav_norm"] + (["potential"] if case["gravity"] == "theta" else [])
        st["restore"] = _keep(c, ["grav_norm"]) if case["gravity"] == "reference" else []
        st["out"] = {f: _view(c, f) for f in fields}
    elif call == "density":
        c.sort()
        st["restore"] = _keep(c, ["h"])
        st["out"] = {f: _view(c, f) for f in ("h", "rho", "pressure", "grad_term", "sound_speed", "balsara")}
    elif call == "accel":
        c.sort()
        c.densityPass()
        st["restore"] = _keep(c, ["acc"])
        st["out"] = {f: _view(c, f) for f in ("acc", "du", "dhdt", "next_active_time", "dt")}
    elif call == "step":
        fields = _state_fields(case)
        st["steps"] = case["steps"]
        st["restore"] = _keep(c, fields + (["grav_norm"] if case["gravity"] == "reference" else []))
        st["out"] = {f: _view(c, f) for f in fields if f != "pos" or "pos64" not in fields}
    else:
        if case.get("learned"):
            # the seed network is trained on the solver's own first passes
            c.sort()
            c.hseed_capture(True)
            c.densityPass()
            c.hseed_train(300)
            c.upload("h", ic["h"])
            c.set_form(h_seed="learned", **_form(case))
            c.hseed_online(4)
        pos = "pos64" if case["precision"] == "mixed" else "pos"
        st["in"], st["res"] = {}, {}
        for f, a in ((pos, ic["pos"]), ("vel", ic["vel"]), ("u", ic["u"]), ("h", ic["h"]), ("rho", ic["rho"])):
            t = torch.empty(a.shape, dtype=torch.float64 if f == "pos64" else torch.float32, pin_memory=True)
            t.copy_(torch.from_numpy(a))
            o = torch.zeros_like(t).pin_memory()
            st["out"][f] = o
            st["in"][f], st["res"][f] = t.numpy(), o.numpy()
        if case["gravity"] == "reference":
            st["restore"] = _keep(c, ["grav_norm"])
    return st


def run(st):
    for dst, src in st["restore"]:
        dst.copy_(src)
    call = st["call"]
    if call == "cells":
        o = st["out"]
        status = st["lib"].sph_sort_cells_noalloc(
            ctypes.c_void_p(st["pos"].data_ptr()), st["n"], ctypes.c_void_p(o["cell_key"].data_ptr()),
            ctypes.c_void_p(o["cell_index"].data_ptr()), ctypes.c_void_p(0))
        pkg._lib.check(status, "sph_sort_cells_noalloc")
    elif call == "sort":
        st["c"].sort()
    elif call == "gravity":
        st["c"].updateOctreeBuffer()
        st["c"].gravitationalPass()
    elif call == "density":
        st["c"].densityPass()
    elif call == "accel":
        st["c"].accelerationPass()
    elif call == "step":
        st["c"].step_all(st["steps"])
    elif call == "host":
        st["c"].step_host(st["in"], st["res"])
    else:
        st["e"].step(1)
    return st["out"]


# ---- what a pass cannot do without -------------------------------------------

# About 60 neighbours lie within 2 h.  Operations per particle: density, one
# sweep to confirm h (12 a pair) and the gradient sweep (45 a pair); the
# acceleration pass 70 a pair; gravity an expansion of order two evaluated at
# the particle plus its near neighbours, about 100 interactions of 40.
_FLOPS = dict(sort=20, gravity=4000, density=60 * 57, accel=60 * 70, step=40)
# Bytes per particle, every input read once and every output written once.
_BYTES = dict(cells=20, sort=32, gravity=36, density=57, accel=88, step=92)


def work(case):
    call = case["call"]
    n = sum(_sizes(case)) if call == "ensemble" else case["n"]
    if call in ("cells", "sort"):
        return {"bytes": n * _BYTES[call], "flops": n * _FLOPS["sort"]}
    if call in ("gravity", "density", "accel"):
        return {"bytes": n * _BYTES[call], "flops": n * _FLOPS[call]}
    steps = case.get("steps", 1)
    per = sum(_BYTES[k] for k in ("sort", "gravity", "density", "accel", "step"))
    if call == "host":
        per += 2 * 48  # the state in and out
    return {"bytes": n * steps * per, "flops": n * steps * sum(_FLOPS.values())}


# ---- tolerances --------------------------------------------------------------

def tolerance(case):
    """Four times what was seen between this library's build and one that sums
    in another order without fused multiply-adds, or where noted otherwise."""
    call = case["call"]
    if call in ("cells", "sort"):
        return "exact"
    # a particle on the h iteration's threshold may take one sweep more, which
    # moves its h by up to half a per cent: a few in a million do
    n = case["n"]
    flips = 0.02 / math.sqrt(n)
    if call == "gravity":
        if case["gravity"] == "reference":
            return {"rel": 2e-4, "max": 0.02}
        # what is accepted for a group of particles depends on the grouping:
        # four times the opening-angle form's own error against the direct sum
        return {"rel": {0.5: 3e-3, 0.6: 6e-3, 0.7: 1.2e-2}[case["theta"]], "max": 0.3}
    if call == "density":
        return {"rel": 4e-5 + flips, "max": 0.04}
    if call == "accel":
        return {"rel": 6e-5 + flips, "max": 0.03, "differ": 1e-4}
    if case.get("learned"):
        # trained with atomics, so the seeds are never twice the same; they
        # start an iteration that stops within half a per cent
        return {"rel": 5e-3, "max": 0.03}
    if case["gravity"] == "theta":
        return {"rel": 2.5e-4 + flips, "max": 0.02}
    return {"rel": 2e-5 + flips, "max": 0.02}


# ---- 64-bit results ----------------------------------------------------------

def _w(q):
    """Cubic spline times pi h^3."""
    return torch.where(q > 2, 0.0, torch.where(q > 1, 0.25 * (2 - q) ** 3, 1 - 1.5 * q * q * (1 - 0.5 * q)))


def _dw(q):
    """Its derivative in q (times pi h^4 as a gradient)."""
    return torch.where(q > 2, 0.0, torch.where(q > 1, -0.75 * (2 - q) ** 2, 3 * (0.75 * q - 1) * q))


def _dwdh(q):
    """-pi h^4 / 3 times the derivative in h, in the reference's polynomials."""
    far = 2 - 4 * q + 2.5 * q * q - 0.5 * q ** 3
    return torch.where(q > 2, 0.0, torch.where(q > 1, far, 1 + 0.5 * (3 * q - 5) * q * q))


def _chunks(n):
    rows = max(1, min(n, (1 << 26) // n))
    return [slice(a, min(a + rows, n)) for a in range(0, n, rows)]


def _tables():
    """The two EOS tables as (res, res, 2) grids of (P, c) in 64 bits: the text
    files resampled as the reference does it (its interpolation weights, lower
    and upper swapped, included)."""
    grids = []
    paths = pkg.eos_tables.ensure_tables()
    for name in ("forsterite", "Fe85Si15"):
        with open(paths[name]) as f:
            words = " ".join(f.read().split("\n")[13:]).split()
        nr, nt = int(words[0]), int(words[1])
        v = np.array(words[2:], dtype=np.float64)
        rho = v[:nr]
        t = v[nr + nt:nr + nt + 4 * nr * nt].reshape(nt, nr, 4).transpose(1, 0, 2)  # [rho][T]
        u, val = t[:, :, 0], t[:, :, 1:3] * np.array([1e-18, 1e-6])
        res = 2048
        gr = 1e6 ** (np.arange(res) / res)
        gu = 100.0 * 1e10 ** (np.arange(res) / res)
        lo = np.clip(np.searchsorted(rho, gr, side="left") - 1, 0, nr - 2)
        rl = ((gr - rho[lo]) / (rho[lo + 1] - rho[lo]))[:, None, None]

        def row(i):
            k = np.clip(np.searchsorted(u[i], gu, side="left") - 1, 0, nt - 2)
            w = ((gu - u[i][k]) / (u[i][k + 1] - u[i][k]))[:, None]
            return val[i][k] * w + val[i][k + 1] * (1 - w)

        rows = np.stack([row(i) for i in range(nr)])
        grids.append(torch.from_numpy(rl * rows[lo] + (1 - rl) * rows[lo + 1]).cuda())
    return grids


def _eos(mat, rho, u):
    out = torch.zeros(rho.shape[0], 2, dtype=torch.float64, device="cuda")
    for grid, sel in zip(_tables(), (mat == 400, mat != 400)):
        res = grid.shape[0]
        x = (torch.log(u[sel] / 1e-10) / math.log(1e10)).clamp(0, 1) * res - 0.5
        y = (torch.log(rho[sel] / 1e-6) / math.log(1e6)).clamp(0, 1) * res - 0.5
        fx, fy = (x - x.floor())[:, None], (y - y.floor())[:, None]
        x0, y0 = x.floor().long(), y.floor().long()
        x1, y1 = (x0 + 1).clamp(0, res - 1), (y0 + 1).clamp(0, res - 1)
        x0, y0 = x0.clamp(0, res - 1), y0.clamp(0, res - 1)
        out[sel] = (grid[y0, x0] * (1 - fx) + grid[y0, x1] * fx) * (1 - fy) + \
            (grid[y1, x0] * (1 - fx) + grid[y1, x1] * fx) * fy
    return out[:, 0], out[:, 1]


class _State64:
    def __init__(self, ic):
        f = lambda k: torch.from_numpy(np.asarray(ic[k])).cuda().double()  # noqa: E731
        self.x, self.v, self.m, self.u, self.h = f("pos"), f("vel"), f("mass"), f("u"), f("h")
        self.mat = torch.from_numpy(ic["material"]).cuda()
        self.n = self.x.shape[0]

    def gravity(self):
        """Direct sum with the cubic-spline softening: (acceleration, potential), per unit G."""
        acc, phi = torch.zeros_like(self.x), torch.zeros_like(self.m)
        for s in _chunks(self.n):
            d = [self.x[s, k, None] - self.x[None, :, k] for k in range(3)]
            r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
            q = r / SOFTENING
            q2 = q * q
            near = (4 / 3 * q - 1.2 * q2 * q + 0.5 * q2 * q2) / SOFTENING ** 2
            mid = (8 / 3 * q - 3 * q2 + 1.2 * q2 * q - q2 * q2 / 6 - 1 / (15 * q2)) / SOFTENING ** 2
            fr = torch.where(q >= 2, 1 / (r * r), torch.where(q > 1, mid, near))
            fr = torch.where(r > 0, self.m * fr / r, torch.zeros_like(r))
            near = (2 / 3 * q2 - 0.3 * q2 * q2 + 0.1 * q2 * q2 * q - 1.4) / SOFTENING
            mid = (4 / 3 * q2 - q2 * q + 0.3 * q2 * q2 - q2 * q2 * q / 30 - 1.6 + 1 / (15 * q)) / SOFTENING
            pot = torch.where(q >= 2, -1 / r, torch.where(q > 1, mid, near))
            phi[s] = torch.where(r > 0, self.m * pot, torch.zeros_like(r)).sum(dim=1)
            for k in range(3):
                acc[s, k] = -(fr * d[k]).sum(dim=1)
        return acc, phi

    def density(self):
        n = self.n
        self.rho, self.f, self.bal = (torch.zeros_like(self.m) for _ in range(3))
        div, curl = torch.zeros_like(self.m), torch.zeros_like(self.m)
        for s in _chunks(n):
            d = [self.x[None, :, k] - self.x[s, k, None] for k in range(3)]
            r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
            h = self.h[s].clone()
            live = torch.ones_like(h, dtype=torch.bool)
            rho = torch.zeros_like(h)
            for _ in range(50):
                at = live.nonzero()[:, 0]
                if not at.numel():
                    break
                hh = h[at]
                rho[at] = (self.m * _w(r[at] / hh[:, None])).sum(dim=1) / (math.pi * hh ** 3)
                new = 0.5 * (hh + torch.clamp(ETA_RES * (self.m[s][at] / rho[at]) ** (1 / 3), max=H_MAX))
                go = (new - hh).abs() / hh > ETA_TOL
                h[at] = torch.where(go, new, hh)
                live[at] = go
            q = r / h[:, None]
            many = (r <= 2 * h[:, None]).sum(dim=1) >= 128  # the reference sums these twice
            rho = rho + torch.where(many, (self.m * _w(q)).sum(dim=1) / (math.pi * h ** 3), torch.zeros_like(rho))
            dh = -3 / (math.pi * h ** 4) * (self.m * _dwdh(q)).sum(dim=1)
            g = torch.where(r > 1e-12, self.m * _dw(q) / (math.pi * h ** 4)[:, None] / r, torch.zeros_like(r))
            g = [g * d[k] for k in range(3)]
            v = [self.v[None, :, k] - self.v[s, k, None] for k in range(3)]
            div[s] = (v[0] * g[0] + v[1] * g[1] + v[2] * g[2]).sum(dim=1).abs() / rho
            c = [(v[1] * g[2] - v[2] * g[1]).sum(dim=1), (v[2] * g[0] - v[0] * g[2]).sum(dim=1),
                 (v[0] * g[1] - v[1] * g[0]).sum(dim=1)]
            curl[s] = torch.sqrt(c[0] ** 2 + c[1] ** 2 + c[2] ** 2) / rho
            self.h[s], self.rho[s] = h, rho
            self.f[s] = 1 / (1 + h / (3 * rho) * dh)
        self.P, self.c = _eos(self.mat, self.rho, self.u)
        self.bal = div / (div + curl + 1e-4 * self.c / self.h)

    def acceleration(self):
        """Pressure and viscosity terms: acceleration, du/dt, dh/dt, ticks."""
        n = self.n
        acc, du, dh, ticks = torch.zeros_like(self.x), torch.zeros_like(self.m), torch.zeros_like(self.m), None
        sig = torch.zeros_like(self.m)
        fact = self.f * self.P / self.rho ** 2
        x32 = self.x.float()
        cell = torch.floor(x32 / float(CELL))
        lo = torch.floor((x32 - (2 * self.h.clamp(max=H_MAX)).float()[:, None]) / float(CELL))
        hi = torch.floor((x32 + (2 * self.h.clamp(max=H_MAX)).float()[:, None]) / float(CELL))
        for s in _chunks(n):
            d = [self.x[s, k, None] - self.x[None, :, k] for k in range(3)]
            r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
            inside = torch.ones_like(r, dtype=torch.bool)
            for k in range(3):  # a pair is seen only inside the particle's own box of cells
                inside &= (cell[None, :, k] >= lo[s, k, None]) & (cell[None, :, k] <= hi[s, k, None])
            see = inside & (r > 1e-6) & (r <= 2 * torch.maximum(self.h[s, None], self.h[None, :]))
            at, j = see.nonzero(as_tuple=True)
            i = at + s.start
            r = r[at, j]
            rh = torch.stack([d[k][at, j] for k in range(3)], dim=1) / r[:, None]
            v = self.v[i] - self.v[j]
            si = _dw(r / self.h[i]) / (math.pi * self.h[i] ** 4)
            sj = _dw(r / self.h[j]) / (math.pi * self.h[j] ** 4)
            vr = (v * rh).sum(dim=1)
            mu = torch.where(vr < 0, vr, torch.zeros_like(vr))
            vs = self.c[i] + self.c[j] - 3 * mu
            nu = -0.5 * 1.5 * 0.5 * (self.bal[i] + self.bal[j]) * mu * vs / (0.5 * (self.rho[i] + self.rho[j]))
            mean = 0.5 * (si + sj)
            push = -self.m[j] * (fact[i] * si + fact[j] * sj + nu * mean)
            acc.index_add_(0, i, push[:, None] * rh)
            du.index_add_(0, i, self.m[j] * (fact[i] * si + 0.5 * nu * mean) * vr)
            dh.index_add_(0, i, self.m[j] / self.rho[j] * vr * si)
            sig.index_reduce_(0, i, vs, "amax")
        goal = 2 * 0.2 * 1.825742 * self.h / sig.clamp(min=1e-12)
        level = torch.ceil(torch.log2(32.0 / goal)).clamp(0, 16)
        ticks = (65536 * 0.5 ** level).int()
        return acc, du, dh, ticks

    def step(self):
        g, _ = self.gravity()
        self.density()
        a, du, dh, ticks = self.acceleration()
        a = a + G * g
        dt = TICK * int(ticks.min())
        self.x = self.x + dt * self.v + 0.5 * dt * dt * a
        self.v = self.v + dt * a
        self.u = self.u + dt * du
        rate = dh / self.h * dt
        self.h = (self.h * torch.exp(rate)).clamp(max=H_MAX)
        self.rho = self.rho * torch.exp(-3 * rate)


def exact(case, seed):
    call = case["call"]
    if call in ("cells", "sort"):
        return None  # whole numbers, compared as they are
    if call == "ensemble":
        got = [_exact_steps(_initial(case["bodies"], k, seed + 31 * i), case, 1) if k <= EXACT_MOST else None
               for i, k in enumerate(_sizes(case))]
        return got if any(g is not None for g in got) else None
    if case["n"] > EXACT_MOST:
        return None
    ic = _initial(case["bodies"], case["n"], seed)
    if call in ("step", "host"):
        return _exact_steps(ic, case, case.get("steps", 1))
    s = _State64(ic)
    if call == "gravity":
        g, phi = s.gravity()
        got = {"acc": G * g, "grav_norm": torch.sqrt((g * g).sum(dim=1))}
        if case["gravity"] == "theta":
            got["potential"] = G * phi
        return got
    s.density()
    if call == "density":
        return {"h": s.h, "rho": s.rho, "pressure": s.P, "grad_term": s.f, "sound_speed": s.c, "balsara": s.bal}
    a, du, dh, ticks = s.acceleration()
    acc = torch.from_numpy((G * ic["grav"]).astype(np.float32)).cuda().double()
    return {"acc": acc + a, "du": du, "dhdt": dh, "next_active_time": None, "dt": None}


def _exact_steps(ic, case, steps):
    s = _State64(ic)
    for _ in range(steps):
        s.step()
    pos = "pos64" if case["precision"] == "mixed" else "pos"
    return {pos: s.x, "vel": s.v, "u": s.u, "h": s.h, "rho": s.rho}
