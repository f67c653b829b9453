"""Performance cases of mesh_gb300: what a lattice-gauge user has the library
do, each one pass through the public Python entry points, and the same values
in plain FP64 torch (`exact`).

A case is a dict of plain values: "kind" (which entry points), "group" (u1,
su2, su3), "prec" (32 or 64), "dims" ("12x20x14x30") and the parameters of the
kind. The links look like a thermalised configuration at the usual couplings:
independent links around the identity with a plaquette of about 0.6, in a
Haar-random gauge; Markov chains with their own accept step start closer to
the cold configuration.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import mesh_gb300 as mesh

GPU = "cuda"
NC = {"u1": 1, "su2": 2, "su3": 3}
NREAL = {"u1": 2, "su2": 4, "su3": 18}
NALG = {"u1": 1, "su2": 3, "su3": 8}
TAG_MOMENTUM, TAG_METROPOLIS, TAG_HEATBATH = 1, 3, 5
FFT_EXTENTS = (4, 6, 8, 12, 16, 24, 32)


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # an observable on a small lattice: one launch and its result on the host
        {"name": "plaquette-su3-f64-8x4", "kind": "plaquette", "group": "su3", "prec": 64, "dims": "8x8x8x8"},
        # molecular dynamics of compact U(1) in three dimensions
        {"name": "hmd-u1-f32-3d", "kind": "hmd", "group": "u1", "prec": 32, "dims": "64x96x80", "scheme": "2lf",
         "eps": 0.5, "steps": 10, "beta": 2.0},
        # the reference's own configuration: FP64 SU(3), 8^4, beta 5.7, ten leapfrog steps, graph-replayed chain
        {"name": "chain-su3-f64-8x4", "kind": "chain", "group": "su3", "prec": 64, "dims": "8x8x8x8",
         "scheme": "2lf", "eps": 0.5, "steps": 10, "beta": 5.7},
        # mixed-precision trajectory on a lattice whose extents are no powers of two
        {"name": "trajectory-su3-f32-ragged", "kind": "trajectory", "group": "su3", "prec": 32,
         "dims": "12x20x14x30", "scheme": "2mn", "eps": 0.5, "steps": 10, "beta": 6.0},
        # the production run: mixed precision SU(3) 32^4 at beta 6.0, twenty Omelyan steps
        {"name": "trajectory-su3-f32-32x4", "kind": "trajectory", "group": "su3", "prec": 32,
         "dims": "32x32x32x32", "scheme": "2mn", "eps": 0.5, "steps": 20, "beta": 6.0},
        # an ensemble of SU(2) replicas of several sizes advanced together, then written out
        {"name": "batch-su2-f32", "kind": "batch", "group": "su2", "prec": 32, "replicas": 24, "extents": "4,6,8,10,12",
         "sizes": 99, "scheme": "2lf", "eps": 0.5, "steps": 16, "beta": 2.4, "count": 3},
        # local updates: one heat-bath and three overrelaxation sweeps in FP64
        {"name": "sweeps-su3-f64", "kind": "sweeps", "group": "su3", "prec": 64, "dims": "12x12x12x24", "heatbath": 1,
         "overrelax": 3, "beta": 6.0},
        # overrelaxation of a large single-precision lattice
        {"name": "overrelax-su3-f32-32x4", "kind": "sweeps", "group": "su3", "prec": 32, "dims": "32x32x32x32",
         "heatbath": 0, "overrelax": 3, "beta": 6.0},
        # the static potential: all Wilson loops up to 8 x 12
        {"name": "wilson-su3-f32-24x4", "kind": "wilson", "group": "su3", "prec": 32, "dims": "24x24x24x24",
         "max_r": 8, "max_t": 12},
        # Landau gauge by overrelaxation: two blocks of ten sweeps from a random gauge
        {"name": "landau-or-su3-f64-24x4", "kind": "landau_or", "group": "su3", "prec": 64, "dims": "24x24x24x24",
         "sweeps": 20},
        # Landau gauge by Fourier-accelerated steepest descent: five steps
        {"name": "landau-fa-su3-f64-24x4", "kind": "landau_fa", "group": "su3", "prec": 64, "dims": "24x24x24x24",
         "steps": 5},
        # the reference's conjugate gradient for Landau gauge, SU(2), ragged extents
        {"name": "landau-cg-su2-f64", "kind": "landau_cg", "group": "su2", "prec": 64, "dims": "16x12x18x10",
         "steps": 8},
    ]


def _extent(rng, lo, hi):
    return 2 * max(1, round(math.exp(rng.uniform(math.log(lo), math.log(hi))) / 2))


def _lattice(rng, nd, vmin, vmax, choices=None):
    """extents whose volume is spread over [vmin, vmax] by its logarithm"""
    for _ in range(1000):
        v = math.exp(rng.uniform(math.log(vmin), math.log(vmax)))
        side = v ** (1.0 / nd)
        dims = [rng.choice(choices) if choices else _extent(rng, max(2.0, side / 1.8), side * 1.8) for _ in range(nd)]
        if vmin <= math.prod(dims) <= vmax and max(dims) < 256:
            return "x".join(map(str, dims))
    return "x".join(["16"] * nd)


def draw(rng):
    kind = rng.choice(["plaquette", "hmd", "chain", "trajectory", "trajectory", "batch", "sweeps", "wilson",
                       "landau_or", "landau_fa", "landau_cg"])
    c = {"kind": kind, "group": "su3", "prec": 64}
    if kind == "plaquette":
        c |= {"group": rng.choice(["u1", "su2", "su3"]), "dims": _lattice(rng, rng.choice([2, 3, 4]), 64, 1 << 17)}
    elif kind == "hmd":
        c |= {"group": rng.choice(["u1", "su2", "su3"]), "prec": rng.choice([32, 64])}
        c |= {"dims": _lattice(rng, rng.choice([2, 3, 4]), 1 << 10, 1 << (19 if c["prec"] == 32 else 16)),
              "scheme": rng.choice(["2lf", "2mn"]), "eps": 0.5, "steps": rng.randint(5, 15), "beta": 2.0 * NC[c["group"]]}
    elif kind == "chain":
        c |= {"group": rng.choice(["su2", "su3"]), "dims": _lattice(rng, 4, 1 << 8, 1 << 15), "scheme": "2lf",
              "eps": 0.5, "steps": rng.randint(8, 16)}
        c |= {"beta": 5.7 if c["group"] == "su3" else 2.3}
    elif kind == "trajectory":
        c |= {"prec": 32, "dims": _lattice(rng, 4, 1 << 12, 1 << 20), "scheme": rng.choice(["2lf", "2mn"]),
              "eps": 0.5, "steps": rng.randint(8, 20), "beta": round(rng.uniform(5.6, 6.2), 2)}
    elif kind == "batch":
        c |= {"group": "su2", "prec": 32, "replicas": rng.randint(8, 32), "extents": "4,6,8,10,12",
              "sizes": rng.randint(0, 10**6), "scheme": "2lf", "eps": 0.5, "steps": rng.randint(10, 16),
              "beta": round(rng.uniform(2.2, 2.6), 2), "count": rng.randint(1, 3)}
    elif kind == "sweeps":
        c |= {"prec": rng.choice([32, 64])}
        c |= {"dims": _lattice(rng, 4, 1 << 10, 1 << (20 if c["prec"] == 32 else 16)),
              "heatbath": 0 if c["prec"] == 32 else 1, "overrelax": rng.randint(1, 4),
              "beta": round(rng.uniform(5.6, 6.2), 2)}
    elif kind == "wilson":
        c |= {"prec": 32, "dims": _lattice(rng, 4, 1 << 14, 1 << 19)}
        dims = _dims(c)
        c |= {"max_r": min(rng.randint(3, 10), *dims[:3]), "max_t": min(rng.randint(4, 14), dims[3])}
    elif kind == "landau_or":
        c |= {"dims": _lattice(rng, 4, 1 << 10, 1 << 18), "sweeps": rng.choice([10, 20])}
    elif kind == "landau_fa":
        c |= {"dims": _lattice(rng, 4, 1 << 10, 1 << 18, FFT_EXTENTS), "steps": rng.randint(3, 6)}
    else:
        c |= {"group": rng.choice(["su2", "su3"]), "dims": _lattice(rng, 4, 1 << 10, 1 << 15),
              "steps": rng.randint(5, 8)}
    return c


def _dims(case):
    return tuple(int(x) for x in case["dims"].split("x"))


def _batch_dims(case):
    r = random.Random(case["sizes"])
    ext = [int(x) for x in case["extents"].split(",")]
    return [(r.choice(ext),) * 4 for _ in range(case["replicas"])]


def _n_force(case):
    """momentum steps of one trajectory (link updates: one more)"""
    return (1 if case["scheme"] == "2lf" else 2) * case["steps"]


# FP operations of one 3x3 (2x2, 1x1) complex product, as the group's own
# representation multiplies (quaternions for SU(2))
_MUL = {"u1": 6, "su2": 28, "su3": 198}


def work(case):
    """each input read and each output written once; link products counted as
    products of the group's elements"""
    kind, b = case["kind"], case["prec"] // 8
    if kind == "batch":
        V, nd = sum(math.prod(d) for d in _batch_dims(case)), 4
    else:
        V, nd = math.prod(_dims(case)), len(_dims(case))
    nr, na, m = NREAL[case["group"]], NALG[case["group"]], _MUL[case["group"]]
    planes = nd * (nd - 1) // 2
    link, alg = nr * b * V, na * b * V
    # a momentum step: two products a plane, its closure, the lower staples and
    # theirs; a link update: the exponential (two products) and the product
    md = (planes * 3 + 2 * planes + nd) * m * V, 3 * nd * m * V
    if kind == "plaquette":
        return {"bytes": nd * link, "flops": planes * 2.2 * m * V}
    if kind in ("hmd", "chain", "trajectory", "batch"):
        n, count = _n_force(case), case.get("count", 1)
        # every step reads and writes what it updates: the links and momenta are larger than the chip's caches
        return {"bytes": count * ((n + 1) * (2 * nd * link + nd * alg) + n * (nd * link + 2 * nd * alg)),
                "flops": count * (n * md[0] + (n + 1) * md[1])}
    if kind == "sweeps":
        n = case["heatbath"] + case["overrelax"]
        return {"bytes": n * 2 * nd * link, "flops": n * nd * (2 * 2 * (nd - 1) + 2) * m * V}
    if kind == "wilson":
        return {"bytes": 4 * link, "flops": case["max_r"] * case["max_t"] * 3 * 2.2 * m * V}
    if kind == "landau_cg":
        return {"bytes": case["steps"] * 6 * (nd + 2) * link, "flops": case["steps"] * (4 * nd + 5 * 2 * nd) * m * V}
    if kind == "landau_or":
        return {"bytes": case["sweeps"] * (nd + 2) * link, "flops": case["sweeps"] * (2 * nd + 2) * m * V}
    return {"bytes": case["steps"] * ((nd + 2) * link + 8 * 4 * 2 * na * V), "flops": case["steps"] * (2 * nd + 3) * m * V}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _mul(a, b):
    """matrix product over the two leading axes"""
    return (a.unsqueeze(2) * b.unsqueeze(0)).sum(1)


def _adj(a):
    return a.transpose(0, 1).conj()


def _eye(n, like):
    e = torch.zeros_like(like)
    for i in range(n):
        e[i, i] = 1
    return e


def _exp(x, terms=16):
    r = _eye(x.shape[0], x)
    for k in range(terms, 0, -1):
        r = _mul(x, r) / k
        for i in range(x.shape[0]):
            r[i, i] += 1
    return r


def _tr(a):
    return sum(a[i, i] for i in range(a.shape[0]))


def _alg_from_reals(group, p):
    """Gaussian algebra element of DIM normals (leading axis)"""
    if group == "u1":
        return (1j * p[0] * math.sqrt(0.5))[None, None]
    if group == "su2":
        return _quat([torch.zeros_like(p[0]), 0.5 * p[0], 0.5 * p[1], 0.5 * p[2]])
    r3 = 1 / math.sqrt(3.0)
    a0, a1 = 0.5j * (p[2] + p[7] * r3), 0.5j * (-p[2] + p[7] * r3)
    b01, b02, b12 = 0.5 * torch.complex(p[1], p[0]), 0.5 * torch.complex(p[4], p[3]), 0.5 * torch.complex(p[6], p[5])
    return torch.stack([torch.stack([a0, b01, b02]), torch.stack([-b01.conj(), a1, b12]),
                        torch.stack([-b02.conj(), -b12.conj(), -(a0 + a1)])])


def _quat(q):
    return torch.stack([torch.stack([torch.complex(q[0], q[1]), torch.complex(q[2], q[3])]),
                        torch.stack([torch.complex(-q[2], q[3]), torch.complex(q[0], -q[1])])])


def _haar(group, shape, gen):
    n = lambda k: torch.randn((k, *shape), generator=gen, device=GPU, dtype=torch.float64)  # noqa: E731
    if group == "u1":
        z = torch.complex(*n(2))[None, None]
        return z / z.abs()
    if group == "su2":
        q = n(4)
        return _quat(q / q.norm(dim=0))
    r, rows = torch.complex(n(9), n(9)).reshape(3, 3, *shape), []
    for i in range(2):
        v = r[i]
        for u in rows:
            v = v - (u.conj() * v).sum(0) * u
        rows.append(v / (v.abs() ** 2).sum(0).sqrt())
    return torch.stack([*rows, _cross_conj(*rows)])


def _cross_conj(a, b):
    return torch.stack([a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]]).conj()


def _fwd(a, mu):
    """a(x + mu), the lattice in the trailing axes of a (two matrix axes first)"""
    return torch.roll(a, -1, 2 + mu)


def _bwd(a, mu):
    return torch.roll(a, 1, 2 + mu)


# spread of the links around the identity: a plaquette near 0.6, or (chains
# that decide for themselves whether to accept) near the cold start, from
# where the first trajectories of a run are accepted
_WIDTH, _COLD = {"u1": 0.5, "su2": 0.5, "su3": 0.42}, 0.1


def _links(group, prec, dims, gen, cold=False):
    """links (nd, V, reals) in the host layout, in the case's precision"""
    g, out = _haar(group, dims, gen), []
    for mu in range(len(dims)):
        p = torch.randn((NALG[group], *dims), generator=gen, device=GPU, dtype=torch.float64)
        v = _exp((_COLD if cold else _WIDTH[group]) * _alg_from_reals(group, p))
        out.append(_reals(group, _mul(_mul(g, v), _adj(_fwd(g, mu)))))
    return torch.stack(out).to(torch.float32 if prec == 32 else torch.float64)


def _momenta(group, prec, dims, gen):
    out = []
    for _ in dims:
        p = torch.randn((NALG[group], *dims), generator=gen, device=GPU, dtype=torch.float64)
        out.append(_reals(group, _alg_from_reals(group, p)))
    return torch.stack(out).to(torch.float32 if prec == 32 else torch.float64)


def _reals(group, m):
    """matrices (n, n, *dims) -> host objects (V, reals)"""
    if group == "su2":
        r = torch.stack([m[0, 0].real, m[0, 0].imag, m[0, 1].real, m[0, 1].imag])
    else:
        r = torch.view_as_real(m).movedim(-1, 2).reshape(-1, *m.shape[2:])
    return r.reshape(r.shape[0], -1).T.contiguous()


def _matrices(group, v, dims):
    """host objects (V, reals) -> complex128 matrices (n, n, *dims)"""
    r = v.double().T.reshape(NREAL[group], *dims)
    if group == "su2":
        return _quat(r)
    n = NC[group]
    z = torch.complex(r[0::2], r[1::2])
    return z.reshape(n, n, *dims).contiguous()


def _host(t):
    return t.cpu().numpy()


def _generator(seed):
    return torch.Generator(device=GPU).manual_seed(int(seed) * 7919 + 17)


# ---------------------------------------------------------------------------
# outputs: a field's device storage (even/odd structure of arrays)
# ---------------------------------------------------------------------------
class _Storage:
    """a field's device memory for torch; keeps its owners alive"""

    def __init__(self, field, reals, owners):
        self.owners = (field, owners)
        t = "<f4" if field.prec == mesh.F32 else "<f8"
        n = field.nstack * field.grid.size * reals
        self.__cuda_array_interface__ = {"shape": (n,), "typestr": t, "data": (field.device_ptr, False), "version": 3}


def _view(state, field):
    """the field's storage as a tensor, made again when the field's memory moves"""
    key, p = id(field), field.device_ptr
    got = state["views"].get(key)
    if got is None or got[0] != p:
        reals = mesh.NREAL[field.group] if field.kind == mesh.GROUP else mesh.NALG[field.group]
        got = (p, torch.as_tensor(_Storage(field, reals, state.get("owner")), device=GPU))
        state["views"][key] = got
    return got[1]


def _device_layout(group, prec, x, algebra, dims):
    """objects (components, V, host reals) in the order of the device storage"""
    V = math.prod(dims)
    coords = torch.meshgrid(*[torch.arange(d, device=GPU) for d in dims], indexing="ij")
    order = torch.argsort(sum(coords).reshape(-1) & 1, stable=True)  # even sites first, each parity lexicographic
    if algebra:
        pick = {"u1": [1], "su2": [1, 2, 3], "su3": [1, 9, 2, 3, 4, 5, 10, 11]}[group]
        x = x[..., pick]
    x, out = x[:, order], []
    nr, wide, k = x.shape[-1], 4 if prec == 32 else 2, 0
    while k < nr:
        w = wide if nr - k >= wide else 2 if nr - k >= 2 else 1
        out.append(x[..., k:k + w].reshape(x.shape[0], V * w))
        k += w
    return torch.cat(out, 1).reshape(-1)


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
_context = None


def _ctx():
    global _context
    if _context is None:
        _context = mesh.Context(0)
    return _context


def _prec(case):
    return mesh.F32 if case["prec"] == 32 else mesh.F64


def _inputs(case, seed):
    """the case's links and momenta (host layout, on the GPU)"""
    gen = _generator(seed)
    if case["kind"] == "batch":
        return {"links": [_links(case["group"], case["prec"], d, gen, True) for d in _batch_dims(case)]}
    inp = {"links": _links(case["group"], case["prec"], _dims(case), gen, case["kind"] == "chain")}
    if case["kind"] in ("hmd", "trajectory"):
        inp["momenta"] = _momenta(case["group"], case["prec"], _dims(case), gen)
    return inp


def prepare(case, seed):
    kind, prec, ctx, inp = case["kind"], _prec(case), _ctx(), _inputs(case, seed)
    s = {"case": case, "seed": int(seed), "views": {}}
    if "scheme" in case:
        s["deltas"] = mesh.make_deltas(case["scheme"], case["eps"], case["steps"])
    if kind == "batch":
        dims = _batch_dims(case)
        s["chain"] = mesh.HmcBatch(ctx, case["group"], prec, dims, [int(seed) + r for r in range(len(dims))])
        for r, u in enumerate(inp["links"]):
            s["chain"].import_(r, _host(u))
        s["betas"] = [case["beta"]] * len(dims)
        return s
    grid = mesh.Grid(_dims(case))
    if kind in ("chain", "trajectory"):
        h = s["owner"] = s["chain"] = mesh.Hmc(ctx, case["group"], prec, grid, int(seed))
        s["U"], s["P"] = h.U, h.P
        s["U"].import_(_host(inp["links"]))
        if kind == "trajectory":
            s["P0"] = mesh.Momenta(ctx, case["group"], prec, grid).import_(_host(inp["momenta"]))
        return s
    s["U"] = mesh.GaugeField(ctx, case["group"], prec, grid).import_(_host(inp["links"]))
    if kind == "hmd":
        s["P"] = mesh.Momenta(ctx, case["group"], prec, grid).import_(_host(inp["momenta"]))
    elif kind.startswith("landau"):
        s["landau"] = mesh.Landau(s["U"])
        if kind == "landau_fa":
            s["fa"] = mesh.LandauFA(s["U"])
            s["fa"].set_plain(0.08)
        s["owner"] = (s["landau"], s.get("fa"))
    s["sweep"] = 0
    return s


def run(state):
    c = state["case"]
    kind = c["kind"]
    if kind == "plaquette":
        return mesh.plaquette(state["U"])
    if kind == "hmd":
        mesh.run_hmd(state["U"], state["P"], c["beta"], state["deltas"])
        return {"U": _view(state, state["U"]), "P": _view(state, state["P"])}
    if kind == "chain":
        state["chain"].run(c["beta"], state["deltas"], 1)
        return {"U": _view(state, state["U"])}
    if kind == "trajectory":
        # the trajectory on supplied momenta; uniform 0 accepts it
        state["chain"].update_supplied(state["P0"], 0.0, c["beta"], state["deltas"])
        return {"U": _view(state, state["U"]), "P": _view(state, state["P"])}
    if kind == "batch":
        h = state["chain"]
        h.run(state["betas"], state["deltas"], c["count"])
        return [h.export(r) for r in range(h.R)]
    if kind == "sweeps":
        for _ in range(c["heatbath"]):
            mesh.heatbath_sweep(state["U"], c["beta"], state["seed"], state["sweep"])
            state["sweep"] += 1
        for _ in range(c["overrelax"]):
            mesh.overrelax_sweep(state["U"])
        return {"U": _view(state, state["U"])}
    if kind == "wilson":
        return mesh.wilson_loops(state["U"], c["max_r"], c["max_t"])
    g = state["landau"].g
    state["landau"].reset()
    if kind == "landau_or":
        _, theta = state["landau"].overrelax(omega=1.7, tol=1e-14, max_sweeps=c["sweeps"], check_every=10)
    elif kind == "landau_fa":
        _, _, theta = state["fa"].run(g, tol=1e-14, max_iter=c["steps"])
    else:
        _, theta = state["landau"].run(c["steps"], tol=1e-14)
    return {"g": _view(state, g), "theta": theta}


# ---------------------------------------------------------------------------
# the same in 64 bits, in plain torch
# ---------------------------------------------------------------------------
def _proj(m):
    """antihermitian, for N > 1 traceless, part"""
    n, a = m.shape[0], 0.5 * (m - _adj(m))
    if n > 1:
        t = _tr(a) / n
        for i in range(n):
            a[i, i] -= t
    return a


def _staple(U, mu):
    S = torch.zeros_like(U[mu])
    for nu in range(len(U)):
        if nu != mu:
            S += _mul(_fwd(U[nu], mu), _adj(_mul(U[nu], _fwd(U[mu], nu))))
            S += _bwd(_mul(_adj(_mul(U[mu], _fwd(U[nu], mu))), U[nu]), nu)
    return S


def _reunit(m):
    r = 1.5 * m - 0.5 * _mul(_mul(m, _adj(m)), m)
    if m.shape[0] < 3:
        return r
    det = sum(r[0, i] * (r[1, (i + 1) % 3] * r[2, (i + 2) % 3] - r[1, (i + 2) % 3] * r[2, (i + 1) % 3]) for i in range(3))
    return r * (4.0 / 3.0 - det / 3.0)


def _gram_schmidt(m):
    if m.shape[0] < 3:
        return m / (m[0].abs() ** 2).sum(0).sqrt()
    a = m[0] / (m[0].abs() ** 2).sum(0).sqrt()
    b = m[1] - (a.conj() * m[1]).sum(0) * a
    b = b / (b.abs() ** 2).sum(0).sqrt()
    return torch.stack([a, b, _cross_conj(a, b)])


def _plaq(U):
    n, nd, tot = U[0].shape[0], len(U), 0.0
    for mu in range(nd):
        for nu in range(mu + 1, nd):
            ab, dc = _mul(U[mu], _fwd(U[nu], mu)), _mul(U[nu], _fwd(U[mu], nu))
            tot += float((ab * dc.conj()).real.sum())
    return tot / (nd * (nd - 1) / 2 * U[0][0, 0].numel()) / n


def _md(U, P, beta, deltas):
    """alternating link updates and momentum steps, in place"""
    n = U[0].shape[0]
    for i, d in enumerate(deltas):
        for mu in range(len(U)) if i % 2 == 0 else ():
            U[mu] = _mul(_exp(d * P[mu]), U[mu])
        if i % 2:
            F = [_proj(_mul(U[mu], _staple(U, mu))) * (beta / (2 * n)) for mu in range(len(U))]
            for mu in range(len(U)):
                P[mu] = P[mu] - d * F[mu]


def _philox(site, word1, ctr, seed):
    """Philox4x32-10 of Salmon et al. 2011: four 32-bit words per site"""
    m32 = 0xFFFFFFFF
    c = [site, torch.full_like(site, word1 & m32), torch.full_like(site, ctr & m32), torch.full_like(site, ctr >> 32)]
    k0, k1 = seed & m32, (seed >> 32) & m32
    for _ in range(10):
        p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((p1 >> 32) & m32) ^ c[1] ^ k0, p1 & m32, ((p0 >> 32) & m32) ^ c[3] ^ k1, p0 & m32]
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return c


def _u53(a, b):
    return (((a << 21) ^ (b >> 11)).double() + 0.5) * 2.0**-53


def _u24(a):
    return ((a >> 8).double() + 0.5) * 2.0**-24


def _drawn_momenta(group, prec, dims, seed, traj):
    """the momenta a chain with this seed draws for trajectory `traj`"""
    site = torch.arange(math.prod(dims), device=GPU)
    out = []
    for mu in range(len(dims)):
        p, blk = [], 0
        while len(p) < NALG[group]:
            w = _philox(site, (TAG_MOMENTUM << 24) | (mu << 8) | blk, traj, seed)
            pairs = [(_u24(w[0]), _u24(w[1])), (_u24(w[2]), _u24(w[3]))] if prec == 32 else [(_u53(w[0], w[1]), _u53(w[2], w[3]))]
            for a, b in pairs:
                rad = torch.sqrt(-2.0 * torch.log(a))
                p += [rad * torch.cos(2 * math.pi * b), rad * torch.sin(2 * math.pi * b)]
            blk += 1
        out.append(_alg_from_reals(group, torch.stack(p[:NALG[group]]).reshape(-1, *dims)))
    return out


def _energy(U, P, beta):
    nd, V = len(U), U[0][0, 0].numel()
    return (1 - _plaq(U)) * beta * (nd * (nd - 1) / 2) * V + sum(float((p.abs() ** 2).sum()) for p in P)


def _chain(case, U, dims, seed, count):
    """`count` trajectories of runHmcUpdate on the chain's own streams"""
    deltas = mesh.make_deltas(case["scheme"], case["eps"], case["steps"]).tolist()
    for k in range(count):
        P = _drawn_momenta(case["group"], case["prec"], dims, seed, k)
        h_old, new = _energy(U, P, case["beta"]), [u.clone() for u in U]
        _md(new, P, case["beta"], deltas)
        new = [_reunit(u) for u in new]
        w = _philox(torch.zeros(1, dtype=torch.int64, device=GPU), TAG_METROPOLIS << 24, k, seed)
        if float(_u53(w[0], w[1])) < math.exp(min(50.0, h_old - _energy(new, P, case["beta"]))):
            U = new
    return U


def _block(W, i, j):
    """SU(2)-like part of rows and columns i, j"""
    return 0.5 * (W[i, i] + W[j, j].conj()), 0.5 * (W[i, j] - W[j, i].conj())


def _rotate(M, i, j, p, q):
    x, y = M[i].clone(), M[j].clone()
    M[i], M[j] = p * x + q * y, -q.conj() * x + p.conj() * y


def _su2_heatbath(alpha, site, mu, sub, seed, ctr):
    """SU(2) elements with density exp(alpha x0): Kennedy-Pendleton above
    alpha = 1, Creutz below; (x0 + i x3, x2 + i x1) and where one was found"""
    def draw(call):
        w = _philox(site, (TAG_HEATBATH << 24) | (mu << 8) | (sub << 6) | call, ctr, seed)
        return _u53(w[0], w[1]), _u53(w[2], w[3])

    x0, done = torch.zeros_like(alpha), torch.zeros_like(alpha, dtype=torch.bool)
    for a in range(24):
        (u0, u1), (u2, u3) = draw(1 + 2 * a), draw(2 + 2 * a)
        t = 1 + torch.log(u0 + (1 - u0) * torch.exp(-2 * alpha)) / alpha
        d = -(torch.log(u0) + torch.cos(2 * math.pi * u1) ** 2 * torch.log(u2)) / alpha
        low = alpha < 1
        ok = torch.where(low, u1 * u1 <= 1 - t * t, u3 * u3 <= 1 - 0.5 * d) & ~done
        x0, done = torch.where(ok, torch.where(low, t, 1 - d), x0), done | ok
        if bool(done.all()):
            break
    u0, u1 = draw(0)
    ct = 2 * u0 - 1
    r, st = torch.sqrt((1 - x0 * x0).clamp(min=0)), torch.sqrt((1 - ct * ct).clamp(min=0))
    x1, x2, x3 = r * st * torch.cos(2 * math.pi * u1), r * st * torch.sin(2 * math.pi * u1), r * ct
    return torch.complex(x0, x3), torch.complex(x2, x1), done


def _sweep(U, dims, beta, heatbath, seed, ctr):
    """a checkerboard sweep of SU(3) links by their SU(2) subgroups, in place"""
    coords = torch.meshgrid(*[torch.arange(d, device=GPU) for d in dims], indexing="ij")
    parity, lex = sum(coords) & 1, torch.arange(math.prod(dims), device=GPU).reshape(dims)
    for mu in range(len(U)):
        for par in range(2):
            at = parity == par
            u = U[mu][:, :, at].clone()
            W = _mul(u, _staple(U, mu)[:, :, at])
            for sub, (i, j) in enumerate(((0, 1), (1, 2), (0, 2))):
                a, b = _block(W, i, j)
                k = torch.sqrt(a.abs() ** 2 + b.abs() ** 2)
                a, b = a / k, b / k
                if heatbath:
                    xp, xq, ok = _su2_heatbath(2 * beta * k / 3, lex[at], mu, sub, seed, ctr)
                else:
                    xp, xq, ok = a.conj(), -b, torch.ones_like(k, dtype=torch.bool)
                p, q = xp * a.conj() + xq * b.conj(), -xp * b + xq * a
                p, q = torch.where(ok, p, torch.ones_like(p)), torch.where(ok, q, torch.zeros_like(q))
                _rotate(u, i, j, p, q)
                _rotate(W, i, j, p, q)
            U[mu][:, :, at] = _reunit(u)


def _theta(U, g):
    D = torch.zeros_like(g)
    for mu in range(len(U)):
        A = _proj(_mul(_mul(g, U[mu]), _adj(_fwd(g, mu))))
        D += A - _bwd(A, mu)
    return D, float((D.abs() ** 2).sum()) / (len(U) * g[0, 0].numel())


def _or_power(h, w):
    c, a = 0.5 * w * (w - 1), h[0] - 1
    v2 = h[1] ** 2 + h[2] ** 2 + h[3] ** 2
    f = w + 2 * c * a
    r = torch.stack([1 + w * a + c * (a * a - v2), h[1] * f, h[2] * f, h[3] * f])
    return r / r.norm(dim=0)


def _closing(U, g):
    K = torch.zeros_like(g)
    for mu in range(len(U)):
        K += _mul(U[mu], _adj(_fwd(g, mu))) + _adj(_bwd(_mul(g, U[mu]), mu))
    return K


def _landau_or(U, g, sweeps, dims):
    coords = torch.meshgrid(*[torch.arange(d, device=GPU) for d in dims], indexing="ij")
    parity = sum(coords) & 1
    for _ in range(sweeps):
        for par in range(2):
            at = parity == par
            G = g[:, :, at].clone()
            W = _mul(G, _closing(U, g)[:, :, at])
            for i, j in ((0, 1), (0, 2), (1, 2)):
                a, b = _block(W, i, j)
                q = torch.stack([a.real, b.imag, b.real, a.imag])
                h = _or_power(q / q.norm(dim=0) * torch.tensor([1.0, -1, -1, -1], device=GPU, dtype=q.dtype)[:, None], 1.7)
                p, q = torch.complex(h[0], h[3]), torch.complex(h[2], h[1])
                _rotate(G, i, j, p, q)
                _rotate(W, i, j, p, q)
            g[:, :, at] = G
    return _gram_schmidt(g)


def _landau_fa(U, g, steps, dims):
    p2 = sum((4 * torch.sin(math.pi * torch.arange(d, device=GPU, dtype=torch.float64) / d) ** 2).reshape(
        [-1 if k == mu else 1 for k in range(len(dims))]) for mu, d in enumerate(dims))
    m = 0.08 * float(p2.max()) / torch.where(p2 > 0, p2, torch.full_like(p2, math.inf))
    D, th = _theta(U, g)
    axes = tuple(range(2, 2 + len(dims)))
    for _ in range(steps):
        trial = _gram_schmidt(_mul(_exp(-torch.fft.ifftn(m * torch.fft.fftn(D, dim=axes), dim=axes), 24), g))
        D2, th2 = _theta(U, trial)
        if not th2 < th:
            trial = _landau_or(U, g, 10, dims)
            D2, th2 = _theta(U, trial)
        g, D, th = trial, D2, th2
    return g, th


def _landau_cg(U, g, steps):
    n, nd, V = g.shape[0], len(U), g[0, 0].numel()
    fac = 1.0 / (n * nd * V)

    def functional(h):
        return sum(float((_mul(h, U[mu]) * _fwd(h, mu).conj()).real.sum()) for mu in range(nd)) * fac

    def stepped(F, e):
        k = max(0, math.ceil(math.log2(max(1e-300, abs(e) * float(F.abs().max()) * 4))))
        x = _exp(F * (e / 2**k))
        for _ in range(k):
            x = _mul(x, x)
        return _mul(x, g)

    eps = 3000.0
    for _ in range(steps):
        F = _proj(_mul(g, _closing(U, g))) * (-0.5 * fac)
        base, y1 = functional(g), functional(stepped(F, eps))
        while y1 <= base:
            eps *= 0.5
            y1 = functional(stepped(F, eps))
        x1, x2, x3 = eps, 1.2 * eps, 0.8 * eps
        y2 = functional(stepped(F, x2))
        if y2 > y1:
            eps = x2
        else:
            y3 = functional(stepped(F, x3))
            eps = 0.5 * ((x2**2 - x3**2) * y1 - (x1**2 - x3**2) * y2 + (x1**2 - x2**2) * y3) / (
                (x2 - x3) * y1 - (x1 - x3) * y2 + (x1 - x2) * y3)
        g = _reunit(stepped(F, eps))
    return g, _theta(U, g)[1]


def _wilson(U, dims, max_r, max_t):
    out, V, n = np.zeros((max_r, max_t)), math.prod(dims), U[0].shape[0]
    T = [U[3]]
    for t in range(1, max_t):
        T.append(_mul(T[-1], torch.roll(U[3], -t, 5)))
    for mu in range(3):
        S = U[mu]
        for r in range(1, max_r + 1):
            if r > 1:
                S = _mul(S, torch.roll(U[mu], -(r - 1), 2 + mu))
            for t in range(1, max_t + 1):
                ab, dc = _mul(S, torch.roll(T[t - 1], -r, 2 + mu)), _mul(T[t - 1], torch.roll(S, -t, 5))
                out[r - 1, t - 1] += float((ab * dc.conj()).real.sum())
    return out / (3 * V * n)


def exact(case, seed):
    kind, group, prec = case["kind"], case["group"], case["prec"]
    inp = _inputs(case, seed)
    if kind == "batch":
        out = []
        for r, (d, u) in enumerate(zip(_batch_dims(case), inp["links"])):
            U = _chain(case, [_matrices(group, c, d) for c in u], d, int(seed) + r, case["count"])
            out.append(torch.stack([_reals(group, m) for m in U]).cpu().numpy())
        return out
    dims = _dims(case)
    U = [_matrices(group, c, dims) for c in inp["links"]]

    def stored(ms, algebra=False):
        return _device_layout(group, prec, torch.stack([_reals(group, m) for m in ms]), algebra, dims)

    if kind == "plaquette":
        return _plaq(U)
    if kind == "wilson":
        return _wilson(U, dims, case["max_r"], case["max_t"])
    if kind in ("hmd", "trajectory"):
        P = [_matrices(group, c, dims) for c in inp["momenta"]]
        _md(U, P, case["beta"], mesh.make_deltas(case["scheme"], case["eps"], case["steps"]).tolist())
        if kind == "trajectory":
            U = [_reunit(u) for u in U]
        return {"U": stored(U), "P": stored(P, True)}
    if kind == "chain":
        return {"U": stored(_chain(case, U, dims, int(seed), 1))}
    if kind == "sweeps":
        for k in range(case["heatbath"]):
            _sweep(U, dims, case["beta"], True, int(seed), k)
        for _ in range(case["overrelax"]):
            _sweep(U, dims, case["beta"], False, 0, 0)
        return {"U": stored(U)}
    g = _eye(NC[group], U[0])
    if kind == "landau_or":
        for _ in range(case["sweeps"] // 10):
            g = _landau_or(U, g, 10, dims)
        theta = _theta(U, g)[1]
    elif kind == "landau_fa":
        g, theta = _landau_fa(U, g, case["steps"], dims)
    else:
        g, theta = _landau_cg(U, g, case["steps"])
    return {"g": stored([g]), "theta": theta}
