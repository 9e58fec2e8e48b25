"""The work that users of this package have it do, as cases that can be timed
and compared: pressure solves from a few thousand to 29 million cells, single
trees and forests of independent problems, 2D and 3D, from device memory and
from host TreeData buffers, and the calls around a solve in a flow solver's
time step (a moving body's new fractions, a regrid, the projection step).

listed()             the cases
draw(rng)            one more case of the same ranges
prepare(case, seed)  a program's state before the call
run(state)           one pass through the public entry points, and its outputs
work(case)           bytes and operations that a pass cannot do without
exact(case, seed)    the outputs in 64 bits from plain torch, or None

The tree and the shape of the bodies belong to a case; the density ratio, the
right-hand side and the velocities come from the seed.
"""
import ctypes
import functools
import math

import numpy as np
import torch

import sayakaamr_gb300 as sg
from sayakaamr_gb300 import workloads as W

# cut cells and faces below this fraction are solid
MIN_FRACTION = 1e-2
# the relative tolerance of the repository's parity solves, and that of an
# ensemble, whose cut cells (up to 7 levels, density ratio up to 1000) let a
# true residual reach about 1e-10 in 64 bits
TOL, TOL_BATCH = 1e-10, 1e-9
# the largest solve for which a plain 64-bit solve takes a few seconds
EXACT_CELLS = 2_500_000


def _solve(name, **kw):
    c = dict(name=name, kind="solve", dim=2, nb=16, roots=1, min_level=4, max_level=7, band=1.0, problems=1,
             geometry=1, precision=1, smoother=0, n_post=2, inner_sweeps=2, omega=1.0, host=False)
    c.update(kw)
    return c


def listed():
    return [
        # a small 2D domain: 8x8-cell blocks, four levels around the bodies
        # (16 thousand cells), the quick start's parameters
        _solve("solve_2d_small", nb=8, roots=4, min_level=1, max_level=4, geometry=2),
        # one 2D two-phase problem with a solid (6 levels, about 340 thousand
        # cells), block-hybrid smoothing, the setting that suits this size
        _solve("solve_2d", roots=2, min_level=2, max_level=6, band=1.5, geometry=3, smoother=1, n_post=4),
        # an ensemble of a few independent 2D problems solved as one forest
        _solve("batch_16", problems=16, geometry=4, omega=1.1),
        # the same from and to the caller's pinned TreeData host buffers
        _solve("batch_64_host", problems=64, geometry=4, omega=1.1, host=True),
        # the benchmark's ensemble: 256 problems, about 29 million cells
        _solve("batch_256", problems=256, geometry=4, omega=1.1),
        # a caller who wants the whole preconditioner in 64 bits
        _solve("batch_32_fp64", problems=32, geometry=4, precision=0),
        # 3D, 16^3-cell blocks: one body, 2 and 16 million cells
        _solve("solve_3d", dim=3, min_level=2, max_level=4, band=1.5, geometry=5, smoother=1, n_post=3),
        _solve("solve_3d_large", dim=3, min_level=2, max_level=5, band=3.0, geometry=5, smoother=1, n_post=3),
        # a time step of a flow solver with a moving body between regrids:
        # new level set and right-hand side, one solve (3D, 8^3-cell blocks)
        _elbow("step_3d", "step", 5),
        _elbow("step_3d_large", "step", 7),
        # the step after a regrid: a new solver on the new tree that starts
        # from the old solution
        _elbow("regrid_3d", "regrid", 6),
        # the pressure step of a projection method from host face velocities:
        # divergence, solve, velocity correction
        _solve("project_2d", kind="project", roots=2, min_level=2, max_level=6, band=1.5, geometry=3, omega=1.1),
    ]


def _elbow(name, kind, max_level, **kw):
    c = dict(name=name, kind=kind, dim=3, nb=8, max_level=max_level, position=0.37, precision=1, smoother=0, n_post=4,
             inner_sweeps=2, omega=1.1)
    c.update(kw)
    return c


def draw(rng):
    kind = rng.choice(["single", "single", "forest", "forest", "box", "step", "regrid", "project"])
    geometry = rng.randrange(10, 1 << 20)
    omega = rng.choice([1.0, 1.1])
    smoother = rng.choice([0, 0, 1])
    n_post = rng.choice([3, 4]) if smoother else 2
    if kind in ("single", "project"):
        c = _solve("", nb=rng.choice([6, 8, 12, 16]), roots=rng.choice([1, 2, 3, 4]), min_level=rng.choice([1, 2]),
                   max_level=rng.choice([3, 4, 5, 6]), band=rng.choice([1.0, 1.5]), geometry=geometry,
                   precision=rng.choice([1, 1, 1, 0]), smoother=smoother, n_post=n_post, omega=omega)
        if kind == "project":
            c["kind"] = "project"
    elif kind == "forest":
        c = _solve("", problems=int(round(math.exp(rng.uniform(math.log(3), math.log(200))))), geometry=geometry,
                   precision=rng.choice([1, 1, 1, 0]), omega=omega, host=rng.choice([False, False, True]))
    elif kind == "box":
        c = _solve("", dim=3, nb=rng.choice([8, 12, 16]), min_level=2, max_level=rng.choice([3, 4]),
                   band=rng.choice([1.0, 1.5, 2.0]), geometry=geometry, smoother=smoother, n_post=n_post + 1,
                   omega=omega)
    else:
        c = _elbow("", kind, rng.choice([4, 5, 6]), position=round(rng.uniform(0.15, 0.8), 3), omega=omega,
                   n_post=rng.choice([2, 3, 4]))
    del c["name"]
    return c


# ---- trees and bodies (host) ----------------------------------------------
def _dist(xp, p, s):
    """distance-like function of the ellipse (2D) or ball (3D) s = (centre x,
    y, z, semi-axes a, b, angle), negative inside; s may carry leading axes"""
    x, y = p[..., 0] - s[..., 0], p[..., 1] - s[..., 1]
    ct, st = xp.cos(s[..., 5]), xp.sin(s[..., 5])
    u, v = (x * ct + y * st) / s[..., 3], (-x * st + y * ct) / s[..., 4]
    q = u * u + v * v
    if p.shape[-1] == 3:
        z = (p[..., 2] - s[..., 2]) / s[..., 3]
        q = q + z * z
    return (xp.sqrt(q) - 1.0) * xp.minimum(s[..., 3], s[..., 4])


def _bodies(c):
    """per problem: up to four solids (an unused one lies far outside), one
    density front, and the finest level"""
    rng = np.random.default_rng(c["geometry"])
    out = []
    for _ in range(c["problems"]):
        solids = np.tile(np.array([9.0, 9.0, 9.0, 0.1, 0.1, 0.0]), (4, 1))
        if c["dim"] == 3:
            solids[0] = [0.5, 0.5, 0.5, 0.08, 0.08, 0.0]
            r = rng.uniform(0.12, 0.18)
            front = np.array([*rng.uniform(0.35, 0.65, 3), r, r, 0.0])
            out.append((solids, front, c["max_level"]))
            continue
        for k in range(int(rng.integers(1, 5)) if c["problems"] > 1 else 1):
            a = rng.uniform(0.04, 0.10)
            s = [*rng.uniform(0.2, 0.8, 2), 0.0, a, a * rng.uniform(0.4, 1.0), rng.uniform(0, math.pi)]
            # bodies that touch could close off a pocket of fluid, which has
            # no solution of its own
            if all(math.hypot(s[0] - q[0], s[1] - q[1]) > a + q[3] + 0.05 for q in solids[:k] if q[0] < 5):
                solids[k] = s
        a = rng.uniform(0.12, 0.22)
        front = np.array([*rng.uniform(0.3, 0.7, 2), 0.0, a, a * rng.uniform(0.5, 1.0), rng.uniform(0, math.pi)])
        top = int(rng.integers(min(5, c["max_level"]), c["max_level"] + 1)) if c["problems"] > 1 else c["max_level"]
        out.append((solids, front, top))
    return out


def _near(s, lo, hi, band):
    """block [lo, hi] within `band` block widths of the surface of s"""
    c, h = 0.5 * (lo + hi), np.max(hi - lo, axis=1)
    return np.abs(_dist(np, c, s)) < (0.5 + band) * h


def _one_tree(c, solids, front, top):
    nd = c["dim"]
    if nd == 3:
        shapes = [np.array([0.5, 0.5, 0.5, 0.2, 0.2, 0.0])]
    else:
        shapes = [front] + [s for s in solids if s[0] < 5]

    def need(lo, hi, level):
        m = np.zeros(len(lo), dtype=bool)
        for s in shapes:
            m |= _near(s, lo, hi, c["band"])
        return m
    roots = (c["roots"], c["roots"], c["roots"] if nd == 3 else 1)
    while True:
        t = W.refine_tree(nd, c["nb"], roots, (0, 0, 0), (1, 1, 1 if nd == 3 else 0), c["min_level"], top, need,
                          capacity=40000)
        tb = t.tables()
        if c["problems"] == 1 or (tb["node_type"] == 1).sum() <= 1024 or top <= 5:
            return tb
        top -= 1


def _key(c):
    return tuple(sorted((k, v) for k, v in c.items() if k not in (
        "name", "precision", "smoother", "n_post", "inner_sweeps", "omega", "host")))


def _geometry(c):
    """(tables, problem of every block, bodies); for the elbow (tables before
    the regrid, tables after it or None)"""
    return _geometry_of(_key(c))


@functools.lru_cache(maxsize=32)
def _geometry_of(key):
    c = dict(key)
    if c["kind"] in ("step", "regrid"):
        t = W.elbow_tree(W.elbow_point(c["position"]), nb=c["nb"], max_level=c["max_level"])
        before = t.tables()
        if c["kind"] == "step":
            return before, None
        W.elbow_regrid(t, W.elbow_point(c["position"] + 0.04), c["max_level"])
        return before, t.tables()
    bodies = _bodies(c)
    tbs = [_one_tree(c, *b) for b in bodies]
    off = np.cumsum([0] + [t["num_blocks"] for t in tbs[:-1]])
    tb = dict(ndim=c["dim"], nb=c["nb"], num_blocks=int(sum(t["num_blocks"] for t in tbs)),
              min_level=c["min_level"], max_level=max(int(t["max_level"]) for t in tbs))
    for k in ("level", "which_child", "node_type", "block_len", "block_lo"):
        tb[k] = np.concatenate([t[k] for t in tbs])
    for k in ("neighbor", "child", "parent"):
        tb[k] = np.concatenate([np.where(t[k] >= 0, t[k] + o, t[k]) for t, o in zip(tbs, off)]).astype(np.int32)
    problem = np.repeat(np.arange(len(tbs)), [t["num_blocks"] for t in tbs])
    return tb, problem, (np.stack([b[0] for b in bodies]), np.stack([b[1] for b in bodies]))


def _bc(tb, dirichlet):
    """p = 0 on one face of the domain, walls elsewhere"""
    nd, n = tb["ndim"], tb["num_blocks"]
    nbr = tb["neighbor"].reshape(n, 6)
    bc = np.full((n, 6), -1, dtype=np.int32)
    for f in range(2 * nd):
        bc[nbr[:, f] <= sg.PHYS_BNDRY, f] = sg.DIRICHLET if f == dirichlet else sg.NEUMANN
    return bc.reshape(-1)


# ---- fields (GPU) ----------------------------------------------------------
def _points(tb, shift, extra=(0, 0, 0)):
    """[block, point, dim]: the points (i + shift) * dx of every block, nb +
    extra per dimension, first dimension fastest"""
    nd, nb, n = tb["ndim"], tb["nb"], tb["num_blocks"]
    ax = [torch.arange(nb + extra[d], dtype=torch.float64, device="cuda") + shift[d] for d in range(nd)]
    g = torch.meshgrid(*ax[::-1], indexing="ij")[::-1]
    idx = torch.stack([a.reshape(-1) for a in g], 1)
    lo = torch.as_tensor(tb["block_lo"].reshape(n, 3)[:, :nd].copy(), device="cuda")
    dx = torch.as_tensor(tb["block_len"].reshape(n, 3)[:, :nd] / nb, device="cuda")
    return lo[:, None, :] + idx[None] * dx[:, None, :]


def _gaussians(p, problem, count, g, sigma):
    nd = p.shape[-1]
    amp = torch.randn(count, 8, generator=g, dtype=torch.float64).cuda()
    cen = (0.1 + 0.8 * torch.rand(count, 8, nd, generator=g, dtype=torch.float64)).cuda()
    f = torch.zeros(p.shape[:2], dtype=torch.float64, device="cuda")
    for q in range(8):
        d2 = ((p - cen[problem, q][:, None, :]) ** 2).sum(-1)
        f += amp[problem, q][:, None] * torch.exp(d2 / (-2.0 * sigma * sigma))
    return f


def _fields(c, seed):
    """fractions, face coefficient 1/rho and right-hand side of a solve"""
    tb, problem, (solids, fronts) = _geometry(c)
    nd, nb, n = tb["ndim"], tb["nb"], tb["num_blocks"]
    g = torch.Generator().manual_seed(seed)
    prob = torch.as_tensor(problem, device="cuda")
    sol, fro = torch.as_tensor(solids, device="cuda"), torch.as_tensor(fronts, device="cuda")
    ratio = (10.0 ** (1.0 + 2.0 * torch.rand(c["problems"], generator=g, dtype=torch.float64))).cuda()[prob][:, None]
    h = torch.as_tensor(tb["block_len"].reshape(n, 3)[:, :1] / nb, device="cuda")

    def frac(p):
        v = torch.ones(p.shape[:2], dtype=torch.float64, device="cuda")
        for k in range(solids.shape[1]):
            if (solids[:, k, 0] < 5).any():
                v = torch.minimum(v, torch.clamp(_dist(torch, p, sol[prob, k][:, None, :]) / h + 0.5, 0.0, 1.0))
        return torch.where(v < MIN_FRACTION, torch.zeros_like(v), v)

    half = [0.5] * nd
    vol, closed = frac(_points(tb, half)), None
    area, bface = [], []
    for d in range(nd):
        ext = tuple(int(q == d) for q in range(3))
        at = lambda s: _points(tb, [s if q == d else 0.5 for q in range(nd)], ext)  # noqa: E731
        a = frac(at(0.0))
        # a face is open only between two fluid cells
        a = torch.where((frac(at(-0.5)) > 0) & (frac(at(0.5)) > 0), a, torch.zeros_like(a))
        rho = 1.0 + (ratio - 1.0) * torch.clamp(0.5 - _dist(torch, at(0.0), fro[prob][:, None, :]) / (2.0 * h), 0, 1)
        area.append(a)
        bface.append(1.0 / rho)
        av = a.reshape([n] + [nb + ext[q] for q in range(nd)][::-1])
        shut = (av.narrow(nd - d, 0, nb) == 0) & (av.narrow(nd - d, 1, nb) == 0)
        closed = shut if closed is None else closed & shut
    vol = torch.where(closed.reshape(n, -1), torch.zeros_like(vol), vol)
    f = _gaussians(_points(tb, half), prob, c["problems"], g, 0.05 if nd == 2 else 0.08)
    leaf = torch.as_tensor(tb["node_type"] == 1, device="cuda")
    f = f * leaf[:, None]
    top = torch.zeros(c["problems"], dtype=torch.float64, device="cuda")
    top.scatter_reduce_(0, prob, (f.abs() * (vol > 0)).amax(1), "amax")
    rhs = -f / top[prob][:, None]
    return tb, vol, area, bface, rhs.contiguous(), g


def _level_set(p, centre):
    """inside the elbow's tube and outside the sphere at `centre`"""
    c, R = torch.as_tensor(W.ELBOW_C, device="cuda"), W.ELBOW_R

    def seg(a, b):
        a, b = (torch.tensor(v, dtype=torch.float64, device="cuda") for v in (a, b))
        t = torch.clamp(((p - a) * (b - a)).sum(-1) / ((b - a) ** 2).sum(), 0.0, 1.0)
        return torch.linalg.norm(p - (a + t[..., None] * (b - a)), dim=-1)
    x, y, z = (p[..., q] - c[q] for q in range(3))
    arc = torch.sqrt((torch.hypot(x, y) - R) ** 2 + z * z)
    d = torch.where((x >= 0) & (y >= 0), arc, torch.full_like(arc, math.inf))
    cx, cy, cz = (float(v) for v in W.ELBOW_C)
    d = torch.minimum(d, seg([cx + R, 0.0, cz], [cx + R, cy, cz]))
    d = torch.minimum(d, seg([cx, cy + R, cz], [0.0, cy + R, cz]))
    sphere = torch.linalg.norm(p - torch.as_tensor(centre, device="cuda"), dim=-1) - W.SPHERE_R
    return torch.minimum(W.ELBOW_TUBE - d, sphere)


def _elbow_fields(c, tb, seed, position):
    """level set on the grown boxes (one ghost layer) and right-hand side"""
    g = torch.Generator().manual_seed(seed)
    ls = _level_set(_points(tb, [-0.5] * 3, (2, 2, 2)), W.elbow_point(position))
    prob = torch.zeros(tb["num_blocks"], dtype=torch.int64, device="cuda")
    f = _gaussians(_points(tb, [0.5] * 3), prob, 1, g, 0.08)
    leaf = torch.as_tensor(tb["node_type"] == 1, device="cuda")
    return ls.contiguous(), (-f * leaf[:, None]).contiguous()


# ---- states ----------------------------------------------------------------
def _params(c):
    p = dict(tol_rel=TOL_BATCH if c.get("problems", 1) > 1 else TOL, tol_abs=0.0, use_mg_precond=1, bottom=1,
             precision=c["precision"], n_post_smooth=c["n_post"], smoother=c["smoother"], inner_sweeps=c["inner_sweeps"],
             relax_omega=c["omega"], max_iter=2000)
    if c["kind"] in ("step", "regrid"):
        # a time-stepping program keeps the small bottom level's inverse
        p.update(bottom_level=1, bottom_refresh=0)
    return p


def _host(t):
    return t.reshape(-1).cpu().numpy()


def _grown(cells, tb):
    """compact cells as a pinned TreeData buffer with one ghost layer"""
    nd, nb, n = tb["ndim"], tb["nb"], tb["num_blocks"]
    out = torch.zeros([n] + [nb + 2] * nd, dtype=torch.float64)
    out[(slice(None),) + (slice(1, nb + 1),) * nd] = cells.cpu().reshape([n] + [nb] * nd)
    return out.reshape(-1).pin_memory()


def prepare(case, seed):
    c = case
    if c["kind"] in ("step", "regrid"):
        before, after = _geometry(c)
        s = sg.MacSolver(before)
        s.set_bc(_bc(before, 0))
        s.set_params(**_params(c))
        ls, rhs = _elbow_fields(c, before, seed, c["position"])
        torch.cuda.synchronize()
        s.set_ib_frac_by_ls_device(ls.data_ptr(), ngrow=1)
        s.set_rhs_device(rhs.data_ptr())
        s.set_zero_sol()
        s.prepare()
        st = dict(kind=c["kind"], solver=s)
        tb, where = before, c["position"] + 0.01
        if c["kind"] == "regrid":
            # the sequence has solved on the old tree, and its later trees
            # use the smoother variant that the first one tuned
            s.cg_solve()
            tb, where = after, c["position"] + 0.04
            st.update(tables=after, bc=_bc(after, 0),
                      params=dict(_params(c), smooth_variant=s.tuned_smoother(c["precision"])[0]))
        # the step's data, computed on the GPU where the solver reads them
        st["ls"], st["rhs"] = _elbow_fields(c, tb, seed + 1, where)
        st["sol"] = torch.zeros_like(st["rhs"]).reshape(-1)
        return st
    tb, vol, area, bface, rhs, g = _fields(c, seed)
    s = sg.MacSolver(tb)
    s.set_bc(_bc(tb, 2 * c["dim"] - 1))
    s.set_ib_frac_compact(_host(vol), [_host(a) for a in area])
    for d in range(c["dim"]):
        s.set_coef_b(d, _host(bface[d]))
    s.set_params(**_params(c))
    st = dict(kind=c["kind"], solver=s, host=c["host"])
    if c["kind"] == "project":
        st["u"] = [_host(u) for u in _velocity(c, tb, area, g)]
        st["dt"] = 1e-3
    elif c["host"]:
        st["rhs"] = _grown(rhs, tb)
        st["sol"] = torch.zeros_like(st["rhs"]).pin_memory()
    else:
        st["rhs"] = rhs.reshape(-1)
        st["sol"] = torch.zeros_like(st["rhs"])
    torch.cuda.synchronize()
    s.prepare()
    return st


def _velocity(c, tb, area, g):
    """face velocities of a smooth flow, zero on closed faces"""
    nd = tb["ndim"]
    k = (1.0 + 3.0 * torch.rand(nd, 3, generator=g, dtype=torch.float64)).cuda()
    out = []
    for d in range(nd):
        p = _points(tb, [0.0 if q == d else 0.5 for q in range(nd)], tuple(int(q == d) for q in range(3)))
        u = torch.ones(p.shape[:2], dtype=torch.float64, device="cuda")
        for q in range(nd):
            u = u * torch.sin(math.pi * k[d, q] * p[..., q] + q + d)
        out.append(u * (area[d] > 0))
    return out


# ---- one pass --------------------------------------------------------------
def _solution(s, out):
    """the solution into device memory"""
    if s.lib.sayaka_mac_get_sol_compact(s.h, ctypes.c_void_p(out.data_ptr()), 1) != sg.OK:
        raise RuntimeError("get_sol failed")
    return out


def run(state):
    s, kind = state["solver"], state["kind"]
    if kind == "project":
        u = [a.copy() for a in state["u"]]
        s.set_rhs_div(u, -1.0 / state["dt"])
        s.set_zero_sol()
        info = s.cg_solve()
        for d, a in enumerate(u):
            s.correct_vel(d, state["dt"], a)
        return {"p": s.get_sol_compact(), "u": u, "status": info["status"]}
    if kind == "regrid":
        old, s = s, sg.MacSolver(state["tables"])
        s.set_bc(state["bc"])
        s.set_ib_frac_by_ls_device(state["ls"].data_ptr(), ngrow=1)
        s.set_params(**state["params"])
        s.init_from(old, prolong="centered_linear")
        s.set_rhs_device(state["rhs"].data_ptr())
        info = s.cg_solve()
        return {"p": _solution(s, state["sol"]), "status": info["status"]}
    if kind == "step":
        s.set_ib_frac_by_ls_device(state["ls"].data_ptr(), ngrow=1)
        s.set_rhs_device(state["rhs"].data_ptr())
        s.set_zero_sol()
        info = s.cg_solve()
        return {"p": _solution(s, state["sol"]), "status": info["status"]}
    if state["host"]:
        s.set_rhs(state["rhs"].numpy(), ncomp=1, ngrow=1)
        s.set_zero_sol()
        info = s.cg_solve()
        s.get_sol(state["sol"].numpy(), ncomp=1, ngrow=1)
        return {"p": state["sol"], "status": info["status"]}
    s.set_rhs_device(state["rhs"].data_ptr())
    s.set_zero_sol()
    info = s.cg_solve()
    return {"p": _solution(s, state["sol"]), "status": info["status"]}


def work(case):
    c = case
    g = _geometry(c)
    tb = g[1] if c["kind"] == "regrid" else g[0]
    nd = c["dim"]
    cells = int((tb["node_type"] == 1).sum()) * c["nb"] ** nd
    if c["kind"] in ("step", "regrid"):
        per = 8 * 3  # level set and right-hand side read, solution written (regrid: the old solution too)
        per += 8 if c["kind"] == "regrid" else 0
    elif c["kind"] == "project":
        per = 8 * (2 + 4 * nd + 1)  # velocities read and written, B, areas, volumes read, solution written
    else:
        per = 8 * (2 + 2 * nd + 1)  # right-hand side, B, areas, volumes read, solution written
    # one application of the operator: the least that says whether p solves it
    return {"bytes": cells * per, "flops": cells * (4 * nd + 3)}


# ---- 64-bit solutions in plain torch ---------------------------------------
def _assemble(tb, vol, area, bface, bc):
    """The composite operator over the leaf cells, rows scaled by cell volume
    and fraction: K p = dv vf rhs.  Same-level faces T = ds/dx B a; a fine
    face at a coarser leaf T/1.5 to the coarse cell behind it, and the same
    back; the coarse cell's own diagonal takes ds/(0.75 dx) with B and a
    averaged over the fine faces; p = 0 faces 2 T.  Returns (row, column,
    value, diagonal, scale, leaf-cell number of every cell)."""
    dev = "cuda"
    nd, nb, n = tb["ndim"], tb["nb"], tb["num_blocks"]
    nc = nb ** nd
    T_ = lambda a: torch.as_tensor(np.ascontiguousarray(a), device=dev).long()  # noqa: E731
    nbr, child, parent = T_(tb["neighbor"]).reshape(n, 6), T_(tb["child"]).reshape(n, 8), T_(tb["parent"])
    which, leaf = T_(tb["which_child"]), torch.as_tensor(tb["node_type"] == 1, device=dev)
    bct = T_(bc).reshape(n, 6)
    dx = torch.as_tensor(tb["block_len"].reshape(n, 3)[:, :nd] / nb, device=dev)
    dv = dx.prod(1)
    L = torch.nonzero(leaf).reshape(-1)
    uid = torch.full((n, nc), -1, dtype=torch.int64, device=dev)
    uid[L] = torch.arange(len(L) * nc, device=dev).reshape(len(L), nc)
    fluid = vol > 0
    ijk = torch.stack([(torch.arange(nc, device=dev) // nb ** q) % nb for q in range(nd)])
    enc = lambda v: sum(v[q] * nb ** q for q in range(nd))  # noqa: E731

    def face(d, v, s):  # index of face s of cell v in direction d
        out, stride = 0, 1
        for q in range(nd):
            out = out + (v[q] + (s if q == d else 0)) * stride
            stride *= nb + (q == d)
        return out
    diag = torch.zeros(len(L) * nc, dtype=torch.float64, device=dev)
    rows, cols, vals = [], [], []

    def link(r, cidx, v):
        rows.append(r.reshape(-1)), cols.append(cidx.reshape(-1)), vals.append(v.reshape(-1))

    def onto(r, v):
        diag.index_add_(0, r.reshape(-1), v.reshape(-1))
    half = nb // 2
    for d in range(nd):
        k = dv[:, None] / (dx[:, d] ** 2)[:, None]
        T = k * bface[d] * area[d]
        for s in (0, 1):
            f = 2 * d + s
            inner = torch.nonzero(ijk[d] != (nb - 1 if s else 0)).reshape(-1)
            edge = torch.nonzero(ijk[d] == (nb - 1 if s else 0)).reshape(-1)
            tf = T[L][:, face(d, ijk[:, inner], s)]
            link(uid[L][:, inner], uid[L][:, inner + (nb ** d if s else -nb ** d)], tf)
            onto(uid[L][:, inner], tf)
            ev = ijk[:, edge]
            fx = face(d, ev, s)
            nb_f = nbr[L, f]
            mirror = [ev[q].clone() for q in range(nd)]
            mirror[d] = torch.full_like(ev[d], 0 if s else nb - 1)
            there = nb_f >= 0
            same = there & leaf[nb_f.clamp(min=0)]
            S = L[same]
            link(uid[S][:, edge], uid[nb_f[same]][:, enc(mirror)], T[S][:, fx])
            onto(uid[S][:, edge], T[S][:, fx])
            # a coarser leaf behind the face
            fine = L[nb_f == -1]
            if len(fine):
                C = nbr[parent[fine], f]
                cc = [((which[fine] >> q) & 1)[:, None] * half + (ev[q] // 2)[None] if q != d
                      else torch.full((len(fine), len(edge)), 0 if s else nb - 1, device=dev) for q in range(nd)]
                v = T[fine][:, fx] / 1.5
                r, q_ = uid[fine][:, edge], uid[C[:, None], enc(cc)]
                link(r, q_, v)
                onto(r, v)
                link(q_, r, v)
            # finer blocks behind the face: the coarse cell's own diagonal
            crs = L[there & ~same]
            if len(crs):
                up = [(ev[q] >= half).long() for q in range(nd)]
                ck = (1 - s) << d
                for q in range(nd):
                    if q != d:
                        ck = ck + (up[q] << q)
                F = child[nbr[crs, f]][:, ck]
                bm = am = 0.0
                for a in range(2 ** (nd - 1)):
                    v, j = [], 0
                    for q in range(nd):
                        if q == d:
                            v.append(torch.full_like(ev[q], 0 if s else nb - 1))
                        else:
                            v.append(2 * (ev[q] - up[q] * half) + ((a >> j) & 1))
                            j += 1
                    ff = face(d, v, 1 - s)
                    bm = bm + bface[d][F, ff]
                    am = am + area[d][F, ff]
                m = 0.5 ** (nd - 1)
                onto(uid[crs][:, edge], k[crs] / 0.75 * (bm * m) * (am * m))
            wall = nb_f <= sg.PHYS_BNDRY
            zero = wall & (bct[L, f] == sg.DIRICHLET)
            onto(uid[L[zero]][:, edge], 2.0 * T[L[zero]][:, fx])
    row, col, val = torch.cat(rows), torch.cat(cols), torch.cat(vals)
    scale = (dv[:, None] * vol)[L].reshape(-1)
    solid = ~fluid[L].reshape(-1)
    keep = (val != 0) & ~solid[row] & ~solid[col]
    diag = torch.where(solid, torch.ones_like(diag), diag)
    return row[keep], col[keep], val[keep], diag, torch.where(solid, torch.zeros_like(scale), scale), uid


def _solve64(row, col, val, diag, b):
    """K x = b by conjugate gradients (diagonal preconditioner) with iterative
    refinement"""
    n = len(diag)
    i = torch.arange(n, device=b.device)
    K = torch.sparse_coo_tensor(torch.stack([torch.cat([row, i]), torch.cat([col, i])]), torch.cat([-val, diag]),
                                (n, n)).coalesce().to_sparse_csr()
    x = torch.zeros_like(b)
    r = b.clone()
    b0 = float(b.norm())
    for _ in range(4):
        if float(r.norm()) < 1e-14 * b0:
            break
        d, res, stop = torch.zeros_like(b), r.clone(), 1e-9 * float((r * r / diag).sum().sqrt())
        z = res / diag
        p, rz = z.clone(), (res * z).sum()
        for k in range(20000):
            q = K @ p
            a = rz / (p * q).sum()
            d += a * p
            res -= a * q
            z = res / diag
            new = (res * z).sum()
            p = z + (new / rz) * p
            rz = new
            if k % 100 == 99 and not float(rz) > stop * stop:
                break
        x += d
        r = b - K @ x
    return x


def exact(case, seed):
    c = case
    if c["kind"] == "regrid":
        return None
    if work(c)["flops"] / (4 * c["dim"] + 3) > EXACT_CELLS:
        return None
    if c["kind"] == "step":
        tb = _geometry(c)[0]
        ls, rhs = _elbow_fields(c, tb, seed + 1, c["position"] + 0.01)
        n, nb = tb["num_blocks"], tb["nb"]
        wet = (ls > 0).reshape(n, nb + 2, nb + 2, nb + 2)
        mid = slice(1, nb + 1)
        vol = wet[:, mid, mid, mid].double().reshape(n, -1)
        area, bface = [], []
        for d in range(3):
            w = wet.narrow(3 - d, 0, nb + 1) & wet.narrow(3 - d, 1, nb + 1)
            w = w[tuple([slice(None)] + [slice(None) if q == d else mid for q in (2, 1, 0)])]
            area.append(w.double().reshape(n, -1))
            bface.append(torch.ones_like(area[d]))
        bc = _bc(tb, 0)
    else:
        tb, vol, area, bface, rhs, g = _fields(c, seed)
        bc = _bc(tb, 2 * c["dim"] - 1)
        if c["kind"] == "project":
            u = _velocity(c, tb, area, g)
            nd, nb, n = tb["ndim"], tb["nb"], tb["num_blocks"]
            dx = torch.as_tensor(tb["block_len"].reshape(n, 3)[:, :nd] / nb, device="cuda")
            rhs = torch.zeros_like(vol)
            for d in range(nd):
                v = u[d].reshape([n] + [nb + (q == d) for q in range(nd)][::-1])
                rhs += -1.0 / 1e-3 / dx[:, d:d + 1] * (v.narrow(nd - d, 1, nb) - v.narrow(nd - d, 0, nb)).reshape(n, -1)
    row, col, val, diag, scale, uid = _assemble(tb, vol, area, bface, bc)
    leaf = uid >= 0
    x = _solve64(row, col, val, diag, scale * rhs[leaf])
    p = torch.zeros_like(rhs)
    p[leaf] = x
    if c["kind"] == "project":
        return {"p": p.reshape(-1), "u": [None] * c["dim"], "status": None}
    if c.get("host"):
        return {"p": _grown(p, tb), "status": None}
    return {"p": p.reshape(-1), "status": None}
