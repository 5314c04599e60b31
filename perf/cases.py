"""What this framework is used for, as cases that can be timed and checked.

Every case goes through the public entry points (``Instance``, ``Batch``,
``Server`` and the C ABI's allocation-free update). The meshes and materials
are the repository's own: the 200 mm hole plate and the thick ring of the
benchmark's configurations and of ``cudaplasticity_b200.workload``, as 4-node
quads, triangles or 8-node quads, from 2 k DOF (the smallest request of the
batch stream) to 2.1 M DOF (configuration 2).

Kinds of cases:

* ``solve``  -- an instance that a program keeps; one pass sets the loads,
  resets the state, runs the whole elasto-plastic solve and reads the result.
  Tolerances are those of the parity tests, so that the result is determined
  to well below 1e-9 whatever the order of the sums. Above 40 k DOF, where
  such a solve takes many seconds, a pass is a few of its outer steps: from
  the displacements of a neighbouring state, with capped iterations
  (``max_cg``, ``max_outer``).
* ``update`` -- the secant update (strain, stress, diagram, exit norm) on
  device buffers that the caller owns.
* ``batch``  -- uneven instances solved together in mixed precision.
* ``serve``  -- a burst of uneven FP64 requests through the solve service,
  from host arrays to host results.

``exact`` restates a case in torch with dense FP64 factorisations.
"""
import ctypes
import math
import time

import numpy as np
import torch

import cudaplasticity_b200 as cp
from cudaplasticity_b200 import _capi

E_MPA, NU = 210000.0, 0.3
READ = ("uv", "sxx", "syy", "tau", "sig_i", "eps_p_i")
READ_FEW = ("uv", "sig_i", "eps_p_i")
READ_MANY = ("uv", "sig_i")  # per instance of a batch or a burst
#: the options of the benchmark's headline solve at the parity tests' tolerances
FP64_KW = dict(cg_tol=1e-13, outer_tol=1e-11, max_outer=2000, max_cg=2_000_000, aitken=1, adaptive_cg=2, precond=1,
               predict=1, recycle=6)
MIXED_KW = dict(cg_tol=1e-12, outer_tol=1e-11, inner_tol=1e-3, max_outer=2000, max_cg=2_000_000, aitken=1,
                adaptive_cg=1, precond=1, predict=1)
EXACT_DOF = 9000  # the largest problem that exact() factorises densely


def listed():
    solve = dict(kind="solve", elem="q4", diagram="linear", levels=1, precision="fp64", cap_cg=0, cap_outer=0)
    return [
        # the update alone, called on every outer step by a program with its own linear solver: configuration 1's
        # mesh (the smallest call: latency) and configuration 2's (throughput, Hollomon hardening)
        dict(kind="update", name="update 4k linear", shape="plate", n_c=64, n_r=64, diagram="linear"),
        dict(kind="update", name="update 1M hollomon", shape="plate", n_c=1024, n_r=1024, diagram="hollomon"),
        # the smallest request of the batch stream
        dict(solve, name="plate 2k", shape="plate", n_c=32, n_r=31, diagram="piecewise"),
        # configuration 1, the headline: 64 x 64 O-grid, bilinear hardening, load increments
        dict(solve, name="plate 8k config1", shape="plate", n_c=64, n_r=64, levels=10),
        # the same plate in triangles
        dict(solve, name="plate 8k triangles", shape="plate", elem="t3", n_c=64, n_r=64, levels=2,
             diagram="hollomon"),
        # 8-node quads: a pressurised ring with curved edges
        dict(solve, name="ring 14k q8", shape="ring", elem="q8", n_c=48, n_r=47),
        # a middling request of the batch and served streams, ragged sizes
        dict(solve, name="ring 32k piecewise", shape="ring", n_c=132, n_r=121, diagram="piecewise"),
        # configuration 3: mixed precision on configuration 1's mesh
        dict(solve, name="plate 8k mixed", shape="plate", n_c=64, n_r=64, levels=2, precision="mixed"),
        # the batch stream's largest request, and configuration 2: outer steps with capped linear solves
        dict(solve, name="plate 200k capped", shape="plate", n_c=316, n_r=315, diagram="piecewise", cap_cg=200,
             cap_outer=3),
        dict(solve, name="plate 2.1M config2 capped", shape="plate", n_c=1024, n_r=1024, diagram="hollomon",
             cap_cg=200, cap_outer=2),
        # uneven instances together (configuration 4's form) and a burst of requests (configuration 5's form)
        dict(kind="batch", name="batch 24", count=24, dof_min=2000, dof_max=16000),
        dict(kind="serve", name="serve 8", count=8, dof_min=2000, dof_max=30000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _grid(dof, rng):
    """An uneven O-grid or ring of about dof unknowns (4-node elements)."""
    n_c = max(8, 4 * int(round(math.sqrt(dof / 2.0) * rng.uniform(0.8, 1.25) / 4.0)))
    return n_c, max(4, int(round(dof / 2.0 / n_c)) - 1)


def draw(rng):
    kind = rng.choice(["update", "solve", "solve", "solve", "mixed", "capped", "batch", "serve"])
    diagram = rng.choice(["linear", "hollomon", "piecewise"])
    if kind == "update":
        n_c, n_r = _grid(_log_int(rng, 2000, 1_900_000), rng)
        return dict(kind="update", shape="plate", n_c=n_c, n_r=n_r, diagram=diagram)
    if kind == "batch":
        return dict(kind="batch", count=rng.randint(4, 24), dof_min=2000, dof_max=_log_int(rng, 5000, 16000))
    if kind == "serve":
        return dict(kind="serve", count=rng.randint(2, 8), dof_min=2000, dof_max=_log_int(rng, 6000, 30000))
    elem, precision, cap_cg, cap_outer, levels = "q4", "fp64", 0, 0, rng.randint(1, 2)
    if kind == "solve":
        elem = rng.choice(["q4", "q4", "t3", "q8"])
        dof = _log_int(rng, 2000, 14000 if elem == "q8" else 32000)
    elif kind == "mixed":
        dof, precision, levels = _log_int(rng, 2000, 9000), "mixed", rng.randint(1, 2)
    else:
        dof, cap_cg, cap_outer, levels = _log_int(rng, 40000, 1_900_000), rng.randint(100, 200), 2, 1
    shape = rng.choice(["plate", "ring"])
    n_c, n_r = _grid(dof / (3.0 if elem == "q8" else 1.0), rng)
    return dict(kind="solve", shape=shape, elem=elem, n_c=n_c, n_r=n_r, diagram=diagram, levels=levels,
                precision=precision, cap_cg=cap_cg, cap_outer=cap_outer)


# ------------------------------------------------------------------- inputs --

def _material(diagram, rng):
    sy = 250.0 * rng.uniform(0.95, 1.05)
    if diagram == "linear":
        p = dict(diagram="linear", sigma_t=sy, k_t=2000.0)
    elif diagram == "hollomon":
        p = dict(diagram="hollomon", sigma_y=sy, eps0=0.002, n=0.2)
    else:  # five segments with falling slopes, as in the batch stream
        pts = [(sy / E_MPA, sy)]
        for h, w in zip((20000.0, 8000.0, 3000.0, 1200.0, 500.0), rng.uniform(0.5e-3, 2e-3, size=5)):
            pts.append((pts[-1][0] + w, pts[-1][1] + h * w))
        p = dict(diagram="piecewise", points=pts)
    return sy, p


def _problem(c, rng):
    """Mesh arrays, material parameters and loads of one plate or ring. The loads take it well past first yield
    and well below the limit load."""
    sy, mat = _material(c["diagram"], rng)
    elem = c.get("elem", "q4")
    order = 2 if elem == "q8" else 1
    L = cp.Loads()
    if c["shape"] == "plate":
        n1 = c["n_c"] // 4
        mesh = cp.Mesh.rect_with_hole(-100.0, 100.0, -100.0, 100.0, 20.0, n1, n1, rad_n=c["n_r"], order=order)
        L.set_force(2, 0.0, sy * rng.uniform(0.6, 0.7)).fix_border_hor(0).fix_point(-100.0, -100.0)
    else:
        b = rng.uniform(95.0, 120.0)
        mesh = cp.Mesh.ring(50.0, b, c["n_c"], c["n_r"], order=order)
        onset = sy * (1.0 - 2500.0 / (b * b)) / math.sqrt(3.0)
        L.set_force(0, onset * rng.uniform(1.15, 1.25), 0.0, True)
        xy = mesh.arrays()["node_xy"]
        r = np.hypot(xy[:, 0], xy[:, 1])
        for axis, dof in ((1, 1), (0, 0)):  # symmetry: no displacement across the axes
            for nd in np.where(np.abs(xy[:, axis]) <= 1e-9 * r)[0]:
                L.fix_dof(2 * int(nd) + dof)
    if elem == "t3":
        mesh.split_t3()
    rp, mask, uv = L.build(mesh, h=1.0)
    a = mesh.arrays()
    if c.get("cap_cg"):  # the free displacements start from a neighbouring state
        x, y = a["node_xy"][:, 0], a["node_xy"][:, 1]
        if c["shape"] == "plate":
            start = _tension(x, y, sy / E_MPA * rng.uniform(0.7, 0.9))
        else:
            k = onset / E_MPA * rng.uniform(1.1, 1.3) * 2500.0 / (b * b - 2500.0)
            s = k * ((1.0 - NU) + (1.0 + NU) * b * b / (x * x + y * y))
            start = np.stack([s * x, s * y], axis=1).ravel()
        uv = np.where(mask.astype(bool), start, uv)
    return dict(mesh=a, mat=mat, rp=rp, mask=mask, uv=uv)


def _tension(x, y, eps):
    """Displacements of a tension test in y with strain eps far from the hole and its concentration at the hole."""
    r2 = x * x + y * y
    q = 400.0 / r2
    return np.stack([-NU * eps * x * (1.0 + 1.5 * q), eps * y * (1.0 + 2.0 * q * x * x / r2)], axis=1).ravel()


def _many(c, rng):
    """The problems of a batch or a burst: plates and rings in turn, sizes spread evenly over the logarithm of the
    range, small and large ones mixed."""
    out = []
    for i in range(c["count"]):
        at = ((i * 7) % c["count"] if c["count"] % 7 else i) + 0.5
        n = math.sqrt(0.5 * c["dof_min"] * (c["dof_max"] / c["dof_min"]) ** (at / c["count"]))
        n_c = max(8, 4 * int(round(n / 4.0)))
        out.append(_problem(dict(shape="plate" if i % 2 == 0 else "ring", n_c=n_c,
                                 n_r=max(4, int(round(n * n / n_c)) - 1), diagram="piecewise"), rng))
    return out


def _update_inputs(c, rng):
    """The plate and the displacements of a tension test in it: a uniform strain plus the hole's concentration,
    with strains on both sides of first yield."""
    sy, mat = _material(c["diagram"], rng)
    n1 = c["n_c"] // 4
    mesh = cp.Mesh.rect_with_hole(-100.0, 100.0, -100.0, 100.0, 20.0, n1, n1, rad_n=c["n_r"])
    a = mesh.arrays()
    u = _tension(a["node_xy"][:, 0], a["node_xy"][:, 1], sy / E_MPA * rng.uniform(0.7, 0.9))
    return a, mat, np.ascontiguousarray(u)


_KEPT = {}


def _context():
    if "ctx" not in _KEPT:
        _KEPT["ctx"] = cp.Context(0)
    return _KEPT["ctx"]


def _server():
    if "server" not in _KEPT:
        _KEPT["server"] = cp.Server(0)
    return _KEPT["server"]


def _cp_material(p):
    return cp.material(E_MPA, NU, h=1.0, **p)


def _options(c):
    if c["precision"] == "mixed":
        return dict(MIXED_KW, precision=cp.CP_PREC_MIXED, levels=c["levels"])
    kw = dict(FP64_KW, precision=cp.CP_PREC_FP64, levels=c["levels"])
    if c["cap_cg"]:
        kw.update(max_cg=c["cap_cg"], max_outer=c["cap_outer"], adaptive_cg=0)
    return kw


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    c = dict(case)
    if c["kind"] == "update":
        a, mat, u = _update_inputs(c, rng)
        ne, dev = a["elem4"].shape[0], "cuda"
        t = lambda v, dt: torch.from_numpy(np.ascontiguousarray(v).ravel()).to(dev, dt)  # noqa: E731
        full = lambda v: torch.full((ne,), v, dtype=torch.float64, device=dev)  # noqa: E731
        return dict(case=c, mat=_cp_material(mat), xy=t(a["node_xy"], torch.float64), e4=t(a["elem4"], torch.int32),
                    u=t(u, torch.float64), E_c=full(E_MPA), nu_c=full(NU), psi=full(1.0),
                    fields=torch.zeros(9, ne, dtype=torch.float64, device=dev), ne=ne, nn=a["node_xy"].shape[0])
    if c["kind"] == "solve":
        p = _problem(c, rng)
        inst = cp.Instance(_context(), p["mesh"], _cp_material(p["mat"]))
        return dict(case=c, inst=inst, rp=p["rp"], mask=p["mask"], uv=p["uv"], options=_options(c))
    problems = _many(c, rng)
    if c["kind"] == "serve":
        return dict(case=c, server=_server(), problems=problems, mats=[_cp_material(p["mat"]) for p in problems])
    ctx = _context()
    insts = [cp.Instance(ctx, p["mesh"], _cp_material(p["mat"])) for p in problems]
    return dict(case=c, batch=cp.Batch(ctx, max_instances=c["count"]), insts=insts, problems=problems)


# --------------------------------------------------------------------- pass --

def _read(inst, names=READ):
    return {k: inst.field(k) for k in names}


def run(state):
    c = state["case"]
    if c["kind"] == "update":
        err = ctypes.c_double()
        s = state
        st = _capi.lib().cp_secant_update_noalloc(
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(s["mat"]), s["nn"],
            s["xy"].data_ptr(), s["ne"], s["e4"].data_ptr(), s["u"].data_ptr(), s["E_c"].data_ptr(),
            s["nu_c"].data_ptr(), s["psi"].data_ptr(), s["fields"].data_ptr(), ctypes.byref(err))
        if st != 0:
            raise cp.CuplastError(st)
        return dict(fields=s["fields"], E_c=s["E_c"], nu_c=s["nu_c"], psi=s["psi"], rel_err=err.value)
    if c["kind"] == "solve":
        inst = state["inst"]
        inst.set_loads(state["rp"], state["mask"], state["uv"])
        inst.reset_state()
        inst.solve(allow_not_converged=c["cap_cg"] > 0, **state["options"])
        return _read(inst, READ_FEW if c["cap_cg"] else READ)
    if c["kind"] == "serve":
        kw = dict(FP64_KW, precision=cp.CP_PREC_FP64)
        ids = [state["server"].submit(p["mesh"], m, p["rp"], p["mask"], p["uv"], **kw)
               for p, m in zip(state["problems"], state["mats"])]
        out = []
        for rid in ids:
            inst, rep, _ = state["server"].wait(rid)
            if rep["status"] != 0:
                raise cp.CuplastError(rep["status"])
            out.append(_read(inst, READ_MANY))
            inst.close()
        return out
    slots = {}
    for inst, p in zip(state["insts"], state["problems"]):
        inst.set_loads(p["rp"], p["mask"], p["uv"])
        inst.reset_state()
        slots[state["batch"].add(inst, **MIXED_KW)] = inst
    state["batch"].run()
    for slot, inst, rep in state["batch"].harvest():
        if rep["status"] != 0 or slots[slot] is not inst:
            raise cp.CuplastError(rep["status"])
    return [_read(inst, READ_MANY) for inst in state["insts"]]


# --------------------------------------------------------------------- work --

def _sizes(c):
    """Nodes, elements and 2 x 2 blocks of K of a plate or ring."""
    q8 = c.get("elem") == "q8"
    ring = c["n_c"] * (c["n_r"] + 1)
    ne = c["n_c"] * c["n_r"] * (2 if c.get("elem") == "t3" else 1)
    if q8:
        return ring + c["n_c"] * (2 * c["n_r"] + 1), ne, 21 * ring + 13 * 2 * ring
    return ring, ne, (7 if c.get("elem") == "t3" else 9) * ring


def _solve_bytes(n, ne, blocks, iters, read):
    """A pass reads the mesh and loads and writes the results, and every CG iteration reads K and the vectors of a
    preconditioned CG (x, r, p read and written, K p written and read, M read)."""
    return n * (16 + 16 + 16 + 2) + ne * 16 + n * 16 + ne * 8 * (read - 1) + iters * (36.0 * blocks + n * 160.0)


def work(case):
    c = case
    if c["kind"] == "update":
        n, ne, _ = _sizes(c)
        # coordinates, displacements, connectivity, E_c, nu_c read; nine fields, E_c, nu_c, psi written
        return dict(bytes=n * 32.0 + ne * (16 + 16 + 12 * 8), flops=ne * 150.0)
    if c["kind"] == "solve":
        n, ne, blocks = _sizes(c)
        # about sqrt(DOF) iterations per linear solve, and a few outer steps per load level at the very least
        iters = c["cap_cg"] * c["cap_outer"] if c["cap_cg"] else c["levels"] * 5 * math.sqrt(2 * n)
        return dict(bytes=_solve_bytes(n, ne, blocks, iters, 3 if c["cap_cg"] else 6), flops=iters * (8.0 * blocks + 30.0 * n))
    dof = (c["dof_max"] - c["dof_min"]) / math.log(c["dof_max"] / c["dof_min"]) * c["count"]
    n = dof / 2.0
    iters = 5 * math.sqrt(dof / c["count"])
    return dict(bytes=_solve_bytes(n, n, 9 * n, iters, 2), flops=iters * 102.0 * n)


# -------------------------------------------------------------------- exact --

def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f64(v):
    return torch.as_tensor(np.ascontiguousarray(v), dtype=torch.float64, device=_device())


def _shape(kind, r, s):
    """dN/dr and dN/ds of the 4- and 8-node quads at (r, s)."""
    ri, si = [1.0, -1.0, -1.0, 1.0], [1.0, 1.0, -1.0, -1.0]
    if kind == 4:
        return ([0.25 * a * (1 + b * s) for a, b in zip(ri, si)], [0.25 * b * (1 + a * r) for a, b in zip(ri, si)])
    dr = [0.25 * a * (1 + s * b) * (2 * r * a + s * b) for a, b in zip(ri, si)]
    ds = [0.25 * b * (1 + r * a) * (r * a + 2 * s * b) for a, b in zip(ri, si)]
    dr += [-r * (1 + s), -0.5 * (1 - s * s), -r * (1 - s), 0.5 * (1 - s * s)]
    ds += [0.5 * (1 - r * r), -s * (1 - r), -0.5 * (1 - r * r), -s * (1 + r)]
    return dr, ds


def _gradients(mesh):
    """Per element group: nodes (ne, k), shape gradients (points, ne, k) in x and y, and the stiffness and mean-strain
    weights (points, ne)."""
    xy, out = _f64(mesh["node_xy"]), []
    e3, e4, e8 = (mesh.get(k) for k in ("elem3", "elem4", "elem8"))
    if e3 is not None and len(e3):
        nd = torch.as_tensor(e3, dtype=torch.int64, device=_device())
        x, y = xy[nd, 0], xy[nd, 1]
        a2 = (x[:, 1] - x[:, 0]) * (y[:, 2] - y[:, 0]) - (x[:, 2] - x[:, 0]) * (y[:, 1] - y[:, 0])
        bx = torch.stack([y[:, 1] - y[:, 2], y[:, 2] - y[:, 0], y[:, 0] - y[:, 1]], 1) / a2[:, None]
        by = torch.stack([x[:, 2] - x[:, 1], x[:, 0] - x[:, 2], x[:, 1] - x[:, 0]], 1) / a2[:, None]
        out.append((nd, bx[None], by[None], (0.5 * a2)[None], torch.ones_like(a2)[None]))
    for el, kind in ((e4, 4), (e8, 8)):
        if el is None or not len(el):
            continue
        nd = torch.as_tensor(el, dtype=torch.int64, device=_device())
        x, y = xy[nd, 0], xy[nd, 1]
        g = math.sqrt(0.6)
        pts = [(-0.577350269189626, 1.0), (0.577350269189626, 1.0)] if kind == 4 else \
            [(-g, 5 / 9), (0.0, 8 / 9), (g, 5 / 9)]
        bxs, bys, ws, ms = [], [], [], []
        for r, wr in pts:
            for s, ws_ in pts:
                dr, ds = (torch.tensor(v, dtype=torch.float64, device=_device()) for v in _shape(kind, r, s))
                xr, yr, xs, ys = x @ dr, y @ dr, x @ ds, y @ ds
                det = xr * ys - yr * xs
                bxs.append((dr * ys[:, None] - ds * yr[:, None]) / det[:, None])
                bys.append((ds * xr[:, None] - dr * xs[:, None]) / det[:, None])
                ws.append(det * (wr * ws_))
                ms.append(torch.full_like(det, wr * ws_ / 4.0))
        out.append((nd, torch.stack(bxs), torch.stack(bys), torch.stack(ws), torch.stack(ms)))
    return out


def _curve(mat, eps):
    """The hardening diagram sigma = f(eps)."""
    if mat["diagram"] == "linear":
        et = mat["sigma_t"] / E_MPA
        return torch.where(eps < et, eps * E_MPA, mat["sigma_t"] + (eps - et) * mat["k_t"])
    if mat["diagram"] == "hollomon":
        sy, e0, n = mat["sigma_y"], mat["eps0"], mat["n"]
        s = torch.full_like(eps, sy)
        for _ in range(60):
            t = (s / sy) ** (1.0 / n)
            s = s - (s / E_MPA + e0 * (t - 1.0) - eps) / (1.0 / E_MPA + e0 * t / (n * s))
        return torch.where(eps < sy / E_MPA, eps * E_MPA, s)
    pts = mat["points"]
    out = eps * E_MPA
    for k in range(len(pts) - 1):
        slope = (pts[k + 1][1] - pts[k][1]) / (pts[k + 1][0] - pts[k][0])
        out = torch.where(eps >= pts[k][0], pts[k][1] + (eps - pts[k][0]) * slope, out)
    return out


def _strain(groups, u):
    """Element-mean strains."""
    u = u.reshape(-1, 2)
    parts = []
    for nd, bx, by, _, m in groups:
        ux, uy = u[nd, 0], u[nd, 1]
        ex, ey = (bx * ux).sum(-1), (by * uy).sum(-1)
        g = (by * ux).sum(-1) + (bx * uy).sum(-1)
        parts.append(torch.stack([(ex * m).sum(0), (ey * m).sum(0), (g * m).sum(0)]))
    return torch.cat(parts, 1)


def _stress(eps, E, nu):
    """Plane-stress stresses and the stress intensity."""
    c = E / (1 - nu * nu)
    sx, sy, t = c * (eps[0] + nu * eps[1]), c * (nu * eps[0] + eps[1]), c * (1 - nu) * 0.5 * eps[2]
    return sx, sy, t, torch.sqrt(0.5 * (sx * sx + sy * sy + (sx - sy) ** 2 + 6 * t * t))


def _stiffness(groups, n, E, nu):
    """Dense K."""
    K = torch.zeros(4 * n * n, dtype=torch.float64, device=_device())
    e0 = 0
    for nd, bx, by, w, _ in groups:
        ne, k = nd.shape
        Ee, ve = E[e0:e0 + ne], nu[e0:e0 + ne]
        e0 += ne
        c = Ee / (1 - ve * ve)
        xx, yy, xy = (torch.einsum("ge,gei,gej->eij", w, a, b) for a, b in ((bx, bx), (by, by), (bx, by)))
        yx = xy.transpose(1, 2)
        c0, c1, c2 = (v[:, None, None] for v in (c, c * ve, c * (1 - ve) * 0.5))
        blocks = ((0, 0, c0 * xx + c2 * yy), (0, 1, c1 * xy + c2 * yx), (1, 0, c1 * yx + c2 * xy),
                  (1, 1, c0 * yy + c2 * xx))
        for a, b, v in blocks:
            at = (2 * nd[:, :, None] + a) * (2 * n) + 2 * nd[:, None, :] + b
            K.index_add_(0, at.reshape(-1), v.reshape(-1))
    return K.reshape(2 * n, 2 * n)


def _fixed_point(p, limit_s):
    """The converged state: the secant iteration on E / psi with Aitken's relaxation, each linear system factorised."""
    n = p["mesh"]["node_xy"].shape[0]
    groups, mat = _gradients(p["mesh"]), p["mat"]
    free = torch.as_tensor(np.flatnonzero(p["mask"]), device=_device())
    b, u = _f64(p["rp"]), _f64(p["uv"]).clone()
    ne = sum(g[0].shape[0] for g in groups)
    psi = torch.ones(ne, dtype=torch.float64, device=_device())
    held, omega, best, began = None, 1.0, math.inf, time.monotonic()
    for it in range(600):
        E, nu = E_MPA / psi, 0.5 * (1 - (1 - 2 * NU) / psi)
        K = _stiffness(groups, n, E, nu)
        Kf = K.index_select(0, free).index_select(1, free)
        C = torch.linalg.cholesky(Kf)
        for _ in range(3):  # iterative refinement
            r = (b - K @ u).index_select(0, free)
            u[free] += torch.cholesky_solve(r[:, None], C)[:, 0]
        eps = _strain(groups, u)
        sx, sy, t, si = _stress(eps, E, nu)
        ei = si / E
        tab = _curve(mat, ei)
        rel = float((si - tab).norm() / tab.norm())
        if rel < 2e-14 or (rel < 1e-12 and rel > 0.9 * best):
            break
        best = min(best, rel)
        if time.monotonic() - began > limit_s:
            return None
        res = E_MPA * ei / tab - psi
        if held is not None:
            d = res - held
            omega = min(10.0, max(0.1, -omega * float(held @ d) / max(float(d @ d), 1e-300)))
        held = res
        psi = torch.clamp(psi + omega * res, min=1.0)
    ps = E_MPA * ei / tab
    Ec, nc = E_MPA / ps, 0.5 * (1 - (1 - 2 * NU) / ps)
    xp, yp = (1 / Ec - 1 / E_MPA) * sx, (1 / Ec - 1 / E_MPA) * sy
    gp = (2 * (1 + nc) / Ec - 2 * (1 + NU) / E_MPA) * t
    ep = math.sqrt(2.0) / 3.0 * torch.sqrt((xp - yp) ** 2 + 6 * gp * gp)
    return {k: v.cpu().numpy() for k, v in zip(READ, (u, sx, sy, t, si, ep))}


def exact(case, seed):
    rng = np.random.default_rng(seed)
    c = dict(case)
    if c["kind"] == "update":
        a, mat, u = _update_inputs(c, rng)
        eps = _strain(_gradients(a), _f64(u))
        one = torch.ones_like(eps[0])
        sx, sy, t, si = _stress(eps, E_MPA * one, NU * one)
        ei = si / E_MPA
        tab = _curve(mat, ei)
        psi = E_MPA * ei / tab
        return dict(fields=torch.stack([eps[0], eps[1], eps[2], ei, sx, sy, t, si, tab]), E_c=E_MPA / psi,
                    nu_c=0.5 * (1 - (1 - 2 * NU) / psi), psi=psi, rel_err=float((si - tab).norm() / tab.norm()))
    if c["kind"] == "solve":
        if c["cap_cg"] or 2 * _sizes(c)[0] > EXACT_DOF:
            return None
        return _fixed_point(_problem(c, rng), 15.0)
    out, began = [], time.monotonic()
    for p in _many(c, rng):
        small = p["rp"].size <= 5000 and time.monotonic() - began < 12.0
        f = _fixed_point(p, 4.0) if small else None
        out.append({k: f[k] if f else None for k in READ_MANY})
    return out
