"""The work this package is used for, as measurable cases.

A case is one call sequence that a user's program makes through the public
entry points (ns3d_gb300, include/ns3d_capi.h): a permeability request on one
voxel image (open, solve, read the fields, close), a pressure-drop sweep on a
handle that is kept, a batch or a served stream of images, or one linear
system through the allocation-free entry point.  Images are seeded packs of
spheres or fibres rasterised by ns3d_generate_image, as in
ns3d_gb300/workloads.py.

Outer loops are capped (`outer`) where a converged solve would take minutes:
every outer iteration does the same work, so the cap changes how often it is
repeated and nothing else.

  listed()           the cases
  draw(rng)          one more case of the same ranges
  prepare(case, s)   inputs of seed s and the handles a program keeps
  run(state)         one pass; returns every output whole
  work(case)         bytes and operations the path cannot do without
  exact(case, s)     the outputs in 64 bits by plain torch, where they have
                     such a value
"""
import ctypes as C

import numpy as np
import torch

import ns3d_gb300
from ns3d_gb300 import capi, synth

DX = 1e-6
# linear-solver and outer-loop settings
TIGHT = dict(alpha=0.8, vsolvertol=1e-8, psolvertol=1e-8, pcsolvertol=1e-8, simpletol=1e-4,
             maxitsolver=2000)  # the serving stream's
LOOSE = dict(alpha=0.8, vsolvertol=1e-5, psolvertol=1e-6, pcsolvertol=1e-3, simpletol=1e-4,
             maxitsolver=500)   # the reference's compare_algorithms.ini
PRECISION = {"fp64": 0, "mixed": 1, "mixed_mg": 2}


def _case(path, name=None, **kw):
    c = {"path": path}
    if name:
        c["name"] = name
    c.update(kw)
    return c


def _request(name, nx, ny, nz, kind, radius, porosity, method, precision, outer, numerics="tight", direction=1,
             border=0):
    return _case("request", name, nx=nx, ny=ny, nz=nz, kind=kind, radius=radius, porosity=porosity, method=method,
                 precision=precision, outer=outer, numerics=numerics, direction=direction, border=border)


def listed():
    return [
        # one linear system in device memory, from a host that must not
        # allocate: the smallest call, launches and barriers decide
        _case("noalloc", "noalloc_20", edge=20, porosity=0.7, tol=1e-8),
        # the smallest image anyone solves: a crop of a scan, all latency
        _request("fp64_simplec_24", 24, 20, 16, "spheres", 3, 0.6, "SIMPLEC", "fp64", 8),
        # odd box, flow along y, border of one voxel, SIMPLER with the loose
        # settings of the reference's comparison input
        _request("fp64_simpler_49x33x41", 49, 33, 41, "spheres", 4, 0.62, "SIMPLER", "fp64", 10, "loose", 2, 1),
        # the reference's published benchmark size and settings (64^3)
        _request("fp64_simplec_64_loose", 64, 64, 64, "spheres", 6, 0.55, "SIMPLEC", "fp64", 40, "loose"),
        # mid-size plain FP64 request, odd edge, fibres, flow along z
        _request("fp64_ideal_97", 97, 97, 97, "fibres", 3, 0.8, "IDEAL", "fp64", 2, "tight", 3),
        # the 128^3 sphere pack of the parity records
        _request("fp64_simplec_128", 128, 128, 128, "spheres", 8, 0.5, "SIMPLEC", "fp64", 3),
        # a large plain FP64 request: more rows than the loop kernels hold
        # one chunk per group for
        _request("fp64_simplec_171", 171, 150, 163, "fibres", 3, 0.85, "SIMPLEC", "fp64", 1),
        # mixed precision with Jacobi preconditioning (precision = MIXED)
        _request("mixed_simplec_56", 56, 56, 56, "spheres", 5, 0.6, "SIMPLEC", "mixed", 10),
        # a small and a large request of the serving stream as it is served
        _request("mg_ideal_70", 70, 70, 70, "fibres", 2, 0.6, "IDEAL", "mixed_mg", 6, "tight", 1),
        _request("mg_simplec_159", 159, 159, 159, "fibres", 3, 0.9, "SIMPLEC", "mixed_mg", 6, "tight", 2),
        # many small images driven from one thread, plain FP64
        _case("lockstep", "lockstep_fp64_8", count=8, lo=32, hi=48, precision="fp64", outer=6),
        # six requests in flight in the continuous-batching server
        _case("serve", "serve_mg_6", count=6, lo=48, hi=112, precision="mixed_mg", outer=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    """One more case of the ranges above (no name)."""
    path = rng.choice(("noalloc", "request", "request", "request", "request", "lockstep", "serve"))
    if path == "noalloc":
        return _case(path, edge=_log_int(rng, 8, 40), porosity=round(rng.uniform(0.5, 0.95), 3), tol=1e-8)
    if path == "lockstep":
        return _case(path, count=rng.randint(2, 8), lo=_log_int(rng, 20, 32), hi=_log_int(rng, 33, 48),
                     precision=rng.choice(("fp64", "mixed_mg")), outer=rng.randint(2, 6))
    if path == "serve":
        return _case(path, count=rng.randint(2, 6), lo=_log_int(rng, 32, 56), hi=_log_int(rng, 57, 112),
                     precision=rng.choice(("fp64", "mixed_mg")), outer=rng.randint(1, 4))
    precision = rng.choice(("fp64", "fp64", "mixed", "mixed_mg", "mixed_mg"))
    e = _log_int(rng, 20, 150 if precision == "mixed_mg" else 128)
    nx, ny, nz = (max(12, int(round(e * rng.uniform(0.75, 1.05)))) for _ in range(3))
    if rng.random() < 0.5:
        kind, radius, porosity = "spheres", rng.randint(3, 8), round(rng.uniform(0.45, 0.95), 3)
    else:
        kind, radius, porosity = "fibres", rng.randint(2, 4), round(rng.uniform(0.5, 0.95), 3)
    method = rng.choice(("SIMPLEC", "SIMPLEC", "SIMPLER", "SIMPLERR", "IDEAL"))
    outer = 1 if e > 90 else rng.randint(1, 2) if e > 60 else rng.randint(2, 8)
    return _request(None, nx, ny, nz, kind, radius, porosity, method, precision, outer,
                    rng.choice(("tight", "tight", "loose")), rng.randint(1, 3), rng.choice((0, 0, 1)))


# ---- inputs ------------------------------------------------------------------
def _image(shape, kind, radius, porosity, seed):
    img, _, _ = capi.generate_image(ns3d_gb300.lib(), 1 if kind == "fibres" else 0, shape, radius, porosity, seed,
                                    max_prims=1 << 12)
    return synth.to_raw(img)


def _params(shape, method, direction, border, precision, outer, numerics):
    return ns3d_gb300.default_params(
        dx=DX, mu=1e-3, rho=1.0, p0=1.0, gradp=1.0 / (shape[direction - 1] * DX), beta=1.0, N1=2, N2=2,
        direction=direction, border=border, method=method, precision=PRECISION[precision], maxitSIMPLE=outer,
        **(LOOSE if numerics == "loose" else TIGHT))


def _many(case, seed):
    """The images and parameters of a lockstep or served case: sizes, packs
    and methods by the case, the packs themselves by the seed."""
    rng = np.random.default_rng([case["count"], case["lo"], case["hi"]])
    out = []
    for i in range(case["count"]):
        e = int(round(np.exp(rng.uniform(np.log(case["lo"]), np.log(case["hi"])))))
        shape = (e, e, e) if case["path"] == "serve" else tuple(int(rng.integers(case["lo"], case["hi"] + 1))
                                                                for _ in range(3))
        fibres = bool(rng.integers(2))
        radius = int(rng.integers(2, 5)) if fibres else int(rng.integers(3, 7))
        raw = _image(shape, "fibres" if fibres else "spheres", radius, float(rng.uniform(0.5, 0.9)), seed * 131 + i)
        direction = int(rng.integers(1, 4)) if case["path"] == "serve" else 1
        method = ("SIMPLEC", "IDEAL")[int(rng.integers(2))]
        out.append((_params(shape, method, direction, 0, case["precision"], case["outer"], "tight"), raw, shape))
    return out


def _grid_system(case, seed):
    """A 7-point momentum-like system on the pores of a random pack: face
    conductances around 1, solid faces as walls (so it is regular), columns in
    the layout of ns3d_bicgstab_noalloc."""
    e = case["edge"]
    raw = _image((e, e, e), "spheres", 3, case["porosity"], seed)
    fluid = torch.from_numpy(raw.reshape(e, e, e) == 0).permute(2, 1, 0).contiguous()
    n = int(fluid.sum())
    npad = (e ** 3 + 1023) // 1024 * 1024
    index = torch.full((e, e, e), -1, dtype=torch.int64)
    index[fluid] = torch.arange(n)
    g = torch.Generator().manual_seed(seed)
    coef = torch.zeros(7, npad, dtype=torch.float64)
    nbr = torch.full((6, npad), -1, dtype=torch.int32)
    diag = torch.zeros(n, dtype=torch.float64)
    for axis in range(3):
        face = 0.5 + torch.rand((e + 1, e, e), generator=g, dtype=torch.float64)  # conductance of face i along `axis`
        idx = index.movedim(axis, 0)
        for side in range(2):
            col = torch.full_like(idx, -1)
            if side == 0:
                col[1:] = idx[:-1]
                cond = face[:-1]
            else:
                col[:-1] = idx[1:]
                cond = face[1:]
            col = col.movedim(0, axis)[fluid]
            cond = cond.movedim(0, axis)[fluid]
            slot = 2 * axis + side  # W, E, S, N, B, T
            nbr[slot, :n] = col.to(torch.int32)
            coef[slot + 1, :n] = torch.where(col >= 0, cond, torch.zeros_like(cond))
            diag += cond
    coef[0, :n] = -diag
    rhs = torch.zeros(npad, dtype=torch.float64)
    rhs[:n] = torch.randn(n, generator=g, dtype=torch.float64)
    return coef, nbr, rhs, n, npad


def _noalloc(lib):
    f = lib.ns3d_bicgstab_noalloc
    f.restype = C.c_int
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_void_p, C.c_void_p, C.c_int32, C.c_int32, C.c_double, C.c_int32,
                  C.c_void_p, C.POINTER(capi.SolveInfo)]
    return f


def _field_buffers(cells):
    """Pinned host buffers for p, u, v, w, as long as any image of this size needs."""
    return [torch.zeros(c, dtype=torch.float64, pin_memory=True) for c in cells]


def _cells(params, shape):
    nx, ny, nz = shape
    if params.direction == 2:
        nx, ny = ny, nx
    elif params.direction == 3:
        nx, nz = nz, nx
    nx += 2 * params.border
    return nx * ny * nz, (nx + 1) * ny * nz, nx * ny * nz, nx * ny * nz


def _doubles(buffers):
    return [C.cast(C.c_void_p(b.data_ptr()), C.POINTER(C.c_double)) for b in buffers]


def prepare(case, seed):
    lib = ns3d_gb300.lib()
    if case["path"] == "noalloc":
        coef, nbr, rhs, n, npad = _grid_system(case, seed)
        return {"case": case, "call": _noalloc(lib), "coef": coef.cuda(), "nbr": nbr.cuda(), "rhs": rhs.cuda(),
                "x": torch.zeros(npad, dtype=torch.float64, device="cuda"), "n": n, "npad": npad}
    if case["path"] == "request":
        shape = (case["nx"], case["ny"], case["nz"])
        raw = _image(shape, case["kind"], case["radius"], case["porosity"], seed)
        prm = _params(shape, case["method"], case["direction"], case["border"], case["precision"], case["outer"],
                      case["numerics"])
        return {"case": case, "lib": lib, "raw": raw, "params": prm, "shape": shape,
                "fields": _field_buffers(_cells(prm, shape))}
    jobs = _many(case, seed)
    state = {"case": case, "lib": lib, "fields": [_field_buffers(_cells(p, shape)) for p, _, shape in jobs]}
    if case["path"] == "lockstep":
        state["solvers"] = [capi.Solver(lib, *j) for j in jobs]
    else:
        state["jobs"] = jobs
        state["server"] = capi.Server(lib, max_active=6)
    return state


# ---- one pass ------------------------------------------------------------------
_SCALARS = ("K", "Q", "v_moy", "RMR", "normdiv", "reldiv", "velocityNorm", "maxdiv", "MaxDeltaV")
_COUNTS = ("iterations", "converged", "it_u", "it_v", "it_w", "it_p", "krylov_iterations")


def _outputs(result, fields):
    out = {"scalars": np.array([getattr(result, k) for k in _SCALARS]),
           "counts": np.array([getattr(result, k) for k in _COUNTS], np.int64)}
    out.update(zip(("p", "u", "v", "w"), fields))
    return out


def _checked(rc, what):
    if rc != 0:
        raise RuntimeError("%s returned %d" % (what, rc))


def run(state):
    path = state["case"]["path"]
    if path == "noalloc":
        x = state["x"]
        x.zero_()
        info = capi.SolveInfo()
        _checked(state["call"](state["coef"].data_ptr(), state["nbr"].data_ptr(), state["rhs"].data_ptr(),
                               x.data_ptr(), state["n"], state["npad"], state["case"]["tol"], 2000,
                               torch.cuda.current_stream().cuda_stream, C.byref(info)), "ns3d_bicgstab_noalloc")
        return {"x": x, "info": np.array([info.iterations, info.info], np.int64)}
    lib = state["lib"]
    if path == "request":
        s = capi.Solver(lib, state["params"], state["raw"], state["shape"])
        result = s.solve()
        _checked(lib.ns3d_get_fields(s.h, *_doubles(state["fields"])), "ns3d_get_fields")
        s.close()
        return _outputs(result, state["fields"])
    if path == "lockstep":
        for s in state["solvers"]:
            s.set_initial_fields()
        rc, status = capi.solve_lockstep(lib, state["solvers"])
        _checked(rc or int(status.min()), "ns3d_solve_lockstep")
        for s, buffers in zip(state["solvers"], state["fields"]):
            _checked(lib.ns3d_get_fields(s.h, *_doubles(buffers)), "ns3d_get_fields")
        return [_outputs(s.result(), buffers) for s, buffers in zip(state["solvers"], state["fields"])]
    srv = state["server"]
    tickets = [srv.submit(*j, keep_fields=True) for j in state["jobs"]]
    out = []
    for t, buffers in zip(tickets, state["fields"]):
        result, _ = srv.wait(t)
        _checked(lib.ns3d_server_fields(srv.h, t, *_doubles(buffers)), "ns3d_server_fields")
        out.append(_outputs(result, buffers))
    return out


# ---- what a pass cannot do without ------------------------------------------------
def _solve_work(cells, edge, case):
    """Counts of one capped solve on `cells` voxels: the BiCGSTAB iterations
    that such a pack needs (about 4.8 per voxel of edge at 1e-8 with Jacobi,
    about 45 with the multilevel preconditioner; loose tolerances a quarter),
    each with two sparse products and the vector updates, and the assembly of
    the four systems per outer iteration."""
    method = case.get("method", "SIMPLEC")
    solves = {"SIMPLEC": 1, "SIMPLER": 1 + 2, "SIMPLERR": 2 + 2, "IDEAL": 4}[method] * case["outer"]
    rows = cells * case.get("porosity", 0.7)
    loose = case.get("numerics") == "loose"
    word = 8 if case["precision"] == "fp64" else 4
    its = 45.0 if case["precision"] == "mixed_mg" else 4.8 * edge * (0.25 if loose else 1.0)
    per_iter = rows * (2 * 7 + 2 * 3 + 17) * word
    extra = 2 * rows * 12 * word if case["precision"] == "mixed_mg" else 0  # two V-cycles: fine level once each
    assembly = 4 * rows * 21 * 8.0 * case["outer"]
    momentum = 3 * rows * (2 * 7 + 2 * 3 + 17) * word * 10 * case["outer"]
    return {"bytes": solves * its * (per_iter + extra) + assembly + momentum,
            "flops": solves * its * rows * 50.0 + 4 * rows * 100.0 * case["outer"]}


def work(case):
    if case["path"] == "noalloc":
        rows = case["edge"] ** 3 * case["porosity"]
        its = 1.1 * case["edge"]
        return {"bytes": its * rows * 8.0 * 37, "flops": its * rows * 50.0}
    if case["path"] == "request":
        cells = (case["nx"] + 2 * case["border"]) * case["ny"] * case["nz"]
        return _solve_work(cells, max(case["nx"], case["ny"], case["nz"]), case)
    e = (case["lo"] * case["hi"]) ** 0.5
    one = _solve_work(e ** 3, e, case)
    return {k: case["count"] * 2.0 * v for k, v in one.items()}  # half of the images run IDEAL, with four solves


# ---- 64-bit values ------------------------------------------------------------------
def exact(case, seed):
    """The solution of the linear system by conjugate gradients in 64 bits,
    run until the residual stops falling.  A capped outer loop has no such
    value: its fields are those of an iteration count, not of an equation."""
    if case["path"] != "noalloc":
        return None
    coef, nbr, rhs, n, npad = _grid_system(case, seed)
    coef, cols, b = -coef[:, :n].cuda(), nbr[:, :n].cuda().long(), -rhs[:n].cuda()
    cols = torch.where(cols >= 0, cols, torch.arange(n, device="cuda"))  # missing entries have a zero coefficient

    def product(v):
        return coef[0] * v + (coef[1:] * v[cols]).sum(0)

    x = torch.zeros_like(b)
    for _ in range(3):  # restarts from the true residual
        r = b - product(x)
        p, rr = r.clone(), torch.dot(r, r)
        for _ in range(20 * case["edge"]):
            q = product(p)
            a = rr / torch.dot(p, q)
            x += a * p
            r -= a * q
            new = torch.dot(r, r)
            if float(new) <= 1e-40 * float(torch.dot(b, b)):
                break
            p = r + (new / rr) * p
            rr = new
    return {"x": torch.nn.functional.pad(x, (0, npad - n)), "info": None}
