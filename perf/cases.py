"""What a user of the cavity solver has it do, as cases that can be timed.

A user builds a mesh, binds a solver to it (one case, a batch of uneven cases,
or plain device arrays of one pressure system) and then calls it again and
again: whole SIMPLE outer iterations, the routines they consist of, pressure
solves to a tight residual, or the host-array drop-in.  ``prepare`` does the
first part -- mesh, solver and a developing flow to start from -- and ``run``
is one such call with the transfer of its fields in and out.

Sizes, forms and parameters are those of the repository's workloads: hex,
tet-split, prism, pyramid and mixed meshes of the unit-cube cavity, interior
nodes jittered by 0, 10 or 20% of the spacing, Re log-uniform in 10..1000,
alpha 0.7 / 0.3 for the steady form and the reference's dt = 0.01, rho = 5 for
the transient one.
"""
import ctypes as C
import math
import os
import random
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "cfd-lite_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)
import cfdl  # noqa: E402
import workloads  # noqa: E402

# fields an outer iteration starts from, and those a user reads back
STATE = ("u", "v", "w", "p", "u0", "v0", "w0", "gu", "gv", "gw", "gp", "mip", "mip0")
RESULT = ("u", "v", "w", "p", "gu", "gv", "gw", "gp", "mip")
KINDS = ("hex", "tet", "prism", "pyramid", "mixed")
PER_CUBE = {"hex": 1, "tet": 6, "prism": 2, "pyramid": 6, "mixed": 3.5}


def listed():
    return [
        # the smallest call: one outer iteration of a small served cavity (edge 24 is the lower end of the served
        # requests), where latency and launches are all there is
        {"name": "step24_p3", "path": "step", "kind": "hex", "n": 24, "jitter": 0.0, "precision": 3, "steps": 1},
        # the plain FP64 method on the 32^3 cavity, ten outer iterations between two looks at the fields
        {"name": "step32_fp64", "path": "step", "kind": "hex", "n": 32, "jitter": 0.0, "precision": 0, "steps": 10},
        # an unstructured (tet-split) mesh of odd size, four couplings per row, FP64
        {"name": "step45tet_fp64", "path": "step", "kind": "tet", "n": 45, "jitter": 0.1, "precision": 0, "steps": 8},
        # the 128^3 jittered cavity, the benchmark's default workload, FP64
        {"name": "step128_fp64", "path": "step", "kind": "hex", "n": 128, "jitter": 0.2, "precision": 0, "steps": 12},
        # the same mesh with the mixed forms of pressure solve, momentum corrections and explicit face terms
        {"name": "step128_p3", "path": "step", "kind": "hex", "n": 128, "jitter": 0.2, "precision": 3, "steps": 16},
        # a batch of uneven cases, half of them tet-split, as one graph launch, FP64
        {"name": "batch_fp64", "path": "batch", "count": 12, "n_lo": 16, "n_hi": 64, "precision": 0, "steps": 6},
        # the same in the mixed form, more cases
        {"name": "batch_p3", "path": "batch", "count": 24, "n_lo": 16, "n_hi": 64, "precision": 3, "steps": 5},
        # the energy equation solved after every outer iteration, odd edge
        {"name": "energy77_fp64", "path": "energy", "kind": "hex", "n": 77, "jitter": 0.1, "precision": 0, "steps": 5},
        # one mixed-precision pressure solve of a large mesh to a 1e-8 relative residual (FP64 refinement around FP32)
        {"name": "pressure176_mixed", "path": "pressure", "kind": "hex", "n": 176, "jitter": 0.1, "precision": 1},
        # the transient form, routine by routine, as a host that replaces one reference routine at a time calls it;
        # five-slot rows
        {"name": "routines41prism_fp64", "path": "routines", "kind": "prism", "n": 41, "jitter": 0.1, "precision": 0,
         "steps": 3},
        # the allocation-free pressure solve on the caller's own device arrays
        {"name": "noalloc40", "path": "noalloc", "n": 40, "rtol": 1e-12},
        # the drop-in with host arrays: upload u, v, w, p, one outer iteration, download of every field
        {"name": "host96_fp64", "path": "host", "kind": "hex", "n": 96, "jitter": 0.2, "precision": 0},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    path = rng.choice(("step", "step", "step", "batch", "energy", "pressure", "routines", "noalloc", "host"))
    if path == "noalloc":
        return {"path": path, "n": _log_int(rng, 9, 50), "rtol": rng.choice((1e-11, 1e-12, 1e-13))}
    if path == "batch":
        lo = rng.randrange(16, 33)
        return {"path": path, "count": rng.randrange(2, 17), "n_lo": lo, "n_hi": rng.randrange(lo, 61),
                "precision": rng.choice((0, 1, 2, 3)), "steps": rng.randrange(2, 6)}
    kind = rng.choice(("hex", "hex", "tet") + KINDS)
    # edge of the cube lattice such that every kind reaches about the same cell counts
    top = {"step": 2.0e6, "energy": 6e5, "pressure": 4e6, "routines": 5e5, "host": 1.2e6}[path]
    hi = int((top / PER_CUBE[kind]) ** (1 / 3))
    case = {"path": path, "kind": kind, "n": _log_int(rng, 16, hi), "jitter": rng.choice((0.0, 0.1, 0.2)),
            "precision": rng.choice((0, 0, 1, 2, 3, 3))}
    if path == "pressure":
        case["precision"] = rng.choice((0, 1, 1))
    if path in ("step", "energy", "routines"):
        cap = {"step": 2.0e7, "energy": 2.5e6, "routines": 1.5e6}[path]
        case["steps"] = max(1, min(rng.randrange(1, 13), int(cap / _cells(case))))
    return case


def _cells(case):
    return case["n"] ** 3 * PER_CUBE[case["kind"]]


def _params(seed):
    """Reynolds number of an input: log-uniform in 10..1000 (rho = 1, lid speed 1, mu = 1/Re)."""
    return 1.0 / math.exp(random.Random(seed).uniform(math.log(10.0), math.log(1000.0)))


def _pinned(n):
    return torch.empty(int(n), dtype=torch.float64, pin_memory=True)


def _fields(tensors):
    return cfdl.Fields(**{k: C.c_void_p(v.data_ptr()) for k, v in tensors.items()})


def _check(st, what):
    if st != cfdl.CFDL_OK:
        raise cfdl.CfdlError(st, what)


class State:
    pass


def prepare(case, seed):
    path = case["path"]
    s = State()
    s.case, s.path = case, path
    if path == "noalloc":
        _prepare_noalloc(s, case, seed)
        return s
    if path == "batch":
        _prepare_batch(s, case, seed)
        return s
    # the mesh: interior nodes jittered from the seed
    zone = cfdl.Zone(case["n"], kind=case["kind"], jitter=case["jitter"], seed=seed)
    s.setup = cfdl.Setup(zone, device=True)
    mu, prec = _params(seed), case["precision"]
    if path == "pressure":
        s.config = cfdl.steady(mu=mu, precision=prec, solve_mode=1, tight_rtol=1e-8)
    elif path == "routines":
        s.config = cfdl.default_config(precision=prec)       # the reference's transient form: rho 5, mu 0.01, dt 0.01
    else:
        s.config = cfdl.steady(mu=mu, precision=prec)
    s.solver = g = cfdl.Solver(s.setup, s.config)
    if path == "energy":
        g.energy_init()
    if path == "routines":
        # the transient form starts from a disturbed flow drawn from the seed
        r = np.random.default_rng(seed)
        for f in ("u", "v", "w"):
            a = g.get(f)
            a[:s.setup.ne] = 0.05 * r.standard_normal() + 0.01 * r.standard_normal(s.setup.ne)
            g.set(f, a)
    # a developing flow, a few outer iterations from the initial state
    g.step(3, 3 if path == "routines" else 0)
    if path == "pressure":
        # the pressure-correction system of the next outer iteration
        g.update_boundaries()
        g.calc_coef_uvw()
        g.solve_momentum()
        g.calc_grad("uvw")
        g.calc_mip(True)
        g.calc_coef_p()
        s.out = {"phic": _pinned(g.ne + g.nbf)}
        return s
    s.start = {f: _pinned(g._len(f)) for f in STATE}
    s.c_start = _fields(s.start)
    _check(cfdl.lib().cfdl_download_fields(g._h, C.byref(s.c_start)), "download")
    if path == "host":
        names = ("u", "v", "w", "p", "gu", "gv", "gw", "gp", "gpc", "mip")
        s.host = {f: _pinned(g._len(f)) for f in names}
        s.c_host = _fields(s.host)
        _check(cfdl.lib().cfdl_download_fields(g._h, C.byref(s.c_host)), "download")
        s.keep = sum(cfdl.FIELD_BITS[k] for k in names if k not in ("u", "v", "w", "p"))
        return s
    s.out = {f: _pinned(g._len(f)) for f in RESULT}
    s.c_out = _fields(s.out)
    if path == "energy":
        s.more = {f: g.get(f) for f in ("t", "e", "e0")}
    if path == "routines":
        s.extra = {f: _pinned(g._len(f)) for f in ("bu", "d", "dc", "b", "phic")}
    return s


def _prepare_batch(s, case, seed):
    lo, hi = case["n_lo"], case["n_hi"]
    # edges spread evenly over the range so that every input is as much work; the tet-split half, the order and the
    # Reynolds numbers come from the seed
    k = case["count"]
    r = random.Random(seed)
    edges = [int(round(lo + (hi - lo) * (i + 0.5) / k)) for i in range(k)]
    specs = [{"n": e, "tet": i % 2 == 1, "re": 1.0 / _params(seed * 1000 + i)} for i, e in enumerate(edges)]
    r.shuffle(specs)
    setups = workloads.build_setups(specs, jitter=0.1, seed=seed)
    s.batch = cfdl.Batch(setups, [cfdl.steady(mu=1.0 / c["re"], precision=case["precision"]) for c in specs])
    s.ids = s.batch.ids()
    s.batch.set_run(3)
    s.batch.run(3)
    sizes = [q.ne + q.nbf for q in setups]
    s.at = np.concatenate([[0], np.cumsum(sizes)])
    s.out = {f: _pinned(s.at[-1]) for f in ("u", "v", "w", "p")}


def _noalloc_system(case, seed):
    """A pressure-correction system of an n^3 cavity in the reference's CSR layout: the symmetric zero-row-sum matrix
    of face coefficients area/(dr.n) times a smoothly varying factor, and the net inflow of random face fluxes."""
    n = case["n"]
    ne, nbf = n ** 3, 6 * n * n
    r = np.random.default_rng(seed)
    cell = np.arange(ne).reshape(n, n, n)                     # z, y, x
    nb = np.full((ne, 6), -1, dtype=np.int64)
    a = np.zeros((ne, 6))
    b = np.zeros(ne)
    for axis in range(3):
        lo = np.take(cell, np.arange(n - 1), axis=2 - axis).ravel()
        hi = np.take(cell, np.arange(1, n), axis=2 - axis).ravel()
        c = (1.0 / n) * np.exp(0.2 * r.standard_normal(lo.size))
        q = r.standard_normal(lo.size) / (n * n)
        nb[lo, 2 * axis + 1], nb[hi, 2 * axis] = hi, lo
        a[lo, 2 * axis + 1], a[hi, 2 * axis] = c, c
        np.subtract.at(b, lo, q)
        np.add.at(b, hi, q)
    inside = nb >= 0
    halo = ne + np.cumsum(~inside.ravel()).reshape(ne, 6) - 1
    slot = np.arange(6)[None, :] ^ 1                          # the face as the neighbour numbers it, 1-based
    ef1 = np.where(inside, ((nb + 1) << 5) | (slot + 1), (halo + 1) << 5)
    idx = 1 + 6 * np.arange(ne + 1)
    assert halo.max() == ne + nbf - 1
    return ef1.astype(np.int32).ravel(), idx.astype(np.int32), a.sum(1), a.ravel(), b, nb


def _prepare_noalloc(s, case, seed):
    ef1, idx, ap, anb, b, _ = _noalloc_system(case, seed)
    s.ne, s.nh = ap.size, anb.size
    s.dev = [torch.from_numpy(x).cuda() for x in (ef1, idx, ap, anb, b)]
    s.x = torch.empty(s.ne, dtype=torch.float64, device="cuda")
    s.iters, s.rnorm = C.c_int(), C.c_double()
    torch.cuda.synchronize()


def run(state):
    s, L = state, cfdl.lib()
    if s.path == "noalloc":
        d = [C.c_void_p(t.data_ptr()) for t in s.dev]
        _check(L.cfdl_solve_pc_noalloc(s.ne, s.nh, d[0], d[1], d[2], d[3], d[4], C.c_void_p(s.x.data_ptr()),
                                       s.case["rtol"], 20000, C.byref(s.iters), C.byref(s.rnorm)), "solve_pc_noalloc")
        return {"phic": s.x}
    if s.path == "batch":
        s.batch.set_run(s.case["steps"])
        s.batch.run(s.case["steps"])
        for i, cid in enumerate(s.ids):
            for f, t in s.out.items():
                _check(L.cfdl_case_get_array(s.batch._h, cid, f.encode(),
                                             C.c_void_p(t.data_ptr() + 8 * int(s.at[i]))), "case_get " + f)
        return s.out
    g = s.solver
    if s.path == "pressure":
        g.solve_pc()
        _check(L.cfdl_get_array(g._h, b"phic", C.c_void_p(s.out["phic"].data_ptr())), "get phic")
        return s.out
    if s.path == "host":
        _check(L.cfdl_step_host_keep(g._h, C.byref(s.c_host), s.keep, 1, 0, None), "step_host_keep")
        return s.host
    # restart from the saved flow, advance, read back
    _check(L.cfdl_upload_fields(g._h, C.byref(s.c_start)), "upload")
    if s.path == "energy":
        for f, v in s.more.items():
            g.set(f, v)
    if s.path == "routines":
        for k in range(s.case["steps"]):
            g.update_boundaries()
            g.calc_coef_uvw()
            g.solve_momentum()
            g.calc_grad("uvw")
            g.calc_mip(True)
            g.calc_coef_p()
            g.solve_pc()
            g.adjust_pc()
            g.calc_grad("phic")
            g.update_uvwp()
        g.update_time()
    else:
        g.step(s.case["steps"], 0)
    _check(L.cfdl_download_fields(g._h, C.byref(s.c_out)), "download")
    out = dict(s.out)
    if s.path == "energy":
        out["t"] = g.get("t")
    if s.path == "routines":
        for f, t in s.extra.items():
            _check(L.cfdl_get_array(g._h, f.encode(), C.c_void_p(t.data_ptr())), "get " + f)
        out.update(s.extra)
    return out


def _sizes(kind, n):
    """Cells, faces and slots per row of one mesh."""
    c = n ** 3
    if kind == "hex":
        return c, 3 * n ** 2 * (n + 1), 6
    w = {"tet": 4, "prism": 5, "pyramid": 5, "mixed": 6}[kind]
    ne = PER_CUBE[kind] * c
    per_row = {"tet": 4, "prism": 5, "pyramid": 5, "mixed": 5.15}[kind]
    return ne, 0.5 * per_row * ne + 6 * n * n, w


def _iteration_bytes(ne, nf, w):
    # connectivity, gradient stencil, volume; geometry and property planes of the faces; fields in and out
    mesh = ne * (8 * w + 24 * w + 8) + nf * 8 * (15 + 10 + 1)
    fields = ne * 8 * (4 + 4 + 2 * 15) + nf * 16
    return mesh + fields


def _iteration_flops(ne, nf):
    # assembly, gradients, fluxes, one BiCGStab iteration of three components and five V-cycles
    return 2 * (ne * 560 + nf * 75)


def work(case):
    path = case["path"]
    if path == "noalloc":
        ne = case["n"] ** 3
        its = 4 * case["n"]                                   # CG iterations grow with the edge
        return {"bytes": ne * (6 * 12 + 4 + 3 * 8), "flops": its * ne * (2 * 7 + 12)}
    if path == "batch":
        k, lo, hi = case["count"], case["n_lo"], case["n_hi"]
        b = f = 0.0
        for i in range(k):
            ne, nf, w = _sizes("tet" if i % 2 else "hex", round(lo + (hi - lo) * (i + 0.5) / k))
            b += case["steps"] * _iteration_bytes(ne, nf, w) + 4 * 8 * ne
            f += case["steps"] * _iteration_flops(ne, nf)
        return {"bytes": b, "flops": f}
    ne, nf, w = _sizes(case["kind"], case["n"])
    if path == "pressure":
        return {"bytes": ne * (4 * w + 8 * w + 24), "flops": 40 * ne * 100}
    steps = case.get("steps", 1)
    b, f = steps * _iteration_bytes(ne, nf, w), steps * _iteration_flops(ne, nf)
    if path == "energy":
        b, f = b + steps * ne * 8 * 30, f + steps * ne * 900
    return {"bytes": b + ne * 8 * 40 + nf * 24, "flops": f}


def exact(case, seed):
    """The pressure correction of the allocation-free solve, by conjugate gradients in 64 bits on the plain system.  The
    other paths are sequences of whole nonlinear iterations with inner solves stopped at a residual drop: no plain value."""
    if case["path"] != "noalloc":
        return None
    _, _, ap, anb, b, nb = _noalloc_system(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    ap, b = torch.from_numpy(ap).to(dev), torch.from_numpy(b).to(dev)
    a = torch.from_numpy(anb.reshape(-1, 6)).to(dev)
    j = torch.from_numpy(np.where(nb >= 0, nb, 0)).to(dev)

    def amul(x):
        return ap * x - (a * x[j]).sum(1)

    b = b - b.mean()
    x = torch.zeros_like(b)
    # restarted: each restart's true residual takes out what rounding left
    for _ in range(4):
        r = b - amul(x)
        r = r - r.mean()
        z = r / ap
        p, rz, r0 = z.clone(), torch.dot(r, z), torch.linalg.norm(r)
        for it in range(40 * case["n"]):
            q = amul(p)
            alpha = rz / torch.dot(p, q)
            x = x + alpha * p
            r = r - alpha * q
            if it % 16 == 0 and torch.linalg.norm(r) <= 1e-12 * r0:
                break
            z = r / ap
            rn = torch.dot(r, z)
            p = z + (rn / rz) * p
            rz = rn
    # A has the constants in its kernel; conjugate gradients with Jacobi scaling, from zero, stay where the sum weighted
    # by the diagonal is zero
    return {"phic": x - torch.dot(ap, x) / ap.sum()}
