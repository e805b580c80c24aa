"""The operator applies a boundary-element program runs, as timed cases.

Every case goes through the package's public entry points (``tbempy.ThreeD``,
``tbempy.TwoD``, ``tbempy.autograd``): the operators are built once, as a
solver or an inversion builds them, and one pass is one call of the kind such
a program makes in its inner loop.

Kinds of case:
  apply      FMMOperator.apply on device tensors (any form, 3D or 2D)
  density    forward and transposed apply: the gradient of a misfit with
             respect to the density (autograd.fmm_apply)
  geometry   the gradient of a misfit with respect to both point sets and the
             density (autograd.fmm_apply_geometry)
  step       displacement and traction of one fault as one CUDA graph
  batch      many meshes and many right-hand sides in one operator
  csr        the sparse nearfield correction (SparseOperator.apply)
  boundary   the assembled boundary operator (IntegralOperator.apply)
  direct     the direct FP64 sum (DirectOperator.apply)
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "3bem_gb300"))

from tbempy import ThreeD, TwoD, autograd, meshes  # noqa: E402

MU, NU = 1.0, 0.25
MAC, D = 0.3, 0.05


def listed():
    return [
        # the smallest call: a coarse sphere inside a solver's inner loop, all latency
        {"name": "sphere_960_mixed", "kind": "apply", "dim": 3, "kernel": "LaplaceSingle", "precision": "mixed",
         "mesh": "icosphere", "size": 2, "order": 152, "leaf": 30, "n_rhs": 1},
        # the headline step: both elastic operators of a 98,304-point dipping fault, one graph
        {"name": "fault_98k_step_graph", "kind": "step", "dim": 3, "mesh": "fault", "size": 128, "order": 296,
         "leaf": 64, "n_rhs": 1},
        # a slip inversion's iteration: traction forward and transposed, 24,576 points
        {"name": "fault_24k_density_gradient", "kind": "density", "dim": 3, "kernel": "ElasticTraction",
         "precision": "mixed", "mesh": "fault", "size": 64, "order": 296, "leaf": 64, "n_rhs": 1},
        # a geometry inversion's iteration: observers on the free surface over a warped fault
        {"name": "fault_geometry_gradient", "kind": "geometry", "dim": 3, "kernel": "ElasticDisplacement",
         "precision": "mixed", "mesh": "warped_fault", "size": 32, "n_obs": 4096, "order": 296, "leaf": 64,
         "n_rhs": 1},
        # the drop-in of the reference's operator: plain FP64, one right-hand side
        {"name": "sphere_15k_plain", "kind": "apply", "dim": 3, "kernel": "LaplaceSingle", "precision": "fp64",
         "mesh": "icosphere", "size": 4, "order": 152, "leaf": 50, "n_rhs": 1},
        # the same form for an elastic kernel on a small mesh of an odd size, at a lower order
        {"name": "fault_3k_plain_elastic", "kind": "apply", "dim": 3, "kernel": "ElasticDisplacement",
         "precision": "fp64", "mesh": "fault", "size": 23, "order": 99, "leaf": 40, "n_rhs": 1},
        # the FP64 residual operator of iterative refinement on the bumpy sphere
        {"name": "bumpy_61k_fp64_compressed", "kind": "apply", "dim": 3, "kernel": "LaplaceDouble",
         "precision": "fp64_compressed", "mesh": "bumpy", "size": 5, "order": 296, "leaf": 64, "n_rhs": 1},
        # many meshes of uneven size, 64 right-hand sides
        {"name": "batch_16_spheres_64rhs", "kind": "batch", "dim": 3, "kernel": "LaplaceDouble", "size": 16,
         "max_level": 4, "order": 152, "leaf": 128, "n_rhs": 64},
        # a 2D crack problem in the plain form
        {"name": "circle_20k_2d_elastic", "kind": "apply", "dim": 2, "kernel": "ElasticTraction", "precision": "fp64",
         "mesh": "circle", "size": 20000, "order": 24, "leaf": 32, "n_rhs": 1},
        # the sparse nearfield correction of a 20,480-facet sphere: 184,320 rows, 9.2 M entries
        {"name": "nearfield_csr_20k_facets", "kind": "csr", "size": 20480, "nnz_per_row": 50, "n_rhs": 1},
        # the whole boundary operator of a 1,280-facet sphere, as GMRES calls it
        {"name": "boundary_1280_facets", "kind": "boundary", "dim": 3, "kernel": "LaplaceDouble", "size": 3,
         "precision": "fp64", "order": 75, "leaf": 20, "n_rhs": 1},
        # the exact check every result is reported against
        {"name": "direct_6k_traction", "kind": "direct", "dim": 3, "kernel": "ElasticTraction", "mesh": "fault",
         "size": 32, "n_rhs": 1},
    ]


KERNELS = ["LaplaceSingle", "LaplaceDouble", "ElasticDisplacement", "ElasticTraction"]


def _between(rng, lo, hi):
    """An integer spread over the logarithm of its range."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["mixed", "mixed", "plain", "compressed", "2d", "step", "density", "geometry", "batch", "csr",
                       "boundary", "direct"])
    kernel = rng.choice(KERNELS)
    elastic = kernel.startswith("Elastic")
    # the double layer vanishes on a plane
    mesh = "spiral" if kernel == "LaplaceDouble" else "fault"
    if kind == "mixed":
        return {"kind": "apply", "dim": 3, "kernel": kernel, "precision": "mixed",
                "mesh": mesh, "size": _between(rng, 12, 120),
                "order": 296 if elastic else 152, "leaf": rng.choice([30, 40, 50, 64]), "n_rhs": rng.choice([1, 1, 2, 7])}
    if kind == "plain":
        return {"kind": "apply", "dim": 3, "kernel": kernel, "precision": "fp64", "mesh": mesh,
                "size": _between(rng, 12, 32 if elastic else 48), "order": 99 if elastic else rng.choice([75, 152]),
                "leaf": rng.choice([25, 40, 50]), "n_rhs": rng.choice([1, 1, 3])}
    if kind == "compressed":
        k = rng.choice(["LaplaceSingle", "LaplaceDouble"])
        return {"kind": "apply", "dim": 3, "kernel": k, "precision": "fp64_compressed", "mesh": "spiral",
                "size": _between(rng, 20, 90), "order": rng.choice([152, 296]), "leaf": rng.choice([40, 64]),
                "n_rhs": rng.choice([1, 1, 2])}
    if kind == "2d":
        return {"kind": "apply", "dim": 2, "kernel": kernel, "precision": "fp64", "mesh": "circle",
                "size": _between(rng, 900, 24000), "order": rng.choice([16, 20, 24]), "leaf": rng.choice([20, 32]),
                "n_rhs": rng.choice([1, 3])}
    if kind == "step":
        return {"kind": "step", "dim": 3, "mesh": "fault", "size": _between(rng, 12, 120), "order": 296, "leaf": 64,
                "n_rhs": 1}
    if kind == "density":
        return {"kind": "density", "dim": 3, "kernel": kernel, "precision": "mixed", "mesh": mesh,
                "size": _between(rng, 12, 96), "order": 296 if elastic else 152, "leaf": rng.choice([40, 64]),
                "n_rhs": rng.choice([1, 1, 4])}
    if kind == "geometry":
        return {"kind": "geometry", "dim": 3, "kernel": rng.choice(["LaplaceSingle", "ElasticDisplacement"]),
                "precision": "mixed", "mesh": "warped_fault", "size": _between(rng, 12, 34),
                "n_obs": _between(rng, 500, 4500), "order": 296, "leaf": 64, "n_rhs": 1}
    if kind == "batch":
        return {"kind": "batch", "dim": 3, "kernel": rng.choice(["LaplaceSingle", "LaplaceDouble"]),
                "size": _between(rng, 3, 16), "max_level": rng.choice([3, 4]), "order": 152, "leaf": 128,
                "n_rhs": rng.choice([5, 16, 33, 64])}
    if kind == "csr":
        return {"kind": "csr", "size": _between(rng, 600, 20000), "nnz_per_row": rng.choice([12, 27, 50]),
                "n_rhs": rng.choice([1, 1, 3])}
    if kind == "boundary":
        return {"kind": "boundary", "dim": 3, "kernel": rng.choice(["LaplaceSingle", "LaplaceDouble"]),
                "size": rng.choice([2, 3]), "precision": "fp64", "order": rng.choice([75, 99]),
                "leaf": rng.choice([20, 30, 40]), "n_rhs": rng.choice([1, 2])}
    return {"kind": "direct", "dim": 3, "kernel": kernel, "mesh": mesh, "size": _between(rng, 8, 32),
            "n_rhs": rng.choice([1, 1, 4])}


# ---------------------------------------------------------------- geometry

def _points(case):
    """(locs, normals, weights) of the case's mesh, numpy FP64."""
    mesh, size = case["mesh"], case["size"]
    if mesh == "icosphere":
        return meshes.sphere_points(size)
    if mesh == "fault":
        return meshes.fault_points(size)[:3]
    if mesh == "warped_fault":
        v, t, _ = meshes.dipping_fault(size, 45.0)
        v = v.copy()
        v[:, 2] += 0.05 * np.sin(3 * v[:, 0]) * np.cos(2 * v[:, 1])
        return meshes.points_from_mesh(v, t)
    if mesh == "bumpy":
        return meshes.points_from_mesh(*meshes.bumpy_sphere(size))
    if mesh == "spiral":  # 6 size^2 + 1 points spread over the unit sphere on a golden spiral
        n = 6 * size * size + 1
        i = np.arange(n) + 0.5
        z = 1.0 - 2.0 * i / n
        a = math.pi * (1.0 + 5.0 ** 0.5) * i
        s = np.sqrt(1.0 - z * z)
        p = np.ascontiguousarray(np.stack([s * np.cos(a), s * np.sin(a), z], axis=1))
        return p, p.copy(), np.full(n, 4.0 * math.pi / n)
    n = size  # circle
    a = 2.0 * math.pi * (np.arange(n) + 0.5) / n
    r = 1.0 + 0.1 * np.cos(5 * a)
    p = np.ascontiguousarray(np.stack([r * np.cos(a), r * np.sin(a)], axis=1))
    t = np.stack([np.gradient(p[:, 0]), np.gradient(p[:, 1])], axis=1)
    length = np.linalg.norm(t, axis=1)
    return p, np.ascontiguousarray(np.stack([t[:, 1], -t[:, 0]], axis=1) / length[:, None]), length


def _observers(case):
    rng = np.random.default_rng(5)
    n = case["n_obs"]
    return (np.column_stack([rng.uniform(-3, 3, n), rng.uniform(-3, 3, n), np.zeros(n)]),
            np.tile([0.0, 0.0, 1.0], (n, 1)))


def _kernel(case, name=None):
    k = getattr(TwoD if case["dim"] == 2 else ThreeD, name or case["kernel"])
    return k(MU, NU) if k.__name__.startswith("Elastic") else k()


def _components(case, name=None):
    return case["dim"] if (name or case["kernel"]).startswith("Elastic") else 1


def _vectors(seed, n_rhs, n):
    """Densities uniform in [-1, 1], [n] or [n_rhs, n], on the GPU."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    x = torch.rand((n_rhs, n), generator=g, device="cuda", dtype=torch.float64) * 2 - 1
    return x[0] if n_rhs == 1 else x


def _config(case):
    return ThreeD.FMMConfig(MAC, case["order"], case["leaf"], D, False)


def _batch_points(case):
    """Icospheres of levels 2 .. max_level in turn, radii and centres as in the batched workload."""
    rng = np.random.default_rng(2)
    L, N, W, off = [], [], [], [0]
    base = {}
    for m in range(case["size"]):
        lev = 2 + m % (case["max_level"] - 1)
        if lev not in base:
            base[lev] = meshes.sphere_points(lev)
        l0, n0, w0 = base[lev]
        r, c = rng.lognormal(0.0, 0.5), rng.uniform(-100.0, 100.0, 3)
        L.append(l0 * r + c)
        N.append(n0)
        W.append(w0 * r * r)
        off.append(off[-1] + len(l0))
    return np.concatenate(L), np.concatenate(N), np.concatenate(W), np.asarray(off, dtype=np.int64)


def _csr(case):
    """A nearfield matrix's pattern: the nine observation points of a facet share the three columns of each of its
    neighbouring facets, whose number varies about the mean; the facets' numbering keeps neighbours close."""
    nf = case["size"]
    rng = np.random.default_rng(7)
    mean = case["nnz_per_row"] / 3.0
    count = np.minimum(rng.integers(max(1, int(0.6 * mean)), int(1.4 * mean) + 2, nf), nf)
    width = int(1.4 * mean) + 2
    near = (np.arange(nf)[:, None] - 2 * width + np.cumsum(rng.integers(1, 7, (nf, width)), axis=1)) % nf
    keep = np.arange(width)[None, :] < count[:, None]
    rows = np.repeat(np.arange(nf), 9)
    near, keep = near[rows], keep[rows]
    cols = (3 * near[keep])[:, None] + np.arange(3)[None, :]
    row_ptrs = np.concatenate([[0], np.cumsum(3 * count[rows])]).astype(np.int64)
    cols = np.ascontiguousarray(cols.reshape(-1).astype(np.int64))
    return 9 * nf, 3 * nf, rng.standard_normal(len(cols)), cols, row_ptrs


# ------------------------------------------------------------------- cases

def prepare(case, seed):
    kind, n_rhs = case["kind"], case["n_rhs"]
    if kind == "csr":
        op = ThreeD.SparseOperator(*_csr(case))
        return {"kind": kind, "op": op, "x": _vectors(seed, n_rhs, op.n_cols())}
    if kind == "boundary":
        mesh = ThreeD.Mesh(*meshes.icosphere(case["size"]))
        mthd = ThreeD.make_sinh_integrator(5, 3, 3, 3, 8, 3.0, _kernel(case))
        op = ThreeD.boundary_operator(mesh, mesh, mthd, _config(case), mesh, precision=case["precision"])
        return {"kind": kind, "op": op, "x": _vectors(seed, n_rhs, op.n_cols())}
    if kind == "batch":
        op = ThreeD.BatchedFMMOperator(_kernel(case), *_batch_points(case), _config(case))
        return {"kind": kind, "op": op, "x": _vectors(seed, n_rhs, op.n_cols())}
    sl, sn, sw = _points(case)
    if kind == "direct":
        op = ThreeD.DirectOperator(_kernel(case), sl, sn, sl, sn, sw)
        return {"kind": kind, "op": op, "x": _vectors(seed, n_rhs, op.n_cols())}
    if kind == "step":
        ops = [ThreeD.FMMOperator(_kernel(case, k), sl, sn, sl, sn, sw, _config(case), precision="mixed")
               for k in ("ElasticDisplacement", "ElasticTraction")]
        x = _vectors(seed, n_rhs, ops[0].n_cols())
        ys = [torch.empty(op.n_rows(), dtype=torch.float64, device="cuda") for op in ops]
        torch.cuda.synchronize()
        return {"kind": kind, "graph": ThreeD.FMMGraph(ops, [x, x], ys), "ys": ys}
    ol, on = _observers(case) if kind == "geometry" else (sl, sn)
    op = ThreeD.FMMOperator(_kernel(case), ol, on, sl, sn, sw, _config(case), precision=case["precision"])
    state = {"kind": kind, "op": op, "x": _vectors(seed, n_rhs, op.n_cols())}
    if kind in ("density", "geometry"):
        state["data"] = _vectors(seed + 1000003, n_rhs, op.n_rows())
        state["x"].requires_grad_()
    if kind == "geometry":
        state["points"] = [torch.tensor(a, device="cuda", requires_grad=True) for a in (ol, on, sl, sn, sw)]
    return state


def run(state):
    kind = state["kind"]
    if kind == "step":
        stream = torch.cuda.current_stream().cuda_stream
        state["graph"].launch(stream if stream else 1)
        return state["ys"]
    op, x = state["op"], state["x"]
    if kind == "density":
        y = autograd.fmm_apply(op, x)
        (g,) = torch.autograd.grad(0.5 * ((y - state["data"]) ** 2).sum(), [x])
        return {"y": y.detach(), "density": g}
    if kind == "geometry":
        pts = state["points"]
        y = autograd.fmm_apply_geometry(op, *pts, x)
        g = torch.autograd.grad(0.5 * ((y - state["data"]) ** 2).sum(), [pts[0], pts[2], pts[4], x])
        return {"y": y.detach(), "observers": g[0], "sources": g[1], "weights": g[2], "density": g[3]}
    return op.apply(x)


# ------------------------------------------------------------ work of a pass

# operations of one kernel value applied to one density (multiply-add = 2)
_PAIR = {"LaplaceSingle": 12, "LaplaceDouble": 19, "ElasticDisplacement": 48, "ElasticTraction": 90}


def _n_points(case):
    s = case["size"]
    return {"icosphere": 60 * 4 ** s, "bumpy": 60 * 4 ** s, "fault": 6 * s * s, "warped_fault": 6 * s * s,
            "spiral": 6 * s * s + 1, "circle": s}[case["mesh"]]


def _fmm_flops(case, name, n_src, n_obs):
    """The FMM's kernel evaluations: every point with the points of the leaves around its own (on a surface about ten
    leaves of half their limit; in the plane six) and with its leaf's two translation surfaces."""
    near = (10 if case["dim"] == 3 else 6) * case["leaf"] / 2.0
    return _PAIR[name] * (n_obs * near + case["order"] * (n_src + n_obs))


def work(case):
    kind, r = case["kind"], case["n_rhs"]
    if kind == "csr":
        nnz = 9.0 * case["size"] * case["nnz_per_row"]
        # values, 32-bit columns, row starts, input and output
        return {"bytes": 12 * nnz + 8 * 9 * case["size"] + 8 * r * 12 * case["size"], "flops": 2 * nnz * r}
    if kind == "boundary":
        nf = 20 * 4 ** case["size"]
        # corrections (about 30 entries a row, three rows a facet, two matrices) and the FMM over nine points a facet
        return {"bytes": 12.0 * 2 * 3 * nf * 30 + 8 * r * 6 * nf,
                "flops": r * _fmm_flops(case, case["kernel"], 9 * nf, 9 * nf)}
    if kind == "batch":
        n = sum(60 * 4 ** (2 + m % (case["max_level"] - 1)) for m in range(case["size"]))
        # the kernel value is shared by the right-hand sides
        f = _fmm_flops(case, case["kernel"], n, n)
        return {"bytes": 16.0 * n * r + 56.0 * n, "flops": f * (1 + 2.0 * r / _PAIR[case["kernel"]])}
    n = _n_points(case)
    if kind == "step":
        return {"bytes": 8.0 * 3 * n * 3 + 56.0 * n,
                "flops": _fmm_flops(case, "ElasticDisplacement", n, n) + _fmm_flops(case, "ElasticTraction", n, n)}
    C = _components(case)
    if kind == "direct":
        return {"bytes": 16.0 * C * n * r + 104.0 * n, "flops": float(_PAIR[case["kernel"]]) * n * n * r}
    n_obs = case.get("n_obs", n)
    flops = _fmm_flops(case, case["kernel"], n, n_obs) * r
    bytes_ = 8.0 * C * (n + n_obs) * r + 8.0 * (2 * case["dim"] * (n + n_obs) + n)
    passes = {"apply": 1, "density": 2, "geometry": 4}[kind]
    return {"bytes": bytes_ * passes, "flops": flops * passes}


# -------------------------------------------------------------- exact values

def _blocks(name, dim, o, on, s, sn):
    """The kernel's R x R blocks for all pairs of o [m, dim] and s [n, dim], FP64; zero where the points coincide."""
    d = [s[None, :, k] - o[:, None, k] for k in range(dim)]
    r2 = sum(c * c for c in d)
    ok = r2 >= 1e-12
    r2 = torch.where(ok, r2, torch.ones_like(r2))
    ir2 = 1.0 / r2
    ir = torch.sqrt(ir2)
    one = ok.to(torch.float64)
    if name == "LaplaceSingle":
        return [[one * (ir / (4 * math.pi) if dim == 3 else 0.5 * torch.log(r2) / (2 * math.pi))]]
    if name == "LaplaceDouble":
        dn = sum(d[k] * sn[None, :, k] for k in range(dim))
        return [[one * dn * (ir2 * ir / (4 * math.pi) if dim == 3 else ir2 / (2 * math.pi))]]
    e = range(dim)
    if name == "ElasticDisplacement":
        c2 = 3 - 4 * NU
        if dim == 3:
            f, diag, rad = 1 / (16 * math.pi * MU * (1 - NU)), c2 * ir, ir * ir2
        else:
            f, diag, rad = 1 / (8 * math.pi * MU * (1 - NU)), -0.5 * c2 * torch.log(r2), ir2
        f = f * one
        return [[f * (diag + d[k] * d[j] * rad if k == j else d[k] * d[j] * rad) for j in e] for k in e]
    c2, q = 1 - 2 * NU, dim
    f = -one * (ir2 if dim == 3 else ir) / ((8 if dim == 3 else 4) * math.pi * (1 - NU))
    m = [sn[None, :, k] for k in e]
    drdm = sum(d[k] * m[k] for k in e) * ir
    return [[f * ((q * d[k] * d[j] * ir2 + (c2 if k == j else 0.0)) * drdm - c2 * (m[j] * d[k] - m[k] * d[j]) * ir)
             for j in e] for k in e]


def _dense(name, dim, o, on, s, sn, w, x, z=None):
    """A x [n_rhs, R n_obs], and A^T z where z is given, by chunks of observation points."""
    R = dim if name.startswith("Elastic") else 1
    n, m = s.shape[0], o.shape[0]
    xs = x.reshape(-1, R, n) * w
    y = torch.empty((xs.shape[0], R, m), dtype=torch.float64, device=o.device)
    t = torch.zeros((xs.shape[0], R, n), dtype=torch.float64, device=o.device)
    step = max(1, int(2e8 / n) // R)
    for b in range(0, m, step):
        K = _blocks(name, dim, o[b:b + step], on[b:b + step], s, sn)
        for k in range(R):
            y[:, k, b:b + step] = sum(xs[:, j] @ K[k][j].T for j in range(R))
            if z is not None:
                for j in range(R):
                    t[:, j] += z.reshape(-1, R, m)[:, k, b:b + step] @ K[k][j]
    return y.reshape(xs.shape[0], -1), (t * w).reshape(xs.shape[0], -1)


def _cuda(*arrays):
    return [torch.tensor(a, device="cuda") for a in arrays]


def exact(case, seed):
    kind, r = case["kind"], case["n_rhs"]

    def like(y):
        return y[0] if r == 1 else y

    if kind == "boundary":
        return None  # its singular integrals have no plain form
    if kind == "csr":
        nr, nc, v, c, p = _csr(case)
        x = _vectors(seed, r, nc).reshape(r, -1)
        v, c, rows = _cuda(v, c, np.repeat(np.arange(nr), np.diff(p)))
        y = torch.zeros((r, nr), dtype=torch.float64, device="cuda")
        for q in range(r):
            y[q].index_add_(0, rows, v * x[q, c])
        return like(y)
    if kind == "batch":
        L, N, W, off = _batch_points(case)
        l, n, w = _cuda(L, N, W)
        x = _vectors(seed, r, len(L)).reshape(r, -1)
        y = torch.empty_like(x)
        for a, b in zip(off[:-1], off[1:]):
            y[:, a:b] = _dense(case["kernel"], 3, l[a:b], n[a:b], l[a:b], n[a:b], w[a:b], x[:, a:b])[0]
        return like(y)
    sl, sn, sw = _cuda(*_points(case))
    dim = case["dim"]
    if kind == "step":
        x = _vectors(seed, r, 3 * len(sl))
        return [like(_dense(k, 3, sl, sn, sl, sn, sw, x)[0]) for k in ("ElasticDisplacement", "ElasticTraction")]
    R = _components(case)
    ol, on = _cuda(*_observers(case)) if kind == "geometry" else (sl, sn)
    x = _vectors(seed, r, R * len(sl))
    y = like(_dense(case["kernel"], dim, ol, on, sl, sn, sw, x)[0])
    if kind not in ("density", "geometry"):
        return y
    res = y - _vectors(seed + 1000003, r, R * len(ol))
    g = like(_dense(case["kernel"], dim, ol, on, sl, sn, sw, x, res)[1])
    if kind == "density":
        return {"y": y, "density": g}
    # the misfit's derivatives with respect to the points: r^T A x differentiated with r held
    leaf = [sl.clone().requires_grad_(), sw.clone().requires_grad_()]
    acc, g_obs = [torch.zeros_like(a) for a in leaf], torch.empty_like(ol)
    step = max(1, int(1e7 / len(sl)))
    for b in range(0, len(ol), step):
        o = ol[b:b + step].clone().requires_grad_()
        K = _blocks(case["kernel"], dim, o, on[b:b + step], leaf[0], sn)
        total = 0.0
        for k in range(R):
            z = res.reshape(R, -1)[k, b:b + step]
            for j in range(R):
                total = total + z @ (K[k][j] @ (x.reshape(R, -1)[j] * leaf[1]))
        g_obs[b:b + step], *more = torch.autograd.grad(total, [o] + leaf)
        for a, q in zip(acc, more):
            a += q
    return {"y": y, "observers": g_obs, "sources": acc[0], "weights": acc[1], "density": g}
