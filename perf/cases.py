"""The work a user of this framework has it do, as cases to time.

A case is a plain dict.  ``prepare`` makes what a program holds before the
call (model, solver, inputs on the GPU), ``run`` is one pass through the public
entry points, ``work`` what that pass cannot do without and ``exact`` the same
outputs in plain 64-bit torch, where they have such a value.

Kinds:

* ``state``    one state solve of the optimisation loop: densities -> moduli,
               Galerkin assembly, multigrid-preconditioned CG for every load
               case; a box cantilever or an irregular domain, FP64 or with the
               FP32 V-cycle.
* ``super``    the same for a super-element model (ft = 2): sub-voxel density
               filter, densities -> moduli, assembly, CG.
* ``step``     the design-dependent part of an iteration around the solve:
               state solve, element energies, PDE-filtered sensitivities.
* ``optimize`` the whole optimisation loop in one call.
* ``adjoint``  gradient of a nodal displacement through the PDE filter: state
               and adjoint solve on an i.i.d. design, to a tight tolerance.
* ``product``  y = K(E) u, for a program that iterates by itself.
* ``vcycle``   z = M r, the preconditioner by itself.
* ``filter``   the PDE density filter by itself.
* ``gather``   the two node/element MEX gateways around a user's element step.
* ``galerkin`` the two Galerkin MEX gateways of an ordinary model.

State solves run to a relative residual of 1e-8 or tighter, so that what is
compared is the solution and not where an iteration happened to stop.
"""
import functools
import math

import numpy as np
import torch

from top_gpu_on_matlab_b200 import mex
from top_gpu_on_matlab_b200.fea import Mesh, Solver

E0, EMIN, PENAL, NU = 1.0, 1e-9, 3.0, 0.3


def listed():
    return [
        # the precision configuration: the 96x192x96 cantilever, FP32 V-cycle
        dict(name="state_mixed_96x192x96", kind="state", domain="box", ny=96, nx=192, nz=96, mixed=True, control=400, tol=1e-9),
        # the plain FP64 configuration: 24x48x24, four levels; launches and latency count
        dict(name="state_fp64_24x48x24", kind="state", domain="box", ny=24, nx=48, nz=24, mixed=False, control=54, tol=1e-9),
        # the batching configuration at half its size: irregular domain, four load cases in one batched solve
        dict(name="state_mixed_irregular_4loads", kind="state", domain="irregular", ny=96, nx=192, nz=96, mixed=True, control=400, tol=1e-9),
        # an ordinary FP64 solve at the size of the sensitivity configuration
        dict(name="state_fp64_64x128x64", kind="state", domain="box", ny=64, nx=128, nz=64, mixed=False, control=1000, tol=1e-9),
        # the super-element configuration: 10x60x10 super elements of 4x4x4 voxels, MBB supports
        dict(name="super_fp64_10x60x10", kind="super", ny=10, nx=60, nz=10, mixed=False, control=20000, tol=1e-9),
        # an iteration's work around the solve on a ragged grid (padded levels, void margins), FP32 V-cycle
        dict(name="step_mixed_37x75x41", kind="step", ny=37, nx=75, nz=41, mixed=True, control=400, tol=1e-9),
        # the loop itself in one call, the reference's small cantilever, sensitivity filter
        dict(name="optimize_fp64_24x48x24", kind="optimize", ny=24, nx=48, nz=24, mixed=False, control=54, tol=1e-9, loops=4, ft=1),
        # the differentiation configuration: displacement objective chained through the PDE filter
        dict(name="adjoint_fp64_64x128x64", kind="adjoint", ny=64, nx=128, nz=64, mixed=False, control=20000, tol=1e-10),
        # the fine product at the benchmark's size
        dict(name="product_fp64_96x192x96", kind="product", ny=96, nx=192, nz=96, mixed=False, control=400, tol=1e-6),
        # the PDE filter at the benchmark's size (the reference runs it twice or three times an iteration with ft = 2)
        dict(name="filter_fp64_96x192x96", kind="filter", ny=96, nx=192, nz=96, rmin=2.5, control=400, tol=1e-6),
        # drop-in use from MATLAB: gather and scatter of a 64x128x64 model in double
        dict(name="gather_fp64_64x128x64", kind="gather", ny=64, nx=128, nz=64, single=False),
        # drop-in use from MATLAB: the Galerkin gateways of a 64x128x64 model in double
        dict(name="galerkin_fp64_64x128x64", kind="galerkin", ny=64, nx=128, nz=64, single=False),
    ]


def _size(rng, lo, hi):
    """A size spread over the logarithm of [lo, hi], every value possible."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["state", "state", "state", "super", "step", "optimize", "adjoint", "product", "vcycle", "filter",
                       "gather", "galerkin"])
    if kind == "state":
        mixed = rng.random() < 0.5
        if rng.random() < 0.3:      # the ellipsoids need room: from a quarter of the configuration's grid
            n = _size(rng, 48, 88)
            return dict(kind=kind, domain="irregular", ny=n, nx=2 * n - rng.randrange(4), nz=n - rng.randrange(4), mixed=mixed, control=400, tol=1e-9)
        return dict(kind=kind, domain="box", ny=_size(rng, 12, 88), nx=_size(rng, 24, 176), nz=_size(rng, 12, 88), mixed=mixed,
                    control=rng.choice([400, 1000]), tol=1e-9)
    if kind == "super":
        return dict(kind=kind, ny=2 * _size(rng, 3, 8), nx=2 * _size(rng, 8, 32), nz=_size(rng, 6, 16), mixed=rng.random() < 0.5, control=20000, tol=1e-9)
    if kind == "step":
        return dict(kind=kind, ny=_size(rng, 16, 64), nx=_size(rng, 32, 128), nz=_size(rng, 16, 64), mixed=rng.random() < 0.5,
                    control=rng.choice([400, 1000]), tol=1e-9)
    if kind == "optimize":
        return dict(kind=kind, ny=_size(rng, 12, 32), nx=_size(rng, 24, 64), nz=_size(rng, 12, 32), mixed=False, control=400,
                    tol=1e-9, loops=rng.choice([2, 3, 4]), ft=rng.choice([0, 1, 2]))
    if kind == "adjoint":
        return dict(kind=kind, ny=_size(rng, 16, 60), nx=_size(rng, 32, 120), nz=_size(rng, 16, 60), mixed=False, control=rng.choice([1000, 20000]), tol=1e-10)
    if kind in ("product", "vcycle"):
        return dict(kind=kind, ny=_size(rng, 12, 96), nx=_size(rng, 24, 192), nz=_size(rng, 12, 96), mixed=False, control=1000, tol=1e-6)
    if kind == "filter":
        return dict(kind=kind, ny=_size(rng, 12, 96), nx=_size(rng, 24, 192), nz=_size(rng, 12, 96), rmin=rng.choice([math.sqrt(3.0), 2.5, 4.0]),
                    control=1000, tol=1e-6)
    n = lambda hi: 8 * _size(rng, 2, hi // 8)  # noqa: E731  (the drop-ins' two levels, spans 4 and 2, without padding)
    return dict(kind=kind, ny=n(64), nx=n(128), nz=n(64), single=rng.random() < 0.5)


# ---- inputs ---------------------------------------------------------------
def _element_grid(mesh):
    """(ey, ex, ez) of the solid elements in compact order."""
    lv = mesh.info()[0]
    g = mesh.get(0, "eleMapBack").astype(np.int64) - 1
    return g % lv["resY"], (g // lv["resY"]) % lv["resX"], g // (lv["resY"] * lv["resX"])


def _smooth(ey, ex, ez, seed):
    """A design on its way to members of ten to twenty voxels, densities in [0.3, 0.95]."""
    r = np.random.default_rng(seed)
    fx, fy, fz = r.uniform(0.42, 0.58, 3) * (1 / 3, 1 / 5, 1 / 4)
    px, pz = r.uniform(0, 2 * np.pi, 2)
    return 0.3 + 0.65 * np.sin(fx * ex + px) ** 2 * np.cos(fz * ez + fy * ey + pz) ** 2


def _domain_mask(ny, nx, nz):
    """Three ellipsoids and a bar along x, in proportion to the grid; about a third of it is solid."""
    r = np.random.default_rng(34)
    y, x, z = np.meshgrid(np.arange(ny) + 0.5, np.arange(nx) + 0.5, np.arange(nz) + 0.5, indexing="ij")
    m = np.zeros((ny, nx, nz), bool)
    for _ in range(3):
        c = (r.uniform(0.3, 0.7) * ny, r.uniform(0.25, 0.75) * nx, r.uniform(0.3, 0.7) * nz)
        a = r.uniform(40, 90, 3) * (ny / 192, nx / 384, nz / 192)
        m |= ((y - c[0]) / a[0]) ** 2 + ((x - c[1]) / a[1]) ** 2 + ((z - c[2]) / a[2]) ** 2 <= 1
    return m | ((y - ny / 2) ** 2 + (z - nz / 2) ** 2 <= (30 / 192 * min(ny, nz)) ** 2)


def _four_loads(mesh, patch=50):
    """x = 0 face fixed; four load cases, each spread over a patch of the x = max face."""
    lv = mesh.info()[0]
    NY, NX = lv["resY"] + 1, lv["resX"] + 1
    fwd = mesh.get(0, "nodMapForward")
    act = np.flatnonzero(fwd)
    X = (act // NY) % NX
    fixed = fwd[act[X == 0]]
    face = act[X == X.max()]
    fy, fz = face % NY, face // (NY * NX)
    r = np.random.default_rng(1)
    loads = []
    for d in ((0, -1, 0), (0, 0, 1), (0, 0, -1), (0, 1, 0)):
        c = r.integers(len(face))
        near = np.argsort((fy - fy[c]) ** 2 + (fz - fz[c]) ** 2, kind="stable")[:patch]
        loads.append(np.column_stack([fwd[face[near]], np.tile(np.array(d, float) / len(near), (len(near), 1))]))
    mesh.apply_bc(np.column_stack([fixed, np.ones((len(fixed), 3))]), loads)


@functools.lru_cache(maxsize=4)
def _mesh(ny, nx, nz, control, domain, optcase, sup):
    """The model: a program builds it once and solves on it for every design."""
    mask = _domain_mask(ny, nx, nz) if domain == "irregular" else np.ones((ny, nx, nz), bool)
    m = Mesh(mask, control=control, nu=NU, super_element=sup)
    if domain == "irregular":
        _four_loads(m)
    else:
        m.apply_optcase(optcase)
    return m


@functools.lru_cache(maxsize=1)
def _shared_solver(ny, nx, nz, control, domain, optcase, sup, mixed, tol, omega, rmin):
    """The solver of a model, kept over its designs (every pass that uses it sets the densities first)."""
    s = Solver(_mesh(ny, nx, nz, control, domain, optcase, sup), E0=E0, Emin=EMIN, penal=PENAL, tol=tol, maxIT=4000, omega=omega, mixed=mixed)
    if rmin and sup:
        s.super_filter_setup(rmin)
    elif rmin:
        s.filter_setup(rmin)
    return s


def _box_nodes(ny, nx, nz):
    """[nElem x 8] 1-based node ids of a full box, in the element node order of the library."""
    ey, ex, ez = (a.ravel(order="F") for a in np.meshgrid(np.arange(ny), np.arange(nx), np.arange(nz), indexing="ij"))
    return np.stack([1 + (ey + dy) + (ny + 1) * ((ex + dx) + (nx + 1) * (ez + dz)) for dy, dx, dz in _CORNERS], 1).astype(np.int32)


_CORNERS = [(1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 0), (1, 0, 1), (1, 1, 1), (0, 1, 1), (0, 0, 1)]


def _hex_stiffness(cell):
    """24x24 stiffness of a cube of unit modulus (2x2x2 Gauss points)."""
    lam, mu = NU / ((1 + NU) * (1 - 2 * NU)), 0.5 / (1 + NU)
    D = np.diag([lam + 2 * mu] * 3 + [mu] * 3)
    D[:3, :3] += lam * (1 - np.eye(3))
    xyz = np.array([(dx, 1 - dy, dz) for dy, dx, dz in _CORNERS], float)
    K = np.zeros((24, 24))
    for p in np.ndindex(2, 2, 2):
        g = 0.5 + (np.array(p) - 0.5) / math.sqrt(3.0)
        f, df = np.where(xyz > 0, g, 1 - g), np.where(xyz > 0, 1.0, -1.0)
        N = np.stack([df[:, 0] * f[:, 1] * f[:, 2], f[:, 0] * df[:, 1] * f[:, 2], f[:, 0] * f[:, 1] * df[:, 2]])
        B = np.zeros((6, 24))
        for a in range(8):
            x, y, z = N[:, a]
            B[:, 3 * a:3 * a + 3] = [[x, 0, 0], [0, y, 0], [0, 0, z], [y, x, 0], [0, z, y], [z, 0, x]]
        K += B.T @ D @ B / 8
    return K * cell


def _prolongation(span):
    """[24 x 24 x span^3] trilinear interpolation from a cell's corners to each child's, children y fastest."""
    P = np.zeros((24, 24, span ** 3))
    for s in range(span ** 3):
        o = (s % span, s // span % span, s // span ** 2)
        for i, ci in enumerate(_CORNERS):
            t = [(o[k] + ci[k]) / span for k in range(3)]
            for j, cj in enumerate(_CORNERS):
                w = np.prod([t[k] if cj[k] else 1 - t[k] for k in range(3)])
                for c in range(3):
                    P[3 * i + c, 3 * j + c, s] = w
    return P


def _children(ny, nx, nz, span):
    """[nCoarse x span^3] 1-based child ids of the cells of a box of ny x nx x nz children."""
    cy, cx, cz = (a.ravel(order="F") for a in np.meshgrid(np.arange(ny // span), np.arange(nx // span), np.arange(nz // span), indexing="ij"))
    s = np.arange(span ** 3)
    y, x, z = span * cy[:, None] + s % span, span * cx[:, None] + s // span % span, span * cz[:, None] + s // span ** 2
    return (1 + y + ny * (x + nx * z)).astype(np.int32)


def _galerkin_inputs(case, seed):
    """Moduli, element matrices of the cells on the fixed x = 0 face, the maps and transfer blocks."""
    ny, nx, nz = case["ny"], case["nx"], case["nz"]
    ne = ny * nx * nz
    e = np.arange(ne)
    E = EMIN + _smooth(e % ny, e // ny % nx, e // (ny * nx), seed) ** PENAL * (E0 - EMIN)
    K = _hex_stiffness(1.0 / nx)
    onFace = np.flatnonzero(e // ny % nx == 0)
    mapUnique = np.zeros(ne, np.int32)
    mapUnique[onFace] = 1 + np.arange(len(onFace))
    fixedRows = np.array([3 * i + c for i, (_, dx, _) in enumerate(_CORNERS) if dx == 0 for c in range(3)])
    free = K.copy()
    free[fixedRows, :] = 0
    free[:, fixedRows] = 0
    y, z = onFace % ny, onFace // (ny * nx)
    fixed = np.zeros((576, len(onFace)))
    for i, (dy, dx, dz) in enumerate(_CORNERS):
        if dx == 0:     # the fixed diagonal shared by the elements around the node
            share = np.where((y + dy > 0) & (y + dy < ny), 2, 1) * np.where((z + dz > 0) & (z + dz < nz), 2, 1)
            for c in range(3):
                fixed[(3 * i + c) * 25] = E0 / share
    return dict(E=E, K0=K.ravel(order="F"), P4=_prolongation(4), P2=_prolongation(2), up1=_children(ny, nx, nz, 4),
                up2=_children(ny // 4, nx // 4, nz // 4, 2), mapUnique=mapUnique,
                uFree=np.repeat(free.ravel(order="F")[:, None], len(onFace), 1), uFixed=fixed)


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


# ---- prepare / run ----------------------------------------------------------
def prepare(case, seed):
    kind, ny, nx, nz = case["kind"], case["ny"], case["nx"], case["nz"]
    r = np.random.default_rng([seed, 7])
    if kind == "gather":
        dt = np.float32 if case["single"] else np.float64
        tt = torch.float32 if case["single"] else torch.float64
        nn, ne = (ny + 1) * (nx + 1) * (nz + 1), ny * nx * nz
        return dict(kind=kind, eNod=mex.gpu_array(_box_nodes(ny, nx, nz)), u=mex.gpu_array(r.standard_normal((nn, 3)).astype(dt)),
                    uMat=mex.zeros((ne, 24), dtype=tt), Y=mex.zeros((nn, 3), dtype=tt))
    if kind == "galerkin":
        dt = np.float32 if case["single"] else np.float64
        tt = torch.float32 if case["single"] else torch.float64
        st = {k: mex.gpu_array(v if v.dtype == np.int32 else v.astype(dt)) for k, v in _galerkin_inputs(case, seed).items()}
        st.update(kind=kind, K1=mex.zeros((24, 24, len(st["up1"])), dtype=tt), K2=mex.zeros((24, 24, len(st["up2"])), dtype=tt))
        return st
    if kind == "super":
        s = _shared_solver(ny, nx, nz, case["control"], "box", 2, 1, case["mixed"], case["tol"], 0.6, math.sqrt(3.0))
        q, e = np.arange(64)[:, None], np.arange(ny * nx * nz)[None, :]
        x = _smooth(4 * (e % ny) + q % 4, 4 * (e // ny % nx) + q // 4 % 4, 4 * (e // (ny * nx)) + q // 16, seed)
        return dict(kind=kind, solver=s, x=_dev(x.ravel(order="F")))
    domain = case.get("domain", "box")
    if kind in ("product", "vcycle", "filter"):      # one design, many calls: a solver of its own
        m = _mesh(ny, nx, nz, case["control"], domain, 1, 0)
        s = Solver(m, E0=E0, Emin=EMIN, penal=PENAL, tol=case["tol"], maxIT=4000, omega=0.6, mixed=case.get("mixed", False))
        x = _dev(_smooth(*_element_grid(m), seed))
        if kind == "filter":
            s.filter_setup(case["rmin"])
            return dict(kind=kind, solver=s, x=x)
        s.set_density(x)
        if kind == "vcycle":
            s.assemble()
        return dict(kind=kind, solver=s, u=_dev(r.standard_normal(s.numDOFs)))
    omega = 0.4 if kind == "adjoint" else 0.6
    rmin = {"step": math.sqrt(3.0), "adjoint": 2.5}.get(kind, 0.0)
    s = _shared_solver(ny, nx, nz, case["control"], domain, 1, 0, case["mixed"], case["tol"], omega, rmin)
    if kind == "optimize":      # the loop starts from a uniform design; its volume fraction is the user's input
        return dict(kind=kind, solver=s, V0=0.12 + 0.2 * float(r.random()), loops=case["loops"], ft=case["ft"])
    if kind == "adjoint":
        x = _dev(0.05 + 0.95 * r.random(s.num_design))
        loaded = np.flatnonzero(s.mesh.get(0, "F"))
        return dict(kind=kind, solver=s, x=x, dof=int(loaded[len(loaded) // 2]), tol=case["tol"])
    return dict(kind=kind, solver=s, x=_dev(_smooth(*_element_grid(s.mesh), seed)))


def run(state):
    kind = state["kind"]
    if kind == "gather":
        state["Y"].zero_()
        mex.Gathering_inplace(state["uMat"], state["u"], state["eNod"])
        mex.Scattering_inplace(state["Y"], state["eNod"], state["uMat"])
        return state["uMat"], state["Y"]
    if kind == "galerkin":
        mex.assembleKs_level2_inplace(state["K1"], state["up1"], state["E"], state["K0"], state["P4"], state["mapUnique"],
                                      state["uFree"], state["uFixed"])
        mex.assembleKs_higherLevel_inplace(state["K2"], state["up2"], state["K1"], state["P2"])
        return state["K1"], state["K2"]
    s = state["solver"]
    if kind == "product":
        return s.matvec(0, state["u"])
    if kind == "vcycle":
        return s.vcycle(state["u"])
    if kind == "filter":
        return s.filter(state["x"])[0]
    if kind == "optimize":
        x, rows, c = s.optimize(V0=state["V0"], rMin=math.sqrt(3.0), nLoop=state["loops"], ft=state["ft"])
        return x, c, [[q["c"], q["vol"]] for q in rows]
    if kind == "adjoint":
        g, J, _ = s.sensitivity(state["x"], "displacement", dof=state["dof"], ft=2, tol=state["tol"])
        return g, J
    x = s.super_filter(state["x"], 1) if kind == "super" else state["x"]
    s.set_density(x)
    s.assemble()
    if kind == "super":
        return x, s.pcg(0)[0]
    U = s.pcg_all()[0]
    if kind == "state":
        return U
    ce = s.unit_compliance(U)
    return U, ce, s.filter(ce)[0]


# ---- what a pass cannot do without -------------------------------------------
_ITERATIONS = {"state": 40, "super": 60, "step": 40, "adjoint": 60}      # CG iterations of a solve, about


def work(case):
    kind, ny, nx, nz = case["kind"], case["ny"], case["nx"], case["nz"]
    ne, nn = ny * nx * nz, (ny + 1) * (nx + 1) * (nz + 1)
    w = 4 if case.get("single") else 8
    if kind == "gather":
        return dict(bytes=2 * (32 * ne + 3 * nn * w + 24 * ne * w), flops=24 * ne)
    if kind == "galerkin":
        n1 = ne // 64
        return dict(bytes=ne * (w + 4) + n1 * (64 * 4 + 2 * 576 * w) + n1 // 8 * (32 + 576 * w), flops=n1 * 2 * 64 * 576 + n1 * 4 * 24 ** 3)
    if kind == "filter":        # about ten conjugate-gradient steps on one value a node
        return dict(bytes=16 * ne + 10 * 8 * 8 * nn, flops=10 * nn * 140)
    loads, sub = (4, 1) if case.get("domain") == "irregular" else (1, 1)
    if case.get("domain") == "irregular":
        ne, nn = ne // 3, nn // 3
    prod_b, prod_f = 8 * (6 * nn + ne), 190 * ne
    if kind == "super":
        prod_b, prod_f = 8 * (6 * nn + 300 * ne), 1152 * ne
    if kind == "product":
        return dict(bytes=prod_b, flops=prod_f)
    if kind == "vcycle":
        return dict(bytes=2 * prod_b + 8 * 9 * nn, flops=2.5 * prod_f)
    v = 0.5 if case["mixed"] else 1.0       # the V-cycle's share at its precision
    per = loads * (prod_b + 8 * 3 * nn * 8 + v * (2 * prod_b + 8 * 9 * nn))
    its = _ITERATIONS.get(kind, 0)
    if kind == "optimize":
        its = 30 * (case["loops"] + 1)
    if kind == "adjoint":
        its *= 2
    return dict(bytes=its * per, flops=its * loads * 3.5 * prod_f)


# ---- the outputs in 64 bits ----------------------------------------------------
def _box_product(ny, nx, nz, E, eNod, K, fixedNodes):
    """u -> K(E) u on a box, fixed nodes' rows E0 u and out of the other rows."""
    def apply(u):
        v = u.clone()
        v[fixedNodes] = 0
        y = torch.zeros_like(v)
        for a in range(0, len(eNod), 1 << 18):
            n = eNod[a:a + (1 << 18)]
            f = (v[n].reshape(-1, 24) @ K) * E[a:a + (1 << 18), None]
            y.index_add_(0, n.reshape(-1), f.reshape(-1, 3))
        y[fixedNodes] = E0 * u[fixedNodes]
        return y
    return apply


def _box_setup(case, seed):
    ny, nx, nz = case["ny"], case["nx"], case["nz"]
    e = np.arange(ny * nx * nz)
    x = _dev(_smooth(e % ny, e // ny % nx, e // (ny * nx), seed))
    E = EMIN + x ** PENAL * (E0 - EMIN)
    eNod = _dev(_box_nodes(ny, nx, nz).astype(np.int64) - 1)
    node = np.arange((ny + 1) * (nx + 1) * (nz + 1))
    fixed = _dev(np.flatnonzero(node // (ny + 1) % (nx + 1) == 0))
    return x, E, eNod, fixed


def _cg(apply, b, invD, tol):
    x = torch.zeros_like(b)
    r = b.clone()
    z = invD * r
    p = z.clone()
    rho, nb = (r * z).sum(), float(b.norm())
    for k in range(20000):
        q = apply(p)
        a = rho / (p * q).sum()
        x += a * p
        r -= a * q
        if k % 20 == 0 and float(r.norm()) < tol * nb:
            break
        z = invD * r
        new = (r * z).sum()
        p = z + (new / rho) * p
        rho = new
    return x


def _exact_filter(x, eNod, nn, rmin):
    """The Helmholtz filter of the reference: nodal, its derivatives in the [-1, 1] coordinates of the element."""
    s = np.array([(-1, -1, -1), (1, -1, -1), (1, 1, -1), (-1, 1, -1), (-1, -1, 1), (1, -1, 1), (1, 1, 1), (-1, 1, 1)], float)
    K = np.zeros((8, 8))
    for p in np.ndindex(2, 2, 2):
        f = 1 + s * ((np.array(p) * 2 - 1) / math.sqrt(3.0))
        N = f.prod(1) / 8
        dN = np.stack([s[:, k] * np.delete(f, k, 1).prod(1) / 8 for k in range(3)])
        K += (rmin / 2 / math.sqrt(3.0)) ** 2 * dN.T @ dN + np.outer(N, N) / 8
    Kd = _dev(K)
    diag = torch.zeros(nn, dtype=torch.float64, device="cuda").index_add_(0, eNod.reshape(-1), Kd.diagonal().repeat(len(eNod)))

    def apply(v):
        return torch.zeros_like(v).index_add_(0, eNod.reshape(-1), (v[eNod] @ Kd).reshape(-1))
    rhs = torch.zeros_like(diag).index_add_(0, eNod.reshape(-1), (x / 8).repeat_interleave(8))
    return _cg(apply, rhs, 1 / diag, 1e-14)[eNod].mean(1)


def exact(case, seed):
    kind, ny, nx, nz = case["kind"], case["ny"], case["nx"], case["nz"]
    nn = (ny + 1) * (nx + 1) * (nz + 1)
    r = np.random.default_rng([seed, 7])
    if kind == "gather":
        dt = np.float32 if case["single"] else np.float64
        u = _dev(r.standard_normal((nn, 3)).astype(dt).astype(np.float64))
        eNod = _dev(_box_nodes(ny, nx, nz).astype(np.int64) - 1)
        m = u[eNod].reshape(-1, 24)
        Y = torch.zeros_like(u).index_add_(0, eNod.reshape(-1), m.reshape(-1, 3))
        return m, Y
    if kind == "galerkin":
        q = _galerkin_inputs(case, seed)
        if case["single"]:      # the values the single gateways are given
            q = {k: v if v.dtype == np.int32 else v.astype(np.float32).astype(np.float64) for k, v in q.items()}
        d = {k: _dev(v) for k, v in q.items()}
        mat = lambda v: v.reshape(24, 24, -1).permute(2, 1, 0)  # noqa: E731  column-major 24x24 per column
        K0, free, fixed = mat(d["K0"]), mat(d["uFree"]), mat(d["uFixed"])
        K1 = torch.zeros(len(q["up1"]), 24, 24, dtype=torch.float64, device="cuda")
        for s in range(64):
            f = d["up1"][:, s].long() - 1
            u = d["mapUnique"][f].long() - 1
            K = K0 * d["E"][f, None, None]
            on = u >= 0
            K[on] = free[u[on]] * d["E"][f[on], None, None] + fixed[u[on]]
            P = d["P4"][:, :, s]
            K1 += P.T @ K @ P
        K2 = torch.zeros(len(q["up2"]), 24, 24, dtype=torch.float64, device="cuda")
        for s in range(8):
            P = d["P2"][:, :, s]
            K2 += P.T @ K1[d["up2"][:, s].long() - 1] @ P
        return K1.permute(1, 2, 0), K2.permute(1, 2, 0)
    if kind == "product":
        _, E, eNod, fixed = _box_setup(case, seed)
        u = _dev(r.standard_normal(3 * nn)).reshape(-1, 3)
        return _box_product(ny, nx, nz, E, eNod, _dev(_hex_stiffness(1.0 / nx)), fixed)(u).reshape(-1)
    if kind == "filter":
        x, _, eNod, _ = _box_setup(case, seed)
        return _exact_filter(x, eNod, nn, case["rmin"])
    if kind == "state" and case["domain"] == "box" and ny * nx * nz <= 40000:
        _, E, eNod, fixed = _box_setup(case, seed)
        K = _dev(_hex_stiffness(1.0 / nx))
        b = torch.zeros(nn, 3, dtype=torch.float64, device="cuda")
        zt = int(math.floor(nz / 6.0 + 1.5))
        z, y = np.meshgrid(np.arange(zt), np.arange(ny + 1), indexing="ij")
        b[_dev((y + (ny + 1) * (nx + (nx + 1) * z)).ravel()), 2] = -1.0 / z.size
        diag = torch.zeros_like(b).index_add_(0, eNod.reshape(-1), (E[:, None] * K.diagonal()).reshape(-1, 3))
        diag[fixed] = E0
        return _cg(_box_product(ny, nx, nz, E, eNod, K, fixed), b, 1 / diag, 1e-13).reshape(-1)
    return None
