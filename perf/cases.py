"""The work that a user of this library has it do, as timed cases.

A case is a dict of plain values.  `listed()` gives the fixed cases, `draw(rng)`
one more of the same ranges, `prepare(case, seed)` what a program has in hand
before the call (mesh, loads, a context with its mesh set up), `run(state)` one
pass through the public entry points, `work(case)` the bytes and operations
that a pass cannot do without and `exact(case, seed)` the outputs in 64 bits
from plain torch.

Kinds of work:
  ke      batched element stiffness on host arrays (GpuContext.element_ke)
  static  solve_linear on a host model: upload, pattern, assembly, solve, u back
  block   a mesh kept on the device: assemble, then the two-level mixed solve on
          device vectors (the step of a parameter study or a time loop)
  loads   many load cases on one assembled matrix (solve_batched)
  cubes   many independent meshes in one context (solve_multi)
  simp    compliance and its gradient for a density field (forward, backward)
  recover stresses, strains, von Mises, reactions of a displacement field
  kff     the caller's own triplets (solve_kff), optionally with multi-point
          constraints (solve_reduced)
"""
from __future__ import annotations

import functools
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "axia-fem_gb300")
if os.path.isdir(_PKG) and _PKG not in sys.path:
    sys.path.insert(0, _PKG)
if os.path.isdir("axia-fem_gb300") and os.path.abspath("axia-fem_gb300") not in sys.path:
    sys.path.insert(0, os.path.abspath("axia-fem_gb300"))

DEV = "cuda"
NU = 0.3
E_STEEL = 210000.0
RTOL = 1e-10


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def listed():
    return [
        # the smallest call: stiffness matrices of one group of quadratic bricks
        dict(name="ke_c3d20_37", kind="ke", nn=20, reduced=0, n=37),
        # a small cantilever from host arrays in the default FP64 backend: all latency
        dict(name="static_c3d8_20x4x4_fp64", kind="static", nn=8, mixed=0, nx=20, ny=4, nz=4),
        # an ordinary FP64 solve (the reference's algorithm), odd edges
        dict(name="static_c3d8_45x31x23_fp64", kind="static", nn=8, mixed=0, nx=45, ny=31, nz=23),
        # an ordinary tetrahedral model (six per cell) from host arrays, mixed backend
        dict(name="static_c3d10_13x11x12_mixed", kind="static", nn=10, mixed=1, nx=13, ny=11, nz=12),
        # the benchmark block: a million bricks, perturbed, pressure on one face
        dict(name="block_c3d8_100x100x100", kind="block", nn=8, reduced=0, nx=100, ny=100, nz=100),
        # the quadratic block with a random traction on its top face
        dict(name="block_c3d20_50x50x50", kind="block", nn=20, reduced=0, nx=50, ny=50, nz=50),
        # a full batch of 32 load cases on a large block (the largest case)
        dict(name="loads32_c3d8_80x80x80", kind="loads", nn=8, nrhs=32, host=0, nx=80, ny=80, nz=80),
        # a handful of load cases of an ordinary part, host arrays in and out
        dict(name="loads7_c3d8_41x29x23", kind="loads", nn=8, nrhs=7, host=1, nx=41, ny=29, nz=23),
        # a family of 64 uneven cubes solved together
        dict(name="cubes64_10to40", kind="cubes", count=64, lo=10, hi=40, mix=20261203),
        # one iteration of a density optimisation: forward and backward
        dict(name="simp_c3d8_100x50x50", kind="simp", nx=100, ny=50, nz=50),
        # the output step after a large solve
        dict(name="recover_c3d8_100x100x100", kind="recover", nn=8, nx=100, ny=100, nz=100),
        # a caller that builds its own K_ff and hands over the triplets
        dict(name="kff_c3d8_17x16x19", kind="kff", mpc=0, nx=17, ny=16, nz=19),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def _edges(rng, lo, hi, cells):
    """Three edge counts, each spread over its logarithm, with at most `cells` cells; no edge over
    three times another (a slender beam's solution moves by more than the solver's tolerance)."""
    while True:
        n = [_log_int(rng, lo, hi) for _ in range(3)]
        if n[0] * n[1] * n[2] <= cells and max(n) <= 3 * min(n):
            return dict(nx=n[0], ny=n[1], nz=n[2])


def draw(rng):
    kind = rng.choice(["ke", "static", "static", "block", "block", "loads", "loads", "cubes", "simp", "recover", "kff"])
    if kind == "ke":
        return dict(kind=kind, nn=rng.choice([8, 20]), reduced=0, n=_log_int(rng, 1, 3000))
    if kind == "static":
        nn, mixed = rng.choice([(8, 0), (8, 1), (20, 0), (20, 1), (10, 0), (10, 1)])
        return dict(kind=kind, nn=nn, mixed=mixed,
                    **{8: lambda: _edges(rng, 4, 64, 40000), 20: lambda: _edges(rng, 3, 32, 5000),
                       10: lambda: _edges(rng, 3, 20, 2500)}[nn]())
    if kind == "block":
        nn, reduced = rng.choice([(8, 0), (8, 0), (20, 0), (20, 1)])
        return dict(kind=kind, nn=nn, reduced=reduced,
                    **(_edges(rng, 12, 110, 1000000) if nn == 8 else _edges(rng, 7, 55, 125000)))
    if kind == "loads":
        return dict(kind=kind, nn=8, nrhs=rng.choice([2, 3, 7, 13, 24, 32, 33, 45]), host=rng.choice([0, 1]),
                    **_edges(rng, 8, 60, 100000))
    if kind == "cubes":
        lo = rng.randint(3, 12)
        return dict(kind=kind, count=_log_int(rng, 2, 80), lo=lo, hi=rng.randint(lo + 1, 34), mix=rng.randrange(1 << 30))
    if kind == "simp":
        return dict(kind=kind, **_edges(rng, 8, 110, 250000))
    if kind == "recover":
        nn = rng.choice([8, 20])
        return dict(kind=kind, nn=nn, **(_edges(rng, 8, 110, 1000000) if nn == 8 else _edges(rng, 5, 50, 100000)))
    return dict(kind=kind, mpc=rng.choice([0, 1]), **_edges(rng, 3, 30, 7000))


# ---------------------------------------------------------------------------
# models
# ---------------------------------------------------------------------------
@functools.lru_cache(maxsize=4)
def _grid(nx, ny, nz, nn):
    """Unit-cell grid: coords, connectivity and the lattice position of each node."""
    from axia_gpu import meshgen

    if nn == 10:
        return meshgen.structured_tets(nx, ny, nz, nn)
    return meshgen.structured_block(nx, ny, nz, nn)


def _model(nx, ny, nz, nn, seed, reduced=0, perturb=0.1):
    """A block clamped at x = 0 with its inner nodes moved by up to `perturb` cells
    (corner-node elements only: a straight-sided mesh of quadratic ones)."""
    from axia_gpu import meshgen

    coords, conn, lat = _grid(nx, ny, nz, nn)
    top = np.array([nx, ny, nz]) * (1 if nn == 8 else 2)
    rng = np.random.default_rng([seed, 1])
    coords = meshgen.perturb_interior(coords, lat, top, perturb, 1.0, seed) if nn == 8 else coords * rng.uniform(0.8, 1.25, 3)
    clamped = np.nonzero(lat[:, 0] == 0)[0].astype(np.int64)
    bc = (3 * clamped[:, None] + np.arange(3)).ravel()
    n_elem = conn.shape[0]
    m = meshgen.Model("block", coords, conn, nn, np.full(n_elem, E_STEEL), NU, bc, np.zeros(bc.shape[0]),
                      np.zeros(3 * coords.shape[0]), reduced=reduced, shape=(nx, ny, nz))
    if nn == 10:  # nodal forces on the far face
        tip = np.nonzero(lat[:, 0] == top[0])[0]
        m.cload[3 * tip] = rng.uniform(5.0, 15.0, tip.shape[0])
    else:  # pressure on the far face (C3D8: even, C3D20: random per element on the top)
        el = np.arange(n_elem, dtype=np.int64)
        if nn == 8:
            el = el[el % nx == nx - 1]
            face, p = meshgen.FACE_XMAX, np.full(el.shape[0], rng.uniform(0.5, 2.0))
        else:
            el = el[el // (nx * ny) == nz - 1]
            face, p = meshgen.FACE_ZMAX, rng.standard_normal(el.shape[0])
        m.dload_elem, m.dload_face, m.dload_p = el, np.full(el.shape[0], face, np.int32), p
    return m


def _surface_loads(m, seed, nrhs):
    """nrhs force fields on the GPU: each loads 5 % of the surface nodes, N(0, 1) per component."""
    _, _, lat = _grid(*m.shape, m.nn)
    top = np.array(m.shape) * (1 if m.nn == 8 else 2)
    surf = torch.from_numpy(np.nonzero(((lat == 0) | (lat == top)).any(axis=1))[0]).to(DEV)
    g = torch.Generator(device=DEV).manual_seed(int(seed) % (1 << 62))
    k = max(1, round(0.05 * surf.numel()))
    F = torch.zeros(nrhs, m.n_nodes, 3, dtype=torch.float64, device=DEV)
    for r in range(nrhs):
        pick = surf[torch.randperm(surf.numel(), generator=g, device=DEV)[:k]]
        F[r, pick] = torch.randn(k, 3, generator=g, device=DEV, dtype=torch.float64)
    return F.reshape(nrhs, -1)


def _random_elements(nn, n, seed):
    """n distorted elements at random places, and their moduli."""
    from axia_gpu import meshgen

    rng = np.random.default_rng(seed)
    xi = meshgen.HEX20_XI[:nn].astype(np.float64)
    xyz = 0.5 * xi[None] + rng.uniform(-0.08, 0.08, (n, nn, 3)) + rng.uniform(-50.0, 50.0, (n, 1, 3))
    return xyz, rng.uniform(1e3, 2.1e5, n)


def _cube_models(case, seed):
    sizes = np.random.default_rng(case["mix"]).integers(case["lo"], case["hi"] + 1, size=case["count"])
    return [_model(int(n), int(n), int(n), 8, seed + 97 * i, perturb=0.0) for i, n in enumerate(sizes)]


def _rho(case, seed):
    return np.random.default_rng([seed, 2]).uniform(0.3, 1.0, case["nx"] * case["ny"] * case["nz"])


def _simp_model(case, seed):
    m = _model(case["nx"], case["ny"], case["nz"], 8, seed, perturb=0.0)
    _, _, lat = _grid(*m.shape, 8)
    tip = np.nonzero((lat[:, 0] == case["nx"]) & (lat[:, 1] == case["ny"] // 2) & (lat[:, 2] == case["nz"] // 2))[0]
    f = np.zeros(m.ndof)
    f[3 * tip[0] + 2] = -1.0
    return m, f


def _displacement(m, seed):
    """A bent and stretched body with a little noise, and a load field."""
    rng = np.random.default_rng([seed, 3])
    x = m.coords / np.asarray(m.shape).max()
    c = rng.uniform(-1e-3, 1e-3, (3, 6))
    basis = np.stack([x[:, 0], x[:, 1], x[:, 2], x[:, 0] ** 2, x[:, 0] * x[:, 1], x[:, 0] * x[:, 2]], axis=1)
    u = basis @ c.T + rng.standard_normal(x.shape) * 1e-7
    return np.ascontiguousarray(u.ravel()), rng.standard_normal(m.ndof)


def _kff_problem(case, seed):
    """Full-DOF element triplets of a brick mesh in element order, Ke row-major."""
    m = _model(case["nx"], case["ny"], case["nz"], 8, seed)
    ke, _ = _stiffness(m)
    d = (3 * m.conn[:, :, None].astype(np.int64) + np.arange(3)).reshape(m.n_elem, -1)
    i = np.repeat(d, 24, axis=1).ravel()
    j = np.tile(d, (1, 24)).ravel()
    f = np.random.default_rng([seed, 4]).standard_normal(m.ndof)
    return m, i, j, ke.cpu().numpy().ravel(), f


def _ties(m):
    """The far face's z displacements follow one of its nodes (a rigid platen)."""
    _, _, lat = _grid(*m.shape, 8)
    tip = np.nonzero(lat[:, 0] == m.shape[0])[0]
    return int(tip[0]), tip[1:]


# ---------------------------------------------------------------------------
# prepare and run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    from axia_gpu import GpuContext, SparseBackend
    from axia_gpu import _lib as L

    kind = case["kind"]
    st = dict(kind=kind, case=case, ctx=GpuContext(0), L=L)
    ctx = st["ctx"]
    if kind == "ke":
        st["xyz"], st["e"] = _random_elements(case["nn"], case["n"], seed)
        return st
    if kind == "static":
        st["model"] = _model(case["nx"], case["ny"], case["nz"], case["nn"], seed)
        st["backend"] = SparseBackend.GpuMixed if case["mixed"] else SparseBackend.Gpu
        return st
    mixed = dict(rtol=RTOL, precision=L.PREC_MIXED, refine_mode=L.REFINE_RELIABLE, inner_rtol=0.01,
                 matrix_format=L.FORMAT_BSR3, preconditioner=L.PRECOND_COARSE)
    st["opts"] = mixed
    if kind == "block":
        m = _model(case["nx"], case["ny"], case["nz"], case["nn"], seed, case["reduced"], perturb=0.15)
        ctx.setup(m)
        st["f"] = torch.from_numpy(ctx.load_vector(m)).to(DEV)
        st["u"] = torch.zeros_like(st["f"])
    elif kind == "loads":
        m = _model(case["nx"], case["ny"], case["nz"], 8, seed)
        ctx.setup(m)
        ctx.assemble_ex(L.ASM_BSR64 | L.ASM_BSR32 | L.ASM_BSR32LO)
        F = _surface_loads(m, seed, case["nrhs"])
        st["opts"] = dict(rtol=RTOL, inner_rtol=0.01, preconditioner=L.PRECOND_COARSE)
        if case["host"]:
            st["F"] = F.cpu().numpy()
        else:
            st["F"], st["U"] = F, torch.zeros_like(F)
    elif kind == "cubes":
        models = _cube_models(case, seed)
        ctx.setup_multi(models)
        ctx.assemble_ex(L.ASM_BSR64 | L.ASM_BSR32)
        st["opts"] = dict(rtol=RTOL, inner_rtol=0.01, preconditioner=L.PRECOND_COARSE)
        st["f"] = torch.cat([_surface_loads(m, seed + i, 1)[0] for i, m in enumerate(models)])
        st["u"] = torch.zeros_like(st["f"])
    elif kind == "simp":
        m, st["load"] = _simp_model(case, seed)
        ctx.setup(m)
        st["rho"] = _rho(case, seed)
        st["opts"] = dict(mixed, rtol=1e-12)
    elif kind == "recover":
        m = _model(case["nx"], case["ny"], case["nz"], case["nn"], seed, perturb=0.15)
        ctx.setup(m)
        u, f = _displacement(m, seed)
        st["u"], st["f"] = torch.from_numpy(u).to(DEV), torch.from_numpy(f).to(DEV)
        z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=DEV)  # noqa: E731
        st["out"] = dict(stress=z(m.n_nodes, 6), strain=z(m.n_nodes, 6), vm=z(m.n_nodes), rf=z(m.ndof),
                         elem=z(m.n_elem, 6))
    elif kind == "kff":
        m, i, j, v, f = _kff_problem(case, seed)
        if case["mpc"]:
            from axia_gpu.dofmap import DofMap

            master, slaves = _ties(m)
            st["map"] = DofMap(m.ndof, m.bc_dof, m.bc_val,
                               [(3 * int(s) + 2, [(3 * master + 2, 1.0)], 0.0) for s in slaves])
            st["trips"], st["rhs"] = (i, j, v), f
        else:
            free = m.free_mask()
            ind = np.full(m.ndof, -1, np.int64)
            ind[free] = np.arange(int(free.sum()))
            keep = (ind[i] >= 0) & (ind[j] >= 0)
            st["n"], st["trips"], st["rhs"] = int(free.sum()), (ind[i[keep]], ind[j[keep]], v[keep]), f[free]
    return st


def run(st):
    kind, ctx, L, case = st["kind"], st["ctx"], st["L"], st["case"]
    if kind == "ke":
        ke, vol = ctx.element_ke(st["xyz"], st["e"], NU, reduced=case["reduced"])
        return {"ke": ke, "vol": vol}
    if kind == "static":
        from axia_gpu import solve_linear

        return {"u": solve_linear(st["model"], backend=st["backend"], rtol=RTOL, ctx=ctx).u}
    if kind == "block":
        ctx.assemble_ex(L.ASM_BSR64 | L.ASM_BSR32)
        ctx.solve_device(st["f"].data_ptr(), st["u"].data_ptr(), **st["opts"])
        return {"u": st["u"]}
    if kind == "loads":
        if case["host"]:
            return {"u": ctx.solve_batched(st["F"], **st["opts"])[0]}
        ctx.solve_batched_device(case["nrhs"], st["F"].data_ptr(), st["U"].data_ptr(), **st["opts"])
        return {"u": st["U"]}
    if kind == "cubes":
        ctx.solve_multi_device(st["f"].data_ptr(), st["u"].data_ptr(), **st["opts"])
        return {"u": st["u"]}
    if kind == "simp":
        u, c, _ = ctx.compliance_forward(st["rho"], 3.0, 1.0, st["load"], **st["opts"])
        return {"u": u, "c": c, "grad": ctx.compliance_backward()}
    if kind == "recover":
        o = st["out"]
        ctx.recover_device(st["u"].data_ptr(), st["f"].data_ptr(), E_STEEL, o["stress"].data_ptr(),
                           o["strain"].data_ptr(), o["vm"].data_ptr(), o["rf"].data_ptr(), o["elem"].data_ptr())
        return o
    if case["mpc"]:
        return {"u": ctx.solve_reduced(st["map"], st["trips"], st["rhs"], rtol=RTOL)[0]}
    return {"u": ctx.solve_kff(st["n"], st["trips"], st["rhs"], rtol=RTOL)[0]}


# ---------------------------------------------------------------------------
# work
# ---------------------------------------------------------------------------
def _counts(case):
    """(elements, nodes, nodes per element, Gauss points, 3x3 node blocks of K)."""
    kind = case["kind"]
    if kind == "cubes":
        ns = np.random.default_rng(case["mix"]).integers(case["lo"], case["hi"] + 1, size=case["count"]).astype(float)
        return float((ns ** 3).sum()), float(((ns + 1) ** 3).sum()), 8, 8, float(((3 * ns + 1) ** 3).sum())
    nn = case.get("nn", 8)
    n = np.array([case["nx"], case["ny"], case["nz"]], float)
    if nn == 8:
        return n.prod(), (n + 1).prod(), 8, 8, (3 * n + 1).prod()
    corner, edge = (n + 1).prod(), sum(n[k] * np.delete(n + 1, k).prod() for k in range(3))
    if nn == 20:
        return n.prod(), corner + edge, 20, 8 if case.get("reduced") else 27, 81 * corner + 51 * edge
    return 6 * n.prod(), (2 * n + 1).prod(), 10, 4, 28 * (2 * n + 1).prod()


def work(case):
    """Inputs read once and outputs written once; the flops of the element stiffness (the
    closed isotropic form on the upper triangle) and, for a solve, of one product with K
    per right-hand side: how many more an iterative solve takes is not the path's own."""
    kind = case["kind"]
    if kind == "ke":
        nn, n = case["nn"], case["n"]
        return {"bytes": 8 * n * (3 * nn + 1 + 9 * nn * nn + 1), "flops": n * _ke_flops(nn, 8 if nn == 8 else 27)}
    ne, nodes, nn, ng, nb = (float(v) for v in _counts(case))
    nn, ng = int(nn), int(ng)
    mesh = ne * (4 * nn + 8) + 24 * nodes
    vec = 24 * nodes
    if kind in ("static", "block"):
        return {"bytes": mesh + 2 * vec, "flops": ne * _ke_flops(nn, ng) + 18 * nb}
    if kind == "loads":  # the assembled matrix (FP32 blocks and columns) is an input
        return {"bytes": 40 * nb + 2 * case["nrhs"] * vec, "flops": 18 * nb * case["nrhs"]}
    if kind == "cubes":
        return {"bytes": 40 * nb + 2 * vec, "flops": 18 * nb}
    if kind == "simp":
        return {"bytes": mesh + 16 * ne + 2 * vec, "flops": ne * (_ke_flops(8, 8) + 1200) + 18 * nb}
    if kind == "recover":
        return {"bytes": mesh + 2 * vec + vec + nodes * 13 * 8 + ne * 48, "flops": ne * ng * (60 * nn + 150)}
    return {"bytes": ne * 576 * 24 + 2 * vec, "flops": 18 * nb}


def _ke_flops(nn, ng):
    return ng * (18 * nn + 60 + 15 * nn + 9 * nn * (nn + 1)) + 9 * nn * (nn + 1)


# ---------------------------------------------------------------------------
# the outputs in 64 bits, from plain torch
# ---------------------------------------------------------------------------
_XI8 = np.array([[-1, -1, -1], [1, -1, -1], [1, 1, -1], [-1, 1, -1], [-1, -1, 1], [1, -1, 1], [1, 1, 1], [-1, 1, 1]], float)
_XI20 = np.concatenate([_XI8, np.array([[0, -1, -1], [1, 0, -1], [0, 1, -1], [-1, 0, -1], [0, -1, 1], [1, 0, 1],
                                        [0, 1, 1], [-1, 0, 1], [-1, -1, 0], [1, -1, 0], [1, 1, 0], [-1, 1, 0]], float)])
_TET_EDGES = [(0, 1), (1, 2), (2, 0), (0, 3), (1, 3), (2, 3)]


def _shape(nn, p):
    """Shape functions at the (possibly complex) point p."""
    x, y, z = p
    if nn == 10:
        l = [1 - x - y - z, x, y, z]
        return np.array([v * (2 * v - 1) for v in l] + [4 * l[a] * l[b] for a, b in _TET_EDGES])
    out = []
    for x0, y0, z0 in _XI8 if nn == 8 else _XI20:
        fx, fy, fz = 1 + x * x0, 1 + y * y0, 1 + z * z0
        if nn == 8:
            out.append(fx * fy * fz / 8)
        elif x0 and y0 and z0:
            out.append(fx * fy * fz * (x * x0 + y * y0 + z * z0 - 2) / 8)
        else:
            out.append((1 - x * x if not x0 else fx) * (1 - y * y if not y0 else fy) * (1 - z * z if not z0 else fz) / 4)
    return np.array(out)


def _gauss(nn, ng):
    if nn == 10:
        a, b = 0.5854101966249685, 0.1381966011250105
        return [(np.array([a if q == k else b for q in (1, 2, 3)]), 1.0 / 24.0) for k in range(4)]
    x, w = np.polynomial.legendre.leggauss(2 if ng == 8 else 3)
    return [(np.array([x[i], x[j], x[k]]), w[i] * w[j] * w[k])
            for i in range(len(x)) for j in range(len(x)) for k in range(len(x))]


def _gradients(nn, p):
    """dN/dxi at p by complex-step differentiation (exact to rounding)."""
    h = 1e-40
    return np.stack([_shape(nn, p + 1j * h * np.eye(3)[q]).imag / h for q in range(3)], axis=1)


def _at_gauss(xyz, nn, ng):
    """For each Gauss point: (dN/dx (n, nn, 3), weight x det (n,))."""
    for p, w in _gauss(nn, ng):
        dn = torch.from_numpy(_gradients(nn, p)).to(xyz)
        jac = torch.einsum("nai,aj->nij", xyz, dn)  # dx_i / dxi_j
        c = torch.stack([torch.linalg.cross(jac[:, :, (k + 1) % 3], jac[:, :, (k + 2) % 3]) for k in range(3)], dim=1)
        det = (jac[:, :, 0] * c[:, 0, :]).sum(1)
        yield torch.einsum("ak,nki->nai", dn, c) / det[:, None, None], w * det


def _element_ke(xyz, e, nn, ng):
    """Stiffness (n, 3nn, 3nn) and volume of elements with node positions xyz (n, nn, 3)."""
    n = xyz.shape[0]
    a = torch.zeros(n, nn * 3, nn * 3, dtype=torch.float64, device=xyz.device)
    vol = torch.zeros(n, dtype=torch.float64, device=xyz.device)
    for g, wd in _at_gauss(xyz, nn, ng):
        v = g.reshape(n, -1)
        a += (wd[:, None] * v)[:, :, None] * v[:, None, :]
        vol += wd
    a = a.reshape(n, nn, 3, nn, 3)
    lam = (e * NU / ((1 + NU) * (1 - 2 * NU)))[:, None, None, None, None]
    mu = (e / (2 * (1 + NU)))[:, None, None, None, None]
    tr = a.diagonal(dim1=2, dim2=4).sum(-1)[:, :, None, :, None]
    ke = lam * a + mu * a.transpose(2, 4) + mu * tr * torch.eye(3, dtype=torch.float64, device=xyz.device)[:, None, :]
    return ke.reshape(n, 3 * nn, 3 * nn), vol


def _stiffness(m, e=None):
    """Ke of all elements of a model and the element DOFs, in chunks on the GPU."""
    conn = torch.from_numpy(m.conn.astype(np.int64)).to(DEV)
    x = torch.from_numpy(np.ascontiguousarray(m.coords)).to(DEV)
    e = torch.from_numpy(m.e_elem if e is None else e).to(DEV)
    ng = {8: 8, 10: 4, 20: 8 if m.reduced else 27}[m.nn]
    nd = 3 * m.nn
    ke = torch.empty(m.n_elem, nd, nd, dtype=torch.float64, device=DEV)
    step = max(1, 20_000_000 // (nd * nd))
    for s in range(0, m.n_elem, step):
        ke[s:s + step] = _element_ke(x[conn[s:s + step]], e[s:s + step], m.nn, ng)[0]
    return ke, (3 * conn[:, :, None] + torch.arange(3, device=DEV)).reshape(m.n_elem, nd)


def _solve(ke, dof, F, free, rep=None, tol=1e-14):
    """U (ndof, k) of K U = F (zero elsewhere than on `free`) by Jacobi CG on the element
    matrices, with true residuals now and then; rep: the DOF that each DOF follows."""
    n, k = F.shape
    ne, nd = dof.shape

    def gather(y):  # T^T y on the free DOFs
        if rep is not None:
            y = torch.zeros_like(y).index_add_(0, rep, y)
        return y * free[:, None]

    def mul(v):
        if rep is not None:
            v = v[rep]
        y = torch.bmm(ke, v[dof.reshape(-1)].reshape(ne, nd, k))
        return gather(torch.zeros_like(v).index_add_(0, dof.reshape(-1), y.reshape(-1, k)))

    d = torch.zeros(n, 1, dtype=torch.float64, device=DEV)
    d.index_add_(0, dof.reshape(-1), ke.diagonal(dim1=1, dim2=2).reshape(-1, 1))
    d = gather(d) if rep is None else _tied_diag(ke, dof, rep, n) * free[:, None]
    inv = torch.where(d != 0, 1.0 / d, torch.ones_like(d))
    b = gather(F)
    x = torch.zeros_like(b)
    bn = b.norm(dim=0).clamp_min(1e-300)
    r = b.clone()
    for _ in range(4):
        z = inv * r
        p, rz = z.clone(), (r * z).sum(0)
        goal = torch.maximum(tol * bn, 1e-9 * r.norm(dim=0))
        for it in range(6000):
            q = mul(p)
            alpha = rz / (p * q).sum(0).clamp_min(1e-300)
            x += alpha * p
            r -= alpha * q
            if it % 20 == 19 and bool((r.norm(dim=0) <= goal).all()):
                break
            z = inv * r
            new = (r * z).sum(0)
            p = z + (new / rz.clamp_min(1e-300)) * p
            rz = new
        r = b - mul(x)
        if bool((r.norm(dim=0) <= 1e-13 * bn).all()):
            break
    return x if rep is None else x[rep]


def _tied_diag(ke, dof, rep, n):
    """Diagonal of T^T K T: the couplings of DOFs of one element that follow the same one."""
    d = torch.zeros(n, 1, dtype=torch.float64, device=DEV)
    r = rep[dof]
    same = r[:, :, None] == r[:, None, :]
    return d.index_add_(0, r.reshape(-1), (ke * same).sum(2).reshape(-1, 1))


def _free(m):
    return torch.from_numpy(m.free_mask().astype(np.float64)).to(DEV)


def _face_forces(m):
    """Consistent forces of the model's face pressures (positive compresses) plus its nodal loads."""
    f = torch.from_numpy(m.cload.copy()).to(DEV)
    if not m.dload_elem.shape[0]:
        return f
    nn = m.nn
    xi = _XI8 if nn == 8 else _XI20
    axis, side = (0, 1.0) if nn == 8 else (2, 1.0)
    x = torch.from_numpy(m.coords).to(DEV)[torch.from_numpy(m.conn[m.dload_elem].astype(np.int64)).to(DEV)]
    p = torch.from_numpy(m.dload_p).to(DEV)
    pts, wts = np.polynomial.legendre.leggauss(2 if nn == 8 else 3)
    t1, t2 = (axis + 1) % 3, (axis + 2) % 3
    fe = torch.zeros(x.shape[0], nn, 3, dtype=torch.float64, device=DEV)
    for i, a in enumerate(pts):
        for j, b in enumerate(pts):
            q = np.zeros(3)
            q[axis], q[t1], q[t2] = side, a, b
            dn = _gradients(nn, q)
            g = [torch.einsum("nai,a->ni", x, torch.from_numpy(dn[:, t].copy()).to(DEV)) for t in (t1, t2)]
            normal = torch.linalg.cross(g[0], g[1])  # outward times area
            shp = torch.from_numpy(_shape(nn, q) * (xi[:, axis] == side)).to(DEV)
            fe -= wts[i] * wts[j] * p[:, None, None] * shp[None, :, None] * normal[:, None, :]
    dof = torch.from_numpy((3 * m.conn[m.dload_elem][:, :, None].astype(np.int64) + np.arange(3)).reshape(-1)).to(DEV)
    return f.index_add_(0, dof, fe.reshape(-1))


def _recovered(m, u, f):
    """Averaged nodal stress, strain, von Mises, K u - f and element means."""
    nn, ng = m.nn, 8 if m.nn == 8 else 27
    conn = torch.from_numpy(m.conn.astype(np.int64)).to(DEV)
    x, u, f = torch.from_numpy(m.coords).to(DEV), torch.from_numpy(u).to(DEV), torch.from_numpy(f).to(DEV)
    pts = np.polynomial.legendre.leggauss(2 if ng == 8 else 3)[0]
    xi = _XI8 if nn == 8 else _XI20
    lag = lambda i, t: np.prod([(t - pts[j]) / (pts[i] - pts[j]) for j in range(len(pts)) if j != i], axis=0)  # noqa: E731
    ext = np.stack([lag(i, xi[:, 0]) * lag(j, xi[:, 1]) * lag(k, xi[:, 2])
                    for i in range(len(pts)) for j in range(len(pts)) for k in range(len(pts))], axis=1)  # (nn, ng)
    ext = torch.from_numpy(ext).to(DEV)
    lam, mu = E_STEEL * NU / ((1 + NU) * (1 - 2 * NU)), E_STEEL / (2 * (1 + NU))
    z = lambda *s: torch.zeros(*s, dtype=torch.float64, device=DEV)  # noqa: E731
    acc, cnt, rf, mean = z(m.n_nodes, 6), z(m.n_nodes, 1), z(m.n_nodes, 3), z(m.n_elem, 6)
    step = 100000
    for s in range(0, m.n_elem, step):
        c = conn[s:s + step]
        ue, fe, sig = u.reshape(-1, 3)[c], 0.0, []
        for g, wd in _at_gauss(x[c], nn, ng):
            h = torch.einsum("nai,naj->nij", ue, g)
            t = lam * (h[:, 0, 0] + h[:, 1, 1] + h[:, 2, 2])[:, None, None] * torch.eye(3, dtype=h.dtype, device=DEV)
            t = t + mu * (h + h.transpose(1, 2))
            fe = fe + wd[:, None, None] * torch.einsum("nai,nij->naj", g, t)
            sig.append(torch.stack([t[:, 0, 0], t[:, 1, 1], t[:, 2, 2], t[:, 0, 1], t[:, 1, 2], t[:, 2, 0]], 1))
        nodal = torch.einsum("am,nmc->nac", ext, torch.stack(sig, dim=1))
        mean[s:s + step] = nodal.mean(1)
        acc.index_add_(0, c.reshape(-1), nodal.reshape(-1, 6))
        cnt.index_add_(0, c.reshape(-1), torch.ones(c.numel(), 1, dtype=torch.float64, device=DEV))
        rf.index_add_(0, c.reshape(-1), fe.reshape(-1, 3))
    a = acc / cnt
    d = a[:, :3] - a[:, [1, 2, 0]]
    strain = ((1 + NU) * a - NU * torch.cat([a[:, :3].sum(1, keepdim=True).expand(-1, 3), 0 * a[:, 3:]], 1)) / E_STEEL
    vm = torch.sqrt(0.5 * (d * d).sum(1) + 3.0 * (a[:, 3:] ** 2).sum(1))
    return dict(stress=a, strain=strain, vm=vm, rf=rf.reshape(-1) - f, elem=mean)


def exact(case, seed):
    kind = case["kind"]
    if kind == "ke":
        xyz, e = _random_elements(case["nn"], case["n"], seed)
        ke, vol = _element_ke(torch.from_numpy(xyz).to(DEV), torch.from_numpy(e).to(DEV), case["nn"],
                              8 if case["nn"] == 8 else 27)
        return {"ke": ke.cpu().numpy(), "vol": vol.cpu().numpy()}
    if kind in ("static", "block"):
        m = _model(case["nx"], case["ny"], case["nz"], case["nn"], seed, case.get("reduced", 0),
                   perturb=0.15 if kind == "block" else 0.1)
        u = _solve(*_stiffness(m), _face_forces(m)[:, None], _free(m))[:, 0]
        return {"u": u if kind == "block" else u.cpu().numpy()}
    if kind == "loads":
        m = _model(case["nx"], case["ny"], case["nz"], 8, seed)
        if m.n_elem * case["nrhs"] > 2_000_000:  # over 20 seconds of FP64 products
            return None
        U = _solve(*_stiffness(m), _surface_loads(m, seed, case["nrhs"]).T.contiguous(), _free(m)).T.contiguous()
        return {"u": U.cpu().numpy() if case["host"] else U}
    if kind == "cubes":
        parts = []
        for i, m in enumerate(_cube_models(case, seed)):
            parts.append(_solve(*_stiffness(m), _surface_loads(m, seed + i, 1).T.contiguous(), _free(m))[:, 0])
        return {"u": torch.cat(parts)}
    if kind == "simp":
        m, f = _simp_model(case, seed)
        rho = _rho(case, seed)
        ke, dof = _stiffness(m, rho ** 3)
        f = torch.from_numpy(f).to(DEV)
        u = _solve(ke, dof, f[:, None], _free(m))[:, 0]
        ue = u[dof]
        energy = (torch.bmm(ke, ue[:, :, None])[:, :, 0] * ue).sum(1)
        grad = -3.0 * energy / torch.from_numpy(rho).to(DEV)
        return {"u": u.cpu().numpy(), "c": float(f @ u), "grad": grad.cpu().numpy()}
    if kind == "recover":
        m = _model(case["nx"], case["ny"], case["nz"], case["nn"], seed, perturb=0.15)
        return _recovered(m, *_displacement(m, seed))
    m, _, _, _, f = _kff_problem(case, seed)
    ke, dof = _stiffness(m)
    rep, free = None, _free(m)
    if case["mpc"]:
        master, slaves = _ties(m)
        rep = torch.arange(m.ndof, device=DEV)
        sl = torch.from_numpy(3 * slaves + 2).to(DEV)
        rep[sl] = 3 * master + 2
        free[sl] = 0.0
    u = _solve(ke, dof, torch.from_numpy(f).to(DEV)[:, None], free, rep)[:, 0].cpu().numpy()
    return {"u": u if case["mpc"] else u[m.free_mask()]}
