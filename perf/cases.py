"""The work a user of this package has it do, as cases that can be timed and compared.

A design program meshes a magnet, evaluates the coils' source field, assembles and solves the
nonlinear curl-curl system and maps the field; programs that keep snoo.py's own loops call
the assemblers and the ``fem_c`` functions instead.  The cases cover that path through its public
entry points, from the smallest meshes (30k tetrahedra and below, where launches count) to the
1.2M tetrahedra of the headline benchmark, with both precisions of the Newton solver, plain and
diluted steel, quadrature orders 2 (4 points) and the solvers' default 6 (64 points), odd
element counts throughout.  Meshes and materials are the package's own window-frame and
bar-conductor families; a seed draws the DoF vectors, coil currents and iron saturation.

A vector potential is fixed only up to gradients, so whole solves return B = curl A in every
element, driven to a relative residual of 1e-10 so that B is determined to the float64 bounds.
The reference-semantics ``solve`` (CG to 1e-5 per Newton step) leaves its answer undetermined
beyond that level and is represented by its parts: CSR assembly, source field and CSR CG.
"""

import functools
import math

import numpy as np
import torch

import snoopy_b200 as S
from snoopy_b200 import evaluators, fem_c
from snoopy_b200 import finite_element as FE
from snoopy_b200 import materials as MAT
from snoopy_b200 import mesh as M
from snoopy_b200.laplace_subdomain_solver import LaplaceSubdomainSolver

NU0 = 0.25 / math.pi * 1e7


def listed():
    return [
        # a snoo.py program's own loop over fem_c with host arrays, on a small iron domain
        {"name": "fem_c_12k", "kind": "fem_c", "tets": 12000, "order": 2},
        # the drop-in assembler, matrices left on the GPU: a mid-size mesh, the headline mesh, and
        # diluted steel at the default quadrature order
        {"name": "csr_40k", "kind": "csr", "tets": 40000, "order": 2, "diluted": False},
        {"name": "csr_1160k", "kind": "csr", "tets": 1164240, "order": 2, "diluted": False},
        {"name": "csr_diluted_150k", "kind": "csr", "tets": 150000, "order": 6, "diluted": True},
        # scalar-potential Newton matrices with a B-spline permeability
        {"name": "gradgrad_300k", "kind": "gradgrad", "tets": 300000, "order": 4},
        # the electric potential of a conductor: grad-grad assembly and CSR CG to 1e-14
        {"name": "laplace_200k", "kind": "laplace", "tets": 200000},
        # the coils' field at the iron's quadrature points, evaluated anew for every solve
        {"name": "source_1160k", "kind": "source", "tets": 1164240, "order": 2},
        # one inexact Newton step from zero (assembly, block-Jacobi CG, line search): a small mesh,
        # mixed precision at the default quadrature order, the headline mesh
        {"name": "newton_step_35k", "kind": "newton_step", "tets": 38000, "order": 2, "precision": "fp64"},
        {"name": "newton_step_mixed_290k", "kind": "newton_step", "tets": 300000, "order": 6, "precision": "mixed"},
        {"name": "newton_step_1160k", "kind": "newton_step", "tets": 1164240, "order": 2, "precision": "fp64"},
        # the headline solve, whole
        {"name": "solve_1160k", "kind": "solve", "tets": 1164240, "order": 2, "precision": "fp64"},
        # B along a path through the solved magnet by nodal averages, as the field-map drivers do
        {"name": "field_map_290k", "kind": "field_map", "tets": 300000, "points": 20000},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fem_c", "csr", "csr", "gradgrad", "laplace", "source", "newton_step", "newton_step", "solve",
                       "field_map"])
    case = {"kind": kind}
    if kind == "fem_c":
        case.update(tets=_log(rng, 3000, 60000), order=rng.choice([1, 2, 3]))
    elif kind == "csr":
        diluted = rng.random() < 0.3
        case.update(tets=_log(rng, 10000, 300000 if diluted else 1150000), order=rng.choice([2, 2, 3, 6]) if not diluted
                    else rng.choice([2, 6]), diluted=diluted)
        if case["order"] == 6:
            case["tets"] = min(case["tets"], 200000 + case["tets"] % 1000)
    elif kind == "gradgrad":
        case.update(tets=_log(rng, 20000, 900000), order=rng.choice([2, 4, 8]))
    elif kind == "laplace":
        case.update(tets=_log(rng, 20000, 300000))
    elif kind == "source":
        case.update(tets=_log(rng, 20000, 1150000), order=rng.choice([1, 2, 3]))
    elif kind == "newton_step":
        case.update(tets=_log(rng, 20000, 1150000), order=2, precision=rng.choice(["fp64", "mixed"]))
        if case["tets"] < 200000:
            case["order"] = rng.choice([2, 6])
    elif kind == "solve":
        case.update(tets=_log(rng, 20000, 900000), order=2, precision=rng.choice(["fp64", "mixed"]))
    else:
        case.update(tets=_log(rng, 20000, 400000), points=_log(rng, 500, 50000))
    return case


# ---------------------------------------------------------------- inputs


@functools.lru_cache(maxsize=4)
def _mesh(tets):
    """The window-frame mesh of about ``tets`` tetrahedra (the solvers' benchmark family)."""
    return M.window_frame_mesh(tets, jitter=0.15, seed=7)


@functools.lru_cache(maxsize=4)
def _bar_mesh(tets):
    return M.bar_conductor_mesh(tets, seed=3)


def _potential(msh, rng):
    """Edge DoFs of a smooth field of a tesla or so and a few per cent of noise, the size of a
    Newton iterate: the line integral of A = B0 x r / 2 along every edge."""
    b0 = rng.normal(0.0, 0.7, 3)
    p0, p1 = msh.nodes[msh.edges[:, 0]], msh.nodes[msh.edges[:, 1]]
    x = ((0.25 * np.cross(b0, p0 + p1)) * (p1 - p0)).sum(1)
    return x + rng.normal(0.0, 0.03 * np.abs(x).max(), len(x))


def _iron(rng):
    return MAT.atan_reluctance(mu_r=rng.uniform(1000.0, 5000.0), Js=rng.uniform(1.6, 2.1))


def _coils(msh, rng):
    g = msh.geometry
    coils = g.coils()
    scale = rng.uniform(0.4, 1.6)
    for c in coils:
        c.current *= scale
    return coils


def _dilution():
    return MAT.Dilution(0.0, 0.30, 0.35, 0.75, 0.02, 0.40, 0.45, 0.80, z_pos=-0.25, z_len=0.5, mag_type=1)


def _inputs(case, seed):
    """Host inputs of a case, from the seed alone."""
    rng = np.random.default_rng([int(seed), int(case["tets"])])
    kind = case["kind"]
    if kind == "laplace":
        return {"mesh": _bar_mesh(case["tets"]), "phi": rng.uniform(0.2, 3.0) * (1.0 if rng.random() < 0.5 else -1.0)}
    msh = _mesh(case["tets"])
    d = {"mesh": msh, "rel": _iron(rng), "coils": _coils(msh, rng)}
    if kind in ("fem_c", "csr", "field_map"):
        d["x"] = _potential(msh, rng)
    if kind in ("fem_c", "csr"):
        nq = len(FE.quadrature_rule(case["order"])[0])
        n_iron = len(msh.domain_elements(M.TAG_IRON))
        # the coils' field: a smooth part and its variation over the iron
        d["B_s"] = rng.normal(0.0, 0.3, 3) + rng.normal(0.0, 0.1, (n_iron * nq, 3))
    if kind == "gradgrad":
        h = rng.normal(0.0, 1.0, 3)
        h *= 10.0 ** rng.uniform(1.5, 4.0) / np.linalg.norm(h)
        v = msh.nodes @ h
        d["x"] = v + rng.normal(0.0, 0.02 * np.abs(v).max(), len(v))
        d["mu"] = MAT.atan_permeability(mu_r=rng.uniform(1000.0, 5000.0), Js=rng.uniform(1.6, 2.1))
    if kind == "field_map":
        e = np.sort(rng.integers(0, msh.num_elements, case["points"]))
        bary = rng.dirichlet(np.full(4, 2.0), len(e))
        d.update(elements=e, bary=bary, points=np.einsum("pi,pid->pd", bary, msh.nodes[msh.cells[e]]))
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    kind, msh = case["kind"], d["mesh"]
    s = {"kind": kind}
    if kind == "laplace":
        t1, t2 = msh.coil_terminals[M.TAG_COIL_1]
        s.update(solver=LaplaceSubdomainSolver(msh, M.TAG_COIL_1, (t1, t2)), phi=d["phi"])
        s["solver"].matrix_factory.pattern
        return s
    if kind == "fem_c":
        w, q = FE.quadrature_rule(case["order"])
        el = msh.domain_elements(M.TAG_IRON)
        curls, _ = FE.curl_edge_basis_functions(q)
        s["args"] = (msh.nodes, msh.cells[el], msh.elem_edges[el], curls, FE.evaluate_basis_derivative(q),
                     msh.orientations[el], d["x"], d["B_s"], d["rel"], q, w, msh.num_dofs, 6)
        return s
    tags = [M.TAG_IRON, M.TAG_AIR]
    if kind == "gradgrad":
        s.update(asm=S.GradGradAssembler(msh, tags), mu=[d["mu"], S.ConstantPermeability(4e-7 * math.pi)],
                 order=case["order"], x=torch.from_numpy(d["x"]).cuda())
        s["asm"].pattern
        return s
    if kind == "csr":
        mats = [d["rel"], S.ConstantReluctance(NU0)]
        asm = (S.CurlCurlAssemblerDiluted(msh, tags, mats, [_dilution(), None]) if case["diluted"]
               else S.CurlCurlAssembler(msh, tags, mats))
        asm.pattern
        asm.tables(case["order"])
        s.update(asm=asm, order=case["order"], x=torch.from_numpy(d["x"]).cuda(),
                 B_s=[torch.from_numpy(d["B_s"].reshape(-1)).cuda(), np.zeros((0, 3))])
        return s
    solver = S.RedMVPSolver(msh, d["coils"], [M.TAG_IRON], [M.TAG_AIR], [d["rel"]], max_newton_iterations=60,
                            quad_order=case.get("order", 2))
    solver.verbose = False
    s.update(solver=solver, precision=case.get("precision"))
    if kind == "field_map":
        solver.curl_curl_factory._device_state()
        msh.index()
        s.update(mesh=msh, coils=d["coils"], points=d["points"], x=torch.from_numpy(d["x"]).cuda())
    else:
        s["eng"] = solver.newton_engine()
    return s


def run(s):
    kind = s["kind"]
    if kind == "fem_c":
        K, dK, rhs = fem_c.compute_stiffness_and_jacobi_matrix_curl_curl(*s["args"])
        return {"indptr": K.indptr, "indices": K.indices, "K": K.data, "dK": dK.data, "rhs": rhs}
    if kind == "csr":
        K, J, rhs = s["asm"].compute_stiffness_and_jacobi_matrix_c(s["x"], quad_order=s["order"],
                                                                   source_fields=s["B_s"], device=True)
        return {"indptr": J.crow_indices(), "indices": J.col_indices(), "K": K.values(), "J": J.values(), "rhs": rhs}
    if kind == "gradgrad":
        K, J = s["asm"].compute_stiffness_and_jacobi_matrix_c(s["x"], s["mu"], quad_order=s["order"], device=True)
        return {"indptr": J.crow_indices(), "indices": J.col_indices(), "K": K.values(), "J": J.values()}
    if kind == "laplace":
        return s["solver"].solve(s["phi"])
    if kind == "source":
        return s["solver"].compute_source_fields(refresh=True)[0]
    if kind == "newton_step":
        x, _ = s["eng"].solve(None, tol=1e-8, max_newton=1, precision={"fp64": 0, "mixed": 1}[s["precision"]],
                              raise_on_failure=False)
        return x
    if kind == "solve":
        x, _ = s["solver"].solve_to_residual(1e-10, precision=s["precision"], return_device=True)
        return s["solver"].curl_curl_factory.element_B_device(x)
    return evaluators.evaluate_fem_solution_node_interpolation(s["mesh"], s["points"], s["solver"], s["coils"], s["x"],
                                                               [M.TAG_IRON, M.TAG_AIR])


def work(case):
    """Bytes and operations a pass cannot do without, from the element count E (1.2 edges and
    0.18 nodes per element, 16 stored entries per edge row and 15 per node row on these meshes)."""
    kind, E = case["kind"], float(case["tets"])
    n, N = 1.2 * E, 0.18 * E
    nnz, nnz_p = 16.2 * n, 15.0 * N
    nq = {1: 1, 2: 4, 3: 5, 4: 27, 6: 64, 8: 125}[case.get("order", 2)]
    iron = 0.22 * E
    mesh = 44.0 * E + 24.0 * N  # cells, edge ids, orientations; nodes
    if kind in ("fem_c", "csr"):
        if kind == "fem_c":  # the iron alone; matrices and their structure come back to the host
            return {"bytes": 0.22 * mesh + 24.0 * nq * iron + 8.0 * n + 20.0 * 0.3 * nnz + 8.0 * n,
                    "flops": iron * (600.0 + 90.0 * nq)}
        return {"bytes": mesh + 24.0 * nq * iron + 8.0 * n + 2 * 8.0 * nnz + 8.0 * n + 2 * (4.0 * nnz + 4.0 * n),
                "flops": E * 600.0 + iron * 90.0 * nq}
    if kind == "gradgrad":
        return {"bytes": 16.0 * E + 32.0 * N + 2 * 8.0 * nnz_p + 2 * (4.0 * nnz_p + 4.0 * N), "flops": E * 400.0}
    if kind == "laplace":  # the bar holds 1/36 of the box; CG iterations as the nodes along it
        its = 2.3 * E ** (1.0 / 3.0)
        return {"bytes": 16.0 * E / 36.0 + 24.0 * N + its * (12.0 * nnz_p / 36.0 + 72.0 * N / 36.0) + 16.0 * N,
                "flops": E / 36.0 * 300.0 + its * nnz_p / 36.0 * 2.0}
    segments = 384.0
    if kind == "source":
        return {"bytes": 16.0 * iron + 24.0 * N + 24.0 * nq * iron, "flops": 45.0 * segments * nq * iron}
    if kind == "field_map":
        P = float(case["points"])
        return {"bytes": mesh + 8.0 * n + 24.0 * E + 2 * 24.0 * N + 48.0 * P, "flops": 45.0 * segments * N + 60.0 * E}
    # Newton: per CG iteration the element operator (DoF words, slots, tensors) and the DoF state
    # (row starts, nine words, the float32 block row); iterations as measured on these meshes
    wd = 8.0 if case["precision"] == "fp64" else 4.0
    it_bytes = E * (48.0 + 6 * wd) + n * (4.0 + 8 * wd + 34.0)
    asm = mesh + 24.0 * nq * iron + 8.0 * n + 6 * wd * E + 16.0 * n
    steps, per = (1.0, 7.0) if kind == "newton_step" else (15.0, 1.8)  # assemblies per step
    total = (2.5 if kind == "newton_step" else 14.3) * E ** (1.0 / 3.0)
    src = 0.0 if kind == "newton_step" else 45.0 * segments * nq * iron
    return {"bytes": steps * per * asm + total * it_bytes, "flops": steps * per * E * 200.0 + total * E * 90.0 + src}


# ---------------------------------------------------------------- the same in 64 bits, plain torch


def _t(a, dtype=torch.float64):
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    return torch.as_tensor(np.ascontiguousarray(a), dtype=dtype, device=dev)


def _jacobian(nodes, cells, dphi):
    """dX/dxi of affine tetrahedra [E, 3, 3], and its determinant."""
    J = torch.einsum("eik,il->ekl", nodes[cells], dphi)
    return J, torch.linalg.det(J)


def _pchip(rel, b):
    """nu and dnu/dB of a piecewise cubic with its last piece continued; 0 below the first knot."""
    if not hasattr(rel, "spl"):
        return torch.full_like(b, rel.value), torch.zeros_like(b)
    c, x = _t(rel.spl.c), _t(rel.spl.x)
    i = (torch.searchsorted(x, b, right=True) - 1).clamp(0, len(x) - 2)
    t = b - x[i]
    c0, c1, c2, c3 = (c[k][i] for k in range(4))
    ok = (b >= x[0]).to(b.dtype)
    return ok * (((c0 * t + c1) * t + c2) * t + c3), ok * ((3 * c0 * t + 2 * c1) * t + c2)


def _curl_terms(nodes, cells, gids, curls, dphi, w, phi, x, B_s, rel, dil):
    """Element matrices K, dK [E, 6, 6] and reduced rhs terms [E, 6] of one material."""
    J, det = _jacobian(nodes, cells, dphi)
    c = torch.einsum("ekl,ejl->ejk", J, curls)
    B = torch.einsum("ejk,ej->ek", c, x[gids]) / det[:, None]
    A = torch.zeros_like(J)
    kfac, r = torch.zeros_like(det), torch.zeros_like(c[:, :, 0])
    for q in range(len(w)):
        bs = B_s[:, q] if B_s is not None else torch.zeros_like(B)
        b = B + bs
        bm = torch.linalg.vector_norm(b, dim=1)
        f = torch.ones_like(bm)
        if dil is not None and B_s is not None:
            z = nodes[cells][:, :, 2] @ phi[q]
            f = (dil.c_num + z * dil.m_num) / (dil.c_den + z * dil.m_den)
        nu, dnu = _pchip(rel, f * bm)
        nu, dnu = f * nu, f * f * dnu
        kfac += nu * w[q] / det
        a = torch.where(bm >= 1e-14, dnu * w[q] / det / bm.clamp_min(1e-300), torch.zeros_like(bm))
        A += a[:, None, None] * b[:, :, None] * b[:, None, :]
        if B_s is not None:
            r += torch.einsum("ejk,ek->ej", c, bs) * ((NU0 - nu) * w[q])[:, None]
    return kfac[:, None, None] * (c @ c.transpose(1, 2)), c @ A @ c.transpose(1, 2), r


def _csr(rows, n, *values):
    """Row pointers, column indices and summed values of element matrices over the DoFs ``rows`` [E, k]."""
    k = rows.shape[1]
    keys = (rows[:, :, None].expand(-1, k, k) * n + rows[:, None, :].expand(-1, k, k)).reshape(-1)
    uniq, inv = torch.unique(keys, return_inverse=True)
    out = [torch.zeros(len(uniq), dtype=torch.float64, device=rows.device).index_add_(0, inv, v.reshape(-1)) for v in values]
    ptr = torch.searchsorted(uniq, torch.arange(n + 1, device=rows.device) * n)
    return ptr, uniq % n, out


def _exact_curl(case, d):
    msh = d["mesh"]
    w, q = FE.quadrature_rule(case["order"])
    tab = _t(FE.curl_edge_basis_functions(q)[0])[:, 0]
    dphi, phi = _t(FE.evaluate_basis_derivative(q))[0], _t(FE.evaluate_basis(q)).reshape(len(w), 4)
    nodes, x, wt = _t(msh.nodes), _t(d["x"]), _t(w)
    parts = [(M.TAG_IRON, d["rel"])] + ([(M.TAG_AIR, S.ConstantReluctance(NU0))] if case["kind"] == "csr" else [])
    K, dK, rows, rhs = [], [], [], torch.zeros(msh.num_dofs, dtype=torch.float64, device=nodes.device)
    for tag, rel in parts:
        el = msh.domain_elements(tag)
        g = _t(msh.elem_edges[el], torch.int64)
        bs = _t(d["B_s"]).reshape(len(el), len(w), 3) if tag == M.TAG_IRON else None
        k, dk, r = _curl_terms(nodes, _t(msh.cells[el], torch.int64), g, tab[_t(msh.orientations[el], torch.int64)],
                               dphi, wt, phi, x, bs, rel, _dilution() if case.get("diluted") else None)
        K.append(k)
        dK.append(dk)
        rows.append(g)
        rhs.index_add_(0, g.reshape(-1), r.reshape(-1))
    K, dK, rows = torch.cat(K), torch.cat(dK), torch.cat(rows)
    second = dK if case["kind"] == "fem_c" else K + dK
    ptr, col, (v, v2) = _csr(rows, msh.num_dofs, K, second)
    out = {"indptr": ptr.int(), "indices": col.int(), "K": v, "dK" if case["kind"] == "fem_c" else "J": v2, "rhs": rhs}
    return out if case["kind"] == "csr" else {k: t.cpu().numpy() for k, t in out.items()}


def _exact_gradgrad(case, d):
    msh = d["mesh"]
    w, q = FE.quadrature_rule(case["order"])
    dphi, nodes, x = _t(FE.evaluate_basis_derivative(q))[0], _t(msh.nodes), _t(d["x"])
    total, K, J, rows = float(np.sum(w)), [], [], []
    for tag, mat in ((M.TAG_IRON, d["mu"]), (M.TAG_AIR, None)):
        cells = _t(msh.cells[msh.domain_elements(tag)], torch.int64)
        Jm, det = _jacobian(nodes, cells, dphi)
        g = torch.einsum("elk,il->eik", torch.linalg.inv(Jm), dphi)
        H = torch.einsum("eik,ei->ek", g, x[cells])
        hm = torch.linalg.vector_norm(H, dim=1)
        if mat is None:
            mu, dmu = torch.full_like(hm, 4e-7 * math.pi), torch.zeros_like(hm)
        else:
            h = hm.cpu().numpy()
            low = h < mat.H_min
            mu, dmu = _t(mat.evaluate_mu(h)), _t(np.where(low, 0.0, mat.evaluate_mu_derivative(h)))
        k = (mu * det * total)[:, None, None] * (g @ g.transpose(1, 2))
        p = torch.einsum("eik,ek->ei", g, H)
        f = torch.where(hm >= 1e-14, dmu * det * total / hm.clamp_min(1e-300), torch.zeros_like(hm))
        dk = f[:, None, None] * p[:, :, None] * p[:, None, :]
        # J adds the running K after every domain: the first domain's K counts twice
        K.append(k)
        J.append(dk + (2.0 if tag == M.TAG_IRON else 1.0) * k)
        rows.append(cells)
    ptr, col, (v, v2) = _csr(torch.cat(rows), msh.num_nodes, torch.cat(K), torch.cat(J))
    return {"indptr": ptr.int(), "indices": col.int(), "K": v, "J": v2}


def _biot_savart(coils, pts):
    """Field of straight filaments, uniform current density inside a filament's core radius."""
    out = torch.zeros_like(pts)
    for c in coils:
        seg = _t(c.get_segments())
        for i in range(0, len(pts), 16384):
            p = pts[i:i + 16384, None, :]
            a, b = seg[None, :, :3] - p, seg[None, :, 3:] - p
            n = seg[None, :, 3:] - seg[None, :, :3]
            la, lb = torch.linalg.vector_norm(a, dim=2), torch.linalg.vector_norm(b, dim=2)
            t = -(a * n).sum(2) / (n * n).sum(2)
            perp = -(a + t[:, :, None] * n)
            dmin = torch.linalg.vector_norm(perp, dim=2)
            inside = ((dmin < c.rad) & (t >= 0) & (t <= 1)) | (la < c.rad) | (lb < c.rad)
            far = torch.linalg.cross(a, b) * ((la + lb) / ((la * lb + (a * b).sum(2)) * la * lb))[:, :, None]
            u = torch.linalg.cross(n.expand_as(perp), perp)
            near = u * (2.0 * dmin / c.rad ** 2 / torch.linalg.vector_norm(u, dim=2))[:, :, None]
            out[i:i + 16384] += c.current * 1e-7 * torch.where(inside[:, :, None], near, far).sum(1)
    return out


def _exact_field_map(d):
    msh = d["mesh"]
    nodes, cells = _t(msh.nodes), _t(msh.cells, torch.int64)
    _, q = FE.quadrature_rule(1)
    tab = _t(FE.curl_edge_basis_functions(q)[0])[:, 0][_t(msh.orientations, torch.int64)]
    J, det = _jacobian(nodes, cells, _t(FE.evaluate_basis_derivative(q))[0])
    B = torch.einsum("ekl,ejl,ej->ek", J, tab, _t(d["x"])[_t(msh.elem_edges, torch.int64)]) / det[:, None]
    coil = _biot_savart(d["coils"], nodes)
    e, bary = _t(d["elements"], torch.int64), _t(d["bary"])
    out = torch.zeros((len(e), 3), dtype=torch.float64, device=nodes.device)
    tag_of = _t(msh.elem_domain, torch.int64)
    for tag in (M.TAG_IRON, M.TAG_AIR):
        sel = tag_of == tag
        at = cells[sel].reshape(-1)
        total = torch.zeros_like(nodes).index_add_(0, at, B[sel].repeat_interleave(4, 0))
        count = torch.zeros(len(nodes), dtype=torch.float64, device=nodes.device).index_add_(0, at, torch.ones_like(at, dtype=torch.float64))
        nodal = total / count.clamp_min(1.0)[:, None] + coil
        mine = tag_of[e] == tag
        out[mine] = torch.einsum("pi,pik->pk", bary[mine], nodal[cells[e[mine]]])
    return out.cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind in ("newton_step", "solve"):
        return None  # hundreds of CG iterations in 64 bits on the host: minutes
    d = _inputs(case, seed)
    if kind in ("fem_c", "csr"):
        return _exact_curl(case, d)
    if kind == "gradgrad":
        return _exact_gradgrad(case, d)
    msh = d["mesh"]
    if kind == "laplace":  # a straight bar between flat terminals: linear along it, 0 outside
        z, inside = msh.nodes[:, 2], msh.domain_nodes_mask(M.TAG_COIL_1)
        return np.where(inside, d["phi"] * z / (z.max() - z.min()), 0.0)
    if kind == "source":
        el = msh.domain_elements(M.TAG_IRON)
        phi = _t(FE.evaluate_basis(FE.quadrature_rule(case["order"])[1])).reshape(-1, 4)
        pts = torch.einsum("qi,eik->eqk", phi, _t(msh.nodes)[_t(msh.cells[el], torch.int64)]).reshape(-1, 3)
        return _biot_savart(d["coils"], pts).reshape(-1)
    return _exact_field_map(d)
