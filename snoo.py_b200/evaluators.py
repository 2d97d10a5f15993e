"""Field-map evaluation with the reference's interface (``snoopy/evaluators.py``).

Points are located on the device mesh index (``mesh_index.MeshIndex``: bucket grid + barycentric
test) instead of gmsh's ``get_element_by_coordinates``; ``gmsh_model`` is the ``TetMesh`` the
solvers use.  A point counts as inside the volumes ``vol_tags`` when the element holding it
belongs to one of them (the reference asks gmsh's ``is_inside`` per volume first).
"""

import numpy as np

from . import _lib
from . import finite_element as fe
from .curl_curl_assembler import CurlCurlAssembler
from .device import torch, upload, zeros
from .fem_c import biot_savart_device
from .racetrack_coil import RacetrackCoil


# the methods that have a form on the device
_RACETRACK_B = RacetrackCoil.compute_B
_NODAL_FIELDS = CurlCurlAssembler.compute_nodal_fields


def _method_of(obj, name):
    """The plain function behind a method bound to ``obj`` itself, else None."""
    method = getattr(obj, name)
    return getattr(method, "__func__", None) if getattr(method, "__self__", None) is obj else None


def _nodal_fields(assembler, x, tag):
    """``assembler.compute_nodal_fields(x, [tag])`` as a CUDA tensor [N, 3]."""
    if _method_of(assembler, "compute_nodal_fields") is _NODAL_FIELDS:
        return assembler.nodal_fields_device(x, [tag])
    return upload(assembler.compute_nodal_fields(x, [tag]), np.float64).view(-1, 3)


def _located(mesh, positions, vol_tags):
    """Device element ids (-1 outside the volumes), barycentric coordinates and the index of
    each point's volume in ``vol_tags`` (-1 outside)."""
    pts = upload(np.asarray(positions, dtype=np.float64).reshape(-1, 3), np.float64)
    elem, bary = mesh.index().locate_device(pts)
    el = elem.cpu().numpy().astype(np.int64)
    dom = np.full(len(el), -1, dtype=np.int32)
    ok = el >= 0
    tag_of = mesh.elem_domain[el[ok]]
    found = np.full(len(tag_of), -1, dtype=np.int32)
    for i, t in enumerate(vol_tags):  # a repeated tag: its last position
        found[tag_of == t] = i
    dom[ok] = found
    el[dom < 0] = -1
    return upload(el, np.int32), bary, upload(dom, np.int32), el


def evaluate_curl_curl_solution(positions, gmsh_model, vol_tags, solution, glob_ids=None):
    """B = curl A at ``positions`` [M, 3] inside the volumes ``vol_tags`` (0 elsewhere), for the
    vector potential ``solution`` (``evaluators.py:155-295``).  ``glob_ids`` is accepted for the
    reference's signature; the mesh's own edge ids are used."""
    mesh = gmsh_model
    el_d, _, _, _ = _located(mesh, positions, vol_tags)
    n = int(el_d.numel())
    w, q = fe.quadrature_rule(1)
    d_phi = upload(fe.evaluate_basis_derivative(q), np.float64)
    curls, n_orient = fe.curl_edge_basis_functions(q)
    curls_d = upload(curls, np.float64)
    nodes_d = upload(mesh.nodes, np.float64)
    cells_d, gids_d, or_d = (upload(mesh.cells, np.int32), upload(mesh.elem_edges, np.int32),
                             upload(mesh.orientations, np.int32))
    x_d = solution if hasattr(solution, "data_ptr") else upload(solution, np.float64)
    B = zeros(3 * n)
    _lib.call("snp_b_at_elements", n, _lib.ptr(el_d), _lib.ptr(nodes_d), _lib.ptr(cells_d), _lib.ptr(gids_d),
              _lib.ptr(or_d), _lib.ptr(curls_d), n_orient, _lib.ptr(d_phi), len(w), _lib.ptr(x_d), _lib.ptr(B),
              _lib.stream_ptr())
    return B[: 3 * n].cpu().numpy().reshape(-1, 3)


def evaluate_interpolation(positions, gmsh_model, vol_tags, nodal_values):
    """Linear interpolation of nodal values at ``positions`` (``evaluators.py:297-410``):
    a point in volume ``vol_tags[j]`` interpolates ``nodal_values[j]`` ([N] or [N, C]).
    Returns [M, C] (C = 1 for scalar values); 0 outside the volumes."""
    mesh = gmsh_model
    t = torch()
    el_d, bary, dom_d, _ = _located(mesh, positions, vol_tags)
    first = nodal_values[0] if hasattr(nodal_values[0], "data_ptr") else np.asarray(nodal_values[0])
    nc = 1 if first.ndim == 1 else int(first.shape[1])
    stack = []
    for v in nodal_values:
        v_d = v if hasattr(v, "data_ptr") else upload(np.asarray(v, dtype=np.float64), np.float64)
        if int(v_d.numel()) != mesh.num_nodes * nc:
            raise ValueError(f"every nodal value set needs {mesh.num_nodes} x {nc} values")
        stack.append(v_d.reshape(-1))
    nodal_d = t.cat(stack) if len(stack) > 1 else stack[0].contiguous()
    out = mesh.index().interpolate(el_d, bary, nodal_d, nc, len(stack), dom_d)
    return out.cpu().numpy()


def evaluate_fem_solution_node_interpolation(gmsh_model, points, solver, coil_list, x, domain_list):
    """B at ``points`` by interpolating nodal averages (``evaluators.py:413-454``): per domain of
    ``domain_list`` the element fields averaged at the nodes plus the coils' field at the nodes."""
    asm = solver.curl_curl_factory
    nodes_d = upload(asm.nodes, np.float64)
    b_coil = torch().zeros_like(nodes_d)
    for coil in coil_list:
        if _method_of(coil, "compute_B") is _RACETRACK_B:  # the same without the copies to the host and back
            b = biot_savart_device(upload(coil.get_segments(), np.float64), nodes_d, coil.current, coil.rad)
        else:  # any value that broadcasts over the nodes
            b = upload(np.broadcast_to(coil.compute_B(asm.nodes), asm.nodes.shape), np.float64)
        b_coil = b_coil + b[: nodes_d.numel()]
    b_coil = b_coil.view(-1, 3)
    b_node_list = [_nodal_fields(asm, x, indx) + b_coil for indx in domain_list]
    return evaluate_interpolation(points, gmsh_model, domain_list, b_node_list)
