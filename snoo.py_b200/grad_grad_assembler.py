"""``GradGradAssembler`` with the reference's interface (``snoopy/matrix_assembly.py:92-1135``,
duplicated as ``snoopy/grad_grad_assembler.py``), plus the sparse row/column helpers of
``matrix_assembly.py:16-90``.

Nodal P1 assembly of div(mu grad phi) and its Newton Jacobian through the sm_100a kernel
``snp_gradgrad_system``; one CSR pattern over all domains is built once and cached.
"""

import numpy as np

from . import _lib
from . import finite_element as fe
from .device import Pattern, permeability_spec, torch, upload


def recover_full_solution(u, u_g, b):
    """Insert the reduced solution into the lifting vector (``matrix_assembly.py:16-46``)."""
    num_nodes = len(u_g)
    indx_rem = np.delete(np.arange(num_nodes, dtype=np.int64), b)
    u_ret = np.array(u_g, dtype=np.float64).copy()
    u_ret[indx_rem] = u
    return u_ret


def delete_rows_sparse(M, rows):
    """``matrix_assembly.py:48-68``."""
    mask = np.ones(M.shape[0], dtype=bool)
    mask[rows] = False
    return M[np.flatnonzero(mask), :]


def delete_cols_sparse(M, cols):
    """``matrix_assembly.py:70-90``."""
    mask = np.ones(M.shape[1], dtype=bool)
    mask[cols] = False
    return M[:, np.flatnonzero(mask)]


class GradGradAssembler:
    """P1 scalar-potential assembler (``matrix_assembly.py:92``)."""

    def __init__(self, mesh, domain_tags):
        self.mesh = mesh
        self.nodes = mesh.nodes
        self.num_materials = len(domain_tags)
        self.cell_types = []
        self.cells = []
        self._elems = []
        for tag in domain_tags:
            el = mesh.domain_elements(tag)
            self._elems.append(el)
            self.cell_types.append(np.array([4]))
            self.cells.append([(mesh.cells[el].astype(np.int64) + 1).reshape(-1)])
        self.domain_tags = list(domain_tags)
        self._dev = None
        self._tables = {}

    def get_quadrature_rule(self, ct, quad_order):
        w, q = fe.quadrature_rule(quad_order)
        return q, w

    def _device_state(self):
        if self._dev is None:
            _lib.require_cuda()
            cells = [self.mesh.cells[el] for el in self._elems]
            allc = np.concatenate(cells) if cells else np.zeros((0, 4), dtype=np.int32)
            cd = upload(allc, np.int32)
            offs = np.cumsum([0] + [len(el) for el in self._elems])
            self._dev = {"nodes": upload(self.nodes, np.float64), "cells": cd, "offsets": offs,
                         "pattern": Pattern(cd, len(allc), 4, self.nodes.shape[0])}
        return self._dev

    def _tabs(self, quad_order):
        if quad_order not in self._tables:
            w, q = fe.quadrature_rule(quad_order)
            self._tables[quad_order] = (len(w), upload(w, np.float64), upload(fe.evaluate_basis_derivative(q), np.float64))
        return self._tables[quad_order]

    @property
    def pattern(self):
        return self._device_state()["pattern"]

    def _assemble(self, x, mu_list, quad_order, K, dK, J, running):
        """K, dK, J (device, or None) of the domains that ``mu_list`` covers.  ``running``: J adds
        the sum of K so far after every domain, else K once."""
        d = self._device_state()
        nq, w_d, dphi_d = self._tabs(quad_order)
        pat, offs, cells = d["pattern"], d["offsets"], d["cells"]
        x_d = x if hasattr(x, "data_ptr") else upload(x, np.float64)
        t = torch()
        K, dK, J = (t.empty(max(pat.nnz, 1), dtype=t.float64, device=cells.device) if want else None
                    for want in (K, dK, J))
        specs = [permeability_spec(perm) for perm in mu_list]
        # all splines' knots and control points in one upload
        parts, where, n = [], [], 0
        for typ, k, nc, knots, ctrl, _, _ in specs:
            if typ == 1:
                parts += [np.asarray(knots, dtype=np.float64).reshape(-1), np.asarray(ctrl, dtype=np.float64).reshape(-1)]
                where.append((n, n + len(parts[-2])))
                n += len(parts[-2]) + len(parts[-1])
            else:
                where.append(None)
        tab = upload(np.concatenate(parts), np.float64) if parts else None
        mats = (_lib.GradGradMaterial * max(len(specs), 1))()
        for i, (typ, k, nc, _, _, hmin, muh) in enumerate(specs):
            at = where[i]
            mats[i] = _lib.GradGradMaterial(
                int(offs[i + 1] - offs[i]), cells.data_ptr() + 16 * int(offs[i]),
                tab.data_ptr() + 8 * at[0] if at else None, tab.data_ptr() + 8 * at[1] if at else None, hmin, muh,
                float(len(specs) - i) if running else 1.0, typ, k, nc, 0)
        _lib.call("snp_gradgrad_system", pat.handle, len(specs), mats, _lib.ptr(d["nodes"]), _lib.ptr(dphi_d),
                  _lib.ptr(w_d), nq, _lib.ptr(x_d), _lib.ptr(K), _lib.ptr(dK), _lib.ptr(J), _lib.stream_ptr())
        return pat, K, dK, J

    def assemble_device(self, x, mu_list, quad_order=8, K=True, dK=False, J=True):
        """Assemble into the cached pattern; returns CUDA tensors (those requested) and ``pattern``."""
        pat, K, dK, J = self._assemble(x, mu_list, quad_order, K, dK, J, running=False)
        return {"pattern": pat, "K": K, "dK": dK, "J": J}

    def compute_stiffness_and_jacobi_matrix_c(self, x, mu_list, quad_order=8, device=False):
        """``(K, J)`` (``matrix_assembly.py:1059-1135``), scipy CSR without exact zeros; with
        ``device=True`` torch sparse CSR tensors on the GPU (full structural pattern).

        The reference adds the running K to dK after every material (``dK += K`` inside the
        material loop), so J = dK + sum_n (K of materials 0..n).  This is kept as is: with one
        domain, the Laplace subdomain case, it is K + dK.
        """
        pat, K, _, J = self._assemble(x, mu_list, quad_order, True, False, True, running=True)
        if device:
            return pat.to_torch(K), pat.to_torch(J)
        return pat.to_scipy(K, drop_zeros=True), pat.to_scipy(J, drop_zeros=True)
