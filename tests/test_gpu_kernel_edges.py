"""Kernels at the sizes where their launch shapes change: remainders of a warp or a tile, the
smallest problems, every branch of a dispatch.  Each against the CPU oracle or a plain float64
evaluation of the same formula."""

import ctypes

import numpy as np
import pytest

import snoopy_b200 as S
from helpers import rel_max
from snoopy_b200 import fem_c
from snoopy_b200 import finite_element as FE
from snoopy_b200 import materials as MAT
from snoopy_b200 import mesh as M

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pts", [1, 7, 8, 9, 257])
@pytest.mark.parametrize("tets", [800, 12000])
def test_locate_point_counts(oracle_mod, n_pts, tets):
    """One warp per point: fewer points than a block's warps, whole blocks and a remainder, few
    buckets (the search window clipped on every side) and many."""
    msh = M.window_frame_mesh(tets, jitter=0.1, seed=5)
    rng = np.random.default_rng(n_pts)
    pts = rng.uniform(-0.62, 0.62, (n_pts, 3)) * [1.0, 1.0, 1.2]
    el, bary = msh.locate(pts)
    elo, baryo = oracle_mod.locate_points(msh.nodes, msh.cells, pts)
    assert np.array_equal(el, elo)
    # barycentric coordinates: a few float64 roundings of ratios of order-one determinants
    assert np.abs(bary - baryo).max() < 1e-12


NU0 = 0.25e7 / np.pi


def _assert_rows_close(a, b, row_ptr, tol):
    a, b, rp = a.double().cpu().numpy(), b.double().cpu().numpy(), row_ptr.cpu().numpy()
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    rmax = np.zeros(len(rp) - 1)
    np.maximum.at(rmax, rows, np.abs(b))
    assert (np.abs(a - b) <= tol * rmax[rows]).all()


@pytest.mark.parametrize("order", [1, 2, 3, 4])
@pytest.mark.parametrize("n_iron", [1, 127, 129])
def test_packed_assembly_matches_atomic(order, n_iron):
    """The packed two-phase assembly: every quadrature branch, iron ranges below, at and above an
    element tile, against the kernels that add into the CSR (other order of the same sums: a
    few roundings of the row's largest entry)."""
    msh = M.window_frame_mesh(2000, jitter=0.15, seed=3)
    dom = np.full(msh.num_elements, M.TAG_AIR, dtype=np.int32)
    dom[100:100 + n_iron] = M.TAG_IRON
    msh.elem_domain = dom
    A = S.CurlCurlAssembler(msh, [M.TAG_AIR, M.TAG_IRON], [S.ConstantReluctance(NU0), MAT.atan_reluctance()])
    rng = np.random.default_rng(order)
    x = rng.normal(0, 2e-3, msh.num_dofs)
    bs = rng.normal(0, 0.5, (n_iron * A.tables(order).nq, 3))
    sf = [np.zeros((0, 3)), bs]
    kw = dict(K=True, J=True, dK=True, rhs=True, F=True)
    R, T = (A.assemble_device(x, order, sf, method=m, **kw) for m in ("rows", "atomic"))
    for key in ("K", "dK", "J"):
        _assert_rows_close(R[key], T[key], A.pattern.row_ptr, 1e-12)
    for key in ("rhs", "F"):
        assert rel_max(R[key].cpu().numpy(), T[key].cpu().numpy()) < 1e-12


def test_packed_assembly_many_ranges():
    """40 materials, every other one without a source field and with constant reluctance: more
    separate ranges than the packed form's tables hold."""
    msh = M.window_frame_mesh(3000, jitter=0.15, seed=3)
    n_mat = 40
    msh.elem_domain = (100 + np.arange(msh.num_elements) * n_mat // msh.num_elements).astype(np.int32)
    rel = MAT.atan_reluctance()
    mats = [S.ConstantReluctance(NU0) if i % 2 else rel for i in range(n_mat)]
    A = S.CurlCurlAssembler(msh, [100 + i for i in range(n_mat)], mats)
    rng = np.random.default_rng(1)
    x = rng.normal(0, 2e-3, msh.num_dofs)
    nq = A.tables(2).nq
    sf = [np.zeros((0, 3)) if i % 2 else rng.normal(0, 0.5, (len(A._elems[i]) * nq, 3)) for i in range(n_mat)]
    for kw in (dict(K=True, J=True, dK=True, rhs=True, F=True), dict(K=True, J=True, dK=True, rhs=False, F=True)):
        R, T = (A.assemble_device(x, 2, sf, method=m, **kw) for m in ("rows", "atomic"))
        for key in ("K", "dK", "J"):
            _assert_rows_close(R[key], T[key], A.pattern.row_ptr, 1e-12)
        assert rel_max(R["F"].cpu().numpy(), T["F"].cpu().numpy()) < 1e-12
        if kw["rhs"]:
            assert rel_max(R["rhs"].cpu().numpy(), T["rhs"].cpu().numpy()) < 1e-12


def test_block_and_packed_element_values_agree():
    """The C entry points with the documented block layout and the whole-system call sum the same
    values in the same order: bitwise equal."""
    import ctypes

    import torch
    from snoopy_b200 import _lib

    msh = M.window_frame_mesh(3000, jitter=0.15, seed=9)
    A = S.CurlCurlAssembler(msh, [M.TAG_IRON, M.TAG_AIR], [MAT.atan_reluctance(), S.ConstantReluctance(NU0)])
    rng = np.random.default_rng(2)
    x = torch.from_numpy(rng.normal(0, 2e-3, msh.num_dofs)).cuda()
    tb, d, pat = A.tables(2), A._device_state(), A.pattern
    sf = [rng.normal(0, 0.5, (d["mats"][0]["count"] * tb.nq, 3)), np.zeros((0, 3))]
    R = A.assemble_device(x, 2, sf, method="rows", K=True, J=True, dK=True, rhs=True, F=True)
    bs = A.upload_source_fields(sf)
    parts, stride = 1 | 2 | 8 | 16, ctypes.c_int32()
    _lib.call("snp_curlcurl_terms_stride", parts, ctypes.byref(stride))
    terms = torch.empty(pat.n_elems * stride.value, dtype=torch.float64, device="cuda")
    for n, m in enumerate(d["mats"]):
        n_int, rc, rx = d["rel"][n]
        _lib.call("snp_curlcurl_terms", pat.handle, m["offset"], m["count"], _lib.ptr(d["nodes"]), _lib.ptr(m["cells"]),
                  _lib.ptr(m["gids"]), _lib.ptr(m["orient"]), _lib.ptr(tb.curls_d), tb.n_orient, None,
                  _lib.ptr(tb.d_phi_d), _lib.ptr(tb.w_d), tb.nq, _lib.ptr(x), _lib.ptr(bs[n]), n_int, _lib.ptr(rc),
                  _lib.ptr(rx), None, parts, _lib.ptr(terms), _lib.stream_ptr())
    out = {k: torch.empty_like(R[k]) for k in ("K", "dK", "J", "rhs", "F")}
    _lib.call("snp_curlcurl_rows", pat.handle, _lib.ptr(terms), parts, _lib.ptr(out["K"]), _lib.ptr(out["dK"]),
              _lib.ptr(out["J"]), None, _lib.ptr(out["rhs"]), _lib.ptr(out["F"]), _lib.stream_ptr())
    for k in out:
        assert torch.equal(out[k], R[k]), k


@pytest.mark.parametrize("n_tar", [1, 31, 1000, 12000, 25000, 50000, 80000])
@pytest.mark.parametrize("n_src", [1, 15, 16, 129])
def test_biot_savart_shapes(oracle_mod, n_tar, n_src):
    """Every lane split, tiles with a remainder; targets inside cores, near their surface, in line
    with segments and far away.  The sums of both sides differ by rounding only: within 1e-12 of
    the sum of the terms' magnitudes, here bounded by the field of the nearest filaments."""
    rng = np.random.default_rng(n_tar + n_src)
    a = rng.uniform(-1, 1, (n_src, 3))
    src = np.concatenate([a, a + rng.normal(0, 0.3, (n_src, 3))], axis=1)
    rad = 0.02
    tar = rng.uniform(-1.5, 1.5, (n_tar, 3))
    k = min(n_tar, 400)
    j = rng.integers(0, n_src, k)
    t = rng.uniform(-1.0, 2.0, k)[:, None]
    axis = src[j, 3:] - src[j, :3]
    off = np.cross(axis, rng.normal(size=(k, 3)))
    off *= (rad * rng.choice([0.1, 0.5, 0.999, 1.001, 1.5, 40.0], k) / np.linalg.norm(off, axis=1))[:, None]
    tar[:k] = src[j, :3] + t * axis + off
    got = fem_c.compute_B_line_segs_cpp(src, tar, 250.0, rad)
    ref = oracle_mod.compute_B_line_segs_cpp(src, tar, 250.0, rad)
    scale = 250.0 * 1e-7 * 2.0 / rad * max(1.0, np.sqrt(n_src))  # field at the surface of a core
    assert np.isfinite(ref).all() and np.abs(got - ref).max() < 1e-12 * scale


def _window_solver(tets, **kw):
    msh = M.window_frame_mesh(tets, jitter=0.15, seed=11)
    s = S.RedMVPSolver(msh, msh.geometry.coils(), [M.TAG_IRON], [M.TAG_AIR], [MAT.atan_reluctance()],
                       max_newton_iterations=60, quad_order=2, **kw)
    s.verbose = False
    return s


@pytest.mark.parametrize("tets", [900, 700000])
def test_krylov_passes_apply_the_jacobian(tets):
    """Each form of the float64 CG passes (direct and staged DoF pass) in one Newton step from zero:
    the step h it takes satisfies J h = -F to the CG tolerance it was given, with J applied by
    the product kernels."""
    import torch

    precision = "fp64"

    s = _window_solver(tets)
    eng = s.newton_engine()
    x0 = torch.zeros(eng.n, dtype=torch.float64, device="cuda")
    F = eng.assemble_tensors(x0, precision, torch.empty_like(x0))
    free = eng.free_mask.bool()
    h, _ = eng.solve(None, tol=1e-8, max_newton=1, cg_rtol=1e-3, raise_on_failure=False, line_search=False)
    eng.assemble_tensors(x0, precision, torch.empty_like(x0))
    Jh = eng.jacobian_apply(h, torch.zeros_like(h), precision)
    rel = float(torch.linalg.vector_norm((Jh + F)[free]) / torch.linalg.vector_norm(F[free]))
    assert rel <= 1.0001e-3  # the recursive residual met 1e-3; the true one differs by rounding


@pytest.mark.parametrize("size", [1, 3, 8])
def test_staged_dof_pass_blocks_and_padding(size):
    """The staged DoF pass with blocks of 1, 3 and 8 DoFs (packed rows of 1 to 36 entries, tiles
    ended by shorter blocks, a last tile with padding) against the direct pass, which smaller
    systems take: the same preconditioner, so the same solve to rounding."""
    import torch

    s = _window_solver(620000)
    eng = s.newton_engine()
    assert (eng.n + 255) // 256 >= 4 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    free = eng.free_mask.cpu().numpy().astype(bool)
    keys = np.arange(eng.n) // size
    from snoopy_b200.newton import dof_blocks

    eng.set_preconditioner("block", meta=dof_blocks(keys, free))
    x, st = eng.solve(None, tol=1e-8, max_newton=1, cg_rtol=1e-2, raise_on_failure=False, line_search=False)
    F = eng.assemble_tensors(torch.zeros_like(x), "fp64", torch.empty_like(x))
    Jh = eng.jacobian_apply(x, torch.zeros_like(x))
    fm = eng.free_mask.bool()
    rel = float(torch.linalg.vector_norm((Jh + F)[fm]) / torch.linalg.vector_norm(F[fm]))
    assert rel <= 1.0001e-2 and st["cg_iterations"] > 10


def _masked_system(n, nf, seed, row_len=12):
    """A symmetric matrix with A_ii = 1 + sum_j |A_ij| (so ||A^-1|| <= 1) on n rows, nf of them free."""
    import scipy.sparse as sp

    rng = np.random.default_rng(seed)
    i = np.repeat(np.arange(n), row_len // 2)
    j = np.clip(i + rng.integers(1, max(2, min(n, 400)), len(i)), 0, n - 1)
    keep = i < j
    off = sp.coo_matrix((rng.uniform(-1.0, 1.0, int(keep.sum())), (i[keep], j[keep])), shape=(n, n)).tocsr()
    off = off + off.T
    A = (off + sp.diags(1.0 + np.asarray(abs(off).sum(axis=1)).ravel())).tocsr()
    A.sort_indices()
    free = np.zeros(n, bool)
    free[rng.permutation(n)[:nf]] = True
    return A, free, rng


def _pcg(A, free, b, x0, pad=0, rtol=1e-12, atol=0.0, maxiter=-1):
    """(rc, x, iterations) of snp_pcg; `pad` constrained rows of one entry are appended."""
    from snoopy_b200 import _lib
    from snoopy_b200.device import to_host, upload

    n = A.shape[0] + pad
    rp = np.concatenate([A.indptr, A.nnz + np.arange(1, pad + 1)])
    ci = np.concatenate([A.indices, np.arange(A.shape[0], n)])
    if free is None and pad:
        free = np.ones(A.shape[0], bool)
    fm = None if free is None else upload(np.concatenate([free, np.zeros(pad, bool)]).astype(np.uint8), np.uint8)
    x = upload(np.concatenate([x0, np.zeros(pad)]), np.float64)
    args = [upload(rp, np.int32), upload(ci, np.int32), upload(np.concatenate([A.data, np.ones(pad)]), np.float64), fm,
            upload(np.concatenate([b, np.zeros(pad)]), np.float64), x]
    its, res = ctypes.c_int64(-1), ctypes.c_double(-1.0)
    rc = _lib.load().snp_pcg(n, *[_lib.ptr(a) for a in args], rtol, atol, maxiter, ctypes.byref(its),
                             ctypes.byref(res), _lib.stream_ptr())
    return rc, to_host(x)[:A.shape[0]], its.value


@pytest.mark.parametrize("n,nf,row_len", [(1, 1, 2), (40, 7, 8), (40, 8, 8), (1000, 9, 12), (5000, 1023, 12),
                                          (5000, 1025, 40), (70001, 4100, 12), (9000, 8192, 12), (9000, 8193, 12),
                                          (8192, 8192, 4), (8192, 8192, 12), (8192, 8192, 60), (262144, 300, 4)])
def test_small_pcg_matches_the_general_path(n, nf, row_len):
    """Few free rows: the cluster solve against the same system padded to more rows than it takes.

    ||x - A^-1 b|| <= ||A^-1|| ||r|| <= 1e-12 ||b|| for either, ten times that for the drift of the
    recursive residual; the counts may differ where ||r|| meets the tolerance within its rounding."""
    A, free, rng = _masked_system(n, nf, 7 + nf, row_len)
    b = rng.normal(size=n)
    x0 = rng.normal(size=n)
    x0[~free] = np.nan  # never read
    b[~free] = np.nan
    mask = None if nf == n else free
    for maxiter in (-1, 0, 3):
        rc, x, its = _pcg(A, mask, b, x0, maxiter=maxiter)
        rc_g, x_g, its_g = _pcg(A, mask, b, x0, 262145 - n, maxiter=maxiter)
        assert rc == rc_g and abs(its - its_g) <= (1 if maxiter < 0 else 0)
        assert not x[~free].any()
        assert np.linalg.norm((x - x_g)[free]) <= 2e-11 * np.linalg.norm(b[free])
    x = _pcg(A, mask, b, x0)[1][free]
    assert np.linalg.norm(A[free][:, free] @ x - b[free]) <= 1e-11 * np.linalg.norm(b[free])


def test_small_pcg_status_codes_match_the_general_path():
    A, free, rng = _masked_system(3000, 600, 3)
    b, x0 = rng.normal(size=3000), rng.normal(size=3000)
    row = int(np.flatnonzero(free)[77])
    cases = {"zero rhs": (A, np.zeros(3000), x0), "exact start": (A, A @ (x0 * free), x0)}
    for name, value in (("zero pivot", 0.0), ("nan pivot", np.nan)):
        Z = A.copy()
        Z.data[(Z.indices == row) & (np.repeat(np.arange(3000), np.diff(Z.indptr)) == row)] = value
        cases[name] = (Z, b, x0)
    Z = cases["zero pivot"][0].copy()
    Z.eliminate_zeros()
    cases["no diagonal entry"] = (Z, b, x0)
    nan_b = b.copy()
    nan_b[row] = np.nan
    cases["nan rhs"] = (A, nan_b, x0)
    for name, (mat, rhs, start) in cases.items():
        rc, x, its = _pcg(mat, free, rhs, start)
        rc_g, x_g, its_g = _pcg(mat, free, rhs, start, 262145 - 3000)
        assert (rc, its) == (rc_g, its_g), name
        np.testing.assert_allclose(x, x_g, rtol=0, atol=1e-11 * np.linalg.norm(b), err_msg=name)


@pytest.mark.parametrize("wanted", ["K", "dK", "J", "K,dK", "K,J", "dK,J", "K,dK,J"])
@pytest.mark.parametrize("sizes", [[1], [128, 129], [127, 0, 1, 300], [40] * 17 + [1000]])
def test_gradgrad_system_matches_material_by_material(sizes, wanted):
    """One launch over all materials (17 and more take two) against the accumulating call per
    material, by atomics: sums of the same values in another order."""
    from snoopy_b200 import _lib
    from snoopy_b200.device import Pattern, permeability_tables, upload, zeros

    msh = M.window_frame_mesh(4000, jitter=0.1, seed=4)
    n = sum(sizes)
    cells = upload(msh.cells[: n + 50], np.int32)  # 50 elements of no material
    pat = Pattern(cells, n + 50, 4, msh.num_nodes)
    w, q = FE.quadrature_rule(2)
    tabs = [upload(a, np.float64) for a in (msh.nodes, FE.evaluate_basis_derivative(q), w)]
    x = upload(np.random.default_rng(1).normal(0, 30.0, msh.num_nodes), np.float64)
    spline = permeability_tables(MAT.atan_permeability())
    flat = permeability_tables(S.ConstantPermeability(3e-6))
    mats = (_lib.GradGradMaterial * len(sizes))()
    ref = {k: zeros(pat.nnz) for k in ("K", "dK", "J")}
    weights = [1.0 if wanted == "K,dK,J" else float(len(sizes) - i) for i in range(len(sizes))]
    off = 0
    for i, cnt in enumerate(sizes):
        typ, k, nc, t, c, hmin, muh = spline if i % 2 == 0 else flat
        cp = cells.data_ptr() + 16 * off
        mats[i] = _lib.GradGradMaterial(cnt, cp, t.data_ptr(), c.data_ptr(), hmin, muh, weights[i], typ, k, nc, 0)
        part = {k: zeros(pat.nnz) for k in ("K", "dK")}
        with pytest.MonkeyPatch.context() as mp:
            mp.setenv("SNP_ASSEMBLY", "atomic")
            _lib.call("snp_gradgrad_assemble", pat.handle, off, cnt, _lib.ptr(tabs[0]), ctypes.c_void_p(cp),
                      _lib.ptr(tabs[1]), _lib.ptr(tabs[2]), len(w), _lib.ptr(x), typ, k, nc, _lib.ptr(t), _lib.ptr(c),
                      hmin, muh, _lib.ptr(part["K"]), _lib.ptr(part["dK"]), None, _lib.stream_ptr())
        ref["K"] += part["K"]
        ref["dK"] += part["dK"]
        ref["J"] += part["dK"] + weights[i] * part["K"]
        off += cnt
    for mode in ("rows", "atomic"):
        out = {k: zeros(pat.nnz).fill_(7.0) if k in wanted.split(",") else None for k in ("K", "dK", "J")}
        with pytest.MonkeyPatch.context() as mp:
            mp.setenv("SNP_ASSEMBLY", mode)
            _lib.call("snp_gradgrad_system", pat.handle, len(sizes), mats, _lib.ptr(tabs[0]), _lib.ptr(tabs[1]),
                      _lib.ptr(tabs[2]), len(w), _lib.ptr(x), _lib.ptr(out["K"]), _lib.ptr(out["dK"]),
                      _lib.ptr(out["J"]), _lib.stream_ptr())
        for k, v in out.items():
            if v is not None:
                # a row's entries are sums of up to 30 values no larger than its diagonal's
                _assert_rows_close(v, ref[k], pat.row_ptr, 1e-12)
    # entry by entry the accumulating call (rows) is the system call's sum
    if sizes == [1] and wanted == "K,dK":
        acc = {k: zeros(pat.nnz) for k in ("K", "dK")}
        typ, k, nc, t, c, hmin, muh = spline
        _lib.call("snp_gradgrad_assemble", pat.handle, 0, 1, _lib.ptr(tabs[0]), _lib.ptr(cells), _lib.ptr(tabs[1]),
                  _lib.ptr(tabs[2]), len(w), _lib.ptr(x), typ, k, nc, _lib.ptr(t), _lib.ptr(c), hmin, muh,
                  _lib.ptr(acc["K"]), _lib.ptr(acc["dK"]), None, _lib.stream_ptr())
        _assert_rows_close(acc["K"], ref["K"], pat.row_ptr, 1e-12)
        _assert_rows_close(acc["dK"], ref["dK"], pat.row_ptr, 1e-12)


@pytest.mark.parametrize("tets,precision", [(900, "fp64"), (900, "mixed"), (60000, "mixed"), (620000, "fp64")])
def test_overlapping_passes_give_one_answer(tets, precision, monkeypatch):
    """CG passes that may start while the previous one drains, captured in the loop body and
    launched one by one: bitwise the same solve, and the same again."""
    import torch

    s = _window_solver(tets)
    out = []
    for graph in ("1", "0", "1"):
        monkeypatch.setenv("SNP_PCG_GRAPH", graph)
        eng = s.newton_engine()
        x, st = eng.solve(None, tol=1e-8, max_newton=2, precision={"fp64": 0, "mixed": 1}[precision],
                          raise_on_failure=False)
        out.append((x.clone(), st["cg_iterations"]))
        s._newton = None
    assert out[0][1] == out[1][1] == out[2][1] > 10
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][0], out[2][0])


@pytest.mark.parametrize("diluted", [False, True])
@pytest.mark.parametrize("n_iron", [1, 63, 65, 400])
@pytest.mark.parametrize("order", [3, 4, 6])
def test_point_sums_in_their_own_launch(order, n_iron, diluted):
    """Many quadrature points: the launch that sums them, four lanes per element, behind every set of
    wanted outputs, against the kernels that do it element by element and add into the CSR."""
    msh = M.window_frame_mesh(2000, jitter=0.15, seed=3)
    dom = np.full(msh.num_elements, M.TAG_AIR, dtype=np.int32)
    dom[100:100 + n_iron] = M.TAG_IRON
    msh.elem_domain = dom
    tags, mats = [M.TAG_AIR, M.TAG_IRON], [S.ConstantReluctance(NU0), MAT.atan_reluctance()]
    if diluted:
        A = S.CurlCurlAssemblerDiluted(msh, tags, mats, [None, MAT.Dilution(0.0, 0.30, 0.35, 0.75, 0.02, 0.40, 0.45, 0.80,
                                                                                z_pos=-0.25, z_len=0.5)])
    else:
        A = S.CurlCurlAssembler(msh, tags, mats)
    rng = np.random.default_rng(order)
    x = rng.normal(0, 2e-3, msh.num_dofs)
    sf = [np.zeros((0, 3)), rng.normal(0, 0.5, (n_iron * A.tables(order).nq, 3))]
    T = A.assemble_device(x, order, sf, method="atomic", K=True, J=True, dK=True, rhs=True, F=True)
    for wanted in ("K,dK,J,rhs,F", "J,F", "dK", "K,rhs", "rhs,F"):
        kw = {k: k in wanted.split(",") for k in ("K", "dK", "J", "rhs", "F")}
        R = A.assemble_device(x, order, sf, method="rows", **kw)
        for key in wanted.split(","):
            if key in ("rhs", "F"):
                assert rel_max(R[key].cpu().numpy(), T[key].cpu().numpy()) < 1e-12
            else:
                _assert_rows_close(R[key], T[key], A.pattern.row_ptr, 1e-12)


@pytest.mark.parametrize("order", [1, 2, 3, 4, 6])
def test_tensor_kernel_point_loads(order):
    """Element tensors with points loaded in pairs (even counts), with a single one left over (odd
    counts) and with one point only: F and J x against the CSR system's."""
    import torch

    s = _window_solver(900)
    s.quad_order = order
    eng = s.newton_engine()
    x = torch.from_numpy(np.random.default_rng(order).normal(0, 1e-3, eng.n)).cuda()
    v = torch.from_numpy(np.random.default_rng(9).normal(0, 1.0, eng.n)).cuda()
    free = eng.free_mask.bool()
    v[~free] = 0.0
    F = eng.assemble_tensors(x, "fp64", torch.empty_like(x))
    Jv = eng.jacobian_apply(v, torch.zeros_like(v))
    out = s.curl_curl_factory.assemble_device(x, order, s.compute_source_fields(), K=False, J=True, rhs=False, F=True)
    ref = out["pattern"].to_torch(out["J"]).matmul(v)
    # sums of a few tens of element terms of the same magnitude in another order
    for a, b in ((F[free], out["F"][:eng.n][free]), (Jv[free], ref[free])):
        assert float((a - b).abs().max()) <= 1e-12 * float(b.abs().max())


@pytest.mark.parametrize("order", ["mesh", "shuffled", "reversed"])
def test_tile_pass_and_its_fallback(order):
    """The float64 element pass over tiles of elements (mesh order and its reverse, a last tile with
    a remainder, and the direct DoF pass behind it) and an element order that shares too few edges in
    a tile: one Newton step satisfies J h = -F to the CG tolerance, with J from the product kernels."""
    import torch

    msh = M.window_frame_mesh(330000, jitter=0.15, seed=11)
    n = msh.num_elements
    assert n >= 300000 and n % 256
    perm = {"mesh": np.arange(n), "shuffled": np.random.default_rng(3).permutation(n),
            "reversed": np.arange(n)[::-1]}[order]
    other = M.TetMesh(msh.nodes, msh.cells[perm], msh.elem_domain[perm], grid=msh.grid,
                      boundary_node_mask=msh._boundary_node_mask)
    s = S.RedMVPSolver(other, msh.geometry.coils(), [M.TAG_IRON], [M.TAG_AIR], [MAT.atan_reluctance()],
                       max_newton_iterations=60, quad_order=2)
    s.verbose = False
    eng = s.newton_engine()
    x0 = torch.zeros(eng.n, dtype=torch.float64, device="cuda")
    F = eng.assemble_tensors(x0, "fp64", torch.empty_like(x0))
    free = eng.free_mask.bool()
    h, _ = eng.solve(None, tol=1e-8, max_newton=1, cg_rtol=1e-3, raise_on_failure=False, line_search=False)
    eng.assemble_tensors(x0, "fp64", torch.empty_like(x0))
    Jh = eng.jacobian_apply(h, torch.zeros_like(h), "fp64")
    rel = float(torch.linalg.vector_norm((Jh + F)[free]) / torch.linalg.vector_norm(F[free]))
    assert rel <= 1.0001e-3  # the recursive residual met 1e-3; the true one differs by rounding


@pytest.mark.parametrize("precision", [0, 1])
def test_first_solves_are_ordered_without_the_default_stream(precision):
    """A solver's first Krylov solve clears its state on its own stream: two solvers at once, with the
    default stream busy meanwhile, answer as they do the second time, bit by bit."""
    import torch

    from snoopy_b200 import _lib

    solvers = [_window_solver(20000) for _ in range(2)]
    for s in solvers:
        s.stream = torch.cuda.Stream()
    engs = [s.newton_engine() for s in solvers]
    opts = (_lib.SolveOpts * 2)(*[_lib.SolveOpts(1, 1e-6, 50000, 60, 0.1, precision, 0, 1, 0.0)] * 2)
    out = []
    for busy in (True, False):
        xs = [torch.zeros(e.n, dtype=torch.float64, device="cuda") for e in engs]
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(400_000_000)  # about 0.2 s
        stats, status = (_lib.SolveStats * 2)(), (ctypes.c_int32 * 2)()
        rc = _lib.load().snp_solver_solve_many((ctypes.c_void_p * 2)(*[e.handle.value for e in engs]), 2,
                                               (ctypes.c_void_p * 2)(*[x.data_ptr() for x in xs]), opts, stats, 2,
                                               status)
        torch.cuda.synchronize()
        assert rc == 0, _lib.load().snp_last_error()
        out.append(xs)
    for a, b in zip(*out):
        assert torch.equal(a, b)
