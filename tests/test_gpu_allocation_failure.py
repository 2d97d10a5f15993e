"""Memory exhaustion inside a call: it ends with SNP_NO_MEMORY, and the same handle answers the next
call as one that never met it.  The refusals come from the library's own allocator
(``snp_alloc_probe``), not from a full device."""

import ctypes

import pytest

import snoopy_b200 as S
from snoopy_b200 import _lib
from snoopy_b200 import materials as MAT
from snoopy_b200 import mesh as M

pytestmark = pytest.mark.gpu

NO_MEMORY = 6


@pytest.fixture
def allowed():
    """Sets how many allocations are served from now on (negative: all) and how many are refused
    behind them (negative: all); returns those made so far."""

    def probe(n, refused=-1):
        made = ctypes.c_int64()
        _lib.call("snp_alloc_probe", n, refused, ctypes.byref(made))
        return made.value

    yield probe
    probe(-1)


def _solver(tets, **kw):
    msh = M.window_frame_mesh(tets, jitter=0.15, seed=11)
    s = S.RedMVPSolver(msh, msh.geometry.coils(), [M.TAG_IRON], [M.TAG_AIR], [MAT.atan_reluctance()],
                       max_newton_iterations=60, quad_order=2, **kw)
    s.verbose = False
    return s


@pytest.mark.parametrize("method,precision", [("cg", 0), ("cg", 1), ("gmres", 0)])
def test_krylov_work_space_refused_in_the_middle(method, precision, allowed):
    import torch

    s = _solver(900)

    def solve(eng):
        return eng.solve(None, tol=1e-8, max_newton=2, precision=precision, raise_on_failure=False)[0].clone()

    def engine():
        s._newton = None
        eng = s.newton_engine()
        eng.set_krylov(method)
        return eng

    eng = engine()
    before = allowed(-1)
    want = solve(eng)
    need = allowed(-1) - before
    assert need >= 6  # state, 1 / diag, partials, scalars (device and host), flag
    for k in range(need):
        eng = engine()
        for served in (k, 0):  # and once more, behind a call that left off in the middle
            allowed(served)
            with pytest.raises(_lib.SnpError) as err:
                solve(eng)
            allowed(-1)
            assert err.value.status == NO_MEMORY
        assert torch.equal(solve(eng), want), k


def test_block_partition_refused_in_the_middle(allowed):
    """A refused new partition leaves point Jacobi; the next one takes over completely."""
    import numpy as np
    import torch
    from snoopy_b200.newton import dof_blocks

    eng = _solver(900).newton_engine()
    free = eng.free_mask.cpu().numpy().astype(bool)
    other = dof_blocks(np.arange(eng.n) // 3, free)

    def solve():
        return eng.solve(None, tol=1e-8, max_newton=2, raise_on_failure=False)[0].clone()

    lower_node = solve()
    before = allowed(-1)
    eng.set_preconditioner("block", meta=other)
    need = allowed(-1) - before
    threes = solve()
    eng.set_preconditioner("jacobi")
    point = solve()
    assert not torch.equal(point, threes) and not torch.equal(lower_node, threes)
    for k in range(need):
        eng.set_preconditioner("block")
        assert torch.equal(solve(), lower_node)
        allowed(k)
        with pytest.raises(_lib.SnpError) as err:
            eng.set_preconditioner("block", meta=other)
        allowed(-1)
        assert err.value.status == NO_MEMORY and not eng.block_jacobi
        assert torch.equal(solve(), point), k
        eng.set_preconditioner("block", meta=other)
        assert torch.equal(solve(), threes), k


def _frame(n_tets, order):
    import numpy as np

    msh = M.window_frame_mesh(n_tets, jitter=0.15, seed=11)
    if order == "mesh":
        return msh
    perm = np.random.default_rng(3).permutation(msh.num_elements)
    return M.TetMesh(msh.nodes, msh.cells[perm], msh.elem_domain[perm], grid=msh.grid,
                     boundary_node_mask=msh._boundary_node_mask)


def test_tile_plan_refused_in_the_middle(allowed):
    """The tiles of the float64 element pass are an option: a solver for which one of their arrays could
    not be had keeps a slot per element edge, and every other refusal ends the set-up."""
    import torch

    meshes = {o: _frame(330000, o) for o in ("mesh", "shuffled")}
    coils = _frame(900, "mesh").geometry.coils()

    def engine(order, *probe):
        s = S.RedMVPSolver(meshes[order], coils, [M.TAG_IRON], [M.TAG_AIR], [MAT.atan_reluctance()],
                           max_newton_iterations=60, quad_order=2)
        s.verbose = False
        s.curl_curl_factory.pattern  # the assembler's own allocations come first
        s.compute_source_fields()
        before = allowed(*(probe or (-1,)))
        try:
            eng = s.newton_engine()
        finally:
            made = allowed(-1) - before
        return eng, made

    def step(eng):  # twelve CG iterations
        x, st = eng.solve(None, tol=1e-8, max_newton=1, cg_rtol=1e-12, cg_maxiter=12, raise_on_failure=False,
                          line_search=False)
        assert st["cg_iterations"] == 12
        return x.clone()

    eng, total = engine("mesh")
    tiles = step(eng)
    # a mesh order whose tiles share too few edges stops after three of the plan's allocations
    plan = total - engine("shuffled")[1] + 3
    assert plan >= 15
    # behind the plan: 18 arrays of the solver, 9 of each assembled-matrix CG, 11 of the block partition
    end = total - (18 + 2 * 9 + 11)
    first = None
    for k in range(end - plan, end):
        eng, _ = engine("mesh", k, 1)
        x = step(eng)
        first = x if first is None else first
        assert torch.equal(x, first), k
    assert not torch.equal(first, tiles)  # the other sums
    # the same iterate to rounding: a few 1e-16 per iteration, and room for twelve iterations to carry
    # them on by a factor of three each
    assert float((first - tiles).abs().max()) <= 1e-10 * float(tiles.abs().max())
    for k in (end - plan - 1, end):
        with pytest.raises(_lib.SnpError) as err:
            engine("mesh", k, 1)
        assert err.value.status == NO_MEMORY


@pytest.mark.parametrize("n,nf", [(9000, 9000), (9000, 8193), (40000, 20000)])
def test_pcg_too_large_for_the_cluster_allocates_as_any_other(n, nf, allowed):
    """snp_pcg on systems that the cluster solve does not take: the buffers of the general path, which
    the same system padded beyond the cluster's limit takes unasked, and no more."""
    from test_gpu_kernel_edges import _masked_system, _pcg

    A, free, rng = _masked_system(n, nf, 5)
    b, x0 = rng.normal(size=n), rng.normal(size=n)
    made = []
    for pad in (0, 262145 - n):
        before = allowed(-1)
        rc, _, its = _pcg(A, None if nf == n else free, b, x0, pad)
        made.append((allowed(-1) - before, rc))
    assert made[0] == made[1] == (10, 0)  # diagonal positions; nine of the Krylov work space
