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
    """Sets how many allocations are served from now on (negative: all); returns those made so far."""

    def probe(n):
        made = ctypes.c_int64()
        _lib.call("snp_alloc_probe", n, ctypes.byref(made))
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
