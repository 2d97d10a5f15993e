"""The staged DoF pass of the float64 CG (tiles of 256 DoFs copied into shared memory, packed block
inverses) against the one-launch CG, which reads the unpacked rows and a slot per element edge: the
same iteration, term by term, in another order of the sums."""

import functools

import numpy as np
import pytest

import snoopy_b200 as S
from snoopy_b200 import materials as MAT
from snoopy_b200 import mesh as M
from snoopy_b200.newton import dof_blocks

pytestmark = pytest.mark.gpu

TILE, INC_CAP, WIDE = 256, 1536, 16383  # DoFs of a tile, slots it stages, slots its words count


@functools.lru_cache(maxsize=1)
def _base_mesh():
    return M.window_frame_mesh(620000, jitter=0.15, seed=11)


def _crowded(order, extra):
    """The mesh in the given element order, with the edges of ``extra`` scattered elements identified
    with the 252 first DoFs of a tile without constrained ones.  Every DoF keeps an element, and the matrix
    stays a sum of element matrices, so it is positive semidefinite and the system consistent."""
    src = _base_mesh()
    n = src.num_elements
    perm = np.arange(n) if order == "mesh" else np.random.default_rng(3).permutation(n)
    msh = M.TetMesh(src.nodes, src.cells[perm], src.elem_domain[perm], grid=src.grid,
                    boundary_node_mask=src._boundary_node_mask)
    gids = np.array(msh.elem_edges)
    n_dofs = msh.num_dofs
    free = np.ones(n_dofs, bool)
    free[msh.dirichlet_edge_ids()] = False
    tile = int(np.flatnonzero(free[:n_dofs // TILE * TILE].reshape(-1, TILE).all(axis=1))[5])
    valence = np.bincount(gids.ravel(), minlength=n_dofs)
    inner = np.flatnonzero((valence[gids] >= 4).all(axis=1) & (gids // TILE != tile).all(axis=1))
    chosen = inner[:: max(1, len(inner) // max(extra, 1))][:extra]
    gids[chosen] = tile * TILE + 42 * np.arange(6) + (np.arange(len(chosen)) % 42)[:, None]
    assert len(chosen) == extra and np.bincount(gids.ravel(), minlength=n_dofs).min() > 0
    msh.elem_edges = gids
    return msh, tile


def _slots_per_tile(msh, tile_plan):
    """Slot values of every DoF tile: one per element edge, or one per DoF and tile of 256 elements."""
    g = np.asarray(msh.elem_edges, dtype=np.int64)
    if not tile_plan:
        return np.bincount(g.ravel() // TILE)
    e_tile = np.repeat(np.arange(len(g)) // 256, 6)
    pairs = np.unique(e_tile * msh.num_dofs + g.ravel())
    assert len(pairs) <= 3 * len(g)  # else there is no plan
    return np.bincount(pairs % msh.num_dofs // TILE)


@pytest.mark.parametrize("order,extra,size", [("mesh", 0, 1), ("mesh", 0, 3), ("mesh", 0, 8), ("shuffled", 0, 8),
                                              ("mesh", 600, 3), ("shuffled", 600, 3), ("mesh", 4000, 8),
                                              ("shuffled", 4000, 8)])
def test_staged_dof_pass_is_the_one_launch_iteration(order, extra, size, monkeypatch):
    """Blocks of 1, 3 and 8 DoFs; element orders with and without a tile plan; a tile with more slots than
    are staged, and one with more than the plan's words count.

    Twenty iterations of either: the sums differ by the order of at most a few thousand terms, 1e-13 of
    their magnitudes, which the recurrence carries on (through the hundreds of iterations of a whole
    solve it grows to 1e-6); a wrong entry of the preconditioner or a missing slot changes the iterate by
    parts in a thousand."""
    import torch

    msh, tile = _crowded(order, extra)
    slots = _slots_per_tile(msh, order == "mesh")
    if extra == 600:
        assert INC_CAP < slots[tile] <= WIDE and slots.max() == slots[tile]
    elif extra == 4000:
        assert slots[tile] > WIDE
    s = S.RedMVPSolver(msh, _base_mesh().geometry.coils(), [M.TAG_IRON], [M.TAG_AIR], [MAT.atan_reluctance()],
                       max_newton_iterations=60, quad_order=2)
    s.verbose = False
    eng = s.newton_engine()
    assert (eng.n + TILE - 1) // TILE >= 4 * 4 * torch.cuda.get_device_properties(0).multi_processor_count
    free = eng.free_mask.cpu().numpy().astype(bool)
    eng.set_preconditioner("block", meta=dof_blocks(np.arange(eng.n) // size, free))

    def step():
        x, st = eng.solve(None, tol=1e-8, max_newton=1, cg_rtol=1e-8, cg_maxiter=20, raise_on_failure=False,
                          line_search=False)
        return x.clone(), st["cg_iterations"]

    monkeypatch.delenv("SNP_PCG_COOP", raising=False)
    x, its = step()
    monkeypatch.setenv("SNP_PCG_COOP", "1")
    ref, its_ref = step()
    assert its == its_ref == 20
    assert float((x - ref).abs().max()) <= 1e-9 * float(ref.abs().max())
