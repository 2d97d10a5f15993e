"""Kernels at the sizes where their launch shapes change: remainders of a warp or a tile, the
smallest problems, every branch of a dispatch.  Each against the CPU oracle or a plain float64
evaluation of the same formula."""

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
