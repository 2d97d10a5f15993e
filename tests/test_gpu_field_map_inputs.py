"""Field maps of coils and assemblers that are not the package's own."""

import types

import numpy as np
import pytest

import snoopy_b200 as S
from snoopy_b200 import evaluators as EV
from snoopy_b200 import materials as MAT
from snoopy_b200 import mesh as M

pytestmark = pytest.mark.gpu

TAGS = [M.TAG_AIR, M.TAG_IRON]


@pytest.fixture(scope="module")
def case():
    msh = M.window_frame_mesh(3000, jitter=0.15, seed=7)
    solver = S.RedMVPSolver(msh, msh.geometry.coils(), [M.TAG_IRON], [M.TAG_AIR], [MAT.atan_reluctance()], quad_order=2)
    rng = np.random.default_rng(3)
    return msh, solver, rng.normal(0, 1e-3, msh.num_dofs), rng.uniform(-0.4, 0.4, (200, 3))


def _map(case, solver=None, coils=()):
    msh, own, x, pts = case
    return EV.evaluate_fem_solution_node_interpolation(msh, pts, solver or own, coils, x, TAGS)


@pytest.mark.parametrize("value", [0.25, [0.1, -0.2, 0.3], [[0.1, -0.2, 0.3]], "column"])
def test_coil_fields_that_broadcast_over_the_nodes(case, value):
    """A coil's ``compute_B`` may return anything that adds to an [N, 3] array."""
    nodes = case[0].nodes
    value = nodes[:, :1] * 0.5 if value == "column" else np.asarray(value)
    coil = types.SimpleNamespace(compute_B=lambda p: value)
    whole = types.SimpleNamespace(compute_B=lambda p: value + 0.0 * p)
    assert np.array_equal(_map(case, coils=[coil]), _map(case, coils=[whole]))


def test_racetrack_coils_with_a_field_of_their_own(case):
    """A racetrack coil's field is evaluated on the device unless it has another ``compute_B``: by
    subclass or on the object; one with other segments keeps them."""
    kind = type(case[0].geometry.coils()[0])

    class Halved(kind):
        def compute_B(self, positions, disc_arc=5):
            return 0.5 * super().compute_B(positions, disc_arc)

    class Coarse(kind):
        def get_segments(self, disc_arc=5, enable_plot=False):
            return super().get_segments(2)

    def as_kind(cls):
        return [cls(c.kp, c.y, c.rad, c.current) for c in case[0].geometry.coils()]

    def on_host(coils):
        return [types.SimpleNamespace(compute_B=c.compute_B) for c in coils]

    own = as_kind(kind)
    own[0].compute_B = lambda positions: np.ones((len(positions), 3))
    for coils in (as_kind(kind), as_kind(Halved), as_kind(Coarse), own):
        assert np.array_equal(_map(case, coils=coils), _map(case, coils=on_host(coils)))


def test_assemblers_with_nodal_fields_of_their_own(case):
    """An assembler needs its nodes and ``compute_nodal_fields``; a subclass's own is the one used."""
    msh, solver, x, _ = case
    asm = solver.curl_curl_factory
    want = _map(case)
    plain = types.SimpleNamespace(nodes=asm.nodes, compute_nodal_fields=asm.compute_nodal_fields)
    assert np.array_equal(_map(case, types.SimpleNamespace(curl_curl_factory=plain)), want)

    class Doubled(S.CurlCurlAssembler):
        def compute_nodal_fields(self, x, mat_ids):
            return 2.0 * super().compute_nodal_fields(x, mat_ids)

    twice = Doubled(msh, TAGS, [S.ConstantReluctance(1e6), MAT.atan_reluctance()])
    assert np.array_equal(_map(case, types.SimpleNamespace(curl_curl_factory=twice)), 2.0 * want)
