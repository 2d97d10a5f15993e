"""``snp_curlcurl_system`` against what its description promises: the bits of the two-call form, and
dK = 0 where the reluctance is constant."""

import ctypes

import numpy as np
import pytest

import snoopy_b200 as S
from snoopy_b200 import _lib
from snoopy_b200 import materials as MAT
from snoopy_b200 import mesh as M

pytestmark = pytest.mark.gpu

NU0 = 0.25e7 / np.pi


def _two_calls(A, x, order, sf, parts, keys, like):
    """K, dK, J, rhs, F of ``snp_curlcurl_terms`` per material and ``snp_curlcurl_rows``."""
    import torch

    tb, d, pat = A.tables(order), A._device_state(), A.pattern
    bs, stride = A.upload_source_fields(sf), ctypes.c_int32()
    _lib.call("snp_curlcurl_terms_stride", parts, ctypes.byref(stride))
    terms = torch.empty(pat.n_elems * stride.value, dtype=torch.float64, device="cuda")
    for n, m in enumerate(d["mats"]):
        n_int, rc, rx = d["rel"][n]
        coef = A._dilution_coef(n)
        _lib.call("snp_curlcurl_terms", pat.handle, m["offset"], m["count"], _lib.ptr(d["nodes"]), _lib.ptr(m["cells"]),
                  _lib.ptr(m["gids"]), _lib.ptr(m["orient"]), _lib.ptr(tb.curls_d), tb.n_orient,
                  _lib.ptr(tb.phi_d) if coef is not None else None, _lib.ptr(tb.d_phi_d), _lib.ptr(tb.w_d), tb.nq,
                  _lib.ptr(x), _lib.ptr(bs[n]), n_int, _lib.ptr(rc), _lib.ptr(rx), coef, parts, _lib.ptr(terms),
                  _lib.stream_ptr())
    out = {k: torch.empty_like(like[k]) if k in keys else None for k in ("K", "dK", "J", "rhs", "F")}
    _lib.call("snp_curlcurl_rows", pat.handle, _lib.ptr(terms), parts, _lib.ptr(out["K"]), _lib.ptr(out["dK"]),
              _lib.ptr(out["J"]), None, _lib.ptr(out["rhs"]), _lib.ptr(out["F"]), _lib.stream_ptr())
    return out


@pytest.mark.parametrize("diluted", [False, True])
@pytest.mark.parametrize("order", [1, 2, 3, 4, 5, 6])
def test_system_has_the_bits_of_terms_and_rows(order, diluted):
    """At every number of quadrature points, those of the points' own launch included, for plain and
    diluted steel and every set of outputs."""
    import torch

    msh = M.window_frame_mesh(3000, jitter=0.15, seed=9)
    tags, mats = [M.TAG_IRON, M.TAG_AIR], [MAT.atan_reluctance(), S.ConstantReluctance(NU0)]
    if diluted:
        dil = MAT.Dilution(0.0, 0.30, 0.35, 0.75, 0.02, 0.40, 0.45, 0.80, z_pos=-0.25, z_len=0.5)
        A = S.CurlCurlAssemblerDiluted(msh, tags, mats, [dil, None])
    else:
        A = S.CurlCurlAssembler(msh, tags, mats)
    rng = np.random.default_rng(order)
    x = torch.from_numpy(rng.normal(0, 2e-3, msh.num_dofs)).cuda()
    sf = [rng.normal(0, 0.5, (len(A._elems[0]) * A.tables(order).nq, 3)), np.zeros((0, 3))]
    K, DK, F, RHS = _lib.TERMS_K, _lib.TERMS_DK, _lib.TERMS_F, _lib.TERMS_RHS
    for parts, keys in ((K | DK | F | RHS, ("K", "dK", "J", "rhs", "F")), (K | DK, ("J",)), (DK, ("dK",)),
                        (K | F, ("K", "F")), (F | RHS, ("rhs", "F"))):
        R = A.assemble_device(x, order, sf, method="rows", **{k: k in keys for k in ("K", "dK", "J", "rhs", "F")})
        T = _two_calls(A, x, order, sf, parts, keys, R)
        for k in keys:
            assert torch.equal(T[k], R[k]), (keys, k)


@pytest.mark.parametrize("value", [np.nan, np.inf, 1e200])
@pytest.mark.parametrize("order,air_field", [(2, False), (2, True), (4, True)])
def test_constant_reluctance_keeps_what_is_not_finite(order, air_field, value):
    """dK of a material with constant reluctance is nu' times something: 0 for a finite B, else what the
    products give.  An infinity, a NaN or a large number in x shows in dK and J as in the two-call form."""
    import torch

    msh = M.window_frame_mesh(3000, jitter=0.15, seed=9)
    A = S.CurlCurlAssembler(msh, [M.TAG_IRON, M.TAG_AIR], [MAT.atan_reluctance(), S.ConstantReluctance(NU0)])
    rng = np.random.default_rng(order)
    x = torch.from_numpy(rng.normal(0, 2e-3, msh.num_dofs)).cuda()
    gids = A._device_state()["mats"][1]["gids"].view(-1, 6)
    x[gids[[0, 200, 201], [0, 3, 5]].long()] = value
    nq = A.tables(order).nq
    sf = [rng.normal(0, 0.5, (len(A._elems[0]) * nq, 3)),
          rng.normal(0, 0.5, (len(A._elems[1]) * nq, 3)) if air_field else np.zeros((0, 3))]
    K, DK, F, RHS = _lib.TERMS_K, _lib.TERMS_DK, _lib.TERMS_F, _lib.TERMS_RHS
    for parts, keys in ((K | DK | F | RHS, ("K", "dK", "J", "rhs", "F")), (K | DK, ("J",)), (DK, ("dK",))):
        R = A.assemble_device(x, order, sf, method="rows", **{k: k in keys for k in ("K", "dK", "J", "rhs", "F")})
        T = _two_calls(A, x, order, sf, parts, keys, R)
        for k in keys:
            assert torch.equal(T[k].isnan(), R[k].isnan()) and torch.equal(T[k].nan_to_num(), R[k].nan_to_num()), (keys, k)
        matrix = "dK" if "dK" in keys else "J"
        assert bool(T[matrix].isfinite().all()) == np.isfinite(value)  # 0 times a large B is 0
