"""Meshes whose doubled sizes have no compile-time kernels: their transforms are
padded to the next lengths that have them.  The field against the FP64 oracle (fed the
device's tensor: 1e-12 FP64, 1e-5 FP32 field, as for every other mesh), and against
the run-time-plan kernels at the mesh's own lengths over the forms both take
(scalar and per-cell Ms, terms with parameter fields, rows of odd, even and
4-divisible lengths; field, energy and dm/dt): 1e-12 and 1e-5."""
import numpy as np
import pytest

import maf_oracle as O
from helpers import random_m, rel_l2, rel_max

M = pytest.importorskip("magnumaf")

pytestmark = pytest.mark.gpu

MS = 8.6e5
HEXT = (0.011 / O.mu0, -0.027 / O.mu0, 0.019 / O.mu0)

# x rows odd, even and 4-divisible, one below and one above a compile-time length; single
# rows and columns; every z length (8, 16, 32, 64, 96, 128); one axis ragged at a time
MESHES = [
    (100, 25, 1), (33, 7, 1), (1, 13, 1), (15, 1, 1), (98, 64, 1), (63, 33, 1), (26, 130, 1),
    (64, 32, 2), (25, 18, 3), (20, 65, 5), (50, 21, 9), (16, 8, 15), (35, 10, 20), (12, 9, 39), (7, 20, 50), (130, 16, 4),
]


def _terms(gm, d):
    return [d, M.ExchangeField(1.3e-11), M.DmiField(1e-3), M.CubicAnisotropyField(-1e4, 3e3, -2e3),
            M.UniaxialAnisotropyField(2e5, (0.6, 0.0, 0.8)), M.ExternalField.uniform(*HEXT)]


@pytest.mark.parametrize("shape", MESHES)
def test_padded_field_vs_oracle_and_own_lengths(shape):
    gm = M.Mesh(*shape, 3e-9, 2e-9, 4e-9)
    om = O.Mesh(*shape, 3e-9, 2e-9, 4e-9)
    m = random_m(shape, 41)
    d = M.DemagField(gm)
    od = O.DemagField(om, N_real=d.get_N(symmetric=True))
    oterms = [od, O.ExchangeField(1.3e-11), O.DmiField(1e-3), O.CubicAnisotropyField(-1e4, 3e3, -2e3),
              O.UniaxialAnisotropyField(2e5, (0.6, 0.0, 0.8)), O.ExternalField(np.array(HEXT))]
    ref = O.Heff_in_Apm(oterms, O.State(om, MS, m))
    llg = M.LLGIntegrator(0.1, _terms(gm, d), "DP45")
    for prec, tol in (("fp64", 1e-12), ("fp32_field", 1e-5)):
        s = M.State(gm, MS, m, precision=prec)
        got = {}
        for generic in (False, True, False):
            d.generic = generic
            h, e, k = llg.H_in_Apm(s), llg.Eeff_in_J(s), llg.dmdt(s)
            assert rel_l2(h, ref) < tol and rel_max(h, ref) < tol, (generic, rel_l2(h, ref), rel_max(h, ref))
            got[generic] = (h, e, k)
        assert abs(got[False][1] - got[True][1]) <= tol * abs(got[True][1])
        assert rel_l2(got[False][2], got[True][2]) < tol


# 3-D meshes where x keeps its own length beside padded y and z (DemagField.lengths): a spectrum
# that would grow by more than 1.6, and by more than 1.25 beside 4096 points along y; one axis
# padded, two, rows of odd length
@pytest.mark.parametrize("shape", [(9, 130, 20), (3, 64, 33), (1, 200, 16), (6, 300, 12), (20, 1040, 2)])
def test_own_x_length_beside_padded_axes(shape):
    lengths = M.DemagField.lengths(*shape)
    assert lengths[0] == 2 * shape[0] and lengths != tuple(2 * n for n in shape)
    test_padded_field_vs_oracle_and_own_lengths(shape)


def test_attempt_with_own_x_length():
    """A whole Runge-Kutta attempt of that form (the stage's epilogue writes the next stage's m)."""
    shape = (9, 130, 20)
    gm, om = M.Mesh(*shape, 3e-9, 2e-9, 4e-9), O.Mesh(*shape, 3e-9, 2e-9, 4e-9)
    m = random_m(shape, 41)
    d = M.DemagField(gm)
    os_ = O.State(om, MS, m)
    sumbk, _ = O.LLGIntegrator(0.1, [O.DemagField(om, N_real=d.get_N(symmetric=True)), O.ExchangeField(1.3e-11)],
                               "DP45").attempt(os_, 2e-14)
    llg = M.LLGIntegrator(0.1, [d, M.ExchangeField(1.3e-11)], "DP45")
    for prec, tol in (("fp64", 1e-12), ("fp32_field", 1e-6)):
        got, _ = llg.rk_attempt(M.State(gm, MS, m, precision=prec), "DP45", 2e-14)
        assert rel_max(got, os_.m + sumbk) < tol


@pytest.mark.parametrize("shape", [(100, 25, 1), (33, 20, 3), (50, 18, 10)])
def test_padded_ms_field_and_parameter_fields(shape):
    gm = M.Mesh(*shape, 3e-9, 3e-9, 3e-9)
    m = random_m(shape, 42)
    rng = np.random.default_rng(7)
    x = (np.arange(shape[0]) + 0.5) / shape[0] - 0.5
    y = (np.arange(shape[1]) + 0.5) / shape[1] - 0.5
    m[x[:, None] ** 2 + y[None, :] ** 2 > 0.25] = 0.0  # empty cells: a field of Ms
    d = M.DemagField(gm)
    ku = rng.uniform(1e4, 2e5, size=shape)
    llg = M.LLGIntegrator(0.1, [d, M.ExchangeField(1.3e-11), M.UniaxialAnisotropyField(ku, (0.0, 0.0, 1.0))], "RKF45")
    for prec, tol in (("fp64", 1e-12), ("fp32_field", 1e-5)):
        s = M.State(gm, MS, m, precision=prec)
        got = []
        for generic in (False, True):
            d.generic = generic
            got.append((llg.H_in_Apm(s), llg.dmdt(s), llg.Eeff_in_J(s)))
        for a, b in zip(*got):
            assert rel_l2(a, b) < tol


def test_padded_tensor_stays_the_meshs_own():
    """The spectral tensor a user reads (or caches on disk) keeps the mesh's lengths."""
    gm = M.Mesh(50, 18, 10, 3e-9, 3e-9, 3e-9)
    d = M.DemagField(gm)
    before = d.spectral_tensor()
    assert before.shape == (6, 11, 19, 51)
    d.H_in_Apm(M.State(gm, MS, random_m((50, 18, 10), 1)))
    assert np.array_equal(d.spectral_tensor(), before)
