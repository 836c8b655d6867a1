"""Size rules of the time step and the minimiser: up to 2^18 cells the epilogue of a
Runge-Kutta stage writes the next stage's magnetisation, above a combine kernel does; up
to 196608 values per vector the LBFGS recursion is one cluster launch, above a chain of
launches.  Both sides of each line against the oracle (1e-12 for an attempt, 1e-9 relative
for the energy after a few iterations), local terms only.  Ensembles: members of more
transform lengths than there are chains share chains, bit for bit their own trajectories."""
import numpy as np
import pytest

import maf_lbfgs_oracle as L
import maf_oracle as O
from helpers import mesh_pair, random_m, rel_max

M = pytest.importorskip("magnumaf")

pytestmark = pytest.mark.gpu


def _terms():
    return ([M.ExchangeField(1.3e-11), M.UniaxialAnisotropyField(3e5, (0.0, 0.0, 1.0)), M.DmiField(1e-3)],
            [O.ExchangeField(1.3e-11), O.UniaxialAnisotropyField(3e5), O.DmiField(1e-3)])


@pytest.mark.parametrize("scheme", ["RKF45", "DP45", "BS23"])
@pytest.mark.parametrize("shape,ms_field", [((9, 7, 1), False), ((12, 5, 3), True), ((512, 512, 1), False),
                                            ((513, 512, 1), False), ((264, 250, 4), True)])
def test_attempt_on_both_sides_of_the_stage_rule(shape, ms_field, scheme):
    gm, om = mesh_pair(*shape, 3e-9, 3e-9, 3e-9)
    m0 = random_m(shape, 5)
    if ms_field:
        m0[::3, 1::2] = 0.0
    gterms, oterms = _terms()
    gs, os_ = M.State(gm, 8e5, m0), O.State(om, 8e5, m0)
    m_new, err = M.LLGIntegrator(0.1, gterms, scheme).rk_attempt(gs, scheme, 2e-14)
    sumbk, err_ref = O.LLGIntegrator(0.1, oterms, scheme).attempt(os_, 2e-14)
    assert rel_max(m_new, os_.m + sumbk) < 1e-12
    # the norm is a difference of nearly equal sums of terms up to 1e-2 / 1e-6 in its units
    assert abs(err - err_ref) < 1e-8 * err_ref + 1e-11
    s32 = M.State(gm, 8e5, m0, precision="fp32_field")
    m32, _ = M.LLGIntegrator(0.1, gterms, scheme).rk_attempt(s32, scheme, 2e-14)
    assert rel_max(m32, os_.m + sumbk) < 1e-6


@pytest.mark.parametrize("shape", [(3, 2, 1), (73, 75, 1), (256, 256, 1), (257, 256, 1)])
def test_minimiser_on_both_sides_of_the_recursion_rule(shape):
    gm, om = mesh_pair(*shape, 2e-9, 2e-9, 1e-9)
    x = np.linspace(0, 3, shape[0])[:, None, None]
    y = np.linspace(0, 2, shape[1])[None, :, None]
    m0 = np.stack([np.cos(x) * np.cos(y), np.sin(x) * np.cos(y), np.sin(y) + 0 * x], axis=-1)
    m0 = m0 / np.linalg.norm(m0, axis=3, keepdims=True)
    gterms, oterms = _terms()
    gs, os_ = M.State(gm, 8e5, m0), O.State(om, 8e5, m0)
    mini = M.LBFGS_Minimizer(gterms, tol=1e-6, maxiter=9)
    E = mini.minimize(gs)
    E_ref, it_ref = L.minimize(os_, oterms, tolerance=1e-6, maxIter=9)
    assert abs(E - E_ref) <= 1e-9 * abs(E_ref)
    assert mini.stats()["iterations"] == it_ref
    assert np.abs(gs.m - os_.m).max() < 1e-8


@pytest.mark.parametrize("prec", ["fp32_field", "fp64"])
@pytest.mark.parametrize("members", [1, 16, 17, 23])
def test_ensemble_chains_on_both_sides_of_their_bound(members, prec):
    sides = [(nx, ny) for nx in (10, 33, 66, 100, 130) for ny in (6, 20, 35, 65, 99)][:members]
    made = []
    for _ in range(2):
        group = []
        for i, (nx, ny) in enumerate(sides):
            mesh = M.Mesh(nx, ny, 1, 2e-9, 2e-9, 1e-9)
            st = M.State(mesh, 7e5, random_m((nx, ny, 1), 60 + i), precision=prec)
            terms = [M.DemagField(mesh), M.ExchangeField(1.5e-11), M.UniaxialAnisotropyField(6e5)]
            group.append((M.Stochastic_LLG(0.1, 300.0, 5e-14, st, terms, "Heun", seed=11, member=i), st))
        made.append(group)
    batch = M.StochasticBatch(made[0], fused=True)
    batch.steps(5)
    assert batch.fused_active
    for (_, sb), (it, ss) in zip(*made):
        it.steps(ss, 5)
        assert np.array_equal(np.asarray(sb.m), np.asarray(ss.m))


@pytest.mark.parametrize("prec", ["fp64", "fp32_field"])
@pytest.mark.parametrize("shape", [(9, 7, 1), (10, 7, 1), (300, 301, 1), (301, 301, 1)])
def test_error_norm_is_nan_where_a_quotient_is(shape, prec):
    """The norm's quotients err / (atol + rtol |m|) in meshes of odd and even cell counts (two
    kernels): 0 / 0 in empty cells with atol = 0, and a NaN in one cell, wherever it lies."""
    gm, _ = mesh_pair(*shape, 3e-9, 3e-9, 3e-9)
    terms = _terms()[0]
    m0 = random_m(shape, 5)
    s = M.State(gm, 8e5, m0, precision=prec)
    for atol in (1e-6, 0.0):
        assert np.isfinite(M.LLGIntegrator(0.1, terms, "RKF45", atol=atol).rk_attempt(s, "RKF45", 2e-14)[1])
    holes = m0.copy()
    holes[::3, 1::2] = 0.0
    s = M.State(gm, 8e5, holes, precision=prec)
    llg = M.LLGIntegrator(0.1, terms, "RKF45", atol=0.0)
    assert np.isnan(llg.rk_attempt(s, "RKF45", 2e-14)[1])
    with pytest.raises(M.MafError) as e:
        llg.step(s)
    assert e.value.code == 4
    last = m0.copy()
    for cell in ((0, 0, 0), (shape[0] - 1, shape[1] - 1, 0), (shape[0] // 2, shape[1] // 2, 0)):
        zeeman = np.zeros(shape + (3,))
        zeeman[cell] = np.nan
        s = M.State(gm, 8e5, last, precision=prec)
        err = M.LLGIntegrator(0.1, terms + [M.ExternalField(zeeman)], "RKF45").rk_attempt(s, "RKF45", 2e-14)[1]
        assert np.isnan(err)
