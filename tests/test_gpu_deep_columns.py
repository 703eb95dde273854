"""Columns of more than one pass of 32 levels: the warp-per-column kernels carry the
fluxes below a level from one pass to the next (terrain stage) or gather a level's
neighbours across passes (adjoint), and an ensemble's members differ in their number of
chunks. KMAX on, below and above multiples of 32, and the deepest."""
import numpy as np
import pytest

import helpers
import oracle
from scale_b200 import adjoint, hevi, mkinit
from scale_b200.ensemble import STATE, Ensemble
from test_gpu_terrain import SHORT_KW, _short_inputs, _stage_kw, with_terrain

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib(gpu):
    yield hevi
    hevi.finalize()


@pytest.mark.parametrize("scheme", ["UD3", "CD4", "UD5"])
@pytest.mark.parametrize("kmax", [31, 32, 33, 64, 65, 97, 256])
def test_terrain_stage(lib, scheme, kmax):
    g = helpers.small_grid(IMAX=17, JMAX=5, KMAX=kmax, DZ=12000.0 / kmax, halo=helpers.halo_of(scheme))
    c = helpers.small_case(g, scheme)
    helpers.perturb_state(c)
    a = with_terrain(helpers.short_inputs(c, dtrk=0.5, full=True), g)
    ref, got = helpers.stage_outputs(g), helpers.stage_outputs(g)
    oracle.tstep_short(g, scheme, ref, a)
    lib.setup(g.index_dict(), scheme, scheme)
    lib.ATMOS_DYN_Tstep_short_fvm_hevi(**_stage_kw(a, got))
    for n in ref:
        assert helpers.same(got[n], ref[n]), f"{n}: max rel diff {helpers.max_rel(got[n], ref[n]):.3e}"


@pytest.mark.parametrize("scheme", ["UD3", "CD4", "UD5"])
@pytest.mark.parametrize("kmax", [33, 64, 97])
def test_terrain_rk4(lib, scheme, kmax):
    g = helpers.small_grid(IMAX=9, JMAX=7, KMAX=kmax, DZ=12000.0 / kmax, halo=helpers.halo_of(scheme))
    a, ref = _short_inputs(g, scheme)
    got = {n: v.copy(order="F") for n, v in ref.items()}
    oracle.tinteg_short_rk4(g, scheme, ref, dict(a, dt=0.2))
    lib.setup(g.index_dict(), scheme, scheme)
    lib.ATMOS_DYN_Tinteg_short_rk4(**a, **got, **SHORT_KW, dt=0.2)
    for n in ref:
        assert helpers.same(got[n], ref[n]), f"{n}: max rel diff {helpers.max_rel(got[n], ref[n]):.3e}"


@pytest.mark.parametrize("scheme", ["UD3", "CD4", "UD3KOREN1993"])
@pytest.mark.parametrize("kmax", [32, 33, 34, 64, 70])
def test_adjoint(lib, scheme, kmax):
    """The pass form reproduces the fused step and the adjoint is the transpose of the
    tangent-linear model, with the bounds of the shallow cases."""
    g = helpers.small_grid(IMAX=10, JMAX=9, KMAX=kmax, DZ=12000.0 / kmax)
    c = helpers.small_case(g, scheme)
    c.dt = 0.25
    lib.setup(g.index_dict(), scheme, scheme)
    m = adjoint.Model(c)
    X = m.state()
    m.boundary(X)
    m.step(X)
    Xa, Xb = X.clone(), X.clone()
    m.step(Xa)
    m.step_passes(Xb)
    hevi.check()
    assert (Xa - Xb).abs().max().item() <= 1e-12 * Xa.abs().max().item()
    r = adjoint.dot_product_test(m, X, 2)
    assert r["rel_diff"] < 1e-11, r


def _run(cases, nsteps):
    e = Ensemble(cases)
    try:
        e.run(nsteps)
        return e.members()
    finally:
        e.close()


# few tiles: one chunk per thread block; many: each block marches up its columns
@pytest.mark.parametrize("size", [(9, 7), (64, 60)], ids=["split", "march"])
@pytest.mark.parametrize("scheme", ["UD3", "UD5"])
def test_ensemble_of_unequal_depths(gpu, scheme, size):
    I, J = size
    sizes = [(I, J, 20), (I + 3, J, 33), (I, J + 5, 64), (I + 1, J + 2, 97)]
    cases = mkinit.ensemble(sizes=sizes, scheme=scheme)
    together = _run(cases, 2)
    for m, c in enumerate(cases):
        alone = _run([c], 2)[0]
        for n in STATE:
            d = np.max(np.abs(together[m][n] - alone[n]))
            assert np.array_equal(together[m][n], alone[n]), f"member {m} {n}: max diff {d:.3e}"
