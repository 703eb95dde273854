"""The stage kernels form their quotients without the compiler's division and
fall back to it where a divisor or a quotient leaves the range that covers;
these inputs leave it. The results equal, bit for bit (NaN where it has NaN), those
of the fused stage kernel, which divides with `/`."""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu

INF, NAN = np.inf, np.nan
# (field, value) put at a few cells of the stage input
SPECIAL = [
    ("DENS", 0.0), ("DENS", -1.0), ("DENS", INF), ("DENS", NAN), ("DENS", 1e-310), ("DENS", 1e305), ("DENS", 2.0 - 2.0**-52),
    ("RHOT", INF), ("RHOT", NAN), ("RHOT", 0.0), ("MOMX", INF), ("MOMY", -INF), ("MOMZ", NAN), ("MOMX", -0.0), ("MOMZ", 1e-200),
]


@pytest.fixture
def lib(gpu):
    from scale_b200 import hevi

    yield hevi
    hevi.finalize()


@pytest.mark.parametrize("scheme", ["UD3", "CD4", "UD5"])
@pytest.mark.parametrize("field,value", SPECIAL, ids=lambda v: str(v))
def test_stage_special_values(lib, scheme, field, value):
    # 70 levels: an interior chunk of 32 levels between two that touch a wall
    g = helpers.small_grid(IMAX=9, JMAX=6, KMAX=97 if scheme == "UD5" else 70, DZ=200.0, halo=helpers.halo_of(scheme))
    c = helpers.small_case(g, scheme)
    helpers.perturb_state(c)
    a = helpers.short_inputs(c, dtrk=0.5, full=True)
    for k, i, j in ((g.KS + 1, g.IS + 2, g.JS + 1), (g.KS + 40, g.IS + 4, g.JS + 3), (g.KE - 1, g.IE, g.JE)):
        a[field][k - 1, i - 1, j - 1] = value
    kw = dict(a)
    kw.update(PROG_RK=None, PROG0=None, PROG=None, FLAG_FCT_MOMENTUM=False, FLAG_FCT_T=False,
              FLAG_FCT_ALONG_STREAM=True, BND_W=False, BND_E=False, BND_S=False, BND_N=False, last=False)
    lib.setup(g.index_dict(), scheme, scheme)
    out, codes = [], []
    for tile_x in (0, 16):  # the staged form, the fused kernel
        lib.stage_shape(tile_x, 16)
        out.append(helpers.stage_outputs(g))
        try:
            lib.ATMOS_DYN_Tstep_short_fvm_hevi(**kw, **out[-1])
            codes.append(0)
        except lib.HeviError as e:  # SCALE_HEVI_ERR_NONFINITE; the outputs have come back
            codes.append(e.code)
    assert codes[0] == codes[1] and codes[0] in (0, 4)
    for n in out[0]:
        assert helpers.same(out[0][n], out[1][n]), n


# the levels at which the split march joins its chunks: a chunk's first own level is
# KS + 32, KS + 62, ..., and the level below it is run along for its fluxes
@pytest.mark.parametrize("scheme,size", [("UD3", (9, 6)), ("CD4", (148, 32)), ("UD5", (9, 6))], ids=lambda v: str(v))
@pytest.mark.parametrize("field,value", [("DENS", INF), ("DENS", NAN), ("DENS", 1e305), ("MOMZ", INF), ("MOMX", -INF),
                                         ("MOMY", INF)], ids=lambda v: str(v))
def test_stage_special_values_at_chunk_joins(lib, scheme, size, field, value):
    g = helpers.small_grid(IMAX=size[0], JMAX=size[1], KMAX=97, DZ=120.0, halo=helpers.halo_of(scheme))
    c = helpers.small_case(g, scheme)
    helpers.perturb_state(c)
    a = helpers.short_inputs(c, dtrk=0.5, full=True)
    for n, lev in enumerate((30, 31, 32, 60, 61, 62, 63, 91)):
        a[field][g.KS + lev - 1, g.IS + n - 1, g.JS + n % 6 - 1] = value
    kw = dict(a)
    kw.update(PROG_RK=None, PROG0=None, PROG=None, FLAG_FCT_MOMENTUM=False, FLAG_FCT_T=False,
              FLAG_FCT_ALONG_STREAM=True, BND_W=False, BND_E=False, BND_S=False, BND_N=False, last=False)
    lib.setup(g.index_dict(), scheme, scheme)
    out = []
    for tile_x in (0, 16):  # the staged form, the fused kernel
        lib.stage_shape(tile_x, 16)
        out.append(helpers.stage_outputs(g))
        try:
            lib.ATMOS_DYN_Tstep_short_fvm_hevi(**kw, **out[-1])
        except lib.HeviError as e:  # the outputs have come back
            assert e.code == 4
    for n in out[0]:
        assert helpers.same(out[0][n], out[1][n]), n
