"""The explicit kernel of the tiled stage takes a column's chunks of 32 levels either
one per thread block, 30 levels apart with two ghost levels (few tiles), or one after
another in one block (enough tiles to fill the chip). Both give the bits of the fused
stage kernel, at the depths where the number of chunks and the last one's levels change."""
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib(gpu):
    from scale_b200 import hevi

    yield hevi
    hevi.stage_shape(0, 0)
    hevi.finalize()


# few tiles: one chunk per block; 296 tiles of 4x4 (148 for the 6-point schemes): a march
@pytest.mark.parametrize("kmax", [31, 32, 33, 34, 35, 61, 62, 63, 64, 65, 92, 93, 123])
@pytest.mark.parametrize("scheme,size", [("UD3", (6, 5)), ("CD4", (148, 32)), ("UD5", (5, 4)), ("CD6", (148, 16))],
                         ids=lambda v: str(v))
def test_split_and_marched_columns(lib, scheme, size, kmax):
    g = helpers.small_grid(IMAX=size[0], JMAX=size[1], KMAX=kmax, DZ=12000.0 / kmax, halo=helpers.halo_of(scheme))
    c = helpers.small_case(g, scheme)
    helpers.perturb_state(c)
    kw = dict(helpers.short_inputs(c, dtrk=0.5, full=True))
    kw.update(PROG_RK=None, PROG0=None, PROG=None, FLAG_FCT_MOMENTUM=False, FLAG_FCT_T=False,
              FLAG_FCT_ALONG_STREAM=True, BND_W=False, BND_E=False, BND_S=False, BND_N=False, last=False)
    lib.setup(g.index_dict(), scheme, scheme)
    out = []
    for tile_x in (0, 16):  # the tiled form, the fused kernel
        lib.stage_shape(tile_x, 16)
        out.append(helpers.stage_outputs(g))
        lib.ATMOS_DYN_Tstep_short_fvm_hevi(**kw, **out[-1])
    for n in out[0]:
        assert helpers.same(out[0][n], out[1][n]), n


# tiles that reach beyond the domain, and beyond the array, by 1 to 3 columns; odd KA stages
# with cp.async, which leaves what lies beyond the array as it was
@pytest.mark.parametrize("kmax", [40, 41, 65])
@pytest.mark.parametrize("size", [(5, 6), (6, 7), (7, 5), (8, 8), (33, 29)], ids=str)
@pytest.mark.parametrize("scheme", ["UD3", "UD3KOREN1993", "UD5"])
def test_ragged_tiles(lib, scheme, size, kmax):
    test_split_and_marched_columns(lib, scheme, size, kmax)
