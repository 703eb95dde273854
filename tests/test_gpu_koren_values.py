"""The Koren limiter forms only the upwind side of a face, by quotients without the
compiler's division, where its values are of ordinary size, and both sides with `/`
elsewhere. Bit for bit the oracle, over fields that lie in, across and out of that range."""
import numpy as np
import pytest

import helpers
import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib(gpu):
    from scale_b200 import hevi

    yield hevi
    hevi.finalize()


@pytest.mark.parametrize("value", [0.0, 1e-310, 1e-200, 1e29, -3e29, 1e31, -1e35, 1e290], ids=str)
@pytest.mark.parametrize("fct", [False, True], ids=["plain", "fct"])
def test_koren_values(lib, value, fct):
    from test_gpu_parity import _tracer_inputs

    scheme = "UD3KOREN1993"
    g = helpers.small_grid(IMAX=9, JMAX=6, KMAX=34, DZ=12000.0 / 34)
    c = helpers.small_case(g)
    helpers.perturb_state(c)
    q0, q, d0, d, mflx, rhoq, GS, MAPF = _tracer_inputs(g, c)
    # single cells, and a block of equal values (the ratio's divisor vanishes there)
    for k, i, j in ((g.KS, g.IS, g.JS), (g.KS + 10, g.IS + 4, g.JS + 2), (g.KE, g.IE, g.JE)):
        q[k - 1, i - 1, j - 1] = value
    q[g.KS + 19:g.KS + 25, g.IS + 1:g.IS + 6, g.JS:g.JS + 4] = value
    ref = np.full(g.shape, np.nan, order="F")
    oracle.tstep_tracer(g, scheme, ref, q, q0, rhoq, d0, d, mflx, g.zeros(3), GS, MAPF, 2.5, fct, False)
    got = np.full(g.shape, np.nan, order="F")
    lib.setup(g.index_dict(), scheme, scheme)
    lib.ATMOS_DYN_Tstep_tracer_fvm_heve(QTRCo=got, QTRC=q, QTRC0=q0, RHOQ_t=rhoq, DENS0=d0, DENS=d, mflx_hi=mflx,
                                        num_diff=g.zeros(3), GSQRT=GS, MAPF=MAPF, CDZ=g.CDZ, RCDZ=g.RCDZ,
                                        RCDX=g.RCDX, RCDY=g.RCDY, dtl=2.5, FLAG_FCT_TRACER=fct,
                                        FLAG_FCT_ALONG_STREAM=False)
    assert helpers.same(got, ref), f"max rel diff {helpers.max_rel(got, ref):.3e}"
