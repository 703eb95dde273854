"""The tiled stage and filter stage their boxes by bulk tensor copies where the
arrays admit tensor maps and with cp.async otherwise. Here the same arrays lie on
and 8 bytes off a 16-byte boundary; both give the same bits. (Odd KA and ensembles,
which always take cp.async, are compared with the oracle and with single domains in
the edge-size and ensemble tests.)"""
import numpy as np
import pytest

import helpers

pytestmark = pytest.mark.gpu


@pytest.fixture
def lib(gpu):
    from scale_b200 import hevi

    yield hevi
    hevi.finalize()


@pytest.mark.parametrize("size", [(2, 3, 4, "CD4"), (9, 6, 28, "UD3"), (17, 5, 64, "UD3KOREN1993"), (7, 13, 96, "CD6")],
                         ids=lambda s: "x".join(map(str, s)))
def test_unaligned_arrays_give_the_same_bits(lib, size):
    import torch

    I, J, K, scheme = size
    if scheme == "CD6":
        I, J = max(I, 3), max(J, 3)
    g = helpers.small_grid(IMAX=I, JMAX=J, KMAX=K, DZ=12000.0 / K, halo=helpers.halo_of(scheme))
    c = helpers.small_case(g, scheme)
    helpers.perturb_state(c)
    a = helpers.short_inputs(c, dtrk=0.5, full=True)
    n3 = int(np.prod(g.shape))
    res = []
    for off in (0, 1):

        def dev(x, k=1):
            buf = torch.full((k * n3 + 2,), float("nan"), dtype=torch.float64, device="cuda")
            v = buf[off:off + k * n3]
            if x is not None:
                v.copy_(torch.from_numpy(np.ravel(x, order="F").copy()))
            return v

        lib.setup(g.index_dict(), scheme, scheme)
        kw = {}
        for n, v in a.items():
            big = isinstance(v, np.ndarray) and v.ndim >= 3 and n not in ("GSQRT", "J13G", "J23G", "MAPF")
            kw[n] = dev(v, v.size // n3) if big else v
        for n in ("GSQRT", "J13G", "J23G", "MAPF"):
            kw[n] = None
        kw["CORIOLI"] = torch.from_numpy(np.ravel(a["CORIOLI"], order="F").copy()).cuda()
        out = {n: dev(None) for n in ("DENS_RK", "MOMZ_RK", "MOMX_RK", "MOMY_RK", "RHOT_RK")}
        out.update(mflx_hi=dev(None, 3), tflx_hi=dev(None, 3))
        kw.update(PROG_RK=None, PROG0=None, PROG=None, FLAG_FCT_MOMENTUM=False, FLAG_FCT_T=False,
                  FLAG_FCT_ALONG_STREAM=True, BND_W=False, BND_E=False, BND_S=False, BND_N=False, last=False)
        lib.ATMOS_DYN_Tstep_short_fvm_hevi_dev(**kw, **out)
        nd = dev(None, 15)
        X = {n: kw[n] for n in ("DENS", "MOMZ", "MOMX", "MOMY", "RHOT")}
        lib.ATMOS_DYN_numfilter_coef_dev(num_diff=nd, DT=0.5, REF_dens=kw["REF_dens"], REF_pott=dev(c.ref["REF_pott"]),
                                         ND_COEF=1e-3, ND_ORDER=1, ND_SFC_FACT=0.7, ND_USE_RS=True, **X,
                                         **{n: getattr(g, n) for n in ("CDZ", "CDX", "CDY", "FDZ", "FDX", "FDY")})
        lib.check()
        res.append({n: v.cpu().numpy() for n, v in dict(out, num_diff=nd).items()})
    for n in res[0]:
        assert helpers.same(res[0][n], res[1][n]), n
