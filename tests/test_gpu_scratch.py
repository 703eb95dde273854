"""The device memory the library holds for itself: what the stage kernels use and no
more. At setup the three RK buffers (15 fields), the flux sums (6), the column sources
(4) and the column right-hand side (1); 13 work fields more for terrain-following
metrics. The allocator rounds each buffer up to 2 MiB; half a field covers that."""
import numpy as np
import pytest

import helpers
from scale_b200 import hevi
from test_gpu_terrain import _stage_kw, with_terrain

pytestmark = pytest.mark.gpu


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_setup_holds_26_fields(gpu):
    g = helpers.small_grid(IMAX=244, JMAX=244, KMAX=128, DZ=100.0)
    field = 8 * int(np.prod(g.shape))
    for _ in range(2):  # the first setup also brings up the context
        before = _free()
        hevi.setup(g.index_dict(), "UD3", "UD3")
        held = before - _free()
        hevi.finalize()
    assert 26 * field <= held <= 26.5 * field, held / field


@pytest.mark.parametrize("short", ["HEVI", "HEVE"])
def test_terrain_holds_13_fields_more(gpu, short):
    import torch

    held = None
    for n in (8, 140):  # the small domain loads the kernels
        g = helpers.small_grid(IMAX=n, JMAX=n, KMAX=120, DZ=100.0)
        c = helpers.small_case(g, "UD3")
        a = with_terrain(helpers.short_inputs(c, dtrk=0.1, full=False), g)
        o = helpers.stage_outputs(g, 0.0)
        dev = lambda x: torch.from_numpy(np.ravel(x, order="F").copy()).cuda()  # noqa: E731
        ad = {k: dev(v) if isinstance(v, np.ndarray) and v.ndim >= 2 else v for k, v in a.items()}
        od = {k: dev(v) for k, v in o.items()}
        hevi.setup(g.index_dict(), "UD3", "UD3")
        try:
            before = _free()
            fn = hevi.ATMOS_DYN_Tstep_short_fvm_hevi_dev if short == "HEVI" else hevi.ATMOS_DYN_Tstep_short_fvm_heve_dev
            fn(**_stage_kw(ad, od))
            hevi.check()
            held = (before - _free()) / (8 * int(np.prod(g.shape)))
        finally:
            hevi.finalize()
    assert 13 <= held <= 13.5, held
