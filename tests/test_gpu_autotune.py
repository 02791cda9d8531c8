"""The autotuners time each launch shape once: a precision-form tile height that the
tracer count gives by itself (rows 32) is no second candidate; and batches of the
precision form at the tracer counts whose kernels differ equal their domains stepped
alone, bit for bit."""
import re

import numpy as np
import pytest

from mom5_gb300 import grid

pytestmark = pytest.mark.gpu


def load(capi, ntr, sizes, precision):
    from mom5_gb300 import harness
    out = []
    for n, (ni, nj, nk, cx) in enumerate(sizes):
        sp = grid.DomainSpec(ni=ni, nj=nj, nk=nk, lon0=0.0, lon1=float(ni) * 0.5, lat0=-25.0, lat1=25.0, cyclic_x=cx,
                             continent=(ni // 3, nj // 3, max(2, ni // 8), max(2, nj // 8)), wavelength_cells=6.0,
                             ntracers=ntr, seed=7 + n)
        d = harness.load(grid.make_domain(sp),
                         options=capi.default_options(barotropic_time_stepping_B=1, precision=precision))
        d.barotropic_init(dtuv=200.0, dtbt=20.0)
        out.append(d)
    return out


SIZES = [(57, 33, 9, True), (29, 41, 6, False), (84, 24, 5, False)]


# heights by tracer count: one domain 16 up to 4 tracers, 20 above; batch 16 (1, 2, 7 to 10), 24 (3, 4), 20 (5, 6)
@pytest.mark.parametrize("ntr,one,batch", [(2, [24, 32], [24, 32]), (4, [24, 32], [16, 32]),
                                           (6, [16, 24, 32], [16, 24, 32]), (7, [16, 24, 32], [24, 32])])
def test_each_height_is_timed_once(gpu_lib, ntr, one, batch):
    capi = gpu_lib
    ds = load(capi, ntr, SIZES[:2], capi.PRECISION_MIXED)
    report = ds[0].autotune(3600.0)
    assert sorted(int(x) for x in re.findall(r"rows=(\d+): ", report)) == one, report
    b = capi.Batch(ds)
    report = b.autotune(3600.0)
    assert sorted(int(x) for x in re.findall(r"rows=(\d+) tj", report.split("chosen")[0])) == batch, report
    assert b.tuning[0] in batch
    b.close()
    for d in ds:
        d.close()


@pytest.mark.parametrize("ntr", [1, 6, 7])
def test_batch_of_the_precision_form_equals_single_steps(gpu_lib, ntr):
    capi = gpu_lib
    single, batched = (load(capi, ntr, SIZES, capi.PRECISION_MIXED) for _ in range(2))
    b = capi.Batch(batched)
    for p in (0, 1):
        b.step(3600.0, parity=p)
        for d in single:
            d.tracer_advection_step(1 + p, 1 + p, 2 - p, 3600.0)
            d.update_ocean_barotropic(1 + p, 2 - p)
    for s, t in zip(single, batched):
        for n in range(1, ntr + 1):
            assert np.array_equal(s.get(capi.F.TRACER, n=n, level=1), t.get(capi.F.TRACER, n=n, level=1)), n
        assert np.array_equal(s.get(capi.F.ETA_T_BAR, level=1), t.get(capi.F.ETA_T_BAR, level=1))
    b.close()
    for d in single + batched:
        d.close()
