"""The timing sections (mom5gpu_timing_query): every whole step counts as a call of
"tracer_update" whichever kernels form the update, with a time of its own where it is a
launch of its own."""
import pytest

from mom5_gb300 import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", ["ADVECT_MDFL_SWEBY", "ADVECT_UPWIND"])
def test_update_calls_are_counted(gpu_lib, scheme):
    capi = gpu_lib
    from mom5_gb300 import harness
    sp = grid.DomainSpec(ni=40, nj=30, nk=6, lon0=0.0, lon1=40.0, lat0=-20.0, lat1=20.0, cyclic_x=True,
                         wavelength_cells=6.0, ntracers=2, seed=3)
    d = harness.load(grid.make_domain(sp), options=capi.default_options(), scheme=getattr(capi, scheme))
    d.enable_timing(True)
    for _ in range(3):
        d.tracer_advection_step(1, 1, 2, 3600.0)
    update_ms, update_calls = d.timing("tracer_update")
    assert update_calls == 3
    if scheme == "ADVECT_UPWIND":
        assert update_ms > 0
    else:
        ms, calls = d.timing("mdfl")
        assert calls == 3 and ms > 0
    d.enable_timing(True)
    assert d.timing("tracer_update") == (0.0, 0)
    d.close()
