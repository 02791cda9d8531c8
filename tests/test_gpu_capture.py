"""Steps captured by the caller into a CUDA graph of its own (mom5gpu_set_stream): the
kernels launched as programmatic dependents (advection of small domains, both grids'
subcycles), the precision form, and schemes with scratch launches of their own, also
behind a copy that joins from another stream.  Replays give the values of the same
steps launched one by one."""
import numpy as np
import pytest

from mom5_gb300 import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme,mixed,cgrid,ni,nj,nk", [
    ("ADVECT_MDFL_SWEBY", False, False, 37, 29, 12), ("ADVECT_MDFL_SWEBY", False, True, 61, 33, 4),
    ("ADVECT_MDFL_SWEBY", True, False, 57, 41, 9), ("ADVECT_MDFL_SWEBY", False, False, 363, 241, 2),
    ("ADVECT_MDPPM", False, False, 45, 37, 6), ("ADVECT_PSOM", False, False, 131, 35, 33)])
def test_replayed_steps(gpu_lib, scheme, mixed, cgrid, ni, nj, nk):
    capi = gpu_lib
    import torch
    from mom5_gb300 import harness
    sp = grid.DomainSpec(ni=ni, nj=nj, nk=nk, lon0=0.0, lon1=min(360.0, float(ni)), lat0=-30.0, lat1=30.0, cyclic_x=True,
                         continent=(ni // 3, nj // 3, max(1, ni // 8), max(1, nj // 8)), wavelength_cells=6.0,
                         ntracers=2, seed=ni)
    ds = []
    for _ in range(2):
        d = harness.load(grid.make_domain(sp), scheme=getattr(capi, scheme),
                         options=capi.default_options(barotropic_time_stepping_B=1,
                                                      precision=capi.PRECISION_MIXED if mixed else capi.PRECISION_FP64),
                         horz_grid=capi.CGRID if cgrid else capi.BGRID)
        d.barotropic_init(dtuv=100.0, dtbt=20.0)
        ds.append(d)
    single, captured = ds
    main, side = torch.cuda.Stream(), torch.cuda.Stream()
    for d in ds:
        d.set_stream(main.cuda_stream)
    surface = torch.zeros(single.count(capi.F.PME), dtype=torch.float64).pin_memory()

    def steps(d, join):
        for p in (0, 1):
            if join:  # an upload on another stream between the steps
                side.wait_stream(main)
                d.copy_field_async(capi.F.PME, surface.data_ptr(), 1, side.cuda_stream)
                main.wait_stream(side)
            d.tracer_advection_step(1 + p, 1 + p, 2 - p, 3600.0)
            d.update_ocean_barotropic(1 + p, 2 - p)

    with torch.cuda.stream(main):
        for d in ds:  # the first calls allocate
            steps(d, False)
            d.copy_field_async(capi.F.PME, surface.data_ptr(), 1, main.cuda_stream)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        g.capture_begin()
        steps(captured, True)
        g.capture_end()
        for _ in range(2):
            g.replay()
            steps(single, False)
    torch.cuda.synchronize()
    for level in (1, 2):
        for n in (1, 2):
            a, b = (d.get(capi.F.TRACER, n=n, level=level) for d in ds)
            assert np.isfinite(a).all() and np.array_equal(a, b), (level, n)
        for f in (capi.F.ETA_T_BAR, capi.F.UDRHO_U, capi.F.UDRHO_V):
            a, b = (d.get(f, level=level) for d in ds)
            assert np.array_equal(a, b), (level, f)
    g.reset()
    for d in ds:
        d.close()
