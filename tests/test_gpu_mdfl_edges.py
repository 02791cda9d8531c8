"""The whole MDFL Sweby step (advection of every tracer, explicit update, halo
update) where its launches change: around the 127 cells of an x block, on domains
small enough that each tracer gets blocks of its own and just above, with one to
five tracers, one level to several level segments, closed and periodic sides.
Tracers and th_tendency, with their halos, equal the restatement value for value
(advect_tracer_mdfl_sweby, ocean_tracer_advect.F90:3806-4066; update_tracer,
ocean_tracer.F90:2341-2350), also where the halos held something else before."""
import numpy as np
import pytest

from mom5_gb300 import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cx,cy,ni,nj,nk,ntr", [
    (False, False, 127, 9, 1, 2), (True, False, 128, 11, 2, 3), (True, True, 126, 10, 5, 2), (False, True, 129, 7, 4, 1),
    (True, False, 130, 40, 20, 3), (False, False, 255, 33, 12, 5), (True, True, 254, 32, 10, 2), (True, True, 3, 4, 6, 2)])
def test_step_equals_restatement(gpu_lib, oracle_lib, cx, cy, ni, nj, nk, ntr):
    capi, O = gpu_lib, oracle_lib
    from mom5_gb300 import harness
    sp = grid.DomainSpec(ni=ni, nj=nj, nk=nk, lon0=0.0, lon1=float(ni), lat0=-20.0, lat1=20.0, cyclic_x=cx,
                         cyclic_y=cy, continent=(ni // 3, nj // 3, max(1, ni // 8), max(1, nj // 8)),
                         wavelength_cells=6.0, ntracers=ntr, seed=ni + nk)
    dom = grid.make_domain(sp)
    d = harness.load(dom, options=capi.default_options())
    dt = 3600.0
    g = O.domain_arrays(dom)
    dims = O.dims(sp)
    shape = g["T"][0].shape
    before = np.random.default_rng(5).standard_normal(shape)
    for n in range(1, ntr + 1):
        d.set(capi.F.TH_TENDENCY, before, n=n)
    d.tracer_advection_step(1, 1, 2, dt)
    for n in range(1, ntr + 1):
        T = g["T"][n - 1].copy()
        th = O.advect_mdfl_sweby(dims, g, T, dt)
        ref = O.update_tracer(dims, g, T, th, dt)
        assert np.array_equal(d.get(capi.F.TRACER, n=n, level=2).reshape(shape), ref), n
        assert np.array_equal(d.get(capi.F.TH_TENDENCY, n=n).reshape(shape), th.reshape(shape)), n
    d.close()
