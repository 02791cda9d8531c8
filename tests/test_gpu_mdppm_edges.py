"""MDPPM where its lines change shape: lengths around the cells a segment closes (16,
32, 40, 56, 72, 88, 120, 184), single levels, each edge limiter, closed and periodic
sides.
Tendencies equal the restatement value for value (advect_tracer_mdppm,
ocean_tracer_advect.F90:5990-6507)."""
import numpy as np
import pytest

from mom5_gb300 import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cx,cy,ni,nj,nk,limiter", [
    (False, False, 56, 24, 16, 2), (True, False, 57, 25, 17, 1), (True, True, 88, 40, 33, 3),
    (False, True, 89, 41, 1, 2), (True, False, 184, 56, 2, 2), (False, False, 185, 57, 5, 3),
    (True, True, 4, 5, 57, 1), (False, False, 121, 73, 6, 2), (True, True, 40, 33, 20, 3)])
def test_line_lengths(gpu_lib, oracle_lib, cx, cy, ni, nj, nk, limiter):
    capi, O = gpu_lib, oracle_lib
    from mom5_gb300 import harness
    sp = grid.DomainSpec(ni=ni, nj=nj, nk=nk, lon0=0.0, lon1=float(ni), lat0=-20.0, lat1=20.0, cyclic_x=cx,
                         cyclic_y=cy, continent=(ni // 3, nj // 3, max(1, ni // 8), max(1, nj // 8)),
                         wavelength_cells=6.0, ntracers=1, seed=ni + nk)
    dom = grid.make_domain(sp)
    d = harness.load(dom, options=capi.default_options(), scheme=capi.ADVECT_MDPPM)
    d.set_ppm_limiter(1, limiter)
    g = O.domain_arrays(dom)
    dims = O.dims(sp)
    dt = 3600.0
    d.zero_th_tendency(1)
    d.horz_advect_tracer(1, 1, 1, dt)
    d.vert_advect_tracer(1, 1, 1, dt)
    got = d.get(capi.F.TH_TENDENCY, n=1)
    ref = O.advect_mdppm(dims, g, g["T"][0].copy(), dt, limiter)
    assert np.abs(ref).max() > 0
    assert np.array_equal(got.reshape(ref.shape), ref), np.abs(got.reshape(ref.shape) - ref).max()
    d.close()
