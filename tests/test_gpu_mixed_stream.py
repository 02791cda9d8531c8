"""The precision form's tile at its edges: domains around multiples of the 28
columns and of the 12, 16 and 20 rows a tile advances, one to ten tracers (an odd
count leaves half a tracer pair empty), columns of one level to several level
segments, both halo modes.  One step against the FP64 drop-in, itself equal value
for value to the restatement of advect_tracer_mdfl_sweby
(ocean_tracer_advect.F90:3806-4066), within the form's 1e-6 of the tracer's
maximum; and the tile heights, which cut a domain into different tiles and
segments, against each other bit for bit."""
import numpy as np
import pytest

from mom5_gb300 import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cx,cy,ni,nj,nk,ntr", [
    (False, False, 28, 12, 1, 1), (True, False, 29, 13, 2, 2), (True, True, 27, 11, 3, 3), (False, True, 57, 41, 24, 5),
    (True, False, 84, 40, 31, 6), (False, False, 31, 37, 9, 7), (True, True, 56, 33, 12, 9), (True, False, 13, 21, 50, 10)])
def test_tile_edges(gpu_lib, cx, cy, ni, nj, nk, ntr):
    capi = gpu_lib
    from mom5_gb300 import harness
    sp = grid.DomainSpec(ni=ni, nj=nj, nk=nk, lon0=0.0, lon1=float(ni), lat0=-20.0, lat1=20.0, cyclic_x=cx,
                         cyclic_y=cy, continent=(ni // 3, nj // 3, max(2, ni // 8), max(2, nj // 8)),
                         wavelength_cells=6.0, ntracers=ntr, seed=ni + nk)
    dom = grid.make_domain(sp)
    out = {}
    for prec, rows in ((capi.PRECISION_FP64, 0), (capi.PRECISION_MIXED, 32), (capi.PRECISION_MIXED, 16),
                       (capi.PRECISION_MIXED, 24)):
        d = harness.load(dom, options=capi.default_options(precision=prec))
        if rows:
            d.tuning = (rows, 0, 0)
        d.tracer_advection_step(1, 1, 2, 3600.0)
        out[rows] = [d.get(capi.F.TRACER, n=n, level=2) for n in range(1, ntr + 1)]
        d.close()
    for n in range(ntr):
        err = np.abs(out[32][n] - out[0][n]).max() / np.abs(out[0][n]).max()
        assert err <= 1e-6, (n, err)
        for rows in (16, 24):
            assert np.array_equal(out[rows][n], out[32][n]), (rows, n)
