"""PSOM on lines of several segments: rows above 126 cells, columns of rows above 30
and more than 30 levels, on domains whose launches are many times larger than what
the GPU holds at once, so that a segment runs after its neighbours have updated their
cells in place.  Three calls (the sweep orders xyz, zxy, yzx), every tendency and
moment equal to the restatement value for value (advect_tracer_psom,
ocean_tracer_advect.F90:4549-4660), and with the sides closed the tendencies sum to
zero: the two sides of a segment's end face form the same flux."""
import numpy as np
import pytest

from mom5_gb300 import grid

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cx,cy,ni,nj,nk,mode", [
    (False, False, 181, 101, 50, "mh"), (True, True, 253, 61, 31, "mh"), (True, False, 126, 91, 33, "prather"),
    (False, True, 127, 30, 61, "none"), (True, True, 379, 31, 30, "mh"), (False, False, 252, 120, 32, "prather")])
def test_segments(gpu_lib, oracle_lib, cx, cy, ni, nj, nk, mode):
    capi, O = gpu_lib, oracle_lib
    from mom5_gb300 import harness
    sp = grid.DomainSpec(ni=ni, nj=nj, nk=nk, lon0=0.0, lon1=float(ni) / 4, lat0=-20.0, lat1=20.0, cyclic_x=cx,
                         cyclic_y=cy, continent=(ni // 3, nj // 3, ni // 8, nj // 8), wavelength_cells=6.0,
                         ntracers=1, seed=ni + nk)
    dom = grid.make_domain(sp)
    d = harness.load(dom, options=capi.default_options(psom_limit_prather=int(mode == "prather")),
                     scheme=capi.ADVECT_PSOM)
    d.set_psom_limit(1, mode != "none")
    g = O.domain_arrays(dom)
    dims = O.dims(sp)
    dt = 3600.0
    shape = g["T"][0].shape
    inner = (slice(None), slice(1, -1), slice(1, -1))
    mom = np.zeros((9,) + shape)
    for itt0 in range(3):
        d.set_itt0(itt0)
        d.zero_th_tendency(1)
        d.horz_advect_tracer(1, 1, 1, dt)
        got = d.get(capi.F.TH_TENDENCY, n=1).reshape(shape)
        ref, s0 = O.advect_psom(dims, g, g["T"][0].copy(), dt, mom, itt0=itt0, limit=mode != "none",
                                prather=mode == "prather")
        assert np.abs(ref).max() > 0
        assert np.array_equal(got, ref), (itt0, int((got != ref).sum()), float(np.abs(got - ref).max()))
        if not (cx or cy):
            flux = got[inner] * g["dat"].reshape(shape[1:])[1:-1, 1:-1]
            assert abs(flux.sum()) <= 1e-12 * np.abs(flux).sum()
    for q in range(9):
        m = d.get(capi.F.PSOM_SX + q, n=1).reshape(shape)[inner]
        assert np.array_equal(m, mom[q][inner]), q
    assert np.array_equal(d.get(capi.F.PSOM_S0, n=1).reshape(shape)[inner], s0[inner])
    d.close()
