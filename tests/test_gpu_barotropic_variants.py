"""The barotropic subcycle's kernels at sizes on each side of the rules that choose
them by the number of columns: products on the FP64 or the integer pipe, loads before
or after the wait for the previous launch, blocks of 64 or 128 threads; exact form on
both grids, precision form, batches, odd extents, closed and periodic sides, both time
steppings, a few subcycles.  The exact form equals the restatement of
update_ocean_barotropic (ocean_barotropic.F90:2763-3033) value for value; the
precision form stays within its 1e-6; a batch equals its domains stepped alone."""
import numpy as np
import pytest

from mom5_gb300 import grid

pytestmark = pytest.mark.gpu

DTBT = 20.0
LEVEL_FIELDS = ("eta_t_bar", "udrho_u", "udrho_v", "conv_rho_ud_t", "eta_u")
FIELDS = ("ps", "grad_ps_x", "grad_ps_y")


def domain(ni, nj, cx, cy, ntr=0, nk=1, seed=0):
    sp = grid.DomainSpec(ni=ni, nj=nj, nk=nk, lon0=0.0, lon1=min(360.0, float(ni)), lat0=-55.0, lat1=55.0,
                         cyclic_x=cx, cyclic_y=cy, hmin=None, ridge_amp=1200.0, ntracers=ntr, seed=seed + ni,
                         continent=None if cy else (ni // 3, nj // 3, max(2, ni // 9), max(2, nj // 9)))
    return sp, grid.make_domain(sp)


# columns of the data domain: 5538, 88935, 111325, 125139, 316713
SIZES = [(69, 76), (361, 243), (363, 303), (411, 301), (577, 545)]


@pytest.mark.parametrize("cgrid", [False, True])
@pytest.mark.parametrize("ni,nj", SIZES)
@pytest.mark.parametrize("cx,cy,step_b", [(True, False, True), (False, False, False), (True, True, True)])
def test_exact_form(gpu_lib, oracle_lib, ni, nj, cx, cy, step_b, cgrid):
    capi, O = gpu_lib, oracle_lib
    from mom5_gb300 import harness
    sp, dom = domain(ni, nj, cx, cy)
    d = harness.load(dom, options=capi.default_options(barotropic_time_stepping_A=int(not step_b),
                                                       barotropic_time_stepping_B=int(step_b)),
                     horz_grid=capi.CGRID if cgrid else capi.BGRID)
    nts = d.barotropic_init(dtuv=7 * DTBT / 2, dtbt=DTBT)
    g, dims = O.domain_arrays(dom), O.dims(sp)
    st = {k: dom[k].numpy().copy() for k in ("eta_t", "eta_t_bar", "udrho_u", "udrho_v")}
    tau = 1
    for step in range(2):
        d.update_ocean_barotropic(tau, 3 - tau)
        out = O.update_ocean_barotropic(dims, g, st, nts, DTBT, time_stepping_B=step_b, cgrid=cgrid)
        for k in LEVEL_FIELDS + FIELDS:
            got = d.get(getattr(capi.F, k.upper()), **({"level": 3 - tau} if k in LEVEL_FIELDS else {})).ravel()
            ref = np.asarray(out[k]).ravel()
            assert np.array_equal(got, ref), (step, k, int((got != ref).sum()), float(np.abs(got - ref).max()))
        st = {"eta_t": st["eta_t"], **{k: out[k] for k in ("eta_t_bar", "udrho_u", "udrho_v")}}
        d.set(capi.F.ETA_T, np.ascontiguousarray(st["eta_t"]), level=3 - tau)
        tau = 3 - tau
    assert np.abs(out["udrho_u"]).max() > 0
    d.close()


@pytest.mark.parametrize("ni,nj", SIZES)
@pytest.mark.parametrize("cx,cy,step_b", [(True, False, True), (False, False, False), (True, True, True)])
def test_precision_form(gpu_lib, oracle_lib, ni, nj, cx, cy, step_b):
    capi, O = gpu_lib, oracle_lib
    from mom5_gb300 import harness
    sp, dom = domain(ni, nj, cx, cy)
    d = harness.load(dom, options=capi.default_options(barotropic_time_stepping_A=int(not step_b),
                                                       barotropic_time_stepping_B=int(step_b),
                                                       precision=capi.PRECISION_MIXED))
    nts = d.barotropic_init(dtuv=7 * DTBT / 2, dtbt=DTBT)
    g, dims = O.domain_arrays(dom), O.dims(sp)
    st = {k: dom[k].numpy().copy() for k in ("eta_t", "eta_t_bar", "udrho_u", "udrho_v")}
    d.update_ocean_barotropic(1, 2)
    out = O.update_ocean_barotropic(dims, g, st, nts, DTBT, time_stepping_B=step_b)
    for k in ("eta_t_bar", "udrho_u", "udrho_v"):
        got = d.get(getattr(capi.F, k.upper()), level=2).ravel()
        ref = np.asarray(out[k]).ravel()
        assert np.abs(got - ref).max() <= 1e-6 * np.abs(ref).max(), k
    d.close()


@pytest.mark.parametrize("fusion", [1, 2])
@pytest.mark.parametrize("ni,nj", [(69, 76), (411, 301), (577, 545)])
def test_one_launch_forms(gpu_lib, ni, nj, fusion):
    """One launch per subcycle, and one for all of them, whose blocks walk the columns
    in one round on 411x301 and in three on 577x545: the bits of the default form."""
    capi = gpu_lib
    from mom5_gb300 import harness
    _, dom = domain(ni, nj, True, False)
    out = {}
    for form in (0, fusion):
        d = harness.load(dom, options=capi.default_options(barotropic_time_stepping_B=1))
        d.barotropic_init(dtuv=7 * DTBT / 2, dtbt=DTBT)
        d.set_barotropic_fusion(form)
        d.update_ocean_barotropic(1, 2)
        d.synchronize()
        out[form] = [d.get(getattr(capi.F, k.upper()), level=2) for k in LEVEL_FIELDS]
        d.close()
    for k, x, y in zip(LEVEL_FIELDS, out[0], out[fusion]):
        assert np.array_equal(x, y), k


# columns of the lists, each domain rounded up to blocks of 128: about 89000, 119000 and 346000
LISTS = [[(200, 150), (180, 160), (170, 165)], [(200, 150), (180, 160), (170, 165), (251, 117)],
         [(577, 545), (200, 150)]]


@pytest.mark.parametrize("sizes", LISTS)
@pytest.mark.parametrize("mixed", [False, True])
def test_batch_equals_single_steps(gpu_lib, sizes, mixed):
    capi = gpu_lib
    from mom5_gb300 import harness
    prec = capi.PRECISION_MIXED if mixed else capi.PRECISION_FP64
    sets = []
    for _ in range(2):
        ds = []
        for n, (ni, nj) in enumerate(sizes):
            _, dom = domain(ni, nj, n % 2 == 0, False, ntr=1, nk=2, seed=n)
            ds.append(harness.load(dom, options=capi.default_options(barotropic_time_stepping_B=1, precision=prec)))
            ds[-1].barotropic_init(dtuv=7 * DTBT / 2, dtbt=DTBT)
        sets.append(ds)
    single, batched = sets
    b = capi.Batch(batched)
    for p in (0, 1):
        b.step(600.0, parity=p)
        for d in single:
            d.tracer_advection_step(1 + p, 1 + p, 2 - p, 600.0)
            d.update_ocean_barotropic(1 + p, 2 - p)
    for n, (s, t) in enumerate(zip(single, batched)):
        assert np.array_equal(s.get(capi.F.TRACER, n=1, level=1), t.get(capi.F.TRACER, n=1, level=1)), n
        for k in LEVEL_FIELDS:
            f = getattr(capi.F, k.upper())
            x, y = s.get(f, level=1), t.get(f, level=1)
            assert np.array_equal(x, y), (n, k, float(np.abs(x - y).max()))
    b.close()
    for d in single + batched:
        d.close()
