"""GPU tests of the packed column kernels at the column counts where they take another
form: soil_temperature! with 1, 2 or 4 columns per warp or 32 per block (a partial last
group, and blocks that share columns sorted by snow-layer count), and the packed Richards
solve with 1 to 16 columns per warp.  The bits are the oracle's, over columns of every
kind: snow counts, ponded water, unresolved snow, excess ice, bedrock, wetland, ice and
urban landunits, several patches, masks, out-of-range counts and patch ranges, and ground
fluxes that make the band elimination exchange rows."""
import numpy as np
import pytest

from clmgb import abi, api, synth
from clmgb.state import ColumnState
from oracle import oracle as O
from parity import FLOAT_OUT, INT_OUT, bit_mismatches

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

ST_OUT = [k for k in FLOAT_OUT if k not in ("smp_l", "hk_l", "qcharge", "num_substeps", "forc_lwrad", "t_ssbef",
                                            "t_h2osfc_bef", "eff_porosity", "icefrac")] + INT_OUT


def _varied(nc, seed):
    """Snow and frozen-soil columns (two patches each) with every kind of column among them."""
    rng = np.random.default_rng(seed)
    one = synth.make_workload(1, nc=nc, seed=seed, nsteps=1).state
    st = ColumnState(one.vp, nc, 2 * nc, 4)
    for k, (_, _, kind, _) in st.spec.items():
        if kind == "p":
            st[k][:] = np.repeat(one[k], 2, axis=-1)
        elif kind == "c":
            st[k][:] = one[k]
    a, some = st.arrays, lambda p: rng.random(nc) < p  # noqa: E731
    c1 = np.arange(1, nc + 1)
    a["lun_itype"][:] = [1, 6, 4, 1]                  # soil, wetland, ice, urban
    a["lun_urbpoi"][:] = [0, 0, 0, 1]
    lu = np.where(some(0.8), 1, rng.integers(2, 5, nc))
    a["col_landunit"][:] = lu
    a["patch_landunit"][:] = np.repeat(lu, 2)
    a["patch_column"][:] = np.repeat(c1, 2)
    a["col_patchi"][:], a["col_patchf"][:] = 2 * c1 - 1, 2 * c1
    w = rng.uniform(0.1, 0.9, nc)
    a["patch_wtcol"][:] = np.stack([w, 1.0 - w], axis=1).ravel()
    a["patch_wtcol"][rng.random(2 * nc) < 0.05] = 0.0
    a["mask_nolakep"][rng.random(2 * nc) < 0.05] = 0
    for k, sd in (("eflx_sh_grnd", 30.0), ("eflx_sh_soil", 30.0), ("eflx_sh_snow", 30.0), ("eflx_sh_h2osfc", 30.0),
                  ("dlrad", 40.0), ("qflx_evap_soi", 2e-5), ("qflx_ev_soil", 2e-5), ("qflx_ev_snow", 2e-5)):
        a[k][:] = rng.normal(0.0, sd, 2 * nc)
    # ground-flux derivatives up to where a row's diagonal vanishes: the rows are exchanged
    a["cgrnd"][:] = np.where(rng.random(2 * nc) < 0.3, rng.uniform(-3000.0, 0.0, 2 * nc), rng.uniform(0.0, 40.0, 2 * nc))
    a["col_nbedrock"][:] = rng.integers(1, st.vp.nlevsoi + 1, nc)
    ponded, none = some(0.25), a["col_snl"] == 0
    a["frac_h2osfc"][:] = np.where(ponded, rng.uniform(0.05, 0.6, nc), 0.0)
    a["frac_sno_eff"][:] = np.where(ponded, 0.3, a["frac_sno_eff"])
    a["h2osfc"][:] = np.where(ponded, rng.uniform(0.0, 20.0, nc), 0.0)
    a["t_h2osfc"][:] = np.where(ponded, rng.uniform(265.0, 280.0, nc), a["t_h2osfc"])
    a["h2osno_no_layers"][:] = np.where(none & some(0.4), rng.uniform(0.0, 30.0, nc), 0.0)
    a["snow_depth"][:] = np.where(none, a["h2osno_no_layers"] / 200.0, a["snow_depth"])
    a["h2osoi_liq"][:st.vp.nlevsno] = np.where(a["h2osoi_ice"][:st.vp.nlevsno] > 0.0,
                                               rng.uniform(0.0, 3.0, (st.vp.nlevsno, nc)), 0.0)
    a["excess_ice"][:5] = np.where(some(0.2), rng.uniform(0.0, 30.0, (5, nc)), 0.0)
    a["mask_nolakec"][some(0.04)] = 0
    a["mask_hydrology"][some(0.04)] = 0
    a["col_snl"][some(0.02)] = -(st.vp.nlevsno + 1)
    a["col_patchf"][some(0.02)] = 2 * nc + 5
    a["eflx_snomelt_r"][:] = 3.0
    return st


def _limit():
    h = api.Handle(synth.clm5_varpar())
    sms = h.get_option(abi.OPT_NUM_SMS)
    h.close()
    return sms


# per SM: up to 12 columns one per warp, then 2, then 4, and beyond 40 in blocks of 32
COUNTS = [lambda n: 1, lambda n: 5, lambda n: 12 * n, lambda n: 12 * n + 1, lambda n: 24 * n + 3, lambda n: 40 * n,
          lambda n: 40 * n + 1, lambda n: 40 * n + 290]


@pytest.mark.parametrize("count", range(len(COUNTS)))
@pytest.mark.parametrize("snow", [abi.SNOW_JORDAN1991, abi.SNOW_STURM1997])
def test_soil_temperature_forms(count, snow):
    nc = COUNTS[count](_limit())
    st = _varied(nc, 31 + count)
    ref = st.copy()
    h = api.Handle(st.vp)
    d = st.to_device()
    status = torch.full((nc,), 99, dtype=torch.int32, device="cuda")
    s_ref = np.zeros(nc, dtype=np.uint32)
    for _ in range(2):
        api.soil_temperature(h, d, 1800.0, snow, col_status=status)
        s_ref = O.soil_temperature(ref, 1800.0, snow)
    got = d.to_host()
    dev = h.device_status()
    h.close()
    s = status.cpu().numpy().astype(np.uint32)
    assert np.array_equal(s, s_ref)
    assert dev == np.bitwise_or.reduce(s_ref, initial=0)
    # a column whose patch range is invalid stops there: the kernels have written its fact
    # by then, the oracle has not
    stopped = (s_ref & abi.COL_PATCH_RANGE) != 0
    got["fact"][:, stopped] = ref["fact"][:, stopped]
    mism = bit_mismatches(got, ref, ST_OUT)
    assert not mism, mism


@pytest.mark.parametrize("count", [1, 4, 7])
def test_column_step_forms_and_substep_log(count):
    """The step's first half (saved temperatures, fractions) and its logged form leave the
    same state as the separate calls."""
    nc = COUNTS[count](_limit())
    st = _varied(nc, 77 + count)
    st["col_patchf"][:] = np.arange(1, nc + 1) * 2
    cfg = abi.SwmConfig.clm5_default()
    ref = st.copy()
    O.soil_temperature(ref, 1800.0)
    O.soil_water_fractions(ref)
    fields = ST_OUT + ["eff_porosity", "icefrac", "t_ssbef"]
    m = st["mask_nolakec"] == 1
    for logged in (False, True):
        h = api.Handle(st.vp)
        h.reserve(nc)
        d = st.to_device()
        if logged:
            api.column_step_logged(h, d, 1800.0, api.SubstepLog(nc, 8), cfg)
        else:
            api.column_step(h, d, 1800.0, cfg)
        got = d.to_host()
        h.close()
        j0 = st.vp.nlevsno
        ref["t_ssbef"][:] = np.where(m, st["t_soisno"], 0.0)
        got["h2osoi_liq"][j0:j0 + st.vp.nlevsoi] = ref["h2osoi_liq"][j0:j0 + st.vp.nlevsoi]   # the water solve's
        mism = bit_mismatches(got, ref, fields)
        assert not mism, (logged, mism)


@pytest.mark.parametrize("per_sm", [0, 10, 80, 160])
@pytest.mark.parametrize("more", [1, 3])
def test_packed_richards_columns_per_warp(per_sm, more):
    """Up to 10 columns per SM run one per warp, more share warps, up to 16 each; above
    160 per SM the queue refills them."""
    nc = per_sm * _limit() + more
    wl = synth.make_workload(2, nc=nc, seed=9 + per_sm, nsteps=1)
    st = wl.state
    st["col_nbedrock"][:] = np.random.default_rng(per_sm).integers(1, st.vp.nlevsoi + 1, nc)
    O.soil_water_fractions(st)
    cfg = abi.SwmConfig.clm5_default()
    cfg.lower_boundary_condition = abi.BC_FLUX
    ref = st.copy()
    O.soil_water(ref, wl.dtime, cfg)
    h = api.Handle(st.vp)
    h.reserve(nc)
    d = st.to_device()
    api.soil_water(h, d, wl.dtime, cfg)
    got = d.to_host()
    assert h.device_status() == 0
    h.close()
    mism = bit_mismatches(got, ref, ["h2osoi_liq", "qcharge", "num_substeps", "smp_l", "hk_l"])
    assert not mism, mism
