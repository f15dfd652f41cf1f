"""GPU test of the hand-over of long columns from the per-lane work-queue Richards kernel to
the warp-per-column finish (CLMGB_OPT_QUEUE_DEFER with CLMGB_OPT_QUEUE_PACKED_REFRESH 0; the
packed kernel hands nothing over).  That columns are handed over is read from the work the
finish counts (CLMGB_OPT_COUNT_WORK); the results are the oracle's bits for every lower
boundary, both flux calculations, every batch of refreshes, and the normal bounded wait."""
import numpy as np
import pytest

from clmgb import abi, api, synth
from oracle import oracle as O
from parity import bit_mismatches

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

OUT = ["h2osoi_liq", "smp_l", "hk_l", "qcharge", "num_substeps"]


def _inputs(nc, seed, bc, flux):
    wl = synth.make_workload(2, nc=nc, seed=seed, nsteps=1)
    st = wl.state
    rng = np.random.default_rng(seed)
    st["col_nbedrock"][:] = rng.integers(1, st.vp.nlevsoi + 1, nc)
    st["zwt"][:] = rng.uniform(0.3, 12.0, nc)
    O.soil_water_fractions(st)
    cfg = abi.SwmConfig.clm5_default()
    cfg.lower_boundary_condition, cfg.flux_calculation = bc, flux
    ref = st.copy()
    O.soil_water(ref, wl.dtime, cfg)
    return wl, cfg, ref


def _solve(wl, cfg, defer, batch=None):
    """(state, work counted by the finish, column status, device status)"""
    st = wl.state
    h = api.Handle(st.vp)
    h.reserve(st.nc)
    h.set_option(abi.OPT_QUEUE_PACKED_REFRESH, 0)
    h.set_option(abi.OPT_QUEUE_DEFER, defer)
    if batch is not None:
        h.set_option(abi.OPT_QUEUE_FRESH_BATCH, batch)
    h.set_option(abi.OPT_COUNT_WORK, 1)
    d = st.to_device()
    status = torch.full((st.nc,), 3, dtype=torch.int32, device="cuda")
    api.soil_water(h, d, wl.dtime, cfg, col_status=status)
    work = (h.get_option(abi.OPT_WORK_LEVEL_ATTEMPTS), h.get_option(abi.OPT_WORK_LEVEL_REFRESHES))
    out = d.to_host(), work, status.cpu().numpy(), h.device_status()
    h.close()
    return out


@pytest.mark.parametrize("bc", [abi.BC_ZERO_FLUX, abi.BC_FLUX, abi.BC_WATERTABLE])
@pytest.mark.parametrize("flux", [1, 42])
def test_handed_over_columns_keep_the_bits(bc, flux):
    wl, cfg, ref = _inputs(5000, 5, bc, flux)
    levels = wl.state["col_nbedrock"].astype(np.int64)
    for defer in (0, 2, 6):
        out, work, status, dev = _solve(wl, cfg, defer)
        # columns with more attempts than `defer` leave the queue at their next accepted one
        most = int((np.maximum(ref["num_substeps"] - defer, 0) * levels).sum()) if defer else 0
        assert (0 < work[1] <= work[0] <= most) if defer else work == (0, 0), (defer, work, most)
        assert not bit_mismatches(out, ref, OUT), defer
        assert np.all(status == 0) and dev == 0


@pytest.mark.parametrize("batch", [0, 1, 8, 32])
def test_handed_over_columns_with_any_batch_of_refreshes(batch):
    wl, cfg, ref = _inputs(3000, 8, abi.BC_FLUX, 1)
    for defer in (0, 6):
        out, work, status, dev = _solve(wl, cfg, defer, batch)
        assert (work[0] > 0) == (defer > 0)
        assert not bit_mismatches(out, ref, OUT), defer
        assert np.all(status == 0) and dev == 0


def test_normal_bounded_wait_leaves_no_trace():
    wl, cfg, ref = _inputs(16384, 12, abi.BC_ZERO_FLUX, 1)
    out, work, status, dev = _solve(wl, cfg, 4)
    assert work[0] > 0
    assert not bit_mismatches(out, ref, OUT)
    assert np.all(status == 0) and dev == 0
