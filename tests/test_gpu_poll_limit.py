"""CLMGB_OPT_QUEUE_POLL_LIMIT bounds a wait of the per-lane Richards kernel.  By itself it
leaves the solve to the packed kernel: the same bits, the same counted work."""
import pytest

from clmgb import abi, api, synth
from parity import bit_mismatches

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("polls", [0, 1000])
def test_poll_limit_alone_leaves_the_solve_to_the_packed_kernel(polls):
    wl = synth.make_workload(2, nc=2000, seed=3, nsteps=1)
    runs = []
    for limit in (None, polls):
        h = api.Handle(wl.state.vp)
        h.reserve(wl.state.nc)
        if limit is not None:
            h.set_option(abi.OPT_QUEUE_POLL_LIMIT, limit)
            assert h.get_option(abi.OPT_QUEUE_POLL_LIMIT) == limit
        h.set_option(abi.OPT_COUNT_WORK, 1)
        d = wl.state.to_device()
        api.set_soil_water_fractions(h, d)
        api.soil_water(h, d, wl.dtime)
        work = (h.get_option(abi.OPT_WORK_LEVEL_ATTEMPTS), h.get_option(abi.OPT_WORK_LEVEL_REFRESHES))
        runs.append((work, d.to_host()))
        assert h.device_status() == 0
        h.close()
    assert runs[0][0][0] > 0 and runs[1][0] == runs[0][0]
    assert not bit_mismatches(runs[1][1], runs[0][1], ["h2osoi_liq", "qcharge", "num_substeps", "smp_l", "hk_l"])
