"""GPU test of the Richards work order (a counting sort by the previous substep count, in one
block or in two kernels): every listed column is solved once, whatever the counts, at the
edges of the two forms.  The solve without reserved scratch lists no order: the same bits."""
import numpy as np
import pytest

from clmgb import abi, api, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nc", [1, 33, 1023, 1025, 4095, 4096, 4097, 6000])
@pytest.mark.parametrize("counts", ["one", "any"])
def test_ordered_solve_is_the_unordered_one(nc, counts):
    wl = synth.make_workload(2, nc=nc, seed=nc, nsteps=1)
    st, rng = wl.state, np.random.default_rng(nc)
    st["icefrac"][:] = np.where(rng.random(st["icefrac"].shape) < 0.5, 0.0, rng.random(st["icefrac"].shape))
    st["num_substeps"][:] = 2.0 if counts == "one" else rng.choice([np.nan, -1.0, 0.0, 0.5, 1.0, 7.0, 62.0, 63.0, 1e9],
                                                                   nc)
    if nc > 1:
        st["mask_hydrology"][rng.random(nc) < 0.2] = 0
    cfg = abi.SwmConfig.clm5_default()
    out = []
    for reserve in (False, True):
        h, s = api.Handle(st.vp), st.to_device()
        if reserve:
            h.reserve(nc)
        status = torch.full((nc,), 7, dtype=torch.int32, device="cuda")
        api.soil_water(h, s, wl.dtime, cfg, col_status=status)
        out.append([status] + [s[k] for k in ("h2osoi_liq", "smp_l", "hk_l", "qcharge", "num_substeps")])
        torch.cuda.synchronize()
        h.close()
    for x, y in zip(*out):
        assert torch.equal(x.view(torch.uint8), y.view(torch.uint8))
