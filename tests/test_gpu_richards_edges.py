"""GPU test of the packed Richards solve at the column counts where it takes another form or a
warp another number of columns, per SM: up to 10 columns one a warp, up to 80 eight a warp
and an attempt's quotients and powers in line (ten warps), beyond 18 warps of eight, which
the queue refills above 144; with 25 levels one block of nine warps fits an SM, refilled
above 72.  The bits are the oracle's for every lower boundary."""
import numpy as np
import pytest

from clmgb import abi, api, synth
from oracle import oracle as O
from parity import bit_mismatches

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

OUT = ["h2osoi_liq", "qcharge", "num_substeps", "smp_l", "hk_l"]
ALL = [abi.BC_ZERO_FLUX, abi.BC_FLUX, abi.BC_WATERTABLE]
CASES = ([(20, 1, n, m, abi.BC_FLUX) for n in (10, 144) for m in (0, 1)] +
         [(20, 1, 80, m, bc) for m in (0, 1) for bc in ALL] +
         [(20, 42, n, 1, abi.BC_ZERO_FLUX) for n in (10, 80)] +
         [(25, 1, n, m, abi.BC_WATERTABLE) for n in (72, 80) for m in (0, 1)])


@pytest.mark.parametrize("levels,flux,per_sm,more,bc", CASES)
def test_bits_at_the_edges_of_the_forms(levels, flux, per_sm, more, bc):
    vp = abi.Varpar(12, 25, levels, 5, 25, 0)
    h = api.Handle(vp)
    nc = per_sm * h.get_option(abi.OPT_NUM_SMS) + more
    wl = synth.make_workload(2, nc=nc, seed=per_sm + levels, nsteps=1, vp=vp)
    st = wl.state
    rng = np.random.default_rng(nc)
    st["col_nbedrock"][:] = rng.integers(1, levels + 1, nc)
    st["zwt"][:] = rng.uniform(0.3, 20.0, nc)
    O.soil_water_fractions(st)
    cfg = abi.SwmConfig.clm5_default()
    cfg.lower_boundary_condition, cfg.flux_calculation = bc, flux
    ref = st.copy()
    O.soil_water(ref, wl.dtime, cfg)
    h.reserve(nc)
    d = st.to_device()
    api.soil_water(h, d, wl.dtime, cfg)
    got = d.to_host()
    assert h.device_status() == 0
    h.close()
    mism = bit_mismatches(got, ref, OUT)
    assert not mism, mism
