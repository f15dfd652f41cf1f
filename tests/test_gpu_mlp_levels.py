"""GPU test of the warm-start features on soil grids with more levels than the features hold
(20): the conductivity of level 20 is that of its interface with level 21 where the column
goes on below.  Against a numpy restatement in binary64; the kernels form it in binary32:
some ten operations with a relative error of 2^-24 on terms up to 100, and the features
kernel rounds to bfloat16 (2^-9)."""
import ctypes as C

import numpy as np
import pytest

from clmgb import abi, api, mlp, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _log_conductivity(st, e_ice):
    """Feature 40 + j - 1 of levels 1..20, [20, nc]; the columns reach to col_nbedrock."""
    joff, n = st.vp.nlevsno, st["col_nbedrock"]
    s = st["h2osoi_liq"][joff:joff + st.vp.nlevsoi] / (1000.0 * st["dz"][joff:joff + st.vp.nlevsoi] *
                                                       st["watsat"][:st.vp.nlevsoi])
    out = np.full((20, st.nc), -30.0)
    for j in range(1, min(20, st.vp.nlevsoi) + 1):
        lowest = n == j
        k = min(j, st.vp.nlevsoi - 1)
        s1 = np.where(lowest, s[j - 1], 0.5 * (s[j - 1] + s[k]))
        ice = np.where(lowest, st["icefrac"][j - 1], 0.5 * (st["icefrac"][j - 1] + st["icefrac"][k]))
        v = (np.log10(st["hksat"][j - 1]) + (2.0 * st["bsw"][j - 1] + 3.0) * np.log10(np.clip(s1, 0.01, 1.0)) -
             e_ice * ice)
        out[j - 1] = np.where(j <= n, v, -30.0)
    return out


@pytest.mark.parametrize("nlevsoi", [19, 20, 21, 25])
def test_conductivity_of_the_lowest_feature_level(nlevsoi):
    vp = abi.Varpar(12, 25, nlevsoi, 5, 25, 0)
    nc = 300
    wl = synth.make_workload(1, nc=nc, seed=nlevsoi, vp=vp, nsteps=1)
    wl.state["col_nbedrock"][:] = np.random.default_rng(nlevsoi).integers(18, nlevsoi + 1, nc)
    h = api.Handle(vp)
    st = wl.state.to_device()
    api.set_soil_water_fractions(h, st)
    ref = _log_conductivity(st.to_host(), abi.SwmConfig.clm5_default().e_ice)
    net = mlp.WarmStartMLP(h, seed=0)
    X = net.features(st, wl.dtime)[:, 40:60].float().cpu().numpy().T
    F = torch.empty((nc, 64), device="cuda")
    T, cnt = torch.empty((nc, 32), device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    api.check(h.lib.clmgb_mlp_samples(h.h, C.byref(st.bounds()), C.byref(st.soilwater_fields()),
                                      C.byref(abi.SwmConfig.clm5_default()), float(wl.dtime), 1, C.c_void_p(F.data_ptr()),
                                      C.c_void_p(T.data_ptr()), C.c_void_p(cnt.data_ptr()), nc, None, None))
    assert int(cnt.item()) == nc
    h.close()
    np.testing.assert_allclose(X, ref, rtol=2.0 ** -8, atol=1e-4)
    F = F[:, 40:60].cpu().numpy().T
    np.testing.assert_allclose(np.sort(F, axis=1), np.sort(ref, axis=1), rtol=1e-5, atol=1e-4)
