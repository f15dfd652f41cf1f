"""GPU test: the Zeng-Decker solve on a grid whose soil levels are all its ground levels reads
no temperature behind the last one, in both of its forms, and gives the oracle's bits."""
import numpy as np
import pytest

import zd09_last_level as Z
from clmgb import abi, api, zd09
from oracle import oracle as O

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("behind", Z.BEHIND)
@pytest.mark.parametrize("nc", [200, 9000])
def test_no_temperature_behind_the_last_level_is_read(behind, nc):
    wl, zs, t = Z.make(behind, nc)
    h = api.Handle(zs.vp)
    d = zs.to_device()
    rows = torch.from_numpy(t).cuda()
    d["t_soisno"] = rows[:-1]
    zd09.soil_water_zd09(h, d, wl.dtime)
    out = d.to_host()
    h.close()
    ref = Z.make(Z.BEHIND[1], nc)[1]
    O.soil_water_zd09(ref, wl.dtime)
    for (n, _, _, _) in abi.ZD09_FIELDS:
        assert np.array_equal(out[n], ref[n], equal_nan=True), n
