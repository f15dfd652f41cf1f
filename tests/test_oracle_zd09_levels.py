"""CPU check: the oracle's Zeng-Decker solve reads no temperature behind the last level."""
import numpy as np

import zd09_last_level as Z
from clmgb import abi
from oracle import oracle as O


def test_no_temperature_behind_the_last_level_is_read():
    out = []
    for behind in Z.BEHIND:
        wl, zs, _ = Z.make(behind)
        O.soil_water_zd09(zs, wl.dtime)
        out.append(zs)
    for (n, _, _, _) in abi.ZD09_FIELDS:
        assert np.array_equal(out[0][n], out[1][n], equal_nan=True), n
