"""Zeng-Decker inputs on a grid whose soil levels are all its ground levels, with water tables
below the soil column.  The temperature array is the front of a longer one, whose next
row a solve must not look at.  TEST INFRASTRUCTURE."""
import numpy as np

from clmgb import abi, synth, zd09

BEHIND = (200.0, 300.0)          # what lies behind the last level: frozen, thawed


def make(behind, nc=200, levels=25):
    vp = abi.Varpar(12, levels, levels, 5, levels, 0)
    wl = synth.make_workload(1, nc=nc, seed=6, vp=vp, nsteps=1)
    st = wl.state
    bottom = st["zi"][vp.nlevsno + levels]
    st["t_soisno"][vp.nlevsno + levels - 1, ::2] = 268.0
    zs = zd09.Zd09State.from_column_state(st, zwt=bottom + np.linspace(-2.0, 6.0, nc))
    t = np.full((zs["t_soisno"].shape[0] + 1, nc), behind)
    t[:-1] = zs["t_soisno"]
    zs["t_soisno"] = t[:-1]
    return wl, zs, t
