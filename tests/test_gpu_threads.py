"""Two host threads, each with its own handle, stream and arrays, call the same entry point
with sizes that need different amounts of shared memory: no call is refused.  (The limit of
a kernel's dynamic shared memory belongs to the function, so a call that set it to its own
need could lower it between the other thread's setting and its launch.)"""
import ctypes as C
import threading

import numpy as np
import pytest

from clmgb import abi, api, synth, zd09

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

CALLS = 8000


def _soil_temperature(nc, stream):
    wl = synth.make_workload(1, nc=nc, seed=nc, nsteps=1)
    d, h = wl.state.to_device(), api.Handle(wl.state.vp)
    f, b = d.soiltemp_fields(), d.bounds()
    keep = (d, h, f, b)
    return keep, lambda: h.lib.clmgb_soil_temperature(h.h, C.byref(b), C.byref(f), wl.dtime, abi.SNOW_JORDAN1991, 0,
                                                      None, C.c_void_p(stream.cuda_stream))


def _zengdecker(nc, stream):
    wl = synth.make_workload(1, nc=nc, seed=nc, nsteps=1)
    z = zd09.Zd09State.from_column_state(wl.state, zwt=np.full(nc, 3.0)).to_device()
    h, cfg = api.Handle(wl.state.vp), zd09.zd09_config()
    f, b = z.fields(), z.bounds()
    keep = (z, h, cfg, f, b)
    return keep, lambda: h.lib.clmgb_soil_water_zd09(h.h, C.byref(b), C.byref(f), C.byref(cfg), wl.dtime,
                                                     C.c_void_p(stream.cuda_stream))


def _tridiagonal(levels, stream):
    h, nc = api.Handle(synth.clm5_varpar()), 300
    g = torch.Generator(device="cuda").manual_seed(levels)
    u, a, b, c, r = (torch.rand((levels, nc), generator=g, dtype=torch.float64, device="cuda") for _ in range(5))
    b += 3.0
    jtop, mask = torch.ones(nc, dtype=torch.int64, device="cuda"), torch.ones(nc, dtype=torch.uint8, device="cuda")
    keep = (h, u, a, b, c, r, jtop, mask)
    p = [C.c_void_p(t.data_ptr()) for t in keep[1:]]
    return keep, lambda: h.lib.clmgb_tridiagonal_multi(h.h, nc, nc, levels, *p, C.c_void_p(stream.cuda_stream))


def _soil_water(levels, stream):
    vp = abi.Varpar(12, 25, levels, 5, 25, 0)
    wl = synth.make_workload(0, nc=61, seed=levels, vp=vp, nsteps=1)
    d, h, cfg = wl.state.to_device(), api.Handle(vp), abi.SwmConfig.clm5_default()
    h.reserve(61)
    f, b = d.soilwater_fields(), d.bounds()
    keep = (d, h, cfg, f, b)
    return keep, lambda: h.lib.clmgb_soil_water(h.h, C.byref(b), C.byref(f), C.byref(cfg), wl.dtime, None,
                                                C.c_void_p(stream.cuda_stream))


@pytest.mark.parametrize("make,small,large", [(_soil_temperature, 61, 4500), (_zengdecker, 61, 5000),
                                              (_tridiagonal, 4, 60), (_soil_water, 10, 25)])
def test_calls_of_two_threads_are_not_refused(make, small, large):
    streams = [torch.cuda.Stream(), torch.cuda.Stream()]
    kept = [make(size, s) for size, s in zip((small, large), streams)]
    torch.cuda.synchronize()
    refused = [0, 0]

    def go(i):
        for k in range(CALLS):
            refused[i] += kept[i][1]() != 0
            if k % 64 == 63:
                streams[i].synchronize()

    threads = [threading.Thread(target=go, args=(i,)) for i in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert refused == [0, 0]
