"""GPU tests of the perceptron's one-launch passes at the edges of their tiles, against
the per-layer entry points and the numpy reference (tests/mlp_reference.py)."""
import ctypes as C

import numpy as np
import pytest

import mlp_reference as R
from clmgb import abi, api, mlp, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def h():
    assert torch.cuda.is_available()
    hd = api.Handle(synth.clm5_varpar())
    yield hd
    hd.close()


def _p(t):
    return C.c_void_p(t.data_ptr())


def _new(M, n, dtype):
    return torch.empty((M, n), dtype=dtype, device="cuda")


def _layers(h, net, X, st):
    """The forward pass layer by layer."""
    M, lib = X.shape[0], h.lib
    Z1, Z2, H1, H2 = (_new(M, 128, t) for t in (torch.float32, torch.float32, torch.bfloat16, torch.bfloat16))
    Y = _new(M, 32, torch.float32)
    for o, i, x, l, act, z, y in ((128, 64, X, 0, 1, Z1, H1), (128, 128, H1, 1, 1, Z2, H2), (32, 128, H2, 2, 0, Y, None)):
        api.check(lib.clmgb_mlp_linear(h.h, M, o, i, _p(x), i, _p(net.wb[l]), _p(net.b[l]), act, _p(z), o,
                                       None if y is None else _p(y), o, st))
    return Y, (X, Z1, H1, Z2, H2)


def _signals(h, net, acts, dY, st):
    """The backward signals dZ2, dZ1 layer by layer."""
    (X, Z1, H1, Z2, H2), M, lib = acts, dY.shape[0], h.lib
    out, up, n = [], dY, 32
    for l, z in ((2, Z2), (1, Z1)):
        dh, dz = _new(M, 128, torch.bfloat16), _new(M, 128, torch.bfloat16)
        api.check(lib.clmgb_mlp_linear(h.h, M, 128, n, _p(up), n, _p(net.wt[l]), None, 0, None, 128, _p(dh), 128, st))
        api.check(lib.clmgb_mlp_silu_backward(h.h, M * 128, _p(z), _p(dh), _p(dz), st))
        out.append(dz)
        up, n = dz, 128
    return out


@pytest.mark.parametrize("M", [1, 15, 16, 17, 31, 33, 63, 64, 65, 1000, 4097, 20011])
def test_passes_match_the_layers(h, M):
    g = torch.Generator(device="cuda").manual_seed(M)
    net = mlp.WarmStartMLP(h, seed=M)
    for b in net.b:
        b.copy_(torch.randn(b.shape, generator=g, device="cuda") * 0.1)
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    X = torch.randn((M, 64), generator=g, device="cuda").to(torch.bfloat16)
    T = torch.zeros((M, 32), device="cuda")
    T[:, :R.OUT] = torch.randn((M, R.OUT), generator=g, device="cuda")
    Yl, al = _layers(h, net, X, st)
    Y, acts = net.forward(X, keep=True)
    # the same products in the same order with the same rounding points: the same bits
    assert torch.equal(Y, Yl) and torch.equal(net.forward(X), Yl)
    assert all(torch.equal(a, b) for a, b in zip(acts, al))
    # loss: fp32 sums of at most 4 + 5 + 8 + M/32 terms; its gradient rounds once to bf16
    loss, dY = net.loss(Y, T)
    Lr, dYr = R.loss_and_dy(Y.double().cpu().numpy(), T.double().cpu().numpy())
    assert abs(float(loss) - Lr) <= (32 + M / 32) * 2.0 ** -23 * Lr
    assert np.all(np.abs(dY.double().cpu().numpy() - dYr) <= 2.0 ** -7 * np.abs(dYr))
    # gradients: sums in another order, each off by at most one rounding (or truncation)
    # per addition of the terms' magnitudes
    dW, db = net.gradients(acts, dY)
    dZ2, dZ1 = _signals(h, net, al, dY, st)
    tol = (128 + M / 32) * 2.0 ** -22
    for i, (dz, x) in enumerate(((dZ1, X), (dZ2, al[2]), (dY, al[4]))):
        d, x = dz.double(), x.double()
        assert bool(((dW[i].double() - d.T @ x).abs() <= tol * (d.abs().T @ x.abs())).all()), i
        assert bool(((db[i].double() - d.sum(0)).abs() <= tol * d.abs().sum(0)).all()), i
    # the optimiser on all parameters against the per-array entry: the same expressions
    ref = [[t.clone() for t in ts] for ts in (net.w, net.b, net.mw, net.vw, net.mb, net.vb, net.wb, net.wt)]
    net.adam(dW, db, lr=2e-3)
    w, b, mw, vw, mb, vb, wb, wt = ref
    for i, (o, n) in enumerate(mlp.LAYERS):
        api.check(h.lib.clmgb_mlp_adam(h.h, o, n, _p(w[i]), _p(dW[i]), _p(mw[i]), _p(vw[i]), 2e-3, 0.9, 0.999, 1e-8, 1,
                                       _p(wb[i]), _p(wt[i]), st))
        api.check(h.lib.clmgb_mlp_adam(h.h, 1, o, _p(b[i]), _p(db[i]), _p(mb[i]), _p(vb[i]), 2e-3, 0.9, 0.999, 1e-8, 1,
                                       None, None, st))
    for ts, rs in zip((net.w, net.b, net.mw, net.vw, net.mb, net.vb, net.wb, net.wt), ref):
        assert all(torch.equal(a, b) for a, b in zip(ts, rs))


def test_misaligned_rows_give_the_same(h):
    net = mlp.WarmStartMLP(h, seed=2)
    X = torch.randn((100, 64), device="cuda").to(torch.bfloat16)
    odd = torch.empty(100 * 64 + 1, dtype=torch.bfloat16, device="cuda")[1:].view(100, 64)
    odd.copy_(X)
    assert torch.equal(net.forward(odd), net.forward(X))
    n = abi.MlpNet(C.sizeof(abi.MlpNet), *(mlp._P3(*(t.data_ptr() for t in ts)) for ts in (
        net.w, net.b, net.wb, net.wt, net.mw, net.vw, net.mb, net.vb)))
    Y = torch.empty((100, 32), device="cuda")
    e = h.lib.clmgb_mlp_forward(h.h, 100, _p(odd), C.byref(n), None, None, None, None, _p(Y), None)
    assert e == -4                                     # CLMGB_ERR_UNSUPPORTED


@pytest.mark.parametrize("nc", [1, 31, 32, 33, 1000])
@pytest.mark.parametrize("offset", [0, 1])
def test_features_are_those_of_the_recorded_samples(h, nc, offset):
    """The features of the columns with a solve are the ones the solver records at its first
    substep start (in any order); the other columns' rows are the normalised zeros."""
    wl = synth.make_workload(2, nc=nc, seed=nc, nsteps=1)
    st = wl.state.to_device()
    hh = api.Handle(wl.state.vp)
    api.set_soil_water_fractions(hh, st)
    if nc > 1:
        st["mask_hydrology"][nc // 2] = 0
    net = mlp.WarmStartMLP(hh, seed=0)
    X = torch.empty(nc * 64 + offset, dtype=torch.bfloat16, device="cuda")[offset:].view(nc, 64)
    net.features(st, wl.dtime, out=X)
    F, T = _new(nc, 64, torch.float32), _new(nc, 32, torch.float32)
    cnt = torch.zeros(1, dtype=torch.int32, device="cuda")
    live = st["mask_hydrology"][:nc].bool()
    api.check(hh.lib.clmgb_mlp_samples(hh.h, C.byref(st.bounds()), C.byref(st.soilwater_fields()),
                                       C.byref(abi.SwmConfig.clm5_default()), float(wl.dtime), 1, _p(F), _p(T), _p(cnt),
                                       nc, None, None))
    n = int(cnt.item())
    assert n == int(live.sum())
    key = lambda t: sorted(map(tuple, t.float().cpu().numpy().tolist()))  # noqa: E731
    assert key(X[live]) == key(F[:n].to(torch.bfloat16))
    assert not bool(X[~live].any())
    hh.close()
