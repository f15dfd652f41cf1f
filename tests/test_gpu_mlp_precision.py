"""GPU test of the precision of the perceptron's weight and bias gradients: FP32 sums rounded
to nearest over the 128 rows of a block, one atomic addition a block, as in the per-layer
entry points.  Up to one block's rows the bits are theirs.  Over many blocks, where the
order of the atomic additions is open, the error of the hidden layers' weights against
64-bit sums, over the sum of magnitudes so that each of their 8,192 and 16,384 numbers counts
alike, has a root mean square no larger than theirs but for that order (10 %).  The outputs'
weights and the biases, too few for such a mean, are within the rounding of each addition:
2^-24 of the sum so far, which is below the sum of magnitudes."""
import ctypes as C

import pytest

from clmgb import api, mlp, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def _p(t):
    return C.c_void_p(t.data_ptr())


def _both(h, M):
    """Backward signals and layer inputs, the gradients of the layers and of the one launch."""
    st = C.c_void_p(torch.cuda.current_stream().cuda_stream)
    g = torch.Generator(device="cuda").manual_seed(M)
    net = mlp.WarmStartMLP(h, seed=M)
    X = torch.randn((M, 64), generator=g, device="cuda").to(torch.bfloat16)
    T = torch.zeros((M, 32), device="cuda")
    T[:, :21] = torch.randn((M, 21), generator=g, device="cuda")
    y, acts = net.forward(X, keep=True)
    _, dY = net.loss(y, T)
    _, Z1, H1, Z2, H2 = acts
    sig, up, n = [dY], dY, 32
    for l, z in ((2, Z2), (1, Z1)):
        dh, dz = (torch.empty((M, 128), dtype=torch.bfloat16, device="cuda") for _ in range(2))
        api.check(h.lib.clmgb_mlp_linear(h.h, M, 128, n, _p(up), n, _p(net.wt[l]), None, 0, None, 128, _p(dh), 128, st))
        api.check(h.lib.clmgb_mlp_silu_backward(h.h, M * 128, _p(z), _p(dh), _p(dz), st))
        sig.append(dz)
        up, n = dz, 128
    dW, db = net.gradients(acts, dY)
    out = []
    for i, (dz, x) in enumerate(zip(reversed(sig), (X, H1, H2))):
        w, b = torch.zeros_like(dW[i]), torch.zeros_like(db[i])
        api.check(h.lib.clmgb_mlp_linear_dw(h.h, M, *w.shape, _p(dz), w.shape[0], _p(x), w.shape[1], _p(w), _p(b), st))
        out.append((dz.double(), x.double(), (w, b), (dW[i], db[i])))
    return out


@pytest.mark.parametrize("M", [1, 16, 17, 64, 65, 127, 128])
def test_gradients_of_one_block_are_the_layers_bits(M):
    h = api.Handle(synth.clm5_varpar())
    for dz, x, layer, fused in _both(h, M):
        assert torch.equal(layer[0], fused[0]) and torch.equal(layer[1], fused[1])
    h.close()


@pytest.mark.parametrize("M", [1000, 4096, 9000, 16384, 65537])
def test_error_of_the_gradients_is_no_larger_than_the_layers(M):
    h = api.Handle(synth.clm5_varpar())
    adds = 128 + (M + 127) // 128
    for i, (dz, x, layer, fused) in enumerate(_both(h, M)):
        w, b, size = dz.T @ x, dz.sum(0), dz.abs().T @ x.abs()
        if i < 2:
            rms = [((g[0].double() - w) / size.clamp_min(1e-300)).square().mean().sqrt().item() for g in (layer, fused)]
            assert rms[1] <= 1.1 * rms[0]
        assert bool(((fused[0].double() - w).abs() <= 1.01 * adds * 2.0 ** -24 * size).all())
        assert bool(((fused[1].double() - b).abs() <= 1.01 * adds * 2.0 ** -24 * dz.abs().sum(0)).all())
    h.close()
