"""GPU test of the step's reverse at levels whose saturation is clamped at 1 from an infinite
value (no pore space): the derivative of the clamp is zero there, so the gradient is finite
and the one of a pore space too small to matter.  A relative pore space of 1e-12 moves the
conductivity's derivative in watsat, dke dksat log(mixture), by a relative 1e-12."""
import numpy as np
import pytest

from clmgb import adjoint, api, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("logged", [False, True])
def test_gradient_of_a_level_without_pore_space(logged):
    wl = synth.make_workload(0, nc=40, seed=4, nsteps=1)
    st = wl.state
    st["mask_hydrology"][:] = 0                       # soil_temperature! alone
    levels = np.arange(st.nc) % st.vp.nlevsoi
    G, I = (torch.from_numpy(x).cuda() for x in wl.forcing_block(range(1)))
    grads = []
    for ws in (0.0, 1.0e-12):
        st["watsat"][levels, np.arange(st.nc)] = ws
        h = api.Handle(st.vp)
        h.reserve(st.nc)
        h.reserve_adjoint(st.nc, 256)
        a = st.to_device()
        api.synth_forcing(h, a, G[0], I[0])
        log = api.SubstepLog(st.nc, 8) if logged else None
        if logged:
            api.column_step_logged(h, a.copy(), wl.dtime, log)
        adj = adjoint.StepAdjointBuffers(a)
        adj.zero_()
        g = torch.Generator(device="cuda").manual_seed(1)
        adj.lam_t_soisno.copy_(torch.randn(adj.lam_t_soisno.shape, generator=g, device="cuda", dtype=torch.float64))
        api.column_step_vjp(h, a, wl.dtime, adj, log=log)
        assert h.device_status() == 0
        grads.append([adj.grad["watsat"].cpu().numpy(), adj.lam_h2osoi_liq.cpu().numpy(),
                      adj.lam_t_soisno.cpu().numpy()])
        h.close()
    for x, y in zip(*grads):
        assert np.all(np.isfinite(x)) and np.any(y != 0.0)
        np.testing.assert_allclose(x, y, rtol=1e-9, atol=1e-12 * np.abs(y).max())
