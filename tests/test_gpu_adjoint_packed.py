"""GPU test of the solve's reverse with a thread per level (logged columns) against the one
on a thread per column (no log): the same functions of a level in the same order, so the
same bits, at the edges of a block's 16 columns, over ragged bedrock, inactive columns, all
lower boundaries, odd level counts and columns whose solve the log does not hold."""
import numpy as np
import pytest

from clmgb import abi, adjoint, api, synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# what the reverse leaves of the forward step with a log (without one it replays the whole step)
STATE = ("t_soisno", "h2osoi_liq", "h2osoi_ice", "fact", "t_grnd", "t_h2osfc", "icefrac", "eff_porosity", "qcharge",
         "num_substeps", "smp_l", "hk_l", "t_ssbef", "t_h2osfc_bef")


@pytest.mark.parametrize("nc", [1, 15, 16, 17, 100])
@pytest.mark.parametrize("lower", [abi.BC_FLUX, abi.BC_ZERO_FLUX, abi.BC_WATERTABLE])
@pytest.mark.parametrize("cap,reserve,nlevsoi", [(24, True, 20), (2, False, 20), (24, False, 7), (24, True, 25)])
def test_reverse_per_level_gives_the_bits_of_the_reverse_per_column(nc, lower, cap, reserve, nlevsoi):
    cfg = abi.SwmConfig.clm5_default()
    cfg.lower_boundary_condition = lower
    rng = np.random.default_rng(nc + 7 * lower)
    vp = synth.clm5_varpar()
    vp.nlevsoi = nlevsoi
    wl = synth.make_workload(1, nc=nc, seed=nc, nsteps=3, vp=vp)
    st = wl.state
    st["col_nbedrock"][:] = rng.integers(1, st.vp.nlevsoi + 1, nc)
    st["zwt"][:] = rng.uniform(0.3, 12.0, nc)
    if nc > 4:
        st["col_nbedrock"][1] = 0
        st["mask_hydrology"][2] = 0
        st["mask_nolakec"][3] = 0
    h = api.Handle(st.vp)
    h.reserve_adjoint(nc, 256)
    if reserve:
        h.reserve(nc)
    a = st.to_device()
    G, I = (torch.from_numpy(x).cuda() for x in wl.forcing_block(range(3)))
    log = api.SubstepLog(nc, cap)
    for t in range(3):
        api.synth_forcing(h, a, G[t], I[t])
        b, f = a.copy(), a.copy()
        api.column_step_logged(h, f, wl.dtime, log, cfg)
        out = []
        for s, lg in ((b, None), (a, log)):
            adj = adjoint.StepAdjointBuffers(s)
            g = torch.Generator(device="cuda").manual_seed(nc + t)
            for x in vars(adj).values():
                for y in (x.values() if isinstance(x, dict) else [x]):
                    if torch.is_tensor(y):
                        y.copy_(torch.randn(y.shape, generator=g, device="cuda", dtype=y.dtype))
            status = torch.zeros(nc, dtype=torch.int32, device="cuda")
            if lg is None:
                api.column_step_vjp(h, s, wl.dtime, adj, cfg, col_status=status)
            else:
                api.column_step_vjp(h, s, wl.dtime, adj, cfg, col_status=status, log=lg)
            out.append([status] + [y for x in vars(adj).values() for y in (x.values() if isinstance(x, dict) else [x])
                                   if torch.is_tensor(y)] + [s[k] for k in STATE])
        assert len(out[0]) > 10
        for i, (x, y) in enumerate(zip(*out)):
            assert torch.equal(x.view(torch.uint8), y.view(torch.uint8)), (t, i)
    h.close()
