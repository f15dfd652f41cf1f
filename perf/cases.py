"""The work a host model has this library do, as timed cases.

A land model calls the column solve every timestep for every column it holds, so most
cases are whole column steps through the drop-in calls, from a single-site ensemble of a
few columns (where launches and the longest chain of substeps count) to the quarter of a
million columns of the scale workload.  The others are the calls such a program makes
beside them: a host-resident step, the calibration gradient, the reference's default
Zeng-Decker water solve, the stand-alone banded and tridiagonal solvers, and the training
step and inference of the warm-start network.

Column states come from clmgb.synth (the workloads' distributions); solver systems and
training pairs are drawn here.  A step case advances its state on every pass, as a model
does, with the workload's forcing of the next hour or half hour (24 steps, repeated).
"""
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "clm.jl_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

from clmgb import abi, adjoint, api, hoststep, mlp, synth, zd09  # noqa: E402

FORCING_STEPS = 24
LOWER = {"zero_flux": abi.BC_ZERO_FLUX, "free_drainage": abi.BC_FLUX, "water_table": abi.BC_WATERTABLE}
SNOW = {"jordan": abi.SNOW_JORDAN1991, "sturm": abi.SNOW_STURM1997}


def listed():
    return [
        # one site: an ensemble of 61 columns with snow and frozen soil; latency of the step's launches
        {"name": "step_site_61", "kind": "step", "cfg": 1, "nc": 61, "lower": "zero_flux", "snow": "jordan",
         "bedrock": False, "one_call": False},
        # a regional run without snow: the 1,024 columns of the plain workload
        {"name": "step_plain_1024", "kind": "step", "cfg": 0, "nc": 1024, "lower": "zero_flux", "snow": "jordan",
         "bedrock": False, "one_call": False},
        # a ragged domain: an odd column count, bedrock at any depth, a water table, the other snow scheme
        {"name": "step_ragged_10007", "kind": "step", "cfg": 1, "nc": 10007, "lower": "water_table", "snow": "sturm",
         "bedrock": True, "one_call": False},
        # the snow and frozen-soil workload, free drainage, through the one-call step
        {"name": "step_snow_65536", "kind": "step", "cfg": 1, "nc": 65536, "lower": "free_drainage", "snow": "jordan",
         "bedrock": False, "one_call": True},
        # the scale workload: diurnal forcing, infiltration pulses, hourly steps
        {"name": "step_scale_262144", "kind": "step", "cfg": 2, "nc": 262144, "lower": "zero_flux", "snow": "jordan",
         "bedrock": False, "one_call": False},
        # a host-resident model: the step's inputs up, the four calls, every written field back
        {"name": "host_step_50021", "kind": "host", "cfg": 2, "nc": 50021},
        # calibration: the gradient of a trajectory's loss with respect to four parameters of every level
        {"name": "gradient_16384", "kind": "gradient", "cfg": 1, "nc": 16384, "steps": 6, "every": 3},
        # the water solve of the reference's default configuration
        {"name": "zengdecker_40009", "kind": "zengdecker", "cfg": 1, "nc": 40009},
        # the reference's batched band solver on snow + surface water + soil systems
        {"name": "band_65537", "kind": "band", "nc": 65537},
        # the reference's batched tridiagonal solver on soil + aquifer systems
        {"name": "tridiagonal_100003", "kind": "tridiagonal", "nc": 100003, "levels": 21},
        # one optimiser step of the warm-start network on a minibatch
        {"name": "train_4096", "kind": "train", "batch": 4096},
        # the network's proposals for every column: features and forward pass
        {"name": "propose_131072", "kind": "propose", "cfg": 2, "nc": 131072},
    ]


def _between(rng, lo, hi):
    """A whole number spread over the logarithm of lo..hi."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["host", "gradient", "zengdecker", "band", "tridiagonal", "train", "propose"])
    if kind == "step":
        return {"kind": kind, "cfg": rng.choice([0, 1, 1, 2, 2]), "nc": _between(rng, 40, 262144),
                "lower": rng.choice(["zero_flux", "zero_flux", "free_drainage", "water_table"]),
                "snow": rng.choice(["jordan", "jordan", "sturm"]), "bedrock": rng.random() < 0.3,
                "one_call": rng.random() < 0.4}
    if kind == "host":
        return {"kind": kind, "cfg": rng.choice([1, 2]), "nc": _between(rng, 1000, 50021)}
    if kind == "gradient":
        return {"kind": kind, "cfg": 1, "nc": _between(rng, 300, 16384), "steps": rng.randint(2, 6),
                "every": rng.randint(1, 4)}
    if kind == "zengdecker":
        return {"kind": kind, "cfg": rng.choice([0, 1]), "nc": _between(rng, 500, 40009)}
    if kind == "band":
        return {"kind": kind, "nc": _between(rng, 500, 65537)}
    if kind == "tridiagonal":
        return {"kind": kind, "nc": _between(rng, 500, 100003), "levels": rng.randint(10, 50)}
    if kind == "train":
        return {"kind": kind, "batch": _between(rng, 250, 16384)}
    return {"kind": kind, "cfg": rng.choice([1, 2]), "nc": _between(rng, 1000, 131072)}


# ---------------------------------------------------------------- preparation
def _workload(case, seed, steps=FORCING_STEPS):
    return synth.make_workload(case["cfg"], nc=case["nc"], seed=7919 * int(seed) + 11, nsteps=steps)


def _handle(vp, nc):
    h = api.Handle(vp)
    h.reserve(nc)
    return h


def _forcing(wl, steps):
    G, I = wl.forcing_block(range(steps))
    return torch.from_numpy(G).cuda(), torch.from_numpy(I).cuda()


class _Step:
    """A device-resident model: its state, forcing, handle and configuration."""

    def __init__(self, case, seed):
        wl = _workload(case, seed)
        rng = np.random.default_rng(int(seed) + 5)
        st = wl.state
        if case["bedrock"]:
            st["col_nbedrock"][:] = rng.integers(6, st.vp.nlevsoi + 1, st.nc)
        if case["lower"] == "water_table":
            st["zwt"][:] = rng.uniform(0.5, 12.0, st.nc)
        self.dtime, self.snow, self.one_call = wl.dtime, SNOW[case["snow"]], case["one_call"]
        self.cfg = abi.SwmConfig.clm5_default()
        self.cfg.lower_boundary_condition = LOWER[case["lower"]]
        self.G, self.I = _forcing(wl, FORCING_STEPS)
        self.state = st.to_device()
        self.h = _handle(st.vp, st.nc)
        self.t = 0

    def run(self):
        k, s = self.t % FORCING_STEPS, self.state
        self.t += 1
        api.synth_forcing(self.h, s, self.G[k], self.I[k])
        if self.one_call:
            api.column_step(self.h, s, self.dtime, self.cfg, self.snow)
        else:
            api.soil_temperature(self.h, s, self.dtime, self.snow)
            api.set_soil_water_fractions(self.h, s)
            api.soil_water(self.h, s, self.dtime, self.cfg)
        return {n: s[n] for n in hoststep.WRITTEN_TEMPERATURE + hoststep.WRITTEN_WATER}


class _Host:
    """A model whose arrays live in pinned host memory."""

    def __init__(self, case, seed):
        wl = _workload(case, seed)
        st = wl.state
        self.G, self.I = _forcing(wl, FORCING_STEPS)
        self.h = _handle(st.vp, st.nc)
        self.host = {k: torch.from_numpy(np.ascontiguousarray(v)).pin_memory() for k, v in st.arrays.items()}
        self.stepper = hoststep.HostStepper(self.h, self.host, st.to_device(), wl.dtime)
        self.t = 0

    def run(self):
        k = self.t % FORCING_STEPS
        self.t += 1
        self.stepper.step(forcing=lambda dev: api.synth_forcing(self.h, dev, self.G[k], self.I[k]))
        torch.cuda.current_stream().synchronize()      # the model goes on with the host arrays
        return {n: self.host[n] for n in hoststep.WRITTEN_TEMPERATURE + hoststep.WRITTEN_WATER}


class _Gradient:
    """A calibration: initial state, observations, trajectory."""

    def __init__(self, case, seed):
        n = case["steps"]
        wl = _workload(case, seed, n)
        cfg = abi.SwmConfig.clm5_default()
        cfg.lower_boundary_condition = abi.BC_FLUX
        self.h = _handle(wl.state.vp, case["nc"])
        self.h.reserve_adjoint(case["nc"], 256)
        self.G, self.I = _forcing(wl, n)
        self.traj = adjoint.Trajectory(self.h, n, wl.dtime, self._force, cfg,
                                       forcing_reverse=adjoint.synth_forcing_reverse)
        self.start = wl.state.to_device()
        truth = wl.state.copy()
        adjoint.perturb_parameters(truth, np.random.default_rng(int(seed) + 3))
        s = truth.to_device()
        obs = adjoint.CalibrationLoss(self.start, wl.dtime)
        for t in range(n):
            self.traj.step(t, s)
            obs.observe(t, s)
        self.target, self.every = torch.stack(obs.y), case["every"]

    def _force(self, t, s):
        api.synth_forcing(self.h, s, self.G[t], self.I[t])

    def run(self):
        s = self.start.copy()
        loss = adjoint.CalibrationLoss(s, self.traj.dtime, self.target)
        adj = adjoint.multistep_reverse(self.traj, s, loss.seed, loss.observe, checkpoint_every=self.every)
        out = {"grad_" + p: adj.grad[p] for p in adjoint.PARAMS}
        out.update(loss=loss.per_column(), lam_t_soisno=adj.lam_t_soisno, lam_h2osoi_liq=adj.lam_h2osoi_liq,
                   lam_h2osoi_ice=adj.lam_h2osoi_ice, lam_t_grnd=adj.lam_t_grnd)
        out.update({n: s[n] for n in hoststep.WRITTEN_TEMPERATURE + hoststep.WRITTEN_WATER})
        return out


class _ZengDecker:
    """The state of the reference's default water solve, water tables at every depth."""

    def __init__(self, case, seed):
        wl = _workload(case, seed, 1)
        vp = wl.state.vp
        rng = np.random.default_rng(int(seed) + 9)
        bottom = float(wl.state["zi"][vp.nlevsno + vp.nlevsoi, 0])
        zwt = np.where(rng.random(case["nc"]) < 0.7, rng.uniform(0.1, bottom, case["nc"]),
                       bottom + rng.uniform(0.3, 5.0, case["nc"]))
        self.state = zd09.Zd09State.from_column_state(wl.state, zwt=zwt).to_device()
        self.h, self.dtime = _handle(vp, case["nc"]), wl.dtime

    def run(self):
        zd09.soil_water_zd09(self.h, self.state, self.dtime)
        return {n: self.state[n] for n in ("h2osoi_liq", "h2osoi_vol", "qcharge", "smp_l", "hk_l")}


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(1000003 * int(seed) + 17)


def _uniform(g, shape, lo, hi):
    return torch.rand(shape, generator=g, dtype=torch.float64, device="cuda") * (hi - lo) + lo


class _Band:
    """Heat-conduction systems over up to 12 snow levels, the surface-water row and 25
    soil levels: diagonally dominant, with the small outer couplings of that row."""
    SNO, GRND = 12, 25

    def __init__(self, case, seed):
        nc, nlev, g = case["nc"], self.SNO + 1 + self.GRND, _gen(seed)
        self.h = api.Handle(synth.clm5_varpar())
        up, lo = _uniform(g, (nlev, nc), 0.0, 5.0), _uniform(g, (nlev, nc), 0.0, 5.0)
        b = torch.empty((nlev, 5, nc), dtype=torch.float64, device="cuda")
        b[:, 0], b[:, 1], b[:, 3], b[:, 4] = _uniform(g, (nlev, nc), -0.05, 0.05), -up, -lo, \
            _uniform(g, (nlev, nc), -0.05, 0.05)
        b[:, 2] = 1.0 + up + lo
        self.b, self.r = b, _uniform(g, (nlev, nc), 240.0, 300.0)
        self.jtop = -torch.randint(0, self.SNO + 1, (nc,), generator=g, device="cuda")
        self.jbot = torch.full((nc,), self.GRND, dtype=torch.int64, device="cuda")
        self.mask = (torch.rand(nc, generator=g, device="cuda") < 0.98).to(torch.uint8)
        self.x = torch.zeros((nlev, nc), dtype=torch.float64, device="cuda")

    def run(self):
        api.batched_band_solve(self.h, self.x, self.b, self.r, self.jtop, self.jbot, self.mask, kl=2, ku=2,
                               nlevsno_off=self.SNO)
        return {"x": self.x}

    def exact(self):
        nlev, _, nc = self.b.shape
        row = torch.arange(nlev, device="cuda")
        top = self.jtop + self.SNO                      # first row of the system, from 0
        x = torch.zeros((nlev, nc), dtype=torch.float64, device="cuda")
        for c0 in range(0, nc, 8192):
            c = slice(c0, min(nc, c0 + 8192))
            live = row[:, None] >= top[None, c]
            a = torch.zeros((live.shape[1], nlev, nlev), dtype=torch.float64, device="cuda")
            for band in range(5):                       # band = row - column + 2
                for i in range(nlev):
                    j = i - (band - 2)
                    if 0 <= j < nlev:
                        a[:, i, j] = torch.where(live[i] & live[j], self.b[i, band, c],
                                                 torch.zeros_like(self.b[i, band, c]))
            a += torch.diag_embed((~live).T.to(torch.float64))
            r = torch.where(live, self.r[:, c], torch.zeros_like(self.r[:, c]))
            x[:, c] = torch.linalg.solve(a, r.T.unsqueeze(-1)).squeeze(-1).T * self.mask[c].to(torch.float64)
        return {"x": x}


class _Tridiagonal:
    """Soil-water systems, some of which start below the first level."""

    def __init__(self, case, seed):
        nc, n, g = case["nc"], case["levels"], _gen(seed)
        self.h = api.Handle(synth.clm5_varpar())
        self.a, self.c = -_uniform(g, (n, nc), 0.0, 2.0), -_uniform(g, (n, nc), 0.0, 2.0)
        self.b, self.r = 1.0 - self.a - self.c, _uniform(g, (n, nc), -1.0, 1.0)
        self.jtop = torch.where(torch.rand(nc, generator=g, device="cuda") < 0.8, 1,
                                torch.randint(1, 4, (nc,), generator=g, device="cuda"))
        self.mask = (torch.rand(nc, generator=g, device="cuda") < 0.98).to(torch.uint8)
        self.u = torch.zeros((n, nc), dtype=torch.float64, device="cuda")

    def run(self):
        api.tridiagonal_multi(self.h, self.u, self.a, self.b, self.c, self.r, self.jtop, self.mask)
        return {"u": self.u}

    def exact(self):
        n = self.u.shape[0]
        live = (torch.arange(1, n + 1, device="cuda")[:, None] >= self.jtop[None]) & (self.mask[None] > 0)
        zero = torch.zeros_like(self.a)
        first = torch.arange(1, n + 1, device="cuda")[:, None] == self.jtop[None]
        a = torch.where(live & ~first, self.a, zero)
        b, c, r = torch.where(live, self.b, zero + 1.0), torch.where(live, self.c, zero), torch.where(live, self.r, zero)
        b, r = b.clone(), r.clone()
        for i in range(1, n):
            w = a[i] / b[i - 1]
            b[i] -= w * c[i - 1]
            r[i] -= w * r[i - 1]
        u = zero.clone()
        u[n - 1] = r[n - 1] / b[n - 1]
        for i in range(n - 2, -1, -1):
            u[i] = (r[i] - c[i] * u[i + 1]) / b[i]
        return {"u": torch.where(live, u, zero)}


def _silu(z):
    return z / (1.0 + torch.exp(-z))


class _Train:
    """A network in training and its current minibatch."""
    LR = 2.0e-3

    def __init__(self, case, seed):
        g, m = _gen(seed), case["batch"]
        self.h = api.Handle(synth.clm5_varpar())
        self.net = mlp.WarmStartMLP(self.h, seed=int(seed))
        self.x = torch.randn((m, mlp.IN), generator=g, device="cuda").to(torch.bfloat16)
        self.y = torch.zeros((m, mlp.OUTP), device="cuda")
        self.y[:, 0] = torch.randint(0, 7, (m,), generator=g, device="cuda").to(torch.float32)
        self.y[:, 1:mlp.OUT] = torch.randn((m, mlp.OUT - 1), generator=g, device="cuda")

    def run(self):
        net = self.net
        y, acts = net.forward(self.x, keep=True)
        loss, dy = net.loss(y, self.y)
        dw, db = net.gradients(acts, dy)
        net.adam(dw, db, lr=self.LR)
        return {"y": y, "loss": loss, "dw": dw, "db": db, "w": list(net.w), "b": list(net.b)}

    def exact(self):
        w, b = [v.double() for v in self.net.wb], [v.double() for v in self.net.b]
        x, t, m = self.x.double(), self.y.double(), self.x.shape[0]
        z1 = x @ w[0].T + b[0]
        h1 = _silu(z1)
        z2 = h1 @ w[1].T + b[1]
        h2 = _silu(z2)
        y = h2 @ w[2].T + b[2]
        k = torch.zeros(mlp.OUTP, dtype=torch.float64, device="cuda")
        k[0], k[1:mlp.OUT] = 1.0, 1.0 / (mlp.OUT - 1)
        loss = (k * (y - t) ** 2).sum().reshape(1) / m

        def slope(z):
            s = torch.sigmoid(z)
            return s * (1.0 + z * (1.0 - s))
        d3 = 2.0 * k * (y - t) / m
        d2 = (d3 @ w[2]) * slope(z2)
        d1 = (d2 @ w[1]) * slope(z1)
        dw, db = [d1.T @ x, d2.T @ h1, d3.T @ h2], [d1.sum(0), d2.sum(0), d3.sum(0)]

        def adam(p, q):                                 # the first step: both moments start at zero
            return p.double() - self.LR * q / (q.abs() + 1.0e-8)
        return {"y": y, "loss": loss, "dw": dw, "db": db, "w": [adam(p, q) for p, q in zip(self.net.w, dw)],
                "b": [adam(p, q) for p, q in zip(self.net.b, db)]}


class _Propose:
    """A trained network's normalisation and a state at the start of the water solve."""

    def __init__(self, case, seed):
        wl = _workload(case, seed, 1)
        self.h = _handle(wl.state.vp, case["nc"])
        self.dtime, self.state = wl.dtime, wl.state.to_device()
        api.set_soil_water_fractions(self.h, self.state)
        self.net = mlp.WarmStartMLP(self.h, seed=int(seed))
        raw = self._raw()
        sd = raw.std(0)
        self.net.mean = raw.mean(0).float().contiguous()
        self.net.istd = torch.where(sd > 1e-6, 1.0 / sd, torch.ones_like(sd)).float().contiguous()

    def _raw(self):
        """The network's inputs (clmgb_mlp_features' definition) in 64 bits."""
        s, v = self.state, self.state.vp
        n, j0, e_ice = v.nlevsoi, v.nlevsno, abi.SwmConfig.clm5_default().e_ice
        sat = s["h2osoi_liq"][j0:j0 + n] / (1000.0 * s["dz"][j0:j0 + n] * s["watsat"][:n])
        ice = s["icefrac"][:n]
        below = torch.cat([sat[1:], sat[-1:]])
        mid = torch.clamp(0.5 * (sat + below), 0.01, 1.0)
        mid_ice = 0.5 * (ice + torch.cat([ice[1:], ice[-1:]]))
        cond = torch.log10(s["hksat"][:n]) + (2.0 * s["bsw"][:n] + 3.0) * torch.log10(mid) - e_ice * mid_ice
        one = torch.ones_like(s["qflx_infl"])
        tail = torch.stack([s["qflx_infl"] * 1.0e3, s["qflx_rootsoi"][:n].sum(0) * 1.0e3, one,
                            one * (math.log2(self.dtime / 60.0) / 6.0)])
        return torch.cat([sat, ice, cond, tail]).T

    def run(self):
        x = self.net.features(self.state, self.dtime)
        return {"x": x, "y": self.net.forward(x)}

    def exact(self):
        x = (self._raw() - self.net.mean.double()) * self.net.istd.double()
        w, b = [v.double() for v in self.net.wb], [v.double() for v in self.net.b]
        h = _silu(_silu(x @ w[0].T + b[0]) @ w[1].T + b[1])
        return {"x": x, "y": h @ w[2].T + b[2]}


KINDS = {"step": _Step, "host": _Host, "gradient": _Gradient, "zengdecker": _ZengDecker, "band": _Band,
         "tridiagonal": _Tridiagonal, "train": _Train, "propose": _Propose}


def prepare(case, seed):
    return KINDS[case["kind"]](case, seed)


def run(state):
    return state.run()


def exact(case, seed):
    """64-bit values where the outputs are a closed form of the inputs.  The column steps,
    their gradient and the Zeng-Decker solve are long 64-bit programs whose melt, freeze
    and substep decisions depend on the last bits: a second 64-bit restatement has no
    better claim to be exact than the first."""
    cls = KINDS[case["kind"]]
    return cls(case, seed).exact() if hasattr(cls, "exact") else None


def work(case):
    """Bytes: every field a pass reads or writes once (8-byte words, active levels only;
    the mean number of snow levels of the workload).  Operations: additions,
    multiplications, divisions and powers of the reference's expressions, each as one, with
    the workloads' usual four substep attempts and three accepted substeps a column."""
    kind = case["kind"]
    if kind in ("step", "host", "gradient"):
        snow = {0: 0.0, 1: 6.0, 2: 2.6}[case["cfg"]]
        words = 21 * 25 + 6 * 20 + 55 + 16 * snow
        ops = 130 * (25 + snow) + 20 * (4 * 18 + 3 * 39)
        if kind == "gradient":
            # forward, then per step its reverse: state and adjoints in and out, about three forwards' operations
            return {"bytes": 8 * case["nc"] * (words + case["steps"] * (2 * words + 4 * 45 + 160)),
                    "flops": 4 * case["nc"] * case["steps"] * ops}
        return {"bytes": 8 * case["nc"] * words, "flops": case["nc"] * ops}
    if kind == "zengdecker":
        return {"bytes": 8 * case["nc"] * (20 * 15 + 12), "flops": case["nc"] * 20 * 90}
    if kind == "band":
        return {"bytes": 8 * case["nc"] * 32 * 7, "flops": case["nc"] * 32 * 32}
    if kind == "tridiagonal":
        return {"bytes": 8 * case["nc"] * case["levels"] * 5, "flops": case["nc"] * case["levels"] * 9}
    layers = mlp.IN * mlp.HID + mlp.HID * mlp.HID + mlp.HID * mlp.OUT
    if kind == "train":
        return {"bytes": case["batch"] * (2 * mlp.IN + 8 * mlp.OUTP) + 28 * layers, "flops": 6 * case["batch"] * layers}
    return {"bytes": case["nc"] * (8 * 7 * 20 + 2 * mlp.IN + 4 * mlp.OUTP), "flops": 2 * case["nc"] * layers}
