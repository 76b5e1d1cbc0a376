"""The work that a program built on this framework has it do, as measured cases.

Each case is one short piece of a run: a flow in motion (never a state at rest,
which takes fewer of the solver's branches) is put into the stepper, the clock is
set, and a few steps are taken, so that every pass does the same work. The kinds:

  steps      a device-resident patch, `solver.PatchStepper`, stepped eagerly or by
             replaying a captured graph; 5 fields, or all 7 with segregation and
             entrainment
  host       `PatchStepper.step_host`: the state stays in (pinned) host memory
  patch      `patch.Patch`: the step2-style calls a Fortran driver makes in turn
  rollout    `solver.rollout_peak` / `rollout`: the differentiable port's calls,
             which set up a stepper and pick the time step themselves
  ensemble   `ensemble.EnsembleStepper`: flumes of uneven sizes with their own
             parameters and time steps
  gradient   `adjoint.rollout_states` and its backward pass, gauge loss
  ensemble_gradient   the same over an ensemble of channels

Everything is float64, the only type the framework takes.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from dclaw_b200.adjoint import ensemble_rollout_states, rollout_states, theta_of
from dclaw_b200.ensemble import EnsembleStepper, Member
from dclaw_b200.params import DClawParams
from dclaw_b200.patch import Patch
from dclaw_b200.solver import Grid, PatchStepper, rollout, rollout_peak

GHOST = 2            # ghost cells on each side of a patch-call array
CFL = 0.4


# ---- cases ------------------------------------------------------------------
def _case(name, kind, mx, my, steps, **options):
    case = {"name": name, "kind": kind, "mx": mx, "my": my, "steps": steps, "dx": 1.0, "tilt": 20.0,
            "wet": 0.3, "sources": 32, "order": 2, "limiter": 4, "src2method": 0, "manning": 0.0,
            "walls": True, "graph": False, "peak": True, "members": 0}
    case.update(options)
    return case


def listed():
    return [
        # a small patch of a level, or a quick look: the launches and the latency of one step count
        _case("patch_64", "steps", 64, 64, 10, tilt=30.0, sources=2, wet=0.2),
        # the 200 x 200 slope with runout, run as a production loop runs it: a replayed graph
        _case("slope_200_graph", "steps", 200, 200, 10, tilt=30.0, sources=1, wet=0.12, graph=True),
        # a mid-size ragged patch with open boundaries and Manning friction
        _case("ragged_1000x731_manning", "steps", 1000, 731, 4, manning=0.03, walls=False),
        # the benchmark's field: one large patch
        _case("field_4096", "steps", 4096, 4096, 2, dx=0.5),
        # the explicit quadrant-wise integration of the source terms, first order, other limiter
        _case("quadrants_777x1024", "steps", 1024, 777, 2, src2method=2, limiter=1),
        # the whole state: segregation and entrainment
        _case("full_state_1024", "steps_full", 1024, 1024, 2),
        # a driver that keeps its state in host memory between steps
        _case("host_2048", "host", 2048, 2048, 1, dx=0.5),
        # a driver that calls the patch routines one by one (stepgrid's loop)
        _case("patch_calls_500x300", "patch", 500, 300, 2),
        # the port's call: set-up, time-step choice, running peak, read-back
        _case("rollout_peak_333x200", "rollout", 333, 200, 30, sources=4),
        # particles of a filter: flumes of uneven sizes and parameters
        _case("flumes_24", "ensemble", 4096, 128, 4, dx=0.05, members=24, tilt=31.0),
        # calibration: the gradient of a gauge misfit through a run
        _case("gradient_512", "gradient", 512, 512, 12),
        # the particles' gradients
        _case("channel_gradient_8", "ensemble_gradient", 1024, 256, 6, dx=0.05, members=8, tilt=31.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["steps", "steps", "steps", "steps_full", "host", "patch", "rollout", "ensemble", "gradient",
                       "gradient", "ensemble_gradient"])
    top = {"steps": 4096, "steps_full": 1500, "host": 2048, "patch": 1024, "rollout": 800, "gradient": 512}
    o = {"dx": rng.choice([0.5, 1.0, 2.0]), "tilt": rng.uniform(10.0, 32.0), "wet": rng.uniform(0.1, 0.5),
         "walls": rng.random() < 0.7}
    if kind.startswith("ensemble"):
        members = _log_int(rng, 2, 24 if kind == "ensemble" else 8)
        o.update(dx=0.05, tilt=rng.uniform(25.0, 33.0), members=members, walls=True)
        mx, my = (4096, 128) if kind == "ensemble" else (1024, 256)
        mx = _log_int(rng, 512, mx)
        steps = 2 * rng.randint(1, 2) if kind == "ensemble" else rng.randint(2, 6)
        o["graph"] = kind == "ensemble" and rng.random() < 0.5
    else:
        mx, my = (_log_int(rng, 40, top[kind]) for _ in range(2))
        o["sources"] = rng.randint(1, 32)
        cells = mx * my
        if kind in ("steps", "steps_full"):
            steps = 10 if cells < 200_000 else 4 if cells < 3_000_000 else 2
            o["graph"] = rng.random() < 0.4
            if kind == "steps":
                o["src2method"] = rng.choice([0, 0, 0, 1, 2, -1])
                o["order"] = rng.choice([2, 2, 2, 1])
                o["limiter"] = rng.choice([4, 4, 4, 1, 2, 3, 0])
                o["manning"] = rng.choice([0.0, 0.0, 0.03])
        elif kind == "host":
            steps = 1
        elif kind == "patch":
            steps = 2
        elif kind == "rollout":
            steps = rng.randint(10, 30)
            o["peak"] = rng.random() < 0.6
        else:
            steps = rng.randint(2, 12)
            o["manning"] = rng.choice([0.0, 0.0, 0.03])
    case = _case("", kind, mx, my, steps, **o)
    del case["name"]
    return case


# ---- inputs -------------------------------------------------------------------
def _noise(gen, my, mx, slope=-3.0):
    """A Gaussian random field with power spectrum k^slope, unit variance."""
    white = torch.randn(my, mx, generator=gen, device="cuda", dtype=torch.float64)
    kx = torch.fft.rfftfreq(mx, device="cuda", dtype=torch.float64)
    ky = torch.fft.fftfreq(my, device="cuda", dtype=torch.float64)
    k2 = kx[None, :] ** 2 + ky[:, None] ** 2
    k2[0, 0] = math.inf
    f = torch.fft.irfft2(torch.fft.rfft2(white) * k2 ** (slope / 4.0), s=(my, mx))
    f = f - f.mean()
    return f / f.std()


def _flow(case, gen, params):
    """(q (5, my, mx), b (my, mx), first dt): paraboloid masses with velocities of
    metres a second, mostly down the tilt, on rough terrain, about `wet` of it covered."""
    mx, my, dx = case["mx"], case["my"], case["dx"]
    x = (torch.arange(mx, device="cuda", dtype=torch.float64) + 0.5) * dx
    y = (torch.arange(my, device="cuda", dtype=torch.float64) + 0.5) * dx
    b = math.tan(math.radians(case["tilt"])) * (mx * dx - x)[None, :] + _noise(gen, my, mx) * min(5.0, 0.02 * mx * dx)
    n = case["sources"]
    draws = torch.rand(n, 8, generator=gen, device="cuda", dtype=torch.float64).tolist()
    radius = math.sqrt(case["wet"] * mx * my * dx * dx / (n * math.pi))
    h = torch.zeros_like(b)
    hm, hu, hv, pb = (torch.zeros_like(b) for _ in range(4))
    for r in draws:
        cx, cy = (0.08 + 0.84 * r[0]) * mx * dx, (0.08 + 0.84 * r[1]) * my * dx
        reach = radius * (0.85 + 0.3 * r[2])
        hk = ((0.5 + 2.5 * r[3]) * (1.0 - ((x - cx)[None, :] ** 2 + (y - cy)[:, None] ** 2) / reach**2)).clamp_min(0.0)
        h += hk
        hm += hk * (0.55 + 0.09 * r[4])
        hu += hk * (6.0 * r[5])
        hv += hk * (3.0 * (r[6] - 0.5))
        pb += hk * (0.4 + 0.6 * r[7])
    swing = 1.0 + 0.2 * _noise(gen, my, mx, -2.0).clamp(-2.0, 2.0)
    q = torch.stack([h, hu * swing, hv * swing, hm, params.rho_f * params.grav * pb])
    q *= (h > params.dry_tolerance)
    return q, b, _first_dt(q, dx, params)


def _first_dt(q, dx, params):
    h = q[0].clamp_min(1.0e-12)
    speed = torch.where(q[0] > 0.0, torch.maximum(q[1].abs(), q[2].abs()) / h + (params.grav * h).sqrt(), 0.0 * h)
    return CFL * dx / max(float(speed.max()), 1.0)


def _params(case, **more):
    side = "wall" if case["walls"] else "extrap"
    return DClawParams(bc_lower=(side, side), bc_upper=(side, side), order=case["order"], limiter=case["limiter"],
                       transverse_waves=case["order"] if case["order"] == 2 else 0, src2method=case["src2method"],
                       alphamethod=1 if case["src2method"] == 2 else 0, friction_forcing=case["manning"] > 0.0,
                       manning_coefficient=case["manning"], cfl_desired=CFL, **more)


def _members(case, seed):
    """Channels of uneven sizes with parameters from the priors (phi U[28, 40] deg,
    log10 kref U[-11, -8], m0 U[0.55, 0.65], alpha U[0.005, 0.05]); each holds a
    release that is somewhere between its block and a thin sheet along the channel."""
    rng, sizes = np.random.default_rng(seed), np.random.default_rng([case["mx"], case["my"], case["members"]])
    out = []
    for _ in range(case["members"]):
        w = int(sizes.integers(max(16, case["my"] // 4), case["my"] + 1))
        n = int(sizes.integers(max(128, case["mx"] // 4), case["mx"] + 1)) if case["kind"] == "ensemble" else case["mx"]
        p = DClawParams(phi=float(rng.uniform(28.0, 40.0)), kref=float(10.0 ** rng.uniform(-11.0, -8.0)),
                        m0=float(rng.uniform(0.55, 0.65)), alpha_c=float(rng.uniform(0.005, 0.05)), cfl_desired=CFL)
        dx = case["dx"]
        x, y = (np.arange(n) + 0.5) * dx, (np.arange(w) + 0.5) / w
        b = np.broadcast_to(math.tan(math.radians(case["tilt"])) * np.maximum(0.75 * n * dx - x, 0.0), (w, n))
        length = min(3.0 * float(np.exp(rng.uniform(0.0, 2.5))), 0.6 * n * dx)
        depth = 3.0 / length
        front = 0.5 + length
        profile = np.where(x >= 0.5, np.clip(1.0 - ((x - 0.5) / length) ** 2, 0.0, None), 0.0)
        h = depth * profile[None, :] * (1.0 + 0.1 * np.sin(9.0 * y[:, None] + 40.0 * x[None, :] / front))
        h = np.where(h > 2.0e-3, h, 0.0)
        u = rng.uniform(1.0, 4.0) * (0.3 + 0.7 * x / front)[None, :]
        v = 0.3 * rng.uniform(-1.0, 1.0) * np.cos(7.0 * y)[:, None]
        q = np.stack([h, h * u, h * v, h * p.m0, rng.uniform(0.4, 1.0) * p.rho_f * p.grav * h])
        speed = np.where(h > 0.0, np.maximum(np.abs(u), np.abs(v)) + np.sqrt(p.grav * h), 0.0).max()
        out.append(Member(q, np.ascontiguousarray(b), p, dx, dx, CFL * dx / float(speed)))
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    kind = case["kind"]
    s = {"case": case}
    if kind.startswith("ensemble"):
        s["members"] = _members(case, seed)
        st = EnsembleStepper(s["members"])
        s["q"] = st.qa.clone()
        if kind == "ensemble":
            s["stepper"], s["clocks"] = st, st.clocks.clone()
            if case["graph"]:
                st.step(2)
                st.capture(case["steps"])
        else:
            s["theta"] = torch.stack([theta_of(m.params, "cuda") for m in s["members"]])
            s["gauges"] = torch.cat([
                st.cm[k].q_off + (int(st.my[k]) // 2) * int(st.mx[k])
                + torch.linspace(20, 0.5 * float(st.mx[k]), 16, device="cuda").to(torch.int64)
                for k in range(st.n)])
            s["target"] = 0.1 * torch.rand(case["steps"], s["gauges"].numel(), generator=gen, device="cuda",
                                           dtype=torch.float64)
        return s
    full = kind == "steps_full"
    p = _params(case, **(dict(segregation=1, beta_seg=0.3, entrainment=1, entrainment_method=0) if full else {}))
    if kind == "gradient":
        p = p.replace(speed_limit=30.0)
    q, b, dt = _flow(case, gen, p)
    dx = case["dx"]
    s.update(q=q, b=b, dt=dt, params=p)
    if full:
        s["q"] = torch.cat([q, p.chi0 * q[:1], torch.zeros_like(q[:1])])
        erodible = 0.5 * torch.ones_like(b)
        s["stepper"] = PatchStepper(s["q"], b, p, dx, dx, h_e=erodible)
    elif kind in ("steps", "host"):
        s["stepper"] = PatchStepper(q, b, p, dx, dx)
    if kind in ("steps", "steps_full") and case["graph"]:
        s["stepper"].init_clock(dt)
        s["stepper"].step(2)
        s["stepper"].capture(case["steps"])
    elif kind == "host":
        s["q_host"], s["out"] = q.cpu().pin_memory(), torch.empty(q.shape, dtype=torch.float64).pin_memory()
        del s["q"]
    elif kind == "patch":
        s["patch"] = Patch(p, case["mx"], case["my"])
        s["q_pad"], s["aux"] = (torch.zeros(nf, case["my"] + 2 * GHOST, case["mx"] + 2 * GHOST, device="cuda",
                                            dtype=torch.float64) for nf in (5, 6))
        s["aux"][0, GHOST:-GHOST, GHOST:-GHOST] = b
    elif kind == "rollout":
        s["q_nx"], s["b_nx"] = q.permute(0, 2, 1).contiguous(), b.t().contiguous()
    elif kind == "gradient":
        s["theta"] = theta_of(p, "cuda")
        wet = torch.nonzero(q[0].reshape(-1) > 0.0).reshape(-1)
        s["gauges"] = wet[torch.randint(wet.numel(), (64,), generator=gen, device="cuda")]
        s["target"] = torch.rand(case["steps"], 64, generator=gen, device="cuda", dtype=torch.float64)
    return s


# ---- one pass -------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind, n, dx = case["kind"], case["steps"], case["dx"]
    if kind in ("steps", "steps_full"):
        st = s["stepper"]
        st.qa.copy_(s["q"])
        st.init_clock(s["dt"])
        if case["graph"]:
            st.replay()
        else:
            st.step(n)
        return {"q": st.state(), "clock": st.clock[:4]}
    if kind == "host":
        st = s["stepper"]
        st.init_clock(s["dt"])
        st.step_host(s["q_host"], s["out"])
        clock = st.read_clock()          # the driver's next time step; the state is back when it is
        return {"q": s["out"], "dt": clock.dt, "cfl": clock.cfl}
    if kind == "patch":
        pt, q, aux = s["patch"], s["q_pad"], s["aux"]
        q[:, GHOST:-GHOST, GHOST:-GHOST].copy_(s["q"])
        t, dt = 0.0, s["dt"]
        for _ in range(n):
            pt.bc2amr(q)
            pt.setaux(aux)
            pt.b4step2(q, aux, dx, dx, t, dt)
            cfl = pt.step2(q, aux, dx, dx, dt)
            pt.src2(q, aux, dx, dx, t, dt)
            t += dt
        return {"q": q, "aux": aux, "cfl": cfl}
    if kind == "rollout":
        grid = Grid(case["mx"], case["my"], dx, dx)
        side = "wall" if case["walls"] else "open"
        call = rollout_peak if case["peak"] else rollout
        q, t, kept, *_ = call(s["q_nx"], s["b_nx"], s["params"], grid, 1.0e3, CFL, side, side, n_steps=n)
        return {"q": q, "t": t, "kept": kept}
    if kind == "ensemble":
        st = s["stepper"]
        st.qa.copy_(s["q"])
        st.clocks.copy_(s["clocks"])
        if case["graph"]:
            st.replay()
        else:
            st.step(n)
        return {"q": st.qa, "clocks": st.clocks.view(st.n, -1)[:, :4]}
    q0, theta = s["q"].detach().requires_grad_(), s["theta"].detach().requires_grad_()
    outs = range(1, n + 1)
    if kind == "gradient":
        got = rollout_states(q0, theta, s["b"], s["params"], dx, dx, n, outs, s["dt"], select=s["gauges"])
    else:
        got = ensemble_rollout_states(q0, theta, s["members"], n, outs, select=s["gauges"])
    loss = (got - s["target"]).square().sum()
    gq, gt = torch.autograd.grad(loss, (q0, theta))
    return {"gauges": got.detach(), "loss": loss.detach(), "gq": gq, "gtheta": gt}


# ---- what one pass cannot do without -----------------------------------------------
def work(case):
    """Bytes: state in and out and the bed, for every cell and step (once more in and
    out, and the adjoint state, where a gradient is taken). Operations: about 2500 a
    covered cell and step forward (four interface solves' share, limiter, two
    transverse splits, source terms, counting a division, a root and each elementary
    function as its polynomial), three times that for the reverse of a step."""
    kind = case["kind"]
    cells = case["mx"] * case["my"]
    wet = case["wet"]
    if kind.startswith("ensemble"):
        mean = 0.625 * (0.625 if kind == "ensemble" else 1.0)
        cells, wet = int(cells * mean * case["members"]), 0.1
    fields = 7 if kind == "steps_full" else 5
    total, flops = 8.0 * cells * (2 * fields + 1) * case["steps"], 2500.0 * wet * cells * case["steps"]
    if kind.endswith("gradient"):
        return {"bytes": 3.0 * total, "flops": 4.0 * flops}
    return {"bytes": total, "flops": flops}


def exact(case, seed):
    """None throughout: the outputs are D-Claw's own float64 scheme, whose limiter and
    wet/dry branches have no more exact value than the scheme itself computes."""
    return None
