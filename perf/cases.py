"""The work a user of this framework has it do, as cases that can be timed.

A case is a dict of plain values.  `prepare` makes what a program holds before
the call (a context, particles, a time stepper), `run` is one pass through the
public entry points, `exact` the same results in 64 bits from plain torch, and
`work` the bytes and operations a pass cannot do without.

Kinds:
  step      particles in (float3 x, v in lattice order), `steps` PM steps,
            particles out: a simulation, or a part of one between outputs.
            `calls`: "run_steps" (the fused loop) or "phases" (the phase
            functions one by one, as the reference's driver calls them);
            `io`: "device" (the caller's arrays are on the GPU) or "host".
  ensemble  boxes of mixed sizes loaded into slots, advanced together.
  classes   size classes advanced each at its own pace, as the serving loop does.
  pk        the power spectrum of a loaded particle state.
  ic        initial conditions from a seed and a P(k) table.
  fft       the 3D complex transform of a caller's grid.

The particles are what a run meets at its middle (a = 0.46 of a run from
z = 50): a Gaussian field with a CDM spectrum on 1 Mpc/h cells, its particles
moved through its linear potential, so that they have flowed into filaments
and clumps and crossed there.
"""
import math

import numpy as np
import torch

import hacc_gpm_b200 as H
from hacc_gpm_b200 import ensemble as E
from hacc_gpm_b200 import ipk

SIDES = (16, 24, 32, 40, 48, 64, 80, 96, 120, 128, 160, 192, 200, 240, 256, 320, 384, 400, 480, 512, 640, 768, 800,
         960, 1000, 1024)
Z_INI, N_STEPS, MID_STEP = 50.0, 100, 45  # the headline run: 100 steps from z = 50, timed at its middle


def _step(name, ng, np_side, steps, calls="run_steps", io="device"):
    return {"name": name, "kind": "step", "ng": ng, "np": np_side, "steps": steps, "calls": calls, "io": io}


def listed():
    return [
        # a parameter scan's or a test's box: launches and latency
        _step("step 32", 32, 32, 10),
        # the smallest production box (50-step runs of 64^3), driven from numpy arrays
        _step("step 64 host", 64, 64, 5, io="host"),
        # a side that is no multiple of 16, so particles in 8^3 blocks, and of radices 3, 5 and 8
        _step("step 120", 120, 120, 4),
        # phase by phase, as the reference's serial() drives the drop-in; radices 5, 5, 8
        _step("phases 200", 200, 200, 2, calls="phases"),
        # fewer particles than cells (half the side, mass 8)
        _step("step 256 of 128", 256, 128, 4),
        # the medium production box
        _step("step 256", 256, 256, 4),
        # the headline workload
        _step("step 512", 512, 512, 4),
        # the largest grid, with half as many particles per side
        _step("step 1024 of 512", 1024, 512, 2),
        # batched ensemble: the five sides of the 96-box workload
        {"name": "ensemble 32-128", "kind": "ensemble", "sides": "32,48,64,96,128", "slots": 4, "steps": 16},
        # the serving loop's classes, one side of them outside the multi-class launch
        {"name": "classes 48-192", "kind": "classes", "sides": "48,80,192", "slots": 3, "steps": 8},
        # the power spectrum with the reference's 221 linear bins
        {"name": "pk 256", "kind": "pk", "ng": 256, "np": 256, "bins": 221, "log": False, "fold": 0},
        # one transform of a caller's grid, a side of radix 5
        {"name": "fft 320", "kind": "fft", "ng": 320, "inverse": False},
    ]


def _of_log(rng, lo, hi):
    """A whole number in [lo, hi], spread over its logarithm."""
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _side(rng, lo, hi):
    """A grid side near a size spread over its logarithm."""
    at = rng.uniform(math.log(lo), math.log(hi))
    return min((s for s in SIDES if lo <= s <= hi), key=lambda s: abs(math.log(s) - at))


def draw(rng):
    kind = rng.choices(("step", "ensemble", "classes", "pk", "ic", "fft"), (12, 2, 2, 2, 1, 2))[0]
    if kind == "step":
        most = work(_step("", 1024, 512, 2))["bytes"]
        while True:
            ng = _side(rng, 16, 1024)
            np_side = rng.choice((ng, ng, ng, ng // 2, 2 * ng))
            c = _step("", ng, np_side, _of_log(rng, 1, 24), rng.choice(("run_steps", "run_steps", "phases")),
                      rng.choice(("device", "device", "host")) if ng <= 128 else "device")
            del c["name"]
            if np_side in SIDES and work(c)["bytes"] <= 0.8 * most:
                return c
    if kind == "ensemble":
        sides = sorted(rng.sample((32, 48, 64, 96, 128), rng.randint(1, 5)))
        return {"kind": kind, "sides": ",".join(map(str, sides)), "slots": rng.randint(1, 6), "steps": _of_log(rng, 2, 24)}
    if kind == "classes":
        sides = sorted(rng.sample((24, 32, 40, 48, 64, 80, 96, 120, 128, 160, 192), rng.randint(1, 3)))
        return {"kind": kind, "sides": ",".join(map(str, sides)), "slots": rng.randint(1, 4), "steps": _of_log(rng, 2, 16)}
    if kind == "pk":
        ng = _side(rng, 32, 512)
        return {"kind": kind, "ng": ng, "np": rng.choice((ng, ng, ng // 2)) if ng // 2 in SIDES else ng,
                "bins": rng.choice((32, 64, 221)), "log": rng.random() < 0.5, "fold": rng.choice((0, 0, 1, 2))}
    if kind == "ic":
        return {"kind": kind, "ng": _side(rng, 32, 512)}
    return {"kind": kind, "ng": _side(rng, 16, 512), "inverse": rng.random() < 0.5}


# ---- inputs ------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _params_text(ng, np_side, seed):
    return ipk.lcdm_params_text(ng, np_side, float(ng), Z_INI, N_STEPS, seed=seed)


def _displacement(n, seed):
    """The linear displacement field on n^3 cells of 1 Mpc/h, [3][n^3], with an rms of 2 cells an axis."""
    k1 = 2 * math.pi * torch.fft.fftfreq(n, device="cuda")
    kz = 2 * math.pi * torch.fft.rfftfreq(n, device="cuda")
    k2 = k1[:, None, None] ** 2 + k1[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    k = k2.sqrt()
    # a CDM transfer function (Bardeen et al. 1986) of shape 0.21, cut off below the cell
    q = k / 0.21
    t = torch.log1p(2.34 * q) / (2.34 * q)
    t *= (1 + 3.89 * q + (16.1 * q) ** 2 + (5.46 * q) ** 3 + (6.71 * q) ** 4) ** -0.25
    f = torch.fft.rfftn(torch.randn(n, n, n, device="cuda", generator=_generator(seed)))
    f *= k ** 0.48 * t * torch.exp(-0.5 * k2) / k2
    f[0, 0, 0] = 0
    del k2, k, q, t
    psi = torch.empty(3, n ** 3, device="cuda")
    for d, kd in enumerate((k1[:, None, None], k1[None, :, None], kz[None, None, :])):
        psi[d] = torch.fft.irfftn(1j * kd * f, s=(n, n, n)).reshape(-1)
    psi *= 2.0 / psi.square().mean().sqrt()
    return psi


def _particles(ng, np_side, seed):
    """(x, v) of np^3 particles in lattice order, float32 [np^3, 3]: x in grid units, in [0, ng), v in the run's units."""
    n = np_side
    psi = _displacement(n, seed)
    q = torch.arange(n, device="cuda", dtype=torch.float32)
    x = torch.stack([a.reshape(-1) for a in torch.meshgrid(q, q, q, indexing="ij")])
    u = psi.clone()
    x += 0.1 * u
    for s in range(9):  # du/dD = 3/(2D) (psi(x) - u): motion in the linear potential, D from 0.1 to 1
        d = 0.1 * (s + 1)
        i = torch.remainder(x.round(), n).long()
        i = (i[0] * n + i[1]) * n + i[2]
        for a in range(3):
            u[a] += 0.15 / d * (psi[a][i] - u[a])
        x += 0.1 * u
        del i
    x *= ng / np_side
    x = torch.remainder(x, ng)
    x[x >= ng] = 0.0
    a, dt, adot, _ = _epochs(ng, np_side)[0]
    # D grows by about 2 % in a step at mid-run; a step drifts by v deltaT / (a^2 adot)
    v = u * (0.02 * (ng / np_side) * a * a * adot / dt)
    return x.t().contiguous(), v.t().contiguous()


def _free():
    torch.cuda.synchronize()
    torch.cuda.empty_cache()


def _stepper(params):
    ts = H.Timestepper(params)
    ts.set_initial_z(params.z_ini)
    for _ in range(2 * MID_STEP):
        ts.advance_half_step()
    return ts


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fft":
        n = case["ng"]
        g = _generator(seed)
        grid = torch.complex(*(torch.randn(n, n, n, device="cuda", generator=g) for _ in range(2)))
        return {"case": case, "grid": grid, "out": torch.empty_like(grid)}
    if kind in ("ensemble", "classes"):
        sides = [int(s) for s in case["sides"].split(",")]
        ens = E.Ensemble([(s, s, case["slots"]) for s in sides])
        state = {"case": case, "ens": ens, "boxes": [], "x": {}, "v": {}}
        for c, side in enumerate(sides):
            state["x"][str(side)] = torch.empty(case["slots"], side ** 3, 3, device="cuda")
            state["v"][str(side)] = torch.empty(case["slots"], side ** 3, 3, device="cuda")
            for k in range(case["slots"]):
                params = H.parse_params(_params_text(side, side, seed))
                x, v = _particles(side, side, seed + 1000 * c + k)
                state["boxes"].append((c, k, params, _stepper(params), x, v, state["x"][str(side)][k], state["v"][str(side)][k]))
        _free()
        return state
    np_side = case.get("np", case["ng"])
    params = H.parse_params(_params_text(case["ng"], np_side, seed % 100000000))
    if kind == "ic":
        header, table = ipk.make_ipk(ipk.cosmo_from_params(params), Z_INI, k_max=10.0)
        state = {"case": case, "table": table, "k_delta": float(header[3])}
    else:
        x, v = _particles(case["ng"], np_side, seed)
        state = {"case": case, "x": x, "v": v, "ts": _stepper(params)}
    _free()
    state["sim"] = H.Simulation(params)
    if kind == "pk":
        state["sim"].load_state_device(x.data_ptr(), v.data_ptr())
        state["sim"].sync()
    elif case.get("io") == "host":
        state["x"], state["v"] = x.cpu().numpy(), v.cpu().numpy()
    else:
        state["xo"] = torch.empty(np_side ** 3, 3, device="cuda")
        state["vo"] = torch.empty(np_side ** 3, 3, device="cuda")
    return state


# ---- one pass ------------------------------------------------------------------
def _run_step(state):
    case, sim, ts = state["case"], state["sim"], state["ts"].copy()
    host = case["io"] == "host"
    if host:
        sim.load_state(state["x"], state["v"])
    else:
        sim.load_state_device(state["x"].data_ptr(), state["v"].data_ptr())
    if case["calls"] == "run_steps":
        sim.run_steps(ts, case["steps"])
    else:
        for _ in range(case["steps"]):
            sim.update_positions(ts)
            sim.cic()
            sim.solve_gradient()
            ts.advance_half_step()
            sim.update_velocities(ts)
            ts.advance_half_step()
            sim.update_positions(ts)
    if host:
        x, v = sim.store_state()
        return {"x": x, "v": v}
    sim.store_state_device(state["xo"].data_ptr(), state["vo"].data_ptr())
    return {"x": state["xo"], "v": state["vo"]}


def _run_boxes(state):
    case, ens = state["case"], state["ens"]
    for c, k, params, ts, x, v, _, _ in state["boxes"]:
        ens.slot(c, k, params).load_state_device(x.data_ptr(), v.data_ptr())
        ens.start(c, k, ts.copy(), case["steps"])
    if case["kind"] == "ensemble":
        ens.step(case["steps"])
        ens.sync()
    else:
        for c in range(len(ens.classes)):
            ens.step_class(c, case["steps"])
        for c in range(len(ens.classes)):
            ens.sync_class(c)
    for c, k, _, _, _, _, x, v in state["boxes"]:
        ens.views[(c, k)].store_state_device(x.data_ptr(), v.data_ptr())
        ens.release(c, k)
    return {"x": state["x"], "v": state["v"]}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "step":
        return _run_step(state)
    if kind in ("ensemble", "classes"):
        return _run_boxes(state)
    if kind == "pk":
        k, p, n = state["sim"].power_spectrum(case["bins"], case["log"], case["fold"])
        return {"k": k, "p": p, "n": n}
    if kind == "ic":
        state["sim"].generate_ic(state["table"], state["k_delta"])
        state["sim"].store_state_device(state["xo"].data_ptr(), state["vo"].data_ptr())
        return {"x": state["xo"], "v": state["vo"]}
    state["out"].copy_(state["grid"])
    H.binding.fft_c2c(state["out"].data_ptr(), case["ng"], case["inverse"], torch.cuda.current_stream().cuda_stream)
    return state["out"]


# ---- the same in 64 bits -----------------------------------------------------
def _epochs(ng, np_side, steps=1):
    """(a, deltaT, adot, fscal) at the start of the pass and after each half step (timestepper.cpp:13-68)."""
    text = dict(line.split(None, 1) for line in _params_text(ng, np_side, 0).splitlines() if " " in line)
    p = {k: float(np.float32(float(text[k]))) for k in ("OMEGA_CDM", "DEUT", "HUBBLE", "T_CMB", "N_EFF_MASSLESS")}
    cb = p["OMEGA_CDM"] + p["DEUT"] / p["HUBBLE"] ** 2
    rad = 2.471e-5 * (p["T_CMB"] / 2.725) ** 4 / p["HUBBLE"] ** 2
    rad *= 1 + p["N_EFF_MASSLESS"] * 7 / 8 * (4 / 11) ** (4 / 3)
    dt = (1.0 - 1.0 / (Z_INI + 1.0)) / N_STEPS
    a, out = 1.0 / (Z_INI + 1.0) + MID_STEP * dt, []
    for _ in range(2 * steps + 1):
        adot = math.sqrt((cb + rad / a + (1 - cb - rad) * a ** 3) / a)
        out.append((a, dt, adot, 1.5 * cb * float(np.float32(1 / adot)) / a))
        a += 0.5 * dt
    return out


def _corners(x, ng):
    """(weight, linear cell index) of each of the 8 cells around every particle."""
    lo = x.floor()
    d, i = x - lo, torch.remainder(lo, ng).long()
    for c in range(8):
        b = [c >> 2 & 1, c >> 1 & 1, c & 1]
        j = [torch.remainder(i[:, a] + b[a], ng) for a in range(3)]
        w = 1.0
        for a in range(3):
            w = w * (d[:, a] if b[a] else 1 - d[:, a])
        yield w, (j[0] * ng + j[1]) * ng + j[2]


def _density(x, ng, mass):
    rho = torch.zeros(ng ** 3, dtype=torch.float64, device="cuda")
    for w, i in _corners(x, ng):
        rho.index_add_(0, i, w * mass)
    return rho.view(ng, ng, ng)


def _potential(rho):
    ng = rho.shape[0]
    # the framework's Green's function takes its cosines in single precision, as the reference does
    c = torch.cos(torch.arange(ng, device="cuda").float() * np.float32(2 * math.pi / ng)).double() - 1.0
    s = c[:, None, None] + c[None, :, None] + c[None, None, : ng // 2 + 1]
    s[0, 0, 0] = math.inf
    f = torch.fft.rfftn(rho)
    f *= 0.5 / ng ** 3 / s
    return torch.fft.irfftn(f, s=rho.shape, norm="forward")


def _exact_steps(ng, np_side, seed, steps):
    x, v = (t.double() for t in _particles(ng, np_side, seed))
    ep = _epochs(ng, np_side, steps)

    def drift(x, a, dt, adot, _):
        return torch.remainder(x + v * float(np.float32(0.5 * dt / (a * a * adot))), ng)

    for s in range(steps):
        x = drift(x, *ep[2 * s])
        phi = _potential(_density(x, ng, (ng / np_side) ** 3))
        _, dt, _, fscal = ep[2 * s + 1]
        for d in range(3):
            f = (0.5 * (torch.roll(phi, 1, d) - torch.roll(phi, -1, d))).view(-1)
            for w, i in _corners(x, ng):
                v[:, d] += w * (dt * fscal) * f[i]
            del f
        x = drift(x, *ep[2 * s + 2])
    x[x.float() >= ng] = 0.0  # a position that rounds to the box side is 0
    return {"x": x, "v": v}


def _exact_pk(case, seed):
    ng, fold = case["ng"], case["fold"]
    x = _particles(ng, case["np"], seed)[0].double()
    x = torch.remainder(x * 2 ** fold, ng)
    f = torch.fft.rfftn(_density(x, ng, (ng / case["np"]) ** 3) - 1.0)
    i = torch.arange(ng, device="cuda")
    m = torch.where(i > ng // 2 - 1, i - ng, i).double()
    # the bins' edges follow the folded box in k, the power the unfolded one (power.cu:174-227)
    d = 2 * math.pi / ng * 2 ** fold
    kf = (m * d).float()
    kz = kf[: ng // 2 + 1]
    k = (kf[:, None, None] ** 2 + kf[None, :, None] ** 2 + kz[None, None, :] ** 2).sqrt().double()
    h = 0.5 * m * (2 * math.pi / ng)
    w = torch.where(m == 0, 1.0, (torch.sin(h) / h) ** -4)
    p = f.abs().square() / ng ** 3 * w[:, None, None] * w[None, :, None] * w[None, None, : ng // 2 + 1]
    k_max = math.sqrt(3 * (ng // 2) ** 2) * d
    centres = np.arange(case["bins"]) + 0.5
    if case["log"]:
        step = math.log(k_max / d) / case["bins"]
        b = torch.log(k / d) / step
        centres = d * np.exp(step * centres)
    else:
        step = (k_max - d) / case["bins"]
        b = (k - d) / step
        centres = d + step * centres
    two = torch.full_like(p, 2.0)
    two[:, :, 0] = two[:, :, ng // 2] = 1.0
    two[0, 0, 0] = two[ng // 2, ng // 2, ng // 2] = 0.0
    ok = (b > -1) & (b < case["bins"])
    b = torch.where(ok, b, 0.0).long()
    two *= ok
    n = torch.zeros(case["bins"], dtype=torch.float64, device="cuda").index_add_(0, b.reshape(-1), two.reshape(-1))
    s = torch.zeros_like(n).index_add_(0, b.reshape(-1), (p * two).reshape(-1))
    return {"k": centres, "p": torch.where(n > 0, s / n.clamp(min=1), 0.0), "n": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "step":
        return _exact_steps(case["ng"], case["np"], seed, case["steps"])
    if kind in ("ensemble", "classes"):
        out = {"x": {}, "v": {}}
        for c, side in enumerate(int(s) for s in case["sides"].split(",")):
            got = [_exact_steps(side, side, seed + 1000 * c + k, case["steps"]) for k in range(case["slots"])]
            for key in out:
                out[key][str(side)] = torch.stack([g[key] for g in got])
        return out
    if kind == "pk":
        return _exact_pk(case, seed)
    if kind == "fft":
        grid = prepare(case, seed)["grid"].to(torch.complex128)
        return torch.fft.ifftn(grid, norm="forward") if case["inverse"] else torch.fft.fftn(grid)
    return None  # initial conditions start from cuRAND's draws, which plain torch does not make


# ---- what a pass cannot do without -----------------------------------------------
def _step_work(ng, np_side, steps):
    """Particles in and out (48 B each) and, in each step, 16 B a particle for the deposit, 56 for the kick and the
    drifts, and 32 B a cell for the transforms of the density and the potential in single precision."""
    part, cell = np_side ** 3, ng ** 3
    fft = 5 * cell * math.log2(cell)  # a real transform and back
    return 48 * part + steps * (72 * part + 32 * cell), steps * (200 * part + fft + 10 * cell)


def work(case):
    kind = case["kind"]
    if kind == "step":
        b, f = _step_work(case["ng"], case["np"], case["steps"])
    elif kind in ("ensemble", "classes"):
        b = f = 0
        for s in case["sides"].split(","):
            w = _step_work(int(s), int(s), case["steps"])
            b, f = b + case["slots"] * w[0], f + case["slots"] * w[1]
    elif kind == "pk":
        part, cell = case["np"] ** 3, case["ng"] ** 3
        b, f = 16 * part + 20 * cell, 60 * part + 2.5 * cell * math.log2(cell) + 10 * cell
    elif kind == "ic":
        cell = case["ng"] ** 3
        b, f = 80 * cell, 10 * cell * math.log2(cell) + 200 * cell
    else:
        cell = case["ng"] ** 3
        # the grid's copy to the buffer transformed in place, then the transform
        b, f = 32 * cell, 5 * cell * math.log2(cell)
    return {"bytes": b, "flops": f}
