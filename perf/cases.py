"""The work that users of this framework have it do, as cases that can be timed and checked.

A case is a dict with a "kind":

  induced   the velocity of vortex-ring sheets at points: ``InducedVelocity`` on host arrays, or (where "device") the
            allocation-free C entry on device arrays
  advect    one ``AdvectFactory(scheme).Advect`` of a wake behind its wings
  solve     ``dense_solve`` of a wing's influence matrix
  rings     ``rings.AdvectParallel``: the legacy array-of-rings loop's wake advection
  step      one MainLoop of ``SimpleSimulator`` on a wake held at a fixed length, and the state after it
  sweep     a whole batched sweep: create, run, read the loads
  mlp       forward and backward of the warm-start network over a batch of panels

Everything is drawn from the seed with NumPy.  The "mixed" form computes its velocities in single precision, so a
program that asks for it keeps what it gives in single precision; FP64 results stay in 64 bits.  ``exact`` restates the
mathematics in 64 bits with plain torch.
"""
import ctypes as C
import math

import numpy as np
import torch

import uvlm_b200 as U
from uvlm_b200.batch import make_batch
from uvlm_b200.warmstart import MLP

FLOP_PER_PAIR = 59  # one (point, lattice segment) interaction of the Biot-Savart law
FREE_FLIGHT = (-1.0, 0.0, 0.0)
IGNORE_ROWS = 5  # RK2 and RK4 move the newest wake rows by Euler


def listed():
    return [
        # the smallest call: a few points of a small wing's field (a unit test, a probe in a loop)
        {"name": "point_fp64", "kind": "induced", "precision": "fp64", "device": False, "num": 1, "rows": 4, "cols": 8,
         "targets": 9},
        # the velocity-field tools on a grid around three wings' wakes, sizes that fill no tile
        {"name": "field_fp64", "kind": "induced", "precision": "fp64", "device": False, "num": 3, "rows": 61,
         "cols": 47, "targets": 9001},
        # one evaluation over a full-length wake at its own nodes, single precision
        {"name": "wake_mixed", "kind": "induced", "precision": "mixed", "device": False, "num": 1, "rows": 400,
         "cols": 128, "targets": 32768},
        # the advection object of a program with its own time loop: four wings in formation, RK2
        {"name": "advect_rk2_fp64", "kind": "advect", "scheme": "RK2", "precision": "fp64", "num": 4, "rows": 16,
         "cols": 64, "wake": 40},
        # the reference's dense solve for a 24 x 96 wing
        {"name": "solve_fp64", "kind": "solve", "method": "fp64", "rows": 24, "cols": 96},
        # the accelerated solve at the size of the 32 x 128 wing
        {"name": "solve_tf32", "kind": "solve", "method": "tf32", "rows": 32, "cols": 128},
        # the legacy loop: an 8 x 16 wing and 60 wake rows as an array of rings
        {"name": "rings_advect", "kind": "rings", "rows": 8, "cols": 16, "wake": 60},
        # the smallest simulation, the 8 x 16 plunging wing: launches and latency
        {"name": "step_small_fp64", "kind": "step", "precision": "fp64", "scheme": "euler", "num": 1, "rows": 8,
         "cols": 16, "wake": 50},
        # an ordinary simulation in the plain form: dense solve and N-body both count
        {"name": "step_fp64", "kind": "step", "precision": "fp64", "scheme": "RK2", "num": 1, "rows": 24, "cols": 96,
         "wake": 100},
        # the headline simulation: 32 x 128 wing, 51,200-ring wake, RK2, mixed form
        {"name": "step_mixed", "kind": "step", "precision": "mixed", "scheme": "RK2", "num": 1, "rows": 32,
         "cols": 128, "wake": 400},
        # a parameter study: many seeded flapping wings from rest, batched
        {"name": "sweep_mixed", "kind": "sweep", "precision": "mixed", "cases": 40, "steps": 24},
        # training of the learned warm start: gradients over the panels of one large step
        {"name": "mlp_gradients", "kind": "mlp", "batch": 4096},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["induced", "induced", "advect", "advect", "solve", "rings", "step", "step", "sweep", "mlp"])
    prec = rng.choice(["fp64", "mixed"])
    if kind == "induced":
        if rng.random() < 0.35:  # the allocation-free entry, within its scratch
            return {"kind": kind, "precision": prec, "device": True, "num": rng.randint(1, 3), "rows": _log(rng, 4, 100),
                    "cols": _log(rng, 4, 130), "targets": _log(rng, 5, 20000)}
        most = 400 if prec == "mixed" else 100
        return {"kind": kind, "precision": prec, "device": False, "num": rng.randint(1, 4 if most == 100 else 1),
                "rows": _log(rng, 4, most), "cols": _log(rng, 4, 128), "targets": _log(rng, 1, 32000)}
    if kind == "advect":
        return {"kind": kind, "scheme": rng.choice(["euler", "RK2", "RK4", "AB2"]), "precision": prec,
                "num": rng.randint(1, 4), "rows": _log(rng, 3, 16), "cols": _log(rng, 6, 64), "wake": _log(rng, 3, 60)}
    if kind == "solve":
        return {"kind": kind, "method": rng.choice(["fp64", "tf32", "bf16"]), "rows": _log(rng, 4, 32),
                "cols": _log(rng, 8, 128)}
    if kind == "rings":
        return {"kind": kind, "rows": rng.randint(3, 12), "cols": 2 * rng.randint(3, 16), "wake": _log(rng, 4, 90)}
    if kind == "step":
        num = rng.randint(1, 4)
        return {"kind": kind, "precision": prec, "scheme": rng.choice(["euler", "RK2"]), "num": num,
                "rows": _log(rng, 4, 32 if num == 1 else 16), "cols": 2 * _log(rng, 4, 48 if num == 1 else 32),
                "wake": _log(rng, 8, (300 if prec == "mixed" else 100) // num)}
    if kind == "sweep":
        most = 40 if prec == "mixed" else 12
        return {"kind": kind, "precision": prec, "cases": rng.randint(3, most), "steps": rng.randint(6, 24 if most == 40 else 12)}
    return {"kind": kind, "batch": _log(rng, 64, 16384)}


# ------------------------------------------------------------------ inputs
def _rng(case, seed):
    return np.random.default_rng([int(seed), len(case["kind"]), int(case.get("rows", 1)), int(case.get("cols", 1))])


def _kinematics(rng, n):
    """Heave and pitch of wing n about its leading edge, as the workloads of the benchmark have them."""
    w = rng.uniform(0.6, 1.0)
    ph = n * math.pi / 2 + rng.uniform(-0.2, 0.2)
    return {"alpha": rng.uniform(0.0, 0.06), "plug_amp": rng.uniform(0.1, 0.2), "plug_omega": w, "plug_phase": ph,
            "twist_amp": math.radians(rng.uniform(8, 14)), "twist_omega": w, "twist_phase": ph + math.pi / 2}


def _origin(n):
    return (1.5 * (n // 2), 0.0, 0.5 * (n % 2))  # the 2 x 2 tandem/biplane formation


def _lattice(rows, cols, span):
    """Nodes of a flat wing of chord 1 (rows + 1, cols + 1, 3)."""
    x, y = np.meshgrid(np.linspace(0, 1, rows + 1), np.linspace(-span / 2, span / 2, cols + 1), indexing="ij")
    return np.stack([x, y, np.zeros_like(x)], -1)


def _move(kin, x, t, origin):
    """Reference nodes x (..., 3), given without their origin, moved by heave and pitch at time t."""
    m = _Motion(kin)
    return m.at(torch.from_numpy(x), t).numpy() + np.asarray(origin)


def _wake(rng, kins, cols, span, rows, dt, t):
    """rows + 1 node rows shed by the moving trailing edges and convected, with some roll-up: older rows wave and the
    tips curl; circulations follow the motion."""
    y = np.linspace(-span / 2, span / 2, cols + 1)
    edge = np.stack([np.ones(cols + 1), y, np.zeros(cols + 1)], -1)
    pos = np.zeros((len(kins), rows + 1, cols + 1, 3))
    gamma = np.zeros((len(kins), rows, cols))
    mid = 0.5 * (y[1:] + y[:-1]) / (span / 2)
    for n, k in enumerate(kins):
        a, b, c = rng.uniform(0, 2 * math.pi, 3)
        tip = np.abs(2 * y / span) ** 6 * np.sign(y)
        for i in range(rows + 1):
            p = _move(k, edge, t - i * dt, _origin(n))
            age = 1 - math.exp(-i * dt / 3)
            p[:, 0] += i * dt + 0.03 * age * np.sin(1.3 * y + a + 0.9 * i * dt)
            p[:, 1] += age * (0.02 * np.sin(2.1 * y + b + 0.7 * i * dt) - 0.1 * tip)
            p[:, 2] += age * (0.05 * np.sin(1.1 * y + c + 1.1 * i * dt) + 0.1 * np.abs(tip) * math.sin(0.8 * i * dt))
            pos[n, i] = p
        shape = np.sqrt(np.clip(1 - mid ** 2, 0, None)) * rng.uniform(0.2, 0.4)
        when = t - dt * np.arange(rows)[:, None]
        gamma[n] = shape * (0.3 + np.sin(k["plug_omega"] * when + k["plug_phase"]))
    gamma += 1e-3 * rng.standard_normal(gamma.shape)
    pos += 1e-3 * rng.standard_normal(pos.shape)
    return pos, gamma


def _formation(case, seed):
    """Wings and wake of an "advect" or "step" case."""
    rng = _rng(case, seed)
    num, rows, cols, wake = case["num"], case["rows"], case["cols"], case["wake"]
    span = 8.0 if num == 1 else 4.0
    kins = [_kinematics(rng, n) for n in range(num)]
    dt = 2 * math.pi / kins[0]["plug_omega"] / 40
    step = wake + 1 + int(rng.integers(0, 40))
    t = (step - 1) * dt
    base = _lattice(rows, cols, span)
    wing = np.stack([_move(k, base, t, _origin(n)) for n, k in enumerate(kins)])
    pos, wg = _wake(rng, kins, cols, span, wake, dt, t)
    mid = (np.arange(cols) + 0.5) / cols * 2 - 1
    g = np.sqrt(np.clip(1 - mid ** 2, 0, None)) * np.linspace(1, 0.3, rows)[:, None]
    gamma = np.stack([g * rng.uniform(0.1, 0.3) for _ in range(num)]) + 1e-3 * rng.standard_normal((num, rows, cols))
    prev = gamma * 0.97
    pos[:, 0] = wing[:, -1]
    return {"kins": kins, "dt": dt, "step": step, "span": span, "wing_pos": wing, "wing_gamma": gamma,
            "wing_gamma_prev": prev, "wake_pos": pos, "wake_gamma": wg}


def _sheets(case, seed):
    """Sheets, circulations and points of an "induced" case: wakes with some of their own nodes and points around."""
    rng = _rng(case, seed)
    kins = [_kinematics(rng, n) for n in range(case["num"])]
    span = 8.0 if case["cols"] > 64 else 4.0
    pos, gamma = _wake(rng, kins, case["cols"], span, case["rows"], 0.157, 20.0)
    flat = pos.reshape(-1, 3)
    n = case["targets"]
    own = flat[rng.integers(0, len(flat), n - n // 4)]
    free = rng.uniform(flat.min(0) - 0.5, flat.max(0) + 0.5, (n // 4, 3))
    return pos, gamma, np.concatenate([own, free])


def _ring_loop(case, seed):
    """The legacy loop's containers: a wing and its wake as rings (n, 4, 3), and their circulations."""
    rng = _rng(case, seed)
    k = _kinematics(rng, 0)
    rows, cols, wake = case["rows"], case["cols"], case["wake"]
    wing = _move(k, _lattice(rows, cols, 4.0), 20.0, _origin(0))
    pos, wg = _wake(rng, [k], cols, 4.0, wake, 0.125, 20.0)

    def rings(p):
        return np.ascontiguousarray(np.stack([p[:-1, :-1], p[1:, :-1], p[1:, 1:], p[:-1, 1:]], 2).reshape(-1, 4, 3))

    bound, shed = rings(wing), rings(pos[0])
    gammas = np.concatenate([0.2 + 0.05 * rng.standard_normal(len(bound)), wg.ravel()])
    return np.concatenate([bound, shed]), gammas, shed, np.array([1.0, 0.0, 0.05]), 0.125


def _system(case, seed):
    """The influence matrix of a cambered, pitched wing and a right-hand side."""
    rng = _rng(case, seed)
    rows, cols = case["rows"], case["cols"]
    p = _lattice(rows, cols, 8.0)
    p[..., 2] = 0.05 * p[..., 0] * (1 - p[..., 0]) + 0.02 * rng.uniform() * p[..., 1] ** 2
    p = p + 2e-3 / max(rows, cols / 8) * rng.standard_normal(p.shape)
    nodes = torch.from_numpy(p)[None].to(_device())
    centre, normal, _ = _panels(nodes)
    A = _influence(nodes, centre, normal)
    b = -normal.reshape(-1, 3) @ torch.tensor([1.0, 0.0, rng.uniform(0.05, 0.2)], dtype=torch.float64, device=A.device)
    return A.cpu().numpy(), (b.cpu().numpy() + 1e-3 * rng.standard_normal(rows * cols))


def _network(case, seed):
    rng = _rng(case, seed)
    dims = [8, 256, 256, 256, 1]
    params = []
    for i in range(4):
        params += [rng.standard_normal(dims[i] * dims[i + 1]) * math.sqrt(2.0 / dims[i]),
                   0.1 * rng.standard_normal(dims[i + 1])]
    X = rng.standard_normal((case["batch"], 8)).astype(np.float32)
    T = (0.2 * np.tanh(X[:, 0] - 0.5 * X[:, 3]) + 0.05 * X[:, 6] * X[:, 7]).astype(np.float32)
    mean = (0.1 * rng.standard_normal(8)).astype(np.float32)
    std = (0.5 + rng.random(8)).astype(np.float32)
    return np.concatenate(params).astype(np.float32), X, T, mean, std, 0.7


def _sweep_cases(case, seed):
    """The seeded flapping-wing sweep: rows 4..16, even columns 8..64, aspect ratio 2..10, reduced frequency 0.1..1."""
    rng = _rng(case, seed)
    out = []
    for _ in range(case["cases"]):
        w = 2 * float(rng.uniform(0.1, 1.0))
        out.append(dict(rows=int(rng.integers(4, 17)), cols=2 * int(rng.integers(4, 33)), chord=1.0,
                        span=float(rng.uniform(2, 10)), omega=w, heave=float(rng.uniform(0.05, 0.3)),
                        pitch_deg=float(rng.uniform(0, 20)), dt=2 * math.pi / w / 40))
    return out


def prepare(case, seed):
    k = case["kind"]
    s = {"case": case}
    if k == "induced":
        pos, gamma, targets = _sheets(case, seed)
        if case["device"]:
            s["pos"], s["gamma"], s["targets"] = (torch.from_numpy(a).cuda() for a in (pos, gamma, targets))
            s["out"] = torch.empty_like(s["targets"])
        else:
            s["pos"], s["gamma"], s["targets"] = pos, gamma, targets
    elif k == "advect":
        s.update(_formation(case, seed))
        s["advection"] = U.AdvectFactory(case["scheme"], case["precision"])
    elif k == "solve":
        s["A"], s["b"] = _system(case, seed)
    elif k == "rings":
        s["rings"], s["gammas"], s["wake"], s["stream"], s["dt"] = _ring_loop(case, seed)
    elif k == "step":
        f = _formation(case, seed)
        sim = U.SimpleSimulator(precision=case["precision"], max_wake_rows=case["wake"] + 8,
                                erase_wake_after=case["wake"],
                                warm_start="extrapolate" if case["precision"] == "mixed" else "previous")
        for n, q in enumerate(f["kins"]):
            m = U.Morphing().set_alpha(q["alpha"]).set_plug(q["plug_amp"], q["plug_omega"], q["plug_phase"])
            m.set_twist(q["twist_amp"], q["twist_omega"], q["twist_phase"])
            sim.AddWing(U.RectGenerator(), m, 1.0, f["span"], case["rows"], case["cols"], _origin(n))
        sim.set_forward_flight(FREE_FLIGHT)
        sim.set_advection(case["scheme"])
        sim.begin()
        sim.set_state(case["wake"], f["wing_pos"], f["wake_pos"], f["wing_gamma"], f["wing_gamma_prev"],
                      f["wake_gamma"])
        s.update(sim=sim, step=f["step"], dt=f["dt"])
    elif k == "sweep":
        s["cases"] = _sweep_cases(case, seed)
    else:
        params, s["X"], s["T"], mean, std, scale = _network(case, seed)
        s["net"] = MLP(seed=0)
        s["net"].set_params(params)
        s["net"].set_normalization(mean, std, scale)
    return s


def _kept(case, v):
    return v.astype(np.float32) if case.get("precision") == "mixed" else v


def run(s):
    case = s["case"]
    k = case["kind"]
    if k == "induced":
        if not case["device"]:
            return _kept(case, U.InducedVelocity(s["targets"], s["pos"], s["gamma"], case["precision"]))
        D = C.POINTER(C.c_double)
        pos, gamma, targets, out = (C.cast(s[n].data_ptr(), D) for n in ("pos", "gamma", "targets", "out"))
        rc = U.lib().uvlm_sheet_induced_velocity_noalloc(pos, gamma, case["num"], case["rows"], case["cols"], targets,
                                                         case["targets"], out, int(case["precision"] == "mixed"),
                                                         torch.cuda.current_stream().cuda_stream)
        if rc:
            raise RuntimeError(U.lib().uvlm_global_last_error().decode())
        return s["out"].float() if case["precision"] == "mixed" else s["out"]
    if k == "advect":
        return _kept(case, s["advection"].Advect(s["wing_pos"], s["wing_gamma"], s["wake_pos"], s["wake_gamma"],
                                                 FREE_FLIGHT, s["dt"]))
    if k == "solve":
        return U.dense_solve(s["A"], s["b"], case["method"])[0]
    if k == "rings":
        return U.rings.AdvectParallel(s["rings"], s["gammas"], s["wake"], s["stream"], s["dt"])
    if k == "step":
        row = s["sim"].step(s["step"], s["dt"])
        s["step"] += 1
        st = s["sim"].state()
        return {"loads": _kept(case, row[1:]), "wing_gamma": _kept(case, st["wing_gamma"]),
                "wake_pos": _kept(case, st["wake_pos"])}
    if k == "sweep":
        sim = make_batch(s["cases"], precision=case["precision"], max_steps=case["steps"])
        sim.run(case["steps"])
        loads = sim.loads()
        sim.close()
        return _kept(case, loads)
    g, loss = s["net"].gradients(s["X"], s["T"])
    return {"gradients": g, "loss": loss}


# ------------------------------------------------------------------- work
def _segments(num, rows, cols):
    return num * ((rows + 1) * cols + rows * (cols + 1))


def work(case):
    k = case["kind"]
    if k == "induced":
        nodes = case["num"] * (case["rows"] + 1) * (case["cols"] + 1)
        pairs = case["targets"] * _segments(case["num"], case["rows"], case["cols"])
        return {"bytes": 24 * nodes + 8 * case["num"] * case["rows"] * case["cols"] + 48 * case["targets"],
                "flops": FLOP_PER_PAIR * pairs}
    if k == "advect":
        num, rows, cols, wake = case["num"], case["rows"], case["cols"], case["wake"]
        segs = _segments(num, rows, cols) + _segments(num, wake, cols)
        evals = {"euler": 1, "AB2": 1, "RK2": 1, "RK4": 2}[case["scheme"]]
        last = max(0, wake - IGNORE_ROWS) if case["scheme"] in ("RK2", "RK4") else 0
        return {"bytes": num * (cols + 1) * (24 * (rows + 1) + 48 * (wake + 1)) + 8 * num * cols * (rows + wake),
                "flops": FLOP_PER_PAIR * segs * num * (cols + 1) * (evals * wake + last)}
    if k == "solve":
        n = case["rows"] * case["cols"]
        return {"bytes": 8 * n * n + 16 * n, "flops": 2 * n ** 3 / 3 + 2 * n * n}
    if k == "rings":
        bound, shed = case["rows"] * case["cols"], case["wake"] * case["cols"]
        return {"bytes": 104 * (bound + shed) + 192 * shed, "flops": FLOP_PER_PAIR * 4 * (bound + shed) * 4 * shed}
    if k == "step":
        num, rows, cols, wake = case["num"], case["rows"], case["cols"], case["wake"] + 1
        n = num * rows * cols
        bound, shed = _segments(num, rows, cols), _segments(num, wake, cols)
        lines = num * rows * (2 * cols + 1)
        nodes = num * (cols + 1) * wake
        moved = nodes + (num * (cols + 1) * (wake - IGNORE_ROWS) if case["scheme"] == "RK2" else 0)
        pairs = n * shed + lines * (bound + shed) + moved * (bound + shed)
        solve = 2 * n ** 3 / 3 if case["precision"] == "fp64" else 20 * n * n
        return {"bytes": 48 * nodes + 8 * num * cols * wake + 24 * n, "flops": FLOP_PER_PAIR * (pairs + n * bound) + solve}
    if k == "sweep":
        flops = 0.0
        for rows, cols in ((10, 36),):  # the mean wing of the sweep
            for wake in range(case["steps"]):
                n = rows * cols
                bound, shed = _segments(1, rows, cols), _segments(1, wake, cols) if wake else 0
                pairs = n * (bound + shed) + rows * (2 * cols + 1) * (bound + shed) + wake * (cols + 1) * (bound + shed)
                flops += FLOP_PER_PAIR * pairs + 4 * n * n
        return {"bytes": 24 * case["cases"] * case["steps"], "flops": case["cases"] * flops}
    dense = 2 * 256 * 256 + 8 * 256 + 256
    return {"bytes": case["batch"] * 36 + 8 * (dense + 769), "flops": case["batch"] * 6 * dense}


# --------------------------------------------- the same mathematics in 64 bits
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _velocity(a, b, g, x, most=1 << 24):
    """Velocity at points x (n, 3) of the segments a -> b (m, 3) with strengths g (m,): the Biot-Savart law with the
    cut-offs |r1 x r2|^2 < 1e-10 and |r| < 1e-10."""
    out = torch.zeros_like(x)
    if not len(a):
        return out
    r0 = (b - a)[None]
    at = 0
    while at < len(x):
        n = max(1, min(len(x) - at, most // len(a)))
        for sa in range(0, len(a), most):
            s = slice(sa, sa + most)
            out[at:at + n] += _law(a[s], b[s], r0[:, s], g[s], x[at:at + n])
        at += n
    return out / (4 * math.pi)


def _law(a, b, r0, g, x, keep=False):
    r1, r2 = x[:, None] - a[None], x[:, None] - b[None]
    n1, n2 = r1.norm(dim=-1), r2.norm(dim=-1)
    d = torch.linalg.cross(r0.expand_as(r1), r1)
    d2 = (d * d).sum(-1)
    dot = (r1 * r2).sum(-1)
    del r1, r2
    nn = n1 * n2
    # r0.(r1/|r1| - r2/|r2|) / |d|^2 in the two forms that do not cancel
    f = torch.where(dot >= 0, (n1 + n2) / (nn * (nn + dot)), (n1 + n2) * (nn - dot) / (nn * d2))
    f = torch.where((d2 < 1e-10) | (n1 < 1e-10) | (n2 < 1e-10), torch.zeros_like(f), f)
    if keep:
        return d * f[..., None]
    return torch.einsum("xs,xsc->xc", f * g, d)


def _lattice_segments(p, g):
    """Unique segments of sheets p (num, R + 1, C + 1, 3) and the ring circulations g (num, R, C) they carry."""
    z = torch.nn.functional.pad(g, (1, 1, 1, 1))
    span = z[:, 1:, 1:-1] - z[:, :-1, 1:-1]
    chord = z[:, 1:-1, :-1] - z[:, 1:-1, 1:]
    a = torch.cat([p[:, :, :-1].reshape(-1, 3), p[:, :-1].reshape(-1, 3)])
    b = torch.cat([p[:, :, 1:].reshape(-1, 3), p[:, 1:].reshape(-1, 3)])
    return a, b, torch.cat([span.reshape(-1), chord.reshape(-1)])


def _sheet_velocity(sheets, x):
    """Velocity at x of several (nodes, circulations) sheet sets."""
    parts = [_lattice_segments(p, g) for p, g in sheets if g.numel()]
    if not parts:
        return torch.zeros_like(x)
    a, b, g = (torch.cat(v) for v in zip(*parts))
    return _velocity(a, b, g, x)


def _panels(p):
    """Collocation points, unit normals and areas of every panel."""
    p00, p01, p10, p11 = p[:, :-1, :-1], p[:, :-1, 1:], p[:, 1:, :-1], p[:, 1:, 1:]
    n = torch.linalg.cross(p11 - p00, p01 - p10)
    area = torch.linalg.cross(p10 - p00, p01 - p00).norm(dim=-1)
    return (p00 + p10 + p11 + p01) / 4, n / n.norm(dim=-1, keepdim=True), area


def _influence(p, centre, normal):
    """A[k][l]: normal velocity at panel k of ring l with unit circulation."""
    num, R1, C1, _ = p.shape
    R, Cc = R1 - 1, C1 - 1
    x, n = centre.reshape(-1, 3), normal.reshape(-1, 3)
    A = torch.empty(len(x), num * R * Cc, dtype=torch.float64, device=p.device)
    step = max(1, (1 << 23) // (num * R1 * C1))
    sa, sb = p[:, :, :-1].reshape(-1, 3), p[:, :, 1:].reshape(-1, 3)
    ha, hb = p[:, :-1].reshape(-1, 3), p[:, 1:].reshape(-1, 3)
    for k in range(0, len(x), step):
        xk, nk = x[k:k + step], n[k:k + step]
        S = (_law(sa, sb, (sb - sa)[None], None, xk, True) * nk[:, None]).sum(-1).reshape(-1, num, R1, Cc)
        H = (_law(ha, hb, (hb - ha)[None], None, xk, True) * nk[:, None]).sum(-1).reshape(-1, num, R, C1)
        A[k:k + step] = (S[:, :, :-1] + H[..., 1:] - S[:, :, 1:] - H[..., :-1]).reshape(len(xk), -1)
    return A / (4 * math.pi)


class _Motion:
    """x = heave + attack (twist x_ref): the reference's closed-form kinematics without flap and bend."""

    def __init__(self, k):
        self.k = k

    def at(self, x, t):
        k = self.k
        y = x[..., 1].abs()
        beta = k["twist_amp"] * math.sin(k["twist_omega"] * t + k["twist_phase"])
        th = k.get("alpha", 0.0) + beta  # two rotations about the same axis
        z = k["plug_amp"] * math.sin(k["plug_omega"] * t + k.get("plug_phase", 0.0))
        c, s = math.cos(th), math.sin(th)
        return torch.stack([c * x[..., 0] + s * x[..., 2], torch.where(x[..., 1] < 0, -y, y),
                            -s * x[..., 0] + c * x[..., 2] + z], -1)

    def velocity(self, x, t, h=1e-6):
        return (self.at(x, t + h) - self.at(x, t - h)) / (2 * h)


class _Loop:
    """MainLoop of the time-stepper: kinematics, shed, matrix, right-hand side, solve, loads, advection."""

    def __init__(self, motions, bases, origins, span, scheme):
        self.m, self.span, self.scheme = motions, span, scheme
        self.base, self.origin = bases, origins
        self.ff = torch.tensor(FREE_FLIGHT, dtype=torch.float64, device=bases.device)

    def moved(self, fn, x):
        return torch.stack([fn(m, x[n]) for n, m in enumerate(self.m)])

    def step(self, step, dt, gamma, wake, wake_gamma):
        t = step * dt
        pos = self.moved(lambda m, x: m.at(x, t), self.base) + self.origin
        wake = torch.cat([pos[:, -1:], wake], 1)
        if step > 0:
            wake_gamma = torch.cat([gamma[:, -1:], wake_gamma], 1)
        centre, normal, area = _panels(pos)
        centre0, _, _ = _panels(self.base)
        own = self.moved(lambda m, x: m.velocity(x, t), centre0)
        flat = centre.reshape(-1, 3)
        u = _sheet_velocity([(wake, wake_gamma)], flat) - own.reshape(-1, 3) - self.ff
        b = -(u * normal.reshape(-1, 3)).sum(-1)
        before, gamma = gamma, torch.linalg.solve(_influence(pos, centre, normal), b).reshape(gamma.shape)
        both = [(pos, gamma), (wake, wake_gamma)]
        loads = self.loads(pos, gamma, before, normal, area, both, t, dt)
        wake = self.advect(pos, gamma, wake, wake_gamma, dt)
        return loads, gamma, wake, wake_gamma

    def loads(self, pos, gamma, before, normal, area, sheets, t, dt):
        z = torch.nn.functional.pad(gamma, (1, 1, 1, 1))
        out = []
        for n, m in enumerate(self.m):
            p, q = pos[n], self.base[n]
            a = torch.cat([p[:-1, :-1].reshape(-1, 3), p[:-1].reshape(-1, 3)])  # the trailing edge carries no load
            b = torch.cat([p[:-1, 1:].reshape(-1, 3), p[1:].reshape(-1, 3)])
            a0 = torch.cat([q[:-1, :-1].reshape(-1, 3), q[:-1].reshape(-1, 3)])
            b0 = torch.cat([q[:-1, 1:].reshape(-1, 3), q[1:].reshape(-1, 3)])
            g = torch.cat([(z[n, 1:-1, 1:-1] - z[n, :-2, 1:-1]).reshape(-1), (z[n, 1:-1, :-1] - z[n, 1:-1, 1:]).reshape(-1)])
            u = _sheet_velocity(sheets, (a + b) / 2) - self.ff - m.velocity((a0 + b0) / 2, t)
            F = (torch.linalg.cross(u, b - a) * g[:, None]).sum(0)
            F = F + (normal[n] * ((gamma[n] - before[n]) / dt * area[n])[..., None]).sum((0, 1))
            c = F / (0.5 * (self.ff * self.ff).sum() * self.span[n])
            out += [c[0], c[2]]
        return torch.stack(out)

    def advect(self, pos, gamma, wake, wake_gamma, dt):
        return _advected(self.scheme, pos, gamma, wake, wake_gamma, self.ff, dt)


def _advected(scheme, pos, gamma, wake, wake_gamma, ff, dt):
    def velocity(w, first=1):
        v = torch.zeros_like(w) - ff
        if w.shape[1] > first:
            x = w[:, first:]
            v[:, first:] += _sheet_velocity([(pos, gamma), (w, wake_gamma)], x.reshape(-1, 3)).reshape(x.shape)
        return v

    k1 = velocity(wake)
    late = (torch.arange(wake.shape[1], device=wake.device) > IGNORE_ROWS)[None, :, None, None]
    if scheme == "RK2":
        k2 = velocity(wake + k1 * dt, IGNORE_ROWS + 1)
        return wake + torch.where(late, (k1 + k2) / 2, k1) * dt
    if scheme == "RK4":  # the reference takes its third slope twice
        k2 = velocity(wake + k1 * dt / 2)
        k3 = velocity(wake + k2 * dt / 2, IGNORE_ROWS + 1)
        return wake + torch.where(late, (k1 + 2 * k2 + 3 * k3) / 6, k1) * dt
    return wake + k1 * dt  # Euler, and the first call of AB2


def _f64(a):
    return torch.from_numpy(np.ascontiguousarray(a)).double().to(_device())


def exact(case, seed):
    k = case["kind"]
    if k == "induced":
        pos, gamma, targets = _sheets(case, seed)
        return _sheet_velocity([(_f64(pos), _f64(gamma))], _f64(targets))
    if k == "advect":
        f = _formation(case, seed)
        return _advected(case["scheme"], *(_f64(f[n]) for n in ("wing_pos", "wing_gamma", "wake_pos", "wake_gamma")),
                         _f64(FREE_FLIGHT), f["dt"])
    if k == "solve":
        A, b = _system(case, seed)
        return torch.linalg.solve(_f64(A), _f64(b))
    if k == "rings":
        rings, gammas, shed, stream, dt = _ring_loop(case, seed)
        r, x = _f64(rings), _f64(shed)
        v = _velocity(r.roll(-1, 1).reshape(-1, 3), r.reshape(-1, 3), _f64(gammas).repeat_interleave(4), x.reshape(-1, 3))
        return x + (v.reshape(x.shape) + _f64(stream)) * dt
    if k == "step":
        f = _formation(case, seed)
        num = case["num"]
        base = _f64(np.stack([_lattice(case["rows"], case["cols"], f["span"])] * num))
        origin = _f64(np.array([_origin(n) for n in range(num)]))[:, None, None]
        loop = _Loop([_Motion(q) for q in f["kins"]], base, origin, [f["span"]] * num, case["scheme"])
        loads, gamma, wake, _ = loop.step(f["step"], f["dt"], *(_f64(f[n]) for n in ("wing_gamma", "wake_pos", "wake_gamma")))
        return {"loads": loads, "wing_gamma": gamma, "wake_pos": wake[:, :-1]}
    if k == "sweep":
        out = torch.zeros(case["steps"], case["cases"], 3, dtype=torch.float64)
        for c, d in enumerate(_sweep_cases(case, seed)):
            m = _Motion({"plug_amp": d["heave"], "plug_omega": d["omega"], "twist_amp": math.radians(d["pitch_deg"]),
                         "twist_omega": d["omega"], "twist_phase": math.pi / 2})
            base = _f64(_lattice(d["rows"], d["cols"], d["span"]))[None]
            loop = _Loop([m], base, torch.zeros(1, 1, 1, 3, dtype=torch.float64, device=base.device), [d["span"]], "euler")
            gamma = torch.zeros(1, d["rows"], d["cols"], dtype=torch.float64, device=base.device)
            wake = torch.zeros(1, 0, d["cols"] + 1, 3, dtype=torch.float64, device=base.device)
            wake_gamma = torch.zeros(1, 0, d["cols"], dtype=torch.float64, device=base.device)
            for s in range(case["steps"]):
                loads, gamma, wake, wake_gamma = loop.step(s, d["dt"], gamma, wake, wake_gamma)
                out[s, c, 0] = s * d["dt"]
                out[s, c, 1:] = loads.cpu()
        return out
    params, X, T, mean, std, scale = _network(case, seed)
    dims, at, w, h = [8, 256, 256, 256, 1], 0, [], (_f64(X) - _f64(mean)) / _f64(std)
    for i in range(4):
        n = dims[i] * dims[i + 1]
        W = torch.from_numpy(params[at:at + n]).bfloat16().double().reshape(dims[i], dims[i + 1]).to(_device())
        b = _f64(params[at + n:at + n + dims[i + 1]])
        at += n + dims[i + 1]
        w += [W.requires_grad_(), b.requires_grad_()]
        z = h @ W + b
        h = 0.5 * z * (1 + torch.erf(z / math.sqrt(2))) if i < 3 else z
    loss = ((h[:, 0] - _f64(T) / scale) ** 2).mean()
    loss.backward()
    return {"gradients": torch.cat([v.grad.reshape(-1) for v in w]), "loss": loss.detach()}
