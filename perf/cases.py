"""The solves that a user of this library runs, as measurable cases.

A case is a batched ``diffeqsolve`` -- forward, or forward and the gradient of a
loss -- on one of the registered fields, through the public call with its
defaults.  Families and the sizes that they span:

  vdp       Van der Pol, Dopri5 + PID(1e-6, 1e-9), one t1 per trajectory; forward
            and RecursiveCheckpointAdjoint; 1 to 65536 trajectories
  lv        Lotka-Volterra, Tsit5 + PID(1e-6, 1e-8), saves at many times; FP32 and
            FP64 state; 1 to 16384 trajectories
  ou        Ornstein-Uhlenbeck SDE, Heun, virtual Brownian tree; 64 to 65536
  node      neural ODE 64-128-128-64, Tsit5 or Dopri5 + PID(1e-5, 1e-7), value at
            t1; forward and RecursiveCheckpointAdjoint(64); 64 to 32768
  wide      neural ODE 64-256-256-64, 32 saves; forward and BacksolveAdjoint under
            either norm; 64 to 16384
  nsde      neural SDE 32-64-64-32 with a tanh diagonal diffusion, Heun, dt 0.01;
            forward and RecursiveCheckpointAdjoint; 64 to 32768
"""
import math

import torch

import diffrax_gb300 as dfx

DEV = "cuda"
WIDTHS = {"node": (64, 128, 128, 64), "wide": (64, 256, 256, 64), "nsde": (32, 64, 64, 32)}


def listed():
    return [
        # one trajectory: a simulation inside an outer program, where launches and
        # the latency of a step are all there is
        {"name": "vdp_one", "family": "vdp", "batch": 1, "t1": 20.0, "grad": False},
        # trajectories to compare with measured time series: many saves, few rows
        {"name": "lv_saves_1024", "family": "lv", "batch": 1024, "n_ts": 100, "t1": 140.0,
         "dtype": "float32"},
        # the same model in double precision at an odd batch: reference solutions
        {"name": "lv_f64_777", "family": "lv", "batch": 777, "n_ts": 17, "t1": 40.0,
         "dtype": "float64"},
        # a parameter sweep with horizons of its own per trajectory: the largest
        # analytic batch
        {"name": "vdp_uneven_65536", "family": "vdp", "batch": 65536, "t1": 50.0, "grad": False},
        # fitting initial values and parameters of an analytic model
        {"name": "vdp_grad_30011", "family": "vdp", "batch": 30011, "t1": 50.0, "grad": True},
        # Monte-Carlo paths of an analytic SDE
        {"name": "ou_paths_16384", "family": "ou", "batch": 16384, "n_steps": 100},
        # neural ODE: inference, and a training step at an odd batch
        {"name": "node_fwd_8192", "family": "node", "batch": 8192, "solver": "tsit5",
         "grad": False},
        {"name": "node_train_3001", "family": "node", "batch": 3001, "solver": "tsit5",
         "grad": True},
        # latent-trajectory model with 32 observation times: decode, and a training
        # step with the memory-free adjoint
        {"name": "wide_fwd_16384", "family": "wide", "batch": 16384, "norm": "rms",
         "grad": False},
        {"name": "wide_train_16384", "family": "wide", "batch": 16384, "norm": "rms",
         "grad": True},
        # neural SDE: sample paths, and a training step at an odd batch
        {"name": "nsde_fwd_32768", "family": "nsde", "batch": 32768, "n_steps": 100,
         "grad": False},
        {"name": "nsde_train_9001", "family": "nsde", "batch": 9001, "n_steps": 100,
         "grad": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    family = rng.choice(["vdp", "vdp", "lv", "ou", "node", "node", "wide", "wide", "nsde", "nsde"])
    grad = rng.random() < 0.5
    if family == "vdp":
        return {"family": family, "batch": _log_int(rng, 1, 65536),
                "t1": round(rng.uniform(6.0, 50.0), 3), "grad": grad}
    if family == "lv":
        return {"family": family, "batch": _log_int(rng, 1, 16384), "n_ts": _log_int(rng, 1, 200),
                "t1": round(rng.uniform(5.0, 140.0), 3),
                "dtype": rng.choice(["float32", "float64"])}
    if family == "ou":
        return {"family": family, "batch": _log_int(rng, 64, 65536),
                "n_steps": rng.randint(10, 200)}
    if family == "node":
        return {"family": family, "batch": _log_int(rng, 64, 32768),
                "solver": rng.choice(["tsit5", "dopri5"]), "grad": grad}
    if family == "wide":
        return {"family": family, "batch": _log_int(rng, 64, 16384),
                "norm": rng.choice(["rms", "seminorm"]), "grad": grad}
    return {"family": family, "batch": _log_int(rng, 64, 32768), "n_steps": rng.randint(10, 100),
            "grad": grad}


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------


def _bf16(x):
    """BF16 values held in FP32, as a model trained in BF16 hands them over."""
    return x.to(torch.bfloat16).float()


def _inputs(case, seed):
    """The case's inputs as tensors on the GPU, from the seed alone."""
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 1000003 + 17)
    B, family = case["batch"], case["family"]

    def uniform(shape, lo, hi):
        return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64) * (hi - lo) + lo

    if family == "vdp":
        return {"mu": uniform((B, 1), math.log(0.1), math.log(10.0)).exp().float(),
                "y0": uniform((B, 2), -2.0, 2.0).float(),
                "t1": uniform((B,), 0.1 * case["t1"], case["t1"])}
    if family == "lv":
        dtype = getattr(torch, case["dtype"])
        base = torch.tensor([0.1, 0.02, 0.4, 0.02], dtype=torch.float64, device=DEV)
        return {"y0": uniform((B, 2), 5.0, 15.0).to(dtype),
                "args": (base * uniform((4,), 0.95, 1.05)).to(dtype),
                "ts": torch.linspace(0.0, case["t1"], case["n_ts"] + 1, dtype=torch.float64,
                                     device=DEV)[1:].contiguous()}
    if family == "ou":
        return {"y0": uniform((B, 2), -2.0, 2.0).float(),
                "args": torch.tensor([1.5, 0.5, 0.6], device=DEV), "key": int(seed) % 100003 + 1}
    w = WIDTHS[family]

    def normal(*shape):
        return torch.randn(shape, generator=g, device=DEV)

    d = {"y0": normal(B, w[0]),
         "W": [_bf16(normal(w[i + 1], w[i]) / math.sqrt(w[i])) for i in range(3)],
         "b": [_bf16(0.1 * normal(w[i + 1])) for i in range(3)]}
    if family == "wide":
        d["ts"] = torch.linspace(0.0, 1.0, 32, dtype=torch.float64, device=DEV)
    if family == "nsde":
        d["Ws"] = _bf16(normal(w[0], w[0]) / math.sqrt(w[0]))
        d["bs"] = _bf16(0.1 * normal(w[0]))
        d["key"] = int(seed) % 100003 + 1
    return d


def prepare(case, seed):
    d = _inputs(case, seed)
    family, grad = case["family"], case.get("grad", False)
    s = {"case": case, "in": d, "leaves": []}
    if family == "vdp":
        s["terms"] = dfx.ODETerm(dfx.VanDerPol())
        s["leaves"] = [d["y0"], d["mu"]]
    elif family == "lv":
        s["terms"] = dfx.ODETerm(dfx.LotkaVolterra())
    elif family == "ou":
        ou = dfx.OrnsteinUhlenbeck()
        bm = dfx.VirtualBrownianTree(0.0, 1.0, 1e-3, (2,), key=d["key"])
        s["terms"] = dfx.MultiTerm(dfx.ODETerm(ou), dfx.ControlTerm(ou, bm))
    else:
        drift = dfx.ODETerm(dfx.MLPField(d["W"], d["b"]))
        s["leaves"] = [d["y0"], *d["W"], *d["b"]]
        s["terms"] = drift
        if family == "nsde":
            bm = dfx.VirtualBrownianTree(0.0, 1.0, 1e-3, (WIDTHS["nsde"][0],), key=d["key"])
            s["terms"] = dfx.MultiTerm(drift, dfx.ControlTerm(
                dfx.TanhDiagonalDiffusion(d["Ws"], d["bs"]), bm))
            s["leaves"] += [d["Ws"], d["bs"]]
    if grad:
        for x in s["leaves"]:
            x.requires_grad_(True)
    return s


def _solve(s):
    case, d, terms = s["case"], s["in"], s["terms"]
    family = case["family"]
    if family == "vdp":
        return dfx.diffeqsolve(
            terms, dfx.Dopri5(), 0.0, d["t1"], None, d["y0"], d["mu"],
            stepsize_controller=dfx.PIDController(rtol=1e-6, atol=1e-9, pcoeff=0.3, icoeff=0.4))
    if family == "lv":
        return dfx.diffeqsolve(
            terms, dfx.Tsit5(), 0.0, case["t1"], 0.1, d["y0"], d["args"],
            saveat=dfx.SaveAt(ts=d["ts"]),
            stepsize_controller=dfx.PIDController(rtol=1e-6, atol=1e-8))
    if family in ("ou", "nsde"):
        return dfx.diffeqsolve(terms, dfx.Heun(), 0.0, 1.0, 1.0 / case["n_steps"], d["y0"],
                               d.get("args"))
    pid = dfx.PIDController(rtol=1e-5, atol=1e-7)
    if family == "node":
        solver = dfx.Tsit5() if case["solver"] == "tsit5" else dfx.Dopri5()
        return dfx.diffeqsolve(terms, solver, 0.0, 1.0, None, d["y0"], stepsize_controller=pid,
                               adjoint=dfx.RecursiveCheckpointAdjoint(checkpoints=64))
    if case["norm"] == "seminorm":
        adjoint = dfx.BacksolveAdjoint(stepsize_controller=dfx.PIDController(
            rtol=1e-5, atol=1e-7, norm=dfx.adjoint_rms_seminorm))
    else:
        adjoint = dfx.BacksolveAdjoint()
    return dfx.diffeqsolve(terms, dfx.Tsit5(), 0.0, 1.0, None, d["y0"],
                           saveat=dfx.SaveAt(ts=d["ts"]), stepsize_controller=pid,
                           adjoint=adjoint)


def _loss(family, ys):
    """Sum of squares of the saved values for the analytic fields, their mean over
    the batch (times a weight of the order of a regression loss) for the MLPs."""
    loss = ys.square().sum()
    return loss if family == "vdp" else loss / (ys.shape[0] * ys.shape[-1])


def run(state):
    case = state["case"]
    if not case.get("grad", False):
        sol = _solve(state)
        return {"ts": sol.ts, "ys": sol.ys, "result": sol.result}
    sol = _solve(state)
    grads = torch.autograd.grad(_loss(case["family"], sol.ys), state["leaves"])
    return {"ys": sol.ys.detach(), "result": sol.result, "grads": list(grads)}


# ---------------------------------------------------------------------------
# Work that a pass cannot do without
# ---------------------------------------------------------------------------


def work(case):
    """Inputs read once and outputs written once; the operations of the solver's
    own field evaluations and stage arithmetic at the fewest steps that the
    tolerance takes (adaptive solves: the mean over these input distributions)."""
    B, family, grad = case["batch"], case["family"], case.get("grad", False)
    if family in ("vdp", "lv", "ou"):
        size = 8 if case.get("dtype") == "float64" else 4
        n_save = case.get("n_ts", 1)
        nbytes = B * (2 * size + n_save * (2 * size + 8) + 4)
        if family == "vdp":
            steps = 8.0 * 0.55 * case["t1"]
            nbytes += B * 12
        else:
            steps = 1.6 * case["t1"] if family == "lv" else case["n_steps"]
        flops = B * steps * (40 if family == "ou" else 186)
        if grad:
            nbytes += B * 12
            flops *= 3.5
        return {"bytes": nbytes, "flops": flops}
    w = WIDTHS[family]
    weights = sum(w[i] * w[i + 1] for i in range(3)) + (w[0] ** 2 if family == "nsde" else 0)
    params = weights + sum(w[1:]) + (w[0] if family == "nsde" else 0)
    n_save = 32 if family == "wide" else 1
    evals = 2 * case["n_steps"] if family == "nsde" else 25
    nbytes = B * (4 * w[0] + n_save * (4 * w[0] + 8) + 4) + 4 * params
    flops = 2.0 * weights * B * evals
    if grad:
        nbytes += B * 4 * w[0] + 4 * params
        # reverse solve over 31 segments of one step, f and both VJPs per stage; or
        # recompute and both VJPs of every forward stage
        flops += 2.0 * weights * B * (31 * 7 * 3 if family == "wide" else 3 * evals)
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# The same in 64 bits, as plain torch gives it
# ---------------------------------------------------------------------------

_C = (0.0, 1 / 5, 3 / 10, 4 / 5, 8 / 9, 1.0, 1.0)
_A = ((), (1 / 5,), (3 / 40, 9 / 40), (44 / 45, -56 / 15, 32 / 9),
      (19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729),
      (9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656),
      (35 / 384, 0.0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84))
_E = (71 / 57600, 0.0, -71 / 16695, 71 / 1920, -17253 / 339200, 22 / 525, -1 / 40)


def _adaptive64(f, y, span, h, rtol=1e-9, atol=1e-12):
    """y(span) from y(0) of the autonomous y' = f(y) to a tight tolerance, every
    row with steps of its own; also the rows' last step sizes."""
    t = torch.zeros_like(span)
    k0 = f(y)
    for n in range(200000):
        if n % 8 == 0 and bool((t >= span).all()):
            break
        left = span - t
        hh = torch.minimum(h, left)
        ks, col = [k0], hh[:, None]
        for i in range(1, 7):
            inc = sum(a * k for a, k in zip(_A[i], ks) if a)
            y1 = y + col * inc
            ks.append(f(y1))
        err = col * sum(e * k for e, k in zip(_E, ks) if e)
        scale = atol + rtol * torch.maximum(y.abs(), y1.abs())
        r = (err / scale).square().mean(1).sqrt()
        live = t < span
        ok = (r <= 1) & live
        t = torch.where(ok, torch.where(h >= left, span, t + hh), t)
        y = torch.where(ok[:, None], y1, y)
        k0 = torch.where(ok[:, None], ks[6], k0)
        grown = hh * (0.9 * r.clamp(min=1e-12) ** -0.2).clamp(0.2, 5.0)
        h = torch.where(live & ~((h >= left) & (r <= 1)), grown, h)
    return y, h


def _exact_vdp(case, d):
    y0, mu, t1 = d["y0"].double(), d["mu"].double()[:, 0], d["t1"]
    h = torch.full_like(t1, 1e-3)
    if not case["grad"]:
        def f(y):
            x, v = y[:, 0], y[:, 1]
            return torch.stack((v, mu * (1 - x * x) * v - x), 1)
        y, _ = _adaptive64(f, y0, t1, h)
        return {"ts": t1[:, None], "ys": y[:, None], "result": None}

    def f(z):  # the state, then its derivatives by x0, v0 and mu
        x, v = z[:, 0], z[:, 1]
        dx, dv = z[:, 2::2], z[:, 3::2]
        q = mu * (1 - x * x)
        force = torch.zeros_like(dv)
        force[:, 2] = (1 - x * x) * v
        ddv = (-2 * mu * x * v - 1)[:, None] * dx + q[:, None] * dv + force
        return torch.cat((torch.stack((v, q * v - x), 1),
                          torch.stack((dv, ddv), 2).reshape(-1, 6)), 1)
    z0 = torch.zeros(len(t1), 8, dtype=torch.float64, device=DEV)
    z0[:, :2] = y0
    z0[:, 2] = z0[:, 5] = 1.0
    z, _ = _adaptive64(f, z0, t1, h)
    y, s = z[:, :2], z[:, 2:].reshape(-1, 3, 2)
    g = 2 * (s * y[:, None]).sum(2)
    return {"ys": y[:, None], "result": None, "grads": [g[:, :2], g[:, 2:]]}


def _exact_lv(case, d):
    a, b, c, e = d["args"].double().tolist()

    def f(y):
        x, v = y[:, 0], y[:, 1]
        return torch.stack((a * x - b * x * v, -c * v + e * x * v), 1)
    y = d["y0"].double()
    h = torch.full((len(y),), 0.05, dtype=torch.float64, device=DEV)
    out, t = [], 0.0
    for u in d["ts"].tolist():
        y, h = _adaptive64(f, y, torch.full_like(h, u - t), h)
        out.append(y)
        t = u
    return {"ts": d["ts"].expand(len(y), -1), "ys": torch.stack(out, 1), "result": None}


def _philox(counter, key):
    """Philox4x32-10 of four int64 tensors that hold 32-bit words."""
    m32 = 0xFFFFFFFF
    c0, c1, c2, c3 = counter
    k0, k1 = key & m32, (key >> 32) & m32
    for _ in range(10):
        p, q = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = (((q >> 32) & m32) ^ c1 ^ k0, q & m32, ((p >> 32) & m32) ^ c3 ^ k1,
                          p & m32)
        k0, k1 = (k0 + 0x9E3779B9) & m32, (k1 + 0xBB67AE85) & m32
    return c0, c1, c2, c3


def _tree_normals(B, dim, key, node, kind):
    """The [B, dim] normals of one node of the trajectories' Brownian trees."""
    quads = (dim + 3) // 4
    traj = torch.arange(B, device=DEV)[:, None].expand(B, quads)
    quad = torch.arange(quads, device=DEV)[None, :].expand(B, quads)
    c = _philox((traj, torch.full_like(traj, node), quad + (kind << 24),
                 torch.full_like(traj, 0x5EED)), key)
    out = []
    for p in (0, 2):
        u = ((c[p] >> 8).double() + 0.5) / 16777216.0
        v = ((c[p + 1] >> 8).double() + 0.5) / 16777216.0
        rad = (-2 * u.log()).sqrt()
        out += [rad * torch.cos(2 * math.pi * v), rad * torch.sin(2 * math.pi * v)]
    return torch.stack(out, 2).reshape(B, 4 * quads)[:, :dim]


def _brownian(B, dim, key, r, tol):
    """W(r) on the unit interval by bridge descent to intervals of at most tol."""
    lo, width, node = 0.0, 1.0, 1
    w_lo = torch.zeros(B, dim, dtype=torch.float64, device=DEV)
    dw = _tree_normals(B, dim, key, 0, 0)
    while width > tol:
        mid = lo + width / 2
        bridge = math.sqrt(width) / 2 * _tree_normals(B, dim, key, node, 1)
        right = r > mid
        if right:
            w_lo, dw, lo = w_lo + dw / 2 + bridge, dw / 2 - bridge, mid
        else:
            dw = dw / 2 + bridge
        node, width = 2 * node + int(right), width / 2
    a, b = max(r - lo, 0.0), max(width - max(r - lo, 0.0), 0.0)
    return w_lo + a / width * dw + math.sqrt(a * b / width) * _tree_normals(B, dim, key, node, 2)


def _heun64(case, d, y, f, g):
    """Heun's method on the case's grid and Brownian paths; g = 0 on none."""
    n, (B, dim), w = case["n_steps"], y.shape, None
    for i in range(n + 1):
        # a path is looked up at the FP32 value of its time
        r = float(torch.tensor(i / n, dtype=torch.float64).float())
        with torch.no_grad():
            w1 = _brownian(B, dim, d["key"], r, 1e-3)
        if i:
            h, dw = 1.0 / n, w1 - w
            k0 = f(y) * h + g(y) * dw
            y = y + 0.5 * (k0 + f(y + k0) * h + g(y + k0) * dw)
        w = w1
    return y


def _exact_ou(case, d):
    theta, mu, sigma = d["args"].double().tolist()
    y = _heun64(case, d, d["y0"].double(), lambda y: theta * (mu - y), lambda y: sigma)
    return {"ts": torch.ones(len(y), 1, dtype=torch.float64, device=DEV), "ys": y[:, None],
            "result": None}


def _exact_mlp(case, d):
    family, grad = case["family"], case["grad"]
    W, b = [x.double() for x in d["W"]], [x.double() for x in d["b"]]
    y0 = d["y0"].double()
    leaves = [y0, *W, *b]

    def f(y):
        h = torch.tanh(torch.addmm(b[0], y, W[0].t()))
        h = torch.tanh(torch.addmm(b[1], h, W[1].t()))
        return torch.addmm(b[2], h, W[2].t())
    if family == "nsde":
        Ws, bs = d["Ws"].double(), d["bs"].double()
        leaves += [Ws, bs]
    for x in leaves:
        x.requires_grad_(grad)
    with torch.set_grad_enabled(grad):
        if family == "nsde":
            ys = _heun64(case, d, y0, f,
                         lambda y: 0.1 * torch.tanh(torch.addmm(bs, y, Ws.t())))[:, None]
        else:  # classical Runge-Kutta steps far below the tolerance
            n = 62
            y, h, saved = y0, 1.0 / n, [y0]
            for i in range(n):
                k1 = f(y)
                k2 = f(y + 0.5 * h * k1)
                k3 = f(y + 0.5 * h * k2)
                k4 = f(y + h * k3)
                y = y + (h / 6) * (k1 + 2 * k2 + 2 * k3 + k4)
                if i % 2:
                    saved.append(y)
            ys = torch.stack(saved, 1) if family == "wide" else y[:, None]
        if grad:
            grads = torch.autograd.grad(_loss(family, ys), leaves)
            return {"ys": ys.detach(), "result": None, "grads": list(grads)}
    ts = d["ts"] if family == "wide" else torch.ones(1, dtype=torch.float64, device=DEV)
    return {"ts": ts.expand(len(y0), -1), "ys": ys, "result": None}


def exact(case, seed):
    d = _inputs(case, seed)
    return {"vdp": _exact_vdp, "lv": _exact_lv, "ou": _exact_ou}.get(
        case["family"], _exact_mlp)(case, d)
