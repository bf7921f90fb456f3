"""Performance cases: what programs built on henon_map_cpp_b200 have it do.

Every case is a dict of plain values; `kind` names the entry points that it
goes through and the rest are its sizes and options.  `prepare` builds what
a program holds before the call (the tracker with its modulation tables,
constructs, initial conditions), `run` makes one pass through the public
API, `work` counts the operations that a pass cannot do without, and `exact`
restates a pass in plain torch where that is quick enough.

A tracker's turn budget counts a particle set's turns for good (reset() does
not give them back), so a pass creates its particle set, as the programs do.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import henon_map_cpp_b200 as hm
from henon_map_cpp_b200 import _capi as C
from henon_map_cpp_b200 import autograd, sweep

TUNES = (0.168, 0.201)
BARRIER = 10.0
WINDOWS = 13  # log-spaced indicator windows
GHOST_MODULE = 1e-6
SPS = ((1.000e-4, 1), (0.218e-4, 2), (0.708e-4, 3), (0.254e-4, 6), (0.100e-4, 7), (0.078e-4, 10),
       (0.218e-4, 12))


def listed():
    return [
        # The per-turn construct loop of the notebooks: one call per
        # construct and turn on a small set; launches and host time count.
        dict(name="construct_loop", kind="loop", n=1000, turns=40, epsilon=32.0, mu=0.0,
             extent=0.4),
        # Survival of an unmodulated 100 x 100 grid through the facade: a
        # quick look at a working point, bound by the turns' latency.
        dict(name="survival_small", kind="track", n=10_000, turns=10_000, epsilon=0.0, mu=0.0,
             extent=0.5, arith="exact", kick=0.0, back=0),
        # Forward tracking and backward tracking of an odd-sized set with the
        # octupole: reversibility checks.
        dict(name="there_and_back", kind="track", n=17_711, turns=5_000, epsilon=16.0, mu=0.2,
             extent=0.3, arith="exact", kick=0.0, back=4_000),
        # The dynamic-aperture scan at full size, host arrays in and out.
        dict(name="aperture_scan", kind="track", n=1_048_576, turns=100_000, epsilon=16.0, mu=0.2,
             extent=0.6, arith="exact", kick=0.0, back=0),
        # The same scan in fast arithmetic on device arrays, odd-sized.
        dict(name="aperture_scan_fast", kind="device", n=491_401, turns=100_000, epsilon=64.0,
             mu=0.0, extent=0.6, arith="fast"),
        # The long horizon of the scan on a coarse grid: few chains, many turns.
        dict(name="long_horizon", kind="device", n=40_000, turns=1_000_000, epsilon=1.0, mu=0.0,
             extent=0.5, arith="exact"),
        # Tracking with a random kick every turn (noise studies).
        dict(name="noise", kind="track", n=262_144, turns=4_000, epsilon=16.0, mu=0.2, extent=0.4,
             arith="exact", kick=1e-5, back=0),
        # All the indicators of the modulated grid in one fused call.
        dict(name="indicators", kind="indicators", n=65_025, turns=10_000, epsilon=32.0, mu=0.0,
             extent=0.4),
        # Displacement Lyapunov estimate with two ghosts per particle.
        dict(name="ghost_lyapunov", kind="ghost", n=65_536, turns=2_000, every=10, epsilon=16.0,
             mu=0.2, extent=0.4),
        # Birkhoff and FFT tunes over windows of the orbit: a smooth full
        # orbit and ragged windows.
        dict(name="tunes", kind="tunes", n=16_384, turns=10_000, cut1=1_000, cut2=5_000,
             epsilon=16.0, mu=0.0, extent=0.4),
        # Gradient of the orbit loss with respect to the initial conditions
        # and the parameters, forward and backward, as an optimiser calls it.
        dict(name="orbit_loss", kind="loss", n=65_536, turns=10_000, every=100, epsilon=16.0,
             mu=0.1, extent=0.3),
        # A sweep of mixed-size parameter sets as one batch, set-up included.
        dict(name="sweep", kind="sweep", sets=64, n_min=1_000, n_max=64_000, t_min=1_000,
             t_max=200_000),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the listed kinds; sizes over the same ranges."""
    kind = rng.choice(("loop", "track", "track", "track", "device", "device", "noise",
                       "indicators", "ghost", "tunes", "loss", "sweep"))
    eps = rng.choice((0.0, 1.0, 16.0, 32.0, 64.0))
    mu = rng.choice((0.0, 0.2))
    extent = rng.choice((0.3, 0.4, 0.5, 0.6))
    if kind == "loop":
        return dict(kind="loop", n=_log_int(rng, 64, 20_000), turns=_log_int(rng, 5, 100),
                    epsilon=eps, mu=mu, extent=0.4)
    if kind == "track":
        n = _log_int(rng, 500, 1_000_000)
        turns = _log_int(rng, 500, min(200_000, int(5e10 / n)))
        back = rng.choice((0, 0, turns // 2))
        return dict(kind="track", n=n, turns=turns, epsilon=eps, mu=mu, extent=extent,
                    arith=rng.choice(("exact", "exact", "fast")), kick=0.0, back=back)
    if kind == "device":
        n = _log_int(rng, 500, 1_000_000)
        return dict(kind="device", n=n, turns=_log_int(rng, 500, min(500_000, int(5e10 / n))),
                    epsilon=eps, mu=mu, extent=extent, arith=rng.choice(("exact", "fast")))
    if kind == "noise":
        n = _log_int(rng, 1_000, 300_000)
        return dict(kind="track", n=n, turns=_log_int(rng, 200, min(10_000, int(1e9 / n))),
                    epsilon=eps, mu=mu, extent=0.4, arith="exact", kick=rng.choice((1e-6, 1e-4)),
                    back=0)
    if kind == "indicators":
        return dict(kind="indicators", n=_log_int(rng, 500, 65_000), turns=_log_int(rng, 400, 8_000),
                    epsilon=eps, mu=mu, extent=0.4)
    if kind == "ghost":
        every = rng.choice((1, 5, 10, 17))
        return dict(kind="ghost", n=_log_int(rng, 1_000, 100_000),
                    turns=every * rng.randint(20, 150), every=every, epsilon=eps, mu=mu, extent=0.4)
    if kind == "tunes":
        turns = _log_int(rng, 500, 10_000)
        cut1 = rng.randint(100, turns // 2)
        return dict(kind="tunes", n=_log_int(rng, 500, 16_000), turns=turns, cut1=cut1,
                    cut2=rng.randint(cut1 + 50, turns), epsilon=eps, mu=mu, extent=0.4)
    if kind == "loss":
        return dict(kind="loss", n=_log_int(rng, 1_000, 65_000), turns=_log_int(rng, 500, 10_000),
                    every=100, epsilon=16.0, mu=rng.choice((0.0, 0.1)), extent=0.3)
    return dict(kind="sweep", sets=rng.randint(4, 64), n_min=1_000,
                n_max=_log_int(rng, 4_000, 64_000), t_min=1_000, t_max=_log_int(rng, 10_000, 200_000))


# ---- inputs ----------------------------------------------------------------------

def _start(case, seed):
    """Initial conditions (x, px, y, py) on the host: points of [0, extent]^2
    with px = py = 0 (the scans' grids); each seed has another grid, slightly
    smaller and shifted."""
    rng = np.random.default_rng(1000 + seed)
    n = case["n"]
    side = math.isqrt(n - 1) + 1
    v = np.linspace(0.0, case["extent"] * (1 - 0.05 * rng.uniform()), side)
    x, y = np.meshgrid(v, v)
    x = x.ravel()[:n] + 1e-3 * rng.uniform()
    y = y.ravel()[:n] + 1e-3 * rng.uniform()
    return x, np.zeros(n), y, np.zeros(n)


def _windows(turns):
    lo = max(2.0, turns / 100)
    return sorted({int(round(w)) for w in np.geomspace(lo, turns, WINDOWS)})


def _constructs(case):
    n, wins = case["n"], _windows(case["turns"])
    return dict(matrix=hm.matrix_4d_vector(n), old=hm.matrix_4d_vector(n),
                jac=hm.matrix_4d_vector(n), megno=hm.megno_construct(n),
                megno_b=hm.megno_birkhoff_construct(n, wins),
                vectors=hm.vector_4d(np.tile([1.0, 0.0, 0.0, 0.0], (n, 1))),
                lyapunov=hm.lyapunov_birkhoff_construct_multi(n, wins),
                tune=hm.tune_birkhoff_construct(n, [max(1, w // 2) for w in wins]))


def prepare(case, seed):
    kind = case["kind"]
    s = dict(case=case)
    if kind == "sweep":
        # the case's particle counts and turn budgets; tunes, modulation,
        # octupole and points from the seed
        rng = np.random.default_rng(1000 + seed)
        span = lambda lo, hi, u: int(round(lo * (hi / lo) ** u))  # noqa: E731
        sizes = np.random.default_rng(7).uniform(size=(case["sets"], 2))
        s["sets"] = [dict(omega_x=rng.uniform(0.15, 0.32), omega_y=rng.uniform(0.15, 0.32),
                          epsilon=rng.uniform(0.0, 64.0), mu=rng.uniform(-0.5, 0.5),
                          n_particles=span(case["n_min"], case["n_max"], u),
                          n_turns=span(case["t_min"], case["t_max"], v), barrier=BARRIER)
                     for u, v in sizes]
        points = [sweep.ball_points(rng, k["n_particles"], 0.6) for k in s["sets"]]
        s["coords"] = tuple(np.concatenate([p[q] for p in points]) for q in range(4))
        return s
    if kind == "loss":
        rng = np.random.default_rng(1000 + seed)
        n = case["n"]
        pts = (rng.uniform(0, case["extent"], n), rng.normal(0, 0.01, n),
               rng.uniform(0, case["extent"], n), rng.normal(0, 0.01, n))
        s["leaves"] = [torch.tensor(p, device="cuda", requires_grad=True) for p in pts]
        # an optimiser moves the parameters a little from step to step
        s["leaves"].append(torch.tensor(
            [2 * math.pi * TUNES[0], 2 * math.pi * TUNES[1],
             case["epsilon"] + 1e-3 * rng.uniform(), case["mu"]],
            dtype=torch.float64, requires_grad=True))
        return s
    s["start"] = _start(case, seed)
    s["seed"] = seed
    turns = case["turns"]
    if kind == "device":
        s["tracker"] = C.Tracker(turns, *TUNES, "sps", float("nan"), case["epsilon"], 0)
        s["tracker"].arith = C.ARITH_FAST if case["arith"] == "fast" else C.ARITH_EXACT
        s["start"] = [torch.from_numpy(a).cuda() for a in s["start"]]
        s["now"] = [torch.empty_like(a) for a in s["start"]]
        s["steps"] = torch.empty(case["n"], dtype=torch.int32, device="cuda")
        s["work"] = torch.empty(C.load().hm_track_workspace_bytes(case["n"]), dtype=torch.uint8,
                                device="cuda")
        return s
    s["tracker"] = hm.henon_tracker(turns + 1, *TUNES, "sps", epsilon=case["epsilon"])
    if kind == "track":
        s["tracker"].set_arith(case["arith"])
    if kind in ("loop", "indicators"):
        s.update(_constructs(case))
    return s


# ---- one pass --------------------------------------------------------------------

def _state_of(p):
    return dict(x=p.get_x(), px=p.get_px(), y=p.get_y(), py=p.get_py(), steps=p.get_steps())


def _reset(s):
    for k in ("matrix", "old", "jac", "megno", "megno_b", "lyapunov", "tune"):
        s[k].reset()
    s["vectors"].set_vectors(np.array([1.0, 0.0, 0.0, 0.0]))


def _values(s, p):
    return dict(_state_of(p), matrix=s["matrix"].get_matrix(), megno=s["megno"].get_values(),
                megno_b=s["megno_b"].get_values(), vectors=s["vectors"].get_vectors(),
                ly_raw=s["lyapunov"].get_values_raw(), ly_b=s["lyapunov"].get_values_b(),
                t1x=s["tune"].get_tune1_x(), t1y=s["tune"].get_tune1_y(),
                t2x=s["tune"].get_tune2_x(), t2y=s["tune"].get_tune2_y())


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "sweep":
        out = sweep.run_sweep(s["sets"], s["coords"])
        return {k: np.concatenate([r[k] for r in out]) for k in ("x", "px", "y", "py", "steps")}
    if kind == "loss":
        *xs, theta = s["leaves"]
        for leaf in s["leaves"]:
            leaf.grad = None
        loss = autograd.orbit_loss(*xs, theta, n_turns=case["turns"], barrier=BARRIER,
                                   checkpoint_every=case["every"])
        loss.backward()
        return dict(loss=loss.detach(), grads=[leaf.grad for leaf in s["leaves"]])
    mu, turns = case["mu"], case["turns"]
    if kind == "device":
        for now, start in zip(s["now"], s["start"]):
            now.copy_(start)
        s["steps"].zero_()
        C.call("hm_track_device", *[a.data_ptr() for a in s["now"]], s["steps"].data_ptr(),
               case["n"], s["tracker"].device_tables(), turns, 0, turns, mu, BARRIER, 0,
               s["tracker"].arith, s["work"].data_ptr(),
               ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        return dict(zip(("x", "px", "y", "py"), s["now"]), steps=s["steps"])
    p = hm.particles(*s["start"])
    tracker = s["tracker"]
    if kind == "track":
        if case["kick"]:
            p.kick_seed = s["seed"]
        tracker.track(p, turns, mu, BARRIER, case["kick"] or np.nan)
        out = _state_of(p)
        if case["back"]:
            tracker.track(p, case["back"], mu, BARRIER, inverse=True)
            out = dict(there=out, back=_state_of(p))
        return out
    if kind == "ghost":
        p.add_ghost(GHOST_MODULE, "x")
        p.add_ghost(GHOST_MODULE, "y")
        lyap = tracker.track_ghost_lyapunov(p, turns // case["every"], case["every"], mu,
                                            GHOST_MODULE, BARRIER)
        return dict(_state_of(p), lyapunov=lyap)
    if kind == "tunes":
        frame = tracker.tune_all(p, turns, mu, BARRIER,
                                 from_idx=np.array([0, case["cut1"], case["cut2"]]),
                                 to_idx=np.array([case["cut1"], case["cut2"], turns]))
        cols = ("tune_x_birkhoff", "tune_y_birkhoff", "tune_x_fft", "tune_y_fft")
        return dict({c: [np.asarray(v) for v in frame[c]] for c in cols}, state=_state_of(p))
    _reset(s)
    s["tune"].first_add(p)
    if kind == "indicators":
        samples = tracker.track_indicators(
            p, turns, mu, BARRIER, matrix=s["matrix"], megno=s["megno"],
            megno_birkhoff=s["megno_b"], vectors=s["vectors"], lyapunov=s["lyapunov"],
            tune=s["tune"], megno_sample_turns=_windows(turns))
        return dict(_values(s, p), samples=samples)
    for _ in range(turns):  # the notebooks' loop
        s["old"].explicit_copy(s["matrix"])
        tracker.track(p, 1, mu, BARRIER)
        s["matrix"].structured_multiply(tracker, p, mu)
        s["megno"].add(s["matrix"], s["old"])
        s["megno_b"].add(s["matrix"], s["old"])
        s["jac"].set_with_tracker(tracker, p, mu)
        s["vectors"].multiply(s["jac"])
        s["lyapunov"].add(s["vectors"])
        s["vectors"].normalize()
        s["tune"].add(p)
    return _values(s, p)


# ---- what a pass cannot do without -------------------------------------------------

def _map_flops(mu):
    return 42.0 if mu else 26.0  # every *, + and - of one particle-turn


def work(case):
    """Operations of one pass.  Particles lost on the way stop costing turns:
    about half of the turns of a scan of [0, 0.6]^2 are run, nearly all on
    [0, 0.4]^2."""
    kind = case["kind"]
    if kind == "sweep":
        ln = lambda lo, hi: (hi - lo) / math.log(hi / lo)  # noqa: E731  mean of a log-uniform
        n, t = ln(case["n_min"], case["n_max"]), ln(case["t_min"], case["t_max"])
        return dict(bytes=case["sets"] * (n * 68 + t * 32), flops=0.35 * case["sets"] * n * t * 42)
    n, turns = float(case["n"]), float(case["turns"])
    io = n * 68 + turns * 32  # coordinates in and out, steps, the turn records
    kept = {0.3: 0.95, 0.4: 0.9, 0.5: 0.7, 0.6: 0.55}[case["extent"]]
    per_turn = _map_flops(case["mu"])
    if kind in ("track", "device"):
        turns += case.get("back", 0)
        if case.get("kick"):
            per_turn += 60  # a uniform direction and the kick
        return dict(bytes=io, flops=kept * n * turns * per_turn)
    if kind == "ghost":
        return dict(bytes=3 * io, flops=kept * n * (3 * turns * per_turn
                                                    + 2 * turns / case["every"] * 60))
    if kind == "loss":
        # forward turn with the loss, reverse turn with the gradients, and the
        # checkpoints written and read once
        return dict(bytes=io + n * 64 + 64 * n * turns / case["every"],
                    flops=kept * n * turns * (per_turn + 8 + 90))
    wins = len(_windows(case["turns"]))
    if kind == "tunes":
        spans = (case["cut1"], case["cut2"] - case["cut1"], case["turns"] - case["cut2"],
                 case["turns"])
        fft = 2 * sum(5.0 * m * math.log2(max(2, m)) for m in spans)
        return dict(bytes=io + n * 128, flops=n * (turns * per_turn + 2 * turns * 40 + fft))
    # indicators: DF, DF.M, the norm, v <- DF v, log10, log, two atan2 and the
    # open windows' sums
    return dict(bytes=io + n * (256 + 64 + 8 * 9 * wins),
                flops=kept * n * turns * (per_turn + 24 + 128 + 33 + 32 + 8 + 4 * 25 + 20))


# ---- the same in plain torch, in 64 bits ---------------------------------------------

def _angles(turns, case, seed=0):
    """(sin, cos) of omega_x(n) and omega_y(n), from the C library."""
    two_pi = 2 * math.pi
    base = two_pi / 868.12
    rows = []
    for n in range(turns):
        ripple = 0.0
        for c, k in SPS:
            ripple += c * math.cos(k * base * n)
        w = [two_pi * t * (1 + case["epsilon"] * ripple) for t in TUNES]
        rows.append((math.sin(w[0]), math.cos(w[0]), math.sin(w[1]), math.cos(w[1])))
    return rows


def _turn(x, px, y, py, a, mu):
    sx, cx, sy, cy = a
    xx, yy = x * x, y * y
    px = px + (xx - yy)
    py = py + (-2.0 * x) * y
    if mu:
        px, py = (px + mu * (xx * x - ((3.0 * y) * y) * x),
                  py + mu * (yy * y - ((3.0 * x) * x) * y))
    return x * cx + px * sx, -x * sx + px * cx, y * cy + py * sy, -y * sy + py * cy


def _turn_back(x, px, y, py, a, mu):
    sx, cx, sy, cy = a
    x, px = x * cx - px * sx, x * sx + px * cx
    y, py = y * cy - py * sy, y * sy + py * cy
    xx, yy = x * x, y * y
    if mu:
        px, py = (px - mu * (xx * x - ((3.0 * y) * y) * x),
                  py - mu * (yy * y - ((3.0 * x) * x) * y))
    return x, px - (xx - yy), y, py - (-2.0 * x) * y


def _inside(x, px, y, py):
    return (x * x + px * px) + (y * y + py * py) < BARRIER * BARRIER


class _Orbit:
    """Tracked points; lost ones become NaN and keep their turns."""

    def __init__(self, start):
        self.c = [torch.as_tensor(a, device="cuda") for a in start]
        self.steps = torch.zeros(len(start[0]), dtype=torch.int64, device="cuda")

    def turn(self, a, mu, back=False):
        c = (_turn_back if back else _turn)(*self.c, a, mu)
        keep = _inside(*c)
        self.c = [torch.where(keep, v, math.nan) for v in c]
        self.steps += torch.where(keep, -1 if back else 1, 0)

    def state(self):
        return dict(zip(("x", "px", "y", "py"), self.c), steps=None)


def _weights(n):
    t = torch.arange(n, dtype=torch.float64, device="cuda") / n
    w = torch.exp(-1 / (t * (1 - t)))
    return w / w.sum()


def _exact_track(case, start):
    o, a = _Orbit(start), _angles(case["turns"], case)
    for t in a:
        o.turn(t, case["mu"])
    out = o.state()
    if case["back"]:
        for k in range(case["back"]):
            o.turn(a[case["turns"] - 1 - k], case["mu"], back=True)
        out = dict(there=out, back=o.state())
    return out


def _exact_constructs(case, start):
    o, a = _Orbit(start), _angles(case["turns"] + 1, case)
    n, mu, wins = case["n"], case["mu"], _windows(case["turns"])
    new = lambda *shape: torch.zeros(*shape, n, dtype=torch.float64, device="cuda")  # noqa: E731
    M = torch.eye(4, dtype=torch.float64, device="cuda")[:, :, None].expand(4, 4, n).clone()
    v = new(4)
    v[0] = 1.0
    norm = M.square().sum((0, 1)).sqrt()
    l1, l2, l3, b1 = new(), new(), new(), new()
    mb, raw, lb = new(len(wins)), new(len(wins)), new(len(wins))
    tw = [max(1, w // 2) for w in wins]
    t1, t2 = new(2, len(wins)), new(2, len(wins))
    pad = lambda w: torch.nn.functional.pad(_weights(w), (0, case["turns"] + 2 - w))  # noqa: E731
    w_ly = torch.stack([pad(w) for w in wins])
    w_t1 = torch.stack([pad(w) for w in tw])
    w_t2 = torch.stack([torch.roll(pad(w), w) for w in tw])
    idx = torch.arange(case["turns"] + 2, device="cuda")[None, :]
    over = lambda w: torch.tensor(w, device="cuda")[:, None]  # noqa: E731
    in_ly, in_mb = idx < over(wins), idx <= over(wins)
    in_t1, in_t2 = idx < over(tw), (idx >= over(tw)) & (idx < 2 * over(tw))
    lens = over(wins).double()
    angle = torch.stack([torch.atan2(o.c[1], o.c[0]), torch.atan2(o.c[3], o.c[2])])
    samples = []
    add = lambda acc, live, term: torch.where(live[:, None], acc + term, acc)  # noqa: E731
    for k in range(case["turns"]):
        o.turn(a[k], mu)
        x, y = o.c[0], o.c[2]
        sx, cx, sy, cy = a[k + 1]
        da = 2 * x + 3 * mu * (x * x - y * y)
        db = -2 * y - 6 * mu * x * y
        rows = ((cx + sx * da, sx, sx * db, 0.0), (-sx + cx * da, cx, cx * db, 0.0),
                (sy * db, 0.0, cy - sy * da, sy), (cy * db, 0.0, -sy - cy * da, cy))
        # a lost point's whole matrix is NaN: 0 * NaN
        apply = lambda m: torch.stack([sum(r[q] * m[q] for q in range(4)) for r in rows])  # noqa: E731
        M = apply(M)
        old, norm = norm, M.square().sum((0, 1)).sqrt()
        lr = torch.log10(norm / old)
        i = float(k + 1)
        l1 = l1 + lr * i
        l2 = l2 + l1 / i
        l3 = l2 / i
        if k + 1 in wins:
            samples.append(l3)
        b1 = b1 + lr * i
        mb = add(mb, in_mb[:, k + 1], b1 * w_ly[:, k, None] / i)
        v = apply(v)
        nv = v.square().sum(0).sqrt()
        lv = torch.log(nv)
        raw = add(raw, in_ly[:, k], lv / lens)
        lb = add(lb, in_ly[:, k], lv * w_ly[:, k, None])
        v = v / nv
        now = torch.stack([torch.atan2(o.c[1], x), torch.atan2(o.c[3], y)])
        d = now - angle
        d = torch.where(d > 0, d, d + 2 * math.pi)
        angle = now
        for plane in range(2):
            t1[plane] = add(t1[plane], in_t1[:, k + 1], d[plane] * w_t1[:, k + 1, None])
            t2[plane] = add(t2[plane], in_t2[:, k + 1], d[plane] * w_t2[:, k + 1, None])
    s = dict(o.state(), matrix=M.permute(2, 0, 1), megno=l3, megno_b=mb, vectors=v.T, ly_raw=raw,
             ly_b=lb)
    # the construct's tunes are read out by its own convention
    s.update(t1x=None, t1y=None, t2x=None, t2y=None)
    if case["kind"] == "indicators":
        s["samples"] = torch.stack(samples)
    return s


def _exact_ghost(case, start):
    n, mu = case["n"], case["mu"]
    c = [np.tile(a, 3) for a in start]
    c[0][n:2 * n] += GHOST_MODULE
    c[2][2 * n:] += GHOST_MODULE
    o, a = _Orbit(c), _angles(case["turns"], case)
    lyap = torch.zeros(2, n, dtype=torch.float64, device="cuda")
    for k, t in enumerate(a):
        o.turn(t, mu)
        if (k + 1) % case["every"] == 0:
            base = torch.stack([v[:n] for v in o.c])
            for g in range(2):
                cut = slice((1 + g) * n, (2 + g) * n)
                off = torch.stack([v[cut] for v in o.c]) - base
                d = off.square().sum(0).sqrt()
                lyap[g] += torch.log(d / GHOST_MODULE)
                moved = base + off * (GHOST_MODULE / d)
                for q in range(4):
                    o.c[q][cut] = moved[q]
    # the displacements are small differences: the coordinates of the ghosts
    # and the sums are as sensitive as the orbit, so only the base is exact
    return dict({k: None for k in ("x", "px", "y", "py", "steps")}, lyapunov=lyap.T)


def _interpolated_peak(z):
    """Peak of |FFT| over the last axis, interpolated between its neighbours."""
    m = torch.fft.fft(z).abs()
    n = m.shape[1]
    at = m.argmax(1)
    ends = (at == 0) | (at == n - 1)
    k = at.clamp(1, n - 2)
    get = lambda j: m.gather(1, j[:, None])[:, 0]  # noqa: E731
    k = torch.where(get(k - 1) > get(k + 1), k - 1, k)
    a, b, c = get(k), get(k + 1), math.cos(2 * math.pi / n)
    root = torch.sqrt(c * c * (a + b) ** 2 - 2 * a * b * (2 * c * c - c - 1))
    A = (-(a + b * c) * (a - b) + b * root) / (a * a + b * b + 2 * a * b * c)
    v = (1 - (k / n + torch.asin(A * math.sin(2 * math.pi / n)) / (2 * math.pi))).abs()
    return torch.where(ends, torch.where(at == 0, 1.0, 0.0).double(), v)


def _exact_tunes(case, start):
    o, turns = _Orbit(start), case["turns"]
    orbit = torch.empty(turns + 1, 4, case["n"], dtype=torch.float64, device="cuda")
    orbit[0] = torch.stack(o.c)
    for k, t in enumerate(_angles(turns, case)):
        o.turn(t, case["mu"])
        orbit[k + 1] = torch.stack(o.c)
    orbit -= orbit.mean(0)
    cuts = (0, case["cut1"], case["cut2"], turns)
    wins = list(zip(cuts[:3], cuts[1:])) + [None]
    out = {c: [] for c in ("tune_x_birkhoff", "tune_y_birkhoff", "tune_x_fft", "tune_y_fft")}
    for w in wins:
        for plane, q in (("x", 0), ("y", 2)):
            f, t = w or (0, turns)
            part = orbit[f:t + 1, q:q + 2]
            theta = torch.atan2(part[:, 1], part[:, 0])
            d = theta[1:] - theta[:-1]
            d = torch.where(d < 0, d + 2 * math.pi, d)
            out[f"tune_{plane}_birkhoff"].append(
                1 - (_weights(t - f)[:, None] * d).sum(0) / (2 * math.pi))
            if w is None:
                part = orbit[1:, q:q + 2]
            m = part.shape[0]
            hann = 2 * torch.sin(math.pi * torch.arange(m, dtype=torch.float64,
                                                       device="cuda") / m) ** 2
            peaks = []
            for some in torch.split(part, 2048, dim=2):
                z = torch.complex(some[:, 0] * hann[:, None], some[:, 1] * hann[:, None]).T
                peak = _interpolated_peak(torch.nan_to_num(z).contiguous())
                peaks.append(torch.where(z.isnan().any(1), math.nan, peak))
            out[f"tune_{plane}_fft"].append(torch.cat(peaks))
    return dict(out, state=o.state())


def exact(case, seed):
    """The pass in plain torch.  Orbits repeat the map's own order of
    operations, so chaotic ones agree as well; what amplifies rounding beyond
    that (gradients through chaos) has no value."""
    kind = case["kind"]
    if kind not in ("track", "loop", "indicators", "ghost", "tunes") or case["turns"] > 10_000:
        return None
    if kind == "track" and (case["kick"] or case["arith"] != "exact" or case["n"] > 200_000):
        return None
    start = _start(case, seed)
    if kind == "track":
        return _exact_track(case, start)
    if kind == "ghost":
        return _exact_ghost(case, start)
    if kind == "tunes":
        return _exact_tunes(case, start)
    return _exact_constructs(case, start)
