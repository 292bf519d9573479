"""The work that programs give this particle-filter engine, as cases to time.

A case is a dict of plain values; prepare() builds what such a program keeps
between calls (filters, device arrays of inputs and estimates, host records),
run() makes one pass through the public entry points, work() counts what the
pass cannot do without.

Every trace is periodic: the ground truth returns to its start after `period`
steps, so a filter can be stepped for as long as wanted and keeps tracking
(the inputs wrap around at the array's end).

Kinds of pass:
  step      pf_step, one host input in and one host estimate out per call
  submit    pf_step_submit / pf_step_collect: the pipelined form of the same
  run       pf_run_device: inputs and estimates in device memory, one graph
            replay per step; optionally the particles read back at the end
  batch     pf_batch_submit: many filters of uneven sizes, one period of steps
  serve     pf_server_update / launch / poll: resident filters of two models,
            an update of each one per round
  estimate  pfk_estimate_noalloc: the posterior estimate of particles and
            weights that the caller holds in device memory
"""
import math

import numpy as np
import torch

import esthera_b200 as E

UNICYCLE, DHARM, REFARM, BEACON, CAMARM = 0, 1, 2, 3, 4
STATE = {UNICYCLE: 3, DHARM: 12, REFARM: 9, BEACON: 3, CAMARM: 9}
NOISE = {UNICYCLE: 3, DHARM: 6, REFARM: 9, BEACON: 3, CAMARM: 9}
NONE, RING, TORUS, ALL2ALL = 0, 1, 2, 3
REFERENCE, SYSTEMATIC, VOSE = 0, 1, 2
FUSED, PHASED, SPLIT = 0, 1, 2
EST_WORDS = 27  # 8-byte words of one estimate record


def filter_case(name, kind, model, m, n, t, exchange, resampler, steps, **more):
    c = {"name": name, "kind": kind, "model": model, "m": m, "n": n, "t": t, "exchange": exchange,
         "resampler": resampler, "steps": steps, "pipeline": SPLIT, "reference_rng": False, "linear": False,
         "freq": 1.0, "ess": 0.0, "period": 64, "particles": False}
    c.update(more)
    return c


def listed():
    return [
        # a robot's own pose filter: 4096 particles as 8 sub-filters of 512, no exchange, one
        # synchronous call per sensor reading -- launches and copies are most of it
        filter_case("step_unicycle_4k", "step", UNICYCLE, 512, 8, 0, NONE, SYSTEMATIC, 8),
        # a mid-size tracker fed from the host as readings arrive, calls not waited for one by one
        filter_case("submit_unicycle_64k", "submit", UNICYCLE, 256, 256, 2, TORUS, SYSTEMATIC, 32),
        # an offline run over a recorded trace with an odd number of sub-filters; the particle
        # cloud is read back at the end
        filter_case("run_unicycle_25k_ring", "run", UNICYCLE, 256, 100, 1, RING, SYSTEMATIC, 64, particles=True),
        # the large unicycle filter, 2^20 particles on a 32 x 64 torus, systematic resampling
        filter_case("run_unicycle_1m", "run", UNICYCLE, 512, 2048, 2, TORUS, SYSTEMATIC, 16),
        # the same with Vose alias resampling
        filter_case("run_unicycle_1m_vose", "run", UNICYCLE, 512, 2048, 2, TORUS, VOSE, 16),
        # the 6-joint arm, 2^18 particles on a 32 x 32 torus
        filter_case("run_dharm_256k", "run", DHARM, 256, 1024, 1, TORUS, SYSTEMATIC, 16, period=256),
        # the range-only unicycle with the configuration of its program's loop: ring exchange,
        # multinomial resampling
        filter_case("run_beacon_128k", "run", BEACON, 512, 256, 1, RING, REFERENCE, 16),
        # the default pipeline (one kernel per step), camera arm
        filter_case("run_camarm_64k_fused", "run", CAMARM, 512, 128, 1, RING, SYSTEMATIC, 16, pipeline=FUSED),
        # the drop-in robot-arm loop: one kernel per phase, the reference's random-number layout,
        # linear weights, multinomial resampling, host steps
        filter_case("step_refarm_32k_phased", "step", REFARM, 512, 64, 1, RING, REFERENCE, 8, pipeline=PHASED,
                    reference_rng=True, linear=True),
        # many independent trackers of very uneven sizes stepped together
        {"name": "batch_uneven_512", "kind": "batch", "model": UNICYCLE, "m": 256, "ppt": 4, "filters": 512,
         "lo": 256, "hi": 65536, "t": 2, "exchange": RING, "resampler": SYSTEMATIC, "cadence": 4, "period": 32},
        # a tracking service: 48 resident filters of two models, each round an update of all of them
        {"name": "serve_mixed_48", "kind": "serve", "m": 256, "ppt": 4, "filters": 48, "lo": 1024, "hi": 262144,
         "t": 2, "exchange": RING, "resampler": SYSTEMATIC, "rounds": 4, "period": 256},
        # the posterior mean of a particle set held by the caller
        {"name": "estimate_1m", "kind": "estimate", "state": 3, "angles": 1, "m": 512, "n": 2048, "linear": False},
    ]


def log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: every model, exchange, resampler and form, odd counts among them."""
    kind = rng.choice(["run", "run", "run", "run", "step", "submit", "batch", "serve", "estimate"])
    if kind == "estimate":
        state = rng.choice([1, 2, 3, 4, 6, 9, 12, 16])
        m = rng.choice([32, 64, 100, 128, 250, 256, 512, 777, 1024])
        n = min(log_uniform(rng, 1, 4096), (1 << 22) // (m * state))
        return {"kind": "estimate", "state": state, "angles": rng.randint(0, min(state, 6)), "m": m, "n": max(n, 1),
                "linear": rng.random() < 0.3}
    if kind == "batch":
        lo = rng.choice([256, 1024])
        model = rng.choice([UNICYCLE, UNICYCLE, BEACON, DHARM])
        return {"kind": "batch", "model": model, "m": rng.choice([128, 256, 512]), "ppt": rng.choice([2, 4]),
                "filters": log_uniform(rng, 3, 48 if model == DHARM else 192),
                "lo": lo, "hi": log_uniform(rng, 4096, 65536), "t": rng.choice([1, 2]), "exchange": RING,
                "resampler": rng.choice([SYSTEMATIC, SYSTEMATIC, VOSE, REFERENCE]), "cadence": rng.choice([1, 2, 4]),
                "period": 32}
    if kind == "serve":
        return {"kind": "serve", "m": rng.choice([128, 256, 512]), "ppt": rng.choice([0, 4]),
                "filters": log_uniform(rng, 2, 48), "lo": 1024, "hi": log_uniform(rng, 8192, 262144),
                "t": rng.choice([1, 2]), "exchange": rng.choice([NONE, RING]),
                "resampler": rng.choice([SYSTEMATIC, SYSTEMATIC, VOSE]), "rounds": rng.randint(1, 4), "period": 256}
    model = rng.choice([UNICYCLE, UNICYCLE, DHARM, REFARM, BEACON, CAMARM])
    m = rng.choice([32, 64, 128, 256, 256, 512, 512, 1024])
    most = (1 << 20) // m if STATE[model] <= 3 else (1 << 18) // m
    n = log_uniform(rng, 1, most if kind == "run" else max(2, most // 8))
    exchange = rng.choice([NONE, RING, TORUS, TORUS, ALL2ALL])
    if exchange == TORUS:  # N = dx dy with dx the power of two nearest below sqrt(N)
        dx = 1 << int(math.log2(max(1.0, math.sqrt(n))))
        n = dx * max(dx, n // dx)
        while n // dx >= 4 * dx:
            dx *= 2
            n = dx * (n // dx)
    if exchange == ALL2ALL:
        n = min(n, 2048)
    t = rng.randint(1, 2) if exchange != NONE else 0
    resampler = rng.choice([SYSTEMATIC, SYSTEMATIC, VOSE, REFERENCE])
    pipeline = rng.choice([SPLIT, SPLIT, SPLIT, FUSED, PHASED])
    return {"kind": kind, "model": model, "m": m, "n": n, "t": t, "exchange": exchange, "resampler": resampler,
            "steps": rng.randint(4, 16), "pipeline": pipeline, "reference_rng": pipeline == PHASED,
            "linear": False, "freq": rng.choice([1.0, 1.0, 1.0, 0.8]), "ess": rng.choice([0.0, 0.0, 0.0, 0.5]),
            "period": 256 if model == DHARM else 64, "particles": kind == "run" and n * m * STATE[model] <= 1 << 17}


# ---- periodic traces -----------------------------------------------------------
def wrap(a):
    return (a + np.pi) % (2 * np.pi) - np.pi


def arm_camera(angles, x, y):
    """The camera arm's chain: the cart's coordinates in the last link's frame, [steps] each."""
    cx = cy = cz = None
    for i in range(5):
        s, c = np.sin(angles[:, i]), np.cos(angles[:, i])
        if i == 0:
            cx, cy, cz = x * c + y * s, -x * s + y * c, np.zeros_like(x)
        else:
            cy, cz = cy * c - cz * s, cy * s + cz * c - 3.0
    return cx, cy, cz


def dh_pose(p, q):
    """Position and yaw / pitch / roll of the DH chain for joint angles q [steps, 6]."""
    n = len(q)
    R = np.broadcast_to(np.eye(3), (n, 3, 3)).copy()
    pos = np.zeros((n, 3))
    for i in range(6):
        ct, st = np.cos(q[:, i]), np.sin(q[:, i])
        ca, sa = math.cos(p.alpha[i]), math.sin(p.alpha[i])
        A = np.zeros((n, 3, 3))
        A[:, 0, 0], A[:, 0, 1], A[:, 0, 2] = ct, -st * ca, st * sa
        A[:, 1, 0], A[:, 1, 1], A[:, 1, 2] = st, ct * ca, -ct * sa
        A[:, 2, 1], A[:, 2, 2] = sa, ca
        pos = pos + np.einsum("nij,nj->ni", R, np.stack([p.a[i] * ct, p.a[i] * st, np.full(n, p.d[i])], 1))
        R = R @ A
    return np.concatenate([pos, np.stack([np.arctan2(R[:, 1, 0], R[:, 0, 0]),
                                          np.arctan2(-R[:, 2, 0], np.hypot(R[:, 2, 1], R[:, 2, 2])),
                                          np.arctan2(R[:, 2, 1], R[:, 2, 2])], 1)], 1)


def trace(model, period, seed):
    """(model parameters, inputs [period] STEP_INPUT_DTYPE): truth back at its start after `period` steps."""
    rng = np.random.default_rng(seed)
    inputs = np.zeros(period, E.STEP_INPUT_DTYPE)
    k = np.arange(1, period + 1)
    if model == UNICYCLE or model == BEACON:
        p = E.unicycle_params(seed & 0xFFFF) if model == UNICYCLE else E.beacon_params()
        dt = p.dt
        turn = 2 * np.pi / period  # one full circle
        v = 1.0
        th0 = p.init_state[2]
        th = th0 + turn * k
        r = v * dt / turn
        x = p.init_state[0] + r * (np.sin(th) - math.sin(th0))
        y = p.init_state[1] - r * (np.cos(th) - math.cos(th0))
        inputs["control"][:, 0], inputs["control"][:, 1] = v, turn / dt
        if model == UNICYCLE:
            L = p.num_landmarks
            for j in range(L):
                dx, dy = p.landmarks[j][0] - x, p.landmarks[j][1] - y
                inputs["meas"][:, j] = np.hypot(dx, dy) + rng.normal(0, p.sigma_range, period)
                inputs["meas"][:, L + j] = wrap(np.arctan2(dy, dx) - th + rng.normal(0, p.sigma_bearing, period))
        else:
            for j in range(p.num_beacons):
                d = np.sqrt((x - p.beacons[j][0]) ** 2 + (y - p.beacons[j][1]) ** 2 + p.beacons[j][2] ** 2)
                inputs["meas"][:, j] = d + rng.normal(0, p.sigma_range, period)
    elif model == DHARM:
        p = E.dharm_params(seed & 0xFFFF)
        w = 2 * np.pi / (period * p.dt)
        phase = rng.uniform(0, 2 * np.pi, 6)
        amp = 0.01 / (w * w * p.dt)  # the largest velocity change per step is the process noise's deviation
        q0 = np.array(p.init_state[:6])
        q = q0 + amp * (np.sin(w * p.dt * k[:, None] + phase) - np.sin(phase))
        for i in range(6):
            p.init_state[6 + i] = amp * w * math.cos(phase[i])
        z = dh_pose(p, q)
        z[:, :3] += rng.normal(0, p.sigma_pos, (period, 3))
        z[:, 3:] = wrap(z[:, 3:] + rng.normal(0, p.sigma_ang, (period, 3)))
        inputs["meas"][:, :6] = z
    else:
        p = E.refarm_params() if model == REFARM else E.camarm_params()
        turn = 2 * np.pi / period
        phase = rng.uniform(0, 2 * np.pi, 5)
        a0 = np.array(p.init_state[:5])
        ang = a0 + 0.3 * (np.sin(turn * k[:, None] + phase) - np.sin(phase))
        before = a0 + 0.3 * (np.sin(turn * (k[:, None] - 1) + phase) - np.sin(phase))
        inputs["control"][:, :5] = (ang - before) / p.dt
        x = p.init_state[5] + 1.0 - np.cos(turn * k)
        y = p.init_state[6] + np.sin(turn * k)
        cx, cy, cz = arm_camera(ang, x, y)
        inputs["meas"][:, :5] = ang + rng.normal(0, 0.1, (period, 5))
        if model == CAMARM:
            xn, yn = cx / cz, cy / cz
            r2 = xn * xn + yn * yn
            rad = 1 + p.kc[0] * r2 + p.kc[1] * r2 * r2
            cx = p.fc[0] * (rad * xn + 2 * p.kc[2] * xn * yn + p.kc[3] * (3 * xn * xn + yn * yn)) + p.cc[0]
            cy = p.fc[1] * (rad * yn + p.kc[2] * (3 * yn * yn + xn * xn) + 2 * p.kc[3] * xn * yn) + p.cc[1]
        inputs["meas"][:, 5] = cx + rng.normal(0, 1.0, period)
        inputs["meas"][:, 6] = cy + rng.normal(0, 1.0, period)
    return p, inputs


def uneven_counts(case, seed):
    """Particle counts log-uniform over [lo, hi], multiples of lo: one count per equal slice of the
    logarithm, so that every seed gives about the same total, in an order of the seed's."""
    rng = np.random.default_rng(seed)
    n = case["filters"]
    u = rng.permutation((np.arange(n) + 0.5) / n)
    x = np.exp(math.log(case["lo"]) + u * math.log(case["hi"] / case["lo"]))
    return np.clip(np.rint(x / case["lo"]).astype(np.int64) * case["lo"], case["lo"], None).astype(np.int32)


# ---- prepare / run -------------------------------------------------------------
def to_device(records):
    return torch.from_numpy(np.ascontiguousarray(records).view(np.uint8).reshape(-1).copy()).cuda()


def estimate_fields(raw, *shape):
    """Views of the estimate records in a device buffer: every field of pf_estimate."""
    d = raw.view(torch.float64).view(*shape, EST_WORDS)
    f = raw.view(torch.float32).view(*shape, 2 * EST_WORDS)
    i = raw.view(torch.int32).view(*shape, 2 * EST_WORDS)
    return {"mean": d[..., :16], "log_norm": d[..., 16], "best": f[..., 34:50], "best_key": f[..., 50],
            "best_subfilter": i[..., 51], "step": i[..., 52], "flags": i[..., 53]}


def record_fields(rec):
    return {k: rec[k] for k in ("mean", "log_norm", "best", "best_key", "best_subfilter", "step", "flags")}


def prepare(case, seed):
    kind = case["kind"]
    state = {"case": case}
    if kind == "estimate":
        T = case["m"] * case["n"]
        g = torch.Generator(device="cuda").manual_seed(seed)
        x = 2.0 * torch.randn(case["state"], T, generator=g, device="cuda")
        # log-likelihoods of particles spread about the mode, or their exponentials
        keys = -0.5 * torch.randn(T, generator=g, device="cuda").square() * 9.0
        state["keys"] = keys.exp() if case["linear"] else keys
        state["state"] = x
        state["out"] = torch.zeros(8 * EST_WORDS, dtype=torch.uint8, device="cuda")
        state["fields"] = estimate_fields(state["out"])
        return state
    if kind == "batch":
        counts = uneven_counts(case, seed)
        params, inputs = zip(*[trace(case["model"], case["period"], 1000 * seed + i) for i in range(len(counts))])
        state["filter"] = E.FilterBatch(case["model"], list(params), counts, particles_per_subfilter=case["m"],
                                        particles_per_thread=case["ppt"], num_transfer=case["t"],
                                        exchange=case["exchange"], resampler=case["resampler"],
                                        exchange_period=case["cadence"], seed=seed)
        state["in"] = to_device(np.stack(inputs))
        state["est"] = torch.zeros(len(counts) * case["period"] * 8 * EST_WORDS, dtype=torch.uint8, device="cuda")
        state["fields"] = estimate_fields(state["est"], len(counts), case["period"])
        return state
    if kind == "serve":
        counts = uneven_counts(dict(case, lo=max(case["lo"], case["m"])), seed)
        server = E.Server(8 << 30, len(counts), particles_per_subfilter=case["m"], particles_per_thread=case["ppt"],
                          num_transfer=case["t"], exchange=case["exchange"], resampler=case["resampler"])
        ids, inputs = [], []
        for i, n in enumerate(counts):
            model = DHARM if i % 10 >= 7 else UNICYCLE
            p, inp = trace(model, case["period"], 1000 * seed + i)
            ids.append(server.open(model, p, int(n), (seed + 1000 * i) & 0xFFFFFFFF))
            inputs.append(inp)
        state.update(filter=server, ids=ids, inputs=inputs, at=0)
        return state
    model = case["model"]
    p, inputs = trace(model, case["period"], seed)
    f = E.ParticleFilter(model, p, particles_per_subfilter=case["m"], num_subfilters=case["n"],
                         num_transfer=case["t"], exchange=case["exchange"], resampler=case["resampler"],
                         pipeline=case["pipeline"], rng=1 if case["reference_rng"] else 0,
                         mtgp_streams=120, log_weights=0 if case["linear"] else 1, resampling_freq=case["freq"],
                         ess_fraction=case["ess"], seed=seed & 0xFFFFFFFF)
    state["filter"] = f
    if kind == "run":
        state["in"] = to_device(inputs)
        state["est"] = torch.zeros(case["period"] * 8 * EST_WORDS, dtype=torch.uint8, device="cuda")
        state["fields"] = estimate_fields(state["est"], case["period"])
        f.run_device(state["in"].data_ptr(), state["est"].data_ptr(), case["period"], 0)
    else:
        state["inputs"] = [E.step_input(inputs[k]) for k in range(case["period"])]
        state["at"] = 0
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "estimate":
        E.estimate_noalloc(state["keys"].data_ptr(), state["state"].data_ptr(), case["state"],
                           case["m"] * case["n"], case["m"], state["out"].data_ptr(),
                           angle_mask=((1 << case["angles"]) - 1) << (case["state"] - case["angles"]),
                           log_weights=0 if case["linear"] else 1, stream=torch.cuda.current_stream().cuda_stream)
        return state["fields"]
    f = state["filter"]
    if kind == "run":
        f.run_continue(case["steps"])
        if case["particles"]:
            return dict(state["fields"], particles=f.particles())
        return state["fields"]
    if kind == "batch":
        f.submit(state["in"].data_ptr(), state["est"].data_ptr(), case["period"], case["period"])
        return state["fields"]
    out = []
    if kind == "serve":
        for _ in range(case["rounds"]):
            k = state["at"] % case["period"]
            state["at"] += 1
            for fid, inp in zip(state["ids"], state["inputs"]):
                f.update(fid, inp[k:k + 1], tag=k)
            f.launch()
            r = f.poll(wait=True)
            out.append(dict(record_fields(r["estimate"]), filter=r["filter"], updates=r["step"]))
        return out
    for _ in range(case["steps"]):
        inp = state["inputs"][state["at"] % case["period"]]
        state["at"] += 1
        if kind == "step":
            out.append(f.step(inp))
        else:
            f.submit(inp)
    return record_fields(np.array(out) if kind == "step" else f.collect(case["steps"]))


# ---- work ----------------------------------------------------------------------
def step_flops(model):
    """Floating-point operations of one particle's step: Box-Muller, propagation, likelihood."""
    body = {UNICYCLE: 40 + 4 * 45, DHARM: 6 * 70 + 100, REFARM: 130, BEACON: 40 + 10 * 10, CAMARM: 170}
    return 20 * NOISE[model] + body[model]


def work(case):
    """Each particle's state read and written once a step, an input read and an estimate written."""
    if case["kind"] == "estimate":
        T = case["m"] * case["n"]
        return {"bytes": 4 * T * (1 + case["state"]) + 8 * EST_WORDS, "flops": T * (10 + 4 * case["state"])}
    if case["kind"] == "batch":
        P, n = int(uneven_counts(case, 0).sum()), case["filters"]
        per, fl, steps = 8 * STATE[case["model"]], step_flops(case["model"]), case["period"]
        return {"bytes": steps * (P * per + n * (128 + 8 * EST_WORDS)), "flops": steps * P * fl}
    if case["kind"] == "serve":
        counts = uneven_counts(dict(case, lo=max(case["lo"], case["m"])), 0)
        P, n = int(counts.sum()), len(counts)
        arm = sum(1 for i in range(n) if i % 10 >= 7) / n  # counts come in a random order
        per = 8 * (arm * STATE[DHARM] + (1 - arm) * STATE[UNICYCLE])
        fl = arm * step_flops(DHARM) + (1 - arm) * step_flops(UNICYCLE)
        return {"bytes": case["rounds"] * (P * per + n * (128 + 8 * EST_WORDS)), "flops": case["rounds"] * P * fl}
    T = case["m"] * case["n"]
    per = 8 * STATE[case["model"]]
    return {"bytes": case["steps"] * (T * per + 128 + 8 * EST_WORDS) + (T * per / 2 if case["particles"] else 0),
            "flops": case["steps"] * T * step_flops(case["model"])}


def exact(case, seed):
    """The estimate of given particles in 64 bits.  A filter's own steps have no such value: their
    random numbers come from the engine's streams and one changed rounding in a weight changes
    which particles are drawn."""
    if case["kind"] != "estimate":
        return None
    s = prepare(case, seed)
    k, x = s["keys"].double().cpu(), s["state"].double().cpu()
    top = k.max()
    w = k if case["linear"] else (k - top).exp()
    W = w.sum()
    mean = torch.zeros(16, dtype=torch.float64)
    S, first = case["state"], case["state"] - case["angles"]
    for v in range(S):
        if v < first:
            mean[v] = (w * x[v]).sum() / W
        else:
            mean[v] = torch.atan2((w * x[v].sin()).sum(), (w * x[v].cos()).sum())
    at = int(k.argmax())
    best = torch.zeros(16, dtype=torch.float32)
    best[:S] = s["state"][:, at].cpu()
    return {"mean": mean, "log_norm": W.log() + (0.0 if case["linear"] else top), "best": best,
            "best_key": s["keys"][at].cpu(), "best_subfilter": torch.tensor(at // case["m"], dtype=torch.int32),
            "step": None, "flags": None}
