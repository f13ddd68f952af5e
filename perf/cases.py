"""The calls whose time matters to a program that plans with this library, over the range of sizes
it makes them at: whole plans of each dynamics model (plain, learned and in batches), and the
stages that programs call on their own — segment propagation, swept-box queries, the learned
proposal's inference pass and its training gradient.

Sizes are those of the presets, the benchmark workloads (bench.py) and the tests, with odd sizes
and smaller calls beside them.
"""
from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

PACKAGE = Path(__file__).resolve().parent.parent / "kino-pax-fork_b200"
if str(PACKAGE) not in sys.path:
    sys.path.insert(0, str(PACKAGE))

import kpax  # noqa: E402
import kpax_autotune  # noqa: E402
import kpax_envs as envs  # noqa: E402
import kpax_learn  # noqa: E402

MODELS = {"di": 1, "dubins": 2, "quad": 3}
PRESETS = {"di": kpax.PRESET_DI, "dubins": kpax.PRESET_DUBINS, "quad": kpax.PRESET_QUAD}
# FP32 operations of one integration step (a fused multiply-add counts two)
STEP_FLOPS = {"di": 18, "dubins": 63, "quad": 498}
# steps of an average segment: it ends at its first failing check, or after the drawn number
STEPS_RUN = {"di": 4.5, "dubins": 14.0, "quad": 17.0}
MLP_FLOPS = 2 * (51 * 256 + 256 * 256 + 256 * 88)


def listed() -> list[dict]:
    return [
        # a replanning cycle: a goal some metres away among the building's boxes, a small budget and
        # few iterations, so the call's fixed costs count as much as its expansions
        {"name": "plan quad near", "kind": "plan", "model": "quad", "obstacles": 1000, "budget": 1 << 14, "tree": 1 << 17,
         "iterations": 20, "near": True, "learned": False},
        # the quadrotor benchmark: the preset in the building scene, a goal on its far side
        {"name": "plan quad", "kind": "plan", "model": "quad", "obstacles": 1000, "budget": 1 << 16, "tree": 1 << 20,
         "iterations": 300, "near": False, "learned": False},
        # the Dubins benchmark: the preset in the forest
        {"name": "plan dubins", "kind": "plan", "model": "dubins", "obstacles": 200, "budget": 1 << 16, "tree": 1 << 20,
         "iterations": 300, "near": False, "learned": False},
        # the double integrator among the benchmark's boxes at the tests' speeds (|v| <= 5): short
        # segments, a frontier of many nodes, a tree that grows until it is full
        {"name": "plan di", "kind": "plan", "model": "di", "obstacles": 20, "budget": 1 << 14, "tree": 1 << 20,
         "iterations": 300, "near": False, "learned": False, "speed": 5},
        # a quadrotor plan that draws its controls from the proposal network
        {"name": "plan learned", "kind": "plan", "model": "quad", "obstacles": 700, "budget": 1 << 16, "tree": 1 << 20,
         "iterations": 120, "near": False, "learned": True},
        # a planning server: many mixed queries of uneven size in one call
        {"name": "batch", "kind": "batch", "queries": 96, "tree": 1 << 20, "obstacles": 5000, "iterations": 150},
        # the propagation benchmark: independent Dubins segments, draws made by the library
        {"name": "segments dubins 4M", "kind": "segments", "model": "dubins", "n": 1 << 22, "obstacles": 200,
         "draws": False, "entry": "env"},
        # a caller's own sampler: some ten thousand quadrotor segments with given draws
        {"name": "segments quad 30k", "kind": "segments", "model": "quad", "n": 30011, "obstacles": 1000,
         "draws": True, "entry": "env"},
        # a control loop: a thousand segments against this cycle's obstacles, nothing allocated
        {"name": "segments di 1k", "kind": "segments", "model": "di", "n": 1021, "obstacles": 20, "draws": True,
         "entry": "noalloc"},
        # collision checking on its own: the swept boxes of single integration steps
        {"name": "collide 4M", "kind": "collide", "n": 1 << 22, "obstacles": 1000},
        # the proposal network's records for a set of states
        {"name": "propose 64k", "kind": "propose", "n": 65536, "obstacles": 1000},
        # the proposal network's training: loss and gradient of one mini-batch of the training recipe
        {"name": "gradient 4096", "kind": "gradient", "n": 4096},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["plan", "plan", "plan", "segments", "segments", "collide", "propose", "gradient", "batch"])
    if kind == "plan":
        model = rng.choice(["quad", "quad", "dubins", "di"])
        obstacles = _log_int(rng, 100, 2000) if model == "quad" else _log_int(rng, 10, 400)
        return {"kind": kind, "model": model, "obstacles": obstacles, "budget": _log_int(rng, 1 << 11, 1 << 16),
                "tree": _log_int(rng, 1 << 15, 1 << 20), "iterations": _log_int(rng, 5, 200),
                "near": rng.random() < 0.4, "learned": model == "quad" and rng.random() < 0.3,
                "speed": rng.choice([1, 5]) if model == "di" else 0}
    if kind == "segments":
        model = rng.choice(["quad", "dubins", "di"])
        noalloc = rng.random() < 0.4
        return {"kind": kind, "model": model, "n": _log_int(rng, 100, 1 << 17 if noalloc else 1 << 21),
                "obstacles": _log_int(rng, 10, 1000), "draws": rng.random() < 0.5, "entry": "noalloc" if noalloc else "env"}
    if kind == "collide":
        return {"kind": kind, "n": _log_int(rng, 200, 1 << 22), "obstacles": _log_int(rng, 20, 2000)}
    if kind == "propose":
        return {"kind": kind, "n": _log_int(rng, 50, 1 << 17), "obstacles": _log_int(rng, 200, 2000)}
    if kind == "gradient":
        return {"kind": kind, "n": _log_int(rng, 128, 8192)}
    return {"kind": kind, "queries": _log_int(rng, 3, 90), "tree": _log_int(rng, 1 << 15, 1 << 19),
            "obstacles": _log_int(rng, 100, 4000), "iterations": _log_int(rng, 20, 100)}


# ---------------------------------------------------------------------------------------------
# inputs


def _scene(model: str, n: int, seed: int):
    """(obstacles, start, goal) of a model's benchmark scene with n obstacles."""
    if model == "quad":
        return envs.quad_scene(seed=seed, n_total=max(n, 20))
    if model == "dubins":
        _, start, goal = envs.dubins_scene()
        trees = envs.forest(n, seed)
        keep = [b for b in trees if not any(np.all(b[:3] <= p[:3]) and np.all(p[:3] <= b[3:]) for p in (start, goal))]
        return np.asarray(keep, np.float32).reshape(-1, 6), start, goal
    _, start, goal = envs.di_scene()
    return envs.random_boxes(n, seed, avoid=(start, goal)), start, goal


def _uniform(g, n: int, lo: list[float], hi: list[float]):
    u = torch.rand((n, len(lo)), generator=g, device="cuda", dtype=torch.float32)
    lo_t, hi_t = torch.tensor(lo, device="cuda"), torch.tensor(hi, device="cuda")
    return (lo_t + u * (hi_t - lo_t)).contiguous()


def _parents(model: str, n: int, g):
    """States uniform within the model's bounds, as the benchmarks draw them."""
    pi = math.pi
    if model == "di":
        return _uniform(g, n, [0, 0, 0, -1, -1, -1], [100, 100, 100, 1, 1, 1])
    if model == "dubins":
        return _uniform(g, n, [0, 0, 0, -pi, -pi / 3, 0.5], [100, 100, 100, pi, pi / 3, 2])
    return _uniform(g, n, [0] * 3 + [-0.5] * 3 + [-5] * 3 + [-0.5] * 3, [100] * 3 + [0.5] * 3 + [5] * 3 + [0.5] * 3)


def _generator(seed: int):
    return torch.Generator(device="cuda").manual_seed(seed)


def _segment_inputs(case: dict, seed: int):
    """Obstacles, parents and (where the caller draws) uniforms in (0, 1] on a 2^-24 grid."""
    obs, _, _ = _scene(case["model"], case["obstacles"], seed)
    g = _generator(seed)
    parents = _parents(case["model"], case["n"], g)
    draws = None
    if case["draws"]:
        draws = torch.randint(1, (1 << 24) + 1, (case["n"], 5), generator=g, device="cuda").float() * 2.0 ** -24
    return obs, parents, draws


def _propose_inputs(case: dict, seed: int):
    obs, _, _ = _scene("quad", case["obstacles"], seed)
    g = _generator(seed)
    return obs, _parents("quad", case["n"], g), _uniform(g, case["n"], [5] * 3, [95] * 3)


def _gradient_inputs(case: dict, seed: int):
    """Features as harvested trees give them (scaled states, scaled goal offsets, occupancy bits of
    the neighbouring cells) and the logits of the draw uniforms; freshly initialised parameters."""
    n, g = case["n"], _generator(seed)
    x = torch.zeros((n, kpax.MLP_FEATURES), device="cuda")
    x[:, :12] = _uniform(g, n, [0] * 3 + [-1] * 3 + [-1] * 3 + [-0.5] * 3, [1] * 3 + [1] * 6 + [0.5] * 3)
    x[:, 12:15] = _uniform(g, n, [0.05] * 3, [0.95] * 3) - x[:, :3]
    x[:, 15:24] = -x[:, 3:12]
    x[:, 24:51] = (torch.rand((n, 27), generator=g, device="cuda") < 0.3).float()
    u = torch.rand((n, 5), generator=g, device="cuda").clamp(1e-4, 1 - 1e-4)
    return x, torch.log(u / (1 - u)).contiguous(), kpax_learn.init_params(seed)


def _plan_config(case: dict, n_obs: int) -> kpax.Config:
    cfg = kpax.preset(PRESETS[case["model"]])
    cfg.expansions_per_iter, cfg.max_tree_size, cfg.max_iter = case["budget"], case["tree"], case["iterations"]
    if case.get("speed") == 5:  # the tests' faster double integrator
        cfg.v_min, cfg.v_max = -5.0, 5.0
        for d in range(3):
            cfg.ctrl_min[d], cfg.ctrl_max[d] = -4.0, 4.0
    return kpax_autotune.tuned(cfg, n_obs)[0]


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "plan":
        if case["learned"] and not case["near"]:  # goals within a plan's reach: the learned family
            obs, start, goal = envs.learned_family(seed, obs_range=(case["obstacles"], case["obstacles"]))
        else:
            obs, start, goal = _scene(case["model"], case["obstacles"], seed)
            if case["near"]:
                pair = envs.free_queries(obs, 1, seed, *((6.0, 15.0) if case["model"] == "quad" else (8.0, 20.0)))[0]
                start, goal = start.copy(), goal.copy()
                start[:3], goal[:3] = pair[:3], pair[3:]
        planner = kpax.KPAX(_plan_config(case, obs.shape[0]))
        if case["learned"]:
            planner.set_proposal(kpax_learn.load_network(), 0.2)
        return {"case": case, "planner": planner, "obs": torch.from_numpy(obs).cuda(), "start": start, "goal": goal}
    if kind == "batch":
        queries = envs.batch_queries(case["queries"], seed, obs_range=(10, case["obstacles"]), tree_range=(1 << 14, case["tree"]))
        cfgs = []
        for q in queries:
            cfg = kpax.preset({1: kpax.PRESET_DI, 2: kpax.PRESET_DUBINS, 3: kpax.PRESET_QUAD}[q["model"]])
            cfg.max_tree_size, cfg.max_iter, cfg.block_size = q["tree"], case["iterations"], 256
            cfgs.append(cfg)
        obs = [torch.from_numpy(q["obstacles"]).cuda() for q in queries]
        return {"case": case, "batch": kpax.Batch(cfgs), "obs": obs, "start": [q["start"] for q in queries],
                "goal": [q["goal"] for q in queries], "n_obs": [q["n_obs"] for q in queries]}
    if kind == "segments":
        obs, parents, draws = _segment_inputs(case, seed)
        cfg, n = kpax.preset(PRESETS[case["model"]]), case["n"]
        d_obs = torch.from_numpy(obs).cuda()
        env = kpax.Env(cfg, d_obs.data_ptr(), obs.shape[0]) if case["entry"] == "env" else None
        return {"case": case, "cfg": cfg, "env": env, "obs": d_obs, "parents": parents, "draws": draws, "stream": seed % 1000,
                "rows": torch.zeros((n, cfg.sample_dim), device="cuda"),
                "valid": torch.zeros(n, dtype=torch.uint8, device="cuda"),
                "steps": torch.zeros(n, dtype=torch.int32, device="cuda")}
    if kind == "collide":
        obs, _, _ = _scene("quad", case["obstacles"], seed)
        cfg = kpax.preset(kpax.PRESET_QUAD)
        d_obs = torch.from_numpy(obs).cuda()
        g = _generator(seed)
        lo = _uniform(g, case["n"], [0] * 3, [100] * 3)
        hi = lo + _uniform(g, case["n"], [0] * 3, [0.2] * 3)
        return {"case": case, "env": kpax.Env(cfg, d_obs.data_ptr(), obs.shape[0]), "obs": d_obs, "lo": lo, "hi": hi,
                "free": torch.zeros(case["n"], dtype=torch.uint8, device="cuda")}
    if kind == "propose":
        obs, states, goals = _propose_inputs(case, seed)
        d_obs = torch.from_numpy(obs).cuda()
        env = kpax.Env(kpax.preset(kpax.PRESET_QUAD), d_obs.data_ptr(), obs.shape[0])
        return {"case": case, "env": env, "obs": d_obs, "net": kpax_learn.load_network(), "states": states, "goals": goals,
                "mix": torch.zeros((case["n"], kpax.MLP_MIX), device="cuda")}
    x, y, params = _gradient_inputs(case, seed)
    net = kpax.MLP(max_batch=case["n"])
    net.set_params(params)
    return {"case": case, "net": net, "x": x, "y": y, "grad": torch.zeros(net.num_params, device="cuda")}


def _rows(path: np.ndarray, case: dict) -> np.ndarray:
    """A plan's path with zero rows up to the longest one that its iterations allow."""
    out = np.zeros((case["iterations"] + 2, path.shape[1]), np.float32)
    out[: path.shape[0]] = path
    return out


def run(state: dict):
    case = state["case"]
    kind = case["kind"]
    if kind == "plan":
        planner = state["planner"]
        r = planner.plan(state["start"], state["goal"], state["obs"].data_ptr(), state["obs"].shape[0])
        return {"path": _rows(planner.h_controlPathToGoal_, case), "cost": float(r.path_cost),
                "counts": np.array([r.found, r.goal_idx, r.path_len, r.tree_size, r.iters, r.tree_full, r.expansions,
                                    r.valid_expansions], np.int64)}
    if kind == "batch":
        res, stats = state["batch"].plan(state["start"], state["goal"], [o.data_ptr() for o in state["obs"]], state["n_obs"])
        fields = ("found", "goal_idx", "path_len", "tree_size", "iters", "tree_full", "expansions", "valid_expansions")
        return {"paths": np.concatenate([_rows(r["path"], case).ravel() for r in res]),
                "costs": np.array([r["path_cost"] for r in res], np.float64),
                "counts": np.array([[r[f] for f in fields] for r in res], np.int64),
                "totals": np.array([stats[f] for f in ("iters", "found", "expansions", "valid_expansions", "steps")], np.int64)}
    if kind == "segments":
        draws = state["draws"].data_ptr() if state["draws"] is not None else None
        args = (state["parents"].data_ptr(), draws, state["stream"], case["n"], state["rows"].data_ptr(),
                state["valid"].data_ptr(), state["steps"].data_ptr())
        if case["entry"] == "env":
            kpax.propagate_batch(state["cfg"], state["env"], *args)
        else:
            kpax.propagate_batch_noalloc(state["cfg"], state["obs"].data_ptr(), state["obs"].shape[0], *args)
        return {"rows": state["rows"], "valid": state["valid"], "steps": state["steps"]}
    if kind == "collide":
        kpax.collide_batch(state["env"], state["lo"].data_ptr(), state["hi"].data_ptr(), case["n"], state["free"].data_ptr())
        return state["free"]
    if kind == "propose":
        state["net"].propose(state["env"], state["states"].data_ptr(), 12, state["goals"].data_ptr(), case["n"],
                             state["mix"].data_ptr())
        return state["mix"]
    loss = state["net"].loss_grad(state["x"].data_ptr(), state["y"].data_ptr(), case["n"], state["grad"].data_ptr())
    return {"loss": loss, "grad": state["grad"]}


def work(case: dict) -> dict:
    """Bytes and operations of one pass: inputs and results once; of a plan, the children's
    integration steps and the nodes it keeps (at most what its tree and iterations allow)."""
    kind = case["kind"]
    if kind == "plan":
        m, sd = case["model"], 12 if case["model"] == "quad" else 6
        iters = min(case["iterations"], 6 if case["near"] else 10 ** 9)
        children = iters * case["budget"]
        nodes = min(case["tree"], children // 4 + 1)
        flops = children * STEPS_RUN[m] * STEP_FLOPS[m]
        if case["learned"]:
            flops += children / 32 * MLP_FLOPS
        return {"bytes": nodes * (4 * sd + 37) + 24 * case["obstacles"], "flops": flops}
    if kind == "batch":
        per = case["iterations"] * (0.4 * (1 << 14) * STEPS_RUN["di"] * STEP_FLOPS["di"] +
                                    0.3 * (1 << 16) * STEPS_RUN["dubins"] * STEP_FLOPS["dubins"] +
                                    0.3 * (1 << 16) * STEPS_RUN["quad"] * STEP_FLOPS["quad"]) / 2
        return {"bytes": case["queries"] * case["tree"] / 4 * 80, "flops": case["queries"] * per}
    if kind == "segments":
        sd, cd = (12, 4) if case["model"] == "quad" else (6, 3)
        bytes_ = case["n"] * (4 * sd + (20 if case["draws"] else 0) + 4 * (sd + cd + 1) + 5) + 24 * case["obstacles"]
        return {"bytes": bytes_, "flops": case["n"] * STEPS_RUN[case["model"]] * STEP_FLOPS[case["model"]]}
    if kind == "collide":
        return {"bytes": 25 * case["n"] + 24 * case["obstacles"], "flops": 12 * case["n"]}
    if kind == "propose":
        return {"bytes": case["n"] * 4 * (12 + 3 + kpax.MLP_MIX) + 2 * kpax_learn.NUM_PARAMS, "flops": case["n"] * MLP_FLOPS}
    return {"bytes": case["n"] * 4 * (64 + 5) + 8 * kpax_learn.NUM_PARAMS, "flops": 3 * case["n"] * MLP_FLOPS}


# ---------------------------------------------------------------------------------------------
# 64-bit values


def _philox_uniforms(n: int, stream: int, seed: int):
    """The library's draws of segments 0..n-1: Philox4x32-10 (Salmon et al., 2011) with counter
    (index, 0, sub-stream, stream) and key `seed`; ((x >> 8) + 1) * 2^-24."""
    mask = 0xFFFFFFFF

    def words(sub: int):
        c = [torch.arange(n, device="cuda", dtype=torch.int64)] + [torch.full((n,), v, device="cuda", dtype=torch.int64)
                                                                  for v in (0, sub, stream)]
        k0, k1 = seed & mask, (seed >> 32) & mask
        for _ in range(10):
            p0, p1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
            c = [((p1 >> 32) & mask) ^ c[1] ^ k0, p1 & mask, ((p0 >> 32) & mask) ^ c[3] ^ k1, p0 & mask]
            k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
        return c

    a, b = words(0), words(1)
    return torch.stack([((w >> 8) + 1).double() * 2.0 ** -24 for w in (a[0], a[1], a[2], a[3], b[0])], dim=1)


def _quad_rates(s, c):
    """Derivative of the quadrotor's state (NU 10e-3, MU 2e-6, inertia 1, 1, 2, mass 1, g 9.81)."""
    f, t, p, u, v, w, P, Q, R = s[:, 3:].unbind(1)
    sf, cf, st, ct, sp, cp = f.sin(), f.cos(), t.sin(), t.cos(), p.sin(), p.cos()
    drag = -10e-3 * torch.sqrt(u * u + v * v + w * w)
    spin = -2e-6 * torch.sqrt(P * P + Q * Q + R * R)
    g = -9.81
    return torch.stack([
        ct * cp * u + (sf * st * cp - cf * sp) * v + (cf * st * cp + sf * sp) * w,
        ct * sp * u + (sf * st * sp + cf * cp) * v + (cf * st * sp - sf * cp) * w,
        -st * u + sf * ct * v + cf * ct * w,
        P + (Q * sf + R * cf) * st / ct, Q * cf - R * sf, (Q * sf + R * cf) / ct,
        R * v - Q * w - g * st + drag * u, P * w - R * u + g * ct * sf + drag * v,
        Q * u - P * v + g * ct * cf + drag * w + c[:, 0],
        -Q * R + spin * P + c[:, 1], P * R + spin * Q + c[:, 2], 0.5 * (spin * R + c[:, 3])], dim=1)


def _step(model: str, s, c, h: float):
    if model == "di":
        v, a = s[:, 3:], c[:, :3]
        return torch.cat([s[:, :3] + (5 * v + 2 * a * h) * h / 6, v + a * h], dim=1)
    if model == "dubins":
        def rates(q):
            ct, st, cy, sy = q[:, 4].cos(), q[:, 4].sin(), q[:, 3].cos(), q[:, 3].sin()
            return torch.stack([q[:, 5] * ct * cy, q[:, 5] * ct * sy, q[:, 5] * st, c[:, 1], c[:, 2], c[:, 0]], dim=1)
    else:
        def rates(q):
            return _quad_rates(q, c)
    k1 = rates(s)
    k2 = rates(s + 0.5 * h * k1)
    k3 = rates(s + 0.5 * h * k2)
    k4 = rates(s + h * k3)
    return s + h / 6 * (k1 + 2 * k2 + 2 * k3 + k4)


def _exact_segments(case: dict, seed: int):
    model = case["model"]
    cfg = kpax.preset(PRESETS[model])
    obs, parents, draws = _segment_inputs(case, seed)
    boxes = torch.from_numpy(obs).cuda().double()
    n, cd = case["n"], 4 if model == "quad" else 3
    u = draws.double() if draws is not None else _philox_uniforms(n, seed % 1000, int(cfg.seed))
    lo = torch.tensor([float(x) for x in cfg.ctrl_min], device="cuda", dtype=torch.float64)
    hi = torch.tensor([float(x) for x in cfg.ctrl_max], device="cuda", dtype=torch.float64)
    h, most = float(cfg.step_size), int(cfg.max_propagation_duration)
    states, controls, durations = [], [], []
    for i in range(0, n, 1 << 17):
        s, uc = parents[i: i + (1 << 17)].double(), u[i: i + (1 << 17)]
        c = lo + uc[:, :4] * (hi - lo)
        steps = (torch.full((s.shape[0],), most, device="cuda") if cfg.fixed_steps
                 else 1 + (uc[:, 4].float() * most).to(torch.int64))
        alive = torch.ones(s.shape[0], dtype=torch.bool, device="cuda")
        for k in range(int(steps.max())):
            idx = torch.nonzero(alive & (steps > k)).ravel()
            if not idx.numel():
                break
            a = s[idx]
            b = _step(model, a, c[idx], h)
            v = {"di": b[:, 3:6], "dubins": b[:, 5:6], "quad": b[:, 6:9]}[model]
            ok = ((v >= cfg.v_min) & (v <= cfg.v_max)).all(1)
            if model == "dubins":
                ok &= (b[:, 4] >= cfg.pitch_min) & (b[:, 4] <= cfg.pitch_max)
            ok &= ((b[:, :3] >= cfg.w_min) & (b[:, :3] <= cfg.w_max)).all(1)
            p, q = torch.minimum(a[:, :3], b[:, :3]), torch.maximum(a[:, :3], b[:, :3])
            hit = torch.ones((idx.numel(), boxes.shape[0]), dtype=torch.bool, device="cuda")
            for d in range(3):
                hit &= (q[:, d, None] > boxes[None, :, d]) & (boxes[None, :, 3 + d] > p[:, d, None])
            s[idx] = b
            alive[idx] = ok & ~hit.any(1)
        states.append(s)
        controls.append(c[:, [1, 2, 0]] if model == "dubins" else c[:, :cd])
        durations.append(h * steps.double()[:, None])
    rows = torch.cat([torch.cat(states), torch.cat(controls), torch.cat(durations)], dim=1)
    return {"rows": rows, "valid": None, "steps": None}


def _unpack(w):
    W1, b1, W2, b2, W3, b3 = torch.split(w, [256 * 64, 256, 256 * 256, 256, 96 * 256, 96])
    return W1.view(256, 64), b1, W2.view(256, 256), b2, W3.view(96, 256), b3


def _network(w, x):
    W1, b1, W2, b2, W3, b3 = _unpack(w)
    silu = torch.nn.functional.silu
    return (silu(silu(x @ W1.T + b1) @ W2.T + b2) @ W3.T + b3)[:, :88]


def _exact_propose(case: dict, seed: int):
    obs, states, goals = _propose_inputs(case, seed)
    boxes, s = torch.from_numpy(obs).cuda().double(), states.double()
    # occupancy of the 8^3 cells (12.5 m): at least 32 of 4^3 lattice points inside boxes
    at = (torch.arange(32, device="cuda").double() + 0.5) * 3.125
    pts = torch.stack(torch.meshgrid(at, at, at, indexing="ij"), dim=-1).reshape(-1, 3)
    inside = torch.zeros(pts.shape[0], dtype=torch.bool, device="cuda")
    for b in boxes:
        inside |= ((pts >= b[:3]) & (pts <= b[3:])).all(1)
    blocked = inside.view(8, 4, 8, 4, 8, 4).sum((1, 3, 5)) >= 32
    padded = torch.ones((10, 10, 10), dtype=torch.float64, device="cuda")
    padded[1:9, 1:9, 1:9] = blocked.double()
    cell = (8 * states[:, :3] / 100).to(torch.int64).clamp(0, 7) + 1
    scale = torch.tensor([0.01] * 3 + [1.0] * 3 + [0.1] * 3 + [1.0] * 3, device="cuda", dtype=torch.float64)
    goal = torch.zeros_like(s)
    goal[:, :3] = goals.double()
    bits = [padded[cell[:, 0] + j % 3 - 1, cell[:, 1] + j // 3 % 3 - 1, cell[:, 2] + j // 9 - 1][:, None] for j in range(27)]
    x = torch.cat([s * scale, (goal - s) * scale] + bits + [torch.zeros((s.shape[0], 13), device="cuda")], dim=1)
    w = torch.from_numpy(np.load(PACKAGE / "weights" / "quad_proposal.npz")["params"].astype(np.float64)).cuda()
    return _network(w, x)


def _exact_gradient(case: dict, seed: int):
    x, y, params = _gradient_inputs(case, seed)
    w = torch.from_numpy(params.astype(np.float64)).cuda().requires_grad_()
    o = _network(w, x.double()).view(-1, 8, 11)
    s = -2 + 5 * torch.tanh(o[:, :, 6:] / 5)
    r = (y.double()[:, None] - o[:, :, 1:6]) * torch.exp(-s)
    logs = torch.log_softmax(o[:, :, 0], dim=1) + (-0.5 * r * r - s - 0.5 * math.log(2 * math.pi)).sum(2)
    loss = -torch.logsumexp(logs, dim=1).mean()
    loss.backward()
    return {"loss": float(loss.detach()), "grad": w.grad}


def exact(case: dict, seed: int):
    """What run() returns in 64 bits: the segments' rows, the mixture records, the loss and gradient.
    Plans are chains of decisions and verdicts are bytes; they have none."""
    if case["kind"] == "segments":
        return _exact_segments(case, seed)
    if case["kind"] == "propose":
        return _exact_propose(case, seed)
    return _exact_gradient(case, seed) if case["kind"] == "gradient" else None
