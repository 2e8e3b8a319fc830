"""Performance cases of the crowd-tick library: what a program that uses it has
it do, each through the entry point that program calls.

    listed()             the fixed cases
    draw(rng)            one more case of the same ranges
    prepare(case, seed)  what the program holds before the call
    run(state)           one pass, with its whole outputs
    exact(case, seed)    the outputs in 64 bits, where they have such a value
    work(case)           the bytes and operations a pass cannot do without

Maps are fixed and kept per process (a program loads its map once); the crowd,
its goals and paths, the network's weights and the training rows come from the
seed.  Crowds follow workloads.py: radius U[0.2, 0.35] m, preferred speed
U[1.2, 1.5] m/s, time horizons 2 s, neighbours within 5 m, dt = 1/60 s.
"""
from __future__ import annotations

import ctypes
import functools

import numpy as np
import torch

from ecmgenerator_gb300 import _lib
from ecmgenerator_gb300 import agents as ag
from ecmgenerator_gb300.proposal import N_HID, N_IN, N_OUT, ProposalModel, param_layout, split_params
from ecmgenerator_gb300.scene import BoxIndex
from ecmgenerator_gb300.simulator import BatchSimulator, Planner, Simulator, set_neighbor_mode
from ecmgenerator_gb300.workloads import DT, ORCA, add_spawn_areas

MAP_SEED = 1
TRAINED = "ecmgenerator_gb300/data/proposal.npy"


def listed():
    return [
        # a small crowd rolled out half a second ahead from a given state (what-if
        # runs, planning around people): launches and latency count
        dict(name="rollout_boxes_1k", kind="rollout", map="boxes", side=100, agents=1000, k=10, ticks=30),
        # the editor's running scene: spawn and goal areas keep a mid-size crowd
        # going, every tick's positions and velocities are drawn
        dict(name="spawn_boxes_25k", kind="tick", map="boxes", side=500, agents=25000, k=10, mode="spawn"),
        # dense crossing flows, drawn every tick: an ordinary large crowd
        dict(name="crossing_100k", kind="tick", map="crossing", side=400, agents=100000, k=16, mode="plain"),
        # the headline workload: a million agents in crossing flows
        dict(name="crossing_1m", kind="tick", map="crossing", side=400, agents=1000000, k=16, mode="plain"),
        # independent scenes stepped together (parameter sweeps, learning
        # environments): reset to a state, eight ticks, read back
        dict(name="batch_rollout_24", kind="batch", scenes=24, agents=65000, k=10, ticks=8),
        # the tick with the trained proposal network asked on every tick
        dict(name="learned_boxes_25k", kind="tick", map="boxes", side=500, agents=25000, k=10, mode="learned"),
        # the reference's own neighbour lists (kd-tree mode), for trajectories
        # identical to the original simulator's
        dict(name="kdtree_crossing_250k", kind="tick", map="crossing", side=400, agents=250000, k=16, mode="kdtree"),
        # the stand-alone neighbour query in somebody else's frame loop: small ...
        dict(name="knn_3k", kind="knn", n=3000, k=8, radius=5.0),
        # ... and large
        dict(name="knn_1m", kind="knn", n=1000000, k=16, radius=5.0),
        # training the proposal network: a few Adam steps at the batch size that
        # train_proposal.py uses
        dict(name="train_65k", kind="train", rows=400000, batch=65536, steps=4),
        # loss and gradient over a validation set with a ragged last tile
        dict(name="grad_3001", kind="grad", rows=3001),
        # classes of a recorded set
        dict(name="predict_250k", kind="predict", rows=250000),
    ]


def _log_int(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["tick", "tick", "tick", "rollout", "batch", "kdtree", "knn", "knn", "train", "grad", "predict"])
    k = rng.choice([5, 7, 8, 10, 11, 16, 16, 20])
    if kind == "tick":
        if rng.random() < 0.5:
            return dict(kind="tick", map="crossing", side=400, agents=_log_int(rng, 20000, 600000), k=min(k, 16),
                        mode="plain")
        side = rng.choice([200, 500])
        return dict(kind="tick", map="boxes", side=side, agents=_log_int(rng, 500, 0.1 * side * side), k=k,
                    mode=rng.choice(["plain", "spawn", "learned"]))
    if kind == "rollout":
        return dict(kind="rollout", map="boxes", side=100, agents=_log_int(rng, 60, 1500), k=k,
                    ticks=rng.randint(8, 24))
    if kind == "batch":
        return dict(kind="batch", scenes=rng.randint(2, 24), agents=_log_int(rng, 4000, 65000), k=k,
                    ticks=rng.randint(2, 8))
    if kind == "kdtree":
        return dict(kind="tick", map="crossing", side=400, agents=_log_int(rng, 10000, 250000), k=min(k, 16),
                    mode="kdtree")
    if kind == "knn":
        return dict(kind="knn", n=_log_int(rng, 1000, 900000), k=min(k, 16), radius=rng.choice([2.0, 5.0, 10.0]))
    if kind == "train":
        return dict(kind="train", rows=_log_int(rng, 20000, 400000), batch=_log_int(rng, 1000, 65000),
                    steps=rng.randint(1, 4))
    if kind == "grad":
        return dict(kind="grad", rows=_log_int(rng, 130, 60000))
    return dict(kind="predict", rows=_log_int(rng, 500, 240000))


# ---- maps and crowds --------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _map(kind, side):
    """(configuration, scene, planner, obstacle index) of a fixed map: "boxes"
    has the box density of workloads.py's 1000 m scene, "crossing" is its
    400 m scene with crossing flows from bands along the four sides"""
    if kind == "crossing":
        cfg = ag.scaled("c3", w=float(side), h=float(side))
    else:
        cfg = ag.scaled("c2", w=float(side), h=float(side), boxes=int(side * side / 250), overlap=True)
    scene = ag.build_scene(cfg, MAP_SEED)
    return cfg, scene, Planner(scene), BoxIndex(scene)


def _crowd(kind, side, n, seed):
    """positions, radii, speeds and paths of n agents.  Up to 65,536 routes are
    planned; further agents share a route and start within 1.5 m of its start,
    as groups do."""
    cfg, scene, planner, boxes = _map(kind, side)
    m = min(n, 65536)
    st = ag.spawn_agents(dict(cfg, agents=m), scene, seed)
    routes = planner.find_paths(st.pos[:m], st.goal[:m], st.clear[:m], cap=128)
    routes = [p if p is not None else np.stack([st.pos[i], st.goal[i]]) for i, p in enumerate(routes)]
    if n == m:
        return scene, st.pos[:m], st.clear[:m], st.pref_speed[:m], routes
    rng = np.random.default_rng(seed + 31)
    of = np.arange(n) % m
    room = boxes.clearance(st.pos[:m, 0], st.pos[:m, 1], reach=2.5) - 0.35
    r = np.clip(0.8 * room, 0.0, 1.5)[of] * np.sqrt(rng.random(n))
    a = rng.random(n) * 2 * np.pi
    pos = st.pos[:m][of] + np.stack([r * np.cos(a), r * np.sin(a)], 1)
    return (scene, pos.astype(np.float32), rng.uniform(0.2, 0.35, n).astype(np.float32),
            rng.uniform(1.2, 1.5, n).astype(np.float32), [routes[i] for i in of])


def _kept(sim):
    return dict(position=sim.get_position_data(), velocity=sim.get_velocity_data(),
                attraction=sim.get_attraction_point_data())


class _View(np.ndarray):
    """a host array of the simulator's, which stays alive with it"""


def _views(sim, *fields):
    out = {}
    for f in fields:
        out[f] = sim.view(f).view(_View)
        out[f].owner = sim
    return out


# ---- the cases --------------------------------------------------------------
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, int(seed))


def run(state):
    return state["run"](state)


def _prepare_tick(case, seed):
    """a running simulation, two ticks old, whose host arrays follow it"""
    n, mode = case["agents"], case["mode"]
    scene, pos, clear, speed, paths = _crowd(case["map"], case["side"], n, seed)
    slots = n + n // 2 if mode == "spawn" else n
    sim = Simulator(scene, slots, DT, max_neighbors=case["k"], **ORCA)
    sim.add_agents(pos, clear, speed, paths)
    s = dict(sim=sim, run=_run_tick)
    if mode == "kdtree":
        set_neighbor_mode(sim, "kdtree")
    elif mode == "learned":
        s["model"] = ProposalModel()
        s["model"].load(TRAINED)
        sim.set_proposal(s["model"])
        sim.set_proposal_gate(0.0)
    elif mode == "spawn":
        add_spawn_areas(sim, scene, rate=60.0, seed=seed)
        rng = np.random.default_rng(seed + 5)
        sim.push_spawn_random(rng.integers(0, 2**31 - 1, 400000, dtype=np.int32))
    sim.set_host_mirror(True)
    sim.update(ticks=2)
    return s


def _run_tick(s):
    sim = s["sim"]
    sim.update()
    return dict(_views(sim, "position", "velocity", "active"), agents=sim.get_num_agents())


def _prepare_rollout(case, seed):
    scene, pos, clear, speed, paths = _crowd(case["map"], case["side"], case["agents"], seed)
    sim = Simulator(scene, case["agents"], DT, max_neighbors=case["k"], **ORCA)
    sim.add_agents(pos, clear, speed, paths)
    sim.update(ticks=2)
    return dict(sim=sim, at=_kept(sim), ticks=case["ticks"], run=_run_rollout)


def _prepare_batch(case, seed):
    n_sc = case["scenes"]
    sides = [(60, 100, 150, 200)[i % 4] for i in range(n_sc)]
    share = 10.0 ** (np.arange(n_sc) * 7 % n_sc / n_sc) # tenfold between the smallest crowd and the largest
    counts = np.maximum(20, np.round(case["agents"] * share / share.sum())).astype(int)
    crowds = [_crowd("boxes", side, int(c), seed + 101 * i) for i, (side, c) in enumerate(zip(sides, counts))]
    sim = BatchSimulator([c[0] for c in crowds], counts, DT, max_neighbors=case["k"], **ORCA)
    for i, c in enumerate(crowds):
        sim.add_agents(*c[1:], scene=i)
    sim.update(ticks=2)
    return dict(sim=sim, at=_kept(sim), ticks=case["ticks"], run=_run_rollout)


def _run_rollout(s):
    """back to the given state, `ticks` ticks, the state read back"""
    sim = s["sim"]
    for field, value in s["at"].items():
        sim.set_state(field, value)
    sim.update(ticks=s["ticks"])
    return _views(sim, "position", "velocity", "attraction", "active")


def _prepare_knn(case, seed):
    """points at 6 per square metre, a third of them in groups; 2 % inactive"""
    n = case["n"]
    side = float(np.sqrt(n / 6.0))
    g = torch.Generator(device="cuda").manual_seed(seed)
    pos = torch.rand((n, 2), generator=g, device="cuda") * side
    m = n // 3
    c = torch.randint(0, m, (m,), generator=g, device="cuda") // 20 * 20
    pos[:m] = (pos[c] + torch.randn((m, 2), generator=g, device="cuda") * 1.5).clamp(0.0, side)
    active = (torch.rand(n, generator=g, device="cuda") >= 0.02).to(torch.uint8)
    lib = _lib.load()
    cell = float(np.sqrt(case["k"] / 6.0)) * 0.5
    box = tuple(map(ctypes.c_float, (0.0, 0.0, side, side, cell)))
    scratch = torch.empty(lib.ecmg_knn_scratch_bytes(n, *box), dtype=torch.uint8, device="cuda")
    ids = torch.zeros((n, case["k"]), dtype=torch.int32, device="cuda")
    count = torch.zeros(n, dtype=torch.int32, device="cuda")
    return dict(lib=lib, pos=pos, active=active, box=box, scratch=scratch, ids=ids, count=count, n=n, k=case["k"],
                radius=case["radius"], run=_run_knn)


def _run_knn(s):
    rc = s["lib"].ecmg_knn(s["pos"].data_ptr(), s["active"].data_ptr(), s["n"], s["k"], s["radius"], *s["box"],
                           s["ids"].data_ptr(), s["count"].data_ptr(), s["scratch"].data_ptr(), s["scratch"].numel(),
                           torch.cuda.current_stream().cuda_stream)
    if rc:
        raise RuntimeError(f"ecmg_knn: {rc}")
    return dict(ids=s["ids"], count=s["count"])


def _weights(seed):
    """He-style initial weights"""
    rng = np.random.default_rng(seed)
    return np.concatenate([(rng.standard_normal(shp) * np.sqrt(2.0 / shp[0])).reshape(-1) if len(shp) == 2
                           else np.zeros(shp) for _, shp in param_layout()]).astype(np.float32)


def _rows(n, seed):
    """feature rows like the tick's (16 neighbours x 5, preferred velocity,
    zero padding) and labels with its class frequencies"""
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn((n, N_IN), generator=g, device="cuda") * 0.4
    x[:, 82:] = 0.0
    p = torch.full((N_OUT,), 0.0, device="cuda")
    p[0], p[1:17], p[17:137], p[137:153], p[153] = 0.57, 0.29 / 16, 0.09 / 120, 0.03 / 16, 0.02
    y = torch.multinomial(p, n, replacement=True, generator=g).to(torch.uint8)
    return x.to(torch.bfloat16), y


def _model(seed):
    m = ProposalModel()
    m.set_params(_weights(seed))
    return m


def _prepare_train(case, seed):
    x, y = _rows(case["rows"], seed)
    return dict(model=_model(seed), x=x, y=y, steps=case["steps"], batch=case["batch"], seed=seed, run=_run_train)


def _run_train(s):
    loss, acc = s["model"].train(s["x"], s["y"], steps=s["steps"], batch=s["batch"], lr=1e-3, seed=s["seed"])
    return dict(loss=loss, weights=s["model"].get_params())


def _prepare_grad(case, seed):
    x, y = _rows(case["rows"], seed)
    return dict(model=_model(seed), x=x, y=y, run=_run_grad)


def _run_grad(s):
    loss, grad = s["model"].loss_grad(s["x"], s["y"])
    return dict(loss=loss, grad=grad)


def _prepare_predict(case, seed):
    x, _ = _rows(case["rows"], seed)
    m = ProposalModel()
    m.load(TRAINED)
    return dict(model=m, x=x, run=_run_predict)


def _run_predict(s):
    return s["model"].predict(s["x"])


# ---- 64-bit values ----------------------------------------------------------
def _net64(flat):
    return {k: torch.from_numpy(np.array(v)).double().cuda().requires_grad_() for k, v in split_params(flat).items()}


def _loss64(P, x, y):
    a = torch.nn.functional.gelu(x @ P["W1"] + P["b1"], approximate="tanh")
    a = torch.nn.functional.gelu(a @ P["W2"] + P["b2"], approximate="tanh")
    return torch.nn.functional.cross_entropy(a @ P["W3"] + P["b3"], y.long())


def _flat(P, grad=False):
    return torch.cat([(P[n].grad if grad else P[n].detach()).reshape(-1) for n, _ in param_layout()]).cpu().numpy()


def _minibatch(n, batch, seed):
    """the training's rows: splitmix64 of the seed and the row, modulo n"""
    with np.errstate(over="ignore"):
        z = np.uint64(seed) + np.uint64(0x9E3779B97F4A7C15) * np.arange(1, batch + 1, dtype=np.uint64)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        z ^= z >> np.uint64(31)
    return torch.from_numpy((z % np.uint64(n)).astype(np.int64)).cuda()


def exact(case, seed):
    """Ticks have no 64-bit value: which half-planes are active, and so where
    an agent goes, is decided on the rounded 32-bit numbers (tests/ hold them to
    the oracle bit for bit).  Neighbour ids and classes are whole numbers."""
    seed = int(seed)
    if case["kind"] == "grad":
        x, y = _rows(case["rows"], seed)
        P = _net64(_weights(seed))
        loss = _loss64(P, x.double(), y)
        loss.backward()
        return dict(loss=float(loss), grad=_flat(P, grad=True))
    if case["kind"] == "train":
        x, y = _rows(case["rows"], seed)
        P = _net64(_weights(seed))
        opt = torch.optim.Adam(P.values(), lr=1e-3, betas=(0.9, 0.999), eps=1e-8)
        losses = []
        for it in range(case["steps"]):
            i = _minibatch(case["rows"], case["batch"], seed + 0x51ED27 * (it + 1))
            opt.zero_grad()
            loss = _loss64(P, x[i].double(), y[i])
            loss.backward()
            opt.step()
            losses.append(float(loss))
        return dict(loss=np.array(losses), weights=_flat(P))
    return None


# ---- what a pass cannot do without ------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("tick", "rollout", "batch"):
        n, k = case["agents"], case["k"]
        t = case.get("ticks", 1)
        # per agent and tick: position, velocity, radius, speed, flag, attraction
        # point and path record in, position, velocity, attraction point and
        # preferred velocity out; once per pass the arrays handed to the program
        b = n * t * (8 + 8 + 4 + 4 + 1 + 8 + 8 + 32) + n * (16 if kind == "tick" else 24 + 24)
        # per neighbour: distance, half-plane, one step of the linear program
        return dict(bytes=b, flops=n * t * k * 120)
    if kind == "knn":
        return dict(bytes=case["n"] * (8 + 1 + 4 * case["k"] + 4), flops=case["n"] * case["k"] * 5)
    weights = N_IN * N_HID + N_HID * N_HID + N_HID * N_OUT
    if kind == "predict":
        return dict(bytes=case["rows"] * (2 * N_IN + 1) + 4 * weights, flops=2 * weights * case["rows"])
    rows, steps = (case["batch"], case["steps"]) if kind == "train" else (case["rows"], 1)
    return dict(bytes=steps * (rows * (2 * N_IN + 1) + 4 * weights * (6 if kind == "train" else 2)),
                flops=6 * weights * rows * steps)
