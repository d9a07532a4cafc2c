"""Workloads for timing the framework through its public entry points.

A case is a dict of plain values; `kind` says which entry points it goes
through:

  step    a host loop that hands the state in, advances it and reads it back:
          Engine.set_state, Engine.step, Engine.get_state.  `scene` is one of
          the repository's configurations (the falling cubes, the chain net,
          the batch of uneven scenes), `form` the solver's option: plain FP64,
          mixed precision, the learned warm start, one step length per contact
          group.
  frame   the drop-in class as the reference's viewer drives it: NewtonAbd
          history in, step(), history, compute_V() and get_contact_points().
  newton  one Newton system of a scene through the handle: energy, gradient
          and increment (Engine.energy, Engine.assemble, Engine.solve), as a
          program that runs its own outer loop calls them.
  pairs   edge-edge candidate pairs of device buffers (abd_ee_pairs_static).
  mlp     the warm-start network on rows of features (Engine.mlp_forward).
  train   one pass of the trainer over a data set (Trainer.epoch).

Geometry is fixed by a case; a seed draws velocities, rows or positions.
"""
import ctypes
import functools
import math
import os

import numpy as np
import torch

from colb_b200 import fixtures, learned, params as P, scene as S
from colb_b200.abd import NewtonAbd
from colb_b200.engine import MLP_IN, MLP_NPARAM, MLP_OUT, Engine, Trainer, load_library

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CHAIN_SCENE = os.path.join(ROOT, "tests", "golden", "chains_scene.npz")
FALL = 15 * P.REFERENCE["dt"]
CAPS = (-5, -6, -7)     # Krylov, Newton and CCD caps end a step with the iterate reached


def listed():
    return [
        # the smallest call: eight cubes falling onto the ground (launches and round trips count)
        dict(name="cubes8", kind="step", scene="cubes", form="fp64", size=8, count=1, steps=8),
        # the reference's own scene with its constants, one viewer frame after another
        dict(name="chain144_frame", kind="frame", links=144, steps=3),
        # an ordinary net, odd side, every interlocked pair in contact from the first step
        dict(name="net9", kind="step", scene="net", form="fp64", size=9, count=1, steps=1),
        # the chain-net configuration at rest: the benchmark's workload
        dict(name="net16_rest", kind="step", scene="net_rest", form="fp64", size=16, count=1, steps=1),
        # the same net in the mixed-precision form
        dict(name="net16_rest_mixed", kind="step", scene="net_rest", form="mixed", size=16, count=1, steps=1),
        # the same net with the learned warm start (features, network, energy-guarded start)
        dict(name="net16_rest_learned", kind="step", scene="net_rest", form="learned", size=16, count=1, steps=1),
        # eight nets in one handle: the batched form of the benchmark
        dict(name="nets8_rest", kind="step", scene="net_rest", form="fp64", size=16, count=8, steps=1),
        # the batched-scenes configuration: 512 uneven scenes of 4..64 cubes and tori, 10,801 bodies
        dict(name="batch512", kind="step", scene="batch", form="fp64", size=512, count=1, steps=2),
        # the largest scene: a Newton system of the landing 4096-sphere pile
        dict(name="pile4096_newton", kind="newton", spheres=4096),
        # allocation-free detection on 64 links' 55,296 edges
        dict(name="pairs55k", kind="pairs", side=8, dist=0.12),
        # the network on a large ragged set of rows
        dict(name="mlp50k", kind="mlp", rows=50021),
        # a training pass with the trainer's usual mini-batch and a short last one
        dict(name="train10k", kind="train", rows=10007, batch=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["cubes", "frame", "net", "net", "nets", "rest", "batch", "batch", "newton", "newton", "pairs",
                       "mlp", "mlp", "train", "train"])
    if what == "cubes":
        return dict(kind="step", scene="cubes", form=rng.choice(["fp64", "mixed"]), size=8, count=_log(rng, 1, 100),
                    steps=rng.randint(1, 8))
    if what == "frame":
        return dict(kind="frame", links=rng.randint(20, 144), steps=rng.randint(1, 3))
    if what == "net":
        return dict(kind="step", scene="net", form=rng.choice(["fp64", "fp64", "learned", "groups"]),
                    size=rng.randint(3, 11), count=1, steps=1)
    if what == "nets":
        return dict(kind="step", scene="net", form=rng.choice(["fp64", "groups"]), size=rng.randint(4, 8),
                    count=rng.randint(2, 6), steps=1)
    if what == "rest":
        form = rng.choice(["fp64", "mixed", "learned"])
        return dict(kind="step", scene="net_rest", form=form, size=16,
                    count=rng.randint(2, 6 if form == "fp64" else 3), steps=1)
    if what == "batch":
        return dict(kind="step", scene="batch", form=rng.choice(["fp64", "mixed"]), size=_log(rng, 5, 500), count=1,
                    steps=rng.randint(1, 2))
    if what == "newton":
        return dict(kind="newton", spheres=_log(rng, 30, 4000))
    if what == "pairs":
        return dict(kind="pairs", side=rng.randint(1, 8), dist=round(rng.uniform(0.02, 0.14), 4))
    if what == "mlp":
        return dict(kind="mlp", rows=_log(rng, 1, 50000))
    batch = rng.choice([64, 100, 256, 512, 777])
    return dict(kind="train", rows=_log(rng, 100, min(10000, 18 * batch)), batch=batch)


# ------------------------------------------------------------------ scenes
@functools.lru_cache(maxsize=None)
def _scenes(scene, size, count):
    """The scenes of a `step` case, without the seed's velocities."""
    if scene == "cubes":
        return [S.config1_cubes(seed=k) for k in range(count)]
    if scene == "net":
        # links 1.5 - 5e-4 apart: every interlocked pair starts within the barrier's reach
        return [S.config2_chain_net(n=size, seed=k, pitch=1.5 - 5e-4) for k in range(count)]
    if scene == "net_rest":
        state, _, seed = fixtures.load_net16()
        return [dict(S.config2_chain_net(n=16, seed=seed), state=state)] * count
    # lowered until the lowest vertex of each scene is 5 mm above the ground: some scenes land in the
    # first steps, the others fall freely
    out = []
    for sc in S.config3_batch(n_scenes=size, seed=0):
        st = sc["state"].copy()
        drop = S.transform(sc)[:, 1].min() - 5e-3
        st[:, [S.ST_NOW + 1, S.ST_NXT + 1]] -= drop
        out.append(dict(sc, state=st))
    return out


@functools.lru_cache(maxsize=None)
def _pile(spheres):
    """The pile while it lands (its stored state), cut to its first spheres."""
    state, _, seed = fixtures.load_pile()
    return dict(S.config5_pile(n=spheres, seed=seed), state=state[:spheres])


@functools.lru_cache(maxsize=None)
def _chain(links):
    """The reference chain scene, cut to its first links, FALL seconds after
    its start: the free links have fallen and turned with the scene's initial
    spin, and meet their neighbours in the next frames."""
    sc = S.load_npz_scene(CHAIN_SCENE)
    st = sc["state"].copy()
    free = np.flatnonzero(sc["mass"] > 0)
    w = np.array([3.0, 3.0, 0.0])
    turn, n = np.linalg.norm(w) * FALL, S.skew(w / np.linalg.norm(w))
    q = np.eye(3) + np.sin(turn) * n + (1 - np.cos(turn)) * n @ n
    for base in (S.ST_NOW, S.ST_NXT):
        st[free, base + 1] -= 5.0 * FALL * FALL
        st[free, base + S.ST_Q:base + S.ST_Q + 9] = q.reshape(9)
        st[free, base + S.ST_V + 1] -= 10.0 * FALL
        st[free, base + S.ST_QD:base + S.ST_QD + 9] = (S.skew(w) @ q).reshape(9)
    sc = dict(sc, state=st)
    if links == len(sc["mass"]):
        return sc
    v = sc["vert_body"] < links
    nv = int(v.sum())
    return dict(sc, xbar=sc["xbar"][:nv], vert_body=sc["vert_body"][:nv],
                edges=sc["edges"][(sc["edges"] < nv).all(1)], mass=sc["mass"][:links],
                inertia_J=sc["inertia_J"][:links], state=sc["state"][:links])


def _with_velocity(sc, dv):
    """The scene's state with dv added to the centre velocities of its dynamic bodies."""
    st = sc["state"].copy()
    dv = dv * (sc["mass"] > 0)[:, None]
    for base in (S.ST_NOW, S.ST_NXT):
        st[:, base + S.ST_V:base + S.ST_V + 3] += dv
    return st


def _step_states(case, scenes, rng):
    out = []
    for sc in scenes:
        nb = len(sc["mass"])
        if case["scene"] == "cubes":
            dv = rng.uniform(-1, 1, (nb, 3)) + [0.0, -1.5, 0.0]
        elif case["scene"] == "batch":
            dv = rng.uniform(-0.5, 0.5, (nb, 3))
        else:
            dv = rng.uniform(-1e-3, 1e-3, (nb, 3))
        out.append(_with_velocity(sc, dv))
    return out


def _rows(rng, n):
    """Features and targets of the scale the trainer normalises them to."""
    x = rng.standard_normal((n, MLP_IN)).astype(np.float32)
    w = rng.standard_normal((MLP_IN, MLP_OUT)).astype(np.float32) / 7
    y = (np.tanh(x @ w) + 0.1 * rng.standard_normal((n, MLP_OUT))).astype(np.float32)
    return x, y


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "step":
        scenes = _scenes(case["scene"], case["size"], case["count"])
        states = _step_states(case, scenes, rng)
        form = case["form"]
        dt = 1.0 / 240.0 if case["scene"] in ("net", "net_rest") else 1.0 / 120.0
        p = P.config_params(dt=dt, precision=1 if form == "mixed" else 0, warm_start=3 if form == "learned" else 0,
                            ls_groups=1 if form == "groups" else 0)
        e = Engine(p, [dict(sc, state=st) for sc, st in zip(scenes, states)])
        if form == "learned":
            net, norm, _ = learned.load()
            e.set_mlp(net, norm)
        start = torch.from_numpy(np.concatenate(states)).pin_memory().numpy()
        out = torch.zeros((e.nb, 48), dtype=torch.float64).pin_memory().numpy()
        return dict(kind=kind, engine=e, start=start, out=out, steps=case["steps"])
    if kind == "frame":
        sc = _chain(case["links"])
        start = _with_velocity(sc, rng.uniform(-0.05, 0.05, (len(sc["mass"]), 3)))
        # the viewer's point buffers
        points = [np.zeros((4096, 4)) for _ in range(case["steps"])]
        return dict(kind=kind, solver=NewtonAbd(P.REFERENCE["dt"], dict(sc, state=start)), start=start, points=points)
    if kind == "newton":
        sc = _pile(case["spheres"])
        start = _with_velocity(sc, rng.uniform(-0.05, 0.05, (len(sc["mass"]), 3)))
        return dict(kind=kind, engine=Engine(P.config_params(), dict(sc, state=start)), start=start)
    if kind == "pairs":
        sc = S.config2_chain_net(n=case["side"], seed=0)
        st = sc["state"].copy()
        st[:, S.ST_NXT:S.ST_NXT + 3] += rng.uniform(-1e-2, 1e-2, (len(st), 3))
        x = torch.from_numpy(S.transform(sc, st)).cuda()
        cap = 16 * len(sc["edges"])
        return dict(kind=kind, lib=load_library(), x=x, edges=torch.from_numpy(sc["edges"]).cuda(), dist=case["dist"],
                    out=torch.zeros((cap, 4), dtype=torch.int32, device="cuda"),
                    n=torch.zeros(1, dtype=torch.int32, device="cuda"))
    if kind == "mlp":
        net, norm, _ = learned.load()
        e = Engine(P.config_params(), S.config1_cubes())
        e.set_mlp(net, norm)
        x = (rng.standard_normal((case["rows"], MLP_IN)) * norm[MLP_IN:2 * MLP_IN] + norm[:MLP_IN]).astype(np.float32)
        return dict(kind=kind, engine=e, x=x)
    x, y = _rows(rng, case["rows"])
    t = Trainer(learned.init_params(seed % 1000))
    t.set_data(x, y)
    return dict(kind=kind, trainer=t, order=rng.permutation(case["rows"]).astype(np.int32), batch=case["batch"])


LR = 5e-4       # the middle of the trainer's cosine schedule


def run(state):
    kind = state["kind"]
    if kind == "step":
        e = state["engine"]
        e.set_state(state["start"])
        e.step(state["steps"], allow=CAPS)
        return e.get_state(out=state["out"])
    if kind == "frame":
        s = state["solver"]
        s.history = state["start"]
        out = []
        for points in state["points"]:
            s.step()
            pts, depth = s.get_contact_points()
            points[:len(pts), :3], points[:len(pts), 3], points[len(pts):] = pts, depth, 0.0
            out.append([s.compute_V(), points])
        return [s.history.view(np.float64).reshape(-1, 48), out]
    if kind == "newton":
        e = state["engine"]
        e.set_state(state["start"])
        energy = e.energy()
        grad, _ = e.assemble(dense=False)
        du, _ = e.solve()
        return [energy, grad, du]
    if kind == "pairs":
        x, edges, out, n = state["x"], state["edges"], state["out"], state["n"]
        ptr = lambda t: ctypes.c_void_p(t.data_ptr())
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        rc = state["lib"].abd_ee_pairs_static(ptr(x), ptr(edges), len(x), len(edges), state["dist"], ptr(out), len(out),
                                              ptr(n), stream)
        if rc != 0:
            raise RuntimeError("abd_ee_pairs_static: %d" % rc)
        return [int(n.item()), out]
    if kind == "mlp":
        return state["engine"].mlp_forward(state["x"])
    t = state["trainer"]
    loss = t.epoch(state["order"], state["batch"], LR)
    return [float(loss), t.params()]


# ------------------------------------------------------------------ work and 64-bit values
def _geometry_bytes(sc):
    return 24 * len(sc["xbar"]) + 4 * len(sc["xbar"]) + 8 * len(sc["edges"]) + 12 * len(sc["tris"])


MACS = MLP_IN * 256 + 2 * 256 * 256 + 256 * MLP_OUT


def work(case):
    kind = case["kind"]
    if kind == "step":
        # every step reads the geometry and the state once and writes the state once
        scenes = _scenes(case["scene"], case["size"], case["count"])
        nb = sum(len(sc["mass"]) for sc in scenes)
        nv = sum(len(sc["xbar"]) for sc in scenes)
        return dict(bytes=case["steps"] * (sum(_geometry_bytes(sc) for sc in scenes) + 2 * 384 * nb), flops=case["steps"] * 18 * nv)
    if kind == "frame":
        sc = _chain(case["links"])
        nv, nb = len(sc["xbar"]), len(sc["mass"])
        return dict(bytes=case["steps"] * (_geometry_bytes(sc) + 2 * 384 * nb + 24 * nv), flops=case["steps"] * 18 * nv)
    if kind == "newton":
        # geometry and state in; gradient, one 12 x 12 block per body and the increment
        sc = _pile(case["spheres"])
        nb = len(sc["mass"])
        return dict(bytes=_geometry_bytes(sc) + nb * (384 + 96 + 1152 + 96), flops=18 * len(sc["xbar"]) + 1152 * nb)
    if kind == "pairs":
        n = case["side"] ** 2
        return dict(bytes=n * (288 * 24 + 864 * 8), flops=0)
    if kind == "mlp":
        n = case["rows"]
        return dict(bytes=4 * n * (MLP_IN + MLP_OUT) + 2 * MLP_NPARAM, flops=2 * MACS * n)
    n, steps = case["rows"], -(-case["rows"] // case["batch"])
    # per row the forward and the two backward products; per mini-batch the weights and both moments in and out
    return dict(bytes=4 * n * (MLP_IN + MLP_OUT) + steps * 24 * MLP_NPARAM, flops=6 * MACS * n)


def _split(p):
    """The parameter blob as four (weight, bias) pairs."""
    out, at = [], 0
    for o, i in ((256, MLP_IN), (256, 256), (256, 256), (MLP_OUT, 256)):
        w = p[at:at + o * i].reshape(o, i)
        at += o * i
        out.append((w, p[at:at + o]))
        at += o
    return out


def _forward(p, x):
    h = x
    layers = _split(p)
    for k, (w, b) in enumerate(layers):
        h = h @ w.T + b
        if k < 3:
            h = torch.nn.functional.gelu(h)
    return h


def exact(case, seed):
    """64-bit values for the network and the trainer; the steps' and systems' reference is the repository's oracle,
    which takes longer than a case may."""
    if case["kind"] == "mlp":
        s = prepare(case, seed)
        net, norm, _ = learned.load()
        norm = torch.from_numpy(norm).double()
        x = (torch.from_numpy(s["x"]).double() - norm[:MLP_IN]) / norm[MLP_IN:2 * MLP_IN]
        y = _forward(torch.from_numpy(net).double(), x)
        return y * norm[2 * MLP_IN + MLP_OUT:] + norm[2 * MLP_IN:2 * MLP_IN + MLP_OUT]
    if case["kind"] == "train":
        rng = np.random.default_rng(seed)
        x, y = (torch.from_numpy(a).double() for a in _rows(rng, case["rows"]))
        order = torch.from_numpy(rng.permutation(case["rows"]))
        p = torch.from_numpy(learned.init_params(seed % 1000)).double().requires_grad_()
        m, v, losses = torch.zeros(MLP_NPARAM).double(), torch.zeros(MLP_NPARAM).double(), []
        for t, at in enumerate(range(0, case["rows"], case["batch"]), 1):
            rows = order[at:at + case["batch"]]
            loss = ((_forward(p, x[rows]) - y[rows]) ** 2).mean()
            g, = torch.autograd.grad(loss, p)
            losses.append(float(loss.detach()))
            m = 0.9 * m + 0.1 * g
            v = 0.999 * v + 0.001 * g * g
            step = (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
            p = (p.detach() - LR * step).requires_grad_()
        return [float(np.mean(losses)), p.detach()]
    return None
