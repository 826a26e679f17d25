"""The framework's workloads as measurable cases.

A case names a family (``what``) and its sizes and options; ``prepare``
builds what a program holds before the call (scene handle, inputs, graph),
``run`` makes the calls.  Families:

``nodes``    a planner's own loop: ``indicator(q)`` for one sampled node after
             the other, host in, host out (latency).
``vertices`` one batched vertex check, device or host buffers.
``edges``    one batched edge check (roadmap candidates: the k nearest free
             neighbours of free samples, or short random edges as a growing
             tree proposes them), device or host buffers.
``batch``    many independent problems: the captured vertex and edge checks
             of all of them.
``knn``      index a roadmap's nodes and find every node's k nearest.
``predict``  collision-probability inference.
``train``    a predictor trained from given initial weights.
``plan``     a whole multi-query planning call (lazy or plain roadmap).

Scenes, samples, weights and queries all come from the seed.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from gpuprm_b200 import GPRM_EDGES_ALL_STEPS, GPRM_EDGES_EARLY_EXIT, GPRM_MODE_FAST, GPRM_MODE_FP64_BAND, scenes
from gpuprm_b200.batch import CONFIGS, EDGES, ProblemBatch, offsets_of
from gpuprm_b200.configspace import RobotConfigspace
from gpuprm_b200.mlp import CollisionMLP, param_shapes
from gpuprm_b200.neighbours import NeighbourIndex, knn_pairs
from gpuprm_b200.planner import lazy_prm, make_queries, plain_prm

DEV = "cuda:0"
NDOF = {"box4": 4, "hull6": 6, "wall7": 7}
PAIRS = {"box4": 67, "hull6": 394, "wall7": 4117}
FREE = {"box4": 0.85, "hull6": 0.46, "wall7": 0.37}     # free share of uniform samples, for work()
DQ = {"box4": 0.02, "hull6": 0.01, "wall7": 0.005}      # the resolutions the configurations name


def listed():
    return [
        # the reference's planner checks every sampled node by a call of its own
        dict(name="nodes_box4", what="nodes", scene="box4", fast=False, n=32),
        # one growth step of the drop-in planner: the new nodes' candidate edges, host buffers
        dict(name="edges_step_box4", what="edges", scene="box4", source="tree", n=500, fast=False, early=False,
             host=True),
        # the benchmark's roadmap: the candidate edges of 2^20 samples
        dict(name="edges_hull6_roadmap", what="edges", scene="hull6", source="knn", n=1 << 20, k=10,
             edges=2500000, fast=True, early=False, host=False),
        # a smaller roadmap through the drop-in interface: the reference's exact codes, host buffers
        dict(name="edges_hull6_exact_host", what="edges", scene="hull6", source="knn", n=150001, k=10,
             edges=350003, fast=False, early=False, host=True),
        # cluttered 7-DOF scene, 512 obstacles, fine steps: a part of its roadmap's edges
        dict(name="edges_wall7", what="edges", scene="wall7", source="knn", n=1 << 18, k=16, edges=70001,
             fast=True, early=False, host=False),
        # the sampling phase of a large roadmap
        dict(name="vertices_hull6", what="vertices", scene="hull6", n=1 << 20, fast=True, host=False),
        # the same in the cluttered scene, exact codes, a ragged count
        dict(name="vertices_wall7_exact", what="vertices", scene="wall7", n=100003, fast=False, host=False),
        # many mixed robots and obstacle sets at once, replayed as a planner service does
        dict(name="batch_mixed", what="batch", problems=24, lo=13.0, hi=15.0, fast=True),
        # connecting a large roadmap
        dict(name="knn_6d", what="knn", ndof=6, n=480001, k=10),
        # pruning a planner's samples
        dict(name="predict_1m", what="predict", ndof=6, n=(1 << 20) + 77),
        # training the predictor of a scene
        dict(name="train_128_steps", what="train", ndof=6, n=1 << 18, batch=4096, epochs=2),
        # a whole multi-query plan
        dict(name="plan_lazy_hull6", what="plan", scene="hull6", n=1 << 18, k=10, queries=1000, lazy=True),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["nodes", "vertices", "vertices", "edges", "edges", "edges", "edges", "batch", "knn", "predict",
                       "train", "plan"])
    scene = rng.choice(["box4", "hull6", "hull6", "wall7"])
    fast = rng.random() < 0.6
    if what == "nodes":
        return dict(what=what, scene=scene, fast=fast, n=rng.randint(8, 64))
    if what == "vertices":
        top = {"box4": 1 << 20, "hull6": 1 << 20, "wall7": 1 << 18}[scene]
        return dict(what=what, scene=scene, n=_log(rng, 32, top), fast=fast, host=rng.random() < 0.3)
    if what == "edges":
        if rng.random() < 0.4:
            return dict(what=what, scene=scene, source="tree", n=_log(rng, 16, 40000), fast=fast,
                        early=rng.random() < 0.25, host=rng.random() < 0.5)
        n = {"box4": _log(rng, 2000, 300000), "hull6": _log(rng, 2000, 600000), "wall7": _log(rng, 4000, 260000)}[scene]
        k = rng.choice([6, 10, 16])
        edges = _log(rng, 5000, 30000) if scene == "wall7" else min(int(0.25 * n * k), 1000000)
        return dict(what=what, scene=scene, source="knn", n=n, k=k, edges=edges, fast=fast,
                    early=rng.random() < 0.25, host=rng.random() < 0.3)
    if what == "batch":
        lo = rng.uniform(10.0, 13.0)
        return dict(what=what, problems=rng.randint(6, 24), lo=round(lo, 2), hi=round(lo + 2.0, 2), fast=fast)
    if what == "knn":
        return dict(what=what, ndof=rng.randint(4, 7), n=_log(rng, 1500, 400000), k=rng.choice([5, 10, 16]))
    if what == "predict":
        return dict(what=what, ndof=rng.randint(4, 7), n=_log(rng, 200, 1 << 20))
    if what == "train":
        batch = rng.choice([1024, 2048, 4096])
        return dict(what=what, ndof=rng.randint(4, 7), n=batch * rng.randint(4, 48) + rng.randint(0, 500), batch=batch,
                    epochs=rng.randint(1, 2))
    return dict(what="plan", scene=rng.choice(["box4", "hull6"]), n=_log(rng, 4000, 200000), k=10,
                queries=_log(rng, 20, 1000), lazy=rng.random() < 0.6)


# ---------------------------------------------------------------- inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _space(scene, dq, fast):
    cs = RobotConfigspace(scene, dq=dq)
    cs.init()
    cs.set_mode(GPRM_MODE_FP64_BAND | (GPRM_MODE_FAST if fast else 0))
    return cs


def _uniform(scene, n, seed):
    """(ndof, n) uniform in the joint box."""
    lo = torch.tensor(scene.mins, device=DEV)[:, None]
    hi = torch.tensor(scene.maxs, device=DEV)[:, None]
    return (lo + (hi - lo) * torch.rand((scene.ndof, n), device=DEV, generator=_gen(seed))).contiguous()


def _free(cs, q):
    codes = torch.empty(q.shape[1], dtype=torch.int32, device=DEV)
    cs.check_configs_device(q, codes)
    return q[:, codes == 0].contiguous()


def _roadmap_edges(cs, q, k, count):
    """The first `count` candidate edges of the roadmap (from the start again where it has fewer)."""
    qf = _free(cs, q)
    i, j = knn_pairs(qf, k)
    pick = torch.arange(count, device=DEV) % i.numel()
    i, j = i[pick], j[pick]
    return qf[:, i].contiguous(), qf[:, j].contiguous()


def _weights(seed, gain=1.0):
    """Weights as a flat float32 vector, uniform +-gain/sqrt(fan-in): 1 is the
    framework's own initial range, 2.5 gives logits of a trained network's size."""
    rng = np.random.default_rng(seed)
    parts = []
    for name, shape in param_shapes():
        fan = 16 if name in ("W1", "b1") else 256
        parts.append(gain * rng.uniform(-1.0, 1.0, int(np.prod(shape))) / math.sqrt(fan))
    return np.concatenate(parts).astype(np.float32)


def _configs(ndof, n, seed):
    return ((torch.rand((ndof, n), device=DEV, generator=_gen(seed)) * 2 - 1) * math.pi).contiguous()


def _labels(q):
    """A learnable stand-in for a scene's verdicts: the tip of a planar arm in a disc or below a line."""
    th = torch.cumsum(q.double(), 0)
    x, y = torch.cos(th).sum(0), torch.sin(th).sum(0)
    return ((x * x + y * y < 1.5) | (y < -1.0)).float().contiguous()


def prepare(case, seed):
    what = case["what"]
    if what in ("nodes", "vertices", "edges", "plan"):
        scene = scenes.make_scene(case["scene"], seed % 100003)
        cs = _space(scene, DQ[case["scene"]], case.get("fast", True))
        s = dict(what=what, cs=cs, scene=scene)
        if what == "nodes":
            s["q"] = scenes.uniform_configs(scene, case["n"], seed + 1)
        elif what == "vertices":
            q = _uniform(scene, case["n"], seed + 1)
            s["host"] = case["host"]
            if case["host"]:
                s["q"] = q.cpu().numpy().reshape(-1)
                s["res"] = np.zeros(case["n"], np.int32)
            else:
                s["q"] = q
                s["res"] = torch.empty(case["n"], dtype=torch.int32, device=DEV)
            s["n"] = case["n"]
        elif what == "edges":
            cs.set_edge_policy(GPRM_EDGES_EARLY_EXIT if case["early"] else GPRM_EDGES_ALL_STEPS)
            if case["source"] == "tree":
                a, b = scenes.random_edges(scene, case["n"], seed + 1, 0.5)
                qs = torch.tensor(np.ascontiguousarray(a.T), device=DEV)
                qe = torch.tensor(np.ascontiguousarray(b.T), device=DEV)
            else:
                qs, qe = _roadmap_edges(cs, _uniform(scene, case["n"], seed + 1), case["k"], case["edges"])
            n = int(qs.shape[1])
            s.update(host=case["host"], n=n)
            if case["host"]:
                s.update(qs=qs.cpu().numpy().reshape(-1), qe=qe.cpu().numpy().reshape(-1), res=np.zeros(n, np.int32))
            else:
                s.update(qs=qs, qe=qe, res=torch.empty(n, dtype=torch.int32, device=DEV))
        else:
            cs.set_edge_policy(GPRM_EDGES_ALL_STEPS)
            starts, goals = make_queries(cs, scene, case["queries"], seed + 3)
            s.update(starts=starts, goals=goals, n=case["n"], k=case["k"], seed=seed + 4, lazy=case["lazy"])
        return s
    if what == "batch":
        rng = np.random.default_rng(seed)
        spaces, qv, qa, qb = [], [], [], []
        for p in range(case["problems"]):
            scene = scenes.make_mixed((seed * 131 + p) % 1000003)
            cs = _space(scene, 0.01, case["fast"])
            n = int(round(2.0 ** (case["lo"] + (case["hi"] - case["lo"]) * (0.618034 * (p + 1) % 1.0))))
            radius = float(rng.uniform(0.4, 0.8))
            q = _uniform(scene, n, seed * 7 + p)
            a, b = _roadmap_edges(cs, q, 10, int(2.2 * n))
            length = torch.linalg.vector_norm(b - a, dim=0, keepdim=True)
            b = a + (b - a) * torch.clamp(radius / length.clamp(min=1e-30), max=1.0)
            spaces.append(cs)
            qv.append(q)
            qa.append(a)
            qb.append(b)

        def pack(parts, offs):
            out = torch.zeros((7, int(offs[-1])), dtype=torch.float32, device=DEV)
            for x, o in zip(parts, offs[:-1]):
                out[:x.shape[0], int(o):int(o) + x.shape[1]] = x
            return out
        ov, oe = offsets_of([x.shape[1] for x in qv]), offsets_of([x.shape[1] for x in qa])
        pb = ProblemBatch(spaces)
        pb.set_layout(CONFIGS, ov)
        pb.set_layout(EDGES, oe)
        s = dict(what=what, pb=pb, q=pack(qv, ov), qs=pack(qa, oe), qe=pack(qb, oe),
                 rv=torch.empty(int(ov[-1]), dtype=torch.int32, device=DEV),
                 re=torch.empty(int(oe[-1]), dtype=torch.int32, device=DEV))
        torch.cuda.synchronize()
        pb.capture(CONFIGS, s["q"], None, s["rv"])
        pb.capture(EDGES, s["qs"], s["qe"], s["re"])
        return s
    if what == "knn":
        return dict(what=what, x=_configs(case["ndof"], case["n"], seed), index=NeighbourIndex(case["ndof"]),
                    k=case["k"])
    if what == "predict":
        mlp = CollisionMLP(case["ndof"], seed=seed % 1000)
        mlp.set_params(_weights(seed + 1, 2.5))
        return dict(what=what, mlp=mlp, q=_configs(case["ndof"], case["n"], seed))
    q = _configs(case["ndof"], case["n"], seed)
    return dict(what=what, q=q, y=_labels(q), w=_weights(seed + 1), ndof=case["ndof"], batch=case["batch"],
                epochs=case["epochs"])


# ---------------------------------------------------------------- the calls

def run(s):
    what = s["what"]
    if what == "nodes":
        return np.array([s["cs"].indicator(q) for q in s["q"]], np.int32)
    if what == "vertices":
        if s["host"]:
            s["cs"].indicator(s["q"], s["res"], s["n"], s["n"])
        else:
            s["cs"].check_configs_device(s["q"], s["res"])
        return s["res"]
    if what == "edges":
        if s["host"]:
            s["cs"].indicator2(s["qs"], s["qe"], s["res"], s["n"], s["n"])
        else:
            s["cs"].check_edges_device(s["qs"], s["qe"], s["res"])
        return s["res"]
    if what == "batch":
        s["pb"].replay(CONFIGS)
        s["pb"].replay(EDGES)
        return [s["rv"], s["re"]]
    if what == "knn":
        s["index"].build(s["x"])
        idx, dist = s["index"].knn(s["k"])
        return [idx, dist]
    if what == "predict":
        return s["mlp"].predict(s["q"])
    if what == "train":
        mlp = CollisionMLP(s["ndof"], seed=0)
        mlp.set_params(s["w"])
        losses = mlp.train(s["q"], s["y"], epochs=s["epochs"], batch=s["batch"], lr=1e-3, seed=5)
        return [mlp.get_params(), losses]
    plan = lazy_prm if s["lazy"] else plain_prm
    r = plan(s["cs"], s["scene"], s["starts"], s["goals"], s["n"], k=s["k"], seed=s["seed"])
    p = r.device_paths
    # the paths one after the other, filled up to a size that does not depend on them
    room = 128 * len(r.success)
    flat = torch.full((max(room, int(p.flat.numel())),), -1, dtype=torch.int32, device=DEV)
    flat[:p.flat.numel()] = p.flat
    points = torch.zeros((flat.numel(), p.verts.shape[1]), dtype=torch.float32, device=DEV)
    points[:p.flat.numel()] = p.verts[p.flat.long()]
    return [r.success, p.length, p.off, flat, points]


# ---------------------------------------------------------------- the work of a pass

def work(case):
    """Bytes: inputs once, outputs once.  Flops: for checks, per configuration
    its forward kinematics (about 100 per joint) and one ball-distance test
    (9) per polytope pair, the least that answers a free check here."""
    what = case["what"]
    if what in ("nodes", "vertices", "edges", "plan"):
        kind = case["scene"]
        d = NDOF[kind]
        per = 100 * d + 9 * PAIRS[kind]
        n = case["n"]
        if what in ("nodes", "vertices"):
            return {"bytes": n * (4 * d + 4), "flops": n * per}
        if what == "edges" and case["source"] == "tree":
            edges, steps = n, n * (1 + 0.25 / DQ[kind])
        else:
            nf = max(2.0, n * FREE[kind])
            edges = 0.6 * nf * min(case["k"], nf - 1)
            ref_n, ref_len = {"box4": (14000, 0.24), "hull6": (484714, 0.70), "wall7": (1550000, 0.83)}[kind]
            mean = ref_len * (ref_n / nf) ** (1.0 / d)
            edges = min(edges, case.get("edges", edges))
            steps = edges * (1 + mean / DQ[kind])
        if what == "edges":
            return {"bytes": edges * (8 * d + 4), "flops": steps * per}
        # a lazy plan has to check at least one edge per vertex; a plain one all of them
        if case["lazy"]:
            steps = steps * n * FREE[kind] / edges
        return {"bytes": n * (4 * d + 4), "flops": n * per + steps * per}
    if what == "batch":
        n = case["problems"] * 2.0 ** (0.5 * (case["lo"] + case["hi"]))
        edges = 2.2 * n
        return {"bytes": n * 32 + edges * 60, "flops": (n + 55 * edges) * (550 + 9 * 300)}
    if what == "knn":
        n, d, k = case["n"], case["ndof"], case["k"]
        return {"bytes": n * (4 * d + 8 * k), "flops": n * 3.0 ** d * 3 * d}
    macs = 2 * case["ndof"] * 256 + 3 * 256 * 256 + 256
    if what == "predict":
        return {"bytes": case["n"] * (4 * case["ndof"] + 4) + 2 * macs, "flops": 2 * macs * case["n"]}
    rows = case["n"] // case["batch"] * case["batch"] * case["epochs"]
    return {"bytes": rows * (4 * case["ndof"] + 8) + 8 * macs, "flops": 6 * macs * rows}


# ---------------------------------------------------------------- the answers in 64 bits

def _gelu(z):
    return 0.5 * z * (1.0 + torch.tanh(math.sqrt(2.0 / math.pi) * (z + 0.044715 * z ** 3)))


def _unflat(w):
    out, o = [], 0
    for _, shape in param_shapes():
        n = int(np.prod(shape))
        out.append(w[o:o + n].reshape(shape))
        o += n
    return out


def _features(q):
    X = torch.zeros((q.shape[1], 16), dtype=torch.float64, device=q.device)
    d = q.shape[0]
    X[:, 0:2 * d:2] = torch.sin(q.double()).T
    X[:, 1:2 * d:2] = torch.cos(q.double()).T
    return X


def _logit(w, X):
    P = _unflat(w)
    h = X
    for l in range(4):
        h = _gelu(h @ P[2 * l].T + P[2 * l + 1])
    return (h @ P[8].T)[:, 0] + P[9]


def exact(case, seed):
    what = case["what"]
    if what == "predict":
        w = torch.tensor(_weights(seed + 1, 2.5), device=DEV, dtype=torch.float64)
        X = _features(_configs(case["ndof"], case["n"], seed))
        return torch.cat([torch.sigmoid(_logit(w, x)) for x in X.split(1 << 17)])
    if what == "knn":
        x = _configs(case["ndof"], case["n"], seed).double()
        n, d, k = case["n"], case["ndof"], case["k"]
        xt = x.T.contiguous()
        out = torch.empty((n, k), dtype=torch.float64, device=DEV)
        rows = max(1, (1 << 28) // n)
        sq = (xt * xt).sum(1)
        for a in range(0, n, rows):
            b = min(n, a + rows)
            near = (sq[a:b, None] + sq[None, :] - 2.0 * (xt[a:b] @ xt.T))
            near[torch.arange(b - a, device=DEV), torch.arange(a, b, device=DEV)] = math.inf
            idx = torch.topk(near, k, dim=1, largest=False).indices
            dist = torch.zeros((b - a, k), dtype=torch.float64, device=DEV)
            for c in range(d):
                dist += (xt[a:b, c, None] - xt[:, c][idx]) ** 2
            out[a:b] = torch.sort(torch.sqrt(dist), dim=1).values
        return [None, out]
    if what == "train":
        q = _configs(case["ndof"], case["n"], seed)
        y = _labels(q).double()
        X = _features(q)
        w = torch.tensor(_weights(seed + 1), device=DEV, dtype=torch.float64)
        g = torch.Generator(device=DEV)
        g.manual_seed(5)
        order = [torch.randperm(case["n"], device=DEV, generator=g) for _ in range(case["epochs"])]
        m, v, t, losses = torch.zeros_like(w), torch.zeros_like(w), 0, []
        for perm in order:
            steps, total = case["n"] // case["batch"], 0.0
            for k in range(steps):
                pick = perm[k * case["batch"]:(k + 1) * case["batch"]]
                w.requires_grad_(True)
                loss = torch.nn.functional.binary_cross_entropy_with_logits(_logit(w, X[pick]), y[pick])
                grad, = torch.autograd.grad(loss, w)
                w = w.detach()
                t += 1
                m = 0.9 * m + 0.1 * grad
                v = 0.999 * v + 0.001 * grad * grad
                w = w - 1e-3 * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
                total += float(loss)
            losses.append(total / steps)
        return [w.cpu().numpy(), np.array(losses)]
    return None
