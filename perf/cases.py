"""The work that the speed of this package is judged by, through its public entry points.

A planner calls the expansion for one popped node, for a round of nodes, or for a whole frontier;
it ranks candidates with the surrogate, trains the surrogate, checks candidates lazily, and runs the
search that is built from these.  ``listed()`` has one case for each of these at the sizes of the
package's workloads (``workloads.CONFIGS`` and the search problems of ``bench.py``), ``draw()`` more of
the same ranges.  ``prepare`` makes what a program has in hand before the call, ``run`` is one call.
"""
import math

import numpy as np
import torch

from dynoplan_gb300 import gpu as G
from dynoplan_gb300 import search as S
from dynoplan_gb300 import surrogate as SG
from dynoplan_gb300 import workloads as W

DEV = "cuda:0"

# per robot: steps of a motion, environment, obstacle sides, delta, and the share of all (node, motion)
# pairs that lie in the ball of radius delta / 2 (for the sizes of buffers and the work of a pass)
ROBOTS = {
    "unicycle1": dict(kind=W.UNICYCLE1, steps=(5, 50), extent=(6.0, 6.0), side=(0.2, 1.0), delta=0.3, share=0.0955),
    "car1": dict(kind=W.CAR1, steps=(5, 100), extent=(10.0, 10.0), side=(0.2, 1.5), delta=0.3, share=0.0165),
    "quadrotor": dict(kind=W.QUAD3D, steps=(50, 300), extent=(6.0, 6.0, 3.0), side=(0.2, 1.0), delta=0.8, share=0.127),
    "quad2d": dict(kind=W.QUAD2D, steps=(20, 150), extent=(8.0, 4.0), side=(0.2, 1.0), delta=0.5, share=0.82),
}
HIDDEN, OUT_PAD, FEAT, EMB = 256, 16, 80, 16


def listed():
    return [
        # the plain drop-in: Expander::expand_lazy plus the checks, called for one popped node, host arrays
        dict(name="expand one node", op="expand", robot="car1", P=5000, N=1, obs=80, host=True, fp64=False, gap=True),
        # a round of the batched search: 32 popped nodes of quad2d against 10,000 motions, host arrays
        dict(name="expand search round", op="expand", robot="quad2d", P=10000, N=32, obs=40, host=True, fp64=False, gap=True),
        # a frontier with end states in FP64 and every output, as a FP64 planner keeps them
        dict(name="expand unicycle fp64", op="expand", robot="unicycle1", P=1000, N=10000, obs=30, host=False, fp64=True, gap=True),
        # the headline frontier: 100,000 car-with-trailer nodes x 5,000 motions on the device
        dict(name="expand car", op="expand", robot="car1", P=5000, N=100000, obs=80, host=False, fp64=False, gap=False),
        # the same as a host program gets it: nodes from, and results in, page-locked host memory
        dict(name="expand car host", op="expand", robot="car1", P=5000, N=100000, obs=80, host=True, fp64=False, gap=False),
        # long motions, 3-D, most results: the largest call
        dict(name="expand quadrotor", op="expand", robot="quadrotor", P=5000, N=50000, obs=40, host=False, fp64=False, gap=False),
        # limit_branching_factor over a frontier: the in-ball pairs, then 20 valid motions a node
        dict(name="lazy check car", op="lazy", robot="car1", P=5000, N=30011, obs=80, limit=20),
        # the surrogate over a search round's successors (32 nodes, the next 40 motions of each)
        dict(name="surrogate round", op="forward", P=10000, N=32, pairs=1280),
        # the surrogate over a frontier's candidates
        dict(name="surrogate frontier", op="forward", P=5000, N=100000, pairs=1048576),
        # its inputs for that frontier
        dict(name="node features", op="features", robot="car1", N=100000, obs=80, goal=True),
        # four steps of training, the weights read back
        dict(name="train surrogate", op="train", P=5000, N=20000, batch=65536, steps=4),
        # the whole call: db-A* on a quad2d problem, up to 1,024 expansions
        dict(name="search quad2d", op="search", P=10000, batch=32, expands=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["expand", "expand", "expand", "expand", "expand", "lazy", "forward", "forward", "features", "train", "search"])
    if op == "expand":
        robot = rng.choice(list(ROBOTS))
        most = {"unicycle1": (1000, 10000), "car1": (5000, 100000), "quadrotor": (5000, 50000), "quad2d": (10000, 1500)}[robot]
        host = rng.random() < 0.4
        return dict(op=op, robot=robot, P=_log(rng, 64, most[0]), N=_log(rng, 1, most[1] // (4 if host else 1)),
                    obs=rng.randint(0, 60 if robot in ("unicycle1", "quad2d") else 120), host=host, fp64=rng.random() < 0.3, gap=rng.random() < 0.5)
    if op == "lazy":
        return dict(op=op, robot=rng.choice(["car1", "unicycle1"]), P=_log(rng, 200, 5000), N=_log(rng, 16, 30000),
                    obs=rng.randint(5, 100), limit=rng.randint(5, 30))
    if op == "forward":
        return dict(op=op, P=_log(rng, 64, 10000), N=_log(rng, 1, 100000), pairs=_log(rng, 1, 1048576))
    if op == "features":
        return dict(op=op, robot=rng.choice(list(ROBOTS)), N=_log(rng, 1, 100000), obs=rng.randint(0, 120), goal=rng.random() < 0.5)
    if op == "train":
        return dict(op=op, P=_log(rng, 64, 10000), N=_log(rng, 64, 50000), batch=_log(rng, 256, 65536), steps=rng.randint(1, 6))
    return dict(op=op, P=_log(rng, 1000, 10000), batch=_log(rng, 1, 64), expands=_log(rng, 64, 1024))


# ------------------------------------------------------------------ inputs --

def _canon_gap(m, env, x):
    """smallest separating-axis gap of every state (torch, FP64) to the environment's boxes"""
    t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    c, h = t(0.5 * (env.obs_lo + env.obs_hi)), t(0.5 * (env.obs_hi - env.obs_lo))
    if not len(c):
        return torch.full((len(x),), math.inf, dtype=torch.float64, device=DEV)
    if m.kind == W.QUAD3D:
        d = (x[:, None, :3] - c).abs() - h
        g = torch.where((d.amax(2) <= 0), d.amax(2), d.clamp(min=0).norm(dim=2)) - m.radius
        return g.amin(1)
    parts = [(x[:, 0], x[:, 1], x[:, 2])]
    if m.kind == W.CAR1:
        parts.append((x[:, 0] - m.hitch * x[:, 3].cos(), x[:, 1] - m.hitch * x[:, 3].sin(), x[:, 3]))
    a, b, best = 0.5 * m.box[0], 0.5 * m.box[1], None
    for px, py, th in parts:
        ct, st = th.cos()[:, None], th.sin()[:, None]
        ac, sn, dx, dy = ct.abs(), st.abs(), px[:, None] - c[:, 0], py[:, None] - c[:, 1]
        g = torch.stack([dx.abs() - (a * ac + b * sn + h[:, 0]), dy.abs() - (a * sn + b * ac + h[:, 1]),
                         (dx * ct + dy * st).abs() - (a + h[:, 0] * ac + h[:, 1] * sn),
                         (dy * ct - dx * st).abs() - (b + h[:, 0] * sn + h[:, 1] * ac)]).amax(0).amin(1)
        best = g if best is None else torch.minimum(best, g)
    return best


def _free_nodes(m, env, N, seed):
    """N collision-free frontier states, uniform in position"""
    g = torch.Generator(device=DEV).manual_seed(seed)
    lo, hi = (torch.from_numpy(np.asarray(v, dtype=np.float64)).to(DEV) for v in (env.lo, env.hi))
    out, have = [], 0
    while have < N:
        k = min(max(256, 2 * (N - have)), 65536)
        u = lambda *s: torch.rand(*s, generator=g, device=DEV, dtype=torch.float64)
        z = lambda *s: torch.randn(*s, generator=g, device=DEV, dtype=torch.float64)
        x = torch.zeros((k, m.nx), dtype=torch.float64, device=DEV)
        d = len(env.lo)
        x[:, :d] = lo + (hi - lo) * u(k, d)
        if m.kind == W.QUAD3D:
            q = z(k, 4)
            x[:, 3:7] = q / q.norm(dim=1, keepdim=True)
            x[:, 7:13] = 0.5 * z(k, 6)
        else:
            x[:, 2] = math.pi * (2 * u(k) - 1)
        if m.kind == W.CAR1:
            x[:, 3] = x[:, 2] + 0.25 * math.pi * (2 * u(k) - 1)
        if m.kind == W.QUAD2D:
            x[:, 2] *= 0.1
            x[:, 3:6] = 0.5 * z(k, 3)
        x = x[_canon_gap(m, env, x) > 1e-3]
        out.append(x)
        have += len(x)
    return torch.cat(out)[:N].contiguous()


def _motions(r, P, seed):
    m = W.robot_model(r["kind"])
    if m.kind == W.QUAD2D:  # motions that chain, as the search uses them
        return m, W.make_primitives_hover(m, P, *r["steps"], seed=seed)
    return m, W.make_primitives(m, P, *r["steps"], seed=seed)


def _world(case, seed):
    r = ROBOTS[case["robot"]]
    m = W.robot_model(r["kind"])
    env = W.make_env(r["extent"], case["obs"], *r["side"], seed=seed * 7919 + 7)
    return r, m, env, _free_nodes(m, env, case["N"], seed * 7919 + 13)


def _pairs(case, seed):
    """feature rows (state part, occupancy part), and candidate pairs grouped by motion"""
    g = torch.Generator(device=DEV).manual_seed(seed * 7919 + 29)
    n = case["pairs"] if case["op"] == "forward" else case["batch"] * case["steps"]
    f = torch.zeros((case["N"], FEAT), device=DEV)
    f[:, :4] = 2 * torch.rand((case["N"], 4), generator=g, device=DEV) - 1
    f[:, 13:15] = 2 * torch.rand((case["N"], 2), generator=g, device=DEV) - 1
    f[:, 16:] = (torch.rand((case["N"], FEAT - 16), generator=g, device=DEV) < 0.25).float()
    node = torch.randint(case["N"], (n,), generator=g, device=DEV, dtype=torch.int32)
    prim = torch.randint(case["P"], (n,), generator=g, device=DEV, dtype=torch.int32)
    if case["op"] == "forward":
        prim = prim.sort().values
    coll = (torch.rand(n, generator=g, device=DEV) < 0.6).float()
    ctg = torch.rand(n, generator=g, device=DEV)
    shapes = [("W1", (HIDDEN, 128), 96), ("W2", (HIDDEN, HIDDEN), HIDDEN), ("W3", (HIDDEN, HIDDEN), HIDDEN),
              ("W4", (OUT_PAD, HIDDEN), HIDDEN), ("emb", (case["P"], EMB), 4)]
    weights = {k: torch.randn(s, generator=g, device=DEV) / math.sqrt(fan) for k, s, fan in shapes}
    weights["W4"][2:] = 0
    for i in (1, 2, 3):
        weights["b%d" % i] = 0.05 * torch.randn(HIDDEN, generator=g, device=DEV)
    weights["b4"] = torch.zeros(OUT_PAD, device=DEV)
    return f.to(torch.bfloat16), node, prim, torch.stack([coll, ctg], 1).contiguous(), weights


def _rows(case):
    return min(case["N"] * case["P"], int(1.6 * ROBOTS[case["robot"]]["share"] * case["N"] * case["P"]) + 8192)


def _buffers(case, m):
    cap, fp64, gap, host = _rows(case), case.get("fp64"), case.get("gap"), case.get("host")
    new = lambda shape, dt: torch.zeros(shape, dtype=dt, pin_memory=True) if host else torch.zeros(shape, dtype=dt, device=DEV)
    out = dict(node=new(cap, torch.int32), prim=new(cap, torch.int32), verdict=new(cap, torch.uint8),
               first_invalid=new(cap, torch.int16), end_state=new((cap, m.nx), torch.float64 if fp64 else torch.float32),
               flags=new(cap, torch.uint8))
    if gap:
        out["min_gap"] = new(cap, torch.float32)
    return cap, out


def prepare(case, seed):
    op = case["op"]
    if op in ("expand", "lazy", "features"):
        r, m, env, x = _world(case, seed)
        s = dict(case=case, ctx=G.Context(m), radius=0.5 * r["delta"], N=case["N"], x=x)
        s["ctx"].upload_env(env)
        if op == "features":
            s["goal"] = x[0].cpu().numpy().copy() if case["goal"] else None
            return s
        s["ctx"].upload_primitives(_motions(r, case["P"], seed * 7919)[1])
        s["cap"], s["out"] = _buffers(case, m)
        if case.get("host"):
            s["x"] = torch.empty(x.shape, dtype=x.dtype, pin_memory=True).copy_(x).numpy()
            s["np"] = {k: v.numpy().view({"node": np.uint32, "prim": np.uint32}.get(k, v.numpy().dtype)) for k, v in s["out"].items()}
        else:
            s["ptr"] = {k: v.data_ptr() for k, v in s["out"].items()}
        return s
    if op in ("forward", "train"):
        feat, node, prim, target, weights = _pairs(case, seed)
        rows = 65536 if op == "forward" else case["batch"]
        net = SG.Surrogate(case["P"], max_rows=rows)
        for k, v in weights.items():
            net.set(k, v.cpu().numpy())
        s = dict(case=case, net=net, feat=feat, node=node, prim=prim, target=target)
        if op == "forward":
            s["out"] = torch.empty((case["pairs"], 2), device=DEV)
        else:
            s["parts"] = [tuple(t[i * rows:(i + 1) * rows].contiguous() for t in (node, prim, target)) for i in range(case["steps"])]
        return s
    m, prims = _motions(ROBOTS["quad2d"], case["P"], 1005)
    env, start, goal = W.make_search_problem(m, (8.0, 4.0), (20, 60), (0.2, 1.0), seed=1005 + 17 * seed)
    ctx = G.Context(m)
    ctx.upload_primitives(prims)
    ctx.upload_env(env)
    opts = S.options(0.5, batch=case["batch"], max_expands=case["expands"], time_limit_ms=60000.0)
    return dict(case=case, ctx=ctx, start=start, goal=goal, opts=opts,
                path=(np.zeros(4096, np.int32), np.zeros((4097, m.nx))))


def run(s):
    case = s["case"]
    op, ctx = case["op"], s.get("ctx")
    if op == "expand":
        prec = 1 if case["fp64"] else 0
        if case["host"]:
            r = ctx.expand(s["x"], s["radius"], precision=prec, capacity=s["cap"], outputs=s["np"])
            return {"n_pairs": r["n_pairs"], **s["out"]}  # whole buffers: the rows past n_pairs stay zero
        r = ctx.expand_device(s["x"].data_ptr(), s["N"], s["radius"], s["ptr"], s["cap"], precision=prec)
        return {"n_pairs": r["n_pairs"], **s["out"]}
    if op == "lazy":
        o, p = s["out"], s["ptr"]
        r = ctx.expand_device(s["x"].data_ptr(), s["N"], s["radius"], dict(node=p["node"], prim=p["prim"]), s["cap"], ball_only=True)
        n = r["n_pairs"]
        st = ctx.lazy_check_device(s["x"].data_ptr(), s["N"], n, p["node"], p["prim"],
                                   {k: p[k] for k in ("verdict", "first_invalid", "end_state", "flags")}, case["limit"])
        return {"stats": [st["n_checked"], st["n_valid"], st["n_accepted"]], **o}
    if op == "features":
        return SG.node_features(ctx, s["x"], s["goal"])
    if op == "forward":
        return s["net"].forward(s["feat"], s["node"], s["prim"], s["out"])
    if op == "train":
        loss = [s["net"].train_step(s["feat"], n, p, t, lr=1e-3) for n, p, t in s["parts"]]
        return {"loss": loss, **{k: s["net"].get(k) for k in SG.PARAMS}}
    r, motions, states = S.search(ctx, s["start"], s["goal"], s["opts"])
    n = r["path_len"] if r["solved"] else 0
    s["path"][0][:n], s["path"][1][:n + 1] = motions[:n], states[:n + 1]
    return {"solved": r["solved"], "status": r["status"], "cost": r["cost"], "expands": r["expands"], "nodes": r["nodes"],
            "checked_pairs": r["checked_pairs"], "length": n, "motions": s["path"][0], "states": s["path"][1]}


def work(case):
    op = case["op"]
    if op in ("expand", "lazy"):
        r = ROBOTS[case["robot"]]
        m = W.robot_model(r["kind"])
        L = 0.5 * sum(r["steps"]) + 1
        pairs = max(1.0, r["share"] * case["N"] * case["P"])
        es = 8 if case.get("fp64") else 4
        out = 4 + 4 + 1 + 2 + m.nx * es + 1 + (4 if case.get("gap") else 0)
        tables = min(case["P"], pairs) * L * m.nx * 4
        # a pair's states (half of them before it ends): moved, bounds-tested, one separating-axis test a part
        return dict(bytes=case["N"] * m.nx * 8 + tables + pairs * out, flops=pairs * 0.5 * L * (10 + 20 * m.n_parts))
    if op == "features":
        return dict(bytes=case["N"] * (W.robot_model(ROBOTS[case["robot"]]["kind"]).nx * 8 + FEAT * 2), flops=case["N"] * 64 * 8)
    net = 2 * ((FEAT + EMB) * HIDDEN + 2 * HIDDEN * HIDDEN + 2 * HIDDEN)
    params = HIDDEN * 128 + 2 * HIDDEN * HIDDEN + OUT_PAD * HIDDEN + 3 * HIDDEN + OUT_PAD + case["P"] * EMB
    if op == "forward":
        return dict(bytes=case["N"] * FEAT * 2 + params * 2 + case["pairs"] * 16, flops=case["pairs"] * net)
    if op == "train":
        rows = case["batch"] * case["steps"]
        return dict(bytes=case["N"] * FEAT * 2 + rows * 16 + case["steps"] * params * 32, flops=3 * rows * net)
    r = ROBOTS["quad2d"]
    pairs = r["share"] * case["expands"] * case["P"]
    return dict(bytes=case["P"] * 86 * 24 + pairs * 11, flops=pairs * 0.5 * 86 * 30)


# ------------------------------------------------- the same in plain FP64 --

def _canonical(m, prims):
    """FP64 states of every motion: the stored ones, or the rollout of the stored start"""
    st, off = torch.from_numpy(prims.states).to(DEV), prims.soff()
    if m.kind not in (W.QUAD2D, W.QUAD3D):
        return st, off
    T, P = int(prims.length.max()), prims.P
    U = np.zeros((P, T - 1, m.nu))
    a = prims.aoff()
    for p in range(P):
        U[p, :prims.length[p] - 1] = prims.actions[a[p]:a[p] + prims.length[p] - 1]
    U = torch.from_numpy(U).to(DEV)
    x = st[torch.from_numpy(off).to(DEV)]
    rows = [x]
    for k in range(T - 1):
        u, dt, n = U[:, k], m.dt, x.clone()
        if m.kind == W.QUAD2D:
            acc = (u[:, 0] + u[:, 1]) * m.g * 0.5
            th = x[:, 2] + x[:, 5] * dt
            n[:, :2] = x[:, :2] + x[:, 3:5] * dt
            n[:, 2] = th - 2 * math.pi * torch.floor((th + math.pi) / (2 * math.pi))
            n[:, 3] = x[:, 3] - acc * x[:, 2].sin() * dt
            n[:, 4] = x[:, 4] + (acc * x[:, 2].cos() - m.g) * dt
            n[:, 5] = x[:, 5] + m.ang_gain * m.g * 0.5 * (u[:, 0] - u[:, 1]) * dt
        else:
            f = u * (m.mass * m.g * 0.25)
            lever = m.arm / math.sqrt(2.0)
            sx, sy, sz = ([-1, -1, 1, 1], [-1, 1, 1, -1], [-1, 1, -1, 1])
            tau = torch.stack([c * (f * torch.tensor(v, dtype=f.dtype, device=DEV)).sum(1) for c, v in ((lever, sx), (lever, sy), (m.t2t, sz))], 1)
            qx, qy, qz, qw = x[:, 3], x[:, 4], x[:, 5], x[:, 6]
            am = f.sum(1) / m.mass
            acc = torch.stack([2 * (qx * qz + qy * qw) * am, 2 * (qy * qz - qx * qw) * am, (1 - 2 * (qx * qx + qy * qy)) * am - m.g], 1)
            J, w = torch.tensor(m.inertia, dtype=f.dtype, device=DEV), x[:, 10:13]
            h = 0.5 * dt * w
            a_ = h.norm(dim=1, keepdim=True)
            e, ew = h * torch.sinc(a_ / math.pi), a_[:, 0].cos()
            v, q3 = x[:, 3:6], torch.cross(x[:, 3:6], e, dim=1)
            q = torch.cat([qw[:, None] * e + v * ew[:, None] + q3, (qw * ew - (v * e).sum(1))[:, None]], 1)
            n[:, :3] = x[:, :3] + x[:, 7:10] * dt
            n[:, 3:7] = q / q.norm(dim=1, keepdim=True)
            n[:, 7:10] = x[:, 7:10] + acc * dt
            n[:, 10:13] = w + (tau - torch.cross(w, w * J, dim=1)) / J * dt
        x = n
        rows.append(x)
    X = torch.stack(rows, 1)
    return torch.cat([X[p, :prims.length[p]] for p in range(P)]), off


def _exact_ends(case, seed):
    """end states of the in-ball pairs: motions by falling length, nodes in cell order"""
    r, m, env, x = _world(case, seed)
    prims = _motions(r, case["P"], seed * 7919)[1]
    st, off = _canonical(m, prims)
    lo, hi = (torch.from_numpy(np.asarray(v, dtype=np.float64)).to(DEV) for v in (env.lo, env.hi))
    d, N = len(env.lo), case["N"]
    if N >= 2048:  # Z-order of 64 x 64 (16^3) cells, ascending index in a cell
        bits = 4 if d == 3 else 6
        q = ((x[:, :d] - lo) / (hi - lo)).clamp(0, 1).mul(1 << bits).to(torch.int64).clamp(max=(1 << bits) - 1)
        code = sum((((q[:, i] >> b) & 1) << (d * b + i)) for i in range(d) for b in range(bits))
        x = x[torch.argsort(code, stable=True)]
    ang = lambda a, b: (lambda v: torch.minimum(v, 2 * math.pi - v))((a - b).abs().remainder(2 * math.pi))
    w, radius, out = m.w, 0.5 * r["delta"], []
    V = {W.QUAD2D: slice(3, 5), W.QUAD3D: slice(7, 10)}.get(m.kind)
    t_all = torch.arange(int(prims.length.max()), dtype=torch.float64, device=DEV) * m.dt
    for p in sorted(range(prims.P), key=lambda p: -int(prims.length[p])):
        L, c = int(prims.length[p]), st[int(off[p]):int(off[p]) + int(prims.length[p])]
        s = c[0]
        if m.kind == W.QUAD3D:
            dist = (w[0] * s[:3].norm() + w[1] * torch.acos((x[:, 3:7] @ s[3:7]).abs().clamp(max=1)) + w[2] * s[7:10].norm()
                    + w[3] * (x[:, 10:13] - s[10:13]).norm(dim=1))
        else:
            dist = w[0] * s[:2].norm() + w[1] * ang(x[:, 2], s[2])
            if m.kind == W.CAR1:
                dist = dist + w[2] * ang(x[:, 3], s[3])
            if m.kind == W.QUAD2D:
                dist = dist + w[2] * s[3:5].norm() + w[3] * (x[:, 5] - s[5]).abs()
        y = x[dist <= radius]
        if not len(y):
            continue
        pos = c[None, :, :d] + y[:, None, :d]
        if V is not None:
            pos = pos + t_all[None, :L, None] * y[:, None, V]
        bad = ((pos < lo) | (pos > hi)).any(2)
        e = torch.where(bad.any(1), bad.to(torch.uint8).argmax(1), L - 1)
        end = c[e].clone()
        end[:, :d] = pos[torch.arange(len(y), device=DEV), e]
        if V is not None:
            end[:, V] += y[:, V]
        out.append(end)
    n = sum(len(e) for e in out)
    return torch.cat(out + [torch.zeros((_rows(case) - n, m.nx), dtype=torch.float64, device=DEV)])


def _net(weights, f, node, prim):
    h = torch.cat([f[node.long()], weights["emb"][prim.long()]], 1) @ weights["W1"][:, :FEAT + EMB].T + weights["b1"]
    gelu = lambda z: 0.5 * z * (1 + torch.tanh(math.sqrt(2 / math.pi) * (z + 0.044715 * z ** 3)))
    for i in (2, 3):
        h = gelu(h) @ weights["W%d" % i].T + weights["b%d" % i]
    return (gelu(h) @ weights["W4"].T + weights["b4"])[:, :2]


def exact(case, seed):
    op = case["op"]
    if op == "expand":
        names = ["n_pairs", "node", "prim", "verdict", "first_invalid", "end_state", "flags"] + (["min_gap"] if case["gap"] else [])
        return {k: _exact_ends(case, seed) if k == "end_state" else None for k in names}
    if op == "features":
        r, m, env, x = _world(case, seed)
        lo, hi = (torch.from_numpy(np.asarray(v, dtype=np.float64)).to(DEV) for v in (env.lo, env.hi))
        d, f = len(env.lo), torch.zeros((case["N"], FEAT), dtype=torch.float64, device=DEV)
        f[:, :d] = 2 * (x[:, :d] - lo) / (hi - lo) - 1
        for i in range(d, m.nx):
            planar_angle = m.kind != W.QUAD3D and (i == 2 or (m.kind == W.CAR1 and i == 3))
            raw = m.kind == W.QUAD3D and i < 7
            f[:, i] = ((x[:, i] + math.pi).remainder(2 * math.pi) - math.pi) / math.pi if planar_angle else (x[:, i] if raw else x[:, i] / 4)
        if case["goal"]:
            f[:, 13:13 + d] = 2 * (x[:1, :d] - x[:, :d]) / (hi - lo)
        olo, ohi = (torch.from_numpy(np.asarray(v)).to(DEV) for v in (env.obs_lo, env.obs_hi))
        for c in range(64):
            cen = x[:, :d].clone()
            cen[:, 0] += (c % 8 - 3.5) * 0.75
            cen[:, 1] += (c // 8 - 3.5) * 0.75
            if len(olo):
                f[:, 16 + c] = ((cen[:, None] - 0.375 <= ohi) & (cen[:, None] + 0.375 >= olo)).all(2).any(1).double()
        return f
    if op not in ("forward", "train"):
        return None
    feat, node, prim, target, weights = _pairs(case, seed)
    weights, f, target = {k: v.double() for k, v in weights.items()}, feat.double(), target.double()
    if op == "forward":
        return torch.cat([_net(weights, f, a, b) for a, b in zip(node.split(65536), prim.split(65536))])
    m1 = {k: torch.zeros_like(v) for k, v in weights.items()}
    m2 = {k: torch.zeros_like(v) for k, v in weights.items()}
    losses, B = [], case["batch"]
    for i in range(case["steps"]):
        w = {k: v.clone().requires_grad_() for k, v in weights.items()}
        a, b, t = (v[i * B:(i + 1) * B] for v in (node, prim, target))
        o = _net(w, f, a, b)
        loss = (torch.nn.functional.softplus(o[:, 0]) - t[:, 0] * o[:, 0] + 0.5 * (o[:, 1] - t[:, 1]) ** 2).mean()
        loss.backward()
        losses.append(float(loss.detach()))
        for k in weights:
            g = w[k].grad
            m1[k] = 0.9 * m1[k] + 0.1 * g
            m2[k] = 0.999 * m2[k] + 0.001 * g * g
            step = (m1[k] / (1 - 0.9 ** (i + 1))) / ((m2[k] / (1 - 0.999 ** (i + 1))).sqrt() + 1e-8)
            weights[k] = weights[k] - 1e-3 * step
    return {"loss": losses, **{k: weights[k].detach() for k in SG.PARAMS}}
