"""What the framework is timed on: whole robust updates of one graph, an online
session, a batch of graphs, and the stages that a program with its data in GPU
memory calls by themselves.

A case is a dict of plain values; `prepare` makes what a program has in hand
before the call from a seed, `run` is one pass through the public entry
points, `work` is what a pass cannot do without, `exact` the same outputs in
64 bits by plain numpy or torch where they are computed numbers.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "kimera-rpgo_gb300"))

from rpgo_gb300 import capi, synth  # noqa: E402
from rpgo_gb300.graph import symbol  # noqa: E402
from rpgo_gb300.params import QUIET, RobustSolverParams  # noqa: E402

# per-factor and per-pair operation counts used by work()
PAIR_FLOPS = {(3, 0): 4600.0, (3, 1): 500.0, (2, 0): 700.0, (2, 1): 200.0}
FACTOR_FLOPS = {3: 3000.0, 2: 500.0}


# ------------------------------------------------------------------ cases
def listed():
    return [
        # a small planar map, as one robot builds in a building: PCM2D and LM, the reference's default solver
        {"name": "update_2d_500_lm", "kind": "update", "dim": 2, "poses": 500, "inliers": 100, "outliers": 20,
         "gnc": False},
        # a short 3D mission, PCM then GNC-TLS: the smallest whole call, where launches and waits count
        {"name": "update_3d_300_gnc", "kind": "update", "dim": 3, "poses": 300, "inliers": 60, "outliers": 20,
         "gnc": True},
        # an ordinary 3D map, PCM then GNC-TLS (the second benchmark graph's sizes)
        {"name": "update_3d_5000_gnc", "kind": "update", "dim": 3, "poses": 5000, "inliers": 1000, "outliers": 333,
         "gnc": True},
        # a large map with a fifth as many closures as poses, PCM then GNC-TLS
        {"name": "update_3d_20000_gnc", "kind": "update", "dim": 3, "poses": 20000, "inliers": 2800,
         "outliers": 1200, "gnc": True},
        # the largest map (the headline graph's sizes) with the default solver, PCM then LM
        {"name": "update_3d_50000_lm", "kind": "update", "dim": 3, "poses": 50000, "inliers": 14000,
         "outliers": 6000, "gnc": False},
        # a robot's online session: a map, then an update per few new keyframes, each re-optimised
        {"name": "session_3d_1000", "kind": "session", "poses": 1000, "inliers": 200, "outliers": 60, "steps": 10,
         "step_poses": 5, "step_closures": 3},
        # Monte-Carlo trials: independent graphs of 200 to 2,000 poses in one call, lock-step form
        {"name": "batch_joint_16", "kind": "batch", "graphs": 16, "most": 2000, "joint": True},
        # the odometry chain with its covariances, a whole mission at once
        {"name": "trajectory_3d_20000", "kind": "trajectory", "dim": 3, "count": 20000},
        # all pairs of a group of closures, 3D with covariances (the default test), an odd count
        {"name": "pairwise_3d_4001", "kind": "pairwise", "dim": 3, "mode": 0, "poses": 8000, "n": 4001},
        # new rows only, 2D, as an incremental user adds closures to a group
        {"name": "pairwise_2d_rows", "kind": "pairwise", "dim": 2, "mode": 0, "poses": 4000, "n": 3000,
         "row_begin": 2000},
        # the greedy clique of a large group's consistency matrix
        {"name": "clique_6000", "kind": "clique", "poses": 15000, "n": 6000},
        # one training step of the closure network at the trainer's batch size
        {"name": "mlp_train_8192", "kind": "mlp_train", "n": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["update", "update", "update", "session", "batch", "trajectory", "pairwise", "clique",
                       "mlp_train"])
    if kind == "update":
        dim = rng.choice([2, 3, 3])
        gnc = rng.random() < 0.6
        n = _log_int(rng, 150, 4000 if dim == 2 else (12000 if gnc else 30000))
        lc = max(4, int(n * rng.uniform(0.10, 0.30)))
        out = int(lc * rng.uniform(0.0, 0.4))
        return {"kind": kind, "dim": dim, "poses": n, "inliers": lc - out, "outliers": out, "gnc": gnc}
    if kind == "session":
        n = _log_int(rng, 200, 3000)
        return {"kind": kind, "poses": n, "inliers": n // 5, "outliers": n // 16, "steps": rng.randint(5, 12),
                "step_poses": rng.randint(1, 9), "step_closures": rng.randint(1, 5)}
    if kind == "batch":
        return {"kind": kind, "graphs": rng.randint(5, 24), "most": _log_int(rng, 500, 2500),
                "joint": rng.random() < 0.5}
    if kind == "trajectory":
        return {"kind": kind, "dim": rng.choice([2, 3, 3]), "count": _log_int(rng, 50, 50000)}
    if kind == "pairwise":
        n = _log_int(rng, 60, 7000)
        case = {"kind": kind, "dim": rng.choice([2, 3, 3]), "mode": rng.choice([0, 0, 1]), "n": n,
                "poses": max(200, 2 * n)}
        if rng.random() < 0.4:
            case["row_begin"] = rng.randrange(n)
        return case
    if kind == "clique":
        n = _log_int(rng, 100, 7000)
        return {"kind": kind, "poses": max(200, 2 * n), "n": n}
    return {"kind": kind, "n": _log_int(rng, 200, 20000)}


# ------------------------------------------------------------------ inputs
def _params(case):
    p = RobustSolverParams()
    if case.get("dim", 3) == 2:
        p.setPcm2DParams(1.0, 1.0, QUIET)
    else:
        p.setPcm3DParams(10.0, 5.0, QUIET)
    if case.get("gnc"):
        p.setGncInlierCostThresholdsAtProbability(0.9)
    return p


def _graph(dim, poses, inliers, outliers, seed):
    make = synth.grid2d if dim == 2 else synth.walk3d
    return make(poses, inliers, outliers, seed=seed).graph


class _Part:
    """A graph given by the arrays of the C ABI's layout (what capi.Batch takes)."""

    def __init__(self, arrays):
        self._a = arrays

    def arrays(self):
        return self._a


def _session_parts(case, seed):
    """The map of the first `poses` poses with the closures between them, then
    per step its new poses, their odometry and the closures that reach them."""
    total = case["poses"] + case["steps"] * case["step_poses"]
    extra = case["steps"] * case["step_closures"]
    a = _graph(3, total, case["inliers"] + extra, case["outliers"], seed).arrays()
    n_f, index = len(a["kind"]), lambda k: (k & np.uint64((1 << 56) - 1)).astype(np.int64)
    # the step in which a factor (a pose) arrives: 0 for the map
    newest = np.where(a["kind"] == 0, np.maximum(index(a["key1"]), index(a["key2"])), index(a["key1"]))
    step_of = lambda i: np.maximum(0, (i - case["poses"]) // case["step_poses"] + 1)
    f_step, v_step = step_of(newest), step_of(index(a["value_keys"]))
    # closures of the map's poses that are beyond its own share arrive one by one in the steps
    late = np.flatnonzero((f_step == 0) & (np.arange(n_f) >= total))[case["inliers"] + case["outliers"]:]
    f_step[late] = 1 + np.arange(len(late)) % case["steps"]
    parts = []
    for s in range(case["steps"] + 1):
        f, v = f_step == s, v_step == s
        part = {k: np.ascontiguousarray(a[k][f]) for k in ("kind", "key1", "key2", "measured", "cov", "sqrt_info")}
        part |= {k: np.ascontiguousarray(a[k][v]) for k in ("value_keys", "value_poses")}
        parts.append(capi.Batch(_Part(part)))
    return parts


def _odometry(dim, count, seed):
    """`count` odometry measurements and their covariances (numpy): a random
    walk's increments with noise, each with a covariance scale of its own."""
    rng = np.random.default_rng(seed)
    if dim == 3:
        w = rng.normal(0.0, 0.1, (count, 3))
        th = np.linalg.norm(w, axis=1)[:, None, None]
        K = np.zeros((count, 3, 3))
        K[:, 0, 1], K[:, 0, 2], K[:, 1, 2] = -w[:, 2], w[:, 1], -w[:, 0]
        K[:, 1, 0], K[:, 2, 0], K[:, 2, 1] = w[:, 2], -w[:, 1], w[:, 0]
        R = np.eye(3) + np.sin(th) / th * K + (1.0 - np.cos(th)) / th ** 2 * (K @ K)
        t = np.array([0.5, 0.0, 0.0]) + rng.normal(0.0, 0.02, (count, 3))
        pose = np.concatenate([R.reshape(count, 9), t], axis=1)
        sig = np.array([0.005] * 3 + [0.02] * 3)
    else:
        th = rng.normal(0.0, 0.1, count)
        t = np.array([1.0, 0.0]) + rng.normal(0.0, 0.05, (count, 2))
        pose = np.stack([np.cos(th), np.sin(th), t[:, 0], t[:, 1]], axis=1)
        sig = np.array([0.05, 0.05, 0.01])
    d = len(sig)
    cov = np.zeros((count, d, d))
    cov[:, range(d), range(d)] = (sig * np.exp(rng.normal(0.0, 0.2, (count, 1)))) ** 2
    return pose, cov


def _dev(x):
    return torch.from_numpy(np.ascontiguousarray(x)).cuda()


def _ptr(t):
    return t.data_ptr()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _call(name, *args):
    rc = getattr(capi.load(), name)(*args)
    if rc:
        raise RuntimeError("%s: %d" % (name, rc))


def _chain(dim, mode, pose, cov):
    """A chain's inputs and trajectory arrays on the GPU, slot 0 at the identity."""
    n = len(pose)
    st, d = (12, 6) if dim == 3 else (4, 3)
    s = {"dim": dim, "mode": mode, "count": n,
         "src": torch.arange(n, dtype=torch.int32, device="cuda"),
         "dst": torch.arange(1, n + 1, dtype=torch.int32, device="cuda"),
         "dpose": _dev(pose), "dcov": _dev(cov),
         "pose": torch.zeros(n + 1, st, dtype=torch.float64, device="cuda"),
         "cov": torch.zeros(n + 1, d, d, dtype=torch.float64, device="cuda"),
         "node": torch.zeros(n + 1, dtype=torch.int32, device="cuda"),
         "rot": torch.ones(n + 1, dtype=torch.uint8, device="cuda")}
    s["pose"][0, [0, 4, 8] if dim == 3 else [0]] = 1.0
    return s


def _scan(s):
    _call("rpgo_trajectory_scan_dev", s["dim"], s["mode"], s["count"], _ptr(s["src"]), _ptr(s["dst"]),
          _ptr(s["dpose"]), _ptr(s["dcov"]), _ptr(s["pose"]), _ptr(s["cov"]), _ptr(s["node"]), _ptr(s["rot"]),
          _stream())


def _closures(case, seed):
    """A walk's trajectory and a group of n closures on the GPU: 70 % of them
    true ones, in arrival order."""
    dim, mode, n = case.get("dim", 3), case.get("mode", 0), case["n"]
    out = int(0.3 * n)
    while True:
        a = _graph(dim, case["poses"], n - out, out, seed).arrays()
        odo, lc = case["poses"] - 1, case["poses"]
        if len(a["kind"]) - lc >= n:
            break
        out += n - (len(a["kind"]) - lc)  # a walk with too few close pairs: more false ones instead
    s = _chain(dim, mode, a["measured"][:odo], a["cov"][:odo])
    _scan(s)
    index = lambda k: (k - np.uint64(symbol("a", 0))).astype(np.int32)
    s |= {"n": n, "row_begin": case.get("row_begin", 0), "words": (n + 31) // 32,
          "a": _dev(index(a["key1"][lc:lc + n])), "b": _dev(index(a["key2"][lc:lc + n])),
          "flip": torch.zeros(n, dtype=torch.uint8, device="cuda"),
          "z": _dev(a["measured"][lc:lc + n]), "zc": _dev(a["cov"][lc:lc + n]),
          # PCM's thresholds: a Mahalanobis distance, or mean metres and radians per pose
          "th": ((5.0 if dim == 3 else 1.0), 0.0) if mode == 0 else (0.01, 0.002)}
    s["adj"] = torch.zeros(n, s["words"], dtype=torch.int32, device="cuda")
    return s


def _pairs(s, row_begin):
    _call("rpgo_pairwise_adjacency_dev", s["dim"], s["mode"], s["n"], row_begin, _ptr(s["a"]), _ptr(s["b"]),
          _ptr(s["flip"]), _ptr(s["z"]), _ptr(s["zc"]), _ptr(s["pose"]), _ptr(s["cov"]), _ptr(s["node"]),
          _ptr(s["rot"]), s["th"][0], s["th"][1], _ptr(s["adj"]), s["words"], _stream())


def _mlp_arrays(case, seed):
    """Network parameters, Adam moments of a training in progress, features
    and labels (numpy FP32)."""
    rng, n = np.random.default_rng(seed), case["n"]
    f = lambda *s: rng.standard_normal(s).astype(np.float32)
    x = f(n, 16) * 2.0 + 1.0
    y = (rng.random(n) < 0.89).astype(np.float32)
    p = np.concatenate([np.ones(16, np.float32), np.full(16, 0.5, np.float32), 0.3 * f(1024), 0.1 * f(64),
                        0.15 * f(4096), 0.1 * f(64), 0.2 * f(64), 0.1 * f(1)]).astype(np.float32)
    m, v = 1e-3 * f(5345), (1e-3 * f(5345)) ** 2 + np.float32(1e-8)
    m[:32] = v[:32] = 0.0
    return x, y, p, m, v


# ------------------------------------------------------------------ prepare and run
def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind, "case": case}
    if kind == "update":
        g = _graph(case["dim"], case["poses"], case["inliers"], case["outliers"], seed)
        return s | {"params": _params(case), "graph": capi.Batch(g)}
    if kind == "session":
        return s | {"params": _params(case), "parts": _session_parts(case, seed)}
    if kind == "batch":
        rng = np.random.default_rng(seed)
        graphs = []
        for k in range(case["graphs"]):
            # sizes spread over the range, the same ones for every seed
            n = int(200 + (case["most"] - 200) * (k + 0.5) / case["graphs"])
            lc = int((0.10 + 0.20 * (7 * k % 11) / 10) * n)
            out = int(0.5 * (5 * k % 7) / 6 * lc)
            graphs.append(capi.Batch(_graph(3, n, lc - out, out, int(rng.integers(1 << 30)))))
        return s | {"params": _params({"gnc": True}), "graphs": graphs}
    if kind == "trajectory":
        return s | _chain(case["dim"], 0, *_odometry(case["dim"], case["count"], seed))
    if kind == "pairwise":
        s |= _closures(case, seed)
        if s["row_begin"]:
            _pairs(s, 0)  # the group's earlier rows
        return s
    if kind == "clique":
        s |= _closures(case, seed)
        _pairs(s, 0)
        s["clique"], s["size"] = np.zeros(s["n"], dtype=np.int32), np.zeros(1, dtype=np.int32)
        return s
    x, y, p, m, v = (_dev(t) for t in _mlp_arrays(case, seed))
    return s | {"x": x, "y": y, "p": p, "m": m, "v": v, "grad": torch.zeros_like(p), "step": 100,
                "loss": ctypes.c_double()}


def _padded(w, n):
    """Weights in an array of n entries: how many factors PCM leaves depends on the inputs."""
    out = np.zeros(n)
    out[:len(w)] = w
    return out


def _result(solver, graphs):
    c = solver.counts()
    return {"poses": solver.estimate()[1], "weights": _padded(solver.gnc_weights(), sum(g.f.count for g in graphs)),
            "factors": int(c.num_factors), "inliers": int(c.num_lc_inliers)}


def run(s):
    kind = s["kind"]
    if kind == "update":
        solver = capi.RobustSolver(s["params"])
        if solver.update(s["graph"]):
            raise RuntimeError("update failed")
        return _result(solver, [s["graph"]])
    if kind == "session":
        solver = capi.RobustSolver(s["params"])
        for part in s["parts"]:
            if solver.update(part):
                raise RuntimeError("update failed")
        return _result(solver, s["parts"])
    if kind == "batch":
        res = capi.solve_batch(s["params"], s["graphs"], joint=s["case"]["joint"])
        return {"status": np.array([r[0] for r in res], dtype=np.int32),
                "poses": np.concatenate([r[2] for r in res]),
                "weights": np.concatenate([_padded(r[3], g.f.count) for r, g in zip(res, s["graphs"])])}
    if kind == "trajectory":
        _scan(s)
        return {"pose": s["pose"], "cov": s["cov"]}
    if kind == "pairwise":
        _pairs(s, s["row_begin"])
        return s["adj"]
    if kind == "clique":
        _call("rpgo_max_clique_heu_dev", s["n"], _ptr(s["adj"]), s["words"], 0, -1, s["clique"].ctypes.data,
              s["size"].ctypes.data, _stream())
        return {"size": int(s["size"][0]), "clique": s["clique"]}
    s["step"] += 1
    _call("rpgo_mlp_train_step_dev", _ptr(s["p"]), _ptr(s["m"]), _ptr(s["v"]), s["step"], 1e-3, s["case"]["n"],
          _ptr(s["x"]), _ptr(s["y"]), _ptr(s["grad"]), ctypes.byref(s["loss"]), _stream())
    return {"loss": s["loss"].value, "grad": s["grad"], "params": s["p"], "m": s["m"], "v": s["v"]}


# ------------------------------------------------------------------ work
def _update_work(dim, poses, closures, gnc):
    st, d = (12, 6) if dim == 3 else (4, 3)
    factors = poses + closures
    # every graph is read once and its estimate written; all pairs of its
    # closures; one linearisation and one block factorisation of the chain's
    # own blocks per damped system, for the fewest systems such a solve takes
    # (an LM run of five; under GNC a dozen of them)
    solves = 60 if gnc else 5
    return {"bytes": 8.0 * factors * (st + 2 * d * d + 3) + 8.0 * poses * (2 * st + 1),
            "flops": PAIR_FLOPS[dim, 0] * closures * (closures - 1) / 2
            + solves * (FACTOR_FLOPS[dim] * factors + 6.0 * d ** 3 * (poses + closures))}


def work(case):
    kind = case["kind"]
    if kind == "update":
        return _update_work(case["dim"], case["poses"], case["inliers"] + case["outliers"], case["gnc"])
    if kind == "session":
        w = _update_work(3, case["poses"], case["inliers"] + case["outliers"], False)
        # the pairs once; every step solves the whole graph again
        solve = 5 * (FACTOR_FLOPS[3] + 6.0 * 216) * (case["poses"] + case["inliers"] + case["outliers"])
        return {"bytes": w["bytes"], "flops": w["flops"] + case["steps"] * solve}
    if kind == "batch":
        n = 0.5 * (200 + case["most"])
        w = _update_work(3, n, 0.2 * n, True)
        return {k: case["graphs"] * v for k, v in w.items()}
    st, d = (12, 6) if case.get("dim", 3) == 3 else (4, 3)
    if kind == "trajectory":
        return {"bytes": case["count"] * (2.0 * 8 * (st + d * d) + 9),
                "flops": case["count"] * 2.0 * (2 * d ** 3 + d * d + 36)}
    if kind == "pairwise":
        n, r = case["n"], case.get("row_begin", 0)
        pairs = n * (n - 1) / 2 - r * (r - 1) / 2
        return {"bytes": 8.0 * (n + 2 * n) * (st + d * d) + 4.0 * n * ((n + 31) // 32),
                "flops": PAIR_FLOPS[case["dim"], case["mode"]] * pairs}
    if kind == "clique":
        n = case["n"]
        # the matrix read once; one AND and population count per row and word for a walk from every vertex's row
        return {"bytes": 4.0 * n * ((n + 31) // 32), "flops": 2.0 * n * ((n + 31) // 32)}
    return {"bytes": 4.0 * (17 * case["n"] + 8 * 5345), "flops": 6.0 * 5184 * case["n"]}


# ------------------------------------------------------------------ exact
def _exact_trajectory(case, seed):
    dim, n = case["dim"], case["count"]
    pose, cov = _odometry(dim, n, seed)
    if dim == 3:
        T, S = np.eye(4), np.zeros((6, 6))
        P, C = np.zeros((n + 1, 12)), np.zeros((n + 1, 6, 6))
        P[0, [0, 4, 8]] = 1.0
        R = pose[:, :9].reshape(n, 3, 3)
        Ri = R.transpose(0, 2, 1)
        ti = -np.einsum("nij,nj->ni", Ri, pose[:, 9:])
        tx = np.zeros((n, 3, 3))
        tx[:, 0, 1], tx[:, 0, 2], tx[:, 1, 2] = -ti[:, 2], ti[:, 1], -ti[:, 0]
        tx[:, 1, 0], tx[:, 2, 0], tx[:, 2, 1] = ti[:, 2], -ti[:, 1], ti[:, 0]
        A = np.zeros((n, 6, 6))
        A[:, :3, :3] = A[:, 3:, 3:] = Ri
        A[:, 3:, :3] = tx @ Ri
        D = np.tile(np.eye(4), (n, 1, 1))
        D[:, :3, :3], D[:, :3, 3] = R, pose[:, 9:]
        for k in range(n):
            T, S = T @ D[k], A[k] @ S @ A[k].T + cov[k]
            P[k + 1, :9], P[k + 1, 9:], C[k + 1] = T[:3, :3].reshape(9), T[:3, 3], S
        return {"pose": P, "cov": C}
    M, S = np.eye(3), np.zeros((3, 3))
    P, C = np.zeros((n + 1, 4)), np.zeros((n + 1, 3, 3))
    P[0, 0] = 1.0
    c, s, x, y = pose.T
    D = np.zeros((n, 3, 3))
    D[:, 0, 0] = D[:, 1, 1] = c
    D[:, 0, 1], D[:, 1, 0], D[:, 0, 2], D[:, 1, 2], D[:, 2, 2] = -s, s, x, y, 1.0
    A = np.linalg.inv(D)
    # Ad of the inverse [[R, (y, -x)], [0, 1]] for the tangent (v_x, v_y, omega)
    A[:, 0, 2], A[:, 1, 2] = A[:, 1, 2].copy(), -A[:, 0, 2].copy()
    for k in range(n):
        M, S = M @ D[k], A[k] @ S @ A[k].T + cov[k]
        P[k + 1], C[k + 1] = (M[0, 0], M[1, 0], M[0, 2], M[1, 2]), S
    return {"pose": P, "cov": C}


def _exact_mlp(case, seed):
    x, y, p, m, v = (torch.from_numpy(t).double() for t in _mlp_arrays(case, seed))
    n = case["n"]
    # the network is defined with its weights rounded to BF16, its biases not
    r = lambda t: t.float().bfloat16().double()
    W1, b1 = r(p[32:1056]).view(64, 16), p[1056:1120]
    W2, b2 = r(p[1120:5216]).view(64, 64), p[5216:5280]
    W3, b3 = r(p[5280:5344]), p[5344]
    xn = (x - p[:16]) * p[16:32]
    h1 = (xn @ W1.T + b1).clamp(min=0)
    h2 = (h1 @ W2.T + b2).clamp(min=0)
    z = h2 @ W3 + b3
    loss = (z.clamp(min=0) - z * y + torch.log1p(torch.exp(-z.abs()))).mean()
    dz = (torch.sigmoid(z) - y) / n
    d2 = torch.outer(dz, W3) * (h2 > 0)
    d1 = (d2 @ W2) * (h1 > 0)
    g = torch.cat([torch.zeros(32, dtype=torch.float64), (d1.T @ xn).reshape(-1), d1.sum(0), (d2.T @ h1).reshape(-1),
                   d2.sum(0), h2.T @ dz, dz.sum().reshape(1)])
    step, lr = 101, 1e-3
    t = slice(32, None)
    m, v, p = m.clone(), v.clone(), p.clone()
    m[t], v[t] = 0.9 * m[t] + 0.1 * g[t], 0.999 * v[t] + 0.001 * g[t] ** 2
    p[t] -= lr * (m[t] / (1 - 0.9 ** step)) / ((v[t] / (1 - 0.999 ** step)).sqrt() + 1e-8)
    return {"loss": float(loss), "grad": g, "params": p, "m": m, "v": v}


def exact(case, seed):
    if case["kind"] == "trajectory":
        return _exact_trajectory(case, seed)
    if case["kind"] == "mlp_train":
        return _exact_mlp(case, seed)
    # adjacency bits and clique indices are whole numbers; an update's estimate is the iterate at which hundreds of
    # damped solves stop, which takes a second solver and minutes
    return None
