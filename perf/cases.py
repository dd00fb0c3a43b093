"""The calls whose speed counts, as a program makes them.

Eight kinds of work, each through the public entry points of b12_b200: the subdivision
driver one call at a time, whole subdivision jobs with their transition matrix and
invariant measure, unstable-manifold continuations, parameter scans, selective refinement
(leaves of several depths), matrices of stored box coverings, insertions of points, power
iterations on larger matrices, and bursts of jobs on the server.  A long-running program
keeps its trees, matrices, batches, servers and result buffers; the results it reads are
copied to pinned host memory, or left on the device where the next step would use them.
Result buffers hold more than a job of their size gives; the room behind a result stays zero.
"""
import math

import numpy as np
import torch

import b12_b200 as B
from b12_b200 import workloads as W
from b12_b200.server import JobServer, stream_job_args

DUFFING_CENTER, DUFFING_RADIUS = (0.0,) * 4, (2.0,) * 4
DOMAIN = {"henon": (W.HENON_CENTER, W.HENON_RADIUS), "lorenz": (W.LORENZ_CENTER, W.LORENZ_RADIUS),
          "forced": (W.FORCED_CENTER, W.FORCED_RADIUS)}


def listed():
    return [
        # the smallest calls: the documented driver loop call by call on a small Henon tree
        {"name": "henon_steps_d12", "kind": "steps", "map": "henon", "fma": False, "depth": 12, "grid": 4},
        # the reference's introductory job: 20 steps and the matrix
        {"name": "henon_job_d20", "kind": "job", "map": "henon", "fma": False, "depth": 20, "grid": 4, "iters": 0},
        # an ordinary job with the default (strict) arithmetic
        {"name": "lorenz_job_d22_strict", "kind": "job", "map": "lorenz", "fma": False, "depth": 22, "grid": 5,
         "iters": 0},
        # the headline job: depth 27, fused multiply-adds, matrix and 200 power iterations
        {"name": "lorenz_job_d27_fma", "kind": "job", "map": "lorenz", "fma": True, "depth": 27, "grid": 5,
         "iters": 200},
        # a period map of 200 integrator steps per point, the third family of the served stream
        {"name": "forced_job_d19", "kind": "job", "map": "forced", "fma": False, "depth": 19, "grid": 4, "iters": 0},
        # the four-dimensional continuation benchmark: 49 sweeps to ten million boxes
        {"name": "continuation_d24", "kind": "continuation", "depth": 24, "points": 64},
        # a scan over rho: many small instances advanced together
        {"name": "scan_64_d18_25", "kind": "scan", "n": 64, "low": 18, "high": 25, "matrices": False},
        # refinement of half the domain only: leaves of several depths
        {"name": "selective_d20_6", "kind": "selective", "depth": 20, "more": 6, "fma": True},
        # a stored covering of a trajectory loaded from the host, its matrix with lost points kept
        {"name": "matrix_d25", "kind": "matrix", "depth": 25, "boxes": 100000, "grid": 5, "absolute": False,
         "lost": True, "fma": False},
        # two clouds of a million points each inserted into one tree
        {"name": "insert_1m_d24", "kind": "insert", "points": 1000000, "depth": 24},
        # the power iteration on a matrix too large for one chip's shared memory
        {"name": "measure_600k", "kind": "measure", "n": 600000, "points": 16, "iters": 50},
        # a burst of mixed jobs on the server, every result read
        {"name": "served_48", "kind": "served", "jobs": 48},
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["steps", "job", "job", "job", "continuation", "scan", "selective", "matrix", "insert",
                       "measure", "served"])
    if kind == "steps":
        return {"kind": kind, "map": "henon", "fma": False, "depth": rng.randint(6, 20), "grid": rng.randint(2, 5)}
    if kind == "job":
        m = rng.choice(["henon", "lorenz", "lorenz", "forced"])
        low, high = {"henon": (14, 22), "lorenz": (15, 26), "forced": (14, 20)}[m]
        return {"kind": kind, "map": m, "fma": m == "lorenz" and rng.random() < 0.5, "depth": rng.randint(low, high),
                "grid": rng.randint(3, 5) if m == "lorenz" else rng.randint(3, 6), "iters": rng.choice([0, 0, 50, 200])}
    if kind == "continuation":
        return {"kind": kind, "depth": rng.randint(13, 23), "points": rng.randint(20, 64)}
    if kind == "scan":
        matrices = rng.random() < 0.4
        low = rng.randint(12, 18)
        return {"kind": kind, "n": _log(rng, 5, 60), "low": low, "high": low + rng.randint(0, 3 if matrices else 6),
                "matrices": matrices}
    if kind == "selective":
        return {"kind": kind, "depth": rng.randint(14, 20), "more": rng.randint(2, 6), "fma": rng.random() < 0.5}
    if kind == "matrix":
        return {"kind": kind, "depth": rng.randint(15, 30), "boxes": _log(rng, 500, 100000), "grid": rng.randint(2, 5),
                "absolute": rng.random() < 0.5, "lost": rng.random() < 0.5, "fma": rng.random() < 0.5}
    if kind == "insert":
        return {"kind": kind, "points": _log(rng, 1000, 1000000), "depth": rng.randint(10, 40)}
    if kind == "measure":
        return {"kind": kind, "n": _log(rng, 2000, 600000), "points": rng.randint(5, 16), "iters": rng.randint(20, 60)}
    return {"kind": kind, "jobs": _log(rng, 6, 48)}


# ---------------------------------------------------------------- inputs
def _map_args(case, seed):
    """(map parameters, integrator arguments) of a job: the usual parameters, a little moved by the seed."""
    u = float(np.random.default_rng([seed, 7]).uniform(-1.0, 1.0))
    if case["map"] == "henon":
        return (1.4 - 0.01 * abs(u), 0.3)
    if case["map"] == "lorenz":
        return (10.0, 28.0 + 0.1 * u, 8.0 / 3.0)
    return (0.25, -1.0, 1.0, 0.3 + 0.002 * u)


def _scheme(case, seed):
    p = _map_args(case, seed)
    m = {"henon": lambda: B.henon(*p), "lorenz": lambda: B.lorenz(*p, fma=case["fma"]),
         "forced": lambda: B.forced_duffing(200, *p)}[case["map"]]()
    return B.Scheme(m, B.inner_grid(case["grid"]))


def _boxes(case):
    """About how many leaves a job of this kind ends with (they roughly fill the attractor's dimension)."""
    d = case["depth"]
    if case["map"] == "henon":
        return 15000.0 * 2.0 ** (0.63 * (d - 20))
    if case["map"] == "lorenz":
        return 250000.0 * 2.0 ** (0.69 * (d - 27))
    return 27000.0 * 2.0 ** (0.75 * (d - 19))


def _trajectory_boxes(depth, boxes, seed):
    """The boxes of one depth that a set of Lorenz trajectories passes through, about `boxes`
    of them (at most), sorted: what a program that covers simulated data loads."""
    g = np.random.default_rng([seed, 11])
    x = g.normal(size=(3, 4000)) * 5.0 + np.array([[0.0], [0.0], [25.0]])
    c, r = (np.array(v)[:, None] for v in DOMAIN["lorenz"])
    h, got, found = 0.01, [], 0
    f = lambda y: np.stack([10.0 * (y[1] - y[0]), 28.0 * y[0] - y[1] - y[0] * y[2], y[0] * y[1] - 8.0 / 3.0 * y[2]])  # noqa: E731
    k = [depth // 3 + (j < depth % 3) for j in range(3)]
    for step in range(600):
        k1 = f(x)
        k2 = f(x + 0.5 * h * k1)
        k3 = f(x + 0.5 * h * k2)
        x = x + h / 6.0 * (k1 + 2.0 * k2 + 2.0 * k3 + f(x + h * k3))
        if step < 150 or step % 3:
            continue
        u = (x - c) / r * 0.5 + 0.5
        bits = [np.minimum((u[j] * 2.0 ** k[j]).astype(np.uint64), np.uint64(2 ** k[j] - 1)) for j in range(3)]
        code = np.zeros(x.shape[1], dtype=np.uint64)
        for t in range(depth):
            j = t % 3
            code = (code << np.uint64(1)) | ((bits[j] >> np.uint64(k[j] - 1 - t // 3)) & np.uint64(1))
        got.append(code)
    codes = np.unique(np.concatenate(got))
    return np.sort(g.permutation(codes)[:boxes])


def _targets(case, seed):
    """Row-major target boxes of n source boxes with P test points each: an expanding map of
    a line of boxes with a spread, every box mapped over its neighbourhood's image."""
    n, P = case["n"], case["points"]
    g = torch.Generator().manual_seed(seed)
    i = torch.arange(n, dtype=torch.int64)[:, None]
    spread = torch.randint(0, 24, (n, P), generator=g)
    return ((2 * i + spread + (i % 7) * (n // 7)) % n).to(torch.int32)


def _pinned(n, dtype):
    t = {np.uint32: torch.int32, np.uint64: torch.int64, np.uint8: torch.uint8, np.float64: torch.float64}[dtype]
    return torch.zeros(max(int(n), 1), dtype=t, pin_memory=True).numpy().view(dtype)


def _matrix_room(rows, nnz):
    return {"rowptr": _pinned(rows + 1, np.uint32), "cols": _pinned(nnz, np.uint32), "vals": _pinned(nnz, np.float64),
            "measure": _pinned(rows, np.float64)}


def _leaf_room(n):
    n = int(n)
    return {"codes": torch.zeros(n, dtype=torch.int64, device="cuda"),
            "depth": torch.zeros(n, dtype=torch.uint8, device="cuda"),
            "flags": torch.zeros(n, dtype=torch.uint8, device="cuda")}


def _read_matrix(m, room):
    m.to_host_into(room["rowptr"][:m.n_rows + 1], room["cols"][:m.nnz], room["vals"][:m.nnz])
    return {"shape": np.array([m.n_rows, m.n_cols]), "rowptr": room["rowptr"].view(np.int32),
            "cols": room["cols"].view(np.int32), "vals": room["vals"]}


def _read_leaves(tree, room):
    for to, x in zip((room["codes"], room["depth"], room["flags"]), tree.leaves_device("cuda")):
        to[:len(x)] = x
    return dict(room)


def _put(room, parts):
    """The parts one after another at the start of a kept array."""
    at = 0
    for x in parts:
        room[at:at + len(x)] = x
        at += len(x)
    return room


def _job_room(map_name, depth):
    """Leaves of a job at most, with room to spare."""
    return int(2.0 * _boxes({"map": map_name, "depth": depth})) + 1000


def _continuation_boxes(depth):
    return 9.9e6 * 2.0 ** (0.75 * (depth - 24))


def prepare(case, seed):
    kind = case["kind"]
    g = np.random.default_rng([seed, 3])
    if kind in ("steps", "job"):
        n = _job_room(case["map"], case["depth"])
        s = {"tree": B.ImplicitBoxTree(*DOMAIN[case["map"]]), "scheme": _scheme(case, seed)}
        if kind == "job":
            s.update(matrix=None, leaf_room=_leaf_room(n), room=_matrix_room(n, 9 * n))
        else:
            s["host"] = [np.zeros(n, np.uint64), np.zeros(n, np.uint8), np.zeros(n, np.uint8)]
    elif kind == "continuation":
        s = {"tree": B.ImplicitBoxTree(DUFFING_CENTER, DUFFING_RADIUS), "x0": g.uniform(-1e-3, 1e-3, size=4),
             "scheme": B.Scheme(B.coupled_duffing(), B.philox_grid(case["points"], int(seed) & 0xFFFFFFFF)),
             "counts": np.zeros(1000, np.uint32), "leaf_room": _leaf_room(2 * _continuation_boxes(case["depth"]) + 1000)}
    elif kind == "scan":
        # the depths in use spread evenly over the instances, rho at random
        rho = g.uniform(15.0, 35.0, size=case["n"])
        depth = [case["high"] - i % (case["high"] - case["low"] + 1) for i in range(case["n"])]
        n = sum(_job_room("lorenz", d) for d in depth)
        s = {"batch": B.Batch(*DOMAIN["lorenz"], B.Scheme(B.lorenz(fma=True), B.inner_grid(5)),
                              [(10.0, x, 8.0 / 3.0) for x in rho], depth),
             "host": {"codes": np.zeros(n, np.uint64), "flags": np.zeros(n, np.uint8)}}
        if case["matrices"]:
            s["host"].update(rowptr=np.zeros(n + case["n"], np.uint32), cols=np.zeros(9 * n, np.uint32),
                             vals=np.zeros(9 * n))
    elif kind == "selective":
        job = {"map": "lorenz", "fma": case["fma"], "depth": case["depth"], "grid": 5}
        s = {"tree": B.ImplicitBoxTree(*DOMAIN["lorenz"]), "scheme": _scheme(job, seed),
             "leaf_room": _leaf_room(_job_room("lorenz", case["depth"] + case["more"]))}
    elif kind == "matrix":
        codes = _trajectory_boxes(case["depth"], case["boxes"], seed)
        n = len(codes)
        s = {"tree": B.ImplicitBoxTree(*DOMAIN["lorenz"]), "matrix": None,
             "room": _matrix_room(case["boxes"], 20 * case["boxes"]),
             "scheme": _scheme({"map": "lorenz", "fma": case["fma"], "grid": case["grid"]}, seed),
             "leaves": (codes, np.full(n, case["depth"], np.uint8), np.zeros(n, np.uint8))}
    elif kind == "insert":
        clouds = []
        for _ in range(2):
            p = torch.empty((case["points"], 4), dtype=torch.float64, pin_memory=True).numpy()
            p[:] = np.clip(0.6 * g.standard_normal(size=p.shape, dtype=np.float32), -1.99, 1.99)
            clouds.append(p)
        s = {"tree": B.ImplicitBoxTree(DUFFING_CENTER, DUFFING_RADIUS), "clouds": clouds,
             "leaf_room": _leaf_room(2 * case["points"])}
    elif kind == "measure":
        n = case["n"]
        tree = B.ImplicitBoxTree(*DOMAIN["henon"])
        tree.load_leaves(np.arange(n, dtype=np.uint64), np.full(n, 20, np.uint8), np.zeros(n, np.uint8))
        s = {"matrix": tree.transition_rows(_targets(case, seed).cuda(), case["points"], n),
             "out": _pinned(n, np.float64)}
        tree.close()
    else:
        # the stream's families and depths, with other parameters of its ranges for each seed
        u = g.uniform(size=case["jobs"])
        stream = []
        for j, x in zip(W.job_stream(case["jobs"], 1.0, 0), u):
            if j["family"] == "henon":
                j = dict(j, params=(1.0 + 0.4 * x, 0.3))
            elif j["family"] == "lorenz":
                j = dict(j, params=(10.0, 15.0 + 20.0 * x, 8.0 / 3.0))
            stream.append(j)
        names = {"forced_duffing": "forced"}
        n = sum(_job_room(names.get(j["family"], j["family"]), j["depth"]) for j in stream)
        s = {"server": JobServer(), "stream": stream,
             "host": {"counts": np.zeros(sum(j["depth"] for j in stream), np.uint32), "codes": np.zeros(n, np.uint64),
                      "rowptr": np.zeros(n + len(stream), np.uint32), "cols": np.zeros(9 * n, np.uint32),
                      "vals": np.zeros(9 * n)}}
    s["case"] = case
    return s


# ---------------------------------------------------------------- one pass
def run(s):
    case = s["case"]
    return {"steps": _run_steps, "job": _run_job, "continuation": _run_continuation, "scan": _run_scan,
            "selective": _run_selective, "matrix": _run_matrix, "insert": _run_insert, "measure": _run_measure,
            "served": _run_served}[case["kind"]](s, case)


def _signed(a):
    return a.view({4: np.int32, 8: np.int64}[a.itemsize]) if a.dtype.kind == "u" and a.itemsize > 1 else a


def _run_steps(s, case):
    t, sc, counts = s["tree"], s["scheme"], []
    t.delete_depth(0)
    t.set_flags(B.SD)
    for _ in range(case["depth"]):
        t.subdivide(B.SD)
        t.set_flags_by_image(sc, B.HIT)
        t.remove(B.HIT)
        t.unset_flags(B.HIT)
        counts.append(t.count())
    return [np.array(counts)] + [_signed(_put(room, [x])) for room, x in zip(s["host"], t.leaves())]


def _run_job(s, case):
    t = s["tree"]
    t.delete_depth(0)
    counts = t.subdivision_run(s["scheme"], case["depth"])
    s["matrix"] = m = t.transition_matrix(s["scheme"], into=s["matrix"])
    out = {"counts": _signed(counts), **_read_leaves(t, s["leaf_room"]), **_read_matrix(m, s["room"])}
    if case["iters"]:
        m.invariant_measure(case["iters"], out=s["room"]["measure"][:m.n_rows])
        out["measure"] = s["room"]["measure"]
    return out


def _run_continuation(s, case):
    counts = s["tree"].continuation_run(s["scheme"], s["x0"], case["depth"], max_sweeps=1000)
    return {"counts": _signed(_put(s["counts"], [counts])), **_read_leaves(s["tree"], s["leaf_room"])}


def _run_scan(s, case):
    b, host = s["batch"], s["host"]
    b.run()
    if case["matrices"]:
        b.transition_matrices()
    counts = np.concatenate([b.counts(i) for i in range(b.n)])
    got = [b.leaves(i) for i in range(b.n)]
    out = {"counts": counts, "codes": _put(host["codes"], [x[0] for x in got]),
           "flags": _put(host["flags"], [x[2] for x in got])}
    if case["matrices"]:
        rows = [b.csr(i) for i in range(b.n)]
        for k, name in enumerate(("rowptr", "cols", "vals")):
            out[name] = _put(host[name], [x[k] for x in rows])
    return {k: _signed(v) for k, v in out.items()}


def _run_selective(s, case):
    t, sc, counts = s["tree"], s["scheme"], []
    t.delete_depth(0)
    t.subdivision_run(sc, case["depth"])
    codes, depth, flags = t.leaves()
    lower = (codes >> np.uint64(case["depth"] - 1)) == 0
    t.load_leaves(codes, depth, ((flags & ~np.uint8(B.SD)) | np.where(lower, B.SD, 0)).astype(np.uint8))
    for _ in range(case["more"]):
        t.subdivide(B.SD)
        t.set_flags_by_image(sc, B.HIT)
        t.remove(B.HIT)
        t.unset_flags(B.HIT)
        counts.append(t.count())
    return {"counts": np.array(counts), **_read_leaves(t, s["leaf_room"])}


def _run_matrix(s, case):
    t = s["tree"]
    t.load_leaves(*s["leaves"])
    s["matrix"] = t.transition_matrix(s["scheme"], case["absolute"], case["lost"], into=s["matrix"])
    return _read_matrix(s["matrix"], s["room"])


def _run_insert(s, case):
    t = s["tree"]
    t.delete_depth(0)
    new = [t.insert_points(s["clouds"][0], case["depth"], B.INS),
           t.insert_points(s["clouds"][1], case["depth"], B.INS, B.HIT)]
    return {"new": np.array(new), **_read_leaves(t, s["leaf_room"])}


def _run_measure(s, case):
    return {"measure": s["matrix"].invariant_measure(case["iters"], out=s["out"])}


def _run_served(s, case):
    srv = s["server"]
    ids = [srv.submit(*stream_job_args(j)) for j in s["stream"]]
    srv.wait_all(ids)
    got = []
    for i in ids:
        got.append(srv.result(i))
        srv.release(i)
    return {k: _signed(_put(room, [x[k] for x in got])) for k, room in s["host"].items()}


# ---------------------------------------------------------------- what a pass cannot do without
#: floating-point operations of one image point: every +, *, / of the map counts 1
POINT_FLOPS = {"henon": 5, "lorenz": 1560, "forced": 12800, "duffing": 280}


def work(case):
    kind = case["kind"]
    if kind in ("steps", "job"):
        n, dim = _boxes(case), 3 if case["map"] == "lorenz" else 2
        images = 2.0 * n / (1.0 - 2.0 ** (-0.69)) * 0.63
        nnz = 6.5 * n if kind == "job" else 0.0
        its = case.get("iters", 0)
        return {"bytes": 10.0 * n + 12.0 * nnz + 8.0 * n * (its > 0),
                "flops": images * case["grid"] ** dim * POINT_FLOPS[case["map"]] + 2.0 * nnz * its}
    if kind == "continuation":
        n = _continuation_boxes(case["depth"])
        return {"bytes": 10.0 * n, "flops": n * case["points"] * POINT_FLOPS["duffing"]}
    if kind == "scan":
        mid = [_boxes({"map": "lorenz", "depth": d}) for d in range(case["low"], case["high"] + 1)]
        n = case["n"] * sum(mid) / len(mid) * 0.6
        return {"bytes": 10.0 * n + (80.0 * n if case["matrices"] else 0.0), "flops": 3.3 * n * 125 * POINT_FLOPS["lorenz"]}
    if kind == "selective":
        n = _boxes({"map": "lorenz", "depth": case["depth"]})
        images = n * 3.3 + sum(0.5 * n * (1.0 + 2.0 ** (0.69 * k)) for k in range(1, case["more"] + 1))
        return {"bytes": 10.0 * n * 2.0 ** (0.35 * case["more"]), "flops": images * 125 * POINT_FLOPS["lorenz"]}
    if kind == "matrix":
        n = case["boxes"]
        return {"bytes": 10.0 * n + 12.0 * 8 * n, "flops": n * case["grid"] ** 3 * POINT_FLOPS["lorenz"]}
    if kind == "insert":
        return {"bytes": 2.0 * case["points"] * (32 + 10), "flops": 2.0 * case["points"] * 12}
    if kind == "measure":
        nnz = 0.75 * case["n"] * case["points"]
        return {"bytes": 12.0 * nnz + 16.0 * case["n"], "flops": 2.0 * nnz * case["iters"]}
    n = case["jobs"] * 25000.0
    return {"bytes": 90.0 * n, "flops": n * 2.2 * (125 * POINT_FLOPS["lorenz"] + 2 * 16 * POINT_FLOPS["forced"]) / 3.0}


# ---------------------------------------------------------------- the values in 64 bits, without the library
class _Plain:
    """Subdivision and transition matrices of one depth in plain float64 torch."""

    def __init__(self, name, params, grid):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.name, self.p = name, params
        c, r = DOMAIN[name]
        self.dim = len(c)
        self.c, self.r = [float(x) for x in c], [float(x) for x in r]
        i = torch.arange(grid ** self.dim, device=self.dev)
        self.grid = [((i // grid ** j % grid).double() * 2.0 + 1.0 - grid) / grid for j in range(self.dim)]
        self.P = grid ** self.dim

    def rhs(self, x, cos):
        p = self.p
        if self.name == "lorenz":
            return [p[0] * (x[1] - x[0]), p[1] * x[0] - x[1] - x[0] * x[2], -p[2] * x[2] + x[0] * x[1]]
        return [x[1], -p[0] * x[1] - p[1] * x[0] - p[2] * (x[0] * x[0] * x[0]) + p[3] * cos]

    def image(self, x):
        if self.name == "henon":
            return [1.0 - self.p[0] * x[0] * x[0] + x[1], self.p[1] * x[0]]
        steps, h = (20, 0.01) if self.name == "lorenz" else (200, 2.0 * math.pi / 200)
        at = [math.cos(j * (h * steps / (2 * steps))) for j in range(2 * steps + 1)]
        for s in range(steps):
            k = self.rhs(x, at[2 * s])
            res = [u + h / 6.0 * v for u, v in zip(x, k)]
            for scale, weight, j in ((h / 2.0, h / 3.0, 1), (h / 2.0, h / 3.0, 1), (h, h / 6.0, 2)):
                k = self.rhs([u + scale * v for u, v in zip(x, k)], at[2 * s + j])
                res = [u + weight * v for u, v in zip(res, k)]
            x = res
        return x

    def targets(self, codes, depth):
        """Codes of the boxes that the test points of `codes` land in, -1 outside the domain."""
        k = [depth // self.dim + (j < depth % self.dim) for j in range(self.dim)]
        out = torch.empty(len(codes), self.P, dtype=torch.int64, device=self.dev)
        for a in range(0, len(codes), 1 << 15):
            part = codes[a:a + (1 << 15)]
            bits = [torch.zeros_like(part) for _ in k]
            for t in range(depth):
                bits[t % self.dim] = bits[t % self.dim] * 2 + (part >> (depth - 1 - t) & 1)
            x = []
            for j in range(self.dim):
                rk = self.r[j] * 2.0 ** -k[j]
                mid = (bits[j].double() * 2.0 ** (1 - k[j]) - 1.0) * self.r[j] + self.c[j] + rk
                x.append((mid[:, None] + self.grid[j][None, :] * rk).reshape(-1))
            y = self.image(x)
            inside = torch.ones_like(y[0], dtype=torch.bool)
            code = torch.zeros(y[0].shape, dtype=torch.int64, device=self.dev)
            to = []
            for j in range(self.dim):
                inside &= (y[j] >= self.c[j] - self.r[j]) & (y[j] < self.c[j] + self.r[j])
                u = ((y[j] - self.c[j]) / self.r[j] + 1.0) * 0.5
                to.append(torch.where(inside, u * 2.0 ** k[j], 0.0).floor().long() & (2 ** k[j] - 1))
            for t in range(depth):
                j = t % self.dim
                code = code * 2 + (to[j] >> (k[j] - 1 - t // self.dim) & 1)
            out[a:a + (1 << 15)] = torch.where(inside, code, -1).reshape(-1, self.P)
        return out

    def subdivide(self, depth):
        codes = torch.zeros(1, dtype=torch.int64, device=self.dev)
        for d in range(1, depth + 1):
            codes = (codes[:, None] * 2 + torch.arange(2, device=self.dev)).reshape(-1)
            hit = torch.unique(self.targets(codes, d))
            codes = codes[torch.isin(codes, hit)]
        return codes

    def matrix(self, codes, depth, absolute=False, lost=False):
        """(rows, columns, values) of the transition matrix, row by row, lost points in column n + 1."""
        t = self.targets(codes, depth)
        n = len(codes)
        at = torch.searchsorted(codes, t).clamp_(max=n - 1)
        col = torch.where((codes[at] == t) & (t >= 0), at, n + 1)
        row = torch.arange(n, device=self.dev)[:, None].expand_as(col)
        key, count = torch.unique((row * (n + 2) + col).reshape(-1), return_counts=True)
        if not lost:
            keep = key % (n + 2) < n
            key, count = key[keep], count[keep]
        return key // (n + 2), key % (n + 2), count.double() if absolute else count.double() / self.P


def _plain_measure(n, rows, cols, vals, iters):
    v = torch.full((n,), 1.0 / n, dtype=torch.float64, device=vals.device)
    for _ in range(iters):
        v = torch.zeros_like(v).index_add_(0, cols, vals * v[rows])
        v = v / v.abs().sum()
    return v


def exact(case, seed):
    kind = case["kind"]
    def padded(values, n):
        return torch.nn.functional.pad(values, (0, n - len(values)))

    if kind == "job" and case["depth"] <= 22:
        plain = _Plain(case["map"], _map_args(case, seed), case["grid"])
        codes = plain.subdivide(case["depth"])
        n = _job_room(case["map"], case["depth"])
        rows, cols, vals = plain.matrix(codes, case["depth"])
        out = {"counts": None, "codes": None, "depth": None, "flags": None, "shape": None, "rowptr": None,
               "cols": None, "vals": padded(vals, 9 * n)}
        if case["iters"]:
            out["measure"] = padded(_plain_measure(len(codes), rows, cols, vals, case["iters"]), n)
        return out
    if kind == "matrix":
        plain = _Plain("lorenz", _map_args({"map": "lorenz"}, seed), case["grid"])
        codes = torch.from_numpy(_trajectory_boxes(case["depth"], case["boxes"], seed).view(np.int64)).to(plain.dev)
        vals = plain.matrix(codes, case["depth"], case["absolute"], case["lost"])[2]
        return {"shape": None, "rowptr": None, "cols": None, "vals": padded(vals, 20 * case["boxes"])}
    if kind == "measure":
        n, P = case["n"], case["points"]
        t = _targets(case, seed).long()
        key, count = torch.unique((torch.arange(n)[:, None] * n + t).reshape(-1), return_counts=True)
        if torch.cuda.is_available():
            key, count = key.cuda(), count.cuda()
        return {"measure": _plain_measure(n, key // n, key % n, count.double() / P, case["iters"])}
    return None
