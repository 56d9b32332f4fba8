"""The measured workloads of this framework: populations of weighing-matrix
searches through the batch, whole-call and serving entry points, and the exact
batched rescoring.  Every output is a whole number: the same inputs give the
same trajectories, scores and matrices bit for bit.

Populations of `batch` cases are reset to their uploaded starts at the
beginning of a pass, so that each pass is one search from its start.  Where a
replica may solve, it stops at its own solve (stop rule 2), which is the rule
whose results do not depend on launch timing.
"""
import ctypes as C

import numpy as np
import torch

import xtax_b200 as X

# the tempering ladder and candidate rule of the benchmark's populations
LADDER = dict(tempering=1, t_min=0.1, t_init=6.0, objective=0, squared_objective_fraction=0.0,
              parity_objective_fraction=0.0, stop_on_solve=0)


def listed():
    return [
        # One annealing search alone on the device: squared objective, within-row
        # swaps, cooling (the single-replica W(12,11) configuration).  The
        # smallest call: its speed is the latency of one Markov chain.
        {"name": "search_w12", "kind": "batch", "set": "single", "orders": "12:11", "jobs": 1, "replicas": 1,
         "iters": 5000, "round": 5000},
        # A small whole call, host buffers in and out: four searches of 64
        # replicas with the default parameters (the reference's mix of objectives).
        {"name": "solve_w14", "kind": "solve", "set": "default", "orders": "14:13", "jobs": 4, "replicas": 64,
         "iters": 2000, "round": 2000},
        # The uniform tempering population: 128 instances of a 32-rung ladder on
        # W(26,25), one exchange interval of 10^4 iterations.
        {"name": "ladder_w26", "kind": "batch", "set": "ladder", "orders": "26:25", "jobs": 128, "replicas": 32,
         "iters": 10000, "round": 10000},
        # Uneven orders in one launch: 16-rung ladders of five orders, 1024
        # replicas of each.
        {"name": "uneven_w14_30", "kind": "batch", "set": "ladder", "orders": "14:13 18:17 20:19 24:23 30:29",
         "jobs": 64, "replicas": 16, "iters": 4000, "round": 2000},
        # What the drop-in command line runs: one search, a device full of
        # replicas, default parameters, one launch of 4096 iterations.
        {"name": "default_w24", "kind": "batch", "set": "default", "orders": "24:23", "jobs": 1, "replicas": 2368,
         "iters": 4096, "round": 4096},
        # The sparse family of the request mix, W(n,4), at orders of one and two
        # rows per lane, odd ones among them, 256 replicas per request.
        {"name": "sparse_w17_64", "kind": "batch", "set": "default", "orders": "17:4 23:4 31:4 35:4 42:4 49:4 56:4 64:4",
         "jobs": 1, "replicas": 256, "iters": 2000, "round": 2000},
        # Orders of four rows per lane, half the entries nonzero.
        {"name": "mid_w100", "kind": "batch", "set": "default", "orders": "100:50", "jobs": 1, "replicas": 592,
         "iters": 1000, "round": 1000},
        # The largest order whose state sits in shared memory.
        {"name": "wide_w256", "kind": "batch", "set": "default", "orders": "256:255", "jobs": 1, "replicas": 148,
         "iters": 1000, "round": 1000},
        # Beyond shared memory: the reference's own largest order at w = n - 1.
        {"name": "large_w276", "kind": "batch", "set": "large", "orders": "276:275", "jobs": 1, "replicas": 2368,
         "iters": 1000, "round": 1000},
        # Exact rescoring of 65536 matrices resident on the device, the largest
        # order of the tensor-core configuration.
        {"name": "rescore_n128", "kind": "rescore", "n": 128, "w": 64, "count": 65536, "gram": False},
        # The same check at an order off the 32-grid, as populations of W(n,n-1) need it.
        {"name": "rescore_n100", "kind": "rescore", "n": 100, "w": 99, "count": 8192, "gram": False},
        # The serving loop on its request mix: 24 requests of 256 replicas at
        # once, each with a budget of 6000 iterations per replica.
        {"name": "serve_mix24", "kind": "serve", "requests": 24, "replicas": 256, "iters": 6000},
    ]


def _log(rng, lo, hi):
    return int(round(np.exp(rng.uniform(np.log(lo), np.log(hi)))))


def draw(rng):
    kind = rng.choice(["single", "solve", "ladder", "default", "default", "sparse", "mid", "wide", "large",
                       "rescore", "rescore", "rescore", "serve"])
    if kind == "single":
        n = rng.randrange(6, 32)
        return {"kind": "batch", "set": "single", "orders": f"{n}:{n - 1}", "jobs": 1, "replicas": 1,
                "iters": _log(rng, 500, 8000), "round": 4000}
    if kind == "solve":
        n = rng.randrange(8, 40)
        return {"kind": "solve", "set": "default", "orders": f"{n}:{max(1, n - rng.randrange(0, 4))}",
                "jobs": rng.randrange(1, 9), "replicas": _log(rng, 1, 128), "iters": _log(rng, 200, 2000),
                "round": 1000}
    if kind == "ladder":
        n = rng.randrange(10, 33)
        return {"kind": "batch", "set": "ladder", "orders": f"{n}:{n - 1}", "jobs": _log(rng, 8, 128),
                "replicas": rng.choice([8, 16, 32]), "iters": _log(rng, 500, 6000), "round": 2000}
    if kind == "default":
        n = rng.randrange(10, 33)
        w = rng.choice([n - 1, n - 1, max(2, n // 2), max(2, n - 3)])
        return {"kind": "batch", "set": "default", "orders": f"{n}:{w}", "jobs": rng.randrange(1, 4),
                "replicas": _log(rng, 64, 1200), "iters": _log(rng, 300, 4000), "round": 4096}
    if kind == "sparse":
        orders = " ".join(f"{rng.randrange(16, 65)}:4" for _ in range(rng.randrange(1, 8)))
        return {"kind": "batch", "set": "default", "orders": orders, "jobs": 1, "replicas": _log(rng, 32, 256),
                "iters": _log(rng, 300, 2000), "round": 2000}
    if kind == "mid":
        n = rng.randrange(65, 129)
        return {"kind": "batch", "set": "default", "orders": f"{n}:{rng.randrange(2, n + 1)}", "jobs": 1,
                "replicas": _log(rng, 32, 592), "iters": _log(rng, 100, 1000), "round": 500}
    if kind == "wide":
        n = rng.randrange(129, 257)
        return {"kind": "batch", "set": "default", "orders": f"{n}:{rng.randrange(2, n + 1)}", "jobs": 1,
                "replicas": _log(rng, 8, 148), "iters": _log(rng, 50, 300), "round": 150}
    if kind == "large":
        n = _log(rng, 257, 512)
        return {"kind": "batch", "set": "large", "orders": f"{n}:{rng.choice([n - 1, n // 2, 20])}", "jobs": 1,
                "replicas": _log(rng, 16, 600), "iters": _log(rng, 30, 200), "round": 100}
    if kind == "rescore":
        n = rng.choice([32, 64, 96, 128, _log(rng, 8, 256), _log(rng, 8, 256)])
        most = max(64, min(65536, 65536 * 128 * 128 // (4 * n * n)) if n % 32 == 0 and n <= 128
                   else 8192 * 1000000 // max(n ** 3, 125000))
        return {"kind": "rescore", "n": n, "w": rng.choice([max(1, n // 2), max(1, n - 1), min(n, 4)]),
                "count": _log(rng, 16, most), "gram": rng.random() < 0.25 and most <= 16384}
    return {"kind": "serve", "requests": rng.randrange(2, 25), "replicas": _log(rng, 32, 256),
            "iters": _log(rng, 1000, 6000)}


def _orders(case):
    return [tuple(int(v) for v in o.split(":")) for o in case["orders"].split()]


def _jobs(case, seed):
    return [{"n": n, "w": w, "seed": 1 + 7919 * seed + 1000 * i + k, "replicas": case["replicas"]}
            for i, (n, w) in enumerate(_orders(case)) for k in range(case["jobs"])]


def _params(case, seed):
    if case["set"] == "single":
        return X.Params(seed=seed + 1, t_init=4.0, t_min=0.05, cooling=(0.05 / 4.0) ** (1.0 / 2000.0),
                        moves_per_cool=500, stuck_threshold=2_000_000_000, objective=1, move_set=1, start_kind=1,
                        stop_on_solve=2, moves_per_launch=case["round"])
    if case["set"] == "ladder":
        return X.Params(seed=seed + 1, exchange_interval=case["round"], moves_per_launch=case["round"], **LADDER)
    if case["set"] == "large":
        return X.Params(seed=seed + 1, t_init=6.0, t_min=0.1, squared_objective_fraction=0.0,
                        parity_objective_fraction=0.0, stop_on_solve=0, moves_per_launch=case["round"])
    return X.Params(seed=seed + 1, stop_on_solve=2, moves_per_launch=case["round"])


def _requests(case, seed):
    """The request mix: 70% W(n, n-1), 30% W(n, 4) with n in 16..64; the
    orders belong to the case, the searches' seeds to `seed`."""
    rng = np.random.default_rng(1234 + case["requests"])
    out = []
    for k in range(case["requests"]):
        if rng.random() < 0.7:
            n = int(rng.choice([12, 14, 18, 20, 24, 26, 30]))
            out.append((n, n - 1, 1000 + 4001 * seed + k))
        else:
            out.append((int(rng.integers(16, 65)), 4, 1000 + 4001 * seed + k))
    return out


def _matrices(case, seed):
    """`count` row-major n x n ternary matrices, w nonzeros per row, on the device."""
    n, w, count = case["n"], case["w"], case["count"]
    gen = torch.Generator(device="cuda").manual_seed(1 + seed)
    W = torch.zeros((count, n, n), dtype=torch.int8, device="cuda")
    step = max(1, (1 << 26) // (n * n))
    for lo in range(0, count, step):
        c = min(step, count - lo)
        cols = torch.rand((c, n, n), device="cuda", generator=gen).topk(w, dim=2).indices
        signs = (torch.randint(0, 2, (c, n, w), device="cuda", generator=gen) * 2 - 1).to(torch.int8)
        W[lo:lo + c].scatter_(2, cols, signs)
    return W


def prepare(case, seed):
    if case["kind"] == "rescore":
        n, count = case["n"], case["count"]
        return {"case": case, "W": _matrices(case, seed),
                "stats": torch.zeros((count, 4), dtype=torch.int32, device="cuda"),
                "gram": torch.zeros((count, n, n), dtype=torch.int32, device="cuda") if case["gram"] else None}
    if case["kind"] == "serve":
        return {"case": case, "server": X.Server(), "requests": _requests(case, seed)}
    st = {"case": case, "jobs": _jobs(case, seed), "params": _params(case, seed)}
    if case["kind"] == "batch":
        st["batch"] = X.Batch(st["jobs"], st["params"])
    return st


_COUNTERS = ("score", "conflicts", "best_replica", "solved", "verified", "error", "moves", "candidate_evaluations",
             "iterations", "solved_iteration", "accepted_moves", "accepted_rows", "two_row_evaluations")

_STATE = ("iterations", "moves", "candidate_evaluations", "score", "conflicts", "best_score", "best_conflicts",
          "objective_total", "moves_since_improvement", "cooling_counter", "rung", "objective_kind", "status", "error",
          "accepted_moves", "accepted_rows", "two_row_evaluations")


def _table(results, fields):
    return np.array([[getattr(r, f) for f in fields] for r in results], dtype=np.int64)


def run(state):
    case = state["case"]
    if case["kind"] == "rescore":
        W, stats, gram = state["W"], state["stats"], state["gram"]
        rc = X.lib().xw_rescore_device(C.c_void_p(W.data_ptr()), case["count"], case["n"], case["w"],
                                       C.c_void_p(stats.data_ptr()),
                                       C.c_void_p(gram.data_ptr() if gram is not None else 0), 0,
                                       C.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != X.XW_OK:
            raise X.XwError(rc, X.lib().xw_last_error().decode())
        return [stats] if gram is None else [stats, gram]
    if case["kind"] == "serve":
        srv = state["server"]
        ids = [srv.submit(n, w, seed, replicas=case["replicas"], max_moves=case["replicas"] * case["iters"])
               for n, w, seed in state["requests"]]
        out = [srv.wait(i) for i in ids]
        for i in ids:
            srv.release(i)
        return {"results": _table([r for r, _ in out],
                                  ("state", "solved", "verified", "sylvester", "best_replica", "score", "conflicts",
                                   "moves", "candidate_evaluations", "iterations", "solved_iteration")),
                "best": np.concatenate([W for _, W in out])}
    if case["kind"] == "solve":
        res, best = X.batch_solve(state["jobs"], state["params"], iters=case["iters"])
        return {"results": _table(res, _COUNTERS), "best": best}
    b = state["batch"]
    b.reset()
    b.run(case["iters"])
    out = b.results()
    # the whole state of the first job's first replicas, as a program that
    # continues or inspects single replicas reads it
    reps = [b.replica(0, r) for r in range(min(4, case["replicas"]))]
    return {"results": _table([r for r, _ in out], _COUNTERS), "best": np.concatenate([W for _, W in out]),
            "states": _table([s for s, _, _, _ in reps], _STATE),
            "temperature_bits": np.array([s.temperature for s, _, _, _ in reps]).view(np.int64),
            "W": np.stack([W for _, W, _, _ in reps]), "best_W": np.stack([B for _, _, B, _ in reps]),
            "minority": np.stack([M for _, _, _, M in reps]).astype(np.int64)}


# Of one iteration: candidates evaluated on average (one, or four with
# probability 1/2), rows of the Gram matrix a candidate changes, and integer
# operations per entry of such a row (two products, two sums, two absolute
# values, the two sums of the score and the conflicts).
_CANDIDATES, _ROWS, _OPS = 2.5, 1.5, 8.0


def _anneal_work(n, w, replicas, iters):
    record = 128 + 2 * n * n + n * min(w, n - w)
    return {"bytes": 2.0 * replicas * record, "flops": replicas * iters * _CANDIDATES * _ROWS * _OPS * n}


def work(case):
    if case["kind"] == "rescore":
        n, count = case["n"], case["count"]
        out = 16 + (4 * n * n if case["gram"] else 0)
        # G is symmetric: n(n+1)/2 dot products of n terms
        return {"bytes": float(count * (n * n + out)), "flops": float(count) * n * (n + 1) * n}
    if case["kind"] == "serve":
        parts = [_anneal_work(n, w, case["replicas"], case["iters"]) for n, w, _ in _requests(case, 0)]
    else:
        parts = [_anneal_work(j["n"], j["w"], j["replicas"], case["iters"]) for j in _jobs(case, 0)]
    return {k: float(sum(p[k] for p in parts)) for k in ("bytes", "flops")}


def exact(case, seed):
    """The rescoring's statistics (and Gram matrices) in 64 bits; searches have
    no value but their trajectory."""
    if case["kind"] != "rescore" or case["count"] * case["n"] ** 3 > 4e9:
        return None
    n, w = case["n"], case["w"]
    W = _matrices(case, seed).cpu().numpy().astype(np.float64)
    G = np.matmul(W, W.transpose(0, 2, 1)).astype(np.int64)
    off = G * (1 - np.eye(n, dtype=np.int64))
    a = np.abs(off)
    ok = (G == w * np.eye(n, dtype=np.int64)).all(axis=(1, 2))
    stats = np.stack([a.sum((1, 2)) // 2, (a != 0).sum((1, 2)) // 2, (off * off).sum((1, 2)) // 2,
                      ok.astype(np.int64)], axis=1)
    return [stats] if not case["gram"] else [stats, G]
