"""The kernel for orders above the shared-memory classes, in its three
forms: bit planes in shared memory with the Gram matrix in HBM (the default
for orders up to 448, XW_LARGE_PLANES=2); the Gram matrix and masks in HBM
(larger orders, XW_LARGE_PLANES=0); bit planes with every Gram entry
recomputed (XW_LARGE_PLANES=1).

Its replicas follow the same draw layout and move rules as the shared-memory
kernel, so the CPU oracle replays them bit for bit: W, best W, minority
lists, counters, scores, temperature.  XW_LARGE_MIN_ORDER lowers the order
from which a batch uses it, which lets the small parity cases run through
it too, and the two kernels must then agree on every replica.
"""
import numpy as np
import pytest

import oracle_lib as O
import xtax_b200 as X
from test_gpu_parity import compare, oracle_job, start_of

pytestmark = pytest.mark.gpu


@pytest.fixture
def large_from(monkeypatch):
    def set_order(n):
        monkeypatch.setenv("XW_LARGE_MIN_ORDER", str(n))
    return set_order


FORMS = {"gram": "0", "planes": "1", "hybrid": "2"}


@pytest.fixture(params=list(FORMS))
def form(request, monkeypatch):
    """Every form of the large-order kernel."""
    monkeypatch.setenv("XW_LARGE_PLANES", FORMS[request.param])
    return request.param


def run_and_replay(n, w, R, iters, kw, seed):
    p = X.Params(stop_on_solve=0, **kw)
    batch = X.Batch([{"n": n, "w": w, "seed": seed, "replicas": R}], p)
    temps = [batch.replica(0, r)[0].reheat_temperature for r in range(R)]
    batch.run(iters)
    batch.synchronize()
    job = oracle_job(n, w, seed, p)
    for r in range(R):
        rep = O.Replica(job, r, start_of(n, w, seed, r, p), temps[r], r)
        rep.run(iters, stop_on_solve=False)
        assert rep.check() == 0
        compare(batch, 0, r, rep)
    return batch


SMALL_CASES = [
    (12, 11, 4, 2000, dict(t_init=4.0, moves_per_launch=700, stuck_threshold=500, moves_per_cool=50)),
    (16, 4, 4, 1500, dict(t_init=3.0, moves_per_launch=500, double_sign_fraction=0.4)),
    (13, 9, 3, 1200, dict(t_init=4.0, moves_per_launch=600, target_samples=12, candidate_samples=7)),
    (20, 10, 3, 1000, dict(t_init=5.0, moves_per_launch=1000, move_set=1, start_kind=1, objective=1)),
    (30, 29, 3, 800, dict(t_init=6.0, moves_per_launch=400, objective=2)),
    (8, 8, 3, 800, dict(t_init=3.0, moves_per_launch=400)),
    (9, 1, 3, 600, dict(t_init=1.0, moves_per_launch=300)),
    (70, 30, 2, 200, dict(t_init=8.0, moves_per_launch=100)),
    (200, 20, 1, 60, dict(t_init=6.0, moves_per_launch=30)),
]


@pytest.mark.parametrize("n,w,R,iters,kw", SMALL_CASES, ids=lambda v: str(v) if not isinstance(v, dict) else "")
def test_small_orders_through_the_large_kernel_match_oracle(large_from, form, n, w, R, iters, kw):
    large_from(1)
    run_and_replay(n, w, R, iters, kw, 3000 + n * 7 + w).close()


LARGE_CASES = [
    # just above the shared-memory classes; the reference's own limit is about 276
    (260, 259, 2, 40, dict(t_init=8.0, moves_per_launch=20)),
    (276, 275, 1, 30, dict(t_init=8.0, moves_per_launch=30)),
    (300, 20, 2, 40, dict(t_init=6.0, moves_per_launch=40, double_sign_fraction=0.3)),
    (320, 4, 2, 40, dict(t_init=2.0, moves_per_launch=20, move_set=1, start_kind=1, objective=1)),
    (333, 150, 1, 30, dict(t_init=10.0, moves_per_launch=30, objective=2)),
    (384, 384, 1, 30, dict(t_init=8.0, moves_per_launch=30)),
    (1024, 1000, 1, 12, dict(t_init=10.0, moves_per_launch=12)),
]


@pytest.mark.parametrize("n,w,R,iters,kw", LARGE_CASES, ids=lambda v: str(v) if not isinstance(v, dict) else "")
def test_large_orders_match_oracle(form, n, w, R, iters, kw):
    run_and_replay(n, w, R, iters, kw, 5000 + n * 7 + w).close()


@pytest.mark.parametrize("objective", [0, 1, 2])
@pytest.mark.parametrize("n,same,iters", [(264, 200, 60), (264, 122, 400), (271, 123, 400), (280, 122, 400)])
def test_gram_entries_around_the_byte_limit(n, same, iters, objective):
    """The hybrid form's G in bytes holds entries up to 123: a start above it
    (halfwords from the load on) and starts at it, which the walk leaves."""
    rng = np.random.default_rng(n + same)
    w = n - 1 if n % 2 == 0 else n
    W = rng.choice(np.array([-1, 1], np.int8), size=(n, n))
    if w < n:
        W[np.arange(n), np.arange(n) // 2 * 2] = 0
    for i in range(0, n - 1, 2):   # pairs of rows with a product of `same` or one more
        W[i + 1] = W[i]
        W[i + 1, rng.permutation(np.flatnonzero(W[i]))[:(w - same) // 2]] *= -1
    start = np.ascontiguousarray(W.T)   # column-major
    p = X.Params(stop_on_solve=0, t_init=1e6, t_min=1e5, moves_per_launch=iters // 2, candidate_samples=2,
                 sign_fraction=0.6, objective=objective)
    batch = X.Batch([{"n": n, "w": w, "seed": 5, "replicas": 1}], p, starts=start)
    rep = O.Replica(oracle_job(n, w, 5, p), 0, start, batch.replica(0, 0)[0].reheat_temperature, 0)

    def largest():
        G = rep.get()[4].copy()
        np.fill_diagonal(G, 0)
        return np.abs(G).max()

    assert (largest() > 123) == (same > 123)
    seen = 0
    for _ in range(20):
        rep.run(iters // 20, stop_on_solve=False)
        seen = max(seen, largest())
    assert seen > 127   # no longer a byte
    batch.run(iters)
    batch.synchronize()
    compare(batch, 0, 0, rep)
    batch.close()


@pytest.mark.parametrize("n,w,planes", [(276, 275, True), (448, 447, True), (449, 448, False), (1024, 1000, False)])
def test_large_class_reports_its_form(monkeypatch, n, w, planes):
    """The bit-plane forms up to order 448 (the hybrid by default), the
    stored Gram matrix above it."""
    for wanted in ("", "0", "1", "2"):
        monkeypatch.setenv("XW_LARGE_PLANES", wanted)
        b = X.Batch([{"n": n, "w": w, "seed": 1, "replicas": 2}], X.Params(stop_on_solve=0))
        (c,) = b.classes()
        assert c["large"] == (1 + int(wanted or "2") if planes else 1)
        b.close()


def test_both_kernels_agree_on_a_mixed_batch(large_from):
    """A batch of several orders gives the same results whichever kernel
    runs which jobs (here: the shared-memory kernel for all, then the large
    kernel for orders from 20 while the rest stay in shared memory)."""
    jobs = [{"n": n, "w": w, "seed": 11 + n, "replicas": 6} for n, w in ((12, 11), (18, 9), (26, 25), (40, 8))]
    p = X.Params(stop_on_solve=0, t_init=5.0, moves_per_launch=500)
    out = []
    for threshold in (257, 20):
        large_from(threshold)
        b = X.Batch(jobs, p)
        b.run(1500)
        b.synchronize()
        out.append([(r.score, r.conflicts, r.best_replica, r.moves, r.candidate_evaluations, W.tobytes())
                    for r, W in b.results()])
        out.append([tuple(np.concatenate([a.ravel().astype(np.int64) for a in b.replica(j, k)[1:]]).tolist())
                    for j in range(len(jobs)) for k in range(6)])
        b.close()
    assert out[0] == out[2]
    assert out[1] == out[3]


def test_large_tempering_matches_oracle():
    n, w, R, interval, rounds = 264, 263, 4, 15, 3
    p = X.Params(stop_on_solve=0, tempering=1, exchange_interval=interval, t_min=0.1, t_init=6.0,
                 squared_objective_fraction=0.0, parity_objective_fraction=0.0)
    seed = 91
    batch = X.Batch([{"n": n, "w": w, "seed": seed, "replicas": R}], p)
    batch.run(interval * rounds)
    batch.synchronize()
    # the host builds the ladder by repeated multiplication
    ratio = (6.0 / 0.1) ** (1.0 / (R - 1))
    ladder, t = [], 0.1
    for _ in range(R):
        ladder.append(t)
        t *= ratio
    job = oracle_job(n, w, seed, p)
    reps = [O.Replica(job, r, start_of(n, w, seed, r, p), ladder[r], r) for r in range(R)]
    for k in range(rounds):
        for rep in reps:
            rep.run(interval, stop_on_solve=False)
        O.exchange(job, reps, ladder, k)
    for r in range(R):
        compare(batch, 0, r, reps[r])
    batch.close()


def test_large_snapshot_resume_equals_uninterrupted(tmp_path):
    """A snapshot holds no Gram arena: the kernel rebuilds it on resume and
    the trajectory continues unchanged."""
    jobs = [{"n": 270, "w": 269, "seed": 7, "replicas": 3}]
    p = X.Params(stop_on_solve=0, t_init=8.0, moves_per_launch=25)
    a = X.Batch(jobs, p)
    a.run(100)
    a.synchronize()
    b = X.Batch(jobs, p)
    b.run(50)
    b.synchronize()
    path = str(tmp_path / "large.xwpop")
    b.save(path)
    b.close()
    c = X.Batch.load(path, jobs)
    c.run(50)
    c.synchronize()
    for r in range(3):
        sa, Wa, Ba, Ma = a.replica(0, r)
        sc, Wc, Bc, Mc = c.replica(0, r)
        assert sc.error == 0
        assert (sa.iterations, sa.moves, sa.score, sa.best_score) == (sc.iterations, sc.moves, sc.score, sc.best_score)
        assert (Wa == Wc).all() and (Ba == Bc).all() and (Ma == Mc).all()
    a.close()
    c.close()


def test_large_order_solves_and_verifies():
    """W(300, 1) from row-only starts needs column changes: the within-row
    swap finds a signed permutation matrix, which the host verifies (the
    oracle's replay of these replicas solves within 60000 iterations)."""
    p = X.Params(stop_on_solve=1, t_init=0.15, t_min=0.05, moves_per_launch=20000, move_set=1, start_kind=1,
                 squared_objective_fraction=0.0, parity_objective_fraction=0.0)
    res, best = X.batch_solve([{"n": 300, "w": 1, "seed": 3, "replicas": 8}], p, iters=400000)
    assert res[0].error == 0
    assert res[0].solved == 1 and res[0].verified == 1
    W = best[: 300 * 300].reshape(300, 300).T.astype(np.int64)
    assert (W @ W.T == np.eye(300, dtype=np.int64)).all()


def test_order_above_the_maximum_is_refused():
    with pytest.raises(X.XwError):
        X.Batch([{"n": X.MAX_ORDER_CUDA + 1, "w": 4, "seed": 1, "replicas": 1}], X.Params())


def test_elite_restarts_at_a_large_order():
    """Restarts replace W and the 16-bit minority lists of HBM-resident
    replicas: the kernel must rebuild their Gram from the new W (a stale
    Gram would fail the score check at the next load and the run)."""
    # a random walk at a very high fixed temperature stops improving on its
    # best almost at once, so the stagnation trigger fires
    p = X.Params(seed=3, replicas=32, moves_per_launch=200, max_seconds=2.0, restart_interval=0.05,
                 restart_fraction=0.5, t_init=1000.0, t_min=1000.0)
    r = X.run_annealer(264, 263, p)
    restarts = [line for line in r.log if line.startswith("[restart] seconds=")]
    assert restarts and r.restarted_replicas > 0
    assert X.score(264, 263, r.best.entries)[0] == r.best.score


def test_cli_runs_a_large_order(tmp_path):
    """The drop-in CLI beyond the reference's shared-memory limit: it runs,
    reports, and writes its best W."""
    import os
    import subprocess
    cli = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xtax_b200", "bin", "xweigh_cuda")
    out = tmp_path / "w.csv"
    r = subprocess.run([cli, "300", "299", "--seed", "5", "--replicas", "64", "--max-seconds", "2", "-o", str(out)],
                       capture_output=True, text=True, timeout=300)
    # not solved in 2 s: the reference's finish() still exits 0 and says so
    assert r.returncode == 0, r.stderr
    assert f"No weighing matrix found; wrote the best fixed-weight candidate to {out}" in r.stdout
    assert any(line.startswith("done moves=") for line in r.stdout.splitlines())
    final = [line for line in r.stdout.splitlines() if line.startswith("Final best score: ")][0]
    rows = [list(map(int, line.split(","))) for line in out.read_text().splitlines()]
    W = np.array(rows, dtype=np.int8).T.reshape(-1)
    st = X.score(300, 299, W)
    assert final == f"Final best score: {st[0]} conflicts={st[1]}"


def test_restarts_at_a_large_order_with_weight_near_half_stay_quick():
    """The escape scan of W(512,256) would take about 4e12 operations, many
    seconds per restart: past the scan budget a restart kicks without an
    escape move, so a short run still restarts several times."""
    p = X.Params(seed=4, replicas=32, moves_per_launch=100, max_seconds=6.0, restart_interval=0.05,
                 restart_fraction=0.5, t_init=1000.0, t_min=1000.0)
    r = X.run_annealer(512, 256, p)
    restarts = [line for line in r.log if line.startswith("[restart] seconds=")]
    assert len(restarts) >= 2
    assert all("min_escape_delta=0" in line for line in restarts)
    # once the search stagnates, restarts follow one another within the
    # interval plus a launch, not seconds of scanning apart
    t = [float(line.split("seconds=")[1].split()[0]) for line in restarts]
    assert max(b - a for a, b in zip(t, t[1:])) < 2.0
    assert X.score(512, 256, r.best.entries)[0] == r.best.score


@pytest.mark.parametrize("small,n,w", [(False, 257, 256), (False, 258, 5), (False, 259, 130), (False, 260, 259), (False, 271, 271),
                                       (False, 320, 319), (False, 447, 446), (False, 448, 4), (True, 5, 4), (True, 6, 3),
                                       (True, 16, 15), (True, 17, 4), (True, 64, 63), (True, 65, 2), (True, 130, 129)])
def test_rounds_of_a_few_iterations(large_from, small, n, w):
    """W and G pass from launch to launch through the arena: many launches of
    two iterations, at orders of every remainder by a word, from the start
    again after a reset."""
    if small:
        large_from(1)
    p = X.Params(stop_on_solve=0, t_init=3.0, moves_per_launch=2, moves_per_cool=3)
    batch = X.Batch([{"n": n, "w": w, "seed": 70 + n, "replicas": 2}], p)
    temps = [batch.replica(0, r)[0].reheat_temperature for r in range(2)]
    for iters in (21, 14):
        batch.reset()
        batch.run(iters)
        batch.synchronize()
        for r in range(2):
            rep = O.Replica(oracle_job(n, w, 70 + n, p), r, start_of(n, w, 70 + n, r, p), temps[r], r)
            rep.run(iters, stop_on_solve=False)
            compare(batch, 0, r, rep)
    batch.close()
