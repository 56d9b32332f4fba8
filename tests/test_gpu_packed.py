"""The packed-row annealing kernels at the edges of their layouts, against the
oracle: every replica's whole state, bit for bit.

Orders around each class's limits (a lane's words, a row's pad, bytes against
halfwords of G, the permuted rows above order 248), the candidate and
tournament counts that take several passes, coins of probability 0 and 1,
runs of one-candidate iterations of every length, temperatures above the
32-bit threshold table, and index draws in Lemire's rejection zone.
"""
import struct

import pytest

import oracle_lib as O
import xtax_b200 as X
from test_gpu_parity import compare, oracle_job, start_of

pytestmark = pytest.mark.gpu


def replay(n, w, R, iters, seed, **kw):
    kw.setdefault("t_init", 4.0)
    kw.setdefault("moves_per_launch", max(1, iters // 2 - 3))
    p = X.Params(stop_on_solve=0, warps_per_replica=kw.pop("warps_per_replica", 1), **kw)
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
    batch.close()


EDGES = [(1, 1), (2, 1), (3, 2), (5, 5), (16, 15), (17, 16), (31, 30), (32, 31), (32, 32), (33, 3), (33, 32), (48, 24),
         (63, 62), (64, 63), (64, 64), (65, 33), (79, 78), (80, 79), (81, 4), (112, 111), (127, 126), (127, 127),
         (128, 127), (128, 128), (129, 64), (135, 134), (136, 4), (192, 96), (241, 240), (248, 124), (249, 124),
         (250, 125), (255, 254), (256, 256)]


@pytest.mark.parametrize("n,w", EDGES)
def test_orders_at_the_edges_of_the_classes(n, w):
    replay(n, w, 3 if n < 100 else 2, 700 if n < 100 else 150, 40 + n)


@pytest.mark.parametrize("greedy", [0.0, 0.1, 1.0])
@pytest.mark.parametrize("n,w", [(14, 13), (26, 25), (40, 20), (100, 99)])
def test_runs_of_one_candidate_iterations(n, w, greedy):
    # rejections of every number before an accept: a cold replica and a warm one
    replay(n, w, 4, 900, 7 + n, greedy_fraction=greedy, t_init=3.0, t_min=0.2, moves_per_cool=37, stuck_threshold=101)


@pytest.mark.parametrize("cs,ts", [(1, 1), (2, 4), (4, 5), (5, 8), (32, 9), (8, 64)])
@pytest.mark.parametrize("n,w", [(15, 8), (30, 29), (70, 69), (130, 66)])
def test_candidate_and_tournament_counts(n, w, cs, ts):
    replay(n, w, 2, 200 if n < 100 else 60, 3 * n + cs, candidate_samples=cs, target_samples=ts)


@pytest.mark.parametrize("coins", [dict(target_fraction=1.0), dict(target_fraction=0.0), dict(sign_fraction=1.0),
                                   dict(sign_fraction=0.0, double_sign_fraction=0.0), dict(double_sign_fraction=1.0),
                                   dict(switch_sign_fraction=1.0, sign_fraction=0.0, double_sign_fraction=0.0)],
                         ids=lambda c: "-".join(f"{k}={v}" for k, v in c.items()))
@pytest.mark.parametrize("n,w", [(9, 8), (26, 25), (50, 25), (140, 139)])
def test_certain_and_impossible_coins(n, w, coins):
    replay(n, w, 3, 400 if n < 100 else 80, 90 + n, **coins)


@pytest.mark.parametrize("n,w", [(12, 11), (64, 9), (150, 20)])
@pytest.mark.parametrize("t", [1e-3, 1e10, 1e13])
def test_temperatures_beyond_the_threshold_table(n, w, t):
    replay(n, w, 2, 300 if n < 100 else 60, 11 + n, t_init=t, t_min=min(t, 0.25))


@pytest.mark.parametrize("n,w,kw", [(8, 1, {}), (20, 19, {}), (33, 32, {}), (90, 45, {}), (150, 149, {}),
                                    (40, 6, dict(objective=1)), (200, 199, dict(objective=2))])
def test_within_row_swaps_of_every_class(n, w, kw):
    replay(n, w, 3, 300 if n < 100 else 80, 5 + n, move_set=1, start_kind=1, sign_fraction=0.2, **kw)


def test_an_index_draw_in_the_rejection_zone():
    # W(122, 61), seed 6: iteration 186996 of replica 0 draws the second row
    # of candidate 3's double flip from a word that Lemire's test rejects (by
    # exhaustive search of the draws); the whole trajectory is replayed past it
    replay(122, 61, 1, 187050, 6, greedy_fraction=1.0, double_sign_fraction=1.0, t_init=2.0, t_min=2.0,
           moves_per_launch=100000)


@pytest.mark.parametrize("n,w", [(13, 12), (26, 24), (32, 31)])
def test_latency_mode_at_odd_counts(n, w):
    replay(n, w, 2, 500, 60 + n, warps_per_replica=6, candidate_samples=6, t_init=0.7, t_min=0.1, moves_per_cool=23)


def set_stagnation(path, value):
    """Sets the moves since the last improvement of every replica of a
    snapshot file (the header's field at byte 64 of its record)."""
    d = bytearray(open(path, "rb").read())
    job, header, params, jobs = struct.unpack_from("<4I", d, 8)
    replicas, arena, rungs = struct.unpack_from("<3Q", d, 24)
    assert header == 128
    off = 48 + params + job * jobs
    records = struct.unpack_from(f"<{replicas}Q", d, off)
    base = off + 8 * (replicas + rungs + jobs)
    assert len(d) == base + arena
    for r in records:
        struct.pack_into("<i", d, base + r + 64, value)
    open(path, "wb").write(bytes(d))


@pytest.mark.parametrize("n,w,R,kw", [(12, 11, 4, dict(warps_per_replica=1)), (13, 6, 4, dict(warps_per_replica=1)),
                                      (14, 13, 5, dict(warps_per_replica=1, replicas_per_warp=2)),
                                      (12, 11, 4, dict(warps_per_replica=8)), (24, 23, 4, dict(warps_per_replica=32)),
                                      (16, 4, 4, dict(warps_per_replica=64, objective=1)), (40, 20, 4, {}), (100, 99, 4, {}),
                                      (150, 149, 4, {}), (260, 259, 4, {}),
                                      (12, 11, 1, dict(warps_per_replica=1, t_min=1e3, reheat=3.0)),
                                      (12, 11, 1, dict(warps_per_replica=16, t_min=1e3, reheat=3.0)),
                                      (260, 130, 1, dict(t_min=1e3, reheat=3.0))], ids=str)
def test_a_tempering_replica_is_never_reheated(n, w, R, kw, tmp_path):
    # replicas whose count of moves without improvement passes 2^31 - 1 early
    # in the second half of the run: the upper rungs of a hot ladder, which a
    # reheat (factor 1e-6) would freeze, or a ladder of one, whose temperature
    # no exchange sets again
    p = X.Params(**{**dict(stop_on_solve=0, tempering=1, exchange_interval=300, t_min=50.0, t_init=1e4, reheat=1e-6, greedy_fraction=0.0,
                           squared_objective_fraction=0.0, parity_objective_fraction=0.0), **kw})
    seed, top = 600 + n, 2 ** 31 - 1 - 5
    jobs = [{"n": n, "w": w, "seed": seed, "replicas": R}]
    first = X.Batch(jobs, p)
    first.run(300)
    first.synchronize()
    path = str(tmp_path / "population")
    first.save(path)
    first.close()
    set_stagnation(path, top)
    batch = X.Batch.load(path, jobs)
    batch.run(300)
    batch.synchronize()
    ratio = (p.t_init / p.t_min) ** (1.0 / max(R - 1, 1))
    ladder = [p.t_min]
    while len(ladder) < R:
        ladder.append(ladder[-1] * ratio)
    job = oracle_job(n, w, seed, p)
    reps = [O.Replica(job, r, start_of(n, w, seed, r, p), ladder[r], r) for r in range(R)]
    for k in range(2):
        for rep in reps:
            rep.run(300, stop_on_solve=False)
        if R > 1:
            O.exchange(job, reps, ladder, k)
    for r, rep in enumerate(reps):
        st, W, B, M = batch.replica(0, r)
        s, oW, oB, oM, _, _ = rep.get()
        assert (st.error, st.iterations, st.moves, st.candidate_evaluations) == (0, s.it, s.moves, s.cand_evals), r
        assert (st.score, st.conflicts, st.best_score, st.best_conflicts) == (s.score, s.conflicts, s.best_score,
                                                                              s.best_conflicts), r
        assert (st.temperature, st.rung, st.objective_total) == (s.temperature, s.rung, s.obj_total), r
        assert (W == oW).all() and (B == oB).all() and (M == oM).all(), r
        # counted from the last improvement, or on from the snapshot's count,
        # which wraps
        assert st.moves_since_improvement == (s.msi if s.msi < 300 else top + 300 - 2 ** 32), r
        assert st.cooling_counter == s.cool_ctr, r
    batch.close()


@pytest.mark.parametrize("n,w,kw", [(12, 11, dict(warps_per_replica=1)), (12, 4, dict(warps_per_replica=1, replicas_per_warp=2)),
                                    (20, 13, dict(warps_per_replica=8)), (40, 20, {}), (100, 99, {}), (150, 20, {}),
                                    (260, 259, {})], ids=str)
def test_a_certain_sign_flip_is_never_a_row_swap(n, w, kw):
    # iteration 78 of replica 0 at this seed draws 2^32 - 1 for the flip's
    # coin (by exhaustive search), which lies below the threshold 2^32 of
    # probability 1
    seed = 4352672
    assert O.philox([1, 78, 0, 0], X.philox_key(seed))[3] == 2 ** 32 - 1
    replay(n, w, 1, 120, seed, move_set=1, start_kind=1, sign_fraction=1.0, greedy_fraction=0.0, objective=0,
           t_init=1e9, t_min=1e9, **kw)


@pytest.mark.parametrize("ts,target", [(9, 0.0), (9, 0.05), (64, 0.0), (64, 0.05), (64, 1.0)])
@pytest.mark.parametrize("n,w,kw", [(12, 11, dict(replicas_per_warp=2)), (14, 5, dict(warps_per_replica=8)), (26, 25, {}),
                                    (40, 20, {}), (100, 99, {}), (140, 70, {})], ids=str)
def test_long_tournaments_that_few_candidates_need(n, w, kw, ts, target):
    replay(n, w, 2, 250 if n < 100 else 60, 8 * n + ts, target_samples=ts, target_fraction=target, **kw)


@pytest.mark.parametrize("wpr", [6, 16, 32, 64])
@pytest.mark.parametrize("mpc,stuck,launch", [(m, 10 ** 6, 64) for m in (1, 6, 16, 64)] +
                         [(500, 12, 50), (500, 64, 100), (7, 13, 6), (500, 50000, 1)])
def test_latency_mode_with_steps_at_the_ends_of_rounds(wpr, mpc, stuck, launch):
    # a cold replica, whose rounds are mostly rejections: cooling steps,
    # reheats and launch ends that fall on a round's last call, before it and
    # after it
    replay(12, 11, 2, 400, 9, warps_per_replica=wpr, t_init=0.4, t_min=0.2, cooling=0.99, reheat=1.5, moves_per_cool=mpc,
           stuck_threshold=stuck, moves_per_launch=launch)
