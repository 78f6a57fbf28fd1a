"""GPU parity of the long-row construction kernel (k > 32, full rows
included; k_construct_rows.cu) against the port: its two modes of the same
colony, rows longer than one scan round (n > 1024), candidate lists of
64 and 100 with the best-choice fallback, coincident cities (infinite
weights), ants that blend their fitness after convergence, and batches whose
instances differ in size."""
import os
import tempfile

import numpy as np
import pytest

import oracle
import acogpu_gb300 as aco
from acogpu_gb300 import _abi, instances
from acogpu_gb300.prior import EdgePrior, candidate_heuristic
from helpers import assert_same_state, bits, instance

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4
GOLDEN_STEP = np.uint64(0x9E3779B97F4A7C15)


def run_vs_port(d, p, iters, ctx, mode=_abi.ACO_CONSTRUCT_AUTO):
    q_ = _abi.AcoParams.from_buffer_copy(p)
    q_.construct_mode = mode
    g = aco.Colony(d, params=q_, num_ants=p.num_ants)
    g.initialize()
    q = oracle.Port(p, d, threads=THREADS)
    q.initialize()
    for it in range(iters):
        g.constructSolution()
        q.iterate()
        assert_same_state(g, q, aging=bool(p.aging), ctx=f"{ctx} iteration {it}")
    g.close()
    q.close()


@pytest.mark.parametrize("mode", [_abi.ACO_CONSTRUCT_ROWS, _abi.ACO_CONSTRUCT_GLOBAL])
def test_rows_and_general_kernels_agree_with_the_port(mode):
    _, _, d = instance(700, 71, kind="clustered")
    p = _abi.default_params(num_ants=300, aging=1, cand_k=0, rho=0.1, beta=2.0, seed=71)
    run_vs_port(d, p, 4, f"mode {mode}", mode)


def test_rows_longer_than_one_scan_round():
    """n = 2000: two rounds of 1024 row entries per scan, and the guess taken
    from the compacted buffer."""
    _, _, d = instance(2000, 72)
    p = _abi.default_params(num_ants=160, cand_k=0, rho=0.1, beta=2.0, seed=72)
    run_vs_port(d, p, 3, "n=2000")


@pytest.mark.parametrize("k,variant", [(64, _abi.ACO_ANT_SYSTEM), (100, _abi.ACO_RANK_BASED)])
def test_candidate_lists_longer_than_32(k, variant):
    _, _, d = instance(600, 73 + k, kind="clustered")
    p = _abi.default_params(num_ants=200, variant=variant, rank_w=6, cand_k=k, rho=0.2,
                            beta=2.0, nn_order=_abi.ACO_NN_STABLE,
                            heuristic=_abi.ACO_HEURISTIC_DEVICE, fallback=_abi.ACO_FALLBACK_BEST,
                            tau0_mode=_abi.ACO_TAU0_DORIGO, seed=73 + k)
    run_vs_port(d, p, 5, f"k={k}")


def test_coincident_cities_full_rows():
    """Cities at distance 0 give infinite weights: +inf sums and the walk
    past the row into select_local_best, as the reference does."""
    x, y = instances.uniform_instance(120, seed=74)
    x = np.asarray(x, np.float32).copy()
    y = np.asarray(y, np.float32).copy()
    for a, b in ((3, 40), (7, 41), (90, 91)):
        x[b], y[b] = x[a], y[a]
    d = instances.euc2d_distances(x, y)
    p = _abi.default_params(num_ants=60, cand_k=0, rho=0.3, beta=2.0, seed=74)
    run_vs_port(d, p, 6, "coincident")


def test_blending_ants_after_convergence():
    """Small aging limits so the colony converges early: recruits blend
    their fitness (tau and eta read from L2) for min_ret iterations."""
    _, _, d = instance(220, 75, kind="clustered")
    p = _abi.default_params(num_ants=90, aging=1, cand_k=0, rho=0.2, beta=2.0, seed=75)
    (p.min_retirement_age, p.max_retirement_age, p.local_performance, p.global_performance,
     p.min_population_limit, p.max_population_limit) = (4, 7, 10, 2, 20, 100)
    g = aco.Colony(d, params=p, num_ants=90)
    g.initialize()
    q = oracle.Port(p, d, threads=THREADS)
    q.initialize()
    blended = False
    for it in range(45):
        g.constructSolution()
        q.iterate()
        a = q.aging()
        blended = blended or (a["isconverged"] and bool(((a["age"] < 4) & (a["valid"] > 0)).any()))
        assert_same_state(g, q, aging=True, ctx=f"iteration {it}")
    assert blended
    g.close()
    q.close()


def test_batch_of_long_rows_of_uneven_size():
    """One launch over instances of 300, 1500 and 2000 cities (full rows,
    aging): the per-ant regions are sized for the largest; every instance
    against its own port."""
    insts = [instances.clustered_instance(n, seed=76 + i) for i, n in enumerate((300, 1500, 2000))]
    p = _abi.default_params(num_ants=120, aging=1, cand_k=0, rho=0.1, beta=2.0, seed=76)
    b = aco.Batch(insts, params=p, num_ants=120)
    b.initialize()
    ports = []
    for i, (x, y) in enumerate(insts):
        qi = _abi.AcoParams.from_buffer_copy(p)
        with np.errstate(over="ignore"):
            qi.seed = int(np.uint64(p.seed) + np.uint64(i) * GOLDEN_STEP)
        q = oracle.Port(qi, instances.euc2d_distances(x, y), threads=THREADS)
        q.initialize()
        ports.append(q)
    for it in range(3):
        b.run(1)
        b.synchronize()
        for i, q in enumerate(ports):
            q.iterate()
            assert_same_state(b.colony(i), q, aging=True, ctx=f"instance {i} iteration {it}")
    t = b.autotune()
    assert t["ants_per_block"] in (2, 4, 6, 8, 11)
    for q in ports:
        q.close()
    b.close()


@pytest.mark.parametrize("n,k", [(33, 0), (64, 0), (127, 0), (128, 0), (129, 0), (1023, 0),
                                 (1024, 0), (1025, 0), (2051, 0), (300, 33), (300, 127),
                                 (300, 128), (300, 129), (1100, 1099), (4100, 40)])
@pytest.mark.parametrize("aging", [0, 1])
def test_row_edges_match_the_port(n, k, aging):
    """Row lengths around a lane's four entries, a chunk (128) and a round
    (1024), full rows and candidate lists; bit for bit."""
    _, _, d = instance(n, 400 + n + k, kind="clustered" if n % 2 else "uniform")
    more = dict(nn_order=_abi.ACO_NN_STABLE, heuristic=_abi.ACO_HEURISTIC_DEVICE,
                fallback=_abi.ACO_FALLBACK_BEST, tau0_mode=_abi.ACO_TAU0_DORIGO) if k else {}
    p = _abi.default_params(num_ants=60 if n < 1000 else 24, aging=aging, cand_k=k, rho=0.2,
                            beta=2.0, seed=n + k, **more)
    run_vs_port(d, p, 3 if n < 1000 else 2, f"n={n} k={k}")


@pytest.mark.parametrize("n,k", [(90, 0), (200, 70)])
def test_long_rows_with_a_prior_match_the_port(n, k):
    """A learned prior on long rows: the candidate heuristic is no longer the
    plain one, so full rows are summed in row order; a checkpoint of the colony
    continues the same way, and initialising drops the prior again."""
    x, y, d = instance(n, 500 + n)
    p = _abi.default_params(num_ants=40, cand_k=k, rho=0.2, beta=2.0, seed=9,
                            fallback=_abi.ACO_FALLBACK_BEST if k else _abi.ACO_FALLBACK_REFERENCE)
    g = aco.Colony(coords=(x, y), params=p, num_ants=40)
    g.initialize()
    g.run(1)
    pr = EdgePrior(seed=5)
    g.initialize()
    pr.apply(g, floor=0.05)
    q = oracle.Port(p, d, threads=THREADS)
    q.initialize()
    q.set_candidate_heuristic(candidate_heuristic(g))
    for it in range(3):
        g.constructSolution()
        q.iterate()
        assert_same_state(g, q, ctx=f"prior iteration {it}")
    with tempfile.TemporaryDirectory() as tmp:
        g.save(os.path.join(tmp, "c"))
        h = aco.Colony(coords=(x, y), params=p, num_ants=40)
        h.initialize()
        h.load(os.path.join(tmp, "c"))
    q.iterate()
    for col in (g, h):
        col.constructSolution()
        assert_same_state(col, q, ctx="after the checkpoint")
    g.initialize()
    q2 = oracle.Port(p, d, threads=THREADS)
    q2.initialize()
    for it in range(2):
        g.constructSolution()
        q2.iterate()
        assert_same_state(g, q2, ctx=f"plain again {it}")
    for col in (g, h, q, q2):
        col.close()
    pr.close()


@pytest.mark.parametrize("side,aging", [(8, 0), (20, 1), (34, 0)])
def test_lattice_rows_match_the_port(side, aging):
    """Cities on an integer lattice: few distinct distances, so weights repeat,
    running sums fall halfway between floats and thresholds land on them."""
    x, y = np.meshgrid(np.arange(side, dtype=np.float32), np.arange(side, dtype=np.float32))
    d = instances.euc2d_distances(x.ravel(), y.ravel())
    p = _abi.default_params(num_ants=40, aging=aging, cand_k=0, rho=0.5, beta=2.0, seed=side)
    run_vs_port(d, p, 4, f"lattice {side}")


@pytest.mark.parametrize("n,aging", [(129, 0), (300, 1), (1100, 0)])
def test_prior_on_rows_in_city_order_matches_the_port(n, aging):
    """Full rows of more than 128 cities are summed in city order from the plain
    choice matrix, but not while a prior is installed: through apply, a second
    apply, a checkpoint into another colony, and initialising again."""
    x, y, d = instance(n, 800 + n)
    p = _abi.default_params(num_ants=40 if n < 1000 else 20, cand_k=0, rho=0.2, beta=2.0, seed=9,
                            aging=aging)
    g = aco.Colony(coords=(x, y), params=p, num_ants=p.num_ants)
    g.initialize()
    pr = EdgePrior(seed=5)
    q = oracle.Port(p, d, threads=THREADS)
    q.initialize()
    for floor in (0.05, 0.5):
        pr.apply(g, floor=floor)
        q.set_candidate_heuristic(candidate_heuristic(g))
        for it in range(2):
            g.constructSolution()
            q.iterate()
            assert_same_state(g, q, aging=bool(aging), ctx=f"floor {floor} iteration {it}")
    with tempfile.TemporaryDirectory() as tmp:
        g.save(os.path.join(tmp, "c"))
        h = aco.Colony(coords=(x, y), params=p, num_ants=p.num_ants)
        h.initialize()
        h.run(1)
        h.load(os.path.join(tmp, "c"))
    q.iterate()
    for col in (g, h):
        col.run(1)
        col.synchronize()
        assert_same_state(col, q, aging=bool(aging), ctx="after the checkpoint")
    q2 = oracle.Port(p, d, threads=THREADS)
    q2.initialize()
    g.initialize()
    for it in range(2):
        g.constructSolution()
        q2.iterate()
        assert_same_state(g, q2, aging=bool(aging), ctx=f"plain again {it}")
    # a checkpoint without a prior, into a colony that has one
    with tempfile.TemporaryDirectory() as tmp:
        g.save(os.path.join(tmp, "c"))
        h.load(os.path.join(tmp, "c"))
    q2.iterate()
    h.constructSolution()
    assert_same_state(h, q2, aging=bool(aging), ctx="plain checkpoint")
    for col in (g, h, q, q2):
        col.close()
    pr.close()


def coincident(n, seed):
    x, y = instances.uniform_instance(n, seed=seed)
    x, y = np.array(x, np.float32), np.array(y, np.float32)
    for a, b in ((3, n // 3), (7, n // 3 + 1), (n - 30, n - 2), (n // 2, n - 3)):
        x[b], y[b] = x[a], y[a]
    return x, y


@pytest.mark.parametrize("n,aging", [(200, 0), (700, 1), (1100, 0)])
def test_coincident_cities_on_rows_in_city_order(n, aging):
    """Infinite weights where a masked one becomes a NaN in the city-order sum,
    in one mask word a lane and in more."""
    x, y = coincident(n, 90 + n)
    p = _abi.default_params(num_ants=40 if n < 1000 else 16, aging=aging, cand_k=0, rho=0.3,
                            beta=2.0, seed=n)
    run_vs_port(instances.euc2d_distances(x, y), p, 4 if n < 1000 else 3, f"coincident n={n}")


@pytest.mark.parametrize("sizes", [(200, 300), (200, 1100)])
def test_batch_with_a_prior_and_coincident_cities(sizes):
    """The batch kernel's sums of full rows, one mask word a lane (largest
    instance up to 1024 cities) and more: one instance with a prior, one with
    infinite weights, then without the prior again."""
    insts = [instances.uniform_instance(sizes[0], seed=4), coincident(sizes[1], 5),
             instances.uniform_instance(150, seed=6)]
    p = _abi.default_params(num_ants=30, cand_k=0, rho=0.2, beta=2.0, seed=77)
    b = aco.Batch(insts, params=p, num_ants=30)
    pr = EdgePrior(seed=5)

    def ports():
        out = []
        for i, (x, y) in enumerate(insts):
            qi = _abi.AcoParams.from_buffer_copy(p)
            with np.errstate(over="ignore"):
                qi.seed = int(np.uint64(p.seed) + np.uint64(i) * GOLDEN_STEP)
            out.append(oracle.Port(qi, instances.euc2d_distances(x, y), threads=THREADS))
            out[-1].initialize()
        return out

    for prior in (True, False):
        b.initialize()
        qs = ports()
        if prior:
            pr.apply(b.colony(0), floor=0.1)
            qs[0].set_candidate_heuristic(candidate_heuristic(b.colony(0)))
        for it in range(3):
            b.run(1)
            b.synchronize()
            for i, q in enumerate(qs):
                q.iterate()
                assert_same_state(b.colony(i), q, ctx=f"prior={prior} instance {i} iteration {it}")
        for q in qs:
            q.close()
    pr.close()
    b.close()
