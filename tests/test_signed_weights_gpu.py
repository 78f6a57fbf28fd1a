"""Negative weights: the bounded picks of the fast construction kernels hold for
weights that are not negative, so a colony where a caller's pheromone, tau0,
prior or distances made some negative goes to the general kernel, which adds
entry by entry.  Against the port, bit for bit, whatever kernel was asked for."""
import os

import numpy as np
import pytest

import oracle
import acogpu_gb300 as aco
from acogpu_gb300 import _abi
from acogpu_gb300.prior import EdgePrior, candidate_heuristic
from helpers import assert_same_state, instance

pytestmark = pytest.mark.gpu
THREADS = os.cpu_count() or 4
FAST = dict(nn_order=_abi.ACO_NN_STABLE, heuristic=_abi.ACO_HEURISTIC_DEVICE,
            fallback=_abi.ACO_FALLBACK_BEST)
# (n, k, mode): the staged, cluster, direct and general kernels; long rows
# staged, in row order and in city order, in one mask word a lane and in more.
SHAPES = [(60, 16, _abi.ACO_CONSTRUCT_STAGED), (1100, 20, _abi.ACO_CONSTRUCT_CLUSTER),
          (2100, 24, _abi.ACO_CONSTRUCT_CLUSTER), (1100, 32, _abi.ACO_CONSTRUCT_DIRECT),
          (60, 16, _abi.ACO_CONSTRUCT_GLOBAL), (28, 0, _abi.ACO_CONSTRUCT_AUTO),
          (60, 0, _abi.ACO_CONSTRUCT_ROWS), (300, 64, _abi.ACO_CONSTRUCT_ROWS),
          (260, 0, _abi.ACO_CONSTRUCT_ROWS), (1100, 0, _abi.ACO_CONSTRUCT_ROWS)]


def pair(n, k, mode, d=None, **kw):
    x, y, e = instance(n, 300 + n + k)
    p = _abi.default_params(num_ants=24, cand_k=k, rho=0.2, beta=2.0, seed=n + k, **{**FAST, **kw})
    q_ = _abi.AcoParams.from_buffer_copy(p)
    q_.construct_mode = mode
    g = aco.Colony(**({"coords": (x, y)} if d is None else {"distances": d}), params=q_, num_ants=24)
    g.initialize()
    q = oracle.Port(p, e if d is None else d, threads=THREADS)
    q.initialize()
    return g, q


def follow(g, q, iters, aging, ctx):
    for it in range(iters):
        g.constructSolution()
        q.iterate()
        assert_same_state(g, q, aging=bool(aging), ctx=f"{ctx} iteration {it}")
    g.close()
    q.close()


@pytest.mark.parametrize("n,k,mode", SHAPES)
@pytest.mark.parametrize("aging", [0, 1])
def test_negative_initial_pheromone(n, k, mode, aging):
    """Every weight negative: no sum is positive, so every step falls back."""
    g, q = pair(n, k, mode, tau0_mode=_abi.ACO_TAU0_VALUE, tau0=-0.25, aging=aging)
    follow(g, q, 2, aging, f"n={n} k={k} mode={mode}")


@pytest.mark.parametrize("n,k,mode", SHAPES)
@pytest.mark.parametrize("share", [0.02, 0.5])
def test_pheromone_of_both_signs(n, k, mode, share):
    g, q = pair(n, k, mode)
    rng = np.random.default_rng(n + k)
    tau = rng.uniform(0.01, 1.0, (n, n)).astype(np.float32)
    tau[rng.random((n, n)) < share] *= -1
    tau = np.triu(tau) + np.triu(tau, 1).T  # the port keeps it symmetric
    g.set_pheromone(tau)
    q.set_pheromone(tau)
    follow(g, q, 2, 0, f"n={n} k={k} mode={mode}")


@pytest.mark.parametrize("n,k,mode", SHAPES)
def test_prior_with_a_negative_floor(n, k, mode):
    g, q = pair(n, k, mode)
    pr = EdgePrior(seed=5)
    pr.apply(g, floor=-0.5)
    eta = candidate_heuristic(g)
    assert (eta < 0).any()
    q.set_candidate_heuristic(eta)
    follow(g, q, 3, 0, f"n={n} k={k} mode={mode}")
    pr.close()


@pytest.mark.parametrize("n,k,mode", SHAPES)
def test_negative_distances(n, k, mode):
    """Tours of negative length: the best is the lowest, and its deposits make
    pheromone negative between two iterations of one run."""
    rng = np.random.default_rng(7 * n)
    d = np.triu(3 * rng.integers(-20, 7, (n, n)), 1)
    d[d == 0] = 3
    d = np.triu(d, 1) + np.triu(d, 1).T
    np.fill_diagonal(d, 0x7FFFFFFF)
    g, q = pair(n, k, mode, d=d.astype(np.int32), nn_order=_abi.ACO_NN_REFERENCE_QSORT)
    g.run(3)
    g.synchronize()
    for _ in range(3):
        q.iterate()
    assert q.glob_best() < 0
    follow(g, q, 1, 0, f"n={n} k={k} mode={mode}")


@pytest.mark.parametrize("sizes,k", [((60, 300, 1100), 0), ((50, 400, 1500), 20)])
def test_batch_with_one_signed_instance(sizes, k):
    insts = [instance(n, 40 + n)[:2] for n in sizes]
    p = _abi.default_params(num_ants=24, cand_k=k, rho=0.2, beta=2.0, seed=9, **FAST)
    b = aco.Batch(insts, params=p, num_ants=24)
    b.initialize()
    ports = []
    for i, n in enumerate(sizes):
        qi = _abi.AcoParams.from_buffer_copy(p)
        with np.errstate(over="ignore"):
            qi.seed = int(np.uint64(p.seed) + np.uint64(i) * np.uint64(0x9E3779B97F4A7C15))
        q = oracle.Port(qi, instance(n, 40 + n)[2], threads=THREADS)
        q.initialize()
        if i != 1:
            rng = np.random.default_rng(n)
            tau = rng.uniform(-0.2, 1.0, (n, n)).astype(np.float32)
            tau = np.triu(tau) + np.triu(tau, 1).T
            b.colony(i).set_pheromone(tau)
            q.set_pheromone(tau)
        ports.append(q)
    for it in range(2):
        b.run(1)
        b.synchronize()
        for i, q in enumerate(ports):
            q.iterate()
            assert_same_state(b.colony(i), q, ctx=f"instance {i} iteration {it}")
    for q in ports:
        q.close()
    b.close()


@pytest.mark.parametrize("sentinel", [-1, -7])
def test_a_negative_own_distance_keeps_the_fast_kernel(sentinel):
    """No tour uses a city's distance to itself, so a negative sentinel there
    changes neither the tours nor the kernel that builds them."""
    _, _, d = instance(300, 12)
    e = d.copy()
    np.fill_diagonal(e, sentinel)
    cols = []
    for m in (d, e):
        p = _abi.default_params(num_ants=24, cand_k=16, rho=0.2, beta=3.0, seed=4, **FAST)
        cols.append(aco.Colony(m, params=p, num_ants=24))
        cols[-1].initialize()
        cols[-1].run(2)
        cols[-1].synchronize()
    a, b = cols
    assert np.array_equal(b.tours(), a.tours())
    # the autotuner times the kernels that take the colony: the general one is last
    assert _abi.ACO_CONSTRUCT_GLOBAL not in [c.autotune()["construct_mode"] for c in cols]
    for c in cols:
        c.close()
