"""Colonies and batches of different sizes in one program: setting up one must
not change what another can launch (a kernel's shared-memory limit is shared by
all of them), whether they take turns in one thread or run in several."""
import threading

import numpy as np
import pytest

import acogpu_gb300 as aco
from acogpu_gb300 import _abi, instances

pytestmark = pytest.mark.gpu

FAST = dict(nn_order=_abi.ACO_NN_STABLE, heuristic=_abi.ACO_HEURISTIC_DEVICE,
            fallback=_abi.ACO_FALLBACK_BEST, tau0_mode=_abi.ACO_TAU0_DORIGO)


def colony(n, k, **kw):
    p = _abi.default_params(num_ants=8, cand_k=k, beta=2.0, rho=0.1, seed=n, **{**FAST, **kw})
    return aco.Colony(coords=instances.uniform_instance(n, seed=n), params=p, num_ants=8)


def batch(sizes, k, **kw):
    p = _abi.default_params(num_ants=64, cand_k=k, beta=2.0, rho=0.1, seed=5, **{**FAST, **kw})
    return aco.Batch([instances.uniform_instance(n, seed=n) for n in sizes], params=p, num_ants=64)


def tours_of(x):
    return [c.tours() for c in ([x] if isinstance(x, aco.Colony) else map(x.colony, range(len(x))))]


def same(a, b):
    return all(np.array_equal(p, q) for p, q in zip(tours_of(a), tours_of(b), strict=True))


# Each pair's larger one needs more than the default 48 KB in some kernel: the
# staged table, the row pass, the batch kernel's table, its row pass.
MAKERS = {"staged": (lambda: colony(1000, 30), lambda: colony(200, 30)),
          "staged_aging": (lambda: colony(900, 30, aging=1), lambda: colony(60, 30, aging=1)),
          "row_pass": (lambda: colony(6000, 20), lambda: colony(100, 20)),
          "staged_rows": (lambda: colony(180, 0), lambda: colony(60, 0)),
          "cluster": (lambda: colony(3000, 32), lambda: colony(1500, 32)),
          "batch": (lambda: batch((1000, 900), 20), lambda: batch((100, 90), 20)),
          "batch_row_pass": (lambda: batch((4000, 900), 40), lambda: batch((100, 90), 40))}


@pytest.mark.parametrize("kind", MAKERS)
def test_a_smaller_one_set_up_between_initialise_and_run(kind):
    large, small = MAKERS[kind]
    alone = large()
    alone.initialize()
    alone.run(2)
    alone.synchronize()
    a, b = large(), small()
    a.initialize()
    b.initialize()
    a.run(2)
    a.synchronize()
    b.run(2)
    b.synchronize()
    assert same(a, alone)
    for x in (a, b, alone):
        x.close()


# The setup kernels: stable lists by selection and by the whole sort, the
# reference's quicksort order, the greedy tour (in the first two).
@pytest.mark.parametrize("large,small,k,kw", [
    (6000, 2500, 20, {}), (2500, 1100, 400, {}),
    (1500, 600, 0, dict(nn_order=_abi.ACO_NN_REFERENCE_QSORT))])
def test_threads_initialise_colonies_of_two_sizes(large, small, k, kw):
    cols = [colony(large, k, **kw), colony(small, k, **kw)]
    lists = []
    for c in cols:
        c.initialize()
        lists.append(c.nn_list())
    failed, start = [], threading.Barrier(2)

    def setup(c):
        start.wait()
        for i in range(60):
            try:
                c.initialize()
            except Exception as e:  # a thread's failure is the test's
                failed.append((c.n, i, str(e)))

    threads = [threading.Thread(target=setup, args=(c,)) for c in cols]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, (len(failed), failed[:3])
    for c, nn in zip(cols, lists, strict=True):
        assert np.array_equal(c.nn_list(), nn)
        c.close()
