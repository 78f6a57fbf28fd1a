"""The work that a user of the engine has it do, as cases to be timed and compared.

Every pass is a whole call sequence of a user's program through the public
classes (acogpu_gb300.Colony, Batch, run.TSP, prior.EdgePrior): a colony or
batch that exists is initialised, run for some iterations and its results
are read, so a pass starts from the same state each time and can be repeated.
Sizes are those of the repository's configurations, tests and benchmark (5 to
8192 cities, candidate lists of 16 to 100 cities and full rows, 10 to 1024
ants), and generic odd ones.  All instances are seeded synthetic ones.
"""
import math

import numpy as np
import torch

import acogpu_gb300 as aco
from acogpu_gb300 import _abi, instances
from acogpu_gb300.prior import EdgePrior
from acogpu_gb300.run import TSP

FEATURES, HIDDEN = 12, 128


def listed():
    return [
        # The reference program's own call: TSP.execute on a small instance,
        # its stage timers read after every iteration (launches and latency).
        {"name": "execute_n52", "kind": "execute", "n": 52, "m": 52, "k": 0, "beta": 5.0,
         "rho": 0.1, "aging": 0, "rank": 0, "cluster": 0, "iters": 10},
        # Plain Ant System, the small configured run: 100 cities, 100 ants.
        {"name": "as_full_n100", "kind": "solve", "n": 100, "m": 100, "k": 0, "beta": 2.0,
         "rho": 0.5, "aging": 0, "rank": 0, "cluster": 0, "iters": 100},
        # A program that looks at every iteration's best before it goes on, on
        # a mid-size instance of odd size with the aging variant.
        {"name": "as_aging_full_n783", "kind": "step", "n": 783, "m": 783, "k": 0, "beta": 2.0,
         "rho": 0.1, "aging": 1, "rank": 0, "cluster": 0, "iters": 5},
        # The reference's largest instance size, full rows.
        {"name": "as_full_n2392", "kind": "solve", "n": 2392, "m": 512, "k": 0, "beta": 2.0,
         "rho": 0.1, "aging": 0, "rank": 0, "cluster": 0, "iters": 2},
        # The benchmark's default: eight instances of 1000 clustered cities, the
        # reference's own algorithm with aging.
        {"name": "batch8_full_n1000", "kind": "batch", "count": 8, "lo": 1000, "hi": 1000,
         "m": 1000, "k": 0, "beta": 2.0, "rho": 0.1, "aging": 1, "rank": 0, "iters": 5},
        # Rank-based Ant System with aging on candidate lists of 30.
        {"name": "rbas_aging_n1000_k30", "kind": "solve", "n": 1000, "m": 1000, "k": 30,
         "beta": 2.0, "rho": 0.1, "aging": 1, "rank": 6, "cluster": 1, "iters": 100},
        # Candidate lists longer than 32, ragged size.
        {"name": "rbas_n1501_k64", "kind": "solve", "n": 1501, "m": 500, "k": 64, "beta": 2.0,
         "rho": 0.2, "aging": 0, "rank": 6, "cluster": 1, "iters": 10},
        # One large instance on candidate lists of 32.
        {"name": "as_n4096_k32", "kind": "solve", "n": 4096, "m": 512, "k": 32, "beta": 2.0,
         "rho": 0.1, "aging": 0, "rank": 0, "cluster": 0, "iters": 50},
        # From coordinates to the first tours of a large instance: creation,
        # setup and one iteration in the atomic-deposit mode.
        {"name": "create_n4096_atomic", "kind": "create", "n": 4096, "m": 512, "k": 32,
         "beta": 2.0, "rho": 0.1, "aging": 0, "rank": 0, "cluster": 0, "iters": 1},
        # 512 instances of 50 to 2000 cities advanced together.
        {"name": "batch512_uneven_k20", "kind": "batch", "count": 512, "lo": 50, "hi": 2000,
         "m": 1024, "k": 20, "beta": 2.0, "rho": 0.1, "aging": 0, "rank": 0, "iters": 3},
        # Training of the edge-scoring network on the edges of solved instances.
        {"name": "prior_train", "kind": "train", "count": 128, "lo": 100, "hi": 500, "k": 20,
         "batch": 65536, "epochs": 4},
        # Loss, gradient and scores of a labelled set held by the host (odd size).
        {"name": "prior_score_100003", "kind": "score", "edges": 100003},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["execute", "solve", "solve", "solve", "step", "create", "batch", "batch",
                       "train", "score"])
    if kind == "train":
        lo = _log(rng, 60, 200)
        return {"kind": kind, "count": _log(rng, 16, 128), "lo": lo,
                "hi": lo + _log(rng, 20, 300), "k": rng.choice([16, 20, 30]),
                "batch": 128 * _log(rng, 32, 512), "epochs": rng.randint(1, 4)}
    if kind == "score":
        return {"kind": kind, "edges": _log(rng, 100, 200000)}
    common = {"beta": rng.choice([1.0, 2.0, 2.0, 3.0, 5.0]),
              "rho": round(rng.uniform(0.05, 0.5), 3), "aging": rng.randint(0, 1),
              "rank": rng.choice([0, 0, 5, 6])}
    full = rng.random() < 0.5
    if kind == "batch":
        lo = _log(rng, 50, 600)
        hi = min(_log(rng, lo, 4 * lo), 1100 if full else 2000)
        return {"kind": kind, "count": _log(rng, 2, 12 if full else 64), "lo": lo,
                "hi": max(lo, hi), "m": _log(rng, 64, 1024),
                "k": 0 if full else rng.choice([16, 20, 27, 30, 32, 48, 100]),
                "iters": rng.randint(1, 4), **common}
    if kind == "execute":
        n = _log(rng, 5, 400)
        k = 0
    elif full:
        n = _log(rng, 20, 2392)
        k = 0
    else:
        n = _log(rng, 40, 4500)
        k = min(n - 1, rng.choice([10, 16, 20, 25, 30, 32, 32, 50, 64, 100]))
    m = min(n, _log(rng, 10, 512 if n > 1100 else 1024))
    return {"kind": kind, "n": n, "m": m, "k": k, "cluster": rng.randint(0, 1),
            "iters": 1 if kind == "create" else rng.randint(1, 4) if full else rng.randint(2, 20),
            **common}


def _params(case, seed):
    """The reference's own algorithm for full rows, else the published
    candidate-list methods, as the repository's benchmark configures them."""
    p = _abi.default_params(num_ants=case["m"], beta=case["beta"], rho=case["rho"],
                            aging=case["aging"], cand_k=case["k"], seed=1000 + seed)
    if case["rank"]:
        p.variant, p.rank_w = _abi.ACO_RANK_BASED, case["rank"]
    if case["k"]:
        p.nn_order, p.heuristic = _abi.ACO_NN_STABLE, _abi.ACO_HEURISTIC_DEVICE
        p.fallback, p.tau0_mode = _abi.ACO_FALLBACK_BEST, _abi.ACO_TAU0_DORIGO
    if case["kind"] == "create":
        p.deposit = _abi.ACO_DEPOSIT_ATOMIC
    return p


def _instance(n, seed, clustered):
    if clustered:
        return instances.clustered_instance(n, seed=seed)
    return instances.uniform_instance(n, box=100000 if n > 2500 else 10000, seed=seed)


def _sizes(case):
    if case["lo"] == case["hi"]:
        return [case["lo"]] * case["count"]
    return [int(n) for n in instances.batch_sizes(case["count"], lo=case["lo"], hi=case["hi"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        sizes = _sizes(case)
        same = case["lo"] == case["hi"]
        insts = [_instance(n, 100000 * (seed + 1) + i, same or i % 2)
                 for i, n in enumerate(sizes)]
        return {"kind": kind, "iters": case["iters"],
                "batch": aco.Batch(insts, params=_params(case, seed), num_ants=case["m"])}
    if kind == "train":
        insts = [_instance(n, 100000 * (seed + 1) + i, i % 2)
                 for i, n in enumerate(_sizes(case))]
        p = _abi.default_params(cand_k=case["k"], beta=2.0, rho=0.1, seed=1000 + seed,
                                nn_order=_abi.ACO_NN_STABLE, heuristic=_abi.ACO_HEURISTIC_DEVICE,
                                fallback=_abi.ACO_FALLBACK_BEST, tau0_mode=_abi.ACO_TAU0_DORIGO)
        b = aco.Batch(insts, params=p, num_ants=64)
        b.initialize()
        b.run(10)
        b.synchronize()
        prior = EdgePrior(seed=seed)
        for i in range(len(insts)):
            prior.add_examples(b.colony(i))
        b.close()
        return {"kind": kind, "prior": prior, "start": prior.weights(), "batch": case["batch"],
                "epochs": case["epochs"], "seed": seed}
    if kind == "score":
        prior = EdgePrior(seed=seed)
        prior.set_weights(_weights(seed))
        feats, labels = _examples(case["edges"], seed)
        return {"kind": kind, "prior": prior, "feats": feats, "labels": labels,
                "pos_weight": 9.0}
    x, y = _instance(case["n"], 1 + seed, case["cluster"])
    p = _params(case, seed)
    state = {"kind": kind, "iters": case["iters"]}
    if kind == "create":
        return {**state, "coords": (x, y), "params": p, "m": case["m"]}
    return {**state, "colony": aco.Colony(coords=(x, y), params=p, num_ants=case["m"])}


def _weights(seed):
    """He-initialised layers with small biases, packed W1 b1 W2 b2 w3 b3."""
    g = np.random.default_rng(7000 + seed)
    parts = [g.normal(0.0, (2.0 / FEATURES) ** 0.5, HIDDEN * FEATURES),
             g.normal(0.0, 0.05, HIDDEN),
             g.normal(0.0, (2.0 / HIDDEN) ** 0.5, HIDDEN * HIDDEN),
             g.normal(0.0, 0.05, HIDDEN),
             g.normal(0.0, (1.0 / HIDDEN) ** 0.5, HIDDEN), g.normal(0.0, 0.05, 1)]
    return np.concatenate(parts).astype(np.float32)


def _examples(edges, seed):
    """Features as candidate edges have them (ratios, ranks, a flag), a tenth
    of the edges positive, near ones above all."""
    g = np.random.default_rng(seed)
    f = np.empty((edges, FEATURES), dtype=np.float32)
    f[:, 0:2] = g.gamma(2.0, 0.35, (edges, 2))
    f[:, 2:4] = g.integers(0, 21, (edges, 2)) / 20.0
    f[:, 4:6] = g.normal(0.0, 0.5, (edges, 2))
    f[:, 6:9] = g.uniform(0.0, 1.0, (edges, 3))
    f[:, 9:11] = g.gamma(4.0, 0.25, (edges, 2))
    f[:, 11] = g.random(edges) < 0.2
    near = np.exp(-3.0 * f[:, 0])
    labels = (g.random(edges) < 0.4 * near).astype(np.float32)
    return f, labels


def _results(c):
    """What a user reads after a run: the best tour and its length, the last
    iteration's tours and lengths, and the pheromone a later run goes on from."""
    return {"best": c.getGlobBestDist(), "best_tour": c.best_tour(), "tours": c.tours(),
            "lengths": c.tour_lengths(), "pheromone": c.pheromone()}


def run(state):
    kind = state["kind"]
    if kind == "batch":
        b = state["batch"]
        b.initialize()
        b.run(state["iters"])
        best = b.glob_best()
        colonies = [b.colony(i) for i in range(len(b))]
        return {"best": best, "best_tours": np.concatenate([c.best_tour() for c in colonies]),
                "lengths": np.concatenate([c.tour_lengths() for c in colonies])}
    if kind == "train":
        p = state["prior"]
        p.set_weights(state["start"])
        loss = p.train(epochs=state["epochs"], batch=state["batch"], lr=1e-3, seed=state["seed"])
        return {"loss": loss, "weights": p.weights()}
    if kind == "score":
        p = state["prior"]
        loss, grads = p.loss_and_grads(state["feats"], state["labels"], state["pos_weight"])
        return {"loss": loss, "grads": grads, "probs": p.predict(state["feats"])}
    if kind == "create":
        c = aco.Colony(coords=state["coords"], params=state["params"], num_ants=state["m"])
        c.initialize()
        c.run(state["iters"])
        out = _results(c)
        c.close()
        return out
    c = state["colony"]
    if kind == "execute":
        stats, _ = TSP(max_iter=state["iters"]).execute(c)
        return {"iter_bests": np.array([s["iterbest"] for s in stats], dtype=np.int64),
                **_results(c)}
    c.initialize()
    if kind == "step":
        bests = []
        for _ in range(state["iters"]):
            c.constructSolution()
            bests.append(c.getIterBestDist())
        return {"iter_bests": np.array(bests, dtype=np.int64), **_results(c)}
    c.run(state["iters"])
    return _results(c)


def work(case):
    kind = case["kind"]
    if kind in ("train", "score"):
        if kind == "train":
            edges = case["epochs"] * case["k"] * sum(_sizes(case))
            read = 2 * FEATURES * edges + 4 * edges
        else:
            edges = case["edges"]
            read = 4 * FEATURES * edges + 8 * edges
        macs = FEATURES * HIDDEN + HIDDEN * HIDDEN + HIDDEN  # forward; twice that backward
        passes = 3 if kind == "train" else 4
        return {"bytes": read, "flops": 2 * macs * passes * edges}
    total = {"bytes": 0, "flops": 0}
    for n in _sizes(case) if kind == "batch" else [case["n"]]:
        m, k = min(case["m"], n) if kind == "batch" else case["m"], case["k"] or n
        # A step adds the weights of the row's unvisited candidates, and looks
        # for the crossing among them; a converged row is read once an iteration.
        steps = m * sum(min(k, n - x) for x in (1, n // 4, n // 2, 3 * n // 4)) * (n - 1) // 4
        total["flops"] += case["iters"] * 2 * steps
        total["bytes"] += case["iters"] * (6 * n * k + 4 * m * n + 12 * n * n)
        total["bytes"] += 12 * n * n + 4 * n * k  # setup: distances, heuristic, lists
    return total


def exact(case, seed):
    """64-bit loss, gradient and scores of the network on a labelled set.  The
    other cases' outputs are draws of a random process (tours and what they
    deposit) or a training run in shuffled batches: no 64-bit value exists that
    does not follow the engine's own 32-bit draws."""
    if case["kind"] != "score":
        return None
    shapes = {"W1": (HIDDEN, FEATURES), "b1": (HIDDEN,), "W2": (HIDDEN, HIDDEN),
              "b2": (HIDDEN,), "w3": (HIDDEN,), "b3": (1,)}
    parts = torch.from_numpy(_weights(seed)).double().split([math.prod(s) for s in shapes.values()])
    w = {k: v.reshape(s).clone().requires_grad_(True)
         for (k, s), v in zip(shapes.items(), parts)}
    feats, labels = _examples(case["edges"], seed)
    x, y = torch.from_numpy(feats).double(), torch.from_numpy(labels).double()
    h = torch.relu(x @ w["W1"].T + w["b1"])
    z = torch.relu(h @ w["W2"].T + w["b2"]) @ w["w3"] + w["b3"]
    sp = torch.nn.functional.softplus
    loss = (9.0 * y * sp(-z) + (1.0 - y) * sp(z)).sum() / len(labels)
    loss.backward()
    grads = torch.cat([v.grad.reshape(-1) for v in w.values()])
    return {"loss": loss.item(), "grads": grads.numpy(),
            "probs": torch.sigmoid(z).detach().numpy()}
