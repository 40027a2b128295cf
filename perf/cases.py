"""Workloads of the framework, one pass each through its public entry points.

Run from the repository root (the package lives in cuda-moea_b200/).  A case
is a dict of plain values; its "path" says what a pass is:

- "run": a complete optimisation.  The program keeps one Algorithm and restarts
  it for every further seeded repetition (reset(), then run()), which is how
  statistics over repeated runs are taken.  Returns the final population.
- "callback": the same with a problem that the user evaluates in torch.
- "batch": twenty generations of many independent instances advancing together.
- "select": one NSGA-III environmental selection of a merged population, the
  call that another framework's generation loop makes.
- "igd": the quality indicator of a population against a sampled front.

Runs are chaotic in their rounding (one changed bit changes later survivors),
so a 64-bit restatement has no value to offer for them; the selection's ideal
point and the indicator have one.
"""
from __future__ import annotations

import math
import os
import sys

import torch

_PACKAGE = os.path.abspath("cuda-moea_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import cuda_moea as cm  # noqa: E402
from cuda_moea import metrics, stages  # noqa: E402

BATCH_GENERATIONS = 20  # even: every population is back in the slot its view shows


def listed():
    return [
        # The small textbook configuration: 91 directions, 92 points.  Nothing but
        # the latency of the chain of stages counts.
        {"name": "nsga3_small", "path": "run", "algorithm": "NSGA3", "problem": "DTLZ2", "N": 92, "M": 3, "D": 12,
         "T": 100, "partitions": 12, "copy": 0.0},
        # The population size and operators of the usual quality comparisons.
        {"name": "nsga3_medium", "path": "run", "algorithm": "NSGA3", "problem": "DTLZ2", "N": 1024, "M": 3,
         "D": 12, "T": 100, "partitions": 43, "copy": 0.5},
        # A ragged mid-size population with five objectives and a multimodal problem,
        # directions picked from the population size.
        {"name": "nsga3_ragged", "path": "run", "algorithm": "NSGA3", "problem": "DTLZ3", "N": 3002, "M": 5,
         "D": 14, "T": 50, "partitions": 0, "copy": 0.0},
        # The large-population throughput configuration.
        {"name": "nsga3_large", "path": "run", "algorithm": "NSGA3", "problem": "DTLZ1", "N": 32768, "M": 3,
         "D": 7, "T": 50, "partitions": 254, "copy": 0.0},
        # Many objectives: nearly every point is non-dominated, 6435 directions.
        {"name": "nsga3_many", "path": "run", "algorithm": "NSGA3", "problem": "DTLZ2", "N": 6436, "M": 8,
         "D": 17, "T": 50, "partitions": 8, "copy": 0.0},
        # Constrained, ten objectives, few directions (two layers, 275).
        {"name": "nsga3_constrained", "path": "run", "algorithm": "NSGA3", "problem": "C3DTLZ4", "N": 16384,
         "M": 10, "D": 14, "T": 20, "partitions": -1, "copy": 0.0},
        # RVEA at the size of the usual quality comparisons.
        {"name": "rvea_medium", "path": "run", "algorithm": "RVEA", "problem": "DTLZ2", "N": 990, "M": 3, "D": 12,
         "T": 100, "partitions": 0, "copy": 0.5},
        # RVEA with very many decision variables: memory-bound variation and evaluation.
        {"name": "rvea_wide", "path": "run", "algorithm": "RVEA", "problem": "DTLZ2", "N": 1024, "M": 8,
         "D": 131072, "T": 50, "partitions": 0, "copy": 0.0},
        # The user's own problem, evaluated in torch on the algorithm's stream.
        {"name": "nsga3_callback", "path": "callback", "N": 2048, "M": 3, "D": 16, "T": 20},
        # Many small instances of uneven size, objectives and problem at once.
        {"name": "batch_mixed", "path": "batch", "count": 256, "low": 92, "high": 4096, "mix": 0},
        # One selection of a merged population inside somebody else's loop.
        {"name": "select_ragged", "path": "select", "n": 20014, "M": 5, "partitions": 20, "infeasible": 0.0},
        # The indicator of a population against the usual 20000 front samples.
        {"name": "igd_medium", "path": "igd", "n": 1024, "R": 20000, "M": 3, "filter": True},
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _even(n):
    return n + n % 2


def draw(rng):
    path = rng.choice(["run", "run", "run", "rvea", "wide", "callback", "batch", "select", "igd"])
    if path == "run":
        M = rng.choice([2, 3, 3, 3, 5, 8, 10])
        N = _even(_log_int(rng, 92, 32768 if M <= 3 else 16384 if M <= 5 else 6436))
        problem = rng.choice(["DTLZ1", "DTLZ2", "DTLZ3", "DTLZ4", "DTLZ5", "DTLZ6", "DTLZ7", "C1DTLZ1", "C2DTLZ2"])
        return {"path": "run", "algorithm": "NSGA3", "problem": problem, "N": N, "M": M,
                "D": M + rng.randint(4, 19), "T": rng.randint(20, 60) if N <= 4096 else 20, "partitions": 0,
                "copy": rng.choice([0.0, 0.5])}
    if path == "rvea":
        M = rng.choice([2, 3, 5, 8])
        return {"path": "run", "algorithm": "RVEA", "problem": rng.choice(["DTLZ1", "DTLZ2", "DTLZ3", "DTLZ4"]),
                "N": _log_int(rng, 92, 8192), "M": M, "D": M + rng.randint(4, 200), "T": rng.randint(20, 100),
                "partitions": 0, "copy": rng.choice([0.0, 0.5])}
    if path == "wide":
        M = rng.choice([2, 3, 5, 8])
        N = _log_int(rng, 128, 2048)
        D = _log_int(rng, 1000, min(131072, (1 << 26) // N))
        return {"path": "run", "algorithm": "RVEA", "problem": rng.choice(["DTLZ1", "DTLZ2", "DTLZ3", "DTLZ4"]),
                "N": N, "M": M, "D": D, "T": 20, "partitions": 0, "copy": rng.choice([0.0, 0.5])}
    if path == "callback":
        M = rng.choice([2, 3, 5])
        return {"path": "callback", "N": _even(_log_int(rng, 92, 8192)), "M": M, "D": rng.randint(M + 1, 40), "T": 20}
    if path == "batch":
        low = _log_int(rng, 92, 1000)
        return {"path": "batch", "count": _log_int(rng, 32, 256), "low": low, "high": rng.randint(low + 40, 4096),
                "mix": rng.randint(1, 1 << 20)}
    if path == "select":
        M = rng.choice([2, 3, 5, 8])
        return {"path": "select", "n": _even(_log_int(rng, 184, 40000 if M <= 5 else 16000)), "M": M,
                "partitions": rng.randint(*{2: (50, 400), 3: (12, 120), 5: (4, 20), 8: (2, 8)}[M]),
                "infeasible": rng.choice([0.0, 0.0, 0.4])}
    return {"path": "igd", "n": _log_int(rng, 92, 8192), "R": _log_int(rng, 1000, 50000),
            "M": rng.choice([2, 3, 5, 8]), "filter": rng.random() < 0.7}


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _sphere_rows(n, M, spread, gen):
    """Objectives of a population on its way to the unit-sphere front: directions
    of the positive orthant, radius 1 plus an exponential excess."""
    u = torch.rand((n, M), generator=gen, device="cuda").clamp_min(1e-6)
    g = -torch.log(torch.rand((n, 1), generator=gen, device="cuda").clamp_min(1e-6)) * spread
    return u / u.norm(dim=1, keepdim=True) * (1.0 + g)


class Spheres(cm.PythonProblem):
    """Squared distances to M seeded centres."""

    def __init__(self, dimension, objectives, seed):
        super().__init__(dimension, objectives)
        self.centres = torch.rand((objectives, dimension), generator=_generator(seed), device="cuda")

    def evaluate(self, variables, context):
        return (variables[:, None, :] - self.centres).square().sum(2)


def _algorithm(case, seed):
    directions = None
    if case["algorithm"] == "NSGA3":
        directions = (cm.UserDefinedDirections(cm.two_layer_directions(case["M"], 3, 2))
                      if case["partitions"] < 0 else cm.DasDennisDirections(case["partitions"]))
    return cm.Algorithm(case["algorithm"], population_size=case["N"], max_generations=case["T"],
                        problem=getattr(cm, case["problem"])(case["D"], case["M"]),
                        crossover=cm.SBX(variable_copy_probability=case["copy"]), reference_directions=directions,
                        seed=seed, print_progress=False)


def _batch_specs(case):
    gen = torch.Generator().manual_seed(case["mix"])

    def pick(low, high):
        return int(torch.randint(low, high, (1,), generator=gen))
    specs = []
    for i in range(case["count"]):
        kind, M = pick(1, 8), (3, 5, 8)[pick(0, 3)]
        specs.append((kind, M, _even(pick(case["low"], case["high"] + 1) & ~1), M + (19 if kind == 7 else 9)))
    return specs


def _directions(M, partitions):
    return stages.reference_directions(1, partitions, M).cuda()


def prepare(case, seed):
    path = case["path"]
    if path == "run":
        algorithm = _algorithm(case, seed)
        algorithm.initialize()
        return {"path": path, "algorithm": algorithm}
    if path == "callback":
        algorithm = cm.NSGA3(population_size=case["N"], max_generations=case["T"],
                             problem=Spheres(case["D"], case["M"], seed), seed=seed, print_progress=False)
        algorithm.initialize()
        return {"path": path, "algorithm": algorithm}
    if path == "batch":
        batch = cm.Batch([cm.NSGA3(population_size=N, max_generations=20000, problem=getattr(cm, f"DTLZ{k}")(D, M),
                                   seed=seed + i, print_progress=False)
                          for i, (k, M, N, D) in enumerate(_batch_specs(case))])
        populations = [batch.population(i, copy=False) for i in range(len(batch))]
        return {"path": path, "batch": batch,
                "variables": [p.variables.reshape(-1) for p in populations],
                "objectives": [p.objectives.t().reshape(-1) for p in populations]}
    gen = _generator(seed)
    if path == "select":
        n, M = case["n"], case["M"]
        refs = _directions(M, case["partitions"])
        half = n // 2
        objs = torch.cat([_sphere_rows(half, M, 0.05, gen), _sphere_rows(n - half, M, 0.08, gen)]).t().contiguous()
        cv = torch.rand(n, generator=gen, device="cuda")
        cv = torch.where(torch.rand(n, generator=gen, device="cuda") < case["infeasible"], cv, torch.zeros_like(cv))
        return {"path": path, "workspace": stages.Workspace(n, M, refs.shape[1]), "objs": objs, "cv": cv,
                "refs": refs, "seed": int(seed) & 0x7FFFFFFF, "ideal": objs[:, :half].amin(dim=1)}
    front = _sphere_rows(case["n"], case["M"], 0.01, gen)
    samples = _sphere_rows(case["R"], case["M"], 0.0, gen).double()
    return {"path": path, "workspace": stages.Workspace(max(2, case["n"]), case["M"], 1), "front": front,
            "samples": samples, "filter": case["filter"]}


def run(state):
    path = state["path"]
    if path in ("run", "callback"):
        algorithm = state["algorithm"]
        if algorithm.finished:
            algorithm.reset()
        r = algorithm.run()
        # RVEA lists the non-dominated rows (a number of them that depends on the run)
        indices = torch.nn.functional.pad(r.auxiliary_indices, (0, r.variables.shape[0] - len(r.auxiliary_indices)),
                                          value=-1)
        return {"variables": r.variables, "objectives": r.objectives, "constraints": r.constraints,
                "indices": indices, "active": r.active_count}
    if path == "batch":
        state["batch"].run(BATCH_GENERATIONS)
        return {"variables": torch.cat(state["variables"]), "objectives": torch.cat(state["objectives"])}
    if path == "select":
        return stages.nsga3_select(state["workspace"], state["cv"], state["objs"], state["refs"], state["seed"], 0,
                                   state["ideal"])
    return metrics.igd(state["front"], state["samples"], filter_nondominated=state["filter"],
                       workspace=state["workspace"])


def exact(case, seed):
    if case["path"] == "select":
        s = prepare(case, seed)
        return {"survivors": None, "fronts": None, "sizes": None, "offset": None,
                "ideal": s["objs"].double().amin(dim=1)}
    if case["path"] != "igd":
        return None
    s = prepare(case, seed)
    front = s["front"].double()
    if case["filter"]:
        keep = []
        for q in front.split(256):
            no_worse = (front[:, None, :] <= q[None, :, :]).all(2)
            better = (front[:, None, :] < q[None, :, :]).any(2)
            keep.append(~(no_worse & better).any(0))
        front = front[torch.cat(keep)]
    nearest = [(q[:, None, :] - front[None, :, :]).square().sum(2).amin(1).sqrt()
               for q in s["samples"].split(max(1, (1 << 24) // (front.shape[0] * case["M"])))]
    return float(torch.cat(nearest).mean())


def _generation(N, M, D):
    """Bytes and operations that one generation cannot do without: parents read,
    children and survivors written; about 60 operations per variable (the draws and
    two powers), the objective sums, and one sort of the merged objectives."""
    n = 2 * N
    return 4.0 * N * (3 * (D + M) + 5), 60.0 * N * D + 2.0 * M * n * math.log2(n)


def work(case):
    path = case["path"]
    if path in ("run", "callback"):
        b, f = _generation(case["N"], case["M"], case["D"])
        return {"bytes": b * case["T"], "flops": f * case["T"]}
    if path == "batch":
        N = (case["low"] + case["high"]) / 2
        b, f = _generation(N, 5, 15)
        return {"bytes": b * case["count"] * BATCH_GENERATIONS, "flops": f * case["count"] * BATCH_GENERATIONS}
    if path == "select":
        n, M = case["n"], case["M"]
        H = math.comb(case["partitions"] + M - 1, M - 1)
        return {"bytes": 4.0 * (n * (M + 1) + M * H + n + M), "flops": 2.0 * M * n * math.log2(n)}
    n, R, M = case["n"], case["R"], case["M"]
    return {"bytes": 4.0 * n * M + 8.0 * R * M + 8.0, "flops": 3.0 * M * n * R}
