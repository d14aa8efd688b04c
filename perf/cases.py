"""The work that a user of this framework has it do, as timed cases.

Every case goes through a public entry point: the local-search strategies
(`improve` / `improve_batch`), the population operators of one modular generation, the
fused GA solvers, and the learned candidate lists. Instances are uniform cities or
Gaussian clusters in a 1000 x 1000 square with EUC_2D distances, as the repository's own
workloads are; starting tours are random permutations. Each pass of a GA case builds the
problem from its coordinates, as a program with a new instance does; the batch case keeps
its instances' k-NN tables, as the repository's uneven batch workload does.

A case is a dict of plain values; `op` picks the entry point and the rest are its sizes
and options.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from tsp_gpu_clean_b200.batch import FusedBatchSolver
from tsp_gpu_clean_b200.device import candidate_list
from tsp_gpu_clean_b200.fused import FusedMemeticSolver, LocalSearchConfig
from tsp_gpu_clean_b200.learned import EdgeScorer, LearnedCandidates, device_instance
from tsp_gpu_clean_b200.problem import Problem, ProblemContext
from tsp_gpu_clean_b200.strategies import (
  CrossoverB200PermOrder,
  CrossoverB200PermPartiallyMapped,
  EvaluationB200Cost,
  LocalSearchB200OrOpt,
  LocalSearchB200ThreeOpt,
  LocalSearchB200TourTwoOpt,
  MutationB200PermInversion,
  MutationB200PermSwap,
  SelectionB200Tournament,
)

#: "until a local optimum": more passes than any refinement here takes
ALL = 10**9

#: parameter block of the edge-scoring MLP: W1 (16 x 64, five rows used), b1, W2, b2, w3, b3
HIDDEN, INPUTS, FEATURES = 64, 16, 5
OFF_B1 = INPUTS * HIDDEN
OFF_W2 = OFF_B1 + HIDDEN
OFF_B2 = OFF_W2 + HIDDEN * HIDDEN
OFF_W3 = OFF_B2 + HIDDEN
OFF_B3 = OFF_W3 + HIDDEN
PARAMS = OFF_B3 + 1
TRAIN_STEP = 200  # Adam steps behind the training case's state
LR = 3e-3


def listed() -> list[dict]:
  return [
    # one route polished with the strategy's defaults (exhaustive best improvement, ten
    # passes): the smallest call, bound by latency; NumPy in and out
    {"name": "polish_one", "op": "two_opt", "n": 200, "tours": 1, "mode": "best", "k": 0, "iters": 10, "host": True,
     "clustered": False},
    # one generation of the modular GA, strategy by strategy, on a device-resident
    # population: evaluation, tournament, crossover, mutation, evaluation
    {"name": "operators", "op": "operators", "n": 1000, "rows": 512, "crossover": "pmx", "mutation": "inversion",
     "host": False},
    # the repository's 2-opt benchmark: random tours of a clustered instance refined to a
    # local optimum with k-NN candidates, best improvement, NumPy in and out
    {"name": "refine_best", "op": "two_opt", "n": 1000, "tours": 1024, "mode": "best", "k": 20, "iters": ALL,
     "host": True, "clustered": True},
    # the same with first improvement on device tensors
    {"name": "refine_first", "op": "two_opt", "n": 1000, "tours": 1024, "mode": "first", "k": 20, "iters": ALL,
     "host": False, "clustered": True},
    # the exhaustive neighbourhood (no candidate list) for a population to a local optimum
    {"name": "refine_exhaustive", "op": "two_opt", "n": 500, "tours": 128, "mode": "best", "k": 0, "iters": ALL,
     "host": False, "clustered": False},
    # many moves per pass, as a post-mutation local search of a population uses it
    {"name": "refine_multi", "op": "two_opt", "n": 1002, "tours": 256, "mode": "multi_move", "k": 20, "iters": 10,
     "host": False, "clustered": False},
    # the repository's Or-opt benchmark
    {"name": "or_opt", "op": "or_opt", "n": 1000, "tours": 1024, "k": 20, "segment": 3, "iters": 50, "host": False,
     "clustered": True},
    # the 3-opt strategy's defaults (exhaustive steepest descent, ten passes)
    {"name": "three_opt", "op": "three_opt", "n": 200, "tours": 32, "mode": "batch", "k": 0, "inner": 0, "iters": 10,
     "host": False},
    # a whole memetic GA run on a new 1000-city instance, problem set-up included
    {"name": "ga_run", "op": "ga", "n": 1000, "rows": 512, "gens": 100, "elite": 64, "crossover": "pmx",
     "mutation": "inversion", "init": "nn", "stage": "none", "clustered": True},
    # many GA runs of uneven size in one batch, from coordinates and k-NN tables in hand
    {"name": "ga_batch", "op": "ga_batch", "count": 128, "n_min": 50, "n_max": 5000, "rows": 64, "gens": 50, "elite": 8},
    # learned candidate lists of a new 10,000-city instance: distance matrix, k-NN pool,
    # edge features, MLP inference, top-k selection
    {"name": "learned_table", "op": "table", "n": 10000, "pool": 30, "k": 10},
    # one optimiser step of the edge-scoring MLP on a full batch
    {"name": "train_step", "op": "train", "edges": 65536},
  ]


def _log(rng, lo: int, hi: int) -> int:
  return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
  op = rng.choice(["two_opt_knn", "two_opt_knn", "two_opt_all", "multi", "or_opt", "three_opt", "operators", "ga", "ga",
                   "ga_batch", "table", "train"])
  host = rng.random() < 0.5
  if op == "two_opt_knn":
    return {"op": "two_opt", "n": _log(rng, 100, 2000), "tours": _log(rng, 1, 512), "mode": rng.choice(["best", "first"]),
            "k": rng.choice([8, 10, 15, 20]), "iters": rng.choice([10, ALL]), "host": host,
            "clustered": rng.random() < 0.5}
  if op == "two_opt_all":
    return {"op": "two_opt", "n": _log(rng, 50, 500), "tours": _log(rng, 1, 128), "mode": rng.choice(["best", "first"]),
            "k": 0, "iters": rng.choice([10, ALL]), "host": host, "clustered": rng.random() < 0.5}
  if op == "multi":
    return {"op": "two_opt", "n": _log(rng, 100, 1200), "tours": _log(rng, 1, 256), "mode": "multi_move",
            "k": rng.choice([10, 15, 20]), "iters": rng.choice([5, 10]), "host": host, "clustered": rng.random() < 0.5}
  if op == "or_opt":
    return {"op": "or_opt", "n": _log(rng, 100, 1500), "tours": _log(rng, 1, 600), "k": rng.choice([10, 15, 20]),
            "segment": rng.choice([1, 2, 3]), "iters": rng.choice([10, 50]), "host": host,
            "clustered": rng.random() < 0.5}
  if op == "three_opt":
    k = rng.choice([0, 0, 8, 10])
    n = _log(rng, 20, 200) if k == 0 else _log(rng, 50, 500)
    return {"op": "three_opt", "n": n, "tours": _log(rng, 1, 32), "mode": rng.choice(["batch", "multi_move"]) if k else
            "batch", "k": k, "inner": rng.choice([0, 4]) if k else 0, "iters": rng.choice([5, 10]), "host": host}
  if op == "operators":
    return {"op": "operators", "n": _log(rng, 100, 2000), "rows": _log(rng, 64, 512),
            "crossover": rng.choice(["pmx", "ox"]), "mutation": rng.choice(["inversion", "swap"]), "host": host}
  if op == "ga":
    rows = _log(rng, 64, 512)
    stage = rng.choice(["none", "none", "post_mutation"])
    return {"op": "ga", "n": _log(rng, 100, 1500), "rows": rows, "gens": rng.randrange(20, 101),
            "elite": 0 if stage == "post_mutation" else max(1, rows // 8), "crossover": rng.choice(["pmx", "ox"]),
            "mutation": rng.choice(["inversion", "swap"]), "init": rng.choice(["nn", "random"]), "stage": stage,
            "clustered": rng.random() < 0.5}
  if op == "ga_batch":
    return {"op": "ga_batch", "count": _log(rng, 8, 100), "n_min": 50, "n_max": _log(rng, 500, 5000),
            "rows": rng.choice([32, 48, 64]), "gens": rng.randrange(10, 51), "elite": rng.choice([4, 8])}
  if op == "table":
    return {"op": "table", "n": _log(rng, 500, 9999), "pool": rng.choice([16, 20, 30]), "k": rng.choice([8, 10])}
  return {"op": "train", "edges": _log(rng, 2000, 65535)}


# ------------------------------------------------------------------------------ inputs
def _coords(n: int, clustered: bool, rng) -> np.ndarray:
  if not clustered:
    return rng.uniform(0.0, 1000.0, (n, 2))
  centres = rng.uniform(0.0, 1000.0, (20, 2))
  return np.clip(centres[rng.integers(0, 20, n)] + rng.normal(0.0, 30.0, (n, 2)), 0.0, 1000.0)


def _tours(n: int, count: int, rng) -> np.ndarray:
  return np.argsort(rng.random((count, n)), axis=1).astype(np.int32)


def _batch_coords(case: dict, rng) -> list[np.ndarray]:
  out = []
  order = np.random.default_rng(case["count"]).permutation(case["count"])
  for i in range(case["count"]):  # sizes log-uniform over the range, the same for every seed
    n = int(round(case["n_min"] * (case["n_max"] / case["n_min"]) ** ((order[i] + 0.5) / case["count"])))
    out.append(_coords(n, i % 2 == 1, rng))
  return out


def _mlp_params(rng) -> np.ndarray:
  p = np.zeros(PARAMS, dtype=np.float32)
  p[: FEATURES * HIDDEN] = rng.normal(0.0, math.sqrt(2.0 / FEATURES), FEATURES * HIDDEN)
  p[OFF_B1:OFF_W2] = rng.normal(0.0, 0.1, HIDDEN)
  p[OFF_W2:OFF_B2] = rng.normal(0.0, math.sqrt(2.0 / HIDDEN), HIDDEN * HIDDEN)
  p[OFF_B2:OFF_W3] = rng.normal(0.0, 0.1, HIDDEN)
  p[OFF_W3:OFF_B3] = rng.normal(0.0, math.sqrt(1.0 / HIDDEN), HIDDEN)
  p[OFF_B3] = -2.0
  return p


def _train_inputs(case: dict, seed: int):
  """Parameters, Adam state, features (BF16, padded to 16 columns) and labels of one batch."""
  rng = np.random.default_rng(seed)
  E = case["edges"]
  p = _mlp_params(rng)
  used = p != 0
  m = np.where(used, rng.normal(0.0, 1e-3, PARAMS), 0.0).astype(np.float32)
  v = np.where(used, rng.uniform(0.5e-4, 2e-4, PARAMS), 0.0).astype(np.float32)
  rank = rng.integers(0, 30, E)
  near = (rank + rng.uniform(0.0, 1.0, E)) / 30.0  # distance relative to the farthest of the pool
  angle = rng.uniform(0.0, 2.0 * math.pi, E)
  x = np.zeros((E, INPUTS), dtype=np.float32)
  x[:, 0] = np.sqrt(near)
  x[:, 1] = rank / 30.0
  x[:, 2] = np.clip(rank + rng.integers(-6, 7, E), 0, 30) / 30.0
  x[:, 3] = x[:, 0] * np.cos(angle)
  x[:, 4] = x[:, 0] * np.sin(angle)
  y = (rng.random(E) < np.where(rank < 4, 0.4, 0.02)).astype(np.float32)
  return p, m, v, torch.from_numpy(x).to(torch.bfloat16), torch.from_numpy(y)


# ------------------------------------------------------------------------------ state
def _two_opt(case):
  return LocalSearchB200TourTwoOpt(max_iterations=case["iters"], mode=case["mode"], candidate_k=case["k"] or None)


def _or_opt(case):
  return LocalSearchB200OrOpt(max_iterations=case["iters"], candidate_k=case["k"], max_segment=case["segment"])


def _three_opt(case):
  return LocalSearchB200ThreeOpt(max_iterations=case["iters"], mode=case["mode"], candidate_k=case["k"] or None,
                                 inner_candidate_k=case["inner"] or None)


SEARCHES = {"two_opt": _two_opt, "or_opt": _or_opt, "three_opt": _three_opt}


def prepare(case: dict, seed: int):
  op = case["op"]
  rng = np.random.default_rng(seed)
  if op in SEARCHES:
    ctx = ProblemContext(Problem.from_coordinates(_coords(case["n"], case.get("clustered", False), rng)), seed=seed)
    tours = _tours(case["n"], case["tours"], rng)
    return {"op": op, "search": SEARCHES[op](case), "ctx": ctx, "one": case["tours"] == 1,
            "tours": tours if case["host"] else torch.from_numpy(tours).cuda()}
  if op == "operators":
    ctx = ProblemContext(Problem.from_coordinates(_coords(case["n"], True, rng)), seed=seed)
    pop = _tours(case["n"], case["rows"], rng)
    return {
      "op": op, "ctx": ctx, "pop": pop if case["host"] else torch.from_numpy(pop).cuda(),
      "eval": EvaluationB200Cost(), "select": SelectionB200Tournament(k=5),
      "cross": CrossoverB200PermPartiallyMapped() if case["crossover"] == "pmx" else CrossoverB200PermOrder(),
      "mutate": MutationB200PermInversion() if case["mutation"] == "inversion" else MutationB200PermSwap(),
    }
  if op == "ga":
    return {"op": op, "case": case, "coords": _coords(case["n"], case["clustered"], rng), "seed": seed}
  if op == "ga_batch":
    coords, tables = _batch_coords(case, rng), []
    for x in coords:
      ctx = ProblemContext(Problem.from_coordinates(x), seed=0)
      tables.append({k: candidate_list(ctx, k) for k in (5, 20)})
    return {"op": op, "case": case, "coords": coords, "tables": tables, "seed": seed}
  if op == "table":
    coords = _coords(case["n"], False, rng)
    learned = LearnedCandidates(pool_k=case["pool"], seed=0)
    learned.scorer.params.copy_(torch.from_numpy(_mlp_params(rng)))
    return {"op": op, "coords": coords, "learned": learned, "pool": case["pool"], "k": case["k"]}
  p, m, v, x, y = _train_inputs(case, seed)
  scorer = EdgeScorer(0)
  scorer.params.copy_(torch.from_numpy(p))
  scorer.m.copy_(torch.from_numpy(m))
  scorer.v.copy_(torch.from_numpy(v))
  scorer.step = TRAIN_STEP
  return {"op": op, "scorer": scorer, "x": x.view(torch.int16).cuda(), "y": y.cuda()}


# ------------------------------------------------------------------------------ one pass
def run(state):
  op = state["op"]
  if op in SEARCHES:
    if state["one"]:
      return state["search"].improve(state["tours"][0], state["ctx"])
    return state["search"].improve_batch(state["tours"], state["ctx"])
  if op == "operators":
    ctx, pop = state["ctx"], state["pop"]
    fitness = state["eval"].evaluate_batch(pop, ctx)
    parents = state["select"].select_batch(pop, fitness, context=ctx)
    children = state["cross"].crossover_batch(parents, ctx)
    children = state["mutate"].mutate_batch(children, 0.05, ctx)
    return {"fitness": fitness, "children": children, "cost": state["eval"].evaluate_batch(children, ctx)}
  if op == "ga":
    c = state["case"]
    ctx = ProblemContext(Problem.from_coordinates(state["coords"]), seed=state["seed"])
    solver = FusedMemeticSolver(population_size=c["rows"], mutation_rate=0.05, tournament_k=5, nn_k=5,
                                local_search=LocalSearchConfig("best", 10, 20), elite_count=c["elite"],
                                post_init=c["stage"] == "none", crossover=c["crossover"], mutation=c["mutation"],
                                init=c["init"], local_search_stage=c["stage"])
    best, stats = solver.evolve(ctx, list(range(c["n"])), c["gens"], patience=ALL)
    return {"best": best, "history": np.asarray(stats["convergence_history"]), "population": solver.final_population,
            "fitness": solver.final_fitness}
  if op == "ga_batch":
    c = state["case"]
    ctxs = [ProblemContext(Problem.from_coordinates(x), seed=state["seed"] + i, candidate_cache=dict(t))
            for i, (x, t) in enumerate(zip(state["coords"], state["tables"]))]
    solver = FusedBatchSolver(population_size=c["rows"], mutation_rate=0.05, tournament_k=5, nn_k=5,
                              local_search=LocalSearchConfig("best", 10, 20), elite_count=c["elite"], post_init=True)
    runs = solver.evolve(ctxs, c["gens"], patience=ALL)
    return {"best": np.concatenate([best for best, _ in runs]),
            "history": np.asarray([stats["convergence_history"] for _, stats in runs])}
  if op == "table":
    inst = device_instance(state["coords"], state["pool"])
    return {"dist": inst.dist, "pool": inst.pool, "table": state["learned"].table(inst, state["k"])}
  scorer = state["scorer"]
  loss = scorer.train_step(state["x"], state["y"], LR)
  return {"loss": loss, "params": scorer.params, "m": scorer.m, "v": scorer.v}


# ------------------------------------------------------------------------------ what a pass needs
def work(case: dict) -> dict:
  """Inputs read once and outputs written once; the MLP step also counts its products. The
  searches do integer arithmetic and comparisons only."""
  op = case["op"]
  if op in SEARCHES:
    n = case["n"]  # tours in and out, the distance matrix, the k-NN table with its distances
    return {"bytes": 8 * n * case["tours"] + 4 * n * n + 8 * n * case["k"], "flops": 0}
  if op == "operators":
    n, rows = case["n"], case["rows"]  # population in, children out, both fitness vectors, the matrix
    return {"bytes": 8 * n * rows + 16 * rows + 4 * n * n, "flops": 0}
  if op == "ga":
    n, rows = case["n"], case["rows"]  # coordinates in; population, fitness, tour and history out
    return {"bytes": 20 * n + 4 * n * rows + 8 * rows + 8 * case["gens"], "flops": 0}
  if op == "ga_batch":
    mean = (case["n_max"] - case["n_min"]) / math.log(case["n_max"] / case["n_min"])
    return {"bytes": int(case["count"] * (20 * mean + 8 * case["gens"])), "flops": 0}
  if op == "table":
    n = case["n"]  # coordinates in; matrix, pool and table out (the matrix is part of the instance)
    edges = n * case["pool"]
    return {"bytes": 16 * n + 4 * n * n + 4 * edges + 4 * n * case["k"],
            "flops": 2 * edges * (FEATURES * HIDDEN + HIDDEN * HIDDEN + HIDDEN)}
  E = case["edges"]
  products = FEATURES * HIDDEN + HIDDEN * HIDDEN + HIDDEN
  return {"bytes": E * (2 * INPUTS + 4) + 6 * 4 * PARAMS, "flops": 2 * E * (3 * products - FEATURES * HIDDEN)}


# ------------------------------------------------------------------------------ 64-bit values
def _exact_costs(coords: np.ndarray, tours: np.ndarray) -> np.ndarray:
  p = coords[tours]
  d = np.roll(p, -1, axis=1) - p
  return np.floor(np.sqrt((d * d).sum(axis=2)) + 0.5).sum(axis=1)


def _exact_train(case: dict, seed: int) -> dict:
  p, m, v, x, y = (torch.as_tensor(a).double() for a in _train_inputs(case, seed))
  p.requires_grad_(True)
  w1, b1 = p[:OFF_B1].view(INPUTS, HIDDEN), p[OFF_B1:OFF_W2]
  w2, b2 = p[OFF_W2:OFF_B2].view(HIDDEN, HIDDEN), p[OFF_B2:OFF_W3]
  h = torch.relu(torch.relu(x @ w1 + b1) @ w2 + b2)
  loss = torch.nn.functional.binary_cross_entropy_with_logits(h @ p[OFF_W3:OFF_B3] + p[OFF_B3], y)
  loss.backward()
  g, t = p.grad, TRAIN_STEP + 1
  m = 0.9 * m + 0.1 * g
  v = 0.999 * v + 0.001 * g * g
  q = p.detach() - LR * (m / (1.0 - 0.9**t)) / (torch.sqrt(v / (1.0 - 0.999**t)) + 1e-8)
  return {"loss": float(loss.detach()), "params": q, "m": m, "v": v}


def exact(case: dict, seed: int):
  """Tours and tables are whole numbers; GA histories are whole-number lengths of runs that
  plain NumPy would take minutes for. Tour costs and the MLP step have 64-bit values."""
  if case["op"] == "operators":
    rng = np.random.default_rng(seed)
    coords = _coords(case["n"], True, rng)
    return {"fitness": _exact_costs(coords, _tours(case["n"], case["rows"], rng)), "children": None, "cost": None}
  if case["op"] == "train":
    return _exact_train(case, seed)
  return None
