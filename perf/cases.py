"""Performance cases: the work that users of paragraph_gb300 have it do, through its public calls.

A case is one call (or one driver's sequence of stage calls) on data of the repository's own
generator (paragraph_gb300.datagen: Gaussian mixture base, training queries of another modality,
exact top-128 ground truth).  Kinds:

  build    an index build from device tensors (projection + two link rounds), plain FP32 or
           screened on the tensor cores
  host     the same from pinned host buffers, results copied back: the whole call counts
  batched  many uneven sub-indexes in one call, replayed from a CUDA graph
  index    the driver's whole index: build, MatchSup rounds, FusionNN, FusionFinal
  stages   a driver that calls the pipeline's stages one by one
  query    beam search of external queries over a built graph
  gt       exact inner-product top-k of every query
"""
from __future__ import annotations

import math

import torch

import paragraph_gb300 as pg
from paragraph_gb300 import datagen

GT_K = 128
PROJ = 16
MATCH_ROUNDS, M_NN, M_FINAL = 6, 40, 70
SCREENS = {"none": pg.SCREEN_NONE, "fp16": pg.SCREEN_FP16, "bf16": pg.SCREEN_BF16}


def listed():
    return [
        # a shard of a few hundred points rebuilt on the fly: launches and latency
        dict(name="build-1k", kind="build", n=1000, q=1000, d=200, degree=32, beam=64,
             screen="fp16", cosine=False, centers=64),
        # the 100k x 200 configuration
        dict(name="build-100k", kind="build", n=100_000, q=100_000, d=200, degree=32, beam=64,
             screen="fp16", cosine=False, centers=64),
        # the headline 1M x 200 inner-product build of bench.py
        dict(name="build-1m", kind="build", n=1_000_000, q=1_000_000, d=200, degree=32, beam=64,
             screen="fp16", cosine=False, centers=64),
        # the precision configuration: 1M x 512 cosine, M = 48, L = 96
        dict(name="build-cosine-1m", kind="build", n=1_000_000, q=1_000_000, d=512, degree=48,
             beam=96, screen="fp16", cosine=True, centers=128),
        # default parameters (no screening) at the reference driver's own degree, ragged size
        dict(name="build-plain-120k", kind="build", n=120_007, q=90_001, d=512, degree=55, beam=64,
             screen="none", cosine=True, centers=128),
        # data in host memory: pinned buffers in, graph and projection out
        dict(name="host-250k", kind="host", n=250_000, q=250_000, d=200, degree=32, beam=64,
             screen="fp16", cosine=False, centers=64),
        # uneven sub-indexes (log-uniform sizes, D = 512) in one replayed CUDA graph
        dict(name="batched-16", kind="batched", count=16, smallest=5_000, largest=80_000, d=512,
             degree=32, beam=64, screen="fp16", cosine=False, centers=64),
        # the file that the reference's driver writes, from device tensors
        dict(name="index-200k", kind="index", n=200_000, q=200_000, d=200, degree=32, beam=64,
             screen="fp16", cosine=False, centers=64),
        # a driver that swaps the reference's launches one for one, odd size
        dict(name="stages-33k", kind="stages", n=33_333, q=25_000, d=128, degree=32, beam=64,
             screen="none", cosine=False, centers=64),
        # evaluation run over a held-out query set
        dict(name="query-20k", kind="query", n=400_000, q=200_000, nq=20_000, d=200, degree=32,
             beam=96, topk=10, screen="fp16", cosine=False, centers=64),
        # a few online queries: the latency of one small call
        dict(name="query-16", kind="query", n=100_000, q=100_000, nq=16, d=200, degree=32, beam=64,
             topk=10, screen="fp16", cosine=False, centers=64),
        # ground truth for a training set
        dict(name="gt-300k", kind="gt", n=300_001, q=250_000, d=200, k=128, cosine=False,
             centers=64),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["build", "build", "build", "host", "batched", "index", "stages", "query",
                       "gt"])
    cosine = rng.random() < 0.4
    case = dict(kind=kind, d=4 * rng.randint(16, 128), cosine=cosine, centers=rng.choice([64, 128]))
    if kind == "gt":
        case.update(n=_log_int(rng, 1000, 500_000), q=_log_int(rng, 500, 400_000),
                    k=rng.choice([10, 100, 128]))
        return case
    case.update(degree=rng.choice([16, 24, 32, 48, 55]), beam=rng.choice([64, 64, 96, 128]),
                screen=rng.choice(["fp16", "fp16", "bf16", "none"]))
    if kind == "batched":
        smallest = _log_int(rng, 500, 10_000)
        case.update(count=rng.randint(3, 24), smallest=smallest,
                    largest=int(smallest * rng.uniform(2, 10)))
        return case
    top = {"build": 600_000, "host": 400_000, "index": 250_000, "stages": 150_000,
           "query": 300_000}[kind]
    n = _log_int(rng, 800, top)
    case.update(n=n, q=max(200, int(n * rng.uniform(0.3, 1.2))))
    if kind == "query":
        case.update(nq=_log_int(rng, 1, 20_000), topk=rng.choice([1, 10, 50]))
    return case


def _sizes(case):
    """Points of each sub-index: log-spaced from the smallest to the largest, shuffled evenly."""
    c, lo, hi = case["count"], case["smallest"], case["largest"]
    s = [int(round(lo * (hi / lo) ** (i / (c - 1)))) for i in range(c)]
    return s[1::2] + s[::2][::-1]


def _ground_truth(base, queries, k, gt):
    with pg.Handle(0) as h:
        h.ground_truth(base, queries, gt)


def _data(case, n, q, seed, extra=0):
    """base (n x d), gt (q x 128) and `extra` held-out queries, on the GPU."""
    base, _, queries = datagen.make_dataset_cuda(n, case["d"], q + extra, seed=seed,
                                                 cosine=case["cosine"], centers=case["centers"],
                                                 with_gt=False)
    gt = torch.empty((q, GT_K), dtype=torch.int32, device="cuda")
    _ground_truth(base, queries[:q], GT_K, gt)
    return base, gt, queries[q:].clone()


def _ids(*shape, pinned=False):
    if pinned:
        return torch.full(shape, -1, dtype=torch.int32).pin_memory()
    return torch.full(shape, -1, dtype=torch.int32, device="cuda")


def prepare(case, seed):
    kind, d = case["kind"], case["d"]
    s = dict(case)
    if kind == "gt":
        s["base"], _, s["queries"] = datagen.make_dataset_cuda(
            case["n"], d, case["q"], seed=seed, cosine=case["cosine"], centers=case["centers"],
            with_gt=False)
        s["h"] = pg.Handle(0)
        s["out"] = _ids(case["q"], case["k"])
        return s
    degree = case["degree"]
    s["params"] = pg.default_params(degree, case["beam"], screen=SCREENS[case["screen"]])
    if kind == "batched":
        sizes = _sizes(case)
        parts = [_data(case, n, n, seed * 1000 + i) for i, n in enumerate(sizes)]
        s["base"] = torch.cat([p[0] for p in parts])
        s["gt"] = torch.cat([p[1] for p in parts])
        off = [0]
        for n in sizes:
            off.append(off[-1] + n)
        s["off"] = off
        s["params"].flags |= pg.FLAG_CUDA_GRAPH
        s["stream"] = torch.cuda.Stream()
        s["h"] = pg.Handle(0, stream=s["stream"])
        s["graph"], s["proj"] = _ids(off[-1], degree), _ids(off[-1], PROJ)
        torch.cuda.synchronize()
        return s
    n, q = case["n"], case["q"]
    s["base"], s["gt"], held_out = _data(case, n, q, seed, case.get("nq", 0))
    s["h"] = pg.Handle(0)
    if kind == "host":
        s["base"], s["gt"] = s["base"].cpu().pin_memory(), s["gt"].cpu().pin_memory()
        s["graph"], s["proj"] = _ids(n, degree, pinned=True), _ids(n, PROJ, pinned=True)
        return s
    s["graph"], s["proj"] = _ids(n, degree), _ids(n, PROJ)
    if kind == "query":
        s["h"].build_device(s["base"], s["gt"], s["graph"], s["proj"], s["params"])
        s["queries"] = held_out
        s["out"] = _ids(case["nq"], case["topk"])
    elif kind == "index":
        s["out"], s["cnt"] = _ids(n, 2 * M_NN + M_FINAL), _ids(n)
    elif kind == "stages":
        reverse = GT_K - 2 - degree
        s["cand"], s["found"] = _ids(n, GT_K), _ids(n, case["beam"])
        s["pruned"], s["pruned_num"] = _ids(n, degree), _ids(n)
        s["reverse"], s["reverse_num"] = _ids(n, reverse), _ids(n)
        s["pruned1"], s["reverse1"] = _ids(n, 15), _ids(n, 111)
        s["pruned1_num"], s["reverse1_num"] = _ids(n), _ids(n)
    return s


def _run_stages(s):
    """The reference driver's launches of the projection and one link round."""
    h, base = s["h"], s["base"]
    h.match_top1(s["gt"], s["n"], s["cand"])
    e = [h.prune_reverse(base, s["cand"], s["pruned1"], s["pruned1_num"], s["reverse1"],
                         s["reverse1_num"], False)]
    e.append(h.merge_prune(base, s["pruned1"], s["pruned1_num"], s["reverse1"], s["reverse1_num"],
                           s["proj"], False))
    e.extend(h.search(base, s["proj"], s["found"], km=s["beam"] - 32))
    e.append(h.prune_reverse(base, s["found"], s["pruned"], s["pruned_num"], s["reverse"],
                             s["reverse_num"], True))
    e.append(h.merge_prune(base, s["pruned"], s["pruned_num"], s["reverse"], s["reverse_num"],
                           s["graph"], True))
    return [s[k] for k in ("cand", "pruned1", "pruned1_num", "reverse1", "reverse1_num", "proj",
                           "found", "pruned", "pruned_num", "reverse", "reverse_num", "graph")] + e


def run(state):
    s, kind = state, state["kind"]
    h = s["h"]
    if kind == "gt":
        h.ground_truth(s["base"], s["queries"], s["out"])
        return s["out"]
    if kind == "query":
        evals, iters = h.query_search(s["base"], s["graph"], s["queries"], s["out"],
                                      km=s["beam"] - 32)
        return s["out"], evals, iters
    if kind == "stages":
        return _run_stages(s)
    if kind == "index":
        st = h.build_index(s["base"], s["gt"], s["out"], s["cnt"], s["params"], MATCH_ROUNDS, M_NN,
                           M_FINAL)
        return s["out"], s["cnt"], st.evals_total
    if kind == "batched":
        st = h.build_batched(s["base"], s["gt"], s["off"], s["off"], s["graph"], s["proj"],
                             s["params"])
    elif kind == "host":
        st = h.build_host_ptr(s["base"].data_ptr(), s["n"], s["d"], s["gt"].data_ptr(), s["q"],
                              s["graph"].data_ptr(), s["proj"].data_ptr(), s["params"])
    else:
        st = h.build_device(s["base"], s["gt"], s["graph"], s["proj"], s["params"])
    return s["graph"], s["proj"], st.evals_total


# Distance evaluations per point of a build (both link rounds) and per external query on the
# generator's data, by beam width: the counts that the algorithm itself makes, rounded.
EVALS_POINT = {64: 570, 96: 1800, 128: 2500}
EVALS_QUERY = {64: 250, 96: 500, 128: 700}


def work(case):
    """Inputs read once, outputs written once; 2 d operations per distance evaluation."""
    kind, d = case["kind"], case["d"]
    if kind == "gt":
        n, q, k = case["n"], case["q"], case["k"]
        return {"bytes": 4 * (n * d + q * d + q * k), "flops": 2 * n * q * d}
    if kind == "query":
        nq = case["nq"]
        evals = nq * EVALS_QUERY[case["beam"]]
        rows = min(case["n"], evals)  # base rows and graph rows that the queries reach
        return {"bytes": 4 * (nq * (d + case["topk"]) + rows * (d + 16)), "flops": 2 * d * evals}
    if kind == "batched":
        n = q = sum(_sizes(case))
    else:
        n, q = case["n"], case["q"]
    out = n * (case["degree"] + PROJ)
    evals = n * EVALS_POINT[case["beam"]]
    if kind == "index":
        out = n * (2 * M_NN + M_FINAL + 1)
    elif kind == "stages":
        out = n * (GT_K + 15 + 111 + PROJ + case["beam"] + GT_K - 2 + case["degree"] + 4)
        evals //= 2
    return {"bytes": 4 * (n * d + q * GT_K + out), "flops": 2 * d * evals}


def exact(case, seed):
    """Every output is an id, a count of ids or a count of evaluations: there is no computed
    number to compare."""
    return None
