"""The calls this framework answers in earnest, as cases to time and compare.

A case is one call of a public entry point on an index (or the construction of
the sampling probabilities an index is built from). Four kinds:

  scan           an exact or flat index, or a precision strategy of one:
                 query_batch (host queries), query_device_batch, or query_many
                 in consecutive batches
  hierarchy      a sampled and projected index: query_device_batch
  batch          hierarchies of uneven sizes answered by one QueryBatch run
  probabilities  importance probabilities of a matrix on the device

Sizes follow the configurations of bench.py and the tests: d = 60,660 columns,
33 class centroids, 7,028 or 65,536 rows, T = 8 to 128 repetitions, p = 16 to
256 projected coordinates, batches of 1 to 4,096 queries. Values follow
ultrahigh_ann_b200/synthetic.py: log2(1 + Gamma(0.5, 200)) class centroids, 40%
of the columns zero in every row, rows and queries their centroid plus
N(0, 0.8^2) noise, clipped at 0. Rows of flat and hierarchical indexes are held
in BF16 where bench.py holds them so (65,536 rows).

The direct strategy reports a certified binary32 distance (widened to binary64
by the API), so its distances are returned as binary32; the precision
strategies and the probabilities compute in binary64 and are returned so.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import ultrahigh_ann_b200 as uha

SIGMA = 0.8
CLASSES = 33
# the law's probabilities are taken from this many rows of the matrix
PROBABILITY_ROWS = 256


# ------------------------------------------------------------------- cases

def listed():
    return [
        # The smallest call: one host query against 33 class centroids.
        dict(name="flat_l2_centroids_host1", kind="scan", index="flat", metric="l2", rows=33,
             d=60660, T=8, storage="float32", count=1, batch=1, host=True, strategy="direct"),
        # A service loop answering device-resident queries one at a time.
        dict(name="flat_l2_r7028_one_by_one", kind="scan", index="flat", metric="l2", rows=7028,
             d=60660, T=32, storage="float32", count=512, batch=1, host=False,
             strategy="direct"),
        # A full serving batch on the largest flat index.
        dict(name="flat_l1_r65536_b256", kind="scan", index="flat", metric="l1", rows=65536,
             d=60660, T=32, storage="bfloat16", count=256, batch=256, host=False,
             strategy="direct"),
        # One exact query over all columns: the headline call.
        dict(name="exact_l2_r7028_b1", kind="scan", index="exact", metric="l2", rows=7028,
             d=60660, T=0, storage="float32", count=1, batch=1, host=False, strategy="direct"),
        # Host queries in batches of 64, as a program holding numpy arrays calls it.
        dict(name="exact_l2_r7028_host64", kind="scan", index="exact", metric="l2", rows=7028,
             d=60660, T=0, storage="float32", count=64, batch=64, host=True,
             strategy="direct"),
        # The largest exact batch.
        dict(name="exact_l2_r7028_b1024", kind="scan", index="exact", metric="l2", rows=7028,
             d=60660, T=0, storage="float32", count=1024, batch=1024, host=False,
             strategy="direct"),
        # Exact L1 of a ragged batch.
        dict(name="exact_l1_r7028_b333", kind="scan", index="exact", metric="l1", rows=7028,
             d=60660, T=0, storage="float32", count=333, batch=333, host=False,
             strategy="direct"),
        # Bulk labelling with the tensor-core strategy in calls of two batches.
        dict(name="exact_l2_bf16_rerank_b1024", kind="scan", index="exact", metric="l2",
             rows=7028, d=60660, T=0, storage="float32", count=2048, batch=1024, host=False,
             strategy="gemm_bf16_rerank", candidates=8),
        # The hierarchies at the largest row count.
        dict(name="hier_l2_r65536_p64_b4096", kind="hierarchy", metric="l2", rows=65536,
             d=60660, T=32, p=64, storage="bfloat16", count=4096),
        dict(name="hier_l1_r65536_p64_b4096", kind="hierarchy", metric="l1", rows=65536,
             d=60660, T=32, p=64, storage="bfloat16", count=4096),
        # Hierarchies of uneven rows and p, both metrics, in one captured launch.
        dict(name="hier_batch_6", kind="batch", rows=16384, d=60660, T=32, p_small=16,
             p_large=256, storage="bfloat16", count=1000, indexes=6),
        # Sampling probabilities of a labelled training set.
        dict(name="probabilities_l2_r384", kind="probabilities", metric="l2", rows=384,
             d=60660),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["exact", "exact", "flat", "flat", "precision", "hierarchy", "hierarchy",
                       "batch", "probabilities"])
    metric = rng.choice(["l2", "l1"])
    if kind == "exact":
        rows = _log_int(rng, 500, 8192)
        d = rng.randrange(4099, 60661)
        # no more than 1,024 queries over 7,028 x 60,660 values (L1: half of it)
        most = min(1024, int((4.2e11 if metric == "l2" else 2.1e11) / (rows * d)))
        count = _log_int(rng, 1, most)
        return dict(kind="scan", index="exact", metric=metric, rows=rows, d=d, T=0,
                    storage="float32", count=count, batch=count, host=rng.random() < 0.25,
                    strategy="direct")
    if kind == "flat":
        rows = _log_int(rng, 33, 65536)
        T = _log_int(rng, 8, 128)
        batch = _log_int(rng, 1, 512)
        host = rng.random() < 0.25
        count = batch if host or batch > 8 else batch * rng.randrange(1, 65)
        return dict(kind="scan", index="flat", metric=metric, rows=rows,
                    d=rng.randrange(20011, 60661), T=T,
                    storage="bfloat16" if rows > 16384 else "float32", count=count, batch=batch,
                    host=host, strategy="direct")
    if kind == "precision":
        batch = _log_int(rng, 1, 1024)
        return dict(kind="scan", index=rng.choice(["exact", "flat"]), metric="l2",
                    rows=_log_int(rng, 1000, 8192), d=rng.randrange(20011, 60661),
                    T=rng.choice([32, 128]), storage="float32",
                    count=batch * rng.randrange(1, 3), batch=batch, host=False,
                    strategy=rng.choice(["gemm_bf16_rerank", "gemm_fp8_rerank"]),
                    candidates=rng.choice([8, 32]))
    if kind == "hierarchy":
        rows = _log_int(rng, 1024, 65536)
        p = _log_int(rng, 16, 256)
        # no more than 4,096 queries over 65,536 x 64 values
        most = min(4096, int(4096.0 * 65536 * 64 / (rows * p)))
        return dict(kind="hierarchy", metric=metric, rows=rows, d=rng.randrange(20011, 60661),
                    T=rng.choice([16, 32, 64]), p=p, storage=rng.choice(["float32", "bfloat16"]),
                    count=_log_int(rng, 16, most))
    if kind == "batch":
        return dict(kind="batch", rows=_log_int(rng, 2048, 16384), d=rng.randrange(20011, 60661),
                    T=32, p_small=rng.randrange(16, 65), p_large=rng.randrange(65, 257),
                    storage="bfloat16", count=_log_int(rng, 64, 1000),
                    indexes=rng.randrange(2, 7))
    return dict(kind="probabilities", metric=metric, rows=_log_int(rng, 33, 384),
                d=rng.randrange(4099, 60661))


# ------------------------------------------------------------------ inputs

class _State:
    pass


def _values(case, seed, rows, count):
    """(rows, queries) on the device."""
    d = case["d"]
    device = torch.device("cuda", 0)
    host = np.random.default_rng([seed, rows, d])
    centroids = np.log2(1.0 + host.gamma(0.5, 200.0, size=(CLASSES, d)))
    keep = host.random(d) >= 0.4
    centroids[:, ~keep] = 0.0
    centroids = torch.from_numpy(centroids.astype(np.float32)).to(device)
    keep = torch.from_numpy(keep).to(device)
    gen = torch.Generator(device=device)
    gen.manual_seed(seed)
    storage = torch.bfloat16 if case.get("storage") == "bfloat16" else torch.float32

    def noisy(labels, dtype, masked):
        out = torch.empty((labels.size, d), dtype=dtype, device=device)
        labels = torch.from_numpy(labels).to(device)
        for s in range(0, out.shape[0], 1024):
            lab = labels[s:s + 1024]
            block = torch.randn((lab.shape[0], d), generator=gen, device=device)
            block.mul_(SIGMA).add_(centroids[lab]).clamp_(min=0.0)
            if masked:
                block.mul_(keep)
            # queries take the values of the rows' storage type
            out[s:s + 1024] = block.to(storage)
        return out

    if rows == CLASSES:
        matrix = centroids.to(storage)
    else:
        matrix = noisy(host.integers(0, CLASSES, rows), storage, True)
    queries = noisy(host.integers(0, CLASSES, count), torch.float32, False) if count else None
    # the engine reads them on streams of its own
    torch.cuda.synchronize()
    return matrix, queries


def _probabilities(matrix, metric):
    few = matrix[:PROBABILITY_ROWS].float().contiguous()
    torch.cuda.synchronize()
    compute = (uha.compute_l2_importance_probabilities_gpu if metric == "l2"
               else uha.compute_l1_importance_probabilities_gpu)
    return compute(few).probabilities


def _hierarchy(matrix, probabilities, metric, T, p, engine):
    cls = (uha.CudaHierarchicalL2AnnIndex if metric == "l2" else uha.CudaHierarchicalL1AnnIndex)
    return cls(matrix, T, p, engine, importance_probabilities=probabilities)


def _batch_members(case):
    """(metric, rows, p, queries) of each index of a batch case."""
    out = []
    for i in range(case["indexes"]):
        out.append(("l2" if i % 2 == 0 else "l1", max(1024, case["rows"] >> (i // 2)),
                    (case["p_large"], case["p_small"])[(i // 2) % 2],
                    max(1, case["count"] - 7 * i)))
    return out


def prepare(case, seed):
    s = _State()
    s.case = case
    kind = case["kind"]
    if kind == "probabilities":
        s.matrix, _ = _values(case, seed, case["rows"], 0)
    elif kind == "batch":
        members = _batch_members(case)
        matrix, queries = _values(case, seed, case["rows"], max(m[3] for m in members))
        probabilities = {m: _probabilities(matrix, m) for m in ("l2", "l1")}
        engine = uha.MT19937_64(seed)
        s.indexes = [_hierarchy(matrix[:rows], probabilities[metric], metric, case["T"], p,
                                engine) for metric, rows, p, _ in members]
        s.batch = uha.QueryBatch([(ix, m[3]) for ix, m in zip(s.indexes, members)])
        s.queries = queries
        s.pointers = [queries.data_ptr()] * len(members)
    else:
        matrix, queries = _values(case, seed, case["rows"], case["count"])
        engine = uha.MT19937_64(seed)
        metric = case["metric"]
        if kind == "hierarchy":
            s.index = _hierarchy(matrix, _probabilities(matrix, metric), metric, case["T"],
                                 case["p"], engine)
        elif case["index"] == "exact":
            s.index = (uha.CudaExactL2Index if metric == "l2" else uha.CudaExactL1Index)(matrix)
        else:
            cls = (uha.CudaSampledCoordinateL2AnnIndex if metric == "l2"
                   else uha.CudaSampledCoordinateL1AnnIndex)
            s.index = cls(matrix, _probabilities(matrix, metric), case["T"], engine)
        s.workspace = s.index.make_query_workspace(case.get("batch", case["count"]))
        if case.get("candidates"):
            s.workspace.set_candidates(case["candidates"])
        s.strategy = uha.QueryStrategy[case.get("strategy", "direct")]
        s.queries = queries.cpu().numpy() if case.get("host") else queries
        s.rows = np.zeros(case["count"], np.uint64)
        s.distances = np.zeros(case["count"], np.float64)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------- calls

def run(s):
    case = s.case
    if case["kind"] == "probabilities":
        compute = (uha.compute_l2_importance_probabilities_gpu if case["metric"] == "l2"
                   else uha.compute_l1_importance_probabilities_gpu)
        return {"probabilities": compute(s.matrix).probabilities}
    if case["kind"] == "batch":
        answers = s.batch.run(s.pointers, on_device=True)
        return [{"rows": r, "distances": d.astype(np.float32)} for r, d in answers]
    count = case["count"]
    if case.get("host"):
        s.index.query_batch(s.queries, count, s.rows, s.workspace, s.strategy, s.distances)
    elif case.get("batch", count) == count:
        s.index.query_device_batch(s.queries.data_ptr(), count, s.rows, s.workspace, s.strategy,
                                   s.distances)
    else:
        s.index.query_many(s.queries.data_ptr(), count, case["batch"], s.rows, s.workspace,
                           s.strategy, s.distances, on_device=True)
    direct = s.strategy == uha.QueryStrategy.direct
    return {"rows": s.rows,
            "distances": s.distances.astype(np.float32) if direct else s.distances}


# -------------------------------------------------------------------- work

def _sample_size(case):
    """About the sampled columns of a flat or hierarchical index: T repetitions
    of probabilities that sum to about 11.5 (L2) or 4 (L1) for 256 rows, most
    columns sampled once."""
    return min(0.6 * case["d"], case["T"] * (11.5 if case["metric"] == "l2" else 4.0))


def _hier_work(metric, rows, p, count, d, T):
    k = _sample_size(dict(metric=metric, d=d, T=T))
    return (count * k * 4 + rows * p * 4 + p * k * 4 + count * 16,
            2 * count * k * p + 3 * count * rows * p)


def work(case):
    kind = case["kind"]
    if kind == "probabilities":
        pairs = case["rows"] * (case["rows"] - 1) / 2
        # the distance of each pair, then each column's largest ratio
        return {"bytes": case["rows"] * case["d"] * 4 + case["d"] * 8,
                "flops": pairs * case["d"] * 6}
    if kind == "batch":
        both = [_hier_work(m, r, p, n, case["d"], case["T"]) for m, r, p, n in
                _batch_members(case)]
        return {"bytes": sum(b for b, _ in both), "flops": sum(f for _, f in both)}
    n = case["count"]
    if kind == "hierarchy":
        b, f = _hier_work(case["metric"], case["rows"], case["p"], n, case["d"], case["T"])
        return {"bytes": b, "flops": f}
    columns = case["d"] if case["index"] == "exact" else _sample_size(case)
    return {"bytes": (case["rows"] + n) * columns * 4 + n * 16,
            "flops": 3 * n * case["rows"] * columns}


# ------------------------------------------------------------------- exact

def _nearest_l2(rows, queries):
    """Index and squared distance of each query's nearest row, in 64 bits: the
    norm identity picks a few rows, whose distances are then summed directly."""
    rows = rows.double()
    norms = (rows * rows).sum(1)
    keep = min(4, rows.shape[0])
    index, distance = [], []
    for s in range(0, queries.shape[0], 256):
        q = queries[s:s + 256].double()
        near = (norms - 2.0 * (q @ rows.T)).topk(keep, 1, largest=False).indices.sort(1).values
        d = torch.stack([(rows[near[:, i]] - q).square().sum(1) for i in range(keep)], 1)
        best = d.min(1)
        # the first of equal distances has the lowest row
        first = (d == best.values[:, None]).int().argmax(1)
        index.append(near.gather(1, first[:, None])[:, 0])
        distance.append(best.values)
    return torch.cat(index), torch.cat(distance)


def _nearest_l1(rows, queries, weights):
    index, distance = [], []
    rows = rows.double()
    queries = queries.double()
    if weights is not None:
        rows = rows * weights
        queries = queries * weights
    for s in range(0, queries.shape[0], 64):
        d = torch.zeros((min(64, queries.shape[0] - s), rows.shape[0]), dtype=torch.float64,
                        device=rows.device)
        for c in range(0, rows.shape[1], 8192):
            d += torch.cdist(queries[s:s + 64, c:c + 8192].contiguous(),
                             rows[:, c:c + 8192].contiguous(), p=1.0)
        best = d.min(1)
        index.append((d == best.values[:, None]).int().argmax(1))
        distance.append(best.values)
    return torch.cat(index), torch.cat(distance)


def _nearest_median(rows, queries):
    """Index and median |difference| of each query's nearest row, in 64 bits.
    A row with fewer than p/2 binary32 differences below 1.001 times some row's
    median is not the nearest; the medians of the others are sorted out."""
    p = rows.shape[1]
    lower, upper = (p - 1) // 2, p // 2
    rows32 = rows.float()

    def medians(r, q):
        v = (r - q).abs().sort(-1).values
        return v[..., lower] + (v[..., upper] - v[..., lower]) * 0.5

    some = rows[:: max(1, rows.shape[0] // 512)]
    index, distance = [], []
    step = max(1, int(2e8 / (rows.shape[0] * p)))
    for s in range(0, queries.shape[0], step):
        q = queries[s:s + step]
        bound = medians(some, q[:, None, :]).min(1).values * 1.001
        near = (rows32 - q.float()[:, None, :]).abs() <= bound.float()[:, None, None]
        a, r = ((near.sum(2) >= (p + 1) // 2)).nonzero(as_tuple=True)
        m = medians(rows[r], q[a])
        best = torch.full((q.shape[0],), math.inf, dtype=torch.float64, device=rows.device)
        best.scatter_reduce_(0, a, m, "amin")
        row = torch.full((q.shape[0],), rows.shape[0], dtype=torch.int64, device=rows.device)
        hit = m == best[a]
        row.scatter_reduce_(0, a[hit], r[hit], "amin")
        index.append(row)
        distance.append(best)
    return torch.cat(index), torch.cat(distance)


def _answer(found):
    index, distance = found
    return {"rows": index.cpu().numpy().astype(np.uint64), "distances": distance.cpu().numpy()}


def _hierarchy_exact(index, matrix, queries, metric):
    columns = torch.from_numpy(index.coordinate_sample.source_columns.astype(np.int64)).cuda()
    # the drawn p x k projection is an input of the answer
    projection = torch.from_numpy(np.asarray(index.projection)).double().cuda()
    rows = matrix[:, columns].double() @ projection.T
    q = queries[:, columns].double() @ projection.T
    return _answer(_nearest_l2(rows, q) if metric == "l2" else _nearest_median(rows, q))


def exact(case, seed):
    kind = case["kind"]
    if kind == "probabilities":
        matrix, _ = _values(case, seed, case["rows"], 0)
        rows = matrix.double()
        most = torch.zeros(case["d"], dtype=torch.float64, device=rows.device)
        for a in range(case["rows"] - 1):
            diff = (rows[a + 1:] - rows[a]).abs()
            if case["metric"] == "l2":
                diff = diff.square()
            total = diff.sum(1, keepdim=True)
            diff = torch.where(total > 0, diff / total, torch.zeros_like(diff))
            most = torch.maximum(most, diff.max(0).values)
        return {"probabilities": most.cpu().numpy()}
    s = prepare(case, seed)
    if kind == "batch":
        members = _batch_members(case)
        matrix, queries = _values(case, seed, case["rows"], max(m[3] for m in members))
        return [_hierarchy_exact(ix, matrix[:m[1]], queries[:m[3]], m[0])
                for ix, m in zip(s.indexes, members)]
    matrix, queries = _values(case, seed, case["rows"], case["count"])
    metric = case["metric"]
    if kind == "hierarchy":
        return _hierarchy_exact(s.index, matrix, queries, metric)
    weights = None
    if case["index"] == "flat":
        sample = s.index.coordinate_sample
        columns = torch.from_numpy(sample.source_columns.astype(np.int64)).cuda()
        matrix, queries = matrix[:, columns].float(), queries[:, columns]
        scale = torch.from_numpy(sample.multiplicities * sample.inverse_probabilities).cuda()
        if metric == "l2":
            # the embedded values of a flat L2 index are binary32 products
            scale = scale.sqrt().float()
            matrix, queries = matrix * scale, queries * scale
        else:
            weights = scale
    return _answer(_nearest_l2(matrix, queries) if metric == "l2"
                   else _nearest_l1(matrix, queries, weights))
