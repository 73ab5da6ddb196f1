"""The work a user of this library has it do, as a list of measured cases.

A case is a plain dict.  Its "kind" says which public entry point it goes through:

  layer     one aggregation of a graph layer, AggregationPlan.spmm: forward (A^T . X) or backward (A . X), with the
            stored coefficients or in the value-free form with a row scale, with or without the ReLU in the store
  gcn       forward and backward of a whole graph-convolution model, gcn.GCN
  pagerank  power iterations with a fixed count, or the delta job run to its end over the parts of an EBV partition
  cc, sssp  one run of the minimum-propagation jobs from their start values to the fixed point

Graphs are seeded and synthetic, in the two shapes the repository's benchmark uses: R-MAT with 2^scale vertices, and
power-law graphs with a given number of vertices and drawn pairs (both from graphgen).
"""
import ctypes as C
import math
import types

import numpy as np
import torch

import drone_b200 as db
from drone_b200 import gcn, graphgen as gg, graphsum as gs, minprop as mpj, pagerank as prk, partition as pt
from drone_b200._lib import check, lib

ITERATIONS, DAMPING = 20, 0.85    # the fixed-iteration PageRank configuration
JOB_EPS = 1e-6                    # push threshold of the delta job, as the reference's GPU job sets it


def listed():
    layer = dict(kind="layer", graph="rmat", edge_factor=16, symmetrise=False, op="AT", form="plain", relu=False)
    return [
        # the size of a citation graph and of the test graphs: a few microseconds of work, so launches count
        dict(layer, name="layer_rmat12_f16", scale=12, symmetrise=True, features=16),
        # the single-GPU headline configuration, forward
        dict(layer, name="layer_rmat20_f64", scale=20, symmetrise=True, features=64),
        # forward of a hidden layer in the value-free form: unit coefficients, row factor and ReLU in the store
        dict(layer, name="layer_rmat22_f32_value_free_relu", scale=22, features=32, form="value_free", relu=True),
        # the large-scale propagation configuration, at the largest size whose graph is made in about a second
        dict(layer, name="layer_rmat24_f32", scale=24, features=32),
        # backward of a wide hidden layer on the products-shaped graph (operands of 2.5 GB, mean degree 52)
        dict(kind="layer", graph="powerlaw", name="layer_products_f256_backward", vertices=2449029, pairs=61900000,
             features=256, op="A", form="plain", relu=False),
        # first aggregation of a backward pass on the Reddit-shaped graph: as wide as the classes, rows of 164 bytes
        dict(kind="layer", graph="powerlaw", name="layer_reddit_f41_backward", vertices=232965, pairs=57200000,
             features=41, op="A", form="plain", relu=False),
        # one training step of the two-layer model on the Reddit-shaped graph
        dict(kind="gcn", name="gcn_reddit_602_128_41", vertices=232965, pairs=57200000, dims="602-128-41"),
        # the propagation at feature width 1, one part
        dict(kind="pagerank", name="pagerank_rmat22_float", scale=22, parts=1, double=False, schedule="power"),
        # the small PageRank configuration: two EBV parts, 20 iterations, double
        dict(kind="pagerank", name="pagerank_rmat16_2parts_double", scale=16, parts=2, double=True, schedule="power"),
        # the job as a master drives it, superstep by superstep until no part has anything to send
        dict(kind="pagerank", name="pagerank_job_rmat16_4parts", scale=16, parts=4, double=True, schedule="delta"),
        # labels of the connected components of an undirected graph
        dict(kind="cc", name="cc_rmat20", scale=20, symmetrise=True, lengths=False),
        # distances with unit lengths, which is what the reference's graph builder stores
        dict(kind="sssp", name="sssp_rmat22", scale=22, symmetrise=False, lengths=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["layer"] * 6 + ["gcn"] + ["pagerank"] * 3 + ["cc", "sssp"])
    if kind == "layer":
        case = dict(kind="layer", op=rng.choice(["AT", "A"]))
        if rng.random() < 0.5:
            case.update(graph="rmat", scale=rng.randint(12, 24), edge_factor=_log_int(rng, 4, 32),
                        symmetrise=rng.random() < 0.5)
            edges = (case["edge_factor"] << case["scale"]) * (2 if case["symmetrise"] else 1)
            while edges > 16 << 24:      # as many stored entries as the largest listed graph at most
                case["scale"] -= 1
                edges //= 2
            n = 1 << case["scale"]
        else:
            n = _log_int(rng, 3000, 2449029)
            pairs = min(int(n * math.exp(rng.uniform(math.log(2), math.log(245)))), 61900000)
            case.update(graph="powerlaw", vertices=n, pairs=pairs)
            edges = 2 * pairs
        most = max(1, min(512, (61900000 * 2 * 256) // (edges + n), (2449029 * 256 * 4) // n))
        features = _log_int(rng, 1, most)
        if rng.random() < 0.5:           # hidden widths are multiples of 8, class counts are any number
            features = max(8, features // 8 * 8)
        case.update(features=features, form=rng.choice(["plain", "plain", "value_free"]), relu=rng.random() < 0.3)
        return case
    if kind == "gcn":
        n = _log_int(rng, 3000, 232965)
        dims = [_log_int(rng, 32, 602), _log_int(rng, 16, 128) // 8 * 8, rng.randint(5, 47)]
        return dict(kind="gcn", vertices=n, pairs=int(n * math.exp(rng.uniform(math.log(2), math.log(245)))),
                    dims="-".join(str(d) for d in dims))
    if kind == "pagerank":
        if rng.random() < 1 / 3:
            return dict(kind=kind, scale=rng.randint(16, 22), parts=1, double=rng.random() < 0.5, schedule="power")
        if rng.random() < 0.5:
            return dict(kind=kind, scale=rng.randint(12, 18), parts=rng.randint(2, 8), double=rng.random() < 0.5,
                        schedule="power")
        return dict(kind=kind, scale=rng.randint(12, 16), parts=rng.randint(2, 4), double=True, schedule="delta")
    return dict(kind=kind, scale=rng.randint(14, 22 if kind == "sssp" else 20), symmetrise=kind == "cc",
                lengths=kind == "sssp" and rng.random() < 0.5)


# ----- inputs -----

def _device():
    return torch.device("cuda", torch.cuda.current_device())


def _generator(seed):
    gen = torch.Generator(device=_device())
    gen.manual_seed(seed)
    return gen


def _edges(case, seed, self_loops):
    """(n, u, v) on the GPU: sorted by source, no duplicates; "add" gives every vertex its self-loop."""
    if case.get("graph") == "powerlaw" or "pairs" in case:
        return gg.powerlaw_graph(case["vertices"], case["pairs"], seed=seed, device=_device(), self_loops=self_loops)
    return gg.rmat_graph(case["scale"], case.get("edge_factor", 16), seed=seed, device=_device(),
                         symmetrise=case.get("symmetrise", False), self_loops=self_loops)


def _array(owner, pointer, n, typestr):
    """A tensor over n values of device memory that belongs to the handle `owner`, which lives as long as the tensor."""
    return torch.as_tensor(types.SimpleNamespace(owner=owner, __cuda_array_interface__={
        "shape": (n,), "typestr": typestr, "data": (pointer, False), "version": 2}), device=_device())


def _one_part(n, index, dst, out_degree=None):
    """A whole graph as the only part, in the shape graphsum.DeviceGraph has."""
    host = types.SimpleNamespace(rank=0, n_parts=1, n_local=n, l2g=np.arange(n, dtype=np.int32),
                                 mirror2worker=np.full(n, -1, np.int32), master_worker_index=np.zeros(n + 1, np.int32),
                                 master2workers=np.zeros(0, np.int32))
    return types.SimpleNamespace(host=host, n_local=n, device=_device(), index=index, dst=dst, out_degree=out_degree,
                                 mirror2worker=torch.full((n,), -1, dtype=torch.int32, device=_device()),
                                 xplan=pt.ExchangePlan(host, 1))


def _prepare_layer(case, seed):
    n, u, v = _edges(case, seed, "add")
    index, dst = gg.csr_by_source(u, v, n)
    in_degree, out_degree = gg.degrees(u, v, n)
    del u, v
    plan = db.AggregationPlan(index, dst, in_degree=in_degree, out_degree=out_degree)
    f = case["features"]
    x = torch.randn((n, f), device=_device(), generator=_generator(seed))
    options = {"relu": True} if case["relu"] else {}
    op = db.OP_AT if case["op"] == "AT" else db.OP_A
    if case["form"] == "value_free":     # the factor of the gathered side sits in X, the other one is the row scale
        in_scale, out_scale = db.degree_scales(in_degree, out_degree)
        row, column = (in_scale, out_scale) if op == db.OP_AT else (out_scale, in_scale)
        x *= column[:, None]
        options.update(unit_values=True, row_scale=row)
    return {"plan": plan, "op": op, "x": x, "out": torch.empty((n, f), device=_device()), "options": options}


def _prepare_gcn(case, seed):
    n, u, v = _edges(case, seed, "add")
    index, dst = gg.csr_by_source(u, v, n)
    in_degree, out_degree = gg.degrees(u, v, n)
    del u, v
    dims = [int(d) for d in case["dims"].split("-")]
    plan = db.AggregationPlan(index, dst, in_degree=in_degree, out_degree=out_degree)
    plan.reserve(max(dims[1:]), padded_rows=True)
    graph = types.SimpleNamespace(plan=plan, mirror2worker=None)
    gen = _generator(seed)
    x = torch.randn((n, dims[0]), device=_device(), generator=gen)
    truth = torch.randint(0, dims[-1], (n,), device=_device(), generator=gen, dtype=torch.int32)
    truth[torch.rand(n, device=_device(), generator=gen) < 0.34] = -1        # vertices of the other splits
    return {"model": gcn.GCN(graph, x, truth, gg.glorot_weights(dims, _device(), seed=seed))}


def _prepare_pagerank(case, seed):
    n, u, v = _edges(case, seed, "drop")
    parts = case["parts"]
    eps = JOB_EPS if case["schedule"] == "delta" else 0.0
    if parts == 1:
        index, dst = gg.csr_by_source(u, v, n)
        _, out_degree = gg.degrees(u, v, n)
        graphs, isolated = [_one_part(n, index, dst, out_degree)], 0
    else:
        in_degree, out_degree = (d.cpu().numpy() for d in gg.degrees(u, v, n))
        part = pt.ebv_partition(n, u.cpu().numpy(), v.cpu().numpy(), parts, keep_self_loops=False)
        graphs = [gs.DeviceGraph(part.local_graph(p), in_degree, out_degree, _device(), max_features=1)
                  for p in range(parts)]
        isolated = int((part.replicas == 0).sum())
    jobs = [prk.PageRank(g, n, use_double=case["double"], eps=eps, n_isolated=isolated) for g in graphs]
    values, own, ids = [], [], []
    for job, g in zip(jobs, graphs):
        p = C.c_void_p(0)
        check(lib().drone_pr_device_arrays(job.handle, C.byref(p), None, None, None, None))
        values.append(_array(job, p.value, job.n_local, "<f8" if case["double"] else "<f4"))
        if parts > 1:
            own.append(torch.nonzero(g.mirror2worker < 0)[:, 0])      # masters and unreplicated vertices
            ids.append(torch.as_tensor(g.host.l2g, device=_device()).long()[own[-1]])
    ranks = torch.zeros(n, dtype=values[0].dtype, device=_device()) if parts > 1 else None
    return {"jobs": jobs, "values": values, "own": own, "ids": ids, "ranks": ranks, "schedule": case["schedule"]}


def _prepare_minprop(case, seed):
    n, u, v = _edges(case, seed, "drop")
    index, dst = gg.csr_by_source(u, v, n)
    _, out_degree = gg.degrees(u, v, n)
    source = int(torch.argmax(out_degree)) if case["kind"] == "sssp" else -1
    lengths = None
    if case["lengths"]:
        lengths = torch.rand(dst.numel(), device=_device(), generator=_generator(seed)) * 0.99 + 0.01
    graph = _one_part(n, index, dst)
    job = mpj.MinProp(graph, mpj.SSSP if case["kind"] == "sssp" else mpj.CC, edge_len=lengths)
    p = C.c_void_p(0)
    check(lib().drone_mp_device_arrays(job.handle, C.byref(p), None, None))
    return {"job": job, "source": source, "values": _array(job, p.value, n, "<f4" if case["kind"] == "sssp" else "<i4")}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "layer":
        state = _prepare_layer(case, seed)
    elif kind == "gcn":
        state = _prepare_gcn(case, seed)
    elif kind == "pagerank":
        state = _prepare_pagerank(case, seed)
    else:
        state = _prepare_minprop(case, seed)
    state["kind"] = kind
    return state


def run(state):
    kind = state["kind"]
    if kind == "layer":
        return state["plan"].spmm(state["op"], state["x"], out=state["out"], **state["options"])
    if kind == "gcn":
        model = state["model"]
        loss = model.forward()
        gradients = model.backward()
        return {"loss": loss, "gradients": list(gradients), "hidden": model.z[:-1], "logits": model.z[-1]}
    if kind == "pagerank":
        sent = {}
        if state["schedule"] == "delta":
            steps, sizes = prk.run_job_local(state["jobs"])
            sent = {"steps": steps, "sizes": np.sum(np.array(sizes, np.int64), axis=0)}
        elif len(state["jobs"]) == 1:
            state["jobs"][0].power_iterate(ITERATIONS, DAMPING)
            return state["values"][0]
        else:
            prk.power_iterate_local(state["jobs"], ITERATIONS, DAMPING)
        for values, own, ids in zip(state["values"], state["own"], state["ids"]):    # ranks by global id
            state["ranks"].index_copy_(0, ids, values.index_select(0, own))
        return {"ranks": state["ranks"], **sent}
    response = state["job"].peval(state["source"])
    return {"values": state["values"], "visited": int(response.VisitedSize)}


# ----- what a pass cannot do without -----

def _rmat_entries(scale, drawn, symmetrise):
    """Expected number of distinct directed edges, without self-loops, among `drawn` R-MAT edges (probabilities a, b, c
    with b = c): every cell of the adjacency matrix has the probability a^i b^j d^l with i + j + l = scale, and
    scale! / (i! j! l!) 2^j cells share it."""
    a, b, _ = gg.RMAT_ABC
    d = 1 - a - 2 * b
    total = 0.0
    for j in range(1, scale + 1):        # j = 0 is the diagonal
        for i in range(scale - j + 1):
            p = a ** i * b ** j * d ** (scale - j - i)
            cells = math.comb(scale, j) * math.comb(scale - j, i) * 2.0 ** j
            total -= cells * math.expm1(drawn * math.log1p(-p * (2 if symmetrise else 1)))
    return total


def _powerlaw_entries(n, pairs, exponent=0.4, offset=100.0):
    """The same for graphgen.powerlaw_graph (both directions of every distinct pair): its vertices in groups of nearly
    equal weight."""
    edges = np.unique(np.round(np.geomspace(offset, n + offset, 400) - offset).astype(np.int64))
    size = np.diff(edges).astype(np.float64)
    w = (0.5 * (edges[:-1] + edges[1:] - 1) + offset) ** -exponent
    p = w / (size * w).sum()
    return float((size[:, None] * size[None, :] * -np.expm1(-2.0 * pairs * p[:, None] * p[None, :])).sum())


def _shape(case):
    """(vertices, stored entries without self-loops)"""
    if "pairs" in case:
        return case["vertices"], _powerlaw_entries(case["vertices"], case["pairs"])
    n = 1 << case["scale"]
    return n, _rmat_entries(case["scale"], case.get("edge_factor", 16) * n, case.get("symmetrise", False))


def work(case):
    n, entries = _shape(case)
    kind = case["kind"]
    if kind == "layer":
        nnz, f = entries + n, case["features"]
        coefficients = 4 * nnz if case["form"] == "plain" else 4 * n
        return {"bytes": 4 * nnz + coefficients + 4 * (n + 1) + 8 * n * f, "flops": 2 * nnz * f}
    if kind == "gcn":
        nnz = entries + n
        d = [int(x) for x in case["dims"].split("-")]
        layers = len(d) - 1
        stored = 2 * (8 * nnz + 4 * (n + 1))                          # both orientations, each read once
        outputs = 4 * n * sum(d[1:]) + 4 * sum(d[i] * d[i + 1] for i in range(layers))
        dense = sum((2 if i == 0 else 3) * 2 * n * d[i] * d[i + 1] for i in range(layers))
        return {"bytes": 4 * n * d[0] + 4 * n + stored + outputs, "flops": dense + 4 * nnz * sum(d[1:])}
    if kind == "pagerank":
        # the job's vertices move by less than JOB_EPS after log(JOB_EPS) / log(damping) supersteps
        steps = ITERATIONS if case["schedule"] == "power" else int(math.log(JOB_EPS) / math.log(DAMPING))
        value = 8 if case["double"] else 4
        return {"bytes": steps * (4 * entries + 8 * n + 2 * value * n), "flops": steps * (entries + 4 * n)}
    # every edge offers its source's value at least once
    return {"bytes": (8 if case["lengths"] else 4) * entries + 12 * n, "flops": entries}


def tolerance(case):
    kind = case["kind"]
    if kind == "layer":
        return {"rel": 1e-5}                    # float sums of a row's terms in another order
    if kind == "gcn":
        return {"rel": 2e-5}                    # the same through two layers and the sums over all vertices of dW
    if kind == "pagerank":
        return {"rel": 1e-10} if case["double"] else {"rel": 1e-5}
    return "exact"                              # minima do not depend on the order
