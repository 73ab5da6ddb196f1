"""PageRank on the device against the oracles: DRONE's GPU-job schedule in double (1e-9) and float,
synchronous power iteration (the 20-iteration, damping 0.85 configuration), all parts on one GPU or
one process per GPU over NCCL."""
import ctypes as C
import os
import types

import numpy as np
import pytest
import torch

import drone_b200 as db
from drone_b200._lib import check
from helpers import run_ranks
from drone_b200 import graphgen as gg
from drone_b200 import graphsum as gs
from drone_b200 import pagerank as prk
from drone_b200 import partition as pt
from test_pagerank_oracle import pr_case

pytestmark = pytest.mark.gpu

PR_TOL = 1e-9   # relative, double mode against the double oracle running the same schedule


def build_parts(part, n, u, v, dev, use_double, eps):
    in_deg = np.bincount(v, minlength=n).astype(np.int32)
    out_deg = np.bincount(u, minlength=n).astype(np.int32)
    graphs = [gs.DeviceGraph(part.local_graph(p), in_deg, out_deg, dev, max_features=1) for p in range(part.n_parts)]
    n_iso = int((part.replicas == 0).sum())
    prs = [prk.PageRank(g, n, comm=None, use_double=use_double, eps=eps, n_isolated=n_iso) for g in graphs]
    return graphs, prs


@pytest.mark.parametrize("parts", [2, 4])
def test_delta_schedule_double_matches_oracle(cuda_device, oracle, parts):
    n, u, v, out_deg, part = pr_case(scale=10, seed=31, parts=parts)
    want, want_steps, want_sizes = oracle.pr_drone_cuda(n, part.part_u, part.part_v, out_deg, part.owner, eps=1e-6,
                                                        dtype=np.float64)
    graphs, prs = build_parts(part, n, u, v, cuda_device, True, 1e-6)
    steps, sizes = prk.run_job_local(prs)
    got = prk.gather_global(prs, graphs, n)
    assert steps == want_steps
    # per superstep, the four exchange counts summed over parts
    got_sizes = np.array([[sum(s[i] for s in step) for i in range(4)] for step in sizes])
    assert np.array_equal(got_sizes, want_sizes)
    touched = part.replicas > 0
    assert np.max(np.abs(got[touched] - want[touched]) / np.abs(want[touched])) < PR_TOL
    # every replica of a vertex holds the same value at the end
    seen = {}
    for pr_, g in zip(prs, graphs):
        vals = pr_.values()
        for loc in np.nonzero(part.replicas[g.host.l2g] > 1)[0][:200]:
            gid = int(g.host.l2g[loc])
            assert seen.setdefault(gid, vals[loc]) == vals[loc]


def test_delta_schedule_float_close_to_reference_semantics(cuda_device, oracle):
    n, u, v, out_deg, part = pr_case(scale=10, seed=32, parts=2)
    want, want_steps, _ = oracle.pr_drone_cuda(n, part.part_u, part.part_v, out_deg, part.owner, eps=1e-6,
                                               dtype=np.float32)
    graphs, prs = build_parts(part, n, u, v, cuda_device, False, 1e-6)
    steps, _ = prk.run_job_local(prs)
    got = prk.gather_global(prs, graphs, n)
    touched = part.replicas > 0
    # float sums in a different (fixed) order than the oracle's; thresholded pushes may flip near eps
    assert np.max(np.abs(got[touched] - want[touched]) / want[touched]) < 2e-4
    assert abs(steps - want_steps) <= max(3, want_steps // 5)


@pytest.mark.parametrize("parts", [1, 2, 8])
def test_power_iteration_rmat16_config(cuda_device, oracle, parts):
    """R-MAT scale 16, edge factor 16, self-loops and duplicates removed, damping 0.85, 20 iterations, 1/|V| start."""
    n, u, v = gg.rmat_graph(16, 16, seed=20261125, symmetrise=False, self_loops="drop")
    u, v = u.numpy(), v.numpy()
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    part = pt.ebv_partition(n, u, v, parts, keep_self_loops=False)
    graphs, prs = build_parts(part, n, u, v, cuda_device, True, 0.0)
    prk.power_iterate_local(prs, 20, 0.85)
    got = prk.gather_global(prs, graphs, n)
    touched = part.replicas > 0
    assert np.max(np.abs(got[touched] - want[touched]) / want[touched]) < PR_TOL
    # float mode: same procedure, float accuracy
    graphs32, prs32 = build_parts(part, n, u, v, cuda_device, False, 0.0)
    prk.power_iterate_local(prs32, 20, 0.85)
    got32 = prk.gather_global(prs32, graphs32, n)
    assert np.max(np.abs(got32[touched] - want[touched]) / want[touched]) < 1e-4


@pytest.mark.parametrize("parts", [1, 3])
def test_pairs_laid_out_by_gather_frequency(cuda_device, oracle, parts, monkeypatch):
    """Large parts publish their {delta, pushed} pairs in the order of how often they are gathered and renumber the pull
    lists' columns to match (forced here on a small graph): only the addresses of the gathers change, so the values
    and the superstep count are bit for bit those of the plain layout, in both schedules."""
    n, u, v = gg.rmat_graph(13, 16, seed=36, symmetrise=False, self_loops="drop")
    u, v = u.numpy(), v.numpy()
    part = pt.ebv_partition(n, u, v, parts, keep_self_loops=False)
    results = []
    for min_rows in ("0", "1"):
        monkeypatch.setenv("DRONE_PR_ORDER_MIN_ROWS", min_rows)
        graphs, prs = build_parts(part, n, u, v, cuda_device, False, 1e-6)
        steps, _ = prk.run_job_local(prs)
        delta = prk.gather_global(prs, graphs, n)
        prk.power_iterate_local(prs, 20, 0.85)
        results.append((steps, delta, prk.gather_global(prs, graphs, n)))
    assert results[0][0] == results[1][0]
    assert np.array_equal(results[0][1], results[1][1]) and np.array_equal(results[0][2], results[1][2])
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    touched = part.replicas > 0
    assert np.max(np.abs(results[1][2][touched] - want[touched]) / want[touched]) < 1e-4


def test_against_cpu_job_restatement(cuda_device, oracle):
    """DRONE's CPU job (float, eps 0.01, at most 200 supersteps) and the GPU schedule agree to the
    accuracy the CPU job's threshold allows."""
    n, u, v, out_deg, part = pr_case(scale=10, seed=33, parts=2)
    cpu, _, _ = oracle.pr_drone_cpu(n, part.part_u, part.part_v, out_deg, part.owner, eps=0.01, max_steps=200)
    graphs, prs = build_parts(part, n, u, v, cuda_device, True, 1e-9)
    prk.run_job_local(prs)
    got = prk.gather_global(prs, graphs, n)
    touched = (part.replicas > 0) & (out_deg > 0)
    # the CPU job ignores dangling mass; three dangling vertices of 1024 shift values by well under its threshold
    assert np.median(np.abs(got[touched] - cpu[touched]) / cpu[touched]) < 0.05


def test_call_order_is_checked(cuda_device, oracle):
    n, u, v, out_deg, part = pr_case(scale=8, seed=34, parts=1)
    graphs, prs = build_parts(part, n, u, v, cuda_device, False, 1e-6)
    with pytest.raises(db.DroneError, match="before PR_PEVal"):
        prs[0].inceval()
    res = prs[0].peval()
    assert res.LocalVertexSize == graphs[0].n_local and res.is_empty()
    assert res.VisitedSize > 0


def _nccl_rank(rank, world, port, ok):
    import torch.distributed as dist
    from oracle import oracle
    os.environ["MASTER_ADDR"] = "127.0.0.1"
    os.environ["MASTER_PORT"] = str(port)
    os.environ.setdefault("NCCL_NVLS_ENABLE", "0")
    torch.cuda.set_device(rank)
    dev = torch.device("cuda", rank)
    dist.init_process_group("gloo", rank=rank, world_size=world)
    try:
        n, u, v, out_deg, part = pr_case(scale=10, seed=35, parts=world)
        want, want_steps, _ = oracle.pr_drone_cuda(n, part.part_u, part.part_v, out_deg, part.owner, eps=1e-6,
                                                   dtype=np.float64)
        in_deg = np.bincount(v, minlength=n).astype(np.int32)
        comm = gs.Comm(rank, world)
        g = gs.DeviceGraph(part.local_graph(rank), in_deg, out_deg, dev, max_features=1)
        pr_ = prk.PageRank(g, n, comm=comm, use_double=True, eps=1e-6, n_isolated=int((part.replicas == 0).sum()))
        res = pr_.peval()
        steps = 1
        while True:
            flag = torch.tensor([0 if res.is_empty() else 1])
            dist.all_reduce(flag)                      # the master's "any worker has messages" (master.go:283-287)
            if int(flag) == 0:
                break
            res = pr_.inceval()
            steps += 1
        assert steps == want_steps
        vals = pr_.values()
        keep = g.host.mirror2worker == -1
        gid = g.host.l2g[keep]
        assert np.max(np.abs(vals[keep] - want[gid]) / want[gid]) < PR_TOL
        pr_.power_iterate(20, 0.85)
        index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
        wantp = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
        vals = pr_.values()
        assert np.max(np.abs(vals[keep] - wantp[gid]) / wantp[gid]) < PR_TOL
        # the same job with the boundary entries stored straight into the peer's memory: same supersteps, same values
        g2 = gs.DeviceGraph(part.local_graph(rank), in_deg, out_deg, dev, max_features=4)
        g2.xplan.enable_p2p(comm)
        pr2 = prk.PageRank(g2, n, comm=comm, use_double=True, eps=1e-6, n_isolated=int((part.replicas == 0).sum()))
        assert pr2.transport_name().startswith("peer memory")
        res = pr2.peval()
        steps2 = 1
        while True:
            flag = torch.tensor([0 if res.is_empty() else 1])
            dist.all_reduce(flag)
            if int(flag) == 0:
                break
            res = pr2.inceval()
            steps2 += 1
        assert steps2 == want_steps
        vals2 = pr2.values()
        assert np.max(np.abs(vals2[keep] - want[gid]) / want[gid]) < PR_TOL
        pr2.power_iterate(20, 0.85)
        assert np.array_equal(pr2.values(), vals)
        ok[rank] = 1
        dist.barrier()
        pr2.close()
        pr_.close()
        comm.close()
    finally:
        dist.destroy_process_group()


def test_pagerank_over_nccl_two_gpus():
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    run_ranks(_nccl_rank, 2, (29700 + os.getpid() % 2000,))


@pytest.mark.parametrize("scale,parts,use_double", [(5, 2, True), (12, 12, True), (15, 9, False), (15, 1, True), (16, 3, False)])
def test_supersteps_in_one_launch(cuda_device, oracle, scale, parts, use_double):
    """The persistent kernel at its edges: fewer vertices than a block has threads, more than eight parts, values that do
    and do not all fit the shared-memory table, rows of many partial sums.  The job in one launch takes the supersteps,
    and sends the entries, that the same job driven one superstep at a time does."""
    n, u, v, out_deg, part = pr_case(scale=scale, seed=50 + scale, parts=parts)
    graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 1e-6)
    steps, sizes = prk.run_job_local(prs)
    got = prk.gather_global(prs, graphs, n)
    alone = [[(r.Mirror2MasterSendSize, r.Mirror2MasterRecvSize, r.Master2MirrorSendSize, r.Master2MirrorRecvSize)
              for r in prk.step_local(prs, True)]]
    while any(any(s) for s in alone[-1]):
        alone.append([(r.Mirror2MasterSendSize, r.Mirror2MasterRecvSize, r.Master2MirrorSendSize, r.Master2MirrorRecvSize)
                      for r in prk.step_local(prs, False)])
    assert steps == len(alone) and sizes == alone
    assert np.array_equal(got, prk.gather_global(prs, graphs, n))
    capped, _ = prk.run_job_local(prs, max_steps=1)
    assert capped == 1
    prk.power_iterate_local(prs, 20, 0.85)
    got = prk.gather_global(prs, graphs, n)
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    touched = part.replicas > 0
    assert np.max(np.abs(got[touched] - want[touched]) / want[touched]) < (PR_TOL if use_double else 1e-4)


def test_barrier_count_passes_its_end(cuda_device, monkeypatch):
    """The count of arrivals at the barriers of a launch is modulo 2^32: started just below that it changes nothing."""
    n, u, v, out_deg, part = pr_case(scale=13, seed=70, parts=2)
    results = []
    for start in ("0", str(2 ** 32 - 100)):
        monkeypatch.setenv("DRONE_BARRIER_START", start)
        graphs, prs = build_parts(part, n, u, v, cuda_device, True, 1e-6)
        steps, sizes = prk.run_job_local(prs)
        delta = prk.gather_global(prs, graphs, n)
        prk.power_iterate_local(prs, 20, 0.85)
        results.append((steps, sizes, delta, prk.gather_global(prs, graphs, n)))
    assert results[0][:2] == results[1][:2] and results[0][0] > 3
    assert np.array_equal(results[0][2], results[1][2]) and np.array_equal(results[0][3], results[1][3])
    assert np.ptp(results[1][3]) > 0                    # not the start values


@pytest.mark.parametrize("parts,use_double", [(1, False), (3, True), (12, False)])
def test_a_wait_that_runs_out_is_reported(cuda_device, oracle, monkeypatch, parts, use_double):
    """A barrier between the blocks of a run gives up after a bounded number of looks (here: none).  The synchronous calls
    report that themselves, the asynchronous power iteration through drone_pr_values of every part; a run that should have
    finished leaves no plausible values; the handle and the device stay usable."""
    n, u, v, out_deg, part = pr_case(scale=13, seed=71, parts=parts)
    monkeypatch.setenv("DRONE_BARRIER_POLLS", "0")
    graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 1e-6)
    prk.power_iterate_local(prs, 20, 0.85)
    for pr_ in prs:
        with pytest.raises(db.DroneError, match="ran out"):
            pr_.values()
    out = np.zeros(prs[0].n_local, np.float64 if use_double else np.float32)
    assert db.lib().drone_pr_values(prs[0].handle, out.ctypes.data, None) == -4 and np.isnan(out).all()
    with pytest.raises(db.DroneError, match="ran out"):
        prk.step_local(prs, True)
    with pytest.raises(db.DroneError, match="before PR_PEVal"):
        prk.step_local(prs, False)
    with pytest.raises(db.DroneError, match="ran out"):
        prk.run_job_local(prs)
    monkeypatch.delenv("DRONE_BARRIER_POLLS")
    graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 1e-6)
    prk.power_iterate_local(prs, 20, 0.85)
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    got = prk.gather_global(prs, graphs, n)
    touched = part.replicas > 0
    assert np.max(np.abs(got[touched] - want[touched]) / want[touched]) < (PR_TOL if use_double else 1e-4)


def test_handles_allocate_when_they_are_made(cuda_device):
    """drone_pr_create makes everything a handle needs: the first job and the first power iteration over several parts take no
    device memory (the exchange plans' own copies, made on their first use, are there already)."""
    n, u, v, out_deg, part = pr_case(scale=19, seed=73, parts=3)
    graphs, prs = build_parts(part, n, u, v, cuda_device, True, 1e-6)
    prk.step_local(prs, True)
    fresh = [prk.PageRank(g, n, use_double=True, eps=1e-6) for g in graphs]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info(cuda_device)[0]
    prk.step_local(fresh, True)
    prk.power_iterate_local(fresh, 2, 0.85)
    torch.cuda.synchronize()
    assert torch.cuda.mem_get_info(cuda_device)[0] >= free


@pytest.mark.parametrize("scale,parts,use_double", [(5, 2, True), (13, 1, False), (13, 3, True), (15, 4, True), (16, 2, False),
                                                    (12, 12, False)])
def test_separate_steps_of_one_process_per_gpu(cuda_device, oracle, monkeypatch, scale, parts, use_double):
    """The kernels and the order of steps that a job takes with one process per GPU (pull, pack and apply of both directions,
    dangling mass, isolated vertices), here with all parts in one process and copies for messages: against the double oracle
    of both schedules, and against the persistent kernel in supersteps, exchange sizes, visited vertices and values."""
    n, u, v, out_deg, part = pr_case(scale=scale, seed=80 + scale, parts=parts)
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want_power = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    touched = part.replicas > 0
    tol = PR_TOL if use_double else 1e-4
    results = []
    for separate in ("0", "1"):
        monkeypatch.setenv("DRONE_PR_SEPARATE_STEPS", separate)
        graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 1e-6)
        before = db.lib().drone_kernel_launch_count()
        steps, sizes = prk.run_job_local(prs)
        delta = prk.gather_global(prs, graphs, n)
        visited = [[r.VisitedSize for r in prk.step_local(prs, first)] for first in (True, False)]
        prk.power_iterate_local(prs, 20, 0.85)
        launches = db.lib().drone_kernel_launch_count() - before
        assert (launches > 20 * parts) == (separate == "1")
        power = prk.gather_global(prs, graphs, n)
        assert np.max(np.abs(power[touched] - want_power[touched]) / want_power[touched]) < tol
        # every replica of a vertex ends with its master's value, bit for bit
        for p, g in zip(prs, graphs):
            assert np.array_equal(p.values(), power[g.host.l2g])
        results.append((steps, sizes, visited, delta))
    if use_double:
        want, want_steps, want_sizes = oracle.pr_drone_cuda(n, part.part_u, part.part_v, out_deg, part.owner, eps=1e-6, dtype=np.float64)
        assert results[1][0] == want_steps
        assert np.array_equal(np.array([[sum(s[i] for s in step) for i in range(4)] for step in results[1][1]]), want_sizes)
        assert np.max(np.abs(results[1][3][touched] - want[touched]) / np.abs(want[touched])) < PR_TOL
        assert results[0][:3] == results[1][:3]
    assert np.max(np.abs(results[0][3][touched] - results[1][3][touched]) / np.abs(results[0][3][touched])) < (PR_TOL if use_double else 2e-4)


@pytest.mark.parametrize("use_double", [False, True])
@pytest.mark.parametrize("scale,edge_factor", [(18, 24), (18, 96), (20, 8)])
def test_power_iterations_over_a_stream_of_edges(cuda_device, oracle, scale, edge_factor, use_double):
    """One part of many edges: rows that several pieces of the stream share, rows without edges, vertices without out-edges;
    the same bits every time."""
    n, u, v = gg.rmat_graph(scale, edge_factor, seed=90 + edge_factor, symmetrise=False, self_loops="drop")
    u, v = u.numpy(), v.numpy()
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 5, 0.85)
    part = pt.ebv_partition(n, u, v, 1, keep_self_loops=False)
    graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 0.0)
    touched = part.replicas > 0
    runs = []
    for _ in range(2):
        prk.power_iterate_local(prs, 5, 0.85)
        runs.append(prk.gather_global(prs, graphs, n))
    assert np.max(np.abs(runs[0][touched] - want[touched]) / want[touched]) < (PR_TOL if use_double else 1e-4)
    assert np.array_equal(runs[0], runs[1])
    prk.power_iterate_local(prs, 0, 0.85)
    assert np.ptp(prk.gather_global(prs, graphs, n)[touched]) == 0


@pytest.mark.parametrize("scale,parts,use_double", [(4, 1, True), (5, 2, False), (9, 3, True), (12, 12, True), (13, 1, False),
                                                    (15, 9, True), (16, 1, True), (16, 4, True), (17, 2, False)])
def test_slices_in_shared_memory(cuda_device, oracle, monkeypatch, scale, parts, use_double):
    """Graphs whose edges fit the SMs' shared memory, against the kernels for larger ones: fewer rows than threads, rows that
    many threads share, rows without edges, more than eight parts, masters with more than four mirrors; the job at once and
    superstep by superstep, with everything a caller can see of its state."""
    n, u, v, out_deg, part = pr_case(scale=scale, seed=110 + scale, parts=parts)
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    touched = part.replicas > 0
    tol = PR_TOL if use_double else 1e-4
    results = []
    for slices in ("0", "1"):
        monkeypatch.setenv("DRONE_PR_SLICES", slices)
        graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 1e-6)
        steps, sizes = prk.run_job_local(prs)
        delta = prk.gather_global(prs, graphs, n)
        some = [[(r.Mirror2MasterSendSize, r.Master2MirrorRecvSize, r.VisitedSize) for r in prk.step_local(prs, first)]
                for first in (True, False, False)]
        prk.step_local(prs, True)
        prk.step_local(prs, False)
        state = [device_state(p) for p in prs]
        prk.power_iterate_local(prs, 20, 0.85)
        power = prk.gather_global(prs, graphs, n)
        assert np.max(np.abs(power[touched] - want[touched]) / want[touched]) < tol
        for p, g in zip(prs, graphs):
            assert np.array_equal(p.values(), power[g.host.l2g])
        results.append((steps, sizes, some, delta, state))
    a, b = results
    assert np.max(np.abs(a[3][touched] - b[3][touched]) / np.abs(a[3][touched])) < (PR_TOL if use_double else 2e-4)
    if use_double:
        assert a[:3] == b[:3]
    for x, y in zip(a[4], b[4]):
        for name in ("active", "ubm"):
            assert np.array_equal(x[name], y[name])
        for name in ("pr", "acc", "diff"):
            # values start at 1, and so do the terms of a sum, whatever cancels in it: a float sum is off by a few 2^-24 of that
            assert np.max(np.abs(x[name] - y[name]) / np.maximum(np.abs(x[name]), 1e-3 if use_double else 1.0)) < (PR_TOL if use_double else 1e-4), name


def hub_graph(n, edges, hubs, seed):
    """Random edges, and for every (vertex, in-edges) of `hubs` that many sources more."""
    rng = np.random.default_rng(seed)
    u, v = [rng.integers(0, n, edges)], [rng.integers(0, n, edges)]
    for vertex, count in hubs:
        u.append(rng.permutation(n)[:count])
        v.append(np.full(count, vertex))
    u, v = np.concatenate(u), np.concatenate(v)
    key = np.unique((u * n + v)[u != v])
    return (key // n).astype(np.int32), (key % n).astype(np.int32)


@pytest.mark.parametrize("use_double", [False, True])
@pytest.mark.parametrize("n,edges,hubs", [(20000, 60000, [(13, 19999)]), (20000, 0, [(19999, 19000), (0, 4097), (1, 4098), (7, 300)]),
                                          (33333, 50000, [(k, 1000 + 700 * k) for k in range(45)])])
def test_rows_of_many_pieces(cuda_device, oracle, monkeypatch, n, edges, hubs, use_double):
    """One part's edges as a stream with rows that reach over a few and over many of its pieces, several of them in one warp."""
    monkeypatch.setenv("DRONE_PR_SLICES", "0")
    u, v = hub_graph(n, edges, hubs, seed=len(hubs))
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    part = pt.ebv_partition(n, u, v, 1, keep_self_loops=False)
    graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 0.0)
    prk.power_iterate_local(prs, 20, 0.85)
    got = prk.gather_global(prs, graphs, n)
    touched = part.replicas > 0
    assert np.max(np.abs(got[touched] - want[touched]) / want[touched]) < (PR_TOL if use_double else 1e-4)
    prk.power_iterate_local(prs, 20, 0.85)
    assert np.array_equal(prk.gather_global(prs, graphs, n), got)


@pytest.mark.parametrize("parts,use_double,hub,kept", [(1, False, 30000, False), (1, True, 20000, False), (1, True, 2000, True),
                                                       (2, True, 60000, False)])
def test_slices_of_a_vertex_with_many_edges(cuda_device, oracle, monkeypatch, parts, use_double, hub, kept):
    """A vertex whose edges would make one block's slice much larger than the others' keeps a run out of the slices, whose sums
    add in another order: the values are bit for bit those of a handle without slices."""
    n = 65536
    u, v = hub_graph(n, 8 * n, [(13, hub)], seed=hub)
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    part = pt.ebv_partition(n, u, v, parts, keep_self_loops=False)
    touched, power = part.replicas > 0, []
    for slices in ("0", "1"):
        monkeypatch.setenv("DRONE_PR_SLICES", slices)
        graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 1e-6)
        prk.power_iterate_local(prs, 20, 0.85)
        power.append(prk.gather_global(prs, graphs, n))
        assert np.max(np.abs(power[-1][touched] - want[touched]) / want[touched]) < (PR_TOL if use_double else 1e-4)
    assert np.array_equal(power[0], power[1]) == (not kept)


@pytest.mark.parametrize("use_double", [False, True])
def test_job_of_one_part_takes_no_slices(cuda_device, monkeypatch, use_double):
    """One superstep does not repay filling the slices: whole or step by step the job of one part has the bits of a handle without."""
    n, u, v, _, part = pr_case(scale=14, seed=79, parts=1)
    seen = []
    for slices in ("0", "1"):
        monkeypatch.setenv("DRONE_PR_SLICES", slices)
        graphs, prs = build_parts(part, n, u, v, cuda_device, use_double, 1e-6)
        steps, sizes = prk.run_job_local(prs)
        seen.append((steps, sizes, prk.gather_global(prs, graphs, n)))
        prk.step_local(prs, True)
        prk.step_local(prs, False)
        seen[-1] += (prk.gather_global(prs, graphs, n), device_state(prs[0])["acc"])
    for a, b in zip(*seen):
        assert np.array_equal(a, b)


def test_state_after_the_whole_job(cuda_device, monkeypatch):
    """What a job that runs in slices to its end leaves of every part's state, against the kernel without them."""
    n, u, v, _, part = pr_case(scale=13, seed=77, parts=3)
    states = []
    for slices in ("0", "1"):
        monkeypatch.setenv("DRONE_PR_SLICES", slices)
        _, prs = build_parts(part, n, u, v, cuda_device, True, 1e-6)
        prk.run_job_local(prs)
        states.append([device_state(p) for p in prs])
    for x, y in zip(*states):
        for name in ("active", "ubm"):
            assert np.array_equal(x[name], y[name])
        for name in ("pr", "acc", "diff"):
            assert np.max(np.abs(x[name] - y[name]) / np.maximum(np.abs(x[name]), 1e-3)) < PR_TOL, name


def device_state(job):
    """The arrays of drone_pr_device_arrays, copied."""
    ptrs = [C.c_void_p(0) for _ in range(5)]
    check(db.lib().drone_pr_device_arrays(job.handle, *[C.byref(p) for p in ptrs]))
    kinds = ["<f8" if job.use_double else "<f4"] * 3 + ["<i4"] * 2
    out = {}
    for name, p, t in zip(("pr", "acc", "diff", "active", "ubm"), ptrs, kinds):
        view = types.SimpleNamespace(__cuda_array_interface__={"shape": (job.n_local,), "typestr": t, "data": (p.value, False), "version": 2})
        out[name] = torch.as_tensor(view, device="cuda").cpu().numpy()
    return out
