"""The grid barriers of the persistent PageRank kernels, in each of their forms: a count of arrivals that passes its end, and a
wait that runs out."""
import numpy as np
import pytest
import torch

import drone_b200 as db
from drone_b200 import graphgen as gg
from drone_b200 import pagerank as prk
from drone_b200 import partition as pt
from test_pagerank_gpu import PR_TOL, build_parts
from test_pagerank_oracle import pr_case

pytestmark = pytest.mark.gpu

# (parts, double): rows in shared memory, columns in global memory, and one part's edges as a stream
FORMS = [("slices", 2, True), ("columns", 1, False), ("columns", 3, True), ("columns", 12, False), ("stream", 1, False), ("stream", 1, True)]


def handles(form, parts, use_double, dev, monkeypatch):
    monkeypatch.setenv("DRONE_PR_SLICES", "1" if form == "slices" else "0")
    if form == "stream":      # more edges than shared memory holds, in the order of how often they are gathered
        n, u, v = gg.rmat_graph(18, 24, seed=114, symmetrise=False, self_loops="drop")
        u, v = u.numpy(), v.numpy()
        part = pt.ebv_partition(n, u, v, 1, keep_self_loops=False)
    else:
        n, u, v, _, part = pr_case(scale=13, seed=70, parts=parts)
    graphs, prs = build_parts(part, n, u, v, dev, use_double, 1e-6)
    index, dst = gg.csr_by_source(torch.as_tensor(u), torch.as_tensor(v), n)
    return n, index, dst, part, graphs, prs


@pytest.mark.parametrize("form,parts,use_double", FORMS)
def test_barrier_count_passes_its_end_in_every_form(cuda_device, monkeypatch, form, parts, use_double):
    """The count of arrivals is modulo 2^32: started just below that it changes nothing."""
    results = []
    for start in ("0", str(2 ** 32 - 100)):
        monkeypatch.setenv("DRONE_BARRIER_START", start)
        n, _, _, _, graphs, prs = handles(form, parts, use_double, cuda_device, monkeypatch)
        prk.power_iterate_local(prs, 20, 0.85)
        power = prk.gather_global(prs, graphs, n)
        steps, sizes = prk.run_job_local(prs)
        results.append((steps, sizes, power, prk.gather_global(prs, graphs, n)))
    assert results[0][:2] == results[1][:2]
    assert np.array_equal(results[0][2], results[1][2]) and np.array_equal(results[0][3], results[1][3])
    assert np.ptp(results[1][2]) > 0


@pytest.mark.parametrize("form,parts,use_double", FORMS)
def test_a_wait_that_runs_out_is_reported_in_every_form(cuda_device, oracle, monkeypatch, form, parts, use_double):
    """No look at the count at all: every block gives up at its first barrier.  The job reports it, the power iteration through
    drone_pr_values of every part, whose values are NaN; new handles work."""
    monkeypatch.setenv("DRONE_BARRIER_POLLS", "0")
    n, index, dst, part, graphs, prs = handles(form, parts, use_double, cuda_device, monkeypatch)
    for _ in range(2):
        prk.power_iterate_local(prs, 20, 0.85)
        out = np.zeros(prs[0].n_local, np.float64 if use_double else np.float32)
        assert db.lib().drone_pr_values(prs[0].handle, out.ctypes.data, None) == -4 and np.isnan(out).all()
        for p in prs:
            with pytest.raises(db.DroneError, match="ran out"):
                p.values()
    with pytest.raises(db.DroneError, match="ran out"):
        prk.step_local(prs, True)
    with pytest.raises(db.DroneError, match="ran out"):
        prk.run_job_local(prs)
    monkeypatch.delenv("DRONE_BARRIER_POLLS")
    n, index, dst, part, graphs, prs = handles(form, parts, use_double, cuda_device, monkeypatch)
    prk.power_iterate_local(prs, 20, 0.85)
    want = oracle.pagerank_power_f64(index.numpy(), dst.numpy(), 20, 0.85)
    got = prk.gather_global(prs, graphs, n)
    touched = part.replicas > 0
    assert np.max(np.abs(got[touched] - want[touched]) / want[touched]) < (PR_TOL if use_double else 1e-4)
