"""Making a PageRank handle where one of its launches or allocations fails: an error, or a handle that gives the right values.  The
failing calls are a fake's, in a child process (failing_calls.c): nothing reaches the GPU in their place."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

CHILD = """
import ctypes, os, sys
sys.path[:0] = [%(root)r, %(here)r]
import numpy as np, torch
import drone_b200 as db
from drone_b200 import graphgen as gg, pagerank as prk, partition as pt
from test_pagerank_gpu import build_parts
fake, dev = ctypes.CDLL(%(fake)r), torch.device("cuda", 0)
stream = sys.argv[1] == "stream"
os.environ["DRONE_PR_SLICES"] = "0" if stream else "1"
os.environ["DRONE_PR_ORDER_MIN_ROWS"] = "1"
n, u, v = gg.rmat_graph(12, 16, seed=5, symmetrise=False, self_loops="drop")
part = pt.ebv_partition(n, u.numpy(), v.numpy(), 1, keep_self_loops=False)
graphs, prs = build_parts(part, n, u.numpy(), v.numpy(), dev, False, 1e-6)
fake.fail_launch(-1)
fake.fail_allocation(-1)
make = lambda: prk.PageRank(graphs[0], n, use_double=False, eps=1e-6, n_isolated=int((part.replicas == 0).sum()))
def values(job):
    prk.power_iterate_local([job], 20, 0.85)
    return job.values()
want = values(make())
fake.fail_launch(-1)
fake.fail_allocation(-1)
job = make()
launches, allocations = fake.launches_made(), fake.allocations_made()
assert launches > 5 and allocations > 2
for k in range(launches):
    fake.fail_launch(k)
    try:
        make()
    except db.DroneError:
        continue
    raise SystemExit("launch %%d of %%d failed and nobody said so" %% (k, launches))
fake.fail_launch(-1)
did_without = 0
for k in range(allocations):
    fake.fail_allocation(k)
    try:
        job = make()
    except db.DroneError:
        continue
    fake.fail_allocation(-1)
    did_without += 1
    got = values(job)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
assert did_without == (2 if stream else 0), did_without
fake.fail_allocation(-1)
assert np.array_equal(values(make()), want)
print("ok")
"""


@pytest.mark.parametrize("form", ["slices", "stream"])
def test_failing_calls_while_a_handle_is_made(cuda_device, tmp_path, form):
    fake = str(tmp_path / "failing_calls.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-o", fake, os.path.join(HERE, "failing_calls.c"), "-ldl"], check=True)
    code = CHILD % {"root": os.path.dirname(HERE), "here": HERE, "fake": fake}
    done = subprocess.run([sys.executable, "-c", code, form], env=dict(os.environ, LD_PRELOAD=fake), capture_output=True, text=True,
                          timeout=300)
    assert done.returncode == 0 and done.stdout.strip().endswith("ok"), done.stdout + done.stderr
