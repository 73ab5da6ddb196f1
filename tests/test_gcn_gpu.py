"""End-to-end check of the aggregation path inside the reference's 2-layer GCN step: outputs and gradients against
the double-precision oracle (1e-5 relative), on one GPU and, with two GPUs, as two EBV parts over NCCL."""
import os

import numpy as np
import pytest
import torch

import drone_b200 as db
from drone_b200 import gcn, graphgen as gg, graphsum as gs, partition as pt
from helpers import run_ranks, graph_case
from oracle import gcn_oracle

pytestmark = pytest.mark.gpu
GCN_TOL = 1e-5


def glorot(seed, fan_in, fan_out):
    """(U - 0.5) * 2 * sqrt(6 / (in + out)) (cuda_gcn/src/cuda/cuda_kernel.cu:469-474), from a fixed seed."""
    rng = np.random.default_rng(seed)
    return ((rng.random((fan_in, fan_out)) - 0.5) * 2 * np.sqrt(6.0 / (fan_in + fan_out))).astype(np.float32)


def make_case(scale=10, dims=(40, 32, 7)):
    n, u, v = gg.rmat_graph(scale, 12, seed=51, symmetrise=True, self_loops="add")
    u, v = u.numpy(), v.numpy()
    x = gg.seeded_normal(3, (n, dims[0]))
    truth = np.random.default_rng(4).integers(-1, dims[2], n).astype(np.int32)     # -1: unlabelled
    return n, u, v, x, truth, glorot(5, dims[0], dims[1]), glorot(6, dims[1], dims[2])


def rel(got, want):
    return float(np.abs(np.asarray(got, np.float64) - want).max() / max(np.abs(want).max(), 1e-30))


def test_gcn_step_single_gpu(cuda_device, oracle):
    n, u, v, x, truth, w1, w2 = make_case()
    index, dst, in_deg, out_deg, val = graph_case(gg, oracle, n, u, v)
    want = gcn_oracle.gcn_step(index, dst, val, x, w1, w2, truth)
    part = pt.ebv_partition(n, u, v, 1)
    lg = part.local_graph(0)
    g = gs.DeviceGraph(lg, in_deg, out_deg, cuda_device, max_features=32)
    t = lambda a: torch.as_tensor(a, device=cuda_device)
    torch.backends.cuda.matmul.allow_tf32 = False
    step = gcn.GCNStep(g, t(x[lg.l2g]), t(truth[lg.l2g]), t(w1), t(w2))
    loss = step.forward()
    step.backward()
    torch.cuda.synchronize()
    inv = lg.l2g
    assert rel(step.logits.cpu().numpy(), want["logits"][inv]) < GCN_TOL
    assert rel(step.z1.cpu().numpy(), want["z1"][inv]) < GCN_TOL
    assert abs(float(loss) - want["loss"]) < GCN_TOL * max(1.0, abs(want["loss"]))
    assert rel(step.d_h2.cpu().numpy(), want["d_h2"][inv]) < GCN_TOL
    assert rel(step.d_h1.cpu().numpy(), want["d_h1"][inv]) < GCN_TOL
    assert rel(step.d_w2.cpu().numpy(), want["d_w2"]) < GCN_TOL
    assert rel(step.d_w1.cpu().numpy(), want["d_w1"]) < GCN_TOL


def _rank(rank, world, port, ok):
    import torch.distributed as dist
    from oracle import oracle
    os.environ["MASTER_ADDR"], os.environ["MASTER_PORT"] = "127.0.0.1", str(port)
    os.environ.setdefault("NCCL_NVLS_ENABLE", "0")
    torch.cuda.set_device(rank)
    dev = torch.device("cuda", rank)
    dist.init_process_group("gloo", rank=rank, world_size=world)
    try:
        n, u, v, x, truth, w1, w2 = make_case()
        index, dst, in_deg, out_deg, val = graph_case(gg, oracle, n, u, v)
        want = gcn_oracle.gcn_step(index, dst, val, x, w1, w2, truth)
        part = pt.ebv_partition(n, u, v, world)
        lg = part.local_graph(rank)
        g = gs.DeviceGraph(lg, in_deg, out_deg, dev, max_features=32)
        comm = gs.Comm(rank, world)
        t = lambda a: torch.as_tensor(a, device=dev)
        torch.backends.cuda.matmul.allow_tf32 = False
        step = gcn.GCNStep(g, t(x[lg.l2g]), t(truth[lg.l2g]), t(w1), t(w2), comm=comm, worker_num=world)
        if rank != 0:                     # weights live on rank 0 and are broadcast at the start of every forward pass
            step.weights[0].zero_()
            step.weights[1].zero_()
        step.broadcast_weights()          # weight_broadcast_value_nccl (cuda_communicate.cu:99-105)
        step.forward()
        d_w1, d_w2 = step.backward()
        step.reduce_gradients()           # weight_reduce_grad_nccl: the sums land on rank 0 (cuda_communicate.cu:107-115)
        torch.cuda.synchronize()
        assert rel(step.logits.cpu().numpy(), want["logits"][lg.l2g]) < GCN_TOL
        # mirror rows of the layer gradients are zeroed in place before dW, as clear_mirror_grad does
        masters = lg.mirror2worker == -1
        assert rel(step.d_h1.cpu().numpy()[masters], want["d_h1"][lg.l2g][masters]) < GCN_TOL
        assert not step.d_h1.cpu().numpy()[~masters].any()
        if rank == 0:
            assert rel(d_w2.cpu().numpy(), want["d_w2"]) < GCN_TOL
            assert rel(d_w1.cpu().numpy(), want["d_w1"]) < GCN_TOL
        ok[rank] = 1
        dist.barrier()
        comm.close()
    finally:
        dist.destroy_process_group()


def test_gcn_step_two_gpus():
    if torch.cuda.device_count() < 2:
        pytest.skip("needs two GPUs")
    run_ranks(_rank, 2, (29800 + os.getpid() % 2000,))


@pytest.mark.parametrize("classes", [1, 7, 8, 9, 16, 17, 33, 41, 64, 65, 256, 257, 1000])
@pytest.mark.parametrize("n,share", [(1, 1.0), (37, 0.0), (5003, 0.66), (200001, 0.66)])
def test_loss_and_relu_mask(cuda_device, n, share, classes):
    """The loss kernel at the edges of its lane groups, without labelled rows, and with rows of infinities, against the same
    steps in double; the mask of the ReLU's gradient, where it is read as vectors and where not."""
    if n * classes > 3e7:
        pytest.skip("the shape is covered with fewer classes")
    gen = torch.Generator(cuda_device).manual_seed(n + classes)
    model = gcn.GCN(None, torch.zeros((n, 4), device=cuda_device),
                    torch.randint(0, classes, (n,), device=cuda_device, generator=gen, dtype=torch.int32),
                    [torch.zeros((4, classes), device=cuda_device)], aggregate=lambda *a: None)
    model.labelled = torch.rand(n, device=cuda_device, generator=gen) < share
    logits = torch.randn((n, classes), device=cuda_device, generator=gen) * 4
    z, lab = logits.double(), model.labelled
    p = torch.softmax(z, 1)
    want_loss = -(torch.log_softmax(z, 1).gather(1, model.safe_truth[:, None])[:, 0] * lab).sum() / max(int(lab.sum()), 1)
    want = (p - torch.nn.functional.one_hot(model.safe_truth, classes)) * lab[:, None]
    loss = model._softmax_loss(logits)
    # exponentials, a sum of `classes` terms and a quotient in float
    assert (model.d_logits - want).abs().max() <= (8 + classes / 8) * 2.0 ** -24
    assert abs(float(loss) - float(want_loss)) <= 1e-6 * max(1.0, float(want_loss))
    assert torch.equal(model._softmax_loss(logits), loss)
    if n > 30 and classes > 4:      # what torch makes of infinities and NaN, entry by entry
        odd = logits.clone()
        odd[3, 1], odd[5, 2], odd[7, 0], odd[9] = float("inf"), float("nan"), -float("inf"), -float("inf")
        model._softmax_loss(odd)
        want = (torch.softmax(odd, 1) - torch.nn.functional.one_hot(model.safe_truth, classes)) * lab[:, None]
        assert torch.equal(model.d_logits.isnan(), want.isnan())
        fine = ~want.isnan()
        assert (model.d_logits - want)[fine].abs().max() <= (8 + classes / 8) * 2.0 ** -23
    grad, out = torch.randn_like(logits), torch.randn_like(logits).clamp_(min=0)
    want = grad * (out > 0)
    assert torch.equal(model._relu_mask(grad, out), want)


def test_labels_outside_the_classes_are_refused(cuda_device):
    with pytest.raises(ValueError, match="label"):
        gcn.GCN(None, torch.zeros((3, 4), device=cuda_device), torch.tensor([0, 5, -1], dtype=torch.int32, device=cuda_device),
                [torch.zeros((4, 5), device=cuda_device)])


@pytest.mark.parametrize("k,m,n", [(1, 1, 1), (15, 3, 5), (17, 64, 64), (63, 65, 7), (64, 128, 64), (65, 129, 65), (1000, 602, 128),
                                   (3001, 100, 16), (9999, 33, 47), (20000, 128, 41), (300, 700, 300), (0, 5, 6)])
def test_weight_gradient(cuda_device, k, m, n):
    """Tiles and shares at their edges, odd widths and leading dimensions, against double; the same bits every time."""
    gen = torch.Generator(cuda_device).manual_seed(k + m + n)
    model = gcn.GCN(None, torch.zeros((1, 4), device=cuda_device), torch.zeros(1, dtype=torch.int32, device=cuda_device),
                    [torch.zeros((4, 5), device=cuda_device)], aggregate=lambda *a: None)
    a = torch.randn((k, m + 3), device=cuda_device, generator=gen)[:, 1:m + 1]
    g = torch.randn((k, n), device=cuda_device, generator=gen)
    got, want = model._weight_gradient(a, g), a.double().t() @ g.double()
    # a chain of k additions of terms of size 1: sqrt(k) roundings of a sum that has grown to sqrt(k), and some to spare
    assert (got - want).abs().max() <= 6 * 2.0 ** -24 * (k + 30) if k else (got == 0).all()
    assert torch.equal(got, model._weight_gradient(a, g))
    assert torch.equal(model._weight_gradient(a.contiguous(), g), got)
