"""The kernels of a graph-convolution training step beside the aggregation: loss, mask of the ReLU's gradient, weight gradients."""
import pytest
import torch

from drone_b200 import gcn

pytestmark = pytest.mark.gpu


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


def test_weight_gradient_of_rows_that_overlap(cuda_device):
    """Inputs whose rows are one row of memory (expanded), or begin inside the one before."""
    gen = torch.Generator(cuda_device).manual_seed(5)
    model = gcn.GCN(None, torch.zeros((1, 4), device=cuda_device), torch.zeros(1, dtype=torch.int32, device=cuda_device),
                    [torch.zeros((4, 5), device=cuda_device)], aggregate=lambda *a: None)
    flat, g = torch.randn(600, device=cuda_device, generator=gen), torch.randn((100, 24), device=cuda_device, generator=gen)
    for a in (flat[:40].expand(100, 40), flat.as_strided((100, 40), (3, 1))):
        want = a.double().t() @ g.double()
        assert (model._weight_gradient(a, g) - want).abs().max() <= 6 * 2.0 ** -24 * 130


def test_labels_elsewhere_are_refused(cuda_device):
    """Labels that are not one a row on the model's device do not reach the kernel: torch refuses them."""
    def model(truth):
        return gcn.GCN(None, torch.zeros((6, 4), device=cuda_device), truth, [torch.zeros((4, 5), device=cuda_device)],
                       aggregate=lambda *a: None)
    logits = torch.zeros((6, 5), device=cuda_device)
    for truth in (torch.zeros(6, dtype=torch.int32), torch.zeros(4, dtype=torch.int32, device=cuda_device)):
        with pytest.raises(RuntimeError):
            model(truth)._softmax_loss(logits)


def test_sizes_beyond_the_row_numbers_are_refused(cuda_device):
    """Rows are numbered in 32 bits, a share beyond the last one: more than 2^30 rows are an error before anything is launched."""
    import ctypes as C
    from drone_b200._lib import lib
    size = C.c_longlong(0)
    assert lib().drone_weight_gradient_scratch(2 ** 30 + 1, 4, 4, C.byref(size)) == -1
    assert lib().drone_weight_gradient_scratch(2 ** 30, 4, 4, C.byref(size)) == 0 and size.value > 0


@pytest.mark.parametrize("default", [torch.float64, torch.bfloat16, torch.float16])
def test_default_dtype_changed_after_the_model_was_made(cuda_device, default):
    """What the kernels write into is float32 whatever torch makes by default when the step runs."""
    gen = torch.Generator(cuda_device).manual_seed(11)
    n, dims = 5003, (65, 24, 7)
    x = torch.randn((n, dims[0]), device=cuda_device, generator=gen)
    truth = torch.randint(-1, dims[-1], (n,), device=cuda_device, generator=gen, dtype=torch.int32)
    weights = [torch.randn((a, b), device=cuda_device, generator=gen) / 8 for a, b in zip(dims, dims[1:])]
    model = gcn.GCN(None, x, truth, weights, aggregate=lambda op, src, out: out.copy_(src))
    assert model._kernels
    want = [model.forward(), *model.backward()]
    try:
        torch.set_default_dtype(default)
        got = [model.forward(), *model.backward()]
    finally:
        torch.set_default_dtype(torch.float32)
    for a, b in zip(got, want):
        assert a.dtype == torch.float32 and torch.equal(a, b)


def bare_model(device, classes=5):
    return gcn.GCN(None, torch.zeros((6, 4), device=device), torch.zeros(6, dtype=torch.int32, device=device),
                   [torch.zeros((4, classes), device=device)], aggregate=lambda *a: None)


def test_what_the_kernels_cannot_read_goes_to_torch(cuda_device):
    """Operands of a weight gradient, a mask or a loss that differ in rows, device or type, or do not lie in rows: torch's result
    or torch's refusal."""
    model, gen = bare_model(cuda_device), torch.Generator(cuda_device).manual_seed(13)
    a, g = torch.randn((300, 40), device=cuda_device, generator=gen), torch.randn((300, 24), device=cuda_device, generator=gen)
    for other in (g[:299], torch.cat([g, g]), g.cpu(), g.double(), g.half()):
        with pytest.raises(RuntimeError) as ours:
            model._weight_gradient(a, other)
        with pytest.raises(RuntimeError) as torchs:
            a.t() @ other
        assert str(ours.value) == str(torchs.value)
    want = a.double().t() @ g.double()
    assert (model._weight_gradient(a, g[:, 0]) - want[:, 0]).abs().max() <= 6 * 2.0 ** -24 * 330
    for other in (g.t().contiguous().t(), torch.cat([g, g], dim=1)[:, :24], torch.randn((600, 24), device=cuda_device)[::2].copy_(g)):
        assert (model._weight_gradient(a, other) - want).abs().max() <= 6 * 2.0 ** -24 * 330
    assert torch.equal(model._weight_gradient(a.double(), g.double()), want)
    assert model._weight_gradient(a[:, :0], g).shape == (0, 24)
    grad, out = torch.randn((9, 12), device=cuda_device, generator=gen), torch.randn((9, 12), device=cuda_device, generator=gen)
    for x, z in ((grad.double(), out.double()), (grad.t().contiguous().t(), out), (grad.clone(), out.t().contiguous().t()), (grad.clone(), out[:1])):
        assert torch.equal(model._relu_mask(x, z), grad.to(x.dtype) * (z > 0))
    logits = torch.randn((6, 5), device=cuda_device, generator=gen)
    want = model._softmax_loss(logits).clone()
    assert abs(float(model._softmax_loss(logits.double())) - float(want)) < 1e-6 and model.d_logits.dtype == torch.float64


@pytest.mark.parametrize("classes", [5, 41, 300])
def test_labels_changed_to_classes_that_do_not_exist(cuda_device, classes):
    """Labels set on a model are looked at like those it was made with; changed in place they leave no plausible loss."""
    for outside in (-1, classes, 2 ** 40):
        model = bare_model(cuda_device, classes)
        logits = torch.randn((6, classes), device=cuda_device)
        assert torch.isfinite(model._softmax_loss(logits))
        truth = model.safe_truth.clone()
        truth[4] = outside
        with pytest.raises(ValueError, match="label"):
            model.safe_truth = truth
        model.safe_truth = torch.full_like(truth, classes - 1)
        assert torch.isfinite(model._softmax_loss(logits))
        model.safe_truth[4] = outside
        assert model._softmax_loss(logits).isnan()
        assert model.d_logits[4].isnan().all() and torch.isfinite(model.d_logits[[0, 1, 2, 3, 5]]).all()
