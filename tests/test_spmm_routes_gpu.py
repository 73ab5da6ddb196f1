"""Routes of an aggregation call that its operands, the plan's buffers or the stream decide, and what must not depend on them."""
import ctypes as C

import pytest
import torch

import drone_b200 as db
from drone_b200 import graphgen as gg

pytestmark = pytest.mark.gpu


def uniform_plan(dev, n, degree, seed):
    """Rows of equally many columns drawn at random: forward rows are short, rows of the transpose differ in length."""
    gen = torch.Generator(dev).manual_seed(seed)
    index = (torch.arange(n + 1, device=dev) * degree).int()
    dst = torch.randint(0, n, (n, degree), device=dev, generator=gen).sort(dim=1).values.int().reshape(-1)
    val = torch.rand(n * degree, device=dev, generator=gen) - 0.5
    return (lambda: db.AggregationPlan(index, dst, values=val)), gen


@pytest.mark.parametrize("n,degree,first,wider", [(30000, 40, 41, 63),         # copies of X and Y, by a wider call of an odd width
                                                  (300000, 24, 29, 232),       # the copy of X, by a call on aligned rows
                                                  (0, 0, 32, 64)])             # partial sums
def test_buffers_of_a_captured_call_outlive_their_replacement(cuda_device, n, degree, first, wider):
    """A graph captured from a call runs on with what the call used, also after a wider call has replaced the plan's buffers by
    larger ones and other tensors lie where memory came free."""
    if n:
        make, gen = uniform_plan(cuda_device, n, degree, n)
        plan = make()
    else:
        n, u, v = gg.rmat_graph(13, 16, seed=3, device=cuda_device, symmetrise=True, self_loops="add")
        index, dst = gg.csr_by_source(u, v, n)
        in_deg, out_deg = gg.degrees(u, v, n)
        plan, gen = db.AggregationPlan(index, dst, in_degree=in_deg, out_degree=out_deg), torch.Generator(cuda_device).manual_seed(1)
        assert plan.stats().n_partials[db.OP_AT] > 0
    x = torch.randn((n, first), device=cuda_device, generator=gen)
    want = plan.spmm(db.OP_AT, x)
    out, graph = torch.zeros_like(want), torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        plan.spmm(db.OP_AT, x, out=out)
    for width in (wider, 2 * wider):
        wide = torch.randn((n, width), device=cuda_device, generator=gen)
        again = plan.spmm(db.OP_AT, wide)
        torch.cuda.synchronize()
        junk = [torch.full((size,), float("nan"), device=cuda_device) for size in [1 << 16] * 64 + [1 << 22] * 16]
        out.zero_()
        graph.replay()
        assert torch.equal(out, want)
        assert torch.equal(plan.spmm(db.OP_AT, wide), again)      # what the graph writes is not the wider call's
        assert torch.equal(plan.spmm(db.OP_AT, x), want)
        del junk
    del graph
    plan.close()


@pytest.mark.parametrize("n,degree,f", [(300000, 40, 180), (300000, 24, 232),       # X copied to rows on lines for its slices
                                        (300000, 24, 256), (200000, 30, 128),       # slices of X where it lies: by counts, and that fit L2
                                        (200000, 33, 127), (300000, 64, 159)])      # odd widths, whose copies run in slices
def test_same_bits_in_classes_under_capture_and_without_room(cuda_device, n, degree, f):
    """Calls that run in column slices: class by class, captured on a plan that has no copies yet, and where copies find no room
    the result has the bits of the whole, eager call."""
    make, gen = uniform_plan(cuda_device, n, degree, n + f)
    x = torch.randn((n, f), device=cuda_device, generator=gen)
    narrow = torch.randn((n, 9), device=cuda_device, generator=gen)
    plan, fresh = make(), make()
    for op in (db.OP_A, db.OP_AT):
        want = plan.spmm(op, x)
        assert plan.stats().last_slice_width == 64 and plan.stats().n_partials[op] == 0
        out, graph = torch.empty_like(x), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            fresh.spmm(op, x, out=out)
        graph.replay()
        assert torch.equal(out, want)
        del graph
        if f % 4:      # copies neither reserved nor made by the call
            bare = make()
            bare.reserve(f)
            assert torch.equal(bare.spmm(op, x), want)
            bare.close()
    for classes in (3, 16):
        row_class = torch.randint(0, classes, (n,), device=cuda_device, generator=gen, dtype=torch.int32)
        plan.set_row_classes(row_class, classes)
        for op in (db.OP_A, db.OP_AT):
            want, out = plan.spmm(op, x), torch.full_like(x, 7.0)
            plan.spmm(op, x, out=out, row_class=1)
            assert (out[row_class != 1] == 7.0).all()
            for c in (0, *range(2, classes)):
                plan.spmm(op, x, out=out, row_class=c)
            assert torch.equal(out, want)
    assert torch.equal(plan.spmm(db.OP_AT, narrow), fresh.spmm(db.OP_AT, narrow))


@pytest.mark.parametrize("n,degree,f,split", [(300000, 40, 180, False), (300000, 24, 256, False), (200000, 30, 128, False),
                                              (200000, 33, 127, False), (300000, 30, 256, True), (200000, 62, 255, True)])
def test_static_scratch_runs_in_the_same_slices(cuda_device, n, degree, f, split):
    """drone_spmm_static_scratch cuts the columns as drone_spmm does and gives its bits, before the plan has copies and after; with
    rows of many chunks, whose partial sums lie in the built-in array."""
    make, gen = uniform_plan(cuda_device, n, degree, n + f)
    if split:
        index = torch.full((n + 1,), degree, device=cuda_device, dtype=torch.int64)
        index[0], index[1], index[7] = 0, 10000, 900
        index = torch.cumsum(index, 0)
        nnz = int(index[-1])
        dst = torch.randint(0, n, (nnz,), device=cuda_device, generator=gen, dtype=torch.int32)
        val = torch.rand(nnz, device=cuda_device, generator=gen) - 0.5
        index = index.int()
        make = lambda: db.AggregationPlan(index, dst, values=val)
    x = torch.randn((n, f), device=cuda_device, generator=gen)
    plan, fresh = make(), make()
    for op in (db.OP_A, db.OP_AT):
        want = plan.spmm(op, x)
        assert plan.stats().last_slice_width == 64 and (plan.stats().n_partials[db.OP_A] > 0) == split
        for p in (fresh, plan):
            out = torch.full_like(x, float("nan"))
            rc = db.lib().drone_spmm_static_scratch(p.handle, op, f, C.c_void_p(x.data_ptr()), f, C.c_void_p(out.data_ptr()), f,
                                                    C.c_void_p(torch.cuda.current_stream().cuda_stream))
            assert rc == 0, db.lib().drone_last_error()
            assert p.stats().last_slice_width == 64
            assert torch.equal(out, want)
    assert fresh.stats().scratch_bytes == 0


@pytest.mark.parametrize("f,width", [(16, 4), (32, 4), (32, 8), (48, 12), (60, 12), (32, 16)])
def test_forced_slices_narrower_than_a_short_rest(cuda_device, monkeypatch, f, width):
    """Forced slices of fewer than 16 columns are all of that width, the last one as well: partial sums have room for no more.  On
    a fresh plan, whose partial sums no wider call has made larger; each slice has the bits of a call on its own columns."""
    n, u, v = gg.rmat_graph(12, 16, seed=36, device=cuda_device, symmetrise=False, self_loops="add")
    index, dst = gg.csr_by_source(u, v, n)
    val = torch.rand(dst.numel(), device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(2)) - 0.5
    monkeypatch.setenv("DRONE_SLICE_WIDTH", str(width))
    sliced = db.AggregationPlan(index, dst, values=val)
    monkeypatch.setenv("DRONE_SLICE_WIDTH", "0")
    whole = db.AggregationPlan(index, dst, values=val)
    x = torch.randn((n, f), device=cuda_device, generator=torch.Generator(cuda_device).manual_seed(f))
    for op in (db.OP_A, db.OP_AT):
        partials = sliced.stats().n_partials[op]
        assert partials > 0
        got = sliced.spmm(op, x)
        assert sliced.stats().last_slice_width == width
        assert sliced.stats().scratch_bytes == 4 * width * max(partials, sliced.stats().n_partials[db.OP_A])
        for c0 in range(0, f, width):
            assert torch.equal(got[:, c0:c0 + width], whole.spmm(op, x[:, c0:c0 + width].contiguous()))


@pytest.mark.parametrize("n,per_row", [(8000, 200), (8000, 300), (100000, 31), (11000, 143),      # one launch: long rows, and not
                                       (100000, 190), (100000, 215), (40000, 1080), (400000, 53), (40000, 1590), (40000, 1700)])   # 20, 40 and 64 M
def test_narrow_widths_take_fewer_batches(cuda_device, n, per_row):
    """Widths of 1 to 8 where chunks take fewer batches of gathers at a time, and beside it, against double; the same bits for the
    rows class by class."""
    gen = torch.Generator(cuda_device).manual_seed(n + per_row)
    lengths = torch.randint(per_row * 9 // 10, per_row * 11 // 10 + 1, (n,), device=cuda_device, generator=gen)
    lengths[::97], lengths[1::97], lengths[5] = 3, 0, 5000
    index = torch.zeros(n + 1, dtype=torch.int64, device=cuda_device)
    torch.cumsum(lengths, 0, out=index[1:])
    nnz = int(index[-1])
    dst = torch.randint(0, n, (nnz,), device=cuda_device, generator=gen, dtype=torch.int32)
    val = torch.rand(nnz, device=cuda_device, generator=gen) - 0.5
    index = index.int()
    plan = db.AggregationPlan(index, dst, values=val, orientations=1)
    scale = torch.rand(n, device=cuda_device, generator=gen)
    row_class = torch.randint(0, 2, (n,), device=cuda_device, generator=gen, dtype=torch.int32)
    x = torch.randn((n, 8), device=cuda_device, generator=gen)
    plain = torch.sparse_csr_tensor(index.long(), dst.long(), val.double(), (n, n)) @ x.double()
    unit = (torch.sparse_csr_tensor(index.long(), dst.long(), torch.ones_like(val).double(), (n, n)) @ x.double()) * scale[:, None]
    results = {}
    for f in (1, 2, 4, 8):
        xf = x[:, :f].contiguous()
        got = results[f, 0] = plan.spmm(db.OP_A, xf)
        free = results[f, 1] = plan.spmm(db.OP_A, xf, unit_values=True, row_scale=scale)
        # float sums of up to 5000 terms of size 1, in pieces of at most 256
        for y, want in ((got, plain[:, :f]), (free, unit[:, :f])):
            assert (y - want).abs().max() <= 2e-5 * want.abs().max()
    plan.set_row_classes(row_class, 2)
    for (f, form), want in results.items():
        options = dict(unit_values=True, row_scale=scale) if form else {}
        out = torch.empty_like(want)
        for c in range(2):
            plan.spmm(db.OP_A, x[:, :f].contiguous(), out=out, row_class=c, **options)
        assert torch.equal(out, want)
