"""Host-side mirror of the reference's GCN step around the aggregation path (CUDAGCN::forward / backward,
cuda_gcn/src/cuda/cuda_gcn.cu:44-83,119-170), for any number of layers.  Only the GraphSum layers, the masking of
mirror rows, the loss, the ReLU's gradient, the weight gradients and the weight broadcast / gradient reduce are this library's
kernels and NCCL calls; the other products of the dense layers stay on cuBLAS (torch.matmul).  Used to time an epoch and to check gradients end to end.

Layer l = 1..L:  H_l = A_{l-1} · W_l  (Matmul)  ->  Z_l = Â^T-aggregation of H_l + mirror/master sync (GraphSum)
                 ->  A_l = ReLU(Z_l) for l < L, logits = Z_L.
The reference's module list is this with L = 2 (cuda_gcn.cu:44-83); its layer interface allows more.
"""
import ctypes as C

import torch

from ._lib import LOSS_SCRATCH, OP_A, OP_AT, check, lib
from .graphsum import aggregate_and_exchange, clear_mirror_rows, exchange_sum


class GCN:
    """forward + backward of [Matmul -> GraphSum -> ReLU] x (L-1) -> Matmul -> GraphSum -> cross-entropy on one rank.

    weights: list of L tensors [d_{l-1}, d_l].
    aggregate(op, x, out, relu): the sparse aggregation (default: graph.plan.spmm with the ReLU done in the store
    when fuse_relu is set); sync(rows): the mirror/master exchange (default: over `comm` when worker_num > 1).
    With fuse_relu = False the ReLU runs as its own pass, as CUDAReLU::forward does (cuda_module.cu:498-511)."""

    def __init__(self, graph, x, truth, weights, comm=None, worker_num=1, aggregate=None, fuse_relu=True, sync=None):
        self.g, self.x, self.truth = graph, x, truth
        self.weights = list(weights)
        self.n_layers = len(self.weights)
        self.comm, self.worker_num = comm, worker_num
        self.fuse_relu = bool(fuse_relu) and aggregate is None
        self.aggregate = aggregate or (lambda op, src, out, relu=False: graph.plan.spmm(op, src, out=out, relu=relu))
        self._custom_aggregate = aggregate is not None
        self._sync = sync
        n, dev = x.shape[0], x.device
        dims = [w.shape[1] for w in self.weights]
        self.h = [torch.empty((n, d), device=dev) for d in dims]        # Matmul outputs
        self.z = [torch.empty((n, d), device=dev) for d in dims]        # GraphSum outputs (after ReLU for l < L)
        self.d_h = [torch.empty((n, d), device=dev) for d in dims]      # gradients w.r.t. the Matmul outputs
        self.d_a = [torch.empty((n, d), device=dev) for d in dims[:-1]] # gradients w.r.t. the ReLU outputs (masked in place)
        self.mirror2worker = graph.mirror2worker if worker_num > 1 else None
        # element-wise steps: one kernel each on the GPU, torch elsewhere
        self._kernels = x.is_cuda and all(t.dtype == torch.float32 for t in (x, *self.weights))
        self.labelled = truth >= 0
        self.safe_truth = truth.clamp(min=0).long()
        if self._kernels:
            self._scratch = torch.empty(LOSS_SCRATCH, dtype=torch.float64, device=dev)
            self._shares = {}
        self.d_w = [None] * self.n_layers
        self.loss = None

    @property
    def safe_truth(self):
        return self._safe_truth

    @safe_truth.setter
    def safe_truth(self, classes):
        """The rows' classes, also where they are not labelled.  They are looked at when they are set: torch would stop the step
        at one that does not exist, the kernel makes the loss NaN (as it does when the tensor is changed in place)."""
        most = self.weights[-1].shape[1]
        if self._kernels and classes.numel() > 0 and not torch.cuda.is_current_stream_capturing():
            least, largest = (int(t) for t in classes.aminmax())
            if least < 0 or largest >= most:
                raise ValueError("a label is outside 0..%d" % (most - 1))
        self._safe_truth = classes

    # ----- pieces -----
    def sync(self, rows):
        if self._sync is not None:
            self._sync(rows)
        elif self.worker_num > 1:
            exchange_sum(self.g.xplan, self.comm, rows)

    def _aggregate_and_sync(self, op, src, out):
        """GraphSum of one layer and direction: aggregation + mirror/master sync.  With the library's own aggregation
        and its peer-memory transport the two are one fused sequence (mirror rows leave from the aggregation's
        store); with a custom aggregation or sync they run one after the other."""
        if not self._custom_aggregate and self._sync is None and self.worker_num > 1:
            aggregate_and_exchange(self.g.plan, self.g.xplan, self.comm, op, src, out)
            return out
        self._aggregate(op, src, out)
        self.sync(out)
        return out

    def _aggregate(self, op, src, out, relu=False):
        if self._custom_aggregate:
            self.aggregate(op, src, out)
            if relu:
                out.clamp_(min=0)
        else:
            self.aggregate(op, src, out, relu)
        return out

    def broadcast_weights(self):
        """weight_broadcast_value_nccl at the start of every forward pass (cuda_communicate.cu:99-105)."""
        if self.worker_num > 1:
            for w in self.weights:
                self.comm.bcast(w, root=0)

    def reduce_gradients(self):
        """weight_reduce_grad_nccl after the backward pass (cuda_communicate.cu:107-115): sums land on rank 0."""
        if self.worker_num > 1:
            for dw in self.d_w:
                self.comm.reduce_sum(dw, root=0)

    # ----- the step -----
    def forward(self):
        a = self.x
        last = self.n_layers - 1
        for l, w in enumerate(self.weights):
            torch.matmul(a, w, out=self.h[l])                              # CUDAMatmul::forward
            relu = l < last
            # The mirror/master sync adds partial sums, so the ReLU can sit in the aggregation's store only when there
            # is nothing to add afterwards (one worker); with several workers it follows the sync.
            fused = relu and self.fuse_relu and self.worker_num == 1 and self._sync is None
            if fused:
                self._aggregate(OP_AT, self.h[l], self.z[l], relu=True)    # CUDAGraphSum::forward + CUDAReLU::forward
            else:
                self._aggregate_and_sync(OP_AT, self.h[l], self.z[l])      # CUDAGraphSum::forward with its sync
            if relu and not fused:
                self.z[l].clamp_(min=0)                                    # CUDAReLU::forward, in place
            a = self.z[l]
        return self._softmax_loss(self.z[last])

    def _stream(self):
        return torch._C._cuda_getCurrentRawStream(self.x.device.index)

    def _call(self, name, *args):
        """A library call on the model's device."""
        if torch.cuda.current_device() == self.x.device.index:
            check(getattr(lib(), name)(*args))
        else:
            with torch.cuda.device(self.x.device):
                check(getattr(lib(), name)(*args))

    def _per_row(self, t, dtype, n):
        """Whether t is one value of this type a row, side by side on the model's device."""
        return t.dtype == dtype and t.shape == (n,) and t.device == self.x.device and t.is_contiguous()

    def _float_matrix(self, t):
        """Whether t is a matrix of floats on the model's device."""
        return t.dtype == torch.float32 and t.dim() == 2 and t.device == self.x.device

    def _softmax_loss(self, logits):
        """CUDACrossEntropyLoss::forward: loss = mean over labelled rows; gradient not divided by the count."""
        n, classes = logits.shape
        if (self._kernels and self._float_matrix(logits) and logits.is_contiguous() and self._per_row(self.labelled, torch.bool, n)
                and self._per_row(self.safe_truth, torch.int64, n)):
            self.d_logits, self.loss = torch.empty_like(logits), torch.empty((), dtype=torch.float32, device=logits.device)
            self._call("drone_softmax_loss", n, classes, logits.data_ptr(), classes, self.safe_truth.data_ptr(),
                       self.labelled.data_ptr(), self.d_logits.data_ptr(), classes, self.loss.data_ptr(), self._scratch.data_ptr(),
                       self._stream())
            return self.loss
        zmax = logits.max(dim=1, keepdim=True).values
        e = torch.exp(logits - zmax)
        s = e.sum(dim=1, keepdim=True)
        self.d_logits = e / s
        picked = logits.gather(1, self.safe_truth.unsqueeze(1))
        per_row = (torch.log(s) - (picked - zmax)).squeeze(1)
        count = self.labelled.sum().clamp(min=1)
        self.loss = (per_row * self.labelled).sum() / count
        self.d_logits.scatter_add_(1, self.safe_truth.unsqueeze(1), -torch.ones_like(picked))
        self.d_logits.mul_(self.labelled.unsqueeze(1))
        return self.loss

    def _relu_mask(self, grad, out):
        if not (self._kernels and grad.shape == out.shape and all(self._float_matrix(t) and t.is_contiguous() for t in (grad, out))):
            return grad.mul_(out > 0)
        n, f = grad.shape
        self._call("drone_relu_mask", n, f, grad.data_ptr(), f, out.data_ptr(), f, self._stream())
        return grad

    def _weight_gradient(self, a, g):
        # what the kernel cannot read goes to torch, which computes or refuses it
        if not self._kernels or not all(self._float_matrix(t) for t in (a, g)) or a.shape[0] != g.shape[0]:
            return a.t() @ g
        (k, m), n = a.shape, g.shape[1]
        # rows one after the other: an expanded or overlapping input has none to step over
        in_rows = all(t.stride(1) == 1 and (k <= 1 or t.shape[1] <= t.stride(0) < 1 << 31) for t in (a, g))
        if not in_rows or min(m, n) == 0 or max(m, n) > 1 << 15 or k > 1 << 30:
            return a.t() @ g
        floats = self._shares.get((k, m, n))
        if floats is None:      # a property of the shape
            size = C.c_longlong(0)
            self._call("drone_weight_gradient_scratch", k, m, n, C.byref(size))
            floats = self._shares[(k, m, n)] = size.value
        out, parts = (torch.empty(shape, dtype=torch.float32, device=g.device) for shape in ((m, n), floats))
        lda, ldb = (t.stride(0) if k > 1 else t.shape[1] for t in (a, g))
        self._call("drone_weight_gradient", k, m, n, a.data_ptr(), lda, g.data_ptr(), ldb, out.data_ptr(),
                   parts.data_ptr(), floats, self._stream())
        return out

    def backward(self):
        g = self.d_logits
        for l in range(self.n_layers - 1, -1, -1):
            self._aggregate_and_sync(OP_A, g, self.d_h[l])                 # CUDAGraphSum::backward with its sync
            a_prev = self.z[l - 1] if l > 0 else self.x
            if l > 0:
                d_a = torch.matmul(self.d_h[l], self.weights[l].t(), out=self.d_a[l - 1])   # CUDAMatmul::backward: dA first ...
            if self.mirror2worker is not None:
                clear_mirror_rows(self.d_h[l], self.mirror2worker)         # ... clear_mirror_grad (in place) ...
            self.d_w[l] = self._weight_gradient(a_prev, self.d_h[l])       # ... then dW
            if l > 0:
                g = self._relu_mask(d_a, self.z[l - 1])                    # CUDAReLU::backward: the mask is (output > 0)
                if l == 1:
                    self.d_z1 = g
        return tuple(self.d_w)


class GCNStep(GCN):
    """The reference's own two-layer model, with the names its variables carry (cuda_gcn.cu:44-83)."""

    def __init__(self, graph, x, truth, w1, w2, comm=None, worker_num=1, aggregate=None, fuse_relu=True):
        super().__init__(graph, x, truth, [w1, w2], comm=comm, worker_num=worker_num, aggregate=aggregate,
                         fuse_relu=fuse_relu)

    w1 = property(lambda self: self.weights[0])
    w2 = property(lambda self: self.weights[1])
    h1 = property(lambda self: self.h[0])
    z1 = property(lambda self: self.z[0])
    h2 = property(lambda self: self.h[1])
    logits = property(lambda self: self.z[1])
    d_h1 = property(lambda self: self.d_h[0])
    d_h2 = property(lambda self: self.d_h[1])
    d_w1 = property(lambda self: self.d_w[0])
    d_w2 = property(lambda self: self.d_w[1])
