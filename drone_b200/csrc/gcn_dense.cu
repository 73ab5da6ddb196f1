// The element-wise steps beside the aggregation of a graph-convolution model: softmax cross-entropy with its gradient
// (CUDACrossEntropyLoss::forward, cuda_gcn/src/cuda/cuda_kernel.cu:326-370) and the mask of a ReLU's gradient
// (CUDAReLU::backward, cuda_module.cu:513-523).
//
// As a dozen and a half element-wise launches the loss read and wrote the logits about ten times, at 5 us of host work a
// launch; here a group of lanes holds a row in registers.  Bound: HBM, one read of the logits and one write of the gradient, and
// with few rows the two launches.
#include "common.cuh"

#include <algorithm>

#include "../../include/drone_b200.h"

namespace drone {

constexpr int kLossBlocks = DRONE_LOSS_SCRATCH / 2;

template <int L>
__device__ __forceinline__ float lanes_max(float v) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
template <int L>
__device__ __forceinline__ float lanes_sum(float v) {
#pragma unroll
    for (int o = L / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Rows of at most L * PER classes (PER > 0), L lanes a row with PER values each in registers; PER == 0: of any number, read three
// times.  block_sums[b] = {sum of the labelled rows' losses, number of labelled rows} of block b, in a fixed order.
template <int L, int PER>
__global__ void __launch_bounds__(256) softmax_loss_kernel(const float *__restrict__ logits, long long ld, const long long *__restrict__ truth,
                                                           const unsigned char *__restrict__ labelled, int n, int classes,
                                                           float *__restrict__ grad, long long ld_grad, double2 *block_sums) {
    const int gl = threadIdx.x & (L - 1);
    double loss = 0, count = 0;
    const int rows_at_once = (int)(gridDim.x * blockDim.x) / L;
    for (int row0 = (int)(blockIdx.x * blockDim.x + threadIdx.x) / L; row0 - (int)(threadIdx.x & 31) / L < n; row0 += rows_at_once) {
        const bool live = row0 < n;      // whole warps stay for the shuffles
        const int row = live ? row0 : n - 1;
        const float *x = logits + (long long)row * ld;
        float *g = grad + (long long)row * ld_grad;
        const long long t = __ldg(truth + row);
        // a class that does not exist: nothing plausible comes out
        const float mask = t < 0 || t >= classes ? NAN : __ldg(labelled + row) ? 1.f : 0.f;
        constexpr int REGS = PER > 0 ? PER : 1;
        float v[REGS], m = -INFINITY, s = 0, at_truth = 0;
        if (PER > 0) {
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                v[u] = gl + u * L < classes ? __ldg(x + gl + u * L) : -INFINITY;
                m = fmaxf(m, v[u]);
            }
        } else {
            for (int c = gl; c < classes; c += L) m = fmaxf(m, __ldg(x + c));
        }
        m = lanes_max<L>(m);
        if (PER > 0) {
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                const int c = gl + u * L;
                if (c < classes) {
                    if (c == t) at_truth = v[u];
                    v[u] = expf(v[u] - m);
                    s += v[u];
                }
            }
        } else {
            for (int c = gl; c < classes; c += L) {
                const float e = __ldg(x + c);
                if (c == t) at_truth = e;
                s += expf(e - m);
            }
        }
        s = lanes_sum<L>(s);
        at_truth = lanes_sum<L>(at_truth);
        if (live) {
            if (PER > 0) {
#pragma unroll
                for (int u = 0; u < PER; ++u) {
                    const int c = gl + u * L;
                    if (c < classes) g[c] = (v[u] / s - (c == t ? 1.f : 0.f)) * mask;
                }
            } else {
                for (int c = gl; c < classes; c += L) g[c] = (expf(__ldg(x + c) - m) / s - (c == t ? 1.f : 0.f)) * mask;
            }
            if (gl == 0) {
                loss += (double)((logf(s) - (at_truth - m)) * mask);
                count += mask;
            }
        }
    }
    __shared__ double2 of_warp[8];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        loss += __shfl_down_sync(0xffffffffu, loss, o);
        count += __shfl_down_sync(0xffffffffu, count, o);
    }
    if ((threadIdx.x & 31) == 0) of_warp[threadIdx.x >> 5] = make_double2(loss, count);
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) {
            loss += of_warp[w].x;
            count += of_warp[w].y;
        }
        block_sums[blockIdx.x] = make_double2(loss, count);
    }
}

__global__ void __launch_bounds__(256) fold_loss_kernel(const double2 *block_sums, int blocks, float *out) {
    __shared__ double2 sm[256];
    double2 mine = make_double2(0, 0);
    for (int i = threadIdx.x; i < blocks; i += 256) {
        mine.x += block_sums[i].x;
        mine.y += block_sums[i].y;
    }
    sm[threadIdx.x] = mine;
    for (int o = 128; o > 0; o >>= 1) {
        __syncthreads();
        if ((int)threadIdx.x < o) {
            sm[threadIdx.x].x += sm[threadIdx.x + o].x;
            sm[threadIdx.x].y += sm[threadIdx.x + o].y;
        }
    }
    if (threadIdx.x == 0) *out = (float)(sm[0].x / fmax(sm[0].y, 1.0));
}

// grad = grad * (out > 0), V = float4 or float
__device__ __forceinline__ float masked(float g, float z) { return g * (z > 0.f ? 1.f : 0.f); }
__device__ __forceinline__ float4 masked(const float4 &g, const float4 &z) {
    return make_float4(masked(g.x, z.x), masked(g.y, z.y), masked(g.z, z.z), masked(g.w, z.w));
}
template <typename V>
__global__ void __launch_bounds__(256) relu_mask_kernel(V *__restrict__ grad, long long ld, const V *__restrict__ out, long long ld_out,
                                                        int n, int width) {
    const long long first = blockIdx.x * (long long)blockDim.x + threadIdx.x, step = (long long)gridDim.x * blockDim.x;
    for (RowColumn at(first, step, width); at.row < n; at.advance()) {
        V *g = grad + (long long)at.row * ld + at.col;
        *g = masked(*g, __ldg(out + (long long)at.row * ld_out + at.col));
    }
}

template <int L, int PER>
static int launch_loss(const float *logits, int ld, const long long *truth, const unsigned char *labelled, int n, int classes, float *grad,
                       int ld_grad, float *loss, double *scratch, cudaStream_t st) {
    const int blocks = std::max(1, (int)std::min<long long>(kLossBlocks, ((long long)n * L + 255) / 256));
    if (n > 0) {
        softmax_loss_kernel<L, PER><<<blocks, 256, 0, st>>>(logits, ld, truth, labelled, n, classes, grad, ld_grad, (double2 *)scratch);
        DRONE_LAUNCH_CHECK("softmax_loss_kernel");
    }
    fold_loss_kernel<<<1, 256, 0, st>>>((const double2 *)scratch, n > 0 ? blocks : 0, loss);
    DRONE_LAUNCH_CHECK("fold_loss_kernel");
    return DRONE_OK;
}

}  // namespace drone

using namespace drone;

extern "C" {

int drone_softmax_loss(int n_rows, int classes, const float *d_logits, int ld, const long long *d_truth, const unsigned char *d_labelled,
                       float *d_grad, int ld_grad, float *d_loss, double *d_scratch, void *stream) {
    DRONE_REQUIRE(n_rows >= 0 && classes >= 1 && ld >= classes && ld_grad >= classes,
                  "drone_softmax_loss: n_rows=%d classes=%d ld=%d ld_grad=%d", n_rows, classes, ld, ld_grad);
    DRONE_REQUIRE(d_loss && d_scratch && (n_rows == 0 || (d_logits && d_truth && d_labelled && d_grad)), "drone_softmax_loss: NULL argument");
    DRONE_REQUIRE((reinterpret_cast<uintptr_t>(d_scratch) & 15) == 0, "drone_softmax_loss: d_scratch is not 16-byte aligned");
    cudaStream_t st = (cudaStream_t)stream;
#define DRONE_LOSS(L, PER) launch_loss<L, PER>(d_logits, ld, d_truth, d_labelled, n_rows, classes, d_grad, ld_grad, d_loss, d_scratch, st)
    if (classes <= 8) return DRONE_LOSS(8, 1);
    if (classes <= 16) return DRONE_LOSS(8, 2);
    if (classes <= 32) return DRONE_LOSS(8, 4);
    if (classes <= 64) return DRONE_LOSS(8, 8);
    if (classes <= 256) return DRONE_LOSS(32, 8);
    return DRONE_LOSS(32, 0);
#undef DRONE_LOSS
}

int drone_relu_mask(int n_rows, int F, float *d_grad, int ld_grad, const float *d_out, int ld_out, void *stream) {
    DRONE_REQUIRE(n_rows >= 0 && F >= 1 && ld_grad >= F && ld_out >= F, "drone_relu_mask: n_rows=%d F=%d ld_grad=%d ld_out=%d", n_rows, F,
                  ld_grad, ld_out);
    if (n_rows == 0) return DRONE_OK;
    DRONE_REQUIRE(d_grad && d_out, "drone_relu_mask: NULL argument");
    cudaStream_t st = (cudaStream_t)stream;
    const bool vec4 = F % 4 == 0 && ld_grad % 4 == 0 && ld_out % 4 == 0 &&
                      ((reinterpret_cast<uintptr_t>(d_grad) | reinterpret_cast<uintptr_t>(d_out)) & 15) == 0;
    const int width = vec4 ? F / 4 : F;
    const int grid = (int)std::min<long long>(((long long)n_rows * width + 255) / 256, 148 * 16);
    if (vec4) relu_mask_kernel<<<grid, 256, 0, st>>>((float4 *)d_grad, ld_grad / 4, (const float4 *)d_out, ld_out / 4, n_rows, width);
    else relu_mask_kernel<<<grid, 256, 0, st>>>(d_grad, ld_grad, d_out, ld_out, n_rows, width);
    DRONE_LAUNCH_CHECK("relu_mask_kernel");
    return DRONE_OK;
}

}  // extern "C"
