// Weight gradients of a dense layer: C[M, N] = sum over k of A[k, :]^T B[k, :], A [K, M] the layer's input and B [K, N] the gradient
// of its output, with K (vertices) far above M and N (widths): CUDAMatmul::backward, cuda_gcn/src/cuda/cuda_module.cu:63-86.
//
// The result is a few tiles at most, so K is cut as well: every block adds an outer product a row over its share of the rows,
// one tile of C in registers, and a second kernel adds the shares in order.  All in float, a share's chain of additions being
// K / shares long, the shares added in double.  Bound: the FMA pipes (72 TFLOP/s) for wide layers, the two launches for small graphs.
// us with cuBLAS, which gives a tile to one block whatever K is / here, and the relative error of the result (2-norm): 232,965 x
// 602 x 128 842 / 767, 1.4e-6 / 1.1e-6; 232,965 x 128 x 41 361 / 117, 1.7e-6 / 5e-7; 100,000 x 602 x 128 401 / 341; 30,000 x 300 x 64
// 104 / 53; 3,000 x 16 x 7 49 / 18; 2.4 M x 100 x 256 3424 / 3180.
#include "common.cuh"

#include <algorithm>

#include "../../include/drone_b200.h"

namespace drone {

constexpr int kStepRows = 16;        // rows of A and B in shared memory at a time ...
constexpr int kStages = 3;           // ... of which this many are there or on their way

__device__ __forceinline__ void copy_async(float *shared, const float *global, bool live) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" :: "r"((unsigned)__cvta_generic_to_shared(shared)), "l"(global), "r"(live ? 4 : 0));
}

// Columns [col0, col0 + W) of rows [row0, row0 + kStepRows), 0 beyond the last row or column.  4 bytes a copy: rows of an odd
// width start anywhere.
template <int W>
__device__ __forceinline__ void copy_rows(float (*to)[W], const float *from, long long ld, int row0, int rows, int col0, int cols) {
    constexpr int ROWS = 256 / W;      // a thread stays in its column
    const int r = threadIdx.x / W, c = threadIdx.x % W;
    const bool in_row = col0 + c < cols;
    const float *at = from + (long long)(row0 + r) * ld + col0 + c;
#pragma unroll
    for (int u = 0; u < kStepRows; u += ROWS, at += ROWS * ld) {
        const bool live = in_row && row0 + r + u < rows;
        copy_async(&to[r + u][c], live ? at : from, live);
    }
}

// Two floats in a register pair: one instruction multiplies and adds both, each rounded as fmaf does.  (The scalar instruction
// reaches half the rate: 233,000 x 602 x 128 in 1083 us with it, 767 with this one.)
using Pair = unsigned long long;
__device__ __forceinline__ void fma_pair(Pair &acc, Pair a, Pair b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }
__device__ __forceinline__ Pair pair_of(float x) {
    Pair p;
    asm("mov.b64 %0, {%1, %1};" : "=l"(p) : "f"(x));
    return p;
}

template <int BM, int BN>
__global__ void __launch_bounds__(256, 2)
weight_gradient_kernel(const float *__restrict__ A, long long lda, const float *__restrict__ B, long long ldb, int M, int N, int K, int share,
                       float *__restrict__ out) {
    constexpr int TM = BM / 16, TN = BN / 16;
    struct Stage { float a[kStepRows][BM], b[kStepRows][BN]; };
    extern __shared__ __align__(16) char stage_bytes[];
    Stage *stage = reinterpret_cast<Stage *>(stage_bytes);
    const int tiles_n = (N + BN - 1) / BN, m0 = ((int)blockIdx.x / tiles_n) * BM, n0 = ((int)blockIdx.x % tiles_n) * BN;
    const int k0 = (int)blockIdx.y * share, k1 = min(K, k0 + share), steps = (k1 - k0 + kStepRows - 1) / kStepRows;
    const int tm = threadIdx.x / 16, tn = threadIdx.x % 16;
    Pair acc[TM][TN / 2];      // rows and columns of the tile in fours, 64 apart
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0;
    auto request = [&](int s) {
        if (s < steps) {
            copy_rows<BM>(stage[s % kStages].a, A, lda, k0 + s * kStepRows, k1, m0, M);
            copy_rows<BN>(stage[s % kStages].b, B, ldb, k0 + s * kStepRows, k1, n0, N);
        }
        asm volatile("cp.async.commit_group;");
    };
#pragma unroll
    for (int s = 0; s < kStages - 1; ++s) request(s);
#pragma unroll 1
    for (int s = 0; s < steps; ++s) {
        asm volatile("cp.async.wait_group %0;" :: "n"(kStages - 2));
        __syncthreads();      // step s has landed for everybody, and everybody has left the stage that is filled next
        request(s + kStages - 1);
        const Stage &now = stage[s % kStages];
#pragma unroll
        for (int k = 0; k < kStepRows; ++k) {
            Pair a[TM], b[TN / 2];
#pragma unroll
            for (int h = 0; h < TM / 4; ++h) {
                const float4 x = *reinterpret_cast<const float4 *>(now.a[k] + h * 64 + tm * 4);
                a[h * 4] = pair_of(x.x);
                a[h * 4 + 1] = pair_of(x.y);
                a[h * 4 + 2] = pair_of(x.z);
                a[h * 4 + 3] = pair_of(x.w);
            }
#pragma unroll
            for (int h = 0; h < TN / 4; ++h) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2 *>(now.b[k] + h * 64 + tn * 4);
                b[h * 2] = x.x;
                b[h * 2 + 1] = x.y;
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) fma_pair(acc[i][j], a[i], b[j]);
        }
    }
    asm volatile("cp.async.wait_group 0;");
    float *c = out + (long long)blockIdx.y * M * N;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + (i / 4) * 64 + tm * 4 + i % 4;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + (j / 4) * 64 + tn * 4 + j % 4;
            if (m < M && n < N) c[(long long)m * N + n] = __uint_as_float((unsigned)(acc[i][j / 2] >> (j & 1) * 32));
        }
    }
}

__global__ void __launch_bounds__(256) add_shares_kernel(const float *__restrict__ parts, int shares, int count, float *__restrict__ out) {
    for (int i = blockIdx.x * 256 + threadIdx.x; i < count; i += gridDim.x * 256) {
        double sum = 0;
#pragma unroll 8
        for (int s = 0; s < shares; ++s) sum += __ldg(parts + (long long)s * count + i);
        out[i] = (float)sum;
    }
}

struct GradientSplit {
    int bm, bn, tiles, shares, share;
};

// Two blocks an SM, but a share of at least 64 rows; tiles no wider than what they have to hold.
static GradientSplit split_gradient(int K, int M, int N, int sms) {
    GradientSplit s;
    s.bm = M <= 64 ? 64 : 128;
    s.bn = N <= 64 ? 64 : 128;
    if (s.bm == 64) s.bn = 64;
    s.tiles = ceil_div(M, s.bm) * ceil_div(N, s.bn);
    const int most = std::max(1, 2 * sms / s.tiles);
    s.share = std::max(64, ceil_div(ceil_div(K, most), kStepRows) * kStepRows);
    s.shares = std::max(1, ceil_div(K, s.share));
    return s;
}

template <int BM, int BN>
static int launch_gradient(const GradientSplit &s, const float *A, int lda, const float *B, int ldb, int M, int N, int K, float *out, cudaStream_t st) {
    constexpr size_t bytes = sizeof(float) * kStages * kStepRows * (BM + BN);
    weight_gradient_kernel<BM, BN><<<dim3(s.tiles, s.shares), 256, bytes, st>>>(A, lda, B, ldb, M, N, K, s.share, out);
    DRONE_LAUNCH_CHECK("weight_gradient_kernel");
    return DRONE_OK;
}

static int device_sms(int *sms) {
    int dev = 0;
    DRONE_CUDA(cudaGetDevice(&dev));
    DRONE_CUDA(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
    return DRONE_OK;
}

}  // namespace drone

using namespace drone;

extern "C" {

int drone_weight_gradient_scratch(int K, int M, int N, long long *n_floats) {
    DRONE_REQUIRE(K >= 0 && K <= 1 << 30 && M >= 1 && N >= 1 && M <= 1 << 15 && N <= 1 << 15 && n_floats, "drone_weight_gradient_scratch: K=%d M=%d N=%d", K, M, N);
    int sms = 0;
    const int rc = device_sms(&sms);
    if (rc) return rc;
    const GradientSplit s = split_gradient(K, M, N, sms);
    *n_floats = s.shares > 1 ? (long long)s.shares * M * N : 0;
    return DRONE_OK;
}

int drone_weight_gradient(int K, int M, int N, const float *d_A, int lda, const float *d_B, int ldb, float *d_C, float *d_scratch,
                          long long n_scratch, void *stream) {
    DRONE_REQUIRE(K >= 0 && K <= 1 << 30 && M >= 1 && N >= 1 && M <= 1 << 15 && N <= 1 << 15 && lda >= M && ldb >= N,
                  "drone_weight_gradient: K=%d M=%d N=%d lda=%d ldb=%d", K, M, N, lda, ldb);
    DRONE_REQUIRE(d_C && (K == 0 || (d_A && d_B)), "drone_weight_gradient: NULL argument");
    cudaStream_t st = (cudaStream_t)stream;
    if (K == 0) {
        DRONE_CUDA(cudaMemsetAsync(d_C, 0, sizeof(float) * (size_t)M * (size_t)N, st));
        return DRONE_OK;
    }
    int sms = 0, rc = device_sms(&sms);
    if (rc) return rc;
    const GradientSplit s = split_gradient(K, M, N, sms);
    const long long need = s.shares > 1 ? (long long)s.shares * M * N : 0;
    DRONE_REQUIRE(n_scratch >= need && (need == 0 || d_scratch), "drone_weight_gradient: %lld floats of scratch, %lld needed", n_scratch, need);
    float *out = s.shares > 1 ? d_scratch : d_C;
    rc = s.bm == 64 ? launch_gradient<64, 64>(s, d_A, lda, d_B, ldb, M, N, K, out, st)
         : s.bn == 64 ? launch_gradient<128, 64>(s, d_A, lda, d_B, ldb, M, N, K, out, st)
                      : launch_gradient<128, 128>(s, d_A, lda, d_B, ldb, M, N, K, out, st);
    if (rc || s.shares == 1) return rc;
    const int count = M * N;
    add_shares_kernel<<<std::min(ceil_div(count, 256), sms * 8), 256, 0, st>>>(d_scratch, s.shares, count, d_C);
    DRONE_LAUNCH_CHECK("add_shares_kernel");
    return DRONE_OK;
}

}  // extern "C"
