// hhp_blas1.cu -- BLAS-1 on device vectors: the reference's device_vector_dot / device_vector_scale /
// device_vector_axpy / device_vector_GPUtoGPU (src/util/hhp_cuda.c:163-202: cuBLAS Ddot, Dscal,
// Daxpy and a device-to-device copy), and the device-pointer-mode Ddot of the dp loop
// (src/entry/bicgstab_gpu_dp.c:163-190), on the context's stream.
//
// The dot product is deterministic (cuBLAS's is not guaranteed to be): each thread sums a fixed
// strided subset with fused multiply-adds, each block folds its threads in a fixed tree, and the
// block that finishes last (an atomic count; no block waits for another) adds the block partials
// in block order and stores the result. One launch; the partials live in context-owned scratch,
// so calls on one context are serialised on its stream.
#include <algorithm>

#include "hhp_device.cuh"
#include "hhp_internal.h"

namespace hhp {

namespace {

constexpr int kThreads = 256;
constexpr int kDotMaxBlocks = 1024;

// All kernels work on units of two consecutive elements, one 16-byte access where every vector starts
// on a 16-byte boundary (VEC), two 8-byte ones elsewhere; unit u belongs to the same thread either
// way, so the alignment changes no result. HBM bounds the long vectors: a thread keeps kUnits units of
// each in flight (64 KB per SM and vector at the dot's 2 blocks per SM). 16M elements, one 8-byte load
// in flight before: dot 72 -> 45 us (5.7 TB/s), axpy 78 -> 60 us (6.4 TB/s), scal 68 -> 48 us. Short
// ones are a chain of latencies and take one unit per thread on as many blocks as there are units.
constexpr int kUnits = 4;

template <bool VEC>
__device__ __forceinline__ double2 ld2(const double *p, long long u) {
    if (VEC) return __ldg(reinterpret_cast<const double2 *>(p) + u);
    return make_double2(__ldg(p + 2 * u), __ldg(p + 2 * u + 1));
}
// the same through an ordinary load: for a vector that the kernel also writes
template <bool VEC>
__device__ __forceinline__ double2 ldw2(const double *p, long long u) {
    if (VEC) return reinterpret_cast<const double2 *>(p)[u];
    return make_double2(p[2 * u], p[2 * u + 1]);
}
template <bool VEC>
__device__ __forceinline__ void st2(double *p, long long u, double2 v) {
    if (VEC) {
        reinterpret_cast<double2 *>(p)[u] = v;
    } else {
        p[2 * u] = v.x;
        p[2 * u + 1] = v.y;
    }
}

// fn(u) for units u0, u0 + stride, ... below nu, kUnits of them at a time: load(k, u) for each, then use.
template <typename Load, typename Use>
__device__ __forceinline__ void walk_units(long long u, long long stride, long long nu, Load load, Use use) {
    for (; u + (kUnits - 1) * stride < nu; u += kUnits * stride) {
#pragma unroll
        for (int k = 0; k < kUnits; ++k) load(k, u + k * stride);
#pragma unroll
        for (int k = 0; k < kUnits; ++k) use(k, u + k * stride);
    }
    for (; u < nu; u += stride) {
        load(0, u);
        use(0, u);
    }
}

// Sum over the block, in thread 0: a butterfly in every warp, one over the warps' sums.
__device__ __forceinline__ double block_total(double v, double *red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    v = warp_sum(v);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    v = threadIdx.x < kThreads / 32 ? red[threadIdx.x] : 0.0;
    if (warp == 0) {
#pragma unroll
        for (int o = kThreads / 64; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    }
    return v;
}

template <bool VEC>
__global__ void __launch_bounds__(kThreads, 4) k_dot(const double *__restrict__ x, const double *__restrict__ y,
                                                  long long n, double *part, unsigned *count, double *out) {
    __shared__ double red[kThreads / 32];
    __shared__ int last;
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    const long long u0 = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    double acc = 0.0;
    double2 a[kUnits], b[kUnits];
    walk_units(
        u0, stride, n / 2,
        [&](int k, long long u) {
            a[k] = ld2<VEC>(x, u);
            b[k] = ld2<VEC>(y, u);
        },
        [&](int k, long long) { acc = fma(a[k].y, b[k].y, fma(a[k].x, b[k].x, acc)); });
    if ((n & 1) && u0 == 0) acc = fma(__ldg(x + n - 1), __ldg(y + n - 1), acc);
    const double s = block_total(acc, red);
    if (threadIdx.x == 0) {
        part[blockIdx.x] = s;
        __threadfence();
        last = atomicAdd(count, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    double t = 0.0;
    for (unsigned i = threadIdx.x; i < gridDim.x; i += kThreads) t += __ldcg(part + i);
    t = block_total(t, red);
    if (threadIdx.x == 0) {
        *out = t;
        *count = 0u;  // ready for the next launch
    }
}

template <bool VEC>
__global__ void __launch_bounds__(kThreads) k_axpy(long long n, double alpha, const double *__restrict__ x, double *y) {
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    const long long u0 = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    double2 a[kUnits], b[kUnits];
    walk_units(
        u0, stride, n / 2,
        [&](int k, long long u) {
            a[k] = ld2<VEC>(x, u);
            b[k] = ldw2<VEC>(y, u);
        },
        [&](int k, long long u) { st2<VEC>(y, u, make_double2(fma(alpha, a[k].x, b[k].x), fma(alpha, a[k].y, b[k].y))); });
    if ((n & 1) && u0 == 0) y[n - 1] = fma(alpha, x[n - 1], y[n - 1]);
}

template <bool VEC>
__global__ void __launch_bounds__(kThreads) k_scal(long long n, double alpha, double *x) {
    const long long stride = static_cast<long long>(gridDim.x) * blockDim.x;
    const long long u0 = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
    double2 a[kUnits];
    walk_units(
        u0, stride, n / 2, [&](int k, long long u) { a[k] = ldw2<VEC>(x, u); },
        [&](int k, long long u) { st2<VEC>(x, u, make_double2(alpha * a[k].x, alpha * a[k].y)); });
    if ((n & 1) && u0 == 0) x[n - 1] = alpha * x[n - 1];
}

bool aligned16(const void *a, const void *b) {
    return (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) % 16 == 0;
}

// One unit per thread until the SMs hold `per_sm` blocks each (dot: 2, every block more is a partial
// more for the last one; 1M elements 8.3 us at 2, 10.3 us at 4. axpy, scal: 8).
int unit_grid(const hhp_ctx *ctx, long long n, int per_sm) {
    const long long units = (n + 1) / 2;
    return static_cast<int>(std::max(1LL, std::min<long long>((units + kThreads - 1) / kThreads, 1LL * per_sm * ctx->num_sms)));
}

hhp_status ensure_dot_scratch(hhp_ctx *ctx) {
    if (ctx->dot_part) return HHP_OK;
    if (cudaMalloc(&ctx->dot_part, sizeof(double) * kDotMaxBlocks) != cudaSuccess ||
        cudaMalloc(&ctx->dot_count, sizeof(unsigned)) != cudaSuccess ||
        cudaMemsetAsync(ctx->dot_count, 0, sizeof(unsigned), ctx->stream) != cudaSuccess) {
        set_error("dot: out of device memory for the partials");
        return HHP_ERR_OOM;
    }
    return HHP_OK;
}

hhp_status dot_launch(hhp_ctx *ctx, int n, const double *x, const double *y, double *out_dev) {
    if (!ctx || n < 0 || (n > 0 && (!x || !y)) || !out_dev) {
        set_error("dot: null argument or negative length");
        return HHP_ERR_ARG;
    }
    if (n == 0) {
        HHP_CUDA(cudaMemsetAsync(out_dev, 0, sizeof(double), ctx->stream));
        return HHP_OK;
    }
    HHP_TRY(ensure_dot_scratch(ctx));
    const int grid = std::min(unit_grid(ctx, n, 2), kDotMaxBlocks - 1);
    (aligned16(x, y) ? k_dot<true> : k_dot<false>)<<<grid, kThreads, 0, ctx->stream>>>(x, y, n, ctx->dot_part,
                                                                                      ctx->dot_count, out_dev);
    HHP_CUDA(cudaGetLastError());
    ctx->kernel_launches += 1;
    return HHP_OK;
}

}  // namespace

void release_blas1(hhp_ctx *ctx) {
    cudaFree(ctx->dot_part);
    cudaFree(ctx->dot_count);
    ctx->dot_part = nullptr;
    ctx->dot_count = nullptr;
}

}  // namespace hhp

using namespace hhp;

hhp_status hhp_dot_dev(hhp_ctx *ctx, int n, const double *x_dev, const double *y_dev, double *result_dev) {
    return dot_launch(ctx, n, x_dev, y_dev, result_dev);
}

hhp_status hhp_dot(hhp_ctx *ctx, int n, const double *x_dev, const double *y_dev, double *result) {
    if (!result) {
        set_error("dot: result is NULL");
        return HHP_ERR_ARG;
    }
    if (!ctx) {
        set_error("dot: null context");
        return HHP_ERR_ARG;
    }
    HHP_TRY(ensure_dot_scratch(ctx));
    double *slot = ctx->dot_part + (kDotMaxBlocks - 1);  // never a block partial: grids stay below
    HHP_TRY(dot_launch(ctx, n, x_dev, y_dev, slot));
    HHP_CUDA(cudaMemcpyAsync(result, slot, sizeof(double), cudaMemcpyDeviceToHost, ctx->stream));
    HHP_CUDA(cudaStreamSynchronize(ctx->stream));
    return HHP_OK;
}

hhp_status hhp_axpy_dev(hhp_ctx *ctx, int n, double alpha, const double *x_dev, double *y_dev) {
    if (!ctx || n < 0 || (n > 0 && (!x_dev || !y_dev))) {
        set_error("axpy: null argument or negative length");
        return HHP_ERR_ARG;
    }
    if (n == 0) return HHP_OK;
    (aligned16(x_dev, y_dev) ? k_axpy<true> : k_axpy<false>)<<<unit_grid(ctx, n, 8), kThreads, 0, ctx->stream>>>(
        n, alpha, x_dev, y_dev);
    HHP_CUDA(cudaGetLastError());
    ctx->kernel_launches += 1;
    return HHP_OK;
}

hhp_status hhp_scal_dev(hhp_ctx *ctx, int n, double alpha, double *x_dev) {
    if (!ctx || n < 0 || (n > 0 && !x_dev)) {
        set_error("scal: null argument or negative length");
        return HHP_ERR_ARG;
    }
    if (n == 0) return HHP_OK;
    (aligned16(x_dev, x_dev) ? k_scal<true> : k_scal<false>)<<<unit_grid(ctx, n, 8), kThreads, 0, ctx->stream>>>(
        n, alpha, x_dev);
    HHP_CUDA(cudaGetLastError());
    ctx->kernel_launches += 1;
    return HHP_OK;
}

hhp_status hhp_copy_dev(hhp_ctx *ctx, int n, const double *src_dev, double *dst_dev) {
    if (!ctx || n < 0 || (n > 0 && (!src_dev || !dst_dev))) {
        set_error("copy: null argument or negative length");
        return HHP_ERR_ARG;
    }
    if (n == 0) return HHP_OK;
    HHP_CUDA(cudaMemcpyAsync(dst_dev, src_dev, sizeof(double) * static_cast<size_t>(n), cudaMemcpyDeviceToDevice,
                             ctx->stream));
    return HHP_OK;
}
