// The operators of the reference's `Backend` trait either side of attention
// (crates/yaxus-model/src/lib.rs:124-171), as the CPU backend computes them
// (crates/yaxus-backend-cpu/src/lib.rs:485-562): embedding gather, RMSNorm, the fused residual
// step, matmul against bf16 weights, SwiGLU, add, row gather, argmax.
//
// All of them are bandwidth-bound or a chain of latencies.  The one with real traffic, the matmul, is in
// matmul_tc.cu; here is its form for shapes that one does not take.
#include <cuda_bf16.h>
#include <string.h>

#include <algorithm>

#include "yx_device.cuh"

namespace yx {
namespace {

using namespace dev;

// Any shape the tensor-core kernel does not take (K not a multiple of 128): a warp per output, pass rows in the grid's y
// extent (a thread's number among all outputs' does not fit in 32 bits from 2^27 outputs on).
__global__ void matmul_any_kernel(const float *__restrict__ x, const __nv_bfloat16 *__restrict__ w, uint32_t N, uint32_t K,
                                  float *__restrict__ out) {
    const uint32_t n = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), t = blockIdx.y, lane = threadIdx.x & 31;
    if (n >= N) return;
    float s = 0.0f;
    for (uint32_t k = lane; k < K; k += 32) s += __bfloat162float(w[(size_t)n * K + k]) * x[(size_t)t * K + k];
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    if (lane == 0) out[(size_t)t * N + n] = s;
}

__global__ void swiglu_kernel(const float *__restrict__ x, uint32_t rows, uint32_t inner, float *__restrict__ out) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= (size_t)rows * inner) return;
    const size_t r = idx / inner, j = idx - r * inner;
    const float g = x[r * 2 * inner + j], u = x[r * 2 * inner + inner + j];
    out[idx] = g / (1.0f + expf(-g)) * u;
}

__global__ void add_assign_kernel(float *__restrict__ a, const float *__restrict__ b, size_t n) {
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx < n) a[idx] += b[idx];
}

// Up to this many row indices ride in kernel-parameter space; longer lists go through idx_dev.  The
// copy they replace (its call, the copy itself, the ordering after it) cost a decode step 5 us.
constexpr uint32_t PARAM_IDS = 512;
struct RowIds {
    const uint32_t *dev;   // null: use v
    uint32_t v[PARAM_IDS];
};

__device__ __forceinline__ void record_bad_row(yx_dev_status *status, int where, uint32_t id, uint32_t r) {
    if (atomicCAS(&status->code, 0, 1) == 0) {
        status->where = where;
        status->a = (int)id;
        status->b = (int)r;
    }
}

// out[r] = f32(table[ids[r]]) (cpu lib.rs:485-497); an id outside the table is recorded and its row zeroed.
// Latency-bound at decode: a CTA takes 2048 columns of a row, eight to a thread in one 16-byte load where the
// rows allow it (16 rows x 4096: 9.3 us with one scalar element at a time and a CTA per row).  A grid's y extent ends
// at 65535, so where a row has more parts than that a CTA takes several of them.
constexpr uint32_t EMBED_COLS = 2048;
dim3 gather_grid(uint32_t rows, uint32_t cols) { return dim3(rows, std::min((cols - 1) / EMBED_COLS + 1, 65535u)); }
template <bool VEC>
__global__ void __launch_bounds__(256) embed_kernel(const __nv_bfloat16 *__restrict__ table, uint32_t vocab, uint32_t h,
                                                    const __grid_constant__ RowIds ids, float *__restrict__ out, yx_dev_status *status) {
    dependent_entry();
    const uint32_t r = blockIdx.x, id = ids.dev ? ids.dev[r] : ids.v[r];
    const bool ok = id < vocab;
    if (!ok && threadIdx.x == 0 && blockIdx.y == 0) record_bad_row(status, 400, id, r);
    const __nv_bfloat16 *src = table + (size_t)(ok ? id : 0u) * h;
    float *dst = out + (size_t)r * h;
    for (size_t c0 = (size_t)blockIdx.y * EMBED_COLS; c0 < h; c0 += (size_t)gridDim.y * EMBED_COLS) {
        if constexpr (VEC) {
            const size_t c = c0 + threadIdx.x * 8;
            if (c >= h) return;
            const uint4 v = ok ? *(const uint4 *)(src + c) : make_uint4(0, 0, 0, 0);
            auto lo = [](uint32_t w) { return __uint_as_float(w << 16); };
            auto hi = [](uint32_t w) { return __uint_as_float(w & 0xffff0000u); };
            *(float4 *)(dst + c) = make_float4(lo(v.x), hi(v.x), lo(v.y), hi(v.y));
            *(float4 *)(dst + c + 4) = make_float4(lo(v.z), hi(v.z), lo(v.w), hi(v.w));
        } else {
            for (size_t c = c0 + threadIdx.x; c < min((size_t)h, c0 + EMBED_COLS); c += blockDim.x) dst[c] = ok ? __bfloat162float(src[c]) : 0.0f;
        }
    }
}

template <bool VEC>
__global__ void __launch_bounds__(256) select_rows_kernel(const float *__restrict__ x, uint32_t src_rows, uint32_t cols,
                                                          const __grid_constant__ RowIds ids, float *__restrict__ out,
                                                          yx_dev_status *status) {
    dependent_entry();
    const uint32_t r = blockIdx.x, src = ids.dev ? ids.dev[r] : ids.v[r];
    if (src >= src_rows) {
        if (threadIdx.x == 0 && blockIdx.y == 0) record_bad_row(status, 401, src, r);
        return;
    }
    const float *s = x + (size_t)src * cols;
    float *d = out + (size_t)r * cols;
    for (size_t c0 = (size_t)blockIdx.y * EMBED_COLS; c0 < cols; c0 += (size_t)gridDim.y * EMBED_COLS) {
        const size_t end = min((size_t)cols, c0 + EMBED_COLS);
        if constexpr (VEC) {
#pragma unroll
            for (uint32_t i = 0; i < EMBED_COLS / 1024; i++) {
                const size_t c = c0 + i * 1024 + threadIdx.x * 4;
                if (c < end) *(float4 *)(d + c) = *(const float4 *)(s + c);
            }
        } else {
            for (size_t c = c0 + threadIdx.x; c < end; c += blockDim.x) d[c] = s[c];
        }
    }
}

// Sum over the CTA (at most 16 warps); `scratch` is the caller's alone until the CTA's next barrier but one.
__device__ __forceinline__ float block_sum(float v, float *scratch) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(0xffffffffu, v, d);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, n_warps = blockDim.x >> 5;
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    float s = lane < n_warps ? scratch[lane] : 0.0f;
#pragma unroll
    for (int d = 8; d > 0; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    return __shfl_sync(0xffffffffu, s, 0);
}

// One CTA per row.  With `x_inout`: d = rmsnorm(delta, post); x += d; out = rmsnorm(x, pre)
// (crates/yaxus-model/src/lib.rs:149-162).  Without: out = rmsnorm(delta, post) (cpu lib.rs:296-302).
//
// A decode step has a handful of rows, so this is one SM's chain of latencies, not bandwidth: every
// operand is asked for at once, in 16-byte loads, and the row stays in registers between the two sums
// (V vectors of four a thread).  16 rows x 4096: 15.4 us when each pass over the row read it again.
template <int V, bool ADD>
__global__ void __launch_bounds__(512) norm_rows_kernel(float *__restrict__ x_inout, const float *__restrict__ delta,
                                                        const float *__restrict__ post_w, float post_offset,
                                                        const float *__restrict__ pre_w, float pre_offset, float eps, uint32_t cols,
                                                        float *__restrict__ out) {
    __shared__ float scratch[2][16];
    dependent_entry();
    const size_t base = (size_t)blockIdx.x * cols;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 d[V], pw[V], x[V], qw[V];
#pragma unroll
    for (int i = 0; i < V; i++) {
        const uint32_t c = (i * blockDim.x + threadIdx.x) * 4;
        const bool in = c < cols;
        d[i] = in ? *(const float4 *)(delta + base + c) : zero;
        if (ADD) x[i] = in ? *(const float4 *)(x_inout + base + c) : zero;
        pw[i] = in ? __ldg((const float4 *)(post_w + c)) : zero;
        if (ADD) qw[i] = in ? __ldg((const float4 *)(pre_w + c)) : zero;
    }
    float ss = 0.0f;
#pragma unroll
    for (int i = 0; i < V; i++) ss += d[i].x * d[i].x + d[i].y * d[i].y + d[i].z * d[i].z + d[i].w * d[i].w;
    const float r1 = 1.0f / sqrtf(block_sum(ss, scratch[0]) / (float)cols + eps);
    float ss2 = 0.0f;
#pragma unroll
    for (int i = 0; i < V; i++) {
        d[i] = make_float4((post_offset + pw[i].x) * (d[i].x * r1), (post_offset + pw[i].y) * (d[i].y * r1),
                           (post_offset + pw[i].z) * (d[i].z * r1), (post_offset + pw[i].w) * (d[i].w * r1));
        const uint32_t c = (i * blockDim.x + threadIdx.x) * 4;
        if (ADD) {
            x[i] = make_float4(x[i].x + d[i].x, x[i].y + d[i].y, x[i].z + d[i].z, x[i].w + d[i].w);
            if (c < cols) {
                *(float4 *)(x_inout + base + c) = x[i];
                ss2 += x[i].x * x[i].x + x[i].y * x[i].y + x[i].z * x[i].z + x[i].w * x[i].w;
            }
        } else if (c < cols) {
            *(float4 *)(out + base + c) = d[i];
        }
    }
    if constexpr (ADD) {
        const float r2 = 1.0f / sqrtf(block_sum(ss2, scratch[1]) / (float)cols + eps);
#pragma unroll
        for (int i = 0; i < V; i++) {
            const uint32_t c = (i * blockDim.x + threadIdx.x) * 4;
            if (c < cols)
                *(float4 *)(out + base + c) = make_float4((pre_offset + qw[i].x) * (x[i].x * r2), (pre_offset + qw[i].y) * (x[i].y * r2),
                                                          (pre_offset + qw[i].z) * (x[i].z * r2), (pre_offset + qw[i].w) * (x[i].w * r2));
        }
    }
}

// The same for rows that are no multiple of four wide, wider than 8192, or unaligned.
__global__ void __launch_bounds__(256) norm_any_kernel(float *__restrict__ x_inout, const float *__restrict__ delta,
                                                       const float *__restrict__ post_w, float post_offset,
                                                       const float *__restrict__ pre_w, float pre_offset, float eps, uint32_t cols,
                                                       float *__restrict__ out) {
    __shared__ float scratch[2][16];
    dependent_entry();
    const size_t base = (size_t)blockIdx.x * cols;
    float ss = 0.0f;
    for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
        const float v = delta[base + c];
        ss += v * v;
    }
    const float r1 = 1.0f / sqrtf(block_sum(ss, scratch[0]) / (float)cols + eps);
    if (!x_inout) {
        for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) out[base + c] = (post_offset + post_w[c]) * (delta[base + c] * r1);
        return;
    }
    float ss2 = 0.0f;
    for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) {
        const float v = x_inout[base + c] + (post_offset + post_w[c]) * (delta[base + c] * r1);
        x_inout[base + c] = v;
        ss2 += v * v;
    }
    const float r2 = 1.0f / sqrtf(block_sum(ss2, scratch[1]) / (float)cols + eps);
    for (uint32_t c = threadIdx.x; c < cols; c += blockDim.x) out[base + c] = (pre_offset + pre_w[c]) * (x_inout[base + c] * r2);
}

int launch_norm(yx_ctx *ctx, float *x_inout, const float *delta, const float *post_w, float post_offset, const float *pre_w,
                float pre_offset, float eps, uint32_t rows, uint32_t cols, float *out) {
    const uintptr_t all = (uintptr_t)x_inout | (uintptr_t)delta | (uintptr_t)post_w | (uintptr_t)pre_w | (uintptr_t)out;
    ctx->last_launch = yx_ctx::LAST_OTHER;
    auto go = [&](auto kernel, unsigned threads) {
        return launch_dependent(ctx, "norm kernel launch", kernel, dim3(rows), dim3(threads), 0, x_inout, delta, post_w, post_offset, pre_w,
                                pre_offset, eps, cols, out);
    };
    if (cols % 4 != 0 || cols > 8192 || (all & 15u) != 0) return go(norm_any_kernel, 256);
    // The fewest threads that hold the row in one or two vectors each: a barrier among 512 is cheaper than among
    // 1024, and rows of up to 1024 leave half of those idle.
    const bool add = x_inout != nullptr;
    if (cols <= 1024) return add ? go(norm_rows_kernel<1, true>, 256) : go(norm_rows_kernel<1, false>, 256);
    if (cols <= 2048) return add ? go(norm_rows_kernel<1, true>, 512) : go(norm_rows_kernel<1, false>, 512);
    if (cols <= 4096) return add ? go(norm_rows_kernel<2, true>, 512) : go(norm_rows_kernel<2, false>, 512);
    return add ? go(norm_rows_kernel<4, true>, 512) : go(norm_rows_kernel<4, false>, 512);
}

// The first largest value of each row; NaNs never win, a row of NaNs gives 0 (cpu lib.rs:430-441).
//
// A row of a vocabulary is 100 to 600 KB, and a greedy step has one to a few rows: one CTA per row left
// 147 SMs idle (28 us for one row of 32000, 42 us for one of 50257).  Here a row is cut into parts of
// ARGMAX_COLS, a CTA each, with all of a thread's loads in flight at once; the row's last CTA to finish
// (a counter in global scratch, which it leaves at zero) takes the best of the parts.  The result goes
// straight to mapped host memory: the read-back is the stream's completion, with no copy behind it.
constexpr uint32_t ARGMAX_COLS = 2048;
struct Best {
    float v;
    uint32_t i;   // 0xffffffff: nothing above -inf seen
};
__device__ __forceinline__ Best better(Best a, Best b) { return b.v > a.v || (b.v == a.v && b.i < a.i) ? b : a; }
__device__ __forceinline__ Best best_of_cta(Best b, Best *scratch) {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1)
        b = better(b, Best{__shfl_xor_sync(0xffffffffu, b.v, d), __shfl_xor_sync(0xffffffffu, b.i, d)});
    if ((threadIdx.x & 31) == 0) scratch[threadIdx.x >> 5] = b;
    __syncthreads();
    b = scratch[0];
    for (int i = 1; i < (int)(blockDim.x >> 5); i++) b = better(b, scratch[i]);
    return b;
}

__global__ void __launch_bounds__(256) argmax_rows_kernel(const float *__restrict__ x, uint32_t cols, Best *__restrict__ parts,
                                                          uint32_t *__restrict__ counters, uint32_t *out) {
    __shared__ Best scratch[2][8];
    __shared__ bool last;
    dependent_entry();
    const float *row = x + (size_t)blockIdx.y * cols;
    const uint32_t n_parts = gridDim.x, c0 = blockIdx.x * ARGMAX_COLS;
    float v[ARGMAX_COLS / 256];
#pragma unroll
    for (uint32_t j = 0; j < ARGMAX_COLS / 256; j++) {
        const uint32_t c = c0 + j * 256 + threadIdx.x;
        v[j] = c < cols ? row[c] : -INFINITY;
    }
    Best b{-INFINITY, 0xffffffffu};
#pragma unroll
    for (uint32_t j = 0; j < ARGMAX_COLS / 256; j++)
        if (v[j] > b.v) b = Best{v[j], c0 + j * 256 + threadIdx.x};
    b = best_of_cta(b, scratch[0]);
    if (n_parts > 1) {
        Best *mine = parts + (size_t)blockIdx.y * n_parts;
        if (threadIdx.x == 0) {
            __stcg((float2 *)(mine + blockIdx.x), make_float2(b.v, __uint_as_float(b.i)));
            __threadfence();
            last = atomicAdd(counters + blockIdx.y, 1u) + 1 == n_parts;
        }
        __syncthreads();
        if (!last) return;
        __threadfence();
        b = Best{-INFINITY, 0xffffffffu};
        for (uint32_t p = threadIdx.x; p < n_parts; p += blockDim.x) {
            const float2 e = __ldcg((const float2 *)(mine + p));
            b = better(b, Best{e.x, __float_as_uint(e.y)});
        }
        b = best_of_cta(b, scratch[1]);
        if (threadIdx.x == 0) counters[blockIdx.y] = 0u;
    }
    if (threadIdx.x == 0) out[blockIdx.y] = b.i == 0xffffffffu ? 0u : b.i;
}

int launched(yx_ctx *ctx, const char *what) {
    ctx->launches++;
    ctx->last_launch = yx_ctx::LAST_OTHER;
    return check_cuda(ctx, cudaGetLastError(), what);
}

struct Guard {
    int prev = -1;
    explicit Guard(int dev) {
        cudaGetDevice(&prev);
        if (prev != dev) cudaSetDevice(dev);
        else prev = -1;
    }
    ~Guard() {
        if (prev >= 0) cudaSetDevice(prev);
    }
};

int ready(yx_ctx *ctx) {
    if (!ctx) return YX_ERR_INVALID;
    return ctx->status;
}

int matmul_impl(yx_ctx *ctx, const float *x, const void *w_bf16, uint32_t T, uint32_t N, uint32_t K, int glu, float *out) {
    if (int rc = ready(ctx)) return rc;
    if (T == 0 || N == 0) return YX_OK;
    if (!x || !w_bf16 || !out || K == 0) return fail(ctx, YX_ERR_INVALID, "matmul: null tensor or empty inner dimension");
    if (glu && N % 2 != 0) return fail(ctx, YX_ERR_INVALID, "matmul_glu: the weight must hold gate and up rows (even N)");
    Guard guard(ctx->device);
    const __nv_bfloat16 *w = (const __nv_bfloat16 *)w_bf16;
    const uint32_t cols = glu ? N / 2 : N;
    const bool tensor = K % 128 == 0 && ((uintptr_t)w & 15u) == 0 && ((uintptr_t)x & 7u) == 0;
    if (tensor && (!glu || cols % 16 == 0)) return launch_matmul_tc(ctx, x, w, T, N, K, glu != 0, out);
    float *dst = out;
    if (glu) {
        // (room for 32 rows at least: see matmul_few_rows)
        if (int rc = ensure_buffer(ctx, (void **)&ctx->mm_sums, &ctx->mm_sums_cap, (size_t)std::max(T, 32u) * N * sizeof(float))) return rc;
        dst = ctx->mm_sums;
    }
    if (tensor) {
        if (int rc = launch_matmul_tc(ctx, x, w, T, N, K, false, dst)) return rc;
    } else {
        for (uint32_t t0 = 0; t0 < T; t0 += 65535u) {   // (the y extent's end)
            matmul_any_kernel<<<dim3(N / 8 + 1, std::min(T - t0, 65535u)), 256, 0, ctx->stream>>>(x + (size_t)t0 * K, w, N, K, dst + (size_t)t0 * N);
            if (int rc = launched(ctx, "matmul kernel (any shape)")) return rc;
        }
    }
    if (!glu) return YX_OK;
    const uint64_t n = (uint64_t)T * cols;
    swiglu_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(dst, T, cols, out);
    return launched(ctx, "swiglu kernel");
}

}  // namespace

}  // namespace yx

using namespace yx;

extern "C" {

int yx_matmul(yx_ctx *ctx, const float *x_dev, const void *w_bf16_dev, uint32_t rows, uint32_t n, uint32_t k, float *out_dev) {
    return matmul_impl(ctx, x_dev, w_bf16_dev, rows, n, k, 0, out_dev);
}

int yx_matmul_glu(yx_ctx *ctx, const float *x_dev, const void *w_bf16_dev, uint32_t rows, uint32_t n, uint32_t k,
                  float *out_dev) {
    return matmul_impl(ctx, x_dev, w_bf16_dev, rows, n, k, 1, out_dev);
}

int yx_swiglu(yx_ctx *ctx, const float *x_dev, uint32_t rows, uint32_t inner, float *out_dev) {
    if (int rc = ready(ctx)) return rc;
    const uint64_t n = (uint64_t)rows * inner;
    if (n == 0) return YX_OK;
    if (!x_dev || !out_dev) return fail(ctx, YX_ERR_INVALID, "swiglu: null tensor");
    Guard guard(ctx->device);
    swiglu_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(x_dev, rows, inner, out_dev);
    return launched(ctx, "swiglu kernel");
}

int yx_add_assign(yx_ctx *ctx, float *a_dev, const float *b_dev, size_t n) {
    if (int rc = ready(ctx)) return rc;
    if (n == 0) return YX_OK;
    if (!a_dev || !b_dev) return fail(ctx, YX_ERR_INVALID, "add_assign: null tensor");
    Guard guard(ctx->device);
    add_assign_kernel<<<(unsigned)((n + 255) / 256), 256, 0, ctx->stream>>>(a_dev, b_dev, n);
    return launched(ctx, "add_assign kernel");
}

int yx_rmsnorm(yx_ctx *ctx, const float *x_dev, const float *w_dev, uint32_t rows, uint32_t cols, float offset, float eps,
               float *out_dev) {
    if (int rc = ready(ctx)) return rc;
    if (rows == 0) return YX_OK;
    if (!x_dev || !w_dev || !out_dev || cols == 0) return fail(ctx, YX_ERR_INVALID, "rmsnorm: null tensor or no columns");
    Guard guard(ctx->device);
    return launch_norm(ctx, nullptr, x_dev, w_dev, offset, nullptr, 0.0f, eps, rows, cols, out_dev);
}

int yx_add_norm(yx_ctx *ctx, float *x_dev, const float *delta_dev, const float *post_w_dev, float post_offset,
                const float *pre_w_dev, float pre_offset, float eps, uint32_t rows, uint32_t cols, float *out_dev) {
    if (int rc = ready(ctx)) return rc;
    if (rows == 0) return YX_OK;
    if (!x_dev || !delta_dev || !post_w_dev || !pre_w_dev || !out_dev || cols == 0)
        return fail(ctx, YX_ERR_INVALID, "add_norm: null tensor or no columns");
    Guard guard(ctx->device);
    return launch_norm(ctx, x_dev, delta_dev, post_w_dev, post_offset, pre_w_dev, pre_offset, eps, rows, cols, out_dev);
}

// The row indices of a gather, checked against `limit` (already done by the caller): in the kernel's
// parameters where they fit, else uploaded.
static int row_ids(yx_ctx *ctx, const uint32_t *host, uint32_t n, RowIds &ids) {
    ids.dev = nullptr;
    if (n <= PARAM_IDS) {
        memcpy(ids.v, host, (size_t)n * 4);
        return YX_OK;
    }
    if (int rc = ensure_buffer(ctx, (void **)&ctx->idx_dev, &ctx->idx_cap, (size_t)n * 4)) return rc;
    ids.dev = ctx->idx_dev;
    return upload_ordered(ctx, ctx->idx_dev, host, (size_t)n * 4);
}

int yx_embed(yx_ctx *ctx, const void *table_bf16_dev, uint32_t vocab, uint32_t h, const uint32_t *ids_host, uint32_t rows,
             float *out_dev) {
    if (int rc = ready(ctx)) return rc;
    if (rows == 0) return YX_OK;
    if (!table_bf16_dev || !ids_host || !out_dev || h == 0) return fail(ctx, YX_ERR_INVALID, "embed: null tensor");
    for (uint32_t r = 0; r < rows; r++)
        if (ids_host[r] >= vocab) return fail(ctx, YX_ERR_INVALID, "embed: a token id is outside the table");
    Guard guard(ctx->device);
    RowIds ids;
    if (int rc = row_ids(ctx, ids_host, rows, ids)) return rc;
    const bool vec = h % 8 == 0 && (((uintptr_t)table_bf16_dev | (uintptr_t)out_dev) & 15u) == 0;
    ctx->last_launch = yx_ctx::LAST_OTHER;
    return launch_dependent(ctx, "embed kernel launch", vec ? embed_kernel<true> : embed_kernel<false>,
                            gather_grid(rows, h), dim3(256), 0, (const __nv_bfloat16 *)table_bf16_dev, vocab, h, ids,
                            out_dev, ctx->dev_status);
}

int yx_select_rows(yx_ctx *ctx, const float *x_dev, uint32_t src_rows, uint32_t cols, const uint32_t *rows_host, uint32_t n,
                   float *out_dev) {
    if (int rc = ready(ctx)) return rc;
    if (n == 0 || cols == 0) return YX_OK;
    if (!x_dev || !rows_host || !out_dev) return fail(ctx, YX_ERR_INVALID, "select_rows: null tensor");
    for (uint32_t r = 0; r < n; r++)
        if (rows_host[r] >= src_rows) return fail(ctx, YX_ERR_INVALID, "select_rows: a row index is outside the tensor");
    Guard guard(ctx->device);
    RowIds ids;
    if (int rc = row_ids(ctx, rows_host, n, ids)) return rc;
    const bool vec = cols % 4 == 0 && (((uintptr_t)x_dev | (uintptr_t)out_dev) & 15u) == 0;
    ctx->last_launch = yx_ctx::LAST_OTHER;
    return launch_dependent(ctx, "select_rows kernel launch", vec ? select_rows_kernel<true> : select_rows_kernel<false>,
                            gather_grid(n, cols), dim3(256), 0, x_dev, src_rows, cols, ids, out_dev,
                            ctx->dev_status);
}

int yx_argmax_rows(yx_ctx *ctx, const float *logits_dev, uint32_t rows, uint32_t cols, uint32_t *out_host) {
    if (int rc = ready(ctx)) return rc;
    if (rows == 0) return YX_OK;
    if (!logits_dev || !out_host || cols == 0) return fail(ctx, YX_ERR_INVALID, "argmax_rows: null tensor or no columns");
    Guard guard(ctx->device);
    const uint32_t n_parts = (cols + ARGMAX_COLS - 1) / ARGMAX_COLS;
    if (rows > ctx->pick_cap) {
        // The counters start at zero and every launch leaves them there; the picks are pinned host memory.
        if (int rc = check_cuda(ctx, cudaStreamSynchronize(ctx->stream), "argmax_rows: sync before growing")) return rc;
        if (ctx->pick_counters) cudaFree(ctx->pick_counters);
        if (ctx->pick_host) cudaFreeHost(ctx->pick_host);
        ctx->pick_counters = ctx->pick_host = nullptr;
        ctx->pick_cap = 0;
        const size_t want = std::max<size_t>(64, (size_t)rows + rows / 2);
        if (int rc = check_cuda(ctx, cudaMalloc((void **)&ctx->pick_counters, want * 4), "argmax_rows: counters")) return rc;
        if (int rc = check_cuda(ctx, cudaMemsetAsync(ctx->pick_counters, 0, want * 4, ctx->stream), "argmax_rows: counters")) return rc;
        if (int rc = check_cuda(ctx, cudaHostAlloc((void **)&ctx->pick_host, want * 4, cudaHostAllocMapped), "argmax_rows: result")) return rc;
        ctx->pick_cap = want;
    }
    if (int rc = ensure_buffer(ctx, (void **)&ctx->idx_dev, &ctx->idx_cap, (size_t)rows * n_parts * sizeof(Best))) return rc;
    ctx->last_launch = yx_ctx::LAST_OTHER;
    // (a grid's y extent ends at 65535)
    for (uint32_t r0 = 0; r0 < rows; r0 += 65535u) {
        const uint32_t n = std::min(rows - r0, 65535u);
        if (int rc = launch_dependent(ctx, "argmax_rows kernel launch", argmax_rows_kernel, dim3(n_parts, n), dim3(256), 0,
                                      logits_dev + (size_t)r0 * cols, cols, (Best *)ctx->idx_dev + (size_t)r0 * n_parts,
                                      ctx->pick_counters + r0, ctx->pick_host + r0))
            return rc;
    }
    // A read-back: the one place the model waits for the device (crates/yaxus-model/src/lib.rs:177-185).
    if (int rc = yx_sync(ctx)) return rc;
    memcpy(out_host, ctx->pick_host, (size_t)rows * 4);
    return YX_OK;
}

}  // extern "C"
