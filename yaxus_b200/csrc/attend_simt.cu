// Split-key attention on CUDA cores, for f32 KV storage (the reference's own cache type) and
// as a second, independent implementation the tensor-core kernel is checked against.
//
// Same contract as the reference's `attn_split` (crates/yaxus-backend-gpu/src/shaders.rs:1466-1579):
// per item (rows, one KV head, a run of keys) it emits, for every query head of the KV head's
// group, the running maximum m, the sum of exponentials l and the unnormalised output o.
// A CTA of four warps walks the items the planner gave it.  A warp takes every fourth key, eight of
// them in flight;
// a lane holds four of the 128 dims, so a K or V row is one coalesced 512-byte (f32) or
// 256-byte (16-bit) read per warp; the four warps' triples are merged in shared memory.
// K and V are read straight from global memory: each byte is used once per head chunk.  The parts of a row are
// merged by whichever of its CTAs comes last, without a launch of their own.
// Bound by issue slots and latencies, not yet by HBM: twelve sequences of 600 to 2500 keys on 4 f32 KV heads (77 MB)
// take 31 us, launch and merge included, where separate sums over the warp for every key and head and a merge kernel
// took 28 + 9 us with twice the exchanges (two layers: 109 -> 84 us); one sequence of 1024 keys 49 -> 43 us.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "yx_device.cuh"

namespace yx {
namespace {

constexpr int WARPS = 4;
constexpr int HC = 4;  // query heads per sweep over the keys
constexpr int KU = 8;  // keys a warp has in flight
constexpr float LOG2E = 1.4426950408889634f;

__device__ __forceinline__ float4 load4(const char *arena, int kv_dtype, uint32_t page, int hkv, int kvh, int tok,
                                        int lane) {
    int dim = lane * 4;
    if (kv_dtype == YX_F32) return *(const float4 *)((const float *)arena + kv_off32(page, hkv, kvh, tok, dim));
    uint2 raw = *(const uint2 *)((const uint16_t *)arena + kv_off16(page, hkv, kvh, tok, dim));
    float4 r;
    if (kv_dtype == YX_F16) {
        float2 a = __half22float2(*(const __half2 *)&raw.x), b = __half22float2(*(const __half2 *)&raw.y);
        r = make_float4(a.x, a.y, b.x, b.y);
    } else {
        float2 a = __bfloat1622float2(*(const __nv_bfloat162 *)&raw.x), b = __bfloat1622float2(*(const __nv_bfloat162 *)&raw.y);
        r = make_float4(a.x, a.y, b.x, b.y);
    }
    return r;
}

__device__ __forceinline__ float4 load_q4(const void *q, int q_dtype, size_t elem) {
    if (q_dtype == YX_F32) return *(const float4 *)((const float *)q + elem);
    uint2 raw = *(const uint2 *)((const uint16_t *)q + elem);
    if (q_dtype == YX_F16) {
        float2 a = __half22float2(*(const __half2 *)&raw.x), b = __half22float2(*(const __half2 *)&raw.y);
        return make_float4(a.x, a.y, b.x, b.y);
    }
    float2 a = __bfloat1622float2(*(const __nv_bfloat162 *)&raw.x), b = __bfloat1622float2(*(const __nv_bfloat162 *)&raw.y);
    return make_float4(a.x, a.y, b.x, b.y);
}

// The lanes whose bit `bit` is clear get a + their partner's a, the others b + their partner's b.
__device__ __forceinline__ float halve(float a, float b, int bit, int lane) {
    const bool upper = (lane & bit) != 0;
    return (upper ? b : a) + __shfl_xor_sync(0xffffffffu, upper ? a : b, bit);
}
// Where a call's merged rows go (any of out and the triple's three may be null), and what the merge needs.
struct RowMerge {
    const Merge *merges;
    uint32_t *counters;      // one per (row, KV head), zero between launches
    void *out;
    int out_dtype;
    float *m, *l, *o;
};

// The merge of combine.cu for one (row, query head), by a warp: lane c weighs part c, then all of them are added up in
// order, eight vectors asked for at once.  Every part of this kernel has been written, so empty ones (l <= 0) may be
// read; they are left out by their weight, whatever they hold.
__device__ __forceinline__ void merge_parts(const RowMerge &fin, const Merge &mg, const float *part_o, const float *part_ml, int g, int group,
                                            size_t idx, int lane) {
    float mx = -1e30f, l = 0.0f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (uint32_t c0 = 0; c0 < mg.count; c0 += 32) {
        const uint32_t nc = min(32u, mg.count - c0);
        float2 ml = make_float2(-1e30f, 0.0f);
        if ((uint32_t)lane < nc) ml = __ldcg((const float2 *)(part_ml + ((size_t)(mg.first + c0 + lane) * group + g) * 2));
        const bool live = ml.y > 0.0f;
        float cm = live ? ml.x : -1e30f;
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) cm = fmaxf(cm, __shfl_xor_sync(0xffffffffu, cm, off));
        const float nm = fmaxf(mx, cm), r = __expf(mx - nm), w = live ? __expf(ml.x - nm) : 0.0f;
        float ls = ml.y * w;   // (a sum that is no number has weight 0 and stays no number: the row shows it)
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) ls += __shfl_xor_sync(0xffffffffu, ls, off);
        l = l * r + ls;
        acc = make_float4(acc.x * r, acc.y * r, acc.z * r, acc.w * r);
        mx = nm;
        for (uint32_t j0 = 0; j0 < nc; j0 += 8) {
            float4 po[8];
#pragma unroll
            for (uint32_t j = 0; j < 8; j++)
                po[j] = j0 + j < nc ? __ldcg((const float4 *)(part_o + ((size_t)(mg.first + c0 + j0 + j) * group + g) * D + lane * 4)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) {
                const float wj = __shfl_sync(0xffffffffu, w, (int)((j0 + j) & 31u));
                if (j0 + j < nc && wj != 0.0f) acc = make_float4(acc.x + po[j].x * wj, acc.y + po[j].y * wj, acc.z + po[j].z * wj, acc.w + po[j].w * wj);
            }
        }
    }
    if (fin.out) {
        const float inv = 1.0f / l;   // a row always sees its own key, so l > 0 for whole attention
        dev::store4(fin.out, fin.out_dtype, idx * D + lane * 4, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
    }
    if (fin.o) {
        *(float4 *)(fin.o + idx * D + lane * 4) = acc;
        if (lane == 0) {
            fin.m[idx] = mx;
            fin.l[idx] = l;
        }
    }
}
static_assert(HC == 4 && KU == 8, "a lane ends up with one of 8 keys x 4 heads");

__global__ void __launch_bounds__(WARPS * 32, 4)
attend_simt_kernel(const void *__restrict__ q, int q_dtype, int hq, int group, const char *__restrict__ k_arena,
                   const char *__restrict__ v_arena, int hkv, int kv_dtype, uint32_t kv_pages, uint32_t window,
                   const uint32_t *__restrict__ pos, const uint32_t *__restrict__ pages, const Item *__restrict__ items,
                   const uint32_t *__restrict__ cta_begin, float *part_o, float *part_ml, const RowMerge fin, yx_dev_status *status) {
    __shared__ float sm_o[WARPS][HC][D];
    __shared__ float sm_ml[WARPS][HC][2];
    __shared__ __align__(16) float sm_e[WARPS][KU + 1][HC];
    __shared__ bool last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const float scale = 0.08838834764831845f;   // 1 / sqrt(128), the reference's f32 value
    dev::dependent_entry();
    const uint32_t ib = cta_begin[blockIdx.x], ie = cta_begin[blockIdx.x + 1];
    for (uint32_t ii = ib; ii < ie; ii++) {
        const Item it = items[ii];
        const int kvh = it.kv_head;
        for (int r = 0; r < it.n_rows; r++) {
            const uint32_t row = it.rows[r];
            const uint32_t p = pos[row];
            uint32_t lo = 0;
            if (window > 0 && p + 1 > window) lo = p + 1 - window;
            uint32_t k0 = max(max(lo, it.key_lo), it.tile_begin * TILE_KEYS);
            uint32_t k1 = min(min(p, it.key_hi), it.tile_end * TILE_KEYS - 1);   // inclusive
            for (int h0 = 0; h0 < group; h0 += HC) {
                float4 qv[HC];
                float4 o[HC];
                float m = -INFINITY, l = 0.0f;   // of head h0 + lane / 8; l over the keys lane % 8 of every round
#pragma unroll
                for (int g = 0; g < HC; g++) {
                    int hh = min(h0 + g, group - 1);
                    qv[g] = load_q4(q, q_dtype, ((size_t)row * hq + kvh * group + hh) * D + lane * 4);
                    o[g] = make_float4(0.f, 0.f, 0.f, 0.f);
                }
                // KU keys of this warp at a time: their page ids, then their K and V rows, are asked
                // for together, so a round costs two memory latencies instead of two per key.
                for (uint64_t key0 = (uint64_t)k0 + warp; key0 <= k1; key0 += (uint64_t)WARPS * KU) {
                    float4 kk[KU], vv[KU];
                    bool live[KU];
                    uint32_t page[KU];
#pragma unroll
                    for (int u = 0; u < KU; u++) {
                        const uint64_t key = key0 + (uint64_t)u * WARPS;
                        live[u] = key <= k1;
                        page[u] = live[u] ? pages[it.pt_off + (uint32_t)(key / PAGE)] : 0u;
                    }
                    uint32_t dead = 0;   // keys of the round that do not count
#pragma unroll
                    for (int u = 0; u < KU; u++) {
                        const uint64_t key = key0 + (uint64_t)u * WARPS;
                        if (live[u] && page[u] >= kv_pages) {   // recorded, the access is skipped
                            if (lane == 0 && atomicCAS(&status->code, 0, 1) == 0) {
                                status->where = 100;
                                status->a = (int)page[u];
                                status->b = (int)row;
                            }
                            live[u] = false;
                        }
                        kk[u] = vv[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                        if (live[u]) {
                            const int tok = (int)(key % PAGE);
                            kk[u] = load4(k_arena, kv_dtype, page[u], hkv, kvh, tok, lane);
                            vv[u] = load4(v_arena, kv_dtype, page[u], hkv, kvh, tok, lane);
                        } else {
                            dead |= 1u << u;
                        }
                    }
                    // KU x HC dot products over 32 lanes end with one in each lane, key lane % 8 of head lane / 8: at
                    // every step a lane hands half of what it holds to its partner and keeps the other half, 31 exchanges
                    // where a sum of each over all lanes takes 160.
                    float s[KU];
#pragma unroll
                    for (int u = 0; u < KU; u++) {
                        float d[HC];
#pragma unroll
                        for (int g = 0; g < HC; g++)
                            d[g] = qv[g].x * kk[u].x + qv[g].y * kk[u].y + qv[g].z * kk[u].z + qv[g].w * kk[u].w;
                        const float a = halve(d[0], d[2], 16, lane), b = halve(d[1], d[3], 16, lane);
                        s[u] = halve(a, b, 8, lane);
                    }
#pragma unroll
                    for (int u = 0; u < 4; u++) s[u] = halve(s[u], s[u + 4], 4, lane);
                    s[0] = halve(s[0], s[2], 2, lane);
                    s[1] = halve(s[1], s[3], 2, lane);
                    const float sc = halve(s[0], s[1], 1, lane) * scale;
                    const bool counts = ((dead >> (lane & 7)) & 1u) == 0;
                    float mx = counts ? sc : -INFINITY;
#pragma unroll
                    for (int off = 4; off > 0; off >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
                    const float mn = fmaxf(m, mx);
                    const float f = m == -INFINITY ? 0.0f : exp2f((m - mn) * LOG2E);
                    const float e = counts ? exp2f((sc - mn) * LOG2E) : 0.0f;
                    l = l * f + e;
                    m = mn;
                    // Back to every lane through shared memory: [key][head], the rescales behind them.
                    __syncwarp();
                    sm_e[warp][lane & 7][lane >> 3] = e;
                    if ((lane & 7) == 0) sm_e[warp][KU][lane >> 3] = f;
                    __syncwarp();
                    {
                        const float4 fs = *(const float4 *)sm_e[warp][KU];
                        const float fg[HC] = {fs.x, fs.y, fs.z, fs.w};
#pragma unroll
                        for (int g = 0; g < HC; g++) o[g] = make_float4(o[g].x * fg[g], o[g].y * fg[g], o[g].z * fg[g], o[g].w * fg[g]);
                    }
#pragma unroll
                    for (int u = 0; u < KU; u++) {
                        const float4 es = *(const float4 *)sm_e[warp][u];
                        const float eg[HC] = {es.x, es.y, es.z, es.w};
#pragma unroll
                        for (int g = 0; g < HC; g++) {
                            o[g].x += eg[g] * vv[u].x;
                            o[g].y += eg[g] * vv[u].y;
                            o[g].z += eg[g] * vv[u].z;
                            o[g].w += eg[g] * vv[u].w;
                        }
                    }
                }
#pragma unroll
                for (int off = 4; off > 0; off >>= 1) l += __shfl_xor_sync(0xffffffffu, l, off);
#pragma unroll
                for (int g = 0; g < HC; g++) *(float4 *)&sm_o[warp][g][lane * 4] = o[g];
                if ((lane & 7) == 0) {
                    sm_ml[warp][lane >> 3][0] = m;
                    sm_ml[warp][lane >> 3][1] = l;
                }
                __syncthreads();
                // Thread t merges dim t of the four warps' triples, head by head.
                const int t = threadIdx.x;
#pragma unroll
                for (int g = 0; g < HC; g++) {
                    if (h0 + g >= group) break;
                    float mx = -INFINITY;
#pragma unroll
                    for (int w = 0; w < WARPS; w++) mx = fmaxf(mx, sm_ml[w][g][0]);
                    float ls = 0.0f, acc = 0.0f;
#pragma unroll
                    for (int w = 0; w < WARPS; w++) {
                        float mw = sm_ml[w][g][0];
                        float f = mw == -INFINITY ? 0.0f : exp2f((mw - mx) * LOG2E);
                        ls += sm_ml[w][g][1] * f;
                        acc += sm_o[w][g][t] * f;
                    }
                    size_t slot = (size_t)it.part[r] * group + h0 + g;
                    __stcg(part_o + slot * D + t, acc);
                    // An item without a live key for this row: the reference's empty mark.
                    if (t == 0) __stcg((float2 *)(part_ml + slot * 2), make_float2(mx == -INFINITY ? -1e30f : mx, ls));
                }
                __syncthreads();
            }
            if (!fin.merges) continue;   // (measurement hook)
            // The last of a row and KV head's parts to be written merges them all, a warp to a query head.
            const Merge mg = fin.merges[(size_t)row * hkv + kvh];
            __threadfence();
            __syncthreads();
            if (threadIdx.x == 0) {
                uint32_t *counter = fin.counters + (size_t)row * hkv + kvh;
                last = mg.count == 1 || atomicAdd(counter, 1u) == mg.count - 1;
                if (last && mg.count > 1) *counter = 0u;
            }
            __syncthreads();
            if (last) {
                __threadfence();
                for (int g = warp; g < group; g += WARPS) merge_parts(fin, mg, part_o, part_ml, g, group, (size_t)row * hq + kvh * group + g, lane);
            }
            __syncthreads();   // (`last` is the next row's)
        }
    }
}

}  // namespace

int launch_attend_simt(yx_ctx *ctx, const AttendArgs &a, const Merge *merges) {
    const RowMerge fin{ctx->skip_merge ? nullptr : merges, a.counters, a.out, a.out_dtype, a.m_out, a.l_out, a.o_out};
    return launch_dependent(ctx, "attend_simt kernel launch", attend_simt_kernel, dim3((unsigned)a.n_ctas), dim3(WARPS * 32), 0, a.q, a.q_dtype,
                            a.hq, a.group, a.k_arena, a.v_arena, a.hkv, a.kv_dtype, a.kv_pages, (uint32_t)std::max<int64_t>(a.window, 0),
                            ctx->d_pos, ctx->d_pages, a.items, a.cta_begin, a.part_o, a.part_ml, fin, ctx->dev_status);
}

}  // namespace yx
