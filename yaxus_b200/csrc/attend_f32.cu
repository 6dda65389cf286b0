// Split-key attention over f32 caches (the reference's own cache type), in f32 on the CUDA cores.
//
// Same contract as the reference's `attn_split` (crates/yaxus-backend-gpu/src/shaders.rs:1466-1579): per item
// (rows, one KV head, a run of keys) the running maximum m, the sum of exponentials l and the unnormalised
// output o of every query head of the KV head's group.
//
// For passes that bring enough queries to the same keys (api.cu, f32_tiles_pay, says which those are).
// An item brings up to 64 queries (rows x heads of the group) to the same keys, and a tile of 32 keys is used for
// all of them out of shared memory: with one row an item, a prompt of 1000 rows read every key 1000 times and was
// bound by the shuffles of its dot products.  128 threads, two CTAs an SM: thread (ty, tx) of 8 x 16 holds rows
// ty * RT .. of the queries (RT = 8, 4 or 2 for 64, 32 or 16 of them) against keys tx and tx + 16, then the same
// rows' outputs for dims 4 tx .. and 64 + 4 tx ..  A row's probabilities stay inside half a warp, so they pass
// through shared memory without a barrier.  Products are packed pairs (fma.rn.f32x2): two products an issue slot.
// Rows of K, V and Q lie 132 floats apart, which spreads sixteen of them over all banks; a bulk copy each puts
// them there, two tiles in flight.
//
// Bound by the latencies of its own arithmetic at two warps a scheduler (FMA pipe half busy), not by memory.  A
// 1000-row prompt behind 1000 keys, 16 query / 4 KV heads, two layers: a whole step 5415 -> 1340 us.
// Sums are blocked by 32 dims and 32 keys, which costs 36 us of that: the error against 64 bits over 300 rows behind
// 1000 keys is 2.0e-7 with it, 4.0e-7 without, and 3.3e-7 for the kernel that takes a row at a time.
#include <type_traits>

#include "yx_device.cuh"

namespace yx {
namespace {

using namespace dev;

constexpr int THREADS = 128;
constexpr int KEYS = 32;                       // keys of a tile
constexpr int QUERIES = 64;                    // most queries of an item
constexpr int STRIDE = 132;                    // floats between rows of Q, K and V
constexpr int P_STRIDE = 36;
constexpr int TILE_FLOATS = KEYS * STRIDE;
constexpr int SMEM_BYTES = (QUERIES * STRIDE + 4 * TILE_FLOATS + QUERIES * P_STRIDE) * 4;   // Q, two stages of K and V, P
constexpr float LOG2E = 1.4426950408889634f;
constexpr float SCALE = 0.08838834764831845f;  // 1 / sqrt(128), the reference's f32 value

struct Params {
    const void *q;
    int q_dtype, hq, group, hkv;
    const char *k_arena, *v_arena;
    uint32_t kv_pages, window;
    const uint32_t *pos, *pages;
    const Item *items;
    const uint32_t *cta_begin;
    float *part_o, *part_ml;
    yx_dev_status *status;
};

struct Shared {
    uint64_t full[2], empty[2];
    int abort_flag;
    volatile int bad_page[2];
    uint32_t first[QUERIES], last[QUERIES];    // keys a query sees, inclusive
    uint32_t all_from, all_to;                 // keys every query sees
};

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t both(float x) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(x));
    return d;
}
__device__ __forceinline__ float2 halves(uint64_t x) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(x));
    return r;
}

// One item with RT query rows a thread.  `turn` counts the CTA's tiles: stage turn & 1, phase (turn >> 1) & 1.
template <int RT>
__device__ __forceinline__ void run_item(const Params &P, const Item &it, Shared &sh, float *s_q, float *s_kv, float *s_p, uint32_t &turn) {
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const uint32_t n_q = (uint32_t)it.n_rows * P.group;
    const uint32_t key_begin = max(it.key_lo, it.tile_begin * TILE_KEYS), key_end = min(it.key_hi, it.tile_end * TILE_KEYS - 1);   // inclusive
    const uint32_t t_begin = key_begin / KEYS, t_end = key_end / KEYS + 1;

    // Tile t (its keys in range) into stage `stage`, by the first warp: a bulk copy of 512 bytes a row.
    auto load = [&](uint32_t t, uint32_t stage) {
        const int lane = threadIdx.x;
        const uint32_t k0 = max(key_begin, t * KEYS), k1 = min(key_end, t * KEYS + KEYS - 1), n = k1 - k0 + 1;
        const uint32_t page = P.pages[it.pt_off + t * KEYS / PAGE], bar = smem_u32(&sh.full[stage]);
        const bool bad = page >= P.kv_pages;   // recorded, the copies are left out
        if (lane == 0) {
            if (bad && atomicCAS(&P.status->code, 0, 1) == 0) {
                P.status->where = 100;
                P.status->a = (int)page;
                P.status->b = (int)it.rows[0];
            }
            sh.bad_page[stage] = bad;
            mbar_expect_tx(bar, bad ? 0u : n * 1024u);
        }
        __syncwarp();
        if (bad || (uint32_t)lane >= n) return;
        const uint32_t key = k0 + lane, r = key % KEYS;
        const size_t at = kv_off32(page, P.hkv, it.kv_head, (int)(key % PAGE), 0) * 4;
        const uint32_t dst = smem_u32(s_kv + stage * 2 * TILE_FLOATS + r * STRIDE);
        bulk_g2s(dst, P.k_arena + at, 512, bar);
        bulk_g2s(dst + TILE_FLOATS * 4, P.v_arena + at, 512, bar);
    };

    if (threadIdx.x < 32) {
        load(t_begin, turn & 1u);
        if (t_begin + 1 < t_end) load(t_begin + 1, (turn + 1) & 1u);
    }
    for (int i = threadIdx.x; i < 8 * RT * 32; i += THREADS) {
        const uint32_t qi = i >> 5, c = (i & 31) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (qi < n_q) v = load4_as_f32(P.q, P.q_dtype, ((size_t)it.rows[qi / P.group] * P.hq + it.kv_head * P.group + qi % P.group) * D + c);
        *(float4 *)(s_q + qi * STRIDE + c) = v;
    }
    if (threadIdx.x < 32) {
        uint32_t from = 0, to = 0xffffffffu;
        for (uint32_t qi = threadIdx.x; qi < 8 * RT; qi += 32) {
            uint32_t lo = 1, hi = 0;                       // (a query past the item's sees nothing)
            if (qi < n_q) {
                const uint32_t p = P.pos[it.rows[qi / P.group]];
                lo = max(key_begin, P.window > 0 && p + 1 > P.window ? p + 1 - P.window : 0u);
                hi = min(key_end, p);
                from = max(from, lo);
                to = min(to, hi);
            }
            sh.first[qi] = lo;
            sh.last[qi] = hi;
        }
        __syncwarp();
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) {
            from = max(from, __shfl_xor_sync(0xffffffffu, from, d));
            to = min(to, __shfl_xor_sync(0xffffffffu, to, d));
        }
        if (threadIdx.x == 0) {
            sh.all_from = from;
            sh.all_to = to;
        }
    }
    __syncthreads();

    float m[RT], l[RT];
    uint64_t o[RT][4];
#pragma unroll
    for (int r = 0; r < RT; r++) {
        m[r] = -INFINITY;
        l[r] = 0.0f;
        o[r][0] = o[r][1] = o[r][2] = o[r][3] = 0ull;
    }
    const float *q_rows = s_q + ty * RT * STRIDE;
    float *p_rows = s_p + ty * RT * P_STRIDE;

    for (uint32_t t = t_begin; t < t_end; t++, turn++) {
        const uint32_t stage = turn & 1u;
        mbar_wait(smem_u32(&sh.full[stage]), (turn >> 1) & 1u, &sh.abort_flag, P.status, 101);
        __syncwarp();
        // The tile before this one is done with once the slowest warp is, and its stage filled again.
        if (threadIdx.x < 32 && t > t_begin && t + 1 < t_end) {
            mbar_wait(smem_u32(&sh.empty[stage ^ 1u]), ((turn - 1) >> 1) & 1u, &sh.abort_flag, P.status, 102);
            __syncwarp();
            load(t + 1, stage ^ 1u);
            __syncwarp();
        }
        const float *k = s_kv + stage * 2 * TILE_FLOATS, *v = k + TILE_FLOATS;
        if (!sh.bad_page[stage]) {   // (uniform over the CTA)
            // Scores of RT rows against keys tx and tx + 16: even dims in one half of the pair, odd ones in the other, 32 dims
            // at a time, so that no chain of rounded sums is longer than 16.
            uint64_t s2[RT][2];
#pragma unroll 1
            for (int d0 = 0; d0 < D; d0 += 32) {
                uint64_t part[RT][2];
#pragma unroll
                for (int d = 0; d < 32; d += 4) {
                    const ulonglong2 ka = *(const ulonglong2 *)(k + tx * STRIDE + d0 + d), kb = *(const ulonglong2 *)(k + (tx + 16) * STRIDE + d0 + d);
                    uint64_t q_hi[RT];
#pragma unroll
                    for (int r = 0; r < RT; r++) {
                        const ulonglong2 qv = *(const ulonglong2 *)(q_rows + r * STRIDE + d0 + d);
                        part[r][0] = d == 0 ? mul2(qv.x, ka.x) : fma2(qv.x, ka.x, part[r][0]);
                        part[r][1] = d == 0 ? mul2(qv.x, kb.x) : fma2(qv.x, kb.x, part[r][1]);
                        q_hi[r] = qv.y;
                    }
                    // (the other two dims only now: back to back, each would wait for the sum before it)
#pragma unroll
                    for (int r = 0; r < RT; r++) {
                        part[r][0] = fma2(q_hi[r], ka.y, part[r][0]);
                        part[r][1] = fma2(q_hi[r], kb.y, part[r][1]);
                    }
                }
#pragma unroll
                for (int r = 0; r < RT; r++) {
                    s2[r][0] = d0 == 0 ? part[r][0] : add2(s2[r][0], part[r][0]);
                    s2[r][1] = d0 == 0 ? part[r][1] : add2(s2[r][1], part[r][1]);
                }
            }
            // Every key of the tile live for every query: no masks.
            const bool edge = t * KEYS < sh.all_from || t * KEYS + KEYS - 1 > sh.all_to;
            const uint32_t key_a = t * KEYS + tx, key_b = key_a + 16;
            float rescale[RT];
#pragma unroll
            for (int r = 0; r < RT; r++) {
                const float2 a = halves(s2[r][0]), b = halves(s2[r][1]);
                const float sa = (a.x + a.y) * SCALE, sb = (b.x + b.y) * SCALE;
                bool live_a = true, live_b = true;
                if (edge) {
                    const uint32_t lo = sh.first[ty * RT + r], hi = sh.last[ty * RT + r];
                    live_a = key_a >= lo && key_a <= hi;
                    live_b = key_b >= lo && key_b <= hi;
                }
                float mx = fmaxf(live_a ? sa : -INFINITY, live_b ? sb : -INFINITY);
#pragma unroll
                for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
                const float mn = fmaxf(m[r], mx);
                const float f = m[r] == -INFINITY ? 0.0f : exp2f((m[r] - mn) * LOG2E);
                const float ea = live_a ? exp2f((sa - mn) * LOG2E) : 0.0f, eb = live_b ? exp2f((sb - mn) * LOG2E) : 0.0f;
                m[r] = mn;
                l[r] = l[r] * f + (ea + eb);
                rescale[r] = f;
                // (a masked key is marked, so that its V row, which may hold anything, is left out altogether)
                p_rows[r * P_STRIDE + tx] = live_a ? ea : -1.0f;
                p_rows[r * P_STRIDE + tx + 16] = live_b ? eb : -1.0f;
            }
            __syncwarp();
            // The tile's outputs are summed by themselves and then added to the rescaled ones before: chains of 32 keys.
            auto products = [&](auto masked) {
                uint64_t sum[RT][4];
#pragma unroll
                for (int r = 0; r < RT; r++) sum[r][0] = sum[r][1] = sum[r][2] = sum[r][3] = 0ull;
#pragma unroll 1
                for (int k4 = 0; k4 < KEYS; k4 += 4) {
                    float p[RT][4];
#pragma unroll
                    for (int r = 0; r < RT; r++) *(float4 *)p[r] = *(const float4 *)(p_rows + r * P_STRIDE + k4);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const ulonglong2 va = *(const ulonglong2 *)(v + (k4 + j) * STRIDE + tx * 4), vb = *(const ulonglong2 *)(v + (k4 + j) * STRIDE + 64 + tx * 4);
#pragma unroll
                        for (int r = 0; r < RT; r++) {
                            if (decltype(masked)::value && p[r][j] < 0.0f) continue;
                            const uint64_t pp = both(p[r][j]);
                            sum[r][0] = fma2(pp, va.x, sum[r][0]);
                            sum[r][1] = fma2(pp, va.y, sum[r][1]);
                            sum[r][2] = fma2(pp, vb.x, sum[r][2]);
                            sum[r][3] = fma2(pp, vb.y, sum[r][3]);
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < RT; r++) {
                    const uint64_t f = both(rescale[r]);
#pragma unroll
                    for (int c = 0; c < 4; c++) o[r][c] = fma2(o[r][c], f, sum[r][c]);
                }
            };
            if (edge) products(std::true_type{});
            else products(std::false_type{});
        }
        __syncwarp();
        if ((threadIdx.x & 31) == 0) mbar_arrive(smem_u32(&sh.empty[stage]));
    }

#pragma unroll
    for (int r = 0; r < RT; r++) {
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) l[r] += __shfl_xor_sync(0xffffffffu, l[r], w);
        const uint32_t qi = ty * RT + r;
        if (qi < n_q) {
            const size_t slot = (size_t)it.part[qi / P.group] * P.group + qi % P.group;
            float *dst = P.part_o + slot * D + tx * 4;
            *(ulonglong2 *)dst = make_ulonglong2(o[r][0], o[r][1]);
            *(ulonglong2 *)(dst + 64) = make_ulonglong2(o[r][2], o[r][3]);
            if (tx == 0) {
                // An item without a live key for this row: the reference's empty mark.
                P.part_ml[slot * 2] = m[r] == -INFINITY && l[r] == 0.0f ? -1e30f : m[r];
                P.part_ml[slot * 2 + 1] = l[r];
            }
        }
        __syncwarp();
    }
}

__global__ void __launch_bounds__(THREADS, 2) attend_f32_kernel(const Params P) {
    extern __shared__ __align__(128) float smem[];
    __shared__ Shared sh;
    __shared__ Item item_s;
    float *s_q = smem, *s_kv = s_q + QUERIES * STRIDE, *s_p = s_kv + 4 * TILE_FLOATS;
    if (threadIdx.x == 0) {
        sh.abort_flag = 0;
        mbar_init(smem_u32(&sh.full[0]), 1);
        mbar_init(smem_u32(&sh.full[1]), 1);
        mbar_init(smem_u32(&sh.empty[0]), THREADS / 32);
        mbar_init(smem_u32(&sh.empty[1]), THREADS / 32);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    dependent_entry();
    const uint32_t begin = P.cta_begin[blockIdx.x], end = P.cta_begin[blockIdx.x + 1];
    uint32_t turn = 0;
    for (uint32_t i = begin; i < end; i++) {
        __syncthreads();   // the item before is through with everything in shared memory
        if (threadIdx.x < sizeof(Item) / 16) ((uint4 *)&item_s)[threadIdx.x] = ((const uint4 *)(P.items + i))[threadIdx.x];
        __syncthreads();
        const uint32_t n_q = (uint32_t)item_s.n_rows * P.group;
        if (n_q <= 16) run_item<2>(P, item_s, sh, s_q, s_kv, s_p, turn);
        else if (n_q <= 32) run_item<4>(P, item_s, sh, s_q, s_kv, s_p, turn);
        else run_item<8>(P, item_s, sh, s_q, s_kv, s_p, turn);
    }
    __syncthreads();
    if (sh.abort_flag)
        for (int i = 0; i < 64; i++) __nanosleep(1000);   // copies in flight come to rest
}

}  // namespace

int launch_attend_f32(yx_ctx *ctx, const AttendArgs &a) {
    if (!ctx->smem_configured[8]) {
        if (int rc = check_cuda(ctx, cudaFuncSetAttribute(attend_f32_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES),
                                "attend_f32: shared memory attribute"))
            return rc;
        ctx->smem_configured[8] = true;
    }
    Params P{};
    P.q = a.q;
    P.q_dtype = a.q_dtype;
    P.hq = a.hq;
    P.group = a.group;
    P.hkv = a.hkv;
    P.k_arena = a.k_arena;
    P.v_arena = a.v_arena;
    P.kv_pages = a.kv_pages;
    P.window = (uint32_t)(a.window > 0 ? a.window : 0);
    P.pos = ctx->d_pos;
    P.pages = ctx->d_pages;
    P.items = a.items;
    P.cta_begin = a.cta_begin;
    P.part_o = a.part_o;
    P.part_ml = a.part_ml;
    P.status = ctx->dev_status;
    return launch_dependent(ctx, "attend_f32 kernel launch", attend_f32_kernel, dim3((unsigned)a.n_ctas), dim3(THREADS), SMEM_BYTES, P);
}

}  // namespace yx
