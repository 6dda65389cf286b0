// out [T, N] f32 = x [T, K] f32 . w [N, K]^T (bf16) for passes of many rows, on the fifth-generation
// tensor cores, and the same with silu(gate) * up taken in the epilogue (crates/yaxus-model/src/lib.rs:128,164-168).
//
// Activations keep 16 bits of mantissa: x = hi + lo, two bf16 matrices, and every weight tile that reaches
// shared memory is multiplied by both, into one f32 accumulator in tensor memory.  The arithmetic is twice
// that of a plain bf16 product; what a tile costs in weight traffic, accumulator reads and stores is not.
//
// The products are taken transposed, out^T = w x^T, by pairs of CTAs (cta_group::2): a tile is 256 weight
// rows (128 in each CTA) by up to 256 pass rows (half of them in each CTA), so a lane of tensor memory is a
// weight row, a warp's store of one pass row is one 128-byte line, and a pass of 33 rows fills the 256-row
// side as well as one of 2048 does.  A k step of 64 costs a CTA 16 KiB of weights and up to 32 KiB of
// activations for 2 x 256 x 256 x 64 multiply-adds: 32 bytes a clock and SM, half of what L2 delivers.
//
// Tiles are dealt to the pairs in whole rounds, pass rows fastest, so that the pairs that run together share
// weight rows and activations in L2.  What is left after the last whole round is cut along k into one equal
// share a pair (stream-K): such a share's sums go to scratch, and the CTA that comes last at a tile adds them
// up in order.  The shares come first in a pair's work, so that the adding up hides under whole tiles.  Adding up
// is a chain of L2 latencies: with one warp to a lane quarter and one share at a time it took 15 to 20 us.
//
// Large passes are bound by the tensor cores: 2048 rows on 4096 -> 28672 (gate and up) take 608 us, 1.58 PFLOP/s
// of bf16 products; 80 rows by the weights' way through L2 and shared memory: 412 MB in 100 us.  Against two
// library products (high part, then low part added to it) and a SwiGLU kernel, whole steps of one layer went from
// 2151 to 1700 us (2048 rows) and from 1244 to 399 us (80 rows).
//
// Warps 0-7 epilogue (two to each 32 lanes of tensor memory, taking turns at 32 pass rows), warp 8 TMA, warp 9
// issues the MMAs (first CTA of the pair).  All waits are bounded; on expiry the CTA records where, stops waiting
// anywhere, frees its tensor memory together with its partner and returns.
#include <cuda.h>

#include <algorithm>

#include "yx_tcgen05.cuh"

namespace yx {
namespace {

using namespace dev;

constexpr uint32_t TC_M = 256;              // weight rows of a pair's tile
constexpr uint32_t TC_KSTEP = 64;           // k of a stage: one 128-byte swizzled row
constexpr uint32_t TC_MAX_BT = 256;         // pass rows of a tile
constexpr int TC_MAX_STAGES = 12;
constexpr int TC_THREADS = 10 * 32;
constexpr int TC_TMA_WARP = 8, TC_MMA_WARP = 9;
constexpr uint32_t W_BYTES = 128 * 128;     // a CTA's share of a stage's weights
constexpr uint32_t TC_SMEM_BUDGET = 220 * 1024;
// k steps summed in tensor memory before the epilogue takes them over into its own f32 sums: the tensor core drops what
// lies below its accumulator's last place at each of a step's eight additions (see ROWS_CHAIN below).  Whole rounds of tiles of
// more than 128 rows and 32 k steps or more take chains of 16.  Error of the result against 64-bit products, 512 rows x
// [28672, 4096] with a GLU: one chain 1.9e-5, two library products 0.97e-5, chains of 16 0.64e-5; there, a piece begins with
// a longer chain where only two accumulators fit: it is what the tensor cores have to do while the epilogue stores the
// piece before (2048 rows x [28672, 4096]: 608 us, with chains of eight throughout 665, without chains 590).
// Everything else takes chains that lose no more than two library products would, whose accumulators take half the
// additions (one part each) and which cut k for small results: eight steps, half of the k steps where there are fewer than
// 16 of them, six where every tile is cut along k.  Errors with chains of 16, now, and the library's (2.44e-6 of each is
// the activations' two parts'): 275 rows x [34914, 1152] 3.19, 2.67 and 2.70e-6; 262 x [1460, 6784] 3.27, 2.60 and 2.60e-6;
// 558 x [41408, 1024] with a GLU 5.70, 4.22 and 4.09e-6.  Over 110 shapes of 33 to 900 rows at most 1.05 times the
// library's (1.39 before).  It costs 1 % in the mean, 6 % where it costs most (the last of these: 90 and 96 us); a step of
// 80 rows pays 19 us of 399 for chains of eight in place of 16.
constexpr uint32_t TC_CHAIN = 16, TC_FIRST_CHAIN = 32, TC_SHORT_CHAIN = 8, TC_CUT_CHAIN = 6, TC_LEAST_CHAIN = 4;
constexpr int TC_MAX_BUFS = 4;
constexpr uint32_t GLU_GROUP = 16;          // gate and up rows alternate in a tile sixteen by sixteen: a warp holds both

struct PairArgs {
    uint32_t T, cols;                 // pass rows; columns of the result
    uint32_t bt, t_tiles;             // pass rows of a tile (multiple of 32), tiles of them
    uint32_t ksteps;
    uint32_t pairs;                   // CTA pairs of the grid
    uint32_t rounds;                  // whole rounds of tiles
    uint32_t rest_units, rest_pairs;  // k steps of the tiles after them, and the pairs that share those
    uint32_t stages;
    uint32_t bufs, buf_columns;       // accumulators in tensor memory
    uint32_t chain, long_first;       // k steps summed in one of them; whether a piece begins with more
    float *out;
    float *part;                      // [2 * rest_pairs shares][2 CTAs][bt][128]
    uint32_t *counters;               // [tiles left over][2 CTAs], zero between launches
    yx_dev_status *status;
};

// One stretch of k steps of one tile.
struct Piece {
    uint32_t tile, k0, k1;
    bool whole;
};

__device__ __forceinline__ uint32_t rest_begin(const PairArgs &a, uint32_t p) { return (uint32_t)((uint64_t)p * a.rest_units / a.rest_pairs); }
// The pair whose share holds unit u.
__device__ __forceinline__ uint32_t rest_owner(const PairArgs &a, uint32_t u) {
    return (uint32_t)((((uint64_t)u + 1) * a.rest_pairs - 1) / a.rest_units);
}

// Walks a pair's pieces: its share of the left-over tiles (at most two pieces), then its whole tiles.
struct Walk {
    uint32_t u, u_end, round;
    __device__ __forceinline__ Walk(const PairArgs &a, uint32_t pair) : u(0), u_end(0), round(0) {
        if (pair < a.rest_pairs) {
            u = rest_begin(a, pair);
            u_end = rest_begin(a, pair + 1);
        }
    }
    __device__ __forceinline__ bool next(const PairArgs &a, uint32_t pair, Piece &p) {
        if (u < u_end) {
            const uint32_t tile = u / a.ksteps;
            p.k0 = u - tile * a.ksteps;
            p.k1 = min(a.ksteps, p.k0 + (u_end - u));
            u += p.k1 - p.k0;
            p.tile = a.rounds * a.pairs + tile;
            p.whole = p.k1 - p.k0 == a.ksteps;
            return true;
        }
        if (round >= a.rounds) return false;
        p = Piece{round * a.pairs + pair, 0, a.ksteps, true};
        round++;
        return true;
    }
};

// Where the chain of k steps that begins at k ends.
__device__ __forceinline__ uint32_t chain_end(const PairArgs &a, const Piece &p, uint32_t k) {
    const uint32_t n = k == p.k0 && a.long_first ? min(TC_FIRST_CHAIN, max(a.chain, (p.k1 - p.k0) * 3 / 8)) : a.chain;
    return min(p.k1, k + n);
}
// Accumulators in turn, and the parity of the current round of them.
struct AccTurn {
    uint32_t buf = 0, round = 0;
    __device__ __forceinline__ void next(uint32_t bufs) {
        if (++buf == bufs) {
            buf = 0;
            round++;
        }
    }
};

__device__ __forceinline__ uint32_t mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
}

// 32 pass rows from `t0` on of this lane's weight row.
template <bool GLU>
__device__ __forceinline__ void store_rows(const PairArgs &a, const float (&v)[32], uint32_t t0, uint32_t row, int lane) {
    if constexpr (!GLU) {
        if (row >= a.cols) return;
        float *dst = a.out + (size_t)t0 * a.cols + row;
        if (t0 + 32 <= a.T) {
#pragma unroll
            for (int i = 0; i < 32; i++) dst[(size_t)i * a.cols] = v[i];
        } else {
#pragma unroll
            for (int i = 0; i < 32; i++)
                if (t0 + i < a.T) dst[(size_t)i * a.cols] = v[i];
        }
    } else {
        // Lanes 0-15 hold gate rows, lanes 16-31 the same rows' up: the lower half finishes the first sixteen
        // pass rows, the upper half the others.  `row` counts both kinds, so its 32 are 16 columns.
        const uint32_t col = (row >> 5) * GLU_GROUP + (lane & 15), t = t0 + (lane & 16);
        float *dst = a.out + (size_t)t * a.cols + col;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const float other = __shfl_xor_sync(0xffffffffu, lane < 16 ? v[16 + i] : v[i], 16);
            const float g = lane < 16 ? v[i] : other, u = lane < 16 ? other : v[16 + i];
            if (col < a.cols && t + i < a.T) dst[(size_t)i * a.cols] = g / (1.0f + expf(-g)) * u;
        }
    }
}

// CHUNKS: 64-row chunks of a tile, what an epilogue thread keeps in registers (two for up to
// 128 pass rows, three for up to 192: before the chains of eight above, steps of 80 and of 311 rows took 391 and 453 us with
// room for four, 382 and 437 so; with them 399 and 440).
template <bool GLU, int CHUNKS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(TC_THREADS, 1)
matmul_pair_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ CUtensorMap x_map, const PairArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar_store[2 * TC_MAX_STAGES + 2 * TC_MAX_BUFS];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_flag;
    __shared__ int last_s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = blockIdx.x & 1u, pair = blockIdx.x >> 1;
    const uint32_t S = a.stages, x_bytes = a.bt * 128u, stage_bytes = W_BYTES + x_bytes;   // x: bt / 2 rows, high and low part
    const uint32_t base = smem_u32(smem);
    const uint32_t b_full = smem_u32(bar_store), b_empty = b_full + 8 * TC_MAX_STAGES;
    const uint32_t b_acc_full = b_empty + 8 * TC_MAX_STAGES, b_acc_empty = b_acc_full + 8 * TC_MAX_BUFS;
    volatile int *abortp = &abort_flag;

    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (uint32_t s = 0; s < S; s++) {
            mbar_init(b_full + 8 * s, 1);
            mbar_init(b_empty + 8 * s, 1);
        }
        for (int b = 0; b < TC_MAX_BUFS; b++) {
            mbar_init(b_acc_full + 8 * b, 1);
            mbar_init(b_acc_empty + 8 * b, 16);   // a warp's arrival each, from both CTAs
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == TC_TMA_WARP && lane == 0) {
        prefetch_tensormap(&w_map);
        prefetch_tensormap(&x_map);
    }
    if (warp == TC_MMA_WARP) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "n"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;

    if (warp == TC_TMA_WARP && lane == 0) {
        // ---- producer -------------------------------------------------------------------------
        const uint32_t full0 = mapa(b_full, 0);   // the first CTA's barriers count both CTAs' bytes
        auto load_w = [&](uint32_t s, const Piece &p, uint32_t k) {
            const uint32_t m0 = (p.tile / a.t_tiles) * TC_M + rank * 128u;
            if (rank == 0) mbar_expect_tx(b_full + 8 * s, 2 * stage_bytes);
            tma_load_4d_pair(base + s * stage_bytes, &w_map, (int)(k * TC_KSTEP), GLU ? 0 : (int)m0, 0, GLU ? (int)(m0 / (2 * GLU_GROUP)) : 0,
                             full0 + 8 * s);
        };
        auto load_x = [&](uint32_t s, const Piece &p, uint32_t k) {
            const uint32_t t0 = (p.tile % a.t_tiles) * a.bt + rank * (a.bt / 2);
            tma_load_3d_pair(base + s * stage_bytes + W_BYTES, &x_map, (int)(k * TC_KSTEP), (int)t0, 0, full0 + 8 * s);
        };
        // The kernel ahead (the split of the activations) let this one start only after its own wait, so nothing
        // that may still run writes the weights: the ring's first weights are on their way before the wait.
        uint32_t ahead = 0;
        {
            Walk walk(a, pair);
            Piece p;
            while (ahead < S && walk.next(a, pair, p))
                for (uint32_t k = p.k0; k < p.k1 && ahead < S; k++) load_w(ahead++, p, k);
        }
        asm volatile("griddepcontrol.wait;" ::: "memory");
        asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        Walk walk(a, pair);
        Piece p;
        uint32_t it = 0, s = 0, phase = 0;
        while (walk.next(a, pair, p)) {
            for (uint32_t k = p.k0; k < p.k1; k++, it++) {
                if (it >= ahead) {
                    mbar_wait(b_empty + 8 * s, phase ^ 1u, abortp, a.status, 501);
                    if (*abortp) break;
                    load_w(s, p, k);
                }
                load_x(s, p, k);
                if (++s == S) {
                    s = 0;
                    phase ^= 1u;
                }
            }
            if (*abortp) break;
        }
    } else if (warp == TC_MMA_WARP && lane == 0 && rank == 0) {
        // ---- MMA issuer -----------------------------------------------------------------------
        const uint32_t idesc = f16_instr_desc(true, false, TC_M, a.bt);
        Walk walk(a, pair);
        Piece p;
        uint32_t s = 0, phase = 0;
        AccTurn turn;
        while (!*abortp && walk.next(a, pair, p)) {
            for (uint32_t k0 = p.k0; k0 < p.k1 && !*abortp; turn.next(a.bufs)) {
                const uint32_t acc = tmem + turn.buf * a.buf_columns, k_end = chain_end(a, p, k0);
                if (turn.round > 0) mbar_wait(b_acc_empty + 8 * turn.buf, (turn.round - 1) & 1u, abortp, a.status, 502);
                tc_fence_after();
                for (uint32_t k = k0; k < k_end; k++) {
                    mbar_wait(b_full + 8 * s, phase, abortp, a.status, 503);
                    if (*abortp) break;
                    tc_fence_after();
                    const uint32_t w_lo = desc_lo(base + s * stage_bytes, 0), h_lo = w_lo + W_BYTES / 16, l_lo = h_lo + x_bytes / 32;
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) umma2_ss_lo(acc, w_lo + 2 * kk, h_lo + 2 * kk, idesc, k > k0 || kk > 0);
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) umma2_ss_lo(acc, w_lo + 2 * kk, l_lo + 2 * kk, idesc, 1);
                    umma2_commit(b_empty + 8 * s);
                    if (++s == S) {
                        s = 0;
                        phase ^= 1u;
                    }
                }
                umma2_commit(b_acc_full + 8 * turn.buf);
                k0 = k_end;
            }
        }
    } else if (warp < 8) {
        // ---- epilogue -------------------------------------------------------------------------
        Walk walk(a, pair);
        Piece p;
        AccTurn turn;
        while (walk.next(a, pair, p)) {
            const uint32_t wr = (warp & 3) * 32 + lane;   // weight row of this CTA's 128
            const uint32_t row = (p.tile / a.t_tiles) * TC_M + rank * 128u + wr, t0 = (p.tile % a.t_tiles) * a.bt;
            const uint32_t rest = p.whole ? 0u : p.tile - a.rounds * a.pairs;
            // The pairs that share left-over tile `rest`, found while it is being summed.  Only the first of them may
            // have begun in the tile before it, which makes this tile its second piece.
            uint32_t q0 = 0, q1 = 0, second = 0;
            if (!p.whole) {
                q0 = rest_owner(a, rest * a.ksteps);
                q1 = rest_owner(a, (rest + 1) * a.ksteps - 1);
                second = rest - rest_begin(a, q0) / a.ksteps;
            }
            // This thread's sums: its weight row, 32 pass rows out of every 64.
            const uint32_t c0 = 32u * (warp >> 2);
            float sum[CHUNKS][32];
#pragma unroll
            for (int j = 0; j < CHUNKS; j++)
#pragma unroll
                for (int i = 0; i < 32; i++) sum[j][i] = 0.0f;
            for (uint32_t k = p.k0; k < p.k1; k = chain_end(a, p, k), turn.next(a.bufs)) {
                const uint32_t acc = tmem + turn.buf * a.buf_columns + ((uint32_t)(warp & 3) << 21);
                mbar_wait(b_acc_full + 8 * turn.buf, turn.round & 1u, abortp, a.status, 504);
                __syncwarp();   // (after a wait that ran out the warps go on, on whatever is there: their barriers below count all of them)
                tc_fence_after();
#pragma unroll
                for (int j = 0; j < CHUNKS; j++) {
                    if (c0 + 64 * j >= a.bt) break;
#pragma unroll
                    for (int h = 0; h < 32; h += 16) {   // (sixteen at a time: 32 more registers would spill)
                        uint32_t r[16];
                        tmem_ld16(acc + c0 + 64 * j + h, r);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i++) sum[j][h + i] += __uint_as_float(r[i]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(mapa(b_acc_empty + 8 * turn.buf, 0)) : "memory");
            }
            // A share's sums: four pass rows of each of 128 weight rows, then the next four.
            auto share = [&](uint32_t q) { return (float4 *)(a.part + ((size_t)(2 * q + (q == q0 ? second : 0u)) * 2 + rank) * a.bt * 128u) + wr; };
#pragma unroll
            for (int j = 0; j < CHUNKS; j++) {
                const uint32_t c = c0 + 64 * j;
                if (c >= a.bt) break;
                if (p.whole) {
                    store_rows<GLU>(a, sum[j], t0 + c, row, lane);
                } else {
                    float4 *mine = share(pair) + c / 4 * 128u;
#pragma unroll
                    for (int i = 0; i < 8; i++) __stcg(mine + i * 128, make_float4(sum[j][4 * i], sum[j][4 * i + 1], sum[j][4 * i + 2], sum[j][4 * i + 3]));
                }
            }
            if (p.whole) continue;
            // The last of the tile's shares to arrive adds all of them up, in the order of k.
            __threadfence();
            asm volatile("bar.sync 1, 256;" ::: "memory");
            if (threadIdx.x == 0) {
                uint32_t *counter = a.counters + 2 * rest + rank;
                const int last = atomicAdd(counter, 1u) == q1 - q0;
                if (last) *counter = 0u;
                last_s = last;
            }
            asm volatile("bar.sync 1, 256;" ::: "memory");
            const bool last = last_s != 0;
            if (!last) continue;
            __threadfence();
            // (a chain of L2 latencies: six shares' sums are asked for at once)
            for (uint32_t c = 32u * (warp >> 2); c < a.bt && t0 + c < a.T; c += 64) {
                alignas(16) float v[32];
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    float4 sum[4] = {};
                    for (uint32_t q = q0; q <= q1; q += 6) {
                        float4 w[6][4];
#pragma unroll
                        for (int b = 0; b < 6; b++) {
                            const float4 *src = share(min(q + b, q1)) + (c / 4 + 4 * h) * 128u;
#pragma unroll
                            for (int i = 0; i < 4; i++) w[b][i] = q + b <= q1 ? __ldcg(src + i * 128) : make_float4(0.f, 0.f, 0.f, 0.f);
                        }
#pragma unroll
                        for (int b = 0; b < 6; b++)
#pragma unroll
                            for (int i = 0; i < 4; i++) {
                                sum[i].x += w[b][i].x;
                                sum[i].y += w[b][i].y;
                                sum[i].z += w[b][i].z;
                                sum[i].w += w[b][i].w;
                            }
                    }
#pragma unroll
                    for (int i = 0; i < 4; i++) *(float4 *)(v + 16 * h + 4 * i) = sum[i];
                }
                store_rows<GLU>(a, v, t0 + c, row, lane);
            }
        }
    }
    __syncwarp();
    if (*abortp)
        for (int i = 0; i < 64; i++) __nanosleep(1000);   // copies and products in flight come to rest
    tc_fence_before();
    __syncthreads();
    cluster_sync();   // the partner's copies and completions still land in this CTA
    tc_fence_after();
    if (warp == TC_MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(512) : "memory");
}

// x [n] f32 -> its high and its low bf16 part, x = hi + lo to 16 bits of mantissa; eight elements a thread.
template <bool VEC16>
__global__ void __launch_bounds__(256) split_rows_kernel(const float *__restrict__ x, size_t n, uint4 *__restrict__ hi, uint4 *__restrict__ lo) {
    dependent_entry();
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx * 8 >= n) return;
    float v[8];
    if constexpr (VEC16) {
        *(float4 *)v = *(const float4 *)(x + idx * 8);
        *(float4 *)(v + 4) = *(const float4 *)(x + idx * 8 + 4);
    } else {
#pragma unroll
        for (int j = 0; j < 4; j++) *(float2 *)(v + 2 * j) = *(const float2 *)(x + idx * 8 + 2 * j);
    }
    uint32_t h[4], l[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
        h[j] = pack2<true>(v[2 * j], v[2 * j + 1]);
        const float2 b = unpack2<true>(h[j]);
        l[j] = pack2<true>(v[2 * j] - b.x, v[2 * j + 1] - b.y);
    }
    hi[idx] = make_uint4(h[0], h[1], h[2], h[3]);
    lo[idx] = make_uint4(l[0], l[1], l[2], l[3]);
}

// ---- passes of few rows ------------------------------------------------------------------------------------
//
// At most 32 pass rows: the weights stream through the chip once and everything else must stay out of their way.
// One launch: the activations are split into their bf16 parts on the way into shared memory by eight warps, each
// with every eighth k step, so that eight steps' loads are in flight; a step's operand is the high parts' rows and
// the low parts' rows one below the other, one MMA per 16 k takes both, and the epilogue adds the two halves of
// the accumulator.  128 weight rows by 64 k make a stage; the k steps of all tiles are laid end to end and cut
// into one equal share a CTA, so that every SM streams the same number of bytes whatever N and K are.
// A share that ends inside a tile leaves its sums in scratch, and the CTA that comes last at a tile adds them up
// in the order of k.
// The kernel starts under the one ahead of it and asks its first stages into L2 before it waits: weights are not
// written by the kernel ahead, and even if they were, L2 is where such writes land.
//
// Bound by HBM from some 200 MB on (one row on 28672 x 4096: 45 us, the part above a launch's fixed 8 to 12 us at
// 7.2 TB/s), by a chain of latencies below.  The kernel with weights straight from global memory into mma.sync
// fragments, a packing kernel before it and a finishing kernel behind took 58 us for sixteen rows of that weight;
// steps went from 419 to 360 us (one row, large), 538 to 424 us (sixteen rows), 417 to 340 us (one row, small).
constexpr int ROWS_THREADS = 14 * 32;
constexpr int ROWS_CONVERT_WARP = 6, ROWS_CONVERTERS = 8;
constexpr uint32_t ROWS_M = 128;
constexpr uint32_t ROWS_MAX = 32;           // pass rows
// k steps summed in tensor memory before the epilogue takes them over into its own f32 sums.  The tensor core drops
// what lies below its accumulator's last place: chains of 64 steps erred by 8.1e-6 of a GLU's result (16 rows x
// [28672, 4096]), the mma.sync kernel by 4.2e-6.  Chains of 16 are
// at 4.0e-6 (but 3.9e-6 against 3.7e-6 for twenty rows x [11264, 2048]), chains of eight at 3.7e-6 for 1.5 % of a step.
constexpr uint32_t ROWS_CHAIN = 8, ROWS_BUFS = 4;   // (and four accumulators: the tensor cores run on while an epilogue adds shares up)

struct RowsArgs {
    const float *x;
    uint32_t T, K, cols, ksteps, units, ctas, stages;
    uint32_t x_vec16;
    float *out;
    float *part;          // [2 * ctas shares][TP][128]
    uint32_t *counters;   // one a tile, zero between launches
    yx_dev_status *status;
};
__device__ __forceinline__ uint32_t share_begin(const RowsArgs &a, uint32_t p) { return (uint32_t)((uint64_t)p * a.units / a.ctas); }
__device__ __forceinline__ uint32_t share_owner(const RowsArgs &a, uint32_t u) { return (uint32_t)((((uint64_t)u + 1) * a.ctas - 1) / a.units); }

// TP pass rows of this lane's weight row.
template <int TP, bool GLU>
__device__ __forceinline__ void store_few(const RowsArgs &a, const float (&v)[TP], uint32_t row, int lane) {
    if constexpr (!GLU) {
        if (row >= a.cols) return;
#pragma unroll
        for (int i = 0; i < TP; i++)
            if (i < (int)a.T) a.out[(size_t)i * a.cols + row] = v[i];
    } else {
        // (see store_rows: the lower half of the warp finishes the first half of the pass rows)
        const uint32_t col = (row >> 5) * GLU_GROUP + (lane & 15), t = lane < 16 ? 0 : TP / 2;
#pragma unroll
        for (int i = 0; i < TP / 2; i++) {
            const float other = __shfl_xor_sync(0xffffffffu, lane < 16 ? v[TP / 2 + i] : v[i], 16);
            const float g = lane < 16 ? v[i] : other, u = lane < 16 ? other : v[TP / 2 + i];
            if (col < a.cols && t + i < a.T) a.out[(size_t)(t + i) * a.cols + col] = g / (1.0f + expf(-g)) * u;
        }
    }
}

template <int TP, bool GLU>
__global__ void __launch_bounds__(ROWS_THREADS, 1)
matmul_rows_kernel(const __grid_constant__ CUtensorMap w_map, const __grid_constant__ RowsArgs a) {
    extern __shared__ __align__(1024) unsigned char smem[];
    __shared__ __align__(8) uint64_t bar_store[2 * TC_MAX_STAGES + 2 * ROWS_BUFS];
    __shared__ uint32_t tmem_base_s;
    __shared__ int abort_flag;
    __shared__ int last_s;
    constexpr uint32_t NB = 2 * TP, X_BYTES = NB * 128, STAGE = W_BYTES + X_BYTES;
    constexpr uint32_t TMEM = ROWS_BUFS * NB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t S = a.stages, base = smem_u32(smem);
    const uint32_t b_full = smem_u32(bar_store), b_empty = b_full + 8 * TC_MAX_STAGES;
    const uint32_t b_acc_full = b_empty + 8 * TC_MAX_STAGES, b_acc_empty = b_acc_full + 8 * ROWS_BUFS;
    volatile int *abortp = &abort_flag;
    const uint32_t u0 = share_begin(a, blockIdx.x), u1 = share_begin(a, blockIdx.x + 1);

    auto weight_rows = [&](uint32_t u, int &x, int &y, int &z) {
        const uint32_t tile = u / a.ksteps;
        x = (int)((u - tile * a.ksteps) * TC_KSTEP);
        y = GLU ? 0 : (int)(tile * ROWS_M);
        z = GLU ? (int)(tile * (ROWS_M / (2 * GLU_GROUP))) : 0;
    };
    if (warp == 4 && lane == 0) {
        prefetch_tensormap(&w_map);
        for (uint32_t u = u0; u < u1 && u - u0 < S; u++) {
            int x, y, z;
            weight_rows(u, x, y, z);
            tma_prefetch_4d(&w_map, x, y, 0, z);
        }
    }
    if (threadIdx.x == 0) {
        abort_flag = 0;
        for (uint32_t s = 0; s < S; s++) {
            mbar_init(b_full + 8 * s, 2);    // the weights' copy and the converting warp
            mbar_init(b_empty + 8 * s, 1);
        }
        for (uint32_t b = 0; b < ROWS_BUFS; b++) {
            mbar_init(b_acc_full + 8 * b, 1);
            mbar_init(b_acc_empty + 8 * b, 4);
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_s)), "n"(TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    if (warp == 4) {
        // ---- weights --------------------------------------------------------------------------
        if (lane == 0) {
            uint32_t s = 0, phase = 0;
            for (uint32_t u = u0; u < u1; u++) {
                if (u - u0 >= S) mbar_wait(b_empty + 8 * s, phase ^ 1u, abortp, a.status, 511);
                if (*abortp) break;
                int x, y, z;
                weight_rows(u, x, y, z);
                mbar_expect_tx(b_full + 8 * s, W_BYTES);
                tma_load_4d(base + s * STAGE, &w_map, x, y, 0, z, b_full + 8 * s);
                if (++s == S) {
                    s = 0;
                    phase ^= 1u;
                }
            }
        }
    } else if (warp == 5) {
        // ---- MMA issuer -----------------------------------------------------------------------
        if (lane == 0) {
            constexpr uint32_t idesc = f16_instr_desc(true, false, ROWS_M, NB);
            uint32_t s = 0, phase = 0, n = 0, piece_end = u0;
            for (uint32_t u = u0; u < u1 && !*abortp; n++) {
                if (u == piece_end) piece_end = min(u1, (u / a.ksteps + 1) * a.ksteps);
                const uint32_t end = min(piece_end, u + ROWS_CHAIN);
                const uint32_t buf = n % ROWS_BUFS, acc = tmem + buf * NB;
                if (n >= ROWS_BUFS) mbar_wait(b_acc_empty + 8 * buf, (n / ROWS_BUFS - 1) & 1u, abortp, a.status, 512);
                tc_fence_after();
                for (uint32_t first = u; u < end; u++) {
                    mbar_wait(b_full + 8 * s, phase, abortp, a.status, 513);
                    if (*abortp) break;
                    tc_fence_after();
                    const uint32_t w_lo = desc_lo(base + s * STAGE, 0), x_lo = w_lo + W_BYTES / 16;
#pragma unroll
                    for (uint32_t kk = 0; kk < 4; kk++) umma_ss_lo(acc, w_lo + 2 * kk, x_lo + 2 * kk, idesc, u > first || kk > 0);
                    umma_commit(b_empty + 8 * s);
                    if (++s == S) {
                        s = 0;
                        phase ^= 1u;
                    }
                }
                umma_commit(b_acc_full + 8 * buf);
            }
        }
    } else if (warp >= ROWS_CONVERT_WARP) {
        // ---- activations: every eighth step is this warp's ------------------------------------------
        for (uint32_t u = u0 + (uint32_t)(warp - ROWS_CONVERT_WARP); u < u1; u += ROWS_CONVERTERS) {
            const uint32_t it = u - u0, s = it % S, use = it / S;
            const float *src = a.x + (size_t)(u % a.ksteps) * TC_KSTEP;
            constexpr int R = TP / 4;          // 16-byte operand chunks (eight k of a pass row) a lane
            float v[R][8];
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint32_t t = r * 4 + (lane >> 3);
                if (t >= a.T) continue;        // (rows past T only reach accumulator columns that nobody reads)
                const float *p = src + (size_t)t * a.K + (lane & 7) * 8;
                if (a.x_vec16) {
                    *(float4 *)&v[r][0] = *(const float4 *)p;
                    *(float4 *)&v[r][4] = *(const float4 *)(p + 4);
                } else {
#pragma unroll
                    for (int j = 0; j < 4; j++) *(float2 *)&v[r][2 * j] = *(const float2 *)(p + 2 * j);
                }
            }
            if (use > 0) mbar_wait(b_empty + 8 * s, (use - 1) & 1u, abortp, a.status, 514);
            if (__any_sync(0xffffffffu, *abortp)) break;
            unsigned char *dst = smem + s * STAGE + W_BYTES;
#pragma unroll
            for (int r = 0; r < R; r++) {
                const uint32_t t = r * 4 + (lane >> 3);
                if (t >= a.T) continue;
                uint32_t h[4], l[4];
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    h[j] = pack2<true>(v[r][2 * j], v[r][2 * j + 1]);
                    const float2 b = unpack2<true>(h[j]);
                    l[j] = pack2<true>(v[r][2 * j] - b.x, v[r][2 * j + 1] - b.y);
                }
                unsigned char *at = dst + t * 128 + (((lane & 7) ^ (t & 7)) << 4);
                *(uint4 *)at = make_uint4(h[0], h[1], h[2], h[3]);
                *(uint4 *)(at + TP * 128) = make_uint4(l[0], l[1], l[2], l[3]);
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(b_full + 8 * s);
        }
    } else {
        // ---- epilogue -------------------------------------------------------------------------
        uint32_t n = 0;
        for (uint32_t u = u0; u < u1;) {
            const uint32_t tile = u / a.ksteps, end = min(u1, (tile + 1) * a.ksteps);
            const bool whole = end - u == a.ksteps;
            const uint32_t wr = warp * 32 + lane, row = tile * ROWS_M + wr;
            // The CTAs that share this tile, found while the tile is being summed (the divisions take a third of a
            // microsecond).  Only the first of them may have begun in a tile before it: then this is its last piece.
            uint32_t q0 = 0, q1 = 0, later = 0;
            if (!whole) {
                q0 = share_owner(a, tile * a.ksteps);
                q1 = share_owner(a, (tile + 1) * a.ksteps - 1);
                later = share_begin(a, q0) < tile * a.ksteps;
            }
            float v[TP];
#pragma unroll
            for (int i = 0; i < TP; i++) v[i] = 0.0f;
            for (; u < end; n++) {
                u = min(end, u + ROWS_CHAIN);
                const uint32_t buf = n % ROWS_BUFS, acc = tmem + buf * NB + ((uint32_t)warp << 21);
                mbar_wait(b_acc_full + 8 * buf, (n / ROWS_BUFS) & 1u, abortp, a.status, 515);
                __syncwarp();   // (a wait that ran out does not stop these warps: their barriers below count all of them)
                tc_fence_after();
                if constexpr (TP == 8) {
                    uint32_t r[16];
                    tmem_ld16(acc, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 8; i++) v[i] += __uint_as_float(r[i]) + __uint_as_float(r[8 + i]);
                } else {
#pragma unroll
                    for (int h = 0; h < TP / 16; h++) {
                        uint32_t r[16], q[16];
                        tmem_ld16(acc + 16 * h, r);
                        tmem_ld16(acc + TP + 16 * h, q);
                        tmem_ld_wait();
#pragma unroll
                        for (int i = 0; i < 16; i++) v[16 * h + i] += __uint_as_float(r[i]) + __uint_as_float(q[i]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(b_acc_empty + 8 * buf);
            }
            if (whole) {
                store_few<TP, GLU>(a, v, row, lane);
                continue;
            }
            auto share = [&](uint32_t q) { return a.part + (size_t)(2 * q + (q == q0 ? later : 0u)) * TP * 128u + wr; };
            float *mine = share(blockIdx.x);
#pragma unroll
            for (int i = 0; i < TP; i++)
                if (i < (int)a.T) __stcg(mine + i * 128, v[i]);
            __threadfence();
            asm volatile("bar.sync 1, 128;" ::: "memory");
            if (threadIdx.x == 0) {
                const int last = atomicAdd(a.counters + tile, 1u) == q1 - q0;
                if (last) a.counters[tile] = 0u;
                last_s = last;
            }
            asm volatile("bar.sync 1, 128;" ::: "memory");
            const bool last = last_s != 0;
            if (!last) continue;
            __threadfence();
#pragma unroll
            for (int i = 0; i < TP; i++) v[i] = 0.0f;
            constexpr int B = 64 / TP;   // shares read at once
            for (uint32_t q = q0; q <= q1; q += B) {
                float w[B][TP];
#pragma unroll
                for (int b = 0; b < B; b++) {
                    const float *src = share(min(q + b, q1));
#pragma unroll
                    for (int i = 0; i < TP; i++) w[b][i] = i < (int)a.T && q + b <= q1 ? __ldcg(src + i * 128) : 0.0f;
                }
#pragma unroll
                for (int b = 0; b < B; b++)
#pragma unroll
                    for (int i = 0; i < TP; i++) v[i] += w[b][i];
            }
            store_few<TP, GLU>(a, v, row, lane);
        }
    }
    __syncwarp();
    if (*abortp)
        for (int i = 0; i < 64; i++) __nanosleep(1000);   // copies and products in flight come to rest
    tc_fence_before();
    __syncthreads();
    if (warp == 5) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMEM) : "memory");
}

using EncodeTiled = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            p = nullptr;
        return (EncodeTiled)p;
    }();
    return fn;
}

// A map of a bf16 tensor, innermost dimension dense, 128-byte swizzle; rows outside it read as zero.
int encode(yx_ctx *ctx, CUtensorMap *map, uint32_t rank, const void *p, const cuuint64_t *dims, const cuuint64_t *strides, const cuuint32_t *box) {
    const cuuint32_t ones[4] = {1, 1, 1, 1};
    if (!encode_tiled()) return fail(ctx, YX_ERR_CUDA, "matmul: the driver has no cuTensorMapEncodeTiled");
    const CUresult r = encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void *>(p), dims, strides, box, ones,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? YX_OK : fail(ctx, YX_ERR_CUDA, "matmul: cuTensorMapEncodeTiled failed with " + std::to_string((int)r));
}

// The weights in boxes of 128 rows by 64 k; for a GLU four groups of 16 gate rows and the 16 up rows of the same columns.
int encode_weights(yx_ctx *ctx, CUtensorMap *map, const void *w, uint32_t N, uint32_t K, bool glu) {
    const cuuint64_t row = (cuuint64_t)K * 2;
    if (glu) {
        const cuuint64_t dims[4] = {K, GLU_GROUP, 2, N / 2 / GLU_GROUP};
        const cuuint64_t strides[3] = {row, N / 2 * row, GLU_GROUP * row};
        const cuuint32_t box[4] = {TC_KSTEP, GLU_GROUP, 2, 128 / (2 * GLU_GROUP)};
        return encode(ctx, map, 4, w, dims, strides, box);
    }
    const cuuint64_t dims[4] = {K, N, 1, 1};
    const cuuint64_t strides[3] = {row, N * row, N * row};
    const cuuint32_t box[4] = {TC_KSTEP, 128, 1, 1};
    return encode(ctx, map, 4, w, dims, strides, box);
}

int ensure_counters(yx_ctx *ctx, size_t n) {
    const size_t before = ctx->mm_counters_cap;
    if (int rc = ensure_buffer(ctx, (void **)&ctx->mm_counters, &ctx->mm_counters_cap, std::max<size_t>(n, 512) * sizeof(uint32_t))) return rc;
    if (ctx->mm_counters_cap == before) return YX_OK;
    return check_cuda(ctx, cudaMemsetAsync(ctx->mm_counters, 0, ctx->mm_counters_cap, ctx->stream), "matmul: counters");
}

// CTA pairs that are on the chip together (a GPC with an odd number of SMs leaves one out).
template <bool GLU, int CHUNKS>
int resident_pairs(yx_ctx *ctx, int *out) {
    int &n = ctx->mm_pairs[GLU][CHUNKS - 2];
    if (n == 0) {
        auto *kernel = matmul_pair_kernel<GLU, CHUNKS>;
        if (int rc = check_cuda(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_BUDGET),
                                "matmul: shared memory attribute"))
            return rc;
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)ctx->sm_count / 2 * 2);
        cfg.blockDim = dim3(TC_THREADS);
        cfg.dynamicSmemBytes = TC_SMEM_BUDGET;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        int found = 0;
        if (int rc = check_cuda(ctx, cudaOccupancyMaxActiveClusters(&found, kernel, &cfg), "matmul: resident pairs")) return rc;
        n = std::max(1, std::min(found, ctx->sm_count / 2));
    }
    *out = n;
    return YX_OK;
}

// Pass rows are spread evenly over as few tiles as hold them: 300 rows are two tiles of 160, not 256 and 64.
uint32_t tile_rows(uint32_t T) {
    const uint32_t tiles = (T + TC_MAX_BT - 1) / TC_MAX_BT;
    return ((T + tiles - 1) / tiles + 31) / 32 * 32;
}

// How many pairs share the k steps of `tiles` left-over tiles.  Either every tile is cut into the same number of
// shares, which leaves some pairs idle, or all pairs take an equal share, which lets shares run over the end of a
// tile: one more epilogue and one more share to add up for most pairs.  A k step takes 0.26 us and 2 ns a pass row
// (62 GB/s into each SM, measured at 96 to 256 rows), the extra epilogue 3 us, adding up at all another 6; behind
// whole rounds both are hidden.  A share of fewer than four k steps costs more to add up than it saves.
uint32_t share_rest(uint32_t tiles, uint32_t ksteps, uint32_t pairs, uint32_t bt, bool hidden) {
    const uint32_t most = std::max(1u, ksteps / 4), each = std::min(pairs / tiles, most);
    const uint32_t all = std::min(pairs, tiles * most);
    const float step = 0.26f + 0.002f * (float)bt, overrun = hidden ? 1.0f : each == 1 ? 9.0f : 3.0f;
    const float even = step * (float)((ksteps + each - 1) / each), equal = step * (float)(tiles * ksteps) / (float)all;
    return even <= equal + overrun ? tiles * each : all;
}

template <bool GLU, int CHUNKS>
int matmul_pair_rows(yx_ctx *ctx, const float *x, const void *w, uint32_t T, uint32_t N, uint32_t K, float *out) {
    const size_t n = (size_t)T * K;
    if (int rc = ensure_buffer(ctx, (void **)&ctx->mm_packed, &ctx->mm_packed_cap, n * 4)) return rc;
    int pairs = 0;
    if (int rc = resident_pairs<GLU, CHUNKS>(ctx, &pairs)) return rc;

    PairArgs a{};
    a.T = T;
    a.cols = GLU ? N / 2 : N;
    a.t_tiles = (T + TC_MAX_BT - 1) / TC_MAX_BT;
    a.bt = tile_rows(T);
    a.ksteps = K / TC_KSTEP;
    const uint32_t tiles = ((N + TC_M - 1) / TC_M) * a.t_tiles;
    a.pairs = (uint32_t)pairs;
    a.rounds = tiles / a.pairs;
    a.rest_units = (tiles - a.rounds * a.pairs) * a.ksteps;
    if (a.rest_units > 0) a.rest_pairs = share_rest(tiles - a.rounds * a.pairs, a.ksteps, a.pairs, a.bt, a.rounds > 0);
    const uint32_t stage_bytes = W_BYTES + a.bt * 128u;
    a.stages = std::min<uint32_t>(TC_MAX_STAGES, (TC_SMEM_BUDGET - 1024) / stage_bytes);
    a.bufs = a.bt <= 128 ? 4 : a.bt <= 160 ? 3 : 2;
    a.buf_columns = 512 / a.bufs / 32 * 32;
    const bool large = a.bufs < TC_MAX_BUFS && a.rounds > 0 && a.ksteps >= 2 * TC_CHAIN;
    a.chain = large ? TC_CHAIN : std::min(a.rounds > 0 ? TC_SHORT_CHAIN : TC_CUT_CHAIN, std::max(TC_LEAST_CHAIN, a.ksteps / 2));
    a.long_first = large && a.bufs == 2;
    a.out = out;
    a.status = ctx->dev_status;
    // The most any pass needs (39 MB), so that a call that is being recorded into a graph finds it whatever passes came
    // before: the shares' room does not grow with the rows (512 rows may leave no tile over, 100 rows many).
    if (int rc = ensure_buffer(ctx, (void **)&ctx->mm_part, &ctx->mm_part_cap, (size_t)a.pairs * 2 * 2 * TC_MAX_BT * 128 * sizeof(float))) return rc;
    a.part = ctx->mm_part;
    if (int rc = ensure_counters(ctx, 2 * a.pairs)) return rc;
    a.counters = ctx->mm_counters;

    CUtensorMap w_map, x_map;
    if (int rc = encode_weights(ctx, &w_map, w, N, K, GLU)) return rc;
    uint4 *hi = (uint4 *)ctx->mm_packed, *lo = hi + n / 8;
    {
        const cuuint64_t dims[3] = {K, T, 2};
        const cuuint64_t strides[2] = {(cuuint64_t)K * 2, (cuuint64_t)T * K * 2};
        const cuuint32_t box[3] = {TC_KSTEP, a.bt / 2, 2};
        if (int rc = encode(ctx, &x_map, 3, hi, dims, strides, box)) return rc;
    }
    ctx->last_launch = yx_ctx::LAST_OTHER;
    if (int rc = launch_dependent(ctx, "matmul: activation split kernel launch", ((uintptr_t)x & 15u) == 0 ? split_rows_kernel<true> : split_rows_kernel<false>,
                                  dim3((unsigned)((n / 8 + 255) / 256)), dim3(256), 0, x, n, hi, lo))
        return rc;
    const uint32_t grid = 2 * (a.rounds > 0 ? a.pairs : a.rest_pairs);
    return launch_dependent(ctx, "matmul kernel launch", matmul_pair_kernel<GLU, CHUNKS>, dim3(grid), dim3(TC_THREADS), a.stages * stage_bytes, w_map, x_map, a);
}

template <int TP, bool GLU>
int matmul_few_rows(yx_ctx *ctx, const float *x, const void *w, uint32_t T, uint32_t N, uint32_t K, float *out) {
    constexpr uint32_t stage_bytes = W_BYTES + 2 * TP * 128, stages = std::min<uint32_t>(TC_MAX_STAGES, TC_SMEM_BUDGET / stage_bytes);
    auto *kernel = matmul_rows_kernel<TP, GLU>;
    bool &configured = ctx->mm_rows_configured[GLU][TP / 16];
    if (!configured) {
        if (int rc = check_cuda(ctx, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, stages * stage_bytes),
                                "matmul: shared memory attribute"))
            return rc;
        configured = true;
    }
    RowsArgs a{};
    // Other CTAs still read the rows when a tile's result is written: a result over its own rows takes them from a copy.
    const uintptr_t x0 = (uintptr_t)x, o0 = (uintptr_t)out;
    if (o0 < x0 + (size_t)T * K * 4 && x0 < o0 + (size_t)T * (GLU ? N / 2 : N) * 4) {
        if (int rc = ensure_buffer(ctx, (void **)&ctx->mm_packed, &ctx->mm_packed_cap, (size_t)ROWS_MAX * K * 4)) return rc;
        if (int rc = check_cuda(ctx, cudaMemcpyAsync(ctx->mm_packed, x, (size_t)T * K * 4, cudaMemcpyDeviceToDevice, ctx->stream), "matmul: rows under the result"))
            return rc;
        x = (const float *)ctx->mm_packed;
    }
    a.x = x;
    a.T = T;
    a.K = K;
    a.cols = GLU ? N / 2 : N;
    a.ksteps = K / TC_KSTEP;
    const uint32_t tiles = (N + ROWS_M - 1) / ROWS_M;
    a.units = tiles * a.ksteps;
    a.ctas = std::min((uint32_t)ctx->sm_count, std::max(1u, a.units / 2));
    a.stages = stages;
    a.x_vec16 = ((uintptr_t)x & 15u) == 0;
    a.out = out;
    a.status = ctx->dev_status;
    // (for any number of rows and any weight, as in matmul_pair_rows: one row may be followed by sixteen in a recording)
    if (int rc = ensure_buffer(ctx, (void **)&ctx->mm_part, &ctx->mm_part_cap, (size_t)2 * ctx->sm_count * ROWS_MAX * 128 * sizeof(float))) return rc;
    if (int rc = ensure_counters(ctx, tiles)) return rc;
    a.part = ctx->mm_part;
    a.counters = ctx->mm_counters;
    CUtensorMap w_map;
    if (int rc = encode_weights(ctx, &w_map, w, N, K, GLU)) return rc;
    ctx->last_launch = yx_ctx::LAST_OTHER;
    return launch_dependent(ctx, "matmul kernel launch", kernel, dim3(a.ctas), dim3(ROWS_THREADS), stages * stage_bytes, w_map, a);
}

template <bool GLU>
int matmul_tc(yx_ctx *ctx, const float *x, const void *w, uint32_t T, uint32_t N, uint32_t K, float *out) {
    if (T <= 8) return matmul_few_rows<8, GLU>(ctx, x, w, T, N, K, out);
    if (T <= 16) return matmul_few_rows<16, GLU>(ctx, x, w, T, N, K, out);
    if (T <= 32) return matmul_few_rows<32, GLU>(ctx, x, w, T, N, K, out);
    const uint32_t rows = tile_rows(T);
    if (rows <= 128) return matmul_pair_rows<GLU, 2>(ctx, x, w, T, N, K, out);
    if (rows <= 192) return matmul_pair_rows<GLU, 3>(ctx, x, w, T, N, K, out);
    return matmul_pair_rows<GLU, 4>(ctx, x, w, T, N, K, out);
}

}  // namespace

// Takes K a multiple of 128, w 16-byte aligned, x 8-byte aligned; with `glu`, a multiple of 16 result columns.
int launch_matmul_tc(yx_ctx *ctx, const float *x, const void *w, uint32_t T, uint32_t N, uint32_t K, bool glu, float *out) {
    return glu ? matmul_tc<true>(ctx, x, w, T, N, K, out) : matmul_tc<false>(ctx, x, w, T, N, K, out);
}

}  // namespace yx
