// tcgen05 FP8 E4M3 GEMM on CTA pairs (cta_group::2), for batches of more rows than the decode tiles take:
//     D[m, n] = epilogue( a_scale[m] * ( w_scale[n] * sum_k A[m, k] * W[n, k] ) )
// Operands, epilogue arithmetic and tolerances are those of fp8_gemm_tc.cuh (A [M, K], W [N, K], row-major fp8).
//
// Two CTAs on neighbouring SMs form one 256 x BN tile: a 256-row slab of W is the MMA's M operand (128 rows in each
// CTA's shared memory), BN batch rows are its N operand (BN / 2 rows in each CTA), and each CTA's TMEM holds the
// 128 x BN f32 accumulator of its own weight rows.  A 128 x 256 one-CTA tile moves 48 KB of L2 -> shared memory per
// 128 bytes of K, the pair 32 KB per CTA for the same MMA work.  BN is a run-time value (a multiple of 32 up to 256) so
// that the tile fits the batch.
//
//   warp 0      TMA producer: this CTA's 128 weight rows and BN / 2 batch rows per stage (128-byte swizzle).  Both
//               CTAs' loads complete on the leader's (even rank) "full" barrier.
//   warp 1      leader only: an elected lane issues the pair's MMAs and commits the stage's "empty" barrier of both CTAs.
//   warp 2      tensor memory: 512 columns, two accumulators, so that the epilogue of one tile overlaps the next
//               tile's main loop.
//   warps 4-11  epilogue: warp w reads lanes 32 * (w % 4) and every second 16-column group of the accumulator.
//
// Persistent form (S == 1): a cluster is one pair and walks the tiles, batch tiles innermost, so that the weights are
// read from HBM about once.  Split-K form (S = 2, 3): a cluster is S pairs on one tile; column group g is finished by
// pair g % S, the others push their partials into its (then idle) operand ring: no global scratch, no atomics, bitwise
// reproducible.
//
// The sum over K is defined apart from its distribution: it is cut into V ranges (V >= S), each accumulated by itself and
// all added in order.  A pair keeps the partials of its ranges side by side in tensor memory.  Up to 128 rows V is the
// split-K factor the one-CTA form's plan gives the shape, so that a batch decodes to the same bytes whichever kernel
// takes it (a decoder stack amplifies the rounding of another order to the size of its FP8 steps within a few layers).
//
// Large batches are bound by the tensor pipe and the power cap, small ones by the weights' stream.  Measured, us, a one-CTA
// form with 256-row batch tiles and a pull reduction against pairs: [8192 x 5376] at M = 500 / 2048: 30 / 125 against 22 / 66;
// [43008 x 5376] 162 / 725 against 92 / 305 (3.1 PFLOP/s); [5376 x 21504] + residual 133 / 517 against 53 / 190; at M = 128
// the four projections 20 / 17 / 48 / 33 against 13 / 11 / 45 / 26.
//
// Every wait is bounded and reports through the status word of fp8_gemm_tc.cuh.
#pragma once
#include "fp8_gemm_tc.cuh"

namespace rvpair {

using namespace rvtc;

constexpr int PAIR_THREADS = 384;
constexpr int PAIR_EPI_WARP0 = 4, PAIR_EPI_WARPS = 8;
constexpr int PAIRS = rv::SMS / 2;
constexpr int PAIR_MAX_STAGES = 8, PAIR_HEADER = 4096;

struct PairParams {
    const float* a_scale;
    const float* w_scale;
    void* out;
    const void* residual;
    int M, N, kblocks;
    int bn, nb, tiles;  // batch columns per tile, batch tiles, tiles in all
    int stages, splits;
    int ranges, npart, sets;  // K ranges (V), most of them in one pair, sets of npart accumulators in tensor memory
    RopeKv rope;     // EPI_QKV_ROPE only
    int rope_pairs;  // EPI_QKV_ROPE: tables 4-byte, Q and caches 2-byte aligned (a lane's two elements move as one)
    float* arg_val;  // EPI_ARGMAX only: as in TcParams
    int* arg_idx;
    float softcap;
};
// EPI_QKV_ROPE: staging of finished 16-column groups (two per half of the epilogue warps), positions and slots of the rows
constexpr int PAIR_ROPE_STAGE = 4 * 16 * TILE_W * 4, PAIR_ROPE_BYTES = PAIR_ROPE_STAGE + 4096;
constexpr int PAIR_ARG_BYTES = 2 * 4 * 256 * 8;  // EPI_ARGMAX: winners per accumulator, 32-row quarter and batch column
constexpr int pair_extra_bytes(int epi) { return epi == EPI_QKV_ROPE ? PAIR_ROPE_BYTES : epi == EPI_ARGMAX ? PAIR_ARG_BYTES : 0; }

// ---- PTX wrappers of the pair forms -----------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_rank(uint32_t saddr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
// Tile load into this CTA's shared memory that completes on the mbarrier at `bar` (an address of this CTA or its pair peer).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar)
        : "memory");
}
__device__ __forceinline__ void umma_f8_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f8f6f4 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc),
        "r"(accumulate)
        : "memory");
}
// Arrives on the barrier at this offset in the CTAs of `mask` once every MMA issued so far has completed.
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar, uint32_t mask) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                     smem_u32(bar)),
                 "h"((uint16_t)mask)
                 : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* holder) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(holder)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(512u) : "memory");
}
__device__ __forceinline__ void pair_epi_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

// M = 256 over the pair, N = bn, E4M3 x E4M3 -> F32, both operands K-major.
__device__ __forceinline__ uint32_t pair_instr_desc(int bn) { return (1u << 4) | ((uint32_t)(bn >> 3) << 17) | (16u << 24); }

template <int EPI, typename OutT>
__global__ void __launch_bounds__(PAIR_THREADS, 1)
fp8_gemm_pair_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_a, PairParams p) {
    constexpr bool ROPE = EPI == EPI_QKV_ROPE, ARG = EPI == EPI_ARGMAX, RES = EPI == EPI_RESIDUAL;
    extern __shared__ uint8_t raw[];
    uint8_t* header = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* ring = header + PAIR_HEADER + pair_extra_bytes(EPI);
    uint64_t* full = reinterpret_cast<uint64_t*>(header);  // leader: both CTAs' tiles of the stage have landed
    uint64_t* empty = full + PAIR_MAX_STAGES;              // both: the stage has been read
    uint64_t* acc_full = empty + PAIR_MAX_STAGES;          // both: accumulator b is complete
    uint64_t* acc_empty = acc_full + 2;                    // leader: accumulator b has been read by both CTAs
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 2);
    float* s_as = reinterpret_cast<float*>(header + 1024);  // [2][256] activation scales of the tile's batch rows
    int* s_pos = reinterpret_cast<int*>(header + PAIR_HEADER + PAIR_ROPE_STAGE);  // (ROPE) [2][256] positions, then slots
    int* s_slot = s_pos + 512;

    const int warp = rv::uniform_warp(), lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank(), half = rank & 1u, lead = rank & ~1u;
    const int S = p.splits, pair = (int)(rank >> 1);
    const int cluster_id = (int)blockIdx.x / (2 * S), clusters = (int)gridDim.x / (2 * S);
    const int BN = p.bn, STAGES = p.stages;
    const int b_rows = BN >> 1, b_bytes = b_rows * BK, stage_bytes = TILE_W * BK + b_bytes;
    // K block at which range v begins; ranges of this pair
    auto range_kb = [&](int v) -> int { return (int)((long long)v * p.kblocks / p.ranges); };
    auto first_range = [&](int q) -> int { return q * p.ranges / S; };
    const int v_lo = first_range(pair), my_parts = first_range(pair + 1) - v_lo;
    const int kb_lo = range_kb(v_lo), nkb = range_kb(v_lo + my_parts) - kb_lo;
    const int set_cols = p.npart * BN;

    if (threadIdx.x == 0) {
        rv::prefetch_map(&map_w);
        rv::prefetch_map(&map_a);
        for (int s = 0; s < STAGES; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int b = 0; b < 2; b++) {
            mbar_init(acc_full + b, 1);
            mbar_init(acc_empty + b, 2 * PAIR_EPI_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == 2) tmem_alloc_pair(tmem_holder);
    tc_fence_before();
    __syncthreads();
    cluster_arrive();
    cluster_wait();  // the pair's barriers exist, its tensor memory is allocated
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    // (after the allocation: a dependent kernel that starts now must not find tensor memory this grid still needs)
    rv::pdl_launch();

    if (warp == 0) {
        const uint32_t ring_addr = smem_u32(ring);
        const uint32_t full_addr = map_rank(smem_u32(full), lead);
        const bool one = rv::elect_one();
        int s = 0;
        uint32_t ph = 1;  // (a fresh barrier's previous phase counts as complete: the first pass over the ring does not wait)
        bool alive = true, waited = false;
        for (int t = cluster_id; t < p.tiles && alive; t += clusters) {
            const int n0 = (t / p.nb) * 256 + (int)half * TILE_W, m0 = (t % p.nb) * BN + (int)half * b_rows;
            // Weights never depend on the previous kernel: the first ring of weight tiles goes out before the wait
            // for it, the activation tiles of those stages follow.  (That is early only where this CTA found its SM empty:
            // its shared memory is the whole SM's, so it never starts beside a CTA of the kernel before it.)
            const int pre = waited ? 0 : (nkb < STAGES ? nkb : STAGES);
            if (!waited) {
                for (int i = 0; i < pre; i++) {
                    if (one) {
                        if (half == 0) mbar_expect_tx(full + i, 2u * (uint32_t)stage_bytes);
                        tma_load_2d_pair(ring_addr + (uint32_t)(i * stage_bytes), &map_w, (kb_lo + i) * BK, n0, full_addr + 8u * i);
                    }
                }
                rv::pdl_wait();
                waited = true;
                for (int i = 0; i < pre; i++)
                    if (one)
                        tma_load_2d_pair(ring_addr + (uint32_t)(i * stage_bytes) + TILE_W * BK, &map_a, (kb_lo + i) * BK, m0,
                                         full_addr + 8u * i);
                s = pre;
                if (s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
            for (int i = pre; i < nkb; i++) {
                alive = mbar_wait(empty + s, ph, 21);
                if (!alive) break;
                const uint32_t dst = ring_addr + (uint32_t)(s * stage_bytes);
                if (one) {
                    if (half == 0) mbar_expect_tx(full + s, 2u * (uint32_t)stage_bytes);
                    tma_load_2d_pair(dst, &map_w, (kb_lo + i) * BK, n0, full_addr + 8u * s);
                    tma_load_2d_pair(dst + TILE_W * BK, &map_a, (kb_lo + i) * BK, m0, full_addr + 8u * s);
                }
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
    } else if (warp == 1) {
        if (half == 0) {
            const uint32_t idesc = pair_instr_desc(BN), mask = 3u << rank;
            const uint64_t desc0 = smem_desc_sw128(smem_u32(ring)), desc_stage = (uint64_t)(stage_bytes >> 4);
            const bool one = rv::elect_one();
            int s = 0, b = 0;
            uint32_t ph = 0, set_ph = 1;  // (the first pass over the sets does not wait)
            bool alive = true;
            rv::pdl_wait();  // (the first product needs the activations: no bounded wait while the preceding kernel runs)
            for (int t = cluster_id; t < p.tiles && alive; t += clusters) {
                alive = mbar_wait_cluster(acc_empty + b, set_ph, 22);
                if (!alive) break;
                tc_fence_after();
                uint32_t acc = tmem_base + (uint32_t)(b * set_cols);
                int v = v_lo, next = range_kb(v_lo + 1) - kb_lo;
                bool first = true;
                for (int i = 0; i < nkb; i++) {
                    if (i == next) {  // the next range has an accumulator of its own
                        v++;
                        next = range_kb(v + 1) - kb_lo;
                        acc += (uint32_t)BN;
                        first = true;
                    }
                    alive = mbar_wait_cluster(full + s, ph, 23);
                    if (!alive) break;
                    tc_fence_after();
                    const uint64_t adesc = desc0 + desc_stage * (uint64_t)s, bdesc = adesc + (uint64_t)(TILE_W * BK >> 4);
                    if (one) {
#pragma unroll
                        for (int k = 0; k < BK / UMMA_K; k++)
                            umma_f8_pair(acc, adesc + (uint64_t)(k * UMMA_K >> 4), bdesc + (uint64_t)(k * UMMA_K >> 4), idesc,
                                         (!first || k > 0) ? 1u : 0u);
                        umma_commit_pair(empty + s, mask);
                    }
                    first = false;
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
                if (one) umma_commit_pair(acc_full + b, mask);
                if (++b == p.sets) {
                    b = 0;
                    set_ph ^= 1u;
                }
            }
        }
    }
    __syncwarp();

    const int ew = warp - PAIR_EPI_WARP0, quarter = warp & 3, wg = ew >> 2;
    const int r = quarter * 32 + lane, groups = BN >> 4;
    const uint32_t lane_addr = tmem_base + ((uint32_t)(quarter * 32) << 16);
    // one 16-column group: scale, residual, narrow, store (64 contiguous bytes of an output row per warp and column)
    auto store_group = [&](int m_base, int n, float ws, const float* as, const float* v, const unsigned short* res) {
        if (n >= p.N) return;
#pragma unroll
        for (int j = 0; j < 16; j++) {
            const int m = m_base + j;
            if (m < p.M) {
                const size_t o = (size_t)m * p.N + n;
                if constexpr (EPI == EPI_F32)
                    reinterpret_cast<float*>(p.out)[o] = as[j] * (ws * v[j]);
                else if constexpr (RES)
                    reinterpret_cast<OutT*>(p.out)[o] = rv::T16<OutT>::from_f32_sat(
                        fmaf(as[j], ws * v[j], rv::T16<OutT>::to_f32(*reinterpret_cast<const OutT*>(res + j))));
                else
                    reinterpret_cast<OutT*>(p.out)[o] = rv::T16<OutT>::from_f32_sat(as[j] * (ws * v[j]));
            }
        }
    };
    // 16 residual values as stored (rows past the end re-read the last one: a branch per element would serialise the
    // loads, which at M = 2048 cost the O projection 2.5 times its main loop)
    auto load_res = [&](int m_base, int n, unsigned short* res) {
        if constexpr (RES) {
            const unsigned short* src = reinterpret_cast<const unsigned short*>(p.residual) + (n < p.N ? n : p.N - 1);
#pragma unroll
            for (int j = 0; j < 16; j++) {
                const int m = m_base + j < p.M ? m_base + j : p.M - 1;
                res[j] = src[(size_t)m * p.N];
            }
        }
    };
    // Fused QKV epilogue: the weight tile of a CTA is one head (128 output channels), so a finished column group holds
    // whole heads of 16 tokens.  Round to the activation type (the bytes the unfused GEMM would have stored), exchange
    // through shared memory, then a warp per token: rotate (half-split pairs d, d + 64), head absmax, quantise, write Q or
    // the paged K / V row with its scale — the arithmetic of the RoPE + KV-write kernel.
    int rope_use = 0;
    auto rope_group = [&](int b, int g, int tile, int m_base, float ws, const float* as, const float* v) {
        if constexpr (ROPE) {
            const RopeKv& rk = p.rope;
            // An odd number of heads leaves the last pair's second CTA without one (the whole CTA returns: nobody waits below).
            if (tile >= rk.heads + 2 * rk.kv_heads) return;
            const int kind = tile < rk.heads ? 0 : (tile < rk.heads + rk.kv_heads ? 1 : 2);
            const int head = kind == 0 ? tile : (kind == 1 ? tile - rk.heads : tile - rk.heads - rk.kv_heads);
            float* stage = reinterpret_cast<float*>(header + PAIR_HEADER) + (size_t)((wg * 2 + (rope_use++ & 1)) * 16) * TILE_W;
            uint32_t cw[4], sw[4];
            int pos[4];
#pragma unroll
            for (int i = 0; i < 4; i++) {  // table entries of this warp's tokens, ahead of the exchange
                pos[i] = s_pos[b * 256 + g * 16 + quarter * 4 + i];
                cw[i] = sw[i] = 0u;
                if (kind != 2 && pos[i] >= 0 && pos[i] < rk.max_positions) {
                    const size_t e = (size_t)pos[i] * 32 + lane;  // this lane's pair of table elements
                    if (p.rope_pairs) {
                        cw[i] = __ldg(reinterpret_cast<const uint32_t*>(rk.cos_t) + e);
                        sw[i] = __ldg(reinterpret_cast<const uint32_t*>(rk.sin_t) + e);
                    } else {
                        const unsigned short *ct = reinterpret_cast<const unsigned short*>(rk.cos_t) + 2 * e,
                                             *st = reinterpret_cast<const unsigned short*>(rk.sin_t) + 2 * e;
                        cw[i] = (uint32_t)ct[0] | (uint32_t)ct[1] << 16;
                        sw[i] = (uint32_t)st[0] | (uint32_t)st[1] << 16;
                    }
                }
            }
#pragma unroll
            for (int j = 0; j < 16; j++)
                stage[j * TILE_W + r] = rv::T16<OutT>::to_f32(rv::T16<OutT>::from_f32_sat(as[j] * (ws * v[j])));
            asm volatile("bar.sync %0, 128;" ::"r"(2 + wg) : "memory");
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const int c = quarter * 4 + i, m = m_base + c;
                const bool live = m < p.M && pos[i] >= 0 && pos[i] < rk.max_positions;
                const float2 a = *reinterpret_cast<const float2*>(stage + c * TILE_W + 2 * lane);
                const float2 h = *reinterpret_cast<const float2*>(stage + c * TILE_W + 64 + 2 * lane);
                float2 lo = a, hi = h;
                if (kind != 2) {
                    const float2 cs = rv::T16<OutT>::to_f32x2(cw[i]), sn = rv::T16<OutT>::to_f32x2(sw[i]);
                    lo.x = a.x * cs.x - h.x * sn.x;
                    hi.x = a.x * sn.x + h.x * cs.x;
                    lo.y = a.y * cs.y - h.y * sn.y;
                    hi.y = a.y * sn.y + h.y * cs.y;
                }
                // (+inf carries "a value was not finite": an absmax of finite values never is)
                float am = fmaxf(fmaxf(fabsf(lo.x), fabsf(hi.x)), fmaxf(fabsf(lo.y), fabsf(hi.y)));
                if (!isfinite(lo.x) || !isfinite(hi.x) || !isfinite(lo.y) || !isfinite(hi.y)) am = CUDART_INF_F;
                am = rv::warp_max(am);
                const float sc = isinf(am) ? CUDART_NAN_F : fmaxf(am / 448.0f, 1e-12f);
                const float inv = 1.0f / sc;
                const uint32_t q = rv::f32x4_to_e4m3x4(lo.x * inv, lo.y * inv, hi.x * inv, hi.y * inv);
                if (!live) continue;
                uint8_t* o = nullptr;
                float* so = nullptr;
                if (kind == 0) {
                    o = rk.q_fp8 + ((size_t)m * rk.heads + head) * TILE_W;
                    so = rk.q_scale + (size_t)m * rk.heads + head;
                } else {
                    const int slot = s_slot[b * 256 + g * 16 + c];
                    if (slot < 0 || slot >= rk.num_cache_slots) continue;
                    const size_t sidx = (size_t)slot * rk.kv_heads + head;
                    o = (kind == 1 ? rk.k_cache : rk.v_cache) + sidx * TILE_W;
                    so = (kind == 1 ? rk.k_scale : rk.v_scale) + sidx;
                }
                if (p.rope_pairs) {
                    reinterpret_cast<unsigned short*>(o)[lane] = (unsigned short)(q & 0xffffu);
                    reinterpret_cast<unsigned short*>(o)[32 + lane] = (unsigned short)(q >> 16);
                } else {
                    o[2 * lane] = (uint8_t)q;
                    o[2 * lane + 1] = (uint8_t)(q >> 8);
                    o[64 + 2 * lane] = (uint8_t)(q >> 16);
                    o[65 + 2 * lane] = (uint8_t)(q >> 24);
                }
                if (lane == 0) *so = sc;
            }
        }
    };
    // Greedy-argmax epilogue: the best (value, channel) of each column over the warp's 32 channels.  Candidates are 64-bit
    // keys (the value's order-preserving code, then the complement of the channel, so that the lower channel wins a tie;
    // 0 = none), and the 16 columns are reduced by halving: 16 exchanges instead of 5 per column.
    unsigned long long* s_arg = reinterpret_cast<unsigned long long*>(header + PAIR_HEADER);
    auto arg_group = [&](int b, int g, int n, float ws, const float* as, const float* v) {
        if constexpr (ARG) {
            const float inv_cap = p.softcap > 0.0f ? 1.0f / p.softcap : 0.0f;
            unsigned long long k[16];
#pragma unroll
            for (int j = 0; j < 16; j++) {
                float val = as[j] * (ws * v[j]);
                if (p.softcap > 0.0f) val = p.softcap * tanhf(val * inv_cap);
                uint32_t u = __float_as_uint(val + 0.0f);  // (-0 and +0 are a tie)
                u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
                k[j] = (val == val && n < p.N) ? ((unsigned long long)u << 32 | (0xffffffffu - (uint32_t)n)) : 0ull;
            }
#pragma unroll
            for (int o = 16, h = 8; o > 1; o >>= 1, h >>= 1) {
                const bool up = (lane & o) != 0;
#pragma unroll
                for (int j = 0; j < h; j++) {
                    const unsigned long long mine = up ? k[j + h] : k[j];
                    const unsigned long long got = __shfl_xor_sync(0xffffffffu, up ? k[j] : k[j + h], o);
                    k[j] = mine > got ? mine : got;
                }
            }
            const unsigned long long got = __shfl_xor_sync(0xffffffffu, k[0], 1);
            const int col = ((lane >> 4) & 1) * 8 + ((lane >> 3) & 1) * 4 + ((lane >> 2) & 1) * 2 + ((lane >> 1) & 1);
            if ((lane & 1) == 0) s_arg[(size_t)(b * 4 + quarter) * 256 + g * 16 + col] = k[0] > got ? k[0] : got;
        }
    };
    // the tile's per-row operands into shared memory: activation scales and, for ROPE, positions and cache slots
    auto stage_rows = [&](int b, int et, int m0) {
        if (et < BN) {
            const bool in = m0 + et < p.M;
            s_as[b * 256 + et] = in ? p.a_scale[m0 + et] : 0.0f;
            if constexpr (ROPE) {
                s_pos[b * 256 + et] = in ? p.rope.positions[m0 + et] : -1;
                s_slot[b * 256 + et] = in ? p.rope.slot_mapping[m0 + et] : -1;
            }
        }
    };
    // sum of `n` accumulators BN columns apart, in order, added to v
    auto add_parts = [&](uint32_t col, int n, bool ready, float* v) {
#pragma unroll 1
        for (int i = 0; i < n; i++) {
            uint32_t u[16];
            tmem_ld16(lane_addr + col + (uint32_t)(i * BN), u);
            tmem_ld_wait();
#pragma unroll
            for (int j = 0; j < 16; j++) v[j] += ready ? __uint_as_float(u[j]) : 0.0f;
        }
    };
    const int et = (int)threadIdx.x - PAIR_EPI_WARP0 * 32;
    if (S == 1) {
        if (warp >= PAIR_EPI_WARP0) {
            rv::pdl_wait();
            int b = 0;
            uint32_t set_ph = 0;
            bool ready = true;
            for (int t = cluster_id; t < p.tiles; t += clusters) {
                const int m0 = (t % p.nb) * BN, n = (t / p.nb) * 256 + (int)half * TILE_W + r;
                // scales and the first residual group are fetched while the main loop runs
                const float* as = s_as + b * 256;
                stage_rows(b, et, m0);
                const float ws = n < p.N ? p.w_scale[n] : 0.0f;
                unsigned short res_nx[RES ? 16 : 1];
                load_res(m0 + wg * 16, n, res_nx);
                pair_epi_sync();
                if (ready) ready = mbar_wait(acc_full + b, set_ph, 24);
                tc_fence_after();
#pragma unroll 1
                for (int g = wg; g < groups; g += 2) {
                    uint32_t u[16];
                    float v[16];
                    unsigned short res[RES ? 16 : 1];
                    const uint32_t col = (uint32_t)(b * set_cols + g * 16);
                    tmem_ld16(lane_addr + col, u);
                    if constexpr (RES) {
#pragma unroll
                        for (int j = 0; j < 16; j++) res[j] = res_nx[j];
                        // (one group ahead: out may be the residual buffer, but no other thread writes these elements)
                        load_res(m0 + (g + 2 < groups ? g + 2 : g) * 16, n, res_nx);
                    }
                    tmem_ld_wait();
#pragma unroll
                    for (int j = 0; j < 16; j++) v[j] = ready ? __uint_as_float(u[j]) : 0.0f;
                    if (my_parts > 1) {
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = 0.0f + v[j];
                        add_parts(col + (uint32_t)BN, my_parts - 1, ready, v);
                    }
                    if (g + 2 >= groups) {  // last read of this accumulator: give it back before the stores
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive_peer(acc_empty + b, lead);
                    }
                    if constexpr (ROPE)
                        rope_group(b, g, n / TILE_W, m0 + g * 16, ws, as + g * 16, v);
                    else if constexpr (ARG)
                        arg_group(b, g, n, ws, as + g * 16, v);
                    else
                        store_group(m0 + g * 16, n, ws, as + g * 16, v, res);
                }
                if constexpr (ARG) {  // the tile's winner per batch row, over its four 32-channel quarters
                    pair_epi_sync();
                    const int wtiles = (p.N + TILE_W - 1) / TILE_W, wt = (t / p.nb) * 2 + (int)half;
                    if (et < BN && m0 + et < p.M && wt < wtiles) {
                        unsigned long long best = 0ull;
#pragma unroll
                        for (int q = 0; q < 4; q++) {
                            const unsigned long long c = s_arg[(size_t)(b * 4 + q) * 256 + et];
                            best = c > best ? c : best;
                        }
                        const uint32_t u = (uint32_t)(best >> 32);
                        const size_t o = (size_t)(m0 + et) * wtiles + wt;
                        p.arg_val[o] = best ? __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u) : -CUDART_INF_F;
                        p.arg_idx[o] = best ? (int)(0xffffffffu - (uint32_t)best) : -1;
                    }
                }
                if (++b == p.sets) {
                    b = 0;
                    set_ph ^= 1u;
                }
            }
        }
        rv::pdl_wait();
    } else {
        // Split-K: one tile per cluster.
        const int t = cluster_id, m0 = (t % p.nb) * BN, n = (t / p.nb) * 256 + (int)half * TILE_W + r;
        const bool epi = warp >= PAIR_EPI_WARP0;
        float ws = 0.0f;
        bool ready = true;
        rv::pdl_wait();
        if (epi) {
            stage_rows(0, et, m0);
            ws = n < p.N ? p.w_scale[n] : 0.0f;
            pair_epi_sync();
            ready = mbar_wait(acc_full, 0, 25);
            tc_fence_after();
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();  // every pair's MMAs are complete: the operand rings are idle
        const int gmax = (groups + S - 1) / S;  // column groups an owner finishes; receive slots [slot][gmax][16][128] f32
        // Pair 0's partials are a prefix of the sum and travel as one; every other pair sends its partials one by one, for
        // the owner to add them in order.
        auto sent_by = [&](int q) -> int { return q == 0 ? 1 : first_range(q + 1) - first_range(q); };
        if (epi) {
            int owner = wg % S, gi = wg / S;
#pragma unroll 1
            for (int g = wg; g < groups; g += 2) {
                if (owner != pair) {
                    int slot = 0;
                    for (int q = 0; q < pair; q++)
                        if (q != owner) slot += sent_by(q);
                    const int n_sent = sent_by(pair), per = pair == 0 ? my_parts : 1;
#pragma unroll 1
                    for (int i = 0; i < n_sent; i++) {
                        float v[16];
#pragma unroll
                        for (int j = 0; j < 16; j++) v[j] = 0.0f;
                        add_parts((uint32_t)(i * BN + g * 16), per, ready, v);
                        const uint32_t dst = map_rank(smem_u32(ring) + (uint32_t)(((((slot + i) * gmax + gi) * 16) * TILE_W + r) * 4),
                                                      (uint32_t)(owner * 2) + half);
#pragma unroll
                        for (int j = 0; j < 16; j++)
                            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst + (uint32_t)(j * TILE_W * 4)), "f"(v[j])
                                         : "memory");
                    }
                }
                owner += 2;
                while (owner >= S) {
                    owner -= S;
                    gi++;
                }
            }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();  // the partials are in place
        if (epi) {
            const float* recv = reinterpret_cast<const float*>(ring);
#pragma unroll 1
            for (int gi = wg; gi < gmax; gi += 2) {
                const int g = gi * S + pair;
                if (g >= groups) break;
                float v[16];
                unsigned short res[RES ? 16 : 1];
                load_res(m0 + g * 16, n, res);
#pragma unroll
                for (int j = 0; j < 16; j++) v[j] = 0.0f;
                int slot = 0;
#pragma unroll 1
                for (int q = 0; q < S; q++) {
                    if (q == pair) {
                        add_parts((uint32_t)(g * 16), my_parts, ready, v);
                    } else {
                        for (const int end = slot + sent_by(q); slot < end; slot++) {
                            const float* src = recv + (size_t)((slot * gmax + gi) * 16) * TILE_W + r;
#pragma unroll
                            for (int j = 0; j < 16; j++) v[j] += src[(size_t)j * TILE_W];
                        }
                    }
                }
                if constexpr (ROPE)
                    rope_group(0, g, n / TILE_W, m0 + g * 16, ws, s_as + g * 16, v);
                else
                    store_group(m0 + g * 16, n, ws, s_as + g * 16, v, res);
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    // nobody leaves while a peer may still signal its barriers, read its operands or write its ring
    cluster_arrive();
    cluster_wait();
    if (warp == 2) {
        tc_fence_after();
        tmem_dealloc_pair(tmem_base);
    }
}

// ---- host side --------------------------------------------------------------------------------------------------------
struct PairPlan {
    int bn, nb, tiles, splits, ranges, npart, sets;
};
// K ranges of a shape: up to 128 rows the split-K factor of the one-CTA form's plan for the batch tile (a power of two from
// 16) that holds the rows; above, whatever the distribution over pairs is (0).
inline int pair_ranges(int M, int N, int K) {
    if (M > 128) return 0;
    return pick_splits(M, N, K, M <= 16 ? 16 : M <= 32 ? 32 : M <= 64 ? 64 : 128);
}
// Most partials an owner receives when V ranges are dealt to S pairs (pair 0 sends one, the others all of theirs).
inline int pair_recv_slots(int V, int S) {
    int most = 0;
    for (int o = 0; o < S; o++) {
        int n = 0;
        for (int q = 0; q < S; q++)
            if (q != o) n += q == 0 ? 1 : (q + 1) * V / S - q * V / S;
        most = n > most ? n : most;
    }
    return most;
}
// Tile width and split-K factor of a shape: the cheapest of the candidates under a cost model in microseconds.  All widths are
// candidates: weights of few rows fill the chip only with narrow batch tiles (512 x 512 at 1400 rows: 12 tiles of 256 columns 10.8
// us, 88 of 32 5.7), and a short K spends its time in the epilogue between two tiles.  Over 16 weight shapes (512 x 512 to
// 43008 x 5376) and 9 batch sizes (48 to 2048) the choice is 2 % off the best width on average, 15 % at worst.
inline PairPlan pair_plan(int M, int N, int K, int ranges) {
    const int nw = (N + 255) / 256, kblocks = (K + BK - 1) / BK;
    PairPlan best = {};
    double best_cost = 0.0;
    // (many rows run at the power cap, where a narrower tile, which moves more and pads more, must be worth it, as must a split: 43008 x
    // 5376 at 1000 rows 158 us with 256 columns, 175 with 160, which the model puts 1 % ahead)
    const double worth = M > 512 ? 0.96 : 1.0;
    for (int bn = M > 224 ? 256 : (M + 31) / 32 * 32; bn >= 32; bn -= 32) {
        const int nb = (M + bn - 1) / bn, tiles = nw * nb;
        for (int S = 1; S <= 3; S++) {
            // (clusters of 4 and 6 CTAs: 32 and 21 of them were resident at once where measured, 35 and 25 were not)
            if (S > 1 && (tiles > (S == 2 ? 32 : 21) || kblocks / S < 2)) break;
            const int V = ranges > 0 ? ranges : S;
            const int npart = (V + S - 1) / S;
            // a tile's partials fit tensor memory; the receive slots (all partials but the owner's) fit the operand ring
            if (V < S || npart * bn > 512 || pair_recv_slots(V, S) * ((bn / 16 + S - 1) / S) * 8192 > 144 * 1024) continue;
            const int sets = 2 * npart * bn <= 512 ? 2 : 1;
            const int waves = S > 1 ? 1 : (tiles + PAIRS - 1) / PAIRS;
            const double per_kb = fmax(1.464e-3 * bn, 0.178 + 2.4e-4 * bn);  // tensor pipe / issue and feed of 128 bytes of K
            const double epi = 1.6 + 0.019 * bn + 2e-3 * bn * (npart - 1);  // an epilogue between two tiles
            double us = ((kblocks + S - 1) / S) * per_kb;
            us += (waves - 1) * (sets == 2 ? fmax(us, epi) : us + epi);  // (the last one's is in the constants below)
            us = fmax(us, (double)N * K / 7.88e6);  // the weights' stream
            us += 1.8 + 0.021 * bn + 2e-3 * bn * (npart - 1) + (S > 1 ? 0.86 + 8.2e-3 * bn * (1 + 0.5 * (npart - 1)) : 0.0);
            if (best.bn == 0 || us < worth * best_cost) {
                best = {bn, nb, tiles, S, V, npart, sets};
                best_cost = us;
            }
        }
    }
    return best;  // (V is at most 8: a width of 32 or 64 always fits)
}

// Which shapes the pair kernel takes.  Above 32 rows all of them: over the sweep of pair_plan() it is faster than the
// one-CTA form was from 33 rows on (43008 x 5376: equal up to 64 rows), 1.3 times at 96 rows, 2 to 4 times above 128.  Up
// to 32 rows only weights that the one-CTA form splits into more CTAs than are resident (three per SM), two uneven waves:
// 223 to 240 tiles of 128 rows, split in two.  Measured at 1, 8, 16, 17 and 32 rows, K 1024 to 8192, one-CTA time / pair
// time: there 1.10 to 1.67 (28672 x 4096: 26.3 / 21.8 us at one row, 32.7 / 22.7 at 32).  Next to it the one-CTA form wins
// or ties, its three small CTAs per SM start faster: 149 to 222 tiles 0.77 to 1.03 up to 16 rows (0.86 to 1.3 at 17 to 32,
// where the short K gain), 241 to 295 tiles, not split, 0.75 to 1.13, mostly 0.95 to 1.02.
inline bool prefer_pair(int M, int N, int K) {
    if (K % 16 != 0) return false;
    const int tiles = (N + TILE_W - 1) / TILE_W, splits = splits_of(tiles, (K + BK - 1) / BK, SPLIT_TARGET);
    return M > 32 || (splits > 1 && tiles * splits > 3 * rv::SMS);
}

template <int EPI, typename OutT>
int launch_pair_one(const TcArgs& g, const PairPlan& pl, cudaStream_t s, const RopeKv* rope = nullptr) {
    CUtensorMap mw, ma;
    if (!cached_map(&mw, g.w, g.N, g.K, TILE_W) || !cached_map(&ma, g.a, g.M, g.K, pl.bn / 2))
        return rvhost::fail_msg(-2, "cuTensorMapEncodeTiled failed (driver entry point missing or bad operand layout)");
    auto kern = fp8_gemm_pair_kernel<EPI, OutT>;
    constexpr int SMEM = 227 * 1024;  // the whole SM: nothing that allocates tensor memory may run beside this kernel
    static RvDeviceOnce smem_once;
    if (rv_allow_smem(smem_once, kern, SMEM))
        return rvhost::fail_msg(-2, "cannot raise dynamic shared memory for the pair GEMM");
    PairParams p;
    p.a_scale = g.a_scale;
    p.w_scale = g.w_scale;
    p.out = g.out;
    p.residual = g.residual;
    p.M = g.M;
    p.N = g.N;
    p.kblocks = (g.K + BK - 1) / BK;
    p.bn = pl.bn;
    p.nb = pl.nb;
    p.tiles = pl.tiles;
    p.splits = pl.splits;
    p.ranges = pl.ranges;
    p.npart = pl.npart;
    p.sets = pl.sets;
    p.rope = rope ? *rope : RopeKv{};
    p.rope_pairs = rope && rv_aligned(rope->cos_t, 4) && rv_aligned(rope->sin_t, 4) && rv_aligned(rope->q_fp8, 2) &&
                   rv_aligned(rope->k_cache, 2) && rv_aligned(rope->v_cache, 2);
    p.arg_val = g.arg_val;
    p.arg_idx = g.arg_idx;
    p.softcap = g.softcap;
    const int stage_bytes = TILE_W * BK + pl.bn / 2 * BK;
    p.stages = (SMEM - 1024 - PAIR_HEADER - pair_extra_bytes(EPI)) / stage_bytes;
    if (p.stages > PAIR_MAX_STAGES) p.stages = PAIR_MAX_STAGES;
    const int clusters = pl.splits > 1 ? pl.tiles : (pl.tiles < PAIRS ? pl.tiles : PAIRS);
    if (rv_launch(kern, dim3(clusters * 2 * pl.splits), dim3(PAIR_THREADS), SMEM, s, dim3(2 * pl.splits, 1, 1), mw, ma, p) !=
        cudaSuccess) {
        cudaGetLastError();
        return rvhost::fail_msg(-2, "pair GEMM launch failed");
    }
    return 0;
}

inline int launch_pair(const TcArgs& g, cudaStream_t s) {
    const PairPlan pl = pair_plan(g.M, g.N, g.K, pair_ranges(g.M, g.N, g.K));
    if (g.out_kind == 2) return launch_pair_one<EPI_F32, __half>(g, pl, s);
    if (g.out_kind == 0)
        return g.residual ? launch_pair_one<EPI_RESIDUAL, __half>(g, pl, s) : launch_pair_one<EPI_SCALE, __half>(g, pl, s);
    return g.residual ? launch_pair_one<EPI_RESIDUAL, __nv_bfloat16>(g, pl, s)
                      : launch_pair_one<EPI_SCALE, __nv_bfloat16>(g, pl, s);
}

// LM head with the greedy argmax in the epilogue: per-tile winners into arg_val / arg_idx (the merge is the caller's).
inline int launch_pair_argmax(const TcArgs& g, cudaStream_t s) {
    return launch_pair_one<EPI_ARGMAX, __half>(g, pair_plan(g.M, g.N, g.K, 1), s);
}

// QKV projection with RoPE, Q quantisation and the paged KV write in the epilogue, 33 to 128 rows; otherwise as
// rvtc::launch_qkv_rope.
inline int launch_pair_qkv_rope(const TcArgs& g, const RopeKv& rk, int dtype, cudaStream_t s) {
    if (g.K % 16 != 0 || g.M > 128 || g.N != (rk.heads + 2 * rk.kv_heads) * TILE_W)
        return rvhost::fail_msg(-3, "fused QKV epilogue: shape not taken");
    const PairPlan pl = pair_plan(g.M, g.N, g.K, pair_ranges(g.M, g.N, g.K));
    return dtype == 0 ? launch_pair_one<EPI_QKV_ROPE, __half>(g, pl, s, &rk)
                      : launch_pair_one<EPI_QKV_ROPE, __nv_bfloat16>(g, pl, s, &rk);
}

}  // namespace rvpair
