// FP8-KV paged GQA decode attention on tcgen05 / TMEM / TMA: one CTA, many (sequence, KV head) items.
//
// The form of paged_decode_fp8_umma.cuh for sequences that are not split: same contract, grid (kv_heads, 1, batch), tile arithmetic
// and partial layout (of one chunk).  What differs is how the grid's blocks become work.  A batch of short
// contexts is thousands of blocks of one or two tiles, each a chain of dependent latencies (launch, tensor memory,
// context length -> table -> TMA -> scores -> softmax -> product -> store) of 6-8 us around a microsecond of work.  Here a
// resident CTA takes over blocks that have not started (clusterlaunchcontrol.try_cancel, the hardware's own queue: no
// counters, nothing to reset) and runs them through the same ring, tensor memory and barriers:
//
//   warp 0   : scheduler and producer.  Claims the next block when it issues the last tile of the current one, looks up
//              the item's geometry, publishes it as a record in shared memory, issues the TMA loads of Q, K and V.  It runs
//              ahead of the other warps by the depth of the ring, across item boundaries.
//   warp 1   : MMA issuer, one stream of tiles over all items; the next item's score product runs under the current
//              item's softmax and epilogue.
//   warps 2-5: softmax and epilogue; while an item's last product runs they fetch the next item's scales.
//
// Blocks are handed out in grid order.  Where the grid takes more than one wave of CTAs and the contexts differ, that order is
// made the order of falling length (a permutation of the batch in shared memory), so that the longest sequences do not start last.
//
// What bounds it: the softmax warps' chain per item for short contexts (5 us of latencies per block become 2), the KV stream for
// long ones.
#pragma once
#include "paged_decode_fp8_umma.cuh"

namespace rvua {

constexpr int ITEM_SLOTS = 4;     // records in flight between the scheduler and the other warps
constexpr int ITEM_AUX_BYTES = 2048;

// A value that is the same in all lanes, in a uniform register (where the warp reduction leaves its result)
__device__ __forceinline__ int uniform(int v) { return (int)__reduce_or_sync(0xffffffffu, (unsigned)v); }

// ---- sequences by falling length ---------------------------------------------------------------------------------------
// Blocks start in grid order, the batch outermost.  Where the grid takes more than one wave, that order is made the order of
// falling length, so that the longest sequences do not start last (64 sequences of 512 to 32768 tokens, head_dim 256: 1614 us in the
// callers' order, 1290 in this one).  Nothing is kept: every CTA sorts the batch, by counting, in its first microsecond.
constexpr int ORDER_MAX = 256;  // sequences it is done for (a thread or two each)
// Keys that fall with the length (no window: all of it is attended), then with the sequence's number.  True if this thread saw two lengths.
__device__ __forceinline__ bool order_keys(const Params& p, int* key, int tid) {
    constexpr int cap = 0x7fffff;
    const int first = min(p.context_lens[0], cap);
    bool differ = false;
    for (int i = tid; i < ORDER_MAX; i += THREADS) {
        const int len = i < p.batch ? min(p.context_lens[i], cap) : 0;
        key[i] = i < p.batch ? (max(len, 0) << 8) + (ORDER_MAX - 1 - i) : -1;
        differ |= i < p.batch && len != first;
    }
    return differ;
}
// Rank of a sequence = how many keys are larger.
__device__ __forceinline__ void order_ranks(const Params& p, const int* key, uint8_t* perm, int tid) {
    for (int i = tid; i < p.batch; i += THREADS) {
        const int mine = key[i];
        int rank = 0;
        for (int j = 0; j < p.batch; j += 4) {
            const int4 k = *reinterpret_cast<const int4*>(key + j);
            rank += (k.x > mine ? 1 : 0) + (k.y > mine ? 1 : 0) + (k.z > mine ? 1 : 0) + (k.w > mine ? 1 : 0);
        }
        perm[rank] = (uint8_t)i;
    }
}

struct Item {
    int b, kvh;
    int t_begin, t_end, tile0, ntiles;  // ntiles 0: nothing attended (fill says what to store), -1: no more items
    int fill, pad;                      // 1: zeros, 2: NaN
};

// Claims a block of the grid that has not started; the 16-byte answer lands at `dst`, counted on `bar`.
__device__ __forceinline__ void claim_block(void* dst, uint64_t* bar) {
    asm volatile("clusterlaunchcontrol.try_cancel.async.shared::cta.mbarrier::complete_tx::bytes.b128 [%0], [%1];" ::"r"(smem_u32(dst)),
                 "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ bool claimed_block(const void* src, int& x, int& z) {
    uint32_t ok, bx = 0, by = 0, bz = 0;
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b128 r;\n\t"
        "ld.shared.b128 r, [%4];\n\t"
        "clusterlaunchcontrol.query_cancel.is_canceled.pred.b128 p, r;\n\t"
        "selp.u32 %3, 1, 0, p;\n\t"
        "mov.u32 %0, 0;\n\tmov.u32 %1, 0;\n\tmov.u32 %2, 0;\n\t"
        "@p clusterlaunchcontrol.query_cancel.get_first_ctaid.v4.b32.b128 {%0, %1, %2, _}, r;\n\t}"
        : "=&r"(bx), "=&r"(by), "=&r"(bz), "=r"(ok)
        : "r"(smem_u32(src))
        : "memory");
    x = (int)bx;
    z = (int)bz;
    return ok != 0;
}
// (try_wait may suspend the thread for a while: a loop that polls several barriers in turn tests instead)
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
// N consecutive TMEM columns of this thread's lane
template <int N> __device__ __forceinline__ void tmem_ldn(uint32_t taddr, uint32_t* r) {
    if constexpr (N == 1)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(r[0]) : "r"(taddr));
    else if constexpr (N == 2)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
    else if constexpr (N == 4)
        asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
                     : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                     : "r"(taddr));
    else
        tmem_ld8(taddr, r);
}

template <int N> __device__ __forceinline__ void tmem_stn(uint32_t taddr, const uint32_t* r) {
    if constexpr (N == 1)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x1.b32 [%0], {%1};" ::"r"(taddr), "r"(r[0]) : "memory");
    else if constexpr (N == 2)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x2.b32 [%0], {%1,%2};" ::"r"(taddr), "r"(r[0]), "r"(r[1]) : "memory");
    else if constexpr (N == 4)
        asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                     : "memory");
    else
        tmem_st8(taddr, r);
}

// Shared memory: ring, two Q buffers of the eight rows that can hold query heads, P tile, scratch.  The upper eight rows of the
// score product's B operand are zeros, and so are the last eight of P's 32: one block serves both, the stride between a Q
// buffer's two 8-row groups leads there.  With that, three units (four CTAs per SM) and four at head_dim 256 (three) fit.
template <int HD> struct ItemCfg : Cfg<HD> {
    using C = Cfg<HD>;
    static constexpr int QP = 8 * PANEL;                  // a panel of a Q buffer
    static constexpr int Q_BUFS = 2 * C::HALVES * QP;
    static constexpr int ZERO_AT = Q_BUFS + 24 * PANEL;   // from the first Q buffer
    static constexpr int smem_bytes(int units) { return units * UNIT + Q_BUFS + C::P_BYTES + ITEM_AUX_BYTES; }
    static __device__ __forceinline__ uint64_t q_desc(uint32_t q_addr, int buf, int h) {
        const int at = (buf * C::HALVES + h) * QP;
        uint64_t d = (uint64_t)(((q_addr + (uint32_t)at) & 0x3ffffu) >> 4);
        d |= (uint64_t)1 << 16;
        d |= (uint64_t)((ZERO_AT - at) >> 4) << 32;
        d |= (uint64_t)1 << 46;
        d |= (uint64_t)2 << 61;
        return d;
    }
};

template <int HD, int GT, typename OutT>
__global__ void __launch_bounds__(THREADS, HD == 512 ? 1 : ctas_per_sm<HD, GT>())
paged_decode_fp8_items_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                              const __grid_constant__ CUtensorMap map_q, Params p, int nunits, int ordered) {
    static_assert(HD == 128 || HD == 256 || HD == 512, "one, two or four 128-byte panels per cache row");
    static_assert(GT >= 1 && GT <= 8, "up to 8 query heads share the score tile");
    using C = ItemCfg<HD>;
    constexpr int HALVES = C::HALVES, UPT = C::UPT;
    const int NUNITS = nunits;
    constexpr int PSTRIDE = HD + 2;
    extern __shared__ __align__(1024) uint8_t item_smem[];
    uint8_t* ring = item_smem;                           // NUNITS x 16 KB
    uint8_t* q_tile = ring + NUNITS * UNIT;              // two of HALVES x [8 rows][128 B], swizzled
    uint8_t* p_tile = q_tile + C::Q_BUFS;                // [32 rows][128 token bytes], swizzled
    uint8_t* aux = p_tile + C::P_BYTES;
    uint64_t* full = reinterpret_cast<uint64_t*>(aux);   // [NUNITS] TMA landed
    uint64_t* empty = full + MAX_UNITS;                  // [NUNITS] MMAs that read the unit are done
    uint64_t* s_ready = empty + MAX_UNITS;               // [2] score tile in TMEM
    uint64_t* s_free = s_ready + 2;                      // [2] softmax has read the score tile
    uint64_t* p_ready = s_free + 2;                      // P tile written (and accumulator rescaled)
    uint64_t* pv_done = p_ready + 1;                     // the tile's second product has completed
    uint64_t* q_full = pv_done + 1;                      // [2] Q of an item landed
    uint64_t* q_free = q_full + 2;                       // [2] its score products are done
    uint64_t* item_full = q_free + 2;                    // [ITEM_SLOTS] record published
    uint64_t* item_free = item_full + ITEM_SLOTS;        // [ITEM_SLOTS] record read by the five other warps
    uint64_t* claim_bar = item_free + ITEM_SLOTS;        // the claimed block is known
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(claim_bar + 1);
    uint8_t* claim = aux + 384;                          // 16 bytes: answer of the last claim
    float* red = reinterpret_cast<float*>(aux + 400);    // [2][4][8] tile maxima, then [4][8] sums, [12] masks and flags (108 floats)
    Item* items = reinterpret_cast<Item*>(aux + 832);    // [ITEM_SLOTS]
    uint8_t* s_perm = aux + 1024;                        // [ORDER_MAX] sequences by falling length
    int* s_key = reinterpret_cast<int*>(ring);           // [ORDER_MAX] their sort keys, before the ring is used
    static_assert(384 >= (2 * MAX_UNITS + 10 + 2 * ITEM_SLOTS + 1) * 8 + 4 && 400 + 108 * 4 <= 832 &&
                      832 + ITEM_SLOTS * sizeof(Item) <= 1024 && 1024 + ORDER_MAX <= ITEM_AUX_BYTES, "scratch layout");

    rv::pdl_launch();
    const int tid = threadIdx.x, warp = rv::uniform_warp(), lane = tid & 31;
    const int group = p.heads / p.kv_heads;
    const int nh = group < GT ? group : GT;  // query heads of a KV head (the launcher guarantees group <= GT)
    const int bs = p.block_size;
    OutT* out = reinterpret_cast<OutT*>(p.out);

    // ---- set-up that does not depend on the preceding kernel ----
    if (tid == 0) {
        rv::prefetch_map(&map_k);
        rv::prefetch_map(&map_v);
        rv::prefetch_map(&map_q);
        for (int i = 0; i < NUNITS; i++) {
            mbar_init(full + i, 1);
            mbar_init(empty + i, 1);
        }
        for (int i = 0; i < 2; i++) {
            mbar_init(s_ready + i, 1);
            mbar_init(s_free + i, 4);
            mbar_init(q_full + i, 1);
            mbar_init(q_free + i, 1);
        }
        mbar_init(p_ready, 4);
        mbar_init(pv_done, 1);
        for (int i = 0; i < ITEM_SLOTS; i++) {
            mbar_init(item_full + i, 1);
            mbar_init(item_free + i, 5);
        }
        mbar_init(claim_bar, 1);
        fence_barrier_init();
    }
    if (warp == 1) tmem_alloc(tmem_holder, C::TMEM_COLS);
    for (int i = tid; i < (C::Q_BUFS + C::P_BYTES) / 16; i += THREADS)  // zero Q and P tiles (padding rows stay zero)
        reinterpret_cast<uint4*>(q_tile)[i] = make_uint4(0, 0, 0, 0);
    const bool early = p.early_meta != 0;
    if (!early) rv::pdl_wait();
    const bool differ = ordered && order_keys(p, s_key, tid);
    fence_proxy_async();  // the zeroes (and the keys in the ring) come before the tensor core's reads and the TMA's writes
    tc_fence_before();
    const bool reorder = __syncthreads_or(differ) != 0;
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    if (reorder) {
        order_ranks(p, s_key, s_perm, tid);
        fence_proxy_async();
        __syncthreads();
    }

    // physical block of the page holding `tok` (integer divisions only off the common power-of-two path)
    auto block_of = [&](const int* table, int tok) -> int {
        const int page = p.bs_shift >= 0 ? (tok >> p.bs_shift) : tok / bs;
        return table[p.window_size_left >= 0 ? page % p.max_blocks_per_seq : page];
    };

    // Waits until use `use` of ring unit `slot` has landed.  A parity wait cannot tell "this use has landed" from "the use before
    // last has", so the unit's previous occupant must be known to be consumed first; the one before that always is: the ring is
    // filled in order, and the unit in front of this one, which this role has seen landed or consumed, was sent after it was freed.
    auto landed = [&](int slot, int use, int site) -> bool {
        return (use == 0 || mbar_wait(empty + slot, (uint32_t)(use - 1) & 1u, site)) && mbar_wait(full + slot, (uint32_t)use & 1u, site);
    };

    if (warp == 0) {
        // ------------------------------------------------------------------ scheduler and producer (whole warp)
        // Lane j looks page j of every tile up; one elected lane issues the loads.
        const int ppt = TOK / bs;  // pages per tile (<= 16)
        int x = blockIdx.x, z = blockIdx.z;
        int slot = 0, use = 0;     // ring position of the next unit
        int n = 0, active = 0, q_sent = 0;  // items published, items with tiles among them, Q loads issued
        uint32_t claims = 0, answers = 0;
        bool alive = true, waited = !early, more = true;
        const bool one = rv::elect_one();
        auto wait_one = [&](uint64_t* bar, uint32_t parity, int site) { return __all_sync(0xffffffffu, mbar_wait(bar, parity, site)) != 0; };
        while (alive) {
            // (one value in all lanes: the loads below are issued by one elected lane from uniform registers)
            Item it;
            x = uniform(x);
            it.b = uniform(reorder ? (int)s_perm[z] : z);
            it.kvh = x;
            it.t_begin = it.t_end = it.tile0 = it.ntiles = it.fill = 0;
            if (more) {
                const int ctx = uniform(p.context_lens[it.b]);
                if (ctx <= 0 || (p.window_size_left < 0 && (long long)ctx > (long long)bs * p.max_blocks_per_seq)) {
                    it.fill = ctx == 0 ? 1 : 2;
                } else {
                    int start, len;
                    rvattn::attend_interval(ctx, p.window_size_left, start, len);
                    it.t_begin = start;
                    it.t_end = start + len;
                    it.tile0 = (it.t_begin / bs) * bs;  // first tile starts on a page boundary
                    it.ntiles = (it.t_end - it.tile0 + TOK - 1) / TOK;
                }
            } else {
                it.ntiles = -1;
            }
            const int sl = n & (ITEM_SLOTS - 1);
            // (the other warps read their first record after the dependency wait: no bounded wait for them ahead of it)
            if (n >= ITEM_SLOTS && !waited) {
                rv::pdl_wait();
                waited = true;
            }
            if (n >= ITEM_SLOTS) alive = wait_one(item_free + sl, (uint32_t)(n / ITEM_SLOTS - 1) & 1u, 11);
            if (!alive) break;
            if (lane == 0) {
                items[sl] = it;
                mbar_arrive(item_full + sl);
            }
            n++;
            if (!more) break;
            bool q_out = false;
            auto send_q = [&]() {  // Q comes from the preceding kernel
                if (!waited) rv::pdl_wait();
                waited = true;
                q_out = true;
                const int qb = active & 1;
                if (active >= 2) alive = wait_one(q_free + qb, (uint32_t)(active / 2 - 1) & 1u, 12);
                if (lane == 0 && alive) {
                    mbar_expect_tx(q_full + qb, (uint32_t)(nh * HD));
                    for (int h = 0; h < HALVES; h++)
                        tma_load_3d(smem_u32(q_tile + (qb * HALVES + h) * C::QP), &map_q, h * PANEL, 0, it.b * p.heads + it.kvh * group,
                                    smem_u32(q_full + qb));
                }
                q_sent += alive ? 1 : 0;
                __syncwarp();
            };
            if (waited && it.ntiles > 0) send_q();
            const int* table = p.block_tables + (size_t)it.b * p.max_blocks_per_seq;
            for (int i = 0; i < it.ntiles && alive; i++) {
                // (early: everything but Q and the newest token's K / V rows, which are in the last tile, is older than the
                // preceding kernel; Q goes out before the first wait that depends on the score products)
                if (!q_out && (i == it.ntiles - 1 || use > 0)) send_q();
                // pages of the tile that hold attended tokens; the rest are not fetched (their rows of the unit keep stale
                // bytes: masked in the scores, zeroed by the softmax warps for the V panels)
                const int np = min(ppt, (it.t_end - (it.tile0 + i * TOK) + bs - 1) / bs);
                int zz = 0;
                if (lane < np) {
                    const int ph = block_of(table, it.tile0 + i * TOK + lane * bs);
                    zz = (unsigned)ph < (unsigned)p.num_blocks_total ? ph * bs : 0;  // (the softmax warps poison the row)
                }
                if (i == it.ntiles - 1) {
                    if (lane == 0) {
                        fence_proxy_async();  // (the last answer was read through the generic proxy)
                        mbar_expect_tx(claim_bar, 16u);
                        claim_block(claim, claim_bar);
                    }
                    claims++;
                    __syncwarp();
                }
#pragma unroll 1
                for (int u = 0; u < UPT && alive; u++) {
                    if (use > 0) {
                        if (!q_out) send_q();
                        alive = alive && wait_one(empty + slot, (uint32_t)(use - 1) & 1u, 1);
                    }
                    if (!alive) break;
                    if (one) mbar_expect_tx(full + slot, (uint32_t)(np * bs * PANEL));
                    load_pages(smem_u32(ring) + (uint32_t)(slot * UNIT), bs * PANEL, u < HALVES ? &map_k : &map_v, (u % HALVES) * PANEL, it.kvh,
                               zz, np, one, smem_u32(full + slot));
                    if (++slot == NUNITS) {
                        slot = 0;
                        use++;
                    }
                }
            }
            if (!alive) break;
            if (it.ntiles > 0) {
                active++;
            } else {
                if (lane == 0) {
                    fence_proxy_async();
                    mbar_expect_tx(claim_bar, 16u);
                    claim_block(claim, claim_bar);
                }
                claims++;
                __syncwarp();
            }
            alive = wait_one(claim_bar, (claims - 1) & 1u, 13);
            answers = claims;
            more = __all_sync(0xffffffffu, alive && claimed_block(claim, x, z)) != 0;  // (after a refusal there is no further claim)
        }
        if (!waited) rv::pdl_wait();
        if (!alive) {  // a wait gave up: this warp's copies in flight land before the block leaves
            if (claims != answers) wait_one(claim_bar, (claims - 1) & 1u, 13);
            if (q_sent > 0) wait_one(q_full + ((q_sent - 1) & 1), (uint32_t)((q_sent - 1) / 2) & 1u, 12);
            for (int i = 0; i < NUNITS; i++) {
                const int last = i < slot ? use : use - 1;
                if (last >= 0) wait_one(full + i, (uint32_t)last & 1u, 1);
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        // Issue whichever product has its inputs first: the score MMA of the next tile (its K panels have landed and its TMEM
        // buffer is free) or the second product of the oldest open tile (its P tile is written and its V panels have landed).
        // Waiting for one in program order would hold the other back, and with it the release of the ring units the producer is
        // waiting for.  (The second product from a softmax warp, behind a barrier of the four: 15.3 against 14.5 us at 128
        // sequences of 48 tokens, head_dim 128, and 34.3 against 29.3 at 256.)
        const bool one = rv::elect_one();
        if (early) rv::pdl_wait();  // (the first product needs Q: the poll limit below must not run while the preceding kernel does)
        constexpr uint32_t idesc_qk = instr_desc(NQ, false), idesc_pv = instr_desc(NP, true);
        const uint64_t rdesc = desc_kmajor(smem_u32(ring)), vdesc0 = desc_mnmajor(smem_u32(ring)), pdesc = desc_kmajor(smem_u32(p_tile));
        // A product is issued when everything that it reads is there: its barriers are tested in one go, by the elected lane, which
        // a barrier that is not complete may suspend for a while.  (One barrier per stream and round, tested without suspension: a
        // product was seen to be ready up to three rounds late, and the warp took issue slots from the others.  256 sequences of
        // 4000 tokens, 64 / 8 heads, head_dim 128, three units: 548 us so, 518 this way.)
        int next_qk = 0, next_pv = 0;        // tiles, over all items
        int left = 0, item = 0, active = 0;  // score tiles left in the current item; records read; items with tiles begun
        uint32_t firsts = 0;                 // bit t & 7: tile t opens an item (next_qk runs at most three ahead of next_pv)
        uint32_t idle = 0;
        bool alive = true, ended = false, opens = false;
        // ring position (slot, use count) of the first K panel of tile next_qk and of the first V panel of tile next_pv
        int q_slot = 0, q_use = 0, v_slot = HALVES % NUNITS, v_use = HALVES / NUNITS;
        auto step = [&](int& slot, int& use, int by) {
            slot += by;
            while (slot >= NUNITS) {
                slot -= NUNITS;
                use++;
            }
        };
        // A unit's barrier may only be polled once the unit's previous occupant has been consumed here:
        // a parity wait cannot tell "this use has landed" from "the use before last has", so polling
        // while the previous use is still loading would report the data as present.
        auto prev_consumed = [&](int g) {
            g -= NUNITS;
            if (g < 0) return true;
            const int tile = g / UPT;
            return g % UPT < HALVES ? tile < next_qk : tile < next_pv;
        };
        while (alive && !(ended && next_pv == next_qk)) {
            bool did = false;
            // ---- scores: a record, then the TMEM buffer, Q and the K panels ----
            if (left == 0) {
                const int sl = item & (ITEM_SLOTS - 1);
                if (!ended && __all_sync(0xffffffffu, mbar_test(item_full + sl, (uint32_t)(item / ITEM_SLOTS) & 1u))) {
                    const int t = items[sl].ntiles;
                    __syncwarp();
                    if (lane == 0) mbar_arrive(item_free + sl);
                    item++;
                    ended = t < 0;
                    left = t > 0 ? t : 0;
                    opens = t > 0;
                    active += t > 0 ? 1 : 0;
                    did = true;
                }
            } else {
                const int i = next_qk, qb = (active - 1) & 1;
                bool ok = one && (i < 2 || mbar_try_wait(s_free + (i & 1), (uint32_t)((i >> 1) - 1) & 1u));
                if (opens) ok = ok && mbar_try_wait(q_full + qb, (uint32_t)((active - 1) / 2) & 1u);
                int slot[HALVES];
#pragma unroll
                for (int h = 0; h < HALVES; h++) {
                    int sl = q_slot + h, us = q_use;
                    if (sl >= NUNITS) {
                        sl -= NUNITS;
                        us++;
                    }
                    slot[h] = sl;
                    ok = ok && prev_consumed(i * UPT + h) && mbar_try_wait(full + sl, (uint32_t)us & 1u);
                }
                if (__any_sync(0xffffffffu, ok)) {
                    tc_fence_after();
                    left--;
                    if (one) {
#pragma unroll
                        for (int h = 0; h < HALVES; h++) {
                            const uint64_t kdesc = rdesc + (uint64_t)((slot[h] * UNIT) >> 4), qd = C::q_desc(smem_u32(q_tile), qb, h);
#pragma unroll
                            for (int k = 0; k < PANEL / 32; k++)
                                umma_f8(tmem_base + (uint32_t)(i & 1) * NQ, kdesc + (uint64_t)(2 * k), qd + (uint64_t)(2 * k), idesc_qk,
                                        (h > 0 || k > 0) ? 1u : 0u);
                            umma_commit(empty + slot[h]);
                        }
                        umma_commit(s_ready + (i & 1));
                        if (left == 0) umma_commit(q_free + qb);
                    }
                    firsts = (firsts & ~(1u << (i & 7))) | ((opens ? 1u : 0u) << (i & 7));
                    opens = false;
                    next_qk++;
                    step(q_slot, q_use, UPT);
                    did = true;
                }
            }
            // ---- second product: the P tile and the V panels ----
            if (next_pv < next_qk) {
                const int i = next_pv;
                bool ok = one && mbar_try_wait(p_ready, (uint32_t)i & 1u);
                int slot[HALVES];
#pragma unroll
                for (int h = 0; h < HALVES; h++) {
                    int sl = v_slot + h, us = v_use;
                    if (sl >= NUNITS) {
                        sl -= NUNITS;
                        us++;
                    }
                    slot[h] = sl;
                    ok = ok && prev_consumed(i * UPT + HALVES + h) && mbar_try_wait(full + sl, (uint32_t)us & 1u);
                }
                if (__any_sync(0xffffffffu, ok)) {
                    tc_fence_after();
                    if (one) {
                        const uint32_t add = (firsts >> (i & 7)) & 1u ? 0u : 1u;
#pragma unroll
                        for (int h = 0; h < HALVES; h++) {
                            const uint64_t vdesc = vdesc0 + (uint64_t)((slot[h] * UNIT) >> 4);
#pragma unroll
                            for (int k = 0; k < TOK / 32; k++)
                                umma_f8(tmem_base + C::O_COL + (uint32_t)h * NP, vdesc + (uint64_t)((32 * PANEL * k) >> 4),
                                        pdesc + (uint64_t)(2 * k), idesc_pv, k > 0 ? 1u : add);
                            umma_commit(empty + slot[h]);
                        }
                        umma_commit(pv_done);
                    }
                    next_pv++;
                    step(v_slot, v_use, UPT);
                    did = true;
                }
            }
            if (did) {
                idle = 0;
            } else if (++idle > WAIT_LIMIT) {
                if (one) atomicCAS(&g_status, 0, (2 << 16) | (int)(blockIdx.x & 0xffff));
                alive = false;
            }
        }
    } else {
        // ------------------------------------------------------------------ softmax (128 threads)
        const int quarter = warp & 3;             // TMEM lanes this warp may touch: 32 * quarter ..
        const int row = quarter * 32 + lane;      // token of the tile (scores) / head dim of the panel (accumulator)
        const uint32_t lane_base = tmem_base + ((uint32_t)(quarter * 32) << 16);
        const bool k_perslot = p.k_scale_cache != nullptr, v_perslot = p.v_scale_cache != nullptr;
        float* sums = red + 64;                                // [4][8]
        unsigned* bads = reinterpret_cast<unsigned*>(red + 96);  // [4] heads whose result is NaN, then [2][4] a wait gave up
        int g = 0, n = 0;                  // tiles so far, records read
        int v_slot = HALVES % NUNITS, v_use = HALVES / NUNITS;  // ring position of tile g's first V panel
        bool alive = true;
        int b = 0, kvh = 0, t_begin = 0, t_end = 0, tile0 = 0, ntiles = -1;
        auto next_item = [&]() {
            const int sl = n & (ITEM_SLOTS - 1);
            alive = alive && mbar_wait(item_full + sl, (uint32_t)(n / ITEM_SLOTS) & 1u, 14);
            const Item& it = items[sl];
            b = it.b;
            kvh = it.kvh;
            t_begin = it.t_begin;
            t_end = it.t_end;
            tile0 = it.tile0;
            ntiles = alive ? it.ntiles : -1;
            n++;
        };
        // The four warps leave together: whether a wait has given up is agreed on once per record, where they meet.
        auto meet = [&]() {
            unsigned* gave_up = bads + 4 + 4 * (n & 1);
            if (lane == 0) gave_up[warp - 2] = alive ? 0u : 1u;
            bar_softmax();
            alive = (gave_up[0] | gave_up[1] | gave_up[2] | gave_up[3]) == 0;
            if (!alive) ntiles = -1;
        };
        auto drop_item = [&](int i) {  // record i has been read for the last time
            __syncwarp();
            if (lane == 0) mbar_arrive(item_free + (i & (ITEM_SLOTS - 1)));
        };
        // this thread's token of a tile: validity, block, K / V scales; a table entry outside the cache poisons the whole row
        unsigned bad = 0;
        bool valid_n = false;
        float ks_n = 0.0f, vs_n = 0.0f;
        auto fetch = [&](int i) {
            const int tok = tile0 + i * TOK + row;
            valid_n = i < ntiles && tok >= t_begin && tok < t_end;
            if (valid_n) {
                int ph = block_of(p.block_tables + (size_t)b * p.max_blocks_per_seq, tok);
                if ((unsigned)ph >= (unsigned)p.num_blocks_total) {
                    bad = 0xffffffffu;
                    ph = 0;
                }
                const size_t sidx = ((size_t)ph * bs + (tok % bs)) * p.kv_heads + kvh;
                ks_n = k_perslot ? p.k_scale_cache[sidx] : *p.k_descale;
                vs_n = v_perslot ? p.v_scale_cache[sidx] : *p.v_descale;
            }
        };
        float qsc[GT];  // q scale * softmax scale * log2(e): the softmax runs in base 2
        auto open_item = [&]() {  // what the first tile of an item needs, requested together
            bad = 0;
#pragma unroll
            for (int k = 0; k < GT; k++) {
                qsc[k] = 0.0f;
                if (k < nh) {
                    const int head = kvh * group + k;
                    qsc[k] = p.q_scale_cache ? p.q_scale_cache[(size_t)b * p.heads + head] : *p.q_descale;
                }
            }
            fetch(0);
        };
        if (early) rv::pdl_wait();  // the newest token's scales and Q's come from the preceding kernel
        next_item();
        meet();
        if (ntiles > 0) open_item();
        while (ntiles >= 0) {
            const int cur = n - 1;  // the record is kept until the item's results are stored
            if (ntiles == 0) {
                const float fill = items[cur & (ITEM_SLOTS - 1)].fill == 1 ? 0.0f : CUDART_NAN_F;
                const size_t head0 = (size_t)b * p.heads + (size_t)kvh * group;
                if (p.force_partial) {
                    for (int i = tid - 64; i < group * PSTRIDE; i += 128) {
                        const int d = i % PSTRIDE;
                        p.workspace[head0 * PSTRIDE + i] = d < HD ? fill : (d == HD ? -1e20f : 0.0f);
                    }
                } else {
                    for (int i = tid - 64; i < group * HD; i += 128) out[head0 * HD + i] = rv::T16<OutT>::from_f32(fill);
                }
                drop_item(cur);
                next_item();
                meet();
                if (ntiles > 0) open_item();
                continue;
            }
            float m_run[GT], l_part[GT];
#pragma unroll
            for (int k = 0; k < GT; k++) {
                m_run[k] = -1e20f;
                l_part[k] = 0.0f;
                if (k < nh && rvattn::bad_scale(qsc[k])) bad |= 1u << k;
                qsc[k] = qsc[k] * p.scale * 1.4426950408889634f;
            }
            for (int i = 0; i < ntiles; i++, g++) {  // (no way out: the warps meet in every tile)
                const bool valid = valid_n;
                const float ks = ks_n, vs = vs_n;
                fetch(i + 1);
                if (valid && (rvattn::bad_scale(ks) || rvattn::bad_scale(vs))) bad = 0xffffffffu;
                const float lv = valid ? __log2f(vs) : 0.0f;
                // ---- scores of this token ----
                alive = alive && mbar_wait(s_ready + (g & 1), (uint32_t)(g >> 1) & 1u, 6);
                tc_fence_after();
                uint32_t sraw[GT];
                tmem_ldn<GT>(lane_base + (uint32_t)(g & 1) * NQ, sraw);
                tmem_ld_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(s_free + (g & 1));
                float s2[GT];  // base-2 score without / with the V scale folded in
                float* mx = red + (g & 1) * 32 + (warp - 2) * 8;
#pragma unroll
                for (int k = 0; k < GT; k++) {
                    float s = __uint_as_float(sraw[k]) * qsc[k] * ks;
                    if (valid && k < nh && !isfinite(s)) {
                        bad |= 1u << k;
                        s = -1e30f;
                    }
                    s2[k] = valid ? s : -1e30f;
                    const float wm = rv::warp_max(s2[k] + lv);
                    if (lane == 0) mx[k] = wm;
                }
                bar_softmax();
                float corr[GT];
                bool moved = false;
                uint8_t term[GT][3];
#pragma unroll
                for (int k = 0; k < GT; k++) {
                    const float* all = red + (g & 1) * 32 + k;
                    const float tm = fmaxf(fmaxf(all[0], all[8]), fmaxf(all[16], all[24]));
                    const float m_new = fmaxf(m_run[k], tm);
                    corr[k] = fast_exp2(m_run[k] - m_new);
                    moved |= k < nh && m_new > m_run[k];
                    m_run[k] = m_new;
                    const float x = valid ? fast_exp2(s2[k] + lv - m_new + 8.0f) : 0.0f;  // p * v_scale, in (0, 256]
                    const float y = valid ? fast_exp2(s2[k] - m_new + 8.0f) : 0.0f;       // p, same normalisation
                    l_part[k] = l_part[k] * corr[k] + y;
                    split3(x, term[k][0], term[k][1], term[k][2]);
                }
                // ---- the previous tile's second product must be done before P is overwritten / O rescaled (the one
                // before an item's first tile was awaited by that item's epilogue) ----
                if (i > 0) alive = alive && mbar_wait(pv_done, (uint32_t)(g - 1) & 1u, 7);
#pragma unroll
                for (int k = 0; k < GT; k++)
                    if (k < nh) {
                        const uint32_t off = (uint32_t)((((row >> 4) ^ k) << 4) + (row & 15));
#pragma unroll
                        for (int t = 0; t < 3; t++) p_tile[(t * 8 + k) * PANEL + off] = term[k][t];
                    }
                // rows of the tile outside the attended interval: zero their V bytes (stale cache bytes may be NaN codes; a
                // lane starts at a chunk of its own, so that eight lanes' stores cover all banks)
                if (tile0 + i * TOK < t_begin || tile0 + (i + 1) * TOK > t_end) {
                    int sh = v_slot, us = v_use;
#pragma unroll
                    for (int h = 0; h < HALVES; h++) {
                        alive = alive && landed(sh, us, 8);
                        if (alive && !valid) {
                            uint4* vrow = reinterpret_cast<uint4*>(ring + (size_t)sh * UNIT + row * PANEL);
#pragma unroll
                            for (int c = 0; c < PANEL / 16; c++) vrow[(c + lane) & 7] = make_uint4(0, 0, 0, 0);
                        }
                        if (++sh == NUNITS) {
                            sh = 0;
                            us++;
                        }
                    }
                }
                if (i > 0 && moved) {  // block-uniform: every thread sees the same maxima
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < HALVES; h++)
#pragma unroll
                        for (int t = 0; t < 3; t++) {
                            uint32_t o[GT];
                            const uint32_t addr = lane_base + C::O_COL + (uint32_t)(h * NP + t * 8);
                            tmem_ldn<GT>(addr, o);
                            tmem_ld_wait();
#pragma unroll
                            for (int k = 0; k < GT; k++) o[k] = __float_as_uint(__uint_as_float(o[k]) * corr[k]);
                            tmem_stn<GT>(addr, o);
                        }
                    tmem_st_wait();
                }
                fence_proxy_async();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(p_ready);
                v_slot += UPT;
                while (v_slot >= NUNITS) {
                    v_slot -= NUNITS;
                    v_use++;
                }
            }
            // ---- epilogue: accumulator (thread = head dim) / denominators -> output or partial ----
            float* my_sums = sums + (warp - 2) * 8;
#pragma unroll
            for (int k = 0; k < GT; k++) {
                const float ws = rv::warp_sum(l_part[k]);
                if (lane == 0) my_sums[k] = ws;
            }
            bad = __reduce_or_sync(0xffffffffu, bad);
            if (lane == 0) bads[warp - 2] = bad;
            // the next item's record and what its first tile needs, while the last product runs
            next_item();
            if (ntiles > 0) open_item();
            if (alive) alive = mbar_wait(pv_done, (uint32_t)(g - 1) & 1u, 9);
            tc_fence_after();
            meet();
            const unsigned bad_mask = alive ? (bads[0] | bads[1] | bads[2] | bads[3]) : 0xffffffffu;
            const Item& it = items[cur & (ITEM_SLOTS - 1)];
            const size_t head0 = (size_t)it.b * p.heads + (size_t)it.kvh * group;
#pragma unroll
            for (int h = 0; h < HALVES; h++) {
                float acc[GT];
                uint32_t o[3][GT];
#pragma unroll
                for (int t = 0; t < 3; t++) tmem_ldn<GT>(lane_base + C::O_COL + (uint32_t)(h * NP + t * 8), o[t]);
                tmem_ld_wait();
#pragma unroll
                for (int k = 0; k < GT; k++) {
                    acc[k] = 0.0f;
#pragma unroll
                    for (int t = 0; t < 3; t++) acc[k] += __uint_as_float(o[t][k]);
                }
                const int d = h * PANEL + row;
#pragma unroll
                for (int k = 0; k < GT; k++)
                    if (k < nh) {
                        const float L = sums[k] + sums[8 + k] + sums[16 + k] + sums[24 + k];
                        const bool any_bad = (bad_mask >> k) & 1u;
                        if (!p.force_partial) {
                            float v = L > 0.0f ? acc[k] / L : acc[k];
                            if (any_bad) v = CUDART_NAN_F;
                            out[(head0 + k) * HD + d] = rv::T16<OutT>::from_f32(v);
                        } else {
                            float* ws = p.workspace + (head0 + k) * PSTRIDE;
                            ws[d] = any_bad ? CUDART_NAN_F : acc[k];
                            if (d == 0) {
                                ws[HD] = (m_run[k] - 8.0f) * 0.6931471805599453f;  // back to base e
                                ws[HD + 1] = any_bad ? CUDART_NAN_F : L;
                            }
                        }
                    }
            }
            tc_fence_before();
            drop_item(cur);
        }
    }
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, C::TMEM_COLS);
    }
}

// ---- host side -------------------------------------------------------------------------
// Which launches take this kernel: one chunk per sequence and more blocks than the one-item kernel keeps resident at once; with a
// window, where nothing is reordered, from two waves on.  Lengths are not known here, and what it gives depends on them.  Measured,
// us, one-item kernel (in the callers' order) / this one, 16-token pages:
//   short       128 sequences of 48 tokens, 16 KV heads, head_dim 128 28.7 / 20.6; 256 of 516 123.0 / 114.1; 64 of 516, head_dim 512
//               143 / 125
//   unequal     64 of 500 to 16000, head_dim 128 397 / 381; 64 of 100 to 4000, 64 / 8 heads 105 / 72, head_dim 512 266 / 200, 32 / 16
//               heads 360 / 335
//   with a window of 1024: 256 of 16 to 400 tokens, head_dim 128 69.7 / 62.0; 256 of 100 to 4000, 64 / 8 heads, head_dim 256 229 / 215
//   equal, long 64 of 2000, 16 KV heads, head_dim 128 102.7 / 106.6; 256 of 4000 652 / 690, with a window of 1024 184 / 192; 128 of 4000,
//               64 / 8 heads, head_dim 256 390 / 382
// So the cost is with equal long contexts at head_dim 128 and one or two query heads per KV head, which stream at the copy rate in
// either kernel: 3 to 6 %.  Over 1018 shapes with 20 to 256 sequences, grids of one wave among them, the time is 0.92 on average.
// A grid that is resident at once gains nothing and pays for the records and claims: 33 sequences of 22 to 411 tokens 12.0 / 13.3.
// So do grids whose blocks are chunks that short sequences leave empty (15 sequences of up to 56 tokens, a whole layer
// 126.5 / 132.8), and the form that leaves maxima for the O projection, which is part of a chain of dependent launches (32 rows, a
// 12-layer stack: 1465 / 1476 us per step).
template <int HD, int GT> inline bool prefer_items(const Params& p) {
    if (p.max_chunks > 1 || p.amax_out) return false;
    const long long ctas = (long long)p.kv_heads * p.batch;
    const int fit = (228 * 1024) / (Cfg<HD>::smem_bytes(pick_units<Cfg<HD>>(ctas, ctas_per_sm<HD, GT>())) + 1024);
    const long long resident = (long long)(fit < ctas_per_sm<HD, GT>() ? fit : ctas_per_sm<HD, GT>()) * rv::SMS;
    return ctas > (p.window_size_left < 0 ? resident : 2 * resident);
}

}  // namespace rvua
