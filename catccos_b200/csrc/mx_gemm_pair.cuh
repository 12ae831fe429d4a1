// MXFP8 block-scaled GEMM on CTA pairs (clusters of two SMs, tcgen05 cta_group::2).
//
// Same operator, operands, layouts and flag gating as mx_gemm.cuh; what changes is the tile: a pair of
// CTAs owns a 256 x 256 output tile.  CTA r of the pair loads A rows [m0 + 128 r, +128) and B columns
// [n0 + 128 r, +128) of every K tile (32 KB per K tile per SM instead of 48 KB; a ragged last column of tiles is split
// in two halves of what it has), the leader CTA (r = 0)
// issues one tcgen05.mma.cta_group::2 (M = 256, N = 256, K = 32) that reads both CTAs' shared memory, and
// each CTA ends up with the accumulator of its own 128 rows x 256 columns in its own tensor memory.
// Every CTA loads its own tiles with plain TMA (no cluster multicast anywhere); what crosses the pair is
// only barrier traffic:
//   full[s]                     lives in the leader; both CTAs' TMA bytes go there
//   empty[s], tmem_full[a]      live in each CTA; the leader's tcgen05.commit arrives on both copies
//   tmem_empty[a], overlap_free[a]  live in the leader; the epilogue warps of both CTAs arrive there
//   atoms[b], sf_full[b]        live in the leader, sf_empty[b] in each CTA: see below
//
// Two rings.  The operand ring carries nothing but TMA and is as deep as shared memory allows.  The scale factors have a
// ring of their own that moves in groups of four K tiles: the scale-loader warps load the E8M0 bytes one group ahead into
// registers, write the atoms, and an elected lane of each of the leader's warps copies one K tile's atoms of both CTAs
// into tensor memory; two groups are in flight.
//
// What bounds it: about 600 SM cycles per K tile against 512 of MMA (slope over K, whole tiles; 8192 x 2304 and
// 16384 x 3456 at 1.46 GHz under the power cap, 1024 x 2304 at 1.965 GHz: 601, 587, 601 cycles).  It is not the ring's
// depth: five stages take 616, 580, 611, four 625, 601, 751.  Which of the rest it is has not been shown: a K tile moves
// 32 KB into and 32 KB out of each SM's shared memory (500 cycles at 128 bytes), and 51 bytes per cycle and SM leave L2.
// The cycles are the same under the power cap, which lowers the clock.  Pairs on 256 x 128 tiles (48 KB per 256 MMA
// cycles) were measured 1.4 to 1.6 times slower.
// Measured (B200, kernel alone, three operand sets in turn, 40 calls queued behind an idle GPU, so near the full clock; in
// brackets a second without a pause, at 1.3 to 1.8 GHz), against one ring of five stages that also carried the scales, no split
// behind whole tiles, and stores straight from registers: 1024 x 2304 x 7168 27.0 -> 21.5 us (26.7 -> 22.3), 3001 x 2064 x
// 5120 42.3 -> 32.3 (44.6 -> 37.9), 4096 x 3456 x 5120 68.0 -> 57.2 (77.0 -> 67.8), 8192 x 2304 x 7168 103.5 -> 96.0
// (122 -> 113), 32768 x 3456 x 5120 440 -> 414 (515 -> 488).
//
// Work units.  num_tiles = rounds * pairs + rem: the rem tiles that would leave pairs idle in a round of their own are
// cut into ksplit parts along K, one (tile, part) per pair, and every pair takes `rounds` whole tiles.  The parts
// exchange fp32 pieces through the rank's split-K scratch: every part owns an equal share of the tile's 32-column chunks
// and adds the parts' pieces in a fixed order, so the result does not depend on timing.  A pair with whole tiles starts
// with its part: the exchange (4 to 6 us when it comes last) then passes beside the products of the tiles that follow.
// A gated launch (flags) ends with it, because its last tiles' rows arrive last.
#pragma once

#include "mx_gemm.cuh"

namespace catccos {

constexpr uint32_t kPairBlockM = 256;
constexpr uint32_t kPairBlockN = 256;
constexpr uint32_t kSfGroup = 4;  // K tiles whose scale factors travel together (one per scale-loader warp)

struct PairSmem {
    static constexpr uint32_t kStages = 6;
    static constexpr uint32_t kABytes = 128 * kGemmBlockK;  // this CTA's 128 rows
    static constexpr uint32_t kBBytes = 128 * kGemmBlockK;  // this CTA's 128 columns
    static constexpr uint32_t kSfaBytes = 512;              // per K tile
    static constexpr uint32_t kSfbBytes = 1024;  // all 256 columns: each CTA multiplies by the whole N tile
    static constexpr uint32_t kSfBufBytes = kSfGroup * (kSfaBytes + kSfbBytes);
    static constexpr uint32_t kOffA = 0;
    static constexpr uint32_t kOffB = kOffA + kStages * kABytes;
    static constexpr uint32_t kOffOut = kOffB + kStages * kBBytes;
    static constexpr uint32_t kOffSf = kOffOut + 4 * kOutStageBytes;
    static constexpr uint32_t kOffBar = kOffSf + 2 * kSfBufBytes;
    // full[S], empty[S], tmem_full[2], tmem_empty[2], overlap_free[2], sf_full[2], sf_empty[2], atoms[2], red[4]
    static constexpr uint32_t kNumBars = 2 * kStages + 12 + 4;
    static constexpr uint32_t kOffTmemPtr = kOffBar + kNumBars * 8;
    static constexpr uint32_t kOffGate = kOffTmemPtr + 8;  // K-tile iterations whose rows this CTA's producer has seen ready
    static constexpr uint32_t kBytes = kOffTmemPtr + 16;
    static constexpr uint32_t kDynamicBytes = kBytes + 1024;
    static_assert(kDynamicBytes <= 232448, "one CTA's shared memory");
    static_assert(4 * kSplitRedBytes <= kOffOut, "the split-K pieces land in the idle operand stages");
    static_assert(4 * 4 * kOutStageBytes <= kOffOut, "the last tile's output is staged in the idle operand stages");
    // Tensor memory: two 256-column accumulators that share 96 columns (the epilogue drains those first and then lets
    // the next tile start), and two groups of four scale sets (SFA 4 + SFB 8 columns).
    static constexpr uint32_t kAccCol1 = 160;
    static constexpr uint32_t kSfCol = 416;
    static constexpr uint32_t kSfSetCols = 12;
    static constexpr uint32_t kSfGroupCols = kSfGroup * kSfSetCols;
    static_assert(kAccCol1 + 256 <= kSfCol && kSfCol + 2 * kSfGroupCols <= 512, "tensor memory columns");
};

// Tile order for pairs: as tile_coord, with 256-row tiles.
__host__ __device__ __forceinline__ TileCoord pair_tile_coord(uint32_t idx, uint32_t n_tiles, uint32_t m_tiles, const GemmParams& p)
{
    uint32_t mo = idx / n_tiles;
    TileCoord t;
    t.n_tile = idx - mo * n_tiles;
    t.m_tile = mo;
    if (p.flags != nullptr && p.world > 1) {
        if (p.m_local % kPairBlockM == 0) {
            t.m_tile = arrival_m_tile(mo, p.m_local / kPairBlockM, p);
        } else {
            t.m_tile = (mo + (p.rank * p.m_local) / kPairBlockM) % m_tiles;
        }
    }
    return t;
}

// The launch of `tiles` tiles on at most `pairs` resident pairs: whole rounds, then the rest cut along K in at most `parts` parts
// each (<= 1: it stays whole).
struct PairGrid {
    uint32_t pairs, ksplit;
};

inline PairGrid pair_grid(uint32_t tiles, uint32_t pairs, uint32_t parts)
{
    const uint32_t rem = tiles % pairs;
    if (rem == 0 || parts <= 1) {
        return {tiles < pairs ? tiles : pairs, 1};
    }
    parts = parts < pairs / rem ? parts : pairs / rem;
    return {tiles < pairs ? rem * parts : pairs, parts};
}

// One work unit of a pair: a whole tile, or one K part of a tile of the last round.
struct PairUnit {
    uint32_t m0, n0, n_tile;  // first row and column of the pair's tile
    uint32_t width;           // columns that are multiplied: 256, or what a ragged last tile has, rounded up to 32
    uint32_t kt0, kt1;        // K tiles
    uint32_t part, rem_ix;    // split units: which part, and which of the rem tiles
    bool split;
    bool last;                // no other unit follows on this pair
};

struct PairWork {
    uint32_t m_tiles, n_tiles, num_tiles, k_tiles, pair, num_pairs, rounds, rem, ksplit, units, split_at;

    __host__ __device__ __forceinline__ PairWork(const GemmParams& p, uint32_t pair_, uint32_t num_pairs_)
    {
        m_tiles = (p.Mg + kPairBlockM - 1) / kPairBlockM;
        n_tiles = (p.N + kPairBlockN - 1) / kPairBlockN;
        num_tiles = m_tiles * n_tiles;
        k_tiles = p.K / kGemmBlockK;
        pair = pair_;
        num_pairs = num_pairs_;
        ksplit = p.ksplit > 1u ? p.ksplit : 1u;
        // a grid of exactly num_tiles * ksplit pairs splits every tile
        rounds = ksplit > 1u && num_tiles * ksplit == num_pairs ? 0u : num_tiles / num_pairs;
        rem = num_tiles - rounds * num_pairs;
        units = p.gemm_off ? 0u : rounds + (pair < rem * ksplit ? 1u : 0u);
        // the position of the unit from the incomplete round
        split_at = units > rounds ? (ksplit > 1u && p.flags == nullptr ? 0u : rounds) : units;
    }

    // pairs that have a split unit
    __host__ __device__ __forceinline__ uint32_t split_units() const { return ksplit > 1u && units > 0u ? rem * ksplit : 0u; }

    __host__ __device__ __forceinline__ PairUnit unit(uint32_t i, const GemmParams& p) const
    {
        PairUnit u;
        uint32_t tile = pair + (i - (i > split_at ? 1u : 0u)) * num_pairs;
        u.part = 0;
        u.rem_ix = 0;
        u.kt0 = 0;
        u.kt1 = k_tiles;
        u.split = i == split_at && ksplit > 1u;
        u.last = i + 1u == units;
        if (i == split_at) {
            u.part = pair / rem;
            u.rem_ix = pair - u.part * rem;
            tile = rounds * num_pairs + u.rem_ix;
            u.kt0 = u.part * k_tiles / ksplit;
            u.kt1 = (u.part + 1u) * k_tiles / ksplit;
        }
        const TileCoord tc = pair_tile_coord(tile, n_tiles, m_tiles, p);
        u.m0 = tc.m_tile * kPairBlockM;
        u.n0 = tc.n_tile * kPairBlockN;
        u.n_tile = tc.n_tile;
        const uint32_t left = p.N - u.n0;
        u.width = left < kPairBlockN ? (left + 31u) / 32u * 32u : kPairBlockN;
        return u;
    }
};

template <typename OutT, bool FUSED_QUANT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(FUSED_QUANT ? kGemmFusedThreads : kGemmThreads, 1)
mx_gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                    const __grid_constant__ CUtensorMap tmap_c, const __grid_constant__ GemmParams p)
{
    using S = PairSmem;
    constexpr uint32_t kStages = S::kStages;

    grid_dep_launch();  // as in mx_gemm_kernel
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + S::kOffBar);
    uint64_t* full = bars;
    uint64_t* empty = full + kStages;
    uint64_t* tmem_full = empty + kStages;
    uint64_t* tmem_empty = tmem_full + 2;
    uint64_t* overlap_free = tmem_empty + 2;
    uint64_t* sf_full = overlap_free + 2;
    uint64_t* sf_empty = sf_full + 2;
    uint64_t* atoms = sf_empty + 2;
    uint64_t* red_bar = atoms + 2;
    uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + S::kOffTmemPtr);
    uint32_t* gate = reinterpret_cast<uint32_t*>(smem + S::kOffGate);
    uint32_t* push_turn = gate + 1;  // the pushers of this CTA store one after the other (mx_quant.cuh, push_worker)

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t cta = cluster_ctarank();  // 0 = leader
    const uint64_t bar_ns = p.bar_timeout_ns;
    const PairWork work(p, blockIdx.x >> 1, gridDim.x >> 1);

    if (threadIdx.x == 0) {
        CATCCOS_TR_STAMP(p.trace, kTrCtaStart);
        *gate = 0u;
        *push_turn = 0u;
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 2);  // both CTAs' producers (expect_tx)
            mbar_init(&empty[s], 1);
        }
        for (uint32_t a = 0; a < 2; ++a) {
            mbar_init(&tmem_full[a], 1);
            mbar_init(&tmem_empty[a], 8);    // four epilogue warps in each CTA
            mbar_init(&overlap_free[a], 8);
            mbar_init(&sf_full[a], kSfGroup);  // one commit behind each K tile's copies
            mbar_init(&sf_empty[a], 1);
            mbar_init(&atoms[a], 8);           // four scale-loader warps in each CTA
        }
        for (uint32_t w = 0; w < 4; ++w) {
            mbar_init(&red_bar[w], 1);
        }
        mbar_fence_init();
    }
    if (warp == 5) {
        tmem_alloc_pair(tmem_ptr_smem, kTmemCols);
        tmem_relinquish_pair();
    }
    if (warp == 4 && lane == 0) {
        tma_prefetch_desc(&tmap_a);
        tma_prefetch_desc(&tmap_b);
        tma_prefetch_desc(&tmap_c);
    }
    tcgen05_fence_before();
    __syncthreads();
    cluster_sync_all();  // both CTAs' barriers exist before anybody arrives on the other's
    tcgen05_fence_after();
    const uint32_t tmem_base = *tmem_ptr_smem;
    bool alive = true;  // false once a wait of this role has given up

    if (threadIdx.x == 0) {
        CATCCOS_TR_STAMP(p.trace, kTrSetupDone);
    }

    if (warp == 4) {
        // ------------------------------- TMA producer (both CTAs) -------------------------
        uint32_t it = 0;
        // packed 4-bit operands arrive as half the bytes they occupy in shared memory (the gaps are not written)
        const uint32_t tx_bytes = (p.a_fmt == 5u ? S::kABytes / 2u : S::kABytes) + (p.b_fmt == 5u ? S::kBBytes / 2u : S::kBBytes);
        auto load_b = [&](const PairUnit& u, uint32_t kt, uint32_t s, uint32_t leader_bar) {
            const int32_t n = (int32_t)(u.n0 + cta * (u.width / 2u)), k = (int32_t)(kt * kGemmBlockK);
            if (p.b_kmajor) {  // the transposed copy [N, K]: this CTA's columns are rows of it
                tma_load_2d_pair(smem + S::kOffB + s * S::kBBytes, &tmap_b, leader_bar, k, n);
            } else {
                tma_load_2d_pair(smem + S::kOffB + s * S::kBBytes, &tmap_b, leader_bar, n, k);
            }
        };
        uint32_t early = 0;  // iterations whose B tile is already on its way
        if (p.flags == nullptr) {
            if (p.b_early && work.units > 0u) {
                // the weights do not come from the kernel launched just before: fill the ring's B half meanwhile
                const PairUnit u = work.unit(0, p);
                early = min(kStages, u.kt1 - u.kt0);
                if (lane == 0) {
                    for (uint32_t s = 0; s < early; ++s) {
                        const uint32_t leader_bar = map_to_cta(smem_u32(&full[s]), 0);
                        mbar_arrive_expect_tx_cluster(leader_bar, tx_bytes);
                        load_b(u, u.kt0 + s, s, leader_bar);
                    }
                }
            }
            grid_dep_wait();  // A is the output of the kernel launched just before (no-op for a plain launch);
        }                     // with flags, the flags say when its rows are there
        for (uint32_t ui = 0; alive && ui < work.units; ++ui) {
            const PairUnit u = work.unit(ui, p);
            const uint32_t m0 = u.m0 + cta * 128u;
            uint32_t ready_end = u.kt0;  // K tiles below this index are known to be there
            for (uint32_t kt = u.kt0; alive && kt < u.kt1; ++kt, ++it) {
                if (p.flags != nullptr && kt >= ready_end) {
                    const unsigned long long t0 = CATCCOS_TR_NOW();
                    (void)t0;
                    const uint32_t seg0 = kt / p.seg_ktiles;
                    const uint32_t nready = wait_rows_ready(p, m0, lane, seg0);
                    alive = nready != 0u;
                    ready_end = min((seg0 + nready) * p.seg_ktiles, u.kt1);
                    fence_proxy_async_all();
                    if (lane == 0) {
                        st_release_cta_shared(gate, it + (ready_end - kt));
                        CATCCOS_TR_ADD(p.trace, kTrProdFlagWaitNs, CATCCOS_TR_NOW() - t0);
                    }
                }
                if (!alive) {
                    break;
                }
                // as in the MMA issuer the warp stays together and one elected lane issues
                const uint32_t s = it % kStages;
                const uint32_t leader_bar = map_to_cta(smem_u32(&full[s]), 0);
                if (it >= early) {
                    const unsigned long long t1 = CATCCOS_TR_NOW();
                    (void)t1;
                    alive = mbar_wait_warp(&empty[s], ((it / kStages) & 1u) ^ 1u, p.status, 200, s, bar_ns);
                    if (lane == 0) {
                        CATCCOS_TR_ADD(p.trace, kTrProdEmptyWaitNs, CATCCOS_TR_NOW() - t1);
                    }
                    if (!alive) {
                        break;
                    }
                }
                if (elect_one()) {
                    if (it >= early) {
                        mbar_arrive_expect_tx_cluster(leader_bar, tx_bytes);
                    }
                    if (kt == u.kt0 && ui < kTraceTiles) {
                        CATCCOS_TR_STAMP(p.trace, kTrTileStart + ui);
                    }
                    CATCCOS_TR_STAMP_FIRST(p.trace, kTrProdFirstTma);
                    tma_load_2d_pair(smem + S::kOffA + s * S::kABytes, &tmap_a, leader_bar, (int32_t)(kt * kGemmBlockK),
                                     (int32_t)m0);
                    if (it >= early) {
                        load_b(u, kt, s, leader_bar);
                    }
                    CATCCOS_TR_STAMP(p.trace, kTrProdLastTma);
                }
                __syncwarp();
            }
        }
    } else if (warp == 5) {
        // ------------------------------- MMA issuer (leader CTA only) ---------------------
        // The whole warp runs the loop and one elected lane issues: inside a branch on the lane the operands of a tcgen05
        // instruction cannot stay in uniform registers, and each then takes about 70 cycles to get out.  The issuer
        // issues the MMAs and the commits, nothing else.
        if (cta == 0) {
            const bool bk = p.b_kmajor != 0u;
            const uint32_t idesc0 = make_idesc_mxf8(kPairBlockM, 0, !bk) | ((p.a_fmt & 7u) << 7) |
                                    ((p.b_fmt & 7u) << 10);  // operand formats: E4M3 = 0, E5M2 = 1, E2M1 = 5
            const uint32_t hi_a = (uint32_t)(make_smem_desc(0, 16, 1024, 2) >> 32);
            // B, MN-major: each CTA's 128 columns are one 128-byte swizzle row per K row
            const uint64_t desc_b = bk ? make_smem_desc(0, 16, 1024, 2) : make_smem_desc(0, 16384, 1024, 2);
            const uint32_t hi_b = (uint32_t)(desc_b >> 32);
            const uint32_t a_lo0 = (uint32_t)make_smem_desc(0, 16, 1024, 2) | (smem_u32(smem + S::kOffA) >> 4);
            const uint32_t b_lo0 = (uint32_t)desc_b | (smem_u32(smem + S::kOffB) >> 4);
            const uint32_t kb_step_b = (bk ? 32u : 4096u) >> 4;
            uint32_t s = 0, ph = 0;   // operand stage and its phase
            uint32_t group = 0;       // scale groups consumed
            for (uint32_t ui = 0; alive && ui < work.units; ++ui) {
                const PairUnit u = work.unit(ui, p);
                const uint32_t acc = ui & 1u;
                const uint32_t acc_ph = (ui >> 1) & 1u;
                const uint32_t d_col = tmem_base + (acc ? S::kAccCol1 : 0u);
                const unsigned long long t0 = CATCCOS_TR_NOW();
                (void)t0;
                alive = mbar_wait_warp(&tmem_empty[acc], acc_ph ^ 1u, p.status, 201, acc, bar_ns);
                if (ui > 0 && alive) {
                    alive = mbar_wait_warp(&overlap_free[acc ^ 1u], ((ui - 1) >> 1) & 1u, p.status, 202, acc, bar_ns);
                }
                if (lane == 0) {
                    CATCCOS_TR_ADD(p.trace, kTrMmaAccWaitNs, CATCCOS_TR_NOW() - t0);
                }
                const uint32_t n_it = u.kt1 - u.kt0;
                const uint32_t idesc = idesc0 | ((u.width >> 3) << 17);
                for (uint32_t i = 0; alive && i < n_it; ++i) {
                    const uint32_t buf = group & 1u;
                    const unsigned long long t1 = CATCCOS_TR_NOW();
                    (void)t1;
                    if (i % kSfGroup == 0u) {
                        alive = mbar_wait_warp(&sf_full[buf], (group >> 1) & 1u, p.status, 207, buf, bar_ns);
                    }
                    alive = alive && mbar_wait_warp(&full[s], ph, p.status, 203, s, bar_ns);
                    if (!alive) {
                        break;  // nothing is issued, and the accumulator never reported, after a wait has given up
                    }
                    tcgen05_fence_after();
                    if (lane == 0) {
                        CATCCOS_TR_ADD(p.trace, kTrMmaFullWaitNs, CATCCOS_TR_NOW() - t1);
                        CATCCOS_TR_STAMP_FIRST(p.trace, kTrMmaFirst);
                    }
                    const uint32_t a_lo = a_lo0 + s * (S::kABytes >> 4);
                    const uint32_t b_lo = b_lo0 + s * (S::kBBytes >> 4);
                    const uint32_t sf = tmem_base + S::kSfCol + buf * S::kSfGroupCols + (i % kSfGroup) * S::kSfSetCols;
                    const bool group_end = i % kSfGroup == kSfGroup - 1u || i + 1u == n_it;
                    if (elect_one()) {
#pragma unroll
                        for (uint32_t kb = 0; kb < 4; ++kb) {
                            umma_mxf8_pair_lohi(d_col, a_lo + kb * (32u >> 4), hi_a, b_lo + kb * kb_step_b, hi_b,
                                                idesc_with_sf_id(idesc, kb), sf, sf + 4, (kb != 0u || i != 0u) ? 1u : 0u);
                        }
                        tcgen05_commit_pair(&empty[s], 3);
                        if (group_end) {
                            tcgen05_commit_pair(&sf_empty[buf], 3);
                        }
                        if (i + 1u == n_it) {
                            tcgen05_commit_pair(&tmem_full[acc], 3);
                        }
                    }
                    __syncwarp();
                    group += group_end ? 1u : 0u;
                    s = (s + 1 == kStages) ? 0u : s + 1;
                    ph ^= s == 0u ? 1u : 0u;
                }
                if (lane == 0) {
                    if (ui < kTraceTiles) {
                        CATCCOS_TR_STAMP(p.trace, kTrTileEnd + ui);
                    }
                    CATCCOS_TR_STAMP(p.trace, kTrMmaLast);
                }
            }
        }
    } else if (FUSED_QUANT && warp >= 10) {
        // ------------------------------- quantise-and-push producer -----------------------
        // Of the fourteen extra warps, eight quantise this rank's shard into the local stage (warps 10-19
        // except 13 and 17, which share a scheduler with the MMA issuer and must not compete with that
        // single thread for issue slots).  The other six (13, 17, 20-23) run the pusher, a copy loop that
        // issues an instruction only every few hundred cycles, and send finished items on to the peers.
        if (warp < 20u && (warp & 3u) != (5u & 3u)) {
            const uint32_t qw = warp - 10u - (warp > 13u ? 1u : 0u) - (warp > 17u ? 1u : 0u);  // 0..7
            quant_push_producer<true>(p.q, qw * 32u + lane, blockIdx.x, gridDim.x, 1);
        } else {
            const uint32_t pw = warp == 13u ? 0u : (warp == 17u ? 1u : warp - 18u);  // 0..5
            push_worker(p.push, lane, pw * gridDim.x + blockIdx.x, gridDim.x * kPushWarps, pw, gridDim.x, push_turn);
        }
    } else if (warp >= 6) {
        // ------------------------------- scale loaders (both CTAs) ------------------------
        // Warp j loads the A scales of this CTA's rows [32 j, +32) for all four K tiles of a group (16 bytes per row) and
        // the B scales of all columns of the pair's tile for K tile j.
        constexpr uint32_t kNB = kPairBlockN / 32;
        const uint32_t j = warp - 6;
        const uint32_t sf_row_bytes = p.K / 32;
        const bool a_wide = p.K % 512u == 0u && ((uintptr_t)p.a_scales & 15u) == 0u;
        uint32_t cur_lo[kNB], cur_hi[kNB], nxt_lo[kNB], nxt_hi[kNB];
        uint4 cur_a, nxt_a;
        uint32_t known_end = 0;  // K-tile iterations below this index have their rows in place

        // where this warp is: unit ui, first K tile of the group, running index of that K tile
        struct Cursor {
            uint32_t ui, kt, it;
            PairUnit u;
        };
        auto next = [&](Cursor& c) {
            c.kt += kSfGroup;
            c.it += kSfGroup;
            if (c.kt >= c.u.kt1) {
                c.it -= c.kt - c.u.kt1;
                if (++c.ui < work.units) {
                    c.u = work.unit(c.ui, p);
                    c.kt = c.u.kt0;
                }
            }
        };
        auto load_b = [&](const Cursor& c, uint32_t (&rlo)[kNB], uint32_t (&rhi)[kNB]) {
            const uint32_t kt = c.kt + j;
#pragma unroll
            for (uint32_t i = 0; i < kNB; ++i) {
                const uint32_t n = c.u.n0 + i * 32 + lane;
                rlo[i] = 0x7F7Fu;
                rhi[i] = 0x7F7Fu;
                if (n < p.N && kt < c.u.kt1) {
                    rlo[i] = __ldcg(reinterpret_cast<const uint16_t*>(p.b_scales + ((size_t)(2 * kt) * p.N + n) * 2));
                    rhi[i] = __ldcg(reinterpret_cast<const uint16_t*>(p.b_scales + ((size_t)(2 * kt + 1) * p.N + n) * 2));
                }
            }
        };
        auto load_a = [&](const Cursor& c, uint4& ra) {
            const uint32_t m0 = c.u.m0 + cta * 128u;
            const uint32_t last = min(c.kt + kSfGroup, c.u.kt1);  // K tiles [c.kt, last) of the group exist
            while (p.flags != nullptr && alive && c.it + (last - c.kt) > known_end) {
                // this CTA's producer has usually seen these rows' flags already and said so in shared memory
                // one lane reads the word for the warp: the producer may be updating it, and the branch below holds
                // warp-wide operations, so every lane has to take the same side
                const uint32_t g = __shfl_sync(0xFFFFFFFFu, ld_acquire_cta_shared(gate), 0);
                __syncwarp();  // lane 0 acquired it
                if (g >= c.it + (last - c.kt)) {
                    known_end = g;
                } else {
                    const unsigned long long t0 = CATCCOS_TR_NOW();
                    (void)t0;
                    // the first K tile of the group that is not known to be there
                    const uint32_t kt = max(known_end, c.it) - c.it + c.kt;
                    const uint32_t seg0 = kt / p.seg_ktiles;
                    const uint32_t nready = wait_rows_ready(p, m0, lane, seg0);
                    alive = nready != 0u;
                    known_end = c.it + (min((seg0 + nready) * p.seg_ktiles, c.u.kt1) - c.kt);
                    if (lane == 0) {
                        CATCCOS_TR_ADD(p.trace, kTrSfGateWaitNs + j, CATCCOS_TR_NOW() - t0);
                    }
                }
            }
            const uint32_t row = m0 + j * 32 + lane;
            ra = make_uint4(0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
            if (row < p.Mg) {
                const uint32_t* src = reinterpret_cast<const uint32_t*>(p.a_scales + (size_t)row * sf_row_bytes) + c.kt;
                if (a_wide && c.kt % kSfGroup == 0u) {
                    ra = __ldcg(reinterpret_cast<const uint4*>(src));  // K % 512 == 0: the four K tiles are in the row
                } else {
                    ra.x = __ldcg(src);
                    ra.y = c.kt + 1u < last ? __ldcg(src + 1) : ra.y;
                    ra.z = c.kt + 2u < last ? __ldcg(src + 2) : ra.z;
                    ra.w = c.kt + 3u < last ? __ldcg(src + 3) : ra.w;
                }
            }
        };

        Cursor c;
        c.ui = 0;
        c.it = 0;
        c.kt = 0;
        if (work.units > 0u) {
            c.u = work.unit(0, p);
            c.kt = c.u.kt0;
            if (p.flags == nullptr && !p.b_early) {
                grid_dep_wait();
            }
            load_b(c, cur_lo, cur_hi);
            if (p.flags == nullptr && p.b_early) {
                grid_dep_wait();  // only the A scales are the output of the kernel launched just before
            }
            load_a(c, cur_a);
        }
        uint32_t group = 0;
        while (alive && c.ui < work.units) {
            const bool real = c.kt + j < c.u.kt1;  // the last group of a unit may be short
            next(c);
            if (c.ui < work.units) {
                load_b(c, nxt_lo, nxt_hi);
                load_a(c, nxt_a);
            }
            const uint32_t buf = group & 1u, ph = (group >> 1) & 1u;
            const unsigned long long t1 = CATCCOS_TR_NOW();
            (void)t1;
            alive = mbar_wait_warp(&sf_empty[buf], ph ^ 1u, p.status, 205, buf, bar_ns) && alive;
            if (lane == 0) {
                CATCCOS_TR_ADD(p.trace, kTrSfEmptyWaitNs + j, CATCCOS_TR_NOW() - t1);
            }
            uint8_t* sfa = smem + S::kOffSf + buf * S::kSfBufBytes;
            uint8_t* sfb = sfa + kSfGroup * S::kSfaBytes + j * S::kSfbBytes;
            {
                // an atom row holds the words of tile rows lane, lane + 32, lane + 64, lane + 96: this warp's is word j
                uint32_t* dst = reinterpret_cast<uint32_t*>(sfa + lane * 16u) + j;
                dst[0] = cur_a.x;
                dst[S::kSfaBytes / 4] = cur_a.y;
                dst[2 * S::kSfaBytes / 4] = cur_a.z;
                dst[3 * S::kSfaBytes / 4] = cur_a.w;
            }
#pragma unroll
            for (uint32_t h = 0; h < kNB / 4; ++h) {
                uint4 v;
                v.x = cur_lo[h * 4 + 0] | (cur_hi[h * 4 + 0] << 16);
                v.y = cur_lo[h * 4 + 1] | (cur_hi[h * 4 + 1] << 16);
                v.z = cur_lo[h * 4 + 2] | (cur_hi[h * 4 + 2] << 16);
                v.w = cur_lo[h * 4 + 3] | (cur_hi[h * 4 + 3] << 16);
                *reinterpret_cast<uint4*>(sfb + h * 512u + lane * 16u) = v;
            }
            fence_proxy_async_shared();
            __syncwarp();
            // All loader warps of both CTAs report their atoms to the leader; the leader's warp j then copies K tile
            // j's atoms of both CTAs into both CTAs' tensor memory (one cta_group::2 copy does the same offsets in
            // the two).
            if (lane == 0) {
                mbar_arrive_cluster(map_to_cta(smem_u32(&atoms[buf]), 0));
            }
            if (cta == 0) {
                alive = mbar_wait_warp(&atoms[buf], ph, p.status, 208, buf, bar_ns) && alive;
                tcgen05_fence_after();
                if (elect_one()) {
                    if (real) {
                        const uint32_t hi_sf = (uint32_t)(make_smem_desc(0, 0, 128, 0) >> 32);
                        const uint32_t sf_t = tmem_base + S::kSfCol + buf * S::kSfGroupCols + j * S::kSfSetCols;
                        tcgen05_cp_sf_pair_lohi(sf_t, smem_u32(sfa + j * S::kSfaBytes) >> 4, hi_sf);
#pragma unroll
                        for (uint32_t h = 0; h < kPairBlockN / 128; ++h) {
                            tcgen05_cp_sf_pair_lohi(sf_t + 4 + 4 * h, (smem_u32(sfb) >> 4) + h * (512u >> 4), hi_sf);
                        }
                    }
                    tcgen05_commit_pair(&sf_full[buf], 1);
                }
                __syncwarp();
            }
            ++group;
            cur_a = nxt_a;
#pragma unroll
            for (uint32_t i = 0; i < kNB; ++i) {
                cur_lo[i] = nxt_lo[i];
                cur_hi[i] = nxt_hi[i];
            }
        }
    } else {
        // ------------------------------- epilogue (both CTAs, own 128 rows) ---------------
        const uint32_t q = warp;
        OutT* c = reinterpret_cast<OutT*>(p.c);
        constexpr uint32_t kChunks = kPairBlockN / 32;
        const uint32_t lane_base = tmem_base + ((q * 32u) << 16);
        uint8_t* stage_out = smem + S::kOffOut + q * kOutStageBytes;
        uint32_t split_ep = 0;
        if (work.split_units() > work.pair) {
            if (p.flags == nullptr) {
                grid_dep_wait();  // a gated launch's quantiser has waited for the launch before it
            }
            split_ep = split_epoch(p.splitk_state, work.split_units() * 8u, lane);
        }
        for (uint32_t ui = 0; alive && ui < work.units; ++ui) {
            const PairUnit u = work.unit(ui, p);
            const uint32_t row0 = u.m0 + cta * 128u + q * 32u;  // this warp's first row
            const uint32_t row = row0 + lane;
            const uint32_t acc = ui & 1u;
            const uint32_t d_col = acc ? S::kAccCol1 : 0u;
            const unsigned long long t0 = CATCCOS_TR_NOW();
            (void)t0;
            alive = mbar_wait_warp(&tmem_full[acc], (ui >> 1) & 1u, p.status, 206, acc, bar_ns);
            if (q == 0 && lane == 0) {
                CATCCOS_TR_ADD(p.trace, kTrEpiWaitNs, CATCCOS_TR_NOW() - t0);
            }
            if (!alive) {
                break;  // an accumulator that never filled is not written out
            }
            tcgen05_fence_after();
            if (u.split) {
                SplitExchange<OutT, kChunks> x;
                x.epoch = split_ep;
                const uint32_t slot = u.rem_ix * work.ksplit * 2u + cta;
                x.ws = p.splitk_ws + (size_t)slot * (128u * kPairBlockN);
                x.part_stride = (size_t)2u * 128u * kPairBlockN;
                x.flags = p.splitk_flags + slot * 4u + q;
                x.flag_stride = 8u;
                if (u.last) {
                    // the operand stages are idle by now and receive the other parts' pieces
                    x.red = smem + S::kOffA + q * kSplitRedBytes;
                    x.bar = &red_bar[q];
                    alive = x.run(p, c, lane_base + d_col, u.part, work.ksplit, q, lane, row0, u.n0, u.rem_ix, bar_ns);
                } else {
                    x.put(p, lane_base + d_col, u.part, q, lane, row0, u.n0);
                    tcgen05_fence_before();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive_cluster(map_to_cta(smem_u32(&overlap_free[acc]), 0));
                        mbar_arrive_cluster(map_to_cta(smem_u32(&tmem_empty[acc]), 0));
                    }
                    alive = x.take(p, c, u.part, work.ksplit, q, lane, row0, u.n0, u.rem_ix);
                }
                continue;
            }
            // The half that holds the columns shared with the other accumulator goes first, columns 128..255 of
            // accumulator 0, 0..127 of accumulator 1.  A half is pulled into registers as a whole and its columns are given
            // back before anything is converted or stored: the next tile's products wait for them.
            constexpr uint32_t kPull = FUSED_QUANT ? 2 : 4;  // 32-column chunks (the fused kernel's threads have 80 registers)
            for (uint32_t hi = 0; hi < 2; ++hi) {
                const uint32_t col0 = (acc == 0u ? 1u - hi : hi) * 128u;
                const bool inside = row0 < p.Mg && u.n0 + col0 < p.N;
                uint32_t scale_word = 0;
#pragma unroll
                for (uint32_t g0 = 0; g0 < 4; g0 += kPull) {
                    uint32_t r[kPull][32];
#pragma unroll
                    for (uint32_t i = 0; i < kPull; ++i) {
                        tmem_ld_32x32(lane_base + d_col + col0 + (g0 + i) * 32u, r[i]);
                    }
                    tmem_ld_wait();
                    if (g0 + kPull == 4u) {
                        tcgen05_fence_before();
                        __syncwarp();
                        if (lane == 0) {
                            uint64_t* b = hi == 0u ? &overlap_free[acc] : &tmem_empty[acc];
                            mbar_arrive_cluster(map_to_cta(smem_u32(b), 0));
                        }
                    }
#pragma unroll
                    for (uint32_t i = 0; i < kPull; i += 2) {
                        const uint32_t g = g0 + i;  // chunks g and g + 1: 64 columns
                        const uint32_t col = u.n0 + col0 + g * 32u;
                        if constexpr (std::is_same<OutT, ScatterOut>::value) {
                            store_c_chunk<OutT>(c, p, row, col, r[i]);
                            store_c_chunk<OutT>(c, p, row, col + 32u, r[i + 1]);
                        } else if constexpr (std::is_same<OutT, MxOut>::value) {
                            if (g == 0u) {
                                out_stage_free(lane);
                            }
                            uint32_t o[8], byte0, byte1;
                            mx_quantise_chunk(p, r[i], o, byte0);
                            out_stage_put(stage_out, lane, g * 2u, o);
                            mx_quantise_chunk(p, r[i + 1], o, byte1);
                            out_stage_put(stage_out, lane, g * 2u + 2u, o);
                            scale_word |= (byte0 | (byte1 << 8)) << (8u * g);
                            if (g == 2u) {
                                out_stage_send(stage_out, &tmap_c, lane, inside, u.n0 + col0, row0);
                                store_scale_word(p, row, u.n0 + col0, scale_word);
                            }
                        } else {
                            // A send waits until the one before it has been read.  The next tile's products hide that; the last
                            // tile has none, but its accumulator is complete only when nothing uses the operand stages any
                            // more, so each of its four sends takes a buffer there and none waits (1024x2304x256 6.5 -> 6.0 us,
                            // 2000x4096x1024 12.8 -> 12.5).  A quantised tile has two sends and gains nothing.
                            uint8_t* out = stage_out;
                            if (u.last) {
                                out = smem + S::kOffA + (q * 4u + hi * 2u + g / 2u) * kOutStageBytes;
                            } else {
                                out_stage_free(lane);
                            }
                            out_stage_put_chunk<OutT>(out, lane, 0u, r[i]);
                            out_stage_put_chunk<OutT>(out, lane, 4u, r[i + 1]);
                            out_stage_send(out, &tmap_c, lane, inside && col < p.N, col, row0);
                        }
                    }
                }
            }
            publish_tile_rows<OutT>(p, row0, u.n_tile, work.n_tiles, lane);
            if (lane == 0 && q == 0) {
                CATCCOS_TR_STAMP(p.trace, kTrEpiLast);
            }
        }
        if (lane == 0) {
            bulk_store_wait_all();  // the output is written before the CTA ends
        }
    }

    tcgen05_fence_before();
    if (__syncthreads_or(alive ? 0 : 1)) {
        drain_after_abort(p.status);  // both CTAs stay while loads that report to the other's barriers may be in flight
    }
    cluster_sync_all();  // nobody leaves while the other CTA may still arrive on its barriers
    if (p.flags != nullptr) {
        grid_dep_wait();
    }
    if (threadIdx.x == 0) {
        CATCCOS_TR_STAMP(p.trace, kTrCtaEnd);
    }
    if (warp == 5) {
        tcgen05_fence_after();
        tmem_dealloc_pair(tmem_base, kTmemCols);
    }
}

}  // namespace catccos
