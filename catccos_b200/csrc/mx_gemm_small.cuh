// MXFP8 block-scaled GEMM for few output tiles (decode and small batches): C[M, N] = X[M, K] x W[K, N].
//
// Same operands and layouts as mx_gemm.cuh, one GPU, no flags.  Such a call is bound by latencies and by streaming the
// weights once, not by the tensor pipe, so this kernel is built the other way round:
//   * The operands are swapped: 128 weight columns are the M side of tcgen05.mma, MT activation rows (16 or 32)
//     its N side.  A call with 16 rows pays for 16, not for a padded tile of 128, and an accumulator has MT columns.
//   * K is cut over the CTAs of a cluster (1, 2, 4 or 8 of them), so that a few output tiles still stream the weights
//     with every SM.  The partial sums meet in distributed shared memory: part p owns MT / parts of the rows (four at least), the others
//     push theirs into its shared memory, it adds them in ascending part order (the result does not depend on timing).
//     Through global memory (partials, fence, flag, poll, load) the same exchange takes 3 to 5 us.
//   * About 110 KB of shared memory and 64 tensor-memory columns a CTA: two CTAs per SM, one fills and drains
//     while the other streams.  CTAs of different clusters never wait for one another, so any grid is fine.
//   * With QUANT the four epilogue warps, idle until the accumulator is ready, quantise the bf16 rows straight into the
//     operand ring (every CTA for itself): a fused call is one launch and has no quantised copy of X anywhere.
//
// Tiles of 64 and 128 rows were measured too: no faster than mx_gemm.cuh's tiles at the sizes that fill them.
// Measured (B200, 200 calls queued in the stream, against a quantise kernel and mx_gemm.cuh's tiles without programmatic
// launches): fused 16 x 4096 x 7168 18.5 to 20.3 -> 8.6 us, 1 x 2432 x 2432 12.3 -> 4.5, 8 x 1024 x 7168 14.5 -> 6.2, 12 x
// 3008 x 4992 18.5 -> 6.2, 64 x 1024 x 1024 13.8 -> 5.4; the matmul alone 16 x 4096 x 7168 14.4 -> 8.6.
//
// 320 threads: warps 0-3 X scales (or, QUANT, X codes and scales), then the epilogue; warp 4 TMA; warp 5 MMA issuer, which
// also copies the stage's scale factors into tensor memory; warps 6-9 W scales, warp j every fourth K tile.
#pragma once

#include "mx_gemm.cuh"

namespace catccos {

constexpr uint32_t kSmallBlockN = 128;  // weight columns of a tile
constexpr uint32_t kSmallMaxParts = 8;

struct SmallParams {
    const void* x;            // QUANT: bf16 [M, K]
    const uint8_t* x_scales;  // otherwise: E8M0 [M, K/32] (the codes come through the tensor map)
    const uint8_t* w_scales;  // [K/64, N, 2]
    void* c;                  // [M, N]
    uint8_t* c_scales;        // MxOut: E8M0 [M, N/32]
    uint32_t M, N, K;
    uint32_t parts;           // cluster size: K parts of a tile
    uint32_t x_fmt, w_fmt;    // as GemmParams::a_fmt, b_fmt
    uint32_t w_kmajor;        // 1: W is the transposed copy [N, K]
    uint32_t w_early;         // 1: W and its scales were in place before the kernel launched just before this one
    uint32_t device_tiny;     // QUANT, MxOut: tiny blocks follow the reference device kernel
    uint64_t bar_timeout_ns;
    StatusBlock* status;
    StatusBlock* records;     // kWaitRecords wait records of which all but `status` are to be cleared (or nullptr)
};

template <uint32_t MT>
struct SmallSmem {
    static constexpr uint32_t kStages = MT == 16 ? 5 : 4;
    // A scale-loader warp serves every kSfStride-th K tile.  Its wait for the stage looks at a parity, so the phase before
    // the one it waits for must be known to be over: its own wait before this one says so as long as the stride is not
    // larger than the ring.
    static constexpr uint32_t kSfStride = 4;
    static_assert(kSfStride <= kStages, "a scale loader would take a stale phase for the one it waits for");
    static constexpr uint32_t kWBytes = kSmallBlockN * kGemmBlockK;
    static constexpr uint32_t kXBytes = MT * kGemmBlockK;
    static constexpr uint32_t kOffW = 0;
    static constexpr uint32_t kOffX = kOffW + kStages * kWBytes;
    static constexpr uint32_t kOffSf = kOffX + kStages * kXBytes;  // per stage: 512 bytes of W scales, 512 of X scales
    static constexpr uint32_t kOffRed = kOffSf + kStages * 1024;
    // the other parts' pieces: [part][128 columns][rows a part owns] floats; a part owns at least four rows
    static constexpr uint32_t kRedBytes = (kSmallMaxParts - 1) * 4 * 512;
    static_assert(MT <= 4 * kSmallMaxParts, "with fewer parts the pieces get larger, but not more of them");
    static constexpr uint32_t kOffBar = kOffRed + kRedBytes;
    static constexpr uint32_t kNumBars = 2 * kStages + 1;  // full[S], empty[S], acc_full
    static constexpr uint32_t kOffTmemPtr = kOffBar + kNumBars * 8;
    static constexpr uint32_t kOffDead = kOffTmemPtr + 4;  // a part of this cluster has given up
    static constexpr uint32_t kBytes = kOffTmemPtr + 16;
    static constexpr uint32_t kDynamicBytes = kBytes + 1024;
    static_assert(kDynamicBytes <= 113 * 1024, "two CTAs per SM");
    static constexpr uint32_t kSfCol = MT;  // tensor memory: the accumulator, then 8 scale columns a stage
    static constexpr uint32_t kTmemCols = 64;
    static_assert(kSfCol + kStages * 8 <= kTmemCols, "tensor memory columns");
};

// 32 lanes x 16 consecutive 32-bit columns -> 16 registers per thread
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

__device__ __forceinline__ void st_shared_cluster_u32(uint32_t cluster_addr, uint32_t v)
{
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(cluster_addr), "r"(v) : "memory");
}

__device__ __forceinline__ void st_shared_cluster_v4(uint32_t cluster_addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d)
{
    asm volatile("st.shared::cluster.v4.u32 [%0], {%1, %2, %3, %4};" ::"r"(cluster_addr), "r"(a), "r"(b), "r"(c), "r"(d)
                 : "memory");
}

__device__ __forceinline__ void cluster_arrive()
{
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}

__device__ __forceinline__ void cluster_wait()
{
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// One output row's 32 columns of this warp: lane holds column n (the caller keeps lanes right of the matrix out for the
// 16-bit types; MX blocks are inside or outside as a whole).
template <typename OutT>
__device__ __forceinline__ void store_small(const SmallParams& p, uint32_t row, uint32_t n, uint32_t lane, float v)
{
    if constexpr (std::is_same<OutT, MxOut>::value) {
        const uint32_t bits = pack2<__nv_bfloat16>(v, 0.f) & 0xFFFFu;
        const uint32_t amax = __reduce_max_sync(0xFFFFFFFFu, bits & 0x7FFFu);
        uint32_t byte;
        float mul;
        bool nonfinite;
        block_scale(amax, p.device_tiny != 0u, 8u, byte, mul, nonfinite);
        const uint32_t code = nonfinite ? 0x7Fu : (cvt_e4m3x2(__uint_as_float(bits << 16) * mul, 0.f) & 0xFFu);
        if (n < p.N) {
            static_cast<uint8_t*>(p.c)[(size_t)row * p.N + n] = (uint8_t)code;
            if (lane == 0) {
                p.c_scales[(size_t)row * (p.N / 32u) + n / 32u] = (uint8_t)byte;
            }
        }
    } else {
        if (n < p.N) {
            static_cast<OutT*>(p.c)[(size_t)row * p.N + n] = static_cast<OutT>(v);
        }
    }
}

template <uint32_t MT, typename OutT, bool QUANT>
__global__ void __launch_bounds__(kGemmThreads, 2)
mx_gemm_small_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x,
                     const __grid_constant__ SmallParams p)
{
    using S = SmallSmem<MT>;
    constexpr uint32_t kStages = S::kStages;

    grid_dep_launch();
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + S::kOffBar);
    uint64_t* empty = full + kStages;
    uint64_t* acc_full = empty + kStages;
    uint32_t* tmem_ptr_smem = reinterpret_cast<uint32_t*>(smem + S::kOffTmemPtr);
    uint32_t* dead = reinterpret_cast<uint32_t*>(smem + S::kOffDead);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint64_t bar_ns = p.bar_timeout_ns;
    const uint32_t parts = p.parts;
    const uint32_t part = blockIdx.x & (parts - 1u);  // == the CTA's rank in its cluster
    const uint32_t tile = blockIdx.x / parts;
    const uint32_t n_tiles = (p.N + kSmallBlockN - 1) / kSmallBlockN;
    const uint32_t m0 = tile / n_tiles * MT, n0 = (tile % n_tiles) * kSmallBlockN;
    const uint32_t k_tiles = p.K / kGemmBlockK;
    const uint32_t kt0 = part * k_tiles / parts, n_it = (part + 1u) * k_tiles / parts - kt0;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 2 + (QUANT ? 4 : 1));  // TMA bytes, the W scales, the X scales (QUANT: and codes)
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        *dead = 0u;
        mbar_fence_init();
    }
    for (uint32_t i = threadIdx.x; i < kStages * 1024 / 16; i += kGemmThreads) {
        // scale atoms of rows and columns outside the matrix, and of rows beyond MT, stay at 1.0
        reinterpret_cast<uint4*>(smem + S::kOffSf)[i] = make_uint4(0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
    }
    if (warp == 5) {
        tmem_alloc(tmem_ptr_smem, S::kTmemCols);
        tmem_relinquish();
    }
    if (warp == 4 && lane == 0) {
        tma_prefetch_desc(&tmap_w);
        if (!QUANT) {
            tma_prefetch_desc(&tmap_x);
        }
    }
    fence_proxy_async_shared();
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    if (parts > 1u) {
        cluster_arrive();  // "this CTA runs": waited for before anything is pushed into it
    }
    const uint32_t tmem_base = *tmem_ptr_smem;
    bool alive = true;  // false once a wait of this role has given up

    if (warp == 4) {
        // ------------------------------- TMA producer -------------------------------------
        const uint32_t tx_bytes = (p.w_fmt == 5u ? S::kWBytes / 2u : S::kWBytes) +
                                  (QUANT ? 0u : (p.x_fmt == 5u ? S::kXBytes / 2u : S::kXBytes));
        auto load_w = [&](uint32_t it) {
            const uint32_t s = it % kStages;
            const int32_t k = (int32_t)((kt0 + it) * kGemmBlockK);
            mbar_arrive_expect_tx(&full[s], tx_bytes);
            tma_load_2d(smem + S::kOffW + s * S::kWBytes, &tmap_w, &full[s], p.w_kmajor ? k : (int32_t)n0,
                        p.w_kmajor ? (int32_t)n0 : k);
        };
        uint32_t early = 0;
        if (p.w_early) {
            early = min(kStages, n_it);
            if (lane == 0) {
                for (uint32_t it = 0; it < early; ++it) {
                    load_w(it);
                }
            }
        }
        grid_dep_wait();
        if (p.records != nullptr && blockIdx.x == 0 && lane < kWaitRecords && p.records + lane != p.status) {
            p.records[lane] = StatusBlock{};  // what the call before left: it has finished
        }
        __syncwarp();
        // the warp stays together and one elected lane issues (mx_gemm.cuh)
        for (uint32_t it = 0; it < n_it; ++it) {
            const uint32_t s = it % kStages;
            if (it >= early) {
                alive = mbar_wait_warp(&empty[s], ((it / kStages) & 1u) ^ 1u, p.status, 300, s, bar_ns);
                if (!alive) {
                    break;
                }
            }
            if (elect_one()) {
                if (it >= early) {
                    load_w(it);
                }
                if (!QUANT) {
                    tma_load_2d(smem + S::kOffX + s * S::kXBytes, &tmap_x, &full[s], (int32_t)((kt0 + it) * kGemmBlockK),
                                (int32_t)m0);
                }
            }
            __syncwarp();
        }
    } else if (warp == 5) {
        // ------------------------------- MMA issuer ---------------------------------------
        const bool wk = p.w_kmajor != 0u;
        // the M side (A in the descriptor's terms) is W, MN-major unless it is the transposed copy; the N side is X, K-major
        const uint32_t idesc = make_idesc_mxf8(128, MT, false) | (wk ? 0u : 1u << 15) | ((p.w_fmt & 7u) << 7) |
                               ((p.x_fmt & 7u) << 10);
        const uint64_t desc_w = wk ? make_smem_desc(0, 16, 1024, 2) : make_smem_desc(0, 16384, 1024, 2);
        const uint32_t hi_w = (uint32_t)(desc_w >> 32), hi_x = (uint32_t)(make_smem_desc(0, 16, 1024, 2) >> 32);
        const uint32_t hi_sf = (uint32_t)(make_smem_desc(0, 0, 128, 0) >> 32);
        const uint32_t w_lo0 = (uint32_t)desc_w | (smem_u32(smem + S::kOffW) >> 4);
        const uint32_t x_lo0 = (uint32_t)make_smem_desc(0, 16, 1024, 2) | (smem_u32(smem + S::kOffX) >> 4);
        const uint32_t sf_lo0 = smem_u32(smem + S::kOffSf) >> 4;
        const uint32_t w_step = (wk ? 32u : 4096u) >> 4;
        uint32_t s = 0, ph = 0;
        for (uint32_t it = 0; it < n_it; ++it) {
            alive = mbar_wait_warp(&full[s], ph, p.status, 303, s, bar_ns);
            if (!alive) {
                break;
            }
            tcgen05_fence_after();
            const uint32_t w_lo = w_lo0 + s * (S::kWBytes >> 4), x_lo = x_lo0 + s * (S::kXBytes >> 4);
            const uint32_t sf = tmem_base + S::kSfCol + s * 8u;
            if (elect_one()) {
                // copies and products of one thread run in the order they are issued
                tcgen05_cp_sf_lohi(sf, sf_lo0 + s * (1024u >> 4), hi_sf);
                tcgen05_cp_sf_lohi(sf + 4, sf_lo0 + s * (1024u >> 4) + (512u >> 4), hi_sf);
#pragma unroll
                for (uint32_t kb = 0; kb < 4; ++kb) {
                    umma_mxf8_lohi(tmem_base, w_lo + kb * w_step, hi_w, x_lo + kb * (32u >> 4), hi_x, idesc_with_sf_id(idesc, kb),
                                   sf, sf + 4, (kb != 0u || it != 0u) ? 1u : 0u);
                }
                tcgen05_commit(&empty[s]);
                if (it + 1u == n_it) {
                    tcgen05_commit(acc_full);
                }
            }
            __syncwarp();
            s = (s + 1 == kStages) ? 0u : s + 1;
            ph ^= s == 0u ? 1u : 0u;
        }
    } else if (warp >= 6) {
        // ------------------------------- W scales -----------------------------------------
        const uint32_t j = warp - 6;
        uint32_t lo[4], hi[4], nlo[4], nhi[4];
        auto load = [&](uint32_t it, uint32_t (&l)[4], uint32_t (&h)[4]) {
            const uint32_t kt = kt0 + it;
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t n = n0 + i * 32 + lane;
                l[i] = h[i] = 0x7F7Fu;
                if (n < p.N) {
                    l[i] = __ldcg(reinterpret_cast<const uint16_t*>(p.w_scales + ((size_t)(2 * kt) * p.N + n) * 2));
                    h[i] = __ldcg(reinterpret_cast<const uint16_t*>(p.w_scales + ((size_t)(2 * kt + 1) * p.N + n) * 2));
                }
            }
        };
        if (!p.w_early) {
            grid_dep_wait();
        }
        if (j < n_it) {
            load(j, lo, hi);
        }
        for (uint32_t it = j; alive && it < n_it; it += S::kSfStride) {
            if (it + S::kSfStride < n_it) {
                load(it + S::kSfStride, nlo, nhi);
            }
            const uint32_t s = it % kStages;
            alive = mbar_wait_warp(&empty[s], ((it / kStages) & 1u) ^ 1u, p.status, 305, s, bar_ns);
            *reinterpret_cast<uint4*>(smem + S::kOffSf + s * 1024u + lane * 16u) =
                make_uint4(lo[0] | (hi[0] << 16), lo[1] | (hi[1] << 16), lo[2] | (hi[2] << 16), lo[3] | (hi[3] << 16));
            fence_proxy_async_shared();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full[s]);
            }
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                lo[i] = nlo[i];
                hi[i] = nhi[i];
            }
        }
    } else if (QUANT) {
        // ------------------------------- X: quantise into the ring ------------------------
        // Every warp takes MT / 4 rows of every K tile, four rows (8 lanes of 16 values each) a step; four steps are
        // loaded together, the next four travel while these are encoded.
        constexpr uint32_t kSteps = MT / 16;  // of a K tile
        const uint32_t c8 = lane & 7u;
        const uint32_t total = n_it * kSteps;
        const bool e5m2 = p.x_fmt == 1u, tiny = p.device_tiny != 0u;
        uint4 v[4][2], nv[4][2];
        auto load = [&](uint32_t st, uint4& a, uint4& b) {
            const uint32_t row = m0 + warp * (MT / 4) + (st % kSteps) * 4u + (lane >> 3);
            a = b = make_uint4(0, 0, 0, 0);
            if (st < total && row < p.M) {
                load_half_block(static_cast<const uint16_t*>(p.x) + (size_t)row * p.K + (kt0 + st / kSteps) * kGemmBlockK + c8 * 16u, a, b);
            }
        };
        grid_dep_wait();
#pragma unroll
        for (uint32_t i = 0; i < 4; ++i) {
            load(i, v[i][0], v[i][1]);
        }
        for (uint32_t st0 = 0; alive && st0 < total; st0 += 4) {
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                load(st0 + 4 + i, nv[i][0], nv[i][1]);
            }
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                const uint32_t st = st0 + i;
                if (st >= total || !alive) {
                    break;
                }
                const uint32_t it = st / kSteps, s = it % kStages;
                if (st % kSteps == 0u) {
                    alive = mbar_wait_warp(&empty[s], ((it / kStages) & 1u) ^ 1u, p.status, 306, s, bar_ns);
                }
                uint32_t byte;
                const uint4 o = quant16(v[i][0], v[i][1], tiny, e5m2, byte);
                const uint32_t r = warp * (MT / 4) + (st % kSteps) * 4u + (lane >> 3);
                *reinterpret_cast<uint4*>(smem + S::kOffX + s * S::kXBytes + r * 128u + ((c8 ^ (r & 7u)) << 4)) = o;
                uint32_t w = (lane & 1u) ? 0u : byte << (4u * c8);  // lanes 0, 2, 4, 6 of a row: bytes 0 .. 3
                w |= __shfl_xor_sync(0xFFFFFFFFu, w, 2);
                w |= __shfl_xor_sync(0xFFFFFFFFu, w, 4);
                if (c8 == 0u) {
                    *reinterpret_cast<uint32_t*>(smem + S::kOffSf + s * 1024u + 512u + r * 16u) = w;
                }
                if (st % kSteps == kSteps - 1u) {
                    fence_proxy_async_shared();
                    __syncwarp();
                    if (lane == 0) {
                        mbar_arrive(&full[s]);
                    }
                }
            }
#pragma unroll
            for (uint32_t i = 0; i < 4; ++i) {
                v[i][0] = nv[i][0];
                v[i][1] = nv[i][1];
            }
        }
    } else {
        // ------------------------------- X scales -----------------------------------------
        uint32_t w = 0, nw = 0;
        const uint32_t row_bytes = p.K / 32;
        auto load = [&](uint32_t it) {
            const uint32_t row = m0 + lane;
            return lane < MT && row < p.M
                       ? __ldcg(reinterpret_cast<const uint32_t*>(p.x_scales + (size_t)row * row_bytes + (kt0 + it) * 4u))
                       : 0x7F7F7F7Fu;
        };
        grid_dep_wait();
        if (warp < n_it) {
            w = load(warp);
        }
        for (uint32_t it = warp; alive && it < n_it; it += S::kSfStride) {
            if (it + S::kSfStride < n_it) {
                nw = load(it + S::kSfStride);
            }
            const uint32_t s = it % kStages;
            alive = mbar_wait_warp(&empty[s], ((it / kStages) & 1u) ^ 1u, p.status, 306, s, bar_ns);
            *reinterpret_cast<uint32_t*>(smem + S::kOffSf + s * 1024u + 512u + lane * 16u) = w;
            fence_proxy_async_shared();
            __syncwarp();
            if (lane == 0) {
                mbar_arrive(&full[s]);
            }
            w = nw;
        }
    }

    // ------------------------------- reduction and output ---------------------------------
    const uint32_t q = warp;  // epilogue warps: tensor-memory lane quarter == 32 of the tile's columns
    const uint32_t n = n0 + q * 32u + lane;
    const uint32_t acc = tmem_base + ((q & 3u) << 21);
    const uint32_t rows = min(MT, p.M - m0);
    const uint32_t per = max(4u, MT / parts), shift = __ffs(per) - 1;  // rows a part owns (a power of two)
    const uint32_t col_of_tile = (q & 3u) * 32u + lane;
    // float index of four rows (group j of a part's own) of this lane's column: the groups are rotated by the column so that
    // a warp's 16-byte accesses spread over the banks
    auto piece = [&](uint32_t slot, uint32_t j) {
        return ((slot * 128u + col_of_tile) << shift) + ((j ^ (col_of_tile & ((per >> 2) - 1u))) << 2);
    };
    if (warp < 4) {
        alive = alive && mbar_wait_warp(acc_full, 0, p.status, 308, 0, bar_ns);
        tcgen05_fence_after();
    }
    __syncwarp();
    if (parts > 1u) {
        const uint32_t red = smem_u32(smem + S::kOffRed);
        cluster_wait();
        if (!alive && lane == 0) {
            for (uint32_t d = 0; d < parts; ++d) {
                st_shared_cluster_u32(map_to_cta(smem_u32(dead), d), 1u);
            }
        }
        __syncwarp();
        if (warp < 4 && alive) {
            for (uint32_t c0 = 0; c0 < rows; c0 += 16) {
                uint32_t r[16];
                tmem_ld_32x16(acc + c0, r);
                tmem_ld_wait();
#pragma unroll
                for (uint32_t g = 0; g < 4; ++g) {
                    const uint32_t col = c0 + 4u * g, d = col >> shift;
                    if (col < rows && d != part) {
                        const uint32_t at = piece(part - (part > d ? 1u : 0u), (col - (d << shift)) >> 2);
                        st_shared_cluster_v4(map_to_cta(red + at * 4u, d), r[4 * g], r[4 * g + 1], r[4 * g + 2], r[4 * g + 3]);
                    }
                }
            }
        }
        __syncwarp();
        cluster_sync_all();
        if (*reinterpret_cast<volatile uint32_t*>(dead) != 0u) {
            alive = false;
        }
        if (warp < 4 && alive) {
            const float* pieces = reinterpret_cast<const float*>(smem + S::kOffRed);
            const uint32_t own0 = part << shift, own1 = min(own0 + per, rows);
            for (uint32_t c0 = own0 & ~15u; c0 < own1; c0 += 16) {
                uint32_t r[16];
                tmem_ld_32x16(acc + c0, r);
                tmem_ld_wait();
#pragma unroll
                for (uint32_t g = 0; g < 4; ++g) {
                    const uint32_t col = c0 + 4u * g;
                    if (col < own0 || col >= own1) {
                        continue;
                    }
                    float4 v[kSmallMaxParts];
#pragma unroll
                    for (uint32_t src = 0; src < kSmallMaxParts; ++src) {
                        v[src] = make_float4(__uint_as_float(r[4 * g]), __uint_as_float(r[4 * g + 1]),
                                             __uint_as_float(r[4 * g + 2]), __uint_as_float(r[4 * g + 3]));
                        if (src < parts && src != part) {
                            v[src] = *reinterpret_cast<const float4*>(
                                pieces + piece(src - (src > part ? 1u : 0u), (col - own0) >> 2));
                        }
                    }
                    float4 sum = v[0];
#pragma unroll
                    for (uint32_t src = 1; src < kSmallMaxParts; ++src) {
                        if (src < parts) {
                            sum.x += v[src].x;
                            sum.y += v[src].y;
                            sum.z += v[src].z;
                            sum.w += v[src].w;
                        }
                    }
                    const float out[4] = {sum.x, sum.y, sum.z, sum.w};
#pragma unroll
                    for (uint32_t e = 0; e < 4; ++e) {
                        if (col + e < own1) {
                            store_small<OutT>(p, m0 + col + e, n, lane, out[e]);
                        }
                    }
                }
            }
        }
    } else if (warp < 4 && alive) {
        for (uint32_t c0 = 0; c0 < rows; c0 += 16) {
            uint32_t r[16];
            tmem_ld_32x16(acc + c0, r);
            tmem_ld_wait();
#pragma unroll
            for (uint32_t e = 0; e < 16; ++e) {
                if (c0 + e < rows) {
                    store_small<OutT>(p, m0 + c0 + e, n, lane, __uint_as_float(r[e]));
                }
            }
        }
    }

    tcgen05_fence_before();
    if (__syncthreads_or(alive ? 0 : 1)) {
        drain_after_abort(p.status);
    }
    if (warp == 5) {
        tcgen05_fence_after();
        tmem_dealloc(tmem_base, S::kTmemCols);
    }
}

}  // namespace catccos
