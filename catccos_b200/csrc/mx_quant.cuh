// MX quantise-and-push kernel for sm_100a: bf16 [M, K] -> E4M3 codes + one E8M0 scale per 32
// K-elements, stored straight into every destination rank's buffer (peer-mapped over NVLink), with a
// ready flag per (source rank, 16-row chunk).
//
// It replaces the vector-core program of the reference:
//   arithmetic   include/catccos/comm/block/comm_block_mx_quant.hpp:413-523,569-664 (ComputeMxQuant, FP8)
//   streaming    include/catccos/comm/block/comm_block_mx_quant.hpp:155-207 (operator())
//   allgather    include/catccos/comm/kernel/mx_quant_allgather.hpp:132-287 (quantise into the symmetric
//                stage, signal, peers GET) - here the direction is PUT: quantise once, store to all.
//
// Arithmetic per 32-element block (bit-exact with the reference's CPU golden, "native" rounding):
//   E = biased exponent of the largest |x|;  scale byte = E - 8;  code = RNE_sat_E4M3(x * 2^(127 - byte)).
//   Blocks whose largest |x| is below 1e-12 follow the golden (scale byte 0x7F, signed-zero codes) or,
//   in mode kQuantDeviceTiny, the reference device kernel (byte = max(E - 8, 0)).  Inf/NaN blocks: 0xFF / 0x7F.
#pragma once

#include <cuda_fp4.h>

#include "common.cuh"
#include "wait_records.hpp"
#include "trace.cuh"

namespace catccos {

constexpr uint32_t kQuantThreads = 256;
constexpr uint32_t kQuantRowsPerItem = 16;  // == kRowsPerChunk of the GEMM gate: 8 warps x 2 rows
constexpr uint32_t kQuantColsPerWarpStep = 512;
constexpr uint32_t kQuantGolden = 0;        // tiny blocks follow the CPU golden
constexpr uint32_t kQuantDeviceTiny = 1;    // tiny blocks follow the reference device kernel
constexpr uint32_t kQuantPreQuantised = 2;  // input is already codes + scales: copy and publish only

struct QuantPushParams {
    // producer: this rank's shard
    const void* in;           // bf16 [M, K]  (or, for the pre-quantised push, E4M3 codes [M, K])
    const uint8_t* in_scales; // pre-quantised push only: E8M0 [M, K/32]
    uint32_t M, K;
    uint32_t mode;            // kQuantGolden / kQuantDeviceTiny / kQuantPreQuantised
    uint32_t e5m2;            // 0 = E4M3 codes (emax 8, +-448), 1 = E5M2 codes (emax 15, +-57344)
    uint32_t produce;         // 0: skip the producer part (the harness that runs the two parts apart)
    uint32_t publish;         // 0: nobody waits on this shard's flags (single rank, plain quantise)
    uint32_t sys_scope;       // 1: some destination is another GPU (system-scope fences), 0: all local
    uint32_t rank, world, epoch;
    uint32_t segs_per_chunk;  // a 16-row chunk is split into this many column segments (work items)
    uint32_t seg_cols;        // columns per segment (multiple of 512)
    uint32_t group_chunks;    // work items are ordered group by group (this many chunks), segment-major inside
    uint32_t seg_order_n;     // 0, or the number of entries of seg_order
    uint8_t seg_order[32];    // the order in which the K segments are visited (a split-K consumer wants the first
                              // segment of each of its K parts first, then the second of each, ...)
    uint32_t num_dst;
    uint8_t* dst_codes[kMaxRanks];   // where this shard's codes [M, K] go at destination d
    uint8_t* dst_scales[kMaxRanks];  // where this shard's scales [M, K/32] go at destination d
    uint32_t* dst_flags[kMaxRanks];  // destination d's flag words for this source, one per (chunk, segment)
                                     // at index chunk * segs_per_chunk + segment, or nullptr
    // consumer (standalone quantise + allgather with outputs outside symmetric memory):
    // copy the peers' shards from this GPU's stage to the caller's outputs as their flags arrive
    uint32_t consume;
    const uint8_t* stage_codes;   // [world][M][K]
    const uint8_t* stage_scales;  // [world][M][K/32]
    uint8_t* out_codes;           // [world * M, K]
    uint8_t* out_scales;          // [world * M, K/32]
    const uint32_t* flags;        // this GPU's flag words [world][flag_stride]
    uint32_t flag_stride;
    uint64_t timeout_ns;
    StatusBlock* status;
    unsigned long long* trace;    // timeline side buffer (trace build only), else nullptr
};

__device__ __forceinline__ uint32_t absmax_bits8(uint4 v)
{
    uint32_t m = __vmaxu2(__vmaxu2(v.x & 0x7FFF7FFFu, v.y & 0x7FFF7FFFu), __vmaxu2(v.z & 0x7FFF7FFFu, v.w & 0x7FFF7FFFu));
    return max(m & 0xFFFFu, m >> 16);
}

// two fp32 -> two E4M3 codes (round to nearest even, saturate to +-448), first value in the low byte
__device__ __forceinline__ uint32_t cvt_e4m3x2(float lo, float hi)
{
    uint16_t r;
    asm("cvt.rn.satfinite.e4m3x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ uint32_t cvt_e5m2x2(float lo, float hi)
{
    uint16_t r;
    asm("cvt.rn.satfinite.e5m2x2.f32 %0, %1, %2;" : "=h"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ uint32_t encode4(uint32_t a, uint32_t b, float mul, bool e5m2)
{
    const float a0 = __uint_as_float(a << 16) * mul, a1 = __uint_as_float(a & 0xFFFF0000u) * mul;
    const float b0 = __uint_as_float(b << 16) * mul, b1 = __uint_as_float(b & 0xFFFF0000u) * mul;
    if (e5m2) {
        return cvt_e5m2x2(a0, a1) | (cvt_e5m2x2(b0, b1) << 16);
    }
    return cvt_e4m3x2(a0, a1) | (cvt_e4m3x2(b0, b1) << 16);
}

// Scale byte and multiplier for a block whose largest |bf16 bits| is amax.
__device__ __forceinline__ void block_scale(uint32_t amax, bool device_tiny, uint32_t emax, uint32_t& byte, float& mul,
                                            bool& nonfinite)
{
    const uint32_t E = amax >> 7;
    nonfinite = (E == 0xFFu);
    if (device_tiny) {
        byte = E > emax ? E - emax : 0u;
        mul = byte == 0u ? 0.0f : __uint_as_float((254u - byte) << 23);
    } else {
        const bool tiny = amax <= 0x2B8Cu;  // |x| < 1e-12 for every bf16 in the block
        byte = tiny ? 0x7Fu : E - emax;
        mul = tiny ? 0.0f : __uint_as_float((254u - byte) << 23);
    }
    if (nonfinite) {
        byte = 0xFFu;
    }
}

// Quantises 16 bf16 values held by one lane (two lanes share a 32-block).
__device__ __forceinline__ uint4 quant16(uint4 v0, uint4 v1, bool device_tiny, bool e5m2, uint32_t& byte)
{
    uint32_t amax = max(absmax_bits8(v0), absmax_bits8(v1));
    amax = max(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    float mul;
    bool nonfinite;
    block_scale(amax, device_tiny, e5m2 ? 15u : 8u, byte, mul, nonfinite);
    uint4 o;
    o.x = encode4(v0.x, v0.y, mul, e5m2);
    o.y = encode4(v0.z, v0.w, mul, e5m2);
    o.z = encode4(v1.x, v1.y, mul, e5m2);
    o.w = encode4(v1.z, v1.w, mul, e5m2);
    if (nonfinite) {
        o = make_uint4(0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu, 0x7F7F7F7Fu);
    }
    return o;
}

// 16 bf16 values (half a 32-block) of one lane.  The caller's pointer is 16-byte aligned at least; where it is 32-byte
// aligned (the same answer for every lane) one full-sector load takes both halves.
__device__ __forceinline__ void load_half_block(const void* p, uint4& v0, uint4& v1)
{
    if (((uintptr_t)p & 31u) == 0u) {
        ld_global_stream_v8(p, v0, v1);
    } else {
        v0 = __ldcs(static_cast<const uint4*>(p));
        v1 = __ldcs(static_cast<const uint4*>(p) + 1);
    }
}

// Barrier among the 256 threads of one quantise group (barrier 0 when the group is the whole CTA).
__device__ __forceinline__ void quant_group_sync(uint32_t bar_id)
{
    asm volatile("bar.sync %0, %1;" ::"r"(bar_id), "r"(kQuantThreads) : "memory");
}

// Publishing a finished work item: every thread's stores are ordered before the flag words.  The fences
// are system-scope only when a destination is another GPU; a single-GPU run stays at GPU scope.
// Order of the work items.  Inside a group of `group_chunks` chunks the items run segment-major (the first
// K segment of every row of the group first), so a consumer that walks K in order can start early and
// follow the quantiser; groups follow one another, so a consumer with several waves of tiles gets complete
// rows for its first wave while the rest is still on its way.  group_chunks >= chunks: one group.
// `order` (n entries, n == segs, or n == 0 for the natural order) maps the position in that walk to the segment.
__host__ __device__ __forceinline__ void item_coord(uint32_t item, uint32_t chunks, uint32_t segs, uint32_t group_chunks,
                                           const uint8_t* order, uint32_t order_n, uint32_t& chunk, uint32_t& seg)
{
    const uint32_t gc = group_chunks == 0u || group_chunks > chunks ? chunks : group_chunks;
    const uint32_t per_group = gc * segs;
    const uint32_t g = item / per_group;
    const uint32_t rem = item - g * per_group;
    const uint32_t cg = min(gc, chunks - g * gc);
    seg = rem / cg;
    chunk = g * gc + (rem - seg * cg);
    if (order_n == segs) {
        seg = order[seg];
    }
}

// One work item = one (16-row chunk, column segment), owned by exactly one group, which publishes it alone.
__device__ __forceinline__ void publish_item(const QuantPushParams& p, uint32_t flag_index, uint32_t tid, uint32_t bar_id)
{
    const unsigned long long t0 = CATCCOS_TR_NOW();
    (void)t0;
    quant_group_sync(bar_id);
    if (tid == 0) {
        if (p.sys_scope) {
            __threadfence_system();
        } else {
            __threadfence();
        }
#pragma unroll
        for (uint32_t d = 0; d < (uint32_t)kMaxRanks; ++d) {
            if (d < p.num_dst && p.dst_flags[d] != nullptr) {
                // the fence above already ordered the data; the flag itself can be a relaxed store
                asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p.dst_flags[d] + flag_index), "r"(p.epoch)
                             : "memory");
            }
        }
        CATCCOS_TR_ADD(p.trace, kTrQuantPublishNs, CATCCOS_TR_NOW() - t0);
        CATCCOS_TR_ADD(p.trace, kTrQuantItems, 1ull);
        CATCCOS_TR_STAMP_FIRST(p.trace, kTrQuantFirstDone);
        CATCCOS_TR_STAMP(p.trace, kTrQuantDone);
    }
}

// The producer: a group of 256 threads (tid 0..255) takes work items worker, worker + num_workers, ...
// and for each quantises (or copies) 16 rows x one column segment, stores the result at every
// destination and publishes the item's flag.  It never waits on anybody.
// kPrefetch: the loads of the next 512-column step are issued before the current one is encoded (eight
// 16-byte loads in flight per lane).  Worth its registers where only one producer group runs per SM
// (inside the GEMM kernel); the stand-alone kernel prefers more resident CTAs.
template <bool kPrefetch>
__device__ __forceinline__ void quant_push_producer(const QuantPushParams& p, uint32_t tid, uint32_t worker,
                                                    uint32_t num_workers, uint32_t bar_id)
{
    const uint32_t warp = tid >> 5;
    const uint32_t lane = tid & 31;
    const uint32_t chunks = (p.M + kQuantRowsPerItem - 1) / kQuantRowsPerItem;
    const uint32_t items = p.produce ? chunks * p.segs_per_chunk : 0u;
    const uint32_t sf_cols = p.K / 32;
    const bool sf_vec = (sf_cols % 4u) == 0u;
    const bool prequant = p.mode == kQuantPreQuantised;
    const bool device_tiny = p.mode == kQuantDeviceTiny;
    const bool e5m2 = p.e5m2 != 0u;

    // loads one 512-column step (two rows of this warp) of the item whose first row for this warp is row0
    auto load_step = [&](uint32_t row0, uint32_t cb, uint32_t c_end, uint4 (&dst)[2][2]) {
        const uint32_t col = cb + lane * 16;
#pragma unroll
        for (uint32_t r = 0; r < 2; ++r) {
            const uint32_t row = row0 + r;
            dst[r][0] = dst[r][1] = make_uint4(0, 0, 0, 0);
            if (col < c_end && row < p.M) {
                if (prequant) {
                    dst[r][0] = __ldcs(reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(p.in) +
                                                                     (size_t)row * p.K + col));
                } else {
                    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.in) +
                                                                      (size_t)row * p.K + col);
                    dst[r][0] = __ldcs(src);
                    dst[r][1] = __ldcs(src + 1);
                }
            }
        }
    };
    uint4 v[2][2], vn[2][2];
    bool first_loaded = false;  // kPrefetch: the item's first step was requested while the previous item finished

    for (uint32_t item = worker; item < items; item += num_workers) {
        uint32_t chunk, seg;
        item_coord(item, chunks, p.segs_per_chunk, p.group_chunks, p.seg_order, p.seg_order_n, chunk, seg);
        const uint32_t c_begin = seg * p.seg_cols;
        const uint32_t c_end = min(p.K, c_begin + p.seg_cols);
        const uint32_t row0 = chunk * kQuantRowsPerItem + warp * 2;

        if (kPrefetch && !first_loaded) {
            load_step(row0, c_begin, c_end, v);
        }
        for (uint32_t cb = c_begin; cb < c_end; cb += kQuantColsPerWarpStep) {
            const uint32_t col = cb + lane * 16;
            const bool col_ok = col < c_end;
            const bool has_next = kPrefetch && cb + kQuantColsPerWarpStep < c_end;
            if (kPrefetch) {
                if (has_next) {
                    load_step(row0, cb + kQuantColsPerWarpStep, c_end, vn);
                }
            } else {
                load_step(row0, cb, c_end, v);  // both rows first: four 16-byte loads in flight per lane
            }
            uint4 o[2];
            uint32_t byte[2];
#pragma unroll
            for (uint32_t r = 0; r < 2; ++r) {
                const uint32_t row = row0 + r;
                if (prequant) {
                    o[r] = v[r][0];
                    byte[r] = 0;
                    if (col_ok && row < p.M && (lane & 1u) == 0u) {
                        byte[r] = p.in_scales[(size_t)row * sf_cols + col / 32];
                    }
                } else {
                    o[r] = quant16(v[r][0], v[r][1], device_tiny, e5m2, byte[r]);
                }
                // scale bytes of 8 lanes (4 blocks) packed into one word on lanes 0, 8, 16, 24
                const uint32_t base = lane & ~7u;
                uint32_t w = __shfl_sync(0xFFFFFFFFu, byte[r], base) |
                             (__shfl_sync(0xFFFFFFFFu, byte[r], base + 2) << 8) |
                             (__shfl_sync(0xFFFFFFFFu, byte[r], base + 4) << 16) |
                             (__shfl_sync(0xFFFFFFFFu, byte[r], base + 6) << 24);
                if (col_ok && row < p.M) {
                    const size_t code_off = (size_t)row * p.K + col;
                    const size_t sf_off = (size_t)row * sf_cols + col / 32;
#pragma unroll
                    for (uint32_t d = 0; d < (uint32_t)kMaxRanks; ++d) {
                        if (d >= p.num_dst || p.dst_codes[d] == nullptr) {
                            continue;
                        }
                        *reinterpret_cast<uint4*>(p.dst_codes[d] + code_off) = o[r];
                        if (sf_vec) {
                            if ((lane & 7u) == 0u) {
                                *reinterpret_cast<uint32_t*>(p.dst_scales[d] + sf_off) = w;
                            }
                        } else if ((lane & 1u) == 0u) {
                            p.dst_scales[d][sf_off] = (uint8_t)byte[r];
                        }
                    }
                }
            }
            if (has_next) {
#pragma unroll
                for (uint32_t r = 0; r < 2; ++r) {
                    v[r][0] = vn[r][0];
                    v[r][1] = vn[r][1];
                }
            }
        }
        first_loaded = false;
        if (kPrefetch && item + num_workers < items) {
            // the next item's first step travels while this item is published (a barrier, a fence, the flags)
            uint32_t chunk2, seg2;
            item_coord(item + num_workers, chunks, p.segs_per_chunk, p.group_chunks, p.seg_order, p.seg_order_n, chunk2, seg2);
            const uint32_t cb2 = seg2 * p.seg_cols;
            load_step(chunk2 * kQuantRowsPerItem + warp * 2, cb2, min(p.K, cb2 + p.seg_cols), v);
            first_loaded = true;
        }
        if (p.publish) {
            publish_item(p, chunk * p.segs_per_chunk + seg, tid, bar_id);
        }
    }
}

// The quantiser for one destination and no flags (a single rank, the plain quantise calls).  Rows hold whole 32-blocks
// and all three arrays are dense, so the matrix is a flat run of blocks whatever its shape: a lane takes 16 consecutive
// values (32 bytes in, 16 bytes of codes out, two lanes share a scale), a warp 1 KiB, and every block of the grid is one
// such step per warp and ends.  HBM-bound: the loads of a few hundred resident warps are all in flight at once, ragged
// shapes split evenly, nothing loops.  Measured (B200, back to back): bf16 [4096, 7168] 24.4 us with the item loop of
// quant_push_producer, 14.4 us here (6.2 TB/s); [1024, 7168] 8.4 -> 3.5 us.  More steps per warp, or a grid of one wave
// that loops, measure 1-5 % slower.
template <bool kE5m2>
__global__ void __launch_bounds__(kQuantThreads) mx_quant_flat_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ codes,
                                                                      uint8_t* __restrict__ scales, uint64_t halves,
                                                                      uint32_t device_tiny, StatusBlock* reset)
{
    grid_dep_wait();
    if (reset != nullptr && blockIdx.x == 0 && threadIdx.x < kWaitRecords) {
        reset[threadIdx.x] = StatusBlock{};
        __threadfence();  // before the GEMM behind this kernel may look at it
    }
    grid_dep_launch();
    const uint64_t i = (uint64_t)blockIdx.x * kQuantThreads + threadIdx.x;
    uint4 v0 = make_uint4(0, 0, 0, 0), v1 = v0;
    if (i < halves) {
        load_half_block(in + i * 32, v0, v1);
    }
    uint32_t byte;
    const uint4 o = quant16(v0, v1, device_tiny != 0u, kE5m2, byte);
    if (i < halves) {
        *reinterpret_cast<uint4*>(codes + i * 16) = o;
        if ((i & 1u) == 0u) {
            scales[i >> 1] = (uint8_t)byte;
        }
    }
}

// What a pusher warp needs: where this rank's quantised shard lives locally and where it goes.
struct PushParams {
    const uint8_t* src_codes;   // this rank's shard in its own stage: codes [M, K]
    const uint8_t* src_scales;  //                                      scales [M, K/32]
    const uint32_t* src_flags;  // this GPU's flag words for its own shard (published by the quantise warps), or
                                // nullptr when the shard was complete before the kernel started
    uint8_t* dst_codes[kMaxRanks];   // the same shard's place in rank d's stage (nullptr for d == rank)
    uint8_t* dst_scales[kMaxRanks];
    uint32_t* dst_flags[kMaxRanks];  // rank d's flag words for this source
    uint32_t M, K, rank, world, epoch;
    uint32_t segs_per_chunk, seg_cols, group_chunks, seg_order_n;
    uint8_t seg_order[32];
    uint64_t timeout_ns;
    StatusBlock* status;
    unsigned long long* trace;  // timeline side buffer (trace build only), else nullptr
};

// The pusher: one warp forwards finished work items of this rank's shard from the local stage to the peers.
// Pusher `worker` of `num_workers` takes items worker, worker + num_workers, ... in item order, so early K
// segments leave first.  For an item it waits (bounded) for the quantise warps' local flag, then moves the
// 16 rows x one K segment in passes of 4 KiB: eight 16-byte loads in flight per lane, each value stored to
// every peer (the local stage is read once, whatever the number of ranks; the peers are visited starting
// behind this rank so that the ranks of a box do not all store to the same GPU at the same moment).  One
// system-scope fence per item orders the stores before the peers' flag words.
//
// The pushers of a CTA take turns (`turn`, a word in shared memory that counts the CTA's items): a pusher loads
// its item's first pass, waits until the item before it has been stored, fenced and flagged, and then does the
// same.  Every CTA thus feeds NVLink one item after the other, in item order, and all CTAs together keep about
// one bandwidth-delay product in flight.  When all pushers fire at once instead, the link delivers all items at
// the same slow pace and the first rows the GEMM needs arrive with the last.
// `pw` names the pusher inside its CTA, `grid` is the number of CTAs (worker = pw * grid + CTA index).
__device__ __forceinline__ void push_worker(const PushParams& p, uint32_t lane, uint32_t worker, uint32_t num_workers,
                                            uint32_t pw, uint32_t grid, uint32_t* turn)
{
    (void)pw;
    if (p.world < 2) {
        return;
    }
    const uint32_t chunks = (p.M + kQuantRowsPerItem - 1) / kQuantRowsPerItem;
    const uint32_t items = chunks * p.segs_per_chunk;
    const uint32_t peers = p.world - 1;
    const uint32_t sf_cols = p.K / 32;
    for (uint32_t item = worker; item < items; item += num_workers) {
        const uint32_t seq = item / grid;  // this item's place among the CTA's items
        uint32_t chunk, seg;
        item_coord(item, chunks, p.segs_per_chunk, p.group_chunks, p.seg_order, p.seg_order_n, chunk, seg);
        const uint32_t flag_index = chunk * p.segs_per_chunk + seg;
        if (p.src_flags != nullptr) {
            const unsigned long long t0 = CATCCOS_TR_NOW();
            (void)t0;
            bool ok = true;
            if (lane == 0 && !wait_flag_ge(p.src_flags + flag_index, p.epoch, p.timeout_ns, p.status)) {
                report_status(p.status, kStatusFlagTimeout, p.rank, chunk, p.epoch);
                ok = false;
            }
            if (!__all_sync(0xFFFFFFFFu, ok)) {
                return;  // the quantise warps of this launch will not deliver: nothing sensible left to push
            }
            __syncwarp();  // lane 0 acquired the flag; a vote orders no memory
            if (lane == 0) {
                CATCCOS_TR_ADD(p.trace, kTrPushFlagWaitNs + pw, CATCCOS_TR_NOW() - t0);
            }
        }
        if (lane == 0) {
            CATCCOS_TR_STAMP_FIRST(p.trace, kTrPushFirst + pw);
        }
        const uint32_t c_begin = seg * p.seg_cols;
        const uint32_t cols = min(p.K, c_begin + p.seg_cols) - c_begin;
        const uint32_t r_begin = chunk * kQuantRowsPerItem;
        const uint32_t rows = min(p.M, r_begin + kQuantRowsPerItem) - r_begin;
        // codes: rows x cols bytes, 16 bytes per lane per step, eight steps in flight
        const uint32_t per_row = cols / 16;
        const uint32_t n16 = rows * per_row;
        uint4 v[8];
        size_t off[8];
        auto load_pass = [&](uint32_t i) {
#pragma unroll
            for (uint32_t j = 0; j < 8; ++j) {
                const uint32_t e = i + j * 32;
                const uint32_t r = e / per_row;
                off[j] = (size_t)(r_begin + r) * p.K + c_begin + (size_t)(e - r * per_row) * 16;
                if (e < n16) {
                    v[j] = __ldcg(reinterpret_cast<const uint4*>(p.src_codes + off[j]));
                }
            }
        };
        load_pass(lane);  // the first pass travels while this pusher waits for its turn
        if (turn != nullptr) {
            bool ok = true;
            if (lane == 0) {
                const uint64_t t0 = globaltimer_ns();
                uint32_t spins = 0;
                while (*reinterpret_cast<volatile uint32_t*>(turn) != seq) {
                    if ((++spins & 0x3Fu) == 0u) {
                        if (globaltimer_ns() - t0 > p.timeout_ns || status_tripped(p.status)) {
                            ok = false;
                            break;
                        }
                        __nanosleep(64);
                    }
                }
            }
            if (!__all_sync(0xFFFFFFFFu, ok)) {
                return;  // an earlier pusher of this CTA gave up
            }
        }
        for (uint32_t i = lane; i < n16; i += 256) {
            if (i != lane) {
                load_pass(i);
            }
            for (uint32_t t = 0; t < peers; ++t) {
                uint8_t* dst = p.dst_codes[(p.rank + 1 + t) % p.world];
#pragma unroll
                for (uint32_t j = 0; j < 8; ++j) {
                    if (i + j * 32 < n16) {
                        *reinterpret_cast<uint4*>(dst + off[j]) = v[j];
                    }
                }
            }
        }
        // scales: rows x cols/32 bytes
        const uint32_t sf_per_row = cols / 32;
        if ((sf_per_row % 4u) == 0u && (sf_cols % 4u) == 0u) {
            const uint32_t w_per_row = sf_per_row / 4;
            for (uint32_t e = lane; e < rows * w_per_row; e += 32) {
                const uint32_t r = e / w_per_row;
                const size_t so = (size_t)(r_begin + r) * sf_cols + c_begin / 32 + (size_t)(e - r * w_per_row) * 4;
                const uint32_t w = __ldcg(reinterpret_cast<const uint32_t*>(p.src_scales + so));
                for (uint32_t t = 0; t < peers; ++t) {
                    *reinterpret_cast<uint32_t*>(p.dst_scales[(p.rank + 1 + t) % p.world] + so) = w;
                }
            }
        } else {
            for (uint32_t e = lane; e < rows * sf_per_row; e += 32) {
                const uint32_t r = e / sf_per_row;
                const size_t so = (size_t)(r_begin + r) * sf_cols + c_begin / 32 + (e - r * sf_per_row);
                const uint8_t b = __ldcg(p.src_scales + so);
                for (uint32_t t = 0; t < peers; ++t) {
                    p.dst_scales[(p.rank + 1 + t) % p.world][so] = b;
                }
            }
        }
        __syncwarp();
        if (lane == 0) {
            const unsigned long long t1 = CATCCOS_TR_NOW();
            (void)t1;
            __threadfence_system();
            CATCCOS_TR_ADD(p.trace, kTrPushFenceNs + pw, CATCCOS_TR_NOW() - t1);
            for (uint32_t t = 0; t < peers; ++t) {
                asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p.dst_flags[(p.rank + 1 + t) % p.world] + flag_index),
                             "r"(p.epoch)
                             : "memory");
            }
            if (turn != nullptr) {
                // The turn passes on only now.  A fence waits for the stores the whole SM has in flight, not only
                // for this warp's: were the next item's stores let out before it, this item's flags would wait
                // for them too, and so on down the line, and every flag would arrive with the last item.
                *reinterpret_cast<volatile uint32_t*>(turn) = seq + 1u;
            }
            CATCCOS_TR_ADD(p.trace, kTrPushItems + pw, 1ull);
            CATCCOS_TR_STAMP(p.trace, kTrPushLast + pw);
        }
    }
}

// kPrefetch: see quant_push_producer; chosen by the host when only one or two CTAs run per SM (a grid cut down so
// that the items of a multi-rank push leave in order) and every CTA works through several items.
template <bool kPrefetch>
__global__ void __launch_bounds__(kQuantThreads) mx_quant_push_kernel(QuantPushParams p)
{
    grid_dep_wait();    // `in` may be the predecessor's output, and the outputs may be what it still reads
    grid_dep_launch();  // a GEMM launched behind this kernel may set itself up while the quantiser drains
#ifdef CATCCOS_TRACE
    if (p.trace != nullptr && threadIdx.x == 0) {
        atomicMin(p.trace + kTrQuantKernelStart, globaltimer_ns());
    }
    QuantPushParams pq = p;
    pq.trace = nullptr;  // the per-CTA rows belong to the GEMM kernel's CTAs
    quant_push_producer<kPrefetch>(pq, threadIdx.x, blockIdx.x, gridDim.x, 0);
    if (p.trace != nullptr) {
        __syncthreads();
        if (threadIdx.x == 0) {
            atomicMax(p.trace + kTrQuantKernelEnd, globaltimer_ns());
        }
    }
#else
    quant_push_producer<kPrefetch>(p, threadIdx.x, blockIdx.x, gridDim.x, 0);
#endif

    if (!p.consume) {
        return;
    }
    const uint32_t chunks = (p.M + kQuantRowsPerItem - 1) / kQuantRowsPerItem;
    const uint32_t sf_cols = p.K / 32;
    // ---- consumer: stage -> caller's outputs, chunk by chunk as the peers' flags arrive ----
    const uint32_t peer_items = (p.world - 1) * chunks;
    for (uint32_t item = blockIdx.x; item < peer_items; item += gridDim.x) {
        const uint32_t chunk = item / (p.world - 1);
        const uint32_t src = (p.rank + 1 + item % (p.world - 1)) % p.world;
        if (threadIdx.x < p.segs_per_chunk) {
            const uint32_t* f = p.flags + (size_t)src * p.flag_stride + chunk * p.segs_per_chunk + threadIdx.x;
            if (!wait_flag_ge(f, p.epoch, p.timeout_ns, p.status)) {
                report_status(p.status, kStatusFlagTimeout, src, chunk, p.epoch);
            }
        }
        __syncthreads();
        const uint32_t r_begin = chunk * kQuantRowsPerItem;
        const uint32_t r_end = min(p.M, r_begin + kQuantRowsPerItem);
        const size_t shard = (size_t)src * p.M;
        // codes: rows are contiguous in both buffers, so the chunk is one flat span
        {
            const size_t off = (shard + r_begin) * p.K;
            const size_t bytes = (size_t)(r_end - r_begin) * p.K;
            const uint4* s = reinterpret_cast<const uint4*>(p.stage_codes + off);
            uint4* d = reinterpret_cast<uint4*>(p.out_codes + off);
            for (size_t i = threadIdx.x; i < bytes / 16; i += kQuantThreads) {
                __stcs(d + i, __ldcg(s + i));
            }
        }
        {
            const size_t off = (shard + r_begin) * sf_cols;
            const size_t bytes = (size_t)(r_end - r_begin) * sf_cols;
            if (((off | bytes) & 3u) == 0u) {
                const uint32_t* s = reinterpret_cast<const uint32_t*>(p.stage_scales + off);
                uint32_t* d = reinterpret_cast<uint32_t*>(p.out_scales + off);
                for (size_t i = threadIdx.x; i < bytes / 4; i += kQuantThreads) {
                    d[i] = __ldcg(s + i);
                }
            } else {
                for (size_t i = threadIdx.x; i < bytes; i += kQuantThreads) {
                    p.out_scales[off + i] = __ldcg(p.stage_scales + off + i);
                }
            }
        }
        __syncthreads();
    }
}

// The quantise-and-push kernel for several ranks when the GEMM runs beside it: one CTA per SM (or two) works through
// its items strictly one after the other, and for every item
//   1. has all of the item's input in flight at once (up to sixteen 16-byte loads per lane: one trip to HBM),
//   2. quantises, and requests the next item's input before it stores anything,
//   3. stores the item to this rank's own stage, fences at GPU scope and sets the local flag - the GEMM's tiles
//      over this rank's own rows can start while the item is still on its way to the peers,
//   4. stores the same registers to every peer, fences at system scope and sets the peers' flags.
// A fence waits for the stores the whole SM has in flight, so an SM that keeps one item in flight publishes
// each item as soon as that item has landed; all SMs together keep about one bandwidth-delay product of NVLink
// busy, and the items arrive in item order (the rows of the GEMM's first wave first).
// Needs seg_cols <= kOrderedMaxSteps * 512 (the host caps the K segments accordingly).
constexpr uint32_t kOrderedMaxSteps = 4;

// (launch bounds: at most 128 registers per thread, so that this CTA and the GEMM's CTA fit one SM's register file)
__global__ void __launch_bounds__(kQuantThreads, 2) mx_quant_push_ordered_kernel(QuantPushParams p)
{
    grid_dep_launch();
#ifdef CATCCOS_TRACE
    if (p.trace != nullptr && threadIdx.x == 0) {
        atomicMin(p.trace + kTrQuantKernelStart, globaltimer_ns());
    }
#endif
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t chunks = (p.M + kQuantRowsPerItem - 1) / kQuantRowsPerItem;
    const uint32_t items = p.produce ? chunks * p.segs_per_chunk : 0u;
    const uint32_t sf_cols = p.K / 32;
    const bool sf_vec = (sf_cols % 4u) == 0u;
    const bool prequant = p.mode == kQuantPreQuantised;
    const bool device_tiny = p.mode == kQuantDeviceTiny;
    const bool e5m2 = p.e5m2 != 0u;

    uint4 in[kOrderedMaxSteps][2][2];
    auto load_item = [&](uint32_t item) {
        uint32_t chunk, seg;
        item_coord(item, chunks, p.segs_per_chunk, p.group_chunks, p.seg_order, p.seg_order_n, chunk, seg);
        const uint32_t c_begin = seg * p.seg_cols;
        const uint32_t c_end = min(p.K, c_begin + p.seg_cols);
        const uint32_t row0 = chunk * kQuantRowsPerItem + warp * 2;
#pragma unroll
        for (uint32_t st = 0; st < kOrderedMaxSteps; ++st) {
            const uint32_t col = c_begin + st * kQuantColsPerWarpStep + lane * 16;
#pragma unroll
            for (uint32_t r = 0; r < 2; ++r) {
                const uint32_t row = row0 + r;
                in[st][r][0] = in[st][r][1] = make_uint4(0, 0, 0, 0);
                if (col < c_end && row < p.M) {
                    if (prequant) {
                        in[st][r][0] = __ldcs(reinterpret_cast<const uint4*>(static_cast<const uint8_t*>(p.in) +
                                                                            (size_t)row * p.K + col));
                    } else {
                        const uint4* src = reinterpret_cast<const uint4*>(static_cast<const uint16_t*>(p.in) +
                                                                          (size_t)row * p.K + col);
                        in[st][r][0] = __ldcs(src);
                        in[st][r][1] = __ldcs(src + 1);
                    }
                }
            }
        }
    };

    uint32_t item = blockIdx.x;
    if (item < items) {
        load_item(item);
    }
    for (; item < items; item += gridDim.x) {
        uint32_t chunk, seg;
        item_coord(item, chunks, p.segs_per_chunk, p.group_chunks, p.seg_order, p.seg_order_n, chunk, seg);
        const uint32_t c_begin = seg * p.seg_cols;
        const uint32_t c_end = min(p.K, c_begin + p.seg_cols);
        const uint32_t row0 = chunk * kQuantRowsPerItem + warp * 2;
        const uint32_t flag_index = chunk * p.segs_per_chunk + seg;

        uint4 o[kOrderedMaxSteps][2];
        uint32_t w[kOrderedMaxSteps][2], byte[kOrderedMaxSteps][2];
#pragma unroll
        for (uint32_t st = 0; st < kOrderedMaxSteps; ++st) {
            const uint32_t col = c_begin + st * kQuantColsPerWarpStep + lane * 16;
#pragma unroll
            for (uint32_t r = 0; r < 2; ++r) {
                const uint32_t row = row0 + r;
                if (prequant) {
                    o[st][r] = in[st][r][0];
                    byte[st][r] = 0;
                    if (col < c_end && row < p.M && (lane & 1u) == 0u) {
                        byte[st][r] = p.in_scales[(size_t)row * sf_cols + col / 32];
                    }
                } else {
                    o[st][r] = quant16(in[st][r][0], in[st][r][1], device_tiny, e5m2, byte[st][r]);
                }
                const uint32_t base = lane & ~7u;
                w[st][r] = __shfl_sync(0xFFFFFFFFu, byte[st][r], base) | (__shfl_sync(0xFFFFFFFFu, byte[st][r], base + 2) << 8) |
                           (__shfl_sync(0xFFFFFFFFu, byte[st][r], base + 4) << 16) |
                           (__shfl_sync(0xFFFFFFFFu, byte[st][r], base + 6) << 24);
            }
        }
        if (item + gridDim.x < items) {
            load_item(item + gridDim.x);  // travels while this item is stored, fenced and flagged
        }
        auto store_to = [&](uint32_t d) {
#pragma unroll
            for (uint32_t st = 0; st < kOrderedMaxSteps; ++st) {
                const uint32_t col = c_begin + st * kQuantColsPerWarpStep + lane * 16;
#pragma unroll
                for (uint32_t r = 0; r < 2; ++r) {
                    const uint32_t row = row0 + r;
                    if (col < c_end && row < p.M) {
                        *reinterpret_cast<uint4*>(p.dst_codes[d] + (size_t)row * p.K + col) = o[st][r];
                        const size_t sf_off = (size_t)row * sf_cols + col / 32;
                        if (sf_vec) {
                            if ((lane & 7u) == 0u) {
                                *reinterpret_cast<uint32_t*>(p.dst_scales[d] + sf_off) = w[st][r];
                            }
                        } else if ((lane & 1u) == 0u) {
                            p.dst_scales[d][sf_off] = (uint8_t)byte[st][r];
                        }
                    }
                }
            }
        };
        // this rank's own stage first: its rows are the first the GEMM beside this kernel works on
        if (p.rank < p.num_dst && p.dst_codes[p.rank] != nullptr) {
            store_to(p.rank);
            __syncthreads();
            if (tid == 0 && p.dst_flags[p.rank] != nullptr) {
                __threadfence();
                asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p.dst_flags[p.rank] + flag_index), "r"(p.epoch)
                             : "memory");
            }
        }
        // then the peers, starting behind this rank so that the ranks of a box do not all store to the same GPU
        bool any_peer = false;
        for (uint32_t t = 1; t < p.num_dst; ++t) {
            const uint32_t d = (p.rank + t) % p.num_dst;
            if (p.dst_codes[d] != nullptr) {
                store_to(d);
                any_peer = true;
            }
        }
        if (any_peer) {
            __syncthreads();
            if (tid == 0) {
                __threadfence_system();
                for (uint32_t t = 1; t < p.num_dst; ++t) {
                    const uint32_t d = (p.rank + t) % p.num_dst;
                    if (p.dst_flags[d] != nullptr) {
                        asm volatile("st.relaxed.sys.global.u32 [%0], %1;" ::"l"(p.dst_flags[d] + flag_index), "r"(p.epoch)
                                     : "memory");
                    }
                }
            }
        }
    }
#ifdef CATCCOS_TRACE
    if (p.trace != nullptr) {
        __syncthreads();
        if (threadIdx.x == 0) {
            atomicMax(p.trace + kTrQuantKernelEnd, globaltimer_ns());
        }
    }
#endif
}

// Routing-side producer of a packed MoE dispatch: every token (a bf16 row of N values) is quantised once and the
// same packed row is written to each of its top_k destinations.  A packed row is
// [N E4M3 codes | ceil(N / 32) E8M0 scales, padded to an even count | zero padding to a multiple of 32 bytes];
// expanded_row_idx[token * top_k + route] names the destination row, a negative entry drops the route.
// It replaces CommBlockMxQuant::QuantScatterPacked (include/catccos/comm/block/comm_block_mx_quant.hpp:312-368).
__host__ __device__ __forceinline__ uint32_t packed_row_bytes(uint32_t n)
{
    const uint32_t scale_bytes = ((n + 31u) / 32u + 1u) / 2u * 2u;
    return (n + scale_bytes + 31u) / 32u * 32u;
}

// One warp per (token, 512-column step): a lane quantises 16 consecutive values (two lanes share a 32-block) and stores
// its 16 bytes of codes once per route; the warp of a token's last step also writes the padding.  Bound by the writes
// (top_k packed rows per token): every warp has all its loads, then all its stores in flight, and a token's steps run
// side by side instead of one after the other.
__global__ void __launch_bounds__(kQuantThreads) mx_quant_scatter_packed_kernel(const uint16_t* __restrict__ in,
                                                                               const int32_t* __restrict__ expanded_row_idx,
                                                                               uint8_t* __restrict__ packed_out, uint32_t tokens,
                                                                               uint32_t n, uint32_t top_k, uint32_t device_tiny)
{
    grid_dep_wait();
    grid_dep_launch();
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t steps = (n + kQuantColsPerWarpStep - 1) / kQuantColsPerWarpStep;
    const uint64_t w = (uint64_t)blockIdx.x * (kQuantThreads / 32) + (threadIdx.x >> 5);
    const uint32_t token = (uint32_t)(w / steps), step = (uint32_t)(w % steps);
    if (token >= tokens) {
        return;
    }
    const uint32_t row_bytes = packed_row_bytes(n);
    const uint32_t col = step * kQuantColsPerWarpStep + lane * 16;
    const bool ok = col < n;
    uint4 v0 = make_uint4(0, 0, 0, 0), v1 = v0;
    if (ok) {
        load_half_block(in + (size_t)token * n + col, v0, v1);
    }
    const int32_t* routes = expanded_row_idx + (size_t)token * top_k;
    const bool last = step == steps - 1;
    uint32_t byte = 0;
    uint4 o = v0;
    for (uint32_t r0 = 0; r0 < top_k; r0 += 32) {
        const int32_t mine = r0 + lane < top_k ? __ldg(routes + r0 + lane) : -1;
        if (r0 == 0) {
            o = quant16(v0, v1, device_tiny != 0u, false, byte);
        }
        const uint32_t here = min(32u, top_k - r0);
        for (uint32_t r = 0; r < here; ++r) {
            const int32_t dst = __shfl_sync(0xFFFFFFFFu, mine, r);
            if (dst < 0) {
                continue;
            }
            uint8_t* row = packed_out + (size_t)dst * row_bytes;
            if (ok) {
                *reinterpret_cast<uint4*>(row + col) = o;
                if ((lane & 1u) == 0u) {
                    row[n + col / 32u] = (uint8_t)byte;
                }
            }
            // the tail of the row: the scale count rounded up to even, then zeros up to the 32-byte boundary
            if (last && n + n / 32u + lane < row_bytes) {
                row[n + n / 32u + lane] = 0;
            }
        }
    }
}

// Transposed copy of a packed E2M1 weight: in [K, N/2] (two N-neighbours per byte, low nibble = even column, the
// reference's file layout, examples/utils/gen_data_fp4_mx_allgather_matmul.py:521-544) -> out [N, K/2] (two
// K-neighbours per byte).  The tensor core reads 4-bit operands K-major only.  A warp takes 64 (K) x 64 (N) values: lane
// (kw, ng) the eight K rows 8 kw .. and sixteen columns 16 ng .., so a load instruction reads whole 32-byte sectors of
// eight rows and a store instruction writes whole sectors of four; the 8 x 8 blocks of nibbles turn in registers.  Bound
// by memory (the weight in and out once); one value per byte through shared memory: a
// launch of [7168, 2304] 11.5 us, 6.8 us here (cold caches).
// Needs N % 64 == 0 and K % 64 == 0 (the GEMM asks for multiples of 128) and 8-byte aligned pointers.
__device__ __forceinline__ void transpose_nibbles_8x8(const uint32_t (&a)[8], uint32_t (&b)[8])
{
    uint32_t h[2][4];  // [n half][k]: four nibbles of row k, then of row k + 4
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) {
        h[0][k] = __byte_perm(a[k], a[k + 4], 0x5410);
        h[1][k] = __byte_perm(a[k], a[k + 4], 0x7632);
    }
#pragma unroll
    for (uint32_t i = 0; i < 2; ++i) {
#pragma unroll
        for (uint32_t j = 0; j < 2; ++j) {  // columns 4 i + 2 j and the next
            const uint32_t sel = j == 0u ? 0x6240 : 0x7351;
            const uint32_t even = __byte_perm(h[i][0], h[i][2], sel), odd = __byte_perm(h[i][1], h[i][3], sel);
            b[4 * i + 2 * j] = (even & 0x0F0F0F0Fu) | ((odd & 0x0F0F0F0Fu) << 4);
            b[4 * i + 2 * j + 1] = ((even >> 4) & 0x0F0F0F0Fu) | (odd & 0xF0F0F0F0u);
        }
    }
}

constexpr uint32_t kFp4TransTile = 64;
__global__ void __launch_bounds__(256) fp4_transpose_kernel(const uint8_t* __restrict__ in, uint8_t* __restrict__ out, uint32_t K,
                                                            uint32_t N)
{
    grid_dep_wait();
    grid_dep_launch();
    const uint32_t lane = threadIdx.x & 31, kw = lane & 7u, ng = lane >> 3;
    const uint32_t n_tiles = N / kFp4TransTile, tile = blockIdx.x * 8u + (threadIdx.x >> 5);
    if (tile >= n_tiles * (K / kFp4TransTile)) {
        return;
    }
    const uint32_t k0 = tile / n_tiles * kFp4TransTile + kw * 8u, n0 = tile % n_tiles * kFp4TransTile + ng * 16u;
    uint32_t lo[8], hi[8], t[8];
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        const uint2 v = __ldcs(reinterpret_cast<const uint2*>(in + (size_t)(k0 + i) * (N / 2) + n0 / 2));
        lo[i] = v.x;
        hi[i] = v.y;
    }
    uint8_t* dst = out + (size_t)n0 * (K / 2) + k0 / 2;
    transpose_nibbles_8x8(lo, t);
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        *reinterpret_cast<uint32_t*>(dst + (size_t)i * (K / 2)) = t[i];
    }
    transpose_nibbles_8x8(hi, t);
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) {
        *reinterpret_cast<uint32_t*>(dst + (size_t)(i + 8) * (K / 2)) = t[i];
    }
}

// bf16 [rows, K] -> FP4 E2M1 codes, two per byte (low nibble = even column), + one E8M0 scale per 32 elements.
// The FP4 branch of the reference's quantiser (include/catccos/comm/block/comm_block_mx_quant.hpp:525-568, emax
// constant block_epilogue_dynamic_mx_quant.hpp:53): the same exponent rule with emax 2, saturation at +-6,
// round to nearest even (cvt.rn.satfinite.e2m1x2.f32).  Flat, as mx_quant_flat_kernel: a lane quantises 16 consecutive
// values (two lanes share a 32-block) and stores 8 bytes of codes.  [1024, 7168]: 12.8 us with a warp walking each row.
__global__ void __launch_bounds__(kQuantThreads) mx_quant_e2m1_kernel(const uint8_t* __restrict__ in, uint64_t halves,
                                                                      uint8_t* __restrict__ packed,
                                                                      uint8_t* __restrict__ scales, uint32_t device_tiny)
{
    grid_dep_wait();
    grid_dep_launch();
    const uint64_t i = (uint64_t)blockIdx.x * kQuantThreads + threadIdx.x;
    uint4 v0 = make_uint4(0, 0, 0, 0), v1 = v0;
    if (i < halves) {
        load_half_block(in + i * 32, v0, v1);
    }
    uint32_t amax = max(absmax_bits8(v0), absmax_bits8(v1));
    amax = max(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, 1));
    uint32_t byte;
    float mul;
    bool nonfinite;
    block_scale(amax, device_tiny != 0u, 2u, byte, mul, nonfinite);
    const uint32_t w[8] = {v0.x, v0.y, v0.z, v0.w, v1.x, v1.y, v1.z, v1.w};
    uint32_t o[2] = {0u, 0u};
#pragma unroll
    for (uint32_t k = 0; k < 8; ++k) {
        const float lo = __uint_as_float(w[k] << 16) * mul, hi = __uint_as_float(w[k] & 0xFFFF0000u) * mul;
        const uint32_t b = __nv_cvt_float2_to_fp4x2(make_float2(lo, hi), __NV_E2M1, cudaRoundNearest);
        o[k >> 2] |= (b & 0xFFu) << (8u * (k & 3u));
    }
    if (nonfinite) {
        o[0] = o[1] = 0x77777777u;  // E2M1 has no NaN: the largest magnitude stands in
    } else if (mul == 0.0f && device_tiny == 0u) {
        o[0] = o[1] = 0u;  // the golden writes +0 for every element of a block below 1e-12
    }
    if (i < halves) {
        *reinterpret_cast<uint2*>(packed + i * 8) = make_uint2(o[0], o[1]);
        if ((i & 1u) == 0u) {
            scales[i >> 1] = (uint8_t)byte;
        }
    }
}

}  // namespace catccos
