// C ABI of libcatccos_b200.so (declarations and reference citations: include/catccos_b200.h).
// Host logic only: rank contexts, symmetric buffers (cuMem/VMM, peer mapped), epochs, launches.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include "../../include/catccos_b200.h"
#include "bootstrap.hpp"
#include "internal_options.h"
#include "common.cuh"
#include "mx_gemm.cuh"
#include "mx_gemm_pair.cuh"
#include "mx_gemm_small.cuh"
#include "mx_quant.cuh"

using namespace catccos;

static_assert(sizeof(catccos_b200_tiling_t) == 17 * sizeof(uint32_t), "must match CocTilingParams");

#define ERROR_LOG(fmt, ...) fprintf(stdout, "[ERROR] " fmt "\n", ##__VA_ARGS__)

// Same shape as the reference's ACL_CHECK (utils/utils.h:28-34): print and carry the code on.
#define CUDA_TRY(expr)                                                                              \
    do {                                                                                            \
        cudaError_t err__ = (expr);                                                                 \
        if (err__ != cudaSuccess) {                                                                 \
            fprintf(stderr, "%s:%d cudaError:%d (%s)\n", __FILE__, __LINE__, (int)err__,            \
                    cudaGetErrorString(err__));                                                     \
            return CATCCOS_B200_ECUDA;                                                              \
        }                                                                                           \
    } while (0)

#define CU_TRY(expr)                                                                                \
    do {                                                                                            \
        CUresult err__ = (expr);                                                                    \
        if (err__ != CUDA_SUCCESS) {                                                                \
            fprintf(stderr, "%s:%d cudaError:%d (driver)\n", __FILE__, __LINE__, (int)err__);       \
            return CATCCOS_B200_ECUDA;                                                              \
        }                                                                                           \
    } while (0)

namespace {

// ---------------------------------------------------------------------------------------------
// driver entry points (resolved at run time so that the library links against cudart only)
// ---------------------------------------------------------------------------------------------
struct Driver {
    decltype(&cuMemCreate) MemCreate = nullptr;
    decltype(&cuMemRelease) MemRelease = nullptr;
    decltype(&cuMemExportToShareableHandle) MemExport = nullptr;
    decltype(&cuMemImportFromShareableHandle) MemImport = nullptr;
    decltype(&cuMemAddressReserve) MemAddressReserve = nullptr;
    decltype(&cuMemAddressFree) MemAddressFree = nullptr;
    decltype(&cuMemMap) MemMap = nullptr;
    decltype(&cuMemUnmap) MemUnmap = nullptr;
    decltype(&cuMemSetAccess) MemSetAccess = nullptr;
    decltype(&cuMemGetAllocationGranularity) MemGetGranularity = nullptr;
    decltype(&cuTensorMapEncodeTiled) TensorMapEncodeTiled = nullptr;
    bool ok = false;

    template <typename F>
    bool Get(const char* name, F& fn)
    {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint(name, &p, cudaEnableDefault, &q) != cudaSuccess || p == nullptr) {
            ERROR_LOG("driver entry point %s not found", name);
            return false;
        }
        fn = reinterpret_cast<F>(p);
        return true;
    }

    bool Load()
    {
        if (ok) {
            return true;
        }
        ok = Get("cuMemCreate", MemCreate) && Get("cuMemRelease", MemRelease) &&
             Get("cuMemExportToShareableHandle", MemExport) && Get("cuMemImportFromShareableHandle", MemImport) &&
             Get("cuMemAddressReserve", MemAddressReserve) && Get("cuMemAddressFree", MemAddressFree) &&
             Get("cuMemMap", MemMap) && Get("cuMemUnmap", MemUnmap) && Get("cuMemSetAccess", MemSetAccess) &&
             Get("cuMemGetAllocationGranularity", MemGetGranularity) &&
             Get("cuTensorMapEncodeTiled", TensorMapEncodeTiled);
        return ok;
    }
};

// ---------------------------------------------------------------------------------------------
// state
// ---------------------------------------------------------------------------------------------
constexpr size_t kHeaderBytes = 1u << 20;       // counters + flag words at the start of a symmetric buffer
constexpr uint32_t kMaxFlags = 24576;           // flag words per source rank: (16-row chunks) x (K segments)
constexpr size_t kFlagsOff = 256u << 10;        // uint32 [kMaxRanks][kMaxFlags]; the first 256 KiB are reserved
static_assert(kFlagsOff + (size_t)kMaxRanks * kMaxFlags * 4 <= kHeaderBytes, "header layout");

constexpr size_t kSplitKTileBytes = 128u * 256u * 4u;  // one fp32 partial tile of the widest GEMM tile

struct RankCtx {
    int device = 0;
    int num_sms = 0;
    StatusBlock* status = nullptr;  // device memory
    uint8_t* fp4_bt = nullptr;  // the transposed copy of a packed E2M1 weight, made on every call that gets one
    size_t fp4_bt_bytes = 0;
    // split-K scratch of this rank's GEMM launches: one fp32 partial tile and four flag words per SM, then the 64-bit
    // word that counts the split launches (the flags are epochs, split_epoch).  Launches of one rank are stream-ordered.
    float* splitk_ws = nullptr;
    uint32_t* splitk_flags = nullptr;
    // copy-engine allgather: one stream per peer (the transfers to the peers run side by side), an event that
    // marks "this rank's shard is quantised" and one per stream that marks "everything for that peer has left"
    cudaStream_t side = nullptr;  // the quantise-and-push kernel runs here, beside the GEMM on the caller's stream
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    cudaStream_t copy[kMaxRanks] = {};
    cudaEvent_t ev_quant = nullptr;
    cudaEvent_t ev_copy[kMaxRanks] = {};
#ifdef CATCCOS_TRACE
    unsigned long long* trace = nullptr;  // [SMs][kTraceSlots] timeline words of the armed launch
    int trace_grid = 0;
#endif
};

struct SymmAlloc {
    size_t size = 0;                       // bytes per rank
    std::vector<uint8_t*> base;            // base[r]: address of rank r's copy, valid for the acting rank's device
    std::vector<uint32_t> epoch;           // per acting rank: collectives issued on this buffer
    std::vector<bool> released;          // local mode: which ranks have fetched their pointer
    // VMM bookkeeping (one process per rank)
    bool vmm = false;
    CUdeviceptr va = 0;
    size_t va_size = 0;
    std::vector<CUmemGenericAllocationHandle> handles;
};

enum class Mode { kNone, kProcess, kLocal };

struct State {
    std::mutex mu;
    Mode mode = Mode::kNone;
    int world = 1;
    int rank = 0;  // acting rank
    std::vector<RankCtx> ranks;
    std::vector<std::unique_ptr<SymmAlloc>> allocs;
    Bootstrap boot;
    Driver drv;
    // options
    // options a caller may set (include/catccos_b200.h)
    int tiny_block_rule = 0;
    int c_dtype = 0;
    // test and tuning hooks (internal_options.h)
    int block_n = 0;
    int phase_mask = 3;
    int cta_pair = 0;        // 0 = automatic, 1 = always CTA pairs (cta_group::2), 2 = never
    int fuse_mode = -1;      // -1 = automatic, 0 = quantise warps inside the GEMM kernel, 3 = (one rank only) quantise
                             // kernel, then GEMM kernel, 4 = quantise kernel, then GEMM-and-push kernel
    int a_dtype = 0;         // element type of the A codes (what the quantiser writes, what the GEMM reads): 0 = E4M3, 1 = E5M2
    int b_dtype = 0;         // element type of the B codes the caller passes
    int split_k = 0;         // 0 = automatic, 1 = never split K, 2..8 = split K in that many parts when it fits
    int b_lsu = 0;           // 0 = automatic, 1 = B through the load/store units, 2 = through TMA
    int small_tile = 0;      // 0 = automatic, 1 = always the small-tile kernel where it can run, 2 = never
    int small_quant = 0;     // 0 = automatic, 1 = the small-tile kernel quantises a fused call itself, 2 = never
    int tile_order = -1;     // gated GEMM: -1 = automatic, 1 = own shard first, 0 = slice by slice over all ranks
    uint64_t timeout_ns = 2000ull * 1000000ull;
#ifdef CATCCOS_TRACE
    bool trace_armed = false;  // the next GEMM launch of the acting rank writes its timeline
#endif
    std::vector<uint32_t> local_alloc_cursor;  // local mode: next allocation index per rank
};

State g;
std::atomic<uint64_t> g_launches{0};

int setup_rank_ctx(RankCtx& rc, int device)
{
    rc.device = device;
    CUDA_TRY(cudaSetDevice(device));
    CUDA_TRY(cudaFree(nullptr));
    CUDA_TRY(cudaDeviceGetAttribute(&rc.num_sms, cudaDevAttrMultiProcessorCount, device));
    CUDA_TRY(cudaMalloc(&rc.status, sizeof(StatusBlock)));
    CUDA_TRY(cudaMemset(rc.status, 0, sizeof(StatusBlock)));
    CUDA_TRY(cudaMalloc(&rc.fp4_bt, 1u << 20));
    rc.fp4_bt_bytes = 1u << 20;
    CUDA_TRY(cudaMalloc(&rc.splitk_ws, (size_t)rc.num_sms * kSplitKTileBytes));
    CUDA_TRY(cudaMalloc(&rc.splitk_flags, ((size_t)rc.num_sms * 4 + 2) * sizeof(uint32_t)));
    CUDA_TRY(cudaMemset(rc.splitk_flags, 0, ((size_t)rc.num_sms * 4 + 2) * sizeof(uint32_t)));
    {
        int lo = 0, hi = 0;
        CUDA_TRY(cudaDeviceGetStreamPriorityRange(&lo, &hi));
        CUDA_TRY(cudaStreamCreateWithPriority(&rc.side, cudaStreamNonBlocking, hi));
    }
    CUDA_TRY(cudaEventCreateWithFlags(&rc.ev_fork, cudaEventDisableTiming));
    CUDA_TRY(cudaEventCreateWithFlags(&rc.ev_join, cudaEventDisableTiming));
    CUDA_TRY(cudaEventCreateWithFlags(&rc.ev_quant, cudaEventDisableTiming));
    for (int t = 0; t < kMaxRanks; ++t) {
        CUDA_TRY(cudaStreamCreateWithFlags(&rc.copy[t], cudaStreamNonBlocking));
        CUDA_TRY(cudaEventCreateWithFlags(&rc.ev_copy[t], cudaEventDisableTiming));
    }
#ifdef CATCCOS_TRACE
    CUDA_TRY(cudaMalloc(&rc.trace, (size_t)rc.num_sms * kTraceSlots * sizeof(unsigned long long)));
    CUDA_TRY(cudaMemset(rc.trace, 0, (size_t)rc.num_sms * kTraceSlots * sizeof(unsigned long long)));
#endif
    return 0;
}

void destroy_rank_ctx(RankCtx& rc)
{
    cudaSetDevice(rc.device);
    if (rc.status) cudaFree(rc.status);
    if (rc.fp4_bt) cudaFree(rc.fp4_bt);
    if (rc.splitk_ws) cudaFree(rc.splitk_ws);
    if (rc.splitk_flags) cudaFree(rc.splitk_flags);
    if (rc.side) cudaStreamDestroy(rc.side);
    if (rc.ev_fork) cudaEventDestroy(rc.ev_fork);
    if (rc.ev_join) cudaEventDestroy(rc.ev_join);
    if (rc.ev_quant) cudaEventDestroy(rc.ev_quant);
    for (int t = 0; t < kMaxRanks; ++t) {
        if (rc.copy[t]) cudaStreamDestroy(rc.copy[t]);
        if (rc.ev_copy[t]) cudaEventDestroy(rc.ev_copy[t]);
    }
#ifdef CATCCOS_TRACE
    if (rc.trace) cudaFree(rc.trace);
#endif
    rc = RankCtx();
}

// A world of one needs no set-up call: the first operator call adopts the current device.
int ensure_init()
{
    if (g.mode != Mode::kNone) {
        return 0;
    }
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    g.world = 1;
    g.rank = 0;
    g.ranks.resize(1);
    int rc = setup_rank_ctx(g.ranks[0], dev);
    if (rc != 0) {
        return rc;
    }
    g.mode = Mode::kProcess;
    return 0;
}

RankCtx& cur() { return g.ranks[g.mode == Mode::kLocal ? g.rank : 0]; }

SymmAlloc* find_symm(const void* p)
{
    for (auto& a : g.allocs) {
        if (a && a->base[g.rank] == p) {
            return a.get();
        }
    }
    return nullptr;
}

// The symmetric allocation that holds [p, p + bytes) on the acting rank, and p's offset inside it.
SymmAlloc* find_symm_containing(const void* p, size_t bytes, size_t* offset)
{
    const uint8_t* q = static_cast<const uint8_t*>(p);
    for (auto& a : g.allocs) {
        if (a && a->base[g.rank] != nullptr && q >= a->base[g.rank] && q + bytes <= a->base[g.rank] + a->size) {
            *offset = (size_t)(q - a->base[g.rank]);
            return a.get();
        }
    }
    return nullptr;
}

size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

struct StageLayout {
    size_t stage_bytes, codes_off, scales_off;
};

// Two stages after the header; a stage holds the gathered codes [W*M, K] then the scales [W*M, K/32].
bool stage_layout(size_t symm_bytes, uint32_t W, uint32_t M, uint32_t K, StageLayout& L)
{
    if (symm_bytes < kHeaderBytes + 2048) {
        return false;
    }
    L.stage_bytes = ((symm_bytes - kHeaderBytes) / 2) & ~(size_t)1023;
    L.codes_off = 0;
    L.scales_off = align_up((size_t)W * M * K, 1024);
    size_t need = L.scales_off + align_up((size_t)W * M * (K / 32), 1024);
    return need <= L.stage_bytes;
}

// ---------------------------------------------------------------------------------------------
// launches
// ---------------------------------------------------------------------------------------------
// Every kernel of this library that waits for its predecessor with grid_dep_wait() before it touches memory is
// launched with programmatic stream serialisation: its launch latency and set-up pass while the predecessor drains.
// Measured (B200, back to back on one stream, a 3 us kernel): 6.2 us per launch without the attribute (a plain
// dependency is picked up in steps of 2.05 us), 3.6 us with it.
template <typename... KArgs, typename... Args>
cudaError_t launch_after(void (*kern)(KArgs...), dim3 grid, uint32_t threads, size_t smem, cudaStream_t st, Args&&... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    g_launches++;
    return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

int quant_grid(const RankCtx& rc)
{
    int per_sm = 0;
    const void* fn = (const void*)mx_quant_push_kernel<false>;
    // An SM keeps one shared-memory carve-out for all resident CTAs.  The GEMM needs the largest one;
    // asking for the same carve-out here lets quantise CTAs and a GEMM CTA share an SM when the two run
    // as separate kernels.
    static bool carveout_set[kMaxRanks * 2] = {};
    if (rc.device < kMaxRanks * 2 && !carveout_set[rc.device]) {
        cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
        cudaGetLastError();
        carveout_set[rc.device] = true;
    }
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, kQuantThreads, 0) != cudaSuccess || per_sm < 1) {
        per_sm = 1;
    }
    if (per_sm > 6) {
        per_sm = 6;
    }
    return per_sm * rc.num_sms;
}

// The ordered quantise-and-push kernel (several ranks, GEMM beside it): per_sm CTAs per SM.
int launch_quant_push_ordered(RankCtx& rc, cudaStream_t st, QuantPushParams& p, bool prequant, int per_sm);

uint32_t quant_mode(bool prequant)
{
    return prequant ? kQuantPreQuantised : (g.tiny_block_rule != 0 ? kQuantDeviceTiny : kQuantGolden);
}

uint32_t quant_sys_scope(uint32_t world) { return world > 1 ? 1u : 0u; }

constexpr uint32_t kQuantItemsPerSm = 4;  // work items per SM the quantiser's K-segment choice aims for

// max_cols (0 = none): an upper bound on the columns of a K segment.
void choose_segments(uint32_t M, uint32_t K, int num_sms, QuantPushParams& p, uint32_t max_cols = 0)
{
    const uint32_t chunks = (M + kQuantRowsPerItem - 1) / kQuantRowsPerItem;
    const uint32_t max_segs = (K + kQuantColsPerWarpStep - 1) / kQuantColsPerWarpStep;
    uint32_t want = ((uint32_t)num_sms * kQuantItemsPerSm + chunks - 1) / chunks;
    if (want < 1) want = 1;
    if (want > max_segs) want = max_segs;
    uint32_t seg_cols = (uint32_t)align_up((K + want - 1) / want, kQuantColsPerWarpStep);
    if (max_cols != 0 && seg_cols > max_cols) {
        seg_cols = max_cols;
    }
    p.seg_cols = seg_cols;
    p.segs_per_chunk = (K + seg_cols - 1) / seg_cols;
}

// bf16 [M, K] -> codes and scales in one place, nobody waiting on flags: the flat quantiser.
// `reset` (or nullptr): the wait records of the allocation-free entry point, cleared for this call.
int launch_quant_flat(cudaStream_t st, const void* in, uint32_t M, uint32_t K, uint8_t* codes, uint8_t* scales,
                      StatusBlock* reset = nullptr)
{
    const uint64_t halves = (uint64_t)M * (K / 16);
    const dim3 grid((unsigned)((halves + kQuantThreads - 1) / kQuantThreads));
    CUDA_TRY(launch_after(g.a_dtype == 1 ? mx_quant_flat_kernel<true> : mx_quant_flat_kernel<false>, grid, kQuantThreads, 0, st,
                          static_cast<const uint8_t*>(in), codes, scales, halves, g.tiny_block_rule != 0 ? 1u : 0u, reset));
    return 0;
}

// max_grid (0 = no limit): an upper bound on the CTAs, for a push that has to leave in item order.
int launch_quant_push(RankCtx& rc, cudaStream_t st, QuantPushParams& p, bool prequant, bool produce,
                      bool local_only = false, int max_grid = 0)
{
    int grid = quant_grid(rc);
    if (max_grid > 0 && grid > max_grid) grid = max_grid;
    const uint32_t chunks = (p.M + kQuantRowsPerItem - 1) / kQuantRowsPerItem;
    uint32_t items = produce ? chunks * p.segs_per_chunk : 0;
    if (p.consume) {
        uint32_t peer_items = (p.world - 1) * chunks;
        if (peer_items > items) items = peer_items;
    }
    if (items == 0) {
        return 0;
    }
    if ((uint32_t)grid > items) grid = (int)items;
    p.produce = produce ? 1u : 0u;
    p.mode = quant_mode(prequant);
    p.e5m2 = g.a_dtype == 1 ? 1u : 0u;
    p.sys_scope = local_only ? quant_sys_scope(1) : quant_sys_scope(p.world);  // no peer sees these stores directly
    const bool prefetch = grid <= 2 * rc.num_sms && items > (uint32_t)grid;
    CUDA_TRY(launch_after(prefetch ? mx_quant_push_kernel<true> : mx_quant_push_kernel<false>, dim3(grid), kQuantThreads, 0, st, p));
    return 0;
}

int launch_quant_push_ordered(RankCtx& rc, cudaStream_t st, QuantPushParams& p, bool prequant, int per_sm)
{
    const uint32_t chunks = (p.M + kQuantRowsPerItem - 1) / kQuantRowsPerItem;
    const uint32_t items = chunks * p.segs_per_chunk;
    if (items == 0 || p.seg_cols > kOrderedMaxSteps * kQuantColsPerWarpStep) {
        return CATCCOS_B200_EINVAL;
    }
    static bool carveout_set[kMaxRanks * 2] = {};
    if (rc.device < kMaxRanks * 2 && !carveout_set[rc.device]) {
        // the GEMM's CTA, which needs the largest shared-memory carve-out, shares the SM with these CTAs
        cudaFuncSetAttribute((const void*)mx_quant_push_ordered_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                             cudaSharedmemCarveoutMaxShared);
        cudaGetLastError();
        carveout_set[rc.device] = true;
    }
    uint32_t grid = (uint32_t)(per_sm * rc.num_sms);
    if (grid > items) grid = items;
    p.produce = 1u;
    p.consume = 0u;
    p.mode = quant_mode(prequant);
    p.e5m2 = g.a_dtype == 1 ? 1u : 0u;
    p.sys_scope = 1u;
    mx_quant_push_ordered_kernel<<<grid, kQuantThreads, 0, st>>>(p);
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// Tensor maps depend on (address, extents, box) only; a decode loop calls with the same few buffers over and
// over, and an encode costs about as much as the launch it precedes.  A small most-recently-used table keeps the
// last maps (calls of one process are serialised by its callers: one host thread per rank).
struct MapKey {
    const void* base;
    uint64_t inner, outer;
    uint32_t box_inner, box_outer;
    bool fp4;
    uint32_t elem;
    bool operator==(const MapKey& o) const
    {
        return base == o.base && inner == o.inner && outer == o.outer && box_inner == o.box_inner &&
               box_outer == o.box_outer && fp4 == o.fp4 && elem == o.elem;
    }
};
constexpr int kMapCacheSize = 16;
struct MapCache {
    MapKey key[kMapCacheSize] = {};
    CUtensorMap map[kMapCacheSize];
    uint64_t used[kMapCacheSize] = {};
    uint64_t clock = 0;
} g_maps;

int encode_map_2d_uncached(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
                           uint32_t box_outer, bool fp4, uint32_t elem);

// inner / outer / box in elements of `elem` bytes; fp4: two E2M1 values per byte in global memory
int encode_map_2d(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
                  uint32_t box_outer, bool fp4 = false, uint32_t elem = 1)
{
    const MapKey k{base, inner, outer, box_inner, box_outer, fp4, elem};
    int victim = 0;
    for (int i = 0; i < kMapCacheSize; ++i) {
        if (g_maps.used[i] != 0 && g_maps.key[i] == k) {
            g_maps.used[i] = ++g_maps.clock;
            *map = g_maps.map[i];
            return 0;
        }
        if (g_maps.used[i] < g_maps.used[victim]) {
            victim = i;
        }
    }
    int rc = encode_map_2d_uncached(map, base, inner, outer, box_inner, box_outer, fp4, elem);
    if (rc == 0) {
        g_maps.key[victim] = k;
        g_maps.map[victim] = *map;
        g_maps.used[victim] = ++g_maps.clock;
    }
    return rc;
}

int encode_map_2d_uncached(CUtensorMap* map, const void* base, uint64_t inner, uint64_t outer, uint32_t box_inner,
                           uint32_t box_outer, bool fp4, uint32_t elem)
{
    cuuint64_t dims[2] = {inner, outer};
    cuuint64_t strides[1] = {fp4 ? inner / 2 : inner * elem};  // bytes; 4-bit elements are packed in pairs
    cuuint32_t box[2] = {box_inner, box_outer};
    cuuint32_t estr[2] = {1, 1};
    // packed 4-bit values land in shared memory sixteen to a 16-byte chunk (8 bytes of values, 8 bytes of gap):
    // the same 128 bytes per 128 values as the 8-bit types, so boxes, swizzle and descriptors stay as they are
    const CUtensorMapDataType dt = fp4 ? CU_TENSOR_MAP_DATA_TYPE_16U4_ALIGN16B
                                       : (elem == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8);
    CU_TRY(g.drv.TensorMapEncodeTiled(map, dt, 2, const_cast<void*>(base), dims, strides, box,
                                      estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                      !fp4 && box_inner * elem == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
    return 0;
}

template <uint32_t BLOCK_N, typename OutT, bool FUSED>
int launch_gemm_inst(int grid, cudaStream_t st, const CUtensorMap& ta, const CUtensorMap& tb, const GemmParams& p,
                     bool overlap_predecessor)
{
    auto kern = mx_gemm_kernel<BLOCK_N, OutT, FUSED>;
    static bool attr_done[kMaxRanks * 2] = {};
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < kMaxRanks * 2 && !attr_done[dev]) {
        CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)GemmSmem<BLOCK_N>::kDynamicBytes));
        attr_done[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(FUSED ? kGemmFusedThreads : kGemmThreads + (p.b_lsu ? kBLoadWarps * 32 : 0));
    cfg.dynamicSmemBytes = GemmSmem<BLOCK_N>::kDynamicBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    // Without flags the kernel waits for its predecessor itself; with flags it does not, and only the quantise kernel
    // that feeds it may still be running.
    cfg.numAttrs = (overlap_predecessor || (!FUSED && p.flags == nullptr)) ? 1 : 0;
    CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, ta, tb, p));
    g_launches++;
    CUDA_TRY(cudaGetLastError());
    return 0;
}

// CTA pairs that can be resident at once.  A launch never has more: CTAs of one launch wait on flags that other CTAs of
// the same launch publish.
template <typename OutT, bool FUSED>
int resident_pairs(uint32_t max_pairs, uint32_t* pairs)
{
    auto kern = mx_gemm_pair_kernel<OutT, FUSED>;
    static bool attr_done[kMaxRanks * 2] = {};
    static int max_clusters[kMaxRanks * 2] = {};
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= kMaxRanks * 2 || !attr_done[dev]) {
        CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PairSmem::kDynamicBytes));
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2 * max_pairs);
        cfg.blockDim = dim3(FUSED ? kGemmFusedThreads : kGemmThreads);
        cfg.dynamicSmemBytes = PairSmem::kDynamicBytes;
        cudaLaunchAttribute attr;
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 2;
        attr.val.clusterDim.y = 1;
        attr.val.clusterDim.z = 1;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess || n < 1) {
            cudaGetLastError();
            n = (int)max_pairs;
        }
        if (dev >= kMaxRanks * 2) {
            *pairs = std::min((uint32_t)n, max_pairs);
            return 0;
        }
        max_clusters[dev] = n;
        attr_done[dev] = true;
    }
    *pairs = std::min((uint32_t)max_clusters[dev], max_pairs);
    return 0;
}

template <typename OutT, bool FUSED>
int launch_gemm_pair_inst(uint32_t max_pairs, uint32_t tiles, uint32_t parts, cudaStream_t st, const CUtensorMap& ta,
                          const CUtensorMap& tb, const CUtensorMap& tc, GemmParams& p, bool overlap_predecessor)
{
    uint32_t pairs = 0;
    int rc = resident_pairs<OutT, FUSED>(max_pairs, &pairs);
    if (rc != 0) return rc;
    const PairGrid grid = pair_grid(tiles, pairs, parts);
    p.ksplit = grid.ksplit;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * grid.pairs);
    cfg.blockDim = dim3(FUSED ? kGemmFusedThreads : kGemmThreads);
    cfg.dynamicSmemBytes = PairSmem::kDynamicBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr;  // the cluster shape is the kernel's own (__cluster_dims__)
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    // Without flags the kernel waits for its predecessor itself; with flags it does not, and only the quantise kernel
    // that feeds it may still be running.
    cfg.numAttrs = (overlap_predecessor || (!FUSED && p.flags == nullptr)) ? 1 : 0;
    CUDA_TRY(cudaLaunchKernelEx(&cfg, mx_gemm_pair_kernel<OutT, FUSED>, ta, tb, tc, p));
    g_launches++;
    return 0;
}

// What the tilings cost, in microseconds (kernel alone, back to back): a launch, each K tile of a round, and what splitting
// K adds (partial tiles written, flagged, read, added; more where more of them cross).  Used only to pick one.  The
// constants are fitted to 390 sizes x up to 17 variants measured on B200 (64 <= M <= 4096, N and K to 8192): estimates are
// off by 6 %.  In 150 sizes left out of the fit the tiling they choose is 0.4 % from the fastest (mean; 8 % at worst).
// Larger M (to 32768) is not in the fit: such launches are many rounds of pairs whatever the constants say.
constexpr double kBasePair = 5.42, kBaseSingle256 = 4.05, kBaseSingle128 = 3.4, kBaseSingle64 = 3.13;
constexpr double kOutput = 0.223e-6;  // per output element
// with few SMs busy; the loads of a full GPU take kBusy more (pairs 0.30 to 0.36 us, 128 columns 0.30 to 0.34)
constexpr double kPeriodPair = 0.291, kPeriodSingle256 = 0.378, kPeriodSingle128 = 0.276, kPeriodSingle64 = 0.255, kBusy = 0.2;
constexpr double kRagged = 1.11;  // N no multiple of 32: every other K row of B starts inside a sector
constexpr double kSplitCostPair = 3.16, kSplitCostPairPerCta = 0.0216;
// single CTAs: the bytes that cross go with the tile's width, and each part adds a piece to wait for
constexpr double kSplitCost = 1.75, kSplitCostPerCta256 = 0.0314, kSplitCostPerPart = 0.353;
// pairs with whole tiles to follow, beside which the exchange passes (but the partial tiles' traffic does not)
constexpr double kSplitFirstCost = 2.32, kSplitFirstCostPerCta = 0.019;

struct GemmPlan {
    bool use_pair;
    uint32_t block_n, ksplit;  // ksplit: CTA pairs: most parts of a last-round tile; single CTAs: parts of every tile
    double time;               // what the launch is expected to take, microseconds
};

// Tiling of one GEMM launch: CTA pairs or single CTAs, tile width, and the number of K parts.
// whole_tiles: K stays in one piece; wide: only the tile widths every variant of the kernel has (128 and more).
GemmPlan plan_gemm(const RankCtx& rc, uint32_t Mg, uint32_t N, uint32_t K, bool whole_tiles = false, bool wide = false)
{
    const uint32_t m128 = (Mg + 127) / 128, m256 = (Mg + 255) / 256;
    const uint32_t n256 = (N + 255) / 256;
    const uint32_t sms = (uint32_t)rc.num_sms, max_pairs = sms / 2;
    const uint32_t k_tiles = K / kGemmBlockK;
    // Splitting needs the scratch (the allocation-free entry point has none).
    const bool may_split = rc.splitk_ws != nullptr && g.split_k != 1 && !whole_tiles;
    const uint32_t cap = may_split ? (g.split_k >= 2 ? (uint32_t)g.split_k : kSplitKMax) : 1u;
    const bool forced_split = g.split_k >= 2;
    const double ragged = N % 32u != 0u ? kRagged : 1.0;
    auto busy = [&](uint32_t ctas) { return ragged * (1.0 + kBusy * std::min(1.0, (double)ctas / sms)); };

    // CTA pairs: whole rounds, and a last round whose tiles are cut in as many parts as shorten it
    const uint32_t tiles = m256 * n256, rem = tiles % max_pairs;
    uint32_t pair_parts = 1;
    double last = rem != 0 ? k_tiles * kPeriodPair * busy(2 * tiles) : 0.0;
    for (uint32_t s = 2; rem != 0 && s <= std::min(std::min(cap, max_pairs / rem), k_tiles); ++s) {
        const uint32_t ctas = 2 * rem * s;
        const double cost = tiles >= max_pairs ? kSplitFirstCost + kSplitFirstCostPerCta * ctas
                                               : kSplitCostPair + kSplitCostPairPerCta * ctas;
        const double t = ((k_tiles + s - 1) / s) * kPeriodPair * busy(tiles >= max_pairs ? sms : ctas) + cost;
        if (t < last) {
            last = t;
            pair_parts = s;
        }
    }
    const double t_pair = kBasePair + (tiles / max_pairs) * k_tiles * kPeriodPair * busy(sms) + last;

    // single CTAs: rounds of whole tiles, or, when the tiles leave at least half of the SMs idle, every (tile, K part) on
    // its own CTA (a power of two that divides the K tiles, at least four K tiles per part, one part per 32 columns)
    auto single = [&](uint32_t bn, uint32_t* parts) {
        const uint32_t t1 = m128 * ((N + bn - 1) / bn);
        const double base = bn == 256 ? kBaseSingle256 : (bn == 128 ? kBaseSingle128 : kBaseSingle64);
        const double period = bn == 256 ? kPeriodSingle256 : (bn == 128 ? kPeriodSingle128 : kPeriodSingle64);
        double best = base + (double)((t1 + sms - 1) / sms) * k_tiles * period * busy(t1);
        *parts = 1;
        for (uint32_t s = 2; s <= std::min(std::min(cap, sms / t1), bn / 32u); s *= 2) {
            if (k_tiles % s != 0 || k_tiles / s < 4) {
                continue;
            }
            const double t = base + k_tiles / s * period * busy(t1 * s) + kSplitCost + kSplitCostPerCta256 * t1 * s * bn / 256 +
                             kSplitCostPerPart * s;
            if (t < best || forced_split) {
                best = t;
                *parts = s;
            }
        }
        return best;
    };
    const uint32_t widths[3] = {256, 128, 64};
    const uint32_t asked = wide && g.block_n == 64 ? 0u : (uint32_t)g.block_n;
    uint32_t bn = 0, parts = 1;
    double t_single = 0.0;
    for (uint32_t w : widths) {
        if (asked != 0 ? w != asked : ((w == 64 && wide) || (w == 256 && N <= 128))) {
            continue;
        }
        uint32_t s = 1;
        const double t = single(w, &s);
        if (bn == 0 || t < t_single) {
            bn = w;
            parts = s;
            t_single = t;
        }
    }

    GemmPlan plan;
    plan.use_pair = g.cta_pair == 1 || (g.cta_pair == 0 && g.block_n == 0 && t_pair < t_single);
    plan.block_n = plan.use_pair ? kPairBlockN : bn;
    plan.ksplit = plan.use_pair ? pair_parts : parts;
    plan.time = (plan.use_pair ? t_pair : t_single) + kOutput * Mg * N;
    return plan;
}

// The small-tile kernel (mx_gemm_small.cuh) for a call: activation rows of a tile, K parts, and whether it quantises.
struct SmallPlan {
    bool use, quant;
    uint32_t mt, parts;
};

// What it costs, in microseconds, as a launch of one K tile; each further K tile of a CTA while loads are latency-bound
// (with the quantisation inside, four warps' work); or, if that is longer, streaming every tile's weights (rows of N
// bytes that are no multiple of 128 straddle two lines each); and the exchange of the parts.  A quantiser in front costs
// a launch and a dependency.  The constants are fitted to 54 sizes x 4 to 8 variants measured on B200 (1 <= M <= 256,
// 1024 <= N <= 7168, 1024 <= K <= 7168; above 16 rows with tiles of 32 only, so tiles of 16 are not considered there):
// estimates are off by 8 %, and the variant they choose by 0.7 % from the fastest.
constexpr double kSmallBase = 2.9, kSmallPeriod16 = 0.23, kSmallPeriod32 = 0.24, kSmallQuant16 = 0.37, kSmallQuant32 = 0.79;
constexpr double kSmallQuantShared = 1.45;  // two CTAs on an SM
constexpr double kSmallBytesPerUs = 7.4e6, kSmallBytesPerUsRagged = 5.1e6, kSmallHidden = 0.73;
constexpr double kSmallExchange16 = 0.6, kSmallExchange32 = 1.5, kSmallExchange32PerRow = 0.03;
constexpr double kSmallShortK = 0.5;  // 32-row tiles, up to four K tiles: 64 sizes read 0.2 to 0.4 above the estimate, others 0.2 below
constexpr double kSmallMxOutPerRow = 0.08;  // a warp takes the block maximum of one row at a time
constexpr double kQuantiserSmall = 1.6, kQuantiserLarge = 1.8;

// Clusters of `parts` CTAs that are resident at once, two CTAs on an SM (148, 71 and 33 of 2, 4 and 8 on 148 SMs).
uint32_t small_clusters(uint32_t sms, uint32_t parts)
{
    return parts == 1 ? 2 * sms : (parts == 2 ? sms : (parts == 4 ? sms * 71 / 148 : sms * 33 / 148));
}

SmallPlan plan_small(const RankCtx& rc, uint32_t M, uint32_t N, uint32_t K, bool bf16_in, bool mx_out = false)
{
    SmallPlan s = {};
    if (g.small_tile == 2 || g.cta_pair != 0 || g.block_n != 0) {
        return s;  // another tiling is asked for
    }
#ifdef CATCCOS_TRACE
    if (g.trace_armed && rc.trace != nullptr) {
        return s;  // this kernel keeps no timeline: the call is recorded on the general ones
    }
#endif
    s.mt = M <= 16 ? 16 : 32;
    const uint32_t tiles = ((M + s.mt - 1) / s.mt) * ((N + kSmallBlockN - 1) / kSmallBlockN), k_tiles = K / kGemmBlockK;
    const uint32_t cap = std::min(g.split_k >= 1 ? (uint32_t)g.split_k : kSmallMaxParts, k_tiles);
    const uint32_t sms = (uint32_t)rc.num_sms;
    const double stream = (double)tiles * k_tiles * (kSmallBlockN * kGemmBlockK) /
                          (N % 128u == 0u ? kSmallBytesPerUs : kSmallBytesPerUsRagged);
    double best = 0.0;
    for (uint32_t quant = 0; quant <= (bf16_in ? 1u : 0u); ++quant) {
        if (bf16_in && g.small_quant != 0 && (quant != 0) != (g.small_quant == 1)) {
            continue;
        }
        for (uint32_t parts = 1; parts <= cap; parts *= 2) {
            const uint32_t resident = small_clusters(sms, parts);
            if (parts > 1 && tiles > resident && g.split_k <= 1) {
                break;  // clusters that wait for a place pay their start again
            }
            const double rounds = (double)((tiles + resident - 1) / resident);
            double period = s.mt == 16 ? kSmallPeriod16 : kSmallPeriod32;
            if (quant) {
                period = (s.mt == 16 ? kSmallQuant16 : kSmallQuant32) * (tiles * parts > sms ? kSmallQuantShared : 1.0);
            }
            const double loop = ((k_tiles + parts - 1) / parts) * period * rounds;
            double t = rounds * kSmallBase + std::max(loop, stream) + (1.0 - kSmallHidden) * std::min(loop, stream);
            if (parts > 1) {
                t += s.mt == 16 ? kSmallExchange16 : kSmallExchange32 + kSmallExchange32PerRow * (s.mt / parts);
            }
            t += bf16_in && !quant ? kQuantiserSmall : 0.0;
            t += mx_out ? kSmallMxOutPerRow * (s.mt / parts) : 0.0;
            if (s.parts == 0 || t < best || (g.split_k > 1 && parts * 2 > cap && quant == (uint32_t)s.quant)) {
                best = t;
                s.parts = parts;
                s.quant = quant != 0;
            }
        }
    }
    best += s.mt == 32 && k_tiles <= 4 ? kSmallShortK : 0.0;
    s.use = g.small_tile == 1 || best < plan_gemm(rc, M, N, K).time + (bf16_in ? kQuantiserLarge : 0.0);
    return s;
}

template <uint32_t MT, typename OutT, bool QUANT>
int launch_small_inst(cudaStream_t st, const CUtensorMap& tw, const CUtensorMap& tx, const SmallParams& p)
{
    auto kern = mx_gemm_small_kernel<MT, OutT, QUANT>;
    static bool attr_done[kMaxRanks * 2] = {};
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev >= kMaxRanks * 2 || !attr_done[dev]) {
        CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SmallSmem<MT>::kDynamicBytes));
        CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
        if (dev < kMaxRanks * 2) attr_done[dev] = true;
    }
    const uint32_t tiles = ((p.M + MT - 1) / MT) * ((p.N + kSmallBlockN - 1) / kSmallBlockN);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(tiles * p.parts);
    cfg.blockDim = dim3(kGemmThreads);
    cfg.dynamicSmemBytes = SmallSmem<MT>::kDynamicBytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = p.parts;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    g_launches++;
    CUDA_TRY(cudaLaunchKernelEx(&cfg, kern, tw, tx, p));
    return 0;
}

// p: x or x_scales, w_scales, c, c_scales, M, N, K, w_early, w_kmajor, records filled in.
int launch_small(RankCtx& rc, cudaStream_t st, const SmallPlan& plan, const void* x_codes, const void* w, SmallParams p,
                 bool mx_out)
{
    if (!g.drv.Load()) {
        return CATCCOS_B200_ECUDA;
    }
    p.parts = plan.parts;
    p.status = rc.status;
    p.bar_timeout_ns = 2 * g.timeout_ns + 1000000000ull;
    p.x_fmt = g.a_dtype == 2 ? 5u : (g.a_dtype == 1 ? 1u : 0u);
    p.w_fmt = g.b_dtype == 2 ? 5u : (g.b_dtype == 1 ? 1u : 0u);
    p.device_tiny = g.tiny_block_rule != 0 ? 1u : 0u;
    CUtensorMap tw, tx;
    int rcode = p.w_kmajor ? encode_map_2d(&tw, w, p.K, p.N, kGemmBlockK, kSmallBlockN, g.b_dtype == 2)
                           : encode_map_2d(&tw, w, p.N, p.K, kSmallBlockN, kGemmBlockK);
    if (rcode != 0) return rcode;
    tx = tw;  // not read by a quantising launch
    if (!plan.quant) {
        rcode = encode_map_2d(&tx, x_codes, p.K, p.M, kGemmBlockK, plan.mt, g.a_dtype == 2);
        if (rcode != 0) return rcode;
    }
    const bool f16 = g.c_dtype == 1;
#define CATCCOS_SMALL_CASE(MT)                                                                   \
    if (plan.mt == MT) {                                                                         \
        if (mx_out) {                                                                            \
            return launch_small_inst<MT, MxOut, false>(st, tw, tx, p);                           \
        }                                                                                        \
        if (plan.quant) {                                                                        \
            return f16 ? launch_small_inst<MT, __half, true>(st, tw, tx, p)                      \
                       : launch_small_inst<MT, __nv_bfloat16, true>(st, tw, tx, p);              \
        }                                                                                        \
        return f16 ? launch_small_inst<MT, __half, false>(st, tw, tx, p)                         \
                   : launch_small_inst<MT, __nv_bfloat16, false>(st, tw, tx, p);                 \
    }
    CATCCOS_SMALL_CASE(16)
    CATCCOS_SMALL_CASE(32)
#undef CATCCOS_SMALL_CASE
    return CATCCOS_B200_EINVAL;
}

// overlap_predecessor: the kernel launched just before on `st` is this library's quantise kernel, whose output
// the GEMM reads only behind grid_dep_wait(); the GEMM may then be scheduled while that kernel drains.
// epilogue: what the epilogue warps do with a finished tile (never combined with the quantise warps inside)
enum Epilogue { kEpiStore = 0,    // round to bf16 / fp16 and store C
                kEpiMxQuant = 1,  // MX-quantise the output (p.c = codes, p.c_scales)
                kEpiScatter = 2 };  // Matmul + ReduceScatter: fp32 partial rows to the stage of the rank that owns them

int launch_gemm(RankCtx& rc, cudaStream_t st, const void* a, const void* b, GemmParams& p, bool fused_quant = false,
                bool overlap_predecessor = false, Epilogue epilogue = kEpiStore)
{
    const bool mx_out = epilogue == kEpiMxQuant, scatter = epilogue == kEpiScatter;
    if (!g.drv.Load()) {
        return CATCCOS_B200_ECUDA;
    }
    if (p.Mg == 0 || p.N == 0 || p.K == 0 || p.K % kGemmBlockK != 0 || p.N % 16 != 0) {
        ERROR_LOG("mx gemm needs K %% 128 == 0 and N %% 16 == 0 (got M=%u N=%u K=%u)", p.Mg, p.N, p.K);
        return CATCCOS_B200_EINVAL;
    }
    if ((((uintptr_t)a | (uintptr_t)b) & 15u) || (!scatter && ((uintptr_t)p.c & 31u)) || ((uintptr_t)p.a_scales & 3u) ||
        ((uintptr_t)p.b_scales & 1u)) {
        ERROR_LOG("mx gemm operands must be 16-byte aligned (the output 32-byte aligned)");
        return CATCCOS_B200_EINVAL;
    }
    const bool f16 = g.c_dtype == 1;
    p.status = rc.status;
    p.timeout_ns = g.timeout_ns;
    // a barrier inside the kernel may have to wait for as long as the flag wait it depends on
    p.bar_timeout_ns = 2 * g.timeout_ns + 1000000000ull;
    p.a_fmt = g.a_dtype == 2 ? 5u : (g.a_dtype == 1 ? 1u : 0u);
    p.b_fmt = g.b_dtype == 2 ? 5u : (g.b_dtype == 1 ? 1u : 0u);
    const bool a_fp4 = g.a_dtype == 2, b_fp4 = g.b_dtype == 2;
    if ((a_fp4 && (((uintptr_t)a & 31u) || p.K % 128 != 0)) || (b_fp4 && (((uintptr_t)b & 31u) || p.N % 128 != 0))) {
        ERROR_LOG("mx gemm: packed E2M1 operands must be 32-byte aligned, with K a multiple of 128 (and N, for B)");
        return CATCCOS_B200_EINVAL;
    }
    if (b_fp4) {
        // the tensor core takes 4-bit operands K-major only: transpose the weight [K, N/2] -> [N, K/2] into this
        // rank's scratch (grown on first use; a few microseconds for a weight of some megabytes)
        const size_t need = (size_t)p.N * (p.K / 2);
        if (rc.fp4_bt == nullptr) {
            return CATCCOS_B200_ESTATE;  // the allocation-free entry point has no scratch for it
        }
        if (need > rc.fp4_bt_bytes) {
            CUDA_TRY(cudaStreamSynchronize(st));
            CUDA_TRY(cudaFree(rc.fp4_bt));
            CUDA_TRY(cudaMalloc(&rc.fp4_bt, need));
            rc.fp4_bt_bytes = need;
        }
        const dim3 tg(((p.N / kFp4TransTile) * (p.K / kFp4TransTile) + 7) / 8);  // a warp per tile
        CUDA_TRY(launch_after(fp4_transpose_kernel, tg, 256, 0, st, static_cast<const uint8_t*>(b), rc.fp4_bt, p.K, p.N));
        b = rc.fp4_bt;
        p.b_kmajor = 1;
        p.b_early = 0;  // the copy is the kernel launched just before
        overlap_predecessor = false;
    }
    if (p.flags == nullptr && !fused_quant && !scatter) {
        const SmallPlan small = plan_small(rc, p.Mg, p.N, p.K, false, mx_out);
        if (small.use) {
            SmallParams sp = {};
            sp.x_scales = p.a_scales;
            sp.w_scales = p.b_scales;
            sp.c = p.c;
            sp.c_scales = p.c_scales;
            sp.M = p.Mg;
            sp.N = p.N;
            sp.K = p.K;
            sp.w_kmajor = p.b_kmajor;
            sp.w_early = p.b_early;
            return launch_small(rc, st, small, a, b, sp, mx_out);
        }
    }
#ifdef CATCCOS_TRACE
    if (g.trace_armed && rc.trace != nullptr) {
        g.trace_armed = false;
        p.trace = p.q.trace = p.push.trace = rc.trace;
    }
#endif
    const GemmPlan plan = plan_gemm(rc, p.Mg, p.N, p.K, scatter, scatter || fused_quant || p.flags != nullptr);  // scatter: the owner adds whole tiles, K stays in one piece
    const bool use_pair = plan.use_pair;
    const uint32_t bn = plan.block_n, ksplit = plan.ksplit;
    const uint32_t m256 = (p.Mg + 255) / 256;
    const uint32_t max_pairs = (uint32_t)rc.num_sms / 2;
    if (ksplit > 1) {
        p.splitk_ws = rc.splitk_ws;
        p.splitk_flags = rc.splitk_flags;
        p.splitk_state = reinterpret_cast<unsigned long long*>(rc.splitk_flags + (size_t)rc.num_sms * 4);
    }
    if (use_pair) {
        CUtensorMap pa, pb, pc;
        int rc2 = encode_map_2d(&pa, a, p.K, p.Mg, kGemmBlockK, 128, a_fp4);
        if (rc2 != 0) return rc2;
        rc2 = b_fp4 ? encode_map_2d(&pb, b, p.K, p.N, kGemmBlockK, 128, true)
                    : encode_map_2d(&pb, b, p.N, p.K, 128, kGemmBlockK, false);
        if (rc2 != 0) return rc2;
        if (scatter) {
            pc = pa;  // the epilogue stores to several ranks without a map
        } else {
            rc2 = mx_out ? encode_map_2d(&pc, p.c, p.N, p.Mg, 128, 32) : encode_map_2d(&pc, p.c, p.N, p.Mg, 64, 32, false, 2);
            if (rc2 != 0) return rc2;
        }
        const uint32_t tiles = m256 * ((p.N + kPairBlockN - 1) / kPairBlockN);
#ifdef CATCCOS_TRACE
        rc.trace_grid = (int)(2 * pair_grid(tiles, max_pairs, ksplit).pairs);
#endif
#define CATCCOS_PAIR(OUT, FUSED) \
    launch_gemm_pair_inst<OUT, FUSED>(max_pairs, tiles, ksplit, st, pa, pb, pc, p, overlap_predecessor)
        if (mx_out) {
            return CATCCOS_PAIR(MxOut, false);
        }
        if (scatter) {
            return CATCCOS_PAIR(ScatterOut, false);
        }
        if (fused_quant) {
            return f16 ? CATCCOS_PAIR(__half, true) : CATCCOS_PAIR(__nv_bfloat16, true);
        }
        return f16 ? CATCCOS_PAIR(__half, false) : CATCCOS_PAIR(__nv_bfloat16, false);
#undef CATCCOS_PAIR
    }
    CUtensorMap ta, tb;
    int rcode = encode_map_2d(&ta, a, p.K, p.Mg, kGemmBlockK, kGemmBlockM, a_fp4);
    if (rcode != 0) return rcode;
    rcode = b_fp4 ? encode_map_2d(&tb, b, p.K, p.N, kGemmBlockK, bn, true)
                  : encode_map_2d(&tb, b, p.N, p.K, std::min(bn, 128u), kGemmBlockK, false);
    if (rcode != 0) return rcode;
    const uint32_t tiles = ((p.Mg + kGemmBlockM - 1) / kGemmBlockM) * ((p.N + bn - 1) / bn);
    int grid = (int)(tiles < (uint32_t)rc.num_sms ? tiles : (uint32_t)rc.num_sms);
    p.ksplit = ksplit;
    p.b = static_cast<const uint8_t*>(b);
    p.b_lsu = bn == 64 && !b_fp4 && (g.b_lsu == 0 ? p.N % 32u != 0u : g.b_lsu == 1) ? 1u : 0u;
    if (ksplit > 1) {
        grid = (int)(tiles * ksplit);  // <= SMs by construction: all units are resident at once
    }
#ifdef CATCCOS_TRACE
    rc.trace_grid = grid;
#endif
#define CATCCOS_GEMM_CASE(BN)                                                                         \
    if (bn == BN) {                                                                                   \
        if (mx_out) {                                                                                 \
            return launch_gemm_inst<BN, MxOut, false>(grid, st, ta, tb, p, overlap_predecessor);      \
        }                                                                                             \
        if (scatter) {                                                                                \
            return launch_gemm_inst<BN, ScatterOut, false>(grid, st, ta, tb, p, overlap_predecessor); \
        }                                                                                             \
        if (fused_quant) {                                                                            \
            return f16 ? launch_gemm_inst<BN, __half, true>(grid, st, ta, tb, p, overlap_predecessor)         \
                       : launch_gemm_inst<BN, __nv_bfloat16, true>(grid, st, ta, tb, p, overlap_predecessor); \
        }                                                                                             \
        return f16 ? launch_gemm_inst<BN, __half, false>(grid, st, ta, tb, p, overlap_predecessor)           \
                   : launch_gemm_inst<BN, __nv_bfloat16, false>(grid, st, ta, tb, p, overlap_predecessor);   \
    }
    CATCCOS_GEMM_CASE(256)
    CATCCOS_GEMM_CASE(128)
#undef CATCCOS_GEMM_CASE
    if (bn == 64) {
        if (mx_out) {
            return launch_gemm_inst<64, MxOut, false>(grid, st, ta, tb, p, overlap_predecessor);
        }
        return f16 ? launch_gemm_inst<64, __half, false>(grid, st, ta, tb, p, overlap_predecessor)
                   : launch_gemm_inst<64, __nv_bfloat16, false>(grid, st, ta, tb, p, overlap_predecessor);
    }
    return CATCCOS_B200_EINVAL;
}

// Sets n flag words to the epoch (the rows they stand for were put in place by stream-ordered copies).
__global__ void fill_flags_kernel(uint32_t* flags, uint32_t n, uint32_t epoch)
{
    grid_dep_wait();
    grid_dep_launch();
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        flags[i] = epoch;
    }
}

// Ends once every listed flag word carries the epoch (bounded): what follows on the stream may read the rows the
// peers' copy engines wrote.  One thread per word.
__global__ void wait_flags_kernel(const uint32_t* flags, uint32_t flag_stride, uint32_t world, uint32_t rank, uint32_t chunks,
                                  uint32_t segs, uint32_t epoch, uint64_t timeout_ns, StatusBlock* status)
{
    grid_dep_wait();
    grid_dep_launch();
    for (uint32_t i = threadIdx.x; i + 1 < world; i += blockDim.x) {
        const uint32_t src = (rank + 1 + i) % world;
        const uint32_t last_chunk = chunks - 1u;
        // the last word a peer's stream writes: everything before it on that stream has landed
        const uint32_t* f = flags + (size_t)src * flag_stride + (size_t)last_chunk * segs + (segs - 1u);
        if (!wait_flag_ge(f, epoch, timeout_ns, status)) {
            report_status(status, kStatusFlagTimeout, src, last_chunk, epoch);
        }
    }
}

constexpr uint32_t kCopySliceRows = 256;  // rows the copy engines move (and flag) at a time: one row of GEMM tiles

// AllGather of this rank's quantised shard by the copy engines.  Behind the quantise kernel on `st` (an event),
// one stream per peer copies the shard into that peer's stage: all scales first (they are small), then slice by
// slice the codes followed by the slice's flag words, which the quantise kernel has set to the epoch in this
// rank's own flag array.  Copies of one stream run in order, so a peer sees a slice's flags only after the
// slice's data; the streams of the peers run side by side and share the NVLink egress, which hides the few
// microseconds every copy costs to start.  No SM takes part: the GEMM that runs meanwhile keeps its load/store
// units to itself, and the slices arrive in the order the GEMM visits them.
int copy_engine_push(RankCtx& rc, cudaStream_t st, uint32_t W, uint32_t rank, uint32_t M, uint32_t K, uint32_t segs,
                     uint32_t slice_rows, const uint8_t* src_codes, const uint8_t* src_scales, const uint32_t* src_flags,
                     uint8_t* const* dst_codes, uint8_t* const* dst_scales, uint32_t* const* dst_flags,
                     size_t code_row_bytes = 0)
{
    const uint32_t sf = K / 32;
    const size_t row_bytes = code_row_bytes != 0 ? code_row_bytes : K;  // a row of codes: K bytes, K / 2 for packed E2M1
    CUDA_TRY(cudaEventRecord(rc.ev_quant, st));
    for (uint32_t t = 0; t + 1 < W; ++t) {
        const uint32_t d = (rank + 1 + t) % W;
        cudaStream_t cs = rc.copy[t];
        CUDA_TRY(cudaStreamWaitEvent(cs, rc.ev_quant, 0));
        CUDA_TRY(cudaMemcpyAsync(dst_scales[d], src_scales, (size_t)M * sf, cudaMemcpyDeviceToDevice, cs));
        for (uint32_t r0 = 0; r0 < M; r0 += slice_rows) {
            const uint32_t rows = std::min(slice_rows, M - r0);
            const uint32_t c0 = r0 / kRowsPerChunk, chunks = (rows + kRowsPerChunk - 1) / kRowsPerChunk;
            CUDA_TRY(cudaMemcpyAsync(dst_codes[d] + (size_t)r0 * row_bytes, src_codes + (size_t)r0 * row_bytes,
                                     (size_t)rows * row_bytes, cudaMemcpyDeviceToDevice, cs));
            CUDA_TRY(cudaMemcpyAsync(dst_flags[d] + (size_t)c0 * segs, src_flags + (size_t)c0 * segs,
                                     (size_t)chunks * segs * sizeof(uint32_t), cudaMemcpyDeviceToDevice, cs));
        }
        CUDA_TRY(cudaEventRecord(rc.ev_copy[t], cs));
    }
    return 0;
}

// The caller's stream does not run past the call before this rank's shard has left: the next call but one
// writes the same stage, and the flag words the copies read are rewritten by the very next call.
int copy_engine_join(RankCtx& rc, cudaStream_t st, uint32_t W)
{
    for (uint32_t t = 0; t + 1 < W; ++t) {
        CUDA_TRY(cudaStreamWaitEvent(st, rc.ev_copy[t], 0));
    }
    return 0;
}

// Alignment that the quantisers' and TMA's 16-byte accesses, the output's whole sectors and the 16-bit reads of the weight
// scales need.  Checked at the entry: the quantiser, which runs first, checks nothing.
bool matmul_operands_ok(const char* op, const void* a, const void* b, const void* b_scale, const void* c)
{
    if ((((uintptr_t)a | (uintptr_t)b) & 15u) || ((uintptr_t)c & 31u) || ((uintptr_t)b_scale & 1u)) {
        ERROR_LOG("%s: a and b must be 16-byte aligned, c 32-byte aligned, b_scale 2-byte aligned", op);
        return false;
    }
    return true;
}

bool share_memory(const void* p, size_t p_bytes, const void* q, size_t q_bytes)
{
    return (uintptr_t)p < (uintptr_t)q + q_bytes && (uintptr_t)q < (uintptr_t)p + p_bytes;
}

// Common part of the two AllGather-Matmul entry points.
int allgather_matmul(void* stream, const void* a, const void* a_scale, bool prequant, const void* b,
                     const void* b_scale, void* c, void* symm, const catccos_b200_tiling_t* t)
{
    if (!t || !a || !b || !b_scale || !c || (prequant && !a_scale)) {
        return CATCCOS_B200_EINVAL;
    }
    const uint32_t M = t->m, K = t->k, N = t->n, W = t->rankSize;
    if (M == 0 || K == 0 || N == 0 || K % kGemmBlockK != 0 || N % 16 != 0) {
        ERROR_LOG("allgather matmul: M=%u K=%u N=%u unsupported (K a multiple of 128, N of 16)", M, K, N);
        return CATCCOS_B200_EINVAL;
    }
    if (!matmul_operands_ok("allgather matmul", a, b, b_scale, c)) {
        return CATCCOS_B200_EINVAL;
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    if (W != (uint32_t)g.world) {
        ERROR_LOG("allgather matmul: rankSize %u (world %d)", W, g.world);
        return CATCCOS_B200_EINVAL;
    }
    SymmAlloc* sa = find_symm(symm);
    if (sa == nullptr) {
        ERROR_LOG("allgather matmul: symm must come from catccos_b200_symm_alloc");
        return CATCCOS_B200_ENOTSYMM;
    }
    RankCtx& rc = cur();
    StageLayout L;
    const uint32_t chunks = (M + kRowsPerChunk - 1) / kRowsPerChunk;
    QuantPushParams seg = {};
    // the same split on every rank and in both kernels; with several ranks a work item is at most 2048 columns wide
    // (what the ordered quantise-and-push kernel keeps in registers)
    choose_segments(M, K, rc.num_sms, seg, W > 1 ? kOrderedMaxSteps * kQuantColsPerWarpStep : 0u);
    if (!stage_layout(sa->size, W, M, K, L) || (size_t)chunks * seg.segs_per_chunk > kMaxFlags) {
        ERROR_LOG("allgather matmul: symmetric buffer of %zu bytes too small", sa->size);
        return CATCCOS_B200_ENOMEM;
    }
    CUDA_TRY(cudaSetDevice(rc.device));
    cudaStream_t st = (cudaStream_t)stream;
    const bool produce = (g.phase_mask & 1) != 0, consume = (g.phase_mask & 2) != 0;
    if (produce) {
        sa->epoch[g.rank] += 1;
    }
    const uint32_t epoch = sa->epoch[g.rank];
    const size_t stage_off = kHeaderBytes + (size_t)(epoch & 1u) * L.stage_bytes;
    const uint32_t rank = (uint32_t)g.rank;

    QuantPushParams q = {};
    q.in = a;
    q.in_scales = (const uint8_t*)a_scale;
    q.M = M;
    q.K = K;
    q.rank = rank;
    q.world = W;
    q.epoch = epoch;
    q.num_dst = W;
    q.publish = 1;
    q.segs_per_chunk = seg.segs_per_chunk;
    q.seg_cols = seg.seg_cols;
    {
        // A GEMM with more tiles than SMs runs in waves: send complete 256-row groups one after another so
        // that the first wave's rows are whole early.  A single-wave GEMM starts every tile at once and is
        // better served by one group (segment-major over all rows).
        const uint32_t tiles = ((W * M + 127) / 128) * ((N + 255) / 256);
        q.group_chunks = tiles > (uint32_t)rc.num_sms ? 256u / kRowsPerChunk : 0u;
    }
    {
        // a split-K GEMM on this rank wants the first K segment of each of its K parts first, then the second
        // of each, ... (every rank takes the same decision)
        const GemmPlan plan = plan_gemm(rc, W * M, N, K, false, true);
        const uint32_t segs = seg.segs_per_chunk;
        if (plan.ksplit > 1 && segs <= 32 && segs > 1) {
            const uint32_t kper = K / kGemmBlockK / plan.ksplit, seg_ktiles = seg.seg_cols / kGemmBlockK;
            uint32_t start[9];
            for (uint32_t a = 0; a < plan.ksplit; ++a) {
                start[a] = a * kper / seg_ktiles;
            }
            start[plan.ksplit] = segs;
            uint32_t n = 0;
            for (uint32_t round = 0; n < segs && round < segs; ++round) {
                for (uint32_t a = 0; a < plan.ksplit; ++a) {
                    const uint32_t sg = start[a] + round;
                    if (sg < start[a + 1]) {
                        q.seg_order[n++] = (uint8_t)sg;
                    }
                }
            }
            q.seg_order_n = n == segs ? n : 0u;
        }
    }
    for (uint32_t d = 0; d < W; ++d) {
        uint8_t* base = sa->base[d] + stage_off;
        q.dst_codes[d] = base + L.codes_off + (size_t)rank * M * K;
        q.dst_scales[d] = base + L.scales_off + (size_t)rank * M * (K / 32);
        q.dst_flags[d] = reinterpret_cast<uint32_t*>(sa->base[d] + kFlagsOff) + (size_t)rank * kMaxFlags;
    }
    q.status = rc.status;
    q.timeout_ns = g.timeout_ns;

    GemmParams p = {};
    {
        uint8_t* base = sa->base[rank] + stage_off;
        p.a_scales = base + L.scales_off;
        p.b_scales = (const uint8_t*)b_scale;
        p.c = c;
        p.Mg = W * M;
        p.N = N;
        p.K = K;
        p.flags = reinterpret_cast<const uint32_t*>(sa->base[rank] + kFlagsOff);
        p.flag_stride = kMaxFlags;
        p.segs = seg.segs_per_chunk;
        p.seg_ktiles = seg.seg_cols / kGemmBlockK;
        p.world = W;
        p.rank = rank;
        p.m_local = M;
        p.epoch = epoch;
    }
    const uint8_t* a_stage = sa->base[rank] + stage_off + L.codes_off;

    // With one rank there is no transfer to hide: the quantise kernel uses every SM for a few microseconds and
    // the GEMM follows it on the same stream, which measures faster than sharing the SMs between the two.
    // Several ranks: the quantise kernel stores every item to all ranks and the flag-gated GEMM follows on the
    // same stream (mode 6).  Measured at 2 and 4 ranks it is the fastest arrangement for the prefill shape and,
    // by a third, for the decode shape (one short dependency chain: quantise, store, fence, flag).
    const int auto_mode = 6;
    const int fuse_mode = W == 1 ? ((g.fuse_mode == 5 || g.fuse_mode < 0) ? 3 : g.fuse_mode)
                                 : (g.fuse_mode == 3 ? 0 : (g.fuse_mode >= 0 ? g.fuse_mode : auto_mode));
    // Tile order of the gated GEMM.  Where this rank's shard is in its own stage long before the peers' rows
    // (quantise kernel first, warps or copy engines forward it), the own shard's tiles go first.  Where the
    // quantiser stores an item to every rank before it takes the next, the own rows appear at the pace of the
    // transfer like everybody's: the tiles then follow the send groups, slice by slice over all ranks.
    p.own_first = g.tile_order >= 0 ? (uint32_t)g.tile_order : ((fuse_mode == 6 || fuse_mode == 7) ? 0u : 1u);
    if (produce && consume && fuse_mode == 3) {
        // C may lie in A's memory (a caller's buffer used twice): A is then quantised or copied into the stage first.  A kernel
        // that still reads A where it is while others of its CTAs store C needs the two apart.
        const bool apart = !share_memory(c, (size_t)M * N * 2, a, (size_t)M * K * (prequant ? 1 : 2)) &&
                           !(prequant && share_memory(c, (size_t)M * N * 2, a_scale, (size_t)M * (K / 32)));
        if (prequant && apart && ((uintptr_t)a_scale & 3u) == 0u) {
            // nothing to quantise and nobody to send to: the GEMM reads the caller's operands in place (scales that are not
            // aligned for its word loads go through the stage)
            p.a_scales = (const uint8_t*)a_scale;
            p.flags = nullptr;
            return launch_gemm(rc, st, a, b, p);
        }
        const SmallPlan small = plan_small(rc, M, N, K, !prequant);
        if (!prequant && apart && small.use && small.quant && g.b_dtype != 2) {
            SmallParams sp = {};
            sp.x = a;
            sp.w_scales = (const uint8_t*)b_scale;
            sp.c = c;
            sp.M = M;
            sp.N = N;
            sp.K = K;
            return launch_small(rc, st, small, nullptr, b, sp, false);
        }
        if (prequant) {
            q.publish = 0;
            rcode = launch_quant_push(rc, st, q, prequant, true);
        } else {
            rcode = launch_quant_flat(st, a, M, K, q.dst_codes[0], q.dst_scales[0]);
        }
        if (rcode != 0) return rcode;
        p.flags = nullptr;  // stream order is the only dependency
        // The quantiser waits for its own predecessor before it lets this launch go, so the weights are in place.
        p.b_early = prequant ? 0u : 1u;
        return launch_gemm(rc, st, a_stage, b, p, false, true);
    }
    if (fuse_mode == 6) {
        // Two kernels on the caller's stream.  The quantise kernel stores every work item to all ranks (one pass:
        // quantise and allgather) and flags it; the flag-gated GEMM kernel follows (with programmatic stream
        // serialisation: it may set itself up while the quantise kernel drains).  The quantise grid shrinks with
        // the number of ranks so that about the same number of bytes is on its way at any time.
        if (produce) {
            const int cap = std::max(rc.num_sms, (4 * rc.num_sms) / (int)std::max(1u, W - 1u) / rc.num_sms * rc.num_sms);
            rcode = launch_quant_push(rc, st, q, prequant, true, false, cap);
            if (rcode != 0) return rcode;
        }
        if (consume) {
            return launch_gemm(rc, st, a_stage, b, p, false, produce);
        }
        return 0;
    }
    if (fuse_mode == 7) {
        // Two kernels side by side.  The ordered quantise-and-push kernel (mx_quant.cuh), on a side stream of high
        // priority, one CTA per SM, never waits for anybody; the GEMM kernel, launched after it on the caller's
        // stream, takes one CTA per SM beside it and follows the flags, its own rows included.
        if (produce && consume) {
            CUDA_TRY(cudaEventRecord(rc.ev_fork, st));
            CUDA_TRY(cudaStreamWaitEvent(rc.side, rc.ev_fork, 0));
        }
        if (produce) {
#ifdef CATCCOS_TRACE
            if (g.trace_armed && rc.trace != nullptr) {
                q.trace = rc.trace;
            }
#endif
            rcode = launch_quant_push_ordered(rc, consume ? rc.side : st, q, prequant, 1);
            if (rcode != 0) return rcode;
            if (consume) {
                CUDA_TRY(cudaEventRecord(rc.ev_join, rc.side));
            }
        }
        if (consume) {
            rcode = launch_gemm(rc, st, a_stage, b, p);
            if (rcode != 0) return rcode;
            if (produce) {
                CUDA_TRY(cudaStreamWaitEvent(st, rc.ev_join, 0));
            }
        }
        return 0;
    }
    if (fuse_mode == 5) {
        if (produce) {
            QuantPushParams ql = q;  // the quantise kernel writes this rank's stage and its own flag words only
            for (uint32_t d = 0; d < W; ++d) {
                if (d != rank) {
                    ql.dst_codes[d] = nullptr;
                    ql.dst_scales[d] = nullptr;
                    ql.dst_flags[d] = nullptr;
                }
            }
            rcode = launch_quant_push(rc, st, ql, prequant, true, true);
            if (rcode != 0) return rcode;
            rcode = copy_engine_push(rc, st, W, rank, M, K, seg.segs_per_chunk, kCopySliceRows, q.dst_codes[rank],
                                     q.dst_scales[rank], q.dst_flags[rank], q.dst_codes, q.dst_scales, q.dst_flags);
            if (rcode != 0) return rcode;
        }
        if (consume) {
            rcode = launch_gemm(rc, st, a_stage, b, p);  // gated on the flags, own rows included
            if (rcode != 0) return rcode;
        }
        return produce ? copy_engine_join(rc, st, W) : 0;
    }
    if (produce) {
        // one GEMM launch: quantise warps fill the local stage, pusher warps forward it to the peers, the GEMM
        // warps of all ranks consume behind them.  The producer half alone (the harness that hosts several ranks
        // on one GPU runs every rank's producer before any consumer) is the same launch with the GEMM warps idle.
        p.gemm_off = consume ? 0u : 1u;
        p.q = q;
        p.q.produce = 1;
        p.q.mode = quant_mode(prequant);
        p.q.e5m2 = g.a_dtype == 1 ? 1u : 0u;
        p.q.sys_scope = 0;
        const bool quant_first = fuse_mode == 4;
        PushParams& ps = p.push;
        ps.src_codes = q.dst_codes[rank];
        ps.src_scales = q.dst_scales[rank];
        ps.src_flags = q.dst_flags[rank];
        for (uint32_t d = 0; d < W; ++d) {
            ps.dst_codes[d] = d == rank ? nullptr : q.dst_codes[d];
            ps.dst_scales[d] = d == rank ? nullptr : q.dst_scales[d];
            ps.dst_flags[d] = d == rank ? nullptr : q.dst_flags[d];
            if (d != rank) {
                p.q.dst_codes[d] = nullptr;  // the quantise warps write the local stage only
                p.q.dst_scales[d] = nullptr;
                p.q.dst_flags[d] = nullptr;
            }
        }
        ps.M = M;
        ps.K = K;
        ps.rank = rank;
        ps.world = W;
        ps.epoch = epoch;
        ps.segs_per_chunk = seg.segs_per_chunk;
        ps.seg_cols = seg.seg_cols;
        ps.group_chunks = q.group_chunks;
        ps.seg_order_n = q.seg_order_n;
        memcpy(ps.seg_order, q.seg_order, sizeof(ps.seg_order));
        ps.timeout_ns = g.timeout_ns;
        ps.status = rc.status;
        if (quant_first) {
            // the quantiser runs first, alone on every SM (48 resident warps per SM instead of the eight inside
            // the GEMM kernel) and fills the local stage (p.q names no peer any more); the GEMM-and-push kernel
            // follows on the same stream and may be scheduled while the quantiser drains
            QuantPushParams ql = p.q;
            rcode = launch_quant_push(rc, st, ql, prequant, true, true);
            if (rcode != 0) return rcode;
            p.q.produce = 0;
        }
        return launch_gemm(rc, st, a_stage, b, p, true, quant_first);
    }
    if (consume) {  // the consumer half alone: the flag-gated GEMM
        return launch_gemm(rc, st, a_stage, b, p);
    }
    return 0;
}

}  // namespace

// =============================================================================================
// C ABI
// =============================================================================================
extern "C" {

int catccos_b200_init(int rank, int world, int device, const char* ip_port)
{
    std::lock_guard<std::mutex> lock(g.mu);
    if (g.mode != Mode::kNone) {
        ERROR_LOG("catccos_b200_init: already initialised");
        return CATCCOS_B200_ESTATE;
    }
    if (world < 1 || world > kMaxRanks || rank < 0 || rank >= world) {
        ERROR_LOG("catccos_b200_init: rank %d of %d unsupported (at most %d ranks)", rank, world, kMaxRanks);
        return CATCCOS_B200_EINVAL;
    }
    g.world = world;
    g.rank = rank;
    g.ranks.resize(1);
    int rc = setup_rank_ctx(g.ranks[0], device);
    if (rc != 0) return rc;
    if (world > 1) {
        if (!g.drv.Load()) return CATCCOS_B200_ECUDA;
        if (!g.boot.Init(rank, world, ip_port)) {
            ERROR_LOG("catccos_b200_init: rendezvous failed: %s", g.boot.error().c_str());
            return CATCCOS_B200_ENET;
        }
    }
    g.mode = Mode::kProcess;
    return 0;
}

int catccos_b200_init_local(int world, const int* devices)
{
    std::lock_guard<std::mutex> lock(g.mu);
    if (g.mode != Mode::kNone) {
        ERROR_LOG("catccos_b200_init_local: already initialised");
        return CATCCOS_B200_ESTATE;
    }
    if (world < 1 || world > kMaxRanks || devices == nullptr) {
        return CATCCOS_B200_EINVAL;
    }
    g.world = world;
    g.rank = 0;
    g.ranks.resize(world);
    g.local_alloc_cursor.assign(world, 0);
    for (int r = 0; r < world; ++r) {
        int rc = setup_rank_ctx(g.ranks[r], devices[r]);
        if (rc != 0) return rc;
    }
    // ranks on different GPUs reach one another's memory through peer access
    for (int r = 0; r < world; ++r) {
        for (int s = 0; s < world; ++s) {
            if (devices[r] != devices[s]) {
                cudaSetDevice(devices[r]);
                cudaError_t e = cudaDeviceEnablePeerAccess(devices[s], 0);
                if (e != cudaSuccess && e != cudaErrorPeerAccessAlreadyEnabled) {
                    fprintf(stderr, "%s:%d cudaError:%d (peer access %d->%d)\n", __FILE__, __LINE__, (int)e, devices[r],
                            devices[s]);
                    return CATCCOS_B200_ECUDA;
                }
                cudaGetLastError();
            }
        }
    }
    g.mode = Mode::kLocal;
    return 0;
}

int catccos_b200_set_rank(int rank)
{
    if (g.mode != Mode::kLocal || rank < 0 || rank >= g.world) {
        return CATCCOS_B200_ESTATE;
    }
    g.rank = rank;
    CUDA_TRY(cudaSetDevice(g.ranks[rank].device));
    return 0;
}

int catccos_b200_finalize(void)
{
    std::lock_guard<std::mutex> lock(g.mu);
    if (g.mode == Mode::kNone) {
        return 0;
    }
    for (auto& rc : g.ranks) {
        cudaSetDevice(rc.device);
        cudaDeviceSynchronize();
    }
    for (auto& a : g.allocs) {
        if (!a) continue;
        if (a->vmm) {
            g.drv.MemUnmap(a->va, a->va_size);
            for (auto h : a->handles) g.drv.MemRelease(h);
            g.drv.MemAddressFree(a->va, a->va_size);
        } else if (g.mode == Mode::kLocal) {
            for (int r = 0; r < g.world; ++r) {
                cudaSetDevice(g.ranks[r].device);
                cudaFree(a->base[r]);
            }
        } else {
            cudaFree(a->base[0]);
        }
    }
    g.allocs.clear();
    for (auto& rc : g.ranks) destroy_rank_ctx(rc);
    g.ranks.clear();
    g.boot.Close();
    g.mode = Mode::kNone;
    g.world = 1;
    g.rank = 0;
    return 0;
}

int catccos_b200_symm_alloc(size_t bytes, void** local_ptr)
{
    if (local_ptr == nullptr || bytes == 0) {
        return CATCCOS_B200_EINVAL;
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    std::lock_guard<std::mutex> lock(g.mu);
    const int W = g.world;
    if (g.mode == Mode::kLocal) {
        // the k-th call of every rank names the same allocation
        uint32_t idx = g.local_alloc_cursor[g.rank]++;
        uint32_t seen = 0;
        SymmAlloc* sa = nullptr;
        for (auto& a : g.allocs) {
            if (a && seen++ == idx) {
                sa = a.get();
                break;
            }
        }
        if (sa == nullptr) {
            auto na = std::make_unique<SymmAlloc>();
            na->size = align_up(bytes, 1024);
            na->base.assign(W, nullptr);
            na->epoch.assign(W, 0);
            na->released.assign(W, false);
            for (int r = 0; r < W; ++r) {
                CUDA_TRY(cudaSetDevice(g.ranks[r].device));
                CUDA_TRY(cudaMalloc(&na->base[r], na->size));
                CUDA_TRY(cudaMemset(na->base[r], 0, na->size));
            }
            for (int r = 0; r < W; ++r) {
                CUDA_TRY(cudaSetDevice(g.ranks[r].device));
                CUDA_TRY(cudaDeviceSynchronize());
            }
            CUDA_TRY(cudaSetDevice(g.ranks[g.rank].device));
            sa = na.get();
            g.allocs.push_back(std::move(na));
        } else if (sa->size < bytes) {
            ERROR_LOG("symm_alloc: ranks disagree on the size of allocation %u", idx);
            return CATCCOS_B200_EINVAL;
        }
        *local_ptr = sa->base[g.rank];
        return 0;
    }
    RankCtx& rc = g.ranks[0];
    CUDA_TRY(cudaSetDevice(rc.device));
    auto na = std::make_unique<SymmAlloc>();
    na->base.assign(W, nullptr);
    na->epoch.assign(W, 0);
    if (W == 1) {
        na->size = align_up(bytes, 1024);
        CUDA_TRY(cudaMalloc(&na->base[0], na->size));
        CUDA_TRY(cudaMemset(na->base[0], 0, na->size));
        CUDA_TRY(cudaDeviceSynchronize());
    } else {
        Driver& d = g.drv;
        CUmemAllocationProp prop = {};
        prop.type = CU_MEM_ALLOCATION_TYPE_PINNED;
        prop.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
        prop.location.id = rc.device;
        prop.requestedHandleTypes = CU_MEM_HANDLE_TYPE_POSIX_FILE_DESCRIPTOR;
        size_t gran = 0;
        CU_TRY(d.MemGetGranularity(&gran, &prop, CU_MEM_ALLOC_GRANULARITY_RECOMMENDED));
        na->size = align_up(bytes, gran);
        na->vmm = true;
        na->handles.assign(W, 0);
        CU_TRY(d.MemCreate(&na->handles[g.rank], na->size, &prop, 0));
        int my_fd = -1;
        CU_TRY(d.MemExport(&my_fd, na->handles[g.rank], CU_MEM_HANDLE_TYPE_POSIX_FILE_DESCRIPTOR, 0));
        std::vector<int> fds;
        if (!g.boot.ExchangeFds(my_fd, fds)) {
            ERROR_LOG("symm_alloc: handle exchange failed: %s", g.boot.error().c_str());
            return CATCCOS_B200_ENET;
        }
        for (int r = 0; r < W; ++r) {
            if (r != g.rank) {
                CU_TRY(d.MemImport(&na->handles[r], (void*)(uintptr_t)fds[r], CU_MEM_HANDLE_TYPE_POSIX_FILE_DESCRIPTOR));
            }
            close(fds[r]);
        }
        na->va_size = na->size * W;
        CU_TRY(d.MemAddressReserve(&na->va, na->va_size, gran, 0, 0));
        CUmemAccessDesc acc = {};
        acc.location.type = CU_MEM_LOCATION_TYPE_DEVICE;
        acc.location.id = rc.device;
        acc.flags = CU_MEM_ACCESS_FLAGS_PROT_READWRITE;
        for (int r = 0; r < W; ++r) {
            CU_TRY(d.MemMap(na->va + (size_t)r * na->size, na->size, 0, na->handles[r], 0));
            na->base[r] = reinterpret_cast<uint8_t*>(na->va + (size_t)r * na->size);
        }
        CU_TRY(d.MemSetAccess(na->va, na->va_size, &acc, 1));
        CUDA_TRY(cudaMemset(na->base[g.rank], 0, na->size));
        CUDA_TRY(cudaDeviceSynchronize());
        if (!g.boot.Barrier()) {  // nobody pushes into a buffer that is still being cleared
            return CATCCOS_B200_ENET;
        }
    }
    *local_ptr = na->base[g.rank];
    g.allocs.push_back(std::move(na));
    return 0;
}

int catccos_b200_symm_free(void* local_ptr)
{
    std::lock_guard<std::mutex> lock(g.mu);
    for (auto& a : g.allocs) {
        if (!a || a->base[g.rank] != local_ptr) {
            continue;
        }
        if (g.mode == Mode::kLocal) {
            a->released[g.rank] = true;  // freed once every rank has let go
            bool all = true;
            for (int r = 0; r < g.world; ++r) all = all && a->released[r];
            if (!all) return 0;
            for (int r = 0; r < g.world; ++r) {
                cudaSetDevice(g.ranks[r].device);
                cudaDeviceSynchronize();
                cudaFree(a->base[r]);
            }
            cudaSetDevice(g.ranks[g.rank].device);
        } else {
            CUDA_TRY(cudaDeviceSynchronize());
            if (a->vmm) {
                g.boot.Barrier();  // peers may still be storing into this rank's copy
                g.drv.MemUnmap(a->va, a->va_size);
                for (auto h : a->handles) g.drv.MemRelease(h);
                g.drv.MemAddressFree(a->va, a->va_size);
            } else {
                cudaFree(a->base[0]);
            }
        }
        a.reset();
        return 0;
    }
    return CATCCOS_B200_ENOTSYMM;
}

size_t catccos_b200_symm_bytes_needed(const catccos_b200_tiling_t* t, int quant_op)
{
    if (t == nullptr) return 0;
    const size_t W = t->rankSize ? t->rankSize : 1;
    const size_t M = t->m;
    if (quant_op == 2) {  // Matmul + ReduceScatter: two stages of the whole fp32 product (m is the whole M there)
        return kHeaderBytes + 2 * align_up(M * (size_t)t->n * sizeof(float), 1024) + 2048;
    }
    const size_t K = quant_op ? t->n : t->k;
    return kHeaderBytes + 2 * (align_up(W * M * K, 1024) + align_up(W * M * (K / 32), 1024)) + 2048;
}

int catccos_b200_mx_quant(void* stream, const void* in_bf16, uint32_t rows, uint32_t k, void* codes, void* scales)
{
    if (!in_bf16 || !codes || !scales || rows == 0 || k == 0 || k % 32 != 0) {
        return CATCCOS_B200_EINVAL;
    }
    if (((uintptr_t)in_bf16 | (uintptr_t)codes) & 15u) {
        return CATCCOS_B200_EINVAL;
    }
    if (k % 128 == 0 && ((uintptr_t)scales & 3u)) {
        return CATCCOS_B200_EINVAL;  // a row of whole words: the GEMMs, which take such rows, read the scales as 32-bit words
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    return launch_quant_flat((cudaStream_t)stream, in_bf16, rows, k, (uint8_t*)codes, (uint8_t*)scales);
}

int catccos_b200_mx_quant_fp4(void* stream, const void* in_bf16, uint32_t rows, uint32_t k, void* packed, void* scales)
{
    if (!in_bf16 || !packed || !scales || rows == 0 || k == 0 || k % 32 != 0) {
        return CATCCOS_B200_EINVAL;
    }
    if (((uintptr_t)in_bf16 & 15u) || ((uintptr_t)packed & 7u)) {
        return CATCCOS_B200_EINVAL;
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    const uint64_t halves = (uint64_t)rows * (k / 16);
    CUDA_TRY(launch_after(mx_quant_e2m1_kernel, dim3((unsigned)((halves + kQuantThreads - 1) / kQuantThreads)), kQuantThreads, 0,
                          (cudaStream_t)stream, static_cast<const uint8_t*>(in_bf16), halves, static_cast<uint8_t*>(packed),
                          static_cast<uint8_t*>(scales), g.tiny_block_rule != 0 ? 1u : 0u));
    return 0;
}

int catccos_b200_mx_quant_allgather(void* stream, const void* in_bf16, void* out_codes, void* out_scales, void* symm,
                                    const catccos_b200_tiling_t* t, uint32_t magic)
{
    (void)magic;
    if (!t || !in_bf16 || !out_codes || !out_scales) {
        return CATCCOS_B200_EINVAL;
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    const uint32_t M = t->m, K = t->n, W = t->rankSize;  // the quantised axis is called n here
    if (W != (uint32_t)g.world || M == 0 || K == 0 || K % 32 != 0) {
        ERROR_LOG("mx quant allgather: rankSize %u (world %d), M=%u N=%u: N must be a positive multiple of 32", W,
                  g.world, M, K);
        return CATCCOS_B200_EINVAL;
    }
    if (((uintptr_t)in_bf16 | (uintptr_t)out_codes) & 15u) {
        return CATCCOS_B200_EINVAL;
    }
    if (K % 128 == 0 && ((uintptr_t)out_scales & 3u)) {
        return CATCCOS_B200_EINVAL;  // several ranks copy such rows as 32-bit words, and the GEMMs read them so
    }
    RankCtx& rc = cur();
    CUDA_TRY(cudaSetDevice(rc.device));
    const uint32_t rank = (uint32_t)g.rank;
    QuantPushParams q = {};
    q.in = in_bf16;
    q.M = M;
    q.K = K;
    q.rank = rank;
    q.world = W;
    q.num_dst = W;
    q.status = rc.status;
    q.timeout_ns = g.timeout_ns;
    choose_segments(M, K, rc.num_sms, q);
    uint8_t* oc = (uint8_t*)out_codes;
    uint8_t* os = (uint8_t*)out_scales;
    if (W == 1) {
        return launch_quant_flat((cudaStream_t)stream, in_bf16, M, K, oc, os);
    }
    SymmAlloc* sa = find_symm(symm);
    if (sa == nullptr) {
        ERROR_LOG("mx quant allgather: symm must come from catccos_b200_symm_alloc");
        return CATCCOS_B200_ENOTSYMM;
    }
    StageLayout L;
    const uint32_t chunks = (M + kRowsPerChunk - 1) / kRowsPerChunk;
    if (!stage_layout(sa->size, W, M, K, L) || (size_t)chunks * q.segs_per_chunk > kMaxFlags) {
        ERROR_LOG("mx quant allgather: symmetric buffer of %zu bytes too small", sa->size);
        return CATCCOS_B200_ENOMEM;
    }
    const bool produce = (g.phase_mask & 1) != 0, consume = (g.phase_mask & 2) != 0;
    if (produce) {
        sa->epoch[g.rank] += 1;
    }
    const uint32_t epoch = sa->epoch[g.rank];
    const size_t stage_off = kHeaderBytes + (size_t)(epoch & 1u) * L.stage_bytes;
    cudaStream_t st = (cudaStream_t)stream;
    uint32_t* my_flags = reinterpret_cast<uint32_t*>(sa->base[rank] + kFlagsOff);
    // Outputs that live in symmetric memory (the same offset on every rank) receive the peers' shards directly;
    // other outputs receive them through this rank's stage and one more local copy.
    size_t off_c = 0, off_s = 0;
    SymmAlloc* sc = find_symm_containing(oc, (size_t)W * M * K, &off_c);
    SymmAlloc* ss = find_symm_containing(os, (size_t)W * M * (K / 32), &off_s);
    const bool direct = sc != nullptr && ss != nullptr;
    // the quantise kernel writes this rank's shard into the caller's output and sets this rank's own flag words
    q.epoch = epoch;
    q.publish = 1;
    q.dst_codes[rank] = oc + (size_t)rank * M * K;
    q.dst_scales[rank] = os + (size_t)rank * M * (K / 32);
    q.dst_flags[rank] = my_flags + (size_t)rank * kMaxFlags;
    if (produce) {
        rcode = launch_quant_push(rc, st, q, false, true, true);
        if (rcode != 0) return rcode;
        // the copy engines forward it, slice by slice, to every peer: into the peer's output or its stage
        uint8_t* dc[kMaxRanks] = {};
        uint8_t* ds[kMaxRanks] = {};
        uint32_t* df[kMaxRanks] = {};
        for (uint32_t d = 0; d < W; ++d) {
            if (d == rank) continue;
            uint8_t* base = sa->base[d] + stage_off;
            dc[d] = (direct ? sc->base[d] + off_c : base + L.codes_off) + (size_t)rank * M * K;
            ds[d] = (direct ? ss->base[d] + off_s : base + L.scales_off) + (size_t)rank * M * (K / 32);
            df[d] = reinterpret_cast<uint32_t*>(sa->base[d] + kFlagsOff) + (size_t)rank * kMaxFlags;
        }
        // nobody consumes this operator's rows early: one slice per peer (three copies: scales, codes, flags)
        // keeps the copies long and their fixed start-up cost small
        const uint32_t slice_rows = (uint32_t)align_up(M, kRowsPerChunk);
        rcode = copy_engine_push(rc, st, W, rank, M, K, q.segs_per_chunk, slice_rows, q.dst_codes[rank], q.dst_scales[rank],
                                 q.dst_flags[rank], dc, ds, df);
        if (rcode != 0) return rcode;
    }
    if (consume) {
        if (direct) {
            CUDA_TRY(launch_after(wait_flags_kernel, dim3(1), 128, 0, st, my_flags, kMaxFlags, W, rank, chunks, q.segs_per_chunk,
                                  epoch, g.timeout_ns, rc.status));
        } else {
            QuantPushParams qc = q;
            qc.consume = 1;
            qc.stage_codes = sa->base[rank] + stage_off + L.codes_off;
            qc.stage_scales = sa->base[rank] + stage_off + L.scales_off;
            qc.out_codes = oc;
            qc.out_scales = os;
            qc.flags = my_flags;
            qc.flag_stride = kMaxFlags;
            rcode = launch_quant_push(rc, st, qc, false, false);
            if (rcode != 0) return rcode;
        }
    }
    return produce ? copy_engine_join(rc, st, W) : 0;
}

int catccos_b200_fp8_mx_allgather_matmul(void* stream, const void* a, const void* b, const void* a_scale,
                                         const void* b_scale, void* c, void* symm, const catccos_b200_tiling_t* t,
                                         uint32_t magic)
{
    (void)magic;
    return allgather_matmul(stream, a, a_scale, true, b, b_scale, c, symm, t);
}

int catccos_b200_fp4_mx_allgather_matmul(void* stream, const void* a, const void* b, const void* a_scale,
                                         const void* b_scale, void* c, void* symm, const catccos_b200_tiling_t* t,
                                         uint32_t magic)
{
    (void)magic;
    if (!t || !a || !b || !a_scale || !b_scale || !c) {
        return CATCCOS_B200_EINVAL;
    }
    const uint32_t M = t->m, K = t->k, N = t->n, W = t->rankSize;
    if (M == 0 || K == 0 || N == 0) {
        ERROR_LOG("fp4 allgather matmul: M=%u K=%u N=%u unsupported", M, K, N);
        return CATCCOS_B200_EINVAL;
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    if (W != (uint32_t)g.world || K % kGemmBlockK != 0 || N % 16 != 0) {
        ERROR_LOG("fp4 allgather matmul: rankSize %u (world %d), M=%u K=%u N=%u unsupported", W, g.world, M, K, N);
        return CATCCOS_B200_EINVAL;
    }
    RankCtx& rc = cur();
    CUDA_TRY(cudaSetDevice(rc.device));
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t rank = (uint32_t)g.rank;
    // both operands are packed E2M1 for the length of this call, whatever the options say
    struct DtypeGuard {
        int a, b;
        DtypeGuard() : a(g.a_dtype), b(g.b_dtype) { g.a_dtype = 2; g.b_dtype = 2; }
        ~DtypeGuard() { g.a_dtype = a; g.b_dtype = b; }
    } guard;
    GemmParams p = {};
    p.a_scales = (const uint8_t*)a_scale;
    p.b_scales = (const uint8_t*)b_scale;
    p.c = c;
    p.Mg = W * M;
    p.N = N;
    p.K = K;
    p.world = W;
    p.rank = rank;
    p.m_local = M;
    if (W == 1) {
        return launch_gemm(rc, st, a, b, p);
    }
    SymmAlloc* sa = find_symm(symm);
    if (sa == nullptr) {
        ERROR_LOG("fp4 allgather matmul: symm must come from catccos_b200_symm_alloc");
        return CATCCOS_B200_ENOTSYMM;
    }
    // a stage: the gathered packed codes [W * M, K / 2], then the gathered scales [W * M, K / 32]
    const size_t row_bytes = K / 2, sf = K / 32;
    const size_t stage_bytes = ((sa->size - kHeaderBytes) / 2) & ~(size_t)1023;
    const size_t scales_off = align_up((size_t)W * M * row_bytes, 1024);
    const uint32_t chunks = (M + kRowsPerChunk - 1) / kRowsPerChunk;
    if (sa->size < kHeaderBytes + 2048 || scales_off + align_up((size_t)W * M * sf, 1024) > stage_bytes || chunks > kMaxFlags) {
        ERROR_LOG("fp4 allgather matmul: symmetric buffer of %zu bytes too small", sa->size);
        return CATCCOS_B200_ENOMEM;
    }
    const bool produce = (g.phase_mask & 1) != 0, consume = (g.phase_mask & 2) != 0;
    if (produce) {
        sa->epoch[g.rank] += 1;
    }
    const uint32_t epoch = sa->epoch[g.rank];
    const size_t stage_off = kHeaderBytes + (size_t)(epoch & 1u) * stage_bytes;
    uint8_t* dc[kMaxRanks] = {};
    uint8_t* ds[kMaxRanks] = {};
    uint32_t* df[kMaxRanks] = {};
    for (uint32_t d = 0; d < W; ++d) {
        uint8_t* base = sa->base[d] + stage_off;
        dc[d] = base + (size_t)rank * M * row_bytes;
        ds[d] = base + scales_off + (size_t)rank * M * sf;
        df[d] = reinterpret_cast<uint32_t*>(sa->base[d] + kFlagsOff) + (size_t)rank * kMaxFlags;
    }
    if (produce) {
        // A arrives quantised: this rank's shard goes into its own stage by two copies, its flag words are set,
        // and the copy engines forward all three to the peers (one flag word per 16-row chunk, one K segment)
        CUDA_TRY(cudaMemcpyAsync(dc[rank], a, (size_t)M * row_bytes, cudaMemcpyDeviceToDevice, st));
        CUDA_TRY(cudaMemcpyAsync(ds[rank], a_scale, (size_t)M * sf, cudaMemcpyDeviceToDevice, st));
        CUDA_TRY(launch_after(fill_flags_kernel, dim3((chunks + 255) / 256), 256, 0, st, df[rank], chunks, epoch));
        rcode = copy_engine_push(rc, st, W, rank, M, K, 1, kCopySliceRows, dc[rank], ds[rank], df[rank], dc, ds, df, row_bytes);
        if (rcode != 0) return rcode;
    }
    if (consume) {
        p.a_scales = sa->base[rank] + stage_off + scales_off;
        p.flags = reinterpret_cast<const uint32_t*>(sa->base[rank] + kFlagsOff);
        p.flag_stride = kMaxFlags;
        p.segs = 1;
        p.seg_ktiles = K / kGemmBlockK;
        p.epoch = epoch;
        rcode = launch_gemm(rc, st, sa->base[rank] + stage_off, b, p);
        if (rcode != 0) return rcode;
    }
    return produce ? copy_engine_join(rc, st, W) : 0;
}

int catccos_b200_mx_quant_allgather_matmul(void* stream, const void* a_bf16, const void* b, const void* b_scale,
                                           void* c, void* symm, const catccos_b200_tiling_t* t, uint32_t magic)
{
    (void)magic;
    return allgather_matmul(stream, a_bf16, nullptr, false, b, b_scale, c, symm, t);
}

int catccos_b200_mx_gemm(void* stream, const void* a, const void* a_scale, const void* b, const void* b_scale, void* c,
                         uint32_t m, uint32_t n, uint32_t k)
{
    if (!a || !a_scale || !b || !b_scale || !c) {
        return CATCCOS_B200_EINVAL;
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    RankCtx& rc = cur();
    GemmParams p = {};
    p.a_scales = (const uint8_t*)a_scale;
    p.b_scales = (const uint8_t*)b_scale;
    p.c = c;
    p.Mg = m;
    p.N = n;
    p.K = k;
    p.flags = nullptr;
    p.world = 1;
    p.m_local = m;
    return launch_gemm(rc, (cudaStream_t)stream, a, b, p);
}

int catccos_b200_mx_gemm_quant_out(void* stream, const void* a, const void* a_scale, const void* b, const void* b_scale,
                                   void* c_codes, void* c_scales, uint32_t m, uint32_t n, uint32_t k)
{
    if (!a || !a_scale || !b || !b_scale || !c_codes || !c_scales) {
        return CATCCOS_B200_EINVAL;
    }
    if (n % 32 != 0) {
        ERROR_LOG("mx gemm with quantised output: n must be a multiple of 32 (got %u)", n);
        return CATCCOS_B200_EINVAL;
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    RankCtx& rc = cur();
    GemmParams p = {};
    p.a_scales = (const uint8_t*)a_scale;
    p.b_scales = (const uint8_t*)b_scale;
    p.c = c_codes;
    p.c_scales = (uint8_t*)c_scales;
    p.c_tiny_rule = g.tiny_block_rule != 0 ? kQuantDeviceTiny : kQuantGolden;
    p.Mg = m;
    p.N = n;
    p.K = k;
    p.flags = nullptr;
    p.world = 1;
    p.m_local = m;
    return launch_gemm(rc, (cudaStream_t)stream, a, b, p, false, false, kEpiMxQuant);
}

// Matmul + ReduceScatter: what plan_gemm will choose for the N tile (the reducer walks the same tiles)
static uint32_t scatter_block_n(const RankCtx& rc, uint32_t M, uint32_t N, uint32_t K)
{
    return plan_gemm(rc, M, N, K, true, true).block_n;
}

int catccos_b200_mxfp8_matmul_reduce_scatter(void* stream, const void* a, const void* b, const void* a_scale,
                                             const void* b_scale, void* d, void* symm, const catccos_b200_tiling_t* t,
                                             uint32_t magic)
{
    (void)magic;
    if (!t || !a || !b || !a_scale || !b_scale || !d) {
        return CATCCOS_B200_EINVAL;
    }
    const uint32_t M = t->m, K = t->k, N = t->n, W = t->rankSize;  // m is the whole M: every rank holds all rows of its K slice
    if (M == 0 || K == 0 || N == 0) {
        ERROR_LOG("matmul reduce scatter: M=%u K=%u N=%u unsupported", M, K, N);
        return CATCCOS_B200_EINVAL;
    }
    if ((uintptr_t)d & 7u) {
        ERROR_LOG("matmul reduce scatter: d must be 8-byte aligned (32-byte with one rank)");
        return CATCCOS_B200_EINVAL;  // the reducer stores four 16-bit results at a time
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    if (W != (uint32_t)g.world || K % kGemmBlockK != 0 || N % 16 != 0 || M % W != 0 || (M / W) % 32 != 0) {
        ERROR_LOG("matmul reduce scatter: rankSize %u (world %d), M=%u K=%u N=%u unsupported (M / rankSize must be a "
                  "multiple of 32, K of 128, N of 16)", W, g.world, M, K, N);
        return CATCCOS_B200_EINVAL;
    }
    RankCtx& rc = cur();
    CUDA_TRY(cudaSetDevice(rc.device));
    cudaStream_t st = (cudaStream_t)stream;
    const uint32_t rank = (uint32_t)g.rank, rows = M / W;
    const bool produce = (g.phase_mask & 1) != 0, consume = (g.phase_mask & 2) != 0;
    if (W == 1) {
        // nothing to reduce: the plain GEMM writes D
        GemmParams p = {};
        p.a_scales = (const uint8_t*)a_scale;
        p.b_scales = (const uint8_t*)b_scale;
        p.c = d;
        p.Mg = M;
        p.N = N;
        p.K = K;
        p.world = 1;
        p.m_local = M;
        return launch_gemm(rc, st, a, b, p);
    }
    SymmAlloc* sa = find_symm(symm);
    if (sa == nullptr) {
        ERROR_LOG("matmul reduce scatter: symm must come from catccos_b200_symm_alloc");
        return CATCCOS_B200_ENOTSYMM;
    }
    const uint32_t bn = scatter_block_n(rc, M, N, K);
    const uint32_t n_tiles = (N + bn - 1) / bn;
    const size_t stage_bytes = ((sa->size - kHeaderBytes) / 2) & ~(size_t)1023;
    const size_t need = (size_t)M * N * sizeof(float);  // world slots of [rows, N] fp32
    if (sa->size < kHeaderBytes + 2048 || need > stage_bytes || (size_t)(rows / 32) * n_tiles > kMaxFlags) {
        ERROR_LOG("matmul reduce scatter: symmetric buffer of %zu bytes too small (needs %zu)", sa->size,
                  kHeaderBytes + 2 * need + 2048);
        return CATCCOS_B200_ENOMEM;
    }
    if (produce) {
        sa->epoch[g.rank] += 1;
    }
    const uint32_t epoch = sa->epoch[g.rank];
    const size_t stage_off = kHeaderBytes + (size_t)(epoch & 1u) * stage_bytes;
    if (produce) {
        GemmParams p = {};
        p.a_scales = (const uint8_t*)a_scale;
        p.b_scales = (const uint8_t*)b_scale;
        p.c = nullptr;
        p.Mg = M;
        p.N = N;
        p.K = K;
        p.world = W;
        p.rank = rank;
        p.m_local = M;
        p.epoch = epoch;
        p.rs_rows = rows;
        for (uint32_t dr = 0; dr < W; ++dr) {
            p.rs_dst[dr] = reinterpret_cast<float*>(sa->base[dr] + stage_off);
            p.rs_flags[dr] = reinterpret_cast<uint32_t*>(sa->base[dr] + kFlagsOff) + (size_t)rank * kMaxFlags;
        }
        rcode = launch_gemm(rc, st, a, b, p, false, false, kEpiScatter);
        if (rcode != 0) return rcode;
    }
    if (consume) {
        const uint32_t units = (rows / 32) * n_tiles;
        const uint32_t grid = std::min(units, (uint32_t)rc.num_sms * 4u);
        const float* parts = reinterpret_cast<const float*>(sa->base[rank] + stage_off);
        const uint32_t* flags = reinterpret_cast<const uint32_t*>(sa->base[rank] + kFlagsOff);
        if (g.c_dtype == 1) {
            CUDA_TRY(launch_after(mx_reduce_scatter_kernel<__half>, dim3(grid), 256, 0, st, parts, flags, kMaxFlags, W, rows, N, bn,
                                  epoch, (__half*)d, g.timeout_ns, rc.status));
        } else {
            CUDA_TRY(launch_after(mx_reduce_scatter_kernel<__nv_bfloat16>, dim3(grid), 256, 0, st, parts, flags, kMaxFlags, W, rows,
                                  N, bn, epoch, (__nv_bfloat16*)d, g.timeout_ns, rc.status));
        }
    }
    return 0;
}

size_t catccos_b200_packed_row_bytes(uint32_t n) { return packed_row_bytes(n); }

int catccos_b200_mx_quant_scatter_packed(void* stream, const void* in_bf16, const int32_t* expanded_row_idx, void* packed_out,
                                         uint32_t tokens, uint32_t n, uint32_t top_k)
{
    if (!in_bf16 || !expanded_row_idx || !packed_out || n == 0 || n % 32 != 0 || top_k == 0) {
        return CATCCOS_B200_EINVAL;
    }
    if ((((uintptr_t)in_bf16 | (uintptr_t)packed_out) & 15u) != 0) {
        return CATCCOS_B200_EINVAL;  // rows are read and written 16 bytes at a time
    }
    if (tokens == 0) {
        return 0;
    }
    int rcode = ensure_init();
    if (rcode != 0) return rcode;
    const uint64_t warps = (uint64_t)tokens * ((n + kQuantColsPerWarpStep - 1) / kQuantColsPerWarpStep);
    const unsigned grid = (unsigned)((warps + kQuantThreads / 32 - 1) / (kQuantThreads / 32));
    CUDA_TRY(launch_after(mx_quant_scatter_packed_kernel, dim3(grid), kQuantThreads, 0, (cudaStream_t)stream,
                          static_cast<const uint16_t*>(in_bf16), expanded_row_idx, static_cast<uint8_t*>(packed_out), tokens, n,
                          top_k, g.tiny_block_rule != 0 ? 1u : 0u));
    return 0;
}

int catccos_b200_last_status(uint32_t out[4])
{
    if (out == nullptr || g.mode == Mode::kNone) {
        return CATCCOS_B200_ESTATE;
    }
    RankCtx& rc = cur();
    CUDA_TRY(cudaSetDevice(rc.device));
    CUDA_TRY(cudaDeviceSynchronize());
    StatusBlock sb;
    CUDA_TRY(cudaMemcpy(&sb, rc.status, sizeof(sb), cudaMemcpyDeviceToHost));
    out[0] = sb.code;
    out[1] = sb.rank;
    out[2] = sb.chunk;
    out[3] = sb.epoch;
    if (sb.code != 0) {
        ERROR_LOG("device wait ran out: code %u rank/barrier %u chunk/stage %u epoch %u", sb.code, sb.rank, sb.chunk,
                  sb.epoch);
        CUDA_TRY(cudaMemset(rc.status, 0, sizeof(sb)));
        return CATCCOS_B200_ETIMEOUT;
    }
    return 0;
}

int catccos_b200_set_option(const char* key, int64_t value)
{
    if (key == nullptr) return CATCCOS_B200_EINVAL;
    std::string k = key;
    if (k == "tiny_block_rule" && (value == 0 || value == 1)) {
        g.tiny_block_rule = (int)value;
    } else if (k == "c_dtype" && (value == 0 || value == 1)) {
        g.c_dtype = (int)value;
    } else if (k == "a_dtype" && value >= 0 && value <= 2) {
        g.a_dtype = (int)value;
    } else if (k == "b_dtype" && value >= 0 && value <= 2) {
        g.b_dtype = (int)value;
    } else if (k == "timeout_ms" && value > 0 && value <= 600000) {
        g.timeout_ns = (uint64_t)value * 1000000ull;
    } else if (k == CATCCOS_B200_OPT_BLOCK_N && (value == 0 || value == 64 || value == 128 || value == 256)) {
        g.block_n = (int)value;
    } else if (k == CATCCOS_B200_OPT_PHASE_MASK && value >= 1 && value <= 3) {
        g.phase_mask = (int)value;
    } else if (k == CATCCOS_B200_OPT_CTA_PAIR && value >= 0 && value <= 2) {
        g.cta_pair = (int)value;
    } else if (k == CATCCOS_B200_OPT_FUSE_MODE && (value == -1 || value == 0 || (value >= 3 && value <= 7))) {
        g.fuse_mode = (int)value;
    } else if (k == CATCCOS_B200_OPT_SPLIT_K && value >= 0 && value <= 8) {
        g.split_k = (int)value;
    } else if (k == CATCCOS_B200_OPT_B_LSU && value >= 0 && value <= 2) {
        g.b_lsu = (int)value;
    } else if (k == CATCCOS_B200_OPT_SMALL_TILE && value >= 0 && value <= 2) {
        g.small_tile = (int)value;
    } else if (k == CATCCOS_B200_OPT_SMALL_QUANT && value >= 0 && value <= 2) {
        g.small_quant = (int)value;
    } else if (k == CATCCOS_B200_OPT_TILE_ORDER && value >= -1 && value <= 1) {
        g.tile_order = (int)value;
    } else {
        ERROR_LOG("set_option: unknown key or bad value: %s = %lld", key, (long long)value);
        return CATCCOS_B200_EINVAL;
    }
    return 0;
}

uint64_t catccos_b200_launch_count(void) { return g_launches.load(); }

}  // extern "C"

// =============================================================================================
// Allocation-free single-GPU entry point
// =============================================================================================
namespace {

// Scratch of catccos_b200_mx_quant_matmul_static: the quantised copy of A lives in
// this file-scope device array instead of a buffer from catccos_b200_symm_alloc.  Every GPU that
// loads the library carries it (about 8.3 MiB) until the process exits.
constexpr size_t kStaticMaxElems = size_t(8) << 20;  // m * k may not exceed this
constexpr size_t kStaticStatusOff = 0;
constexpr size_t kStaticScalesOff = kStaticStatusOff + 1024;
constexpr size_t kStaticCodesOff = kStaticScalesOff + kStaticMaxElems / 32;
constexpr size_t kStaticBytes = kStaticCodesOff + kStaticMaxElems;
static_assert(kStaticScalesOff % 256 == 0 && kStaticCodesOff % 1024 == 0, "TMA and vector stores need these aligned");

static __device__ __align__(256) uint8_t g_static_scratch[kStaticBytes];

struct StaticDeviceState {
    uint8_t* ptr = nullptr;  // device address of g_static_scratch on this device
    int num_sms = 0;
    WaitRecordTurn turn;
};
StaticDeviceState g_static_dev[kMaxRanks * 2];
std::mutex g_static_mu;

}  // namespace

extern "C" int catccos_b200_mx_quant_matmul_static(void* stream, const void* a_bf16, const void* b, const void* b_scale,
                                                   void* c, uint32_t m, uint32_t n, uint32_t k)
{
    if (!a_bf16 || !b || !b_scale || !c || m == 0 || n == 0 || k == 0) {
        return CATCCOS_B200_EINVAL;
    }
    if (k % kGemmBlockK != 0 || n % 16 != 0) {
        ERROR_LOG("mx_quant_matmul_static: k must be a multiple of 128 and n of 16 (got n=%u k=%u)", n, k);
        return CATCCOS_B200_EINVAL;
    }
    if (!matmul_operands_ok("mx_quant_matmul_static", a_bf16, b, b_scale, c)) {
        return CATCCOS_B200_EINVAL;  // refused before the shared array or the stream is touched
    }
    if ((size_t)m * k > kStaticMaxElems) {
        ERROR_LOG("mx_quant_matmul_static: m * k = %zu exceeds the built-in scratch of %zu elements; "
                  "use catccos_b200_mx_quant_allgather_matmul with a buffer from catccos_b200_symm_alloc",
                  (size_t)m * k, kStaticMaxElems);
        return CATCCOS_B200_ENOMEM;
    }
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxRanks * 2) {
        return CATCCOS_B200_EINVAL;
    }
    std::lock_guard<std::mutex> lock(g_static_mu);
    StaticDeviceState& sd = g_static_dev[dev];
    if (sd.ptr == nullptr) {
        // One-time set-up for this device (it is current).  In host code the array's name is only a
        // stand-in; the address a kernel may use comes from the runtime.
        void* p = nullptr;
        int sms = 0;
        CUDA_TRY(cudaGetSymbolAddress(&p, g_static_scratch));
        CUDA_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        if (!g.drv.Load()) {
            return CATCCOS_B200_ECUDA;
        }
        sd.num_sms = sms;  // the state is filled in only once every step of the set-up has succeeded
        sd.ptr = static_cast<uint8_t*>(p);
    }
    RankCtx rc;  // a view for the launcher: nothing is created or owned here
    rc.device = dev;
    rc.num_sms = sd.num_sms;
    StatusBlock* records = reinterpret_cast<StatusBlock*>(sd.ptr + kStaticStatusOff);
    cudaStream_t st = (cudaStream_t)stream;
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    CUDA_TRY(cudaStreamIsCapturing(st, &capture));
    const bool captured = capture != cudaStreamCaptureStatusNone;

    if (g.b_dtype == 2) {
        return CATCCOS_B200_ESTATE;  // packed weights need a transposed copy, and this path has no scratch for it
    }
    const SmallPlan small = plan_small(rc, m, n, k, true);
    if (small.use && small.quant) {
        // one launch (wait_records.hpp: how it comes by a clear record)
        rc.status = records + sd.turn.one_launch(captured);
        if (captured) {
            CUDA_TRY(cudaMemsetAsync(rc.status, 0, sizeof(StatusBlock), st));
        }
        SmallParams sp = {};
        sp.x = a_bf16;
        sp.w_scales = (const uint8_t*)b_scale;
        sp.c = c;
        sp.M = m;
        sp.N = n;
        sp.K = k;
        sp.records = records;
        return launch_small(rc, st, small, nullptr, b, sp, false);
    }
    // Two launches on the caller's stream, as catccos_b200_mx_quant_allgather_matmul at one rank: the quantiser on every
    // SM, then the GEMM (K in one piece: the array has no room for partial tiles).  One kernel that does both measured
    // 36 us on 509 x 2320 x 3968.
    rc.status = records + sd.turn.two_launches(captured);
    uint8_t* codes = sd.ptr + kStaticCodesOff;
    uint8_t* scales = sd.ptr + kStaticScalesOff;
    int rcode = launch_quant_flat(st, a_bf16, m, k, codes, scales, records);
    if (rcode != 0) return rcode;
    GemmParams p = {};
    p.a_scales = scales;
    p.b_scales = (const uint8_t*)b_scale;
    p.c = c;
    p.Mg = m;
    p.N = n;
    p.K = k;
    p.world = 1;
    p.m_local = m;
    p.b_early = 1;
    return launch_gemm(rc, st, codes, b, p, false, true);
}

#ifdef CATCCOS_TRACE
// =============================================================================================
// Device-side timeline (trace build only; declarations: include/catccos_b200_trace.h)
// =============================================================================================
extern "C" int catccos_b200_trace_arm(void)
{
    if (g.mode == Mode::kNone) {
        return CATCCOS_B200_ESTATE;
    }
    RankCtx& rc = cur();
    CUDA_TRY(cudaSetDevice(rc.device));
    CUDA_TRY(cudaDeviceSynchronize());
    CUDA_TRY(cudaMemset(rc.trace, 0, (size_t)rc.num_sms * kTraceSlots * sizeof(unsigned long long)));
    // the stand-alone quantise kernel keeps the minimum of its CTAs' start times in this word
    const unsigned long long big = ~0ull;
    CUDA_TRY(cudaMemcpy(rc.trace + kTrQuantKernelStart, &big, sizeof(big), cudaMemcpyHostToDevice));
    g.trace_armed = true;
    return 0;
}

extern "C" int catccos_b200_trace_read(unsigned long long* out, uint32_t max_words, uint32_t* grid, uint32_t* slots)
{
    if (out == nullptr || grid == nullptr || slots == nullptr || g.mode == Mode::kNone) {
        return CATCCOS_B200_ESTATE;
    }
    RankCtx& rc = cur();
    const size_t words = (size_t)rc.trace_grid * kTraceSlots;
    if (rc.trace == nullptr || words == 0 || words > max_words) {
        return CATCCOS_B200_EINVAL;
    }
    CUDA_TRY(cudaSetDevice(rc.device));
    CUDA_TRY(cudaDeviceSynchronize());
    CUDA_TRY(cudaMemcpy(out, rc.trace, words * sizeof(unsigned long long), cudaMemcpyDeviceToHost));
    *grid = (uint32_t)rc.trace_grid;
    *slots = kTraceSlots;
    return 0;
}
#endif

// The device-side wait record of the allocation-free entry point lives in the built-in array too (the regular
// record belongs to a rank context, which that entry point never creates).  Synchronises the device and copies
// the 16 bytes out; nothing is allocated.
extern "C" int catccos_b200_mx_quant_matmul_static_status(uint32_t out[4])
{
    if (out == nullptr) {
        return CATCCOS_B200_EINVAL;
    }
    int dev = 0;
    CUDA_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxRanks * 2) {
        return CATCCOS_B200_EINVAL;
    }
    std::lock_guard<std::mutex> lock(g_static_mu);
    StaticDeviceState& sd = g_static_dev[dev];
    if (sd.ptr == nullptr) {
        return CATCCOS_B200_ESTATE;  // no call has been made on this device yet
    }
    CUDA_TRY(cudaDeviceSynchronize());
    StatusBlock records[kWaitRecords];
    CUDA_TRY(cudaMemcpy(records, sd.ptr + kStaticStatusOff, sizeof(records), cudaMemcpyDeviceToHost));
    StatusBlock sb = records[0];
    for (const StatusBlock& r : records) {
        if (sb.code == 0) {
            sb = r;  // a call clears the records it does not use: at most one is set
        }
    }
    out[0] = sb.code;
    out[1] = sb.rank;
    out[2] = sb.chunk;
    out[3] = sb.epoch;
    if (sb.code != 0) {
        ERROR_LOG("device wait ran out in mx_quant_matmul_static: code %u rank/barrier %u chunk/stage %u epoch %u", sb.code,
                  sb.rank, sb.chunk, sb.epoch);
        return CATCCOS_B200_ETIMEOUT;
    }
    return 0;
}
