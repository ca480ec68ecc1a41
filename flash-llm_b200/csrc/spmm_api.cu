// Host side of libSpMM_API.so: argument checks, launch-plan choice and kernel launches behind the reference's
// SpMM_SplitK_API interface (reference csrc/SpMM_API.cu:22-130), plus the C-linkage aliases.
#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <mutex>
#include <new>
#include <type_traits>

#include "../../include/SpMM_API.cuh"
#include "launch.h"
#include "spmm_kernel_direct_sm100.cuh"
#include "spmm_kernel_sm100.cuh"
#include "spmm_kernel_stream_sm100.cuh"
#include "spmm_kernel_wide_sm100.cuh"
#include "tiled_csl_host.h"
#include "tiling.h"

namespace flashllm {

__device__ unsigned int g_status_word = 0;

// Scratch of the allocation-free entry point FlashLLM_SpMM_SplitK_NoAlloc: room for the fp32 partial matrices the
// K split parks between the SpMM kernel and its reduction.  It lives in the library image, so every GPU that loads
// the library carries these 8 MiB until the process exits.  In host code this name is only a handle for
// cudaGetSymbolAddress; the device address obtained from it (once per device) is what the kernels receive.
constexpr size_t kNoAllocScratchBytes = size_t(8) << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Arrival counters of the in-kernel split-K sum: kCounterSets sets of one word per output tile, all zero between
// launches.  Launches of one stream are ordered (the sum of one is over before the next one's B loader is let
// through), so a set is bound to a stream; calls on other streams take other sets, and a call that finds no free
// set, or has more output tiles than a set holds, sums with the second kernel instead.
constexpr int kCounterSets = 32, kCounterTiles = 2048;
static __device__ unsigned int g_tile_counters[kCounterSets * kCounterTiles];

static std::atomic<unsigned long long> g_launches{0};

void count_launch()
{
    g_launches.fetch_add(1, std::memory_order_relaxed);
}

// ---------------------------------------------------------------- per-device state

constexpr int kMaxDevices = 64;

// Scratch of the streaming form: one counter per tile row and two fp32 [N][128] parts per CTA of the largest grid at the
// largest N it takes.  Launches on one stream follow one another, so a scratch belongs to a stream (by its unique id: a
// handle may be reused while its old stream's work still runs).  It is allocated at the stream's first such call and kept,
// at most kScratchStreams per device; further streams run the other forms.  Nobody tells the library that a stream has been
// destroyed or that its work has ended (a word that every CTA stores at its end made every launch 0.3 us longer, an event
// behind every launch more), so a place stays its stream's until FlashLLM_ReleaseStreamScratch or FlashLLM_ReleaseScratch.
constexpr int    kScratchStreams = 8, kScratchRows = 4096, kScratchCtas = 2 * 160, kScratchMaxN = 64;
constexpr size_t kScratchBytes   = kScratchRows * sizeof(unsigned int)
                                 + size_t(2) * kScratchCtas * kScratchMaxN * kTileM * sizeof(float);
// Calls of streams without a scratch between an allocation that failed and the next one.
constexpr unsigned int kScratchRetryCalls = 256;

struct StreamScratch {
    unsigned long long stream_id = 0;
    bool               taken     = false;  // by the stream of that id; a place that was given back keeps its memory
    unsigned char*     memory    = nullptr;
};

struct DeviceState {
    std::mutex     mutex;
    bool           ready      = false;  // set once every step of the set-up has succeeded; a failed set-up is retried
    int            sm_count   = 0;
    int            smem_optin = 0;
    unsigned int*  status     = nullptr;
    unsigned char* noalloc_scratch = nullptr;  // device address of g_noalloc_scratch on this device
    unsigned int*  tile_counters   = nullptr;  // device address of g_tile_counters on this device
    int            counter_streams = 0;        // streams that own a counter set so far
    cudaStream_t   counter_stream[kCounterSets] = {nullptr};
    StreamScratch  scratch[kScratchStreams];
    unsigned int   scratch_retry = 0;  // calls to go until an allocation that failed is tried again
};

// The place of the stream with this id, or nullptr.
static StreamScratch* scratch_with_id(DeviceState* st, unsigned long long id)
{
    for (StreamScratch& place : st->scratch)
        if (place.taken && place.stream_id == id)
            return &place;
    return nullptr;
}

// The scratch of `stream` on this device, set up on first use; nullptr while the stream is being captured (a graph may be
// replayed on any stream), when all places are taken, or when memory is short.
static unsigned char* scratch_of_stream(DeviceState* st, cudaStream_t stream)
{
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    unsigned long long      id      = 0;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone
        || cudaStreamGetId(stream, &id) != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(st->mutex);
    if (StreamScratch* mine = scratch_with_id(st, id))
        return mine->memory;
    StreamScratch* place = nullptr;  // a free one, with memory if there is such
    for (StreamScratch& other : st->scratch)
        if (!other.taken && (place == nullptr || (place->memory == nullptr && other.memory != nullptr)))
            place = &other;
    if (place == nullptr)
        return nullptr;
    if (place->memory == nullptr && st->scratch_retry > 0) {
        --st->scratch_retry;
        return nullptr;
    }
    // Another thread may be capturing: allocate in relaxed mode, and clear the counters in this stream's own order.
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (place->memory == nullptr && cudaMalloc(reinterpret_cast<void**>(&place->memory), kScratchBytes) != cudaSuccess) {
        place->memory     = nullptr;
        st->scratch_retry = kScratchRetryCalls;
    }
    const bool ok = place->memory != nullptr
                    && cudaMemsetAsync(place->memory, 0, kScratchRows * sizeof(unsigned int), stream) == cudaSuccess;
    cudaThreadExchangeStreamCaptureMode(&mode);
    if (!ok) {
        cudaGetLastError();
        return nullptr;
    }
    place->stream_id = id;
    place->taken     = true;
    return place->memory;
}

// The counter set of `stream` on this device, or nullptr when all sets are taken by other streams.
static unsigned int* counters_of_stream(DeviceState* st, cudaStream_t stream)
{
    std::lock_guard<std::mutex> lock(st->mutex);
    for (int i = 0; i < st->counter_streams; ++i)
        if (st->counter_stream[i] == stream)
            return st->tile_counters + static_cast<size_t>(i) * kCounterTiles;
    if (st->counter_streams >= kCounterSets)
        return nullptr;
    st->counter_stream[st->counter_streams] = stream;
    return st->tile_counters + static_cast<size_t>(st->counter_streams++) * kCounterTiles;
}

static DeviceState g_devices[kMaxDevices];

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
using ReplaceAddressFn = CUresult (*)(CUtensorMap*, void*);
static EncodeTiledFn    g_encode_tiled    = nullptr;
static ReplaceAddressFn g_replace_address = nullptr;
static std::once_flag g_encode_once;

// Register budget of the register-streaming kernel: vectors per lane kept in registers (tiles of up to 768 vectors,
// i.e. 62.5 % sparsity, need no overflow loop), for its two shapes: 8 scatter warps and one CTA per SM; 4 scatter
// warps and two CTAs per SM.
#ifndef FLASHLLM_NARROW_CAP
#define FLASHLLM_NARROW_CAP 14
#endif
#ifndef FLASHLLM_PAIR_CAP
#define FLASHLLM_PAIR_CAP 8
#endif
// ... and of its shape with two warps per tile (4 stages, 8 scatter warps, two CTAs per SM): rows per warp
#ifndef FLASHLLM_DIRECT_BLOCKS
#define FLASHLLM_DIRECT_BLOCKS 2
#endif
constexpr int kDirectBlocks = FLASHLLM_DIRECT_BLOCKS;  // CTAs per SM of the 4-stage shapes
constexpr int kDirectCapWide = 24, kDirectCapNarrow = FLASHLLM_NARROW_CAP, kDirectCapPair = FLASHLLM_PAIR_CAP;

template<typename Kernel>
static cudaError_t raise_smem_limit_of(Kernel kernel, int optin)
{
    cudaFuncAttributes attr{};
    cudaError_t        e = cudaFuncGetAttributes(&attr, kernel);
    if (e != cudaSuccess)
        return e;
    // the opt-in limit covers static and dynamic shared memory together
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                optin - static_cast<int>(attr.sharedSizeBytes));
}

// Vectors per lane the streaming form keeps in registers: what 96 registers (two CTAs of 10 warps per SM) have room for.
constexpr int kStreamCap = 14;

template<int N_TILE>
static cudaError_t raise_smem_limit(int optin)
{
    cudaError_t e = raise_smem_limit_of(spmm_tcgen05_kernel<N_TILE>, optin);
    auto direct   = [&](auto push) {
        if (e == cudaSuccess)
            e = raise_smem_limit_of(spmm_tcgen05_direct_kernel<N_TILE, kDirectCapWide, 8, 1, 1, push>, optin);
        if (e == cudaSuccess)
            e = raise_smem_limit_of(spmm_tcgen05_direct_kernel<N_TILE, kDirectCapNarrow, 4, kDirectBlocks, 1, push>, optin);
        if (e == cudaSuccess)
            e = raise_smem_limit_of(spmm_tcgen05_direct_kernel<N_TILE, kDirectCapPair, 4, 2, 2, push>, optin);
    };
    direct(std::false_type{});
    if constexpr (N_TILE <= kPushMaxN)
        direct(std::true_type{});
    if constexpr (N_TILE <= kScratchMaxN)
        if (e == cudaSuccess)
            e = raise_smem_limit_of(spmm_tcgen05_stream_kernel<N_TILE, kStreamCap>, optin);
    return e;
}

static DeviceState* device_state(cudaError_t* err)
{
    int dev = 0;
    *err    = cudaGetDevice(&dev);
    if (*err != cudaSuccess)
        return nullptr;
    if (dev < 0 || dev >= kMaxDevices) {
        *err = cudaErrorInvalidDevice;
        return nullptr;
    }
    DeviceState* st = &g_devices[dev];
    std::lock_guard<std::mutex> lock(st->mutex);
    if (st->ready) {
        *err = cudaSuccess;
        return st;
    }
    // Nothing here allocates.  A failure (for instance a first call made while a stream is being captured) is
    // returned to this caller only; the next call tries again.
    cudaError_t e = cudaDeviceGetAttribute(&st->sm_count, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
        e = cudaDeviceGetAttribute(&st->smem_optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e == cudaSuccess)
        e = cudaGetSymbolAddress(reinterpret_cast<void**>(&st->status), g_status_word);
    if (e == cudaSuccess)
        e = cudaGetSymbolAddress(reinterpret_cast<void**>(&st->noalloc_scratch), g_noalloc_scratch);
    if (e == cudaSuccess)
        e = cudaGetSymbolAddress(reinterpret_cast<void**>(&st->tile_counters), g_tile_counters);
    // The opt-in limit is a per-device property of each kernel; raise it once instead of on every call
    // (the reference calls cudaFuncSetAttribute per launch, csrc/SpMM_API.cu:36-37).
    if (e == cudaSuccess)
        e = raise_smem_limit<16>(st->smem_optin);
    if (e == cudaSuccess)
        e = raise_smem_limit<32>(st->smem_optin);
    if (e == cudaSuccess)
        e = raise_smem_limit<64>(st->smem_optin);
    if (e == cudaSuccess)
        e = raise_smem_limit<128>(st->smem_optin);
    if (e == cudaSuccess)
        e = raise_smem_limit_of(spmm_tcgen05_wide_kernel<256, kWideCap>, st->smem_optin);
    if (e == cudaSuccess)
        e = raise_smem_limit_of(spmm_tcgen05_wide_kernel<384, kWideCap>, st->smem_optin);
    if (e == cudaSuccess)
        e = raise_smem_limit_of(spmm_tcgen05_wide_kernel<512, kWideCap>, st->smem_optin);
    st->ready = (e == cudaSuccess);
    *err      = e;
    return st->ready ? st : nullptr;
}

int device_status_pointer(unsigned int** status)
{
    cudaError_t  err = cudaSuccess;
    DeviceState* st  = device_state(&err);
    if (!st)
        return static_cast<int>(err);
    *status = st->status;
    return 0;
}

static cudaError_t load_encode_tiled()
{
    std::call_once(g_encode_once, []() {
        void*                           fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) == cudaSuccess
            && qres == cudaDriverEntryPointSuccess)
            g_encode_tiled = reinterpret_cast<EncodeTiledFn>(fn);
        if (cudaGetDriverEntryPoint("cuTensorMapReplaceAddress", &fn, cudaEnableDefault, &qres) == cudaSuccess
            && qres == cudaDriverEntryPointSuccess)
            g_replace_address = reinterpret_cast<ReplaceAddressFn>(fn);
    });
    return g_encode_tiled && g_replace_address ? cudaSuccess : cudaErrorNotSupported;
}

// ---------------------------------------------------------------- launch plan

struct PlanOverride {
    int v[kPlanFieldCount] = {0};
};
static PlanOverride g_override;
static std::mutex   g_override_mutex;
static std::atomic<unsigned> g_override_version{0};  // counts FlashLLM_SetPlan calls
static std::atomic<int> g_launch_overlap{0};


constexpr int kDefaultPath = kPathDirect;
constexpr int kSmemPerSm   = 228 * 1024;  // for all resident CTAs, 1 KB of it each for the system; L1 then keeps 28 KB
constexpr int kSmemForL1   = 196 * 1024;  // the next lower carveout, with 60 KB of L1

static int n_tile_for(int N)
{
    return N <= 16 ? 16 : (N <= 32 ? 32 : (N <= 64 ? 64 : 128));
}

static int plan_smem_bytes(const SpmmPlan& pl)
{
    const int bars = 8 * (2 * pl.ring_slots + 2 * pl.a_stages + 2 * pl.b_stages + 2) + 16 + 4 * pl.offsets_staged;
    return pl.a_stages * kDenseTileBytes + pl.b_stages * pl.b_batch * pl.n_tile * kTileK * 2
           + pl.ring_slots * pl.chunk_vectors * 16 + pl.sum_bytes + bars;
}

static bool is_pow2(int v)
{
    return v > 0 && (v & (v - 1)) == 0;
}

static int stream_smem_bytes(const SpmmPlan& pl)
{
    return kStreamStages * kDenseTileBytes + pl.b_stages * pl.b_batch * pl.n_tile * kTileK * 2
           + 8 * (2 * kStreamStages + 4 + 2 * pl.b_stages) + 16 + kStreamSumBytes + 4 * pl.offsets_staged;
}

// The streaming form: as many CTAs as the GPU holds, fewer only when there are fewer tiles.
static cudaError_t make_stream_plan(const DeviceState* st, SpmmPlan pl, int tile_rows, int k_tiles, int chunk_tiles, SpmmPlan* out)
{
    const long long tiles = static_cast<long long>(tile_rows) * k_tiles;
    long long       ctas  = static_cast<long long>(kStreamCtasPerSm) * st->sm_count;
    ctas                  = ctas < kScratchCtas ? ctas : kScratchCtas;
    ctas                  = ctas < tiles ? ctas : tiles;
    if (pl.n_tile > kScratchMaxN || tile_rows > kScratchRows || tiles > 0x7FFFFFFFll)
        return cudaErrorInvalidConfiguration;
    pl.ctas           = static_cast<int>(ctas);
    pl.chunk_tiles    = chunk_tiles;
    pl.cluster_k      = 1;
    pl.workspace_k    = 1;
    pl.scatter_warps  = kStreamStages;
    pl.a_stages       = kStreamStages;
    pl.producers      = 1;
    pl.reduce         = kReduceLastCta;
    pl.b_batch        = 8192 / (pl.n_tile * kTileK * 2);  // 8 KB per TMA instruction ...
    pl.b_stages       = pl.n_tile <= 32 ? 2 : 3;          // ... and four to eight tiles' worth of B ahead of the MMAs
    const int longest = static_cast<int>((tiles + ctas - 1) / ctas);
    pl.offsets_staged = longest + 1 <= 2048 ? ((longest + 1 + 3) / 4) * 4 : 0;
    pl.smem_bytes     = stream_smem_bytes(pl);
    *out              = pl;
    return cudaSuccess;
}

// Clusters of S CTAs resident at a time on 148 SMs (measured), two CTAs or one per SM.
constexpr int kClustersResident2[kMaxClusterK + 1] = {0, 296, 148, 92, 71, 56, 45, 37, 33};
constexpr int kClustersResident1[kMaxClusterK + 1] = {0, 148, 74, 45, 33, 26, 22, 15, 15};

static long long clusters_resident(const DeviceState* st, const int* table, int s)
{
    const long long c = static_cast<long long>(table[s]) * st->sm_count / 148;
    return c < 1 ? 1ll : c;
}

// What a launch with N <= 64 costs, in us, back to back on one stream, at 80 % sparsity on a B200.  Fitted to 8..288 tile rows (with
// overlap 2..288) by 16..288 K tiles, every cluster size, one to four workspace parts and the streaming form timed at each; what
// the choice then loses to the fastest of them, on average and at most, overlap off: N = 16 0.8 % (12 %; these prices are older
// and the rule about SMs is not), 32 0.3 % (5 %), 64 0.3 % (9 %); on, where CTAs pair up by luck: 0.4 % (9 %), 0.8 % (12 %),
// 1.1 % (15 %).  Over 45 further sizes at 60 to 95 % the calls took 0.892 of the time of one cost for all K cuts.
struct FormCosts {
    double whole, cluster, per_rank;  // fixed part: uncut, in clusters, and what their sum adds for the rows a CTA sums
    double crowded, full;             // more with two CTAs per SM, and when a grid leaves no place for the next one's clusters
    double tile_alone, tile_shared;   // per tile of a CTA with an SM to itself, or not
    double second_kernel;             // of a sum over workspace parts
    double stream, stream_tile, stream_part;
};
static const FormCosts kFormCosts[2][3] = {{{3.3, 4.0, 1.3, 0.35, 0.5, 0.280, 0.46, 2.5, 6.2, 0.450, 0.07},
                                            {3.75, 4.2, 1.7, 1.4, 0.9, 0.305, 0.46, 2.5, 6.9, 0.475, 0.17},
                                            {4.75, 5.6, 2.9, 2.4, 0.8, 0.335, 0.51, 2.5, 8.7, 0.525, 0.47}},
                                           {{2.1, 3.6, 0.0, 0.0, 0.4, 0.330, 0.39, 2.0, 5.2, 0.375, 0.10},
                                            {3.9, 4.9, 0.0, 0.0, 0.9, 0.375, 0.46, 2.4, 6.2, 0.465, 0.17},
                                            {4.0, 7.2, 0.0, 0.0, 0.9, 0.365, 0.48, 2.0, 7.5, 0.495, 0.41}}};

static const FormCosts& form_costs(bool overlap, int n_tile)
{
    return kFormCosts[overlap ? 1 : 0][n_tile == 16 ? 0 : n_tile == 32 ? 1 : 2];
}

// Who has an SM to itself, and with it a tile in 0.3 us instead of 0.45 to 0.5.  The last few clusters of three and more do not
// find their SMs empty (25 of five, of which 148 SMs hold 26, took 17.7 us where 24 take 12.5), but for those of four (33 of 33
// do).  With overlap the next launch's CTAs are there early and pair up: hardly ever up to 32 CTAs, or 48 with a second kernel in
// between, and from 64 on more often than not (8 clusters of eight 0.35 us per tile, 7 of them 0.46: the luck of the launch),
// unless there is one for every SM (148 rows by 144 tiles, N = 16 and 32: 0.31 us per tile, 136 rows 0.48).
static bool sm_to_itself(const DeviceState* st, int ctas_flat, int s, int g, bool overlap)
{
    const long long clusters = static_cast<long long>(ctas_flat) * g, apart = clusters_resident(st, kClustersResident1, s);
    const bool      sparse   = s <= 2 || s == 4 ? clusters <= apart : 100 * clusters <= 93 * apart;
    return sparse && (!overlap || clusters * s <= (g > 1 ? 48 : 32) || (s == 1 && 100 * clusters > 98 * apart));
}

// Hardly a place is left for the clusters of the next launch.
static bool grid_is_full(const DeviceState* st, long long clusters, int s)
{
    return 10 * clusters > 9 * clusters_resident(st, kClustersResident2, s);
}

// One CTA or cluster of S CTAs per tile row (and workspace part).
static double row_form_us(const DeviceState* st, int ctas_flat, int k_tiles, int s, int g, int n_tile, bool overlap)
{
    const FormCosts& f        = form_costs(overlap, n_tile);
    const long long  clusters = static_cast<long long>(ctas_flat) * g;
    const long long  held     = clusters_resident(st, kClustersResident2, s);
    const double     fixed    = s == 1 ? f.whole : f.cluster + f.per_rank / s;
    const double     crowded  = s == 1 ? 0.0 : f.crowded + (grid_is_full(st, clusters, s) ? f.full : 0.0);
    const double     tiles    = static_cast<double>((k_tiles + s * g - 1) / (s * g));
    const double     alone    = fixed + f.tile_alone * tiles;
    const double     shared   = fixed + crowded + f.tile_shared * tiles;
    return (sm_to_itself(st, ctas_flat, s, g, overlap) ? alone : (clusters + held - 1) / held * shared)
           + (g > 1 ? f.second_kernel + 0.1 * g : 0.0);
}

// Most of the matrices that the row form was fitted to stay in L2 from call to call, large ones do not.  One size says how much
// that is, 288 rows by 144 tiles: 75.9 us from DRAM where the prices say 69.5.  Up to 4000 tiles (26 MB) nothing is added.
static double row_form_margin(int tile_rows, int k_tiles)
{
    return static_cast<long long>(tile_rows) * k_tiles < 4000 ? 1.0 : 1.05;
}

// The streaming form: a CTA's tiles, and the parts that the CTA which completes a row adds up.
static double stream_form_us(const SpmmPlan& pl, int tile_rows, int k_tiles, bool overlap)
{
    const FormCosts& f     = form_costs(overlap, pl.n_tile);
    const double     tiles = static_cast<double>(tile_rows) * k_tiles / pl.ctas;
    return f.stream + f.stream_tile * tiles + f.stream_part * (1.0 + static_cast<double>(pl.ctas) / tile_rows);
}

// N >= 256: output columns per CTA, cluster parts S and workspace parts G by the cheapest estimate, in SM cycles; what the
// caller pinned is kept.  A CTA of the wide form takes kTileCycles per tile (by hundreds of columns; 128 columns are the
// register-streaming form, whose own choice follows when that is the cheapest: then cudaErrorInvalidConfiguration), 8000 to
// 14000 around them, 2000 per 128 columns more for a cluster sum; a second kernel costs 5000 and its bytes.  The cycles were
// fitted when 384 columns had 6 + 5 stages.  With the shapes as they are, over six matrices (36864x9216, 18944x9216,
// 9216x9216, 4736x7232, 9472x4096, 2048x8192) at N = 256, 384, 512, 640, 768 against every width at its cheapest S: the choice
// is the fastest or within 5 %, but for N = 384 at 4736x7232 (36.7 us, 384 columns in 3 parts 34.5) and at 9472x4096 (33.1 us,
// 256 columns uncut 29.5).
static cudaError_t make_wide_plan(const DeviceState* st, SpmmPlan pl, const PlanOverride& ov, int tile_rows, int k_tiles, int N,
                                  int max_extra, SpmmPlan* out)
{
    static const int kTileCycles[5] = {0, 600, 780, 1080, 1300};
    double           best = 0.0;
    int              width = 0;  // in 128 columns
    for (int w = 1; w <= 4 && (w - 1) * 128 < N; ++w) {
        if (ov.v[kPlanProducers] && ov.v[kPlanProducers] != w)
            continue;
        const int n_tiles = (N + w * 128 - 1) / (w * 128);
        for (int s = 1; s <= kMaxClusterK && s <= k_tiles; ++s) {
            // the cluster sum parks fp32 [columns][128] over the pipeline buffers
            if ((w == 4 && s > 1) || (ov.v[kPlanClusterK] && ov.v[kPlanClusterK] != s))
                continue;
            const int capacity = kClustersResident1[s] * st->sm_count / 148;
            for (int g = 1; g <= max_extra && g <= 32 && s * g <= k_tiles; ++g) {
                if (ov.v[kPlanWorkspaceK] && ov.v[kPlanWorkspaceK] != g)
                    continue;
                const long long clusters = static_cast<long long>(tile_rows) * n_tiles * g;
                const double    waves    = static_cast<double>((clusters + capacity - 1) / (capacity < 1 ? 1 : capacity));
                const double    per_cta  = static_cast<double>((k_tiles + s * g - 1) / (s * g)) * kTileCycles[w] + 6000.0 + w * 2000.0
                                       + (s > 1 ? w * 2000.0 : 0.0);
                const double cost = waves * per_cta + (g > 1 ? 5000.0 + 0.03 * g * tile_rows * N : 0.0);
                if (width == 0 || cost < best) {
                    width          = w;
                    best           = cost;
                    pl.cluster_k   = s;
                    pl.workspace_k = g;
                }
            }
        }
    }
    if (width < 2)
        return cudaErrorInvalidConfiguration;
    pl.path          = kPathWide;
    pl.reduce        = kReduceSecondKernel;
    pl.n_tile        = width * 128;
    pl.producers     = width;
    pl.a_stages      = wide_a_stages(pl.n_tile);
    pl.scatter_warps = pl.a_stages;
    pl.b_stages      = wide_b_stages(pl.n_tile);
    pl.b_batch       = 1;
    const int buffers = pl.a_stages * kDenseTileBytes + pl.b_stages * wide_mma_n(pl.n_tile) * kTileK * 2;
    const int bars    = 8 * (2 * pl.a_stages + 2 * pl.b_stages + 1) + 16;
    const int longest = (k_tiles + pl.cluster_k * pl.workspace_k - 1) / (pl.cluster_k * pl.workspace_k) + 1;
    const int staged  = ((longest + 1 + 3) / 4) * 4;
    pl.offsets_staged = buffers + bars + 4 * staged <= st->smem_optin ? staged : 0;
    pl.smem_bytes     = buffers + bars + 4 * pl.offsets_staged;
    *out              = pl;
    return cudaSuccess;
}

// Chooses how to cut K and how deep to pipeline.  Takes the place of the reference's per-N switch over
// TilingConfig instances (csrc/SpMM_API.cu:79-118) and of its hand-tuned Split_K tables
// (kernel_benchmark/benchmark.sh:13-15).
// `max_parts`: workspace parts the caller has room for (Split_K / 2 for a caller's Reduction_Workspace, whose Split_K
// fp16 matrices hold half as many fp32 ones).
// `sends`: the call is the sending half of a fused all-reduce, where workspace parts are always summed by the last
// CTA of a tile, which then also stores the sum to every GPU.
// `may_stream`: the call may use the streaming form (the stream's scratch is at hand).
// `parts_fit`: workspace and C are aligned for workspace parts; a plan's are dropped otherwise.
static cudaError_t make_plan(const DeviceState* st, int M, int N, int K, int max_parts, SpmmPlan* out, bool sends = false,
                             bool may_stream = true, bool parts_fit = true)
{
    PlanOverride ov;
    {
        std::lock_guard<std::mutex> lock(g_override_mutex);
        ov = g_override;
    }
    SpmmPlan pl{};
    pl.n_tile           = n_tile_for(N);
    const int tile_rows = M / kTileM;
    const int k_tiles   = K / kTileK;
    const int n_tiles   = (N + pl.n_tile - 1) / pl.n_tile;
    const int ctas_flat = tile_rows * n_tiles;
    const int slab      = pl.n_tile * kTileK * 2;

    // Two pipelines per SM (4 scatter warps, 4 stages each) where they fit; wide-N tiles need the shared memory for
    // their B batches, so they run one deeper pipeline per SM instead.
    pl.path               = ov.v[kPlanPath] ? ov.v[kPlanPath] : kDefaultPath;
    bool pinned           = false;
    for (int v : ov.v)
        pinned |= v != 0;
    if (pl.path == kPathStream)  // pinned: other fields do not apply to it
        return may_stream && !sends ? make_stream_plan(st, pl, tile_rows, k_tiles, (k_tiles + 1) / 2, out)
                                    : cudaErrorInvalidConfiguration;
    if (pl.path == kPathWide || (N >= 256 && !pinned && !sends)) {
        if (N < 256 || N % 128 != 0 || sends)
            return cudaErrorInvalidConfiguration;
        const cudaError_t e = make_wide_plan(st, pl, ov, tile_rows, k_tiles, N, max_parts > 1 ? max_parts : 1, out);
        if (e == cudaSuccess || pl.path == kPathWide)
            return e;
    }
    const bool direct     = pl.path == kPathDirect;
    pl.scatter_warps      = ov.v[kPlanScatterWarps] ? ov.v[kPlanScatterWarps]
                                                    : (direct ? (pl.n_tile <= 64 ? 4 : 8) : (pl.n_tile <= 32 ? 4 : 8));
    const bool two_per_sm = direct ? pl.scatter_warps < 8 : pl.n_tile <= 32;
    pl.producers       = ov.v[kPlanProducers] ? ov.v[kPlanProducers] : 1;
    pl.chunk_vectors   = ov.v[kPlanChunkVectors] ? ov.v[kPlanChunkVectors] : 512;
    pl.ring_slots      = ov.v[kPlanRingSlots] ? ov.v[kPlanRingSlots]
                                              : (two_per_sm ? kMaxTileVectors / pl.chunk_vectors + 1 : 8);
    if (!ov.v[kPlanRingSlots])
        pl.ring_slots = (pl.ring_slots + pl.producers - 1) / pl.producers * pl.producers;
    pl.a_stages        = ov.v[kPlanAStages] ? ov.v[kPlanAStages] : pl.scatter_warps;
    pl.b_batch         = ov.v[kPlanBBatch] ? ov.v[kPlanBBatch] : (4096 / slab > 0 ? 4096 / slab : 1);
    pl.b_stages        = ov.v[kPlanBStages] ? ov.v[kPlanBStages] : 2;
    if (direct) {  // one stage per scatter warp, no copy ring; B batches split evenly between the MMA issuers
        if (!ov.v[kPlanBBatch])
            pl.b_batch = (pl.b_batch + kDirectIssuers - 1) / kDirectIssuers * kDirectIssuers;
        pl.a_stages      = pl.scatter_warps;
        // `producers` of the register-streaming form = warps that share one tile (1, or 2 with four stages)
        pl.producers     = (ov.v[kPlanProducers] == 2 && pl.scatter_warps == 4) ? 2 : 1;
        pl.ring_slots    = 0;
        pl.chunk_vectors = 0;
    }
    // How to cut K.  A CTA that owns a whole tile row needs no reduction and pays its set-up and pipeline fill once,
    // so K is cut only to fill the GPU.  S parts are summed inside a thread-block cluster (distributed shared memory),
    // G parts through fp32 partial tiles in the workspace (summed by the last CTA of a tile to finish, or by a second
    // kernel).  A launch of rows*G clusters of S CTAs runs in ceil(rows*G / capacity(S)) waves, where capacity(S) is
    // the number of clusters of S CTAs the GPU holds at a time -- measured, and well below slots/S for S >= 3 (71
    // clusters of 4, 33 of 8 on 296 slots): one cluster more than that and the launch takes twice as long.  Up to 64
    // columns row_form_us prices a cut.  Elsewhere it is cut by tiles: every CTA processes k_tiles/(S*G) tiles after a
    // fixed cost worth about 16 tiles; a cluster sum costs about 3 more, the sum by the last CTA 2 + 0.1 per part (8 + 0.1
    // per part in a fused all-reduce, where the peers wait for that CTA: measured on 2 GPUs, 9216x1152 ... 9216x18432), a
    // second kernel half a tile per part.  The cheapest (S, G) wins, fewer parts on a tie.  Replaces the reference's
    // hand-tuned Split_K tables (kernel_benchmark/benchmark.sh:13-15).
    const bool two_resident = two_per_sm && ((direct && pl.producers == 1) ? kDirectBlocks : 2) == 2;
    const int* resident     = two_resident ? kClustersResident2 : kClustersResident1;
    const int max_extra = max_parts > 1 ? max_parts : 1;
    // (measured on eleven shapes from 9216x1152 to 9216x36864: with launch overlap the second kernel hides behind its
    // neighbours and beats the sum by the last CTA, which sits on every tile's critical path, by ~2 us per call;
    // without overlap the two are level.  The fused all-reduce always sums by the last CTA: that CTA also sends.)
    pl.reduce           = sends ? kReduceLastCta : (ov.v[kPlanReduce] ? ov.v[kPlanReduce] : kReduceSecondKernel);
    if (ctas_flat > kCounterTiles)
        pl.reduce = kReduceSecondKernel;
    // (Without launch overlap a second kernel used to cost a whole launch, and small problems did better with clusters alone.
    // This rule and the costs in tiles below were fitted before every kernel was launched with programmatic serialisation.)
    const bool overlap   = g_launch_overlap.load(std::memory_order_relaxed) != 0;
    const bool few_tiles = static_cast<long long>(tile_rows) * k_tiles <= 4096 && !overlap;
    // The cut by tiles.
    struct Cut {
        int s, g;
    };
    auto cut_by_tiles = [&](int reduce) {
        Cut    best{1, 1};
        double best_cost = 0.0;
        for (int s_ = 1; s_ <= kMaxClusterK && s_ <= k_tiles; ++s_) {
            for (int g = 1; g <= max_extra && g <= 32 && s_ * g <= k_tiles; ++g) {
                if (g > 1 && reduce == kReduceSecondKernel && few_tiles)
                    break;
                const long long clusters = static_cast<long long>(ctas_flat) * g, capacity = clusters_resident(st, resident, s_);
                const double    waves    = static_cast<double>((clusters + capacity - 1) / capacity);
                const double    per_cta  = static_cast<double>((k_tiles + s_ * g - 1) / (s_ * g)) + 16.0 + (s_ > 1 ? 3.0 : 0.0)
                                        + (g > 1 && reduce == kReduceLastCta ? (sends ? 8.0 : 2.0) + 0.1 * g : 0.0);
                const double cost = waves * per_cta + (g > 1 && reduce == kReduceSecondKernel ? 0.5 * g : 0.0);
                if ((s_ == 1 && g == 1) || cost < best_cost - 1e-9 || (cost < best_cost + 1e-9 && s_ * g < best.s * best.g)) {
                    best_cost = cost;
                    best      = {s_, g};
                }
            }
        }
        return best;
    };
    // It also bounds the sums of every other cut: the tensor core truncates each of its additions, so the error of a sum grows
    // with the tiles added up in one accumulator (measured: 0.7e-7 to 1.4e-7 of the sum per tile of four).  No cut that is
    // cheaper may add up more of them, in four accumulators, than this one in two; and where two of them would hold more than if
    // K were cut into as many parts as fill the GPU, it takes the four.
    auto      in_one_of_two = [&](int parts) { return ((k_tiles + parts - 1) / parts + 1) / 2; };
    const Cut by_tiles      = cut_by_tiles(kReduceSecondKernel);
    const int bound         = in_one_of_two(by_tiles.s * (parts_fit ? by_tiles.g : 1));
    const int fill          = std::min(kStreamCtasPerSm * st->sm_count / tile_rows, kMaxClusterK * max_extra);
    const int full_parts    = std::max(by_tiles.s * by_tiles.g, fill);
    Cut       best          = pl.reduce == kReduceSecondKernel ? by_tiles : cut_by_tiles(pl.reduce);
    // The cut by us, where the row form with two CTAs per SM and the streaming form are the choice.
    const bool priced    = direct && two_resident && pl.n_tile <= kScratchMaxN && !sends;
    double     best_cost = -1.0;
    for (int s_ = 1; priced && s_ <= kMaxClusterK && s_ <= k_tiles; ++s_) {
        for (int g = 1; g <= (parts_fit ? max_extra : 1) && g <= 32 && s_ * g <= k_tiles; ++g) {
            if (g > 1 && pl.reduce == kReduceSecondKernel && few_tiles)
                break;
            const int accumulators = direct_accumulators(pl.n_tile), longest = (k_tiles + s_ * g - 1) / (s_ * g);
            if ((longest + accumulators - 1) / accumulators > bound)
                continue;
            const double cost = row_form_us(st, ctas_flat, k_tiles, s_, g, pl.n_tile, overlap);
            if (best_cost < 0.0 || cost < best_cost) {
                best_cost = cost;
                best      = {s_, g};
            }
        }
    }
    if (may_stream && !pinned && priced) {
        SpmmPlan sp = pl;
        sp.path     = kPathStream;
        // a chunk holds what any of these cuts would put into one of two accumulators
        const int chunk_tiles = in_one_of_two(std::max(full_parts, best.s * best.g));
        if (make_stream_plan(st, sp, tile_rows, k_tiles, chunk_tiles, &sp) == cudaSuccess
            && stream_form_us(sp, tile_rows, k_tiles, overlap) < row_form_margin(tile_rows, k_tiles) * best_cost) {
            *out = sp;
            return cudaSuccess;
        }
    }
    pl.cluster_k = ov.v[kPlanClusterK] ? ov.v[kPlanClusterK] : best.s;
    if (pl.cluster_k > k_tiles)
        pl.cluster_k = k_tiles;
    int extra = ov.v[kPlanWorkspaceK] ? ov.v[kPlanWorkspaceK] : best.g;
    if (extra > max_extra)
        extra = max_extra;  // the workspace is promised to hold Split_K fp16 matrices = Split_K/2 fp32 partials
    if (extra * pl.cluster_k > k_tiles)
        extra = k_tiles / pl.cluster_k;
    if (extra < 1)
        extra = 1;
    pl.workspace_k = extra;
    const int parts = pl.cluster_k * (parts_fit ? extra : 1);
    pl.accumulators = kDirectIssuers;
    if (direct && (k_tiles + parts - 1) / parts > kDirectIssuers * in_one_of_two(full_parts))
        pl.accumulators = direct_accumulators(pl.n_tile);
    // room for this CTA's slice of TileOffsets (K tiles of the longest part, plus one), up to 8 KB
    const int longest = (k_tiles + pl.cluster_k * pl.workspace_k - 1) / (pl.cluster_k * pl.workspace_k) + 1;
    pl.offsets_staged = longest + 1 <= 2048 ? ((longest + 1 + 3) / 4) * 4 : 0;
    // Room of its own for the peers' partial sums where it costs no resident CTA: they may then arrive while this CTA still
    // multiplies.  (Wide outputs take the operands' buffers, once everybody's MMAs are over.)  That saves a call 0.1 to 0.6 us,
    // but an L1 too small for the loads in flight (8 warps x 13 rows of 512 bytes at 80 %) costs every tile: two CTAs of 32
    // columns leave 28 KB with such room and 92 without, and 9216x36864 70 % in clusters of two took 102.5 us instead of 97.8.
    // They have it for short K ranges only; time without it / with it by tiles per CTA (72 x 4 and 148 x 2 CTAs, 65 to 80 %):
    // overlap off 0.98 .. 0.99 at 4, 0.97 at 8, 0.95 at 24; on 1.00 .. 1.04 at 8, 0.96 .. 1.01 at 16, 0.96 .. 0.98 at 24 (92 %:
    // 1.00 .. 1.07).
    // Where large clusters leave no place for the next launch's, a CTA's end counts for more: off, 56 clusters of five 1.04 at 8,
    // 1.07 at 13, 1.02 at 29, 45 of six 1.00, 0.99, 0.96 at 7, 11, 24, 33 of eight 1.02, 1.03, 1.00 at 5, 8, 18.
    // Up to 64 CTAs do not meet the next launch's on an SM, and have the area at any length: 1.00 at 65 and 80 %, 1.02 at 92 %.
    // 64 columns are sent where CTAs have an SM to themselves (kPushMaxN), also from the next launch's (overlap on, sent / parked: 4
    // clusters of eight by 46 tiles 7.2 / 8.4 us, 8 of four by 16 6.8 / 7.6, but 16 of four 9.1 / 8.2, 8 of six 8.7 / 7.4).
    // The fused all-reduce parks: its CTAs then store whole columns of 512 bytes to the other GPUs, not runs of 64.
    pl.push = direct && pl.cluster_k > 1 && pl.n_tile <= kPushMaxN && !sends
              && (pl.n_tile <= 32 || !two_resident
                  || sm_to_itself(st, ctas_flat, pl.cluster_k, extra, overlap));
    if (pl.push) {
        pl.sum_bytes       = cluster_sum_bytes(pl.n_tile, pl.cluster_k);
        const bool full    = pl.cluster_k >= 5 && grid_is_full(st, static_cast<long long>(ctas_flat) * extra, pl.cluster_k);
        const bool short_k = (k_tiles + parts - 1) / parts <= (overlap || full ? 16 : 4) || ctas_flat * extra * pl.cluster_k <= 64;
        const int  room    = two_resident ? (short_k ? kSmemPerSm : kSmemForL1) / 2 - 1024 : st->smem_optin;
        if (plan_smem_bytes(pl) > room)
            pl.sum_bytes = 0;
    }
    pl.smem_bytes     = plan_smem_bytes(pl);

    const bool ring_ok = pl.scatter_warps >= 4 && pl.scatter_warps <= kMaxScatterWarps
                         && pl.producers >= 1 && pl.producers <= kMaxProducers && is_pow2(pl.chunk_vectors)
                         && pl.chunk_vectors >= 64 && pl.ring_slots <= kMaxRingSlots
                         // a slot is always refilled by the same producer warp, and a stage's successive tiles are
                         // taken by groups that cannot be two uses ahead: both keep every mbarrier parity wait within
                         // one phase
                         && pl.ring_slots % pl.producers == 0 && pl.a_stages >= pl.scatter_warps
                         && pl.ring_slots * pl.chunk_vectors >= kMaxTileVectors + pl.chunk_vectors;
    const bool direct_ok = (pl.scatter_warps == 4 || pl.scatter_warps == 8)
                           && pl.a_stages == pl.scatter_warps && pl.b_batch % kDirectIssuers == 0;
    const bool ok = (pl.path == kPathRing || pl.path == kPathDirect) && (direct ? direct_ok : ring_ok)
                    && pl.a_stages >= 1 && pl.a_stages <= kMaxAStages && pl.b_stages >= 1 && pl.b_stages <= kMaxBStages
                    && pl.b_batch >= 1 && pl.b_batch <= 256 && pl.cluster_k >= 1 && pl.cluster_k <= kMaxClusterK
                    && pl.workspace_k >= 1 && (pl.reduce == kReduceSecondKernel || pl.reduce == kReduceLastCta)
                    && pl.smem_bytes <= st->smem_optin
                    // the fp32 partial tiles of the cluster reduction are parked over the pipeline buffers
                    && pl.smem_bytes - 1024 - 4 * pl.offsets_staged >= pl.n_tile * kTileM * 4
                    && (!pl.push || pl.sum_bytes > 0
                        || pl.a_stages * kDenseTileBytes + pl.b_stages * pl.b_batch * slab
                               >= cluster_sum_bytes(pl.n_tile, pl.cluster_k));
    if (!ok)
        return cudaErrorInvalidConfiguration;
    *out = pl;
    return cudaSuccess;
}

// B as a 3-D tensor {64 K-elements (inner), N, K/64}: one box = b_batch K tiles of [n_tile x 64] (wide form: of one MMA's
// columns), each stored as a 128-byte-swizzled slab; rows past N and K tiles past K/64 read as 0.  ldb: halves from one row of
// B to the next.
static cudaError_t encode_b_map(const half* B, int N, int K, int ldb, const SpmmPlan& pl, CUtensorMap* map)
{
    const cuuint64_t dims[3]    = {static_cast<cuuint64_t>(kTileK), static_cast<cuuint64_t>(N), static_cast<cuuint64_t>(K / kTileK)};
    const cuuint64_t strides[2] = {static_cast<cuuint64_t>(ldb) * 2, static_cast<cuuint64_t>(kTileK) * 2};
    const int        columns    = pl.path == kPathWide ? wide_mma_n(pl.n_tile) : pl.n_tile;
    const cuuint32_t box[3]     = {static_cast<cuuint32_t>(kTileK), static_cast<cuuint32_t>(columns),
                                   static_cast<cuuint32_t>(pl.b_batch)};
    const cuuint32_t estr[3]    = {1, 1, 1};
    const CUresult   r = g_encode_tiled(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<half*>(B), dims, strides, box, estr,
                                        CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                        CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS ? cudaSuccess : cudaErrorInvalidValue;
}

// What a call derives from its sizes alone, kept per thread: a decode loop repeats a few dozen calls, and the search over
// K cuts and the tensor map's encoding are 2 us of each, a third of a small call.  The map's address is set on every call.
struct CallKey {
    const DeviceState* device;
    int                M, N, K, ldb, max_parts;
    bool               sends, may_stream, overlap, parts_fit;
    unsigned           override_version;
    bool operator==(const CallKey& o) const
    {
        return device == o.device && M == o.M && N == o.N && K == o.K && ldb == o.ldb && max_parts == o.max_parts && sends == o.sends
               && may_stream == o.may_stream && overlap == o.overlap && parts_fit == o.parts_fit
               && override_version == o.override_version;
    }
};
struct CallMemo {
    CallKey     key{};
    SpmmPlan    plan{};
    bool        has_map = false;
    CUtensorMap map{};
};

static cudaError_t plan_call(const CallKey& key, CallMemo** out)
{
    constexpr unsigned kEntries = 64;
    static thread_local CallMemo memo[kEntries];
    const unsigned hash = (static_cast<unsigned>(key.M) / kTileM * 2654435761u) ^ (static_cast<unsigned>(key.K) / kTileK * 40503u)
                          ^ (static_cast<unsigned>(key.N) * 97u) ^ static_cast<unsigned>(key.max_parts + key.may_stream);
    CallMemo& m = memo[(hash ^ (hash >> 16)) % kEntries];
    if (!(m.key == key)) {
        SpmmPlan          plan{};
        const cudaError_t err = make_plan(key.device, key.M, key.N, key.K, key.max_parts, &plan, key.sends, key.may_stream,
                                          key.parts_fit);
        if (err != cudaSuccess)
            return err;
        m.key     = key;
        m.plan    = plan;
        m.has_map = false;
    }
    *out = &m;
    return cudaSuccess;
}

template<int N_TILE>
static cudaError_t launch_spmm(cudaStream_t stream, const CUtensorMap& tmap, const SpmmParams& params, int tile_rows,
                               int n_tiles)
{
    const SpmmPlan& pl = params.plan;
    const dim3      grid(pl.cluster_k, tile_rows, n_tiles * pl.workspace_k);
    auto            launch = [&](auto kernel, int warps) {
        return launch_in_stream_order(kernel, grid, dim3(warps * 32), pl.smem_bytes, stream, pl.cluster_k, tmap, params);
    };
    if (pl.path == kPathStream) {
        if constexpr (N_TILE <= kScratchMaxN)
            return launch_in_stream_order(spmm_tcgen05_stream_kernel<N_TILE, kStreamCap>, dim3(pl.ctas), dim3(kStreamWarps * 32),
                                          pl.smem_bytes, stream, 1, tmap, params);
        return cudaErrorInvalidConfiguration;
    }
    if (pl.path == kPathDirect) {
        const int warps  = 1 + kDirectIssuers + pl.scatter_warps * pl.producers;
        auto      direct = [&](auto push) {
            if (pl.scatter_warps == 8)
                return launch(spmm_tcgen05_direct_kernel<N_TILE, kDirectCapWide, 8, 1, 1, push>, warps);
            if (pl.producers == 2)
                return launch(spmm_tcgen05_direct_kernel<N_TILE, kDirectCapPair, 4, 2, 2, push>, warps);
            return launch(spmm_tcgen05_direct_kernel<N_TILE, kDirectCapNarrow, 4, kDirectBlocks, 1, push>, warps);
        };
        if constexpr (N_TILE <= kPushMaxN)
            if (pl.push || pl.cluster_k == 1)
                return direct(std::true_type{});
        return direct(std::false_type{});
    }
    return launch(spmm_tcgen05_kernel<N_TILE>, pl.producers + 2 + pl.scatter_warps);
}

template<int N_TILE>
static cudaError_t launch_wide(cudaStream_t stream, const CUtensorMap& tmap, const SpmmParams& params, int tile_rows,
                               int n_tiles)
{
    const SpmmPlan& pl = params.plan;
    return launch_in_stream_order(spmm_tcgen05_wide_kernel<N_TILE, kWideCap>,
                                  dim3(pl.cluster_k, tile_rows, n_tiles * pl.workspace_k),
                                  dim3((kWideFirstScatter + wide_a_stages(N_TILE)) * 32), pl.smem_bytes, stream, pl.cluster_k, tmap,
                                  params);
}

static cudaError_t reduce_partials(cudaStream_t stream, half* C, const float* ws, long long count, int parts,
                                   const half* bias, int M, int activation, const half* residual)
{
    const int       threads = 256;
    const long long groups  = (count + 3) / 4;
    const unsigned  blocks  = static_cast<unsigned>((groups + threads - 1) / threads);
    return launch_in_stream_order(splitk_reduce_f32_kernel, dim3(blocks), dim3(threads), 0, stream, 1, C, ws, count, parts, bias, M,
                                  activation, residual);
}

static cudaError_t reduce_workspace(cudaStream_t stream, half* C, const half* ws, long long count, int parts)
{
    const int       threads = 256;
    const long long groups  = (count + 7) / 8;
    const unsigned  blocks  = static_cast<unsigned>((groups + threads - 1) / threads);
    return launch_in_stream_order(splitk_reduce_kernel, dim3(blocks), dim3(threads), 0, stream, 1, C, ws, count, parts);
}

static bool n_supported(int N)
{
    // the reference's dispatch list (csrc/SpMM_API.cu:79-118)
    return N == 8 || N == 16 || N == 32 || N == 64 || (N > 0 && N % 128 == 0);
}

}  // namespace flashllm

using namespace flashllm;

// Receive buffers of a GPU group for the fused row-parallel SpMM + all-reduce.  Every GPU owns one buffer with two
// sets (used by alternate calls) of `world` fp32 slots [max_elems] and `world` x kCommFlagsPerRank flag words:
//   [set 0 slots][set 1 slots][set 0 flags][set 1 flags][own partial matrices][own arrival counters]
// Slot w / flag row w of a GPU's buffer is written only by GPU w.  While one call's sums are still being read on a
// slow GPU, a fast GPU's next call writes the other set; it cannot start the call after that before the slow GPU has
// taken part in the next one, so two sets are enough.
constexpr int kCommFlagsPerRank = 8192;

struct FlashLLMComm {
    int            rank = 0, world = 0;
    long long      max_elems = 0;
    unsigned char* buffer[kMaxPushWorld] = {nullptr};  // buffer[w]: GPU w's receive buffer as mapped in this process
    unsigned int   epoch = 0;                          // calls made so far; every GPU of the group makes the same calls
    // How long the summing kernel waits for the slowest GPU of the group before it gives up (status bit 32).  The
    // GPUs of a group enter a layer at slightly different times; the limit only has to end a wait for a partner that
    // never comes.
    unsigned long long wait_limit_ns = 2000ull * 1000ull * 1000ull;
};

static size_t comm_slot_bytes(int world, long long max_elems)
{
    return static_cast<size_t>(world) * static_cast<size_t>(max_elems) * sizeof(float);
}

static size_t comm_flag_bytes(int world)
{
    return static_cast<size_t>(world) * kCommFlagsPerRank * sizeof(unsigned int);
}

// ... followed by what only the owning GPU touches: room for kCommLocalParts fp32 partial matrices of its own K
// split, and the arrival counters of that split's in-kernel sum (zero between calls).
constexpr int kCommLocalParts = 8, kCommCounterTiles = 4096;

static size_t comm_buffer_bytes(int world, long long max_elems)
{
    return 2 * comm_slot_bytes(world, max_elems) + 2 * comm_flag_bytes(world)
           + kCommLocalParts * static_cast<size_t>(max_elems) * sizeof(float) + kCommCounterTiles * sizeof(unsigned int);
}

// SpMM_SplitK_API plus the output epilogue (bias of output feature m, activation) the public entry points select.
static cudaError_t spmm_launch_all(cudaStream_t stream,
                                   const uint4* Compressed_A,
                                   const int*   TileOffsets,
                                   const half*  B,
                                   half*        C,
                                   const int    M_Global,
                                   const int    N_Global,
                                   const int    K_Global,
                                   half*        Reduction_Workspace,
                                   int          Split_K,
                                   const half*  bias,
                                   int          activation,
                                   const half*  residual = nullptr,
                                   FlashLLMComm* comm = nullptr,
                                   int           phases = 3,
                                   bool          may_allocate = true,
                                   int           ldb          = 0)  // halves between the rows of B, 0 = K_Global
{
    if (!n_supported(N_Global)) {
        printf("MM_Sparse_API Error: Unsupported N dimension %d!\n", N_Global);
        return cudaErrorUnknown;
    }
    if (M_Global <= 0 || K_Global <= 0 || M_Global % kTileM != 0 || K_Global % kTileK != 0 || Split_K < 1
        || Compressed_A == nullptr || TileOffsets == nullptr || B == nullptr || C == nullptr
        || (reinterpret_cast<uintptr_t>(Compressed_A) & 15u) != 0 || (reinterpret_cast<uintptr_t>(B) & 15u) != 0
        || (ldb != 0 && (ldb < K_Global || ldb % 8 != 0)) || (reinterpret_cast<uintptr_t>(C) & 1u) != 0
        || (Split_K > 1 && Reduction_Workspace == nullptr))
        return cudaErrorInvalidValue;

    cudaError_t  err = cudaSuccess;
    DeviceState* st  = device_state(&err);
    if (!st)
        return err;
    if ((err = load_encode_tiled()) != cudaSuccess)
        return err;

    SpmmParams params{};
    SpmmPlan&  pl = params.plan;
    // The sum over workspace parts reads 16-byte groups of the workspace and writes 8-byte groups of C.
    const bool parts_fit = comm != nullptr || Split_K < 4 || ((reinterpret_cast<uintptr_t>(Reduction_Workspace) & 15u) == 0
                                                              && (reinterpret_cast<uintptr_t>(C) & 7u) == 0);
    CallKey    key{st,           M_Global,     N_Global, K_Global, ldb ? ldb : K_Global, comm ? kCommLocalParts : Split_K / 2,
                comm != nullptr, may_allocate, g_launch_overlap.load(std::memory_order_relaxed) != 0, parts_fit,
                g_override_version.load(std::memory_order_relaxed)};
    CallMemo*  memo = nullptr;
    if ((err = plan_call(key, &memo)) != cudaSuccess)
        return err;
    if (memo->plan.path == kPathStream) {
        unsigned char* scratch = scratch_of_stream(st, stream);
        if (scratch != nullptr) {
            params.tile_counters = reinterpret_cast<unsigned int*>(scratch);
            params.partial       = reinterpret_cast<float*>(scratch + kScratchRows * sizeof(unsigned int));
        }
        else {
            key.may_stream = false;
            if ((err = plan_call(key, &memo)) != cudaSuccess)
                return err;
        }
    }
    pl = memo->plan;
    if (!parts_fit)
        pl.workspace_k = 1;

    params.compressed   = Compressed_A;
    params.tile_offsets = TileOffsets;
    params.out          = C;
    if (pl.workspace_k > 1)
        params.partial = reinterpret_cast<float*>(Reduction_Workspace);
    if (!comm && pl.workspace_k > 1 && pl.reduce == kReduceLastCta) {
        params.tile_counters = counters_of_stream(st, stream);
        if (params.tile_counters == nullptr)
            pl.reduce = kReduceSecondKernel;  // every counter set belongs to another stream
    }
    params.status       = st->status;
    params.bias         = bias;
    params.activation   = activation;
    params.early_weights = g_launch_overlap.load(std::memory_order_relaxed);
    params.residual     = residual;
    params.M            = M_Global;
    params.N            = N_Global;
    params.K            = K_Global;
    params.k_tiles      = K_Global / kTileK;
    if (pl.path == kPathStream) {
        const unsigned long long tiles = static_cast<unsigned long long>(M_Global / kTileM) * params.k_tiles;
        params.stream_share            = ((tiles << 32) + pl.ctas - 1) / pl.ctas;
        params.ctas_per_tile           = static_cast<float>(static_cast<double>(pl.ctas) / static_cast<double>(tiles));
    }

    if (memo->has_map) {
        if (g_replace_address(&memo->map, const_cast<half*>(B)) != CUDA_SUCCESS)
            return cudaErrorInvalidValue;
    }
    else {
        if ((err = encode_b_map(B, N_Global, K_Global, key.ldb, pl, &memo->map)) != cudaSuccess)
            return err;
        memo->has_map = true;
    }
    const CUtensorMap& tmap = memo->map;

    const int tile_rows = M_Global / kTileM;
    const int n_tiles   = (N_Global + pl.n_tile - 1) / pl.n_tile;
    const int grid_ctas = pl.cluster_k * tile_rows * n_tiles * pl.workspace_k;
    // flags a sender raises per call: one per CTA, or one per output tile when the last CTA of a tile sends its sum
    const int comm_flags = pl.workspace_k > 1 ? tile_rows * n_tiles : grid_ctas;
    size_t    set_slots = 0, set_flags = 0;
    if (comm) {
        const long long elems = static_cast<long long>(M_Global) * N_Global;
        if (elems > comm->max_elems || elems % 4 != 0 || comm_flags > kCommFlagsPerRank
            || (pl.workspace_k > 1 && tile_rows * n_tiles > kCommCounterTiles) || (reinterpret_cast<uintptr_t>(C) & 7u) != 0)
            return cudaErrorInvalidValue;
        if (pl.workspace_k > 1) {  // own K split: parts parked in the own buffer, summed and sent by the last CTA
            unsigned char* own   = comm->buffer[comm->rank] + 2 * comm_slot_bytes(comm->world, comm->max_elems)
                                 + 2 * comm_flag_bytes(comm->world);
            pl.reduce            = kReduceLastCta;
            params.partial       = reinterpret_cast<float*>(own);
            params.tile_counters = reinterpret_cast<unsigned int*>(own + kCommLocalParts * static_cast<size_t>(comm->max_elems)
                                                                                 * sizeof(float));
        }
        if (phases & 1)
            comm->epoch += 1;  // a new call; a sum-only call belongs to the call whose stores went out last
        const int set       = static_cast<int>(comm->epoch & 1u);
        set_slots           = static_cast<size_t>(set) * comm_slot_bytes(comm->world, comm->max_elems);
        set_flags           = 2 * comm_slot_bytes(comm->world, comm->max_elems)
                    + static_cast<size_t>(set) * comm_flag_bytes(comm->world);
        params.push_world   = comm->world;
        params.push_epoch   = comm->epoch;
        for (int w = 0; w < comm->world; ++w) {
            params.push_slot[w] = reinterpret_cast<float*>(comm->buffer[w] + set_slots) + comm->rank * comm->max_elems;
            params.push_flag[w] = reinterpret_cast<unsigned int*>(comm->buffer[w] + set_flags) + comm->rank * kCommFlagsPerRank;
        }
    }
    if (!comm || (phases & 1)) {
        switch (pl.n_tile) {
            case 16: err = launch_spmm<16>(stream, tmap, params, tile_rows, n_tiles); break;
            case 32: err = launch_spmm<32>(stream, tmap, params, tile_rows, n_tiles); break;
            case 64: err = launch_spmm<64>(stream, tmap, params, tile_rows, n_tiles); break;
            case 256: err = launch_wide<256>(stream, tmap, params, tile_rows, n_tiles); break;
            case 384: err = launch_wide<384>(stream, tmap, params, tile_rows, n_tiles); break;
            case 512: err = launch_wide<512>(stream, tmap, params, tile_rows, n_tiles); break;
            default: err = launch_spmm<128>(stream, tmap, params, tile_rows, n_tiles); break;
        }
        if (err != cudaSuccess)
            return err;
    }
    if (comm && !(phases & 2))
        return cudaSuccess;
    if (comm) {
        // second kernel: waits (bounded) for every GPU's flags of this call, then adds the slots up in rank order
        const long long     count   = static_cast<long long>(M_Global) * N_Global;
        const int           threads = 256;
        const unsigned      blocks  = static_cast<unsigned>((count / 4 + threads - 1) / threads);
        cudaLaunchConfig_t  cfg{};
        cudaLaunchAttribute attr[1];
        cfg.gridDim  = dim3(blocks, 1, 1);
        cfg.blockDim = dim3(threads, 1, 1);
        cfg.stream   = stream;
        if (g_launch_overlap.load(std::memory_order_relaxed)) {
            attr[0].id                                         = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs                                          = attr;
            cfg.numAttrs                                       = 1;
        }
        unsigned char* mine = comm->buffer[comm->rank];
        count_launch();
        return cudaLaunchKernelEx(&cfg, allreduce_sum_kernel, C, reinterpret_cast<const float*>(mine + set_slots),
                                  comm->max_elems, reinterpret_cast<const unsigned int*>(mine + set_flags), kCommFlagsPerRank,
                                  comm->epoch, comm->world, pl.workspace_k > 1 ? 1 : pl.cluster_k, tile_rows, pl.n_tile, count, bias,
                                  M_Global, activation, residual, st->status, comm->wait_limit_ns, phases == 3 ? 0 : 1);
    }
    if (pl.workspace_k > 1 && pl.reduce == kReduceSecondKernel)
        return reduce_partials(stream, C, params.partial, static_cast<long long>(M_Global) * N_Global, pl.workspace_k,
                               bias, M_Global, activation, residual);
    return cudaSuccess;
}

cudaError_t SpMM_SplitK_API(cudaStream_t stream,
                            const half*  A,
                            const uint4* Compressed_A,
                            const int*   TileOffsets,
                            const half*  B,
                            half*        C,
                            const int    M_Global,
                            const int    N_Global,
                            const int    K_Global,
                            half*        Reduction_Workspace,
                            int          Split_K)
{
    (void)A;  // kept for signature compatibility; callers pass nullptr
    return spmm_launch_all(stream, Compressed_A, TileOffsets, B, C, M_Global, N_Global, K_Global, Reduction_Workspace,
                           Split_K, nullptr, kActNone);
}

extern "C" {

int FlashLLM_SpMM_SplitK_BiasAct(void*       stream,
                                 const void* Compressed_A,
                                 const int*  TileOffsets,
                                 const void* B,
                                 void*       C,
                                 int         M,
                                 int         N,
                                 int         K,
                                 void*       Reduction_Workspace,
                                 int         Split_K,
                                 const void* bias,
                                 int         activation)
{
    if (activation != kActNone && activation != kActRelu)
        return static_cast<int>(cudaErrorInvalidValue);
    return static_cast<int>(spmm_launch_all(static_cast<cudaStream_t>(stream), static_cast<const uint4*>(Compressed_A),
                                            TileOffsets, static_cast<const half*>(B), static_cast<half*>(C), M, N, K,
                                            static_cast<half*>(Reduction_Workspace), Split_K,
                                            static_cast<const half*>(bias), activation));
}

int FlashLLM_SpMM_SplitK_Epilogue(void*       stream,
                                  const void* Compressed_A,
                                  const int*  TileOffsets,
                                  const void* B,
                                  void*       C,
                                  int         M,
                                  int         N,
                                  int         K,
                                  void*       Reduction_Workspace,
                                  int         Split_K,
                                  const void* bias,
                                  int         activation,
                                  const void* residual)
{
    if ((activation != kActNone && activation != kActRelu) || (residual != nullptr && residual == C))
        return static_cast<int>(cudaErrorInvalidValue);
    return static_cast<int>(spmm_launch_all(static_cast<cudaStream_t>(stream), static_cast<const uint4*>(Compressed_A),
                                            TileOffsets, static_cast<const half*>(B), static_cast<half*>(C), M, N, K,
                                            static_cast<half*>(Reduction_Workspace), Split_K,
                                            static_cast<const half*>(bias), activation,
                                            static_cast<const half*>(residual)));
}

int FlashLLM_SpMM_SplitK_Strided(void*       stream,
                                 const void* Compressed_A,
                                 const int*  TileOffsets,
                                 const void* B,
                                 int         ldb,
                                 void*       C,
                                 int         M,
                                 int         N,
                                 int         K,
                                 void*       Reduction_Workspace,
                                 int         Split_K,
                                 const void* bias,
                                 int         activation,
                                 const void* residual)
{
    if ((activation != kActNone && activation != kActRelu) || (residual != nullptr && residual == C) || ldb <= 0)
        return static_cast<int>(cudaErrorInvalidValue);
    return static_cast<int>(spmm_launch_all(static_cast<cudaStream_t>(stream), static_cast<const uint4*>(Compressed_A),
                                            TileOffsets, static_cast<const half*>(B), static_cast<half*>(C), M, N, K,
                                            static_cast<half*>(Reduction_Workspace), Split_K, static_cast<const half*>(bias),
                                            activation, static_cast<const half*>(residual), nullptr, 3, true, ldb));
}

int FlashLLM_SpMM_SplitK(void*       stream,
                         const void* A,
                         const void* Compressed_A,
                         const int*  TileOffsets,
                         const void* B,
                         void*       C,
                         int         M,
                         int         N,
                         int         K,
                         void*       Reduction_Workspace,
                         int         Split_K)
{
    return static_cast<int>(SpMM_SplitK_API(static_cast<cudaStream_t>(stream),
                                            static_cast<const half*>(A),
                                            static_cast<const uint4*>(Compressed_A),
                                            TileOffsets,
                                            static_cast<const half*>(B),
                                            static_cast<half*>(C),
                                            M,
                                            N,
                                            K,
                                            static_cast<half*>(Reduction_Workspace),
                                            Split_K));
}

int FlashLLM_SpMM_SplitK_NoAlloc(void*       stream,
                                 const void* Compressed_A,
                                 const int*  TileOffsets,
                                 const void* B,
                                 void*       C,
                                 int         M,
                                 int         N,
                                 int         K,
                                 int         Split_K)
{
    if (M <= 0 || N <= 0 || K <= 0 || Split_K < 1)
        return static_cast<int>(cudaErrorInvalidValue);
    // Split_K fp16 matrices, the room a caller-owned workspace would have; Split_K = 1 never touches the scratch
    const unsigned long long need = Split_K > 1 ? 2ull * static_cast<unsigned long long>(Split_K) * M * N : 0ull;
    if (need > kNoAllocScratchBytes) {
        fprintf(stderr,
                "FlashLLM_SpMM_SplitK_NoAlloc: Split_K*M*N*2 = %llu bytes exceeds the built-in %zu-byte scratch; lower "
                "Split_K (Split_K = 1 needs no scratch and is accepted at any size) or use FlashLLM_SpMM_SplitK with a "
                "workspace of your own.\n",
                need, kNoAllocScratchBytes);
        return static_cast<int>(cudaErrorInvalidValue);
    }
    cudaError_t  err = cudaSuccess;
    DeviceState* st  = device_state(&err);  // first call on a device: looks the scratch address up, allocates nothing
    if (!st)
        return static_cast<int>(err);
    return static_cast<int>(spmm_launch_all(static_cast<cudaStream_t>(stream), static_cast<const uint4*>(Compressed_A),
                                            TileOffsets, static_cast<const half*>(B), static_cast<half*>(C), M, N, K,
                                            reinterpret_cast<half*>(st->noalloc_scratch), Split_K, nullptr, kActNone, nullptr,
                                            nullptr, 3, false));
}

unsigned long long FlashLLM_Comm_BufferBytes(int world, long long max_elems)
{
    if (world < 1 || world > kMaxPushWorld || max_elems < 4)
        return 0;
    return comm_buffer_bytes(world, max_elems);
}

int FlashLLM_Comm_AllocBuffer(int world, long long max_elems, void** buffer, void* ipc_handle)
{
    if (buffer == nullptr || world < 1 || world > kMaxPushWorld || max_elems < 4 || max_elems % 4 != 0)
        return static_cast<int>(cudaErrorInvalidValue);
    const size_t bytes = comm_buffer_bytes(world, max_elems);
    cudaError_t  e     = cudaMalloc(buffer, bytes);
    if (e == cudaSuccess)
        e = cudaMemset(*buffer, 0, bytes);  // flags start below every epoch
    if (e == cudaSuccess && ipc_handle != nullptr)
        e = cudaIpcGetMemHandle(static_cast<cudaIpcMemHandle_t*>(ipc_handle), *buffer);
    if (e == cudaSuccess)
        e = cudaDeviceSynchronize();
    return static_cast<int>(e);
}

int FlashLLM_Comm_OpenPeerBuffer(const void* ipc_handle, void** buffer)
{
    if (ipc_handle == nullptr || buffer == nullptr)
        return static_cast<int>(cudaErrorInvalidValue);
    return static_cast<int>(cudaIpcOpenMemHandle(buffer, *static_cast<const cudaIpcMemHandle_t*>(ipc_handle),
                                                 cudaIpcMemLazyEnablePeerAccess));
}

int FlashLLM_Comm_ClosePeerBuffer(void* buffer)
{
    return static_cast<int>(cudaIpcCloseMemHandle(buffer));
}

int FlashLLM_Comm_FreeBuffer(void* buffer)
{
    return static_cast<int>(cudaFree(buffer));
}

int FlashLLM_Comm_Create(void** comm, int rank, int world, long long max_elems, void* const* buffers)
{
    if (comm == nullptr || buffers == nullptr || world < 1 || world > kMaxPushWorld || rank < 0 || rank >= world
        || max_elems < 4 || max_elems % 4 != 0)
        return static_cast<int>(cudaErrorInvalidValue);
    for (int w = 0; w < world; ++w)
        if (buffers[w] == nullptr || (reinterpret_cast<uintptr_t>(buffers[w]) & 15u) != 0)
            return static_cast<int>(cudaErrorInvalidValue);
    FlashLLMComm* c = new (std::nothrow) FlashLLMComm();
    if (c == nullptr)
        return static_cast<int>(cudaErrorMemoryAllocation);
    c->rank      = rank;
    c->world     = world;
    c->max_elems = max_elems;
    for (int w = 0; w < world; ++w)
        c->buffer[w] = static_cast<unsigned char*>(buffers[w]);
    *comm = c;
    return 0;
}

int FlashLLM_Comm_SetWaitLimit(void* comm, int milliseconds)
{
    if (comm == nullptr || milliseconds < 1 || milliseconds > 60000)
        return static_cast<int>(cudaErrorInvalidValue);
    static_cast<FlashLLMComm*>(comm)->wait_limit_ns = static_cast<unsigned long long>(milliseconds) * 1000000ull;
    return 0;
}

int FlashLLM_Comm_Destroy(void* comm)
{
    delete static_cast<FlashLLMComm*>(comm);
    return 0;
}

int FlashLLM_SpMM_SplitK_AllReduce(void*       comm,
                                   void*       stream,
                                   const void* Compressed_A,
                                   const int*  TileOffsets,
                                   const void* B,
                                   void*       C,
                                   int         M,
                                   int         N,
                                   int         K,
                                   const void* bias,
                                   int         activation,
                                   const void* residual,
                                   int         phases)
{
    if (comm == nullptr || (activation != kActNone && activation != kActRelu) || phases < 1 || phases > 3
        || (residual != nullptr && residual == C))
        return static_cast<int>(cudaErrorInvalidValue);
    return static_cast<int>(spmm_launch_all(static_cast<cudaStream_t>(stream), static_cast<const uint4*>(Compressed_A),
                                            TileOffsets, static_cast<const half*>(B), static_cast<half*>(C), M, N, K,
                                            nullptr, 1, static_cast<const half*>(bias), activation,
                                            static_cast<const half*>(residual), static_cast<FlashLLMComm*>(comm), phases));
}

int FlashLLM_SplitK_Reduction(void* stream, void* C, const void* Reduction_Workspace, int M, int N, int Split_K)
{
    const long long count = static_cast<long long>(M) * N;
    if (C == nullptr || Reduction_Workspace == nullptr || M <= 0 || N <= 0 || Split_K < 1 || count % 8 != 0
        || (reinterpret_cast<uintptr_t>(C) & 15u) != 0 || (reinterpret_cast<uintptr_t>(Reduction_Workspace) & 15u) != 0)
        return static_cast<int>(cudaErrorInvalidValue);
    return static_cast<int>(reduce_workspace(static_cast<cudaStream_t>(stream), static_cast<half*>(C),
                                             static_cast<const half*>(Reduction_Workspace), count, Split_K));
}

int FlashLLM_ReleaseScratch(void)
{
    cudaError_t  err = cudaSuccess;
    DeviceState* st  = device_state(&err);
    if (!st)
        return static_cast<int>(err);
    if ((err = cudaDeviceSynchronize()) != cudaSuccess)
        return static_cast<int>(err);
    std::lock_guard<std::mutex> lock(st->mutex);
    for (StreamScratch& place : st->scratch) {
        cudaFree(place.memory);
        place = StreamScratch();
    }
    st->scratch_retry = 0;
    return 0;
}

int FlashLLM_ReleaseStreamScratch(void* stream)
{
    cudaError_t  err = cudaSuccess;
    DeviceState* st  = device_state(&err);
    if (!st)
        return static_cast<int>(err);
    const cudaStream_t s  = static_cast<cudaStream_t>(stream);
    unsigned long long id = 0;
    if ((err = cudaStreamGetId(s, &id)) != cudaSuccess || (err = cudaStreamSynchronize(s)) != cudaSuccess)
        return static_cast<int>(err);
    std::lock_guard<std::mutex> lock(st->mutex);
    if (StreamScratch* place = scratch_with_id(st, id))
        place->taken = false;
    return 0;
}

void FlashLLM_SetLaunchOverlap(int enable)
{
    g_launch_overlap.store(enable ? 1 : 0, std::memory_order_relaxed);
}

void FlashLLM_SetPlan(const int* fields, int count)
{
    std::lock_guard<std::mutex> lock(g_override_mutex);
    for (int i = 0; i < kPlanFieldCount; ++i)
        g_override.v[i] = (fields != nullptr && i < count) ? fields[i] : 0;
    g_override_version.fetch_add(1, std::memory_order_relaxed);
}

int FlashLLM_GetPlan(int M, int N, int K, int Split_K, int* out, int count)
{
    if (out == nullptr || !n_supported(N) || M <= 0 || K <= 0 || M % kTileM != 0 || K % kTileK != 0 || Split_K < 1)
        return static_cast<int>(cudaErrorInvalidValue);
    cudaError_t  err = cudaSuccess;
    DeviceState* st  = device_state(&err);
    if (!st)
        return static_cast<int>(err);
    SpmmPlan pl{};
    if ((err = make_plan(st, M, N, K, Split_K / 2, &pl)) != cudaSuccess)
        return static_cast<int>(err);
    const int values[kPlanFieldCount + 1] = {pl.cluster_k,  pl.workspace_k,   pl.a_stages,      pl.b_stages,  pl.b_batch,
                                             pl.ring_slots, pl.chunk_vectors, pl.scatter_warps, pl.producers, pl.path,
                                             pl.reduce,     pl.smem_bytes};
    for (int i = 0; i < count && i <= kPlanFieldCount; ++i)
        out[i] = values[i];
    return 0;
}

unsigned int FlashLLM_ConsumeStatus(void)
{
    cudaError_t  err = cudaSuccess;
    DeviceState* st  = device_state(&err);
    if (!st)
        return 0x80000000u;
    unsigned int value = 0;
    if (cudaDeviceSynchronize() != cudaSuccess)
        return 0x80000000u;
    if (cudaMemcpy(&value, st->status, sizeof(value), cudaMemcpyDeviceToHost) != cudaSuccess)
        return 0x80000000u;
    if (value != 0)
        cudaMemset(st->status, 0, sizeof(value));
    return value;
}

#ifdef FLASHLLM_CTA_TIMES
// Launch-shape builds only: copies the per-CTA stamps (4 per CTA, up to 4096 CTAs) to the host.
int FlashLLM_DebugCtaTimes(unsigned long long* out, int count)
{
    cudaDeviceSynchronize();
    return static_cast<int>(cudaMemcpyFromSymbol(out, flashllm::g_cta_times, sizeof(unsigned long long) * count));
}
#endif

#ifdef FLASHLLM_TRACE
// Timeline builds only: copies the recorded timestamps (kinds x depth) to the host.
int FlashLLM_DebugTrace(long long* out, int count)
{
    cudaDeviceSynchronize();
    return static_cast<int>(cudaMemcpyFromSymbol(out, flashllm::g_trace, sizeof(long long) * count));
}
#endif

unsigned long long FlashLLM_LaunchCount(void)
{
    return g_launches.load(std::memory_order_relaxed);
}

}  // extern "C"
