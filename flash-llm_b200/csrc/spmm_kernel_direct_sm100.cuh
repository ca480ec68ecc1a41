// Load-as-Sparse / Compute-as-Dense SpMM for sm_100a, register-streaming form.
//
// Same work, roles of the B loader, MMA issuer and epilogue, K split and bounded waits as spmm_tcgen05_kernel, but
// the compressed words never pass through shared memory as a stream:
//
//   * Every scatter warp owns one 16 KB stage and takes every NSW-th tile of the CTA's K range.  It fetches the words
//     of its NEXT tile straight from global memory into registers (ld.global, 16 bytes per lane and instruction,
//     the reference's LDG.128 scheme, csrc/SpMM_Kernel.cuh:17-62) right after it has published the current one, so
//     a whole hand-back period of the stage (several microseconds) hides the memory latency, and as many tiles as
//     there are scatter warps are in flight per CTA.  No copy ring, no producer warps, no per-chunk barriers.
//   * A stage is cleared with 32 16-byte stores per lane: clearing only the cells the previous tile wrote (their
//     locations kept in registers) takes more, and slower, store instructions and measured slower.  Tiles with more vectors than the register budget (CAP per lane) fetch and scatter
//     the excess in a plain loop.
#pragma once
#include "spmm_kernel_sm100.cuh"

namespace flashllm {

// Warp-collective bounded wait: every lane probes (the probe parks the warp for a while), one answer for all lanes.
__device__ __forceinline__ bool
wait_bounded_converged(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status)
{
    if (ptx::mbar_try_wait(bar, parity))
        return true;
    uint64_t t0 = 0;
    bool     ok = true;
    for (uint32_t it = 1; ok && !ptx::mbar_try_wait(bar, parity); ++it) {
        if ((it & 255u) == 0u) {
            if (*abort_flag)
                ok = false;
            else if (abort_flag[kDepsResolved] == 0u)  // still behind the previous kernel of the stream: no clock yet
                t0 = 0;
            else {
                const uint64_t now = ptx::globaltimer_ns();
                if (t0 == 0)
                    t0 = now;
                else if (now - t0 > kWaitLimitNs) {
                    *abort_flag = 1u;
                    atomicOr(status, kStatusWaitExpired);
                    ok = false;
                }
            }
        }
    }
    return ok;
}

// Warp-collective bounded wait for what the CTAs of the cluster store here: every lane probes (the probe parks the warp for a
// while).  A peer that is late is late by its own bounded waits, so the clock runs twice as long.  A CTA that gave up
// on the way sends what it has, so that its peers' waits end.
__device__ __forceinline__ bool
wait_bounded_cluster(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, unsigned int* status)
{
    uint64_t t0 = 0;
    for (uint32_t it = 1; !ptx::mbar_try_wait_cluster(bar, parity); ++it) {
        if ((it & 255u) == 0u) {
            const uint64_t now = ptx::globaltimer_ns();
            if (t0 == 0)
                t0 = now;
            else if (now - t0 > 2 * kWaitLimitNs) {
                *abort_flag = 1u;
                atomicOr(status, kStatusWaitExpired);
                return false;
            }
        }
    }
    return true;
}

// Words are read once, so they get no line of L1; not through the read-only path (ld.global.nc): a kernel is launched before
// its predecessors have ended, and that path is for data that nobody writes in a kernel's lifetime.
#ifndef FLASHLLM_LDG_FLAVOUR
#define FLASHLLM_LDG_FLAVOUR "ld.global.L1::no_allocate.v4.u32"
#endif

// Straight-line forms for the scatter warps' per-tile path.  That path is bound by the number of instructions and
// branches a warp has to get through per tile, so a row of 32 vectors is loaded / scattered by predicated instructions
// behind ONE comparison (`rem` = vectors of the tile from this lane's first one on, against the row's constant offset)
// instead of being guarded by branches, and row addresses are one base register plus a constant.
template<int VEC_OFFSET>
__device__ __forceinline__ void ldg_row_if(uint4& v, const uint4* lane_base, int rem)
{
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.gt.s32 p, %5, %6;\n"
        "@p " FLASHLLM_LDG_FLAVOUR " {%0, %1, %2, %3}, [%4 + %7];\n"
        "}\n"
        : "+r"(v.x), "+r"(v.y), "+r"(v.z), "+r"(v.w)
        : "l"(lane_base), "r"(rem), "n"(VEC_OFFSET), "n"(VEC_OFFSET * 16));
}

template<int VEC_OFFSET>
__device__ __forceinline__ void scatter_row_if(uint32_t stage, const uint4& w, int rem)
{
    const uint32_t a0 = stage + ((w.x >> 15) & 0x3FFEu), a1 = stage + ((w.y >> 15) & 0x3FFEu);
    const uint32_t a2 = stage + ((w.z >> 15) & 0x3FFEu), a3 = stage + ((w.w >> 15) & 0x3FFEu);
#if (FLASHLLM_ABLATE & 32)  // timing only: whole-word stores in place of the 16-bit ones (neighbours get clobbered)
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.gt.s32 p, %8, %9;\n"
        "@p st.shared.u32 [%0], %4;\n"
        "@p st.shared.u32 [%1], %5;\n"
        "@p st.shared.u32 [%2], %6;\n"
        "@p st.shared.u32 [%3], %7;\n"
        "}\n" ::"r"(a0 & ~3u),
        "r"(a1 & ~3u), "r"(a2 & ~3u), "r"(a3 & ~3u), "r"(w.x << 16), "r"(w.y << 16), "r"(w.z << 16), "r"(w.w << 16), "r"(rem),
        "n"(VEC_OFFSET)
        : "memory");
    return;
#endif
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.gt.s32 p, %8, %9;\n"
        "@p st.shared.u16 [%0], %4;\n"
        "@p st.shared.u16 [%1], %5;\n"
        "@p st.shared.u16 [%2], %6;\n"
        "@p st.shared.u16 [%3], %7;\n"
        "}\n" ::"r"(a0),
        "r"(a1), "r"(a2), "r"(a3), "h"(static_cast<unsigned short>(w.x & 0xFFFFu)),
        "h"(static_cast<unsigned short>(w.y & 0xFFFFu)), "h"(static_cast<unsigned short>(w.z & 0xFFFFu)),
        "h"(static_cast<unsigned short>(w.w & 0xFFFFu)), "r"(rem), "n"(VEC_OFFSET)
        : "memory");
}

// Rows [FIRST, LAST) of a warp's share of a tile: the warp's row q is the tile's row q * WPT + its index among the
// WPT warps that share the tile (already folded into lane_base and rem).
template<int FIRST, int LAST, int WPT, int CAP>
__device__ __forceinline__ void load_rows(uint4 (&buf)[CAP], const uint4* lane_base, int rem)
{
    if constexpr (FIRST < LAST) {
        ldg_row_if<FIRST * WPT * 32>(buf[FIRST], lane_base, rem);
        load_rows<FIRST + 1, LAST, WPT, CAP>(buf, lane_base, rem);
    }
}

template<int FIRST, int LAST, int WPT, int CAP>
__device__ __forceinline__ void scatter_rows(uint32_t stage, const uint4 (&buf)[CAP], int rem)
{
    if constexpr (FIRST < LAST) {
        scatter_row_if<FIRST * WPT * 32>(stage, buf[FIRST], rem);
        scatter_rows<FIRST + 1, LAST, WPT, CAP>(stage, buf, rem);
    }
}

// A warp's batch of up to CAP rows: the lower half always, the upper half only when the tile reaches it (one branch),
// so that sparse tiles do not pay for rows they do not have.
template<int WPT, int CAP>
__device__ __forceinline__ void load_batch(uint4 (&buf)[CAP], const uint4* lane_base, int rem_uniform, int rem)
{
    load_rows<0, CAP / 2, WPT, CAP>(buf, lane_base, rem);
    if (rem_uniform > (CAP / 2) * WPT * 32)
        load_rows<CAP / 2, CAP, WPT, CAP>(buf, lane_base, rem);
}

template<int WPT, int CAP>
__device__ __forceinline__ void scatter_batch(uint32_t stage, const uint4 (&buf)[CAP], int rem_uniform, int rem)
{
    scatter_rows<0, CAP / 2, WPT, CAP>(stage, buf, rem);
    if (rem_uniform > (CAP / 2) * WPT * 32)
        scatter_rows<CAP / 2, CAP, WPT, CAP>(stage, buf, rem);
}

// Scatters a warp's share of a tile of n_in vectors whose first CAP rows are in buf.  Rows beyond them are fetched half a
// batch at a time into the registers just emptied, so that their latency hides behind the other half's stores
// (9216x36864 N = 32 at 70 %, 614 vectors a tile: 110.0 -> 107.3 us; 2048x32768 N = 16 at 70 %: 27.8 -> 26.9).
template<int WPT, int CAP>
__device__ __forceinline__ void scatter_tile(uint32_t stage, uint4 (&buf)[CAP], const uint4* lane_base, int n_in, int rem)
{
    constexpr int H = CAP / 2, V = H * WPT * 32;  // rows and vectors of half a batch
    if (n_in <= 2 * V) {
        scatter_batch<WPT, CAP>(stage, buf, n_in, rem);
        return;
    }
    for (int v0 = 0;; v0 += 2 * V) {
        scatter_rows<0, H, WPT, CAP>(stage, buf, rem - v0);
        if (n_in > v0 + 2 * V)
            load_rows<0, H, WPT, CAP>(buf, lane_base + v0 + 2 * V, rem - v0 - 2 * V);
        if (n_in <= v0 + V)
            break;
        scatter_rows<H, CAP, WPT, CAP>(stage, buf, rem - v0);
        if (n_in > v0 + 3 * V)
            load_rows<H, CAP, WPT, CAP>(buf, lane_base + v0 + 2 * V, rem - v0 - 2 * V);
        if (n_in <= v0 + 2 * V)
            break;
    }
}

// How many of its own tiles ahead a scatter warp asks the memory system to bring into L2 (its register loads run one
// tile ahead).
#ifndef FLASHLLM_PREFETCH_AHEAD
#define FLASHLLM_PREFETCH_AHEAD 2
#endif
constexpr int kPrefetchAhead = FLASHLLM_PREFETCH_AHEAD;

// Warps of the register-streaming kernel: one B loader, kDirectIssuers MMA issuers, then the scatter warps.
constexpr int kDirectIssuers = 2;

// The most accumulators that the tiles of a CTA may take turns with (plan.accumulators: this many or kDirectIssuers).  The
// tensor core truncates every addition, so a sum's error grows with the tiles added up in one accumulator: with four of them a
// K range may be twice as long as with two.
__host__ __device__ constexpr int direct_accumulators(int n_tile)
{
    return n_tile <= 64 ? 2 * kDirectIssuers : kDirectIssuers;
}

// Sum over the CTAs of a cluster: rank q finishes rows [128 q / S, 128 (q + 1) / S) of the output tile, and every CTA sends it
// those rows of its partial tile, [S ranks][rows][columns + 4 for the banks' sake].  The stores count themselves in on the
// receiver's mbarrier, so nobody asks a peer for data or waits for it beyond that.  With the partial tiles parked at home and
// fetched between two cluster barriers the sum took 2.4 of the 6.3 us of 1024x1024 N = 8 in clusters of eight.  us per call
// before and after, with the waits that park the warp in place of sleeping ones: that call 5.6 -> 4.5, 4096x4096 N = 16
// (eight) 9.9 -> 8.7, 9216x1152 N = 16 (three) 9.1 -> 8.1, 4736x7232 N = 32 (seven) 19.0 -> 18.6.
//
// 128 columns are parked at home and fetched as before: a row per lane makes for stores of 16 bytes to as many places, and
// 2688x8960 N = 128 in clusters of six takes 16.6 us that way instead of 15.4.  64 columns, for which there is no area but the
// operands' buffers, too where CTAs share SMs (plan.push): us per call parked / sent, 4096x4096 in clusters of eight 12.3 / 13.0,
// of six 13.8 / 14.8; 5120x1024 in sixes 9.1 / 10.5; but with an SM to every CTA 1024x4096 in clusters of two 17.9 / 17.0, of
// four 11.8 / 11.2, of eight 9.2 / 8.4.
constexpr int kPushMaxN = 64;

__host__ __device__ constexpr int cluster_sum_rows(int S)
{
    return (kTileM + S - 1) / S;
}
__host__ __device__ constexpr int cluster_sum_bytes(int n_tile, int S)
{
    return S * cluster_sum_rows(S) * (n_tile + 4) * 4;
}

// One scatter warp's share of the accumulators (as in accumulators_to_output) to the CTAs that finish its rows; NaN from a
// CTA that gave up, whose tensor memory may hold anything.
template<int N_TILE>
__device__ __forceinline__ void accumulators_to_peers(uint32_t tmem_acc, int accumulators, int n_valid, int quarter, int lane, int sw,
                                                      int per_quarter, int S, int rank, uint32_t sum_base, uint32_t sum_bar, bool ok)
{
    if (sw >= 4 * per_quarter)
        return;
    const int col_share = (N_TILE / per_quarter) < 8 ? 8 : (N_TILE / per_quarter);
    const int col_begin = (sw / 4) * col_share;
    const int col_end   = (col_begin + col_share) < n_valid ? (col_begin + col_share) : n_valid;
    const int row = quarter * 32 + lane;
    const int q   = ((row + 1) * S - 1) / kTileM;  // who finishes this row
    const uint32_t bar = ptx::map_to_rank(sum_bar, q);
    const uint32_t to  = ptx::map_to_rank(sum_base, q)
                        + static_cast<uint32_t>((rank * cluster_sum_rows(S) + row - kTileM * q / S) * (N_TILE + 4)) * 4u;
    const uint32_t acc = tmem_acc + (static_cast<uint32_t>(quarter * 32) << 16);
    constexpr int  A   = direct_accumulators(N_TILE);
    const float    none = ok ? 0.0f : __int_as_float(0x7FFFFFFF);
    for (int c0 = col_begin; c0 < col_end; c0 += 8) {
        float    v[8];
        uint32_t t[A][8];
#pragma unroll
        for (int a = 0; a < A; ++a)
            if (a < accumulators)
                ptx::tmem_ld_x8(acc + a * N_TILE + c0, t[a]);
        ptx::tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 8; ++i)
            v[i] = ok && accumulators > 0 ? __uint_as_float(t[0][i]) : none;
#pragma unroll
        for (int a = 1; a < A; ++a)
            if (a < accumulators)
#pragma unroll
                for (int i = 0; i < 8; ++i)
                    v[i] += __uint_as_float(t[a][i]);
        ptx::st_async_v4_f32(to + c0 * 4, v, bar);
        ptx::st_async_v4_f32(to + c0 * 4 + 16, v + 4, bar);
    }
}

// The rows this CTA finishes, once all its peers' parts are there (`arrived`): added in rank order, four columns per thread.
// What a thread's first outputs need from memory is asked for before that.
template<int N_TILE, typename Arrived>
__device__ __forceinline__ void finish_cluster_rows(const SpmmParams& p, uint32_t sum_base, int rank, int S, int G, int g, int n_idx,
                                                    int tile_row, int n_valid, int tid, int threads, Arrived arrived)
{
    const int    row0     = kTileM * rank / S;
    const int    rows     = kTileM * (rank + 1) / S - row0;
    const size_t tile_off = static_cast<size_t>(n_idx) * N_TILE * p.M + static_cast<size_t>(tile_row) * kTileM;
    const uint32_t step  = static_cast<uint32_t>(cluster_sum_rows(S) * (N_TILE + 4)) * 4u;
    const int      shift = 32 - __clz(rows - 1);  // rows, rounded up to a power of two, are 16 to 64
    const int      r_1   = tid & ((1 << shift) - 1), c_1 = (tid >> shift) * 4;
    const bool     first = G == 1 && r_1 < rows && c_1 < n_valid;
    float          bias_1 = -0.0f;
    half           res_1[4];
    if (first)
        bias_1 = bias_of(p, tile_row * kTileM + row0 + r_1);
    if (first && p.residual != nullptr)
        load_residual<4>(p, res_1, tile_off + static_cast<size_t>(c_1) * p.M + row0 + r_1);
    if (!arrived())
        return;
    for (int e = tid; e < (n_valid / 4) << shift; e += threads) {
        const int r = e & ((1 << shift) - 1), c = (e >> shift) * 4;
        if (r >= rows)
            continue;
        const uint32_t from = sum_base + static_cast<uint32_t>(r * (N_TILE + 4) + c) * 4u;
        float          v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        uint4          w[kMaxClusterK];
#pragma unroll
        for (int s = 0; s < kMaxClusterK; ++s)
            if (s < S)
                w[s] = lds16(from + s * step);
#pragma unroll
        for (int s = 0; s < kMaxClusterK; ++s)
            if (s < S) {
                v[0] += __uint_as_float(w[s].x);
                v[1] += __uint_as_float(w[s].y);
                v[2] += __uint_as_float(w[s].z);
                v[3] += __uint_as_float(w[s].w);
            }
        const int    m  = row0 + r;
        const size_t at = static_cast<size_t>(c) * p.M + m;
        if (G > 1) {
            float* const part = p.partial + static_cast<size_t>(g) * p.M * p.N + tile_off + at;
#pragma unroll
            for (int i = 0; i < 4; ++i)
                part[static_cast<size_t>(i) * p.M] = v[i];
        }
        else if (e == tid)
            finish_columns<4>(p, v, tile_off + at, 4, bias_1, res_1);
        else
            finish_columns<4>(p, v, tile_off + at, 4, bias_of(p, tile_row * kTileM + m));
    }
    if (G > 1 && p.tile_counters != nullptr)
        __threadfence();
}

// CAP: vectors per lane kept in registers.  WARPS: stages = tiles in flight per CTA.  WPT: warps that share one tile
// (row q of warp h is the tile's row q * WPT + h), so a tile of up to 32 * CAP * WPT vectors is handled without the
// overflow loop and a warp's instruction stream per tile is 1 / WPT as long.  MIN_BLOCKS: CTAs per SM the register
// budget is sized for.  PUSH: the CTAs of a cluster send one another their sums (a kernel of its own, since both ways in one
// cost every call 0.2 us).
//
// One thread cannot issue tcgen05.mma as fast as the tensor core retires them (measured: 4 MMAs and the commit that
// hands a stage back cost an issuing thread ~400 cycles, the tensor core ~180), so tiles alternate between
// kDirectIssuers issuing threads, each with accumulators of its own in tensor memory; the epilogue adds them.
template<int N_TILE, int CAP, int WARPS, int MIN_BLOCKS, int WPT, bool PUSH>
__global__ void __launch_bounds__((1 + kDirectIssuers + WARPS * WPT) * 32, MIN_BLOCKS)
    spmm_tcgen05_direct_kernel(const __grid_constant__ CUtensorMap tmap_b, const SpmmParams p)
{
    static_assert(N_TILE == 16 || N_TILE == 32 || N_TILE == 64 || N_TILE == 128, "unsupported MMA N");
    static_assert(WARPS >= 4 && WARPS <= 12, "four warps cover the TMEM lane quarters in the epilogue");
    static_assert(!PUSH || N_TILE <= kPushMaxN, "wider outputs are parked");
    static_assert(WPT == 1 || WPT == 2, "a tile is decompressed by one warp or by a pair");
    static_assert(CAP % 2 == 0 && 32 % WPT == 0, "batches are issued in two halves; the clear is split evenly");
    constexpr uint32_t kBSlab    = N_TILE * kTileK * 2;  // one K tile of B in shared memory
    constexpr int      MI        = kDirectIssuers;
    static_assert(WARPS % MI == 0, "every issuer serves the same stages on every lap");
    constexpr uint32_t kTmemCols = direct_accumulators(N_TILE) * N_TILE;  // a power of two
    constexpr int      NSW       = WARPS * WPT;  // scatter warps
    constexpr int      a_stages  = WARPS;

#ifdef FLASHLLM_TRACE
    __shared__ unsigned int s_trace[kTraceKinds * kTraceDepth];
    for (int i = threadIdx.x; i < kTraceKinds * kTraceDepth; i += blockDim.x)
        s_trace[i] = 0;
#endif
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t raw_addr = ptx::smem_u32(smem_raw);
    const uint32_t base     = (raw_addr + 1023u) & ~1023u;  // swizzled operands need 1024-byte alignment
    uint8_t* const smem     = smem_raw + (base - raw_addr);

    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0)
        FL_CTA_TIME(0);

    const SpmmPlan& plan     = p.plan;
    const int       b_stages = plan.b_stages;
    const int       KB       = plan.b_batch;
    const int       S        = plan.cluster_k;
    const int       G        = plan.workspace_k;
    const int       accs     = plan.accumulators;  // a power of two
    constexpr int   b_warp   = 0;  // warp that loads B
    constexpr int   mma_warp = 1;       // first of the MI warps that issue MMAs; it owns the TMEM allocation
    constexpr int   first_sw = 1 + MI;  // first scatter warp
    constexpr int   NTS      = NSW * 32;

    // ---- shared memory carve-up
    const uint32_t a_base   = base;
    const uint32_t b_base   = a_base + a_stages * kDenseTileBytes;
    const uint32_t sum_area = b_base + b_stages * KB * kBSlab;  // plan.sum_bytes: the peers' partial sums
    const uint32_t bar_base = sum_area + plan.sum_bytes;
    const uint32_t a_full   = bar_base;
    const uint32_t a_empty  = a_full + 8u * a_stages;
    const uint32_t b_full   = a_empty + 8u * a_stages;
    const uint32_t b_empty  = b_full + 8u * b_stages;
    const uint32_t acc_full = b_empty + 8u * b_stages;
    const uint32_t sum_full = acc_full + 8u;
    const uint32_t misc_off = (sum_full + 8u) - base;
    const uint32_t sum_base = plan.sum_bytes > 0 ? sum_area : a_base;
    volatile uint32_t* const tmem_slot  = reinterpret_cast<volatile uint32_t*>(smem + misc_off);
    volatile uint32_t* const abort_flag = reinterpret_cast<volatile uint32_t*>(smem + misc_off + 4);
    int* const               offs_stage = reinterpret_cast<int*>(smem + misc_off + 16);  // plan.offsets_staged ints

    // ---- work assignment: blockIdx.x = K part inside the cluster, y = tile row, z = (N tile, workspace part)
    const int rank     = blockIdx.x;
    const int tile_row = blockIdx.y;
    const int g        = blockIdx.z % G;
    const int n_idx    = blockIdx.z / G;
    const int parts    = S * G;
    const int part     = g * S + rank;
    const int k_begin  = static_cast<int>(static_cast<long long>(p.k_tiles) * part / parts);
    const int k_end    = static_cast<int>(static_cast<long long>(p.k_tiles) * (part + 1) / parts);
    const int L        = k_end - k_begin;
    const int* const offs_global = p.tile_offsets + static_cast<long long>(tile_row) * p.k_tiles + k_begin;
    const bool       staged      = (L + 1 <= plan.offsets_staged);
    const int* const offs        = staged ? offs_stage : offs_global;  // valid after the set-up barrier

    if (raw_addr != base) {  // the launch did not honour the 1024-byte alignment: nothing below would be valid
        if (threadIdx.x == 0)
            atomicOr(p.status, kStatusSmemMisaligned);
        return;
    }

    // ---- scatter warps: the first tile's words are requested before anything else, so that the set-up below
    // (barrier initialisation, tensor-memory allocation, offset staging and checking: ~1.5 us) hides behind their
    // latency instead of preceding it.  The two offsets are read straight from global memory and checked on the spot.
    const int sw        = warp - first_sw;
    const int st        = sw % WARPS;       // the stage, and the tile stream st, st + WARPS, ... this warp works on
    const int h         = sw / WARPS;       // its index among the WPT warps that share those tiles
    const int first_vec = h * 32 + lane;    // this lane's vector in row 0 of the warp's share
    uint4     nxt[CAP];                     // words of the tile about to be scattered (loads in flight)
    int          n_in = 0;                  // vectors of the whole tile whose share is in nxt
    const uint4* src  = p.compressed;
    bool         bad  = false;
    auto fetch_first_tile = [&]() {
        if (st < L) {
            const int vb = offs_global[st], ve = offs_global[st + 1];
            bad          = (ve < vb) || (ve - vb > kMaxTileVectors) || (vb < 0);
            n_in         = bad ? 0 : ve - vb;
            src          = p.compressed + (bad ? 0 : vb);
            load_batch<WPT, CAP>(nxt, src + first_vec, n_in, n_in - first_vec);
        }
    };
    if (warp >= first_sw) {
#pragma unroll
        for (int q = 0; q < CAP; ++q)
            nxt[q] = make_uint4(0u, 0u, 0u, 0u);
        if (p.early_weights)
            fetch_first_tile();
    }

    // ---- set-up
    if (threadIdx.x == 0) {
        for (int i = 0; i < a_stages; ++i) {
            ptx::mbar_init(a_full + 8u * i, WPT);  // every warp that shares the tile publishes its part
            ptx::mbar_init(a_empty + 8u * i, 1);
        }
        for (int i = 0; i < b_stages; ++i) {
            ptx::mbar_init(b_full + 8u * i, 1);
            ptx::mbar_init(b_empty + 8u * i, MI);  // every issuer hands a batch back
        }
        ptx::mbar_init(acc_full, MI);
        ptx::mbar_init(sum_full, 1);
        abort_flag[0]             = 0u;  // a launch never inherits a give-up from an earlier one: the status word only reports
        abort_flag[kDepsResolved] = 0u;
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tmap_b);
    }
    if (warp == mma_warp) {
        ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
        ptx::tmem_relinquish();
    }
    if (!p.early_weights) {
        ptx::grid_dependency_wait();
        if (warp >= first_sw)
            fetch_first_tile();
    }
    if (staged) {
        // This CTA's slice of TileOffsets is read once, together, instead of one dependent load per tile.
        for (int i = threadIdx.x; i <= L; i += blockDim.x)
            offs_stage[i] = offs_global[i];
    }
    // Offsets that run backwards, or tiles above 2048 vectors, would make the roles below disagree about who owns
    // which vectors; the whole slice is checked before any of them starts.
    bool bad_slice = offsets_slice_is_bad(offs_global, L);
    ptx::tc_fence_before_sync();
    bad_slice = __syncthreads_or(bad_slice ? 1 : 0) != 0;
    ptx::tc_fence_after_sync();
    const bool go = !bad_slice && (*abort_flag == 0u);  // false: every role skips its work and no sum leaves this CTA
    if (bad_slice && threadIdx.x == 0) {
        atomicOr(p.status, kStatusBadTileOffsets);
        *abort_flag = 1u;
    }
    const uint32_t tmem_acc = *tmem_slot;
    const int      n_valid  = (p.N - n_idx * N_TILE) < N_TILE ? (p.N - n_idx * N_TILE) : N_TILE;
    if (PUSH && S > 1) {
        if (threadIdx.x == 0)  // everything the peers (and this CTA) will store here
            ptx::mbar_arrive_expect_tx(sum_full,
                                       static_cast<uint32_t>(S * (kTileM * (rank + 1) / S - kTileM * rank / S) * n_valid) * 4u);
        __syncwarp();
        if (plan.sum_bytes > 0)
            ptx::cluster_arrive_relaxed();  // this CTA runs and its barrier is ready
    }
    // A following kernel of this library may start its set-up and weight streaming while this grid drains; it waits
    // (in its B loader) before it touches anything this grid or its predecessors produce.
    if (threadIdx.x == 0)
        ptx::grid_launch_dependents();
    if (threadIdx.x == 0)
        FL_CTA_TIME(1);

    bool acc_ok = false;  // scatter warps: the CTA's sums are complete
    if (warp == b_warp) {
        // ================================================================ B loader: KB K tiles per TMA instruction
        if (lane == 0 && L > 0 && go) {
            load_b_batches(&tmap_b, (L + KB - 1) / KB, KB, b_stages, kBSlab, b_base, b_full, b_empty, n_idx * N_TILE, k_begin,
                           abort_flag, p.status);
        }
    }
    else if (warp < first_sw) {
        // ================================================================ MMA issuers: issuer m takes tiles m, m + MI, ...
        // The B batches hold a multiple of MI tiles, so every issuer has work in every full batch and hands it back
        // itself; the last, partial batch is never waited for.
        if (lane == 0 && go) {
            const int m = warp - mma_warp;
            if (m < L) {
                const uint32_t idesc   = ptx::umma_idesc_f16_f32(kTileM, N_TILE);
                const uint64_t a_desc0 = ptx::umma_desc_kmajor_sw128(a_base);
                const uint64_t b_desc0 = ptx::umma_desc_kmajor_sw128(b_base);
                int            s = m, bs = 0, kb = m;
                uint32_t       a_par = 0, b_par = 0;
                bool           ready = false, first_in_batch = true;
                for (int j = m; j < L; j += MI) {
                    if (m == 0)
                        FL_TRACE(7, j);
                    if (!ready) {
                        if (!wait_bounded(a_full + 8u * s, a_par, abort_flag, p.status))
                            break;
                        if (first_in_batch && !wait_bounded(b_full + 8u * bs, b_par, abort_flag, p.status))
                            break;
                    }
                    if (m == 0)
                        FL_TRACE(9, j);
                    int      s_n = s + MI, kb_n = kb + MI, bs_n = bs;
                    uint32_t a_par_n = a_par, b_par_n = b_par;
                    if (s_n >= a_stages) {
                        s_n -= a_stages;
                        a_par_n ^= 1u;
                    }
                    const bool batch_done = kb_n >= KB;
                    if (batch_done) {
                        kb_n -= KB;
                        if (++bs_n == b_stages) {
                            bs_n = 0;
                            b_par_n ^= 1u;
                        }
                    }
                    const bool has_next = j + MI < L;
                    ptx::tc_fence_after_sync();
#if (FLASHLLM_ABLATE & 4)
                    ptx::umma_commit(a_empty + 8u * s);  // timing only: hand-backs without any MMA
                    if (batch_done || !has_next)
                        ptx::umma_commit(b_empty + 8u * bs);
                    ready = false;
                    if (false)
#endif
                    ready = ptx::umma_tile_commit_probe(
                        tmem_acc + static_cast<uint32_t>((j & (accs - 1)) * N_TILE),
                        a_desc0 + static_cast<uint32_t>(s * (kDenseTileBytes >> 4)),
                        b_desc0 + static_cast<uint32_t>((bs * KB + kb) * (kBSlab >> 4)), idesc, j >= accs ? 1u : 0u, a_empty + 8u * s,
                        b_empty + 8u * bs, (batch_done || !has_next) ? 1u : 0u, a_full + 8u * s_n, a_par_n, b_full + 8u * bs_n,
                        b_par_n, has_next ? 1u : 0u, (has_next && batch_done) ? 1u : 0u);
                    if (m == 0)
                        FL_TRACE(10, j);
                    first_in_batch = batch_done;
                    s     = s_n;
                    kb    = kb_n;
                    bs    = bs_n;
                    a_par = a_par_n;
                    b_par = b_par_n;
                }
            }
            ptx::umma_commit(acc_full);
        }
    }
    else {
        // ================================================================ scatter warps: WPT warps per stage
        if (L > 0 && go) {
            const uint32_t stage     = a_base + st * kDenseTileBytes;
            const uint32_t full_bar  = a_full + 8u * st;
            const uint32_t empty_bar = a_empty + 8u * st;
            // the tile after the first one is pulled from DRAM into L2 (its register loads come one tile from now)
            if (st < L && lane == 0 && h == 0) {
                for (int a = 1; a < kPrefetchAhead; ++a) {
                    const int t = st + a * WARPS;
                    if (t < L && offs[t + 1] > offs[t])
                        ptx::prefetch_l2_bulk(p.compressed + offs[t], static_cast<uint32_t>(offs[t + 1] - offs[t]) * 16u);
                }
            }
            uint32_t use = 0;
            for (int j = st; j < L; j += WARPS, ++use) {
                if (bad)
                    atomicOr(p.status, kStatusBadTileOffsets);
                if (lane == 0)
                    FL_TRACE(0, j);
                bool ok = !bad;
                if (ok && use > 0)
                    ok = __all_sync(0xFFFFFFFFu, wait_bounded_converged(empty_bar, (use & 1u) ^ 1u, abort_flag, p.status));
                if (!ok) {  // uniform across the warps that share the tile: they watch the same barrier and flag
                    if (bad)
                        *abort_flag = 1u;
                    break;
                }
                if (lane == 0)
                    FL_TRACE(3, j);
                // Offsets of this warp's following tile.  Two places are wrong for these two shared-memory loads: right
                // behind the previous tile's global loads (they queue behind them in the load/store unit: ~700 cycles at
                // the loop's top) and behind the proxy fence below (they wait for it, and the loads that need them wait
                // for them: the refill then takes ~7000 cycles instead of ~650).  Here the unit is idle.
                const bool has_next = j + WARPS < L;
                int        vb2 = 0, ve2 = 0;
                if (has_next) {
                    vb2 = offs[j + WARPS];
                    ve2 = offs[j + WARPS + 1];
                }
                // ---- clear the stage (each sharing warp its part), then scatter the new tile
                if (!(FLASHLLM_ABLATE & 1)) {
#pragma unroll
                    for (int q = 0; q < 32 / WPT; ++q)
                        sts_zero16(stage + static_cast<uint32_t>((q * WPT + h) * 32 + lane) * 16u);
                }
                // another lane's (or the partner warp's) zero must not land on top of a new value
                if (WPT == 1)
                    __syncwarp();
                else
                    ptx::named_barrier_sync(1u + static_cast<uint32_t>(st), 32u * WPT);
                if (lane == 0)
                    FL_TRACE(2, j);
                {
                    const int rem = n_in - first_vec;
#if (FLASHLLM_ABLATE & 2)
#pragma unroll
                    for (int q = 0; q < CAP; ++q)
                        if ((nxt[q].x ^ nxt[q].y ^ nxt[q].z ^ nxt[q].w) == 0x9E3779B9u)  // keeps the loads alive
                            scatter_word(stage, nxt[q].x);
#else
                    scatter_tile<WPT, CAP>(stage, nxt, src + first_vec, n_in, rem);
#endif
                }
                if (lane == 0)
                    FL_TRACE(5, j);
#if !(FLASHLLM_ABLATE & 16)  // timing only: without the proxy fence the tensor core may read stale words
                ptx::fence_proxy_async_smem();
#endif
                __syncwarp();
                if (lane == 0)
                    ptx::mbar_arrive(full_bar);
                if (lane == 0)
                    FL_TRACE(6, j);
                // ---- start fetching the following tile
                if (has_next) {
                    bad  = (ve2 < vb2) || (ve2 - vb2 > kMaxTileVectors) || (vb2 < 0);
                    n_in = bad ? 0 : ve2 - vb2;
                    src  = p.compressed + (bad ? 0 : vb2);
                    if (!(FLASHLLM_ABLATE & 8))
                        load_batch<WPT, CAP>(nxt, src + first_vec, n_in, n_in - first_vec);
                    // ... and pull the one after it from DRAM into L2, so that its register loads, issued one tile
                    // from now, only have the L2 latency left to hide
                    if (lane == 0 && h == 0 && j + kPrefetchAhead * WARPS < L) {
                        const int pb = offs[j + kPrefetchAhead * WARPS], pe = offs[j + kPrefetchAhead * WARPS + 1];
                        if (pe > pb)
                            ptx::prefetch_l2_bulk(p.compressed + pb, static_cast<uint32_t>(pe - pb) * 16u);
                    }
                }
                if (lane == 0)
                    FL_TRACE(13, j);
            }
        }

        // ================================================================ epilogue (same warps)
        acc_ok = go;
        if (L > 0 && go)
            acc_ok = wait_bounded_converged(acc_full, 0u, abort_flag, p.status);
        acc_ok = __all_sync(0xFFFFFFFFu, acc_ok && (*abort_flag == 0u));
        ptx::tc_fence_after_sync();
        if (sw == 0 && lane == 0)
            FL_CTA_TIME(2);

        if (!PUSH || S == 1)
            accumulators_to_output<N_TILE>(p, tmem_acc, L < accs ? L : accs, N_TILE, warp & 3, lane, sw, NSW >= 8 ? 2 : 1, S, G, g,
                                           n_idx, tile_row, acc_ok, reinterpret_cast<float*>(smem));
    }

    // ================================================================ cluster reduction and tear-down
    if (!PUSH && S > 1) {
        __syncwarp();
        ptx::cluster_sync_all();  // every CTA's partial tile is parked in its shared memory
        if (warp >= first_sw)
            cluster_reduce_store<N_TILE>(p, base, rank, S, G, g, n_idx, tile_row, threadIdx.x - first_sw * 32, NTS,
                                         *abort_flag == 0u);
        __syncwarp();
        ptx::cluster_sync_all();  // nobody leaves while a peer may still read its shared memory
    }
    else if (S > 1) {
        __syncwarp();
        if (plan.sum_bytes > 0)
            ptx::cluster_wait();  // long over: the peers have started
        else
            ptx::cluster_sync_all();  // nobody multiplies any more, the stages are free
        if (warp >= first_sw) {
            ptx::tc_fence_after_sync();
            accumulators_to_peers<N_TILE>(tmem_acc, L < accs ? L : accs, n_valid, warp & 3, lane, sw, NSW >= 8 ? 2 : 1, S, rank,
                                          sum_base, sum_full, acc_ok);
            finish_cluster_rows<N_TILE>(p, sum_base, rank, S, G, g, n_idx, tile_row, n_valid, threadIdx.x - first_sw * 32, NTS, [&]() {
                return __all_sync(0xFFFFFFFFu, wait_bounded_cluster(sum_full, 0u, abort_flag, p.status)) && *abort_flag == 0u;
            });
        }
    }
    ptx::tc_fence_before_sync();
    __syncthreads();
    // A CTA that gave up leaves only when its peers have left or given up too: until then they may store into its shared memory.
    if (PUSH && S > 1 && *abort_flag != 0u) {
        __syncwarp();
        ptx::cluster_sync_all();
    }
    finish_tile<N_TILE>(p, S, G, n_idx, tile_row, abort_flag);
    if (threadIdx.x == 0)
        FL_CTA_TIME(3);
    if (warp == mma_warp) {
        __syncwarp();
        ptx::tmem_dealloc(tmem_acc, kTmemCols);
    }
#ifdef FLASHLLM_TRACE
    if (blockIdx.y == FLASHLLM_TRACE && blockIdx.x == 0)
        for (int i = threadIdx.x; i < kTraceKinds * kTraceDepth; i += blockDim.x)
            g_trace[i] = s_trace[i];
#endif
}

}  // namespace flashllm
