// Load-as-Sparse / Compute-as-Dense SpMM for sm_100a, streaming form: a persistent grid over the linear tile sequence.
//
// The tiles of A in the order of TileOffsets (tile row by tile row, K tile by K tile) are ONE sequence, and so are their
// words in Compressed_A.  CTA c of P takes tiles T*c/P up to T*(c+1)/P of it (to a rounding), whatever rows they belong to, so every SM gets
// the same share of the matrix for any number of tile rows.  (One CTA per tile row leaves SMs idle whenever the rows do
// not fill the last wave: 216 rows on 296 CTA slots, 384 rows on 296.)  A maximal run of a CTA's tiles inside one tile row
// is a segment:
//
//   * scatter warps decompress tile after tile as in the register-streaming form and know nothing of rows;
//   * the MMA-issuing warp multiplies a segment in chunks of at most plan.chunk_tiles tiles, each in the other one of two
//     tensor-memory accumulators than the chunk before, and changes over without draining anything;
//   * four epilogue warps read a finished accumulator while the next chunk is being multiplied and add a segment's chunks
//     up in fp32, in tensor memory.  The tensor core truncates every one of its additions: with a segment in one accumulator
//     36864x9216 N = 16 at 80 % was 2.07501e-4 off its exact values in the 2-norm, in chunks it is 2.07427e-4 (rounding to
//     fp16 alone: 2.07382e-4), and a layer of four such matmuls 3.03e-4 instead of 3.49e-4.  A segment that is a
//     whole row becomes output at once; a part of a row is parked as an fp32 tile in the stream's scratch and counted in
//     on the row's counter, and whoever completes the count adds the parts up in CTA order (the same bits whoever comes
//     last) and finishes the output.  No CTA waits for another.
//
// What a call takes after its last MMA is no other CTA's work any more, so it is kept short.  The first of two CTAs that share
// a row usually finds the other's part parked, takes it into tensor memory while its own is being multiplied and finishes the
// row without parking.  Other rows are added up when the CTA's roles are done, by all of its threads instead of the four
// epilogue warps: a part is an L2 round trip away.  Both together, us per call with two matrices in turn: 2048x32768 N=16 70 %
// (19 parts a row) 26.5 -> 24.5, 9216x36864 N=32 70 % (5 parts) 97.1 -> 93.4, 49152x12288 N=64 143.8 -> 141.1, 36864x9216 N=16
// 71.4 -> 70.6.
//
// The MMA-issuing warp runs converged and elects one lane inside the instruction block: operands then stay in uniform
// registers.  Issued from a branch taken by one lane, the four MMAs and the commit of a tile cost 271 cycles instead of
// the 170 the tensor core needs for them (M128 N16 K16), which took two issuing warps to hide.
//
// Measured (B200, back to back on one stream, two matrices in turn, against one CTA or cluster per tile row): 27648x9216 N=8
// 90 % 62.2 -> 45.4 us, 2048x32768 N=16 70 % 27.0 -> 24.5, 9216x36864 N=32 70 % 100 -> 93, 49152x12288 N=64 80 % 170 -> 141,
// 36864x9216 N=16 80 % (288 rows: hardly any quantisation to begin with) 75.9 -> 70.6.  (With another matrix on every call, none
// of which L2 holds, the large ones take 2 to 15 % longer.)  The chunks cost 0 to 0.7 % of that, at N = 64 1.3 %; as short as 24
// tiles there, which the cut by tiles asks of 27648x12288 with a workspace, 4.8 % (85.2 -> 89.3).
// A CTA's share is bound by the shared-memory work of its tiles: of ~3300 cycles from one tile of a stage to the next at
// 80 % (8 stages per SM: 412 per tile), 570 go to clearing the stage, 1140 to the 16-bit scatter stores (they wait for the
// tensor core's operand reads), 1070 to getting the next tile's loads issued behind the other warps' stores, 430 to the
// stage's hand-back.  Six stages per CTA, or one CTA of 8 or 12 warps per SM, are slower.
#pragma once
#include "spmm_kernel_direct_sm100.cuh"

namespace flashllm {

constexpr int kStreamStages       = 4;  // decompressed tiles in flight per CTA, one scatter warp each
constexpr int kStreamCtasPerSm    = 2;
constexpr int kStreamFirstScatter = 2;  // warp 0 loads B, warp 1 issues MMAs
constexpr int kStreamFirstEpi     = kStreamFirstScatter + kStreamStages;
constexpr int kStreamWarps        = kStreamFirstEpi + 4;
constexpr int kStreamSumBytes     = 32;    // two rows' number, first and last CTA
constexpr int kStreamLooks        = 4096;  // at another CTA's arrival while this one's own sums are being completed

// First tile of CTA c's share, and the CTA whose share holds tile t.  No division, which the last part of
// a row would wait for.  stream_share = 2^32 tiles / CTAs, rounded up: exact at c = 0 and c = CTAs.
__host__ __device__ __forceinline__ int stream_begin(unsigned long long stream_share, int c)
{
    return static_cast<int>((stream_share * static_cast<unsigned>(c)) >> 32);
}
__device__ __forceinline__ int stream_owner(const SpmmParams& p, int ctas, int t)
{
    int c = static_cast<int>(t * p.ctas_per_tile);  // a guess, right to a CTA
    c     = c < ctas ? c : ctas - 1;
    while (stream_begin(p.stream_share, c) > t)
        --c;
    while (stream_begin(p.stream_share, c + 1) <= t)
        ++c;
    return c;
}

// A scatter warp's tiles sw, sw + STAGES, ... of a CTA's L tiles: the words of the next one wait in registers (up to CAP
// 16-byte vectors per lane) while the warp's stage is still being multiplied.
template<int CAP, int STAGES>
struct TileStream {
    uint4        nxt[CAP];
    int          n_in;  // vectors of the tile in nxt
    const uint4* src;
    bool         bad;

    __device__ __forceinline__ void clear()
    {
        n_in = 0;
        src  = nullptr;
        bad  = false;
#pragma unroll
        for (int q = 0; q < CAP; ++q)
            nxt[q] = make_uint4(0u, 0u, 0u, 0u);
    }

    __device__ __forceinline__ void fetch(const SpmmParams& p, int vb, int ve, int lane)
    {
        bad  = (ve < vb) || (ve - vb > kMaxTileVectors) || (vb < 0);
        n_in = bad ? 0 : ve - vb;
        src  = p.compressed + (bad ? 0 : vb);
        load_batch<1, CAP>(nxt, src + lane, n_in, n_in - lane);
    }

    // The first tile, by offsets straight from global memory, before the CTA's set-up.
    __device__ __forceinline__ void fetch_first(const SpmmParams& p, const int* offs_global, int sw, int L, int lane)
    {
        if (sw < L)
            fetch(p, offs_global[sw], offs_global[sw + 1], lane);
    }

    __device__ __forceinline__ void run(const SpmmParams& p, const int* offs, int sw, int L, int lane, uint32_t stage,
                                        uint32_t full_bar, uint32_t empty_bar, volatile uint32_t* abort_flag)
    {
        if (lane == 0) {
            for (int a = 1; a < kPrefetchAhead; ++a) {
                const int t = sw + a * STAGES;
                if (t < L && offs[t + 1] > offs[t])
                    ptx::prefetch_l2_bulk(p.compressed + offs[t], static_cast<uint32_t>(offs[t + 1] - offs[t]) * 16u);
            }
        }
        uint32_t use = 0;
        for (int j = sw; j < L; j += STAGES, ++use) {
            bool ok = !bad;
            if (use > 0)
                ok = wait_bounded_converged(empty_bar, (use & 1u) ^ 1u, abort_flag, p.status) && ok;
            if (!__all_sync(0xFFFFFFFFu, ok))
                break;
            // offsets of this warp's following tile: read here, where the load/store unit is idle (see the
            // register-streaming form)
            const bool has_next = j + STAGES < L;
            int        vb2 = 0, ve2 = 0;
            if (has_next) {
                vb2 = offs[j + STAGES];
                ve2 = offs[j + STAGES + 1];
            }
            zero_fill_stage(stage, lane);
            __syncwarp();  // another lane's zero must not land on top of a new value
            scatter_tile<1, CAP>(stage, nxt, src + lane, n_in, n_in - lane);
            ptx::fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0)
                ptx::mbar_arrive(full_bar);
            if (has_next) {  // start fetching the following tile, and pull the one after it into L2
                fetch(p, vb2, ve2, lane);
                if (lane == 0 && j + kPrefetchAhead * STAGES < L) {
                    const int pb = offs[j + kPrefetchAhead * STAGES], pe = offs[j + kPrefetchAhead * STAGES + 1];
                    if (pe > pb)
                        ptx::prefetch_l2_bulk(p.compressed + pb, static_cast<uint32_t>(pe - pb) * 16u);
                }
            }
        }
    }
};

// Adds the parked parts of tile row `row` up in CTA order and finishes the output.  Called by all `threads` threads of a CTA
// when its other work is done: a part is an L2 round trip away, so what counts is how many loads are in flight.
template<int N_TILE>
__device__ __forceinline__ void
sum_row_parts(const SpmmParams& p, int row, int c_first, int c_last, const float* first, int tid, int threads)
{
    const size_t slot     = static_cast<size_t>(N_TILE) * kTileM;
    const bool   wide_out = (reinterpret_cast<uintptr_t>(p.out) & 7u) == 0;
    // Q groups of four outputs per thread and P parts at a time, added in CTA order: ten or twelve 16-byte loads in flight.
    // More and the kernel needs local memory, which costs every launch 0.5 us.
    constexpr int Q = N_TILE <= 32 ? 2 : 4, P = N_TILE <= 32 ? 5 : 2;
    const int     quads = p.N * (kTileM / 4);
    for (int q0 = tid; q0 < quads; q0 += Q * threads) {
        float4 acc[Q];
#pragma unroll
        for (int i = 0; i < Q; ++i)
            if (q0 + i * threads < quads)
                acc[i] = __ldcg(reinterpret_cast<const float4*>(first) + q0 + i * threads);
        for (int c = c_first + 1; c <= c_last; c += P) {
            float4 v[P][Q];
#pragma unroll
            for (int j = 0; j < P; ++j)
#pragma unroll
                for (int i = 0; i < Q; ++i)
                    if (c + j <= c_last && q0 + i * threads < quads)
                        v[j][i] = __ldcg(reinterpret_cast<const float4*>(p.partial + slot * (2 * (c + j))) + q0 + i * threads);
#pragma unroll
            for (int j = 0; j < P; ++j)
#pragma unroll
                for (int i = 0; i < Q; ++i)
                    if (c + j <= c_last) {
                        acc[i].x += v[j][i].x;
                        acc[i].y += v[j][i].y;
                        acc[i].z += v[j][i].z;
                        acc[i].w += v[j][i].w;
                    }
        }
#pragma unroll
        for (int i = 0; i < Q; ++i) {
            const int q = q0 + i * threads;
            if (q >= quads)
                break;
            const int    n = q / (kTileM / 4), out_row = row * kTileM + (q % (kTileM / 4)) * 4;
            const size_t at = static_cast<size_t>(n) * p.M + out_row;
            uint2        o;
            half*        oh = reinterpret_cast<half*>(&o);
            oh[0]           = finish_output(acc[i].x, p.bias, out_row, p.activation, p.residual, at);
            oh[1]           = finish_output(acc[i].y, p.bias, out_row + 1, p.activation, p.residual, at + 1);
            oh[2]           = finish_output(acc[i].z, p.bias, out_row + 2, p.activation, p.residual, at + 2);
            oh[3]           = finish_output(acc[i].w, p.bias, out_row + 3, p.activation, p.residual, at + 3);
            if (wide_out)
                *reinterpret_cast<uint2*>(p.out + at) = o;
            else
                for (int e = 0; e < 4; ++e)
                    p.out[at + e] = oh[e];
        }
    }
}

template<int N_TILE, int CAP>
__global__ void __launch_bounds__(kStreamWarps * 32, kStreamCtasPerSm)
    spmm_tcgen05_stream_kernel(const __grid_constant__ CUtensorMap tmap_b, const SpmmParams p)
{
    static_assert(N_TILE == 16 || N_TILE == 32 || N_TILE == 64, "unsupported MMA N");
    constexpr uint32_t kBSlab    = N_TILE * kTileK * 2;              // one K tile of B in shared memory
    constexpr uint32_t kTmemCols = 4 * N_TILE;  // two accumulators and the sum of a segment's finished chunks; a power of two

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t raw_addr = ptx::smem_u32(smem_raw);
    const uint32_t base     = (raw_addr + 1023u) & ~1023u;  // swizzled operands need 1024-byte alignment
    uint8_t* const smem     = smem_raw + (base - raw_addr);

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);  // uniform: the issuing warp stays converged
    const int lane = threadIdx.x & 31;

    const int       b_stages = p.plan.b_stages;
    const int       KB       = p.plan.b_batch;
    const int       chunk    = p.plan.chunk_tiles;
    const int       ctas     = gridDim.x;
    const int       cta      = blockIdx.x;
    const int       t_begin  = stream_begin(p.stream_share, cta);
    const int       L        = stream_begin(p.stream_share, cta + 1) - t_begin;  // >= 1: the grid has at most `tiles` CTAs
    const int       row0     = t_begin / p.k_tiles;
    const int       k0       = t_begin - row0 * p.k_tiles;  // K tile the CTA starts at

    // ---- shared memory carve-up
    const uint32_t a_base    = base;
    const uint32_t b_base    = a_base + kStreamStages * kDenseTileBytes;
    const uint32_t a_full    = b_base + b_stages * KB * kBSlab;
    const uint32_t a_empty   = a_full + 8u * kStreamStages;
    const uint32_t acc_full  = a_empty + 8u * kStreamStages;  // two of each: the accumulators take turns
    const uint32_t acc_empty = acc_full + 16u;
    const uint32_t b_full    = acc_empty + 16u;
    const uint32_t b_empty   = b_full + 8u * b_stages;
    const uint32_t misc_off  = (b_empty + 8u * b_stages) - base;
    volatile uint32_t* const tmem_slot  = reinterpret_cast<volatile uint32_t*>(smem + misc_off);
    volatile uint32_t* const abort_flag = reinterpret_cast<volatile uint32_t*>(smem + misc_off + 4);
    int* const               sums       = reinterpret_cast<int*>(smem + misc_off + 16);  // rows to add up at the end
    int* const               offs_stage = reinterpret_cast<int*>(smem + misc_off + 16 + kStreamSumBytes);  // plan.offsets_staged ints

    const int* const offs_global = p.tile_offsets + t_begin;
    const bool       staged      = (L + 1 <= p.plan.offsets_staged);
    const int* const offs        = staged ? offs_stage : offs_global;  // valid after the set-up barrier

    if (raw_addr != base) {  // the launch did not honour the 1024-byte alignment: nothing below would be valid
        if (threadIdx.x == 0)
            atomicOr(p.status, kStatusSmemMisaligned);
        return;
    }

    // ---- scatter warps request their first tile before anything else (see the register-streaming form)
    const bool scatters = warp >= kStreamFirstScatter && warp < kStreamFirstEpi;
    const int  sw       = warp - kStreamFirstScatter;  // the stage, and the tile stream sw, sw + kStreamStages, ...
    TileStream<CAP, kStreamStages> stream;
    if (scatters) {
        stream.clear();
        if (p.early_weights)
            stream.fetch_first(p, offs_global, sw, L, lane);
    }

    // ---- set-up
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStreamStages; ++i) {
            ptx::mbar_init(a_full + 8u * i, 1);
            ptx::mbar_init(a_empty + 8u * i, 1);
        }
        for (int i = 0; i < 2; ++i) {
            ptx::mbar_init(acc_full + 8u * i, 1);
            ptx::mbar_init(acc_empty + 8u * i, 4);  // every epilogue warp hands its quarter back
        }
        for (int i = 0; i < b_stages; ++i) {
            ptx::mbar_init(b_full + 8u * i, 1);
            ptx::mbar_init(b_empty + 8u * i, 1);
        }
        abort_flag[0]             = 0u;
        abort_flag[kDepsResolved] = 0u;
        ptx::fence_mbar_init();
        ptx::prefetch_tensormap(&tmap_b);
    }
    if (warp == 1) {
        ptx::tmem_alloc(ptx::smem_u32(const_cast<uint32_t*>(tmem_slot)), kTmemCols);
        ptx::tmem_relinquish();
    }
    if (!p.early_weights) {
        // The offsets are the first of two memory latencies in a row that a call starts with.  No value may be read before the
        // wait, but they may be on their way to L2: 36864x9216 N=16 70.6 -> 69.9 us, 9216x36864 N=32 93.5 -> 92.8.
        if (warp >= kStreamFirstEpi)
            for (int i = (threadIdx.x - kStreamFirstEpi * 32) * 32; i <= L; i += 128 * 32)
                ptx::prefetch_l2(offs_global + i);
        ptx::grid_dependency_wait();
        if (scatters)
            stream.fetch_first(p, offs_global, sw, L, lane);
    }
    if (staged) {
        for (int i = threadIdx.x; i <= L; i += blockDim.x)
            offs_stage[i] = offs_global[i];
    }
    bool bad_slice = offsets_slice_is_bad(offs_global, L);
    ptx::tc_fence_before_sync();
    bad_slice = __syncthreads_or(bad_slice ? 1 : 0) != 0;
    ptx::tc_fence_after_sync();
    const bool go = !bad_slice;  // false: every role skips its work and nothing is stored
    if (bad_slice && threadIdx.x == 0) {
        atomicOr(p.status, kStatusBadTileOffsets);
        *abort_flag = 1u;
    }
    const uint32_t tmem_acc = *tmem_slot;
    if (threadIdx.x == 0)
        ptx::grid_launch_dependents();

    if (warp == 0) {
        // ================================================================ B loader: KB K tiles per TMA instruction
        if (lane == 0 && go) {
            ptx::grid_dependency_wait();
            abort_flag[kDepsResolved] = 1u;
            int      bs = 0, issued = 0;
            uint32_t use = 0;
            bool     ok  = true;
            for (int j = 0, k = k0; ok && j < L; k = 0) {
                const int len = L - j < p.k_tiles - k ? L - j : p.k_tiles - k;  // this segment
                for (int b = 0; b < len; b += KB) {
                    if (!wait_bounded_relaxed(b_empty + 8u * bs, (use & 1u) ^ 1u, abort_flag, p.status)) {
                        ok = false;
                        break;
                    }
                    ptx::mbar_arrive_expect_tx(b_full + 8u * bs, KB * kBSlab);
                    ptx::tma_load_3d(b_base + bs * KB * kBSlab, &tmap_b, 0, 0, k + b, b_full + 8u * bs);
                    ++issued;
                    if (++bs == b_stages) {
                        bs = 0;
                        ++use;
                    }
                }
                j += len;
            }
            if (*abort_flag) {  // give copies already issued a bounded chance to land before the CTA may exit
                const uint64_t t_leave = ptx::globaltimer_ns();
                for (int back = 1; back <= b_stages && back <= issued; ++back) {
                    const int bb = issued - back;
                    while (!ptx::mbar_test_wait(b_full + 8u * (bb % b_stages), (bb / b_stages) & 1u)
                           && ptx::globaltimer_ns() - t_leave < 2000000ull) {}
                }
            }
        }
    }
    else if (warp == 1) {
        // ================================================================ MMA issuer (converged warp)
        if (go) {
            const uint32_t idesc   = ptx::umma_idesc_f16_f32(kTileM, N_TILE);
            const uint64_t a_desc0 = ptx::umma_desc_kmajor_sw128(a_base);
            const uint64_t b_desc0 = ptx::umma_desc_kmajor_sw128(b_base);
            int            s = 0, bs = 0, q = 0;
            uint32_t       a_par = 0, b_par = 0;
            bool           ok = true;
            for (int j = 0, k = k0; ok && j < L; k = 0) {
                const int len = L - j < p.k_tiles - k ? L - j : p.k_tiles - k;
                int       kb  = 0;
                for (int i0 = 0; ok && i0 < len; i0 += chunk, ++q) {
                    const int      n   = len - i0 < chunk ? len - i0 : chunk;
                    const uint32_t acc = tmem_acc + static_cast<uint32_t>((q & 1) * N_TILE);
                    ok = __all_sync(0xFFFFFFFFu, wait_bounded_converged(acc_empty + 8u * (q & 1), ((q >> 1) & 1u) ^ 1u, abort_flag,
                                                                        p.status));
                    for (int i = 0; ok && i < n; ++i) {
                        ok = wait_bounded_converged(a_full + 8u * s, a_par, abort_flag, p.status);
                        if (kb == 0)
                            ok = wait_bounded_converged(b_full + 8u * bs, b_par, abort_flag, p.status) && ok;
                        ok = __all_sync(0xFFFFFFFFu, ok);
                        if (!ok)
                            break;
                        const bool batch_done = kb + 1 == KB || i0 + i + 1 == len;
                        ptx::tc_fence_after_sync();
                        ptx::umma_tile_elect(acc, a_desc0 + static_cast<uint32_t>(s * (kDenseTileBytes >> 4)),
                                             b_desc0 + static_cast<uint32_t>((bs * KB + kb) * (kBSlab >> 4)), idesc, i != 0 ? 1u : 0u,
                                             a_empty + 8u * s, b_empty + 8u * bs, batch_done ? 1u : 0u);
                        if (++s == kStreamStages) {
                            s = 0;
                            a_par ^= 1u;
                        }
                        ++kb;
                        if (batch_done) {
                            kb = 0;
                            if (++bs == b_stages) {
                                bs = 0;
                                b_par ^= 1u;
                            }
                        }
                    }
                    if (ok)
                        ptx::umma_commit_elect(acc_full + 8u * (q & 1));
                }
                j += len;
            }
        }
    }
    else if (warp < kStreamFirstEpi) {
        // ================================================================ scatter warps: one whole tile at a time
        if (go)
            stream.run(p, offs, sw, L, lane, a_base + sw * kDenseTileBytes, a_full + 8u * sw, a_empty + 8u * sw, abort_flag);
    }
    else {
        // ================================================================ epilogue warps
        const int tid     = threadIdx.x - kStreamFirstEpi * 32;
        const int quarter = warp & 3;  // the tensor-memory lanes this warp may read
        const int r       = quarter * 32 + lane;
        const uint32_t tmem_lanes = tmem_acc + (static_cast<uint32_t>(quarter * 32) << 16);
        const uint32_t tmem_sum   = tmem_lanes + 2u * N_TILE;
        // eight columns of chunk q, added to the sum of the segment's chunks before it (`more`: there are such)
        auto read_columns = [&](int q, int c0, bool more, float (&v)[8]) {
            uint32_t t[8];
            ptx::tmem_ld_x8(tmem_lanes + static_cast<uint32_t>((q & 1) * N_TILE + c0), t);
            ptx::tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 8; ++e)
                v[e] = __uint_as_float(t[e]);
            if (more) {
                ptx::tmem_ld_x8(tmem_sum + c0, t);
                ptx::tmem_wait_ld();
#pragma unroll
                for (int e = 0; e < 8; ++e)
                    v[e] += __uint_as_float(t[e]);
            }
            if (c0 + 8 == N_TILE) {  // the accumulator has been read: the issuer may start the chunk after next in it
                ptx::tc_fence_before_sync();
                __syncwarp();
                if (lane == 0)
                    ptx::mbar_arrive(acc_empty + 8u * (q & 1));
            }
        };
        int          q    = 0;
        unsigned int todo = 0;  // tid 0: rows this CTA has completed the count of, its first or its last or both
        for (int row = row0;; ++row) {
            const int j = row == row0 ? 0 : (row - row0) * p.k_tiles - k0;
            if (j >= L)
                break;
            const int      len   = j == 0 ? min(L, p.k_tiles - k0) : min(L - j, p.k_tiles);
            const bool     whole = len == p.k_tiles;
            bool           ok    = go;
            int            i     = 0;
            // A row of two CTAs, the first one's last segment: usually the other, which began with its part, has parked that
            // long ago.  Then this CTA takes it into tensor memory ahead of time and finishes the row, parking nothing.
            const int  row_begin = row * p.k_tiles;
            const int  c_last    = whole ? cta : stream_owner(p, ctas, row_begin + p.k_tiles - 1);
            const bool ask       = c_last == cta + 1 && t_begin <= row_begin;
            bool       asked = false, complete = false;
            float      bias  = 0.0f;
            auto       other_has_parked = [&](bool look) {  // every epilogue warp asks once
                asked             = true;
                unsigned int seen = 0u;
                if (look && tid == 0) {
                    ptx::grid_dependency_wait();  // counters may be in use by the stream's previous launch until it is over
                    seen = ptx::ld_relaxed_gpu_u32(p.tile_counters + row);
                    for (int n = 1; seen == 0u && n < kStreamLooks && !ptx::mbar_test_wait(acc_full + 8u * (q & 1), (q >> 1) & 1u);
                         ++n)
                        seen = ptx::ld_relaxed_gpu_u32(p.tile_counters + row);
                    ptx::fence_acq_rel_gpu();
                }
                return barrier_any(1u, 128u, seen == 1u);
            };
            for (; ok; i += chunk, ++q) {
                const bool last_chunk = i + chunk >= len;
                if (last_chunk && ask) {
                    complete = other_has_parked(true);
                    if (complete) {
                        const float* from = p.partial + static_cast<size_t>(N_TILE * kTileM) * (2 * c_last) + r;
#pragma unroll 1
                        for (int c0 = 0; c0 < N_TILE; c0 += 8, from += 8 * kTileM) {
                            float v[8];
#pragma unroll
                            for (int e = 0; e < 8; ++e)
                                v[e] = c0 < p.N ? __ldcg(from + e * kTileM) : 0.0f;
                            ptx::tmem_st_x8(tmem_sum + N_TILE + c0, v);
                        }
                        ptx::tmem_wait_st();
                    }
                }
                ok = __all_sync(0xFFFFFFFFu, wait_bounded_converged(acc_full + 8u * (q & 1), (q >> 1) & 1u, abort_flag, p.status));
                ptx::tc_fence_after_sync();
                // Bias and residual may be the stream's earlier work.  With launch overlap on these warps have not waited for that,
                // but a full accumulator has: it took a B that was loaded after the wait.  (A wait of their own costs 0.6 %.)
                if (i == 0)
                    bias = ok ? bias_of(p, row * kTileM + r) : 0.0f;
                if (!ok || last_chunk)
                    break;
#pragma unroll 1
                for (int c0 = 0; c0 < N_TILE; c0 += 8) {
                    float v[8];
                    read_columns(q, c0, i != 0, v);
                    ptx::tmem_st_x8(tmem_sum + c0, v);
                }
                ptx::tmem_wait_st();
            }
            if (ask && !asked)  // gave up on the way
                complete = other_has_parked(false);
            float* const park = whole || complete ? nullptr
                                                  : p.partial + static_cast<size_t>(N_TILE) * kTileM * (2 * cta + (j == 0 ? 0 : 1)) + r;
            if (ok) {  // the segment's last chunk
#pragma unroll 1
                for (int c0 = 0; c0 < N_TILE; c0 += 8) {
                    float v[8];
                    read_columns(q, c0, i != 0, v);
                    if (complete) {
                        uint32_t t[8];
                        ptx::tmem_ld_x8(tmem_sum + N_TILE + c0, t);
                        ptx::tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            v[e] += __uint_as_float(t[e]);
                    }
                    if (park != nullptr) {
#pragma unroll
                        for (int e = 0; e < 8; ++e)
                            if (c0 + e < p.N)
                                __stcg(park + (c0 + e) * kTileM, v[e]);
                    }
                    else
                        finish_columns<8>(p, v, static_cast<size_t>(c0) * p.M + row * kTileM + r, p.N - c0, bias);
                }
                ++q;
            }
            if (complete) {
                if (tid == 0)
                    p.tile_counters[row] = 0u;  // nobody else touches it again in this launch
            }
            else if (!whole) {
                const bool gave_up = barrier_any(1u, 128u, !ok);
                if (tid == 0) {
                    // arrivals in the low half of the counter; a CTA that gave up also marks the high half, so that the
                    // last one knows the row's sum is not to be trusted
                    const unsigned int mine = gave_up ? 0x10001u : 1u;
                    ptx::grid_dependency_wait();  // (as above)
                    const int          c_first = stream_owner(p, ctas, row_begin);
                    const unsigned int before  = ptx::atom_add_acq_rel_gpu(p.tile_counters + row, mine);
                    if ((before & 0xFFFFu) + 1u == static_cast<unsigned int>(c_last - c_first + 1)) {
                        p.tile_counters[row] = 0u;  // nobody else touches it again in this launch
                        if (((before + mine) >> 16) == 0u) {
                            sums[3 * todo]     = row;
                            sums[3 * todo + 1] = c_first;
                            sums[3 * todo + 2] = c_last;
                            ++todo;
                        }
                    }
                }
            }
        }
        if (tid == 0)
            abort_flag[kLastOfTile] = todo;
    }

    // ================================================================ tear-down, and the sums of rows that became complete here
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (warp == 1)
        ptx::tmem_dealloc(tmem_acc, kTmemCols);
    const unsigned int todo = abort_flag[kLastOfTile];
#pragma unroll 1
    for (unsigned int i = 0; i < todo; ++i) {
        const int row = sums[3 * i], c_first = sums[3 * i + 1], c_last = sums[3 * i + 2];
        // only the row's first CTA may have begun before the row: this is then its last segment, in its second slot
        const int slot = 2 * c_first + (stream_begin(p.stream_share, c_first) < row * p.k_tiles ? 1 : 0);
        sum_row_parts<N_TILE>(p, row, c_first, c_last, p.partial + static_cast<size_t>(N_TILE) * kTileM * slot, threadIdx.x,
                              kStreamWarps * 32);
    }
}

}  // namespace flashllm
