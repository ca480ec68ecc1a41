// Load-as-Sparse / Compute-as-Dense SpMM for sm_100a, wide form: prompt processing, N >= 256.
//
// Decompressing a tile of A costs an SM 400..500 cycles of shared-memory work whatever N is, its MMAs 2 cycles per output
// column.  With 128 columns per CTA every tile is decompressed N / 128 times, and an M128 N128 MMA asks for 128 bytes of
// operands per cycle, all that the shared-memory read path has, so that the 16-bit scatter stores starve behind it.  Here
// a CTA owns one tile row, a range of K tiles and up to 512 output columns (all of tensor memory): a tile is decompressed
// once and multiplied by one or two slabs of B of up to 256 columns (M128 N256: 96 bytes of operands per cycle).
//
//   * warp 0 loads B, one slab [kMmaN x 64] per TMA instruction, in the order the MMAs take them;
//   * warp 1, converged, issues the MMAs of a tile slab by slab; the last one hands the A stage back;
//   * one scatter warp per A stage, as in the streaming form; they are the epilogue warps at the end.
//
// Measured (B200, 80 %, us per call, 128 columns per CTA -> this form): 36864x9216 N = 256 / 384 / 512: 211 / 397 / 408 ->
// 135 / 207 / 223 (1.56 PFLOP/s of dense contraction); 9216x9216: 55 / 103 / 108 -> 45 / 62 / 65; 4736x7232 at 75 %:
// 32 / 44 / 42 -> 29 / 35 / 36.  512 columns are bound by the MMAs (1024 cycles of the 1300 per tile), 256 by the shared-memory path.  Tried
// and not kept: CTA pairs (cta_group::2, M = 256, half of B each), 1..6 % faster where the rows come out even and up to
// 40 % slower where K has to be cut (33 clusters of four fit the GPU, 74 of two).
#pragma once
#include "spmm_kernel_stream_sm100.cuh"

namespace flashllm {

// Columns of one MMA, number of them per tile, A stages (= scatter warps) and B stages for `n_tile` output columns a CTA:
// 224 of the 227 KB of one CTA per SM.  Measured both ways (18944x9216 / 9472x4096 / 2048x8192 at 62..95 %): 384 columns with
// 8 + 4 stages instead of 6 + 5 1..8 % faster (all eight warps share the epilogue), 512 columns with 8 + 3 or 7 + 3 4..15 %
// slower (a slab of B is 512 MMA cycles, three of them less than its way from L2), 256 with 6 + 4 or 4 + 5 up to 20 % slower.
__host__ __device__ constexpr int wide_mma_n(int n_tile) { return n_tile <= 256 ? n_tile : n_tile / 2; }
__host__ __device__ constexpr int wide_slabs(int n_tile) { return n_tile / wide_mma_n(n_tile); }
__host__ __device__ constexpr int wide_a_stages(int n_tile) { return n_tile <= 384 ? 8 : 6; }
__host__ __device__ constexpr int wide_b_stages(int n_tile) { return n_tile == 256 ? 3 : 4; }
// Accumulators that the tiles take turns in.  Two halve the truncated additions of a sum; 384 and 512 columns leave no room
// for a second one (a sum loses 7e-8 of itself per tile in one accumulator): 36864x9216 N = 512 at 80 % is 2.0755e-4 off its exact values in the 2-norm,
// with 256 columns and two accumulators 2.0736e-4 and 29 % slower, where rounding to fp16 alone is 2.0730e-4.
__host__ __device__ constexpr int wide_accumulators(int n_tile) { return n_tile <= 256 ? 2 : 1; }
constexpr int kWideFirstScatter = 2;
constexpr int kWideCap          = 24;  // vectors per lane kept in registers: tiles of up to 62.5 % sparsity

template<int N_TILE, int CAP>
__global__ void __launch_bounds__((kWideFirstScatter + wide_a_stages(N_TILE)) * 32, 1)
    spmm_tcgen05_wide_kernel(const __grid_constant__ CUtensorMap tmap_b, const SpmmParams p)
{
    static_assert(N_TILE == 256 || N_TILE == 384 || N_TILE == 512, "unsupported width");
    constexpr int      kMmaN     = wide_mma_n(N_TILE), kSlabs = wide_slabs(N_TILE);
    constexpr int      STAGES    = wide_a_stages(N_TILE), B_STAGES = wide_b_stages(N_TILE);
    constexpr uint32_t kBSlab    = kMmaN * kTileK * 2;
    constexpr int      kAccs     = wide_accumulators(N_TILE);
    constexpr uint32_t kTmemCols = 512;

    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t base = ptx::smem_u32(smem_raw);  // 1024-byte aligned, checked below
    uint8_t* const smem = smem_raw;

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);  // uniform: the issuing warp stays converged
    const int lane = threadIdx.x & 31;

    // ---- shared memory carve-up
    const uint32_t a_base   = base;
    const uint32_t b_base   = a_base + STAGES * kDenseTileBytes;
    const uint32_t a_full   = b_base + B_STAGES * kBSlab;
    const uint32_t a_empty  = a_full + 8u * STAGES;
    const uint32_t b_full   = a_empty + 8u * STAGES;
    const uint32_t b_empty  = b_full + 8u * B_STAGES;
    const uint32_t acc_full = b_empty + 8u * B_STAGES;
    const uint32_t misc_off = (acc_full + 8u) - base;
    volatile uint32_t* const tmem_slot  = reinterpret_cast<volatile uint32_t*>(smem + misc_off);
    volatile uint32_t* const abort_flag = reinterpret_cast<volatile uint32_t*>(smem + misc_off + 4);
    int* const               offs_stage = reinterpret_cast<int*>(smem + misc_off + 16);  // plan.offsets_staged ints

    // ---- work assignment: blockIdx.x = K part inside the cluster, y = tile row, z = (N tile, workspace part)
    const int S        = p.plan.cluster_k;
    const int G        = p.plan.workspace_k;
    const int rank     = blockIdx.x;
    const int tile_row = blockIdx.y;
    const int g        = blockIdx.z % G;
    const int n_idx    = blockIdx.z / G;
    const int parts    = S * G;
    const int part     = g * S + rank;
    const int k_begin  = static_cast<int>(static_cast<long long>(p.k_tiles) * part / parts);
    const int L        = static_cast<int>(static_cast<long long>(p.k_tiles) * (part + 1) / parts) - k_begin;  // >= 1
    const int* const offs_global = p.tile_offsets + static_cast<long long>(tile_row) * p.k_tiles + k_begin;
    const bool       staged      = (L + 1 <= p.plan.offsets_staged);
    const int* const offs        = staged ? offs_stage : offs_global;  // valid after the set-up barrier

    TileStream<CAP, STAGES> stream;
    const bool              scatters = warp >= kWideFirstScatter;
    const int               sw       = warp - kWideFirstScatter;
    if (scatters) {
        stream.clear();
        if (p.early_weights)
            stream.fetch_first(p, offs_global, sw, L, lane);
    }

    // ---- set-up
    if (threadIdx.x == 0) {
        for (int i = 0; i < STAGES; ++i) {
            ptx::mbar_init(a_full + 8u * i, 1);
            ptx::mbar_init(a_empty + 8u * i, 1);
        }
        for (int i = 0; i < B_STAGES; ++i) {
            ptx::mbar_init(b_full + 8u * i, 1);
            ptx::mbar_init(b_empty + 8u * i, 1);
        }
        ptx::mbar_init(acc_full, 1);
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
    const bool aligned = (base & 1023u) == 0u;
    const bool go      = aligned && !bad_slice;  // false: every role skips its work and no sum leaves this CTA
    if (!go && threadIdx.x == 0) {
        atomicOr(p.status, bad_slice ? kStatusBadTileOffsets : kStatusSmemMisaligned);
        *abort_flag = 1u;
    }
    const uint32_t tmem_acc = *tmem_slot;
    if (threadIdx.x == 0)
        ptx::grid_launch_dependents();

    if (warp == 0) {
        // ================================================================ B loader: slab after slab
        if (lane == 0 && go) {
            ptx::grid_dependency_wait();
            abort_flag[kDepsResolved] = 1u;
            int       bs = 0, issued = 0;
            uint32_t  use   = 0;
            const int slabs = L * kSlabs;
            for (int i = 0; i < slabs; ++i) {
                if (!wait_bounded_relaxed(b_empty + 8u * bs, (use & 1u) ^ 1u, abort_flag, p.status))
                    break;
                ptx::mbar_arrive_expect_tx(b_full + 8u * bs, kBSlab);
                ptx::tma_load_3d(b_base + bs * kBSlab, &tmap_b, 0, n_idx * N_TILE + (i % kSlabs) * kMmaN, k_begin + i / kSlabs,
                                 b_full + 8u * bs);
                ++issued;
                if (++bs == B_STAGES) {
                    bs = 0;
                    ++use;
                }
            }
            if (*abort_flag) {  // copies already issued get a bounded chance to land before the CTA may exit
                const uint64_t t_leave = ptx::globaltimer_ns();
                for (int back = 1; back <= B_STAGES && back <= issued; ++back) {
                    const int bb = issued - back;
                    while (!ptx::mbar_test_wait(b_full + 8u * (bb % B_STAGES), (bb / B_STAGES) & 1u)
                           && ptx::globaltimer_ns() - t_leave < 2000000ull) {}
                }
            }
        }
        __syncwarp();
    }
    else if (warp == 1) {
        // ================================================================ MMA issuer (converged warp)
        if (go) {
            const uint32_t idesc   = ptx::umma_idesc_f16_f32(kTileM, kMmaN);
            const uint64_t a_desc0 = ptx::umma_desc_kmajor_sw128(a_base);
            const uint64_t b_desc0 = ptx::umma_desc_kmajor_sw128(b_base);
            int            s = 0, bs = 0;
            uint32_t       a_par = 0, b_par = 0;
            bool           ok = true;
            for (int j = 0; ok && j < L; ++j) {
                ok = __all_sync(0xFFFFFFFFu, wait_bounded_converged(a_full + 8u * s, a_par, abort_flag, p.status));
#pragma unroll
                for (int h = 0; h < kSlabs; ++h) {
                    ok = ok && __all_sync(0xFFFFFFFFu, wait_bounded_converged(b_full + 8u * bs, b_par, abort_flag, p.status));
                    if (!ok)
                        break;
                    ptx::tc_fence_after_sync();
                    // hands the B slab back, and with the tile's last slab the A stage
                    ptx::umma_tile_elect(tmem_acc + static_cast<uint32_t>(j % kAccs * N_TILE + h * kMmaN),
                                         a_desc0 + static_cast<uint32_t>(s * (kDenseTileBytes >> 4)),
                                         b_desc0 + static_cast<uint32_t>(bs * (kBSlab >> 4)), idesc, j >= kAccs ? 1u : 0u,
                                         b_empty + 8u * bs, a_empty + 8u * s, h + 1 == kSlabs ? 1u : 0u);
                    if (++bs == B_STAGES) {
                        bs = 0;
                        b_par ^= 1u;
                    }
                }
                if (++s == STAGES) {
                    s = 0;
                    a_par ^= 1u;
                }
            }
            if (ok)
                ptx::umma_commit_elect(acc_full);
        }
    }
    else {
        // ================================================================ scatter warps, then the epilogue
        bool acc_ok = go;
        if (go) {
            stream.run(p, offs, sw, L, lane, a_base + sw * kDenseTileBytes, a_full + 8u * sw, a_empty + 8u * sw, abort_flag);
            acc_ok = wait_bounded_warp(acc_full, 0u, abort_flag, p.status);
        }
        acc_ok = __all_sync(0xFFFFFFFFu, acc_ok && (*abort_flag == 0u));
        ptx::tc_fence_after_sync();
        accumulators_to_output<N_TILE, 32>(p, tmem_acc, L < kAccs ? L : kAccs, N_TILE, warp & 3, lane, sw, STAGES >= 8 ? 2 : 1, S, G,
                                           g, n_idx, tile_row, acc_ok, reinterpret_cast<float*>(smem));
    }

    // ================================================================ cluster reduction and tear-down
    ptx::tc_fence_before_sync();
    __syncthreads();
    if (S > 1) {
        ptx::cluster_sync_all();  // every CTA's partial tile is parked in its shared memory
        if (scatters)
            cluster_reduce_store<N_TILE>(p, base, rank, S, G, g, n_idx, tile_row, threadIdx.x - kWideFirstScatter * 32, STAGES * 32,
                                         *abort_flag == 0u);
        __syncwarp();
        ptx::cluster_sync_all();  // nobody leaves while a peer may still read its shared memory
    }
    if (warp == 1)
        ptx::tmem_dealloc(tmem_acc, kTmemCols);
}

}  // namespace flashllm
