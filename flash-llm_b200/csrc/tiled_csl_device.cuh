// Device tiled-CSL encoder: dense fp16 A in HBM -> TileOffsets and packed words, bit-identical to the host encoder
// and therefore to the reference's InitSparseMatrixA_API / _NoReorder (reference csrc/SpMM_API.cu:163-489).
//
// One warp encodes one 128x64 tile.  For the reordered format lane k owns shared-memory bank k of the decompressed
// tile: the two cells (r, 2k ^ ((r&7)<<3)) and the one after it in every row r, which is exactly the reference's
// bucket k in its row-major scan order (:248-271).  The reference's greedy deal (always pop the newest word of the
// fullest bucket, :299-320) is a level-order walk over bucket heights, so the word at height h of bucket k is pick
//     q = sum_k' max(0, c[k'] - h) + #{k' < k : c[k'] >= h}
// and the two lane-queue passes (:323-346) map q to a fixed slot.
//
// Bound by HBM: the dense matrix has to be read twice, because the size of the result is only known after the first pass.
// 36864x9216 at 80 % (680 MB dense, 272 MB of words), both passes with the host's wait and
// the allocation between them: 322 us (906 with every tile read twice and its words stored one by one); counting alone
// 113 us, 6.0 TB/s.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "ptx_sm100.cuh"
#include "tiling.h"

namespace flashllm {

constexpr unsigned kStatusOffsetsOverflow  = 4u;  // more 16-byte vectors than an int can count
constexpr unsigned kStatusOffsetsMismatch  = 8u;  // TileOffsets do not match the matrix being packed

constexpr int kEncodeWarps   = 8;
constexpr int kHeightEntries = kTileM * kTileK / 32 + kVectorWords + 1;  // bucket heights 0..259

__device__ __forceinline__ bool keeps_cell(uint32_t h16)
{
    const uint32_t a = h16 & 0x7FFFu;  // the reference keeps finite non-zeros and infinities, drops +-0 and NaN
    return a != 0u && a <= 0x7C00u;
}

__device__ __forceinline__ uint32_t lanemask_lt()
{
    uint32_t m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// Output slot of the q-th pick of the reference's deal, inside a tile of `vectors` 16-byte vectors.
__device__ __forceinline__ int slot_of_pick(int q, int vectors)
{
    const int repeat = vectors >> 5, remain = vectors & 31;
    if (q < 4 * remain) {
        const int v = q / remain, b = q - v * remain;
        return repeat * 128 + b * 4 + (3 - v);
    }
    const int qm   = q - 4 * remain;
    const int push = qm >> 5, b = qm & 31;
    const int w    = 4 * repeat - 1 - push;
    return (w >> 2) * 128 + b * 4 + (w & 3);
}

// The cells of a pair that keeps_cell would keep, as 1.0 / 0.0: not equal to zero and not NaN.
__device__ __forceinline__ uint32_t kept_pair(uint32_t pair)
{
    uint32_t d;
    asm("set.ne.f16x2.f16x2 %0, %1, %2;" : "=r"(d) : "r"(pair), "r"(0u));
    return d;
}

__device__ __forceinline__ uint32_t add_f16x2(uint32_t a, uint32_t b)
{
    uint32_t d;
    asm("add.f16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

__device__ __forceinline__ const uint16_t* tile_start(const uint16_t* A, int K, int k_tiles, int t)
{
    return A + static_cast<size_t>(t / k_tiles) * kTileM * K + static_cast<size_t>(t % k_tiles) * kTileK;
}

// Step 1a: offs[t + 1] = 16-byte vectors (non-zeros rounded up to a multiple of four) of tile t and of the tiles before it
// in its CTA's group of kCountTiles.  A warp counts a quarter of the rows of four neighbouring tiles, eight lanes to a tile and
// 16 bytes to a lane, so that it reads 512 bytes of a row in one piece; counts are kept in fp16 pairs, exact up to 2048 and
// never above 128 here.  (With one warp to all rows of its tiles the counts of 1024x1024 took eight memory latencies in a row:
// both launches of this step 12.2 us, in quarters 8.0; an encoding of 36864x9216 in all 326 -> 323.)
constexpr int kCountTiles = 32, kCountRowParts = 4, kCountWarps = kCountTiles / 4 * kCountRowParts;

__global__ void __launch_bounds__(kCountWarps * 32)
    csl_count_kernel(const uint16_t* A, int K, int tiles, int k_tiles, int* offs)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    __shared__ int s_words[kCountRowParts][kCountTiles];
    static_assert(kCountTiles == 32, "one lane per tile of the group");
    constexpr int kRows = kTileM / kCountRowParts;
    const int lane = threadIdx.x & 31, part = (threadIdx.x >> 5) % kCountRowParts;
    const int slot = (threadIdx.x >> 5) / kCountRowParts * 4 + (lane >> 3);
    const int t    = blockIdx.x * kCountTiles + slot;
    uint32_t  n2   = 0;
    if (t < tiles) {
        const uint16_t* src   = tile_start(A, K, k_tiles, t) + static_cast<size_t>(part * kRows) * K + (lane & 7) * 8;
        auto            count = [&](uint4 v) {
            n2 = add_f16x2(n2, add_f16x2(add_f16x2(kept_pair(v.x), kept_pair(v.y)), add_f16x2(kept_pair(v.z), kept_pair(v.w))));
        };
        if ((reinterpret_cast<uintptr_t>(A) & 15u) == 0) {
#pragma unroll 16
            for (int r = 0; r < kRows; ++r)
                count(*reinterpret_cast<const uint4*>(src + static_cast<size_t>(r) * K));
        }
        else {  // A is 4-byte aligned
#pragma unroll 4
            for (int r = 0; r < kRows; ++r) {
                const uint32_t* row = reinterpret_cast<const uint32_t*>(src + static_cast<size_t>(r) * K);
                count(make_uint4(row[0], row[1], row[2], row[3]));
            }
        }
    }
    const __half2 h = *reinterpret_cast<const __half2*>(&n2);
    int           n = static_cast<int>(__low2float(h)) + static_cast<int>(__high2float(h));
    for (int d = 1; d < 8; d <<= 1)
        n += __shfl_xor_sync(0xFFFFFFFFu, n, d);
    if ((lane & 7) == 0)
        s_words[part][slot] = n;
    __syncthreads();
    if (threadIdx.x < 32) {
        int words = 0;
#pragma unroll
        for (int i = 0; i < kCountRowParts; ++i)
            words += s_words[i][lane];
        int v = (words + kVectorWords - 1) / kVectorWords;
        for (int d = 1; d < 32; d <<= 1) {
            const int below = __shfl_up_sync(0xFFFFFFFFu, v, d);
            v += lane >= d ? below : 0;
        }
        const int mine = blockIdx.x * kCountTiles + lane;
        if (mine < tiles)
            offs[mine + 1] = v;
    }
}

// Step 1b: adds to every entry the sums of the groups before its own; offs[0] = 0, offs[tiles + 1] = offs[tiles].  One CTA,
// 1024 groups at a time: it scans the groups' sums and then runs over their entries.
__global__ void __launch_bounds__(1024) csl_scan_kernel(int* offs, int tiles, unsigned int* status)
{
    // No launch_dependents, here and in the kernels that end an encoding: an SpMM with launch overlap on that follows reads
    // offsets and words before its own wait.
    ptx::grid_dependency_wait();
    __shared__ int       s_before[1024];  // sum of the groups before this one
    __shared__ long long s_warp[32];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int groups = (tiles + kCountTiles - 1) / kCountTiles;
    long long done   = 0;  // sum of the groups of earlier rounds
    for (int g0 = 0; g0 < groups; g0 += 1024) {
        const int       g   = g0 + tid;
        const long long end = (static_cast<long long>(g) + 1) * kCountTiles;
        const int       sum = g < groups ? offs[end < tiles ? end : tiles] : 0;
        long long       upto = sum;  // inclusive
        for (int d = 1; d < 32; d <<= 1) {
            const long long below = __shfl_up_sync(0xFFFFFFFFu, upto, d);
            upto += lane >= d ? below : 0;
        }
        if (lane == 31)
            s_warp[warp] = upto;
        __syncthreads();
        long long base = done;
        for (int w = 0; w < 32; ++w) {
            base += w < warp ? s_warp[w] : 0;
            done += s_warp[w];
        }
        s_before[tid] = static_cast<int>(base + upto - sum);
        __syncthreads();
        const int first = g0 * kCountTiles, last = tiles - first < 1024 * kCountTiles ? tiles : first + 1024 * kCountTiles;
#pragma unroll 8
        for (int i = first + tid; i < last; i += 1024)
            offs[i + 1] += s_before[(i - first) / kCountTiles];
        __syncthreads();  // s_before and s_warp may be written again
    }
    if (tid == 0) {
        if (done > 0x7FFFFFFFll)
            atomicOr(status, kStatusOffsetsOverflow);
        offs[0]         = 0;
        offs[tiles + 1] = static_cast<int>(done);
    }
    __threadfence();  // the offsets are in place for whatever starts once this grid has ended
}

// Step 2, reordered format, tiles with buckets of any height: counts, tabulates the per-height terms of q in shared
// memory (s_mask: buckets at least this high; s_above: words lying above this height), reads the tile again and places
// every word on its own.
__device__ __forceinline__ void pack_any_tile(const uint16_t* __restrict__ tile, int K, int vectors, uint32_t* __restrict__ dst,
                                              uint32_t* s_mask, uint16_t* s_above, int lane, unsigned int* status)
{
    const int words = vectors * kVectorWords;
    // pass 1: bucket sizes and each bucket's first zero cell
    int count = 0, zero_loc = -1;
#pragma unroll 8
    for (int r = 0; r < kTileM; ++r) {
        const int      x    = (r & 7) << 3;
        const int      c0   = (2 * lane) ^ x;  // the bucket's two cells sit at columns c0, c0 + 1
        const uint32_t pair = *reinterpret_cast<const uint32_t*>(tile + static_cast<size_t>(r) * K + c0);
        const bool     k0 = keeps_cell(pair & 0xFFFFu), k1 = keeps_cell(pair >> 16);
        count += (k0 ? 1 : 0) + (k1 ? 1 : 0);
        if (zero_loc < 0 && !(k0 && k1))
            zero_loc = r * kTileK + 2 * lane + (k0 ? 1 : 0);
    }
    const int nnz  = __reduce_add_sync(0xFFFFFFFFu, count);
    const int pads = words - nnz;
    if (pads < 0 || pads >= kVectorWords || vectors < 0 || vectors > kMaxTileVectors) {
        if (lane == 0)
            atomicOr(status, kStatusOffsetsMismatch);
        return;
    }
    // padding words join the emptiest bucket, one at a time, lowest bucket on ties
    int total = count;
    for (int p = 0; p < pads; ++p) {
        const unsigned best = __reduce_min_sync(0xFFFFFFFFu, (static_cast<unsigned>(total) << 5) | lane);
        if ((best & 31u) == static_cast<unsigned>(lane))
            ++total;
    }
    const int top = __reduce_max_sync(0xFFFFFFFFu, total);
    // per-height tables, from the top down
    int running = 0;
    for (int h = top; h >= 1; --h) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, total >= h);
        if (lane == 0) {
            s_mask[h]  = m;
            s_above[h] = static_cast<uint16_t>(running);
        }
        running += __popc(m);
    }
    __syncwarp();
    const uint32_t lower = lanemask_lt();

    // pass 2: place every word
    int h = 0;
#pragma unroll 8
    for (int r = 0; r < kTileM; ++r) {
        const int      x    = (r & 7) << 3;
        const int      c0   = (2 * lane) ^ x;
        const uint32_t pair = *reinterpret_cast<const uint32_t*>(tile + static_cast<size_t>(r) * K + c0);
        const uint32_t v0 = pair & 0xFFFFu, v1 = pair >> 16;
        if (keeps_cell(v0)) {
            ++h;
            const int q             = s_above[h] + __popc(s_mask[h] & lower);
            dst[slot_of_pick(q, vectors)] = v0 | (static_cast<uint32_t>(r * kTileK + 2 * lane) << 16);
        }
        if (keeps_cell(v1)) {
            ++h;
            const int q             = s_above[h] + __popc(s_mask[h] & lower);
            dst[slot_of_pick(q, vectors)] = v1 | (static_cast<uint32_t>(r * kTileK + 2 * lane + 1) << 16);
        }
    }
    for (; h < total;) {  // this bucket's padding words: +0.0 at its first zero cell
        ++h;
        const int q                   = s_above[h] + __popc(s_mask[h] & lower);
        dst[slot_of_pick(q, vectors)] = static_cast<uint32_t>(zero_loc) << 16;
    }
}

__device__ __noinline__ void pack_tall_tile(const uint16_t* tile, int K, int vectors, uint32_t* dst, uint32_t* s_mask,
                                            uint16_t* s_above, int lane, unsigned int* status)
{
    pack_any_tile(tile, K, vectors, dst, s_mask, s_above, lane, status);
}

// The tiles of more than kListVectors vectors, which csl_pack_reorder_kernel leaves out: a matrix of such tiles wants
// more warps per SM than that kernel's shared memory allows.  Persistent, so that it costs 4 to 9 us where there are none.
constexpr int kListVectors = 1088;  // 136 words to a bucket: hardly ever one above 164

__global__ void __launch_bounds__(kEncodeWarps * 32) csl_pack_dense_kernel(const uint16_t* A,
                                                                           int K,
                                                                           int tiles,
                                                                           int k_tiles,
                                                                           const int* offs,
                                                                           uint32_t* out,
                                                                           unsigned int* status)
{
    ptx::grid_launch_dependents();
    ptx::grid_dependency_wait();
    __shared__ uint32_t s_mask[kEncodeWarps][kHeightEntries];
    __shared__ uint16_t s_above[kEncodeWarps][kHeightEntries];
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int t = blockIdx.x * kEncodeWarps + w; t < tiles; t += gridDim.x * kEncodeWarps) {
        const int first = offs[t], vectors = offs[t + 1] - first;
        if (vectors > kListVectors) {
            pack_any_tile(tile_start(A, K, k_tiles, t), K, vectors, out + static_cast<size_t>(first) * kVectorWords, s_mask[w],
                          s_above[w], lane, status);
            __syncwarp();
        }
    }
}

// Step 2, reordered format.
//
// A lane appends its bucket's words to a column of shared memory, the newest on top (height h in row kListRows - h: bank =
// lane, no conflicts).  From the height of the lowest bucket down every level holds 32 words, which already lie in pick
// order; only the levels above it are walked, top first, and their words moved to the front of the same memory (a level
// is read before anything can be written over it).  The words then leave as whole 16-byte vectors.
//
// The grid is persistent: while the words of a tile are dealt and stored, the next one is on its way into registers and the
// one after it into L2.  Bound by its own instructions (0.59 of the issue slots, hardly a stall on memory): the lists take
// the shared memory that more warps would need, and L1 needs what they leave for the loads in flight.  us per 36864x9216
// pack at 80 %: six CTAs per SM 244, five 224, four 210, four with the L2 prefetch 195, three 241 (lists of 140 rows).
constexpr int kPackWarps = 2, kPackCtasPerSm = 4;
constexpr int kListRows = 168, kSpareRows = 8;  // 44 KB of shared memory per CTA: the buckets of tiles of 50 % sparsity and more
constexpr int kPackCarveoutPercent = 82;        // of 228 KB: kPackCtasPerSm CTAs and 1 KB for each

// This lane's pair of cells of every row: bucket `lane` owns columns c0, c0 + 1 with c0 = 2 * lane ^ ((r & 7) << 3).
__device__ __forceinline__ void load_bucket(uint32_t (&pair)[kTileM], const uint16_t* tile, int K, int lane)
{
#pragma unroll
    for (int r = 0; r < kTileM; ++r) {
        pair[r] = *reinterpret_cast<const uint32_t*>(tile + ((2 * lane) ^ ((r & 7) << 3)));
        tile += K;
    }
}

// Asks for a tile's rows (128 bytes each, at most two lines of L2) to be in L2 when load_bucket comes for them.
__device__ __forceinline__ void prefetch_tile(const uint16_t* tile, int K, int lane)
{
#pragma unroll
    for (int r = 0; r < kTileM; r += 32)
        asm volatile("prefetch.global.L2 [%0];" ::"l"(tile + static_cast<size_t>(r + lane) * K));
}

__global__ void __launch_bounds__(kPackWarps * 32, kPackCtasPerSm) csl_pack_reorder_kernel(const uint16_t* A,
                                                                                           int K,
                                                                                           int tiles,
                                                                                           int k_tiles,
                                                                                           const int* offs,
                                                                                           uint32_t* out,
                                                                                           unsigned int* status)
{
    ptx::grid_dependency_wait();  // no launch_dependents (see csl_scan_kernel)
    // spare rows in front: words beyond kListRows land there
    __shared__ uint32_t s_list[kPackWarps][(kListRows + kSpareRows) * 32];
    static_assert(sizeof(s_list[0]) >= kHeightEntries * (sizeof(uint32_t) + sizeof(uint16_t)), "tables of a tall tile");
    const int       w      = threadIdx.x >> 5;
    const int       lane   = threadIdx.x & 31;
    uint32_t* const list   = s_list[w];
    uint32_t* const lists  = list + kSpareRows * 32;  // row kListRows - h holds height h
    const uint32_t  bottom = ptx::smem_u32(list) + (kListRows + kSpareRows - 1) * 128 + lane * 4;
    const uint32_t  limit  = ptx::smem_u32(list) + kSpareRows * 128 + lane * 4;
    const int       stride = static_cast<int>(gridDim.x) * kPackWarps;
    const uint32_t  lower  = lanemask_lt();
    const bool      wide   = (reinterpret_cast<uintptr_t>(out) & 15u) == 0;
    uint32_t        pair[kTileM];
    // last tiles first: the counting pass has just read them and L2 still holds the end of the matrix
    int t = tiles - 1 - (static_cast<int>(blockIdx.x) * kPackWarps + w);
    auto vectors_of = [&](int tile) { return tile >= 0 ? offs[tile + 1] - offs[tile] : kListVectors + 1; };
    int  vectors = vectors_of(t), vectors1 = vectors_of(t - stride);  // of this tile and the next one
    if (vectors <= kListVectors)
        load_bucket(pair, tile_start(A, K, k_tiles, t), K, lane);
    for (int vectors2; t >= 0; t -= stride, vectors = vectors1, vectors1 = vectors2) {
        vectors2 = vectors_of(t - 2 * stride);
        if (vectors > kListVectors) {  // csl_pack_dense_kernel's
            if (vectors1 <= kListVectors)
                load_bucket(pair, tile_start(A, K, k_tiles, t - stride), K, lane);
            continue;
        }
        const int       first = offs[t];
        const int       words = vectors * kVectorWords;
        uint32_t* const dst   = out + static_cast<size_t>(first) * kVectorWords;

        // ---- the bucket's words, oldest in the last row
        __syncwarp();  // the previous tile's words have been read
        uint32_t at  = bottom;                           // where the next word goes
        uint32_t loc = static_cast<uint32_t>(2 * lane) * 0x10001u + 0x10000u;  // of the row's two cells, low half first
#pragma unroll
        for (int r = 0; r < kTileM; ++r) {
            const uint32_t w0 = __byte_perm(pair[r], loc, 0x5410), w1 = __byte_perm(pair[r], loc, 0x7632);
            if (r % (kSpareRows / 2) == 0)  // at most kSpareRows words until the next look
                at = static_cast<int>(at) > static_cast<int>(limit) ? at : limit;
            // (a position that a store has yet to read cannot be overwritten: it moves on through fresh registers)
            uint32_t at1, at2;
            asm volatile(
                "{\n"
                ".reg .pred p, q;\n"
                ".reg .u32 s, t;\n"
                "setp.ne.f16x2 p|q, %3, %6;\n"
                "selp.u32 s, 128, 0, p;\n"
                "selp.u32 t, 128, 0, q;\n"
                "sub.u32 %0, %2, s;\n"
                "sub.u32 %1, %0, t;\n"
                "@p st.shared.u32 [%2], %4;\n"
                "@q st.shared.u32 [%0], %5;\n"
                "}\n"
                : "=&r"(at1), "=&r"(at2)
                : "r"(at), "r"(pair[r]), "r"(w0), "r"(w1), "r"(0u)
                : "memory");
            at = at2;
            loc += kTileK * 0x10001u;
        }
        if (vectors1 <= kListVectors)
            load_bucket(pair, tile_start(A, K, k_tiles, t - stride), K, lane);
        if (vectors2 <= kListVectors)
            prefetch_tile(tile_start(A, K, k_tiles, t - 2 * stride), K, lane);
        const int count = static_cast<int>(bottom - at) >> 7;
        if (__any_sync(0xFFFFFFFFu, count > kListRows - kVectorWords)) {  // (a column that overflowed counts at least kListRows - 1)
            __syncwarp();
            pack_tall_tile(tile_start(A, K, k_tiles, t), K, vectors, dst, list, reinterpret_cast<uint16_t*>(list + kHeightEntries),
                           lane, status);
            continue;
        }
        const int nnz  = __reduce_add_sync(0xFFFFFFFFu, count);
        const int pads = words - nnz;
        if (pads < 0 || pads >= kVectorWords || vectors < 0 || vectors > kMaxTileVectors) {
            if (lane == 0)
                atomicOr(status, kStatusOffsetsMismatch);
            continue;
        }
        // padding words join the emptiest bucket, one at a time, lowest bucket on ties: +0.0 at the bucket's first zero cell
        int total = count;
        for (int p = 0; p < pads; ++p) {
            const unsigned best = __reduce_min_sync(0xFFFFFFFFu, (static_cast<unsigned>(total) << 5) | lane);
            if ((best & 31u) == static_cast<unsigned>(lane))
                ++total;
        }
        if (total > count) {
            int cell = 0;  // in the bucket's scan order; the words lie in that order, so the first gap is the first zero cell
            while (cell < count) {
                const uint32_t l = lists[(kListRows - 1 - cell) * 32 + lane] >> 16;
                if (static_cast<int>(((l >> 6) << 1) | (l & 1u)) != cell)
                    break;
                ++cell;
            }
            const uint32_t zero_loc = static_cast<uint32_t>((cell >> 1) * kTileK + 2 * lane + (cell & 1));
            for (int h = count + 1; h <= total; ++h)
                lists[(kListRows - h) * 32 + lane] = zero_loc << 16;
        }
        const int top  = __reduce_max_sync(0xFFFFFFFFu, total);
        const int full = __reduce_min_sync(0xFFFFFFFFu, total);  // levels 1 .. full hold 32 words each
        __syncwarp();
        // ---- the levels above, in pick order, to the front
        int           above = 0;
        constexpr int H     = 4;  // levels at a time: all read, then moved
        for (int h0 = top; h0 > full; h0 -= H) {
            uint32_t word[H], m[H];
#pragma unroll
            for (int i = 0; i < H; ++i) {
                const int  h    = h0 - i;
                const bool mine = h > full && total >= h;
                m[i]            = __ballot_sync(0xFFFFFFFFu, mine);
                word[i]         = mine ? lists[(kListRows - h) * 32 + lane] : 0u;
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < H; ++i) {
                if ((m[i] >> lane) & 1u)
                    lists[above + __popc(m[i] & lower)] = word[i];
                above += __popc(m[i]);
            }
        }
        __syncwarp();
        // ---- pick q lies at lists[q], or from the full levels on at lists[q + skip]
        const int skip = (kListRows - full) * 32 - above;
        auto      pick = [&](int q) { return lists[q < above ? q : q + skip]; };
        const int repeat = vectors >> 5, remain = vectors & 31;
        auto      put  = [&](int vector, uint4 v) {
            uint32_t* const to = dst + vector * kVectorWords;
            if (wide)
                *reinterpret_cast<uint4*>(to) = v;
            else {
                to[0] = v.x;
                to[1] = v.y;
                to[2] = v.z;
                to[3] = v.w;
            }
        };
        if (lane < remain)
            put(repeat * 32 + lane, make_uint4(pick(3 * remain + lane), pick(2 * remain + lane), pick(remain + lane), pick(lane)));
        int q = 4 * remain + lane;
#pragma unroll 4
        for (int i = repeat - 1; i >= 0; --i, q += 128)
            put(i * 32 + lane, make_uint4(pick(q + 96), pick(q + 64), pick(q + 32), pick(q)));
    }
    __threadfence();  // the words are in place for whatever starts once this grid has ended
}

// Step 2, scan-order format (reference csrc/SpMM_API.cu:441-476): non-zeros in row-major order, with the first
// `pads` zero-testing cells of the tile kept in place as padding words (their bits preserved).
__device__ __forceinline__ void pack_scan_tile(const uint16_t* __restrict__ tile, int K, int words, uint32_t* __restrict__ dst,
                                               int lane, unsigned int* status)
{
    int nnz = 0;
#pragma unroll 8
    for (int r = 0; r < kTileM; ++r) {
        const uint32_t pair = *reinterpret_cast<const uint32_t*>(tile + static_cast<size_t>(r) * K + 2 * lane);
        nnz += (keeps_cell(pair & 0xFFFFu) ? 1 : 0) + (keeps_cell(pair >> 16) ? 1 : 0);
    }
    nnz            = __reduce_add_sync(0xFFFFFFFFu, nnz);
    const int pads = words - nnz;
    if (pads < 0 || pads >= kVectorWords) {
        if (lane == 0)
            atomicOr(status, kStatusOffsetsMismatch);
        return;
    }
    const uint32_t lower   = lanemask_lt();
    int            emitted = 0, zeros = 0;
    for (int r = 0; r < kTileM; ++r) {
        const int      x    = (r & 7) << 3;
        const uint32_t pair = *reinterpret_cast<const uint32_t*>(tile + static_cast<size_t>(r) * K + 2 * lane);
        const uint32_t v0 = pair & 0xFFFFu, v1 = pair >> 16;
        const bool     k0 = keeps_cell(v0), k1 = keeps_cell(v1);
        bool           e0 = k0, e1 = k1;
        if (zeros < pads) {  // some padding still to place: rank the zero cells of this row
            const uint32_t z0 = __ballot_sync(0xFFFFFFFFu, !k0), z1 = __ballot_sync(0xFFFFFFFFu, !k1);
            const int      zr = zeros + __popc(z0 & lower) + __popc(z1 & lower);
            e0                = k0 || (zr < pads);
            e1                = k1 || (zr + (k0 ? 0 : 1) < pads);
            zeros += __popc(z0) + __popc(z1);
        }
        const uint32_t b0 = __ballot_sync(0xFFFFFFFFu, e0), b1 = __ballot_sync(0xFFFFFFFFu, e1);
        int            pos = emitted + __popc(b0 & lower) + __popc(b1 & lower);
        if (e0)
            dst[pos++] = v0 | (static_cast<uint32_t>(r * kTileK + ((2 * lane) ^ x)) << 16);
        if (e1)
            dst[pos] = v1 | (static_cast<uint32_t>(r * kTileK + ((2 * lane + 1) ^ x)) << 16);
        emitted += __popc(b0) + __popc(b1);
    }
}

__global__ void __launch_bounds__(kEncodeWarps * 32) csl_pack_scan_kernel(const uint16_t* A,
                                                                          int K,
                                                                          int tiles,
                                                                          int k_tiles,
                                                                          const int* offs,
                                                                          uint32_t* out,
                                                                          unsigned int* status)
{
    ptx::grid_dependency_wait();  // no launch_dependents (see csl_scan_kernel)
    const int lane = threadIdx.x & 31;
    const int t    = blockIdx.x * kEncodeWarps + (threadIdx.x >> 5);
    if (t >= tiles)
        return;
    const int first = offs[t];
    pack_scan_tile(tile_start(A, K, k_tiles, t), K, (offs[t + 1] - first) * kVectorWords,
                   out + static_cast<size_t>(first) * kVectorWords, lane, status);
    __threadfence();
}

}  // namespace flashllm
