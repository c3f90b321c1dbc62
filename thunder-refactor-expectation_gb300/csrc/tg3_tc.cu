// tg3_tc.cu -- the likelihood cross term on the 5th-generation tensor cores.
//
// C[b][i][j] = alpha * sum_k A[b][i][k] B[b][j][k] + nrm[b][i], with each FP32
// operand stored as two bf16 planes, hi = bf16(x) and lo = bf16(x - hi), and
// the product formed as Ah Bh + Ah Bl + Al Bh (the lo x lo term, ~2^-16 of
// the product, is dropped), accumulated in FP32 in tensor memory.
//
// A tile is (128 rows of A, batch item); N (<= 256) columns in one UMMA of
// shape 128 x N x 16.  One CTA an SM walks the tiles, 320 threads:
//   warp 0 lane 0 : TMA producer (cp.async.bulk.tensor),
//   warp 1 lane 0 : tcgen05.mma issuer, commits to the stage's empty barrier,
//   warps 2-9     : epilogue (tcgen05.ld 32x32b, + nrm, store), two warps to a
//                   quarter of the rows, alternate 32 columns each.
// Two accumulators in tensor memory: while the epilogue drains one, the MMAs
// of the next tile fill the other and the copies run ahead of both.  (With a
// CTA per tile the set-up, the pipeline's fill and the epilogue stood between
// the tiles' products: 4.8 ms for 6,912 x 98,000 x 768, the short K of a box-64
// search, where they are most of a tile; now 2.1 ms, 1.5 PFLOP/s executed.)
// Every mbarrier wait is bounded (clock64 budget); on expiry the CTA records
// TG3 flag bit 4, stops issuing, waits (bounded) for its own copies and MMAs,
// frees its tensor memory and returns.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "tg3_internal.cuh"
#include "tg3_tcgen05.cuh"

namespace tg3 {

namespace {

using namespace tc;

constexpr int TC_M = 128;          // rows of A per CTA (UMMA M)
constexpr int TC_BK = 64;          // bf16 elements per K block (one 128-byte row)
constexpr int TC_EPI = 8;            // epilogue warps
constexpr int TC_THREADS = 64 + 32 * TC_EPI;
constexpr int TC_PITCH = 36;         // row pitch of the transposition buffer (16-byte rows, no conflicts)
constexpr int TC_SEGS = 8;           // column groups of a tile whose norms are fetched ahead
constexpr int TC_ROWS = 8;           // rows of it
constexpr int TC_STAGE = TC_ROWS * TC_PITCH;
struct TcParams {
    int M, N, Kd;            // rows of A per item, columns (rows of B) per item, K
    int aRowsPerItem;        // A row offset between items (0: A shared by all items)
    int bRowsPerItem;        // B row offset between items
    int nTotal;              // > 0: columns of the whole problem (the last item is partial)
    int colPerItem;          // column offset between items (column-group remap)
    int cGroup;              // > 0: column j goes to group j / cGroup, position j % cGroup
    long long cGroupStride;  // element stride between column groups
    int ntile;               // N rounded up to 16 (the UMMA N)
    int tmemCols;            // power of two >= ntile
    int stages;
    float* C;
    long long sC;
    int ldc;
    const float* nrm;
    long long sN;
    float alpha;
    int* flag;
    // with best: the largest C + norm of every (column group, group of rows),
    // as ordered ints (float_key): best[l bestGroups + row / bestRows], the norm
    // of row r in column group l at bestNrm[r bestNs + l]
    int* best;
    int bestRows, bestGroups;
    const float* bestNrm;
    int bestNs;
    int mTiles, tiles;       // row tiles of an item, tiles of the problem
};

// K-major operand descriptors: 128-byte rows with the 128-byte swizzle
// (K blocks of 64 bf16) or 64-byte rows with the 64-byte swizzle (K blocks
// of 32, half the stage bytes and so twice the stages in flight).
template <int BK>
__device__ __forceinline__ uint64_t desc(uint32_t saddr)
{
    return BK == 64 ? umma_desc(saddr) : umma_desc_sw64(saddr);
}

// The norms that a warp's rows need for the tile's first TC_SEGS column
// groups, lane = row, fetched before the tile's products are waited for.
__device__ __forceinline__ void load_norms(const TcParams& p, float* ad, int lane, int rowBase,
                                           int item, int nValid)
{
    const int j0 = item * p.colPerItem;
    const int l0 = j0 / p.cGroup, l1 = (j0 + nValid - 1) / p.cGroup;
    const float* src = p.bestNrm + (size_t)min(rowBase + lane, p.M - 1) * p.bestNs + l0;
    for (int k = 0; k < min(l1 - l0 + 1, TC_SEGS); k++) ad[k * 32 + lane] = src[k];
}

// Largest value of each of the chunk's column groups (columns c0 .. c0 + cn - 1
// of the tile, v[] of this lane's row) with the row's norm, then over the
// warp's rows of every row group, into best.  fl(x + norm) grows with x, so the
// norm is added to the largest x only.  A sum that is not a number is no maximum
// (fmaxf over the columns skips one, and so does the weights' own pass).
__device__ __forceinline__ void chunk_best(const TcParams& p, const float* v, int cn, const float* ad,
                                           int lane, int rowBase, int rows, int j0, int c0)
{
    const bool rowOk = lane < rows;
    const int row = rowBase + lane;
    const int g0 = rowBase / p.bestRows, g1 = (rowBase + rows - 1) / p.bestRows;
    const int g = rowOk ? row / p.bestRows : -1;
    const int lTile = j0 / p.cGroup;
    int l = (j0 + c0) / p.cGroup;
    auto put = [&](float m) {                                   // m: group l's largest of the row
        const float n = l - lTile < TC_SEGS ? ad[(l - lTile) * 32 + lane]
                                            : p.bestNrm[(size_t)min(row, p.M - 1) * p.bestNs + l];
        const float sum = m + n;
        const int key = sum == sum ? float_key(sum) : kFloatKeyNegInf;
        for (int k = g0; k <= g1; k++) {
            const int top = __reduce_max_sync(0xffffffffu, g == k ? key : kFloatKeyNegInf);
            if (lane == 0) atomicMax(p.best + (size_t)l * p.bestGroups + k, top);
        }
    };
    int end = (l + 1) * p.cGroup - (j0 + c0);                   // group l's end in the chunk
    if (end >= cn && cn == 32) {                                // one group
        float m = v[0];
#pragma unroll
        for (int i = 1; i < 32; i++) m = fmaxf(m, v[i]);
        put(m);
    } else if (p.cGroup >= 32) {                                // two, or the tile's last columns
        float m0 = -INFINITY, m1 = -INFINITY;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            m0 = fmaxf(m0, i < end && i < cn ? v[i] : -INFINITY);
            m1 = fmaxf(m1, i >= end && i < cn ? v[i] : -INFINITY);
        }
        put(m0);
        if (end < cn) {
            l++;
            put(m1);
        }
    } else {
        float m = -INFINITY;
#pragma unroll
        for (int i = 0; i < 32; i++) {
            if (i >= cn) break;
            m = fmaxf(m, v[i]);
            if (i + 1 == end || i + 1 == cn) {
                put(m);
                m = -INFINITY;
                l++;
                end += p.cGroup;
            }
        }
    }
}

// Half `half` of the accumulator's 32 lanes of this warp to C: lane = row;
// columns go through the warp's buffer 32 at a time (TC_ROWS rows a time), so
// that a store covers neighbouring columns.
__device__ __forceinline__ void store_tile(const TcParams& p, uint32_t acc, float* stage,
                                           const float* ad, int lane, int rowBase, int item,
                                           int nValid, int half)
{
    const int rows = min(32, p.M - rowBase);
    const float add = (lane < rows && p.nrm) ? p.nrm[item * p.sN + rowBase + lane] : 0.f;
    float* cbase = p.C + item * p.sC + (size_t)rowBase * p.ldc;
    const int j0 = item * p.colPerItem;
    for (int c0 = 32 * half; c0 < nValid; c0 += 64) {
        float v[32];
        tmem_ld32(acc + (uint32_t)c0, v);
        if (rows <= 0) continue;
#pragma unroll
        for (int i = 0; i < 32; i++) v[i] = fmaf(p.alpha, v[i], add);
        const int cn = min(32, nValid - c0);
        if (p.best) chunk_best(p, v, cn, ad, lane, rowBase, rows, j0, c0);
        size_t off = c0 + lane;
        if (p.cGroup > 0) {
            const int jj = j0 + c0 + lane, l = jj / p.cGroup;
            off = (size_t)l * p.cGroupStride + (jj - l * p.cGroup);
        }
        float* dst = cbase + off;
#pragma unroll
        for (int h = 0; h < 32; h += TC_ROWS) {
            if (lane / TC_ROWS == h / TC_ROWS)
#pragma unroll
                for (int i = 0; i < 8; i++)
                    *reinterpret_cast<float4*>(stage + (lane - h) * TC_PITCH + 4 * i) =
                        make_float4(v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
            __syncwarp();
            if (lane < cn) {
                if (rows >= h + TC_ROWS) {
                    float t[TC_ROWS];
#pragma unroll
                    for (int rr = 0; rr < TC_ROWS; rr++) t[rr] = stage[rr * TC_PITCH + lane];
#pragma unroll
                    for (int rr = 0; rr < TC_ROWS; rr++) dst[(long long)(h + rr) * p.ldc] = t[rr];
                } else {
                    for (int rr = 0; rr < rows - h; rr++)
                        dst[(long long)(h + rr) * p.ldc] = stage[rr * TC_PITCH + lane];
                }
            }
            __syncwarp();
        }
    }
}

template <int BK>
__global__ void __launch_bounds__(TC_THREADS, 1)
k_gemm_bf16x3(const __grid_constant__ CUtensorMap tmAh, const __grid_constant__ CUtensorMap tmAl,
              const __grid_constant__ CUtensorMap tmBh, const __grid_constant__ CUtensorMap tmBl,
              const TcParams p)
{
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // 1024-byte aligned stage buffers
    uint8_t* smem = reinterpret_cast<uint8_t*>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    const int aBytes = TC_M * BK * 2;                  // 16 KB (BK 64) or 8 KB (32)
    const int bBytes = p.ntile * BK * 2;               // ntile rows of 2 BK bytes
    const int stageBytes = 2 * aBytes + 2 * bBytes;
    float* outStage = reinterpret_cast<float*>(smem + p.stages * stageBytes);
    float* norms = outStage + TC_EPI * TC_STAGE;                 // with best: [TC_EPI][32 TC_SEGS]
    uint64_t* full =
        reinterpret_cast<uint64_t*>(norms + (p.best ? TC_EPI * 32 * TC_SEGS : 0));
    uint64_t* empty = full + p.stages;
    uint64_t* accFull = empty + p.stages;              // [2]
    uint64_t* accEmpty = accFull + 2;                  // [2]
    uint64_t* drained = accEmpty + 2;                  // abort only: the issued MMAs are done
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(drained + 1);
    int* abortFlag = reinterpret_cast<int*>(tmemSlot + 1);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int nkb = p.Kd / BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; s++) {
            mbar_init(full + s, 1);
            mbar_init(empty + s, 1);
        }
        for (int a = 0; a < 2; a++) {
            mbar_init(accFull + a, 1);
            mbar_init(accEmpty + a, TC_EPI);
        }
        mbar_init(drained, 1);
        *abortFlag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmemSlot)),
                     "r"(2 * p.tmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmemSlot;
    // a wait that ran out anywhere in the CTA ends every role's loop
    auto wait = [&](uint64_t* bar, int parity) {
        if (mbar_wait(bar, parity, kWaitBudget) && *(volatile int*)abortFlag == 0) return true;
        if (atomicExch(abortFlag, 1) == 0) atomicOr(p.flag, 4);
        return false;
    };

    int issuedTma = 0;      // K blocks whose copies were issued (producer)
    int issuedMma = 0;      // K blocks whose MMAs were issued (issuer)
    if (warp == 0 && lane == 0) {
        // ---------------- TMA producer
        bool ok = true;
        for (int t = blockIdx.x; ok && t < p.tiles; t += gridDim.x) {
            const int item = t / p.mTiles;
            const int aRow0 = item * p.aRowsPerItem + (t - item * p.mTiles) * TC_M;
            const int bRow0 = item * p.bRowsPerItem;
            for (int kb = 0; kb < nkb; kb++) {
                const int s = issuedTma % p.stages, round = issuedTma / p.stages;
                if (round > 0 && !wait(empty + s, (round - 1) & 1)) {
                    ok = false;
                    break;
                }
                uint8_t* st = smem + s * stageBytes;
                mbar_expect_tx(full + s, stageBytes);
                tma_load_2d(st, &tmAh, full + s, kb * BK, aRow0);
                tma_load_2d(st + aBytes, &tmAl, full + s, kb * BK, aRow0);
                tma_load_2d(st + 2 * aBytes, &tmBh, full + s, kb * BK, bRow0);
                tma_load_2d(st + 2 * aBytes + bBytes, &tmBl, full + s, kb * BK, bRow0);
                issuedTma++;
            }
        }
    } else if (warp == 1 && lane == 0) {
        // ---------------- MMA issuer
        const uint32_t idesc = umma_idesc(TC_M, p.ntile);
        bool ok = true;
        int i = 0;
        for (int t = blockIdx.x; ok && t < p.tiles; t += gridDim.x, i++) {
            const uint32_t acc = tmem + (i & 1) * p.tmemCols;
            if (i >= 2 && !wait(accEmpty + (i & 1), ((i >> 1) - 1) & 1)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int kb = 0; kb < nkb; kb++) {
                const int s = issuedMma % p.stages;
                if (!wait(full + s, (issuedMma / p.stages) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                uint8_t* st = smem + s * stageBytes;
                const uint32_t ah = smem_u32(st), al = smem_u32(st + aBytes);
                const uint32_t bh = smem_u32(st + 2 * aBytes),
                               bl = smem_u32(st + 2 * aBytes + bBytes);
#pragma unroll
                for (int kk = 0; kk < BK / 16; kk++) {
                    const uint32_t off = kk * 32;      // 16 bf16 = 32 bytes along K
                    umma_bf16(acc, desc<BK>(ah + off), desc<BK>(bh + off), idesc, (kb | kk) != 0);
                    umma_bf16(acc, desc<BK>(ah + off), desc<BK>(bl + off), idesc, 1);
                    umma_bf16(acc, desc<BK>(al + off), desc<BK>(bh + off), idesc, 1);
                }
                umma_commit(empty + s);    // stage free once these MMAs have read it
                issuedMma++;
            }
            if (ok) umma_commit(accFull + (i & 1));
        }
    } else if (warp >= 2) {
        // ---------------- epilogue: tensor-memory lanes 32 (warp mod 4) ..
        const int q = warp & 3;
        int i = 0;
        for (int t = blockIdx.x; t < p.tiles; t += gridDim.x, i++) {
            const int item = t / p.mTiles;
            const int rowBase = (t - item * p.mTiles) * TC_M + q * 32;
            const int nValid = p.nTotal > 0 ? min(p.N, p.nTotal - item * p.N) : p.N;
            float* ad = norms + (warp - 2) * 32 * TC_SEGS;
            if (p.best) load_norms(p, ad, lane, rowBase, item, nValid);
            // one lane waits for the warp: the loads below are warp-collective
            int ok = lane == 0 ? wait(accFull + (i & 1), (i >> 1) & 1) : 0;
            if (!__shfl_sync(0xffffffffu, ok, 0)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            store_tile(p, tmem + (i & 1) * p.tmemCols + ((uint32_t)(q * 32) << 16),
                       outStage + (warp - 2) * TC_STAGE, ad, lane, rowBase, item, nValid,
                       (warp - 2) >> 2);
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(accEmpty + (i & 1));
        }
    }
    __syncwarp();
    __syncthreads();
    if (*(volatile int*)abortFlag) {
        // let the copies and the MMAs that this CTA issued finish before leaving
        if (warp == 0 && lane == 0)
            for (int kb = max(0, issuedTma - p.stages); kb < issuedTma; kb++)
                mbar_wait(full + kb % p.stages, (kb / p.stages) & 1, kWaitBudget / 4);
        if (warp == 1 && lane == 0 && issuedMma > 0) {
            umma_commit(drained);
            mbar_wait(drained, 0, kWaitBudget / 4);
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                     "r"(2 * p.tmemCols)
                     : "memory");
    }
}

}  // namespace

bool bf16x3_available() { return tc::encode_fn() != nullptr; }

size_t bf16x3_scratch_bytes(int, int, int, int) { return 256; }

// A and B point at the hi planes; the lo plane of each follows its hi plane
// (rows * Kd bf16 elements later).  lda / ldb must equal Kd.
// General form.  A: hi plane at A, lo plane rowsA x Kd elements later; B the
// same with rowsB.  Item i uses A rows i * aRowsPerItem + (0 .. M) and B rows
// i * bRowsPerItem + (0 .. N); it writes C + i * sC (+ row * ldc + col) for
// row < M and col < N (col < nTotal - i * N when nTotal > 0).
cudaError_t launch_gemm_bf16x3(const void* A, long long rowsA, const void* B, long long rowsB,
                               int M, int N, int Kd, int items, int aRowsPerItem,
                               int bRowsPerItem, int nTotal, float* C, long long sC, int ldc,
                               const float* nrm, long long sN, float alpha, int* flag,
                               cudaStream_t st, int cGroup, long long cGroupStride, int bk,
                               const TileBest* best, bool besideProjections)
{
    if (bk != 64 && bk != 32) return cudaErrorInvalidValue;
    if (N <= 0 || N > 256 || M <= 0 || items <= 0 || Kd <= 0 || Kd % bk)
        return cudaErrorInvalidValue;
    const __nv_bfloat16* Ah = reinterpret_cast<const __nv_bfloat16*>(A);
    const __nv_bfloat16* Al = Ah + rowsA * Kd;
    const __nv_bfloat16* Bh = reinterpret_cast<const __nv_bfloat16*>(B);
    const __nv_bfloat16* Bl = Bh + rowsB * Kd;
    TcParams p;
    p.M = M;
    p.N = N;
    p.Kd = Kd;
    p.aRowsPerItem = aRowsPerItem;
    p.bRowsPerItem = bRowsPerItem;
    p.nTotal = nTotal;
    p.colPerItem = N;
    p.cGroup = cGroup;
    p.cGroupStride = cGroupStride;
    p.ntile = (N + 15) / 16 * 16;
    p.tmemCols = 32;
    while (p.tmemCols < p.ntile) p.tmemCols <<= 1;
    p.best = best ? best->key : nullptr;
    if (best) {
        if (cGroup <= 0 || best->rows <= 0) return cudaErrorInvalidValue;
        p.bestRows = best->rows;
        p.bestGroups = best->groups;
        p.bestNrm = best->nrm;
        p.bestNs = best->nrmStride;
    }
    const int stageBytes = 2 * TC_M * bk * 2 + 2 * p.ntile * bk * 2;
    // all of the shared memory; beside projections 131 KB (the 132 KB split of
    // an SM's 228 KB with the CTA's own KB), at least two stages
    const size_t extra = 1024 + 256 +
                         sizeof(float) * TC_EPI * (TC_STAGE + (best ? 32 * TC_SEGS : 0));
    p.stages = (int)(((besideProjections ? 131 : 227) * 1024 - extra) / stageBytes);
    if (p.stages < 2) p.stages = (int)((227 * 1024 - extra) / stageBytes);
    const int maxStages = bk == 64 ? 4 : 6;
    if (p.stages > maxStages) p.stages = maxStages;
    if (p.stages < 2) return cudaErrorInvalidValue;
    p.C = C;
    p.sC = sC;
    p.ldc = ldc;
    p.nrm = nrm;
    p.sN = sN;
    p.alpha = alpha;
    p.flag = flag;
    const bool sw64 = bk == 32;
    CUtensorMap mAh, mAl, mBh, mBl;
    if (!tc::make_map(&mAh, Ah, rowsA, Kd, TC_M, bk, sw64) ||
        !tc::make_map(&mAl, Al, rowsA, Kd, TC_M, bk, sw64) ||
        !tc::make_map(&mBh, Bh, rowsB, Kd, p.ntile, bk, sw64) ||
        !tc::make_map(&mBl, Bl, rowsB, Kd, p.ntile, bk, sw64))
        return cudaErrorInvalidValue;
    const int mTiles = (M + TC_M - 1) / TC_M;
    if ((long long)mTiles * items > 0x7fffffffLL) return cudaErrorInvalidValue;
    p.mTiles = mTiles;
    p.tiles = mTiles * items;
    const size_t smem = (size_t)p.stages * stageBytes + extra;
    void (*kern)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap,
                 const TcParams) = bk == 64 ? k_gemm_bf16x3<64> : k_gemm_bf16x3<32>;
    cudaError_t e = allow_shared(kern);
    if (e != cudaSuccess) return e;
    kern<<<std::min(p.tiles, 152), TC_THREADS, smem, st>>>(mAh, mAl, mBh, mBl, p);
    return cudaGetLastError();
}

// Batched form: item b multiplies A rows [b M, (b + 1) M) with B rows
// [b N, (b + 1) N).  lda / ldb must equal Kd and the batch strides M Kd / N Kd.
cudaError_t launch_gemm_nt_bf16x3(const float* A, long long sA, int lda, const float* B,
                                  long long sB, int ldb, int M, int N, int Kd, int batch,
                                  float* C, long long sC, int ldc, const float* nrm,
                                  long long sN, float alpha, void*, size_t, int* flag,
                                  cudaStream_t st, int bk, bool besideProjections)
{
    if (lda != Kd || ldb != Kd || sA != (long long)M * Kd || sB != (long long)N * Kd)
        return cudaErrorInvalidValue;
    return launch_gemm_bf16x3(A, (long long)batch * M, B, (long long)batch * N, M, N, Kd, batch, M,
                              N, 0, C, sC, ldc, nrm, sN, alpha, flag, st, 0, 0,
                              Kd % bk == 0 ? bk : 64, nullptr, besideProjections);
}

}  // namespace tg3
