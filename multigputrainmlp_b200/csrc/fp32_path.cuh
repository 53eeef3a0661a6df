// The reference's non-fp16 data flows (--linear-fp16 0 and/or --input-grad-fp16 0), on CUDA cores.
//
// These flags select fp32 activations and weights for the linear layers, and an fp32 (instead of fp16)
// gradient operand for the embedding table (native/cuda/mlp_backward.cu:1273-1510 with use_half_linear /
// use_half_input_grad false; the reference runs them as TF32 cuBLAS GEMMs). Plain fp32 multiply-adds with fixed
// summation orders: results are deterministic and at least as accurate as the reference's TF32. Used by engine.cu only.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "embedding_gather.cuh"
#include "launch.cuh"

namespace mgt {
namespace fp32path {

// ---- dense layers --------------------------------------------------------------------------------------------------
// C[M x N] = op(A)[M x K] * op(B)[K x N]
//   TA = false: A is [M][lda] (K contiguous)     TA = true: A is [K][lda] (M contiguous)
//   TB = false: B is [K][ldb] (N contiguous)     TB = true: B is [N][ldb] (K contiguous)
// blockIdx.z = group * splits + split: groups are equal problems `stride_*` floats apart, splits share K. With splits > 1
// the result is a plane of partial sums, added up in order with the sums of the step; otherwise the epilogue applies,
// each step optional:   v = relu((acc + bias[n] + add[m][n])) * [mask[m][n] > 0]   and column sums of v per tile row.
struct SgemmArgs {
    const float* A;
    const float* B;
    float* C;
    uint64_t stride_a, stride_b, stride_c;
    uint32_t M, N, K, lda, ldb, ldc, splits;
    const float* bias;
    const float* add;
    const float* mask;
    uint32_t ld_add, ld_mask, relu;
    float* colsum;  // [gridDim.y][N]
    bool vec_a, vec_b;
};

__device__ __forceinline__ uint64_t PackPair(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void UnpackPair(uint64_t v, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v)); }
// two independent, correctly rounded fp32 multiply-adds in one instruction
__device__ __forceinline__ void FmaPair(uint64_t& acc, uint64_t a, uint64_t b) { asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b)); }

// One float4 of a tile operand. kKContig: the operand is [rows][ld] with K inside, element (row, k..k+3); otherwise
// [K][ld] with the rows inside, element (k, row..row+3). Outside the matrix: zeros.
template <bool kKContig>
__device__ __forceinline__ float4 LoadQuad(const float* __restrict__ p, uint32_t ld, uint32_t rows, uint32_t K, uint32_t row, uint32_t k, bool vec) {
    float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (kKContig) {
        if (row >= rows || k >= K) return v;
        const float* q = p + static_cast<uint64_t>(row) * ld + k;
        if (vec && k + 4U <= K) return __ldg(reinterpret_cast<const float4*>(q));
        v.x = __ldg(q);
        if (k + 1U < K) v.y = __ldg(q + 1);
        if (k + 2U < K) v.z = __ldg(q + 2);
        if (k + 3U < K) v.w = __ldg(q + 3);
    } else {
        if (row >= rows || k >= K) return v;
        const float* q = p + static_cast<uint64_t>(k) * ld + row;
        if (vec && row + 4U <= rows) return __ldg(reinterpret_cast<const float4*>(q));
        v.x = __ldg(q);
        if (row + 1U < rows) v.y = __ldg(q + 1);
        if (row + 2U < rows) v.z = __ldg(q + 2);
        if (row + 3U < rows) v.w = __ldg(q + 3);
    }
    return v;
}

// A CTA computes a BM x BN tile, a thread TM x TN of it; KG groups of threads share the tile's K chunks and are added in
// shared memory at the end (small problems: the K loop of one tile is the critical path). Operands are staged through
// registers into double-buffered shared memory, BK deep, one barrier per chunk. Bound by the fp32 pipes: with pairs of
// rows in one fma.rn.f32x2 the inner loop needs TM * TN / 2 of them, TN duplications and (TM + TN) / 4 vector reads.
// (The first version of this path read scalars through a 4 x 4 tile without prefetch and never split K: the 34 weight
// gradients of p888 at 8 192 samples took 45.2 ms, now 1.1 ms.)
template <int BM, int BN, int TM, int TN, int KG, int BK, bool TA, bool TB>
__global__ void __launch_bounds__((BM / TM) * (BN / TN) * KG)
SgemmKernel(const __grid_constant__ SgemmArgs a) {
    constexpr uint32_t NT = (BM / TM) * (BN / TN);
    constexpr uint32_t QA = BM * BK / 4 / NT, QB = BN * BK / 4 / NT;  // float4 loads per thread and chunk
    constexpr uint32_t LDA = BM + 4, LDB = BN + 4;
    constexpr int VW = TN < 4 ? TN : 4, NV = TN / VW;  // a thread's columns: NV vectors of VW
    static_assert(QA >= 1 && QB >= 1 && QA * NT * 4 == BM * BK && QB * NT * 4 == BN * BK && BK % 16 == 0, "whole quads per thread");
    __shared__ __align__(16) float As[KG][2][BK][LDA];
    __shared__ __align__(16) float Bs[KG][2][BK][LDB];
    const uint32_t group_k = threadIdx.x / NT, tid = threadIdx.x % NT;
    const uint32_t tx = tid % (BN / TN), ty = tid / (BN / TN);
    const uint32_t m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const uint32_t group = blockIdx.z / a.splits, split = blockIdx.z - group * a.splits;
    const float* A = a.A + group * a.stride_a;
    const float* B = a.B + group * a.stride_b;
    const uint32_t chunks = (a.K + BK - 1U) / BK;
    const uint32_t c_begin = static_cast<uint32_t>(static_cast<uint64_t>(split) * chunks / a.splits);
    const uint32_t c_end = static_cast<uint32_t>(static_cast<uint64_t>(split + 1U) * chunks / a.splits);
    const uint32_t turns = (c_end - c_begin + KG - 1U) / KG;

    // quad q of an operand with K inside: 16 columns of K at a time, four lanes to a row of them
    auto k_of = [](uint32_t q, uint32_t rows) { return q / (rows * 4U) * 16U + (q % 4U) * 4U; };
    auto row_of = [](uint32_t q, uint32_t rows) { return q % (rows * 4U) / 4U; };
    float4 qa[QA], qb[QB];
    auto fetch = [&](uint32_t turn) {
        const uint32_t c = c_begin + turn * KG + group_k;
        const uint32_t K = c < c_end ? a.K : 0U;  // past the range: zeros
#pragma unroll
        for (uint32_t i = 0; i < QA; ++i) {
            const uint32_t q = tid + i * NT;
            if (TA) qa[i] = LoadQuad<false>(A, a.lda, a.M, K, m0 + (q % (BM / 4)) * 4U, c * BK + q / (BM / 4), a.vec_a);
            else qa[i] = LoadQuad<true>(A, a.lda, a.M, K, m0 + row_of(q, BM), c * BK + k_of(q, BM), a.vec_a);
        }
#pragma unroll
        for (uint32_t i = 0; i < QB; ++i) {
            const uint32_t q = tid + i * NT;
            if (TB) qb[i] = LoadQuad<true>(B, a.ldb, a.N, K, n0 + row_of(q, BN), c * BK + k_of(q, BN), a.vec_b);
            else qb[i] = LoadQuad<false>(B, a.ldb, a.N, K, n0 + (q % (BN / 4)) * 4U, c * BK + q / (BN / 4), a.vec_b);
        }
    };
    // An operand with K inside is transposed on its way into shared memory: the four scalars of a quad go to four K rows. Rows
    // 8..15 of every 16 hold the columns with bit 3 flipped, so that the quads of eight rows meet in 32 different banks.
    auto stage = [&](uint32_t buf) {
#pragma unroll
        for (uint32_t i = 0; i < QA; ++i) {
            const uint32_t q = tid + i * NT;
            if (TA) {
                *reinterpret_cast<float4*>(&As[group_k][buf][q / (BM / 4)][(q % (BM / 4)) * 4U]) = qa[i];
            } else {
                const uint32_t k = k_of(q, BM), r = row_of(q, BM) ^ (k & 8U);
                As[group_k][buf][k][r] = qa[i].x; As[group_k][buf][k + 1][r] = qa[i].y; As[group_k][buf][k + 2][r] = qa[i].z; As[group_k][buf][k + 3][r] = qa[i].w;
            }
        }
#pragma unroll
        for (uint32_t i = 0; i < QB; ++i) {
            const uint32_t q = tid + i * NT;
            if (!TB) {
                *reinterpret_cast<float4*>(&Bs[group_k][buf][q / (BN / 4)][(q % (BN / 4)) * 4U]) = qb[i];
            } else {
                const uint32_t k = k_of(q, BN), r = row_of(q, BN) ^ (k & 8U);
                Bs[group_k][buf][k][r] = qb[i].x; Bs[group_k][buf][k + 1][r] = qb[i].y; Bs[group_k][buf][k + 2][r] = qb[i].z; Bs[group_k][buf][k + 3][r] = qb[i].w;
            }
        }
    };

    uint64_t acc[TM / 2][TN];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ULL;
    dependent_begin();
    fetch(0);
    stage(0);
    __syncthreads();
    for (uint32_t turn = 0; turn < turns; ++turn) {
        const uint32_t buf = turn & 1U;
        if (turn + 1U < turns) fetch(turn + 1U);
#pragma unroll 16
        for (uint32_t k = 0; k < BK; ++k) {
            uint64_t av[TM / 2];
            float bv[TN];
#pragma unroll
            for (int i = 0; i < TM / 4; ++i) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&As[group_k][buf][k][(ty * TM + i * 4) ^ (TA ? 0U : k & 8U)]);
                av[2 * i] = v.x;
                av[2 * i + 1] = v.y;
            }
#pragma unroll
            for (int j = 0; j < NV; ++j) {
                // (a thread's vectors lie BN / NV columns apart: the warp reads consecutive ones)
                const float* b = &Bs[group_k][buf][k][(j * (BN / NV) + tx * VW) ^ (TB ? k & 8U : 0U)];
                if constexpr (VW == 4) {
                    const float4 v = *reinterpret_cast<const float4*>(b);
                    bv[4 * j] = v.x; bv[4 * j + 1] = v.y; bv[4 * j + 2] = v.z; bv[4 * j + 3] = v.w;
                } else {
                    const float2 v = *reinterpret_cast<const float2*>(b);
                    bv[2 * j] = v.x; bv[2 * j + 1] = v.y;
                }
            }
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const uint64_t bb = PackPair(bv[j], bv[j]);
#pragma unroll
                for (int i = 0; i < TM / 2; ++i) FmaPair(acc[i][j], av[i], bb);
            }
        }
        if (turn + 1U < turns) stage(buf ^ 1U);
        __syncthreads();
    }
    float v[TM][TN];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) UnpackPair(acc[i][j], v[2 * i][j], v[2 * i + 1][j]);
    if (KG > 1) {
        float* spill = &As[0][0][0][0];  // (KG - 1) tiles: the operand buffers are free now
        static_assert(KG == 1 || (KG - 1) * BM * BN <= KG * 2 * static_cast<int>(BK * LDA), "partial tiles fit the operand buffer");
        if (group_k > 0U) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) spill[((group_k - 1U) * TM * TN + i * TN + j) * NT + tid] = v[i][j];
        }
        __syncthreads();
        if (group_k > 0U) return;
#pragma unroll
        for (uint32_t g = 1; g < KG; ++g)
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) v[i][j] += spill[((g - 1U) * TM * TN + i * TN + j) * NT + tid];
    }
    const bool partial = a.splits > 1U;
    float* C = a.C + (partial ? static_cast<uint64_t>(blockIdx.z) * a.M * a.N : group * a.stride_c);
    const uint32_t ldc = partial ? a.N : a.ldc;
    const bool vec_c = (ldc & 3U) == 0U && (reinterpret_cast<uintptr_t>(C) & 15U) == 0U;
    float cs[TN] = {};
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const uint32_t m = m0 + ty * TM + i;
        if (m >= a.M) break;
#pragma unroll
        for (int jq = 0; jq < NV; ++jq) {
            const uint32_t n = n0 + jq * (BN / NV) + tx * VW;
#pragma unroll
            for (int e = 0; e < VW; ++e) {
                if (n + e >= a.N) continue;
                float x = v[i][jq * VW + e];
                if (!partial) {
                    if (a.bias != nullptr) x += __ldg(a.bias + n + e);
                    if (a.add != nullptr) x += a.add[static_cast<uint64_t>(m) * a.ld_add + n + e];
                    if (a.relu != 0U) x = fmaxf(x, 0.0f);
                    if (a.mask != nullptr) x = __ldg(a.mask + static_cast<uint64_t>(m) * a.ld_mask + n + e) > 0.0f ? x : 0.0f;
                    cs[jq * VW + e] += x;
                }
                v[i][jq * VW + e] = x;
            }
            float* dst = C + static_cast<uint64_t>(m) * ldc + n;
            if (vec_c && n + VW <= a.N) {
                if constexpr (VW == 4) *reinterpret_cast<float4*>(dst) = make_float4(v[i][jq * 4], v[i][jq * 4 + 1], v[i][jq * 4 + 2], v[i][jq * 4 + 3]);
                else *reinterpret_cast<float2*>(dst) = make_float2(v[i][jq * 2], v[i][jq * 2 + 1]);
            } else {
#pragma unroll
                for (int e = 0; e < VW; ++e)
                    if (n + e < a.N) dst[e] = v[i][jq * VW + e];
            }
        }
    }
    if (a.colsum != nullptr && !partial) {
        // rows of the tile in a fixed order: a thread's own, then the row groups of the CTA
        float* red = &Bs[0][0][0][0];
        constexpr uint32_t kRowGroups = BM / TM;
        static_assert(kRowGroups * BN <= KG * 2 * BK * LDB, "column sums fit the operand buffer");
        if (KG > 1) asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); else __syncthreads();  // (with KG > 1 only the first group is still here)
#pragma unroll
        for (int jq = 0; jq < NV; ++jq)
#pragma unroll
            for (int e = 0; e < VW; ++e) red[ty * BN + jq * (BN / NV) + tx * VW + e] = cs[jq * VW + e];
        if (KG > 1) asm volatile("bar.sync 1, %0;" ::"n"(NT) : "memory"); else __syncthreads();
        for (uint32_t c = tid; c < BN; c += NT) {
            if (n0 + c >= a.N) break;
            float sum = 0.0f;
            for (uint32_t g = 0; g < kRowGroups; ++g) sum += red[g * BN + c];
            a.colsum[static_cast<uint64_t>(blockIdx.y) * a.N + n0 + c] = sum;
        }
    }
}

// Tile choice. The large tile has the best ratio of multiply-adds to shared-memory reads but needs two waves of the 148 SMs
// to balance; the middle one (four CTAs per SM) covers the rest of the range; below one CTA per SM the K loop of a single
// tile is what takes the time, so small tiles. Gradients split K over four groups of threads there. The forward product (neither
// operand transposed) adds in the order of k whatever its tile: its results decide the ReLUs, and every other order opens or
// closes one here and there, which moves the gradient by up to 1e-4, where a gradient product's own order moves it by 1e-7. So one
// K group, chunks of 64 to keep loads in flight and 4 x 2 results a thread for a shorter turn (a step of 1 024 samples, hd1 256,
// hd2 64, 2 blocks: 186 us with four groups, 195 us with 4 x 4 results, 190 us like this).
enum class SgemmTile { kLarge, kMiddle, kSmall };
inline uint32_t SgemmTileRows(SgemmTile t) { return t == SgemmTile::kLarge ? 128U : (t == SgemmTile::kMiddle ? 64U : 32U); }
inline SgemmTile PickSgemmTile(uint32_t M, uint32_t N, uint64_t batches, uint32_t sm_count) {
    auto tiles = [&](uint32_t t) { return static_cast<uint64_t>((M + t - 1) / t) * ((N + t - 1) / t) * batches; };
    if (tiles(128U) >= 2ULL * sm_count && N > 64U) return SgemmTile::kLarge;
    return tiles(64U) >= sm_count ? SgemmTile::kMiddle : SgemmTile::kSmall;
}

inline bool SgemmAligned(const float* p, uint32_t ld, uint64_t stride) {
    return (reinterpret_cast<uintptr_t>(p) & 15U) == 0U && (ld & 3U) == 0U && (stride & 3ULL) == 0ULL;
}
template <bool TA, bool TB>
inline cudaError_t Sgemm(LaunchOn st, SgemmArgs a, uint32_t groups, SgemmTile tile) {
    a.vec_a = SgemmAligned(a.A, a.lda, a.stride_a);
    a.vec_b = SgemmAligned(a.B, a.ldb, a.stride_b);
    const uint32_t t = SgemmTileRows(tile);
    const dim3 grid((a.N + t - 1) / t, (a.M + t - 1) / t, groups * a.splits);
    if (tile == SgemmTile::kLarge) Launch(SgemmKernel<128, 128, 8, 8, 1, 16, TA, TB>, grid, 256, 0, st, a);
    else if (tile == SgemmTile::kMiddle) Launch(SgemmKernel<64, 64, 8, 4, 1, 16, TA, TB>, grid, 128, 0, st, a);
    else if constexpr (!TA && !TB) Launch(SgemmKernel<32, 32, 4, 2, 1, 64, TA, TB>, grid, 128, 0, st, a);
    else Launch(SgemmKernel<32, 32, 4, 4, 4, 16, TA, TB>, grid, 256, 0, st, a);
    return cudaGetLastError();
}

// ---- embedding layer -------------------------------------------------------------------------------------------------
// a1[s][h] = relu(b_in[h] + sum over positions, in position order, of W_in[pos*V + state[s][pos]][h])  (mlp_backward.cu:696-753)
// A warp owns SPW samples and 32 * W columns, a CTA 8 * SPW samples of the same columns, and all walk the positions in step:
// the V rows of a position that the CTA's samples pick from stay in L1 while they are used (72 rows of 512 bytes), so L2
// serves each row about once per CTA and position instead of once per sample. SPW = 8 at large batches (0.92 -> 0.31 ms
// at 8 192 samples x 2 560 columns), SPW = 1 where there would be too few warps otherwise. W = 4: H1 a multiple of four.
template <int SPW, int W>
__global__ void __launch_bounds__(256)
EmbeddingForwardKernel(const uint8_t* __restrict__ states, const float* __restrict__ w_in, const float* __restrict__ b_in, uint32_t B, uint32_t L, uint32_t V,
                       uint32_t H1, float* __restrict__ a1, uint32_t ld) {
    constexpr uint32_t kSamples = 8U * SPW;
    __shared__ uint8_t cls[80][kSamples];  // [position][sample]
    const uint32_t s0 = blockIdx.x * kSamples, warp = threadIdx.x >> 5, lane = threadIdx.x & 31U;
    dependent_begin();
    for (uint32_t i = threadIdx.x; i < kSamples * L; i += 256U) {
        const uint32_t s = i / L, p = i - s * L;
        cls[p][s] = s0 + s < B ? states[static_cast<uint64_t>(s0 + s) * 80U + p] : 0U;
    }
    __syncthreads();
    const uint32_t h = (blockIdx.y * 32U + lane) * W;
    if (h >= H1) return;
    float acc[SPW][W];
#pragma unroll
    for (int q = 0; q < SPW; ++q)
#pragma unroll
        for (int e = 0; e < W; ++e) acc[q][e] = __ldg(b_in + h + e);
    const uint32_t rows = L * V;
#pragma unroll(SPW == 1 ? 8 : 2)
    for (uint32_t p = 0; p < L; ++p) {
#pragma unroll
        for (int q = 0; q < SPW; ++q) {
            const uint32_t row = min(p * V + cls[p][warp * SPW + q], rows - 1U);
            const float* src = w_in + static_cast<uint64_t>(row) * H1 + h;
            if (W == 4) {
                const float4 x = __ldg(reinterpret_cast<const float4*>(src));
                acc[q][0] += x.x; acc[q][1 % W] += x.y; acc[q][2 % W] += x.z; acc[q][3 % W] += x.w;
            } else {
                acc[q][0] += __ldg(src);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < SPW; ++q) {
        const uint32_t s = s0 + warp * SPW + q;
        if (s >= B) break;
        float* dst = a1 + static_cast<uint64_t>(s) * ld + h;
        if (W == 4) *reinterpret_cast<float4*>(dst) = make_float4(fmaxf(acc[q][0], 0.0f), fmaxf(acc[q][1 % W], 0.0f), fmaxf(acc[q][2 % W], 0.0f), fmaxf(acc[q][3 % W], 0.0f));
        else dst[0] = fmaxf(acc[q][0], 0.0f);
    }
}
inline cudaError_t EmbeddingForward(LaunchOn st, const uint8_t* states, const float* w_in, const float* b_in, uint32_t B, uint32_t L, uint32_t V, uint32_t H1,
                                    float* a1, uint32_t ld, uint32_t sm_count) {
    const bool quads = (H1 & 3U) == 0U && (ld & 3U) == 0U && (reinterpret_cast<uintptr_t>(w_in) & 15U) == 0U;
    const uint32_t col_blocks = (H1 + (quads ? 128U : 32U) - 1U) / (quads ? 128U : 32U);
    // eight samples per warp once that still leaves four CTAs for every SM
    const bool many = static_cast<uint64_t>((B + 63U) / 64U) * col_blocks >= 4ULL * sm_count;
    const dim3 grid(many ? (B + 63U) / 64U : (B + 7U) / 8U, col_blocks);
    if (quads && many) Launch(EmbeddingForwardKernel<8, 4>, grid, 256, 0, st, states, w_in, b_in, B, L, V, H1, a1, ld);
    else if (quads) Launch(EmbeddingForwardKernel<1, 4>, grid, 256, 0, st, states, w_in, b_in, B, L, V, H1, a1, ld);
    else if (many) Launch(EmbeddingForwardKernel<8, 1>, grid, 256, 0, st, states, w_in, b_in, B, L, V, H1, a1, ld);
    else Launch(EmbeddingForwardKernel<1, 1>, grid, 256, 0, st, states, w_in, b_in, B, L, V, H1, a1, ld);
    return cudaGetLastError();
}

// Table gradient: grad[p*V + v][h] = sum of dz1[s][h] over the samples with class v at position p (zero where there are
// none), in sample order. A warp owns one table row and 32 * W columns and adds the listed rows of dz1, eight loads in flight;
// the column blocks are the slow grid dimension, so the slice of dz1 in use stays in L2. Bound by L2: every dz1 row is read
// once per position. (Adding every sample into shared-memory rows, one CTA per position and 64 columns, was a chain of
// dependent read-modify-writes: 8.24 ms at 16 384 samples x 2 560 columns, now 0.64 ms with the sort.)
template <int W>
__global__ void __launch_bounds__(256)
EmbeddingGradKernel(const uint32_t* __restrict__ order, const uint32_t* __restrict__ first, const float* __restrict__ dz1, uint32_t ld, uint32_t B, uint32_t L,
                    uint32_t V, uint32_t H1, float* __restrict__ grad_table) {
    const uint32_t row = blockIdx.x * 8U + (threadIdx.x >> 5), lane = threadIdx.x & 31U;
    if (row >= L * V) return;
    const uint32_t p = row / V, v = row - p * V;
    const uint32_t h = (blockIdx.y * 32U + lane) * W;
    dependent_begin();
    first = after_begin(first);
    const uint32_t lo = __ldg(first + p * (V + 1U) + v), hi = __ldg(first + p * (V + 1U) + v + 1U);
    const uint32_t* list = order + static_cast<uint64_t>(p) * B;
    float acc[W] = {};
    const bool in = h < H1;
    for (uint32_t i = lo; i < hi; i += 32U) {
        const uint32_t mine = i + lane < hi ? __ldg(list + i + lane) : 0U;
        const uint32_t n = min(32U, hi - i);
#pragma unroll 8
        for (uint32_t j = 0; j < n; ++j) {
            const uint32_t s = __shfl_sync(0xFFFFFFFFU, mine, j);
            if (in) {
                const float* src = dz1 + static_cast<uint64_t>(s) * ld + h;
                if (W == 4) {
                    const float4 x = __ldg(reinterpret_cast<const float4*>(src));
                    acc[0] += x.x; acc[1 % W] += x.y; acc[2 % W] += x.z; acc[3 % W] += x.w;
                } else {
                    acc[0] += __ldg(src);
                }
            }
        }
    }
    if (!in) return;
    float* dst = grad_table + static_cast<uint64_t>(row) * H1 + h;
    if (W == 4) *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1 % W], acc[2 % W], acc[3 % W]);
    else dst[0] = acc[0];
}
// `lists`: gather::ListWords words of scratch; `sorted`: gather::SortByClassKernel has left its lists there
inline cudaError_t EmbeddingGrad(LaunchOn st, const uint8_t* states, const float* dz1, uint32_t ld, uint32_t B, uint32_t L, uint32_t V, uint32_t H1,
                                 uint32_t* lists, bool sorted, float* grad_table) {
    uint32_t* first = lists + static_cast<uint64_t>(L) * B;
    if (!sorted) Launch(gather::SortByClassKernel, L, 1024, 0, st, states, B, V, lists, first);
    const bool quads = (H1 & 3U) == 0U && (ld & 3U) == 0U && (reinterpret_cast<uintptr_t>(grad_table) & 15U) == 0U;
    const uint32_t cols = quads ? 128U : 32U;
    const dim3 grid((L * V + 7U) / 8U, (H1 + cols - 1U) / cols);
    if (quads) Launch(EmbeddingGradKernel<4>, grid, 256, 0, st, lists, first, dz1, ld, B, L, V, H1, grad_table);
    else Launch(EmbeddingGradKernel<1>, grid, 256, 0, st, lists, first, dz1, ld, B, L, V, H1, grad_table);
    return cudaGetLastError();
}

// fp16 rounding of the embedding-gradient operand (--linear-fp16 0 --input-grad-fp16 1)
__global__ void RoundHalfKernel(float* __restrict__ x, uint64_t total) {
    dependent_begin();
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) x[i] = __half2float(__float2half_rn(x[i]));
}

}  // namespace fp32path
}  // namespace mgt
