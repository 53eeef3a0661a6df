// The embedding layer as what it is, sums of table rows: every sample of the batch picks one row per position, forward adds
// the picked rows, the table gradient adds the rows of dz1 that picked a table row. 16-bit operands, fp32 sums, the same
// results as the one-hot GEMMs of onehot_pair.cuh up to the order of the additions.
//
// Per sample both read L rows of H1 values and do nothing else; the GEMMs multiply by L * V - L zeros per sample to get the
// tensor cores to do it. Gathering runs at what L2 delivers (measured 20 TB/s: 256-byte and longer row segments, tables and
// slices that fit L2), scales with the batch from one sample on and does not care how many classes a position has, while a
// one-hot GEMM needs a wave of 256 x 512 tiles, two CTAs to each, with L * V / 64 K chunks. engine.cu picks the cheaper of the
// two by size.
#pragma once

#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.cuh"
#include "ptx_sm100.cuh"

namespace mgt {
namespace gather {

// A row vector, and below the adds, as volatile assembly: they stay in the order written, all loads of a batch before its
// first add (left to itself the compiler waits for each load in turn to save registers).
__device__ __forceinline__ uint4 LoadRow(const uint16_t* p) {
    uint4 u;
    asm volatile("ld.global.nc.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(u.x), "=r"(u.y), "=r"(u.z), "=r"(u.w) : "l"(p));
    return u;
}

// acc[0..7] += the eight 16-bit values of a 16-byte vector (mixed-precision adds: the fp32 sum of an fp32 and a 16-bit value)
template <bool kBf16>
__device__ __forceinline__ void AddEight(float (&acc)[8], const uint4& u) {
    const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint16_t lo = static_cast<uint16_t>(w[i] & 0xFFFFU), hi = static_cast<uint16_t>(w[i] >> 16);
        if (kBf16) {
            asm volatile("add.f32.bf16 %0, %1, %0;" : "+f"(acc[2 * i]) : "h"(lo));
            asm volatile("add.f32.bf16 %0, %1, %0;" : "+f"(acc[2 * i + 1]) : "h"(hi));
        } else {
            asm volatile("add.f32.f16 %0, %1, %0;" : "+f"(acc[2 * i]) : "h"(lo));
            asm volatile("add.f32.f16 %0, %1, %0;" : "+f"(acc[2 * i + 1]) : "h"(hi));
        }
    }
}

// a1T[h][s] = relu(bias[h] + sum over positions of table[p*V + state[s][p]][h]) in the operand format, and one sign word of
// the fp32 sums per h and 32 samples - what the one-hot forward writes. The bias is table row L*V.
// A CTA owns 32 samples x 64 columns; eight lanes share a sample and read 128 bytes of a row, and two such groups share the
// positions of a sample: half the chain of loads where the batch is small, no difference where L2 is the bound. The result is
// turned in shared memory so that rows of 32 samples are written whole. 1 024 samples x 256 columns 8 us, 3 001 x 2 560
// 70 us, 53 248 x 2 560 1.1 ms = 17 TB/s. (Four samples per group of lanes, for row hits in L1: 121 us and 1.6 ms.)
constexpr int kForwardSplit = 2;
template <int SPLIT, bool kBf16>
__global__ void __launch_bounds__(256 * SPLIT)
ForwardKernel(const uint8_t* __restrict__ states, const uint16_t* __restrict__ table, uint32_t ld_table, uint32_t B, uint32_t L, uint32_t V, uint32_t H1,
              uint16_t* __restrict__ a1_t, uint32_t ld, uint32_t* __restrict__ bits, uint32_t ld_bits) {
    constexpr uint32_t kThreads = 256U * SPLIT;
    constexpr uint32_t NB = 9U;  // loads in flight per thread
    __shared__ uint8_t cls[80][32];
    __shared__ float tile[SPLIT][64][33];
    const uint32_t s0 = blockIdx.x * 32U, h0 = blockIdx.y * 64U, t = threadIdx.x, group = (t >> 3) & 31U, part = t >> 8, sub = t & 7U;
    dependent_begin();
    for (uint32_t i = t; i < 32U * L; i += kThreads) {
        const uint32_t s = i / L, p = i - s * L;
        cls[p][s] = s0 + s < B ? states[static_cast<uint64_t>(s0 + s) * 80U + p] : 0U;
    }
    __syncthreads();
    const uint32_t rows = L * V, h = h0 + sub * 8U;
    float acc[8] = {};
    if (h < H1) {  // (rows are padded to eight columns)
        const uint16_t* col = table + h;
        if (part == 0U) AddEight<kBf16>(acc, __ldg(reinterpret_cast<const uint4*>(col + static_cast<uint64_t>(rows) * ld_table)));
        const uint32_t p_end = (part + 1U) * L / SPLIT;
        auto row = [&](uint32_t p) { return LoadRow(col + static_cast<uint64_t>(min(p * V + cls[p][group], rows - 1U)) * ld_table); };
        uint32_t p = part * L / SPLIT;
        for (; p + NB <= p_end; p += NB) {  // (whole batches without conditions, or the loads do not overlap)
            uint4 u[NB];
#pragma unroll
            for (uint32_t j = 0; j < NB; ++j) u[j] = row(p + j);
#pragma unroll
            for (uint32_t j = 0; j < NB; ++j) AddEight<kBf16>(acc, u[j]);
        }
        for (; p < p_end; ++p) AddEight<kBf16>(acc, row(p));
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) tile[part][sub * 8U + e][group] = acc[e];
    __syncthreads();
    const uint32_t warp = t >> 5, lane = t & 31U, s = s0 + lane;
#pragma unroll
    for (uint32_t i = 0; i < 8U / SPLIT; ++i) {
        const uint32_t c = warp + 8U * SPLIT * i;
        if (h0 + c >= H1) break;
        float v = tile[0][c][lane];
#pragma unroll
        for (int q = 1; q < SPLIT; ++q) v += tile[q][c][lane];
        const uint32_t word = __ballot_sync(0xFFFFFFFFU, s < B && v > 0.0f);
        if (lane == 0) bits[static_cast<uint64_t>(h0 + c) * ld_bits + (s0 >> 5)] = word;
        if (s < B) a1_t[static_cast<uint64_t>(h0 + c) * ld + s] = ptx::to_operand(fmaxf(v, 0.0f), kBf16);
    }
}

// The samples of each position in the order of their class there (stable, so sums over a class keep the sample order):
// order[p][first[p][v] .. first[p][v+1]) = samples with class v at position p. One CTA per position: every warp counts the
// classes of its own stretch of samples, the counts are scanned class by class, and the same sweep places the samples.
__global__ void __launch_bounds__(1024)
SortByClassKernel(const uint8_t* __restrict__ states, uint32_t B, uint32_t V, uint32_t* __restrict__ order, uint32_t* __restrict__ first) {
    __shared__ uint32_t count[32][80];
    __shared__ uint32_t base[81];
    const uint32_t p = blockIdx.x, warp = threadIdx.x >> 5, lane = threadIdx.x & 31U;
    for (uint32_t v = lane; v < 80U; v += 32U) count[warp][v] = 0U;
    __syncwarp();
    dependent_begin();
    const uint32_t stretch = ((B + 31U) / 32U + 31U) / 32U * 32U;
    const uint32_t lo = min(B, warp * stretch), hi = min(B, lo + stretch);
    for (uint32_t s = lo; s < hi; s += 32U) {
        const uint32_t v = s + lane < hi ? states[static_cast<uint64_t>(s + lane) * 80U + p] : 0xFFU;
        const uint32_t same = __match_any_sync(0xFFFFFFFFU, v);
        if (v < V && lane == static_cast<uint32_t>(__ffs(static_cast<int>(same))) - 1U) count[warp][v] += static_cast<uint32_t>(__popc(same));
        __syncwarp();
    }
    __syncthreads();
    if (threadIdx.x < V) {
        uint32_t sum = 0;
        for (uint32_t w = 0; w < 32U; ++w) {
            const uint32_t c = count[w][threadIdx.x];
            count[w][threadIdx.x] = sum;
            sum += c;
        }
        base[threadIdx.x + 1U] = sum;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        base[0] = 0U;
        for (uint32_t v = 1; v <= V; ++v) base[v] += base[v - 1U];
    }
    __syncthreads();
    if (threadIdx.x <= V) first[p * (V + 1U) + threadIdx.x] = base[threadIdx.x];
    for (uint32_t s = lo; s < hi; s += 32U) {
        const uint32_t v = s + lane < hi ? states[static_cast<uint64_t>(s + lane) * 80U + p] : 0xFFU;
        const uint32_t same = __match_any_sync(0xFFFFFFFFU, v);
        if (v < V) order[static_cast<uint64_t>(p) * B + base[v] + count[warp][v] + static_cast<uint32_t>(__popc(same & ((1U << lane) - 1U)))] = s + lane;
        __syncwarp();
        if (v < V && lane == static_cast<uint32_t>(__ffs(static_cast<int>(same))) - 1U) count[warp][v] += static_cast<uint32_t>(__popc(same));
        __syncwarp();
    }
}
// words of scratch for `order` and, behind it, `first`
inline uint64_t ListWords(uint32_t B, uint32_t L, uint32_t V) { return static_cast<uint64_t>(L) * B + static_cast<uint64_t>(L) * (V + 1U); }

// Table gradient from 16-bit dz1 [samples][ld]: grad[p*V + v][h] = sum of dz1[s][h] over the listed samples, zero where there
// are none. Eight lanes own 64 columns of a table row; SHARE = 4: four such groups share a row and take eight listed samples
// each in turn, added up at the end (few classes: few rows with long lists). The next sample numbers are fetched while the
// rows of the current ones are on their way. The column blocks are the slow grid dimension, so the slice of dz1 in use stays in
// L2. 3 001 samples x 2 560 columns, 72 classes: 82 us.
template <int SHARE, bool kBf16>
__global__ void __launch_bounds__(256)
GradKernel(const uint32_t* __restrict__ order, const uint32_t* __restrict__ first, const uint16_t* __restrict__ dz1, uint32_t ld, uint32_t B, uint32_t L, uint32_t V,
           uint32_t H1, float* __restrict__ grad_table, bool vec) {
    const uint32_t group = threadIdx.x >> 3, sub = threadIdx.x & 7U, lane = threadIdx.x & 31U;
    const uint32_t row = blockIdx.x * (32U / SHARE) + group / SHARE, part = group % SHARE;
    const uint32_t p = min(row / V, L - 1U), v = row - p * V;
    const bool live = row < L * V;
    const uint32_t h = blockIdx.y * 64U + sub * 8U;
    dependent_begin();
    first = after_begin(first);
    const uint32_t lo = live ? __ldg(first + p * (V + 1U) + v) : 0U, hi = live ? __ldg(first + p * (V + 1U) + v + 1U) : 0U;
    const uint32_t* list = order + static_cast<uint64_t>(p) * B;
    const uint32_t mask = 0xFFU << (lane & 24U);  // the eight lanes of this group
    float acc[8] = {};
    const bool in = h < H1;
    const uint16_t* col = dz1 + (in ? h : 0U);  // (lanes past the last column read the first ones and write nothing)
    uint32_t i = lo + part * 8U;
    uint32_t mine = i + sub < hi ? __ldg(list + i + sub) : 0U;
    while (i < hi) {
        const uint32_t n = i + 8U * SHARE;
        const uint32_t ahead = n + sub < hi ? __ldg(list + n + sub) : 0U;
        // loads without conditions, or they do not overlap: past the end of a list they read the first sample's row
        uint4 u[8];
#pragma unroll
        for (uint32_t j = 0; j < 8U; ++j) u[j] = LoadRow(col + static_cast<uint64_t>(__shfl_sync(mask, mine, j, 8)) * ld);
        if (i + 8U > hi) {
#pragma unroll
            for (uint32_t j = 0; j < 8U; ++j)
                if (i + j >= hi) u[j] = make_uint4(0U, 0U, 0U, 0U);
        }
#pragma unroll
        for (uint32_t j = 0; j < 8U; ++j) AddEight<kBf16>(acc, u[j]);
        i = n;
        mine = ahead;
    }
    if (SHARE > 1) {
        __syncwarp();
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            acc[e] += __shfl_xor_sync(0xFFFFFFFFU, acc[e], 8);
            acc[e] += __shfl_xor_sync(0xFFFFFFFFU, acc[e], 16);
        }
    }
    if (!in || !live || part != 0U) return;
    float* dst = grad_table + static_cast<uint64_t>(row) * H1 + h;
    if (vec) {
        *reinterpret_cast<float4*>(dst) = make_float4(acc[0], acc[1], acc[2], acc[3]);
        if (h + 4U < H1) *reinterpret_cast<float4*>(dst + 4) = make_float4(acc[4], acc[5], acc[6], acc[7]);
    } else {
#pragma unroll
        for (uint32_t e = 0; e < 8U; ++e)
            if (h + e < H1) dst[e] = acc[e];
    }
}

}  // namespace gather
}  // namespace mgt
