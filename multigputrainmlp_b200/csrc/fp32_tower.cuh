// The residual tower of the fp32 data flow in ONE launch per direction, on the CUDA cores (fma.rn.f32x2).
//
//   forward, block k :  T = relu(S * W1_k + b1_k)               -> r1[k]
//                       S = relu((T * W2_k + b2_k) + S)         -> x[k + 1]
//   backward, block k:  T = (S * W2_k^T) * [r1[k] > 0]          -> dz1t[k],  column sums in slot k
//   (k = R-1 .. 0)      S = (T * W1_k^T + S) * [x[k] > 0]       -> dz2[k],   column sums in slot R + k
//
// (mlp_backward.cu:1294-1323 and 1367-1413 are the reference's loops.) A CTA owns 8 W samples and carries them through all
// blocks. S and T lie in shared memory, one row per hidden unit, so that a warp's eight samples of a unit are two 16-byte
// broadcasts. A warp works on 8 samples x 32 NJ columns, a lane on columns 32 apart; CG warps side by side cover the width.
// One more warp fetches the weights into a ring of cp.async stages; the others wait for a stage on its mbarrier and not for each
// other, so that one is in its epilogue while its neighbour on the scheduler multiplies.
//
// Forward sums run in the order of k, as the tiles of SgemmKernel do: their results decide the ReLUs. Backward products are
// summed in pieces of at most 32 terms, a stage of weights each, that are then added up.
//
// What bounds it: the fp32 pipes where the batch fills the chip (a warp of 8 x 224 takes 78 cycles a k alone on its scheduler, two
// of them 142, for 28 fma.rn.f32x2 each), the chain of a warp where it does not. p888 (hd2 224, 16 blocks) at 8 192 samples: 0.70 ms
// forward and 0.75 ms backward; as 64 launches of tiled products 1.05 and 1.27 ms. Scalar multiply-adds take 211 cycles where pairs
// take 142.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>

#include "fp32_path.cuh"
#include "ptx_sm100.cuh"

namespace mgt {
namespace fp32path {

struct TowerArgs {
    uint32_t B, H, R, pitch;    // pitch: floats per sample of every activation and gradient
    // W1_0, W2_0, W1_1, ... w_step floats apart, rows of ld_w (a multiple of four, 16-byte aligned); their biases bias_step apart
    const float* w;
    const float* bias;
    uint64_t w_step, bias_step;
    uint32_t ld_w;
    float* state_tape;          // x[0..R] (forward) or dz2[0..R] (backward), tape_stride floats apart
    float* inner_tape;          // r1[0..R) or dz1t[0..R)
    uint64_t tape_stride;
    uint32_t* bits;             // ReLU signs of a sample, `words` per entry: entry k is r1[k], entry R + k is x[k]; entry_stride words apart
    uint64_t entry_stride;
    uint32_t words;
    float* colsum;              // backward: slot j at colsum + j * colsum_slot, one row of H per CTA
    uint64_t colsum_slot;
    uint32_t row_groups, col_groups;  // W and CG
    uint32_t chunk, stages;     // depth of a weight stage (a multiple of 8) and their number: kTowerStages, but as a constant it makes the kernel
                                // slower (p888 at 8 192 samples 3 670 -> 3 748 us a step)
    int* status;
};

// How a batch is cut. Columns of a warp: 32 NJ; the more, the fewer shared-memory reads a multiply-add needs, but the fewer warps.
struct TowerPlan {
    uint32_t nj, row_groups, col_groups, tiles, chunk;
    size_t smem;
    uint32_t rounds;  // of the chip, a tile to every place that an SM has for one
    double us;        // what a product of all samples takes in that many rounds, as measured (widths of 129 to 256)
};
constexpr uint32_t kTowerSmem = 227U * 1024U, kTowerBarBytes = 128U, kTowerStages = 3U;
inline uint32_t TowerThreads(uint32_t nj) { return nj >= 7U ? 256U : 512U; }          // of a CTA at most
inline uint32_t TowerResidentThreads(uint32_t nj) { return nj <= 2U ? 1024U : TowerThreads(nj); }  // of an SM, by registers
inline size_t TowerSmem(uint32_t H, uint32_t W, uint32_t padded, uint32_t chunk) {
    const size_t rows = (H + 15U) / 16U * 16U;
    return (2U * rows * (8U * W + 4U) + kTowerStages * static_cast<size_t>(padded) * (chunk + 4U) + 2U * W * padded) * sizeof(float) + kTowerBarBytes;
}
// words of sign bits of a sample
inline uint32_t TowerSampleWords(uint32_t H) { return H <= 128U || H > 224U ? (H + 31U) / 32U : 7U; }
// Picks the cut with the least estimated time: rounds of the chip x (cycles a k x H + 3 000 for epilogue and waits of a product). The
// cycles of a k are measured: those of one warp on its scheduler, and what every further one adds. So is the time of a round, for
// 100 units in us, with one warp on a scheduler and with more: by the steps of two rounds and more in the list at FusedFp32Tower.
inline TowerPlan PlanTower(uint32_t B, uint32_t H, uint32_t sm) {
    struct Width { uint32_t nj; double alone, each, round_alone, round; };
    constexpr Width kWidths[] = {{1U, 20.0, 20.0, 8.3, 8.3}, {2U, 46.0, 26.0, 8.3, 8.3}, {4U, 66.0, 45.0, 12.1, 12.1}, {7U, 78.0, 71.0, 8.4, 10.8}, {8U, 88.0, 81.0, 10.0, 13.2}};
    TowerPlan best{};
    double best_cost = 1e30;
    for (const Width& width : kWidths) {
        const uint32_t nj = width.nj, cg = (H + 32U * nj - 1U) / (32U * nj), padded = cg * nj * 32U;
        if (nj >= 7U && (cg > 1U || nj > TowerSampleWords(H))) continue;  // (never the best; a sample has TowerSampleWords words)
        for (uint32_t w = 1U; w <= 8U; ++w) {
            if ((w * cg + 1U) * 32U > TowerThreads(nj)) break;
            uint32_t chunk = 32U;  // the deepest stages of which three fit (of eight k they do for every width up to 256)
            while (chunk > 8U && (TowerSmem(H, w, padded, chunk) > kTowerSmem || chunk >= 2U * H)) chunk /= 2U;
            const size_t smem = TowerSmem(H, w, padded, chunk);
            const uint32_t tiles = (B + 8U * w - 1U) / (8U * w), warps = w * cg;
            const uint32_t resident = std::max<uint32_t>(1U, std::min<uint32_t>({static_cast<uint32_t>(kTowerSmem / (smem + 1024U)), TowerResidentThreads(nj) / (warps * 32U + 32U), tiles / sm}));
            const uint32_t rounds = (tiles + sm * resident - 1U) / (sm * resident);
            const double cost = rounds * (std::max(width.alone, width.each * ((warps * resident + 3U) / 4U)) * H + 3000.0 * resident);
            if (cost < best_cost) {
                best_cost = cost;
                best = {nj, w, cg, tiles, chunk, smem, rounds, rounds * (H / 100.0) * (warps * resident <= 4U ? width.round_alone : width.round)};
            }
        }
    }
    return best;
}
// words of one entry of sign bits, and rows of column sums of one slot, for any plan: neither falls with a larger batch
inline uint64_t TowerBitWords(uint32_t B, uint32_t H) { return static_cast<uint64_t>(B) * TowerSampleWords(H); }
inline uint64_t TowerSumRows(uint32_t B) { return (static_cast<uint64_t>(B) + 7U) / 8U; }

__device__ __forceinline__ void CopyAsync16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(ptx::smem_u32(dst)), "l"(src) : "memory");
}
// one arrival on the barrier once this thread's copies so far have landed
__device__ __forceinline__ void CopyAsyncArrive(uint64_t* bar) { asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(ptx::smem_u32(bar)) : "memory"); }
__device__ __forceinline__ void CopyAsyncWaitAll() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void AddPair(uint64_t& acc, uint64_t a) { asm("add.rn.f32x2 %0, %0, %1;" : "+l"(acc) : "l"(a)); }

// N k of a warp's 8 x 32 NJ tile; A as [k][row], B as [k][column], or as [column][k] with rows of 4 modulo 8 words (a quad of four
// k a lane, no bank conflicts)
template <int NJ, bool TB, uint32_t N>
__device__ __forceinline__ void TowerMultiply(uint64_t (&acc)[4][NJ], const float* a, uint32_t ld_a, const float* b, uint32_t ld_b) {
#pragma unroll
    for (uint32_t k4 = 0; k4 < N; k4 += 4U) {
        float q[4][NJ];
#pragma unroll
        for (int j = 0; j < NJ; ++j) {
            if (TB) {
                const float4 v = *reinterpret_cast<const float4*>(b + 32U * j * ld_b + k4);
                q[0][j] = v.x; q[1][j] = v.y; q[2][j] = v.z; q[3][j] = v.w;
            } else {
#pragma unroll
                for (uint32_t e = 0; e < 4U; ++e) q[e][j] = b[(k4 + e) * ld_b + 32U * j];
            }
        }
#pragma unroll
        for (uint32_t e = 0; e < 4U; ++e) {
            const ulonglong2 lo = *reinterpret_cast<const ulonglong2*>(a + (k4 + e) * ld_a), hi = *reinterpret_cast<const ulonglong2*>(a + (k4 + e) * ld_a + 4U);
            const uint64_t av[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const uint64_t bb = PackPair(q[e][j], q[e][j]);
#pragma unroll
                for (int i = 0; i < 4; ++i) FmaPair(acc[i][j], av[i], bb);
            }
        }
    }
}

// The tower's matrices with rows of whole quads, for widths and addresses that are none: matrix m of [H][H] at src + m * src_step goes to
// [pitch][pitch] at dst + m * pitch * pitch, the padding as zeros. A warp copies a row.
__global__ void __launch_bounds__(256)
PadMatricesKernel(const float* __restrict__ src, uint64_t src_step, uint32_t H, uint32_t pitch, float* __restrict__ dst) {
    const uint32_t row = blockIdx.x * 8U + (threadIdx.x >> 5), lane = threadIdx.x & 31U;
    dependent_begin();
    if (row >= pitch) return;
    const float* s = src + blockIdx.y * src_step + static_cast<uint64_t>(row) * H;
    float* d = dst + (static_cast<uint64_t>(blockIdx.y) * pitch + row) * pitch;
    for (uint32_t c = lane; c < pitch; c += 32U) d[c] = row < H && c < H ? __ldg(s + c) : 0.0f;
}

template <int NJ, bool BWD>
__global__ void __launch_bounds__(NJ >= 7 ? 256 : 512, NJ <= 2 ? 2 : 1)
TowerKernel(const __grid_constant__ TowerArgs a) {
    extern __shared__ __align__(16) float tower_f32[];
    const uint32_t H = a.H, W = a.row_groups, CG = a.col_groups, R = a.R;
    const uint32_t rows = (H + 15U) & ~15U, ld = 8U * W + 4U, padded = CG * NJ * 32U;
    const uint32_t pitch_w = BWD ? a.chunk + 4U : padded;                 // of a weight stage: [column][k] backward, [k][column] forward
    const uint32_t stage_floats = padded * (a.chunk + 4U);
    float* S = tower_f32;                      // [unit][sample]
    float* T = S + rows * ld;
    float* ring = T + rows * ld;
    float* red = ring + a.stages * stage_floats;  // backward: [product & 1][row group][column]
    uint64_t* full = reinterpret_cast<uint64_t*>(red + 2U * W * padded);
    uint64_t* empty = full + a.stages;
    volatile int* cta_abort = reinterpret_cast<volatile int*>(empty + a.stages);
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31U, warps = W * CG;
    const uint32_t chunks = (H + a.chunk - 1U) / a.chunk, products = 2U * R;
    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < a.stages; ++s) {
            ptx::mbar_init(&full[s], 32);
            ptx::mbar_init(&empty[s], warps);
        }
        *cta_abort = 0;
        ptx::fence_barrier_init();
    }
    __syncthreads();
    dependent_begin();

    // matrix of product p: W1_0, W2_0, W1_1, ... forward, W2_{R-1}, W1_{R-1}, W2_{R-2}, ... backward
    auto matrix = [&](uint32_t p) { return BWD ? 2U * R - 1U - p : p; };
    if (warp == warps) {
        // ------------------------------- weights ------------------------------------------
        uint32_t stage = 0, phase = 1;
        bool ok = true;
        for (uint32_t p = 0; p < products && ok; ++p) {
            for (uint32_t c = 0; c < chunks; ++c) {
                if (!ptx::mbar_wait_warp(&empty[stage], phase, cta_abort, ptx::kAbortProducerWait)) { ok = false; break; }
                const uint32_t k0 = c * a.chunk, deep = min(a.chunk, H - k0), quads = (deep + 3U) / 4U;
                float* dst = ring + stage * stage_floats;
                // (pieces of 128 bytes of as many rows as there are lanes for: whole rows one after the other are the same few lines for all
                // CTAs at once, and took the forward tower of p888 at 8 192 samples from 0.70 to 1.50 ms)
                const float* src = a.w + matrix(p) * a.w_step;
                if (BWD) {
                    // columns of the product are rows of the matrix: 4 `quads` neighbours of K of each
                    const uint32_t per = a.chunk / 4U, q = lane % per;  // 8, 4 or 2 lanes a column
                    for (uint32_t n = lane / per; n < H && q < quads; n += 32U / per) CopyAsync16(dst + n * pitch_w + 4U * q, src + static_cast<uint64_t>(n) * a.ld_w + k0 + 4U * q);
                } else {
                    for (uint32_t k = lane >> 3; k < 4U * quads; k += 4U)
                        for (uint32_t n = 4U * (lane & 7U); n < H; n += 32U) CopyAsync16(dst + k * pitch_w + n, src + static_cast<uint64_t>(k0 + k) * a.ld_w + n);
                }
                CopyAsyncArrive(&full[stage]);
                if (++stage == a.stages) {
                    stage = 0;
                    phase ^= 1U;
                }
            }
        }
        CopyAsyncWaitAll();
    } else {
        const uint32_t rg = warp / CG, cg = warp - rg * CG;
        const uint32_t col0 = cg * NJ * 32U + lane;                       // this lane's columns: col0 + 32 j
        const uint32_t row0 = blockIdx.x * 8U * W + rg * 8U;
        // sign words: this lane keeps word `lane` and word 32 + lane of the warp's 8 x NJ, counted row by row. Columns past the width
        // have none (but with one warp of 224 or 256 columns: asking there too costs that kernel 1 %), nor have rows past the batch: a
        // unit counts as closed there in the backward pass, whatever the forward pass made of their zeros (weights without bound make
        // NaN of them, which must not get into the column sums).
        constexpr uint32_t kWords = 8U * NJ;
        auto has_word = [&](uint32_t i) { return i < kWords && row0 + i / NJ < a.B && (NJ >= 7 || cg * NJ + i % NJ < a.words); };
        const bool word0 = has_word(lane), word1 = has_word(32U + lane);
        auto word_at = [&](uint32_t entry, uint32_t i) -> uint32_t* {
            return a.bits + entry * a.entry_stride + static_cast<uint64_t>(row0 + i / NJ) * a.words + cg * NJ + i % NJ;
        };
        auto store_words = [&](uint32_t entry, uint32_t w0, uint32_t w1) {
            if (word0) *word_at(entry, lane) = w0;
            if (word1) *word_at(entry, 32U + lane) = w1;
        };
        // the CG warps that share rows meet here after an epilogue (with column sums all warps of the CTA do)
        auto meet = [&]() {
            if (CG == 1U) __syncwarp();
            else ptx::named_bar_sync(1U + rg, 32U * CG);
        };
        // the state the tile starts with; rows past the batch and units past H are zeros
        {
            const float* src = a.state_tape + (BWD ? R * a.tape_stride : 0ULL);
            uint32_t w0 = 0, w1 = 0;
#pragma unroll
            for (int j = 0; j < NJ; ++j) {
                const uint32_t col = col0 + 32U * j;
                float v[8];
#pragma unroll
                for (uint32_t i = 0; i < 8U; ++i) v[i] = row0 + i < a.B && col < H ? src[static_cast<uint64_t>(row0 + i) * a.pitch + col] : 0.0f;
                if (col < rows) {
                    float4* d = reinterpret_cast<float4*>(S + col * ld + rg * 8U);
                    d[0] = make_float4(v[0], v[1], v[2], v[3]);
                    d[1] = make_float4(v[4], v[5], v[6], v[7]);
                    if (col >= H) {
                        float4* z = reinterpret_cast<float4*>(T + col * ld + rg * 8U);
                        z[0] = z[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    }
                }
                if (!BWD) {
#pragma unroll
                    for (uint32_t i = 0; i < 8U; ++i) {
                        const uint32_t word = __ballot_sync(0xFFFFFFFFU, v[i] > 0.0f), at = i * NJ + j;
                        if (at < 32U) w0 = lane == at ? word : w0;
                        else w1 = lane == at - 32U ? word : w1;
                    }
                }
            }
            if (!BWD) store_words(R, w0, w1);
            meet();
        }

        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (uint32_t p = 0; p < products; ++p) {  // (a warp whose wait has run out does no more work, but it still meets the others)
            const uint32_t k = BWD ? R - 1U - (p >> 1) : p >> 1;
            const bool second = (p & 1U) != 0U;
            const float* A = (second ? T : S) + rg * 8U;
            float bias[NJ];
            uint32_t m0 = 0, m1 = 0;
            if (BWD) {
                const uint32_t entry = second ? R + k : k;
                if (word0) m0 = *word_at(entry, lane);
                if (word1) m1 = *word_at(entry, 32U + lane);
            } else {
                const float* b = a.bias + matrix(p) * a.bias_step;
#pragma unroll
                for (int j = 0; j < NJ; ++j) bias[j] = col0 + 32U * j < H ? __ldg(b + col0 + 32U * j) : 0.0f;
            }
            uint64_t acc[4][NJ], sum[4][NJ];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < NJ; ++j) acc[i][j] = sum[i][j] = 0ULL;
            for (uint32_t c = 0; c < chunks && ok; ++c) {
                if (!ptx::mbar_wait_warp(&full[stage], phase, cta_abort, ptx::kAbortMmaWait)) { ok = false; break; }
                const float* as = A + c * a.chunk * ld;
                const float* bs = ring + stage * stage_floats + (BWD ? col0 * pitch_w : col0);
                const uint32_t deep = min(a.chunk, H - c * a.chunk);
                uint32_t kk = 0;
#pragma unroll 1
                for (; kk + 8U <= deep; kk += 8U) TowerMultiply<NJ, BWD, 8U>(acc, as + kk * ld, ld, BWD ? bs + kk : bs + kk * pitch_w, pitch_w);
#pragma unroll 1
                for (; kk < deep; kk += 4U) TowerMultiply<NJ, BWD, 4U>(acc, as + kk * ld, ld, BWD ? bs + kk : bs + kk * pitch_w, pitch_w);
                __syncwarp();
                if (lane == 0) ptx::mbar_arrive(&empty[stage]);
                if (BWD) {
#pragma unroll
                    for (int i = 0; i < 4; ++i)
#pragma unroll
                        for (int j = 0; j < NJ; ++j) {
                            AddPair(sum[i][j], acc[i][j]);
                            acc[i][j] = 0ULL;
                        }
                }
                if (++stage == a.stages) {
                    stage = 0;
                    phase ^= 1U;
                }
            }
            // epilogue: the rows it overwrites were read by the product before last, which the warps that share them have left
            float* out_s = second ? S : T;
            float* tape = (second ? a.state_tape + (BWD ? k : k + 1U) * a.tape_stride : a.inner_tape + k * a.tape_stride) + static_cast<uint64_t>(row0) * a.pitch;
            uint32_t w0 = 0, w1 = 0;
#pragma unroll
            for (int j = 0; j < NJ && ok; ++j) {
                const uint32_t col = col0 + 32U * j;
                const bool in = col < H;
                float v[8], old[8] = {};
#pragma unroll
                for (int i = 0; i < 4; ++i) UnpackPair(BWD ? sum[i][j] : acc[i][j], v[2 * i], v[2 * i + 1]);
                float4* d = reinterpret_cast<float4*>(out_s + col * ld + rg * 8U);
                if (second && in) {
                    const float4 lo = d[0], hi = d[1];
                    old[0] = lo.x; old[1] = lo.y; old[2] = lo.z; old[3] = lo.w;
                    old[4] = hi.x; old[5] = hi.y; old[6] = hi.z; old[7] = hi.w;
                }
                float total = 0.0f;
#pragma unroll
                for (uint32_t i = 0; i < 8U; ++i) {
                    const uint32_t at = i * NJ + j;
                    if (BWD) {
                        if (second) v[i] += old[i];
                        const uint32_t word = __shfl_sync(0xFFFFFFFFU, at < 32U ? m0 : m1, at & 31U);
                        v[i] = ((word >> lane) & 1U) != 0U && in ? v[i] : 0.0f;
                        total += v[i];
                    } else {
                        v[i] += bias[j];
                        if (second) v[i] += old[i];
                        v[i] = fmaxf(v[i], 0.0f);
                        const uint32_t word = __ballot_sync(0xFFFFFFFFU, in && v[i] > 0.0f);
                        if (at < 32U) w0 = lane == at ? word : w0;
                        else w1 = lane == at - 32U ? word : w1;
                    }
                }
                if (BWD) red[((p & 1U) * W + rg) * padded + col] = total;
                if (in) {
                    d[0] = make_float4(v[0], v[1], v[2], v[3]);
                    d[1] = make_float4(v[4], v[5], v[6], v[7]);
#pragma unroll
                    for (uint32_t i = 0; i < 8U; ++i)
                        if (row0 + i < a.B) tape[i * a.pitch + col] = v[i];
                }
            }
            if (BWD) {
                // column sums of the tile: a warp's eight rows, then the row groups in order
                ptx::named_bar_sync(15U, 32U * warps);
                for (uint32_t col = threadIdx.x; col < H && ok; col += 32U * warps) {
                    float total = 0.0f;
                    for (uint32_t g = 0; g < W; ++g) total += red[((p & 1U) * W + g) * padded + col];
                    a.colsum[(second ? R + k : k) * a.colsum_slot + static_cast<uint64_t>(blockIdx.x) * H + col] = total;
                }
            } else {
                if (ok && !(second && k + 1U == R)) store_words(second ? R + k + 1U : k, w0, w1);
                meet();
            }
        }
        if (!ok && lane == 0 && a.status != nullptr) atomicCAS(a.status, 0, *cta_abort);
    }
}

template <int NJ, bool BWD>
inline cudaError_t TowerRun(int device, LaunchOn st, const TowerArgs& a, const TowerPlan& plan) {
    // the opt-in shared-memory size is a per-device attribute of each kernel instantiation
    static std::mutex attr_mu;
    static bool attr_done[64] = {};
    if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
    {
        std::lock_guard<std::mutex> lock(attr_mu);
        if (!attr_done[device]) {
            const cudaError_t r = cudaFuncSetAttribute(TowerKernel<NJ, BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kTowerSmem));
            if (r != cudaSuccess) return r;
            attr_done[device] = true;
        }
    }
    return Launch(TowerKernel<NJ, BWD>, plan.tiles, 32U * (plan.row_groups * plan.col_groups + 1U), plan.smem, st, a);
}
template <bool BWD>
inline cudaError_t LaunchTower(int device, LaunchOn st, const TowerPlan& plan, TowerArgs a) {
    a.row_groups = plan.row_groups;
    a.col_groups = plan.col_groups;
    a.chunk = plan.chunk;
    a.stages = kTowerStages;
    a.words = TowerSampleWords(a.H);
    switch (plan.nj) {
        case 1: return TowerRun<1, BWD>(device, st, a, plan);
        case 2: return TowerRun<2, BWD>(device, st, a, plan);
        case 4: return TowerRun<4, BWD>(device, st, a, plan);
        case 7: return TowerRun<7, BWD>(device, st, a, plan);
        case 8: return TowerRun<8, BWD>(device, st, a, plan);
    }
    return cudaErrorInvalidValue;
}

}  // namespace fp32path
}  // namespace mgt
