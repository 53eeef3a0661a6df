// Warp-specialised, persistent tcgen05 GEMM for sm_100a.
//
//   D[M x N] (fp32, TMEM) = A[M x K] * B[K x N]      fp16 operands, 128B-swizzled shared memory
//
// One CTA per SM. Warp 0 feeds operands with TMA (plain per-CTA loads, no multicast), warp 1
// issues tcgen05.mma from one thread and owns TMEM, warps 2-9 drain the accumulator
// (tcgen05.ld -> registers -> fused epilogue -> global). The embedding layer has kernels of its own
// (onehot_pair.cuh, embedding_gather.cuh).
//
// Operand forms
//   A  K-major  : global [M][K] (K contiguous), one TMA box 64(K) x 128(M) per stage
//   A  MN-major : global [K][M] (M contiguous), two TMA boxes 64(M) x 64(K) per stage
//   B  K-major  : global [N][K] (K contiguous), one TMA box 64(K) x BN(N)
//   B  MN-major : global [K][N] (N contiguous), ceil(BN/64) TMA boxes 64(N) x 64(K)
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "launch.cuh"
#include "ptx_sm100.cuh"

namespace mgt {

enum class BSource : int { kTmaK = 0, kTmaMN = 1 };

enum class Epi : int {
    kBiasReluF16 = 0,      // out_f16 = relu(acc + bias)
    kBiasReluF32F16,       // out_f32 = out_f16 = relu(acc + bias)
    kBiasResReluF32F16,    // v = relu(add + (acc + bias)); out_f32 = v (may alias add); out_f16 = v
    kMaskF16,              // out_f16 = acc * [mask > 0]
    kAddMaskF32F16,        // v = (acc + add) * [mask > 0]; out_f32 = v (may alias add); out_f16 = v
    kPartialF32,           // partial[split][m][n] = acc
    kBiasF32,              // out_f32 = acc + bias                 (a pre-activation kept in fp32: input of batch normalisation)
    kBiasF32Moments,       // the same, with the sums and the sums of squares of its columns in `moments`
    kMaskRowsumF16,        // out_f16[m][n] = acc * [bit n of bits[m]]; rowsum[(n tile, warp of the quadrant)][m] = sum over the warp's columns
    kMaskRowsumF16Tma,     // the same result by TMA stores through shared memory
    kMaskRowsumF32,        // the same values unrounded and transposed: out_f32[n][m] (the lanes of a warp write 32 neighbouring columns of one row)
    kMaskRowsumF16T,       // ... in the operand format: out_f16[n][m]
};

struct GemmArgs {
    uint32_t M, N, K;
    uint32_t m_tiles, n_tiles, splits, k_chunks;
    uint32_t groups;         // number of stacked problems (grouped form), else 1
    const float* bias;
    float* out_f32;
    uint32_t ld_f32;
    __half* out_f16;
    uint32_t ld_f16;
    const float* add_f32;
    uint32_t ld_add;
    const __half* mask;
    uint32_t ld_mask;
    float* partial;
    // Optional fp32 column sums of the values the kMaskF16 / kAddMaskF32F16 epilogues produce
    // (bias gradients): row (blockIdx.x * 8 + epilogue warp) of colsum[gridDim.x * 8][N] accumulates
    // what that warp handled. The buffer must be zero before the launch.
    float* colsum;
    // kBiasF32Moments: row (blockIdx.x * 4 + TMEM lane quadrant) of moments[gridDim.x * 4][2][N] gets what the quadrant's warps
    // handled; one N tile, every slot of a launch is written (no zeroing needed)
    float* moments;
    // kMaskRowsumF16: fp32 row sums of the masked values, one partial row of M floats per (N tile, warp of a lane quadrant):
    // rowsum[(n_tile * EPI_WARPS / 4 + w)][m]; every slot of a launch is written (no zeroing needed)
    float* rowsum;
    // kMaskRowsumF16 reads (the embedding forward wrote it): one 32-bit word per row and 32 columns, ld_bits words per row
    uint32_t* bits;
    uint32_t ld_bits;
    uint32_t bf16;           // operands and 16-bit outputs are bfloat16 instead of fp16
    int* status;             // device status word, 0 = ok
};

// BSTAT_: "B-stationary" - for short reductions (K <= 64*SB_) the whole B operand of the CTA's N tile is loaded
// once and stays in shared memory while the CTA streams its M tiles (all units of a CTA then share the N tile).
// GROUPED_: one launch computes args.groups independent products of the same shape; operand g is slice g
// (third coordinate) of the 3-D tensors behind the two descriptors, result g goes to its own partial planes.
template <int BN_, bool A_MN_, BSource BSRC_, Epi EPI_, int SA_, int SB_, bool BSTAT_ = false, bool GROUPED_ = false, int EPI_WARPS_ = 8>
struct GemmCfg {
    static constexpr bool BSTAT = BSTAT_;
    static constexpr bool GROUPED = GROUPED_;
    static constexpr int BM = 128;
    static constexpr int BK = 64;
    static constexpr int BN = BN_;
    static constexpr bool A_MN = A_MN_;
    static constexpr BSource BSRC = BSRC_;
    static constexpr Epi EPI = EPI_;
    static constexpr int SA = SA_;
    static constexpr int SB = SB_;
    static constexpr bool B_MN = (BSRC_ == BSource::kTmaMN);
    static constexpr int N_GROUPS = (BN_ + 63) / 64;
    static constexpr int A_STAGE_BYTES = BM * 128;
    static constexpr int B_STAGE_BYTES = B_MN ? N_GROUPS * 8192 : BN_ * 128;
    static constexpr int ACC_BUFS = 2;
    static constexpr int ACC_COLS = 256;  // TMEM columns reserved per accumulator
    static constexpr int EPI_WARPS = EPI_WARPS_;        // a multiple of four: EPI_WARPS/4 warps share a TMEM lane quadrant
    static constexpr int EPI_STRIDE = EPI_WARPS_ / 4;  // ... and take every EPI_STRIDE-th 32-column chunk
    static constexpr int THREADS = 64 + 32 * EPI_WARPS;
    static constexpr int EPI_TILE_PITCH = 36;
    static constexpr bool MOMENTS = EPI_ == Epi::kBiasF32Moments;
    // per epilogue warp: a padded 32x32 fp32 tile, 32 words of ReLU-mask bits and four rows of column-sum accumulators (eight for moments)
    // (the row-sum epilogues without TMA stores write from registers and need no staging)
    static constexpr bool TMA_OUT = EPI_ == Epi::kMaskRowsumF16Tma;  // two 32 x 32 tiles of the output per epilogue warp
    static constexpr int EPI_OFFSET = TMA_OUT ? 1024 : 256;          // behind the barriers; a swizzled tile starts on 512 bytes
    static constexpr int EPI_WARP_BYTES = TMA_OUT ? 2 * 2048 : (EPI_ == Epi::kMaskRowsumF16 || EPI_ == Epi::kMaskRowsumF32 || EPI_ == Epi::kMaskRowsumF16T) ? 0 : (32 * EPI_TILE_PITCH * 4 + 128 + (MOMENTS ? 8 : 4) * 32 * 4);
    static constexpr int EPI_STAGE_BYTES = EPI_WARPS * EPI_WARP_BYTES;
    static constexpr int SMEM_BYTES = 1024 + SA_ * A_STAGE_BYTES + SB_ * B_STAGE_BYTES + EPI_OFFSET + EPI_STAGE_BYTES;
    static_assert(BN_ % 16 == 0 && BN_ >= 16 && BN_ <= 256, "UMMA N");
    static_assert(BN_ % 32 == 0, "epilogue drains 32 columns at a time");
    static_assert(EPI_WARPS_ == 8 || EPI_WARPS_ == 16, "epilogue warps");
    static_assert(B_STAGE_BYTES % 1024 == 0, "swizzle atoms must stay 1024-byte aligned");
    static_assert(!GROUPED_ || (EPI_ == Epi::kPartialF32 && A_MN_ && BSRC_ == BSource::kTmaMN && !BSTAT_), "grouped form: split-K weight gradients");
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

template <class Cfg>
__global__ void __launch_bounds__(Cfg::THREADS, 1)
umma_gemm_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_b, const __grid_constant__ CUtensorMap tma_out, const GemmArgs args) {
    using namespace ptx;
    constexpr int BM = Cfg::BM, BN = Cfg::BN, SA = Cfg::SA, SB = Cfg::SB;
    // equal rings of A and B advance together: one barrier pair a stage
    constexpr bool kJoint = !Cfg::BSTAT && SA == SB;
    constexpr int ACC_BUFS = Cfg::ACC_BUFS;

    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    const uint32_t pad = ((raw_addr + 1023U) & ~1023U) - raw_addr;
    uint8_t* smem = smem_raw + pad;
    uint8_t* a_ring = smem;
    uint8_t* b_ring = smem + SA * Cfg::A_STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(b_ring + SB * Cfg::B_STAGE_BYTES);
    uint64_t* full_a = bars;
    uint64_t* empty_a = full_a + SA;
    uint64_t* full_b = empty_a + SA;
    uint64_t* empty_b = full_b + SB;
    uint64_t* acc_full = empty_b + SB;
    uint64_t* acc_empty = acc_full + ACC_BUFS;
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + ACC_BUFS);
    volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_holder + 1);
    float* epi_stage = reinterpret_cast<float*>(b_ring + SB * Cfg::B_STAGE_BYTES + Cfg::EPI_OFFSET);

    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t lane = threadIdx.x & 31U;
    const uint32_t units_per_group = args.m_tiles * args.n_tiles * args.splits;
    const uint32_t total_units = units_per_group * (Cfg::GROUPED ? args.groups : 1U);

    if (threadIdx.x == 0) {
        for (int s = 0; s < SA; ++s) {
            mbar_init(&full_a[s], 1);
            mbar_init(&empty_a[s], 1);
        }
        for (int s = 0; s < SB; ++s) {
            mbar_init(&full_b[s], 1);
            mbar_init(&empty_b[s], 1);
        }
        for (int s = 0; s < ACC_BUFS; ++s) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 32 * Cfg::EPI_WARPS);
        }
        *cta_abort = 0;
        fence_barrier_init();
        prefetch_tensormap(&tma_a);
        prefetch_tensormap(&tma_b);
        if (Cfg::TMA_OUT) prefetch_tensormap(&tma_out);
    }
    if (warp == 1) {
        tmem_alloc(tmem_holder, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    dependent_begin();
    // unit -> (m tile, n tile, split): splits of one tile are neighbours
    auto group_of = [&](uint32_t unit) { return Cfg::GROUPED ? unit / units_per_group : 0U; };
    auto decode = [&](uint32_t unit, uint32_t& mt, uint32_t& nt, uint32_t& sp) {
        if (Cfg::GROUPED) unit %= units_per_group;
        sp = unit % args.splits;
        const uint32_t rest = unit / args.splits;
        nt = rest % args.n_tiles;
        mt = rest / args.n_tiles;
    };
    auto chunk_begin = [&](uint32_t sp) { return static_cast<uint32_t>((static_cast<uint64_t>(sp) * args.k_chunks) / args.splits); };

    if (warp == 0) {
        // ------------------------------- TMA producer -------------------------------------
        // (a whole converged warp, as the issuer's: in one lane's loop the waits, expectations and six loads of a chunk of
        // 128 x 256 took twice its 512 cycles of MMAs)
        const uint32_t lead = elect_one();
        uint32_t it = 0;
        bool ok = true;
        for (uint32_t unit = blockIdx.x; unit < total_units && ok; unit += gridDim.x) {
            uint32_t mt, nt, sp;
            decode(unit, mt, nt, sp);
            const uint32_t c0 = chunk_begin(sp), c1 = chunk_begin(sp + 1);
            const int32_t m0 = static_cast<int32_t>(mt * BM), n0 = static_cast<int32_t>(nt * BN), z = Cfg::GROUPED ? static_cast<int32_t>(group_of(unit)) : 0;
            for (uint32_t c = c0; c < c1; ++c, ++it) {
                const uint32_t sa = it % SA, pa = (it / SA) & 1U;
                const int32_t k0 = static_cast<int32_t>(c * 64);
                if (!mbar_wait_warp(&empty_a[sa], pa ^ 1U, cta_abort, kAbortProducerWait)) { ok = false; break; }
                if (lead) {
                    uint8_t* a_dst = a_ring + sa * Cfg::A_STAGE_BYTES;
                    mbar_arrive_expect_tx(&full_a[sa], Cfg::A_STAGE_BYTES + (kJoint ? Cfg::B_STAGE_BYTES : 0));
                    if (Cfg::GROUPED) {
                        tma_load_3d(a_dst, &tma_a, m0, k0, z, &full_a[sa]);
                        tma_load_3d(a_dst + 8192, &tma_a, m0 + 64, k0, z, &full_a[sa]);
                    } else if (Cfg::A_MN) {
                        tma_load_2d(a_dst, &tma_a, m0, k0, &full_a[sa]);
                        tma_load_2d(a_dst + 8192, &tma_a, m0 + 64, k0, &full_a[sa]);
                    } else {
                        tma_load_2d(a_dst, &tma_a, k0, m0, &full_a[sa]);
                    }
                }
                if (!Cfg::BSTAT || unit == blockIdx.x) {
                    // B-stationary: chunk c of B lives in stage c for the whole kernel, loaded with the first unit
                    const uint32_t sb = Cfg::BSTAT ? (c - c0) : it % SB, pb = Cfg::BSTAT ? 0U : (it / SB) & 1U;
                    if (!Cfg::BSTAT && !kJoint && !mbar_wait_warp(&empty_b[sb], pb ^ 1U, cta_abort, kAbortProducerWait)) { ok = false; break; }
                    if (lead) {
                        uint8_t* b_dst = b_ring + sb * Cfg::B_STAGE_BYTES;
                        uint64_t* full = kJoint ? &full_a[sa] : &full_b[sb];
                        if (!kJoint) mbar_arrive_expect_tx(full, Cfg::B_STAGE_BYTES);
                        if (Cfg::GROUPED) {
#pragma unroll
                            for (int g = 0; g < Cfg::N_GROUPS; ++g) tma_load_3d(b_dst + g * 8192, &tma_b, n0 + g * 64, k0, z, full);
                        } else if (Cfg::B_MN) {
#pragma unroll
                            for (int g = 0; g < Cfg::N_GROUPS; ++g) tma_load_2d(b_dst + g * 8192, &tma_b, n0 + g * 64, k0, full);
                        } else {
                            tma_load_2d(b_dst, &tma_b, k0, n0, full);
                        }
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------- UMMA issuer --------------------------------------
        {
            const uint32_t lead = elect_one();
            const uint32_t idesc = make_idesc_f16(BM, BN, Cfg::A_MN, Cfg::B_MN, args.bf16 != 0U);
            uint32_t it = 0, unit_iter = 0;
            bool ok = true;
            for (uint32_t unit = blockIdx.x; unit < total_units && ok; unit += gridDim.x, ++unit_iter) {
                uint32_t mt, nt, sp;
                decode(unit, mt, nt, sp);
                const uint32_t c0 = chunk_begin(sp), c1 = chunk_begin(sp + 1);
                const uint32_t ab = unit_iter % ACC_BUFS, aph = (unit_iter / ACC_BUFS) & 1U;
                if (!mbar_wait_warp(&acc_empty[ab], aph ^ 1U, cta_abort, kAbortMmaWait)) { ok = false; break; }
                tc_fence_after();
                const uint32_t d_base = tmem_base + ab * Cfg::ACC_COLS;
                for (uint32_t c = c0; c < c1; ++c, ++it) {
                    const uint32_t sa = it % SA, pa = (it / SA) & 1U;
                    const uint32_t sb = Cfg::BSTAT ? (c - c0) : it % SB, pb = Cfg::BSTAT ? 0U : (it / SB) & 1U;
                    if (!mbar_wait_warp(&full_a[sa], pa, cta_abort, kAbortMmaWait)) { ok = false; break; }
                    if (!kJoint && (!Cfg::BSTAT || unit == blockIdx.x)) {
                        if (!mbar_wait_warp(&full_b[sb], pb, cta_abort, kAbortMmaWait)) { ok = false; break; }
                    }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(a_ring + sa * Cfg::A_STAGE_BYTES);
                    const uint32_t b_addr = smem_u32(b_ring + sb * Cfg::B_STAGE_BYTES);
                    const uint32_t k_left = args.K - c * 64U;
                    const uint32_t ksteps = k_left >= 64U ? 4U : (k_left + 15U) / 16U;
                    // Descriptors of the chunk's first K step; a later step only moves the start address (bits [0,14) in
                    // units of 16 bytes, no carry: shared-memory addresses are below 2^18). The fewer
                    // dependent instructions stand between two MMAs the better: the full chunk is unrolled.
                    constexpr uint64_t kStepA = Cfg::A_MN ? 2048U / 16U : 32U / 16U, kStepB = Cfg::B_MN ? 2048U / 16U : 32U / 16U;
                    const uint64_t a_desc0 = Cfg::A_MN ? make_smem_desc(a_addr, 8192U, 1024U) : make_smem_desc(a_addr, 16U, 1024U);
                    const uint32_t first = c > c0 ? 1U : 0U;
                    const uint64_t b_desc0 = Cfg::B_MN ? make_smem_desc(b_addr, 8192U, 1024U) : make_smem_desc(b_addr, 16U, 1024U);
                    if (ksteps == 4U) {
#pragma unroll
                        for (uint32_t kk = 0; kk < 4U; ++kk) umma_f16(lead, d_base, a_desc0 + kk * kStepA, b_desc0 + kk * kStepB, idesc, kk == 0U ? first : 1U);
                    } else {
                        for (uint32_t kk = 0; kk < ksteps; ++kk) umma_f16(lead, d_base, a_desc0 + kk * kStepA, b_desc0 + kk * kStepB, idesc, kk == 0U ? first : 1U);
                    }
                    umma_commit(lead, &empty_a[sa]);
                    if (!Cfg::BSTAT && !kJoint) umma_commit(lead, &empty_b[sb]);
                }
                if (ok) umma_commit(lead, &acc_full[ab]);
            }
        }
        __syncwarp();
    } else {
        // ------------------------------- epilogue -----------------------------------------
        // Eight warps: TMEM lanes [32*quad, 32*quad+32) can only be read by warps with warp%4 == quad, so two
        // warps share a quadrant and take alternate 32-column chunks.
        const uint32_t ew = warp - 2U;
        const uint32_t quad = warp & 3U;
        const uint32_t chunk_parity = ew >> 2;
        uint32_t unit_iter = 0;
        bool ok = true;
        if constexpr (Cfg::TMA_OUT || Cfg::EPI == Epi::kMaskRowsumF16 || Cfg::EPI == Epi::kMaskRowsumF32 || Cfg::EPI == Epi::kMaskRowsumF16T) {
            // D and the output have a row per TMEM lane and the warp's 32 columns side by side in that row: 64 bytes per lane,
            // written as four 16-byte vectors straight from registers; the mask of a chunk is one word per lane; the row
            // sum is a sum over the lane's own registers. (Full 32-byte sectors; whole rows per warp are not needed.)
            // TMA_OUT: a warp turns 32 rows x 32 columns into the operand format in a shared-memory tile of its own and a TMA store writes it,
            // while the next chunk goes into the other tile: a lane storing its 64 bytes straight from registers touches 32 lines per
            // instruction, and the load/store unit then bounds a CTA with more than one unit (a step of p888 at 53 248 samples
            // 3 044 -> 2 999 us, with batch normalisation 5 463 -> 5 395).
            const bool vec_ok = (args.ld_f16 & 7U) == 0U;
            [[maybe_unused]] uint8_t* tiles = reinterpret_cast<uint8_t*>(epi_stage) + ew * Cfg::EPI_WARP_BYTES;
            [[maybe_unused]] uint32_t stores = 0;
            constexpr int CPW = (BN / 32 + Cfg::EPI_STRIDE - 1) / Cfg::EPI_STRIDE;  // chunks of a unit per warp
            // the mask words of a unit do not depend on its MMAs: those of the NEXT unit are requested while this one is drained
            auto request = [&](uint32_t unit, uint32_t (&words)[CPW]) {
                uint32_t mt, nt, sp;
                decode(unit, mt, nt, sp);
                const uint32_t m = mt * BM + quad * 32U + lane;
#pragma unroll
                for (int ci = 0; ci < CPW; ++ci) {
                    const uint32_t n0 = nt * BN + (chunk_parity + ci * Cfg::EPI_STRIDE) * 32U;
                    words[ci] = (unit < total_units && m < args.M && n0 < args.N) ? __ldg(args.bits + static_cast<uint64_t>(m) * args.ld_bits + (n0 >> 5)) : 0U;
                }
            };
            uint32_t mw_next[CPW];
            request(blockIdx.x, mw_next);
            for (uint32_t unit = blockIdx.x; unit < total_units && ok; unit += gridDim.x, ++unit_iter) {
                uint32_t mt, nt, sp;
                decode(unit, mt, nt, sp);
                const uint32_t ab = unit_iter % ACC_BUFS, aph = (unit_iter / ACC_BUFS) & 1U;
                const uint32_t m = mt * BM + quad * 32U + lane;
                const bool m_ok = m < args.M;
                uint32_t mw[CPW];
#pragma unroll
                for (int ci = 0; ci < CPW; ++ci) mw[ci] = mw_next[ci];
                request(unit + gridDim.x, mw_next);
                if (!__all_sync(0xFFFFFFFFU, mbar_wait(&acc_full[ab], aph, cta_abort, kAbortEpilogueWait))) { ok = false; break; }
                tc_fence_after();
                float row_sum = 0.0f;
#pragma unroll
                for (int ci = 0; ci < CPW; ++ci) {
                    const uint32_t cc = chunk_parity + ci * Cfg::EPI_STRIDE;
                    const uint32_t n0 = nt * BN + cc * 32U;
                    if (cc >= static_cast<uint32_t>(BN / 32) || n0 >= args.N) continue;  // (warp-uniform)
                    const uint32_t valid = min(32U, args.N - n0);
                    const bool vec = valid == 32U && vec_ok;
                    uint32_t r[32];
                    tmem_ld_32x32(tmem_base + ((quad * 32U) << 16) + ab * Cfg::ACC_COLS + cc * 32, r);
                    tmem_ld_wait();
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = ((mw[ci] >> j) & 1U) ? __uint_as_float(r[j]) : 0.0f;
#pragma unroll
                    for (int j = 0; j < 32; ++j) row_sum += v[j];  // (columns past N were masked with zeros above)
                    if (Cfg::EPI == Epi::kMaskRowsumF32 || Cfg::EPI == Epi::kMaskRowsumF16T) {
                        if (m_ok) {
#pragma unroll
                            for (int j = 0; j < 32; ++j) {
                                if (static_cast<uint32_t>(j) >= valid) continue;
                                if (Cfg::EPI == Epi::kMaskRowsumF32) args.out_f32[static_cast<uint64_t>(n0 + j) * args.ld_f32 + m] = v[j];
                                else reinterpret_cast<uint16_t*>(args.out_f16)[static_cast<uint64_t>(n0 + j) * args.ld_f16 + m] = to_operand(v[j], args.bf16 != 0U);
                            }
                        }
                    } else if (Cfg::TMA_OUT) {
                        // (rows past M and columns past N are outside the map)
                        uint8_t* tile = tiles + (stores & 1U) * 2048U;
                        if (lane == 0) bulk_wait_read_but_one();  // the store before last has read this tile
                        __syncwarp();
#pragma unroll
                        for (uint32_t q = 0; q < 4U; ++q) {
                            uint4 u;
                            u.x = pack_operand_pair(v[8 * q + 0], v[8 * q + 1], args.bf16 != 0U);
                            u.y = pack_operand_pair(v[8 * q + 2], v[8 * q + 3], args.bf16 != 0U);
                            u.z = pack_operand_pair(v[8 * q + 4], v[8 * q + 5], args.bf16 != 0U);
                            u.w = pack_operand_pair(v[8 * q + 6], v[8 * q + 7], args.bf16 != 0U);
                            *reinterpret_cast<uint4*>(tile + lane * 64U + ((q ^ ((lane >> 1) & 3U)) << 4)) = u;  // 64-byte swizzle
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&tma_out, tile, static_cast<int32_t>(n0), static_cast<int32_t>(mt * BM + quad * 32U));
                            bulk_commit_group();
                        }
                        ++stores;
                    } else if (m_ok) {
                        uint16_t* dst = reinterpret_cast<uint16_t*>(args.out_f16) + static_cast<uint64_t>(m) * args.ld_f16 + n0;
                        if (vec) {
#pragma unroll
                            for (int q = 0; q < 4; ++q) {
                                uint4 u;
                                u.x = pack_operand_pair(v[8 * q + 0], v[8 * q + 1], args.bf16 != 0U);
                                u.y = pack_operand_pair(v[8 * q + 2], v[8 * q + 3], args.bf16 != 0U);
                                u.z = pack_operand_pair(v[8 * q + 4], v[8 * q + 5], args.bf16 != 0U);
                                u.w = pack_operand_pair(v[8 * q + 6], v[8 * q + 7], args.bf16 != 0U);
                                reinterpret_cast<uint4*>(dst)[q] = u;
                            }
                        } else {
#pragma unroll
                            for (int j = 0; j < 32; ++j)
                                if (static_cast<uint32_t>(j) < valid) dst[j] = to_operand(v[j], args.bf16 != 0U);
                        }
                    }
                }
                if (args.rowsum != nullptr && m_ok) args.rowsum[(static_cast<uint64_t>(nt) * Cfg::EPI_STRIDE + chunk_parity) * args.M + m] = row_sum;
                tc_fence_before();
                mbar_arrive(&acc_empty[ab]);
            }
            if (Cfg::TMA_OUT && lane == 0) bulk_wait_all();  // the stores read this CTA's shared memory until they complete
        } else {
            // Row-major tensors: a TMEM lane holds one row, but global memory wants a warp on whole rows. Each warp
            // stages operands and results through its own padded 32x32 fp32 tile in shared memory, so that every
            // global access is a full 64/128-byte row segment: 16-byte vectors, four (fp32) or eight (fp16) rows per
            // instruction. The global operands of a chunk (residual/skip values, ReLU mask source, bias) are
            // requested one chunk ahead - for the first chunk of a tile before the tile's MMAs have even finished -
            // so their latency is off the critical path. Ragged shapes take a scalar form without prefetch.
            constexpr bool kPlainF32 = Cfg::EPI == Epi::kBiasF32 || Cfg::MOMENTS;  // fp32 out only: no ReLU, no 16-bit copy
            constexpr bool kHasBias = Cfg::EPI == Epi::kBiasReluF16 || Cfg::EPI == Epi::kBiasReluF32F16 || Cfg::EPI == Epi::kBiasResReluF32F16 || kPlainF32;
            constexpr bool kHasAdd = Cfg::EPI == Epi::kBiasResReluF32F16 || Cfg::EPI == Epi::kAddMaskF32F16;
            constexpr bool kHasMask = Cfg::EPI == Epi::kMaskF16 || Cfg::EPI == Epi::kAddMaskF32F16;
            constexpr bool kOutF32 = Cfg::EPI == Epi::kBiasReluF32F16 || Cfg::EPI == Epi::kBiasResReluF32F16 || Cfg::EPI == Epi::kAddMaskF32F16 || kPlainF32;
            constexpr bool kPartial = Cfg::EPI == Epi::kPartialF32;
            constexpr uint32_t TP = Cfg::EPI_TILE_PITCH;  // floats per staged row (16-byte aligned, bank-friendly)
            float* tile = epi_stage + ew * (Cfg::EPI_WARP_BYTES / 4);
            uint32_t* mask_words = reinterpret_cast<uint32_t*>(tile + 32 * TP);
            // B-stationary kernels keep one N tile per CTA, so a warp meets the same (at most four) column chunks in every
            // unit: their column sums are accumulated here and written once at the end instead of a global
            // read-modify-write per chunk
            float* col_acc = reinterpret_cast<float*>(mask_words + 32);
            constexpr bool kColsumLocal = Cfg::BSTAT && kHasMask && BN / (32 * Cfg::EPI_STRIDE) <= 4;
            if (kColsumLocal || Cfg::MOMENTS) {
#pragma unroll
                for (int i = 0; i < (Cfg::MOMENTS ? 8 : 4); ++i) col_acc[i * 32 + lane] = 0.0f;
                __syncwarp();
            }
            const uint32_t r4 = lane >> 3, c4 = (lane & 7U) * 4U;  // fp32 vectors: 4 rows x 8 lanes
            const uint32_t r8 = lane >> 2, c8 = (lane & 3U) * 8U;  // fp16 vectors: 8 rows x 4 lanes
            const bool ld_vec = (!kHasAdd || (args.ld_add & 3U) == 0U) && (!kHasMask || (args.ld_mask & 7U) == 0U) &&
                                (!kOutF32 || (args.ld_f32 & 3U) == 0U) && (kPartial ? (args.N & 3U) == 0U : (kPlainF32 || (args.ld_f16 & 7U) == 0U));
            struct Operands {
                float4 add[kHasAdd ? 8 : 1];
                uint4 mask[kHasMask ? 4 : 1];
                float bias;
            };
            // requests the global operands of chunk n0 of the tile whose first row is m_base (vector form only)
            auto request = [&](Operands& o, uint32_t m_base, uint32_t rows_ok, uint32_t n0) {
                if (n0 + 32U > args.N || !ld_vec) return;
                if constexpr (kHasBias) o.bias = __ldg(args.bias + n0 + lane);
                if constexpr (kHasAdd) {
#pragma unroll
                    for (uint32_t i = 0; i < 8U; ++i) {
                        const uint32_t rr = r4 + 4U * i;
                        o.add[i] = rr < rows_ok ? *reinterpret_cast<const float4*>(args.add_f32 + static_cast<uint64_t>(m_base + rr) * args.ld_add + n0 + c4)
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
                    }
                }
                if constexpr (kHasMask) {
#pragma unroll
                    for (uint32_t i = 0; i < 4U; ++i) {
                        const uint32_t rr = r8 + 8U * i;
                        o.mask[i] = rr < rows_ok ? *reinterpret_cast<const uint4*>(args.mask + static_cast<uint64_t>(m_base + rr) * args.ld_mask + n0 + c8)
                                                 : make_uint4(0, 0, 0, 0);
                    }
                }
            };
            for (uint32_t unit = blockIdx.x; unit < total_units && ok; unit += gridDim.x, ++unit_iter) {
                uint32_t mt, nt, sp;
                decode(unit, mt, nt, sp);
                const uint32_t ab = unit_iter % ACC_BUFS, aph = (unit_iter / ACC_BUFS) & 1U;
                const uint32_t m_base = mt * BM + quad * 32U;
                const uint32_t rows_ok = m_base < args.M ? min(32U, args.M - m_base) : 0U;
                Operands next{};
                request(next, m_base, rows_ok, nt * BN + chunk_parity * 32U);
                // the TMEM loads below are warp-collective, so the whole warp takes the same way out
                if (!__all_sync(0xFFFFFFFFU, mbar_wait(&acc_full[ab], aph, cta_abort, kAbortEpilogueWait))) { ok = false; break; }
                tc_fence_after();
#pragma unroll 1
                for (int cc = static_cast<int>(chunk_parity); cc < BN / 32; cc += Cfg::EPI_STRIDE) {
                    const uint32_t n0 = nt * BN + cc * 32;
                    if (n0 >= args.N) break;
                    const Operands cur = next;
                    if (cc + Cfg::EPI_STRIDE < BN / 32) request(next, m_base, rows_ok, n0 + 32U * Cfg::EPI_STRIDE);
                    uint32_t r[32];
                    tmem_ld_32x32(tmem_base + ((quad * 32U) << 16) + ab * Cfg::ACC_COLS + cc * 32, r);
                    tmem_ld_wait();
                    const uint32_t valid = min(32U, args.N - n0);
                    const bool vec = valid == 32U && ld_vec;
                    const bool col_ok = lane < valid;
                    float v[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
                    if constexpr (kHasBias) {
                        const float bias_l = vec ? cur.bias : (col_ok ? __ldg(args.bias + n0 + lane) : 0.0f);
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] += __shfl_sync(0xFFFFFFFFU, bias_l, j);
                    }
                    if constexpr (kHasAdd) {
                        if (vec) {
#pragma unroll
                            for (uint32_t i = 0; i < 8U; ++i) *reinterpret_cast<float4*>(tile + (r4 + 4U * i) * TP + c4) = cur.add[i];
                        } else {
                            for (uint32_t rr = 0; rr < 32U; ++rr)
                                tile[rr * TP + lane] = (rr < rows_ok && col_ok) ? args.add_f32[static_cast<uint64_t>(m_base + rr) * args.ld_add + n0 + lane] : 0.0f;
                        }
                        __syncwarp();
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const float4 x = *reinterpret_cast<const float4*>(tile + lane * TP + q * 4);
                            v[q * 4] = x.x + v[q * 4];
                            v[q * 4 + 1] = x.y + v[q * 4 + 1];
                            v[q * 4 + 2] = x.z + v[q * 4 + 2];
                            v[q * 4 + 3] = x.w + v[q * 4 + 3];
                        }
                        __syncwarp();
                    }
                    if constexpr (kHasMask) {
                        uint32_t bits = 0;
                        if (vec) {
                            uint8_t* mask_bytes = reinterpret_cast<uint8_t*>(mask_words);
#pragma unroll
                            for (uint32_t i = 0; i < 4U; ++i) {
                                const uint32_t w4[4] = {cur.mask[i].x, cur.mask[i].y, cur.mask[i].z, cur.mask[i].w};
                                uint32_t byte = 0;
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    // a positive non-zero half: sign clear, magnitude non-zero
                                    const uint32_t lo = w4[e] & 0xFFFFU, hi = w4[e] >> 16;
                                    byte |= (lo != 0U && lo < 0x8000U) ? (1U << (2 * e)) : 0U;
                                    byte |= (hi != 0U && hi < 0x8000U) ? (1U << (2 * e + 1)) : 0U;
                                }
                                mask_bytes[(r8 + 8U * i) * 4U + (lane & 3U)] = static_cast<uint8_t>(byte);
                            }
                            __syncwarp();
                            bits = mask_words[lane];
                            __syncwarp();
                        } else {
                            for (uint32_t rr = 0; rr < 32U; ++rr) {
                                const uint16_t mh = (rr < rows_ok && col_ok) ? reinterpret_cast<const uint16_t*>(args.mask)[static_cast<uint64_t>(m_base + rr) * args.ld_mask + n0 + lane] : 0U;
                                const bool positive = mh != 0U && mh < 0x8000U;
                                const uint32_t row_bits = __ballot_sync(0xFFFFFFFFU, positive);
                                if (lane == rr) bits = row_bits;
                            }
                        }
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = ((bits >> j) & 1U) ? v[j] : 0.0f;
                    } else if constexpr (!kPartial && !kPlainF32) {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = fmaxf(v[j], 0.0f);
                    }
#pragma unroll
                    for (int q = 0; q < 8; ++q)
                        *reinterpret_cast<float4*>(tile + lane * TP + q * 4) = make_float4(v[q * 4], v[q * 4 + 1], v[q * 4 + 2], v[q * 4 + 3]);
                    __syncwarp();
                    if constexpr (kPartial || kOutF32) {
                        float* base = kPartial ? args.partial + ((static_cast<uint64_t>(group_of(unit)) * args.splits + sp) * args.M + m_base) * args.N + n0
                                               : args.out_f32 + static_cast<uint64_t>(m_base) * args.ld_f32 + n0;
                        const uint64_t ld = kPartial ? args.N : args.ld_f32;
                        if (vec) {
#pragma unroll
                            for (uint32_t i = 0; i < 8U; ++i) {
                                const uint32_t rr = r4 + 4U * i;
                                if (rr < rows_ok) *reinterpret_cast<float4*>(base + rr * ld + c4) = *reinterpret_cast<const float4*>(tile + rr * TP + c4);
                            }
                        } else {
                            for (uint32_t rr = 0; rr < rows_ok; ++rr)
                                if (col_ok) base[rr * ld + lane] = tile[rr * TP + lane];
                        }
                    }
                    if constexpr (!kPartial && !kPlainF32) {
                        if (vec) {
#pragma unroll
                            for (uint32_t i = 0; i < 4U; ++i) {
                                const uint32_t rr = r8 + 8U * i;
                                if (rr < rows_ok) {
                                    const float4 x0 = *reinterpret_cast<const float4*>(tile + rr * TP + c8);
                                    const float4 x1 = *reinterpret_cast<const float4*>(tile + rr * TP + c8 + 4U);
                                    const bool bf = args.bf16 != 0U;
                                    uint4 u;
                                    u.x = pack_operand_pair(x0.x, x0.y, bf);
                                    u.y = pack_operand_pair(x0.z, x0.w, bf);
                                    u.z = pack_operand_pair(x1.x, x1.y, bf);
                                    u.w = pack_operand_pair(x1.z, x1.w, bf);
                                    *reinterpret_cast<uint4*>(args.out_f16 + static_cast<uint64_t>(m_base + rr) * args.ld_f16 + n0 + c8) = u;
                                }
                            }
                        } else {
                            for (uint32_t rr = 0; rr < rows_ok; ++rr)
                                if (col_ok) reinterpret_cast<uint16_t*>(args.out_f16)[static_cast<uint64_t>(m_base + rr) * args.ld_f16 + n0 + lane] = to_operand(tile[rr * TP + lane], args.bf16 != 0U);
                        }
                    }
                    if constexpr (Cfg::MOMENTS) {
                        float s1 = 0.0f, s2 = 0.0f;  // column `lane` of the staged tile, rows in order
#pragma unroll 8
                        for (uint32_t rr = 0; rr < 32U; ++rr) {
                            const float x = rr < rows_ok ? tile[rr * TP + lane] : 0.0f;
                            s1 += x;
                            s2 += x * x;
                        }
                        col_acc[(cc / Cfg::EPI_STRIDE) * 64 + lane] += s1;  // this lane is the only user of the slots
                        col_acc[(cc / Cfg::EPI_STRIDE) * 64 + 32 + lane] += s2;
                    }
                    if constexpr (kHasMask) {
                        if (args.colsum != nullptr) {
                            float total = 0.0f;  // column `lane` of the staged tile, rows in order
#pragma unroll 8
                            for (uint32_t rr = 0; rr < 32U; ++rr) total += rr < rows_ok ? tile[rr * TP + lane] : 0.0f;
                            if (kColsumLocal) {
                                col_acc[(cc / Cfg::EPI_STRIDE) * 32 + lane] += total;  // this lane is the only user of the slot
                            } else if (col_ok) {
                                float* dst = args.colsum + (static_cast<uint64_t>(blockIdx.x) * Cfg::EPI_WARPS + ew) * args.N + n0 + lane;
                                *dst += total;  // this warp is the only writer of its row
                            }
                        }
                    }
                    __syncwarp();
                }
                tc_fence_before();
                mbar_arrive(&acc_empty[ab]);
            }
            if (Cfg::MOMENTS) {
                float* row = args.moments + (static_cast<uint64_t>(blockIdx.x) * 4U + quad) * 2U * args.N;
                for (int cc = static_cast<int>(chunk_parity); cc < BN / 32; cc += Cfg::EPI_STRIDE) {
                    const uint32_t n = cc * 32 + lane;
                    if (n < args.N) {
                        row[n] = col_acc[(cc / Cfg::EPI_STRIDE) * 64 + lane];
                        row[args.N + n] = col_acc[(cc / Cfg::EPI_STRIDE) * 64 + 32 + lane];
                    }
                }
            }
            if (kColsumLocal && args.colsum != nullptr && blockIdx.x < total_units) {
                const uint32_t nt = blockIdx.x % args.n_tiles;  // the N tile of every unit of this CTA
                for (int cc = static_cast<int>(chunk_parity); cc < BN / 32; cc += Cfg::EPI_STRIDE) {
                    const uint32_t n = nt * BN + cc * 32 + lane;
                    if (n < args.N) args.colsum[(static_cast<uint64_t>(blockIdx.x) * Cfg::EPI_WARPS + ew) * args.N + n] = col_acc[(cc / Cfg::EPI_STRIDE) * 32 + lane];
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (*cta_abort != 0) {
        // give copies that are still in flight time to land before the CTA's memory is released
        for (int i = 0; i < 2000; ++i) __nanosleep(1000);
        if (threadIdx.x == 0 && args.status != nullptr) atomicCAS(args.status, 0, *cta_abort);
        __syncthreads();
    }
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace mgt
