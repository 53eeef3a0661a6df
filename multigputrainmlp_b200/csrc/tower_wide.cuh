// The residual tower for widths of 257 to 512, one kernel per direction, a pair of CTAs per tile (sm_100a, tcgen05 + TMEM).
//
// As tower_chain.cuh - 128 samples carried through all blocks, the fp32 state S and the product D in TMEM, epilogues that
// write the next operand, tapes by TMA store - but S and D of a tile take 2 H columns of TMEM and only 512 are there. So the
// two CTAs of a cluster share a tile: each computes half of the columns (whole 64-column panels) and keeps S and D of those,
// and both hold the whole A operand in shared memory. A panel that one CTA's epilogue finishes is copied into the other's
// shared memory (cp.async.bulk between the CTAs, counted on the barrier the other's MMAs wait for); an MMA starts with the
// panels of its own CTA while the others are on their way. One operand buffer serves S and T in turn: an epilogue starts
// when the MMAs of both CTAs have read it.
//
// Layer by layer these widths took four GEMM launches a block that each moved the fp32 stream, the operand and its copy
// through HBM: hd2 512, 32 blocks, 131 072 samples 17.7 ms, 13.2 ms here.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "launch.cuh"
#include "onehot_pair.cuh"
#include "ptx_sm100.cuh"
#include "tower_chain.cuh"

namespace mgt {

struct WideCfg {
    static constexpr int EPI_WARPS = 16;            // a multiple of four: EPI_WARPS/4 warps share a TMEM lane quadrant
    static constexpr int COPY_WARP = 2 + EPI_WARPS;
    static constexpr int THREADS = 32 * (COPY_WARP + 1);
    static constexpr int SW = 3;                    // weight ring stages
    static constexpr int ACT_BYTES = 8 * 16384;     // the operand: up to eight 64-column panels of 128 rows x 128 bytes
    static constexpr int W_STAGE_BYTES = 32768;
    static constexpr int SMEM_BYTES = ACT_BYTES + SW * W_STAGE_BYTES + 256 + 2048;  // + barriers + bias slices
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

namespace detail {

// arrives on the barrier at this offset in both CTAs of the cluster once every MMA of this CTA issued so far has completed
__device__ __forceinline__ void umma_commit_pair(uint32_t lead, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
        ::"r"(ptx::smem_u32(bar)), "h"(static_cast<uint16_t>(3)), "r"(lead)
        : "memory");
}
// shared memory of this CTA -> shared memory of another, bytes counted on a barrier there
__device__ __forceinline__ void copy_to_cluster(uint32_t dst_cluster, uint32_t src, uint32_t bytes, uint32_t bar_cluster) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst_cluster), "r"(src), "r"(bytes), "r"(bar_cluster) : "memory");
}

}  // namespace detail

template <bool BWD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(WideCfg::THREADS, 1)
tower_wide_kernel(const __grid_constant__ CUtensorMap tma_w, const __grid_constant__ CUtensorMap tma_tape_s,
                   const __grid_constant__ CUtensorMap tma_tape_t, const ChainArgs args) {
    using namespace ptx;
    constexpr int SW = WideCfg::SW;
    constexpr uint32_t kStateCol = 256;  // first TMEM column of S

    extern __shared__ __align__(1024) uint8_t tower_smem[];
    uint8_t* smem = tower_smem;
    uint8_t* act = smem;                            // the A operand of the MMA at hand: S or T rounded, all H columns
    uint8_t* w_ring = smem + WideCfg::ACT_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(w_ring + SW * WideCfg::W_STAGE_BYTES);
    uint64_t* w_full = bars;
    uint64_t* w_empty = w_full + SW;
    uint64_t* ready = w_empty + SW;     // [8] K chunk c of the operand is there: own chunks from the epilogue, the others by copy
    uint64_t* mma_done = ready + 8;     // [2] D / S complete in both CTAs and the operand's panels stored
    uint64_t* sums_done = mma_done + 2; // [2] backward: every epilogue warp has read its bias sums out of D / out of S
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(sums_done + 2);
    volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_holder + 1);
    float* bias_slots = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(bars) + 256);  // [products of a block][warps per quadrant][chunks per warp][32]

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31U;
    const uint32_t H = args.H, R = args.R, rank = pair::cluster_rank();
    const uint32_t HC = ((H + 127U) / 128U) * 64U;  // columns of the first CTA: half of them in whole panels
    const uint32_t col0 = rank * HC;                // this CTA's columns: [col0, col0 + own), worked on in chunks of 32
    const uint32_t own = rank == 0U ? HC : H - HC;
    const uint32_t NC = (own + 31U) / 32U;          // 32-column chunks of an epilogue
    const uint32_t KC = (H + 63U) / 64U;            // K chunks of an MMA
    const uint32_t PC = (own + 63U) / 64U, p0 = rank * (HC / 64U);  // the chunks this CTA writes: [p0, p0 + PC)
    // K chunks in the order this CTA takes them: its own first, they are there sooner
    auto chunk_at = [&](uint32_t i) { return i < PC ? p0 + i : (rank == 0U ? i : i - PC); };
    auto mine = [&](uint32_t c) { return c - p0 < PC; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < SW; ++s) {
            mbar_init(&w_full[s], 1);
            mbar_init(&w_empty[s], 1);
        }
        for (uint32_t c = 0; c < 8U; ++c) {
            // one arrival per epilogue warp that owns a 32-column chunk inside K chunk c; for a copied one the byte count's
            const uint32_t chunks = mine(c) ? (NC - 2U * (c - p0) >= 2U ? 2U : 1U) : 1U;
            mbar_init(&ready[c], mine(c) ? 4U * chunks : 1U);
        }
        mbar_init(&mma_done[0], 3);  // the commits of both CTAs and the storing warp
        mbar_init(&mma_done[1], 3);
        mbar_init(&sums_done[0], WideCfg::EPI_WARPS);
        mbar_init(&sums_done[1], WideCfg::EPI_WARPS);
        *cta_abort = 0;
        fence_barrier_init();
        prefetch_tensormap(&tma_w);
        prefetch_tensormap(&tma_tape_s);
        prefetch_tensormap(&tma_tape_t);
    }
    if (warp == 1) {
        tmem_alloc(tmem_holder, 512);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    pair::cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    dependent_begin();
    const uint32_t cluster = blockIdx.x >> 1, clusters = gridDim.x >> 1;

    if (warp == 0) {
        // ------------------------------- weight stream ------------------------------------
        if (lane == 0) {
            const uint32_t stage_bytes = HC * 128U;
            uint32_t it = 0;
            bool ok = true;
            for (uint32_t tile = cluster; tile < args.tiles && ok; tile += clusters) {
                for (uint32_t l = 0; l < 2U * R && ok; ++l) {
                    // forward visits W1_0, W2_0, W1_1, ...; backward W2_{R-1}, W1_{R-1}, W2_{R-2}, ...
                    const int32_t z = static_cast<int32_t>(BWD ? (2U * (R - 1U - (l >> 1)) + ((l & 1U) ^ 1U)) : l);
                    for (uint32_t i = 0; i < KC; ++i, ++it) {
                        const uint32_t c = chunk_at(i);
                        const uint32_t s = it % SW, ph = (it / SW) & 1U;
                        if (!mbar_wait_spin(&w_empty[s], ph ^ 1U, cta_abort, kAbortChainWait)) { ok = false; break; }
                        uint8_t* dst = w_ring + s * WideCfg::W_STAGE_BYTES;
                        mbar_arrive_expect_tx(&w_full[s], stage_bytes);
                        if (BWD) {
                            // B[N = in][K = out], K contiguous: one box 64(K) x HC(N)
                            tma_load_3d(dst, &tma_w, static_cast<int32_t>(c * 64U), static_cast<int32_t>(col0), z, &w_full[s]);
                        } else {
                            // B[K = in][N = out], N contiguous: boxes 64(N) x 64(K)
                            for (uint32_t g = 0; g < HC / 64U; ++g)
                                tma_load_3d(dst + g * 8192U, &tma_w, static_cast<int32_t>(col0 + g * 64U), static_cast<int32_t>(c * 64U), z, &w_full[s]);
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
            const uint32_t idesc = make_idesc_f16(128, NC * 32U, false, !BWD, args.bf16 != 0U);
            uint32_t it = 0, step = 0;
            bool ok = true;
            for (uint32_t tile = cluster; tile < args.tiles && ok; tile += clusters) {
                for (uint32_t kb = 0; kb < R && ok; ++kb) {
                    for (uint32_t half = 0; half < 2U && ok; ++half, ++step) {
                        // (the bias sums are read after the panels are handed on, and a panel may be in before they are: see tower_chain.cuh)
                        if (BWD && !mbar_wait_warp(&sums_done[half], ((step >> 1) & 1U) ^ 1U, cta_abort, kAbortChainWait)) { ok = false; break; }
                        const uint32_t a_base = smem_u32(act);
                        const uint32_t d_addr = tmem_base + (half ? kStateCol : 0U);
                        for (uint32_t c = 0; c < KC; ++c)
                            if (lead && !mine(c)) mbar_arrive_expect_tx(&ready[c], 16384U);
                        for (uint32_t i = 0; i < KC; ++i, ++it) {
                            const uint32_t c = chunk_at(i);
                            const uint32_t s = it % SW, ph = (it / SW) & 1U;
                            if (!mbar_wait_warp(&ready[c], step & 1U, cta_abort, kAbortChainWait)) { ok = false; break; }
                            if (!mbar_wait_warp(&w_full[s], ph, cta_abort, kAbortChainWait)) { ok = false; break; }
                            tc_fence_after();
                            const uint32_t a_addr = a_base + c * 16384U;
                            const uint32_t b_addr = smem_u32(w_ring + s * WideCfg::W_STAGE_BYTES);
                            const uint32_t k_left = H - c * 64U;
                            const uint32_t ksteps = k_left >= 64U ? 4U : (k_left + 15U) / 16U;
                            // descriptors of the chunk's first K step; a later step only moves the start address (units of 16
                            // bytes, no carry out of the field).
                            const uint64_t a_desc0 = make_smem_desc(a_addr, 16U, 1024U);
                            const uint64_t b_desc0 = BWD ? make_smem_desc(b_addr, 16U, 1024U) : make_smem_desc(b_addr, 8192U, 1024U);
                            constexpr uint64_t kStepA = 32U / 16U, kStepB = BWD ? 32U / 16U : 2048U / 16U;
                            // the second product of a block adds onto the state that already sits in TMEM
                            const uint32_t first = (half != 0U || i > 0U) ? 1U : 0U;
                            if (ksteps == 4U) {
#pragma unroll
                                for (uint32_t kk = 0; kk < 4U; ++kk) umma_f16(lead, d_addr, a_desc0 + kk * kStepA, b_desc0 + kk * kStepB, idesc, kk == 0U ? first : 1U);
                            } else {
                                for (uint32_t kk = 0; kk < ksteps; ++kk) umma_f16(lead, d_addr, a_desc0 + kk * kStepA, b_desc0 + kk * kStepB, idesc, kk == 0U ? first : 1U);
                            }
                            umma_commit(lead, &w_empty[s]);
                        }
                        if (ok) detail::umma_commit_pair(lead, &mma_done[half]);
                    }
                }
            }
        }
        __syncwarp();
    } else if (warp == WideCfg::COPY_WARP) {
        // ------------------------------- panels to the other CTA and to the tape ----------
        // Every panel this CTA's epilogue finishes goes to the same place in the other CTA's shared memory, counted on the barrier
        // its MMAs wait for, and, being a 64-column slice of a tape entry too, to the tape (T of this block, or the S the
        // previous block produced; the S a tile starts with is on its tape already).
        if (lane == 0) {
            uint32_t step = 0;
            bool ok = true;
            for (uint32_t tile = cluster; tile < args.tiles && ok; tile += clusters) {
                for (uint32_t kb = 0; kb < R && ok; ++kb) {
                    for (uint32_t half = 0; half < 2U && ok; ++half, ++step) {
                        const uint32_t k = BWD ? R - 1U - kb : kb;
                        const uint32_t entry = half ? k : (BWD ? k + 1U : k);
                        for (uint32_t i = 0; i < PC; ++i) {
                            const uint32_t c = p0 + i;
                            if (!mbar_wait_spin(&ready[c], step & 1U, cta_abort, kAbortChainWait)) { ok = false; break; }
                            const uint32_t src = smem_u32(act + c * 16384U);
                            detail::copy_to_cluster(pair::map_to(src, rank ^ 1U), src, 16384U, pair::map_to(smem_u32(&ready[c]), rank ^ 1U));
                        }
                        if (ok && (half != 0U || kb > 0U))  // (behind the copies: the other CTA waits for them)
                            for (uint32_t c = p0; c < p0 + PC; ++c)
                                tma_store_3d(half ? &tma_tape_t : &tma_tape_s, act + c * 16384U, static_cast<int32_t>(c * 64U), static_cast<int32_t>(tile * 128U),
                                             static_cast<int32_t>(entry));
                        bulk_commit_group();
                        bulk_wait_read_all();  // the epilogue that follows overwrites the panels
                        if (ok) mbar_arrive(&mma_done[half]);
                    }
                }
            }
            bulk_wait_all();  // the tape stores read this CTA's shared memory until they complete
        }
        __syncwarp();
    } else {
        // ------------------------------- epilogue -----------------------------------------
        const uint32_t ew = warp - 2U;
        const uint32_t quad = warp & 3U;       // TMEM lanes [32*quad, 32*quad+32)
        constexpr uint32_t SUBS = WideCfg::EPI_WARPS / 4;  // warps per quadrant
        constexpr uint32_t WPW = 8U / SUBS;                  // 32-column chunks (and sign-bit words) per warp at most
        static_assert(WPW == 2U, "sign words move as pairs");
        const uint32_t par = ew >> 2;          // this warp takes 32-column chunks par, par+SUBS, ...
        const uint32_t r = quad * 32U + lane;  // row inside the tile
        const uint32_t lane_addr = (quad * 32U) << 16;
        // byte offset of 16-byte unit u (0..7) of this row inside a 64-column panel, 128B swizzle
        auto unit_off = [&](uint32_t u) { return r * 128U + ((u ^ (r & 7U)) << 4); };
        auto store_operand = [&](uint32_t cc, const uint32_t (&h)[16]) {
            uint8_t* panel = act + (p0 + (cc >> 1)) * 16384U;
#pragma unroll
            for (uint32_t q = 0; q < 4U; ++q)
                *reinterpret_cast<uint4*>(panel + unit_off((cc & 1U) * 4U + q)) = make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
        };
        auto store_tape = [&](__half* row_ptr, uint32_t cc, const uint32_t (&h)[16]) {
            uint4* dst = reinterpret_cast<uint4*>(row_ptr + col0 + cc * 32U);
#pragma unroll
            for (uint32_t q = 0; q < 4U; ++q)
                if (col0 + cc * 32U + 8U * q < args.ld_s) dst[q] = make_uint4(h[4 * q], h[4 * q + 1], h[4 * q + 2], h[4 * q + 3]);
        };
        // lane 0 polls, the warp follows: the result is warp-uniform
        auto warp_wait = [&](uint64_t* bar, uint32_t parity) -> bool {
            uint32_t done = 0;
            if (lane == 0) done = mbar_wait_spin(bar, parity, cta_abort, kAbortChainWait) ? 1U : 0U;
            return __shfl_sync(0xFFFFFFFFU, done, 0) != 0U;
        };
        auto publish = [&](uint64_t* bar) {
            fence_proxy_async_smem();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar);
        };
        // Bias of a layer: before the warp waits for the MMAs each lane fetches one value per chunk of its warp into a shared-memory
        // slot, so that every thread can read all 32 of a chunk as broadcast vectors. The warps of one quadrant set share
        // slots and write identical values; a slot is rewritten two products later, after MMAs that needed every warp's
        // epilogue in between.
        auto stage_bias = [&](uint32_t layer) {
            if (!BWD) {
#pragma unroll
                for (uint32_t ci = 0; ci < WPW; ++ci) {
                    const uint32_t cc = par + SUBS * ci;
                    bias_slots[(layer & 1U) * 256U + (par * WPW + ci) * 32U + lane] = col0 + cc * 32U + lane < H ? __ldg(args.bias + layer * args.bias_stride + col0 + cc * 32U + lane) : 0.0f;
                }
                __syncwarp();
            }
        };
        auto store_words = [&](uint32_t* dst, const uint32_t (&wd)[WPW]) { *reinterpret_cast<uint2*>(dst) = make_uint2(wd[0], wd[1]); };
        auto load_words = [&](const uint32_t* src, uint32_t (&wd)[WPW]) {
            const uint2 m = *reinterpret_cast<const uint2*>(src);
            wd[0] = m.x; wd[1] = m.y;
        };
        auto apply_mask = [&](uint32_t (&v)[32], uint32_t bits) {
#pragma unroll
            for (int j = 0; j < 32; ++j) v[j] = ((bits >> j) & 1U) ? v[j] : 0U;
        };
        // bias sums of a product (its columns from `taddr` on), when the panels are handed on; `done`: the columns may be overwritten
        auto column_sums = [&](uint32_t taddr, uint32_t tile, uint32_t slot, uint64_t* done) {
            tmem_st_wait();
#pragma unroll
            for (uint32_t ci = 0; ci < WPW; ++ci) {
                const uint32_t cc = par + SUBS * ci;
                if (cc >= NC) break;
                uint32_t j;
                const float total = detail::column_sums(taddr + cc * 32U, lane, &j);
                const uint32_t col = col0 + cc * 32U + j;
                if (col < H) args.colsum[slot * args.colsum_stride + (static_cast<uint64_t>(tile) * 4U + quad) * H + col] = total;
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(done);
        };

        uint32_t uses = 0;
        bool ok = true;
        for (uint32_t tile = cluster; tile < args.tiles && ok; tile += clusters) {
            const uint64_t row = static_cast<uint64_t>(tile) * 128U + r;
            const bool row_ok = row < args.samples;
            const uint64_t bits_row = row * 16U + rank * 8U + par * WPW;  // this warp's words of the row

            // ---- load the state: TMEM S, fp16 operand, (forward) sign bits of x_0
            {
                uint32_t words[WPW] = {0, 0};
#pragma unroll
                for (uint32_t ci = 0; ci < WPW; ++ci) {
                    const uint32_t cc = par + SUBS * ci;
                    if (cc >= NC) break;
                    float v[32];
                    if (row_ok && col0 + cc * 32U + 32U > H) {
#pragma unroll
                        for (uint32_t j = 0; j < 32U; ++j) v[j] = col0 + cc * 32U + j < H ? args.state_f32[row * args.ld_f32 + col0 + cc * 32U + j] : 0.0f;
                    } else if (row_ok) {
                        const float4* src = reinterpret_cast<const float4*>(args.state_f32 + row * args.ld_f32 + col0 + cc * 32U);
#pragma unroll
                        for (int q = 0; q < 8; ++q) {
                            const float4 f = src[q];
                            v[4 * q] = f.x; v[4 * q + 1] = f.y; v[4 * q + 2] = f.z; v[4 * q + 3] = f.w;
                        }
                    } else {
#pragma unroll
                        for (int j = 0; j < 32; ++j) v[j] = 0.0f;
                    }
                    uint32_t raw[32];
#pragma unroll
                    for (int j = 0; j < 32; ++j) raw[j] = __float_as_uint(v[j]);
                    tmem_st_32x32(tmem_base + lane_addr + kStateCol + cc * 32U, raw);
                    uint32_t h[16];
                    detail::pack_operands(raw, h, args.bf16 != 0U);
                    if (!BWD) words[ci] = detail::positive_bits(raw);
                    store_operand(cc, h);
                    tmem_st_wait();
                    publish(&ready[p0 + (cc >> 1)]);
                }
                if (!BWD) store_words(args.bits_s + bits_row, words);
            }

            for (uint32_t kb = 0; kb < R && ok; ++kb, ++uses) {
                const uint32_t k = BWD ? R - 1U - kb : kb;
                const bool last = kb + 1U == R;
                // ================= first epilogue: T from D =================
                {
                    uint32_t mwords[WPW] = {0, 0};
                    if (BWD) load_words(args.bits_t + k * args.bits_stride + bits_row, mwords);
                    uint32_t words[WPW] = {0, 0};
                    stage_bias(2U * k);
                    if (!warp_wait(&mma_done[0], uses & 1U)) { ok = false; break; }
                    tc_fence_after();
#pragma unroll
                    for (uint32_t ci = 0; ci < WPW; ++ci) {
                        const uint32_t cc = par + SUBS * ci;
                        if (cc >= NC) break;
                        uint32_t raw[32];
                        tmem_ld_32x32(tmem_base + lane_addr + cc * 32U, raw);
                        tmem_ld_wait();
                        uint32_t h[16];
                        if (BWD) {
                            apply_mask(raw, mwords[ci]);
                            tmem_st_32x32(tmem_base + lane_addr + cc * 32U, raw);  // (for the column sums)
                        } else {
                            detail::add_bias_relu(raw, bias_slots + (par * WPW + ci) * 32U);
                        }
                        detail::pack_operands(raw, h, args.bf16 != 0U);
                        store_operand(cc, h);
                        publish(&ready[p0 + (cc >> 1)]);
                        if (!BWD) words[ci] = detail::positive_bits(raw);
                    }
                    if (BWD) column_sums(tmem_base + lane_addr, tile, k, &sums_done[0]);
                    if (!BWD) store_words(args.bits_t + k * args.bits_stride + bits_row, words);
                }
                // ================= second epilogue: new S =================
                {
                    uint32_t mwords[WPW] = {0, 0};
                    if (BWD) load_words(args.bits_s + k * args.bits_stride + bits_row, mwords);
                    uint32_t words[WPW] = {0, 0};
                    stage_bias(2U * k + 1U);
                    if (!warp_wait(&mma_done[1], uses & 1U)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t entry = BWD ? k : k + 1U;
                    __half* tape_row = args.tape_s + entry * args.tape_s_stride + row * args.ld_s;
#pragma unroll
                    for (uint32_t ci = 0; ci < WPW; ++ci) {
                        const uint32_t cc = par + SUBS * ci;
                        if (cc >= NC) break;
                        uint32_t raw[32];
                        tmem_ld_32x32(tmem_base + lane_addr + kStateCol + cc * 32U, raw);
                        tmem_ld_wait();
                        uint32_t h[16];
                        if (BWD) apply_mask(raw, mwords[ci]);
                        else detail::add_bias_relu(raw, bias_slots + 256U + (par * WPW + ci) * 32U);
                        detail::pack_operands(raw, h, args.bf16 != 0U);
                        if (BWD || !last) tmem_st_32x32(tmem_base + lane_addr + kStateCol + cc * 32U, raw);
                        if (!last) {
                            store_operand(cc, h);
                            tmem_st_wait();
                            publish(&ready[p0 + (cc >> 1)]);
                        }
                        if (!BWD) words[ci] = detail::positive_bits(raw);
                        if (row_ok && last) {  // no MMA consumes the last S of a tile, so no panel store either
                            store_tape(tape_row, cc, h);
                            if (!BWD) {
                                float4* dst = reinterpret_cast<float4*>(args.state_f32 + row * args.ld_f32 + col0 + cc * 32U);
#pragma unroll
                                for (int q = 0; q < 8; ++q)
                                    if (col0 + cc * 32U + 4U * q < args.ld_f32) dst[q] = make_float4(__uint_as_float(raw[4 * q]), __uint_as_float(raw[4 * q + 1]), __uint_as_float(raw[4 * q + 2]), __uint_as_float(raw[4 * q + 3]));
                            }
                        }
                    }
                    if (BWD) column_sums(tmem_base + lane_addr + kStateCol, tile, R + k, &sums_done[1]);
                    if (!BWD) store_words(args.bits_s + (k + 1U) * args.bits_stride + bits_row, words);
                    if (last) tc_fence_before();  // the next tile's state load overwrites the TMEM columns read here
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
    pair::cluster_sync_all();  // no CTA leaves while the other may still copy into it
    if (warp == 1) {
        tc_fence_after();
        tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace mgt
