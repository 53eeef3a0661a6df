// The two GEMMs of the embedding layer with a one-hot operand, for pairs of CTAs (sm_100a, tcgen05.cta_group::2).
//
//   forward    D[h][s] = table^T[h][k] * onehot[k][s]      K = L*V table rows + 1 all-ones row (the bias)
//   gradient   D[h][r] = dz1T[h][s] * onehot^T[s][r]       K = samples, r = table rows
//
// The one-hot matrix is synthesised in shared memory from the 80-byte states and never exists in HBM. A pair owns a tile of
// 256 rows (h) x up to 512 columns: each CTA holds its own 128 rows of the A operand, half of the columns of the one-hot
// operand, and its 128 rows of both 256-column accumulators (all of its TMEM). One thread of the pair's first CTA issues
// tcgen05.mma for both.
//
// Why pairs: with one CTA per tile the kernel is bound by shared-memory bandwidth, not by the tensor cores. A K chunk of 64
// is 8 MMAs of 128 x 256 x 16 = 1 024 tensor cycles; it reads 96 KB of operands (768 cycles at 128 bytes a cycle), takes in
// 16 KB by TMA (128) and scatters about a thousand 2-byte stores into the one-hot rows, up to eight to a bank (400): 1 640
// cycles measured. In a pair each SM reads 64 KB, and synthesises half the rows. p888 at 53 248 samples, forward 0.96 ms
// and gradient 0.92 ms with one CTA per tile, 0.72 and 0.73 ms in pairs (the latter with the zeroing of the result): 1.96 and
// 1.92 PFLOP/s executed. What is left beside the MMAs is the epilogue of a piece (6 000 cycles, both accumulators being all of
// tensor memory) and, in the gradient, scattered stores that get in the way of the MMAs' operand reads.
//
// How a pair's work is cut. Forward: the columns of all row tiles form one line and every pair takes an equal stretch of it, in
// steps of 64 columns, and cuts that into equal pieces of at most 512 (no partly filled last round). Gradient: the K chunks of
// all tiles form one line; a stretch is at least as long as a tile, so at most two pairs share one and add into the zeroed
// result in either order with the same bits (0 + a + b = 0 + b + a); shorter lines are cut into whole tiles or halves.
#pragma once

#include <cuda.h>
#include <cuda_fp16.h>

#include "launch.cuh"
#include "ptx_sm100.cuh"

namespace mgt {

struct PairArgs {
    uint32_t M;              // rows of D (hd1)
    uint32_t N;              // columns of D (samples / table rows)
    uint32_t K;              // table rows + 1 / samples
    uint32_t k_chunks;
    uint32_t tile_cols;      // gradient: columns per tile (a multiple of 32, at most 512)
    uint32_t n_tiles;        // gradient: tiles of a row of tiles
    uint32_t workers;        // pairs that have work
    uint64_t line;           // length of the line: forward m_tiles * row_len, gradient tiles * k_chunks
    uint32_t row_len;        // forward: N rounded up to 64
    __half* out_f16;         // forward: relu(D) as [M][ld_f16]
    uint32_t ld_f16;
    uint32_t* bits;          // forward: sign words of D, [M][ld_bits]
    uint32_t ld_bits;
    float* out_f32;          // gradient: [N][ld_f32]
    uint32_t ld_f32;
    const uint8_t* states;   // [samples][80]
    uint32_t state_len, value_pad, samples;
    uint32_t in_rows;        // forward: state_len * value_pad, the all-ones row
    uint32_t bf16;
    int* status;
};

template <bool GRAD>
struct PairCfg {
    static constexpr int STAGES = 4;                  // of both operands together
    static constexpr int A_BYTES = 128 * 128;         // 128 rows x 64 K
    static constexpr int B_ACC_BYTES = 128 * 128;     // this CTA's half of one accumulator's columns x 64 K
    static constexpr int STAGE_BYTES = A_BYTES + 2 * B_ACC_BYTES;
    static constexpr int EPI_WARPS = 8;
    static constexpr int SYNTH_WARPS = 8;             // that fill one stage
    // The gradient's samples change with every chunk: fetching their classes, finding the places and handing the stage over take
    // a warp longer (1 160 cycles) than the chunk's MMAs, so two groups of warps take chunks in turn.
    static constexpr int SYNTH_GROUPS = GRAD ? 2 : 1;
    static constexpr int FIRST_SYNTH_THREAD = 64 + 32 * EPI_WARPS;
    static constexpr int THREADS = FIRST_SYNTH_THREAD + 32 * SYNTH_WARPS * SYNTH_GROUPS;
    // forward: per epilogue warp 32 rows x 32 columns of the result; gradient, few classes: per group two chunks' classes by position
    static constexpr int EXTRA_BYTES = GRAD ? SYNTH_GROUPS * 2 * 80 * 64 : EPI_WARPS * 32 * 64;
    static constexpr int SMEM_BYTES = 1024 + STAGES * STAGE_BYTES + EXTRA_BYTES + 256;
    static_assert(SMEM_BYTES <= 232448, "shared memory budget");
};

namespace pair {

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the same shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to(uint32_t smem_addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
    return r;
}
// Arrival on a barrier of either CTA. What it announces is in this CTA's own shared memory (or tensor memory) and goes to the
// async proxy, so the CTA-scope release that is the default is enough: a cluster-scope release would wait for this thread's
// global accesses too and took microseconds per chunk.
__device__ __forceinline__ void arrive_cluster(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
// A plain (not multicast) TMA load into this CTA's shared memory whose bytes are counted on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const void* map, int32_t x, int32_t y, uint32_t bar_cluster_addr) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(ptx::smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y)
        : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_holder, uint32_t columns) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(ptx::smem_u32(smem_holder)), "r"(columns) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t columns) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(columns) : "memory");
}
// (predicated for a converged warp: see ptx::umma_f16)
__device__ __forceinline__ void umma_f16(uint32_t lead, uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(lead)
        : "memory");
}
// arrives on the barrier at this offset in both CTAs once every MMA issued so far by this thread has completed
__device__ __forceinline__ void umma_commit_both(uint32_t lead, uint64_t* bar) {
    asm volatile(
        "{\n\t.reg .pred q;\n\t"
        "setp.ne.b32 q, %2, 0;\n\t"
        "@q tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n\t}"
        ::"r"(ptx::smem_u32(bar)), "h"(static_cast<uint16_t>(3)), "r"(lead)
        : "memory");
}

// One piece of a pair's stretch: 256 rows from mt * 256, columns [n0, n0 + cols), K chunks [c0, c1).
struct Piece {
    uint32_t mt, n0, cols, c0, c1;
};
// Walks the stretch [x, end) of the line that belongs to pair `worker`.
template <bool GRAD>
struct Pieces {
    const PairArgs& a;
    uint64_t x, end;
    uint32_t row_len;  // forward: columns of a row tile on the line
    __device__ __forceinline__ Pieces(const PairArgs& args, uint32_t worker) : a(args) {
        row_len = GRAD ? args.k_chunks : args.row_len;
        const uint64_t unit = GRAD ? 1U : 64U, units = args.line / unit;
        x = worker < args.workers ? units * worker / args.workers * unit : 0U;
        end = worker < args.workers ? units * (worker + 1U) / args.workers * unit : 0U;
    }
    __device__ __forceinline__ bool next(Piece& p) {
        if (x >= end) return false;
        const uint32_t tile = static_cast<uint32_t>(x / row_len), at = static_cast<uint32_t>(x - static_cast<uint64_t>(tile) * row_len);
        const uint32_t left = static_cast<uint32_t>(min(end - x, static_cast<uint64_t>(row_len - at)));
        if (GRAD) {
            p.mt = tile / a.n_tiles;
            p.n0 = (tile - p.mt * a.n_tiles) * a.tile_cols;
            p.cols = min(a.tile_cols, ((a.N + 31U) & ~31U) - p.n0);
            p.c0 = at;
            p.c1 = at + left;
            x += left;
        } else {
            const uint32_t pieces = (left + 511U) / 512U;
            p.mt = tile;
            p.n0 = at;
            p.cols = min(left, (left / 64U + pieces - 1U) / pieces * 64U);
            p.c0 = 0U;
            p.c1 = a.k_chunks;
            x += p.cols;
        }
        return true;
    }
};

}  // namespace pair

template <bool GRAD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<GRAD>::THREADS, 1)
onehot_pair_kernel(const __grid_constant__ CUtensorMap tma_a, const __grid_constant__ CUtensorMap tma_out, const __grid_constant__ PairArgs args) {
    using namespace ptx;
    constexpr uint32_t ST = PairCfg<GRAD>::STAGES;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw_addr = smem_u32(smem_raw);
    uint8_t* smem = smem_raw + (((raw_addr + 1023U) & ~1023U) - raw_addr);
    uint8_t* extra = smem + ST * PairCfg<GRAD>::STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(extra + PairCfg<GRAD>::EXTRA_BYTES);
    uint64_t* full = bars;               // [ST], used in the first CTA: its own arrival with the byte count of both, 16 synthesis warps
    uint64_t* empty = full + ST;         // [ST] in both: the MMAs that read the stage are done
    uint64_t* acc_full = empty + ST;     // in both
    uint64_t* acc_empty = acc_full + 1;  // in the first CTA: 16 epilogue warps
    uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(acc_empty + 1);
    volatile int* cta_abort = reinterpret_cast<volatile int*>(tmem_holder + 1);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31U;
    const uint32_t rank = pair::cluster_rank(), worker = blockIdx.x >> 1;

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < ST; ++s) {
            mbar_init(&full[s], 1U + 2U * PairCfg<GRAD>::SYNTH_WARPS);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_empty, 2U * PairCfg<GRAD>::EPI_WARPS);
        *cta_abort = 0;
        fence_barrier_init();
        prefetch_tensormap(&tma_a);
        if (!GRAD) prefetch_tensormap(&tma_out);
    }
    {
        // the one-hot ring starts as all zeros; the fast forms only set and clear single halfs afterwards
        uint4* z = reinterpret_cast<uint4*>(smem);
        for (uint32_t i = threadIdx.x; i < ST * PairCfg<GRAD>::STAGE_BYTES / 16; i += PairCfg<GRAD>::THREADS) z[i] = make_uint4(0, 0, 0, 0);
        fence_proxy_async_smem();
    }
    if (warp == 1) pair::tmem_alloc(tmem_holder, 512);
    tc_fence_before();
    __syncthreads();
    pair::cluster_sync_all();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_holder;
    dependent_begin();
    pair::Pieces<GRAD> pieces(args, worker);
    pair::Piece p;

    if (warp == 0) {
        // ------------------------------- TMA producer: this CTA's 128 rows of A -----------
        const uint32_t lead = elect_one();
        uint32_t it = 0;
        bool ok = true;
        while (ok && pieces.next(p)) {
            const int32_t m = static_cast<int32_t>(p.mt * 256U + rank * 128U);
            for (uint32_t c = p.c0; c < p.c1; ++c, ++it) {
                const uint32_t s = it % ST;
                if (!mbar_wait_warp(&empty[s], ((it / ST) & 1U) ^ 1U, cta_abort, kAbortProducerWait)) { ok = false; break; }
                if (!lead) continue;
                uint8_t* dst = smem + s * PairCfg<GRAD>::STAGE_BYTES;
                const uint32_t bar = pair::map_to(smem_u32(&full[s]), 0);
                if (rank == 0U) mbar_arrive_expect_tx(&full[s], 2U * PairCfg<GRAD>::A_BYTES);
                if (GRAD) {
                    pair::tma_load_2d(dst, &tma_a, static_cast<int32_t>(c * 64U), m, bar);
                } else {
                    pair::tma_load_2d(dst, &tma_a, m, static_cast<int32_t>(c * 64U), bar);
                    pair::tma_load_2d(dst + 8192, &tma_a, m + 64, static_cast<int32_t>(c * 64U), bar);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------- MMA issuer: one thread of the pair ---------------
        if (rank == 0U) {
            const uint32_t lead = elect_one();
            uint32_t it = 0, unit = 0;
            bool ok = true;
            while (ok && pieces.next(p)) {
                if (!mbar_wait_warp(acc_empty, (unit & 1U) ^ 1U, cta_abort, kAbortMmaWait)) { ok = false; break; }
                tc_fence_after();
                const uint32_t cols0 = min(256U, p.cols), cols1 = p.cols - cols0;
                const uint32_t idesc0 = make_idesc_f16(256, cols0, !GRAD, false, args.bf16 != 0U);
                const uint32_t idesc1 = make_idesc_f16(256, cols1, !GRAD, false, args.bf16 != 0U);
                for (uint32_t c = p.c0; c < p.c1; ++c, ++it) {
                    const uint32_t s = it % ST;
                    // (one wait and one commit a chunk: with separate rings for A and B, two of each, a chunk took 170 cycles more)
                    if (!mbar_wait_warp(&full[s], (it / ST) & 1U, cta_abort, kAbortMmaWait)) { ok = false; break; }
                    tc_fence_after();
                    const uint32_t a_addr = smem_u32(smem + s * PairCfg<GRAD>::STAGE_BYTES), b_addr = a_addr + PairCfg<GRAD>::A_BYTES;
                    const uint32_t k_left = args.K - c * 64U;
                    const uint32_t ksteps = k_left >= 64U ? 4U : (k_left + 15U) / 16U;
                    // descriptors of the chunk's first K step; a later step only moves the start address
                    constexpr uint64_t kStepA = GRAD ? 32U / 16U : 2048U / 16U, kStepB = 32U / 16U;
                    const uint64_t a_desc = GRAD ? make_smem_desc(a_addr, 16U, 1024U) : make_smem_desc(a_addr, 8192U, 1024U);
                    const uint64_t b_desc0 = make_smem_desc(b_addr, 16U, 1024U), b_desc1 = make_smem_desc(b_addr + PairCfg<GRAD>::B_ACC_BYTES, 16U, 1024U);
                    const uint32_t first = c > p.c0 ? 1U : 0U;
                    if (ksteps == 4U && cols1 != 0U) {
#pragma unroll
                        for (uint32_t kk = 0; kk < 4U; ++kk) pair::umma_f16(lead, tmem_base, a_desc + kk * kStepA, b_desc0 + kk * kStepB, idesc0, kk == 0U ? first : 1U);
#pragma unroll
                        for (uint32_t kk = 0; kk < 4U; ++kk) pair::umma_f16(lead, tmem_base + 256U, a_desc + kk * kStepA, b_desc1 + kk * kStepB, idesc1, kk == 0U ? first : 1U);
                    } else {
                        for (uint32_t kk = 0; kk < ksteps; ++kk) pair::umma_f16(lead, tmem_base, a_desc + kk * kStepA, b_desc0 + kk * kStepB, idesc0, kk == 0U ? first : 1U);
                        if (cols1 != 0U)
                            for (uint32_t kk = 0; kk < ksteps; ++kk) pair::umma_f16(lead, tmem_base + 256U, a_desc + kk * kStepA, b_desc1 + kk * kStepB, idesc1, kk == 0U ? first : 1U);
                    }
                    pair::umma_commit_both(lead, &empty[s]);
                }
                if (ok) pair::umma_commit_both(lead, acc_full);
                ++unit;
            }
        }
        __syncwarp();
    } else if (warp < 2U + PairCfg<GRAD>::EPI_WARPS) {
        // ------------------------------- epilogue: this CTA's 128 rows of D ---------------
        // Eight warps, two per TMEM lane quadrant, each with one half of the columns. Forward: the activation is kept the way D
        // lies ([hd1][samples]); a warp turns 32 rows x 32 columns into the operand format in its own shared-memory tile and a
        // TMA store writes it (a lane storing its row's 64 bytes straight from registers touches 32 lines per instruction: the
        // load/store unit made an epilogue of that 20 000 cycles, a fifth of a piece). The sign words of the 64 columns are one
        // 8-byte store per lane. Gradient: D is the transposed table gradient; the 32 lanes of a warp write consecutive
        // addresses of a table row.
        const uint32_t quad = warp & 3U, half = (warp - 2U) >> 2;
        uint8_t* tile = extra + (warp - 2U) * (32U * 64U);
        const uint32_t empty_addr = pair::map_to(smem_u32(acc_empty), 0);
        uint32_t unit = 0;
        bool ok = true;
        while (ok && pieces.next(p)) {
            if (!__all_sync(0xFFFFFFFFU, mbar_wait(acc_full, unit & 1U, cta_abort, kAbortEpilogueWait))) { ok = false; break; }
            tc_fence_after();
            const uint32_t m = p.mt * 256U + rank * 128U + quad * 32U + lane;
            const bool m_ok = m < args.M;
            const bool shared_tile = GRAD && !(p.c0 == 0U && p.c1 == args.k_chunks);
            if (!GRAD) {
                const uint32_t chunks = p.cols / 64U, mine0 = half * ((chunks + 1U) / 2U), mine1 = half == 0U ? (chunks + 1U) / 2U : chunks;
#pragma unroll 1
                for (uint32_t cc = mine0; cc < mine1; ++cc) {
                    const uint32_t n0 = p.n0 + cc * 64U;
                    uint32_t words[2];
#pragma unroll
                    for (uint32_t hh = 0; hh < 2U; ++hh) {
                        uint32_t r[32];
                        tmem_ld_32x32(tmem_base + ((quad * 32U) << 16) + cc * 64U + hh * 32U, r);
                        tmem_ld_wait();
                        // ReLU, and "is positive" of the fp32 value: with r >= +0, the sign bit of 0 - r as an integer
                        uint32_t word = 0;
#pragma unroll
                        for (int j = 31; j >= 0; --j) {
                            r[j] = __float_as_uint(fmaxf(__uint_as_float(r[j]), 0.0f));
                            word = __funnelshift_l(0U - r[j], word, 1);
                        }
                        const uint32_t at = n0 + hh * 32U;
                        if (lane == 0) bulk_wait_read_all();  // the store of the previous tile has read it
                        __syncwarp();
                        words[hh] = at + 32U <= args.N ? word : (at < args.N ? word & ((1U << (args.N - at)) - 1U) : 0U);
#pragma unroll
                        for (uint32_t q = 0; q < 4U; ++q) {
                            uint4 u;
                            u.x = pack_operand_pair(__uint_as_float(r[8 * q + 0]), __uint_as_float(r[8 * q + 1]), args.bf16 != 0U);
                            u.y = pack_operand_pair(__uint_as_float(r[8 * q + 2]), __uint_as_float(r[8 * q + 3]), args.bf16 != 0U);
                            u.z = pack_operand_pair(__uint_as_float(r[8 * q + 4]), __uint_as_float(r[8 * q + 5]), args.bf16 != 0U);
                            u.w = pack_operand_pair(__uint_as_float(r[8 * q + 6]), __uint_as_float(r[8 * q + 7]), args.bf16 != 0U);
                            *reinterpret_cast<uint4*>(tile + lane * 64U + ((q ^ ((lane >> 1) & 3U)) << 4)) = u;  // 64-byte swizzle
                        }
                        fence_proxy_async_smem();
                        __syncwarp();
                        if (lane == 0) {
                            tma_store_2d(&tma_out, tile, static_cast<int32_t>(at), static_cast<int32_t>(p.mt * 256U + rank * 128U + quad * 32U));
                            bulk_commit_group();
                        }
                    }
                    if (m_ok && n0 < args.N) *reinterpret_cast<uint2*>(args.bits + static_cast<uint64_t>(m) * args.ld_bits + (n0 >> 5)) = make_uint2(words[0], words[1]);
                }
            } else {
                const uint32_t chunks = p.cols / 32U;
#pragma unroll 1
                for (uint32_t cc = half; cc < chunks; cc += 2U) {
                    const uint32_t n0 = p.n0 + cc * 32U;
                    uint32_t r[32];
                    tmem_ld_32x32(tmem_base + ((quad * 32U) << 16) + cc * 32U, r);
                    tmem_ld_wait();
                    const uint32_t valid = n0 < args.N ? min(32U, args.N - n0) : 0U;
                    if (m_ok) {
                        float* dst = args.out_f32 + static_cast<uint64_t>(n0) * args.ld_f32 + m;
#pragma unroll
                        for (int j = 0; j < 32; ++j) {
                            if (static_cast<uint32_t>(j) < valid) {
                                if (shared_tile) atomicAdd(dst, __uint_as_float(r[j])); else *dst = __uint_as_float(r[j]);
                            }
                            dst += args.ld_f32;
                        }
                    }
                    __syncwarp();  // the next load needs the whole warp
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) pair::arrive_cluster(empty_addr);
            ++unit;
        }
        if (!GRAD && lane == 0) bulk_wait_all();  // the stores read this CTA's shared memory
        __syncwarp();
    } else {
        // ------------------------------- one-hot synthesis --------------------------------
        // This CTA's half of the columns of each accumulator: column j of accumulator q belongs to CTA j / (columns / 2). A
        // shared-memory row is one column of the one-hot operand, 64 K values of 2 bytes, 128-byte swizzled. Every place is
        // owned by one warp, so the warps never wait for one another.
        constexpr uint32_t GROUPS = PairCfg<GRAD>::SYNTH_GROUPS;
        const uint32_t group = (threadIdx.x - PairCfg<GRAD>::FIRST_SYNTH_THREAD) >> 8, t = (threadIdx.x - PairCfg<GRAD>::FIRST_SYNTH_THREAD) & 255U;
        const uint32_t V = args.value_pad, L = args.state_len;
        const uint16_t one = operand_one(args.bf16 != 0U);
        auto stage_b = [&](uint32_t it) { return smem + (it % ST) * PairCfg<GRAD>::STAGE_BYTES + PairCfg<GRAD>::A_BYTES; };
        auto acquire = [&](uint32_t it) -> bool {
            return __all_sync(0xFFFFFFFFU, mbar_wait_spin(&empty[it % ST], ((it / ST) & 1U) ^ 1U, cta_abort, kAbortSynthWait));
        };
        auto publish = [&](uint32_t it) {
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) pair::arrive_cluster(pair::map_to(smem_u32(&full[it % ST]), 0));
        };
        auto place = [&](uint32_t row, uint32_t k) -> uint32_t { return row * 128U + ((((k >> 3) ^ (row & 7U)) << 4) | ((k & 7U) << 1)); };
        constexpr uint32_t kNone = 0xFFFFFFFFU;
        // a row of ones at the set bits of a 64-bit mask, written whole: eight 16-byte units
        auto write_row = [&](uint8_t* buf, uint32_t row, uint64_t mask) {
            const uint32_t unit = one;
#pragma unroll
            for (uint32_t q = 0; q < 8U; ++q) {
                const uint32_t b = static_cast<uint32_t>(mask >> (8U * q)) & 0xFFU;
                uint4 u;
                u.x = ((b & 1U) | ((b & 2U) << 15)) * unit;
                u.y = (((b >> 2) & 1U) | ((b & 8U) << 13)) * unit;
                u.z = (((b >> 4) & 1U) | ((b & 32U) << 11)) * unit;
                u.w = (((b >> 6) & 1U) | ((b & 128U) << 9)) * unit;
                *reinterpret_cast<uint4*>(buf + row * 128U + ((q ^ (row & 7U)) << 4)) = u;
            }
        };
        uint32_t it = group;  // the chunks of this group: group, group + GROUPS, ...
        bool ok = true;
        if constexpr (!GRAD) {
            // thread = one column: accumulator t / 128, row t % 128 of this CTA's half
            const uint32_t q = t >> 7, j = t & 127U, row = t;
            if (V >= 64U && (reinterpret_cast<uintptr_t>(args.states) & 3U) == 0U) {  // (the classes are fetched as words)
                // A column's ones sit at k_p = p*V + s[p], increasing in p, and the chunks of a piece are visited in increasing
                // k, so each column keeps a cursor; with V >= 64 a chunk holds at most two of its ones (plus the all-ones row,
                // in the last chunk). The places of the NEXT chunk are worked out while the MMAs of the current ones run;
                // between "stage released" and "stage published" a thread only stores: zeros at the places it remembers from
                // four chunks ago, ones at the new places.
                uint32_t hist[ST][3];
#pragma unroll
                for (uint32_t a = 0; a < ST; ++a)
#pragma unroll
                    for (uint32_t b = 0; b < 3U; ++b) hist[a][b] = kNone;
                uint32_t next[3] = {kNone, kNone, kNone};
                uint32_t pos = 0, cur = 0, ahead = 0;  // classes from position pos on: the rest of a word of four, and the next word
                const uint32_t* st = reinterpret_cast<const uint32_t*>(args.states);
                bool active = false;
                auto start = [&](const pair::Piece& u) {
                    const uint32_t cols = q == 0U ? min(256U, u.cols) : (u.cols > 256U ? u.cols - 256U : 0U);
                    const uint32_t sample = u.n0 + q * 256U + rank * (cols / 2U) + j;
                    active = j < cols / 2U && sample < args.samples;
                    st = reinterpret_cast<const uint32_t*>(args.states + static_cast<uint64_t>(active ? sample : 0U) * 80U);
                    pos = active ? 0U : L;
                    cur = __ldg(st);
                    ahead = __ldg(st + 1);
                };
                auto prepare = [&](uint32_t c) {
                    const uint32_t k0 = c * 64U, kb = args.in_rows - k0;
#pragma unroll
                    for (uint32_t b = 0; b < 2U; ++b) {
                        const uint32_t k = pos * V + (cur & 0xFFU) - k0;  // never below the chunk: earlier chunks consumed those
                        const bool hit = pos < L && k < 64U;
                        next[b] = hit ? place(row, k) : kNone;
                        if (hit) {
                            ++pos;
                            cur >>= 8;
                            if ((pos & 3U) == 0U) {
                                cur = ahead;
                                ahead = __ldg(st + min((pos >> 2) + 1U, 19U));  // (a record is twenty words)
                            }
                        }
                    }
                    next[2] = (kb < 64U && active) ? place(row, kb) : kNone;
                };
                bool have = pieces.next(p);
                uint32_t c = 0;
                if (have) { start(p); prepare(0); }
                while (have) {
                    if (!acquire(it)) break;
                    uint8_t* buf = stage_b(it);
#pragma unroll
                    for (uint32_t b = 0; b < 3U; ++b)
                        if (hist[0][b] != kNone) *reinterpret_cast<uint16_t*>(buf + hist[0][b]) = 0;
#pragma unroll
                    for (uint32_t b = 0; b < 3U; ++b) {
                        if (next[b] != kNone) *reinterpret_cast<uint16_t*>(buf + next[b]) = one;
#pragma unroll
                        for (uint32_t a = 0; a + 1U < ST; ++a) hist[a][b] = hist[a + 1U][b];
                        hist[ST - 1U][b] = next[b];
                    }
                    publish(it);
                    ++it;
                    if (++c >= p.c1) {
                        c = 0;
                        have = pieces.next(p);
                        if (have) start(p);
                    }
                    if (have) prepare(c);
                }
            } else {
                // few classes: many ones per column and chunk, so a thread writes its whole row (right for any number of classes, and
                // for records that do not start at a word)
                while (ok && pieces.next(p)) {
                    const uint32_t cols = q == 0U ? min(256U, p.cols) : (p.cols > 256U ? p.cols - 256U : 0U);
                    const uint32_t sample = p.n0 + q * 256U + rank * (cols / 2U) + j;
                    const bool active = j < cols / 2U && sample < args.samples;
                    const uint8_t* st = args.states + static_cast<uint64_t>(active ? sample : 0U) * 80U;
                    for (uint32_t c = p.c0; c < p.c1; ++c, ++it) {
                        const uint32_t k0 = c * 64U;
                        uint64_t mask = 0;
                        if (active) {
                            const uint32_t hi = min((k0 + 63U) / V, L - 1U);
                            for (uint32_t pp = k0 / V; pp <= hi; ++pp) {
                                const uint32_t k = pp * V + __ldg(st + pp) - k0;
                                if (k < 64U) mask |= 1ULL << k;
                            }
                            const uint32_t kb = args.in_rows - k0;
                            if (kb < 64U) mask |= 1ULL << kb;
                        }
                        if (!acquire(it)) { ok = false; break; }
                        write_row(stage_b(it), row, mask);
                        publish(it);
                    }
                }
            }
        } else {
            const uint32_t max_positions = (args.tile_cols + V - 1U) / V + 1U;
            if (max_positions <= 12U) {
                // thread (sample k = t/4, quarter = t%4) owns up to three of the tile's positions of its sample. Classes are fetched
                // two of the group's chunks ahead and turned into places before the stage is free; what was set in a stage is cleared from
                // registers.
                const uint32_t k = t >> 2, quarter = t & 3U;
                constexpr uint32_t HD = ST / GROUPS;  // stages this group fills
                static_assert(ST % GROUPS == 0, "a group meets the same stages");
                uint32_t hist[HD][3];
#pragma unroll
                for (uint32_t a = 0; a < HD; ++a)
#pragma unroll
                    for (uint32_t b = 0; b < 3U; ++b) hist[a][b] = kNone;
                struct At {
                    pair::Pieces<GRAD> walk;
                    pair::Piece u;
                    uint32_t c;
                    bool have;
                };
                auto begin = [&](At& x) { x.have = x.walk.next(x.u); x.c = x.u.c0; };
                auto advance = [&](At& x, uint32_t steps) {
                    x.c += steps;
                    while (x.have && x.c >= x.u.c1) {
                        const uint32_t over = x.c - x.u.c1;
                        begin(x);
                        x.c += over;
                    }
                };
                auto fetch = [&](const At& x, uint32_t (&cls)[3]) {
                    const uint32_t sample = x.c * 64U + k, p_lo = x.u.n0 / V, p_hi = min((x.u.n0 + x.u.cols - 1U) / V, L - 1U);
                    const bool in = x.have && sample < args.samples;
                    const uint8_t* st = args.states + static_cast<uint64_t>(in ? sample : 0U) * 80U;
#pragma unroll
                    for (uint32_t b = 0; b < 3U; ++b) {
                        const uint32_t pp = p_lo + quarter + 4U * b;
                        cls[b] = (in && pp <= p_hi) ? __ldg(st + pp) : kNone;
                    }
                };
                At now{pieces, p, 0, false}, far{pieces, p, 0, false};
                begin(now);
                begin(far);
                advance(now, group);
                advance(far, group);
                uint32_t cls0[3], cls1[3];
                fetch(far, cls0);
                advance(far, GROUPS);
                fetch(far, cls1);
                advance(far, GROUPS);
                while (now.have) {
                    const uint32_t p_lo = now.u.n0 / V;
                    uint32_t off[3];
#pragma unroll
                    for (uint32_t b = 0; b < 3U; ++b) {
                        const uint32_t n = (p_lo + quarter + 4U * b) * V + cls0[b] - now.u.n0;
                        off[b] = kNone;
                        if (cls0[b] != kNone && n < now.u.cols) {
                            const uint32_t q = n >> 8, cols = q == 0U ? min(256U, now.u.cols) : now.u.cols - 256U, local = (n & 255U) - rank * (cols / 2U);
                            if (local < cols / 2U) off[b] = q * PairCfg<GRAD>::B_ACC_BYTES + place(local, k);
                        }
                        cls0[b] = cls1[b];
                    }
                    fetch(far, cls1);
                    advance(far, GROUPS);
                    advance(now, GROUPS);
                    if (!acquire(it)) break;
                    uint8_t* buf = stage_b(it);
#pragma unroll
                    for (uint32_t b = 0; b < 3U; ++b)
                        if (hist[0][b] != kNone) *reinterpret_cast<uint16_t*>(buf + hist[0][b]) = 0;
                    __syncwarp();  // a place cleared by one lane may be set by another lane of this warp
#pragma unroll
                    for (uint32_t b = 0; b < 3U; ++b) {
                        if (off[b] != kNone) *reinterpret_cast<uint16_t*>(buf + off[b]) = one;
#pragma unroll
                        for (uint32_t a = 0; a + 1U < HD; ++a) hist[a][b] = hist[a + 1U][b];
                        hist[HD - 1U][b] = off[b];
                    }
                    publish(it);
                    it += GROUPS;
                }
            } else {
                // few classes: thread = one table row (p, v); the classes of the chunk's 64 samples at the tile's positions are
                // turned in shared memory, and the row is the comparison of 64 of them with v
                const uint32_t q = t >> 7, j = t & 127U, row = t;
                uint32_t count = 0;
                while (ok && pieces.next(p)) {
                    const uint32_t cols = q == 0U ? min(256U, p.cols) : (p.cols > 256U ? p.cols - 256U : 0U);
                    const uint32_t n = p.n0 + q * 256U + rank * (cols / 2U) + j;
                    const bool active = j < cols / 2U && n < L * V;
                    const uint32_t pp = active ? n / V : 0U, v = active ? n - pp * V : 0xFFU;
                    const uint32_t p_lo = p.n0 / V, p_hi = min((p.n0 + p.cols - 1U) / V, L - 1U), npos = p_hi - p_lo + 1U;
                    for (uint32_t c = p.c0; c < p.c1; ++c, ++count) {
                        if (count % GROUPS != group) continue;
                        uint8_t* cls = extra + (group * 2U + ((it / GROUPS) & 1U)) * (80U * 64U);  // [position][64 samples]
                        for (uint32_t i = t; i < 64U * npos; i += 256U) {
                            const uint32_t k = i / npos, x = i - k * npos, sample = c * 64U + k;
                            cls[x * 64U + k] = sample < args.samples ? __ldg(args.states + static_cast<uint64_t>(sample) * 80U + p_lo + x) : 0xFFU;
                        }
                        named_bar_sync(1U + 2U * group, 32U * PairCfg<GRAD>::SYNTH_WARPS);
                        uint64_t mask = 0;
                        if (active) {
                            const uint32_t* w = reinterpret_cast<const uint32_t*>(cls + (pp - p_lo) * 64U);
#pragma unroll
                            for (uint32_t i = 0; i < 16U; ++i) {
                                const uint32_t eq = __vcmpeq4(w[i], v * 0x01010101U) & 0x08040201U;  // one bit per equal byte
                                mask |= static_cast<uint64_t>((eq | (eq >> 8) | (eq >> 16) | (eq >> 24)) & 0xFU) << (4U * i);
                            }
                        }
                        // (all warps leave together when a wait runs out: the barrier above needs every one of them)
                        if (!named_bar_and(2U + 2U * group, 32U * PairCfg<GRAD>::SYNTH_WARPS, acquire(it))) { ok = false; break; }
                        write_row(stage_b(it), row, mask);
                        publish(it);
                        it += GROUPS;
                    }
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
    pair::cluster_sync_all();  // no CTA leaves while the other may still arrive on its barriers or read its operands
    if (warp == 1) {
        tc_fence_after();
        pair::tmem_dealloc(tmem_base, 512);
    }
}

}  // namespace mgt
