// On-GPU random-walk generator, bit-exact with the reference generator for the same
// (seed, epoch, step, rank, sample): native/cuda/random_walk_kernel.cu:7-64 and
// native/src/random_walk_cpu.cpp:32-66. Integer-only; HBM traffic is 100 bytes per sample.
//
// The moves of a walk must be drawn one after the other (the generator never repeats the previous move, so what a draw means
// depends on the one before), but they need not be applied to the state one after the other: new[i] = old[move[i]] for
// every move makes the final value of position i target[m_1[m_2[... m_d[i] ...]]], a chain of lookups that starts at i and
// never touches the other positions. So a CTA works in two phases: one thread per sample draws the moves of its walk, then
// all threads trace positions, four per thread (one word of the record), eighteen threads per sample. While the moves are
// drawn the other warps compose the 18 x 18 pairs of permutations in shared memory, which halves the length of every trace.
// The states of the generator form a chain of their own whatever the moves are, so the drawing loop takes one state per
// turn and both remainders of it, and decides afterwards what they were for: no lane waits for another's repeated move.
// What bounds it: that chain at small batches, the lookups in shared memory at large ones. Before, one thread carried the
// 72-byte state of a sample through every pair of moves and the repeated-move branch was taken by nearly every warp: 30 us
// at 1 024 samples and 41 us at 53 248 (depths 1..29), now 7 us and 26 us.
// The generator's `rng % bound` on the full 64-bit state is computed exactly with 32-bit multiplies
// (x mod b = ((hi mod b) * (2^32 mod b) + lo mod b) mod b, each step by a multiply-high with ceil(2^32 / b) and one
// correction), which is several times cheaper than a 64-bit remainder.
#include "../../include/mgt_b200.h"
#include "launch.cuh"

#include <cuda_runtime.h>

namespace {

constexpr uint32_t kWalkThreads = 512;
constexpr uint32_t kWalkBlockMoves = 32;  // moves drawn between two trace phases; a longer walk takes several rounds
constexpr uint32_t kStateWords = MGT_STATE_STORAGE_LEN / 4;  // 20 words hold the 72 positions (and the 8 pad bytes)

__host__ __device__ inline uint64_t Mix64(uint64_t x) {
    x += 0x9e3779b97f4a7c15ULL;
    x = (x ^ (x >> 30)) * 0xbf58476d1ce4e5b9ULL;
    x = (x ^ (x >> 27)) * 0x94d049bb133111ebULL;
    return x ^ (x >> 31);
}

struct Bound {
    uint32_t b, magic, r32;  // magic = ceil(2^32 / b), r32 = 2^32 mod b; valid for 2 <= b <= 65535
};
__device__ inline Bound MakeBound(uint32_t b) {
    Bound q{b, 0U, 0U};
    if (b >= 2U && b <= 65535U) {
        q.magic = 0xFFFFFFFFU / b + 1U;
        q.r32 = (0xFFFFFFFFU % b + 1U) % b;
    }
    return q;
}
__device__ inline uint32_t Mod32(uint32_t n, const Bound& q) {
    if (q.magic == 0U) return q.b <= 1U ? 0U : n % q.b;
    uint32_t r = n - __umulhi(n, q.magic) * q.b;  // the quotient estimate is exact or one too large
    return r >= q.b ? r + q.b : r;
}
// x % bound on the full 64 bits
__device__ inline uint32_t Mod64(uint64_t x, const Bound& q) {
    if (q.b <= 1U) return 0U;  // (a bound of 0 is a division by zero in the reference; never reached with valid configurations)
    if (q.magic == 0U) return static_cast<uint32_t>(x % q.b);
    const uint32_t h = Mod32(static_cast<uint32_t>(x >> 32), q), l = Mod32(static_cast<uint32_t>(x), q);
    return Mod32(h * q.r32 + l, q);
}

// The same for the bounds of the drawing loop (at most MGT_MOVE_COUNT), without a branch: a remainder that came out
// negative wraps to a large number and is then larger than itself plus b.
__device__ inline uint32_t SmallMod32(uint32_t n, const Bound& q) {
    const uint32_t r = n - __umulhi(n, q.magic) * q.b;
    return q.b <= 1U ? 0U : min(r, r + q.b);
}
__device__ inline uint32_t SmallMod64(uint64_t x, const Bound& q) {
    const uint32_t h = SmallMod32(static_cast<uint32_t>(x >> 32), q), l = SmallMod32(static_cast<uint32_t>(x), q);
    return SmallMod32(h * q.r32 + l, q);
}

template <uint32_t kWalkSamples>
__global__ void __launch_bounds__(kWalkThreads)
RandomWalkKernel(mgt_random_walk_config_t config, uint64_t base_seed, uint64_t epoch, uint64_t step, uint32_t global_rank,
                 const mgt_train_state_t* __restrict__ moves, const mgt_train_state_t* __restrict__ target,
                 mgt_train_state_t* __restrict__ states, float* __restrict__ labels, mgt_walk_meta_t* __restrict__ meta) {
    __shared__ __align__(4) uint8_t s_moves[MGT_MOVE_COUNT * MGT_STATE_STORAGE_LEN];  // pad positions map to themselves
    // s_pairs[a][b][i] = moves[a][moves[b][i]]: "move a, then move b" as one lookup
    __shared__ __align__(4) uint8_t s_pairs[MGT_MOVE_COUNT * MGT_MOVE_COUNT * MGT_STATE_STORAGE_LEN];
    __shared__ uint32_t s_target[kStateWords];
    __shared__ __align__(4) uint8_t s_seq[kWalkSamples][kWalkBlockMoves];  // the moves of this round, in the order drawn
    __shared__ uint8_t s_count[kWalkSamples];                              // and how many
    __shared__ uint32_t s_state[kWalkSamples][kStateWords];                // only used by walks longer than one round

    const uint32_t tid = threadIdx.x;
    // Word wd of a record: the given bytes for positions below state_len. For a move (`as_move`) a pad position maps to
    // itself, and so does a source position outside the record - a malformed table must not make the lookups below index
    // outside the shared arrays; for a state the pad bytes are zero.
    auto keep_valid = [&](uint32_t given, uint32_t wd, bool as_move) -> uint32_t {
        uint32_t out = 0;
#pragma unroll
        for (uint32_t k = 0; k < 4U; ++k) {
            const uint32_t pos = wd * 4U + k;
            uint32_t byte = (given >> (8U * k)) & 0xFFU;
            if (as_move && byte >= static_cast<uint32_t>(MGT_STATE_STORAGE_LEN)) byte = pos;
            if (pos >= config.state_len) byte = as_move ? pos : 0U;
            out |= byte << (8U * k);
        }
        return out;
    };
    // the records are 80 bytes long and the arrays come from the device allocator: whole words can be read
    constexpr uint32_t kMoveWords = MGT_MOVE_COUNT * kStateWords;
    const bool drawer = tid < kWalkSamples;
    if (!drawer) {
        constexpr uint32_t kHelpers = kWalkThreads - kWalkSamples;
        mgt::dependent_begin();
        for (uint32_t i = tid - kWalkSamples; i < kMoveWords; i += kHelpers) {
            const uint32_t mv = i / kStateWords, wd = i - mv * kStateWords;
            const uint32_t given = mv < config.move_count ? reinterpret_cast<const uint32_t*>(moves[mv].v)[wd] : 0U;
            const uint32_t identity = 0x03020100U + wd * 0x04040404U;  // moves the puzzle does not have: never drawn, kept well-formed
            reinterpret_cast<uint32_t*>(s_moves)[i] = mv < config.move_count ? keep_valid(given, wd, true) : identity;
        }
        if (tid - kWalkSamples < kStateWords) s_target[tid - kWalkSamples] = keep_valid(__ldg(reinterpret_cast<const uint32_t*>(target->v) + (tid - kWalkSamples)), tid - kWalkSamples, false);
        asm volatile("bar.sync 1, %0;" ::"n"(kHelpers) : "memory");
        // compose the pairs: one word (four positions) per item; pairs with a move the puzzle does not have are never read
        for (uint32_t i = tid - kWalkSamples; i < MGT_MOVE_COUNT * kMoveWords; i += kHelpers) {
            const uint32_t wd = i % kStateWords, ab = i / kStateWords;
            const uint32_t a = ab / MGT_MOVE_COUNT, b = ab - a * MGT_MOVE_COUNT;
            if (a >= config.move_count || b >= config.move_count) continue;
            const uint32_t inner = reinterpret_cast<const uint32_t*>(s_moves + b * MGT_STATE_STORAGE_LEN)[wd];
            const uint8_t* outer = s_moves + a * MGT_STATE_STORAGE_LEN;
            uint32_t packed = 0;
#pragma unroll
            for (uint32_t k = 0; k < 4U; ++k) packed |= static_cast<uint32_t>(outer[(inner >> (8U * k)) & 0xFFU]) << (8U * k);
            reinterpret_cast<uint32_t*>(s_pairs)[i] = packed;
        }
    }

    const uint32_t first_sample = blockIdx.x * kWalkSamples;
    const uint32_t sample = first_sample + tid;  // of a drawing thread
    uint64_t rng = 0;
    uint32_t depth = 0, left = 0, last_move = config.move_count;
    Bound all_moves{}, other_moves{};
    if (drawer) {
        rng = base_seed;
        rng ^= Mix64(epoch + 0x100000001b3ULL);
        rng ^= Mix64(step + 0x9e3779b97f4a7c15ULL);
        rng ^= Mix64(static_cast<uint64_t>(global_rank) << 32);
        rng ^= Mix64(sample);
        const Bound span = MakeBound(config.k_max - config.k_min + 1U);
        all_moves = MakeBound(config.move_count);
        other_moves = MakeBound(config.move_count - 1U);
        rng = Mix64(rng);
        depth = sample < config.sample_count ? config.k_min + Mod64(rng, span) : 0U;
        left = depth;
    }
    uint32_t repeated = 0U;  // 1: the last state drew the previous move again, the next one picks among the others
    const uint32_t rounds = (config.k_max - 1U) / kWalkBlockMoves + 1U;  // k_max >= 1, up to the largest of 32 bits
    for (uint32_t round = 0; round < rounds; ++round) {
        if (drawer) {
            const uint32_t now = min(left, kWalkBlockMoves);
            left -= now;
            // native/cuda/random_walk_kernel.cu:40-47: a draw equal to the previous move is replaced by one of the others,
            // picked by the generator's next state
            // Software pipeline: while turn n decides what its state was for, the remainders of state n + 1 and the state
            // n + 2 are on their way, so a turn takes about as long as one step of the state chain.
            uint64_t cur = Mix64(rng), ahead = Mix64(cur);
            uint32_t plain = SmallMod64(cur, all_moves), other = SmallMod64(cur, other_moves);
            for (uint32_t done = 0; done < now;) {
                const uint64_t ahead2 = Mix64(ahead);
                const uint32_t plain1 = SmallMod64(ahead, all_moves), other1 = SmallMod64(ahead, other_moves);
                const bool emit = repeated != 0U || plain != last_move;
                const uint32_t replaced = last_move + 1U + other;  // below 2 * move_count
                last_move = repeated != 0U ? (replaced >= config.move_count ? replaced - config.move_count : replaced) : plain;  // (when nothing is emitted plain is last_move)
                repeated = emit ? 0U : 1U;
                s_seq[tid][done] = static_cast<uint8_t>(last_move);  // (overwritten by the next turn when this one emits nothing)
                done += emit ? 1U : 0U;
                rng = cur;
                cur = ahead; ahead = ahead2; plain = plain1; other = other1;
            }
            s_count[tid] = static_cast<uint8_t>(now);
            // (the moves of the first round are drawn while the kernel ahead still runs: they are a matter of the arguments alone)
            if (round == 0U) mgt::dependent_begin();
        }
        __syncthreads();
        const bool final_round = round + 1U == rounds;
        constexpr uint32_t kItems = kWalkSamples * kStateWords, kPerThread = (kItems + kWalkThreads - 1U) / kWalkThreads;
        uint32_t result[kPerThread];
#pragma unroll
        for (uint32_t r = 0; r < kPerThread; ++r) {
            const uint32_t item = tid + r * kWalkThreads;
            const uint32_t ls = item / kStateWords, wd = item - ls * kStateWords;
            uint32_t packed = 0;
            result[r] = 0U;
            if (item >= kItems || first_sample + ls >= config.sample_count) continue;
            if (wd * 4U < config.state_len) {
                const uint32_t count = s_count[ls];
                uint32_t pos[4];
                const uint32_t odd = (count & 1U) ? s_seq[ls][count - 1U] * MGT_STATE_STORAGE_LEN : 0U;
#pragma unroll
                for (uint32_t k = 0; k < 4U; ++k) {
                    pos[k] = wd * 4U + k;
                    if (count & 1U) pos[k] = s_moves[odd + pos[k]];
                }
                for (uint32_t j = count / 2U; j > 0U; --j) {
                    const uint32_t both = reinterpret_cast<const uint16_t*>(s_seq[ls])[j - 1U];
                    const uint8_t* pair = s_pairs + ((both & 0xFFU) * MGT_MOVE_COUNT + (both >> 8)) * MGT_STATE_STORAGE_LEN;
#pragma unroll
                    for (uint32_t k = 0; k < 4U; ++k) pos[k] = pair[pos[k]];
                }
                const uint8_t* old = reinterpret_cast<const uint8_t*>(round == 0U ? s_target : s_state[ls]);
#pragma unroll
                for (uint32_t k = 0; k < 4U; ++k) {
                    const bool pad = wd * 4U + k >= config.state_len;  // the pad bytes of a record are zero
                    packed |= (pad ? 0U : static_cast<uint32_t>(old[pos[k]])) << (8U * k);
                }
            }
            if (final_round) reinterpret_cast<uint32_t*>(states + first_sample + ls)[wd] = packed;
            result[r] = packed;
        }
        if (!final_round) {
            __syncthreads();  // every trace of this round has read the old states
#pragma unroll
            for (uint32_t r = 0; r < kPerThread; ++r) {
                const uint32_t item = tid + r * kWalkThreads;
                if (item < kItems) s_state[item / kStateWords][item % kStateWords] = result[r];
            }
        }
    }
    if (drawer && sample < config.sample_count) {
        labels[sample] = static_cast<float>(depth);
        mgt_walk_meta_t m;
        m.depth = depth;
        m.last_move = last_move;
        m.rng_counter = rng;
        meta[sample] = m;
    }
}

__global__ void ExpandScalarLabelsKernel(const float* __restrict__ scalar_labels, uint32_t samples, uint32_t output_dim, float* __restrict__ labels) {
    const uint64_t item = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    const uint64_t total = static_cast<uint64_t>(samples) * output_dim;
    mgt::dependent_begin();
    if (item >= total) return;
    labels[item] = scalar_labels[item / output_dim];
}

}  // namespace

extern "C" {

mgt_status_t mgt_validate_random_walk_config(const mgt_random_walk_config_t* c) {
    if (c == nullptr) return MGT_INVALID_CONFIG;
    if (c->sample_count == 0 || c->k_min == 0 || c->k_min > c->k_max || c->move_count == 0 || c->move_count > MGT_MOVE_COUNT ||
        c->state_len == 0 || c->state_len > MGT_STATE_LEN || c->state_storage_len < c->state_len ||
        c->state_storage_len > MGT_STATE_STORAGE_LEN) {
        return MGT_INVALID_CONFIG;
    }
    return MGT_OK;
}

mgt_status_t mgt_launch_random_walk(const mgt_random_walk_config_t* config, uint64_t base_seed, uint64_t epoch, uint64_t step,
                                    uint32_t global_rank, const mgt_train_state_t* device_moves,
                                    const mgt_train_state_t* device_target, mgt_train_state_t* device_states,
                                    float* device_labels, mgt_walk_meta_t* device_meta, void* stream) {
    if (mgt_validate_random_walk_config(config) != MGT_OK || device_moves == nullptr || device_target == nullptr ||
        device_states == nullptr || device_labels == nullptr || device_meta == nullptr) {
        return MGT_INVALID_CONFIG;
    }
    // the kernel reads moves and target as words and writes a state record as words (16 bytes is what the other kernels want)
    if ((reinterpret_cast<uintptr_t>(device_moves) & 3U) != 0 || (reinterpret_cast<uintptr_t>(device_target) & 3U) != 0 ||
        (reinterpret_cast<uintptr_t>(device_states) & 15U) != 0 || (reinterpret_cast<uintptr_t>(device_labels) & 3U) != 0 ||
        (reinterpret_cast<uintptr_t>(device_meta) & 7U) != 0) {
        return MGT_INVALID_CONFIG;
    }
    // Up to 32 samples for each of 148 SMs a CTA takes 32: one word of positions per thread, the shortest path. Beyond that
    // 128 per CTA, so that the pair table is composed a quarter as often (three CTAs share an SM).
    const mgt::LaunchOn st(static_cast<cudaStream_t>(stream), true);
    if (config->sample_count <= 148U * 32U) {
        mgt::Launch(RandomWalkKernel<32>, (config->sample_count + 31U) / 32U, kWalkThreads, 0, st, *config, base_seed, epoch, step, global_rank, device_moves, device_target, device_states, device_labels, device_meta);
    } else {
        mgt::Launch(RandomWalkKernel<128>, (config->sample_count + 127U) / 128U, kWalkThreads, 0, st, *config, base_seed, epoch, step, global_rank, device_moves, device_target, device_states, device_labels, device_meta);
    }
    return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
}

mgt_status_t mgt_launch_expand_scalar_labels(const float* device_scalar_labels, uint32_t samples, uint32_t output_dim,
                                             float* device_labels, void* stream) {
    if (device_scalar_labels == nullptr || device_labels == nullptr || samples == 0 || output_dim == 0) return MGT_INVALID_CONFIG;
    const uint64_t total = static_cast<uint64_t>(samples) * output_dim;
    const uint32_t blocks = static_cast<uint32_t>((total + 255ULL) / 256ULL);
    mgt::Launch(ExpandScalarLabelsKernel, blocks, 256, 0, {static_cast<cudaStream_t>(stream), true}, device_scalar_labels, samples, output_dim, device_labels);
    return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
}

}  // extern "C"
