// Loss + gradient engine: forward, MSE loss and backward of the residual MLP on tcgen05 tensor
// cores, behind the C ABI of include/mgt_b200.h. Follows the data flow of the reference's fp16
// path (native/cuda/mlp_backward.cu:1228-1510): fp16 operands rounded at the same tensors, fp32
// accumulation, fp32 master biases for the hidden/residual layers, fp16 mirror for the embedding
// table and its bias. What differs is how it is computed:
//   * the embedding layer and its gradient are one-hot GEMMs whose one-hot operand is synthesised
//     in shared memory from the 80-byte states (never materialised in HBM), or sums of gathered rows
//     where the batch is small for the GEMMs;
//   * bias, ReLU, residual add, ReLU-mask and the fp16 down-cast are epilogues of the GEMMs;
//   * bias gradients are fp32 column sums taken in the epilogue that produces each dz tensor
//     (the reference sums the fp32 dz, not its fp16 copy: tiny gradients that underflow in fp16
//     still reach the bias), reduced over CTAs in a fixed order;
//   * activations are kept once (fp16 tape + one in-place fp32 residual stream).
#include "../../include/mgt_b200.h"
#include "batch_norm.cuh"
#include "embedding_gather.cuh"
#include "fp32_path.cuh"
#include "fp32_tower.cuh"
#include "onehot_pair.cuh"
#include "tower_chain.cuh"
#include "tower_wide.cuh"
#include "umma_gemm.cuh"

#include <cuda.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace mgt {
namespace {

// ---- flat parameter layout (native/cuda/mlp_backward.cu:25-36) -----------------------------
inline uint64_t BlockParams(const mgt_mlp_shape_t& s) { return 2ULL * ((uint64_t)s.hd2 * s.hd2 + s.hd2); }
inline uint64_t InputBias(const mgt_mlp_shape_t& s) { return (uint64_t)s.state_len * s.state_value_pad * s.hd1; }
inline uint64_t HiddenWeight(const mgt_mlp_shape_t& s) { return InputBias(s) + s.hd1; }
inline uint64_t HiddenBias(const mgt_mlp_shape_t& s) { return HiddenWeight(s) + (uint64_t)s.hd1 * s.hd2; }
inline uint64_t ResidualBase(const mgt_mlp_shape_t& s) { return HiddenBias(s) + s.hd2; }
inline uint64_t OutputWeight(const mgt_mlp_shape_t& s) { return ResidualBase(s) + (uint64_t)s.residual_blocks * BlockParams(s); }
inline uint64_t OutputBias(const mgt_mlp_shape_t& s) { return OutputWeight(s) + (uint64_t)s.hd2 * s.output_dim; }
inline uint64_t ParamCount(const mgt_mlp_shape_t& s) { return OutputBias(s) + s.output_dim; }
inline uint64_t Fc1W(const mgt_mlp_shape_t& s, uint32_t b) { return ResidualBase(s) + (uint64_t)b * BlockParams(s); }
inline uint64_t Fc1B(const mgt_mlp_shape_t& s, uint32_t b) { return Fc1W(s, b) + (uint64_t)s.hd2 * s.hd2; }
inline uint64_t Fc2W(const mgt_mlp_shape_t& s, uint32_t b) { return Fc1B(s, b) + s.hd2; }
inline uint64_t Fc2B(const mgt_mlp_shape_t& s, uint32_t b) { return Fc2W(s, b) + (uint64_t)s.hd2 * s.hd2; }

inline uint64_t RoundUp(uint64_t v, uint64_t a) { return (v + a - 1) / a * a; }

bool ValidShape(const mgt_mlp_shape_t* s) {
    return s != nullptr && s->state_len > 0 && s->state_len <= MGT_STATE_LEN && s->state_value_pad > 0 &&
           s->state_value_pad <= MGT_STATE_VALUE_PAD && s->hd1 > 0 && s->hd1 <= MGT_MAX_HD1 && s->hd2 > 0 &&
           s->hd2 <= MGT_MAX_HD2 && s->residual_blocks <= MGT_MAX_RESIDUAL_BLOCKS && s->output_dim > 0;
}

// ---- workspace ------------------------------------------------------------------------------
// All offsets are in bytes from a 1024-byte aligned base inside the caller's float arena.
struct Workspace {
    uint32_t B, H1, H2, R, OUT, IN;
    uint32_t p_bt;    // pitch (halfs) of the tensors kept with one row per hd1 column (a1, dz1): samples rounded to 8
    uint64_t off_rowsum, rowsum_rows;  // partial row sums of the hidden layer's dX GEMM (input-bias gradient)
    uint64_t off_bits_h1;              // sign words of the embedding layer's pre-activation: [hd1][ld_bits_h1]
    uint32_t ld_bits_h1;
    uint32_t p_act;   // pitch (halfs) of x_h / r1_h, rounded to 8
    uint32_t p_dz;    // pitch (halfs) of dz tensors over H2
    uint32_t p_f32;   // pitch (floats) of the fp32 residual / gradient streams
    uint32_t p_w1, p_w2, p_wout;  // pitches of the internal fp16 weight copy
    uint64_t off_a1, off_x, off_r1, off_xf, off_dzf, off_dz2, off_dz1t, off_dz1, off_partial, off_partial_fc2, off_partial_fc1, off_partial_out, off_head, off_wint, off_dy, off_dyh, off_colsum;
    uint64_t colsum_floats, colsum_slot_floats, dz_stride;
    uint64_t off_bits, bits_stride;  // ReLU sign bits of the residual tower: 2R+1 entries of bits_stride words
    uint64_t x_stride, r1_stride;  // bytes between consecutive blocks' tensors
    uint64_t head_blocks;
    // batch normalisation (only planned when it is on): fp32 pre-activations of the R+1 normalised layers, their saved
    // mean / rstd, partial sums of the reductions, the statistics vector when the caller gives no exchange buffer
    // the embedding layer by gathering rows instead of one-hot GEMMs (sample lists of the table gradient, dz1 as rows of samples)
    bool gather_fwd, gather_grad;
    uint32_t p_dz1_rows;
    uint64_t off_lists;
    uint64_t off_bn_z, bn_z_stride, off_bn_save, off_bn_partial, off_bn_bias, off_bn_stats;
    uint64_t total_bytes;
};

constexpr uint32_t kHeadBlocks = 296;   // two CTAs per SM on a 148-SM part
constexpr uint32_t kHeadThreads = 256;
// per CTA: { grad W_out, grad b_out, loss, column sums of dz } with one output, { loss, column sums of dz, grad b_out } with more
inline uint64_t HeadPartialFloats(const mgt_mlp_shape_t& s) { return s.output_dim == 1U ? 2ULL * s.hd2 + 2ULL : (uint64_t)s.hd2 + 1ULL + s.output_dim; }

// The scratch for per-CTA partial sums is sized by the SM count: never below the B200's 148, so that the size the
// query reports (it has no engine, it asks the current device) covers the launch on any sm_100 part.
inline uint32_t PlanSmCount(int device_sms) { return device_sms > 148 ? static_cast<uint32_t>(device_sms) : 148U; }
inline uint32_t CurrentDeviceSmCount() {
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) {
        cudaGetLastError();
        return 148U;
    }
    return PlanSmCount(sms);
}

// ---- the embedding layer: one-hot GEMMs for CTA pairs (onehot_pair.cuh) or gathered rows (embedding_gather.cuh) -------------
// How the pairs cut their work, and an estimate of what it takes in microseconds (fitted to a B200, within a fifth or so).
struct PairPlan {
    uint32_t workers, tile_cols, n_tiles, row_len;
    uint64_t line;
    bool shared_tiles;  // gradient: two pairs add into some tiles, the result has to be zeroed before
    double us;
};
// Forward: every pair an equal number of 64-column steps of the line; below four full pieces per pair the pieces of a row tile
// instead (a stretch across a row tile's end is one piece more).
PairPlan PlanPairForward(const mgt_mlp_shape_t& s, uint32_t B, uint32_t sm) {
    PairPlan p{};
    const uint32_t m_tiles = (s.hd1 + 255U) / 256U, pairs = sm / 2U, k_chunks = (s.state_len * s.state_value_pad + 64U) / 64U;
    const bool by_tile = m_tiles <= pairs && B <= 2048U * (pairs / m_tiles);
    p.row_len = (B + 63U) / 64U * 64U;
    p.line = (uint64_t)m_tiles * p.row_len;
    p.workers = (uint32_t)std::min<uint64_t>(by_tile ? m_tiles * (pairs / m_tiles) : pairs, p.line / 64U);
    const double cols = (double)p.line / p.workers, pieces = std::ceil(cols / 512.0) + (by_tile ? 0.0 : 0.5);
    p.us = 12.0 + pieces * (k_chunks * std::max(700.0, 2.0 * cols / pieces + 25.0) + 6000.0) / 1845.0;
    return p;
}
// Gradient: tiles of up to 512 columns - the more columns, the fewer times A is read; with few classes the synthesis is what
// takes the time, so narrower ones as long as there are pairs for them. Stretches of at least a tile for every pair; with fewer
// tiles than pairs whole tiles, or halves where they all fit.
PairPlan PlanPairGrad(const mgt_mlp_shape_t& s, uint32_t B, uint32_t sm) {
    PairPlan p{};
    const uint32_t m_tiles = (s.hd1 + 255U) / 256U, pairs = sm / 2U, k_chunks = (B + 63U) / 64U, rows = s.state_len * s.state_value_pad;
    p.n_tiles = (rows + 511U) / 512U;
    if (s.state_value_pad < 64U) p.n_tiles = std::max(p.n_tiles, std::min((rows + 63U) / 64U, pairs / 2U / m_tiles));
    p.tile_cols = ((rows + p.n_tiles - 1U) / p.n_tiles + 31U) & ~31U;
    p.n_tiles = (rows + p.tile_cols - 1U) / p.tile_cols;
    const uint32_t tiles = m_tiles * p.n_tiles;
    p.workers = tiles >= pairs ? pairs : (2U * tiles <= pairs && k_chunks >= 2U ? 2U * tiles : tiles);
    p.line = (uint64_t)tiles * k_chunks;
    p.shared_tiles = tiles % p.workers != 0U;
    const double share = (double)tiles / p.workers;
    p.us = 12.0 + (share * k_chunks * std::max(1100.0, 2.0 * p.tile_cols + 230.0) + (share > 1.0 ? share + 1.0 : 1.0) * 27000.0) / 1845.0 +
           (p.shared_tiles ? 3.0 + (double)rows * s.hd1 * 4.0 / 6.0e6 : 0.0);
    return p;
}
// Gathering adds about 8 (forward) or 6.7 (gradient) values a picosecond, after a few us of start-up and, in the backward
// direction, the sort of the samples.
struct EmbeddingForms { bool gather_fwd, gather_grad; };
EmbeddingForms PickEmbeddingForms(const mgt_mlp_shape_t& s, uint32_t B, uint32_t sm) {
    const double sums = (double)B * s.state_len * s.hd1;
    return {4.0 + sums / 8.0e6 < PlanPairForward(s, B, sm).us, 8.0 + B * 0.0019 + sums / 6.7e6 < PlanPairGrad(s, B, sm).us};
}

// Columns of a product's tile: 224 serves the p888 residual width without padded MMA columns.
inline uint32_t PickBN(uint32_t n) { return n <= 224 ? 224U : 256U; }
// K splits of a weight gradient: at most one wave of [128 x 256] tiles.
inline uint32_t MostSplits(uint32_t M, uint32_t N, uint32_t groups, uint32_t sm_count) {
    const uint64_t tiles = (uint64_t)((M + 127U) / 128U) * ((N + PickBN(N) - 1U) / PickBN(N)) * groups;
    return tiles >= sm_count ? 1U : (uint32_t)(sm_count / tiles);
}

// No term may fall with a larger batch: a caller sizes its scratch for the largest batch and runs smaller ones in it. So what a
// form of the embedding layer needs is planned whichever form this batch takes (288 bytes a sample of 72 positions). half_ig: the
// table gradient is the 16-bit one (the fp32 one keeps its lists behind this workspace).
Workspace PlanWorkspace(const mgt_mlp_shape_t& s, uint32_t B, uint32_t sm_count, bool half_ig, bool batch_norm = false) {
    Workspace w{};
    w.B = B; w.H1 = s.hd1; w.H2 = s.hd2; w.R = s.residual_blocks; w.OUT = s.output_dim;
    w.IN = s.state_len * s.state_value_pad;
    w.p_act = (uint32_t)RoundUp(s.hd2, 8);
    w.p_dz = (uint32_t)RoundUp(s.hd2, 8);
    w.p_bt = (uint32_t)RoundUp(B, 8);
    w.p_f32 = (uint32_t)RoundUp(s.hd2, 4);
    w.p_w1 = (uint32_t)RoundUp(s.hd1, 8);
    w.p_w2 = (uint32_t)RoundUp(s.hd2, 8);
    w.p_wout = (uint32_t)RoundUp(s.output_dim, 8);
    uint64_t off = 0;
    auto take = [&](uint64_t bytes) { const uint64_t o = off; off = RoundUp(off + bytes, 1024); return o; };
    // a1 and dz1 lie as [hd1][samples]: the way the two embedding GEMMs produce and consume them
    const uint64_t hidden_act_bytes = (uint64_t)s.hd1 * w.p_bt * 2;
    w.off_a1 = take(hidden_act_bytes);
    w.x_stride = RoundUp((uint64_t)B * w.p_act * 2, 1024);
    w.off_x = take(w.x_stride * (w.R + 1));
    w.r1_stride = w.x_stride;
    w.off_r1 = take(w.r1_stride * (w.R > 0 ? w.R : 1));
    w.off_xf = take((uint64_t)B * w.p_f32 * 4);
    w.off_dzf = take((uint64_t)B * w.p_f32 * 4);
    // gradients w.r.t. pre-activations, kept for the whole backward pass so that the weight gradients of all
    // residual blocks can be computed by two grouped GEMMs at the end: tape[0] belongs to the hidden layer,
    // tape[k+1] to fc2 of block k; dz1t[k] to fc1 of block k
    w.dz_stride = RoundUp((uint64_t)B * w.p_dz * 2, 1024);
    w.off_dz2 = take(w.dz_stride * (w.R + 1));
    w.off_dz1t = take(w.dz_stride * (w.R > 0 ? w.R : 1));
    const EmbeddingForms forms = PickEmbeddingForms(s, B, sm_count);
    w.gather_fwd = forms.gather_fwd;
    w.gather_grad = forms.gather_grad;
    w.p_dz1_rows = (uint32_t)RoundUp(s.hd1, 8);
    w.off_dz1 = take(std::max<uint64_t>(hidden_act_bytes, half_ig ? (uint64_t)B * w.p_dz1_rows * 2 : 0));
    w.off_lists = take(half_ig ? gather::ListWords(B, s.state_len, s.state_value_pad) * 4 : 0);
    // split-K partials, of every product until the sums of the step are launched
    const uint32_t r = w.R > 0 ? w.R : 1;
    w.off_partial = take((uint64_t)MostSplits(s.hd1, s.hd2, 1, sm_count) * s.hd1 * s.hd2 * 4);
    w.off_partial_fc2 = take((uint64_t)MostSplits(s.hd2, s.hd2, r, sm_count) * r * s.hd2 * s.hd2 * 4);
    w.off_partial_fc1 = take((uint64_t)MostSplits(s.hd2, s.hd2, r, sm_count) * r * s.hd2 * s.hd2 * 4);
    w.off_partial_out = take(s.output_dim > 1 ? (uint64_t)MostSplits(s.hd2, s.output_dim, 1, sm_count) * s.hd2 * s.output_dim * 4 : 0);
    w.head_blocks = kHeadBlocks;
    w.off_head = take((uint64_t)kHeadBlocks * HeadPartialFloats(s) * 4);
    // per-warp column sums: one slot per residual dX GEMM (2R of them)
    const uint64_t chain_tiles = (B + 127) / 128;
    const uint64_t slot_rows = (uint64_t)sm_count * 16 > chain_tiles * 4 ? (uint64_t)sm_count * 16 : chain_tiles * 4;  // up to 16 epilogue warps per CTA
    w.colsum_slot_floats = slot_rows * s.hd2;
    w.colsum_floats = w.colsum_slot_floats * 2 * (w.R > 0 ? w.R : 1);
    w.off_colsum = take(w.colsum_floats * 4);
    w.rowsum_rows = 2ULL * ((B + 255) / 256);  // two epilogue warps per lane quadrant, one N tile per 256 samples
    w.off_rowsum = take(w.rowsum_rows * s.hd1 * 4);
    w.ld_bits_h1 = (uint32_t)RoundUp((B + 31) / 32, 8);  // (32-byte rows)
    w.off_bits_h1 = take((uint64_t)s.hd1 * w.ld_bits_h1 * 4);
    w.bits_stride = chain_tiles * 128 * (s.hd2 > 256U ? 16 : 8);  // words: one per 32 of 256 columns, twice that in the wide tower
    w.off_bits = take(w.bits_stride * 4 * (2 * w.R + 1));
    // internal fp16 weight copy (used when the caller's mirror cannot be addressed by TMA as it lies)
    const uint64_t wint_halfs = (uint64_t)(w.IN + 1) * w.p_w1 + (uint64_t)s.hd1 * w.p_w2 + 2ULL * w.R * s.hd2 * w.p_w2 + (uint64_t)s.hd2 * w.p_wout;
    w.off_wint = take(wint_halfs * 2 + 1024ULL * (2 * w.R + 4));
    w.off_dy = take((uint64_t)B * s.output_dim * 4);
    w.off_dyh = take((uint64_t)B * w.p_wout * 2);
    if (batch_norm) {
        w.bn_z_stride = RoundUp((uint64_t)B * w.p_f32 * 4, 1024);
        w.off_bn_z = take(w.bn_z_stride * (w.R + 1));
        w.off_bn_save = take((uint64_t)(w.R + 1) * 2 * s.hd2 * 4);
        w.off_bn_partial = take((uint64_t)bn::kMaxBlocks * 2 * s.hd2 * 4);
        w.off_bn_bias = take((uint64_t)(w.R + 1) * bn::kMaxBlocks * s.hd2 * 4);
        w.off_bn_stats = take(2ULL * s.hd2 * 4);
    }
    w.total_bytes = off + 1024;  // slack to align the caller's base
    return w;
}

// ---- engine -----------------------------------------------------------------------------------
using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

struct MapKey {
    const void* base;
    uint64_t inner, outer, pitch;
    uint32_t box_inner, box_outer;
    CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B;
    uint64_t layers = 0, layer_stride = 0;  // 3-D maps only
    bool operator==(const MapKey& o) const {
        return base == o.base && inner == o.inner && outer == o.outer && pitch == o.pitch && box_inner == o.box_inner && box_outer == o.box_outer && swizzle == o.swizzle &&
               layers == o.layers && layer_stride == o.layer_stride;
    }
};
struct MapKeyHash {
    size_t operator()(const MapKey& k) const {
        uint64_t h = reinterpret_cast<uint64_t>(k.base);
        auto mix = [&](uint64_t v) { h ^= v + 0x9e3779b97f4a7c15ULL + (h << 6) + (h >> 2); };
        mix(k.inner); mix(k.outer); mix(k.pitch); mix(k.box_inner); mix(k.box_outer); mix(k.swizzle); mix(k.layers); mix(k.layer_stride);
        return (size_t)h;
    }
};

}  // namespace
}  // namespace mgt

namespace mgt {
// A second stream and the events that tie it to the caller's. Taken by an engine's first pass on a stream that wants one and given
// back when the engine goes: the pool keeps kPooled idle ones per device (a program that makes engines one after the other would
// pay 0.1 ms each for new ones). A stream that a capture still holds is neither handed out nor destroyed.
struct SideStream {
    cudaStream_t stream = nullptr;
    cudaEvent_t events[3] = {nullptr, nullptr, nullptr};
};
// 0: the stream is not being captured, ~0: it cannot be told or the capture is invalid, else the id of the capture
inline unsigned long long CaptureOf(cudaStream_t stream) {
    cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
    unsigned long long id = 0;
    if (cudaStreamGetCaptureInfo(stream, &status, &id) != cudaSuccess) {
        cudaGetLastError();
        return ~0ULL;
    }
    if (status == cudaStreamCaptureStatusNone) return 0;
    return status == cudaStreamCaptureStatusActive ? id + 1U : ~0ULL;
}
class SidePool {
    static constexpr size_t kPooled = 4;
    std::mutex mu;
    std::vector<SideStream> idle[64];

public:
    static SidePool& Get() {
        static SidePool* pool = new SidePool();  // (never destroyed: the CUDA runtime may be gone before it)
        return *pool;
    }
    // make = false: only an idle one (nothing is created while a stream is being captured)
    bool Take(int device, bool make, SideStream* out) {
        if (device < 0 || device >= 64) return false;
        {
            std::lock_guard<std::mutex> lock(mu);
            for (size_t i = idle[device].size(); i-- > 0;) {
                if (CaptureOf(idle[device][i].stream) != 0) continue;
                *out = idle[device][i];
                idle[device].erase(idle[device].begin() + static_cast<ptrdiff_t>(i));
                return true;
            }
        }
        if (!make) return false;
        // (ahead of the caller's stream where both have blocks to place: the embedding gradient then ends the pass with the whole
        // chip; 3 001 samples of p888 550 -> 523 us a step)
        SideStream s;
        int least = 0, greatest = 0;
        bool ok = cudaDeviceGetStreamPriorityRange(&least, &greatest) == cudaSuccess && cudaStreamCreateWithPriority(&s.stream, cudaStreamNonBlocking, greatest) == cudaSuccess;
        for (cudaEvent_t& ev : s.events) ok = ok && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess;
        if (!ok) {
            Destroy(s);
            return false;
        }
        *out = s;
        return true;
    }
    void GiveBack(int device, const SideStream& s) {
        if (s.stream == nullptr) return;
        {
            std::lock_guard<std::mutex> lock(mu);
            if (idle[device].size() < kPooled || CaptureOf(s.stream) != 0) {
                idle[device].push_back(s);
                return;
            }
        }
        Destroy(s);
    }

private:
    static void Destroy(const SideStream& s) {
        for (cudaEvent_t ev : s.events)
            if (ev) cudaEventDestroy(ev);
        if (s.stream) cudaStreamDestroy(s.stream);
    }
};
}  // namespace mgt

struct mgt_engine {
    int device = 0;
    int sm_count = 148;
    int* status_word = nullptr;  // device
    mgt::EncodeTiledFn encode = nullptr;
    std::unordered_map<mgt::MapKey, CUtensorMap, mgt::MapKeyHash> maps;
    std::mutex mu;
    cudaEvent_t ev_last = nullptr, ev_now = nullptr;
    // second streams for the weight gradients of small batches (SideBranch), one for each of the streams this engine was called on
    struct SideOf {
        cudaStream_t main;
        mgt::SideStream side;
    };
    std::vector<SideOf> sides;
    size_t side_turn = 0;
    std::mutex side_mu;    // of the two above; and an event is recorded and waited for in one piece
    uint64_t launches = 0;  // kernels launched through this engine (host-side count)
    uint64_t forks = 0;     // passes of which a part ran on a second stream
    bool layered_tower = false;  // MGT_RESIDUAL_PATH=layered: per-layer GEMMs instead of the fused residual-tower kernels (both are tested)
    enum { kBySize, kGather, kOneHot } embedding_form = kBySize;  // MGT_EMBEDDING_FORM=gather|onehot: one form of the embedding layer for all sizes (both are tested)
    mgt_gradient_ready_fn early_fn = nullptr;  // mgt_engine_set_early_range_hook
    void* early_user = nullptr;
    mgt_train_options_t options{MGT_OPERAND_FP16, MGT_LOSS_MSE, 0, 1.0e-5f};  // mgt_engine_set_train_options
    // mgt_engine_set_batch_norm_state
    float* bn_running = nullptr;
    float bn_momentum = 0.1f;
    uint32_t bn_world = 1;
    float* bn_exchange_buffer = nullptr;
    mgt_stats_exchange_fn bn_exchange = nullptr;
    void* bn_exchange_user = nullptr;
    bool bf16_now = false;  // operand format of the launch being enqueued (set by mgt_launch_mlp_loss_grad, off otherwise)

    // fp16 3-D tensor map (a stack of `layers` equal matrices `layer_stride_bytes` apart), 128-byte swizzle, box depth 1
    bool Map3D(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t layers, uint64_t pitch_elems, uint64_t layer_stride_bytes,
               uint32_t box_inner, uint32_t box_outer) {
        mgt::MapKey key{base, inner, outer, pitch_elems, box_inner, box_outer};
        key.layers = layers;
        key.layer_stride = layer_stride_bytes;
        std::lock_guard<std::mutex> lock(mu);
        auto it = maps.find(key);
        if (it != maps.end()) { *out = it->second; return true; }
        if ((reinterpret_cast<uintptr_t>(base) & 15U) != 0 || ((pitch_elems * 2) & 15U) != 0 || (layer_stride_bytes & 15U) != 0 || box_inner * 2 > 128 || box_outer > 256) return false;
        const cuuint64_t dims[3] = {inner, outer, layers};
        const cuuint64_t strides[2] = {pitch_elems * 2, layer_stride_bytes};
        const cuuint32_t box[3] = {box_inner, box_outer, 1};
        const cuuint32_t elem[3] = {1, 1, 1};
        CUtensorMap m;
        const CUresult r = encode(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box, elem,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return false;
        if (maps.size() > 4096) maps.clear();
        maps.emplace(key, m);
        *out = m;
        return true;
    }

    // fp16 2-D tensor map: `inner` contiguous elements per row, `outer` rows; the swizzle spans a box row (128 bytes, or 64 with
    // a box of 32 elements).
    bool Map(CUtensorMap* out, const void* base, uint64_t inner, uint64_t outer, uint64_t pitch_elems, uint32_t box_inner, uint32_t box_outer,
             CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
        const mgt::MapKey key{base, inner, outer, pitch_elems, box_inner, box_outer, swizzle};
        std::lock_guard<std::mutex> lock(mu);
        auto it = maps.find(key);
        if (it != maps.end()) { *out = it->second; return true; }
        if ((reinterpret_cast<uintptr_t>(base) & 15U) != 0 || ((pitch_elems * 2) & 15U) != 0 || box_inner * 2 > 128 || box_outer > 256) return false;
        const cuuint64_t dims[2] = {inner, outer};
        const cuuint64_t strides[1] = {pitch_elems * 2};
        const cuuint32_t box[2] = {box_inner, box_outer};
        const cuuint32_t elem[2] = {1, 1};
        CUtensorMap m;
        const CUresult r = encode(&m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<void*>(base), dims, strides, box, elem,
                                  CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
        if (r != CUDA_SUCCESS) return false;
        if (maps.size() > 4096) maps.clear();
        maps.emplace(key, m);
        *out = m;
        return true;
    }
};

namespace mgt {
namespace {

template <class Cfg>
mgt_status_t LaunchGemm(mgt_engine* e, const CUtensorMap& ta, const CUtensorMap& tb, GemmArgs args, LaunchOn stream, const CUtensorMap* to = nullptr) {
    // the opt-in shared-memory size is a per-device attribute of each kernel instantiation
    static std::mutex attr_mu;
    static bool attr_done[64] = {};
    if (e->device < 0 || e->device >= 64) return MGT_INVALID_CONFIG;
    {
        std::lock_guard<std::mutex> lock(attr_mu);
        if (!attr_done[e->device]) {
            if (cudaFuncSetAttribute(umma_gemm_kernel<Cfg>, cudaFuncAttributeMaxDynamicSharedMemorySize, Cfg::SMEM_BYTES) != cudaSuccess) return MGT_CUDA_FAILURE;
            attr_done[e->device] = true;
        }
    }
    const uint64_t units = (uint64_t)args.m_tiles * args.n_tiles * args.splits * (Cfg::GROUPED ? args.groups : 1U);
    if (units == 0) return MGT_INVALID_CONFIG;
    uint32_t grid = (uint32_t)(units < (uint64_t)e->sm_count ? units : (uint64_t)e->sm_count);
    if (Cfg::BSTAT) {
        // every unit of a CTA must share the N tile: unit = mt * n_tiles + nt advances by the grid size
        if (args.splits != 1 || args.k_chunks > (uint32_t)Cfg::SB || args.n_tiles > (uint32_t)e->sm_count) return MGT_INVALID_CONFIG;
        if (grid >= args.n_tiles) grid = grid / args.n_tiles * args.n_tiles;
    }
    args.status = e->status_word;
    args.bf16 = e->bf16_now ? 1U : 0U;
    Launch(umma_gemm_kernel<Cfg>, grid, Cfg::THREADS, Cfg::SMEM_BYTES, stream, ta, tb, to != nullptr ? *to : ta, args);
    ++e->launches;
    return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
}

template <bool GRAD>
mgt_status_t LaunchPair(mgt_engine* e, const CUtensorMap& ta, const CUtensorMap& to, PairArgs args, LaunchOn stream) {
    static std::mutex attr_mu;
    static bool attr_done[64] = {};
    if (e->device < 0 || e->device >= 64) return MGT_INVALID_CONFIG;
    {
        std::lock_guard<std::mutex> lock(attr_mu);
        if (!attr_done[e->device]) {
            if (cudaFuncSetAttribute(onehot_pair_kernel<GRAD>, cudaFuncAttributeMaxDynamicSharedMemorySize, PairCfg<GRAD>::SMEM_BYTES) != cudaSuccess) return MGT_CUDA_FAILURE;
            attr_done[e->device] = true;
        }
    }
    args.status = e->status_word;
    args.bf16 = e->bf16_now ? 1U : 0U;
    Launch(onehot_pair_kernel<GRAD>, 2U * args.workers, PairCfg<GRAD>::THREADS, PairCfg<GRAD>::SMEM_BYTES, stream, ta, to, args);
    ++e->launches;
    return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
}

// Tile configurations.
template <int BN, Epi EPI> using CfgFwd = GemmCfg<BN, false, BSource::kTmaMN, EPI, 3, 3>;   // act[K-major] x W[K][N]
template <int BN, Epi EPI> using CfgDx = GemmCfg<BN, false, BSource::kTmaK, EPI, 3, 3>;     // dz[K-major] x W[N][K]
// B-stationary forms for reductions of at most 256 (the residual width): weights stay in shared memory
template <int BN, Epi EPI> using CfgFwdS = GemmCfg<BN, false, BSource::kTmaMN, EPI, 3, 4, true>;
template <int BN, Epi EPI> using CfgDxS = GemmCfg<BN, false, BSource::kTmaK, EPI, 3, 4, true>;
template <int BN> using CfgDw = GemmCfg<BN, true, BSource::kTmaMN, Epi::kPartialF32, 3, 3>; // act^T x dz
// The hidden layer with its wide side (hd1) as rows: a1 and dz1 are kept as [hd1][samples], the way the two embedding GEMMs
// produce and consume them, so that their epilogues and the hidden dX epilogue move 64 contiguous bytes per lane
template <int BN, Epi EPI> using CfgFwdRows = GemmCfg<BN, true, BSource::kTmaMN, EPI, 3, 3>;        // a1T[K][M] x W[K][N]
template <int BN> using CfgDwRows = GemmCfg<BN, false, BSource::kTmaMN, Epi::kPartialF32, 3, 3>;    // a1T[M][K] x dz[K][N]
using CfgDxRows = GemmCfg<256, false, BSource::kTmaK, Epi::kMaskRowsumF16, 4, 4>;                   // W[M][K] x dz[N][K] -> dz1T[M][N]
using CfgDxRowsTma = GemmCfg<256, false, BSource::kTmaK, Epi::kMaskRowsumF16Tma, 4, 4>;             // ... by TMA stores
using CfgDxRowsF32 = GemmCfg<256, false, BSource::kTmaK, Epi::kMaskRowsumF32, 4, 4>;                // the same -> dz1[N][M] in fp32
using CfgDxRowsF16T = GemmCfg<256, false, BSource::kTmaK, Epi::kMaskRowsumF16T, 4, 4>;               // the same -> dz1[N][M]
template <int BN> using CfgDwG = GemmCfg<BN, true, BSource::kTmaMN, Epi::kPartialF32, 3, 3, false, true>; // R stacked act^T x dz
using CfgDbgKK = GemmCfg<256, false, BSource::kTmaK, Epi::kPartialF32, 3, 3>;
using CfgDbgKM = GemmCfg<256, false, BSource::kTmaMN, Epi::kPartialF32, 3, 3>;
using CfgDbgMK = GemmCfg<256, true, BSource::kTmaK, Epi::kPartialF32, 3, 3>;

GemmArgs BaseArgs(uint32_t M, uint32_t N, uint32_t K, uint32_t bn_total, uint32_t splits) {
    GemmArgs a{};
    a.M = M; a.N = N; a.K = K;
    a.m_tiles = (M + 127) / 128;
    a.n_tiles = (N + bn_total - 1) / bn_total;
    a.k_chunks = (K + 63) / 64;
    a.groups = 1;
    a.splits = splits < 1 ? 1 : (splits > a.k_chunks ? a.k_chunks : splits);
    return a;
}

// ---- small kernels ------------------------------------------------------------------------------

// The weight matrices as fp16 or bfloat16 with padded rows, all of them in one launch: matrix i is fp32 [rows][cols] at
// src + src_off[i] and goes to [rows][8 * units[i]] halfs at dst + dst_off[i] (bytes), the padding as zeros. A thread writes
// one 16-byte unit of eight columns; unit_begin[i] is the running number of the matrix's first unit. A copy through HBM (6
// bytes a parameter); as one memset and one scalar kernel per matrix the 67 matrices of a 40 M parameter model took 490 us, this
// kernel 43 us.
struct RepackPlan {
    static constexpr int kMax = 2 * MGT_MAX_RESIDUAL_BLOCKS + 3;
    uint64_t src_off[kMax], dst_off[kMax], unit_begin[kMax + 1];
    uint32_t cols[kMax], units[kMax];
    uint32_t count;
};
__global__ void __launch_bounds__(256)
RepackHalfKernel(const float* __restrict__ src, uint8_t* __restrict__ dst, const __grid_constant__ RepackPlan plan, bool bf16) {
    dependent_begin();
    const uint64_t total = plan.unit_begin[plan.count];
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    uint32_t i = 0;
    for (uint64_t u = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; u < total; u += stride) {
        while (u >= plan.unit_begin[i + 1]) ++i;
        const uint64_t local = u - plan.unit_begin[i];
        const uint32_t cols = plan.cols[i], units = plan.units[i];
        const uint64_t row = local / units;
        const uint32_t c0 = (uint32_t)(local - row * units) * 8U;
        const float* p = src + plan.src_off[i] + row * cols + c0;
        float v[8];
        if (c0 + 8U <= cols && (reinterpret_cast<uintptr_t>(p) & 15U) == 0U) {
            const float4 x = __ldg(reinterpret_cast<const float4*>(p)), y = __ldg(reinterpret_cast<const float4*>(p) + 1);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w; v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
        } else {
#pragma unroll
            for (uint32_t j = 0; j < 8U; ++j) v[j] = c0 + j < cols ? __ldg(p + j) : 0.0f;
        }
        *reinterpret_cast<uint4*>(dst + plan.dst_off[i] + local * 16U) =
            make_uint4(ptx::pack_operand_pair(v[0], v[1], bf16), ptx::pack_operand_pair(v[2], v[3], bf16), ptx::pack_operand_pair(v[4], v[5], bf16),
                       ptx::pack_operand_pair(v[6], v[7], bf16));
    }
}

// Sums over partial results, each in a fixed order: out[group][i] = sum over terms t of src[group][t * stride + i]. The sums of a
// step that nothing in the step waits for - split-K planes, bias sums of the tiles, what the head's CTAs leave - are collected and
// go in one launch: as six of 2 to 14 us each, with a gap before it, they were a seventh of the smallest steps (us a step with six, with
// one, and with one since launches overlap too: 64 samples of hd1 8, hd2 8 85, 73, 56; 1 024 of hd1 256, hd2 64, 2 blocks 118, 103, 82;
// p888 at 53 248 3 059, 3 051, where they do not overlap).
// Few items with many terms (kLanes): eight items a CTA, each of 32 lanes adds terms g, g + 32, ... and the lanes are then
// added 0..31. Many items with few terms: an item (kItem) or four neighbouring ones (kQuad) a thread, terms in order.
struct SumJob {
    enum Form : uint32_t { kLanes, kItem, kQuad };
    const float* src;
    float* dst;
    uint64_t src_group, dst_group, stride;  // floats from one group, one term to the next
    uint64_t items;
    uint32_t terms, per_group, first_cta;
    Form form;
};
struct SumJobs {
    static constexpr int kMax = 12;
    SumJob job[kMax];
    uint32_t count, ctas;
};
constexpr uint32_t kReduceCols = 8;
template <class T>
__device__ __forceinline__ T SumTerms(const float* src, uint64_t stride, uint32_t terms, uint64_t i) {
    auto at = [&](uint32_t t) { return __ldg(reinterpret_cast<const T*>(src + t * stride) + i); };
    auto add = [](float4& x, const float4& y) { x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w; };
    auto add1 = [](float& x, float y) { x += y; };
    T sum = at(0);
    uint32_t t = 1;
    for (; t + 8U <= terms; t += 8U) {  // eight loads in flight
        T x[8];
#pragma unroll
        for (uint32_t q = 0; q < 8U; ++q) x[q] = at(t + q);
#pragma unroll
        for (uint32_t q = 0; q < 8U; ++q) {
            if constexpr (sizeof(T) == 16) add(sum, x[q]); else add1(sum, x[q]);
        }
    }
    for (; t < terms; ++t) {
        const T x = at(t);
        if constexpr (sizeof(T) == 16) add(sum, x); else add1(sum, x);
    }
    return sum;
}
__global__ void __launch_bounds__(256)
SumKernel(const __grid_constant__ SumJobs jobs) {
    __shared__ float s_part[32][kReduceCols + 1];
    uint32_t at = 0;
    while (at + 1U < jobs.count && blockIdx.x >= jobs.job[at + 1U].first_cta) ++at;
    const SumJob& job = jobs.job[at];
    dependent_begin();
    const uint32_t local = blockIdx.x - job.first_cta, group = local / job.per_group, cta = local - group * job.per_group;
    const float* src = job.src + group * job.src_group;
    float* dst = job.dst + group * job.dst_group;
    if (job.form == SumJob::kLanes) {
        const uint32_t cl = threadIdx.x & (kReduceCols - 1U), g = threadIdx.x / kReduceCols, c = cta * kReduceCols + cl;
        float sum = 0.0f;
        if (c < job.items) {
            const float* p = src + c;
            uint32_t r = g;
            for (; r + 96U < job.terms; r += 128U) {
                const float a0 = p[r * job.stride], a1 = p[(r + 32U) * job.stride], a2 = p[(r + 64U) * job.stride], a3 = p[(r + 96U) * job.stride];
                sum += a0; sum += a1; sum += a2; sum += a3;
            }
            for (; r < job.terms; r += 32U) sum += p[r * job.stride];
        }
        s_part[g][cl] = sum;
        __syncthreads();
        if (g == 0 && c < job.items) {
            float total = s_part[0][cl];
#pragma unroll
            for (int q = 1; q < 32; ++q) total += s_part[q][cl];
            dst[c] = total;
        }
        return;
    }
    const uint64_t i = cta * 256ULL + threadIdx.x;
    if (job.form == SumJob::kQuad) {
        if (i < job.items / 4U) reinterpret_cast<float4*>(dst)[i] = SumTerms<float4>(src, job.stride, job.terms, i);
    } else if (i < job.items) {
        dst[i] = SumTerms<float>(src, job.stride, job.terms, i);
    }
}

// Output head for output_dim == 1 (native/cuda/mlp_backward.cu:891-931): y = b + <x, w> with fp32
// master weights, diff, dy = 2 diff / B, loss term diff^2 / B, dcur = w * dy, then the ReLU mask of
// the last block. One warp per sample (grid-stride); per-CTA partial sums go to
// partials[CTA][2*H2+2] = { grad W_out[H2], grad b_out, loss, column sums of dz[H2] } and are added
// in a fixed order.
constexpr int kHeadMaxPerLane = MGT_MAX_HD2 / 32;
__global__ void __launch_bounds__(kHeadThreads)
HeadOut1Kernel(const float* __restrict__ w_out, const float* __restrict__ b_out, const float* __restrict__ labels, const float* __restrict__ x,
               uint32_t p_f32, uint32_t B, uint32_t H2, float* __restrict__ dzf, __half* __restrict__ dz_h, uint32_t p_dz, float* __restrict__ partials,
               bool bf16) {
    __shared__ float s_acc[kHeadThreads / 32][2 * MGT_MAX_HD2 + 2];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31U;
    const uint32_t warps_total = gridDim.x * (kHeadThreads / 32);
    const float inv_n = 1.0f / static_cast<float>(B);
    dependent_begin();
    w_out = after_begin(w_out);
    const float bias = *after_begin(b_out);
    float wreg[kHeadMaxPerLane], gacc[kHeadMaxPerLane], dacc[kHeadMaxPerLane];
#pragma unroll
    for (int q = 0; q < kHeadMaxPerLane; ++q) {
        const uint32_t j = q * 32 + lane;
        wreg[q] = j < H2 ? w_out[j] : 0.0f;
        gacc[q] = 0.0f;
        dacc[q] = 0.0f;
    }
    float gb = 0.0f, loss = 0.0f;
    // The row and the label of the warp's next sample are fetched before the current one is worked on: one sample is a
    // chain of load -> five shuffles -> stores, and a warp that waits for each load in turn leaves HBM idle.
    float xn[kHeadMaxPerLane], label_next = 0.0f;
    auto fetch = [&](uint32_t b) {
        const float* row = x + (uint64_t)b * p_f32;
#pragma unroll
        for (int q = 0; q < kHeadMaxPerLane; ++q) {
            const uint32_t j = q * 32 + lane;
            xn[q] = (b < B && j < H2) ? row[j] : 0.0f;
        }
        label_next = b < B ? labels[b] : 0.0f;
    };
    fetch(blockIdx.x * (kHeadThreads / 32) + warp);
    for (uint32_t b = blockIdx.x * (kHeadThreads / 32) + warp; b < B; b += warps_total) {
        float xv[kHeadMaxPerLane];
        const float label = label_next;
        float dot = 0.0f;
#pragma unroll
        for (int q = 0; q < kHeadMaxPerLane; ++q) {
            xv[q] = xn[q];
            dot += xv[q] * wreg[q];
        }
        fetch(b + warps_total);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) dot += __shfl_xor_sync(0xFFFFFFFFU, dot, o);
        const float diff = (bias + dot) - label;
        const float dy = 2.0f * diff * inv_n;
        if (lane == 0) { gb += dy; loss += diff * diff * inv_n; }
#pragma unroll
        for (int q = 0; q < kHeadMaxPerLane; ++q) {
            const uint32_t j = q * 32 + lane;
            if (j < H2) {
                gacc[q] += xv[q] * dy;
                const float d = xv[q] > 0.0f ? wreg[q] * dy : 0.0f;
                dacc[q] += d;
                dzf[(uint64_t)b * p_f32 + j] = d;
                if (dz_h != nullptr) reinterpret_cast<uint16_t*>(dz_h)[(uint64_t)b * p_dz + j] = ptx::to_operand(d, bf16);
            }
        }
    }
#pragma unroll
    for (int q = 0; q < kHeadMaxPerLane; ++q) {
        const uint32_t j = q * 32 + lane;
        if (j < H2) { s_acc[warp][j] = gacc[q]; s_acc[warp][H2 + 2 + j] = dacc[q]; }
    }
    if (lane == 0) { s_acc[warp][H2] = gb; s_acc[warp][H2 + 1] = loss; }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < 2 * H2 + 2; j += kHeadThreads) {
        float sum = 0.0f;
        for (int wi = 0; wi < kHeadThreads / 32; ++wi) sum += s_acc[wi][j];
        partials[(uint64_t)blockIdx.x * (2 * H2 + 2) + j] = sum;
    }
}

// ---- output head for output_dim > 1 (native/cuda/mlp_backward.cu:1341-1363) -------------------------------------------
// 16-bit operands, fp32 accumulate, dy rounded to the operand format for the two products that follow; kF32: fp32 operands
// throughout. kCrossEntropy = false: the reference's MSE against the labels. kCrossEntropy = true (no counterpart in the
// reference): the outputs are per-depth logits, class = depth - 1 (the labels carry the walk depth in every output slot),
// loss = mean over the batch of -log softmax(y)[class], dy = (softmax(y) - onehot(class)) / B.
// Both kernels leave one row of partial sums per CTA: { loss, column sums of dz[H2], column sums of dy[OUT] }.
struct HeadArgs {
    const void* w_out;       // [H2][p_wout] operand format, or fp32
    uint32_t p_wout;
    const float* b_out;
    const float* labels;
    const __half* x_h;       // operand copy of x (unused with kF32)
    uint32_t p_act;
    const float* x_f32;
    uint32_t p_f32;
    uint32_t B, H2, OUT;
    float* dy;
    __half* dy_h;            // (unused with kF32)
    uint32_t p_dy;
    float* dzf;
    __half* dz_h;            // (unused with kF32)
    uint32_t p_dz;
    float* partials;
    bool bf16;
};

// dL/dy of one sample, a lane per output (and every 32nd): y and dy in `row` (the logits come in, the operand of the two
// products goes out), the plain dy to memory. Adds the sample's loss term to `loss` and its dy to `dyb`, if kept there.
template <bool kCrossEntropy, bool kF32, int kKept>
__device__ __forceinline__ void HeadLossRow(const HeadArgs& a, uint32_t b, float inv_n, float* row, uint32_t lane, float& loss, float (&dyb)[kKept]) {
    float mx = -3.0e38f, log_sum = 0.0f;
    uint32_t cls = 0;
    if (kCrossEntropy) {
        for (uint32_t o = lane; o < a.OUT; o += 32) mx = fmaxf(mx, row[o]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFU, mx, o));
        float sum = 0.0f;
        for (uint32_t o = lane; o < a.OUT; o += 32) sum += expf(row[o] - mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xFFFFFFFFU, sum, o);
        log_sum = logf(sum) + mx;
        // a depth outside 1..OUT cannot come from the walk generator with k_max <= OUT; clamp instead of reading out of bounds
        const int c = __float2int_rn(a.labels[(uint64_t)b * a.OUT]) - 1;
        cls = static_cast<uint32_t>(c < 0 ? 0 : (c >= static_cast<int>(a.OUT) ? static_cast<int>(a.OUT) - 1 : c));
    }
#pragma unroll 1
    for (uint32_t o = lane, i = 0; o < a.OUT; o += 32, ++i) {
        const float y = row[o];
        float d;
        if (kCrossEntropy) {
            d = (expf(y - log_sum) - (o == cls ? 1.0f : 0.0f)) * inv_n;
            if (o == cls) loss += (log_sum - y) * inv_n;
        } else {
            const float diff = y - a.labels[(uint64_t)b * a.OUT + o];
            d = 2.0f * diff * inv_n;
            loss += diff * diff * inv_n;
        }
        a.dy[(uint64_t)b * a.OUT + o] = d;
        if (kF32) {
            row[o] = d;
        } else {
            const uint16_t dh = ptx::to_operand(d, a.bf16);
            reinterpret_cast<uint16_t*>(a.dy_h)[(uint64_t)b * a.p_dy + o] = dh;
            row[o] = ptx::from_operand(dh, a.bf16);
        }
#pragma unroll
        for (int q = 0; q < kKept; ++q) dyb[q] += static_cast<int>(i) == q ? d : 0.0f;
    }
}

// Up to 64 outputs: a CTA takes 64 samples at a time. Forward as a small register-tiled product (a thread: four samples x
// OP / 16 outputs) from x staged 64 columns at a time and the weights staged once; the loss by a warp per sample; backward
// with a thread per hidden column, its OP weights in registers, so that dy is read as broadcast vectors and rows of dz are
// written whole. Bound by the multiply-adds of both products on the CUDA cores and the shared-memory reads that feed them: 0.68 ms at
// batch 131 072, hd2 512, 29 outputs, where the 0.8 GB it moves (x in the operand format and in fp32 for the ReLU mask, dz in
// both) take 0.13. One warp per sample with a scalar read of x and of a weight for every multiply-add took 1.83 ms.
constexpr uint32_t kHeadTile = 64;
template <int OP>
constexpr size_t HeadTileSmem(uint32_t H2) { return ((size_t)H2 * OP + 64U * (kHeadTile + 4U) + kHeadTile * OP) * sizeof(float); }
template <int OP, bool kCrossEntropy, bool kF32>
__global__ void __launch_bounds__(kHeadThreads)
HeadTileKernel(const __grid_constant__ HeadArgs a) {
    extern __shared__ __align__(16) float s_head[];
    constexpr uint32_t NO = OP / 16, XP = kHeadTile + 4U;
    float* ws = s_head;                                // [H2][OP]
    float* xs = ws + (size_t)a.H2 * OP;                // [64 columns][XP]: x of the tile, transposed
    float* ys = xs + 64U * XP;                         // [64 samples][OP]
    const uint32_t t = threadIdx.x, warp = t >> 5, lane = t & 31U;
    dependent_begin();
    for (uint32_t i = t; i < a.H2 * OP; i += kHeadThreads) {
        const uint32_t j = i / OP, o = i % OP;
        float w = 0.0f;
        if (o < a.OUT) w = kF32 ? static_cast<const float*>(a.w_out)[(uint64_t)j * a.p_wout + o] : ptx::from_operand(static_cast<const uint16_t*>(a.w_out)[(uint64_t)j * a.p_wout + o], a.bf16);
        ws[i] = w;
    }
    const float inv_n = 1.0f / static_cast<float>(kCrossEntropy ? (uint64_t)a.B : (uint64_t)a.B * a.OUT);
    float loss = 0.0f, dyb[2] = {0.0f, 0.0f};
    const uint32_t hj = min(kHeadThreads, (a.H2 + 31U) & ~31U), groups = kHeadThreads / hj, jg = t / hj, jl = t % hj;
    float dacc[2] = {0.0f, 0.0f};
    const uint32_t tiles = (a.B + kHeadTile - 1U) / kHeadTile;
    for (uint32_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        const uint32_t b0 = tile * kHeadTile;
        float acc[4][NO] = {};
        const uint32_t og = t % 16U, sg = t / 16U;
        for (uint32_t j0 = 0; j0 < a.H2; j0 += 64U) {
            // a thread stages sixteen columns of one sample; consecutive lanes take consecutive samples
            const uint32_t s = t % kHeadTile, jb = (t / kHeadTile) * 16U;
            __syncthreads();
#pragma unroll
            for (uint32_t q = 0; q < 2U; ++q) {
                const uint32_t j = j0 + jb + q * 8U;
                float v[8];
#pragma unroll
                for (int e = 0; e < 8; ++e) v[e] = 0.0f;
                if (b0 + s < a.B && j < a.H2) {
                    if (kF32) {
#pragma unroll
                        for (uint32_t e = 0; e < 8U; ++e)
                            if (j + e < a.H2) v[e] = __ldg(a.x_f32 + (uint64_t)(b0 + s) * a.p_f32 + j + e);
                    } else {
                        // (rows are padded to eight elements; what lies past H2 meets nothing: the product stops at H2)
                        const uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(a.x_h) + (uint64_t)(b0 + s) * a.p_act + j);
                        const uint32_t w4[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            v[2 * e] = ptx::from_operand(static_cast<uint16_t>(w4[e] & 0xFFFFU), a.bf16);
                            v[2 * e + 1] = ptx::from_operand(static_cast<uint16_t>(w4[e] >> 16), a.bf16);
                        }
                    }
                }
#pragma unroll
                for (uint32_t e = 0; e < 8U; ++e) xs[(jb + q * 8U + e) * XP + s] = v[e];
            }
            __syncthreads();
            const uint32_t jn = min(64U, a.H2 - j0);
#pragma unroll 8
            for (uint32_t j = 0; j < jn; ++j) {
                const float4 x4 = *reinterpret_cast<const float4*>(xs + j * XP + sg * 4U);
                const float* w = ws + (size_t)(j0 + j) * OP + og * NO;
#pragma unroll
                for (uint32_t n = 0; n < NO; ++n) {
                    acc[0][n] += x4.x * w[n];
                    acc[1][n] += x4.y * w[n];
                    acc[2][n] += x4.z * w[n];
                    acc[3][n] += x4.w * w[n];
                }
            }
        }
#pragma unroll
        for (uint32_t n = 0; n < NO; ++n) {
            const uint32_t o = og * NO + n;
            const float bias = o < a.OUT ? __ldg(a.b_out + o) : 0.0f;
#pragma unroll
            for (uint32_t i = 0; i < 4U; ++i) ys[(sg * 4U + i) * OP + o] = acc[i][n] + bias;
        }
        __syncthreads();
        for (uint32_t i = 0; i < kHeadTile / (kHeadThreads / 32U); ++i) {
            const uint32_t s = warp * (kHeadTile / (kHeadThreads / 32U)) + i;
            if (b0 + s >= a.B) break;
            HeadLossRow<kCrossEntropy, kF32, 2>(a, b0 + s, inv_n, ys + s * OP, lane, loss, dyb);
        }
        __syncthreads();
        if (jg < groups) {
            for (uint32_t cb = 0; cb < 2U; ++cb) {
                const uint32_t j = jl + cb * kHeadThreads;
                if (j >= a.H2) break;
                float w[OP];
#pragma unroll
                for (int o = 0; o < OP; o += 4) {
                    const float4 w4 = *reinterpret_cast<const float4*>(ws + (size_t)j * OP + o);
                    w[o] = w4.x; w[o + 1] = w4.y; w[o + 2] = w4.z; w[o + 3] = w4.w;
                }
                const uint32_t rows = min(kHeadTile, a.B - b0);
                float sum = 0.0f;
#pragma unroll 4
                for (uint32_t s = jg; s < rows; s += groups) {
                    const uint64_t b = b0 + s;
                    const float x = __ldg(a.x_f32 + b * a.p_f32 + j);
                    float d = 0.0f;
#pragma unroll
                    for (int o = 0; o < OP; o += 4) {
                        const float4 g = *reinterpret_cast<const float4*>(ys + s * OP + o);
                        d += g.x * w[o];
                        d += g.y * w[o + 1];
                        d += g.z * w[o + 2];
                        d += g.w * w[o + 3];
                    }
                    d = x > 0.0f ? d : 0.0f;
                    sum += d;
                    a.dzf[b * a.p_f32 + j] = d;
                    if (!kF32) reinterpret_cast<uint16_t*>(a.dz_h)[b * a.p_dz + j] = ptx::to_operand(d, a.bf16);
                }
                dacc[cb] += sum;
            }
        }
        // (outputs past OUT: their weights are zero, and ys holds acc + bias = 0 there)
    }
    __syncthreads();
    // partial sums of the CTA, in a fixed order: warps for the loss and dy, sample groups for the columns
    float* red = xs;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFU, loss, o);
    if (lane == 0) red[warp] = loss;
    red[8U + warp * 64U + lane] = dyb[0];
    red[8U + warp * 64U + 32U + lane] = dyb[1];
    float* cols = red + 8U + 8U * 64U;  // [groups][H2], groups * H2 <= 512
    if (jg < groups) {
        if (jl < a.H2) cols[jg * a.H2 + jl] = dacc[0];
        if (jl + kHeadThreads < a.H2) cols[jl + kHeadThreads] = dacc[1];
    }
    __syncthreads();
    float* out = a.partials + (uint64_t)blockIdx.x * (1U + a.H2 + a.OUT);
    for (uint32_t i = t; i < 1U + a.H2 + a.OUT; i += kHeadThreads) {
        float sum = 0.0f;
        if (i == 0U) {
            for (uint32_t w = 0; w < 8U; ++w) sum += red[w];
        } else if (i <= a.H2) {
            for (uint32_t g = 0; g < groups; ++g) sum += cols[g * a.H2 + i - 1U];
        } else {
            for (uint32_t w = 0; w < 8U; ++w) sum += red[8U + w * 64U + i - 1U - a.H2];
        }
        out[i] = sum;
    }
}

// More than 64 outputs: one warp per sample, plain SIMT. Column sums of dy are left to HeadOutNBiasGradKernel.
template <bool kCrossEntropy, bool kF32>
__global__ void __launch_bounds__(kHeadThreads)
HeadOutNKernel(const __grid_constant__ HeadArgs a) {
    extern __shared__ float s_dyn[];  // per warp: OUT floats (logits, then rounded dy)
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31U;
    const uint32_t warps_total = gridDim.x * (kHeadThreads / 32), H2 = a.H2, OUT = a.OUT;
    dependent_begin();
    float* s_dy = s_dyn + warp * OUT;
    auto weight = [&](uint32_t j, uint32_t o) -> float {
        return kF32 ? static_cast<const float*>(a.w_out)[(uint64_t)j * a.p_wout + o] : ptx::from_operand(static_cast<const uint16_t*>(a.w_out)[(uint64_t)j * a.p_wout + o], a.bf16);
    };
    const float inv_n = 1.0f / static_cast<float>(kCrossEntropy ? (uint64_t)a.B : (uint64_t)a.B * OUT);
    float loss = 0.0f, none[1] = {0.0f};
    float dacc[kHeadMaxPerLane];
#pragma unroll
    for (int q = 0; q < kHeadMaxPerLane; ++q) dacc[q] = 0.0f;
    for (uint32_t b = blockIdx.x * (kHeadThreads / 32) + warp; b < a.B; b += warps_total) {
        const uint16_t* row = reinterpret_cast<const uint16_t*>(a.x_h) + (uint64_t)b * a.p_act;
        const float* row_f = a.x_f32 + (uint64_t)b * a.p_f32;
        for (uint32_t o = lane; o < OUT; o += 32) {
            float acc = 0.0f;
            for (uint32_t j = 0; j < H2; ++j) acc += (kF32 ? row_f[j] : ptx::from_operand(row[j], a.bf16)) * weight(j, o);
            s_dy[o] = acc + a.b_out[o];
        }
        __syncwarp();
        HeadLossRow<kCrossEntropy, kF32, 1>(a, b, inv_n, s_dy, lane, loss, none);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < kHeadMaxPerLane; ++q) {
            const uint32_t j = q * 32 + lane;
            if (j < H2) {
                float acc = 0.0f;
                for (uint32_t o = 0; o < OUT; ++o) acc += s_dy[o] * weight(j, o);
                const float d = row_f[j] > 0.0f ? acc : 0.0f;
                dacc[q] += d;
                a.dzf[(uint64_t)b * a.p_f32 + j] = d;
                if (!kF32) reinterpret_cast<uint16_t*>(a.dz_h)[(uint64_t)b * a.p_dz + j] = ptx::to_operand(d, a.bf16);
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) loss += __shfl_xor_sync(0xFFFFFFFFU, loss, o);
    __shared__ float s_part[kHeadThreads / 32][MGT_MAX_HD2 + 1];
    if (lane == 0) s_part[warp][0] = loss;
#pragma unroll
    for (int q = 0; q < kHeadMaxPerLane; ++q) {
        const uint32_t j = q * 32 + lane;
        if (j < H2) s_part[warp][1 + j] = dacc[q];
    }
    __syncthreads();
    for (uint32_t j = threadIdx.x; j < H2 + 1; j += kHeadThreads) {
        float sum = 0.0f;
        for (int wi = 0; wi < kHeadThreads / 32; ++wi) sum += s_part[wi][j];
        a.partials[(uint64_t)blockIdx.x * (1U + H2 + OUT) + j] = sum;
    }
}

// grad b_out[o] = sum_b dy[b][o]: one CTA per output, rows dealt to the threads and added in a fixed tree.
__global__ void __launch_bounds__(256)
HeadOutNBiasGradKernel(const float* __restrict__ dy, uint32_t B, uint32_t OUT, float* __restrict__ grad_b) {
    __shared__ float s_sum[256];
    dependent_begin();
    const uint32_t o = blockIdx.x;
    float sum = 0.0f;
    for (uint32_t b = threadIdx.x; b < B; b += 256U) sum += dy[(uint64_t)b * OUT + o];
    s_sum[threadIdx.x] = sum;
    __syncthreads();
    for (uint32_t w = 128U; w > 0U; w >>= 1) {
        if (threadIdx.x < w) s_sum[threadIdx.x] += s_sum[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) grad_b[o] = s_sum[0];
}

// The dynamic shared memory a kernel may take is an attribute that every thread of the process shares: it is set once per device,
// to all that is left beside the kernel's static arrays, never to what this launch needs (another thread's launch may want more
// at that moment, and a kernel with static arrays needs it set below 48 KB too).
template <void (*kKernel)(HeadArgs)>
bool LaunchHeadKernel(int device, uint32_t grid, size_t smem, LaunchOn st, const HeadArgs& a) {
    static std::mutex attr_mu;
    static size_t most[64] = {};
    if (device < 0 || device >= 64) return false;
    {
        std::lock_guard<std::mutex> lock(attr_mu);
        if (most[device] == 0) {
            cudaFuncAttributes attr{};
            int limit = 0;
            if (cudaFuncGetAttributes(&attr, kKernel) != cudaSuccess || cudaDeviceGetAttribute(&limit, cudaDevAttrMaxSharedMemoryPerBlockOptin, device) != cudaSuccess) return false;
            const size_t left = static_cast<size_t>(limit) - attr.sharedSizeBytes;
            if (cudaFuncSetAttribute(kKernel, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(left)) != cudaSuccess) return false;
            most[device] = left;
        }
        if (smem > most[device]) return false;
    }
    Launch(kKernel, grid, kHeadThreads, smem, st, a);
    return true;
}

// The sums of a step that wait to be launched. Pass() launches them when the caller wants finished ranges on the way or the stages
// timed (`at_once`), or when kMostWaiting bytes of partial results wait: those are still in L2 then (p888: the planes of a weight
// gradient are 13 to 16 MB). Sums that find the list full launch what waits first; whether that worked is told by the next
// Pass() or LaunchAll(). They go to the stream `on`, which every kernel that left the partial results has to be ahead of.
struct Sums {
    static constexpr uint64_t kMostWaiting = 8ULL << 20;
    mgt_engine* e;
    bool at_once;
    LaunchOn on;
    SumJobs jobs{};
    uint64_t waiting = 0;
    mgt_status_t full = MGT_OK;  // of the launches that made room

    void Add(SumJob j, uint32_t groups) {
        if (groups == 0U) return;
        if (jobs.count == SumJobs::kMax && full == MGT_OK) full = LaunchAll();
        if (full != MGT_OK) return;
        const uint32_t per_cta = j.form == SumJob::kLanes ? kReduceCols : (j.form == SumJob::kQuad ? 1024U : 256U);
        j.per_group = (uint32_t)((j.items + per_cta - 1U) / per_cta);
        j.first_cta = jobs.ctas;
        jobs.ctas += j.per_group * groups;
        waiting += j.items * j.terms * groups * sizeof(float);
        jobs.job[jobs.count++] = j;
    }
    // dst[i] = sum over `rows` rows of src[r * stride + i]
    void Rows(const float* src, uint32_t rows, uint64_t stride, uint32_t items, float* dst, uint32_t groups = 1, uint64_t src_group = 0, uint64_t dst_group = 0) {
        Add({src, dst, src_group, dst_group, stride, items, rows, 0, 0, SumJob::kLanes}, groups);
    }
    // dst[group][i] = sum over the group's `splits` planes of `count` floats
    void Planes(const float* src, uint32_t splits, uint64_t count, float* dst, uint32_t groups = 1, uint64_t dst_group = 0) {
        const bool quads = ((count | dst_group) & 3ULL) == 0ULL && ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15U) == 0U;
        Add({src, dst, splits * count, dst_group, count, count, splits, 0, 0, quads ? SumJob::kQuad : SumJob::kItem}, groups);
    }
    // what HeadOut1Kernel's CTAs leave: rows of { grad W_out, grad b_out, loss, column sums of dz }
    void Head(const float* src, uint32_t rows, uint32_t H2, float* grad_out_layer, float* loss, float* bias_below) {
        const uint32_t width = 2U * H2 + 2U;
        Rows(src, rows, width, H2 + 1U, grad_out_layer);
        Rows(src + H2 + 1U, rows, width, 1, loss);
        if (bias_below != nullptr) Rows(src + H2 + 2U, rows, width, H2, bias_below);
    }
    // bias gradients of the tower from its column sums: slot k -> b1_k, slot R + k -> b2_{k-1} (the hidden bias for k = 0)
    void TowerBiases(const mgt_mlp_shape_t& s, const float* colsum, uint32_t rows, uint64_t slot, float* grad, bool second) {
        const uint32_t H = s.hd2, R = s.residual_blocks;
        Rows(colsum, rows, H, H, grad + Fc1B(s, 0), R, slot, BlockParams(s));
        if (!second) return;
        Rows(colsum + slot * R, rows, H, H, grad + HiddenBias(s));
        Rows(colsum + slot * (R + 1ULL), rows, H, H, grad + Fc2B(s, 0), R - 1U, slot, BlockParams(s));
    }
    mgt_status_t Pass() { return at_once || waiting > kMostWaiting ? LaunchAll() : full; }
    mgt_status_t LaunchAll() {
        if (full != MGT_OK || jobs.count == 0U) return full;
        mgt::Launch(SumKernel, jobs.ctas, 256, 0, on, jobs);
        jobs.count = jobs.ctas = 0U;
        waiting = 0;
        ++e->launches;
        return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
    }
};

// Output layer with several outputs, its loss and the gradient entering the layer below, enqueued; all gradients of the head
// except W_out's, which is a product over the batch.
template <bool kCrossEntropy, bool kF32>
mgt_status_t LaunchHeadN(mgt_engine* e, LaunchOn st, const HeadArgs& a, Sums& sums, float* loss, float* bias_below, float* grad_b) {
    const bool tiled = a.OUT <= 64U;
    const uint32_t tiles = tiled ? (a.B + kHeadTile - 1U) / kHeadTile : (a.B + 7U) / 8U;
    const uint32_t grid = tiles < kHeadBlocks ? tiles : kHeadBlocks;
    bool ok;
    if (a.OUT <= 16U) ok = LaunchHeadKernel<HeadTileKernel<16, kCrossEntropy, kF32>>(e->device, grid, HeadTileSmem<16>(a.H2), st, a);
    else if (a.OUT <= 32U) ok = LaunchHeadKernel<HeadTileKernel<32, kCrossEntropy, kF32>>(e->device, grid, HeadTileSmem<32>(a.H2), st, a);
    else if (tiled) ok = LaunchHeadKernel<HeadTileKernel<64, kCrossEntropy, kF32>>(e->device, grid, HeadTileSmem<64>(a.H2), st, a);
    else {
        // With more than a CTA an SM not before the kernel ahead has ended: this one has its weights through L1, and a CTA that begins beside a
        // tower's keeps the split of the SM that the tower asked for, all shared memory (8 433 samples, hd2 256: 128 outputs 2 671 us a step,
        // 1 634 like this; 70 outputs 732, 550; 2 000 samples 240, 241; but 500 samples, hd2 64 103, 105).
        ok = LaunchHeadKernel<HeadOutNKernel<kCrossEntropy, kF32>>(e->device, grid, (kHeadThreads / 32) * a.OUT * sizeof(float), {st.stream, st.overlap && grid <= (uint32_t)e->sm_count}, a);
    }
    if (!ok) return MGT_CUDA_FAILURE;
    // the partial rows of the CTAs: { loss, column sums of dz, with up to 64 outputs column sums of dy }
    const uint32_t width = 1U + a.H2 + a.OUT;
    sums.Rows(a.partials, grid, width, 1, loss);
    if (bias_below != nullptr) sums.Rows(a.partials + 1U, grid, width, a.H2, bias_below);
    if (tiled) sums.Rows(a.partials + 1U + a.H2, grid, width, a.OUT, grad_b);
    else Launch(HeadOutNBiasGradKernel, a.OUT, 256, 0, st, a.dy, a.B, a.OUT, grad_b);
    e->launches += tiled ? 1 : 2;
    return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
}

inline uint32_t GridFor(uint64_t items, uint32_t threads, int sm_count) {
    const uint64_t want = (items + threads - 1) / threads;
    const uint64_t cap = (uint64_t)sm_count * 8;
    return (uint32_t)(want < 1 ? 1 : (want < cap ? want : cap));
}

// Work of the backward pass on a second stream, beside the caller's: from Fork() on, until the object ends (on every path, so that
// the caller's stream is never ahead of it). Every stream the engine is called on has a second one of its own: on a shared one a
// step would wait for the step of another stream. (Beyond kSides streams they do share; only the time differs.) Fork() may find no
// second stream - none can be made, or a capture of other streams holds it - and then all work stays on the caller's, with the same
// bits.
struct SideBranch {
    static constexpr size_t kSides = 4;
    mgt_engine* e;
    cudaStream_t main;
    SideStream side{};
    bool open = false;

    bool TieLocked(int event, cudaStream_t from, cudaStream_t to) {
        return cudaEventRecord(side.events[event], from) == cudaSuccess && cudaStreamWaitEvent(to, side.events[event], 0) == cudaSuccess;
    }
    bool Tie(int event, cudaStream_t from, cudaStream_t to) {
        std::lock_guard<std::mutex> lock(e->side_mu);
        return TieLocked(event, from, to);
    }
    bool Fork() {
        std::lock_guard<std::mutex> lock(e->side_mu);
        const unsigned long long capture = CaptureOf(main);
        bool ok = capture != ~0ULL;
        mgt_engine::SideOf* slot = nullptr;
        for (auto& known : e->sides)
            if (ok && known.main == main) slot = &known;
        if (ok && slot == nullptr && e->sides.size() < kSides) {
            SideStream taken;
            if ((ok = SidePool::Get().Take(e->device, capture == 0, &taken))) {
                e->sides.push_back({main, taken});
                slot = &e->sides.back();
            }
        } else if (ok && slot == nullptr) {
            slot = &e->sides[e->side_turn++ % kSides];
            slot->main = main;
        }
        if (ok) {
            side = slot->side;
            const unsigned long long held = CaptureOf(side.stream);
            ok = held == 0 || held == capture;
            open = ok && TieLocked(0, main, side.stream);
            e->forks += open ? 1U : 0U;
        }
        if (!open) cudaGetLastError();
        return open;
    }
    bool Join() {
        const bool was = open;
        open = false;
        return !was || Tie(2, side.stream, main);
    }
    ~SideBranch() { Join(); }
};

struct StageTimer {
    mgt_engine* e;
    cudaStream_t stream;
    mgt_backward_profile_t* profile;
    bool Start() {
        if (!profile) return true;
        std::memset(profile, 0, sizeof(*profile));
        if (!e->ev_last && cudaEventCreate(&e->ev_last) != cudaSuccess) return false;
        if (!e->ev_now && cudaEventCreate(&e->ev_now) != cudaSuccess) return false;
        return cudaEventRecord(e->ev_last, stream) == cudaSuccess;
    }
    // As in the reference, every mark synchronises the host (native/cuda/mlp_backward.cu:211-221).
    bool Mark(float* dst) {
        if (!profile) return true;
        float ms = 0.0f;
        if (cudaEventRecord(e->ev_now, stream) != cudaSuccess) return false;
        if (cudaEventSynchronize(e->ev_now) != cudaSuccess) return false;
        if (cudaEventElapsedTime(&ms, e->ev_last, e->ev_now) != cudaSuccess) return false;
        *dst += ms;  // a stage may be visited twice (its dX part and, later, its dW part): Start() zeroed the profile
        std::swap(e->ev_last, e->ev_now);
        return true;
    }
};

#define MGT_TRY(...)                          \
    do {                                      \
        const mgt_status_t _st = (__VA_ARGS__); \
        if (_st != MGT_OK) return _st;        \
    } while (0)
#define MGT_MAP(...)                               \
    do {                                           \
        if (!(__VA_ARGS__)) return MGT_CUDA_FAILURE; \
    } while (0)

// D = act[M x K, K-major] * W[K x N, row-major] with a forward epilogue.
template <Epi EPI>
mgt_status_t GemmForward(mgt_engine* e, LaunchOn st, const __half* act, uint32_t act_pitch, const __half* w, uint32_t w_pitch,
                         uint32_t M, uint32_t N, uint32_t K, GemmArgs epi) {
    const uint32_t bn = PickBN(N);
    GemmArgs a = BaseArgs(M, N, K, bn, 1);
    a.bias = epi.bias; a.out_f32 = epi.out_f32; a.ld_f32 = epi.ld_f32; a.out_f16 = epi.out_f16; a.ld_f16 = epi.ld_f16;
    a.add_f32 = epi.add_f32; a.ld_add = epi.ld_add; a.mask = epi.mask; a.ld_mask = epi.ld_mask; a.moments = epi.moments;
    CUtensorMap ta, tb;
    MGT_MAP(e->Map(&ta, act, K, M, act_pitch, 64, 128));
    MGT_MAP(e->Map(&tb, w, N, K, w_pitch, 64, 64));
    if (a.k_chunks <= 4) return bn == 224 ? LaunchGemm<CfgFwdS<224, EPI>>(e, ta, tb, a, st) : LaunchGemm<CfgFwdS<256, EPI>>(e, ta, tb, a, st);
    return bn == 224 ? LaunchGemm<CfgFwd<224, EPI>>(e, ta, tb, a, st) : LaunchGemm<CfgFwd<256, EPI>>(e, ta, tb, a, st);
}

// The same product with the activation stored as actT[K][M] (one row per input column): an MN-major A operand.
template <Epi EPI>
mgt_status_t GemmForwardRows(mgt_engine* e, LaunchOn st, const __half* act_t, uint32_t act_t_pitch, const __half* w, uint32_t w_pitch,
                             uint32_t M, uint32_t N, uint32_t K, GemmArgs epi) {
    const uint32_t bn = PickBN(N);
    GemmArgs a = BaseArgs(M, N, K, bn, 1);
    a.bias = epi.bias; a.out_f32 = epi.out_f32; a.ld_f32 = epi.ld_f32; a.out_f16 = epi.out_f16; a.ld_f16 = epi.ld_f16;
    a.add_f32 = epi.add_f32; a.ld_add = epi.ld_add; a.mask = epi.mask; a.ld_mask = epi.ld_mask; a.moments = epi.moments;
    CUtensorMap ta, tb;
    MGT_MAP(e->Map(&ta, act_t, M, K, act_t_pitch, 64, 64));
    MGT_MAP(e->Map(&tb, w, N, K, w_pitch, 64, 64));
    return bn == 224 ? LaunchGemm<CfgFwdRows<224, EPI>>(e, ta, tb, a, st) : LaunchGemm<CfgFwdRows<256, EPI>>(e, ta, tb, a, st);
}

// How a dX GEMM is run: tile width, form, grid, and the rows of its column-sum scratch (one per epilogue warp of every CTA).
struct BackpropPlan {
    uint32_t bn;
    bool stationary;
    uint32_t grid, rows;
};
BackpropPlan PlanBackprop(const mgt_engine* e, uint32_t M, uint32_t N, uint32_t K) {
    BackpropPlan p{};
    const uint32_t sm = (uint32_t)e->sm_count;
    p.bn = PickBN(N);
    const GemmArgs a = BaseArgs(M, N, K, p.bn, 1);
    p.stationary = a.k_chunks <= 4 && a.n_tiles <= sm;
    const uint64_t units = (uint64_t)a.m_tiles * a.n_tiles;
    p.grid = (uint32_t)(units < (uint64_t)sm ? units : (uint64_t)sm);
    if (p.stationary && p.grid >= a.n_tiles) p.grid = p.grid / a.n_tiles * a.n_tiles;  // as LaunchGemm picks it
    p.rows = p.grid * 8U;
    return p;
}

// dX[M x N] = dz[M x K, K-major] * W[N x K, row-major]^T with a backward epilogue that produces the
// next dz tensor; its fp32 column sums (a bias gradient) go to `colsum` (zeroed by the caller,
// PlanBackprop().rows rows of N).
template <Epi EPI>
mgt_status_t GemmBackpropInput(mgt_engine* e, LaunchOn st, const __half* dz, uint32_t dz_pitch, const __half* w, uint32_t w_pitch,
                               uint32_t M, uint32_t N, uint32_t K, GemmArgs epi, float* colsum) {
    const BackpropPlan p = PlanBackprop(e, M, N, K);
    GemmArgs a = BaseArgs(M, N, K, p.bn, 1);
    a.out_f32 = epi.out_f32; a.ld_f32 = epi.ld_f32; a.out_f16 = epi.out_f16; a.ld_f16 = epi.ld_f16;
    a.add_f32 = epi.add_f32; a.ld_add = epi.ld_add; a.mask = epi.mask; a.ld_mask = epi.ld_mask;
    a.colsum = colsum;
    CUtensorMap ta, tb;
    MGT_MAP(e->Map(&ta, dz, K, M, dz_pitch, 64, 128));
    MGT_MAP(e->Map(&tb, w, K, N, w_pitch, 64, p.bn));
    if (p.stationary) return p.bn == 224 ? LaunchGemm<CfgDxS<224, EPI>>(e, ta, tb, a, st) : LaunchGemm<CfgDxS<256, EPI>>(e, ta, tb, a, st);
    return p.bn == 224 ? LaunchGemm<CfgDx<224, EPI>>(e, ta, tb, a, st) : LaunchGemm<CfgDx<256, EPI>>(e, ta, tb, a, st);
}

// The weight gradients of all residual blocks for one of the two linear layers in ONE launch:
// grad_g[in x out] = act_g^T * dz_g for g = 0..groups-1, where act_g / dz_g are slices of two tapes and
// grad_g lie `grad_group_stride` floats apart. Split-K.
mgt_status_t GemmGradWeightsGrouped(mgt_engine* e, LaunchOn st, const __half* act_tape, uint32_t act_pitch, uint64_t act_stride_bytes,
                                    const __half* dz_tape, uint32_t dz_pitch, uint64_t dz_stride_bytes, uint32_t groups, uint32_t samples,
                                    uint32_t in_dim, uint32_t out_dim, float* partial, Sums& sums, float* grad_first, uint64_t grad_group_stride) {
    const uint32_t bn = PickBN(out_dim);
    GemmArgs a = BaseArgs(in_dim, out_dim, samples, bn, MostSplits(in_dim, out_dim, groups, (uint32_t)e->sm_count));
    a.groups = groups;
    a.partial = partial;
    CUtensorMap ta, tb;
    MGT_MAP(e->Map3D(&ta, act_tape, in_dim, samples, groups, act_pitch, act_stride_bytes, 64, 64));
    MGT_MAP(e->Map3D(&tb, dz_tape, out_dim, samples, groups, dz_pitch, dz_stride_bytes, 64, 64));
    MGT_TRY(bn == 224 ? LaunchGemm<CfgDwG<224>>(e, ta, tb, a, st) : LaunchGemm<CfgDwG<256>>(e, ta, tb, a, st));
    sums.Planes(partial, a.splits, (uint64_t)in_dim * out_dim, grad_first, groups, grad_group_stride);
    return MGT_OK;
}

// grad[in x out] = act^T * dz, reduced over the batch with split-K.
mgt_status_t GemmGradWeights(mgt_engine* e, LaunchOn st, const __half* act, uint32_t act_pitch, const __half* dz, uint32_t dz_pitch,
                             uint32_t samples, uint32_t in_dim, uint32_t out_dim, float* partial, Sums& sums, float* grad_out) {
    const uint32_t bn = PickBN(out_dim);
    GemmArgs a = BaseArgs(in_dim, out_dim, samples, bn, MostSplits(in_dim, out_dim, 1, (uint32_t)e->sm_count));
    a.partial = partial;
    CUtensorMap ta, tb;
    MGT_MAP(e->Map(&ta, act, in_dim, samples, act_pitch, 64, 64));
    MGT_MAP(e->Map(&tb, dz, out_dim, samples, dz_pitch, 64, 64));
    MGT_TRY(bn == 224 ? LaunchGemm<CfgDw<224>>(e, ta, tb, a, st) : LaunchGemm<CfgDw<256>>(e, ta, tb, a, st));
    sums.Planes(partial, a.splits, (uint64_t)in_dim * out_dim, grad_out);
    return MGT_OK;
}

// grad[in x out] = act^T * dz with the activation stored as actT[in][samples]: a K-major A operand.
mgt_status_t GemmGradWeightsRows(mgt_engine* e, LaunchOn st, const __half* act_t, uint32_t act_t_pitch, const __half* dz, uint32_t dz_pitch,
                                 uint32_t samples, uint32_t in_dim, uint32_t out_dim, float* partial, Sums& sums, float* grad_out) {
    const uint32_t bn = PickBN(out_dim);
    GemmArgs a = BaseArgs(in_dim, out_dim, samples, bn, MostSplits(in_dim, out_dim, 1, (uint32_t)e->sm_count));
    a.partial = partial;
    CUtensorMap ta, tb;
    MGT_MAP(e->Map(&ta, act_t, samples, in_dim, act_t_pitch, 64, 128));
    MGT_MAP(e->Map(&tb, dz, out_dim, samples, dz_pitch, 64, 64));
    MGT_TRY(bn == 224 ? LaunchGemm<CfgDwRows<224>>(e, ta, tb, a, st) : LaunchGemm<CfgDwRows<256>>(e, ta, tb, a, st));
    sums.Planes(partial, a.splits, (uint64_t)in_dim * out_dim, grad_out);
    return MGT_OK;
}

// dxT[N_in x samples] = (W[N_in x K] * dz[samples x K]^T) * [mask bit]: the hidden layer's dX with its wide side as rows; the
// mask words are the ones the embedding forward wrote beside its activation.
// Row sums of the result (the bias gradient of the layer below) go to bias_grad[N_in] with the step's sums. With
// dx_f32 the result goes there instead, in fp32 and with one row per sample; with dx_rows it goes to dx_t in the operand format
// with one row per sample.
mgt_status_t GemmBackpropInputRows(mgt_engine* e, LaunchOn st, const __half* w, uint32_t w_pitch, const __half* dz, uint32_t dz_pitch, uint32_t samples,
                                   uint32_t in_dim, uint32_t out_dim, uint32_t* mask_bits, uint32_t ld_bits, __half* dx_t, uint32_t t_pitch, float* dx_f32, uint32_t f32_pitch, bool dx_rows, uint32_t dx_rows_pitch, float* rowsum,
                                   uint64_t rowsum_rows, Sums& sums, float* bias_grad) {
    GemmArgs a = BaseArgs(in_dim, samples, out_dim, CfgDxRows::BN, 1);
    const uint64_t rows = (uint64_t)a.n_tiles * CfgDxRows::EPI_STRIDE;
    if (rows > rowsum_rows) return MGT_CAPACITY_EXCEEDED;
    a.bits = mask_bits; a.ld_bits = ld_bits; a.out_f16 = dx_t; a.ld_f16 = t_pitch; a.out_f32 = dx_f32; a.ld_f32 = f32_pitch; a.rowsum = rowsum;
    if (dx_rows) a.ld_f16 = dx_rows_pitch;
    CUtensorMap ta, tb;
    MGT_MAP(e->Map(&ta, w, out_dim, in_dim, w_pitch, 64, 128));
    MGT_MAP(e->Map(&tb, dz, out_dim, samples, dz_pitch, 64, CfgDxRows::BN));
    if (dx_f32 != nullptr) {
        MGT_TRY(LaunchGemm<CfgDxRowsF32>(e, ta, tb, a, st));
    } else if (dx_rows) {
        MGT_TRY(LaunchGemm<CfgDxRowsF16T>(e, ta, tb, a, st));
    } else if ((uint64_t)a.m_tiles * a.n_tiles > (uint64_t)e->sm_count) {
        CUtensorMap to;
        MGT_MAP(e->Map(&to, dx_t, samples, in_dim, t_pitch, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B));
        MGT_TRY(LaunchGemm<CfgDxRowsTma>(e, ta, tb, a, st, &to));
    } else {  // (a CTA with one unit only waits for its stores at the end: 4 096 samples of hd1 1024 199.4 us a step, 200.3 with TMA stores)
        MGT_TRY(LaunchGemm<CfgDxRows>(e, ta, tb, a, st));
    }
    sums.Rows(rowsum, (uint32_t)rows, in_dim, in_dim, bias_grad);
    return MGT_OK;
}

// The residual tower in one launch per direction. hd2 up to 256: tower_chain.cuh, a CTA per tile of 128 samples (the tile's
// state and product take two TMEM columns per hidden unit). Up to the largest width, 512: tower_wide.cuh, a pair of CTAs per tile.
bool ChainEligible(const mgt_engine* e, const mgt_mlp_shape_t& s) {
    return s.residual_blocks > 0 && !e->layered_tower;
}

template <bool BWD>
mgt_status_t LaunchChain(mgt_engine* e, LaunchOn st, const __half* w_first, uint32_t w_pitch, uint64_t w_layer_stride_bytes, uint32_t tape_s_entries,
                         uint32_t tape_t_entries, ChainArgs a) {
    static std::mutex attr_mu;
    static bool attr_done[64] = {};
    {
        std::lock_guard<std::mutex> lock(attr_mu);
        if (e->device >= 0 && e->device < 64 && !attr_done[e->device]) {
            if (cudaFuncSetAttribute(tower_chain_kernel<BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, ChainCfg::SMEM_BYTES) != cudaSuccess ||
                cudaFuncSetAttribute(tower_wide_kernel<BWD>, cudaFuncAttributeMaxDynamicSharedMemorySize, WideCfg::SMEM_BYTES) != cudaSuccess) return MGT_CUDA_FAILURE;
            attr_done[e->device] = true;
        }
    }
    const bool wide = a.H > 256U;
    CUtensorMap tw, ts, tt;
    // (backward: a box of weight rows for the columns of one CTA)
    MGT_MAP(e->Map3D(&tw, w_first, a.H, a.H, 2ULL * a.R, w_pitch, w_layer_stride_bytes, 64, !BWD ? 64U : (wide ? (a.H + 127U) / 128U * 64U : (a.H + 31U) & ~31U)));
    // the tapes as stacks of [samples][H] matrices; a store box is one operand panel: 64 columns x 128 rows
    MGT_MAP(e->Map3D(&ts, a.tape_s, a.H, a.samples, tape_s_entries, a.ld_s, a.tape_s_stride * 2, 64, 128));
    MGT_MAP(e->Map3D(&tt, a.tape_t, a.H, a.samples, tape_t_entries, a.ld_t, a.tape_t_stride * 2, 64, 128));
    a.status = e->status_word;
    a.bf16 = e->bf16_now ? 1U : 0U;
    const uint32_t units = wide ? (uint32_t)e->sm_count / 2U : (uint32_t)e->sm_count, grid = a.tiles < units ? a.tiles : units;
    if (wide) Launch(tower_wide_kernel<BWD>, 2U * grid, WideCfg::THREADS, WideCfg::SMEM_BYTES, st, tw, ts, tt, a);
    else Launch(tower_chain_kernel<BWD>, grid, ChainCfg::THREADS, ChainCfg::SMEM_BYTES, st, tw, ts, tt, a);
    ++e->launches;
    return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
}

// ---- the fp32 data flow (use_half_linear == 0), mlp_backward.cu:1273-1510 without the fp16 copies -----------------
// Every activation and every gradient w.r.t. a pre-activation is kept (as in the tensor-core flow), so that the weight
// gradients of all blocks are two grouped products at the end. Rows are padded to four floats.
struct Fp32Workspace {
    uint32_t p1, p2;
    uint64_t a1, x, r1, dz2, dz1t, dz1, dy, head, partial, partial_fc2, partial_fc1, partial_out, colsum, colsum_slot, colsum_in, bits, bits_entry, tower_w, lists, total;  // float offsets
};
// The blocks in one launch per direction (fp32_tower.cuh). Widths up to 128: always (us a step, by layers and fused: 1 000 samples of hd2
// 128, 16 blocks 680, 490; 30 000 of hd2 128, 8 blocks 1 960, 1 800; 300 of hd2 8, 32 blocks 900, 200). Up to 256: a CTA streams every
// matrix through one warp, which is the longest part with few samples to a CTA (2 000 samples, 6 blocks, hd2 160 441, 365; 192 440, 416; 224
// 526, 573; 256 598, 654; 2 500 of hd2 160 466, 426; 224 765, 668; 256 812, 752). From there on it is the faster form while one round of the
// chip takes all samples (8 blocks: 5 000 of hd2 160 920, 690; 7 000 of hd2 240 1 531, 1 426). Beyond, both go in steps, the tower of 32 to
// 56 samples an SM, the products of a tile an SM, and an estimate of both decides (hd2 224: 9 500 2 013, 2 420; 12 000 2 393, 2 507; 20 000
// 4 468, 3 573; hd2 160: 9 500 1 372, 1 257; 12 000 1 506, 1 699). Of 119 steps of 8 400 to 42 000 samples it took the slower form for
// 10, by 4.6 % at most. Wider ones are products of their own (2 500 of hd2 510, 8 blocks 3 260, 4 330).
constexpr uint32_t kFusedFp32Batch = 2500U;
// whether any batch of up to B samples is fused: scratch is planned by this
bool MayFuseFp32Tower(const mgt_mlp_shape_t& s, uint32_t B) { return s.residual_blocks > 0 && (s.hd2 <= 128U || (s.hd2 <= 256U && B >= kFusedFp32Batch)); }
bool FusedFp32Tower(const mgt_mlp_shape_t& s, uint32_t B, uint32_t sm) {
    if (!MayFuseFp32Tower(s, B)) return false;
    if (s.hd2 <= 128U) return true;
    const fp32path::TowerPlan plan = fp32path::PlanTower(B, s.hd2, sm);
    if (plan.rounds == 1U) return true;
    auto each = [&](uint32_t t) { return ((uint64_t)((B + t - 1U) / t) * ((s.hd2 + t - 1U) / t) + sm - 1U) / sm; };  // tiles for the fullest SM
    const bool large = fp32path::PickSgemmTile(B, s.hd2, 1, sm) == fp32path::SgemmTile::kLarge;
    return plan.us < (large ? 20.0 + 0.130 * s.hd2 * (double)each(128U) : 13.2 + 0.0284 * s.hd2 * (double)each(64U));
}
struct DwPlan {
    fp32path::SgemmTile tile;
    uint32_t splits;
};
// Weight gradients: few tiles, a long sum over the batch. Enough K splits for eight CTAs of the middle tile per SM, as long as
// a split keeps 256 samples (16 products of 224 x 224 over 8 192 samples: 3, 6, 9 splits 428, 380, 365 us).
DwPlan PlanDw(uint32_t M, uint32_t N, uint32_t K, uint32_t groups, uint32_t sm) {
    DwPlan p{M > 32U && N > 32U ? fp32path::SgemmTile::kMiddle : fp32path::SgemmTile::kSmall, 1U};
    const uint32_t t = fp32path::SgemmTileRows(p.tile);
    const uint64_t tiles = (uint64_t)((M + t - 1) / t) * ((N + t - 1) / t) * groups;
    const uint64_t want = (8ULL * sm + tiles - 1) / tiles, most = K / 256U > 0U ? K / 256U : 1U;
    p.splits = (uint32_t)(want < most ? want : most);
    return p;
}
Fp32Workspace PlanFp32(const mgt_mlp_shape_t& s, uint32_t B, uint32_t sm) {
    Fp32Workspace w{};
    uint64_t off = 0;
    auto take = [&](uint64_t n) { const uint64_t at = off; off += (n + 63) & ~63ULL; return at; };
    w.p1 = (uint32_t)RoundUp(s.hd1, 4);
    w.p2 = (uint32_t)RoundUp(s.hd2, 4);
    const uint64_t bh2 = (uint64_t)B * w.p2, bh1 = (uint64_t)B * w.p1, r = s.residual_blocks > 0 ? s.residual_blocks : 1ULL;
    w.a1 = take(bh1);
    w.x = take(bh2 * (s.residual_blocks + 1ULL));
    w.r1 = take(bh2 * r);
    w.dz2 = take(bh2 * (s.residual_blocks + 1ULL));
    w.dz1t = take(bh2 * r);
    w.dz1 = take(bh1);
    w.dy = take((uint64_t)B * s.output_dim);
    w.head = take((uint64_t)kHeadBlocks * HeadPartialFloats(s));
    auto planes = [&](uint32_t M, uint32_t N, uint32_t groups) { return (uint64_t)PlanDw(M, N, B, groups, sm).splits * groups * M * N; };
    w.partial = take(planes(s.hd1, s.hd2, 1));
    w.partial_fc2 = take(planes(s.hd2, s.hd2, (uint32_t)r));
    w.partial_fc1 = take(planes(s.hd2, s.hd2, (uint32_t)r));
    w.partial_out = take(s.output_dim > 1 ? planes(s.hd2, s.output_dim, 1) : 0);
    const bool fused = MayFuseFp32Tower(s, B);
    w.colsum_slot = (fused ? fp32path::TowerSumRows(B) : (uint64_t)((B + 31U) / 32U)) * s.hd2;  // one row per tile of at least 32 samples, 8 in the tower
    w.colsum = take(w.colsum_slot * 2 * r);
    w.colsum_in = take((uint64_t)((B + 31U) / 32U) * s.hd1);
    w.bits_entry = fp32path::TowerBitWords(B, s.hd2);
    w.bits = take(fused ? w.bits_entry * 2 * r : 0);
    w.tower_w = take(fused ? 2 * r * (uint64_t)w.p2 * w.p2 : 0);  // (the tower's matrices padded, where it cannot take them as they lie)
    w.lists = take(gather::ListWords(B, s.state_len, s.state_value_pad));
    w.total = off + 64;
    return w;
}
uint64_t Fp32WorkspaceFloats(const mgt_mlp_shape_t& s, uint32_t B, uint32_t sm) { return PlanFp32(s, B, sm).total; }

template <class F>
mgt_status_t LaunchFp32Path(mgt_engine* e, const mgt_mlp_shape_t& s, const float* w, const uint8_t* states, const float* labels, uint32_t B, float* loss,
                            float* grad, float* workspace, bool half_ig, bool told, mgt_backward_profile_t* profile, F&& notify, LaunchOn st) {
    using namespace mgt::fp32path;
    const uint32_t sm = PlanSmCount(e->sm_count);
    const Fp32Workspace ws = PlanFp32(s, B, sm);
    float* base = reinterpret_cast<float*>(RoundUp(reinterpret_cast<uintptr_t>(workspace), 256));
    const uint32_t H1 = s.hd1, H2 = s.hd2, R = s.residual_blocks, OUT = s.output_dim, L = s.state_len, V = s.state_value_pad, p1 = ws.p1, p2 = ws.p2;
    const uint64_t bh2 = (uint64_t)B * p2;
    float* a1 = base + ws.a1;
    auto x = [&](uint32_t k) { return base + ws.x + bh2 * k; };
    auto r1 = [&](uint32_t k) { return base + ws.r1 + bh2 * k; };
    auto dz2 = [&](uint32_t k) { return base + ws.dz2 + bh2 * k; };    // [0] hidden layer, [k + 1] fc2 of block k
    auto dz1t = [&](uint32_t k) { return base + ws.dz1t + bh2 * k; };  // fc1 of block k
    float *dy = base + ws.dy, *dz1 = base + ws.dz1, *colsum = base + ws.colsum;
    const SgemmTile tile_h2 = PickSgemmTile(B, H2, 1, sm), tile_h1 = PickSgemmTile(B, H1, 1, sm);
    const uint32_t rows_h2 = (B + SgemmTileRows(tile_h2) - 1U) / SgemmTileRows(tile_h2), rows_h1 = (B + SgemmTileRows(tile_h1) - 1U) / SgemmTileRows(tile_h1);
    const bool fused = FusedFp32Tower(s, B, sm);
    const TowerPlan tower = fused ? PlanTower(B, H2, sm) : TowerPlan{};
    TowerArgs tower_args{};
    tower_args.B = B; tower_args.H = H2; tower_args.R = R; tower_args.pitch = p2;
    tower_args.w = w + Fc1W(s, 0); tower_args.ld_w = H2; tower_args.w_step = BlockParams(s) / 2;
    tower_args.bias = w + Fc1B(s, 0); tower_args.bias_step = BlockParams(s) / 2;
    const bool pad_tower = fused && ((H2 & 3U) != 0U || (reinterpret_cast<uintptr_t>(tower_args.w) & 15U) != 0U);
    if (pad_tower) { tower_args.w = base + ws.tower_w; tower_args.ld_w = p2; tower_args.w_step = (uint64_t)p2 * p2; }
    tower_args.tape_stride = bh2;
    tower_args.bits = reinterpret_cast<uint32_t*>(base + ws.bits); tower_args.entry_stride = ws.bits_entry;
    tower_args.status = e->status_word;
    auto ok = [&]() { return cudaGetLastError() == cudaSuccess; };
    // out[B x N] = act[B x K] W[K x N] + bias, ReLU (with the residual added before it)
    auto forward = [&](const float* act, uint32_t ld_act, uint32_t K, const float* weight, const float* bias, const float* res, float* out) {
        SgemmArgs a{};
        a.A = act; a.lda = ld_act; a.B = weight; a.ldb = H2; a.C = out; a.ldc = p2; a.M = B; a.N = H2; a.K = K; a.splits = 1; a.bias = bias; a.add = res; a.ld_add = p2; a.relu = 1U;
        ++e->launches;
        return Sgemm<false, false>(st, a, 1, tile_h2) == cudaSuccess;
    };
    // out[B x N] = (dz[B x H2] W[N x H2]^T (+ skip)) * [act > 0], with its column sums per tile
    auto backward = [&](const float* dz, const float* weight, uint32_t N, const float* skip, const float* act, uint32_t ld, float* out, float* sums, SgemmTile tile) {
        SgemmArgs a{};
        a.A = dz; a.lda = p2; a.B = weight; a.ldb = H2; a.C = out; a.ldc = ld; a.M = B; a.N = N; a.K = H2; a.splits = 1; a.add = skip; a.ld_add = ld; a.mask = act; a.ld_mask = ld;
        a.colsum = sums;
        ++e->launches;
        return Sgemm<false, true>(st, a, 1, tile) == cudaSuccess;
    };
    // (the sums of the step in one launch at its end, unless the caller is told of finished ranges or times the stages)
    Sums sums{e, told, st};
    // grad_g[M x N] = act_g^T dz_g over the batch
    auto weight_grad = [&](const float* act, uint32_t ld_act, uint64_t act_stride, uint32_t M, const float* dz, uint32_t ld_dz, uint64_t dz_stride, uint32_t N, uint32_t groups,
                           float* partial, float* out, uint64_t out_stride) {
        const DwPlan plan = PlanDw(M, N, B, groups, sm);
        SgemmArgs a{};
        a.A = act; a.lda = ld_act; a.stride_a = act_stride; a.B = dz; a.ldb = ld_dz; a.stride_b = dz_stride; a.M = M; a.N = N; a.K = B; a.splits = plan.splits;
        a.C = plan.splits > 1U ? partial : out; a.ldc = N; a.stride_c = out_stride;
        if (Sgemm<true, false>(st, a, groups, plan.tile) != cudaSuccess) return false;
        ++e->launches;
        if (plan.splits > 1U) sums.Planes(partial, plan.splits, (uint64_t)M * N, out, groups, out_stride);
        return ok();
    };
    StageTimer timer{e, st, profile};
    if (!timer.Start()) return MGT_CUDA_FAILURE;

    if (pad_tower) {
        Launch(PadMatricesKernel, dim3((p2 + 7U) / 8U, 2U * R), 256, 0, st, w + Fc1W(s, 0), BlockParams(s) / 2, H2, p2, base + ws.tower_w);
        ++e->launches;
    }
    if (EmbeddingForward(st, states, w, w + InputBias(s), B, L, V, H1, a1, p1, sm) != cudaSuccess) return MGT_CUDA_FAILURE;
    ++e->launches;
    if (!timer.Mark(profile ? &profile->input_forward_ms : nullptr)) return MGT_CUDA_FAILURE;
    if (!forward(a1, p1, H1, w + HiddenWeight(s), w + HiddenBias(s), nullptr, x(0))) return MGT_CUDA_FAILURE;
    if (!timer.Mark(profile ? &profile->hidden_forward_ms : nullptr)) return MGT_CUDA_FAILURE;
    if (fused) {
        TowerArgs t = tower_args;
        t.state_tape = x(0); t.inner_tape = r1(0);
        if (LaunchTower<false>(e->device, st, tower, t) != cudaSuccess) return MGT_CUDA_FAILURE;
        ++e->launches;
    }
    for (uint32_t k = 0; k < R && !fused; ++k) {
        if (!forward(x(k), p2, H2, w + Fc1W(s, k), w + Fc1B(s, k), nullptr, r1(k)) || !forward(r1(k), p2, H2, w + Fc2W(s, k), w + Fc2B(s, k), x(k), x(k + 1U))) return MGT_CUDA_FAILURE;
    }
    if (!timer.Mark(profile ? &profile->residual_forward_ms : nullptr)) return MGT_CUDA_FAILURE;
    // output layer, loss, and the masked gradient entering the tower with its column sums
    float* head_bias_dst = grad + (R > 0 ? Fc2B(s, R - 1) : HiddenBias(s));
    if (OUT == 1U) {
        const uint32_t grid = (B + 7U) / 8U < kHeadBlocks ? (B + 7U) / 8U : kHeadBlocks;
        Launch(HeadOut1Kernel, grid, kHeadThreads, 0, st, w + OutputWeight(s), w + OutputBias(s), labels, x(R), p2, B, H2, dz2(R), nullptr, 0, base + ws.head, false);
        sums.Head(base + ws.head, grid, H2, grad + OutputWeight(s), loss, head_bias_dst);
        ++e->launches;
    } else {
        const HeadArgs h{w + OutputWeight(s), OUT, w + OutputBias(s), labels, nullptr, 0, x(R), p2, B, H2, OUT, dy, nullptr, 0, dz2(R), nullptr, 0, base + ws.head, false};
        MGT_TRY(LaunchHeadN<false, true>(e, st, h, sums, loss, head_bias_dst, grad + OutputBias(s)));
        if (!weight_grad(x(R), p2, 0, H2, dy, OUT, 0, OUT, 1, base + ws.partial_out, grad + OutputWeight(s), 0)) return MGT_CUDA_FAILURE;
    }
    if (!ok()) return MGT_CUDA_FAILURE;
    MGT_TRY(sums.Pass());
    MGT_TRY(notify(OutputWeight(s), (uint64_t)H2 * OUT + OUT));
    if (!timer.Mark(profile ? &profile->output_ms : nullptr)) return MGT_CUDA_FAILURE;
    // input gradients down the tower and through the hidden layer
    if (fused) {
        TowerArgs t = tower_args;
        t.state_tape = dz2(0); t.inner_tape = dz1t(0); t.colsum = colsum; t.colsum_slot = ws.colsum_slot;
        if (LaunchTower<true>(e->device, st, tower, t) != cudaSuccess) return MGT_CUDA_FAILURE;
        ++e->launches;
    }
    for (uint32_t rb = R; rb > 0 && !fused; --rb) {
        const uint32_t k = rb - 1U;
        if (!backward(dz2(k + 1U), w + Fc2W(s, k), H2, nullptr, r1(k), p2, dz1t(k), colsum + ws.colsum_slot * k, tile_h2) ||
            !backward(dz1t(k), w + Fc1W(s, k), H2, dz2(k + 1U), x(k), p2, dz2(k), colsum + ws.colsum_slot * (R + k), tile_h2)) return MGT_CUDA_FAILURE;
    }
    // The weight gradients of all blocks, bias gradients from the column sums, and then those of the hidden layer come before the
    // table gradient: their ranges are announced as soon as they are enqueued, and a caller's exchange of them runs beside it.
    if (R > 0) {
        if (!weight_grad(r1(0), p2, bh2, H2, dz2(1), p2, bh2, H2, R, base + ws.partial_fc2, grad + Fc2W(s, 0), BlockParams(s)) ||
            !weight_grad(x(0), p2, bh2, H2, dz1t(0), p2, bh2, H2, R, base + ws.partial_fc1, grad + Fc1W(s, 0), BlockParams(s))) return MGT_CUDA_FAILURE;
        sums.TowerBiases(s, colsum, fused ? tower.tiles : rows_h2, ws.colsum_slot, grad, true);
        MGT_TRY(sums.Pass());
        for (uint32_t rb = R; rb > 0; --rb) {
            MGT_TRY(notify(Fc2W(s, rb - 1U), (uint64_t)H2 * H2 + H2));
            MGT_TRY(notify(Fc1W(s, rb - 1U), (uint64_t)H2 * H2 + H2));
        }
    }
    if (!ok() || !timer.Mark(profile ? &profile->residual_backward_ms : nullptr)) return MGT_CUDA_FAILURE;
    if (!backward(dz2(0), w + HiddenWeight(s), H1, nullptr, a1, p1, dz1, base + ws.colsum_in, tile_h1)) return MGT_CUDA_FAILURE;
    if (!weight_grad(a1, p1, 0, H1, dz2(0), p2, 0, H2, 1, base + ws.partial, grad + HiddenWeight(s), 0)) return MGT_CUDA_FAILURE;
    MGT_TRY(sums.Pass());
    MGT_TRY(notify(HiddenWeight(s), (uint64_t)H1 * H2 + H2));
    // the input-bias gradient sums the fp32 dz1 (mlp_backward.cu:1505)
    sums.Rows(base + ws.colsum_in, rows_h1, H1, H1, grad + InputBias(s));
    MGT_TRY(sums.Pass());
    if (half_ig) {
        Launch(RoundHalfKernel, GridFor((uint64_t)B * p1, 256, e->sm_count), 256, 0, st, dz1, (uint64_t)B * p1);
        ++e->launches;
    }
    if (!ok() || !timer.Mark(profile ? &profile->hidden_backward_ms : nullptr)) return MGT_CUDA_FAILURE;
    if (EmbeddingGrad(st, states, dz1, p1, B, L, V, H1, reinterpret_cast<uint32_t*>(base + ws.lists), false, grad) != cudaSuccess) return MGT_CUDA_FAILURE;
    e->launches += 2;
    MGT_TRY(sums.LaunchAll());
    MGT_TRY(notify(0, (uint64_t)L * V * H1 + H1));
    if (!timer.Mark(profile ? &profile->input_grad_ms : nullptr)) return MGT_CUDA_FAILURE;
    return MGT_OK;
}

// Whether the kernels of a step begin before those ahead of them have ended (launch.cuh): where a step is a row of short kernels.
// 4 096 samples of hd1 1024 210 -> 200 us, 5 003 of hd1 333 172 -> 157, 1 024 of hd1 256 103 -> 82; 3 001 samples of hd1 2560 make no
// difference, and with kernels that fill the chip the next one's CTAs are in the way: 9 001 samples of hd1 1000 445 -> 491, 8 192 of
// hd1 2560 in fp32 4 701 -> 5 230. The many passes of batch normalisation stream and gain at any size (53 248 of hd1 2560 5 884 -> 5 510).
bool OverlapLaunches(const mgt_mlp_shape_t& s, uint32_t B, bool batch_norm) { return batch_norm || (uint64_t)B * s.hd1 <= 6000000ULL; }
// All in fp32 the kernels have their operands through L1, and lose some of it to the shared memory of the next one, as soon as a
// product has more than one or two tiles for an SM. Counted in tiles of 32 x 32, of the products by hd1 (the input gradient) and of those
// by hd2 (the blocks): us a step without and with, by samples / hd1 / hd2 / blocks. Few tiles: 250 / 512 / 64 / 4 176 -> 153; 128 / 1000 /
// 192 / 6 373 -> 322; 1 000 / 256 / 192 / 6 400 -> 379. Too many by hd1: 256 / 1000 / 128 / 4 265 -> 292; 102 / 2500 / 192 / 6 470 -> 534;
// by hd2: 2 000 / 64 / 128 / 4 223 -> 249; 3 800 / 64 / 256 / 6 899 -> 1 099; 320 / 400 / 400 / 6 528 -> 558. A narrow hd2 leaves the chip
// emptier: 512 / 1000 / 24 / 4 173 -> 149, 1 000 / 512 / 64 / 4 193 -> 184, but 8 000 / 64 / 24 / 4 170 -> 177.
bool OverlapFp32Launches(const mgt_mlp_shape_t& s, uint32_t B) {
    auto tiles = [&](uint32_t n) { return (uint64_t)((B + 31U) / 32U) * ((n + 31U) / 32U); };
    const uint64_t by_hd1 = s.hd2 <= 32U || (s.hd2 <= 64U && s.hd1 <= 512U) ? 518U : (s.hd1 <= 512U ? 256U : 160U);
    return tiles(s.hd1) <= by_hd1 && tiles(s.hd2) <= (s.hd2 <= 320U ? 200U : 112U);
}

struct HalfWeights {
    const __half* in_table; uint32_t p1;     // [(IN+1)][p1], row IN is the input bias
    const __half* wh; uint32_t p2;            // [H1][p2]
    const __half* w1[MGT_MAX_RESIDUAL_BLOCKS];
    const __half* w2[MGT_MAX_RESIDUAL_BLOCKS];
    const __half* wout; uint32_t pout;        // [H2][pout]
};

}  // namespace
}  // namespace mgt

using namespace mgt;

extern "C" {

const char* mgt_status_name(mgt_status_t status) {
    switch (status) {
        case MGT_OK: return "ok";
        case MGT_INVALID_CONFIG: return "invalid_config";
        case MGT_INVALID_PUZZLE: return "invalid_puzzle";
        case MGT_CAPACITY_EXCEEDED: return "capacity_exceeded";
        case MGT_CUDA_FAILURE: return "cuda_failure";
        case MGT_NCCL_FAILURE: return "nccl_failure";
        case MGT_IO_FAILURE: return "io_failure";
        case MGT_DEVICE_TIMEOUT: return "device_timeout";
    }
    return "unknown";
}

const char* mgt_version(void) { return "mgt_b200 0.1 (sm_100a)"; }

mgt_status_t mgt_validate_mlp_shape(const mgt_mlp_shape_t* shape) { return ValidShape(shape) ? MGT_OK : MGT_INVALID_CONFIG; }

uint64_t mgt_mlp_param_count(const mgt_mlp_shape_t* shape) { return ValidShape(shape) ? ParamCount(*shape) : 0; }

mgt_status_t mgt_engine_create(int32_t device_id, mgt_engine_t** out_engine) {
    if (out_engine == nullptr || device_id < 0) return MGT_INVALID_CONFIG;
    *out_engine = nullptr;
    if (cudaSetDevice(device_id) != cudaSuccess) return MGT_CUDA_FAILURE;
    cudaDeviceProp prop{};
    if (cudaGetDeviceProperties(&prop, device_id) != cudaSuccess) return MGT_CUDA_FAILURE;
    if (prop.major != 10) {
        std::fprintf(stderr, "mgt_b200: device %d is sm_%d%d; this library only runs on sm_100a (B200)\n", device_id, prop.major, prop.minor);
        return MGT_CUDA_FAILURE;
    }
    auto* e = new mgt_engine();
    e->device = device_id;
    e->sm_count = prop.multiProcessorCount;
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult qres;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || fn == nullptr) {
        delete e;
        return MGT_CUDA_FAILURE;
    }
    e->encode = reinterpret_cast<EncodeTiledFn>(fn);
    if (const char* path = std::getenv("MGT_RESIDUAL_PATH")) e->layered_tower = std::strcmp(path, "layered") == 0;
    if (const char* form = std::getenv("MGT_EMBEDDING_FORM"))
        e->embedding_form = std::strcmp(form, "gather") == 0 ? mgt_engine::kGather : (std::strcmp(form, "onehot") == 0 ? mgt_engine::kOneHot : mgt_engine::kBySize);
    if (cudaMalloc(&e->status_word, sizeof(int)) != cudaSuccess || cudaMemset(e->status_word, 0, sizeof(int)) != cudaSuccess) {
        delete e;
        return MGT_CUDA_FAILURE;
    }
    *out_engine = e;
    return MGT_OK;
}

mgt_status_t mgt_engine_destroy(mgt_engine_t* e) {
    if (e == nullptr) return MGT_OK;
    if (e->ev_last) cudaEventDestroy(e->ev_last);
    if (e->ev_now) cudaEventDestroy(e->ev_now);
    for (const auto& known : e->sides) SidePool::Get().GiveBack(e->device, known.side);
    if (e->status_word) cudaFree(e->status_word);
    delete e;
    return MGT_OK;
}

uint64_t mgt_engine_launch_count(const mgt_engine_t* e) { return e == nullptr ? 0 : e->launches; }
uint64_t mgt_engine_fork_count(const mgt_engine_t* e) { return e == nullptr ? 0 : e->forks; }

mgt_status_t mgt_engine_check(mgt_engine_t* e, void* stream, int32_t* out_device_code) {
    if (e == nullptr) return MGT_INVALID_CONFIG;
    int code = 0;
    if (cudaStreamSynchronize(static_cast<cudaStream_t>(stream)) != cudaSuccess) return MGT_CUDA_FAILURE;
    if (cudaMemcpy(&code, e->status_word, sizeof(int), cudaMemcpyDeviceToHost) != cudaSuccess) return MGT_CUDA_FAILURE;
    if (out_device_code) *out_device_code = code;
    if (code != 0) {
        cudaMemset(e->status_word, 0, sizeof(int));
        return MGT_DEVICE_TIMEOUT;
    }
    return MGT_OK;
}

// The fp32 operand of the table gradient behind the tensor-core workspace: dz1 [samples][hd1], rows padded to four floats,
// then the sample lists of its classes (and slack: to align the start, and for the rounding of what the 16-bit gradient plans
// instead, so that scratch of this size does for either).
static uint64_t Fp32TableFloats(const mgt_mlp_shape_t& s, uint32_t B) {
    return (uint64_t)B * RoundUp(s.hd1, 4) + gather::ListWords(B, s.state_len, s.state_value_pad) + 64 + 512;
}

static uint64_t WorkspaceFloats(const mgt_mlp_shape_t* shape, uint32_t sample_count, uint32_t chunks, int32_t use_half_input_grad, int32_t use_half_linear,
                                bool batch_norm) {
    if (!ValidShape(shape) || sample_count == 0 || chunks == 0) return 0;
    if (!use_half_linear) return batch_norm ? 0 : Fp32WorkspaceFloats(*shape, sample_count, CurrentDeviceSmCount());
    const Workspace w = PlanWorkspace(*shape, sample_count, CurrentDeviceSmCount(), use_half_input_grad != 0, batch_norm);
    return (w.total_bytes + 3) / 4 + (use_half_input_grad ? 0 : Fp32TableFloats(*shape, sample_count));
}

uint64_t mgt_mlp_loss_grad_workspace_floats(const mgt_mlp_shape_t* shape, uint32_t sample_count, uint32_t chunks,
                                            int32_t use_half_input_grad, int32_t use_half_linear) {
    return WorkspaceFloats(shape, sample_count, chunks, use_half_input_grad, use_half_linear, false);
}

uint64_t mgt_mlp_loss_grad_workspace_floats_with_options(const mgt_mlp_shape_t* shape, uint32_t sample_count, uint32_t chunks, int32_t use_half_input_grad,
                                                         int32_t use_half_linear, const mgt_train_options_t* options) {
    return WorkspaceFloats(shape, sample_count, chunks, use_half_input_grad, use_half_linear, options != nullptr && options->batch_norm != 0);
}

uint64_t mgt_bn_param_count(const mgt_mlp_shape_t* shape) { return ValidShape(shape) ? 2ULL * (shape->residual_blocks + 1ULL) * shape->hd2 : 0; }

mgt_status_t mgt_engine_set_batch_norm_state(mgt_engine_t* e, float* device_running_stats, float momentum, uint32_t world_size, float* device_exchange_buffer,
                                             mgt_stats_exchange_fn exchange, void* user) {
    if (e == nullptr || !(momentum >= 0.0f && momentum <= 1.0f) || world_size == 0) return MGT_INVALID_CONFIG;
    if ((exchange != nullptr) != (device_exchange_buffer != nullptr)) return MGT_INVALID_CONFIG;
    e->bn_running = device_running_stats;
    e->bn_momentum = momentum;
    e->bn_world = world_size;
    e->bn_exchange_buffer = device_exchange_buffer;
    e->bn_exchange = exchange;
    e->bn_exchange_user = user;
    return MGT_OK;
}

mgt_status_t mgt_launch_mlp_loss_grad(mgt_engine_t* e, const mgt_mlp_shape_t* shape, const float* w, const uint16_t* w_half_u16,
                                      const mgt_train_state_t* states, const float* labels, uint32_t B, float* loss, float* grad,
                                      float* workspace, uint64_t workspace_floats, uint32_t chunks, uint32_t ppb, int32_t half_ig,
                                      int32_t half_lin, mgt_backward_profile_t* profile, mgt_gradient_ready_fn ready, void* ready_user,
                                      void* stream_v, uint32_t position_tile) {
    (void)position_tile;
    if (e == nullptr || !ValidShape(shape) || w == nullptr || states == nullptr || labels == nullptr || loss == nullptr || grad == nullptr ||
        B == 0 || workspace == nullptr || chunks == 0 || ppb == 0) {
        return MGT_INVALID_CONFIG;
    }
    const mgt_mlp_shape_t s = *shape;
    const bool bnorm = e->options.batch_norm != 0;
    const bool options_set = e->options.operand_format != MGT_OPERAND_FP16 || e->options.loss_kind != MGT_LOSS_MSE || bnorm;
    if (options_set && !half_lin) return MGT_INVALID_CONFIG;  // the options belong to the tensor-core data flow
    if (e->options.loss_kind == MGT_LOSS_CROSS_ENTROPY && s.output_dim < 2U) return MGT_INVALID_CONFIG;
    struct FormatScope {  // the operand format applies to the kernels enqueued by this call only
        mgt_engine* e;
        ~FormatScope() { e->bf16_now = false; }
    } format_scope{e};
    e->bf16_now = half_lin && e->options.operand_format == MGT_OPERAND_BF16;
    if (!half_lin) {
        // fp32 linear layers: the CUDA-core path (fp32_path.cuh); half_ig only selects the rounding of its embedding-gradient operand
        if (workspace_floats < Fp32WorkspaceFloats(s, B, PlanSmCount(e->sm_count))) return MGT_CAPACITY_EXCEEDED;
        uint32_t id = 0;
        auto tell = [&](uint64_t off, uint64_t count) -> mgt_status_t {
            if (ready == nullptr) return MGT_OK;
            return ready(ready_user, id++, off, count, stream_v) == MGT_OK ? MGT_OK : MGT_CUDA_FAILURE;
        };
        return LaunchFp32Path(e, s, w, reinterpret_cast<const uint8_t*>(states), labels, B, loss, grad, workspace, half_ig != 0, ready != nullptr || profile != nullptr, profile, tell,
                              {static_cast<cudaStream_t>(stream_v), OverlapFp32Launches(s, B)});
    }
    Workspace ws = PlanWorkspace(s, B, PlanSmCount(e->sm_count), half_ig != 0, bnorm);
    if (e->embedding_form != mgt_engine::kBySize) ws.gather_fwd = ws.gather_grad = e->embedding_form == mgt_engine::kGather;
    if (workspace_floats < (ws.total_bytes + 3) / 4 + (half_ig ? 0 : Fp32TableFloats(s, B))) return MGT_CAPACITY_EXCEEDED;
    const LaunchOn st(static_cast<cudaStream_t>(stream_v), OverlapLaunches(s, B, bnorm));
    uint8_t* base = reinterpret_cast<uint8_t*>(RoundUp(reinterpret_cast<uintptr_t>(workspace), 1024));
    float* dz1_f32 = reinterpret_cast<float*>(RoundUp(reinterpret_cast<uintptr_t>(workspace + (ws.total_bytes + 3) / 4), 256));  // behind the tensor-core workspace
    const uint32_t p_dz1_f32 = (uint32_t)RoundUp(s.hd1, 4);
    __half* a1_h = reinterpret_cast<__half*>(base + ws.off_a1);
    auto x_h = [&](uint32_t k) { return reinterpret_cast<__half*>(base + ws.off_x + ws.x_stride * k); };
    auto r1_h = [&](uint32_t k) { return reinterpret_cast<__half*>(base + ws.off_r1 + ws.r1_stride * k); };
    float* x_f32 = reinterpret_cast<float*>(base + ws.off_xf);
    float* dzf = reinterpret_cast<float*>(base + ws.off_dzf);
    auto dz_tape = [&](uint32_t k) { return reinterpret_cast<__half*>(base + ws.off_dz2 + ws.dz_stride * k); };   // [0] hidden, [k+1] fc2 of block k
    auto dz1_tape = [&](uint32_t k) { return reinterpret_cast<__half*>(base + ws.off_dz1t + ws.dz_stride * k); };  // fc1 of block k
    __half* dz1_h = reinterpret_cast<__half*>(base + ws.off_dz1);
    float* head_partial = reinterpret_cast<float*>(base + ws.off_head);
    float* colsum = reinterpret_cast<float*>(base + ws.off_colsum);
    const uint32_t H1 = s.hd1, H2 = s.hd2, R = s.residual_blocks, OUT = s.output_dim, IN = ws.IN;

    StageTimer timer{e, st, profile};
    if (!timer.Start()) return MGT_CUDA_FAILURE;
    // Nothing in the step waits for the sums over partial results: they are a launch at its end.
    const bool told = ready != nullptr || e->early_fn != nullptr || profile != nullptr;
    Sums sums{e, told, st};
    uint32_t ready_id = 0;
    auto notify = [&](uint64_t off, uint64_t count) -> mgt_status_t {
        if (ready == nullptr) return MGT_OK;
        const mgt_status_t r = ready(ready_user, ready_id++, off, count, stream_v);
        return r == MGT_OK ? MGT_OK : MGT_CUDA_FAILURE;  // the reference maps a failing callback to kCudaFailure
    };

    // ---- batch normalisation (opt-in): fp32 pre-activations z of every normalised layer are kept, layer 0 = hidden
    // layer, layer k + 1 = fc2 of block k; gamma/beta and their gradients follow the reference's parameters
    const uint64_t bn_base = ParamCount(s);
    auto z_tape = [&](uint32_t layer) { return reinterpret_cast<float*>(base + ws.off_bn_z + ws.bn_z_stride * layer); };
    auto bn_mean = [&](uint32_t layer) { return reinterpret_cast<float*>(base + ws.off_bn_save) + 2ULL * layer * H2; };
    auto bn_rstd = [&](uint32_t layer) { return bn_mean(layer) + H2; };
    float* bn_partial = reinterpret_cast<float*>(base + ws.off_bn_partial);
    auto bn_bias = [&](uint32_t layer) { return reinterpret_cast<float*>(base + ws.off_bn_bias) + (uint64_t)layer * bn::kMaxBlocks * H2; };  // partial sums of a bias gradient
    float* bn_stats = bnorm && e->bn_exchange_buffer != nullptr ? e->bn_exchange_buffer : reinterpret_cast<float*>(base + ws.off_bn_stats);
    const uint32_t bn_blocks = bn::BlocksFor(B, e->sm_count);
    const uint32_t bn_reduce_grid = (H2 + bn::kReduceCols - 1U) / bn::kReduceCols, bn_reduce_threads = bn::kReduceCols * bn::kReduceParts;
    auto bn_exchange = [&]() -> mgt_status_t {
        if (e->bn_exchange == nullptr) return MGT_OK;
        return e->bn_exchange(e->bn_exchange_user, bn_stats, 2ULL * H2, stream_v) == MGT_OK ? MGT_OK : MGT_CUDA_FAILURE;
    };
    // Widths of one tile: the GEMM that makes z leaves its column moments too, as four rows of partial sums a CTA. As a kernel of its
    // own they read z again: p888 at 53 248 samples 5 485 -> 5 415 us a step. (The moments of the backward pass in the epilogue of
    // the product before them as well: it needs z there, and 5 485 us again.)
    const uint32_t bn_rows = 4U * std::min((B + 127U) / 128U, (uint32_t)e->sm_count);
    const bool bn_fused = H2 <= 256U && bn_rows <= bn::kMaxBlocks;
    // z_tape(layer) -> x_f32 / x_h(layer): x = relu(bn(z)) for the hidden layer, relu(x + bn(z)) for a block
    auto bn_forward = [&](uint32_t layer) -> mgt_status_t {
        if (!bn_fused) Launch(bn::ColumnMomentsKernel<false>, bn_blocks, bn::kThreads, 0, st, z_tape(layer), ws.p_f32, nullptr, 0, nullptr, nullptr, B, H2, bn_partial);
        Launch(bn::ReduceMomentsKernel, bn_reduce_grid, bn_reduce_threads, 0, st, bn_partial, bn_fused ? bn_rows : bn_blocks, H2, 1.0f / (float)B, bn_stats, nullptr, nullptr);
        MGT_TRY(bn_exchange());
        const float* gamma = w + bn_base + 2ULL * layer * H2;
        float* running = e->bn_running != nullptr ? e->bn_running + 2ULL * layer * H2 : nullptr;
        const double n = (double)B * e->bn_world;
        const float unbias = n > 1.0 ? (float)(n / (n - 1.0)) : 1.0f;
        uint16_t* xh = reinterpret_cast<uint16_t*>(x_h(layer));
        if (layer == 0U) {
            Launch(bn::ApplyForwardKernel<false>, bn_blocks, bn::kThreads, 0, st, z_tape(layer), ws.p_f32, bn_stats, gamma, gamma + H2, e->options.bn_eps, B, H2, x_f32,
                                                                             ws.p_f32, xh, ws.p_act, e->bf16_now, bn_mean(layer), bn_rstd(layer), running,
                                                                             e->bn_momentum, unbias);
        } else {
            Launch(bn::ApplyForwardKernel<true>, bn_blocks, bn::kThreads, 0, st, z_tape(layer), ws.p_f32, bn_stats, gamma, gamma + H2, e->options.bn_eps, B, H2, x_f32,
                                                                            ws.p_f32, xh, ws.p_act, e->bf16_now, bn_mean(layer), bn_rstd(layer), running,
                                                                            e->bn_momentum, unbias);
        }
        e->launches += bn_fused ? 2 : 3;
        return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
    };
    // dzf (gradient w.r.t. the sum entering the ReLU above the layer) -> dz_tape(layer) = gradient w.r.t. z, plus the
    // gradients of gamma, beta and of the bias inside z
    auto bn_backward = [&](uint32_t layer) -> mgt_status_t {
        Launch(bn::ColumnMomentsKernel<true>, bn_blocks, bn::kThreads, 0, st, dzf, ws.p_f32, z_tape(layer), ws.p_f32, bn_mean(layer), bn_rstd(layer), B, H2, bn_partial);
        float* dgamma = grad + bn_base + 2ULL * layer * H2;
        Launch(bn::ReduceMomentsKernel, bn_reduce_grid, bn_reduce_threads, 0, st, bn_partial, bn_blocks, H2, 1.0f / (float)B, bn_stats, dgamma + H2, dgamma);
        MGT_TRY(bn_exchange());
        Launch(bn::ApplyBackwardKernel, bn_blocks, bn::kThreads, 0, st, dzf, ws.p_f32, z_tape(layer), ws.p_f32, bn_mean(layer), bn_rstd(layer), w + bn_base + 2ULL * layer * H2,
                                                                    bn_stats, B, H2, reinterpret_cast<uint16_t*>(dz_tape(layer)), ws.p_dz, e->bf16_now, bn_bias(layer));
        e->launches += 3;
        return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
    };

    // ---- fp16 weights: the caller's mirror as it lies when TMA can address it, else a padded copy
    HalfWeights hw{};
    const __half* w_half = reinterpret_cast<const __half*>(w_half_u16);
    // (the caller's mirror is fp16 by contract: with bfloat16 operands the copy is rebuilt from the fp32 weights each call)
    const bool direct = w_half != nullptr && !e->bf16_now && (H1 % 8U) == 0 && (H2 % 8U) == 0 && (reinterpret_cast<uintptr_t>(w_half) & 15U) == 0;
    if (direct) {
        hw.in_table = w_half; hw.p1 = H1;
        hw.wh = w_half + HiddenWeight(s); hw.p2 = H2;
        for (uint32_t k = 0; k < R; ++k) { hw.w1[k] = w_half + Fc1W(s, k); hw.w2[k] = w_half + Fc2W(s, k); }
        hw.wout = w_half + OutputWeight(s); hw.pout = OUT;
    } else {
        uint64_t cur = 0;
        RepackPlan plan{};
        auto repack = [&](uint64_t src_off, uint32_t rows, uint32_t cols, uint32_t pitch) -> const __half* {
            const uint32_t i = plan.count++;
            plan.src_off[i] = src_off; plan.dst_off[i] = cur; plan.cols[i] = cols; plan.units[i] = pitch / 8U;
            plan.unit_begin[i + 1] = plan.unit_begin[i] + (uint64_t)rows * plan.units[i];
            const __half* dst = reinterpret_cast<const __half*>(base + ws.off_wint + cur);
            cur += RoundUp((uint64_t)rows * pitch * 2, 1024);
            return dst;
        };
        hw.p1 = ws.p_w1; hw.p2 = ws.p_w2; hw.pout = ws.p_wout;
        hw.in_table = repack(0, IN + 1, H1, ws.p_w1);
        hw.wh = repack(HiddenWeight(s), H1, H2, ws.p_w2);
        for (uint32_t k = 0; k < R; ++k) {
            hw.w1[k] = repack(Fc1W(s, k), H2, H2, ws.p_w2);
            hw.w2[k] = repack(Fc2W(s, k), H2, H2, ws.p_w2);
        }
        hw.wout = repack(OutputWeight(s), H2, OUT, ws.p_wout);
        Launch(RepackHalfKernel, GridFor(plan.unit_begin[plan.count], 256, e->sm_count), 256, 0, st, w, base + ws.off_wint, plan, e->bf16_now);
        ++e->launches;
        if (cudaGetLastError() != cudaSuccess) return MGT_CUDA_FAILURE;
    }

    // ---- embedding forward: a1 = relu([onehot | 1] * [W_in ; b_in])  (mlp_backward.cu:755-832)
    if (ws.gather_fwd) {
        auto run = [&](auto kernel) {
            Launch(kernel, dim3((B + 31U) / 32U, (H1 + 63U) / 64U), 256 * gather::kForwardSplit, 0, st, reinterpret_cast<const uint8_t*>(states), reinterpret_cast<const uint16_t*>(hw.in_table), hw.p1, B, s.state_len, s.state_value_pad, H1,
                reinterpret_cast<uint16_t*>(a1_h), ws.p_bt, reinterpret_cast<uint32_t*>(base + ws.off_bits_h1), ws.ld_bits_h1);
        };
        if (e->bf16_now) run(gather::ForwardKernel<gather::kForwardSplit, true>); else run(gather::ForwardKernel<gather::kForwardSplit, false>);
        ++e->launches;
        if (cudaGetLastError() != cudaSuccess) return MGT_CUDA_FAILURE;
    } else {
        PairArgs a{};
        a.M = H1; a.N = B; a.K = IN + 1U; a.k_chunks = (IN + 64U) / 64U;
        const PairPlan plan = PlanPairForward(s, B, (uint32_t)e->sm_count);
        a.row_len = plan.row_len; a.line = plan.line; a.workers = plan.workers;
        a.out_f16 = a1_h; a.ld_f16 = ws.p_bt;
        a.bits = reinterpret_cast<uint32_t*>(base + ws.off_bits_h1); a.ld_bits = ws.ld_bits_h1;
        a.states = reinterpret_cast<const uint8_t*>(states); a.state_len = s.state_len; a.value_pad = s.state_value_pad; a.samples = B; a.in_rows = IN;
        CUtensorMap ta, to;
        MGT_MAP(e->Map(&ta, hw.in_table, H1, IN + 1, hw.p1, 64, 64));
        MGT_MAP(e->Map(&to, a1_h, B, H1, ws.p_bt, 32, 32, CU_TENSOR_MAP_SWIZZLE_64B));
        MGT_TRY(LaunchPair<false>(e, ta, to, a, st));
    }
    if (!timer.Mark(profile ? &profile->input_forward_ms : nullptr)) return MGT_CUDA_FAILURE;

    // ---- hidden layer: x0 = relu(a1 * Wh + bh)  (mlp_backward.cu:1281-1291)
    {
        GemmArgs epi{};
        epi.bias = w + HiddenBias(s); epi.out_f32 = x_f32; epi.ld_f32 = ws.p_f32; epi.out_f16 = x_h(0); epi.ld_f16 = ws.p_act;
        if (bnorm) {
            epi.out_f32 = z_tape(0);
            epi.moments = bn_partial;
            MGT_TRY(bn_fused ? GemmForwardRows<Epi::kBiasF32Moments>(e, st, a1_h, ws.p_bt, hw.wh, hw.p2, B, H2, H1, epi)
                             : GemmForwardRows<Epi::kBiasF32>(e, st, a1_h, ws.p_bt, hw.wh, hw.p2, B, H2, H1, epi));
            MGT_TRY(bn_forward(0));
        } else {
            MGT_TRY(GemmForwardRows<Epi::kBiasReluF32F16>(e, st, a1_h, ws.p_bt, hw.wh, hw.p2, B, H2, H1, epi));
        }
    }
    if (!timer.Mark(profile ? &profile->hidden_forward_ms : nullptr)) return MGT_CUDA_FAILURE;

    // ---- residual blocks forward (mlp_backward.cu:1294-1323)
    const bool chain = ChainEligible(e, s) && !bnorm;  // batch statistics need the whole batch between two layers: one kernel per layer
    const uint64_t w_layer_stride = R > 0 ? (uint64_t)(reinterpret_cast<const uint8_t*>(hw.w2[0]) - reinterpret_cast<const uint8_t*>(hw.w1[0])) : 16;
    ChainArgs ca{};
    ca.samples = B; ca.H = H2; ca.R = R; ca.tiles = (B + 127U) / 128U;
    ca.ld_f32 = ws.p_f32;
    ca.bits_s = reinterpret_cast<uint32_t*>(base + ws.off_bits);
    ca.bits_t = ca.bits_s + ws.bits_stride * (R + 1);
    ca.bits_stride = ws.bits_stride;
    if (chain) {
        ChainArgs f = ca;
        f.state_f32 = x_f32;
        f.bias = w + Fc1B(s, 0); f.bias_stride = (uint64_t)H2 * H2 + H2;
        f.tape_s = x_h(0); f.tape_s_stride = ws.x_stride / 2; f.ld_s = ws.p_act;
        f.tape_t = r1_h(0); f.tape_t_stride = ws.r1_stride / 2; f.ld_t = ws.p_act;
        MGT_TRY(LaunchChain<false>(e, st, hw.w1[0], hw.p2, w_layer_stride, R + 1, R, f));
    }
    for (uint32_t k = 0; k < R && !chain; ++k) {
        GemmArgs e1{};
        e1.bias = w + Fc1B(s, k); e1.out_f16 = r1_h(k); e1.ld_f16 = ws.p_act;
        MGT_TRY(GemmForward<Epi::kBiasReluF16>(e, st, x_h(k), ws.p_act, hw.w1[k], hw.p2, B, H2, H2, e1));
        GemmArgs e2{};
        e2.bias = w + Fc2B(s, k); e2.add_f32 = x_f32; e2.ld_add = ws.p_f32; e2.out_f32 = x_f32; e2.ld_f32 = ws.p_f32;
        e2.out_f16 = x_h(k + 1); e2.ld_f16 = ws.p_act;
        if (bnorm) {
            e2.out_f32 = z_tape(k + 1U);
            e2.moments = bn_partial;
            MGT_TRY(bn_fused ? GemmForward<Epi::kBiasF32Moments>(e, st, r1_h(k), ws.p_act, hw.w2[k], hw.p2, B, H2, H2, e2)
                             : GemmForward<Epi::kBiasF32>(e, st, r1_h(k), ws.p_act, hw.w2[k], hw.p2, B, H2, H2, e2));
            MGT_TRY(bn_forward(k + 1U));
            continue;
        }
        MGT_TRY(GemmForward<Epi::kBiasResReluF32F16>(e, st, r1_h(k), ws.p_act, hw.w2[k], hw.p2, B, H2, H2, e2));
    }
    if (!timer.Mark(profile ? &profile->residual_forward_ms : nullptr)) return MGT_CUDA_FAILURE;

    // ---- output head, loss and the gradient entering the last block (mlp_backward.cu:1327-1364)
    __half* dz_cur = dz_tape(R);   // fp16 copy of the gradient w.r.t. the pre-activation the head feeds
    // the head also yields the fp32 column sums of dz: the bias gradient of the layer below it, unless that is normalised
    float* head_bias_dst = bnorm ? nullptr : grad + (R > 0 ? Fc2B(s, R - 1) : HiddenBias(s));
    if (OUT == 1U) {
        Launch(HeadOut1Kernel, kHeadBlocks, kHeadThreads, 0, st, w + OutputWeight(s), w + OutputBias(s), labels, x_f32, ws.p_f32, B, H2, dzf, dz_cur, ws.p_dz, head_partial, e->bf16_now);
        sums.Head(head_partial, kHeadBlocks, H2, grad + OutputWeight(s), loss, head_bias_dst);
        ++e->launches;
    } else {
        float* dy = reinterpret_cast<float*>(base + ws.off_dy);
        __half* dy_h = reinterpret_cast<__half*>(base + ws.off_dyh);
        const HeadArgs h{hw.wout, hw.pout, w + OutputBias(s), labels, x_h(R), ws.p_act, x_f32, ws.p_f32, B, H2, OUT, dy, dy_h, ws.p_wout, dzf, dz_cur, ws.p_dz, head_partial, e->bf16_now};
        MGT_TRY(e->options.loss_kind == MGT_LOSS_CROSS_ENTROPY ? LaunchHeadN<true, false>(e, st, h, sums, loss, head_bias_dst, grad + OutputBias(s))
                                                               : LaunchHeadN<false, false>(e, st, h, sums, loss, head_bias_dst, grad + OutputBias(s)));
        // grad W_out = x_R^T * dy (16-bit operands, fp32 accumulate, mlp_backward.cu:1349-1354): the split-K weight-gradient GEMM
        MGT_TRY(GemmGradWeights(e, st, x_h(R), ws.p_act, dy_h, ws.p_wout, B, H2, OUT, reinterpret_cast<float*>(base + ws.off_partial_out), sums, grad + OutputWeight(s)));
    }
    if (cudaGetLastError() != cudaSuccess) return MGT_CUDA_FAILURE;
    MGT_TRY(sums.Pass());
    MGT_TRY(notify(OutputWeight(s), (uint64_t)H2 * OUT + OUT));
    if (!timer.Mark(profile ? &profile->output_ms : nullptr)) return MGT_CUDA_FAILURE;

    // ---- residual blocks backward (mlp_backward.cu:1367-1413). First the chain of input-gradient GEMMs,
    // block R-1 down to 0; every dz tensor is kept. dzf holds the running fp32 gradient (skip connection).
    const uint32_t dx_rows = PlanBackprop(e, B, H2, H2).rows;
    if (R > 0 && !chain && cudaMemsetAsync(colsum, 0, ws.colsum_floats * sizeof(float), st) != cudaSuccess) return MGT_CUDA_FAILURE;
    uint32_t colsum_rows = dx_rows;
    if (chain) {
        ChainArgs b = ca;
        b.state_f32 = dzf;
        b.tape_s = dz_tape(0); b.tape_s_stride = ws.dz_stride / 2; b.ld_s = ws.p_dz;
        b.tape_t = dz1_tape(0); b.tape_t_stride = ws.dz_stride / 2; b.ld_t = ws.p_dz;
        b.colsum = colsum; b.colsum_stride = ws.colsum_slot_floats;
        MGT_TRY(LaunchChain<true>(e, st, hw.w1[0], hw.p2, w_layer_stride, R + 1, R, b));
        colsum_rows = ca.tiles * 4U;
    }
    for (uint32_t rb = R; rb > 0 && !chain; --rb) {
        const uint32_t k = rb - 1U;
        if (bnorm) MGT_TRY(bn_backward(k + 1U));  // dz_tape(k + 1) = gradient w.r.t. the fc2 output; dzf goes down the skip path as it is
        GemmArgs d2{};  // dz1 = (dz2 * W2^T) * [r1 > 0]
        d2.mask = r1_h(k); d2.ld_mask = ws.p_act; d2.out_f16 = dz1_tape(k); d2.ld_f16 = ws.p_dz;
        MGT_TRY(GemmBackpropInput<Epi::kMaskF16>(e, st, dz_tape(k + 1), ws.p_dz, hw.w2[k], hw.p2, B, H2, H2, d2, colsum + ws.colsum_slot_floats * k));
        GemmArgs d1{};  // next dz = (dz1 * W1^T + dz2) * [x_k > 0]: ReLU of the previous block (or of the hidden layer)
        d1.add_f32 = dzf; d1.ld_add = ws.p_f32; d1.out_f32 = dzf; d1.ld_f32 = ws.p_f32; d1.mask = x_h(k); d1.ld_mask = ws.p_act;
        d1.out_f16 = dz_tape(k); d1.ld_f16 = ws.p_dz;
        MGT_TRY(GemmBackpropInput<Epi::kAddMaskF32F16>(e, st, dz1_tape(k), ws.p_dz, hw.w1[k], hw.p2, B, H2, H2, d1, colsum + ws.colsum_slot_floats * (R + k)));
    }
    if (!timer.Mark(profile ? &profile->residual_backward_ms : nullptr)) return MGT_CUDA_FAILURE;

    // Order of what follows: the dX GEMMs run first, down to the embedding gradient; the weight-gradient GEMMs of the tower
    // and of the hidden layer (which only read tapes) come last. The embedding table is 86 % of the parameters: this way
    // its gradient is complete - and the early-range hook can hand it to the exchange - while a third of a millisecond
    // of weight-gradient work is still to run. The gradient-ready notifications keep the reference's order.

    // ---- hidden layer backward, dX part (mlp_backward.cu:1417-1438): dz_tape(0) = dcur * [x0 > 0]
    dz_cur = dz_tape(0);
    if (bnorm) {
        MGT_TRY(bn_backward(0));
        // the gradients of the biases in front of the normalisations, of all layers
        sums.Rows(bn_bias(0), bn_blocks, H2, H2, grad + HiddenBias(s));
        sums.Rows(bn_bias(1), bn_blocks, H2, H2, grad + Fc2B(s, 0), R, (uint64_t)bn::kMaxBlocks * H2, BlockParams(s));
        MGT_TRY(sums.Pass());
    }
    // Small batches: the weight gradients run beside the dX products and the embedding gradient, on the second stream. Neither
    // branch fills the SMs there (the dX product has fewer than two tiles an SM), and every launch is a gap: 9 001 samples of
    // hd1 1000, hd2 200, 8 blocks 510 -> 453 us a step, 1 024 of hd1 256, hd2 64, 2 blocks 91 -> 82. With more tiles each kernel has the
    // whole chip anyway, and beyond some 16 000 samples of a small model the gradient's gathers lose more to the shared memory of the
    // GEMMs beside them than they gain (54 025 of hd1 88: 611 -> 660 us).
    // The fork is six calls more for the host, which bounds the shortest steps: whatever runs beside what, they take 61 to 66 us with it
    // (by host). So not where the chain of kernels is shorter than that. It grows with the blocks and, from some thousand samples x hd1
    // on, with the embedding layer; without and with the fork, samples / hd1 / hd2: no blocks 500 / 64 / 16 51, 57; one 64 / 8 / 8 60, 66,
    // 300 / 16 / 16 65, 66, 64 / 256 / 16 67, 66, 1 000 / 32 / 16 70, 66; two 64 / 8 / 16 61, 67, 64 / 64 / 16 67, 62, 256 / 8 / 16 69, 62,
    // 1 024 / 56 / 16 76, 66; four 64 / 8 / 64 71, 66, 256 / 64 / 64 84, 76, 3 000 / 16 / 64 96, 87; 24 256 / 8 / 256 427, 415.
    // Not with callers that are told of finished ranges or time the stages: they rely on the order.
    const uint64_t dx_tiles = (uint64_t)((H1 + 127U) / 128U) * ((B + 255U) / 256U);
    constexpr uint64_t kLeast[] = {65536U, 16384U, 2048U, 0U};  // samples x hd1, by the number of blocks
    SideBranch branch{e, st};
    if (dx_tiles < 2ULL * e->sm_count && B <= 16384U && (uint64_t)B * H1 >= kLeast[std::min(R, 3U)] && !told) branch.Fork();
    const LaunchOn st_dw(branch.open ? branch.side.stream : st.stream, st.overlap);
    uint32_t* order = half_ig ? reinterpret_cast<uint32_t*>(base + ws.off_lists) : reinterpret_cast<uint32_t*>(dz1_f32 + (uint64_t)B * p_dz1_f32);
    uint32_t* first = order + (uint64_t)s.state_len * B;
    auto sort_classes = [&](LaunchOn stream) {
        Launch(gather::SortByClassKernel, s.state_len, 1024, 0, stream, reinterpret_cast<const uint8_t*>(states), B, s.state_value_pad, order, first);
        ++e->launches;
    };
    // The sort of a gathered table gradient goes first on the second stream. Behind the dX product it finds no room beside the weight
    // gradients there (registers), and the table gradient waits for them: fp32 table, 2 blocks, samples / hd1 / hd2 16 384 / 64 / 32 184 us
    // a step on one stream's order, 210 with launches that overlap, 180 like this; 6 000 / 256 / 96 172, 166, 150. With longer gathers, which leave
    // the weight gradients no room in turn, it costs more than it saves: 10 000 / 512 / 200, 6 blocks 364 -> 387; 16 384 / 512 / 96 352 -> 392.
    const bool sort_aside = branch.open && (half_ig ? ws.gather_grad : H1 <= 256U || (H1 <= 512U && B <= 4096U));
    if (sort_aside) sort_classes(st_dw);
    sums.on = st_dw;
    Sums own{e, true, st};  // (the sums that wait are launched on the second stream, which does not see the dX product)
    Sums& dx_sums = branch.open ? own : sums;
    // dz1T = (Wh * dzh^T) * [pre-activation of a1 > 0], the input-bias gradient from its row sums. With --input-grad-fp16 0 the
    // embedding gradient wants dz1 in fp32 (mlp_backward.cu:1433-1504, float one-hot GEMM): the same product of fp16 operands
    // with fp32 accumulation, written unrounded as rows of samples.
    MGT_TRY(GemmBackpropInputRows(e, st, hw.wh, hw.p2, dz_cur, ws.p_dz, B, H1, H2, reinterpret_cast<uint32_t*>(base + ws.off_bits_h1), ws.ld_bits_h1, dz1_h,
                                  ws.p_bt, half_ig ? nullptr : dz1_f32, p_dz1_f32, half_ig && ws.gather_grad, ws.p_dz1_rows, reinterpret_cast<float*>(base + ws.off_rowsum), ws.rowsum_rows, dx_sums, grad + InputBias(s)));
    MGT_TRY(dx_sums.Pass());
    if (!timer.Mark(profile ? &profile->hidden_backward_ms : nullptr)) return MGT_CUDA_FAILURE;

    // ---- embedding gradient: grad W_in = onehot^T * dz1  (mlp_backward.cu:1440-1504); the input-bias
    // gradient (mlp_backward.cu:1505) is the column sum written by the GEMM above
    if (sort_aside && !branch.Tie(1, branch.side.stream, st)) return MGT_CUDA_FAILURE;  // (of the branch only the sort is enqueued yet)
    if (!half_ig) {
        if (fp32path::EmbeddingGrad(st, reinterpret_cast<const uint8_t*>(states), dz1_f32, p_dz1_f32, B, s.state_len, s.state_value_pad, H1,
                                    order, sort_aside, grad) != cudaSuccess) return MGT_CUDA_FAILURE;
        e->launches += sort_aside ? 1 : 2;
    } else if (ws.gather_grad) {
        const bool vec = (H1 & 3U) == 0U && (reinterpret_cast<uintptr_t>(grad) & 15U) == 0U;
        auto run = [&](auto kernel, uint32_t rows_per_cta) {
            Launch(kernel, dim3((IN + rows_per_cta - 1U) / rows_per_cta, (H1 + 63U) / 64U), 256, 0, st, order, first, reinterpret_cast<const uint16_t*>(dz1_h), ws.p_dz1_rows, B,
                                                                                               s.state_len, s.state_value_pad, H1, grad, vec);
        };
        if (!sort_aside) sort_classes(st);
        // a group of lanes per table row, four groups where that leaves fewer than 16 warps for an SM
        const bool few = (uint64_t)IN * ((H1 + 63U) / 64U) < 64ULL * e->sm_count;
        if (few) { if (e->bf16_now) run(gather::GradKernel<4, true>, 8U); else run(gather::GradKernel<4, false>, 8U); }
        else { if (e->bf16_now) run(gather::GradKernel<1, true>, 32U); else run(gather::GradKernel<1, false>, 32U); }
        ++e->launches;
        if (cudaGetLastError() != cudaSuccess) return MGT_CUDA_FAILURE;
    } else {
        PairArgs a{};
        a.M = H1; a.N = IN; a.K = B; a.k_chunks = (B + 63U) / 64U;
        const PairPlan plan = PlanPairGrad(s, B, (uint32_t)e->sm_count);
        a.n_tiles = plan.n_tiles; a.tile_cols = plan.tile_cols; a.workers = plan.workers; a.line = plan.line;
        a.out_f32 = grad; a.ld_f32 = H1;
        a.states = reinterpret_cast<const uint8_t*>(states); a.state_len = s.state_len; a.value_pad = s.state_value_pad; a.samples = B;
        if (plan.shared_tiles && cudaMemsetAsync(grad, 0, (uint64_t)IN * H1 * sizeof(float), st) != cudaSuccess) return MGT_CUDA_FAILURE;
        CUtensorMap ta;
        MGT_MAP(e->Map(&ta, dz1_h, B, H1, ws.p_bt, 64, 128));
        MGT_TRY(LaunchPair<true>(e, ta, ta, a, st));
    }
    // table and input bias are complete: tell a caller who asked to hear of it before the weight-gradient GEMMs are enqueued
    if (e->early_fn != nullptr && e->early_fn(e->early_user, 2U * R + 2U, 0, InputBias(s) + H1, stream_v) != MGT_OK) return MGT_CUDA_FAILURE;
    if (!timer.Mark(profile ? &profile->input_grad_ms : nullptr)) return MGT_CUDA_FAILURE;

    if (R > 0) {
        // weight gradients of all blocks: two grouped split-K GEMMs (fc2: r1_k^T dz2_k, fc1: x_k^T dz1_k)
        MGT_TRY(GemmGradWeightsGrouped(e, st_dw, r1_h(0), ws.p_act, ws.r1_stride, dz_tape(1), ws.p_dz, ws.dz_stride, R, B, H2, H2,
                                       reinterpret_cast<float*>(base + ws.off_partial_fc2), sums, grad + Fc2W(s, 0), BlockParams(s)));
        MGT_TRY(sums.Pass());
        MGT_TRY(GemmGradWeightsGrouped(e, st_dw, x_h(0), ws.p_act, ws.x_stride, dz1_tape(0), ws.p_dz, ws.dz_stride, R, B, H2, H2,
                                       reinterpret_cast<float*>(base + ws.off_partial_fc1), sums, grad + Fc1W(s, 0), BlockParams(s)));
        // (with batch normalisation b2_k and the hidden bias got their gradients from the normalisation's backward pass)
        sums.TowerBiases(s, colsum, colsum_rows, ws.colsum_slot_floats, grad, !bnorm);
        MGT_TRY(sums.Pass());
        if (cudaGetLastError() != cudaSuccess) return MGT_CUDA_FAILURE;
        for (uint32_t rb = R; rb > 0; --rb) {
            MGT_TRY(notify(Fc2W(s, rb - 1U), (uint64_t)H2 * H2 + H2));
            MGT_TRY(notify(Fc1W(s, rb - 1U), (uint64_t)H2 * H2 + H2));
        }
    }
    if (!timer.Mark(profile ? &profile->residual_backward_ms : nullptr)) return MGT_CUDA_FAILURE;

    // ---- hidden layer backward, dW part; every kernel that reads the hidden weights was enqueued long before, so a caller
    // may update the range in place as soon as it is announced
    MGT_TRY(GemmGradWeightsRows(e, st_dw, a1_h, ws.p_bt, dz_cur, ws.p_dz, B, H1, H2, reinterpret_cast<float*>(base + ws.off_partial), sums, grad + HiddenWeight(s)));
    MGT_TRY(sums.LaunchAll());  // (on the second stream they are done while the table gradient still runs)
    if (!branch.Join()) return MGT_CUDA_FAILURE;
    MGT_TRY(notify(HiddenWeight(s), (uint64_t)H1 * H2 + H2));
    if (!timer.Mark(profile ? &profile->hidden_backward_ms : nullptr)) return MGT_CUDA_FAILURE;
    MGT_TRY(notify(0, InputBias(s) + H1));
    if (bnorm) MGT_TRY(notify(bn_base, 2ULL * (R + 1ULL) * H2));
    return MGT_OK;
}

mgt_status_t mgt_engine_set_train_options(mgt_engine_t* e, const mgt_train_options_t* options) {
    if (e == nullptr || options == nullptr) return MGT_INVALID_CONFIG;
    if (options->operand_format != MGT_OPERAND_FP16 && options->operand_format != MGT_OPERAND_BF16) return MGT_INVALID_CONFIG;
    if (options->loss_kind != MGT_LOSS_MSE && options->loss_kind != MGT_LOSS_CROSS_ENTROPY) return MGT_INVALID_CONFIG;
    if (options->batch_norm != 0 && !(options->bn_eps > 0.0f)) return MGT_INVALID_CONFIG;
    e->options = *options;
    return MGT_OK;
}

mgt_status_t mgt_engine_set_early_range_hook(mgt_engine_t* e, mgt_gradient_ready_fn fn, void* user) {
    if (e == nullptr) return MGT_INVALID_CONFIG;
    e->early_fn = fn;
    e->early_user = user;
    return MGT_OK;
}

mgt_status_t mgt_debug_gemm(mgt_engine_t* e, const uint16_t* a, uint32_t lda, int32_t a_mn, const uint16_t* b, uint32_t ldb, int32_t b_mn,
                            float* d, uint32_t m, uint32_t n, uint32_t k, uint32_t splits, float* partial_scratch, void* stream) {
    if (e == nullptr || a == nullptr || b == nullptr || d == nullptr || m == 0 || n == 0 || k == 0 || splits == 0) return MGT_INVALID_CONFIG;
    if (splits > 1 && partial_scratch == nullptr) return MGT_INVALID_CONFIG;
    const LaunchOn st(static_cast<cudaStream_t>(stream), false);
    GemmArgs args = BaseArgs(m, n, k, 256, splits);
    // with a single split the accumulator tiles go straight into d, as 16-byte vectors when n is a multiple of 4
    if (args.splits == 1 && (n & 3U) == 0U && (reinterpret_cast<uintptr_t>(d) & 15U) != 0U) return MGT_INVALID_CONFIG;
    if ((reinterpret_cast<uintptr_t>(d) & 3U) != 0U) return MGT_INVALID_CONFIG;
    if (args.splits > 1 && (n & 3U) == 0U && (reinterpret_cast<uintptr_t>(partial_scratch) & 15U) != 0U) return MGT_INVALID_CONFIG;
    args.partial = args.splits > 1 ? partial_scratch : d;
    CUtensorMap ta, tb;
    const __half* ah = reinterpret_cast<const __half*>(a);
    const __half* bh = reinterpret_cast<const __half*>(b);
    if (a_mn) { MGT_MAP(e->Map(&ta, ah, m, k, lda, 64, 64)); } else { MGT_MAP(e->Map(&ta, ah, k, m, lda, 64, 128)); }
    if (b_mn) { MGT_MAP(e->Map(&tb, bh, n, k, ldb, 64, 64)); } else { MGT_MAP(e->Map(&tb, bh, k, n, ldb, 64, 256)); }
    mgt_status_t r;
    if (a_mn && b_mn) r = LaunchGemm<CfgDw<256>>(e, ta, tb, args, st);
    else if (a_mn) r = LaunchGemm<CfgDbgMK>(e, ta, tb, args, st);
    else if (b_mn) r = LaunchGemm<CfgDbgKM>(e, ta, tb, args, st);
    else r = LaunchGemm<CfgDbgKK>(e, ta, tb, args, st);
    if (r != MGT_OK) return r;
    if (args.splits > 1) {
        Sums sums{e, true, st};
        sums.Planes(partial_scratch, args.splits, (uint64_t)m * n, d);
        MGT_TRY(sums.LaunchAll());
    }
    return MGT_OK;
}

mgt_status_t mgt_debug_sums(mgt_engine_t* e, const float* src, uint32_t terms, uint32_t items, uint32_t jobs, int32_t planes, float* dst, void* stream) {
    if (e == nullptr || src == nullptr || dst == nullptr || terms == 0 || items == 0 || jobs == 0) return MGT_INVALID_CONFIG;
    Sums sums{e, false, {static_cast<cudaStream_t>(stream), false}};
    for (uint32_t j = 0; j < jobs; ++j) {
        const float* at = src + (uint64_t)j * terms * items;
        if (planes) sums.Planes(at, terms, items, dst + (uint64_t)j * items);
        else sums.Rows(at, terms, items, items, dst + (uint64_t)j * items);
    }
    return sums.LaunchAll();
}

}  // extern "C"

// ---- split-K GEMM whose scratch is part of the library image ------------------------------------
// Device memory that this library reserves at load time on every GPU that uses it: the split-K
// partial sums of mgt_gemm_split_k_static_scratch and that entry point's status word.
static __device__ __align__(256) float g_static_partials[MGT_STATIC_SCRATCH_FLOATS];
static __device__ int g_static_status;

namespace {
struct StaticSlot {
    mgt_engine* engine = nullptr;   // host-side object only: descriptor cache, SM count, status-word address
    float* partials = nullptr;      // device address of g_static_partials on that device
};
StaticSlot g_static_slots[64];
std::mutex g_static_mu;

// One-time set-up per device, with that device current: resolve the DEVICE addresses of the two
// symbols above (in host code their names are only host-side handles) and look up the tensor-map
// encoder. Allocates no device memory.
mgt_status_t StaticSlotFor(int device, StaticSlot** out) {
    if (device < 0 || device >= 64) return MGT_INVALID_CONFIG;
    std::lock_guard<std::mutex> lock(g_static_mu);
    StaticSlot& slot = g_static_slots[device];
    if (slot.engine == nullptr) {
        void* partials = nullptr;
        void* status = nullptr;
        if (cudaGetSymbolAddress(&partials, g_static_partials) != cudaSuccess || partials == nullptr) return MGT_CUDA_FAILURE;
        if (cudaGetSymbolAddress(&status, g_static_status) != cudaSuccess || status == nullptr) return MGT_CUDA_FAILURE;
        cudaDeviceProp prop{};
        if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return MGT_CUDA_FAILURE;
        if (prop.major != 10) {
            std::fprintf(stderr, "mgt_b200: device %d is sm_%d%d; this library only runs on sm_100a (B200)\n", device, prop.major, prop.minor);
            return MGT_CUDA_FAILURE;
        }
        void* fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres) != cudaSuccess || fn == nullptr) return MGT_CUDA_FAILURE;
        auto* e = new mgt_engine();
        e->device = device;
        e->sm_count = prop.multiProcessorCount;
        e->encode = reinterpret_cast<EncodeTiledFn>(fn);
        e->status_word = static_cast<int*>(status);
        slot.engine = e;
        slot.partials = static_cast<float*>(partials);
    }
    *out = &slot;
    return MGT_OK;
}
}  // namespace

extern "C" mgt_status_t mgt_gemm_split_k_static_scratch(const uint16_t* a, uint32_t lda, int32_t a_mn, const uint16_t* b, uint32_t ldb, int32_t b_mn,
                                                        float* d, uint32_t m, uint32_t n, uint32_t k, uint32_t splits, void* stream) {
    if (a == nullptr || b == nullptr || d == nullptr || m == 0 || n == 0 || k == 0 || splits == 0) return MGT_INVALID_CONFIG;
    const uint32_t k_chunks = (k + 63U) / 64U;
    const uint64_t used_splits = splits > k_chunks ? k_chunks : splits;
    if (used_splits > 1 && used_splits * m * n > static_cast<uint64_t>(MGT_STATIC_SCRATCH_FLOATS)) {
        std::fprintf(stderr, "mgt_gemm_split_k_static_scratch: %llu splits of a %u x %u result need %llu floats of scratch, the built-in buffer holds %u\n",
                     static_cast<unsigned long long>(used_splits), m, n, static_cast<unsigned long long>(used_splits * m * n),
                     static_cast<unsigned>(MGT_STATIC_SCRATCH_FLOATS));
        return MGT_CAPACITY_EXCEEDED;
    }
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return MGT_CUDA_FAILURE;
    StaticSlot* slot = nullptr;
    MGT_TRY(StaticSlotFor(device, &slot));
    // every valid element of the partial planes is written before the reduction reads it, so nothing
    // needs clearing between calls; what an earlier call left beyond that is never read
    return mgt_debug_gemm(slot->engine, a, lda, a_mn, b, ldb, b_mn, d, m, n, k, splits, slot->partials, stream);
}

extern "C" mgt_status_t mgt_static_scratch_check(void* stream, int32_t* out_device_code) {
    int device = 0;
    if (cudaGetDevice(&device) != cudaSuccess) return MGT_CUDA_FAILURE;
    StaticSlot* slot = nullptr;
    MGT_TRY(StaticSlotFor(device, &slot));
    // the hidden per-device engine's status word is the built-in g_static_status: same read-and-clear as mgt_engine_check
    return mgt_engine_check(slot->engine, stream, out_device_code);
}
