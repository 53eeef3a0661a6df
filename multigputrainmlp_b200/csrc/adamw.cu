// Element-wise AdamW with optional fp16 weight mirror: native/cuda/adamw.cu:8-46.
// HBM-bound: 28 bytes (30 with the mirror) per parameter; 16-byte accesses, one per thread and array.
#include "../../include/mgt_b200.h"
#include "adamw_math.cuh"
#include "launch.cuh"

#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace {

constexpr uint32_t kAdamWThreads = 128;
constexpr uint64_t kOverlapParams = 8ULL << 20;  // a longer update does not notice the gap before it, and its CTAs crowd what still runs

template <bool kMirror>
__global__ void __launch_bounds__(kAdamWThreads)
AdamWKernel(mgt_adamw_config_t config, float* __restrict__ w, __half* __restrict__ w_half, const float* __restrict__ g,
            float* __restrict__ m, float* __restrict__ v) {
    const mgt::AdamWScalars sc = mgt::MakeAdamWScalars(config.step, config.learning_rate, config.beta1, config.beta2, config.eps, config.weight_decay);
    const uint64_t n4 = config.param_count >> 2;
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    mgt::dependent_begin();
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += stride) {
        float4 wv = reinterpret_cast<float4*>(w)[i];
        const float4 gv = reinterpret_cast<const float4*>(g)[i];
        float4 mv = reinterpret_cast<float4*>(m)[i];
        float4 vv = reinterpret_cast<float4*>(v)[i];
        wv.x = mgt::AdamWUpdateOne(sc, wv.x, gv.x, &mv.x, &vv.x);
        wv.y = mgt::AdamWUpdateOne(sc, wv.y, gv.y, &mv.y, &vv.y);
        wv.z = mgt::AdamWUpdateOne(sc, wv.z, gv.z, &mv.z, &vv.z);
        wv.w = mgt::AdamWUpdateOne(sc, wv.w, gv.w, &mv.w, &vv.w);
        reinterpret_cast<float4*>(w)[i] = wv;
        reinterpret_cast<float4*>(m)[i] = mv;
        reinterpret_cast<float4*>(v)[i] = vv;
        if (kMirror) {
            const __half2 h01 = __floats2half2_rn(wv.x, wv.y);
            const __half2 h23 = __floats2half2_rn(wv.z, wv.w);
            uint2 u;
            u.x = *reinterpret_cast<const uint32_t*>(&h01);
            u.y = *reinterpret_cast<const uint32_t*>(&h23);
            reinterpret_cast<uint2*>(w_half)[i] = u;
        }
    }
    // tail (param_count % 4)
    const uint64_t tail0 = n4 << 2;
    const uint64_t t = tail0 + static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < config.param_count) {
        float mm = m[t], vv = v[t];
        const float nw = mgt::AdamWUpdateOne(sc, w[t], g[t], &mm, &vv);
        w[t] = nw;
        m[t] = mm;
        v[t] = vv;
        if (kMirror) w_half[t] = __float2half_rn(nw);
    }
}

__global__ void FloatToHalfKernel(const float* __restrict__ src, uint64_t count, __half* __restrict__ dst) {
    mgt::dependent_begin();
    const uint64_t stride = static_cast<uint64_t>(gridDim.x) * blockDim.x;
    for (uint64_t i = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < count; i += stride) dst[i] = __float2half_rn(src[i]);
}

int SmCount() {
    int dev = 0, sms = 148;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 148;
}

bool Aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15U) == 0U; }

}  // namespace

extern "C" {

mgt_status_t mgt_validate_adamw_config(const mgt_adamw_config_t* c) {
    if (c == nullptr) return MGT_INVALID_CONFIG;
    if (c->param_count == 0 || c->step == 0 || !(c->learning_rate > 0.0f) || c->beta1 < 0.0f || c->beta1 >= 1.0f ||
        c->beta2 < 0.0f || c->beta2 >= 1.0f || !(c->eps > 0.0f) || c->weight_decay < 0.0f) {
        return MGT_INVALID_CONFIG;
    }
    return MGT_OK;
}

static mgt_status_t LaunchAdamW(const mgt_adamw_config_t* config, float* w, uint16_t* w_half, const float* g, float* m, float* v,
                                void* stream, bool mirror) {
    if (mgt_validate_adamw_config(config) != MGT_OK || w == nullptr || g == nullptr || m == nullptr || v == nullptr ||
        (mirror && w_half == nullptr)) {
        return MGT_INVALID_CONFIG;
    }
    if (!Aligned16(w) || !Aligned16(g) || !Aligned16(m) || !Aligned16(v) || (mirror && (reinterpret_cast<uintptr_t>(w_half) & 7U))) {
        return MGT_INVALID_CONFIG;
    }
    // One 16-byte item per thread in CTAs of 128 threads: 0.076 ms for the 15.46 M parameters of p888 against 0.080 ms as a
    // grid-stride loop over 16 CTAs per SM. The loop in the kernel only serves counts beyond the grid limit.
    const uint64_t n4 = config->param_count >> 2;
    const uint64_t want = (n4 + kAdamWThreads - 1ULL) / kAdamWThreads;
    const uint64_t cap = 1ULL << 30;
    const uint32_t blocks = static_cast<uint32_t>(want < 1 ? 1 : (want < cap ? want : cap));
    const mgt::LaunchOn s(static_cast<cudaStream_t>(stream), config->param_count <= kOverlapParams);
    if (mirror) {
        mgt::Launch(AdamWKernel<true>, blocks, kAdamWThreads, 0, s, *config, w, reinterpret_cast<__half*>(w_half), g, m, v);
    } else {
        mgt::Launch(AdamWKernel<false>, blocks, kAdamWThreads, 0, s, *config, w, nullptr, g, m, v);
    }
    return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
}

mgt_status_t mgt_launch_adamw(const mgt_adamw_config_t* config, float* w, const float* g, float* m, float* v, void* stream) {
    return LaunchAdamW(config, w, nullptr, g, m, v, stream, false);
}

mgt_status_t mgt_launch_adamw_with_half_mirror(const mgt_adamw_config_t* config, float* w, uint16_t* w_half, const float* g,
                                               float* m, float* v, void* stream) {
    return LaunchAdamW(config, w, w_half, g, m, v, stream, true);
}

mgt_status_t mgt_launch_float_to_half(const float* values, uint64_t count, uint16_t* half, void* stream) {
    if (values == nullptr || half == nullptr || count == 0) return MGT_INVALID_CONFIG;
    const uint64_t want = (count + 255ULL) / 256ULL;
    const uint64_t cap = static_cast<uint64_t>(SmCount()) * 16ULL;
    const uint32_t blocks = static_cast<uint32_t>(want < cap ? want : cap);
    mgt::Launch(FloatToHalfKernel, blocks, 256, 0, {static_cast<cudaStream_t>(stream), true}, values, count, reinterpret_cast<__half*>(half));
    return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_CUDA_FAILURE;
}

}  // extern "C"
