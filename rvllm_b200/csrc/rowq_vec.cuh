// The C launcher's forms of the row kernels: the arithmetic — and so every byte and scale — of the entry points in
// rowq_rmsnorm.cu, rowq_act.cuh and rope_kv_write.cu, without the launch geometry those take from the reference's launchers.
//
// What bounds the reference geometry at prefill-sized row counts is not bandwidth: 1024 threads per row hold one vector
// each, spend their time in four block-wide barriers, and two such blocks fill an SM; a (token, head) block of 64 threads
// per RoPE head does 500 bytes of work per launch slot.  Measured on [1000 x 5376 / 21504], us, reference geometry / here:
// add + norm + quant 17.6 / 7.0, RoPE + KV write 33.9 / 7.4 (16-byte loads, see its launcher), act + quant 47.3 / 28.4,
// per-token quant (4096) 8.0 / 3.1; on 32 rows the norm 4.1 / 2.9.
//
// (What a preceding kernel wrote is read with plain loads: see rv::ldg128.)
#pragma once
#include "common.cuh"
#include "rowq_act.cuh"

namespace rvrow {

// ---- RMSNorm + quant ----------------------------------------------------------------------------------------------------
// A thread holds up to NV 16-byte vectors of the row and stands for eight threads of the reference block of `nt` threads:
// vector t + j * (nt / 8) holds elements 8 t + k + j nt, the ones reference thread 8 t + k sums.  Eight partial sums per
// thread, combined over lanes first (the reference butterfly's offsets 16 and 8), then inside the thread (4, 2, 1), are
// bit for bit the reference's warp sums; 128 threads per row instead of 1024, one barrier per reduction, and the row never
// leaves registers.
template <typename T, int NV, bool RES>
__global__ void __launch_bounds__(128) norm_quant_vec_kernel(uint8_t* __restrict__ out, float* __restrict__ scales, T* residual_out,
                                                             const T* in, const T* residual,
                                                             const T* __restrict__ gamma, float eps, int hidden, int nt) {
    __shared__ float s_sum[32], s_max[4];
    const int t = threadIdx.x, lane = t & 31, per = nt >> 3, nvec = hidden >> 3;
    const size_t base = (size_t)blockIdx.x * nvec;
    rv::pdl_launch();
    uint4 g[NV], x[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) {  // gamma is a weight: fetched ahead of the wait for the kernel before
        const int v = t + j * per;
        g[j] = make_uint4(0, 0, 0, 0);
        if (t < per && v < nvec) g[j] = rv::ldg128(reinterpret_cast<const uint4*>(gamma) + v);
    }
    rv::pdl_wait();
    uint4 r[RES ? NV : 1];
#pragma unroll
    for (int j = 0; j < NV; j++) {
        const int v = t + j * per;
        x[j] = make_uint4(0, 0, 0, 0);
        if (RES) r[j] = make_uint4(0, 0, 0, 0);
        if (t < per && v < nvec) {
            x[j] = reinterpret_cast<const uint4*>(in)[base + v];
            if (RES) r[j] = reinterpret_cast<const uint4*>(residual)[base + v];
        }
    }
    float ss[8];
#pragma unroll
    for (int k = 0; k < 8; k++) ss[k] = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; j++) {
        uint32_t* xp = &x[j].x;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float2 a = rv::T16<T>::to_f32x2(xp[k]);
            if (RES) {
                const float2 b = rv::T16<T>::to_f32x2((&r[RES ? j : 0].x)[k]);
                a.x = a.x + b.x;
                a.y = a.y + b.y;
                xp[k] = rv::pack2<T>(a.x, a.y);  // the sum of squares is of the unrounded sum, the norm of the rounded one
            }
            ss[2 * k] += a.x * a.x;
            ss[2 * k + 1] += a.y * a.y;
        }
        if (RES) {
            const int v = t + j * per;
            if (t < per && v < nvec) reinterpret_cast<uint4*>(residual_out)[base + v] = x[j];
        }
    }
#pragma unroll
    for (int o = 2; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 8; k++) ss[k] += __shfl_xor_sync(0xffffffffu, ss[k], o);
    const float w = ((ss[0] + ss[4]) + (ss[2] + ss[6])) + ((ss[1] + ss[5]) + (ss[3] + ss[7]));
    if ((t & 3) == 0 && t < per) s_sum[t >> 2] = w;
    __syncthreads();
    const float sum_sq = rv::warp_sum(lane < (nt >> 5) ? s_sum[lane] : 0.0f);
    const float rms = rsqrtf(sum_sq / (float)hidden + eps);
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; j++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 a = rv::T16<T>::to_f32x2((&x[j].x)[k]), b = rv::T16<T>::to_f32x2((&g[j].x)[k]);
            amax = fmaxf(amax, fmaxf(fabsf(a.x * rms * b.x), fabsf(a.y * rms * b.y)));
        }
    amax = rv::warp_max(amax);
    if (lane == 0) s_max[t >> 5] = amax;
    __syncthreads();
    amax = s_max[0];
    for (int i = 1; i < (int)(blockDim.x >> 5); i++) amax = fmaxf(amax, s_max[i]);
    const float scale = rv::row_scale(amax);
    if (t == 0) scales[blockIdx.x] = scale;
    const float inv = 1.0f / scale;
#pragma unroll
    for (int j = 0; j < NV; j++) {
        const int v = t + j * per;
        float f[8];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 a = rv::T16<T>::to_f32x2((&x[j].x)[k]), b = rv::T16<T>::to_f32x2((&g[j].x)[k]);
            f[2 * k] = a.x * rms * b.x * inv;
            f[2 * k + 1] = a.y * rms * b.y * inv;
        }
        if (t < per && v < nvec)
            reinterpret_cast<uint2*>(out)[base + v] =
                make_uint2(rv::f32x4_to_e4m3x4(f[0], f[1], f[2], f[3]), rv::f32x4_to_e4m3x4(f[4], f[5], f[6], f[7]));
    }
}

// ---- per-token quant ------------------------------------------------------------------------------------------------------
// Up to four vectors per thread in registers, as few warps per row as that takes.
template <typename T>
__global__ void __launch_bounds__(1024) quant_vec_kernel(uint8_t* __restrict__ out, float* __restrict__ scales,
                                                         const T* in, int dim) {
    constexpr int NV = 4;
    __shared__ float s_max[32];
    const int t = threadIdx.x, lane = t & 31, nt = blockDim.x, nvec = dim >> 3;
    const size_t base = (size_t)blockIdx.x * nvec;
    rv::pdl_launch();
    rv::pdl_wait();
    uint4 x[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) {
        const int v = t + j * nt;
        x[j] = v < nvec ? reinterpret_cast<const uint4*>(in)[base + v] : make_uint4(0, 0, 0, 0);
    }
    float amax = 0.0f;
#pragma unroll
    for (int j = 0; j < NV; j++)
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 a = rv::T16<T>::to_f32x2((&x[j].x)[k]);
            amax = fmaxf(amax, fmaxf(fabsf(a.x), fabsf(a.y)));
        }
    amax = rv::warp_max(amax);
    if (nt > 32) {
        if (lane == 0) s_max[t >> 5] = amax;
        __syncthreads();
        amax = rv::warp_max(lane < (nt >> 5) ? s_max[lane] : 0.0f);
    }
    const float scale = rv::row_scale(amax);
    if (t == 0) scales[blockIdx.x] = scale;
    const float inv = 1.0f / scale;
#pragma unroll
    for (int j = 0; j < NV; j++) {
        const int v = t + j * nt;
        float f[8];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float2 a = rv::T16<T>::to_f32x2((&x[j].x)[k]);
            f[2 * k] = a.x * inv;
            f[2 * k + 1] = a.y * inv;
        }
        if (v < nvec)
            reinterpret_cast<uint2*>(out)[base + v] =
                make_uint2(rv::f32x4_to_e4m3x4(f[0], f[1], f[2], f[3]), rv::f32x4_to_e4m3x4(f[4], f[5], f[6], f[7]));
    }
}

// ---- act(gate) * up + quant, many long rows -------------------------------------------------------------------------------
// Persistent: one block of 1024 threads per SM, two row buffers in shared memory filled by bulk copies, so that a row's
// loads overlap the arithmetic of the row before (about 35 instructions per element: exponential, division, conversions —
// the arithmetic, not the 5 bytes per element, is the longer side).  Products stay in registers between the row maximum
// and the encode; the maximum is taken over the magnitudes' bit patterns, where a non-finite product is the largest.
__device__ __forceinline__ uint32_t saddr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
constexpr uint32_t ROW_WAIT_LIMIT = 1u << 24;

template <int ACT, typename T, int NC>
__global__ void __launch_bounds__(1024, 1) act_mul_quant_stream_kernel(uint8_t* __restrict__ out, float* __restrict__ scales,
                                                                       const T* gate_up, int inter, int rows) {
    extern __shared__ __align__(128) uint8_t raw[];
    __shared__ uint64_t full[2];
    __shared__ uint32_t red[2][32];
    const int t = threadIdx.x, lane = t & 31, nvec = inter >> 3;
    const uint32_t row_bytes = 4u * (uint32_t)inter;
    rv::pdl_launch();
    auto fetch = [&](int row, int b) {  // (one thread)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(saddr(full + b)), "r"(row_bytes) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                         saddr(raw + (size_t)b * row_bytes)),
                     "l"(gate_up + (size_t)row * 2 * inter), "r"(row_bytes), "r"(saddr(full + b))
                     : "memory");
    };
    if (t == 0) {
        for (int b = 0; b < 2; b++) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(saddr(full + b)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    rv::pdl_wait();
    __syncthreads();
    if (t == 0)
        for (int b = 0; b < 2; b++)
            if ((int)blockIdx.x + b * (int)gridDim.x < rows) fetch((int)blockIdx.x + b * (int)gridDim.x, b);
    int b = 0;
    uint32_t ph = 0;
    for (int row = blockIdx.x; row < rows; row += gridDim.x) {
        bool landed = false;
        for (uint32_t i = 0; i < ROW_WAIT_LIMIT && !landed; i++) {
            uint32_t ok;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(ok)
                : "r"(saddr(full + b)), "r"(ph)
                : "memory");
            landed = ok != 0;
        }
        const uint8_t* src = raw + (size_t)b * row_bytes;
        float y[NC][8];
        uint32_t mx = landed ? 0u : 0x7fffffffu;  // (a copy that never landed: the row's scale becomes NaN)
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const int v = t + c * 1024;
            if (v < nvec) {
                rvact::mul8<ACT, T>(reinterpret_cast<const uint4*>(src)[v], reinterpret_cast<const uint4*>(src + 2 * (size_t)inter)[v], y[c]);
#pragma unroll
                for (int k = 0; k < 8; k++) mx = max(mx, __float_as_uint(y[c][k]) & 0x7fffffffu);
            }
        }
        mx = __reduce_max_sync(0xffffffffu, mx);
        if (lane == 0) red[b][t >> 5] = mx;
        __syncthreads();  // every thread is done with the buffer; the maxima are in place
        if (t == 0 && row + 2 * (int)gridDim.x < rows) fetch(row + 2 * (int)gridDim.x, b);
        mx = __reduce_max_sync(0xffffffffu, red[b][lane]);
        const float scale = mx >= 0x7f800000u ? CUDART_NAN_F : rv::row_scale(__uint_as_float(mx));
        if (t == 0) scales[row] = scale;
        const float inv = 1.0f / scale;
        uint2* o = reinterpret_cast<uint2*>(out + (size_t)row * inter);
#pragma unroll
        for (int c = 0; c < NC; c++) {
            const int v = t + c * 1024;
            if (v < nvec)
                o[v] = make_uint2(rv::f32x4_to_e4m3x4(y[c][0] * inv, y[c][1] * inv, y[c][2] * inv, y[c][3] * inv),
                                  rv::f32x4_to_e4m3x4(y[c][4] * inv, y[c][5] * inv, y[c][6] * inv, y[c][7] * inv));
        }
        b ^= 1;
        ph ^= b == 0 ? 1u : 0u;
    }
}

// ---- RoPE + Q quant + paged KV write --------------------------------------------------------------------------------------
// A head row is a sub-warp group of head_dim / (2 VE) lanes, each with VE elements of the lower half and their partners of
// the upper half: vector loads and stores, shuffles instead of a block barrier, and 256-thread blocks over the token's
// Q, K and V heads alike.
template <typename T, int VE>
__global__ void __launch_bounds__(256)
rope_fp8kv_vec_kernel(const T* q_in, const T* k_in, const T* v_in, int stride,
                      uint8_t* __restrict__ q_fp8, uint8_t* __restrict__ k_cache, uint8_t* __restrict__ v_cache,
                      float* __restrict__ k_scale, float* __restrict__ v_scale, float* __restrict__ q_scale,
                      const T* cos_t, const T* sin_t, const int* positions, const int* slot_mapping,
                      int heads, int kv_heads, int head_dim, int half_rot,
                      int max_positions, int num_cache_slots) {
    rv::pdl_launch();
    rv::pdl_wait();
    const int half = head_dim >> 1, lanes = half / VE;  // a power of two up to 32
    const int idx = blockIdx.x * 256 + threadIdx.x, item = idx / lanes, l = idx & (lanes - 1), tok = blockIdx.y;
    const int kind = item < heads ? 0 : (item < heads + kv_heads ? 1 : 2);
    const int head = kind == 0 ? item : (kind == 1 ? item - heads : item - heads - kv_heads);
    const bool in = item < heads + 2 * kv_heads;
    const int pos = positions[tok];
    const int slot = kind == 0 ? 0 : slot_mapping[tok];
    const bool live = in && pos >= 0 && pos < max_positions && (kind == 0 || (slot >= 0 && slot < num_cache_slots));
    struct alignas(2 * VE) Vec {
        uint32_t w[VE / 2];
    };
    Vec lo16 = {}, hi16 = {}, c16 = {}, s16 = {};
    const bool rot = kind != 2 && l * VE < half_rot;
    if (live) {
        const T* row = (kind == 0 ? q_in : kind == 1 ? k_in : v_in) + (size_t)tok * stride + (size_t)head * head_dim + l * VE;
        lo16 = *reinterpret_cast<const Vec*>(row);
        hi16 = *reinterpret_cast<const Vec*>(row + half);
        if (rot) {
            c16 = *reinterpret_cast<const Vec*>(cos_t + (size_t)pos * half_rot + l * VE);
            s16 = *reinterpret_cast<const Vec*>(sin_t + (size_t)pos * half_rot + l * VE);
        }
    }
    float lo[VE], hi[VE], am = 0.0f;
#pragma unroll
    for (int j = 0; j < VE / 2; j++) {
        const float2 a = rv::T16<T>::to_f32x2(lo16.w[j]), b = rv::T16<T>::to_f32x2(hi16.w[j]);
        const float2 c = rv::T16<T>::to_f32x2(c16.w[j]), s = rv::T16<T>::to_f32x2(s16.w[j]);
        lo[2 * j] = rot ? a.x * c.x - b.x * s.x : a.x;
        hi[2 * j] = rot ? a.x * s.x + b.x * c.x : b.x;
        lo[2 * j + 1] = rot ? a.y * c.y - b.y * s.y : a.y;
        hi[2 * j + 1] = rot ? a.y * s.y + b.y * c.y : b.y;
    }
#pragma unroll
    for (int j = 0; j < VE; j++) {
        const float m = (!isfinite(lo[j]) || !isfinite(hi[j])) ? CUDART_INF_F : fmaxf(fabsf(lo[j]), fabsf(hi[j]));
        am = fmaxf(am, m);
    }
    for (int o = lanes >> 1; o > 0; o >>= 1) am = fmaxf(am, __shfl_xor_sync(0xffffffffu, am, o));
    if (!live) return;
    const float sc = isinf(am) ? CUDART_NAN_F : rv::row_scale(am);
    const float inv = 1.0f / sc;
    size_t row_out;
    uint8_t* o;
    float* so;
    if (kind == 0) {
        row_out = (size_t)tok * heads + head;
        o = q_fp8;
        so = q_scale;
    } else {
        row_out = (size_t)slot * kv_heads + head;
        o = kind == 1 ? k_cache : v_cache;
        so = kind == 1 ? k_scale : v_scale;
    }
    o += row_out * head_dim + l * VE;
    struct alignas(VE) Codes {
        uint32_t w[VE / 4];
    } clo, chi;
#pragma unroll
    for (int j = 0; j < VE; j += 4) {
        clo.w[j / 4] = rv::f32x4_to_e4m3x4(lo[j] * inv, lo[j + 1] * inv, lo[j + 2] * inv, lo[j + 3] * inv);
        chi.w[j / 4] = rv::f32x4_to_e4m3x4(hi[j] * inv, hi[j + 1] * inv, hi[j + 2] * inv, hi[j + 3] * inv);
    }
    *reinterpret_cast<Codes*>(o) = clo;
    *reinterpret_cast<Codes*>(o + half) = chi;
    if (l == 0) so[row_out] = sc;
}

}  // namespace rvrow
