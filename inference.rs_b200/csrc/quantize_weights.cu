// Weight quantizers and dequantizers on the device: f32 rows -> packed Q8_0 / Q4_K / Q6_K blocks, byte for byte what the
// reference's CPU quantizer produces in its default mode (`Quantizer::LlamaCpp`, no importance matrix), and back.
//
// Reference: `QTensor::quantize` (crates/inference-tensor/src/quantized/mod.rs:903-918) -> `BlockQ8_0::from_float`
// (k_quants.rs:923-949 via quantize_block32, mod.rs:43-56), `BlockQ4K::quantize_with` (k_quants.rs:1949-2015) with
// `make_qkx2_quants` (utils.rs:268-361), `BlockQ6K::quantize_with` (k_quants.rs:2590-2646) with `make_qx_quants`
// (utils.rs:135-264); `to_float` (k_quants.rs:905-921,2096-2123,2649-2680); the embedding row gather `get_rows`
// (crates/inference-tensor/src/quantized/cuda.rs:151-242). The reference runs the K-quant searches on the host even
// for CUDA tensors (cuda.rs:340-361) and has device quantizers for Q6_K / Q8_0 only
// (crates/inference-quant/kernels/cuda/gguf_quantize/k_quantize_instance_ggufq.cu:1-6).
//
// The scale searches compare sums of f32 products whose rounding decides which candidate wins, so the arithmetic is
// the reference's operation for operation: this file is compiled with -fmad=false (no multiply-add contraction, as the
// reference's LlamaCpp mode, utils.rs:37-45), divisions and square roots are IEEE, and sums run in the same order.
// One thread searches one sub-block (32 values of Q4_K, 16 of Q6_K) held in registers; the lanes of a superblock then meet in
// shuffles to agree on its scales and to write its bytes. The searches are bound by the f32 pipe, not by memory: a sub-block
// of Q4_K tries 21 scales over 32 values, a dozen operations each, and every sum has one order to run in.
#include "common.cuh"
#include "runtime.h"
#include <type_traits>

namespace b200q {

constexpr float ROUNDING_MAGIC = 12582912.0f;  // 1.5 * 2^23: adding it rounds to the nearest integer, ties to even
constexpr float GROUP_MAX_EPS = 1e-15f;

__device__ __forceinline__ int nearest_int(float v) {  // utils.rs:32-35
    const float r = v + ROUNDING_MAGIC;
    return (int)(__float_as_uint(r) & 0x007fffffu) - 0x00400000;
}
__device__ __forceinline__ int nearest_int_mul(float a, float b) { return nearest_int(a * b); }  // utils.rs:70-73, unfused
__device__ __forceinline__ int clampi(int v, int lo, int hi) { return v < lo ? lo : (v > hi ? hi : v); }
__device__ __forceinline__ unsigned short f16_bits(float v) { return __half_as_ushort(__float2half_rn(v)); }
__device__ __forceinline__ float f16_value(unsigned short b) { return __half2float(__ushort_as_half(b)); }
// Rust's `as i8` on a float: saturating, NaN -> 0
__device__ __forceinline__ int sat_i8(float v) {
    if (v != v) return 0;
    if (v <= -128.0f) return -128;
    if (v >= 127.0f) return 127;
    return (int)v;
}

// ---------------------------------------------------------------------------------------------
// Q8_0: d = amax / 127, q = round_half_away(x * (1 / d))
// ---------------------------------------------------------------------------------------------
// HBM-bound: 4 bytes in and 1.06 out per value. Eight lanes share a block (one 128-bit load each); the 32 blocks of a CTA
// are 1088 bytes, a multiple of 16, so they are put together in shared memory and leave as 128-bit stores.
constexpr int Q8_CTA_BLOCKS = 32;
__global__ void __launch_bounds__(256) quantize_q8_0_kernel(const float* __restrict__ x, uint8_t* __restrict__ out, long long nblocks, int vec_in,
                                                           int vec_out) {
    __shared__ __align__(16) uint8_t stage[Q8_CTA_BLOCKS * Q8_0_BYTES];
    const int tid = threadIdx.x, sub = tid & 7, local = tid >> 3;
    const long long b0 = (long long)blockIdx.x * Q8_CTA_BLOCKS, b = b0 + local;
    float v[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    if (b < nblocks) {
        const float* xb = x + b * 32 + 4 * sub;
        if (vec_in) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(xb));
            v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = xb[i];
        }
    }
    float amax = 0.0f;  // and not v[0]: fmaxf passes a NaN over, so a block of nothing else has the scale 0
#pragma unroll
    for (int i = 0; i < 4; ++i) amax = fmaxf(amax, fabsf(v[i]));
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, m));
    const float d = amax / 127.0f;
    const float id = d != 0.0f ? 1.0f / d : 0.0f;
    unsigned short* o = reinterpret_cast<unsigned short*>(stage + local * Q8_0_BYTES);
    if (sub == 0) o[0] = f16_bits(d);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const unsigned lo = (unsigned)sat_i8(roundf(v[2 * i] * id)) & 0xffu;
        const unsigned hi = (unsigned)sat_i8(roundf(v[2 * i + 1] * id)) & 0xffu;
        o[1 + 2 * sub + i] = (unsigned short)(lo | (hi << 8));
    }
    __syncthreads();
    const int bytes = (int)min((long long)Q8_CTA_BLOCKS, nblocks - b0) * Q8_0_BYTES;
    uint8_t* dst = out + b0 * Q8_0_BYTES;
    const int whole = vec_out ? bytes / 16 : 0;
    for (int i = tid; i < whole; i += 256) reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(stage)[i];
    for (int i = whole * 8 + tid; i < bytes / 2; i += 256)
        reinterpret_cast<unsigned short*>(dst)[i] = reinterpret_cast<const unsigned short*>(stage)[i];
}

// ---------------------------------------------------------------------------------------------
// Q4_K
// ---------------------------------------------------------------------------------------------
// make_qkx2_quants(n = 32, nmax = 15, rmin = -1, rdelta = 0.1, nstep = 20, squared error): the weighted least-squares
// search for (scale, min) of one sub-block. Returns the scale; *the_min = -min. This plain form serves the sub-blocks whose
// range is too near the ends of the f32 range for the bounds of the register form below, and those with a NaN or an infinity.
__device__ __noinline__ float search_scale_min_q4(const float* x, const float* weights, uint8_t* L, float* the_min) {
    constexpr int n = 32, nmax = 15, nstep = 20;
    const float rmin = -1.0f, rdelta = 0.1f;
    float mn = x[0], mx = x[0];
    float sum_w = weights[0];
    float sum_x = sum_w * x[0];
    for (int i = 1; i < n; ++i) {
        mn = fminf(mn, x[i]);
        mx = fmaxf(mx, x[i]);
        sum_w += weights[i];
        sum_x = weights[i] * x[i] + sum_x;
    }
    if (mn > 0.0f) mn = 0.0f;
    if (mx == mn) {
        for (int i = 0; i < n; ++i) L[i] = 0;
        *the_min = -mn;
        return 0.0f;
    }
    float iscale = (float)nmax / (mx - mn);
    float scale = 1.0f / iscale;
    float best_error = 0.0f;
    for (int i = 0; i < n; ++i) {
        const int li = clampi(nearest_int_mul(iscale, x[i] - mn), 0, nmax);
        L[i] = (uint8_t)li;
        float diff = (scale * (float)li + mn) - x[i];
        diff = diff * diff;
        best_error = weights[i] * diff + best_error;
    }
    uint8_t laux[n];
    for (int is = 0; is <= nstep; ++is) {
        iscale = ((rdelta * (float)is + rmin) + (float)nmax) / (mx - mn);
        float sum_l = 0.0f, sum_l2 = 0.0f, sum_xl = 0.0f;
        for (int i = 0; i < n; ++i) {
            const int li = clampi(nearest_int_mul(iscale, x[i] - mn), 0, nmax);
            laux[i] = (uint8_t)li;
            const float wl = weights[i] * (float)li;
            sum_l += wl;
            sum_l2 = wl * (float)li + sum_l2;
            sum_xl = wl * x[i] + sum_xl;
        }
        const float d = sum_w * sum_l2 - sum_l * sum_l;
        if (d > 0.0f) {
            float this_scale = -(sum_x * sum_l - sum_w * sum_xl) / d;
            float this_min = (sum_l2 * sum_x - sum_l * sum_xl) / d;
            if (this_min > 0.0f) {
                this_min = 0.0f;
                this_scale = sum_xl / sum_l2;
            }
            float cur_error = 0.0f;
            for (int i = 0; i < n; ++i) {
                float diff = (this_scale * (float)laux[i] + this_min) - x[i];
                diff = diff * diff;
                cur_error = weights[i] * diff + cur_error;
            }
            if (cur_error < best_error) {
                for (int i = 0; i < n; ++i) L[i] = laux[i];
                best_error = cur_error;
                scale = this_scale;
                mn = this_min;
            }
        }
    }
    *the_min = -mn;
    return scale;
}

__device__ __forceinline__ void scale_min_k4(int j, const uint8_t* q, int& sc, int& m) {  // utils.rs:119-129
    if (j < 4) {
        sc = q[j] & 63;
        m = q[j + 4] & 63;
    } else {
        sc = (q[j + 4] & 0xF) | ((q[j - 4] >> 6) << 4);
        m = (q[j + 4] >> 4) | ((q[j] >> 6) << 4);
    }
}

// clampi(nearest_int_mul(iscale, xm), 0, 15) as a float; HIGH: the product may be above 15
template <bool HIGH> __device__ __forceinline__ float q4_level(float iscale, float xm) {
    const float l = fmaxf(iscale * xm + ROUNDING_MAGIC, ROUNDING_MAGIC) - ROUNDING_MAGIC;
    return HIGH ? fminf(l, 15.0f) : l;
}
// The same search with the sub-block in registers, levels as floats. The candidates depend on one another (a better one moves
// the minimum that the next one's levels start from), so all 21 run, in the reference's order; about 18 f32 operations per value
// and candidate are what this kernel is made of (14336 x 4096: 1262 us with a superblock per thread in local memory, 864 now; the
// f32 pipe alone would need about 640). *bad: the range left the band in which a level's product is below 2^22 (then the
// integer form above decides); *best_iscale, *best_mn: what the winning levels were made with.
__device__ __forceinline__ float search_scale_min_q4_regs(const float (&x)[32], const float (&w)[32], float mn, float mx, float* the_min,
                                                          float* best_iscale, float* best_mn, bool* bad) {
    float best_error = 0.0f, sum_w = 0.0f, sum_x = 0.0f;
    float iscale = 15.0f / (mx - mn);
    float scale = 1.0f / iscale;
    *best_iscale = iscale;
    *best_mn = mn;
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        sum_w = i == 0 ? w[0] : sum_w + w[i];
        sum_x = i == 0 ? w[0] * x[0] : w[i] * x[i] + sum_x;
        float diff = (scale * q4_level<true>(iscale, x[i] - mn) + mn) - x[i];
        diff = diff * diff;
        best_error = w[i] * diff + best_error;
    }
    auto candidate = [&](auto clamp_high, int is) {
        const float range = mx - mn;
        if (!(range > 1e-36f)) *bad = true;
        iscale = ((0.1f * (float)is + -1.0f) + 15.0f) / range;
        float l[32];
        float sum_l = 0.0f, sum_l2 = 0.0f, sum_xl = 0.0f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            l[i] = q4_level<decltype(clamp_high)::value>(iscale, x[i] - mn);
            const float wl = w[i] * l[i];
            sum_l += wl;
            sum_l2 = wl * l[i] + sum_l2;
            sum_xl = wl * x[i] + sum_xl;
        }
        const float d = sum_w * sum_l2 - sum_l * sum_l;
        float this_scale = -(sum_x * sum_l - sum_w * sum_xl) / d;
        float this_min = (sum_l2 * sum_x - sum_l * sum_xl) / d;
        if (this_min > 0.0f) {
            this_min = 0.0f;
            this_scale = sum_xl / sum_l2;
        }
        float err = 0.0f;
#pragma unroll
        for (int i = 0; i < 32; ++i) {
            float diff = (this_scale * l[i] + this_min) - x[i];
            diff = diff * diff;
            err = w[i] * diff + err;
        }
        if (d > 0.0f && err < best_error) {
            best_error = err;
            scale = this_scale;
            *best_iscale = iscale;
            *best_mn = mn;
            mn = this_min;
        }
    };
    // up to candidate 10 the largest product is 15 (1 + 2u), which rounds to 15 by itself
#pragma unroll 1
    for (int is = 0; is <= 10; ++is) candidate(std::false_type{}, is);
#pragma unroll 1
    for (int is = 11; is <= 20; ++is) candidate(std::true_type{}, is);
    *the_min = -mn;
    return scale;
}

// One lane per sub-block, eight lanes per superblock.
constexpr int Q4_CTA_THREADS = 128;
__global__ void __launch_bounds__(Q4_CTA_THREADS, 4) quantize_q4_k_kernel(const float* __restrict__ xs, uint8_t* __restrict__ out, long long nblocks,
                                                                       int vec_in, int vec_out) {
    __shared__ uint8_t slow_l[Q4_CTA_THREADS][32];  // levels of sub-blocks that took the plain search
    const int tid = threadIdx.x, j = tid & 7;
    const long long b_raw = ((long long)blockIdx.x * Q4_CTA_THREADS + tid) >> 3;
    const bool valid = b_raw < nblocks;
    const long long b = valid ? b_raw : nblocks - 1;  // (the lanes of a warp stay together: shuffles below)
    const float* src = xs + b * QK_K + 32 * j;
    float x[32], w[32];
    float sumsq = 0.0f, mn, mx;
    if (vec_in) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(src) + i);
            x[4 * i] = t.x; x[4 * i + 1] = t.y; x[4 * i + 2] = t.z; x[4 * i + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 32; ++i) x[i] = src[i];
    }
    mn = mx = x[0];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        sumsq = sumsq + x[i] * x[i];  // k_quants.rs:302-305
        mn = fminf(mn, x[i]);
        mx = fmaxf(mx, x[i]);
    }
    {
        const float av_x = sqrtf(sumsq / 32.0f);
#pragma unroll
        for (int i = 0; i < 32; ++i) w[i] = av_x + fabsf(x[i]);
    }
    if (mn > 0.0f) mn = 0.0f;
    float scale, the_min, best_iscale, best_mn;
    bool plain = !(sumsq < 1e35f);  // (false for a NaN as well)
    if (mx == mn) {
        scale = 0.0f;
        the_min = -mn;
        best_iscale = 0.0f;
        best_mn = 0.0f;
    } else {
        scale = search_scale_min_q4_regs(x, w, mn, mx, &the_min, &best_iscale, &best_mn, &plain);
        if (plain) {
            float xv[32], wv[32];
            for (int i = 0; i < 32; ++i) {
                xv[i] = x[i];
                wv[i] = w[i];
            }
            scale = search_scale_min_q4(xv, wv, slow_l[tid], &the_min);
        }
    }
    float max_scale = fmaxf(scale, 0.0f), max_min = fmaxf(the_min, 0.0f);
#pragma unroll
    for (int m = 4; m > 0; m >>= 1) {
        max_scale = fmaxf(max_scale, __shfl_xor_sync(0xffffffffu, max_scale, m));
        max_min = fmaxf(max_min, __shfl_xor_sync(0xffffffffu, max_min, m));
    }
    const float inv_scale = max_scale > 0.0f ? 63.0f / max_scale : 0.0f;
    const float inv_min = max_min > 0.0f ? 63.0f / max_min : 0.0f;
    const int lsi = nearest_int_mul(inv_scale, scale);
    const int lmi = nearest_int_mul(inv_min, the_min);
    const unsigned ls = (uint8_t)(lsi < 63 ? lsi : 63), lm = (uint8_t)(lmi < 63 ? lmi : 63);
    // every lane of the superblock builds the twelve bytes of packed 6-bit scales and mins (utils.rs:119-129 read backwards)
    uint32_t sc_w = 0, m_w = 0, hi_w = 0;
    {
        const unsigned mine = ls | (lm << 8);
        const int base = (tid & 31) & ~7;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const unsigned a = __shfl_sync(0xffffffffu, mine, base + q), c = __shfl_sync(0xffffffffu, mine, base + 4 + q);
            const unsigned als = a & 0xffu, alm = a >> 8, cls = c & 0xffu, clm = c >> 8;
            sc_w |= ((als | ((cls >> 4) << 6)) & 0xffu) << (8 * q);
            m_w |= ((alm | ((clm >> 4) << 6)) & 0xffu) << (8 * q);
            hi_w |= (((cls & 0xFu) | ((clm & 0xFu) << 4)) & 0xffu) << (8 * q);
        }
    }
    const unsigned short dh = f16_bits(max_scale / 63.0f), mh = f16_bits(max_min / 63.0f);
    const float dv = f16_value(dh), mv = f16_value(mh);
    // the scale and min as they are stored, and every value again against them (k_quants.rs:1995-2005)
    int sc, m;
    {
        const uint32_t words[3] = {sc_w, m_w, hi_w};
        uint8_t packed[12];
#pragma unroll
        for (int i = 0; i < 12; ++i) packed[i] = (uint8_t)(words[i >> 2] >> (8 * (i & 3)));
        // (both decodings, selected: j differs between the lanes)
        int sc_lo = 0, m_lo = 0, sc_hi = 0, m_hi = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            int s0, m0, s1, m1;
            scale_min_k4(q, packed, s0, m0);
            scale_min_k4(q + 4, packed, s1, m1);
            if ((j & 3) == q) {
                sc_lo = s0; m_lo = m0; sc_hi = s1; m_hi = m1;
            }
        }
        sc = j < 4 ? sc_lo : sc_hi;
        m = j < 4 ? m_lo : m_hi;
    }
    const float d = dv * (float)sc, dm = mv * (float)m;
    uint32_t lw[8];
    if (d != 0.0f) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            lw[i] = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) lw[i] |= (uint32_t)clampi(nearest_int((x[4 * i + q] + dm) / d), 0, 15) << (8 * q);
        }
    } else {
        // a sub-block whose stored scale is zero keeps the levels of its search
        const bool from_plain = plain && mx != mn;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            lw[i] = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int e = 4 * i + q;
                const uint32_t level = mx == mn ? 0u : (from_plain ? (uint32_t)slow_l[tid][e] : (uint32_t)(int)q4_level<true>(best_iscale, x[e] - best_mn));
                lw[i] |= level << (8 * q);
            }
        }
    }
    // sub-blocks 2c and 2c + 1 share 32 bytes, low and high nibbles: each of the two lanes writes one half
    uint32_t o4[4];
    const bool odd = (j & 1) != 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const uint32_t got = __shfl_xor_sync(0xffffffffu, odd ? lw[i] : lw[4 + i], 1);
        o4[i] = odd ? (got | (lw[4 + i] << 4)) : (lw[i] | (got << 4));
    }
    if (!valid) return;
    uint8_t* o = out + b * Q4_K_BYTES;
    uint8_t* oq = o + 16 + 32 * (j >> 1) + (odd ? 16 : 0);
    const uint32_t head[4] = {(uint32_t)dh | ((uint32_t)mh << 16), sc_w, m_w, hi_w};
    if (vec_out) {
        *reinterpret_cast<uint4*>(oq) = make_uint4(o4[0], o4[1], o4[2], o4[3]);
        if (j == 0) *reinterpret_cast<uint4*>(o) = make_uint4(head[0], head[1], head[2], head[3]);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            reinterpret_cast<unsigned short*>(oq)[2 * i] = (unsigned short)o4[i];
            reinterpret_cast<unsigned short*>(oq)[2 * i + 1] = (unsigned short)(o4[i] >> 16);
            if (j == 0) {
                reinterpret_cast<unsigned short*>(o)[2 * i] = (unsigned short)head[i];
                reinterpret_cast<unsigned short*>(o)[2 * i + 1] = (unsigned short)(head[i] >> 16);
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// Q6_K
// ---------------------------------------------------------------------------------------------
// make_qx_quants(n = 16, nmax = 32, rmse_type = 1, no importance weights): weights x^2, 18 nudged candidates.
__device__ __noinline__ float search_scale_q6(const float* x, int8_t* ls) {
    constexpr int n = 16, nmax = 32;
    float mx = 0.0f, amax = 0.0f;
    for (int i = 0; i < n; ++i) {
        if (fabsf(x[i]) > amax) {
            amax = fabsf(x[i]);
            mx = x[i];
        }
    }
    if (amax < GROUP_MAX_EPS) {
        for (int i = 0; i < n; ++i) ls[i] = 0;
        return 0.0f;
    }
    float iscale = -(float)nmax / mx;
    float w[n];
    for (int i = 0; i < n; ++i) w[i] = x[i] * x[i];
    float sumlx = 0.0f, suml2 = 0.0f;
    for (int i = 0; i < n; ++i) {
        const float l = (float)clampi(nearest_int_mul(iscale, x[i]), -nmax, nmax - 1);
        sumlx = (w[i] * x[i]) * l + sumlx;
        suml2 = (w[i] * l) * l + suml2;
    }
    for (int i = 0; i < n; ++i) ls[i] = (int8_t)(nmax + clampi(nearest_int_mul(iscale, x[i]), -nmax, nmax - 1));
    float scale = suml2 != 0.0f ? sumlx / suml2 : 0.0f;
    float best = scale * sumlx;
    for (int is = -9; is <= 9; ++is) {
        if (is == 0) continue;
        const float isc = -(0.1f * (float)is + (float)nmax) / mx;
        sumlx = 0.0f;
        suml2 = 0.0f;
        for (int i = 0; i < n; ++i) {
            const float l = (float)clampi(nearest_int_mul(isc, x[i]), -nmax, nmax - 1);
            sumlx = w[i] * x[i] * l + sumlx;
            suml2 = w[i] * l * l + suml2;
        }
        if (suml2 > 0.0f && sumlx * sumlx > best * suml2) {
            for (int i = 0; i < n; ++i) ls[i] = (int8_t)(nmax + clampi(nearest_int_mul(isc, x[i]), -nmax, nmax - 1));
            scale = sumlx / suml2;
            best = scale * sumlx;
        }
    }
    return scale;
}

// The same search on 16 values in registers, the levels as floats; *best_is: the candidate whose levels won (0: the first).
// Every candidate has to run in the reference's order here: the test is against a running product, not an error.
__device__ __forceinline__ float q6_candidate_iscale(int is, float mx) {
    return is == 0 ? -32.0f / mx : -(0.1f * (float)is + 32.0f) / mx;
}
__device__ __forceinline__ float q6_level(float iscale, float x) {  // clampi(nearest_int_mul(iscale, x), -32, 31) as a float
    return fminf(fmaxf((iscale * x + ROUNDING_MAGIC) - ROUNDING_MAGIC, -32.0f), 31.0f);
}
__device__ __forceinline__ float search_scale_q6_regs(const float (&x)[16], float mx, int* best_is) {
    float w[16], wx[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        w[i] = x[i] * x[i];
        wx[i] = w[i] * x[i];
    }
    float scale = 0.0f, best = 0.0f;
    *best_is = 0;
#pragma unroll 1
    for (int it = 0; it < 19; ++it) {  // the first guess, then -9 .. -1, 1 .. 9
        const int is = it == 0 ? 0 : (it <= 9 ? it - 10 : it - 9);
        const float isc = q6_candidate_iscale(is, mx);
        float sumlx = 0.0f, suml2 = 0.0f;
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const float l = q6_level(isc, x[i]);
            sumlx = wx[i] * l + sumlx;
            suml2 = (w[i] * l) * l + suml2;
        }
        if (it == 0) {
            scale = suml2 != 0.0f ? sumlx / suml2 : 0.0f;
            best = scale * sumlx;
        } else if (suml2 > 0.0f && sumlx * sumlx > best * suml2) {
            *best_is = is;
            scale = sumlx / suml2;
            best = scale * sumlx;
        }
    }
    return scale;
}

// One lane per 16 values, sixteen lanes per superblock.
constexpr int Q6_CTA_THREADS = 128;
__global__ void __launch_bounds__(Q6_CTA_THREADS) quantize_q6_k_kernel(const float* __restrict__ xs, uint8_t* __restrict__ out, long long nblocks,
                                                                       int vec_in) {
    __shared__ int8_t slow_l[Q6_CTA_THREADS][16];  // levels of groups that took the plain search
    const int tid = threadIdx.x, ib = tid & 15;
    const long long b_raw = ((long long)blockIdx.x * Q6_CTA_THREADS + tid) >> 4;
    const bool valid = b_raw < nblocks;
    const long long b = valid ? b_raw : nblocks - 1;  // (the lanes of a warp stay together: shuffles below)
    const float* src = xs + b * QK_K + 16 * ib;
    float x[16];
    if (vec_in) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = __ldg(reinterpret_cast<const float4*>(src) + i);
            x[4 * i] = t.x; x[4 * i + 1] = t.y; x[4 * i + 2] = t.z; x[4 * i + 3] = t.w;
        }
    } else {
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = src[i];
    }
    float mx = 0.0f, amax = 0.0f, zero = 0.0f;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const float a = fabsf(x[i]);
        if (a > amax) {
            amax = a;
            mx = x[i];
        }
        zero += x[i] * 0.0f;  // NaN where a value is infinite or NaN
    }
    float scale;
    int best_is = 0;
    bool from_plain = false;
    const bool none = amax < GROUP_MAX_EPS;
    if (zero == 0.0f) {
        scale = none ? 0.0f : search_scale_q6_regs(x, mx, &best_is);
    } else {
        float xv[16];
        for (int i = 0; i < 16; ++i) xv[i] = x[i];
        scale = search_scale_q6(xv, slow_l[tid]);
        from_plain = true;
    }
    // the scale of largest magnitude, the first of equals (the reference walks the groups in order)
    float max_abs = fabsf(scale) > 0.0f ? fabsf(scale) : 0.0f, max_scale = max_abs > 0.0f ? scale : 0.0f;
    int who = ib;
#pragma unroll
    for (int m = 8; m > 0; m >>= 1) {
        const float oa = __shfl_xor_sync(0xffffffffu, max_abs, m), os = __shfl_xor_sync(0xffffffffu, max_scale, m);
        const int ow = __shfl_xor_sync(0xffffffffu, who, m);
        if (oa > max_abs || (oa == max_abs && ow < who)) {
            max_abs = oa;
            max_scale = os;
            who = ow;
        }
    }
    // an all-zero superblock gives max_scale = 0, iscale = -inf, d = f16(-0.0), scales 0: as the reference
    const float iscale = -128.0f / max_scale;
    const unsigned short dh = f16_bits(1.0f / iscale);
    const float dv = f16_value(dh);
    // (-inf * 0 is a NaN whose mantissa bits differ between machines: the reference's host turns it into scale 0)
    const int sv = max_abs == 0.0f ? 0 : nearest_int_mul(iscale, scale);
    const int8_t sc8 = (int8_t)(sv < 127 ? sv : 127);
    const float d = dv * (float)sc8;
    uint32_t lw[4];  // sixteen 6-bit levels, four to a word
    if (d != 0.0f) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            lw[i] = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) lw[i] |= (uint32_t)(clampi(nearest_int(x[4 * i + q] / d), -32, 31) + 32) << (8 * q);
        }
    } else {
        // a group whose stored scale is zero keeps the levels of its search
        const float isc = q6_candidate_iscale(best_is, mx);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            lw[i] = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int e = 4 * i + q;
                const uint32_t level = from_plain ? (uint32_t)(uint8_t)slow_l[tid][e] : (none ? 0u : (uint32_t)((int)q6_level(isc, x[e]) + 32));
                lw[i] |= (level & 0xffu) << (8 * q);
            }
        }
    }
    // group ib is half h = ib >> 3, quarter qd, 16-value part g of it. ql byte (qd & 1, g, i) = low nibbles of quarters qd and
    // qd ^ 2, qh byte (g, i) = the high two bits of all four quarters: lanes 4 and 2, 4 apart exchange
    const int qd = (ib >> 1) & 3, g = ib & 1, h = ib >> 3;
    uint32_t ql[2], qh = 0;
    {
        uint32_t lo[4], hi[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            lo[i] = lw[i] & 0x0f0f0f0fu;
            hi[i] = ((lw[i] >> 4) & 0x03030303u) << (2 * qd);
        }
        const bool upper = qd >= 2;  // writes the second eight bytes of the sixteen that the two lanes share
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint32_t got = __shfl_xor_sync(0xffffffffu, upper ? lo[i] : lo[2 + i], 4);
            ql[i] = upper ? (got | (lo[2 + i] << 4)) : (lo[i] | (got << 4));
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t t = hi[i] | __shfl_xor_sync(0xffffffffu, hi[i], 2);
            t |= __shfl_xor_sync(0xffffffffu, t, 4);
            if (i == qd) qh = t;  // lane qd writes word qd
        }
    }
    if (!valid) return;
    uint8_t* o = out + b * Q6_K_BYTES;  // 2-byte aligned
    unsigned short* oql = reinterpret_cast<unsigned short*>(o + 64 * h + 32 * (qd & 1) + 16 * g + (qd >= 2 ? 8 : 0));
    unsigned short* oqh = reinterpret_cast<unsigned short*>(o + 128 + 32 * h + 16 * g + 4 * qd);
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        oql[2 * i] = (unsigned short)ql[i];
        oql[2 * i + 1] = (unsigned short)(ql[i] >> 16);
        oqh[i] = (unsigned short)(qh >> (16 * i));
    }
    o[192 + ib] = (uint8_t)sc8;
    if (ib == 0) *reinterpret_cast<unsigned short*>(o + 208) = dh;
}

// ---------------------------------------------------------------------------------------------
// to_float and the row gather: one thread per 8 consecutive values, so that neighbouring lanes write neighbouring 16 or 32
// bytes; HBM-bound (a thread per 32 values wrote 64-byte strides with 2-byte stores: 62 us for 2048 rows of 4096 Q6_K values,
// now under the 15 us that the call costs the host).
// ---------------------------------------------------------------------------------------------
// Eight values of row `row` from value 8 c on. AL: the packed bytes are 16-byte aligned (Q4_K) / 2-byte aligned (the others);
// without it they are read one by one.
template <bool AL>
__device__ __forceinline__ uint32_t packed_u16(const uint8_t* p) {
    if constexpr (AL) return (uint32_t)__ldg(reinterpret_cast<const unsigned short*>(p));
    else return (uint32_t)p[0] | ((uint32_t)p[1] << 8);
}
template <int TYPE, bool AL>
__device__ __forceinline__ void dequant8(const uint8_t* row, int c, float (&v)[8]) {
    if constexpr (TYPE == TYPE_Q8_0) {
        const uint8_t* blk = row + (size_t)(c >> 2) * Q8_0_BYTES;
        const float d = f16_value((unsigned short)packed_u16<AL>(blk));
        const uint8_t* q = blk + 2 + 8 * (c & 3);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t two = packed_u16<AL>(q + 2 * i);
            v[2 * i] = (float)(int)(int8_t)(two & 0xffu) * d;
            v[2 * i + 1] = (float)(int)(int8_t)(two >> 8) * d;
        }
    } else if constexpr (TYPE == TYPE_Q4_K) {
        const uint8_t* sb = row + (size_t)(c >> 5) * Q4_K_BYTES;
        const int j = (c >> 2) & 7;
        const uint8_t* q = sb + 16 + 32 * (j >> 1) + 8 * (c & 3);
        uint32_t hdr[4], w[2];
        if constexpr (AL) {
            const uint4 t = __ldg(reinterpret_cast<const uint4*>(sb));
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(q));
            hdr[0] = t.x; hdr[1] = t.y; hdr[2] = t.z; hdr[3] = t.w;
            w[0] = u.x; w[1] = u.y;
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) hdr[i] = packed_u16<false>(sb + 4 * i) | (packed_u16<false>(sb + 4 * i + 2) << 16);
#pragma unroll
            for (int i = 0; i < 2; ++i) w[i] = packed_u16<false>(q + 4 * i) | (packed_u16<false>(q + 4 * i + 2) << 16);
        }
        const int sh = 8 * (j & 3);
        const uint32_t a = (hdr[1] >> sh) & 0xffu, b = (hdr[2] >> sh) & 0xffu, e = (hdr[3] >> sh) & 0xffu;
        const uint32_t sc = j < 4 ? (a & 63u) : ((e & 0xFu) | ((a >> 6) << 4)), m = j < 4 ? (b & 63u) : ((e >> 4) | ((b >> 6) << 4));
        const float d1 = f16_value((unsigned short)hdr[0]) * (float)(int)sc, m1 = f16_value((unsigned short)(hdr[0] >> 16)) * (float)(int)m;
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = d1 * (float)(int)((w[i >> 2] >> (8 * (i & 3) + 4 * (j & 1))) & 0xFu) - m1;
    } else {
        const uint8_t* sb = row + (size_t)(c >> 5) * Q6_K_BYTES;
        const int n = (c >> 4) & 1, qd = (c >> 2) & 3, l0 = 8 * (c & 3);
        const float d = f16_value((unsigned short)packed_u16<AL>(sb + 208)) * (float)(int)(int8_t)sb[192 + 8 * n + 2 * qd + (l0 >> 4)];
        const uint8_t* ql = sb + 64 * n + 32 * (qd & 1) + l0;
        const uint8_t* qh = sb + 128 + 32 * n + l0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const uint32_t lo = packed_u16<AL>(ql + 2 * i) >> (4 * (qd >> 1)), hi = packed_u16<AL>(qh + 2 * i) >> (2 * qd);
            v[2 * i] = d * (float)((int)((lo & 0xFu) | ((hi & 3u) << 4)) - 32);
            v[2 * i + 1] = d * (float)((int)(((lo >> 8) & 0xFu) | (((hi >> 8) & 3u) << 4)) - 32);
        }
    }
}

template <typename T>
__device__ __forceinline__ void store8(T* dst, const float (&v)[8], bool vec) {
    if (vec) {
        if constexpr (sizeof(T) == 4) {
            reinterpret_cast<float4*>(dst)[0] = make_float4(v[0], v[1], v[2], v[3]);
            reinterpret_cast<float4*>(dst)[1] = make_float4(v[4], v[5], v[6], v[7]);
        } else {
            __align__(16) T t[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] = from_float<T>(v[i]);
            *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(t);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) dst[i] = from_float<T>(v[i]);
    }
}

// ids == nullptr: row i of the output is row i of the matrix (to_float); else row ids[i] (get_rows). A CTA takes
// DEQUANT_CHUNKS chunks of 8 values of the output, rows one after the other; `vec`: the output is 16-byte aligned.
constexpr int DEQUANT_PER_THREAD = 4, DEQUANT_CHUNKS = 256 * DEQUANT_PER_THREAD;
template <typename T, int TYPE, bool AL>
__global__ void __launch_bounds__(256) dequant_rows_kernel(const uint8_t* __restrict__ w, const int* __restrict__ ids, T* __restrict__ out,
                                                           long long nrows_out, int K, long long nrows_w, int vec, unsigned int* status) {
    const int per_row = K / 8;
    const long long base = (long long)blockIdx.x * DEQUANT_CHUNKS;
    const long long row0 = base / per_row;
    const int off0 = (int)(base - row0 * per_row);
    const size_t row_bytes = (size_t)(K / type_block_elems(TYPE)) * type_block_bytes(TYPE);
#pragma unroll
    for (int u = 0; u < DEQUANT_PER_THREAD; ++u) {
        const int i = off0 + u * 256 + (int)threadIdx.x;  // below per_row + DEQUANT_CHUNKS
        const int dr = i / per_row, c = i - dr * per_row;
        const long long r = row0 + dr;
        if (r >= nrows_out) return;
        const long long src = ids != nullptr ? (long long)__ldg(ids + r) : r;
        float v[8];
        if (src < 0 || src >= nrows_w) {  // an id outside the table: zeros, and the status word says so
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = 0.0f;
            if (c == 0) record_failure(status, STATUS_BAD_ROW_ID, (unsigned int)r);
        } else {
            dequant8<TYPE, AL>(w + (size_t)src * row_bytes, c, v);
        }
        store8<T>(out + r * K + (long long)c * 8, v, vec != 0);
    }
}

int quantize_weights(int type, const float* x, void* out, long long n, cudaStream_t s) {
    if (type_block_bytes(type) == 0) return B200Q_ERR_UNSUPPORTED;
    if (n < 0 || n % type_block_elems(type) != 0 || reinterpret_cast<uintptr_t>(out) % 2 != 0) return B200Q_ERR_INVALID;
    if (n == 0) return 0;
    const long long nb = n / type_block_elems(type);
    const int vec_in = reinterpret_cast<uintptr_t>(x) % 16 == 0, vec_out = reinterpret_cast<uintptr_t>(out) % 16 == 0;
    uint8_t* o = static_cast<uint8_t*>(out);
    const auto ctas = [](long long items, int per_cta) { return (unsigned)((items + per_cta - 1) / per_cta); };
    if (type == TYPE_Q8_0) quantize_q8_0_kernel<<<ctas(nb, Q8_CTA_BLOCKS), 256, 0, s>>>(x, o, nb, vec_in, vec_out);
    else if (type == TYPE_Q4_K) quantize_q4_k_kernel<<<ctas(8 * nb, Q4_CTA_THREADS), Q4_CTA_THREADS, 0, s>>>(x, o, nb, vec_in, vec_out);
    else quantize_q6_k_kernel<<<ctas(16 * nb, Q6_CTA_THREADS), Q6_CTA_THREADS, 0, s>>>(x, o, nb, vec_in);
    return (int)cudaGetLastError();
}

template <typename T>
static int launch_dequant_rows(int type, const void* w, const int* ids, void* out, long long nrows_out, int K, long long nrows_w, cudaStream_t s) {
    const unsigned grid = (unsigned)((nrows_out * (K / 8) + DEQUANT_CHUNKS - 1) / DEQUANT_CHUNKS);
    const uint8_t* wp = static_cast<const uint8_t*>(w);
    const int vec = reinterpret_cast<uintptr_t>(out) % 16 == 0;
    const bool aligned = reinterpret_cast<uintptr_t>(w) % (type == TYPE_Q4_K ? 16 : 2) == 0;
    const auto launch = [&](auto kernel) {
        kernel<<<grid, 256, 0, s>>>(wp, ids, static_cast<T*>(out), nrows_out, K, nrows_w, vec, status_ptr());
        return (int)cudaGetLastError();
    };
    if (type == TYPE_Q8_0) return aligned ? launch(dequant_rows_kernel<T, TYPE_Q8_0, true>) : launch(dequant_rows_kernel<T, TYPE_Q8_0, false>);
    if (type == TYPE_Q4_K) return aligned ? launch(dequant_rows_kernel<T, TYPE_Q4_K, true>) : launch(dequant_rows_kernel<T, TYPE_Q4_K, false>);
    return aligned ? launch(dequant_rows_kernel<T, TYPE_Q6_K, true>) : launch(dequant_rows_kernel<T, TYPE_Q6_K, false>);
}

int dequantize_rows(int type, int elem, const void* w, const int* ids, void* out, long long nrows_out, int K, long long nrows_w,
                    cudaStream_t s) {
    if (type_block_bytes(type) == 0) return B200Q_ERR_UNSUPPORTED;
    if (K <= 0 || K % type_block_elems(type) != 0 || nrows_out < 0 || nrows_w < 0) return B200Q_ERR_INVALID;
    if (nrows_out == 0) return 0;
    if (elem == ELEM_F32) return launch_dequant_rows<float>(type, w, ids, out, nrows_out, K, nrows_w, s);
    if (elem == ELEM_F16) return launch_dequant_rows<__half>(type, w, ids, out, nrows_out, K, nrows_w, s);
    if (elem == ELEM_BF16) return launch_dequant_rows<__nv_bfloat16>(type, w, ids, out, nrows_out, K, nrows_w, s);
    return B200Q_ERR_INVALID;
}

}  // namespace b200q
