// Small batches (1..16 activation rows) on the integer tensor cores: every packed weight block is read from HBM once and decoded
// once for all rows. Takes the place of the reference's tensor-core matvec tier: host side fast_mmvq::tiled_plain
// (crates/inference-quant/src/gguf/fast_mmvq.rs:2049-2126), activation layout kernel mmvq_tc_quantize
// (crates/inference-quant/kernels/cuda/mmvq_gguf/mmvq_quantize.cu:157-190), matvec mmvq_tc_k_kernel
// (crates/inference-quant/kernels/cuda/mmvq_gguf/mmvq_tc_k.cuh:221-329). Same arithmetic as there: activations become int8 with one
// scale per 32 values (d = amax / 127 stored as f16, q = roundf(x / d), integer block sums for the min term), the dot products of
// one scale's values are exact integers, and scales are applied in f32.
//
// Two launches:
//   1. tcq_quantize_kernel: x [M][K] -> int8 quants in the order of the MMA's A fragments, and (d, d * sum q) per block and row.
//   2. gemv_rows_kernel: a CTA owns a run of 16-row tiles. A warp takes two tiles and every W_k-th 256-k superblock of them; its own
//      ring of TMA boxes (no other warp involved) brings the packed bytes, the warp turns them into MMA fragments in registers,
//      multiplies 16 x 8 x 32 (Q6_K, whose scales cover 16 values: 16 x 8 x 16), and applies the scales to the sums where they are:
//      in its registers. The W_k warps of a tile pair add up through shared memory in a fixed order (bit-reproducible).
//
// Bound by latency and issue slots of the unpacking and scaling before HBM (ncu, 28672 rows of Q4_K, 8 activation
// rows: 2.3 of 6.6 TB/s, an instruction on 0.36 of the cycles). What keeps the instructions few: sums come out of the MMA as floats (the
// accumulator starts at the bits of 1.5 * 2^23, so an exact subtraction takes the place of a conversion), scaling works on pairs of
// weight rows (fma.f32x2), a row's block scales are decoded by one lane and passed on through shared memory. mma.sync and not tcgen05: scales differ from block to
// block, so a sum may not stay in the accumulator for more than 32 values; with tcgen05 every such sum goes out to TMEM and back, and
// eight MMAs of 128 x 16 x 32 with their five barrier hand-offs per 256 k took 1400 cycles where HBM needs 420. Both launches,
// matrices out of HBM, tcgen05 -> this: 4096 x 28672 Q4_K 5 rows 36.6 -> 26.2 us, 16 rows 47.1 -> 32.9; 14336 x 4096 Q6_K 16 rows
// 51.4 -> 25.7; 4096 x 1024 Q4_K 16 rows 22.1 -> 7.5.
//
// Every wait is bounded; a wait that gives up records a code in the device status word, and work is skipped.
#include "common.cuh"
#include "runtime.h"
#include "tcgen05.cuh"

namespace b200q {

constexpr int TCQ_TOKENS = 16;
constexpr int TCQ_KC = 256;                     // k per superblock: one box
constexpr int TCQ_ROWS = 16;                    // weight rows of a tile
constexpr int TCQ_MAX_CTAS = 160;               // K-split mode: at most one CTA per SM
constexpr int TCQ_COUNTERS = TCQ_MAX_CTAS;      // one per tile
constexpr size_t TCQ_PARTIAL_BYTES = (size_t)TCQ_MAX_CTAS * TCQ_ROWS * TCQ_TOKENS * sizeof(float);  // sum over tiles of ksplit * 16 * rows
// A warp's record of block scales: per pair of rows and block the float4 (row, row + 1) x (factor, second factor), 144 bytes from pair
// to pair; after the last superblock of its rows, their partial sums [16 activation rows][32 rows], 40 floats from row to row (so that
// the eight lanes that write a column fall on different banks).
constexpr int TCQ_REC_PITCH = 144;
constexpr int TCQ_SUM_PITCH = 40;
constexpr int TCQ_EXCH_BYTES = TCQ_TOKENS * TCQ_SUM_PITCH * 4;
static_assert(TCQ_ROWS * TCQ_REC_PITCH <= TCQ_EXCH_BYTES, "sixteen pairs of rows");

// DEPTH stages in flight per warp, each one superblock of up to two tiles. Boxes of 32 rows: a matrix of 28672 rows of 2304 bytes
// comes in in 16 us that way, in 21 us by boxes of 16 rows. Shared memory stays under 195 KB where it can: the rest is the L1 through
// which the warps of a CTA share the activation fragments. Q8_0 has half the instructions per byte, so half the warps.
template <int TYPE> struct TcqType;
template <> struct TcqType<TYPE_Q4_K> { static constexpr int PITCH = 144, WARPS = 16, DEPTH = 2; };
template <> struct TcqType<TYPE_Q6_K> { static constexpr int PITCH = 240, WARPS = 12, DEPTH = 2; };  // 210 bytes from a 16-byte boundary on
template <> struct TcqType<TYPE_Q8_0> { static constexpr int PITCH = 272, WARPS = 8, DEPTH = 2; };
template <int TYPE> constexpr int TCQ_BOX_BYTES = TCQ_ROWS * TcqType<TYPE>::PITCH;
template <int TYPE>
constexpr size_t TCQ_SMEM = 128 + (size_t)TcqType<TYPE>::WARPS * (TcqType<TYPE>::DEPTH * (2 * TCQ_BOX_BYTES<TYPE> + 8) + TCQ_EXCH_BYTES) + 16;

struct TcqParams {
    void* y;               // [M][ldy]
    const uint4* acts;     // quants: [K / 256][halves][4 block pairs][lane], a lane's two registers of either block
    const float4* scales;  // [K / 256][halves][8 blocks][8 rows]: (d, d, d * sum, d * sum), the pairs the scaling multiplies with
    int M, N, K, ldy;
    int tiles_per_cta, tiles_extra;  // CTA group c owns tiles [c * q + min(c, r), ...)
    int wks;               // warps that share a tile pair's superblocks (a divisor of the CTA's)
    // matrices with too few rows to give every SM a tile are split along K as well: ksplit consecutive CTAs share a group; their
    // partial outputs meet in `partial` [ksplit][16][N] and the last to arrive (a counter per tile, zeroed by the quantize launch)
    // adds them in split order and stores
    int ksplit;
    float* partial;
    unsigned int* counters;
    unsigned int* status;
    const uint8_t* ref_acts;  // REF_ACTS kernels: the activations as the reference's mmvq_tc_quantize lays them out
};

// ---------------------------------------------------------------------------------------------
// Launch 1: a warp quantizes two 32-value blocks of eight activation rows, lane (g, t) the values 4t.. and 16 + 4t.. of row g: what
// the lane of the same number multiplies with in an MMA.
// ---------------------------------------------------------------------------------------------
template <typename src_t> __device__ __forceinline__ void tcq_load4(const src_t* p, bool vec, float* v) {
    if (vec) {
        if constexpr (sizeof(src_t) == 4) {
            const float4 f = *reinterpret_cast<const float4*>(p);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else {
            const uint2 u = *reinterpret_cast<const uint2*>(p);
            const src_t* e = reinterpret_cast<const src_t*>(&u);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[i] = to_float<src_t>(e[i]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) v[i] = to_float<src_t>(p[i]);
    }
}
template <typename src_t>
__global__ void __launch_bounds__(128) tcq_quantize_kernel(const src_t* __restrict__ x, uint4* __restrict__ q, float4* __restrict__ scales, int K, int M,
                                                           int ldx, int halves, int vec, unsigned int* __restrict__ counters) {
    // the matvec launch that follows may start now: until its own dependency wait it only sets up and streams weights
    grid_launch_dependents();
    if (blockIdx.x == 0)
        for (int c = threadIdx.x; c < TCQ_COUNTERS; c += 128) counters[c] = 0u;
    const int unit = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (unit >= K / 64 * halves) return;
    const int pair = unit / halves, h = unit - pair * halves;
    const int g = lane >> 2, t = lane & 3, row = 8 * h + g;
    const size_t slot = ((size_t)(pair >> 2) * halves + h) * 4 + (pair & 3);
    uint32_t w[4];
#pragma unroll
    for (int b = 0; b < 2; ++b) {
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = 0.0f;
        if (row < M) {
            const src_t* p = x + (size_t)row * ldx + 64 * pair + 32 * b + 4 * t;
            tcq_load4<src_t>(p, vec, v);
            tcq_load4<src_t>(p + 16, vec, v + 4);
        }
        // from the first value on, as the reference's warp maximum: a NaN among other values counts as 0, but a block of NaNs alone has
        // a NaN for a scale and makes its row's outputs NaNs
        float amax = fabsf(v[0]);
#pragma unroll
        for (int i = 1; i < 8; ++i) amax = fmaxf(amax, fabsf(v[i]));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 1));
        amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, 2));
        const float d = amax / 127.0f;
        int sum = 0;
        uint32_t u[2] = {0u, 0u};
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int qi = amax == 0.0f ? 0 : (int)roundf(v[i] / d);
            sum += qi;
            u[i >> 2] |= ((uint32_t)qi & 0xffu) << (8 * (i & 3));
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        w[2 * b] = u[0];
        w[2 * b + 1] = u[1];
        const float dh = __half2float(__float2half_rn(d));
        if (t == b) scales[(slot * 2 + b) * 8 + g] = make_float4(dh, dh, dh * (float)sum, dh * (float)sum);
    }
    q[slot * 32 + lane] = make_uint4(w[0], w[1], w[2], w[3]);
}

// The reference tier's own activation layout (crates/inference-quant/kernels/cuda/mmvq_gguf/mmvq_quantize.cu:148-190,
// mmvq_tc_act.cuh:1-7), for hosts that call launch_mmvq_tc_quantize_* / launch_mmvq_tc_gguf_*_plain as a pair: the
// rows in halves of 8, one half after the other; per half nb = gridDim.x blocks of 32 values: nb * 32 int2 (entry
// 4r + t of a block = row r's values 4t..4t+3 then 16+4t..16+4t+3), then nb * 8 f16 scales d = amax / 127, then nb * 8
// int16 sums of the quants q = roundf(x / d). One CTA per (block, half), one warp per row.
constexpr int TCQ_REF_BLOCK_BYTES = 32 * 8 + 8 * 2 + 8 * 2;  // 288
template <typename src_t>
__global__ void __launch_bounds__(256) tcq_ref_quantize_kernel(const src_t* __restrict__ x, uint8_t* __restrict__ vy, int kx, int num_rows) {
    const int ib = blockIdx.x, nb = gridDim.x, row = threadIdx.y, lane = threadIdx.x;
    const int col = ib * 32 + lane;
    const int input_row = blockIdx.y * 8 + row;
    uint8_t* base = vy + (size_t)blockIdx.y * nb * TCQ_REF_BLOCK_BYTES;
    const float xi = (input_row < num_rows && col < kx) ? to_float<src_t>(x[(size_t)input_row * kx + col]) : 0.0f;
    const float amax = warp_max(fabsf(xi));
    const float d = amax / 127.0f;
    const int qi = amax == 0.0f ? 0 : (int)roundf(xi / d);
    const int sum = __reduce_add_sync(0xffffffffu, qi);
    __shared__ __align__(8) int8_t q[8][32];
    q[row][lane] = (int8_t)qi;
    if (lane == 0) {
        reinterpret_cast<__half*>(base + (size_t)nb * 256)[ib * 8 + row] = __float2half_rn(d);
        reinterpret_cast<int16_t*>(base + (size_t)nb * 256 + (size_t)nb * 16)[ib * 8 + row] = (int16_t)sum;
    }
    __syncthreads();
    if (row == 0) {
        const int r = lane >> 2, t = lane & 3;
        reinterpret_cast<int2*>(base)[(size_t)ib * 32 + lane] =
            make_int2(*reinterpret_cast<const int*>(&q[r][4 * t]), *reinterpret_cast<const int*>(&q[r][16 + 4 * t]));
    }
}

__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

// ---------------------------------------------------------------------------------------------
// Register arithmetic
// ---------------------------------------------------------------------------------------------
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ f32x2 pack2(uint32_t a, uint32_t b) { return pack2(__uint_as_float(a), __uint_as_float(b)); }
__device__ __forceinline__ void unpack2(f32x2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// Sums of 32 / 16 products per output as the floats 1.5 * 2^23 + sum (|sum| < 2^22): activation rows g (lo) and g + 8 (hi), weight
// rows 2t, 2t + 1. The weights are the MMA's N side: the factors of a pair of rows then come out of the record as the pair that
// fma.f32x2 takes, where the other way round every factor has to be copied into both halves of a register pair.
constexpr uint32_t TCQ_MAGIC = 0x4B400000u;
__device__ __forceinline__ void mma_k32(const uint32_t (&a)[4], uint32_t b0, uint32_t b1, f32x2& lo, f32x2& hi) {
    uint32_t d[4];
    asm("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "r"(TCQ_MAGIC));
    lo = pack2(d[0], d[1]);
    hi = pack2(d[2], d[3]);
}
__device__ __forceinline__ void mma_k16(uint32_t a0, uint32_t a1, uint32_t b, f32x2& lo, f32x2& hi) {
    uint32_t d[4];
    asm("mma.sync.aligned.m16n8k16.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5}, {%6}, {%7, %7, %7, %7};"
        : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
        : "r"(a0), "r"(a1), "r"(b), "r"(TCQ_MAGIC));
    lo = pack2(d[0], d[1]);
    hi = pack2(d[2], d[3]);
}

// The activations of two neighbouring blocks: fragments and scales of each half of eight rows.
template <int H> struct TcqActs {
    uint4 q[H];
    float4 s[H][2];
};
template <int H, bool REF_ACTS> __device__ __forceinline__ void tcq_load_acts(const TcqParams& p, int sb, int c, int lane, TcqActs<H>& a) {
    const int g = lane >> 2;
#pragma unroll
    for (int h = 0; h < H; ++h) {
        if constexpr (REF_ACTS) {
            // the reference's layout holds the same fragments block by block; scales as f16 and sums as int16
            const size_t nb = (size_t)p.K / 32, blk = 8 * (size_t)sb + 2 * c;
            const uint8_t* base = p.ref_acts + (size_t)h * nb * TCQ_REF_BLOCK_BYTES;
            const uint2 q0 = *(reinterpret_cast<const uint2*>(base) + blk * 32 + lane), q1 = *(reinterpret_cast<const uint2*>(base) + (blk + 1) * 32 + lane);
            a.q[h] = make_uint4(q0.x, q0.y, q1.x, q1.y);
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const float d = __half2float(*(reinterpret_cast<const __half*>(base + nb * 256) + (blk + b) * 8 + g));
                const float s = d * (float)(int)*(reinterpret_cast<const int16_t*>(base + nb * 272) + (blk + b) * 8 + g);
                a.s[h][b] = make_float4(d, d, s, s);
            }
        } else {
            const size_t slot = ((size_t)sb * H + h) * 4 + c;
            a.q[h] = p.acts[slot * 32 + lane];
            a.s[h][0] = p.scales[(slot * 2 + 0) * 8 + g];
            a.s[h][1] = p.scales[(slot * 2 + 1) * 8 + g];
        }
    }
}

// sum[h] = (b == 0) or += the products of one 32-value block for weight rows 2t, 2t + 1 of eight and activation row 8 h + g: `w0 w1` the weights'
// fragment, `f` the rows' factors (Q4_K: d * sc pair, -dmin * m pair; Q6_K: the two halves' d * sc / 4 pairs; Q8_0: d pair, unused),
// `b` the block of the pair held by `x`.
template <int TYPE, int H>
__device__ __forceinline__ void tcq_block(uint32_t w0, uint32_t w1, const TcqActs<H>& x, int b, const uint4& f, f32x2 (&sum)[H]) {
    const f32x2 unbias = pack2(-12582912.0f, -12582912.0f), f0 = pack2(f.x, f.y), f1 = pack2(f.z, f.w);
    const uint32_t a[4] = {b ? x.q[0].z : x.q[0].x, H == 2 ? (b ? x.q[H - 1].z : x.q[H - 1].x) : 0u, b ? x.q[0].w : x.q[0].y,
                           H == 2 ? (b ? x.q[H - 1].w : x.q[H - 1].y) : 0u};
    f32x2 d[2], e[2];
    if constexpr (TYPE == TYPE_Q6_K) {
        mma_k16(a[0], a[1], w0, d[0], d[1]);
        mma_k16(a[2], a[3], w1, e[0], e[1]);
    } else {
        mma_k32(a, w0, w1, d[0], d[1]);
    }
#pragma unroll
    for (int h = 0; h < H; ++h) {
        const f32x2 xd = pack2(x.s[h][b].x, x.s[h][b].y), i = add2(d[h], unbias);
        if constexpr (TYPE == TYPE_Q6_K) {
            const f32x2 t = fma2(f0, i, mul2(f1, add2(e[h], unbias)));
            sum[h] = b == 0 ? mul2(xd, t) : fma2(xd, t, sum[h]);
        } else if constexpr (TYPE == TYPE_Q8_0) {
            const f32x2 f = mul2(f0, xd);  // exact: two f16 values
            sum[h] = b == 0 ? mul2(f, i) : fma2(f, i, sum[h]);
        } else {
            const f32x2 xs = pack2(x.s[h][b].z, x.s[h][b].w);
            sum[h] = fma2(f0, mul2(xd, i), b == 0 ? mul2(f1, xs) : fma2(f1, xs, sum[h]));
        }
    }
}

// ---------------------------------------------------------------------------------------------
// A superblock's scales: a lane decodes one row's. The superblock starts at row_addr (Q6_K: any even address); `rec` = the row's
// place in its pair's record.
// ---------------------------------------------------------------------------------------------
template <int TYPE> __device__ __forceinline__ void tcq_decode_scales(uint32_t row_addr, uint32_t rec) {
    if constexpr (TYPE == TYPE_Q4_K) {
        // {f16 d, f16 dmin, 12 bytes of 6-bit scales / mins}; value = d * sc_j * q - dmin * m_j
        // (crates/inference-tensor/src/quantized/k_quants.rs:2096-2123)
        const uint4 hdr = lds128(row_addr);
        const float d = half_bits_to_float(hdr.x), dmin = -half_bits_to_float(hdr.x >> 16);
        const uint32_t s4[2] = {hdr.y & 0x3f3f3f3fu, (hdr.w & 0x0f0f0f0fu) | ((hdr.y >> 2) & 0x30303030u)};
        const uint32_t m4[2] = {hdr.z & 0x3f3f3f3fu, ((hdr.w >> 4) & 0x0f0f0f0fu) | ((hdr.z >> 2) & 0x30303030u)};
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            sts32(rec + 16 * j, __float_as_uint(d * (float)((s4[j >> 2] >> (8 * (j & 3))) & 0xffu)));
            sts32(rec + 16 * j + 8, __float_as_uint(dmin * (float)((m4[j >> 2] >> (8 * (j & 3))) & 0xffu)));
        }
    } else if constexpr (TYPE == TYPE_Q6_K) {
        // {ql[128], qh[64], int8 scales[16], f16 d}; value = d * sc_s * (q - 32), 16 values per scale
        // (crates/inference-tensor/src/quantized/k_quants.rs:2649-2680); the fragments hold 4 (q - 32)
        const float d4 = half_bits_to_float(lds16(row_addr + 208)) * 0.25f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint32_t two = lds16(row_addr + 192 + 2 * j);
            sts32(rec + 16 * j, __float_as_uint(d4 * (float)(int)(int8_t)(two & 0xffu)));
            sts32(rec + 16 * j + 8, __float_as_uint(d4 * (float)(int)(int8_t)(two >> 8)));
        }
    } else {
        // eight blocks {f16 d, 32 int8} of 34 bytes
#pragma unroll
        for (int j = 0; j < 8; ++j) sts32(rec + 16 * j, __float_as_uint(half_bits_to_float(lds16(row_addr + 34 * j))));
    }
}

// A word of packed bytes at an address that is 2 (ODD) or 0 modulo 4.
template <bool ODD> __device__ __forceinline__ uint32_t tcq_word(uint32_t addr) {
    if constexpr (ODD) return __funnelshift_r(lds32(addr - 2), lds32(addr + 2), 16);
    else return lds32(addr);
}

// One superblock of up to two tiles, i.e. `groups` = 4 or 2 groups of eight rows. Blocks come in pairs c (64 k); a pair's activations
// serve all groups and the next pair's are loaded meanwhile (`cur` enters with pair 0 and leaves with pair 0 of superblock `next_sb`,
// if that is not negative). box: shared address of row g's superblock; the next group's is 8 pitches on.
//
// Sums: a pair of blocks adds up by itself, the pairs of a superblock in `rest`, the superblocks in `acc`; what acc loses to rounding
// stays in `rest` (compensated summation), and the warps' sums meet in double. One chain of f32 additions over a warp's blocks is the
// faster one (28672 x 4096, 8 rows, us: Q4_K 25.2 against 26.5, Q6_K 39.2 / 39.5, Q8_0 36.6 / 40.0; 1024 x 4096 Q4_K 6.3 / 6.4) but
// loses with its length. Relative error of f32 outputs against exact sums, chain / this, 3 rows of 14336 x 4096: Q8_0 1.5e-7 / 0.66e-7,
// Q6_K 1.3e-7 / 0.71e-7, Q4_K 1.6e-7 / 0.86e-7 (the decode GEMV 0.76e-7, 0.77e-7, 1.45e-7; the tcgen05 form 1.1e-7, 1.1e-7, 1.6e-7).
template <int TYPE, int H, bool REF_ACTS, bool ODD>
__device__ __forceinline__ void tcq_superblock(const TcqParams& p, int sb, int next_sb, int lane, uint32_t box, uint32_t rec, int groups,
                                               TcqActs<H>& cur, f32x2 (&acc)[4][H], f32x2 (&rest)[4][H]) {
    constexpr int PITCH = TcqType<TYPE>::PITCH;
    const int t = lane & 3;
    rec += t * TCQ_REC_PITCH;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        TcqActs<H> nxt;
        if (c < 3) tcq_load_acts<H, REF_ACTS>(p, sb, c + 1, lane, nxt);
        else if (next_sb >= 0) tcq_load_acts<H, REF_ACTS>(p, next_sb, 0, lane, nxt);
        else nxt = cur;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            if (u == 2 && groups < 4) break;
            const uint32_t row = box + u * 8 * PITCH + 4 * t;
            uint32_t a[2][2];  // fragments of the pair's blocks: row g at values 4t.. and 16 + 4t..
            if constexpr (TYPE == TYPE_Q4_K) {
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t w = lds32(row + 16 + 32 * c + 16 * i);  // low nibbles are block 2c, high nibbles 2c + 1
                    a[0][i] = w & 0x0f0f0f0fu;
                    a[1][i] = (w >> 4) & 0x0f0f0f0fu;
                }
            } else if constexpr (TYPE == TYPE_Q6_K) {
                // half n = c / 2 of the superblock holds blocks 4n + qd: ql[64 n + 32 (qd & 1) + l] nibble qd >> 1, qh[32 n + l] bits
                // 2 qd; the pair is qd = 2 (c & 1) + 0, 1. Six bits to the top of the byte with the sign bit flipped: 4 (q - 32).
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t hi = tcq_word<ODD>(row + 128 + 32 * (c >> 1) + 16 * i) ^ 0xaaaaaaaau;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const int qd = 2 * (c & 1) + e;
                        const uint32_t l = tcq_word<ODD>(row + 64 * (c >> 1) + 32 * e + 16 * i);
                        a[e][i] = (((c & 1) ? (l >> 2) : (l << 2)) & 0x3c3c3c3cu) | ((hi << (6 - 2 * qd)) & 0xc0c0c0c0u);
                    }
                }
            } else {
                // eight 34-byte blocks {f16 d, 32 int8}: an even block's quants start 2 modulo 4
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    a[0][i] = tcq_word<true>(row + 68 * c + 2 + 16 * i);
                    a[1][i] = tcq_word<false>(row + 68 * c + 36 + 16 * i);
                }
            }
            f32x2 sum[H];
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const uint32_t fa = rec + u * 4 * TCQ_REC_PITCH + 16 * (2 * c + b);
                uint4 f;
                if constexpr (TYPE == TYPE_Q8_0) {
                    const uint2 d = lds64(fa);
                    f = make_uint4(d.x, d.y, 0u, 0u);
                } else {
                    f = lds128(fa);
                }
                tcq_block<TYPE, H>(a[b][0], a[b][1], cur, b, f, sum);
            }
#pragma unroll
            for (int h = 0; h < H; ++h) rest[u][h] = add2(rest[u][h], sum[h]);
        }
        cur = nxt;
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
        if (u == 2 && groups < 4) break;
#pragma unroll
        for (int h = 0; h < H; ++h) {
            const f32x2 sum = add2(acc[u][h], rest[u][h]);
            rest[u][h] = sub2(rest[u][h], sub2(sum, acc[u][h]));
            acc[u][h] = sum;
        }
    }
}

// H: halves of eight activation rows. REF_ACTS: activations in the reference tier's layout (p.ref_acts).
template <int TYPE, typename dst_t, int H, bool REF_ACTS = false>
__global__ void __launch_bounds__(32 * TcqType<TYPE>::WARPS, 1) gemv_rows_kernel(const __grid_constant__ CUtensorMap map_pair, const __grid_constant__ CUtensorMap map_tile, const TcqParams p) {
    using TT = TcqType<TYPE>;
    constexpr int BOX = TCQ_BOX_BYTES<TYPE>, STAGE = 2 * BOX, DEPTH = TT::DEPTH, WARPS = TT::WARPS;
    extern __shared__ uint8_t tcq_smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tcq_smem_raw) + 127) & ~(uintptr_t)127);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    uint8_t* ring = smem + warp * (DEPTH * STAGE);
    const uint32_t exch0 = smem_u32(smem + WARPS * DEPTH * STAGE), exch = exch0 + warp * TCQ_EXCH_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + WARPS * (DEPTH * STAGE + TCQ_EXCH_BYTES));
    uint64_t* full = bars + warp * DEPTH;
    volatile unsigned int* last_flag = reinterpret_cast<volatile unsigned int*>(bars + WARPS * DEPTH);  // K-split mode

    // ---- this CTA's tiles and superblocks, this warp's share of them ----
    const int group = (int)blockIdx.x / p.ksplit, split = (int)blockIdx.x - group * p.ksplit;
    const int tile0 = group * p.tiles_per_cta + min(group, p.tiles_extra);
    const int ntiles = p.tiles_per_cta + (group < p.tiles_extra ? 1 : 0), npairs = (ntiles + 1) >> 1;
    const int nkc = p.K / TCQ_KC, k0 = (int)((long long)split * nkc / p.ksplit), k1 = (int)((long long)(split + 1) * nkc / p.ksplit);
    const int wks = p.wks, wm = warp / wks, wk = warp - wm * wks, wms = WARPS / wks;
    const int first_sb = k0 + wk;

    // ---- the ring: stages in the order they are used, (pair, superblock); lane 0 issues ----
    if (lane == 0) {
        for (int i = 0; i < DEPTH; ++i) mbar_init(&full[i], 1);
        mbar_init_fence();
    }
    __syncwarp();
    int in_pair = wm, in_sb = first_sb, in_slot = 0, issued = 0;
    bool more = in_pair < npairs && first_sb < k1;
    auto issue = [&] {
        if (!more) return;
        if (lane == 0) {
            const bool both = 2 * in_pair + 1 < ntiles;
            mbar_arrive_expect_tx(&full[in_slot], both ? STAGE : BOX);
            const int x = TYPE == TYPE_Q8_0 ? in_sb * (TT::PITCH / 2) : (in_sb * type_block_bytes(TYPE)) & ~15;  // Q8_0 in 16-bit elements
            tma_load_2d(ring + in_slot * STAGE, both ? &map_pair : &map_tile, x, (tile0 + 2 * in_pair) * TCQ_ROWS, &full[in_slot]);
        }
        ++issued;
        if (++in_slot == DEPTH) in_slot = 0;
        in_sb += wks;
        if (in_sb >= k1) {
            in_sb = first_sb;
            in_pair += wms;
            more = in_pair < npairs;
        }
    };
    for (int i = 0; i < DEPTH; ++i) issue();

    // Launched as a programmatic dependent of the quantize launch: what it writes (activations, counters) is read from here on.
    grid_dependency_wait();
    TcqActs<H> cur;
    if (wm < npairs && first_sb < k1) tcq_load_acts<H, REF_ACTS>(p, first_sb, 0, lane, cur);

    int slot = 0, used = 0;
    uint32_t ph = 0;
    bool ok = true;
    for (int pair = wm; pair < npairs; pair += wms) {
        const int tiles = min(2, ntiles - 2 * pair);
        f32x2 acc[4][H], rest[4][H];
#pragma unroll
        for (int i = 0; i < 4 * H; ++i) (&acc[0][0])[i] = (&rest[0][0])[i] = 0ull;
        for (int sb = first_sb; sb < k1; sb += wks) {
            if (ok && !__all_sync(0xffffffffu, mbar_wait_bounded(&full[slot], ph))) {
                if (lane == 0) record_failure(p.status, STATUS_WAIT_FULL_TIMEOUT, sb);
                ok = false;
            }
            if (ok) {
                const int o = TYPE == TYPE_Q6_K ? (sb * Q6_K_BYTES) & 15 : 0;  // where the superblock starts in its box
                const uint32_t stage = smem_u32(ring + slot * STAGE) + o;
                if (lane < tiles * TCQ_ROWS) tcq_decode_scales<TYPE>(stage + lane * TT::PITCH, exch + (lane >> 1) * TCQ_REC_PITCH + 4 * (lane & 1));
                __syncwarp();
                const int next_sb = sb + wks < k1 ? sb + wks : (pair + wms < npairs ? first_sb : -1);
                const uint32_t box = stage + (lane >> 2) * TT::PITCH;
                if (TYPE == TYPE_Q6_K && (o & 2)) tcq_superblock<TYPE, H, REF_ACTS, true>(p, sb, next_sb, lane, box, exch, 2 * tiles, cur, acc, rest);
                else tcq_superblock<TYPE, H, REF_ACTS, false>(p, sb, next_sb, lane, box, exch, 2 * tiles, cur, acc, rest);
                ++used;
                __syncwarp();  // every lane has read the stage and the record
                issue();
                if (++slot == DEPTH) {
                    slot = 0;
                    ph ^= 1u;
                }
            }
        }
        // ---- the pair's W_k partial sums add up in warp order ----
        __syncwarp();
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int h = 0; h < H; ++h) {
                float v0, v1;
                unpack2(add2(acc[u][h], rest[u][h]), v0, v1);
                sts64(exch + ((8 * h + (lane >> 2)) * TCQ_SUM_PITCH + 8 * u + 2 * (lane & 3)) * 4, __float_as_uint(v0), __float_as_uint(v1));
            }
        const auto group_sync = [&] {
            if (wks > 1) named_bar_sync(1 + wm, 32 * wks);
            else __syncwarp();
        };
        group_sync();
        const int grow = (tile0 + 2 * pair) * TCQ_ROWS + lane;
        const bool row_ok = lane < tiles * TCQ_ROWS && grow < p.N;
        dst_t* y = reinterpret_cast<dst_t*>(p.y) + grow;
        for (int tok = wk; tok < min(p.M, 8 * H); tok += wks) {
            const uint32_t src = exch0 + wm * wks * TCQ_EXCH_BYTES + (tok * TCQ_SUM_PITCH + lane) * 4;
            double part[4] = {0.0, 0.0, 0.0, 0.0};
            for (int w = 0; w < wks; w += 4)
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (w + i < wks) part[i] += (double)lds_f32(src + (w + i) * TCQ_EXCH_BYTES);
            const float v = (float)((part[0] + part[1]) + (part[2] + part[3]));
            if (row_ok) {
                if (p.ksplit > 1) p.partial[((size_t)split * TCQ_TOKENS + tok) * p.N + grow] = v;
                else y[(size_t)tok * p.ldy] = from_float<dst_t>(v);
            }
        }
        if (p.ksplit > 1) {  // one tile and one pair per CTA, all warps on it
            __threadfence();
            group_sync();
            if (wk == 0 && lane == 0) *last_flag = atomicAdd(p.counters + group, 1u) == (unsigned int)p.ksplit - 1u;
            group_sync();
            if (*last_flag) {
                __threadfence();
                for (int tok = wk; tok < min(p.M, 8 * H); tok += wks) {
                    double v = 0.0;
                    for (int s = 0; s < p.ksplit && row_ok; ++s) v += (double)__ldcg(p.partial + ((size_t)s * TCQ_TOKENS + tok) * p.N + grow);
                    if (row_ok) y[(size_t)tok * p.ldy] = from_float<dst_t>((float)v);
                }
            }
        }
        group_sync();  // the sums have been read before their space holds scales again
    }
    if (!ok) {  // let the copies still in flight land before the CTA may exit; `used` stages were consumed
        for (int i = used; i < issued; ++i)
            if (!mbar_wait_bounded(&full[i % DEPTH], (uint32_t)(i / DEPTH) & 1u)) {
                if (lane == 0) record_failure(p.status, STATUS_WAIT_DRAIN_TIMEOUT, i);
                break;
            }
    }
}

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
// workspace: int8 activations [16][K] | float4 scales [K / 32][16] | K-split counters | K-split partial outputs
static size_t tcq_quant_bytes(int K) { return (size_t)K * TCQ_TOKENS + (size_t)(K / 32) * TCQ_TOKENS * sizeof(float4); }
size_t gemv_tc_workspace_bytes(int, int K) {
    return ((tcq_quant_bytes(K) + 255) & ~(size_t)255) + TCQ_COUNTERS * sizeof(unsigned int) + TCQ_PARTIAL_BYTES;
}

template <int TYPE, typename T, int H, bool REF_ACTS = false>
static int launch_gemv_rows(const CUtensorMap (&maps)[2], const TcqParams& p, int grid, cudaStream_t s) {
    constexpr auto kernel = gemv_rows_kernel<TYPE, T, H, REF_ACTS>;
    const cudaError_t e = allow_full_smem<kernel>();
    if (e != cudaSuccess) return (int)e;
    // without REF_ACTS the launch directly before this one on the stream is this file's quantizer, which lets its dependents start
    // early; the two overlap safely because the quantizer writes nothing this kernel reads before its wait
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid, 1, 1);
    cfg.blockDim = dim3(32 * TcqType<TYPE>::WARPS, 1, 1);
    cfg.dynamicSmemBytes = TCQ_SMEM<TYPE>;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = REF_ACTS ? 0 : 1;
    return (int)cudaLaunchKernelEx(&cfg, kernel, maps[0], maps[1], p);
}

// Tiles over CTAs, K over CTAs where there are few tiles, and the W_k of a CTA's warps: fills the plan fields of p, returns the grid.
template <int TYPE> static int tcq_plan(TcqParams& p, bool allow_ksplit) {
    constexpr int WARPS = TcqType<TYPE>::WARPS;
    const int sms = runtime_info().sm_count < TCQ_MAX_CTAS ? runtime_info().sm_count : TCQ_MAX_CTAS;
    const int tiles = (p.N + TCQ_ROWS - 1) / TCQ_ROWS, nkc = p.K / TCQ_KC;
    const int groups = tiles < sms ? tiles : sms;
    p.tiles_per_cta = tiles / groups;
    p.tiles_extra = tiles % groups;
    p.ksplit = 1;
    if (allow_ksplit && runtime_info().tc_ksplit && 2 * tiles <= sms && nkc >= 2 * WARPS) {
        p.ksplit = sms / tiles < nkc / WARPS ? sms / tiles : nkc / WARPS;  // every warp keeps a superblock
        p.wks = WARPS;
        return tiles * p.ksplit;
    }
    // rounds of tile pairs x (superblocks of a warp, about 1100 cycles each with all warps busy, + the sum over W_k warps, about 1000)
    const int pairs = (p.tiles_per_cta + (p.tiles_extra ? 1 : 0) + 1) / 2;
    long long best = -1;
    for (int wk = WARPS; wk >= 1; --wk) {
        if (WARPS % wk != 0) continue;
        const int wm = WARPS / wk;
        const long long cost = (long long)((pairs + wm - 1) / wm) * ((nkc + wk - 1) / wk * 1100LL + 1000);
        if (best < 0 || cost < best) {
            best = cost;
            p.wks = wk;
        }
    }
    return groups;
}

// 2-D tensor maps over the packed weight bytes: boxes of 32 and of 16 rows x one superblock
template <int TYPE> static int tcq_encode_w(CUtensorMap (&maps)[2], const void* w, int N, int K) {
    if (encode_tiled_fn() == nullptr) return B200Q_ERR_UNSUPPORTED;
    const int row_bytes = K / type_block_elems(TYPE) * type_block_bytes(TYPE);
    constexpr bool u16 = TYPE == TYPE_Q8_0;  // 272 bytes are more than 256 one-byte elements
    const cuuint64_t dims[2] = {(cuuint64_t)(u16 ? row_bytes / 2 : row_bytes), (cuuint64_t)N};
    for (int i = 0; i < 2; ++i) {
        const cuuint32_t box[2] = {(cuuint32_t)(u16 ? TcqType<TYPE>::PITCH / 2 : TcqType<TYPE>::PITCH), (cuuint32_t)(i == 0 ? 2 * TCQ_ROWS : TCQ_ROWS)};
        if (encode_tiled_2d_cached(&maps[i], u16 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8, w, dims, (cuuint64_t)row_bytes, box,
                                   CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) != CUDA_SUCCESS)
            return B200Q_ERR_INVALID;
    }
    return 0;
}

template <int TYPE, typename T>
static int launch_gemv_tc_i8(const void* w, const void* x, void* y, int M, int N, int K, int ldx, int ldy, void* workspace, cudaStream_t s) {
    const int halves = M > 8 ? 2 : 1;
    uint8_t* ws = static_cast<uint8_t*>(workspace);
    uint8_t* after = ws + ((tcq_quant_bytes(K) + 255) & ~(size_t)255);
    TcqParams p{};
    p.y = y;
    p.acts = reinterpret_cast<const uint4*>(ws);
    p.scales = reinterpret_cast<const float4*>(ws + (size_t)K * 8 * halves);
    p.M = M;
    p.N = N;
    p.K = K;
    p.ldy = ldy;
    p.status = status_ptr();
    p.counters = reinterpret_cast<unsigned int*>(after);
    p.partial = reinterpret_cast<float*>(after + TCQ_COUNTERS * sizeof(unsigned int));
    const int grid = tcq_plan<TYPE>(p, true);
    CUtensorMap maps[2];
    const int rc = tcq_encode_w<TYPE>(maps, w, N, K);
    if (rc != 0) return rc;
    const int vec = reinterpret_cast<uintptr_t>(x) % (4 * sizeof(T)) == 0 && ldx % 4 == 0;
    const int units = K / 64 * halves;
    tcq_quantize_kernel<T><<<(units + 3) / 4, 128, 0, s>>>(static_cast<const T*>(x), reinterpret_cast<uint4*>(ws),
                                                          reinterpret_cast<float4*>(ws + (size_t)K * 8 * halves), K, M, ldx, halves, vec, p.counters);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    return halves == 1 ? launch_gemv_rows<TYPE, T, 1>(maps, p, grid, s) : launch_gemv_rows<TYPE, T, 2>(maps, p, grid, s);
}

// ---------------------------------------------------------------------------------------------
// The reference tier's own pair of launchers (crates/inference-quant/src/gguf/ffi.rs:631-652,954-998): the host
// quantizes with launch_mmvq_tc_quantize_<elem> into ITS scratch (288 bytes per 32-value block and 8-row half,
// fast_mmvq.rs:94,1898-1902) and hands that to launch_mmvq_tc_gguf_<type>_<elem>_plain. The matvec is the kernel
// above with REF_ACTS, which reads that layout's fragments as they are; without a workspace for partial outputs the split
// along K is off. Shapes the TMA path cannot take (packed rows that are not a multiple of 16 bytes, unaligned weights) go
// to a plain one-warp-per-row kernel on the same layout.
// ---------------------------------------------------------------------------------------------
template <int TYPE, typename dst_t>
__global__ void __launch_bounds__(256) gemv_tc_ref_simple_kernel(const uint8_t* __restrict__ w, const uint8_t* __restrict__ acts,
                                                                 dst_t* __restrict__ dst, int K, int N, int stride_dst, int M) {
    const int lane = threadIdx.x & 31;
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (row >= N) return;
    const int nb = K / 32;
    const uint8_t* rp = w + (size_t)row * (K / 256) * type_block_bytes(TYPE);
    float acc[TCQ_TOKENS];
#pragma unroll
    for (int t = 0; t < TCQ_TOKENS; ++t) acc[t] = 0.0f;
    for (int kb = lane; kb < nb; kb += 32) {
        int wq[32];
        float s0 = 0.0f, s1 = 0.0f, mn = 0.0f;  // Q4_K: s0 = d * sc, mn = dmin * m; Q6_K: s0, s1 = d * sc of the two halves
        const int sblk = kb >> 3;
        if (TYPE == TYPE_Q4_K) {
            const int j = kb & 7;
            const uint8_t* sb = rp + (size_t)sblk * Q4_K_BYTES;
            const uint8_t* q = sb + 4;
            int sc, m;
            if (j < 4) { sc = q[j] & 63; m = q[j + 4] & 63; }
            else { sc = (q[j + 4] & 0xF) | ((q[j - 4] >> 6) << 4); m = (q[j + 4] >> 4) | ((q[j] >> 6) << 4); }
            s0 = half_bits_to_float((uint32_t)sb[0] | ((uint32_t)sb[1] << 8)) * (float)sc;
            mn = half_bits_to_float((uint32_t)sb[2] | ((uint32_t)sb[3] << 8)) * (float)m;
            const uint8_t* qs = sb + 16 + 32 * (j >> 1);
            for (int l = 0; l < 32; ++l) wq[l] = (j & 1) ? (qs[l] >> 4) : (qs[l] & 0xF);
        } else {
            const int n = (kb >> 2) & 1, qd = kb & 3;
            const uint8_t* sb = rp + (size_t)sblk * Q6_K_BYTES;
            const uint8_t* ql = sb + 64 * n + 32 * (qd & 1);
            const uint8_t* qh = sb + 128 + 32 * n;
            for (int l = 0; l < 32; ++l) {
                const int lo = (qd & 2) ? (ql[l] >> 4) : (ql[l] & 0xF);
                wq[l] = (lo | (((qh[l] >> (2 * qd)) & 3) << 4)) - 32;
            }
            const float d = half_bits_to_float((uint32_t)sb[208] | ((uint32_t)sb[209] << 8));
            s0 = d * (float)(int)(int8_t)sb[192 + 8 * n + 2 * qd];
            s1 = d * (float)(int)(int8_t)sb[192 + 8 * n + 2 * qd + 1];
        }
        for (int t = 0; t < M; ++t) {
            const uint8_t* base = acts + (size_t)(t >> 3) * nb * TCQ_REF_BLOCK_BYTES;
            const int r = t & 7;
            const int8_t* frag = reinterpret_cast<const int8_t*>(base) + (size_t)kb * 256 + (4 * r) * 8;
            const float xd = __half2float(reinterpret_cast<const __half*>(base + (size_t)nb * 256)[kb * 8 + r]);
            int d0 = 0, d1 = 0;
            for (int l = 0; l < 16; ++l) d0 += wq[l] * (int)frag[(l >> 2) * 8 + (l & 3)];
            for (int l = 16; l < 32; ++l) d1 += wq[l] * (int)frag[((l - 16) >> 2) * 8 + 4 + (l & 3)];
            if (TYPE == TYPE_Q4_K) {
                const int sum = (int)reinterpret_cast<const int16_t*>(base + (size_t)nb * 256 + (size_t)nb * 16)[kb * 8 + r];
                acc[t] += s0 * (xd * (float)(d0 + d1)) - mn * (xd * (float)sum);
            } else {
                acc[t] += xd * (s0 * (float)d0 + s1 * (float)d1);
            }
        }
    }
    for (int t = 0; t < M; ++t) {
        const float v = warp_sum(acc[t]);
        if (lane == 0) dst[(size_t)t * stride_dst + row] = from_float<dst_t>(v);
    }
}

template <typename T>
static int launch_tcq_ref_quantize(const void* x, void* vy, int kx, int num_rows, cudaStream_t s) {
    if (kx <= 0 || num_rows <= 0) return 0;
    const dim3 grid((unsigned)((kx + 31) / 32), (unsigned)((num_rows + 7) / 8), 1);
    tcq_ref_quantize_kernel<T><<<grid, dim3(32, 8, 1), 0, s>>>(static_cast<const T*>(x), static_cast<uint8_t*>(vy), kx, num_rows);
    return (int)cudaGetLastError();
}

template <int TYPE, typename T>
static int launch_gemv_tc_ref(const void* w, const void* vy, void* dst, int K, int N, int stride_col_dst, int b, cudaStream_t s) {
    if (N <= 0 || K <= 0 || b <= 0) return 0;
    if (b > TCQ_TOKENS || K % TCQ_KC != 0) return B200Q_ERR_UNSUPPORTED;
    const int row_bytes = K / 256 * type_block_bytes(TYPE);
    const bool tma_ok = reinterpret_cast<uintptr_t>(w) % 16 == 0 && row_bytes % 16 == 0 && encode_tiled_fn() != nullptr &&
                        reinterpret_cast<uintptr_t>(vy) % 8 == 0;
    if (!tma_ok) {
        gemv_tc_ref_simple_kernel<TYPE, T><<<(N + 7) / 8, 256, 0, s>>>(static_cast<const uint8_t*>(w), static_cast<const uint8_t*>(vy),
                                                                      static_cast<T*>(dst), K, N, stride_col_dst, b);
        return (int)cudaGetLastError();
    }
    TcqParams p{};
    p.y = dst;
    p.M = b;
    p.N = N;
    p.K = K;
    p.ldy = stride_col_dst;
    p.status = status_ptr();
    p.ref_acts = static_cast<const uint8_t*>(vy);
    const int grid = tcq_plan<TYPE>(p, false);
    CUtensorMap maps[2];
    const int rc = tcq_encode_w<TYPE>(maps, w, N, K);
    if (rc != 0) return rc;
    return b <= 8 ? launch_gemv_rows<TYPE, T, 1, true>(maps, p, grid, s) : launch_gemv_rows<TYPE, T, 2, true>(maps, p, grid, s);
}

int gemv_tc_dispatch(int type, int elem, const void* w, const void* x, void* y, int M, int N, int K, int ldx, int ldy, void* workspace,
                     cudaStream_t s) {
    if (M <= 0 || N <= 0) return 0;
    if (M > TCQ_TOKENS || K <= 0 || K % TCQ_KC != 0) return B200Q_ERR_UNSUPPORTED;
    const int row_bytes = K / type_block_elems(type) * type_block_bytes(type);
    if (reinterpret_cast<uintptr_t>(w) % 16 != 0 || row_bytes % 16 != 0) return B200Q_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(workspace) % 128 != 0) return B200Q_ERR_INVALID;
#define B200Q_TCQ_CASE(TYPE)                                                                                              \
    if (type == TYPE) {                                                                                                   \
        if (elem == ELEM_BF16) return launch_gemv_tc_i8<TYPE, __nv_bfloat16>(w, x, y, M, N, K, ldx, ldy, workspace, s);   \
        if (elem == ELEM_F16) return launch_gemv_tc_i8<TYPE, __half>(w, x, y, M, N, K, ldx, ldy, workspace, s);           \
        if (elem == ELEM_F32) return launch_gemv_tc_i8<TYPE, float>(w, x, y, M, N, K, ldx, ldy, workspace, s);            \
        return B200Q_ERR_UNSUPPORTED;                                                                                     \
    }
    B200Q_TCQ_CASE(TYPE_Q4_K)
    B200Q_TCQ_CASE(TYPE_Q6_K)
    B200Q_TCQ_CASE(TYPE_Q8_0)
#undef B200Q_TCQ_CASE
    return B200Q_ERR_UNSUPPORTED;
}

}  // namespace b200q

// The reference's symbols; void, asynchronous, allocation-free. `cfg` selects among the reference kernel's own launch
// shapes (mmvq_tc_k.cuh:352-375) and has no meaning for this kernel.
#define B200Q_TC_QUANTIZE(tag, T)                                                                                          \
    extern "C" void launch_mmvq_tc_quantize_##tag(const void* x, void* vy, int kx, int num_rows, void* stream) {          \
        b200q::note_launch_status(b200q::launch_tcq_ref_quantize<T>(x, vy, kx, num_rows, (cudaStream_t)stream));           \
    }
B200Q_TC_QUANTIZE(bf16, __nv_bfloat16)
B200Q_TC_QUANTIZE(f16, __half)
B200Q_TC_QUANTIZE(f32, float)
#undef B200Q_TC_QUANTIZE

#define B200Q_TC_PLAIN(type_tag, TYPE, tag, T)                                                                             \
    extern "C" void launch_mmvq_tc_gguf_##type_tag##_##tag##_plain(const void* vx, const void* vy, void* dst, int ncols_x,  \
                                                                   int nrows_x, int stride_col_dst, int b_size, int cfg,   \
                                                                   void* stream) {                                         \
        (void)cfg;                                                                                                         \
        b200q::note_launch_status(                                                                                         \
            b200q::launch_gemv_tc_ref<TYPE, T>(vx, vy, dst, ncols_x, nrows_x, stride_col_dst, b_size, (cudaStream_t)stream)); \
    }
B200Q_TC_PLAIN(q4_k, b200q::TYPE_Q4_K, bf16, __nv_bfloat16)
B200Q_TC_PLAIN(q4_k, b200q::TYPE_Q4_K, f16, __half)
B200Q_TC_PLAIN(q4_k, b200q::TYPE_Q4_K, f32, float)
B200Q_TC_PLAIN(q6_k, b200q::TYPE_Q6_K, bf16, __nv_bfloat16)
B200Q_TC_PLAIN(q6_k, b200q::TYPE_Q6_K, f16, __half)
B200Q_TC_PLAIN(q6_k, b200q::TYPE_Q6_K, f32, float)
#undef B200Q_TC_PLAIN
