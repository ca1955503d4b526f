// Prefill GEMM on CTA pairs: Y[m][n] = sum_k X[m][k] * W[n][k] in two steps, for callers that lend a workspace.
//
//   1. expand_weights_kernel writes the packed weights once as bf16 / f16 rows (d * q and the min folded in f32, one
//      rounding: the values the single-launch kernel in gemm_tcgen05.cu forms inside its tiles); quantized activations are
//      expanded the same way;
//   2. gemm_pair_kernel multiplies with tcgen05.mma.cta_group::2: a pair of SMs owns a tile of 256 weight rows x up to 256
//      tokens. Each SM holds 128 of the weight rows and half of the tokens in its shared memory and the tensor cores read
//      both halves, so an SM moves 32 KB of operands into shared memory per 64 k for a 256 x 256 tile.
//
// Why two steps: the single-launch kernel expands a weight tile again for every 256 tokens and, with 128 x 128 instructions on
// single SMs, is bound by shared-memory bandwidth near 0.55 of the tensor peak. Expanding costs N * K * 2 bytes written and read
// once, so it pays from a few hundred tokens on (see gemm_pair_pays). The weights sit on the M side of the instruction: its
// N side, the tokens, then goes in steps of 32, so a ragged prompt length wastes little.
//
// Every wait is bounded; a wait that gives up records a code in the device status word, work is skipped, and the kernel
// still frees its TMEM columns before it returns.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "runtime.h"
#include "tcgen05.cuh"

namespace b200q {

// ---- cta_group::2 forms of the wrappers in tcgen05.cuh -----------------------------------------------------------------------
__device__ __forceinline__ uint32_t cluster_ctarank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of the same shared-memory variable in CTA `rank` of the cluster
__device__ __forceinline__ uint32_t map_to_rank(const void* p, uint32_t rank) {
    uint32_t a;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}
// a load into this CTA's shared memory whose bytes are counted on a barrier of either CTA of the pair
__device__ __forceinline__ void tma_load_2d_pair(void* dst_smem, const CUtensorMap* map, int x, int y, uint32_t bar_addr) {
    asm volatile("cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
                     smem_u32(dst_smem)),
                 "l"(map), "r"(bar_addr), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* dst_smem, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)), "r"(ncols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// arrives at the same barrier of both CTAs once the MMAs issued so far have finished
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((unsigned short)3)
                 : "memory");
}
__device__ __forceinline__ void tc_mma_f16_pair(uint32_t tmem_d, uint64_t desc_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
        "}\n" ::"r"(tmem_d),
        "l"(desc_a), "l"(desc_b), "r"(idesc), "r"(accumulate)
        : "memory");
}

template <typename T> struct PairElem;
template <> struct PairElem<__half> { static constexpr int format = 0; };
template <> struct PairElem<__nv_bfloat16> { static constexpr int format = 1; };

// ---- the GEMM ------------------------------------------------------------------------------------------------------------------
constexpr int GP_ROWS = 128;      // weight rows of one CTA = TMEM lanes
constexpr int GP_TOKENS = 256;    // tokens of a tile at most = TMEM columns of one accumulator
constexpr int GP_BK = 64;         // k per stage: one 128-byte swizzled row of 16-bit elements
constexpr int GP_MAX_STAGES = 12;
constexpr int GP_A_BYTES = GP_ROWS * GP_BK * 2;
constexpr int GP_THREADS = 256;   // warp 0 TMA, warp 1 MMA, warp 2 TMEM, warps 4-7 epilogue
constexpr int GP_TMEM_COLS = 512; // two accumulators

struct GemmPairParams {
    void* y;  // [M][ldy]
    int M, N, K, ldy;
    int bn;               // tokens per tile: a multiple of 32, <= 256
    int stages;           // as many as shared memory holds at this bn
    int tiles_m, tiles_n; // token tiles, weight tiles of 256 rows
    unsigned int* status;
};

struct GemmPairBarriers {
    uint64_t full[GP_MAX_STAGES], empty[GP_MAX_STAGES];
    uint64_t tmem_full[2], tmem_empty[2];
    uint32_t tmem_base;
};
constexpr size_t gp_smem(int stages, int bn) { return 1024 + (size_t)stages * (GP_A_BYTES + bn / 2 * GP_BK * 2) + sizeof(GemmPairBarriers); }

template <typename T, typename OutT>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ CUtensorMap tmap_x, const GemmPairParams p) {
    extern __shared__ uint8_t gp_smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(gp_smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* a_stages = smem;
    const int stages = p.stages, half = p.bn / 2, b_bytes = half * GP_BK * 2;  // bytes: a multiple of 1024
    uint8_t* b_stages = smem + stages * GP_A_BYTES;
    GemmPairBarriers* bars = reinterpret_cast<GemmPairBarriers*>(b_stages + stages * b_bytes);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const uint32_t rank = cluster_ctarank();
    const int pair = blockIdx.x >> 1, npairs = gridDim.x >> 1;
    const int nkb = p.K / GP_BK;
    const int ntiles = p.tiles_m * p.tiles_n;
    const uint32_t stage_bytes = 2u * (GP_A_BYTES + (uint32_t)b_bytes);  // both CTAs' operands of a stage

    if (tid == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&bars->full[s], 1);
            mbar_init(&bars->empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bars->tmem_full[s], 1);
            mbar_init(&bars->tmem_empty[s], 8);  // four epilogue warps of each CTA
        }
        mbar_init_fence();
    }
    if (warp == 2) tmem_alloc_pair(&bars->tmem_base, GP_TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // the other CTA's barriers exist before anything arrives at them
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&bars->tmem_base);
    grid_dependency_wait();  // launched as a programmatic dependent of the expansion: its stores are visible from here on

    if (warp == 0) {
        // ---------------- TMA: this CTA's 128 weight rows and half of the tokens; the leader's barrier counts both CTAs' bytes ----
        int s = 0, g = 0;
        uint32_t ph = 1;
        bool ok = true;
        const uint32_t full0 = map_to_rank(&bars->full[0], 0);
        for (int tile = pair; tile < ntiles && ok; tile += npairs) {
            const int tn = tile / p.tiles_m, tm = tile - tn * p.tiles_m;
            const int row = tn * 2 * GP_ROWS + (int)rank * GP_ROWS, token = tm * p.bn + (int)rank * half;
            for (int kb = 0; kb < nkb; ++kb, ++g) {
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bars->empty[s], ph));
                if (!ok) {
                    if (lane == 0) record_failure(p.status, STATUS_WAIT_EMPTY_TIMEOUT, g);
                    break;
                }
                if (elect_one()) {
                    if (rank == 0) mbar_arrive_expect_tx(&bars->full[s], stage_bytes);
                    tma_load_2d_pair(a_stages + (size_t)s * GP_A_BYTES, &tmap_w, kb * GP_BK, row, full0 + 8u * s);
                    tma_load_2d_pair(b_stages + (size_t)s * b_bytes, &tmap_x, kb * GP_BK, token, full0 + 8u * s);
                }
                __syncwarp();
                if (++s == stages) {
                    s = 0;
                    ph ^= 1u;
                }
            }
        }
        // the leader waits for its last copies before the CTAs may exit (they are counted on its barriers; the MMAs have
        // consumed them unless something gave up)
        if (!ok && rank == 0) {
            for (int q = 0; q < min(g, stages); ++q) {
                if (s == 0) { s = stages - 1; ph ^= 1u; } else --s;
                if (!mbar_wait_bounded(&bars->full[s], ph ^ 1u)) {
                    if (lane == 0) record_failure(p.status, STATUS_WAIT_DRAIN_TIMEOUT, q);
                    break;
                }
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer: an elected lane of the leader, for both SMs ----------------
        if (rank == 0) {
            const uint32_t idesc = make_idesc_f16(PairElem<T>::format, 2 * GP_ROWS, p.bn);
            const uint64_t da0 = make_smem_desc_sw128(smem_u32(a_stages)), db0 = make_smem_desc_sw128(smem_u32(b_stages));
            int s = 0, ti = 0;
            uint32_t ph = 0;
            bool ok = true;
            for (int tile = pair; tile < ntiles && ok; tile += npairs, ++ti) {
                const int buf = ti & 1;
                ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bars->tmem_empty[buf], ((ti >> 1) & 1) ^ 1));
                if (!ok) {
                    if (lane == 0) record_failure(p.status, STATUS_WAIT_MMA_TIMEOUT, 2000 + ti);
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + buf * GP_TOKENS;
                for (int kb = 0; kb < nkb; ++kb) {
                    ok = __all_sync(0xffffffffu, mbar_wait_bounded(&bars->full[s], ph));
                    if (!ok) {
                        if (lane == 0) record_failure(p.status, STATUS_WAIT_FULL_TIMEOUT, kb);
                        break;
                    }
                    tc_fence_after();
                    const uint64_t da = da0 + (uint64_t)(s * (GP_A_BYTES >> 4)), db = db0 + (uint64_t)(s * (b_bytes >> 4));
                    if (elect_one()) {
#pragma unroll
                        for (int k = 0; k < GP_BK / 16; ++k) tc_mma_f16_pair(d, da + 2 * k, db + 2 * k, idesc, (kb > 0 || k > 0) ? 1u : 0u);
                        tc_commit_pair(&bars->empty[s]);  // frees the stage in both CTAs when these MMAs have read it
                        if (kb == nkb - 1) tc_commit_pair(&bars->tmem_full[buf]);
                    }
                    __syncwarp();
                    if (++s == stages) {
                        s = 0;
                        ph ^= 1u;
                    }
                }
            }
        }
    } else if (warp >= 4) {
        // ---------------- epilogue: thread = weight row, 32 tokens at a time; a warp's store is 32 neighbouring outputs ----------------
        const int quarter = warp & 3;
        bool ok = true;
        int ti = 0;
        for (int tile = pair; tile < ntiles; tile += npairs, ++ti) {
            const int buf = ti & 1;
            const int tn = tile / p.tiles_m, tm = tile - tn * p.tiles_m;
            if (!mbar_wait_bounded(&bars->tmem_full[buf], (ti >> 1) & 1)) {
                record_failure(p.status, STATUS_WAIT_MMA_TIMEOUT, ti);
                ok = false;
            }
            ok = __all_sync(0xffffffffu, ok);
            if (!ok) break;
            tc_fence_after();
            const int n = tn * 2 * GP_ROWS + (int)rank * GP_ROWS + quarter * 32 + lane;
            const int tok0 = tm * p.bn;
            const int toks = min(p.bn, p.M - tok0);
            OutT* y = reinterpret_cast<OutT*>(p.y) + (size_t)tok0 * p.ldy + n;
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + buf * GP_TOKENS;
            for (int c = 0; c < toks; c += 32) {
                uint32_t acc[32];
                tmem_ld_32x32(taddr + c, acc);
                if (n < p.N) {
#pragma unroll
                    for (int j = 0; j < 32; ++j) {
                        if (c + j < toks) *y = from_float<OutT>(__uint_as_float(acc[j]));
                        y += p.ldy;
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(map_to_rank(&bars->tmem_empty[buf], 0));  // the accumulator may be reused
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();  // neither CTA leaves while the other may still read its operands or arrive at its barriers
    if (warp == 2) tmem_dealloc_pair(tmem_base, GP_TMEM_COLS);
}

// ---- expansion -------------------------------------------------------------------------------------------------------------------
template <typename T> __device__ __forceinline__ uint32_t pair_pack2(float a, float b);
template <> __device__ __forceinline__ uint32_t pair_pack2<__nv_bfloat16>(float a, float b) {
    __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
template <> __device__ __forceinline__ uint32_t pair_pack2<__half>(float a, float b) {
    __half2 v = __floats2half2_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&v);
}
template <typename T> __device__ __forceinline__ void store_16b(T* dst, const float (&v)[8]) {
    *reinterpret_cast<uint4*>(dst) =
        make_uint4(pair_pack2<T>(v[0], v[1]), pair_pack2<T>(v[2], v[3]), pair_pack2<T>(v[4], v[5]), pair_pack2<T>(v[6], v[7]));
}
// byte `idx` of w as the float 2^23 + byte
template <int idx> __device__ __forceinline__ float magic_byte(uint32_t w) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650 | idx)); }
template <typename Fn> __device__ __forceinline__ void eight_bytes(uint32_t a, uint32_t b, float (&v)[8], Fn fn) {
    v[0] = fn(magic_byte<0>(a)); v[1] = fn(magic_byte<1>(a)); v[2] = fn(magic_byte<2>(a)); v[3] = fn(magic_byte<3>(a));
    v[4] = fn(magic_byte<0>(b)); v[5] = fn(magic_byte<1>(b)); v[6] = fn(magic_byte<2>(b)); v[7] = fn(magic_byte<3>(b));
}
// Eight packed bytes at an even address of shared memory: aligned words and a funnel shift.
__device__ __forceinline__ uint2 lds_eight(uint32_t a) {
    const uint32_t w = a & ~3u, sh = (a & 2u) * 8;
    const uint32_t b = lds32(w + 4);
    return make_uint2(__funnelshift_r(lds32(w), b, sh), __funnelshift_r(b, lds32(w + 8), sh));
}

// Between HBM and the issue slots, about half of either (ncu, 4096 x 14336 Q6_K: 29 us, 3.9 TB/s, an instruction on 0.5 of the cycles):
// a CTA's loads, unpacking and stores follow one another. A thread takes eight packed bytes at a time and writes the 8 (Q8_0), 16 (Q4_K: low and high nibbles) or 32 (Q6_K: four
// quarters) values they hold a part of, in 16-byte stores; neighbouring threads write neighbouring pieces. The 34- and 210-byte blocks
// of Q8_0 and Q6_K are aligned to 2 bytes only: a CTA first brings its values' packed bytes into shared memory by 16-byte loads
// (expansion and product, against reading them by halves: 512 x 4096 x 14336 Q8_0 85.1 -> 81.4 us, 333 x 6144 x 4096 34.3 -> 32.9,
// 333 x 28672 x 4096 139 -> 132, Q6_K 133 -> 130). Q4_K's blocks are aligned and read where they lie: staged, 1024 x 14336 x 4096 takes
// 151 us instead of 148.
constexpr int EXPAND_VALUES = 8192;  // of a CTA
template <int TYPE> constexpr int EXPAND_PER_BLOCK = TYPE == TYPE_Q4_K ? 16 : (TYPE == TYPE_Q6_K ? 8 : 4);  // items per block
template <int TYPE, typename T>
__global__ void __launch_bounds__(256) expand_weights_kernel(const uint8_t* __restrict__ w, T* __restrict__ out, long long blocks) {
    constexpr int BLOCKS = EXPAND_VALUES / type_block_elems(TYPE), BYTES = BLOCKS * type_block_bytes(TYPE);
    static_assert(BYTES % 16 == 0, "CTAs start on 16-byte boundaries of the packed bytes");
    constexpr bool STAGED = TYPE != TYPE_Q4_K;
    __shared__ __align__(16) uint8_t stage[STAGED ? BYTES + 16 : 16];
    grid_launch_dependents();
    const long long first = (long long)blockIdx.x * BLOCKS;
    const int nblocks = (int)(blocks - first < BLOCKS ? blocks - first : BLOCKS), nbytes = nblocks * type_block_bytes(TYPE);
    const uint8_t* src = w + first * type_block_bytes(TYPE);
    if constexpr (STAGED) {
        const int wide = (reinterpret_cast<uintptr_t>(src) & 15) == 0 ? nbytes & ~15 : 0;
        for (int i = threadIdx.x; i < wide / 16; i += 256) reinterpret_cast<uint4*>(stage)[i] = __ldg(reinterpret_cast<const uint4*>(src) + i);
        for (int i = wide + 2 * threadIdx.x; i < nbytes; i += 512)
            *reinterpret_cast<unsigned short*>(stage + i) = __ldg(reinterpret_cast<const unsigned short*>(src + i));
        __syncthreads();
    }
    const uint32_t base = smem_u32(stage);
    out += first * type_block_elems(TYPE);
    for (int i = threadIdx.x; i < nblocks * EXPAND_PER_BLOCK<TYPE>; i += 256) {
        const int blk = i / EXPAND_PER_BLOCK<TYPE>, t = i % EXPAND_PER_BLOCK<TYPE>;
        const uint32_t sb = base + blk * type_block_bytes(TYPE);
        T* dst = out + blk * type_block_elems(TYPE);
        float v[8];
        if constexpr (TYPE == TYPE_Q4_K) {
            const int c = t >> 2, l0 = 8 * (t & 3);  // 64-value chunk and the byte inside its 32
            const uint8_t* gb = src + blk * Q4_K_BYTES;
            const uint4 hdr = __ldg(reinterpret_cast<const uint4*>(gb));
            const uint2 q = __ldg(reinterpret_cast<const uint2*>(gb + 16 + 32 * c + l0));
            const float d = half_bits_to_float(hdr.x), dmin = half_bits_to_float(hdr.x >> 16);
            const int sh = 16 * (c & 1);
            const uint32_t s2 = hdr.y >> sh, m2 = hdr.z >> sh, e2 = hdr.w >> sh;  // sub-blocks 2c, 2c + 1: two bytes each
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t a = (s2 >> (8 * h)) & 0xffu, b = (m2 >> (8 * h)) & 0xffu, e = (e2 >> (8 * h)) & 0xffu;
                const uint32_t sc = c < 2 ? (a & 63u) : ((e & 0xFu) | ((a >> 6) << 4)), m = c < 2 ? (b & 63u) : ((e >> 4) | ((b >> 6) << 4));
                const float dl = d * (float)(int)sc, ml = dmin * (float)(int)m;
                eight_bytes((q.x >> (4 * h)) & 0x0f0f0f0fu, (q.y >> (4 * h)) & 0x0f0f0f0fu, v, [&](float f) { return fmaf(dl, f - 8388608.0f, -ml); });
                store_16b<T>(dst + 64 * c + 32 * h + l0, v);
            }
        } else if constexpr (TYPE == TYPE_Q6_K) {
            const int n = t >> 2, l0 = 8 * (t & 3);
            const float d = half_bits_to_float(lds16(sb + 208));
            const uint2 ql[2] = {lds_eight(sb + 64 * n + l0), lds_eight(sb + 64 * n + 32 + l0)}, qh = lds_eight(sb + 128 + 32 * n + l0);
#pragma unroll
            for (int qd = 0; qd < 4; ++qd) {
                const uint32_t two = lds16(sb + 192 + 8 * n + 2 * qd);
                const float s = d * (float)(int)(int8_t)(two >> (8 * (l0 >> 4)));
                const uint32_t a = ((ql[qd & 1].x >> (4 * (qd >> 1))) & 0x0f0f0f0fu) | (((qh.x >> (2 * qd)) & 0x03030303u) << 4);
                const uint32_t b = ((ql[qd & 1].y >> (4 * (qd >> 1))) & 0x0f0f0f0fu) | (((qh.y >> (2 * qd)) & 0x03030303u) << 4);
                eight_bytes(a, b, v, [&](float f) { return s * (f - 8388640.0f); });  // 2^23 + 32
                store_16b<T>(dst + 128 * n + 32 * qd + l0, v);
            }
        } else {
            const float d = half_bits_to_float(lds16(sb));
            const uint2 q = lds_eight(sb + 2 + 8 * t);
            eight_bytes(q.x ^ 0x80808080u, q.y ^ 0x80808080u, v, [&](float f) { return d * (f - 8388736.0f); });
            store_16b<T>(dst + 8 * t, v);
        }
    }
}

// Activations as the reference's prefill quantizer leaves them (144-byte blocks of 128 values of one token, block (k / 128) * M +
// token) -> bf16 rows: d * q in f32, one rounding. Sixteen threads a block.
template <typename T>
__global__ void __launch_bounds__(256) expand_acts_kernel(const uint8_t* __restrict__ aq, T* __restrict__ out, int M, int K, int ds4, long long threads) {
    grid_launch_dependents();
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= threads) return;
    // sixteen threads share a block, the blocks of one token one after the other: the stores of a row are contiguous
    const int per_row = K / 8;
    const int token = (int)(i / per_row), c = (int)(i - (long long)token * per_row);
    const uint8_t* blk = aq + ((size_t)(c >> 4) * M + token) * MMQ_BLOCK_BYTES;
    const uint2 q = __ldg(reinterpret_cast<const uint2*>(blk + 16 + 8 * (c & 15)));
    const uint32_t sw = __ldg(reinterpret_cast<const uint32_t*>(blk) + ((c & 15) >> 2));
    const float d = ds4 ? half_bits_to_float(sw) : __uint_as_float(sw);
    float v[8];
    eight_bytes(q.x ^ 0x80808080u, q.y ^ 0x80808080u, v, [&](float f) { return d * (f - 8388736.0f); });  // 2^23 + 128
    store_16b<T>(out + (size_t)token * K + 8 * c, v);
}

// ---- host side -------------------------------------------------------------------------------------------------------------------
template <typename Kern, typename... Args>
static cudaError_t launch_dependent(Kern kernel, unsigned grid, unsigned block, size_t smem, cudaStream_t s, bool dependent, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid, 1, 1);
    cfg.blockDim = dim3(block, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = dependent ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

template <int TYPE, typename T>
static cudaError_t launch_expand(const void* w, T* out, long long values, cudaStream_t s) {
    const unsigned grid = (unsigned)((values + EXPAND_VALUES - 1) / EXPAND_VALUES);
    expand_weights_kernel<TYPE, T><<<grid, 256, 0, s>>>(static_cast<const uint8_t*>(w), out, values / type_block_elems(TYPE));
    return cudaGetLastError();
}
template <typename T>
static cudaError_t expand_weights(int type, const void* w, T* out, long long values, cudaStream_t s) {
    if (type == TYPE_Q4_K) return launch_expand<TYPE_Q4_K, T>(w, out, values, s);
    if (type == TYPE_Q6_K) return launch_expand<TYPE_Q6_K, T>(w, out, values, s);
    return launch_expand<TYPE_Q8_0, T>(w, out, values, s);
}

// Tokens per tile. Tiles go out in waves of one per CTA pair, and a wave takes as long as its tile is high, but no less than a tile of
// about 148 tokens (an MMA of 256 rows has a floor near 64 cycles; K = 4096: 12.5 us a wave up to 160 tokens, 15.5 at 192, 21 at
// 256). So the height is the one with the least waves x height, plus some 24 tokens' worth a wave for filling and draining; as few
// tiles as 256 tokens allow unless that is beaten by 5 % (more tiles read the weights again from L2). Against always the fewest:
// 512 x 4096 x 14336 (32 tiles for 74 pairs -> 64) 95 -> 77 us, 1024 x 14336 x 4096 (224 tiles in 4 waves -> 280 in 4) 121 -> 111,
// 1024 x 6144 x 4096 57 -> 48, 333 x 6144 x 4096 32.7 -> 31.3.
static int token_tile(int M, int tiles_n) {
    const int pairs = runtime_info().sm_count / 2;
    long long best = 0;
    int best_bn = 0;
    for (int tm = (M + GP_TOKENS - 1) / GP_TOKENS, last = 0;; ++tm) {
        const int bn = (((M + tm - 1) / tm) + 31) & ~31;
        if (best_bn != 0 && bn < 128) break;
        if (bn == last) continue;
        last = bn;
        const long long waves = ((long long)((M + bn - 1) / bn) * tiles_n + pairs - 1) / pairs;
        const long long cost = waves * ((bn > 148 ? bn : 148) + 24);
        if (best_bn == 0 || cost * 100 < best * 95) {
            best = cost;
            best_bn = bn;
        }
    }
    return best_bn;
}

template <typename T, typename OutT>
static int launch_pair(const T* w16, const T* x, void* y, int M, int N, int K, int ldx, int ldy, cudaStream_t s, bool dependent) {
    GemmPairParams p{};
    p.y = y;
    p.M = M;
    p.N = N;
    p.K = K;
    p.ldy = ldy;
    p.status = status_ptr();
    p.bn = token_tile(M, (N + 2 * GP_ROWS - 1) / (2 * GP_ROWS));
    p.stages = GP_MAX_STAGES;
    while (gp_smem(p.stages, p.bn) > (size_t)runtime_info().smem_optin - 1024) --p.stages;
    p.tiles_m = (M + p.bn - 1) / p.bn;
    p.tiles_n = (N + 2 * GP_ROWS - 1) / (2 * GP_ROWS);
    const CUtensorMapDataType dt = PairElem<T>::format == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
    CUtensorMap map_w, map_x;
    {
        const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)N};
        const cuuint32_t box[2] = {GP_BK, GP_ROWS};
        if (encode_tiled_2d_cached(&map_w, dt, w16, dims, (cuuint64_t)K * sizeof(T), box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) !=
            CUDA_SUCCESS)
            return B200Q_ERR_INVALID;
    }
    {
        const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
        const cuuint32_t box[2] = {GP_BK, (cuuint32_t)(p.bn / 2)};
        if (encode_tiled_2d_cached(&map_x, dt, x, dims, (cuuint64_t)ldx * sizeof(T), box, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B) !=
            CUDA_SUCCESS)
            return B200Q_ERR_INVALID;
    }
    constexpr auto kernel = gemm_pair_kernel<T, OutT>;
    cudaError_t e = allow_full_smem<kernel>();
    if (e != cudaSuccess) return (int)e;
    const int ntiles = p.tiles_m * p.tiles_n, pairs = runtime_info().sm_count / 2;
    e = launch_dependent(kernel, 2u * (unsigned)(ntiles < pairs ? ntiles : pairs), GP_THREADS, gp_smem(p.stages, p.bn), s, dependent, map_w, map_x, p);
    return (int)e;
}

// Where the single-launch kernel of gemm_tcgen05.cu stays: it expands each weight tile in the CTA that multiplies it, so with one tile
// of tokens it expands nothing twice and saves the 16-bit copy, but a tile of 128 weight rows takes an SM the same time however many
// SMs have one. So it stays where it can stage packed rows in shared memory and
//   * every SM has a tile, up to 256 rows (256 x 28672 x 4096 Q4_K 84 us against 106 us; one row more doubles its time), or
//   * up to 128 rows (its tile of tokens), where enough SMs have one. Where the two meet, of 148 tiles, us single / pair at 17 and 128
//     rows: Q4_K K = 4096 88 tiles 39.7 / 36.0, 40.7 / 37.7, 96 39.7 / 38.8, 41.4 / 41.7, 112 39.8 / 44.2, 41.2 / 47.1, K = 14336 88
//     125 / 124, 127 / 127; Q8_0 K = 4096 104 47.0 / 48.0, 48.3 / 49.3, K = 14336 96 151 / 148, 153 / 152; Q6_K, slower to unpack,
//     K = 4096 120 52.0 / 52.9, 53.4 / 54.2, K = 14336 112 167 / 168, 169 / 170. Narrower matrices have less to expand: K = 2048 at 128
//     rows, 128 tiles, Q4_K 23.3 / 25.1, Q8_0 27.1 / 28.9, but Q6_K 29.8 / 27.7.
// From 257 rows on it expands twice or more and is the slower one everywhere.
static bool gemm_pair_pays(int type, int M, int N, int K) {
    const int rows = runtime_info().gemm_pair_rows;
    if (rows >= 0) return M >= rows;
    const bool staged = K % 256 == 0 && (long long)K / type_block_elems(type) * type_block_bytes(type) % 16 == 0;
    if (!staged || M > 256) return true;
    const int tiles = (N + 127) / 128, sms = runtime_info().sm_count;
    if (tiles >= sms) return false;
    if (M > 128) return true;
    // of 148 tiles: 93 / 99 / 111 and more stay (Q4_K / Q8_0 / Q6_K), at narrower K 124 / 124 / 148
    const bool wide = K >= 3072;
    const int twenty_fourths = type == TYPE_Q4_K ? (wide ? 15 : 20) : (type == TYPE_Q8_0 ? (wide ? 16 : 20) : (wide ? 18 : 24));
    return 24 * tiles < twenty_fourths * sms;
}
size_t gemm_pair_workspace_bytes(int type, int M, int N, int K) { return gemm_pair_pays(type, M, N, K) ? (size_t)N * K * 2 : 0; }
// Quantized activations: their 16-bit copy as well. The single-launch kernel expands them in every tile, so this pays at every row count
// on every shape that kernel serves, us launcher / this, Q4_K: 28672 x 4096 17 rows 105 / 99, 128 rows 125 / 100, 256 152 / 108; 14336 x
// 4096 17 rows 58 / 47, 128 63 / 49; 1024 x 1024 17 rows 19.5 / 11.5 (closest: Q8_0 28672 x 4096 at 17 rows, 109 / 108). The shapes it does
// not take are multiplied as integers by its plain kernel, and stay so.
size_t mmq_pair_workspace_bytes(int type, int M, int N, int K) {
    const bool tiles = K % 256 == 0 && (long long)K / type_block_elems(type) * type_block_bytes(type) % 16 == 0;
    return tiles && M >= runtime_info().gemm_pair_rows ? ((size_t)N * K + (size_t)M * K) * 2 : 0;
}

// The reference launchers' product (launch_mmq_gguf_*, gemm_tcgen05.cu) with a workspace: bf16 operands, f32 accumulation.
template <typename OutT>
static int mmq_pair_t(int type, const void* w, const void* aq, void* y, int M, int N, int K, int ldy, void* workspace, cudaStream_t s) {
    __nv_bfloat16* w16 = static_cast<__nv_bfloat16*>(workspace);
    __nv_bfloat16* x16 = w16 + (size_t)N * K;
    cudaError_t e = expand_weights<__nv_bfloat16>(type, w, w16, (long long)N * K, s);
    if (e != cudaSuccess) return (int)e;
    const long long threads = (long long)M * (K / 8);
    expand_acts_kernel<__nv_bfloat16><<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(static_cast<const uint8_t*>(aq), x16, M, K, type == TYPE_Q4_K, threads);
    e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    return launch_pair<__nv_bfloat16, OutT>(w16, x16, y, M, N, K, K, ldy, s, true);
}
int mmq_pair_dispatch(int type, int elem, const void* w, const void* aq, void* y, int M, int N, int K, int ldy, void* workspace, cudaStream_t s) {
    if (M <= 0 || N <= 0) return 0;
    if (encode_tiled_fn() == nullptr) return B200Q_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(w) % 16 != 0 || reinterpret_cast<uintptr_t>(aq) % 16 != 0) return B200Q_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(workspace) % 128 != 0) return B200Q_ERR_INVALID;
    if (elem == ELEM_BF16) return mmq_pair_t<__nv_bfloat16>(type, w, aq, y, M, N, K, ldy, workspace, s);
    if (elem == ELEM_F16) return mmq_pair_t<__half>(type, w, aq, y, M, N, K, ldy, workspace, s);
    if (elem == ELEM_F32) return mmq_pair_t<float>(type, w, aq, y, M, N, K, ldy, workspace, s);
    return B200Q_ERR_UNSUPPORTED;
}

template <typename T>
static int gemm_pair_t(int type, const void* w, const T* x, void* y, int M, int N, int K, int ldx, int ldy, void* workspace, cudaStream_t s) {
    T* w16 = static_cast<T*>(workspace);
    const cudaError_t e = expand_weights<T>(type, w, w16, (long long)N * K, s);
    if (e != cudaSuccess) return (int)e;
    return launch_pair<T, T>(w16, x, y, M, N, K, ldx, ldy, s, true);
}

int gemm_pair_dispatch(int type, int elem, const void* w, const void* x, void* y, int M, int N, int K, int ldx, int ldy, void* workspace,
                       cudaStream_t s) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0 || K % GP_BK != 0 || K % type_block_elems(type) != 0) return B200Q_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(x) % 16 != 0 || ((size_t)ldx * 2) % 16 != 0) return B200Q_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(w) % (type == TYPE_Q4_K ? 16 : 2) != 0 || encode_tiled_fn() == nullptr) return B200Q_ERR_UNSUPPORTED;
    if (reinterpret_cast<uintptr_t>(workspace) % 128 != 0) return B200Q_ERR_INVALID;
    if (elem == ELEM_BF16) return gemm_pair_t<__nv_bfloat16>(type, w, static_cast<const __nv_bfloat16*>(x), y, M, N, K, ldx, ldy, workspace, s);
    if (elem == ELEM_F16) return gemm_pair_t<__half>(type, w, static_cast<const __half*>(x), y, M, N, K, ldx, ldy, workspace, s);
    return B200Q_ERR_UNSUPPORTED;
}

}  // namespace b200q
