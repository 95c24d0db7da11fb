// Causal attention of a block of prompt rows on the 5th-generation tensor cores (attentionKernel, Inference.cu:182-266, intended
// math), from 16 rows on; shorter blocks: prefill.cu.
//
// One CTA takes a head and 256 query rows as two tiles of 128 (upper and lower); both read the same 64-key tiles of K and V, which
// halves the bytes an SM draws from L2 per product (16 KB of K and V per 128 x 64 scores).  Twelve warps:
//   warp 0      TMA producer: the q rows once, then K and V tiles (64 keys x 128 dims, two 64-dim halves, 128-byte swizzle)
//   warp 1      MMA issuer: S = Q K^T (K-major operands from shared memory), O += P V with P from tensor memory and V MN-major as it
//               lies in the cache
//   warps 4..7, 8..11   one row a thread of the upper / lower tile: S from tensor memory, online softmax, P back in its place
// Tensor memory, per tile: O 128 columns, two S buffers of 64.  P goes in as TWO fp16 terms (P = hi + lo, lo the rounding error of
// hi): 32 + 32 columns, exactly the room of the S it comes from.  That is 22 bits from 2^-3 on, below it an absolute error of 2^-25 (the
// last place of fp16), where a row's largest P lies between 1 and 256.
// While the threads work on one S the tensor cores compute the other and the other tile's products.  O is rescaled (a pass of
// tensor memory -> registers -> tensor memory) only when a row's maximum has grown by more than 8 powers of two since the
// last time: P then stays at or below 256 and the quotient O / l is the same.
// 1953 rows at position 2048, 32 heads, a call among others: 590 us with warp-level MMAs (mma.sync, 64 rows a CTA), 164 now, 0.36 of the
// measured bf16 rate in useful operations (the second term of P and the masked halves of the diagonal tiles are not counted).
// Bound: the MMAs, 768 cycles per 128 x 64 scores (256 for S, 256 for each term of P), beside 512 cycles of exponentials.
// All waits are bounded.  After one that gives up the error word is set, rows that are not finished are written as NaN, and the CTA
// leaves when its copies and MMAs in flight are done.
#include <atomic>

#include "tc05.cuh"

namespace qw3 {

constexpr int AT_ROWS = 128, AT_KEYS = 64, AT_STAGES = 4;
constexpr int AT_THREADS = 384;
constexpr int AT_Q_BYTES = AT_ROWS * 256;          // one tile of q rows: two halves of 64 dims
constexpr int AT_KV_BYTES = AT_KEYS * 256;         // one tile of K or V
constexpr size_t AT_SMEM = 2 * AT_Q_BYTES + 2 * (size_t)AT_STAGES * AT_KV_BYTES + 512;

__device__ __forceinline__ float ex2(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

struct AttnParams {
    const __half* qkv;
    const __half* kc;
    const __half* vc;
    long long max_pos;
    __half* ctx;
    int hidden, pos0, rows;
    int* err;   // null: the word below
};
// Error word of calls without a workspace, one on every GPU that loads the library.
static __device__ int g_attn_err;

// One row by a warp, from global memory and in 32-bit arithmetic: rows whose tile holds Inf or NaN in V behind the row.  The tensor
// cores multiply these by the zeros of the masked probabilities, and the sum is NaN; here nothing past the row's last key is read.
__device__ __noinline__ void attn_row(const __half* q, const __half* k, const __half* v, int n_keys, __half* dst, int lane) {
    float m = -INFINITY, l = 0.0f, o[4] = {0.0f, 0.0f, 0.0f, 0.0f};   // outputs 4 lane .. 4 lane + 3
    for (int k0 = 0; k0 < n_keys; k0 += 32) {
        float s = -INFINITY;
        if (k0 + lane < n_keys) {
            const uint4* kr = reinterpret_cast<const uint4*>(k + (size_t)(k0 + lane) * 128);
            const uint4* qr = reinterpret_cast<const uint4*>(q);
            s = 0.0f;
            for (int i = 0; i < 16; ++i) {
                const uint4 a = qr[i], b = kr[i];
                const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float2 x = __half22float2(*reinterpret_cast<const __half2*>(&aw[e])), y = __half22float2(*reinterpret_cast<const __half2*>(&bw[e]));
                    s = fmaf(x.y, y.y, fmaf(x.x, y.x, s));
                }
            }
            s *= 1.0f / sqrtf(128.0f);   // Inference.cu:218
        }
        float mn = fmaxf(m, s);
        for (int d = 16; d > 0; d >>= 1) mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, d));
        const float f = m == -INFINITY ? 0.0f : expf(m - mn), pr = s == -INFINITY ? 0.0f : expf(s - mn);
        m = mn;
        l = l * f + pr;   // this lane's keys
#pragma unroll
        for (int e = 0; e < 4; ++e) o[e] *= f;
        for (int j = 0; j < 32 && k0 + j < n_keys; ++j) {
            const float pj = __shfl_sync(0xffffffffu, pr, j);
            const uint2 w = *reinterpret_cast<const uint2*>(v + (size_t)(k0 + j) * 128 + 4 * lane);
            const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w.x)), b = __half22float2(*reinterpret_cast<const __half2*>(&w.y));
            o[0] = fmaf(pj, a.x, o[0]);
            o[1] = fmaf(pj, a.y, o[1]);
            o[2] = fmaf(pj, b.x, o[2]);
            o[3] = fmaf(pj, b.y, o[3]);
        }
    }
    for (int d = 16; d > 0; d >>= 1) l += __shfl_xor_sync(0xffffffffu, l, d);
    __half2* out = reinterpret_cast<__half2*>(dst + 4 * lane);
    out[0] = __floats2half2_rn(o[0] / l, o[1] / l);
    out[1] = __floats2half2_rn(o[2] / l, o[3] / l);
}

// POLL_ONCE: a wait looks at its barrier once and gives up (qw3_attn_prefill_poll_once).
template <bool POLL_ONCE>
__global__ void __launch_bounds__(AT_THREADS, 1)
attn_prefill_tc_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                       const __grid_constant__ CUtensorMap tm_v, const AttnParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* q_s = smem;
    uint8_t* k_s = q_s + 2 * AT_Q_BYTES;
    uint8_t* v_s = k_s + AT_STAGES * AT_KV_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(v_s + AT_STAGES * AT_KV_BYTES);
    const uint32_t q_full = smem_u32(bars), k_full = q_full + 8, v_full = k_full + 8 * AT_STAGES, k_empty = v_full + 8 * AT_STAGES,
                   v_empty = k_empty + 8 * AT_STAGES, s_full = v_empty + 8 * AT_STAGES /* [tile][buffer] */, p_full = s_full + 32,
                   pv_done = p_full + 32 /* [tile][buffer] */, drain = pv_done + 32;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 2 + 4 * AT_STAGES + 12);
    volatile int* s_dead = reinterpret_cast<volatile int*>(tmem_slot + 1);

    const auto wait = [](uint32_t bar, uint32_t parity) { return POLL_ONCE ? mbar_poll(bar, parity) : mbar_wait(bar, parity); };
    const auto give_up = [&](int code) {
        atomicCAS(p.err != nullptr ? p.err : &g_attn_err, 0, code);
        *s_dead = 1;
    };

    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int head = blockIdx.x, r0 = (int)(gridDim.y - 1 - blockIdx.y) * 2 * AT_ROWS;   // the blocks with the most keys start first
    const int n_keys = p.pos0 + min(r0 + 2 * AT_ROWS, p.rows);
    const int n_tiles = (n_keys + AT_KEYS - 1) / AT_KEYS;

    if (tid == 0) {
        mbar_init(q_full, 1);
        mbar_init(drain, 1);
        for (int s = 0; s < AT_STAGES; ++s) {
            mbar_init(k_full + 8 * s, 1);
            mbar_init(v_full + 8 * s, 1);
            mbar_init(k_empty + 8 * s, 1);
            mbar_init(v_empty + 8 * s, 1);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(s_full + 8 * i, 1);
            mbar_init(p_full + 8 * i, 4);   // the four warps of the tile
            mbar_init(pv_done + 8 * i, 1);
        }
        *s_dead = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;   // O of the tiles at columns 0 and 128, S at 256 + 128 tile + 64 buffer

    if (warp == 0) {
        if (elect_one()) {
            bool ok = true;
            mbar_expect_tx(q_full, 2 * AT_Q_BYTES);
            for (int t = 0; t < 2; ++t)
                for (int h = 0; h < 2; ++h)
                    tma_load_2d(smem_u32(q_s + t * AT_Q_BYTES + h * (AT_Q_BYTES / 2)), &tm_q, head * 128 + 64 * h, r0 + AT_ROWS * t, q_full);
            int j = 0, kv = 0;
            for (; j < n_tiles; ++j) {
                const int s = j % AT_STAGES;
                const uint32_t lap = (uint32_t)(j / AT_STAGES);
                for (kv = 0; kv < 2; ++kv) {
                    const uint32_t full = (kv ? v_full : k_full) + 8 * s, empty = (kv ? v_empty : k_empty) + 8 * s;
                    uint8_t* dst = (kv ? v_s : k_s) + s * AT_KV_BYTES;
                    if (lap > 0) ok = wait(empty, (lap - 1) & 1u);
                    if (*s_dead != 0) ok = false;
                    if (!ok) break;
                    mbar_expect_tx(full, AT_KV_BYTES);
                    for (int h = 0; h < 2; ++h)
                        tma_load_3d(smem_u32(dst + h * (AT_KV_BYTES / 2)), kv ? &tm_v : &tm_k, 64 * h, j * AT_KEYS, head, full);
                }
                if (!ok) break;
            }
            // drain: the last release arrivals land before the CTA may leave
            for (int i = n_tiles < AT_STAGES ? 0 : n_tiles - AT_STAGES; i < n_tiles && ok; ++i) {
                const uint32_t parity = (uint32_t)(i / AT_STAGES) & 1u;
                ok = wait(k_empty + 8 * (i % AT_STAGES), parity) && wait(v_empty + 8 * (i % AT_STAGES), parity);
            }
            if (!ok) {
                give_up(0x30021);
                mbar_wait(q_full, 0);   // the copies in flight
                for (int t = 0; t < 2; ++t) {
                    const int asked = j < n_tiles && t < kv ? j + 1 : j;   // tiles of K, of V
                    for (int i = max(asked - AT_STAGES, 0); i < asked; ++i)
                        mbar_wait((t ? v_full : k_full) + 8 * (i % AT_STAGES), (uint32_t)(i / AT_STAGES) & 1u);
                }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (elect_one()) {
            // D = f32, A = B = f16.  S: N = 64 keys, both K-major.  P V: N = 128 dims, V MN-major (bit 16).
            const uint32_t idesc_s = (1u << 4) | ((uint32_t)(AT_KEYS >> 3) << 17) | ((uint32_t)(AT_ROWS >> 4) << 24);
            const uint32_t idesc_o = (1u << 4) | (1u << 16) | ((uint32_t)(128 >> 3) << 17) | ((uint32_t)(AT_ROWS >> 4) << 24);
            const uint64_t qd = make_smem_desc(smem_u32(q_s), 16, 1024), kd = make_smem_desc(smem_u32(k_s), 16, 1024);
            const uint64_t vd = make_smem_desc(smem_u32(v_s), AT_KV_BYTES / 2, 1024);   // 64-dim halves, 8-key groups
            auto scores = [&](int t, int j) {   // S of tile t against key tile j
                const uint32_t d = tmem + 256 + 128 * t + 64 * (j & 1);
                const uint64_t a = qd + (uint64_t)(t * (AT_Q_BYTES >> 4)), b = kd + (uint64_t)((j % AT_STAGES) * (AT_KV_BYTES >> 4));
#pragma unroll
                for (int ks = 0; ks < 8; ++ks)
                    umma_f16(d, a + (uint64_t)((ks >> 2) * (AT_Q_BYTES >> 5) + (ks & 3) * 2), b + (uint64_t)((ks >> 2) * (AT_KV_BYTES >> 5) + (ks & 3) * 2),
                             idesc_s, ks > 0 ? 1u : 0u);
                umma_commit(s_full + 16 * t + 8 * (j & 1));
            };
            bool ok = wait(q_full, 0);
            for (int j = 0; j < 2 && j < n_tiles && ok; ++j) {
                ok = wait(k_full + 8 * j, 0);
                if (!ok) break;
                scores(0, j);
                scores(1, j);
                umma_commit(k_empty + 8 * j);
            }
            for (int j = 0; j < n_tiles && ok; ++j) {
                const int s = j % AT_STAGES, b = j & 1;
                ok = *s_dead == 0 && wait(v_full + 8 * s, (uint32_t)(j / AT_STAGES) & 1u);
                for (int t = 0; t < 2 && ok; ++t) {
                    ok = wait(p_full + 16 * t + 8 * b, (uint32_t)(j >> 1) & 1u);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t a = tmem + 256 + 128 * t + 64 * b;
                    const uint64_t v = vd + (uint64_t)(s * (AT_KV_BYTES >> 4));
#pragma unroll
                    for (int ks = 0; ks < AT_KEYS / 16; ++ks) {
                        umma_f16_ts(tmem + 128 * t, a + 8 * ks, v + (uint64_t)(ks * (2048 >> 4)), idesc_o, (j > 0 || ks > 0) ? 1u : 0u);
                        umma_f16_ts(tmem + 128 * t, a + 32 + 8 * ks, v + (uint64_t)(ks * (2048 >> 4)), idesc_o, 1u);
                    }
                    umma_commit(pv_done + 16 * t + 8 * b);
                    if (t == 1) umma_commit(v_empty + 8 * s);
                    // the next scores of the buffer: issued after, and so executed after, the product that reads P there
                    if (j + 2 < n_tiles) {
                        const int s2 = (j + 2) % AT_STAGES;
                        if (t == 0) ok = wait(k_full + 8 * s2, (uint32_t)((j + 2) / AT_STAGES) & 1u);
                        if (!ok) break;
                        scores(t, j + 2);
                        if (t == 1) umma_commit(k_empty + 8 * s2);
                    }
                }
            }
            if (!ok) give_up(0x30022);
            if (POLL_ONCE || !ok || *s_dead != 0) {   // the MMAs in flight (a wait that gives up later does so long after they are done)
                umma_commit(drain);
                mbar_wait(drain, 0);
            }
        }
        __syncwarp();
    } else if (warp >= 4) {
        const int t = (warp - 4) >> 2, q = warp & 3;
        const uint32_t lane_base = tmem + ((uint32_t)(32 * q) << 16);
        const uint32_t o_at = lane_base + 128 * t, s_at = lane_base + 256 + 128 * t;
        const int row = r0 + AT_ROWS * t + 32 * q + lane, pos = p.pos0 + row;   // last key the row sees
        const int pos_first = pos - lane;                                      // of the warp's first row
        const float c = (float)(1.4426950408889634 / 11.313708498984761);      // log2(e) / sqrt(128), Inference.cu:218
        float m = -INFINITY, mc = 0.0f, l = 0.0f;   // m: maximum in use (raw scores), mc = m c
        float mr = 0.0f, off = 0.0f;                // m c - mc where that is not small, and then off = 0 and m is taken off s; else off = mc
        bool ok = true;
        for (int j = 0; j < n_tiles && ok; ++j) {
            const int b = j & 1;
            ok = __all_sync(0xffffffffu, *s_dead == 0 && wait(s_full + 16 * t + 8 * b, (uint32_t)(j >> 1) & 1u));
            if (!ok) break;
            tc_fence_after();
            uint32_t sr[64];
            float s[64];
            tmem_ld32(s_at + 64 * b, sr);
            tmem_ld32(s_at + 64 * b + 32, sr + 32);
            tmem_wait_ld();
#pragma unroll
            for (int e = 0; e < 64; ++e) s[e] = __uint_as_float(sr[e]);
            const int k0 = j * AT_KEYS;
            if (k0 + AT_KEYS - 1 > pos_first) {   // some row of the warp does not see the whole tile
#pragma unroll
                for (int e = 0; e < 64; ++e) s[e] = k0 + e <= pos ? s[e] : -INFINITY;
            }
            float mx[4] = {s[0], s[1], s[2], s[3]};
#pragma unroll
            for (int e = 4; e < 64; ++e) mx[e & 3] = fmaxf(mx[e & 3], s[e]);
            const float mt = fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3]));
            if (__any_sync(0xffffffffu, (mt - m) * c > 8.0f || mr != 0.0f)) {   // rare after the first tile
                const float mn = fmaxf(m, mt), nmc = mn == -INFINITY ? 0.0f : mn * c;
                const float nmr = fabsf(nmc) >= 1048576.0f ? fmaf(mn, c, -nmc) : 0.0f;
                const float f = m == -INFINITY ? 0.0f : ex2((mc - nmc) + (mr - nmr));
                if (j > 0) {
                    ok = __all_sync(0xffffffffu, wait(pv_done + 16 * t + 8 * (b ^ 1), (uint32_t)((j - 1) >> 1) & 1u));
                    if (!ok) break;
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        uint32_t o[32];
                        tmem_ld32(o_at + 32 * h, o);
                        tmem_wait_ld();
#pragma unroll
                        for (int e = 0; e < 32; ++e) o[e] = __float_as_uint(__uint_as_float(o[e]) * f);
                        tmem_st32(o_at + 32 * h, o);
                    }
                }
                l *= f;
                m = mn;
                mc = nmc;
                mr = nmr;
                off = mr != 0.0f ? 0.0f : mc;
                if (__any_sync(0xffffffffu, mr != 0.0f)) {
                    const float base = mr != 0.0f ? m : 0.0f;
#pragma unroll
                    for (int e = 0; e < 64; ++e) s[e] -= base;
                }
            }
            float ls[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const float a0 = ex2(fmaf(s[32 * h + 2 * e], c, -off)), a1 = ex2(fmaf(s[32 * h + 2 * e + 1], c, -off));
                    ls[(2 * e) & 3] += a0;
                    ls[(2 * e + 1) & 3] += a1;
                    const __half2 hh = __floats2half2_rn(a0, a1);
                    const float2 hf = __half22float2(hh);
                    const __half2 ll = __floats2half2_rn(a0 - hf.x, a1 - hf.y);
                    hi[e] = *reinterpret_cast<const uint32_t*>(&hh);
                    lo[e] = *reinterpret_cast<const uint32_t*>(&ll);
                }
                tmem_st16(s_at + 64 * b + 16 * h, hi);
                tmem_st16(s_at + 64 * b + 32 + 16 * h, lo);
            }
            l += (ls[0] + ls[1]) + (ls[2] + ls[3]);
            tmem_wait_st();
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full + 16 * t + 8 * b);
        }
        for (int j = n_tiles < 2 ? 0 : n_tiles - 2; j < n_tiles && ok; ++j)
            ok = __all_sync(0xffffffffu, wait(pv_done + 16 * t + 8 * (j & 1), (uint32_t)(j >> 1) & 1u));
        if (!ok && lane == 0) give_up(0x30023);
        __syncwarp();
        tc_fence_after();
        __half* dst = p.ctx + (size_t)row * p.hidden + head * 128;
        const bool wide = (reinterpret_cast<uintptr_t>(p.ctx) & 15) == 0;   // the caller's ctx need only be aligned for pairs
        float finite = 0.0f;   // NaN as soon as an output is NaN or Inf
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            uint32_t o[32];
            __syncwarp();
            tmem_ld32(o_at + 32 * h, o);
            tmem_wait_ld();
            if (row < p.rows) {
#pragma unroll
                for (int e = 0; e < 32; e += 8) {
                    uint32_t w[4];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {   // one rounding to fp16, Inference.cu:257-265
                        const float a = __uint_as_float(o[e + 2 * k]) / l, b = __uint_as_float(o[e + 2 * k + 1]) / l;
                        const __half2 v = __floats2half2_rn(a, b);
                        finite = fmaf(a, 0.0f, fmaf(b, 0.0f, finite));
                        w[k] = ok ? *reinterpret_cast<const uint32_t*>(&v) : 0x7fff7fffu;
                    }
                    if (wide) {
                        *reinterpret_cast<uint4*>(dst + 32 * h + e) = make_uint4(w[0], w[1], w[2], w[3]);
                    } else {
#pragma unroll
                        for (int k = 0; k < 4; ++k) *reinterpret_cast<uint32_t*>(dst + 32 * h + e + 2 * k) = w[k];
                    }
                }
            }
        }
        __syncwarp();   // a row that is done again has been stored
        for (uint32_t redo = ok ? __ballot_sync(0xffffffffu, row < p.rows && finite != 0.0f) : 0u; redo != 0; redo &= redo - 1) {
            const int r = row - lane + __ffs(redo) - 1;
            const size_t at = (size_t)head * p.max_pos * 128;
            attn_row(p.qkv + (size_t)r * 3 * p.hidden + head * 128, p.kc + at, p.vc + at, p.pos0 + r + 1,
                     p.ctx + (size_t)r * p.hidden + head * 128, lane);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// qkv [rows][3 * hidden] (q rotated), caches [heads][max_pos][128].
int attn_prefill_tc_launch(const void* qkv, const void* kc, const void* vc, int heads, int hidden, long long max_pos, int pos0, int rows,
                           void* ctx, int* err, bool poll_once, cudaStream_t st) {
    QW3_REQUIRE(((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15) == 0,
                "qw3_attn_prefill: qkv and both caches must be 16-byte aligned from 16 rows on");
    QW3_REQUIRE((reinterpret_cast<uintptr_t>(ctx) & 3) == 0, "qw3_attn_prefill: ctx must be 4-byte aligned from 16 rows on");
    CUtensorMap tm_q, tm_k, tm_v;
    const uint64_t qd[2] = {(uint64_t)hidden, (uint64_t)rows}, qs[1] = {(uint64_t)hidden * 6};
    const uint32_t qb[2] = {64, AT_ROWS};
    // rows past the block's last one do not exist for the copies: they arrive as zeros, whatever the cache holds there
    const uint64_t kd[3] = {128, (uint64_t)(pos0 + rows), (uint64_t)heads}, ks[2] = {256, (uint64_t)max_pos * 256};
    const uint32_t kb[3] = {64, AT_KEYS, 1};
    int rc = encode_f16_map(&tm_q, qkv, 2, qd, qs, qb);
    if (rc == QW3_OK) rc = encode_f16_map(&tm_k, kc, 3, kd, ks, kb);
    if (rc == QW3_OK) rc = encode_f16_map(&tm_v, vc, 3, kd, ks, kb);
    if (rc != QW3_OK) return rc;
    static std::atomic<bool> attr_set[64];   // per device: the kernel's shared-memory limit is raised once
    int dev = 0;
    QW3_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        QW3_CUDA(cudaFuncSetAttribute(attn_prefill_tc_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AT_SMEM));
        QW3_CUDA(cudaFuncSetAttribute(attn_prefill_tc_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)AT_SMEM));
        if (dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    AttnParams p = {static_cast<const __half*>(qkv), static_cast<const __half*>(kc), static_cast<const __half*>(vc), max_pos,
                    static_cast<__half*>(ctx), hidden, pos0, rows, err};
    const dim3 grid(heads, (rows + 2 * AT_ROWS - 1) / (2 * AT_ROWS));
    if (poll_once) attn_prefill_tc_kernel<true><<<grid, AT_THREADS, AT_SMEM, st>>>(tm_q, tm_k, tm_v, p);
    else attn_prefill_tc_kernel<false><<<grid, AT_THREADS, AT_SMEM, st>>>(tm_q, tm_k, tm_v, p);
    QW3_CUDA(cudaGetLastError());
    return QW3_OK;
}

}  // namespace qw3

extern "C" int qw3_attn_prefill_status(void* stream) {
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    void* word = nullptr;
    int err = 0;
    QW3_CUDA(cudaGetSymbolAddress(&word, qw3::g_attn_err));
    QW3_CUDA(cudaMemcpyAsync(&err, word, 4, cudaMemcpyDeviceToHost, st));
    QW3_CUDA(cudaStreamSynchronize(st));
    if (err == 0) return QW3_OK;
    QW3_CUDA(cudaMemsetAsync(word, 0, 4, st));
    QW3_CUDA(cudaStreamSynchronize(st));
    qw3::set_last_error("a bounded device-side wait of qw3_attn_prefill gave up (device error word = 0x%x)", err);
    return QW3_ERR_TIMEOUT;
}
