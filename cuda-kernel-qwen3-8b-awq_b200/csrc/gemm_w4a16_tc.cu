// Tensor-core W4A16 contraction for several activation rows (prefill / batched rows) on sm_100a:
//   Y[r][i] = sum_j W(i, j) * X[r][j],   W(i, j) = hmul(hsub(half(q), zp[g]), scale[g])  (bit-exact),
// with tcgen05.mma (fp16 x fp16 -> fp32 in tensor memory).  The reference has no batched path: it
// feeds prompts token by token through cublasGemmEx at n = 1 (Inference.cu:1304-1343, 1052-1065);
// this is the same product for `rows` tokens at once.
//
// One CTA computes a tile of 128 outputs x N rows of X (N = 16..256).  Nineteen warps:
//   warp 0      TMA producer: per 64-deep K block one box of activations [N][64] (128-byte swizzle, K-major
//               operand B)
//   warp 1, 18  MMA issuers (one lane each; even / odd K blocks into separate accumulators in tensor memory, which
//               warp 1 allocates), tcgen05.commit frees the stages
//   warps 2..17 read the packed nibbles of the tile straight from global memory (16 bytes per thread and row, one
//               K block ahead; four groups of four warps take the K blocks in turn), unpack them to fp16 with
//               the reference's two roundings and write operand A to shared memory in the MN-major 128-byte-swizzled canonical layout (outputs are
//               contiguous in the packed stream, so MN-major needs no transposition); afterwards the
//               same warps read the accumulators back (tcgen05.ld) and store Y as fp16.
// Within every group of 8 outputs the rows of A are stored in the order the lop3 unpack yields them
// (0,4,1,5,2,6,3,7); the epilogue undoes that permutation when it computes the output index.
// All mbarrier waits are bounded; a wait that gives up sets the workspace error word.
#include <atomic>
#include <cstdlib>
#include <mutex>

#include "tc05.cuh"

namespace qw3 {

const Workspace* ws_struct(qw3_ws_t ws);
const W4Desc* w4_desc(qw3_w4_t w);

constexpr int GM_TILE_M = 128;                 // outputs per CTA
constexpr int GM_BK = 64;                      // K per pipeline stage
constexpr int GM_A_BYTES = GM_TILE_M * GM_BK * 2;        // 16384
constexpr int GM_MAX_STAGES = 24;              // mbarrier slots per ring
// Operand A (16 KB per K block, unpacked) and the activations share one ring depth and ONE release barrier per
// stage: a tcgen05.commit costs the issuing lane ~150 ns, so a K block gets a single commit.  The depth is a template
// parameter (6, or 4 with 256-row tiles).
constexpr int GM_UNPACK_WARPS = 16;           // unpack / epilogue warps: four groups of four, taking K blocks in turn
                                              // (an unpack warp is latency-bound on its own chain: more groups, more K blocks in flight)
constexpr int GM_ISSUER_B = 2 + GM_UNPACK_WARPS;   // warp index of the second MMA issuer
constexpr int GM_THREADS = 32 * (GM_ISSUER_B + 1);

struct GemmParams {
    const uint8_t* packed;   // [K][M/2] bytes; the unpack warps read their 16-byte pieces straight from global memory
    const __half* scale;
    const __half* zp;
    int n_alloc, M, K, Mb, Kb;
    int uniform, exact;
    int rows;          // rows of X / Y
    int n_tile;        // UMMA N: 16..256, multiple of 16
    int tmem_cols;     // power of two >= n_acc * acc_stride
    int n_acc;         // accumulators in tensor memory (2 or 4, half per MMA issuer): the MMAs of a K block go to different ones, so
                       // that they do not wait for each other (an MMA into the same accumulator is ~240 cycles
                       // behind the one before, whatever N); the epilogue adds them in a fixed order
    int acc_stride;    // columns between accumulators
    __half* y;         // [rows][M]
    int epilogue;      // QW3_EPI_STORE, QW3_EPI_RESIDUAL (y = hadd(y, result), Inference.cu:1145-1156) or QW3_EPI_GELU
                       // (Inference.cu:271-279): what the batched prompt phase needs after wo / w2 and after w1
    float* part;       // split-K: fp32 partial products [splits][rows][M] (null: one split, y is written directly)
    int* err;
    int a_lbo, a_sbo, a_kstep;   // operand A descriptor: byte offsets between 64-output blocks, between 8-deep K blocks, per K=16 step
};

// One output element: fp32 sum -> fp16, then the epilogue in fp16 as the decode path does it.
__device__ __forceinline__ __half gemm_epilogue(float v, int epilogue, __half old) {
    const __half h = __float2half_rn(v);
    if (epilogue == QW3_EPI_RESIDUAL) return h_add(old, h);
    if (epilogue == QW3_EPI_GELU) return gelu_h(h);
    return h;
}

template <int GM_STAGES>
__global__ void __launch_bounds__(GM_THREADS, 1)
gemm_w4a16_tc_kernel(const __grid_constant__ CUtensorMap tmap_x, const GemmParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int x_bytes = p.n_tile * 128;                                   // [n_tile][64] fp16
    static_assert(GM_STAGES <= GM_MAX_STAGES && GM_STAGES >= GM_UNPACK_WARPS / 4, "ring depth");
    constexpr int GM_A_STAGES = GM_STAGES, GM_X_STAGES = GM_STAGES;
    uint8_t* a_st = smem;                                                 // GM_A_STAGES x 16 KB (1024-aligned)
    uint8_t* x_st = smem + GM_A_STAGES * GM_A_BYTES;                      // GM_X_STAGES x x_bytes (multiple of 1024)
    uint64_t* bars = reinterpret_cast<uint64_t*>(x_st + GM_X_STAGES * x_bytes);
    const uint32_t a_full = smem_u32(bars + 2 * GM_MAX_STAGES), a_empty = smem_u32(bars + 3 * GM_MAX_STAGES);
    const uint32_t x_full = smem_u32(bars + 4 * GM_MAX_STAGES), x_empty = a_empty;   // one release barrier per stage
    const uint32_t acc_full = smem_u32(bars + 6 * GM_MAX_STAGES), drain = smem_u32(bars);   // drain: one an issuer
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 6 * GM_MAX_STAGES + 1);
    volatile int* s_dead = reinterpret_cast<volatile int*>(tmem_slot + 1);   // bars: (6 * 24 + 2) * 8 bytes < 1280

    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int tile_m = blockIdx.x, tile_n = blockIdx.y;
    // split-K: grid.z CTAs share the K blocks of a tile; each handles [kb_lo, kb_lo + n_kb)
    const int n_kb_all = p.K / GM_BK;
    const int kb_lo = (int)((long long)blockIdx.z * n_kb_all / gridDim.z);
    const int n_kb = (int)((long long)(blockIdx.z + 1) * n_kb_all / gridDim.z) - kb_lo;

    if (tid == 0) {
        for (int s = 0; s < GM_X_STAGES; ++s) {
            mbar_init(x_full + 8 * s, 1);
        }
        for (int s = 0; s < GM_A_STAGES; ++s) {
            mbar_init(a_full + 8 * s, 4);       // the 4 unpack warps of the group that owns the K block
            mbar_init(a_empty + 8 * s, 1);      // commit of the MMAs that read A and X of the stage
        }
        mbar_init(acc_full, 2);             // the last commit of each of the two MMA issuers
        mbar_init(drain, 1);
        mbar_init(drain + 8, 1);
        *s_dead = 0;
        mbar_fence_init();
    }
    if (warp == 1) {   // tensor memory for the accumulators: 128 lanes x tmem_cols 32-bit columns
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(p.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        // ---------------- TMA producer of the activations ------------------------------------------
        // (the packed nibbles do not go through TMA: a 128-output tile is 64 bytes wide, and a box of 64 such rows
        // cost the copy engine more per K block than everything else in the CTA)
        if (elect_one()) {
            tma_prefetch_desc(&tmap_x);
            bool ok = true;
            int issued = 0;
            for (int kb = 0; kb < n_kb && ok; ++kb) {
                const int s = kb % GM_X_STAGES;
                if (kb >= GM_X_STAGES) ok = mbar_wait(x_empty + 8 * s, ((kb / GM_X_STAGES) - 1) & 1);   // freed by the MMAs' commit
                if (!ok) break;
                mbar_expect_tx(x_full + 8 * s, (uint32_t)x_bytes);
                tma_load_2d(smem_u32(x_st + s * x_bytes), &tmap_x, (kb_lo + kb) * GM_BK, tile_n * p.n_tile, x_full + 8 * s);
                ++issued;
            }
            if (!ok) {
                atomicCAS(p.err, 0, 0x30001);
                *s_dead = 1;
                for (int kb = issued > GM_X_STAGES ? issued - GM_X_STAGES : 0; kb < issued; ++kb)   // the copies in flight
                    mbar_wait(x_full + 8 * (kb % GM_X_STAGES), (uint32_t)(kb / GM_X_STAGES) & 1u);
            }
        }
    } else if (warp == 1 || warp == GM_ISSUER_B) {
        // ---------------- MMA issuers ------------------------------------------------------------
        // The instruction chain of an issuing lane (two barrier waits, four MMAs, one commit: ~900 cycles) is what a
        // K block costs a CTA when the row tile is small, so TWO warps issue: warp 1 takes the even K blocks, the
        // last warp the odd ones, each into its own accumulators (summed by the epilogue).  One lane per warp runs
        // the loop; ring indices and phases are running counters, descriptors a constant plus additions.
        if (elect_one()) {
            const int who = warp == 1 ? 0 : 1;
            // instruction descriptor: D = f32, A = B = f16, A MN-major (bit 15), B K-major, N >> 3, M >> 4
            const uint32_t idesc = (1u << 4) | (1u << 15) | ((uint32_t)(p.n_tile >> 3) << 17) | ((uint32_t)(GM_TILE_M >> 4) << 24);
            const uint64_t adesc0 = make_smem_desc(smem_u32(a_st), p.a_lbo, p.a_sbo);
            const uint64_t bdesc0 = make_smem_desc(smem_u32(x_st), 16, 1024);
            const uint32_t a_step = (uint32_t)(p.a_kstep >> 4), a_stage = (uint32_t)(GM_A_BYTES >> 4), x_stage = (uint32_t)(x_bytes >> 4);
            const int half_acc = p.n_acc >> 1;                        // accumulators of this issuer
            const uint32_t my_tmem = tmem_base + (uint32_t)(who * half_acc * p.acc_stride);
            int s = who;                                              // stage of K block `who` (GM_STAGES >= 2)
            uint32_t phase = 0;
            bool first = true;
            for (int kb = who; kb < n_kb; kb += 2) {
                if (*s_dead != 0) break;
                if (!(mbar_wait(x_full + 8 * s, phase) && mbar_wait(a_full + 8 * s, phase))) {
                    atomicCAS(p.err, 0, 0x30002);
                    *s_dead = 1;
                    break;
                }
                // A (MN-major): 64-output blocks 8 KB apart (LBO), 8-deep K blocks 1 KB apart (SBO); K=16 = 2 blocks
                // B (K-major): 8-row groups 1 KB apart (SBO); K=16 = 32 bytes inside the swizzled row
                const uint64_t adesc = adesc0 + (uint64_t)((uint32_t)s * a_stage);
                const uint64_t bdesc = bdesc0 + (uint64_t)((uint32_t)s * x_stage);
#pragma unroll
                for (int ks = 0; ks < GM_BK / 16; ++ks) {
                    const int acc = ks & (half_acc - 1);
                    umma_f16(my_tmem + (uint32_t)(acc * p.acc_stride), adesc + (uint64_t)(ks * a_step), bdesc + (uint64_t)(ks * 2), idesc,
                             (!first || ks >= half_acc) ? 1u : 0u);
                }
                first = false;
                umma_commit(a_empty + 8 * s);    // A and X of the stage are free once these MMAs have read them
                if (kb + 2 >= n_kb) umma_commit(acc_full);   // this issuer's last K block
                s += 2;
                if (s >= GM_STAGES) { s -= GM_STAGES; phase ^= 1u; }
            }
            // Drain: the release arrivals of this issuer's last K blocks are waited for by nobody else (no later block
            // reuses those stages).  They must have landed before the CTA exits, or they would hit the barriers of
            // the next CTA that gets this shared memory.
            for (int kb = who; kb < n_kb; kb += 2) {
                if (kb + GM_STAGES < n_kb || *s_dead != 0) continue;
                if (!mbar_wait(a_empty + 8 * (kb % GM_STAGES), (uint32_t)(kb / GM_STAGES) & 1u)) {
                    atomicCAS(p.err, 0, 0x30006);
                    *s_dead = 1;
                }
            }
            if (*s_dead != 0) {   // some wait gave up: the MMAs in flight
                umma_commit(drain + 8 * who);
                mbar_wait(drain + 8 * who, 0);
            }
        }
        __syncwarp();
    } else {
        // ---------------- unpack warps (2..17), then epilogue -----------------------------------
        const int grp = (warp - 2) >> 2;          // group g unpacks the K blocks g, g + 4, ...
        const int ut = (tid - 64) & 127;          // 0..127 inside the group
        const int c4 = ut & 3, krow = ut >> 2;    // 16-byte chunk (32 outputs) of a row; row 0..31 (+32)
        const int ib = tile_m;                    // the tile is exactly one block of 128 outputs
        const int ibk = ib % p.Kb;
        DqConst ku = {0u, 0u, 0u};
        if (p.uniform) {
            const int g = ibk % p.n_alloc;
            ku = p.exact ? make_const<true>(p.zp[g], p.scale[g]) : make_const<false>(p.zp[g], p.scale[g]);
        }
        bool dead = false;
        // this thread's two 16-byte pieces of a K block (rows krow and krow + 32), requested two own blocks ahead
        const size_t pitch = (size_t)p.M / 2;
        const uint8_t* gsrc = p.packed + (size_t)tile_m * (GM_TILE_M / 2) + c4 * 16;
        auto request = [&](const int kb, uint4 (&dst)[2]) {
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const size_t row = (size_t)(kb_lo + kb) * GM_BK + krow + pass * 32;
                dst[pass] = kb < n_kb ? __ldg(reinterpret_cast<const uint4*>(gsrc + row * pitch)) : make_uint4(0u, 0u, 0u, 0u);
            }
        };
        uint4 nxt[2], nxt2[2];   // two own K blocks in flight
        request(grp, nxt);
        request(grp + GM_UNPACK_WARPS / 4, nxt2);
        for (int kb = grp; kb < n_kb && !dead; kb += GM_UNPACK_WARPS / 4) {
            const int t = kb % GM_A_STAGES;
            const uint4 cur[2] = {nxt[0], nxt[1]};
            nxt[0] = nxt2[0];
            nxt[1] = nxt2[1];
            request(kb + 2 * (GM_UNPACK_WARPS / 4), nxt2);
            if (kb >= GM_A_STAGES && !mbar_wait(a_empty + 8 * t, ((kb / GM_A_STAGES) - 1) & 1)) {
                if (lane == 0) atomicCAS(p.err, 0, 0x30003);
                *s_dead = 1;
                dead = true;
                break;
            }
            uint8_t* adst = a_st + t * GM_A_BYTES + (c4 >> 1) * 8192;
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const int k = krow + pass * 32;
                const uint4 raw = cur[pass];
                DqConst kc = ku;
                if (!p.uniform) {
                    const long long j = (long long)(kb_lo + kb) * GM_BK + k;
                    int g = ibk + (int)((j * p.Mb) % p.Kb);
                    g -= g >= p.Kb ? p.Kb : 0;
                    g %= p.n_alloc;
                    kc = p.exact ? make_const<true>(p.zp[g], p.scale[g]) : make_const<false>(p.zp[g], p.scale[g]);
                }
                const uint32_t w4[4] = {raw.x, raw.y, raw.z, raw.w};
                uint8_t* rowp = adst + (k >> 3) * 1024 + (k & 7) * 128;
#pragma unroll
                for (int wd = 0; wd < 4; ++wd) {
                    uint32_t lo0, hi0, lo1, hi1;
                    if (p.exact) {
                        dq_pair<true>(w4[wd], kc, lo0, hi0);
                        dq_pair<true>(w4[wd] >> 8, kc, lo1, hi1);
                    } else {
                        dq_pair<false>(w4[wd], kc, lo0, hi0);
                        dq_pair<false>(w4[wd] >> 8, kc, lo1, hi1);
                    }
                    const int chunk = 4 * (c4 & 1) + wd;   // 8 outputs, stored in unpack order (0,4,1,5,2,6,3,7)
                    *reinterpret_cast<uint4*>(rowp + ((chunk ^ (k & 7)) << 4)) = make_uint4(lo0, hi0, lo1, hi1);
                }
            }
            // generic-proxy writes of A must be visible to the tensor core (async proxy) before the arrive
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(a_full + 8 * t);
        }
        // ---------------- epilogue: accumulators -> fp16 Y ----------------------------------------
        if (!dead && *s_dead == 0 && !mbar_wait(acc_full, 0)) {
            if (lane == 0) atomicCAS(p.err, 0, 0x30004);
            *s_dead = 1;
            dead = true;
        }
        if (!dead && *s_dead == 0) {
            tc_fence_after();
            const int q = warp & 3;                           // TMEM lanes 32q..32q+31 belong to this warp
            const int m = 32 * q + lane;                      // row of A = TMEM lane
            const int pos = m & 7;                            // position inside the 8-group, in unpack order
            const int nib = (pos >> 1) + ((pos & 1) << 2);    // 0,4,1,5,2,6,3,7
            const int i = tile_m * GM_TILE_M + (m & ~7) + nib;
            // the warps of a lane quarter take the 16-column groups in turn
            for (int c0 = 16 * ((warp - 2) >> 2); c0 < p.n_tile; c0 += 16 * (GM_UNPACK_WARPS / 4)) {
                uint32_t v[16];
                tmem_ld16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, v);
                float f[16];
#pragma unroll
                for (int e = 0; e < 16; ++e) f[e] = __uint_as_float(v[e]);
                for (int acc = 1; acc < p.n_acc; ++acc) {   // fixed order: accumulator 0 + 1 + 2 + 3
                    tmem_ld16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(acc * p.acc_stride + c0), v);
#pragma unroll
                    for (int e = 0; e < 16; ++e) f[e] += __uint_as_float(v[e]);
                }
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const int r = tile_n * p.n_tile + c0 + e;
                    if (r < p.rows) {
                        if (p.part != nullptr) p.part[((size_t)blockIdx.z * p.rows + r) * p.M + i] = f[e];
                        else {
                            __half* dst = p.y + (size_t)r * p.M + i;
                            *dst = gemm_epilogue(f[e], p.epilogue, p.epilogue == QW3_EPI_RESIDUAL ? *dst : __half());
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(p.tmem_cols) : "memory");
    }
}

// Split-K: sums the fp32 partial products of the splits in split order and rounds once to fp16.
__global__ void gemm_splitk_reduce_kernel(const float* __restrict__ part, int splits, long long n, int epilogue, __half* y) {
    const long long i = 2 * ((long long)blockIdx.x * blockDim.x + threadIdx.x);
    if (i >= n) return;
    float2 acc = *reinterpret_cast<const float2*>(part + i);
    for (int z = 1; z < splits; ++z) {
        const float2 v = *reinterpret_cast<const float2*>(part + (size_t)z * n + i);
        acc.x += v.x;
        acc.y += v.y;
    }
    const __half2 old = epilogue == QW3_EPI_RESIDUAL ? *reinterpret_cast<const __half2*>(y + i) : __half2();
    *reinterpret_cast<__half2*>(y + i) =
        __halves2half2(gemm_epilogue(acc.x, epilogue, __low2half(old)), gemm_epilogue(acc.y, epilogue, __high2half(old)));
}

// ---- CTA pairs ------------------------------------------------------------------------------------------------------------------
// Most calls of more than 128 rows, and those with more output tiles than pairs (pair_wanted).  Back to back, one-CTA kernel / pairs:
// 2048 rows of 12288 x 4096 202 / 158 us (0.76 of the measured bf16 rate), 64 rows of 151936 x 4096 250 / 193.  Bound: a K block takes
// 0.33 us from the unpack warps to the freed stage whatever the row count, 0.39 at 256 rows, where its MMAs take 0.28.
// Two SMs of a cluster work on one tile of 256 outputs x n_tile rows (tcgen05 cta_group::2): each CTA unpacks operand A for its
// own 128 outputs and holds half of the activation rows, so that a K block moves half the operand-B bytes through an SM's
// shared memory (A 16 KB written + 16 KB read, B 16 KB + 16 KB, in the 512 cycles the MMAs take at 256 rows) and half through L2.
//   warp 0      TMA producer of this CTA's half of the activation rows
//   warp 1      MMA issuer (leader CTA of the pair only), K blocks in turn into two to four accumulators
//   warps 2..17 unpack (four groups of four warps take the K blocks in turn), epilogue
//   warp 18     loader: the packed bytes of this CTA's outputs into a ring of twelve K blocks (cp.async, 64 bytes of a row; a tensor
//               copy of such a narrow box costs more than all else in the CTA).  The unpack warps must not have loads
//               from global memory in flight: the fence that hands operand A to the tensor cores waits for them.
// Operand A is K-major: a thread takes 8 outputs x 8 inputs (one 32-bit word of eight rows); a byte permute joins
// the same byte of two neighbouring rows, and the masks that pick the nibbles then give half2 pairs along K with no
// more instructions than pairs along the outputs cost.  Row m of A holds output 8 (m & 15) + (m >> 4) of its block, which
// makes the 16-byte stores of a warp free of bank conflicts; the epilogue undoes it through a staging tile and stores
// 16 bytes a thread.  The pairs are persistent and take the work items (tile x K split) round robin.
constexpr int GP_STAGES = 5;
constexpr int GP_PK_STAGES = 12, GP_PK_BYTES = GM_BK * 64;           // ring of packed K blocks: 48 KB on the way to an SM
constexpr int GP_MAX_N = 256;
constexpr int GP_X_BYTES = GP_MAX_N / 2 * 128;                       // this CTA's half of the activation rows, 64 deep
constexpr int GP_WARPS = 16, GP_GROUPS = GP_WARPS / 4;
constexpr int GP_LOADER = 2 + GP_WARPS;                              // warp index of the loader of packed bytes
constexpr int GP_THREADS = 32 * (GP_LOADER + 1);
constexpr int GP_STG_LD = 136;                                       // halves per staged row: 272 B, 16-byte pieces of a row aligned
constexpr int GP_STG_BYTES = 16 * GP_STG_LD * 2;                     // 16 rows x 128 outputs per group
constexpr int GP_TAB = 256;                                          // groups of a column: in_dim / 128 <= 256
constexpr size_t GP_SMEM = (size_t)GP_STAGES * (GM_A_BYTES + GP_X_BYTES) + GP_PK_STAGES * GP_PK_BYTES + GP_GROUPS * GP_STG_BYTES + GP_TAB * 4 + 512;

struct PairParams {
    const uint8_t* packed;
    const __half* scale;
    const __half* zp;
    int n_alloc, M, K, Mb, Kb;
    int rows, n_tile, n_tiles_n, n_tiles_m;
    int n_acc, acc_stride;   // accumulators of a tile, which its K blocks take in turn, and the columns between them
    int full;          // tiles whose K is not split
    int splits;        // parts of the K of each of the tiles after those
    int items;         // full + splits * (the other tiles)
    int epilogue;
    __half* y;         // [rows][M]
    float* part;       // partial products of the split tiles: [tile][split][n_tile][256] in the order of A's rows
    int* err;
};

__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// Arrive on the barrier at the same shared-memory offset in the pair's leader (rank 0; the leader itself included).  What is handed
// over lies in this CTA's own shared or tensor memory, has been fenced for the tensor cores (fence.proxy.async, tcgen05.fence),
// and only they read it.  Without qualifiers the arrive releases at CTA scope; this is the form in which CUTLASS hands
// operands transformed by the peer CTA to the leader's tcgen05 instructions (ClusterBarrier::arrive of a CTA of the cluster).
// Release and acquire at cluster scope, sent by one warp of the peer that does nothing else, take 330 us where this takes 157
// (2048 rows of 12288 x 4096): a memory barrier on each side of every K block.
__device__ __forceinline__ void mbar_arrive_leader(uint32_t bar) {
    asm volatile(
        "{\n\t.reg .b32 a;\n\t"
        "mapa.shared::cluster.u32 a, %0, 0;\n\t"
        "mbarrier.arrive.shared::cluster.b64 _, [a];\n\t}"
        ::"r"(bar) : "memory");
}
// Box of the tensor map into this CTA's shared memory, completing on the leader's barrier (bit 24 of a shared::cluster address
// is the CTA's place in the pair).
__device__ __forceinline__ void tma_load_2d_pair(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(bar & 0xFEFFFFFFu) : "memory");
}
__device__ __forceinline__ void umma_f16_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit_pair(uint32_t bar) {   // arrives at the same offset in both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(bar), "h"((unsigned short)3) : "memory");
}
__device__ __forceinline__ uint32_t h2_add(uint32_t a, uint32_t b) {
    uint32_t r;
    asm("add.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
    return r;
}
__device__ __forceinline__ uint32_t prmt(uint32_t a, uint32_t b, uint32_t sel) {
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
    return r;
}

// A wait of the leader's MMA issuer has given up: it waits for the copies of the activations in flight.  Both producers give up after it
// at the latest (no commit frees their stages) and then leave 1 + the K blocks they have asked for in `asked`, the peer from its own
// SM.  A lap of a stage completes with the leader's expectation and the bytes of both CTAs; they are never more than a lap apart.
__device__ __noinline__ void pair_drain(uint32_t x_full, const volatile int* asked, uint32_t half_bytes) {
    const long long t0 = clock64();
    while (asked[0] == 0 || asked[1] == 0)
        if (clock64() - t0 > (1ll << 32)) return;
    for (int s = 0; s < GP_STAGES; ++s) {
        const int laps0 = (asked[0] - 1 - s + GP_STAGES - 1) / GP_STAGES, laps1 = (asked[1] - 1 - s + GP_STAGES - 1) / GP_STAGES;
        const int laps = max(laps0, laps1);
        if (laps <= 0) continue;
        if (laps1 > laps0) mbar_expect_tx(x_full + 8 * s, half_bytes);   // the peer's half alone is on its way
        else if (laps0 > laps1)                                          // the peer's half will not come
            asm volatile("mbarrier.complete_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(x_full + 8 * s), "r"(half_bytes) : "memory");
        mbar_wait(x_full + 8 * s, (uint32_t)(laps - 1) & 1u);
    }
}

// One work item: tile and K range.  Neighbouring items share the 256 outputs and differ in the rows.
struct PairItem { int tile_m, tile_n, kb_lo, n_kb, slot; };   // slot: place of the partial products, negative: none
__device__ __forceinline__ PairItem pair_item(const PairParams& p, int item) {
    PairItem w;
    const int n_kb = p.K / GM_BK;
    int tile = item;
    w.kb_lo = 0;
    w.n_kb = n_kb;
    w.slot = item - p.full;
    if (w.slot >= 0) {
        const int z = w.slot % p.splits;
        tile = p.full + w.slot / p.splits;
        w.kb_lo = z * n_kb / p.splits;
        w.n_kb = (z + 1) * n_kb / p.splits - w.kb_lo;
    }
    w.tile_n = tile % p.n_tiles_n;
    w.tile_m = tile / p.n_tiles_n;
    return w;
}
// Barrier of the four warps of a group that tells all of them whether one has given up.
__device__ __forceinline__ bool group_any(int id, bool v) {
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %2, 0;\n\t"
        "barrier.cta.red.or.aligned.pred q, %1, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(r) : "r"(id), "r"((uint32_t)v) : "memory");
    return r != 0;
}

template <bool EXACT, bool UNIFORM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(GP_THREADS, 1)
gemm_w4a16_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const PairParams p) {
    extern __shared__ __align__(1024) uint8_t smem[];
    uint8_t* a_st = smem;
    uint8_t* x_st = a_st + GP_STAGES * GM_A_BYTES;
    uint8_t* pk_st = x_st + GP_STAGES * GP_X_BYTES;
    uint8_t* stg = pk_st + GP_PK_STAGES * GP_PK_BYTES;
    uint32_t* tab = reinterpret_cast<uint32_t*>(stg + GP_GROUPS * GP_STG_BYTES);   // (zero point, scale) of a group
    uint64_t* bars = reinterpret_cast<uint64_t*>(tab + GP_TAB);
    const uint32_t a_full = smem_u32(bars), x_full = smem_u32(bars + GP_STAGES), st_empty = smem_u32(bars + 2 * GP_STAGES);
    const uint32_t acc_full = smem_u32(bars + 3 * GP_STAGES), acc_empty = smem_u32(bars + 3 * GP_STAGES + 1);
    const uint32_t pk_full = smem_u32(bars + 3 * GP_STAGES + 2), pk_empty = pk_full + 8 * GP_PK_STAGES;
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * GP_STAGES + 2 + 2 * GP_PK_STAGES);
    volatile int* s_dead = reinterpret_cast<volatile int*>(tmem_slot + 1);
    volatile int* s_asked = s_dead + 1;   // pair_drain
    const uint32_t drain = smem_u32(tmem_slot + 4);

    const int tid = threadIdx.x, warp = warp_index(), lane = tid & 31;
    const int rank = (int)cluster_rank();
    const int first = blockIdx.x >> 1, step = gridDim.x >> 1, items = p.items;

    if (tid == 0) {
        for (int s = 0; s < GP_STAGES; ++s) {
            mbar_init(a_full + 8 * s, 8);       // four unpack warps of each CTA (used in the leader)
            mbar_init(x_full + 8 * s, 1);       // the leader's expect; bytes of both CTAs' copies
            mbar_init(st_empty + 8 * s, 1);     // commit of the MMAs that read the stage
        }
        for (int s = 0; s < GP_PK_STAGES; ++s) {
            mbar_init(pk_full + 8 * s, 32);     // the loader's lanes, each when its copies have landed
            mbar_init(pk_empty + 8 * s, 4);     // the warps of the group that took the block
        }
        mbar_init(acc_full, 1);                 // commit of an item's last MMAs
        mbar_init(acc_empty, 2 * GP_WARPS);     // every epilogue warp of the pair has read its share
        mbar_init(drain, 1);
        *s_dead = s_asked[0] = s_asked[1] = 0;
        mbar_fence_init();
    }
    for (int g = tid; g < p.Kb; g += GP_THREADS) tab[g] = pack_h2(p.zp[g % p.n_alloc], p.scale[g % p.n_alloc]);
    if (warp == 1) {   // all 512 columns
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();   // the peer's barriers are initialised before anything arrives on them
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp == 0) {
        if (elect_one()) {
            tma_prefetch_desc(&tmap_x);
            const int half_n = p.n_tile / 2;
            int s = 0, asked = 0;
            uint32_t phase = 0;
            bool ok = true, wrapped = false;
            for (int item = first; item < items && ok; item += step) {
                const PairItem w = pair_item(p, item);
                for (int kb = 0; kb < w.n_kb; ++kb) {
                    if (wrapped && !(ok = mbar_wait(st_empty + 8 * s, phase ^ 1u))) break;
                    if (*s_dead != 0) { ok = false; break; }
                    if (rank == 0) mbar_expect_tx(x_full + 8 * s, (uint32_t)p.n_tile * 128u);
                    tma_load_2d_pair(smem_u32(x_st + s * GP_X_BYTES), &tmap_x, (w.kb_lo + kb) * GM_BK,
                                     w.tile_n * p.n_tile + rank * half_n, x_full + 8 * s);
                    ++asked;
                    if (++s == GP_STAGES) { s = 0; phase ^= 1u; wrapped = true; }
                }
            }
            // drain: the release arrivals of the last laps land before this CTA may leave
            for (int t = 0; t < GP_STAGES && ok; ++t)
                if (t < s || wrapped) ok = mbar_wait(st_empty + 8 * t, t < s ? phase : phase ^ 1u);
            if (!ok) {
                atomicCAS(p.err, 0, 0x30011);
                *s_dead = 1;
                const uint32_t word = smem_u32(const_cast<int*>(s_asked)) + 4 * rank;   // in the leader
                asm volatile(
                    "{\n\t.reg .b32 a;\n\t"
                    "mapa.shared::cluster.u32 a, %0, 0;\n\t"
                    "st.shared::cluster.u32 [a], %1;\n\t}"
                    ::"r"(word), "r"(asked + 1) : "memory");
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (rank == 0 && elect_one()) {
            // D = f32, A = B = f16, both K-major, N >> 3, M >> 4
            const uint32_t idesc = (1u << 4) | ((uint32_t)(p.n_tile >> 3) << 17) | ((uint32_t)(256 >> 4) << 24);
            const uint64_t adesc0 = make_smem_desc(smem_u32(a_st), 16, 1024), bdesc0 = make_smem_desc(smem_u32(x_st), 16, 1024);
            int s = 0, n = 0;
            uint32_t phase = 0;
            bool ok = true;
            for (int item = first; item < items && ok; item += step, ++n) {
                const PairItem w = pair_item(p, item);
                if (n > 0 && !(ok = mbar_wait(acc_empty, (uint32_t)(n - 1) & 1u))) break;
                tc_fence_after();
                int acc = 0;
                for (int kb = 0; kb < w.n_kb; ++kb) {
                    if (*s_dead != 0 || !mbar_wait(x_full + 8 * s, phase) || !mbar_wait(a_full + 8 * s, phase)) {
                        ok = false;
                        break;
                    }
                    tc_fence_after();
                    const uint64_t adesc = adesc0 + (uint64_t)(uint32_t)(s * (GM_A_BYTES >> 4));
                    const uint64_t bdesc = bdesc0 + (uint64_t)(uint32_t)(s * (GP_X_BYTES >> 4));
                    const uint32_t d = tmem_base + (uint32_t)(acc * p.acc_stride);
#pragma unroll
                    for (int ks = 0; ks < GM_BK / 16; ++ks)
                        umma_f16_pair(d, adesc + (uint64_t)(2 * ks), bdesc + (uint64_t)(2 * ks), idesc, (kb >= p.n_acc || ks > 0) ? 1u : 0u);
                    umma_commit_pair(st_empty + 8 * s);
                    if (++acc == p.n_acc) acc = 0;
                    if (++s == GP_STAGES) { s = 0; phase ^= 1u; }
                }
                if (ok) umma_commit_pair(acc_full);
            }
            if (!ok) {
                atomicCAS(p.err, 0, 0x30012);
                *s_dead = 1;
                asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(drain) : "memory");
                mbar_wait(drain, 0);   // the MMAs in flight
                pair_drain(x_full, s_asked, (uint32_t)p.n_tile * 64u);
            }
        }
        __syncwarp();
    } else if (warp == GP_LOADER) {
        const size_t pitch = (size_t)p.M / 2;
        const int row = lane >> 2, ch = lane & 3;   // 16 bytes of every eighth row
        int s = 0;
        uint32_t phase = 0;
        bool ok = true, wrapped = false;
        for (int item = first; item < items && ok; item += step) {
            const PairItem w = pair_item(p, item);
            const int block = 2 * w.tile_m + rank;
            const uint8_t* src = p.packed + ((size_t)w.kb_lo * GM_BK + row) * pitch + (size_t)block * 64 + ch * 16;
            for (int kb = 0; kb < w.n_kb; ++kb) {
                if (wrapped) ok = __all_sync(0xffffffffu, *s_dead == 0 && mbar_wait(pk_empty + 8 * s, phase ^ 1u));
                if (!ok) break;
                if (block < p.Mb) {
                    const uint32_t dst = smem_u32(pk_st + s * GP_PK_BYTES) + ch * 16;
#pragma unroll
                    for (int q = 0; q < 8; ++q)   // the rows of an odd eight lie swapped in pairs
                        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                                     ::"r"(dst + (uint32_t)((8 * q + (row ^ (q & 1))) * 64)), "l"(src + (size_t)(8 * q) * pitch) : "memory");
                }
                src += (size_t)GM_BK * pitch;
                asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(pk_full + 8 * s) : "memory");
                if (++s == GP_PK_STAGES) { s = 0; phase ^= 1u; wrapped = true; }
            }
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (!ok) {
            if (lane == 0) atomicCAS(p.err, 0, 0x30015);
            *s_dead = 1;
        }
        __syncwarp();
    } else {
        const int grp = (warp - 2) >> 2;
        const int ut = (tid - 64) & 127, c = ut & 15, kc = ut >> 4;   // 8 outputs 8c.., 8 inputs 8kc.. of a K block
        const int d_step = p.Mb % p.Kb;
        // this thread's word of row 8 kc of a packed K block; the swap keeps the two kc of a warp off each other's banks
        const uint32_t* pk_thr = reinterpret_cast<const uint32_t*>(pk_st + kc * 512 + c * 4);
        const int pk_swap = kc & 1;
        const uint32_t a_thr = (uint32_t)(c * 128 + ((kc ^ (c & 7)) << 4));
        int s = grp, lap = 0;   // stage and lap of this group's next K block
        int ps = grp;           // its place in the packed ring (a multiple of the groups: the laps of a group's places agree)
        uint32_t pphase = 0;
        int kb = grp, n = 0;
        bool dead = false;
        PairItem w = pair_item(p, first);
        for (int item = first; item < items; item += step, ++n) {
            const int block = 2 * w.tile_m + rank, ibk = block % p.Kb;
            const bool valid = block < p.Mb;
            DqConst ku = {0u, 0u, 0u};
            if (UNIFORM) {
                const uint32_t e = tab[ibk];
                ku = make_const<EXACT>(__ushort_as_half((unsigned short)e), __ushort_as_half((unsigned short)(e >> 16)));
            }
            for (; kb < w.n_kb; kb += GP_GROUPS) {   // this group's K blocks of the item
                bool ok = mbar_wait(pk_full + 8 * ps, pphase);
                uint32_t cur[8];
#pragma unroll
                for (int r = 0; r < 8; ++r) cur[r] = pk_thr[ps * (GP_PK_BYTES / 4) + (r ^ pk_swap) * 16];
                __syncwarp();
                if (lane == 0) mbar_arrive(pk_empty + 8 * ps);
                ps += GP_GROUPS;
                if (ps >= GP_PK_STAGES) { ps -= GP_PK_STAGES; pphase ^= 1u; }
                ok = ok && (lap == 0 || mbar_wait(st_empty + 8 * s, (uint32_t)(lap - 1) & 1u));
                if (!__all_sync(0xffffffffu, ok && *s_dead == 0)) {
                    if (lane == 0) atomicCAS(p.err, 0, 0x30013);
                    *s_dead = 1;
                    dead = true;
                    break;
                }
                if (valid) {
                    uint8_t* dst = a_st + s * GM_A_BYTES + a_thr;
                    DqConst kq[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) kq[q] = ku;
                    if (!UNIFORM) {   // the group moves by d_step from one input to the next
                        const int j = (w.kb_lo + kb) * GM_BK + kc * 8;
                        int g = (ibk + (j % p.Kb) * d_step) % p.Kb;
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            const uint32_t e0 = tab[g];
                            g += d_step;
                            g -= g >= p.Kb ? p.Kb : 0;
                            const uint32_t e1 = tab[g];
                            g += d_step;
                            g -= g >= p.Kb ? p.Kb : 0;
                            const DqConst k0 = make_const<EXACT>(__ushort_as_half((unsigned short)e0), __ushort_as_half((unsigned short)(e0 >> 16)));
                            const DqConst k1 = make_const<EXACT>(__ushort_as_half((unsigned short)e1), __ushort_as_half((unsigned short)(e1 >> 16)));
                            kq[q].z = prmt(k0.z, k1.z, 0x5410);
                            kq[q].hz = prmt(k0.hz, k1.hz, 0x5410);
                            kq[q].s = prmt(k0.s, k1.s, 0x5410);
                        }
                    }
#pragma unroll
                    for (int b = 0; b < 4; ++b) {   // outputs 2b and 2b + 1
                        uint32_t lo[4], hi[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            dq_pair<EXACT>(prmt(cur[2 * q], cur[2 * q + 1], (uint32_t)(b | b << 4 | (4 + b) << 8 | (4 + b) << 12)), kq[q], lo[q], hi[q]);
                        *reinterpret_cast<uint4*>(dst + (2 * b) * 2048) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
                        *reinterpret_cast<uint4*>(dst + (2 * b + 1) * 2048) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
                    }
                }
                // generic-proxy writes of A must be visible to the tensor core (async proxy) before the arrive
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive_leader(a_full + 8 * s);
                s += GP_GROUPS;
                if (s >= GP_STAGES) { s -= GP_STAGES; ++lap; }
            }
            // ---- epilogue: accumulators -> staging -> Y
            if (!dead && !mbar_wait(acc_full, (uint32_t)n & 1u)) {
                if (lane == 0) atomicCAS(p.err, 0, 0x30014);
                *s_dead = 1;
                dead = true;
            }
            __syncwarp();
            dead = group_any(1 + grp, dead);   // the four warps meet in the staging tile: they go on, or leave, together
            if (dead) break;
            tc_fence_after();
            const int q = warp & 3, m = 32 * q + lane;
            __half* sg = reinterpret_cast<__half*>(stg + grp * GP_STG_BYTES);
            const int i_local = 8 * (m & 15) + (m >> 4);
            for (int c0 = 16 * grp; c0 < p.n_tile; c0 += 16 * GP_GROUPS) {
                const int r0 = w.tile_n * p.n_tile + c0;
                if (r0 >= p.rows) break;       // uniform over the group
                uint32_t v[16];
                float f[16];
                tmem_ld16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)c0, v);
#pragma unroll
                for (int e = 0; e < 16; ++e) f[e] = __uint_as_float(v[e]);
                tmem_ld16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(p.acc_stride + c0), v);
#pragma unroll
                for (int e = 0; e < 16; ++e) f[e] += __uint_as_float(v[e]);
                for (int acc = 2; acc < p.n_acc; ++acc) {   // in a fixed order
                    tmem_ld16(tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(acc * p.acc_stride + c0), v);
#pragma unroll
                    for (int e = 0; e < 16; ++e) f[e] += __uint_as_float(v[e]);
                }
                if (!valid) continue;
                if (w.slot >= 0) {
                    float* dst = p.part + ((size_t)w.slot * p.n_tile + c0) * 256 + rank * 128 + m;
#pragma unroll
                    for (int e = 0; e < 16; ++e) dst[(size_t)e * 256] = f[e];
                    continue;
                }
#pragma unroll
                for (int e = 0; e < 16; ++e) {
                    const __half h = __float2half_rn(f[e]);
                    sg[e * GP_STG_LD + i_local] = p.epilogue == QW3_EPI_GELU ? gelu_h(h) : h;
                }
                named_barrier(1 + grp, 128);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const int piece = ut + 128 * k, e = piece >> 4, o8 = piece & 15;
                    if (r0 + e < p.rows) {
                        uint4 o = *reinterpret_cast<const uint4*>(sg + e * GP_STG_LD + o8 * 8);
                        uint4* dst = reinterpret_cast<uint4*>(p.y + (size_t)(r0 + e) * p.M + (size_t)block * 128 + o8 * 8);
                        if (p.epilogue == QW3_EPI_RESIDUAL) {
                            const uint4 old = *dst;
                            o = make_uint4(h2_add(old.x, o.x), h2_add(old.y, o.y), h2_add(old.z, o.z), h2_add(old.w, o.w));
                        }
                        *dst = o;
                    }
                }
                named_barrier(1 + grp, 128);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_leader(acc_empty);
            kb = (kb - w.n_kb) & (GP_GROUPS - 1);   // first own K block of the next item
            if (item + step < items) w = pair_item(p, item + step);
        }
    }
    // nothing arrives at a CTA that has left: the producers and the epilogue warps have waited for every commit of their CTA
    tc_fence_before();
    __syncthreads();
    cluster_sync_all();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512) : "memory");
    }
}

// Sums the partial products of the split tiles in split order, rounds once to fp16 and stores two outputs a thread.
__global__ void __launch_bounds__(256) gemm_pair_reduce_kernel(const PairParams p) {
    const int tile = p.full + blockIdx.x, r = blockIdx.y * 2 + (threadIdx.x >> 7);
    const int row = (tile % p.n_tiles_n) * p.n_tile + r, i = (threadIdx.x & 127) * 2, out = (tile / p.n_tiles_n) * 256 + i;
    if (row >= p.rows || out >= p.M) return;
    const int at = (i & 128) + 16 * (i & 7) + ((i & 127) >> 3);   // A's row of output i; output i + 1 is 16 rows on
    const float* src = p.part + ((size_t)blockIdx.x * p.splits * p.n_tile + r) * 256 + at;
    float a = src[0], b = src[16];
#pragma unroll 4
    for (int z = 1; z < p.splits; ++z) {
        src += (size_t)p.n_tile * 256;
        a += src[0];
        b += src[16];
    }
    __half2* dst = reinterpret_cast<__half2*>(p.y + (size_t)row * p.M + out);
    const __half2 old = p.epilogue == QW3_EPI_RESIDUAL ? *dst : __half2();
    *dst = __halves2half2(gemm_epilogue(a, p.epilogue, __low2half(old)), gemm_epilogue(b, p.epilogue, __high2half(old)));
}

// ---------------------------------------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

int encode_f16_map(CUtensorMap* map, const void* base, int rank, const uint64_t* dims, const uint64_t* strides, const uint32_t* box) {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult qres;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &qres) == cudaSuccess &&
            qres == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(f);
    });
    if (!fn) {
        set_last_error("cuTensorMapEncodeTiled is not available (no CUDA driver?)");
        return QW3_ERR_CUDA;
    }
    cuuint64_t d[3], s[2] = {0, 0};
    cuuint32_t b[3], estr[3] = {1, 1, 1};
    for (int i = 0; i < rank; ++i) {
        d[i] = dims[i];
        b[i] = box[i];
        if (i + 1 < rank) s[i] = strides[i];
    }
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, (cuuint32_t)rank, const_cast<void*>(base), d, s, b, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_last_error("cuTensorMapEncodeTiled failed with CUresult %d", (int)r);
        return QW3_ERR_CUDA;
    }
    return QW3_OK;
}
// Activation rows [rows][K] in boxes of 64 inputs x box_rows.
static int encode_rows(CUtensorMap* map, const void* x, int64_t rows, int64_t K, int box_rows) {
    const uint64_t dims[2] = {(uint64_t)K, (uint64_t)rows}, strides[1] = {(uint64_t)K * 2};
    const uint32_t box[2] = {GM_BK, (uint32_t)box_rows};
    return encode_f16_map(map, x, 2, dims, strides, box);
}

// How the one-CTA kernel cuts rows x M x K: few rows and few output tiles leave most SMs without a CTA, so K is split over grid.z (fp32
// partial products in the workspace, summed in split order by a second kernel) until ~one CTA per SM, while the partials fit.
struct OneCut { int n_tile, n_acc, ctas, splits; };
static OneCut one_cut(long long rows, long long M, int K, int sm_count) {
    OneCut c;
    c.n_tile = rows <= 16 ? 16 : rows <= 32 ? 32 : rows <= 64 ? 64 : rows <= 128 ? 128 : 256;
    c.n_acc = c.n_tile <= 64 ? 4 : 2;       // half of them per MMA issuer
    const long long ctas = (M / GM_TILE_M) * ((rows + c.n_tile - 1) / c.n_tile);
    c.ctas = (int)ctas;
    c.splits = 1;
    while (c.splits < 8 && ctas * (c.splits * 2) <= sm_count && (K / GM_BK) / (c.splits * 2) >= 8 &&
           (long long)(c.splits * 2) * rows * M <= (long long)WS_PARTIALS)
        c.splits *= 2;
    return c;
}
// MMAs that one accumulator of it sums (an issuer has every other K block, and two accumulators where there are four).  The error grows
// with that (64 rows of 151936 x 4096: 0.53 % of the results are not the nearest fp16 at 64 MMAs, 0.95 % at 128), so the pair kernel
// takes no cut in which it is more.
static int one_sum(const OneCut& c, int K) { return ((K / GM_BK + c.splits - 1) / c.splits + 1) / 2 * (2 * GM_BK / 16) / c.n_acc; }
// Accumulators (fewest: each is one more pass of the epilogue over tensor memory) with which n_kb blocks give sums of at most `longest`
// MMAs; 0: more than 512 columns hold.
static int pair_accumulators(int n_kb, int n_tile, int longest) {
    for (int a = 2; a <= 4 && a * n_tile <= 512; ++a)
        if ((n_kb + a - 1) / a * (GM_BK / 16) <= longest) return a;
    return 0;
}

// How rows x M x K is cut for the pair kernel: the width of a row tile and the K splits of the tiles that do not fill a wave of
// pairs; the cut with the lowest estimate, in us.  A K block takes 0.33 us at up to 128 rows (whatever the rows: the hand-over) and 0.39 at
// 256; an item 2.3 (epilogue) and 0.3 for each further pass over 128 rows of accumulators; the sum of split tiles 4 and 0.7 for a
// million partial products; a call 5.  Over 520 sizes the cut taken is 0.6 % slower than the fastest of those tried in the mean, 7 % in
// the 99th percentile.
struct PairCut { int n_tile, n_acc, full, splits, items; double us; };
static PairCut pair_cut(long long rows, int M, int K, int pairs, int longest) {   // n_tile 0: no cut with sums of at most `longest`
    const int n_kb = K / GM_BK, tiles_m = (M + 255) / 256;
    const int max_z = n_kb / 8 < 16 ? n_kb / 8 : 16;
    int kbs[17];   // K blocks of a part
    for (int z = 1; z <= max_z; ++z) kbs[z] = (n_kb + z - 1) / z;
    PairCut best = {};
    for (int n = 32; n <= GP_MAX_N && n - 32 < rows; n += 32) {
        const long long tiles = tiles_m * ((rows + n - 1) / n);
        const double kb_us = n > 128 ? 0.33 + 0.06 * (n - 128) / 128 : 0.33;
        const long long waves = tiles / pairs;
        const int tail = (int)(tiles - waves * pairs);
        for (int z = 1; z <= max_z; ++z) {   // in more than two waves the parts of a tail are no gain
            if (z > 1 && (tail == 0 || tail * z > 2 * pairs || tail * z * n > (int)(WS_PARTIALS / 256))) break;
            const int n_acc = pair_accumulators(z > 1 && waves == 0 ? kbs[z] : n_kb, n, longest);
            if (n_acc == 0) continue;
            const int tail_waves = tail == 0 ? 0 : tail * z <= pairs ? 1 : 2;
            const double item_us = 2.3 + 0.3 * (n_acc - 1) * n / 128;
            const double us = 5.0 + waves * (n_kb * kb_us + item_us) + tail_waves * (kbs[z] * kb_us + item_us) +
                              (z > 1 ? 4.0 + 0.7e-6 * 256 * tail * z * n : 0.0);
            if (best.n_tile == 0 || us < best.us) {
                best.n_tile = n;
                best.n_acc = n_acc;
                best.full = (int)(z > 1 ? tiles - tail : tiles);
                best.splits = z;
                best.items = best.full + (z > 1 ? tail * z : 0);
                best.us = us;
            }
        }
    }
    return best;
}

// The pairs where their estimate is the lower one (us, one-CTA kernel / pairs; 12288 x 4096: 35 / 28 at 160 rows, 68 / 53 at 512, 101 / 82 at
// 1024, 202 / 165 at 2048; 4096 x 12288 175 / 154 at 2048).  The one-CTA kernel stays ahead where it splits K and the workspace
// does not hold the partial products of as many parts of the pairs' tiles (4096 x 12288 at 280 rows 50 / 64, 8192 x 8192 at 129 rows
// 52 / 62) and with a single block of outputs, which leaves half of each pair idle (128 x 12288 at 1953 rows 26 / 29).  Up to 128 rows
// a call is short and the pairs' start and second kernel show (4096 x 4096 at 64 rows 16.4 / 20.6; 18944 x 2048, one wave of both,
// 20.0 / 20.6), unless there are more 256-output tiles than pairs of SMs (151936 x 4096 at 64 rows 250 / 196).  The result is stored by
// 16 bytes; an item has two K blocks for each unpack group.
static bool pair_wanted(const W4Desc* d, long long rows, const void* d_y, const Workspace* ws, PairCut* cut) {
    const int pairs = ws->sm_count / 2, K = (int)d->K;
    if (K / GM_BK < 2 * GP_GROUPS || pairs < 1 || (reinterpret_cast<uintptr_t>(d_y) & 15) != 0) return false;
    if (rows <= 128 && (d->M + 255) / 256 <= pairs) return false;
    const OneCut one = one_cut(rows, d->M, K, ws->sm_count);
    *cut = pair_cut(rows, (int)d->M, K, pairs, one_sum(one, K));
    if (cut->n_tile == 0) return false;
    if (rows <= 128) return true;
    const long long waves = (one.ctas * one.splits + ws->sm_count - 1) / ws->sm_count;
    const double one_us = 2.4 + waves * ((K / GM_BK + one.splits - 1) / one.splits * 0.433 + 10.5) + (one.splits > 1 ? 2.6 : 0.0);
    return cut->us <= one_us;
}

static int pair_launch(const W4Desc* d, const PairCut& cut, const void* d_x, long long rows, void* d_y, const Workspace* ws, cudaStream_t st,
                       int epilogue) {
    PairParams p = {};
    p.packed = d->packed;
    p.scale = d->scale; p.zp = d->zp; p.n_alloc = (int)d->n_alloc;
    p.M = (int)d->M; p.K = (int)d->K; p.Mb = p.M / 128; p.Kb = p.K / 128;
    p.rows = (int)rows;
    const int pairs = ws->sm_count / 2;
    p.n_acc = cut.n_acc;
    p.acc_stride = 512 / p.n_acc & ~31;
    p.n_tile = cut.n_tile; p.full = cut.full; p.splits = cut.splits; p.items = cut.items;
    p.n_tiles_m = (p.M + 255) / 256;
    p.n_tiles_n = (int)((rows + p.n_tile - 1) / p.n_tile);
    p.epilogue = epilogue;
    p.y = static_cast<__half*>(d_y);
    p.part = ws->partials;
    p.err = ws->err;
    CUtensorMap tmap_x;
    const int rc = encode_rows(&tmap_x, d_x, rows, d->K, p.n_tile / 2);
    if (rc != QW3_OK) return rc;
    static std::atomic<bool> attr_set[64];   // per device: the kernels' shared-memory limit is raised once
    int dev = 0;
    QW3_CUDA(cudaGetDevice(&dev));
    if (dev >= 64 || !attr_set[dev].load(std::memory_order_acquire)) {
        QW3_CUDA(cudaFuncSetAttribute(gemm_w4a16_pair_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GP_SMEM));
        QW3_CUDA(cudaFuncSetAttribute(gemm_w4a16_pair_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GP_SMEM));
        QW3_CUDA(cudaFuncSetAttribute(gemm_w4a16_pair_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GP_SMEM));
        QW3_CUDA(cudaFuncSetAttribute(gemm_w4a16_pair_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GP_SMEM));
        if (dev < 64) attr_set[dev].store(true, std::memory_order_release);
    }
    const unsigned grid = 2u * (unsigned)(p.items < pairs ? p.items : pairs);
    if (d->zp_integral) {
        if (d->uniform) gemm_w4a16_pair_kernel<true, true><<<grid, GP_THREADS, GP_SMEM, st>>>(tmap_x, p);
        else gemm_w4a16_pair_kernel<true, false><<<grid, GP_THREADS, GP_SMEM, st>>>(tmap_x, p);
    } else {
        if (d->uniform) gemm_w4a16_pair_kernel<false, true><<<grid, GP_THREADS, GP_SMEM, st>>>(tmap_x, p);
        else gemm_w4a16_pair_kernel<false, false><<<grid, GP_THREADS, GP_SMEM, st>>>(tmap_x, p);
    }
    QW3_CUDA(cudaGetLastError());
    if (p.splits > 1) {
        const dim3 g((unsigned)(p.n_tiles_m * p.n_tiles_n - p.full), (unsigned)(p.n_tile / 2));
        gemm_pair_reduce_kernel<<<g, 256, 0, st>>>(p);
        QW3_CUDA(cudaGetLastError());
    }
    return QW3_OK;
}

}  // namespace qw3

using namespace qw3;

namespace qw3 {
int gemm_launch(qw3_w4_t w, const void* d_x, int64_t rows, void* d_y, qw3_ws_t ws, void* stream, int epilogue);
}

extern "C" int qw3_gemm_w4a16(qw3_w4_t w, const void* d_x, int64_t rows, void* d_y, qw3_ws_t ws, void* stream) {
    return qw3::gemm_launch(w, d_x, rows, d_y, ws, stream, QW3_EPI_STORE);
}

extern "C" int qw3_gemm_w4a16_epilogue(qw3_w4_t w, const void* d_x, int64_t rows, void* d_y, qw3_ws_t ws, int32_t epilogue, void* stream) {
    return qw3::gemm_launch(w, d_x, rows, d_y, ws, stream, epilogue);
}

// The contraction with an optional epilogue (the engine's batched prompt phase fuses the residual add and the GeLU).
int qw3::gemm_launch(qw3_w4_t w, const void* d_x, int64_t rows, void* d_y, qw3_ws_t ws, void* stream, int epilogue) {
    QW3_REQUIRE(w && d_x && d_y && ws, "qw3_gemm_w4a16: null argument");
    QW3_REQUIRE(epilogue == QW3_EPI_STORE || epilogue == QW3_EPI_RESIDUAL || epilogue == QW3_EPI_GELU, "qw3_gemm_w4a16: epilogue");
    QW3_REQUIRE(rows >= 1 && rows <= (1 << 20), "qw3_gemm_w4a16: rows out of range");
    QW3_REQUIRE((reinterpret_cast<uintptr_t>(d_x) & 15) == 0, "qw3_gemm_w4a16: X must be 16-byte aligned");
    const W4Desc* d = w4_desc(w);
    PairCut pair = {};
    if (pair_wanted(d, rows, d_y, ws_struct(ws), &pair))
        return pair_launch(d, pair, d_x, rows, d_y, ws_struct(ws), static_cast<cudaStream_t>(stream), epilogue);
    GemmParams p = {};
    p.packed = d->packed;
    p.scale = d->scale; p.zp = d->zp; p.n_alloc = (int)d->n_alloc;
    p.M = (int)d->M; p.K = (int)d->K; p.Mb = p.M / 128; p.Kb = p.K / 128;
    p.uniform = d->uniform; p.exact = d->zp_integral;
    p.rows = (int)rows;
    const OneCut cut = one_cut(rows, d->M, p.K, ws_struct(ws)->sm_count);
    p.n_tile = cut.n_tile;
    p.n_acc = cut.n_acc;
    p.acc_stride = p.n_tile < 32 ? 32 : p.n_tile;
    p.tmem_cols = p.n_acc * p.acc_stride;   // 128, 128, 256, 256, 512 columns: powers of two
    p.y = static_cast<__half*>(d_y);
    p.epilogue = epilogue;
    p.err = ws_struct(ws)->err;
    p.a_lbo = 8192; p.a_sbo = 1024; p.a_kstep = 2048;
    CUtensorMap tmap_x;
    int rc;
    rc = encode_rows(&tmap_x, d_x, rows, d->K, p.n_tile);
    if (rc != QW3_OK) return rc;
    // shared memory per stage: 16 KB of operand A + n_tile x 128 bytes of activations; 6 stages (4 with 256-row tiles)
    const int stages = p.n_tile <= 128 ? 6 : 4;
    const size_t smem = (size_t)stages * (GM_A_BYTES + p.n_tile * 128) + 1280;
    static std::once_flag attr_once[16];
    int dev = 0;
    QW3_CUDA(cudaGetDevice(&dev));
    if (dev < 16)
        std::call_once(attr_once[dev], [] {
            cudaFuncSetAttribute(gemm_w4a16_tc_kernel<6>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
            cudaFuncSetAttribute(gemm_w4a16_tc_kernel<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
        });
    const int splits = cut.splits;
    p.part = splits > 1 ? ws_struct(ws)->partials : nullptr;
    dim3 grid((unsigned)(d->M / GM_TILE_M), (unsigned)((rows + p.n_tile - 1) / p.n_tile), (unsigned)splits);
    const cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (stages == 6)
        gemm_w4a16_tc_kernel<6><<<grid, GM_THREADS, smem, st>>>(tmap_x, p);
    else
        gemm_w4a16_tc_kernel<4><<<grid, GM_THREADS, smem, st>>>(tmap_x, p);
    QW3_CUDA(cudaGetLastError());
    if (splits > 1) {
        const long long n = rows * d->M;
        gemm_splitk_reduce_kernel<<<(unsigned)((n / 2 + 255) / 256), 256, 0, st>>>(p.part, splits, n, p.epilogue, p.y);
        QW3_CUDA(cudaGetLastError());
    }
    return QW3_OK;
}
