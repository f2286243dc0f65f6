// Tensor-core lane, chunk-parallel part of the backward: one CTA (512 threads) per (chunk, head) turns the
// adjoints published by the reverse scan into dq, dk, dv, dg, dbeta.  K = V = 128, 64 tokens per chunk, bf16
// UMMA operands, fp32 accumulation.  Thread (I, d) owns channel d and the 16 tokens of row block I, so every
// "channel x token" accumulator row (TMEM lane d) is read by the four threads that share that lane.
//
// Products (all on tcgen05; "^T" = channel-major result, M = 128; token x token results use M = 64):
//   dR^T = H dO^T          dW^T = H dZ^T          dE^T = dH' Z^T            (H, dH' V-first panels: MN-major A)
//   dP^T = dZ^T T          dQ^T = -dW^T T                                   (T row-major: MN-major B)
//   dA   = tril(dO Z^T)    Xraw^T = v dZ^T - (e^G k) dW^T    (X = Xraw diag(beta) is the adjoint of T)
//   Y    = T^T X           dM = -stril(Y T^T)
//   pull-back of dA, dM through the decay-masked products, per 16-row target block I with the block's first
//   row as decay reference (both exponential factors stay in range for g in [-5, 0]):
//     RP_I^T = k~_I^T [dA_I ; beta dM_I]^T      CP_I^T = [q~_I ; k-_I]^T [dA_I ; beta dM_I]
// Restates reference chunk_wy_backward.cu:2818-3331 (local VJP), 3337-3552 (pull-back), 3787-3894 (finalize).

#include <cstdio>

#include "common.cuh"
#include "simt_ws.cuh"
#include "tc_common.cuh"
#include "tc_ws.cuh"

namespace kda {
namespace tc {

int make_map_bf16(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);

namespace {

__device__ __forceinline__ uint32_t pk2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
// one MUFU: the operands here are decay factors in [e^-75, 1], far from the flush-to-zero and overflow ends
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float ld16(const uint8_t* base, uint32_t off) {
    return __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(base + off));
}
// element (row r, column d) of a 128-byte-swizzled panel whose 64-column blocks are blk_bytes apart
__device__ __forceinline__ uint32_t eoff(int r, int d, uint32_t blk_bytes) {
    return (uint32_t)(d >> 6) * blk_bytes + sw128_off(r, (d & 63) >> 3) + (uint32_t)(d & 7) * 2;
}
// 32 lanes x 16 consecutive columns, as pairs of adjacent columns (here: adjacent tokens)
__device__ __forceinline__ void tmem_ld_pairs(uint32_t taddr, f2 (&f)[8]) {
    uint32_t r[16];
    tmem_ld16(taddr, r);
    tmem_ld_wait();
#pragma unroll
    for (int j = 0; j < 8; ++j) f[j] = f2_make(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1]));
}
__device__ __forceinline__ f2 rcp_2(f2 a) {
    const float2 x = f2_get(a);
    return f2_make(rcp_approx(x.x), rcp_approx(x.y));
}
__device__ __forceinline__ f2 neg_2(f2 a) { return f2_mul(a, f2_all(-1.f)); }
__device__ __forceinline__ f2 round_bf16_2(f2 a) { return f2_from_bf16(f2_to_bf16(a)); }
__device__ __forceinline__ f2 ld_2(const float* p) {
    const float2 v = *reinterpret_cast<const float2*>(p);
    return f2_make(v.x, v.y);
}
__device__ __forceinline__ uint4 pack_quad(const f2 (&a)[8], int e) {
    return make_uint4(f2_to_bf16(a[e]), f2_to_bf16(a[e + 1]), f2_to_bf16(a[e + 2]), f2_to_bf16(a[e + 3]));
}

}  // namespace

struct IntraBwdArgs {
    const int* chunk_tok0;
    const int* chunk_len;
    const __nv_bfloat16 *q, *k, *v;   // caller tensors [tokens][H][128]
    const void* g;                    // gate dtype
    const float *qinv, *kinv, *beta;  // [nch][64] from the forward
    const __nv_bfloat16* Mt;          // [nch][64][64] M~ (before beta)
    __nv_bfloat16 *dq, *dk, *dv;
    void *dg, *dbeta;                 // gate dtype
    int l2norm, H;
    float scale;
    int* status;
};

// shared-memory map (bytes, 1024-aligned base)
constexpr int kR1 = 0;         // 64 KB  H | dH' panels            -> later: k~_I source panels (4 x 16 KB)
constexpr int kR2 = 65536;     // 16 KB  dO tile                   -> later: X^T tile (8 KB) | Y tile (8 KB)
constexpr int kR3 = 81920;     // 16 KB  Z^T panel                 -> later: target stacks I = 0,1 (2 x 8 KB)
constexpr int kR4 = 98304;     // 16 KB  dZ^T panel                -> later: target stacks I = 2,3
constexpr int kR5 = 114688;    // 48 KB  q | k | v tiles
constexpr int kR6 = 163840;    //  8 KB  T
constexpr int kR7 = 172032;    // 16 KB  dW^T                      -> later: [dA_I ; beta dM_I] tiles (4 x 4 KB)
constexpr int kR8 = 188416;    // 16 KB  Q' = e^G k
constexpr int kRM = 204800;    //  8 KB  M~ (before beta), row-major [target][source]
constexpr int kSmall = 212992; // floats: gsum[4][128] cref[4][128] part[8][128] tot[4][128] dots[64][8] rowv[3][64]
constexpr int kIntraBwdSmem = kSmall + ((4 + 4 + 8 + 4) * 128 + 64 * 8 + 3 * 64) * 4 + 1024;

// Bound by latency: 225 KB of shared memory allow one CTA per SM, and its products depend on one another (state products
// -> X -> Y -> dM -> pull-back).  So (1) only the operand of the next product is read out before that product is issued,
// and everything else - dv, the dR / dE / dQ contributions, the pull-back's decay panels - runs while it is in flight;
// (2) of the six state products the two that the next phase needs are issued first, the others by warps that have finished
// their share of the work beside them; (3) a warp fetches the inputs
// of the CTA that this SM is likely to run next into L2; (4) token pairs go through packed float32 arithmetic.
// 16,384 chunk-heads: 2,262 -> 1,733 us (7 % of it the prefetch), 384: 81 -> 61 us.  A persistent form that loads the next
// chunk-head's panels during the gradient assembly took 1,830: the loads are not what it waits for any more.
template <bool GB>
__global__ void __launch_bounds__(512, 1)
    tc_intra_bwd_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                        const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mdO,
                        const __grid_constant__ CUtensorMap mT, const __grid_constant__ CUtensorMap mH,
                        const __grid_constant__ CUtensorMap mdH, const __grid_constant__ CUtensorMap mZT,
                        const __grid_constant__ CUtensorMap mdZT, const __grid_constant__ CUtensorMap mMt,
                        IntraBwdArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
    uint8_t* Hs = sm + kR1;
    uint8_t* dHs = sm + kR1 + 32768;
    uint8_t* dOs = sm + kR2;
    uint8_t* ZTs = sm + kR3;
    uint8_t* dZTs = sm + kR4;
    uint8_t* qs = sm + kR5;
    uint8_t* ks = qs + 16384;
    uint8_t* vs = ks + 16384;
    uint8_t* Ts = sm + kR6;
    uint8_t* dWs = sm + kR7;
    uint8_t* Qp = sm + kR8;
    uint8_t* Mts = sm + kRM;
    float* gsum = reinterpret_cast<float*>(sm + kSmall);   // [4][128] block sums of g
    float* cref = gsum + 512;                              // [4][128] G at the first row of each block
    float* part = cref + 512;                              // [8][128] partial sums of dD
    float* tot = part + 1024;                              // [4][128] block sums of dG
    float* dots = tot + 512;                               // [2][4][64] row dots: q | k, channel quarter, row
    float* rowv = dots + 512;                              // [3][64]  qinv | kinv | beta
    __shared__ uint64_t bar_in[2], bar_w, bar_p1, bar_x, bar_q, bar_y, bar_m, bar_pb;
    __shared__ uint32_t tmem_slot;
    __shared__ __align__(8) float dA_diag[64];      // dA[i][i]: applied to dq, dk in float32, outside the pull-back products

    const int slot = blockIdx.x, h = blockIdx.y, H = p.H;
    const int len = p.chunk_len[slot], tok0 = p.chunk_tok0[slot];
    if (len == 0) return;
    const int ch = slot * H + h;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int I = warp >> 2;             // row block of this thread
    const int d = tid & 127;             // channel (and TMEM lane) of this thread
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;

    // The first barrier covers what the critical products and the work beside them need.  The loads are issued by warps 1-4,
    // four each, after their gate loads: one thread issuing all of them held the block back.
    if (tid == 0) {
        mbar_init(&bar_in[0], 1);
        mbar_init(&bar_in[1], 1);
        mbar_init(&bar_w, 1);
        mbar_init(&bar_p1, 4);
        mbar_init(&bar_x, 1);
        mbar_init(&bar_q, 1);
        mbar_init(&bar_y, 1);
        mbar_init(&bar_m, 1);
        mbar_init(&bar_pb, 4);
        mbar_expect_tx(&bar_in[0], 32768 + 16384 * 4);
        mbar_expect_tx(&bar_in[1], 32768 + 16384 * 2 + 8192 * 2);
        mbar_fence_init();
    }
    __syncthreads();
    if (warp == 0) tmem_alloc(&tmem_slot, 512);

    // ---- per-row scalars and the cumulative log-decay of this thread's 16 rows
    if (tid < 64) {
        rowv[tid] = p.qinv[ch * 64 + tid];
        rowv[64 + tid] = p.kinv[ch * 64 + tid];
        rowv[128 + tid] = p.beta[ch * 64 + tid];
    }
    const size_t rstride = (size_t)H * 128;
    const size_t col = ((size_t)tok0 * H + h) * 128 + d;
    float G[16];
    {
#pragma unroll
        for (int r = 0; r < 16; ++r) G[r] = ld_io(p.g, col + (size_t)min(16 * I + r, len - 1) * rstride, GB);
        if (lane == 0) {
            if (warp == 1) {
                for (int mb = 0; mb < 2; ++mb) tma_load_2d(Hs + mb * 16384, &mH, &bar_in[0], mb * 64, ch * 128);
                tma_load_2d(dZTs, &mdZT, &bar_in[0], 0, ch * 128);
                tma_load_2d(Ts, &mT, &bar_in[1], 0, ch * 64);
            } else if (warp == 2) {
                for (int mb = 0; mb < 2; ++mb) {
                    tma_load_2d(vs + mb * 8192, &mv, &bar_in[0], h * 128 + mb * 64, tok0);
                    tma_load_2d(dOs + mb * 8192, &mdO, &bar_in[1], h * 128 + mb * 64, tok0);
                }
            } else if (warp == 3) {
                for (int mb = 0; mb < 2; ++mb) tma_load_2d(ks + mb * 8192, &mk, &bar_in[0], h * 128 + mb * 64, tok0);
                for (int mb = 0; mb < 2; ++mb) tma_load_2d(dHs + mb * 16384, &mdH, &bar_in[1], mb * 64, ch * 128);
            } else if (warp == 4) {
                for (int mb = 0; mb < 2; ++mb) tma_load_2d(qs + mb * 8192, &mq, &bar_in[0], h * 128 + mb * 64, tok0);
                tma_load_2d(ZTs, &mZT, &bar_in[1], 0, ch * 128);
                tma_load_2d(Mts, &mMt, &bar_in[1], 0, ch * 64);
            }
        }
        __syncwarp();
        float run = 0.f;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            run += (16 * I + r < len) ? G[r] : 0.f;
            G[r] = run;
        }
        gsum[I * 128 + d] = run;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    // Only decay factors relative to this thread's own block reference cI = G[first row of the block] are needed:
    // E[r] = e^{G[r] - cI} (in (0, 1], at least e^-75), its reciprocal, and the two per-thread scalars that move the
    // reference to the chunk start (e^{cI}) and to the chunk end (e^{gend - cI}).  One exponential per row instead of
    // eight, and the operand panels and the gradient assembly use bit-identical factors by construction.
    float egend, eEndI;
    f2 eCI, E[8];
    {
        const float s0 = gsum[d], s1 = gsum[128 + d], s2 = gsum[256 + d], s3 = gsum[384 + d];
        const float pre = I == 0 ? 0.f : (I == 1 ? s0 : (I == 2 ? s0 + s1 : s0 + s1 + s2));
        const float gend = s0 + s1 + s2 + s3;
#pragma unroll
        for (int r = 0; r < 16; ++r) G[r] += pre;
        const float cI = G[0];
        cref[I * 128 + d] = cI;
        egend = __expf(gend);
        eEndI = __expf(gend - cI);
        eCI = f2_all(__expf(cI));
#pragma unroll
        for (int e = 0; e < 8; ++e) E[e] = f2_make(__expf(G[2 * e] - cI), __expf(G[2 * e + 1] - cI));
    }

    // TMEM columns
    constexpr uint32_t cR = 0, cW = 64, cA = 128, cP = 192, cX = 256, cE = 384, cQ = 448, cY = cP, cM = cW;

    bool ok = true;
    if (len < 64) {
        // rows past a ragged tail hold the next sequence's tokens: blank them in the dO and v tiles, which feed UMMAs
        // as they are (0 x Inf would otherwise reach this sequence's gradients)
        ok = mbar_wait(&bar_in[0], 0, p.status, 40) && mbar_wait(&bar_in[1], 0, p.status, 40);
        if (ok) {
            for (int idx = tid; idx < (64 - len) * 16; idx += 512) {
                const int r = len + (idx >> 4), c = idx & 15;
                const uint32_t off = (uint32_t)(c >> 3) * 8192 + sw128_off(r, c & 7);
                *reinterpret_cast<uint4*>(dOs + off) = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4*>(vs + off) = make_uint4(0, 0, 0, 0);
            }
        }
        fence_async_smem();
        ok = __syncthreads_and(ok);
    }

    // ================================================================ phase 1: state products
    // dW and the first half of X are what the next product waits for: they go first.  The others follow from warps that
    // have finished their share of the work beside them (a thread that issues into a full queue is held until it drains).
    ok = ok && mbar_wait(&bar_in[0], 0, p.status, 40);
    if (ok && tid == 0) {
        tc_fence_after();
        const uint32_t id_mn_mn = umma_idesc_bf16(128, 64, kMajorMN, kMajorMN);
        const uint32_t id64_k_mn = umma_idesc_bf16(64, 64, kMajorK, kMajorMN);
        const uint32_t aH = smem_u32(Hs), bdZ = smem_u32(dZTs), aV = smem_u32(vs);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dW^T = H dZ^T
            umma_bf16_ss(tmem + cW, umma_smem_desc_sw128(aH + k16 * 2048, 16384, 1024),
                         umma_smem_desc_sw128(bdZ + k16 * 2048, 8192, 1024), id_mn_mn, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // Xraw^T = v dZ^T  (first half)    (M = 64)
            umma_bf16_ss(tmem + cX, umma_smem_desc_sw128(aV + (k16 >> 2) * 8192 + (k16 & 3) * 32, 16, 1024),
                         umma_smem_desc_sw128(bdZ + k16 * 2048, 8192, 1024), id64_k_mn, k16 > 0);
        umma_commit(&bar_w);
    }
    __syncwarp();
    // while the tensor core works: this thread's q and k, the Q' operand, and dD[d] = sum_v dH'[d][v] H[d][v]
    uint32_t qw[8], kw[8];
    // unit k and scaled unit q of this thread's rows from their bf16 words
    auto unit_k = [&](f2 (&x)[8], const uint32_t (&w)[8]) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = f2_mul(f2_from_bf16(w[e]), ld_2(rowv + 64 + 16 * I + 2 * e));
    };
    auto unit_q = [&](f2 (&x)[8], const uint32_t (&w)[8]) {
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = f2_mul(f2_from_bf16(w[e]), f2_mul(ld_2(rowv + 16 * I + 2 * e), f2_all(p.scale)));
    };
    {
        const int nv = ok ? len - 16 * I : 0;            // this thread's rows inside the chunk
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int i = 16 * I + 2 * e;
            uint32_t q0 = 0, q1 = 0, k0 = 0, k1 = 0;
            if (2 * e < nv) {
                q0 = *reinterpret_cast<const uint16_t*>(qs + eoff(i, d, 8192));
                k0 = *reinterpret_cast<const uint16_t*>(ks + eoff(i, d, 8192));
            }
            if (2 * e + 1 < nv) {
                q1 = *reinterpret_cast<const uint16_t*>(qs + eoff(i + 1, d, 8192));
                k1 = *reinterpret_cast<const uint16_t*>(ks + eoff(i + 1, d, 8192));
            }
            qw[e] = q0 | (q1 << 16);
            kw[e] = k0 | (k1 << 16);
        }
        // Q' = e^G k for Xraw^T -= Q' dW^T, stored [key d][token] (MN-major A): this thread's 16 tokens are 32
        // contiguous bytes of row d
        f2 w[8];
        unit_k(w, kw);
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = f2_mul(f2_mul(E[e], eCI), w[e]);
        *reinterpret_cast<uint4*>(Qp + sw128_off(d, 2 * I)) = pack_quad(w, 0);
        *reinterpret_cast<uint4*>(Qp + sw128_off(d, 2 * I + 1)) = pack_quad(w, 4);
        ok = ok && mbar_wait(&bar_in[1], 0, p.status, 40);
        // two adjacent channels and 16 value rows a thread
        f2 acc = f2_all(0.f);
        const int d2 = 2 * (tid & 63), vg = tid >> 6;
        if (ok) {
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const uint32_t off = eoff(16 * vg + r, d2, 16384);
                acc = f2_fma(f2_from_bf16(*reinterpret_cast<const uint32_t*>(Hs + off)),
                             f2_from_bf16(*reinterpret_cast<const uint32_t*>(dHs + off)), acc);
            }
        }
        *reinterpret_cast<float2*>(part + vg * 128 + d2) = f2_get(acc);
    }
    if (ok && (warp & 3) == 3 && lane == 0) {
        tc_fence_after();
        const uint32_t aH = smem_u32(Hs), adH = smem_u32(dHs), bdO = smem_u32(dOs), bZ = smem_u32(ZTs), bdZ = smem_u32(dZTs), bT = smem_u32(Ts);
        if (warp == 3) {
            const uint32_t id_k_mn = umma_idesc_bf16(128, 64, kMajorK, kMajorMN);
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)     // dP^T = dZ^T T
                umma_bf16_ss(tmem + cP, umma_smem_desc_sw128(bdZ + k16 * 32, 16, 1024),
                             umma_smem_desc_sw128(bT + k16 * 2048, 8192, 1024), id_k_mn, k16 > 0);
        } else if (warp == 7) {
            const uint32_t id_mn_k = umma_idesc_bf16(128, 64, kMajorMN, kMajorK);
#pragma unroll
            for (int k16 = 0; k16 < 8; ++k16)     // dR^T = H dO^T
                umma_bf16_ss(tmem + cR, umma_smem_desc_sw128(aH + k16 * 2048, 16384, 1024),
                             umma_smem_desc_sw128(bdO + (k16 >> 2) * 8192 + (k16 & 3) * 32, 16, 1024), id_mn_k, k16 > 0);
        } else if (warp == 11) {
            const uint32_t id64_k_mn = umma_idesc_bf16(64, 64, kMajorK, kMajorMN);
#pragma unroll
            for (int k16 = 0; k16 < 8; ++k16)     // dA = dO Z^T                      (M = 64)
                umma_bf16_ss(tmem + cA, umma_smem_desc_sw128(bdO + (k16 >> 2) * 8192 + (k16 & 3) * 32, 16, 1024),
                             umma_smem_desc_sw128(bZ + k16 * 2048, 8192, 1024), id64_k_mn, k16 > 0);
        } else {
            const uint32_t id_mn_mn = umma_idesc_bf16(128, 64, kMajorMN, kMajorMN);
#pragma unroll
            for (int k16 = 0; k16 < 8; ++k16)     // dE^T = dH' Z^T
                umma_bf16_ss(tmem + cE, umma_smem_desc_sw128(adH + k16 * 2048, 16384, 1024),
                             umma_smem_desc_sw128(bZ + k16 * 2048, 8192, 1024), id_mn_mn, k16 > 0);
        }
        umma_commit(&bar_p1);
    }
    __syncwarp();
    ok = ok && mbar_wait(&bar_w, 0, p.status, 41);
    tc_fence_after();

    // ================================================================ phase 2: X and dQ
    {
        f2 t[8];      // dW^T -> bf16 operand (row = channel d, 16 of its 64 tokens)
        tmem_ld_pairs(tmem + lane_base + cW + 16 * I, t);
        *reinterpret_cast<uint4*>(dWs + sw128_off(d, 2 * I)) = pack_quad(t, 0);
        *reinterpret_cast<uint4*>(dWs + sw128_off(d, 2 * I + 1)) = pack_quad(t, 4);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (ok && tid == 0) {
        tc_fence_after();
        const uint32_t id64_neg = umma_idesc_bf16(64, 64, kMajorMN, kMajorMN, 1);
        const uint32_t id_k_mn = umma_idesc_bf16(128, 64, kMajorK, kMajorMN);
        const uint32_t aQ = smem_u32(Qp), aW = smem_u32(dWs), bT = smem_u32(Ts);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // Xraw^T -= Q' dW^T   (dW^T panel read as MN-major B: [key][token])
            umma_bf16_ss(tmem + cX, umma_smem_desc_sw128(aQ + k16 * 2048, 8192, 1024),
                         umma_smem_desc_sw128(aW + k16 * 2048, 8192, 1024), id64_neg, 1);
        umma_commit(&bar_x);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // (T^T dW)^T = dW^T T ;  dQ = -that
            umma_bf16_ss(tmem + cQ, umma_smem_desc_sw128(aW + k16 * 32, 16, 1024),
                         umma_smem_desc_sw128(bT + k16 * 2048, 8192, 1024), id_k_mn, k16 > 0);
        umma_commit(&bar_q);
    }
    __syncwarp();
    // The q and k tiles have been read by everyone: they become thread-private slots for these words.  At 128 registers a
    // thread q, k, the decay factors and three gradients do not fit together, and beside 225 KB of shared memory too little
    // L1 is left to spill into (it went to L2).
    uint4* qslot = reinterpret_cast<uint4*>(qs) + tid;
    uint4* kslot = reinterpret_cast<uint4*>(ks) + tid;
    qslot[0] = make_uint4(qw[0], qw[1], qw[2], qw[3]);
    qslot[512] = make_uint4(qw[4], qw[5], qw[6], qw[7]);
    kslot[0] = make_uint4(kw[0], kw[1], kw[2], kw[3]);
    kslot[512] = make_uint4(kw[4], kw[5], kw[6], kw[7]);
    auto get_q = [&](f2 (&x)[8]) {
        const uint4 a = qslot[0], b = qslot[512];
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        unit_q(x, w);
    };
    auto get_k = [&](f2 (&x)[8]) {
        const uint4 a = kslot[0], b = kslot[512];
        const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
        unit_k(x, w);
    };
    ok = ok && mbar_wait(&bar_p1, 0, p.status, 41);
    tc_fence_after();
    f2 dqn[8], dG[8];
    {
        f2 t[8];
        // in flight: dv = beta dP, staged [token][channel] in the value tile (only the completed products read it) so that
        // it leaves as 16-byte row segments, and the dR part of dq
        tmem_ld_pairs(tmem + lane_base + cP + 16 * I, t);
        __nv_bfloat16* tv = reinterpret_cast<__nv_bfloat16*>(vs) + 16 * I * 128 + d;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const uint32_t u = f2_to_bf16(f2_mul(ld_2(rowv + 128 + 16 * I + 2 * e), t[e]));
            const __nv_bfloat162 b2 = *reinterpret_cast<const __nv_bfloat162*>(&u);
            tv[2 * e * 128] = b2.x;
            tv[(2 * e + 1) * 128] = b2.y;
        }
        tmem_ld_pairs(tmem + lane_base + cR + 16 * I, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            dqn[e] = f2_mul(t[e], f2_mul(E[e], eCI));
        }
        unit_q(t, qw);
#pragma unroll
        for (int e = 0; e < 8; ++e) dG[e] = f2_mul(dqn[e], t[e]);
    }
    ok = ok && mbar_wait(&bar_x, 0, p.status, 42);
    tc_fence_after();

    // ================================================================ phase 3: Y, dM
    // M = 64 accumulators keep row (16*w + l) in lane l < 16 of warp w < 4.  tcgen05.ld is warp-collective, so all 32
    // lanes of those warps run the loads; lanes >= 16 mirror a row and never store.  All four warp groups see the same lanes, so each takes 16 of the 64 columns.
    const bool rowown = lane < 16;
    const int row = 16 * (warp & 3) + (lane & 15);
    uint8_t* XT = sm + kR2;           // [64 rows s][64 i]   K-major B
    uint8_t* Yt = sm + kR2 + 8192;    // [64 rows j][64 s]   K-major A
    float dbeta_acc = 0.f;
    float* dbp = reinterpret_cast<float*>(Qp);      // [4][64] partial dbeta per column group (Q' has been read once X is complete)
    {
        const f2 bs = f2_all(rowv[128 + row]);
        f2 t[8], acc = f2_all(0.f);
        tmem_ld_pairs(tmem + lane_base + cX + 16 * I, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int i = 16 * I + 2 * e;
            acc = f2_fma(f2_make(ld16(Ts, sw128_off(i, row >> 3) + (row & 7) * 2), ld16(Ts, sw128_off(i + 1, row >> 3) + (row & 7) * 2)),
                         t[e], acc);                                                   // T[i][s] * Xraw[i][s]
            t[e] = f2_mul(bs, t[e]);
        }
        const float2 a = f2_get(acc);
        dbeta_acc = a.x + a.y;
        if (rowown) {
            *reinterpret_cast<uint4*>(XT + sw128_off(row, 2 * I)) = pack_quad(t, 0);
            *reinterpret_cast<uint4*>(XT + sw128_off(row, 2 * I + 1)) = pack_quad(t, 4);
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (ok && tid == 0) {
        tc_fence_after();
        const uint32_t id = umma_idesc_bf16(64, 64, kMajorMN, kMajorK);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // Y = T^T X : A[m=j][k=i] = T[i][j] (MN-major), B[n=s][k=i] = X^T rows
            umma_bf16_ss(tmem + cY, umma_smem_desc_sw128(smem_u32(Ts) + k16 * 2048, 8192, 1024),
                         umma_smem_desc_sw128(smem_u32(XT) + k16 * 32, 16, 1024), id, k16 > 0);
        umma_commit(&bar_y);
    }
    __syncwarp();
    if (ok) {      // in flight: the dv rows leave
        const __nv_bfloat16* tv = reinterpret_cast<const __nv_bfloat16*>(vs);
        const int c = tid & 15;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const int i = pass * 32 + (tid >> 4);
            if (i < len)
                *reinterpret_cast<uint4*>(p.dv + ((size_t)(tok0 + i) * H + h) * 128 + 8 * c) =
                    *reinterpret_cast<const uint4*>(tv + i * 128 + 8 * c);
        }
    }
    ok = ok && mbar_wait(&bar_y, 0, p.status, 43);
    tc_fence_after();
    {
        f2 t[8];
        tmem_ld_pairs(tmem + lane_base + cY + 16 * I, t);
        if (rowown) {
            *reinterpret_cast<uint4*>(Yt + sw128_off(row, 2 * I)) = pack_quad(t, 0);
            *reinterpret_cast<uint4*>(Yt + sw128_off(row, 2 * I + 1)) = pack_quad(t, 4);
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (ok && tid == 0) {
        tc_fence_after();
        const uint32_t id = umma_idesc_bf16(64, 64, kMajorK, kMajorK);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // Y T^T : B[n=l][k=s] = T[l][s]
            umma_bf16_ss(tmem + cM, umma_smem_desc_sw128(smem_u32(Yt) + k16 * 32, 16, 1024),
                         umma_smem_desc_sw128(smem_u32(Ts) + k16 * 32, 16, 1024), id, k16 > 0);
        umma_commit(&bar_m);
    }
    __syncwarp();

    // ================================================================ phase 4: pull-back operands
    uint8_t* Sk = sm + kR1;           // k~_I source panels: [I][128 rows d][64 s], rows of blocks <= I only  K-major A
    uint8_t* Xk = sm + kR3;           // target stacks: [I / 2][128 rows d][32 rows of I even | 32 of I odd] K-major A
    uint8_t* DAt = sm + kR7;          // [I][32 rows: 16 dA rows, 16 beta*dM rows][64 s]   K-major / MN-major B
    const int jb = row >> 4, jr = row & 15;
    {
        // in flight: the decay panels.  Both operand families are stored transposed, [channel d][row], so that this
        // thread's 16 rows are contiguous bytes of row d and leave as 16-byte stores (K-major A operands).
        uint8_t* X = Xk + (I >> 1) * 16384;      // two target blocks share a panel: 32 stack rows each
        const int xc = (I & 1) * 4;
        f2 w[8], x[8];
        get_q(w);
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = f2_mul(w[e], E[e]);       // q~ rows of this block
        *reinterpret_cast<uint4*>(X + sw128_off(d, xc)) = pack_quad(w, 0);
        *reinterpret_cast<uint4*>(X + sw128_off(d, xc + 1)) = pack_quad(w, 4);
        get_k(x);
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = f2_mul(x[e], E[e]);       // k~ rows of this block
        *reinterpret_cast<uint4*>(X + sw128_off(d, xc + 2)) = pack_quad(w, 0);
        *reinterpret_cast<uint4*>(X + sw128_off(d, xc + 3)) = pack_quad(w, 4);
        // these rows as sources of their own and every later block (block I's product sums over the blocks <= I only)
        f2 ei[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) ei[e] = rcp_2(E[e]);
#pragma unroll 1
        for (int ver = I; ver < 4; ++ver) {
            if (ver > I) {
                const f2 fb = f2_all(__expf(cref[ver * 128 + d] - cref[(ver - 1) * 128 + d]));
#pragma unroll
                for (int e = 0; e < 8; ++e) ei[e] = f2_mul(ei[e], fb);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = f2_mul(x[e], ei[e]);
            *reinterpret_cast<uint4*>(Sk + ver * 16384 + sw128_off(d, 2 * I)) = pack_quad(w, 0);
            *reinterpret_cast<uint4*>(Sk + ver * 16384 + sw128_off(d, 2 * I + 1)) = pack_quad(w, 4);
        }
    }
    ok = ok && mbar_wait(&bar_q, 0, p.status, 42);       // the dW^T panel is free from here: it becomes the DAt tiles
    tc_fence_after();
    {   // still in flight: the rows of dA
        f2 t[8];
        // row j of dA = tril(dO Z^T), 16 source columns per warp group.  The diagonal of dA adds q k dA to dG through the
        // row part and takes the same amount away through the column part; left inside two bf16 products those O(1) terms
        // cancel only to bf16 accuracy, which swamps dg when the decay is strong.  It goes to dq and dk directly instead
        // (decay factor 1, no dG term).
        tmem_ld_pairs(tmem + lane_base + cA + 16 * I, t);
        const int nd = row - 16 * I;                     // columns before the diagonal, relative to this group's first
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float2 a = f2_get(t[e]);
            if (rowown && 2 * e == nd) dA_diag[row] = a.x;
            if (rowown && 2 * e + 1 == nd) dA_diag[row] = a.y;
            t[e] = f2_make(2 * e < nd ? a.x : 0.f, 2 * e + 1 < nd ? a.y : 0.f);
        }
        if (rowown) {
            *reinterpret_cast<uint4*>(DAt + jb * 4096 + sw128_off(jr, 2 * I)) = pack_quad(t, 0);
            *reinterpret_cast<uint4*>(DAt + jb * 4096 + sw128_off(jr, 2 * I + 1)) = pack_quad(t, 4);
        }
    }
    ok = ok && mbar_wait(&bar_m, 0, p.status, 44);
    tc_fence_after();
    {
        // row j of dM = -stril(Y T^T); dbeta gets sum_l dM[j][l] M~[j][l]
        const int nd = row - 16 * I;
        f2 t[8], acc = f2_all(0.f);
        tmem_ld_pairs(tmem + lane_base + cM + 16 * I, t);
        const uint4 m0 = *reinterpret_cast<const uint4*>(Mts + sw128_off(row, 2 * I));
        const uint4 m1 = *reinterpret_cast<const uint4*>(Mts + sw128_off(row, 2 * I + 1));
        const uint32_t mw[8] = {m0.x, m0.y, m0.z, m0.w, m1.x, m1.y, m1.z, m1.w};
        const f2 bj = f2_all(rowv[128 + row]);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float2 a = f2_get(t[e]);
            const f2 dm = f2_make(2 * e < nd ? -a.x : 0.f, 2 * e + 1 < nd ? -a.y : 0.f);
            acc = f2_fma(dm, f2_from_bf16(mw[e]), acc);
            t[e] = f2_mul(bj, dm);
        }
        const float2 a = f2_get(acc);
        dbeta_acc += a.x + a.y;
        if (rowown) {
            *reinterpret_cast<uint4*>(DAt + jb * 4096 + sw128_off(16 + jr, 2 * I)) = pack_quad(t, 0);
            *reinterpret_cast<uint4*>(DAt + jb * 4096 + sw128_off(16 + jr, 2 * I + 1)) = pack_quad(t, 4);
            dbp[I * 64 + row] = dbeta_acc;
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    // accumulator columns of the pull-back: RP_I (32 columns each) and CP_I (64 columns each)
    constexpr uint32_t cRP = 0, cCP = 128;
    if (ok && warp < 4 && lane == 0) {     // warp = target block
        tc_fence_after();
        const uint32_t id_rp = umma_idesc_bf16(128, 32, kMajorK, kMajorK);
        const uint32_t id_cp = umma_idesc_bf16(128, 64, kMajorK, kMajorMN);
        const uint32_t aS = smem_u32(Sk + warp * 16384), aX = smem_u32(Xk + (warp >> 1) * 16384) + (warp & 1) * 64;
        const uint32_t bD = smem_u32(DAt + warp * 4096);
#pragma unroll 1
        for (int k16 = 0; k16 <= warp; ++k16)     // RP_I^T[d][n] = sum_{s in blocks <= I} k~_I[s][d] * rows_I[n][s]
            umma_bf16_ss(tmem + cRP + 32 * warp, umma_smem_desc_sw128(aS + k16 * 32, 16, 1024),
                         umma_smem_desc_sw128(bD + k16 * 32, 16, 1024), id_rp, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 2; ++k16)     // CP_I^T[d][s] = sum_{n<32} stack_I[n][d] * rows_I[n][s]
            umma_bf16_ss(tmem + cCP + 64 * warp, umma_smem_desc_sw128(aX + k16 * 32, 16, 1024),
                         umma_smem_desc_sw128(bD + k16 * 2048, 4096, 1024), id_cp, k16 > 0);
        umma_commit(&bar_pb);
    }
    __syncwarp();
    if (tid >= 128 && tid < 192 && tid - 128 < len) {
        const int i = tid - 128;
        st_io(p.dbeta, (size_t)(tok0 + i) * H + h, GB, dbp[i] + dbp[64 + i] + dbp[128 + i] + dbp[192 + i]);
    }
    if (warp == 15) {
        // the inputs of the block that starts when this one ends, 148 further on, into L2
        const unsigned nxt = blockIdx.y * gridDim.x + blockIdx.x + 148u;
        if (nxt < gridDim.x * gridDim.y) {
            const int ns = (int)(nxt % gridDim.x), nh = (int)(nxt / gridDim.x);
            const int nlen = p.chunk_len[ns], nt0 = p.chunk_tok0[ns], nch = ns * H + nh;
            if (nlen > 0) {
                if (lane < 2) {
                    tma_prefetch_2d(&mH, lane * 64, nch * 128);
                    tma_prefetch_2d(&mdH, lane * 64, nch * 128);
                    tma_prefetch_2d(&mdO, nh * 128 + lane * 64, nt0);
                    tma_prefetch_2d(&mq, nh * 128 + lane * 64, nt0);
                    tma_prefetch_2d(&mk, nh * 128 + lane * 64, nt0);
                    tma_prefetch_2d(&mv, nh * 128 + lane * 64, nt0);
                } else if (lane == 2) {
                    tma_prefetch_2d(&mZT, 0, nch * 128);
                    tma_prefetch_2d(&mdZT, 0, nch * 128);
                    tma_prefetch_2d(&mT, 0, nch * 64);
                    tma_prefetch_2d(&mMt, 0, nch * 64);
                }
                for (int i = lane; i < nlen; i += 32) {
                    const char* gp = static_cast<const char*>(p.g) + (((size_t)(nt0 + i) * H + nh) * 128) * (GB ? 2 : 4);
#pragma unroll
                    for (int b = 0; b < (GB ? 256 : 512); b += 128) prefetch_l2(gp + b);
                }
            }
        }
        __syncwarp();
    }
    // in flight: the dE and dQ parts of dk, the diagonal of dA
    f2 dkn[8], kn[8];
    f2 ge2 = f2_all(0.f);
    get_k(kn);
    {
        f2 t[8];
        tmem_ld_pairs(tmem + lane_base + cE + 16 * I, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            dkn[e] = f2_mul(t[e], f2_mul(rcp_2(E[e]), f2_all(eEndI)));
            const f2 eE = f2_mul(dkn[e], kn[e]);    // dE * E
            dG[e] = f2_add(dG[e], neg_2(eE));
            ge2 = f2_add(ge2, eE);
        }
        tmem_ld_pairs(tmem + lane_base + cQ + 16 * I, t);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const f2 dQ = neg_2(f2_mul(f2_mul(t[e], ld_2(rowv + 128 + 16 * I + 2 * e)), f2_mul(E[e], eCI)));   // dQ * beta * e^G
            dkn[e] = f2_add(dkn[e], dQ);
            dG[e] = f2_fma(dQ, kn[e], dG[e]);
        }
        get_q(t);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const f2 dd = ld_2(dA_diag + 16 * I + 2 * e);
            dqn[e] = f2_fma(dd, kn[e], dqn[e]);
            dkn[e] = f2_fma(dd, t[e], dkn[e]);
        }
    }
    ok = ok && mbar_wait(&bar_pb, 0, p.status, 45);
    tc_fence_after();

    // ================================================================ phase 5: assemble the gradients
    {
        f2 t[8];
        // decay factors of this thread's rows relative to its own block reference: E = e^{G - c_own} (<= 1) for the
        // row parts, 1 / E for the column parts (a later block I' contributes e^{c_I' - c_own} / E)
        // The decay gradient is a telescoping sum: a pair (i, s) adds its summand to dG at row i (row part) and takes the
        // same summand away at row s (column part), and only the rows in between keep it after the reverse cumulative
        // sum.  The two parts come from different UMMAs, so they cancel exactly only if both are built from the SAME
        // rounded factors: dG therefore uses the bf16 values that sit in the operand panels (target rows q~, k~ and
        // source rows k-), while dq and dk keep the float32 factors.
        tmem_ld_pairs(tmem + lane_base + cRP + 32 * I + 16, t);     // row part through beta*dM
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            dkn[e] = f2_fma(E[e], t[e], dkn[e]);
            dG[e] = f2_fma(round_bf16_2(f2_mul(kn[e], E[e])), t[e], dG[e]);
        }
        tmem_ld_pairs(tmem + lane_base + cRP + 32 * I, t);          // row part through dA
        {
            const uint4 a = qslot[0], b = qslot[512];
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const f2 q = f2_mul(f2_from_bf16(w[e]), f2_mul(ld_2(rowv + 16 * I + 2 * e), f2_all(p.scale)));
                dqn[e] = f2_fma(E[e], t[e], dqn[e]);
                dG[e] = f2_fma(round_bf16_2(f2_mul(q, E[e])), t[e], dG[e]);
            }
        }
        // column part: sources of block I receive from target blocks I' >= I, each with its own decay reference; the
        // source factor is rebuilt exactly as the panel code built it
#pragma unroll
        for (int e = 0; e < 8; ++e) E[e] = rcp_2(E[e]);
        float cprev = cref[I * 128 + d];
#pragma unroll 1
        for (int Ib = I; Ib < 4; ++Ib) {
            tmem_ld_pairs(tmem + lane_base + cCP + 64 * Ib + 16 * I, t);
            if (Ib > I) {
                const float cn = cref[Ib * 128 + d];
                const f2 fb = f2_all(__expf(cn - cprev));
                cprev = cn;
#pragma unroll
                for (int e = 0; e < 8; ++e) E[e] = f2_mul(E[e], fb);
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                dkn[e] = f2_fma(E[e], t[e], dkn[e]);
                dG[e] = f2_fma(neg_2(round_bf16_2(f2_mul(kn[e], E[e]))), t[e], dG[e]);
            }
        }
    }
    // chunk-end term and reverse cumulative sum of dG over the 64 rows of this channel
    {
        f2 local = dG[0];
#pragma unroll
        for (int e = 1; e < 8; ++e) local = f2_add(local, dG[e]);
        const float2 l2 = f2_get(local), g2 = f2_get(ge2);
        tot[I * 128 + d] = l2.x + l2.y;
        gsum[I * 128 + d] = g2.x + g2.y;   // gsum is free again
    }
    // L2-normalisation VJP needs per-row dots over the channels: unit k is kn, unit q is qn / scale
    const float inv_scale = p.scale != 0.f ? 1.0f / p.scale : 0.f;
    f2 qn[8];
    get_q(qn);
    {
        // 32 per-row products (q and k of 16 rows) summed over the 32 channels of this warp with 31 shuffles: each
        // step halves the values a lane carries, so lane L ends with the warp's total of value L.
        float vals[16];
        {
            const bool up = (lane & 16) != 0;      // first step straight from the operands: value j pairs with value j + 16
#pragma unroll
            for (int e = 0; e < 4; ++e) {          // value 2 * row + {q, k}
                const float2 qa = f2_get(f2_mul(qn[e], dqn[e])), ka = f2_get(f2_mul(kn[e], dkn[e]));
                const float2 qb = f2_get(f2_mul(qn[4 + e], dqn[4 + e])), kb = f2_get(f2_mul(kn[4 + e], dkn[4 + e]));
                vals[4 * e] = (up ? qb.x : qa.x) + __shfl_xor_sync(0xffffffffu, up ? qa.x : qb.x, 16);
                vals[4 * e + 1] = (up ? kb.x : ka.x) + __shfl_xor_sync(0xffffffffu, up ? ka.x : kb.x, 16);
                vals[4 * e + 2] = (up ? qb.y : qa.y) + __shfl_xor_sync(0xffffffffu, up ? qa.y : qb.y, 16);
                vals[4 * e + 3] = (up ? kb.y : ka.y) + __shfl_xor_sync(0xffffffffu, up ? ka.y : kb.y, 16);
            }
        }
#pragma unroll
        for (int o = 8; o >= 1; o >>= 1) {
            const bool up = (lane & o) != 0;
#pragma unroll
            for (int j = 0; j < o; ++j) {
                const float send = up ? vals[j] : vals[j + o];
                const float keep = up ? vals[j + o] : vals[j];
                vals[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
            }
        }
        // lane L holds value L = (row L/2, q or k): quadrant partial
        dots[(lane & 1) * 256 + (warp & 3) * 64 + 16 * I + (lane >> 1)] = vals[0];
    }
    __syncthreads();
    if (p.l2norm) {
        if (tid < 128) {      // the four quadrants of the channels -> one number, in place
            float* q4 = dots + (tid >> 6) * 256 + (tid & 63);
            q4[0] = (q4[0] + q4[64]) + (q4[128] + q4[192]);
        }
        __syncthreads();
    }
    {
        float run = gsum[d] + gsum[128 + d] + gsum[256 + d] + gsum[384 + d];
        {
            float dD = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) dD += part[r * 128 + d];
            run += egend * dD;
        }
#pragma unroll
        for (int Ib = 3; Ib > 0; --Ib)
            if (Ib > I) run += tot[Ib * 128 + d];
        // The gradients of this thread's 16 rows go through shared memory (the source-panel region is free now), so
        // that they leave as 16-byte row segments instead of one 2-byte store per row, tensor and thread.
        __nv_bfloat16* tq = reinterpret_cast<__nv_bfloat16*>(sm + kR1) + 16 * I * 128 + d;      // [64][128] dq
        __nv_bfloat16* tk = tq + 64 * 128;                                                       // [64][128] dk
        __nv_bfloat16* tgb = tk + 64 * 128;                                                      // [64][128] dg when the gate dtype is bf16
        float* tgf = reinterpret_cast<float*>(sm + kR1 + 32768) + 16 * I * 128 + d;              // [64][128] dg when it is float32
#pragma unroll
        for (int e = 7; e >= 0; --e) {
            const int i = 16 * I + 2 * e;
            f2 dqv = f2_mul(dqn[e], f2_all(p.scale)), dkv = dkn[e];
            if (p.l2norm) {
                const f2 pq = ld_2(dots + i), pk = ld_2(dots + 256 + i);
                dqv = f2_mul(ld_2(rowv + i), f2_fma(f2_mul(qn[e], f2_all(-inv_scale)), pq, dqv));
                dkv = f2_mul(ld_2(rowv + 64 + i), f2_fma(neg_2(kn[e]), pk, dkv));
            }
            const uint32_t uq = f2_to_bf16(dqv), uk = f2_to_bf16(dkv);
            const __nv_bfloat162 bq = *reinterpret_cast<const __nv_bfloat162*>(&uq), bk = *reinterpret_cast<const __nv_bfloat162*>(&uk);
            tq[2 * e * 128] = bq.x;
            tq[(2 * e + 1) * 128] = bq.y;
            tk[2 * e * 128] = bk.x;
            tk[(2 * e + 1) * 128] = bk.y;
            const float2 g2 = f2_get(dG[e]);
            const float r1 = run + g2.y, r0 = r1 + g2.x;
            run = r0;
            if (GB) {
                tgb[2 * e * 128] = __float2bfloat16(r0);
                tgb[(2 * e + 1) * 128] = __float2bfloat16(r1);
            } else {
                tgf[2 * e * 128] = r0;
                tgf[(2 * e + 1) * 128] = r1;
            }
        }
    }
    __syncthreads();
    if (ok) {
        const __nv_bfloat16* tq = reinterpret_cast<const __nv_bfloat16*>(sm + kR1);
        const __nv_bfloat16* tk = tq + 64 * 128;
        const __nv_bfloat16* tgb = tk + 64 * 128;
        const float* tgf = reinterpret_cast<const float*>(sm + kR1 + 32768);
        const int c = tid & 15;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const int i = pass * 32 + (tid >> 4);
            if (i < len) {
                const size_t o = ((size_t)(tok0 + i) * H + h) * 128;
                *reinterpret_cast<uint4*>(p.dq + o + 8 * c) = *reinterpret_cast<const uint4*>(tq + i * 128 + 8 * c);
                *reinterpret_cast<uint4*>(p.dk + o + 8 * c) = *reinterpret_cast<const uint4*>(tk + i * 128 + 8 * c);
                if (GB) {
                    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dg) + o + 8 * c) =
                        *reinterpret_cast<const uint4*>(tgb + i * 128 + 8 * c);
                } else {
                    float* dgp = reinterpret_cast<float*>(p.dg) + o;
                    *reinterpret_cast<uint4*>(dgp + 4 * c) = *reinterpret_cast<const uint4*>(tgf + i * 128 + 4 * c);
                    *reinterpret_cast<uint4*>(dgp + 64 + 4 * c) = *reinterpret_cast<const uint4*>(tgf + i * 128 + 64 + 4 * c);
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

}  // namespace tc

int tc_intra_backward(const simt::Ws& w, const tc::TcWs& t, int tokens, const void* q, const void* k, const void* v,
                      const void* g, const void* d_o, int gbf16, int l2norm, float scale, void* dq, void* dk, void* dv,
                      void* dg, void* dbeta, cudaStream_t st) {
    using namespace tc;
    const uint64_t nch = (uint64_t)w.nslots * w.H;
    const uint64_t cols = (uint64_t)w.H * 128;
    CUtensorMap mq, mk, mv, mdO, mT, mH, mdH, mZT, mdZT, mMt;
    int rc = 0;
    rc |= make_map_bf16(&mq, q, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mk, k, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mv, v, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mdO, d_o, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mT, t.Tp, nch * 64, 64, 64, 64);
    rc |= make_map_bf16(&mH, t.Hp, nch * 128, 128, 64, 128);
    rc |= make_map_bf16(&mdH, t.dHp, nch * 128, 128, 64, 128);
    rc |= make_map_bf16(&mZT, t.ZT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mdZT, t.dZT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mMt, t.Mt, nch * 64, 64, 64, 64);
    if (rc) return KDA_ERR_CUDA;
    IntraBwdArgs a;
    a.chunk_tok0 = w.chunk_tok0; a.chunk_len = w.chunk_len;
    a.q = static_cast<const __nv_bfloat16*>(q); a.k = static_cast<const __nv_bfloat16*>(k);
    a.v = static_cast<const __nv_bfloat16*>(v); a.g = g;
    a.qinv = w.qinv; a.kinv = w.kinv; a.beta = w.beta; a.Mt = t.Mt;
    a.dq = static_cast<__nv_bfloat16*>(dq); a.dk = static_cast<__nv_bfloat16*>(dk); a.dv = static_cast<__nv_bfloat16*>(dv);
    a.dg = dg; a.dbeta = dbeta; a.l2norm = l2norm; a.H = w.H; a.scale = scale; a.status = t.status;
    auto kern = gbf16 ? tc_intra_bwd_kernel<true> : tc_intra_bwd_kernel<false>;
    if (set_smem_limit(kern, kIntraBwdSmem)) return KDA_ERR_CUDA;
    KDA_LAUNCH("tc_intra_bwd_kernel", st,
               kern<<<dim3(w.nslots, w.H), 512, kIntraBwdSmem, st>>>(mq, mk, mv, mdO, mT, mH, mdH, mZT, mdZT, mMt, a));
    return launch_status();
}

}  // namespace kda
