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
// 32 lanes x 16 consecutive columns
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&f)[16]) {
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; ++j) f[j] = __uint_as_float(r[j]);
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
    int gbf16, l2norm, H;
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
constexpr int kSmall = 212992; // floats: gsum[4][128] cref[4][128] part[4][128] tot[4][128] dots[64][8] rowv[3][64]
constexpr int kIntraBwdSmem = kSmall + (4 * 4 * 128 + 64 * 8 + 3 * 64) * 4 + 1024;

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
    float* part = cref + 512;                              // [4][128] scratch partials
    float* tot = part + 512;                               // [4][128] scratch partials
    float* dots = tot + 512;                               // [64][8]  row dots: [row][quarter*2 + {q,k}]
    float* rowv = dots + 512;                              // [3][64]  qinv | kinv | beta
    __shared__ uint64_t bar_in, bar_mma;
    __shared__ uint32_t tmem_slot;
    __shared__ float dA_diag[64];      // dA[i][i]: applied to dq, dk in float32, outside the pull-back products

    const int slot = blockIdx.x, h = blockIdx.y, H = p.H;
    const int len = p.chunk_len[slot];
    if (len == 0) return;
    const int tok0 = p.chunk_tok0[slot];
    const int ch = slot * H + h;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int I = warp >> 2;             // row block of this thread
    const int d = tid & 127;             // channel (and TMEM lane) of this thread
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;

    if (tid == 0) {
        mbar_init(&bar_in, 1);
        mbar_init(&bar_mma, 1);
        mbar_fence_init();
        mbar_expect_tx(&bar_in, 65536 + 16384 * 3 + 49152 + 8192 + 8192);
        for (int mb = 0; mb < 2; ++mb) {
            tma_load_2d(Hs + mb * 16384, &mH, &bar_in, mb * 64, ch * 128);
            tma_load_2d(dHs + mb * 16384, &mdH, &bar_in, mb * 64, ch * 128);
            tma_load_2d(dOs + mb * 8192, &mdO, &bar_in, h * 128 + mb * 64, tok0);
            tma_load_2d(qs + mb * 8192, &mq, &bar_in, h * 128 + mb * 64, tok0);
            tma_load_2d(ks + mb * 8192, &mk, &bar_in, h * 128 + mb * 64, tok0);
            tma_load_2d(vs + mb * 8192, &mv, &bar_in, h * 128 + mb * 64, tok0);
        }
        tma_load_2d(ZTs, &mZT, &bar_in, 0, ch * 128);
        tma_load_2d(dZTs, &mdZT, &bar_in, 0, ch * 128);
        tma_load_2d(Ts, &mT, &bar_in, 0, ch * 64);
        tma_load_2d(Mts, &mMt, &bar_in, 0, ch * 64);
    }
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
        for (int r = 0; r < 16; ++r) G[r] = ld_io(p.g, col + (size_t)min(16 * I + r, len - 1) * rstride, p.gbf16);
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
    float gend;
    {
        const float s0 = gsum[d], s1 = gsum[128 + d], s2 = gsum[256 + d], s3 = gsum[384 + d];
        const float pre = I == 0 ? 0.f : (I == 1 ? s0 : (I == 2 ? s0 + s1 : s0 + s1 + s2));
        gend = s0 + s1 + s2 + s3;
#pragma unroll
        for (int r = 0; r < 16; ++r) G[r] += pre;
        cref[I * 128 + d] = G[0];
    }
    bool ok = mbar_wait(&bar_in, 0, p.status, 40);
    if (len < 64 && ok) {
        // rows past a ragged tail hold the next sequence's tokens: blank them in the dO and v tiles, which feed UMMAs
        // as they are (0 x Inf would otherwise reach this sequence's gradients)
        for (int idx = tid; idx < (64 - len) * 16; idx += 512) {
            const int r = len + (idx >> 4), c = idx & 15;
            const uint32_t off = (uint32_t)(c >> 3) * 8192 + sw128_off(r, c & 7);
            *reinterpret_cast<uint4*>(dOs + off) = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(vs + off) = make_uint4(0, 0, 0, 0);
        }
        fence_async_smem();
    }
    ok = __syncthreads_and(ok);          // also publishes cref
    const float egend = __expf(gend);
    // From here on only decay factors relative to this thread's own block reference cI = G[first row of the block] are
    // needed: E[r] = e^{G[r] - cI} (in (0, 1], at least e^-75), its reciprocal, and the two per-thread scalars that move
    // the reference to the chunk start (e^{cI}) and to the chunk end (e^{gend - cI}).  One exponential per row instead
    // of eight, and the operand panels and the gradient assembly use bit-identical factors by construction.
    const float cI = G[0];
    const float eCI = __expf(cI), eEndI = __expf(gend - cI);
#pragma unroll
    for (int r = 0; r < 16; ++r) G[r] = __expf(G[r] - cI);
    float (&E)[16] = G;

    // TMEM columns
    constexpr uint32_t cDa = 0, cDb = 64, cDc = 128, cDd = 192, cDg = 256, cDf = 320, cDe = 384;

    // ================================================================ phase 1: state products
    if (ok && tid == 0) {
        tc_fence_after();
        const uint32_t id_mn_k = umma_idesc_bf16(128, 64, kMajorMN, kMajorK);
        const uint32_t id_mn_mn = umma_idesc_bf16(128, 64, kMajorMN, kMajorMN);
        const uint32_t id_k_mn = umma_idesc_bf16(128, 64, kMajorK, kMajorMN);
        const uint32_t id64_k_mn = umma_idesc_bf16(64, 64, kMajorK, kMajorMN);
        const uint32_t aH = smem_u32(Hs), adH = smem_u32(dHs), bdO = smem_u32(dOs), bZ = smem_u32(ZTs), bdZ = smem_u32(dZTs);
        const uint32_t aV = smem_u32(vs), bT = smem_u32(Ts);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dR^T = H dO^T
            umma_bf16_ss(tmem + cDa, umma_smem_desc_sw128(aH + k16 * 2048, 16384, 1024),
                         umma_smem_desc_sw128(bdO + (k16 >> 2) * 8192 + (k16 & 3) * 32, 16, 1024), id_mn_k, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dW^T = H dZ^T
            umma_bf16_ss(tmem + cDb, umma_smem_desc_sw128(aH + k16 * 2048, 16384, 1024),
                         umma_smem_desc_sw128(bdZ + k16 * 2048, 8192, 1024), id_mn_mn, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dE^T = dH' Z^T
            umma_bf16_ss(tmem + cDc, umma_smem_desc_sw128(adH + k16 * 2048, 16384, 1024),
                         umma_smem_desc_sw128(bZ + k16 * 2048, 8192, 1024), id_mn_mn, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // dP^T = dZ^T T
            umma_bf16_ss(tmem + cDd, umma_smem_desc_sw128(bdZ + k16 * 32, 16, 1024),
                         umma_smem_desc_sw128(bT + k16 * 2048, 8192, 1024), id_k_mn, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dA = dO Z^T                      (M = 64)
            umma_bf16_ss(tmem + cDg, umma_smem_desc_sw128(bdO + (k16 >> 2) * 8192 + (k16 & 3) * 32, 16, 1024),
                         umma_smem_desc_sw128(bZ + k16 * 2048, 8192, 1024), id64_k_mn, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // Xraw^T = v dZ^T  (first half)    (M = 64)
            umma_bf16_ss(tmem + cDf, umma_smem_desc_sw128(aV + (k16 >> 2) * 8192 + (k16 & 3) * 32, 16, 1024),
                         umma_smem_desc_sw128(bdZ + k16 * 2048, 8192, 1024), id64_k_mn, k16 > 0);
        umma_commit(&bar_mma);
    }
    // while the tensor core works: dD[d] = sum_v dH'[d][v] H[d][v] over this thread's 32 value rows
    float kn[16], qn[16];
    {
        float acc = 0.f;
        if (ok) {
#pragma unroll 8
            for (int vv = 32 * I; vv < 32 * I + 32; ++vv) acc += ld16(Hs, eoff(vv, d, 16384)) * ld16(dHs, eoff(vv, d, 16384));
        }
        part[I * 128 + d] = acc;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int i = 16 * I + r;
            float qv = 0.f, kv = 0.f;
            if (ok && i < len) {
                qv = ld16(qs, eoff(i, d, 8192));
                kv = ld16(ks, eoff(i, d, 8192));
            }
            qn[r] = qv * rowv[i] * p.scale;
            kn[r] = kv * rowv[64 + i];
        }
        // Q' = e^G k for Xraw^T -= Q' dW^T, stored [key d][token] (MN-major A): this thread's 16 tokens are 32
        // contiguous bytes of row d
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = pk2(E[2 * e] * eCI * kn[2 * e], E[2 * e + 1] * eCI * kn[2 * e + 1]);
        *reinterpret_cast<uint4*>(Qp + sw128_off(d, 2 * I)) = make_uint4(w[0], w[1], w[2], w[3]);
        *reinterpret_cast<uint4*>(Qp + sw128_off(d, 2 * I + 1)) = make_uint4(w[4], w[5], w[6], w[7]);
    }
    ok = ok && mbar_wait(&bar_mma, 0, p.status, 41);      // no block-wide barrier: see the dv staging below
    tc_fence_after();

    // ================================================================ phase 2a: first read-out
    float dqn[16], dkn[16], dG[16];
    float ge_part = 0.f;
    {
        float t[16];
        // dW^T -> bf16 operand (row = channel d, 16 of its 64 tokens)
        tmem_ld16(tmem + lane_base + cDb + 16 * I, t);
        *reinterpret_cast<uint4*>(dWs + sw128_off(d, 2 * I)) =
            make_uint4(pk2(t[0], t[1]), pk2(t[2], t[3]), pk2(t[4], t[5]), pk2(t[6], t[7]));
        *reinterpret_cast<uint4*>(dWs + sw128_off(d, 2 * I + 1)) =
            make_uint4(pk2(t[8], t[9]), pk2(t[10], t[11]), pk2(t[12], t[13]), pk2(t[14], t[15]));
        // dR, dE
        tmem_ld16(tmem + lane_base + cDa + 16 * I, t);
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            dqn[r] = t[r] * (E[r] * eCI);
            dG[r] = dqn[r] * qn[r];
        }
        tmem_ld16(tmem + lane_base + cDc + 16 * I, t);
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float ee = rcp_approx(E[r]) * eEndI;
            const float eE = t[r] * kn[r] * ee;    // dE * E
            dkn[r] = t[r] * ee;
            dG[r] -= eE;
            ge_part += eE;
        }
        // dv = beta dP, staged [token][channel] so that it leaves as 16-byte row segments.  The staging area is the value
        // tile: only the products that have just completed read it, so no thread needs to wait for the others here (the
        // state panels, in contrast, are still being read by threads that are behind in the dD sums)
        tmem_ld16(tmem + lane_base + cDd + 16 * I, t);
        __nv_bfloat16* tv = reinterpret_cast<__nv_bfloat16*>(vs);
#pragma unroll
        for (int r = 0; r < 16; ++r) tv[(16 * I + r) * 128 + d] = __float2bfloat16(rowv[128 + 16 * I + r] * t[r]);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (ok) {
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
    if (ok && tid == 0) {
        tc_fence_after();
        const uint32_t id64_neg = umma_idesc_bf16(64, 64, kMajorMN, kMajorMN, 1);
        const uint32_t id_k_mn = umma_idesc_bf16(128, 64, kMajorK, kMajorMN);
        const uint32_t aQ = smem_u32(Qp), aW = smem_u32(dWs), bT = smem_u32(Ts);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // Xraw^T -= Q' dW^T   (dW^T panel read as MN-major B: [key][token])
            umma_bf16_ss(tmem + cDf, umma_smem_desc_sw128(aQ + k16 * 2048, 8192, 1024),
                         umma_smem_desc_sw128(aW + k16 * 2048, 8192, 1024), id64_neg, 1);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // (T^T dW)^T = dW^T T ;  dQ = -that
            umma_bf16_ss(tmem + cDe, umma_smem_desc_sw128(aW + k16 * 32, 16, 1024),
                         umma_smem_desc_sw128(bT + k16 * 2048, 8192, 1024), id_k_mn, k16 > 0);
        umma_commit(&bar_mma);
    }
    ok = ok && mbar_wait(&bar_mma, 1, p.status, 42);      // no block-wide barrier: the next phase touches nothing another thread still reads
    tc_fence_after();

    // ================================================================ phase 3: X, Y, dM
    // M = 64 accumulators keep row (16*w + l) in lane l < 16 of warp w < 4.  tcgen05.ld is warp-collective, so all 32
    // lanes of those warps run the loads; lanes >= 16 mirror a row and never store.  All four warp groups see the same lanes, so each takes 16 of the 64 columns.
    const bool rowown = lane < 16;
    const int row = 16 * (warp & 3) + (lane & 15);
    uint8_t* XT = sm + kR2;           // [64 rows s][64 i]   K-major B
    uint8_t* Yt = sm + kR2 + 8192;    // [64 rows j][64 s]   K-major A
    float dbeta_acc = 0.f;
    float* dbp = dots;                // [4][64] partial dbeta per column group (dots is not in use yet)
    {
        // every warp group takes 16 of the 64 columns of row `row`
        const float bs = rowv[128 + row];
        float t[16];
        tmem_ld16(tmem + lane_base + cDf + 16 * I, t);
        uint32_t pkd[8];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int i = 16 * I + j;
            dbeta_acc += ld16(Ts, sw128_off(i, row >> 3) + (row & 7) * 2) * t[j];     // T[i][s] * Xraw[i][s]
            if (j & 1) pkd[j >> 1] = pk2(__uint_as_float(pkd[j >> 1]), bs * t[j]);
            else pkd[j >> 1] = __float_as_uint(bs * t[j]);
        }
        if (rowown) {
            *reinterpret_cast<uint4*>(XT + sw128_off(row, 2 * I)) = make_uint4(pkd[0], pkd[1], pkd[2], pkd[3]);
            *reinterpret_cast<uint4*>(XT + sw128_off(row, 2 * I + 1)) = make_uint4(pkd[4], pkd[5], pkd[6], pkd[7]);
        }
    }
    {   // dQ contributions (all threads)
        float t[16];
        tmem_ld16(tmem + lane_base + cDe + 16 * I, t);
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float dQ = -t[r] * rowv[128 + 16 * I + r] * (E[r] * eCI);   // dQ * beta * e^G
            dkn[r] += dQ;
            dG[r] += dQ * kn[r];
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
            umma_bf16_ss(tmem + cDb, umma_smem_desc_sw128(smem_u32(Ts) + k16 * 2048, 8192, 1024),
                         umma_smem_desc_sw128(smem_u32(XT) + k16 * 32, 16, 1024), id, k16 > 0);
        umma_commit(&bar_mma);
    }
    ok = ok && mbar_wait(&bar_mma, 0, p.status, 43);      // no block-wide barrier: the next phase touches nothing another thread still reads
    tc_fence_after();
    {
        float t[16];
        tmem_ld16(tmem + lane_base + cDb + 16 * I, t);
        if (rowown) {
            *reinterpret_cast<uint4*>(Yt + sw128_off(row, 2 * I)) =
                make_uint4(pk2(t[0], t[1]), pk2(t[2], t[3]), pk2(t[4], t[5]), pk2(t[6], t[7]));
            *reinterpret_cast<uint4*>(Yt + sw128_off(row, 2 * I + 1)) =
                make_uint4(pk2(t[8], t[9]), pk2(t[10], t[11]), pk2(t[12], t[13]), pk2(t[14], t[15]));
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
            umma_bf16_ss(tmem + cDc, umma_smem_desc_sw128(smem_u32(Yt) + k16 * 32, 16, 1024),
                         umma_smem_desc_sw128(smem_u32(Ts) + k16 * 32, 16, 1024), id, k16 > 0);
        umma_commit(&bar_mma);
    }
    ok = ok && mbar_wait(&bar_mma, 1, p.status, 44);      // no block-wide barrier: the next phase touches nothing another thread still reads
    tc_fence_after();

    // ================================================================ phase 4: pull-back operands
    uint8_t* Sk = sm + kR1;           // k~_I source panels: [I][128 rows d][64 s]                        K-major A
    uint8_t* Xk = sm + kR3;           // target stacks: [I / 2][128 rows d][32 rows of I even | 32 of I odd] K-major A
    uint8_t* DAt = sm + kR7;          // [I][32 rows: 16 dA rows, 16 beta*dM rows][64 s]   K-major / MN-major B
    {
        // row j of dM = -stril(Y T^T) and of dA = tril(dO Z^T), 16 source columns per warp group;
        // dbeta gets sum_l dM[j][l] M~[j][l]
        const int j = row, Ib = j >> 4, rr = j & 15;
        const float bj = rowv[128 + j];
        float tm[16], ta[16], mv16[16];
        tmem_ld16(tmem + lane_base + cDc + 16 * I, tm);
        tmem_ld16(tmem + lane_base + cDg + 16 * I, ta);
        {
            const uint4 m0 = *reinterpret_cast<const uint4*>(Mts + sw128_off(j, 2 * I));
            const uint4 m1 = *reinterpret_cast<const uint4*>(Mts + sw128_off(j, 2 * I + 1));
            const __nv_bfloat162* hh = reinterpret_cast<const __nv_bfloat162*>(&m0);
            const __nv_bfloat162* hg = reinterpret_cast<const __nv_bfloat162*>(&m1);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float2 f0 = __bfloat1622float2(hh[e]), f1 = __bfloat1622float2(hg[e]);
                mv16[2 * e] = f0.x; mv16[2 * e + 1] = f0.y; mv16[8 + 2 * e] = f1.x; mv16[8 + 2 * e + 1] = f1.y;
            }
        }
        uint32_t pa[8], pm[8];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
            const int l = 16 * I + e;
            const float dm = (l < j) ? -tm[e] : 0.f;
            // The diagonal of dA adds q k dA to dG through the row part and takes the same amount away through the
            // column part; left inside two bf16 products those O(1) terms cancel only to bf16 accuracy, which swamps dg
            // when the decay is strong.  It goes to dq and dk directly instead (decay factor 1, no dG term).
            const float da = (l < j) ? ta[e] : 0.f;
            if (l == j && rowown) dA_diag[j] = ta[e];
            dbeta_acc += dm * mv16[e];
            if (e & 1) { pa[e >> 1] = pk2(__uint_as_float(pa[e >> 1]), da); pm[e >> 1] = pk2(__uint_as_float(pm[e >> 1]), bj * dm); }
            else { pa[e >> 1] = __float_as_uint(da); pm[e >> 1] = __float_as_uint(bj * dm); }
        }
        if (rowown) {
            uint8_t* tile = DAt + Ib * 4096;
            *reinterpret_cast<uint4*>(tile + sw128_off(rr, 2 * I)) = make_uint4(pa[0], pa[1], pa[2], pa[3]);
            *reinterpret_cast<uint4*>(tile + sw128_off(rr, 2 * I + 1)) = make_uint4(pa[4], pa[5], pa[6], pa[7]);
            *reinterpret_cast<uint4*>(tile + sw128_off(16 + rr, 2 * I)) = make_uint4(pm[0], pm[1], pm[2], pm[3]);
            *reinterpret_cast<uint4*>(tile + sw128_off(16 + rr, 2 * I + 1)) = make_uint4(pm[4], pm[5], pm[6], pm[7]);
            dbp[I * 64 + j] = dbeta_acc;
        }
    }
    {
        // Both operand families are stored transposed, [channel d][row], so that this thread's 16 rows are contiguous
        // bytes of row d and leave as 16-byte stores (K-major A operands of the pull-back products).
        const float c0 = cref[d], c1 = cref[128 + d], c2 = cref[256 + d], c3 = cref[384 + d];
        const float fb0 = __expf(c1 - c0), fb1 = __expf(c2 - c1), fb2 = __expf(c3 - c2);
        uint8_t* X = Xk + (I >> 1) * 16384;      // two target blocks share a panel: 32 stack rows each
        const int xc = (I & 1) * 4;
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            uint32_t a[4], b[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = 8 * hf + 2 * e;
                a[e] = pk2(qn[r] * E[r], qn[r + 1] * E[r + 1]);      // q~ rows of this block
                b[e] = pk2(kn[r] * E[r], kn[r + 1] * E[r + 1]);      // k~ rows of this block
            }
            *reinterpret_cast<uint4*>(X + sw128_off(d, xc + hf)) = make_uint4(a[0], a[1], a[2], a[3]);
            *reinterpret_cast<uint4*>(X + sw128_off(d, xc + 2 + hf)) = make_uint4(b[0], b[1], b[2], b[3]);
            // these rows as sources of their own and every later block (zero for the earlier ones: the products sum
            // over all 64 source rows)
            uint32_t w[4][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = 8 * hf + 2 * e;
                float f0 = kn[r] * rcp_approx(E[r]), f1 = kn[r + 1] * rcp_approx(E[r + 1]);
                w[0][e] = w[1][e] = w[2][e] = 0u;
                if (I == 0) { w[0][e] = pk2(f0, f1); f0 *= fb0; f1 *= fb0; }
                if (I <= 1) { w[1][e] = pk2(f0, f1); f0 *= fb1; f1 *= fb1; }
                if (I <= 2) { w[2][e] = pk2(f0, f1); f0 *= fb2; f1 *= fb2; }
                w[3][e] = pk2(f0, f1);
            }
#pragma unroll
            for (int ver = 0; ver < 4; ++ver)
                *reinterpret_cast<uint4*>(Sk + ver * 16384 + sw128_off(d, 2 * I + hf)) =
                    make_uint4(w[ver][0], w[ver][1], w[ver][2], w[ver][3]);
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid < 64 && tid < len)
        st_io(p.dbeta, (size_t)(tok0 + tid) * H + h, p.gbf16, dbp[tid] + dbp[64 + tid] + dbp[128 + tid] + dbp[192 + tid]);
    // accumulator columns of the pull-back: RP_I (32 columns each) and CP_I (64 columns each)
    constexpr uint32_t cRP = 192;
    const uint32_t cCP[4] = {0, 64, 128, 320};
    if (ok && tid == 0) {
        tc_fence_after();
        const uint32_t id_rp = umma_idesc_bf16(128, 32, kMajorK, kMajorK);
        const uint32_t id_cp = umma_idesc_bf16(128, 64, kMajorK, kMajorMN);
#pragma unroll
        for (int Ib = 0; Ib < 4; ++Ib) {
            const uint32_t aS = smem_u32(Sk + Ib * 16384), aX = smem_u32(Xk + (Ib >> 1) * 16384) + (Ib & 1) * 64;
            const uint32_t bD = smem_u32(DAt + Ib * 4096);
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)     // RP_I^T[d][n] = sum_s k~_I[s][d] * rows_I[n][s]
                umma_bf16_ss(tmem + cRP + 32 * Ib, umma_smem_desc_sw128(aS + k16 * 32, 16, 1024),
                             umma_smem_desc_sw128(bD + k16 * 32, 16, 1024), id_rp, k16 > 0);
#pragma unroll
            for (int k16 = 0; k16 < 2; ++k16)     // CP_I^T[d][s] = sum_{n<32} stack_I[n][d] * rows_I[n][s]
                umma_bf16_ss(tmem + cCP[Ib], umma_smem_desc_sw128(aX + k16 * 32, 16, 1024),
                             umma_smem_desc_sw128(bD + k16 * 2048, 4096, 1024), id_cp, k16 > 0);
        }
        umma_commit(&bar_mma);
    }
    ok = ok && mbar_wait(&bar_mma, 0, p.status, 45);      // no block-wide barrier: the next phase touches nothing another thread still reads
    tc_fence_after();

    // ================================================================ phase 5: assemble the gradients
    {
        float t[16];
        const float c0 = cref[d], c1 = cref[128 + d], c2 = cref[256 + d], c3 = cref[384 + d];
        // decay factors of this thread's rows relative to its own block reference: e1 = e^{G - c_own} (<= 1) for the
        // row parts, e2 = e^{c_own - G} for the column parts (a later block I' contributes e^{c_I' - c_own} e2)
        const float (&e1)[16] = E;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const float dd = dA_diag[16 * I + r];
            dqn[r] += dd * kn[r];
            dkn[r] += dd * qn[r];
        }
        // The decay gradient is a telescoping sum: a pair (i, s) adds its summand to dG at row i (row part) and takes the
        // same summand away at row s (column part), and only the rows in between keep it after the reverse cumulative
        // sum.  The two parts come from different UMMAs, so they cancel exactly only if both are built from the SAME
        // rounded factors: dG therefore uses the bf16 values that sit in the operand panels (target rows q~, k~ and
        // source rows k-), while dq and dk keep the float32 factors.
        auto rb = [](float x) { return __bfloat162float(__float2bfloat16(x)); };
        tmem_ld16(tmem + lane_base + cRP + 32 * I, t);          // row part through dA
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            dqn[r] += e1[r] * t[r];
            dG[r] += rb(qn[r] * e1[r]) * t[r];
        }
        tmem_ld16(tmem + lane_base + cRP + 32 * I + 16, t);     // row part through beta*dM
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            dkn[r] += e1[r] * t[r];
            dG[r] += rb(kn[r] * e1[r]) * t[r];
        }
        // column part: sources of block I receive from target blocks I' >= I, each with its own decay reference; the
        // source factor is rebuilt exactly as the panel code built it (own-block factor, then one block step at a time)
        float fsrc[16], esrc[16];
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            esrc[r] = rcp_approx(E[r]);
            fsrc[r] = kn[r] * esrc[r];
        }
        const float fb0 = __expf(c1 - c0), fb1 = __expf(c2 - c1), fb2 = __expf(c3 - c2);
#pragma unroll
        for (int Ib = 0; Ib < 4; ++Ib) {
            if (Ib >= I) {
                tmem_ld16(tmem + lane_base + cCP[Ib] + 16 * I, t);
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    dkn[r] += esrc[r] * t[r];
                    dG[r] -= rb(fsrc[r]) * t[r];
                }
            }
            const float step = Ib == 0 ? fb0 : (Ib == 1 ? fb1 : fb2);
            if (Ib >= I && Ib < 3) {
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    fsrc[r] *= step;
                    esrc[r] *= step;
                }
            }
        }
    }
    // chunk-end term and reverse cumulative sum of dG over the 64 rows of this channel
    float suffix = 0.f;
    {
        float local = 0.f;
#pragma unroll
        for (int r = 0; r < 16; ++r) local += dG[r];
        tot[I * 128 + d] = local;
        gsum[I * 128 + d] = ge_part;       // gsum is free again
    }
    __syncthreads();
    {
        const float dGend = gsum[d] + gsum[128 + d] + gsum[256 + d] + gsum[384 + d] +
                            egend * (part[d] + part[128 + d] + part[256 + d] + part[384 + d]);
        suffix = dGend;
#pragma unroll
        for (int Ib = 3; Ib > 0; --Ib)
            if (Ib > I) suffix += tot[Ib * 128 + d];
    }
    // L2-normalisation VJP needs per-row dots over the channels: unit k is kn, unit q is qn / scale
    const float inv_scale = p.scale != 0.f ? 1.0f / p.scale : 0.f;
    {
        // 32 per-row products (q and k of 16 rows) summed over the 32 channels of this warp with 31 shuffles: each
        // step halves the values a lane carries, so lane L ends with the warp's total of value L.
        float vals[16];
        {
            const bool up = (lane & 16) != 0;      // first step straight from the operands: value j pairs with value j + 16
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float a = (j & 1) ? kn[j >> 1] * dkn[j >> 1] : qn[j >> 1] * dqn[j >> 1];                  // value j
                const float b = (j & 1) ? kn[8 + (j >> 1)] * dkn[8 + (j >> 1)] : qn[8 + (j >> 1)] * dqn[8 + (j >> 1)];   // j + 16
                vals[j] = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
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
        dots[(16 * I + (lane >> 1)) * 8 + (warp & 3) * 2 + (lane & 1)] = vals[0];
    }
    __syncthreads();
    if (tid < 128) {          // the four quadrant partials of (row, q|k) -> one number, in place
        const int i = tid >> 1, w = tid & 1;
        dots[i * 8 + w] = dots[i * 8 + w] + dots[i * 8 + 2 + w] + dots[i * 8 + 4 + w] + dots[i * 8 + 6 + w];
    }
    __syncthreads();
    {
        // The gradients of this thread's 16 rows go through shared memory (the source-panel region is free now), so
        // that they leave as 16-byte row segments instead of one 2-byte store per row, tensor and thread.
        __nv_bfloat16* tq = reinterpret_cast<__nv_bfloat16*>(sm + kR1);            // [64][128] dq
        __nv_bfloat16* tk = tq + 64 * 128;                                          // [64][128] dk
        __nv_bfloat16* tgb = tk + 64 * 128;                                         // [64][128] dg when the gate dtype is bf16
        float* tgf = reinterpret_cast<float*>(sm + kR1 + 32768);                    // [64][128] dg when it is float32
        float run = suffix;
#pragma unroll
        for (int r = 15; r >= 0; --r) {
            const int i = 16 * I + r;
            run += dG[r];
            float dqv, dkv;
            if (p.l2norm) {
                const float2 pp = *reinterpret_cast<const float2*>(dots + i * 8);
                const float pq = pp.x, pk = pp.y;
                dqv = rowv[i] * (dqn[r] * p.scale - qn[r] * inv_scale * pq);
                dkv = rowv[64 + i] * (dkn[r] - kn[r] * pk);
            } else {
                dqv = dqn[r] * p.scale;
                dkv = dkn[r];
            }
            tq[i * 128 + d] = __float2bfloat16(dqv);
            tk[i * 128 + d] = __float2bfloat16(dkv);
            if (p.gbf16) tgb[i * 128 + d] = __float2bfloat16(run);
            else tgf[i * 128 + d] = run;
        }
        __syncthreads();
        if (ok) {
            const int c = tid & 15;
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
                const int i = pass * 32 + (tid >> 4);
                if (i < len) {
                    const size_t o = ((size_t)(tok0 + i) * H + h) * 128;
                    *reinterpret_cast<uint4*>(p.dq + o + 8 * c) = *reinterpret_cast<const uint4*>(tq + i * 128 + 8 * c);
                    *reinterpret_cast<uint4*>(p.dk + o + 8 * c) = *reinterpret_cast<const uint4*>(tk + i * 128 + 8 * c);
                    if (p.gbf16) {
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
    a.dg = dg; a.dbeta = dbeta; a.gbf16 = gbf16; a.l2norm = l2norm; a.H = w.H; a.scale = scale; a.status = t.status;
    if (set_smem_limit(tc_intra_bwd_kernel, kIntraBwdSmem))
        return launch_status();
    KDA_LAUNCH("tc_intra_bwd_kernel", st,
               tc_intra_bwd_kernel<<<dim3(w.nslots, w.H), 512, kIntraBwdSmem, st>>>(mq, mk, mv, mdO, mT, mH, mdH, mZT, mdZT, mMt, a));
    return launch_status();
}

}  // namespace kda
