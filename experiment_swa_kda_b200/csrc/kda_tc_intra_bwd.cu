// Tensor-core lane, chunk-parallel part of the backward: CTAs of 512 threads, one to an SM, walk over the (chunk, head)s and turn the
// adjoints published by the reverse scan into dq, dk, dv, dg, dbeta.  K = V = 128, 64 tokens per chunk, bf16
// UMMA operands, fp32 accumulation.  Warp (I, w) owns the 16 tokens of row block I and channels 32w .. 32w+31, spread over its
// lanes in 8 x 8 pieces: lane l holds channels l/4 + {0, 8, 16, 24} and tokens 2(l%4) + {0, 1, 8, 9}.  That is what
// tcgen05.ld.16x256b reads, ldmatrix.trans takes from a [token][channel] tile and stmatrix puts back, transposed or not.
//
// Products (all on tcgen05; "^T" = channel-major result, M = 128; token x token results use M = 64):
//   dR^T = H dO^T          dW^T = H dZ^T          dE^T = dH' Z^T            (H, dH' K-major A from a walk, MN-major from split scans)
//   dP^T = dZ^T T          dQ^T = -dW^T T                                   (T row-major: MN-major B)
//   dA   = tril(dO Z^T)    Xraw^T = v dZ^T - (e^G k) dW^T    (X = Xraw diag(beta) is the adjoint of T)
//   Y    = T^T X           dM = -stril(Y T^T)
//   pull-back of dA, dM through the decay-masked products, per 16-row target block I with the block's first
//   row as decay reference (both exponential factors stay in range for g in [-5, 0]):
//     RP_I^T = k~_I^T [dA_I ; beta dM_I]^T      CP_I^T = [q~_I ; k-_I]^T [dA_I ; beta dM_I]
// Restates reference chunk_wy_backward.cu:2818-3331 (local VJP), 3337-3552 (pull-back), 3787-3894 (finalize).

#include <algorithm>

#include "common.cuh"
#include "simt_ws.cuh"
#include "tc_common.cuh"
#include "tc_ws.cuh"

namespace kda {
namespace tc {

int make_map_bf16(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);

namespace {

// one MUFU: the operands here are decay factors in [e^-75, 1], far from the flush-to-zero and overflow ends
__device__ __forceinline__ float rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// Eight 8 x 8 pieces a lane, as pairs of adjacent columns (tokens): x[2c + n] is row l/4 + 8c, columns 8n + 2(l%4) + {0, 1}
__device__ __forceinline__ void tmem_ld_16x16(uint32_t taddr, f2* x) {      // 16 lanes x 16 columns: x[0..3]
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    tmem_ld_wait();
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) x[2 * hf + n] = f2_make(__uint_as_float(r[4 * n + 2 * hf]), __uint_as_float(r[4 * n + 2 * hf + 1]));
}
__device__ __forceinline__ void tmem_ld_32x16(uint32_t taddr, f2 (&x)[8]) {      // 32 lanes x 16 columns
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%16];\n\t"
                 "tcgen05.ld.sync.aligned.16x256b.x2.b32 {%8, %9, %10, %11, %12, %13, %14, %15}, [%17];\n\t"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr), "r"(taddr + (16u << 16))
                 : "memory");
    tmem_ld_wait();
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int hf = 0; hf < 2; ++hf)
                x[4 * m + 2 * hf + n] = f2_make(__uint_as_float(r[8 * m + 4 * n + 2 * hf]), __uint_as_float(r[8 * m + 4 * n + 2 * hf + 1]));
}
__device__ __forceinline__ void ldsm_x4(uint32_t addr, uint32_t* w) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t addr, uint32_t* w) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stsm_x4(uint32_t addr, const uint32_t* w) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}
__device__ __forceinline__ void stsm_x4_t(uint32_t addr, const uint32_t* w) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
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
// Sum over the lanes of a quad that come before this one (0 in the first), and after it (0 in the last)
__device__ __forceinline__ float quad_before(float p, int c4) {
    float a = __shfl_up_sync(0xffffffffu, p, 1, 4);
    a = c4 >= 1 ? a : 0.f;
    const float b = __shfl_up_sync(0xffffffffu, a + p, 2, 4);
    return c4 >= 2 ? a + b : a;
}
__device__ __forceinline__ float quad_after(float p, int c4) {
    float a = __shfl_down_sync(0xffffffffu, p, 1, 4);
    a = c4 <= 2 ? a : 0.f;
    const float b = __shfl_down_sync(0xffffffffu, a + p, 2, 4);
    return c4 <= 1 ? a + b : a;
}

}  // namespace

struct IntraBwdArgs {
    simt::ChunkTable tab;
    const void* g;                    // [tokens][H][128], gate dtype
    const float *qinv, *kinv, *beta;  // [nch][64] from the forward
    __nv_bfloat16 *dq, *dk, *dv;
    void *dg, *dbeta;                 // gate dtype
    int l2norm, H, n_seq, nslots;
    float scale;
    int* status;
    int* next;                        // chunk-heads handed out beyond the blocks' first ones; zeroed by the kernel before this one
};

// shared-memory map (bytes, 1024-aligned base)
constexpr int kR1 = 0;         // 64 KB  H | dH' panels            -> later: k~_I source panels (4 x 16 KB)
constexpr int kR2 = 65536;     // 16 KB  dO tile                   -> later: X^T tile (8 KB) | Y tile (8 KB)
constexpr int kR3 = 81920;     // 16 KB  Z panel                   -> later: target stacks I = 0,1 (2 x 8 KB)
constexpr int kR4 = 98304;     // 16 KB  dZ panel                  -> later: target stacks I = 2,3
constexpr int kR5 = 114688;    // 48 KB  q | k | v tiles           -> later: dq | dk | dv, on their way out
constexpr int kR6 = 163840;    //  8 KB  T
constexpr int kR7 = 172032;    // 16 KB  dW^T                      -> later: [dA_I ; beta dM_I] tiles (4 x 4 KB), dg on its way out
constexpr int kR8 = 188416;    // 16 KB  g tile (bf16 gates)       -> later: Q' = e^G k
constexpr int kRM = 204800;    //  8 KB  M~ (before beta), row-major [target][source]
// floats: gfirst[4][128] gsum[4][128] eC[4][128] eEnd[4][128] fb[4][128] part[4][128] egend[128] dots[2][4][64] rowb[2][64]
//         rowv[2][3][64] (this chunk-head's and the next one's)
constexpr int kSmall = 212992;
constexpr int kIntraBwdSmem = kSmall + (24 * 128 + 128 + 512 + 2 * 64 + 2 * 3 * 64) * 4 + 1024;
constexpr int kBwdCtas = 148;      // one to an SM
// Bound by latency: 225 KB of shared memory allow one CTA per SM, and its products depend on one another (state products
// -> X -> Y -> dM -> pull-back).  So (1) only the operand of the next product is read out before that product is issued,
// and everything else - dv, the dR / dE / dQ contributions, the pull-back's decay panels - runs while it is in flight;
// (2) the products that the chain does not wait for are issued where it leaves a gap; (3) a CTA walks over chunk-heads: a tile's
// next contents are loaded as soon as its last reader is done, all but q, k and the gates behind the pull-back, so that the next
// chunk-head starts without a launch, without an allocation and with its operands there; (4) token pairs go through packed
// float32 arithmetic; (5) a lane's elements lie in 8 x 8 pieces, so that tiles are read and written by ldmatrix / stmatrix, four
// pieces an instruction, a row scalar serves eight of its elements and a row dot takes 7 shuffles: with a channel and 16 tokens a
// lane, its 2-byte accesses, row scalars and 31 shuffles had been a quarter of a block's cycles.
// 16,384 chunk-heads: 1,725 -> 1,207 us (1,490 by (2) and (5), 1,380 with cheaper issue, see elect_one; 2,262 before (1) and (4)),
// 384: 65 -> 50 us.
// KV: the panels are the walk's, states [key][value] and Z, dZ [token][value]; otherwise the split scans', states [value][key] and Z, dZ
// [value][token].
template <bool GB, bool KV>
__global__ void __launch_bounds__(512, 1)
    tc_intra_bwd_kernel(const __grid_constant__ CUtensorMap mq, const __grid_constant__ CUtensorMap mk,
                        const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mdO,
                        const __grid_constant__ CUtensorMap mT, const __grid_constant__ CUtensorMap mH,
                        const __grid_constant__ CUtensorMap mdH, const __grid_constant__ CUtensorMap mZT,
                        const __grid_constant__ CUtensorMap mdZT, const __grid_constant__ CUtensorMap mMt,
                        const __grid_constant__ CUtensorMap mg, const __grid_constant__ CUtensorMap mdq,
                        const __grid_constant__ CUtensorMap mdk, const __grid_constant__ CUtensorMap mdv,
                        const __grid_constant__ CUtensorMap mdg, IntraBwdArgs p) {
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
    float* gfirst = reinterpret_cast<float*>(sm + kSmall); // [4][128] g of the first row of each block
    float* gsum = gfirst + 512;                            // [4][128] sum of g over a block's other rows
    float* eC = gsum + 512;                                // [4][128] e^{c_I}, c_I = G at the first row of block I
    float* eEnd = eC + 512;                                // [4][128] e^{G_end - c_I}
    float* fbk = eEnd + 512;                               // [3][128] e^{c_{I+1} - c_I}
    float* part = fbk + 512;                               // [4][128] partial sums of dD
    float* egend = part + 512;                             // [128]
    float* dots = egend + 128;                             // [2][4][64] row dots: q | k, channel quarter, row
    float* rowb = dots + 512;                              // [2][64]  what the row dots take off q and k, per unit row
    float* rowv2 = rowb + 128;                             // [2][3][64]  qinv * scale | kinv | beta
    float* tot = gsum;                                     // [4][128] block sums of dG (the sums of g are done with)
    float* ge = gfirst;                                    // [4][128] block sums of dE * E
    __shared__ uint64_t bar_g, bar_a, bar_qk, bar_w, bar_x, bar_q, bar_y, bar_r, bar_m, bar_pb;
    __shared__ uint32_t tmem_slot;
    __shared__ int next[3];                         // the next chunk-head: index (past the end: none), length, first token
    __shared__ __align__(8) float dA_diag[64];      // dA[i][i]: applied to dq, dk in float32, outside the pull-back products

    // Chunk-heads in order, heads slowest: the block's own first, then one at a time as blocks become free.  Dealt out in advance,
    // the unused slots of a packed batch could all fall to the same blocks (74 sequences of 64 tokens, 148 slots, 16 heads: 184 us, now
    // 115), and a block that had to wait for an SM kept its share (backward of 8,192 chunk-heads while another stream's kernel holds 12
    // SMs: 1,630 us, now 1,127; alone 1,040 both).
    const int H = p.H, used = p.tab.per_seq > 0 ? p.nslots : p.tab.seq_chunk0[p.n_seq], total = used * H;
    int work = blockIdx.x, len = 0, tok0 = 0;
    if (work >= total) return;
    p.tab.span(work % used, tok0, len);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int I = warp >> 2, wq = warp & 3;       // row block and channel quarter of this warp
    const int c4 = lane & 3, r8 = lane >> 2;      // token pair and channel inside an 8 x 8 piece
    const int mi = lane >> 3, mr = lane & 7;      // the piece and row whose address this lane gives to ldmatrix / stmatrix
    const int tb = 16 * I + 2 * c4;               // this lane's tokens: tb + {0, 1, 8, 9}
    const int cb = 32 * wq + r8;                  // this lane's channels: cb + {0, 8, 16, 24}
    const uint32_t sb = smem_u32(sm);
    // offsets of the pieces: [token][channel] tile (channels + 16: ^ 32), [channel][token] panel (channels + 16: + 2048), tile of
    // 64 rows whose 16 rows 16wq .. belong to this warp; `chunk` is the 16-byte column of the block's first eight tokens
    const uint32_t tile_off = (uint32_t)(wq >> 1) * 8192 + sw128_off(16 * I + 8 * (mi & 1) + mr, 4 * (wq & 1) + (mi >> 1));
    auto panel_off = [&](int chunk) { return sw128_off(32 * wq + 8 * (mi >> 1) + mr, chunk + (mi & 1)); };
    const uint32_t row_off = sw128_off(16 * wq + 8 * (mi >> 1) + mr, 2 * I + (mi & 1));
    auto put_panel = [&](uint32_t panel, int chunk, const f2 (&x)[8]) {
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = f2_to_bf16(x[e]);
        const uint32_t a = panel + panel_off(chunk);
        stsm_x4(a, w);
        stsm_x4(a + 2048, w + 4);
    };
    auto put_tile = [&](uint32_t tile, const f2 (&x)[8]) {
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = f2_to_bf16(x[e]);
        stsm_x4_t(tile + tile_off, w);
        stsm_x4_t(tile + (tile_off ^ 32u), w + 4);
    };
    auto get_tile = [&](uint32_t tile, uint32_t (&w)[8]) {
        ldsm_x4_t(tile + tile_off, w);
        ldsm_x4_t(tile + (tile_off ^ 32u), w + 4);
    };
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;

    constexpr uint32_t kBytesA = 65536 + 3 * 16384 + 2 * 8192;      // H, dH', Z, dZ, dO, T, M~
    // The gates come first, then what the critical products and the work beside them need.  The loads are issued by warps 1-4,
    // a few each: one thread issuing all of them held the block back.
    if (tid == 0) {
        mbar_init(&bar_g, 1);
        mbar_init(&bar_a, 2);
        mbar_init(&bar_qk, 1);
        mbar_init(&bar_w, 1);
        mbar_init(&bar_r, 1);
        mbar_init(&bar_x, 1);
        mbar_init(&bar_q, 1);
        mbar_init(&bar_y, 1);
        mbar_init(&bar_m, 1);
        mbar_init(&bar_pb, 4);
        if (GB) mbar_expect_tx(&bar_g, 16384);
        mbar_expect_tx(&bar_a, kBytesA);
        mbar_expect_tx(&bar_a, 16384);              // v
        mbar_expect_tx(&bar_qk, 32768);
        mbar_fence_init();
    }
    __syncthreads();
    if (warp == 0) tmem_alloc(&tmem_slot, 512);

    auto load_z = [&](uint8_t* dst, const CUtensorMap& m, int c) {
        if (KV)
            for (int mb = 0; mb < 2; ++mb) tma_load_2d(dst + mb * 8192, &m, &bar_a, mb * 64, c * 64);
        else
            tma_load_2d(dst, &m, &bar_a, 0, c * 128);
    };
    // operands out of the panels at step k16 of a product: a state as A (rows: keys, contracted over values), Z or dZ as B (columns:
    // tokens, contracted over values)
    auto state_a = [&](uint32_t a, int k16) {
        return KV ? umma_smem_desc_sw128(a, 16, 1024) + ((k16 >> 2) * 16384 + (k16 & 3) * 32) : umma_smem_desc_sw128(a, 16384, 1024) + (k16 * 2048);
    };
    auto z_b = [&](uint32_t b, int k16) {
        return KV ? umma_smem_desc_sw128(b, 16, 1024) + ((k16 >> 2) * 8192 + (k16 & 3) * 32) : umma_smem_desc_sw128(b, 8192, 1024) + (k16 * 2048);
    };
    constexpr uint32_t kSt = KV ? kMajorK : kMajorMN;       // how states, Z and dZ lie as these operands
    if (warp >= 1 && warp <= 4 && elect_one()) {
        const int h = work / used, ch = (work - h * used) * H + h;
        if (warp == 1) {
            for (int mb = 0; mb < 2; ++mb) tma_load_2d(Hs + mb * 16384, &mH, &bar_a, mb * 64, ch * 128);
            load_z(dZTs, mdZT, ch);
            tma_load_2d(Ts, &mT, &bar_a, 0, ch * 64);
        } else if (warp == 2) {
            for (int mb = 0; mb < 2; ++mb) {
                tma_load_2d(vs + mb * 8192, &mv, &bar_a, h * 128 + mb * 64, tok0);
                tma_load_2d(dOs + mb * 8192, &mdO, &bar_a, h * 128 + mb * 64, tok0);
            }
        } else if (warp == 3) {
            if (GB)
                for (int mb = 0; mb < 2; ++mb) tma_load_2d(Qp + mb * 8192, &mg, &bar_g, h * 128 + mb * 64, tok0);
            for (int mb = 0; mb < 2; ++mb) tma_load_2d(ks + mb * 8192, &mk, &bar_qk, h * 128 + mb * 64, tok0);
            for (int mb = 0; mb < 2; ++mb) tma_load_2d(dHs + mb * 16384, &mdH, &bar_a, mb * 64, ch * 128);
        } else {
            for (int mb = 0; mb < 2; ++mb) tma_load_2d(qs + mb * 8192, &mq, &bar_qk, h * 128 + mb * 64, tok0);
            load_z(ZTs, mZT, ch);
            tma_load_2d(Mts, &mMt, &bar_a, 0, ch * 64);
        }
    }
    __syncwarp();
    // the row scalars of a chunk-head, 64 threads
    auto load_rows = [&](float* dst, int ch) {
        const float* src[3] = {p.qinv, p.kinv, p.beta};
#pragma unroll
        for (int j = 0; j < 3; ++j)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst + 64 * j + tid)), "l"(src[j] + (size_t)ch * 64 + tid) : "memory");
    };
    if (tid < 64) load_rows(rowv2, (work % used) * H + work / used);
    bool ok = true;
#pragma unroll 1
    for (uint32_t ph = 0;; ph ^= 1) {       // every barrier below completes once a round
    const int h = work / used;
    float* rowv = rowv2 + 192 * ph;
    // ---- per-row scalars and the log-decay relative to the block's first row
    if (tid < 64) {
        asm volatile("cp.async.wait_all;" ::: "memory");
        rowv[tid] *= p.scale;
    }
    f2 E[8];
    if constexpr (GB) {
        uint32_t w[8];
        ok = mbar_wait(&bar_g, ph, p.status, 40);
        get_tile(sb + kR8, w);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const float2 x = f2_get(f2_from_bf16(w[e]));
            const int i = tb + 8 * (e & 1);
            E[e] = f2_make(i < len ? x.x : 0.f, i + 1 < len ? x.y : 0.f);
        }
    } else {
        const float* gp = static_cast<const float*>(p.g) + ((size_t)tok0 * H + h) * 128 + cb;
        const size_t rstride = (size_t)H * 128;
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const int i = tb + 8 * (e & 1);
            const float a = gp[(size_t)min(i, len - 1) * rstride + 8 * (e >> 1)], b = gp[(size_t)min(i + 1, len - 1) * rstride + 8 * (e >> 1)];
            E[e] = f2_make(i < len ? a : 0.f, i + 1 < len ? b : 0.f);
        }
    }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        float2 g0 = f2_get(E[2 * c]), g1 = f2_get(E[2 * c + 1]);
        if (c4 == 0) {
            gfirst[I * 128 + cb + 8 * c] = g0.x;
            g0.x = 0.f;
        }
        const float p0 = g0.x + g0.y, p1 = g1.x + g1.y;
        const float b0 = quad_before(p0, c4);
        const float b1 = quad_before(p1, c4) + __shfl_sync(0xffffffffu, b0 + p0, 3, 4);
        if (c4 == 3) gsum[I * 128 + cb + 8 * c] = b1 + p1;
        E[2 * c] = f2_make(b0 + g0.x, b0 + p0);
        E[2 * c + 1] = f2_make(b1 + g1.x, b1 + p1);
    }
    tc_fence_before();
    ok = __syncthreads_and(ok);
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    // Only decay factors relative to a block's own reference c_I = G[first row of the block] are needed per element:
    // E = e^{G - c_I} (in (0, 1], at least e^-75) and its reciprocal; per block and channel there are the factors that move the
    // reference to the chunk start, the chunk end and the next block.  The operand panels and the gradient assembly use
    // bit-identical factors by construction.
    {
        const int dd = tid & 127;
        float after = 0.f, before = 0.f;           // log-decay from the next block's first row to the end; before this block
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const float sj = gfirst[j * 128 + dd] + gsum[j * 128 + dd];
            before += j < I ? sj : 0.f;
            after += j > I ? sj : 0.f;
        }
        const float first = gfirst[I * 128 + dd], rest = gsum[I * 128 + dd];
        eC[tid] = __expf(before + first);
        eEnd[tid] = __expf(rest + after);
        fbk[tid] = I < 3 ? __expf(rest + gfirst[min(I + 1, 3) * 128 + dd]) : 0.f;
        if (I == 0) egend[dd] = __expf(first + rest + after);
    }
#pragma unroll
    for (int e = 0; e < 8; ++e) {
        const float2 x = f2_get(E[e]);
        E[e] = f2_make(__expf(x.x), __expf(x.y));
    }
    auto chan4 = [&](float (&x)[4], const float* tbl) {      // a [128] table at this lane's channels
#pragma unroll
        for (int c = 0; c < 4; ++c) x[c] = tbl[cb + 8 * c];
    };

    // TMEM columns
    constexpr uint32_t cR = 0, cW = 64, cA = 128, cP = 192, cX = 256, cY = 320, cE = 384, cQ = 448, cM = cW;

    if (len < 64) {
        // rows past a ragged tail hold the next sequence's tokens: blank them (0 x Inf would otherwise reach this sequence's
        // gradients)
        ok = ok && mbar_wait(&bar_a, ph, p.status, 40) && mbar_wait(&bar_qk, ph, p.status, 40);
        if (ok) {
            for (int idx = tid; idx < (64 - len) * 16; idx += 512) {
                const int r = len + (idx >> 4), c = idx & 15;
                const uint32_t off = (uint32_t)(c >> 3) * 8192 + sw128_off(r, c & 7);
                *reinterpret_cast<uint4*>(dOs + off) = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4*>(vs + off) = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4*>(qs + off) = make_uint4(0, 0, 0, 0);
                *reinterpret_cast<uint4*>(ks + off) = make_uint4(0, 0, 0, 0);
            }
        }
        fence_async_smem();
    }
    ok = __syncthreads_and(ok);                    // tables; the g tile has been read

    // ================================================================ phase 1: state products
    // One thread issues the products, and they run in that order: dW and the first half of X, what the next link of the chain
    // X -> Y -> dM waits for, go first; the five others (~300 cycles each of operand reads) go where the chain's next product
    // is still being prepared.  Issued all at once from four warps they held those warps, and with them the block, back.
    ok = ok && mbar_wait(&bar_a, ph, p.status, 40);
    if (warp == 12 && elect_one() && ok) {
        tc_fence_after();
        const uint32_t id_st = umma_idesc_bf16(128, 64, kSt, kSt);
        const uint32_t id64_k_z = umma_idesc_bf16(64, 64, kMajorK, kSt);
        const uint32_t aH = smem_u32(Hs), bdZ = smem_u32(dZTs), aV = smem_u32(vs);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dW^T = H dZ^T
            umma_bf16_ss(tmem + cW, state_a(aH, k16), z_b(bdZ, k16), id_st, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // Xraw^T = v dZ^T  (first half)    (M = 64)
            umma_bf16_ss(tmem + cX, umma_smem_desc_sw128(aV, 16, 1024) + ((k16 >> 2) * 8192 + (k16 & 3) * 32), z_b(bdZ, k16), id64_k_z, k16 > 0);
        umma_commit(&bar_w);
    }
    __syncwarp();
    // while the tensor core works: this thread's q and k, the Q' operand, and dD[d] = sum_v dH'[d][v] H[d][v]
    // Unit k and scaled unit q of this lane's elements come from their tiles each time they are needed: at 128 registers a
    // thread q, k, the decay factors and three gradients do not fit together, and beside 226 KB of shared memory too little
    // L1 is left to spill into (it goes to L2).
    auto unit = [&](f2 (&x)[8], uint32_t tile, const float* row) {
        uint32_t w[8];
        get_tile(sb + tile, w);
        const f2 s[2] = {ld_2(row + tb), ld_2(row + tb + 8)};
#pragma unroll
        for (int e = 0; e < 8; ++e) x[e] = f2_mul(f2_from_bf16(w[e]), s[e & 1]);
    };
    constexpr uint32_t kQt = kR5, kKt = kR5 + 16384;
    ok = ok && mbar_wait(&bar_qk, ph, p.status, 40);
    {
        // Q' = e^G k for Xraw^T -= Q' dW^T, stored [key d][token] (MN-major A)
        f2 w[8];
        float ec[4];
        chan4(ec, eC + I * 128);
        unit(w, kKt, rowv + 64);
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = f2_mul(f2_mul(E[e], f2_all(ec[e >> 1])), w[e]);
        put_panel(sb + kR8, 2 * I, w);
        if constexpr (KV) {
            // Eight adjacent values of four key rows a lane; the four lanes that share the rows add up by halving.  The two halves of a
            // sum stay apart until the end: of the forms that were tried (a key row and a quarter of its values a thread; ldmatrix; one sum
            // a row) only this one leaves the rest of the block its registers, and a spill here is a trip to L2 (16,544 chunk-heads 1,324 ->
            // 1,210 us, spilled loads 44 -> 12 bytes).
            const int cg = 4 * wq + mi;
            f2 acc[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] = f2_all(0.f);
            if (ok) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t off = (uint32_t)(cg >> 3) * 16384 + sw128_off(32 * I + 8 * j + mr, cg & 7);
                    const uint4 a = *reinterpret_cast<const uint4*>(Hs + off), b = *reinterpret_cast<const uint4*>(dHs + off);
                    acc[j] = f2_fma(f2_from_bf16(a.x), f2_from_bf16(b.x), acc[j]);
                    acc[j] = f2_fma(f2_from_bf16(a.y), f2_from_bf16(b.y), acc[j]);
                    acc[j] = f2_fma(f2_from_bf16(a.z), f2_from_bf16(b.z), acc[j]);
                    acc[j] = f2_fma(f2_from_bf16(a.w), f2_from_bf16(b.w), acc[j]);
                }
            }
            float v8[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 x = f2_get(acc[e]);
                v8[2 * e] = x.x;
                v8[2 * e + 1] = x.y;
            }
#pragma unroll
            for (int o = 4; o >= 2; o >>= 1) {
                const bool up = (mi & (o >> 1)) != 0;
#pragma unroll
                for (int j = 0; j < o; ++j) {
                    const float send = up ? v8[j] : v8[j + o], keep = up ? v8[j + o] : v8[j];
                    v8[j] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * o);
                }
            }
            part[wq * 128 + 32 * I + 8 * mi + mr] = v8[0] + v8[1];
        } else {
            // eight adjacent channels of four value rows a lane; the warp's eight lanes that share them add up by halving
            const int cg = 4 * wq + mi;
            f2 acc[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[e] = f2_all(0.f);
            if (ok) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const uint32_t off = (uint32_t)(cg >> 3) * 16384 + sw128_off(32 * I + 8 * j + mr, cg & 7);
                    const uint4 a = *reinterpret_cast<const uint4*>(Hs + off), b = *reinterpret_cast<const uint4*>(dHs + off);
                    acc[0] = f2_fma(f2_from_bf16(a.x), f2_from_bf16(b.x), acc[0]);
                    acc[1] = f2_fma(f2_from_bf16(a.y), f2_from_bf16(b.y), acc[1]);
                    acc[2] = f2_fma(f2_from_bf16(a.z), f2_from_bf16(b.z), acc[2]);
                    acc[3] = f2_fma(f2_from_bf16(a.w), f2_from_bf16(b.w), acc[3]);
                }
            }
            float v8[8];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 x = f2_get(acc[e]);
                v8[2 * e] = x.x;
                v8[2 * e + 1] = x.y;
            }
#pragma unroll
            for (int o = 4; o >= 1; o >>= 1) {
                const bool up = (mr & o) != 0;
#pragma unroll
                for (int j = 0; j < o; ++j) {
                    const float send = up ? v8[j] : v8[j + o], keep = up ? v8[j + o] : v8[j];
                    v8[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                }
            }
            part[I * 128 + 8 * cg + mr] = v8[0];
        }
    }
    if (warp == 12 && elect_one() && ok) {
        tc_fence_after();
        const uint32_t aH = smem_u32(Hs), bdO = smem_u32(dOs), bZ = smem_u32(ZTs);
        const uint32_t id_st_k = umma_idesc_bf16(128, 64, kSt, kMajorK);
        const uint32_t id64_k_z = umma_idesc_bf16(64, 64, kMajorK, kSt);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dR^T = H dO^T
            umma_bf16_ss(tmem + cR, state_a(aH, k16),
                         umma_smem_desc_sw128(bdO, 16, 1024) + ((k16 >> 2) * 8192 + (k16 & 3) * 32), id_st_k, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dA = dO Z^T                      (M = 64)
            umma_bf16_ss(tmem + cA, umma_smem_desc_sw128(bdO, 16, 1024) + ((k16 >> 2) * 8192 + (k16 & 3) * 32), z_b(bZ, k16), id64_k_z, k16 > 0);
    }
    __syncwarp();
    ok = ok && mbar_wait(&bar_w, ph, p.status, 41);
    tc_fence_after();

    // ================================================================ phase 2: X and dQ
    {
        f2 t[8];      // dW^T -> bf16 operand (row = channel d)
        tmem_ld_32x16(tmem + lane_base + cW + 16 * I, t);
        put_panel(sb + kR7, 2 * I, t);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (warp == 12 && elect_one() && ok) {
        tc_fence_after();
        const uint32_t id64_neg = umma_idesc_bf16(64, 64, kMajorMN, kMajorMN, 1);
        const uint32_t id_k_mn = umma_idesc_bf16(128, 64, kMajorK, kMajorMN);
        const uint32_t aQ = smem_u32(Qp), aW = smem_u32(dWs), bT = smem_u32(Ts);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // Xraw^T -= Q' dW^T   (dW^T panel read as MN-major B: [key][token])
            umma_bf16_ss(tmem + cX, umma_smem_desc_sw128(aQ, 8192, 1024) + (k16 * 2048),
                         umma_smem_desc_sw128(aW, 8192, 1024) + (k16 * 2048), id64_neg, 1);
        umma_commit(&bar_x);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // (T^T dW)^T = dW^T T ;  dQ = -that
            umma_bf16_ss(tmem + cQ, umma_smem_desc_sw128(aW, 16, 1024) + (k16 * 32),
                         umma_smem_desc_sw128(bT, 8192, 1024) + (k16 * 2048), id_k_mn, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // dP^T = dZ^T T
            umma_bf16_ss(tmem + cP, KV ? umma_smem_desc_sw128(smem_u32(dZTs), 8192, 1024) + (k16 * 2048) : umma_smem_desc_sw128(smem_u32(dZTs), 16, 1024) + (k16 * 32),
                         umma_smem_desc_sw128(bT, 8192, 1024) + (k16 * 2048), KV ? umma_idesc_bf16(128, 64, kMajorMN, kMajorMN) : id_k_mn, k16 > 0);
        umma_commit(&bar_q);
    }
    __syncwarp();
    // The answer is on its way behind the product and goes to shared memory: held in a register up to where it is used it was
    // spilled, and the spill waited for it (323 -> 352 us at 4,096 chunk-heads).
    int taken = 0;
    if (warp == 15 && lane == 0) taken = atomicAdd(p.next, 1);
    ok = ok && mbar_wait(&bar_x, ph, p.status, 42);
    if (warp == 15 && lane == 0) next[0] = gridDim.x + taken;
    tc_fence_after();

    // ================================================================ phase 3: Y, dM
    // M = 64 accumulators keep row (16*w + l) in lane l < 16 of warp w < 4: a 16-lane read takes them whole.  All four warp groups
    // see the same lanes, so each takes 16 of the 64 columns; a lane holds rows row0 and row0 + 8, x[2 hf + n].
    const int row0 = 16 * wq + r8;
    constexpr uint32_t kXT = kR2;           // [64 rows s][64 i]   K-major B
    constexpr uint32_t kYt = kR2 + 8192;    // [64 rows j][64 s]   K-major A
    auto put_rows = [&](uint32_t tile, const f2 (&x)[4]) {
        uint32_t w[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) w[e] = f2_to_bf16(x[e]);
        stsm_x4(tile + row_off, w);
    };
    float dbeta_acc[2];
    float* dbp = reinterpret_cast<float*>(Qp);      // [4][64] partial dbeta per column group (Q' has been read once X is complete)
    {
        f2 t[4];
        tmem_ld_16x16(tmem + lane_base + cX + 16 * I, t);
        uint32_t tw[4];                             // T[i][s] in the accumulator's order (rows s)
        ldsm_x4_t(sb + kR6 + sw128_off(16 * I + 8 * (mi & 1) + mr, 2 * wq + (mi >> 1)), tw);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const f2 bs = f2_all(rowv[128 + row0 + 8 * hf]);
            const float2 a = f2_get(f2_fma(f2_from_bf16(tw[2 * hf]), t[2 * hf], f2_mul(f2_from_bf16(tw[2 * hf + 1]), t[2 * hf + 1])));   // T * Xraw
            dbeta_acc[hf] = a.x + a.y;
            t[2 * hf] = f2_mul(bs, t[2 * hf]);
            t[2 * hf + 1] = f2_mul(bs, t[2 * hf + 1]);
        }
        put_rows(sb + kXT, t);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (warp == 12 && elect_one() && ok) {
        tc_fence_after();
        const uint32_t id = umma_idesc_bf16(64, 64, kMajorMN, kMajorK);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // Y = T^T X : A[m=j][k=i] = T[i][j] (MN-major), B[n=s][k=i] = X^T rows
            umma_bf16_ss(tmem + cY, umma_smem_desc_sw128(smem_u32(Ts), 8192, 1024) + (k16 * 2048),
                         umma_smem_desc_sw128(sb + kXT, 16, 1024) + (k16 * 32), id, k16 > 0);
        umma_commit(&bar_y);
        const uint32_t id_st = umma_idesc_bf16(128, 64, kSt, kSt);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)     // dE^T = dH' Z^T
            umma_bf16_ss(tmem + cE, state_a(smem_u32(dHs), k16), z_b(smem_u32(ZTs), k16), id_st, k16 > 0);
        umma_commit(&bar_r);
    }
    __syncwarp();
    ok = ok && mbar_wait(&bar_q, ph, p.status, 42);
    tc_fence_after();
    {
        // in flight: dv = beta dP, staged [token][channel] in the value tile (only the completed products read it) so that
        // it leaves as 16-byte row segments
        f2 t[8];
        tmem_ld_32x16(tmem + lane_base + cP + 16 * I, t);
        const f2 bt[2] = {ld_2(rowv + 128 + tb), ld_2(rowv + 128 + tb + 8)};
#pragma unroll
        for (int e = 0; e < 8; ++e) t[e] = f2_mul(bt[e & 1], t[e]);
        put_tile(sb + kR5 + 32768, t);
    }
    ok = ok && mbar_wait(&bar_y, ph, p.status, 43);
    tc_fence_after();
    {
        f2 t[4];
        tmem_ld_16x16(tmem + lane_base + cY + 16 * I, t);
        put_rows(sb + kYt, t);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (warp == 12 && elect_one() && ok) {
        tc_fence_after();
        const uint32_t id = umma_idesc_bf16(64, 64, kMajorK, kMajorK);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)     // Y T^T : B[n=l][k=s] = T[l][s]
            umma_bf16_ss(tmem + cM, umma_smem_desc_sw128(sb + kYt, 16, 1024) + (k16 * 32),
                         umma_smem_desc_sw128(smem_u32(Ts), 16, 1024) + (k16 * 32), id, k16 > 0);
        umma_commit(&bar_m);
        if (len == 64) {      // in flight: the dv rows leave
            for (int mb = 0; mb < 2; ++mb) tma_store_2d(&mdv, vs + mb * 8192, h * 128 + mb * 64, tok0);
            tma_store_commit();
        }
    }
    __syncwarp();

    if (len < 64 && ok) {      // the rows past a ragged tail are not this sequence's: the others one by one
        const int c = tid & 15;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const int i = pass * 32 + (tid >> 4);
            if (i < len)
                *reinterpret_cast<uint4*>(p.dv + ((size_t)(tok0 + i) * H + h) * 128 + 8 * c) =
                    *reinterpret_cast<const uint4*>(vs + (c >> 3) * 8192 + sw128_off(i, c & 7));
        }
    }
    ok = ok && mbar_wait(&bar_r, ph, p.status, 42);       // every product up to dE is complete: its operands' tiles are free
    tc_fence_after();

    // ================================================================ phase 4: pull-back operands
    uint8_t* Sk = sm + kR1;           // k~_I source panels: [I][128 rows d][64 s], rows of blocks <= I only  K-major A
    uint8_t* Xk = sm + kR3;           // target stacks: [I / 2][128 rows d][32 rows of I even | 32 of I odd] K-major A
    uint8_t* DAt = sm + kR7;          // [I][32 rows: 16 dA rows, 16 beta*dM rows][64 s]   K-major / MN-major B
    // this warp's 16 rows of dA or dM go to the tile of row block wq
    const uint32_t da_off = kR7 + wq * 4096 + sw128_off(8 * (mi >> 1) + mr, 2 * I + (mi & 1));
    // where the next chunk-head of this CTA lies: on its way behind the panels
    int nlen = 0, ntok0 = 0;
    if (warp == 15) {
        __syncwarp();
        if (next[0] < total) p.tab.span(next[0] % used, ntok0, nlen);
    }
    {
        // in flight: the decay panels.  Both operand families are stored transposed, [channel d][row] (K-major A operands).
        const uint32_t X = sb + kR3 + (I >> 1) * 16384;      // two target blocks share a panel: 32 stack rows each
        const int xc = (I & 1) * 4;
        f2 w[8], x[8];
        unit(w, kQt, rowv);
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = f2_mul(w[e], E[e]);       // q~ rows of this block
        put_panel(X, xc, w);
        unit(x, kKt, rowv + 64);
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = f2_mul(x[e], E[e]);       // k~ rows of this block
        put_panel(X, xc + 2, w);
        // these rows as sources of their own and every later block (block I's product sums over the blocks <= I only)
        f2 ei[8];
#pragma unroll
        for (int e = 0; e < 8; ++e) ei[e] = rcp_2(E[e]);
#pragma unroll 1
        for (int ver = I; ver < 4; ++ver) {
            if (ver > I) {
                float fb[4];
                chan4(fb, fbk + (ver - 1) * 128);
#pragma unroll
                for (int e = 0; e < 8; ++e) ei[e] = f2_mul(ei[e], f2_all(fb[e >> 1]));
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) w[e] = f2_mul(x[e], ei[e]);
            put_panel(sb + kR1 + ver * 16384, 2 * I, w);
        }
    }
    {   // still in flight: the rows of dA
        f2 t[4];
        uint32_t w[4];
        // row j of dA = tril(dO Z^T), 16 source columns per warp group.  The diagonal of dA adds q k dA to dG through the
        // row part and takes the same amount away through the column part; left inside two bf16 products those O(1) terms
        // cancel only to bf16 accuracy, which swamps dg when the decay is strong.  It goes to dq and dk directly instead
        // (decay factor 1, no dG term).
        tmem_ld_16x16(tmem + lane_base + cA + 16 * I, t);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int row = row0 + 8 * (e >> 1), nd = row - (tb + 8 * (e & 1));     // columns before the diagonal, from this pair on
            const float2 a = f2_get(t[e]);
            if (nd == 0) dA_diag[row] = a.x;
            if (nd == 1) dA_diag[row] = a.y;
            w[e] = f2_to_bf16(f2_make(nd > 0 ? a.x : 0.f, nd > 1 ? a.y : 0.f));
        }
        stsm_x4(sb + da_off, w);
    }
    if (warp == 15 && lane == 0) {
        next[1] = nlen;
        next[2] = ntok0;
    }
    ok = ok && mbar_wait(&bar_m, ph, p.status, 44);
    tc_fence_after();
    {
        // row j of dM = -stril(Y T^T); dbeta gets sum_l dM[j][l] M~[j][l]
        f2 t[4];
        uint32_t mw[4], w[4];
        tmem_ld_16x16(tmem + lane_base + cM + 16 * I, t);
        ldsm_x4(sb + kRM + row_off, mw);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            const int row = row0 + 8 * hf;
            const f2 bj = f2_all(rowv[128 + row]);
            f2 acc = f2_all(0.f);
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int nd = row - (tb + 8 * n);
                const float2 a = f2_get(t[2 * hf + n]);
                const f2 dm = f2_make(nd > 0 ? -a.x : 0.f, nd > 1 ? -a.y : 0.f);
                acc = f2_fma(dm, f2_from_bf16(mw[2 * hf + n]), acc);
                w[2 * hf + n] = f2_to_bf16(f2_mul(bj, dm));
            }
            const float2 a = f2_get(acc);
            dbeta_acc[hf] += a.x + a.y;
        }
        stsm_x4(sb + da_off + 2048, w);
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            float x = dbeta_acc[hf];
            x += __shfl_xor_sync(0xffffffffu, x, 1);
            x += __shfl_xor_sync(0xffffffffu, x, 2);
            if (c4 == 0) dbp[I * 64 + row0 + 8 * hf] = x;
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    // accumulator columns of the pull-back: RP_I (32 columns each) and CP_I (16 columns for each source block up to I), beside
    // those of dR, dE and dQ
    constexpr uint32_t cRP = 64;
    auto cCP = [](int b) { return 192u + 8u * (uint32_t)(b * (b + 1)); };
    if (warp >= 12 && elect_one() && ok) {     // wq = target block; the warps with the least work of their own
        tc_fence_after();
        const uint32_t id_rp = umma_idesc_bf16(128, 32, kMajorK, kMajorK);
        const uint32_t id_cp = umma_idesc_bf16(128, 16, kMajorK, kMajorMN) + ((uint32_t)(2 * wq) << 17);      // N = 16 (wq + 1)
        const uint32_t aS = smem_u32(Sk + wq * 16384), aX = smem_u32(Xk + (wq >> 1) * 16384) + (wq & 1) * 64;
        const uint32_t bD = smem_u32(DAt + wq * 4096);
#pragma unroll 1
        for (int k16 = 0; k16 <= wq; ++k16)     // RP_I^T[d][n] = sum_{s in blocks <= I} k~_I[s][d] * rows_I[n][s]
            umma_bf16_ss(tmem + cRP + 32 * wq, umma_smem_desc_sw128(aS, 16, 1024) + (k16 * 32),
                         umma_smem_desc_sw128(bD, 16, 1024) + (k16 * 32), id_rp, k16 > 0);
#pragma unroll
        for (int k16 = 0; k16 < 2; ++k16)     // CP_I^T[d][s] = sum_{n<32} stack_I[n][d] * rows_I[n][s]
            umma_bf16_ss(tmem + cCP(wq), umma_smem_desc_sw128(aX, 16, 1024) + (k16 * 32),
                         umma_smem_desc_sw128(bD, 4096, 1024) + (k16 * 2048), id_cp, k16 > 0);
        umma_commit(&bar_pb);
    }
    __syncwarp();
    if (tid >= 128 && tid < 192 && tid - 128 < len) {
        const int i = tid - 128;
        st_io(p.dbeta, (size_t)(tok0 + i) * H + h, GB, dbp[i] + dbp[64 + i] + dbp[128 + i] + dbp[192 + i]);
    }
    const int nwork = next[0];
    const bool more = nwork < total;
    const int nh = more ? nwork / used : 0, nch = more ? (nwork - nh * used) * H + nh : 0;
    if (more && tid < 64) load_rows(rowv2 + 192 * (ph ^ 1), nch);
    // in flight: the dR part of dq, the dE and dQ parts of dk, the diagonal of dA
    f2 dqn[8], dkn[8], kn[8], dG[8];
    float ge4[4];      // sum of dE * E over this lane's tokens, per channel
    {
        f2 t[8];
        float x4[4];
        tmem_ld_32x16(tmem + lane_base + cR + 16 * I, t);
        chan4(x4, eC + I * 128);
#pragma unroll
        for (int e = 0; e < 8; ++e) dqn[e] = f2_mul(t[e], f2_mul(E[e], f2_all(x4[e >> 1])));
        unit(t, kQt, rowv);
        const f2 dd[2] = {ld_2(dA_diag + tb), ld_2(dA_diag + tb + 8)};
        unit(kn, kKt, rowv + 64);
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            dG[e] = f2_mul(dqn[e], t[e]);
            dqn[e] = f2_fma(dd[e & 1], kn[e], dqn[e]);
            dkn[e] = f2_mul(dd[e & 1], t[e]);
        }
        tmem_ld_32x16(tmem + lane_base + cE + 16 * I, t);
        chan4(x4, eEnd + I * 128);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            f2 s;
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int e = 2 * c + n;
                const f2 dE = f2_mul(t[e], f2_mul(rcp_2(E[e]), f2_all(x4[c])));
                const f2 eE = f2_mul(dE, kn[e]);        // dE * E
                dkn[e] = f2_add(dkn[e], dE);
                dG[e] = f2_fma(eE, f2_all(-1.f), dG[e]);
                s = n == 0 ? eE : f2_add(s, eE);
            }
            const float2 s2 = f2_get(s);
            ge4[c] = s2.x + s2.y;
        }
        tmem_ld_32x16(tmem + lane_base + cQ + 16 * I, t);
        chan4(x4, eC + I * 128);
        const f2 nb[2] = {neg_2(ld_2(rowv + 128 + tb)), neg_2(ld_2(rowv + 128 + tb + 8))};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            const f2 dQ = f2_mul(f2_mul(t[e], nb[e & 1]), f2_mul(E[e], f2_all(x4[e >> 1])));   // dQ * beta * e^G
            dkn[e] = f2_add(dkn[e], dQ);
            dG[e] = f2_fma(dQ, kn[e], dG[e]);
        }
    }
    ok = ok && mbar_wait(&bar_pb, ph, p.status, 45);
    tc_fence_after();
    // The products are done with every operand: the next chunk-head's take their places.
    if (warp == 15 && elect_one() && ok && more) {
        const int nt0 = next[2];
        mbar_expect_tx(&bar_a, kBytesA);
        for (int mb = 0; mb < 2; ++mb) tma_load_2d(Hs + mb * 16384, &mH, &bar_a, mb * 64, nch * 128);
        load_z(dZTs, mdZT, nch);
        for (int mb = 0; mb < 2; ++mb) tma_load_2d(dHs + mb * 16384, &mdH, &bar_a, mb * 64, nch * 128);
        for (int mb = 0; mb < 2; ++mb) tma_load_2d(dOs + mb * 8192, &mdO, &bar_a, nh * 128 + mb * 64, nt0);
        load_z(ZTs, mZT, nch);
        tma_load_2d(Ts, &mT, &bar_a, 0, nch * 64);
        tma_load_2d(Mts, &mMt, &bar_a, 0, nch * 64);
        for (int mb = 0; mb < 2; ++mb) {            // into L2 only: their tiles are still in use
            if (GB) tma_prefetch_2d(&mg, nh * 128 + mb * 64, nt0);
            tma_prefetch_2d(&mk, nh * 128 + mb * 64, nt0);
            tma_prefetch_2d(&mq, nh * 128 + mb * 64, nt0);
        }
    }
    if (!GB && warp == 14 && more) {                // float32 gates go through the threads: their rows into L2 as well (16,544
        // chunk-heads: 1,521 us without, 1,370 to 1,400 with)
        const float* gn = static_cast<const float*>(p.g) + ((size_t)next[2] * H + nh) * 128;
        for (int i = lane; i < 4 * next[1]; i += 32) prefetch_l2(gn + (size_t)(i >> 2) * H * 128 + (i & 3) * 32);
    }
    if (warp == 12 && elect_one() && ok && more) {
        tma_store_wait_read();                      // dv has left the value tile
        mbar_expect_tx(&bar_a, 16384);
        for (int mb = 0; mb < 2; ++mb) tma_load_2d(vs + mb * 8192, &mv, &bar_a, nh * 128 + mb * 64, next[2]);
    }
    __syncwarp();

    // ================================================================ phase 5: assemble the gradients
    {
        f2 t[8];
        // decay factors relative to the block's own reference: E = e^{G - c_own} (<= 1) for the
        // row parts, 1 / E for the column parts (a later block I' contributes e^{c_I' - c_own} / E)
        // The decay gradient is a telescoping sum: a pair (i, s) adds its summand to dG at row i (row part) and takes the
        // same summand away at row s (column part), and only the rows in between keep it after the reverse cumulative
        // sum.  The two parts come from different UMMAs, so they cancel exactly only if both are built from the SAME
        // rounded factors: dG therefore uses the bf16 values that sit in the operand panels (target rows q~, k~ and
        // source rows k-), while dq and dk keep the float32 factors.
        tmem_ld_32x16(tmem + lane_base + cRP + 32 * I + 16, t);     // row part through beta*dM
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            dkn[e] = f2_fma(E[e], t[e], dkn[e]);
            dG[e] = f2_fma(round_bf16_2(f2_mul(kn[e], E[e])), t[e], dG[e]);
            kn[e] = neg_2(kn[e]);                                   // -k from here on: the column part is taken away
        }
        tmem_ld_32x16(tmem + lane_base + cRP + 32 * I, t);          // row part through dA
        {
            f2 q[8];
            unit(q, kQt, rowv);
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                dqn[e] = f2_fma(E[e], t[e], dqn[e]);
                dG[e] = f2_fma(round_bf16_2(f2_mul(q[e], E[e])), t[e], dG[e]);
            }
        }
        // column part: sources of block I receive from target blocks I' >= I, each with its own decay reference; the
        // source factor is rebuilt exactly as the panel code built it
#pragma unroll
        for (int e = 0; e < 8; ++e) E[e] = rcp_2(E[e]);
#pragma unroll 1
        for (int Ib = I; Ib < 4; ++Ib) {
            tmem_ld_32x16(tmem + lane_base + cCP(Ib) + 16 * I, t);
            if (Ib > I) {
                float fb[4];
                chan4(fb, fbk + (Ib - 1) * 128);
#pragma unroll
                for (int e = 0; e < 8; ++e) E[e] = f2_mul(E[e], f2_all(fb[e >> 1]));
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                dkn[e] = f2_fma(E[e], t[e], dkn[e]);
                dG[e] = f2_fma(round_bf16_2(f2_mul(kn[e], E[e])), t[e], dG[e]);
            }
        }
    }
    // reverse cumulative sum of dG inside the block; the block's sums go to the other blocks' lanes through shared memory
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        const float2 g0 = f2_get(dG[2 * c]), g1 = f2_get(dG[2 * c + 1]);
        const float p0 = g0.x + g0.y, p1 = g1.x + g1.y;
        const float a1 = quad_after(p1, c4);
        const float a0 = quad_after(p0, c4) + __shfl_sync(0xffffffffu, a1 + p1, 0, 4);
        if (c4 == 0) tot[I * 128 + cb + 8 * c] = a0 + p0;
        dG[2 * c] = f2_make(a0 + p0, a0 + g0.y);
        dG[2 * c + 1] = f2_make(a1 + p1, a1 + g1.y);
    }
    {
        // sums of dE * E over the quad by halving: lane c4 ends with channel c4's
        const bool u2 = (c4 & 2) != 0, u1 = (c4 & 1) != 0;
        const float a = (u2 ? ge4[2] : ge4[0]) + __shfl_xor_sync(0xffffffffu, u2 ? ge4[0] : ge4[2], 2);
        const float b = (u2 ? ge4[3] : ge4[1]) + __shfl_xor_sync(0xffffffffu, u2 ? ge4[1] : ge4[3], 2);
        ge[I * 128 + cb + 8 * c4] = (u1 ? b : a) + __shfl_xor_sync(0xffffffffu, u1 ? a : b, 1);
    }
    // L2-normalisation VJP needs per-row dots over the channels: unit k is -kn, unit q is qn / scale
    f2 qn[8];
    unit(qn, kQt, rowv);
    {
        // q and k of four rows, summed over this lane's four channels, then over the eight lanes with the same rows by halving
        float v8[8];
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            f2 a = f2_mul(qn[n], dqn[n]), b = f2_mul(kn[n], dkn[n]);
#pragma unroll
            for (int c = 1; c < 4; ++c) {
                a = f2_fma(qn[2 * c + n], dqn[2 * c + n], a);
                b = f2_fma(kn[2 * c + n], dkn[2 * c + n], b);
            }
            const float2 x = f2_get(a), y = f2_get(b);
            v8[2 * n] = x.x;
            v8[2 * n + 1] = x.y;
            v8[4 + 2 * n] = y.x;
            v8[4 + 2 * n + 1] = y.y;
        }
#pragma unroll
        for (int o = 4; o >= 1; o >>= 1) {
            const bool up = (r8 & o) != 0;
#pragma unroll
            for (int j = 0; j < o; ++j) {
                const float send = up ? v8[j] : v8[j + o], keep = up ? v8[j + o] : v8[j];
                v8[j] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * o);
            }
        }
        // lane (r8, c4) holds value r8 = (q or k, n, which of the pair)
        dots[(r8 >> 2) * 256 + wq * 64 + tb + 8 * ((r8 >> 1) & 1) + (r8 & 1)] = v8[0];
    }
    __syncthreads();
    if (GB && warp == 14 && elect_one() && ok && more) {      // Q' and the dbeta sums have been read
        mbar_expect_tx(&bar_g, 16384);
        for (int mb = 0; mb < 2; ++mb) tma_load_2d(Qp + mb * 8192, &mg, &bar_g, nh * 128 + mb * 64, next[2]);
    }
    __syncwarp();
    if (tid < 128) {      // the four quarters of the channels -> what a row's dot takes off its gradient, per unit of q or -k
        const float* q4 = dots + (tid >> 6) * 256 + (tid & 63);
        const float dot = (q4[0] + q4[64]) + (q4[128] + q4[192]);
        const float inv_scale = p.scale != 0.f ? 1.0f / p.scale : 0.f;
        const float f = tid < 64 ? -inv_scale * inv_scale : -1.f;
        const bool far = tid < 64 && !(fabsf(inv_scale) > 1e-15f && fabsf(inv_scale) < 1e15f);      // its square leaves float32
        rowb[tid] = !p.l2norm ? 0.f : (far ? -(dot * inv_scale) * (inv_scale * rowv[tid]) : f * dot * rowv[tid]);
    }
    {
        // what the rows of (I, channel) get from the later blocks and from the chunk's end
        const int dd = tid & 127;
        float run = (ge[dd] + ge[128 + dd]) + (ge[256 + dd] + ge[384 + dd]);
        run = fmaf(egend[dd], (part[dd] + part[128 + dd]) + (part[256 + dd] + part[384 + dd]), run);
#pragma unroll
        for (int Ib = 3; Ib > 0; --Ib)
            if (Ib > I) run += tot[Ib * 128 + dd];
        eC[tid] = run;
    }
    __syncthreads();
    {
        // The gradients go through shared memory, so that they leave as whole rows: dq and dk over q and k, of which a warp
        // overwrites only the pieces that it alone has read, dg over the dead tiles of the pull-back.
        const f2 qa[2] = {ld_2(rowv + tb), ld_2(rowv + tb + 8)}, qb[2] = {ld_2(rowb + tb), ld_2(rowb + tb + 8)};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
            dqn[e] = f2_mul(dqn[e], qa[e & 1]);
            if (p.l2norm) dqn[e] = f2_fma(qn[e], qb[e & 1], dqn[e]);      // without it dq does not depend on q: an infinite one stays out
        }
        put_tile(sb + kQt, dqn);
        const f2 ka[2] = {ld_2(rowv + 64 + tb), ld_2(rowv + 64 + tb + 8)}, kb[2] = {ld_2(rowb + 64 + tb), ld_2(rowb + 64 + tb + 8)};
#pragma unroll
        for (int e = 0; e < 8; ++e) dkn[e] = f2_fma(kn[e], kb[e & 1], f2_mul(dkn[e], ka[e & 1]));
        put_tile(sb + kKt, dkn);
        float run[4];
        chan4(run, eC + I * 128);
#pragma unroll
        for (int e = 0; e < 8; ++e) dG[e] = f2_add(dG[e], f2_all(run[e >> 1]));
        if (GB) {
            put_tile(sb + kR7, dG);
        } else {
            float* tg = reinterpret_cast<float*>(sm + kR7);      // [64][128] (over Q' too), 16-byte columns turned by the row pair
#pragma unroll
            for (int e = 0; e < 8; ++e) {
                const float2 x = f2_get(dG[e]);
                const int i = tb + 8 * (e & 1), d = cb + 8 * (e >> 1), sw = (d & 3) + ((((d >> 2) ^ (i >> 1)) & 31) << 2);
                tg[i * 128 + sw] = x.x;
                tg[(i + 1) * 128 + sw] = x.y;
            }
        }
    }
    if (tid < 64) asm volatile("cp.async.wait_all;" ::: "memory");
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (!ok) break;
    if (len < 64 || !GB) {
        const int c = tid & 15;
#pragma unroll
        for (int pass = 0; pass < 2; ++pass) {
            const int i = pass * 32 + (tid >> 4);
            if (i < len) {
                const size_t o = ((size_t)(tok0 + i) * H + h) * 128;
                const uint32_t off = (c >> 3) * 8192 + sw128_off(i, c & 7);
                if (len < 64) {
                    *reinterpret_cast<uint4*>(p.dq + o + 8 * c) = *reinterpret_cast<const uint4*>(qs + off);
                    *reinterpret_cast<uint4*>(p.dk + o + 8 * c) = *reinterpret_cast<const uint4*>(ks + off);
                }
                if (GB) {
                    *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p.dg) + o + 8 * c) = *reinterpret_cast<const uint4*>(sm + kR7 + off);
                } else {
                    const float* tg = reinterpret_cast<const float*>(sm + kR7) + i * 128;
                    float* dgp = reinterpret_cast<float*>(p.dg) + o;
                    *reinterpret_cast<uint4*>(dgp + 4 * c) = *reinterpret_cast<const uint4*>(tg + ((c ^ (i >> 1)) & 31) * 4);
                    *reinterpret_cast<uint4*>(dgp + 64 + 4 * c) = *reinterpret_cast<const uint4*>(tg + (((16 + c) ^ (i >> 1)) & 31) * 4);
                }
            }
        }
        __syncthreads();
    }
    if (warp == 15 && elect_one()) {
        if (len == 64) {
            for (int mb = 0; mb < 2; ++mb) {
                tma_store_2d(&mdq, qs + mb * 8192, h * 128 + mb * 64, tok0);
                tma_store_2d(&mdk, ks + mb * 8192, h * 128 + mb * 64, tok0);
                if (GB) tma_store_2d(&mdg, sm + kR7 + mb * 8192, h * 128 + mb * 64, tok0);
            }
            tma_store_commit();
        }
        tma_store_wait_read();
        if (more) {
            const int nt0 = next[2];
            mbar_expect_tx(&bar_qk, 32768);
            for (int mb = 0; mb < 2; ++mb) {
                tma_load_2d(ks + mb * 8192, &mk, &bar_qk, nh * 128 + mb * 64, nt0);
                tma_load_2d(qs + mb * 8192, &mq, &bar_qk, nh * 128 + mb * 64, nt0);
            }
        }
    }
    __syncwarp();
    if (!more) break;
    work = nwork;
    len = next[1];
    tok0 = next[2];
    }
    if (!ok && tid == 0) {       // unwinding: copies in flight must land before the block may exit
        for (uint32_t par = 0; par < 2; ++par) {
            mbar_poll(&bar_a, par, kSpinLimit / 8);
            mbar_poll(&bar_qk, par, kSpinLimit / 8);
            mbar_poll(&bar_g, par, kSpinLimit / 8);
        }
    }
    if (warp == 12 && elect_one()) tma_store_wait_read();      // shared memory must outlive the reads of the bulk stores
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_slot, 512);
}

}  // namespace tc

int tc_intra_backward(const simt::Ws& w, const simt::Scr& s, const tc::TcWs& t, int n_seq, int tokens, const void* q, const void* k, const void* v,
                      const void* g, const void* d_o, int gbf16, int l2norm, float scale, void* dq, void* dk, void* dv,
                      void* dg, void* dbeta, cudaStream_t st) {
    using namespace tc;
    const uint64_t nch = (uint64_t)w.nslots * w.H;
    const uint64_t cols = (uint64_t)w.H * 128;
    CUtensorMap mq, mk, mv, mdO, mT, mH, mdH, mZT, mdZT, mMt, mg, mdq, mdk, mdv, mdg;
    int rc = 0;
    rc |= make_map_bf16(&mq, q, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mk, k, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mv, v, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mdO, d_o, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mT, t.Tp, nch * 64, 64, 64, 64);
    rc |= make_map_bf16(&mH, t.Hp, nch * 128, 128, 64, 128);
    rc |= make_map_bf16(&mdH, t.dHp, nch * 128, 128, 64, 128);
    const bool kv = t.nseg == 1;      // who left the panels
    rc |= kv ? make_map_bf16(&mZT, t.ZT, nch * 64, 128, 64, 64) : make_map_bf16(&mZT, t.ZT, nch * 128, 64, 64, 128);
    rc |= kv ? make_map_bf16(&mdZT, t.dZT, nch * 64, 128, 64, 64) : make_map_bf16(&mdZT, t.dZT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mMt, t.Mt, nch * 64, 64, 64, 64);
    rc |= make_map_bf16(&mdq, dq, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mdk, dk, (uint64_t)tokens, cols, 64, 64);
    rc |= make_map_bf16(&mdv, dv, (uint64_t)tokens, cols, 64, 64);
    if (gbf16) rc |= make_map_bf16(&mg, g, (uint64_t)tokens, cols, 64, 64) | make_map_bf16(&mdg, dg, (uint64_t)tokens, cols, 64, 64);
    else mg = mdg = mq;      // float32 gates and their gradients go through the threads
    if (rc) return KDA_ERR_CUDA;
    IntraBwdArgs a;
    a.tab = w.tab;
    a.g = g;
    a.qinv = w.qinv; a.kinv = w.kinv; a.beta = w.beta;
    a.dq = static_cast<__nv_bfloat16*>(dq); a.dk = static_cast<__nv_bfloat16*>(dk); a.dv = static_cast<__nv_bfloat16*>(dv);
    a.dg = dg; a.dbeta = dbeta; a.l2norm = l2norm; a.H = w.H; a.n_seq = n_seq; a.nslots = w.nslots; a.scale = scale; a.status = t.status;
    a.next = s.next;
    auto kern = kv ? (gbf16 ? tc_intra_bwd_kernel<true, true> : tc_intra_bwd_kernel<false, true>)
                   : (gbf16 ? tc_intra_bwd_kernel<true, false> : tc_intra_bwd_kernel<false, false>);
    if (set_smem_limit(kern, kIntraBwdSmem)) return KDA_ERR_CUDA;
    KDA_LAUNCH("tc_intra_bwd_kernel", st,
               kern<<<(unsigned)std::min<uint64_t>(nch, kBwdCtas), 512, kIntraBwdSmem, st>>>(mq, mk, mv, mdO, mT, mH, mdH, mZT, mdZT, mMt, mg, mdq, mdk, mdv, mdg, a));
    return launch_status();
}

}  // namespace kda
