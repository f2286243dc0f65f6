// Tensor-core lane, chunk-parallel part of the forward: one CTA (256 threads, two CTAs per SM) per (chunk, head) builds
// every operand panel the scans consume.  K = V = 128, chunk = 64 tokens, bf16 UMMA operands, fp32 accumulation.
//
//   norms, cumulative log-decay G (fp32)                                       CUDA cores, thread = 4 rows x 8 channels
//   A[t][s], M~[t][s] = sum_d (q|k)[t,d] e^{G_t-c} * k[s,d] e^{c-G_s}         tcgen05, M=128 N=96|32 K=128, two chains
//       c = G at the first row of the 16-row target block, so both factors stay in range for any g in [-5, 0]
//       (restates the per-tile decay centre of reference chunk_wy_forward.cu:312-376, 447-450)
//   T = (I + beta M~)^-1                                                       fp32, block forward substitution
//   U^T = P^T T^T,  W^T = Q^T T^T   (P = beta v, Q = beta e^G k)                tcgen05, M=128 N=64 K=64, MN-major A
//   R = q e^G, E = k e^{G_end-G}, e^{G_end}, A^T, T                            panels for the scans / backward
//   Pn = W^T E,  Rm^T = R^T - W^T A^T   (the chunk's state transition,         tcgen05, M=128 N=128|64 K=64, at the end:
//                                        for split scans only)
//       W^T is staged in shared memory for its store, R, E and A^T are still there as they left
// Every operand panel is written as 16-byte pieces of the 128-byte-swizzled layout the UMMA descriptors read: a thread
// owns 8 adjacent channels of 4 consecutive rows, takes q, k, g straight from global memory (a half-warp reads one
// 256-byte row segment) and needs two exponentials per element.  Only the source rows up to a target block's own end are
// built, 160 instead of 256, so all of them fit at once; the second half's tiles take their place when the products are done.
// 113 KB and <= 128 registers let two CTAs share an SM and fill each other's waits: the kernel is a chain of short phases
// between barriers.  Every panel leaves by TMA from the tile the products read, and nothing comes back: R^T stored from
// registers in 8-byte pieces (32 sectors a warp store), E and A^T fetched again for the transition, with a fence in front,
// and R^T read row by row had taken a fifth of a block's cycles.  16,384 chunk-heads: 1,157 -> 916 us, 384: 46 -> 39 us,
// 2,048 forward-only: 148 -> 126 us; without the transition 798, 34 and 115.
// Restates reference chunk_wy_forward.cu:125-405 and 761-858.

#include <cstdio>

#include "common.cuh"
#include "simt_ws.cuh"
#include "tc_common.cuh"
#include "tc_ws.cuh"

namespace kda {
namespace tc {

int make_map_bf16(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);

namespace {

constexpr int kLDs = 68;      // leading dimension (floats) of the 64x64 fp32 tiles of the inverse
constexpr int kLDt = 36;      // ... and of its 32-row scratch
constexpr int kNT = 256;

__device__ __forceinline__ uint32_t pack2(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint4 pack8(const float (&f)[8]) {
    return make_uint4(pack2(f[0], f[1]), pack2(f[2], f[3]), pack2(f[4], f[5]), pack2(f[6], f[7]));
}
// byte offset of the 16-byte piece holding channels 8*cg .. 8*cg+7 of row r in a K-major / MN-major swizzled panel whose
// 64-column blocks are blk_bytes apart
__device__ __forceinline__ uint32_t piece_off(int r, int cg, uint32_t blk_bytes) {
    return (uint32_t)(cg >> 3) * blk_bytes + sw128_off(r, cg & 7);
}
__device__ __forceinline__ void ld8(const void* base, size_t idx, int bf16, float (&f)[8]) {
    if (bf16) {
        unpack_bf16x8(__ldg(reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(base) + idx)), f);
    } else {
        const float4 a = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + idx));
        const float4 b = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(base) + idx + 4));
        f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
    }
}
__device__ __forceinline__ void lds8(const float* p, float (&f)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
// Per-channel tables (rows of 128 floats read 8 channels per lane): channel ch sits at ((ch >> 2) & 1) * 64 +
// (ch >> 3) * 4 + (ch & 3), i.e. the two float4 halves of a lane's 8 channels live in separate 64-float halves of the
// row, so that each of the two 16-byte accesses has a 16-byte lane stride (32 bytes would use half the banks).
// `row + 4 * cg` is the lane's address for channels 8 cg .. 8 cg + 7; element-wise passes over whole rows need no change
// as long as every table of the pass is in this order.
__device__ __forceinline__ void lds8c(const float* p, float (&f)[8]) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 64);
    f[0] = a.x; f[1] = a.y; f[2] = a.z; f[3] = a.w; f[4] = b.x; f[5] = b.y; f[6] = b.z; f[7] = b.w;
}
__device__ __forceinline__ void sts8c(float* p, const float (&f)[8]) {
    *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
    *reinterpret_cast<float4*>(p + 64) = make_float4(f[4], f[5], f[6], f[7]);
}
__device__ __forceinline__ float fast_ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// dst = alpha * A * B for NP independent S x S problems (row-major fp32, leading dimensions kLDs, LB, LD), all 256 threads busy:
// a thread owns one row piece of CW adjacent columns of one product.
template <int S, int NP, int LB, int LD, class PA, class PB, class PD>
__device__ __forceinline__ void tile_mm(PA pa, PB pb, PD pd, float alpha) {
    constexpr int CW = S * S * NP / kNT;          // columns per thread: 1 (8x8x4), 2 (16x16x2), 4 (32x32x1)
    constexpr int TPR = S / CW;                   // threads per row
    const int tid = threadIdx.x;
    const int prob = tid / (S * TPR), rem = tid % (S * TPR);
    const int i = rem / TPR, j0 = (rem % TPR) * CW;
    const float* A = pa(prob) + i * kLDs;
    const float* B = pb(prob) + j0;
    float acc[CW];
#pragma unroll
    for (int c = 0; c < CW; ++c) acc[c] = 0.f;
#pragma unroll
    for (int t = 0; t < S; ++t) {
        const float a = A[t];
        if (CW == 4) {
            const float4 b = *reinterpret_cast<const float4*>(B + t * LB);
            acc[0] += a * b.x; acc[1 % CW] += a * b.y; acc[2 % CW] += a * b.z; acc[3 % CW] += a * b.w;
        } else if (CW == 2) {
            const float2 b = *reinterpret_cast<const float2*>(B + t * LB);
            acc[0] += a * b.x; acc[1 % CW] += a * b.y;
        } else {
            acc[0] += a * B[t * LB];
        }
    }
    float* D = pd(prob) + i * LD + j0;
#pragma unroll
    for (int c = 0; c < CW; ++c) D[c] = alpha * acc[c];
}

// D = alpha * A * B for S x S fp32 tiles in shared memory (leading dimensions kLDs, LB, LD) on the warp-level tensor-core path:
// mma.sync m16n8k8 with every operand split into two TF32 terms (hi + lo; lo*lo dropped), which keeps float32-class
// accuracy - T feeds every later product - while one product costs a warp S/8 short steps instead of S dependent
// shared-memory round trips.  These few 16..32-wide dependent products are latency-bound; a tcgen05 round trip
// (stage operands, issue, commit, read tensor memory back) costs more than the whole product does here.
// NP problems of S x S; a warp owns one 16 x 8 output tile; warps beyond the tile count idle.
__device__ __forceinline__ void split_tf32(float x, uint32_t& hi, uint32_t& lo) {
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(hi) : "f"(x));
    const float r = x - __uint_as_float(hi);
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(lo) : "f"(r));
}
__device__ __forceinline__ void mma_tf32(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
template <int S, int NP, int LB, int LD, class PA, class PB, class PD>
__device__ __forceinline__ void warp_mm(PA pa, PB pb, PD pd, float alpha) {
    constexpr int TR = S / 16, TC = S / 8;         // output tiles per problem
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp >= NP * TR * TC) return;
    const int prob = warp / (TR * TC), tile = warp % (TR * TC);
    const int r0 = 16 * (tile / TC), c0 = 8 * (tile % TC);
    const int g = lane >> 2, tig = lane & 3;
    const float* A = pa(prob) + (r0 + g) * kLDs + tig;
    const float* B = pb(prob) + tig * LB + c0 + g;
    float d[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int ks = 0; ks < S / 8; ++ks) {
        uint32_t ah[4], al[4], bh[2], bl[2];
        split_tf32(A[8 * ks], ah[0], al[0]);
        split_tf32(A[8 * kLDs + 8 * ks], ah[1], al[1]);
        split_tf32(A[8 * ks + 4], ah[2], al[2]);
        split_tf32(A[8 * kLDs + 8 * ks + 4], ah[3], al[3]);
        split_tf32(B[(8 * ks) * LB], bh[0], bl[0]);
        split_tf32(B[(8 * ks + 4) * LB], bh[1], bl[1]);
        mma_tf32(d, al, bh);
        mma_tf32(d, ah, bl);
        mma_tf32(d, ah, bh);
    }
    float* D = pd(prob) + (r0 + g) * LD + c0 + 2 * tig;
    *reinterpret_cast<float2*>(D) = make_float2(alpha * d[0], alpha * d[1]);
    *reinterpret_cast<float2*>(D + 8 * LD) = make_float2(alpha * d[2], alpha * d[3]);
}

// Ms = (I + Ms)^-1 in place for strictly lower-triangular Ms (64x64, zero on and above the diagonal): 8x8 diagonal solves (a
// short dependent chain per thread), then merges to 16 (CUDA cores), 32 and 64 (warp-level tensor cores) with
//   inv([[A,0],[C,B]]) = [[Ai,0],[-Bi C Ai, Bi]].
// A merge reads all of C into its scratch before it writes over it.
__device__ __forceinline__ void unit_lower_inverse(float* Ms, float* tmp) {
    const int tid = threadIdx.x;
    float* Ts = Ms;
    if (tid < 64) {
        const int b = tid >> 3, j = tid & 7;          // diagonal block, column of the inverse
        const float* Lb = Ms + (8 * b) * kLDs + 8 * b;
        float x[8], L[28];
#pragma unroll
        for (int i = 1; i < 8; ++i)
#pragma unroll
            for (int t = 0; t < i; ++t) L[i * (i - 1) / 2 + t] = Lb[i * kLDs + t];
        __syncwarp();                                 // a block's eight threads sit in one warp: all have read it
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = (i == j) ? 1.f : 0.f;
#pragma unroll
        for (int i = 1; i < 8; ++i) {
            float s = 0.f;
#pragma unroll
            for (int t = 0; t < i; ++t) s += L[i * (i - 1) / 2 + t] * x[t];
            x[i] = (i > j) ? -s : x[i];
        }
        float* Tb = Ts + (8 * b) * kLDs + 8 * b;
#pragma unroll
        for (int i = 0; i < 8; ++i) Tb[i * kLDs + j] = x[i];
    }
    __syncthreads();
    // merges: tmp_p = C_p Ai_p ; T21_p = -Bi_p tmp_p
    tile_mm<8, 4, kLDs, kLDt>([&](int p) { return Ms + (16 * p + 8) * kLDs + 16 * p; }, [&](int p) { return Ts + (16 * p) * kLDs + 16 * p; },
                  [&](int p) { return tmp + p * 8 * kLDt; }, 1.f);
    __syncthreads();
    tile_mm<8, 4, kLDt, kLDs>([&](int p) { return Ts + (16 * p + 8) * kLDs + 16 * p + 8; }, [&](int p) { return tmp + p * 8 * kLDt; },
                  [&](int p) { return Ts + (16 * p + 8) * kLDs + 16 * p; }, -1.f);
    __syncthreads();
    warp_mm<16, 2, kLDs, kLDt>([&](int p) { return Ms + (32 * p + 16) * kLDs + 32 * p; }, [&](int p) { return Ts + (32 * p) * kLDs + 32 * p; },
                   [&](int p) { return tmp + p * 16 * kLDt; }, 1.f);
    __syncthreads();
    warp_mm<16, 2, kLDt, kLDs>([&](int p) { return Ts + (32 * p + 16) * kLDs + 32 * p + 16; }, [&](int p) { return tmp + p * 16 * kLDt; },
                   [&](int p) { return Ts + (32 * p + 16) * kLDs + 32 * p; }, -1.f);
    __syncthreads();
    warp_mm<32, 1, kLDs, kLDt>([&](int) { return Ms + 32 * kLDs; }, [&](int) { return Ts; }, [&](int) { return tmp; }, 1.f);
    __syncthreads();
    warp_mm<32, 1, kLDt, kLDs>([&](int) { return Ts + 32 * kLDs + 32; }, [&](int) { return tmp; }, [&](int) { return Ts + 32 * kLDs; }, -1.f);
    __syncthreads();
}

}  // namespace

struct IntraFwdArgs {
    simt::ChunkTable tab;
    const __nv_bfloat16 *q, *k;       // [tokens][H][128]
    const void* g;                    // [tokens][H][128], gate dtype
    const void* beta;                 // [tokens][H]
    int gbf16, l2norm, H;
    float scale;
    TcWs t;
    simt::Ws w;                       // per-row scalars (inverse norms, beta) kept for the backward
    int* mirror;
    int clear_status;                 // no table kernel ran before this one
    const __nv_bfloat16* xv;          // CONV only: the v convolution's input (q, k above are the q, k convolutions' inputs)
    ConvPrep conv;
};

// shared-memory map (bytes from a 1024-aligned base).  Source rows: a 16-row target block I needs the source rows of the
// blocks <= I scaled to its own decay reference, 16 + 32 + 48 + 64 rows; blocks 3, 2 and 0 fill one 128-row stack exactly,
// block 1 has its own, so that all of them exist at once and the two products run back to back.
constexpr int kFSA = 0;            // 32 KB  sources of target blocks 3 | 2 | 0 (64 | 48 | 16 rows), 2 k-blocks of 16 KB
constexpr int kFSB = 32768;        //  8 KB  sources of target block 1 (32 rows), 2 k-blocks of 4 KB
constexpr int kFXA = 40960;        // 24 KB  targets 3 | 2 | 0 (32 rows each: 16 q~, 16 k~), 2 k-blocks of 12 KB
constexpr int kFXB = 65536;        //  8 KB  targets 1, 2 k-blocks of 4 KB
constexpr int kFQ = 73728;         // 16 KB  Q = beta e^G k: MN-major A of W^T = Q^T T^T
constexpr int kFE = 90112;         // 16 KB  E = k e^{G_end-G}: the panel's store and the B operand of Pn = W^T E
constexpr int kFTab = 106496;      // floats: cref[4][128] eC[4][128] eEnd[4][128] fb[3][128] | bet[64]
constexpr int kTabFloats = 15 * 128 + 64;
// After the A / M~ products the stacks are dead and [0, 72 KB) holds the second half's tiles; the inverse's scratch lies in
// the dead tables.
constexpr int kFMs = 0;            // 17 KB  beta M~, then its inverse (fp32); the two bf16 T operands take its place
constexpr int kFTb = 0, kFTbb = 8192;
constexpr int kFAT = 18432;        //  8 KB  A^T: the panel's store and the B operand of W^T A^T
constexpr int kFMt = 26624;        //  8 KB  M~ panel on its way out, then the identity that adds R^T to the transition
constexpr int kFR = 34816;         // 16 KB  R = q e^G: the panel's store and an A operand of the transition, then Rm^T on its way out
constexpr int kFV = 51200;         // 16 KB  v tile (TMA): MN-major A of U^T = v^T (T diag(beta))^T, then U^T on its way out
static_assert(kFMs + 64 * kLDs * 4 <= kFAT && kFV + 16384 <= kFQ && 32 * kLDt <= 15 * 128, "shared-memory map");
constexpr int kIntraFwdSmem = kFTab + kTabFloats * 4 + 1024;
static_assert(2 * (kIntraFwdSmem + 64 + 1024) <= 228 * 1024, "two CTAs share an SM");

// y = silu(sum_m w[m] x[t - 3 + m]) for this thread's 4 rows x 8 channels from the 7 input rows it needs, in the
// arithmetic of the stand-alone convolution kernel (float32 accumulation in tap order, hardware-tanh sigmoid, one
// rounding to bf16), so that the fused call reproduces "convolution, then forward" bit for bit.
__device__ __forceinline__ void conv4_silu_rows(const uint4 (&xr)[7], const void* wgt, size_t wbase, int wf32, uint4 (&out)[4]) {
    float w[8][4];
#pragma unroll
    for (int c = 0; c < 8; ++c) {
        if (wf32) {
            const float4 f = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(wgt) + wbase + 4 * c));
            w[c][0] = __bfloat162float(__float2bfloat16(f.x)); w[c][1] = __bfloat162float(__float2bfloat16(f.y));
            w[c][2] = __bfloat162float(__float2bfloat16(f.z)); w[c][3] = __bfloat162float(__float2bfloat16(f.w));
        } else {
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(wgt) + wbase + 4 * c));
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
            const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
            w[c][0] = a.x; w[c][1] = a.y; w[c][2] = b.x; w[c][3] = b.y;
        }
    }
    float x[7][8];
#pragma unroll
    for (int j = 0; j < 7; ++j) unpack_bf16x8(xr[j], x[j]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float y[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            float z = 0.f;
#pragma unroll
            for (int m = 0; m < 4; ++m) z += w[c][m] * x[j + m][c];
            float th;
            asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(0.5f * z));
            y[c] = z * fmaf(0.5f, th, 0.5f);
        }
        out[j] = pack8(y);
    }
}

template <bool GBF16, bool CONV>
__global__ void __launch_bounds__(kNT, 2)
    tc_intra_fwd_kernel(const __grid_constant__ CUtensorMap mv, const __grid_constant__ CUtensorMap mUT,
                        const __grid_constant__ CUtensorMap mWT, const __grid_constant__ CUtensorMap mAT,
                        const __grid_constant__ CUtensorMap mMt, const __grid_constant__ CUtensorMap mE,
                        const __grid_constant__ CUtensorMap mP, const __grid_constant__ CUtensorMap mRm,
                        const __grid_constant__ CUtensorMap mTp, const __grid_constant__ CUtensorMap mR, IntraFwdArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
    uint8_t* vs = sm + kFV;
    uint8_t* Qs = sm + kFQ;
    float* cref = reinterpret_cast<float*>(sm + kFTab);      // [4][128] G at the first row of each 16-row block
    float* eC = cref + 512;                                  // [4][128] exp(cref)
    float* eEnd = eC + 512;                                  // [4][128] exp(G_end - cref)
    float* fbk = eEnd + 512;                                 // [3][128] exp(cref[I+1] - cref[I])
    float* bet = fbk + 384;                                  // [64]
    float* wtot = reinterpret_cast<float*>(sm + kFSA);       // [8][128] per-warp sums of g (dead before the stacks are written)
    float* gfirst = wtot + 1024;                             // [4][128] g of the first row of each block (dead with them)
    float* Ms = reinterpret_cast<float*>(sm + kFMs);
    float* tmp = cref;
    __shared__ uint64_t bar_in, bar_am, bar_uw;
    __shared__ uint32_t tmem_slot;

    // heads fastest: blocks that run side by side read neighbouring pieces of the same token rows
    const int H = p.H, slot = blockIdx.x / H, h = blockIdx.x - slot * H;
    if (p.clear_status && blockIdx.x == 0 && threadIdx.x == 0) simt::start_status(p.t.status, p.mirror);
    int len, tok0;
    p.tab.span(slot, tok0, len);
    if (len == 0) return;
    const size_t ch = blockIdx.x;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int cg = lane & 15;                      // channels 8*cg .. 8*cg+7
    const int rq = 2 * warp + (lane >> 4);         // rows 4*rq .. 4*rq+3
    const int J = warp >> 1;                       // 16-row block of this thread's rows
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const bool trans = p.t.nseg > 1;               // the split scans walk over maps of whole chunks, formed at the end

    if (warp == 0 && elect_one()) {
        mbar_init(&bar_in, 1);
        mbar_init(&bar_am, 2);
        mbar_init(&bar_uw, 1);
        mbar_fence_init();
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 256);

    // ---- loads: this thread's 4 rows x 8 channels of g, q, k (row index clamped into the chunk, values masked)
    const size_t rstride = (size_t)H * 128;
    const size_t base = ((size_t)tok0 * H + h) * 128 + 8 * cg;
    float G[4][8];
    uint4 qraw[4], kraw[4];
    float brow[4];
    // CONV: 7 input rows for 4 output rows; the rows before the chunk belong to the previous chunk of the same sequence, or
    // are the zero padding at a sequence start
    const size_t wbase = ((size_t)h * 128 + 8 * cg) * 4;
    auto conv_rows = [&](const __nv_bfloat16* x, uint4 (&xr)[7]) {
        const bool first = p.tab.starts_sequence(slot);
#pragma unroll
        for (int jj = 0; jj < 7; ++jj) {
            const int i = 4 * rq - 3 + jj;
            const long long ic = min(i, len - 1);      // rows past the tail feed masked outputs only
            xr[jj] = (i >= 0 || !first) ? __ldg(reinterpret_cast<const uint4*>(x + ((long long)tok0 + ic) * p.conv.x_ld + h * 128 + 8 * cg))
                                        : make_uint4(0, 0, 0, 0);
        }
    };
    if constexpr (CONV) {      // v's convolution follows once its operand tile is free
        uint4 xr[7];
        conv_rows(p.q, xr);
        conv4_silu_rows(xr, p.conv.w[0], wbase, p.conv.wf32, qraw);
        conv_rows(p.k, xr);
        conv4_silu_rows(xr, p.conv.w[1], wbase, p.conv.wf32, kraw);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const int i = 4 * rq + j, ic = min(i, len - 1);
        ld8(p.g, base + (size_t)ic * rstride, GBF16, G[j]);
        if constexpr (!CONV) {
            qraw[j] = __ldg(reinterpret_cast<const uint4*>(p.q + base + (size_t)ic * rstride));
            kraw[j] = __ldg(reinterpret_cast<const uint4*>(p.k + base + (size_t)ic * rstride));
        }
        brow[j] = ld_io(p.beta, (size_t)(tok0 + ic) * H + h, GBF16);
        if (i >= len) {
#pragma unroll
            for (int c = 0; c < 8; ++c) G[j][c] = 0.f;
            qraw[j] = make_uint4(0, 0, 0, 0);
            kraw[j] = make_uint4(0, 0, 0, 0);
            brow[j] = 0.f;
        }
    }
    if ((rq & 3) == 0) sts8c(gfirst + J * 128 + 4 * cg, G[0]);
    // ---- cumulative log-decay: within the thread, across the two half-warps, then across warps through shared memory
#pragma unroll
    for (int j = 1; j < 4; ++j)
#pragma unroll
        for (int c = 0; c < 8; ++c) G[j][c] += G[j - 1][c];
    float pre[8];      // sum of the rows of the other half-warp (added to the upper half's rows)
#pragma unroll
    for (int c = 0; c < 8; ++c) pre[c] = __shfl_xor_sync(0xffffffffu, G[3][c], 16);
    if (lane < 16) {
        float tot[8];
#pragma unroll
        for (int c = 0; c < 8; ++c) tot[c] = G[3][c] + pre[c];
        sts8c(wtot + warp * 128 + 4 * cg, tot);
#pragma unroll
        for (int c = 0; c < 8; ++c) pre[c] = 0.f;
    }
    // ---- inverse norms of this thread's rows: 16 lanes hold one row
    float qi[4], ki[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float fq[8], fk[8];
        unpack_bf16x8(qraw[j], fq);
        unpack_bf16x8(kraw[j], fk);
        float sq = 0.f, sk = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            sq += fq[c] * fq[c];
            sk += fk[c] * fk[c];
        }
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) {
            sq += __shfl_xor_sync(0xffffffffu, sq, o);
            sk += __shfl_xor_sync(0xffffffffu, sk, o);
        }
        const bool valid = 4 * rq + j < len;
        qi[j] = valid ? (p.l2norm ? rsqrtf(fmaxf(sq, 1e-24f)) : 1.0f) : 0.f;      // 1 / max(|q|, 1e-12)
        ki[j] = valid ? (p.l2norm ? rsqrtf(fmaxf(sk, 1e-24f)) : 1.0f) : 0.f;
        if (cg == 0) {
            const int i = 4 * rq + j;
            bet[i] = brow[j];
            p.w.beta[ch * 64 + i] = brow[j];
            p.w.qinv[ch * 64 + i] = qi[j];
            p.w.kinv[ch * 64 + i] = ki[j];
        }
        qi[j] *= p.scale;
    }
    tc_fence_before();
    __syncthreads();                                   // (1) warp sums, first rows, TMEM slot
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    {
        // per (block, channel) factors, two entries a thread, straight from the warp sums (two warps to a block).  The sums
        // run in the order of a row's own G below, so that a block's first row has the factor 1 exactly.
        const int pos = tid & 127;
        float run[5], wsum = 0.f;                      // G at the first row of each block, then G_end
#pragma unroll
        for (int w2 = 0; w2 < 8; ++w2) {
            if ((w2 & 1) == 0) run[w2 >> 1] = gfirst[(w2 >> 1) * 128 + pos] + wsum;
            wsum += wtot[w2 * 128 + pos];
        }
        run[4] = wsum;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            if ((e & 1) == (tid >> 7)) {
                cref[e * 128 + pos] = run[e];
                eC[e * 128 + pos] = __expf(run[e]);
                eEnd[e * 128 + pos] = __expf(wsum - run[e]);
                if (e < 3) fbk[e * 128 + pos] = __expf(run[e + 1] - run[e]);
            }
        }
        if (tid < 128)      // position -> channel
            p.t.decay_end[ch * 128 + ((pos & 63) >> 2) * 8 + (pos >> 6) * 4 + (pos & 3)] = __expf(wsum);
    }
    {
        for (int w2 = 0; w2 < warp; ++w2) {
            float t[8];
            lds8c(wtot + w2 * 128 + 4 * cg, t);
#pragma unroll
            for (int c = 0; c < 8; ++c) pre[c] += t[c];
        }
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int c = 0; c < 8; ++c) G[j][c] += pre[c];
    }
    __syncthreads();                                   // (2) tables; wtot is dead from here

    // ---- operand panels, one row at a time, four channels at a time in packed pairs: 16-byte pieces of the swizzled
    // layouts.  Bound by instruction issue: two exponentials and reciprocals an element are 6 of its ~20 instructions.
    uint32_t rw[4][4];                                 // R = q e^G, rows 4rq .. 4rq+3, channel pairs (stored once the stacks are dead)
    {
        // row bases of target block b in the stacks: {3, 2, 0} share the first pair, {1} has the second
        uint8_t* X = sm + (J == 1 ? kFXB : kFXA);
        const uint32_t xkb = J == 1 ? 4096u : 12288u;
        const int xr0 = J == 3 || J == 1 ? 0 : (J == 2 ? 32 : 64);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int i = 4 * rq + j;
            const uint32_t qw[4] = {qraw[j].x, qraw[j].y, qraw[j].z, qraw[j].w};
            const uint32_t kw[4] = {kraw[j].x, kraw[j].y, kraw[j].z, kraw[j].w};
            const f2 qi2 = f2_all(qi[j]), ki2 = f2_all(ki[j]), b2 = f2_all(brow[j]);
            uint32_t xq[4], xk[4], src[4][4], ew[4], pw[4];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                const int to = J * 128 + 64 * hf + 4 * cg;
                const float4 cJ = *reinterpret_cast<const float4*>(cref + to);
                const float4 ec = *reinterpret_cast<const float4*>(eC + to);
                const float4 ee = *reinterpret_cast<const float4*>(eEnd + to);
                const f2 cj2[2] = {f2_make(cJ.x, cJ.y), f2_make(cJ.z, cJ.w)};
                const f2 ec2[2] = {f2_make(ec.x, ec.y), f2_make(ec.z, ec.w)};
                const f2 ee2[2] = {f2_make(ee.x, ee.y), f2_make(ee.z, ee.w)};
                f2 f0[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int w = 2 * hf + e;
                    const f2 dG = f2_fma(cj2[e], f2_all(-1.f), f2_make(G[j][2 * w], G[j][2 * w + 1]));
                    const float2 x = f2_get(f2_mul(dG, f2_all(1.44269504f)));
                    const f2 tq = f2_make(fast_ex2(x.x), fast_ex2(x.y));   // e^{G - c_J} in (0, 1]; its reciprocal does not wait for it
                    const f2 q = f2_mul(f2_from_bf16(qw[w]), qi2), k = f2_mul(f2_from_bf16(kw[w]), ki2);
                    xq[w] = f2_to_bf16(f2_mul(q, tq));
                    xk[w] = f2_to_bf16(f2_mul(k, tq));
                    const f2 eg = f2_mul(tq, ec2[e]);                      // e^G
                    pw[w] = f2_to_bf16(f2_mul(f2_mul(b2, eg), k));         // Q = beta e^G k
                    rw[j][w] = f2_to_bf16(f2_mul(q, eg));
                    f0[e] = f2_mul(k, f2_make(fast_ex2(-x.x), fast_ex2(-x.y)));  // source row scaled to its own block
                    ew[w] = f2_to_bf16(f2_mul(f0[e], ee2[e]));             // E = k e^{G_end - G}
                    src[0][w] = f2_to_bf16(f0[e]);
                }
                // ... and to every later block
#pragma unroll
                for (int v = 1; v < 4; ++v) {
                    if (J + v < 4) {
                        const float4 fb = *reinterpret_cast<const float4*>(fbk + (J + v - 1) * 128 + 64 * hf + 4 * cg);
                        f0[0] = f2_mul(f0[0], f2_make(fb.x, fb.y));
                        f0[1] = f2_mul(f0[1], f2_make(fb.z, fb.w));
                        src[v][2 * hf] = f2_to_bf16(f0[0]);
                        src[v][2 * hf + 1] = f2_to_bf16(f0[1]);
                    }
                }
            }
            auto put = [](uint8_t* dst, const uint32_t (&w)[4]) { *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]); };
            put(X + piece_off(xr0 + (i & 15), cg, xkb), xq);
            put(X + piece_off(xr0 + 16 + (i & 15), cg, xkb), xk);
            put(Qs + piece_off(i, cg, 8192), pw);
            put(sm + kFE + piece_off(i, cg, 8192), ew);
#pragma unroll
            for (int v = 0; v < 4; ++v) {
                const int b = J + v;                   // target block
                if (b < 4) {
                    if (b == 1) put(sm + kFSB + piece_off(i, cg, 4096), src[v]);
                    else put(sm + kFSA + piece_off((b == 3 ? 0 : (b == 2 ? 64 : 112)) + i, cg, 16384), src[v]);
                }
            }
        }
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();                                   // (3) operands complete
    if (warp < 2 && elect_one()) {
        // warp 0: targets 3, 2, 0 against the full stack.  warp 1: target 1; its stack has 32 rows, the product's other 96
        // read the bytes behind them and are never looked at.
        tc_fence_after();
        const uint32_t idesc = umma_idesc_bf16(128, warp == 0 ? 96 : 32, kMajorK, kMajorK);
        const uint32_t a0 = smem_u32(sm + (warp == 0 ? kFSA : kFSB)), b0 = smem_u32(sm + (warp == 0 ? kFXA : kFXB));
        const uint32_t akb = warp == 0 ? 16384u : 4096u, bkb = warp == 0 ? 12288u : 4096u;
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)
            umma_bf16_ss(tmem + warp * 96, umma_smem_desc_sw128(a0, 16, 1024) + ((k16 >> 2) * akb + (k16 & 3) * 32),
                         umma_smem_desc_sw128(b0, 16, 1024) + ((k16 >> 2) * bkb + (k16 & 3) * 32), idesc, k16 > 0);
        umma_commit(&bar_am);
    }
    __syncwarp();
    // in flight: the E panel leaves, v's convolution, the next block's inputs
    if (warp == 0 && elect_one()) {
        for (int nb = 0; nb < 2; ++nb) tma_store_2d(&mE, sm + kFE + nb * 8192, nb * 64, (int)(ch * 64));
        tma_store_commit();
    }
    uint4 vr[4];
    if constexpr (CONV) {
        uint4 xr[7];
        conv_rows(p.xv, xr);
        conv4_silu_rows(xr, p.conv.w[2], wbase, p.conv.wf32, vr);
    }
    if (warp == 7) {
        // two blocks to an SM: the one that starts when this one ends is about 296 further on
        const unsigned nxt = blockIdx.x + 296u;
        if (nxt < gridDim.x) {
            const int ns = (int)(nxt / H), nh = (int)(nxt % H);
            int nlen, nt0;
            p.tab.span(ns, nt0, nlen);
            if (!CONV && nlen > 0 && lane < 2) tma_prefetch_2d(&mv, nh * 128 + lane * 64, nt0);
            for (int i = lane; i < nlen; i += 32) {
                const size_t o = ((size_t)(nt0 + i) * H + nh) * 128;
#pragma unroll
                for (int b = 0; b < 128; b += GBF16 ? 64 : 32)
                    prefetch_l2(GBF16 ? static_cast<const void*>(static_cast<const __nv_bfloat16*>(p.g) + o + b)
                                      : static_cast<const void*>(static_cast<const float*>(p.g) + o + b));
                if constexpr (!CONV) {
                    prefetch_l2(p.q + o);
                    prefetch_l2(p.q + o + 64);
                    prefetch_l2(p.k + o);
                    prefetch_l2(p.k + o + 64);
                }
            }
        }
        __syncwarp();
    }
    bool ok = mbar_wait(&bar_am, 0, p.t.status, 31);
    ok = __syncthreads_and(ok);                        // (4) both accumulators complete, stacks dead
    tc_fence_after();
    if (ok) {
        if constexpr (CONV) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = 4 * rq + j;
                *reinterpret_cast<uint4*>(vs + piece_off(i, cg, 8192)) = i < len ? vr[j] : make_uint4(0, 0, 0, 0);
            }
        } else if (warp == 0 && elect_one()) {
            mbar_expect_tx(&bar_in, 16384);
            for (int kb = 0; kb < 2; ++kb) tma_load_2d(vs + kb * 8192, &mv, &bar_in, h * 128 + kb * 64, tok0);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<uint4*>(sm + kFR + piece_off(4 * rq + j, cg, 8192)) = make_uint4(rw[j][0], rw[j][1], rw[j][2], rw[j][3]);
        // ---- A^T panel, M~ panel and beta*M~ (fp32): a thread takes one source row s of one target block Ib, 16 columns
        // of A (q targets) and 16 of M~ (k targets).  Accumulator lanes: block 3 in warps 0, 1, block 2 in warp 2 and half
        // of warp 3, block 0 in the other half, block 1 in warp 4; warps 5 to 7 fill in the sources behind a target block.
        {
            int Ib, s;
            uint32_t t[32];
            if (warp < 2) { Ib = 3; s = 32 * warp + lane; }
            else if (warp == 2) { Ib = 2; s = lane; }
            else if (warp == 3) { Ib = lane < 16 ? 2 : 0; s = lane < 16 ? 32 + lane : lane - 16; }
            else if (warp == 4) { Ib = 1; s = lane; }
            else if (warp == 5) { Ib = 1; s = 32 + lane; }
            else if (warp == 6) { Ib = 0; s = 16 + lane; }
            else { Ib = lane < 16 ? 0 : 2; s = 48 + (lane & 15); }
            if (warp < 5) {
                tmem_ld32(tmem + lane_base + (warp < 2 ? 0 : (warp == 4 ? 96 : 32)), t);
                if (warp == 3) {
                    uint32_t u[32];
                    tmem_ld32(tmem + lane_base + 64, u);
                    tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 32; ++c) t[c] = lane < 16 ? t[c] : u[c];
                }
                tmem_ld_wait();
            } else {
#pragma unroll
                for (int c = 0; c < 32; ++c) t[c] = 0u;
            }
            uint32_t at[8];
#pragma unroll
            for (int c = 0; c < 16; c += 2) {
                const float a0 = (s <= 16 * Ib + c) ? __uint_as_float(t[c]) : 0.f;
                const float a1 = (s <= 16 * Ib + c + 1) ? __uint_as_float(t[c + 1]) : 0.f;
                at[c >> 1] = pack2(a0, a1);
            }
            // both panels leave through shared memory as one TMA store each
            uint8_t* ATs = sm + kFAT;              // [64 s][64 i]  bf16, 128-byte swizzle
            uint8_t* Mts = sm + kFMt;              // [64 tt][64 s]
            *reinterpret_cast<uint4*>(ATs + sw128_off(s, 2 * Ib)) = make_uint4(at[0], at[1], at[2], at[3]);
            *reinterpret_cast<uint4*>(ATs + sw128_off(s, 2 * Ib + 1)) = make_uint4(at[4], at[5], at[6], at[7]);
#pragma unroll
            for (int c = 0; c < 16; ++c) {
                const int tt = 16 * Ib + c;
                const float mt = (s < tt) ? __uint_as_float(t[16 + c]) : 0.f;
                Ms[tt * kLDs + s] = bet[tt] * mt;
                *reinterpret_cast<__nv_bfloat16*>(Mts + sw128_off(tt, s >> 3) + (s & 7) * 2) = __float2bfloat16(mt);
            }
        }
        fence_async_smem();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tma_store_2d(&mAT, sm + kFAT, 0, (int)(ch * 64));
            for (int nb = 0; nb < 2; ++nb) tma_store_2d(&mR, sm + kFR + nb * 8192, nb * 64, (int)(ch * 64));
            if (!p.t.fwd_only) tma_store_2d(&mMt, sm + kFMt, 0, (int)(ch * 64));
            tma_store_commit();
        }
        unit_lower_inverse(Ms, tmp);
        // ---- T: bf16 K-major B operands (plain and column-scaled by beta); 32 bytes of a row each, lanes on
        // consecutive rows (272 bytes apart: every 16-byte access of a quarter-warp lands in its own banks).  The plain
        // operand tile is the T panel as TMA lays it out, so the panel is stored from it below.
        {
            const int i = tid & 63, seg = tid >> 6;
            const float* src = Ms + i * kLDs + 16 * seg;
            const float* bb = bet + 16 * seg;
            uint4 u[2], ub[2];
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                float x[8], b8[8];
                lds8(src + 8 * hh, x);
                lds8(bb + 8 * hh, b8);
                u[hh] = pack8(x);
#pragma unroll
                for (int c = 0; c < 8; ++c) x[c] *= b8[c];
                ub[hh] = pack8(x);
            }
            if (trans && warp == 0 && elect_one()) tma_store_wait_read();       // the M~ panel has left: the identity takes its place
            __syncthreads();                           // everyone has its piece of T: the operands take its place
#pragma unroll
            for (int hh = 0; hh < 2; ++hh) {
                const uint32_t off = sw128_off(i, 2 * seg + hh);
                *reinterpret_cast<uint4*>(sm + kFTb + off) = u[hh];
                *reinterpret_cast<uint4*>(sm + kFTbb + off) = ub[hh];
                if (trans && !p.t.fwd_only) {
                    const int one = i - 16 * seg - 8 * hh;         // this row's element on the diagonal, if it is in these 8
                    const uint32_t w = (one & 1) ? 0x3f800000u : 0x3f80u;
                    *reinterpret_cast<uint4*>(sm + kFMt + off) = make_uint4((one >> 1) == 0 ? w : 0u, (one >> 1) == 1 ? w : 0u, (one >> 1) == 2 ? w : 0u, (one >> 1) == 3 ? w : 0u);
                }
            }
        }
        // the value tile: wait for it, blank the rows past a ragged tail (they hold other tokens)
        if (!CONV) ok = mbar_wait(&bar_in, 0, p.t.status, 30);
        if (!CONV && len < 64 && ok) {
            for (int idx = tid; idx < (64 - len) * 16; idx += kNT) {
                const int r = len + (idx >> 4), c = idx & 15;
                *reinterpret_cast<uint4*>(vs + (c >> 3) * 8192 + sw128_off(r, c & 7)) = make_uint4(0, 0, 0, 0);
            }
        }
        fence_async_smem();
        tc_fence_before();
        ok = __syncthreads_and(ok);
        if (warp == 0 && elect_one() && ok) {
            if (!p.t.fwd_only) {                   // kept for the backward only
                tma_store_2d(&mTp, sm + kFTb, 0, (int)(ch * 64));
                tma_store_commit();
            }
            tc_fence_after();
            const uint32_t idesc = umma_idesc_bf16(128, 64, kMajorMN, kMajorK);
            const uint32_t b0 = smem_u32(sm + kFTb), b1 = smem_u32(sm + kFTbb);
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)     // U^T = v^T (T diag(beta))^T
                umma_bf16_ss(tmem + 128, umma_smem_desc_sw128(smem_u32(vs), 8192, 1024) + (k16 * 2048),
                             umma_smem_desc_sw128(b1, 16, 1024) + (k16 * 32), idesc, k16 > 0);
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)     // W^T = Q^T T^T
                umma_bf16_ss(tmem + 192, umma_smem_desc_sw128(smem_u32(Qs), 8192, 1024) + (k16 * 2048),
                             umma_smem_desc_sw128(b0, 16, 1024) + (k16 * 32), idesc, k16 > 0);
            umma_commit(&bar_uw);
        }
        if (ok) ok = mbar_wait(&bar_uw, 0, p.t.status, 32);
        tc_fence_after();
        const int kt = (warp & 3) * 32 + lane, gt = warp >> 2;      // transition read-out: key row, column half
        if (ok) {
            // lane = value channel (U^T, warps 0-3) / key channel (W^T, warps 4-7): one 128-byte panel row per thread,
            // staged in the swizzled layout over the dead v and Q tiles and stored by TMA, 16 KB per panel
            const int which = warp >> 2;
            const int d = (warp & 3) * 32 + lane;
            uint8_t* stg = which ? Qs : vs;
#pragma unroll
            for (int hb = 0; hb < 2; ++hb) {
                uint32_t r[32];
                tmem_ld32(tmem + lane_base + 128 + which * 64 + hb * 32, r);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    *reinterpret_cast<uint4*>(stg + sw128_off(d, 4 * hb + c)) =
                        make_uint4(pack2(__uint_as_float(r[8 * c]), __uint_as_float(r[8 * c + 1])),
                                   pack2(__uint_as_float(r[8 * c + 2]), __uint_as_float(r[8 * c + 3])),
                                   pack2(__uint_as_float(r[8 * c + 4]), __uint_as_float(r[8 * c + 5])),
                                   pack2(__uint_as_float(r[8 * c + 6]), __uint_as_float(r[8 * c + 7])));
            }
        }
        fence_async_smem();
        tc_fence_before();
        ok = __syncthreads_and(ok);
        if (warp == 0 && elect_one() && ok) {
            tma_store_2d(&mUT, vs, 0, (int)(ch * 128));
            tma_store_2d(&mWT, Qs, 0, (int)(ch * 128));
            tma_store_commit();
            if (trans) {
                // ---- chunk transition, fused: Pn = W^T E and Rm^T = R^T - W^T A^T from the tiles that are still here.  Every
                // accumulator column has been read out: Pn takes columns 0..127, Rm^T columns 128..191.  R lies token by token,
                // so the product with an identity brings it in transposed (exactly: one term a sum).
                tc_fence_after();
                const uint32_t a0 = smem_u32(Qs), bE = smem_u32(sm + kFE);
                const uint32_t id128 = umma_idesc_bf16(128, 128, kMajorK, kMajorMN);
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16)     // Pn = W^T E
                    umma_bf16_ss(tmem, umma_smem_desc_sw128(a0, 16, 1024) + (k16 * 32),
                                 umma_smem_desc_sw128(bE, 8192, 1024) + (k16 * 2048), id128, k16 > 0);
                if (!p.t.fwd_only) {
                    const uint32_t idn = umma_idesc_bf16(128, 64, kMajorK, kMajorMN, 1), idr = umma_idesc_bf16(128, 64, kMajorMN, kMajorK);
                    const uint32_t aR = smem_u32(sm + kFR), bA = smem_u32(sm + kFAT), bI = smem_u32(sm + kFMt);
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16)     // -(A W)^T = -W^T A^T
                        umma_bf16_ss(tmem + 128, umma_smem_desc_sw128(a0, 16, 1024) + (k16 * 32),
                                     umma_smem_desc_sw128(bA, 8192, 1024) + (k16 * 2048), idn, k16 > 0);
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16)     // + R^T I
                        umma_bf16_ss(tmem + 128, umma_smem_desc_sw128(aR, 8192, 1024) + (k16 * 2048),
                                     umma_smem_desc_sw128(bI, 16, 1024) + (k16 * 32), idr, 1);
                }
                // the staging below overwrites E, R and T: their stores must have been read, all but the newest group's
                tma_store_wait_read_but1();
                umma_commit(&bar_uw);
            }
        }
        if (trans) {
            if (ok) ok = mbar_wait(&bar_uw, 1, p.t.status, 34);      // no block-wide barrier: the staging below overwrites only what
            tc_fence_after();                                         // the completed products were the last to read
            if (ok) {
                // both results leave through shared memory in the swizzled layout (Pn over the T operands and the E tile, Rm^T
                // over the R tile, all of them read for the last time) and are stored by TMA
                uint8_t* Pst = sm + (gt ? kFE : kFTb);           // [128 key rows][64 columns of half gt]
#pragma unroll
                for (int b = 0; b < 2; ++b) {
                    uint32_t r[32];
                    tmem_ld32(tmem + lane_base + 64 * gt + 32 * b, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *reinterpret_cast<uint4*>(Pst + sw128_off(kt, 4 * b + c)) =
                            make_uint4(pack2(__uint_as_float(r[8 * c]), __uint_as_float(r[8 * c + 1])),
                                       pack2(__uint_as_float(r[8 * c + 2]), __uint_as_float(r[8 * c + 3])),
                                       pack2(__uint_as_float(r[8 * c + 4]), __uint_as_float(r[8 * c + 5])),
                                       pack2(__uint_as_float(r[8 * c + 6]), __uint_as_float(r[8 * c + 7])));
                }
                if (!p.t.fwd_only) {     // the adjoint scan's operand is not needed in a forward-only call
                    uint32_t r[32];
                    tmem_ld32(tmem + lane_base + 128 + 32 * gt, r);
                    tmem_ld_wait();
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        *reinterpret_cast<uint4*>(sm + kFR + sw128_off(kt, 4 * gt + c)) =
                            make_uint4(pack2(__uint_as_float(r[8 * c]), __uint_as_float(r[8 * c + 1])),
                                       pack2(__uint_as_float(r[8 * c + 2]), __uint_as_float(r[8 * c + 3])),
                                       pack2(__uint_as_float(r[8 * c + 4]), __uint_as_float(r[8 * c + 5])),
                                       pack2(__uint_as_float(r[8 * c + 6]), __uint_as_float(r[8 * c + 7])));
                }
            }
            fence_async_smem();
            ok = __syncthreads_and(ok);
            if (warp == 0 && elect_one() && ok) {
                for (int nb = 0; nb < 2; ++nb) tma_store_2d(&mP, sm + (nb ? kFE : kFTb), nb * 64, (int)(ch * 128));
                if (!p.t.fwd_only) tma_store_2d(&mRm, sm + kFR, 0, (int)(ch * 128));
                tma_store_commit();
            }
        }
        if (warp == 0 && elect_one()) tma_store_wait_read();           // shared memory must outlive the reads of the bulk stores
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 256);
}

}  // namespace tc

int tc_intra_forward(const simt::Ws& w, const tc::TcWs& t, const void* q, const void* k, const void* v, const void* g,
                     const void* beta, int gbf16, int l2norm, float scale, int tokens, const tc::ConvPrep* conv, cudaStream_t st) {
    using namespace tc;
    IntraFwdArgs a;
    a.tab = w.tab; a.mirror = status_mirror(); a.clear_status = w.tab.per_seq > 0;
    a.q = static_cast<const __nv_bfloat16*>(q); a.k = static_cast<const __nv_bfloat16*>(k);
    a.g = g; a.beta = beta; a.gbf16 = gbf16; a.l2norm = l2norm; a.H = w.H; a.scale = scale; a.t = t; a.w = w;
    a.xv = static_cast<const __nv_bfloat16*>(v);
    a.conv = conv != nullptr ? *conv : tc::ConvPrep{{nullptr, nullptr, nullptr}, 0, 0};
    if (conv != nullptr && !t.fwd_only) return KDA_ERR_UNSUPPORTED;      // a backward would need q, k, v in memory
    const uint64_t nch = (uint64_t)w.nslots * w.H;
    CUtensorMap mv, mUT, mWT, mAT, mMt, mE, mP, mRm, mTp, mR;
    int rc = make_map_bf16(&mv, v, (uint64_t)tokens, (uint64_t)w.H * 128, 64, 64);
    rc |= make_map_bf16(&mUT, t.UT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mWT, t.WT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mAT, t.AT, nch * 64, 64, 64, 64);
    rc |= make_map_bf16(&mMt, t.fwd_only ? t.AT : t.Mt, nch * 64, 64, 64, 64);      // not stored in a forward-only call
    rc |= make_map_bf16(&mE, t.E, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mR, t.R, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mTp, t.fwd_only ? t.AT : t.Tp, nch * 64, 64, 64, 64);      // not stored in a forward-only call
    rc |= t.nseg > 1 ? make_map_bf16(&mP, t.Pn, nch * 128, 128, 64, 128) : (mP = mE, 0);      // the split scans' alone
    rc |= t.nseg > 1 && !t.fwd_only ? make_map_bf16(&mRm, t.RmT, nch * 128, 64, 64, 128) : (mRm = mWT, 0);
    if (rc) return KDA_ERR_CUDA;
    auto kern = conv != nullptr ? (gbf16 ? tc_intra_fwd_kernel<true, true> : tc_intra_fwd_kernel<false, true>)
                                : (gbf16 ? tc_intra_fwd_kernel<true, false> : tc_intra_fwd_kernel<false, false>);
    if (set_smem_limit(kern, kIntraFwdSmem)) return KDA_ERR_CUDA;
    KDA_LAUNCH("tc_intra_fwd_kernel", st, kern<<<(unsigned)nch, kNT, kIntraFwdSmem, st>>>(mv, mUT, mWT, mAT, mMt, mE, mP, mRm, mTp, mR, a));
    return launch_status();
}

}  // namespace kda
