// Chunked KDA forward and backward in float32 on the CUDA cores ("fp32 lane").
//
// General shapes: any K, V <= 256, any sequence length, packed sequences, initial / final state.  Every matrix of the
// chunked WY algebra is handled as 64x64 float32 tiles staged in shared memory; rows beyond a ragged chunk tail and
// columns beyond K / V are zero, which makes them inert in every product.
//
// Per chunk (64 tokens of one sequence and head), H = incoming state [K,V]:
//   G = cumsum(g);  A = tril(sum_d qn kn rho);  M = beta * stril(sum_d kn kn rho), rho = exp(G_i - G_s)
//   T = (I + M)^-1;  U = T (beta v);  W = T (beta exp(G) kn);  Z = U - W H
//   O = R H + A Z, R = qn exp(G);  H' = exp(G_end) H + E^T Z, E = kn exp(G_end - G)
// Substituting Z, the recurrence is affine in H with coefficients that do not depend on it:
//   H' = exp(G_end) . H - (E^T W) H + E^T U        dH = exp(G_end) . dH' - (E^T W)^T dH' + (R - A W)^T dO
// so everything but one K x K product per step is formed for all chunks side by side, and the scans carry a quarter of
// the work they would with Z inside: at K = V = 64 and 32 chunks 303 + 533 us became 36 + 36.
// Each kernel but the first of a pass may start while the one before it runs and waits for its end (starts_early).
// The equations restate reference chunk_wy_forward.cu:125-405, 761-858, 940-1275, 1498-1588
// and, for the adjoints, chunk_wy_backward.cu:2445-2562, 2818-3331, 3337-3552, 3787-3894.
//
// Products are 64^3 tiles on 256 threads, 4 x 4 outputs each: two 16-byte shared loads per 16 multiply-adds, both of them
// broadcast or conflict-free, so a tile is bound by the float32 pipe.  The left operand is stored with the contraction
// index leading ("At"), the right one naturally.

#include <cstdlib>

#include "common.cuh"
#include "simt_ws.cuh"
#include "tc_ws.cuh"

namespace kda {
namespace simt {

constexpr int kTile = 64 * kLD;      // floats of one shared tile

// ---------------------------------------------------------------------------------------------
// tile helpers (256 threads)
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ void ld_nat(float* dst, const float* __restrict__ src, size_t ld) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int idx = threadIdx.x + 256 * it, r = idx >> 4, c4 = (idx & 15) << 2;
        *reinterpret_cast<float4*>(dst + r * kLD + c4) = *reinterpret_cast<const float4*>(src + (size_t)r * ld + c4);
    }
}
// transposed: lanes run down the rows, so the four scalar stores of a lane are conflict-free (the 64-byte pieces of a row
// that a warp leaves behind are served by L1 in the next iterations)
__device__ __forceinline__ void ld_tr(float* dst, const float* __restrict__ src, size_t ld) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int idx = threadIdx.x + 256 * it, r = idx & 63, c4 = (idx >> 6) << 2;
        const float4 x = *reinterpret_cast<const float4*>(src + (size_t)r * ld + c4);
        dst[(c4 + 0) * kLD + r] = x.x;
        dst[(c4 + 1) * kLD + r] = x.y;
        dst[(c4 + 2) * kLD + r] = x.z;
        dst[(c4 + 3) * kLD + r] = x.w;
    }
}
// the same two as asynchronous copies: commit with cpa_commit, then cpa_wait and a barrier
__device__ __forceinline__ void cpa_nat(float* dst, const float* __restrict__ src, size_t ld) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int idx = threadIdx.x + 256 * it, r = idx >> 4, c4 = (idx & 15) << 2;
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + (r * kLD + c4) * 4), "l"(src + (size_t)r * ld + c4) : "memory");
    }
}
// transposed, element by element: a warp takes 4 rows x 8 columns, whole 32-byte sectors and 32 different banks
__device__ __forceinline__ void cpa_tr(float* dst, const float* __restrict__ src, size_t ld) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int warp = threadIdx.x >> 5, r0 = threadIdx.x & 3, q0 = (threadIdx.x & 31) >> 2;
#pragma unroll
    for (int it = 0; it < 16; ++it) {
        const int r = 4 * it + r0, c = 8 * warp + q0;
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d + (c * kLD + r) * 4), "l"(src + (size_t)r * ld + c) : "memory");
    }
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cpa_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }
// four adjacent elements of a caller tensor, zero outside nr x nc; vec: the tensor allows 4-element accesses
__device__ __forceinline__ void ld4_io(float (&x)[4], const void* base, int bf16, size_t off, size_t stride, int r, int c4, int nr, int nc, int vec) {
    const size_t i = off + (size_t)r * stride + c4;
    if (r >= nr || c4 >= nc) {
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = 0.f;
    } else if (vec && c4 + 4 <= nc) {
        if (bf16) {
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(base) + i));
            const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
            const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
            x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
        } else {
            const float4 f = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(base) + i));
            x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
        }
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) x[e] = c4 + e < nc ? ld_io(base, i + e, bf16) : 0.f;
    }
}
// 64x64 tile of a caller tensor, each element times scale[row] when scale is given
template <bool TR>
__device__ __forceinline__ void ld_tile_io(float* dst, const void* base, int bf16, size_t off, size_t stride, int nr, int nc, int vec,
                                           const float* scale = nullptr) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
        const int idx = threadIdx.x + 256 * it;
        const int r = TR ? idx & 63 : idx >> 4, c4 = (TR ? idx >> 6 : idx & 15) << 2;
        float x[4];
        ld4_io(x, base, bf16, off, stride, r, c4, nr, nc, vec);
        const float s = scale ? scale[r] : 1.f;
        if (TR) {
#pragma unroll
            for (int e = 0; e < 4; ++e) dst[(c4 + e) * kLD + r] = x[e] * s;
        } else {
            *reinterpret_cast<float4*>(dst + r * kLD + c4) = make_float4(x[0] * s, x[1] * s, x[2] * s, x[3] * s);
        }
    }
}

__device__ __forceinline__ void zero_acc(float (&acc)[4][4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.0f;
}
// The patch as column pairs: 8 packed multiply-adds a step where scalar ones are 16, which leaves issue slots to the loads
// (local backward 186 -> 155 us, scan 35 -> 33 us at 384 chunk-heads and K = V = 64; the float32 pipe's rate is the same).
__device__ __forceinline__ void to_pairs(f2 (&p)[4][2], const float (&acc)[4][4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) p[r][c] = f2_make(acc[r][2 * c], acc[r][2 * c + 1]);
}
__device__ __forceinline__ void from_pairs(float (&acc)[4][4], const f2 (&p)[4][2]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const float2 v = f2_get(p[r][c]);
            acc[r][2 * c] = v.x;
            acc[r][2 * c + 1] = v.y;
        }
}
__device__ __forceinline__ void fma_pairs(f2 (&p)[4][2], const float4& a, const float4& b) {
    const f2 b0 = f2_make(b.x, b.y), b1 = f2_make(b.z, b.w);
    const float ar[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const f2 ad = f2_all(ar[r]);
        p[r][0] = f2_fma(ad, b0, p[r][0]);
        p[r][1] = f2_fma(ad, b1, p[r][1]);
    }
}
// acc[r][c] += sum_{kk < n} ap[kk * lda + r] * bp[kk * ldb + c]: ap, bp already at the thread's rows / columns
__device__ __forceinline__ void mm_at(float (&acc)[4][4], const float* ap, int lda, const float* bp, int ldb, int n) {
    f2 p[4][2];
    to_pairs(p, acc);
#pragma unroll 8
    for (int kk = 0; kk < n; ++kk)
        fma_pairs(p, *reinterpret_cast<const float4*>(ap + kk * lda), *reinterpret_cast<const float4*>(bp + kk * ldb));
    from_pairs(acc, p);
}
__device__ __forceinline__ void mm64(float (&acc)[4][4], const float* At, const float* Bs) {
    mm_at(acc, At + 4 * (threadIdx.x >> 4), kLD, Bs + 4 * (threadIdx.x & 15), kLD, 64);
}

// the thread's 4x4 patch -> shared or global rows, naturally or transposed (16-byte stores either way)
__device__ __forceinline__ void st_nat(float* dst, size_t ld, const float (&acc)[4][4]) {
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll
    for (int r = 0; r < 4; ++r)
        *reinterpret_cast<float4*>(dst + (size_t)(4 * ty + r) * ld + 4 * tx) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
}
__device__ __forceinline__ void st_tr(float* dst, size_t ld, const float (&acc)[4][4]) {
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll
    for (int c = 0; c < 4; ++c)
        *reinterpret_cast<float4*>(dst + (size_t)(4 * tx + c) * ld + 4 * ty) = make_float4(acc[0][c], acc[1][c], acc[2][c], acc[3][c]);
}
__device__ __forceinline__ void ld_patch(float (&x)[4][4], const float* src, size_t ld) {
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float4 f = *reinterpret_cast<const float4*>(src + (size_t)(4 * ty + r) * ld + 4 * tx);
        x[r][0] = f.x; x[r][1] = f.y; x[r][2] = f.z; x[r][3] = f.w;
    }
}
// sum over the 16 lanes that share a patch row
__device__ __forceinline__ float row_sum16(float x) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// ---------------------------------------------------------------------------------------------
// chunk table of a packed batch (or of one without tokens): which tokens each 64-token chunk slot covers
// ---------------------------------------------------------------------------------------------
// A packed batch is described by cu_seqlens, which the caller controls: every segment is checked against the token
// count and the slot budget before it enters the tables, so that no later kernel can be steered outside the tensors.
// A segment that starts before the previous one ends, has a negative length or reaches past `tokens` is treated as
// empty; chunks beyond the slot budget are dropped; either raises the status word (kStatusBadCuSeqlens), as does a
// table that does not start at 0 or does not end at `tokens`.
constexpr int kStatusBadCuSeqlens = 10;
constexpr int kTableThreads = 512;
constexpr int kScanOrderMax = kTableThreads;      // batches up to this many sequences get a longest-first scan order

// One block; every packed forward waits for it, so what counts is the length of its chains.  The check of a segment against the one
// before it is a chain through all of them only when one is wrong: a table that never falls, starts at 0 or later and stays within
// `tokens` passes segment by segment, its chunks fit the slot budget (tokens / 64 + n_seq, sh.seq_len being 0 here), and their places are
// a prefix sum.  Then a thread a slot finds its sequence by bisection.  Whole forwards in us, one thread
// and a thread a sequence / this: 512 sequences of 32 tokens, 2 heads 170 / 139, 1,024 of 16 283 / 230, 4,096 of 16 639 / 442; 22 long
// ones of 65,536 tokens, 1 head 127 / 125.
__global__ void __launch_bounds__(kTableThreads) chunk_table_kernel(Ws w, const int32_t* __restrict__ cu, int n_seq, int tokens, int* status, int* mirror) {
    const ChunkTable& t = w.tab;
    __shared__ __align__(16) int first[kTableThreads + 4];      // first chunk slot of each sequence of the tile, and the end
    __shared__ int tok[kTableThreads], len[kTableThreads], warp_sum[kTableThreads / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    bool good = true;
    if (cu)
        for (int s = tid; s < n_seq; s += kTableThreads) {
            const int t0 = cu[s], t1 = cu[s + 1];
            good = good && t0 <= t1 && t1 <= tokens && (s > 0 || t0 >= 0);
        }
    good = __syncthreads_and(good);
    if (tid == 0) {
        int flag = 0, prev_end = 0;
        if (good) {
            if (cu && n_seq > 0) prev_end = cu[n_seq];
        } else {
            int acc = 0;
            for (int s = 0; s < n_seq; ++s) {
                t.seq_chunk0[s] = acc;
                const int t0 = cu[s], t1 = cu[s + 1];
                int n = t1 - t0;
                if (t0 < prev_end || n < 0 || t1 > tokens) { n = 0; flag = 1; }
                else prev_end = t1;
                int nc = (n + kChunk - 1) / kChunk;
                if (acc + nc > w.nslots) { nc = w.nslots - acc; flag = 1; }
                acc += nc;
            }
            t.seq_chunk0[n_seq] = acc;
        }
        if (cu && (cu[0] != 0 || prev_end != tokens)) flag = 1;
        start_status(status, mirror);
        if (flag) raise_status(status, kStatusBadCuSeqlens);
    }
    if (!good) __syncthreads();
    int base = 0;
    for (int s0 = 0; s0 < n_seq; s0 += kTableThreads) {
        const int s = s0 + tid;
        int t0 = 0, n = 0, nc = 0;
        if (s < n_seq) {
            if (cu) {
                t0 = cu[s];
                n = cu[s + 1] - t0;
            }
            nc = good ? (n + kChunk - 1) / kChunk : t.seq_chunk0[s + 1] - t.seq_chunk0[s];
        }
        int x = nc;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sum[warp] = x;
        __syncthreads();
        int end = base, at = base + x - nc;
#pragma unroll
        for (int i = 0; i < kTableThreads / 32; ++i) {
            const int y = warp_sum[i];
            if (i < warp) at += y;
            end += y;
        }
        first[tid] = at;
        if (tid == 0) first[kTableThreads] = end;
        tok[tid] = t0;
        len[tid] = n;
        if (good && s < n_seq) t.seq_chunk0[s] = at;
        __syncthreads();
        for (int c = base + tid; c < end; c += kTableThreads) {
            int i = 0;      // the last sequence that starts at or before slot c: the ones after it that are empty start later
#pragma unroll
            for (int b = kTableThreads / 2; b > 0; b >>= 1)
                if (first[i + b] <= c) i += b;
            const int j = (c - first[i]) * kChunk;
            t.seq[c] = s0 + i;
            t.tok0[c] = tok[i] + j;
            t.len[c] = min(kChunk, len[i] - j);
        }
        // Scan order: starting the longest chains first keeps the tail of a launch short (longest-processing-time-first).  Rank by
        // counting; identity for large batches, which balance by themselves.
        if (s < n_seq) {
            int rank = s;
            if (n_seq <= kScanOrderMax) {
                rank = 0;
                int f = first[0];
                for (int j = 0; j < n_seq; ++j) {
                    const int g = first[j + 1];
                    rank += (g - f) + (j < s ? 1 : 0) > nc ? 1 : 0;
                    f = g;
                }
            }
            t.seq_order[rank] = s;
        }
        base = end;
        __syncthreads();
    }
    if (good && tid == 0) t.seq_chunk0[n_seq] = base;
    for (int c = base + tid; c < w.nslots; c += kTableThreads) {
        t.seq[c] = -1;
        t.tok0[c] = 0;
        t.len[c] = 0;
    }
}

// ---------------------------------------------------------------------------------------------
// T = (I + M)^-1
// ---------------------------------------------------------------------------------------------
// dst = alpha * A * B for NP independent S x S problems (row-major, leading dimension kLD): a thread owns CW adjacent
// columns of one row
template <int S, int NP, class PA, class PB, class PD>
__device__ __forceinline__ void merge_mm(PA pa, PB pb, PD pd, float alpha) {
    constexpr int CW = S * S * NP / 256, TPR = S / CW;      // 1 (8x8x4), 2 (16x16x2), 4 (32x32x1)
    const int prob = threadIdx.x / (S * TPR), rem = threadIdx.x % (S * TPR);
    const int i = rem / TPR, j0 = (rem % TPR) * CW;
    const float* A = pa(prob) + i * kLD;
    const float* B = pb(prob) + j0;
    float acc[CW];
#pragma unroll
    for (int c = 0; c < CW; ++c) acc[c] = 0.f;
#pragma unroll
    for (int t = 0; t < S; ++t) {
        const float a = A[t];
#pragma unroll
        for (int c = 0; c < CW; ++c) acc[c] += a * B[t * kLD + c];
    }
    float* D = pd(prob) + i * kLD + j0;
#pragma unroll
    for (int c = 0; c < CW; ++c) D[c] = alpha * acc[c];
}

// Ts = (I + Ms)^-1 for strictly lower-triangular Ms: 8x8 diagonal solves, then merges to 16, 32 and 64 with
//   inv([[A,0],[C,B]]) = [[Ai,0],[-Bi C Ai, Bi]];  tmp: 32 rows
__device__ void unit_lower_inverse(const float* Ms, float* Ts, float* tmp) {
    const int tid = threadIdx.x;
    for (int idx = tid; idx < kTile / 4; idx += 256) reinterpret_cast<float4*>(Ts)[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    if (tid < 64) {
        const int b = tid >> 3, j = tid & 7;
        const float* Lb = Ms + (8 * b) * kLD + 8 * b;
        float x[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) x[i] = (i == j) ? 1.f : 0.f;
#pragma unroll
        for (int i = 1; i < 8; ++i) {
            float s = 0.f;
#pragma unroll
            for (int t = 0; t < i; ++t) s += Lb[i * kLD + t] * x[t];
            x[i] = (i > j) ? -s : x[i];
        }
        float* Tb = Ts + (8 * b) * kLD + 8 * b;
#pragma unroll
        for (int i = 0; i < 8; ++i) Tb[i * kLD + j] = x[i];
    }
    __syncthreads();
    merge_mm<8, 4>([&](int p) { return Ms + (16 * p + 8) * kLD + 16 * p; }, [&](int p) { return Ts + (16 * p) * kLD + 16 * p; },
                   [&](int p) { return tmp + p * 8 * kLD; }, 1.f);
    __syncthreads();
    merge_mm<8, 4>([&](int p) { return Ts + (16 * p + 8) * kLD + 16 * p + 8; }, [&](int p) { return tmp + p * 8 * kLD; },
                   [&](int p) { return Ts + (16 * p + 8) * kLD + 16 * p; }, -1.f);
    __syncthreads();
    merge_mm<16, 2>([&](int p) { return Ms + (32 * p + 16) * kLD + 32 * p; }, [&](int p) { return Ts + (32 * p) * kLD + 32 * p; },
                    [&](int p) { return tmp + p * 16 * kLD; }, 1.f);
    __syncthreads();
    merge_mm<16, 2>([&](int p) { return Ts + (32 * p + 16) * kLD + 32 * p + 16; }, [&](int p) { return tmp + p * 16 * kLD; },
                    [&](int p) { return Ts + (32 * p + 16) * kLD + 32 * p; }, -1.f);
    __syncthreads();
    merge_mm<32, 1>([&](int) { return Ms + 32 * kLD; }, [&](int) { return Ts; }, [&](int) { return tmp; }, 1.f);
    __syncthreads();
    merge_mm<32, 1>([&](int) { return Ts + 32 * kLD + 32; }, [&](int) { return tmp; }, [&](int) { return Ts + 32 * kLD; }, -1.f);
    __syncthreads();
}

// ---------------------------------------------------------------------------------------------
// decay factors of the masked products
// ---------------------------------------------------------------------------------------------
// rho(i, s) = exp(G_i - G_s) is taken apart per 16-row target block I around the reference c_I = G at the block's row 8:
//   targets  x~_i = x_i exp(G_i - c_I)        sources for block I  k_s exp(c_I - G_s), s < 16 (I + 1)
// so that the masked products are plain tile products.  Within the block both exponents are at most eight tokens' decay
// (40 at the gate's lowest), for earlier sources the factor only shrinks.  The blocks' sums are kept apart from the prefix
// (L, counted from the block's first row), so a factor's exponent is rounded at its own size, not at G's.  A chunk whose
// decay exceeds kMaxExponent inside a block takes the pairwise exponentials instead (log-decays below -5.5 per token).  The
// line lies just above the gate's 40: sums of cotangents times a source's factor are formed before the target's factor
// brings them down, and from e^44 = 1e19 they have another 1e19 to float32's end (from e^80, 6e3: gradients of 1e4 overflowed).
constexpr float kMaxExponent = 44.f;
constexpr int kSrcCols = 16 + 32 + 48 + 64;
// source array of block I in the forward: [32 d][16 (I + 1)] with 4 floats of padding, after the two target stacks
constexpr int kHalf = 32;
__device__ __forceinline__ int src_ld(int I) { return 16 * (I + 1) + 4; }
__device__ __forceinline__ int src_off(int I) { return kHalf * (8 * I * (I + 1) + 4 * I); }
constexpr int kSrcFloats = kHalf * (kSrcCols + 16);

// ---------------------------------------------------------------------------------------------
// K1  chunk-parallel part of the forward, one CTA per (chunk, head): norms, decay, A, T, W, U and the scan's coefficients
// ---------------------------------------------------------------------------------------------
struct IntraArgs {
    const void *q, *k, *v, *g, *beta;
    int bf16, gbf16, l2norm, vec_v, backward;
    float scale;
    int* mirror;
    int clear_status;      // no table kernel ran before this one
};
// 46 KB and at most 80 registers, so that three CTAs share an SM: the kernel alternates between loads, short products and
// barriers, and two CTAs (64-wide factor tiles, 83 KB) left the issue slots 60 % idle.
constexpr int kIntraFloats = 160 * kLD;                   // factor stacks of 32 channels, later M, T and 32 rows of scratch
static_assert(kIntraFloats >= 2 * kHalf * kLD + kSrcFloats, "factor stacks do not fit");
constexpr size_t kIntraSmem = (kIntraFloats + 64 * 3 + 8 * kHalf + 4 * kHalf) * sizeof(float);

__global__ void __launch_bounds__(256, 3) intra_fwd_kernel(Ws w, IntraArgs p) {
    extern __shared__ __align__(16) float sm[];
    dependents_go();
    float* tq = sm;                      // [d][i] q~
    float* tk = tq + kHalf * kLD;        // [d][i] k~
    float* src = tk + kHalf * kLD;       // four source arrays
    float* qi_s = sm + kIntraFloats;     // [64] inverse norms, beta
    float* ki_s = qi_s + 64;
    float* bet = ki_s + 64;
    float* bsum = bet + 64;              // [8][32] sums of g over 8 rows
    float* cref = bsum + 8 * kHalf;      // [4][32] G at row 8 of each block
    const int slot = blockIdx.x, h = blockIdx.y;
    if (p.clear_status && slot == 0 && h == 0 && threadIdx.x == 0) start_status(w.status, p.mirror);
    int len, tok0;
    w.tab.span(slot, tok0, len);
    if (len == 0) return;
    const int K = w.K, Kp = w.Kp, V = w.V, Vp = w.Vp, H = w.H, KT = Kp / 64, VT = Vp / 64;
    const size_t ch = (size_t)slot * H + h;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

    for (int i = warp; i < 64; i += 8) {
        float qi = 0.f, ki = 0.f, b = 0.f;
        if (i < len) {
            const size_t off = ((size_t)(tok0 + i) * H + h) * K;
            float sq = 0.f, sk = 0.f;
            for (int d = lane; d < K; d += 32) {
                const float x = ld_io(p.q, off + d, p.bf16), y = ld_io(p.k, off + d, p.bf16);
                sq += x * x;
                sk += y * y;
            }
            sq = warp_sum(sq);
            sk = warp_sum(sk);
            qi = p.l2norm ? 1.0f / fmaxf(sqrtf(sq), 1e-12f) : 1.0f;
            ki = p.l2norm ? 1.0f / fmaxf(sqrtf(sk), 1e-12f) : 1.0f;
            b = ld_io(p.beta, (size_t)(tok0 + i) * H + h, p.gbf16);
        }
        if (lane == 0) {
            qi_s[i] = qi;
            ki_s[i] = ki;
            bet[i] = b;
            w.qinv[ch * 64 + i] = qi;
            w.kinv[ch * 64 + i] = ki;
            w.beta[ch * 64 + i] = b;
        }
    }
    float* kn_g = w.kn + ch * 64 * Kp;
    float* G_g = w.G + ch * 64 * Kp;

    // ---- A and M: 320 4x4 tiles of [q~; k~] (32 rows per target block) x sources over 256 threads
    const int t1 = tid < 32 ? 0 : (tid < 96 ? 1 : (tid < 192 ? 2 : 3));
    const int b1 = t1 == 0 ? 0 : (t1 == 1 ? 32 : (t1 == 2 ? 96 : 192));
    const int r1 = (tid - b1) / (4 * (t1 + 1)), c1 = (tid - b1) % (4 * (t1 + 1));      // row tile (0-3 q, 4-7 k), source tile
    const int r2 = (tid + 64) / 16, c2 = (tid + 64) % 16;                              // second tile of threads 0..63: block 3
    float acc1[4][4], acc2[4][4];
    zero_acc(acc1);
    zero_acc(acc2);
    const int I = warp >> 1, i0 = 8 * warp;    // element-wise: channel `lane` of 32, rows i0 .. i0 + 7 of block I
    for (int dt = 0; dt < 2 * KT; ++dt) {
        const int dd = dt * kHalf + lane;
        const bool in = dd < K;
        const size_t col = ((size_t)tok0 * H + h) * K + (in ? dd : 0), rstep = (size_t)H * K;
        float L[8];
        {
            float run = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) L[r] = (i0 + r < len && in) ? ld_io(p.g, col + (size_t)(i0 + r) * rstep, p.gbf16) : 0.f;
            const float first = L[0];
#pragma unroll
            for (int r = 0; r < 8; ++r) L[r] = run += L[r];
            __syncthreads();                   // norms on the first round; the previous round's stacks are free
            bsum[warp * kHalf + lane] = run;
            if (warp & 1) cref[I * kHalf + lane] = first;      // g of row 8, completed below
        }
        __syncthreads();
        float pre = 0.f;
        for (int J = 0; J < 2 * I; ++J) pre += bsum[J * kHalf + lane];
        const float half = bsum[2 * I * kHalf + lane], c = half + cref[I * kHalf + lane];      // L of the block's row 8
        if (warp & 1) {
#pragma unroll
            for (int r = 0; r < 8; ++r) L[r] += half;
        }
        bool far = false;
#pragma unroll
        for (int r = 0; r < 8; ++r) far = far || !(fabsf(L[r] - c) <= kMaxExponent);
        const bool pairwise = __syncthreads_or(far);           // every warp has read the block sums and the rows' g
        if (!(warp & 1)) cref[I * kHalf + lane] = pre + c;
        {
            // e^{G_end - G} from the rows' own sum to the chunk's end: G_end and G are both as large as the chunk's whole decay
            // (300 at the gate's lowest), and their difference keeps that size's rounding, 1e-5 of the last tokens' weight in
            // the state.  g once more (L1): eight registers to hold it would cost the third CTA.
            float run = 0.f;
            for (int J = 7; J > warp; --J) run += bsum[J * kHalf + lane];
            float* ed = w.Ed + (ch * 64 + i0) * Kp + dd;
#pragma unroll
            for (int r = 7; r >= 0; --r) {
                ed[(size_t)r * Kp] = expf(run);
                run += (i0 + r < len && in) ? ld_io(p.g, col + (size_t)(i0 + r) * rstep, p.gbf16) : 0.f;
            }
        }
        __syncthreads();
        float kn[8];
        float* rt = w.RT + (ch * Kp + dd) * 64 + i0;           // R^T: 8 rows of this channel
#pragma unroll
        for (int r4 = 0; r4 < 2; ++r4) {
            float R[4], q[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = 4 * r4 + e, i = i0 + r;
                const bool ok = i < len && in;
                const float qn = ok ? ld_io(p.q, col + (size_t)i * rstep, p.bf16) * qi_s[i] * p.scale : 0.f;
                kn[r] = ok ? ld_io(p.k, col + (size_t)i * rstep, p.bf16) * ki_s[i] : 0.f;
                const float G = pre + L[r];
                kn_g[(size_t)i * Kp + dd] = kn[r];
                G_g[(size_t)i * Kp + dd] = G;
                if (p.backward) w.qn[(ch * 64 + i) * Kp + dd] = qn;
                R[e] = qn * expf(G);
                q[e] = pairwise ? qn : qn * expf(L[r] - c);
            }
            *reinterpret_cast<float4*>(rt + 4 * r4) = make_float4(R[0], R[1], R[2], R[3]);
            *reinterpret_cast<float4*>(tq + lane * kLD + i0 + 4 * r4) = make_float4(q[0], q[1], q[2], q[3]);
        }
        if (!pairwise) {
            float e[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) e[r] = kn[r] * expf(L[r] - c);
            *reinterpret_cast<float4*>(tk + lane * kLD + i0) = make_float4(e[0], e[1], e[2], e[3]);
            *reinterpret_cast<float4*>(tk + lane * kLD + i0 + 4) = make_float4(e[4], e[5], e[6], e[7]);
#pragma unroll
            for (int r = 0; r < 8; ++r) e[r] = kn[r] * expf(c - L[r]);
            for (int T = I; T < 4; ++T) {
                const float f = T == I ? 1.f : expf(cref[T * kHalf + lane] - cref[I * kHalf + lane]);
                float* s = src + src_off(T) + lane * src_ld(T) + i0;
                *reinterpret_cast<float4*>(s) = make_float4(e[0] * f, e[1] * f, e[2] * f, e[3] * f);
                *reinterpret_cast<float4*>(s + 4) = make_float4(e[4] * f, e[5] * f, e[6] * f, e[7] * f);
            }
            __syncthreads();
            mm_at(acc1, (r1 < 4 ? tq : tk) + 16 * t1 + 4 * (r1 & 3), kLD, src + src_off(t1) + 4 * c1, src_ld(t1), kHalf);
            if (tid < 64) mm_at(acc2, (r2 < 4 ? tq : tk) + 48 + 4 * (r2 & 3), kLD, src + src_off(3) + 4 * c2, src_ld(3), kHalf);
        } else {
            float* Gs = src;                   // plain q, k, G columns
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                tk[lane * kLD + i0 + r] = kn[r];
                Gs[lane * kLD + i0 + r] = pre + L[r];
            }
            __syncthreads();
            auto pairs = [&](float (&acc)[4][4], int T, int rt4, int ct) {
                const float* x = (rt4 < 4 ? tq : tk);
                for (int r = 0; r < 4; ++r)
                    for (int s4 = 0; s4 < 4; ++s4) {
                        const int i = 16 * T + 4 * (rt4 & 3) + r, s = 4 * ct + s4;
                        if (s > i) continue;
                        float a = 0.f;
                        for (int e = 0; e < kHalf; ++e) a += x[e * kLD + i] * tk[e * kLD + s] * expf(Gs[e * kLD + i] - Gs[e * kLD + s]);
#pragma unroll
                        for (int rr = 0; rr < 4; ++rr)
#pragma unroll
                            for (int ss = 0; ss < 4; ++ss)
                                if (rr == r && ss == s4) acc[rr][ss] += a;
                    }
            };
            pairs(acc1, t1, r1, c1);
            if (tid < 64) pairs(acc2, 3, r2, c2);
        }
    }
    __syncthreads();
    // ---- A out (both orientations), M and its inverse
    float* Ms = sm;
    float* Ts = Ms + kTile;
    float* tmp = Ts + kTile;             // 32 rows
    float* TT = Ms;                      // [s][i] = T[i][s], once M is done with
    float* op = Ts;                      // operand tile, once T is out
    for (int idx = tid; idx < 2 * kTile / 4; idx += 256) reinterpret_cast<float4*>(sm)[idx] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    auto place = [&](const float (&acc)[4][4], int T, int rt, int ct) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c4 = 0; c4 < 4; ++c4) {
                const int i = 16 * T + 4 * (rt & 3) + r, s = 4 * ct + c4;
                if (rt < 4) Ts[i * kLD + s] = s <= i ? acc[r][c4] : 0.f;      // A, until the inverse overwrites it
                else Ms[i * kLD + s] = s < i ? bet[i] * acc[r][c4] : 0.f;
            }
    };
    place(acc1, t1, r1, c1);
    if (tid < 64) place(acc2, 3, r2, c2);
    __syncthreads();
    for (int idx = tid; idx < 4096; idx += 256) {
        w.AT[ch * 4096 + idx] = Ts[(idx & 63) * kLD + (idx >> 6)];
        if (p.backward) w.A[ch * 4096 + idx] = Ts[(idx >> 6) * kLD + (idx & 63)];
    }
    __syncthreads();
    unit_lower_inverse(Ms, Ts, tmp);
    for (int idx = tid; idx < 4096; idx += 256) {
        const int r = idx >> 6, c = idx & 63;
        TT[r * kLD + c] = Ts[c * kLD + r];
        if (p.backward) w.T[ch * 4096 + idx] = Ts[r * kLD + c];
    }
    // ---- W = T (beta e^G k), U = T (beta v)
    float acc[4][4];
    float* W_g = w.W + ch * 64 * Kp;
    float* Z_g = w.Z + ch * 64 * Vp;
    for (int kt = 0; kt < KT; ++kt) {
        __syncthreads();
        for (int idx = tid; idx < 1024; idx += 256) {
            const int r = idx >> 4, c4 = (idx & 15) << 2;
            const float4 k4 = *reinterpret_cast<const float4*>(kn_g + (size_t)r * Kp + kt * 64 + c4);
            const float4 g4 = *reinterpret_cast<const float4*>(G_g + (size_t)r * Kp + kt * 64 + c4);
            const float b = bet[r];
            *reinterpret_cast<float4*>(op + r * kLD + c4) =
                make_float4(b * expf(g4.x) * k4.x, b * expf(g4.y) * k4.y, b * expf(g4.z) * k4.z, b * expf(g4.w) * k4.w);
        }
        __syncthreads();
        zero_acc(acc);
        mm64(acc, TT, op);
        st_nat(W_g + kt * 64, Kp, acc);
        st_tr(w.WT + (ch * Kp + kt * 64) * 64, 64, acc);
    }
    for (int vt = 0; vt < VT; ++vt) {
        __syncthreads();
        ld_tile_io<false>(op, p.v, p.bf16, ((size_t)tok0 * H + h) * V + vt * 64, (size_t)H * V, len, V - vt * 64, p.vec_v, bet);
        __syncthreads();
        zero_acc(acc);
        mm64(acc, TT, op);
        st_nat(Z_g + vt * 64, Vp, acc);
    }
    // ---- the scan's coefficients: E^T W, E^T U, exp(G_end);  Rm = R - A W for the adjoint scan
    float* Es = sm;                      // [s][k]
    float* Xs = sm + kTile;
    const float* ge = G_g + (size_t)63 * Kp;
    for (int kt = 0; kt < KT; ++kt) {
        __syncthreads();
        for (int idx = tid; idx < 1024; idx += 256) {
            const int r = idx >> 4, c4 = (idx & 15) << 2;
            const float4 k4 = *reinterpret_cast<const float4*>(kn_g + (size_t)r * Kp + kt * 64 + c4);
            const float4 e4 = *reinterpret_cast<const float4*>(w.Ed + (ch * 64 + r) * Kp + kt * 64 + c4);
            *reinterpret_cast<float4*>(Es + r * kLD + c4) = make_float4(k4.x * e4.x, k4.y * e4.y, k4.z * e4.z, k4.w * e4.w);
        }
        if (tid < 64) w.dec[ch * Kp + kt * 64 + tid] = expf(ge[kt * 64 + tid]);
        for (int k2 = 0; k2 < KT; ++k2) {
            __syncthreads();
            ld_nat(Xs, W_g + k2 * 64, Kp);
            __syncthreads();
            zero_acc(acc);
            mm64(acc, Xs, Es);           // [k'][k] = sum_s W[s][k'] E[s][k]
            st_nat(w.PT + (ch * Kp + k2 * 64) * Kp + kt * 64, Kp, acc);
            if (p.backward) st_tr(w.P + (ch * Kp + kt * 64) * Kp + k2 * 64, Kp, acc);
        }
        for (int vt = 0; vt < VT; ++vt) {
            __syncthreads();
            ld_nat(Xs, Z_g + vt * 64, Vp);
            __syncthreads();
            zero_acc(acc);
            mm64(acc, Es, Xs);
            st_nat(w.Hc + (ch * Kp + kt * 64) * Vp + vt * 64, Vp, acc);
        }
    }
    if (p.backward) {
        __syncthreads();
        ld_nat(Es, w.AT + ch * 4096, 64);
        for (int kt = 0; kt < KT; ++kt) {
            __syncthreads();
            ld_nat(Xs, W_g + kt * 64, Kp);
            __syncthreads();
            zero_acc(acc);
            mm64(acc, Es, Xs);           // A W
            float qv[4][4], gv[4][4];
            ld_patch(qv, w.qn + ch * 64 * Kp + kt * 64, Kp);
            ld_patch(gv, G_g + kt * 64, Kp);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int c4 = 0; c4 < 4; ++c4) acc[r][c4] = qv[r][c4] * expf(gv[r][c4]) - acc[r][c4];
            st_nat(w.Rm + ch * 64 * Kp + kt * 64, Kp, acc);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// K2  state scan over the chunks of one (sequence, head, 16-column value strip), in either direction:
//     forward  S = H:   S' = dec . S + B - P S       B = E^T U, leaves the chunk-start states in its place
//     backward S = dH': S' = dec . S + B - P^T S     B = Rm^T dO, leaves the adjoints of the outgoing states
// A step is one Kp x Kp product against a 16-column strip.  What a step reads (its matrix as 64x64 tiles, its strip of B,
// its decay) comes through a ring filled by asynchronous copies three tiles ahead; four groups of two warps share the
// contraction and meet in shared memory, laid out so that no access of the step has a bank conflict.  The strip lives in
// registers (thread = row x 4 columns) and, for the products, in shared memory.  1.9 us a step at K = 64 while B was loaded
// one step ahead into registers and the partial sums conflicted; 1.1 now, a chain of four barriers and 16 x 18 instructions.
// ---------------------------------------------------------------------------------------------
constexpr int kVS = 16, kScanStages = 4;
constexpr int kStageFloats = 4096 + 64 * kVS + 64;      // tile, strip of B, decay of one 64-row block
constexpr int kSLD = 20;                                // row stride of the shared strip
constexpr int kPartBlock = 72;                          // float4s per (group, column quad): row 4 l + r at r * 18 + l

struct ScanArgs {
    const float* M;       // [ch][Kp][Kp], contraction index leading: P^T forward, P backward
    float* B;             // [ch][Kp][Vp]
    const float* s_in;    // [n_seq][H][V][K] or null
    float* s_out;
    int backward;
};
inline size_t scan_smem(int Kp) { return (size_t)(kScanStages * kStageFloats + 16 * kPartBlock * 4 + Kp * kSLD) * sizeof(float); }

template <int KT>
__global__ void __launch_bounds__(256) scan_kernel(Ws w, ScanArgs p) {
    extern __shared__ __align__(16) float sm[];
    dependents_go();
    dependency_wait();
    float* ring = sm;
    float4* part = reinterpret_cast<float4*>(ring + kScanStages * kStageFloats);
    float* S = reinterpret_cast<float*>(part + 16 * kPartBlock);      // [Kp][kSLD]
    const int Kp = 64 * KT, Vp = w.Vp, K = w.K, V = w.V, H = w.H;
    const int seq = blockIdx.x, h = blockIdx.y, v0 = blockIdx.z * kVS, tid = threadIdx.x;
    const int c0 = w.tab.first_chunk(seq), c1 = w.tab.first_chunk(seq + 1), n = c1 - c0;
    const int row = tid & 63, cq = tid >> 6;                          // the state element group this thread owns in every 64-row block
    const int l = tid & 15, pq = (tid >> 4) & 3, kg = tid >> 6;       // product: rows 4 l .., column quad, contraction group
    const int grow = tid >> 2, gc = (tid & 3) << 2;                   // global rows of 64 bytes
    auto chunk = [&](int step) { return (size_t)(p.backward ? c1 - 1 - step : c0 + step) * H + h; };
    const int tiles = n * KT * KT;
    const uint32_t ring_s = (uint32_t)__cvta_generic_to_shared(ring);
    auto cp16 = [](uint32_t dst, const float* src) { asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory"); };
    auto issue = [&](int t) {      // tile t: step, then output block, then contraction block
        if (t < tiles) {
            const int step = t / (KT * KT), rt = (t / KT) % KT, kt = t % KT;
            const size_t ch = chunk(step);
            const float* src = p.M + (ch * Kp + kt * 64) * Kp + rt * 64;
            const uint32_t dst = ring_s + (t % kScanStages) * kStageFloats * 4;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int idx = tid + 256 * i, r = idx >> 4, c = (idx & 15) << 2;
                cp16(dst + (r * 64 + c) * 4, src + (size_t)r * Kp + c);
            }
            if (kt == 0) {
                cp16(dst + (4096 + tid * 4) * 4, p.B + (ch * Kp + rt * 64 + grow) * Vp + v0 + gc);
                if (tid < 16) cp16(dst + (4096 + 64 * kVS + tid * 4) * 4, w.dec + ch * Kp + rt * 64 + tid * 4);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float4 s[KT];
#pragma unroll
    for (int rt = 0; rt < KT; ++rt) {
        s[rt] = make_float4(0.f, 0.f, 0.f, 0.f);
        const int kk = rt * 64 + row, vv = v0 + 4 * cq;
        if (p.s_in && kk < K) {
            const float* src = p.s_in + (((size_t)seq * H + h) * V + vv) * K + kk;
            if (vv + 0 < V) s[rt].x = src[0];
            if (vv + 1 < V) s[rt].y = src[K];
            if (vv + 2 < V) s[rt].z = src[2 * (size_t)K];
            if (vv + 3 < V) s[rt].w = src[3 * (size_t)K];
        }
        *reinterpret_cast<float4*>(S + kk * kSLD + 4 * cq) = s[rt];
    }
    for (int t = 0; t < kScanStages - 1; ++t) issue(t);
    int t = 0;
    for (int step = 0; step < n; ++step) {
        const size_t ch = chunk(step);
#pragma unroll
        for (int rt = 0; rt < KT; ++rt) {
            float acc[4][4];
            zero_acc(acc);
#pragma unroll
            for (int kt = 0; kt < KT; ++kt, ++t) {
                asm volatile("cp.async.wait_group %0;" ::"n"(kScanStages - 2) : "memory");
                __syncthreads();                       // tile t has landed for everyone; tile t - 1 and (rt = 0) the old partials are read out
                issue(t + kScanStages - 1);
                const float* stage = ring + (t % kScanStages) * kStageFloats;
                mm_at(acc, stage + 16 * kg * 64 + 4 * l, 64, S + (kt * 64 + 16 * kg) * kSLD + 4 * pq, kSLD, 16);
                if (kt == 0) {
                    const float* bd = stage + 4096;    // this block's strip of B and decay
                    const float4 b = *reinterpret_cast<const float4*>(bd + row * kVS + 4 * cq);
                    const float dc = bd[64 * kVS + row];
                    // the state the chunk sees takes B's place in memory (B of this block has landed), then the row's own terms
                    *reinterpret_cast<float4*>(p.B + (ch * Kp + rt * 64 + grow) * Vp + v0 + gc) = *reinterpret_cast<const float4*>(S + (rt * 64 + grow) * kSLD + gc);
                    s[rt].x = dc * s[rt].x + b.x;
                    s[rt].y = dc * s[rt].y + b.y;
                    s[rt].z = dc * s[rt].z + b.z;
                    s[rt].w = dc * s[rt].w + b.w;
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) part[(kg * 4 + pq) * kPartBlock + r * 18 + l] = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
            __syncthreads();
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                const float4 y = part[(g * 4 + cq) * kPartBlock + (row & 3) * 18 + (row >> 2)];
                s[rt].x -= y.x; s[rt].y -= y.y; s[rt].z -= y.z; s[rt].w -= y.w;
            }
        }
        if (KT > 1) __syncthreads();                   // every block's products have read the strip (one block: the barrier above)
#pragma unroll
        for (int rt = 0; rt < KT; ++rt) *reinterpret_cast<float4*>(S + (rt * 64 + row) * kSLD + 4 * cq) = s[rt];
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (p.s_out) {
#pragma unroll
        for (int rt = 0; rt < KT; ++rt) {
            const int kk = rt * 64 + row, vv = v0 + 4 * cq;
            if (kk < K) {
                float* dst = p.s_out + (((size_t)seq * H + h) * V + vv) * K + kk;
                if (vv + 0 < V) dst[0] = s[rt].x;
                if (vv + 1 < V) dst[K] = s[rt].y;
                if (vv + 2 < V) dst[2 * (size_t)K] = s[rt].z;
                if (vv + 3 < V) dst[3 * (size_t)K] = s[rt].w;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// K3  Z = U - W H, O = R H + A Z; one 64-column value tile per CTA
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) out_kernel(Ws w, void* __restrict__ o, int bf16) {
    extern __shared__ __align__(16) float sm[];
    float *Wt = sm, *Rt = sm + kTile, *Bs = sm + 2 * kTile;
    dependency_wait();
    const int slot = blockIdx.x, h = blockIdx.y, vt = blockIdx.z;
    int len, tok0;
    w.tab.span(slot, tok0, len);
    if (len == 0) return;
    const size_t ch = (size_t)slot * w.H + h;
    const int Kp = w.Kp, Vp = w.Vp;
    float az[4][4], ao[4][4];
    zero_acc(az);
    zero_acc(ao);
    for (int kt = 0; kt < Kp / 64; ++kt) {
        __syncthreads();
        ld_nat(Wt, w.WT + (ch * Kp + kt * 64) * 64, 64);
        ld_nat(Rt, w.RT + (ch * Kp + kt * 64) * 64, 64);
        ld_nat(Bs, w.Hc + (ch * Kp + kt * 64) * Vp + vt * 64, Vp);
        __syncthreads();
        mm64(az, Wt, Bs);
        mm64(ao, Rt, Bs);
    }
    __syncthreads();
    ld_nat(Wt, w.AT + ch * 4096, 64);
    float* Zg = w.Z + ch * 64 * Vp + vt * 64;
    float u[4][4];
    ld_patch(u, Zg, Vp);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) u[r][c] -= az[r][c];
    st_nat(Zg, Vp, u);
    st_nat(Bs, kLD, u);
    __syncthreads();
    mm64(ao, Wt, Bs);
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = 4 * ty + r;
        if (i >= len) continue;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int vv = vt * 64 + 4 * tx + c;
            if (vv < w.V) st_io(o, ((size_t)(tok0 + i) * w.H + h) * w.V + vv, bf16, ao[r][c]);
        }
    }
}

// ---------------------------------------------------------------------------------------------
// K4  Rm^T dO, the adjoint scan's state-independent term; one (key tile, value tile) per CTA
// ---------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) adjoint_term_kernel(Ws w, Scr s, const void* __restrict__ d_o, int bf16, int vec_v) {
    extern __shared__ __align__(16) float sm[];
    const int slot = blockIdx.x, h = blockIdx.y, VT = w.Vp / 64, kt = blockIdx.z / VT, vt = blockIdx.z % VT;
    dependents_go();
    int len, tok0;
    w.tab.span(slot, tok0, len);
    if (len == 0) return;
    const size_t ch = (size_t)slot * w.H + h;
    ld_nat(sm, w.Rm + ch * 64 * w.Kp + kt * 64, w.Kp);
    ld_tile_io<false>(sm + kTile, d_o, bf16, ((size_t)tok0 * w.H + h) * w.V + vt * 64, (size_t)w.H * w.V, len, w.V - vt * 64, vec_v);
    __syncthreads();
    float acc[4][4];
    zero_acc(acc);
    mm64(acc, sm, sm + kTile);
    st_nat(s.dHn + (ch * w.Kp + kt * 64) * w.Vp + vt * 64, w.Vp, acc);
}

// ---------------------------------------------------------------------------------------------
// K5  chunk-local adjoints, one CTA per (chunk, head): dZ, the products with the states, the adjoint of the inverse, the
//     pull-back through the decay-masked products and the L2-normalisation VJP, in one launch.  16 tile products at
//     K = V = 64; six tiles of shared memory, so that two CTAs share an SM.
// ---------------------------------------------------------------------------------------------
struct LocalArgs {
    const void *q, *k, *v, *g, *d_o;
    void *dq, *dk, *dv, *dg, *dbeta;
    int bf16, gbf16, l2norm, vec_k, vec_v;
    float scale;
};
constexpr size_t kLocalSmem = (6 * kTile + 64 * 3 + 4 * 64 * 3 + KDA_MAX_DIM) * sizeof(float);

// ONE: K, V <= 64, the loops over tiles are gone (and the loop-invariant addresses the compiler would keep for them)
template <bool ONE>
__global__ void __launch_bounds__(256, 2) local_bwd_kernel(Ws w, Scr s, LocalArgs p) {
    extern __shared__ __align__(16) float sm[];
    float *t0 = sm, *t1 = sm + kTile, *t2 = sm + 2 * kTile, *t3 = sm + 3 * kTile, *t4 = sm + 4 * kTile, *t5 = sm + 5 * kTile;
    dependency_wait();
    float* bet = sm + 6 * kTile;         // [64] beta, inverse norms
    float* qi_s = bet + 64;
    float* ki_s = qi_s + 64;
    float* bsum = ki_s + 64;             // [4][64] scratch
    float* cref = bsum + 256;            // [4][64] G at row 8 of each block
    float* tot = cref + 256;             // [4][64] scratch
    float* gend = tot + 256;             // [Kp]    d G_end
    const int slot = blockIdx.x, h = blockIdx.y;
    int len, tok0;
    w.tab.span(slot, tok0, len);
    if (len == 0) return;
    const int K = w.K, Kp = ONE ? 64 : w.Kp, V = w.V, Vp = ONE ? 64 : w.Vp, H = w.H, KT = Kp / 64, VT = Vp / 64;
    const size_t ch = (size_t)slot * H + h;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15, d = tid & 63, I = tid >> 6;
    const float* kn_g = w.kn + ch * 64 * Kp;
    const float* G_g = w.G + ch * 64 * Kp;
    const float* Ed_g = w.Ed + ch * 64 * Kp;
    const float* qn_g = w.qn + ch * 64 * Kp;
    const size_t vrow = (size_t)H * V, krow = (size_t)H * K;
    if (tid < 64) {
        bet[tid] = w.beta[ch * 64 + tid];
        qi_s[tid] = w.qinv[ch * 64 + tid];
        ki_s[tid] = w.kinv[ch * 64 + tid];
    }
    // column d, rows 16 I ..: x(row) -> four 16-byte stores along row d of a transposed tile
    auto st_col = [&](float* t, const float (&x)[16]) {
#pragma unroll
        for (int r4 = 0; r4 < 4; ++r4)
            *reinterpret_cast<float4*>(t + d * kLD + 16 * I + 4 * r4) = make_float4(x[4 * r4], x[4 * r4 + 1], x[4 * r4 + 2], x[4 * r4 + 3]);
    };
    float acc[4][4], accX[4][4];
    float db[4] = {0.f, 0.f, 0.f, 0.f};      // dbeta of this thread's rows (equal in the 16 lanes of a row)
    zero_acc(accX);
    {
        float accA[4][4];
        zero_acc(accA);
        for (int vt = 0; vt < VT; ++vt) {
            const size_t voff = ((size_t)tok0 * H + h) * V + vt * 64;
            const int nc = V - vt * 64;
            // ---- dZ = A^T dO + E dH'; every tile of the step is on its way before the first product
            __syncthreads();
            cpa_nat(t4, w.A + ch * 4096, 64);
            cpa_nat(t2, s.dHn + ch * Kp * Vp + vt * 64, Vp);
            cpa_tr(t1, w.Z + ch * 64 * Vp + vt * 64, Vp);
            if (vt == 0) cpa_nat(t3, w.T + ch * 4096, 64);
            cpa_commit();
            ld_tile_io<false>(t5, p.d_o, p.bf16, voff, vrow, len, nc, p.vec_v);
            ld_tile_io<true>(t0, p.d_o, p.bf16, voff, vrow, len, nc, p.vec_v);
            float e[16];
            auto source_col = [&](int kt) {      // column of E^T
#pragma unroll
                for (int r = 0; r < 16; ++r) {
                    const size_t o = (size_t)(16 * I + r) * Kp + kt * 64 + d;
                    e[r] = kn_g[o] * Ed_g[o];
                }
            };
            source_col(0);
            cpa_wait();
            __syncthreads();
            zero_acc(acc);
            mm64(acc, t4, t5);
            for (int kt = 0; kt < KT; ++kt) {
                __syncthreads();
                if (kt > 0) {
                    source_col(kt);
                    ld_nat(t2, s.dHn + (ch * Kp + kt * 64) * Vp + vt * 64, Vp);
                }
                st_col(t5, e);
                __syncthreads();
                mm64(acc, t5, t2);
            }
            // ---- X += dZ (beta v)^T, dv = beta T^T dZ, dA += dO Z^T
            __syncthreads();
            st_tr(t2, kLD, acc);
            st_nat(t4, kLD, acc);
            if (VT > 1) st_nat(s.dZ + ch * 64 * Vp + vt * 64, Vp, acc);
            ld_tile_io<true>(t5, p.v, p.bf16, voff, vrow, len, nc, p.vec_v, bet);
            __syncthreads();
            mm64(accX, t2, t5);
            zero_acc(acc);
            mm64(acc, t3, t4);
            __syncthreads();
            if (VT == 1) {      // the first key tile's states, behind the last product
                cpa_tr(t4, w.Hc + ch * Kp * Vp, Vp);
                cpa_tr(t5, s.dHn + ch * Kp * Vp, Vp);
                cpa_commit();
            }
            mm64(accA, t0, t1);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = 4 * ty + r;
                float x[4], part = 0.f;
                ld4_io(x, p.v, p.bf16, voff, vrow, i, 4 * tx, len, nc, p.vec_v);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    part += acc[r][c] * x[c];
                    if (i < len && 4 * tx + c < nc) st_io(p.dv, voff + (size_t)i * vrow + 4 * tx + c, p.bf16, bet[i] * acc[r][c]);
                }
                db[r] += row_sum16(part);
            }
        }
        st_nat(s.dA + ch * 4096, 64, accA);      // waits in L2 while the registers serve the key tiles
    }
    for (int kt = 0; kt < KT; ++kt) {
        // Products with the states, one at a time where one value tile is all there is: dR, dE and dW then never live
        // together (with them the kernel spills, and a spill reload costs an L2 round trip next to 218 KB of shared memory).
        float dG[4][4], dk[4][4], aW[4][4], colE[4] = {0.f, 0.f, 0.f, 0.f}, dd = 0.f;
        zero_acc(dG);
        zero_acc(dk);
        zero_acc(aW);
        const size_t so = ch * 64 * Kp + kt * 64;
        if (VT == 1) {
            __syncthreads();
            if (kt > 0) {
                cpa_tr(t4, w.Hc + (ch * Kp + kt * 64) * Vp, Vp);
                cpa_tr(t5, s.dHn + (ch * Kp + kt * 64) * Vp, Vp);
                cpa_commit();
            }
            cpa_wait();
            __syncthreads();
            mm64(aW, t2, t4);
            zero_acc(acc);
            mm64(acc, t0, t4);                   // dR
            mm64(dk, t1, t5);                    // dE
            for (int vv = 16 * I; vv < 16 * I + 16; ++vv) dd += t4[vv * kLD + d] * t5[vv * kLD + d];
        } else {
            zero_acc(acc);
            for (int vt = 0; vt < VT; ++vt) {
                const size_t voff = ((size_t)tok0 * H + h) * V + vt * 64;
                __syncthreads();
                cpa_tr(t4, w.Hc + (ch * Kp + kt * 64) * Vp + vt * 64, Vp);
                cpa_tr(t5, s.dHn + (ch * Kp + kt * 64) * Vp + vt * 64, Vp);
                cpa_tr(t1, w.Z + ch * 64 * Vp + vt * 64, Vp);
                cpa_tr(t2, s.dZ + ch * 64 * Vp + vt * 64, Vp);
                cpa_commit();
                ld_tile_io<true>(t0, p.d_o, p.bf16, voff, vrow, len, V - vt * 64, p.vec_v);
                cpa_wait();
                __syncthreads();
                mm64(aW, t2, t4);
                mm64(acc, t0, t4);
                mm64(dk, t1, t5);
                for (int vv = 16 * I; vv < 16 * I + 16; ++vv) dd += t4[vv * kLD + d] * t5[vv * kLD + d];
            }
        }
        {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const size_t o = (size_t)(4 * ty + r) * Kp + kt * 64 + 4 * tx;
                const float4 g4 = *reinterpret_cast<const float4*>(G_g + o), q4 = *reinterpret_cast<const float4*>(qn_g + o),
                             k4 = *reinterpret_cast<const float4*>(kn_g + o), e4 = *reinterpret_cast<const float4*>(Ed_g + o);
                const float ga[4] = {g4.x, g4.y, g4.z, g4.w}, qa[4] = {q4.x, q4.y, q4.z, q4.w}, ka[4] = {k4.x, k4.y, k4.z, k4.w},
                            ea[4] = {e4.x, e4.y, e4.z, e4.w};
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    acc[r][c] *= expf(ga[c]);                  // dq = dR e^G
                    dk[r][c] *= ea[c];                         // dE e^{G_end - G}
                    const float eE = dk[r][c] * ka[c];
                    dG[r][c] = acc[r][c] * qa[c] - eE;
                    colE[c] += eE;
                }
            }
            st_nat(s.dqn + so, Kp, acc);
        }
        // ---- X -= dW Q^T, T^T dW
        __syncthreads();
        if (kt == KT - 1) {      // dZ^T is read out: T^T for the adjoint of the inverse
            cpa_tr(t2, w.T + ch * 4096, 64);
            cpa_commit();
        }
        st_tr(t4, kLD, aW);
        {
            float x[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const size_t o = (size_t)(16 * I + r) * Kp + kt * 64 + d;
                x[r] = -bet[16 * I + r] * expf(G_g[o]) * kn_g[o];
            }
            st_col(t5, x);
        }
        bsum[I * 64 + d] = dd;
        __syncthreads();
        mm64(accX, t4, t5);
        __syncthreads();
        st_nat(t4, kLD, aW);
        __syncthreads();
        zero_acc(acc);
        mm64(acc, t3, t4);
        // ---- the part through Q: dQ = -(T^T dW)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const size_t o = (size_t)(4 * ty + r) * Kp + kt * 64 + 4 * tx;
            const float4 g4 = *reinterpret_cast<const float4*>(G_g + o), k4 = *reinterpret_cast<const float4*>(kn_g + o);
            const float ga[4] = {g4.x, g4.y, g4.z, g4.w}, ka[4] = {k4.x, k4.y, k4.z, k4.w};
            const float bi = bet[4 * ty + r];
            float brow = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float dQ = -acc[r][c] * expf(ga[c]);
                brow += dQ * ka[c];
                dG[r][c] += dQ * bi * ka[c];
                dk[r][c] += dQ * bi;
            }
            db[r] += row_sum16(brow);
        }
        st_nat(s.dkn + so, Kp, dk);
        st_nat(s.dG + so, Kp, dG);
        *reinterpret_cast<float4*>(t5 + ty * 64 + 4 * tx) = make_float4(colE[0], colE[1], colE[2], colE[3]);      // Q^T is read out
        __syncthreads();
        if (tid < 64) {
            float t = 0.f;
#pragma unroll
            for (int j = 0; j < 16; ++j) t += t5[j * 64 + tid];
            gend[kt * 64 + tid] = t + expf(G_g[(size_t)63 * Kp + kt * 64 + tid]) * (bsum[tid] + bsum[64 + tid] + bsum[128 + tid] + bsum[192 + tid]);
        }
    }
    // ---- dM = -stril(T^T X T^T), dA = tril(dO Z^T)
    float accA[4][4], accM[4][4];
    __syncthreads();
    st_nat(t4, kLD, accX);
    cpa_wait();
    __syncthreads();
    zero_acc(acc);
    mm64(acc, t3, t4);
    st_tr(t5, kLD, acc);
    __syncthreads();
    zero_acc(accM);
    mm64(accM, t5, t2);
    ld_patch(accA, s.dA + ch * 4096, 64);
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = 4 * ty + r, j = 4 * tx + c;
            accA[r][c] = j <= i ? accA[r][c] : 0.f;
            accM[r][c] = j < i ? -accM[r][c] : 0.f;
        }
    // ---- pull-back, one key tile at a time
    const int T0 = ty >> 2;              // 16-row block of this thread's patch rows
    for (int kt = 0; kt < KT; ++kt) {
        const int dd = kt * 64 + d;
        const bool in = dd < K;
        float L[16];
        {
            const size_t col = ((size_t)tok0 * H + h) * K + (in ? dd : 0);
            float run = 0.f;
#pragma unroll
            for (int r = 0; r < 16; ++r) L[r] = (16 * I + r < len && in) ? ld_io(p.g, col + (size_t)(16 * I + r) * krow, p.gbf16) : 0.f;
#pragma unroll
            for (int r = 0; r < 16; ++r) L[r] = run += L[r];
        }
        __syncthreads();
        bsum[I * 64 + d] = L[15];
        __syncthreads();
        float pre = 0.f;
        for (int J = 0; J < I; ++J) pre += bsum[J * 64 + d];
        const float c = L[8];
        cref[I * 64 + d] = pre + c;
        bool far = false;
#pragma unroll
        for (int r = 0; r < 16; ++r) far = far || !(fabsf(L[r] - c) <= kMaxExponent);
        const bool pairwise = __syncthreads_or(far);
        float aq[4][4], am[4][4], a2[4][4];      // with the decay factors applied, below
        zero_acc(aq);
        zero_acc(am);
        zero_acc(a2);
        if (!pairwise) {
            // row part: (dA | dM)[i][s] k_s exp(c_I - G_s); sources of block I: rows 8 I (I + 1) .. of the array at t2
            st_tr(t0, kLD, accA);
            st_tr(t1, kLD, accM);
            float kc[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) kc[r] = kn_g[(size_t)(16 * I + r) * Kp + dd] * expf(c - L[r]);
            for (int T = I; T < 4; ++T) {
                const float f = T == I ? 1.f : expf(cref[T * 64 + d] - cref[I * 64 + d]);
                float* o = t2 + (8 * T * (T + 1) + 16 * I) * kLD + d;
#pragma unroll
                for (int r = 0; r < 16; ++r) o[r * kLD] = kc[r] * f;
            }
#pragma unroll
            for (int r = 0; r < 16; ++r) t5[(16 * I + r) * kLD + d] = L[r] - c;
            __syncthreads();
            {
                const float *x = t0 + 4 * ty, *y = t1 + 4 * ty, *b = t2 + 8 * T0 * (T0 + 1) * kLD + 4 * tx;
                const int n = 16 * (T0 + 1);
                f2 pq[4][2], pm[4][2];
                to_pairs(pq, aq);
                to_pairs(pm, am);
#pragma unroll 4
                for (int kk = 0; kk < n; ++kk) {
                    const float4 bb = *reinterpret_cast<const float4*>(b + kk * kLD);
                    fma_pairs(pq, *reinterpret_cast<const float4*>(x + kk * kLD), bb);
                    fma_pairs(pm, *reinterpret_cast<const float4*>(y + kk * kLD), bb);
                }
                from_pairs(aq, pq);
                from_pairs(am, pm);
            }
            __syncthreads();
            // column part: sum over target blocks of exp(c_T - G_s) sum_{i in T} dA[i][s] q~_i + beta_i dM[i][s] k~_i
            st_nat(t0, kLD, accA);
            {
                float bm[4][4];
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) bm[r][cc] = bet[4 * ty + r] * accM[r][cc];
                st_nat(t1, kLD, bm);
            }
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const float e = expf(t5[(16 * I + r) * kLD + d]);      // L - c, back from this thread's own store
                const size_t o = (size_t)(16 * I + r) * Kp + dd;
                t2[(16 * I + r) * kLD + d] = qn_g[o] * e;
                t3[(16 * I + r) * kLD + d] = kn_g[o] * e;
            }
            __syncthreads();
            for (int T = 3; T >= T0; --T) {
                if (T < 3) {
                    float f[4];
#pragma unroll
                    for (int cc = 0; cc < 4; ++cc) f[cc] = expf(cref[(T + 1) * 64 + 4 * tx + cc] - cref[T * 64 + 4 * tx + cc]);
#pragma unroll
                    for (int r = 0; r < 4; ++r)
#pragma unroll
                        for (int cc = 0; cc < 4; ++cc) a2[r][cc] *= f[cc];
                }
                mm_at(a2, t0 + 16 * T * kLD + 4 * ty, kLD, t2 + 16 * T * kLD + 4 * tx, kLD, 16);
                mm_at(a2, t1 + 16 * T * kLD + 4 * ty, kLD, t3 + 16 * T * kLD + 4 * tx, kLD, 16);
            }
            float x[4][4];
            ld_patch(x, t5, kLD);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    const float e = expf(x[r][cc]), f = expf(-x[r][cc]);
                    aq[r][cc] *= e;
                    am[r][cc] *= e;
                    a2[r][cc] *= f;
                }
        } else {
            st_nat(t0, kLD, accA);
            st_nat(t1, kLD, accM);
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                const size_t o = (size_t)(16 * I + r) * Kp + dd;
                t2[(16 * I + r) * kLD + d] = qn_g[o];
                t3[(16 * I + r) * kLD + d] = kn_g[o];
                t5[(16 * I + r) * kLD + d] = pre + L[r];
            }
            __syncthreads();
            for (int r = 0; r < 4; ++r)
                for (int cc = 0; cc < 4; ++cc) {
                    const int i = 4 * ty + r, col = 4 * tx + cc;
                    const float gi = t5[i * kLD + col];
                    float vq = 0.f, vm = 0.f, v2 = 0.f;
                    for (int ss = 0; ss <= i; ++ss) {
                        const float e = expf(gi - t5[ss * kLD + col]) * t3[ss * kLD + col];
                        vq += t0[i * kLD + ss] * e;
                        vm += t1[i * kLD + ss] * e;
                    }
                    for (int ii = i; ii < 64; ++ii)
                        v2 += expf(t5[ii * kLD + col] - gi) * (t0[ii * kLD + i] * t2[ii * kLD + col] + bet[ii] * t1[ii * kLD + i] * t3[ii * kLD + col]);
#pragma unroll
                    for (int rr = 0; rr < 4; ++rr)
#pragma unroll
                        for (int ss = 0; ss < 4; ++ss)
                            if (rr == r && ss == cc) {
                                aq[rr][ss] = vq;
                                am[rr][ss] = vm;
                                a2[rr][ss] = v2;
                            }
                }
        }
        // ---- assemble
        const size_t so = ch * 64 * Kp + kt * 64;
        {
            float q[4][4], k[4][4], x[4][4];
            ld_patch(q, qn_g + kt * 64, Kp);
            ld_patch(k, kn_g + kt * 64, Kp);
            ld_patch(x, s.dG + so, Kp);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float bi = bet[4 * ty + r];
                float part = 0.f;
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    part += k[r][cc] * am[r][cc];
                    x[r][cc] += q[r][cc] * aq[r][cc] + bi * k[r][cc] * am[r][cc] - k[r][cc] * a2[r][cc];
                    am[r][cc] = bi * am[r][cc] + a2[r][cc];
                }
                db[r] += row_sum16(part);
            }
            st_nat(t4, kLD, x);
            ld_patch(q, s.dqn + so, Kp);
            ld_patch(k, s.dkn + so, Kp);
#pragma unroll
            for (int r = 0; r < 4; ++r)
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    aq[r][cc] += q[r][cc];
                    am[r][cc] += k[r][cc];
                }
        }
        if (KT == 1) {      // a row lies in 16 lanes: normalise here
            const size_t koff = ((size_t)tok0 * H + h) * K;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int i = 4 * ty + r;
                float x[4], y[4], pq = 0.f, pk = 0.f;
                ld4_io(x, p.q, p.bf16, koff, krow, i, 4 * tx, len, K, p.vec_k);
                ld4_io(y, p.k, p.bf16, koff, krow, i, 4 * tx, len, K, p.vec_k);
#pragma unroll
                for (int cc = 0; cc < 4; ++cc) {
                    x[cc] *= qi_s[i];
                    y[cc] *= ki_s[i];
                    aq[r][cc] *= p.scale;
                    pq += x[cc] * aq[r][cc];
                    pk += y[cc] * am[r][cc];
                }
                if (p.l2norm) {
                    pq = row_sum16(pq);
                    pk = row_sum16(pk);
                }
#pragma unroll
                for (int cc = 0; cc < 4; ++cc)
                    if (i < len && 4 * tx + cc < K) {
                        const size_t o = koff + (size_t)i * krow + 4 * tx + cc;
                        st_io(p.dq, o, p.bf16, p.l2norm ? qi_s[i] * (aq[r][cc] - x[cc] * pq) : aq[r][cc]);
                        st_io(p.dk, o, p.bf16, p.l2norm ? ki_s[i] * (am[r][cc] - y[cc] * pk) : am[r][cc]);
                    }
            }
        } else {
            st_nat(s.dqn + so, Kp, aq);
            st_nat(s.dkn + so, Kp, am);
        }
        // reverse cumulative sum of dG down the rows; the chunk-end term enters at the last one
        __syncthreads();
        {
            float x[16], sum = 0.f;
#pragma unroll
            for (int r = 0; r < 16; ++r) sum += x[r] = t4[(16 * I + r) * kLD + d];
            tot[I * 64 + d] = sum;
            __syncthreads();
            float run = gend[dd];
            for (int J = 3; J > I; --J) run += tot[J * 64 + d];
#pragma unroll
            for (int r = 15; r >= 0; --r) {
                run += x[r];
                const int i = 16 * I + r;
                if (i < len && in) st_io(p.dg, ((size_t)tok0 * H + h) * K + (size_t)i * krow + dd, p.gbf16, run);
            }
        }
    }
    if (tx == 0) {
#pragma unroll
        for (int r = 0; r < 4; ++r)
            if (4 * ty + r < len) st_io(p.dbeta, (size_t)(tok0 + 4 * ty + r) * H + h, p.gbf16, db[r]);
    }
    if (KT > 1) {
        __syncthreads();
        const int warp = tid >> 5, lane = tid & 31;
        for (int i = warp; i < len; i += 8) {
            const size_t off = ((size_t)(tok0 + i) * H + h) * K;
            const float* dqn = s.dqn + (ch * 64 + i) * Kp;
            const float* dkn = s.dkn + (ch * 64 + i) * Kp;
            const float qi = qi_s[i], ki = ki_s[i];
            float pq = 0.f, pk = 0.f;
            if (p.l2norm) {
                for (int e = lane; e < K; e += 32) {
                    pq += ld_io(p.q, off + e, p.bf16) * qi * dqn[e] * p.scale;
                    pk += ld_io(p.k, off + e, p.bf16) * ki * dkn[e];
                }
                pq = warp_sum(pq);
                pk = warp_sum(pk);
            }
            for (int e = lane; e < K; e += 32) {
                if (p.l2norm) {
                    st_io(p.dq, off + e, p.bf16, qi * (dqn[e] * p.scale - ld_io(p.q, off + e, p.bf16) * qi * pq));
                    st_io(p.dk, off + e, p.bf16, ki * (dkn[e] - ld_io(p.k, off + e, p.bf16) * ki * pk));
                } else {
                    st_io(p.dq, off + e, p.bf16, dqn[e] * p.scale);
                    st_io(p.dk, off + e, p.bf16, dkn[e]);
                }
            }
        }
    }
}

}  // namespace simt

// ---------------------------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------------------------
using simt::Scr;
using simt::Ws;

int tc_scan_forward(const simt::Ws& w, const tc::TcWs& t, int n_seq, int tokens, const float* h0, float* final_state, void* o,
                    const tc::NormEpilogue& norm, cudaStream_t st);
int tc_walk_forward(const simt::Ws& w, const tc::TcWs& t, int n_seq, int tokens, const float* h0, float* final_state, void* o,
                    const tc::NormEpilogue& norm, cudaStream_t st);
int tc_walk_backward(const simt::Ws& w, const simt::Scr& s, const tc::TcWs& t, int n_seq, int tokens, const void* d_o,
                     const float* d_final, float* dh0, cudaStream_t st);
int tc_intra_forward(const simt::Ws& w, const tc::TcWs& t, const void* q, const void* k, const void* v, const void* g,
                     const void* beta, int gbf16, int l2norm, float scale, int tokens, const tc::ConvPrep* conv, cudaStream_t st);
int tc_scan_backward(const simt::Ws& w, const simt::Scr& s, const tc::TcWs& t, int n_seq, int tokens, const void* d_o,
                     const float* d_final, float* dh0, cudaStream_t st);
int tc_intra_backward(const simt::Ws& w, const simt::Scr& s, const tc::TcWs& t, int n_seq, int tokens, const void* q, const void* k, const void* v,
                      const void* g, const void* d_o, int gbf16, int l2norm, float scale, void* dq, void* dk, void* dv,
                      void* dg, void* dbeta, cudaStream_t st);

template <class Kern>
static int set_smem(Kern kern, size_t bytes) {
    return bytes > 48 * 1024 ? set_smem_limit(kern, bytes) : KDA_OK;
}

// four-element accesses along a tensor's last dimension are aligned
static int vec4(const void* p, int dim) { return dim % 4 == 0 && reinterpret_cast<uintptr_t>(p) % 16 == 0; }

// Whether a kernel starts beside the one before it: with at most one chunk-head to an SM.  More blocks, placed while that one still
// holds some SMs, crowd onto the others (8 chunk-heads forward and backward 127.1 -> 123.1 us, 384 378.9 -> 389.8).
static bool starts_early(const Ws& w) { return w.nslots > 0 && w.nslots * (long long)w.H <= 148; }

static int launch_scan(const Ws& w, int n_seq, const simt::ScanArgs& a, const char* name, cudaStream_t st) {
    const size_t bytes = simt::scan_smem(w.Kp);
    // padding strips hold zeros already: E^T U and Rm^T dO of zero columns
    const dim3 grid(n_seq, w.H, ceil_div(w.V, simt::kVS));
    cudaError_t e = cudaSuccess;
#define KDA_SCAN(KT)                                                                                              \
    case KT:                                                                                                      \
        if (set_smem(simt::scan_kernel<KT>, bytes)) return KDA_ERR_CUDA;                                          \
        KDA_LAUNCH(name, st, e = launch_early(simt::scan_kernel<KT>, grid, 256, bytes, st, starts_early(w), 1, w, a));     \
        break
    switch (w.Kp / 64) {
        KDA_SCAN(1);
        KDA_SCAN(2);
        KDA_SCAN(3);
        KDA_SCAN(4);
        default: return KDA_ERR_BAD_SHAPE;
    }
#undef KDA_SCAN
    return e == cudaSuccess ? launch_status() : KDA_ERR_CUDA;
}

static int chunk_table(const KdaChunkShape* sh, const Ws& w, const int32_t* cu, cudaStream_t st) {
    if (w.tab.per_seq > 0) return KDA_OK;
    KDA_LAUNCH("chunk_table_kernel", st, simt::chunk_table_kernel<<<1, simt::kTableThreads, 0, st>>>(w, cu, sh->n_seq, sh->tokens, w.status, status_mirror()));
    return launch_status();
}

int simt_chunk_fwd(const KdaChunkShape* sh, const void* q, const void* k, const void* v, const void* g, const void* beta,
                   const float* h0, const int32_t* cu, void* o, float* final_state, void* workspace, cudaStream_t st,
                   const tc::NormEpilogue* norm, const tc::ConvPrep* conv) {
    Ws w = simt::carve_ws(*sh, workspace);
    if (conv != nullptr && (sh->lane != KDA_LANE_TC || !sh->forward_only)) return KDA_ERR_UNSUPPORTED;
    if (norm != nullptr && norm->gate != nullptr && sh->lane != KDA_LANE_TC) return KDA_ERR_UNSUPPORTED;
    const int bf16 = sh->io_dtype == KDA_DTYPE_BF16, gbf16 = sh->gate_dtype == KDA_DTYPE_BF16;
    const int VT = w.Vp / 64;
    if (sh->lane == KDA_LANE_TC) {
        // chunk-parallel operand panels and transitions on tcgen05, the affine state scan, then the chunk outputs
        size_t ws_bytes = 0;
        simt::carve_ws(*sh, nullptr, &ws_bytes);
        tc::TcWs t = tc::carve_tc(*sh, static_cast<char*>(workspace) + ws_bytes);
        t.status = w.status;      // one status word per workspace, shared by both lanes
        if (int rc = chunk_table(sh, w, cu, st)) return rc;
        if (w.nslots > 0) {
            int rc = tc_intra_forward(w, t, q, k, v, g, beta, gbf16, sh->l2norm, sh->scale, sh->tokens, conv, st);
            if (rc) return rc;
            const auto recurrence = t.nseg > 1 ? tc_scan_forward : tc_walk_forward;
            rc = recurrence(w, t, sh->n_seq, sh->tokens, h0, final_state, o,
                            norm != nullptr ? *norm : tc::NormEpilogue{nullptr, nullptr, 0.f, nullptr, nullptr, 0}, st);
            if (rc) return rc;
        }
        return launch_status();
    }
    if (int rc = chunk_table(sh, w, cu, st)) return rc;
    const dim3 gch(w.nslots, w.H);
    if (w.nslots > 0) {
        const simt::IntraArgs a{q, k, v, g, beta, bf16, gbf16, sh->l2norm, vec4(v, sh->value_dim), sh->forward_only ? 0 : 1, sh->scale, status_mirror(), w.tab.per_seq > 0};
        if (set_smem(simt::intra_fwd_kernel, simt::kIntraSmem)) return KDA_ERR_CUDA;
        KDA_LAUNCH("intra_fwd_kernel", st, simt::intra_fwd_kernel<<<gch, 256, simt::kIntraSmem, st>>>(w, a));
    }
    if (int rc = launch_scan(w, sh->n_seq, simt::ScanArgs{w.PT, w.Hc, h0, final_state, 0}, "scan_fwd_kernel", st)) return rc;
    if (w.nslots > 0) {
        const size_t sm_out = (size_t)3 * simt::kTile * sizeof(float);
        if (set_smem(simt::out_kernel, sm_out)) return KDA_ERR_CUDA;
        cudaError_t e = cudaSuccess;
        KDA_LAUNCH("out_kernel", st, e = launch_early(simt::out_kernel, dim3(w.nslots, w.H, VT), 256, sm_out, st, starts_early(w), 1, w, o, bf16));
        if (e != cudaSuccess) return KDA_ERR_CUDA;
    }
    return launch_status();
}

// Device status word of a forward / backward pair that used `workspace`: 0, kStatusBadCuSeqlens, or the code of the
// bounded wait that expired in the tensor-core lane.
static int status_code(int v) {
    return v == 0 ? KDA_OK : (v == simt::kStatusBadCuSeqlens ? KDA_ERR_CU_SEQLENS : KDA_ERR_DEVICE_STATUS);
}

// Reads the word back over the stream, i.e. synchronises the stream - for tests and post-mortems, not for the hot
// path (and not under stream capture).
int chunk_status(const KdaChunkShape* sh, const void* workspace, cudaStream_t st) {
    Ws w = simt::carve_ws(*sh, const_cast<void*>(workspace));
    int v = 0;
    if (cudaMemcpyAsync(&v, w.status, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess) return KDA_ERR_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return KDA_ERR_CUDA;
    return status_code(v);
}

// Queues a copy of the word into caller-owned page-locked host memory; nothing waits.
int chunk_status_async(const KdaChunkShape* sh, const void* workspace, int32_t* host_word, cudaStream_t st) {
    Ws w = simt::carve_ws(*sh, const_cast<void*>(workspace));
    return cudaMemcpyAsync(host_word, w.status, sizeof(int), cudaMemcpyDeviceToHost, st) == cudaSuccess ? KDA_OK : KDA_ERR_CUDA;
}

int status_word_to_code(int v) { return status_code(v); }

int simt_chunk_bwd(const KdaChunkShape* sh, const void* q, const void* k, const void* v, const void* g, const void* beta,
                   const int32_t* cu, const void* d_o, const float* d_final, const void* workspace, void* scratch,
                   void* dq, void* dk, void* dv, void* dg, void* dbeta, float* dh0, cudaStream_t st) {
    (void)beta; (void)cu;
    Ws w = simt::carve_ws(*sh, const_cast<void*>(workspace));
    Scr s = simt::carve_scr(*sh, scratch);
    const int bf16 = sh->io_dtype == KDA_DTYPE_BF16, gbf16 = sh->gate_dtype == KDA_DTYPE_BF16;
    const int KT = w.Kp / 64;
    if (sh->lane == KDA_LANE_TC) {
        size_t ws_bytes = 0;
        simt::carve_ws(*sh, nullptr, &ws_bytes);
        tc::TcWs t = tc::carve_tc(*sh, static_cast<char*>(const_cast<void*>(workspace)) + ws_bytes);
        t.status = w.status;
        if (w.nslots > 0) {
            int rc = (t.nseg > 1 ? tc_scan_backward : tc_walk_backward)(w, s, t, sh->n_seq, sh->tokens, d_o, d_final, dh0, st);
            if (rc) return rc;
            rc = tc_intra_backward(w, s, t, sh->n_seq, sh->tokens, q, k, v, g, d_o, gbf16, sh->l2norm, sh->scale, dq, dk, dv, dg, dbeta, st);
            return rc ? rc : launch_status();
        } else if (dh0) {
            return KDA_ERR_UNSUPPORTED;
        }
        return launch_status();
    }
    const int vec_v = vec4(v, sh->value_dim) && vec4(d_o, sh->value_dim);
    if (w.nslots > 0) {
        const size_t sm_term = (size_t)2 * simt::kTile * sizeof(float);
        KDA_LAUNCH("adjoint_term_kernel", st, simt::adjoint_term_kernel<<<dim3(w.nslots, w.H, KT * (w.Vp / 64)), 256, sm_term, st>>>(w, s, d_o, bf16, vec_v));
    }
    if (int rc = launch_scan(w, sh->n_seq, simt::ScanArgs{w.P, s.dHn, d_final, dh0, 1}, "scan_bwd_kernel", st)) return rc;
    if (w.nslots > 0) {
        const simt::LocalArgs a{q, k, v, g, d_o, dq, dk, dv, dg, dbeta, bf16, gbf16, sh->l2norm,
                                vec4(q, sh->key_dim) && vec4(k, sh->key_dim), vec_v, sh->scale};
        const auto kern = KT == 1 && w.Vp == 64 ? simt::local_bwd_kernel<true> : simt::local_bwd_kernel<false>;
        if (set_smem(kern, simt::kLocalSmem)) return KDA_ERR_CUDA;
        cudaError_t e = cudaSuccess;
        KDA_LAUNCH("local_bwd_kernel", st, e = launch_early(kern, dim3(w.nslots, w.H), 256, simt::kLocalSmem, st, starts_early(w), 1, w, s, a));
        if (e != cudaSuccess) return KDA_ERR_CUDA;
    }
    return launch_status();
}

}  // namespace kda
