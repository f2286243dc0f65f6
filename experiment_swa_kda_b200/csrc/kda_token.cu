// Products of a few rows: y[m][n] = sum_k x[m][k] w[n][k] for at most 64 rows of x, the shapes of a decode step.
//
// At these row counts a product is bound by reading the weights once (4 bytes each as float32 masters: 100 MB per token at
// width 2,048), so the kernel takes the masters as they are and rounds them to bf16 in registers: no cast pass, no packed
// copy, and several weight matrices with a common input share the launch.  A CTA owns 16 weight rows; its eight warps split
// k in interleaved 32-wide steps, so a row is read as contiguous kilobytes and about 100 KB per SM are in flight.  The
// contraction runs on mma.sync m16n8k16 with the weights as the 16-row operand (a tcgen05 tile would need the weights
// staged in shared memory as bf16 first, which is the copy this kernel avoids); k is permuted inside a step so that each
// lane's operands are 32 (weights) and 16 (x) contiguous bytes.  Partial sums meet in shared memory in a fixed order: a
// result depends on its row of x and of w alone, not on how many rows the call has.

#include "common.cuh"

namespace kda {
namespace tok {

constexpr int kWarps = 8, kRows = 16, kMaxRows = 64, kItems = 6, kStep = 32;

struct RowsArgs {
    const __nv_bfloat16* x;        // [m][k], rows ldx apart
    long long ldx;
    int m, k, n_items;
    const void* w[kItems];         // [rows][k] each, dense
    int end[kItems];               // running row ends
    __nv_bfloat16* out;            // [m][row], rows ldo apart
    long long ldo;
    // CONV: items 0..2 are the q, k, v projections of one token per row; their results step the short convolutions
    const void* conv_w[3];         // [channels][width]
    void* cache[3];                // [m][channels][width] bf16, shifted in place
    __nv_bfloat16* act;            // [3][m][channels]
    int width, conv_wf32;
};

__device__ __forceinline__ uint32_t pk(float a, float b) {
    __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// NT: 8-row tiles of x.  U: steps whose loads are issued together.
template <int NT, bool F32W, bool CONV, int U>
__global__ void __launch_bounds__(kWarps * 32) rows_kernel(RowsArgs p) {
    __shared__ float red[kWarps][kRows][NT * 8 + 1];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int row0 = blockIdx.x * kRows;
    int item = 0, begin = 0;
#pragma unroll
    for (int i = 1; i < kItems; ++i)
        if (i < p.n_items && row0 >= p.end[i - 1]) {
            item = i;
            begin = p.end[i - 1];
        }
    int end = p.end[0];
    const void* w = p.w[0];
#pragma unroll
    for (int i = 1; i < kItems; ++i)
        if (i == item) {
            end = p.end[i];
            w = p.w[i];
        }
    const int lo = min(row0 + g, end - 1) - begin, hi = min(row0 + g + 8, end - 1) - begin;      // rows past the end repeat the last one
    const size_t olo = (size_t)lo * p.k + 8 * tig, ohi = (size_t)hi * p.k + 8 * tig;
    float acc[NT][4];
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[t][e] = 0.f;
    const int steps = p.k / kStep;
    for (int s0 = warp; s0 < steps; s0 += kWarps * U) {
        uint4 a[U][2];                             // bf16 weights: 8 of each row
        uint4 xb[U][NT];
        if (F32W) {
            float4 f[U][4];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int s = s0 + kWarps * u;
                if (s < steps) {
                    const float4* pl = reinterpret_cast<const float4*>(static_cast<const float*>(w) + olo + (size_t)s * kStep);
                    const float4* ph = reinterpret_cast<const float4*>(static_cast<const float*>(w) + ohi + (size_t)s * kStep);
                    f[u][0] = __ldg(pl); f[u][1] = __ldg(pl + 1);
                    f[u][2] = __ldg(ph); f[u][3] = __ldg(ph + 1);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int r = 0; r < 2; ++r)
                    a[u][r] = make_uint4(pk(f[u][2 * r].x, f[u][2 * r].y), pk(f[u][2 * r].z, f[u][2 * r].w),
                                         pk(f[u][2 * r + 1].x, f[u][2 * r + 1].y), pk(f[u][2 * r + 1].z, f[u][2 * r + 1].w));
        } else {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int s = s0 + kWarps * u;
                if (s < steps) {
                    a[u][0] = __ldg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(w) + olo + (size_t)s * kStep));
                    a[u][1] = __ldg(reinterpret_cast<const uint4*>(static_cast<const __nv_bfloat16*>(w) + ohi + (size_t)s * kStep));
                }
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int s = s0 + kWarps * u;
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                xb[u][t] = make_uint4(0, 0, 0, 0);
                if (s < steps && t * 8 + g < p.m)
                    xb[u][t] = __ldg(reinterpret_cast<const uint4*>(p.x + (size_t)(t * 8 + g) * p.ldx + (size_t)s * kStep + 8 * tig));
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (s0 + kWarps * u < steps) {
                const uint32_t a0[4] = {a[u][0].x, a[u][1].x, a[u][0].y, a[u][1].y}, a1[4] = {a[u][0].z, a[u][1].z, a[u][0].w, a[u][1].w};
#pragma unroll
                for (int t = 0; t < NT; ++t) {
                    mma_bf16(acc[t], a0, xb[u][t].x, xb[u][t].y);
                    mma_bf16(acc[t], a1, xb[u][t].z, xb[u][t].w);
                }
            }
        }
    }
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        red[warp][g][t * 8 + 2 * tig] = acc[t][0];
        red[warp][g][t * 8 + 2 * tig + 1] = acc[t][1];
        red[warp][g + 8][t * 8 + 2 * tig] = acc[t][2];
        red[warp][g + 8][t * 8 + 2 * tig + 1] = acc[t][3];
    }
    __syncthreads();
    for (int i = threadIdx.x; i < kRows * p.m; i += kWarps * 32) {
        const int r = i & (kRows - 1), m = i / kRows;
        if (row0 + r >= end) continue;
        float y = 0.f;
#pragma unroll
        for (int k = 0; k < kWarps; ++k) y += red[k][r][m];
        const __nv_bfloat16 yb = __float2bfloat16(y);
        if (CONV && item < 3) {
            // one token of the short convolution + SiLU, the arithmetic of the stand-alone step: the window drops its oldest
            // value and takes y; the cache is rewritten in place
            void* cache = item == 0 ? p.cache[0] : (item == 1 ? p.cache[1] : p.cache[2]);
            const void* cw = item == 0 ? p.conv_w[0] : (item == 1 ? p.conv_w[1] : p.conv_w[2]);
            const int C = end - begin, c = row0 + r - begin;
            const size_t base = ((size_t)m * C + c) * p.width;
            float z = 0.f;
            for (int j = 0; j < p.width; ++j) {
                const float v = j + 1 < p.width ? ld_io(cache, base + j + 1, 1) : __bfloat162float(yb);
                float wj;
                if (p.conv_wf32) wj = __bfloat162float(__float2bfloat16(static_cast<const float*>(cw)[(size_t)c * p.width + j]));
                else wj = ld_io(cw, (size_t)c * p.width + j, 1);
                z += wj * v;
                st_io(cache, base + j, 1, v);
            }
            float th;
            asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(0.5f * z));
            p.act[((size_t)item * p.m + m) * C + c] = __float2bfloat16(z * fmaf(0.5f, th, 0.5f));
        } else {
            p.out[(size_t)m * p.ldo + row0 + r] = yb;
        }
    }
}

template <bool F32W, bool CONV>
int launch_rows(const RowsArgs& p, cudaStream_t st) {
    const int blocks = ceil_div(p.end[p.n_items - 1], kRows);
    if (p.m <= 8) KDA_LAUNCH("rows_kernel", st, rows_kernel<1, F32W, CONV, 4><<<blocks, kWarps * 32, 0, st>>>(p));
    else if (p.m <= 16) KDA_LAUNCH("rows_kernel", st, rows_kernel<2, F32W, CONV, 4><<<blocks, kWarps * 32, 0, st>>>(p));
    else if (p.m <= 32) KDA_LAUNCH("rows_kernel", st, rows_kernel<4, F32W, CONV, 2><<<blocks, kWarps * 32, 0, st>>>(p));
    else KDA_LAUNCH("rows_kernel", st, rows_kernel<8, F32W, CONV, 2><<<blocks, kWarps * 32, 0, st>>>(p));
    return launch_status();
}

// y[m][n] for one 128-wide product (the low-rank gate projection), a warp per (row of x, weight row): the form the decode
// kernel's prologue uses, so that both give the same bits.
template <bool F32W>
__global__ void __launch_bounds__(256) narrow_kernel(int m, int n, const __nv_bfloat16* __restrict__ x, long long ldx, const void* __restrict__ w,
                                                     __nv_bfloat16* __restrict__ out) {
    const long long i = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= (long long)m * n) return;
    const int lane = threadIdx.x & 31, row = (int)(i % n), mm = (int)(i / n);
    float xv[4], wv[4];
    narrow_x(x + (size_t)mm * ldx, lane, xv);
    narrow_w<F32W>(w, (size_t)row * 128, lane, wv);
    const float y = narrow_sum(xv, wv);
    if (lane == 0) out[(size_t)mm * n + row] = __float2bfloat16(y);
}

}  // namespace tok
}  // namespace kda

using namespace kda;

extern "C" int kda_rows_linear(int32_t m, int32_t k, int32_t n_items, int32_t weight_dtype, const void* x, int64_t x_ld, const void* const* weight,
                               const int32_t* rows, void* out, int64_t out_ld, const KdaTokenConv* conv, void* stream) {
    if (m < 1 || m > tok::kMaxRows || k < 1 || n_items < 1 || n_items > tok::kItems || x_ld < k) return KDA_ERR_BAD_SHAPE;
    if (!x || !weight || !rows || !out) return KDA_ERR_NULL;
    if (k % tok::kStep != 0 || x_ld % 8 != 0 || (weight_dtype != KDA_DTYPE_F32 && weight_dtype != KDA_DTYPE_BF16)) return KDA_ERR_UNSUPPORTED;
    tok::RowsArgs p = {};
    p.x = static_cast<const __nv_bfloat16*>(x);
    p.ldx = x_ld;
    p.m = m; p.k = k; p.n_items = n_items;
    p.out = static_cast<__nv_bfloat16*>(out);
    p.ldo = out_ld;
    uintptr_t al = reinterpret_cast<uintptr_t>(x);
    int end = 0;
    for (int i = 0; i < n_items; ++i) {
        if (!weight[i]) return KDA_ERR_NULL;
        // a 16-row group belongs to one matrix: every matrix but the last fills its groups
        if (rows[i] < 1 || (i + 1 < n_items && rows[i] % tok::kRows != 0)) return KDA_ERR_UNSUPPORTED;
        end += rows[i];
        p.w[i] = weight[i];
        p.end[i] = end;
        al |= reinterpret_cast<uintptr_t>(weight[i]);
    }
    if (al % 16 != 0 || out_ld < (conv ? 0 : end)) return KDA_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    const bool f32 = weight_dtype == KDA_DTYPE_F32;
    if (!conv) return f32 ? tok::launch_rows<true, false>(p, st) : tok::launch_rows<false, false>(p, st);
    if (n_items < 3 || conv->width < 1 || conv->width > 4 || !conv->act) return KDA_ERR_BAD_SHAPE;
    for (int i = 0; i < 3; ++i) {
        if (!conv->weight[i] || !conv->cache[i]) return KDA_ERR_NULL;
        p.conv_w[i] = conv->weight[i];
        p.cache[i] = conv->cache[i];
    }
    p.act = static_cast<__nv_bfloat16*>(conv->act);
    p.width = conv->width;
    p.conv_wf32 = conv->weight_dtype == KDA_DTYPE_F32;
    return f32 ? tok::launch_rows<true, true>(p, st) : tok::launch_rows<false, true>(p, st);
}

extern "C" int kda_narrow_linear(int32_t m, int32_t n, int32_t weight_dtype, const void* x, int64_t x_ld, const void* weight, void* out, void* stream) {
    if (m < 1 || n < 1 || x_ld < 128) return KDA_ERR_BAD_SHAPE;
    if (!x || !weight || !out) return KDA_ERR_NULL;
    if (x_ld % 8 != 0 || (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(weight)) % 16 != 0) return KDA_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned blocks = (unsigned)(((long long)m * n + 7) / 8);
    if (weight_dtype == KDA_DTYPE_F32)
        KDA_LAUNCH("narrow_kernel", st, tok::narrow_kernel<true><<<blocks, 256, 0, st>>>(m, n, static_cast<const __nv_bfloat16*>(x), x_ld, weight, static_cast<__nv_bfloat16*>(out)));
    else
        KDA_LAUNCH("narrow_kernel", st, tok::narrow_kernel<false><<<blocks, 256, 0, st>>>(m, n, static_cast<const __nv_bfloat16*>(x), x_ld, weight, static_cast<__nv_bfloat16*>(out)));
    return launch_status();
}
