// Products of a few rows: y[m][n] = sum_k x[m][k] w[n][k] for at most 64 rows of x, the shapes of a decode step.
//
// At these row counts a product is bound by reading the weights once (4 bytes each as float32 masters: 100 MB per token at
// width 2,048), so the kernel takes the masters as they are and rounds them to bf16 in registers: no cast pass, no packed
// copy, and several weight matrices with a common input share the launch.  A CTA owns 16 weight rows; its eight warps split
// k in interleaved 32-wide steps, so a row is read as contiguous kilobytes and about 100 KB per SM are in flight.  The
// contraction runs on mma.sync m16n8k16 with the weights as the 16-row operand (a tcgen05 tile would need the weights
// staged in shared memory as bf16 first, which is the copy this kernel avoids); k is permuted inside a step so that
// every 16-byte piece of a lane lies next to its neighbours' (a quad covers 64 contiguous bytes of a row; two 16-byte
// halves of a 32-byte sector in different copies would fetch it twice).  Partial sums meet in shared memory in a fixed order: a
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
    int width, conv_wf32, conv_vec;      // conv_vec: width 4, windows and weights aligned for one access each
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

// NT: 8-row tiles of x.  RT: 16-row tiles of weights per CTA; two halve the reads of x (every CTA reads all of it) where
// there are enough rows to give every SM a CTA all the same.
// Weights arrive through a thread-private ring in shared memory filled by 16-byte asynchronous copies, 96 KB per CTA in
// flight and no registers held for it (register-staged loads reached 2.3 TB/s at 2,048 x 8,336 and 32 rows, 68 MB of
// masters); x, which L2 serves, is loaded one step ahead.
// DEEP: no more CTAs than SMs and no convolution, the output projection: the ring takes 192 KB, so that up to 3,072 columns are all on
// their way while the kernel before it still runs.
template <int RT, bool DEEP>
constexpr int kDepth = DEEP ? 12 : (RT == 1 ? 6 : 3);
// Leading dimension of the partial sums: odd for the reads (lanes over rows), and 9 modulo 32 leaves two lanes at most on a bank in the
// writes (lanes over 8 rows x 4 pairs; four lanes at 1 modulo 32).
template <int NT>
constexpr int kLdRed = NT >= 4 ? NT * 8 + 9 : NT * 8 + 1;
// Steps x is loaded ahead.  With one tile of weights a CTA there are few CTAs, latency counts, and registers are there for it (output
// projection of 32 tokens, 2,048 wide, from the end of the kernel before it: 9.0 us with one step ahead and six stages, 8.5 with two,
// 6.4 with the deep ring as well).
template <int RT, int NT>
constexpr int kDepthX = RT == 2 ? 1 : (NT == 1 ? 6 : (NT == 2 ? 3 : 2));

__device__ __forceinline__ void cp16(uint32_t dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}

template <int NT, bool F32W, bool CONV, int RT, bool DEEP>
__global__ void __launch_bounds__(kWarps * 32) rows_kernel(RowsArgs p) {
    constexpr int D = kDepth<RT, DEEP>, PIECES = F32W ? 4 : 2, NTH = kWarps * 32, ROWS = kRows * RT, LD = kLdRed<NT>;
    extern __shared__ __align__(16) uint8_t smem[];
    dependents_go();
    uint4* ring = reinterpret_cast<uint4*>(smem);                    // [D][RT][PIECES][threads]
    float* red = reinterpret_cast<float*>(smem);                     // [warps][ROWS][LD], once the ring is drained
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, tig = lane & 3;
    const int row0 = blockIdx.x * ROWS;
    const uint8_t* src[RT][2];                                       // rows g and g + 8 of each tile; past the end: the last row
    constexpr int ES = F32W ? 4 : 2;
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int hf = 0; hf < 2; ++hf) {
            int row = min(row0 + 16 * r + 8 * hf + g, p.end[p.n_items - 1] - 1), begin = 0;
            const void* w = p.w[0];
#pragma unroll
            for (int i = 1; i < kItems; ++i)
                if (i < p.n_items && row >= p.end[i - 1]) {
                    begin = p.end[i - 1];
                    w = p.w[i];
                }
            src[r][hf] = static_cast<const uint8_t*>(w) + (size_t)(row - begin) * p.k * ES + 16 * tig;
        }
    const int steps = p.k / kStep, mine = steps > warp ? (steps - warp + kWarps - 1) / kWarps : 0;      // steps warp, warp + 8, ...
    const uint32_t slot = (uint32_t)__cvta_generic_to_shared(ring + threadIdx.x);
    auto issue = [&](int i) {
        if (i < mine) {
            const size_t off = (size_t)(warp + kWarps * i) * kStep * ES;
#pragma unroll
            for (int r = 0; r < RT; ++r)
#pragma unroll
                for (int q = 0; q < PIECES; ++q)
                    cp16(slot + (uint32_t)((((i % D) * RT + r) * PIECES + q) * NTH) * 16u, src[r][q / (PIECES / 2)] + off + (q % (PIECES / 2)) * 64);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    constexpr int XD = kDepthX<RT, NT>;
    uint4 xb[XD][NT];
    auto load_x = [&](int i, uint4 (&x)[NT]) {
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            x[t] = make_uint4(0, 0, 0, 0);
            if (i < mine && t * 8 + g < p.m) {
                const __nv_bfloat16* xr = p.x + (size_t)(t * 8 + g) * p.ldx + (size_t)(warp + kWarps * i) * kStep;
                if (F32W) {
                    const uint2 u = ld_after8(xr + 4 * tig), v = ld_after8(xr + 16 + 4 * tig);
                    x[t] = make_uint4(u.x, u.y, v.x, v.y);
                } else {
                    x[t] = ld_after16(xr + 8 * tig);
                }
            }
        }
    };
    float acc[RT][NT][4];
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int t = 0; t < NT; ++t)
#pragma unroll
            for (int e = 0; e < 4; ++e) acc[r][t][e] = 0.f;
#pragma unroll
    for (int i = 0; i < D - 1; ++i) issue(i);
    dependency_wait();                                               // weights are nobody's output; x may be the kernel's before
#pragma unroll
    for (int i = 0; i < XD; ++i) load_x(i, xb[i]);
    // A thread's outputs all belong to one weight row (ROWS divides the block), so its convolution windows and weights can
    // come in now, behind the product, instead of one after another at the end (32 tokens, 16 heads: 24.0 -> 21 us).
    constexpr int NOUT = (ROWS * NT * 8 + NTH - 1) / NTH;
    const int orow = row0 + threadIdx.x % ROWS;
    const bool early = CONV && p.conv_vec && orow < p.end[2];
    const int citem = orow < p.end[0] ? 0 : (orow < p.end[1] ? 1 : 2), cc = orow - citem * p.end[0];      // the three have the same channels
    uint2* const win_at = CONV ? static_cast<uint2*>(citem == 0 ? p.cache[0] : (citem == 1 ? p.cache[1] : p.cache[2])) : nullptr;
    const void* const cw = citem == 0 ? p.conv_w[0] : (citem == 1 ? p.conv_w[1] : p.conv_w[2]);
    uint2 win[CONV ? NOUT : 1];
    float cwt[4];
    if (early) {
#pragma unroll
        for (int o = 0; o < NOUT; ++o) {
            const int m = (threadIdx.x + o * NTH) / ROWS;
            if (m < p.m) win[o] = win_at[(size_t)m * p.end[0] + cc];
        }
        if (p.conv_wf32) {
            const float4 u = __ldg(static_cast<const float4*>(cw) + cc);
            cwt[0] = __bfloat162float(__float2bfloat16(u.x)); cwt[1] = __bfloat162float(__float2bfloat16(u.y));
            cwt[2] = __bfloat162float(__float2bfloat16(u.z)); cwt[3] = __bfloat162float(__float2bfloat16(u.w));
        } else {
            const uint2 u = __ldg(static_cast<const uint2*>(cw) + cc);
            cwt[0] = __uint_as_float(u.x << 16); cwt[1] = __uint_as_float(u.x & 0xffff0000u);
            cwt[2] = __uint_as_float(u.y << 16); cwt[3] = __uint_as_float(u.y & 0xffff0000u);
        }
    }
#pragma unroll 1
    for (int i0 = 0; i0 < mine; i0 += XD)
#pragma unroll
    for (int d = 0; d < XD; ++d) {
        const int i = i0 + d;
        if (XD > 1 && i >= mine) break;
        issue(i + D - 1);
        uint4 xc[NT];
#pragma unroll
        for (int t = 0; t < NT; ++t) xc[t] = xb[d][t];
        load_x(i + XD, xb[d]);
        asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
#pragma unroll
        for (int r = 0; r < RT; ++r) {
            uint4 a[2];                             // 8 bf16 of rows g and g + 8
            const uint4* mem = ring + (((i % D) * RT + r) * PIECES) * NTH + threadIdx.x;
            if (F32W) {
#pragma unroll
                for (int hf = 0; hf < 2; ++hf) {
                    const float4 u = *reinterpret_cast<const float4*>(mem + (2 * hf) * NTH), v = *reinterpret_cast<const float4*>(mem + (2 * hf + 1) * NTH);
                    a[hf] = make_uint4(pk(u.x, u.y), pk(u.z, u.w), pk(v.x, v.y), pk(v.z, v.w));
                }
            } else {
                a[0] = mem[0];
                a[1] = mem[NTH];
            }
            const uint32_t a0[4] = {a[0].x, a[1].x, a[0].y, a[1].y}, a1[4] = {a[0].z, a[1].z, a[0].w, a[1].w};
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                mma_bf16(acc[r][t], a0, xc[t].x, xc[t].y);
                mma_bf16(acc[r][t], a1, xc[t].z, xc[t].w);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                                                 // every warp has drained its ring: the memory becomes the partials
#pragma unroll
    for (int r = 0; r < RT; ++r)
#pragma unroll
        for (int t = 0; t < NT; ++t) {
            float* d = red + (size_t)(warp * ROWS + 16 * r + g) * LD + t * 8 + 2 * tig;
            d[0] = acc[r][t][0];
            d[1] = acc[r][t][1];
            d[8 * LD] = acc[r][t][2];
            d[8 * LD + 1] = acc[r][t][3];
        }
    __syncthreads();
    if (orow >= p.end[p.n_items - 1]) return;
#pragma unroll
    for (int o = 0; o < NOUT; ++o) {
        const int m = (threadIdx.x + o * NTH) / ROWS;
        if (m >= p.m) break;
        float y = 0.f;
#pragma unroll
        for (int k = 0; k < kWarps; ++k) y += red[(size_t)(k * ROWS + threadIdx.x % ROWS) * LD + m];
        const __nv_bfloat16 yb = __float2bfloat16(y);
        if (CONV && orow < p.end[2]) {
            // one token of the short convolution + SiLU, the arithmetic of the stand-alone step: the window drops its oldest
            // value and takes y; the cache is rewritten in place
            const int C = p.end[0];
            float z = 0.f;
            if (early) {
                const uint32_t yw = (uint32_t)*reinterpret_cast<const uint16_t*>(&yb) << 16;
                const uint2 next = make_uint2((win[o].x >> 16) | (win[o].y << 16), (win[o].y >> 16) | yw);
                z += cwt[0] * __uint_as_float(next.x << 16);
                z += cwt[1] * __uint_as_float(next.x & 0xffff0000u);
                z += cwt[2] * __uint_as_float(next.y << 16);
                z += cwt[3] * __uint_as_float(yw);
                win_at[(size_t)m * C + cc] = next;
            } else {
                void* cache = win_at;
                const size_t base = ((size_t)m * C + cc) * p.width;
                for (int j = 0; j < p.width; ++j) {
                    const float v = j + 1 < p.width ? ld_io(cache, base + j + 1, 1) : __bfloat162float(yb);
                    float wj;
                    if (p.conv_wf32) wj = __bfloat162float(__float2bfloat16(static_cast<const float*>(cw)[(size_t)cc * p.width + j]));
                    else wj = ld_io(cw, (size_t)cc * p.width + j, 1);
                    z += wj * v;
                    st_io(cache, base + j, 1, v);
                }
            }
            float th;
            asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(0.5f * z));
            p.act[((size_t)citem * p.m + m) * C + cc] = __float2bfloat16(z * fmaf(0.5f, th, 0.5f));
        } else {
            p.out[(size_t)m * p.ldo + orow] = yb;
        }
    }
}

// 4 counts of row tiles x 2 weight types x (with and without convolutions x 2 heights, deep): one signature
static_assert(kSmemKernels >= 4 * 2 * 5, "set_smem_limit would forget instantiations of rows_kernel");
template <int NT, bool F32W, bool CONV, int RT, bool DEEP = false>
int launch_tile(const RowsArgs& p, bool early, cudaStream_t st) {
    constexpr size_t ring = (size_t)kDepth<RT, DEEP> * RT * (F32W ? 4 : 2) * kWarps * 32 * 16, red = (size_t)kWarps * kRows * RT * kLdRed<NT> * 4;
    constexpr size_t bytes = ring > red ? ring : red;
    if (set_smem_limit(rows_kernel<NT, F32W, CONV, RT, DEEP>, bytes)) return KDA_ERR_CUDA;
    cudaError_t e = cudaSuccess;
    KDA_LAUNCH("rows_kernel", st, e = launch_early(rows_kernel<NT, F32W, CONV, RT, DEEP>, dim3(ceil_div(p.end[p.n_items - 1], kRows * RT)), kWarps * 32, bytes, st, early, 1, p));
    return e == cudaSuccess ? launch_status() : KDA_ERR_CUDA;
}

template <bool F32W, bool CONV>
int launch_rows(const RowsArgs& p, bool early, cudaStream_t st) {
    const bool wide = p.end[p.n_items - 1] >= 148 * kRows * 2;       // at least one CTA of two tiles for every SM
    const bool deep = !CONV && p.end[p.n_items - 1] <= 148 * kRows;  // one CTA of one tile at most
#define KDA_ROWS(NT) (wide ? launch_tile<NT, F32W, CONV, 2>(p, early, st) : (!CONV && deep ? launch_tile<NT, F32W, false, 1, true>(p, early, st) : launch_tile<NT, F32W, CONV, 1>(p, early, st)))
    return p.m <= 8 ? KDA_ROWS(1) : (p.m <= 16 ? KDA_ROWS(2) : (p.m <= 32 ? KDA_ROWS(4) : KDA_ROWS(8)));
#undef KDA_ROWS
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
    narrow_x(*reinterpret_cast<const uint2*>(x + (size_t)mm * ldx + 4 * lane), xv);
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
    const bool early = (weight_dtype & KDA_BEHIND_OWN_LAUNCH) != 0;
    weight_dtype &= ~KDA_BEHIND_OWN_LAUNCH;
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
        if (rows[i] < 1) return KDA_ERR_BAD_SHAPE;
        end += rows[i];
        p.w[i] = weight[i];
        p.end[i] = end;
        al |= reinterpret_cast<uintptr_t>(weight[i]);
    }
    if (al % 16 != 0 || out_ld < (conv ? 0 : end)) return KDA_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    const bool f32 = weight_dtype == KDA_DTYPE_F32;
    if (!conv) return f32 ? tok::launch_rows<true, false>(p, early, st) : tok::launch_rows<false, false>(p, early, st);
    if (n_items < 3 || rows[1] != rows[0] || rows[2] != rows[0] || conv->width < 1 || conv->width > 4 || !conv->act) return KDA_ERR_BAD_SHAPE;
    for (int i = 0; i < 3; ++i) {
        if (!conv->weight[i] || !conv->cache[i]) return KDA_ERR_NULL;
        p.conv_w[i] = conv->weight[i];
        p.cache[i] = conv->cache[i];
    }
    p.act = static_cast<__nv_bfloat16*>(conv->act);
    p.width = conv->width;
    p.conv_wf32 = conv->weight_dtype == KDA_DTYPE_F32;
    uintptr_t cal = 0, wal = 0;
    for (int i = 0; i < 3; ++i) {
        cal |= reinterpret_cast<uintptr_t>(conv->cache[i]);
        wal |= reinterpret_cast<uintptr_t>(conv->weight[i]);
    }
    p.conv_vec = conv->width == 4 && cal % 8 == 0 && wal % 16 == 0;
    return f32 ? tok::launch_rows<true, true>(p, early, st) : tok::launch_rows<false, true>(p, early, st);
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
