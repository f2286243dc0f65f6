// Bandwidth-bound KDA kernels: gate activations, recurrent decode step, short causal
// depthwise convolution (+SiLU) and gated RMSNorm, forward and backward.  All are
// HBM-bound: wide coalesced loads, warp-shuffle reductions, deterministic two-stage
// reductions for the weight gradients (no floating-point atomics).

#include <algorithm>

#include <type_traits>

#include "common.cuh"

namespace kda {
namespace pw {

// sigmoid for the bf16 I/O paths: one hardware tanh (relative error 2^-11, far inside bf16 rounding) instead of an
// exponential and a reciprocal - these kernels are bound by instruction issue, not by DRAM; float32 I/O keeps expf and a
// true divide
template <bool FAST>
__device__ __forceinline__ float sigmoid_t(float x) {
    if (FAST) {
        float t;
        asm("tanh.approx.f32 %0, %1;" : "=f"(t) : "f"(0.5f * x));
        return fmaf(0.5f, t, 0.5f);
    }
    return 1.0f / (1.0f + expf(-x));
}

template <bool BF16>
__device__ __forceinline__ void ld4(float (&d)[4], const void* p, size_t i) {
    if (BF16) {
        uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p) + i);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
        float2 a = __bfloat1622float2(h[0]), b = __bfloat1622float2(h[1]);
        d[0] = a.x; d[1] = a.y; d[2] = b.x; d[3] = b.y;
    } else {
        float4 f = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + i);
        d[0] = f.x; d[1] = f.y; d[2] = f.z; d[3] = f.w;
    }
}
template <bool BF16>
__device__ __forceinline__ void st4(void* p, size_t i, const float (&s)[4]) {
    if (BF16) {
        uint2 u;
        __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
        h[0] = __floats2bfloat162_rn(s[0], s[1]);
        h[1] = __floats2bfloat162_rn(s[2], s[3]);
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p) + i) = u;
    } else {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(p) + i) = make_float4(s[0], s[1], s[2], s[3]);
    }
}

// =============================================================================================
// gate / beta activations
// =============================================================================================
__global__ void gate_fwd_kernel(size_t n_gate, size_t n_beta, int H, int K, int bf16, const void* __restrict__ raw,
                                const void* __restrict__ bl, const float* __restrict__ A_log,
                                const float* __restrict__ dt_bias, float lb, float* __restrict__ g,
                                float* __restrict__ beta) {
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_gate; i += stride) {
        const int kk = (int)(i % K), h = (int)((i / K) % H);
        const float z = expf(A_log[h]) * (ld_io(raw, i, bf16) + dt_bias[h * K + kk]);
        g[i] = lb * sigmoidf_(z);
    }
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_beta; i += stride)
        beta[i] = sigmoidf_(ld_io(bl, i, bf16));
}

constexpr int kGateRows = 32;  // tokens per first-stage reduction block

// stage 1: d_raw, d_beta_logits and per-block column partials of ddt_bias / dA_log
__global__ void gate_bwd_kernel(int tokens, int H, int K, int bf16, const void* __restrict__ raw,
                                const void* __restrict__ bl, const float* __restrict__ A_log,
                                const float* __restrict__ dt_bias, float lb, const float* __restrict__ dg,
                                const float* __restrict__ dbeta, void* __restrict__ d_raw, void* __restrict__ d_bl,
                                float* __restrict__ part_b, float* __restrict__ part_a) {
    dependents_go();
    const int HK = H * K;
    const int t0 = blockIdx.x * kGateRows, t1 = min(tokens, t0 + kGateRows);
    for (int c = threadIdx.x; c < HK; c += blockDim.x) {
        const int h = c / K;
        const float ea = expf(A_log[h]), bias = dt_bias[c];
        float sb = 0.f, sa = 0.f;
        for (int t = t0; t < t1; ++t) {
            const size_t i = (size_t)t * HK + c;
            const float x = ld_io(raw, i, bf16) + bias;
            const float sg = sigmoidf_(ea * x);
            const float dr = dg[i] * lb * sg * (1.f - sg) * ea;
            st_io(d_raw, i, bf16, dr);
            sb += dr;
            sa += dr * x;
        }
        part_b[(size_t)blockIdx.x * HK + c] = sb;
        part_a[(size_t)blockIdx.x * HK + c] = sa;
    }
    for (int c = threadIdx.x; c < H; c += blockDim.x) {
        for (int t = t0; t < t1; ++t) {
            const size_t i = (size_t)t * H + c;
            const float b = sigmoidf_(ld_io(bl, i, bf16));
            st_io(d_bl, i, bf16, dbeta[i] * b * (1.f - b));
        }
    }
}

// stage 2: one block per head, 1024 threads = 8 row segments x 128 columns (wider heads loop over column groups);
// fixed summation order
__global__ void __launch_bounds__(1024) gate_bwd_reduce_kernel(int nblk, int H, int K, const float* __restrict__ part_b,
                                                               const float* __restrict__ part_a, float* __restrict__ ddt_bias,
                                                               float* __restrict__ dA_log) {
    __shared__ float redb[8][128], reda[8][128];
    __shared__ float wsum[4];
    const int h = blockIdx.x, HK = H * K;
    const int col = threadIdx.x & 127, seg = threadIdx.x >> 7;
    dependency_wait();                     // the kernel before wrote the partial sums
    float accA = 0.f;                      // segment 0 only: this column's share of sum_k (dr * x), over all column groups
    for (int k0 = 0; k0 < K; k0 += 128) {
        const int kk = k0 + col, c = h * K + kk;
        float sb = 0.f, sa = 0.f;
        if (kk < K)
            for (int b = seg; b < nblk; b += 8) {
                sb += ld_after_f32(part_b + (size_t)b * HK + c);
                sa += ld_after_f32(part_a + (size_t)b * HK + c);
            }
        redb[seg][col] = sb;
        reda[seg][col] = sa;
        __syncthreads();
        if (seg == 0 && kk < K) {
            float tb = 0.f, ta = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                tb += redb[r][col];
                ta += reda[r][col];
            }
            ddt_bias[c] = tb;
            accA += ta;
        }
        __syncthreads();
    }
    if (seg == 0) {                        // 4 warps hold the head's column sums: warp totals, then one thread
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) accA += __shfl_xor_sync(0xffffffffu, accA, o);
        if ((col & 31) == 0) wsum[col >> 5] = accA;
    }
    __syncthreads();
    if (threadIdx.x == 0) dA_log[h] = (wsum[0] + wsum[1]) + (wsum[2] + wsum[3]);
}

// =============================================================================================
// recurrent decode step
//   S' = S * exp(g);  r = v - k^T S';  S'' = S' + beta k r^T;  o = q^T S''
// The state is V-first [n_seq,H,V,K]: a row (fixed value index) is K contiguous floats.  One
// warp owns a row at a time: a single coalesced read and a single coalesced write per row, two
// shuffle reductions, and o_v = q.S'_v + beta r_v (q.k) so the row is never re-read.
// =============================================================================================
// NV4 > 0: K % 4 == 0, lane owns NV4 float4 of a row (keys 128*j + 4*lane + 0..3); NV4 == 0: scalar layout,
// lane owns keys lane + 32*e.  R rows are kept in flight per warp; every load is issued unconditionally
// (addresses clamped, values masked) so the loads of a row group overlap.
// When raw.A_log is set, g and beta hold the raw gate logits and beta logits instead and are activated here
// (g = lb * sigmoid(exp(A_log[h]) * (raw + dt_bias[h,k])), beta = sigmoid(logit)): one launch less per token and layer.
struct RawGate {
    const float* A_log;      // [H], or nullptr: g and beta are already activated
    const float* dt_bias;    // [H*K]
    float lb;
    long long bl_ld;         // elements between the beta logits of consecutive sequences (heads when dense)
};

// FUSED: the layer's decode step around the recurrence (K = V = 128, bf16, raw gate).  The kernel forms its head's raw
// gate from the low-rank projection, steps the state, and applies the gated RMSNorm to the head's output: three launches
// of a token become one.  Each part repeats the stand-alone kernel's arithmetic, so both forms give the same bits.  The
// block then owns all 128 rows of a state: 32 warps hold the whole 64 KB in flight when there are fewer blocks than SMs,
// eight warps otherwise.  Bound by the state's bytes with many sequences: eight warps are held to 64 registers, four blocks an SM (256 x
// 16 states without the rest: 96 us, 0.86 of the copy rate; with three blocks 101).
// With few, by a chain: the projections' outputs, the gate's weights (64 KB a block out of L2, which at 512 blocks it gave in 4.7 us),
// the head's scalars, rows, norm.  So the gate's weights and the first rows are loaded while the launch before still runs, the blocks of
// one head in four sequences form a cluster and share out the gate's rows, and the scalars are worked out once a block instead of in
// every warp.  From the end of the projections to the end of the kernel: 512 states 17.2 -> 14.6 us, 3 states 5.3 -> 4.3; a whole token of
// 32 x 16 heads 53.8 -> 45.8, of 1 x 3 18.4 -> 14.6 (9.6 in a graph, was 14.3).
struct TokenMix {
    const __nv_bfloat16* fa;       // [n_seq][128], rows ld apart
    const void* fb_w;              // [heads*128][128]
    const __nv_bfloat16* gate;     // [n_seq][heads][128], rows ld apart
    const float* norm_w;           // [128]
    long long ld;
    float eps;
    int fb_f32, n_seq;
};

template <int NV4, int R, int NW, bool FUSED, int CL>
__global__ void __launch_bounds__(NW * 32, NW > 8 ? 32 / NW : (NV4 == 1 ? 4 : 2)) decode_kernel(int H, int K, int V, int bf16, int gbf16, int l2norm, float scale,
                                                     const void* __restrict__ q, const void* __restrict__ k,
                                                     const void* __restrict__ v, const void* __restrict__ g,
                                                     const void* __restrict__ beta, const float* s_in, float* s_out,
                                                     void* __restrict__ o, int rows_per_cta, RawGate raw, TokenMix mix) {
    __shared__ __align__(16) float raw_s[FUSED ? 128 : 4];
    __shared__ __align__(16) float head_s[FUSED ? 388 : 4];      // scaled unit q, unit k, decay, then q.k and beta
    __shared__ __align__(16) __nv_bfloat16 o_s[FUSED ? 128 : 8];
    constexpr int NE = NV4 > 0 ? 4 * NV4 : 8;     // state elements per lane per row
    const int rank = blockIdx.x % CL, first = blockIdx.x - rank, last = CL > 1 ? mix.n_seq * H - 1 : 0;
    const int at = CL > 1 ? min((int)blockIdx.x, last) : blockIdx.x;
    const int head = CL > 1 ? at / mix.n_seq : at % H, seq = CL > 1 ? at - head * mix.n_seq : at / H;
    const bool shared = CL > 1 && first / mix.n_seq == min(first + CL - 1, last) / mix.n_seq;
    const int bh = seq * H + head;
    const int v_base = blockIdx.y * rows_per_cta;
    const int v_end = min(V, v_base + rows_per_cta);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    auto key_of = [&](int e) { return NV4 > 0 ? (128 * (e >> 2) + 4 * lane + (e & 3)) : (lane + 32 * e); };
    auto load_v = [&](int r0, float (&vv)[R]) {      // FUSED: v is the work of the kernel before
#pragma unroll
        for (int j = 0; j < R; ++j) vv[j] = ld_after_bf16(v, (size_t)bh * V + min(r0 + j, v_end - 1));
    };
    auto load_rows = [&](int r0, float (&s)[R][NE], float (&vv)[R]) {
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int row = min(r0 + j, v_end - 1);
            const float* src = s_in + ((size_t)bh * V + row) * K;
            if (NV4 > 0) {
#pragma unroll
                for (int e4 = 0; e4 < NV4; ++e4) {
                    const int kk = min(128 * e4 + 4 * lane, K - 4);
                    const float4 x = __ldcs(reinterpret_cast<const float4*>(src + kk));
                    s[j][4 * e4 + 0] = x.x; s[j][4 * e4 + 1] = x.y; s[j][4 * e4 + 2] = x.z; s[j][4 * e4 + 3] = x.w;
                }
            } else {
#pragma unroll
                for (int e = 0; e < NE; ++e) s[j][e] = src[min(lane + 32 * e, K - 1)];
            }
            if (!FUSED) vv[j] = ld_io(v, (size_t)bh * V + row, bf16);
        }
    };
    // first row group goes out before the per-(sequence, head) scalars are needed
    float s[R][NE], vv[R];
    float qe[NE], ke[NE], dec[NE], bt, qk;
    int r0 = v_base + warp * R;
    if (r0 < v_end) load_rows(r0, s, vv);
    if (FUSED) {
        dependents_go();
        // Everything with an address of its own is on its way before the first of it is needed: the state and the gate's weights ahead
        // of the launch this one may have started beside, the projections' outputs right behind its end.
        constexpr int GR = 128 / (CL * NW), G = GR < 4 ? GR : 4;    // gate rows a warp, and how many at once, NW apart
        float wv[G][4], xv[CL][4];
        auto load_w = [&](int r0) {
#pragma unroll
            for (int i = 0; i < G; ++i) {
                const size_t base = ((size_t)head * 128 + r0 + NW * i + warp) * 128;
                if (mix.fb_f32) narrow_w<true>(mix.fb_w, base, lane, wv[i]);
                else narrow_w<false>(mix.fb_w, base, lane, wv[i]);
            }
        };
        load_w(shared ? GR * NW * rank : 0);
        float ea = 0.f, db = 0.f;
        if (threadIdx.x < 128) {
            ea = expf(raw.A_log[head]);
            db = raw.dt_bias[head * 128 + threadIdx.x];
        }
        if (CL > 1) cluster_sync();                                 // the other blocks have started: their shared memory is there
        dependency_wait();
#pragma unroll
        for (int i = 0; i < CL; ++i) narrow_x(ld_after8(mix.fa + (size_t)(shared ? min(first + i, last) - head * mix.n_seq : seq) * mix.ld + 4 * lane), xv[i]);
        if (warp == 0) {
            bt = ld_after_bf16(beta, (size_t)seq * raw.bl_ld + head);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                qe[e] = ld_after_bf16(q, (size_t)bh * 128 + 4 * lane + e);
                ke[e] = ld_after_bf16(k, (size_t)bh * 128 + 4 * lane + e);
            }
        }
        load_v(r0, vv);
        auto gate_rows = [&](const float (&x)[4], int r0, int to) {
            float y[G];
#pragma unroll
            for (int i = 0; i < G; ++i) y[i] = narrow_sum(x, wv[i]);
            if (lane == 0) {
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    const float r = __bfloat162float(__float2bfloat16(y[i]));
                    if (CL > 1) st_cluster(raw_s + r0 + NW * i + warp, to, r);
                    else raw_s[r0 + NW * i + warp] = r;
                }
            }
        };
        if (shared) {
            static_assert(CL == 1 || G == GR, "a shared block's rows go at once");
#pragma unroll
            for (int c = 0; c < CL; ++c) gate_rows(xv[c], G * NW * rank, c);
        } else {
#pragma unroll 1
            for (int r0 = 0;;) {
                gate_rows(xv[0], r0, rank);
                if ((r0 += G * NW) >= 128) break;
                load_w(r0);
            }
        }
        if (warp == 0) {                                            // the head's q, k and scalars, once for all warps
            float sq = 0.f, sk = 0.f, qk = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                sq += qe[e] * qe[e];
                sk += ke[e] * ke[e];
            }
            sq = warp_sum(sq);
            sk = warp_sum(sk);
            const float qi = 1.f / fmaxf(sqrtf(sq), 1e-12f) * scale, ki = 1.f / fmaxf(sqrtf(sk), 1e-12f);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                qe[e] *= qi;
                ke[e] *= ki;
                qk += qe[e] * ke[e];
            }
            qk = warp_sum(qk);
            *reinterpret_cast<float4*>(head_s + 4 * lane) = make_float4(qe[0], qe[1], qe[2], qe[3]);
            *reinterpret_cast<float4*>(head_s + 128 + 4 * lane) = make_float4(ke[0], ke[1], ke[2], ke[3]);
            if (lane == 0) {
                head_s[384] = qk;
                head_s[385] = sigmoidf_(bt);
            }
        }
        if (CL > 1) cluster_sync();
        else __syncthreads();
        if (CL > 1 && (int)blockIdx.x > last) return;               // there for its share of the gate
        if (threadIdx.x < 128) head_s[256 + threadIdx.x] = expf(raw.lb * sigmoidf_(ea * (raw_s[threadIdx.x] + db)));
        __syncthreads();
        auto get4 = [&](float (&x)[NE], int at) {
            const float4 f = *reinterpret_cast<const float4*>(head_s + at + 4 * lane);
            x[0] = f.x; x[1] = f.y; x[2] = f.z; x[3] = f.w;
        };
        get4(qe, 0);
        get4(ke, 128);
        get4(dec, 256);
        qk = head_s[384];
        bt = head_s[385];
    } else {
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            const size_t i = (size_t)bh * K + min(key_of(e), K - 1);
            qe[e] = ld_io(q, i, bf16);
            ke[e] = ld_io(k, i, bf16);
            dec[e] = ld_io(g, i, gbf16);
        }
        bt = ld_io(beta, raw.A_log != nullptr ? (size_t)(bh / H) * raw.bl_ld + bh % H : (size_t)bh, gbf16);
        if (raw.A_log != nullptr) {
            const int hh = bh % H;
            const float ea = expf(raw.A_log[hh]);
            bt = sigmoidf_(bt);
#pragma unroll
            for (int e = 0; e < NE; ++e)
                dec[e] = raw.lb * sigmoidf_(ea * (dec[e] + raw.dt_bias[hh * K + min(key_of(e), K - 1)]));
        }
        float sq = 0.f, sk = 0.f;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            const bool in = key_of(e) < K;
            qe[e] = in ? qe[e] : 0.f;
            ke[e] = in ? ke[e] : 0.f;
            dec[e] = in ? expf(dec[e]) : 0.f;
            sq += qe[e] * qe[e];
            sk += ke[e] * ke[e];
        }
        sq = warp_sum(sq);
        sk = warp_sum(sk);
        const float qi = (l2norm ? 1.f / fmaxf(sqrtf(sq), 1e-12f) : 1.f) * scale;
        const float ki = l2norm ? 1.f / fmaxf(sqrtf(sk), 1e-12f) : 1.f;
        qk = 0.f;
#pragma unroll
        for (int e = 0; e < NE; ++e) {
            qe[e] *= qi;
            ke[e] *= ki;
            qk += qe[e] * ke[e];
        }
        qk = warp_sum(qk);
    }

    for (; r0 < v_end; r0 += NW * R) {
        float a[R], b[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            a[j] = 0.f;
            b[j] = 0.f;
#pragma unroll
            for (int e = 0; e < NE; ++e) {
                s[j][e] *= dec[e];
                a[j] += ke[e] * s[j][e];
                b[j] += qe[e] * s[j][e];
            }
        }
        // R independent reductions interleaved
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
#pragma unroll
            for (int j = 0; j < R; ++j) {
                a[j] += __shfl_xor_sync(0xffffffffu, a[j], off);
                b[j] += __shfl_xor_sync(0xffffffffu, b[j], off);
            }
        }
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const int row = r0 + j;
            if (row < v_end) {
                const float br = bt * (vv[j] - a[j]);
                float* dst = s_out + ((size_t)bh * V + row) * K;
                if (NV4 > 0) {
#pragma unroll
                    for (int e4 = 0; e4 < NV4; ++e4) {
                        const int kk = 128 * e4 + 4 * lane;
                        if (kk < K)
                            __stcs(reinterpret_cast<float4*>(dst + kk),
                                   make_float4(s[j][4 * e4 + 0] + br * ke[4 * e4 + 0], s[j][4 * e4 + 1] + br * ke[4 * e4 + 1],
                                               s[j][4 * e4 + 2] + br * ke[4 * e4 + 2], s[j][4 * e4 + 3] + br * ke[4 * e4 + 3]));
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < NE; ++e) {
                        const int kk = lane + 32 * e;
                        if (kk < K) dst[kk] = s[j][e] + br * ke[e];
                    }
                }
                if (lane == 0) {
                    if (FUSED) o_s[row] = __float2bfloat16(b[j] + br * qk);
                    else st_io(o, (size_t)bh * V + row, bf16, b[j] + br * qk);
                }
            }
        }
        if (r0 + NW * R < v_end) {
            load_rows(r0 + NW * R, s, vv);
            if (FUSED) load_v(r0 + NW * R, vv);
        }
    }
    if (FUSED) {
        __syncthreads();
        if (warp == 0) {      // the head's 128 outputs: lane = 4 adjacent values, as in the stand-alone norm
            float a[4], gt[4], out[4];
            ld4<true>(a, o_s, 4 * lane);
            narrow_x(ld_after8(mix.gate + (size_t)seq * mix.ld + head * 128 + 4 * lane), gt);
            const float4 ww = *reinterpret_cast<const float4*>(mix.norm_w + 4 * lane);
            const float wa[4] = {ww.x, ww.y, ww.z, ww.w};
            float ss = fmaf(a[3], a[3], fmaf(a[2], a[2], fmaf(a[1], a[1], a[0] * a[0])));
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
            ss += __shfl_xor_sync(0xffffffffu, ss, 16);
            const float inv = rsqrtf(ss * (1.0f / 128.0f) + mix.eps);
#pragma unroll
            for (int e = 0; e < 4; ++e) out[e] = a[e] * inv * wa[e] * sigmoid_t<true>(gt[e]);
            st4<true>(o, (size_t)bh * 128 + 4 * lane, out);
        }
    }
}

// =============================================================================================
// short causal depthwise convolution (+ SiLU)
//   xx = [cache[..., :], x] along time (cache slot p <-> time p - W);  y[t] = act(sum_j w[c][j] xx[t + 1 + j])
// One thread: VEC adjacent channels x kConvTT consecutive tokens, sliding window in registers.
// =============================================================================================
constexpr int kConvTT = 4;

template <int VEC, bool BF16>
__device__ __forceinline__ void ld_vec(float (&dst)[VEC], const void* p, size_t i) {
    if (BF16) {
        if (VEC == 8) {
            uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p) + i);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                float2 f = __bfloat1622float2(h[j]);
                dst[2 * j] = f.x;
                dst[2 * j + 1] = f.y;
            }
        } else {
#pragma unroll
            for (int j = 0; j < VEC; ++j) dst[j] = __bfloat162float(reinterpret_cast<const __nv_bfloat16*>(p)[i + j]);
        }
    } else {
        if (VEC == 4) {
            float4 f = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + i);
            dst[0] = f.x; dst[1] = f.y; dst[2] = f.z; dst[3] = f.w;
        } else {
#pragma unroll
            for (int j = 0; j < VEC; ++j) dst[j] = reinterpret_cast<const float*>(p)[i + j];
        }
    }
}

template <int VEC, bool BF16>
__device__ __forceinline__ void st_vec(void* p, size_t i, const float (&src)[VEC]) {
    if (BF16) {
        if (VEC == 8) {
            uint4 u;
            __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
            for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(src[2 * j], src[2 * j + 1]);
            *reinterpret_cast<uint4*>(reinterpret_cast<__nv_bfloat16*>(p) + i) = u;
        } else {
#pragma unroll
            for (int j = 0; j < VEC; ++j) reinterpret_cast<__nv_bfloat16*>(p)[i + j] = __float2bfloat16(src[j]);
        }
    } else {
        if (VEC == 4) {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(p) + i) = make_float4(src[0], src[1], src[2], src[3]);
        } else {
#pragma unroll
            for (int j = 0; j < VEC; ++j) reinterpret_cast<float*>(p)[i + j] = src[j];
        }
    }
}


// one weight; float32 weights next to bf16 activations are rounded to bf16 first, which is what a cast of the
// weight tensor to the activation dtype would have produced
__device__ __forceinline__ float ld_w(const void* w, size_t i, bool bf16, int wf32) {
    if (wf32) {
        const float f = reinterpret_cast<const float*>(w)[i];
        return bf16 ? __bfloat162float(__float2bfloat16(f)) : f;
    }
    return ld_io(w, i, bf16);
}

__device__ __forceinline__ bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// weights of VEC adjacent channels: W*VEC contiguous elements starting at c0*W.  A weight may be a view into a flat
// parameter buffer at any element offset, so it is the address, not the index, that allows a 16-byte load.
template <int W, int VEC, bool BF16>
__device__ __forceinline__ void ld_weights(float (&wv)[W][VEC], const void* wgt, int c0, int wf32) {
    float flat[W * VEC];
    constexpr int N = W * VEC;
    const size_t base = (size_t)c0 * W;
    if (wf32) {
#pragma unroll
        for (int j = 0; j < N; ++j) flat[j] = ld_w(wgt, base + j, BF16, 1);
    } else if (BF16 && N % 8 == 0 && aligned16(reinterpret_cast<const __nv_bfloat16*>(wgt) + base)) {
#pragma unroll
        for (int j = 0; j < N / 8; ++j) {
            float t[8];
            ld_vec<8, true>(t, wgt, base + 8 * j);
#pragma unroll
            for (int e = 0; e < 8; ++e) flat[8 * j + e] = t[e];
        }
    } else if (!BF16 && N % 4 == 0 && aligned16(reinterpret_cast<const float*>(wgt) + base)) {
#pragma unroll
        for (int j = 0; j < N / 4; ++j) {
            float t[4];
            ld_vec<4, false>(t, wgt, base + 4 * j);
#pragma unroll
            for (int e = 0; e < 4; ++e) flat[4 * j + e] = t[e];
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) flat[j] = ld_io(wgt, base + j, BF16);
    }
#pragma unroll
    for (int e = 0; e < VEC; ++e)
#pragma unroll
        for (int j = 0; j < W; ++j) wv[j][e] = flat[e * W + j];
}

// xx at time tau (tau < 0 reaches into the cache: slot W + tau), for VEC channels starting at c0
template <int VEC, bool BF16>
__device__ __forceinline__ void ld_xx(float (&dst)[VEC], const void* x, const void* cache, int b, int tau, int c0, int T,
                                      int C, int W) {
    if (tau >= 0) {
        ld_vec<VEC, BF16>(dst, x, ((size_t)b * T + tau) * C + c0);
    } else if (cache != nullptr && W + tau >= 0) {
#pragma unroll
        for (int j = 0; j < VEC; ++j) dst[j] = ld_io(cache, ((size_t)b * C + c0 + j) * W + (W + tau), BF16);
    } else {
#pragma unroll
        for (int j = 0; j < VEC; ++j) dst[j] = 0.f;
    }
}

template <int W, int VEC, bool BF16>
__global__ void __launch_bounds__(256) conv_fwd_kernel(int B, int T, int C, int silu, int wf32, const void* __restrict__ x,
                                                       const void* __restrict__ wgt, const void* __restrict__ cache,
                                                       void* __restrict__ y, void* __restrict__ fin) {
    const int ncg = C / VEC, ntile = (T + kConvTT - 1) / kConvTT;
    const size_t gid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (gid >= (size_t)B * ntile * ncg) return;
    const int cg = (int)(gid % ncg), tile = (int)((gid / ncg) % ntile), b = (int)(gid / ((size_t)ncg * ntile));
    const int c0 = cg * VEC, t0 = tile * kConvTT, t1 = min(T, t0 + kConvTT);
    float wv[W][VEC];
    ld_weights<W, VEC, BF16>(wv, wgt, c0, wf32);
    // inputs at times t0-(W-1) .. t0+kConvTT-1.  Interior tiles issue every load unconditionally (so they
    // overlap); only the first and last tile of a sequence take the guarded path.
    float xin[kConvTT + W - 1][VEC];
    if (t0 >= W - 1 && t0 + kConvTT <= T) {
#pragma unroll
        for (int j = 0; j < kConvTT + W - 1; ++j)
            ld_vec<VEC, BF16>(xin[j], x, ((size_t)b * T + (t0 - (W - 1) + j)) * C + c0);
    } else {
#pragma unroll
        for (int j = 0; j < kConvTT + W - 1; ++j) {
            const int tau = t0 - (W - 1) + j;
            if (tau < T) ld_xx<VEC, BF16>(xin[j], x, cache, b, tau, c0, T, C, W);
            else {
#pragma unroll
                for (int e = 0; e < VEC; ++e) xin[j][e] = 0.f;
            }
        }
    }
#pragma unroll
    for (int tt = 0; tt < kConvTT; ++tt) {
        const int t = t0 + tt;
        if (t < t1) {
            float out[VEC];
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                float z = 0.f;
#pragma unroll
                for (int j = 0; j < W; ++j) z += wv[j][e] * xin[tt + j][e];
                out[e] = silu ? z * sigmoid_t<BF16>(z) : z;
            }
            st_vec<VEC, BF16>(y, ((size_t)b * T + t) * C + c0, out);
        }
    }
    if (fin != nullptr && t1 == T) {
        // cache slot j holds xx at time T - W + j
        for (int j = 0; j < W; ++j) {
            float tmp[VEC];
            ld_xx<VEC, BF16>(tmp, x, cache, b, T - W + j, c0, T, C, W);
#pragma unroll
            for (int e = 0; e < VEC; ++e) st_io(fin, ((size_t)b * C + c0 + e) * W + j, BF16, tmp[e]);
        }
    }
}

// One decode token through n same-shaped convolutions (the q, k and v branches of a layer) in ONE launch: every cache
// row [W] is shifted by one, the new input appended, y = act(w . row) - the cache is updated IN PLACE.  Same arithmetic
// order as conv_fwd_kernel, so the result equals the non-mutating call bit for bit.
struct ConvStepItems {
    const void* x[4];
    const void* w[4];
    void* cache[4];
    void* y[4];
};

template <int W, bool BF16>
__global__ void __launch_bounds__(256) conv_step_kernel(int B, int C, int silu, int wf32, ConvStepItems items) {
    const int item = blockIdx.y;
    const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;      // b * C + c
    if (idx >= (size_t)B * C) return;
    const int c = (int)(idx % C);
    void* cache = items.cache[item];
    float xx[W];
#pragma unroll
    for (int j = 0; j + 1 < W; ++j) xx[j] = ld_io(cache, idx * W + j + 1, BF16);
    xx[W - 1] = ld_io(items.x[item], idx, BF16);
    float z = 0.f;
#pragma unroll
    for (int j = 0; j < W; ++j) z += ld_w(items.w[item], (size_t)c * W + j, BF16, wf32) * xx[j];
    st_io(items.y[item], idx, BF16, silu ? z * sigmoid_t<BF16>(z) : z);
#pragma unroll
    for (int j = 0; j < W; ++j) st_io(cache, idx * W + j, BF16, xx[j]);
}

// Lane = channel pair or quad, so every global access of a warp is one contiguous row segment; each thread slides the
// window over 8 consecutive tokens with all of its loads issued up front.
template <bool BF16>
__device__ __forceinline__ float2 ld_pair(const void* p, size_t i) {
    // read-only path: the inputs are never written by the kernel that reads them
    if (BF16) {
        const unsigned u = __ldg(reinterpret_cast<const unsigned*>(reinterpret_cast<const __nv_bfloat16*>(p) + i));
        return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u));
    }
    return __ldg(reinterpret_cast<const float2*>(reinterpret_cast<const float*>(p) + i));
}
template <bool BF16>
__device__ __forceinline__ void st_pair(void* p, size_t i, float a, float b) {
    if (BF16) *reinterpret_cast<__nv_bfloat162*>(reinterpret_cast<__nv_bfloat16*>(p) + i) = __floats2bfloat162_rn(a, b);
    else *reinterpret_cast<float2*>(reinterpret_cast<float*>(p) + i) = make_float2(a, b);
}

// N consecutive weights starting at element `base` (the W taps of N / W adjacent channels), with 16-byte loads when the
// run is 16-byte aligned: a warp then reads one contiguous span instead of 32 scattered words per tap.  The weights
// themselves are 16-byte aligned: the host sends any other to the kernels that read them with ld_weights.
template <int N, bool BF16>
__device__ __forceinline__ void ld_wrun(float (&flat)[N], const void* wgt, size_t base, int wf32) {
    const bool f32 = wf32 || !BF16;
    if (f32 && N % 4 == 0 && base % 4 == 0) {
#pragma unroll
        for (int j = 0; j < N / 4; ++j) {
            const float4 f = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(wgt) + base + 4 * j);
            flat[4 * j] = f.x; flat[4 * j + 1] = f.y; flat[4 * j + 2] = f.z; flat[4 * j + 3] = f.w;
        }
        if (BF16) {
#pragma unroll
            for (int j = 0; j < N; ++j) flat[j] = __bfloat162float(__float2bfloat16(flat[j]));
        }
    } else if (!f32 && N % 8 == 0 && base % 8 == 0) {
#pragma unroll
        for (int j = 0; j < N / 8; ++j) {
            float t[8];
            ld_vec<8, true>(t, wgt, base + 8 * j);
#pragma unroll
            for (int e = 0; e < 8; ++e) flat[8 * j + e] = t[e];
        }
    } else {
#pragma unroll
        for (int j = 0; j < N; ++j) flat[j] = ld_w(wgt, base + j, BF16, wf32);
    }
}

constexpr int kConvPairT = 8;    // tokens per thread

// VEC adjacent channels (2 or 4) as floats
template <int VEC, bool BF16>
__device__ __forceinline__ void ld_cvec(float (&d)[VEC], const void* p, size_t i) {
    if (VEC == 2) {
        const float2 v = ld_pair<BF16>(p, i);
        d[0] = v.x; d[1] = v.y;
    } else if (BF16) {
        const uint2 u = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(p) + i));
        const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
        const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
        d[0] = a.x; d[1] = a.y; d[2] = b.x; d[3] = b.y;
    } else {
        const float4 f = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + i));
        d[0] = f.x; d[1] = f.y; d[2] = f.z; d[3] = f.w;
    }
}
template <int VEC, bool BF16>
__device__ __forceinline__ void st_cvec(void* p, size_t i, const float (&s)[VEC]) {
    if (VEC == 2) {
        st_pair<BF16>(p, i, s[0], s[1]);
    } else if (BF16) {
        uint2 u;
        *reinterpret_cast<__nv_bfloat162*>(&u.x) = __floats2bfloat162_rn(s[0], s[1]);
        *reinterpret_cast<__nv_bfloat162*>(&u.y) = __floats2bfloat162_rn(s[2], s[3]);
        *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p) + i) = u;
    } else {
        *reinterpret_cast<float4*>(reinterpret_cast<float*>(p) + i) = make_float4(s[0], s[1], s[2], s[3]);
    }
}

// The same as channel pairs
template <int VEC, bool BF16>
__device__ __forceinline__ void ld_c2(f2 (&d)[VEC / 2], const void* p, size_t i) {
    if (BF16) {
        const __nv_bfloat16* b = reinterpret_cast<const __nv_bfloat16*>(p) + i;
        if (VEC == 2) {
            d[0] = f2_from_bf16(__ldg(reinterpret_cast<const unsigned*>(b)));
        } else {
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(b));
            d[0] = f2_from_bf16(u.x);
            d[VEC / 2 - 1] = f2_from_bf16(u.y);
        }
    } else {
        float x[VEC];
        ld_cvec<VEC, false>(x, p, i);
#pragma unroll
        for (int e = 0; e < VEC / 2; ++e) d[e] = f2_make(x[2 * e], x[2 * e + 1]);
    }
}
template <int VEC, bool BF16>
__device__ __forceinline__ void st_c2(void* p, size_t i, const f2 (&s)[VEC / 2]) {
    if (BF16) {
        __nv_bfloat16* b = reinterpret_cast<__nv_bfloat16*>(p) + i;
        if (VEC == 2) *reinterpret_cast<unsigned*>(b) = f2_to_bf16(s[0]);
        else *reinterpret_cast<uint2*>(b) = make_uint2(f2_to_bf16(s[0]), f2_to_bf16(s[VEC / 2 - 1]));
    } else {
        float x[VEC];
#pragma unroll
        for (int e = 0; e < VEC / 2; ++e) {
            const float2 v = f2_get(s[e]);
            x[2 * e] = v.x;
            x[2 * e + 1] = v.y;
        }
        st_cvec<VEC, false>(p, i, x);
    }
}
template <bool FAST>
__device__ __forceinline__ f2 sigmoid_2(f2 z) {
    if (FAST) {
        const f2 half = f2_all(0.5f);
        const float2 h = f2_get(f2_mul(half, z));
        float a, b;
        asm("tanh.approx.f32 %0, %1;" : "=f"(a) : "f"(h.x));
        asm("tanh.approx.f32 %0, %1;" : "=f"(b) : "f"(h.y));
        return f2_fma(half, f2_make(a, b), half);
    }
    const float2 x = f2_get(z);
    return f2_make(sigmoid_t<false>(x.x), sigmoid_t<false>(x.y));
}
// gy * d silu(z) / dz
template <bool FAST>
__device__ __forceinline__ f2 silu_vjp_2(f2 gy, f2 z) {
    const f2 one = f2_all(1.f), s = sigmoid_2<FAST>(z);
    return f2_mul(gy, f2_mul(s, f2_fma(z, f2_fma(s, f2_all(-1.f), one), one)));
}

// Gate activations, K % 4 == 0: a thread owns 4 adjacent channels (one head), so raw gate, bias, g and their gradients
// move as 8- / 16-byte accesses and the head's exp(A_log) is computed once for all of a thread's rows.
// Forward: quads of channels in memory order; n_thr is a multiple of a row's quads, and a thread takes quads i, i + n_thr, ..., four
// at most and all in its column, with every load in flight.  No lane is idle whatever the width: with blocks of 128 columns,
// narrower rows left lanes without work (200,000 x 8: 29 us, now 4.6).  Bound by issue (an exponential and a division an element)
// and bytes in about equal parts; one quad at a time, with an index division, the bias and exp(A_log) for each, it took 26.7 us at
// 8,191 x 2,048 bf16, now 21.0 (100 MB: 15 at the copy rate).  The four in one block of 32 rows: 22.6.
template <bool BF16>
__global__ void __launch_bounds__(256) gate_fwd4_kernel(unsigned n_thr, size_t n4, int tokens, int H, int K, const void* __restrict__ raw,
                                                        const void* __restrict__ bl, int bl_ld, const float* __restrict__ A_log,
                                                        const float* __restrict__ dt_bias, float lb, float* __restrict__ g,
                                                        float* __restrict__ beta) {
    const unsigned i = blockIdx.x * 256u + threadIdx.x;
    dependents_go();
    if (i >= n_thr) return;
    constexpr size_t quad = BF16 ? 8 : 16;
    const char* rp = static_cast<const char*>(raw) + i * quad;
    float* gp = g + (size_t)i * 4;
    const bool four = i + 3 * (size_t)n_thr < n4;
    float r[4][4];
    if (four) {
#pragma unroll
        for (int j = 0; j < 4; ++j) ld_cvec<4, BF16>(r[j], rp + j * (n_thr * quad), 0);
    } else {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (i + j * (size_t)n_thr < n4) ld_cvec<4, BF16>(r[j], rp + j * (n_thr * quad), 0);
    }
    // n_thr is a multiple of H too: a thread's beta logits, if it has any, belong to one head
    const bool has_beta = i < (size_t)tokens * H;
    unsigned bt = 0, bh = 0;
    float b0 = 0.f;
    if (has_beta) {
        bt = i / (unsigned)H;
        bh = i - bt * H;
        b0 = ld_io(bl, (size_t)bt * bl_ld + bh, BF16);
    }
    const unsigned c = i % ((unsigned)(H * K) >> 2) * 4;
    const float ea = expf(A_log[c / (unsigned)K]);
    const float4 bias = *reinterpret_cast<const float4*>(dt_bias + c);
    auto put = [&](int j) {
        float4 o;
        o.x = lb * sigmoidf_(ea * (r[j][0] + bias.x));
        o.y = lb * sigmoidf_(ea * (r[j][1] + bias.y));
        o.z = lb * sigmoidf_(ea * (r[j][2] + bias.z));
        o.w = lb * sigmoidf_(ea * (r[j][3] + bias.w));
        *reinterpret_cast<float4*>(gp + j * ((size_t)n_thr * 4)) = o;
    };
    if (four) {
#pragma unroll
        for (int j = 0; j < 4; ++j) put(j);
    } else {
#pragma unroll
        for (int j = 0; j < 3; ++j)
            if (i + j * (size_t)n_thr < n4) put(j);
    }
    if (has_beta) {
        beta[i] = sigmoidf_(b0);
        const unsigned rows = n_thr / (unsigned)H;
        for (size_t t = (size_t)bt + rows; t < (size_t)tokens; t += rows) beta[t * H + bh] = sigmoidf_(ld_io(bl, t * bl_ld + bh, BF16));
    }
    dependency_wait();      // not to end before a launch this one ran beside
}

// grid: x = blocks of 128 columns (lane = 4 channels), y = blocks of kGateRows tokens; warp w takes rows w, w + 8, ...
template <bool BF16>
__global__ void __launch_bounds__(256) gate_bwd4_kernel(int tokens, int H, int K, const void* __restrict__ raw,
                                                        const void* __restrict__ bl, int bl_ld, int bl_pad, const float* __restrict__ A_log,
                                                        const float* __restrict__ dt_bias, float lb, const float* __restrict__ dg,
                                                        const float* __restrict__ dbeta, void* __restrict__ d_raw,
                                                        void* __restrict__ d_bl, float* __restrict__ part_b,
                                                        float* __restrict__ part_a) {
    dependents_go();
    constexpr int RPW = kGateRows / 8;
    __shared__ float red[2][8][128];
    const int HK = H * K;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int c = (blockIdx.x * 32 + lane) * 4;
    const int t0 = blockIdx.y * kGateRows;
    const bool cok = c < HK;
    const int cl = cok ? c : 0;
    const float ea = expf(A_log[cl / K]);
    const float4 bias = *reinterpret_cast<const float4*>(dt_bias + cl);
    const float bz[4] = {bias.x, bias.y, bias.z, bias.w};
    float rv[RPW][4];
    float4 gv[RPW];
#pragma unroll
    for (int j = 0; j < RPW; ++j) {          // every load of the thread in flight at once
        const int t = min(t0 + w + 8 * j, tokens - 1);
        ld_cvec<4, BF16>(rv[j], raw, (size_t)t * HK + cl);
        gv[j] = __ldg(reinterpret_cast<const float4*>(dg + (size_t)t * HK + cl));
    }
    float sb[4] = {0.f, 0.f, 0.f, 0.f}, sa[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int j = 0; j < RPW; ++j) {
        const int t = t0 + w + 8 * j;
        if (t < tokens && cok) {
            const float gg[4] = {gv[j].x, gv[j].y, gv[j].z, gv[j].w};
            float dr[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float x = rv[j][e] + bz[e];
                const float sg = sigmoidf_(ea * x);
                dr[e] = gg[e] * lb * sg * (1.f - sg) * ea;
                sb[e] += dr[e];
                sa[e] += dr[e] * x;
            }
            st_cvec<4, BF16>(d_raw, (size_t)t * HK + c, dr);
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        red[0][w][4 * lane + e] = sb[e];
        red[1][w][4 * lane + e] = sa[e];
    }
    __syncthreads();
    if (threadIdx.x < 128 && blockIdx.x * 128 + threadIdx.x < HK) {
        float tb = 0.f, ta = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            tb += red[0][r][threadIdx.x];
            ta += red[1][r][threadIdx.x];
        }
        const size_t o = (size_t)blockIdx.y * HK + blockIdx.x * 128 + threadIdx.x;
        part_b[o] = tb;
        part_a[o] = ta;
    }
    if (blockIdx.x == 0) {                  // beta logits of this block's rows
        // rows bl_ld apart; columns H .. H + bl_pad - 1 of d_bl pad a wider matrix and are zeroed
        const int wide = H + bl_pad, nb = min(kGateRows, tokens - t0) * wide;
        for (int i = threadIdx.x; i < nb; i += 256) {
            const int t = t0 + i / wide, h = i % wide;
            const size_t o = (size_t)t * bl_ld + h;
            float d = 0.f;
            if (h < H) {
                const float b = sigmoidf_(ld_io(bl, o, BF16));
                d = dbeta[(size_t)t * H + h] * b * (1.f - b);
            }
            st_io(d_bl, o, BF16, d);
        }
    }
}

// Up to kConvItems same-shaped convolutions (the q, k and v branches of a layer) share one launch: blockIdx.z runs over
// item x batch.
constexpr int kConvItems = 4;
struct ConvFwdItems {
    const void* x[kConvItems];
    const void* w[kConvItems];
    void* y[kConvItems];
    const void* cache[kConvItems];     // carried-in windows [B][C][W], or null: zeros before the first token
    void* fin[kConvItems];             // carried-out windows [B][C][W], or null
};
struct ConvBwdItems {
    const void* x[kConvItems];
    const void* w[kConvItems];
    const void* dy[kConvItems];
    void* dx[kConvItems];
};
struct ColumnSumItems {
    void* out[kConvItems];
};
// Entry i of a kernel-parameter array by compile-time indices only: a run-time subscript would make every thread copy the
// whole array to local memory first.
template <class T>
__device__ __forceinline__ T pick_item(T const (&a)[kConvItems], int i) {
    T r = a[0];
    if (i == 1) r = a[1];
    if (i == 2) r = a[2];
    if (i == 3) r = a[3];
    return r;
}

// grid: x = channel blocks of 32*VEC, y = blocks of 8 time groups x kConvPairT tokens, z = item * B + batch.  x rows are
// ldx elements apart (a slice of a wider projection), y rows are dense.  WIN: a window is carried in or out; only the
// threads at either end of a sequence touch it.  The kernel moves 2 x B x T x C elements and is bound by instruction issue
// at 0.63 of the copy rate (129 us at 65,536 x 2,048 bf16; long inputs take the streaming kernel below); the windows used
// to go through a 4-token, 8-channel kernel whose lanes read 16-byte pieces of strided rows: 78 us at 8,191 x 2,048, now 22.
template <int W, int VEC, bool BF16, bool WIN>
__global__ void __launch_bounds__(256) conv_fwd_pair_kernel(int B, int T, int C, int ldx, int silu, int wf32, ConvFwdItems items) {
    const int p = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int c = (blockIdx.x * 32 + p) * VEC;
    const int item = blockIdx.z / B;
    const int t0 = (blockIdx.y * 8 + g) * kConvPairT, b = blockIdx.z - item * B;
    dependents_go();
    if (t0 >= T) return;
    const void* __restrict__ x = pick_item(items.x, item);
    const void* __restrict__ wgt = pick_item(items.w, item);
    void* __restrict__ y = pick_item(items.y, item);
    const bool cok = c < C;
    const int cl = cok ? c : 0;
    f2 wv[W][VEC / 2];
    {
        float flat[W * VEC];
        ld_wrun<W * VEC, BF16>(flat, wgt, (size_t)cl * W, wf32);
#pragma unroll
        for (int e = 0; e < VEC / 2; ++e)
#pragma unroll
            for (int m = 0; m < W; ++m) wv[m][e] = f2_make(flat[2 * e * W + m], flat[(2 * e + 1) * W + m]);
    }
    const size_t rowbase = (size_t)b * T;
    f2 xin[kConvPairT + W - 1][VEC / 2];
    if (t0 >= W - 1 && t0 + kConvPairT <= T) {
        // interior: plain address arithmetic, every load independent
        const size_t base = (rowbase + t0 - (W - 1)) * ldx + cl;
#pragma unroll
        for (int j = 0; j < kConvPairT + W - 1; ++j) ld_c2<VEC, BF16>(xin[j], x, base + (size_t)j * ldx);
    } else {
#pragma unroll
        for (int j = 0; j < kConvPairT + W - 1; ++j) {
            const int t = t0 - (W - 1) + j;
            const int tc = min(max(t, 0), T - 1);
            ld_c2<VEC, BF16>(xin[j], x, (rowbase + tc) * ldx + cl);
            if (t < 0 || t >= T) {
#pragma unroll
                for (int e = 0; e < VEC / 2; ++e) xin[j][e] = f2_all(0.f);
            }
        }
        if (WIN && t0 < W - 1) {
            const void* cache = pick_item(items.cache, item);      // slot s holds the input at time s - W
            if (cache != nullptr) {
#pragma unroll
                for (int j = 0; j < W - 1; ++j) {
                    const int t = t0 - (W - 1) + j;
                    if (t < 0) {
#pragma unroll
                        for (int e = 0; e < VEC / 2; ++e) {
                            const size_t slot = ((size_t)b * C + cl + 2 * e) * W + W + t;
                            xin[j][e] = f2_make(ld_io(cache, slot, BF16), ld_io(cache, slot + W, BF16));
                        }
                    }
                }
            }
        }
    }
#pragma unroll
    for (int tt = 0; tt < kConvPairT; ++tt) {
        f2 out[VEC / 2];
#pragma unroll
        for (int e = 0; e < VEC / 2; ++e) {
            f2 z = f2_mul(wv[0][e], xin[tt][e]);
#pragma unroll
            for (int m = 1; m < W; ++m) z = f2_fma(wv[m][e], xin[tt + m][e], z);
            out[e] = silu ? f2_mul(z, sigmoid_2<BF16>(z)) : z;
        }
        if (t0 + tt < T && cok) st_c2<VEC, BF16>(y, (rowbase + t0 + tt) * C + c, out);
    }
    if (WIN && cok && (t0 + kConvPairT > T - W || t0 == 0)) {
        void* fin = pick_item(items.fin, item);                    // slot s holds the input at time T - W + s
        if (fin != nullptr) {
#pragma unroll
            for (int tt = 0; tt < kConvPairT; ++tt) {
                const int t = t0 + tt, s = t - (T - W);
                if (t < T && s >= 0) {
#pragma unroll
                    for (int e = 0; e < VEC / 2; ++e) {
                        const float2 v = f2_get(xin[tt + W - 1][e]);
                        st_io(fin, ((size_t)b * C + c + 2 * e) * W + s, BF16, v.x);
                        st_io(fin, ((size_t)b * C + c + 2 * e + 1) * W + s, BF16, v.y);
                    }
                }
            }
            if (t0 == 0 && T < W) {                                // a sequence shorter than the window keeps what was carried in
                const void* cache = pick_item(items.cache, item);
                for (int s = 0; s < W - T; ++s)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) {
                        const size_t row = ((size_t)b * C + c + e) * W;
                        st_io(fin, row + s, BF16, cache != nullptr ? ld_io(cache, row + T + s, BF16) : 0.f);
                    }
            }
        }
    }
    dependency_wait();                         // not to end before a launch this one ran beside
}

// The same for long bf16 inputs, C % 128 == 0: a thread walks down a run of tokens, 8 rows at a
// time, and loads the next 8 rows before it computes on the present ones, so that reads stay in flight and the W-1 halo
// rows are read once per run instead of once per 8 tokens.  65,536 x 2,048: 129 -> 96 us (0.86 of the copy rate); with two
// blocks per SM instead of three it takes 108.  A window that is only carried out
// (a prompt from an empty state) is a copy of the last W rows, by one more block row of the grid (fin_row; -1: none); in the
// runs themselves it cost every thread registers (49 -> 57 us at 3 x 8,191 x 2,048).
template <int W>
__global__ void __launch_bounds__(256, W <= 4 ? 3 : 2) conv_fwd_stream_kernel(int B, int T, int C, int ldx, int run, int fin_row, int silu, int wf32, ConvFwdItems items) {
    constexpr int R = 8;                                       // run is a multiple of 2 R
    const int p = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int c = (blockIdx.x * 32 + p) * 4;                   // C % 128 == 0: in range
    const int item = blockIdx.z / B, b = blockIdx.z - item * B;
    dependents_go();
    if ((int)blockIdx.y == fin_row) {                          // slot s holds the input at time T - W + s
        const int t = T - W + g;
        __nv_bfloat16* fin = static_cast<__nv_bfloat16*>(pick_item(items.fin, item));
        if (g < W && fin != nullptr) {
            uint2 u = make_uint2(0u, 0u);
            if (t >= 0) u = __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(pick_item(items.x, item)) + ((size_t)b * T + t) * ldx + c));
            const __nv_bfloat162 lo = *reinterpret_cast<const __nv_bfloat162*>(&u.x), hi = *reinterpret_cast<const __nv_bfloat162*>(&u.y);
            __nv_bfloat16* o = fin + ((size_t)b * C + c) * W + g;
            o[0] = lo.x;
            o[W] = lo.y;
            o[2 * W] = hi.x;
            o[3 * W] = hi.y;
        }
        return;
    }
    const int t0 = (blockIdx.y * 8 + g) * run;
    if (t0 >= T) return;
    const void* __restrict__ wgt = pick_item(items.w, item);
    f2 wv[W][2];
    {
        float flat[W * 4];
        ld_wrun<W * 4, true>(flat, wgt, (size_t)c * W, wf32);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int m = 0; m < W; ++m) wv[m][e] = f2_make(flat[2 * e * W + m], flat[(2 * e + 1) * W + m]);
    }
    const __nv_bfloat16* __restrict__ xp = static_cast<const __nv_bfloat16*>(pick_item(items.x, item)) + ((size_t)b * T + t0) * ldx + c;
    __nv_bfloat16* __restrict__ yp = static_cast<__nv_bfloat16*>(pick_item(items.y, item)) + ((size_t)b * T + t0) * C + c;
    const int n = min(run, T - t0);
    f2 xw[W][2];                                               // rows t - (W-1) .. t as a circular buffer: row t in slot t % W
#pragma unroll
    for (int m = 1; m < W; ++m) {
        xw[W - m][0] = xw[W - m][1] = f2_all(0.f);
        if (t0 > 0) {                                          // then t0 >= run >= W: every halo row exists
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(xp - (size_t)m * ldx));
            xw[W - m][0] = f2_from_bf16(u.x);
            xw[W - m][1] = f2_from_bf16(u.y);
        }
    }
    auto load = [&](uint2 (&d)[R], int i) {                    // rows i .. i + R - 1 of the run; past its end nothing
        if (i + R <= n) {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                d[r] = __ldg(reinterpret_cast<const uint2*>(xp));
                xp += ldx;
            }
        } else {
#pragma unroll
            for (int r = 0; r < R; ++r) {
                if (i + r < n) {
                    d[r] = __ldg(reinterpret_cast<const uint2*>(xp));
                    xp += ldx;
                }
            }
        }
    };
    auto rows = [&](const uint2 (&d)[R], int i, auto full) {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            if (!decltype(full)::value && i + r >= n) break;
            const int s = r % W;
            xw[s][0] = f2_from_bf16(d[r].x);
            xw[s][1] = f2_from_bf16(d[r].y);
            f2 out[2];
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                f2 z = f2_mul(wv[0][e], xw[(s + 1) % W][e]);   // x[t - (W-1) + m]
#pragma unroll
                for (int m = 1; m < W; ++m) z = f2_fma(wv[m][e], xw[(s + 1 + m) % W][e], z);
                out[e] = silu ? f2_mul(z, sigmoid_2<true>(z)) : z;
            }
            st_c2<4, true>(yp, 0, out);
            yp += C;
        }
        if constexpr (R % W != 0) {                            // rotate, so that the next block starts at slot 0 again
            f2 k[W][2];
#pragma unroll
            for (int m = 0; m < W; ++m) { k[m][0] = xw[(m + R) % W][0]; k[m][1] = xw[(m + R) % W][1]; }
#pragma unroll
            for (int m = 0; m < W; ++m) { xw[m][0] = k[m][0]; xw[m][1] = k[m][1]; }
        }
    };
    auto block = [&](const uint2 (&d)[R], int i) {
        if (i + R <= n) rows(d, i, std::true_type());
        else rows(d, i, std::false_type());
    };
    uint2 da[R], db[R];
    load(da, 0);
#pragma unroll 1
    for (int i = 0; i < n; i += 2 * R) {
        load(db, i + R);
        block(da, i);
        load(da, i + 2 * R);
        block(db, i + R);
    }
    dependency_wait();                                         // not to end before a launch this one ran beside
}

// Backward.  blockDim = (16 channel groups, 16 time tiles).  Each thread recomputes the
// pre-activations of its tile plus W-1 following tokens, emits dx for its tile and a
// register partial of dweight; the 8 tiles of a block are summed in shared memory and
// written as one partial per block, reduced in fixed order by column_sum_kernel.
constexpr int kConvBT = 4;   // tokens per thread in the backward

template <int W, int VEC, bool BF16>
__global__ void __launch_bounds__(256) conv_bwd_kernel(int B, int T, int C, int silu, int wf32, const void* __restrict__ x,
                                                       const void* __restrict__ wgt, const void* __restrict__ cache,
                                                       const void* __restrict__ dy, const void* __restrict__ dfin,
                                                       void* __restrict__ dx, void* __restrict__ dcache,
                                                       float* __restrict__ dw_part) {
    dependents_go();
    __shared__ float red[16][16][W * VEC];
    const int ncg = C / VEC, ntile = (T + kConvBT - 1) / kConvBT;
    const int cg = blockIdx.x * 16 + threadIdx.x;
    const int tile = blockIdx.y * 16 + threadIdx.y;
    const int b = blockIdx.z;
    const bool active = cg < ncg && tile < ntile;
    float dwv[W][VEC];
#pragma unroll
    for (int j = 0; j < W; ++j)
#pragma unroll
        for (int e = 0; e < VEC; ++e) dwv[j][e] = 0.f;
    if (active) {
        const int c0 = cg * VEC, t0 = tile * kConvBT, t1 = min(T, t0 + kConvBT);
        float wv[W][VEC];
        ld_weights<W, VEC, BF16>(wv, wgt, c0, wf32);
        if (t0 >= W - 1 && t0 + kConvBT + W <= T) {
            // interior tile: every load is unconditional and independent, then pure register arithmetic
            float xin[kConvBT + 2 * (W - 1)][VEC];   // x at t0-(W-1) .. t0+kConvBT+W-2
            float gy[kConvBT + W - 1][VEC];          // dy, then dz, at t0 .. t0+kConvBT+W-2
#pragma unroll
            for (int j = 0; j < kConvBT + 2 * (W - 1); ++j)
                ld_vec<VEC, BF16>(xin[j], x, ((size_t)b * T + (t0 - (W - 1) + j)) * C + c0);
#pragma unroll
            for (int j = 0; j < kConvBT + W - 1; ++j) ld_vec<VEC, BF16>(gy[j], dy, ((size_t)b * T + t0 + j) * C + c0);
#pragma unroll
            for (int j = 0; j < kConvBT + W - 1; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    float z = 0.f;
#pragma unroll
                    for (int m = 0; m < W; ++m) z += wv[m][e] * xin[j + m][e];
                    if (silu) {
                        const float sg = sigmoid_t<BF16>(z);
                        gy[j][e] *= sg * (1.f + z * (1.f - sg));
                    }
                }
#pragma unroll
            for (int j = 0; j < kConvBT; ++j) {
                float out[VEC];
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    float a = 0.f;
#pragma unroll
                    for (int m = 0; m < W; ++m) {
                        a += wv[m][e] * gy[j + W - 1 - m][e];
                        dwv[m][e] += gy[j][e] * xin[j + m][e];
                    }
                    out[e] = a;
                }
                st_vec<VEC, BF16>(dx, ((size_t)b * T + t0 + j) * C + c0, out);
            }
        } else {
        float win[W][VEC];   // xx window ending at the token whose dz is being produced
        float dzw[W][VEC];   // dzw[m] = dz at token (cur - (W-1) + m)
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
            for (int e = 0; e < VEC; ++e) dzw[j][e] = 0.f;
#pragma unroll
        for (int j = 0; j < W - 1; ++j) ld_xx<VEC, BF16>(win[j + 1], x, cache, b, t0 - (W - 1) + j, c0, T, C, W);
        // walk cur over [t0, t1 + W - 1): produce dz[cur]; once W-1 tokens ahead, emit dx[cur - (W-1)]
#pragma unroll
        for (int step = 0; step < kConvBT + W - 1; ++step) {
            const int cur = t0 + step;
            if (cur >= t1 + W - 1) break;
#pragma unroll
            for (int j = 0; j < W - 1; ++j)
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    win[j][e] = win[j + 1][e];
                    dzw[j][e] = dzw[j + 1][e];
                }
            if (cur < T) {
                ld_vec<VEC, BF16>(win[W - 1], x, ((size_t)b * T + cur) * C + c0);
                float g[VEC];
                ld_vec<VEC, BF16>(g, dy, ((size_t)b * T + cur) * C + c0);
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    float z = 0.f;
#pragma unroll
                    for (int j = 0; j < W; ++j) z += wv[j][e] * win[j][e];
                    if (silu) {
                        const float sg = sigmoid_t<BF16>(z);
                        g[e] *= sg * (1.f + z * (1.f - sg));
                    }
                    dzw[W - 1][e] = g[e];
                    if (cur < t1) {
#pragma unroll
                        for (int j = 0; j < W; ++j) dwv[j][e] += g[e] * win[j][e];
                    }
                }
            } else {
#pragma unroll
                for (int e = 0; e < VEC; ++e) { dzw[W - 1][e] = 0.f; win[W - 1][e] = 0.f; }
            }
            const int t = cur - (W - 1);     // dx[t] = sum_j w[j] dz[t + W-1-j] = sum_j w[j] dzw[W-1-j]
            if (t >= t0 && t < t1) {
                float out[VEC];
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    float a = 0.f;
#pragma unroll
                    for (int j = 0; j < W; ++j) a += wv[j][e] * dzw[W - 1 - j][e];
                    if (dfin != nullptr && t >= T - W) a += ld_io(dfin, ((size_t)b * C + c0 + e) * W + (W + t - T), BF16);
                    out[e] = a;
                }
                st_vec<VEC, BF16>(dx, ((size_t)b * T + t) * C + c0, out);
            }
        }
        }   // guarded (boundary) path
        if (dcache != nullptr && tile == 0) {
            // cache slot p is time p - W (< 0): d = sum_j w[j] dz[p - W + W-1-j] = sum_j w[j] dz[p-1-j], plus the
            // final-state cotangent when the sequence is shorter than the window.  Needs dz[0 .. W-2]: recompute.
            float dz0[W][VEC];
#pragma unroll
            for (int m = 0; m < W; ++m)
#pragma unroll
                for (int e = 0; e < VEC; ++e) dz0[m][e] = 0.f;
            float w2[W][VEC];
#pragma unroll
            for (int j = 0; j < W - 1; ++j) ld_xx<VEC, BF16>(w2[j + 1], x, cache, b, -(W - 1) + j, c0, T, C, W);
            for (int t = 0; t < W - 1 && t < T; ++t) {
#pragma unroll
                for (int j = 0; j < W - 1; ++j)
#pragma unroll
                    for (int e = 0; e < VEC; ++e) w2[j][e] = w2[j + 1][e];
                ld_vec<VEC, BF16>(w2[W - 1], x, ((size_t)b * T + t) * C + c0);
                float g[VEC];
                ld_vec<VEC, BF16>(g, dy, ((size_t)b * T + t) * C + c0);
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    float z = 0.f;
#pragma unroll
                    for (int j = 0; j < W; ++j) z += wv[j][e] * w2[j][e];
                    if (silu) {
                        const float sg = sigmoid_t<BF16>(z);
                        g[e] *= sg * (1.f + z * (1.f - sg));
                    }
#pragma unroll
                    for (int m = 0; m < W; ++m)
                        if (m == t) dz0[m][e] = g[e];
                }
            }
#pragma unroll
            for (int p = 0; p < W; ++p)
#pragma unroll
                for (int e = 0; e < VEC; ++e) {
                    float a = 0.f;
#pragma unroll
                    for (int j = 0; j < W; ++j) {
                        const int m = p - 1 - j;
                        if (m >= 0 && m < W) a += wv[j][e] * dz0[m][e];
                    }
                    if (dfin != nullptr && p - T >= 0) a += ld_io(dfin, ((size_t)b * C + c0 + e) * W + (p - T), BF16);
                    st_io(dcache, ((size_t)b * C + c0 + e) * W + p, BF16, a);
                }
        }
    }
#pragma unroll
    for (int j = 0; j < W; ++j)
#pragma unroll
        for (int e = 0; e < VEC; ++e) red[threadIdx.y][threadIdx.x][j * VEC + e] = dwv[j][e];
    __syncthreads();
    if (threadIdx.y == 0 && cg < ncg) {
        const size_t pblk = (size_t)blockIdx.z * gridDim.y + blockIdx.y;
#pragma unroll
        for (int j = 0; j < W; ++j)
#pragma unroll
            for (int e = 0; e < VEC; ++e) {
                float a = 0.f;
#pragma unroll
                for (int r = 0; r < 16; ++r) a += red[r][threadIdx.x][j * VEC + e];
                dw_part[(pblk * C + cg * VEC + e) * W + j] = a;
            }
    }
}

// Backward without a carried-in window (no initial state, no final-state cotangent: the training path).  One block
// owns 64 tokens x 64 channels.  It stages x (with a W-1 halo on both sides) and dy (W-1 halo after) in shared memory
// as float pairs, turns dy into dz in place (each pre-activation is recomputed once, not once per window position),
// then forms dx from the dz window and the block's dweight partial.  Lane = channel pair, so every global access of a
// warp is one contiguous row segment; warp = row group.
constexpr int kConvTileT = 64, kConvTileC = 64;

template <int W, bool BF16>
__global__ void __launch_bounds__(256) conv_bwd_tile_kernel(int B, int T, int C, int ldx, int silu, int wf32, ConvBwdItems items,
                                                            float* __restrict__ dw_part) {
    dependents_go();
    constexpr int XR = kConvTileT + 2 * (W - 1);   // x rows  t0-(W-1) .. t0+63+(W-1)
    constexpr int GR = kConvTileT + W - 1;         // dy rows t0 .. t0+63+(W-1)
    constexpr int RPW = kConvTileT / 8;            // consecutive rows per warp
    // x stays in its storage type (a bf16 pair is one 32-bit word); dy is widened because dz replaces it in place
    typedef typename std::conditional<BF16, __nv_bfloat162, float2>::type xpair_t;
    __shared__ __align__(16) xpair_t xs[XR][32];
    __shared__ __align__(16) float2 gs[GR][32];
    __shared__ __align__(16) float red[8][W][kConvTileC];
    const int p = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int cb = blockIdx.x * kConvTileC;
    const int c = cb + 2 * p;
    const int item = blockIdx.z / B;
    const int t0 = blockIdx.y * kConvTileT, b = blockIdx.z - item * B;
    const void* __restrict__ x = pick_item(items.x, item);
    const void* __restrict__ wgt = pick_item(items.w, item);
    const void* __restrict__ dy = pick_item(items.dy, item);
    void* __restrict__ dx = pick_item(items.dx, item);
    const bool cok = c < C;
    const int cl = cok ? c : 0;                    // loads stay unconditional: out-of-range lanes read column 0 and are masked
    f2 wv[W];
    {
        float flat[2 * W];
        ld_wrun<2 * W, BF16>(flat, wgt, (size_t)cl * W, wf32);
#pragma unroll
        for (int m = 0; m < W; ++m) wv[m] = f2_make(flat[m], flat[W + m]);
    }
    const size_t rowbase = (size_t)b * T;
    auto xload = [&](int tc) -> xpair_t {
        if constexpr (BF16) {
            const unsigned u = __ldg(reinterpret_cast<const unsigned*>(reinterpret_cast<const __nv_bfloat16*>(x) + (rowbase + tc) * ldx + cl));
            return *reinterpret_cast<const __nv_bfloat162*>(&u);
        } else {
            return __ldg(reinterpret_cast<const float2*>(reinterpret_cast<const float*>(x) + (rowbase + tc) * ldx + cl));
        }
    };
    auto xwide = [](const xpair_t& v) -> f2 {
        if constexpr (BF16) return f2_from_bf16(*reinterpret_cast<const unsigned*>(&v));
        else return f2_make(v.x, v.y);
    };
    if (t0 >= W - 1 && t0 + GR <= T && cb + kConvTileC <= C && (C & 3) == 0 && (ldx & 3) == 0) {
        // interior tile: no clamping, four channels per thread (sixteen threads cover a 64-channel row, a warp two rows),
        // addresses advance by a constant stride
        const int q = threadIdx.x & 15, rg = threadIdx.x >> 4;
        const size_t e0 = (rowbase + t0 - (W - 1) + rg) * ldx + cb + 4 * q;       // x row rg of the tile, this thread's channels
        const size_t xstep = (size_t)16 * ldx, step = (size_t)16 * C;
#pragma unroll
        for (int it = 0; it < (XR + 15) / 16; ++it) {
            const int r = rg + 16 * it;
            if (r < XR) {
                if constexpr (BF16) {
                    const uint2 u = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(x) + e0 + it * xstep));
                    *reinterpret_cast<uint2*>(&xs[r][2 * q]) = u;
                } else {
                    const float4 f = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + e0 + it * xstep));
                    *reinterpret_cast<float4*>(&xs[r][2 * q]) = f;
                }
            }
        }
        const size_t g0 = (rowbase + t0 + rg) * C + cb + 4 * q;
#pragma unroll
        for (int it = 0; it < (GR + 15) / 16; ++it) {
            const int r = rg + 16 * it;
            if (r < GR) {
                float4 f;
                if constexpr (BF16) {
                    const uint2 u = __ldg(reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(dy) + g0 + it * step));
                    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
                    const float2 b2 = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
                    f = make_float4(a.x, a.y, b2.x, b2.y);
                } else {
                    f = __ldg(reinterpret_cast<const float4*>(reinterpret_cast<const float*>(dy) + g0 + it * step));
                }
                *reinterpret_cast<float4*>(&gs[r][2 * q]) = f;
            }
        }
    } else {
#pragma unroll
        for (int r = g; r < XR; r += 8) {
            const int t = t0 - (W - 1) + r;
            xpair_t v = xload(min(max(t, 0), T - 1));
            if (t < 0 || t >= T || !cok) v = xpair_t();
            xs[r][p] = v;
        }
#pragma unroll
        for (int r = g; r < GR; r += 8) {
            const int t = t0 + r;
            float2 v = ld_pair<BF16>(dy, (rowbase + min(t, T - 1)) * C + cl);
            if (t >= T || !cok) v = make_float2(0.f, 0.f);
            gs[r][p] = v;
        }
    }
    __syncthreads();
    f2 dw[W];
#pragma unroll
    for (int m = 0; m < W; ++m) dw[m] = f2_all(0.f);
    // dz for rows r0 .. r0+n-1, walking down with the x window in registers; dweight only from the tile's own rows
    auto dz_rows = [&](int r0, int n, bool own) {
        f2 xw[W];
#pragma unroll
        for (int m = 0; m < W - 1; ++m) xw[m] = xwide(xs[r0 + m][p]);
#pragma unroll
        for (int i = 0; i < RPW; ++i) {
            if (i < n) {
                const int r = r0 + i;
                xw[W - 1] = xwide(xs[r + W - 1][p]);
                f2* gp = reinterpret_cast<f2*>(&gs[r][p]);
                f2 gy = *gp;
                if (silu) {
                    f2 z = f2_mul(wv[0], xw[0]);
#pragma unroll
                    for (int m = 1; m < W; ++m) z = f2_fma(wv[m], xw[m], z);
                    gy = silu_vjp_2<BF16>(gy, z);
                    *gp = gy;                      // dz; element (r, p) is touched by this thread only
                }
                if (own) {
#pragma unroll
                    for (int m = 0; m < W; ++m) dw[m] = f2_fma(gy, xw[m], dw[m]);
                }
#pragma unroll
                for (int m = 0; m < W - 1; ++m) xw[m] = xw[m + 1];
            }
        }
    };
    dz_rows(g * RPW, RPW, true);
    if (g < W - 1) dz_rows(kConvTileT + g, 1, false);   // halo rows: their dweight belongs to the next block
#pragma unroll
    for (int m = 0; m < W; ++m) *reinterpret_cast<f2*>(&red[g][m][2 * p]) = dw[m];
    __syncthreads();
    // dx[t] = sum_m w[m] dz[t + W-1-m], again with a register window over this warp's consecutive rows
    {
        const int r0 = g * RPW;
        f2 dzw[W];
#pragma unroll
        for (int m = 0; m < W - 1; ++m) dzw[m] = *reinterpret_cast<const f2*>(&gs[r0 + m][p]);
#pragma unroll
        for (int i = 0; i < RPW; ++i) {
            const int r = r0 + i, t = t0 + r;
            dzw[W - 1] = *reinterpret_cast<const f2*>(&gs[r + W - 1][p]);
            f2 a[1] = {f2_mul(wv[0], dzw[W - 1])};
#pragma unroll
            for (int m = 1; m < W; ++m) a[0] = f2_fma(wv[m], dzw[W - 1 - m], a[0]);
            if (t < T && cok) st_c2<2, BF16>(dx, (rowbase + t) * ldx + c, a);
#pragma unroll
            for (int m = 0; m < W - 1; ++m) dzw[m] = dzw[m + 1];
        }
    }
    if (threadIdx.x < kConvTileC && cb + threadIdx.x < C) {
        const size_t pblk = (size_t)blockIdx.z * gridDim.y + blockIdx.y;
#pragma unroll
        for (int m = 0; m < W; ++m) {
            float a = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) a += red[r][m][threadIdx.x];
            dw_part[(pblk * C + cb + threadIdx.x) * W + m] = a;
        }
    }
}

// Backward, training path, bf16 with C % 128 == 0.  A thread owns 4 adjacent channels and a run of consecutive tokens
// and streams down its rows once: x and dy rows arrive through a thread-private ring in shared memory filled by
// asynchronous 8-byte copies up to kConvRingDepth rows ahead (no registers held for data in flight, no block-wide barrier
// in the loop), the x window and the dz window live in registers as circular buffers with compile-time indices, and every
// pre-activation, SiLU derivative, dweight and dx multiply-add is done exactly once per element.  Only the W-1 rows
// either side of a run are touched twice.  Block = 8 warps = 8 runs x 128 channels; one dweight partial per block.
// Moves 3 x B x T x C elements and was bound by instruction issue (0.47 of the copy rate): channel pairs in packed
// arithmetic, one copy group per W rows, pointers that walk, and two blocks per SM (at three, 80 registers a thread
// spilled inside the loop): 266 -> 170 us at 65,536 x 2,048, 0.72 of the copy rate.  A ring of 24 rows gave 175.
constexpr int kConvRingDepth = 16;

template <int W>
__global__ void __launch_bounds__(256, 2) conv_bwd_ring_kernel(int B, int T, int C, int ldx, int run, int silu, int wf32, ConvBwdItems items,
                                                               float* __restrict__ dw_part) {
    dependents_go();
    constexpr int NG = kConvRingDepth / W;                     // groups of W rows in the ring
    extern __shared__ __align__(16) uint8_t ring_raw[];
    uint2* ring = reinterpret_cast<uint2*>(ring_raw);          // [NG][W][2: x | dy][256 threads]
    float (*red)[W][128] = reinterpret_cast<float (*)[W][128]>(ring_raw);      // [8][W][128], once the ring is drained
    const int p = threadIdx.x & 31, g = threadIdx.x >> 5;
    const int c = (blockIdx.x * 32 + p) * 4;                   // C % 128 == 0: in range
    const int item = blockIdx.z / B, b = blockIdx.z - item * B;
    const int t0 = (blockIdx.y * 8 + g) * run;
    const __nv_bfloat16* __restrict__ x = static_cast<const __nv_bfloat16*>(pick_item(items.x, item));
    const void* __restrict__ wgt = pick_item(items.w, item);
    const __nv_bfloat16* __restrict__ dy = static_cast<const __nv_bfloat16*>(pick_item(items.dy, item));
    __nv_bfloat16* __restrict__ dx = static_cast<__nv_bfloat16*>(pick_item(items.dx, item));
    f2 wv[W][2], dwv[W][2];
    {
        float flat[W * 4];
        ld_wrun<W * 4, true>(flat, wgt, (size_t)c * W, wf32);
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int m = 0; m < W; ++m) {
                wv[m][e] = f2_make(flat[2 * e * W + m], flat[(2 * e + 1) * W + m]);
                dwv[m][e] = f2_all(0.f);
            }
    }
    if (t0 < T) {
        // stream step j handles token tx = t0 - (W-1) + j: x[tx] enters the window; from tx >= t0 on dz[tx] is formed;
        // from tx >= t0 + W-1 on dx[tx - (W-1)] leaves.  Steps run to a multiple of W so the circular indices are static.
        const int nr = ((run + 2 * (W - 1) + W - 1) / W) * W;
        const size_t rowbase = (size_t)b * T;
        const uint32_t slot0 = (uint32_t)__cvta_generic_to_shared(ring + threadIdx.x);
        // the source pointers walk down the rows: a row outside the sequence reads its nearest row inside and is masked
        const __nv_bfloat16* xp = x + (rowbase + max(t0 - (W - 1), 0)) * ldx + c;
        const __nv_bfloat16* gp = dy + (rowbase + max(t0 - (W - 1), 0)) * C + c;
        __nv_bfloat16* dp = dx + (rowbase + t0) * ldx + c;
        int jn = 0, sn = 0;                                    // next group to fetch: its first step, its slot
        auto fetch = [&]() {
            if (jn < nr) {
                const uint32_t dst = slot0 + (uint32_t)sn * (W * 2 * 256 * 8);
                const int tx = t0 - (W - 1) + jn;
                const bool inner = tx >= 0 && tx + W < T;
#pragma unroll
                for (int u = 0; u < W; ++u) {
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + (2 * u) * 256 * 8), "l"(xp) : "memory");
                    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(dst + (2 * u + 1) * 256 * 8), "l"(gp) : "memory");
                    if (inner || (unsigned)(tx + u) < (unsigned)(T - 1)) {
                        xp += ldx;
                        gp += C;
                    }
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
            jn += W;
            sn = sn + 1 == NG ? 0 : sn + 1;
        };
#pragma unroll 1
        for (int i = 0; i < NG - 1; ++i) fetch();
        f2 xc[W][2], dzc[W][2];
#pragma unroll
        for (int m = 0; m < W; ++m)
#pragma unroll
            for (int e = 0; e < 2; ++e) xc[m][e] = dzc[m][e] = f2_all(0.f);
        // EDGE: rows outside the sequence or the run need their masks; the steps in the middle of a run inside the sequence
        // (all but the first and last few) run without them
        auto step = [&](int jj, int slot, auto edge) {
            constexpr bool EDGE = decltype(edge)::value;
            const uint2* rp = ring + slot * (W * 2 * 256) + threadIdx.x;
#pragma unroll
            for (int u = 0; u < W; ++u) {
                const int tx = t0 - (W - 1) + jj + u;
                const uint2 xr = rp[(2 * u) * 256];
                const uint2 gr = rp[(2 * u + 1) * 256];
                xc[u][0] = f2_from_bf16(xr.x);
                xc[u][1] = f2_from_bf16(xr.y);
                f2 gy[2] = {f2_from_bf16(gr.x), f2_from_bf16(gr.y)};
                if (EDGE && (tx < 0 || tx >= T)) xc[u][0] = xc[u][1] = f2_all(0.f);
                const bool live = !EDGE || (tx >= t0 && tx < T);              // dz[tx] exists and belongs to this run's window
                const bool own = !EDGE || (live && tx < t0 + run);            // ... and its dweight is this run's
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    if (silu) {
                        f2 z = f2_mul(wv[0][e], xc[(u + 1) % W][e]);          // x[tx - (W-1) + m]
#pragma unroll
                        for (int m = 1; m < W; ++m) z = f2_fma(wv[m][e], xc[(u + 1 + m) % W][e], z);
                        gy[e] = silu_vjp_2<true>(gy[e], z);
                    }
                    if (!live) gy[e] = f2_all(0.f);
                    dzc[u][e] = gy[e];
                    if (own) {
#pragma unroll
                        for (int m = 0; m < W; ++m) dwv[m][e] = f2_fma(gy[e], xc[(u + 1 + m) % W][e], dwv[m][e]);
                    }
                }
                const int td = tx - (W - 1);
                if (!EDGE || (td >= t0 && td < t0 + run && td < T)) {
                    f2 a[2];
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        a[e] = f2_mul(wv[0][e], dzc[u][e]);                   // dz[tx - m]
#pragma unroll
                        for (int m = 1; m < W; ++m) a[e] = f2_fma(wv[m][e], dzc[(u - m + W) % W][e], a[e]);
                    }
                    st_c2<4, true>(dp, 0, a);
                    dp += ldx;
                }
            }
        };
        // rows tx of the steps jj .. jj + W - 1 and the outputs tx - (W-1) all inside [t0, min(T, t0 + run))
        const int inner0 = 2 * (W - 1), inner1 = min(T - t0, run) + W - 1;
        int slot = 0;
#pragma unroll 1
        for (int jj = 0; jj < nr; jj += W) {
            fetch();                                           // refills the slot that the previous group was read from
            asm volatile("cp.async.wait_group %0;" ::"n"(NG - 1) : "memory");
            if (jj >= inner0 && jj + W <= inner1) step(jj, slot, std::false_type());
            else step(jj, slot, std::true_type());
            slot = slot + 1 == NG ? 0 : slot + 1;
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();                               // every warp has drained its ring: the memory becomes the partials
#pragma unroll
    for (int m = 0; m < W; ++m)
#pragma unroll
        for (int e = 0; e < 2; ++e) *reinterpret_cast<f2*>(&red[g][m][4 * p + 2 * e]) = dwv[m][e];
    __syncthreads();
    if (threadIdx.x < 128) {
        const size_t pblk = (size_t)blockIdx.z * gridDim.y + blockIdx.y;
#pragma unroll
        for (int m = 0; m < W; ++m) {
            float a = 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) a += red[r][m][threadIdx.x];
            dw_part[(pblk * C + blockIdx.x * 128 + threadIdx.x) * W + m] = a;
        }
    }
}

// =============================================================================================
// gated RMSNorm:  y = x * inv * w * sigmoid(gate),  inv = rsqrt(mean(x^2) + eps).  One warp per row.
// =============================================================================================
// VEC4: dim % 128 == 0, lane owns 4 contiguous elements per 128-wide segment; else scalar stride-32.
template <bool BF16, bool VEC4>
__global__ void __launch_bounds__(256) rmsnorm_fwd_kernel(long long rows, int D, float eps, const void* __restrict__ x,
                                                          const void* __restrict__ gate, const float* __restrict__ w,
                                                          void* __restrict__ y, float* __restrict__ inv_rms) {
    const int lane = threadIdx.x & 31;
    const long long warp0 = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    const long long nwarp = (long long)gridDim.x * 8;
    for (long long row = warp0; row < rows; row += nwarp) {
        const size_t base = (size_t)row * D;
        float ss = 0.f;
        if (VEC4) {
            for (int d = 4 * lane; d < D; d += 128) {
                float a[4];
                ld4<BF16>(a, x, base + d);
                ss += a[0] * a[0] + a[1] * a[1] + a[2] * a[2] + a[3] * a[3];
            }
        } else {
            for (int d = lane; d < D; d += 32) {
                float a = ld_io(x, base + d, BF16);
                ss += a * a;
            }
        }
        ss = warp_sum(ss);
        const float inv = rsqrtf(ss / (float)D + eps);
        if (lane == 0) inv_rms[row] = inv;
        if (VEC4) {
            for (int d = 4 * lane; d < D; d += 128) {
                float a[4], gt[4], out[4];
                ld4<BF16>(a, x, base + d);
                ld4<BF16>(gt, gate, base + d);
                const float4 ww = *reinterpret_cast<const float4*>(w + d);
                const float wa[4] = {ww.x, ww.y, ww.z, ww.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) out[e] = a[e] * inv * wa[e] * sigmoid_t<BF16>(gt[e]);
                st4<BF16>(y, base + d, out);
            }
        } else {
            for (int d = lane; d < D; d += 32)
                st_io(y, base + d, BF16, ld_io(x, base + d, BF16) * inv * w[d] * sigmoid_t<BF16>(ld_io(gate, base + d, BF16)));
        }
    }
}

// Backward: u = n*w, y = u*s;  dgate = dy*u*s*(1-s);  du = dy*s;  dw += du*n;  dn = du*w;
//           dx = inv * (dn - n * mean(dn*n)).
// dweight: every warp accumulates its rows into its own shared-memory row, the block sums the
// eight rows in fixed order and writes one partial per block.
// What a launch writes: everything, or one half of it in a call that has no memory of its own for the partials.
enum RmsParts { kRmsAll, kRmsWeight, kRmsInputs };
template <bool BF16, bool VEC4, int PARTS>
__global__ void __launch_bounds__(256) rmsnorm_bwd_kernel(long long rows, int D, const void* __restrict__ x,
                                                          const void* __restrict__ gate, const float* __restrict__ w,
                                                          const float* __restrict__ inv_rms, const void* __restrict__ dy,
                                                          void* __restrict__ dx, void* __restrict__ dgate,
                                                          float* __restrict__ dw_part) {
    dependents_go();
    extern __shared__ float dws[];   // [8][D]
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    float* mine = dws + (size_t)wid * D;
    for (int d = lane; d < D; d += 32) mine[d] = 0.f;
    const long long warp0 = (long long)blockIdx.x * 8 + wid;
    const long long nwarp = (long long)gridDim.x * 8;
    for (long long row = warp0; row < rows; row += nwarp) {
        const size_t base = (size_t)row * D;
        const float inv = inv_rms[row];
        float dot = 0.f;
        if (VEC4) {
            for (int d = 4 * lane; d < D; d += 128) {
                float a[4], gt[4], gy[4];
                ld4<BF16>(a, x, base + d);
                ld4<BF16>(gt, gate, base + d);
                ld4<BF16>(gy, dy, base + d);
                const float4 ww = *reinterpret_cast<const float4*>(w + d);
                const float wa[4] = {ww.x, ww.y, ww.z, ww.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) dot += gy[e] * sigmoid_t<BF16>(gt[e]) * wa[e] * a[e] * inv;
            }
        } else {
            for (int d = lane; d < D; d += 32)
                dot += ld_io(dy, base + d, BF16) * sigmoid_t<BF16>(ld_io(gate, base + d, BF16)) * w[d] * ld_io(x, base + d, BF16) * inv;
        }
        dot = warp_sum(dot) / (float)D;
        if (VEC4) {
            for (int d = 4 * lane; d < D; d += 128) {
                float a[4], gt[4], gy[4], ox[4], og[4];
                ld4<BF16>(a, x, base + d);
                ld4<BF16>(gt, gate, base + d);
                ld4<BF16>(gy, dy, base + d);
                const float4 ww = *reinterpret_cast<const float4*>(w + d);
                const float wa[4] = {ww.x, ww.y, ww.z, ww.w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float n = a[e] * inv, s = sigmoid_t<BF16>(gt[e]);
                    const float du = gy[e] * s;
                    og[e] = gy[e] * n * wa[e] * s * (1.f - s);
                    ox[e] = inv * (du * wa[e] - n * dot);
                    mine[d + e] += du * n;
                }
                if (PARTS != kRmsWeight) {
                    st4<BF16>(dx, base + d, ox);
                    st4<BF16>(dgate, base + d, og);
                }
            }
        } else {
            for (int d = lane; d < D; d += 32) {
                const float n = ld_io(x, base + d, BF16) * inv, s = sigmoid_t<BF16>(ld_io(gate, base + d, BF16));
                const float gyv = ld_io(dy, base + d, BF16);
                const float du = gyv * s;
                if (PARTS != kRmsWeight) {
                    st_io(dgate, base + d, BF16, gyv * n * w[d] * s * (1.f - s));
                    st_io(dx, base + d, BF16, inv * (du * w[d] - n * dot));
                }
                mine[d] += du * n;
            }
        }
    }
    if (PARTS == kRmsInputs) return;
    __syncthreads();
    for (int d = threadIdx.x; d < D; d += 256) {
        float a = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) a += dws[(size_t)r * D + d];
        dw_part[(size_t)blockIdx.x * D + d] = a;
    }
}

// Rows of exactly 128 elements (the head width of the tensor-core lane): the row lives in registers, and a warp works on
// four rows at a time with all of their loads issued before the first reduction, so that a thread has 8-12 independent
// 8-byte (bf16) loads in flight instead of one row's worth.
constexpr int kRmsRows = 4;

template <bool BF16, bool ROWS>
__global__ void __launch_bounds__(256) rmsnorm_fwd128_kernel(long long rows, int heads, int gate_ld, float eps, const void* __restrict__ x,
                                                             const void* __restrict__ gate, const float* __restrict__ w,
                                                             void* __restrict__ y, float* __restrict__ inv_rms) {
    const int lane = threadIdx.x & 31;
    const long long warp0 = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    const long long nwarp = (long long)gridDim.x * 8;
    const float4 ww = *reinterpret_cast<const float4*>(w + 4 * lane);
    const float wa[4] = {ww.x, ww.y, ww.z, ww.w};
    auto gate_at = [&](long long row) {      // as in the backward below
        const unsigned r = (unsigned)row, tok = r / (unsigned)heads;
        return (size_t)tok * gate_ld + (r - tok * (unsigned)heads) * 128 + 4 * lane;
    };
    for (long long row0 = warp0 * kRmsRows; row0 < rows; row0 += nwarp * kRmsRows) {
        float a[kRmsRows][4], gt[kRmsRows][4], ss[kRmsRows];
#pragma unroll
        for (int r = 0; r < kRmsRows; ++r) {
            const size_t base = (size_t)min(row0 + r, rows - 1) * 128 + 4 * lane;
            ld4<BF16>(a[r], x, base);
            ld4<BF16>(gt[r], gate, ROWS ? gate_at(min(row0 + r, rows - 1)) : base);
        }
#pragma unroll
        for (int r = 0; r < kRmsRows; ++r) ss[r] = fmaf(a[r][3], a[r][3], fmaf(a[r][2], a[r][2], fmaf(a[r][1], a[r][1], a[r][0] * a[r][0])));
        // the halves of a row last: the operator's fused norm (tc_walk_kernel) has them in two blocks and gives the same bits
#pragma unroll
        for (int o = 8; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < kRmsRows; ++r) ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], o);
#pragma unroll
        for (int r = 0; r < kRmsRows; ++r) ss[r] += __shfl_xor_sync(0xffffffffu, ss[r], 16);
#pragma unroll
        for (int r = 0; r < kRmsRows; ++r) {
            if (row0 + r < rows) {
                const float inv = rsqrtf(ss[r] * (1.0f / 128.0f) + eps);
                if (lane == 0) inv_rms[row0 + r] = inv;
                float out[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) out[e] = a[r][e] * inv * wa[e] * sigmoid_t<BF16>(gt[r][e]);
                st4<BF16>(y, (size_t)(row0 + r) * 128 + 4 * lane, out);
            }
        }
    }
}

// ROWS: gate and dgate are the [token][head][128] part of wider rows gate_ld elements apart (a slice of the layer's
// projection), heads rows to a token.
template <bool BF16, bool ROWS, int PARTS = kRmsAll>
__global__ void __launch_bounds__(256) rmsnorm_bwd128_kernel(long long rows, int heads, int gate_ld, const void* __restrict__ x,
                                                             const void* __restrict__ gate, const float* __restrict__ w,
                                                             const float* __restrict__ inv_rms, const void* __restrict__ dy,
                                                             void* __restrict__ dx, void* __restrict__ dgate,
                                                             float* __restrict__ dw_part) {
    dependents_go();
    __shared__ float dws[8][128];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const long long warp0 = (long long)blockIdx.x * 8 + wid;
    const long long nwarp = (long long)gridDim.x * 8;
    const float4 ww = *reinterpret_cast<const float4*>(w + 4 * lane);
    const float wa[4] = {ww.x, ww.y, ww.z, ww.w};
    float dwa[4] = {0.f, 0.f, 0.f, 0.f};
    auto gate_at = [&](long long row) {
        const unsigned r = (unsigned)row, tok = r / (unsigned)heads;
        return (size_t)tok * gate_ld + (r - tok * (unsigned)heads) * 128 + 4 * lane;
    };
    for (long long row0 = warp0 * kRmsRows; row0 < rows; row0 += nwarp * kRmsRows) {
        float a[kRmsRows][4], gt[kRmsRows][4], gy[kRmsRows][4], inv[kRmsRows], dot[kRmsRows];
#pragma unroll
        for (int r = 0; r < kRmsRows; ++r) {
            const long long rr = min(row0 + r, rows - 1);
            const size_t base = (size_t)rr * 128 + 4 * lane;
            ld4<BF16>(a[r], x, base);
            ld4<BF16>(gt[r], gate, ROWS ? gate_at(rr) : base);
            ld4<BF16>(gy[r], dy, base);
            inv[r] = inv_rms[rr];
        }
#pragma unroll
        for (int r = 0; r < kRmsRows; ++r) {
            dot[r] = 0.f;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                gt[r][e] = sigmoid_t<BF16>(gt[r][e]);          // s
                a[r][e] *= inv[r];                             // n
                dot[r] += gy[r][e] * gt[r][e] * wa[e] * a[r][e];
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int r = 0; r < kRmsRows; ++r) dot[r] += __shfl_xor_sync(0xffffffffu, dot[r], o);
#pragma unroll
        for (int r = 0; r < kRmsRows; ++r) {
            if (row0 + r < rows) {
                const float mean = dot[r] * (1.0f / 128.0f);
                float ox[4], og[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float n = a[r][e], sg = gt[r][e];
                    const float du = gy[r][e] * sg;
                    og[e] = gy[r][e] * n * wa[e] * sg * (1.f - sg);
                    ox[e] = inv[r] * (du * wa[e] - n * mean);
                    dwa[e] += du * n;
                }
                const size_t base = (size_t)(row0 + r) * 128 + 4 * lane;
                if (PARTS != kRmsWeight) {
                    st4<BF16>(dx, base, ox);
                    st4<BF16>(dgate, ROWS ? gate_at(row0 + r) : base, og);
                }
            }
        }
    }
    if (PARTS == kRmsInputs) return;
#pragma unroll
    for (int e = 0; e < 4; ++e) dws[wid][4 * lane + e] = dwa[e];
    __syncthreads();
    if (threadIdx.x < 128) {
        float t = 0.f;
#pragma unroll
        for (int r = 0; r < 8; ++r) t += dws[r][threadIdx.x];
        dw_part[(size_t)blockIdx.x * 128 + threadIdx.x] = t;
    }
}

// out[i] = sum over b of part[b][i]: 32 columns per block, 32 row segments summed in a fixed order; bf16: rounded on the way out
__global__ void __launch_bounds__(1024) column_sum_kernel(int nblk, int N, const float* __restrict__ part_all,
                                                          ColumnSumItems outs, int bf16) {
    __shared__ float red[32][33];
    const float* __restrict__ part = part_all + (size_t)blockIdx.y * nblk * N;     // blockIdx.y = item
    void* __restrict__ out = pick_item(outs.out, (int)blockIdx.y);
    const int lane = threadIdx.x & 31, seg = threadIdx.x >> 5;
    const int i = blockIdx.x * 32 + lane;
    float a = 0.f;
    dependency_wait();                    // the kernel before wrote the partial sums
    if (i < N)
        for (int b = seg; b < nblk; b += 32) a += ld_after_f32(part + (size_t)b * N + i);
    red[seg][lane] = a;
    __syncthreads();
    if (seg == 0 && i < N) {
        float t = 0.f;
#pragma unroll
        for (int r = 0; r < 32; ++r) t += red[r][lane];
        st_io(out, i, bf16, t);
    }
}


// Casts to bf16 of several dense float32 (or bf16) arrays laid end to end: the projection weights of a layer gathered
// into one matrix, so that the products on one input become one GEMM.  A null source writes zeros (padding rows).
// Bound by the weights' bytes; one launch instead of one cast per weight (8 x 2.3 us at width 768).
constexpr int kPackItems = 10;
struct PackItems {
    const void* src[kPackItems];
    unsigned long long end8[kPackItems];      // running ends, in groups of 8 elements
};
template <bool F32>
__global__ void __launch_bounds__(256) pack_bf16_kernel(unsigned long long total8, int n, PackItems items, __nv_bfloat16* __restrict__ dst) {
    const unsigned long long step = (unsigned long long)gridDim.x * blockDim.x;
    for (unsigned long long i = (unsigned long long)blockIdx.x * blockDim.x + threadIdx.x; i < total8; i += step) {
        unsigned long long begin = 0;
        const void* src = items.src[0];
#pragma unroll
        for (int k = 1; k < kPackItems; ++k)
            if (k < n && i >= items.end8[k - 1]) {
                begin = items.end8[k - 1];
                src = items.src[k];
            }
        uint4 u = make_uint4(0, 0, 0, 0);
        if (src != nullptr) {
            if (F32) {
                const float4* p = reinterpret_cast<const float4*>(src) + 2 * (i - begin);
                const float4 a = __ldg(p), b = __ldg(p + 1);
                __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
                h[0] = __floats2bfloat162_rn(a.x, a.y); h[1] = __floats2bfloat162_rn(a.z, a.w);
                h[2] = __floats2bfloat162_rn(b.x, b.y); h[3] = __floats2bfloat162_rn(b.z, b.w);
            } else {
                u = __ldg(reinterpret_cast<const uint4*>(src) + (i - begin));
            }
        }
        *reinterpret_cast<uint4*>(dst + 8 * i) = u;
    }
}

}  // namespace pw
}  // namespace kda

// =============================================================================================
// C ABI
// =============================================================================================
using namespace kda;

extern "C" int kda_pack_bf16(int32_t n_items, int32_t src_dtype, const void* const* src, const int64_t* elems, void* dst, void* stream) {
    if (n_items < 1 || n_items > pw::kPackItems) return KDA_ERR_BAD_SHAPE;
    if (!src || !elems || !dst) return KDA_ERR_NULL;
    pw::PackItems it = {};
    unsigned long long end = 0;
    uintptr_t al = reinterpret_cast<uintptr_t>(dst);
    for (int i = 0; i < n_items; ++i) {
        if (elems[i] < 0 || elems[i] % 8 != 0) return KDA_ERR_UNSUPPORTED;
        end += (unsigned long long)elems[i] / 8;
        it.src[i] = src[i];
        it.end8[i] = end;
        al |= reinterpret_cast<uintptr_t>(src[i]);
    }
    if (al % 16 != 0) return KDA_ERR_UNSUPPORTED;
    if (end == 0) return KDA_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const int blocks = (int)std::min<unsigned long long>((end + 255) / 256, 148ULL * 8);
    if (src_dtype == KDA_DTYPE_F32) KDA_LAUNCH("pack_bf16_kernel", st, pw::pack_bf16_kernel<true><<<blocks, 256, 0, st>>>(end, n_items, it, static_cast<__nv_bfloat16*>(dst)));
    else KDA_LAUNCH("pack_bf16_kernel", st, pw::pack_bf16_kernel<false><<<blocks, 256, 0, st>>>(end, n_items, it, static_cast<__nv_bfloat16*>(dst)));
    return launch_status();
}

extern "C" int kda_gate_fwd_rows(int32_t tokens, int32_t heads, int32_t key_dim, int32_t io_dtype, const void* raw_gate,
                                 const void* beta_logits, int32_t bl_ld, const float* A_log, const float* dt_bias, float lower_bound,
                            float* g_out, float* beta_out, void* stream) {
    const bool beside = (io_dtype & KDA_BESIDE_OWN_LAUNCH) != 0;
    io_dtype &= ~KDA_BESIDE_OWN_LAUNCH;
    if (tokens < 0 || heads <= 0 || key_dim <= 0 || bl_ld < heads) return KDA_ERR_BAD_SHAPE;
    if (tokens == 0) return KDA_OK;
    if (!raw_gate || !beta_logits || !A_log || !dt_bias || !g_out || !beta_out) return KDA_ERR_NULL;
    const size_t n = (size_t)tokens * heads * key_dim;
    cudaStream_t fst = (cudaStream_t)stream;
    const bool al = ((reinterpret_cast<uintptr_t>(raw_gate) | reinterpret_cast<uintptr_t>(dt_bias) | reinterpret_cast<uintptr_t>(g_out)) % 16) == 0;
    // quads a thread: one up to four blocks a SM, two up to eight (77 rows of 2,048: 2.6, 2.9 and 3.5 us with 1, 2 and 4; 450:
    // 3.8, 3.5, 3.6; 8,191: 39, 28, 21)
    const int quads = n / 4 <= 148 * 4 * 256 ? 1 : (n / 4 <= 148 * 8 * 256 ? 2 : 4);
    const long long n_thr = (long long)heads * key_dim / 4 * ceil_div(tokens, quads);
    if (key_dim % 4 == 0 && al && (long long)heads * key_dim < (1ll << 31) && n_thr < (1ll << 31)) {      // 2^31 threads: 137 GB of g
        const unsigned thr = (unsigned)n_thr, blocks4 = (thr + 255) / 256;
        cudaError_t e = cudaSuccess;
        const auto kern = io_dtype == KDA_DTYPE_BF16 ? pw::gate_fwd4_kernel<true> : pw::gate_fwd4_kernel<false>;
        KDA_LAUNCH("gate_fwd_kernel", fst, e = launch_early(kern, dim3(blocks4), 256, 0, fst, beside, 1, thr, n / 4, tokens, heads, key_dim, raw_gate, beta_logits, bl_ld, A_log, dt_bias, lower_bound, g_out, beta_out));
        return e == cudaSuccess ? launch_status() : KDA_ERR_CUDA;
    }
    if (bl_ld != heads) return KDA_ERR_UNSUPPORTED;      // strided beta logits: the vector path only
    const int blocks = (int)std::min<size_t>((n + 255) / 256, 148 * 16);
    KDA_LAUNCH("gate_fwd_kernel", (cudaStream_t)stream, pw::gate_fwd_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(n, (size_t)tokens * heads, heads, key_dim,
                                                                   io_dtype == KDA_DTYPE_BF16, raw_gate, beta_logits,
                                                                   A_log, dt_bias, lower_bound, g_out, beta_out));
    return launch_status();
}

extern "C" int kda_gate_fwd(int32_t tokens, int32_t heads, int32_t key_dim, int32_t io_dtype, const void* raw_gate,
                            const void* beta_logits, const float* A_log, const float* dt_bias, float lower_bound,
                            float* g_out, float* beta_out, void* stream) {
    return kda_gate_fwd_rows(tokens, heads, key_dim, io_dtype, raw_gate, beta_logits, heads, A_log, dt_bias, lower_bound, g_out, beta_out, stream);
}

extern "C" size_t kda_gate_bwd_scratch_bytes(int32_t tokens, int32_t heads, int32_t key_dim) {
    const size_t nblk = (size_t)ceil_div(tokens > 0 ? tokens : 1, pw::kGateRows);
    return align_up(2 * nblk * heads * key_dim * sizeof(float), 256);
}

extern "C" int kda_gate_bwd_rows(int32_t tokens, int32_t heads, int32_t key_dim, int32_t io_dtype, const void* raw_gate,
                                 const void* beta_logits, int32_t bl_ld, int32_t bl_pad, const float* A_log, const float* dt_bias,
                                 float lower_bound, const float* dg, const float* dbeta, void* d_raw_gate, void* d_beta_logits,
                                 float* dA_log, float* ddt_bias, void* scratch, size_t scratch_bytes, void* stream) {
    if (tokens < 0 || heads <= 0 || key_dim <= 0 || bl_pad < 0 || bl_ld < heads + bl_pad) return KDA_ERR_BAD_SHAPE;
    if (!A_log || !dt_bias || !dA_log || !ddt_bias) return KDA_ERR_NULL;
    if (tokens > 0 && (!raw_gate || !beta_logits || !dg || !dbeta || !d_raw_gate || !d_beta_logits)) return KDA_ERR_NULL;
    if (!scratch || scratch_bytes < kda_gate_bwd_scratch_bytes(tokens, heads, key_dim)) return KDA_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const int nblk = tokens > 0 ? ceil_div(tokens, pw::kGateRows) : 0;
    float* part_b = static_cast<float*>(scratch);
    float* part_a = part_b + (size_t)(nblk > 0 ? nblk : 1) * heads * key_dim;
    const bool al = ((reinterpret_cast<uintptr_t>(raw_gate) | reinterpret_cast<uintptr_t>(dt_bias) | reinterpret_cast<uintptr_t>(dg) |
                      reinterpret_cast<uintptr_t>(d_raw_gate)) % 16) == 0;
    if (nblk > 0 && key_dim % 4 == 0 && al) {
        const dim3 grid(ceil_div(heads * key_dim, 128), nblk);
        if (io_dtype == KDA_DTYPE_BF16)
            KDA_LAUNCH("gate_bwd_kernel", st, pw::gate_bwd4_kernel<true><<<grid, 256, 0, st>>>(tokens, heads, key_dim, raw_gate, beta_logits, bl_ld, bl_pad, A_log, dt_bias, lower_bound, dg, dbeta, d_raw_gate, d_beta_logits, part_b, part_a));
        else
            KDA_LAUNCH("gate_bwd_kernel", st, pw::gate_bwd4_kernel<false><<<grid, 256, 0, st>>>(tokens, heads, key_dim, raw_gate, beta_logits, bl_ld, bl_pad, A_log, dt_bias, lower_bound, dg, dbeta, d_raw_gate, d_beta_logits, part_b, part_a));
    } else if (nblk > 0 && bl_ld != heads) {
        return KDA_ERR_UNSUPPORTED;      // strided beta logits: the vector path only
    } else if (nblk > 0)
        KDA_LAUNCH("gate_bwd_kernel", st, pw::gate_bwd_kernel<<<nblk, 256, 0, st>>>(tokens, heads, key_dim, io_dtype == KDA_DTYPE_BF16, raw_gate,
                                                  beta_logits, A_log, dt_bias, lower_bound, dg, dbeta, d_raw_gate,
                                                  d_beta_logits, part_b, part_a));
    cudaError_t e = cudaSuccess;
    KDA_LAUNCH("gate_bwd_reduce_kernel", st, e = launch_early(pw::gate_bwd_reduce_kernel, dim3(heads), 1024, 0, st, nblk > 0, 1, nblk, heads, key_dim, part_b, part_a, ddt_bias, dA_log));
    return e == cudaSuccess ? launch_status() : KDA_ERR_CUDA;
}

extern "C" int kda_gate_bwd(int32_t tokens, int32_t heads, int32_t key_dim, int32_t io_dtype, const void* raw_gate,
                            const void* beta_logits, const float* A_log, const float* dt_bias, float lower_bound,
                            const float* dg, const float* dbeta, void* d_raw_gate, void* d_beta_logits, float* dA_log,
                            float* ddt_bias, void* scratch, size_t scratch_bytes, void* stream) {
    return kda_gate_bwd_rows(tokens, heads, key_dim, io_dtype, raw_gate, beta_logits, heads, 0, A_log, dt_bias, lower_bound, dg, dbeta,
                             d_raw_gate, d_beta_logits, dA_log, ddt_bias, scratch, scratch_bytes, stream);
}

static int decode_launch(int n_seq, int heads, int key_dim, int value_dim, int bf16, int gbf16, int l2norm, float scale, const void* q,
                         const void* k, const void* v, const void* g, const void* beta, const float* state_in, float* state_out,
                         void* o, cudaStream_t st, pw::RawGate raw = pw::RawGate{nullptr, nullptr, 0.f, 0}) {
    // four rows in flight per warp: at ~70 registers three to four CTAs share an SM, so one CTA's prologue (norms, decay) hides
    // under the others' streaming; eight rows per warp measured 20 % slower
    // one CTA per (sequence, head) once there are enough of them to fill the GPU; otherwise split the value rows
    const int rows_per_cta = (n_seq * heads >= 148 * 4) ? value_dim : 32;
    dim3 grid(n_seq * heads, ceil_div(value_dim, rows_per_cta));
    const bool vec = (key_dim % 4 == 0) &&
                     ((reinterpret_cast<uintptr_t>(state_in) | reinterpret_cast<uintptr_t>(state_out)) % 16 == 0);
    const pw::TokenMix none = {};
#define KDA_DECODE(NV4) \
    KDA_LAUNCH("decode_kernel", st, pw::decode_kernel<NV4, 4, 8, false, 1><<<grid, 256, 0, st>>>(heads, key_dim, value_dim, bf16, gbf16, l2norm, scale, q, k, v, g, beta, state_in, state_out, o, rows_per_cta, raw, none))
    if (vec && key_dim <= 128) KDA_DECODE(1);
    else if (vec) KDA_DECODE(2);
    else KDA_DECODE(0);
#undef KDA_DECODE
    return launch_status();
}

extern "C" int kda_decode_step_raw_rows(int32_t n_seq, int32_t heads, int32_t key_dim, int32_t value_dim, int32_t io_dtype, float scale,
                                        const void* q, const void* k, const void* v, const void* raw_gate, const void* beta_logits, int64_t bl_ld,
                                        const float* A_log, const float* dt_bias, float lower_bound, const float* state_in,
                                        float* state_out, void* o, void* stream) {
    if (n_seq < 0 || heads <= 0 || key_dim <= 0 || value_dim <= 0 || key_dim > KDA_MAX_DIM || value_dim > KDA_MAX_DIM || bl_ld < heads)
        return KDA_ERR_BAD_SHAPE;
    if (n_seq == 0) return KDA_OK;
    if (!q || !k || !v || !raw_gate || !beta_logits || !A_log || !dt_bias || !state_in || !state_out || !o) return KDA_ERR_NULL;
    const int bf16 = io_dtype == KDA_DTYPE_BF16;
    return decode_launch(n_seq, heads, key_dim, value_dim, bf16, bf16, 1, scale, q, k, v, raw_gate, beta_logits, state_in, state_out, o,
                         (cudaStream_t)stream, pw::RawGate{A_log, dt_bias, lower_bound, bl_ld});
}

extern "C" int kda_decode_step_raw(int32_t n_seq, int32_t heads, int32_t key_dim, int32_t value_dim, int32_t io_dtype, float scale,
                                   const void* q, const void* k, const void* v, const void* raw_gate, const void* beta_logits,
                                   const float* A_log, const float* dt_bias, float lower_bound, const float* state_in,
                                   float* state_out, void* o, void* stream) {
    return kda_decode_step_raw_rows(n_seq, heads, key_dim, value_dim, io_dtype, scale, q, k, v, raw_gate, beta_logits, heads, A_log, dt_bias,
                                    lower_bound, state_in, state_out, o, stream);
}

extern "C" int kda_token_mix(int32_t n_seq, int32_t heads, float scale, const void* q, const void* k, const void* v, const void* fa,
                             const void* beta_logits, const void* gate, int64_t ld, const void* fb_weight, int32_t fb_dtype, const float* A_log,
                             const float* dt_bias, float lower_bound, const float* norm_weight, float eps, const float* state_in,
                             float* state_out, void* mixed, void* stream) {
    const bool early = (fb_dtype & KDA_BEHIND_OWN_LAUNCH) != 0;
    fb_dtype &= ~KDA_BEHIND_OWN_LAUNCH;
    if (n_seq < 0 || heads <= 0 || ld < heads) return KDA_ERR_BAD_SHAPE;
    if (n_seq == 0) return KDA_OK;
    if (!q || !k || !v || !fa || !beta_logits || !gate || !fb_weight || !A_log || !dt_bias || !norm_weight || !state_in || !state_out || !mixed)
        return KDA_ERR_NULL;
    if (ld % 4 != 0 || (reinterpret_cast<uintptr_t>(state_in) | reinterpret_cast<uintptr_t>(state_out) | reinterpret_cast<uintptr_t>(fb_weight) |
                        reinterpret_cast<uintptr_t>(norm_weight)) % 16 != 0 ||
        (reinterpret_cast<uintptr_t>(fa) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(mixed)) % 8 != 0)
        return KDA_ERR_UNSUPPORTED;
    const pw::TokenMix mix{static_cast<const __nv_bfloat16*>(fa), fb_weight, static_cast<const __nv_bfloat16*>(gate), norm_weight, ld, eps,
                           fb_dtype == KDA_DTYPE_F32 ? 1 : 0, n_seq};
    const pw::RawGate raw{A_log, dt_bias, lower_bound, ld};
    cudaStream_t st = (cudaStream_t)stream;
    const int blocks = n_seq * heads;
    cudaError_t e = cudaSuccess;
    // Blocks of 32, 16 and 8 warps go one, two and four to an SM (148 of them).  Clusters share the gate's rows but are placed whole, and
    // unevenly from nine tenths of all places on: blocks are on their own there, and where they come in waves (a token's three launches in us,
    // clusters / alone, 8 warps, 2,048 wide: 480 states 44.0 / 44.6, 528 56.8 / 55.8, 544 60.4 / 55.8, 592 66.1 / 57.4, 608 65.5 / 61.0, 768 69.1 /
    // 67.1, 1,024 75.3 / 74.3; clusters of 16 warps / 8 warps alone: 256 33.3 / 36.9, 264 (768 wide) 26.6 / 29.2, 288 41.0 / 38.4).  And blocks that
    // start beside the projections' take the SMs these leave free, four to one and none to the next: up to three to an SM in the end they
    // start behind them (early in clusters / behind, alone: 288 39.5 / 38.4, 1,536 wide 31.2 / 29.2, 408 41.5 / 39.9, 432 41.0 / 39.9; 448, 2,048
    // wide, 43.5 / 45.6, 480 44.0 / 46.1).
    constexpr int kSms = 148;
    const int nw = blocks <= kSms ? 32 : (10 * blocks <= 9 * 2 * kSms ? 16 : 8);
    const bool behind = nw == 8 && blocks <= 3 * kSms;
    const int cluster = nw == 16 || (nw == 8 && !behind && 10 * blocks <= 9 * 4 * kSms) ? 4 : 1;
    const auto kern = nw == 32 ? pw::decode_kernel<1, 4, 32, true, 1>
                               : (nw == 16 ? pw::decode_kernel<1, 4, 16, true, 4> : (cluster == 4 ? pw::decode_kernel<1, 4, 8, true, 4> : pw::decode_kernel<1, 4, 8, true, 1>));
    KDA_LAUNCH("decode_kernel", st, e = launch_early(kern, dim3(ceil_div(blocks, cluster) * cluster), 32u * nw, 0, st, early && !behind, cluster, heads, 128, 128, 1, 1, 1, scale, q, k, v, nullptr, beta_logits,
                                                     state_in, state_out, mixed, 128, raw, mix));
    if (e != cudaSuccess) return KDA_ERR_CUDA;
    return launch_status();
}

extern "C" int kda_decode_step(int32_t n_seq, int32_t heads, int32_t key_dim, int32_t value_dim, int32_t io_dtype,
                               int32_t gate_dtype, int32_t l2norm, float scale, const void* q, const void* k, const void* v, const void* g,
                               const void* beta, const float* state_in, float* state_out, void* o, void* stream) {
    if (n_seq < 0 || heads <= 0 || key_dim <= 0 || value_dim <= 0 || key_dim > KDA_MAX_DIM || value_dim > KDA_MAX_DIM)
        return KDA_ERR_BAD_SHAPE;
    if (n_seq == 0) return KDA_OK;
    if (!q || !k || !v || !g || !beta || !state_in || !state_out || !o) return KDA_ERR_NULL;
    return decode_launch(n_seq, heads, key_dim, value_dim, io_dtype == KDA_DTYPE_BF16, gate_dtype == KDA_DTYPE_BF16, l2norm, scale, q, k,
                         v, g, beta, state_in, state_out, o, (cudaStream_t)stream);
}

extern "C" int kda_decode_steps(int32_t n_steps, int32_t n_seq, int32_t heads, int32_t key_dim, int32_t value_dim, int32_t io_dtype,
                                int32_t gate_dtype, int32_t l2norm, float scale, const void* q, const void* k, const void* v,
                                const void* g, const void* beta, float* state, void* o, void* stream) {
    if (n_steps < 0 || n_seq < 0 || heads <= 0 || key_dim <= 0 || value_dim <= 0 || key_dim > KDA_MAX_DIM || value_dim > KDA_MAX_DIM)
        return KDA_ERR_BAD_SHAPE;
    if (n_seq == 0 || n_steps == 0) return KDA_OK;
    if (!q || !k || !v || !g || !beta || !state || !o) return KDA_ERR_NULL;
    const int bf16 = io_dtype == KDA_DTYPE_BF16, gbf16 = gate_dtype == KDA_DTYPE_BF16;
    const size_t io_b = bf16 ? 2 : 4, g_b = gbf16 ? 2 : 4;
    const size_t nk = (size_t)n_seq * heads * key_dim, nv = (size_t)n_seq * heads * value_dim, nb = (size_t)n_seq * heads;
    auto at = [](const void* p, size_t bytes) { return static_cast<const void*>(static_cast<const char*>(p) + bytes); };
    for (int i = 0; i < n_steps; ++i) {
        // the state is updated in place: a warp reads a whole row before it writes it, and no row is shared between warps
        int rc = decode_launch(n_seq, heads, key_dim, value_dim, bf16, gbf16, l2norm, scale, at(q, i * nk * io_b), at(k, i * nk * io_b),
                               at(v, i * nv * io_b), at(g, i * nk * g_b), at(beta, i * nb * g_b), state, state,
                               static_cast<char*>(o) + i * nv * io_b, (cudaStream_t)stream);
        if (rc) return rc;
    }
    return KDA_OK;
}

namespace {

// Sums of the partial rows the launch before this one left: early, so that a few small blocks stand ready when its last ones end
// (with the gap a launch of their own cost: norm 4.1 + 2.1 us behind a 8.2 us kernel, convolutions 2.3 + 2.4).
[[nodiscard]] int column_sums(const char* name, int n, int nblk, int N, const float* part, const pw::ColumnSumItems& outs, int bf16, cudaStream_t st) {
    cudaError_t e = cudaSuccess;
    KDA_LAUNCH(name, st, e = launch_early(pw::column_sum_kernel, dim3(ceil_div(N, 32), n), 1024, 0, st, nblk > 0, 1, nblk, N, part, outs, bf16));
    return e == cudaSuccess ? launch_status() : KDA_ERR_CUDA;
}

inline bool conv_grid_ok(int n, int B, int T) { return ceil_div(T, 8 * pw::kConvPairT) <= 65535 && (long long)B * n <= 65535; }

// n same-shaped convolutions in one launch; x rows ldx elements apart
constexpr int kConvRun = 32;      // tokens per thread of the streaming forward
template <int W>
int conv_fwd_fast(int n, int B, int T, int C, int ldx, int bf16, int wf32, int silu, const pw::ConvFwdItems& it, cudaStream_t st, bool beside = false) {
    cudaError_t e = cudaSuccess;
    const bool vec4 = C % 128 == 0 && ldx % 4 == 0;         // channels per thread: 4 when a warp's 128 channels fill a row segment
    const dim3 grid(ceil_div(C, vec4 ? 128 : 64), ceil_div(T, 8 * pw::kConvPairT), B * n);
    bool win = false, carried = false;
    for (int i = 0; i < n; ++i) {
        win = win || it.cache[i] != nullptr || it.fin[i] != nullptr;
        carried = carried || it.cache[i] != nullptr;
    }
    // The streaming kernel unless a window is carried in, where its blocks of eight 32-token runs are many enough.  Filled to four fifths:
    // one and a half a SM, two where a window is carried out (224 blocks: 1.09 and 0.91 times the speed of the other kernel, 288: 1.24
    // and 1.00, 4,000: 1.26 and 1.2).  Where the last block of a sequence leaves more warps idle: filled to a half, and six a SM
    // (5 of 8 runs: 0.8 to 1.1 at 450 to 600 blocks, 1.0 to 1.2 at 864; 1 or 2 of 8: 0.5 to 0.8 at any number; 3 of 8: 0.9 to 1.05).
    // Up to 8 tokens a thread has one step to go, and the copy of the windows is what counts (1.0 to 1.3 up to twelve blocks a SM,
    // 0.9 at 27, 0.7 at 83).
    if (vec4 && bf16 && !carried) {
        const int runs = ceil_div(T, 8 * kConvRun);
        const dim3 sgrid(C / 128, runs + (win ? 1 : 0), B * n);
        const long long blocks = (long long)sgrid.x * runs * sgrid.z;
        const long long room = 8LL * kConvRun * runs;      // tokens a sequence's blocks could take
        const bool filled = 5LL * T >= 4 * room ? blocks >= (win ? 2 * 148 : 148 * 3 / 2) : 2LL * T >= room && blocks >= 148 * 6;
        const bool copied = win && T <= 8 && blocks >= 148 * 3 / 2 && blocks <= 148 * 12;
        if ((filled || copied) && sgrid.y <= 65535) {
            KDA_LAUNCH("conv_fwd_stream_kernel", st, e = launch_early(pw::conv_fwd_stream_kernel<W>, sgrid, 256, 0, st, beside, 1, B, T, C, ldx, kConvRun, win ? runs : -1, silu, wf32, it));
            return e == cudaSuccess ? launch_status() : KDA_ERR_CUDA;
        }
    }
#define KDA_CONV_FWD(VEC, BF, WIN) \
    KDA_LAUNCH("conv_fwd_kernel", st, e = launch_early(pw::conv_fwd_pair_kernel<W, VEC, BF, WIN>, grid, 256, 0, st, beside, 1, B, T, C, ldx, silu, wf32, it))
    if (vec4 && bf16) { if (win) KDA_CONV_FWD(4, true, true); else KDA_CONV_FWD(4, true, false); }
    else if (vec4) { if (win) KDA_CONV_FWD(4, false, true); else KDA_CONV_FWD(4, false, false); }
    else if (bf16) { if (win) KDA_CONV_FWD(2, true, true); else KDA_CONV_FWD(2, true, false); }
    else { if (win) KDA_CONV_FWD(2, false, true); else KDA_CONV_FWD(2, false, false); }
#undef KDA_CONV_FWD
    return e == cudaSuccess ? launch_status() : KDA_ERR_CUDA;
}

template <int W>
int conv_bwd_fast(int n, int B, int T, int C, int ldx, int bf16, int wf32, int silu, const pw::ConvBwdItems& it, float* const* dwgt,
                  float* part, cudaStream_t st, int dwb = 0) {
    dim3 grid(ceil_div(C, pw::kConvTileC), ceil_div(T, pw::kConvTileT), B * n);
    // tokens per thread run of the streaming kernel: long runs amortise the W-1 halo rows.  From one block of 32-token runs per
    // SM on it is the faster one (3 x 8,192 x 384: 22.1 -> 17.6 us); below, the tile kernel's more and smaller blocks are
    const long long warps64 = (long long)(C / 128) * ceil_div(T, 64) * B * n;
    if (bf16 && C % 128 == 0 && ldx % 4 == 0 && warps64 >= 148LL * 4) {
        const int run = warps64 >= 148LL * 48 ? 64 : 32;
        grid = dim3(C / 128, ceil_div(T, 8 * run), B * n);                  // never more partial rows than the tile kernel's
        const size_t ring_bytes = (size_t)pw::kConvRingDepth * 2 * 256 * 8;
        if (set_smem_limit(pw::conv_bwd_ring_kernel<W>, ring_bytes)) return KDA_ERR_CUDA;
        KDA_LAUNCH("conv_bwd_kernel", st, pw::conv_bwd_ring_kernel<W><<<grid, 256, ring_bytes, st>>>(B, T, C, ldx, run, silu, wf32, it, part));
    } else if (bf16) KDA_LAUNCH("conv_bwd_kernel", st, pw::conv_bwd_tile_kernel<W, true><<<grid, 256, 0, st>>>(B, T, C, ldx, silu, wf32, it, part));
    else KDA_LAUNCH("conv_bwd_kernel", st, pw::conv_bwd_tile_kernel<W, false><<<grid, 256, 0, st>>>(B, T, C, ldx, silu, wf32, it, part));
    const int nblk = grid.y * B;                  // partial rows per item
    pw::ColumnSumItems outs = {};
    for (int i = 0; i < n; ++i) outs.out[i] = dwgt[i];
    return column_sums("conv_dw_reduce_kernel", n, nblk, C * W, part, outs, dwb, st);
}

template <int W>
int conv_fwd_w(int B, int T, int C, int bf16, int wf32, int silu, const void* x, const void* w, const void* cache, void* y,
               void* fin, cudaStream_t st) {
    const bool al16 = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(w) | reinterpret_cast<uintptr_t>(y)) % 16) == 0;
    if (C % 2 == 0 && al16 && conv_grid_ok(1, B, T)) {
        pw::ConvFwdItems it = {};
        it.x[0] = x; it.w[0] = w; it.y[0] = y; it.cache[0] = cache; it.fin[0] = fin;
        return conv_fwd_fast<W>(1, B, T, C, C, bf16, wf32, silu, it, st);
    }
    // odd channel counts, unaligned tensors, batches past a grid's y / z extent: one channel per thread
    const unsigned blocks = (unsigned)(((size_t)B * ceil_div(T, pw::kConvTT) * C + 255) / 256);
    if (bf16) KDA_LAUNCH("conv_fwd_kernel", st, pw::conv_fwd_kernel<W, 1, true><<<blocks, 256, 0, st>>>(B, T, C, silu, wf32, x, w, cache, y, fin));
    else KDA_LAUNCH("conv_fwd_kernel", st, pw::conv_fwd_kernel<W, 1, false><<<blocks, 256, 0, st>>>(B, T, C, silu, wf32, x, w, cache, y, fin));
    return launch_status();
}

inline void conv_bwd_grid(int B, int T, int C, int vec, dim3& grid) {
    grid = dim3(ceil_div(C / vec, 16), ceil_div(ceil_div(T, pw::kConvBT), 16), B);
}

template <int W>
int conv_bwd_w(int B, int T, int C, int bf16, int wf32, int silu, const void* x, const void* w, const void* cache, const void* dy,
               const void* dfin, void* dx, void* dcache, float* dwgt, int dwb, float* part, cudaStream_t st) {
    const bool al16 = ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy) | reinterpret_cast<uintptr_t>(dx)) % 16) == 0;
    dim3 grid, block(16, 16);
    if constexpr (W <= 4) {
        // no carried-in window and no final-state cotangent: the tiled kernel (same partial layout: one row of
        // partials per 64-token tile and batch entry)
        if (!cache && !dfin && !dcache && C % 2 == 0 && al16 && reinterpret_cast<uintptr_t>(w) % 16 == 0) {
            pw::ConvBwdItems it = {};
            it.x[0] = x; it.w[0] = w; it.dy[0] = dy; it.dx[0] = dx;
            return conv_bwd_fast<W>(1, B, T, C, C, bf16, wf32, silu, it, &dwgt, part, st, dwb);
        }
    }
    // the vector path keeps W*VEC partials per thread in shared memory; wide windows use the scalar path
    constexpr bool kVecOk = W <= 4;
    if (bf16) {
        if constexpr (kVecOk) {
            if (C % 8 == 0 && al16) {
                conv_bwd_grid(B, T, C, 8, grid);
                KDA_LAUNCH("conv_bwd_kernel", st, pw::conv_bwd_kernel<W, 8, true><<<grid, block, 0, st>>>(B, T, C, silu, wf32, x, w, cache, dy, dfin, dx, dcache, part));
            }
        }
        if (!(kVecOk && C % 8 == 0 && al16)) {
            conv_bwd_grid(B, T, C, 1, grid);
            KDA_LAUNCH("conv_bwd_kernel", st, pw::conv_bwd_kernel<W, 1, true><<<grid, block, 0, st>>>(B, T, C, silu, wf32, x, w, cache, dy, dfin, dx, dcache, part));
        }
    } else {
        if constexpr (kVecOk) {
            if (C % 4 == 0 && al16) {
                conv_bwd_grid(B, T, C, 4, grid);
                KDA_LAUNCH("conv_bwd_kernel", st, pw::conv_bwd_kernel<W, 4, false><<<grid, block, 0, st>>>(B, T, C, silu, wf32, x, w, cache, dy, dfin, dx, dcache, part));
            }
        }
        if (!(kVecOk && C % 4 == 0 && al16)) {
            conv_bwd_grid(B, T, C, 1, grid);
            KDA_LAUNCH("conv_bwd_kernel", st, pw::conv_bwd_kernel<W, 1, false><<<grid, block, 0, st>>>(B, T, C, silu, wf32, x, w, cache, dy, dfin, dx, dcache, part));
        }
    }
    const int nblk = grid.y * grid.z;
    pw::ColumnSumItems outs = {};
    outs.out[0] = dwgt;
    return column_sums("conv_dw_reduce_kernel", 1, nblk, C * W, part, outs, dwb, st);
}

}  // namespace

#define KDA_CONV_SWITCH(CALL)            \
    switch (width) {                     \
        case 1: return CALL(1);          \
        case 2: return CALL(2);          \
        case 3: return CALL(3);          \
        case 4: return CALL(4);          \
        case 5: return CALL(5);          \
        case 6: return CALL(6);          \
        case 7: return CALL(7);          \
        case 8: return CALL(8);          \
        default: return KDA_ERR_UNSUPPORTED; \
    }

extern "C" int kda_conv_fwd(int32_t batch, int32_t seq_len, int32_t channels, int32_t width, int32_t io_dtype,
                            int32_t silu, const void* x, const void* weight, const void* initial_state, void* y,
                            void* final_state, void* stream) {
    if (batch <= 0 || seq_len <= 0 || channels <= 0 || width <= 0) return KDA_ERR_BAD_SHAPE;
    if (!x || !weight || !y) return KDA_ERR_NULL;
    const int wf32 = (io_dtype & KDA_WEIGHT_F32) != 0;
    const int bf16 = (io_dtype & 0xff) == KDA_DTYPE_BF16;
    cudaStream_t st = (cudaStream_t)stream;
#define CALL(WW) conv_fwd_w<WW>(batch, seq_len, channels, bf16, wf32, silu, x, weight, initial_state, y, final_state, st)
    KDA_CONV_SWITCH(CALL)
#undef CALL
}

extern "C" size_t kda_conv_bwd_scratch_bytes(int32_t batch, int32_t seq_len, int32_t channels, int32_t width) {
    const size_t nblk = (size_t)ceil_div(ceil_div(seq_len > 0 ? seq_len : 1, pw::kConvBT), 16) * (batch > 0 ? batch : 1);
    return align_up(nblk * channels * width * sizeof(float), 256);
}

extern "C" int kda_conv_bwd(int32_t batch, int32_t seq_len, int32_t channels, int32_t width, int32_t io_dtype,
                            int32_t silu, const void* x, const void* weight, const void* initial_state, const void* d_y,
                            const void* d_final_state, void* dx, void* dweight, void* d_initial_state, void* scratch,
                            size_t scratch_bytes, void* stream) {
    if (batch <= 0 || seq_len <= 0 || channels <= 0 || width <= 0) return KDA_ERR_BAD_SHAPE;
    if (!x || !weight || !d_y || !dx || !dweight) return KDA_ERR_NULL;
    if (!scratch || scratch_bytes < kda_conv_bwd_scratch_bytes(batch, seq_len, channels, width)) return KDA_ERR_WORKSPACE;
    const int wf32 = (io_dtype & KDA_WEIGHT_F32) != 0;
    const int bf16 = (io_dtype & 0xff) == KDA_DTYPE_BF16;
    cudaStream_t st = (cudaStream_t)stream;
#define CALL(WW)                                                                                                  \
    conv_bwd_w<WW>(batch, seq_len, channels, bf16, wf32, silu, x, weight, initial_state, d_y, d_final_state, dx,  \
                   d_initial_state, static_cast<float*>(dweight), (io_dtype & KDA_DWEIGHT_BF16) != 0, static_cast<float*>(scratch), st)
    KDA_CONV_SWITCH(CALL)
#undef CALL
}

// n same-shaped convolutions (the q, k and v branches of a layer) in one launch each way: width <= 4, even channel count
// and row stride, 16-byte aligned tensors; anything else returns KDA_ERR_UNSUPPORTED and the caller issues the per-tensor
// calls.
namespace {
bool conv_multi_ok(int n, int channels, int width, const void* const* w, const void* const* a, const void* const* b, const void* const* c) {
    if (n < 1 || n > pw::kConvItems || width > 4 || channels % 2 != 0) return false;
    for (int i = 0; i < n; ++i) {
        if (!a[i] || !b[i] || (c && !c[i])) return false;
        if ((reinterpret_cast<uintptr_t>(w[i]) | reinterpret_cast<uintptr_t>(a[i]) | reinterpret_cast<uintptr_t>(b[i]) |
             (c ? reinterpret_cast<uintptr_t>(c[i]) : 0)) % 16) return false;
    }
    return true;
}
}  // namespace

extern "C" int kda_conv_fwd_rows(int32_t n_items, int32_t batch, int32_t seq_len, int32_t channels, int32_t width, int32_t io_dtype,
                                 int32_t silu, const void* const* x, int32_t x_ld, const void* const* weight, const void* const* cache,
                                 void* const* y, void* const* final_state, void* stream) {
    if (batch <= 0 || seq_len <= 0 || channels <= 0 || width <= 0 || x_ld < channels) return KDA_ERR_BAD_SHAPE;
    if (!x || !weight || !y) return KDA_ERR_NULL;
    if (x_ld % 2 != 0 || !conv_grid_ok(n_items, batch, seq_len) ||
        !conv_multi_ok(n_items, channels, width, weight, x, const_cast<const void* const*>(y), nullptr))
        return KDA_ERR_UNSUPPORTED;
    const int wf32 = (io_dtype & KDA_WEIGHT_F32) != 0;
    const int bf16 = (io_dtype & 0xff) == KDA_DTYPE_BF16;
    const bool beside = (io_dtype & KDA_BESIDE_OWN_LAUNCH) != 0;
    pw::ConvFwdItems it = {};
    for (int i = 0; i < n_items; ++i) {
        if (!weight[i]) return KDA_ERR_NULL;
        it.x[i] = x[i]; it.w[i] = weight[i]; it.y[i] = y[i];
        it.cache[i] = cache ? cache[i] : nullptr;
        it.fin[i] = final_state ? final_state[i] : nullptr;
    }
    cudaStream_t st = (cudaStream_t)stream;
    switch (width) {
        case 1: return conv_fwd_fast<1>(n_items, batch, seq_len, channels, x_ld, bf16, wf32, silu, it, st, beside);
        case 2: return conv_fwd_fast<2>(n_items, batch, seq_len, channels, x_ld, bf16, wf32, silu, it, st, beside);
        case 3: return conv_fwd_fast<3>(n_items, batch, seq_len, channels, x_ld, bf16, wf32, silu, it, st, beside);
        default: return conv_fwd_fast<4>(n_items, batch, seq_len, channels, x_ld, bf16, wf32, silu, it, st, beside);
    }
}

extern "C" int kda_conv_fwd_multi(int32_t n_items, int32_t batch, int32_t seq_len, int32_t channels, int32_t width,
                                  int32_t io_dtype, int32_t silu, const void* const* x, const void* const* weight,
                                  void* const* y, void* stream) {
    return kda_conv_fwd_rows(n_items, batch, seq_len, channels, width, io_dtype, silu, x, channels, weight, nullptr, y, nullptr, stream);
}

extern "C" int kda_conv_step_multi(int32_t n_items, int32_t batch, int32_t channels, int32_t width, int32_t io_dtype, int32_t silu,
                                   const void* const* x, const void* const* weight, void* const* cache, void* const* y, void* stream) {
    if (n_items < 1 || n_items > 4 || batch <= 0 || channels <= 0) return KDA_ERR_BAD_SHAPE;
    if (width < 1 || width > 4) return KDA_ERR_UNSUPPORTED;
    if (!x || !weight || !cache || !y) return KDA_ERR_NULL;
    const int wf32 = (io_dtype & KDA_WEIGHT_F32) != 0;
    const int bf16 = (io_dtype & 0xff) == KDA_DTYPE_BF16;
    pw::ConvStepItems it = {};
    for (int i = 0; i < n_items; ++i) {
        if (!x[i] || !weight[i] || !cache[i] || !y[i]) return KDA_ERR_NULL;
        it.x[i] = x[i]; it.w[i] = weight[i]; it.cache[i] = cache[i]; it.y[i] = y[i];
    }
    cudaStream_t st = (cudaStream_t)stream;
    const dim3 grid(ceil_div(batch * channels, 256), n_items);
#define KDA_CONV_STEP(WW)                                                                                                          \
    do {                                                                                                                           \
        if (bf16) KDA_LAUNCH("conv_step_kernel", st, pw::conv_step_kernel<WW, true><<<grid, 256, 0, st>>>(batch, channels, silu, wf32, it)); \
        else KDA_LAUNCH("conv_step_kernel", st, pw::conv_step_kernel<WW, false><<<grid, 256, 0, st>>>(batch, channels, silu, wf32, it));     \
    } while (0)
    switch (width) {
        case 1: KDA_CONV_STEP(1); break;
        case 2: KDA_CONV_STEP(2); break;
        case 3: KDA_CONV_STEP(3); break;
        default: KDA_CONV_STEP(4); break;
    }
#undef KDA_CONV_STEP
    return launch_status();
}

extern "C" size_t kda_conv_bwd_multi_scratch_bytes(int32_t n_items, int32_t batch, int32_t seq_len, int32_t channels, int32_t width) {
    return (size_t)(n_items > 0 ? n_items : 1) * kda_conv_bwd_scratch_bytes(batch, seq_len, channels, width);
}

extern "C" int kda_conv_bwd_rows(int32_t n_items, int32_t batch, int32_t seq_len, int32_t channels, int32_t width,
                                 int32_t io_dtype, int32_t silu, const void* const* x, int32_t x_ld, const void* const* weight,
                                 const void* const* d_y, void* const* dx, float* const* dweight, void* scratch,
                                 size_t scratch_bytes, void* stream) {
    if (batch <= 0 || seq_len <= 0 || channels <= 0 || width <= 0 || x_ld < channels) return KDA_ERR_BAD_SHAPE;
    if (!x || !weight || !d_y || !dx || !dweight) return KDA_ERR_NULL;
    if (x_ld % 2 != 0 || !conv_grid_ok(n_items, batch, seq_len) || !conv_multi_ok(n_items, channels, width, weight, x, d_y, const_cast<const void* const*>(dx))) return KDA_ERR_UNSUPPORTED;
    if (!scratch || scratch_bytes < kda_conv_bwd_multi_scratch_bytes(n_items, batch, seq_len, channels, width)) return KDA_ERR_WORKSPACE;
    const int wf32 = (io_dtype & KDA_WEIGHT_F32) != 0;
    const int bf16 = (io_dtype & 0xff) == KDA_DTYPE_BF16;
    pw::ConvBwdItems it = {};
    for (int i = 0; i < n_items; ++i) {
        if (!weight[i] || !dweight[i]) return KDA_ERR_NULL;
        it.x[i] = x[i]; it.w[i] = weight[i]; it.dy[i] = d_y[i]; it.dx[i] = dx[i];
    }
    cudaStream_t st = (cudaStream_t)stream;
    float* part = static_cast<float*>(scratch);
    switch (width) {
        case 1: return conv_bwd_fast<1>(n_items, batch, seq_len, channels, x_ld, bf16, wf32, silu, it, dweight, part, st);
        case 2: return conv_bwd_fast<2>(n_items, batch, seq_len, channels, x_ld, bf16, wf32, silu, it, dweight, part, st);
        case 3: return conv_bwd_fast<3>(n_items, batch, seq_len, channels, x_ld, bf16, wf32, silu, it, dweight, part, st);
        default: return conv_bwd_fast<4>(n_items, batch, seq_len, channels, x_ld, bf16, wf32, silu, it, dweight, part, st);
    }
}

extern "C" int kda_conv_bwd_multi(int32_t n_items, int32_t batch, int32_t seq_len, int32_t channels, int32_t width,
                                  int32_t io_dtype, int32_t silu, const void* const* x, const void* const* weight,
                                  const void* const* d_y, void* const* dx, float* const* dweight, void* scratch,
                                  size_t scratch_bytes, void* stream) {
    return kda_conv_bwd_rows(n_items, batch, seq_len, channels, width, io_dtype, silu, x, channels, weight, d_y, dx, dweight, scratch,
                             scratch_bytes, stream);
}

namespace {
inline int rms_blocks(long long rows) { return (int)std::min<long long>((rows + 7) / 8, 148LL * 4); }
}  // namespace

extern "C" int kda_rmsnorm_gate_fwd(int64_t rows, int32_t dim, int32_t io_dtype, float eps, const void* x,
                                    const void* gate, const float* weight, void* y, float* inv_rms, void* stream) {
    if (rows < 0 || dim <= 0 || dim > 1024) return KDA_ERR_BAD_SHAPE;
    if (rows == 0) return KDA_OK;
    if (!x || !gate || !weight || !y || !inv_rms) return KDA_ERR_NULL;
    cudaStream_t st = (cudaStream_t)stream;
    const int nb = rms_blocks(rows);
    const bool vec = dim % 128 == 0 &&
                     ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(y) |
                       reinterpret_cast<uintptr_t>(weight)) % 16) == 0;
    if (vec && dim == 128) {
        const int nb4 = (int)std::min<long long>((rows + 8 * pw::kRmsRows - 1) / (8 * pw::kRmsRows), 148LL * 8);
        if (io_dtype == KDA_DTYPE_BF16) KDA_LAUNCH("rmsnorm_fwd_kernel", st, pw::rmsnorm_fwd128_kernel<true, false><<<nb4, 256, 0, st>>>(rows, 1, 128, eps, x, gate, weight, y, inv_rms));
        else KDA_LAUNCH("rmsnorm_fwd_kernel", st, pw::rmsnorm_fwd128_kernel<false, false><<<nb4, 256, 0, st>>>(rows, 1, 128, eps, x, gate, weight, y, inv_rms));
        return launch_status();
    }
    if (io_dtype == KDA_DTYPE_BF16) {
        if (vec) KDA_LAUNCH("rmsnorm_fwd_kernel", st, pw::rmsnorm_fwd_kernel<true, true><<<nb, 256, 0, st>>>(rows, dim, eps, x, gate, weight, y, inv_rms));
        else KDA_LAUNCH("rmsnorm_fwd_kernel", st, pw::rmsnorm_fwd_kernel<true, false><<<nb, 256, 0, st>>>(rows, dim, eps, x, gate, weight, y, inv_rms));
    } else {
        if (vec) KDA_LAUNCH("rmsnorm_fwd_kernel", st, pw::rmsnorm_fwd_kernel<false, true><<<nb, 256, 0, st>>>(rows, dim, eps, x, gate, weight, y, inv_rms));
        else KDA_LAUNCH("rmsnorm_fwd_kernel", st, pw::rmsnorm_fwd_kernel<false, false><<<nb, 256, 0, st>>>(rows, dim, eps, x, gate, weight, y, inv_rms));
    }
    return launch_status();
}

extern "C" int kda_rmsnorm_gate_fwd_rows(int64_t rows, int32_t io_dtype, int32_t heads, int32_t gate_ld, float eps, const void* x,
                                         const void* gate, const float* weight, void* y, float* inv_rms, void* stream) {
    if (rows <= 0 || rows >= (1LL << 31) || heads <= 0 || rows % heads != 0 || gate_ld < heads * 128) return KDA_ERR_BAD_SHAPE;
    if (!x || !gate || !weight || !y || !inv_rms) return KDA_ERR_NULL;
    if (gate_ld % 8 != 0 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(y) |
                              reinterpret_cast<uintptr_t>(weight)) % 16) != 0)
        return KDA_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    const int nb4 = (int)std::min<long long>((rows + 8 * pw::kRmsRows - 1) / (8 * pw::kRmsRows), 148LL * 8);
    if (io_dtype == KDA_DTYPE_BF16) KDA_LAUNCH("rmsnorm_fwd_kernel", st, pw::rmsnorm_fwd128_kernel<true, true><<<nb4, 256, 0, st>>>(rows, heads, gate_ld, eps, x, gate, weight, y, inv_rms));
    else KDA_LAUNCH("rmsnorm_fwd_kernel", st, pw::rmsnorm_fwd128_kernel<false, true><<<nb4, 256, 0, st>>>(rows, heads, gate_ld, eps, x, gate, weight, y, inv_rms));
    return launch_status();
}

extern "C" size_t kda_rmsnorm_gate_bwd_scratch_bytes(int64_t rows, int32_t dim) {
    return align_up((size_t)rms_blocks(rows > 0 ? rows : 1) * dim * sizeof(float), 256);
}

namespace {
// part: one row of partials per block
template <int PARTS>
void rms_bwd_launch(int nb, int64_t rows, int32_t dim, int32_t io_dtype, const void* x, const void* gate, const float* weight, const float* inv_rms,
                    const void* d_y, void* dx, void* dgate, float* part, cudaStream_t st) {
    const size_t smem = (size_t)8 * dim * sizeof(float);
    const bool vec = dim % 128 == 0 &&
                     ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(d_y) |
                       reinterpret_cast<uintptr_t>(dx) | reinterpret_cast<uintptr_t>(dgate) | reinterpret_cast<uintptr_t>(weight)) % 16) == 0;
    const bool bf16 = io_dtype == KDA_DTYPE_BF16;
    if (vec && dim == 128) {
        if (bf16) KDA_LAUNCH("rmsnorm_bwd_kernel", st, pw::rmsnorm_bwd128_kernel<true, false, PARTS><<<nb, 256, 0, st>>>(rows, 1, 128, x, gate, weight, inv_rms, d_y, dx, dgate, part));
        else KDA_LAUNCH("rmsnorm_bwd_kernel", st, pw::rmsnorm_bwd128_kernel<false, false, PARTS><<<nb, 256, 0, st>>>(rows, 1, 128, x, gate, weight, inv_rms, d_y, dx, dgate, part));
    } else if (bf16) {
        if (vec) KDA_LAUNCH("rmsnorm_bwd_kernel", st, pw::rmsnorm_bwd_kernel<true, true, PARTS><<<nb, 256, smem, st>>>(rows, dim, x, gate, weight, inv_rms, d_y, dx, dgate, part));
        else KDA_LAUNCH("rmsnorm_bwd_kernel", st, pw::rmsnorm_bwd_kernel<true, false, PARTS><<<nb, 256, smem, st>>>(rows, dim, x, gate, weight, inv_rms, d_y, dx, dgate, part));
    } else {
        if (vec) KDA_LAUNCH("rmsnorm_bwd_kernel", st, pw::rmsnorm_bwd_kernel<false, true, PARTS><<<nb, 256, smem, st>>>(rows, dim, x, gate, weight, inv_rms, d_y, dx, dgate, part));
        else KDA_LAUNCH("rmsnorm_bwd_kernel", st, pw::rmsnorm_bwd_kernel<false, false, PARTS><<<nb, 256, smem, st>>>(rows, dim, x, gate, weight, inv_rms, d_y, dx, dgate, part));
    }
}
[[nodiscard]] int rms_dw_launch(int nb, int32_t dim, const float* part, float* dweight, cudaStream_t st) {
    pw::ColumnSumItems outs = {};
    outs.out[0] = dweight;
    return column_sums("rmsnorm_dw_reduce_kernel", 1, nb, dim, part, outs, 0, st);
}
}  // namespace

extern "C" int kda_rmsnorm_gate_bwd(int64_t rows, int32_t dim, int32_t io_dtype, const void* x, const void* gate,
                                    const float* weight, const float* inv_rms, const void* d_y, void* dx, void* dgate,
                                    float* dweight, void* scratch, size_t scratch_bytes, void* stream) {
    if (rows < 0 || dim <= 0 || dim > 1024) return KDA_ERR_BAD_SHAPE;
    if (!weight || !dweight) return KDA_ERR_NULL;
    if (rows > 0 && (!x || !gate || !inv_rms || !d_y || !dx || !dgate)) return KDA_ERR_NULL;
    if (!scratch || scratch_bytes < kda_rmsnorm_gate_bwd_scratch_bytes(rows, dim)) return KDA_ERR_WORKSPACE;
    cudaStream_t st = (cudaStream_t)stream;
    const int nb = rows > 0 ? rms_blocks(rows) : 0;
    float* part = static_cast<float*>(scratch);
    if (nb > 0) rms_bwd_launch<pw::kRmsAll>(nb, rows, dim, io_dtype, x, gate, weight, inv_rms, d_y, dx, dgate, part, st);
    return rms_dw_launch(nb, dim, part, dweight, st);
}

extern "C" int kda_rmsnorm_gate_bwd_rows(int64_t rows, int32_t io_dtype, int32_t heads, int32_t gate_ld, const void* x, const void* gate,
                                         const float* weight, const float* inv_rms, const void* d_y, void* dx, void* dgate,
                                         float* dweight, void* scratch, size_t scratch_bytes, void* stream) {
    if (rows <= 0 || rows >= (1LL << 31) || heads <= 0 || rows % heads != 0 || gate_ld < heads * 128) return KDA_ERR_BAD_SHAPE;
    if (!x || !gate || !weight || !inv_rms || !d_y || !dx || !dgate || !dweight) return KDA_ERR_NULL;
    if (!scratch || scratch_bytes < kda_rmsnorm_gate_bwd_scratch_bytes(rows, 128)) return KDA_ERR_WORKSPACE;
    if (gate_ld % 8 != 0 || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(gate) | reinterpret_cast<uintptr_t>(d_y) |
                              reinterpret_cast<uintptr_t>(dx) | reinterpret_cast<uintptr_t>(dgate) | reinterpret_cast<uintptr_t>(weight)) % 16) != 0)
        return KDA_ERR_UNSUPPORTED;
    cudaStream_t st = (cudaStream_t)stream;
    const int nb = rms_blocks(rows);
    float* part = static_cast<float*>(scratch);
    if (io_dtype == KDA_DTYPE_BF16) KDA_LAUNCH("rmsnorm_bwd_kernel", st, pw::rmsnorm_bwd128_kernel<true, true><<<nb, 256, 0, st>>>(rows, heads, gate_ld, x, gate, weight, inv_rms, d_y, dx, dgate, part));
    else KDA_LAUNCH("rmsnorm_bwd_kernel", st, pw::rmsnorm_bwd128_kernel<false, true><<<nb, 256, 0, st>>>(rows, heads, gate_ld, x, gate, weight, inv_rms, d_y, dx, dgate, part));
    pw::ColumnSumItems outs = {};
    outs.out[0] = dweight;
    return column_sums("rmsnorm_dw_reduce_kernel", 1, nb, 128, part, outs, 0, st);
}

// =============================================================================================
// Allocation-free variant of the gated-RMSNorm backward
// =============================================================================================
// The regular backward needs a caller-provided scratch buffer for the per-block partial sums of the
// weight gradient.  Some callers have nowhere to get one: code running against a frozen memory plan
// (a serving engine that sized all of its device memory at start-up), a plugin that is handed tensors
// but no allocator, or anything that must not call cudaMalloc because that call synchronises the
// device.  For them dx holds the partials first - at most ceil(rows / 8) rows of dim floats, about a
// quarter of it in bf16 and an eighth in float32 - and is written after they have been summed.  The
// inputs are read twice for it; in return nothing is shared between calls, so they may overlap on
// different streams and in graphs.  Up to 8 rows need no partials: their one block writes the
// gradient itself.
extern "C" int kda_rmsnorm_gate_bwd_static(int64_t rows, int32_t dim, int32_t io_dtype, const void* x, const void* gate,
                                           const float* weight, const float* inv_rms, const void* d_y, void* dx,
                                           void* dgate, float* dweight, void* stream) {
    constexpr int kStaticMaxDim = 256;
    if (rows < 0 || dim <= 0) return KDA_ERR_BAD_SHAPE;
    if (dim > kStaticMaxDim) return KDA_ERR_UNSUPPORTED;
    if (!weight || !dweight) return KDA_ERR_NULL;
    if (rows > 0 && (!x || !gate || !inv_rms || !d_y || !dx || !dgate)) return KDA_ERR_NULL;
    cudaStream_t st = (cudaStream_t)stream;
    if (rows == 0) return rms_dw_launch(0, dim, nullptr, dweight, st);
    const int nb = rms_blocks(rows);
    // bf16 rows may start at an odd element, floats may not: 2 bytes of slack, and more than 8 rows have room for it
    float* part = nb == 1 ? dweight : reinterpret_cast<float*>((reinterpret_cast<uintptr_t>(dx) + 3) / 4 * 4);
    rms_bwd_launch<pw::kRmsWeight>(nb, rows, dim, io_dtype, x, gate, weight, inv_rms, d_y, dx, dgate, part, st);
    if (nb > 1)
        if (int rc = rms_dw_launch(nb, dim, part, dweight, st)) return rc;
    rms_bwd_launch<pw::kRmsInputs>(nb, rows, dim, io_dtype, x, gate, weight, inv_rms, d_y, dx, dgate, nullptr, st);
    return launch_status();
}
