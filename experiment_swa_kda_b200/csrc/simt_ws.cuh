// Workspace layout of the float32 chunk lane: what the forward leaves for the
// backward (Ws) and the backward's own scratch (Scr).  All arrays are padded to
// 64-wide tiles: Kp = ceil64(K), Vp = ceil64(V); chunk-head index ch = slot*H + h.
#pragma once

#include "common.cuh"

namespace kda {
namespace simt {

// Which tokens each 64-token chunk slot covers.  For a packed batch the lengths live on the device, and a kernel of their own
// tabulates them; a fixed-length batch is arithmetic, which saves that launch and the loads every kernel would start with.
// 77 tokens through a layer 71.7 -> 65.6 us, the chain of 2 x 4,096 tokens 243 -> 235, float32 forward and backward of 256
// tokens 131 -> 127.
struct ChunkTable {
    int *seq, *tok0, *len;      // [nslots]
    int* seq_chunk0;            // [n_seq + 1]
    int* seq_order;             // [n_seq] sequences by falling chunk count: the order the state scans start them in
    int seq_len, per_seq;       // fixed-length batch: tokens and chunks of a sequence; per_seq 0: the tables hold
    __device__ __forceinline__ void span(int slot, int& t0, int& n) const {
        if (per_seq > 0) {
            const int s = slot / per_seq, j = slot - s * per_seq;
            t0 = s * seq_len + j * kChunk;
            n = min(kChunk, seq_len - j * kChunk);
        } else {
            t0 = tok0[slot];
            n = len[slot];
        }
    }
    __device__ __forceinline__ int first_chunk(int s) const { return per_seq > 0 ? s * per_seq : seq_chunk0[s]; }
    __device__ __forceinline__ bool starts_sequence(int slot) const { return per_seq > 0 ? slot % per_seq == 0 : seq_chunk0[seq[slot]] == slot; }
};

// Every forward starts with a clean status word and says where the host mirrors it: its first kernel, one thread.
__device__ __forceinline__ void start_status(int* status, int* mirror) {
    *status = 0;
    *reinterpret_cast<int**>(status + 2) = mirror;
}

struct Ws {
    ChunkTable tab;
    // float32 lane, per chunk-head.  R = qn e^G, E = kn Ed; ...T arrays are transposed
    float *kn, *G;              // [64][Kp]   unit k, cumulative log-decay
    float* Ed;                  // [64][Kp]   e^{G_end - G}, from sums that start at the chunk's end
    float *qn, *Rm;             // [64][Kp]   scaled unit q; R - A W (backward only)
    float *W, *WT, *RT;         // [64][Kp], [Kp][64], [Kp][64]
    float* Z;                   // [64][Vp]   U after the intra-chunk step, Z after the output kernel
    float *AT, *A, *T;          // [64][64]   A and T: backward only
    float *PT, *P;              // [Kp][Kp]   (E^T W)^T, and E^T W for the adjoint scan (backward only)
    float* Hc;                  // [Kp][Vp]   E^T U, replaced by the chunk-start state in the scan
    float* dec;                 // [Kp]       exp(G_end)
    float *qinv, *kinv, *beta;  // [nch][64]
    int* status;                // device status word of the forward / backward pair that owns this workspace (0 = ok)
    int nslots, H, K, V, Kp, Vp;
};

struct Scr {
    float* dHn;             // [nch][Kp][Vp]   Rm^T dO, replaced by the adjoint of each chunk's outgoing state in the scan
    float *dqn, *dkn, *dG;  // [nch][64][Kp]
    float* dA;              // [nch][64][64]
    float* dZ;              // [nch][64][Vp]   only when V > 64 (one value tile stays on chip)
    int* next;              // tensor-core lane: chunk-heads handed out by the intra-chunk backward
};

inline int slots_for(const KdaChunkShape& sh, bool varlen_hint) {
    // Upper bound on the number of 64-token chunk slots.  Packed batches may end every
    // sequence with a ragged chunk; the same bound is used for fixed-length batches so
    // that forward and backward agree without knowing whether cu_seqlens was given.
    (void)varlen_hint;
    if (sh.seq_len > 0 && (long long)sh.n_seq * sh.seq_len == sh.tokens)
        return sh.n_seq * ceil_div(sh.seq_len, kChunk);
    return sh.tokens / kChunk + sh.n_seq;
}

struct Carver {
    char* base;
    size_t off = 0;
    explicit Carver(void* p) : base(static_cast<char*>(p)) {}
    template <class T>
    T* take(size_t n) {
        off = align_up(off, 256);
        T* p = base ? reinterpret_cast<T*>(base + off) : nullptr;
        off += n * sizeof(T);
        return p;
    }
};

// The tensor-core lane keeps only the chunk table and the per-row scalars here (its operand panels live in
// tc::TcWs); the large float32 arrays are carved with zero length for it.
inline Ws carve_ws(const KdaChunkShape& sh, void* mem, size_t* bytes = nullptr) {
    Ws w;
    const size_t big = sh.lane == KDA_LANE_TC ? 0 : 1;
    w.H = sh.heads; w.K = sh.key_dim; w.V = sh.value_dim;
    w.Kp = ceil_div(sh.key_dim, 64) * 64;
    w.Vp = ceil_div(sh.value_dim, 64) * 64;
    w.nslots = slots_for(sh, false);
    const size_t nch = (size_t)w.nslots * w.H;
    Carver c(mem);
    w.tab.seq = c.take<int>(w.nslots + 1);
    w.tab.tok0 = c.take<int>(w.nslots + 1);
    w.tab.len = c.take<int>(w.nslots + 1);
    w.tab.seq_chunk0 = c.take<int>(sh.n_seq + 1);
    w.tab.seq_order = c.take<int>(sh.n_seq);
    w.tab.seq_len = sh.seq_len;      // 0 with cu_seqlens
    w.tab.per_seq = ceil_div(sh.seq_len, kChunk);
    const size_t bw = sh.forward_only ? 0 : big;      // arrays only a backward reads
    w.kn = c.take<float>(big * nch * 64 * w.Kp);
    w.G = c.take<float>(big * nch * 64 * w.Kp);
    w.Ed = c.take<float>(big * nch * 64 * w.Kp);
    w.qn = c.take<float>(bw * nch * 64 * w.Kp);
    w.Rm = c.take<float>(bw * nch * 64 * w.Kp);
    w.W = c.take<float>(big * nch * 64 * w.Kp);
    w.WT = c.take<float>(big * nch * 64 * w.Kp);
    w.RT = c.take<float>(big * nch * 64 * w.Kp);
    w.Z = c.take<float>(big * nch * 64 * w.Vp);
    w.AT = c.take<float>(big * nch * 4096);
    w.A = c.take<float>(bw * nch * 4096);
    w.T = c.take<float>(bw * nch * 4096);
    w.PT = c.take<float>(big * nch * w.Kp * w.Kp);
    w.P = c.take<float>(bw * nch * w.Kp * w.Kp);
    w.Hc = c.take<float>(big * nch * w.Kp * w.Vp);
    w.dec = c.take<float>(big * nch * w.Kp);
    w.qinv = c.take<float>(nch * 64);
    w.kinv = c.take<float>(nch * 64);
    w.beta = c.take<float>(nch * 64);
    w.status = c.take<int>(64);
    if (bytes) *bytes = align_up(c.off, 256);
    return w;
}

inline Scr carve_scr(const KdaChunkShape& sh, void* mem, size_t* bytes = nullptr) {
    Scr s;
    const int Kp = ceil_div(sh.key_dim, 64) * 64, Vp = ceil_div(sh.value_dim, 64) * 64;
    const size_t nch = sh.lane == KDA_LANE_TC ? 0 : (size_t)slots_for(sh, false) * sh.heads;   // float32 lane only
    Carver c(mem);
    s.dHn = c.take<float>(nch * Kp * Vp);
    s.dqn = c.take<float>(nch * 64 * Kp);
    s.dkn = c.take<float>(nch * 64 * Kp);
    s.dG = c.take<float>(nch * 64 * Kp);
    s.dA = c.take<float>(nch * 4096);
    s.dZ = c.take<float>(Vp > 64 ? nch * 64 * Vp : 0);
    s.next = c.take<int>(sh.lane == KDA_LANE_TC ? 64 : 0);
    if (bytes) *bytes = align_up(c.off, 256);
    return s;
}

}  // namespace simt
}  // namespace kda
