// Workspace of the tensor-core lane: bf16 operand panels per chunk-head (ch = slot*H + h), K = V = 128.
#pragma once

#include <cuda_bf16.h>

#include "simt_ws.cuh"

namespace kda {
namespace tc {

// Short causal convolution (width 4, SiLU) folded into the intra-chunk forward of a forward-only call: q, k, v of that
// call are the convolutions' INPUTS and the kernel forms the activations itself, so they are never written to memory.
struct ConvPrep {
    const void* w[3];       // weights of the q, k, v convolutions, [H*128][4]
    int wf32;               // 1: float32 weights (rounded to bf16 as loaded, like the stand-alone kernel), 0: bf16
    long long x_ld;         // elements between consecutive tokens of the convolutions' inputs
};

struct TcWs {
    __nv_bfloat16* WT;          // [nch][128][64]   rows = key, cols = token
    __nv_bfloat16 *R, *E;       // [nch][64][128]   rows = token, cols = key
    __nv_bfloat16* AT;          // [nch][64][64]    A transposed: [source s][target i]
    __nv_bfloat16* UT;          // [nch][128][64]   U transposed: [value][token]
    __nv_bfloat16* Tp;          // [nch][64][64]    T = (I + M)^-1, row-major
    __nv_bfloat16* Mt;          // [nch][64][64]    M before the beta scaling, strictly lower, row-major
    __nv_bfloat16* Hp;          // [nch][128][128]  chunk-start state: [key][value] from a walk, [value][key] from split scans
    __nv_bfloat16* ZT;          // [nch][8192]      Z: [token][value], [value][token]
    __nv_bfloat16* dHp;         // [nch][128][128]  adjoint of each chunk's outgoing state, as Hp
    __nv_bfloat16* dZT;         // [nch][8192]      dZ, as ZT
    // split scans only
    __nv_bfloat16* Pn;          // [nch][128][128]  W^T E: [key k][key k'], the state-to-state part of the chunk transition
    __nv_bfloat16* RmT;         // [nch][128][64]   (R - A W)^T: [key][token]
    __nv_bfloat16* Pp;          // [nch][128][128]  composite state-to-state maps at each chunk start
    __nv_bfloat16* fin_panel;   // [n_seq*H*units][128][128]  final state of every scan unit as a bf16 panel
    float* seg_fin;             // [n_seq*H*units][128][128]  the same in float32
    int nseg;                   // scan_segments(): 1 - no split scans -, or their segments per (sequence, head); units = 2 * nseg - 1
    float* decay_end;           // [nch][128]       exp(G_end)
    int* status;                // device status word (0 = ok); points at the workspace's word (simt::Ws::status)
    int fwd_only;               // 1: the backward-only panels (T, M~, Z, dH', dZ, Rm^T) have no storage and are not written
};

// Optional epilogue of the kernel that forms the outputs (a walk, or the split scans' chunk-output kernel): the gated RMSNorm that follows the operator in the layer
// (y = o * rsqrt(mean(o^2) + eps) * weight * sigmoid(gate) over the 128 values of a token and head), applied to the
// output tile while it is still on chip.  o is written as well when the caller passes it: the norm's backward needs it.
struct NormEpilogue {
    const __nv_bfloat16* gate;   // [tokens][H][128] in rows gate_ld elements apart, or nullptr: no epilogue
    const float* weight;         // [128]
    float eps;
    __nv_bfloat16* y;            // [tokens][H][128]
    float* inv_rms;              // [tokens][H], or nullptr: not wanted (no backward follows)
    long long gate_ld;
};

// How a batch goes through its recurrences: 1 - walks (kda_tc_walk.cu), two blocks to a (sequence, head) -, or the number of segments of
// split scans (kda_tc_pscan.cu).  The decision uses the shape alone, so the forward and the backward of a call agree; split, every sequence of
// the batch is cut into the same number of segments, short ones into segments of one chunk or none.
// A walk's step takes about 1.2 us forward and 1.0 back and has everything behind it done; split scans take a quarter of a step's 0.8 us for
// the chain, but 48 + 176 KB more of memory traffic for every chunk of every recurrence, and three more launches each way.  So the walk
// falls behind where there are few recurrences and many chunks.  Forward and backward in us, four segments / walk, by recurrences x chunks:
// 1 x 16: 86 / 82, 2 x 24: 90 / 96, 6 x 20: 92 / 90, 8 x 24: 107 / 109, 12 x 24: 119 / 113, 12 x 32: 154 / 156 (a whole layer 356 / 352), 14 x 40: 193 /
// 193, 16 x 40: 219 / 213, 16 x 64: 295 / 309, 18 x 64: 328 / 327, 18 x 96: 459 / 469, 20 x 96: 500 / 494, 24 x 96: 608 / 549: chunks * (24 - recurrences) > 384.
// Eight segments halve the chain again and lengthen the fix-up's by four products; worth it where the chain is long and SMs are idle (4 / 8
// segments: 1 x 64 109 / 109, 1 x 128 139 / 125, 2 x 192 219 / 197, 6 x 192 361 / 346; 6 x 128 270 / 266, 6 x 64 166 / 170, 8 x 128 313 / 315).
// A walk is as long as its longest chain.  The lengths of a packed batch live on the device, so that chain is taken for 1.5 times the mean of
// two or three sequences and 2.25 times that of more (uniform lengths between 256 and 8,192 make 1.3 to 1.9, one long document among short ones more).
// Up to 21 recurrences, seven units each to the SMs at once, then split from 16 chunks on (sequences x heads, us split / walk, lengths from 256 to
// 8,192: 20 x 1 406 / 473, 4 x 4 340 / 438, 16 x 1 330 / 418, 2 x 8 307 / 350, 6 x 3 293 / 328, 7 x 3 317 / 340, 10 x 2 481 / 512; up to 3,000: 4 x 4 191 / 201, 10
// x 2 205 / 207, 7 x 3 205 / 197, 5 x 3 158 / 150).  Up to 33 there is little in it for uniform lengths, and two segments are safer (5 x 6 528 / 539, 6 x 4
// 358 / 369, 4 x 8 573 / 571, 31 x 1 571 / 567, 16 x 2 545 / 535, 8 x 4 727 / 678; one document of 900 chunks and 30 of 4: 1,384 / 2,021); with fewer than 32
// chunks the walk's fewer launches count (3 x 8 236 / 223, 31 x 1 244 / 225, 16 x 2 262 / 240).  Beyond, the walk is ahead for those lengths (40 x 1 705 / 647,
// 49 x 1 787 / 709, 3 x 16 1,081 / 912) and behind for a batch that one document makes up.
inline int scan_segments(const KdaChunkShape& sh) {
    if (sh.n_seq <= 0) return 1;
    const bool packed = sh.seq_len <= 0 && sh.n_seq > 1;
    const long long rec = (long long)sh.n_seq * sh.heads;
    const long long chunks = sh.seq_len > 0 ? (sh.seq_len + 63) / 64 : (sh.tokens / 64) / sh.n_seq;      // of a sequence, in the mean
    const int quarters = !packed ? 4 : (sh.n_seq < 4 ? 6 : 9);                                           // of the mean to the longest
    if (rec < (packed ? 22 : 21) && chunks * (6 * quarters - rec) > 384 && (!packed || chunks >= 16)) return rec <= 6 && chunks >= 96 ? 8 : 4;
    return quarters == 9 && rec <= 33 && chunks >= 32 ? 2 : 1;      // 2 nseg - 1 scan units to a recurrence
}

inline TcWs carve_tc(const KdaChunkShape& sh, void* mem, size_t* bytes = nullptr) {
    TcWs t;
    const size_t nch = (size_t)simt::slots_for(sh, false) * sh.heads;
    const size_t bw = sh.forward_only ? 0 : 1;      // panels only the backward reads
    simt::Carver c(mem);
    t.WT = c.take<__nv_bfloat16>(nch * 8192);
    t.R = c.take<__nv_bfloat16>(nch * 8192);
    t.E = c.take<__nv_bfloat16>(nch * 8192);
    t.AT = c.take<__nv_bfloat16>(nch * 4096);
    t.UT = c.take<__nv_bfloat16>(nch * 8192);
    t.Tp = c.take<__nv_bfloat16>(bw * nch * 4096);
    t.Mt = c.take<__nv_bfloat16>(bw * nch * 4096);
    t.nseg = scan_segments(sh);
    const size_t split = t.nseg > 1 ? 1 : 0;         // panels of the split scans and what follows them
    t.Hp = c.take<__nv_bfloat16>((bw | split) * nch * 16384);
    t.ZT = c.take<__nv_bfloat16>(bw * nch * 8192);
    t.dHp = c.take<__nv_bfloat16>(bw * nch * 16384);
    t.dZT = c.take<__nv_bfloat16>(bw * nch * 8192);
    t.Pn = c.take<__nv_bfloat16>(split * nch * 16384);
    t.RmT = c.take<__nv_bfloat16>(split * bw * nch * 8192);
    const size_t units = split * sh.n_seq * sh.heads * (2 * t.nseg - 1);
    t.Pp = c.take<__nv_bfloat16>(split * nch * 16384);
    t.fin_panel = c.take<__nv_bfloat16>(units * 16384);
    t.seg_fin = c.take<float>(units * 16384);
    t.decay_end = c.take<float>(nch * 128);
    t.status = c.take<int>(64);
    t.fwd_only = sh.forward_only ? 1 : 0;
    if (bytes) *bytes = align_up(c.off, 256);
    return t;
}

}  // namespace tc
}  // namespace kda
