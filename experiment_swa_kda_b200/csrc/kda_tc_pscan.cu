// Tensor-core lane (K = V = 128): the state recurrences as affine scans, for batches of so few and so long sequences that their steps
// are cut into segments that run side by side (scan_segments; the others walk, kda_tc_walk.cu).
//
// With Z = U - W H substituted, one chunk maps its incoming state H to
//     H' = exp(G_end) . H  -  (W^T E)^T-contracted H  +  E^T U          i.e.  H'^T = dec . H^T - H^T Pn + U^T E
// and the adjoint recurrence of the backward is its transpose,
//     dH^T = dec . dH'^T - dH'^T Pn^T + dO^T (R - A W).
// Pn = W^T E and Rm = R - A W do not depend on the state, so they are computed for all chunks in parallel
// (at the end of the intra-chunk forward kernel) and the sequential part of a chunk step shrinks to ONE UMMA chain between two register passes:
//     pack state -> bf16 A operand | D = state-independent term (issued a step early) - state x Pn | state = dec . state + D
// Everything else that used to sit inside the scans runs chunk-parallel on all SMs afterwards:
//     forward   Z^T = U^T - (W H)^T,  O^T = (R H)^T + (A Z)^T      from the chunk-start states the scan stored
//     backward  dZ^T = dO^T A + dH'^T E^T                          from the state adjoints the scan stored
// All products are written transposed so that M = 128 (value index = TMEM lane) for every UMMA.
// Restates reference chunk_wy_forward.cu:940-1275 (state scan), 1498-1588 (output) and
// chunk_wy_backward.cu:2445-2562 (adjoint scan); the algebraic regrouping is this implementation's.

#include "common.cuh"
#include "simt_ws.cuh"
#include "tc_common.cuh"
#include "tc_ws.cuh"

namespace kda {
namespace tc {

int make_map_bf16_ld(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_cols, uint32_t box_rows);
int make_map_bf16(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);

// ---------------------------------------------------------------------------------------------
// affine scan: one CTA per unit of a (sequence, head) walks its chunks in order (forward) or in reverse (backward)
//     forward    S = H^T   [v][k]:   S' = dec . S - S Pn   + U^T E           stores S (chunk-start state) per chunk
//     backward   S = dH'^T [v][k]:   S' = dec . S - S Pn^T + dO^T Rm         stores S (adjoint of the chunk's outgoing state)
// Threads are specialised by warp; they meet only through mbarriers:
//   state warpgroups (kScanGroups of them): thread (g, v) owns S[v][g*kScanCols .. (g+1)*kScanCols) in registers
//   next warp   one lane issues the TMA loads, as far ahead as the ring reaches
//   next warp   one lane issues every UMMA
//   last warp   one lane issues the TMA stores of the state panels
// The loads of a step are two 32 KB items of one ring, the state-independent operands and then Pn, each handed back when
// its own product is complete: five slots reach two steps ahead.  With two whole steps in the ring a load
// could start only when the step before the last had ended, and 1,700 of a step's 2,600 cycles went by waiting for it
// (16 recurrences in 4 segments of 32 steps: 60 -> 51 us; 6 of 16: 27 -> 24.5).
// TMEM: the accumulator is double-buffered (columns 0 / 128) so that the state-independent product of step c+1 is
// issued while the state threads still read the accumulator of step c; the bf16 state panel the state product reads as
// its A operand sits at column 256.  Its copy in shared memory, for the TMA store, is written behind the arrival that releases
// the product and has the rest of the step to leave.
// ---------------------------------------------------------------------------------------------
struct AffineScanArgs {
    simt::ChunkTable tab;
    const float* decay_end;   // [nch][128] exp(G_end)
    const float* s_in;        // V-first initial state (forward: h0, backward: cotangent of the final state), or null
    int H;
    int* status;
    // Few long sequences: most SMs would idle behind a handful of 64-step chains.  The steps of every
    // (sequence, head) are cut into nseg segments that run side by side as 2 nseg - 1 units: unit 0 walks segment 0 from
    // s_in; for every later segment k, unit 2k-1 walks it from a zero state (its "local" states L) and unit 2k walks its
    // state-to-state map alone, from the identity and without the state-independent term (the composites P of the
    // affine maps).  The true state at a chunk of segment k is S_k P + L with S_k the state at the segment's start;
    // tc_scan_fixup_kernel forms the S_k (a chain of nseg - 1 small products) and then the chunk states, chunk-parallel.
    // Units leave their final state as float32 (seg_fin) and as a bf16 panel (through mF).
    int nseg;
    float* seg_fin;           // [n_seq*H*(2 nseg - 1)][128][128]
};

// first scan step of segment k of a sequence of n steps
__host__ __device__ __forceinline__ int seg_begin(int k, int nseg, int n) { return (int)(((long long)k * n) / nseg); }

constexpr int kScanItem = 32768;                            // Pn, or X 16 KB (U^T or Rm^T) | Y 16 KB (E or dO)
constexpr int kScanSlots = 5;
constexpr int kScanMapSlots = 3;                            // composites load Pn only; more would outrun the ring of decays
constexpr int kScanPanel = kScanSlots * kScanItem;          // 2 x 32 KB  bf16 state panel of step c in c % 2, [2 k-blocks][128 rows x 128 B]
constexpr int kScanDec = kScanPanel + 65536;                // exp(G_end) of step c in slot c % 4: [4][128] floats
constexpr int kScanBars = kScanDec + 2048;
constexpr int kAffineScanSmem = kScanBars + 256;            // 768 bytes below the limit: no room to align the base, which has to be 1024-aligned as it is
constexpr int kScanGroups = 2;                              // state warpgroups: each thread owns 128 / kScanGroups columns of a row
constexpr int kScanCols = 128 / kScanGroups;
constexpr uint32_t kScanPanelCol = 256;                     // TMEM column of the bf16 state panel (64 columns: 128 keys as pairs)
constexpr int kAffineScanThreads = (4 * kScanGroups + 3) * 32;

template <bool kBwd>
__global__ void __launch_bounds__(kAffineScanThreads, 1)
    tc_affine_scan_kernel(const __grid_constant__ CUtensorMap mP, const __grid_constant__ CUtensorMap mX,
                          const __grid_constant__ CUtensorMap mY, const __grid_constant__ CUtensorMap mS,
                          const __grid_constant__ CUtensorMap mS2, const __grid_constant__ CUtensorMap mF, AffineScanArgs p) {
    extern __shared__ __align__(1024) uint8_t sm[];
    uint8_t* Sop = sm + kScanPanel;
    float (*dec_ring)[128] = reinterpret_cast<float (*)[128]>(sm + kScanDec);
    // full: an item has landed.  free: the product that reads it is complete.  sop: all state threads have packed the state panel
    // into tensor memory, pan: into shared memory.  out: the store has read that panel.  Both have one barrier per buffer: the store
    // warp gives `out` of panel c - 1 before it looks for panel c, and by then a barrier of both buffers could have counted panels c
    // and c + 1, which reads like none; panel c + 2 waits for `out` of panel c.  mma: the step's accumulator is complete.
    uint64_t* bar_full = reinterpret_cast<uint64_t*>(sm + kScanBars);
    uint64_t* bar_free = bar_full + kScanSlots;
    uint64_t &bar_sop = bar_free[kScanSlots], &bar_mma = bar_free[kScanSlots + 1];
    uint64_t *bar_pan = bar_free + kScanSlots + 2, *bar_out = bar_pan + 2;
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bar_out + 2);
    volatile int& abort_flag = *reinterpret_cast<volatile int*>(bar_out + 3);
    if (smem_u32(sm) & 1023u) {      // the swizzled tiles would be misread
        if (threadIdx.x == 0) raise_status(p.status, 56);
        return;
    }

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int v = (warp & 3) * 32 + lane;          // value row = TMEM lane
    const int units = 2 * p.nseg - 1;             // grid (sequences x units, heads)
    const int seq = blockIdx.x / units, role = blockIdx.x % units, h = blockIdx.y, H = p.H;
    const int c_begin = p.tab.first_chunk(seq), c_end = p.tab.first_chunk(seq + 1);
    const int n_total = c_end - c_begin;
    const int seg = (role + 1) >> 1;                             // segment this unit walks
    const int step0 = seg_begin(seg, p.nseg, n_total);           // its first step, in the sequence's scan order
    const int n = seg_begin(seg + 1, p.nseg, n_total) - step0;
    const bool composite = role > 0 && (role & 1) == 0;          // state-to-state map only: no state-independent term
    const int unit = (seq * H + h) * units + role;
    auto slot_of = [&](int c) { return kBwd ? c_end - 1 - (step0 + c) : c_begin + step0 + c; };   // chunk slot of step c

    if (warp == 0 && elect_one()) {
        for (int i = 0; i < kScanSlots; ++i) {
            mbar_init(&bar_full[i], 1);
            mbar_init(&bar_free[i], 1);
        }
        mbar_init(&bar_sop, 4 * kScanGroups);      // one arrival per state warp
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_pan[i], 4 * kScanGroups);
            mbar_init(&bar_out[i], 1);
        }
        mbar_init(&bar_mma, 1);
        mbar_fence_init();
        abort_flag = 0;
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 512);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    // item 2c of the ring is X | Y of step c, item 2c + 1 its Pn; a composite's Pn is item c of a shorter ring
    auto slot_xy = [&](int c) { return (2 * c) % kScanSlots; };
    auto parity_xy = [&](int c) { return (uint32_t)(2 * c / kScanSlots) & 1u; };
    auto slot_p = [&](int c) { return composite ? c % kScanMapSlots : (2 * c + 1) % kScanSlots; };
    auto parity_p = [&](int c) { return (uint32_t)(composite ? c / kScanMapSlots : (2 * c + 1) / kScanSlots) & 1u; };

    if (warp == 4 * kScanGroups) {
        // ------------------------------------------------------------------ load warp
        if (elect_one()) {
            const int depth = composite ? kScanMapSlots : kScanSlots, items = composite ? n : 2 * n;
            auto slot_item = [&](int i) { return i % depth; };
            auto parity_item = [&](int i) { return (uint32_t)(i / depth) & 1u; };
            auto issue_load = [&](int i) {
                const int c = composite ? i : i >> 1, cs = slot_of(c), ch = cs * H + h, sl = slot_item(i);
                uint8_t* b = sm + sl * kScanItem;
                uint64_t* bar = &bar_full[sl];
                if (composite || (i & 1)) {
                    mbar_expect_tx(bar, 32768 + 512);
                    bulk_load_1d(dec_ring[c & 3], p.decay_end + (size_t)ch * 128, 512, bar);
                    for (int nb = 0; nb < 2; ++nb) tma_load_2d(b + nb * 16384, &mP, bar, nb * 64, ch * 128);
                } else {
                    mbar_expect_tx(bar, 32768);
                    tma_load_2d(b, &mX, bar, 0, ch * 128);                  // U^T / Rm^T: [128][64]
                    int tok0 = 0, len;
                    if (kBwd) p.tab.span(cs, tok0, len);
                    for (int nb = 0; nb < 2; ++nb) tma_load_2d(b + 16384 + nb * 8192, &mY, bar, kBwd ? h * 128 + nb * 64 : nb * 64, kBwd ? tok0 : ch * 64);
                }
            };
            int issued = 0;
            for (; issued < depth && issued < items; ++issued) issue_load(issued);
            bool ok = true;
            while (issued < items && ok) {     // a slot is free once the product that reads its item is complete
                ok = mbar_wait(&bar_free[slot_item(issued)], parity_item(issued) ^ 1u, p.status, 50);
                if (ok) issue_load(issued++);
                else abort_flag = 1;
            }
            if (!ok)   // unwinding: the copies in flight must land before the block may exit
                for (int i = issued > depth ? issued - depth : 0; i < issued; ++i) mbar_wait(&bar_full[slot_item(i)], parity_item(i), nullptr, 0);
        }
    } else if (warp == 4 * kScanGroups + 1) {
        // ------------------------------------------------------------------ UMMA thread
        if (kBwd && n > 0 && !composite && step0 == 0) {
            // Only a sequence's last chunk (the adjoint scan's first step) can be ragged; the dO rows past its tail
            // belong to the next sequence and are blanked by the whole warp before lane 0 issues the product on them.
            int tok0, len0;
            p.tab.span(slot_of(0), tok0, len0);
            if (len0 < 64) {
                if (mbar_wait(&bar_full[0], 0, p.status, 51)) {
                    for (int idx = lane; idx < (64 - len0) * 16; idx += 32) {
                        const int r = len0 + (idx >> 4), c = idx & 15;
                        *reinterpret_cast<uint4*>(sm + 16384 + (c >> 3) * 8192 + sw128_off(r, c & 7)) = make_uint4(0, 0, 0, 0);
                    }
                    fence_async_smem();
                }
                __syncwarp();
            }
        }
        if (n > 0 && elect_one()) {
            // state-independent product:  forward U^T E (A K-major, B MN-major), backward dO^T Rm (A MN-major, B K-major)
            const uint32_t id_ind = kBwd ? umma_idesc_bf16(128, 128, kMajorMN, kMajorK) : umma_idesc_bf16(128, 128, kMajorK, kMajorMN);
            // state product, negated:  forward -S Pn (B MN-major: rows of Pn are the contraction index),
            //                          backward -S Pn^T (B K-major: rows of Pn are the output index)
            const uint32_t id_st = umma_idesc_bf16(128, 128, kMajorK, kBwd ? kMajorK : kMajorMN, 1);
            auto issue_independent = [&](int c) {
                const uint32_t s0 = smem_u32(sm + slot_xy(c) * kScanItem);
                const uint32_t d = tmem + 128 * (c & 1);
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16) {
                    if (!kBwd)
                        umma_bf16_ss(d, umma_smem_desc_sw128(s0, 16, 1024) + (k16 * 32),
                                     umma_smem_desc_sw128(s0 + 16384, 8192, 1024) + (k16 * 2048), id_ind, k16 > 0);
                    else
                        umma_bf16_ss(d, umma_smem_desc_sw128(s0 + 16384, 8192, 1024) + (k16 * 2048),
                                     umma_smem_desc_sw128(s0, 16, 1024) + (k16 * 32), id_ind, k16 > 0);
                }
                umma_commit(&bar_free[slot_xy(c)]);
            };
            auto ready = [&](int sl, uint32_t parity) {
                if (mbar_wait(&bar_full[sl], parity, p.status, 51)) return true;
                abort_flag = 1;
                return false;
            };
            const bool ok = composite || ready(slot_xy(0), 0u);
            if (ok && !composite) {
                tc_fence_after();
                issue_independent(0);
            }
            for (int c = 0; c < n && ok; ++c) {
                const int st = c & 1;
                const int sl = slot_p(c);
                const uint32_t s0 = smem_u32(sm + sl * kScanItem);
                if (!ready(sl, parity_p(c))) break;
                if (!mbar_wait(&bar_sop, c & 1, p.status, 52)) { abort_flag = 1; break; }
                tc_fence_after();
#pragma unroll
                for (int k16 = 0; k16 < 8; ++k16) {   // A = the packed state in tensor memory, 8 columns per K = 16
                    const UmmaDesc bd = kBwd ? umma_smem_desc_sw128(s0, 16, 1024) + ((k16 >> 2) * 16384 + (k16 & 3) * 32)
                                             : umma_smem_desc_sw128(s0, 16384, 1024) + (k16 * 2048);
                    umma_bf16_ts(tmem + 128 * st, tmem + kScanPanelCol + 8 * k16, bd, id_st, (composite && k16 == 0) ? 0u : 1u);
                }
                umma_commit(&bar_mma);
                umma_commit(&bar_free[sl]);
                if (c + 1 < n && !composite) {
                    // accumulator (c+1) % 2 was last read by the state threads in step c-1, before they packed panel c
                    if (!ready(slot_xy(c + 1), parity_xy(c + 1))) break;
                    tc_fence_after();
                    issue_independent(c + 1);
                }
            }
        }
    } else if (warp == 4 * kScanGroups + 2) {
        // ------------------------------------------------------------------ panel-store thread: the chunk-start states, and the
        // unit's final state as one more panel
        if (elect_one()) {
            for (int c = 0; c < n + 1; ++c) {
                if (!mbar_wait(&bar_pan[c & 1], (c >> 1) & 1, p.status, 55)) { abort_flag = 1; break; }
                const CUtensorMap* m = c == n ? &mF : (composite ? &mS2 : &mS);      // composites go to their own panel array
                const int row = c == n ? unit * 128 : (slot_of(c) * H + h) * 128;
                for (int nb = 0; nb < 2; ++nb) tma_store_2d(m, Sop + (c & 1) * 32768 + nb * 16384, nb * 64, row);
                tma_store_commit();
                tma_store_wait_read();
                mbar_arrive(&bar_out[c & 1]);
            }
            tma_store_wait_all();
        }
    } else {
        // ------------------------------------------------------------------ state warpgroups
        const int col0 = (warp >> 2) * kScanCols;  // first key column of this thread
        float s[kScanCols];
        if (composite) {
#pragma unroll
            for (int j = 0; j < kScanCols; ++j) s[j] = (col0 + j == v) ? 1.f : 0.f;
        } else if (p.s_in && role == 0) {
            const float4* src = reinterpret_cast<const float4*>(p.s_in + (((size_t)seq * H + h) * 128 + v) * 128 + col0);
#pragma unroll
            for (int j = 0; j < kScanCols / 4; ++j) {
                float4 x = src[j];
                s[4 * j] = x.x; s[4 * j + 1] = x.y; s[4 * j + 2] = x.z; s[4 * j + 3] = x.w;
            }
        } else {
#pragma unroll
            for (int j = 0; j < kScanCols; ++j) s[j] = 0.f;
        }
        // This thread's half of the state row as bf16 pairs: first into tensor memory, where the state product reads its
        // A operand (lane = value row, 32 columns per key half), then - after the arrival that releases the UMMA
        // thread - into the shared-memory panel that the TMA store sends to the chunk-parallel kernels.
        static_assert(kScanCols == 64, "the tensor-memory panel is written with one 32-column store per thread");
        const int kh = col0 / 64;
        // Pn and the decays of step c are observed HERE, before the arrival that lets the UMMA thread run step c: the commit of
        // step c frees the slot for a later load, so a state warp that looked at the slot's barrier only
        // after that commit could find it two phases on and read the parity as "not yet complete".
        auto pack_state = [&](int c) -> bool {
            const bool last = c >= n;      // the final state's panel: shared-memory copy only, nothing consumes it on chip
            if (!last && !mbar_wait(&bar_full[slot_p(c)], parity_p(c), p.status, 54)) return false;
            uint32_t w[32];
#pragma unroll
            for (int j = 0; j < 32; ++j) w[j] = pack_bf16(s[2 * j], s[2 * j + 1]);
            if (!last) {
                tmem_st32(tmem + lane_base + kScanPanelCol + 32 * kh, w);
                tmem_st_wait();
                tc_fence_before();
                warp_arrive(&bar_sop, lane);
            }
            if (c > 1 && !mbar_wait(&bar_out[c & 1], ((c - 2) >> 1) & 1, p.status, 57)) return false;      // the panel before the last has left
            uint8_t* dst = Sop + (c & 1) * 32768 + kh * 16384;
#pragma unroll
            for (int q = 0; q < 8; ++q)
                *reinterpret_cast<uint4*>(dst + sw128_off(v, q)) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
            fence_async_smem();
            warp_arrive(&bar_pan[c & 1], lane);
            return true;
        };
        bool ok = true;
        if (!pack_state(0)) { abort_flag = 1; ok = false; }
        for (int c = 0; c < n && ok; ++c) {
            if (!mbar_wait(&bar_mma, c & 1, p.status, 53)) {
                abort_flag = 1; ok = false;
                break;
            }
            tc_fence_after();
            const float* dc = dec_ring[c & 3] + col0;
            {
                uint32_t r[kScanCols / 32][32];    // every part in flight before the wait
#pragma unroll
                for (int b = 0; b < kScanCols / 32; ++b) tmem_ld32(tmem + lane_base + 128 * (c & 1) + col0 + 32 * b, r[b]);
                tmem_ld_wait();
#pragma unroll
                for (int b = 0; b < kScanCols / 32; ++b)
#pragma unroll
                    for (int j4 = 0; j4 < 8; ++j4) {
                        const float4 dv = *reinterpret_cast<const float4*>(dc + 32 * b + 4 * j4);
                        s[32 * b + 4 * j4 + 0] = dv.x * s[32 * b + 4 * j4 + 0] + __uint_as_float(r[b][4 * j4 + 0]);
                        s[32 * b + 4 * j4 + 1] = dv.y * s[32 * b + 4 * j4 + 1] + __uint_as_float(r[b][4 * j4 + 1]);
                        s[32 * b + 4 * j4 + 2] = dv.z * s[32 * b + 4 * j4 + 2] + __uint_as_float(r[b][4 * j4 + 2]);
                        s[32 * b + 4 * j4 + 3] = dv.w * s[32 * b + 4 * j4 + 3] + __uint_as_float(r[b][4 * j4 + 3]);
                    }
            }
            tc_fence_before();
            if (!pack_state(c + 1)) { abort_flag = 1; ok = false; }
        }
        if (ok && abort_flag == 0) {
            // thread-major (float4 j of state thread tid at [j][tid]): every warp store is one contiguous 512-byte run, and the
            // fix-up's threads own the same elements
            float4* dst = reinterpret_cast<float4*>(p.seg_fin + (size_t)unit * 16384) + tid;
#pragma unroll
            for (int j = 0; j < kScanCols / 4; ++j) dst[j * 256] = make_float4(s[4 * j], s[4 * j + 1], s[4 * j + 2], s[4 * j + 3]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------------------------------------
// split scans, second pass: from the units' local states to the true states (see tc_scan_fixup_kernel)
// ---------------------------------------------------------------------------------------------
struct ScanFixArgs {
    simt::ChunkTable tab;
    const float* seg_fin;      // [rec*units][128][128]
    float* s_out;              // final state of the scan, V-first [n_seq][H][128][128], or null
    int H, nseg, bwd, parts;
    int* status;
};

constexpr int kFixP = 65536, kFixL = 131072;        // S hi | S lo, then two P panels, then two local-state panels
constexpr int kFixSmem = 196608 + 1024;

// D[tmem] = (A_hi + A_lo) B: A K-major [128 v][128 k] in two bf16 terms, B = P [k][n] MN-major
__device__ __forceinline__ void issue_hilo_product(uint32_t tmem, const uint8_t* a_hi, const uint8_t* b) {
    const uint32_t b0 = smem_u32(b);
    const uint32_t idesc = umma_idesc_bf16(128, 128, kMajorK, kMajorMN);
#pragma unroll
    for (int part = 0; part < 2; ++part) {
        const uint32_t a0 = smem_u32(a_hi + part * 32768);
#pragma unroll
        for (int k16 = 0; k16 < 8; ++k16)
            umma_bf16_ss(tmem, umma_smem_desc_sw128(a0, 16, 1024) + ((k16 >> 2) * 16384 + (k16 & 3) * 32),
                         umma_smem_desc_sw128(b0, 16384, 1024) + (k16 * 2048), idesc, (part | k16) != 0);
    }
}

// Fix-up of a split scan, one CTA per part of a segment k >= 1 (a run of its chunks).  The true state at the start of
// segment k obeys S_1 = final state of segment 0, S_{j+1} = S_j Pfin_j + Lfin_j (final composite and final local state of
// segment j).  A CTA walks that short chain itself (k - 1 products), then adds S_k Pp_c to the local state the scan
// published for each chunk c of its part; the last part of the last segment applies that segment's final maps as well when
// the caller wants the scan's final state.  S is carried between products as a bf16 hi + lo pair in shared memory (the A
// operand), so the correction keeps float32-class accuracy.
// A thread owns one accumulator row (TMEM lane), so nothing it touches in global memory is addressed row-per-thread:
// the float32 states come thread-major (see the scan kernel), a chunk's bf16 panel comes by TMA into a buffer, is corrected
// there and leaves from it, and the final state is transposed through shared memory.
// Bound by the latency of the chain, then by bytes (96 KB a chunk).  One CTA per SM, so that every input has a second
// buffer: panels for product j + 2 load during j + 1, and the product of chunk c + 1 runs while chunk c is read out.  One
// CTA per chunk, two to an SM, each walking the chain alone and waiting for its panels in turn, took 66 us at 16 recurrences
// of 128 chunks and 17.5 us at 6 of 64.
__global__ void __launch_bounds__(256, 1)
    tc_scan_fixup_kernel(const __grid_constant__ CUtensorMap mPp, const __grid_constant__ CUtensorMap mF,
                         const __grid_constant__ CUtensorMap mHp, ScanFixArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
    __shared__ uint64_t bar_p[2], bar_l[2], bar_mma[2];
    __shared__ uint32_t tmem_slot;
    const int units = 2 * p.nseg - 1, rec = blockIdx.y, seq = rec / p.H, h = rec - seq * p.H;
    const int k = 1 + (int)blockIdx.x / p.parts, part = (int)blockIdx.x % p.parts;
    const int c_begin = p.tab.first_chunk(seq), c_end = p.tab.first_chunk(seq + 1), n_total = c_end - c_begin;
    const int s0 = seg_begin(k, p.nseg, n_total), sn = seg_begin(k + 1, p.nseg, n_total) - s0;
    const int b0 = s0 + (int)((long long)part * sn / p.parts), nc = s0 + (int)((long long)(part + 1) * sn / p.parts) - b0;
    // an empty sequence's final state is its initial state, which the chain reproduces (identity composites, zero local states)
    const bool fin = p.s_out != nullptr && k == p.nseg - 1 && part == p.parts - 1;
    if (nc == 0 && !fin) return;
    // products 0 .. j0-1 walk the chain S_1 -> S_k, j0 .. j0+nc-1 are the chunks' own, the last one the final state's
    const int j0 = k - 1, np = j0 + nc + (fin ? 1 : 0);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int g = warp >> 2;                        // key half handled by this warpgroup
    const int v = (warp & 3) * 32 + lane;           // value row = TMEM lane;  tid == g * 128 + v
    auto chunk_row = [&](int j) {                   // panel row of chunk product j
        const int step = b0 + j - j0;
        return ((p.bwd ? c_end - 1 - step : c_begin + step) * p.H + h) * 128;
    };
    auto is_chunk = [&](int j) { return j >= j0 && j < j0 + nc; };
    // loads, by thread 0: phase j >> 1 of stage j & 1 for the P panels, phase (j - j0) >> 1 for the local states
    int p_end = 0, l_end = j0;                      // loads issued so far (products below these)
    auto load_p = [&]() {
        if (p_end >= np) return;
        const int j = p_end++;
        uint8_t* dst = sm + kFixP + (j & 1) * 32768;
        mbar_expect_tx(&bar_p[j & 1], 32768);
        for (int nb = 0; nb < 2; ++nb)
            tma_load_2d(dst + nb * 16384, is_chunk(j) ? &mPp : &mF, &bar_p[j & 1], nb * 64,
                        is_chunk(j) ? chunk_row(j) : (rec * units + 2 * (j < j0 ? j + 1 : k)) * 128);
    };
    auto load_l = [&]() {
        if (l_end >= j0 + nc) return;
        const int j = l_end++;
        uint8_t* dst = sm + kFixL + (j & 1) * 32768;
        mbar_expect_tx(&bar_l[j & 1], 32768);
        for (int nb = 0; nb < 2; ++nb) tma_load_2d(dst + nb * 16384, &mHp, &bar_l[j & 1], nb * 64, chunk_row(j));
    };
    if (warp == 0 && elect_one()) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&bar_p[s], 1);
            mbar_init(&bar_l[s], 1);
            mbar_init(&bar_mma[s], 1);
        }
        mbar_fence_init();
        load_p(); load_p();
        load_l(); load_l();
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 256);
    auto split_store = [&](const float (&x)[32], int b) {      // 32 keys starting at 64 g + 32 b -> hi / lo operand panels
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            uint32_t hi[4], lo[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const __nv_bfloat162 hh = __floats2bfloat162_rn(x[8 * c + 2 * e], x[8 * c + 2 * e + 1]);
                const float2 back = __bfloat1622float2(hh);
                hi[e] = *reinterpret_cast<const uint32_t*>(&hh);
                lo[e] = pack_bf16(x[8 * c + 2 * e] - back.x, x[8 * c + 2 * e + 1] - back.y);
            }
            *reinterpret_cast<uint4*>(sm + g * 16384 + sw128_off(v, 4 * b + c)) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
            *reinterpret_cast<uint4*>(sm + 32768 + g * 16384 + sw128_off(v, 4 * b + c)) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
        }
    };
    auto load_f32 = [&](const float* unit_base, float (&x)[32], int b) {     // thread-major float32 state of a scan unit
        const float4* src = reinterpret_cast<const float4*>(unit_base) + tid;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const float4 a = src[(8 * b + c) * 256];
            x[4 * c] = a.x; x[4 * c + 1] = a.y; x[4 * c + 2] = a.z; x[4 * c + 3] = a.w;
        }
    };
    {   // S_1 = final state of segment 0
        float x[2][32];
        load_f32(p.seg_fin + (size_t)rec * units * 16384, x[0], 0);
        load_f32(p.seg_fin + (size_t)rec * units * 16384, x[1], 1);
        split_store(x[0], 0);
        split_store(x[1], 1);
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true;
    int issued = 0;
    for (int j = 0; j < np && ok; ++j) {
        const int st = j & 1;
        const bool own = is_chunk(j);
        if (warp == 0 && elect_one()) {
            // this product and, when it leaves S alone, the next: its accumulator was read out an iteration ago
            while (ok && issued < np && (issued <= j || (issued == j + 1 && j >= j0))) {
                ok = mbar_wait(&bar_p[issued & 1], (issued >> 1) & 1, p.status, 80);
                if (ok) {
                    tc_fence_after();
                    issue_hilo_product(tmem + 128 * (issued & 1), sm, sm + kFixP + (issued & 1) * 32768);
                    umma_commit(&bar_mma[issued & 1]);
                    ++issued;
                }
            }
        }
        __syncwarp();
        float add[2][32];                           // what is added to the product
        if (!own) {
            // the final local state of the segment this step crosses (float32, thread-major): flies during the product
            const float* L = p.seg_fin + (size_t)(rec * units + 2 * (j < j0 ? j + 1 : k) - 1) * 16384;
            load_f32(L, add[0], 0);
            load_f32(L, add[1], 1);
        } else {
            ok = mbar_wait(&bar_l[st], ((j - j0) >> 1) & 1, p.status, 82) && ok;
        }
        ok = mbar_wait(&bar_mma[st], (j >> 1) & 1, p.status, 81) && ok;
        tc_fence_after();
        if (warp == 0 && elect_one() && ok) {
            load_p();                               // product j + 2 into the panel this one has read
            if (j > j0) {
                tma_store_wait_read();              // chunk j - 1 has left its buffer: chunk j + 1 into it
                load_l();
            }
        }
        if (own) {
            // the chunk's true state, in place in its buffer
            uint8_t* Lb = sm + kFixL + st * 32768 + g * 16384;
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                uint32_t r[32];
                tmem_ld32(tmem + lane_base + 128 * st + 64 * g + 32 * b, r);
                tmem_ld_wait();
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    uint4* at = reinterpret_cast<uint4*>(Lb + sw128_off(v, 4 * b + c));
                    const uint4 l = *at;
                    const uint32_t lw[4] = {l.x, l.y, l.z, l.w};
                    uint32_t w[4];
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        w[e] = f2_to_bf16(f2_add(f2_make(__uint_as_float(r[8 * c + 2 * e]), __uint_as_float(r[8 * c + 2 * e + 1])), f2_from_bf16(lw[e])));
                    *at = make_uint4(w[0], w[1], w[2], w[3]);
                }
            }
        } else {
            const bool final_state = j >= j0;
            if (final_state) {                      // the rows go through the panel buffers: their stores must have read them
                if (warp == 0 && elect_one()) tma_store_wait_read();
                ok = __syncthreads_and(ok);
            }
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                uint32_t r[32];
                tmem_ld32(tmem + lane_base + 128 * st + 64 * g + 32 * b, r);
                tmem_ld_wait();
                float x[32];
#pragma unroll
                for (int i = 0; i < 32; ++i) x[i] = __uint_as_float(r[i]) + add[b][i];
                if (final_state) {
                    // row-major for the caller (16-byte pieces XOR-swizzled by row so that the stores spread over the
                    // banks), written out below
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        *reinterpret_cast<float4*>(sm + kFixL + v * 512 + (((16 * g + 8 * b + c) ^ (v & 7)) << 4)) =
                            make_float4(x[4 * c], x[4 * c + 1], x[4 * c + 2], x[4 * c + 3]);
                } else {
                    split_store(x, b);              // S_{j+2}: the next product's A operand
                }
            }
        }
        fence_async_smem();
        tc_fence_before();
        ok = __syncthreads_and(ok);                 // operands rewritten, accumulator read
        tc_fence_after();
        if (warp == 0 && elect_one() && ok && own) {
            for (int nb = 0; nb < 2; ++nb) tma_store_2d(&mHp, sm + kFixL + st * 32768 + nb * 16384, nb * 64, chunk_row(j));
            tma_store_commit();
        }
        if (ok && !own && j >= j0) {
            float4* dst = reinterpret_cast<float4*>(p.s_out + (size_t)rec * 16384);
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int f = i * 256 + tid, row = f >> 5, c16 = f & 31;       // float4 f of the row-major 128 x 128 tile
                dst[f] = *reinterpret_cast<const float4*>(sm + kFixL + row * 512 + ((c16 ^ (row & 7)) << 4));
            }
        }
    }
    if (warp == 0 && elect_one()) {
        if (!ok) {      // unwinding: copies and products in flight must end before the block may exit
            for (int j = p_end > 2 ? p_end - 2 : 0; j < p_end; ++j) mbar_wait(&bar_p[j & 1], (j >> 1) & 1, nullptr, 0);
            for (int j = l_end > j0 + 2 ? l_end - 2 : j0; j < l_end; ++j) mbar_wait(&bar_l[j & 1], ((j - j0) >> 1) & 1, nullptr, 0);
            for (int j = issued > 2 ? issued - 2 : 0; j < issued; ++j) mbar_wait(&bar_mma[j & 1], (j >> 1) & 1, nullptr, 0);
        }
        tma_store_wait_read();            // shared memory must outlive the reads of the bulk store
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------------------------
// chunk output (forward), one CTA per chunk-head, from the chunk-start state the scan stored:
//     (W H)^T = H^T W^T,  (R H)^T = H^T R^T           M=128, N=64 each, K=128
//     Z^T = U^T - (W H)^T                             registers -> bf16 panel (kept for the backward) and A operand
//     (A Z)^T = Z^T A^T                               M=128, N=64,  K=64
//     O^T = (R H)^T + (A Z)^T                         transposed through shared memory into o[token][head][value]
// 256 threads: thread (g, v) handles value row v, tokens 32g .. 32g+31.
// ---------------------------------------------------------------------------------------------
struct ChunkOutArgs {
    simt::ChunkTable tab;
    __nv_bfloat16* ZT;
    __nv_bfloat16* o;          // [tokens][H][128]; nullptr with the norm's epilogue when only y is wanted
    int H;
    int* status;
    NormEpilogue norm;
};

// Z^T reuses the W^T tile and the output tile reuses the state tile: the one is dead once the first UMMA chain has
// completed, the other after the last, and the smaller footprint lets two CTAs share an SM.
constexpr int kOutH = 0, kOutWR = 32768, kOutU = 65536, kOutA = 81920, kOutZ = kOutWR, kOutO = kOutH, kOutG = 90112;
constexpr int kChunkOutSmem = kOutA + 8192 + 1024;
constexpr int kChunkOutNormSmem = kOutG + 16384 + 1024;      // + the norm gate's tile when the epilogue is on

__global__ void __launch_bounds__(256, 2)
    tc_chunk_out_kernel(const __grid_constant__ CUtensorMap mH, const __grid_constant__ CUtensorMap mW,
                        const __grid_constant__ CUtensorMap mR, const __grid_constant__ CUtensorMap mUT,
                        const __grid_constant__ CUtensorMap mAT, const __grid_constant__ CUtensorMap mG,
                        const __grid_constant__ CUtensorMap mZT, ChunkOutArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
    uint8_t* Zop = sm + kOutZ;                     // [128 rows x 128 B] K-major A operand
    __nv_bfloat16* Ot = reinterpret_cast<__nv_bfloat16*>(sm + kOutO);   // [64 tokens][128 values]
    __shared__ uint64_t bar_in, bar_mma1, bar_mma2;
    __shared__ uint32_t tmem_slot;
    const int H = p.H, slot = blockIdx.x / H, h = blockIdx.x - slot * H;      // heads fastest, as in the intra-chunk kernels
    int len, tok0;
    p.tab.span(slot, tok0, len);
    if (len == 0) return;
    const int ch = slot * H + h;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int g = warp >> 2;
    const int v = (warp & 3) * 32 + lane;
    if (warp == 0 && elect_one()) {
        mbar_init(&bar_in, 1);
        mbar_init(&bar_mma1, 1);
        mbar_init(&bar_mma2, 1);
        mbar_fence_init();
        mbar_expect_tx(&bar_in, 32768 + 32768 + 16384 + 8192 + (p.norm.gate != nullptr ? 16384 : 0));
        if (p.norm.gate != nullptr)      // the norm gate's tile, needed last: its latency hides under the products
            for (int kb = 0; kb < 2; ++kb) tma_load_2d(sm + kOutG + kb * 8192, &mG, &bar_in, h * 128 + kb * 64, tok0);
        for (int kb = 0; kb < 2; ++kb) tma_load_2d(sm + kOutH + kb * 16384, &mH, &bar_in, kb * 64, ch * 128);
        tma_load_2d(sm + kOutWR, &mW, &bar_in, 0, ch * 128);
        for (int kb = 0; kb < 2; ++kb) tma_load_2d(sm + kOutWR + 16384 + kb * 8192, &mR, &bar_in, kb * 64, ch * 64);
        tma_load_2d(sm + kOutU, &mUT, &bar_in, 0, ch * 128);
        tma_load_2d(sm + kOutA, &mAT, &bar_in, 0, ch * 64);
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 256);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true;
    if (warp == 0 && elect_one()) {
        ok = mbar_wait(&bar_in, 0, p.status, 60);
        if (ok) {
            tc_fence_after();
            const uint32_t a0 = smem_u32(sm + kOutH), b0 = smem_u32(sm + kOutWR);
            const uint32_t idw = umma_idesc_bf16(128, 64, kMajorK, kMajorMN), idr = umma_idesc_bf16(128, 64, kMajorK, kMajorK);
#pragma unroll
            for (int k16 = 0; k16 < 8; ++k16)     // W^T lies key by key ...
                umma_bf16_ss(tmem, umma_smem_desc_sw128(a0, 16, 1024) + ((k16 >> 2) * 16384 + (k16 & 3) * 32),
                             umma_smem_desc_sw128(b0, 8192, 1024) + (k16 * 2048), idw, k16 > 0);
            umma_commit(&bar_mma1);
#pragma unroll
            for (int k16 = 0; k16 < 8; ++k16)     // ... R token by token; needed with the last product only (the commit behind that covers it)
                umma_bf16_ss(tmem + 64, umma_smem_desc_sw128(a0, 16, 1024) + ((k16 >> 2) * 16384 + (k16 & 3) * 32),
                             umma_smem_desc_sw128(b0 + 16384, 16, 1024) + ((k16 >> 2) * 8192 + (k16 & 3) * 32), idr, k16 > 0);
        }
    }
    ok = mbar_wait(&bar_mma1, 0, p.status, 61) && ok;
    // the U^T tile was written by TMA: every reader observes the barrier it completed on
    ok = mbar_wait(&bar_in, 0, p.status, 60) && ok;
    tc_fence_after();
    {   // Z^T for tokens 32g .. 32g+31 of row v
        const uint8_t* UTs = sm + kOutU;
        uint32_t r[32];
        tmem_ld32(tmem + lane_base + 32 * g, r);
        tmem_ld_wait();
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
            const int c16 = g * 4 + q4;
            float u[8];
            unpack_bf16x8(*reinterpret_cast<const uint4*>(UTs + sw128_off(v, c16)), u);
            uint4 z;
            z.x = pack_bf16(u[0] - __uint_as_float(r[8 * q4 + 0]), u[1] - __uint_as_float(r[8 * q4 + 1]));
            z.y = pack_bf16(u[2] - __uint_as_float(r[8 * q4 + 2]), u[3] - __uint_as_float(r[8 * q4 + 3]));
            z.z = pack_bf16(u[4] - __uint_as_float(r[8 * q4 + 4]), u[5] - __uint_as_float(r[8 * q4 + 5]));
            z.w = pack_bf16(u[6] - __uint_as_float(r[8 * q4 + 6]), u[7] - __uint_as_float(r[8 * q4 + 7]));
            *reinterpret_cast<uint4*>(Zop + sw128_off(v, c16)) = z;
        }
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (warp == 0 && elect_one() && ok) {
        if (p.ZT != nullptr) {                      // kept for the backward only: the operand tile is the panel, as TMA lays it out
            tma_store_2d(&mZT, Zop, 0, ch * 128);
            tma_store_commit();
        }
        tc_fence_after();
        const uint32_t a0 = smem_u32(Zop), b0 = smem_u32(sm + kOutA);
        const uint32_t idesc = umma_idesc_bf16(128, 64, kMajorK, kMajorMN);
#pragma unroll
        for (int k16 = 0; k16 < 4; ++k16)
            umma_bf16_ss(tmem + 128, umma_smem_desc_sw128(a0, 16, 1024) + (k16 * 32),
                         umma_smem_desc_sw128(b0, 8192, 1024) + (k16 * 2048), idesc, k16 > 0);
        umma_commit(&bar_mma2);
    }
    if (ok) ok = mbar_wait(&bar_mma2, 0, p.status, 62);
    tc_fence_after();
    if (ok) {
        uint32_t r1[32], r2[32];
        tmem_ld32(tmem + lane_base + 64 + 32 * g, r1);
        tmem_ld32(tmem + lane_base + 128 + 32 * g, r2);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 32; ++j) Ot[(32 * g + j) * 128 + v] = __float2bfloat16(__uint_as_float(r1[j]) + __uint_as_float(r2[j]));
    }
    ok = __syncthreads_and(ok);
    if (ok && p.norm.gate == nullptr) {
        // 64 token rows of 256 bytes: 16 threads per row, 16 rows per pass
        const int c = tid & 15;
#pragma unroll
        for (int pass = 0; pass < 4; ++pass) {
            const int i = pass * 16 + (tid >> 4);
            if (i < len)
                *reinterpret_cast<uint4*>(p.o + ((size_t)(tok0 + i) * H + h) * 128 + 8 * c) =
                    *reinterpret_cast<const uint4*>(Ot + i * 128 + 8 * c);
        }
    } else if (ok) {
        // Gated RMSNorm on the tile: a warp per token row, lane = 4 adjacent values - the decomposition (per-lane sum of
        // four squares, xor-shuffle tree, one rsqrt) of the stand-alone norm kernel, so both give the same bits.
        const float4 ww = *reinterpret_cast<const float4*>(p.norm.weight + 4 * lane);
        const float wa[4] = {ww.x, ww.y, ww.z, ww.w};
#pragma unroll
        for (int pass = 0; pass < 8; ++pass) {
            const int i = pass * 8 + warp;
            const size_t row = (size_t)(tok0 + min(i, len - 1)) * H + h;
            const uint2 ou = *reinterpret_cast<const uint2*>(Ot + i * 128 + 4 * lane);
            const uint2 gu = *reinterpret_cast<const uint2*>(sm + kOutG + (lane >> 4) * 8192 + sw128_off(i, (lane >> 1) & 7) + (lane & 1) * 8);
            const __nv_bfloat162* oh = reinterpret_cast<const __nv_bfloat162*>(&ou);
            const __nv_bfloat162* gh = reinterpret_cast<const __nv_bfloat162*>(&gu);
            const float2 o01 = __bfloat1622float2(oh[0]), o23 = __bfloat1622float2(oh[1]);
            const float2 g01 = __bfloat1622float2(gh[0]), g23 = __bfloat1622float2(gh[1]);
            const float a[4] = {o01.x, o01.y, o23.x, o23.y}, gt[4] = {g01.x, g01.y, g23.x, g23.y};
            float ss = fmaf(a[3], a[3], fmaf(a[2], a[2], fmaf(a[1], a[1], a[0] * a[0])));
#pragma unroll
            for (int off = 8; off > 0; off >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, off);
            ss += __shfl_xor_sync(0xffffffffu, ss, 16);
            if (i < len) {
                const float inv = rsqrtf(ss * (1.0f / 128.0f) + p.norm.eps);
                if (lane == 0 && p.norm.inv_rms != nullptr) p.norm.inv_rms[row] = inv;
                float out[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float th;
                    asm("tanh.approx.f32 %0, %1;" : "=f"(th) : "f"(0.5f * gt[e]));
                    out[e] = a[e] * inv * wa[e] * fmaf(0.5f, th, 0.5f);
                }
                if (p.o != nullptr) *reinterpret_cast<uint2*>(p.o + row * 128 + 4 * lane) = ou;
                *reinterpret_cast<uint2*>(p.norm.y + row * 128 + 4 * lane) =
                    make_uint2(pack_bf16(out[0], out[1]), pack_bf16(out[2], out[3]));
            }
        }
    }
    if (warp == 0 && elect_one()) tma_store_wait_read();            // the Z^T tile must outlive the reads of its bulk store
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------------------------
// dZ (backward), one CTA per chunk-head, from the state adjoint the scan stored:
//     dZ^T = dO^T A + dH'^T E^T          M=128, N=64: K=64 (MN-major A) then K=128
// ---------------------------------------------------------------------------------------------
struct ChunkDzArgs {
    simt::ChunkTable tab;
    int H;
    int* status;
    int* next;                 // zeroed here for the kernel after this one (tc_intra_bwd_kernel)
};

constexpr int kDzH = 0, kDzE = 32768, kDzO = 49152, kDzA = 65536;
constexpr int kChunkDzSmem = kDzA + 8192 + 1024;

__global__ void __launch_bounds__(256, 3)
    tc_chunk_dz_kernel(const __grid_constant__ CUtensorMap mdH, const __grid_constant__ CUtensorMap mE,
                       const __grid_constant__ CUtensorMap mdO, const __grid_constant__ CUtensorMap mAT,
                       const __grid_constant__ CUtensorMap mdZT, ChunkDzArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
    __shared__ uint64_t bar_in, bar_mma;
    __shared__ uint32_t tmem_slot;
    const int H = p.H, slot = blockIdx.x / H, h = blockIdx.x - slot * H;      // heads fastest, as in the intra-chunk kernels
    if (blockIdx.x == 0 && threadIdx.x == 0) *p.next = 0;
    int len, tok0;
    p.tab.span(slot, tok0, len);
    if (len == 0) return;
    const int ch = slot * H + h;
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int g = warp >> 2;
    const int v = (warp & 3) * 32 + lane;
    if (warp == 0 && elect_one()) {
        mbar_init(&bar_in, 1);
        mbar_init(&bar_mma, 1);
        mbar_fence_init();
        mbar_expect_tx(&bar_in, 32768 + 16384 + 16384 + 8192);
        for (int kb = 0; kb < 2; ++kb) {
            tma_load_2d(sm + kDzH + kb * 16384, &mdH, &bar_in, kb * 64, ch * 128);
            tma_load_2d(sm + kDzE + kb * 8192, &mE, &bar_in, kb * 64, ch * 64);
            tma_load_2d(sm + kDzO + kb * 8192, &mdO, &bar_in, h * 128 + kb * 64, tok0);
        }
        tma_load_2d(sm + kDzA, &mAT, &bar_in, 0, ch * 64);
    }
    if (warp == 1) tmem_alloc(&tmem_slot, 64);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    bool ok = true;
    if (len < 64) {
        // ragged tail: the dO rows past it belong to the next sequence; blank them before they feed the UMMA
        ok = mbar_wait(&bar_in, 0, p.status, 70);
        if (ok) {
            for (int idx = tid; idx < (64 - len) * 16; idx += 256) {
                const int r = len + (idx >> 4), c = idx & 15;
                *reinterpret_cast<uint4*>(sm + kDzO + (c >> 3) * 8192 + sw128_off(r, c & 7)) = make_uint4(0, 0, 0, 0);
            }
            fence_async_smem();
        }
        ok = __syncthreads_and(ok);
    }
    if (warp == 0 && elect_one() && ok) {
        ok = mbar_wait(&bar_in, 0, p.status, 70);
        if (ok) {
            tc_fence_after();
            const uint32_t s0 = smem_u32(sm);
            const uint32_t ida = umma_idesc_bf16(128, 64, kMajorMN, kMajorK);
            const uint32_t idb = umma_idesc_bf16(128, 64, kMajorK, kMajorK);
#pragma unroll
            for (int k16 = 0; k16 < 4; ++k16)     // dO^T A
                umma_bf16_ss(tmem, umma_smem_desc_sw128(s0 + kDzO, 8192, 1024) + (k16 * 2048),
                             umma_smem_desc_sw128(s0 + kDzA, 16, 1024) + (k16 * 32), ida, k16 > 0);
#pragma unroll
            for (int k16 = 0; k16 < 8; ++k16)     // + dH'^T E^T
                umma_bf16_ss(tmem, umma_smem_desc_sw128(s0 + kDzH, 16, 1024) + ((k16 >> 2) * 16384 + (k16 & 3) * 32),
                             umma_smem_desc_sw128(s0 + kDzE, 16, 1024) + ((k16 >> 2) * 8192 + (k16 & 3) * 32), idb, 1);
            umma_commit(&bar_mma);
        }
    }
    ok = mbar_wait(&bar_mma, 0, p.status, 71) && ok;
    ok = __syncthreads_and(ok);
    tc_fence_after();
    if (ok) {
        uint32_t r[32];
        tmem_ld32(tmem + lane_base + 32 * g, r);
        tmem_ld_wait();
        // the panel leaves through the dead dH' tile in the swizzled layout and one TMA store: a thread owns a row, and
        // row-per-thread global stores would touch 32 sectors per warp instruction
#pragma unroll
        for (int c = 0; c < 4; ++c)
            *reinterpret_cast<uint4*>(sm + kDzH + sw128_off(v, 4 * g + c)) =
                make_uint4(pack_bf16(__uint_as_float(r[8 * c]), __uint_as_float(r[8 * c + 1])),
                           pack_bf16(__uint_as_float(r[8 * c + 2]), __uint_as_float(r[8 * c + 3])),
                           pack_bf16(__uint_as_float(r[8 * c + 4]), __uint_as_float(r[8 * c + 5])),
                           pack_bf16(__uint_as_float(r[8 * c + 6]), __uint_as_float(r[8 * c + 7])));
    }
    fence_async_smem();
    tc_fence_before();
    ok = __syncthreads_and(ok);
    if (warp == 0 && elect_one() && ok) {
        tma_store_2d(&mdZT, sm + kDzH, 0, ch * 128);
        tma_store_commit();
        tma_store_wait_read();
    }
    if (warp == 1) tmem_dealloc(tmem, 64);
}

}  // namespace tc

// ---------------------------------------------------------------------------------------------
// host entries used by the chunk forward / backward when the tensor-core lane is selected
// ---------------------------------------------------------------------------------------------
// split scans: segment-start states (and the scan's final state), then the chunk states of segments >= 1
static int scan_fixup(const simt::Ws& w, const tc::TcWs& t, int n_seq, __nv_bfloat16* panels, float* s_out, int bwd,
                      const CUtensorMap& mPp, const CUtensorMap& mF, cudaStream_t st) {
    using namespace tc;
    if (set_smem_limit(tc_scan_fixup_kernel, kFixSmem))
        return KDA_ERR_CUDA;
    // one CTA per SM: as many parts to a segment as fill the GPU once, none of them without a chunk
    const int rec = n_seq * w.H, per_seg = (w.nslots / n_seq + t.nseg - 1) / t.nseg;
    const int parts = std::max(1, std::min(148 / (rec * (t.nseg - 1)), per_seg));
    ScanFixArgs f;
    f.tab = w.tab; f.seg_fin = t.seg_fin; f.s_out = s_out; f.H = w.H; f.nseg = t.nseg; f.bwd = bwd; f.parts = parts;
    f.status = t.status;
    CUtensorMap mHp;
    if (make_map_bf16(&mHp, panels, (uint64_t)w.nslots * w.H * 128, 128, 64, 128)) return KDA_ERR_CUDA;
    KDA_LAUNCH("tc_scan_fixup_kernel", st, tc_scan_fixup_kernel<<<dim3(parts * (t.nseg - 1), rec), 256, kFixSmem, st>>>(mPp, mF, mHp, f));
    return launch_status();
}

int tc_scan_forward(const simt::Ws& w, const tc::TcWs& t, int n_seq, int tokens, const float* h0, float* final_state, void* o,
                    const tc::NormEpilogue& norm, cudaStream_t st) {
    using namespace tc;
    const uint64_t nch = (uint64_t)w.nslots * w.H;
    CUtensorMap mW, mR, mE, mAT, mUT, mH, mP, mG, mZT;
    int rc = 0;
    rc |= make_map_bf16(&mW, t.WT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mR, t.R, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mE, t.E, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mAT, t.AT, nch * 64, 64, 64, 64);
    rc |= make_map_bf16(&mUT, t.UT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mH, t.Hp, nch * 128, 128, 64, 128);
    rc |= make_map_bf16(&mP, t.Pn, nch * 128, 128, 64, 128);
    rc |= make_map_bf16(&mZT, t.fwd_only ? t.UT : t.ZT, nch * 128, 64, 64, 128);      // not stored in a forward-only call
    const bool fused_norm = norm.gate != nullptr;
    if (fused_norm) rc |= make_map_bf16_ld(&mG, norm.gate, (uint64_t)tokens, (uint64_t)w.H * 128, (uint64_t)norm.gate_ld, 64, 64);
    else mG = mAT;
    if (rc) return KDA_ERR_CUDA;
    const int out_smem = fused_norm ? kChunkOutNormSmem : kChunkOutSmem;
    if (set_smem_limit(tc_affine_scan_kernel<false>, kAffineScanSmem) ||
        set_smem_limit(tc_chunk_out_kernel, kChunkOutNormSmem))
        return KDA_ERR_CUDA;
    AffineScanArgs a;
    a.tab = w.tab; a.decay_end = t.decay_end; a.s_in = h0;
    a.H = w.H; a.status = t.status; a.nseg = t.nseg; a.seg_fin = t.seg_fin;
    const int units = 2 * t.nseg - 1;
    const dim3 scan_grid(n_seq * units, w.H);
    CUtensorMap mPp, mF;
    if (make_map_bf16(&mPp, t.Pp, nch * 128, 128, 64, 128) ||
        make_map_bf16(&mF, t.fin_panel, (uint64_t)n_seq * w.H * units * 128, 128, 64, 128))
        return KDA_ERR_CUDA;
    KDA_LAUNCH("tc_affine_scan_fwd_kernel", st,
               tc_affine_scan_kernel<false><<<scan_grid, kAffineScanThreads, kAffineScanSmem, st>>>(mP, mUT, mE, mH, mPp, mF, a));
    if (int e = launch_status()) return e;
    if (int e = scan_fixup(w, t, n_seq, t.Hp, final_state, 0, mPp, mF, st)) return e;
    ChunkOutArgs oa;
    oa.tab = w.tab; oa.ZT = t.fwd_only ? nullptr : t.ZT; oa.o = static_cast<__nv_bfloat16*>(o); oa.H = w.H;
    oa.status = t.status;
    oa.norm = norm;
    KDA_LAUNCH("tc_chunk_out_kernel", st,
               tc_chunk_out_kernel<<<(unsigned)nch, 256, out_smem, st>>>(mH, mW, mR, mUT, mAT, mG, mZT, oa));
    return launch_status();
}

int tc_scan_backward(const simt::Ws& w, const simt::Scr& s, const tc::TcWs& t, int n_seq, int tokens, const void* d_o,
                     const float* d_final, float* dh0, cudaStream_t st) {
    using namespace tc;
    const uint64_t nch = (uint64_t)w.nslots * w.H;
    CUtensorMap mE, mAT, mdO, mdH, mP, mRm, mdZT;
    int rc = 0;
    rc |= make_map_bf16(&mE, t.E, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mAT, t.AT, nch * 64, 64, 64, 64);
    rc |= make_map_bf16(&mdO, d_o, (uint64_t)tokens, (uint64_t)w.H * 128, 64, 64);
    rc |= make_map_bf16(&mdH, t.dHp, nch * 128, 128, 64, 128);
    rc |= make_map_bf16(&mP, t.Pn, nch * 128, 128, 64, 128);
    rc |= make_map_bf16(&mRm, t.RmT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mdZT, t.dZT, nch * 128, 64, 64, 128);
    if (rc) return KDA_ERR_CUDA;
    if (set_smem_limit(tc_affine_scan_kernel<true>, kAffineScanSmem) ||
        set_smem_limit(tc_chunk_dz_kernel, kChunkDzSmem))
        return KDA_ERR_CUDA;
    AffineScanArgs a;
    a.tab = w.tab; a.decay_end = t.decay_end; a.s_in = d_final;
    a.H = w.H; a.status = t.status; a.nseg = t.nseg; a.seg_fin = t.seg_fin;
    const int units = 2 * t.nseg - 1;
    const dim3 scan_grid(n_seq * units, w.H);
    CUtensorMap mPp, mF;
    if (make_map_bf16(&mPp, t.Pp, nch * 128, 128, 64, 128) ||
        make_map_bf16(&mF, t.fin_panel, (uint64_t)n_seq * w.H * units * 128, 128, 64, 128))
        return KDA_ERR_CUDA;
    KDA_LAUNCH("tc_affine_scan_bwd_kernel", st,
               tc_affine_scan_kernel<true><<<scan_grid, kAffineScanThreads, kAffineScanSmem, st>>>(mP, mRm, mdO, mdH, mPp, mF, a));
    if (int e = launch_status()) return e;
    if (int e = scan_fixup(w, t, n_seq, t.dHp, dh0, 1, mPp, mF, st)) return e;
    ChunkDzArgs da;
    da.tab = w.tab; da.H = w.H; da.status = t.status; da.next = s.next;
    KDA_LAUNCH("tc_chunk_dz_kernel", st,
               tc_chunk_dz_kernel<<<(unsigned)nch, 256, kChunkDzSmem, st>>>(mdH, mE, mdO, mAT, mdZT, da));
    return launch_status();
}

}  // namespace kda
