// Tensor-core lane (K = V = 128): a recurrence and everything it feeds, in one walk over its chunks.
//
// Forward, from the intra-chunk panels of a chunk and its incoming state H:
//     Z = U - W H        O = R H + A Z        H' = e^{G_end} . H + E^T U - E^T (W H)
// Backward, with the adjoint H' of the chunk's outgoing state, last chunk first:
//     dZ = A^T dO + E H'        adjoint of H = e^{G_end} . H' + R^T dO - W^T dZ
// What the backward reads of the forward (H, Z) and the intra-chunk backward of this one (H', dZ) leaves on the way.  Split scans
// (kda_tc_pscan.cu) fold W^T E and R - A W into maps of their own first: half the chain of a step, for more traffic.
// Restates reference chunk_wy_forward.cu:940-1275, 1498-1588 and chunk_wy_backward.cu:2445-2562.

#include "common.cuh"
#include "simt_ws.cuh"
#include "tc_common.cuh"
#include "tc_ws.cuh"

namespace kda {
namespace tc {

int make_map_bf16_ld(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint64_t ld, uint32_t box_cols, uint32_t box_rows);
int make_map_bf16(CUtensorMap* m, const void* ptr, uint64_t rows, uint64_t cols, uint32_t box_cols, uint32_t box_rows);

namespace {

// 16 lanes x 8 N columns of an accumulator with M = 64: r[4n + 2a + e] is row l/4 + 8a, column 8n + 2(l%4) + e
__device__ __forceinline__ void tmem_ld_16x32(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x4.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t* w) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t* w) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                 : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void stsm4(uint32_t addr, const uint32_t* w) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}
__device__ __forceinline__ void stsm4_t(uint32_t addr, const uint32_t* w) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(w[0]), "r"(w[1]), "r"(w[2]), "r"(w[3]) : "memory");
}
// A barrier of four output warps: they go on together or not at all.
__device__ __forceinline__ bool output_sync(int id, bool ok) {
    uint32_t all;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.u32 p, %1, 0;\n\t"
        "barrier.cta.red.and.pred q, %2, 128, p;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(all)
        : "r"((uint32_t)ok), "r"(id)
        : "memory");
    return all != 0;
}
// the same shared address in the other block of the pair
__device__ __forceinline__ uint32_t peer_addr(const void* p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, int* status, int code) {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        uint32_t ok;
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(ok)
            : "r"(smem_u32(bar)), "r"(parity)
            : "memory");
        if (ok) return true;
    }
    raise_status(status, code);
    return false;
}

}  // namespace

struct WalkArgs {
    simt::ChunkTable tab;
    const float* decay_end;   // [nch][128] exp(G_end)
    const float* s_in;        // V-first initial state (forward: h0, backward: cotangent of the final state), or null
    float* s_out;             // V-first final state of the walk (forward: final state, backward: dh0), or null
    __nv_bfloat16* o;         // forward: [tokens][H][128]; nullptr with the norm's epilogue when only y is wanted
    int o_map;                // o starts on 16 bytes and is stored through its map; with the norm it may start on 8
    int H;
    int keep;                 // 1: the states and Z go to their panels (a backward follows, or this is one)
    int* status;
    int* next;                // backward: zeroed here for the kernel after this one (tc_intra_bwd_kernel)
    NormEpilogue norm;
};

// Shared memory (bytes).  A stage holds a chunk's operands: W^T [128 k][64 t], R and E [64 t][128 k] (two blocks of 64 k), A^T [64 s][64 i]
// and this block's half of U^T [64 v][64 t] (backward: of dO [64 t][64 v]).
constexpr int kWkW = 0, kWkR = 16384, kWkE = 32768, kWkA = 49152, kWkU = 57344, kWkStage = 65536;
constexpr int kWkH = 2 * kWkStage;             // 2 x 16 KB  state [128 k][64 v] of step c in c % 2: an operand, and the panel that leaves
constexpr int kWkZ = kWkH + 32768;             // 2 x  8 KB  Z (dZ) [64 t][64 v], the same
constexpr int kWkO = kWkZ + 16384;             // 2 x  8 KB  output [64 t][64 v] on its way out
constexpr int kWkG = kWkO + 16384;             // 3 x  8 KB  the norm's gate of chunk c in c % 3, then its output on its way out
constexpr int kWkDec = kWkG + 24576;           // [4][128] floats: exp(G_end) of step c in slot c % 4
constexpr int kWkSs = kWkDec + 2048;           // [4][64] floats: the other block's sums of squares of chunk c in c % 4
constexpr int kWkNw = kWkSs + 1024;            // [64] floats: the norm's weight
constexpr int kWkBars = kWkNw + 256;
constexpr int kWalkSmem = kWkBars + 512 + 1024;
constexpr int kWkState = 8;                    // state warps
constexpr int kWkCols = 256 / kWkState;        // state columns a thread
constexpr int kWkFwdThreads = (kWkState + 12) * 32, kWkBwdThreads = (kWkState + 3) * 32;

// One block per (sequence, head) and half of the value columns: the state's columns do not meet in any product.  State and Z lie as
// [key or token][value], so a product reads them as its B operand from the tile that is also the panel on its way out.  Threads are
// specialised by warp and meet only through mbarriers:
//   state warps (8)     own the state in registers (thread: key row, 32 columns), form Z and the next state
//   next warp           one lane issues the TMA loads, as far ahead as the two stages allow
//   next warp           one lane issues the products: W H (backward: E H'), R H beside it; E^T (W H) (W^T dZ), A Z beside it
//   next warp           one lane stores the panels
//   next warp           forward with the norm: one lane loads the gate's tiles
//   output warps (2x4)  forward: read every other chunk's output out, normalise it if asked, store it
// The terms of the next step without the state, E^T U (backward: A^T dO and R^T dO), are issued behind this step's last product.
// Why not E^T Z in one product: U is in bf16 already, and Z = U - W H would be rounded a second time on its way into the sum that the state
// is.  The final state was then 1.08 to 1.20 times as far from float64 as that of split scans, which have E^T U and H Pn apart as well; now
// 1.00.  W H takes U's place in the stage, piece by piece where a warp has read U.  The price is a product and 8 KB more a step: 1.17 -> 1.32 us
// with 32 recurrences of 128 chunks, 381 -> 398 us below.  The lane that issues products is busy all step long (about 50 cycles a product, more
// a wait), so what E^T U needs comes as one group: with E and A a group of their own 1.39, R and A as well 1.5; E^T Z and E^T times what
// rounding took from Z 1.45; E^T U between W H and R H 1.43.
// The norm needs whole rows: the two blocks of a recurrence are a cluster then and swap their sums of squares, warp by warp.
// Many recurrences: bound by the bytes of the panels, 136 KB a chunk-head forward and 120 backward (16,544 chunk-heads in 352
// recurrences: 398 and 337 us, 0.87 and 0.91 of the copy rate; scan and output kernel took 258 + 305 us, scan and dZ kernel 254 + 219, and the
// intra-chunk forward, which formed the scans' maps, 915 instead of 801).  Few: a step of about 2,400 cycles forward and 1,840 backward,
// of which the products' operands, the loads and the stores keep shared memory busy for 2,050 and 1,800 (a product reads A and B at 128 bytes a
// cycle, no faster than it multiplies them); what a step waits for besides is the way from a product's end to the next one's start, twice.
// Whatever can be there early is therefore looked for while a product runs, a lane that issues products commits three times a step, and
// two sets of output warps have two steps each.  Sixteen state warps of 16 columns were no faster (2,010 backward); four output warps
// that swap sums with a release of their own stores took 4,600 cycles a step, with the gate's tile loaded a step ahead 3,600.
template <bool kBwd>
__global__ void __launch_bounds__(kBwd ? kWkBwdThreads : kWkFwdThreads, 1)
    tc_walk_kernel(const __grid_constant__ CUtensorMap mW, const __grid_constant__ CUtensorMap mR, const __grid_constant__ CUtensorMap mE,
                   const __grid_constant__ CUtensorMap mA, const __grid_constant__ CUtensorMap mU, const __grid_constant__ CUtensorMap mS,
                   const __grid_constant__ CUtensorMap mZ, const __grid_constant__ CUtensorMap mO, const __grid_constant__ CUtensorMap mY,
                   const __grid_constant__ CUtensorMap mG, WalkArgs p) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);   // pointer arithmetic keeps the shared address space
    float (*dec_ring)[128] = reinterpret_cast<float (*)[128]>(sm + kWkDec);
    // full / free: operand groups 0, 1, 2 of a stage (which tile is in which group differs by direction, see the load warp).
    // h, z: the state's and Z's tiles are written; hout, zout: their stores have read them.  m1, m2: the step's two products that the state
    // warps wait for.  o: the output accumulator is complete, of: it has been read.  g, gf: the gate's tile; ss: the other block's sums.
    // Whatever has two buffers has two barriers, so that no waiter can be two phases late.
    uint64_t* bar = reinterpret_cast<uint64_t*>(sm + kWkBars);
    auto bar_full = [&](int g, int s) { return bar + 2 * g + s; };
    uint64_t *bar_m1 = bar + 6, *bar_m2 = bar + 8, *bar_o = bar + 10, *bar_h = bar + 12, *bar_z = bar + 14, *bar_hout = bar + 16, *bar_zout = bar + 18,
             *bar_of = bar + 22, *bar_g = bar + 24, *bar_gf = bar + 27, *bar_ss = bar + 30;      // ss: [4][4 warps]
    // by when a group's tiles have been read: forward all of them with the output's product, backward the first two with the step's
    // first product and the third with its second
    auto bar_free = [&](int g, int s) { return kBwd ? (g < 2 ? bar_m1 : bar_m2) + s : bar_o + s; };
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bar + 46);
    volatile int& abort_flag = *reinterpret_cast<volatile int*>(bar + 47);

    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int half = blockIdx.x & 1, rec = blockIdx.x >> 1, H = p.H, rank = rec / H, h = rec - rank * H;
    const int seq = p.tab.per_seq > 0 ? rank : p.tab.seq_order[rank];       // a packed batch longest first: the first blocks to start are the longest chains
    const int c_begin = p.tab.first_chunk(seq), c_end = p.tab.first_chunk(seq + 1), n = c_end - c_begin;
    const bool norm = !kBwd && p.norm.gate != nullptr;
    auto slot_of = [&](int c) { return kBwd ? c_end - 1 - c : c_begin + c; };   // chunk slot of step c

    if (kBwd && blockIdx.x == 0 && tid == 0) *p.next = 0;
    if (warp == 0 && elect_one()) {
        for (int i = 0; i < 12; ++i) mbar_init(bar + i, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&bar_h[i], kWkState);
            mbar_init(&bar_z[i], kWkState);
            mbar_init(&bar_hout[i], 1);
            mbar_init(&bar_zout[i], 1);
            mbar_init(&bar_of[i], 4);
        }
        for (int i = 0; i < 6; ++i) mbar_init(&bar_g[i], 1);
        for (int i = 0; i < 16; ++i) mbar_init(&bar_ss[i], 1);
        mbar_fence_init();
        abort_flag = 0;
    }
    constexpr uint32_t kTmemCols = kBwd ? 256 : 512;      // 192, 320 in use
    if (warp == 1) tmem_alloc(&tmem_slot, kTmemCols);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (norm) {      // the other block's barriers are there before the first sums go over
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
    const uint32_t tmem = tmem_slot;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    constexpr uint32_t c1 = 0, c2 = 64, c3 = 192;      // accumulators: W H (M = 64); next state (two); forward: output (M = 64, two)
    auto ph = [](int c) { return (uint32_t)(c >> 1) & 1u; };      // parity of step c's phase of a barrier with two buffers
    auto ph3 = [](int c) { return (uint32_t)(c / 3) & 1u; };      // ... with three

    if (warp == kWkState) {
        // ------------------------------------------------------------------ load warp
        if (elect_one()) {
            // groups by when they are wanted: forward U E, decays (2) | W R A (0); backward A dO R | E | W, decays
            auto load = [&](int c, int g) {
                const int cs = slot_of(c), ch = cs * H + h, s = c & 1;
                uint8_t* b = sm + s * kWkStage;
                uint64_t* f = bar_full(g, s);
                auto ld_w = [&]() { tma_load_2d(b + kWkW, &mW, f, 0, ch * 128); };
                auto ld_r = [&]() { for (int nb = 0; nb < 2; ++nb) tma_load_2d(b + kWkR + nb * 8192, &mR, f, nb * 64, ch * 64); };
                auto ld_e = [&]() { for (int nb = 0; nb < 2; ++nb) tma_load_2d(b + kWkE + nb * 8192, &mE, f, nb * 64, ch * 64); };
                auto ld_a = [&]() { tma_load_2d(b + kWkA, &mA, f, 0, ch * 64); };
                if (kBwd && g == 0) {
                    mbar_expect_tx(f, 32768);
                    int tok0, len;
                    p.tab.span(cs, tok0, len);
                    tma_load_2d(b + kWkU, &mU, f, h * 128 + half * 64, tok0);
                    ld_a();
                    ld_r();
                } else if (kBwd && g == 1) {
                    mbar_expect_tx(f, 16384);
                    ld_e();
                } else if (g == 0) {
                    mbar_expect_tx(f, 40960);
                    ld_w();
                    ld_r();
                    ld_a();
                } else {
                    mbar_expect_tx(f, (kBwd ? 16384 : 24576) + 512);
                    bulk_load_1d(dec_ring[c & 3], p.decay_end + (size_t)ch * 128, 512, f);
                    if (kBwd) {
                        ld_w();
                    } else {
                        tma_load_2d(b + kWkU, &mU, f, 0, ch * 128 + half * 64);
                        ld_e();
                    }
                }
            };
            bool ok = true;
            int c = 0;
            for (; c < n && ok; ++c) {
#pragma unroll
                for (int i = 0; i < (kBwd ? 3 : 2); ++i) {
                    const int g = kBwd ? i : 2 - 2 * i;      // in the order in which they are wanted
                    if (ok && c > 1 && (i == 0 || (kBwd && i == 2))) ok = mbar_wait(bar_free(g, c & 1), ph(c - 2), p.status, 100);
                    if (ok) load(c, g);
                }
            }
            if (ok) {      // the products behind the last commits are over before the block may exit
                for (c = n > 2 ? n - 2 : 0; c < n && ok; ++c)
                    ok = mbar_wait(bar_free(2, c & 1), ph(c), p.status, 101);
            } else {       // unwinding: the copies in flight must land first
                abort_flag = 1;
                for (int cc = c > 2 ? c - 3 : 0; cc < c; ++cc)
                    for (int g = 0; g < 3; g += kBwd ? 1 : 2) mbar_poll(bar_full(g, cc & 1), ph(cc), kSpinLimit / 8);
            }
        }
    } else if (warp == kWkState + 1) {
        // ------------------------------------------------------------------ UMMA thread
        if (kBwd && n > 0) {
            // Only a sequence's last chunk (the first step) can be ragged; the dO rows past its tail belong to the next sequence and
            // are blanked by the whole warp before its lane issues the products on them.
            int tok0, len0;
            p.tab.span(slot_of(0), tok0, len0);
            if (len0 < 64) {
                if (mbar_wait(bar_full(0, 0), 0, p.status, 102)) {
                    for (int idx = lane; idx < (64 - len0) * 8; idx += 32)
                        *reinterpret_cast<uint4*>(sm + kWkU + sw128_off(len0 + (idx >> 3), idx & 7)) = make_uint4(0, 0, 0, 0);
                    fence_async_smem();
                }
                __syncwarp();
            }
        }
        if (n > 0 && elect_one()) {
            // In a cluster the shared addresses of the second block carry its rank above bit 24, which a descriptor's address field
            // would pass on to the stride beside it.
            const uint32_t s0 = smem_u32(sm) & 0x3ffffu;
            constexpr uint32_t id64_mn_mn = umma_idesc_bf16(64, 64, kMajorMN, kMajorMN), id64_k_mn = umma_idesc_bf16(64, 64, kMajorK, kMajorMN);
            constexpr uint32_t id128_mn_mn = umma_idesc_bf16(128, 64, kMajorMN, kMajorMN), id128n_k_mn = umma_idesc_bf16(128, 64, kMajorK, kMajorMN, 1);
            constexpr uint32_t id128_mn_k = umma_idesc_bf16(128, 64, kMajorMN, kMajorK), id128n_mn_k = umma_idesc_bf16(128, 64, kMajorMN, kMajorK, 1);
            // a tile [rows][64] whose rows are the contraction index; with several blocks of 64 columns these are `blk` bytes apart
            auto mn = [](uint32_t a) { return umma_smem_desc_sw128(a, 8192, 1024); };
            auto km = [](uint32_t a) { return umma_smem_desc_sw128(a, 16, 1024); };
            auto early = [&](int c) {      // the terms of step c without the state
                const uint32_t st = s0 + (c & 1) * kWkStage;
                if (!kBwd) {
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16)     // E^T U
                        umma_bf16_ss(tmem + c2 + 64 * (c & 1), mn(st + kWkE) + (k16 * 2048), km(st + kWkU) + (k16 * 32), id128_mn_k, k16 > 0);
                    return;
                }
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16)     // A^T dO
                    umma_bf16_ss(tmem + c1, km(st + kWkA) + (k16 * 32), mn(st + kWkU) + (k16 * 2048), id64_k_mn, k16 > 0);
#pragma unroll
                for (int k16 = 0; k16 < 4; ++k16)     // R^T dO
                    umma_bf16_ss(tmem + c2 + 64 * (c & 1), mn(st + kWkR) + (k16 * 2048), mn(st + kWkU) + (k16 * 2048), id128_mn_mn, k16 > 0);
            };
            bool ok = true;
            auto wait = [&](uint64_t* b, uint32_t parity, int code) {
                ok = ok && mbar_wait(b, parity, p.status, code);
                return ok;
            };
            auto early_full = [&](int c) { return kBwd ? wait(bar_full(0, c & 1), ph(c), 103) : wait(bar_full(2, c & 1), ph(c), 103); };
            if (early_full(0)) {
                tc_fence_after();
                early(0);
            }
            for (int c = 0; c < n && ok; ++c) {
                const int s = c & 1;
                const uint32_t st = s0 + s * kWkStage, hs = s0 + kWkH + s * 16384, zs = s0 + kWkZ + s * 8192;
                if (!wait(bar_full(kBwd ? 1 : 0, s), ph(c), 104) || !wait(&bar_h[s], ph(c), 105)) break;
                tc_fence_after();
                if (!kBwd) {
#pragma unroll
                    for (int k16 = 0; k16 < 8; ++k16)     // W H
                        umma_bf16_ss(tmem + c1, mn(st + kWkW) + (k16 * 2048), mn(hs) + (k16 * 2048), id64_mn_mn, k16 > 0);
                    umma_commit(&bar_m1[s]);
                    // the output, while the state warps are at the next state
                    if (c > 1 && !wait(&bar_of[s], ph(c - 2), 106)) break;
                    tc_fence_after();
#pragma unroll
                    for (int k16 = 0; k16 < 8; ++k16)     // R H
                        umma_bf16_ss(tmem + c3 + 64 * s, km(st + kWkR) + ((k16 >> 2) * 8192 + (k16 & 3) * 32), mn(hs) + (k16 * 2048), id64_k_mn, k16 > 0);
                    if (!wait(&bar_z[s], ph(c), 107)) break;
                    tc_fence_after();
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16)     // - E^T (W H), which lies where U did
                        umma_bf16_ss(tmem + c2 + 64 * s, mn(st + kWkE) + (k16 * 2048), km(st + kWkU) + (k16 * 32), id128n_mn_k, 1);
                    umma_commit(&bar_m2[s]);
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16)     // + A Z
                        umma_bf16_ss(tmem + c3 + 64 * s, mn(st + kWkA) + (k16 * 2048), mn(zs) + (k16 * 2048), id64_mn_mn, 1);
                    umma_commit(&bar_o[s]);
                } else {
#pragma unroll
                    for (int k16 = 0; k16 < 8; ++k16)     // + E H'
                        umma_bf16_ss(tmem + c1, km(st + kWkE) + ((k16 >> 2) * 8192 + (k16 & 3) * 32), mn(hs) + (k16 * 2048), id64_k_mn, 1);
                    umma_commit(&bar_m1[s]);
                    if (!wait(bar_full(2, s), ph(c), 104) || !wait(&bar_z[s], ph(c), 107)) break;
                    tc_fence_after();
#pragma unroll
                    for (int k16 = 0; k16 < 4; ++k16)     // - W^T dZ
                        umma_bf16_ss(tmem + c2 + 64 * s, km(st + kWkW) + (k16 * 32), mn(zs) + (k16 * 2048), id128n_k_mn, 1);
                    umma_commit(&bar_m2[s]);
                }
                if (c + 1 < n) {      // the other state accumulator was read a step ago (backward: and dZ's has been)
                    if (!early_full(c + 1)) break;
                    tc_fence_after();
                    early(c + 1);
                }
            }
            if (!ok) abort_flag = 1;
        }
    } else if (warp == kWkState + 2) {
        // ------------------------------------------------------------------ panel-store thread
        if (p.keep && elect_one()) {
            bool ok = true;
            for (int c = 0; c < n && ok; ++c) {
                const int s = c & 1, ch = slot_of(c) * H + h;
                ok = mbar_wait(&bar_h[s], ph(c), p.status, 108);
                if (!ok) break;
                tma_store_2d(&mS, sm + kWkH + s * 16384, half * 64, ch * 128);
                tma_store_commit();
                tma_store_wait_read();
                mbar_arrive(&bar_hout[s]);
                ok = mbar_wait(&bar_z[s], ph(c), p.status, 109);
                if (!ok) break;
                tma_store_2d(&mZ, sm + kWkZ + s * 8192, half * 64, ch * 64);
                tma_store_commit();
                tma_store_wait_read();
                mbar_arrive(&bar_zout[s]);
            }
            if (!ok) abort_flag = 1;
            tma_store_wait_all();
        }
    } else if (warp == kWkState + 3) {
        // ------------------------------------------------------------------ the norm's gate
        if (norm && elect_one()) {
            auto token = [&](int c) {
                int tok0, len;
                p.tab.span(slot_of(c), tok0, len);
                return tok0;
            };
            int c = 0;
            for (; c < n; ++c) {
                if (c > 2 && !mbar_wait(&bar_gf[c % 3], ph3(c - 3), p.status, 110)) {
                    abort_flag = 1;
                    break;
                }
                mbar_expect_tx(&bar_g[c % 3], 8192);
                tma_load_2d(sm + kWkG + (c % 3) * 8192, &mG, &bar_g[c % 3], h * 128 + half * 64, token(c));
                if (c + 3 < n) tma_prefetch_2d(&mG, h * 128 + half * 64, token(c + 3));
            }
            for (int i = c > 3 ? c - 3 : 0; i < c; ++i) mbar_poll(&bar_g[i % 3], ph3(i), kSpinLimit / 8);
        }
    } else if (warp >= kWkState + 4) {
        // ------------------------------------------------------------------ output warps: tokens 16q .. 16q + 15 of every other chunk
        const int q = warp & 3, set = (warp - kWkState - 4) >> 2, c4 = lane & 3, r8 = lane >> 2, mi = lane >> 3, mr = lane & 7;
        const uint32_t s0 = smem_u32(sm), otile = s0 + kWkO + set * 8192;
        const bool lead = q == 0;                  // this warp's lane stores for the set
        // address this lane gives to ldmatrix / stmatrix for the two 8-column pieces 2m, 2m + 1 of its warp's 16 rows
        auto piece = [&](int m) { return sw128_off(16 * q + 8 * (mi & 1) + mr, 2 * m + (mi >> 1)); };
        float* wn = reinterpret_cast<float*>(sm + kWkNw);
        if (norm && set == 0 && q < 2) wn[32 * q + lane] = p.norm.weight[64 * half + 32 * q + lane];      // read behind the first output_sync
        if (norm) asm volatile("bar.sync 3, 256;" ::: "memory");
        bool ok = true;
        int c = set;
        for (; c < n; c += 2) {
            int tok0, len;
            p.tab.span(slot_of(c), tok0, len);
            ok = mbar_wait(&bar_o[set], ph(c), p.status, 111);
            __syncwarp();
            tc_fence_after();
            uint32_t ow[16];       // pieces as bf16 pairs: [2i + a] columns 8i + 2c4 + {0, 1}, row r8 + 8a
            {
                uint32_t r[2][16];
                tmem_ld_16x32(tmem + lane_base + c3 + 64 * set, r[0]);
                tmem_ld_16x32(tmem + lane_base + c3 + 64 * set + 32, r[1]);
                tmem_ld_wait();
                tc_fence_before();
                warp_arrive(&bar_of[set], lane);
#pragma unroll
                for (int i = 0; i < 16; ++i) ow[i] = pack_bf16(__uint_as_float(r[i >> 3][2 * (i & 7)]), __uint_as_float(r[i >> 3][2 * (i & 7) + 1]));
            }
            // The tile of the set's last output has left: the lane that stored it waits for that before it comes here.
            ok = output_sync(1 + set, ok);
            if (!ok) break;
            if (p.o != nullptr) {
#pragma unroll
                for (int m = 0; m < 4; ++m) stsm4(otile + piece(m), ow + 4 * m);
            }
            if (norm) {
                // in the order of the stand-alone kernel's sums (four adjacent values, then the pieces of a half row by halving,
                // then the two halves), so that both give the same bits
                float sum[2];
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    float q4[8];
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float2 x = f2_get(f2_from_bf16(ow[2 * i + a]));
                        const float before = __shfl_xor_sync(0xffffffffu, fmaf(x.y, x.y, x.x * x.x), 1);
                        q4[i] = fmaf(x.y, x.y, fmaf(x.x, x.x, before));      // whole in the odd lanes
                    }
                    const float t = ((q4[0] + q4[4]) + (q4[2] + q4[6])) + ((q4[1] + q4[5]) + (q4[3] + q4[7]));
                    sum[a] = t + __shfl_xor_sync(0xffffffffu, t, 2);
                    sum[a] = __shfl_sync(0xffffffffu, sum[a], lane | 1);
                }
                // To the other block, counted by its barrier: a release of the stores before it would wait for all of them.  It sends chunk
                // c + 4's only once it has this set's of c + 2, which leave here after c's have been read.
                const float* ss = reinterpret_cast<const float*>(sm + kWkSs) + 64 * (c & 3) + 16 * q;
                uint64_t* bss = &bar_ss[4 * (c & 3) + q];
                if (lane == 0) mbar_expect_tx(bss, 64);
                if (c4 < 2)
                    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b32 [%0], %1, [%2];" ::"r"(peer_addr(ss + r8 + 8 * c4, half ^ 1)),
                                 "r"(__float_as_uint(c4 == 0 ? sum[0] : sum[1])), "r"(peer_addr(bss, half ^ 1))
                                 : "memory");
                const uint32_t gt_tile = s0 + kWkG + c % 3 * 8192;
                ok = mbar_wait(&bar_g[c % 3], ph3(c), p.status, 112);
                uint32_t yw[16];
#pragma unroll
                for (int m = 0; m < 4; ++m) ldsm4(gt_tile + piece(m), yw + 4 * m);
                float sg[32];      // its sigmoids, while the other block's sums are on their way
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const float2 gt = f2_get(f2_from_bf16(yw[i]));
                    asm("tanh.approx.f32 %0, %1;" : "=f"(sg[2 * i]) : "f"(0.5f * gt.x));
                    asm("tanh.approx.f32 %0, %1;" : "=f"(sg[2 * i + 1]) : "f"(0.5f * gt.y));
                }
                ok = ok && mbar_wait_cluster(bss, (uint32_t)(c >> 2) & 1u, p.status, 113);
                __syncwarp();
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const float inv = rsqrtf((sum[a] + ss[r8 + 8 * a]) * (1.0f / 128.0f) + p.norm.eps);
                    const int row = 16 * q + r8 + 8 * a;
                    if (half == 0 && c4 == 0 && row < len && p.norm.inv_rms != nullptr) p.norm.inv_rms[(size_t)(tok0 + row) * H + h] = inv;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const float2 x = f2_get(f2_from_bf16(ow[2 * i + a])), w2 = *reinterpret_cast<const float2*>(wn + 8 * i + 2 * c4);
                        yw[2 * i + a] = pack_bf16(x.x * inv * w2.x * fmaf(0.5f, sg[4 * i + 2 * a], 0.5f), x.y * inv * w2.y * fmaf(0.5f, sg[4 * i + 2 * a + 1], 0.5f));
                    }
                }
                // over the gate's tile: this warp alone has read these rows of it
#pragma unroll
                for (int m = 0; m < 4; ++m) stsm4(gt_tile + piece(m), yw + 4 * m);
            }
            fence_async_smem();
            ok = output_sync(1 + set, ok);
            if (!ok) break;
            // The sequence's last chunk goes out row by row: those past a ragged tail are another sequence's.
            const bool whole = len == 64, o_rows = p.o != nullptr && !(whole && p.o_map);
            if (whole && lead && elect_one()) {
                if (p.o != nullptr && p.o_map) tma_store_2d(&mO, sm + kWkO + set * 8192, h * 128 + half * 64, tok0);
                if (norm) tma_store_2d(&mY, sm + kWkG + c % 3 * 8192, h * 128 + half * 64, tok0);
                tma_store_commit();
                tma_store_wait_read();
                if (norm) mbar_arrive(&bar_gf[c % 3]);
            }
            __syncwarp();
            if (!whole || o_rows) {
                for (int i = (tid & 127) >> 3; i < len; i += 16) {
                    const size_t at = ((size_t)(tok0 + i) * H + h) * 128 + half * 64 + 8 * (tid & 7);
                    const uint32_t off = sw128_off(i, tid & 7);
                    if (o_rows) {
                        const uint2* x = reinterpret_cast<const uint2*>(sm + kWkO + set * 8192 + off);
                        reinterpret_cast<uint2*>(p.o + at)[0] = x[0];
                        reinterpret_cast<uint2*>(p.o + at)[1] = x[1];
                    }
                    if (norm && !whole) *reinterpret_cast<uint4*>(p.norm.y + at) = *reinterpret_cast<const uint4*>(sm + kWkG + c % 3 * 8192 + off);
                }
            }
        }
        if (!ok) abort_flag = 1;
        if (lead && elect_one()) tma_store_wait_all();
    } else {
        // ------------------------------------------------------------------ state warps
        const int hf = warp >> 2, q = warp & 3, mi = lane >> 3, mr = lane & 7;
        const int k = 32 * q + lane;               // key row = accumulator lane
        const uint32_t s0 = smem_u32(sm);
        const size_t sbase = ((size_t)seq * H + h) * 16384 + (size_t)(64 * half + kWkCols * hf) * 128 + k;      // V-first: neighbouring lanes, neighbouring keys
        f2 s[kWkCols / 2];
#pragma unroll
        for (int j = 0; j < kWkCols / 2; ++j)
            s[j] = p.s_in != nullptr ? f2_make(p.s_in[sbase + (size_t)(2 * j) * 128], p.s_in[sbase + (size_t)(2 * j + 1) * 128]) : f2_all(0.f);
        auto put_state = [&](int c) {              // the state that step c starts from; its tile is free
            uint8_t* dst = sm + kWkH + (c & 1) * 16384;
#pragma unroll
            for (int j = 0; j < kWkCols / 8; ++j)
                *reinterpret_cast<uint4*>(dst + sw128_off(k, kWkCols / 8 * hf + j)) =
                    make_uint4(f2_to_bf16(s[4 * j]), f2_to_bf16(s[4 * j + 1]), f2_to_bf16(s[4 * j + 2]), f2_to_bf16(s[4 * j + 3]));
            fence_async_smem();
            tc_fence_before();
            warp_arrive(&bar_h[c & 1], lane);
        };
        bool ok = true;
        if (n > 0) put_state(0);
        for (int c = 0; c < n && ok; ++c) {
            const int st = c & 1;
            // What is long there is looked for while the product runs: U and the decays (before the arrival that lets the step go on to
            // free their slots), and that the stores have read the tiles written next.  The products that read those are complete: these
            // warps have waited for later ones.
            ok = mbar_wait(bar_full(2, st), ph(c), p.status, 115);
            constexpr int kPieces = kWkCols / 8;   // 8-column pieces a warp: [2i + a] columns kWkCols hf + 8i + 2(l%4) + {0, 1}, tokens 16q + l/4 + 8a
            uint32_t zw[2 * kPieces];
            // U^T lies value by value: this lane's address of pieces 2m, 2m + 1 of what its warp owns
            auto u_at = [&](int m) { return s0 + st * kWkStage + kWkU + sw128_off(kWkCols * hf + 8 * (2 * m + (mi >> 1)) + mr, 2 * q + (mi & 1)); };
            if (!kBwd && ok) {
#pragma unroll
                for (int m = 0; m < kPieces / 2; ++m) ldsm4_t(u_at(m), zw + 4 * m);
            }
            const f2 dec = f2_all(dec_ring[c & 3][k]);
            if (p.keep && c > 1) ok = ok && mbar_wait(&bar_zout[st], ph(c - 2), p.status, 117);
            ok = ok && mbar_wait(&bar_m1[st], ph(c), p.status, 116);
            if (!ok) break;
            tc_fence_after();
            uint32_t wh[2 * kPieces];
            {
                uint32_t r[4 * kPieces];
                tmem_ld_16x32(tmem + lane_base + c1 + kWkCols * hf, r);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 2 * kPieces; ++i) {
                    const f2 x = f2_make(__uint_as_float(r[2 * i]), __uint_as_float(r[2 * i + 1]));
                    if (!kBwd) wh[i] = f2_to_bf16(x);
                    zw[i] = f2_to_bf16(kBwd ? x : f2_fma(x, f2_all(-1.f), f2_from_bf16(zw[i])));
                }
            }
#pragma unroll
            for (int m = 0; m < kPieces / 2; ++m) {
                stsm4(s0 + kWkZ + st * 8192 + sw128_off(16 * q + 8 * (mi & 1) + mr, kPieces * hf + 2 * m + (mi >> 1)), zw + 4 * m);
                if (!kBwd) stsm4_t(u_at(m), wh + 4 * m);      // over U: its product came before W H, and this warp alone has read these pieces
            }
            fence_async_smem();
            tc_fence_before();
            warp_arrive(&bar_z[st], lane);
            if (p.keep && c > 0 && c + 1 < n) ok = mbar_wait(&bar_hout[st ^ 1], ph(c - 1), p.status, 114);
            ok = ok && mbar_wait(&bar_m2[st], ph(c), p.status, 118);
            if (!ok) break;
            tc_fence_after();
            {
                uint32_t r[kWkCols];
                tmem_ld32(tmem + lane_base + c2 + 64 * st + kWkCols * hf, r);
                tmem_ld_wait();
#pragma unroll
                for (int j = 0; j < kWkCols / 2; ++j) s[j] = f2_fma(dec, s[j], f2_make(__uint_as_float(r[2 * j]), __uint_as_float(r[2 * j + 1])));
            }
            if (c + 1 < n) put_state(c + 1);
        }
        if (!ok) abort_flag = 1;
        if (ok && abort_flag == 0 && p.s_out != nullptr) {
#pragma unroll
            for (int j = 0; j < kWkCols / 2; ++j) {
                const float2 x = f2_get(s[j]);
                p.s_out[sbase + (size_t)(2 * j) * 128] = x.x;
                p.s_out[sbase + (size_t)(2 * j + 1) * 128] = x.y;
            }
        }
    }
    __syncwarp();
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, kTmemCols);
    if (norm) {      // the other block may still be writing its sums into this one
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
    }
}

template <bool kBwd>
static int launch_walk(unsigned grid, bool pair, const CUtensorMap& mW, const CUtensorMap& mR, const CUtensorMap& mE, const CUtensorMap& mA,
                       const CUtensorMap& mU, const CUtensorMap& mS, const CUtensorMap& mZ, const CUtensorMap& mO, const CUtensorMap& mY,
                       const CUtensorMap& mG, const WalkArgs& a, cudaStream_t st) {
    if (set_smem_limit(tc_walk_kernel<kBwd>, kWalkSmem)) return KDA_ERR_CUDA;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kBwd ? kWkBwdThreads : kWkFwdThreads);
    cfg.dynamicSmemBytes = kWalkSmem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 2;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = pair ? 1 : 0;
    cudaError_t e = cudaSuccess;
    KDA_LAUNCH(kBwd ? "tc_walk_bwd_kernel" : "tc_walk_fwd_kernel", st,
               e = cudaLaunchKernelEx(&cfg, tc_walk_kernel<kBwd>, mW, mR, mE, mA, mU, mS, mZ, mO, mY, mG, a));
    return e == cudaSuccess ? launch_status() : KDA_ERR_CUDA;
}

}  // namespace tc

int tc_walk_forward(const simt::Ws& w, const tc::TcWs& t, int n_seq, int tokens, const float* h0, float* final_state, void* o,
                    const tc::NormEpilogue& norm, cudaStream_t st) {
    using namespace tc;
    const uint64_t nch = (uint64_t)w.nslots * w.H, cols = (uint64_t)w.H * 128;
    CUtensorMap mW, mR, mE, mA, mU, mS, mZ, mO, mY, mG;
    int rc = make_map_bf16(&mW, t.WT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mR, t.R, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mE, t.E, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mA, t.AT, nch * 64, 64, 64, 64);
    rc |= make_map_bf16(&mU, t.UT, nch * 128, 64, 64, 64);
    mS = mZ = mO = mY = mG = mA;      // not used where a call has none
    if (!t.fwd_only) {
        rc |= make_map_bf16(&mS, t.Hp, nch * 128, 128, 64, 128);
        rc |= make_map_bf16(&mZ, t.ZT, nch * 64, 128, 64, 64);
    }
    const bool o_map = o != nullptr && reinterpret_cast<uintptr_t>(o) % 16 == 0;
    if (o_map) rc |= make_map_bf16(&mO, o, (uint64_t)tokens, cols, 64, 64);
    if (norm.gate != nullptr) {
        rc |= make_map_bf16(&mY, norm.y, (uint64_t)tokens, cols, 64, 64);
        rc |= make_map_bf16_ld(&mG, norm.gate, (uint64_t)tokens, cols, (uint64_t)norm.gate_ld, 64, 64);
    }
    if (rc) return KDA_ERR_CUDA;
    WalkArgs a;
    a.tab = w.tab; a.decay_end = t.decay_end; a.s_in = h0; a.s_out = final_state; a.o = static_cast<__nv_bfloat16*>(o); a.o_map = o_map; a.H = w.H; a.next = nullptr;
    a.keep = !t.fwd_only; a.status = t.status; a.norm = norm;
    return launch_walk<false>(2u * (unsigned)n_seq * (unsigned)w.H, norm.gate != nullptr, mW, mR, mE, mA, mU, mS, mZ, mO, mY, mG, a, st);
}

int tc_walk_backward(const simt::Ws& w, const simt::Scr& s, const tc::TcWs& t, int n_seq, int tokens, const void* d_o,
                     const float* d_final, float* dh0, cudaStream_t st) {
    using namespace tc;
    const uint64_t nch = (uint64_t)w.nslots * w.H;
    CUtensorMap mW, mR, mE, mA, mU, mS, mZ;
    int rc = make_map_bf16(&mW, t.WT, nch * 128, 64, 64, 128);
    rc |= make_map_bf16(&mR, t.R, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mE, t.E, nch * 64, 128, 64, 64);
    rc |= make_map_bf16(&mA, t.AT, nch * 64, 64, 64, 64);
    rc |= make_map_bf16(&mU, d_o, (uint64_t)tokens, (uint64_t)w.H * 128, 64, 64);
    rc |= make_map_bf16(&mS, t.dHp, nch * 128, 128, 64, 128);
    rc |= make_map_bf16(&mZ, t.dZT, nch * 64, 128, 64, 64);
    if (rc) return KDA_ERR_CUDA;
    WalkArgs a = {};
    a.tab = w.tab; a.decay_end = t.decay_end; a.s_in = d_final; a.s_out = dh0; a.H = w.H; a.keep = 1; a.status = t.status; a.next = s.next;
    return launch_walk<true>(2u * (unsigned)n_seq * (unsigned)w.H, false, mW, mR, mE, mA, mU, mS, mZ, mZ, mZ, mZ, a, st);
}

}  // namespace kda
