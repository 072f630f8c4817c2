// Warp-specialised FlashAttention forward for sm_100a: fp16 Q/K/V, fp32 accumulate in tensor memory, fp32 or fp16 O.
// Stands in for flash_attn_tc_kernel (flash_attn_tc.cu:73-312 of eager-flash-attention) behind the same launch
// interface: same tensor layouts, split-KV partial format (row max in the log2 domain) and completion counters.
//
// Two kernels: this one (fa_fwd_ws_kernel) for d_h = 128, where the tensor pipe and the exponentials are about even (and for d_h = 64 in the persistent
// form), and that of four chains (fa_fwd_chains_kernel, fa_fwd_chains.cuh) for d_h 16, 32 and 64. Few rows (KSPLIT) use this one with the differences
// stated there.
//
// One CTA = 256 query rows (two 128-row Q tiles) of one (head, split), 384 threads:
//   warps 0-3   softmax of Q tile 0        (one thread per row; registers raised with setmaxnreg)
//   warps 4-7   softmax of Q tile 1
//   warp  8     TMA producer: Q tiles once, then K and V 128-key stages through two rings
//   warp  9     tcgen05.mma issuer (one elected lane); owns the tensor-memory allocation
//   warp  10    the second issuer where there is one, else idle; warp 11 idle (they give their registers to the softmax)
// Both Q tiles share each K/V stage, which halves the L2 -> shared-memory traffic per FLOP. Each tile is a
// chain  S(j) -> softmax -> P(j) -> P(j)*V(j) -> Q*K^T(j+1) -> S(j+1)  (P overwrites S in tensor memory, and the
// tensor pipe executes in issue order), and the two chains run half a period apart: the one issuing thread
// serves them in turn,
//     ... PV0(j) QK0(j+1) | PV1(j) QK1(j+1) | PV0(j+1) QK0(j+2) | ...
// so that while one tile's softmax runs on the SIMT pipes (and has the special-function unit to itself) the
// tensor pipe executes the other tile's MMAs. A period is one softmax plus one tile's MMAs; timestamps taken
// inside the kernel (d_h = 128) put it at about 1770 + 1890 cycles against 2048 cycles of pure MMA time for
// both tiles. Two things were tried against that and measured slower: an issuing thread per tile (the tiles fall
// into step, both softmaxes then share the special-function unit and both MMA groups the tensor pipe), and
// 64-key stages with two S buffers per tile so that Q*K^T runs a stage ahead (a 128x64x16 MMA takes 48 cycles,
// not 32, and the issuing thread needs about as long per MMA as the tensor pipe). What did pay: descriptors kept
// in registers as (low, high) words, so that an MMA costs the issuing thread two additions and the instruction
// (it shares its scheduler with two softmax warps); a V ring one slot deeper than the K ring (V(j) is wanted
// right at the start of stage j, K(j+1) a whole stage after its slot is freed); packed fp32 pairs in the softmax.
// Slower were: Q*K^T in two 64-key halves, the upper one issued as soon as its columns of S are in
// registers, with its exponentials under the offset in use while the maximum is still being found: the halves'
// MMAs fetch Q twice (d_h = 128, S = 32768, four heads, causal: 1.27 ms against 1.02).
// Tensor memory (512 columns): S0/P0 [0,128) S1/P1 [128,256) O0 [256,256+D) O1 [384,384+D).
// O is rescaled in tensor memory by the softmax warps themselves, and at d_h 64 and 128 only when a row maximum grew
// by more than 2^8 since the value last used as the exponent offset (P then stays below 256, well
// inside fp16); the final division by the row sum makes the result independent of the offset.
// P reaches the MMA warp in two 64-key halves, each on its own mbarrier, so the first four k-steps of
// P*V start while the exponentials of the second half are still being computed.
//
// Work items (256 rows of one head/split) are taken either one per CTA from the grid, or, in the
// persistent form, by fewer CTAs than SMs from a global counter; the barriers are rebuilt per item.
// The order of the items is strict row order, or bands of rows taken head by head when the caller
// allows rows to complete band by band (see fetch_item).
//
// All waits are bounded; a warp leaves its loop as a whole when a wait fails, every other role then
// runs into its own bounded wait or sees the CTA's abort word, and the CTA frees its tensor memory.
#include "fa_fwd_sm100.cuh"
#include "fa_args.cuh"
#include "host_util.h"
#include "sm100_ptx.cuh"

#include <algorithm>
#include <cmath>

namespace efa {

namespace {

constexpr int WS_BM = 128;          // rows per Q tile
constexpr int WS_BN = 128;          // keys per stage
constexpr int WS_THREADS = 384;
constexpr float kNegInfW = -INFINITY;

template <int D, bool KSPLIT>
struct WsCfg {
    static_assert(D == 128 || (D == 64 && !KSPLIT), "smaller heads take the kernel of four chains");
    static constexpr int SWB        = 128;                        // swizzle width = TMA box row, bytes
    static constexpr int BOXC       = SWB / 2;
    static constexpr int NBOX       = D / BOXC;
    static constexpr int BOX_BYTES  = 128 * SWB;
    static constexpr int TILE_BYTES = 128 * D * 2;
    static constexpr int NSTAGE_K   = D == 128 ? 2 : 4;           // K(j+1) is wanted a whole stage after its slot is freed,
    static constexpr int NSTAGE_V   = D == 128 && !KSPLIT ? 3 : 4; // V(j) right at the start of the stage: the deeper ring
    static constexpr int QTILES     = KSPLIT ? 1 : 2;
    static constexpr int SMEM_BYTES = TILE_BYTES * (QTILES + NSTAGE_K + NSTAGE_V) + 1024;
    static constexpr int TMEM_COLS  = 512;
    // A wait by parity only holds for a thread that waits for every phase of a slot in turn: one that skips a phase
    // finds the parity it wants while the slot is still a phase behind. With KSPLIT an issuer takes every second stage, so
    // each slot has to belong to one issuer.
    static constexpr int STAGE_STEP = KSPLIT ? 2 : 1;
    static_assert(NSTAGE_K % STAGE_STEP == 0 && NSTAGE_V % STAGE_STEP == 0, "an issuer would skip phases of a slot");
    static_assert(!KSPLIT || 3 * WS_BM * (int)sizeof(float) <= TILE_BYTES, "the merge's exchange fits a K slot");
};

__device__ __forceinline__ float max3(float a, float b, float c)
{
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Two fp32 lanes per instruction (fma.rn.f32x2 / add.rn.f32x2: same rounding as the scalar forms): scale-and-offset
// and the row sum of the softmax take half the instructions. Measured: 3 % of the attention launch.
__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}

// Two exponentials 2^x on the FMA and integer pipes: x = n + f with n the nearest integer, 2^f as a polynomial of degree 5: the
// minimax fit of the relative error on [-1/2, 1/2] with the constant term 1 (a linear program over Chebyshev nodes, its coefficients
// rounded to fp32). Off by at most 1.8e-7 with the fp32 roundings below; ex2.approx is specified to 2^-22 = 2.4e-7. Below -127 the result
// is 0, NaN stays NaN.
__device__ __forceinline__ uint64_t exp2_poly2(uint64_t x)
{
    float x0, x1;
    unpack2(x, x0, x1);
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(x0) : "f"(-127.f));
    asm("max.NaN.f32 %0, %0, %1;" : "+f"(x1) : "f"(-127.f));
    x = pack2(x0, x1);
    const uint64_t t = add2(x, pack2(12582912.f, 12582912.f));           // 1.5 * 2^23: n in the low bits
    const uint64_t n = add2(t, pack2(-12582912.f, -12582912.f));
    const uint64_t f = fma2(n, pack2(-1.f, -1.f), x);
    uint64_t p = pack2(0x1.5bba14p-10f, 0x1.5bba14p-10f);
    p = fma2(p, f, pack2(0x1.3cea88p-7f, 0x1.3cea88p-7f));
    p = fma2(p, f, pack2(0x1.c6b752p-5f, 0x1.c6b752p-5f));
    p = fma2(p, f, pack2(0x1.ebf9bcp-3f, 0x1.ebf9bcp-3f));
    p = fma2(p, f, pack2(0x1.62e42ap-1f, 0x1.62e42ap-1f));
    p = fma2(p, f, pack2(1.f, 1.f));
    float t0, t1;
    unpack2(t, t0, t1);
    return mul2(p, pack2(__uint_as_float((__float_as_uint(t0) << 23) + 0x3f800000u), __uint_as_float((__float_as_uint(t1) << 23) + 0x3f800000u)));
}

__device__ __forceinline__ void setmaxnreg_dec_56() { asm volatile("setmaxnreg.dec.sync.aligned.u32 56;"); }
__device__ __forceinline__ void setmaxnreg_inc_224() { asm volatile("setmaxnreg.inc.sync.aligned.u32 224;"); }
__device__ __forceinline__ void setmaxnreg_dec_40() { asm volatile("setmaxnreg.dec.sync.aligned.u32 40;"); }
__device__ __forceinline__ void setmaxnreg_dec_24() { asm volatile("setmaxnreg.dec.sync.aligned.u32 24;"); }
__device__ __forceinline__ void setmaxnreg_inc_104() { asm volatile("setmaxnreg.inc.sync.aligned.u32 104;"); }

#include "fa_fwd_chains.cuh"

// PERSIST = false: one work item (256 rows of one head/split) per CTA, grid (H_local*split, row blocks).
// PERSIST = true: a 1-D grid of fewer CTAs than SMs; each CTA takes work items from a global counter in
// the same row-major order. The SMs left without a CTA stay free for the projection and the AllReduce
// of finished tiles, which otherwise can only start when an attention CTA retires.
// KSPLIT: a work item is 128 rows, and both softmax warpgroups take its one Q tile, warpgroup q the key stages
// q, q + 2, ...: an item is half as long for half as many rows, which fills the GPU where 256-row items do not. The
// two running results are merged at the end, straight from tensor memory (both warpgroups see the same lanes).
template <int D, bool OUT_F16, bool PERSIST, bool KSPLIT>
__global__ void __launch_bounds__(WS_THREADS, 1)
fa_fwd_ws_kernel(const __grid_constant__ CUtensorMap tmQ,
                 const __grid_constant__ CUtensorMap tmK,
                 const __grid_constant__ CUtensorMap tmV,
                 const FaArgs a, int* work_counter, int items_x, int items_total)
{
    using C = WsCfg<D, KSPLIT>;
    constexpr uint32_t SWZ = swizzle_code(C::SWB);
    constexpr uint32_t IDESC_QK = idesc_f16_f32(WS_BM, WS_BN, 0, 0);
    constexpr uint32_t IDESC_PV = idesc_f16_f32(WS_BM, D, 0, 1);
    constexpr int NSK = C::NSTAGE_K, NSV = C::NSTAGE_V;
    constexpr int ISSUERS = KSPLIT ? 2 : 1;             // issuing threads: one per warpgroup where the tiles need not alternate
    // Every fourth pair of exponentials as a polynomial at d_h 128, where one tile's chain is what an item waits for and the special-function
    // unit has time to spare: S = 32768, four heads, causal 1008 -> 1000 us; 2048 rows, eight heads 25.3 -> 24.5; ten heads x 8192 rows
    // 310 -> 302; a third of the pairs is worse (+3 %).
    constexpr bool POLY = D == 128;
    constexpr int ITEM_ROWS = KSPLIT ? WS_BM : 2 * WS_BM;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sQ = smem;                                   // QTILES tiles
    uint8_t* sK = sQ + C::QTILES * C::TILE_BYTES;         // NSK stages
    uint8_t* sV = sK + NSK * C::TILE_BYTES;               // NSV stages

    __shared__ __align__(8) uint64_t q_full[2];
    __shared__ __align__(8) uint64_t k_full[NSK], k_empty[NSK], v_full[NSV], v_empty[NSV];
    __shared__ __align__(8) uint64_t s_full[2], p_full[2][2], o_done[2];
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_word;
    __shared__ int half_done[2][2];                       // [tile][64-row half]: warps that finished their stores
    __shared__ int s_item, s_head, s_split, s_row0;       // the work item

    const int tid  = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);       // known to be one value for the warp
    const int lane = tid & 31;

    // ---- once per CTA
    if (tid == 0) {
        abort_word = 0;
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
    }
    if (warp == 9) tmem_alloc(&tmem_base_smem, C::TMEM_COLS);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_smem, 0);
    const bool behind = KSPLIT && a.tail_first >= 0;     // the rest of the launch before this one: no need to wait for that
    if (!behind) pdl_wait();
    pdl_trigger();
    const int kv_len = a.kv_len;

    struct ItemInfo { int head, split, block_row0, kv_lo, kv_hi, nblk_max; int q_abs0[2], rows_q[2], nblk[2]; };
    // Next work item. Thread 0 rebuilds the barriers for every item (all threads are past the previous one), thread 32 finds the
    // item for everybody (the divisions and what they leave in registers were worth 2 % of a launch at d_h 128).
    // Both role branches below call this the same number of times, so its __syncthreads pair up.
    auto fetch_item = [&](int round, ItemInfo& it) -> bool {
        if (tid == 0) {
            half_done[0][0] = half_done[0][1] = half_done[1][0] = half_done[1][1] = 0;
            if (round > 0) {
                for (int q = 0; q < 2; q++) { mbar_inval(&q_full[q]); mbar_inval(&s_full[q]); mbar_inval(&p_full[q][0]); mbar_inval(&p_full[q][1]); mbar_inval(&o_done[q]); }
                for (int s = 0; s < NSK; s++) { mbar_inval(&k_full[s]); mbar_inval(&k_empty[s]); }
                for (int s = 0; s < NSV; s++) { mbar_inval(&v_full[s]); mbar_inval(&v_empty[s]); }
            }
            for (int q = 0; q < 2; q++) {
                mbar_init(&q_full[q], 1);
                mbar_init(&s_full[q], 1);
                mbar_init(&p_full[q][0], WS_BM / 32);
                mbar_init(&p_full[q][1], WS_BM / 32);
                mbar_init(&o_done[q], 1);
            }
            for (int s = 0; s < NSK; s++) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], 1); }
            for (int s = 0; s < NSV; s++) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], 1); }
            mbar_fence_init();
        }
        if (tid == 32) {
            const int item = PERSIST ? atomicAdd(work_counter, 1) : (int)(blockIdx.y * gridDim.x + blockIdx.x);
            s_item = item;
            if (item < items_total) {
                const bool tail = KSPLIT && a.tail_first >= 0;
                int head, split, row0;
                pick_item(item, a, items_x, items_total, ITEM_ROWS, tail, head, split, row0);
                s_head = head;
                s_split = split;
                s_row0 = row0;
            }
        }
        __syncthreads();
        if (__shfl_sync(0xffffffffu, s_item, 0) >= items_total || abort_word != 0) return false;
        it.head  = __shfl_sync(0xffffffffu, s_head, 0);
        it.split = __shfl_sync(0xffffffffu, s_split, 0);
        it.block_row0 = __shfl_sync(0xffffffffu, s_row0, 0);
        const int rows_valid = min(ITEM_ROWS, a.q_rows - it.block_row0);      // 64, 128, 192 or 256 (in a tail also none)
        it.kv_lo = it.split * kv_len;
        it.kv_hi = it.kv_lo + kv_len;

        // Per Q tile: first absolute row, valid rows, number of key stages.
        #pragma unroll
        for (int q = 0; q < 2; q++) {
            const int tile0 = KSPLIT ? 0 : q * WS_BM;
            it.q_abs0[q] = a.q_start + it.block_row0 + tile0;
            it.rows_q[q] = max(0, min(WS_BM, rows_valid - tile0));
            const int kv_end = a.causal ? min(it.kv_hi, it.q_abs0[q] + it.rows_q[q]) : it.kv_hi;
            it.nblk[q] = (it.rows_q[q] > 0 && kv_end > it.kv_lo) ? (kv_end - it.kv_lo + WS_BN - 1) / WS_BN : 0;
        }
        it.nblk_max = max(it.nblk[0], it.nblk[1]);
        return true;
    };
    auto end_item = [&]() {
        __syncwarp();
        tc_fence_before_sync();
        __syncthreads();
        tc_fence_after_sync();
    };
#define EFA_ITEM_LOCALS \
    const int head = it.head, split = it.split, block_row0 = it.block_row0, kv_lo = it.kv_lo, kv_hi = it.kv_hi, nblk_max = it.nblk_max; \
    const int* q_abs0 = it.q_abs0; const int* rows_q = it.rows_q; const int* nblk = it.nblk; \
    (void)head; (void)split; (void)block_row0; (void)kv_lo; (void)kv_hi; (void)nblk_max; (void)q_abs0; (void)rows_q; (void)nblk;

    if (warp >= 8) {
        setmaxnreg_dec_56();
        for (int round = 0; ; round++) {
            ItemInfo it;
            if (!fetch_item(round, it)) break;
            EFA_ITEM_LOCALS
            // =====================================================================================
            // Producer / MMA warpgroup
            // =====================================================================================
            if (warp == 8 && lane == 0) {
                // ---- TMA producer
                auto load_tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int row) {
                    mbar_expect_tx(bar, C::TILE_BYTES);
                    #pragma unroll
                    for (int b = 0; b < C::NBOX; b++)
                        tma_load_3d(dst + b * C::BOX_BYTES, tm, bar, b * C::BOXC, row, head);
                };
                for (int q = 0; q < C::QTILES; q++)
                    if (nblk[q] > 0) load_tile(sQ + q * C::TILE_BYTES, &tmQ, &q_full[q], q_abs0[q]);
                for (int j = 0; j < nblk_max; j++) {
                    const int sk = j % NSK, uk = j / NSK, sv = j % NSV, uv = j / NSV;
                    if (uk > 0 && !mbar_wait(&k_empty[sk], (uint32_t)((uk - 1) & 1), &abort_word, 21)) break;
                    load_tile(sK + sk * C::TILE_BYTES, &tmK, &k_full[sk], kv_lo + j * WS_BN);
                    if (uv > 0 && !mbar_wait(&v_empty[sv], (uint32_t)((uv - 1) & 1), &abort_word, 22)) break;
                    load_tile(sV + sv * C::TILE_BYTES, &tmV, &v_full[sv], kv_lo + j * WS_BN);
                }
            } else if (warp >= 9 && warp < 9 + ISSUERS) {
                // ---- MMA issuer. The whole warp runs the loop, so that the descriptors are values of the warp (uniform registers,
                // which is where the instruction wants them), and one elected lane issues: always the same, since a commit
                // covers what the thread that executes it has issued. Descriptors as (low, high) words; a k-step or a ring
                // slot only moves the address field of the low word.
                // A commit costs this warp 200 to 300 cycles (time stamps: 630 of a period of 3284 at d_h 128 and of 2968 at d_h 64 went
                // into two of them, while a P was waiting), so there is one per tile and stage (s_full): S = 32768, four heads of 128,
                // causal, 1035 -> 1002 us. Ring slots are given back by the softmax warps that see it: S(j) complete means
                // that all that was issued before is, QK(j) and PV(j-1) of both tiles among it.
                const uint64_t dq0 = smem_desc(smem_u32(sQ), 16, 8 * C::SWB, SWZ);
                const uint64_t dk0 = smem_desc(smem_u32(sK), 16, 8 * C::SWB, SWZ);
                const uint64_t dv0 = smem_desc(smem_u32(sV), C::BOX_BYTES, 8 * C::SWB, SWZ);
                const uint32_t dq_lo = (uint32_t)dq0, dq_hi = (uint32_t)(dq0 >> 32);
                const uint32_t dk_lo = (uint32_t)dk0, dk_hi = (uint32_t)(dk0 >> 32);
                const uint32_t dv_lo = (uint32_t)dv0, dv_hi = (uint32_t)(dv0 >> 32);
                auto wait = [&](uint64_t* bar, int phase, int site) -> bool {
                    const bool done = __all_sync(0xffffffffu, mbar_wait(bar, (uint32_t)(phase & 1), &abort_word, site));
                    tc_fence_after_sync();
                    return done;
                };
                auto issue_qk = [&](int q, int slot) {
                    const uint32_t qa = dq_lo + (KSPLIT ? 0u : (uint32_t)q * (C::TILE_BYTES >> 4));
                    const uint32_t ka = dk_lo + (uint32_t)slot * (C::TILE_BYTES >> 4);
                    const uint32_t tS = tmem_base + q * 128;
                    if (elect_one()) {
                        #pragma unroll
                        for (int ks = 0; ks < D / 16; ks++) {
                            const uint32_t off = ((uint32_t)((ks * 16) / C::BOXC) * C::BOX_BYTES + (uint32_t)((ks * 16) % C::BOXC) * 2u) >> 4;
                            tc_mma_ss_lh(tS, qa + off, dq_hi, ka + off, dk_hi, IDESC_QK, ks > 0 ? 1u : 0u);
                        }
                        tc_commit(&s_full[q]);
                    }
                };
                auto issue_pv = [&](int q, int slot, uint32_t acc0, int half, bool last) {
                    const uint32_t va = dv_lo + (uint32_t)slot * (C::TILE_BYTES >> 4);
                    const uint32_t tP = tmem_base + q * 128, tO = tmem_base + 256 + q * 128;
                    if (elect_one()) {
                        #pragma unroll
                        for (int ks = half * 4; ks < half * 4 + 4; ks++)
                            tc_mma_ts_lh(tO, tP + ks * 8, va + ((ks * 16 * C::SWB) >> 4), dv_hi, IDESC_PV, ks > 0 ? 1u : acc0);
                        if (last) tc_commit(&o_done[q]);
                    }
                };
                bool ok = true;
                if constexpr (ISSUERS == 2) {
                    // One issuer per tile.
                    const int q = warp - 9;
                    const int n = KSPLIT ? (nblk[0] + 1 - q) / 2 : q ? nblk[1] : nblk[0];      // stages with work for this tile
                    auto stage = [&](int i) { return KSPLIT ? 2 * i + q : i; };
                    if (n > 0) ok = wait(&q_full[KSPLIT ? 0 : q], 0, 24);
                    // S(i) = Q K^T of stage i.
                    auto step_qk = [&](int i) -> bool {
                        if (i >= n) return true;
                        const int j = stage(i), sk = j % NSK;
                        if (!wait(&k_full[sk], j / NSK, 27)) return false;
                        issue_qk(q, sk);
                        return true;
                    };
                    auto step_pv = [&](int i) -> bool {
                        const int j = stage(i), sv = j % NSV;
                        if (!wait(&v_full[sv], j / NSV, 25)) return false;
                        if (!wait(&p_full[q][0], i, 26)) return false;
                        issue_pv(q, sv, i > 0 ? 1u : 0u, 0, false);
                        if (!wait(&p_full[q][1], i, 29)) return false;
                        issue_pv(q, sv, 1u, 1, i == n - 1);
                        return true;
                    };
                    ok = ok && step_qk(0);
                    for (int i = 0; i < n && ok; i++)
                        ok = step_pv(i) && step_qk(i + 1);
                } else {
                    if (nblk_max > 0) {
                        ok = wait(&k_full[0], 0, 23);
                        #pragma unroll
                        for (int q = 0; q < 2; q++) {
                            if (nblk[q] == 0 || !ok) continue;
                            ok = wait(&q_full[q], 0, 24);
                            if (ok) issue_qk(q, 0);
                        }
                    }
                    for (int j = 0; j < nblk_max && ok; j++) {
                        const int sv = j % NSV, sk = (j + 1) % NSK;
                        ok = wait(&v_full[sv], j / NSV, 25);
                        if (ok && j + 1 < nblk_max) ok = wait(&k_full[sk], (j + 1) / NSK, 27);
                        #pragma unroll
                        for (int q = 0; q < 2; q++) {
                            if (j >= nblk[q] || !ok) continue;
                            ok = wait(&p_full[q][0], j, 26);
                            if (!ok) continue;
                            issue_pv(q, sv, j > 0 ? 1u : 0u, 0, false);
                            ok = wait(&p_full[q][1], j, 29);
                            if (!ok) continue;
                            issue_pv(q, sv, 1u, 1, j + 1 == nblk[q]);
                            if (j + 1 < nblk[q]) issue_qk(q, sk);
                        }
                    }
                }
            }
            end_item();
            if (!PERSIST) break;
        }
    } else {
        setmaxnreg_inc_224();
        for (int round = 0; ; round++) {
            ItemInfo it;
            if (!fetch_item(round, it)) break;
            EFA_ITEM_LOCALS
            // =====================================================================================
            // Softmax warpgroups: tile q = warp / 4, row = thread index within the warpgroup
            // =====================================================================================
            const int q = warp >> 2;
            const int row = tid - q * WS_BM;
            const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
            const uint32_t tmem_S = tmem_base + q * 128 + lane_base;
            const uint32_t tmem_O = tmem_base + 256 + q * 128 + lane_base;
            const int my_rows = q ? rows_q[1] : rows_q[0];
            const int my_nblk = KSPLIT ? (nblk[0] + 1 - q) / 2 : q ? nblk[1] : nblk[0];
            const int my_abs0 = q ? q_abs0[1] : q_abs0[0];
            // Who gives ring slots back: with an issuer per warpgroup each for its part, else the tile that is issued last. Tile 1 sweeps at most
            // one stage more than tile 0, its very last one, whose slots nothing waits for.
            const bool gives_back = (warp & 3) == 0 && lane == 0 && (ISSUERS == 2 || q == (nblk[1] > 0 ? 1 : 0));
            auto stage_of = [&](int j) { return KSPLIT ? 2 * j + q : j; };

            float m_ref = kNegInfW;     // exponent offset in use (a past row maximum), scaled by scale*log2(e)
            float m_true = kNegInfW;    // true running row maximum, same scaling
            float l_run = 0.f;          // running denominator relative to m_ref
            bool ok = true;

            for (int j = 0; j < my_nblk; j++) {
                const int kb = kv_lo + (KSPLIT ? 2 * j + q : j) * WS_BN;
                ok = __all_sync(0xffffffffu, mbar_wait(&s_full[q], (uint32_t)(j & 1), &abort_word, 31));
                if (!ok) break;
                tc_fence_after_sync();
                if (gives_back) {
                    mbar_arrive(&k_empty[stage_of(j) % NSK]);
                    if (j > 0) mbar_arrive(&v_empty[stage_of(j - 1) % NSV]);
                }

                uint32_t su[4][32];
                #pragma unroll
                for (int c = 0; c < 4; c++) tmem_ld32(tmem_S + c * 32, su[c]);
                tmem_wait_ld();

                const bool need_mask = (kb + WS_BN > kv_hi) || (a.causal && kb + WS_BN - 1 > my_abs0);
                if (need_mask) {
                    int lim = kv_hi - 1 - kb;
                    if (a.causal) lim = min(lim, my_abs0 + row - kb);
                    #pragma unroll
                    for (int c = 0; c < 4; c++)
                        #pragma unroll
                        for (int i = 0; i < 32; i++)
                            if (c * 32 + i > lim) su[c][i] = 0xff800000u;
                }

                // row maximum: four independent chains of three-input max (half the instructions of fmaxf)
                float mx0 = kNegInfW, mx1 = kNegInfW, mx2 = kNegInfW, mx3 = kNegInfW;
                #pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    mx0 = max3(mx0, __uint_as_float(su[0][i]), __uint_as_float(su[0][i + 1]));
                    mx1 = max3(mx1, __uint_as_float(su[1][i]), __uint_as_float(su[1][i + 1]));
                    mx2 = max3(mx2, __uint_as_float(su[2][i]), __uint_as_float(su[2][i + 1]));
                    mx3 = max3(mx3, __uint_as_float(su[3][i]), __uint_as_float(su[3][i + 1]));
                }
                const float mx = fmaxf(fmaxf(mx0, mx1), fmaxf(mx2, mx3));
                m_true = fmaxf(m_true, mx * a.scale_log2e);

                // Move the exponent offset only when the maximum grew by more than the threshold.
                float alpha = 1.f;
                if (m_true - m_ref > a.rescale_above || m_ref == kNegInfW) {     // (-inf) - (-inf) is NaN: second test
                    const float m_new = m_true;
                    const float m_use = (m_new == kNegInfW) ? 0.f : m_new;
                    alpha = (m_ref == kNegInfW) ? 0.f : ex2(m_ref - m_use);
                    m_ref = m_new;
                }
                const float m_off = (m_ref == kNegInfW) ? 0.f : m_ref;

                // P is handed to the MMA warp in two halves of 64 keys: the first four k-steps of P*V run on
                // the tensor pipe while the exponentials of the second half are still being computed.
                const uint64_t scale2 = pack2(a.scale_log2e, a.scale_log2e), off2 = pack2(-m_off, -m_off);
                uint64_t psum2[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
                auto weights = [&](int c, uint32_t (&pk)[16]) {
                    #pragma unroll
                    for (int i = 0; i < 16; i++) {
                        if (POLY && i % 4 == 3) {
                            const uint64_t e = exp2_poly2(fma2(pack2(__uint_as_float(su[c][2 * i]), __uint_as_float(su[c][2 * i + 1])), scale2, off2));
                            float e0, e1;
                            unpack2(e, e0, e1);
                            psum2[i & 1] = add2(psum2[i & 1], e);
                            pk[i] = pack_f16x2(e0, e1);
                            continue;
                        }
                        float x0, x1;
                        unpack2(fma2(pack2(__uint_as_float(su[c][2 * i]), __uint_as_float(su[c][2 * i + 1])), scale2, off2), x0, x1);
                        const float q0 = ex2(x0), q1 = ex2(x1);
                        psum2[i & 1] = add2(psum2[i & 1], pack2(q0, q1));
                        pk[i] = pack_f16x2(q0, q1);
                    }
                };
                uint32_t pk[2][16];

                // O may be rescaled and P overwritten once PV(j-1) of this tile is complete, which S(j) complete implies (the tensor pipe
                // runs in issue order): no part of PV(j) is issued before this warp's first arrival below.
                if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                    #pragma unroll
                    for (int c = 0; c < D / 32; c++) {
                        uint32_t o[32];
                        tmem_ld32(tmem_O + c * 32, o);
                        tmem_wait_ld();
                        #pragma unroll
                        for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st32(tmem_O + c * 32, o);
                    }
                }

                #pragma unroll
                for (int c = 0; c < 4; c++) {
                    weights(c, pk[c & 1]);
                    tmem_st16(tmem_S + c * 16, pk[c & 1]);
                    if (c == 1 || c == 3) {
                        tmem_wait_st();
                        tc_fence_before_sync();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&p_full[q][c >> 1]);
                    }
                }
                float ps0, ps1;
                {
                    float s0, s1, s2, s3;
                    unpack2(psum2[0], s0, s1);
                    unpack2(psum2[1], s2, s3);
                    ps0 = s0 + s2;
                    ps1 = s1 + s3;
                }
                l_run = l_run * alpha + (ps0 + ps1);
            }

            if (ok && my_nblk > 0) {
                ok = __all_sync(0xffffffffu, mbar_wait(&o_done[q], 0u, &abort_word, 32));
                tc_fence_after_sync();
            }

            // KSPLIT: both warpgroups learn each other's offset, maximum and sum; each then merges half of the columns. The
            // exchange goes through K slot q, which only this warpgroup's stages used: all of them are consumed here.
            float w_own = 1.f, w_other = 0.f;
            if constexpr (KSPLIT) {
                float* own = reinterpret_cast<float*>(sK + q * C::TILE_BYTES) + row;
                const float* other = reinterpret_cast<const float*>(sK + (q ^ 1) * C::TILE_BYTES) + row;
                own[0] = m_ref; own[WS_BM] = m_true; own[2 * WS_BM] = l_run;
                tc_fence_before_sync();
                asm volatile("bar.sync 1, 256;" ::: "memory");
                tc_fence_after_sync();
                ok = __all_sync(0xffffffffu, ok && abort_word == 0);
                const float m_ref_o = other[0], l_o = other[2 * WS_BM];
                const float m_all = fmaxf(m_ref, m_ref_o);
                w_own   = (m_ref == kNegInfW) ? 0.f : ex2(m_ref - m_all);
                w_other = (m_ref_o == kNegInfW) ? 0.f : ex2(m_ref_o - m_all);
                m_true = fmaxf(m_true, other[WS_BM]);
                l_run = l_run * w_own + l_o * w_other;
                m_ref = m_all;
            }
            // Columns [c_lo, c_hi) in steps of 16.
            const int c_lo = KSPLIT && q == 1 ? D / 32 : 0, c_hi = KSPLIT && q == 0 ? D / 32 : D / 16;

            // ---- epilogue: this thread's row (warps take this branch as a whole: my_rows is 0, 64 or 128)
            if (ok && (warp & 3) * 32 < my_rows) {
                const int head = *(volatile int*)&s_head, split = *(volatile int*)&s_split, block_row0 = *(volatile int*)&s_row0;   // not kept in registers through the loop
                const size_t ld_o = (size_t)a.H_local * D;
                const size_t orow = (size_t)block_row0 + (KSPLIT ? 0 : q * WS_BM) + row;
                float mult;
                float*  dst32 = nullptr;
                __half* dst16 = nullptr;
                if (a.nsplit == 1) {
                    mult = 1.f / l_run;
                    if constexpr (OUT_F16) dst16 = a.O16 + orow * ld_o + (size_t)head * D;
                    else                   dst32 = a.O32 + orow * ld_o + (size_t)head * D;
                } else {
                    // partials are stored relative to the true row maximum
                    mult = (m_true == kNegInfW) ? 0.f : ex2(m_ref - m_true);
                    dst32 = a.O_part + ((size_t)split * a.part_rows + orow) * ld_o + (size_t)head * D;
                    const size_t s0 = ((size_t)split * a.part_rows + orow) * a.H_local + head;
                    if (!KSPLIT || q == 0) {
                        a.m_part[s0] = m_true;
                        a.l_part[s0] = partial_sum(l_run * mult, !a.causal || split * a.kv_len <= a.q_start + (int)orow);
                    }
                }
                #pragma unroll
                for (int c = 0; c < D / 16; c++) {
                    if (KSPLIT && (c < c_lo || c >= c_hi)) continue;
                    uint32_t o[16];
                    if (my_nblk > 0) {
                        tmem_ld16(tmem_O + c * 16, o);
                        tmem_wait_ld();
                    } else {
                        #pragma unroll
                        for (int i = 0; i < 16; i++) o[i] = 0u;
                    }
                    if constexpr (KSPLIT) {
                        uint32_t o2[16];
                        const bool other_ran = (nblk[0] + q) / 2 > 0;            // stages of the other warpgroup
                        if (other_ran) {
                            tmem_ld16(tmem_base + 256 + (q ^ 1) * 128 + lane_base + c * 16, o2);
                            tmem_wait_ld();
                        }
                        #pragma unroll
                        for (int i = 0; i < 16; i++)
                            o[i] = __float_as_uint(__uint_as_float(o[i]) * w_own + (other_ran ? __uint_as_float(o2[i]) * w_other : 0.f));
                    }
                    if (dst16) {
                        uint4 v0, v1;
                        v0.x = pack_f16x2(__uint_as_float(o[0]) * mult,  __uint_as_float(o[1]) * mult);
                        v0.y = pack_f16x2(__uint_as_float(o[2]) * mult,  __uint_as_float(o[3]) * mult);
                        v0.z = pack_f16x2(__uint_as_float(o[4]) * mult,  __uint_as_float(o[5]) * mult);
                        v0.w = pack_f16x2(__uint_as_float(o[6]) * mult,  __uint_as_float(o[7]) * mult);
                        v1.x = pack_f16x2(__uint_as_float(o[8]) * mult,  __uint_as_float(o[9]) * mult);
                        v1.y = pack_f16x2(__uint_as_float(o[10]) * mult, __uint_as_float(o[11]) * mult);
                        v1.z = pack_f16x2(__uint_as_float(o[12]) * mult, __uint_as_float(o[13]) * mult);
                        v1.w = pack_f16x2(__uint_as_float(o[14]) * mult, __uint_as_float(o[15]) * mult);
                        uint4* d = reinterpret_cast<uint4*>(dst16 + c * 16);
                        d[0] = v0;
                        d[1] = v1;
                    } else {
                        float4* d = reinterpret_cast<float4*>(dst32 + c * 16);
                        #pragma unroll
                        for (int qd = 0; qd < 4; qd++)
                            d[qd] = make_float4(__uint_as_float(o[4 * qd]) * mult, __uint_as_float(o[4 * qd + 1]) * mult,
                                                __uint_as_float(o[4 * qd + 2]) * mult, __uint_as_float(o[4 * qd + 3]) * mult);
                    }
                }

                // ---- completion signal: one count per finished 64-row block, after its rows are visible.
                // A 64-row block is two warps (KSPLIT: of each warpgroup); the last of them to get here publishes the count.
                if (a.tile_counters != nullptr) {
                    if (a.counters_sys) __threadfence_system(); else __threadfence();
                    __syncwarp();
                    if (lane == 0) {
                        const int half = (warp & 3) >> 1;
                        if (atomicAdd(&half_done[KSPLIT ? 0 : q][half], 1) == (KSPLIT ? 3 : 1)) {
                            if (a.counters_sys) __threadfence_system(); else __threadfence();
                            atomicAdd(a.tile_counters + (block_row0 + (KSPLIT ? 0 : q * WS_BM) + half * 64) / a.tile_rows, 1);
                        }
                    }
                }
            }
            end_item();
            if (!PERSIST) break;
        }
    }
#undef EFA_ITEM_LOCALS
    __syncthreads();

    // ---- teardown
    if (abort_word != 0) {
        for (int i = 0; i < 64; i++) __nanosleep(100000);
        if (tid == 0 && a.status != nullptr) {
            if (atomicCAS(a.status, 0, (int)KS_WAIT_TIMEOUT) == 0) {
                a.status[1] = s_item;
                a.status[2] = abort_word;
            }
        }
        __syncthreads();
    }
    if (warp == 9) tmem_dealloc(tmem_base, C::TMEM_COLS);
    if (behind) pdl_wait();
}

// The registers that the softmax warps take come out of what the block was launched with: with less than that they would wait for
// ever, so it is looked at before the first launch.
template <int D, bool OUT_F16, int WAYS>
int configure_chains()
{
    cudaFuncAttributes attr;
    EFA_CUDA(cudaFuncGetAttributes(&attr, fa_fwd_chains_kernel<D, OUT_F16, WAYS>));
    if ((attr.numRegs + 7) / 8 * 8 * CH_THREADS < 512 * 104 + 128 * 40 + 128 * 24) { set_error("attention kernel compiled to %d registers", attr.numRegs); return 1; }
    EFA_CUDA(cudaFuncSetAttribute(fa_fwd_chains_kernel<D, OUT_F16, WAYS>, cudaFuncAttributeMaxDynamicSharedMemorySize, ChainCfg<D, WAYS>::SMEM_BYTES));
    return 0;
}

// The first launch of a head size and output type on a device loads and configures every form of it: which one a launch
// takes depends on its shape, and a later one may be inside a stream capture or find no device memory left.
template <int D, bool OUT_F16>
int configure_forms()
{
    static bool configured[64] = {};
    int dev = 0;
    EFA_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64 || configured[dev]) return 0;
    constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    if constexpr (D == 128) {
        EFA_CUDA(cudaFuncSetAttribute(fa_fwd_ws_kernel<D, OUT_F16, false, false>, attr, WsCfg<D, false>::SMEM_BYTES));
        EFA_CUDA(cudaFuncSetAttribute(fa_fwd_ws_kernel<D, OUT_F16, false, true>, attr, WsCfg<D, true>::SMEM_BYTES));
    } else {
        if (configure_chains<D, OUT_F16, 2>() || configure_chains<D, OUT_F16, 4>()) return 1;
    }
    if constexpr (D >= 64) EFA_CUDA(cudaFuncSetAttribute(fa_fwd_ws_kernel<D, OUT_F16, true, false>, attr, WsCfg<D, false>::SMEM_BYTES));
    else if (fa_tile_preload()) return 1;
    configured[dev] = true;
    return 0;
}

template <int D, bool OUT_F16, int WAYS>
int launch_chains(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& args, cudaStream_t stream, int blocks)
{
    using C = ChainCfg<D, WAYS>;
    const int items_x = args.H_local * args.nsplit, rows = C::TILES * WS_BM;
    const int items_y = (args.q_rows + rows - 1) / rows;
    const dim3 grid = blocks > 0 ? dim3(blocks) : dim3(items_x, items_y);
    // The kernel picks its item, and with an order table reads that, ahead of its wait for the kernels before it (0.3 us of a small launch): with
    // a table, which one of them may be writing, it does not start early.
    const bool early = args.order_tab == nullptr;
    EFA_CUDA(launch_kernel(early, 1, fa_fwd_chains_kernel<D, OUT_F16, WAYS>, grid, CH_THREADS, C::SMEM_BYTES, stream, tq, tk, tv, args, items_x, WAYS == 4 && blocks > 0 ? blocks : items_x * items_y));
    return 0;
}

// reserve_sms >= 0: the persistent form on that many SMs less. blocks: of a 1-D grid; 0: all.
template <int D, bool OUT_F16, bool KSPLIT = false>
int launch_ws(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& args, cudaStream_t stream, int reserve_sms, int blocks)
{
    using C = WsCfg<D, KSPLIT>;
    const int items_x = args.H_local * args.nsplit;
    const int item_rows = KSPLIT ? WS_BM : 2 * WS_BM;
    const int items_y = (args.q_rows + item_rows - 1) / item_rows;
    const int total = items_x * items_y;
    if constexpr (!KSPLIT) {
        if (reserve_sms >= 0) {
            const int ctas = std::min(total, std::max(1, device_sms() - reserve_sms));
            int* counter = work_counter_slot();
            if (!counter) { set_error("no device memory for the work counter"); return 1; }
            EFA_CUDA(cudaMemsetAsync(counter, 0, sizeof(int), stream));
            EFA_CUDA(launch_early(fa_fwd_ws_kernel<D, OUT_F16, true, false>, dim3(ctas), WS_THREADS, C::SMEM_BYTES, stream, tq, tk, tv, args, counter, items_x, total));
            return 0;
        }
    }
    if constexpr (D == 128) {
        const dim3 grid = blocks > 0 ? dim3(blocks) : dim3(items_x, items_y);
        EFA_CUDA(launch_early(fa_fwd_ws_kernel<D, OUT_F16, false, KSPLIT>, grid, WS_THREADS, C::SMEM_BYTES, stream, tq, tk, tv, args, (int*)nullptr, items_x, KSPLIT && blocks > 0 ? blocks : total));
    }
    return 0;
}

// Items of 256 rows (HALVES: 128); blocks: of a 1-D grid, 0: all.
template <int D, bool OUT_F16, bool HALVES>
int launch_items(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& args, cudaStream_t stream, int blocks = 0)
{
    if constexpr (D == 128) return launch_ws<D, OUT_F16, HALVES>(tq, tk, tv, args, stream, -1, blocks);
    else return launch_chains<D, OUT_F16, HALVES ? 4 : 2>(tq, tk, tv, args, stream, blocks);
}

template <int D, bool OUT_F16>
int launch_form(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& a, int reserve_sms, cudaStream_t stream)
{
    if (configure_forms<D, OUT_F16>()) return 1;
    if constexpr (D >= 64)
        if (reserve_sms > 0) return launch_ws<D, OUT_F16>(tq, tk, tv, a, stream, reserve_sms, 0);
    const FaPlan plan = fa_ws_plan(a, D, reserve_sms);
    if (plan.tiles > 0) return fa_forward_tile(tq, tk, tv, a, D, OUT_F16, stream);
    if (plan.items128 > 0 && plan.items256 == 0) return launch_items<D, OUT_F16, true>(tq, tk, tv, a, stream);
    if (plan.items128 > 0) {
        FaArgs t = a;
        t.tail_first = plan.items256;
        t.tail_total = plan.items256 + plan.items128 / 2;
        if (int rc = launch_items<D, OUT_F16, false>(tq, tk, tv, a, stream, t.tail_first)) return rc;
        return launch_items<D, OUT_F16, true>(tq, tk, tv, t, stream, plan.items128);
    }
    return launch_items<D, OUT_F16, false>(tq, tk, tv, a, stream);
}

template <int D>
int launch_form(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& a, bool out_f16,
                int reserve_sms, cudaStream_t stream)
{
    return out_f16 ? launch_form<D, true>(tq, tk, tv, a, reserve_sms, stream) : launch_form<D, false>(tq, tk, tv, a, reserve_sms, stream);
}

template <int D>
void ring_of(FaPlan& plan, bool halves)
{
    if constexpr (D == 128) {
        plan.k_slots = halves ? WsCfg<D, true>::NSTAGE_K : WsCfg<D, false>::NSTAGE_K;
        plan.v_slots = halves ? WsCfg<D, true>::NSTAGE_V : WsCfg<D, false>::NSTAGE_V;
    } else {
        plan.k_slots = halves ? ChainCfg<D, 4>::NSK : ChainCfg<D, 2>::NSK;
        plan.v_slots = halves ? ChainCfg<D, 4>::NSV : ChainCfg<D, 2>::NSV;
    }
    plan.stage_step = halves ? 2 : 1;
}

}  // namespace

// Which items a launch goes as (attention_plan.h) and the rings of their kernel. Host arithmetic only.
FaPlan fa_ws_plan(const FaArgs& a, int d_h, int reserve_sms)
{
    FaPlan plan = plan_items(PlanShape{a.q_start, a.q_rows, a.S, a.H_local, a.nsplit, a.kv_len, a.causal, d_h,
                                       a.order_tab == nullptr && !(reserve_sms > 0 && d_h >= 64), a.group_heads > 0 || a.heavy_first != 0, device_sms()});
    if (plan.tiles > 0) {
        plan.k_slots = plan.v_slots = 2;
        plan.stage_step = 1;
        return plan;
    }
    const bool ks = plan.items128 > 0;
    switch (d_h) {
        case 16:  ring_of<16>(plan, ks);  break;
        case 32:  ring_of<32>(plan, ks);  break;
        case 64:  ring_of<64>(plan, ks);  break;
        case 128: ring_of<128>(plan, ks); break;
    }
    return plan;
}

// Launch of the warp-specialised kernel; the caller has validated the arguments and built the maps.
// reserve_sms > 0 selects the persistent form with that many SMs left free (d_h 64 and 128).
int fa_forward_ws(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& a,
                  int d_h, bool out_f16, int reserve_sms, cudaStream_t stream)
{
    switch (d_h) {
        case 16:  return launch_form<16>(tq, tk, tv, a, out_f16, reserve_sms, stream);
        case 32:  return launch_form<32>(tq, tk, tv, a, out_f16, reserve_sms, stream);
        case 64:  return launch_form<64>(tq, tk, tv, a, out_f16, reserve_sms, stream);
        case 128: return launch_form<128>(tq, tk, tv, a, out_f16, reserve_sms, stream);
    }
    set_error("fa_forward_ws: d_h=%d is not 16, 32, 64 or 128", d_h);
    return 2;
}

int fa_ws_kv_box_rows() { return WS_BN; }


namespace {
template <class K> int touch_kernel(K kernel)
{
    cudaFuncAttributes attr;
    EFA_CUDA(cudaFuncGetAttributes(&attr, kernel));
    return 0;
}
}  // namespace

// Loads the code of every instantiation now. A kernel's first launch may otherwise have to wait for the device to go
// idle, which it never does while a stream sits in a front-end wait on a counter that is not coming.
template <int D, bool OUT_F16>
static int touch_forms()
{
    if constexpr (D >= 64)
        if (touch_kernel(fa_fwd_ws_kernel<D, OUT_F16, true, false>)) return 1;
    if constexpr (D == 128)
        return touch_kernel(fa_fwd_ws_kernel<D, OUT_F16, false, false>) || touch_kernel(fa_fwd_ws_kernel<D, OUT_F16, false, true>);
    else
        return touch_kernel(fa_fwd_chains_kernel<D, OUT_F16, 2>) || touch_kernel(fa_fwd_chains_kernel<D, OUT_F16, 4>);
}

int fa_ws_preload()
{
    return touch_forms<16, true>() || touch_forms<16, false>() || touch_forms<32, true>() || touch_forms<32, false>() ||
           touch_forms<64, true>() || touch_forms<64, false>() || touch_forms<128, true>() || touch_forms<128, false>();
}

}  // namespace efa
