// FlashAttention forward for sm_100a with one Q tile per block, d_h 16 and 32: launches of few keys per row and more than
// one wave. Same arguments, partials and completion counters as fa_fwd_ws_sm100.cu.
//
// What bounds such a launch is the turnover of its blocks: tensor-memory allocation, barriers, the Q load, the first Q*K^T and
// the epilogue of a row block that has only one or two 128-key stages. Two of these small blocks share an SM and hide each
// other's; the kernel of four chains has the SM to itself, but is faster per stage. The line lies at two stages: 592 items of 256 rows, d_h 16 / 32,
// 8.8 / 9.5 us here against 15.1 / 16.1 (one stage), 23.9 / 26.4 against 24.4 / 27.2 (two), 32.1 / 36.5 against 29.9 / 34.8 (three), 48 / 53 against
// 41 / 47 (five). Under a mask, or where a last wave of 256-row items is poorly filled, the smaller blocks also end more evenly, which
// decides between two and six stages of more than one wave: causal, 100 heads x 512 rows 12.2 / 12.8 against 13.3 / 14.4, 75 x 640 12.6 / 13.2 against
// 15.4 / 16.9 (148 x 512 15.0 / 15.9 against 14.1 / 15.3), 90 x rows 320 to 640 (d_h 32) 13.5 against 18.1; without a mask 160 heads x 256
// rows x 384 keys 14.9 / 15.9 against 14.6 / 16.5, 50 x 640 12.4 / 13.2 against 16.8 / 18.4, 110 x 640 24.4 / 25.4 against 27.0 / 29.2, 160 x 384 16.0 / 17.1 against
// 18.6 / 20.5, 250 x 384 23.3 / 24.3 against 25.7 / 28.0 (200 x 384 22.0 / 23.0 against 20.3 / 22.1, 160 x 576 37.1 / 38.9 against 33.6 / 36.2); but 64 x 512, one
// wave, 11.0 / 11.3 against 8.9 / 9.8, four stages (100 x 768) 21.8 / 22.8 against 21.1 / 22.7, 16 x 2048 32.7 / 34.0 against 16.4 / 17.7 (as 128-row items).
//
// One CTA = 128 query rows of one (head, split). K and V stream through shared memory in 128-key stages filled by TMA
// (32- or 64-byte swizzle). S = Q K^T is a tcgen05.mma with both operands in shared memory and the 128x128 fp32 result
// in tensor memory; each of the 128 threads owns one row of S (tcgen05.ld 32x32b), does the online softmax for that row
// without any shuffle, and writes P as fp16 back into tensor memory over S. O += P V is a tcgen05.mma with A = P from
// tensor memory and B = V from shared memory in MN-major form; O stays in tensor memory for the whole key sweep and is
// rescaled there only when a row maximum moved.
#include "fa_fwd_sm100.cuh"
#include "fa_args.cuh"
#include "host_util.h"
#include "sm100_ptx.cuh"

#include <cmath>

namespace efa {

namespace {

constexpr int FA_BM = 128;      // query rows per CTA
constexpr int FA_BN = 128;      // keys per stage
constexpr float kNegInf = -INFINITY;

template <int D>
struct FaCfg {
    static_assert(D == 16 || D == 32, "one box per tile, two blocks per SM");
    static constexpr int SWB        = D * 2;                     // swizzle width = TMA box row, bytes
    static constexpr int TILE_BYTES = 128 * SWB;
    static constexpr int NSTAGE     = 2;
    static constexpr int SMEM_BYTES = TILE_BYTES * (1 + 2 * NSTAGE) + 1024;   // + alignment slack
    static constexpr int TMEM_COLS  = 256;                       // S/P: 128 columns, O: D columns
    static constexpr int OCH        = D >= 32 ? 32 : 16;         // O columns per tcgen05.ld
};

template <int D, bool OUT_F16>
__global__ void __launch_bounds__(128)
fa_fwd_tile_kernel(const __grid_constant__ CUtensorMap tmQ,
              const __grid_constant__ CUtensorMap tmK,
              const __grid_constant__ CUtensorMap tmV,
              const FaArgs a)
{
    using C = FaCfg<D>;
    constexpr uint32_t SWZ = swizzle_code(C::SWB);
    constexpr uint32_t IDESC_QK = idesc_f16_f32(FA_BM, FA_BN, 0, 0);
    constexpr uint32_t IDESC_PV = idesc_f16_f32(FA_BM, D, 0, 1);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sQ = smem;
    uint8_t* sK = sQ + C::TILE_BYTES;
    uint8_t* sV = sK + C::NSTAGE * C::TILE_BYTES;

    __shared__ __align__(8) uint64_t bar_q;
    __shared__ __align__(8) uint64_t bar_k[C::NSTAGE];
    __shared__ __align__(8) uint64_t bar_v[C::NSTAGE];
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_word;

    const int tid  = threadIdx.x;
    const int warp = tid >> 5;

    // x enumerates (head, split) pairs, y the 128-row blocks: blocks are dispatched in query-row order, or the reverse.
    const int head  = blockIdx.x % a.H_local;
    const int split = blockIdx.x / a.H_local;
    const int block_row0 = (a.heavy_first ? gridDim.y - 1 - blockIdx.y : blockIdx.y) * FA_BM;   // first row of this block within the launch
    const int rows_valid = min(FA_BM, a.q_rows - block_row0);      // 64 or 128
    const int q_abs0 = a.q_start + block_row0;                     // absolute index of the block's first row
    const int kv_lo = split * a.kv_len;
    const int kv_hi = kv_lo + a.kv_len;
    const int kv_end = a.causal ? min(kv_hi, q_abs0 + rows_valid) : kv_hi;
    const int nblk = kv_end > kv_lo ? (kv_end - kv_lo + FA_BN - 1) / FA_BN : 0;

    if (tid == 0) {
        abort_word = 0;
        mbar_init(&bar_q, 1);
        for (int s = 0; s < C::NSTAGE; s++) { mbar_init(&bar_k[s], 1); mbar_init(&bar_v[s], 1); }
        mbar_init(&bar_s, 1);
        mbar_fence_init();
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
    }
    __syncwarp();
    if (warp == 0) tmem_alloc(&tmem_base_smem, C::TMEM_COLS);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();

    pdl_wait();
    pdl_trigger();
    const uint32_t tmem_base = tmem_base_smem;
    const uint32_t tmem_S = tmem_base;            // fp32 S, 128 columns; P (fp16 pairs) reuses columns 0..63
    const uint32_t tmem_O = tmem_base + 128;      // fp32 O, D columns
    const uint32_t lane_base = (uint32_t)(warp * 32) << 16;   // this warp's 32 TMEM lanes

    auto load_tile = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int row) {
        mbar_expect_tx(bar, C::TILE_BYTES);
        tma_load_3d(dst, tm, bar, 0, row, head);
    };
    auto issue_qk = [&](int stage) {
        const uint32_t qa = smem_u32(sQ);
        const uint32_t ka = smem_u32(sK + stage * C::TILE_BYTES);
        #pragma unroll
        for (int ks = 0; ks < D / 16; ks++) {
            const uint32_t off = (uint32_t)ks * 32u;
            tc_mma_ss(tmem_S, smem_desc(qa + off, 16, 8 * C::SWB, SWZ), smem_desc(ka + off, 16, 8 * C::SWB, SWZ),
                      IDESC_QK, ks > 0 ? 1u : 0u);
        }
    };
    auto issue_pv = [&](int stage, bool first) {
        const uint32_t va = smem_u32(sV + stage * C::TILE_BYTES);
        #pragma unroll
        for (int ks = 0; ks < FA_BN / 16; ks++) {
            // 16 keys = two 8-row groups of the MN-major layout
            tc_mma_ts(tmem_O, tmem_S + ks * 8, smem_desc(va + ks * 16 * C::SWB, C::TILE_BYTES, 8 * C::SWB, SWZ),
                      IDESC_PV, (!first || ks > 0) ? 1u : 0u);
        }
    };

    float m_run = kNegInf;     // running row max, already multiplied by scale*log2(e)
    float l_run = 0.f;         // running row denominator
    bool  failed = false;

    if (nblk > 0) {
        if (tid == 0) {
            load_tile(sQ, &tmQ, &bar_q, q_abs0);
            for (int s = 0; s < C::NSTAGE && s < nblk; s++)
                load_tile(sK + s * C::TILE_BYTES, &tmK, &bar_k[s], kv_lo + s * FA_BN);
            for (int s = 0; s + 1 < C::NSTAGE && s < nblk; s++)
                load_tile(sV + s * C::TILE_BYTES, &tmV, &bar_v[s], kv_lo + s * FA_BN);
            if (mbar_wait(&bar_q, 0, &abort_word, 1) && mbar_wait(&bar_k[0], 0, &abort_word, 2)) {
                tc_fence_after_sync();
                issue_qk(0);
                tc_commit(&bar_s);
            }
        }

        for (int j = 0; j < nblk; j++) {
            const int stage = j % C::NSTAGE;
            const int kb = kv_lo + j * FA_BN;                       // first key of this stage

            bool ok = mbar_wait(&bar_s, (uint32_t)(j & 1), &abort_word, 3);
            if (__syncthreads_or((!ok) || abort_word != 0)) { failed = true; break; }
            tc_fence_after_sync();

            // S(j) is complete, hence so are QK(j) and PV(j-1): K stage `stage` and the V stage
            // used by block j-1 are free again.
            if (tid == 0) {
                if (j + C::NSTAGE < nblk)
                    load_tile(sK + stage * C::TILE_BYTES, &tmK, &bar_k[stage], kv_lo + (j + C::NSTAGE) * FA_BN);
                const int vb = j + C::NSTAGE - 1;
                if (vb < nblk && vb >= C::NSTAGE - 1)
                    load_tile(sV + (vb % C::NSTAGE) * C::TILE_BYTES, &tmV, &bar_v[vb % C::NSTAGE], kv_lo + vb * FA_BN);
            }

            // ---- this thread's row of S -> registers
            uint32_t su[4][32];
            #pragma unroll
            for (int c = 0; c < 4; c++) tmem_ld32(tmem_S + lane_base + c * 32, su[c]);
            tmem_wait_ld();

            const bool need_mask = (kb + FA_BN > kv_hi) || (a.causal && kb + FA_BN - 1 > q_abs0);
            if (need_mask) {
                int lim = kv_hi - 1 - kb;                            // last admissible column of this stage
                if (a.causal) lim = min(lim, q_abs0 + tid - kb);
                #pragma unroll
                for (int c = 0; c < 4; c++)
                    #pragma unroll
                    for (int i = 0; i < 32; i++)
                        if (c * 32 + i > lim) su[c][i] = 0xff800000u;   // -inf
            }

            float mx = kNegInf;
            #pragma unroll
            for (int c = 0; c < 4; c++)
                #pragma unroll
                for (int i = 0; i < 32; i++) mx = fmaxf(mx, __uint_as_float(su[c][i]));

            const float m_new = fmaxf(m_run, mx * a.scale_log2e);
            const float m_use = (m_new == kNegInf) ? 0.f : m_new;    // rows with no admissible key yet
            const float alpha = ex2(m_run - m_use);                  // 0 on the first stage
            float psum = 0.f;
            #pragma unroll
            for (int c = 0; c < 4; c++) {
                uint32_t pk[16];
                #pragma unroll
                for (int i = 0; i < 16; i++) {
                    const float p0 = ex2(fmaf(__uint_as_float(su[c][2 * i]),     a.scale_log2e, -m_use));
                    const float p1 = ex2(fmaf(__uint_as_float(su[c][2 * i + 1]), a.scale_log2e, -m_use));
                    psum += p0 + p1;
                    pk[i] = pack_f16x2(p0, p1);
                }
                tmem_st16(tmem_S + lane_base + c * 16, pk);
            }
            l_run = l_run * alpha + psum;
            m_run = m_new;

            // ---- rescale the O accumulator when some row of this warp moved its maximum
            if (j > 0 && __any_sync(0xffffffffu, alpha != 1.f)) {
                #pragma unroll
                for (int c = 0; c < D / C::OCH; c++) {
                    if constexpr (C::OCH == 32) {
                        uint32_t o[32];
                        tmem_ld32(tmem_O + lane_base + c * 32, o);
                        tmem_wait_ld();
                        #pragma unroll
                        for (int i = 0; i < 32; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st32(tmem_O + lane_base + c * 32, o);
                    } else {
                        uint32_t o[16];
                        tmem_ld16(tmem_O + lane_base + c * 16, o);
                        tmem_wait_ld();
                        #pragma unroll
                        for (int i = 0; i < 16; i++) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
                        tmem_st16(tmem_O + lane_base + c * 16, o);
                    }
                }
            }
            tmem_wait_st();
            tc_fence_before_sync();
            __syncthreads();

            if (tid == 0) {
                tc_fence_after_sync();
                if (mbar_wait(&bar_v[stage], (uint32_t)((j / C::NSTAGE) & 1), &abort_word, 4)) {
                    issue_pv(stage, j == 0);
                    bool issue_ok = true;
                    if (j + 1 < nblk) {
                        const int ns = (j + 1) % C::NSTAGE;
                        issue_ok = mbar_wait(&bar_k[ns], (uint32_t)(((j + 1) / C::NSTAGE) & 1), &abort_word, 5);
                        if (issue_ok) issue_qk(ns);
                    }
                    if (issue_ok) tc_commit(&bar_s);
                }
            }
        }

        if (!failed) {
            bool ok = mbar_wait(&bar_s, (uint32_t)(nblk & 1), &abort_word, 6);
            if (__syncthreads_or((!ok) || abort_word != 0)) failed = true;
            tc_fence_after_sync();
        }
    }

    // ---- epilogue: this thread's row of O
    if (!failed && tid < rows_valid) {
        const size_t ld_o = (size_t)a.H_local * D;
        const size_t row = (size_t)block_row0 + tid;
        const float inv = (a.nsplit == 1) ? 1.f / l_run : 1.f;
        float*  dst32 = nullptr;
        __half* dst16 = nullptr;
        if (a.nsplit == 1) {
            if constexpr (OUT_F16) dst16 = a.O16 + row * ld_o + (size_t)head * D;
            else                   dst32 = a.O32 + row * ld_o + (size_t)head * D;
        } else {
            dst32 = a.O_part + ((size_t)split * a.part_rows + row) * ld_o + (size_t)head * D;
            const size_t s0 = ((size_t)split * a.part_rows + row) * a.H_local + head;
            a.m_part[s0] = m_run;
            a.l_part[s0] = partial_sum(l_run, !a.causal || kv_lo <= q_abs0 + tid);
        }
        #pragma unroll
        for (int c = 0; c < D / 16; c++) {
            uint32_t o[16];
            if (nblk > 0) {
                tmem_ld16(tmem_O + lane_base + c * 16, o);
                tmem_wait_ld();
            } else {
                #pragma unroll
                for (int i = 0; i < 16; i++) o[i] = 0u;
            }
            if (dst16) {
                uint4 v0, v1;
                v0.x = pack_f16x2(__uint_as_float(o[0]) * inv,  __uint_as_float(o[1]) * inv);
                v0.y = pack_f16x2(__uint_as_float(o[2]) * inv,  __uint_as_float(o[3]) * inv);
                v0.z = pack_f16x2(__uint_as_float(o[4]) * inv,  __uint_as_float(o[5]) * inv);
                v0.w = pack_f16x2(__uint_as_float(o[6]) * inv,  __uint_as_float(o[7]) * inv);
                v1.x = pack_f16x2(__uint_as_float(o[8]) * inv,  __uint_as_float(o[9]) * inv);
                v1.y = pack_f16x2(__uint_as_float(o[10]) * inv, __uint_as_float(o[11]) * inv);
                v1.z = pack_f16x2(__uint_as_float(o[12]) * inv, __uint_as_float(o[13]) * inv);
                v1.w = pack_f16x2(__uint_as_float(o[14]) * inv, __uint_as_float(o[15]) * inv);
                uint4* d = reinterpret_cast<uint4*>(dst16 + c * 16);
                d[0] = v0;
                d[1] = v1;
            } else {
                float4* d = reinterpret_cast<float4*>(dst32 + c * 16);
                #pragma unroll
                for (int q = 0; q < 4; q++)
                    d[q] = make_float4(__uint_as_float(o[4 * q]) * inv, __uint_as_float(o[4 * q + 1]) * inv,
                                       __uint_as_float(o[4 * q + 2]) * inv, __uint_as_float(o[4 * q + 3]) * inv);
            }
        }
    }
    // rows_valid is 64 or 128, so a warp takes the branch above as a whole and every tcgen05.ld in it
    // is executed by a full warp.

    // ---- signal tile completion: one count per finished 64-row block, after the rows are visible
    if (!failed && a.tile_counters != nullptr) {
        if (a.counters_sys) __threadfence_system(); else __threadfence();
        __syncthreads();
        if (tid == 0) {
            for (int sb = 0; sb < rows_valid; sb += 64)
                atomicAdd(a.tile_counters + (block_row0 + sb) / a.tile_rows, 1);
        }
    }

    // ---- teardown
    if (failed) {
        // Give copies that may still be in flight time to land before the shared memory is released.
        for (int i = 0; i < 64; i++) __nanosleep(100000);
        if (tid == 0 && a.status != nullptr) {
            if (atomicCAS(a.status, 0, (int)KS_WAIT_TIMEOUT) == 0) {
                a.status[1] = (int)(blockIdx.y * gridDim.x + blockIdx.x);
                a.status[2] = abort_word;
            }
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, C::TMEM_COLS);
}

template <int D, bool OUT_F16>
int launch_tile(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& args, cudaStream_t stream)
{
    using C = FaCfg<D>;
    static_assert(C::SMEM_BYTES <= 48 * 1024, "no opt-in to larger shared memory needed");
    const dim3 grid(args.H_local * args.nsplit, (args.q_rows + FA_BM - 1) / FA_BM);
    EFA_CUDA(launch_early(fa_fwd_tile_kernel<D, OUT_F16>, grid, 128, C::SMEM_BYTES, stream, tq, tk, tv, args));
    return 0;
}

template <class K> int touch_kernel(K kernel)
{
    cudaFuncAttributes attr;
    EFA_CUDA(cudaFuncGetAttributes(&attr, kernel));
    return 0;
}

}  // namespace

int fa_forward_tile(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FaArgs& a,
                    int d_h, bool out_f16, cudaStream_t stream)
{
    if (d_h == 16) return out_f16 ? launch_tile<16, true>(tq, tk, tv, a, stream) : launch_tile<16, false>(tq, tk, tv, a, stream);
    if (d_h == 32) return out_f16 ? launch_tile<32, true>(tq, tk, tv, a, stream) : launch_tile<32, false>(tq, tk, tv, a, stream);
    set_error("fa_forward_tile: d_h=%d is not 16 or 32", d_h);
    return 2;
}

int fa_tile_preload()
{
    return touch_kernel(fa_fwd_tile_kernel<16, true>) || touch_kernel(fa_fwd_tile_kernel<16, false>) ||
           touch_kernel(fa_fwd_tile_kernel<32, true>) || touch_kernel(fa_fwd_tile_kernel<32, false>);
}

}  // namespace efa
