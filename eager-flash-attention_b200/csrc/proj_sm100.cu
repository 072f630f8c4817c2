// Output projection for sm_100a: out[rows][d] = A[rows][d_local] * W[d_local][d], fp16 operands,
// fp32 accumulation in tensor memory, fp16 result (or the fp32 accumulator itself, the reference's output type).
//
// Stands in for project() of eager-flash-attention (attn_main.cu:262-273), which calls cublasSgemm on
// fp32 data. Warp-specialised: warp 0 streams A (K-major, [128 rows][64 k]) and W (MN-major,
// [64 k][BN columns] as 64-column boxes) through a ring of shared-memory stages with TMA; warp 1
// issues tcgen05.mma (128 x BN x 16) into one of two BN-column fp32 accumulators in tensor memory and frees each
// stage with tcgen05.commit; warps 2-5 read the accumulator (tcgen05.ld), round to fp16, stage 32 rows x 128 bytes
// per warp in shared memory and store them with TMA (which clips ragged edges).
//
// A CTA keeps taking tiles for as long as blocks of its grid are waiting: clusterlaunchcontrol.try_cancel hands it
// the coordinates of a block that has not started. The copies and MMAs of the next tile then run while this tile is
// written, and barriers and tensor memory are set up once per SM, which is most of the time where d_local is small
// (a 128 x 256 tile of d_local = 512 is 4k cycles of MMA). Unlike a grid of one CTA per SM with a fixed share of the
// tiles, it also suits the launch that starts beside the attention kernel: SMs that come free late find only the
// tiles that nobody has taken. Measured, 4160 x 512 x 4096 (17.4 GFLOP): 30.7 us with a block per tile and row-wise
// stores from registers, 24.6 us like this.
#include "fa_fwd_sm100.cuh"
#include "host_util.h"
#include "sm100_ptx.cuh"

namespace efa {

namespace {

constexpr int PJ_BM = 128;
constexpr int PJ_BK = 64;
constexpr int PJ_EPI_WARPS = 4;

template <int BN, bool STAGED>
struct PjCfg {
    static constexpr int A_BYTES    = PJ_BM * PJ_BK * 2;          // 16 KB
    static constexpr int B_BOX      = PJ_BK * 64 * 2;             // one [64 k][64 n] box, 8 KB
    static constexpr int B_BYTES    = B_BOX * (BN / 64);
    static constexpr int STAGE      = A_BYTES + B_BYTES;
    static constexpr int NSTAGE     = BN == 256 ? 4 : 6;
    static constexpr int OUT_BOX    = 32 * 128;                   // 32 rows of 128 bytes: one TMA store of one warp
    static constexpr int OUT_BYTES  = STAGED ? PJ_EPI_WARPS * 2 * OUT_BOX : 0;   // two per warp
    static constexpr int SMEM_BYTES = STAGE * NSTAGE + OUT_BYTES + 1024;
};

__device__ __forceinline__ uint4 pack8(const uint32_t* x)
{
    return make_uint4(pack_f16x2(__uint_as_float(x[0]), __uint_as_float(x[1])), pack_f16x2(__uint_as_float(x[2]), __uint_as_float(x[3])),
                      pack_f16x2(__uint_as_float(x[4]), __uint_as_float(x[5])), pack_f16x2(__uint_as_float(x[6]), __uint_as_float(x[7])));
}

struct PjArgs {
    int M, N, K;
    int heads, d_h;     // HEADS: N = 3 * heads * d_h
    int* status;
    int behind = 0;     // the launch before it in the stream is a projection of other rows of the same A (project_f16)
};

// HEADS = false: one W [K][N] and one out [M][N].
// HEADS = true: the N columns are those of three weight tensors [heads][K][d_h] side by side, and each tensor's
// result is [heads][M][d_h]. d_h is a multiple of 64, so every 64-column box lies in one head of one tensor, and a
// tile may span heads and tensors: A is read once for all of them, and narrow heads still fill wide tiles. Measured,
// 8192 x 4096 to Q, K and V of four heads of 128: 297 us as twelve launches of 64 tiles each, 100 us as one of 384.
template <int TENSORS>
struct PjMaps {
    CUtensorMap A, W[TENSORS], out[TENSORS];
};

template <int BN, bool OUT_F32, bool HEADS>
__global__ void __launch_bounds__(192, 1)
proj_gemm_kernel(const __grid_constant__ PjMaps<HEADS ? 3 : 1> maps, const PjArgs a)
{
    static_assert(!(OUT_F32 && HEADS), "Q, K and V are fp16");
    using C = PjCfg<BN, true>;
    constexpr uint32_t IDESC = idesc_f16_f32(PJ_BM, BN, 0, 1);
    constexpr uint32_t SWZ = swizzle_code(128);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sOut = smem + C::NSTAGE * C::STAGE;

    __shared__ __align__(8) uint64_t bar_full[C::NSTAGE];
    __shared__ __align__(8) uint64_t bar_empty[C::NSTAGE];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];
    __shared__ __align__(8) uint64_t next_full[2], next_empty[2];
    __shared__ __align__(16) uint4 next_tile[2];                  // answers of try_cancel
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_word;

    const int tid  = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int num_k = (a.K + PJ_BK - 1) / PJ_BK;

    if (tid == 0) {
        abort_word = 0;
        for (int s = 0; s < C::NSTAGE; s++) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        for (int s = 0; s < 2; s++) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], PJ_EPI_WARPS);
            mbar_init(&next_full[s], 1);
            mbar_init(&next_empty[s], 1 + PJ_EPI_WARPS);          // everyone but the thread that asks
        }
        mbar_fence_init();
        tma_prefetch_desc(&maps.A);
        for (int t = 0; t < (HEADS ? 3 : 1); t++) { tma_prefetch_desc(&maps.W[t]); tma_prefetch_desc(&maps.out[t]); }
    }
    __syncwarp();
    if (warp == 1) tmem_alloc(&tmem_base_smem, 2 * BN);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = tmem_base_smem;
    if (!a.behind) pdl_wait();
    pdl_trigger();

    // Tile of round `it`: the CTA's own block first, then the answer to request it - 1. false: no more (or gave up).
    auto next = [&](int it, int& bx, int& by) -> bool {
        const int s = it & 1;
        if (!mbar_wait(&next_full[s], (uint32_t)((it >> 1) & 1), &abort_word, 14)) return false;
        return clc_query(&next_tile[s], bx, by);
    };

    // HEADS: tensor, head and column within the head of a column of the whole.
    auto locate = [&](int col, int& t, int& head, int& x) {
        const int h_all = col / a.d_h;
        t = h_all / a.heads;
        head = h_all - t * a.heads;
        x = col - h_all * a.d_h;
    };

    if (warp == 0) {
        // ---- TMA producer; also asks for the next tile at the start of every tile
        if (lane == 0) {
            int bx = blockIdx.x, by = blockIdx.y;
            int g = 0;                                            // stages filled so far, over all tiles
            bool ok = true;
            for (int it = 0; ok; it++) {
                const int ns = it & 1;
                if (it >= 2 && !mbar_wait(&next_empty[ns], (uint32_t)(((it >> 1) - 1) & 1), &abort_word, 15)) break;
                mbar_expect_tx(&next_full[ns], 16);
                clc_try_cancel(&next_tile[ns], &next_full[ns]);
                const int n0 = bx * BN, m0 = by * PJ_BM;
                const int nbox = min(BN / 64, (a.N - n0) / 64);   // N is a multiple of 64
                int wt[BN / 64], wh[BN / 64], wx[BN / 64];
                if constexpr (HEADS) {
                    #pragma unroll
                    for (int nb = 0; nb < BN / 64; nb++) locate(min(n0 + nb * 64, a.N - 64), wt[nb], wh[nb], wx[nb]);
                }
                for (int kb = 0; kb < num_k; kb++, g++) {
                    const int s = g % C::NSTAGE;
                    const int use = g / C::NSTAGE;
                    if (use > 0 && !mbar_wait(&bar_empty[s], (uint32_t)((use - 1) & 1), &abort_word, 11)) { ok = false; break; }
                    uint8_t* sa = smem + s * C::STAGE;
                    uint8_t* sb = sa + C::A_BYTES;
                    mbar_expect_tx(&bar_full[s], C::A_BYTES + nbox * C::B_BOX);
                    tma_load_2d(sa, &maps.A, &bar_full[s], kb * PJ_BK, m0);
                    #pragma unroll
                    for (int nb = 0; nb < BN / 64; nb++) {
                        if (nb >= nbox) break;
                        if constexpr (HEADS) tma_load_3d(sb + nb * C::B_BOX, &maps.W[wt[nb]], &bar_full[s], wx[nb], kb * PJ_BK, wh[nb]);
                        else                 tma_load_2d(sb + nb * C::B_BOX, &maps.W[0], &bar_full[s], n0 + nb * 64, kb * PJ_BK);
                    }
                }
                if (!ok || !next(it, bx, by)) break;
                fence_proxy_async_smem();
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        if (lane == 0) {
            int bx = 0, by = 0, g = 0;
            bool ok = true;
            for (int it = 0; ok; it++) {
                const int acc = it & 1;
                if (it >= 2) {
                    ok = mbar_wait(&acc_empty[acc], (uint32_t)(((it >> 1) - 1) & 1), &abort_word, 16);
                    if (!ok) break;
                    tc_fence_after_sync();
                }
                const uint32_t tmem_acc = tmem_base + acc * BN;
                for (int kb = 0; kb < num_k && ok; kb++, g++) {
                    const int s = g % C::NSTAGE;
                    ok = mbar_wait(&bar_full[s], (uint32_t)((g / C::NSTAGE) & 1), &abort_word, 12);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint32_t sa = smem_u32(smem + s * C::STAGE);
                    const uint32_t sb = sa + C::A_BYTES;
                    #pragma unroll
                    for (int ks = 0; ks < PJ_BK / 16; ks++) {
                        tc_mma_ss(tmem_acc,
                                  smem_desc(sa + ks * 32, 16, 1024, SWZ),                    // K-major: 32 B per 16 k
                                  smem_desc(sb + ks * 16 * 128, C::B_BOX, 1024, SWZ),        // MN-major: 16 k rows of 128 B
                                  IDESC, (kb > 0 || ks > 0) ? 1u : 0u);
                    }
                    tc_commit(&bar_empty[s]);
                }
                if (!ok) break;
                tc_commit(&acc_full[acc]);
                const bool more = next(it, bx, by);
                fence_proxy_async_smem();
                mbar_arrive(&next_empty[it & 1]);
                if (!more) break;
            }
        }
    } else {
        // ---- epilogue: warps 2..5 own TMEM lanes 32*(warp % 4) .. +31
        constexpr int COLS = OUT_F32 ? 32 : 64;                   // columns in 128 bytes
        const int lane_grp = warp & 3;
        uint8_t* box0 = sOut + lane_grp * 2 * C::OUT_BOX;
        int bx = blockIdx.x, by = blockIdx.y;
        int stores = 0;
        for (int it = 0; ; it++) {
            const int acc = it & 1;
            const int row0 = by * PJ_BM + lane_grp * 32, n0 = bx * BN;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (uint32_t)((it >> 1) & 1), &abort_word, 13))) break;
            tc_fence_after_sync();
            const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(lane_grp * 32) << 16);
            #pragma unroll 1
            for (int c = 0; c < BN / COLS; c++, stores++) {
                if (n0 + c * COLS >= a.N) break;
                uint4 v[8];                                       // this lane's row: eight 16-byte chunks
                if constexpr (OUT_F32) {
                    uint32_t r[32];
                    tmem_ld32(taddr + c * 32, r);
                    tmem_wait_ld();
                    #pragma unroll
                    for (int q = 0; q < 8; q++) v[q] = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                } else {
                    uint32_t r[2][32];
                    tmem_ld32(taddr + c * 64, r[0]);
                    tmem_ld32(taddr + c * 64 + 32, r[1]);
                    tmem_wait_ld();
                    #pragma unroll
                    for (int q = 0; q < 8; q++) v[q] = pack8(&r[q >> 2][8 * (q & 3)]);
                }
                uint8_t* box = box0 + (stores & 1) * C::OUT_BOX;
                if (lane == 0) tma_store_wait_read_but_one();     // the store before last has left this box
                __syncwarp();
                #pragma unroll
                for (int q = 0; q < 8; q++)                       // 128-byte swizzle: eight rows hit eight bank groups
                    *reinterpret_cast<uint4*>(box + lane * 128 + ((q ^ (lane & 7)) << 4)) = v[q];
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if (row0 < a.M) {
                        if constexpr (HEADS) {
                            int t, head, x;
                            locate(n0 + c * COLS, t, head, x);
                            tma_store_3d(&maps.out[t], box, x, row0, head);
                        } else {
                            tma_store_2d(&maps.out[0], box, n0 + c * COLS, row0);
                        }
                    }
                    tma_store_commit();                           // also without a store: the waits above count groups
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acc_empty[acc]);
            const bool more = __all_sync(0xffffffffu, next(it, bx, by));
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(&next_empty[it & 1]);
            if (!more) break;
        }
        if (lane == 0) tma_store_wait_all();
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (abort_word != 0) {
        for (int i = 0; i < 64; i++) __nanosleep(100000);
        if (tid == 0 && a.status != nullptr) {
            if (atomicCAS(a.status, 0, (int)KS_WAIT_TIMEOUT) == 0) {
                a.status[1] = (int)(blockIdx.y * gridDim.x + blockIdx.x);
                a.status[2] = abort_word;
            }
        }
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem_base, 2 * BN);
    if (a.behind) pdl_wait();
}

template <int BN, bool OUT_F32, bool HEADS>
int launch_proj(const PjMaps<HEADS ? 3 : 1>& maps, const PjArgs& args, cudaStream_t stream)
{
    using C = PjCfg<BN, true>;
    static bool configured[64] = {};
    int dev = 0;
    EFA_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        EFA_CUDA(cudaFuncSetAttribute(proj_gemm_kernel<BN, OUT_F32, HEADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
        configured[dev] = true;
    }
    dim3 grid((args.N + BN - 1) / BN, (args.M + PJ_BM - 1) / PJ_BM);
    EFA_CUDA(launch_early(proj_gemm_kernel<BN, OUT_F32, HEADS>, grid, 192, C::SMEM_BYTES, stream, maps, args));
    return 0;
}

// The same with two CTAs to a tile of 256 rows: a pair of neighbouring SMs runs one tcgen05.mma (cta_group::2, 256 x 256 x 16).
// Each CTA stages its own 128 rows of A and HALF of the columns of W, so an SM fetches 32 KB per 64 k instead of 48
// and reads W's part of an operand from shared memory half as often, which is both what bounds the one-CTA form and a good part
// of its power. Rank 0 of the pair issues the MMAs and owns the barriers that they wait for (bar_full, acc_empty); its
// commits arrive in both CTAs. Each CTA keeps its 128 rows of the accumulator and writes them as above. A tile is
// taken over by the pair as a whole (the answer of try_cancel goes to both). 8192 x 4096 x 4096: 200 -> 178 us (1545 TFLOP/s),
// 32768 x 4096 x 4096: 820 -> 727, both under the power cap; 8192 x 4096 to Q, K and V of four heads of 128: 84 -> 76.
struct PjPairCfg {
    static constexpr int BN         = 256;
    static constexpr int A_BYTES    = PJ_BM * PJ_BK * 2;          // 16 KB
    static constexpr int B_BOX      = PJ_BK * 64 * 2;             // one [64 k][64 n] box, 8 KB
    static constexpr int NBOX       = BN / 128;                   // boxes of W in each CTA
    static constexpr int STAGE      = A_BYTES + B_BOX * NBOX;
    static constexpr int NSTAGE     = 6;
    static constexpr int OUT_BOX    = 32 * 128;
    static constexpr int OUT_BYTES  = PJ_EPI_WARPS * 2 * OUT_BOX;
    static constexpr int SMEM_BYTES = STAGE * NSTAGE + OUT_BYTES + 1024;
};

template <bool OUT_F32, bool HEADS>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(192, 1)
proj_pair_kernel(const __grid_constant__ PjMaps<HEADS ? 3 : 1> maps, const PjArgs a)
{
    static_assert(!(OUT_F32 && HEADS), "Q, K and V are fp16");
    using C = PjPairCfg;
    constexpr int BN = C::BN;
    constexpr uint32_t IDESC = idesc_f16_f32(2 * PJ_BM, BN, 0, 1);
    constexpr uint32_t SWZ = swizzle_code(128);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sOut = smem + C::NSTAGE * C::STAGE;

    __shared__ __align__(8) uint64_t bar_full[C::NSTAGE];         // used in rank 0 only: both CTAs' copies count there
    __shared__ __align__(8) uint64_t bar_empty[C::NSTAGE];
    __shared__ __align__(8) uint64_t acc_full[2], acc_empty[2];   // acc_empty: rank 0
    __shared__ __align__(8) uint64_t next_full[2], next_empty[2]; // next_empty: rank 0
    __shared__ __align__(16) uint4 next_tile[2];                  // answers of try_cancel
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_word;

    const int tid  = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);       // known to be one value for the warp
    const int lane = tid & 31;
    const int rank = (int)cluster_rank();
    const int num_k = (a.K + PJ_BK - 1) / PJ_BK;

    if (tid == 0) {
        abort_word = 0;
        for (int s = 0; s < C::NSTAGE; s++) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        for (int s = 0; s < 2; s++) {
            mbar_init(&acc_full[s], 1);
            mbar_init(&acc_empty[s], 2 * PJ_EPI_WARPS);
            mbar_init(&next_full[s], 1);
            mbar_init(&next_empty[s], 2 * PJ_EPI_WARPS + 2);      // both epilogues, the issuer, rank 1's producer
        }
        mbar_fence_init();
        tma_prefetch_desc(&maps.A);
        for (int t = 0; t < (HEADS ? 3 : 1); t++) { tma_prefetch_desc(&maps.W[t]); tma_prefetch_desc(&maps.out[t]); }
    }
    __syncwarp();
    if (warp == 1) tmem_alloc_pair(&tmem_base_smem, 2 * BN);
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();                                               // the other CTA's barriers are there
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_smem, 0);
    if (!a.behind) pdl_wait();
    pdl_trigger();

    // Tile of round `it`: the pair's own block first, then the answer to request it - 1. false: no more (or gave up).
    auto next = [&](int it, int& bx, int& by) -> bool {
        const int s = it & 1;
        if (!mbar_wait(&next_full[s], (uint32_t)((it >> 1) & 1), &abort_word, 14)) return false;
        int x;
        if (!clc_query(&next_tile[s], x, by)) return false;
        bx = x >> 1;                                              // the pair's first block
        return true;
    };

    // HEADS: tensor, head and column within the head of a column of the whole.
    auto locate = [&](int col, int& t, int& head, int& x) {
        const int h_all = col / a.d_h;
        t = h_all / a.heads;
        head = h_all - t * a.heads;
        x = col - h_all * a.d_h;
    };

    if (warp == 0) {
        // ---- TMA producer of each CTA; rank 0's also asks for the next tile at the start of every tile
        if (lane == 0) {
            int bx = blockIdx.x >> 1, by = blockIdx.y;
            int g = 0;                                            // stages filled so far, over all tiles
            bool ok = true;
            for (int it = 0; ok; it++) {
                const int ns = it & 1;
                if (rank == 0 && it >= 2 && !mbar_wait(&next_empty[ns], (uint32_t)(((it >> 1) - 1) & 1), &abort_word, 15)) { ok = false; break; }
                mbar_expect_tx(&next_full[ns], 16);
                if (rank == 0) clc_try_cancel_cluster(&next_tile[ns], &next_full[ns]);
                const int n0 = bx * BN + rank * (BN / 2), m0 = (by * 2 + rank) * PJ_BM;
                int wt[C::NBOX], wh[C::NBOX], wx[C::NBOX];
                if constexpr (HEADS) {
                    #pragma unroll
                    for (int nb = 0; nb < C::NBOX; nb++) locate(min(n0 + nb * 64, a.N - 64), wt[nb], wh[nb], wx[nb]);
                }
                for (int kb = 0; kb < num_k; kb++, g++) {
                    const int s = g % C::NSTAGE;
                    const int use = g / C::NSTAGE;
                    if (use > 0 && !mbar_wait(&bar_empty[s], (uint32_t)((use - 1) & 1), &abort_word, 11)) { ok = false; break; }
                    uint8_t* sa = smem + s * C::STAGE;
                    uint8_t* sb = sa + C::A_BYTES;
                    const uint32_t full = cluster_addr(&bar_full[s], 0);
                    if (rank == 0) mbar_expect_tx(&bar_full[s], 2 * C::STAGE);
                    tma_load_2d_pair(sa, &maps.A, full, kb * PJ_BK, m0);      // rows and columns past the end read as zeros
                    #pragma unroll
                    for (int nb = 0; nb < C::NBOX; nb++) {
                        if constexpr (HEADS) tma_load_3d_pair(sb + nb * C::B_BOX, &maps.W[wt[nb]], full, wx[nb], kb * PJ_BK, wh[nb]);
                        else                 tma_load_2d_pair(sb + nb * C::B_BOX, &maps.W[0], full, n0 + nb * 64, kb * PJ_BK);
                    }
                }
                if (!ok || !next(it, bx, by)) break;
                fence_proxy_async_smem();
                if (rank != 0) mbar_arrive_cluster(cluster_addr(&next_empty[it & 1], 0));
            }
            // rank 0's commits arrive here as well: none may be on its way when this CTA ends
            for (int s = max(0, g - C::NSTAGE); ok && s < g; s++)
                ok = mbar_wait(&bar_empty[s % C::NSTAGE], (uint32_t)((s / C::NSTAGE) & 1), &abort_word, 17);
        }
    } else if (warp == 1) {
        // ---- MMA issuer of the pair
        if (rank == 0 && lane == 0) {
            const uint64_t da = smem_desc(smem_u32(smem), 16, 1024, SWZ);                          // K-major
            const uint64_t db = smem_desc(smem_u32(smem) + C::A_BYTES, C::B_BOX, 1024, SWZ);       // MN-major: 16 k rows of 128 B
            const uint32_t da_lo = (uint32_t)da, da_hi = (uint32_t)(da >> 32), db_lo = (uint32_t)db, db_hi = (uint32_t)(db >> 32);
            int bx = 0, by = 0, g = 0;
            bool ok = true;
            for (int it = 0; ok; it++) {
                const int acc = it & 1;
                if (it >= 2) {
                    ok = mbar_wait(&acc_empty[acc], (uint32_t)(((it >> 1) - 1) & 1), &abort_word, 16);
                    if (!ok) break;
                    tc_fence_after_sync();
                }
                const uint32_t tmem_acc = tmem_base + acc * BN;
                for (int kb = 0; kb < num_k && ok; kb++, g++) {
                    const int s = g % C::NSTAGE;
                    ok = mbar_wait(&bar_full[s], (uint32_t)((g / C::NSTAGE) & 1), &abort_word, 12);
                    if (!ok) break;
                    tc_fence_after_sync();
                    const uint32_t off = (uint32_t)(s * (C::STAGE >> 4));
                    #pragma unroll
                    for (int ks = 0; ks < PJ_BK / 16; ks++)
                        tc_mma_ss_pair(tmem_acc, da_lo + off + ks * 2, da_hi, db_lo + off + ks * 128, db_hi,
                                       IDESC, (kb > 0 || ks > 0) ? 1u : 0u);
                    tc_commit_pair(&bar_empty[s]);
                }
                if (!ok) break;
                tc_commit_pair(&acc_full[acc]);
                const bool more = next(it, bx, by);
                fence_proxy_async_smem();
                mbar_arrive(&next_empty[it & 1]);
                if (!more) break;
            }
        }
    } else {
        // ---- epilogue of this CTA's 128 rows: warps 2..5 own TMEM lanes 32*(warp % 4) .. +31
        constexpr int COLS = OUT_F32 ? 32 : 64;                   // columns in 128 bytes
        const int lane_grp = warp & 3;
        uint8_t* box0 = sOut + lane_grp * 2 * C::OUT_BOX;
        int bx = blockIdx.x >> 1, by = blockIdx.y;
        int stores = 0;
        for (int it = 0; ; it++) {
            const int acc = it & 1;
            const int row0 = (by * 2 + rank) * PJ_BM + lane_grp * 32, n0 = bx * BN;
            if (!__all_sync(0xffffffffu, mbar_wait(&acc_full[acc], (uint32_t)((it >> 1) & 1), &abort_word, 13))) break;
            tc_fence_after_sync();
            const uint32_t taddr = tmem_base + acc * BN + ((uint32_t)(lane_grp * 32) << 16);
            #pragma unroll 1
            for (int c = 0; c < BN / COLS; c++, stores++) {
                if (n0 + c * COLS >= a.N || row0 >= a.M) break;
                uint4 v[8];                                       // this lane's row: eight 16-byte chunks
                if constexpr (OUT_F32) {
                    uint32_t r[32];
                    tmem_ld32(taddr + c * 32, r);
                    tmem_wait_ld();
                    #pragma unroll
                    for (int q = 0; q < 8; q++) v[q] = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                } else {
                    uint32_t r[2][32];
                    tmem_ld32(taddr + c * 64, r[0]);
                    tmem_ld32(taddr + c * 64 + 32, r[1]);
                    tmem_wait_ld();
                    #pragma unroll
                    for (int q = 0; q < 8; q++) v[q] = pack8(&r[q >> 2][8 * (q & 3)]);
                }
                uint8_t* box = box0 + (stores & 1) * C::OUT_BOX;
                if (lane == 0) tma_store_wait_read_but_one();     // the store before last has left this box
                __syncwarp();
                #pragma unroll
                for (int q = 0; q < 8; q++)                       // 128-byte swizzle: eight rows hit eight bank groups
                    *reinterpret_cast<uint4*>(box + lane * 128 + ((q ^ (lane & 7)) << 4)) = v[q];
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) {
                    if constexpr (HEADS) {
                        int t, head, x;
                        locate(n0 + c * COLS, t, head, x);
                        tma_store_3d(&maps.out[t], box, x, row0, head);
                    } else {
                        tma_store_2d(&maps.out[0], box, n0 + c * COLS, row0);
                    }
                    tma_store_commit();
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(&acc_empty[acc], 0));
            const bool more = __all_sync(0xffffffffu, next(it, bx, by));
            fence_proxy_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(cluster_addr(&next_empty[it & 1], 0));
            if (!more) break;
        }
        if (lane == 0) tma_store_wait_all();
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (abort_word != 0) {
        for (int i = 0; i < 64; i++) __nanosleep(100000);
        if (tid == 0 && a.status != nullptr) {
            if (atomicCAS(a.status, 0, (int)KS_WAIT_TIMEOUT) == 0) {
                a.status[1] = (int)(blockIdx.y * gridDim.x + blockIdx.x);
                a.status[2] = abort_word;
            }
        }
        __syncthreads();
    }
    cluster_sync();                                               // arrivals and MMAs of the pair reach into both CTAs
    if (warp == 1) tmem_dealloc_pair(tmem_base, 2 * BN);
    if (a.behind) pdl_wait();
}

template <bool OUT_F32, bool HEADS>
int launch_pair(const PjMaps<HEADS ? 3 : 1>& maps, const PjArgs& args, cudaStream_t stream)
{
    using C = PjPairCfg;
    static bool configured[64] = {};
    int dev = 0;
    EFA_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        EFA_CUDA(cudaFuncSetAttribute(proj_pair_kernel<OUT_F32, HEADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
        configured[dev] = true;
    }
    dim3 grid(2 * ((args.N + C::BN - 1) / C::BN), (args.M + 2 * PJ_BM - 1) / (2 * PJ_BM));
    EFA_CUDA(launch_early(proj_pair_kernel<OUT_F32, HEADS>, grid, 192, C::SMEM_BYTES, stream, maps, args));
    return 0;
}

// A block per tile, stored row by row from registers with plain stores, which go wherever the kernel may write. Nothing
// promises that for bulk tensor stores: outputs in mapped host memory, managed memory or another GPU's memory take this
// kernel, and launches that are over in one wave (block_per_tile).
struct PjTileArgs {
    void* out;          // fp16 or fp32 [M][N]
    int M, N, K;
    int* status;
    int behind = 0;
};

template <int BN, bool OUT_F32>
__global__ void __launch_bounds__(192)
proj_tile_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmW, const PjTileArgs a)
{
    using C = PjCfg<BN, false>;
    constexpr uint32_t IDESC = idesc_f16_f32(PJ_BM, BN, 0, 1);
    constexpr uint32_t SWZ = swizzle_code(128);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);

    __shared__ __align__(8) uint64_t bar_full[C::NSTAGE];
    __shared__ __align__(8) uint64_t bar_empty[C::NSTAGE];
    __shared__ __align__(8) uint64_t bar_acc;
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_word;

    const int tid  = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int n0 = blockIdx.x * BN;
    const int m0 = blockIdx.y * PJ_BM;
    const int num_k = (a.K + PJ_BK - 1) / PJ_BK;

    if (tid == 0) {
        abort_word = 0;
        for (int s = 0; s < C::NSTAGE; s++) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        mbar_init(&bar_acc, 1);
        mbar_fence_init();
        tma_prefetch_desc(&tmA);
        tma_prefetch_desc(&tmW);
    }
    __syncwarp();
    if (warp == 1) tmem_alloc(&tmem_base_smem, BN);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_acc = tmem_base_smem;
    if (!a.behind) pdl_wait();
    pdl_trigger();

    if (warp == 0) {
        // ---- TMA producer
        if (lane == 0) {
            for (int kb = 0; kb < num_k; kb++) {
                const int s = kb % C::NSTAGE;
                const int use = kb / C::NSTAGE;
                if (use > 0 && !mbar_wait(&bar_empty[s], (uint32_t)((use - 1) & 1), &abort_word, 11)) break;
                uint8_t* sa = smem + s * C::STAGE;
                uint8_t* sb = sa + C::A_BYTES;
                mbar_expect_tx(&bar_full[s], C::STAGE);
                tma_load_2d(sa, &tmA, &bar_full[s], kb * PJ_BK, m0);
                #pragma unroll
                for (int nb = 0; nb < BN / 64; nb++)
                    tma_load_2d(sb + nb * C::B_BOX, &tmW, &bar_full[s], n0 + nb * 64, kb * PJ_BK);
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        if (lane == 0) {
            bool ok = true;
            for (int kb = 0; kb < num_k && ok; kb++) {
                const int s = kb % C::NSTAGE;
                ok = mbar_wait(&bar_full[s], (uint32_t)((kb / C::NSTAGE) & 1), &abort_word, 12);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t sa = smem_u32(smem + s * C::STAGE);
                const uint32_t sb = sa + C::A_BYTES;
                #pragma unroll
                for (int ks = 0; ks < PJ_BK / 16; ks++) {
                    tc_mma_ss(tmem_acc,
                              smem_desc(sa + ks * 32, 16, 1024, SWZ),                    // K-major: 32 B per 16 k
                              smem_desc(sb + ks * 16 * 128, C::B_BOX, 1024, SWZ),        // MN-major: 16 k rows of 128 B
                              IDESC, (kb > 0 || ks > 0) ? 1u : 0u);
                }
                tc_commit(&bar_empty[s]);
            }
            if (ok) tc_commit(&bar_acc);
        }
    } else {
        // ---- epilogue: warps 2..5 own TMEM lanes 32*(warp % 4) .. +31
        const int lane_grp = warp & 3;
        const int row = m0 + lane_grp * 32 + lane;
        if (mbar_wait(&bar_acc, 0, &abort_word, 13)) {
            tc_fence_after_sync();
            const uint32_t taddr = tmem_acc + ((uint32_t)(lane_grp * 32) << 16);
            #pragma unroll 1
            for (int c = 0; c < BN / 32; c++) {
                uint32_t r[32];
                tmem_ld32(taddr + c * 32, r);
                tmem_wait_ld();
                const int col = n0 + c * 32;
                if (OUT_F32) {
                    if (row < a.M && col < a.N) {
                        uint4* dst = reinterpret_cast<uint4*>(static_cast<float*>(a.out) + (size_t)row * a.N + col);
                        #pragma unroll
                        for (int q = 0; q < 8; q++) dst[q] = make_uint4(r[4 * q], r[4 * q + 1], r[4 * q + 2], r[4 * q + 3]);
                    }
                } else if (row < a.M && col < a.N) {   // N is a multiple of 64, so a 32-column chunk is all in or all out
                    uint4* dst = reinterpret_cast<uint4*>(static_cast<__half*>(a.out) + (size_t)row * a.N + col);
                    #pragma unroll
                    for (int q = 0; q < 4; q++) dst[q] = pack8(&r[8 * q]);
                }
            }
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    if (abort_word != 0) {
        for (int i = 0; i < 64; i++) __nanosleep(100000);
        if (tid == 0 && a.status != nullptr) {
            if (atomicCAS(a.status, 0, (int)KS_WAIT_TIMEOUT) == 0) {
                a.status[1] = (int)(blockIdx.y * gridDim.x + blockIdx.x);
                a.status[2] = abort_word;
            }
        }
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem_acc, BN);
    if (a.behind) pdl_wait();
}

template <int BN, bool OUT_F32>
int launch_tile(const CUtensorMap& ta, const CUtensorMap& tw, const PjTileArgs& args, cudaStream_t stream)
{
    using C = PjCfg<BN, false>;
    static bool configured[64] = {};
    int dev = 0;
    EFA_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        EFA_CUDA(cudaFuncSetAttribute(proj_tile_kernel<BN, OUT_F32>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
        configured[dev] = true;
    }
    dim3 grid((args.N + BN - 1) / BN, (args.M + PJ_BM - 1) / PJ_BM);
    EFA_CUDA(launch_early(proj_tile_kernel<BN, OUT_F32>, grid, 192, C::SMEM_BYTES, stream, ta, tw, args));
    return 0;
}

// Few tiles and a long k loop: the tiles leave most SMs idle while each of the others waits for its own copies (about 0.37 us per
// 64 k, whatever the tile's width). A cluster of CTAs shares a 128 x 128 tile, each with its part of k; the partial sums meet in shared
// memory, where every CTA adds its share of the rows over all of them, in rank order in fp32, and stores it:
// 64 x 3776 x 3712 20.8 -> 10.7 us, 128 x 4096 x 4096 22.5 -> 11.5; 1216 x 2752 to Q, K and V of one head of 64 17.4 -> 10.7.
struct PjSplitCfg {
    static constexpr int BN         = 128;
    static constexpr int A_BYTES    = PJ_BM * PJ_BK * 2;
    static constexpr int B_BOX      = PJ_BK * 64 * 2;
    static constexpr int STAGE      = A_BYTES + 2 * B_BOX;        // 32 KB
    static constexpr int NSTAGE     = 6;
    static constexpr int PITCH      = BN + 4;                     // floats between rows of partial sums: 16 bytes off the banks per row
    static constexpr int SMEM_BYTES = STAGE * NSTAGE + 1024;
    static_assert(PJ_BM * PITCH * 4 <= STAGE * NSTAGE, "the partial sums take the ring's place");
};

struct PjSplitArgs {
    void* out[3];       // fp16 [M][N]; HEADS: of Q, K and V [heads][M][d_h]
    int M, N, K;
    int heads, d_h;
    int* status;
};

template <bool HEADS>
__global__ void __launch_bounds__(192)
proj_split_kernel(const __grid_constant__ PjMaps<HEADS ? 3 : 1> maps, const PjSplitArgs a)
{
    using C = PjSplitCfg;
    constexpr uint32_t IDESC = idesc_f16_f32(PJ_BM, C::BN, 0, 1);
    constexpr uint32_t SWZ = swizzle_code(128);

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);

    __shared__ __align__(8) uint64_t bar_full[C::NSTAGE];
    __shared__ __align__(8) uint64_t bar_empty[C::NSTAGE];
    __shared__ __align__(8) uint64_t bar_acc;
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_word;

    const int tid  = threadIdx.x;
    const int warp = tid >> 5;
    const int lane = tid & 31;
    const int rank = (int)cluster_rank(), parts = (int)gridDim.z;  // the cluster is the grid's third dimension
    const int n0 = blockIdx.x * C::BN;
    const int m0 = blockIdx.y * PJ_BM;
    const int all_k = (a.K + PJ_BK - 1) / PJ_BK;
    const int kb0 = rank * all_k / parts, num_k = (rank + 1) * all_k / parts - kb0;       // at least one: parts <= all_k

    // HEADS: tensor, head and column within the head of a column of the whole.
    auto locate = [&](int col, int& t, int& head, int& x) {
        const int h_all = col / a.d_h;
        t = h_all / a.heads;
        head = h_all - t * a.heads;
        x = col - h_all * a.d_h;
    };

    if (tid == 0) {
        abort_word = 0;
        for (int s = 0; s < C::NSTAGE; s++) { mbar_init(&bar_full[s], 1); mbar_init(&bar_empty[s], 1); }
        mbar_init(&bar_acc, 1);
        mbar_fence_init();
        tma_prefetch_desc(&maps.A);
        for (int t = 0; t < (HEADS ? 3 : 1); t++) tma_prefetch_desc(&maps.W[t]);
    }
    __syncwarp();
    if (warp == 1) tmem_alloc(&tmem_base_smem, C::BN);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_acc = tmem_base_smem;
    pdl_wait();
    pdl_trigger();

    if (warp == 0) {
        // ---- TMA producer
        if (lane == 0) {
            int wt[2], wh[2], wx[2];
            if constexpr (HEADS) {
                #pragma unroll
                for (int nb = 0; nb < 2; nb++) locate(min(n0 + nb * 64, a.N - 64), wt[nb], wh[nb], wx[nb]);
            }
            for (int kb = 0; kb < num_k; kb++) {
                const int s = kb % C::NSTAGE;
                const int use = kb / C::NSTAGE;
                if (use > 0 && !mbar_wait(&bar_empty[s], (uint32_t)((use - 1) & 1), &abort_word, 11)) break;
                uint8_t* sa = smem + s * C::STAGE;
                uint8_t* sb = sa + C::A_BYTES;
                mbar_expect_tx(&bar_full[s], C::STAGE);
                tma_load_2d(sa, &maps.A, &bar_full[s], (kb0 + kb) * PJ_BK, m0);
                #pragma unroll
                for (int nb = 0; nb < 2; nb++) {
                    if constexpr (HEADS) tma_load_3d(sb + nb * C::B_BOX, &maps.W[wt[nb]], &bar_full[s], wx[nb], (kb0 + kb) * PJ_BK, wh[nb]);
                    else                 tma_load_2d(sb + nb * C::B_BOX, &maps.W[0], &bar_full[s], n0 + nb * 64, (kb0 + kb) * PJ_BK);
                }
            }
        }
    } else if (warp == 1) {
        // ---- MMA issuer
        if (lane == 0) {
            bool ok = true;
            for (int kb = 0; kb < num_k && ok; kb++) {
                const int s = kb % C::NSTAGE;
                ok = mbar_wait(&bar_full[s], (uint32_t)((kb / C::NSTAGE) & 1), &abort_word, 12);
                if (!ok) break;
                tc_fence_after_sync();
                const uint32_t sa = smem_u32(smem + s * C::STAGE);
                const uint32_t sb = sa + C::A_BYTES;
                #pragma unroll
                for (int ks = 0; ks < PJ_BK / 16; ks++) {
                    tc_mma_ss(tmem_acc,
                              smem_desc(sa + ks * 32, 16, 1024, SWZ),                    // K-major: 32 B per 16 k
                              smem_desc(sb + ks * 16 * 128, C::B_BOX, 1024, SWZ),        // MN-major: 16 k rows of 128 B
                              IDESC, (kb > 0 || ks > 0) ? 1u : 0u);
                }
                tc_commit(&bar_empty[s]);
            }
            if (ok) tc_commit(&bar_acc);
        }
    } else if (__all_sync(0xffffffffu, mbar_wait(&bar_acc, 0, &abort_word, 13))) {
        // ---- warps 2..5 own TMEM lanes 32*(warp % 4) .. +31: a row of partial sums per thread, to where the ring was (the MMAs
        // that read it are complete)
        tc_fence_after_sync();
        const int lane_grp = warp & 3;
        float4* dst = reinterpret_cast<float4*>(reinterpret_cast<float*>(smem) + (lane_grp * 32 + lane) * C::PITCH);
        const uint32_t taddr = tmem_acc + ((uint32_t)(lane_grp * 32) << 16);
        #pragma unroll 1
        for (int c = 0; c < C::BN / 32; c++) {
            uint32_t r[32];
            tmem_ld32(taddr + c * 32, r);
            tmem_wait_ld();
            #pragma unroll
            for (int q = 0; q < 8; q++)
                dst[c * 8 + q] = make_float4(__uint_as_float(r[4 * q]), __uint_as_float(r[4 * q + 1]), __uint_as_float(r[4 * q + 2]), __uint_as_float(r[4 * q + 3]));
        }
    }

    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();                                               // everybody's partial sums are there
    const int share = PJ_BM / parts;                              // parts is 2, 4 or 8
    for (int e = tid; e < share * (C::BN / 4); e += 192) {
        const int r = rank * share + e / (C::BN / 4), c = (e % (C::BN / 4)) * 4;
        const int row = m0 + r, col = n0 + c;
        if (row >= a.M || col >= a.N) continue;
        const uint32_t at = smem_u32(reinterpret_cast<float*>(smem) + r * C::PITCH + c);
        float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int i = 0; i < parts; i++) {
            float4 v;
            uint32_t peer;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(peer) : "r"(at), "r"(i));
            asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer) : "memory");
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        size_t off = (size_t)row * a.N + col;
        int t = 0;
        if constexpr (HEADS) {
            int head, x;
            locate(col, t, head, x);
            off = ((size_t)head * a.M + row) * a.d_h + x;
        }
        *reinterpret_cast<uint2*>(static_cast<__half*>(a.out[t]) + off) = make_uint2(pack_f16x2(sum.x, sum.y), pack_f16x2(sum.z, sum.w));
    }
    __syncwarp();
    cluster_sync();                                               // nobody reads this CTA's memory any more
    if (abort_word != 0) {
        for (int i = 0; i < 64; i++) __nanosleep(100000);
        if (tid == 0 && a.status != nullptr) {
            if (atomicCAS(a.status, 0, (int)KS_WAIT_TIMEOUT) == 0) {
                a.status[1] = (int)(blockIdx.y * gridDim.x + blockIdx.x);
                a.status[2] = abort_word;
            }
        }
        __syncthreads();
    }
    if (warp == 1) tmem_dealloc(tmem_acc, C::BN);
}

template <bool HEADS>
int launch_split(const PjMaps<HEADS ? 3 : 1>& maps, const PjSplitArgs& args, int parts, cudaStream_t stream)
{
    using C = PjSplitCfg;
    static bool configured[64] = {};
    int dev = 0;
    EFA_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && !configured[dev]) {
        EFA_CUDA(cudaFuncSetAttribute(proj_split_kernel<HEADS>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
        configured[dev] = true;
    }
    const dim3 grid((args.N + C::BN - 1) / C::BN, (args.M + PJ_BM - 1) / PJ_BM, parts);
    EFA_CUDA(launch_early_cluster(parts, proj_split_kernel<HEADS>, grid, 192, C::SMEM_BYTES, stream, maps, args));
    return 0;
}

// Tile width: the one that leaves the busiest SM less to fetch. What bounds the kernel is the rate at which tiles come
// from L2 (48 KB per 64 k for a wide tile, 32 KB for a narrow one, 512 and 256 cycles of MMA), so wide tiles count 3, narrow
// ones 2: 4096 x 4096 x 4096 keeps wide tiles although narrow ones would leave the busiest SM fewer columns.
bool wide_tiles(int rows, int cols)
{
    const long row_tiles = (rows + PJ_BM - 1) / PJ_BM;
    const long sms = device_sms();
    auto waves = [&](int bn) { return (row_tiles * ((cols + bn - 1) / bn) + sms - 1) / sms; };
    return waves(256) * 3 <= waves(128) * 2;
}

// A block per tile where one wave of narrow tiles is the whole launch, so that there is nothing to take over, and
// - there are 64 rows: half of every tile's staged stores would be of nothing (64 x 1024 x 1024: 8.7 against 9.5 us), or
// - d is a power of two and d_local at least 512: the 64 rows of a W box then lie a power of two apart and come in slowly,
//   the k loop is the time, and it runs 3 to 6 % faster in the smaller kernel (4416 x 1536 x 512: 13.2 against 13.9 us; where k is not
//   summed in parts, as in the blocks, 256 x 4096 x 1024: 24.5 against 25.9).
// Otherwise the coalesced stores of the other kernel are worth more (2496 x 512 x 576: 7.7 against 8.8 us; 256 x 704 x 2304:
// 8.4 against 9.1), and in more than one wave always. Durations of single launches.
bool block_per_tile(int rows, int d_local, int d)
{
    const long tiles = (long)((rows + PJ_BM - 1) / PJ_BM) * ((d + 127) / 128);
    return tiles <= device_sms() && !wide_tiles(rows, d) && (rows <= 64 || (d_local >= 512 && (d & (d - 1)) == 0));
}

// A pair of CTAs to a tile costs a cluster's start and a hand-over between two SMs per tile, which is worth it where wide tiles are
// and their k loop is long: from d_local 832 on where there are more tiles than pairs of SMs (12224 x 848 x 2688: 55.8 -> 53.7 us, 16384 x
// 1024 x 1024: 33.2 -> 31.5, 25728 x 2864 x 1344: 179 -> 159, but 4160 x 512 x 4096: 20.6 -> 21.2, 9024 x 368 x 1600: 17.2 -> 18.4,
// 29952 x 176 x 1984: 39 -> 50), from 2048 on also with fewer (1024 x 4096 x 4096: 29.9 -> 29.1; 4096 x 1024 x 1024: 10.7 -> 11.2). From 576
// to 832 the gain is 2 to 6 % (16384 x 576 x 4096: 74.1 -> 71.4, 25728 x 720 x 1344: 56.4 -> 52.9, 8192 x 768 x 2048: 26.1 -> 24.7, 8192 x 640 to Q, K and V of eight
// heads of 128: 33.8 -> 32.2) unless the pairs take a round more than single CTAs (4736 x 640 x 4096, five against four: 24.3 -> 26.1).
bool in_pairs(int rows, int d_local, int cols)
{
    const long wide = (cols + 255) / 256, pairs = device_sms() / 2;
    const long tiles = (long)((rows + 255) / 256) * wide, halves = (long)((rows + PJ_BM - 1) / PJ_BM) * wide;
    if (!wide_tiles(rows, cols)) return false;
    if (d_local >= 2048) return rows >= 256;
    if (tiles <= pairs) return false;
    return d_local >= 832 || (d_local >= 576 && (tiles + pairs - 1) / pairs <= (halves + 2 * pairs - 1) / (2 * pairs));
}

// Parts of k for a tile. A cluster and the sum over it cost 2.5 to 3 us, a k-block that an SM has no longer to wait for gives 0.3:
// two parts from 40 k-blocks on (256 x 4096 x 4096: 22.8 -> 17.5 us, but 2048 x 1472 to Q, K and V of one head of 128: 11.3 -> 12.8), four
// from 16 (512 x 1024 x 1024: 8.1 -> 7.6; 512 x 2048 x 1024: 12.8 -> 8.9), while there are SMs for them in clusters (128: a cluster's
// SMs are neighbours, and not every one finds a cluster); eight for at most eight tiles (64 x 2608 x 320: 15.0 -> 7.2; sixteen
// clusters of eight are not on the GPU at a time: 18.6 -> 15.4, the like of it in fours 17.4 -> 10.7). All this on a GPU that is
// otherwise idle. Beside a kernel that holds every SM a cluster waits until its SMs come free together: on a stream of high priority beside
// an attention of 16384 rows, eight heads of 128, 128 x 4096 x 4096 takes 59 us as one CTA per tile, 66 in two parts, 75 in four;
// 64 x 2048 x 1024 29, 39, 45, and 60 in eight. Only the caller knows which it is; the blocks, which do run it so, do not ask for parts.
int k_parts(int rows, int d_local, int cols)
{
    const long tiles = (long)((rows + PJ_BM - 1) / PJ_BM) * ((cols + 127) / 128);
    const int num_k = (d_local + PJ_BK - 1) / PJ_BK;
    const long clustered = device_sms() * 128l / 148;
    if (tiles <= 8 && num_k >= 32) return 8;
    if (tiles * 4 <= clustered && num_k >= 16) return 4;
    if (tiles * 2 <= clustered && num_k >= 40) return 2;
    return 1;
}

int check_shape(int rows, int d_local, int d)
{
    if (rows <= 0 || rows % 64 != 0) { set_error("project: rows (%d) must be a positive multiple of 64", rows); return 2; }
    if (d_local <= 0 || d_local % 16 != 0) { set_error("project: d_local (%d) must be a positive multiple of 16", d_local); return 2; }
    if (d <= 0 || d % 64 != 0) { set_error("project: d (%d) must be a positive multiple of 64", d); return 2; }
    return 0;
}

int input_map(CUtensorMap* out, const void* A, int rows, int k)
{
    unsigned long long dims[2] = {(unsigned long long)k, (unsigned long long)rows};
    unsigned long long strides[1] = {(unsigned long long)k * 2ull};
    unsigned box[2] = {64u, 128u};
    return make_tmap_f16(out, A, 2, dims, strides, box);
}

}  // namespace

int project_f16(const void* A, const void* W, void* out, int rows, int d_local, int d, cudaStream_t stream, int out_dtype, bool own_out, bool behind, bool beside, bool in_parts)
{
    if (out_dtype != EFA_F16 && out_dtype != EFA_F32) { set_error("project: unknown output type %d", out_dtype); return 2; }
    if (int rc = check_shape(rows, d_local, d)) return rc;
    if (!A || !W || !out) { set_error("project: null pointer"); return 2; }

    PjMaps<1> maps;
    if (input_map(&maps.A, A, rows, d_local)) return 1;
    {
        unsigned long long dims[2] = {(unsigned long long)d, (unsigned long long)d_local};
        unsigned long long strides[1] = {(unsigned long long)d * 2ull};
        unsigned box[2] = {64u, 64u};
        if (make_tmap_f16(&maps.W[0], W, 2, dims, strides, box)) return 1;
    }
    const bool f32 = out_dtype == EFA_F32, wide = wide_tiles(rows, d);
    if (const int parts = in_parts && !f32 ? k_parts(rows, d_local, d) : 1; parts > 1) {
        if (((uintptr_t)out & 15) != 0) { set_error("project: output address not 16-byte aligned"); return 1; }
        const PjSplitArgs a{{out, nullptr, nullptr}, rows, d, d_local, 1, d, kernel_status_word()};
        return launch_split<false>(maps, a, parts, stream);
    }
    if (block_per_tile(rows, d_local, d) || (!own_out && !own_device_memory(out))) {
        if (((uintptr_t)out & 15) != 0) { set_error("project: output address not 16-byte aligned"); return 1; }
        const PjTileArgs a{out, rows, d, d_local, kernel_status_word(), behind};
        if (f32) return launch_tile<128, true>(maps.A, maps.W[0], a, stream);
        return wide ? launch_tile<256, false>(maps.A, maps.W[0], a, stream) : launch_tile<128, false>(maps.A, maps.W[0], a, stream);
    }
    unsigned long long dims[2] = {(unsigned long long)d, (unsigned long long)rows};
    unsigned long long strides[1] = {(unsigned long long)d * (f32 ? 4ull : 2ull)};
    unsigned box[2] = {f32 ? 32u : 64u, 32u};
    if (f32 ? make_tmap_f32(&maps.out[0], out, 2, dims, strides, box) : make_tmap_f16(&maps.out[0], out, 2, dims, strides, box)) return 1;
    const PjArgs a{rows, d, d_local, 1, d, kernel_status_word(), behind};
    if (!beside && in_pairs(rows, d_local, d)) return f32 ? launch_pair<true, false>(maps, a, stream) : launch_pair<false, false>(maps, a, stream);
    if (f32) return wide ? launch_proj<256, true, false>(maps, a, stream) : launch_proj<128, true, false>(maps, a, stream);
    return wide ? launch_proj<256, false, false>(maps, a, stream) : launch_proj<128, false, false>(maps, a, stream);
}

int project_heads_f16(const void* X, const void* const W[3], void* const out[3], int rows, int d, int heads, int d_h,
                      cudaStream_t stream)
{
    if (int rc = check_shape(rows, d, d_h)) return rc;
    if ((long)3 * heads * d_h > 0x7fffff00l) { set_error("project: %d heads of %d are too many columns", heads, d_h); return 2; }
    const int cols = 3 * heads * d_h;
    const int parts = k_parts(rows, d, cols);
    // The clusters along k write with plain stores, which go anywhere: whether k is summed in parts does not depend on the memory.
    if (parts == 1 && (!own_device_memory(out[0]) || !own_device_memory(out[1]) || !own_device_memory(out[2]))) {
        // where the staged stores cannot go: head by head
        for (int h = 0; h < heads; h++)
            for (int t = 0; t < 3; t++)
                if (int rc = project_f16(X, static_cast<const __half*>(W[t]) + (size_t)h * d * d_h,
                                         static_cast<__half*>(out[t]) + (size_t)h * rows * d_h, rows, d, d_h, stream))
                    return rc;
        return 0;
    }
    PjMaps<3> maps;
    if (input_map(&maps.A, X, rows, d)) return 1;
    for (int t = 0; t < 3; t++) {
        // three dimensions, so that rows past d read as zero and not as the next head's
        unsigned long long wdims[3] = {(unsigned long long)d_h, (unsigned long long)d, (unsigned long long)heads};
        unsigned long long wstrides[2] = {(unsigned long long)d_h * 2ull, (unsigned long long)d * d_h * 2ull};
        unsigned wbox[3] = {64u, 64u, 1u};
        if (make_tmap_f16(&maps.W[t], W[t], 3, wdims, wstrides, wbox)) return 1;
        if (((uintptr_t)out[t] & 15) != 0) { set_error("project: output address not 16-byte aligned"); return 1; }
        if (parts > 1) continue;
        unsigned long long odims[3] = {(unsigned long long)d_h, (unsigned long long)rows, (unsigned long long)heads};
        unsigned long long ostrides[2] = {(unsigned long long)d_h * 2ull, (unsigned long long)rows * d_h * 2ull};
        unsigned obox[3] = {64u, 32u, 1u};
        if (make_tmap_f16(&maps.out[t], out[t], 3, odims, ostrides, obox)) return 1;
    }
    if (parts > 1) {
        const PjSplitArgs s{{out[0], out[1], out[2]}, rows, cols, d, heads, d_h, kernel_status_word()};
        return launch_split<true>(maps, s, parts, stream);
    }
    PjArgs a{rows, cols, d, heads, d_h, kernel_status_word()};
    if (in_pairs(rows, d, cols)) return launch_pair<false, true>(maps, a, stream);
    return wide_tiles(rows, cols) ? launch_proj<256, false, true>(maps, a, stream) : launch_proj<128, false, true>(maps, a, stream);
}


namespace {
template <class K> int touch_kernel(K kernel)
{
    cudaFuncAttributes attr;
    EFA_CUDA(cudaFuncGetAttributes(&attr, kernel));
    return 0;
}
}  // namespace

int proj_preload()
{
    return touch_kernel(proj_gemm_kernel<128, false, false>) || touch_kernel(proj_gemm_kernel<128, true, false>) ||
           touch_kernel(proj_gemm_kernel<256, false, false>) || touch_kernel(proj_gemm_kernel<256, true, false>) ||
           touch_kernel(proj_gemm_kernel<128, false, true>) || touch_kernel(proj_gemm_kernel<256, false, true>) ||
           touch_kernel(proj_pair_kernel<false, false>) || touch_kernel(proj_pair_kernel<true, false>) || touch_kernel(proj_pair_kernel<false, true>) ||
           touch_kernel(proj_split_kernel<false>) || touch_kernel(proj_split_kernel<true>) ||
           touch_kernel(proj_tile_kernel<128, false>) || touch_kernel(proj_tile_kernel<128, true>) ||
           touch_kernel(proj_tile_kernel<256, false>);
}

}  // namespace efa
