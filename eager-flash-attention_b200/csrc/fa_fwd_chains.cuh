// The attention kernel for d_h 16, 32 and 64, where the exponentials are the work: four chains S -> softmax -> P -> P*V -> Q*K^T -> S to
// an SM. Included by fa_fwd_ws_sm100.cu, which describes what both kernels have in common, and launches them.
//
// One CTA = 768 threads:
//   warps 0-15   softmax of chain 0 to 3, four warps each (one thread per row; 104 registers)
//   warps 16-19  tcgen05.mma issuer of each chain (one elected lane), which also gives back its K/V slots
//   warp  20     TMA producer; warp 21 owns the tensor memory; 22 and 23 only complete their warpgroup
// A chain takes 64 keys of a 128-key stage at a time, with offset, maximum, sum and O of its own; the chains of a tile are merged at the end,
// straight from tensor memory (all of them see the same lanes). WAYS = 2: 256 rows, two chains to each 128-row tile, one for the lower
// and one for the upper half of every stage. WAYS = 4: 128 rows, chains 0 and 1 take the even stages, 2 and 3 the odd ones.
// Tensor memory (512 columns): S of chain c [64c, 64c + 64), P in its lower half; O [256 + 64c, + D).
//
// What bounds it: the special-function unit, 16 exponentials per clock and SM (2048 cycles for 256 rows x 128 keys). Two warps to a scheduler, one
// per tile, left it idle a quarter of the time, with or without Q*K^T a stage ahead (2650 to 2750 cycles, and 2600 with the MMAs cut to one
// k-step: what they wait for is themselves). With four there is nearly always one in its exponentials: 2410 cycles. A chain then waits
// about 700 of them for its own MMAs (hand-over, P*V and Q*K^T behind the other chains', commit), which nothing needs to hide further:
// Q*K^T ahead with P in columns of its own (d_h 16 and 32, where they fit) costs a wait and a commit per block more and is 5 % slower. Every
// eighth pair of exponentials is a polynomial (none: +3 to +7 %, a fourth: +5 %, a sixteenth: +1 %). An issuer for two chains is 3 to 6 %
// slower; slots given back by a softmax warp instead of the issuer 1 to 3 % (it is what the other three of its chain wait for).
// us, two 128-key chains to an SM -> this: S=4096, 16 heads of 64 104 -> 94, causal 53.8 -> 50.9; S=16384 causal 720 -> 665; S=65536, two heads of
// 64 2710 -> 2594 (power: 1.75 GHz); S=4032, eight heads of 32 54.3 -> 49.0; S=16384, 16 heads of 32 1326 -> 1200, four heads of 16 374 -> 323;
// S=1024, eight heads of 64 (128-row items) 10.7 -> 9.5. One tile of 128 rows without a workspace (offset = maximum, so O is rescaled
// more often) 27.2 -> 23.1 in eight splits with the merge, 110 -> 100 in one.
#pragma once

template <int D, int WAYS>
struct ChainCfg {
    static constexpr int SWB        = D >= 64 ? 128 : D * 2;      // swizzle width = TMA box row, bytes
    static constexpr int TILE_BYTES = 128 * D * 2;
    static constexpr int TILES      = 4 / WAYS;
    // K slots and V slots of 128 keys. Four chains on one tile of 64 take a stage in 0.7 us and give V back a stage of theirs after K; with four slots it is asked
    // for too late where keys come from memory. 13952 rows, four heads, inputs in turn / behind a flush of the L2 (us): two chains 282 / 316, 4 + 4 slots 290 / 329,
    // 6 + 4 286 / 317, 4 + 6 265 / 292, 6 + 6 256 / 283; but of launches between other kernels, 768 rows, two heads behind a fill 12.8, 12.8, 12.8, 12.8, 13.6, and one
    // tile in eight splits with its merge 28.2, 24.7, 25.3, 24.6, 25.3. 256-row items have no room for six and lose nothing with four.
    static constexpr int NSK        = 4;
    static constexpr int NSV        = D == 64 && WAYS == 4 ? 6 : 4;
    static constexpr int SMEM_BYTES = TILE_BYTES * (TILES + NSK + NSV) + 1024;
    static constexpr int USERS      = 2 * TILES;                  // chains that read a slot: each takes 64 of its keys
    static_assert(D <= 64 && NSK % 2 == 0 && NSV % 2 == 0, "a chain that takes every second stage would skip phases of a slot");
};
constexpr int CH_THREADS = 768;

template <int D, bool OUT_F16, int WAYS>
__global__ void __launch_bounds__(CH_THREADS, 1)
fa_fwd_chains_kernel(const __grid_constant__ CUtensorMap tmQ,
                     const __grid_constant__ CUtensorMap tmK,
                     const __grid_constant__ CUtensorMap tmV,
                     const FaArgs a, int items_x, int items_total)
{
    using C = ChainCfg<D, WAYS>;
    constexpr int TILES = C::TILES, NSK = C::NSK, NSV = C::NSV, ITEM_ROWS = TILES * WS_BM;
    constexpr uint32_t SWZ = swizzle_code(C::SWB);
    constexpr uint32_t IDESC_QK = idesc_f16_f32(WS_BM, 64, 0, 0);
    constexpr uint32_t IDESC_PV = idesc_f16_f32(WS_BM, D, 0, 1);
    // Where O is rescaled: behind the first half's exponentials at d_h 64 (S=4096, 16 heads 99.9 -> 93.9 us: the vote's latency is hidden), ahead of them for
    // small heads, where it happens at every new maximum (four heads of 16 323 against 335, eight of 32 the same).
    constexpr bool LATE = D == 64;

    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    uint8_t* sQ = smem;                                   // TILES tiles
    uint8_t* sK = sQ + TILES * C::TILE_BYTES;             // NSK stages
    uint8_t* sV = sK + NSK * C::TILE_BYTES;               // NSV stages

    __shared__ __align__(8) uint64_t q_full[TILES];
    __shared__ __align__(8) uint64_t k_full[NSK], k_empty[NSK], v_full[NSV], v_empty[NSV];
    __shared__ __align__(8) uint64_t s_full[4], p_full[4], o_done[4];
    __shared__ float ends[4][3][WS_BM];                   // offset, maximum and sum of every chain's rows
    __shared__ uint32_t tmem_base_smem;
    __shared__ int abort_word;
    __shared__ int half_done[TILES][2];
    __shared__ int s_head, s_split, s_row0;

    const int tid  = threadIdx.x;
    const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int lane = tid & 31;
    const bool tail = WAYS == 4 && a.tail_first >= 0;     // the rest of the launch before this one: no need to wait for that

    if (tid == 0) {
        abort_word = 0;
        for (int t = 0; t < TILES; t++) { mbar_init(&q_full[t], 1); half_done[t][0] = half_done[t][1] = 0; }
        for (int s = 0; s < NSK; s++) { mbar_init(&k_full[s], 1); mbar_init(&k_empty[s], C::USERS); }
        for (int s = 0; s < NSV; s++) { mbar_init(&v_full[s], 1); mbar_init(&v_empty[s], C::USERS); }
        for (int c = 0; c < 4; c++) { mbar_init(&s_full[c], 1); mbar_init(&p_full[c], WS_BM / 32); mbar_init(&o_done[c], 1); }
        mbar_fence_init();
        tma_prefetch_desc(&tmQ);
        tma_prefetch_desc(&tmK);
        tma_prefetch_desc(&tmV);
    }
    if (tid == 32) {                                       // reads an order table: a launch with one does not start early
        int head, split, row0;
        pick_item((int)(blockIdx.y * gridDim.x + blockIdx.x), a, items_x, items_total, ITEM_ROWS, tail, head, split, row0);
        s_head = head;
        s_split = split;
        s_row0 = row0;
    }
    if (warp == 21) tmem_alloc(&tmem_base_smem, 512);
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, tmem_base_smem, 0);
    if (!tail) pdl_wait();
    pdl_trigger();

    const int block_row0 = __shfl_sync(0xffffffffu, s_row0, 0);
    const int kv_lo = __shfl_sync(0xffffffffu, s_split, 0) * a.kv_len, kv_hi = kv_lo + a.kv_len;
    const int rows_valid = min(ITEM_ROWS, a.q_rows - block_row0);             // 64 to 256 (in a tail also none)
    auto abs0 = [&](int t) { return a.q_start + block_row0 + t * WS_BM; };
    auto rows_of = [&](int t) { return max(0, min(WS_BM, rows_valid - t * WS_BM)); };
    // Blocks of 64 keys that a tile sweeps; block b is half b & 1 of stage b / 2 and belongs to chain b % WAYS of the tile.
    auto blocks_of = [&](int t) {
        const int rows = rows_of(t), end = a.causal ? min(kv_hi, abs0(t) + rows) : kv_hi;
        return rows > 0 && end > kv_lo ? (end - kv_lo + 63) >> 6 : 0;
    };
    auto stage_of = [&](int way, int i) { return WAYS == 2 ? i : 2 * i + (way >> 1); };

    if (warp >= 20) {
        setmaxnreg_dec_24();
        if (warp == 20 && lane == 0) {
            // ---- TMA producer
            const int head = s_head;
            auto load = [&](uint8_t* dst, const CUtensorMap* tm, uint64_t* bar, int row) {
                mbar_expect_tx(bar, C::TILE_BYTES);
                tma_load_3d(dst, tm, bar, 0, row, head);
            };
            int n[TILES], most = 0;
            #pragma unroll
            for (int t = 0; t < TILES; t++) {
                n[t] = blocks_of(t);
                most = max(most, n[t]);
                if (n[t] > 0) load(sQ + t * C::TILE_BYTES, &tmQ, &q_full[t], abs0(t));
            }
            for (int j = 0; 2 * j < most; j++) {
                const int s = j % NSK, u = j / NSK, sv = j % NSV, uv = j / NSV;
                if (u > 0 && !mbar_wait(&k_empty[s], (uint32_t)((u - 1) & 1), &abort_word, 21)) break;
                load(sK + s * C::TILE_BYTES, &tmK, &k_full[s], kv_lo + j * WS_BN);
                if (uv > 0 && !mbar_wait(&v_empty[sv], (uint32_t)((uv - 1) & 1), &abort_word, 22)) break;
                load(sV + sv * C::TILE_BYTES, &tmV, &v_full[sv], kv_lo + j * WS_BN);
                int users = 0;
                #pragma unroll
                for (int t = 0; t < TILES; t++) users += max(0, min(2, n[t] - 2 * j));
                for (; users < C::USERS; users++) {           // for chains that end before this stage
                    mbar_arrive(&k_empty[s]);
                    mbar_arrive(&v_empty[sv]);
                }
            }
        }
    } else if (warp >= 16) {
        setmaxnreg_dec_40();
        // ---- MMA issuers, one to a chain. The whole warp runs the loop, one elected lane issues.
        const int c = warp - 16, tile = c / WAYS, way = c % WAYS;
        const uint64_t dq = smem_desc(smem_u32(sQ), 16, 8 * C::SWB, SWZ);
        const uint64_t dk = smem_desc(smem_u32(sK), 16, 8 * C::SWB, SWZ);
        const uint64_t dv = smem_desc(smem_u32(sV), 128 * C::SWB, 8 * C::SWB, SWZ);
        constexpr uint32_t HALF = (64 * C::SWB) >> 4;             // 64 keys further
        const uint32_t dq_lo = (uint32_t)dq + tile * (C::TILE_BYTES >> 4), dq_hi = (uint32_t)(dq >> 32);
        const uint32_t dk_lo = (uint32_t)dk + (way & 1) * HALF, dk_hi = (uint32_t)(dk >> 32);
        const uint32_t dv_lo = (uint32_t)dv + (way & 1) * HALF, dv_hi = (uint32_t)(dv >> 32);
        const uint32_t tS = tmem_base + c * 64, tO = tmem_base + 256 + c * 64;
        auto wait = [&](uint64_t* bar, int phase, int site) -> bool {
            return __all_sync(0xffffffffu, mbar_wait(bar, (uint32_t)(phase & 1), &abort_word, site));
        };
        auto issue_qk = [&](int slot) {
            #pragma unroll
            for (int ks = 0; ks < D / 16; ks++)
                tc_mma_ss_lh(tS, dq_lo + ks * 2, dq_hi, dk_lo + slot * (C::TILE_BYTES >> 4) + ks * 2, dk_hi, IDESC_QK, ks > 0 ? 1u : 0u);
            tc_commit(&s_full[c]);
        };
        // S(i) complete: so is what was issued before, QK(i) and PV(i-1). Here and not in the softmax warps, which are what a chain waits for.
        auto give_back = [&](int i) -> bool {
            if (!wait(&s_full[c], i, 22)) return false;
            if (lane == 0) {
                mbar_arrive(&k_empty[stage_of(way, i) % NSK]);
                if (i > 0) mbar_arrive(&v_empty[stage_of(way, i - 1) % NSV]);
            }
            __syncwarp();
            return true;
        };
        const int n = (blocks_of(tile) - way + WAYS - 1) / WAYS;
        bool ok = n > 0 && wait(&q_full[tile], 0, 24);
        if (ok) {
            const int j = stage_of(way, 0);
            ok = wait(&k_full[j % NSK], j / NSK, 27);
            tc_fence_after_sync();
            if (ok && elect_one()) issue_qk(j % NSK);
            __syncwarp();
        }
        for (int i = 0; i < n && ok; i++) {
            const int j = stage_of(way, i), next = stage_of(way, i + 1);
            const bool more = i + 1 < n;
            ok = give_back(i) && wait(&v_full[j % NSV], j / NSV, 25) && (!more || wait(&k_full[next % NSK], next / NSK, 28)) && wait(&p_full[c], i, 26);
            tc_fence_after_sync();
            if (!ok) break;
            if (elect_one()) {
                #pragma unroll
                for (int ks = 0; ks < 4; ks++)
                    tc_mma_ts_lh(tO, tS + ks * 8, dv_lo + (j % NSV) * (C::TILE_BYTES >> 4) + ((ks * 16 * C::SWB) >> 4), dv_hi, IDESC_PV, ks > 0 || i > 0 ? 1u : 0u);
                if (more) issue_qk(next % NSK); else tc_commit(&o_done[c]);
            }
            __syncwarp();
        }
    } else {
        setmaxnreg_inc_104();
        // =====================================================================================
        // Softmax: chain c = warp / 4, row = thread index within the warpgroup
        // =====================================================================================
        const int c = warp >> 2, tile = c / WAYS, way = c % WAYS;
        const int row = tid & (WS_BM - 1);
        const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
        const uint32_t tmem_S = tmem_base + c * 64 + lane_base;
        const uint32_t tmem_O = tmem_base + 256 + c * 64 + lane_base;
        const int blocks = blocks_of(tile);
        const int n = (blocks - way + WAYS - 1) / WAYS;
        const int my_abs0 = abs0(tile);

        float m_ref = kNegInfW;     // exponent offset in use (a past row maximum), scaled by scale*log2(e)
        float m_true = kNegInfW;    // true running row maximum, same scaling
        float l_run = 0.f;          // running denominator relative to m_ref
        bool ok = true;

        for (int i = 0; i < n; i++) {
            const int kb = kv_lo + (i * WAYS + way) * 64;
            ok = __all_sync(0xffffffffu, mbar_wait(&s_full[c], (uint32_t)(i & 1), &abort_word, 31));
            if (!ok) break;
            tc_fence_after_sync();
            uint32_t su[2][32];
            tmem_ld32(tmem_S, su[0]);
            tmem_ld32(tmem_S + 32, su[1]);
            tmem_wait_ld();

            if (kb + 64 > kv_hi || (a.causal && kb + 63 > my_abs0)) {
                int lim = kv_hi - 1 - kb;
                if (a.causal) lim = min(lim, my_abs0 + row - kb);
                #pragma unroll
                for (int h = 0; h < 2; h++)
                    #pragma unroll
                    for (int k = 0; k < 32; k++)
                        if (h * 32 + k > lim) su[h][k] = 0xff800000u;
            }

            float mx0 = kNegInfW, mx1 = kNegInfW, mx2 = kNegInfW, mx3 = kNegInfW;
            #pragma unroll
            for (int k = 0; k < 16; k += 2) {
                mx0 = max3(mx0, __uint_as_float(su[0][k]), __uint_as_float(su[0][k + 1]));
                mx1 = max3(mx1, __uint_as_float(su[0][16 + k]), __uint_as_float(su[0][17 + k]));
                mx2 = max3(mx2, __uint_as_float(su[1][k]), __uint_as_float(su[1][k + 1]));
                mx3 = max3(mx3, __uint_as_float(su[1][16 + k]), __uint_as_float(su[1][17 + k]));
            }
            m_true = fmaxf(m_true, fmaxf(max3(mx0, mx1, mx2), mx3) * a.scale_log2e);

            // Move the exponent offset only when the maximum grew by more than the threshold.
            float alpha = 1.f;
            if (m_true - m_ref > a.rescale_above || m_ref == kNegInfW) {     // (-inf) - (-inf) is NaN: second test
                const float m_use = (m_true == kNegInfW) ? 0.f : m_true;
                alpha = (m_ref == kNegInfW) ? 0.f : ex2(m_ref - m_use);
                m_ref = m_true;
            }
            const float m_off = (m_ref == kNegInfW) ? 0.f : m_ref;
            const uint64_t scale2 = pack2(a.scale_log2e, a.scale_log2e), off2 = pack2(-m_off, -m_off);
            uint64_t psum2[2] = {pack2(0.f, 0.f), pack2(0.f, 0.f)};
            // Complete with S(i): PV(i-1), so O may be rescaled and P take the place of S.
            auto rescale = [&]() {
                if (i == 0 || !__any_sync(0xffffffffu, alpha != 1.f)) return;
                constexpr int PART = D < 32 ? D : 32;
                #pragma unroll 1
                for (int x = 0; x < D; x += PART) {
                    uint32_t o[PART];
                    if constexpr (PART == 32) tmem_ld32(tmem_O + x, o); else tmem_ld16(tmem_O + x, o);
                    tmem_wait_ld();
                    #pragma unroll
                    for (int k = 0; k < PART; k++) o[k] = __float_as_uint(__uint_as_float(o[k]) * alpha);
                    if constexpr (PART == 32) tmem_st32(tmem_O + x, o); else tmem_st16(tmem_O + x, o);
                }
            };
            if constexpr (!LATE) rescale();
            #pragma unroll
            for (int h = 0; h < 2; h++) {
                uint32_t pk[16];
                #pragma unroll
                for (int k = 0; k < 16; k++) {
                    const uint64_t x = fma2(pack2(__uint_as_float(su[h][2 * k]), __uint_as_float(su[h][2 * k + 1])), scale2, off2);
                    float p0, p1;
                    if (k % 8 == 7) {
                        unpack2(exp2_poly2(x), p0, p1);
                    } else {
                        unpack2(x, p0, p1);
                        p0 = ex2(p0);
                        p1 = ex2(p1);
                    }
                    psum2[k & 1] = add2(psum2[k & 1], pack2(p0, p1));
                    pk[k] = pack_f16x2(p0, p1);
                }
                if constexpr (LATE) { if (h == 0) rescale(); }
                tmem_st16(tmem_S + h * 16, pk);
            }
            tmem_wait_st();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&p_full[c]);
            float s0, s1, s2, s3;
            unpack2(psum2[0], s0, s1);
            unpack2(psum2[1], s2, s3);
            l_run = l_run * alpha + ((s0 + s2) + (s1 + s3));
        }
        if (ok && n > 0) {
            ok = __all_sync(0xffffffffu, mbar_wait(&o_done[c], 0u, &abort_word, 32));
            tc_fence_after_sync();
        }

        // ---- the chains of a tile learn each other's offset, maximum and sum; each then merges and stores its share of the columns
        ends[c][0][row] = m_ref; ends[c][1][row] = m_true; ends[c][2][row] = l_run;
        tc_fence_before_sync();
        asm volatile("bar.sync %0, %1;" :: "r"(1 + tile), "n"(WAYS * WS_BM) : "memory");
        tc_fence_after_sync();
        ok = __all_sync(0xffffffffu, ok && *(volatile int*)&abort_word == 0);
        float w[WAYS];
        {
            float top = kNegInfW;
            #pragma unroll
            for (int k = 0; k < WAYS; k++) {
                top = fmaxf(top, ends[tile * WAYS + k][0][row]);
                m_true = fmaxf(m_true, ends[tile * WAYS + k][1][row]);
            }
            l_run = 0.f;
            #pragma unroll
            for (int k = 0; k < WAYS; k++) {
                const float m = ends[tile * WAYS + k][0][row];
                w[k] = (m == kNegInfW) ? 0.f : ex2(m - top);
                l_run += w[k] * ends[tile * WAYS + k][2][row];
            }
            m_ref = top;
        }
        constexpr int PER = D / WAYS < 16 ? 16 : D / WAYS;        // columns; with few of them some chains have none
        const int c_lo = way * PER;

        // ---- epilogue: this thread's row (warps take this branch as a whole: rows are 0, 64 or 128)
        if (ok && (warp & 3) * 32 < rows_of(tile)) {
            const int head = s_head, split = s_split;
            const size_t ld_o = (size_t)a.H_local * D;
            const size_t orow = (size_t)block_row0 + tile * WS_BM + row;
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
                if (way == 0) {
                    a.m_part[s0] = m_true;
                    a.l_part[s0] = partial_sum(l_run * mult, !a.causal || split * a.kv_len <= a.q_start + (int)orow);
                }
            }
            if (c_lo < D) {
                #pragma unroll 1
                for (int x = c_lo; x < c_lo + PER; x += 16) {
                    uint32_t o[16];
                    #pragma unroll
                    for (int k = 0; k < 16; k++) o[k] = 0u;
                    #pragma unroll
                    for (int k = 0; k < WAYS; k++) {
                        if (k >= blocks) break;                   // that chain has not run
                        uint32_t part[16];
                        tmem_ld16(tmem_base + 256 + (tile * WAYS + k) * 64 + lane_base + x, part);
                        tmem_wait_ld();
                        #pragma unroll
                        for (int e = 0; e < 16; e++) o[e] = __float_as_uint(__uint_as_float(o[e]) + __uint_as_float(part[e]) * w[k]);
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
                        uint4* d = reinterpret_cast<uint4*>(dst16 + x);
                        d[0] = v0;
                        d[1] = v1;
                    } else {
                        float4* d = reinterpret_cast<float4*>(dst32 + x);
                        #pragma unroll
                        for (int qd = 0; qd < 4; qd++)
                            d[qd] = make_float4(__uint_as_float(o[4 * qd]) * mult, __uint_as_float(o[4 * qd + 1]) * mult,
                                                __uint_as_float(o[4 * qd + 2]) * mult, __uint_as_float(o[4 * qd + 3]) * mult);
                    }
                }
            }

            // ---- completion signal: one count per finished 64-row block, after its rows are visible.
            // A 64-row block is two warps of each chain; the last of them to get here publishes the count.
            if (a.tile_counters != nullptr) {
                if (a.counters_sys) __threadfence_system(); else __threadfence();
                __syncwarp();
                if (lane == 0) {
                    const int half = (warp & 3) >> 1;
                    if (atomicAdd(&half_done[tile][half], 1) == 2 * WAYS - 1) {
                        if (a.counters_sys) __threadfence_system(); else __threadfence();
                        atomicAdd(a.tile_counters + (block_row0 + tile * WS_BM + half * 64) / a.tile_rows, 1);
                    }
                }
            }
        }
    }
    __syncwarp();
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();

    // ---- teardown
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
    if (warp == 21) tmem_dealloc(tmem_base, 512);
    if (tail) pdl_wait();
}
