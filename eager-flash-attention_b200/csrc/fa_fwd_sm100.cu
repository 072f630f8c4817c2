// The attention launch interface (flash_attn_tc_forward of eager-flash-attention, flash_attn_tc.cu:363-399): argument
// checks, tensor maps, the merge of split-KV partials and the entry that allocates nothing. The kernels are in fa_fwd_ws_sm100.cu
// (d_h 128), fa_fwd_chains.cuh (16 to 64) and fa_fwd_tile_sm100.cu (16 and 32, few keys); attention_plan.h says which launch goes as what.
#include "fa_fwd_sm100.cuh"
#include "fa_args.cuh"
#include "host_util.h"
#include "sm100_ptx.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <map>
#include <mutex>
#include <tuple>

namespace efa {

namespace {

// Merge of the split-KV partials (the job of combine_kernel, flash_attn_tc.cu:319-349):
//     O = sum_i w_i O_i / sum_i w_i l_i,   w_i = 2^(m_i - max_k m_k).
// A block takes `per_block` rows. First the normalised weights w_i / sum_k w_k l_k are computed once per (row, head)
// into shared memory; then every thread merges 16-byte column chunks with them, so the row maxima and
// denominators are read and exponentiated once per head and row, not once per output element. HBM-bound:
// (split + 1/2 or 1) * rows * d_local * 4 bytes. With few rows it is a chain of loads that counts: up to CB_ROWS rows to a
// block, but no more than leave two blocks to every SM (128 rows of 16 heads of 64 in eight splits: 24 us as 16 blocks of eight
// rows; attention and merge together 42.4 us so, 29.1 as blocks of one row), and all splits of an element are asked for at once (2, 3, 4 or 8
// of them, else four at a time; one after another 29.0 us, so 26.9). Splits that the mask leaves nothing of are not read: 16384 rows, four heads of 64, causal, four
// splits 203.3 -> 196.8 us with the attention; 4096 rows, 16 heads of 64 in two splits 129.9 -> 123.0. The partials are written while this kernel may already be
// on the GPU (launch_early): the pointers promise nothing, and the loads are ordinary ones, past L1 for what is read once.
constexpr int CB_ROWS = 8;

template <bool OUT_F16, int SPLIT /* 0: any */>
__global__ void __launch_bounds__(256)
combine_splits_kernel(const float* O_part, const float* m_part, const float* l_part, void* O,
                      int row0, int rows, int ws_rows, int d_local, int H_local, int d_h, int split_any, int per_block)
{
    extern __shared__ float weight[];                       // [per_block][H_local][split]
    const int split = SPLIT > 0 ? SPLIT : split_any;
    pdl_wait();
    pdl_trigger();
    const int first = blockIdx.x * per_block;
    const int nrows = min(per_block, rows - first);

    for (int e = threadIdx.x; e < nrows * H_local; e += blockDim.x) {
        const int rr = e / H_local, head = e - rr * H_local;
        const size_t base = (size_t)(row0 + first + rr) * H_local + head;
        const size_t step = (size_t)ws_rows * H_local;      // distance between splits
        float top = -INFINITY, denom = 0.f;
        float* w = weight + (size_t)e * split;
        // An empty split (the mask leaves nothing of it, partial_sum) gets -0 as its weight, and is not read below.
        if constexpr (SPLIT > 0) {
            float m[SPLIT], l[SPLIT];
            #pragma unroll
            for (int i = 0; i < SPLIT; i++) { m[i] = __ldcg(m_part + base + i * step); l[i] = __ldcg(l_part + base + i * step); }
            #pragma unroll
            for (int i = 0; i < SPLIT; i++) top = fmaxf(top, m[i]);
            #pragma unroll
            for (int i = 0; i < SPLIT; i++) {
                const float x = exp2f(m[i] - top);
                denom += x * l[i];
                m[i] = no_keys(m[i], l[i]) ? -0.f : x;
            }
            const float inv = 1.f / denom;
            #pragma unroll
            for (int i = 0; i < SPLIT; i++) w[i] = m[i] * inv;
        } else {
            for (int i = 0; i < split; i++) top = fmaxf(top, m_part[base + i * step]);
            for (int i = 0; i < split; i++) {
                const float m = m_part[base + i * step], l = l_part[base + i * step], x = exp2f(m - top);
                denom += x * l;
                w[i] = no_keys(m, l) ? -0.f : x;
            }
            const float inv = 1.f / denom;
            for (int i = 0; i < split; i++) w[i] *= inv;
        }
    }
    __syncthreads();

    const int chunks = d_local / 4;                         // float4 chunks per row (d_h is a multiple of 16)
    for (int e = threadIdx.x; e < nrows * chunks; e += blockDim.x) {
        const int rr = e / chunks, c = e - rr * chunks;
        const int head = (c * 4) / d_h;
        const float* w = weight + ((size_t)rr * H_local + head) * split;
        const float4* src = reinterpret_cast<const float4*>(O_part + (size_t)(row0 + first + rr) * d_local) + c;
        const size_t step4 = (size_t)ws_rows * d_local / 4;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        auto empty = [](float x) { return __float_as_uint(x) == 0x80000000u; };
        if constexpr (SPLIT > 0) {
            float4 v[SPLIT];
            #pragma unroll
            for (int i = 0; i < SPLIT; i++) v[i] = empty(w[i]) ? make_float4(0.f, 0.f, 0.f, 0.f) : __ldcg(src + i * step4);
            #pragma unroll
            for (int i = 0; i < SPLIT; i++) {
                acc.x = fmaf(w[i], v[i].x, acc.x); acc.y = fmaf(w[i], v[i].y, acc.y);
                acc.z = fmaf(w[i], v[i].z, acc.z); acc.w = fmaf(w[i], v[i].w, acc.w);
            }
        } else {
            // four at a time, with no branch around a load (4096 rows, 16 heads of 64 in 16 splits 57 us; a loop that skips empty ones 89)
            for (int i0 = 0; i0 < split; i0 += 4) {
                float4 v[4];
                #pragma unroll
                for (int k = 0; k < 4; k++) v[k] = i0 + k < split && !empty(w[i0 + k]) ? __ldcg(src + (i0 + k) * step4) : make_float4(0.f, 0.f, 0.f, 0.f);
                #pragma unroll
                for (int k = 0; k < 4; k++) {
                    if (i0 + k >= split) break;
                    acc.x = fmaf(w[i0 + k], v[k].x, acc.x); acc.y = fmaf(w[i0 + k], v[k].y, acc.y);
                    acc.z = fmaf(w[i0 + k], v[k].z, acc.z); acc.w = fmaf(w[i0 + k], v[k].w, acc.w);
                }
            }
        }
        const size_t out = (size_t)(first + rr) * d_local + (size_t)c * 4;
        if constexpr (OUT_F16) {
            uint2 packed;
            packed.x = pack_f16x2(acc.x, acc.y);
            packed.y = pack_f16x2(acc.z, acc.w);
            *reinterpret_cast<uint2*>(reinterpret_cast<__half*>(O) + out) = packed;
        } else {
            *reinterpret_cast<float4*>(reinterpret_cast<float*>(O) + out) = acc;
        }
    }
}

template <int SPLIT>
int launch_combine(const efa_flash_partials& part, void* O, bool f16, int row0, int rows, const efa_flash_params& p, int per_block, int blocks, size_t smem, cudaStream_t stream)
{
    const int d_local = p.H_local * p.d_h;
    if (f16)
        EFA_CUDA(launch_early(combine_splits_kernel<true, SPLIT>, dim3(blocks), 256, smem, stream, part.O_part, part.m_part, part.l_part, O,
                              row0, rows, part.rows, d_local, p.H_local, p.d_h, p.split, per_block));
    else
        EFA_CUDA(launch_early(combine_splits_kernel<false, SPLIT>, dim3(blocks), 256, smem, stream, part.O_part, part.m_part, part.l_part, O,
                              row0, rows, part.rows, d_local, p.H_local, p.d_h, p.split, per_block));
    return 0;
}

__global__ void f32_to_f16_kernel(const float* __restrict__ in, __half* __restrict__ out, size_t n)
{
    size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (; i < n; i += stride) out[i] = __float2half_rn(in[i]);
}

// How far (log2 units) a row maximum may outgrow the exponent offset before the accumulator is rescaled. With the
// maximum itself as the offset the largest softmax weight of a row is exactly 1; under a lagging one it is rounded to fp16
// like the others. Long sweeps of the larger heads lag; small heads (few columns to rescale) and the allocation-free
// entry do not: 2 to 8 % less error against float64 (d_h 32, 4032 keys: 1.94e-4 against 2.07e-4, 2-norm).
constexpr float kRescaleLag = 8.f;

// Heads that a causal launch without counters takes together, longest items first (work_order.h). One head after another, each from its
// last rows, ends on the long items of the last head; row by row over all heads ends on short ones, but all heads' K and V are then live at
// once. So as many as keep theirs in half of the L2, in groups of one size: heads in turn before, in groups now (us): S=8192,
// 16 heads of 64 241 -> 191; S=16384, 16 heads of 64 787 -> 709; S=4096, 16 heads of 64 83.5 -> 53.7; S=8192, 32 heads of 128 540 -> 522; S=32768,
// four heads of 128 928 -> 905; S=16384, four heads of 64 in four splits with the merge 252 -> 220. Groups of 24 or 140 MB are the same but
// for 32 heads of 128 (560, 540). Finding an item takes two steps per split, hence the limit to those.
constexpr size_t kGroupBytes = 64u << 20;
int heads_together(const efa_flash_params& p)
{
    if (!p.causal || p.split > 16) return 0;
    const size_t head_bytes = (size_t)p.S * p.d_h * 2 * sizeof(__half);
    const int most = (int)std::max<size_t>(1, std::min<size_t>((size_t)p.H_local, kGroupBytes / head_bytes));
    const int groups = (p.H_local + most - 1) / most;
    return (p.H_local + groups - 1) / groups;
}

// Tensor maps depend only on (pointer, S, H_local, d_h); drivers launch the same tensors over and over.
struct TmapKey {
    const void* ptr; int S, H, D, rows;
    bool operator<(const TmapKey& o) const { return std::tie(ptr, S, H, D, rows) < std::tie(o.ptr, o.S, o.H, o.D, o.rows); }
};

// box_rows: rows of the tensor per TMA box (128 for Q tiles, the stage length for K and V).
int get_qkv_tmap(const void* ptr, int S, int H_local, int D, int box_rows, CUtensorMap* out)
{
    static std::map<TmapKey, CUtensorMap> cache;
    static std::mutex mu;
    std::lock_guard<std::mutex> lock(mu);
    TmapKey key{ptr, S, H_local, D, box_rows};
    auto it = cache.find(key);
    if (it != cache.end()) { *out = it->second; return 0; }
    const int boxc = D >= 64 ? 64 : D;
    unsigned long long dims[3] = {(unsigned long long)D, (unsigned long long)S, (unsigned long long)H_local};
    unsigned long long strides[2] = {(unsigned long long)D * 2ull, (unsigned long long)S * D * 2ull};
    unsigned box[3] = {(unsigned)boxc, (unsigned)box_rows, 1u};
    CUtensorMap tm;
    if (make_tmap_f16(&tm, ptr, 3, dims, strides, box)) return 1;
    if (cache.size() > 256) cache.clear();
    cache[key] = tm;
    *out = tm;
    return 0;
}

}  // namespace

const char* fa_check_params(const efa_flash_params& p, int q_rows)
{
    if (p.d_h != 16 && p.d_h != 32 && p.d_h != 64 && p.d_h != 128)
        return "tc: d_h must be 16, 32, 64 or 128";
    if (p.S <= 0 || p.S % 64 != 0) return "tc: S must be a multiple of 64";
    if (q_rows <= 0 || q_rows % 64 != 0) return "tc: tile must be a multiple of 64";
    if (p.split < 1 || p.S % (p.split * 64) != 0) return "tc: S must be a multiple of split * 64";
    if (p.H_local < 1) return "tc: H_local must be positive";
    return nullptr;
}

void fa_plan(const efa_flash_params& p, int q_start, int q_rows, efa_flash_plan* out)
{
    FaArgs a{};
    a.q_start = q_start; a.S = p.S;
    a.H_local = p.H_local; a.nsplit = p.split; a.q_rows = q_rows; a.kv_len = p.S / p.split; a.causal = p.causal;
    a.heavy_first = p.causal;                              // without counters
    const FaPlan plan = fa_ws_plan(a, p.d_h, 0);
    *out = efa_flash_plan{plan.items256, plan.items128, plan.tiles, plan.k_slots, plan.v_slots, plan.stage_step};
}

int fa_forward(const void* Q, const void* K, const void* V, void* O, int o_dtype,
               const efa_flash_partials* part, int q_start, int q_rows,
               const efa_flash_params& p, cudaStream_t stream, int* tile_counters, int tile_rows, int reserve_sms,
               int band_rows, int heavy_first, const short* order_tab, int* launches)
{
    if (const char* why = fa_check_params(p, q_rows)) { set_error("flash_attn_tc_forward: %s", why); return 2; }
    if (q_start < 0 || q_start % 64 != 0 || q_start + q_rows > p.S) {
        set_error("flash_attn_tc_forward: rows [%d, %d) outside [0, %d) or not 64-aligned", q_start, q_start + q_rows, p.S);
        return 2;
    }
    if (tile_counters != nullptr && (tile_rows <= 0 || tile_rows % 64 != 0)) {
        set_error("flash_attn_tc_forward: tile_rows must be a positive multiple of 64 when counters are given");
        return 2;
    }
    if (o_dtype != EFA_F32 && o_dtype != EFA_F16) { set_error("flash_attn_tc_forward: unknown O dtype %d", o_dtype); return 2; }
    if (p.split > 1) {
        if (!part || !part->O_part || !part->m_part || !part->l_part || part->rows < q_rows) {
            set_error("flash_attn_tc_forward: split > 1 needs a partials workspace sized for the launch rows");
            return 2;
        }
    } else if (O == nullptr) {
        set_error("flash_attn_tc_forward: O is null");
        return 2;
    }

    CUtensorMap tq, tk, tv;
    if (get_qkv_tmap(Q, p.S, p.H_local, p.d_h, 128, &tq) || get_qkv_tmap(K, p.S, p.H_local, p.d_h, fa_ws_kv_box_rows(), &tk) ||
        get_qkv_tmap(V, p.S, p.H_local, p.d_h, fa_ws_kv_box_rows(), &tv))
        return 1;

    FaArgs a;
    a.O32 = (o_dtype == EFA_F32) ? static_cast<float*>(O) : nullptr;
    a.O16 = (o_dtype == EFA_F16) ? static_cast<__half*>(O) : nullptr;
    a.O_part = part ? part->O_part : nullptr;
    a.m_part = part ? part->m_part : nullptr;
    a.l_part = part ? part->l_part : nullptr;
    a.part_rows = part ? part->rows : 0;
    a.q_start = q_start; a.q_rows = q_rows; a.S = p.S; a.H_local = p.H_local;
    a.nsplit = p.split; a.kv_len = p.S / p.split; a.causal = p.causal;
    a.scale_log2e = p.scale * 1.4426950408889634f;
    a.rescale_above = p.d_h >= 64 ? kRescaleLag : 0.f;
    a.tile_counters = tile_counters; a.tile_rows = tile_rows;
    a.counters_sys = 0;
    if (tile_counters != nullptr) {
        // Counters in (mapped) host memory are read over PCIe by whoever waits for them: fence at system scope then.
        cudaPointerAttributes attr;
        if (cudaPointerGetAttributes(&attr, tile_counters) == cudaSuccess) a.counters_sys = attr.type == cudaMemoryTypeHost ? 1 : 0;
        else (void)cudaGetLastError();
    }
    a.status = kernel_status_word();
    a.band_blocks = (tile_counters == nullptr) ? (q_rows + 255) / 256 : band_rows / 256;
    // Nobody waits for particular rows of a launch without counters, so under a causal mask its longest work
    // items go first and the launch ends on short ones; with counters the caller says in which
    // order it will wait for them (first rows first unless told otherwise).
    a.order_tab = order_tab;
    if (tile_counters == nullptr && order_tab == nullptr && heavy_first < 0) a.group_heads = heads_together(p);
    a.heavy_first = heavy_first >= 0 ? (heavy_first ? 1 : 0) : ((tile_counters == nullptr && p.causal) ? 1 : 0);

    if (launches) {
        const FaPlan plan = fa_ws_plan(a, p.d_h, reserve_sms);
        *launches += plan.items256 > 0 && plan.items128 > 0 ? 2 : 1;
    }
    const bool f16 = (o_dtype == EFA_F16);
    return fa_forward_ws(tq, tk, tv, a, p.d_h, f16, reserve_sms, stream);
}

int fa_combine(const efa_flash_partials& part, void* O, int o_dtype, int row0, int rows,
               const efa_flash_params& p, cudaStream_t stream)
{
    if (p.split <= 1) return 0;
    const int per_block = std::max(1, std::min(CB_ROWS, rows / (2 * device_sms())));
    const int blocks = (rows + per_block - 1) / per_block;
    const size_t smem = (size_t)CB_ROWS * p.H_local * p.split * sizeof(float);
    if (smem > 48 * 1024) { set_error("flash_attn_tc_combine: H_local * split = %d is too large", p.H_local * p.split); return 2; }
    const bool f16 = o_dtype == EFA_F16;
    switch (p.split) {
        case 2:  return launch_combine<2>(part, O, f16, row0, rows, p, per_block, blocks, smem, stream);
        case 3:  return launch_combine<3>(part, O, f16, row0, rows, p, per_block, blocks, smem, stream);
        case 4:  return launch_combine<4>(part, O, f16, row0, rows, p, per_block, blocks, smem, stream);
        case 8:  return launch_combine<8>(part, O, f16, row0, rows, p, per_block, blocks, smem, stream);
        default: return launch_combine<0>(part, O, f16, row0, rows, p, per_block, blocks, smem, stream);
    }
}

int convert_f32_to_f16_dev(const float* in, void* out, size_t n, cudaStream_t stream)
{
    if (n == 0) return 0;
    int blocks = (int)((n + 255) / 256);
    if (blocks > 148 * 16) blocks = 148 * 16;
    f32_to_f16_kernel<<<blocks, 256, 0, stream>>>(in, static_cast<__half*>(out), n);
    EFA_CUDA(cudaGetLastError());
    return 0;
}

}  // namespace efa

// ---------------------------------------------------------------------------------------------
// Split-KV attention without any allocation by the caller or by this library
// ---------------------------------------------------------------------------------------------
// The split-KV path needs scratch for the per-split partial results. Normally the caller owns it
// (efa_flash_partials). Some callers cannot obtain device memory at call time: a serving process
// whose memory pool already holds the whole GPU, so that a plain cudaMalloc fails, or a
// latency-critical loop that cannot afford the device-wide synchronisation cudaMalloc implies.
// For them the partials live in the fixed array below, which is part of the loaded module: every
// GPU that loads this library holds EFA_STATIC_SCRATCH_BYTES of it until the process exits.
namespace efa {
namespace {

static __device__ __align__(256) float g_static_scratch[EFA_STATIC_SCRATCH_BYTES / sizeof(float)];
// Status word of the kernels launched by this entry point ({code, block, site, 0}), in the module for the same
// reason: the status word of the other entry points is allocated memory.
static __device__ int g_noalloc_status[4];

// In host code `g_static_scratch` is only a handle for the symbol, not a device address: the address
// that kernels may use comes from cudaGetSymbolAddress, once per device, with that device current.
int static_scratch_address(float** out, int** status_out)
{
    static float* addr[64] = {};
    static int* status[64] = {};
    static std::mutex mu;
    int dev = 0;
    EFA_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) { set_error("device ordinal %d out of range", dev); return 1; }
    std::lock_guard<std::mutex> lock(mu);
    if (!addr[dev] || !status[dev]) {
        void* p = nullptr;
        void* q = nullptr;
        EFA_CUDA(cudaGetSymbolAddress(&p, g_static_scratch));
        EFA_CUDA(cudaGetSymbolAddress(&q, g_noalloc_status));
        if (!p || !q) { set_error("cudaGetSymbolAddress returned a null address for the static scratch"); return 1; }
        addr[dev] = static_cast<float*>(p);
        status[dev] = static_cast<int*>(q);
    }
    *out = addr[dev];
    *status_out = status[dev];
    return 0;
}

int encode_qkv_tmap_uncached(const void* ptr, int S, int H_local, int D, CUtensorMap* out)
{
    const int boxc = D >= 64 ? 64 : D;
    unsigned long long dims[3] = {(unsigned long long)D, (unsigned long long)S, (unsigned long long)H_local};
    unsigned long long strides[2] = {(unsigned long long)D * 2ull, (unsigned long long)S * D * 2ull};
    unsigned box[3] = {(unsigned)boxc, 128u, 1u};
    return make_tmap_f16(out, ptr, 3, dims, strides, box);
}

}  // namespace

int fa_forward_noalloc(const void* Q, const void* K, const void* V, void* O, int o_dtype,
                       int q_start, int q_rows, const efa_flash_params& p, cudaStream_t stream)
{
    if (const char* why = fa_check_params(p, q_rows)) { set_error("flash_attn_tc_forward_noalloc: %s", why); return 2; }
    if (q_start < 0 || q_start % 64 != 0 || q_start + q_rows > p.S) {
        set_error("flash_attn_tc_forward_noalloc: rows [%d, %d) outside [0, %d) or not 64-aligned", q_start, q_start + q_rows, p.S);
        return 2;
    }
    if (o_dtype != EFA_F32 && o_dtype != EFA_F16) { set_error("flash_attn_tc_forward_noalloc: unknown O dtype %d", o_dtype); return 2; }
    if (!O) { set_error("flash_attn_tc_forward_noalloc: O is null"); return 2; }

    const size_t d_local = (size_t)p.H_local * p.d_h;
    const size_t o_floats = (size_t)p.split * q_rows * d_local;
    const size_t ml_floats = (size_t)p.split * q_rows * p.H_local;
    const size_t need = p.split > 1 ? (o_floats + 2 * ml_floats) * sizeof(float) : 0;
    if (need > (size_t)EFA_STATIC_SCRATCH_BYTES) {
        set_error("flash_attn_tc_forward_noalloc: split=%d rows=%d d_local=%zu needs %zu bytes of scratch, the static "
                  "scratch holds %u; use efa_flash_attn_tc_forward with a caller-owned workspace",
                  p.split, q_rows, d_local, need, (unsigned)EFA_STATIC_SCRATCH_BYTES);
        return 6;
    }
    float* scratch = nullptr;
    int* status = nullptr;
    if (static_scratch_address(&scratch, &status)) return 1;

    CUtensorMap tq, tk, tv;
    if (encode_qkv_tmap_uncached(Q, p.S, p.H_local, p.d_h, &tq) || encode_qkv_tmap_uncached(K, p.S, p.H_local, p.d_h, &tk) ||
        encode_qkv_tmap_uncached(V, p.S, p.H_local, p.d_h, &tv))
        return 1;

    // Every partial that the combine step reads is written by the attention kernel earlier in the
    // same call (idle blocks write zeros and an empty maximum), so nothing has to be cleared.
    efa_flash_partials part{scratch, scratch + o_floats, scratch + o_floats + ml_floats, q_rows};
    FaArgs a;
    a.O32 = (o_dtype == EFA_F32) ? static_cast<float*>(O) : nullptr;
    a.O16 = (o_dtype == EFA_F16) ? static_cast<__half*>(O) : nullptr;
    a.O_part = part.O_part; a.m_part = part.m_part; a.l_part = part.l_part; a.part_rows = q_rows;
    a.q_start = q_start; a.q_rows = q_rows; a.S = p.S; a.H_local = p.H_local;
    a.nsplit = p.split; a.kv_len = p.S / p.split; a.causal = p.causal;
    a.scale_log2e = p.scale * 1.4426950408889634f;
    a.rescale_above = 0.f;
    a.tile_counters = nullptr; a.tile_rows = 0;
    a.counters_sys = 0;
    a.status = status;                       // a word of the module, see noalloc_status()
    a.band_blocks = (q_rows + 255) / 256;
    a.order_tab = nullptr;
    a.heavy_first = p.causal ? 1 : 0;
    a.group_heads = heads_together(p);

    const int rc = fa_forward_ws(tq, tk, tv, a, p.d_h, o_dtype == EFA_F16, 0, stream);
    if (rc) return rc;
    return fa_combine(part, O, o_dtype, 0, q_rows, p, stream);
}

// Status of the kernels launched by fa_forward_noalloc on the current device (and optionally clears it).
// Copies to and from a symbol of the module: no allocation here either.
int noalloc_status(int* out4, int reset)
{
    EFA_CUDA(cudaMemcpyFromSymbol(out4, g_noalloc_status, 4 * sizeof(int)));
    if (reset) {
        const int zero[4] = {0, 0, 0, 0};
        EFA_CUDA(cudaMemcpyToSymbol(g_noalloc_status, zero, sizeof(zero)));
    }
    return 0;
}


namespace {
template <class K> int touch_kernel(K kernel)
{
    cudaFuncAttributes attr;
    EFA_CUDA(cudaFuncGetAttributes(&attr, kernel));
    return 0;
}
}  // namespace

int fa_preload()
{
    return touch_kernel(combine_splits_kernel<true, 2>) || touch_kernel(combine_splits_kernel<false, 2>) ||
           touch_kernel(combine_splits_kernel<true, 3>) || touch_kernel(combine_splits_kernel<false, 3>) ||
           touch_kernel(combine_splits_kernel<true, 4>) || touch_kernel(combine_splits_kernel<false, 4>) ||
           touch_kernel(combine_splits_kernel<true, 8>) || touch_kernel(combine_splits_kernel<false, 8>) ||
           touch_kernel(combine_splits_kernel<true, 0>) || touch_kernel(combine_splits_kernel<false, 0>) ||
           touch_kernel(f32_to_f16_kernel) || fa_ws_preload() || fa_tile_preload();
}

}  // namespace efa
