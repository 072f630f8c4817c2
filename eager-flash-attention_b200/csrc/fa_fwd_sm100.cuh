// Internal C++ interface of the attention kernels (the C ABI in efa_b200.h forwards to these).
#pragma once

#include <cuda_runtime.h>
#include "../../include/efa_b200.h"

namespace efa {

const char* fa_check_params(const efa_flash_params& p, int q_rows);

int fa_forward(const void* Q, const void* K, const void* V, void* O, int o_dtype,
               const efa_flash_partials* part, int q_start, int q_rows,
               const efa_flash_params& p, cudaStream_t stream, int* tile_counters, int tile_rows,
               int reserve_sms = 0,    // > 0 (d_h 64/128 only): persistent grid that leaves that many SMs free
               int band_rows = 0,      // with counters: rows may complete in bands of this many rows
                                       // (better K/V reuse in L2); 0 = strict row order. Without counters the
                                       // order is free and whole heads are processed one after another.
               int heavy_first = -1,  // 1 = take the row blocks (or bands) from the last to the first, 0 = from
                                       // the first; -1 = last first exactly when there are no counters and the mask is causal
               const short* order_tab = nullptr,  // band_rows == 0: the order of the 256-row blocks (device memory)
               int* launches = nullptr);          // counts the kernels launched

// How fa_forward of p over rows q_start .. q_start+q_rows is cut into work items (fa_ws_plan); the caller has checked p.
void fa_plan(const efa_flash_params& p, int q_start, int q_rows, efa_flash_plan* out);

// Split-KV attention + merge with the partials in a fixed device array (no allocation anywhere).
int fa_forward_noalloc(const void* Q, const void* K, const void* V, void* O, int o_dtype,
                       int q_start, int q_rows, const efa_flash_params& p, cudaStream_t stream);

// {code, block, site, 0} written by a kernel of fa_forward_noalloc whose bounded wait ran out; reset != 0 clears it.
int noalloc_status(int* out4, int reset);

int fa_combine(const efa_flash_partials& part, void* O, int o_dtype, int row0, int rows,
               const efa_flash_params& p, cudaStream_t stream);

int convert_f32_to_f16_dev(const float* in, void* out, size_t n, cudaStream_t stream);

// out[rows][d] = A[rows][d_local] * W[d_local][d]; fp16 in, fp32 accumulate, fp16 (EFA_F16) or fp32 (EFA_F32) out.
int project_f16(const void* A, const void* W, void* out, int rows, int d_local, int d, cudaStream_t stream,
                int out_dtype = EFA_F16, bool own_out = false /* the caller knows `out` to be this GPU's own memory */,
                bool behind = false /* the launch before it in the stream is a projection whose output this one does not touch, and
                                       whose inputs were complete when it started: this one need not wait for it to end */,
                bool beside = false /* runs while an attention kernel holds the SMs, which come free one by one and not in pairs */,
                bool in_parts = false /* k may be summed in parts (fp16 results; the blocks of all modes sum it in one go, to the same bits) */);

// Three projections of one input in one launch: out[t][head][rows][d_h] = X[rows][d] * W[t][head][d][d_h], all fp16.
int project_heads_f16(const void* X, const void* const W[3], void* const out[3], int rows, int d, int heads, int d_h,
                      cudaStream_t stream);

}  // namespace efa
