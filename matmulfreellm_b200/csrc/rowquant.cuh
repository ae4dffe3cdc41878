// Internal interface between the row kernels: fused.cu (block per row), rowwarp.cu (warp per row), rowwise.cu (stand-alone ops).
#pragma once
#include "common.cuh"

// Timeline of prenorm_quant (experiments build, see mmf_row_trace): thread 0 of CTA 0 takes a record of eight stamps per launch.
#ifdef MMF_EXPERIMENTS
extern long long* g_row_trace;
__device__ __forceinline__ long long* row_trace_record(long long* buffer) {
    if (!buffer || threadIdx.x || blockIdx.x || blockIdx.y) return nullptr;
    const int idx = atomicAdd(reinterpret_cast<int*>(buffer), 1);
    return idx < 1000 ? buffer + 8 + 8 * idx : nullptr;
}
__device__ __forceinline__ long long row_now() {
    long long t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
#define ROW_TRACE(slot) do { if (trace) trace[slot] = row_now(); } while (0)
#else
#define ROW_TRACE(slot) do { } while (0)
#endif

struct PrenormArgs {
    const void* x; int64_t ld_x;
    const void* res; int64_t ld_res;      // may be null
    void* res_out;                         // [M, D] contiguous, may be null
    void* y_out;                           // [M, D] contiguous: the normed row in T, may be null
    const float* norm_w; float eps_norm;   // block-level RMSNorm
    const float* nws[3]; float eps_bl;     // per-projection BitLinear norm weights
    int8_t* q; float* dq; int32_t* rowsum; // [G][M][D], [G][M], [G][M]
    int64_t M; int D; int G;
    int round_sum_first;                   // 1: the reference added x+residual as a tensor op (rounded to T) before norm
    int gsplit;                            // 1: grid.y = G CTAs per row, CTA y does projection y alone (decode-sized calls: the G
                                           //    prologues of a row run side by side instead of one after the other)
#ifdef MMF_EXPERIMENTS
    long long* trace;                      // experiments build: 8 global-timer stamps of CTA 0 per launch (see mmf_row_trace)
#endif
};

// From this many rows on, rows of 16-bit activations are worked on by one warp each (rowwarp.cu), from 593 on by four where a quarter of
// the row is long enough (see there, with the times of whole prompt passes).  Fewer rows leave warps idle.  Launched back to back, where a
// kernel's start hides behind the one before, the warps win earlier (999 rows of 2048 values, us, CTA per row -> one warp: gate norm 7.1 ->
// 4.6, three-projection prenorm 10.4 -> 7.3), but not between contractions.
#ifndef MMF_ROW_WARP_MIN_M
#define MMF_ROW_WARP_MIN_M 1024
#endif
constexpr int64_t ROW_WARP_MIN_M = MMF_ROW_WARP_MIN_M;
// longest rows those kernels hold in registers: two-input kernels and the plain quantisation
constexpr int64_t ROW_WARP_MAX_D = 4096, ROW_WARP_MAX_D1 = 7168;
bool row_warp_takes(int64_t M, int64_t D, int dtype, int64_t max_d);
int warp_prenorm_quant_launch(const PrenormArgs& a, int dtype, cudaStream_t st);
int warp_gatenorm_quant_launch(const void* g, int64_t ld_g, const void* o, int64_t ld_o, int dtype, const float* gw, float eps_g,
                               const float* nw, float eps_bl, int8_t* q, float* dq, int32_t* rowsum, int64_t M, int64_t D, cudaStream_t st);
int warp_act_quant_launch(const void* x, int dtype, int64_t ld, const float* nw, int use_norm, float eps, int8_t* q, float* dq,
                          int32_t* rowsum, int64_t M, int64_t D, cudaStream_t st);

// longest row the register-resident activation quantisation takes
constexpr int64_t ACT_QUANT_REGS_MAX_K = 8192;

// mmf_act_quant for rows of at most ACT_QUANT_REGS_MAX_K values and a 16-byte aligned norm weight (arguments already checked)
int act_quant_regs_launch(const void* x, int dtype, int64_t ld_x, const float* norm_w, int use_norm, float eps, int8_t* q, float* dq,
                          int32_t* rowsum, int64_t M, int64_t K, cudaStream_t st);
