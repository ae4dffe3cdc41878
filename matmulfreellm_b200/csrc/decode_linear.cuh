// BitLinear of a decode step in one kernel: row work before the contraction (prologue), the contraction, and what the next
// kernel would do first (epilogue).  Steps whose sizes the resident kernel of all blocks takes (decode_step.cuh: 1 row 304 us, 4 rows 454) run
// there; here run the others, and BitLinear calls of one and two rows.
//
// A decode step is a chain of dependent kernels, so its time is the number of links times what a link cannot go below: a
// kernel boundary (0.9 us with programmatic dependent launch) and a read of the previous kernel's rows across the L2 (0.7 us).
// A block of the model used to be eight links (row kernel, contraction, four times).  Here
//   * the gate math and state update of the token mixer and the MLP's silu(gate) * up run in the epilogue of the contraction
//     that produces their inputs (a CTA owns the i, f and g rows, or the gate and up rows, of the same channels), and
//   * for one token row, and for two of at most 2048 values, every CTA repeats the row work that precedes the contraction - norms,
//     statistics, int8 codes - instead of waiting for a kernel that did it: the row work is latency, and the SMs would idle meanwhile.
// That leaves four links per block; up to 16 rows, where repeating the row work costs more than a link, it is a kernel of its
// own that stores the codes in the contraction's operand order (eight links).  Step of a 24-block, 2048-wide model, eight
// links of row kernels and tcgen05 contractions -> here: 1 row 595 -> 435 us, 2 rows 635 -> 500, 4 rows 735 -> 534, 8 rows 737 -> 530, 16 rows 769 -> 663; 32 blocks of 2560: 1 row
// 980 -> 688, 8 rows 1127 -> 831.  What remains is latency.  One row, 2048 wide, a link of 4.3 us on average: 0.85 us from the end
// of the link before it to its release, 0.8 until the row is there, 0.8 - 1.1 until the last norm's statistic is known (down_proj,
// which has one norm: 0.35), 0.45 - 0.95 codes, 0.35 - 1.5 products, 0.2 - 0.4 epilogue.  Four rows: row kernel 1.8 us, of which 0.55 is the row's load;
// contraction 1.2 - 2.4; 0.65 - 1.1 between two of them.
//
// Contraction: mma.sync m16n8k32 (8-bit, int32 accumulators) with 16 weight rows on its M axis and 8 token rows on N.
// tcgen05 is not used: its 128-row tile needs a K split over a cluster to fill the GPU, and the exchange of the split's
// partial sums alone (2.4 us) is longer than this kernel's whole contraction at these sizes.  A CTA (one per SM) owns
// N / 148 output rows and all of K; its 16-row blocks and 256-column groups are split over the warps, each warp keeps a block's
// sums in registers over its groups, and the warps' partial sums meet in shared memory by plain stores (atomics there took
// 45 clocks each and a third of the kernel).  A lane's operands are contiguous: the packed layout gives it 16 bytes (64 weights
// of one row) per group and block, whose 2-bit fields need one mask per register; the order of K inside a group is permuted
// alike for weights and codes, which changes nothing in an integer sum.  Weights are fetched by cp.async into slots private to
// a lane before the grid-dependency wait; ready codes come straight from the L2 (staging them in shared memory first, or
// loading a group ahead, was 10 % slower).  What bounds a link is the number of instructions between the wait and the last
// store, since the next kernel's set-up shares the issue slots: few warps, constants and splits computed on the host.
#pragma once
#include "bitlinear.cuh"
#include "packed.cuh"
#include "rowquant.cuh"

namespace {

constexpr int DL_TS = 20;               // accumulator words per (block, token): 16 rows, padded so that a warp's adds do not collide
constexpr int DL_FUSED_ROWS = MMF_DECODE_LINEAR_FUSED_MAX_M;      // most token rows a CTA takes through the fused prologue
constexpr int DL_CODES = 0;             // prologue of the kernel whose codes were made by decode_rows_kernel
// threads of the kernel with ready codes: 12 warps of up to 80 registers for 8 tokens; 16 tokens' codes and accumulators take
// more than 80, so 8 warps of up to 128
constexpr int dl_codes_threads(int NB) { return NB == 1 ? 384 : 256; }

struct DlParams {
    mmf_decode_linear_args a;
    double inv_k;                       // 1 / K
    int KC, KG;                         // 64-column chunks, groups of four chunks
    int grid, base, extra;              // units (two adjacent output rows; gates, swiglu: channels) per CTA: base, the first `extra` CTAs one more
    float inv_base, inv_base1;          // 1 / base, 1 / (base + 1)
    int inv_kw;                         // warp / kw = warp * inv_kw >> 16
    int kw, bw;                         // warp w takes column groups w % kw, + kw, ... of blocks w / kw, + bw, ...
    int kgw;                            // column groups per warp
    int pf;                             // weight items per warp fetched ahead into shared memory
    int smem_codes, smem_acc, smem_w;   // byte offsets in dynamic shared memory
};

// weights unsigned (2-bit fields in place, up to 2 << 6), codes signed
__device__ __forceinline__ void mma_u8s8(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// the RT threads of a row meet; a row that is the whole CTA uses its barrier
template <int TH, int RT> __device__ __forceinline__ void dl_row_sync() {
    if constexpr (RT == TH) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)(threadIdx.x / RT)), "n"(RT) : "memory");
}
template <int TH, int RT> __device__ __forceinline__ double dl_row_sum(double v, double* slot) {
    constexpr int RW = RT / 32;
    v = warp_sum(v);
    if ((threadIdx.x & 31) == 0) slot[(threadIdx.x % RT) >> 5] = v;
    dl_row_sync<TH, RT>();
    // Every warp folds the partials by shuffles.  Alone on an SM, a whole sum takes 306 / 356 / 438 clocks with 4 / 8 / 16 warps
    // (271 / 319 / 531 with every lane reading all partials).
    constexpr int P = RW <= 2 ? 2 : RW <= 4 ? 4 : RW <= 8 ? 8 : 16;
    const int l = threadIdx.x & (P - 1);
    double t = P == RW || l < RW ? slot[l] : 0.0;
#pragma unroll
    for (int o = P / 2; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    return t;
}
// A kernel parameter in a register from here on: read from the constant bank only where it is first used, it would miss there, on
// the critical path.
template <typename P> __device__ __forceinline__ void pin(P*& p) { asm volatile("" : "+l"(p)); }
__device__ __forceinline__ void pin(int64_t& v) { asm volatile("" : "+l"(v)); }
__device__ __forceinline__ void pin(float& v) { asm volatile("" : "+f"(v)); }

template <int RT> struct __align__(16) DlScratch {      // per row; a member is written once per kernel
    double d0[RT / 32], d1[RT / 32];
    float f[3][RT / 32];
    int i[3][RT / 32];
};

// the prologue's parameters, read before the grid-dependency wait
template <typename T> struct DlRowArgs {
    const T *x, *r;
    T* res_out;
    float eps_norm, eps_bl;
    __device__ __forceinline__ DlRowArgs(const mmf_decode_linear_args& a, int m, bool leader) {
        x = reinterpret_cast<const T*>(a.x);
        if (!a.row_ids) x += m * a.ld_x;
        r = a.residual ? reinterpret_cast<const T*>(a.residual) + m * a.ld_residual : nullptr;
        res_out = a.residual_out && leader ? reinterpret_cast<T*>(a.residual_out) + m * a.K : nullptr;
        eps_norm = a.eps_norm;
        eps_bl = a.eps_bl;
        pin(x); pin(r); pin(res_out); pin(eps_norm); pin(eps_bl);
    }
};

// eight values of a row, as packed pairs
struct DlVec { uint32_t v[4]; };
template <typename T> __device__ __forceinline__ DlVec dl_load(const T* p) {
    const uint4 t = *reinterpret_cast<const uint4*>(p);
    return DlVec{{t.x, t.y, t.z, t.w}};
}

// vector `it` of a thread starts at column c; NVT vectors of eight values cover a row of D values
#define DL_FOREACH(it, c) _Pragma("unroll") for (int it = 0, c = rt * 8; it < NVT; ++it, c += RT * 8) if (c < D)

// Row prologue of row m, RT = TH / MR threads: codes of G projections in the MMA's operand order, absmax and (per-warp) code
// sums beside them.  Columns c .. c + 15 of a 256-column group are the 16-byte piece ((c / 16) % 4) * word + (c / 64) % 4 of
// `codes`; a group is 4 * step pieces, a projection KG groups.
template <typename T, int PRO, int G, int TH, int MR, int NVT>
__device__ __forceinline__ void dl_prologue(const mmf_decode_linear_args& a, const DlRowArgs<T>& ra, int m, int D, int KG, const float* snw, uint8_t* codes,
                                            int word, int step, DlScratch<TH / MR>& red, float (&s_amax)[G], double inv_d) {
    constexpr int RT = TH / MR;
    const int rt = threadIdx.x % RT, lane = threadIdx.x & 31, rw = rt >> 5;
    const T* x = ra.x;
    if (PRO == MMF_PRO_PRENORM && a.row_ids) {
        const int64_t row = a.row_ids[m];
        x += (row < 0 ? 0 : row >= a.x_rows ? a.x_rows - 1 : row) * a.ld_x;    // clamp instead of faulting on a bad id
    }
    const T* r = PRO != MMF_PRO_QUANT ? ra.r : nullptr;
    DlVec u[NVT], v[NVT];
    double s0 = 0.0, s1 = 0.0;
    DL_FOREACH(it, c) u[it] = dl_load(x + c);
    if (r) {
        DL_FOREACH(it, c) v[it] = dl_load(r + c);
    }
    if constexpr (PRO == MMF_PRO_PRENORM) {
        T* ro = ra.res_out;
        const bool plain = !r || a.round_sum_first;        // what is normalised is a row of T values
        DL_FOREACH(it, c) {
            uint32_t o[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (plain) {
                    if (r) u[it].v[i] = narrow<T>(__fadd2_rn(widen<T>(u[it].v[i]), widen<T>(v[it].v[i])));
                    o[i] = u[it].v[i];
                    sumsq_pair<T>(u[it].v[i], s0, s1);
                } else {
                    const float2 t = __fadd2_rn(widen<T>(u[it].v[i]), widen<T>(v[it].v[i]));
                    s0 = fma((double)t.x, (double)t.x, s0);
                    s1 = fma((double)t.y, (double)t.y, s1);
                    o[i] = narrow<T>(t);
                }
            }
            if (ro) *reinterpret_cast<uint4*>(ro + c) = make_uint4(o[0], o[1], o[2], o[3]);
        }
        const float rstd = rstd_from_sumsq(dl_row_sum<TH, RT>(s0 + s1, red.d0), D, inv_d, ra.eps_norm);
        s0 = s1 = 0.0;
        DL_FOREACH(it, c) {
            float2 w[4];
            lds8(snw + c, w);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float2 t = widen<T>(u[it].v[i]);
                if (!plain) t = __fadd2_rn(t, widen<T>(v[it].v[i]));
                u[it].v[i] = narrow<T>(__fmul2_rn(mul2(t, rstd), w[i]));
                sumsq_pair<T>(u[it].v[i], s0, s1);
            }
        }
        snw += D;
    } else if constexpr (PRO == MMF_PRO_GATENORM) {
        DL_FOREACH(it, c) {
#pragma unroll
            for (int i = 0; i < 4; ++i) sumsq_pair<T>(u[it].v[i], s0, s1);
        }
        const float rstd = rstd_from_sumsq(dl_row_sum<TH, RT>(s0 + s1, red.d0), D, inv_d, ra.eps_norm);
        s0 = s1 = 0.0;
        DL_FOREACH(it, c) {
            float2 w[4];
            lds8(snw + c, w);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 o = widen<T>(v[it].v[i]);
                const float2 y = __fmul2_rn(mul2(widen<T>(u[it].v[i]), rstd), w[i]);
                u[it].v[i] = narrow<T>(__fmul2_rn(__fmul2_rn(y, o), sigmoid2(o)));
                sumsq_pair<T>(u[it].v[i], s0, s1);
            }
        }
        snw += D;
    } else {
        DL_FOREACH(it, c) {
#pragma unroll
            for (int i = 0; i < 4; ++i) sumsq_pair<T>(u[it].v[i], s0, s1);
        }
    }
    // BitLinear prologue: y = (v * rstd) * w, absmax -> scale -> int8 codes
    const float rstd = rstd_from_sumsq(dl_row_sum<TH, RT>(s0 + s1, red.d1), D, inv_d, ra.eps_bl);
    float am[G];
#pragma unroll
    for (int g = 0; g < G; ++g) am[g] = 0.0f;
    DL_FOREACH(it, c) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float2 w[4];
            lds8(snw + g * D + c, w);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 y = __fmul2_rn(mul2(widen<T>(u[it].v[i]), rstd), w[i]);
                am[g] = fmaxf(am[g], fmaxf(fabsf(y.x), fabsf(y.y)));
            }
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const uint32_t t = __reduce_max_sync(0xffffffffu, __float_as_uint(am[g]));   // non-negative floats order like their bits
        if (lane == 0) red.f[g][rw] = __uint_as_float(t);
    }
    dl_row_sync<TH, RT>();
    float s[G];
    int sum[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        float t = 1e-5f;
#pragma unroll
        for (int w = 0; w < RT / 32; ++w) t = fmaxf(t, red.f[g][w]);
        s[g] = q127_over(t);
        sum[g] = 0;
        if (rt == 0) s_amax[g] = t;
    }
    DL_FOREACH(it, c) {
        uint8_t* dst = codes + ((c >> 8) * (4 * step) + ((c >> 4) & 3) * word + ((c >> 6) & 3)) * 16 + (c & 15);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float2 w[4];
            lds8(snw + g * D + c, w);
            uint32_t word[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                word[i] = codes4(__fmul2_rn(mul2(widen<T>(u[it].v[2 * i]), rstd), w[2 * i]),
                                 __fmul2_rn(mul2(widen<T>(u[it].v[2 * i + 1]), rstd), w[2 * i + 1]), s[g]);
                sum[g] = __dp4a((int)word[i], 0x01010101, sum[g]);
            }
            uint8_t* d = dst + g * KG * (step * 64);
            *reinterpret_cast<uint2*>(d) = make_uint2(word[0], word[1]);
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const int t = __reduce_add_sync(0xffffffffu, sum[g]);
        if (lane == 0) red.i[g][rw] = t;
    }
}

__device__ __forceinline__ float dl_out(int acc, int rs, float scale) { return __fmul_rn((float)(acc - rs), scale); }

// The row work of a decode step as a kernel of its own: a CTA per token row and projection.  Codes in the operand order of the
// contraction that follows, 8 * NB tokens side by side.
template <typename T, int PRO, int TH, int NVT>
__global__ void __launch_bounds__(TH)
decode_rows_kernel(const __grid_constant__ mmf_decode_linear_args a, int KG, int NB, double inv_k) {
    extern __shared__ __align__(16) uint8_t smem[];
    float* snw = reinterpret_cast<float*>(smem);
    __shared__ DlScratch<TH> red;
    __shared__ float s_amax[1];
    const int m = blockIdx.x, g = blockIdx.y, D = (int)a.K, tid = threadIdx.x;
    pdl_trigger();
    auto stage = [&](float* dst, const float* src) {
        if (src) for (int i = tid * 4; i < D; i += TH * 4) cp_async16(dst + i, src + i);
        else for (int i = tid; i < D; i += TH) dst[i] = 1.0f;
    };
    if (PRO != MMF_PRO_QUANT) stage(snw, a.norm_w);
    stage(snw + (PRO != MMF_PRO_QUANT ? D : 0), a.bl_norm_w[g]);
    cp_async_commit();
    const DlRowArgs<T> ra(a, m, g == 0);
    uint8_t* codes = reinterpret_cast<uint8_t*>(a.codes) + ((int64_t)g * KG * NB * 128 + (m >> 3) * 128 + (m & 7) * 4) * 16;
    float* dq = a.dq + (int64_t)g * a.M + m;
    int32_t* rowsum = a.rowsum + (int64_t)g * a.M + m;
    pin(codes); pin(dq); pin(rowsum);
    cp_async_wait_all();
    __syncthreads();
    pdl_wait();
    dl_prologue<T, PRO, 1, TH, 1, NVT>(a, ra, m, D, KG, snw, codes, 32, 32 * NB, red, s_amax, inv_k);
    __syncthreads();
    if (tid == 0) {
        int t = 0;
#pragma unroll
        for (int w = 0; w < TH / 32; ++w) t += red.i[0][w];
        *rowsum = t;
        *dq = over_127(s_amax[0]);
    }
}

// Fused: TH threads, MR token rows (M <= MR), NVT 8-value vectors of a row per thread of the row.  Codes from
// decode_rows_kernel: MR = 8 NB token rows; at most TH threads.
template <typename T, int PRO, int EPI, int TH, int MR, int NVT>
__global__ void __launch_bounds__(TH, 2)
decode_linear_kernel(const __grid_constant__ DlParams p) {
    const mmf_decode_linear_args& a = p.a;
    constexpr bool FUSED = PRO != DL_CODES, CONST8 = FUSED && TH == 256;
    constexpr int NB = FUSED ? 1 : MR / 8, SC = FUSED ? DL_FUSED_ROWS : MR;
    constexpr int G = EPI == MMF_EPI_GATES ? 3 : 1;          // projections (code sets)
    constexpr int RT = TH / MR, TL = 4 * MR;
    constexpr int BP = EPI == MMF_EPI_SWIGLU ? 4 : 8;        // units per block of 16 MMA rows (swiglu: 8 gate and 8 up rows)
    extern __shared__ __align__(16) uint8_t smem[];
    float* snw = reinterpret_cast<float*>(smem);             // norm weights of the prologue
    uint8_t* scodes = smem + p.smem_codes;                   // [G][KG][4 words][TL lanes] 16-byte pieces
    int* part = reinterpret_cast<int*>(smem + p.smem_acc);   // [block][kw][MR tokens][DL_TS] partial sums
    uint4* wslot = reinterpret_cast<uint4*>(smem + p.smem_w);
    __shared__ DlScratch<FUSED ? RT : 32> red[FUSED ? MR : 1];
    __shared__ float s_amax[DL_FUSED_ROWS][G];
    __shared__ float s_scale[G][SC];                         // dq * mean|w|
    __shared__ int s_rs[G][SC];                              // code sum (weights are stored + 1)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, q = lane & 3;
    pdl_trigger();
    const int bid = blockIdx.x, u0 = bid * p.base + min(bid, p.extra), pairs = p.base + (bid < p.extra ? 1 : 0);
    const int nb = (pairs + BP - 1) / BP * G;                // blocks of this CTA; the last one may be partly empty
    const int D = (int)a.K, M = (int)a.M, KC = p.KC, KG = p.KG, kgw = p.kgw, kw = CONST8 ? 8 : p.kw, bw = CONST8 ? 1 : p.bw;
    const int nthr = FUSED ? TH : (int)blockDim.x;
    const int bq = CONST8 ? 0 : warp * p.inv_kw >> 16, kq = warp - bq * kw;           // this warp's blocks and column groups (bq >= bw: none)

    // Item (block b, j): column group kq + j kw.  Weight rows gq and gq + 8 of the block, 16 bytes (64 weights) of chunk 4 kg + q.
    const int rows_end = 2 * pairs;
    auto fetch = [&](int b, int j, auto&& take) {
        const int chunk = (kq + j * kw) * 4 + q;
        const uint4* w0 = reinterpret_cast<const uint4*>(a.packed) + (int64_t)chunk * MMF_TILE_ROWS;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = EPI == MMF_EPI_SWIGLU ? b * 8 + gq : b / G * 16 + gq + 8 * half;   // row (channel) of the CTA
            int n = 2 * u0 + r;
            if constexpr (EPI == MMF_EPI_GATES) n += (b % 3) * D;                            // i | f | g of D rows each
            if constexpr (EPI == MMF_EPI_SWIGLU) n += half * (int)(a.N >> 1);                // gate rows, then up rows
            // past the end of the CTA's rows or of K: all fields zero, no contribution (codes are stored + 1)
            take(half, chunk < KC && r < rows_end ? w0 + (int64_t)(n >> 7) * KC * MMF_TILE_ROWS + (n & 127) : nullptr);
        }
    };
    {   // the weights do not depend on the preceding kernel: on their way before the grid-dependency wait
        uint4* dst = wslot + (size_t)warp * p.pf * 64 + lane;
        int k = 0;
        for (int b = bq < bw ? bq : nb; b < nb; b += bw)
            for (int j = 0; j < kgw && k < p.pf; ++j, ++k, dst += 64)
                fetch(b, j, [&](int half, const uint4* src) {
                    if (src) cp_async16(dst + half * 32, src);
                    else dst[half * 32] = make_uint4(0, 0, 0, 0);
                });
        cp_async_commit();
    }
    if constexpr (FUSED) {
        auto stage = [&](float* dst, const float* src) {
            if (src) for (int i = tid * 4; i < D; i += TH * 4) cp_async16(dst + i, src + i);
            else for (int i = tid; i < D; i += TH) dst[i] = 1.0f;
        };
        float* sdst = snw;
        if (PRO != MMF_PRO_QUANT) { stage(sdst, a.norm_w); sdst += D; }
#pragma unroll
        for (int g = 0; g < G; ++g) stage(sdst + g * D, a.bl_norm_w[g]);
        cp_async_commit();
    }

    // what the rest needs of the parameters and the model's constants
    const int cg = tid / SC, cm = tid % SC;                  // (projection, token) whose scale this thread combines
    const bool has_const = cg < G && cm < M;
    const float ws = has_const ? a.w_scale[cg] : 0.0f;
    const DlRowArgs<T> ra(a, FUSED ? tid / RT : 0, bid == 0);
    const uint4* codes = reinterpret_cast<const uint4*>(a.codes) + lane;
    const float* dq = a.dq + cg * M + cm;
    const int32_t* rowsum = a.rowsum + cg * M + cm;
    if (!FUSED) { pin(codes); pin(dq); pin(rowsum); }
    T *out = reinterpret_cast<T*>(a.out), *g_out = reinterpret_cast<T*>(a.g_out);
    const T* lb = reinterpret_cast<const T*>(a.lower_bound);
    float* state = a.state;
    const uint8_t* mask = a.mask;
    int64_t ld_out = a.ld_out, N = a.N;
    pin(out); pin(ld_out);
    if (EPI == MMF_EPI_GATES) { pin(g_out); pin(lb); pin(state); pin(mask); }
    if (EPI == MMF_EPI_STORE) pin(N);
    // the (token, unit) this thread finishes first
    // (a division that is exact here: (i + 0.5) / pairs stays 0.5 / pairs away from whole numbers, and i < 32 * pairs)
    const float inv_pairs = bid < p.extra ? p.inv_base1 : p.inv_base;
    auto token_of = [&](int i) { return MR == 1 ? 0 : (int)(((float)i + 0.5f) * inv_pairs); };
    const int m_pre = token_of(tid), pr_pre = tid - m_pre * pairs;
    const bool has_pre = EPI == MMF_EPI_GATES && m_pre < M && pr_pre < pairs;
    uint32_t lb_pre = 0;
    if (has_pre && lb) lb_pre = *reinterpret_cast<const uint32_t*>(lb + (u0 + pr_pre) * 2);
    cp_async_wait_all();
    __syncthreads();
    pdl_wait();

    // gates: the state this thread will advance (and whether its token is padding), on the way during the contraction
    float2 h_pre = make_float2(0.0f, 0.0f);
    bool keep_pre = true;
    if (has_pre) {
        h_pre = *reinterpret_cast<const float2*>(state + (int64_t)m_pre * D + (u0 + pr_pre) * 2);
        if (mask) keep_pre = mask[m_pre] != 0;
    }
    if constexpr (FUSED) {
        const int m = tid / RT;
        if (MR == 1 || m < M)
            dl_prologue<T, PRO, G, TH, MR, NVT>(a, ra, m, D, KG, snw, scodes + m * 64, TL, TL, red[m], s_amax[m], p.inv_k);
        __syncthreads();                                     // codes complete
        if (has_const) {
            int t = 0;
#pragma unroll
            for (int w = 0; w < RT / 32; ++w) t += red[cm < MR ? cm : 0].i[cg][w];
            s_rs[cg][cm] = t;
            s_scale[cg][cm] = __fmul_rn(over_127(s_amax[cm][cg]), ws);
        }
    } else {
        if (has_const) {
            s_scale[cg][cm] = __fmul_rn(*dq, ws);
            s_rs[cg][cm] = *rowsum;
        }
    }


    // the 2-bit fields stay where they are: field f of a byte counts 4^f, one accumulator per field, shifted back at the end
    if (CONST8 ? kq < KG : bq < bw) {
        const uint4* src = wslot + (size_t)warp * p.pf * 64 + lane;
        int* dst = part + ((bq * kw + kq) * MR + 2 * q) * DL_TS + gq;
        int k = 0;
#pragma unroll 1
        for (int b = bq; b < nb; b += bw, dst += bw * kw * MR * DL_TS) {
            int c[4][NB][4] = {};
            const int g = EPI == MMF_EPI_GATES ? b % 3 : 0;
            // codes of the first group.  Fused: tokens MR - 7 do not exist, any code will do
            const uint4* cb = FUSED ? reinterpret_cast<const uint4*>(scodes) + (g * KG + kq) * (TL * 4) + (lane & (TL - 1))
                                    : codes + (g * KG + kq) * (NB * 128);
            const int cstep = FUSED ? kw * TL * 4 : kw * NB * 128;
            constexpr int CW = FUSED ? TL : 32;              // pieces per word
#pragma unroll 1
            for (int j = 0; j < kgw; ++j, ++k, src += 64, cb += cstep) {
                if (kq + j * kw >= KG) continue;
                uint4 wa, wb;
                if (k < p.pf) {
                    wa = src[0];
                    wb = src[32];
                } else {                                     // more weights than the slots hold
                    fetch(b, j, [&](int half, const uint4* s) { (half ? wb : wa) = s ? __ldg(s) : make_uint4(0, 0, 0, 0); });
                }
                const uint32_t xa[4] = {wa.x, wa.y, wa.z, wa.w}, xb[4] = {wb.x, wb.y, wb.z, wb.w};
                uint4 x[NB][4];
#pragma unroll
                for (int t = 0; t < NB; ++t)
#pragma unroll
                    for (int w = 0; w < 4; ++w) x[t][w] = cb[(t * 4 + w) * CW];
#pragma unroll
                for (int w = 0; w < 4; w += 2)
#pragma unroll
                    for (int f = 0; f < 4; ++f) {
                        const uint32_t msk = 0x03030303u << (2 * f);
#pragma unroll
                        for (int t = 0; t < NB; ++t) {
                            const uint32_t B0[4] = {x[t][w].x, x[t][w].y, x[t][w].z, x[t][w].w},
                                           B1[4] = {x[t][w + 1].x, x[t][w + 1].y, x[t][w + 1].z, x[t][w + 1].w};
                            mma_u8s8(c[f][t], xa[w] & msk, xb[w] & msk, xa[w + 1] & msk, xb[w + 1] & msk, B0[f], B1[f]);
                        }
                    }
            }
#pragma unroll
            for (int t = 0; t < NB; ++t)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int v = c[0][t][i] + (c[1][t][i] >> 2) + (c[2][t][i] >> 4) + (c[3][t][i] >> 6);
                    if (!FUSED || 2 * q + (i & 1) < MR) dst[(t * 8 + (i & 1)) * DL_TS + (i >> 1) * 8] = v;
                }
        }
    }
    __syncthreads();

    // ---- epilogue: a thread finishes two adjacent rows (channels) of a token
    for (int i = tid; i < pairs * M; i += nthr) {
        const int m = token_of(i), pr = i - m * pairs;
        // rows r, r + 1 of block b, rounded to T and packed
        auto value = [&](int b, int r, int g) {
            const int* s = part + (b * kw * MR + m) * DL_TS + r;
            int2 v = make_int2(0, 0);
            if constexpr (CONST8) {
                const int np = min(kw, KG);
#pragma unroll
                for (int w = 0; w < 8; ++w)
                    if (w < np) {
                        const int2 t = *reinterpret_cast<const int2*>(s + w * MR * DL_TS);
                        v.x += t.x;
                        v.y += t.y;
                    }
            } else {
#pragma unroll 4
                for (int w = 0; w < kw; ++w, s += MR * DL_TS) {
                    const int2 t = *reinterpret_cast<const int2*>(s);
                    v.x += t.x;
                    v.y += t.y;
                }
            }
            return narrow<T>(make_float2(dl_out(v.x, s_rs[g][m], s_scale[g][m]), dl_out(v.y, s_rs[g][m], s_scale[g][m])));
        };
        if constexpr (EPI == MMF_EPI_STORE) {
            const int64_t n = (int64_t)(u0 + pr) * 2;
            const uint32_t o = value(pr >> 3, (pr & 7) * 2, 0);
            T* dst = out + m * ld_out + n;
            if (n + 2 <= N && (ld_out & 1) == 0) *reinterpret_cast<uint32_t*>(dst) = o;
            else
                for (int k = 0; k < 2 && n + k < N; ++k) dst[k] = reinterpret_cast<const T*>(&o)[k];
        } else if constexpr (EPI == MMF_EPI_SWIGLU) {
            // z = round(silu(round(gate)) * round(up)): block b holds 8 channels, rows 0-7 gate and 8-15 up
            const int b = pr >> 2, r = (pr & 3) * 2;
            const float2 gate = widen<T>(value(b, r, 0)), up = widen<T>(value(b, 8 + r, 0));
            *reinterpret_cast<uint32_t*>(out + m * ld_out + (int64_t)(u0 + pr) * 2) = narrow<T>(silu_mul2(gate, up));
        } else {
            // token mixer of one new token (layers/hgrn_bit.py:113-125 of the reference with T = 1)
            const int unit = pr >> 3, r = (pr & 7) * 2, ch = (u0 + pr) * 2;
            const bool pre = i == tid;
            float2* st = reinterpret_cast<float2*>(state + (int64_t)m * D + ch);
            float2 h = pre ? h_pre : *st;
            float2 xv = raw_gate_floor(widen<T>(value(unit * 3, r, 0))), f = raw_gate_floor(widen<T>(value(unit * 3 + 1, r, 1)));
            float2 lbv = make_float2(0.0f, 0.0f), oml = make_float2(1.0f, 1.0f);
            if (lb) {
                lbv = widen<T>(pre ? lb_pre : *reinterpret_cast<const uint32_t*>(lb + ch));
                oml = make_float2(round_to<T>(__fsub_rn(1.0f, lbv.x)), round_to<T>(__fsub_rn(1.0f, lbv.y)));
            }
            raw_gate_pair<T>(xv, f, lb != nullptr, lbv, oml);
            if (mask && !(pre ? keep_pre : mask[m] != 0)) xv = make_float2(0.0f, 0.0f);      // a padding position contributes no input
            h.x = fmaf(f.x, h.x, xv.x);
            h.y = fmaf(f.y, h.y, xv.y);
            *st = h;
            *reinterpret_cast<uint32_t*>(out + (int64_t)m * D + ch) = narrow<T>(h);
            *reinterpret_cast<uint32_t*>(g_out + (int64_t)m * D + ch) = value(unit * 3 + 2, r, 2);
        }
    }
}

constexpr int DL_SMEM_MAX = 220 * 1024;

template <auto kernel> int dl_go(const DlParams& p, int threads, int smem, cudaStream_t st) {
    MMF_CUDA(mmf_allow_smem<kernel>(DL_SMEM_MAX));
    MMF_CUDA(mmf_launch_pdl(kernel, dim3((unsigned)p.grid), dim3((unsigned)threads), (size_t)smem, st, p));
    MMF_LAUNCH_CHECK("decode_linear_kernel");
    return MMF_OK;
}

template <typename T, int PRO, int TH, int NVT> int dl_rows_go(const mmf_decode_linear_args& a, int G, int KG, int NB, cudaStream_t st) {
    MMF_CUDA(mmf_launch_pdl(decode_rows_kernel<T, PRO, TH, NVT>, dim3((unsigned)a.M, (unsigned)G), dim3(TH),
                            (size_t)(PRO == MMF_PRO_QUANT ? 1 : 2) * a.K * 4, st, a, KG, NB, 1.0 / (double)a.K));
    MMF_LAUNCH_CHECK("decode_rows_kernel");
    return MMF_OK;
}
// the fewest threads (of 8 values each) that hold the row; a plain row of more than 4096 values takes two vectors per thread
template <typename T, int PRO> int dl_rows(const mmf_decode_linear_args& a, int G, int KG, int NB, cudaStream_t st) {
    if (a.K <= 1024) return dl_rows_go<T, PRO, 128, 1>(a, G, KG, NB, st);
    if (a.K <= 2048) return dl_rows_go<T, PRO, 256, 1>(a, G, KG, NB, st);
    if (a.K <= 3072) return dl_rows_go<T, PRO, 384, 1>(a, G, KG, NB, st);
    if (a.K <= 4096) return dl_rows_go<T, PRO, 512, 1>(a, G, KG, NB, st);
    if constexpr (PRO == MMF_PRO_QUANT) {
        if (a.K <= 6144) return dl_rows_go<T, PRO, 384, 2>(a, G, KG, NB, st);
        return dl_rows_go<T, PRO, 512, 2>(a, G, KG, NB, st);
    }
    return mmf_set_error(MMF_ERR_BAD_SHAPE, "mmf_decode_linear: row of %lld values", (long long)a.K);
}

// arguments are checked by mmf_decode_linear
template <typename T> int decode_linear_launch(const mmf_decode_linear_args& a, cudaStream_t st) {
    DlParams p;
    p.a = a;
    p.KC = (int)(a.K / MMF_TILE_K);
    p.KG = (p.KC + 3) / 4;
    p.inv_k = 1.0 / (double)a.K;
    const bool fused = a.codes == nullptr;
    const int G = a.epilogue == MMF_EPI_GATES ? 3 : 1, D = (int)a.K;
    const int NB = fused || a.M <= 8 ? 1 : 2, MR = !fused ? 8 * NB : a.M <= 1 ? 1 : 2;
    // One CTA on every SM, however the rows divide: two kernels of the chain share an SM (the next one waits with its weights),
    // and an SM that this grid left empty would later take two CTAs of the next one, which then finishes late.
    const int units = a.epilogue == MMF_EPI_GATES ? (int)(a.K / 2) : a.epilogue == MMF_EPI_SWIGLU ? (int)(a.N / 4) : (int)((a.N + 1) / 2);
    p.grid = units < 148 ? units : 148;
    p.base = units / p.grid;
    p.extra = units % p.grid;
    p.inv_base = 1.0f / (float)p.base;
    p.inv_base1 = 1.0f / (float)(p.base + 1);
    const int bp = a.epilogue == MMF_EPI_SWIGLU ? 4 : 8;
    const int nb = (p.base + (p.extra ? 1 : 0) + bp - 1) / bp * G;        // most blocks of one CTA
    int threads;
    if (fused) {
        // Every warp repeats a row's scalar work (statistics, scales), and the next kernel's set-up competes for the same issue
        // slots, so one row gets the fewest warps that hold it (8 values a thread).
        threads = MR > 1 ? 512 : D <= 1024 ? 128 : D <= 2048 ? 256 : D <= 3072 ? 384 : D <= 4096 ? 512 : D <= 6144 ? 256 : 512;
        // warps over column groups x blocks: the split with the fewest rounds, then the fewest partial sums
        const int warps = threads / 32;
        int best = 1 << 30;
        for (int kw = 1; kw <= warps && kw <= p.KG; ++kw) {
            const int bw = warps / kw < nb ? warps / kw : nb;
            const int cost = ((p.KG + kw - 1) / kw) * ((nb + bw - 1) / bw) * 64 + kw;
            if (cost < best) { best = cost; p.kw = kw; p.bw = bw; }
        }
        // Eight warps (rows of 1025 - 2048 and 4097 - 6144 values) all split K, whatever that rule says: constants in the kernel instead
        // of loops and divisions.  1024 < K <= 6144 to 2048 outputs 3 - 6 % faster (K = 1088 2.24 us a call against 2.31, 2048 2.43 / 2.50,
        // 6144 3.52 / 3.59), steps of 24 blocks 371 / 375 us (1280 wide), 388 / 388 (1536), 431 / 438 (2048).  It loses where the groups of
        // K do not divide among eight warps and the outputs are many: 11264 outputs at K = 1088 3.53 / 3.27, at 4160 8.63 / 8.33.
        if (threads == 256) { p.kw = 8; p.bw = 1; }
    } else {
        int best = 1 << 30;
        for (int kw = 1; kw <= dl_codes_threads(NB) / 32 && kw <= p.KG; ++kw) {
            const int bw = dl_codes_threads(NB) / 32 / kw < nb ? dl_codes_threads(NB) / 32 / kw : nb;
            const int cost = ((p.KG + kw - 1) / kw) * ((nb + bw - 1) / bw) * 64 + kw * bw;
            if (cost < best) { best = cost; p.kw = kw; p.bw = bw; }
        }
        threads = p.kw * p.bw > 8 ? p.kw * p.bw * 32 : 256;
    }
    if (!(fused && threads == 256))                          // many blocks (lm_head): fewer partial sums per block, so that they fit
        while (p.kw > 1 && nb * p.kw * MR * DL_TS * 4 > 80 * 1024) {
            p.kw = (p.kw + 1) / 2;
            p.bw = threads / 32 / p.kw < nb ? threads / 32 / p.kw : nb;
        }
    p.kgw = (p.KG + p.kw - 1) / p.kw;
    p.inv_kw = 65536 / p.kw + 1;
    int off = fused ? (a.prologue == MMF_PRO_QUANT ? G : G + 1) * D * 4 : 0;
    p.smem_codes = off;
    off += fused ? G * p.KG * 256 * MR : 0;
    p.smem_acc = off;
    off += nb * p.kw * MR * DL_TS * 4;
    p.smem_w = off;
    const int per_item = p.kw * p.bw * 1024, want = (nb + p.bw - 1) / p.bw * p.kgw, room = (DL_SMEM_MAX - off) / per_item;
    MMF_REQUIRE(off <= DL_SMEM_MAX && room >= 0, MMF_ERR_BAD_SHAPE, "mmf_decode_linear: N=%lld K=%lld do not fit in shared memory", (long long)a.N,
                (long long)a.K);
    p.pf = want < room ? want : room;
    const int smem = off + p.pf * per_item;
    // (after every check: a refused call has launched nothing)
    if (!fused) {
        const int rc = a.prologue == MMF_PRO_QUANT     ? dl_rows<T, MMF_PRO_QUANT>(a, G, p.KG, NB, st)
                       : a.prologue == MMF_PRO_PRENORM ? dl_rows<T, MMF_PRO_PRENORM>(a, G, p.KG, NB, st)
                                                       : dl_rows<T, MMF_PRO_GATENORM>(a, G, p.KG, NB, st);
        if (rc != MMF_OK) return rc;
    }

#define DL_K(PRO, EPI, TH, MR, NVT) return dl_go<decode_linear_kernel<T, PRO, EPI, TH, MR, NVT>>(p, threads, smem, st)
#define DL_CODES_K(EPI)                                            \
    if (!fused && a.epilogue == EPI) {                             \
        if (NB == 1) DL_K(DL_CODES, EPI, dl_codes_threads(1), 8, 1);  \
        DL_K(DL_CODES, EPI, dl_codes_threads(2), 16, 1);              \
    }
    DL_CODES_K(MMF_EPI_GATES)
    DL_CODES_K(MMF_EPI_SWIGLU)
    DL_CODES_K(MMF_EPI_STORE)
#undef DL_CODES_K
#define DL_FUSED(PRO, EPI)                                                                                            \
    if (a.prologue == PRO && a.epilogue == EPI) {                                                                     \
        constexpr bool LONG = PRO == MMF_PRO_QUANT;                                                                   \
        if (MR == 1) {                                                                                                \
            if (D <= 1024) DL_K(PRO, EPI, 128, 1, 1);                                                                 \
            if (D <= 2048) DL_K(PRO, EPI, 256, 1, 1);                                                                 \
            if (D <= 3072) DL_K(PRO, EPI, 384, 1, 1);                                                                 \
            if (D <= 4096) DL_K(PRO, EPI, 512, 1, 1);                                                                 \
            if constexpr (LONG) { if (D <= 6144) DL_K(PRO, EPI, 256, 1, 3); DL_K(PRO, EPI, 512, 1, 2); }              \
        } else {                                                                                         \
            if (D <= 2048) DL_K(PRO, EPI, 512, 2, 1);                                                                 \
            if (D <= 4096) DL_K(PRO, EPI, 512, 2, 2);                                                                 \
            if constexpr (LONG) { if (D <= 6144) DL_K(PRO, EPI, 512, 2, 3); DL_K(PRO, EPI, 512, 2, 4); }              \
        }                                                                                                             \
    }
    DL_FUSED(MMF_PRO_PRENORM, MMF_EPI_GATES)
    DL_FUSED(MMF_PRO_GATENORM, MMF_EPI_STORE)
    DL_FUSED(MMF_PRO_PRENORM, MMF_EPI_SWIGLU)
    DL_FUSED(MMF_PRO_QUANT, MMF_EPI_STORE)
    DL_FUSED(MMF_PRO_PRENORM, MMF_EPI_STORE)
#undef DL_FUSED
#undef DL_K
    return mmf_set_error(MMF_ERR_BAD_ARG, "mmf_decode_linear: prologue %d with epilogue %d is not provided", a.prologue, a.epilogue);
}

}  // namespace
