// BitLinear of a decode step in one kernel: row work before the contraction (prologue), the contraction, and what the next
// kernel would do first (epilogue).
//
// A decode step is a chain of dependent kernels, so its time is the number of links times what a link cannot go below: a
// kernel boundary (0.9 us with programmatic dependent launch) and a read of the previous kernel's rows across the L2 (0.7 us).
// A block of the model used to be eight links (row kernel, contraction, four times).  Here
//   * the gate math and state update of the token mixer and the MLP's silu(gate) * up run in the epilogue of the contraction
//     that produces their inputs (a CTA owns the i, f and g rows, or the gate and up rows, of the same channels), and
//   * for a few token rows every CTA repeats the row work that precedes the contraction — norms, statistics, int8 codes —
//     instead of waiting for a kernel that did it: the row work is latency, and the SMs would idle meanwhile.
// That leaves four links per block.  For more rows the codes come from a row kernel (prologue MMF_PRO_CODES).
//
// Contraction: mma.sync m16n8k32 (8-bit, int32 accumulators) with 16 weight rows on its M axis and 8 token rows on N.
// tcgen05 is not used: its 128-row tile needs a K split over a cluster to fill the GPU, and the exchange of the split's
// partial sums alone (2.4 us) is longer than this kernel's whole contraction at these sizes.  A CTA (one per SM) owns
// N / 148 output rows and all of K; the (256-column group, 16-row block) pairs of its share are dealt evenly to the warps.
// A lane's operands are contiguous: the packed layout gives it 16 bytes (64 weights of one row) per group and block, whose
// 2-bit fields need one mask per register; the order of K inside a group is permuted alike for weights and codes, which
// changes nothing in an integer sum.  Weights are fetched by cp.async into slots private to a lane before the
// grid-dependency wait.  Partial sums meet in shared memory by integer atomics (exact, so order does not matter).
#pragma once
#include "bitlinear.cuh"
#include "packed.cuh"

namespace {

constexpr int DL_TS = 20;               // accumulator words per (block, token): 16 rows, padded so that a warp's adds do not collide
constexpr int DL_FUSED_ROWS = MMF_DECODE_LINEAR_FUSED_MAX_M;   // token rows a CTA takes through the fused prologue

struct DlParams {
    mmf_decode_linear_args a;
    int KC, KG;                         // 64-column chunks, groups of four chunks
    int units, grid;                    // unit of work: two adjacent output rows (gates, swiglu: channels)
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
    double t[RW];
#pragma unroll
    for (int w = 0; w < RW; w += 2) {
        const double2 d = *reinterpret_cast<const double2*>(slot + w);
        t[w] = d.x;
        t[w + 1] = d.y;
    }
#pragma unroll
    for (int s = RW / 2; s > 0; s >>= 1)
#pragma unroll
        for (int w = 0; w < s; ++w) t[w] += t[w + s];
    return t[0];
}

template <int RT> struct __align__(16) DlScratch {      // per row; a member is written once per kernel
    double d0[RT / 32], d1[RT / 32];
    float f[3][RT / 32];
    int i[3][RT / 32];
};

// VW packed pairs (2 * VW values) per vector
template <int VW> struct DlVec { uint32_t v[VW]; };
template <int VW, typename T> __device__ __forceinline__ DlVec<VW> dl_load(const T* p) {
    DlVec<VW> r;
    if constexpr (VW == 4) {
        const uint4 t = *reinterpret_cast<const uint4*>(p);
        r.v[0] = t.x; r.v[1] = t.y; r.v[2] = t.z; r.v[3] = t.w;
    } else {
        const uint2 t = *reinterpret_cast<const uint2*>(p);
        r.v[0] = t.x; r.v[1] = t.y;
    }
    return r;
}
template <int VW, typename T> __device__ __forceinline__ void dl_store(T* p, const uint32_t (&o)[VW]) {
    if constexpr (VW == 4) *reinterpret_cast<uint4*>(p) = make_uint4(o[0], o[1], o[2], o[3]);
    else *reinterpret_cast<uint2*>(p) = make_uint2(o[0], o[1]);
}
template <int VW> __device__ __forceinline__ void dl_weights(const float* p, float2 (&w)[VW]) {
#pragma unroll
    for (int i = 0; i < VW; i += 2) {
        const float4 t = *reinterpret_cast<const float4*>(p + 2 * i);
        w[i] = make_float2(t.x, t.y);
        w[i + 1] = make_float2(t.z, t.w);
    }
}

// vector `it` of a thread starts at column c; NVT vectors of 2 * VW values cover a row of D values
#define DL_FOREACH(it, c) \
    _Pragma("unroll") for (int it = 0, c = rt * 2 * VW; it < NVT; ++it, c += RT * 2 * VW) if (c < D)

// Row prologue of row m = thread / RT (m < M <= TH / RT): codes of G projections into shared memory in the MMA's operand
// order, dq and (per-warp) code sums beside them.
template <typename T, int PRO, int G, int TH, int RT, int NVT, int VW>
__device__ __forceinline__ void dl_prologue(const DlParams& p, const float* snw, uint8_t* scodes, DlScratch<RT>& red, float (&s_dq)[3][DL_FUSED_ROWS],
                                            double inv_d) {
    const mmf_decode_linear_args& a = p.a;
    const int D = (int)a.K, m = threadIdx.x / RT, rt = threadIdx.x % RT, lane = threadIdx.x & 31, rw = rt >> 5;
    const T* x = reinterpret_cast<const T*>(a.x) + m * a.ld_x;
    const T* r = PRO != MMF_PRO_QUANT && a.residual ? reinterpret_cast<const T*>(a.residual) + m * a.ld_residual : nullptr;
    DlVec<VW> u[NVT], v[NVT];
    double s0 = 0.0, s1 = 0.0;
    DL_FOREACH(it, c) u[it] = dl_load<VW>(x + c);
    if (r) {
        DL_FOREACH(it, c) v[it] = dl_load<VW>(r + c);
    }
    if constexpr (PRO == MMF_PRO_PRENORM) {
        T* ro = a.residual_out && blockIdx.x == 0 ? reinterpret_cast<T*>(a.residual_out) + m * (int64_t)D : nullptr;
        const bool plain = !r || a.round_sum_first;        // what is normalised is a row of T values
        DL_FOREACH(it, c) {
            uint32_t o[VW];
#pragma unroll
            for (int i = 0; i < VW; ++i) {
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
            if (ro) dl_store<VW>(ro + c, o);
        }
        const float rstd = rstd_from_sumsq(dl_row_sum<TH, RT>(s0 + s1, red.d0), D, inv_d, a.eps_norm);
        s0 = s1 = 0.0;
        DL_FOREACH(it, c) {
            float2 w[VW];
            dl_weights<VW>(snw + c, w);
#pragma unroll
            for (int i = 0; i < VW; ++i) {
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
            for (int i = 0; i < VW; ++i) sumsq_pair<T>(u[it].v[i], s0, s1);
        }
        const float rstd = rstd_from_sumsq(dl_row_sum<TH, RT>(s0 + s1, red.d0), D, inv_d, a.eps_norm);
        s0 = s1 = 0.0;
        DL_FOREACH(it, c) {
            float2 w[VW];
            dl_weights<VW>(snw + c, w);
#pragma unroll
            for (int i = 0; i < VW; ++i) {
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
            for (int i = 0; i < VW; ++i) sumsq_pair<T>(u[it].v[i], s0, s1);
        }
    }
    // BitLinear prologue: y = (v * rstd) * w, absmax -> scale -> int8 codes
    const float rstd = rstd_from_sumsq(dl_row_sum<TH, RT>(s0 + s1, red.d1), D, inv_d, a.eps_bl);
    float am[G];
#pragma unroll
    for (int g = 0; g < G; ++g) am[g] = 0.0f;
    DL_FOREACH(it, c) {
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float2 w[VW];
            dl_weights<VW>(snw + g * D + c, w);
#pragma unroll
            for (int i = 0; i < VW; ++i) {
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
        for (int w = 0; w < RT / 32; w += 4) {
            const float4 f = *reinterpret_cast<const float4*>(&red.f[g][w]);
            t = fmaxf(fmaxf(t, f.x), fmaxf(f.y, fmaxf(f.z, f.w)));
        }
        s[g] = __fdiv_rn(127.0f, t);
        sum[g] = 0;
        if (rt == 0) s_dq[g][m] = __fdiv_rn(t, 127.0f);
    }
    DL_FOREACH(it, c) {
        // column c: group c / 256, lane quarter (c / 64) % 4, word (c / 16) % 4, byte c % 16
        uint8_t* dst = scodes + ((size_t)((c >> 8) * 4 + ((c >> 4) & 3)) * 16 + m * 4 + ((c >> 6) & 3)) * 16 + (c & 15);
#pragma unroll
        for (int g = 0; g < G; ++g) {
            float2 w[VW];
            dl_weights<VW>(snw + g * D + c, w);
            uint32_t word[VW / 2];
#pragma unroll
            for (int i = 0; i < VW / 2; ++i) {
                word[i] = codes4(__fmul2_rn(mul2(widen<T>(u[it].v[2 * i]), rstd), w[2 * i]),
                                 __fmul2_rn(mul2(widen<T>(u[it].v[2 * i + 1]), rstd), w[2 * i + 1]), s[g]);
                sum[g] = __dp4a((int)word[i], 0x01010101, sum[g]);
            }
            uint8_t* d = dst + (size_t)g * p.KG * 1024;
            if constexpr (VW == 4) *reinterpret_cast<uint2*>(d) = make_uint2(word[0], word[VW / 2 - 1]);
            else *reinterpret_cast<uint32_t*>(d) = word[0];
        }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
        const int t = __reduce_add_sync(0xffffffffu, sum[g]);
        if (lane == 0) red.i[g][rw] = t;
    }
}

__device__ __forceinline__ float dl_out(int acc, int rs, float scale) { return __fmul_rn((float)(acc - rs), scale); }

// TH threads; fused prologue: RT threads per row, NVT vectors of 2 * VW values per thread; NB groups of 8 token rows
template <typename T, int PRO, int EPI, int NB, int TH, int RT, int NVT, int VW>
__global__ void __launch_bounds__(TH, 2)
decode_linear_kernel(const __grid_constant__ DlParams p) {
    const mmf_decode_linear_args& a = p.a;
    constexpr bool FUSED = PRO != MMF_PRO_CODES;
    constexpr int G = EPI == MMF_EPI_GATES ? 3 : 1;          // projections (code sets)
    constexpr int TOK = 8 * NB, WARPS = TH / 32;
    constexpr int ROWS = TH / RT;                            // rows the prologue takes side by side
    constexpr int CONST_ROWS = FUSED ? DL_FUSED_ROWS : TOK;
    constexpr int BP = EPI == MMF_EPI_SWIGLU ? 4 : 8;        // units per block of 16 MMA rows (swiglu: 8 gate and 8 up rows)
    extern __shared__ __align__(16) uint8_t smem[];
    float* snw = reinterpret_cast<float*>(smem);             // norm weights of the prologue
    uint8_t* scodes = smem + p.smem_codes;                   // [G][KG][4 words][4 tokens x 4 quarters] 16-byte pieces
    int* acc = reinterpret_cast<int*>(smem + p.smem_acc);    // [blocks][TOK][DL_TS]
    uint4* wslot = reinterpret_cast<uint4*>(smem + p.smem_w);
    __shared__ DlScratch<RT> red[FUSED ? ROWS : 1];
    __shared__ float s_dq[3][DL_FUSED_ROWS];
    __shared__ float s_scale[G][CONST_ROWS];                 // dq * mean|w|
    __shared__ int s_rs[G][CONST_ROWS];                      // code sum (weights are stored + 1)

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, q = lane & 3;
    pdl_trigger();
    const int u0 = (int)((unsigned)blockIdx.x * (unsigned)p.units / (unsigned)p.grid),
              pairs = (int)((unsigned)(blockIdx.x + 1) * (unsigned)p.units / (unsigned)p.grid) - u0;   // units of this CTA
    const int nb = (pairs + BP - 1) / BP * G;                // blocks of this CTA; the last one may be partly empty
    const int items = nb * p.KG, i0 = warp * items / WARPS, i1 = (warp + 1) * items / WARPS;
    const int D = (int)a.K, M = (int)a.M;
    // Order of the (group of 256 columns, block) items.  8 tokens: by block, sums stay in registers until the block changes.
    // More: by group, so that the codes (16 registers per 8 tokens) are loaded once per group.
    struct Item {
        int kg, b, nb, KG;
        __device__ __forceinline__ void next() {
            if constexpr (NB == 1) { if (++kg == KG) { kg = 0; ++b; } }
            else { if (++b == nb) { b = 0; ++kg; } }
        }
    };
    const Item first = NB == 1 ? Item{i0 % p.KG, i0 / p.KG, nb, p.KG} : Item{i0 / nb, i0 % nb, nb, p.KG};

    // weight rows gq and gq + 8 of block b, 16 bytes (64 weights) of chunk 4 * kg + q; nullptr past the end of the CTA's rows or of K
    auto wptr = [&](const Item& it, int half) -> const uint4* {
        const int chunk = it.kg * 4 + q;
        const int r = EPI == MMF_EPI_SWIGLU ? it.b * 8 + gq : it.b / G * 16 + gq + 8 * half;   // row (channel) of the CTA
        int n = 2 * u0 + r;
        if constexpr (EPI == MMF_EPI_GATES) n += (it.b % 3) * D;                               // i | f | g of D rows each
        if constexpr (EPI == MMF_EPI_SWIGLU) n += half * (int)(a.N / 2);                       // gate rows, then up rows
        return chunk < p.KC && r < 2 * pairs
                   ? reinterpret_cast<const uint4*>(a.packed) + ((int64_t)(n >> 7) * p.KC + chunk) * MMF_TILE_ROWS + (n & 127) : nullptr;
    };
    {   // the weights do not depend on the preceding kernel: on their way before the grid-dependency wait
        Item it = first;
        const int n_pf = min(i1 - i0, p.pf);
        for (int k = 0; k < n_pf; ++k, it.next()) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                uint4* dst = wslot + ((size_t)(k * WARPS + warp) * 2 + half) * 32 + lane;
                const uint4* src = wptr(it, half);
                if (src) cp_async16(dst, src);
                else *dst = make_uint4(0, 0, 0, 0);          // all fields zero: no contribution
            }
        }
        cp_async_commit();
    }
    for (int i = tid; i < nb * TOK * DL_TS; i += TH) acc[i] = 0;
    // the thread that will combine scale and code sum of (projection cg, token cm)
    const int cg = tid / CONST_ROWS, cm = tid % CONST_ROWS;
    const bool has_const = cg < G && cm < M;
    const float ws = has_const ? a.w_scale[cg] : 0.0f;
    double inv_d = 0.0;
    if constexpr (FUSED) {
        auto stage = [&](float* dst, const float* src) {
            for (int i = tid * 4; i < D; i += TH * 4) {
                float4 w = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
                if (src) w = *reinterpret_cast<const float4*>(src + i);
                *reinterpret_cast<float4*>(dst + i) = w;
            }
        };
        float* dst = snw;
        if (PRO != MMF_PRO_QUANT) { stage(dst, a.norm_w); dst += D; }
#pragma unroll
        for (int g = 0; g < G; ++g) stage(dst + g * D, a.bl_norm_w[g]);
        inv_d = 1.0 / (double)D;
    }
    __syncthreads();
    pdl_wait();

    float2 h_pre = make_float2(0.0f, 0.0f);                  // gates: the state this thread will advance
    if constexpr (EPI == MMF_EPI_GATES) {
        if (tid < pairs * M) {
            const int m = tid / pairs, pr = tid - m * pairs;
            h_pre = *reinterpret_cast<const float2*>(a.state + (int64_t)m * D + (u0 + pr) * 2);
        }
    }
    if constexpr (FUSED) {
        if (tid / RT < M) dl_prologue<T, PRO, G, TH, RT, NVT, VW>(p, snw, scodes, red[tid / RT], s_dq, inv_d);
    } else if (has_const) {
        s_scale[cg][cm] = __fmul_rn(a.dq[(int64_t)cg * M + cm], ws);
        s_rs[cg][cm] = a.rowsum[(int64_t)cg * M + cm];
    }
    cp_async_wait_all();
    if constexpr (FUSED) {
        __syncthreads();                                     // codes complete
        if (has_const) {
            int t = 0;
#pragma unroll
            for (int w = 0; w < RT / 32; ++w) t += red[cm].i[cg][w];
            s_rs[cg][cm] = t;
            s_scale[cg][cm] = __fmul_rn(s_dq[cg][cm], ws);
        }
    }

    auto weights_of = [&](const Item& it, int k, uint32_t (&xa)[4], uint32_t (&xb)[4]) {
        uint4 wa, wb;
        if (k < p.pf) {
            const uint4* src = wslot + (size_t)(k * WARPS + warp) * 64 + lane;
            wa = src[0];
            wb = src[32];
        } else {                                             // more weights than the slots hold
            const uint4 *pa = wptr(it, 0), *pb = wptr(it, 1);
            wa = pa ? __ldg(pa) : make_uint4(0, 0, 0, 0);
            wb = pb ? __ldg(pb) : make_uint4(0, 0, 0, 0);
        }
        xa[0] = wa.x; xa[1] = wa.y; xa[2] = wa.z; xa[3] = wa.w;
        xb[0] = wb.x; xb[1] = wb.y; xb[2] = wb.z; xb[3] = wb.w;
    };
    auto codes_of = [&](int g, int kg, int t, uint32_t (&B)[4][4]) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
            uint4 c = make_uint4(0, 0, 0, 0);
            if constexpr (FUSED) {                           // tokens 4 - 7 do not exist
                if (lane < 16) c = *reinterpret_cast<const uint4*>(scodes + ((size_t)((g * p.KG + kg) * 4 + w) * 16 + lane) * 16);
            } else {
                const int m = t * 8 + gq, chunk = kg * 4 + q;
                if (m < M && chunk < p.KC) c = *reinterpret_cast<const uint4*>(a.q + ((int64_t)g * M + m) * D + chunk * MMF_TILE_K + w * 16);
            }
            B[w][0] = c.x; B[w][1] = c.y; B[w][2] = c.z; B[w][3] = c.w;
        }
    };
    auto add = [&](int b, int t, const int (&v)[4]) {
        int* d = acc + (b * TOK + t * 8 + 2 * q) * DL_TS + gq;
#pragma unroll
        for (int k = 0; k < 4; ++k) atomicAdd(d + (k & 1) * DL_TS + (k >> 1) * 8, v[k]);
    };
    if constexpr (NB == 1) {
        // the 2-bit fields stay where they are: field i of a byte counts 4^i, one accumulator per field, shifted back at the end
        int c[4][4] = {};
        Item it = first;
        for (int i = i0; i < i1; ++i) {
            uint32_t xa[4], xb[4], B[4][4];
            weights_of(it, i - i0, xa, xb);
            codes_of(EPI == MMF_EPI_GATES ? it.b % 3 : 0, it.kg, 0, B);
#pragma unroll
            for (int w = 0; w < 4; w += 2)
#pragma unroll
                for (int f = 0; f < 4; ++f) {
                    const uint32_t mask = 0x03030303u << (2 * f);
                    mma_u8s8(c[f], xa[w] & mask, xb[w] & mask, xa[w + 1] & mask, xb[w + 1] & mask, B[w][f], B[w + 1][f]);
                }
            const int b = it.b;
            it.next();
            if (it.b != b || i + 1 == i1) {
                int v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    v[k] = c[0][k] + (c[1][k] >> 2) + (c[2][k] >> 4) + (c[3][k] >> 6);
                    c[0][k] = c[1][k] = c[2][k] = c[3][k] = 0;
                }
                add(b, 0, v);
            }
        }
    } else {
        uint32_t B[NB][4][4];
        int have = -1;
        Item it = first;
        for (int i = i0; i < i1; ++i, it.next()) {
            const int g = EPI == MMF_EPI_GATES ? it.b % 3 : 0;
            if (it.kg * G + g != have) {
                have = it.kg * G + g;
#pragma unroll
                for (int t = 0; t < NB; ++t) codes_of(g, it.kg, t, B[t]);
            }
            uint32_t xa[4], xb[4];
            weights_of(it, i - i0, xa, xb);
            int c[NB][4] = {};
#pragma unroll
            for (int w = 0; w < 4; w += 2)
#pragma unroll
                for (int f = 0; f < 4; ++f) {
                    const uint32_t a0 = (xa[w] >> (2 * f)) & 0x03030303u, a1 = (xb[w] >> (2 * f)) & 0x03030303u,
                                   a2 = (xa[w + 1] >> (2 * f)) & 0x03030303u, a3 = (xb[w + 1] >> (2 * f)) & 0x03030303u;
#pragma unroll
                    for (int t = 0; t < NB; ++t) mma_u8s8(c[t], a0, a1, a2, a3, B[t][w][f], B[t][w + 1][f]);
                }
#pragma unroll
            for (int t = 0; t < NB; ++t) add(it.b, t, c[t]);
        }
    }
    __syncthreads();

    // ---- epilogue: a thread finishes two adjacent rows (channels) of a token
    for (int i = tid; i < pairs * M; i += TH) {
        const int m = M == 1 ? 0 : i / pairs, pr = i - m * pairs;
        // rows r, r + 1 of block b, rounded to T and packed
        auto value = [&](int b, int r, int g) {
            const int2 v = *reinterpret_cast<const int2*>(acc + (b * TOK + m) * DL_TS + r);
            return narrow<T>(make_float2(dl_out(v.x, s_rs[g][m], s_scale[g][m]), dl_out(v.y, s_rs[g][m], s_scale[g][m])));
        };
        if constexpr (EPI == MMF_EPI_STORE) {
            const int64_t n = (int64_t)(u0 + pr) * 2;
            const uint32_t o = value(pr >> 3, (pr & 7) * 2, 0);
            T* dst = reinterpret_cast<T*>(a.out) + m * a.ld_out + n;
            if (n + 2 <= a.N && (a.ld_out & 1) == 0) *reinterpret_cast<uint32_t*>(dst) = o;
            else
                for (int k = 0; k < 2 && n + k < a.N; ++k) dst[k] = reinterpret_cast<const T*>(&o)[k];
        } else if constexpr (EPI == MMF_EPI_SWIGLU) {
            // z = round(silu(round(gate)) * round(up)): block b holds 8 channels, rows 0-7 gate and 8-15 up
            const int b = pr >> 2, r = (pr & 3) * 2;
            const float2 gate = widen<T>(value(b, r, 0)), up = widen<T>(value(b, 8 + r, 0));
            *reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(a.out) + m * a.ld_out + (int64_t)(u0 + pr) * 2) = narrow<T>(silu_mul2(gate, up));
        } else {
            // token mixer of one new token (layers/hgrn_bit.py:113-125 of the reference with T = 1)
            const T* lb = reinterpret_cast<const T*>(a.lower_bound);
            const int unit = pr >> 3, r = (pr & 7) * 2, ch = (u0 + pr) * 2;
            float2* st = reinterpret_cast<float2*>(a.state + (int64_t)m * D + ch);
            float2 h = i == tid ? h_pre : *st;
            float2 xv = raw_gate_floor(widen<T>(value(unit * 3, r, 0))), f = raw_gate_floor(widen<T>(value(unit * 3 + 1, r, 1)));
            float2 lbv = make_float2(0.0f, 0.0f), oml = make_float2(1.0f, 1.0f);
            if (lb) {
                lbv = widen<T>(*reinterpret_cast<const uint32_t*>(lb + ch));
                oml = make_float2(round_to<T>(__fsub_rn(1.0f, lbv.x)), round_to<T>(__fsub_rn(1.0f, lbv.y)));
            }
            raw_gate_pair<T>(xv, f, lb != nullptr, lbv, oml);
            if (a.mask && !a.mask[m]) xv = make_float2(0.0f, 0.0f);      // a padding position contributes no input
            h.x = fmaf(f.x, h.x, xv.x);
            h.y = fmaf(f.y, h.y, xv.y);
            *st = h;
            *reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(a.out) + (int64_t)m * D + ch) = narrow<T>(h);
            *reinterpret_cast<uint32_t*>(reinterpret_cast<T*>(a.g_out) + (int64_t)m * D + ch) = value(unit * 3 + 2, r, 2);
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

// arguments are checked by mmf_decode_linear
template <typename T> int decode_linear_launch(const mmf_decode_linear_args& a, cudaStream_t st) {
    DlParams p;
    p.a = a;
    p.KC = (int)(a.K / MMF_TILE_K);
    p.KG = (p.KC + 3) / 4;
    const int G = a.epilogue == MMF_EPI_GATES ? 3 : 1;
    // One CTA on every SM, however the rows divide: two kernels of the chain share an SM (the next one waits with its weights),
    // and an SM that this grid left empty would later take two CTAs of the next one, which then finishes late.
    p.units = a.epilogue == MMF_EPI_GATES ? (int)(a.K / 2) : a.epilogue == MMF_EPI_SWIGLU ? (int)(a.N / 4) : (int)((a.N + 1) / 2);
    p.grid = p.units < 148 ? p.units : 148;
    const int bp = a.epilogue == MMF_EPI_SWIGLU ? 4 : 8;
    const int nb = ((p.units + p.grid - 1) / p.grid + bp - 1) / bp * G;   // most blocks of one CTA
    const int NB = a.prologue == MMF_PRO_CODES ? (a.M <= 8 ? 1 : a.M <= 16 ? 2 : 4) : 1;
    // 16 warps of up to 64 registers; with 16 or 32 tokens' codes in registers 8 warps of up to 128.  Either way two kernels
    // fit on an SM, so that the next one fetches its weights while this one runs.
    const int threads = NB == 1 ? 512 : 256, warps = threads / 32;
    const int D = (int)a.K;
    int off = 0;
    p.smem_codes = 0;
    if (a.prologue != MMF_PRO_CODES) {
        off += (a.prologue == MMF_PRO_QUANT ? G : G + 1) * D * 4;
        p.smem_codes = off;
        off += G * p.KG * 1024;
    }
    p.smem_acc = off;
    off += (nb * 8 * NB * DL_TS * 4 + 15) / 16 * 16;
    p.smem_w = off;
    const int per_item = warps * 1024, want = (nb * p.KG + warps - 1) / warps;
    const int room = (DL_SMEM_MAX - off) / per_item;
    MMF_REQUIRE(room >= 1, MMF_ERR_BAD_SHAPE, "mmf_decode_linear: K=%lld does not fit in shared memory", (long long)a.K);
    p.pf = want < room ? want : room;
    const int smem = off + p.pf * per_item;

// vectors per thread for rows of at most 2048, 4096 and (plain quantisation) 8192 values
#define DL_NVT(PRO, EPI, RT, VW)                                                                                       \
    {                                                                                                                 \
        constexpr int S = 2048 / (2 * (VW)) / (RT);                                                                    \
        if (D <= 2048) return dl_go<decode_linear_kernel<T, PRO, EPI, 1, 512, RT, S, VW>>(p, threads, smem, st);        \
        if (D <= 4096) return dl_go<decode_linear_kernel<T, PRO, EPI, 1, 512, RT, 2 * S, VW>>(p, threads, smem, st);    \
        if constexpr (PRO == MMF_PRO_QUANT) return dl_go<decode_linear_kernel<T, PRO, EPI, 1, 512, RT, 4 * S, VW>>(p, threads, smem, st); \
        return mmf_set_error(MMF_ERR_BAD_SHAPE, "mmf_decode_linear: row of %d values", D);                             \
    }
#define DL_FUSED(PRO, EPI)                                  \
    if (a.prologue == PRO && a.epilogue == EPI) {           \
        if (a.M == 1) DL_NVT(PRO, EPI, 512, 2)              \
        else if (a.M == 2) DL_NVT(PRO, EPI, 256, 4)         \
        else DL_NVT(PRO, EPI, 128, 4)                       \
    }
    DL_FUSED(MMF_PRO_PRENORM, MMF_EPI_GATES)
    DL_FUSED(MMF_PRO_GATENORM, MMF_EPI_STORE)
    DL_FUSED(MMF_PRO_PRENORM, MMF_EPI_SWIGLU)
    DL_FUSED(MMF_PRO_QUANT, MMF_EPI_STORE)
    DL_FUSED(MMF_PRO_PRENORM, MMF_EPI_STORE)
#undef DL_FUSED
#undef DL_NVT
#define DL_CODES(EPI)                                                                                                  \
    if (a.prologue == MMF_PRO_CODES && a.epilogue == EPI) {                                                            \
        if (NB == 1) return dl_go<decode_linear_kernel<T, MMF_PRO_CODES, EPI, 1, 512, 512, 1, 4>>(p, threads, smem, st); \
        if (NB == 2) return dl_go<decode_linear_kernel<T, MMF_PRO_CODES, EPI, 2, 256, 256, 1, 4>>(p, threads, smem, st); \
        return dl_go<decode_linear_kernel<T, MMF_PRO_CODES, EPI, 4, 256, 256, 1, 4>>(p, threads, smem, st);              \
    }
    DL_CODES(MMF_EPI_GATES)
    DL_CODES(MMF_EPI_SWIGLU)
    DL_CODES(MMF_EPI_STORE)
#undef DL_CODES
    return mmf_set_error(MMF_ERR_BAD_ARG, "mmf_decode_linear: prologue %d with epilogue %d is not provided", a.prologue, a.epilogue);
}

}  // namespace
