// Row-wise kernels of a prompt (many token rows, 16-bit activations): one WARP per row, four where they all fit at once.
//
// The arithmetic is that of fused.cu (same rounding points, same operations, same bits); the layout is the one that long
// batches want.  A warp holds its whole row in registers as packed 16-bit pairs (D / 64 registers per lane) and widens a
// pair when it uses it, so that
//   * a row's reductions are warp shuffles and redux instructions: no block barrier, no shared-memory round trip, and the
//     per-row work every thread repeats (rstd, scales, the reductions themselves: about 200 instructions) is spread over
//     64 - 176 values per lane instead of 32 - 44 (fused.cu's layouts);
//   * the next row of the warp is on its way from memory (cp.async into slots that only this lane reads) while the current
//     one is normalised and quantised.
// Bound by memory on paper (one read of each input row, one write of each output row).  Measured at 32768 rows of 2048 bf16
// values, before -> after: three-projection prenorm 162 -> 140 us (4.3 TB/s), one-projection prenorm 92 -> 84 us (5.6 TB/s), gate
// norm 94 -> 79 us (4.2 TB/s); quantisation of 5632-value rows 386 -> 118 us (4.7 TB/s; it was the one-CTA-per-row kernel of
// rowwise.cu), 14 instructions per value instead of 22.  What is left: shared-memory wavefronts (the norm weights are read in
// every pass: pipe 87 / 79 / 67 / 80 % busy in those four) and issue (2.6 / 2.7 / 2.9 / 2.5 instructions per clock of 4).
#include "common.cuh"
#include "packed.cuh"
#include "rowquant.cuh"

namespace {

// Warps (= rows in flight) per CTA, one CTA per SM: the norm weights are staged once per SM and shared memory is left for the
// rows.  24 warps at 80 registers were 8 % slower than 16 at 128 (2048-value rows) and leave a nearly empty last wave earlier.
constexpr int WR_MAX_WARPS = 16;
constexpr int WR_ALL_WARPS = 32;              // ... of the form with four warps per row, whose lanes hold at most four vectors: 64 registers do
__host__ __device__ constexpr int wr_max_warps(int W) { return W > 1 ? WR_ALL_WARPS : WR_MAX_WARPS; }
constexpr size_t WR_SMEM_MAX = 224 * 1024;    // of 227 KB; the rest is static
constexpr int V = 8;                          // values per 16-byte vector
// Rows of at most 2048 values take the short forms of division and root (32768 rows: gate norm 78 -> 71 us, quantisation 43 -> 35).  The
// general ones branch, and without those branches between the passes the compiler reads a longer row's weights, and the prenorm's of more
// than four vectors per lane, ahead and spills (5632 values: 117 us -> 217; one-projection prenorm of 2048 83 -> 87).
__host__ __device__ constexpr bool lean(int NV) { return NV <= 8; }
__host__ __device__ constexpr bool lean_prenorm(int NV) { return NV <= 4; }

// Between two passes over a packed row: the compiler would keep the widened values of the first pass for the second, twice
// as many registers as the packed row (at 22 vectors per lane it spilled 560 bytes, now none), instead of widening again.
// Longer rows still spill a little: the quantisation 64 - 72 bytes at 26 and 28 vectors (rows above 6144 values), the prenorm 4 - 40
// bytes at 12 - 16 (rows above 2560 values).
template <int NV> __device__ __forceinline__ void forget_widened(uint32_t (&u)[NV][4]) {
#pragma unroll
    for (int it = 0; it < NV; ++it)
#pragma unroll
        for (int i = 0; i < 4; ++i) asm volatile("" : "+r"(u[it][i]));
}

// The W warps of a row (lane: 0 .. 32 W - 1): vector `it` of a lane starts at column c = (it * 32 W + lane) * 8.  NV is the even number
// of vectors per lane that holds a row of D values, so only the last two vectors can lie (partly) past its end.
#define WR_FOREACH(it, c) \
    _Pragma("unroll") for (int it = 0, c = lane * V; it < NV; ++it, c += 32 * W * V) if (it < NV - 2 || c < D)

// Where a row's warps meet (W > 1): each leaves its part, and after their barrier every one folds all of them.  Consecutive meetings use
// different arrays, so a part is overwritten only after a barrier that follows its last reader.
struct RowScratch {
    double d[2][WR_ALL_WARPS];
    float f[WR_ALL_WARPS];
    int i[WR_ALL_WARPS];
};
// (barrier 0 is also that of __syncthreads, which no warp calls once it has begun a row)
template <int W> __device__ __forceinline__ void row_sync() {
    if constexpr (W > 1) asm volatile("bar.sync %0, %1;" ::"r"((int)(threadIdx.x / (32 * W))), "n"(32 * W) : "memory");
}
template <int W> __device__ __forceinline__ double row_sum(double v, double* part) {
    v = warp_sum(v);
    if constexpr (W > 1) {
        const int w = threadIdx.x >> 5;
        if ((threadIdx.x & 31) == 0) part[w] = v;
        row_sync<W>();
        v = part[w / W * W];
#pragma unroll
        for (int k = 1; k < W; ++k) v += part[w / W * W + k];
    }
    return v;
}

__device__ __forceinline__ void stage(float* dst, const float* src, int n) {
    for (int i = threadIdx.x * 4; i < n; i += blockDim.x * 4) {
        float4 v = make_float4(1.0f, 1.0f, 1.0f, 1.0f);
        if (src) v = *reinterpret_cast<const float4*>(src + i);
        *reinterpret_cast<float4*>(dst + i) = v;
    }
}

// First row of slot `wid` of this CTA; `step` rows are in flight.  Spread evenly over the CTAs while the passes are few: an SM left without
// rows in the last one is given several CTAs of the next kernel, which waits for the slowest (3000 rows launched back to back, gate norm
// 12.3 -> 10.1 us).  Neighbours where the last pass counts little (32768 rows: spread 2 - 4 % slower).
__device__ __forceinline__ int64_t wr_first(int64_t M, int64_t step, int wid) {
    return M < 8 * step ? (int64_t)wid * gridDim.x + blockIdx.x : blockIdx.x * (step / gridDim.x) + wid;
}

// BitLinear prologue of the packed row u: y = (v * rstd) * w, absmax -> scale -> int8 codes, dq, code sum
template <typename T, int NV, int W, bool LEAN>
__device__ __forceinline__ void warp_quant(uint32_t (&u)[NV][4], int D, float rstd, const float* sw, int8_t* qr, float* dq,
                                           int32_t* rowsum, int lane, RowScratch& red) {
    float am0 = 0.0f, am1 = 0.0f;
    forget_widened<NV>(u);
    WR_FOREACH(it, c) {
        float2 w[4];
        lds8(sw + c, w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 y = __fmul2_rn(mul2(widen<T>(u[it][i]), rstd), w[i]);
            am0 = fmaxf(am0, fabsf(y.x));
            am1 = fmaxf(am1, fabsf(y.y));
        }
    }
    // non-negative floats order like their bit patterns
    float a = fmaxf(__uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(fmaxf(am0, am1)))), 1e-5f);
    const int wid = threadIdx.x >> 5, w0 = wid / W * W;
    if constexpr (W > 1) {
        if ((lane & 31) == 0) red.f[wid] = a;
        row_sync<W>();
#pragma unroll
        for (int k = 0; k < W; ++k) a = fmaxf(a, red.f[w0 + k]);
    }
    const float s = LEAN ? q127_over(a) : __fdiv_rn(127.0f, a);
    int lsum = 0;
    forget_widened<NV>(u);
    WR_FOREACH(it, c) {
        float2 w[4];
        lds8(sw + c, w);
        uint32_t word[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            word[h] = codes4(__fmul2_rn(mul2(widen<T>(u[it][2 * h]), rstd), w[2 * h]),
                             __fmul2_rn(mul2(widen<T>(u[it][2 * h + 1]), rstd), w[2 * h + 1]), s);
            lsum = __dp4a((int)word[h], 0x01010101, lsum);
        }
        *reinterpret_cast<uint2*>(qr + c) = make_uint2(word[0], word[1]);
    }
    lsum = __reduce_add_sync(0xffffffffu, lsum);
    if constexpr (W > 1) {
        if ((lane & 31) == 0) red.i[wid] = lsum;
        row_sync<W>();
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 1; k < W; ++k) lsum += red.i[w0 + k];
        *dq = LEAN ? over_127(a) : __fdiv_rn(a, 127.0f);
        *rowsum = lsum;
    }
}

// ---- RMSNorm + quantisation of given rows (mmf_act_quant)
template <typename T, int NV, int W>
__global__ void __launch_bounds__(wr_max_warps(W) * 32, 1)
warp_act_quant_kernel(const T* __restrict__ x, int64_t ld, const float* __restrict__ nw, int use_norm, float eps,
                      int8_t* __restrict__ q, float* __restrict__ dq, int32_t* __restrict__ rowsum, int64_t M, int D) {
    extern __shared__ __align__(16) float sw[];   // [D] norm weight, then per warp one row in flight
    pdl_trigger();
    stage(sw, use_norm ? nw : nullptr, D);
    const double inv_d = 1.0 / (double)D;
    pdl_wait();
    __syncthreads();
    __shared__ RowScratch red;
    const int lane = threadIdx.x % (32 * W), wid = threadIdx.x / (32 * W);      // in the row; row of the CTA
    T* sx = reinterpret_cast<T*>(sw + D) + (size_t)wid * D;
    auto fetch = [&](int64_t row) {
        WR_FOREACH(it, c) cp_async16(sx + c, x + row * ld + c);
        cp_async_commit();
    };
    const int64_t step = (int64_t)gridDim.x * (int)(blockDim.x / (32 * W));
    int64_t m = wr_first(M, step, wid);
    if (m < M) fetch(m);
    for (; m < M; m += step) {
        cp_async_wait_all();
        uint32_t u[NV][4] = {};
        double s0 = 0.0, s1 = 0.0;
        WR_FOREACH(it, c) {
            const uint4 r = *reinterpret_cast<const uint4*>(sx + c);
            u[it][0] = r.x; u[it][1] = r.y; u[it][2] = r.z; u[it][3] = r.w;
#pragma unroll
            for (int i = 0; i < 4; ++i) sumsq_pair<T>(u[it][i], s0, s1);
        }
        if (m + step < M) fetch(m + step);          // this lane's slots have just been read
        const float rstd = use_norm ? rstd_from_sumsq<lean(NV)>(row_sum<W>(s0 + s1, red.d[0]), D, inv_d, eps) : 1.0f;   // v * 1 * 1 is v itself
        warp_quant<T, NV, W, lean(NV)>(u, D, rstd, sw, q + m * (int64_t)D, dq + m, rowsum + m, lane, red);
    }
}

// ---- [x + residual] -> residual_out; RMSNorm -> T; G BitLinear prologues
template <typename T, int NV, int W>
__global__ void __launch_bounds__(wr_max_warps(W) * 32, 1)
warp_prenorm_quant_kernel(PrenormArgs a) {
    extern __shared__ __align__(16) float sw[];   // [1 + G][D] norm weights, then per warp an x row and a residual row in flight
    const int D = a.D;
    pdl_trigger();
    stage(sw, a.norm_w, D);
    for (int g = 0; g < a.G; ++g) stage(sw + (1 + g) * D, a.nws[g], D);
    const double inv_d = 1.0 / (double)D;
    pdl_wait();
    __syncthreads();
    __shared__ RowScratch red;
    const int lane = threadIdx.x % (32 * W), wid = threadIdx.x / (32 * W);      // in the row; row of the CTA
    T* sx = reinterpret_cast<T*>(sw + (1 + a.G) * D) + (size_t)wid * 2 * D;
    T* sr = sx + D;
    const T* x = reinterpret_cast<const T*>(a.x);
    const T* res = reinterpret_cast<const T*>(a.res);
    auto fetch = [&](int64_t row) {
        WR_FOREACH(it, c) {
            cp_async16(sx + c, x + row * a.ld_x + c);
            if (res) cp_async16(sr + c, res + row * a.ld_res + c);
        }
        cp_async_commit();
    };
    const int64_t step = (int64_t)gridDim.x * (int)(blockDim.x / (32 * W));
    int64_t m = wr_first(a.M, step, wid);
    if (m < a.M) fetch(m);
    for (; m < a.M; m += step) {
        cp_async_wait_all();
        T* ro = a.res_out ? reinterpret_cast<T*>(a.res_out) + m * (int64_t)D : nullptr;
        T* yo = a.y_out ? reinterpret_cast<T*>(a.y_out) + m * (int64_t)D : nullptr;
        uint32_t u[NV][4] = {};
        double s0 = 0.0, s1 = 0.0;
        if (!res || a.round_sum_first) {              // what is normalised is a row of T values
            WR_FOREACH(it, c) {
                const uint4 r = *reinterpret_cast<const uint4*>(sx + c);
                u[it][0] = r.x; u[it][1] = r.y; u[it][2] = r.z; u[it][3] = r.w;
                if (res) {
                    const uint4 q4 = *reinterpret_cast<const uint4*>(sr + c);
                    const uint32_t b[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) u[it][i] = narrow<T>(__fadd2_rn(widen<T>(u[it][i]), widen<T>(b[i])));
                }
                if (ro) *reinterpret_cast<uint4*>(ro + c) = make_uint4(u[it][0], u[it][1], u[it][2], u[it][3]);
#pragma unroll
                for (int i = 0; i < 4; ++i) sumsq_pair<T>(u[it][i], s0, s1);
            }
        } else {                                      // the fp32 sum is normalised: it is formed again from the two rows below
            WR_FOREACH(it, c) {
                const uint4 r = *reinterpret_cast<const uint4*>(sx + c);
                const uint4 q4 = *reinterpret_cast<const uint4*>(sr + c);
                const uint32_t xa[4] = {r.x, r.y, r.z, r.w}, xb[4] = {q4.x, q4.y, q4.z, q4.w};
                uint32_t o[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float2 t = __fadd2_rn(widen<T>(xa[i]), widen<T>(xb[i]));
                    s0 = fma((double)t.x, (double)t.x, s0);
                    s1 = fma((double)t.y, (double)t.y, s1);
                    o[i] = narrow<T>(t);
                }
                if (ro) *reinterpret_cast<uint4*>(ro + c) = make_uint4(o[0], o[1], o[2], o[3]);
            }
        }
        const float rstd1 = rstd_from_sumsq<lean_prenorm(NV)>(row_sum<W>(s0 + s1, red.d[0]), D, inv_d, a.eps_norm);
        s0 = s1 = 0.0;
        forget_widened<NV>(u);
        if (!res || a.round_sum_first) {
            WR_FOREACH(it, c) {
                float2 w[4];
                lds8(sw + c, w);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    u[it][i] = narrow<T>(__fmul2_rn(mul2(widen<T>(u[it][i]), rstd1), w[i]));
                    sumsq_pair<T>(u[it][i], s0, s1);
                }
            }
        } else {
            WR_FOREACH(it, c) {
                const uint4 r = *reinterpret_cast<const uint4*>(sx + c);
                const uint4 q4 = *reinterpret_cast<const uint4*>(sr + c);
                const uint32_t xa[4] = {r.x, r.y, r.z, r.w}, xb[4] = {q4.x, q4.y, q4.z, q4.w};
                float2 w[4];
                lds8(sw + c, w);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    u[it][i] = narrow<T>(__fmul2_rn(mul2(__fadd2_rn(widen<T>(xa[i]), widen<T>(xb[i])), rstd1), w[i]));
                    sumsq_pair<T>(u[it][i], s0, s1);
                }
            }
        }
        if (m + step < a.M) fetch(m + step);          // this lane's slots have been read for the last time
        if (yo) {
            WR_FOREACH(it, c) *reinterpret_cast<uint4*>(yo + c) = make_uint4(u[it][0], u[it][1], u[it][2], u[it][3]);
        }
        if (a.G == 0) { row_sync<W>(); continue; }
        const float rstd2 = rstd_from_sumsq<lean_prenorm(NV)>(row_sum<W>(s0 + s1, red.d[1]), D, inv_d, a.eps_bl);
        for (int g = 0; g < a.G; ++g) {
            const int64_t gm = (int64_t)g * a.M + m;
            warp_quant<T, NV, W, lean_prenorm(NV)>(u, D, rstd2, sw + (1 + g) * D, a.q + gm * D, a.dq + gm, a.rowsum + gm, lane, red);
        }
    }
}

// ---- RMSNorm(g) * w * o * sigmoid(o) -> T; BitLinear prologue
template <typename T, int NV, int W>
__global__ void __launch_bounds__(wr_max_warps(W) * 32, 1)
warp_gatenorm_quant_kernel(const T* __restrict__ gx, int64_t ld_g, const T* __restrict__ o, int64_t ld_o,
                           const float* __restrict__ gw, float eps_g, const float* __restrict__ nw, float eps_bl,
                           int8_t* __restrict__ q, float* __restrict__ dq, int32_t* __restrict__ rowsum, int64_t M, int D) {
    extern __shared__ __align__(16) float sw[];   // [2][D] norm weights, then per warp a g row and an o row in flight
    pdl_trigger();
    stage(sw, gw, D);
    stage(sw + D, nw, D);
    const double inv_d = 1.0 / (double)D;
    pdl_wait();
    __syncthreads();
    __shared__ RowScratch red;
    const int lane = threadIdx.x % (32 * W), wid = threadIdx.x / (32 * W);      // in the row; row of the CTA
    T* sg = reinterpret_cast<T*>(sw + 2 * D) + (size_t)wid * 2 * D;
    T* so = sg + D;
    auto fetch = [&](int64_t row) {
        WR_FOREACH(it, c) {
            cp_async16(sg + c, gx + row * ld_g + c);
            cp_async16(so + c, o + row * ld_o + c);
        }
        cp_async_commit();
    };
    const int64_t step = (int64_t)gridDim.x * (int)(blockDim.x / (32 * W));
    int64_t m = wr_first(M, step, wid);
    if (m < M) fetch(m);
    for (; m < M; m += step) {
        cp_async_wait_all();
        uint32_t u[NV][4] = {};
        double s0 = 0.0, s1 = 0.0;
        WR_FOREACH(it, c) {
            const uint4 r = *reinterpret_cast<const uint4*>(sg + c);
            u[it][0] = r.x; u[it][1] = r.y; u[it][2] = r.z; u[it][3] = r.w;
#pragma unroll
            for (int i = 0; i < 4; ++i) sumsq_pair<T>(u[it][i], s0, s1);
        }
        const float rstd1 = rstd_from_sumsq<lean(NV)>(row_sum<W>(s0 + s1, red.d[0]), D, inv_d, eps_g);
        s0 = s1 = 0.0;
        forget_widened<NV>(u);
        WR_FOREACH(it, c) {
            const uint4 r = *reinterpret_cast<const uint4*>(so + c);
            const uint32_t ob[4] = {r.x, r.y, r.z, r.w};
            float2 w[4];
            lds8(sw + c, w);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float2 ov = widen<T>(ob[i]);
                const float2 y = __fmul2_rn(mul2(widen<T>(u[it][i]), rstd1), w[i]);
                u[it][i] = narrow<T>(__fmul2_rn(__fmul2_rn(y, ov), sigmoid2(ov)));
                sumsq_pair<T>(u[it][i], s0, s1);
            }
        }
        if (m + step < M) fetch(m + step);            // this lane's slots have been read for the last time
        const float rstd2 = rstd_from_sumsq<lean(NV)>(row_sum<W>(s0 + s1, red.d[1]), D, inv_d, eps_bl);
        warp_quant<T, NV, W, lean(NV)>(u, D, rstd2, sw + D, q + m * (int64_t)D, dq + m, rowsum + m, lane, red);
    }
}

// One CTA per SM with up to wr_max_warps warps, as shared memory (weight_bytes once, row_bytes per row) allows, fewer when the rows
// are few: they are then spread over all SMs.
template <auto kernel, int W, typename... Args>
int wr_launch(size_t weight_bytes, size_t row_bytes, int64_t M, cudaStream_t st, const char* name, Args... args) {
    MMF_CUDA(mmf_allow_smem<kernel>((int)WR_SMEM_MAX));
    const int64_t fit = (int64_t)((WR_SMEM_MAX - weight_bytes) / row_bytes), sms = mmf_sms(), share = (M + sms - 1) / sms;
    int64_t rows = fit < wr_max_warps(W) / W ? fit : wr_max_warps(W) / W;
    if (share < rows) rows = share;
    MMF_REQUIRE(rows >= 1, MMF_ERR_CUDA, "%s: a row of this length does not fit in shared memory", name);
    size_t smem = weight_bytes + (size_t)rows * row_bytes;
    // Short rows leave registers and shared memory for two CTAs, and an SM that the kernel before leaves early would be given two while
    // others get none (12000 rows of 256 values to 1408 outputs 27.4 us, 24.9 with one): more than half of the shared memory each.
    if (share > rows && smem < WR_SMEM_MAX / 2 + 4096) smem = WR_SMEM_MAX / 2 + 4096;
    MMF_CUDA(mmf_launch_pdl(kernel, dim3((unsigned)(M < sms ? M : sms)), dim3((unsigned)rows * 32 * W), smem, st, args...));
    MMF_LAUNCH_CHECK(name);
    return MMF_OK;
}

constexpr int wr_vectors(int64_t D, int W) { return (int)((D + 512 * W - 1) / (512 * W)) * 2; }
// Four warps per row: five to eight rows per SM, all in flight at once, of 513 - 4096 values.  Between other kernels the latency of a row
// counts, which is what a pass over 64 values per lane takes.  Prompt passes of 24 blocks, 2048 wide, us with a CTA / one warp / two /
// four per row: 592 tokens 2475 / 2630 / - / 2528, 700 2581 / 2780 / 2748 / 2565, 999 2957 / 3059 / 3065 / 2901, 1184 - / 3171 / 3208 /
// 3010; more rows than fit at once, 1600 - / 3573 / 3542 / 3609, 2368 - / 4499 / 4554 / 4557.
inline bool wr_four(int64_t M, int64_t D) {
    const int64_t sms = mmf_sms();
    return D > 512 && D <= 4096 && M > 4 * sms && M <= 8 * sms;
}
// run `...` with W bound to the warps per row and NV to the even number of 256 W-value vectors per lane that holds a row of D values
#define WR_CASE(N, ...) case N: { constexpr int NV = N; __VA_ARGS__; break; }
#define WR_LAST(N, ...) default: { constexpr int NV = N; __VA_ARGS__; }
#define WR_DISPATCH16(M, D, ...)                                                                                    \
    if (wr_four(M, D)) {                                                                                             \
        constexpr int W = 4;                                                                                         \
        switch (wr_vectors(D, W)) { WR_CASE(2, __VA_ARGS__) WR_LAST(4, __VA_ARGS__) }                                \
    } else {                                                                                                         \
        constexpr int W = 1;                                                                                         \
        switch (wr_vectors(D, W)) {                                                                                  \
            WR_CASE(2, __VA_ARGS__) WR_CASE(4, __VA_ARGS__) WR_CASE(6, __VA_ARGS__) WR_CASE(8, __VA_ARGS__)           \
            WR_CASE(10, __VA_ARGS__) WR_CASE(12, __VA_ARGS__) WR_CASE(14, __VA_ARGS__) WR_LAST(16, __VA_ARGS__)       \
        }                                                                                                            \
    }
#define WR_DISPATCH28(M, D, ...)                                                                                    \
    if (wr_four(M, D)) {                                                                                             \
        constexpr int W = 4;                                                                                         \
        switch (wr_vectors(D, W)) { WR_CASE(2, __VA_ARGS__) WR_LAST(4, __VA_ARGS__) }                                \
    } else {                                                                                                         \
        constexpr int W = 1;                                                                                         \
        switch (wr_vectors(D, W)) {                                                                                  \
            WR_CASE(2, __VA_ARGS__) WR_CASE(4, __VA_ARGS__) WR_CASE(6, __VA_ARGS__) WR_CASE(8, __VA_ARGS__)           \
            WR_CASE(10, __VA_ARGS__) WR_CASE(12, __VA_ARGS__) WR_CASE(14, __VA_ARGS__) WR_CASE(16, __VA_ARGS__)       \
            WR_CASE(18, __VA_ARGS__) WR_CASE(20, __VA_ARGS__) WR_CASE(22, __VA_ARGS__) WR_CASE(24, __VA_ARGS__)       \
            WR_CASE(26, __VA_ARGS__) WR_LAST(28, __VA_ARGS__)                                                        \
        }                                                                                                            \
    }
#define WR_DISPATCH_T(dtype, T, ...)                                              \
    if ((dtype) == MMF_BF16) { using T = __nv_bfloat16; __VA_ARGS__; }            \
    else { using T = __half; __VA_ARGS__; }

}  // namespace

bool row_warp_takes(int64_t M, int64_t D, int dtype, int64_t max_d) {
    return dtype != MMF_F32 && D <= max_d && (M >= ROW_WARP_MIN_M || wr_four(M, D));
}

int warp_act_quant_launch(const void* x, int dtype, int64_t ld, const float* nw, int use_norm, float eps, int8_t* q, float* dq,
                          int32_t* rowsum, int64_t M, int64_t D, cudaStream_t st) {
    const size_t weights = (size_t)D * 4, row = (size_t)D * 2;
    WR_DISPATCH_T(dtype, T, {
        WR_DISPATCH28(M, D, { return wr_launch<warp_act_quant_kernel<T, NV, W>, W>(weights, row, M, st, "warp_act_quant_kernel",
                                                          (const T*)x, ld, nw, use_norm, eps, q, dq, rowsum, M, (int)D); });
    });
    return MMF_OK;
}

int warp_prenorm_quant_launch(const PrenormArgs& a, int dtype, cudaStream_t st) {
    const size_t weights = (size_t)(1 + a.G) * a.D * 4, row = (size_t)a.D * 4;
    WR_DISPATCH_T(dtype, T, {
        WR_DISPATCH16(a.M, a.D, { return wr_launch<warp_prenorm_quant_kernel<T, NV, W>, W>(weights, row, a.M, st,
                                                               "warp_prenorm_quant_kernel", a); });
    });
    return MMF_OK;
}

int warp_gatenorm_quant_launch(const void* g, int64_t ld_g, const void* o, int64_t ld_o, int dtype, const float* gw, float eps_g,
                               const float* nw, float eps_bl, int8_t* q, float* dq, int32_t* rowsum, int64_t M, int64_t D, cudaStream_t st) {
    const size_t weights = (size_t)D * 8, row = (size_t)D * 4;
    WR_DISPATCH_T(dtype, T, {
        WR_DISPATCH16(M, D, { return wr_launch<warp_gatenorm_quant_kernel<T, NV, W>, W>(weights, row, M, st,
                                                               "warp_gatenorm_quant_kernel", (const T*)g, ld_g, (const T*)o, ld_o,
                                                               gw, eps_g, nw, eps_bl, q, dq, rowsum, M, (int)D); });
    });
    return MMF_OK;
}
