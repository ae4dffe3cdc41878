// All blocks of a decode step in one resident kernel: one CTA per SM for the whole step (cooperative launch), rows handed from CTA to
// CTA through words of global memory instead of through kernel boundaries.
//
// A step is a chain of four links per block (mixer projections + gates, o_proj, gate_proj + swiglu, down_proj).  As kernels
// (decode_linear.cuh) a link of one row takes 4.3 us, of which 1.6 are the hand-over: the boundary and the first read across the L2.
// Here an epilogue stores its outputs as they are and the next link's readers poll them: a 32-bit word of a row cannot be two 0xffff (no
// rounding produces that NaN), of codes not four times -128 (codes are -127 .. 127), so a word that differs from the fill has arrived and
// needs no flag, fence or counter.  Every word is written once per step; a kernel in front makes them all absent.
//
// The exchange alone (148 CTAs, each stores 28 bytes and reads 4 KB): 0.7 us if the first look comes 400 - 600 clocks after the stores,
// 2.0 us if at once, because polls of all SMs for the same lines queue in front of the stores.  What a link prepares (weights unpacked
// into registers, states read) fills that time; a wait on top of it changes nothing up to 1000 clocks.  A counter barrier took 1.6 us, with
// flags in the words (8-byte pairs) 1.0, through clusters' shared memory 1.0.
//
// Weights come from a copy laid out for this kernel (decode_step.cu): a CTA's rows of a link are contiguous, one bulk copy, four links
// ahead; fetched with cp.async from the tiles of the other kernels, address arithmetic and issue were a quarter of the step.
//
// What bounds it now is the number of instructions in a row's life: alone on one SM with all inputs present a block takes 21.9 k clocks,
// in the step 22.9 k (2048 wide, MLP 5632), at about one instruction per six clocks and warp (dependent arithmetic), and it does not get
// shorter with more warps.  So: one copy of the code for all four links (unrolled per link it was 120 KB, beyond every instruction cache,
// and a step took 674 us; code that leaves the 32 KB cache by branches costs up to twice the time), fp64 sums by the tensor core, the three
// IEEE roundings of the row arithmetic without the general division, operand pairs of the codes stored side by side.
// Step of a 24-block, 2048-wide model, kernels / this, in turn in one process: 1 row 413 / 304 us, 2 rows 478 / 440, 4 rows 516 / 454, 8 rows
// 516 / 465, 9 rows 622 / 518, 16 rows 655 / 559; 32 blocks of 2560: 1 row 666 / 560, 2 rows 804 / 689, 4 rows 814 / 711, 8 rows 816 / 736.
#pragma once
#include "decode_linear.cuh"
#include "decode_step_plan.cuh"

// Timeline (experiments build): thread 0 of CTA 0 stamps every link with its clock.
#ifdef MMF_EXPERIMENTS
#define DS_TRACE(slot) do { if (trace) trace[slot] = clock64(); } while (0)
#define DS_TRACE_AFTER(slot, value) do { asm volatile("" ::"d"(value)); DS_TRACE(slot); } while (0)   // once `value` is formed
#else
#define DS_TRACE(slot) do { } while (0)
#define DS_TRACE_AFTER(slot, value) do { } while (0)
#endif

namespace {

__device__ __forceinline__ uint4 ds_ld(const void* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void ds_st(void* p, uint32_t v) { asm volatile("st.relaxed.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory"); }
__device__ __forceinline__ bool ds_there(uint4 v, uint32_t none) { return v.x != none && v.y != none && v.z != none && v.w != none; }
__device__ __forceinline__ uint32_t ds_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// A thread's side of the bounded waits.  One that runs out sets the status word; the others see it and stop waiting for rows and codes
// too.  For its own bulk copies (`barrier`) a CTA waits all the same, whatever other CTAs do: none is under way when it ends, and a
// region is not read or filled again before its copy is complete.
struct DsWait {
    const DsParams& p;
    bool dead = false;
#ifdef MMF_EXPERIMENTS
    __device__ __forceinline__ int limit() const { return p.wait_limit; }
#else
    __device__ __forceinline__ int limit() const { return DS_WAIT_LIMIT; }
#endif
    __device__ __forceinline__ void give_up() {        // the host's word too: it is read without synchronising
        *p.status = 1;
        if (p.gave_up) asm volatile("st.relaxed.sys.global.b32 [%0], %1;" ::"l"(p.gave_up), "r"(1) : "memory");
        dead = true;
    }
    __device__ __forceinline__ bool again(int& n) {    // another poll?
        if (dead) return false;
        if ((++n & 4095) == 0 || n >= limit()) {
            int s;
            asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(s) : "l"(p.status) : "memory");
            if (s || n >= limit()) {
                give_up();
                return false;
            }
        }
        return true;
    }
    __device__ __forceinline__ void barrier(uint32_t bar, int parity) {
        int n = 0;
        uint32_t done;
        do {
            asm volatile("{\n\t.reg .pred P1;\n\tmbarrier.try_wait.parity.shared::cta.b64 P1, [%1], %2;\n\tselp.b32 %0, 1, 0, P1;\n\t}"
                         : "=r"(done) : "r"(bar), "r"((uint32_t)parity) : "memory");
        } while (!done && ++n < DS_WAIT_LIMIT);
        if (!done) give_up();
    }
};
__device__ __forceinline__ void ds_expect(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ds_copy(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {      // one thread
    if (bytes)
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                     ::"r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// over the CTA
template <int NW> __device__ __forceinline__ double ds_sum(double s, double* slot) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    s = warp_sum(s);
    if (lane == 0) slot[warp] = s;
    __syncthreads();
    double t = slot[lane & 3];
#pragma unroll
    for (int o = 4; o < NW; o += 4)
        if (o + 4 <= NW || (lane & 3) < NW - o) t += slot[o + (lane & 3)];
    return mma_sum(t);
}
// fold the warps' entries of a 16-byte aligned array
template <int NW> __device__ __forceinline__ float ds_fold_max(const float* v) {
    float t = 1e-5f;
#pragma unroll
    for (int k = 0; k < NW; k += 2) {
        const float2 a = *reinterpret_cast<const float2*>(v + k);
        t = fmaxf(t, fmaxf(a.x, a.y));
    }
    return t;
}
template <int NW> __device__ __forceinline__ int ds_fold_sum(const int* v) {
    int t = 0;
#pragma unroll
    for (int k = 0; k < NW; k += 2) {
        const int2 a = *reinterpret_cast<const int2*>(v + k);
        t += a.x + a.y;
    }
    return t;
}

__device__ __forceinline__ void ds_mma(int (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1, int c0, int c1, int c2, int c3) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %11, %12, %13};"
                 : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(c0), "r"(c1), "r"(c2), "r"(c3));
}
// 16 weight rows x one column group: this lane's rows at wa and wb (64 weights each) as MMA operands.  A byte's 2-bit fields stay where
// they are (masked): one sum per field, shifted back at the end.
struct DsWeights { uint32_t a[8][4]; };                        // [word pair, field]
__device__ __forceinline__ void ds_unpack(DsWeights& o, const uint8_t* wa, const uint8_t* wb) {
    const uint4 a = *reinterpret_cast<const uint4*>(wa), b = *reinterpret_cast<const uint4*>(wb);
    const uint32_t xa[4] = {a.x, a.y, a.z, a.w}, xb[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int f = 0; f < 4; ++f) {
            const uint32_t msk = 0x03030303u << (2 * f);
            o.a[4 * k + f][0] = xa[2 * k] & msk;
            o.a[4 * k + f][1] = xb[2 * k] & msk;
            o.a[4 * k + f][2] = xa[2 * k + 1] & msk;
            o.a[4 * k + f][3] = xb[2 * k + 1] & msk;
        }
}
// Sums of a block over NB tiles of 8 tokens, to shared memory: [token][DS_TS], lane (gq, q) holds rows gq, gq + 8 of tokens 2 q, 2 q + 1.
// Piece 2 k + i of the codes x holds what fields 2 i and 2 i + 1 of the weight words 2 k and 2 k + 1 meet, as two operand pairs.
template <int NB, int MR> __device__ __forceinline__ void ds_block(int* dst, const DsWeights& w, const uint4 (&x)[NB][4], int q) {
    int acc[4][NB][4];
#pragma unroll
    for (int k = 0; k < 2; ++k)
#pragma unroll
        for (int f = 0; f < 4; ++f)
#pragma unroll
            for (int t = 0; t < NB; ++t) {
                const uint32_t(&a)[4] = w.a[4 * k + f];
                const uint4 v = x[t][2 * k + (f >> 1)];
                const uint32_t b0 = f & 1 ? v.z : v.x, b1 = f & 1 ? v.w : v.y;
                int(&c)[4] = acc[f][t];
                if (k == 0) ds_mma(c, a[0], a[1], a[2], a[3], b0, b1, 0, 0, 0, 0);
                else ds_mma(c, a[0], a[1], a[2], a[3], b0, b1, c[0], c[1], c[2], c[3]);
            }
    if (MR < 8 && 2 * q >= MR) return;
#pragma unroll
    for (int t = 0; t < NB; ++t)
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (MR >= 8 || (k & 1) < MR)
                dst[(t * 8 + (k & 1)) * DS_TS + (k >> 1) * 8] = acc[0][t][k] + (acc[1][t][k] >> 2) + (acc[2][t][k] >> 4) + (acc[3][t][k] >> 6);
}
template <typename T> __device__ __forceinline__ uint32_t ds_add16(uint32_t a, uint32_t b) {       // narrow(widen(a) + widen(b)): see raw_gate_pair
    if constexpr (cuda::std::is_same<T, __half>::value) {
        const __half2 r = __hadd2(*reinterpret_cast<const __half2*>(&a), *reinterpret_cast<const __half2*>(&b));
        return *reinterpret_cast<const uint32_t*>(&r);
    } else {
        const __nv_bfloat162 r = __hadd2(*reinterpret_cast<const __nv_bfloat162*>(&a), *reinterpret_cast<const __nv_bfloat162*>(&b));
        return *reinterpret_cast<const uint32_t*>(&r);
    }
}

// MR token rows.  FUSED (one row): every CTA does the row work, and codes never leave a warp: warp w makes the codes of the 256-column
// groups w, w + NW, ... and contracts them.  Otherwise (M <= MR, tiles of 8 tokens) a CTA per (row, projection) does the row work and
// hands the codes round; the contraction is split the same way.  A thread holds 8 columns of a hidden row (NW * 256 >= hidden), up to
// three times 8 of an inner row.  FUSED: the weights of a warp's first PRE (block, column group) items are unpacked into registers while
// the row is on its way (unpacking is two thirds of a product's time: 2.2 k clocks of a block; in the other form the code grew out of the
// instruction cache: a tenth slower at eight rows).
template <typename T, int MR, bool FUSED, int NW, int PRE>
__global__ void __launch_bounds__(NW * 32, 1)
decode_step_kernel(const __grid_constant__ DsParams p) {
    constexpr int TH = NW * 32, TL = FUSED ? 4 : 32, NB = FUSED ? 1 : MR / 8, NVI = 3;
    constexpr int STEP = FUSED ? 256 : NB * 2048;              // bytes of a column group's codes
    extern __shared__ __align__(128) uint8_t smem[];
    int* part = reinterpret_cast<int*>(smem + p.part_off);    // [block][column group][MR][DS_TS]
    __shared__ double s_sum[2][NW];
    __shared__ __align__(16) float s_max[3][NW];
    __shared__ float s_top[3];                                 // absmax by projection
    __shared__ __align__(16) int s_codes[3 * NW];              // code sums: mixer [projection][warp], else [column group]
    __shared__ float s_scale[3][MR];                           // not FUSED: scales and code sums
    __shared__ int s_rs[3][MR];
    __shared__ __align__(8) uint64_t s_bar[6];                 // weights of a link, norm weights of an even / odd link

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, gq = lane >> 2, q = lane & 3, bid = blockIdx.x;
    const int M = FUSED ? 1 : p.M, h = p.h, inner = p.inner, links = 4 * p.L;
    const int row_m = FUSED ? 0 : bid / 3, row_g = FUSED ? 0 : bid - row_m * 3;        // not FUSED: this CTA's row and projection
    const bool has_row = FUSED || row_m < M;
    // not FUSED: the CTAs of a row take turns with the links of one projection
    auto mine = [&](int type) { return FUSED || (has_row && (type == DS_IFG || row_g == (type == DS_O ? 1 : type == DS_GATE ? 0 : 2))); };
    const uint32_t bars = ds_smem(s_bar);
    DsWait wait{p};

    // one thread: weights of link idx into its region, norm weights into the region of even / odd links
    auto fetch = [&](int idx) {
        if (idx >= links) return;
        const int type = idx & 3;
        const DsSizes& z = p.size[type];
        const int bytes_per_pair = ds_rows_per_pair(type) * z.KG * 64, u0 = bid * z.base + min(bid, z.extra), pairs = z.base + (bid < z.extra ? 1 : 0);
        ds_expect(bars + type * 8, pairs * bytes_per_pair);
        ds_copy(ds_smem(smem + z.w_off), reinterpret_cast<const uint8_t*>(p.layer[idx >> 2].weights) + z.w_at + (int64_t)u0 * bytes_per_pair,
                pairs * bytes_per_pair, bars + type * 8);
    };
    auto fetch_norms = [&](int idx) {
        if (idx >= links) return;
        const int type = idx & 3;
        if (!mine(type)) return;
        const uint8_t* src = reinterpret_cast<const uint8_t*>(p.layer[idx >> 2].weights) + p.size[type].n_at;
        const uint32_t dst = ds_smem(smem + p.norm_off[idx & 1]), row = p.size[type].D * 4, bar = bars + 32 + (idx & 1) * 8;
        if (FUSED || type != DS_IFG) {
            ds_expect(bar, row * (type == DS_IFG ? 4 : type == DS_DOWN ? 1 : 2));
            ds_copy(dst, src, row * (type == DS_IFG ? 4 : type == DS_DOWN ? 1 : 2), bar);
        } else {                                               // of the projections' norms the CTA's own
            ds_expect(bar, row * 2);
            ds_copy(dst, src, row, bar);
            ds_copy(dst + row, src + (1 + row_g) * row, row, bar);
        }
    };
    if (tid == 0) {
        for (int i = 0; i < 6; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bars + i * 8) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
#pragma unroll 1
        for (int i = 0; i < 4; ++i) {
            if (i < 2) fetch_norms(i);
            fetch(i);
        }
    }
    __syncthreads();

    int norm_phase = 0;                                        // bit k: parity of the next wait for norm region k
    uint32_t xres[4] = {0, 0, 0, 0};                           // residual stream: this thread's columns
    const bool in_h = tid * 8 < h;
    // Codes of columns 8 lane .. + 7 of a group, row 0 of its tile: chunk lane / 8, weight word w = lane / 2 % 4, fields 2 (lane % 2) and the next
    const int code_at = ((((lane >> 2) & 1) * 2 + (lane & 1)) * TL + (lane >> 3)) * 16 + ((lane >> 1) & 1) * 4 +
                        (FUSED ? 0 : ((row_m >> 3) * 128 + (row_m & 7) * 4) * 16);

#pragma unroll 1
    for (int idx = 0; idx < links; ++idx) {
        const int type = idx & 3, l = idx >> 2, G = type == DS_IFG ? 3 : 1;
        const DsSizes& z = p.size[type];
        const int D = z.D, KG = z.KG, u0 = bid * z.base + min(bid, z.extra), pairs = z.base + (bid < z.extra ? 1 : 0), R = pairs * ds_rows_per_pair(type);
        T* xrows = reinterpret_cast<T*>(p.rows + (int64_t)l * p.rows_layer);
        const int64_t Mh = (int64_t)M * h;
        uint8_t* xcodes = FUSED ? smem : p.codes + (int64_t)l * p.codes_layer + z.codes_at;
        uint8_t* xscale = FUSED ? nullptr : p.codes + (int64_t)l * p.codes_layer + p.code_scales_at + (type == DS_IFG ? 0 : 2 + type) * MR * 8;
#ifdef MMF_EXPERIMENTS
        long long* trace = p.trace && tid == 0 && bid == 0 && idx < 1000 ? p.trace + 8 + 8 * idx : nullptr;
#endif
        DS_TRACE(0);
        // ---- while the row is on its way: what the epilogue will need.  Its lanes: lane vk * per + i of a warp works on the warp's i-th
        // (pair, token): value vk (i, f or g; gate or up), or every fourth partial sum of one value
        const int per = type == DS_IFG ? 10 : type == DS_GATE ? 16 : 8;
        const int vk = type == DS_IFG ? (lane >= 10 ? 1 : 0) + (lane >= 20 ? 1 : 0) : type == DS_GATE ? lane >> 4 : lane >> 3, item0 = warp * per + lane - vk * per;
        const int inv_pairs = MR == 1 ? 0 : (1 << 20) / max(pairs, 1) + 1;
        uint32_t lb_pre = 0;
        float2 h_pre = make_float2(0.0f, 0.0f);
        bool keep_pre = true;
        const T* lb = nullptr;
        if (type == DS_IFG && vk == 0 && item0 < pairs * M) {
            const int m = MR == 1 ? 0 : (item0 * inv_pairs) >> 20, ch = (u0 + item0 - m * pairs) * 2;
            lb = reinterpret_cast<const T*>(p.layer[l].lower_bound);
            if (lb) lb_pre = __ldg(reinterpret_cast<const uint32_t*>(lb + ch));
            h_pre = *reinterpret_cast<const float2*>(p.layer[l].state + (int64_t)m * h + ch);
            if (p.mask) keep_pre = p.mask[m] != 0;
        }
        // weight scale: FUSED, of the projection whose value this lane finishes; else of (projection, token)
        const int cg = FUSED ? (type == DS_IFG ? vk : 0) : tid / MR, cm = FUSED ? 0 : tid % MR;
        const bool has_const = FUSED || (cg < G && cm < M);
        float ws = 0.0f;
        if (has_const) ws = __ldg(reinterpret_cast<const float*>(reinterpret_cast<const uint8_t*>(p.layer[l].weights) + p.scales_at) + (type == DS_IFG ? cg : type + 2));
        // ---- items of this warp: block b of 16 weight rows (of a projection) x column group.  Mixer: the projections one after another; inner
        // row: the warp's groups; else one group
        const int nbp = type == DS_GATE ? (pairs + 3) / 4 : (pairs + 7) / 8;
        const int items = warp >= KG ? 0 : nbp * (type == DS_IFG ? 3 : type == DS_DOWN ? (KG - warp + NW - 1) / NW : 1);
        const int bs = type == DS_GATE ? 8 * 64 : 16 * 64, half = type == DS_GATE ? pairs * 128 : 8 * 64;
        // after the last block of a projection or group: on to the next
        const int next_w = (type == DS_DOWN ? NW * R * 64 : pairs * 128) - nbp * bs, next_d = (type == DS_DOWN ? NW - nbp * KG : 0) * (MR * DS_TS);
        const int next_c = (type == DS_DOWN ? NW : KG) * STEP;
        // (rows past the CTA's last one are whatever follows; nothing reads their sums)
        const uint8_t* wk = smem + z.w_off + (warp * R + gq) * 64 + q * 16;
        int bw = 0;
        [[maybe_unused]] DsWeights pre[PRE ? PRE : 1];
        auto unpack = [&](DsWeights& o) {
            ds_unpack(o, wk, wk + half);
            wk += bs;
            if (++bw == nbp) { bw = 0; wk += next_w; }
        };
        wait.barrier(bars + type * 8, l & 1);
        DS_TRACE(1);

        // ---- row work
        const bool me = mine(type);
        if (me) {
            wait.barrier(bars + 32 + (idx & 1) * 8, norm_phase >> (idx & 1) & 1);
            norm_phase ^= 1 << (idx & 1);
        }
        if (me || (type == DS_GATE && has_row)) {              // every holder of a residual row adds the attention output to it
            const float* w = reinterpret_cast<const float*>(smem + p.norm_off[idx & 1]) + (tid * 8 < D ? tid * 8 : 0);      // (a thread past the row's end reads its start)
            // up to three vectors of 8 values: of an inner row; of o and g; of one row
            uint4 v[NVI];
            {
                const T* src = xrows + (type == DS_DOWN ? 4 * Mh + (int64_t)row_m * inner : (int64_t)row_m * h) + tid * 8;
                if (type == DS_IFG) src += 3 * Mh - p.rows_layer / (int64_t)sizeof(T);       // MLP output of the block before
                if (type == DS_GATE) src += 2 * Mh;
                const T* src1 = src + (type == DS_DOWN ? TH * 8 : Mh);
                const bool use1 = type == DS_DOWN ? (TH + tid) * 8 < D : type == DS_O && in_h, use2 = type == DS_DOWN && (2 * TH + tid) * 8 < D, use0 = tid * 8 < D;
                if (idx == 0) {
                    int64_t row = row_m;
                    if (p.row_ids) {
                        row = p.row_ids[row];
                        row = row < 0 ? 0 : row >= p.x_rows ? p.x_rows - 1 : row;       // clamp instead of faulting on a bad id
                    }
                    src = reinterpret_cast<const T*>(p.x) + row * p.ld_x + tid * 8;
                }
                v[0] = v[1] = v[2] = make_uint4(0, 0, 0, 0);
                auto load = [&]() {
                    if (use0) v[0] = ds_ld(src);
                    if (use1) v[1] = ds_ld(src1);
                    if (use2) v[2] = ds_ld(src1 + TH * 8);
                };
                auto there = [&]() { return idx == 0 || (ds_there(v[0], DS_NO_ROW) && ds_there(v[1], DS_NO_ROW) && ds_there(v[2], DS_NO_ROW)); };    // (a table's values may be anything)
                load();
#pragma unroll
                for (int i = 0; i < PRE; ++i)                  // while the load is under way
                    if (i < items) unpack(pre[i]);
                int n = 0;
                while (!there() && wait.again(n)) load();
                __syncwarp();
            }
            DS_TRACE(2);
            double s0 = 0.0, s1 = 0.0;
            float rstd;
            if (type == DS_DOWN) {
#pragma unroll
                for (int it = 0; it < NVI; ++it) {
                    const uint32_t c[4] = {v[it].x, v[it].y, v[it].z, v[it].w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) sumsq_pair<T>(c[i], s0, s1);
                }
                if (me) rstd = rstd_from_sumsq(ds_sum<NW>(s0 + s1, s_sum[1]), D, z.inv_d, p.layer[l].eps_bl);
            } else {
                const uint32_t a[4] = {v[0].x, v[0].y, v[0].z, v[0].w}, b[4] = {v[1].x, v[1].y, v[1].z, v[1].w};
                uint32_t c[4];
                float2 t[4];
                if (type == DS_GATE) {                         // residual stream; the MLP normalises the fp32 sum, ...
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        t[i] = __fadd2_rn(widen<T>(a[i]), widen<T>(xres[i]));
                        xres[i] = ds_add16<T>(a[i], xres[i]);
                        s0 = fma((double)t[i].x, (double)t[i].x, s0);
                        s1 = fma((double)t[i].y, (double)t[i].y, s1);
                    }
                    if (l == p.L - 1 && (FUSED ? bid == 0 : row_g == 0) && in_h)
                        *reinterpret_cast<uint4*>(reinterpret_cast<T*>(p.residual_out) + (int64_t)row_m * h + tid * 8) = make_uint4(xres[0], xres[1], xres[2], xres[3]);
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (type == DS_IFG) xres[i] = idx ? ds_add16<T>(a[i], xres[i]) : a[i];      // ... the mixer its rounding
                        c[i] = type == DS_IFG ? xres[i] : b[i];
                        sumsq_pair<T>(c[i], s0, s1);
                        t[i] = widen<T>(c[i]);
                    }
                }
                if (me) {
                    float2 n[4], gate[4];
                    lds8(w, n);
                    if (type == DS_O) {
#pragma unroll
                        for (int i = 0; i < 4; ++i) gate[i] = sigmoid2(widen<T>(a[i]));
                    }
#pragma unroll 1
                    for (int pass = 0;; ++pass) {
                        rstd = rstd_from_sumsq(ds_sum<NW>(s0 + s1, s_sum[pass]), D, z.inv_d, pass ? p.layer[l].eps_bl : type == DS_O ? p.layer[l].eps_gate : p.eps_norm);
                        if (pass) break;
                        DS_TRACE_AFTER(3, (double)rstd);
                        s0 = s1 = 0.0;
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            float2 y = __fmul2_rn(mul2(t[i], rstd), n[i]);
                            if (type == DS_O) y = __fmul2_rn(__fmul2_rn(y, widen<T>(a[i])), gate[i]);
                            c[i] = in_h ? narrow<T>(y) : 0;
                            sumsq_pair<T>(c[i], s0, s1);
                        }
                    }
                    v[0] = make_uint4(c[0], c[1], c[2], c[3]);
                    w += D;
                }
            }
            if (me) {
                DS_TRACE_AFTER(4, (double)rstd);
                // Units of 8 columns, with codes of their own: the same of the three projections (mixer), the vectors of an inner row, or one
                const bool down = type == DS_DOWN, each = FUSED && type == DS_IFG, multi = down || each;
                if (each) v[1] = v[2] = v[0];
                const int wstep = down ? TH * 8 : D;
                float2 y[NVI][4];
                float am[NVI];
                auto scaled = [&](int j) {
                    const uint32_t c[4] = {v[j].x, v[j].y, v[j].z, v[j].w};
                    float2 n[4];
                    lds8((down && (j * TH + tid) * 8 >= D) ? w : w + j * wstep, n);
                    am[j] = 0.0f;
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        y[j][k] = __fmul2_rn(mul2(widen<T>(c[k]), rstd), n[k]);
                        am[j] = fmaxf(am[j], fmaxf(fabsf(y[j][k].x), fabsf(y[j][k].y)));
                    }
                    if ((down ? j * TH + tid : tid) * 8 >= D) am[j] = 0.0f;      // (what follows a row in shared memory may be anything)
                };
                auto publish = [&](int j) {
                    const uint32_t m = __reduce_max_sync(0xffffffffu, __float_as_uint(am[j]));
                    if (lane == 0) s_max[j][warp] = __uint_as_float(m);
                };
                scaled(0);
                if (multi) { scaled(1); scaled(2); }
                if (down) am[0] = fmaxf(am[0], fmaxf(am[1], am[2]));
                publish(0);
                if (each) { publish(1); publish(2); }
                __syncthreads();
                float sc[NVI];
                auto scale = [&](int j) {
                    const float top = ds_fold_max<NW>(s_max[j]);
                    sc[j] = q127_over(top);
                    if (tid == 0) s_top[j] = top;
                };
                uint8_t* dst = xcodes + ((FUSED || type != DS_IFG ? 0 : row_g) * KG + warp) * STEP + code_at;
                const int dstep = (down ? NW : KG) * STEP;
                auto put = [&](int j) {
                    const uint32_t lo = codes4(y[j][0], y[j][1], sc[j]), hi = codes4(y[j][2], y[j][3], sc[j]);
                    int sum = 0;
                    if ((down ? j * TH + tid : tid) * 8 < D) {
                        sum = __dp4a((int)lo, 0x01010101, __dp4a((int)hi, 0x01010101, 0));
                        if constexpr (FUSED) {
                            *reinterpret_cast<uint32_t*>(dst + j * dstep) = lo;
                            *reinterpret_cast<uint32_t*>(dst + j * dstep + 8) = hi;
                        } else {
                            ds_st(dst + j * dstep, lo);
                            ds_st(dst + j * dstep + 8, hi);
                        }
                    }
                    __syncwarp();
                    sum = __reduce_add_sync(0xffffffffu, sum);
                    if (lane == 0) s_codes[j * NW + warp] = sum;
                };
                scale(0);
                if (each) { scale(1); scale(2); }
                if (down) sc[1] = sc[2] = sc[0];
                put(0);
                if (multi) { put(1); put(2); }
            }
        }
        if constexpr (FUSED) {
            __syncwarp();                                      // this warp's codes
        } else if (me) {
            __syncthreads();
            if (tid == 0) {
                int sum = 0;
#pragma unroll 1
                for (int k = 0; k < KG; ++k) sum += s_codes[k];
                const uint64_t x = (uint64_t)(uint32_t)sum << 32 | __float_as_uint(over_127(s_top[0]));
                asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(xscale + ((type == DS_IFG ? row_g : 0) * MR + row_m) * 8), "l"(x) : "memory");
            }
        }
        DS_TRACE(5);

        // ---- contraction
        int* dst = part + (warp * MR + (FUSED ? 0 : 2 * q)) * DS_TS + gq;
        if constexpr (FUSED) {
            const uint8_t* cb = xcodes + warp * STEP + (lane & (TL - 1)) * 16;        // this warp's own codes
            int b = 0;
            auto product = [&](const DsWeights& w) {
                uint4 x[1][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) x[0][i] = *reinterpret_cast<const uint4*>(cb + i * (TL * 16));
                ds_block<NB, MR>(dst, w, x, q);
                dst += KG * (MR * DS_TS);
                if (++b == nbp) {
                    b = 0;
                    dst += next_d;
                    cb += next_c;
                }
            };
#pragma unroll
            for (int i = 0; i < PRE; ++i)
                if (i < items) product(pre[i]);
#pragma unroll 1
            for (int i = PRE; i < items; ++i) {
                DsWeights one;
                unpack(one);
                product(one);
            }
        } else {
            const uint8_t* cb = xcodes + warp * STEP + lane * 16;
            int kg = warp, b = 0;
            uint4 x[NB][4];
#pragma unroll 1
            for (int i = 0; i < items; ++i) {
                if (b == 0) {                                  // a projection's or column group's codes, as they come
                    int n = 0;
                    bool ok;
                    do {
                        ok = true;
#pragma unroll
                        for (int t = 0; t < NB; ++t)
#pragma unroll
                            for (int k = 0; k < 4; ++k)
                                x[t][k] = kg * 4 + q < z.KC && t * 8 + gq < M ? ds_ld(cb + (t * 4 + k) * 512) : make_uint4(0, 0, 0, 0);
#pragma unroll
                        for (int t = 0; t < NB; ++t)
#pragma unroll
                            for (int k = 0; k < 4; ++k) ok = ok && ds_there(x[t][k], DS_NO_CODES);
                    } while (!ok && wait.again(n));
                    __syncwarp();
                }
                DsWeights one;
                unpack(one);
                ds_block<NB, MR>(dst, one, x, q);
                dst += KG * (MR * DS_TS);
                if (++b == nbp) {
                    b = 0;
                    dst += next_d;
                    cb += next_c;
                    if (type == DS_DOWN) kg += NW;
                }
            }
        }
        if constexpr (!FUSED) {
            if (has_const) {
                uint64_t u;
                int n = 0;
                do {
                    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(u) : "l"(xscale + (cg * MR + cm) * 8) : "memory");
                } while ((uint32_t)u == DS_NO_CODES && wait.again(n));
                s_scale[cg][cm] = __fmul_rn(__uint_as_float((uint32_t)u), ws);
                s_rs[cg][cm] = (int)(u >> 32);
            }
        }
        __syncthreads();
        DS_TRACE(6);
        if (tid == TH - 32) {                                  // the regions of this link are free again
            fetch_norms(idx + 2);
            fetch(idx + 4);
        }

        // ---- epilogue: two adjacent rows (channels) of a token
#pragma unroll 1
        for (int i = item0, i0 = warp * per; i0 < pairs * M; i += NW * per, i0 += NW * per) {
            const bool on = i < pairs * M && (type != DS_IFG || lane < 30);
            const int m = MR == 1 ? 0 : (i * inv_pairs) >> 20, pr = i - m * pairs, ch = (u0 + pr) * 2;
            const int g = type == DS_IFG ? vk : 0, k0 = per == 8 ? vk : 0, ks = per == 8 ? 4 : 1;
            int2 sum = make_int2(0, 0);                        // rows r, r + 1 of a block
            if (on) {
                const int blk = type == DS_GATE ? pr >> 2 : (pr >> 3) + g * nbp, r = type == DS_GATE ? (pr & 3) * 2 + 8 * vk : (pr & 7) * 2;
                const int* s = part + ((blk * KG + k0) * MR + m) * DS_TS + r;
#pragma unroll
                for (int j = 0; j < NW; ++j)
                    if (k0 + j * ks < KG) {
                        const int2 t = *reinterpret_cast<const int2*>(s + j * ks * (MR * DS_TS));
                        const int cs = FUSED ? s_codes[g * NW + k0 + j * ks] : 0;
                        sum.x += t.x - cs;
                        sum.y += t.y - cs;
                    }
            }
            if (per == 8) {
#pragma unroll
                for (int o = 8; o <= 16; o *= 2) {
                    sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o);
                    sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
                }
            }
            const int rs = FUSED || !on ? 0 : s_rs[g][m];
            float sc;
            if constexpr (FUSED) sc = __fmul_rn(over_127(s_top[g]), ws);
            else sc = on ? s_scale[g][m] : 0.0f;
            uint32_t val = narrow<T>(make_float2(dl_out(sum.x, rs, sc), dl_out(sum.y, rs, sc)));
            const uint32_t v1 = __shfl_sync(0xffffffffu, val, (lane + per) & 31), v2 = __shfl_sync(0xffffffffu, val, (lane + 2 * per) & 31);
            if (on && vk == 0) {
                T* out = xrows + (type == DS_GATE ? 4 * Mh + (int64_t)m * inner : (int64_t)m * h) + ch;
                if (type == DS_IFG) {
                    // token mixer of one new token (layers/hgrn_bit.py:113-125 of the reference with T = 1)
                    const bool first = i == item0;
                    float2* st = reinterpret_cast<float2*>(p.layer[l].state + (int64_t)m * h + ch);
                    float2 hv = first ? h_pre : *st;
                    float2 xv = raw_gate_floor(widen<T>(val)), f = raw_gate_floor(widen<T>(v1));
                    float2 lbv = make_float2(0.0f, 0.0f), oml = make_float2(1.0f, 1.0f);
                    if (lb) {
                        lbv = widen<T>(first ? lb_pre : *reinterpret_cast<const uint32_t*>(lb + ch));
                        oml = make_float2(round_to<T>(__fsub_rn(1.0f, lbv.x)), round_to<T>(__fsub_rn(1.0f, lbv.y)));
                    }
                    raw_gate_pair<T>(xv, f, lb != nullptr, lbv, oml);
                    if (p.mask && !(first ? keep_pre : p.mask[m] != 0)) xv = make_float2(0.0f, 0.0f);      // a padding position contributes no input
                    hv.x = fmaf(f.x, hv.x, xv.x);
                    hv.y = fmaf(f.y, hv.y, xv.y);
                    ds_st(out, narrow<T>(hv));
                    ds_st(out + Mh, v2);
                    *st = hv;
                } else {
                    if (type == DS_GATE) val = narrow<T>(silu_mul2(widen<T>(val), widen<T>(v1)));
                    else if (type == DS_O) out += 2 * Mh;
                    else if (l == p.L - 1) out = reinterpret_cast<T*>(p.out) + (int64_t)m * h + ch;
                    else out += 3 * Mh;
                    ds_st(out, val);
                }
            }
        }
        DS_TRACE(7);
        __syncthreads();                                       // (warps without outputs wait here and not in a loop that would take the others' issue slots)
    }
}

#ifdef MMF_EXPERIMENTS
}  // namespace
extern int g_step_refuse;      // mmf_tuning(MMF_TUNE_STEP_REFUSE, 1)
namespace {
#endif
template <auto kernel> int ds_go(const DsParams& p, const DsPlan& d, cudaStream_t st) {
    MMF_CUDA(mmf_allow_smem<kernel>(DS_SMEM_MAX));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)d.grid);
    cfg.blockDim = dim3((unsigned)d.warps * 32);
    cfg.dynamicSmemBytes = (size_t)d.smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;      // the CTAs wait for one another: all of them resident, or none
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
#ifdef MMF_EXPERIMENTS
    const cudaError_t e = g_step_refuse ? cudaErrorCooperativeLaunchTooLarge : cudaLaunchKernelEx(&cfg, kernel, p);
#else
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, p);
#endif
    // A context of fewer SMs than the device has (the attribute counts the device's), or one without cooperative launches: the caller's call
    // is not lost, the chain of kernels needs no co-residency.
    if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorLaunchOutOfResources || e == cudaErrorNotSupported) {
        (void)cudaGetLastError();
        return mmf_set_error(MMF_ERR_NOT_RESIDENT, "mmf_decode_step: %d CTAs are not resident at once here: %s", d.grid, cudaGetErrorString(e));
    }
    MMF_CUDA(e);
    return MMF_OK;
}

// arguments are checked by mmf_decode_step
template <typename T> int decode_step_launch(const DsParams& p, const DsPlan& d, cudaStream_t st) {
#define DS_K(MR, FUSED, NW, PRE) return ds_go<decode_step_kernel<T, MR, FUSED, NW, PRE>>(p, d, st)
#define DS_ROWS(NW, P1, P8, P16)                     \
    if (d.warps == NW) {                             \
        if (d.fused) DS_K(1, true, NW, P1);          \
        if (d.mr == 8) DS_K(8, false, NW, P8);       \
        DS_K(16, false, NW, P16);                    \
    }
    DS_ROWS(8, 3, 0, 0)
    DS_ROWS(10, 2, 0, 0)
#undef DS_ROWS
#undef DS_K
    return mmf_set_error(MMF_ERR_BAD_SHAPE, "mmf_decode_step: %d warps", d.warps);
}

}  // namespace
