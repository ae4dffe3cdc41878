// How a decode step is split over CTAs, warps and shared memory (kernels: decode_step.cuh).
#pragma once
#include "common.cuh"

constexpr int DS_MAX_LAYERS = 96;
constexpr int DS_WAIT_LIMIT = 1 << 22;           // polls of one wait (each is a round trip to the L2: seconds in all)
constexpr int DS_TS = 20;                        // accumulator words per (block, token): 16 rows, padded so that a warp's stores do not collide
constexpr uint32_t DS_NO_ROW = 0xffffffffu;      // a word of an exchanged row that has not been written: two NaNs no rounding produces
constexpr uint32_t DS_NO_CODES = 0x80808080u;    // a word of exchanged codes that has not been written: codes are -127 .. 127
constexpr int DS_SMEM_MAX = 225 * 1024;          // of 227 KB; the rest is static

// links of a block
constexpr int DS_IFG = 0, DS_O = 1, DS_GATE = 2, DS_DOWN = 3;
__host__ __device__ constexpr int ds_rows_per_pair(int type) { return type == DS_IFG ? 6 : type == DS_GATE ? 4 : 2; }     // weight rows per pair of channels

// sizes of a link, the same in every block
struct DsSizes {
    int D, KC, KG;                               // row, its 64-column chunks and 256-column groups
    int base, extra;                             // pairs of channels per CTA: base, the first `extra` CTAs one more
    int w_off;                                   // its weights in shared memory
    int64_t w_at, n_at;                          // its weights and norm weights in a block's packed bytes
    int64_t codes_at;                            // its codes in a block's exchanged codes
    double inv_d;
};
struct DsParams {
    mmf_decode_step_layer layer[DS_MAX_LAYERS];
    DsSizes size[4];
    int64_t scales_at;                           // six weight scales in a block's packed bytes
    const void* x; int64_t ld_x; const int64_t* row_ids; int64_t x_rows;
    const uint8_t* mask;
    void *out, *residual_out;
    int *status, *gave_up;
    uint8_t* rows;                               // exchanged rows, [layer]: o, g, attention output, MLP output [M][h], act [M][inner]
    uint8_t* codes;                              // exchanged codes and their scales, [layer]
    int64_t rows_layer, codes_layer;             // bytes per layer
    int64_t code_scales_at;                      // scales and code sums in a block's exchanged codes: (projection, row), 8 bytes each
    int L, M, h, inner;
    int norm_off[2], part_off;                   // norm weights of even and odd links, partial sums in shared memory
    float eps_norm;
#ifdef MMF_EXPERIMENTS
    long long* trace;
    int wait_limit;
#endif
};

struct DsPlan {
    bool fused = false;
    int mr = 0, warps = 0, smem = 0, grid = 0;   // mr: rows the kernel is made for, 0: the sizes are not taken
    int64_t layer_bytes = 0;                     // packed weights, norm weights and scales of a block
};

inline DsPlan ds_plan(DsParams& p, int64_t M, int64_t h, int64_t inner, int64_t layers, int sms) {
    DsPlan d;
    if (M < 1 || M > MMF_DECODE_STEP_MAX_M || layers < 1 || layers > DS_MAX_LAYERS || h < MMF_TILE_ROWS || h % MMF_TILE_ROWS || h > 4096 ||
        inner < MMF_TILE_K || inner % MMF_TILE_K || inner > 8192)
        return d;
    // One row: every CTA repeats its row work.  More: a CTA per row and projection does it and hands the codes round, which costs a second
    // exchange per link (two rows of 2048: 429 us a step and 457 with the row work repeated, in turn; four: 443 and 1170).
    d.fused = M == 1;
    const int mr = d.fused ? 1 : M <= 8 ? 8 : 16;
    if (!d.fused && 3 * M > sms) return d;
    // The second exchange and the fill of the codes are not won back by a single block (256 - 1024 wide, 4 rows: 24.7 us as kernels, 26.8
    // here), nor by two rows of at most 1024 (kernels of their own then repeat the row work: 8 blocks of 1024 126 / 131 us, 24 of 256 340 / 342;
    // 4 blocks of 2048 86 / 78).
    if (!d.fused && (layers < 2 || (M == 2 && h <= 1024))) return d;
    d.grid = sms;
    // A thread holds eight columns of a hidden row and three times eight of an inner one.  Eight warps where they suffice: twice or three
    // times as many make no link shorter (they share the issue slots) and leave fewer registers (24 warps: 558 us a step against 329).
    d.warps = h <= 2048 && inner <= 6144 ? 8 : 10;
    if (h > d.warps * 256 || inner > d.warps * 768) return d;
    p.M = (int)M; p.h = (int)h; p.inner = (int)inner; p.L = (int)layers;
    const int kgh = (int)(h / MMF_TILE_K + 3) / 4, kgi = (int)(inner / MMF_TILE_K + 3) / 4;
    int off = d.fused ? (3 * kgh > kgi ? 3 * kgh : kgi) * 256 : 0;      // codes
    p.norm_off[0] = off;
    off += (int)h * 4 * (d.fused ? 4 : 2);
    p.norm_off[1] = off;
    off += (int)((2 * h > inner ? 2 * h : inner) * 4);
    int part = 0;
    int64_t at = 0, codes = 0;
    for (int t = 0; t < 4; ++t) {
        DsSizes& z = p.size[t];
        z.D = (int)(t == DS_DOWN ? inner : h);
        z.KC = z.D / MMF_TILE_K;
        z.KG = t == DS_DOWN ? kgi : kgh;
        z.inv_d = 1.0 / (double)z.D;
        const int units = (int)(t == DS_GATE ? inner / 2 : h / 2);
        z.base = units / sms;
        z.extra = units % sms;
        const int most = z.base + (z.extra > 0);
        z.w_off = off;
        off += most * ds_rows_per_pair(t) * z.KG * 64;
        z.w_at = at;
        at += (int64_t)units * ds_rows_per_pair(t) * z.KG * 64;
        z.codes_at = codes;
        codes += (int64_t)(t == DS_IFG ? 3 : 1) * z.KG * (mr / 8) * 2048;
        const int blocks = t == DS_GATE ? (most + 3) / 4 : (most + 7) / 8 * (t == DS_IFG ? 3 : 1);
        const int sums = blocks * z.KG;
        part = sums > part ? sums : part;
    }
    for (int t = 0; t < 4; ++t) {
        p.size[t].n_at = at;
        at += (t == DS_IFG ? 4 * h : t == DS_DOWN ? inner : 2 * h) * 4;
    }
    p.scales_at = at;
    d.layer_bytes = at + 32;
    p.part_off = off;
    d.smem = off + part * mr * DS_TS * 4 + 1024;      // (the last block of 16 weight rows may reach past the CTA's last row)
    if (d.smem > DS_SMEM_MAX) return d;
    p.rows_layer = (M * (4 * h + inner) * 2 + 255) / 256 * 256;
    p.code_scales_at = codes;
    p.codes_layer = d.fused ? 0 : (codes + 6 * mr * 8 + 255) / 256 * 256;
    d.mr = mr;
    return d;
}
