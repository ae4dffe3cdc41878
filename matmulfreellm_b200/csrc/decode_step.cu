// C ABI of the resident decode step (kernel: decode_step.cuh) and the layout of its weights.
#include "decode_step_plan.cuh"
#include "rowquant.cuh"
#include <algorithm>

int decode_step_bf16(const DsParams& p, const DsPlan& d, cudaStream_t st);
int decode_step_fp16(const DsParams& p, const DsPlan& d, cudaStream_t st);

#ifdef MMF_EXPERIMENTS
int g_step_wait_limit = 0;     // mmf_tuning(MMF_TUNE_STEP_WAIT_LIMIT, polls)
int g_step_refuse = 0;         // mmf_tuning(MMF_TUNE_STEP_REFUSE, 1)
#endif

namespace {

struct PackParams {
    DsSizes size[4];
    const uint4* packed[4];
    int h, inner;
    uint8_t* out;
};
// CTA (x, type): the weights of CTA x of the step, [column group][row][chunk of the group] 16-byte pieces of 64 weights; rows i | f | g
// or gate | up of its channels; columns past the row's end are zero fields, which count nothing.
__global__ void step_pack_kernel(const __grid_constant__ PackParams p) {
    const int type = blockIdx.y, bid = blockIdx.x;
    const DsSizes& z = p.size[type];
    const int u0 = bid * z.base + min(bid, z.extra), pairs = z.base + (bid < z.extra ? 1 : 0), mult = ds_rows_per_pair(type), R = pairs * mult;
    uint4* out = reinterpret_cast<uint4*>(p.out + z.w_at + (int64_t)u0 * mult * z.KG * 64);
    const int skip = (type == DS_GATE ? p.inner : p.h) - 2 * pairs;      // from the end of a part's rows to the next part's
    for (int i = threadIdx.x; i < R * z.KG * 4; i += blockDim.x) {
        const int c = (i >> 2) / R * 4 + (i & 3), r = (i >> 2) % R;
        const int n = 2 * u0 + r + (r >= 2 * pairs ? skip : 0) + (r >= 4 * pairs ? skip : 0);
        out[i] = c < z.KC ? p.packed[type][((int64_t)(n >> 7) * z.KC + c) * MMF_TILE_ROWS + (n & 127)] : make_uint4(0, 0, 0, 0);
    }
}
struct NormParams {
    const float* src[9];                         // attn, i, f, g | gate norm, o | mlp, gate_proj | down
    const float* scale[4];
    int h, inner;
    float* out;
};
__global__ void step_norms_kernel(const __grid_constant__ NormParams p) {
    const int k = blockIdx.y, n = k == 8 ? p.inner : p.h;
    float* out = p.out + (int64_t)k * p.h;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) out[i] = p.src[k] ? p.src[k][i] : 1.0f;
    if (k == 8 && blockIdx.x == 0 && threadIdx.x < 8) {
        const int t = threadIdx.x;
        out[n + t] = t < 3 ? p.scale[0][t] : t < 6 ? p.scale[t - 2][0] : 0.0f;
    }
}

// The words that nobody has written yet: rows (the first `rows` 16-byte pieces), then codes.  One kernel takes less of a step than two
// memory fills.
__global__ void __launch_bounds__(256) step_fill_kernel(uint4* p, int64_t rows, int64_t n) {
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += step) {
        const uint32_t w = i < rows ? DS_NO_ROW : DS_NO_CODES;
        p[i] = make_uint4(w, w, w, w);
    }
}

bool taken(DsParams& p, DsPlan& d, int64_t M, int64_t h, int64_t inner, int64_t layers) {
    int sms = 0;
    if (mmf_sm_count(&sms) != cudaSuccess) return false;
    d = ds_plan(p, M, h, inner, layers, sms);
    return d.mr > 0;
}

}  // namespace

extern "C" int64_t mmf_decode_step_layer_bytes(int64_t hidden, int64_t inner) {
    DsParams p;
    DsPlan d;
    return taken(p, d, 1, hidden, inner, 1) ? d.layer_bytes : 0;
}
extern "C" int64_t mmf_decode_step_workspace_bytes(int64_t M, int64_t hidden, int64_t inner, int64_t layers) {
    DsParams p;
    DsPlan d;
    return taken(p, d, M, hidden, inner, layers) ? layers * (p.rows_layer + p.codes_layer) : 0;
}

extern "C" int mmf_decode_step_pack(const mmf_decode_step_weights* w, int64_t hidden, int64_t inner, void* out, void* stream) {
    MMF_REQUIRE(w && out && mmf_aligned(out, 16), MMF_ERR_BAD_ARG, "mmf_decode_step_pack: null or unaligned pointer");
    MMF_REQUIRE(w->ifg && w->o && w->gate && w->down && w->ifg_scale && w->o_scale && w->gate_scale && w->down_scale, MMF_ERR_BAD_ARG,
                "mmf_decode_step_pack: weight missing");
    MMF_REQUIRE(mmf_aligned(w->ifg, 16) && mmf_aligned(w->o, 16) && mmf_aligned(w->gate, 16) && mmf_aligned(w->down, 16), MMF_ERR_ALIGN,
                "mmf_decode_step_pack: packed weights must be 16-byte aligned");
    DsParams p;
    DsPlan d;
    MMF_REQUIRE(taken(p, d, 1, hidden, inner, 1), MMF_ERR_BAD_SHAPE, "mmf_decode_step_pack: hidden=%lld, inner=%lld is not taken", (long long)hidden, (long long)inner);
    PackParams k = {};
    for (int t = 0; t < 4; ++t) k.size[t] = p.size[t];
    k.packed[DS_IFG] = (const uint4*)w->ifg; k.packed[DS_O] = (const uint4*)w->o; k.packed[DS_GATE] = (const uint4*)w->gate; k.packed[DS_DOWN] = (const uint4*)w->down;
    k.h = (int)hidden; k.inner = (int)inner;
    k.out = (uint8_t*)out;
    step_pack_kernel<<<dim3((unsigned)d.grid, 4), 256, 0, (cudaStream_t)stream>>>(k);
    MMF_LAUNCH_CHECK("step_pack_kernel");
    NormParams n = {{w->attn_norm_w, w->ifg_norm_w[0], w->ifg_norm_w[1], w->ifg_norm_w[2], w->gate_norm_w, w->o_norm_w, w->mlp_norm_w, w->gate_proj_norm_w, w->down_norm_w},
                    {w->ifg_scale, w->o_scale, w->gate_scale, w->down_scale}, (int)hidden, (int)inner, (float*)((uint8_t*)out + p.size[0].n_at)};
    step_norms_kernel<<<dim3(4, 9), 256, 0, (cudaStream_t)stream>>>(n);
    MMF_LAUNCH_CHECK("step_norms_kernel");
    return MMF_OK;
}

extern "C" int mmf_decode_step(const mmf_decode_step_args* args, void* stream) {
    MMF_REQUIRE(args && args->layer, MMF_ERR_BAD_ARG, "mmf_decode_step: null arguments");
    const mmf_decode_step_args& a = *args;
    MMF_REQUIRE(a.dtype == MMF_BF16 || a.dtype == MMF_F16, MMF_ERR_BAD_ARG, "mmf_decode_step: 16-bit activations only (dtype %d)", a.dtype);
    MMF_REQUIRE(a.x && a.out && a.residual_out && a.workspace && a.status, MMF_ERR_BAD_ARG, "mmf_decode_step: null pointer");
    MMF_REQUIRE(mmf_aligned(a.x, 16) && a.ld_x % 8 == 0 && mmf_aligned(a.out, 16) && mmf_aligned(a.residual_out, 16) && mmf_aligned(a.workspace, 256),
                MMF_ERR_ALIGN, "mmf_decode_step: rows must be 16-byte aligned");
    MMF_REQUIRE((a.M <= 1 && !a.row_ids) || a.ld_x >= a.hidden, MMF_ERR_BAD_SHAPE, "mmf_decode_step: row pitch below the row");
    MMF_REQUIRE(!a.row_ids || a.x_rows > 0, MMF_ERR_BAD_ARG, "mmf_decode_step: row ids need a table");
    MMF_REQUIRE(a.M > 0 && a.layers > 0 && a.layers <= DS_MAX_LAYERS, MMF_ERR_BAD_SHAPE, "mmf_decode_step: M=%lld, layers=%lld", (long long)a.M,
                (long long)a.layers);
    DsParams p;
    for (int64_t i = 0; i < a.layers; ++i) {
        const mmf_decode_step_layer& y = a.layer[i];
        MMF_REQUIRE(y.weights && y.state, MMF_ERR_BAD_ARG, "mmf_decode_step: layer %lld has a null pointer", (long long)i);
        MMF_REQUIRE(mmf_aligned(y.weights, 16) && mmf_aligned(y.state, 8) && mmf_aligned(y.lower_bound, 4), MMF_ERR_ALIGN,
                    "mmf_decode_step: layer %lld: weights must be 16-byte aligned", (long long)i);
        p.layer[i] = y;
    }
    DsPlan d;
    MMF_REQUIRE(taken(p, d, a.M, a.hidden, a.inner, a.layers), MMF_ERR_BAD_SHAPE,
                "mmf_decode_step: M=%lld, hidden=%lld, inner=%lld, layers=%lld is not taken (mmf_decode_step_workspace_bytes says 0)", (long long)a.M,
                (long long)a.hidden, (long long)a.inner, (long long)a.layers);
    MMF_REQUIRE(a.workspace_bytes >= a.layers * (p.rows_layer + p.codes_layer), MMF_ERR_WORKSPACE, "mmf_decode_step: workspace of %lld bytes, need %lld",
                (long long)a.workspace_bytes, (long long)(a.layers * (p.rows_layer + p.codes_layer)));
    p.x = a.x; p.ld_x = a.ld_x; p.row_ids = a.row_ids; p.x_rows = a.x_rows;
    p.mask = a.mask;
    p.out = a.out; p.residual_out = a.residual_out;
    p.status = a.status;
    p.gave_up = a.gave_up_host;
    p.rows = (uint8_t*)a.workspace;
    p.codes = p.rows + a.layers * p.rows_layer;
    p.eps_norm = a.eps_norm;
#ifdef MMF_EXPERIMENTS
    p.trace = g_row_trace;
    p.wait_limit = g_step_wait_limit ? g_step_wait_limit : DS_WAIT_LIMIT;
#endif
    const cudaStream_t st = (cudaStream_t)stream;
    const int64_t fill_rows = a.layers * p.rows_layer / 16, fill = fill_rows + a.layers * p.codes_layer / 16;
    step_fill_kernel<<<(unsigned)std::min<int64_t>((fill + 255) / 256, 4 * d.grid), 256, 0, st>>>(reinterpret_cast<uint4*>(p.rows), fill_rows, fill);
    MMF_LAUNCH_CHECK("step_fill_kernel");
    return a.dtype == MMF_BF16 ? decode_step_bf16(p, d, st) : decode_step_fp16(p, d, st);
}
