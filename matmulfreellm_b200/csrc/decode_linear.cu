// C ABI of the fused decode-step BitLinear (kernels: decode_linear.cuh).
#include "common.cuh"

int decode_linear_bf16(const mmf_decode_linear_args& a, cudaStream_t st);
int decode_linear_fp16(const mmf_decode_linear_args& a, cudaStream_t st);

extern "C" int mmf_decode_linear(const mmf_decode_linear_args* args, void* stream) {
    MMF_REQUIRE(args, MMF_ERR_BAD_ARG, "mmf_decode_linear: null arguments");
    const mmf_decode_linear_args& a = *args;
    MMF_REQUIRE(a.dtype == MMF_BF16 || a.dtype == MMF_F16, MMF_ERR_BAD_ARG, "mmf_decode_linear: 16-bit activations only (dtype %d)", a.dtype);
    MMF_REQUIRE(a.packed && a.w_scale && a.out, MMF_ERR_BAD_ARG, "mmf_decode_linear: null pointer");
    MMF_REQUIRE(a.M >= 0 && a.N > 0 && a.K > 0 && a.K % MMF_TILE_K == 0 && a.N < (1ll << 24), MMF_ERR_BAD_SHAPE,
                "mmf_decode_linear: need K %% 64 == 0 (M=%lld N=%lld K=%lld)", (long long)a.M, (long long)a.N, (long long)a.K);
    const int max_m = a.codes ? MMF_DECODE_LINEAR_MAX_M : MMF_DECODE_LINEAR_FUSED_MAX_M;
    MMF_REQUIRE(a.M <= max_m, MMF_ERR_BAD_SHAPE, "mmf_decode_linear: at most %d token rows (M=%lld)", max_m, (long long)a.M);
    MMF_REQUIRE(!a.codes || (a.dq && a.rowsum && mmf_aligned(a.codes, 16)), MMF_ERR_BAD_ARG, "mmf_decode_linear: incomplete workspace");
    MMF_REQUIRE(((a.M <= 1 && !a.row_ids) || a.ld_x >= a.K) && (!a.residual || a.M <= 1 || a.ld_residual >= a.K), MMF_ERR_BAD_SHAPE,
                "mmf_decode_linear: row pitch below K");
    MMF_REQUIRE(a.x && (a.prologue != MMF_PRO_GATENORM || a.residual), MMF_ERR_BAD_ARG, "mmf_decode_linear: input row missing");
    MMF_REQUIRE(mmf_aligned(a.packed, 16) && mmf_aligned(a.out, 16) && mmf_aligned(a.x, 16) && a.ld_x % 8 == 0 &&
                    (!a.residual || (mmf_aligned(a.residual, 16) && a.ld_residual % 8 == 0)) && (!a.residual_out || mmf_aligned(a.residual_out, 16)) &&
                    mmf_aligned(a.norm_w, 16) && mmf_aligned(a.bl_norm_w[0], 16) && mmf_aligned(a.bl_norm_w[1], 16) && mmf_aligned(a.bl_norm_w[2], 16),
                MMF_ERR_ALIGN, "mmf_decode_linear: packed, rows and norm weights must be 16-byte aligned");
    const int64_t max_k = a.prologue == MMF_PRO_QUANT ? 8192 : 4096;
    MMF_REQUIRE(a.K <= max_k, MMF_ERR_BAD_SHAPE, "mmf_decode_linear: rows of at most %lld values", (long long)max_k);
    MMF_REQUIRE(!a.row_ids || (a.prologue == MMF_PRO_PRENORM && !a.residual && a.x_rows > 0), MMF_ERR_BAD_ARG,
                "mmf_decode_linear: row ids go with PRENORM without residual");
    if (a.epilogue == MMF_EPI_GATES) {
        MMF_REQUIRE(a.N == 3 * a.K && a.K % MMF_TILE_ROWS == 0, MMF_ERR_BAD_SHAPE, "mmf_decode_linear: gates need three K x K projections, K %% 128 == 0");
        MMF_REQUIRE(a.state && a.g_out && mmf_aligned(a.state, 8) && mmf_aligned(a.g_out, 4) && (!a.lower_bound || mmf_aligned(a.lower_bound, 4)),
                    MMF_ERR_BAD_ARG, "mmf_decode_linear: state or output missing");
    } else if (a.epilogue == MMF_EPI_SWIGLU) {
        MMF_REQUIRE(a.N % 4 == 0 && a.ld_out % 2 == 0 && a.ld_out >= a.N / 2, MMF_ERR_BAD_SHAPE, "mmf_decode_linear: swiglu needs N %% 4 == 0");
    } else {
        MMF_REQUIRE(a.epilogue == MMF_EPI_STORE && a.ld_out >= a.N, MMF_ERR_BAD_ARG, "mmf_decode_linear: unknown epilogue or ld_out < N");
    }
    MMF_REQUIRE(a.prologue == MMF_PRO_QUANT || a.prologue == MMF_PRO_PRENORM || a.prologue == MMF_PRO_GATENORM, MMF_ERR_BAD_ARG,
                "mmf_decode_linear: prologue %d", a.prologue);
    if (a.M == 0) return MMF_OK;
    return a.dtype == MMF_BF16 ? decode_linear_bf16(a, (cudaStream_t)stream) : decode_linear_fp16(a, (cudaStream_t)stream);
}
