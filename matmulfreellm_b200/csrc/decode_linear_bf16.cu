// Instantiations of decode_linear.cuh for bf16 activations.
#include "decode_linear.cuh"

int decode_linear_bf16(const mmf_decode_linear_args& a, cudaStream_t st) { return decode_linear_launch<__nv_bfloat16>(a, st); }
