// Instantiations of decode_linear.cuh for fp16 activations.
#include "decode_linear.cuh"

int decode_linear_fp16(const mmf_decode_linear_args& a, cudaStream_t st) { return decode_linear_launch<__half>(a, st); }
