// Instantiations of decode_step.cuh for bf16 activations.
#include "decode_step.cuh"

int decode_step_bf16(const DsParams& p, const DsPlan& d, cudaStream_t st) { return decode_step_launch<__nv_bfloat16>(p, d, st); }
