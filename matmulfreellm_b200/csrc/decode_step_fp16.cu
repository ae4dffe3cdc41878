// Instantiations of decode_step.cuh for fp16 activations.
#include "decode_step.cuh"

int decode_step_fp16(const DsParams& p, const DsPlan& d, cudaStream_t st) { return decode_step_launch<__half>(p, d, st); }
