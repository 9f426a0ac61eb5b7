// Host-side launchers of the kernels, one per translation unit.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

namespace dash {
struct TrainArgs;
struct DecodeArgs;

// Each adds the kernels it launched to *launches and returns the first launch error.
cudaError_t launch_generic_forward(int dtype, const TrainArgs &a, cudaStream_t stream, int *launches);
cudaError_t launch_generic_backward(int dtype, const TrainArgs &a, cudaStream_t stream, int *launches);
// (`beside`: beside the kernel launched before it, which must allow it - see launch_beside.)
cudaError_t launch_generic_delta(int dtype, const TrainArgs &a, cudaStream_t stream, int *launches, bool beside);
// Whether launch_decode rotates on its way (DecodeArgs::rope_*): a 16-bit cache on the tensor-core pass, rotated features and
// tables readable 16 bytes at a time.  Other calls rotate with a launch of their own first.
bool decode_fuses_rope(int dtype, const DecodeArgs &a, bool vector_ok);
long long decode_fixed_chunk();
cudaError_t launch_decode(int dtype, const DecodeArgs &a, bool vector_ok, cudaStream_t stream, int *launches);
// The library's own decode scratch: its size in floats, and its address on the current device.
size_t decode_static_capacity_floats();
cudaError_t decode_static_scratch(float **out);
cudaError_t launch_fill_f32(float *dst, float value, long long n, cudaStream_t stream, int *launches);
}  // namespace dash
