// The two-factor FFT kernels in FP32 (fft_two.cuh); a file of its own so that
// the two precisions compile side by side.
#include "fft_two.cuh"

namespace fbse {
template size_t two_plane_smem<float>(const fbse_ctx *);
template int two_plane<float>(fbse_ctx *, const float2 *, float2 *, long, bool, const float2 *, const float *, float, float);
template int two_z<float>(fbse_ctx *, float2 *, long, const KinArgs &);
template int two_y<float>(fbse_ctx *, const float2 *, float2 *, long, int, const float2 *, const float *, float, float);
template int two_x<float>(fbse_ctx *, const float2 *, float2 *, long, int, const float2 *, const float *, float, float);
}  // namespace fbse
