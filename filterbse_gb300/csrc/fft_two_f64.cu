// The two-factor FFT kernels in FP64 (fft_two.cuh); a file of its own so that
// the two precisions compile side by side.
#include "fft_two.cuh"

namespace fbse {
template size_t two_plane_smem<double>(const fbse_ctx *);
template int two_plane<double>(fbse_ctx *, const double2 *, double2 *, long, bool, const double2 *, const double *, double, double);
template int two_z<double>(fbse_ctx *, double2 *, long, const KinArgs &);
template int two_y<double>(fbse_ctx *, const double2 *, double2 *, long, int, const double2 *, const double *, double, double);
template int two_x<double>(fbse_ctx *, const double2 *, double2 *, long, int, const double2 *, const double *, double, double);
}  // namespace fbse
