// Parallel-beam slice geometry and sampling shared by the spectral-NCC and
// image kernels (torch_engine.py:139-234): slice axes from a pose in FP64 and
// their vector-Jacobian product, the phase ramp, one modulated sample.
#pragma once

#include "fvr_pose.cuh"
#include "fvr_stencil.cuh"

namespace fvr {

// u = R[0,:] * scale, v = R[1,:] * scale with R the (lateral-composed) rotation.
__device__ __forceinline__ void slice_axes(const float* p, int lateral, double sx, double sy, double sz,
                                           double* ax) {
  Mat3 R = euler_R(p[0], p[1], p[2]);
  if (lateral) R = mat_mul(R, lateral_rot());
  ax[0] = R.m[0][0] * sx;
  ax[1] = R.m[0][1] * sy;
  ax[2] = R.m[0][2] * sz;
  ax[3] = R.m[1][0] * sx;
  ax[4] = R.m[1][1] * sy;
  ax[5] = R.m[1][2] * sz;
  ax[6] = p[3];
  ax[7] = p[4];
}

// dL/d(yaw, pitch, roll) from dL/du, dL/dv (slice axes) for one view.
__device__ __forceinline__ void axes_vjp(const float* p, int lateral, double sx, double sy, double sz,
                                         const double du[3], const double dv[3], double out[3]) {
  Mat3 G{{{du[0] * sx, du[1] * sy, du[2] * sz}, {dv[0] * sx, dv[1] * sy, dv[2] * sz}, {0.0, 0.0, 0.0}}};
  if (lateral) G = mat_mul_bt(G, lateral_rot());  // R_total = R_pose . L -> dR_pose = dR_total . L^T
  euler_vjp(p[0], p[1], p[2], G, out);
}

// Compensated phase / pi: the products of the float32 grid values and
// translations are exact in FP64; one rounding to float before sincospif.
__device__ __forceinline__ void phase_sincos(double kpi, float ku, float kv, float tx, float ty, float* sn,
                                             float* cs) {
  const double arg =
      kpi * fma(static_cast<double>(ku), static_cast<double>(tx), static_cast<double>(kv) * static_cast<double>(ty));
  sincospif(static_cast<float>(arg), sn, cs);
}

struct SliceArgs {
  Stencil st;
  const double* axes;  // [C][8]
  const float* lin;
  int R;
  double kpi;
  double sx, sy, sz;
  int shift;  // 1: position ifftshift(q) (image path), 0: natural order
};

__device__ __forceinline__ int shifted_pos(int i, int j, int R, int shift) {
  if (shift) {  // ifftshift: element (i, j) lands at ((i - R/2) mod R, (j - R/2) mod R)
    const int h = R / 2;
    i -= h;
    if (i < 0) i += R;
    j -= h;
    if (j < 0) j += R;
  }
  return i * R + j;
}

template <int DT, bool DERIV>
__device__ __forceinline__ void slice_sample(const SliceArgs& a, const double* ax, float ku, float kv, Interp& o,
                                             float& sn, float& cs) {
  const double dku = ku, dkv = kv;
  stencil_sample_d<DT, DERIV, false>(a.st, fma(dkv, ax[3], fma(dku, ax[0], a.sx)),
                                     fma(dkv, ax[4], fma(dku, ax[1], a.sy)), fma(dkv, ax[5], fma(dku, ax[2], a.sz)),
                                     o);
  phase_sincos(a.kpi, ku, kv, static_cast<float>(ax[6]), static_cast<float>(ax[7]), &sn, &cs);
}

// pair_ok: the caller's kernels also read the x-pair storage (the moments kernels).
inline int stencil_from(int dtype, const void* data, const float* scales, int64_t D, int64_t H, int64_t W,
                        Stencil* s, bool pair_ok = false) {
  if (!data || D < 1 || H < 1 || W < 1 || D > 8192 || H > 8192 || W > 8192) return FVR_ERR_ARG;
  if (dtype != FVR_F32 && dtype != FVR_BF16 && dtype != FVR_F16 &&
      !(pair_ok && (dtype == FVR_BF16_PAIR || dtype == FVR_F16_PAIR || dtype == FVR_F32_PAIR)))
    return FVR_ERR_DTYPE;
  if ((dtype == FVR_F16 || dtype == FVR_F16_PAIR) && !scales) return FVR_ERR_ARG;
  if (dtype == FVR_F32_PAIR && (reinterpret_cast<uintptr_t>(data) & 31) != 0) return FVR_ERR_ARG;  // 256-bit loads
  if ((reinterpret_cast<uintptr_t>(data) & 15) != 0) return FVR_ERR_ARG;
  *s = Stencil{data, scales, static_cast<int>(D), static_cast<int>(H), static_cast<int>(W), dtype};
  return FVR_OK;
}

inline double half_extent(int64_t n) { return 0.5 * static_cast<double>(n > 1 ? n - 1 : 1); }

}  // namespace fvr
