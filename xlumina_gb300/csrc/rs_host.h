// Interface between the RS / VRS host entry points (rs.cu) and the kernel
// translation units (rs_q*.cu, one or a few transform lengths each, compiled
// in parallel).
#pragma once

#include "internal.h"

namespace xl {

// Arguments of one RS / VRS launch (device pointers; see XlRsArgs in xlgb.h).
struct RsLaunch {
  int B, cin, cout, ny, nx;
  const float2* in[3];
  long long ibs;
  float2* out[3];
  long long obs;
  const double* x;
  const double* y;
  const double* z;
  const float2* spec;
  long long sstride;
  const int* sidx;
  const float2* const* specs;   // per batch entry (overrides spec / sstride / sidx when set)
  float2* work;
  XlProg pre, post;
  int adjoint;
  int px, py;                   // points of the x and the y transform (px: columns of the intermediate)
  int pol;                      // VRS behind a polarizer: two components, u and Ez (pre without the polarizer)
  float pol_c, pol_s;           // cos and sin of its angle
  int lw;                       // log2 of the intermediate's column-tile width (block engine)
};

// Q = 2^logq is the half transform length: the smallest power of two >= the field
// side, at least 32 (the transfer-spectrum row pass takes G = 256 / T rows per CTA,
// which for Q = 16, P = 32, exceeds P).
inline int rs_logq(int ny, int nx) {
  const int n = ny > nx ? ny : nx;
  const int l = ilog2_ceil(n);
  return l < 5 ? 5 : l;
}

// Fields whose longer side is above 256 run on the block FFT engine, each axis
// with its own transform length, the shortest there is that holds the axis's
// 2 n - 1 points of linear convolution: P = 256 R (R = 4, 6, .. 16) for sides up
// to 2048, two halves of 256 R (R = 10, 12, 14, 16; rs_half.cuh) for longer ones.
// Smaller fields run both axes at 2 Q points on the Stockham engine.
inline bool rs_is_blk(int ny, int nx) { return ny > 256 || nx > 256; }
inline bool rs_is_half(int n) { return n > 2048; }
inline int rs_blk_points(int n) {
  if (rs_is_half(n)) return (n + 511) / 512 * 1024;
  const int r = (2 * n + 511) / 512 * 2;
  return 256 * (r < 4 ? 4 : r);
}
// Points of the x (or y) transform of an ny x nx field.
inline int rs_px(int ny, int nx) { return rs_is_blk(ny, nx) ? rs_blk_points(nx) : 2 << rs_logq(ny, nx); }
inline int rs_py(int ny, int nx) { return rs_is_blk(ny, nx) ? rs_blk_points(ny) : 2 << rs_logq(ny, nx); }

// Block engine passes (explicitly instantiated for R = 4, 6, .. 16 in the
// kernel translation units rs_b*.cu).  hhat_rows: offx / offy wrapped for q2
// points, split into `off` (px + py entries) on the way.
template <int R> int rs_blk_rows(cudaStream_t st, const RsLaunch& p, bool inverse);
template <int R> int rs_blk_cols(cudaStream_t st, const RsLaunch& p);
template <int R>
int rs_blk_hhat_rows(cudaStream_t st, int ny, int nx, int py, const double* offx, const double* offy, int q2, double z,
                     const double* zp, double wavelength, int dz, float2* off, float2* out);
template <int R> int rs_blk_hhat_cols(cudaStream_t st, const float2* in, int px, float scale, float2* out);

// The same for axes of 512 R points in two halves (R = 10, 12, 14, 16, rs_h*.cu).
template <int R> int rs_half_rows(cudaStream_t st, const RsLaunch& p, bool inverse);
template <int R> int rs_half_cols(cudaStream_t st, const RsLaunch& p);
template <int R>
int rs_half_hhat_rows(cudaStream_t st, int ny, int nx, int py, const double* offx, const double* offy, int q2, double z,
                      const double* zp, double wavelength, int dz, float2* off, float2* out);
template <int R> int rs_half_hhat_cols(cudaStream_t st, const float2* in, int px, float scale, float2* out);

// Transfer spectrum and propagation passes for Q = 2^LOGQ (explicitly
// instantiated for LOGQ = 5..8 in a kernel translation unit).
template <int LOGQ>
int rs_spectrum(cudaStream_t st, int ny, int nx, const double* offx, const double* offy, double z,
                const double* zp, double wavelength, double scale, float2* spec, float2* work, int dz);
template <int LOGQ>
int rs_propagate(cudaStream_t st, const RsLaunch& p, int stage);

}  // namespace xl
