// Stand-alone per-pixel kernels: a Jones program applied outside a
// propagator (masks whose result the caller reads directly).
#include <initializer_list>
#include <type_traits>

#include "common.cuh"
#include "internal.h"

namespace xl {

struct ElemLaunch {
  int B, C, ny, nx;
  const float2* in[3];
  long long ibs;
  float2* out[3];
  long long obs;
  XlProg prog;
};

__global__ void apply_ops_kernel(const ElemLaunch p) {
  const long long npix = (long long)p.ny * p.nx;
  const int b = blockIdx.y;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    float2 e[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    const long long off = (long long)b * p.ibs + i;
    e[0] = p.in[0][off];
    if (p.C > 1) e[1] = p.in[1][off];
    if (p.C > 2) e[2] = p.in[2][off];
    const int row = (int)((unsigned)i / (unsigned)p.nx), col = (int)i - row * p.nx;
    PixelCtx px{row, col, i, b};
    apply_prog(p.prog, e, px);
    const long long o = (long long)b * p.obs + i;
    p.out[0][o] = e[0];
    if (p.C > 1) p.out[1][o] = e[1];
    if (p.C > 2) p.out[2][o] = e[2];
  }
}

// A program applied to a field of ones: the mask that an SLM or a lens returns
// beside the light.
__global__ void mask_kernel(const ElemLaunch p) {
  const long long npix = (long long)p.ny * p.nx;
  const int b = blockIdx.y;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    float2 e[3] = {make_float2(1.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
    const int row = (int)((unsigned)i / (unsigned)p.nx), col = (int)i - row * p.nx;
    apply_prog(p.prog, e, PixelCtx{row, col, i, b});
    p.out[0][(long long)b * p.obs + i] = e[0];
  }
}

// exp(i phase) of n phases, two at a time where both arrays are aligned for it
// (8 and 16 bytes): a warp's accesses are then whole lines, and a thread has
// four loads in flight.  The kernel writes 8 bytes a phase and reads 4.
// 16 x 1024^2 take 34 us, 30 at the copy rate (torch.polar on a plane of ones:
// 61).  One launch under the profiler, the last stores still in L2: 28, with
// four phases a thread, whose two 16-byte stores are half lines each, 36.
constexpr int MASK_THREADS = 256, MASK_IPT = 4;
__global__ void __launch_bounds__(MASK_THREADS) phase_mask_kernel(const float* __restrict__ ph,
                                                                  float2* __restrict__ out, long long n, int vec) {
  const long long step = (long long)MASK_THREADS * MASK_IPT, nv = vec ? n / 2 : 0;
  for (long long base = blockIdx.x * step; base < nv; base += gridDim.x * step) {
    float2 f[MASK_IPT];
#pragma unroll
    for (int q = 0; q < MASK_IPT; ++q) {
      const long long i = base + q * MASK_THREADS + threadIdx.x;
      f[q] = i < nv ? ((const float2*)ph)[i] : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < MASK_IPT; ++q) {
      const long long i = base + q * MASK_THREADS + threadIdx.x;
      float4 o;
      phase_sincos(f[q].x, &o.y, &o.x);
      phase_sincos(f[q].y, &o.w, &o.z);
      if (i < nv) ((float4*)out)[i] = o;
    }
  }
  for (long long i = 2 * nv + blockIdx.x * (long long)MASK_THREADS + threadIdx.x; i < n;
       i += (long long)gridDim.x * MASK_THREADS) {
    float2 a;
    phase_sincos(ph[i], &a.y, &a.x);
    out[i] = a;
  }
}

// The reference's quality factor (wave_optics.py:187-191) of distances on the
// device, in float64.
__global__ void quality_factor_kernel(const double* __restrict__ z, int n, double wl, double rmax, double dr,
                                      double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double zz = z[i];
  // products and sums rounded one by one, as the host form of it rounds them
  const double r2 = __dmul_rn(rmax, rmax);
  const double hyp = sqrt(__dadd_rn(r2, __dmul_rn(zz, zz)));
  const double len = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(wl, wl), r2), __dmul_rn(2.0 * wl, hyp)));
  out[i] = (len - rmax) / dr;
}

struct OpsBwdLaunch {
  int B, C, ny, nx;
  const float2* in[3];
  long long ibs;
  const float2* gout[3];
  long long gbs;
  float2* gin[3];
  long long ginbs;
  XlProg prog;
  void* pgrad[XL_MAX_OPS * 4];
};

// One thread per pixel and batch entry, or (when a per-pixel parameter shared
// by the whole batch needs its gradient) one thread per pixel looping over
// the batch, so that the batch sum runs in a fixed order.  The op loops are
// unrolled to KMAX so the per-op intermediates stay in registers.  Dynamic
// shared memory holds, [slot][thread] so that a warp's accesses fall in
// distinct banks: the scalar-parameter partial sums (when any scalar
// gradient is asked for), then the shared-plane batch sums (when needed).
//
// FK: the program's op kinds fixed at compile time (FixedKinds<...>, for the
// programs the tables run), so that the per-op switches fold and the trig
// stays in registers; FixedKinds<> reads them from the program.

// IN: the input's gradient is wanted (otherwise the first op's part of it is not
// formed).
template <int KMAX, bool IN, class FK = FixedKinds<>>
__global__ void __launch_bounds__(128) ops_backward_kernel(const OpsBwdLaunch p, int scalar_acc, int plane_acc) {
  constexpr int NS = XL_MAX_OPS * 4;
  constexpr int NT = 128;
  constexpr bool FIXED = FK::n > 0;
  static_assert(!FIXED || FK::n == KMAX, "a fixed program unrolls to its length");
  extern __shared__ float accm[];
  // the trig of every op the forward recompute applies, for its backward
  // (thread-private slots, so no barrier): evaluated once per pixel and entry.
  // A fixed program keeps it in registers instead.
  __shared__ float4 trig_s[FIXED ? 1 : KMAX - 1][NT];
  float* acc_s = accm;                              // NS x NT, when scalar_acc
  float* acc_p = accm + (scalar_acc ? NS * NT : 0); // NS x NT, when plane_acc
  const long long npix = (long long)p.ny * p.nx;
  const int K = FIXED ? FK::n : p.prog.nops;
  auto kind = [&](int k) { return FIXED ? FK::at(k) : p.prog.ops[k].kind; };
  const int tid = threadIdx.x;
  const int b_lo = gridDim.y > 1 ? blockIdx.y : 0;
  const int b_hi = gridDim.y > 1 ? blockIdx.y + 1 : p.B;
  if (scalar_acc)
    for (int q = 0; q < NS; ++q) acc_s[q * NT + tid] = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)((unsigned)i / (unsigned)p.nx), col = (int)i - row * p.nx;
    if (plane_acc)
      for (int q = 0; q < 4 * K; ++q) acc_p[q * NT + tid] = 0.f;
    // the high-NA lens depends on the pixel only: its coefficients are hoisted out of the batch loop
    float kc[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    int hk = -1;
    {
      PixelCtx px0{row, col, i, 0};
#pragma unroll
      for (int k = 0; k < KMAX; ++k)
        if (k < K && hk < 0 && (kind(k) == XL_OP_HIGHNA || kind(k) == XL_OP_HIGHNA_EZ)) {
          highna_coeffs(p.prog.ops[k], px0, kc);
          hk = k;
        }
    }
    for (int b = b_lo; b < b_hi; ++b) {
      PixelCtx px{row, col, i, b};
      float2 st[KMAX][3];
      float4 trig_r[KMAX];
      float2 e[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      const long long off = (long long)b * p.ibs + i;
      e[0] = p.in[0][off];
      if (p.C > 1 && p.in[1]) e[1] = p.in[1][off];
      if (p.C > 2 && p.in[2]) e[2] = p.in[2][off];
      float2 g[3] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
      const long long go = (long long)b * p.gbs + i;
      float pv[KMAX][2];
      if constexpr (FIXED) {
        // every load of the pixel before the first sine: their slow paths are
        // branches, past which no load is moved up, and each op's loads were
        // waited for by themselves (8 x 2048^2 LCD, sSLM, lens Ez row: 589 us,
        // now 480; LCD and polarizer 448 and 353)
        g[0] = p.gout[0][go];
        if (p.C > 1 && p.gout[1]) g[1] = p.gout[1][go];
        if (p.C > 2 && p.gout[2]) g[2] = p.gout[2][go];
#pragma unroll
        for (int k = 0; k < KMAX; ++k)
#pragma unroll
          for (int q = 0; q < 2; ++q)
            if (kind(k) == XL_OP_LCD || kind(k) == XL_OP_SSLM || (q == 0 && (kind(k) == XL_OP_PHASE || kind(k) == XL_OP_LP)))
              pv[k][q] = op_param(p.prog.ops[k], q, px);
      }
      auto trig_of = [&](int k) {
        const XlOp& op = p.prog.ops[k];
        if constexpr (FIXED) return op_trig_p(kind(k), op, [&](int q) { return pv[k][q]; });
        else return op_trig(kind(k), op, px);
      };
      // forward recompute: the input of every op (the last op's output is not needed)
#pragma unroll
      for (int k = 0; k < KMAX; ++k) {
        if (k < K) {
          st[k][0] = e[0]; st[k][1] = e[1]; st[k][2] = e[2];
          if (k + 1 < K) {
            if (k == hk) {
              if (kind(k) == XL_OP_HIGHNA) apply_highna(kc, e);
              else apply_highna_ez(kc, e);
            } else if (k < KMAX - 1) {
              const float4 t = trig_of(k);
              if constexpr (FIXED) trig_r[k] = t;
              else trig_s[FIXED ? 0 : k][tid] = t;
              apply_op_t(kind(k), p.prog.ops[k], t, e, px);
            }
          }
        }
      }
      if constexpr (!FIXED) {
        g[0] = p.gout[0][go];
        if (p.C > 1 && p.gout[1]) g[1] = p.gout[1][go];
        if (p.C > 2 && p.gout[2]) g[2] = p.gout[2][go];
      }
#pragma unroll
      for (int k = KMAX - 1; k >= 0; --k) {
        if (k < K) {
          const XlOp& op = p.prog.ops[k];
          float pg[4] = {0.f, 0.f, 0.f, 0.f};
          const float2 ek[3] = {st[k][0], st[k][1], st[k][2]};
          if (k == hk) {
            if (kind(k) == XL_OP_HIGHNA) apply_highna_bwd(kc, g);
            else apply_highna_ez_bwd(kc, g);
          }
          else if (k + 1 < K && k < KMAX - 1)
            apply_op_bwd_t(kind(k), op, FIXED ? trig_r[k] : trig_s[FIXED ? 0 : k][tid], ek, g, px, pg);
          else apply_op_bwd_t(kind(k), op, trig_of(k), ek, g, px, pg);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            void* dst = p.pgrad[k * 4 + q];
            if (!dst) continue;
            if (op.pmask & (1 << q)) {
              if (op.pbstride) ((float*)dst)[(long long)b * op.pbstride + i] = pg[q];
              else acc_p[(k * 4 + q) * NT + tid] += pg[q];
            } else {
              acc_s[(k * 4 + q) * NT + tid] += pg[q];
            }
          }
        }
      }
      if constexpr (IN) {
        const long long gi = (long long)b * p.ginbs + i;
        if (p.gin[0]) p.gin[0][gi] = g[0];
        if (p.C > 1 && p.gin[1]) p.gin[1][gi] = g[1];
        if (p.C > 2 && p.gin[2]) p.gin[2][gi] = g[2];
      }
    }
    if (plane_acc)
      for (int k = 0; k < K; ++k)
        for (int q = 0; q < 4; ++q) {
          const XlOp& op = p.prog.ops[k];
          if (p.pgrad[k * 4 + q] && (op.pmask & (1 << q)) && !op.pbstride)
            ((float*)p.pgrad[k * 4 + q])[i] = acc_p[(k * 4 + q) * NT + tid];
        }
  }
  if (!scalar_acc) return;
  // scalar parameters: block reduction, one float64 atomic per block and slot
  __shared__ float red[8];
  const int lane = tid & 31, warp = tid >> 5;
  for (int k = 0; k < K; ++k)
    for (int q = 0; q < 4; ++q) {
      const XlOp& op = p.prog.ops[k];
      if (!p.pgrad[k * 4 + q] || (op.pmask & (1 << q))) continue;
      float v = acc_s[(k * 4 + q) * NT + tid];
      for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) red[warp] = v;
      __syncthreads();
      if (tid == 0) {
        double t = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) t += red[w];
        atomicAdd((double*)p.pgrad[k * 4 + q], t);
      }
      __syncthreads();
    }
}

// Scalar programs of one op, two pixels a thread in 16-byte accesses: a phase
// SLM with its gradient in a plane per batch entry, and a separable mask (no
// parameter gradient; the forward's input is not read).  The kernel above, one
// pixel a thread, does not keep enough bytes in flight: 16 x 1024^2, phase 110
// us, with the input's gradient 121, mask 98; these take 62, 85 and 47 (at the
// copy rate 59, 79 and 40).
template <bool IN>
__global__ void __launch_bounds__(256) phase_backward_kernel(const OpsBwdLaunch p) {
  const long long n2 = (long long)p.ny * p.nx / 2;
  const int b = blockIdx.y;
  const XlOp& op = p.prog.ops[0];
  const float4* e2 = (const float4*)(p.in[0] + (long long)b * p.ibs);
  const float4* g2 = (const float4*)(p.gout[0] + (long long)b * p.gbs);
  const float2* f2 = (const float2*)((const float*)op.ptr[0] + (long long)b * op.pbstride);
  float2* d2 = (float2*)((float*)p.pgrad[0] + (long long)b * op.pbstride);
  float4* o2 = (float4*)(p.gin[0] + (long long)b * p.ginbs);
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n2; i += (long long)gridDim.x * blockDim.x) {
    const float4 e = e2[i], g = g2[i];
    const float2 f = f2[i];
    float2 s, c;
    phase_sincos(f.x, &s.x, &c.x);
    phase_sincos(f.y, &s.y, &c.y);
    const float2 a = cmulc(make_float2(g.x, g.y), make_float2(c.x, s.x));
    const float2 h = cmulc(make_float2(g.z, g.w), make_float2(c.y, s.y));
    d2[i] = make_float2(re_gconj_i(a, make_float2(e.x, e.y)), re_gconj_i(h, make_float2(e.z, e.w)));
    if constexpr (IN) o2[i] = make_float4(a.x, a.y, h.x, h.y);
  }
}

// tc + tr < 1 as float64 arithmetic gives it.  GB300's FP64 pipe takes 16 cycles
// a warp and operation (it was 79 % busy with two a pixel), so the sum is
// formed in float from the operands' bits (truncated, within 1e-6) and float64
// is used only where that is within 1e-4 of 1, or an operand is negative, not
// finite or huge.
__device__ __forceinline__ bool pupil_inside(double tc, double tr) {
  auto bits = [](double v) -> float {   // 0 below 2^-126
    const int hi = __double2hiint(v), lo = __double2loint(v);
    return hi < (897 << 20) ? 0.f : __int_as_float(((hi - (896 << 20)) << 3) | (int)((unsigned)lo >> 29));
  };
  constexpr unsigned BIG = 1150u << 20;   // the high word of 2^127; above it negative values, infinities, NaNs
  if ((unsigned)__double2hiint(tc) < BIG && (unsigned)__double2hiint(tr) < BIG) {
    const float s = bits(tc) + bits(tr);
    if (s < 0.9999f) return true;
    if (s > 1.0001f) return false;
  }
  return tc + tr < 1.0;
}

__global__ void __launch_bounds__(256) sepmask_backward_kernel(const OpsBwdLaunch p) {
  const unsigned n2 = (unsigned)((long long)p.ny * p.nx / 2), half = (unsigned)p.nx / 2;
  const int b = blockIdx.y;
  const XlOp& op = p.prog.ops[0];
  const float4* g2 = (const float4*)(p.gout[0] + (long long)b * p.gbs);
  float4* o2 = (float4*)(p.gin[0] + (long long)b * p.ginbs);
  const float2* fc = (const float2*)op.ptr[0];
  const float2* fr = (const float2*)op.ptr[1];
  const double* tc = (const double*)op.ptr[2];
  const double* tr = (const double*)op.ptr[3];
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n2; i += gridDim.x * blockDim.x) {
    const unsigned row = i / half, col = 2 * (i - row * half);
    const float4 g = g2[i];
    float2 m0 = cmul(fc[col], fr[row]), m1 = cmul(fc[col + 1], fr[row]);
    if (tc) {
      const double t = tr[row];
      if (!pupil_inside(tc[col], t)) m0 = make_float2(0.f, 0.f);
      if (!pupil_inside(tc[col + 1], t)) m1 = make_float2(0.f, 0.f);
    }
    const float2 a = cmulc(make_float2(g.x, g.y), m0), h = cmulc(make_float2(g.z, g.w), m1);
    o2[i] = make_float4(a.x, a.y, h.x, h.y);
  }
}

// Whether one of the two kernels above takes a launch: scalar, one op of its
// kind, planes and strides that keep every pair 16-byte (parameters: 8-byte)
// aligned, a phase plane per entry (its gradient needs no sum over the batch).
static bool pairs_ok(const OpsBwdLaunch& p) {
  if (p.C != 1 || p.prog.nops != 1 || p.B > 65535) return false;
  const XlOp& op = p.prog.ops[0];
  auto al = [](const void* q, int n) { return ((uintptr_t)q % n) == 0; };
  if (((long long)p.ny * p.nx) % 2 || p.gbs % 2 || !al(p.gout[0], 16)) return false;
  if (p.gin[0] && (p.ginbs % 2 || !al(p.gin[0], 16))) return false;
  if (op.kind == XL_OP_PHASE)
    return (op.pmask & 1) && p.pgrad[0] && (op.pbstride || p.B == 1) && op.pbstride % 2 == 0 && p.ibs % 2 == 0 &&
           al(p.in[0], 16) && al(op.ptr[0], 8) && al(p.pgrad[0], 8);
  return op.kind == XL_OP_SEPMASK && p.nx % 2 == 0 && p.gin[0];
}

__global__ void highna_plane_kernel(int ny, int nx, XlOp op, float* out) {
  const long long npix = (long long)ny * nx;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)((unsigned)i / (unsigned)nx);
    PixelCtx px{row, (int)i - row * nx, i, 0};
    float kc[6];
    highna_coeffs(op, px, kc);
#pragma unroll
    for (int q = 0; q < 6; ++q) out[q * npix + i] = kc[q];
  }
}

// ---- intensity MSE (loss_functions.py:137-149) ----
// loss[p] = sum_i (|a_i|^2 - |b_i|^2)^2 / npix for plane p; the sum runs in two
// fixed-order stages (per-block float partials in float64, then per plane),
// so the result does not depend on scheduling.
constexpr int MSE_THREADS = 256;

// Per-plane reductions of a pixel function f(a_i, b_i): KIND 0 the intensity
// MSE term (|a|^2 - |b|^2)^2, KIND 1 the real inner product Re(conj(a) b),
// KIND 2 the amplitude term (|a| - |b|)^2, KIND 3 the phase term
// (arg a - arg b)^2 (loss_functions.py:109-135).
template <int KIND>
__device__ __forceinline__ void plane_sum_block(const float2* __restrict__ a, const float2* __restrict__ b,
                                                long long npix, double* __restrict__ partial) {
  float acc = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    const float2 u = a[i], v = b[i];
    if (KIND == 0) {
      const float d = (u.x * u.x + u.y * u.y) - (v.x * v.x + v.y * v.y);
      acc = fmaf(d, d, acc);
    } else if (KIND == 1) {
      acc = fmaf(u.x, v.x, fmaf(u.y, v.y, acc));
    } else if (KIND == 2) {
      const float d = hypotf(u.x, u.y) - hypotf(v.x, v.y);
      acc = fmaf(d, d, acc);
    } else {
      const float d = atan2f(u.y, u.x) - atan2f(v.y, v.x);
      acc = fmaf(d, d, acc);
    }
  }
  __shared__ float red[MSE_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < MSE_THREADS / 32; ++w) t += red[w];
    *partial = t;
  }
}
template <int KIND>
__global__ void __launch_bounds__(MSE_THREADS) plane_sum_partial(const float2* __restrict__ a, long long aps,
                                                                 const float2* __restrict__ b, long long bps,
                                                                 long long npix, double* __restrict__ partial) {
  const int plane = blockIdx.y;
  plane_sum_block<KIND>(a + (long long)plane * aps, b + (long long)plane * bps, npix,
                        partial + (long long)plane * gridDim.x + blockIdx.x);
}

// The intensity MSE of three components in tensors of their own (grid z), and
// its gradient: one launch each instead of three.  A vector light's loss is a
// chain of short kernels: 1024^2 with gradients, through autograd, 310 us (three
// runs 308 to 319), with a launch a component 510 (499 to 520).
struct Vmse {
  const float2* a[3];
  const float2* b[3];
  float2* ga[3];
  float2* gb[3];
};
__global__ void __launch_bounds__(MSE_THREADS) vmse_partial(const Vmse p, long long aps, long long bps, long long npix,
                                                            double* __restrict__ partial) {
  const int plane = blockIdx.y, c = blockIdx.z;
  plane_sum_block<0>(p.a[c] + plane * aps, p.b[c] + plane * bps, npix,
                     partial + ((long long)c * gridDim.y + plane) * gridDim.x + blockIdx.x);
}

// One warp per plane: lane l sums partials l, l + 32, ... in order, then a
// fixed shuffle tree (the same order on every call).
__global__ void mse_int_finish(const double* __restrict__ partial, int nblk, int planes, double inv_n,
                               float* __restrict__ out) {
  const int plane = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (plane >= planes) return;
  double t = 0.0;
  for (int k = lane; k < nblk; k += 32) t += partial[(long long)plane * nblk + k];
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  if (lane == 0) out[plane] = (float)(t * inv_n);
}

// Gradients of loss[p] with upstream gradient g[p] (torch's convention for
// complex tensors, 2 dL/d conj): ga = 4 g (|a|^2 - |b|^2) a / npix and
// gb = -4 g (|a|^2 - |b|^2) b / npix (either may be NULL).
__device__ __forceinline__ void mse_grad_block(const float2* __restrict__ a, const float2* __restrict__ b,
                                               long long npix, float s, float2* __restrict__ ga,
                                               float2* __restrict__ gb) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    const float2 u = a[i], v = b[i];
    const float d = s * ((u.x * u.x + u.y * u.y) - (v.x * v.x + v.y * v.y));
    if (ga) ga[i] = make_float2(d * u.x, d * u.y);
    if (gb) gb[i] = make_float2(-d * v.x, -d * v.y);
  }
}
__global__ void mse_int_grad(const float2* __restrict__ a, long long aps, const float2* __restrict__ b,
                             long long bps, long long npix, const float* __restrict__ g, float four_inv_n,
                             float2* __restrict__ ga, float2* __restrict__ gb) {
  const long long plane = blockIdx.y, o = plane * npix;
  mse_grad_block(a + plane * aps, b + plane * bps, npix, g[plane] * four_inv_n, ga ? ga + o : nullptr,
                 gb ? gb + o : nullptr);
}
__global__ void vmse_grad(const Vmse p, long long aps, long long bps, long long npix, const float* __restrict__ g,
                          float four_inv_n) {
  const long long plane = blockIdx.y, c = blockIdx.z, o = plane * npix;
  if (!p.ga[c] && !p.gb[c]) return;
  mse_grad_block(p.a[c] + plane * aps, p.b[c] + plane * bps, npix, g[c * gridDim.y + plane] * four_inv_n,
                 p.ga[c] ? p.ga[c] + o : nullptr, p.gb[c] ? p.gb[c] + o : nullptr);
}

// Gradients of the amplitude (KIND 2) and phase (KIND 3) MSE per plane with
// upstream gradient g[p] (torch's convention, 2 dL/d conj):
// amplitude: ga = 2 g (|a| - |b|) a / (|a| npix), gb = -2 g (|a| - |b|) b / (|b| npix);
// phase: ga = 2 g (arg a - arg b) i a / (|a|^2 npix), gb the same with -i b / |b|^2;
// zero where |a| (|b|) is zero, as torch's abs and angle give.
template <int KIND>
__global__ void amp_phase_grad(const float2* __restrict__ a, long long aps, const float2* __restrict__ b,
                               long long bps, long long npix, const float* __restrict__ g, float two_inv_n,
                               float2* __restrict__ ga, float2* __restrict__ gb) {
  const int plane = blockIdx.y;
  a += (long long)plane * aps;
  b += (long long)plane * bps;
  const float s = g[plane] * two_inv_n;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    const float2 u = a[i], v = b[i];
    float2 ru, rv;
    if (KIND == 2) {
      const float au = hypotf(u.x, u.y), av = hypotf(v.x, v.y);
      const float d = s * (au - av);
      const float fu = au > 0.f ? d / au : 0.f, fv = av > 0.f ? -d / av : 0.f;
      ru = make_float2(fu * u.x, fu * u.y);
      rv = make_float2(fv * v.x, fv * v.y);
    } else {
      const float d = s * (atan2f(u.y, u.x) - atan2f(v.y, v.x));
      const float nu = u.x * u.x + u.y * u.y, nv = v.x * v.x + v.y * v.y;
      const float fu = nu > 0.f ? d / nu : 0.f, fv = nv > 0.f ? -d / nv : 0.f;
      ru = make_float2(-fu * u.y, fu * u.x);
      rv = make_float2(-fv * v.y, fv * v.x);
    }
    if (ga) ga[(long long)plane * npix + i] = ru;
    if (gb) gb[(long long)plane * npix + i] = rv;
  }
}

// The z-derivative of the VRS Ez derivation, reduced against the Ez gradient:
// per batch entry b, sum_i Re(conj(g_i) dEz_i/dz) with
// dEz/dz = -(Ex X + Ey Y) z / r^3, r^2 = X^2 + Y^2 + z^2 (vectorized_optics.py:258-261).
__global__ void __launch_bounds__(MSE_THREADS) vrs_dz_ez_partial(const float2* __restrict__ ex,
                                                                 const float2* __restrict__ ey, long long ebs,
                                                                 const float2* __restrict__ g, long long gbs,
                                                                 int ny, int nx, const double* __restrict__ x,
                                                                 const double* __restrict__ y,
                                                                 const double* __restrict__ z,
                                                                 double* __restrict__ partial) {
  const int b = blockIdx.y;
  const long long npix = (long long)ny * nx;
  ex += (long long)b * ebs;
  ey += (long long)b * ebs;
  g += (long long)b * gbs;
  const float zf = (float)z[b];
  float acc = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    const int row = (int)((unsigned)i / (unsigned)nx), col = (int)i - row * nx;
    const float X = (float)x[col], Y = (float)y[row];
    const float ir = rsqrtf(X * X + Y * Y + zf * zf);
    const float w = -zf * ir * ir * ir;
    const float2 u = ex[i], v = ey[i], gg = g[i];
    const float2 d = make_float2(w * (u.x * X + v.x * Y), w * (u.y * X + v.y * Y));
    acc = fmaf(gg.x, d.x, fmaf(gg.y, d.y, acc));
  }
  __shared__ float red[MSE_THREADS / 32];
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w2 = 0; w2 < MSE_THREADS / 32; ++w2) t += red[w2];
    partial[(long long)b * gridDim.x + blockIdx.x] = t;
  }
}

// The whole distance gradient of one RS / VRS call per batch entry b:
// sum_c sum_i Re(conj(g_c) d_c) over the propagated components (d: the
// propagation through the dH/dz spectrum) plus, for VRS, sum_i Re(conj(gez)
// dEz/dz) of the input-plane Ez derivation -- one pass instead of a reduction
// per component.
struct ZGradArgs {
  const float2* g[3];
  const float2* d[3];
  long long bs;          // batch stride of g and d (elements)
  int ncomp;
  const float2* ex;      // VRS: the Jones program's output (NULL: scalar RS)
  const float2* ey;
  long long ebs;
  const float2* gez;     // VRS: the propagated Ez gradient before its fold
  const double* x;
  const double* y;
  const double* z;       // one per batch entry
  int ny, nx;
};

__global__ void __launch_bounds__(MSE_THREADS) rs_zgrad_partial(ZGradArgs p, double* __restrict__ partial) {
  const int b = blockIdx.y;
  const long long npix = (long long)p.ny * p.nx;
  const long long o = (long long)b * p.bs;
  float acc = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < npix;
       i += (long long)gridDim.x * blockDim.x) {
    for (int c = 0; c < p.ncomp; ++c) {
      const float2 u = p.g[c][o + i], v = p.d[c][o + i];
      acc = fmaf(u.x, v.x, fmaf(u.y, v.y, acc));
    }
    if (p.ex) {
      const int row = (int)((unsigned)i / (unsigned)p.nx), col = (int)i - row * p.nx;
      const float X = (float)p.x[col], Y = (float)p.y[row], zf = (float)p.z[b];
      const float ir = rsqrtf(X * X + Y * Y + zf * zf);
      const float w = -zf * ir * ir * ir;
      const float2 u = p.ex[(long long)b * p.ebs + i], v = p.ey[(long long)b * p.ebs + i], gg = p.gez[o + i];
      acc = fmaf(gg.x, w * (u.x * X + v.x * Y), fmaf(gg.y, w * (u.y * X + v.y * Y), acc));
    }
  }
  __shared__ float red[MSE_THREADS / 32];
  for (int s = 16; s > 0; s >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < MSE_THREADS / 32; ++w) t += red[w];
    partial[(long long)b * gridDim.x + blockIdx.x] = t;
  }
}

static int mse_blocks(long long npix) {
  long long nb = (npix + MSE_THREADS * 8 - 1) / (MSE_THREADS * 8);
  if (nb > 152 * 4) nb = 152 * 4;
  return nb < 1 ? 1 : (int)nb;
}

static cudaError_t elem_upload_twiddles(const float2* host) {
  return cudaMemcpyToSymbol(g_tw, host, sizeof(g_tw));
}

static const bool elem_registered = register_device_tables(&elem_upload_twiddles, nullptr);

}  // namespace xl

using namespace xl;

extern "C" int xl_ops_backward(void* stream, int batch, int comps, int ny, int nx, const void* const* in,
                               long long in_bstride, const void* const* gout, long long gout_bstride,
                               void* const* gin, long long gin_bstride, const XlProg* prog,
                               void* const* pgrad) {
  if (batch < 1 || comps < 1 || comps > 3 || ny < 1 || nx < 1 || !in || !gout || !gin || !prog) {
    set_error("xl_ops_backward: bad arguments");
    return XL_EINVAL;
  }
  if (prog->nops < 0 || prog->nops > XL_MAX_OPS) {
    set_error("xl_ops_backward: op program too long");
    return XL_EINVAL;
  }
  OpsBwdLaunch p;
  p.B = batch; p.C = comps; p.ny = ny; p.nx = nx;
  p.ibs = in_bstride; p.gbs = gout_bstride; p.ginbs = gin_bstride;
  for (int c = 0; c < 3; ++c) {
    p.in[c] = c < comps ? (const float2*)in[c] : nullptr;
    p.gout[c] = c < comps ? (const float2*)gout[c] : nullptr;
    p.gin[c] = c < comps ? (float2*)gin[c] : nullptr;
    if (c == 0 && (!p.in[0] || !p.gout[0])) {
      set_error("xl_ops_backward: null plane %d", c);
      return XL_EINVAL;
    }
  }
  p.prog = *prog;
  for (int q = 0; q < XL_MAX_OPS * 4; ++q) p.pgrad[q] = pgrad ? pgrad[q] : nullptr;
  // which gradients need accumulation: scalar parameters (summed over all
  // pixels) and per-pixel parameters shared by the batch (summed over it)
  int scalar_acc = 0, plane_acc = 0;
  for (int k = 0; k < prog->nops; ++k)
    for (int q = 0; q < 4; ++q) {
      if (!p.pgrad[k * 4 + q]) continue;
      const XlOp& op = prog->ops[k];
      if (!(op.pmask & (1 << q))) scalar_acc = 1;
      else if (!op.pbstride) plane_acc = 1;
    }
  const long long npix = (long long)ny * nx;
  if (npix > 0x7fffffffLL) {
    set_error("xl_ops_backward: plane too large");
    return XL_EINVAL;
  }
  const long long need = (npix + 127) / 128;
  // without batch sums, one thread per pixel and batch entry (grid.y = batch)
  const int gy = (plane_acc || batch > 65535) ? 1 : batch;
  const size_t sm = (size_t)(scalar_acc + plane_acc) * XL_MAX_OPS * 4 * 128 * sizeof(float);
  int dev = 0, sms = 152;
  if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    sms = 152;
  // one wave: the CTAs that fit on the device at once (the pixel loop strides
  // over the rest), so that no second, partly empty wave follows
  auto grid_for = [&](auto kernel) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 128, sm) != cudaSuccess || per_sm < 1)
      per_sm = 4;
    long long bx = ((long long)per_sm * sms + gy - 1) / gy;
    if (bx > need) bx = need;
    if (bx < 1) bx = 1;
    return dim3((unsigned)bx, gy);
  };
  // programs the tables and the benchmarks run get a kernel with their op
  // kinds fixed (the high-NA table's LCD-sSLM-lens, the VRS benchmark's
  // LCD-polarizer, the 4f table's phase SLM and thin lens); any other
  // program takes the generic one
  auto is = [&](std::initializer_list<int> ks) {
    if ((int)ks.size() != prog->nops) return false;
    int k = 0;
    for (int v : ks)
      if (prog->ops[k++].kind != v) return false;
    return true;
  };
  cudaStream_t s = (cudaStream_t)stream;
  const bool want_in = p.gin[0] || p.gin[1] || p.gin[2];
  if (pairs_ok(p)) {
    // about 16 blocks an SM over the batch, no more than the pairs need
    long long bx = (npix / 2 + 255) / 256, most = (16LL * sms + batch - 1) / batch;
    if (bx > most) bx = most;
    const dim3 grid((unsigned)(bx < 1 ? 1 : bx), batch);
    if (prog->ops[0].kind == XL_OP_SEPMASK) sepmask_backward_kernel<<<grid, 256, 0, s>>>(p);
    else if (want_in) phase_backward_kernel<true><<<grid, 256, 0, s>>>(p);
    else phase_backward_kernel<false><<<grid, 256, 0, s>>>(p);
    XL_CHECK_LAUNCH("one-op backward");
    return XL_OK;
  }
  auto run = [&](auto kernel) { kernel<<<grid_for(kernel), 128, sm, s>>>(p, scalar_acc, plane_acc); };
  auto pick = [&](auto in) {
    constexpr bool IN = decltype(in)::value;
    if (is({XL_OP_LCD, XL_OP_SSLM, XL_OP_HIGHNA_EZ}))
      run(ops_backward_kernel<3, IN, FixedKinds<XL_OP_LCD, XL_OP_SSLM, XL_OP_HIGHNA_EZ>>);
    else if (is({XL_OP_LCD, XL_OP_SSLM, XL_OP_HIGHNA}))
      run(ops_backward_kernel<3, IN, FixedKinds<XL_OP_LCD, XL_OP_SSLM, XL_OP_HIGHNA>>);
    else if (is({XL_OP_LCD, XL_OP_LP}))
      run(ops_backward_kernel<2, IN, FixedKinds<XL_OP_LCD, XL_OP_LP>>);
    else if (is({XL_OP_PHASE}))
      run(ops_backward_kernel<1, IN, FixedKinds<XL_OP_PHASE>>);
    else if (is({XL_OP_SEPMASK}))
      run(ops_backward_kernel<1, IN, FixedKinds<XL_OP_SEPMASK>>);
    else if (prog->nops <= 4)
      run(ops_backward_kernel<4, IN>);
    else
      run(ops_backward_kernel<XL_MAX_OPS, IN>);
  };
  if (want_in) pick(std::true_type{});
  else pick(std::false_type{});
  XL_CHECK_LAUNCH("ops_backward_kernel");
  return XL_OK;
}

namespace xl {
// The transfer function of the chirp-z prologue and epilogue on a whole grid,
// evaluated by the same device function (rs_kernel_value) as the kernels.
__global__ void __launch_bounds__(256) czt_transfer_plane_kernel(int ny, int nx, const double* __restrict__ x,
                                                                 const double* __restrict__ y, double z,
                                                                 double inv_lambda, float k, float2* out) {
  const long long n = (long long)ny * nx;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    const int r = (int)(i / nx), c = (int)(i - (long long)r * nx);
    out[i] = rs_kernel_value(x[c], y[r], z, inv_lambda, k);
  }
}
}  // namespace xl

extern "C" int xl_czt_transfer_plane(void* stream, int ny, int nx, const double* x, const double* y, double z,
                                     double wavelength, void* out) {
  if (ny < 1 || nx < 1 || !x || !y || !out || !(wavelength > 0)) {
    set_error("xl_czt_transfer_plane: bad arguments");
    return XL_EINVAL;
  }
  if (int rc = ensure_init()) return rc;
  const long long n = (long long)ny * nx;
  long long blocks = (n + 255) / 256;
  if (blocks > 152 * 8) blocks = 152 * 8;
  czt_transfer_plane_kernel<<<(unsigned)blocks, 256, 0, (cudaStream_t)stream>>>(
      ny, nx, x, y, z, 1.0 / wavelength, (float)(2.0 * M_PI / wavelength), (float2*)out);
  XL_CHECK_LAUNCH("czt_transfer_plane_kernel");
  return XL_OK;
}

extern "C" int xl_highna_coefficients(void* stream, int ny, int nx, const double* x, const double* y,
                                      double radius, double f, void* out) {
  if (ny < 1 || nx < 1 || !x || !y || !out || !(radius > 0) || !(f > 0)) {
    set_error("xl_highna_coefficients: bad arguments");
    return XL_EINVAL;
  }
  XlOp op = {};
  op.kind = XL_OP_HIGHNA;
  op.ptr[0] = x;
  op.ptr[1] = y;
  op.dval[0] = radius;
  op.dval[1] = f;
  op.dval[2] = radius / sqrt(radius * radius + f * f);
  op.dval[3] = 1.0 / (radius * radius);
  const long long npix = (long long)ny * nx;
  int blocks = (int)((npix + 255) / 256);
  if (blocks > 152 * 8) blocks = 152 * 8;
  highna_plane_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(ny, nx, op, (float*)out);
  XL_CHECK_LAUNCH("highna_plane_kernel");
  return XL_OK;
}

extern "C" int xl_mask_planes(void* stream, int batch, int ny, int nx, void* out, long long out_bstride,
                              const XlProg* prog) {
  if (batch < 1 || batch > 65535 || ny < 1 || nx < 1 || !out || !prog || (long long)ny * nx > 0x7fffffffLL ||
      prog->nops < 0 || prog->nops > XL_MAX_OPS) {
    set_error("xl_mask_planes: bad arguments");
    return XL_EINVAL;
  }
  const long long npix = (long long)ny * nx;
  cudaStream_t s = (cudaStream_t)stream;
  const XlOp& op = prog->ops[0];
  if (prog->nops == 1 && op.kind == XL_OP_PHASE && (op.pmask & 1) &&
      (batch == 1 || (op.pbstride == npix && out_bstride == npix))) {
    const long long n = npix * batch;
    long long blocks = (n + 2 * MASK_THREADS * MASK_IPT - 1) / (2 * MASK_THREADS * MASK_IPT);
    if (blocks > (1 << 20)) blocks = 1 << 20;
    const int vec = ((uintptr_t)op.ptr[0] & 7) == 0 && ((uintptr_t)out & 15) == 0;
    phase_mask_kernel<<<(unsigned)blocks, MASK_THREADS, 0, s>>>((const float*)op.ptr[0], (float2*)out, n, vec);
    XL_CHECK_LAUNCH("phase_mask_kernel");
    return XL_OK;
  }
  ElemLaunch p = {};
  p.B = batch; p.C = 1; p.ny = ny; p.nx = nx;
  p.out[0] = (float2*)out;
  p.obs = out_bstride;
  p.prog = *prog;
  long long blocks = (npix + 255) / 256;
  if (blocks > 152 * 8) blocks = 152 * 8;
  mask_kernel<<<dim3((unsigned)blocks, batch), 256, 0, s>>>(p);
  XL_CHECK_LAUNCH("mask_kernel");
  return XL_OK;
}

extern "C" int xl_quality_factor(void* stream, const double* z, int n, double wavelength, double rmax, double dr,
                                 double* out) {
  if (n < 1 || !z || !out) {
    set_error("xl_quality_factor: bad arguments");
    return XL_EINVAL;
  }
  quality_factor_kernel<<<(n + 127) / 128, 128, 0, (cudaStream_t)stream>>>(z, n, wavelength, rmax, dr, out);
  XL_CHECK_LAUNCH("quality_factor_kernel");
  return XL_OK;
}

extern "C" int xl_apply_ops(void* stream, int batch, int comps, int ny, int nx, const void* const* in,
                            long long in_bstride, void* const* out, long long out_bstride,
                            const XlProg* prog) {
  if (batch < 1 || comps < 1 || comps > 3 || ny < 1 || nx < 1 || !in || !out || !prog) {
    set_error("xl_apply_ops: bad arguments");
    return XL_EINVAL;
  }
  if (prog->nops < 0 || prog->nops > XL_MAX_OPS) {
    set_error("xl_apply_ops: op program too long");
    return XL_EINVAL;
  }
  ElemLaunch p;
  p.B = batch; p.C = comps; p.ny = ny; p.nx = nx; p.ibs = in_bstride; p.obs = out_bstride;
  for (int c = 0; c < 3; ++c) {
    p.in[c] = c < comps ? (const float2*)in[c] : nullptr;
    p.out[c] = c < comps ? (float2*)out[c] : nullptr;
    if (c < comps && (!p.in[c] || !p.out[c])) {
      set_error("xl_apply_ops: null plane %d", c);
      return XL_EINVAL;
    }
  }
  p.prog = *prog;
  const long long npix = (long long)ny * nx;
  int blocks = (int)((npix + 255) / 256);
  if (blocks > 152 * 8) blocks = 152 * 8;
  apply_ops_kernel<<<dim3(blocks, batch), 256, 0, (cudaStream_t)stream>>>(p);
  XL_CHECK_LAUNCH("apply_ops_kernel");
  return XL_OK;
}

extern "C" size_t xl_mse_intensity_work_bytes(int planes, long long npix) {
  if (planes < 1 || npix < 1) return 0;
  return (size_t)planes * mse_blocks(npix) * sizeof(double);
}

extern "C" int xl_mse_intensity(void* stream, int planes, long long npix, const void* a, long long a_pstride,
                                const void* b, long long b_pstride, void* work, void* out) {
  if (planes < 1 || planes > 65535 || npix < 1 || !a || !b || !work || !out) {
    set_error("xl_mse_intensity: bad arguments");
    return XL_EINVAL;
  }
  const int nb = mse_blocks(npix);
  cudaStream_t st = (cudaStream_t)stream;
  plane_sum_partial<0><<<dim3(nb, planes), MSE_THREADS, 0, st>>>((const float2*)a, a_pstride, (const float2*)b,
                                                                  b_pstride, npix, (double*)work);
  XL_CHECK_LAUNCH("plane_sum_partial");
  mse_int_finish<<<(planes + 3) / 4, 128, 0, st>>>((const double*)work, nb, planes, 1.0 / (double)npix,
                                                    (float*)out);
  XL_CHECK_LAUNCH("mse_int_finish");
  return XL_OK;
}

extern "C" int xl_mse_intensity_grad(void* stream, int planes, long long npix, const void* a, long long a_pstride,
                                     const void* b, long long b_pstride, const void* gloss, void* ga, void* gb) {
  if (planes < 1 || planes > 65535 || npix < 1 || !a || !b || !gloss || (!ga && !gb)) {
    set_error("xl_mse_intensity_grad: bad arguments");
    return XL_EINVAL;
  }
  long long nblk = (npix + 255) / 256;
  if (nblk > 152 * 8) nblk = 152 * 8;
  mse_int_grad<<<dim3((unsigned)nblk, planes), 256, 0, (cudaStream_t)stream>>>(
      (const float2*)a, a_pstride, (const float2*)b, b_pstride, npix, (const float*)gloss,
      (float)(4.0 / (double)npix), (float2*)ga, (float2*)gb);
  XL_CHECK_LAUNCH("mse_int_grad");
  return XL_OK;
}

extern "C" int xl_vmse_intensity(void* stream, int planes, long long npix, const void* const* a, long long a_pstride,
                                 const void* const* b, long long b_pstride, void* work, void* out) {
  bool ok = planes >= 1 && planes <= 65535 && npix >= 1 && a && b && work && out;
  for (int c = 0; ok && c < 3; ++c) ok = a[c] && b[c];
  if (!ok) {
    set_error("xl_vmse_intensity: bad arguments");
    return XL_EINVAL;
  }
  Vmse p = {};
  for (int c = 0; c < 3; ++c) {
    p.a[c] = (const float2*)a[c];
    p.b[c] = (const float2*)b[c];
  }
  const int nb = mse_blocks(npix);
  cudaStream_t st = (cudaStream_t)stream;
  vmse_partial<<<dim3(nb, planes, 3), MSE_THREADS, 0, st>>>(p, a_pstride, b_pstride, npix, (double*)work);
  XL_CHECK_LAUNCH("vmse_partial");
  mse_int_finish<<<(3 * planes + 3) / 4, 128, 0, st>>>((const double*)work, nb, 3 * planes, 1.0 / (double)npix,
                                                        (float*)out);
  XL_CHECK_LAUNCH("mse_int_finish");
  return XL_OK;
}

extern "C" int xl_vmse_intensity_grad(void* stream, int planes, long long npix, const void* const* a,
                                      long long a_pstride, const void* const* b, long long b_pstride,
                                      const void* gloss, void* const* ga, void* const* gb) {
  bool ok = planes >= 1 && planes <= 65535 && npix >= 1 && a && b && gloss && ga && gb;
  for (int c = 0; ok && c < 3; ++c) ok = a[c] && b[c];
  if (!ok) {
    set_error("xl_vmse_intensity_grad: bad arguments");
    return XL_EINVAL;
  }
  Vmse p = {};
  for (int c = 0; c < 3; ++c) {
    p.a[c] = (const float2*)a[c];
    p.b[c] = (const float2*)b[c];
    p.ga[c] = (float2*)ga[c];
    p.gb[c] = (float2*)gb[c];
  }
  long long nblk = (npix + 255) / 256;
  if (nblk > 152 * 8) nblk = 152 * 8;
  vmse_grad<<<dim3((unsigned)nblk, planes, 3), 256, 0, (cudaStream_t)stream>>>(p, a_pstride, b_pstride, npix,
                                                                               (const float*)gloss,
                                                                               (float)(4.0 / (double)npix));
  XL_CHECK_LAUNCH("vmse_grad");
  return XL_OK;
}

extern "C" int xl_plane_mse(void* stream, int kind, int planes, long long npix, const void* a, long long a_pstride,
                            const void* b, long long b_pstride, void* work, void* out) {
  if (kind < 0 || kind > 2) {
    set_error("xl_plane_mse: kind must be 0 (intensity), 1 (amplitude) or 2 (phase), got %d", kind);
    return XL_EINVAL;
  }
  if (kind == 0) return xl_mse_intensity(stream, planes, npix, a, a_pstride, b, b_pstride, work, out);
  if (planes < 1 || planes > 65535 || npix < 1 || !a || !b || !work || !out) {
    set_error("xl_plane_mse: bad arguments");
    return XL_EINVAL;
  }
  const int nb = mse_blocks(npix);
  cudaStream_t st = (cudaStream_t)stream;
  if (kind == 1)
    plane_sum_partial<2><<<dim3(nb, planes), MSE_THREADS, 0, st>>>((const float2*)a, a_pstride, (const float2*)b,
                                                                    b_pstride, npix, (double*)work);
  else
    plane_sum_partial<3><<<dim3(nb, planes), MSE_THREADS, 0, st>>>((const float2*)a, a_pstride, (const float2*)b,
                                                                    b_pstride, npix, (double*)work);
  XL_CHECK_LAUNCH("plane_sum_partial");
  mse_int_finish<<<(planes + 3) / 4, 128, 0, st>>>((const double*)work, nb, planes, 1.0 / (double)npix,
                                                    (float*)out);
  XL_CHECK_LAUNCH("mse_int_finish");
  return XL_OK;
}

extern "C" int xl_plane_mse_grad(void* stream, int kind, int planes, long long npix, const void* a,
                                 long long a_pstride, const void* b, long long b_pstride, const void* gloss, void* ga,
                                 void* gb) {
  if (kind < 0 || kind > 2) {
    set_error("xl_plane_mse_grad: kind must be 0 (intensity), 1 (amplitude) or 2 (phase), got %d", kind);
    return XL_EINVAL;
  }
  if (kind == 0) return xl_mse_intensity_grad(stream, planes, npix, a, a_pstride, b, b_pstride, gloss, ga, gb);
  if (planes < 1 || planes > 65535 || npix < 1 || !a || !b || !gloss || (!ga && !gb)) {
    set_error("xl_plane_mse_grad: bad arguments");
    return XL_EINVAL;
  }
  long long nblk = (npix + 255) / 256;
  if (nblk > 152 * 8) nblk = 152 * 8;
  const dim3 grid((unsigned)nblk, planes);
  const float tn = (float)(2.0 / (double)npix);
  cudaStream_t st = (cudaStream_t)stream;
  if (kind == 1)
    amp_phase_grad<2><<<grid, 256, 0, st>>>((const float2*)a, a_pstride, (const float2*)b, b_pstride, npix,
                                            (const float*)gloss, tn, (float2*)ga, (float2*)gb);
  else
    amp_phase_grad<3><<<grid, 256, 0, st>>>((const float2*)a, a_pstride, (const float2*)b, b_pstride, npix,
                                            (const float*)gloss, tn, (float2*)ga, (float2*)gb);
  XL_CHECK_LAUNCH("amp_phase_grad");
  return XL_OK;
}

extern "C" int xl_re_inner(void* stream, int planes, long long npix, const void* a, long long a_pstride,
                           const void* b, long long b_pstride, void* work, void* out) {
  if (planes < 1 || planes > 65535 || npix < 1 || !a || !b || !work || !out) {
    set_error("xl_re_inner: bad arguments");
    return XL_EINVAL;
  }
  const int nb = mse_blocks(npix);
  cudaStream_t st = (cudaStream_t)stream;
  plane_sum_partial<1><<<dim3(nb, planes), MSE_THREADS, 0, st>>>((const float2*)a, a_pstride, (const float2*)b,
                                                                  b_pstride, npix, (double*)work);
  XL_CHECK_LAUNCH("plane_sum_partial");
  mse_int_finish<<<(planes + 3) / 4, 128, 0, st>>>((const double*)work, nb, planes, 1.0, (float*)out);
  XL_CHECK_LAUNCH("mse_int_finish");
  return XL_OK;
}

extern "C" int xl_vrs_dz_ez(void* stream, int batch, int ny, int nx, const void* ex, const void* ey,
                            long long e_bstride, const void* gez, long long g_bstride, const double* x,
                            const double* y, const double* z, void* work, void* out) {
  if (batch < 1 || batch > 65535 || ny < 1 || nx < 1 || (long long)ny * nx > 0x7fffffffLL || !ex || !ey || !gez ||
      !x || !y || !z || !work || !out) {
    set_error("xl_vrs_dz_ez: bad arguments");
    return XL_EINVAL;
  }
  const long long npix = (long long)ny * nx;
  const int nb = mse_blocks(npix);
  cudaStream_t st = (cudaStream_t)stream;
  vrs_dz_ez_partial<<<dim3(nb, batch), MSE_THREADS, 0, st>>>((const float2*)ex, (const float2*)ey, e_bstride,
                                                             (const float2*)gez, g_bstride, ny, nx, x, y, z,
                                                             (double*)work);
  XL_CHECK_LAUNCH("vrs_dz_ez_partial");
  mse_int_finish<<<(batch + 3) / 4, 128, 0, st>>>((const double*)work, nb, batch, 1.0, (float*)out);
  XL_CHECK_LAUNCH("mse_int_finish");
  return XL_OK;
}

extern "C" int xl_rs_z_gradient(void* stream, int batch, int ny, int nx, int comps, const void* const* g,
                                const void* const* d, long long bstride, const void* ex, const void* ey,
                                long long e_bstride, const void* gez, const double* x, const double* y,
                                const double* z, void* work, void* out) {
  if (batch < 1 || batch > 65535 || ny < 1 || nx < 1 || (long long)ny * nx > 0x7fffffffLL || comps < 1 ||
      comps > 3 || !g || !d || !work || !out || (ex && (!ey || !gez || !x || !y || !z))) {
    set_error("xl_rs_z_gradient: bad arguments");
    return XL_EINVAL;
  }
  ZGradArgs p;
  for (int c = 0; c < 3; ++c) {
    p.g[c] = c < comps ? (const float2*)g[c] : nullptr;
    p.d[c] = c < comps ? (const float2*)d[c] : nullptr;
    if (c < comps && (!p.g[c] || !p.d[c])) {
      set_error("xl_rs_z_gradient: null plane %d", c);
      return XL_EINVAL;
    }
  }
  p.bs = bstride;
  p.ncomp = comps;
  p.ex = (const float2*)ex;
  p.ey = (const float2*)ey;
  p.ebs = e_bstride;
  p.gez = (const float2*)gez;
  p.x = x;
  p.y = y;
  p.z = z;
  p.ny = ny;
  p.nx = nx;
  const int nb = mse_blocks((long long)ny * nx);
  cudaStream_t st = (cudaStream_t)stream;
  rs_zgrad_partial<<<dim3(nb, batch), MSE_THREADS, 0, st>>>(p, (double*)work);
  XL_CHECK_LAUNCH("rs_zgrad_partial");
  mse_int_finish<<<(batch + 3) / 4, 128, 0, st>>>((const double*)work, nb, batch, 1.0, (float*)out);
  XL_CHECK_LAUNCH("mse_int_finish");
  return XL_OK;
}
