// In-place block FFT engine for lines of P = 256 R points (R even, 4..16),
// used as a pair: a forward transform that leaves its output in the order its
// threads hold it, a pointwise product in that order, and the inverse
// transform back to natural order.
//
// A line is R blocks of 256 slots in shared memory.  With n = j + 256 n1 and
// k = k1 + R (k2 + 16 k3), j = j0 + 16 j1:
//
//   phase A   thread of index j: DFT_R over n1, twiddle w_P^(j k1), store to
//             slot (k1, j);
//   phase B   thread (k1, j0): DFT16 over j1, twiddle w_256^(j0 k2), store to
//             slot (k1, k2, j0);
//   phase C   thread (k1, k2): DFT16 over j0 -> k3.
//
// The inverse runs C, B, A backwards (conjugate twiddles before each DFT).
//
// Why this form: every phase stores to the slots it loaded from, so a store
// never races with another thread's load and one barrier per exchange is
// enough (a Stockham exchange needs two, with nothing but loads between them);
// and the exchange between B and C stays among the 16 threads of one k1, half
// a warp, so it needs no CTA barrier at all.  A forward and inverse pair has
// two CTA barriers (A -> B, B -> A) where the Stockham engine has eight, and
// between them the warps drift: one's loads and exchanges run under another's
// arithmetic.
//
// Slots are padded by two every sixteen: the three access patterns (runs of j,
// stride 16 + 2, and 16-byte pieces at stride 18) are then free of bank
// conflicts.
//
// Every function is host+device so that a CPU harness can run the threads of
// a line one after the other.
#pragma once

#include "fft_core.cuh"

#if !defined(__CUDACC__)
struct float4 { float x, y, z, w; };
inline float4 make_float4(float a, float b, float c, float d) { float4 r; r.x = a; r.y = b; r.z = c; r.w = d; return r; }
#endif

namespace xl {

// cos and sin of 2 pi num / den at compile time (Taylor series in float64
// after reduction to the first octant), for the twiddles inside DFT_R.
constexpr double ct_sin_small(double x) {
  double t = x, s = x;
  for (int i = 1; i < 16; ++i) {
    t *= -x * x / ((2 * i) * (2 * i + 1));
    s += t;
  }
  return s;
}
constexpr double ct_cos_small(double x) {
  double t = 1.0, s = 1.0;
  for (int i = 1; i < 16; ++i) {
    t *= -x * x / ((2 * i - 1) * (2 * i));
    s += t;
  }
  return s;
}
constexpr double CT_PI = 3.14159265358979323846;
constexpr double ct_cos(int num, int den) {
  num %= den;
  if (8 * num > 4 * den) num = den - num;                        // cos(2 pi - x) = cos x
  if (8 * num > 2 * den) return -ct_cos(den - 2 * num, 2 * den); // cos x = -cos(pi - x)
  if (8 * num > den) return ct_sin_small(2.0 * CT_PI * (den - 4 * num) / (4.0 * den));
  return ct_cos_small(2.0 * CT_PI * num / den);
}
constexpr double ct_sin(int num, int den) { return ct_cos(4 * num + 3 * den, 4 * den); }   // sin x = cos(x - pi/2)

// a * e^(DIR 2 pi i NUM / DEN)
template <int DIR, int NUM, int DEN> XL_HD float2 cmul_root(float2 a) {
  constexpr int n = NUM % DEN;
  if constexpr (n == 0) return a;
  else if constexpr (4 * n == DEN) return cmul_dir_i<DIR>(a);
  else if constexpr (2 * n == DEN) return make_float2(-a.x, -a.y);
  else if constexpr (4 * n == 3 * DEN) return cmul_dir_i<-DIR>(a);
  else {
    constexpr float c = (float)ct_cos(n, DEN), s = (float)(DIR * ct_sin(n, DEN));
    return cmul(a, make_float2(c, s));
  }
}

// ---- DFT of R points in registers, natural order in and out ----

// Odd prime lengths: real and imaginary parts of the pairs x[n], x[R-n].
template <int R, int DIR> XL_HD void dft_odd(float2 (&a)[R]) {
  constexpr int H = (R - 1) / 2;
  float2 s[H], d[H];
#pragma unroll
  for (int n = 0; n < H; ++n) {
    s[n] = cadd(a[n + 1], a[R - 1 - n]);
    d[n] = csub(a[n + 1], a[R - 1 - n]);
  }
  float2 sum = a[0];
#pragma unroll
  for (int n = 0; n < H; ++n) sum = cadd(sum, s[n]);
  const float2 x0 = a[0];
  a[0] = sum;
  constexpr auto cs = [](int i) constexpr { return (float)ct_cos(i, R); };
  constexpr auto sn = [](int i) constexpr { return (float)(DIR * ct_sin(i, R)); };
  // cos and sin of 2 pi i / R, indexed by i = n k mod R
  constexpr float C[7] = {cs(0), cs(1), cs(2 % R), cs(3 % R), cs(4 % R), cs(5 % R), cs(6 % R)};
  constexpr float S[7] = {sn(0), sn(1), sn(2 % R), sn(3 % R), sn(4 % R), sn(5 % R), sn(6 % R)};
  static_assert(R <= 7, "odd lengths 3, 5 and 7");
#pragma unroll
  for (int k = 1; k <= H; ++k) {
    float2 e = x0, o = make_float2(0.f, 0.f);
#pragma unroll
    for (int n = 1; n <= H; ++n) {
      const int i = (n * k) % R;
      e = make_float2(e.x + C[i] * s[n - 1].x, e.y + C[i] * s[n - 1].y);
      o = n == 1 ? make_float2(S[i] * d[0].x, S[i] * d[0].y)
                 : make_float2(o.x + S[i] * d[n - 1].x, o.y + S[i] * d[n - 1].y);
    }
    a[k] = make_float2(e.x - o.y, e.y + o.x);        // e + i o
    a[R - k] = make_float2(e.x + o.y, e.y - o.x);    // e - i o
  }
}

template <int R, int DIR> XL_HD void dft_n(float2 (&a)[R]);

// X[k] = E[k] + w^k O[k], X[k + Q] = E[k] - w^k O[k]
template <int R, int DIR, int K = 0> XL_HD void dft_merge(float2 (&a)[R], const float2 (&e)[R / 2], const float2 (&o)[R / 2]) {
  if constexpr (K < R / 2) {
    const float2 t = cmul_root<DIR, K, R>(o[K]);
    a[K] = cadd(e[K], t);
    a[K + R / 2] = csub(e[K], t);
    dft_merge<R, DIR, K + 1>(a, e, o);
  }
}

template <int R, int DIR> XL_HD void dft_n(float2 (&a)[R]) {
  if constexpr (R == 1) return;
  else if constexpr (R == 2) dft2<DIR>(a);
  else if constexpr (R == 4) dft4<DIR>(a);
  else if constexpr (R == 8) dft8<DIR>(a);
  else if constexpr (R == 16) dft16<DIR>(a);
  else if constexpr (R % 2 == 1) dft_odd<R, DIR>(a);
  else {
    float2 e[R / 2], o[R / 2];
#pragma unroll
    for (int n = 0; n < R / 2; ++n) {
      e[n] = a[2 * n];
      o[n] = a[2 * n + 1];
    }
    dft_n<R / 2, DIR>(e);
    dft_n<R / 2, DIR>(o);
    dft_merge<R, DIR>(a, e, o);
  }
}

// The same when a[R/2..R-1] are zero: X[2q] = DFT(a), X[2q+1] = DFT(w^n a[n]).
template <int R, int DIR, int N = 0> XL_HD void dft_half_twiddle(const float2 (&a)[R], float2 (&o)[R / 2]) {
  if constexpr (N < R / 2) {
    o[N] = cmul_root<DIR, N, R>(a[N]);
    dft_half_twiddle<R, DIR, N + 1>(a, o);
  }
}
template <int R, int DIR> XL_HD void dft_n_half(float2 (&a)[R]) {
  if constexpr (R == 16) dft16_half<DIR>(a);
  else {
    float2 e[R / 2], o[R / 2];
#pragma unroll
    for (int n = 0; n < R / 2; ++n) e[n] = a[n];
    dft_half_twiddle<R, DIR>(a, o);
    dft_n<R / 2, DIR>(e);
    dft_n<R / 2, DIR>(o);
#pragma unroll
    for (int q = 0; q < R / 2; ++q) {
      a[2 * q] = e[q];
      a[2 * q + 1] = o[q];
    }
  }
}

// ---- the phases ----

template <int R> struct BlkFft {
  static_assert(R >= 4 && R <= 16 && R % 2 == 0, "P = 256 R, R even");
  static constexpr int P = 256 * R;
  static constexpr int RP = R <= 4 ? 4 : (R <= 8 ? 8 : 16);   // R rounded up to a power of two
  static constexpr int T = 16 * RP;          // threads of a line in phase A
  static constexpr int IPT = 16 / RP;        // values of j a thread of phase A takes
  static constexpr int TB = 16 * R;          // threads of a line in phases B and C
  static constexpr int BLK = 288;            // slots of one block of 256
  static constexpr int LINE = R * BLK;       // slots of a line
  static constexpr int NTA = (R - 1) * 256;  // phase A twiddles
  static constexpr int NTB = 15 * 16;        // phase B twiddles
  static constexpr int NTW = NTA + NTB;
};

// Twiddle tables: phase A, w_P^(k1 j) at [(k1 - 1) 256 + j]; phase B,
// w_256^(k2 x) at [NTA + (k2 - 1) 16 + x].  Read as 8-byte words: lanes that
// share a twiddle then share the shared-memory wavefront, which 16-byte reads
// of two twiddles did not (3.3 wavefronts a read against 1).
template <int R> inline void blk_twiddles(float2* t) {
  using F = BlkFft<R>;
  auto root = [](long long num, long long den) {
    const double a = -2.0 * 3.14159265358979323846 * (double)(num % den) / (double)den;
    return make_float2((float)::cos(a), (float)::sin(a));
  };
  for (int k = 1; k < R; ++k)
    for (int j = 0; j < 256; ++j) t[(k - 1) * 256 + j] = root((long long)k * j, F::P);
  for (int k = 1; k < 16; ++k)
    for (int x = 0; x < 16; ++x) t[F::NTA + (k - 1) * 16 + x] = root(k * x, 256);
}

// slot of j within a block
XL_HD int blk_slot(int j) { return (j >> 4) * 18 + (j & 15); }

// Phase A forward: v[i R + n1] = x[t + i T + 256 n1] to the slots of `line`.
// ZU: the upper half of the line (n1 >= R/2) is zero and not read from v.
// tw(i, q, w) gives the twiddles w_P^(k1 j) of k1 = 4 q .. 4 q + 3 (k1 in
// 1..R-1) for this thread's i-th j = t + i T.
template <int R, int DIR, bool ZU, class TW>
XL_HD void blk_a_fwd(const float2 (&v)[16], int t, float2* line, const TW& tw) {
  using F = BlkFft<R>;
  float2* d = line + blk_slot(t);
#pragma unroll
  for (int i = 0; i < F::IPT; ++i) {
    float2 a[R];
#pragma unroll
    for (int n = 0; n < R; ++n) a[n] = (ZU && n >= R / 2) ? make_float2(0.f, 0.f) : v[i * R + n];
    if constexpr (ZU) dft_n_half<R, DIR>(a);
    else dft_n<R, DIR>(a);
#pragma unroll
    for (int q = 0; q < (R + 3) / 4; ++q) {
      float2 w[4];
      tw(i, q, w);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int k = 4 * q + n;
        if (k >= R) continue;
        if (k > 0) a[k] = DIR < 0 ? cmul(a[k], w[n]) : cmulc(a[k], w[n]);
        d[k * F::BLK + i * (F::T / 16) * 18] = a[k];
      }
    }
  }
}

// Phase A inverse: the slots of `line` back to v[i R + n1] = x[t + i T + 256 n1].
// DIR is the direction of this transform (+1 when the forward one was -1).
template <int R, int DIR, class TW>
XL_HD void blk_a_inv(float2 (&v)[16], int t, const float2* line, const TW& tw) {
  using F = BlkFft<R>;
  const float2* s = line + blk_slot(t);
#pragma unroll
  for (int i = 0; i < F::IPT; ++i) {
    float2 a[R];
#pragma unroll
    for (int q = 0; q < (R + 3) / 4; ++q) {
      float2 w[4];
      tw(i, q, w);
#pragma unroll
      for (int n = 0; n < 4; ++n) {
        const int k = 4 * q + n;
        if (k >= R) continue;
        a[k] = s[k * F::BLK + i * (F::T / 16) * 18];
        if (k > 0) a[k] = DIR < 0 ? cmul(a[k], w[n]) : cmulc(a[k], w[n]);
      }
    }
    dft_n<R, DIR>(a);
#pragma unroll
    for (int n = 0; n < R; ++n) v[i * R + n] = a[n];
  }
}

// Phase B forward: thread l = j0 of block `blk` (the line's slots + k1 BLK).
template <int DIR>
XL_HD void blk_b_fwd(float2 (&v)[16], int l, float2* blk, const float2* twb) {
  float2* s = blk + l;
#pragma unroll
  for (int m = 0; m < 16; ++m) v[m] = s[18 * m];
  dft16<DIR>(v);
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    if (k > 0) {
      const float2 w = twb[(k - 1) * 16 + l];
      v[k] = DIR < 0 ? cmul(v[k], w) : cmulc(v[k], w);
    }
    s[18 * k] = v[k];
  }
}

// Phase B inverse.
template <int DIR>
XL_HD void blk_b_inv(float2 (&v)[16], int l, float2* blk, const float2* twb) {
  float2* s = blk + l;
#pragma unroll
  for (int k = 0; k < 16; ++k) {
    v[k] = s[18 * k];
    if (k > 0) {
      const float2 w = twb[(k - 1) * 16 + l];
      v[k] = DIR < 0 ? cmul(v[k], w) : cmulc(v[k], w);
    }
  }
  dft16<DIR>(v);
#pragma unroll
  for (int m = 0; m < 16; ++m) s[18 * m] = v[m];
}

// Phase C: thread l = k2 of block `blk`; its sixteen slots are contiguous and
// move as 16-byte pairs.
template <int DIR> XL_HD void blk_c_fwd(float2 (&v)[16], int l, const float2* blk) {
  const float4* s = (const float4*)(blk + 18 * l);
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const float4 x = s[q];
    v[2 * q] = make_float2(x.x, x.y);
    v[2 * q + 1] = make_float2(x.z, x.w);
  }
  dft16<DIR>(v);
}
template <int DIR> XL_HD void blk_c_inv(float2 (&v)[16], int l, float2* blk) {
  dft16<DIR>(v);
  float4* s = (float4*)(blk + 18 * l);
#pragma unroll
  for (int q = 0; q < 8; ++q) s[q] = make_float4(v[2 * q].x, v[2 * q].y, v[2 * q + 1].x, v[2 * q + 1].y);
}

// Frequency of register m (= k3) of phase C's thread (k1, k2).
template <int R> XL_HD int blk_freq(int k1, int k2, int m) { return k1 + R * (k2 + 16 * m); }

}  // namespace xl
