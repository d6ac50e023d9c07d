// RS / VRS kernels for transforms of P = 512 R points (R = 10, 12, 14, 16),
// sides 2049 to 4096, as two transforms of M = P / 2 points on the block FFT
// engine: the even frequencies are the M-point transform of x[n], the odd ones
// that of x[n] w_P^n (the field's side is at most M, so nothing wraps), and the
// inverse at n < M is the even half's inverse plus w_P^-n times the odd half's.
//
// Positions of an axis: the even half's M in the engine's order (rs_blk.cuh),
// then the odd half's.  The halves go through the same line of shared memory one
// after the other, so a CTA holds what one of M points does; what has to last
// over the other half (a column's input, then its first half's output) stays in
// the thread's own Tensor Memory cells.
//
// 8192-point Stockham transforms, this form: 2 x 4096^2 scalar RS 1809 us, 1088;
// one 4096^2 VRS 2513, 1542.  Shorter lengths: 4 x 2500^2 2979, 930 (5120 points);
// 4 x 300 x 4096 1797, 222 (1024 points in y).
#pragma once

#include "rs_blk.cuh"

namespace xl {

// w_P^n = exp(-2 pi i n / (512 R)), n < 256 R, one length after the other.
__host__ __device__ constexpr int half_tw_off(int r) {
  int o = 0;
  for (int q = 10; q < r; q += 2) o += 256 * q;
  return o;
}
static __device__ float2 g_half_tw[half_tw_off(18)];

template <int R> __device__ __forceinline__ const float2* half_tw() { return g_half_tw + half_tw_off(R); }

static cudaError_t half_upload_twiddles(const float2*) {
  std::vector<float2> t(half_tw_off(18));
  for (int r = 10; r <= 16; r += 2)
    for (int n = 0; n < 256 * r; ++n) {
      const double a = -2.0 * 3.14159265358979323846 * n / (512.0 * r);
      t[half_tw_off(r) + n] = make_float2((float)::cos(a), (float)::sin(a));
    }
  return cudaMemcpyToSymbol(g_half_tw, t.data(), t.size() * sizeof(float2));
}
static const bool half_tw_registered = register_device_tables(&half_upload_twiddles, nullptr);

// Column pass (see rs_cols_b).  A thread's Tensor Memory cells hold the phase A
// twiddles and, per component, its input until the odd half is formed and the
// even half's output from then on; w_P^n is in shared memory, where the lanes of
// a row of four columns share a word.  Spectrum values come from L2 for every
// component.
template <int R> struct HalfCol {
  using F = BlkFft<R>;
  using K = RsColB<R>;
  static_assert(F::IPT == 1 && K::TM, "one j a thread, CTAs alone on an SM");
  static constexpr int P = 2 * F::P;
  static constexpr size_t SMEM = ((size_t)F::NTB + F::P + (size_t)K::CW * K::LINE) * 8;
};

template <int R>
__global__ void __launch_bounds__(RsColB<R>::THREADS, 1) rs_cols_h(const __grid_constant__ RsLaunch p) {
  using F = BlkFft<R>;
  using K = RsColB<R>;
  constexpr int P = HalfCol<R>::P;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned s_tmem;
  float2* twb = (float2*)smraw;   // NTB
  float2* tw2 = twb + F::NTB;     // M
  float2* xch = tw2 + F::P;
  const ColMap<R> m;
  for (int i = threadIdx.x; i < F::NTB; i += K::THREADS) twb[i] = blk_tw<R>()[F::NTA + i];
  for (int i = threadIdx.x; i < F::P; i += K::THREADS) tw2[i] = half_tw<R>()[i];
  const TmemTw<R> twa{tmem_twiddles<R, K::THREADS, 64>(&s_tmem, GlobalTw<R>{blk_tw<R>() + m.jt})};
  const unsigned hold = twa.cell + 32u;
  __syncthreads();
  float2* line = xch + m.wc * K::LINE;
  float2* blk = xch + m.bc * K::LINE + m.k1 * F::BLK;
  const bool active = m.warp < K::WARPS_B;
  const int ny = p.ny, lw = p.lw;
  const int units = p.B * (p.px / K::CW);
#pragma unroll 1
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const int b = u % p.B, g = u / p.B;
    const long long col = (long long)g * K::CW + m.wc;
    const float2* sbase = p.specs ? p.specs[b] : p.spec + (long long)(p.sidx ? p.sidx[b] : 0) * p.sstride;
    const float2* spec = sbase + (long long)g * (K::CW * P) + m.warp * 512 + m.lane;
#pragma unroll 1
    for (int c = 0; c < p.cout; ++c) {
      float2* tile = p.work + ((long long)b * p.cout + c) * ny * p.px + (((col >> lw) * ny) << lw) +
                     (col & ((1 << lw) - 1));
      float2 v[16];
#pragma unroll
      for (int n = 0; n < 16; ++n) {
        const int r = m.jt + 256 * n;
        v[n] = n < R && r < ny ? tile[(long long)r << lw] : make_float2(0.f, 0.f);
      }
#pragma unroll
      for (int q = 0; q < (R + 3) / 4; ++q)
        tmem_st4(hold + 8u * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3], q == 0);
      tmem_wait_st(false);
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        blk_a_fwd<R, -1, false>(v, m.jt, line, twa);
        __syncthreads();
        if (active) {
          blk_b_fwd<-1>(v, m.l, blk, twb);
          __syncwarp();
          blk_c_fwd<-1>(v, m.l, blk);
          const float2* sp = spec + h * (K::CW * F::P);
          asm volatile("" : "+l"(sp));   // the loads stay here: ahead of the transform they would hold 32 registers
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float2 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = __ldg(sp + (4 * q + i) * 32);
#pragma unroll
            for (int i = 0; i < 4; ++i) v[4 * q + i] = p.adjoint ? cmulc(v[4 * q + i], w[i]) : cmul(v[4 * q + i], w[i]);
          }
          blk_c_inv<1>(v, m.l, blk);
          __syncwarp();
          blk_b_inv<1>(v, m.l, blk, twb);
        }
        __syncthreads();
        blk_a_inv<R, 1>(v, m.jt, line, twa);
#pragma unroll
        for (int q = 0; q < (R + 3) / 4; ++q) {
          float2 w[4];
          tmem_ld4(hold + 8u * q, w, false);
          if (h == 0) tmem_st4(hold + 8u * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3], false);
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            if (4 * q + i >= R) continue;
            const float2 t = tw2[m.jt + 256 * (4 * q + i)];
            v[4 * q + i] = h == 0 ? cmul(w[i], t) : cadd(w[i], cmulc(v[4 * q + i], t));
          }
        }
        if (h == 0) tmem_wait_st(false);
      }
#pragma unroll
      for (int n = 0; n < R; ++n) {
        const int r = m.jt + 256 * n;
        if (r < ny) tile[(long long)r << lw] = v[n];
      }
    }
  }
  tmem_release<K::THREADS, 64>(s_tmem);
}

// Transfer spectrum, column transforms (see rs_hhat_cols_b): [group][half][warp]
// [register][lane].  The wrapped response fills all P points, so the even half
// transforms h[n] + h[n + M] and the odd one (h[n] - h[n + M]) w_P^n.
template <int R>
__global__ void __launch_bounds__(RsColB<R>::THREADS, 1)
    rs_hhat_cols_h(const float2* __restrict__ in, int px, float scale, float2* __restrict__ out) {
  using F = BlkFft<R>;
  using K = RsColB<R>;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* twb = (float2*)smraw;
  float2* xch = twb + F::NTB;
  const ColMap<R> m;
  for (int i = threadIdx.x; i < F::NTB; i += K::THREADS) twb[i] = blk_tw<R>()[F::NTA + i];
  float2* blk = xch + m.bc * K::LINE + m.k1 * F::BLK;
  const float2* src = in + (long long)blockIdx.x * K::CW + m.wc;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    float2 v[16];
    const float2* lo = src + (long long)m.jt * px;
    long long half = (long long)F::P * px, step = 256LL * px;
    asm volatile("" : "+l"(lo), "+l"(half), "+l"(step));   // addresses formed here, not 32 of them kept over the halves
#pragma unroll
    for (int n = 0; n < R; ++n) {
      const float2 a = lo[n * step], d = lo[n * step + half];
      v[n] = h == 0 ? cadd(a, d) : cmul(csub(a, d), __ldg(half_tw<R>() + m.jt + 256 * n));
      if (n % 4 == 3) asm volatile("" ::: "memory");
    }
    __syncthreads();   // twb, and the even half's slots
    blk_a_fwd<R, -1, false>(v, m.jt, xch + m.wc * K::LINE, GlobalTw<R>{blk_tw<R>() + m.jt});
    __syncthreads();
    if (m.warp < K::WARPS_B) {
      blk_b_fwd<-1>(v, m.l, blk, twb);
      __syncwarp();
      blk_c_fwd<-1>(v, m.l, blk);
      float2* dst = out + (long long)blockIdx.x * (K::CW * 2 * F::P) + h * (K::CW * F::P) + m.warp * 512 + m.lane;
#pragma unroll
      for (int q = 0; q < 16; ++q) dst[32 * q] = cscale(v[q], scale);
    }
  }
}

// ---- row passes ----
// CTAs of 768 threads, alone on an SM, in three groups of 256: the three
// components of a row, or (scalar) three rows that never meet.
template <int R> struct HalfRow {
  using F = BlkFft<R>;
  static_assert(F::IPT == 1, "one j a thread");
  static constexpr int THREADS = 3 * F::T;
  static constexpr size_t LINES = ((size_t)F::NTB + 3 * F::LINE) * 8;   // bytes of tables and lines
};

// Forward.  MODE 1: scalar; 2: VRS (Ex, Ey in, Ez derived); 3: VRS adjoint.  A
// row's elements after the program stay in shared memory for both halves; the
// phase A twiddles and w_P^n of the thread's elements are in Tensor Memory.
//
// A row's loads are not overlapped with its transform within a group, and a row
// staged ahead by bulk copies does not fit beside three lines and rows, so a
// group's next rows are prefetched into L2 while it transforms (where bulk
// prefetches may read them: 16-byte aligned planes and rows).  2 x 4096^2 scalar
// behind an SLM: 320 us without, 264 with (3.6 TB/s; Stockham 501); one 4096^2 VRS
// 359, 313.
template <int R, int MODE, class FK = FixedKinds<>>
__global__ void __launch_bounds__(HalfRow<R>::THREADS, 1) rs_rows_fwd_h(const __grid_constant__ RsLaunch p, const __grid_constant__ RowStage st) {
  using F = BlkFft<R>;
  constexpr int M = F::P, THREADS = HalfRow<R>::THREADS;
  constexpr bool ONE = MODE == 1;
  constexpr int COUT = ONE ? 1 : 3, NP = ONE ? 4 : 2;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned s_tmem;
  const int nx = p.nx, ny = p.ny, tid = threadIdx.x, cg = tid / F::T, t = tid % F::T;
  float2* twb = (float2*)smraw;
  float2* line = twb + F::NTB + cg * F::LINE;
  float2* rows = twb + F::NTB + 3 * F::LINE;   // 3 x nx
  float* xf = (float*)(rows + 3 * nx);         // nx (VRS: x as float32)
  float2* row = rows + cg * nx;
  for (int i = tid; i < F::NTB; i += THREADS) twb[i] = blk_tw<R>()[F::NTA + i];
  if constexpr (MODE == 2)
    for (int i = tid; i < nx; i += THREADS) xf[i] = (float)p.x[i];
  const TmemTw<R> twa{tmem_twiddles<R, THREADS, 64>(&s_tmem, GlobalTw<R>{blk_tw<R>() + t})};
  const unsigned cell2 = twa.cell + 32u;
#pragma unroll
  for (int q = 0; q < (R + 3) / 4; ++q) {
    float2 w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = 4 * q + i < R ? half_tw<R>()[t + 256 * (4 * q + i)] : make_float2(0.f, 0.f);
    tmem_st4(cell2 + 8u * q, w[0], w[1], w[2], w[3], q == 0);
  }
  tmem_wait_st(false);
  __syncthreads();
  const bool active = t < F::TB;
  float2* blk = line + (t >> 4) * F::BLK;
  auto sync = [&]() { GroupSync{1 + cg, F::T}(); };
  const int total = p.B * ny;
  const int step = ONE ? 3 * gridDim.x : gridDim.x;
#pragma unroll 1
  for (int u = ONE ? 3 * blockIdx.x + cg : blockIdx.x; u < total; u += step) {
    const int b = u % p.B, r = u / p.B;
    const int lane0 = ONE ? t : tid, lanes = ONE ? F::T : THREADS;
    float z2 = 0.f, Y = 0.f;
    if constexpr (MODE == 2) {
      const float zb = (float)p.z[b];
      Y = (float)p.y[r];
      z2 = Y * Y + zb * zb;
    }
#pragma unroll 1
    for (int i0 = lane0; i0 < nx; i0 += lanes * NP) {
      float2 e[NP][3];
      PixelCtx px[NP];
      GlobalParams pr[NP];
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        const int n = min(i0 + q * lanes, nx - 1);
        const long long pix = (long long)r * nx + n;
#pragma unroll
        for (int i = 0; i < 3; ++i)
          e[q][i] = i < MODE ? p.in[i][(long long)b * p.ibs + pix] : make_float2(0.f, 0.f);
        px[q] = PixelCtx{r, n, pix, b};
      }
      if constexpr (FK::n > 0) apply_prog_fixed<FK>(p.pre, e, px, pr);
      else if (p.pre.nops) apply_prog_vec<NP>(p.pre, e, px, pr);
#pragma unroll
      for (int q = 0; q < NP; ++q) {
        const int n = i0 + q * lanes;
        if (n >= nx) continue;
        if constexpr (ONE) {
          row[n] = e[q][0];
        } else {
          if constexpr (MODE == 2) {   // vectorized_optics.py:258-261, Ez = Ex X/r + Ey Y/r
            const float X = xf[n], inv = rsqrtf(X * X + z2);
            e[q][2] = cadd(cscale(e[q][0], X * inv), cscale(e[q][1], Y * inv));
          }
#pragma unroll
          for (int c = 0; c < 3; ++c) rows[c * nx + n] = e[q][c];
        }
      }
    }
    if (lane0 == 0 && u + step < total) prefetch_rows(st, (u + step) % p.B, (u + step) / p.B, 1);
    if constexpr (ONE) sync();
    else __syncthreads();
    const int plane = ONE ? b : b * COUT + cg;
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      float2 v[16];
#pragma unroll
      for (int q = 0; q < (R + 3) / 4; ++q) {
        float2 w[4];
        if (h) tmem_ld4(cell2 + 8u * q, w);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int n = t + 256 * (4 * q + i);
          if (4 * q + i >= R) continue;
          v[4 * q + i] = n < nx ? row[n] : make_float2(0.f, 0.f);
          if (h) v[4 * q + i] = cmul(v[4 * q + i], w[i]);
        }
      }
      blk_a_fwd<R, -1, false>(v, t, line, twa);
      sync();
      if (active) {
        blk_b_fwd<-1>(v, t & 15, blk, twb);
        __syncwarp();
        blk_c_fwd<-1>(v, t & 15, blk);
        float2* o = p.work + (long long)plane * ny * (2 * M) + row_pos((t >> 5) + h * (M / 512), t & 31, r, ny, p.lw);
        long long stp = 32LL * ny;
        asm volatile("" : "+l"(o), "+l"(stp));   // one base, not sixteen addresses live across the loop
#pragma unroll
        for (int q = 0; q < 16; ++q) o[q * stp] = v[q];
      }
      sync();   // the next phase A stores to the slots phase C loads here
    }
    if constexpr (!ONE) __syncthreads();   // every group is done with the rows
  }
  tmem_release<THREADS, 64>(s_tmem);
}

// Inverse (see rs_rows_inv_b): the even half's output waits in Tensor Memory for
// the odd one's; the loads of the next half are in flight over a half.
// EPI: an epilogue program, or the adjoint's fold, over all components of a row,
// which the groups leave in their lines.
template <int R, int COUT, bool EPI>
__global__ void __launch_bounds__(HalfRow<R>::THREADS, 1) rs_rows_inv_h(const __grid_constant__ RsLaunch p) {
  using F = BlkFft<R>;
  constexpr int M = F::P, THREADS = HalfRow<R>::THREADS;
  constexpr bool ONE = COUT == 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned s_tmem;
  const int nx = p.nx, ny = p.ny, tid = threadIdx.x, cg = tid / F::T, t = tid % F::T;
  float2* twb = (float2*)smraw;
  float2* lines = twb + F::NTB;
  float2* line = lines + cg * F::LINE;
  for (int i = tid; i < F::NTB; i += THREADS) twb[i] = blk_tw<R>()[F::NTA + i];
  const TmemTw<R> twa{tmem_twiddles<R, THREADS, 64>(&s_tmem, GlobalTw<R>{blk_tw<R>() + t})};
  const unsigned hold = twa.cell + 32u;
  const float2* tw2 = half_tw<R>() + t;
  __syncthreads();
  const bool active = t < F::TB;
  float2* blk = line + (t >> 4) * F::BLK;
  auto sync = [&]() { GroupSync{1 + cg, F::T}(); };
  const int total = p.B * ny;
  const int step = ONE ? 3 * gridDim.x : gridDim.x;
  auto load = [&](int u, int h, float2 (&d)[16]) {
    const int b = u % p.B, r = u / p.B;
    const int plane = ONE ? b : b * COUT + cg;
    const float2* q = p.work + (long long)plane * ny * (2 * M) + row_pos((t >> 5) + h * (M / 512), t & 31, r, ny, p.lw);
    long long stp = 32LL * ny;
    asm volatile("" : "+l"(q), "+l"(stp));
#pragma unroll
    for (int m = 0; m < 16; ++m) d[m] = q[m * stp];
  };
  float2 nxt[16];
  const int first = ONE ? 3 * blockIdx.x + cg : blockIdx.x;
  if (active && first < total) load(first, 0, nxt);
#pragma unroll 1
  for (int u = first; u < total; u += step) {
    const int b = u % p.B, r = u / p.B;
    float2 v[16];
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      if (active) {
#pragma unroll
        for (int m = 0; m < 16; ++m) v[m] = nxt[m];
        const int un = h ? u + step : u;
        if (un < total) load(un, h ^ 1, nxt);
        blk_c_inv<1>(v, t & 15, blk);
        __syncwarp();
        blk_b_inv<1>(v, t & 15, blk, twb);
      }
      sync();
      blk_a_inv<R, 1>(v, t, line, twa);
      if (h == 0) {
#pragma unroll
        for (int q = 0; q < (R + 3) / 4; ++q)
          tmem_st4(hold + 8u * q, v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3], false);
        tmem_wait_st(false);
        sync();   // the odd half's phase C stores to slots that phase A loads here
      }
    }
#pragma unroll
    for (int q = 0; q < (R + 3) / 4; ++q) {
      float2 w[4];
      tmem_ld4(hold + 8u * q, w, false);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (4 * q + i < R) v[4 * q + i] = cadd(w[i], cmulc(v[4 * q + i], __ldg(tw2 + 256 * (4 * q + i))));
    }
    if constexpr (!EPI) {
      float2* o = p.out[ONE ? 0 : cg] + (long long)b * p.obs + (long long)r * nx;
#pragma unroll
      for (int n1 = 0; n1 < R; ++n1) {
        const int n = t + 256 * n1;
        if (n < nx) o[n] = v[n1];
      }
      sync();
    } else {
      float2* d = line + blk_slot(t);
#pragma unroll
      for (int n1 = 0; n1 < R; ++n1) d[n1 * F::BLK] = v[n1];
      if constexpr (ONE) sync();
      else __syncthreads();
      const bool fold = p.adjoint && COUT == 3;   // VRS adjoint: Ez gradient folded into Ex, Ey
      float Y = 0.f, z2 = 0.f;
      if (fold) {
        const float zb = (float)p.z[b];
        Y = (float)p.y[r];
        z2 = Y * Y + zb * zb;
      }
      const float2* base = ONE ? line : lines;
      for (int n = ONE ? t : tid; n < nx; n += ONE ? F::T : THREADS) {
        const long long o = (long long)b * p.obs + (long long)r * nx + n;
        const float2* s = base + (n >> 8) * F::BLK + blk_slot(n & 255);
        float2 e[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) e[c] = c < COUT ? s[c * F::LINE] : make_float2(0.f, 0.f);
        if (fold) {  // adjoint of Ez = Ex X/r + Ey Y/r (vectorized_optics.py:258-261)
          const float X = (float)p.x[n];
          const float inv = rsqrtf(X * X + z2);
          p.out[0][o] = cadd(e[0], cscale(e[2], X * inv));
          p.out[1][o] = cadd(e[1], cscale(e[2], Y * inv));
          if (p.out[2]) p.out[2][o] = e[2];   // the unfolded Ez gradient, when asked for
          continue;
        }
        const PixelCtx px{r, n, (long long)r * nx + n, b};
        apply_prog(p.post, e, px);
#pragma unroll
        for (int c = 0; c < COUT; ++c) p.out[c][o] = e[c];
      }
      if constexpr (ONE) sync();
      else __syncthreads();
    }
  }
  tmem_release<THREADS, 64>(s_tmem);
}

// Rows of the wrapped impulse response (see rs_hhat_rows_b), one row a CTA.
template <int R, bool DZ>
__global__ void __launch_bounds__(BlkFft<R>::T)
    rs_hhat_rows_h(int ny, int nx, int py, const float2* __restrict__ off, double zh, const double* __restrict__ zp,
                   double inv_lambda, float k, float2* __restrict__ out) {
  using F = BlkFft<R>;
  constexpr int M = F::P, P = 2 * M;
  const RsGeom g = rs_geom(zp ? __ldg(zp) : zh, inv_lambda, k);
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* twb = (float2*)smraw;
  float2* line = twb + F::NTB;
  float2* odd = line + F::LINE;   // M
  const int t = threadIdx.x, i = blockIdx.x;
  for (int j = t; j < F::NTB; j += F::T) twb[j] = blk_tw<R>()[F::NTA + j];
  const bool vy = (i < ny) || (i > py - ny);
  const float2 oy = off[P + i];
  const ffloat y = {oy.x, oy.y};
  const ffloat zy = ff_add(g.z2, ff_mul(y, y));
  auto value = [&](int col) {
    float2 h = make_float2(0.f, 0.f);
    if (vy && ((col < nx) || (col > P - nx))) {
      const float2 ox = off[col];
      const ffloat x = {ox.x, ox.y};
      const ffloat sq = ff_add(zy, ff_mul(x, x));
      h = DZ ? rs_dz_value_s(g, sq) : rs_value_s(g, sq);
    }
    return h;
  };
  float2* own = line + blk_slot(t);
#pragma unroll 2
  for (int n1 = 0; n1 < R; ++n1) {
    const int col = t + 256 * n1;
    const float2 a = value(col), d = value(col + M);
    own[n1 * F::BLK] = cadd(a, d);
    odd[col] = cmul(csub(a, d), half_tw<R>()[col]);
  }
  float2* blk = line + (t >> 4) * F::BLK;
#pragma unroll 1
  for (int h = 0; h < 2; ++h) {
    float2 v[16];
#pragma unroll
    for (int n1 = 0; n1 < R; ++n1) v[n1] = h ? odd[t + 256 * n1] : own[n1 * F::BLK];
    __syncthreads();   // twb, and the even half's slots
    blk_a_fwd<R, -1, false>(v, t, line, GlobalTw<R>{blk_tw<R>() + t});
    __syncthreads();
    if (t >= F::TB) continue;
    blk_b_fwd<-1>(v, t & 15, blk, twb);
    __syncwarp();
    blk_c_fwd<-1>(v, t & 15, blk);
    float2* dst = out + (long long)i * P + h * M + (t >> 5) * 512 + (t & 31);
#pragma unroll
    for (int q = 0; q < 16; ++q) dst[32 * q] = v[q];
  }
}

// ---- launches ----

template <int R, int MODE, class FK = FixedKinds<>> static int launch_rows_fwd_h(cudaStream_t s, const RsLaunch& p) {
  using K = HalfRow<R>;
  const size_t sm = K::LINES + (size_t)p.nx * (3 * 8 + (MODE == 2 ? 4 : 0));
  int per_sm;
  if (int rc = launch_ready<rs_rows_fwd_h<R, MODE, FK>>(K::THREADS, sm, &per_sm, "rs_rows_fwd_h")) return rc;
  const int total = p.B * p.ny, units = MODE == 1 ? (total + 2) / 3 : total;
  RowStage st;   // nothing staged: the rows' planes, to be prefetched
  plan_row_stage(p.cin, p.in, p.ibs, p.nx, p.pre, 1, sm, st, 0);
  rs_rows_fwd_h<R, MODE, FK><<<persistent_grid(1, units), K::THREADS, sm, s>>>(p, st);
  XL_CHECK_LAUNCH("rs_rows_fwd_h");
  return XL_OK;
}

template <int R, int COUT, bool EPI> static int launch_rows_inv_h(cudaStream_t s, const RsLaunch& p) {
  using K = HalfRow<R>;
  int per_sm;
  if (int rc = launch_ready<rs_rows_inv_h<R, COUT, EPI>>(K::THREADS, K::LINES, &per_sm, "rs_rows_inv_h")) return rc;
  const int total = p.B * p.ny, units = COUT == 1 ? (total + 2) / 3 : total;
  rs_rows_inv_h<R, COUT, EPI><<<persistent_grid(1, units), K::THREADS, K::LINES, s>>>(p);
  XL_CHECK_LAUNCH("rs_rows_inv_h");
  return XL_OK;
}

template <int R> int rs_half_rows(cudaStream_t st, const RsLaunch& p, bool inverse) {
  if (!inverse) {
    // the fixed programs of rs_blk_rows (us, generic and fixed: LCD and polarizer,
    // 2 x 2300^2 349 and 346, one 3200^2 334 and 320; SLM 319 and 300, 304 and 277)
    using SlmOnly = FixedKinds<XL_OP_PHASE>;
    using LcdLp = FixedKinds<XL_OP_LCD, XL_OP_LP>;
    using SlmsOnly = FixedKinds<XL_OP_SSLM>;
    if (p.cout == 1)
      return SlmOnly::matches(p.pre) ? launch_rows_fwd_h<R, 1, SlmOnly>(st, p) : launch_rows_fwd_h<R, 1>(st, p);
    if (p.cin == 3) return launch_rows_fwd_h<R, 3>(st, p);
    if (LcdLp::matches(p.pre)) return launch_rows_fwd_h<R, 2, LcdLp>(st, p);
    return SlmsOnly::matches(p.pre) ? launch_rows_fwd_h<R, 2, SlmsOnly>(st, p) : launch_rows_fwd_h<R, 2>(st, p);
  }
  const bool epi = p.post.nops > 0 || (p.adjoint && p.cout == 3);
  if (p.cout == 1) return epi ? launch_rows_inv_h<R, 1, true>(st, p) : launch_rows_inv_h<R, 1, false>(st, p);
  return epi ? launch_rows_inv_h<R, 3, true>(st, p) : launch_rows_inv_h<R, 3, false>(st, p);
}

template <int R> int rs_half_cols(cudaStream_t st, const RsLaunch& p) {
  using K = RsColB<R>;
  RsLaunch q = p;
  if (p.pol) q.cout = 2;
  int per_sm;
  if (int rc = launch_ready<rs_cols_h<R>>(K::THREADS, HalfCol<R>::SMEM, &per_sm, "rs_cols_h")) return rc;
  rs_cols_h<R><<<persistent_grid(1, p.B * (p.px / K::CW)), K::THREADS, HalfCol<R>::SMEM, st>>>(q);
  XL_CHECK_LAUNCH("rs_cols_h");
  return XL_OK;
}

template <int R>
int rs_half_hhat_rows(cudaStream_t st, int ny, int nx, int py, const double* offx, const double* offy, int q2, double z,
                      const double* zp, double wavelength, int dz, float2* off, float2* out) {
  using F = BlkFft<R>;
  constexpr int P = 2 * F::P;
  rs_split_offsets_b<<<(P + py + 255) / 256, 256, 0, st>>>(offx, offy, q2, P, py, off);
  XL_CHECK_LAUNCH("rs_split_offsets_b");
  const size_t sm = ((size_t)F::NTB + F::LINE + F::P) * 8;
  const float k = (float)(2.0 * M_PI / wavelength);
  int per_sm;
  auto run = [&](auto kernel, int rc) {
    if (rc) return rc;
    kernel<<<py, F::T, sm, st>>>(ny, nx, py, off, z, zp, 1.0 / wavelength, k, out);
    XL_CHECK_LAUNCH("rs_hhat_rows_h");
    return (int)XL_OK;
  };
  if (dz) return run(rs_hhat_rows_h<R, true>, launch_ready<rs_hhat_rows_h<R, true>>(F::T, sm, &per_sm, "rs_hhat_rows_h"));
  return run(rs_hhat_rows_h<R, false>, launch_ready<rs_hhat_rows_h<R, false>>(F::T, sm, &per_sm, "rs_hhat_rows_h"));
}

template <int R> int rs_half_hhat_cols(cudaStream_t st, const float2* in, int px, float scale, float2* out) {
  using K = RsColB<R>;
  const size_t sm = ((size_t)BlkFft<R>::NTB + (size_t)K::CW * K::LINE) * 8;
  int per_sm;
  if (int rc = launch_ready<rs_hhat_cols_h<R>>(K::THREADS, sm, &per_sm, "rs_hhat_cols_h")) return rc;
  rs_hhat_cols_h<R><<<px / K::CW, K::THREADS, sm, st>>>(in, px, scale, out);
  XL_CHECK_LAUNCH("rs_hhat_cols_h");
  return XL_OK;
}

}  // namespace xl

#define XL_RS_HALF_INSTANTIATE(R)                                                                             \
  template int xl::rs_half_rows<R>(cudaStream_t, const RsLaunch&, bool);                                      \
  template int xl::rs_half_cols<R>(cudaStream_t, const RsLaunch&);                                            \
  template int xl::rs_half_hhat_rows<R>(cudaStream_t, int, int, int, const double*, const double*, int, double, \
                                        const double*, double, int, float2*, float2*);                        \
  template int xl::rs_half_hhat_cols<R>(cudaStream_t, const float2*, int, float, float2*);
