// RS / VRS kernels on the in-place block FFT engine (fft_block.cuh), for
// transforms of P = 256 R points.
#pragma once

#include <math.h>

#include <type_traits>

#include "blk_common.cuh"
#include "rs_host.h"

namespace xl {

// Column pass, in place on CW columns of a tile: FFT along y of the ny nonzero
// rows, multiply by the transfer spectrum (conjugate for the adjoint), inverse
// FFT, keep the ny surviving rows.  Persistent: CTAs walk the (batch entry,
// column group) units batch entries fastest, so that entries at the same
// distance read one spectrum tile together.  Spectra are stored in the order
// phase C holds them (rs_hhat_cols_b), so a warp reads 256 contiguous bytes.
//
// What bounds it: the shared-memory pipe (60 % busy at 4096 points, the FP32
// pipe 48 %); without any of its global loads and stores it runs 16 % faster.
// So the CTAs of 1024 threads (R > 4) keep what a thread reads again and again
// in its own Tensor Memory cells, which are not on that pipe: the phase A
// twiddles (a thread's j never changes), and a unit's spectrum values for the
// second and third component.  8 x 2048^2 VRS: 1.50 ms with both, 1.58 ms
// without, 1.92 ms on the Stockham engine with its eight barriers a component.
// The smaller CTAs (R = 4, four per SM) keep their tables in shared memory: with
// Tensor Memory they took 291 against 178 us for 16 x 500^2 VRS.
//
// A thread holds 64 of the Tensor Memory columns of its lane, CTAs of 1024
// threads all 512; the 64 registers of a thread allow one such CTA per SM, so
// an allocation never waits for another one's columns.
template <int R>
__global__ void __launch_bounds__(RsColB<R>::THREADS, RsColB<R>::MINB) rs_cols_b(const __grid_constant__ RsLaunch p) {
  using F = BlkFft<R>;
  using K = RsColB<R>;
  constexpr bool TM = K::TM;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned s_tmem;
  float2* tw = (float2*)smraw;   // NTW: an even count, so that the lines stay 16-byte aligned
  float2* xch = tw + F::NTW;
  const ColMap<R> m;
  {
    const float2* g = blk_tw<R>();
    for (int i = threadIdx.x; i < F::NTW; i += K::THREADS) tw[i] = g[i];
  }
  __syncthreads();
  const SmemTw<R> tws{tw + m.jt};
  typename std::conditional<TM, TmemTw<R>, SmemTw<R>>::type twa;
  unsigned scell = 0;
  if constexpr (TM) {
    twa.cell = tmem_twiddles<R, K::THREADS, 64>(&s_tmem, tws);
    scell = twa.cell + 32u;
  } else {
    twa = tws;
  }
  float2* line = xch + m.wc * K::LINE;
  float2* blk = xch + m.bc * K::LINE + m.k1 * F::BLK;
  const float2* twb = tw + F::NTA;
  const bool active = m.warp < K::WARPS_B;
  const int ny = p.ny, lw = p.lw;
  const int units = p.B * (p.px / K::CW);
#pragma unroll 1
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const int b = u % p.B, g = u / p.B;
    const long long col = (long long)g * K::CW + m.wc;
    const float2* sbase = p.specs ? p.specs[b] : p.spec + (long long)(p.sidx ? p.sidx[b] : 0) * p.sstride;
    const float2* spec = sbase + (long long)g * (K::CW * F::P) + m.warp * 512 + m.lane;
#pragma unroll 1
    for (int c = 0; c < p.cout; ++c) {
      float2* tile = p.work + ((long long)b * p.cout + c) * ny * p.px + (((col >> lw) * ny) << lw) +
                     (col & ((1 << lw) - 1));
      float2 v[16];
#pragma unroll
      for (int i = 0; i < F::IPT; ++i)
#pragma unroll
        for (int n = 0; n < R / 2; ++n) {
          const int r = m.jt + i * F::T + 256 * n;
          v[i * R + n] = r < ny ? tile[(long long)r << lw] : make_float2(0.f, 0.f);
        }
      blk_a_fwd<R, -1, true>(v, m.jt, line, twa);
      __syncthreads();
      if (active) {
        blk_b_fwd<-1>(v, m.l, blk, twb);
        __syncwarp();
        blk_c_fwd<-1>(v, m.l, blk);
        const float2* sp = spec;
        asm volatile("" : "+l"(sp));   // the loads stay here: ahead of the transform they would hold 32 registers
        auto mul4 = [&](int q, const float2 (&w)[4]) {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[4 * q + i] = p.adjoint ? cmulc(v[4 * q + i], w[i]) : cmul(v[4 * q + i], w[i]);
        };
        if (TM && c > 0) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float2 w[4];
            tmem_ld4(scell + 8u * q, w, false);
            mul4(q, w);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float2 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = __ldg(sp + (4 * q + i) * 32);
            if (TM && p.cout > 1) tmem_st4(scell + 8u * q, w[0], w[1], w[2], w[3], false);
            mul4(q, w);
          }
          if (TM && p.cout > 1) tmem_wait_st(false);   // complete before the next component's loads
        }
        blk_c_inv<1>(v, m.l, blk);
        __syncwarp();
        blk_b_inv<1>(v, m.l, blk, twb);
      }
      __syncthreads();
      blk_a_inv<R, 1>(v, m.jt, line, twa);
#pragma unroll
      for (int i = 0; i < F::IPT; ++i)
#pragma unroll
        for (int n = 0; n < R / 2; ++n) {
          const int r = m.jt + i * F::T + 256 * n;
          if (r < ny) tile[(long long)r << lw] = v[i * R + n];
        }
    }
  }
  if constexpr (TM) tmem_release<K::THREADS, 64>(s_tmem);
}

// Transfer spectrum, column transforms of the row spectra (`in`: P rows of px
// columns), times `scale`, stored per group of CW columns in the order phase
// C of the column pass holds them: [group][warp][register][lane].
template <int R>
__global__ void __launch_bounds__(RsColB<R>::THREADS, RsColB<R>::MINB)
    rs_hhat_cols_b(const float2* __restrict__ in, int px, float scale, float2* __restrict__ out) {
  using F = BlkFft<R>;
  using K = RsColB<R>;
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* tw = (float2*)smraw;           // NTW: an even count, so that the lines stay 16-byte aligned
  float2* xch = tw + F::NTW;
  const ColMap<R> m;
  {
    const float2* g = blk_tw<R>();
    for (int i = threadIdx.x; i < F::NTW; i += K::THREADS) tw[i] = g[i];
  }
  __syncthreads();
  float2 v[16];
  const float2* src = in + (long long)blockIdx.x * K::CW + m.wc;
#pragma unroll
  for (int i = 0; i < F::IPT; ++i)
#pragma unroll
    for (int n = 0; n < R; ++n) v[i * R + n] = src[(long long)(m.jt + i * F::T + 256 * n) * px];
  blk_a_fwd<R, -1, false>(v, m.jt, xch + m.wc * K::LINE, SmemTw<R>{tw + m.jt});
  __syncthreads();
  if (m.warp >= K::WARPS_B) return;
  float2* blk = xch + m.bc * K::LINE + m.k1 * F::BLK;
  blk_b_fwd<-1>(v, m.l, blk, tw + F::NTA);
  __syncwarp();
  blk_c_fwd<-1>(v, m.l, blk);
  float2* dst = out + (long long)blockIdx.x * (K::CW * F::P) + m.warp * 512 + m.lane;
#pragma unroll
  for (int q = 0; q < 16; ++q) dst[32 * q] = cscale(v[q], scale);
}

// ---- row passes ----
// Positions: the P columns of the intermediate are in the order the row
// passes' phase C threads hold them: thread (k1, k2) = warp wq, lane of its
// line holds register m at position (wq 16 + m) 32 + lane, so a warp's access
// covers 32 positions.  Column groups and transfer spectra are in the same
// order.

// Base of a phase C thread's positions in row r of a column-tiled plane (tiles
// of 2^lw, lw <= 5); register m is 32 m columns, that is 32 ny m elements, further
// on.
__device__ __forceinline__ long long row_pos(int wq, int lane, int r, int ny, int lw) {
  const int c = wq * 512 + lane;
  return (((long long)(c >> lw) * ny + r) << lw) + (c & ((1 << lw) - 1));
}

// Component groups of a forward row CTA: one where a thread runs the program
// for its own elements, all three for the adjoint.  CTAs per SM the registers
// are sized for: two of 256 threads where a thread holds a second component
// (three, 80 registers: 533 us for 8 x 2048^2 fields behind a polarizer, two 467).
constexpr int rows_fwd_nc(int mode) { return mode == 3 ? 3 : 1; }
template <int R, int MODE> constexpr int rows_fwd_minb() {
  return MODE == 1 ? RowB<R, 1>::MINB : (MODE == 3 ? RowB<R, 3>::MINB : 2);
}

// Bytes of the forward row pass's shared memory before its stage.
template <int R, int MODE> __host__ __device__ constexpr size_t rows_fwd_fixed(int nx) {
  constexpr int NC = rows_fwd_nc(MODE);
  using K = RowB<R, NC>;
  constexpr int hold = MODE == 2 ? K::THREADS * BlkFft<R>::IPT * R / 2 : 0;
  return ((size_t)(BlkFft<R>::NTB + K::LINES * BlkFft<R>::LINE + (NC == 1 ? hold : 3 * K::G * nx)) * 8 +
          (MODE == 2 || MODE == 4 ? (size_t)nx * 4 : 0) + 15) / 16 * 16;
}

// Forward row pass.  MODE 1: scalar RS (one component); 2: VRS (Ex, Ey in;
// Ex, Ey, Ez out, Ez derived); 3: VRS adjoint (three gradients in and out, no
// program); 4: VRS behind a polarizer at one angle (the program's last op, left
// out of p.pre): Ex = c u and Ey = s u with u = c Ex' + s Ey', so the row has two
// components, u and Ez = u (c X + s Y) / r.
//
// Persistent: CTA c handles row groups c, c + grid, ...  The thread that needs
// an element of phase A runs the fused program for it itself, in CTAs of 256
// threads (several per SM, each at its own point of a row), and transforms its
// components one after the other; the stage is free after the first phase A and
// the bulk copies of the next row group start.  (VRS with three component groups
// in a CTA of 768 threads and the program's results in a shared buffer between:
// 774 us for 8 x 2048^2 behind an LCD and a polarizer, this form 467 with two
// components; without a program 694 and 502.)  The adjoint, which has no program,
// keeps the three groups.
// FK: the fused program's op kinds fixed at compile time (FixedKinds<...>,
// for the programs the benchmarks and tables run), or FixedKinds<>.
template <int R, int MODE, class FK = FixedKinds<>>
__global__ void __launch_bounds__(RowB<R, rows_fwd_nc(MODE)>::THREADS, rows_fwd_minb<R, MODE>())
    rs_rows_fwd_b(const __grid_constant__ RsLaunch p, const __grid_constant__ RowStage st) {
  constexpr int NC = rows_fwd_nc(MODE);
  constexpr bool TM = RowB<R, NC>::TM;
  __shared__ unsigned s_tmem;
  constexpr int CIN = MODE == 4 ? 2 : MODE;
  using F = BlkFft<R>;
  using K = RowB<R, NC>;
  extern __shared__ __align__(16) unsigned char smraw[];
  const int nx = p.nx, ny = p.ny;
  float2* twb = (float2*)smraw;                                      // NTB
  float2* xch = twb + F::NTB;                                        // LINES x LINE
  // the adjoint's rows (3 x G x nx); VRS: Ey of every thread's elements
  float2* post = xch + K::LINES * F::LINE;
  constexpr int HOLD = MODE == 2 ? K::THREADS * F::IPT * R / 2 : 0;
  float* xf = (float*)(post + (NC == 1 ? HOLD : 3 * K::G * nx));     // nx (VRS: x as float32)
  const size_t soff = rows_fwd_fixed<R, MODE>(nx);
  unsigned char* stage = smraw + soff;
  unsigned long long* mbar = (unsigned long long*)(stage + (size_t)K::G * st.row_bytes);
  const int tid = threadIdx.x;
  const int ln = tid / F::T, t = tid % F::T;
  const int cg = ln / K::G, gi = ln % K::G;
  const int ngb = (ny + K::G - 1) / K::G;
  const int total = p.B * ngb;
  const bool staged = st.n > 0;
  float2* line = xch + ln * F::LINE;
  float2* blk = line + (t >> 4) * F::BLK;
  const bool active = t < F::TB;
  const GlobalTw<R> twg{blk_tw<R>() + t};
  typename std::conditional<TM, TmemTw<R>, GlobalTw<R>>::type twa;
  if constexpr (TM) twa.cell = tmem_twiddles<R, K::THREADS, 32>(&s_tmem, twg);
  else twa = twg;

  if (tid == 0 && staged) {
    mbar_init(mbar, 1);
    fence_mbar_init();
  }
  for (int i = tid; i < F::NTB; i += K::THREADS) twb[i] = blk_tw<R>()[F::NTA + i];
  if constexpr (MODE == 2 || MODE == 4)
    for (int i = tid; i < nx; i += K::THREADS) xf[i] = (float)p.x[i];
  __syncthreads();

  // row groups are taken batch entries fastest: CTAs that run together read the
  // same rows of the parameter planes a batch shares, which then come from L2
  auto issue = [&](int grp) {
    const int b = grp % p.B, r0 = (grp / p.B) * K::G;
    stage_rows(st, stage, mbar, b, r0, min(K::G, ny - r0));
  };
  if (tid == 0 && staged && blockIdx.x < total) issue(blockIdx.x);

  unsigned phase = 0;
  // the copy may still be in flight: let it land, record the event and leave
  // without issuing another
  auto timed_out = [&]() {
    mbar_wait_bounded(mbar, phase);
    if (tid == 0) record_timeout();
    if constexpr (TM) tmem_release<K::THREADS, 32>(s_tmem);
  };
  auto next_stage = [&](int grp) {
    phase ^= 1u;
    if (tid == 0 && staged && grp + gridDim.x < total) {
      fence_proxy_async();
      issue(grp + gridDim.x);
    }
  };
  for (int grp = blockIdx.x; grp < total; grp += gridDim.x) {
    const int b = grp % p.B;
    const int r0 = (grp / p.B) * K::G;
    // a wait that runs out is acted on at the barrier after the prologue
    // (the prologue then works on stale data, and the launch's output is not
    // valid), so that no extra barrier is taken per row group
    const bool got = !staged || mbar_wait_bounded(mbar, phase, g_wait_limit_ns);
    const int r = r0 + gi;
    const bool live = r < ny;
    float2 v[16];
    if constexpr (NC == 1) {
      // this thread's elements, NP at a time (the program's code is laid out once
      // for each), through its own slots of the line: no barrier; positions past
      // the row or the field take a valid pixel and are zeroed
      constexpr int NP = MODE == 1 ? 4 : 2;
      const int rr = live ? r : ny - 1;
      constexpr int H = R / 2, N = F::IPT * H;   // 5 to 8 elements
      float2* own = line + blk_slot(t);
      auto pos = [&](int f) { return t + f / H * F::T + 256 * (f % H); };
      auto slot = [&](int f) { return f % H * F::BLK + f / H * (F::T / 16) * 18; };
#pragma unroll 1
      for (int f0 = 0; f0 < N; f0 += NP) {
        float2 e[NP][3];
        PixelCtx px[NP];
        StagedParams pr[NP];
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          const int n = min(pos(f0 + q), nx - 1);
          const long long pix = (long long)rr * nx + n;
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            e[q][i] = make_float2(0.f, 0.f);
            if (i < CIN) {
              const int fo = st.fld[i];
              e[q][i] = fo >= 0 ? ((const float2*)(stage + fo))[(rr - r0) * nx + n] : p.in[i][(long long)b * p.ibs + pix];
            }
          }
          px[q] = PixelCtx{rr, n, pix, b};
          pr[q] = StagedParams{stage, &st, rr - r0, nx, n};
        }
        if constexpr (FK::n > 0) apply_prog_fixed<FK>(p.pre, e, px, pr);
        else if (p.pre.nops) apply_prog_vec<NP>(p.pre, e, px, pr);
#pragma unroll
        for (int q = 0; q < NP; ++q) {
          if constexpr (MODE == 4) e[q][0] = cadd(cscale(e[q][0], p.pol_c), cscale(e[q][1], p.pol_s));
          if (N % NP == 0 || f0 + q < N) {
            own[slot(f0 + q)] = e[q][0];
            if constexpr (MODE == 2) post[(f0 + q) * K::THREADS + tid] = e[q][1];
          }
        }
      }
#pragma unroll
      for (int f = 0; f < N; ++f)
        v[f / H * R + f % H] = (live && pos(f) < nx) ? own[slot(f)] : make_float2(0.f, 0.f);
    } else {
      const int lim = min(K::G, ny - r0) * nx;
      for (int idx = tid; idx < lim; idx += K::THREADS) {
        const int g2 = K::G == 1 ? 0 : idx / nx, n = idx - g2 * nx;
        const long long pix = (long long)(r0 + g2) * nx + n;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          const int fo = st.fld[c];
          post[c * K::G * nx + idx] = fo >= 0 ? ((const float2*)(stage + fo))[idx] : p.in[c][(long long)b * p.ibs + pix];
        }
      }
      // every thread has read the stage and written its pixels; every thread
      // takes the timeout branch or none does
      if (__syncthreads_or(!got)) return timed_out();
      next_stage(grp);
      const float2* src = post + (cg * K::G + gi) * nx;
#pragma unroll
      for (int i = 0; i < F::IPT; ++i)
#pragma unroll
        for (int n1 = 0; n1 < R / 2; ++n1) {
          const int n = t + i * F::T + 256 * n1;
          v[i * R + n1] = (live && n < nx) ? src[n] : make_float2(0.f, 0.f);
        }
    }
    auto finish = [&](int plane) {   // phases B and C of a row, and its store
      if (!active) return;
      blk_b_fwd<-1>(v, t & 15, blk, twb);
      __syncwarp();
      blk_c_fwd<-1>(v, t & 15, blk);
      if (live) {
        float2* o = p.work + (long long)plane * ny * F::P + row_pos(t >> 5, t & 31, r, ny, p.lw);
        long long step = 32LL * ny;
        asm volatile("" : "+l"(o), "+l"(step));   // one base, not sixteen addresses live across the loop
#pragma unroll
        for (int q = 0; q < 16; ++q) o[q * step] = v[q];
      }
    };
    constexpr bool VRS = MODE == 2 || MODE == 4;
    float2 uz[VRS ? F::IPT * R / 2 : 1];   // Ez of this thread's elements
    if constexpr (VRS) {
      const float zb = (float)p.z[b], Y = (float)p.y[live ? r : ny - 1];
      const float z2 = Y * Y + zb * zb, sY = p.pol_s * Y;
#pragma unroll
      for (int i = 0; i < F::IPT; ++i)
#pragma unroll
        for (int n1 = 0; n1 < R / 2; ++n1) {   // vectorized_optics.py:258-261, Ez = Ex X/r + Ey Y/r
          const int f = i * (R / 2) + n1, n = t + i * F::T + 256 * n1;
          const float X = xf[min(n, nx - 1)], inv = rsqrtf(X * X + z2);
          if constexpr (MODE == 4) {   // Ex = c u, Ey = s u
            uz[f] = cscale(v[i * R + n1], (p.pol_c * X + sY) * inv);
          } else {
            const float2 ey = live && n < nx ? post[f * K::THREADS + tid] : make_float2(0.f, 0.f);
            uz[f] = cadd(cscale(v[i * R + n1], X * inv), cscale(ey, Y * inv));
          }
        }
    }
    blk_a_fwd<R, -1, true>(v, t, line, twa);
    if constexpr (NC == 1) {
      if (__syncthreads_or(!got)) return timed_out();
      next_stage(grp);
    } else {
      __syncthreads();
    }
    constexpr int COUT = MODE == 1 ? 1 : (MODE == 4 ? 2 : 3);
    finish(b * COUT + cg);
    if constexpr (NC == 1) __syncthreads();   // the next phase A stores to the slots phase C loads here
    auto another = [&](int c) {   // component c, in v
      blk_a_fwd<R, -1, true>(v, t, line, twa);
      __syncthreads();
      finish(b * COUT + c);
      __syncthreads();
    };
    if constexpr (MODE == 2) {
#pragma unroll
      for (int i = 0; i < F::IPT; ++i)
#pragma unroll
        for (int n1 = 0; n1 < R / 2; ++n1)
          v[i * R + n1] = live && t + i * F::T + 256 * n1 < nx ? post[(i * (R / 2) + n1) * K::THREADS + tid]
                                                               : make_float2(0.f, 0.f);
      another(1);
    }
    if constexpr (VRS) {
#pragma unroll
      for (int i = 0; i < F::IPT; ++i)
#pragma unroll
        for (int n1 = 0; n1 < R / 2; ++n1) v[i * R + n1] = uz[i * (R / 2) + n1];
      another(COUT - 1);
    }
  }
  if constexpr (TM) tmem_release<K::THREADS, 32>(s_tmem);
}

// Inverse row pass: inverse P-point FFT per row and component, crop to nx
// columns, optional fused epilogue program (or, for the VRS adjoint, the fold
// of the Ez gradient into Ex, Ey), store.  Persistent, with the component
// groups of RowB; each thread's loads of its next row are in flight in
// registers while the current one is transformed.  With an epilogue phase A
// leaves the row in its own slots, since the program needs every component of
// a pixel.
//
// What bounds it: the loads in flight, which occupy L1 by whole 128-byte lines
// (a row's pieces are 64 bytes), so shared memory is kept small: with two sets
// of lines (one barrier a row instead of two) 8 x 2048^2 VRS took 728 us
// against 464, and with the phase A twiddles read through L1 instead of kept
// in Tensor Memory 561; loads that do not allocate in L1 took 628.  Stockham
// engine: 573.  (16 x 1024^2 scalar, three CTAs an SM: 84 us, 123 on Stockham;
// with Tensor Memory 95.)
//
// POL (one component, no epilogue): the planes u and Ez of VRS behind a
// polarizer, as entries 2 b and 2 b + 1: Ex = c u, Ey = s u and Ez.
template <int R, int COUT, bool EPI, bool POL = false>
__global__ void __launch_bounds__(RowB<R, COUT>::THREADS, RowB<R, COUT>::MINB)
    rs_rows_inv_b(const __grid_constant__ RsLaunch p) {
  constexpr bool TM = RowB<R, COUT>::TM;
  __shared__ unsigned s_tmem;
  using F = BlkFft<R>;
  using K = RowB<R, COUT>;
  static_assert(K::CG == COUT, "every component of a row at once");
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* twb = (float2*)smraw;
  float2* line = twb + F::NTB + (threadIdx.x / F::T) * F::LINE;   // LINES x LINE
  const int tid = threadIdx.x;
  const int ln = tid / F::T, t = tid % F::T;
  const int cg = ln / K::G, gi = ln % K::G;
  const int nx = p.nx, ny = p.ny;
  const int ngb = (ny + K::G - 1) / K::G;
  const int total = p.B * ngb;
  const bool active = t < F::TB;
  for (int i = tid; i < F::NTB; i += K::THREADS) twb[i] = blk_tw<R>()[F::NTA + i];
  const GlobalTw<R> twg{blk_tw<R>() + t};
  typename std::conditional<TM, TmemTw<R>, GlobalTw<R>>::type twa;
  if constexpr (TM) twa.cell = tmem_twiddles<R, K::THREADS, 32>(&s_tmem, twg);
  else twa = twg;
  __syncthreads();

  auto load = [&](int grp, float2 (&d)[16]) {   // row groups batch entries fastest
    const int b = grp % p.B;
    int r = (grp / p.B) * K::G + gi;
    r = r < ny ? r : ny - 1;    // rows past the end load a valid row and discard it
    const float2* q = p.work + ((long long)b * COUT + cg) * ny * F::P + row_pos(t >> 5, t & 31, r, ny, p.lw);
    long long step = 32LL * ny;
    asm volatile("" : "+l"(q), "+l"(step));
#pragma unroll
    for (int m = 0; m < 16; ++m) d[m] = q[m * step];
  };

  float2 nxt[16];
  if (active && blockIdx.x < total) load(blockIdx.x, nxt);
  for (int grp = blockIdx.x; grp < total; grp += gridDim.x) {
    const int b = grp % p.B;
    const int r0 = (grp / p.B) * K::G;
    const int r = r0 + gi;
    float2 v[16];
    if (active) {
      float2* blk = line + (t >> 4) * F::BLK;
#pragma unroll
      for (int m = 0; m < 16; ++m) v[m] = nxt[m];
      if (grp + gridDim.x < total) load(grp + gridDim.x, nxt);
      blk_c_inv<1>(v, t & 15, blk);
      __syncwarp();
      blk_b_inv<1>(v, t & 15, blk, twb);
    }
    if constexpr (!EPI && K::CG > 1) GroupSync{1 + cg, K::G * F::T}();   // the component groups never meet
    else __syncthreads();
    blk_a_inv<R, 1>(v, t, line, twa);
    if constexpr (!EPI) {
      if (POL && r < ny) {
        const long long row = (long long)(b >> 1) * p.obs + (long long)r * nx;
        const bool ez = b & 1;
        float2* o = p.out[ez ? 2 : 0] + row;
        float2* o1 = p.out[1] + row;
        const float f = ez ? 1.f : p.pol_c;
#pragma unroll
        for (int i = 0; i < F::IPT; ++i)
#pragma unroll
          for (int n1 = 0; n1 < R / 2; ++n1) {
            const int n = t + i * F::T + 256 * n1;
            if (n < nx) {
              o[n] = ez ? v[i * R + n1] : cscale(v[i * R + n1], f);
              if (!ez) o1[n] = cscale(v[i * R + n1], p.pol_s);
            }
          }
      } else if (r < ny) {
        float2* o = p.out[cg] + (long long)b * p.obs + (long long)r * nx;
#pragma unroll
        for (int i = 0; i < F::IPT; ++i)
#pragma unroll
          for (int n1 = 0; n1 < R / 2; ++n1) {
            const int n = t + i * F::T + 256 * n1;
            if (n < nx) o[n] = v[i * R + n1];
          }
      }
    } else {
      float2* d = line + blk_slot(t);
#pragma unroll
      for (int i = 0; i < F::IPT; ++i)
#pragma unroll
        for (int n1 = 0; n1 < R / 2; ++n1) d[n1 * F::BLK + i * (F::T / 16) * 18] = v[i * R + n1];
      __syncthreads();
      const bool fold = p.adjoint && COUT == 3;   // VRS adjoint: Ez gradient folded into Ex, Ey
      const float zb = fold ? (float)p.z[b] : 0.f;
      int last = -1;
      float Y = 0.f, z2 = 0.f;
      for (int idx = tid; idx < K::G * nx; idx += K::THREADS) {
        const int g2 = K::G == 1 ? 0 : idx / nx, n = idx - g2 * nx, ro = r0 + g2;
        if (ro >= ny) break;
        const long long o = (long long)b * p.obs + (long long)ro * nx + n;
        const float2* s = twb + F::NTB + g2 * F::LINE + (n >> 8) * F::BLK + blk_slot(n & 255);
        float2 e[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) e[c] = c < COUT ? s[c * K::G * F::LINE] : make_float2(0.f, 0.f);
        if (fold) {  // adjoint of Ez = Ex X/r + Ey Y/r (vectorized_optics.py:258-261)
          if (g2 != last) {
            last = g2;
            Y = (float)p.y[ro];
            z2 = Y * Y + zb * zb;
          }
          const float X = (float)p.x[n];
          const float inv = rsqrtf(X * X + z2);
          p.out[0][o] = cadd(e[0], cscale(e[2], X * inv));
          p.out[1][o] = cadd(e[1], cscale(e[2], Y * inv));
          if (p.out[2]) p.out[2][o] = e[2];   // the unfolded Ez gradient, when asked for
          continue;
        }
        PixelCtx px{ro, n, (long long)ro * nx + n, b};
        apply_prog(p.post, e, px);
#pragma unroll
        for (int c = 0; c < COUT; ++c) p.out[c][o] = e[c];
      }
    }
    // the next row's phase C stores to slots that phase A (or the epilogue) loads here
    if constexpr (!EPI && K::CG > 1) GroupSync{1 + cg, K::G * F::T}();
    else __syncthreads();
  }
  if constexpr (TM) tmem_release<K::THREADS, 32>(s_tmem);
}

// ---- transfer spectra ----

// The wrapped offsets (arrays of length 2 Q, Q the power of two the ABI states)
// rewrapped for px x py points and split into float-float (hi, lo) pairs: offx
// into off[0 .. px), offy into off[px .. px + py).  `off` is the spectrum
// buffer, which rs_hhat_cols_b overwrites afterwards.
static __global__ void rs_split_offsets_b(const double* __restrict__ offx, const double* __restrict__ offy, int q2,
                                          int px, int py, float2* __restrict__ off) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= px + py) return;
  const bool isx = i < px;
  const int n = isx ? px : py, k = isx ? i : i - px;
  const int d = k < n - k ? k : k - n;                    // index distance
  const ffloat v = ff_split((isx ? offx : offy)[d < 0 ? d + q2 : d]);
  off[i] = make_float2(v.hi, v.lo);
}

// Rows of the wrapped impulse response -> P-point row spectra, row-major in
// position order.  DZ: the rows of dH/dz instead (the spectrum of the
// z-derivative).
template <int R, bool DZ>
__global__ void __launch_bounds__(RowB<R, 1>::THREADS)
    rs_hhat_rows_b(int ny, int nx, int py, const float2* __restrict__ off, double zh, const double* __restrict__ zp,
                   double inv_lambda, float k, float2* __restrict__ out) {
  using F = BlkFft<R>;
  using K = RowB<R, 1>;
  // a distance in device memory, or the host's value
  const RsGeom g = rs_geom(zp ? __ldg(zp) : zh, inv_lambda, k);
  extern __shared__ __align__(16) unsigned char smraw[];
  float2* twb = (float2*)smraw;
  const int ln = threadIdx.x / F::T, t = threadIdx.x % F::T;
  float2* line = twb + F::NTB + ln * F::LINE;
  for (int i = threadIdx.x; i < F::NTB; i += K::THREADS) twb[i] = blk_tw<R>()[F::NTA + i];
  const int i = blockIdx.x * K::G + ln;   // row of the wrapped response (< py)
  const bool vy = (i < ny) || (i > py - ny);
  const float2 oy = off[F::P + i];
  const ffloat y = {oy.x, oy.y};
  const ffloat zy = ff_add(g.z2, ff_mul(y, y));
  float2 v[16];
#pragma unroll
  for (int it = 0; it < F::IPT; ++it)
#pragma unroll
    for (int n1 = 0; n1 < R; ++n1) {
      const int col = t + it * F::T + 256 * n1;
      const bool vx = (col < nx) || (col > F::P - nx);
      float2 h = make_float2(0.f, 0.f);
      if (vy && vx) {
        const float2 ox = off[col];
        const ffloat x = {ox.x, ox.y};
        const ffloat sq = ff_add(zy, ff_mul(x, x));
        h = DZ ? rs_dz_value_s(g, sq) : rs_value_s(g, sq);
      }
      v[it * R + n1] = h;
    }
  blk_a_fwd<R, -1, false>(v, t, line, GlobalTw<R>{blk_tw<R>() + t});
  __syncthreads();
  if (t >= F::TB) return;
  float2* blk = line + (t >> 4) * F::BLK;
  blk_b_fwd<-1>(v, t & 15, blk, twb);
  __syncwarp();
  blk_c_fwd<-1>(v, t & 15, blk);
  float2* dst = out + (long long)i * F::P + (t >> 5) * 512 + (t & 31);
#pragma unroll
  for (int q = 0; q < 16; ++q) dst[32 * q] = v[q];
}

// ---- launches ----

template <int R> static int launch_cols_b(cudaStream_t st, const RsLaunch& p) {
  using K = RsColB<R>;
  int per_sm;
  if (int rc = launch_ready<rs_cols_b<R>>(K::THREADS, K::SMEM, &per_sm, "rs_cols_b")) return rc;
  const int grid = persistent_grid(per_sm, p.B * (p.px / K::CW));
  rs_cols_b<R><<<grid, K::THREADS, K::SMEM, st>>>(p);
  XL_CHECK_LAUNCH("rs_cols_b");
  return XL_OK;
}

template <int R> static int launch_hhat_cols_b(cudaStream_t st, const float2* in, int px, float scale, float2* out) {
  using K = RsColB<R>;
  int per_sm;
  if (int rc = launch_ready<rs_hhat_cols_b<R>>(K::THREADS, K::SMEM, &per_sm, "rs_hhat_cols_b")) return rc;
  rs_hhat_cols_b<R><<<px / K::CW, K::THREADS, K::SMEM, st>>>(in, px, scale, out);
  XL_CHECK_LAUNCH("rs_hhat_cols_b");
  return XL_OK;
}

template <int R, int MODE, class FK = FixedKinds<>>
static int launch_rows_fwd_b(cudaStream_t s, const RsLaunch& p) {
  using K = RowB<R, rows_fwd_nc(MODE)>;
  const size_t fixed = rows_fwd_fixed<R, MODE>(p.nx);
  RowStage st;
  // the stage takes what leaves room for the CTAs the registers allow
  plan_row_stage(p.cin, p.in, p.ibs, p.nx, p.pre, K::G, fixed, st, (size_t)(227 * 1024) / rows_fwd_minb<R, MODE>() - 1024);
  const size_t sm = fixed + (size_t)K::G * st.row_bytes + 16;
  int per_sm;
  if (int rc = launch_ready<rs_rows_fwd_b<R, MODE, FK>>(K::THREADS, sm, &per_sm, "rs_rows_fwd_b")) return rc;
  const int total = p.B * ((p.ny + K::G - 1) / K::G);
  const int grid = persistent_grid(per_sm, total);
  rs_rows_fwd_b<R, MODE, FK><<<grid, K::THREADS, sm, s>>>(p, st);
  XL_CHECK_LAUNCH("rs_rows_fwd_b");
  return XL_OK;
}

template <int R, int COUT, bool EPI, bool POL = false> static int launch_rows_inv_b(cudaStream_t s, const RsLaunch& p) {
  using K = RowB<R, COUT>;
  const size_t sm = ((size_t)BlkFft<R>::NTB + K::LINES * BlkFft<R>::LINE) * 8;
  int per_sm;
  if (int rc = launch_ready<rs_rows_inv_b<R, COUT, EPI, POL>>(K::THREADS, sm, &per_sm, "rs_rows_inv_b")) return rc;
  const int total = p.B * ((p.ny + K::G - 1) / K::G);
  const int grid = persistent_grid(per_sm, total);
  rs_rows_inv_b<R, COUT, EPI, POL><<<grid, K::THREADS, sm, s>>>(p);
  XL_CHECK_LAUNCH("rs_rows_inv_b");
  return XL_OK;
}

template <int R> int rs_blk_rows(cudaStream_t st, const RsLaunch& p, bool inverse) {
  if (!inverse) {
    // programs that get a kernel with their op kinds fixed: a phase SLM before
    // scalar RS, a double-phase SLM before VRS, an LCD before a polarizer and VRS
    // (us, generic and fixed, at 1024 and 1536 points: 75 x 400^2 107 and 98, 288
    // and 271, 233 and 212; 20 x 768^2 111 and 103, 256 and 245, 205 and 185)
    using SlmOnly = FixedKinds<XL_OP_PHASE>;
    using LcdOnly = FixedKinds<XL_OP_LCD>;
    using SlmsOnly = FixedKinds<XL_OP_SSLM>;
    if (p.pol) return LcdOnly::matches(p.pre) ? launch_rows_fwd_b<R, 4, LcdOnly>(st, p) : launch_rows_fwd_b<R, 4>(st, p);
    if (p.cout == 1) return SlmOnly::matches(p.pre) ? launch_rows_fwd_b<R, 1, SlmOnly>(st, p) : launch_rows_fwd_b<R, 1>(st, p);
    if (p.cin == 2) return SlmsOnly::matches(p.pre) ? launch_rows_fwd_b<R, 2, SlmsOnly>(st, p) : launch_rows_fwd_b<R, 2>(st, p);
    return launch_rows_fwd_b<R, 3>(st, p);
  }
  if (p.pol) {
    RsLaunch q = p;
    q.B = 2 * p.B;
    return launch_rows_inv_b<R, 1, false, true>(st, q);
  }
  const bool epi = p.post.nops > 0 || (p.adjoint && p.cout == 3);
  if (p.cout == 1) return epi ? launch_rows_inv_b<R, 1, true>(st, p) : launch_rows_inv_b<R, 1, false>(st, p);
  return epi ? launch_rows_inv_b<R, 3, true>(st, p) : launch_rows_inv_b<R, 3, false>(st, p);
}

template <int R> int rs_blk_cols(cudaStream_t st, const RsLaunch& p) {
  RsLaunch q = p;
  if (p.pol) q.cout = 2;
  return launch_cols_b<R>(st, q);
}

template <int R>
int rs_blk_hhat_rows(cudaStream_t st, int ny, int nx, int py, const double* offx, const double* offy, int q2, double z,
                     const double* zp, double wavelength, int dz, float2* off, float2* out) {
  using F = BlkFft<R>;
  using K = RowB<R, 1>;
  rs_split_offsets_b<<<(F::P + py + 255) / 256, 256, 0, st>>>(offx, offy, q2, F::P, py, off);
  XL_CHECK_LAUNCH("rs_split_offsets_b");
  const size_t sm = ((size_t)F::NTB + K::LINES * F::LINE) * 8;
  const float k = (float)(2.0 * M_PI / wavelength);
  int per_sm;
  auto run = [&](auto kernel, int rc) {
    if (rc) return rc;
    kernel<<<py / K::G, K::THREADS, sm, st>>>(ny, nx, py, off, z, zp, 1.0 / wavelength, k, out);
    XL_CHECK_LAUNCH("rs_hhat_rows_b");
    return (int)XL_OK;
  };
  if (dz) return run(rs_hhat_rows_b<R, true>, launch_ready<rs_hhat_rows_b<R, true>>(K::THREADS, sm, &per_sm, "rs_hhat_rows_b"));
  return run(rs_hhat_rows_b<R, false>, launch_ready<rs_hhat_rows_b<R, false>>(K::THREADS, sm, &per_sm, "rs_hhat_rows_b"));
}

template <int R> int rs_blk_hhat_cols(cudaStream_t st, const float2* in, int px, float scale, float2* out) {
  return launch_hhat_cols_b<R>(st, in, px, scale, out);
}

}  // namespace xl

#define XL_RS_BLK_INSTANTIATE(R)                                                                             \
  template int xl::rs_blk_rows<R>(cudaStream_t, const RsLaunch&, bool);                                      \
  template int xl::rs_blk_cols<R>(cudaStream_t, const RsLaunch&);                                            \
  template int xl::rs_blk_hhat_rows<R>(cudaStream_t, int, int, int, const double*, const double*, int, double, \
                                       const double*, double, int, float2*, float2*);                        \
  template int xl::rs_blk_hhat_cols<R>(cudaStream_t, const float2*, int, float, float2*);
