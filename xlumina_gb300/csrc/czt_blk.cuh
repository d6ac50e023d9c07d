// Chirp-z x and y transforms on the in-place block FFT engine (fft_block.cuh),
// for Bluestein lengths of 256 R points: the kernels and their launch code,
// included by the czt_b*.cu translation units.  What they compute is stated in
// czt_kernels.cuh, which has the shorter and longer lengths.
//
// A line is chirped, transformed, multiplied by the chirp's spectrum g in the
// order phase C holds it, transformed back and chirped again, so the two
// transforms of a line share two CTA barriers.  The length is the shortest
// 256 R that holds the window (2048 onto 1024 samples: 3072 points where a
// power of two would be 4096).
//
// What bounds them: the x transform its fused prologue (the issue rate is 47 to
// 51 %; without the phases between the two barriers 8 x 2048^2 high-NA tables
// took 666 of 780 us, without sines and cosines 686), the y transform the latency
// of a column's loads in a CTA that has its SM to itself (issue rate 48 to 50 %,
// shared-memory pipe 33 to 39 %, DRAM 10 %).  Measured, x and y transform (us;
// Stockham engine before): 4 x 2048^2 -> 1024^2 full focus 628 and 263 (888 and
// 288), 8 of its Ez alone 740 and 184 (845 and 208), their adjoint 158 and 283
// (196 and 420); 16 x 1024^2 -> 512^2 behind a lens 217 and 88 (295 and 103),
// adjoint 85 and 176 (117 and 221), with a distance for each entry 320 and 133
// (438 and 140); 2 x 1500^2 -> 301^2 VCZT 172 and 29 (216 and 31).
#pragma once

#include <math.h>

#include <type_traits>

#include "czt_host.h"
#include "blk_common.cuh"

namespace xl {

// The chirp spectrum's values of a thread, register m at frequency
// blk_freq(k1, k2, m): in Tensor Memory cells (CTAs that have an SM to
// themselves), else read in block order, [m][thread of phase C], from the
// caller's vector or, where that is in natural order, from a copy in shared
// memory.
template <int R> struct TmemG {
  unsigned cell;
  __device__ __forceinline__ void fill(const float2* g, bool natural, int k1, int k2) const {
    float2 w[16];
#pragma unroll
    for (int i = 0; i < 16; ++i)
      w[i] = __ldg(g + (natural ? blk_freq<R>(k1, k2, i) : i * BlkFft<R>::TB + 16 * k1 + k2));
#pragma unroll
    for (int q = 0; q < 4; ++q) tmem_st4(cell + 8u * q, w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3], q == 0);
    tmem_wait_st(false);
  }
  __device__ __forceinline__ void operator()(int q, float2 (&w)[4]) const { tmem_ld4(cell + 8u * q, w, false); }
};
template <int R> struct BlockG {
  const float2* g;   // + the thread's index in phase C
  __device__ __forceinline__ void operator()(int q, float2 (&w)[4]) const {
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = g[(4 * q + i) * BlkFft<R>::TB];
  }
};
// Shared-memory form of a spectrum: natural order in, [m][thread] out.
template <int R> __device__ __forceinline__ void smem_g_fill(float2* dst, const float2* g, int tid, int threads) {
  for (int i = tid; i < BlkFft<R>::P; i += threads) {
    const int tb = i % BlkFft<R>::TB, m = i / BlkFft<R>::TB;
    dst[i] = __ldg(g + blk_freq<R>(tb >> 4, tb & 15, m));
  }
}

// Thread organisation of the x transform: RowB's, with the CTAs per SM that
// the registers are sized for.  One component: three of 256 threads, but from
// 3072 points two (128 registers, and twice the room for staged planes) for a
// fixed program of several ops (the high-NA table's, 8 fields: 2048^2 -> 1024^2
// 738 us, with three CTAs 803; 1800^2 -> 1000^2 641, 635; 4 x 1600^2 -> 900^2, a
// step shorter, 276 with two, 224 with three).
template <int R, int NC, class FK = FixedKinds<>> struct CztRowB : RowB<R, NC> {
  static constexpr int MB = NC == 1 ? (FK::n > 1 && R >= 12 ? 2 : 3) : 1;
};

// Bytes of the x transform's shared memory before its stage.
template <int R, int NC> __host__ __device__ constexpr size_t czt_rows_fixed(int nx, bool natural, bool vczt) {
  using K = CztRowB<R, NC>;
  return ((size_t)(BlkFft<R>::NTB + K::LINES * BlkFft<R>::LINE +
                   (NC > 1 ? NC * K::G * nx : (natural ? BlkFft<R>::P : 0))) * 8 + (vczt ? (size_t)nx * 4 : 0) + 15) /
         16 * 16;
}

// x transform.  NC: components per row (1, or 3 for VCZT and the high-NA
// focus; a plain transform of 2 components runs as 3 with the third idle).
// One component: the thread that transforms an element runs the fused program
// for it itself; three: the prologue leaves the row's components in a buffer.
// FK: the fused program's op kinds fixed at compile time (FixedKinds<...>,
// for the tables' programs), or FixedKinds<>.
template <int R, int NC, class FK = FixedKinds<>>
__global__ void __launch_bounds__(CztRowB<R, NC, FK>::THREADS, CztRowB<R, NC, FK>::MB)
    czt_rows_b(const __grid_constant__ CztLaunch p, const __grid_constant__ RowStage st) {
  using F = BlkFft<R>;
  using K = CztRowB<R, NC>;
  constexpr bool TM = NC > 1;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned s_tmem;
  const int nx = p.nx, ny = p.ny;
  float2* twb = (float2*)smraw;                       // NTB
  float2* xch = twb + F::NTB;                         // LINES x LINE
  float2* post = xch + K::LINES * F::LINE;            // NC x G x nx; one component: a natural-order spectrum, P
  float* xf = (float*)(post + (size_t)NC * K::G * nx);   // nx (VCZT: x as float32)
  const bool vczt = p.mode == XL_CZT_VECTOR && !p.adjoint;
  const size_t soff = czt_rows_fixed<R, NC>(nx, p.nat_x, vczt);
  unsigned char* stage = smraw + soff;
  unsigned long long* mbar = (unsigned long long*)(stage + (size_t)K::G * st.row_bytes);
  const int tid = threadIdx.x;
  const int ln = tid / F::T, t = tid % F::T;
  const int cg = ln / K::G, gi = ln % K::G;
  const int ngb = (ny + K::G - 1) / K::G;
  const int total = p.B * ngb;
  const bool staged = st.n > 0;
  const bool fwd_phase = p.mode != XL_CZT_PLAIN;
  float2* line = xch + ln * F::LINE;
  float2* blk = line + (t >> 4) * F::BLK;
  const bool active = t < F::TB;
  const GlobalTw<R> twg{blk_tw<R>() + t};

  if (tid == 0 && staged) {
    mbar_init(mbar, 1);
    fence_mbar_init();
  }
  for (int i = tid; i < F::NTB; i += K::THREADS) twb[i] = blk_tw<R>()[F::NTA + i];
  if (NC > 1 && vczt)
    for (int i = tid; i < nx; i += K::THREADS) xf[i] = (float)p.x[i];
  typename std::conditional<TM, TmemTw<R>, GlobalTw<R>>::type twa;
  typename std::conditional<TM, TmemG<R>, BlockG<R>>::type gx;
  if constexpr (TM) {
    twa.cell = tmem_twiddles<R, K::THREADS, 64>(&s_tmem, twg);
    gx.cell = twa.cell + 32u;
    gx.fill(p.g_x, p.nat_x, active ? t >> 4 : 0, t & 15);
  } else {
    twa = twg;
    gx.g = (p.nat_x ? post : p.g_x) + t;
    if (p.nat_x) smem_g_fill<R>(post, p.g_x, tid, K::THREADS);
  }
  __syncthreads();
  // Row groups are taken batch entries fastest: CTAs that run together read the
  // same rows of planes shared by the batch (the lens coefficients, shared
  // masks), so those rows come from L2 after the first entry.  With chirps of
  // its own for every entry a CTA takes a run of one entry's groups instead, so
  // that the spectrum it holds changes once or twice.
  const int per = (total + (int)gridDim.x - 1) / (int)gridDim.x;
  const int first = p.zb ? (int)blockIdx.x * per : (int)blockIdx.x;
  const int last = p.zb ? min(first + per, total) : total;
  const int step = p.zb ? 1 : (int)gridDim.x;
  auto entry_of = [&](int grp) { return p.zb ? grp / ngb : grp % p.B; };
  auto row_of = [&](int grp) { return (p.zb ? grp % ngb : grp / p.B) * K::G; };
  auto issue = [&](int grp) {
    const int b = entry_of(grp), r0 = row_of(grp);
    if (staged) stage_rows(st, stage, mbar, b, r0, min(K::G, ny - r0));
    prefetch_rows(st, b, r0, min(K::G, ny - r0));
  };
  if (tid == 0 && first < last) issue(first);

  unsigned phase = 0;
  // the copy may still be in flight: let it land, record the event and leave
  // without issuing another
  auto timed_out = [&]() {
    mbar_wait_bounded(mbar, phase);
    if (tid == 0) record_timeout();
    if constexpr (TM) tmem_release<K::THREADS, 64>(s_tmem);
  };
  auto next_stage = [&](int grp) {
    phase ^= 1u;
    if (tid == 0 && grp + step < last) {
      if (staged) fence_proxy_async();
      issue(grp + step);
    }
  };
  int held = 0;   // entry whose spectrum is held
  for (int grp = first; grp < last; grp += step) {
    const int b = entry_of(grp);
    const int r0 = row_of(grp);
    const double zd = p.zb ? p.zb[b] : p.z;
    const float zf = (float)zd;
    if (p.zb && b != held) {
      held = b;
      if constexpr (TM) {
        gx.fill(p.g_x + (long long)b * F::P, true, active ? t >> 4 : 0, t & 15);
      } else {
        __syncthreads();
        smem_g_fill<R>(post, p.g_x + (long long)b * F::P, tid, K::THREADS);
        __syncthreads();
      }
    }
    // a wait that runs out is acted on at the barrier after the prologue
    // (the prologue then works on stale data, and the launch's output is not
    // valid), so that no extra barrier is taken per row group
    const bool got = !staged || mbar_wait_bounded(mbar, phase, g_wait_limit_ns);
    const int r = r0 + gi;
    const bool live = r < ny;
    const int c = cg;
    const bool act = live && c < p.cout;
    RsGeom geo;          // where no plane of F is at hand: its constants, with Y^2 of
    int geo_row = -1;    // this row added to z^2 (float64 splits, once a row)
    // the fused program, the VCZT Ez and the input-plane transfer function on
    // NPX pixels: (row of the group, column) of pixel q from at(q), results to
    // put(q, e)
    auto pixels = [&](auto npx, auto at, auto put) {
      constexpr int NPX = decltype(npx)::value;
      float2 e[NPX][3];
      PixelCtx px[NPX];
      StagedParams pr[NPX];
#pragma unroll
      for (int q = 0; q < NPX; ++q) {
        int g2, n;
        at(q, g2, n);
        const long long pix = (long long)(r0 + g2) * nx + n;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          e[q][i] = make_float2(0.f, 0.f);
          if (i < p.cin) {
            const int fo = st.fld[i];
            e[q][i] = fo >= 0 ? ((const float2*)(stage + fo))[g2 * nx + n] : p.in[i][(long long)b * p.ibs + pix];
          }
        }
        px[q] = PixelCtx{r0 + g2, n, pix, b};
        pr[q] = StagedParams{stage, &st, g2, nx, n};
      }
      if constexpr (FK::n > 0) apply_prog_fixed<FK>(p.pre, e, px, pr);
      else if (p.pre.nops) apply_prog_vec<NPX>(p.pre, e, px, pr);
#pragma unroll
      for (int q = 0; q < NPX; ++q) {
        if (fwd_phase) {
          const int rr = px[q].row, n = px[q].col;
          if constexpr (NC > 1) {
            if (vczt) {  // vectorized_optics.py:340-344
              const float X = xf[n], Y = (float)p.y[rr];
              const float d = sqrtf(X * X + Y * Y + zf * zf);
              e[q][2] = cscale(cadd(cscale(e[q][0], X / d), cscale(e[q][1], Y / d)), zf / d);
            }
          }
          // wave_optics.py:341 (F on the input plane); the adjoint applies conj(F0) here
          float2 Fv;
          if (st.aux >= 0) {
            Fv = ((const float2*)(stage + st.aux))[(rr - r0) * nx + n];
          } else if (p.fin) {
            Fv = p.fin[px[q].pix];
          } else {
            if (rr != geo_row) {
              geo_row = rr;
              geo = rs_geom(zd, ffloat{p.invl_hi, p.invl_lo}, p.k);
              const ffloat Y = ff_split(p.y[rr]);
              geo.z2 = ff_add(geo.z2, ff_mul(Y, Y));
            }
            const ffloat X = ff_split(p.x[n]);
            Fv = rs_value_s(geo, ff_add(geo.z2, ff_mul(X, X)));
          }
          if (p.adjoint) Fv = cconj(Fv);
#pragma unroll
          for (int i = 0; i < 3; ++i) e[q][i] = cmul(e[q][i], Fv);
        }
        put(q, e[q]);
      }
    };
    const float2* pre_x = czt_entry(p.pre_x, p, b, nx);
    float2 v[16];
    if constexpr (NC == 1) {
      // this thread's elements, NP at a time, through its own slots of the
      // line (no barrier).  Few, since the fused program's code is laid out once
      // for each and the instruction cache is what bounds it (8 x 2048^2 high-NA
      // tables: 8 at a time 910 us, 4 780, 2 762, 1 796; unrolled over all, with
      // the results in registers, 1181; 16 x 1024^2 behind a lens: 4 253, 2 221).
      // Its j-th element is at t + T j: those inside the window, j0 to j1, follow
      // each other; one past the end takes a valid pixel.
      const int g2 = min(gi, ny - 1 - r0);
      constexpr int N = F::IPT * R, NP = 2;
      float2* own = line + blk_slot(t);
      const int at0 = t - p.ioff_x;   // position in the window of element 0
      const int j0 = at0 < 0 ? (F::T - 1 - at0) / F::T : 0;
      const int j1 = at0 < nx ? min((nx - 1 - at0) / F::T + 1, N) : 0;
#pragma unroll 1
      for (int j = j0; j < j1; j += NP) {
        pixels(std::integral_constant<int, NP>{},
               [&](int q, int& g, int& n) {
                 g = g2;
                 n = min(at0 + (j + q) * F::T, nx - 1);
               },
               [&](int q, const float2 (&e)[3]) {
                 const int f = j + q;
                 if (f < j1) own[f / F::IPT * F::BLK + f % F::IPT * (F::T / 16) * 18] = e[0];
               });
      }
#pragma unroll
      for (int f = 0; f < N; ++f) {
        const int n = at0 + f / R * F::T + 256 * (f % R);
        v[f] = (act && n >= 0 && n < nx) ? cmul(own[f % R * F::BLK + f / R * (F::T / 16) * 18], __ldg(pre_x + n))
                                         : make_float2(0.f, 0.f);
      }
    } else {
      const int lim = min(K::G, ny - r0) * nx;
      for (int base = tid; base < lim; base += K::THREADS)
        pixels(std::integral_constant<int, 1>{},
               [&](int, int& g, int& n) {
                 g = K::G == 1 ? 0 : base / nx;
                 n = base - g * nx;
               },
               [&](int, const float2 (&e)[3]) {
#pragma unroll
                 for (int i = 0; i < NC; ++i) post[(i * K::G) * nx + base] = e[i];
               });
      // every thread has read the stage and written its pixels; every thread
      // takes the timeout branch or none does
      if (__syncthreads_or(!got)) return timed_out();
      next_stage(grp);
      const float2* src = post + (c * K::G + gi) * nx;
#pragma unroll
      for (int f = 0; f < F::IPT * R; ++f) {
        const int n = t + f / R * F::T + 256 * (f % R) - p.ioff_x;
        v[f] = (act && n >= 0 && n < nx) ? cmul(src[n], __ldg(pre_x + n)) : make_float2(0.f, 0.f);
      }
    }
    blk_a_fwd<R, -1, false>(v, t, line, twa);
    if constexpr (NC == 1) {
      if (__syncthreads_or(!got)) return timed_out();
      next_stage(grp);
    } else {
      __syncthreads();
    }
    if (active) {
      blk_b_fwd<-1>(v, t & 15, blk, twb);
      __syncwarp();
      blk_c_fwd<-1>(v, t & 15, blk);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        float2 w[4];
        gx(q, w);
#pragma unroll
        for (int i = 0; i < 4; ++i) v[4 * q + i] = cmul(v[4 * q + i], w[i]);
      }
      blk_c_inv<1>(v, t & 15, blk);
      __syncwarp();
      blk_b_inv<1>(v, t & 15, blk, twb);
    }
    __syncthreads();
    blk_a_inv<R, 1>(v, t, line, twa);
    if (act) {
      float2* plane = p.work + ((long long)b * p.cout + c) * ny * p.mxp;
      const float2* post_x = czt_entry(p.post_x, p, b, p.mx);
#pragma unroll
      for (int f = 0; f < F::IPT * R; ++f) {
        const int o = t + f / R * F::T + 256 * (f % R) - p.ooff_x;
        if (o >= 0 && o < p.mx) plane[tiled_rt(r, o, ny, p.lw)] = cmul(v[f], __ldg(post_x + o));
      }
    }
  }
  if constexpr (TM) tmem_release<K::THREADS, 64>(s_tmem);
}

// y transform over groups of CW columns, with the epilogue.  Persistent: CTAs
// walk the (column group, batch entry) units, groups fastest, a unit's
// components one after the other; cu > 1: a unit for each component, where
// there are few of them.  VALUE: the transfer function F0 is evaluated at each
// output sample (a distance of its own for every entry, or a first call, which
// has no plane of it yet); its code and registers stay out of the other kernel
// (16 x 1024^2 -> 512^2 adjoint: 176 us, one kernel for both 194; with a distance
// for each entry 133).
template <int R, bool VALUE>
__global__ void __launch_bounds__(RsColB<R>::THREADS, RsColB<R>::MINB) czt_cols_b(const __grid_constant__ CztLaunch p, int cu) {
  using F = BlkFft<R>;
  using K = RsColB<R>;
  constexpr bool TM = K::TM;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned s_tmem;
  float2* tw = (float2*)smraw;               // NTW
  float2* xch = tw + F::NTW;                 // CW x LINE
  float2* gs = xch + K::CW * K::LINE;        // a natural-order spectrum, P (no Tensor Memory)
  const ColMap<R> m;
  const int tid = threadIdx.x;
  for (int i = tid; i < F::NTW; i += K::THREADS) tw[i] = blk_tw<R>()[i];
  const bool active = m.warp < K::WARPS_B;
  const SmemTw<R> tws{tw + m.jt};
  typename std::conditional<TM, TmemTw<R>, SmemTw<R>>::type twa;
  typename std::conditional<TM, TmemG<R>, BlockG<R>>::type gy;
  auto hold = [&](int b) {   // the spectrum of entry b
    const float2* g = czt_entry(p.g_y, p, b, F::P);
    if constexpr (TM) gy.fill(g, p.nat_y, active ? m.k1 : 0, m.l);
    else if (p.nat_y) smem_g_fill<R>(gs, g, tid, K::THREADS);
  };
  if constexpr (TM) {
    __syncthreads();
    twa.cell = tmem_twiddles<R, K::THREADS, 64>(&s_tmem, tws);
    gy.cell = twa.cell + 32u;
  } else {
    twa = tws;
    gy.g = (p.nat_y ? gs : p.g_y) + m.k1 * 16 + m.l;
  }
  hold(0);
  __syncthreads();
  float2* line = xch + m.wc * K::LINE;
  float2* blk = xch + m.bc * K::LINE + m.k1 * F::BLK;
  const float2* twb = tw + F::NTA;
  const bool fold = p.adjoint && p.mode == XL_CZT_VECTOR;
  const int ny = p.ny, lw = p.lw;
  const int groups = (p.mx + K::CW - 1) / K::CW;
  const int units = groups * cu * p.B;
  // with chirps of its own for every entry a CTA takes a run of units, so that
  // the spectrum it holds changes once or twice
  const bool runs = VALUE && p.zb;
  const int per = (units + (int)gridDim.x - 1) / (int)gridDim.x;
  const int first = runs ? (int)blockIdx.x * per : (int)blockIdx.x;
  const int last = runs ? min(first + per, units) : units, step = runs ? 1 : (int)gridDim.x;
  int held = 0;
#pragma unroll 1
  for (int u = first; u < last; u += step) {
    const int g = u % groups, b = u / groups / cu;
    const int c0 = cu > 1 ? u / groups % cu : 0, c1 = cu > 1 ? c0 + 1 : p.cout;
    const int col = g * K::CW + m.wc;
    const bool live = col < p.mx;
    const double zd = p.zb ? p.zb[b] : p.z;
    const float zf = (float)zd;
    const float2* pre_y = czt_entry(p.pre_y, p, b, ny);
    const float2* post_y = czt_entry(p.post_y, p, b, p.my);
    if (p.zb && b != held) {
      held = b;
      if constexpr (!TM) __syncthreads();
      hold(b);
      if constexpr (!TM) __syncthreads();
    }
    float2 cte = p.cte;
    if (p.cteb) {
      cte = p.cteb[b];
      if (p.adjoint) cte.y = -cte.y;
    }
#pragma unroll 1
    for (int c = c0; c < c1; ++c) {
      const float2* tile = p.work + ((long long)b * p.cout + c) * ny * p.mxp + (((long long)(col >> lw) * ny) << lw) +
                           (col & ((1 << lw) - 1));
      float2 v[16];
#pragma unroll
      for (int f = 0; f < F::IPT * R; ++f) {
        const int n = m.jt + f / R * F::T + 256 * (f % R) - p.ioff_y;
        v[f] = (live && n >= 0 && n < ny) ? cmul(tile[(long long)n << lw], __ldg(pre_y + n)) : make_float2(0.f, 0.f);
      }
      blk_a_fwd<R, -1, false>(v, m.jt, line, twa);
      __syncthreads();
      if (active) {
        blk_b_fwd<-1>(v, m.l, blk, twb);
        __syncwarp();
        blk_c_fwd<-1>(v, m.l, blk);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          float2 w[4];
          gy(q, w);
#pragma unroll
          for (int i = 0; i < 4; ++i) v[4 * q + i] = cmul(v[4 * q + i], w[i]);
        }
        blk_c_inv<1>(v, m.l, blk);
        __syncwarp();
        blk_b_inv<1>(v, m.l, blk, twb);
      }
      __syncthreads();
      blk_a_inv<R, 1>(v, m.jt, line, twa);
      RsGeom geo;
      ffloat XX;
      if constexpr (VALUE) {
        geo = rs_geom(zd, ffloat{p.invl_hi, p.invl_lo}, p.k);
        const ffloat X = ff_split(p.xo[live ? col : 0]);
        XX = ff_mul(X, X);
      }
#pragma unroll
      for (int f = 0; f < F::IPT * R; ++f) {
        const int o = m.jt + f / R * F::T + 256 * (f % R) - p.ooff_y;
        if (!live || o < 0 || o >= p.my) continue;
        float2 val = cmul(v[f], __ldg(post_y + o));
        if (VALUE || p.mode != XL_CZT_PLAIN) {  // wave_optics.py:340, 355: F0 * U (adjoint: conj F)
          float2 Fv;
          if constexpr (VALUE) {
            const ffloat Y = ff_split(p.yo[o]);
            Fv = rs_value_s(geo, ff_add(ff_add(geo.z2, ff_mul(Y, Y)), XX));
          } else {
            Fv = p.fout[(long long)o * p.mx + col];
          }
          val = p.adjoint ? cmulc(val, Fv) : cmul(val, Fv);
        }
        val = cmul(val, cte);
        const long long pix = (long long)b * p.obs + (long long)o * p.mx + col;
        if (fold && c == 2) {  // adjoint of Ez = (Ex X/r + Ey Y/r) z/r, vectorized_optics.py:341-344
          const float X = (float)p.xo[col], Y = (float)p.yo[o];
          const float r2 = X * X + Y * Y + zf * zf;
          p.out[0][pix] = cadd(p.out[0][pix], cscale(val, X * zf / r2));
          p.out[1][pix] = cadd(p.out[1][pix], cscale(val, Y * zf / r2));
        } else {
          p.out[c][pix] = val;
        }
      }
    }
  }
  if constexpr (TM) tmem_release<K::THREADS, 64>(s_tmem);
}

// ---- launches ----

template <int R, int NC, class FK = FixedKinds<>> static int launch_czt_rows_b(cudaStream_t s, const CztLaunch& p) {
  using K = CztRowB<R, NC, FK>;
  const size_t fixed = czt_rows_fixed<R, NC>(p.nx, p.nat_x, p.mode == XL_CZT_VECTOR && !p.adjoint);
  // the stage takes what leaves room for the CTAs the registers allow; planes
  // that do not fit are read from global memory
  const size_t cap = (size_t)(227 * 1024) / K::MB - 1024;
  RowStage st;
  plan_row_stage(p.cin, p.in, p.ibs, p.nx, p.pre, K::G, fixed, st, cap, p.mode != XL_CZT_PLAIN ? p.fin : nullptr);
  const size_t sm = fixed + (size_t)K::G * st.row_bytes + 16;
  int per_sm;
  if (int rc = launch_ready<czt_rows_b<R, NC, FK>>(K::THREADS, sm, &per_sm, "czt_rows_b")) return rc;
  const int grid = persistent_grid(per_sm, p.B * ((p.ny + K::G - 1) / K::G));
  czt_rows_b<R, NC, FK><<<grid, K::THREADS, sm, s>>>(p, st);
  XL_CHECK_LAUNCH("czt_rows_b");
  return XL_OK;
}

template <int R> int czt_blk_rows(cudaStream_t s, const CztLaunch& p) {
  // programs that get a kernel with their op kinds fixed, at every length: an
  // sSLM before the high-NA lens; an LCD, an sSLM and the lens's Ez row; a thin
  // lens; a phase SLM.  Fixed against generic, rows in us at 1024, 1536, 2048,
  // 2560, .. points: sSLM and lens, 33 x 600^2 440 and 488, 14 x 900^2 490 and
  // 528, 7 x 1300^2 439 and 480, 4 x 1600^2 455 and 498 (4 x 2048^2 646 and 712);
  // the Ez row 320 and 380, 307 and 368, 330 and 392, 224 and 270; a thin lens
  // 170 and 185 at 1024 points, 134 and 153 for 2 x 2040^2 at 4096; a phase SLM
  // 150 and 169 at 1536, 132 and 153 at 4096.
  if (p.cout > 1) {
    using HighNa = FixedKinds<XL_OP_SSLM, XL_OP_HIGHNA>;
    if (HighNa::matches(p.pre)) return launch_czt_rows_b<R, 3, HighNa>(s, p);
    return launch_czt_rows_b<R, 3>(s, p);
  }
  using HighNaEz = FixedKinds<XL_OP_LCD, XL_OP_SSLM, XL_OP_HIGHNA_EZ>;
  using LensOnly = FixedKinds<XL_OP_SEPMASK>;
  using SlmOnly = FixedKinds<XL_OP_PHASE>;
  if (HighNaEz::matches(p.pre)) return launch_czt_rows_b<R, 1, HighNaEz>(s, p);
  if (LensOnly::matches(p.pre)) return launch_czt_rows_b<R, 1, LensOnly>(s, p);
  if (SlmOnly::matches(p.pre)) return launch_czt_rows_b<R, 1, SlmOnly>(s, p);
  return launch_czt_rows_b<R, 1>(s, p);
}

template <int R, bool VALUE> static int launch_czt_cols_b(cudaStream_t s, const CztLaunch& p) {
  using K = RsColB<R>;
  const size_t sm = K::SMEM + (!K::TM && p.nat_y ? (size_t)BlkFft<R>::P * 8 : 0);
  int per_sm;
  if (int rc = launch_ready<czt_cols_b<R, VALUE>>(K::THREADS, sm, &per_sm, "czt_cols_b")) return rc;
  // a unit for each component where there are fewer than two rounds of units
  // (2 x 301^2 VCZT outputs, 76 units for 152 SMs: 32 us, 41 without; 4 x
  // 1024^2, 512 units: 291 and 278), unless the VCZT adjoint folds one into the
  // others
  const long long units = (long long)p.B * ((p.mx + K::CW - 1) / K::CW);
  const bool fold = p.adjoint && p.mode == XL_CZT_VECTOR;
  const int cu = !fold && units < 2LL * per_sm * device_sms() ? p.cout : 1;
  czt_cols_b<R, VALUE><<<persistent_grid(per_sm, units * cu), K::THREADS, sm, s>>>(p, cu);
  XL_CHECK_LAUNCH("czt_cols_b");
  return XL_OK;
}

template <int R> int czt_blk_cols(cudaStream_t s, const CztLaunch& p) {
  return p.mode != XL_CZT_PLAIN && !p.fout ? launch_czt_cols_b<R, true>(s, p) : launch_czt_cols_b<R, false>(s, p);
}

}  // namespace xl

#define XL_CZT_BLK_INSTANTIATE(R)                                         \
  template int xl::czt_blk_rows<R>(cudaStream_t, const xl::CztLaunch&);   \
  template int xl::czt_blk_cols<R>(cudaStream_t, const xl::CztLaunch&);
