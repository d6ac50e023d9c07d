// RS / VRS kernels on the in-place block FFT engine (fft_block.cuh), for
// transforms of P = 256 R points.
#pragma once

#include <type_traits>
#include "fft_block.cuh"
#include "line_fft.cuh"
#include "rs_host.h"

namespace xl {

// ---- the engine's twiddle tables in device memory, one after the other ----
__host__ __device__ constexpr int blk_tw_off(int r) {
  int o = 0;
  for (int q = 4; q < r; q += 2) o += (q - 1) * 256 + 240;
  return o;
}
constexpr int BLK_TW_TOTAL = blk_tw_off(18);
static __device__ float2 g_blk_tw[BLK_TW_TOTAL];

template <int R> __device__ __forceinline__ const float2* blk_tw() { return g_blk_tw + blk_tw_off(R); }

static cudaError_t blk_upload_twiddles(const float2*) {
  std::vector<float2> t(BLK_TW_TOTAL);
  blk_twiddles<4>(t.data() + blk_tw_off(4));
  blk_twiddles<6>(t.data() + blk_tw_off(6));
  blk_twiddles<8>(t.data() + blk_tw_off(8));
  blk_twiddles<10>(t.data() + blk_tw_off(10));
  blk_twiddles<12>(t.data() + blk_tw_off(12));
  blk_twiddles<14>(t.data() + blk_tw_off(14));
  blk_twiddles<16>(t.data() + blk_tw_off(16));
  return cudaMemcpyToSymbol(g_blk_tw, t.data(), sizeof(g_blk_tw));
}
static const bool blk_tw_registered = register_device_tables(&blk_upload_twiddles, nullptr);

// ---- Tensor Memory (tcgen05) as per-thread storage ----
// TMEM is 128 lanes x 512 columns of 32-bit cells per SM.  With the 32x32b
// access shape, thread i of warp w reads and writes lane 32 (w mod 4) + i, so
// each thread owns its own cells; a thread here has 64 consecutive columns of
// its lane (32 complex values).  One warp allocates the CTA's columns and
// hands the base address out through shared memory; the same warp frees them
// before the CTA exits.
__device__ __forceinline__ void tmem_alloc(unsigned* dst_smem, unsigned ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// four complex values into this thread's cells [col, col + 8)
__device__ __forceinline__ void tmem_st4(unsigned taddr, float2 a, float2 b, float2 c, float2 d) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
               "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y), "f"(d.x), "f"(d.y)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// four complex values back; the values pass through the wait so that no use
// is scheduled before the load has completed
__device__ __forceinline__ void tmem_ld4(unsigned taddr, float2 (&o)[4]) {
  float r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7])
               : "r"(taddr)
               : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : "+f"(r[0]), "+f"(r[1]), "+f"(r[2]), "+f"(r[3]), "+f"(r[4]), "+f"(r[5]), "+f"(r[6]), "+f"(r[7])
               :
               : "memory");
#pragma unroll
  for (int i = 0; i < 4; ++i) o[i] = make_float2(r[2 * i], r[2 * i + 1]);
}

// Column CTAs: CW columns, interleaved in the lanes of phase A (a warp's load
// or store of a row is then a whole 32-byte sector), T threads each.
template <int R> struct RsColB {
  using F = BlkFft<R>;
  static constexpr int CW = 4, LPW = 32 / CW;
  static constexpr int THREADS = CW * F::T;
  static constexpr int MINB = 1024 / THREADS;
  static constexpr int LINE = F::LINE + 4;     // the CW columns of a half-warp on distinct banks
  static constexpr int WARPS_B = CW * R / 2;   // warps of phases B and C
  static constexpr bool TM = R > 8;            // Tensor Memory cells beside the registers
  static constexpr unsigned TM_COLS = THREADS / 128 * 64;
  static constexpr size_t SMEM = ((size_t)F::NTW + (size_t)CW * LINE) * 8;
};

// Where a thread of a column CTA works: column wc and index jt in phase A;
// column bc, block k1 and index l in phases B and C (warps below WARPS_B).
template <int R> struct ColMap {
  int wc, jt, warp, lane, bc, k1, l;
  __device__ __forceinline__ ColMap() {
    using K = RsColB<R>;
    const int tid = threadIdx.x;
    warp = tid >> 5;
    lane = tid & 31;
    wc = lane % K::CW;
    jt = warp * K::LPW + lane / K::CW;
    bc = (tid >> 4) % K::CW;
    k1 = (tid >> 4) / K::CW;
    l = tid & 15;
  }
};

// Column pass, in place on CW columns of a tile: FFT along y of the ny nonzero
// rows, multiply by the transfer spectrum (conjugate for the adjoint), inverse
// FFT, keep the ny surviving rows.  Persistent: CTAs walk the (batch entry,
// column group) units batch entries fastest, so that entries at the same
// distance read one spectrum tile together.  Spectra are stored in the order
// phase C holds them (rs_hhat_cols_b), so a warp reads 512 contiguous bytes.
// Phase A twiddles, four at a time, from this thread's Tensor Memory cells or
// from the table in shared memory.
template <int R> struct TmemTw {
  unsigned cell;
  static __device__ __forceinline__ unsigned at(int i, int q) { return (unsigned)(2 * (i * ((R + 3) / 4 * 4) + 4 * q)); }
  __device__ __forceinline__ void operator()(int i, int q, float2 (&w)[4]) const { tmem_ld4(cell + at(i, q), w); }
};
template <int R> struct SmemTw {
  const float2* tw;   // the table at the thread's j
  __device__ __forceinline__ void operator()(int i, int q, float2 (&w)[4]) const {
#pragma unroll
    for (int n = 0; n < 4; ++n)
      if (4 * q + n > 0 && 4 * q + n < R) w[n] = tw[(4 * q + n - 1) * 256 + i * BlkFft<R>::T];
  }
};

// Column pass, in place on CW columns of a tile: FFT along y of the ny nonzero
// rows, multiply by the transfer spectrum (conjugate for the adjoint), inverse
// FFT, keep the ny surviving rows.  Persistent: CTAs walk the (batch entry,
// column group) units batch entries fastest, so that entries at the same
// distance read one spectrum tile together.  Spectra are stored in the order
// phase C holds them (rs_hhat_cols_b), so a warp reads 512 contiguous bytes.
//
// What bounds it: the shared-memory pipe (60 % busy at 4096 points, the FP32
// pipe 48 %); without any of its global loads and stores it runs 16 % faster.
// So the CTAs of 1024 threads (R > 8) keep what a thread reads again and again
// in its own Tensor Memory cells, which are not on that pipe: the phase A
// twiddles (a thread's j never changes), and a unit's spectrum values for the
// second and third component.  8 x 2048^2 VRS: 1.50 ms with both, 1.58 ms
// without, 1.92 ms on the Stockham engine with its eight barriers a component.
// The smaller CTAs (R <= 8, several per SM) keep their tables in shared
// memory: with Tensor Memory they ran a third slower (16 x 1024^2 scalar: 339
// against 250 us; Stockham 313 us).
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
  if constexpr (TM) {
    if (threadIdx.x < 32) tmem_alloc(&s_tmem, K::TM_COLS);
    tmem_fence_before_sync();
  }
  __syncthreads();
  unsigned cell = 0;   // lane 32 (warp mod 4) + lane, 64 columns per warp of a lane quarter
  if constexpr (TM) {
    tmem_fence_after_sync();
    cell = s_tmem + ((32u * ((unsigned)m.warp & 3u)) << 16) + (unsigned)(m.warp >> 2) * 64u;
#pragma unroll
    for (int i = 0; i < F::IPT; ++i)
#pragma unroll
      for (int q = 0; q < (R + 3) / 4; ++q) {
        float2 w[4] = {make_float2(1.f, 0.f), make_float2(1.f, 0.f), make_float2(1.f, 0.f), make_float2(1.f, 0.f)};
        SmemTw<R>{tw + m.jt}(i, q, w);
        tmem_st4(cell + TmemTw<R>::at(i, q), w[0], w[1], w[2], w[3]);
      }
    tmem_wait_st();
  }
  typename std::conditional<TM, TmemTw<R>, SmemTw<R>>::type twa;
  if constexpr (TM) twa.cell = cell;
  else twa.tw = tw + m.jt;
  const unsigned scell = cell + 32u;
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
    const float4* spec = (const float4*)sbase + (long long)g * (K::CW * F::P / 2) + m.warp * 256 + m.lane;
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
        const float4* sp = spec;
        asm volatile("" : "+l"(sp));   // the loads stay here: ahead of the transform they would hold 32 registers
        auto mul4 = [&](int q, const float2 (&w)[4]) {
#pragma unroll
          for (int i = 0; i < 4; ++i) v[4 * q + i] = p.adjoint ? cmulc(v[4 * q + i], w[i]) : cmul(v[4 * q + i], w[i]);
        };
        if (TM && c > 0) {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float2 w[4];
            tmem_ld4(scell + 8u * q, w);
            mul4(q, w);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 s = __ldg(sp + 2 * q * 32), t = __ldg(sp + (2 * q + 1) * 32);
            const float2 w[4] = {make_float2(s.x, s.y), make_float2(s.z, s.w), make_float2(t.x, t.y),
                                 make_float2(t.z, t.w)};
            if (TM && p.cout > 1) tmem_st4(scell + 8u * q, w[0], w[1], w[2], w[3]);
            mul4(q, w);
          }
          if (TM && p.cout > 1) tmem_wait_st();   // complete before the next component's loads
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
  if constexpr (TM) {
    // every thread is done with its cells before the allocating warp frees them
    tmem_fence_before_sync();
    __syncthreads();
    if (threadIdx.x < 32) {
      tmem_fence_after_sync();
      tmem_dealloc(s_tmem, K::TM_COLS);
    }
  }
}

// Transfer spectrum, column transforms of the row spectra (`in`: P rows of px
// columns), times `scale`, stored per group of CW columns in the order phase
// C of the column pass holds them: [group][warp][register pair][lane][2].
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
  float4* dst = (float4*)out + (long long)blockIdx.x * (K::CW * F::P / 2) + m.warp * 256 + m.lane;
#pragma unroll
  for (int q = 0; q < 8; ++q)
    dst[q * 32] = make_float4(v[2 * q].x * scale, v[2 * q].y * scale, v[2 * q + 1].x * scale, v[2 * q + 1].y * scale);
}

template <int R> static int launch_cols_b(cudaStream_t st, const RsLaunch& p) {
  using K = RsColB<R>;
  cudaError_t e = allow_smem(rs_cols_b<R>, K::SMEM);
  if (e != cudaSuccess) return cuda_fail(e, "rs_cols_b smem");
  const int grid = persistent_grid(rs_cols_b<R>, K::THREADS, K::SMEM, p.B * (p.px / K::CW));
  rs_cols_b<R><<<grid, K::THREADS, K::SMEM, st>>>(p);
  XL_CHECK_LAUNCH("rs_cols_b");
  return XL_OK;
}

template <int R> static int launch_hhat_cols_b(cudaStream_t st, const float2* in, int px, float scale, float2* out) {
  using K = RsColB<R>;
  cudaError_t e = allow_smem(rs_hhat_cols_b<R>, K::SMEM);
  if (e != cudaSuccess) return cuda_fail(e, "rs_hhat_cols_b smem");
  rs_hhat_cols_b<R><<<px / K::CW, K::THREADS, K::SMEM, st>>>(in, px, scale, out);
  XL_CHECK_LAUNCH("rs_hhat_cols_b");
  return XL_OK;
}

}  // namespace xl
