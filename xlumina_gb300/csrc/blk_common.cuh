// Pieces shared by the kernels on the in-place block FFT engine (RS / VRS,
// rs_blk.cuh, and chirp-z, czt_blk.cuh): its twiddle tables in device memory,
// Tensor Memory as per-thread storage, and the thread organisation of row and
// column CTAs.
#pragma once

#include <vector>

#include "fft_block.cuh"
#include "line_fft.cuh"

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
//
// The 32 lanes of a warp have to execute each of these instructions together,
// and they are called behind code whose branches depend on the lane (the guards
// of a ragged edge, a strided loop's last round), so each brings the lanes
// together itself.  `first` false leaves that out where the lanes came together
// before (at another of these, a barrier or a __syncwarp) and no branch on the
// lane has been taken since: with it at every one 8 x 2048^2 VRS takes 2490 us
// and one 4096^2 1569, as it is 2476 and 1539, without any 2478 and 1544.
__device__ __forceinline__ void tmem_alloc(unsigned* dst_smem, unsigned ncols) {
  __syncwarp();
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst_smem)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(unsigned taddr, unsigned ncols) {
  __syncwarp();
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tmem_fence_before_sync() {
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}
__device__ __forceinline__ void tmem_fence_after_sync() {
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}
// four complex values into this thread's cells [col, col + 8)
__device__ __forceinline__ void tmem_st4(unsigned taddr, float2 a, float2 b, float2 c, float2 d,
                                         bool first = true) {
  if (first) __syncwarp();
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr),
               "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y), "f"(d.x), "f"(d.y)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st(bool first = true) {
  if (first) __syncwarp();
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// four complex values back; the values pass through the wait so that no use
// is scheduled before the load has completed
__device__ __forceinline__ void tmem_ld4(unsigned taddr, float2 (&o)[4], bool first = true) {
  float r[8];
  if (first) __syncwarp();
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
// or store of a row is then whole 32-byte sectors), T threads each.  CW = 8
// fills a CTA of 1024 threads where a line takes 128 (8 x 1024^2 VRS adjoint:
// 378 us, with two CTAs of 4 columns an SM 403); where a line takes 64, four
// CTAs of 4 columns an SM are the better form (16 x 500^2 VRS: 184 us, two of
// 8 columns 193).
template <int R> struct RsColB {
  using F = BlkFft<R>;
  static constexpr int CW = F::T == 128 ? 8 : 4, LPW = 32 / CW;
  static constexpr int THREADS = CW * F::T;
  static constexpr int MINB = 1024 / THREADS;
  static constexpr int LINE = F::LINE + 16 / CW;   // the CW columns of a half-warp on distinct banks
  static constexpr int WARPS_B = CW * R / 2;   // warps of phases B and C
  static constexpr bool TM = MINB == 1;        // Tensor Memory cells beside the registers
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

// Phase A twiddles, four at a time, from this thread's Tensor Memory cells or
// from the table in shared memory.
template <int R> struct TmemTw {
  unsigned cell;
  static __device__ __forceinline__ unsigned at(int i, int q) { return (unsigned)(2 * (i * ((R + 3) / 4 * 4) + 4 * q)); }
  __device__ __forceinline__ void operator()(int i, int q, float2 (&w)[4]) const {
    tmem_ld4(cell + at(i, q), w, i == 0 && q == 0);   // nothing between a phase's reads branches
  }
};
template <int R> struct SmemTw {
  const float2* tw;   // the table at the thread's j
  __device__ __forceinline__ void operator()(int i, int q, float2 (&w)[4]) const {
#pragma unroll
    for (int n = 0; n < 4; ++n)
      if (4 * q + n > 0 && 4 * q + n < R) w[n] = tw[(4 * q + n - 1) * 256 + i * BlkFft<R>::T];
  }
};

// Thread organisation for NC transformed components: CG component groups of G
// lines of T threads, where CG = NC (every component of a row transformed at
// once) when the CTA can hold them, else 1 (one after the other).
template <int R, int NC> struct RowB {
  using F = BlkFft<R>;
  static constexpr int G = 256 / F::T > 1 ? 256 / F::T : 1;
  static constexpr int CG = (NC * G * F::T <= 1024) ? NC : 1;
  static constexpr int LINES = CG * G;
  static constexpr int THREADS = LINES * F::T;
  static constexpr int MINB = (768 / THREADS) > 1 ? (768 / THREADS) : 1;   // resident CTAs per SM
  static constexpr bool TM = MINB == 1;       // phase A twiddles in Tensor Memory
};

// Phase A twiddles of a row thread: the table in global memory, the same
// entries on every row.
template <int R> struct GlobalTw {
  const float2* tw;   // the table at the thread's j
  __device__ __forceinline__ void operator()(int i, int q, float2 (&w)[4]) const {
#pragma unroll
    for (int n = 0; n < 4; ++n)
      if (4 * q + n > 0 && 4 * q + n < R) w[n] = __ldg(tw + (4 * q + n - 1) * 256 + i * BlkFft<R>::T);
  }
};

// The same entries in Tensor Memory: allocates CELLS cells a thread for a CTA of
// THREADS threads, fills the first 32 and returns the thread's first cell.
template <int THREADS, unsigned CELLS> constexpr unsigned tmem_columns() {
  unsigned n = 32;
  while (n < (THREADS + 127) / 128 * CELLS) n *= 2;
  return n;
}
template <int R, int THREADS, unsigned CELLS, class TW> __device__ __forceinline__ unsigned tmem_twiddles(unsigned* s_tmem, const TW& tw) {
  const int warp = threadIdx.x >> 5;
  if (threadIdx.x < 32) tmem_alloc(s_tmem, tmem_columns<THREADS, CELLS>());
  tmem_fence_before_sync();
  __syncthreads();
  tmem_fence_after_sync();
  const unsigned cell = *s_tmem + ((32u * ((unsigned)warp & 3u)) << 16) + (unsigned)(warp >> 2) * CELLS;
#pragma unroll
  for (int i = 0; i < BlkFft<R>::IPT; ++i)
#pragma unroll
    for (int q = 0; q < (R + 3) / 4; ++q) {
      float2 w[4] = {make_float2(1.f, 0.f), make_float2(1.f, 0.f), make_float2(1.f, 0.f), make_float2(1.f, 0.f)};
      tw(i, q, w);
      tmem_st4(cell + TmemTw<R>::at(i, q), w[0], w[1], w[2], w[3], i == 0 && q == 0);
    }
  tmem_wait_st(false);
  return cell;
}
// Frees them once every thread is done with its cells.
template <int THREADS, unsigned CELLS> __device__ __forceinline__ void tmem_release(unsigned base) {
  tmem_fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) {
    tmem_fence_after_sync();
    tmem_dealloc(base, tmem_columns<THREADS, CELLS>());
  }
}

}  // namespace xl
