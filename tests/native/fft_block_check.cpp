// CPU harness for the in-place block FFT engine: the threads of one line run
// one after the other, phase by phase, on the shared-memory layout the kernels
// use.  Built by tests/test_fft_block_cpu.py with g++ and called through ctypes.
#include <algorithm>
#include <cmath>
#include <vector>

#include "../../xlumina_gb300/csrc/fft_block.cuh"

using namespace xl;

// The phase A twiddles of thread t, four at a time, as the kernels pass them.
template <int R> struct Tw {
  const float2* tw;
  void operator()(int i, int q, float2 (&w)[4]) const {
    for (int n = 0; n < 4; ++n)
      if (4 * q + n > 0 && 4 * q + n < R) w[n] = tw[(4 * q + n - 1) * 256 + i * BlkFft<R>::T];
  }
};

// Forward transform of in (P complex) to out in natural frequency order, then
// the inverse of that back to `back` (scaled by P); zu: the upper half of the
// input is taken as zero and not read.
template <int R> static void run(int zu, const float2* in, float2* out, float2* back) {
  using F = BlkFft<R>;
  std::vector<float2> tw(F::NTW);
  std::vector<float4> smem(F::LINE / 2);
  blk_twiddles<R>(tw.data());
  float2* line = (float2*)smem.data();
  for (int t = 0; t < F::T; ++t) {
    float2 v[16];
    for (int i = 0; i < F::IPT; ++i)
      for (int n = 0; n < R; ++n) v[i * R + n] = in[t + i * F::T + 256 * n];
    if (zu) blk_a_fwd<R, -1, true>(v, t, line, Tw<R>{tw.data() + t});
    else blk_a_fwd<R, -1, false>(v, t, line, Tw<R>{tw.data() + t});
  }
  float2 v[16];
  for (int t = 0; t < F::TB; ++t) blk_b_fwd<-1>(v, t & 15, line + (t >> 4) * F::BLK, tw.data() + F::NTA);
  for (int t = 0; t < F::TB; ++t) {
    float2* blk = line + (t >> 4) * F::BLK;
    blk_c_fwd<-1>(v, t & 15, blk);
    for (int m = 0; m < 16; ++m) out[blk_freq<R>(t >> 4, t & 15, m)] = v[m];
    blk_c_inv<1>(v, t & 15, blk);
  }
  for (int t = 0; t < F::TB; ++t) blk_b_inv<1>(v, t & 15, line + (t >> 4) * F::BLK, tw.data() + F::NTA);
  for (int t = 0; t < F::T; ++t) {
    blk_a_inv<R, 1>(v, t, line, Tw<R>{tw.data() + t});
    for (int i = 0; i < F::IPT; ++i)
      for (int n = 0; n < R; ++n) back[t + i * F::T + 256 * n] = v[i * R + n];
  }
}

extern "C" int fft_block_check(int r, int zu, const float* in, float* out, float* back) {
  const float2* a = (const float2*)in;
  float2 *o = (float2*)out, *b = (float2*)back;
  switch (r) {
    case 4: run<4>(zu, a, o, b); return 0;
    case 6: run<6>(zu, a, o, b); return 0;
    case 8: run<8>(zu, a, o, b); return 0;
    case 10: run<10>(zu, a, o, b); return 0;
    case 12: run<12>(zu, a, o, b); return 0;
    case 14: run<14>(zu, a, o, b); return 0;
    case 16: run<16>(zu, a, o, b); return 0;
  }
  return -1;
}

// Bank conflicts of the three access patterns: the most lanes of one half-warp
// (8-byte accesses, 16 bank pairs) or quarter-warp (16-byte accesses, 8 bank
// quads) that fall on one bank, over every access of a warp; `cols` columns
// interleave in phase A's lanes, lines `stride` slots apart.
extern "C" int fft_block_conflicts(int cols, int stride) {
  int worst = 0;
  auto half = [&](const int* slot) {
    for (int h = 0; h < 2; ++h) {
      int n[16] = {0};
      for (int i = 0; i < 16; ++i) worst = std::max(worst, ++n[slot[16 * h + i] & 15]);
    }
  };
  int s[32];
  for (int j = 0; j + 32 / cols <= 256; j += 32 / cols) {
    for (int i = 0; i < 32; ++i) s[i] = (i % cols) * stride + blk_slot(j + i / cols);
    half(s);
  }
  for (int m = 0; m < 16; ++m) {
    for (int i = 0; i < 32; ++i) s[i] = (i >> 4) * 288 + (i & 15) + 18 * m;
    half(s);
  }
  for (int q = 0; q < 8; ++q)
    for (int g = 0; g < 4; ++g) {
      int n[8] = {0};
      for (int i = 0; i < 8; ++i) {
        const int l = (8 * g + i) & 15;
        worst = std::max(worst, ++n[((18 * l) / 2 + q) & 7]);
      }
    }
  return worst;
}
