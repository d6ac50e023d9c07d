// Rayleigh-Sommerfeld propagation (scalar RS and vectorial VRS): the C ABI
// entry points.  The reference (wave_optics.py:281-289) zero-pads the N x N
// field to (2N-1)^2, multiplies fft2(U) by fft2(H) and crops [N-1:, N-1:];
// the kernels run the same linear convolution on a grid that holds it, in three
// passes: up to 256 pixels a side on the Stockham engine (rs_kernels.cuh), above
// on the block engine (rs_blk.cuh), axes above 2048 in two halves (rs_half.cuh).
#include <math.h>

#include <mutex>

#include "rs_host.h"

namespace xl {

// CALL(LOGQ) for the Stockham engine's lengths.
#define XL_RS_DISPATCH(LOGQ_VAR, CALL)          \
  switch (LOGQ_VAR) {                           \
    case 5: return CALL(5);                     \
    case 6: return CALL(6);                     \
    case 7: return CALL(7);                     \
    case 8: return CALL(8);                     \
    default: break;                             \
  }
// NAME<R>(args) of an axis of P points: 256 R, or two halves of 256 R.
#define XL_RS_BLK_DISPATCH(P, NAME, ...)                      \
  switch (P) {                                                \
    case 1024: return rs_blk_##NAME<4>(__VA_ARGS__);          \
    case 1536: return rs_blk_##NAME<6>(__VA_ARGS__);          \
    case 2048: return rs_blk_##NAME<8>(__VA_ARGS__);          \
    case 2560: return rs_blk_##NAME<10>(__VA_ARGS__);         \
    case 3072: return rs_blk_##NAME<12>(__VA_ARGS__);         \
    case 3584: return rs_blk_##NAME<14>(__VA_ARGS__);         \
    case 4096: return rs_blk_##NAME<16>(__VA_ARGS__);         \
    case 5120: return rs_half_##NAME<10>(__VA_ARGS__);        \
    case 6144: return rs_half_##NAME<12>(__VA_ARGS__);        \
    case 7168: return rs_half_##NAME<14>(__VA_ARGS__);        \
    case 8192: return rs_half_##NAME<16>(__VA_ARGS__);        \
    default: break;                                           \
  }

static int unsupported(const char* what) {
  set_error("%s: unsupported size", what);
  return XL_EUNSUPPORTED;
}

static int blk_rows(cudaStream_t st, const RsLaunch& p, bool inverse) {
  XL_RS_BLK_DISPATCH(p.px, rows, st, p, inverse)
  return unsupported("xl_rs_propagate");
}

static int blk_cols(cudaStream_t st, const RsLaunch& p) {
  XL_RS_BLK_DISPATCH(p.py, cols, st, p)
  return unsupported("xl_rs_propagate");
}

static int blk_propagate(cudaStream_t st, const RsLaunch& p, int stage) {
  for (int s = 0; s < 3; ++s) {
    if (stage >= 0 && s != stage) continue;
    if (int rc = s == 1 ? blk_cols(st, p) : blk_rows(st, p, s == 2)) return rc;
  }
  return XL_OK;
}

static int stockham_propagate(int lq, cudaStream_t st, const RsLaunch& p, int stage) {
#define CALL(L) rs_propagate<L>(st, p, stage)
  XL_RS_DISPATCH(lq, CALL)
#undef CALL
  return unsupported("xl_rs_propagate");
}

// One transfer spectrum.  `scale` is the caller's, for a 2 Q x 2 Q transform
// pair; shorter transforms take it times (2 Q)^2 / (px py).
static int spectrum(cudaStream_t st, int ny, int nx, const double* offx, const double* offy, double z,
                    const double* zp, double wavelength, double scale, float2* spec, float2* work, int dz) {
  const int lq = rs_logq(ny, nx);
  if (rs_is_blk(ny, nx)) {
    const int px = rs_px(ny, nx), py = rs_py(ny, nx), q2 = 2 << lq;
    auto rows = [&]() {
      XL_RS_BLK_DISPATCH(px, hhat_rows, st, ny, nx, py, offx, offy, q2, z, zp, wavelength, dz, spec, work)
      return unsupported("xl_rs_transfer_spectrum");
    };
    const float sc = (float)(scale * ((double)q2 * q2 / ((double)px * py)));
    auto cols = [&]() {
      XL_RS_BLK_DISPATCH(py, hhat_cols, st, work, px, sc, spec)
      return unsupported("xl_rs_transfer_spectrum");
    };
    if (int rc = rows()) return rc;
    return cols();
  }
#define CALL(L) rs_spectrum<L>(st, ny, nx, offx, offy, z, zp, wavelength, scale, spec, work, dz)
  XL_RS_DISPATCH(lq, CALL)
#undef CALL
  return unsupported("xl_rs_transfer_spectrum");
}

}  // namespace xl

using namespace xl;


extern "C" size_t xl_rs_spectrum_bytes(int ny, int nx) {
  if (ny < 2 || nx < 2 || ny > XL_MAX_SIDE || nx > XL_MAX_SIDE) return 0;
  return (size_t)rs_px(ny, nx) * rs_py(ny, nx) * sizeof(float2);
}

extern "C" size_t xl_rs_spectrum_work_bytes(int ny, int nx) { return xl_rs_spectrum_bytes(ny, nx); }

extern "C" size_t xl_rs_work_bytes(int batch, int comps, int ny, int nx) {
  if (ny < 2 || nx < 2 || ny > XL_MAX_SIDE || nx > XL_MAX_SIDE || batch < 1 || comps < 1) return 0;
  return (size_t)batch * comps * ny * rs_px(ny, nx) * sizeof(float2);
}

static int transfer_spectrum(const char* what, void* stream, int ny, int nx, const double* offx,
                             const double* offy, double z, const double* zp, int count, long long sstride,
                             double wavelength, double scale, void* spectrum_out, void* work, int dz) {
  if (ny < 2 || nx < 2 || ny > XL_MAX_SIDE || nx > XL_MAX_SIDE) {
    set_error("%s: field side out of range (2..%d): %d x %d", what, XL_MAX_SIDE, ny, nx);
    return XL_EINVAL;
  }
  if (!offx || !offy || !spectrum_out || !work) {
    set_error("%s: null pointer argument", what);
    return XL_EINVAL;
  }
  if ((!zp && !(z != 0.0)) || !(wavelength > 0.0)) {
    set_error("%s: need z != 0 and wavelength > 0 (got z=%g, wavelength=%g)", what, z, wavelength);
    return XL_EINVAL;
  }
  if (count < 1 || (count > 1 && sstride < (long long)(xl_rs_spectrum_bytes(ny, nx) / sizeof(float2)))) {
    set_error("%s: bad spectrum count %d or stride %lld", what, count, sstride);
    return XL_EINVAL;
  }
  if (int rc = ensure_init()) return rc;
  cudaStream_t st = (cudaStream_t)stream;
  for (int e = 0; e < count; ++e)
    if (int rc = spectrum(st, ny, nx, offx, offy, z, zp ? zp + e : nullptr, wavelength, scale,
                          (float2*)spectrum_out + (long long)e * sstride, (float2*)work, dz))
      return rc;
  return XL_OK;
}

extern "C" int xl_rs_transfer_spectrum(void* stream, int ny, int nx, const double* offx,
                                       const double* offy, double z, double wavelength,
                                       double scale, void* spectrum, void* work) {
  return transfer_spectrum("xl_rs_transfer_spectrum", stream, ny, nx, offx, offy, z, nullptr, 1, 0, wavelength,
                           scale, spectrum, work, 0);
}

extern "C" int xl_rs_transfer_spectrum_dz(void* stream, int ny, int nx, const double* offx,
                                          const double* offy, double z, double wavelength,
                                          double scale, void* spectrum, void* work) {
  return transfer_spectrum("xl_rs_transfer_spectrum_dz", stream, ny, nx, offx, offy, z, nullptr, 1, 0,
                           wavelength, scale, spectrum, work, 1);
}

extern "C" int xl_rs_transfer_spectra_device_z(void* stream, int ny, int nx, const double* offx,
                                               const double* offy, const double* z, int count, double wavelength,
                                               double scale, int dz, void* spectra, long long spectrum_stride,
                                               void* work) {
  if (!z) {
    set_error("xl_rs_transfer_spectra_device_z: null distance array");
    return XL_EINVAL;
  }
  return transfer_spectrum("xl_rs_transfer_spectra_device_z", stream, ny, nx, offx, offy, 0.0, z, count,
                           spectrum_stride, wavelength, scale, spectra, work, dz ? 1 : 0);
}

static int rs_run(void* stream, const XlRsArgs* a, int stage) {
  if (!a) {
    set_error("xl_rs_propagate: null args");
    return XL_EINVAL;
  }
  if (a->ny < 2 || a->nx < 2 || a->ny > XL_MAX_SIDE || a->nx > XL_MAX_SIDE || a->batch < 1) {
    set_error("xl_rs_propagate: bad shape batch=%d ny=%d nx=%d", a->batch, a->ny, a->nx);
    return XL_EINVAL;
  }
  const bool scalar = a->comps_in == 1 && a->comps_out == 1;
  const bool vector = a->adjoint ? (a->comps_in == 3 && a->comps_out == 3)
                                 : (a->comps_in == 2 && a->comps_out == 3);
  if (!scalar && !vector) {
    set_error("xl_rs_propagate: comps_in/comps_out must be 1/1 (RS), 2/3 (VRS) or 3/3 (VRS adjoint), "
              "got %d/%d (adjoint=%d)", a->comps_in, a->comps_out, a->adjoint);
    return XL_EINVAL;
  }
  if (a->adjoint && (a->pre.nops || a->post.nops)) {
    set_error("xl_rs_propagate: the adjoint takes no fused programs");
    return XL_EINVAL;
  }
  const int nout = (a->adjoint && vector) ? 2 : a->comps_out;
  for (int c = 0; c < a->comps_in; ++c)
    if (!a->in[c]) { set_error("xl_rs_propagate: null input plane %d", c); return XL_EINVAL; }
  for (int c = 0; c < nout; ++c)
    if (!a->out[c]) { set_error("xl_rs_propagate: null output plane %d", c); return XL_EINVAL; }
  if ((!a->spectrum && !a->spectra) || !a->work) {
    set_error("xl_rs_propagate: null spectrum or workspace");
    return XL_EINVAL;
  }
  if (vector && (!a->x || !a->y || !a->z)) {
    set_error("xl_rs_propagate: VRS needs x, y and z arrays");
    return XL_EINVAL;
  }
  if (a->pre.nops < 0 || a->pre.nops > XL_MAX_OPS || a->post.nops < 0 || a->post.nops > XL_MAX_OPS) {
    set_error("xl_rs_propagate: op program too long");
    return XL_EINVAL;
  }
  if (int rc = ensure_init()) return rc;
  RsLaunch p;
  p.B = a->batch; p.cin = a->comps_in; p.cout = a->comps_out; p.ny = a->ny; p.nx = a->nx;
  for (int c = 0; c < 3; ++c) {
    p.in[c] = (const float2*)a->in[c];
    p.out[c] = (float2*)a->out[c];
  }
  p.ibs = a->in_bstride; p.obs = a->out_bstride;
  p.x = a->x; p.y = a->y; p.z = a->z;
  p.spec = (const float2*)a->spectrum; p.sstride = a->spectrum_stride; p.sidx = a->spectrum_index;
  p.specs = (const float2* const*)a->spectra;
  p.work = (float2*)a->work;
  p.pre = a->pre; p.post = a->post;
  p.adjoint = a->adjoint ? 1 : 0;
  p.px = rs_px(a->ny, a->nx);
  p.py = rs_py(a->ny, a->nx);
  // column tiles of 8: a row's pieces are then 64 bytes.  4-wide tiles suit the
  // column pass and 16-wide ones the row passes better, but together they are
  // slower (8 x 2048^2 VRS, forward + columns + inverse: 3.5 and 2.8 ms against
  // 2.78; 16 x 1024^2 scalar: 494 and 544 against 470 us)
  p.lw = 3;
  // Light behind a polarizer at one angle has one transverse degree of freedom:
  // its Ex and Ey are c and s times one field, and so are their propagations,
  // so two components are transformed instead of three.
  p.pol = 0;
  if (vector && !a->adjoint && a->pre.nops > 0 && a->post.nops == 0 && rs_is_blk(a->ny, a->nx) &&
      !rs_is_half(a->nx)) {
    const XlOp& lp = a->pre.ops[a->pre.nops - 1];
    if (lp.kind == XL_OP_LP && !(lp.pmask & 1)) {
      p.pol = 1;
      p.pol_c = lp.sval[2];
      p.pol_s = lp.sval[3];
      --p.pre.nops;
    }
  }
  cudaStream_t st = (cudaStream_t)stream;
  if (rs_is_blk(a->ny, a->nx)) return blk_propagate(st, p, stage);
  return stockham_propagate(rs_logq(a->ny, a->nx), st, p, stage);
}

extern "C" int xl_rs_propagate(void* stream, const XlRsArgs* a) { return rs_run(stream, a, -1); }

extern "C" int xl_rs_stage(void* stream, const XlRsArgs* a, int stage) {
  if (stage < 0 || stage > 2) {
    set_error("xl_rs_stage: stage must be 0, 1 or 2 (got %d)", stage);
    return XL_EINVAL;
  }
  return rs_run(stream, a, stage);
}

// ---------------------------------------------------------------------------
// Allocation-free RS / VRS.
//
// Some callers of this library cannot call cudaMalloc.  Two examples: a host
// program that reserves all device memory for its own pool at start-up (a
// later cudaMalloc fails or fragments the pool), and a loop that drives
// optical hardware frame by frame, which cannot take the implicit device
// synchronisation and unbounded latency that cudaMalloc / cudaFree can cause.
// xl_rs_propagate_noalloc serves them.  It runs exactly the passes of
// xl_rs_propagate, but its workspace is the fixed device array below, so the
// caller passes only inputs (fields, transfer spectrum, coordinates) and
// outputs, and the call allocates no device memory.
//
// The array holds XL_RS_NOALLOC_MAX_WORK_BYTES on every GPU that loads the
// library, until the process exits.  All calls share it and it keeps the last
// call's contents; nothing in it needs clearing, because the first pass writes
// every element the later passes read.  Calls whose work overlaps on the GPU
// (different streams, or different host threads) race on the array.
static __device__ __align__(256) float2 g_rs_noalloc_scratch[XL_RS_NOALLOC_MAX_WORK_BYTES / sizeof(float2)];

static std::mutex g_noalloc_mu;
static float2* g_noalloc_ptr[256];

// Device address of the scratch array for the current device.  The array's
// name in host code is only a stand-in for the symbol, so the address is
// looked up once per device, with that device current.  The lookup also
// loads this file's device module, which is when the runtime allocates the
// array.
static cudaError_t noalloc_lookup(float2** out) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 256) return cudaErrorInvalidDevice;
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_ptr[dev]) {
    void* p = nullptr;
    if ((e = cudaGetSymbolAddress(&p, g_rs_noalloc_scratch)) != cudaSuccess) return e;
    g_noalloc_ptr[dev] = (float2*)p;
  }
  if (out) *out = g_noalloc_ptr[dev];
  return cudaSuccess;
}

// Run at every device's set-up (xl_init, or the first call of any entry
// point), so that the array exists from then on: a host that hands the rest
// of device memory to its own pool afterwards still has it.
static cudaError_t noalloc_setup(const float2*) { return noalloc_lookup(nullptr); }
static const bool g_noalloc_registered = register_device_tables(&noalloc_setup, nullptr);

extern "C" int xl_rs_propagate_noalloc(void* stream, const XlRsArgs* a) {
  if (!a) {
    set_error("xl_rs_propagate_noalloc: null args");
    return XL_EINVAL;
  }
  const size_t need = xl_rs_work_bytes(a->batch, a->comps_out, a->ny, a->nx);
  if (need == 0) {
    set_error("xl_rs_propagate_noalloc: bad shape batch=%d comps_out=%d ny=%d nx=%d", a->batch,
              a->comps_out, a->ny, a->nx);
    return XL_EINVAL;
  }
  if (need > (size_t)XL_RS_NOALLOC_MAX_WORK_BYTES) {
    set_error("xl_rs_propagate_noalloc: this call needs %zu bytes of scratch, the fixed limit is %llu "
              "(e.g. one 1024x1024 VRS field or one 2048x2048 scalar field); use xl_rs_propagate with a "
              "caller workspace for larger work",
              need, (unsigned long long)XL_RS_NOALLOC_MAX_WORK_BYTES);
    return XL_EINVAL;
  }
  if (int rc = ensure_init()) return rc;
  int dev = 0, sdev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return cuda_fail(e, "xl_rs_propagate_noalloc: cudaGetDevice");
  if ((e = cudaStreamGetDevice((cudaStream_t)stream, &sdev)) != cudaSuccess)
    return cuda_fail(e, "xl_rs_propagate_noalloc: cudaStreamGetDevice");
  if (sdev != dev) {
    set_error("xl_rs_propagate_noalloc: the stream belongs to device %d, the current device is %d", sdev, dev);
    return XL_EINVAL;
  }
  float2* scratch = nullptr;
  if ((e = noalloc_lookup(&scratch)) != cudaSuccess)
    return cuda_fail(e, "xl_rs_propagate_noalloc: cudaGetSymbolAddress");
  XlRsArgs b = *a;
  b.work = scratch;
  return rs_run(stream, &b, -1);
}
