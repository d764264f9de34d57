// swe_render.cu -- headless frames of the solver's state, written as RGBA
// bytes into a device buffer (and optionally copied to the host).
//
//   swe_render_map    the map panel of WaterView.draw() (src/render.mjs:220-247):
//                     one pixel per interior cell, +y up, the diverging L*a*b*
//                     ramp about mean sea level over water (darkened by the STILL
//                     depth when the bed is shown), the land ramp over dry cells.
//   swe_render_globe  renderGlobe() (src/globe.mjs:770-812): an orthographic view
//                     of a spherical grid through a pixel -> cell table baked
//                     once per (size, tilt, margin, grid) by buildGlobeLut()
//                     (src/globe.mjs:554-629); the frame is a copy of the baked
//                     background plus one thread per modelled pixel.
//
// Bytes are stored as a Uint8ClampedArray stores a double (clamp to [0, 255],
// round half to even, NaN to 0), which is how the reference's ImageData holds
// them.  The colour tables are built on the host with the reference's
// formulas (src/render.mjs:98-131, src/globe.mjs:644-652).
#include "../../include/swe_b200.h"

#include <cuda_runtime.h>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <algorithm>
#include <mutex>
#include <string>
#include <vector>

namespace swe_host {
void set_error(const std::string& msg);
void view_of(swe_sim* s, int* dims, double* opts, const double** b, const double** h, cudaStream_t* st);
int frame_of(swe_sim* s, size_t bytes, unsigned char** out);
}  // namespace swe_host

struct swe_globe_lut {
  int size = 0, count = 0, inside = 0, capped = 0;
  double tilt = 0, margin = 0;
  int nx = 0, ny = 0;
  double lat0 = 0, lat1 = 0;
  int* d_px = nullptr;           // byte offset of the pixel in the frame
  double* d_lon = nullptr;       // longitude of the pixel centre at rotation 0 [deg]
  int* d_rowbase = nullptr;      // padded index of the row's first interior cell
  float* d_lit = nullptr;        // cos(incidence) of the viewer-fixed light
  unsigned char* d_bg = nullptr; // everything that is not modelled ocean or land
  unsigned char* d_out = nullptr; // a frame drawn for the host
  void* d_all = nullptr;         // the allocation that holds them
  double* d_stats = nullptr;     // frame reduction scratch
  unsigned int* d_ticket = nullptr;
  int nblocks = 0;
  // A table serves every simulation of its grid, from several threads: d_out,
  // d_stats and d_ticket are one frame's at a time.
  std::mutex frame;
};

namespace {

int fail(int code, const std::string& m) { swe_host::set_error(m); return code; }

#define RCU(call)                                                                          \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess) return fail(SWE_ECUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
  } while (0)

constexpr int RAMP_N = 1025;                    // odd: entry (N-1)/2 is mean sea level exactly
constexpr int RAMP_MID = (RAMP_N - 1) >> 1;
constexpr double PI_D = 3.141592653589793;

// The tables lie in global memory, not in constant memory, which serves one
// address at a time: a warp's pixels look up different colours.
__device__ double g_ramp[3 * RAMP_N];           // src/render.mjs RAMP (unclamped sRGB)
__device__ __align__(4) unsigned char g_cbytes[4 * RAMP_N];   // src/globe.mjs CBYTES, RGBA

// ---- the colour tables (host) ------------------------------------------------
// CIE L*a*b* (D65) -> sRGB, unclamped (src/render.mjs:98-110).
void lab_to_srgb_raw(double L, double a, double bb, double* out) {
  const double fy = (L + 16) / 116, fx = fy + a / 500, fz = fy - bb / 200;
  auto g = [](double f) { return f * f * f > 0.008856 ? f * f * f : (f - 16.0 / 116) / 7.787; };
  const double X = 0.95047 * g(fx), Y = g(fy), Z = 1.08883 * g(fz);
  auto enc = [](double u) {
    return 255 * (u <= 0.0031308 ? 12.92 * u : 1.055 * std::pow(u > 0 ? u : 0.0, 1 / 2.4) - 0.055);
  };
  out[0] = enc(3.2406 * X - 1.5372 * Y - 0.4986 * Z);
  out[1] = enc(-0.9689 * X + 1.8758 * Y + 0.0415 * Z);
  out[2] = enc(0.0557 * X - 0.2040 * Y + 1.0570 * Z);
}

// Uint8ClampedArray's conversion of a double (ToUint8Clamp).
__host__ __device__ __forceinline__ unsigned char clamp_u8(double x) {
  if (!(x > 0)) return 0;                       // NaN, negative, zero
  if (x >= 255) return 255;
  const double f = floor(x);
  const double d = x - f;
  if (d > 0.5) return (unsigned char)(f + 1);
  if (d < 0.5) return (unsigned char)f;
  const int fi = (int)f;
  return (unsigned char)((fi & 1) ? fi + 1 : fi);
}

// JavaScript Math.max / Math.min / Math.round.
__host__ __device__ __forceinline__ double js_max(double a, double b) {
  if (a != a) return a;
  if (b != b) return b;
  if (a > b) return a;
  if (b > a) return b;
  return signbit(a) ? b : a;
}
__host__ __device__ __forceinline__ double js_min(double a, double b) {
  if (a != a) return a;
  if (b != b) return b;
  if (a < b) return a;
  if (b < a) return b;
  return signbit(a) ? a : b;
}
__host__ __device__ __forceinline__ double js_round(double x) {
  const double f = floor(x);
  return (x - f >= 0.5) ? f + 1 : f;
}

struct Tables {
  double ramp[3 * RAMP_N];
  unsigned char cbytes[3 * RAMP_N];
};

void build_tables(Tables* t) {
  const double TROUGH[3] = {20, 8, -34}, MSL[3] = {53, -4, -14}, CREST[3] = {86, 6, 44};
  for (int i = 0; i < RAMP_N; i++) {                          // buildRamp, src/render.mjs:118-131
    const double tt = -1 + (2.0 * i) / (RAMP_N - 1);
    const double* end = tt >= 0 ? CREST : TROUGH;
    const double q = std::fabs(tt);
    lab_to_srgb_raw(MSL[0] + (end[0] - MSL[0]) * q, MSL[1] + (end[1] - MSL[1]) * q,
                    MSL[2] + (end[2] - MSL[2]) * q, t->ramp + 3 * i);
  }
  for (int i = 0; i < RAMP_N; i++) {                          // CBYTES, src/globe.mjs:644-652
    const double v = -1 + (2.0 * i) / (RAMP_N - 1);
    const double tt = js_max(-1, js_min(1, v / 1));           // surfaceColour(v, 1)
    const double q = js_round(std::fabs(tt) * RAMP_MID);
    const int o = 3 * (tt >= 0 ? RAMP_MID + (int)q : RAMP_MID - (int)q);
    for (int c = 0; c < 3; c++) t->cbytes[3 * i + c] = clamp_u8(t->ramp[o + c]);
  }
}

bool aligned4(const void* p) { return (reinterpret_cast<size_t>(p) & 3) == 0; }

int ensure_tables() {
  static int done = -1;                        // per process; the tables are a copy per device
  static int done_dev = -1;
  int dev = 0;
  RCU(cudaGetDevice(&dev));
  if (done == 1 && done_dev == dev) return SWE_OK;
  static Tables t;
  build_tables(&t);
  static unsigned char rgba[4 * RAMP_N];
  for (int i = 0; i < RAMP_N; i++) {
    for (int c = 0; c < 3; c++) rgba[4 * i + c] = t.cbytes[3 * i + c];
    rgba[4 * i + 3] = 255;
  }
  RCU(cudaMemcpyToSymbol(g_ramp, t.ramp, sizeof t.ramp));
  RCU(cudaMemcpyToSymbol(g_cbytes, rgba, sizeof rgba));
  // a copy from pageable memory may return before it has reached the device,
  // and the handles' streams do not wait for the default stream
  RCU(cudaStreamSynchronize(0));
  done = 1;
  done_dev = dev;
  return SWE_OK;
}

// ---- WaterView map panel -------------------------------------------------------
// surfaceColour (src/render.mjs:142-153): the RAMP entry for elevation v.
__device__ __forceinline__ int ramp_index(double v, double scale) {
  const double t = js_max(-1, js_min(1, v / scale));
  if (t != t) return -1;                       // NaN: the reference reads undefined -> 0
  const int q = (int)js_round(fabs(t) * RAMP_MID);
  return t >= 0 ? RAMP_MID + q : RAMP_MID - q;
}

__device__ __forceinline__ unsigned pixel(unsigned char r, unsigned char g, unsigned char b) {
  return 0xff000000u | (unsigned)b << 16 | (unsigned)g << 8 | r;
}
// Pixel p of a frame: one store where the frame lies on a 4-byte boundary (the
// caller's device buffer may not).
__device__ __forceinline__ void put_pixel(unsigned char* out, long long p, unsigned rgba, bool aligned) {
  if (aligned) reinterpret_cast<unsigned*>(out)[p] = rgba;
  else
    for (int c = 0; c < 4; c++) out[4 * p + c] = (unsigned char)(rgba >> (8 * c));
}

// A block per row, or as many as there are.
constexpr int FRAME_THREADS = 256;
__global__ void __launch_bounds__(FRAME_THREADS)
k_render_map(int nx, int ny, int W, const double* __restrict__ b, const double* __restrict__ h,
             double minDepth, double msl, double scale, int showBed, unsigned char* __restrict__ out, bool aligned) {
  for (int j = blockIdx.x; j < ny; j += gridDim.x) {
    const size_t row = (size_t)(j + 2) * W + 2;
    for (int i = threadIdx.x; i < nx; i += FRAME_THREADS) {
      const double depth = h[row + i], bk = b[row + i];
      double c0, c1, c2;
      if (depth <= minDepth) {                    // landColour, src/render.mjs:193-196
        const double t = js_max(0, js_min(1, bk / 6));
        c0 = 96 + 70 * t; c1 = 88 + 62 * t; c2 = 74 + 52 * t;
      } else {
        const int ro = ramp_index(bk + depth - msl, scale);
        if (ro < 0) { c0 = c1 = c2 = NAN; }
        else { c0 = __ldg(g_ramp + 3 * ro); c1 = __ldg(g_ramp + 3 * ro + 1); c2 = __ldg(g_ramp + 3 * ro + 2); }
        if (showBed) {                            // STILL depth shading, src/render.mjs:238-245
          const double still = js_max(0, msl - bk);
          const double shade = 0.55 + 0.45 * exp(-still / 12);
          c0 = c0 * shade; c1 = c1 * shade; c2 = c2 * shade;
        }
      }
      put_pixel(out, (long long)(ny - 1 - j) * nx + i, pixel(clamp_u8(c0), clamp_u8(c1), clamp_u8(c2)), aligned);  // +y up
    }
  }
}

// ---- renderGlobe ------------------------------------------------------------------
constexpr double LAND_SAT = 2500;               // src/globe.mjs:680-682
__constant__ double c_land_lo[3] = {92, 84, 70};
__constant__ double c_land_hi[3] = {188, 172, 144};

// colOfLon (src/globe.mjs:547-550), with the rotation applied as frameLon()'s
// addition (src/globe.mjs:741).
__device__ __forceinline__ int col_of_lon(double lonDeg, int nx) {
  const double i = floor((lonDeg + 180) * nx / 360);
  if (i >= 0 && i < nx) return (int)i;
  if (i >= nx && i < 2.0 * nx) return (int)(i - nx);
  const long long ii = (long long)i;
  return (int)(((ii % nx) + nx) % nx);
}

// A frame's statistics: the least and largest elevation and three counts.
struct FrameStats { double lo, hi; unsigned int wet, dry, sat; };
__device__ __forceinline__ FrameStats both(FrameStats a, const FrameStats& b) {
  return {fmin(a.lo, b.lo), fmax(a.hi, b.hi), a.wet + b.wet, a.dry + b.dry, a.sat + b.sat};
}
// Over the block, in thread 0.
__device__ __forceinline__ FrameStats block_stats(FrameStats v, FrameStats* warps) {
  const unsigned all = 0xffffffffu;
  for (int o = 16; o > 0; o >>= 1) {
    FrameStats u = {__shfl_down_sync(all, v.lo, o), __shfl_down_sync(all, v.hi, o), __shfl_down_sync(all, v.wet, o),
                    __shfl_down_sync(all, v.dry, o), __shfl_down_sync(all, v.sat, o)};
    v = both(v, u);
  }
  if ((threadIdx.x & 31) == 0) warps[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < FRAME_THREADS / 32; w++) v = both(v, warps[w]);
  return v;
}

// Bound by the gather of the pixels' cells and, at a million pixels, by the
// frame's way to the host.  The last block combines the blocks' statistics
// with all of its threads: one thread reading them in turn took most of the
// launch (900 x 900 pixels: 140 -> 18 us).
__global__ void __launch_bounds__(FRAME_THREADS)
k_render_globe(int count, const int* __restrict__ px, const double* __restrict__ lon,
               const int* __restrict__ rowbase, const float* __restrict__ lit, int nx,
               const double* __restrict__ b, const double* __restrict__ h, double minDepth,
               double rot, double scale, double msl, int landLight, unsigned char* __restrict__ out, bool aligned,
               FrameStats* __restrict__ part, unsigned int* ticket, double* __restrict__ stats) {
  __shared__ FrameStats warps[FRAME_THREADS / 32];
  __shared__ bool s_last;
  FrameStats v = {INFINITY, -INFINITY, 0, 0, 0};
  for (int p = blockIdx.x * FRAME_THREADS + threadIdx.x; p < count; p += gridDim.x * FRAME_THREADS) {
    const long long k = rowbase[p] + col_of_lon(lon[p] + rot, nx);
    const double hk = h[k], bk = b[k];
    unsigned rgba;
    if (hk <= minDepth) {
      v.dry++;
      const double t = js_max(0, js_min(1, bk / LAND_SAT));
      const double s = landLight ? 0.30 + 0.70 * (double)lit[p] : 1;
      unsigned char c[3];
      for (int q = 0; q < 3; q++) c[q] = clamp_u8((c_land_lo[q] + (c_land_hi[q] - c_land_lo[q]) * t) * s);
      rgba = pixel(c[0], c[1], c[2]);
    } else {
      v.wet++;
      const double e = bk + hk - msl;
      if (e < v.lo) v.lo = e;
      if (e > v.hi) v.hi = e;
      if (e >= scale || e <= -scale) v.sat++;
      const int co = ramp_index(e, scale);      // colourOffset, src/globe.mjs:665-669
      rgba = co < 0 ? pixel(0, 0, 0) : __ldg(reinterpret_cast<const unsigned*>(g_cbytes) + co);
    }
    put_pixel(out, px[p] / 4, rgba, aligned);
  }
  v = block_stats(v, warps);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = v;
    __threadfence();
    s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!s_last) return;                          // the last block closes the frame (no waiting)
  __threadfence();
  v = {INFINITY, -INFINITY, 0, 0, 0};
  for (unsigned int g = threadIdx.x; g < gridDim.x; g += FRAME_THREADS) {
    const FrameStats* q = part + g;
    v = both(v, {__ldcg(&q->lo), __ldcg(&q->hi), __ldcg(&q->wet), __ldcg(&q->dry), __ldcg(&q->sat)});
  }
  v = block_stats(v, warps);
  if (threadIdx.x == 0) {
    stats[0] = v.wet; stats[1] = v.dry; stats[4] = v.lo; stats[5] = v.hi; stats[6] = v.sat;
    stats[7] = v.wet > 0 ? (double)v.sat / (double)v.wet : 0;
    *ticket = 0;
  }
}

// ---- the LUT bake (host) --------------------------------------------------------------
struct Cam { double size, margin, r, cx, cy, tilt, sinT, cosT; };

Cam globe_camera(int size, double tilt, double margin) {     // src/globe.mjs:460-466
  Cam c;
  c.size = size; c.margin = margin; c.r = 0.5 * size * margin; c.cx = 0.5 * size; c.cy = 0.5 * size;
  c.tilt = tilt;
  const double D2R = PI_D / 180;
  c.sinT = std::sin(tilt * D2R); c.cosT = std::cos(tilt * D2R);
  return c;
}

int row_of_lat(double latDeg, double lat0, double lat1, int ny) {   // src/globe.mjs:561-568
  if (latDeg < lat0 || latDeg > lat1) return -1;
  int j = (int)std::floor((latDeg - lat0) * ny / (lat1 - lat0));
  if (j >= ny) j = ny - 1;
  else if (j < 0) j = 0;
  return j;
}

}  // namespace

extern "C" {

int swe_render_tables(double* ramp, unsigned char* cbytes) {
  static Tables t;
  build_tables(&t);
  if (ramp) std::memcpy(ramp, t.ramp, sizeof t.ramp);
  if (cbytes) std::memcpy(cbytes, t.cbytes, sizeof t.cbytes);
  return SWE_OK;
}

int swe_render_map(swe_sim* s, double msl, double scale, int show_bed, unsigned char* rgba_host, void* rgba_device) {
  if (!s || (!rgba_host && !rgba_device)) return fail(SWE_EINVAL, "swe_render_map: null handle or no output");
  int dims[5];
  double opts[5];
  const double *b, *h;
  cudaStream_t st;
  swe_host::view_of(s, dims, opts, &b, &h, &st);
  const int nx = dims[0], ny = dims[1], W = dims[2];
  int rc = ensure_tables();
  if (rc) return rc;
  const size_t bytes = (size_t)4 * nx * ny;
  unsigned char* out = static_cast<unsigned char*>(rgba_device);
  if (!out) { rc = swe_host::frame_of(s, bytes, &out); if (rc) return rc; }
  k_render_map<<<std::min(ny, 148 * 32), FRAME_THREADS, 0, st>>>(nx, ny, W, b, h, opts[0], msl, scale, show_bed ? 1 : 0,
                                                                out, aligned4(out));
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess && rgba_host) e = cudaMemcpyAsync(rgba_host, out, bytes, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(SWE_ECUDA, std::string("swe_render_map: ") + cudaGetErrorString(e));
  return SWE_OK;
}

int swe_globe_lut_create(swe_sim* s, int size, double tilt_deg, double margin, const double* sun,
                         const double* bg, const double* halo, swe_globe_lut** out) {
  if (!out) return fail(SWE_EINVAL, "null output");
  *out = nullptr;
  if (!s || size < 1) return fail(SWE_EINVAL, "swe_globe_lut_create: null handle or size < 1");
  int dims[5];
  double opts[5];
  const double *b, *h;
  cudaStream_t st;
  swe_host::view_of(s, dims, opts, &b, &h, &st);
  if (!dims[4])
    return fail(SWE_EINVAL, "globe.mjs draws spherical fields only: sim.geom.kind is cartesian. "
                            "Use the map panel (swe_render_map).");
  const int nx = dims[0], ny = dims[1], W = dims[2];
  const double lat0 = opts[1], lat1 = opts[2];
  double sv[3] = {-0.42, 0.48, 0.77};
  if (sun) { sv[0] = sun[0]; sv[1] = sun[1]; sv[2] = sun[2]; }
  const double m = std::sqrt(sv[0] * sv[0] + sv[1] * sv[1] + sv[2] * sv[2]);   // normalise()
  const double su[3] = {sv[0] / m, sv[1] / m, sv[2] / m};
  const double B[3] = {bg ? bg[0] : 8, bg ? bg[1] : 11, bg ? bg[2] : 16};
  const double HALO[3] = {halo ? halo[0] : 36, halo ? halo[1] : 58, halo ? halo[2] : 84};
  const Cam cam = globe_camera(size, tilt_deg, margin);
  const double R2D = 180 / PI_D;
  const size_t NP = (size_t)size * size;
  std::vector<unsigned char> bgb(4 * NP, 0);
  std::vector<int> px, rowbase;
  std::vector<double> lon;
  std::vector<float> lit;
  int inside = 0, capped = 0;
  for (int y = 0; y < size; y++) {
    for (int x = 0; x < size; x++) {
      const size_t p = (size_t)y * size + x, o = 4 * p;
      // orthoInversePixel at rotation 0 (src/globe.mjs:500-520)
      const double X = (x + 0.5 - cam.cx) / cam.r, Y = (cam.cy - y - 0.5) / cam.r;
      const double ss = X * X + Y * Y;
      if (ss > 1) {
        const double g = std::exp(-(ss - 1) * 5.5);            // limb halo
        for (int c = 0; c < 3; c++) bgb[o + c] = clamp_u8(B[c] + (HALO[c] - B[c]) * g);
        bgb[o + 3] = 255;
        continue;
      }
      inside++;
      const double z = std::sqrt(1 - ss);
      const double phi = std::asin(z * cam.sinT + Y * cam.cosT);
      const double lam = std::atan2(X, z * cam.cosT - Y * cam.sinT);
      const double lonDeg = 0 + lam * R2D, latDeg = phi * R2D;
      const int j = row_of_lat(latDeg, lat0, lat1, ny);
      if (j < 0) {                                             // unmodelled cap: hatched
        capped++;
        const int t = ((x + y) & 7) < 3 ? 1 : 0;
        bgb[o] = 52 + 14 * t; bgb[o + 1] = 56 + 14 * t; bgb[o + 2] = 62 + 14 * t; bgb[o + 3] = 255;
        continue;
      }
      px.push_back((int)o);
      lon.push_back(lonDeg);
      rowbase.push_back((j + 2) * W + 2);
      const double l = X * su[0] + Y * su[1] + z * su[2];
      lit.push_back((float)js_max(0, l));
    }
  }
  swe_globe_lut* L = new swe_globe_lut();
  L->size = size; L->count = (int)px.size(); L->inside = inside; L->capped = capped;
  L->tilt = tilt_deg; L->margin = margin; L->nx = nx; L->ny = ny; L->lat0 = lat0; L->lat1 = lat1;
  const int n = std::max(1, L->count);
  L->nblocks = std::max(1, std::min(148 * 8, (L->count + FRAME_THREADS - 1) / FRAME_THREADS));
  const size_t sizes[8] = {sizeof(double) * n, sizeof(int) * n, sizeof(int) * n, sizeof(float) * n, 4 * NP, 4 * NP,
                           sizeof(double) * 8 + sizeof(FrameStats) * L->nblocks, sizeof(unsigned int)};
  size_t total = 0;
  for (size_t b : sizes) total += (b + 255) & ~size_t(255);
  cudaError_t e = cudaMalloc(&L->d_all, total);
  char* at = static_cast<char*>(L->d_all);
  auto take = [&](int q) { char* p = at; at += (sizes[q] + 255) & ~size_t(255); return p; };
  if (e == cudaSuccess) {
    L->d_lon = reinterpret_cast<double*>(take(0));
    L->d_px = reinterpret_cast<int*>(take(1));
    L->d_rowbase = reinterpret_cast<int*>(take(2));
    L->d_lit = reinterpret_cast<float*>(take(3));
    L->d_bg = reinterpret_cast<unsigned char*>(take(4));
    L->d_out = reinterpret_cast<unsigned char*>(take(5));
    L->d_stats = reinterpret_cast<double*>(take(6));
    L->d_ticket = reinterpret_cast<unsigned int*>(take(7));
  }
  // on the handle's stream, and complete before any other stream may read them
  auto up = [&](void* dst, const void* src, size_t bytes) {
    if (e == cudaSuccess && bytes) e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
  };
  up(L->d_px, px.data(), sizeof(int) * L->count);
  up(L->d_lon, lon.data(), sizeof(double) * L->count);
  up(L->d_rowbase, rowbase.data(), sizeof(int) * L->count);
  up(L->d_lit, lit.data(), sizeof(float) * L->count);
  up(L->d_bg, bgb.data(), 4 * NP);
  if (e == cudaSuccess) e = cudaMemsetAsync(L->d_ticket, 0, sizeof(unsigned int), st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    swe_globe_lut_destroy(L);
    return fail(SWE_ECUDA, std::string("swe_globe_lut_create: ") + cudaGetErrorString(e));
  }
  *out = L;
  return SWE_OK;
}

int swe_globe_lut_destroy(swe_globe_lut* L) {
  if (!L) return SWE_OK;
  cudaFree(L->d_all);
  delete L;
  return SWE_OK;
}

int swe_globe_lut_get(swe_globe_lut* L, int* counts, int* px, double* lon_base, int* row_base, float* lit,
                      unsigned char* bg) {
  if (!L) return fail(SWE_EINVAL, "null LUT");
  if (counts) { counts[0] = L->count; counts[1] = L->inside; counts[2] = L->capped; counts[3] = L->size; }
  const size_t n = L->count;
  if (px && n) RCU(cudaMemcpy(px, L->d_px, sizeof(int) * n, cudaMemcpyDeviceToHost));
  if (lon_base && n) RCU(cudaMemcpy(lon_base, L->d_lon, sizeof(double) * n, cudaMemcpyDeviceToHost));
  if (row_base && n) RCU(cudaMemcpy(row_base, L->d_rowbase, sizeof(int) * n, cudaMemcpyDeviceToHost));
  if (lit && n) RCU(cudaMemcpy(lit, L->d_lit, sizeof(float) * n, cudaMemcpyDeviceToHost));
  if (bg) RCU(cudaMemcpy(bg, L->d_bg, (size_t)4 * L->size * L->size, cudaMemcpyDeviceToHost));
  return SWE_OK;
}

int swe_render_globe(swe_sim* s, swe_globe_lut* L, double rot_deg, double scale, double msl, int land_light,
                     unsigned char* rgba_host, void* rgba_device, double* stats) {
  if (!s || !L) return fail(SWE_EINVAL, "swe_render_globe: null handle or LUT");
  if (!rgba_host && !rgba_device) return fail(SWE_EINVAL, "swe_render_globe: no output");
  int dims[5];
  double opts[5];
  const double *b, *h;
  cudaStream_t st;
  swe_host::view_of(s, dims, opts, &b, &h, &st);
  if (!dims[4]) return fail(SWE_EINVAL, "globe.mjs draws spherical fields only: sim.geom.kind is cartesian.");
  if (dims[0] != L->nx || dims[1] != L->ny || opts[1] != L->lat0 || opts[2] != L->lat1) {
    char buf[240];
    std::snprintf(buf, sizeof buf, "LUT was baked for %d|%.17g|%.17g|%d|%d|%.17g|%.17g, grid is now %d|%d|%.17g|%.17g",
                  L->size, L->tilt, L->margin, L->nx, L->ny, L->lat0, L->lat1, dims[0], dims[1], opts[1], opts[2]);
    return fail(SWE_EINVAL, buf);
  }
  int rc = ensure_tables();
  if (rc) return rc;
  const size_t bytes = (size_t)4 * L->size * L->size;
  unsigned char* out = static_cast<unsigned char*>(rgba_device);
  std::lock_guard<std::mutex> one(L->frame);    // until the frame is complete
  if (!out) out = L->d_out;
  cudaError_t e = cudaMemcpyAsync(out, L->d_bg, bytes, cudaMemcpyDeviceToDevice, st);   // out.set(lut.bg)
  FrameStats* part = reinterpret_cast<FrameStats*>(L->d_stats + 8);
  if (e == cudaSuccess && L->count > 0) {
    k_render_globe<<<L->nblocks, FRAME_THREADS, 0, st>>>(L->count, L->d_px, L->d_lon, L->d_rowbase, L->d_lit,
                                                        dims[0], b, h, opts[0], rot_deg, scale, msl,
                                                        land_light ? 1 : 0, out, aligned4(out), part, L->d_ticket, L->d_stats);
    e = cudaGetLastError();
  }
  double st8[8] = {0, 0, 0, 0, INFINITY, -INFINITY, 0, 0};
  if (e == cudaSuccess && L->count > 0) e = cudaMemcpyAsync(st8, L->d_stats, sizeof st8, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess && rgba_host) e = cudaMemcpyAsync(rgba_host, out, bytes, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return fail(SWE_ECUDA, std::string("swe_render_globe: ") + cudaGetErrorString(e));
  st8[2] = L->capped; st8[3] = L->inside;
  if (stats) std::memcpy(stats, st8, sizeof st8);
  return SWE_OK;
}

}  // extern "C"
