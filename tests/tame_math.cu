// The branch-free divisions, square root and face solve of swe_math.cuh
// against CUDA's correctly rounded intrinsics and the operators' own solve:
// random and structured significands over the exponents the face kernel lets
// through, quotients next to a rounding boundary, and the square roots read
// from standard input (the significands whose root lies nearest to one).
// Prints a mismatch count per function.
#include <cstdio>
#include <cstring>
#include <vector>

#include "swe_math.cuh"
using namespace swe;

__device__ unsigned long long rng(unsigned long long& s) {      // splitmix64
  s += 0x9E3779B97F4A7C15ull;
  unsigned long long z = s;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
// A double of exponent lo <= e < hi: a random significand, one bit clear, one
// bit set, close below or above a power of two, or short.
__device__ double number(unsigned long long& s, int lo, int hi) {
  const unsigned long long r = rng(s);
  unsigned long long m = rng(s) & 0xfffffffffffffull;
  switch (r & 7) {
    case 1: m = 0xfffffffffffffull ^ (1ull << (rng(s) % 52)); break;
    case 2: m = 1ull << (rng(s) % 52); break;
    case 3: m = 0xfffffffffffffull - (rng(s) & 0xff); break;
    case 4: m = rng(s) & 0xff; break;
    case 5: m >>= rng(s) % 52; break;
  }
  const unsigned long long e = lo + (int)((r >> 8) % (unsigned)(hi - lo)) + 1023;
  return __longlong_as_double(((r >> 60) & 1) << 63 | e << 52 | m);
}
__device__ bool same(double a, double b) { return __double_as_longlong(a) == __double_as_longlong(b); }
__device__ double next(double x, int d) { return __longlong_as_double(__double_as_longlong(x) + d); }

enum { RCP, DIV, DIV_HARD, DIV_PRODUCT, SQRT, DIV_G, RCP_SQUARE, VEL, LIMITER, FACE, COUNT };

__global__ void k_check(int iters, unsigned long long* bad) {
  unsigned long long s = 104729ull * (blockIdx.x * blockDim.x + threadIdx.x + 1);
  for (int it = 0; it < iters; it++) {
    const double b = fabs(number(s, -160, 160)), a = number(s, -700, 200);
    if (!same(sqrt_tame(b), __dsqrt_rn(b))) bad[SQRT] = 1;
    const double g = fabs(number(s, -60, 60));
    for (int d = -2; d <= 2; d++)
      if (!same(sqrt_tame(next(g * g, d)), __dsqrt_rn(next(g * g, d)))) bad[SQRT] = 1;
    if (!same(div_g(g), __ddiv_rn(g, SWE_G))) bad[DIV_G] = 1;
    if (!ones_lo(b)) {
      const double y = rcp_tame(b), n = number(s, -700, 60), p = b * n, D = b * b;
      if (!same(y, __drcp_rn(b))) bad[RCP] = 1;
      if (!same(div_tame(a, b, y), __ddiv_rn(a, b)) || !same(div_tame(-0.0, b, y), -0.0)) bad[DIV] = 1;
      // b times the midpoint above a quotient q, and its neighbours
      const double q = number(s, -20, 20);
      const double half = __longlong_as_double(__double_as_longlong(q) & 0x7ff0000000000000ll) * 0x1p-53;
      for (int d = -1; d <= 1; d++) {
        const double h = next(fma(b, q, b * half), d);
        if (!same(div_tame(h, b, y), __ddiv_rn(h, b))) bad[DIV_HARD] = 1;
      }
      if (!same(div_product(p, b, n, y), __ddiv_rn(p, b)) || !same(div_product(-0.0, b, -0.0, y), -0.0))
        bad[DIV_PRODUCT] = 1;
      if (!ones_lo(D) && !same(rcp_refine(D, rcp_refine(D, y * y)), __drcp_rn(D))) bad[RCP_SQUARE] = 1;
    }
    const double h = fabs(number(s, -100, 40)), hu = (it & 7) ? number(s, -700, 100) : copysign(0.0, a);
    const double hv = number(s, -700, 100), eps4 = (it & 1) ? 1e-12 : 1e-48;
    double u, v;
    if (vel_tame(hu, hv, h, eps4, u, v)) {
      const double den = vel_den(h, eps4);
      if (!same(u, __ddiv_rn(vel_num(hu, h), den)) || !same(v, __ddiv_rn(vel_num(hv, h), den))) bad[VEL] = 1;
    }
    // a face between two cells: dry or wet, alike down to rounding or far apart, sub- and supercritical
    const unsigned long long r = rng(s);
    const double amp = (r & 3) == 0 ? 1.0 : (r & 3) == 1 ? 1e-3 : (r & 3) == 2 ? 1e-15 : 0.0;
    const double base = (rng(s) >> 11) * 0x1p-53 * 4, fast = ((r >> 15) & 15) ? 1 : 20;
    double x[2][8];
    for (int c = 0; c < 2; c++) {
      for (int k = 0; k < 8; k++) x[c][k] = amp * ((rng(s) >> 11) * 0x1p-52 - 1);
      x[c][0] *= (r >> 4) & 1;
      x[c][5] *= (r >> 4) & 1;
      x[c][1] = base + x[c][1];
      if (x[c][1] < 0 || ((r >> (5 + 5 * c)) & 31) == 0) x[c][1] = 0;
      x[c][2] *= fast;
    }
    const double *L = x[0], *R = x[1];
    if (!same(limiter_mc_tame(L[2], R[2]), limiter(0, L[2], R[2]))) bad[LIMITER] = 1;
    bool redo;
    const FaceSums f = face_flux_tame(L[0], L[1], L[2], L[3], L[4], L[5], L[6], L[7], R[0], R[1], R[2], R[3], R[4],
                                      R[5], R[6], R[7], 1e-3, redo);
    const Face w = face_flux(L[0], L[1], L[2], L[3], L[4], L[5], L[6], L[7], R[0], R[1], R[2], R[3], R[4], R[5], R[6],
                             R[7], 1e-3);
    if (!redo && (!same(f.M, w.M) || !same(f.T, w.T) || !same(f.NpL, w.N + w.pL) || !same(f.NpR, w.N + w.pR)))
      bad[FACE] = 1;
  }
}

__global__ void k_roots(int n, const double* x, unsigned long long* bad) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= n) return;
  for (int e = -160; e <= 160; e += 2)
    if (!same(sqrt_tame(ldexp(x[q], e)), __dsqrt_rn(ldexp(x[q], e)))) bad[SQRT] = 1;
}

int main() {
  const char* names[COUNT] = {"rcp", "div", "div_hard", "div_product", "sqrt", "div_g", "rcp_square", "vel", "limiter",
                              "face"};
  std::vector<double> roots;
  for (double x; std::scanf("%la", &x) == 1;) roots.push_back(x);
  unsigned long long *bad, out[COUNT];
  double* d;
  if (cudaMalloc(&bad, sizeof out) || cudaMemset(bad, 0, sizeof out) || cudaMalloc(&d, 8 * roots.size() + 8)) return 2;
  cudaMemcpy(d, roots.data(), 8 * roots.size(), cudaMemcpyHostToDevice);
  k_roots<<<1, 64>>>((int)roots.size(), d, bad);
  k_check<<<592, 256>>>(400, bad);
  if (cudaMemcpy(out, bad, sizeof out, cudaMemcpyDeviceToHost)) return 3;
  for (int q = 0; q < COUNT; q++) std::printf("%s %llu\n", names[q], out[q]);
  return roots.size() > 64 ? 4 : 0;
}
