// ep_kernels_impl.cuh - bodies of the point-wise and reduction kernels.
#pragma once
#include "ep_kernels.cuh"
#include "ep_pairpot.h"

// Grid coordinate -xmax + h*i without contraction (x(i) of DFT4He3d.f90:248-256).
EP_DEV double coord(double xmax, double h, int i) { return __dadd_rn(-xmax, __dmul_rn(h, (double)i)); }

// |x - r_imp|^2 in potenimp.f90's order (zt = z^2, yt = y^2 + zt, x^2 + yt)
// without contraction: the table index int(1.5 + r/h) of update() then falls
// on the same side of a node as in an uncontracted FP64 evaluation (an FMA
// here moves r by an ulp, and where r/h sits on a node the parabola switches
// to the neighbouring three table points, a 1e-9 relative change of u_imp).
EP_DEV double rr2_nc(double xx, double yy, double zz) {
  return __dadd_rn(__dmul_rn(xx, xx), __dadd_rn(__dmul_rn(yy, yy), __dmul_rn(zz, zz)));
}

EP_DEV void idx3(const Geo& g, long long p, int& ix, int& iy, int& iz) {
  ix = (int)(p % g.nx);
  const long long r = p / g.nx;
  iy = (int)(r % g.ny);
  iz = (int)(r / g.ny);
}

// Parabolic interpolation in f(0:nint+1), the update() function of
// potenimp.f90:588-632, restated.
EP_DEV double interp_update(double r, int nint, double rmax, const double* __restrict__ f) {
  const double h = rmax / (nint - 1);
  const double c1oh = 1.0 / h;
  const double c1o2h2 = c1oh * c1oh * 0.5;
  int i0 = (int)(1.5 + r / h);
  i0 = min(max(i0, 1), nint);
  const double r0 = (i0 - 1) * h;
  const double f0 = f[i0];
  const bool lo = r < r0;
  const double f1 = f[lo ? i0 - 1 : i0 + 1];
  const double f2 = f[lo ? i0 + 1 : i0 - 1];
  const double aa = (f2 - 2.0 * f0 + f1) * c1o2h2;
  const double bb = ((lo ? f2 : f1) - f0) * c1oh - aa * (2.0 * r0 + h);
  const double cc = f0 - r0 * (bb + r0 * aa);
  return r * (aa * r + bb) + cc;
}

// Pair potential of the U+ integral (Select_Pot subset + Morse).
EP_DEV double pot_eval(const PotDev& v, double r) {
  return ep_pair_potential(v.kind, v.r_cutoff, v.umax, v.par, &v.s, r);
}

// Column mapping of the impurity and energy kernels: a warp takes 32
// neighbouring (x, z) columns and its block's warps share the rows y of the
// block's chunk, so the coordinates x and z (and what depends on them alone)
// are per column instead of per point, no point needs an index division, and
// the neighbour rows a gradient reads are shared by the block's warps.
// setup(x index, z index, offset of (x, 0, z)) opens a column; body(y index,
// offset) takes a point; done() closes the column.  Blocks are 32 x 8 threads;
// UNROLL rows are in flight at once.
struct ColGrid {
  int groups;  // groups of 32 columns
  int rows;    // rows of a y chunk (blockIdx.y)
};
template <int UNROLL = 1, class Setup, class Body, class Done>
EP_DEV void columns(const Geo& g, const ColGrid& cg, Setup&& setup, Body&& body, Done&& done) {
  const int ncol = g.nx * g.nz;
  const int y0 = blockIdx.y * cg.rows, y1 = min(y0 + cg.rows, g.ny);
  for (int grp = blockIdx.x; grp < cg.groups; grp += gridDim.x) {
    const int col = grp * 32 + (int)threadIdx.x;
    if (col < ncol) {
      const int iz = col / g.nx, ix = col - iz * g.nx;
      const long long p0 = ix + (long long)g.nx * g.ny * iz;
      setup(ix, iz, p0);
#pragma unroll UNROLL
      for (int iy = y0 + (int)threadIdx.y; iy < y1; iy += 8) body(iy, p0 + (long long)g.nx * iy);
      done();
    }
  }
}

// V_Pi and the P-state Delta of updatepoten at |x - r_imp|^2 = rr2.  update()
// (potenimp.f90:588-632) evaluates, in both of its branches, the parabola
// through f(i0-1), f(i0), f(i0+1); it is tabulated per node i0 (upload_tables)
// about the node r0 = (i0-1) h.  Coefficients about r = 0, as update() forms
// them, cancel beside a cut-off core (1000 K over h = 0.01 A: aa r^2 = 5e7, 1e-8
// K of rounding at every point within h of it: the excited-impurity job's
// energies and psi were off by 4e-14, and by 2.6e-14 with another order of
// operations).  i0 is update()'s: where r / h falls within 1e-5 of a switch of
// the parabola, or r <= 1e-3 or the table's end, it is taken with update()'s
// quotient.
struct ImpTable {
  const double* coef;  // [npot + 2][8]: f0, slope and curvature / 2 of V_Pi, then of V_Sigma - V_Pi
  int npot;
  double h, rh;        // spacing and its reciprocal
  double umax_sigma;
};
EP_DEV void imp_field(const ImpTable& t, double rr2, double& vp, double& dl) {
  const double r = sqrt(rr2);
  const double q = fma(r, t.rh, 1.5);
  int i0 = (int)q;
  double di = (double)i0;
  // compared in FP32 and, for rr2 > 1.1e-6, by the exponent word (an FP64
  // comparison is an FP64-pipe operation)
  const float fr = (float)(q - di);
  const bool plain = __double2hiint(rr2) > 0x3eb27476 && fr > 1e-5f && fr < 1.0f - 1e-5f && i0 < t.npot;
  if (!plain) {
    i0 = min(max((int)(1.5 + r / t.h), 1), t.npot);
    di = (double)i0;
  }
  const double2* c = reinterpret_cast<const double2*>(t.coef + i0 * 8);
  const double2 c0 = __ldg(c), c1 = __ldg(c + 1), c2 = __ldg(c + 2);
  const double d = fma(1.0 - di, t.h, r);
  vp = d * (c1.x * d + c0.y) + c0.x;
  dl = d * (c2.y * d + c2.x) + c1.y;
  // A zero numerator takes the division's slow path, and with one pair
  // potential for both channels every point has one: 1 is divided in its
  // place, opaque to the compiler, which otherwise folds the choice back into
  // dl / rr2 (96 x 160 x 192 double-float 412 -> 344 us).
  const bool zero = ((__double2hiint(dl) & 0x7fffffff) | __double2loint(dl)) == 0;
  double num = zero ? 1.0 : dl;
  asm volatile("" : "+d"(num));
  const double quo = num / rr2;
  if (!(plain || r > 1e-3)) dl = t.umax_sigma;
  else if (!zero) dl = quo;
}

// A double as a field value.  The double-float split rounds to 24 bits in the
// integer pipe (as (float)d rounds but for ties) and takes two FP64-pipe
// operations, the difference and its conversion, where the converting
// constructor takes four; values outside the FP32 range's middle use that.
template <class T> EP_DEV T to_field(double d) { return (T)d; }
template <> EP_DEV dfloat to_field<dfloat>(double d) {
  const long long b = __double_as_longlong(d);
  if ((b << 1) == 0) return dfloat(0.0f, 0.0f);
  const unsigned e = (unsigned)(b >> 52) & 0x7ffu;
  if (e - 923u > 226u) return dfloat(d);  // below 2^-100 or above 2^126, Inf, NaN
  const long long rb = (b + 0x10000000ll) & ~0x1fffffffll;
  const unsigned m = (unsigned)((rb & 0x7fffffffffffffffll) >> 29) - (896u << 23);
  return dfloat(__uint_as_float(m | ((unsigned)(rb >> 32) & 0x80000000u)), (float)(d - __longlong_as_double(rb)));
}

// The field of the P-state impurity.  Bound by the FP64 pipe (about 50
// operations a point with double-float stores, 44 in FP64; the table
// arithmetic, coordinates and two divisions per point were 120): 96 x 160 x 192
// double-float, two channels, 559 -> 366 us, 64 x 64 x 80 FP64 69 -> 44.  With r
// and 1 / r^2 from one reciprocal root it took 320 and 37 us, but 1 / r^2 lost
// two bits.
template <class T>
__global__ void __launch_bounds__(256) k_potenimp(Geo g, ColGrid cg, double xmax, double ymax, double zmax, double hx,
                                                  double hy, double hz, double r0, double r1, double r2, ImpTable t,
                                                  double2 iv0, double2 iv1, double2 iv2, double2 iv3, double2 iv4,
                                                  double2 iv5, T* __restrict__ vpi, T* __restrict__ delta,
                                                  T* __restrict__ uimp) {
  extern __shared__ __align__(16) unsigned char smraw[];
  double2* ys = reinterpret_cast<double2*>(smraw);  // y - r_imp,y of the chunk's rows and its square
  const int y0 = blockIdx.y * cg.rows;
  for (int i = threadIdx.x + 32 * threadIdx.y; i < cg.rows; i += 32 * blockDim.y) {
    const double yy = coord(ymax, hy, y0 + i) - r1;
    ys[i] = make_double2(yy, __dmul_rn(yy, yy));
  }
  __syncthreads();
  double xx = 0, zz = 0, x2 = 0, z2 = 0, oxc = 0, oyc = 0, exc = 0, eyc = 0;
  columns(
      g, cg,
      [&](int ix, int iz, long long) {
        xx = coord(xmax, hx, ix) - r0;
        zz = coord(zmax, hz, iz) - r2;
        x2 = __dmul_rn(xx, xx);
        z2 = __dmul_rn(zz, zz);
        oxc = iv0.x * xx + iv4.x * zz;
        oyc = iv0.y * xx + iv4.y * zz;
        exc = iv1.x * xx + iv5.x * zz;
        eyc = iv1.y * xx + iv5.y * zz;
      },
      [&](int iy, long long p) {
        const double yy = ys[iy - y0].x;
        const double rr2 = __dadd_rn(x2, __dadd_rn(ys[iy - y0].y, z2));  // rr2_nc's order
        double vp, dl;
        imp_field(t, rr2, vp, dl);
        const double ox = iv2.x * yy + oxc, oy = iv2.y * yy + oyc, ex = iv3.x * yy + exc, ey = iv3.y * yy + eyc;
        const double u = vp + dl * ((ox * ox + oy * oy) + (ex * ex + ey * ey));
        if (vpi) {
          vpi[p] = to_field<T>(vp);
          delta[p] = to_field<T>(dl);
        }
        // fmin(u, 1000) by the exponent word (0x408f4000: 1000; a NaN gives 1000)
        const int hu = __double2hiint(u);
        uimp[p] = to_field<T>(hu < 0x408f4000 && (hu & 0x7ff00000) != 0x7ff00000 ? u : fmin(u, 1000.0));
      },
      [] {});
}

// D-state angular factors at x = r - rimp (potenimp.f90:68-117): the d
// harmonics a = (d1..d5) and the upper triangle of P in DGram's order.
EP_DEV void dstate_factors(double xx, double yy, double zz, double (&a)[5], double (&P)[15]) {
  const double sqr3 = sqrt(3.0), sqr3o2 = sqrt(3.0) / 2.0, insqr3 = 1.0 / sqrt(3.0), in3 = 1.0 / 3.0;
  const double d0 = xx * xx + yy * yy + zz * zz;
  const double d1 = sqr3 * xx * yy, d2 = sqr3 * yy * zz, d3 = (-xx * xx - yy * yy + 2.0 * zz * zz) / 2.0;
  const double d4 = sqr3 * xx * zz, d5 = sqr3o2 * (xx * xx - yy * yy);
  a[0] = d1; a[1] = d2; a[2] = d3; a[3] = d4; a[4] = d5;
  const double sd1 = d1 * d1, sd2 = d2 * d2, sd4 = d4 * d4, sd5 = d5 * d5;
  const double s35 = d3 + insqr3 * d5, f35 = d3 - insqr3 * d5;
  P[0] = in3 * (sd2 + sd4 + 4.0 * sd5);                 // (1,1)
  P[1] = -4.0 * in3 * d1 * d2 + insqr3 * d4 * d0;       // (1,2)
  P[2] = -2.0 * insqr3 * d2 * d4;                       // (1,3)
  P[3] = -4.0 * in3 * d1 * d4 + insqr3 * d2 * d0;       // (1,4)
  P[4] = -4.0 * in3 * d1 * d5;                          // (1,5)
  P[5] = in3 * (sd1 + sd4) + s35 * s35;                 // (2,2)
  P[6] = insqr3 * d1 * d4 - d2 * s35;                   // (2,3)
  P[7] = -4.0 * in3 * d2 * d4 + insqr3 * d1 * d0;       // (2,4)
  P[8] = -d1 * d4 - insqr3 * d2 * s35;                  // (2,5)
  P[9] = sd4 + sd2;                                     // (3,3)
  P[10] = insqr3 * d1 * d2 - d4 * f35;                  // (3,4)
  P[11] = insqr3 * (sd2 - sd4);                         // (3,5)
  P[12] = in3 * (sd1 + sd2) + f35 * f35;                // (4,4)
  P[13] = d1 * d2 + insqr3 * d4 * f35;                  // (4,5)
  P[14] = in3 * (sd2 + sd4 + 4.0 * sd1);                // (5,5)
}

template <class T>
__global__ void k_potenimp_d(Geo g, double xmax, double ymax, double zmax, double hx, double hy, double hz,
                             double r0, double r1, double r2, const double* __restrict__ potdel,
                             const double* __restrict__ potpidel, const double* __restrict__ potsigdel, int npot,
                             double rmax, double umax_pi, double umax_sigma, const __grid_constant__ DGram G,
                             T* __restrict__ delta, T* __restrict__ pidel, T* __restrict__ sigdel,
                             T* __restrict__ uimp) {
  const double gtr = G.g[0] + G.g[5] + G.g[9] + G.g[12] + G.g[14];
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < g.N; p += (long long)gridDim.x * blockDim.x) {
    int ix, iy, iz;
    idx3(g, p, ix, iy, iz);
    const double xx = coord(xmax, hx, ix) - r0;
    const double yy = coord(ymax, hy, iy) - r1;
    const double zz = coord(zmax, hz, iz) - r2;
    const double rr2 = rr2_nc(xx, yy, zz);
    const double r4 = rr2 * rr2;
    const double r = sqrt(rr2);
    const double dl = interp_update(r, npot, rmax, potdel);
    double pd = umax_pi, sd = umax_sigma;
    if (r > 1e-3) {
      pd = interp_update(r, npot, rmax, potpidel) / r4;
      sd = interp_update(r, npot, rmax, potsigdel) / r4;
    }
    double a[5], P[15];
    dstate_factors(xx, yy, zz, a, P);
    double qs = 0.0, qp = 0.0;
    int k = 0;
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = i; j < 5; ++j, ++k) {
        qs += a[i] * a[j] * G.g[k];
        qp += P[k] * G.g[k];
      }
    const double u = dl * gtr + pd * qs + sd * qp;
    delta[p] = (T)dl;
    pidel[p] = (T)pd;
    sigdel[p] = (T)sd;
    uimp[p] = (T)fmin(u, 1000.0);
  }
}

template <class T>
__global__ void k_impmoments_d(Geo g, const T* __restrict__ den, const T* __restrict__ dxd,
                               const T* __restrict__ dyd, const T* __restrict__ dzd, const T* __restrict__ uimp,
                               const T* __restrict__ delta, const T* __restrict__ pidel,
                               const T* __restrict__ sigdel, double xmax, double ymax, double zmax, double hx,
                               double hy, double hz, double r0, double r1, double r2, int izlo, int izhi,
                               double* __restrict__ partials) {
  Acc<double> acc[18];
  for (long long p = blockIdx.x * (long long)blockDim.x + threadIdx.x; p < g.N; p += (long long)gridDim.x * blockDim.x) {
    int ix, iy, iz;
    idx3(g, p, ix, iy, iz);
    const double u = dbl(uimp[p]);
    acc[0].add((double)dxd[p] * u);
    acc[1].add((double)dyd[p] * u);
    if (iz >= izlo && iz < izhi) acc[2].add((double)dzd[p] * u);
    const double xx = coord(xmax, hx, ix) - r0, yy = coord(ymax, hy, iy) - r1, zz = coord(zmax, hz, iz) - r2;
    const double rho = dbl(den[p]);
    const double dvd = (double)delta[p] * rho, dv1 = (double)pidel[p] * rho, dv2 = (double)sigdel[p] * rho;
    double a[5], P[15];
    dstate_factors(xx, yy, zz, a, P);
    int k = 0;
#pragma unroll
    for (int i = 0; i < 5; ++i)
#pragma unroll
      for (int j = i; j < 5; ++j, ++k) acc[3 + k].add(P[k] * dv2 + a[i] * a[j] * dv1 + (i == j ? dvd : 0.0));
  }
  block_reduce_store_acc<18>(acc, partials);
}

// FP32 engine, P state: the impurity field in FP32 arithmetic (float tables,
// 1/h and the coordinates rounded once; a double per point would run on the
// FP64 pipe at 1/64 of the FP32 rate).  update() (potenimp.f90:588-632)
// evaluates, in both of its branches, the parabola through f(i0-1), f(i0),
// f(i0+1); here it is evaluated about r0 = (i0-1) h, which avoids the
// cancellation of its global coefficients in FP32.
EP_DEV float interp_update_f(float r, int nint, float h, float rh, const float* __restrict__ f) {
  int i0 = (int)(1.5f + r * rh);
  i0 = min(max(i0, 1), nint);
  const float r0 = (float)(i0 - 1) * h;
  const float fm = f[i0 - 1], f0 = f[i0], fp = f[i0 + 1];
  const float aa = (fp - 2.0f * f0 + fm) * (0.5f * rh * rh);
  const float b = (fp - f0) * rh - aa * h;
  const float d = r - r0;
  return f0 + d * (b + aa * d);
}

// The coordinates from the impurity are FP64 differences rounded once, per
// column and per row (in FP32 their rounding at the box's size, 2e-6 A, times
// the slope of a cut-off core was 2e-5 of the field's maximum).
static __global__ void __launch_bounds__(256)
    k_potenimp_f(Geo g, ColGrid cg, double xmax, double ymax, double zmax, double hx, double hy, double hz, double r0,
                 double r1, double r2, const float* __restrict__ potpi, const float* __restrict__ potdel, int npot,
                 float h, float rh, float umax_sigma, float2 iv0, float2 iv1, float2 iv2, float2 iv3, float2 iv4,
                 float2 iv5, float* __restrict__ vpi, float* __restrict__ delta, float* __restrict__ uimp) {
  extern __shared__ __align__(16) unsigned char smraw[];
  float* ys = reinterpret_cast<float*>(smraw);  // y - r_imp,y of the chunk's rows
  const int y0 = blockIdx.y * cg.rows;
  for (int i = threadIdx.x + 32 * threadIdx.y; i < cg.rows; i += 32 * blockDim.y)
    ys[i] = (float)(coord(ymax, hy, y0 + i) - r1);
  __syncthreads();
  float xx = 0, zz = 0;
  columns<4>(
      g, cg,
      [&](int ix, int iz, long long) {
        xx = (float)(coord(xmax, hx, ix) - r0);
        zz = (float)(coord(zmax, hz, iz) - r2);
      },
      [&](int iy, long long p) {
        const float yy = ys[iy - y0];
        const float rr2 = xx * xx + (yy * yy + zz * zz);
        const float r = sqrtf(rr2);
        const float vp = interp_update_f(r, npot, h, rh, potpi);
        const float dl = r > 1e-3f ? interp_update_f(r, npot, h, rh, potdel) / rr2 : umax_sigma;
        const float ox = iv0.x * xx + iv2.x * yy + iv4.x * zz, oy = iv0.y * xx + iv2.y * yy + iv4.y * zz;
        const float ex = iv1.x * xx + iv3.x * yy + iv5.x * zz, ey = iv1.y * xx + iv3.y * yy + iv5.y * zz;
        const float u = vp + dl * ((ox * ox + oy * oy) + (ex * ex + ey * ey));
        if (vpi) {
          vpi[p] = vp;
          delta[p] = dl;
        }
        uimp[p] = fminf(u, 1000.0f);
      },
      [] {});
}

// Exact or double-float products of field values for the sums: FP64 in FP64;
// a pair of FP32 values (the product and its FMA error, 2^-47 of it at most)
// for FP32 and double-float fields, whose sums are FP32 pairs (ep_reduce.cuh).
EP_DEV double wmul(double a, double b) { return a * b; }
EP_DEV dfloat wmul(dfloat a, dfloat b) { return a * b; }
EP_DEV dfloat wmul(float a, float b) {
  const float p = __fmul_rn(a, b);
  return dfloat(p, __fmaf_rn(a, b, -p));
}
EP_DEV dfloat wmul(dfloat a, float b) {
  const float p = __fmul_rn(a.hi, b);
  return dd_fast2sum(p, __fmaf_rn(a.lo, b, __fmaf_rn(a.hi, b, -p)));
}
EP_DEV dfloat wmul(float a, dfloat b) { return wmul(b, a); }
// The value of a per-thread sum in the arithmetic of its terms.
EP_DEV double wvalue(const Neumaier<double>& a) { return a.s + a.c; }
EP_DEV dfloat wvalue(const Kahan<dfloat>& a) { return dd_fast2sum(a.s, a.c); }
EP_DEV float wvalue(const Kahan<float>& a) { return a.s - a.c; }
EP_DEV float fmul1(float a, float b) { return a * b; }

// P state: forceimp sums and the six moments (the matrix of the internal
// variables).  Along a column only y varies, so a point adds four moments of
// den Delta and den V_Pi (1, y, y^2) and the column's x and z factors are
// applied once per column: seven products and seven compensated sums a point
// in the fields' own arithmetic (FP32; pairs of FP32 values in double-float;
// FP64).  In double-float a thread's sums are pairs, whose roundings (2^-46 of a
// product, 2^-49 of a sum) average out over points and threads, and the block's
// are FP64: the force is within 5e-17 of its terms' magnitudes, the moments
// within 1e-16 (2e-16 with the block's sums in pairs too).  The FP64
// conversions, products and sums of the one-point form (about 120 operations a
// point on the FP64 pipe) go: 96 x 160 x 192 896 -> 54 us; FP64 64 x 64 x 80 361
// -> 111 us; FP32 256 x 256 x 320 168 -> 120 us (memory: seven fields read).  MOM = false: the force alone
// (three sums, four fields read).
template <class T, bool MOM>
__global__ void __launch_bounds__(256) k_impmoments(Geo g, ColGrid cg, const T* __restrict__ den,
                                                    const T* __restrict__ dxd, const T* __restrict__ dyd,
                                                    const T* __restrict__ dzd, const T* __restrict__ uimp,
                                                    const T* __restrict__ vpi, const T* __restrict__ delta,
                                                    double xmax, double ymax, double zmax, double hx, double hy,
                                                    double hz, double r0, double r1, double r2, int izlo, int izhi,
                                                    double* __restrict__ partials) {
  constexpr bool F = std::is_same<T, float>::value;
  auto mul = [](T a, T b) {
    if constexpr (F) return fmul1(a, b);
    else return wmul(a, b);
  };
  extern __shared__ __align__(16) unsigned char smraw[];
  T* ys = reinterpret_cast<T*>(smraw);  // y - r_imp,y of the chunk's rows
  const int y0 = blockIdx.y * cg.rows;
  for (int i = threadIdx.x + 32 * threadIdx.y; i < cg.rows; i += 32 * blockDim.y)
    ys[i] = T(coord(ymax, hy, y0 + i) - r1);
  __syncthreads();
  constexpr int NQ = MOM ? 9 : 3;
  Acc<T> acc[NQ];
  Acc<T> sv, s0, s1, s2;  // along the column: den V_Pi and den Delta (1, y, y^2)
  T xx = T(0), zz = T(0);
  bool fz = false;
  columns<F ? 4 : 2>(
      g, cg,
      [&](int ix, int iz, long long) {
        xx = T(coord(xmax, hx, ix) - r0);
        zz = T(coord(zmax, hz, iz) - r2);
        fz = iz >= izlo && iz < izhi;
        sv = s0 = s1 = s2 = Acc<T>();
      },
      [&](int iy, long long p) {
        const T u = uimp[p];
        acc[0].add(mul(dxd[p], u));
        acc[1].add(mul(dyd[p], u));
        if (fz) acc[2].add(mul(dzd[p], u));
        if constexpr (MOM) {
          const T a1 = den[p], yy = ys[iy - y0], d = mul(a1, delta[p]), dy = mul(d, yy);
          sv.add(mul(a1, vpi[p]));
          s0.add(d);
          s1.add(dy);
          s2.add(mul(dy, yy));
        }
      },
      [&] {
        if constexpr (MOM) {
        const T V = wvalue(sv), D = wvalue(s0), Dx = mul(xx, D), Dz = mul(zz, D), Dy = wvalue(s1);
        acc[3].add(V);
        acc[3].add(mul(xx, Dx));
        acc[4].add(mul(xx, Dy));
        acc[5].add(mul(xx, Dz));
        acc[6].add(V);
        acc[6].add(wvalue(s2));
        acc[7].add(mul(zz, Dy));
        acc[8].add(V);
        acc[8].add(mul(zz, Dz));
        }
      });
  if constexpr (std::is_same<T, dfloat>::value) {
    double tot[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) tot[q] = acc[q].get();
    block_reduce_store_sums<NQ>(tot, partials);
  } else {
    block_reduce_store_acc<NQ>(acc, partials);
  }
}

// Sum of |psi|^2 (block partials).
template <class T>
__global__ void k_normsum(const C2<T>* __restrict__ psi, long long N, double* __restrict__ partials) {
  Acc<double> acc[1];
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const C2<T> v = psi[i];
    acc[0].add(dbl(v.x) * dbl(v.x) + dbl(v.y) * dbl(v.y));
  }
  block_reduce_store_acc<1>(acc, partials);
}

// Running sum of w_k (a_k - b_k) of complex values: paired FMAs, or the
// unnormalised double-float accumulation of ep_dd.cuh.
template <class T> struct DiffSum {
  C2<T> s;
  EP_DEV DiffSum() : s(cmk<T>(T(0), T(0))) {}
  EP_DEV void add(T w, C2<T> a, C2<T> b) { s = vfma(w, vsub(a, b), s); }
  EP_DEV C2<T> value() const { return s; }
};
#if defined(__CUDA_ARCH__)
template <> struct DiffSum<dfloat> {
  dd2_acc s;
  EP_DEV DiffSum() : s{make_float2(0.0f, 0.0f), make_float2(0.0f, 0.0f)} {}
  EP_DEV void add(dfloat w, dfloat2 a, dfloat2 b) {
    float2 ph, pl;
    dd2_wdiff(w, a, b, ph, pl);
    dd2_add(s, ph, pl);
  }
  EP_DEV dfloat2 value() const { return dd2_value(s); }
};
#endif

// Complex first derivative at c along an axis of n points with element stride
// st (index i), from global memory.  LANE: the index differs across the warp
// (x), so each neighbour wraps by a selection; else (y, z) whole warps are
// inside and step two pointers.
template <class T, bool LANE>
EP_DEV C2<T> d1c_global(const C2<T>* __restrict__ c, int i, int n, long long st, const T* w, int R, int periodic) {
  DiffSum<T> s;
  const C2<T> zero = cmk<T>(T(0), T(0));
  if (!LANE && i >= R && i < n - R) {
    const C2<T>*u = c + st, *d = c - st;
    for (int k = 1; k <= R; ++k, u += st, d -= st) s.add(w[k], __ldg(u), __ldg(d));
  } else {
    for (int k = 1; k <= R; ++k) {
      const bool ou = i + k >= n, od = i - k < 0;
      const long long u = ou ? k - n : k, d = od ? n - k : -k;
      s.add(w[k], ou && !periodic ? zero : __ldg(c + u * st), od && !periodic ? zero : __ldg(c + d * st));
    }
  }
  return s.value();
}

// 1 + tanh(beta (den - den_m)) of the solid penalty.  For 2 beta (den - den_m)
// < -25 (a liquid's density: -28) it is 2 e / (1 + e), e = exp(2 beta (den -
// den_m)) < 1.4e-11, from the FP32 exponential: its error, below 3e-6 e, is
// under the 1.1e-16 that the cancellation in FP64's 1 + tanh leaves there (a
// droplet's sum: 9e-9 of it against 3e-8).
EP_DEV double one_plus_tanh(const Phys& ph, double dn) {
  const float y = (float)(2.0 * ph.beta * (dn - ph.den_m));
  if (y < -25.0f) {
    const float e = expf(y);
    return (double)(2.0f * e);
  }
  return 1.0 + tanh(ph.beta * (dn - ph.den_m));
}
// The same in pairs (an FP32 argument, whose rounding of 2 beta den_m alone is
// 4e-7 of e, put 3.7e-7 into every sum; FP64's 1 + tanh leaves 3e-8).
template <class T>
EP_DEV dfloat one_plus_tanh_f(const Phys& ph, T dn) {
  const dfloat y = dfloat(2.0f, 0.0f) * ph.d.beta * (dfloat(dn) - ph.d.den_m);
  if (y.hi < -25.0f) {
    const dfloat e = dd_exp(y);
    return dfloat(2.0f, 0.0f) * (e - e * e);  // 2 e / (1 + e)
  }
  return dfloat(1.0 + tanh(ph.beta * (dbl(dn) - ph.den_m)));
}

// Energy integrals.  W: the arithmetic of the terms (W = double: FP64; W =
// dfloat: pairs of FP32 values, exact products of FP32 fields, 2^-45 for
// double-float ones, summed in FP32 pairs by a thread and in FP64 by a block:
// each sum within about 1e-16 of its terms' magnitudes, as the FP64 form, but
// the Morse U+ of FP32 fields, 3e-13; the two powers of the coarse-grained
// density apart, whose FP64 coefficients cancel).  The FP64 form of every
// engine was bound by the FP64 pipe (about 380 operations a point:
// conversions, tanh, eight Neumaier sums); FP32 fields in pairs leave the pipe
// to a U+ that is no Morse potential (its distance and pair potential).
// 128^3, impurity with a Morse U+: FP32 1133 -> 174 us, double-float 1333 ->
// 286, FP64 1260 -> 953 (64 x 64 x 80: 460 -> 200).  The caller falls back to W = double where the pairs' FP32
// range does not hold the sums.
template <class T, class W>
__global__ void __launch_bounds__(256) k_energy(Geo g, ColGrid cg, const __grid_constant__ FdW<T> fd, Phys ph, const C2<T>* __restrict__ psi,
                                                const T* __restrict__ den, const T* __restrict__ dencg,
                                                const T* __restrict__ delj4, const T* __restrict__ falfs,
                                                const T* __restrict__ dxd, const T* __restrict__ dyd,
                                                const T* __restrict__ dzd, const T* __restrict__ ix_,
                                                const T* __restrict__ iy_, const T* __restrict__ iz_,
                                                const T* __restrict__ uimp, double xmax, double ymax, double zmax,
                                                double hx, double hy, double hz, double r0, double r1, double r2,
                                                double zexc, const __grid_constant__ PotDev vplus, int impurity,
                                                double* __restrict__ partials) {
  constexpr bool D64 = std::is_same<W, double>::value;
  Acc<W> acc[D64 ? 8 : 9];  // pairs: n cg^2 and, as the ninth, n cg^3
  const bool otc = ph.core == 1;
  // FP32 fields: a Morse U+ in pairs of FP32 values (2^-36 and better; in FP64
  // its root and exponential were 200 us of the 255 at 128^3)
  const bool pair_u = std::is_same<T, float>::value && !D64 && vplus.kind == EP_POT_MORSE && zexc <= 0.0;
  // r in FP64 is needed for the exclusion radius and any other U+ that is not
  // zero everywhere
  const bool need_r = impurity && !pair_u && (vplus.kind != EP_POT_NULL || !(zexc <= 0.0));
  extern __shared__ __align__(16) unsigned char smraw[];
  dfloat* ys = reinterpret_cast<dfloat*>(smraw);  // r_imp,y - y of the chunk's rows (pair_u)
  const int y0 = blockIdx.y * cg.rows;
  dfloat ac(0.0f, 0.0f), De = ac, re = ac, al = ac;
  if (pair_u) {
    De = dfloat(vplus.par[0]);
    re = dfloat(vplus.par[1]);
    al = dfloat(vplus.par[2]);
    for (int i = threadIdx.x + 32 * threadIdx.y; i < cg.rows; i += 32 * blockDim.y)
      ys[i] = dfloat(r1 - coord(ymax, hy, y0 + i));
    __syncthreads();
  }
  int ix = 0, iz = 0;
  double a2 = 0, c2 = 0;
  const long long sz = (long long)g.nx * g.ny;
  columns(
      g, cg,
      [&](int i, int k, long long) {
        ix = i;
        iz = k;
        if (need_r) {
          const double a = r0 - coord(xmax, hx, ix), c = r2 - coord(zmax, hz, iz);
          a2 = __dmul_rn(a, a);
          c2 = __dmul_rn(c, c);
        } else if (pair_u) {
          const double a = r0 - coord(xmax, hx, ix), c = r2 - coord(zmax, hz, iz);
          ac = dfloat(a * a + c * c);
        }
      },
      [&](int iy, long long p) {
        const C2<T> dx = d1c_global<T, true>(psi + p, ix, g.nx, 1, fd.w1[0], fd.R, fd.periodic);
        const C2<T> dy = d1c_global<T, false>(psi + p, iy, g.ny, (long long)g.nx, fd.w1[1], fd.R, fd.periodic);
        const C2<T> dz = d1c_global<T, false>(psi + p, iz, g.nz, sz, fd.w1[2], fd.R, fd.periodic);
        const T dn = den[p], cg_ = dencg[p], lj = delj4[p];
        bool inside = impurity != 0;
        double r = 0.0;
        if (need_r) {
          const double b = r1 - coord(ymax, hy, iy);
          r = sqrt(__dadd_rn(__dadd_rn(a2, __dmul_rn(b, b)), c2));
          inside = inside && r >= zexc;
        }
        if constexpr (D64) {
          const double n = dbl(dn), c = dbl(cg_);
          acc[0].add((dbl(dx.x) * dbl(dx.x) + dbl(dx.y) * dbl(dx.y)) +
                     (dbl(dy.x) * dbl(dy.x) + dbl(dy.y) * dbl(dy.y)) +
                     (dbl(dz.x) * dbl(dz.x) + dbl(dz.y) * dbl(dz.y)));
          acc[1].add(dbl(lj) * n);
          acc[2].add(n * (c * c) * (0.5 * ph.cp4 + (1.0 / 3.0) * ph.cpp4 * c));
          if (otc)
            acc[3].add(dbl(falfs[p]) *
                       (dbl(dxd[p]) * dbl(ix_[p]) + dbl(dyd[p]) * dbl(iy_[p]) + dbl(dzd[p]) * dbl(iz_[p])));
          acc[4].add(n * one_plus_tanh(ph, n));
          if (inside) {
            acc[5].add(n * dbl(uimp[p]));
            if (vplus.kind != EP_POT_NULL) acc[6].add(n * pot_eval(vplus, r));
          }
          acc[7].add(n);
        } else {
          acc[0].add(wmul(dx.x, dx.x));
          acc[0].add(wmul(dx.y, dx.y));
          acc[0].add(wmul(dy.x, dy.x));
          acc[0].add(wmul(dy.y, dy.y));
          acc[0].add(wmul(dz.x, dz.x));
          acc[0].add(wmul(dz.y, dz.y));
          acc[1].add(wmul(lj, dn));
          const dfloat nc2 = wmul(wmul(cg_, cg_), dn);
          acc[2].add(nc2);
          acc[8].add(wmul(nc2, cg_));
          if (otc)
            acc[3].add(wmul((wmul(dxd[p], ix_[p]) + wmul(dyd[p], iy_[p])) + wmul(dzd[p], iz_[p]), falfs[p]));
          acc[4].add(wmul(one_plus_tanh_f(ph, dn), dn));
          if (inside) {
            acc[5].add(wmul(dn, uimp[p]));
            if (pair_u) {
              const dfloat b = ys[iy - y0], rd = sqrt(ac + b * b);
              const float rc = (float)vplus.r_cutoff;
              dfloat V;
              if (rc > 0.0f && fabsf(rd.hi - rc) <= 1e-5f * rc) V = dfloat(pot_eval(vplus, (double)rd));
              else if (rd.hi < rc) V = dfloat(vplus.umax);
              else {
                const dfloat e = dd_exp(-(al * (rd - re)));
                V = De * (e * e - dfloat(2.0f, 0.0f) * e);
              }
              acc[6].add(wmul(V, dn));
            } else if (vplus.kind != EP_POT_NULL) {
              acc[6].add(wmul(dfloat(pot_eval(vplus, r)), dn));
            }
          }
          acc[7].add(dfloat(dn));
        }
      },
      [] {});
  if constexpr (D64) {
    block_reduce_store_acc<8>(acc, partials);
  } else {
    double tot[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) tot[q] = acc[q].get();
    tot[2] = 0.5 * ph.cp4 * tot[2] + (1.0 / 3.0) * ph.cpp4 * acc[8].get();
    block_reduce_store_sums<8>(tot, partials);
  }
}

// ---------------------------------------------------------------------------
// Sine integral Si(x): power series for |x| <= 4, else the continued fraction
// of E1(ix) by the modified Lentz method (Numerical Recipes 6.9).
EP_DEV double si_dev(double x) {
  const double ax = fabs(x);
  double r;
  if (ax <= 4.0) {
    double term = ax, sum = ax;
    const double x2 = ax * ax;
    for (int k = 1; k < 60; ++k) {
      term *= -x2 / ((2.0 * k) * (2.0 * k + 1.0));
      const double t = term / (2.0 * k + 1.0);
      sum += t;
      if (fabs(t) < 1e-18 * fabs(sum)) break;
    }
    r = sum;
  } else {
    double br = 1.0, bi = ax, cr = 1e300, ci = 0.0;
    double den = br * br + bi * bi;
    double dr = br / den, di = -bi / den;
    double hr = dr, hi = di;
    for (int i = 2; i < 1000; ++i) {
      const double a = -(double)(i - 1) * (double)(i - 1);
      br += 2.0;
      // d = 1/(a*d + b)
      const double tr = a * dr + br, ti = a * di + bi;
      den = tr * tr + ti * ti;
      dr = tr / den;
      di = -ti / den;
      // c = b + a/c
      const double cd = cr * cr + ci * ci;
      const double ncr = br + a * cr / cd, nci = bi - a * ci / cd;
      cr = ncr;
      ci = nci;
      const double er = cr * dr - ci * di, ei = cr * di + ci * dr;
      const double nhr = hr * er - hi * ei, nhi = hr * ei + hi * er;
      hr = nhr;
      hi = nhi;
      if (fabs(er - 1.0) + fabs(ei) < 3e-16) break;
    }
    double s, c;
    sincos(ax, &s, &c);
    // h *= (cos x - i sin x)
    const double fi = hi * c - hr * s;
    r = 1.5707963267948966192313216916397514 + fi;
  }
  return x < 0 ? -r : r;
}

EP_DEV double ipow(double x, int n) {
  double r = 1.0;
  for (int i = 0; i < n; ++i) r *= x;
  return r;
}

// Integral of sin(a t)/t^11 and sin(a t)/t^5 from x to infinity, closed forms
// of fforma.f90:73-137 (integration by parts down to Si).
EP_DEV double sinint_tail(double a, double x) {
  const double res = si_dev(a * x);
  return a > 0.0 ? 1.5707963267948966192313216916397514 - res : 1.5707963267948966192313216916397514 + res;
}
EP_DEV double sinx11_dev(double a, double x) {
  const double y = a * x, y2 = y * y;
  const double bd = 40320.0 - 720.0 * y2 + 24.0 * (y2 * y2) - 2.0 * (y2 * y2 * y2) + (y2 * y2 * y2 * y2);
  const double cd = 362880.0 - 5040.0 * y2 + 120.0 * (y2 * y2) - 6.0 * (y2 * y2 * y2) + (y2 * y2 * y2 * y2);
  double s, c;
  sincos(y, &s, &c);
  const double res1 = (a * bd * c + cd * s / x) / (3628800.0 * ipow(x, 9));
  const double res2 = -(ipow(a, 10) * sinint_tail(a, x)) / 3628800.0;
  return res1 + res2;
}
EP_DEV double sinx5_dev(double a, double x) {
  const double y = a * x, y2 = y * y;
  double s, c;
  sincos(y, &s, &c);
  const double res1 = -(a * (-2.0 + y2) * c + (-6.0 + y2) * s / x) / (24.0 * x * x * x);
  const double res2 = (ipow(a, 4) * sinint_tail(a, x)) / 24.0;
  return res1 + res2;
}
EP_DEV double intcore_dev(double a, double x) {
  const double y = a * x, y2 = y * y;
  const double d0 = x / ipow(a, 5), e0 = 1.0 / ipow(a, 6);
  const double bd = -120.0 * d0 + 20.0 * (d0 * y2) - (d0 * y2 * y2);
  const double ce = 120.0 * e0 - 60.0 * (e0 * y2) + 5.0 * (e0 * y2 * y2);
  double s, c;
  sincos(y, &s, &c);
  return bd * c + ce * s;
}

template <class T>
__global__ void k_formfactors(Geo g, const double* __restrict__ px, const double* __restrict__ py,
                              const double* __restrict__ pz, int core, double h4, double eps, double sigma,
                              double bforce, double l, T* __restrict__ fvlj, T* __restrict__ wcgk,
                              T* __restrict__ kalfs) {
  const double pi = 3.14159265358979323846264338327950288;
  const double twopi = 2.0 * pi;
  const double sigma6 = ipow(sigma, 6), aux1 = 8.0 * eps, aux3 = sigma6 / ipow(h4, 6);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < g.Nh; q += (long long)gridDim.x * blockDim.x) {
    const int ipx = (int)(q % g.nxh);
    const long long r = q / g.nxh;
    const int ipy = (int)(r % g.ny), ipz = (int)(r / g.ny);
    const double a = px[ipx], b = py[ipy], c = pz[ipz];
    const double p = sqrt(__dadd_rn(__dadd_rn(__dmul_rn(a, a), __dmul_rn(b, b)), __dmul_rn(c, c)));
    double fv;
    if (fabs(p) < 1e-10) {
      fv = bforce;
    } else {
      const double a2 = twopi * p;
      const double t1 = sinx11_dev(a2, h4), t2 = sinx5_dev(a2, h4);
      if (core == 2) {
        const double v0 = aux1 * aux3 * (aux3 - 1.0) / ipow(h4, 4);
        fv = (aux1 * sigma6 * (sigma6 * t1 - t2) + v0 * intcore_dev(a2, h4)) / p;
      } else {
        fv = (aux1 * sigma6 * (sigma6 * t1 - t2)) / p;
      }
    }
    double wc = 1.0;
    if (p > 0.0) {
      const double arg = twopi * p * h4;
      double s, cc;
      sincos(arg, &s, &cc);
      const double aux = s - arg * cc;
      wc = fabs(aux) < 1e-10 ? 1.0 : 3.0 * aux / (arg * arg * arg);
    }
    const double t = pi * l * p;
    fvlj[q] = (T)fv;
    wcgk[q] = (T)wc;
    kalfs[q] = (T)exp(-(t * t));
  }
}
