// ep_xw.cuh - the X passes of poten: real transforms along contiguous lines
// with poten's and term_alfa's point-wise arithmetic around them, one kernel
// set per half-line length N2 = nx / 2 = A B (A, B <= 18).
//
// A warp owns LW lines from their spectra to their fields and back; nothing is
// shared between warps but the twiddle tables, so no block barrier follows
// their load.  A half-line transform of n = b + B a, k = ka + A kb is
//   inverse: pack    lanes over (line, k): X[k] and X[N2-k] (coalesced), both
//                    Z[k] and Z[N2-k] of c2r's packing from one product, to
//                    shared memory;
//            rows    lanes over (line, ka): B-point DFT in place, twiddles;
//            columns lanes over (line, b): A-point DFT; the pairs x = 2m, 2m+1,
//                    m = b + B a, go to the point-wise arithmetic in registers;
//   forward: columns, rows and unpack, the same in reverse order (both X[k] and
//            X[N2-k] from one product, stores coalesced).
// Columns hold the same points in either direction, so the point-wise results
// that a later transform needs again (dencg, f, the sum grad(den).I) are read
// and written by one lane each, in rows of the warp's own.
//
// The passes it replaces (a block's lines transformed by some of its warps,
// five to nine block barriers around them, real rows shared through shared
// memory) waited at their barriers: 10 to 16 stalls per issue at 96 x 120 x
// 160, 33 % of the warps resident.
#pragma once
#include "ep_fft.cuh"
#include "ep_kernels.cuh"

#define EP_XW_LENGTHS_A(X)                                                                                     \
  X(8, 2, 4) X(9, 3, 3) X(10, 2, 5) X(12, 3, 4) X(15, 3, 5) X(16, 4, 4) X(18, 3, 6) X(20, 4, 5) X(24, 4, 6)     \
  X(25, 5, 5) X(27, 3, 9) X(30, 5, 6) X(32, 4, 8) X(36, 6, 6) X(40, 5, 8)
#define EP_XW_LENGTHS_B(X)                                                                                     \
  X(45, 5, 9) X(48, 6, 8) X(50, 5, 10) X(54, 6, 9) X(60, 6, 10) X(64, 8, 8) X(72, 8, 9) X(75, 5, 15) X(80, 8, 10)
#define EP_XW_LENGTHS_C(X)                                                                                     \
  X(81, 9, 9) X(90, 9, 10) X(96, 8, 12) X(100, 10, 10) X(108, 9, 12) X(120, 10, 12)
#define EP_XW_LENGTHS_D(X)                                                                                     \
  X(128, 8, 16) X(135, 9, 15) X(144, 12, 12) X(150, 10, 15) X(160, 10, 16) X(162, 9, 18)

// Arrays of one launch (the passes use what they need).
template <class T> struct XWArgs {
  const C2<T>* in[4];
  C2<T>* out[4];
  const T *den, *dxd, *dyd, *dzd;
  T *dencg, *delj4, *pot4, *falfs, *intx, *inty, *intz, *gy, *gz, *dgx, *ualphas;
  const T* dyz;
  const C2<T>* twx;
  int keep;  // store the fields that only energy() and the caller read
};

// Host-side description of one length's kernels.
struct XWKernels {
  const void* x[4];
  int lines, threads;  // lines and threads per CTA
  size_t smem[4];
  const void* c2r;     // FP64 only; shared memory as x[3]
};
template <class T> const XWKernels* xw_part_a(int n2);
template <class T> const XWKernels* xw_part_b(int n2);
template <class T> const XWKernels* xw_part_c(int n2);
template <class T> const XWKernels* xw_part_d(int n2);
template <class T> inline const XWKernels* xw_kernels(int n2) {
  const XWKernels* k = xw_part_a<T>(n2);
  if (!k) k = xw_part_b<T>(n2);
  if (!k) k = xw_part_c<T>(n2);
  if (!k) k = xw_part_d<T>(n2);
  return k;
}

template <class T, int A, int B> struct XW {
  static constexpr int N2 = A * B, NX = 2 * N2, NXH = N2 + 1, Q = B | 1;  // Q: odd row pitch
  // 2 warps a CTA of the 16-byte types: small grids spread over more SMs (their
  // arithmetic pipe is per SM; 32 x 50 x 54 in FP64 has 85 CTAs of 4 warps)
  static constexpr int WARPS = sizeof(T) == 4 ? 4 : 2, NT = 32 * WARPS;
  static constexpr int HK = N2 / 2 + 1;  // k of a line's pack / unpack pairs
  static constexpr int rounds(int n) { return (n + 31) / 32; }
  // Lines per warp: the count that wastes the fewest lanes over the column and
  // row rounds, with at most 4 KB (4.5 KB of the 16-byte values) in a warp's
  // row; in FP32 80 pairs on half-lines up to 20, 128 up to 32 and 256 up to 64 (their grids
  // are small: 8 lines a warp left a 64^3 grid on 3 warps an SM, X2 16.3 us
  // against 12.3; the arithmetic-bound types want the lanes full: FP64 X2 70.6
  // us with 8 lines, 84.9 with 4 -- but on the smallest grids, which 8 lines a
  // warp leave with two warps an SM: FP64 32 x 50 x 54 X2 60 us, 35 with 4).
  static constexpr int waste(int lw) {
    return 1000 * 32 * (rounds(lw * B) * A + rounds(lw * A) * B) / (lw * 2 * N2);
  }
  static constexpr int pick() {
    int best = 1;
    const int bytes = sizeof(T) == 4 ? 4096 : 4608;
    const int pairs = N2 <= 20 ? 80
                      : sizeof(T) == 8 ? (N2 <= 27 ? 128 : 1024)
                                       : (N2 <= 32 ? 128 : N2 <= 64 ? 256 : 1024);
    for (int lw = 2; lw <= 16 && lw * N2 * (int)sizeof(C2<T>) <= bytes && lw * N2 <= pairs; ++lw)
      if (waste(lw) <= waste(best)) best = lw;
    return best;
  }
  static constexpr int LW = pick(), LINES = WARPS * LW;
  // Pitch of a line's transform row: the pad with the fewest bank conflicts of
  // a column store and a row load (slots of one access phase: 16 lanes of 8
  // bytes, 8 of 16 bytes).
  static constexpr int PH = sizeof(T) == 4 ? 16 : 8;
  static constexpr int conflicts(int ld) {
    int total = 0;
    for (int mode = 0; mode < 2; ++mode)
      for (int g = 0; g < 32; g += PH) {
        int hit[16] = {}, worst = 0;
        for (int i = g; i < g + PH; ++i) {
          const int l = i / (mode ? A : B), j = i - l * (mode ? A : B);
          const int s = (l * ld + (mode ? j * Q : j)) % PH;
          if (++hit[s] > worst) worst = hit[s];
        }
        total += worst;
      }
    return total;
  }
  static constexpr int pitch() {
    int best = A * Q;
    for (int ld = A * Q + 1; ld < A * Q + PH; ++ld)
      if (conflicts(ld) < conflicts(best)) best = ld;
    return best;
  }
  static constexpr int LD = pitch();
  // Pitch of a line's point-wise row (pairs): consecutive lines B slots apart.
  static constexpr int LDR = N2 + ((B - N2) % PH + PH) % PH;
  static constexpr size_t row_bytes(int nrows) {
    return ((size_t)WARPS * LW * (LD + nrows * LDR) + HK + A * Q) * sizeof(C2<T>);
  }
  // CTAs per SM asked for, by the registers of a column or row.
  static constexpr int REGS = sizeof(T) == 4 ? (B > 12 ? 96 : 80) : (B > 12 ? 168 : 128);
  static constexpr int MINB = 65536 / (REGS * NT);
};

template <class T, int A, int B> struct XWarp {
  typedef XW<T, A, B> X;
  C2<T>*S, *R[3];
  C2<T>*tw, *twt;  // exp(-2 pi i k / nx), k <= N2/2; exp(-2 pi i b ka / N2) at ka Q + b
  int lane, nlv;
  long long line0;
  EP_DEV XWarp(unsigned char* raw, const C2<T>* __restrict__ twx, long long nlines) {
    tw = reinterpret_cast<C2<T>*>(raw);
    twt = tw + X::HK;
    for (int i = threadIdx.x; i < X::HK; i += X::NT) tw[i] = twx[i];
    for (int i = threadIdx.x; i < A * X::Q; i += X::NT) {
      const int ka = i / X::Q, b = i - ka * X::Q;
      twt[i] = twx[b < B ? 2 * b * ka : 0];
    }
    const int warp = threadIdx.x >> 5;
    lane = threadIdx.x & 31;
    S = twt + A * X::Q + warp * X::LW * X::LD;
    C2<T>* r = twt + A * X::Q + X::WARPS * X::LW * X::LD + warp * X::LW * X::LDR;
#pragma unroll
    for (int i = 0; i < 3; ++i) R[i] = r + i * X::WARPS * X::LW * X::LDR;
    line0 = (long long)blockIdx.x * X::LINES + warp * X::LW;
    const long long left = nlines - line0;
    nlv = left < 0 ? 0 : (left < X::LW ? (int)left : X::LW);
    __syncthreads();
  }
  EP_DEV static int at(int l, int k) { return l * X::LD + (k % A) * X::Q + k / A; }

  // c2r packing of the lines' spectra.
  EP_DEV void pack(const C2<T>* __restrict__ spec) {
    // several pairs' loads in flight a lane
    constexpr int PU = sizeof(T) == 4 ? 4 : 2;
    for (int e0 = lane; e0 < X::LW * X::HK; e0 += 32 * PU) {
      C2<T> xk[PU], xc[PU];
#pragma unroll
      for (int u = 0; u < PU; ++u) {
        const int e = e0 + 32 * u, l = e / X::HK, k = e - l * X::HK;
        if (l < nlv) {
          const C2<T>* x = spec + (line0 + l) * X::NXH;
          xk[u] = __ldg(x + k);
          xc[u] = conjg(__ldg(x + (X::N2 - k)));
        }
      }
#pragma unroll
      for (int u = 0; u < PU; ++u) {
        const int e = e0 + 32 * u, l = e / X::HK, k = e - l * X::HK;
        if (l < nlv) {
          const C2<T> a = xk[u] + xc[u], b = cmulc(xk[u] - xc[u], tw[k]);
          S[at(l, k)] = a + mul_i(b);
          if (k > 0 && 2 * k < X::N2) S[at(l, X::N2 - k)] = conjg(a) + mul_i(conjg(b));
        }
      }
    }
    __syncwarp();
  }
  // B-point DFTs in place (inverse: with the twiddles of the columns).
  template <int DIR> EP_DEV void rows() {
#pragma unroll 1
    for (int e = lane; e < X::LW * A; e += 32) {
      const int l = e / A, ka = e - l * A;
      if (l < nlv) {
        C2<T>* s = S + l * X::LD + ka * X::Q;
        C2<T> u[B];
#pragma unroll
        for (int b = 0; b < B; ++b) u[b] = s[b];
        epfft::dft<T, B, DIR>(u);
        if (DIR > 0) {
          const C2<T>* w = twt + ka * X::Q;
#pragma unroll
          for (int b = 1; b < B; ++b) u[b] = cmulc(u[b], w[b]);
        }
#pragma unroll
        for (int b = 0; b < B; ++b) s[b] = u[b];
      }
    }
    __syncwarp();
  }
  // Inverse columns: f(line, b, v) gets the pairs m = b + B a as v[a].
  template <class F> EP_DEV void columns_inverse(T scale, F&& f) {
#pragma unroll 1
    for (int e = lane; e < X::LW * B; e += 32) {
      const int l = e / B, b = e - l * B;
      if (l < nlv) {
        C2<T> v[A];
#pragma unroll
        for (int ka = 0; ka < A; ++ka) v[ka] = S[l * X::LD + ka * X::Q + b];
        epfft::dft<T, A, +1>(v);
#pragma unroll
        for (int a = 0; a < A; ++a) v[a] = cmk<T>(v[a].x * scale, v[a].y * scale);
        f(l, b, v);
      }
    }
    __syncwarp();
  }
  EP_DEV void inverse(const C2<T>* __restrict__ spec) {
    pack(spec);
    rows<+1>();
  }
  // Forward transform of the pairs f(line, m) and the r2c unpacking.
  template <class F> EP_DEV void forward(F&& f, C2<T>* __restrict__ out) {
#pragma unroll 1
    for (int e = lane; e < X::LW * B; e += 32) {
      const int l = e / B, b = e - l * B;
      if (l < nlv) {
        C2<T> v[A];
#pragma unroll
        for (int a = 0; a < A; ++a) v[a] = f(l, b + B * a);
        epfft::dft<T, A, -1>(v);
        const C2<T>* w = twt + b;
#pragma unroll
        for (int ka = 1; ka < A; ++ka) v[ka] = cmul(v[ka], w[ka * X::Q]);
#pragma unroll
        for (int ka = 0; ka < A; ++ka) S[l * X::LD + ka * X::Q + b] = v[ka];
      }
    }
    __syncwarp();
    rows<-1>();
    for (int e = lane; e < X::LW * X::HK; e += 32) {
      const int l = e / X::HK, k = e - l * X::HK;
      if (l < nlv) {
        C2<T>* o = out + (line0 + l) * X::NXH;
        const C2<T> zk = S[at(l, k)], zc = conjg(S[at(l, k == 0 ? 0 : X::N2 - k)]);
        const C2<T> ev = epfft::K<T>::half * (zk + zc), od = cmul(tw[k], epfft::K<T>::half * mul_mi(zk - zc));
        o[k] = ev + od;
        if (2 * k < X::N2) o[X::N2 - k] = conjg(ev - od);
      }
    }
    __syncwarp();
  }
  // Offset of pair m of line l in a real field.
  EP_DEV long long at_field(int l, int m) const { return (line0 + l) * X::NX + 2 * m; }
};

template <class T> EP_DEV void st2(T* p, C2<T> v) { *reinterpret_cast<C2<T>*>(p) = v; }
// The pair at p of an array the kernel does not write (such loads move ahead
// of the stores around them: without that X4 waited on memory point by point,
// 509 us against 122 at 256 x 256 x 320).
template <class T> EP_DEV C2<T> ldn2(const T* p) { return __ldg(reinterpret_cast<const C2<T>*>(p)); }

// X1: den -> r2c along x.
template <class T, int A, int B>
__global__ void __launch_bounds__((XW<T, A, B>::NT), (XW<T, A, B>::MINB))
    k_xw1(long long nlines, Phys ph, const __grid_constant__ FdW<T> fd, const __grid_constant__ XWArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  XWarp<T, A, B> w(smraw, a.twx, nlines);
  w.forward([&](int l, int m) { return ldn2(a.den + w.at_field(l, m)); }, a.out[0]);
}

// X2: c2r of the products of fden -> dencg, delj4 (and denalf for OTC); pot4
// partial = delj4 + dencg^2 (a0 + a1 dencg) (poten.f90:34-92); forward r2c of
// den*dencg*(cp4 + cpp4*dencg) (poten.f90:62-67) and, for OTC, of f*grad(den),
// f = 1 - denalf/den0s (term_alfa.f90:157-170).
template <class T, int A, int B>
__global__ void __launch_bounds__((XW<T, A, B>::NT), (XW<T, A, B>::MINB))
    k_xw2(long long nlines, Phys ph, const __grid_constant__ FdW<T> fd, const __grid_constant__ XWArgs<T> a) {
  typedef XW<T, A, B> X;
  extern __shared__ __align__(16) unsigned char smraw[];
  XWarp<T, A, B> w(smraw, a.twx, nlines);
  const bool otc = ph.core == 1;
  const PConst<T> kc(ph);
  C2<T>*Rcg = w.R[0], *Rf = w.R[1];
#pragma unroll 1
  for (int j = 0; j < (otc ? 3 : 2); ++j) {
    w.inverse(a.in[j]);
    w.columns_inverse(kc.renor, [&](int l, int b, C2<T>(&v)[A]) {
      C2<T>* rc = Rcg + l * X::LDR + b;
      C2<T>* rf = Rf + l * X::LDR + b;
      const long long p = w.at_field(l, b);
      if (j == 0) {
#pragma unroll
        for (int i = 0; i < A; ++i) {
          rc[B * i] = v[i];
          if (a.keep) st2(a.dencg + p + 2 * B * i, v[i]);
        }
      } else if (j == 1) {
#pragma unroll
        for (int i = 0; i < A; ++i) {
          const C2<T> cg = rc[B * i];
          if (a.keep) st2(a.delj4 + p + 2 * B * i, v[i]);
          st2(a.pot4 + p + 2 * B * i, cmk<T>(v[i].x + cg.x * cg.x * (kc.a0 + kc.a1 * cg.x),
                                             v[i].y + cg.y * cg.y * (kc.a0 + kc.a1 * cg.y)));
        }
      } else {
#pragma unroll
        for (int i = 0; i < A; ++i) {
          const C2<T> f = cmk<T>(T(1) - v[i].x * kc.rden0s, T(1) - v[i].y * kc.rden0s);
          rf[B * i] = f;
          st2(a.falfs + p + 2 * B * i, f);
        }
      }
    });
  }
#pragma unroll 1
  for (int c = 0; c < (otc ? 4 : 1); ++c) {
    const T* src = c == 0 ? a.den : c == 1 ? a.dxd : c == 2 ? a.dyd : a.dzd;
    const C2<T>* rr = c == 0 ? Rcg : Rf;
    w.forward(
        [&](int l, int m) {
          const C2<T> d = ldn2(src + w.at_field(l, m)), r = rr[l * X::LDR + m];
          if (c == 0)
            return cmk<T>(d.x * r.x * (kc.cp4 + kc.cpp4 * r.x), d.y * r.y * (kc.cp4 + kc.cpp4 * r.y));
          return cmk<T>(r.x * d.x, r.y * d.y);
        },
        a.out[c]);
  }
}

// X3: c2r of the correlation convolution -> pot4 (+ penalty for OT,
// poten.f90:74,88-92,122-126).  OTC: c2r of the three alpha_s integrals
// (term_alfa.f90:172-181), the x-derivative of f*I_x, f*I_y and f*I_z for the
// divergence (:216-225), and forward r2c of grad(den).I (:194-201).
template <class T, int A, int B>
__global__ void __launch_bounds__((XW<T, A, B>::NT), (XW<T, A, B>::MINB))
    k_xw3(long long nlines, Phys ph, const __grid_constant__ FdW<T> fd, const __grid_constant__ XWArgs<T> a) {
  typedef XW<T, A, B> X;
  extern __shared__ __align__(16) unsigned char smraw[];
  XWarp<T, A, B> w(smraw, a.twx, nlines);
  const bool otc = ph.core == 1;
  const T rn = PConst<T>(ph).renor;
  const Pen<T> pn(ph);
  C2<T>*Rw = w.R[0], *Rc = w.R[1], *Rf = w.R[2];  // grad(den).I, f I_x, f
#pragma unroll 1
  for (int j = 0; j < (otc ? 4 : 1); ++j) {
    w.inverse(a.in[j]);
    const T* gc = j == 1 ? a.dxd : j == 2 ? a.dyd : a.dzd;
    T* ic = j == 1 ? a.intx : j == 2 ? a.inty : a.intz;
    T* fc = j == 2 ? a.gy : a.gz;
    w.columns_inverse(rn, [&](int l, int b, C2<T>(&v)[A]) {
      const long long p = w.at_field(l, b);
      const int o = l * X::LDR + b;
      if (j == 0) {
        T* q = a.pot4 + p;
        C2<T> pt[A];
#pragma unroll
        for (int i = 0; i < A; ++i) pt[i] = ld2((const T*)q + 2 * B * i);
#pragma unroll
        for (int i = 0; i < A; ++i) {
          C2<T> s = cmk<T>(pt[i].x + v[i].x, pt[i].y + v[i].y);
          if (!otc) {
            const C2<T> dn = ldn2(a.den + p + 2 * B * i);
            s.x = s.x + penalty_of(pn, dn.x);
            s.y = s.y + penalty_of(pn, dn.y);
          }
          st2(q + 2 * B * i, s);
        }
        return;
      }
#pragma unroll
      for (int i = 0; i < A; ++i) {
        const long long q = p + 2 * B * i;
        C2<T> f;
        if (j == 1) {
          f = ldn2((const T*)a.falfs + q);
          Rf[o + B * i] = f;
        } else {
          f = Rf[o + B * i];
        }
        const C2<T> g = ldn2(gc + q), fi = cmk<T>(f.x * v[i].x, f.y * v[i].y);
        if (a.keep) st2(ic + q, v[i]);
        if (j == 1) {
          Rc[o + B * i] = fi;
          Rw[o + B * i] = cmk<T>(g.x * v[i].x, g.y * v[i].y);
        } else {
          st2(fc + q, fi);
          const C2<T> s = Rw[o + B * i];
          Rw[o + B * i] = cmk<T>(s.x + g.x * v[i].x, s.y + g.y * v[i].y);
        }
      }
    });
    if (j == 1) {
      // d/dx (f I_x) of the pair m from the pairs m - 3 .. m + 3 of its row
      // (weights beyond the stencil's radius are zero)
      for (int e = w.lane; e < X::LW * X::N2; e += 32) {
        const int l = e / X::N2, m = e - l * X::N2;
        if (l < w.nlv) {
          const C2<T>* row = Rc + l * X::LDR;
          T u[14];
#pragma unroll
          for (int i = -3; i <= 3; ++i) {
            const int mm = m + i;
            const int mw = mm < 0 ? mm + X::N2 : (mm >= X::N2 ? mm - X::N2 : mm);
            C2<T> t = row[mw];
            if (mw != mm && !fd.periodic) t = cmk<T>(T(0), T(0));
            u[2 * (i + 3)] = t.x;
            u[2 * (i + 3) + 1] = t.y;
          }
          C2<T> s = cmk<T>(T(0), T(0));
          if constexpr (std::is_same<T, dfloat>::value) {
#if defined(__CUDA_ARCH__)
            dd2_acc t;
            float2 ph_, pl_;
            dd2_wdiff(fd.w1[0][1], dfloat2{u[7], u[8]}, dfloat2{u[5], u[6]}, t.h, t.l);
#pragma unroll
            for (int k = 2; k <= 6; ++k) {
              dd2_wdiff(fd.w1[0][k], dfloat2{u[6 + k], u[7 + k]}, dfloat2{u[6 - k], u[7 - k]}, ph_, pl_);
              dd2_add(t, ph_, pl_);
            }
            s = dd2_value(t);
#endif
          } else {
#pragma unroll
            for (int k = 1; k <= 6; ++k) {
              s.x += fd.w1[0][k] * (u[6 + k] - u[6 - k]);
              s.y += fd.w1[0][k] * (u[7 + k] - u[7 - k]);
            }
          }
          st2(a.dgx + w.at_field(l, m), s);
        }
      }
      __syncwarp();
    }
  }
  if (otc) w.forward([&](int l, int m) { return Rw[l * X::LDR + m]; }, a.out[0]);
}

// X4 (OTC): c2r of kalfs*FFT(grad(den).I) -> U_alpha = (u/den0s + div(f I))
// * h2o2m4 * alphas (term_alfa.f90:203-236); pot4 += U_alpha + penalty.
template <class T, int A, int B>
__global__ void __launch_bounds__((XW<T, A, B>::NT), (XW<T, A, B>::MINB))
    k_xw4(long long nlines, Phys ph, const __grid_constant__ FdW<T> fd, const __grid_constant__ XWArgs<T> a) {
  extern __shared__ __align__(16) unsigned char smraw[];
  XWarp<T, A, B> w(smraw, a.twx, nlines);
  const PConst<T> kc(ph);
  const Pen<T> pn(ph);
  w.inverse(a.in[0]);
  w.columns_inverse(kc.renor, [&](int l, int b, C2<T>(&v)[A]) {
    const long long p = w.at_field(l, b);
    C2<T> pt[A];
#pragma unroll
    for (int i = 0; i < A; ++i) pt[i] = ld2((const T*)a.pot4 + p + 2 * B * i);
#pragma unroll
    for (int i = 0; i < A; ++i) {
      const long long q = p + 2 * B * i;
      const C2<T> gx = ldn2((const T*)a.dgx + q), yz = ldn2(a.dyz + q), dn = ldn2(a.den + q);
      const C2<T> ua = cmk<T>(((v[i].x * kc.rden0s + gx.x) + yz.x) * kc.h2o2m4 * kc.alphas,
                              ((v[i].y * kc.rden0s + gx.y) + yz.y) * kc.h2o2m4 * kc.alphas);
      if (a.keep) st2(a.ualphas + q, ua);
      st2(a.pot4 + q, cmk<T>((pt[i].x + ua.x) + penalty_of(pn, dn.x), (pt[i].y + ua.y) + penalty_of(pn, dn.y)));
    }
  });
}

// c2r alone, scaled, into a real array (ep_convolve_noalloc).
template <class T, int A, int B>
__global__ void __launch_bounds__((XW<T, A, B>::NT), (XW<T, A, B>::MINB))
    k_xw_c2r(long long nlines, const C2<T>* __restrict__ spec, T* __restrict__ out, const C2<T>* __restrict__ twx,
             T scale) {
  extern __shared__ __align__(16) unsigned char smraw[];
  XWarp<T, A, B> w(smraw, twx, nlines);
  w.inverse(spec);
  w.columns_inverse(scale, [&](int l, int b, C2<T>(&v)[A]) {
    T* p = out + w.at_field(l, b);
#pragma unroll
    for (int i = 0; i < A; ++i) st2(p + 2 * B * i, v[i]);
  });
}
template <class T, int A, int B> const void* xw_c2r() {
  if constexpr (std::is_same<T, double>::value) {
    static_assert(XW<T, A, B>::row_bytes(0) <= 48 * 1024, "launched without a raised shared-memory limit");
    return (const void*)k_xw_c2r<T, A, B>;
  }
  return nullptr;
}

#define EP_XW_CASE(NN, AA, BB)                                                                                   \
  case NN: {                                                                                                     \
    typedef XW<T, AA, BB> X;                                                                                     \
    static_assert(X::N2 == NN, "factors of the length");                                                         \
    static const XWKernels k{{(const void*)k_xw1<T, AA, BB>, (const void*)k_xw2<T, AA, BB>,                      \
                              (const void*)k_xw3<T, AA, BB>, (const void*)k_xw4<T, AA, BB>},                     \
                             X::LINES, X::NT, {X::row_bytes(0), X::row_bytes(2), X::row_bytes(3), X::row_bytes(0)}, \
                             xw_c2r<T, AA, BB>()};                                                               \
    return &k;                                                                                                   \
  }
#define EP_XW_PART(NAME, LENGTHS)                    \
  template <class T> const XWKernels* NAME(int n2) { \
    switch (n2) {                                    \
      LENGTHS(EP_XW_CASE)                            \
      default: return nullptr;                       \
    }                                                \
  }
