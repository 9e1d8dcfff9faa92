// ep_yz.cuh - the Y and Z passes: complex transforms of strided lines of
// N = A B points (A, B <= 20), one kernel pair per length.
//
// A CTA owns LL lines whose first elements are neighbours in memory (x runs
// fastest) and NS slots per line: thread = (line, slot), lines fastest, so
// every global and shared access of a half-warp is one contiguous run.  With
//   n = b + B a (a < A, b < B),   k = ka + A kb (ka < A, kb < B)
//   X[ka + A kb] = sum_b w_B^(b kb) w_N^(b ka) sum_a x[b + B a] w_A^(a ka)
// a pass is
//   columns: slot s takes b = s, s + NS, ..: A loads straight from global
//            memory, the A-point DFT in registers, the twiddles, A stores to
//            shared memory (element-major, S[n LL + line]: no padding, no
//            bank conflicts);
//   rows:    slot s takes ka = s, s + NS, ..: the B-point DFT in registers and
//            B stores straight to global memory.
// One exchange and one barrier a transform.  The convolution runs the rows
// forward, the k-space product and the rows backward on the same registers (a
// row is read and written back by one thread), then the columns backward: two
// barriers for a transform pair.
//
// What bounds it: FP32, the memory system (one read and one write of each
// line); FP64 and double-float, their arithmetic pipes.  The split into two
// factors of at most 20 keeps a column or row in registers for every even
// 2^a 3^b 5^c length up to 324 that has one; other lengths stay on the
// shared-memory engine of ep_fft.cuh (a barrier per radix, a shared-memory
// round trip per radix, index divisions).  Mean launch, that engine against
// these kernels: Z convolutions FP32 320 points (256 x 256 x 320) 312 -> 131
// us, FP32/double-float 160 points (96 x 120 x 160) 41 -> 25 us; Y 120 points
// 20-23 -> 14-16 us; against the power-of-two register transforms they replace
// (lines padded in shared memory, twiddled and exchanged per transform):
// double-float 128 points Z 70 -> 59 us, Y 27-33 -> 26-30; FP32 128 points Z
// 15.7 -> 15.4, Y 11.3-12.1 -> 10.4-11.7; FP64 128 points Z 221 -> 214.
// Conventions are those of ep_fft.cuh: forward exp(-2 pi i k n / N),
// unnormalised both ways.
#pragma once
#include "ep_fft.cuh"
#include "ep_kernels.cuh"

// Every length with its factors (A columns' length first: the global loads in
// flight per thread).
#define EP_YZ_LENGTHS_A(X)                                                                                     \
  X(16, 4, 4) X(18, 6, 3) X(20, 5, 4) X(24, 6, 4) X(30, 6, 5) X(32, 8, 4) X(36, 6, 6) X(40, 8, 5) X(48, 8, 6)   \
  X(50, 10, 5) X(54, 9, 6) X(60, 10, 6) X(64, 8, 8) X(72, 9, 8) X(80, 10, 8) X(90, 10, 9) X(96, 12, 8)          \
  X(100, 10, 10)
#define EP_YZ_LENGTHS_B(X)                                                                                     \
  X(108, 12, 9) X(120, 12, 10) X(128, 16, 8) X(144, 12, 12) X(150, 15, 10) X(160, 16, 10) X(162, 18, 9)         \
  X(180, 15, 12) X(192, 16, 12)
#define EP_YZ_LENGTHS_C(X)                                                                                     \
  X(200, 20, 10) X(216, 18, 12) X(240, 16, 15) X(256, 16, 16)
#define EP_YZ_LENGTHS_D(X)                                                                                     \
  X(270, 18, 15) X(288, 18, 16) X(300, 20, 15) X(320, 20, 16) X(324, 18, 18)

// Host-side description of one length's kernels (null: no such length).
struct YZKernels {
  const void* c2c[2]; // (Arr8<T>, LineSet, twiddles): forward, inverse
  const void* conv;   // (ConvSpec<T>, LineSet, twiddles)
  int lines, threads; // lines and threads per CTA
  size_t line_bytes;  // shared memory of one buffer of `lines` lines
  size_t tw_bytes;    // shared memory of the twiddle table
};
// The kernels of lines of n points in precision T; the pieces are compiled in
// separate units.
template <class T> const YZKernels* yz_part_a(int n);
template <class T> const YZKernels* yz_part_b(int n);
template <class T> const YZKernels* yz_part_c(int n);
template <class T> const YZKernels* yz_part_d(int n);
template <class T> inline const YZKernels* yz_kernels(int n) {
  const YZKernels* k = yz_part_a<T>(n);
  if (!k) k = yz_part_b<T>(n);
  if (!k) k = yz_part_c<T>(n);
  if (!k) k = yz_part_d<T>(n);
  return k;
}

// The limits of dynamic shared memory.  A kernel's limit is its largest use's
// wherever it is set: contexts and ep_convolve_noalloc launch the same FP64
// kernels, and a limit lowered to one caller's use (one line buffer of a
// convolution with one table) refuses the other's launch (two buffers).
inline cudaError_t yz_limit_c2c(const YZKernels& k) {
  for (const void* f : k.c2c) {
    const cudaError_t e =
        cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(k.line_bytes + k.tw_bytes));
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}
inline cudaError_t yz_limit_conv(const YZKernels& k) {
  return cudaFuncSetAttribute(k.conv, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(2 * k.line_bytes + k.tw_bytes));
}

template <class T, int A, int B> struct YZ {
  static constexpr int N = A * B;
  // Lines per CTA: 32 in FP32 (256-byte runs) while their buffer stays within
  // 42 KB, else 16 (the two measure alike on one 128^3 instance and 32 is 5 %
  // faster in a batch); 16 of the 16-byte values (32 leave a 64 x 64 x 80 grid
  // on 66 CTAs: Z 58 us against 45), 8 up to 72 points, whose grids are small,
  // and where two buffers of 16 would not fit.
  static constexpr int LL = sizeof(T) == 4 ? (32 * N * 8 <= 42 * 1024 ? 32 : 16) : (N > 72 && N <= 256 ? 16 : 8);
  // Slots per line: the count with the largest share of busy slots over the
  // column and row rounds, less 5 to 16 % below eight slots (fewer loads in
  // flight) and 4 % where the CTA is no whole number of warps.
  static constexpr int rounds(int n, int ns) { return (n + ns - 1) / ns; }
  static constexpr int score(int ns) {
    const int weight = ns >= 8 ? 100 : ns == 7 ? 97 : ns == 6 ? 95 : ns == 5 ? 90 : ns == 4 ? 84 : 60;
    return 2 * N * weight * (ns * LL % 32 ? 96 : 100) / (ns * (rounds(B, ns) * A + rounds(A, ns) * B));
  }
  static constexpr int pick() {
    int best = 1;
    for (int ns = 2; ns <= (A > B ? A : B) && ns * LL <= 512; ++ns)
      if (score(ns) >= score(best)) best = ns;
    return best;
  }
  static constexpr int NS = pick();
  static constexpr int NT = LL * NS;
  static constexpr int RC = rounds(B, NS), RR = rounds(A, NS);  // column and row rounds
  // FP32 rounds are unrolled (a round's loads ahead of the last one's
  // arithmetic); the 16-byte types' are not: their codelets, a few thousand
  // instructions each in double-float, would not stay in the instruction cache
  // (192-point double-float convolution 202 us unrolled)
  static constexpr bool UNROLL = sizeof(T) == 4;
  // CTAs per SM asked for: 64 registers (FP32) or 128 (16-byte complex values)
  // a thread, more for the longest codelets.
  static constexpr int REGS = sizeof(T) == 4 ? (A > 16 ? 80 : 64) : (A > 12 ? 168 : 128);
  static constexpr int cap(int m) { return m < 1 ? 1 : (m > 8 ? 8 : m); }
  static constexpr int MINB = cap(65536 / (REGS * NT));
  // the convolution holds a row's form-factor values too
  static constexpr int REGS_C = sizeof(T) == 4 ? (A >= 12 ? 96 : 80) : REGS;
  static constexpr int MINB_C = cap(65536 / (REGS_C * NT));
};

// The value, opaque to the compiler: multiples of a stride are then formed
// where they are used instead of being kept in registers across a loop.
EP_DEV int fresh(int v) {
  asm volatile("" : "+r"(v));
  return v;
}

// In-place transforms along a strided axis of up to 8 arrays (blockIdx.y).
template <class T, int A, int B, int DIR>
__global__ void __launch_bounds__((YZ<T, A, B>::NT), (YZ<T, A, B>::MINB))
    k_yz_c2c(const __grid_constant__ Arr8<T> arr, LineSet ls, const C2<T>* __restrict__ twg) {
  typedef YZ<T, A, B> Y;
  constexpr int N = Y::N, LL = Y::LL, NS = Y::NS;
  extern __shared__ __align__(16) unsigned char smraw[];
  C2<T>* S = reinterpret_cast<C2<T>*>(smraw);
  C2<T>* tw = S + N * LL;
  const int line = threadIdx.x % LL, slot = threadIdx.x / LL;
  for (int i = threadIdx.x; i < N; i += Y::NT) tw[i] = twg[i];
  const long long L = (long long)blockIdx.x * LL + line;
  const bool valid = L < ls.nlines;
  C2<T>* a = arr.a[blockIdx.y] + (valid ? (L % ls.Mi) + (L / ls.Mi) * ls.So : 0);
  const int Sa = (int)ls.Sa;
  C2<T> v[A];
  auto load = [&](int b) {
    const int st = fresh(B * Sa);
    const C2<T>* p = a + b * Sa;
#pragma unroll
    for (int m = 0; m < A; ++m) v[m] = valid ? p[m * st] : cmk<T>(T(0), T(0));
  };
  if (slot < B) load(slot);
  __syncthreads();  // tw complete
#pragma unroll (Y::UNROLL ? Y::RC : 1)
  for (int c = 0; c < Y::RC; ++c) {
    const int b = slot + c * NS;
    if (b < B) {
      if (c > 0) load(b);
      epfft::dft<T, A, DIR>(v);
      if (b != 0) {
#pragma unroll
        for (int ka = 1; ka < A; ++ka) v[ka] = DIR < 0 ? cmul(v[ka], tw[b * ka]) : cmulc(v[ka], tw[b * ka]);
      }
#pragma unroll
      for (int ka = 0; ka < A; ++ka) S[(ka * B + b) * LL + line] = v[ka];
    }
  }
  __syncthreads();
#pragma unroll (Y::UNROLL ? Y::RR : 1)
  for (int r = 0; r < Y::RR; ++r) {
    const int ka = slot + r * NS;
    if (ka < A) {
      C2<T> u[B];
#pragma unroll
      for (int b = 0; b < B; ++b) u[b] = S[(ka * B + b) * LL + line];
      epfft::dft<T, B, DIR>(u);
      if (valid) {
        const int st = fresh(A * Sa);
        C2<T>* p = a + ka * Sa;
#pragma unroll
        for (int kb = 0; kb < B; ++kb) p[kb * st] = u[kb];
      }
    }
  }
}

// Forward transform along the pass axis, then per kernel table the k-space
// product (poten.f90:34-36,46-48,69-71,95-97 and term_alfa.f90:172-176,
// 203-205) and the inverse transform.  With several tables the spectrum stays
// in a second buffer of shared memory.
template <class T, int A, int B>
__global__ void __launch_bounds__((YZ<T, A, B>::NT), (YZ<T, A, B>::MINB_C))
    k_yz_conv(const __grid_constant__ ConvSpec<T> cs, LineSet ls, const C2<T>* __restrict__ twg) {
  typedef YZ<T, A, B> Y;
  constexpr int N = Y::N, LL = Y::LL, NS = Y::NS;
  extern __shared__ __align__(16) unsigned char smraw[];
  C2<T>* S = reinterpret_cast<C2<T>*>(smraw);
  C2<T>* tw = S + N * LL;
  C2<T>* K = tw + N;  // the kept spectrum (several tables only)
  const int line = threadIdx.x % LL, slot = threadIdx.x / LL;
  for (int i = threadIdx.x; i < N; i += Y::NT) tw[i] = twg[i];
  const int which = blockIdx.y, nout = cs.nout[which];
  const long long L = (long long)blockIdx.x * LL + line;
  const bool valid = L < ls.nlines;
  const long long base = valid ? (L % ls.Mi) + (L / ls.Mi) * ls.So : 0;
  const int Sa = (int)ls.Sa;
  // FP32: the thread's form-factor values of a table are loaded ahead of the
  // barrier in front of their use, when the column's registers are free; the
  // 16-byte types are arithmetic-bound and load them at their use
  constexpr bool PRE = sizeof(T) == 4 && Y::RR * B <= 20;
  T kv[PRE ? Y::RR : 1][B];
  auto load_ker = [&](int j, int r, T (&k)[B]) {
    const int ka = slot + r * NS, st = fresh(A * Sa);
    const T* ker = cs.ker[which][j] + (base + ka * Sa);
#pragma unroll
    for (int kb = 0; kb < B; ++kb) k[kb] = (valid && ka < A) ? ker[kb * st] : T(0);
  };
  {
    const C2<T>* in = cs.in[which] + base;
    C2<T> v[A];
    auto load = [&](int b) {
#pragma unroll
      for (int m = 0; m < A; ++m) v[m] = valid ? in[(b + B * m) * Sa] : cmk<T>(T(0), T(0));
    };
    if (slot < B) load(slot);
    __syncthreads();  // tw complete
#pragma unroll (Y::UNROLL ? Y::RC : 1)
    for (int c = 0; c < Y::RC; ++c) {
      const int b = slot + c * NS;
      if (b < B) {
        if (c > 0) load(b);
        epfft::dft<T, A, -1>(v);
        if (b != 0) {
#pragma unroll
          for (int ka = 1; ka < A; ++ka) v[ka] = cmul(v[ka], tw[b * ka]);
        }
#pragma unroll
        for (int ka = 0; ka < A; ++ka) S[(ka * B + b) * LL + line] = v[ka];
      }
    }
  }
#pragma unroll 1
  for (int j = 0; j < nout; ++j) {
    if constexpr (PRE) {
#pragma unroll
      for (int r = 0; r < Y::RR; ++r) load_ker(j, r, kv[r]);
    }
    __syncthreads();
#pragma unroll (Y::UNROLL ? Y::RR : 1)
    for (int r = 0; r < Y::RR; ++r) {
      const int ka = slot + r * NS;
      if (ka < A) {
        C2<T> u[B];
        if (j == 0) {
#pragma unroll
          for (int b = 0; b < B; ++b) u[b] = S[(ka * B + b) * LL + line];
          epfft::dft<T, B, -1>(u);
          if (nout > 1) {
#pragma unroll
            for (int kb = 0; kb < B; ++kb) K[(ka * B + kb) * LL + line] = u[kb];
          }
        } else {
#pragma unroll
          for (int kb = 0; kb < B; ++kb) u[kb] = K[(ka * B + kb) * LL + line];
        }
        if constexpr (!PRE) load_ker(j, r, kv[0]);
#pragma unroll
        for (int kb = 0; kb < B; ++kb) {
          const T k = kv[PRE ? r : 0][kb];
          u[kb] = cmk<T>(u[kb].x * k, u[kb].y * k);
        }
        epfft::dft<T, B, +1>(u);
        if (ka != 0) {
#pragma unroll
          for (int b = 1; b < B; ++b) u[b] = cmulc(u[b], tw[b * ka]);
        }
#pragma unroll
        for (int b = 0; b < B; ++b) S[(ka * B + b) * LL + line] = u[b];
      }
    }
    __syncthreads();
    C2<T>* out = cs.out[which][j] + base;
#pragma unroll (Y::UNROLL ? Y::RC : 1)
    for (int c = 0; c < Y::RC; ++c) {
      const int b = slot + c * NS;
      if (b < B) {
        C2<T> v[A];
#pragma unroll
        for (int ka = 0; ka < A; ++ka) v[ka] = S[(ka * B + b) * LL + line];
        epfft::dft<T, A, +1>(v);
        if (valid) {
          const int st = fresh(B * Sa);
          C2<T>* o = out + b * Sa;
#pragma unroll
          for (int m = 0; m < A; ++m) o[m * st] = v[m];
        }
      }
    }
  }
}

#define EP_YZ_CASE(NN, AA, BB)                                                                             \
  case NN: {                                                                                               \
    typedef YZ<T, AA, BB> Y;                                                                               \
    static_assert(Y::N == NN, "factors of the length");                                                    \
    static const YZKernels k{{(const void*)k_yz_c2c<T, AA, BB, -1>, (const void*)k_yz_c2c<T, AA, BB, +1>},  \
                             (const void*)k_yz_conv<T, AA, BB>, Y::LL,   \
                             Y::NT, (size_t)Y::LL * NN * sizeof(C2<T>), (size_t)NN * sizeof(C2<T>)};       \
    return &k;                                                                                             \
  }
#define EP_YZ_PART(NAME, LENGTHS)                 \
  template <class T> const YZKernels* NAME(int n) { \
    switch (n) {                                  \
      LENGTHS(EP_YZ_CASE)                         \
      default: return nullptr;                    \
    }                                             \
  }
