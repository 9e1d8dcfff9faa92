// ep_reduce.cuh - compensated reductions shared by the eff_pot kernels.
//
// Every sum the kernels return (norm, errHe, <psi|H|psi>, the energy
// integrals of energy.f90:67-165, the impurity force and moments) is carried
// as an unevaluated pair (hi, lo) from the first addition to the last:
//  * per thread: Neumaier's variant of Kahan-Babuska summation in FP64,
//    Kahan summation in FP32 for FP32 fields and in the stencil marches;
//  * across a warp, across the warps of a block and across the blocks:
//    pairs added with Knuth's error-free TwoSum, hi + e into hi, the lows
//    and e into lo (FP32 pairs up to the block's result for FP32 fields);
//  * block partials are stored as pairs: partials[b*nq + q] holds hi and
//    partials[nblocks*nq + b*nq + q] holds lo (the buffer holds twice the
//    partial count).
// The result is hi + lo rounded once: its error is about one rounding of the
// sum plus n u^2 times the sum of magnitudes, instead of the log2(n) u of a
// plain pairwise tree, so sums whose terms cancel keep their digits.
#pragma once
#include "ep_common.cuh"

// Knuth's TwoSum: s = fl(a + b) and s + e == a + b exactly.
EP_DEV void two_sum(double a, double b, double& s, double& e) {
  s = a + b;
  const double bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}
EP_DEV void two_sum(float a, float b, float& s, float& e) {
  s = a + b;
  const float bb = s - a;
  e = (a - (s - bb)) + (b - bb);
}

// (s, c) += (s2, c2) for unevaluated pairs.
template <class F>
EP_DEV void pair_add(F& s, F& c, F s2, F c2) {
  F t, e;
  two_sum(s, s2, t, e);
  s = t;
  c = (c + c2) + e;
}

// Per-thread accumulators: the running sum s and its compensation c.
// Neumaier: the correction of each addition, whichever operand is larger in
// magnitude, goes into c (value s + c).
template <class T> struct Neumaier {
  typedef T value_type;
  T s = T(0), c = T(0);
  EP_DEV void add(T v) {
    const T t = s + v;
    c += (fabs(s) >= fabs(v)) ? ((s - t) + v) : ((v - t) + s);
    s = t;
  }
  EP_DEV T lo() const { return c; }
  EP_DEV double get() const { return (double)s + (double)c; }
};
// Kahan: c holds minus the low part lost so far (value s - c); four
// operations per addition, for the per-point sums of the stencil marches,
// whose running sums are short (one term per plane of the CTA's z range).
template <class T> struct Kahan {
  typedef T value_type;
  T s = T(0), c = T(0);
  EP_DEV void add(T v) {
    const T y = v - c;
    const T t = s + y;
    c = (t - s) - y;
    s = t;
  }
  EP_DEV T lo() const { return -c; }
  EP_DEV double get() const { return (double)s - (double)c; }
};
// Double-float terms: the pair (s, c) of FP32 values, each high part added
// to s with the error-free TwoSum and its rounding error and the low part
// collected in c (Ogita, Rump and Oishi's Sum2 kept as a pair: the error is
// about n u^2 of the magnitudes, where Kahan's s - c in FP32 keeps an error
// of up to 2u of the sum -- enough to move the renormalisation factor of the
// double-float path by 1e-12 a step).
template <> struct Kahan<dfloat> {
  typedef float value_type;
  float s = 0.0f, c = 0.0f;
  EP_DEV void add(dfloat v) {
    const float t = s + v.hi;
    const float bb = t - s;
    c += ((s - (t - bb)) + (v.hi - bb)) + v.lo;
    s = t;
  }
  EP_DEV float lo() const { return c; }
  EP_DEV double get() const { return (double)s + (double)c; }
};
// The accumulator of sums of T values: Neumaier in FP64, Kahan in FP32 and
// double-float.
template <class T> struct AccOf { typedef Neumaier<T> type; };
template <> struct AccOf<float> { typedef Kahan<float> type; };
template <> struct AccOf<dfloat> { typedef Kahan<dfloat> type; };
template <class T> using Acc = typename AccOf<T>::type;

template <class F>
EP_DEV void warp_pair_sum(F& s, F& c) {
  for (int o = 16; o > 0; o >>= 1) {
    const F s2 = __shfl_down_sync(0xffffffffu, s, o), c2 = __shfl_down_sync(0xffffffffu, c, o);
    pair_add(s, c, s2, c2);
  }
}

// Warp sums of N pairs at once (N a power of two, at most 32): while more
// than one sum is left, the lanes of one half of the exchange keep one half of
// the sums and hand the other half over, so that a step adds as many pairs as
// it leaves (9 pair additions for 8 sums, 16 for 16, where one tree per sum
// takes 40 and 80: the FP64 pipe needs 16 cycles for a warp instruction).
// Sum multi_index<N>(lane) ends in s[0], c[0] of every lane.
template <int N, int O = 16, class F>
EP_DEV void warp_multi_sum(F* s, F* c) {
  static_assert(N >= 1 && N <= 32 && (N & (N - 1)) == 0, "a power of two of sums");
  if constexpr (O > 0) {
    if constexpr (N > 1) {
      const bool up = (threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z)) & O;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        const F gs = up ? s[i] : s[i + N / 2], gc = up ? c[i] : c[i + N / 2];
        F ks = up ? s[i + N / 2] : s[i], kc = up ? c[i + N / 2] : c[i];
        pair_add(ks, kc, __shfl_xor_sync(0xffffffffu, gs, O), __shfl_xor_sync(0xffffffffu, gc, O));
        s[i] = ks;
        c[i] = kc;
      }
      warp_multi_sum<N / 2, O / 2>(s, c);
    } else {
      pair_add(s[0], c[0], __shfl_xor_sync(0xffffffffu, s[0], O), __shfl_xor_sync(0xffffffffu, c[0], O));
      warp_multi_sum<1, O / 2>(s, c);
    }
  }
}
template <int N>
EP_DEV int multi_index(int lane) {
  int q = 0;
#pragma unroll
  for (int n = N / 2, o = 16; n > 0; n /= 2, o /= 2) q += (lane & o) ? n : 0;
  return q;
}

// The sums of QMASK among NQ: how many, the k-th of them, and their count
// rounded up to a power of two.
template <int NQ, unsigned QMASK> struct QSel {
  static constexpr unsigned M = NQ >= 32 ? QMASK : QMASK & ((1u << NQ) - 1u);
  EP_HD static constexpr int count(unsigned m) { return m ? 1 + count(m & (m - 1)) : 0; }
  EP_HD static constexpr int kth(int k) {
    for (int q = 0; q < NQ; ++q)
      if ((M >> q) & 1u)
        if (k-- == 0) return q;
    return -1;
  }
  static constexpr int N = count(M);
  EP_HD static constexpr int pad(int n) { return n <= 1 ? 1 : 2 * pad((n + 1) / 2); }
  static constexpr int NP = pad(N);
};

// Block reduction of per-thread accumulators into the block's pairs, for
// the sums q whose bit is set in QMASK (the others are not stored).  FP32
// accumulators stay FP32 pairs up to the block's result (the FP64 pipe is
// about 1/64 of the FP32 rate on this part; a pair of FP32 values carries
// about 48 significant bits).
template <int NQ, unsigned QMASK = ~0u, class A>
EP_DEV void block_reduce_store_acc(A (&acc)[NQ], double* __restrict__ partials) {
  typedef typename A::value_type T;
  typedef QSel<NQ, QMASK> Q;
  __shared__ T red_s[Q::NP][32], red_c[Q::NP][32];
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nth = blockDim.x * blockDim.y * blockDim.z;
  const int lane = tid & 31, warp = tid >> 5, nw = (nth + 31) >> 5;
  const int mine = multi_index<Q::NP>(lane);
  const bool first = (lane & (32 / Q::NP - 1)) == 0;  // one lane per sum
  T s[Q::NP], c[Q::NP];
#pragma unroll
  for (int k = 0; k < Q::NP; ++k) {
    s[k] = k < Q::N ? acc[k < Q::N ? Q::kth(k) : 0].s : T(0);
    c[k] = k < Q::N ? acc[k < Q::N ? Q::kth(k) : 0].lo() : T(0);
  }
  warp_multi_sum<Q::NP>(s, c);
  if (first) {
    red_s[mine][warp] = s[0];
    red_c[mine][warp] = c[0];
  }
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < Q::NP; ++k) {
      s[k] = lane < nw ? red_s[k][lane] : T(0);
      c[k] = lane < nw ? red_c[k][lane] : T(0);
    }
    warp_multi_sum<Q::NP>(s, c);
    if (first && mine < Q::N) {
      int q = 0;
#pragma unroll
      for (int k = 0; k < Q::N; ++k)
        if (k == mine) q = Q::kth(k);
      const long long nb = (long long)gridDim.x * gridDim.y * gridDim.z;
      const long long b = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
      // the pair widened to FP64 exactly (an FP32 pair gives its two values;
      // TwoSum of them is exact in FP64)
      double hs, he;
      two_sum((double)s[0], (double)c[0], hs, he);
      partials[b * NQ + q] = hs;
      partials[nb * NQ + b * NQ + q] = he;
    }
  }
}

// The same for per-thread FP64 values, added as they are:
// a block's tree rounds eight times at 2^-53, at random over the blocks, and
// takes one FP64 operation an addition where a pair takes eight (the nine sums
// of k_impmoments at 96 x 160 x 192: 89 us, 148 with pairs).
template <int N, int O = 16>
EP_DEV void warp_multi_add(double* s) {
  if constexpr (O > 0) {
    if constexpr (N > 1) {
      const bool up = (threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z)) & O;
#pragma unroll
      for (int i = 0; i < N / 2; ++i) {
        const double give = up ? s[i] : s[i + N / 2], keep = up ? s[i + N / 2] : s[i];
        s[i] = keep + __shfl_xor_sync(0xffffffffu, give, O);
      }
      warp_multi_add<N / 2, O / 2>(s);
    } else {
      s[0] += __shfl_xor_sync(0xffffffffu, s[0], O);
      warp_multi_add<1, O / 2>(s);
    }
  }
}
template <int NQ>
EP_DEV void block_reduce_store_sums(const double (&tot)[NQ], double* __restrict__ partials) {
  typedef QSel<NQ, ~0u> Q;
  __shared__ double red[Q::NP][32];
  const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
  const int nth = blockDim.x * blockDim.y * blockDim.z;
  const int lane = tid & 31, warp = tid >> 5, nw = (nth + 31) >> 5;
  const int mine = multi_index<Q::NP>(lane);
  const bool first = (lane & (32 / Q::NP - 1)) == 0;  // one lane per sum
  double s[Q::NP];
#pragma unroll
  for (int k = 0; k < Q::NP; ++k) s[k] = k < NQ ? tot[k < NQ ? k : 0] : 0.0;
  warp_multi_add<Q::NP>(s);
  if (first) red[mine][warp] = s[0];
  __syncthreads();
  if (warp == 0) {
#pragma unroll
    for (int k = 0; k < Q::NP; ++k) s[k] = lane < nw ? red[k][lane] : 0.0;
    warp_multi_add<Q::NP>(s);
    if (first && mine < NQ) {
      const long long nb = (long long)gridDim.x * gridDim.y * gridDim.z;
      const long long b = blockIdx.x + (long long)gridDim.x * (blockIdx.y + (long long)gridDim.y * blockIdx.z);
      partials[b * NQ + mine] = s[0];
      partials[nb * NQ + b * NQ + mine] = 0.0;
    }
  }
}

// Sum of the block pairs of a reduction -> sc->sums[out0 + q] for the q in
// qmask: warp w takes q = w, w + nwarps, ... (Neumaier over each lane's
// blocks, then a pair tree across the warp).  mode 1: corrector epilogue
// (norm, mu, renormalisation factor).
EP_DEV void finalize_block(const double* partials, int nblocks, int nq, DevScalars* sc, int out0, int mode,
                           double N, double dxyz, double n4, int renorm, int stats = 1, unsigned qmask = ~0u) {
  const int tid = threadIdx.x + blockDim.x * threadIdx.y;
  const int nth = blockDim.x * blockDim.y;
  const int lane = tid & 31, warp = tid >> 5, nw = (nth + 31) >> 5;
  const double* lo = partials + (long long)nblocks * nq;
  for (int q = warp; q < nq; q += nw) {
    if (!((qmask >> q) & 1u)) continue;
    Acc<double> a;
    double cl = 0.0;
    for (int b = lane; b < nblocks; b += 32) {
      a.add(__ldcg(partials + (long long)b * nq + q));
      cl += __ldcg(lo + (long long)b * nq + q);
    }
    double s = a.s, c = a.c + cl;
    warp_pair_sum(s, c);
    if (lane == 0) sc->sums[out0 + q] = s + c;
  }
  __syncthreads();
  if (tid == 0) {
    bool bad = false;
    for (int q = 0; q < nq; ++q)
      if ((qmask >> q) & 1u) bad |= !isfinite(sc->sums[out0 + q]);
    if (mode == 1) {
      const double norm = sc->sums[out0 + 1] * dxyz;
      sc->norm = norm;
      if (stats) {
        sc->mu = sc->sums[out0 + 2] / sc->sums[out0 + 3];
        sc->errHe = sc->sums[out0] / N;
      }
      sc->scale = (renorm && norm > 0.0) ? sqrt(n4 / norm) : 1.0;
    }
    if (bad) atomicOr(&sc->flags, (unsigned)EP_FLAG_NONFINITE);
  }
}
