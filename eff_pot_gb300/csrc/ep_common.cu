// ep_common.cu - launch accounting and the reduction finalize kernel.
#include <cmath>

#include "ep_engine.h"

int Prof::cls(const char* name) {
  for (size_t i = 0; i < names.size(); ++i)
    if (names[i] == name) return (int)i;
  names.emplace_back(name);
  ms.push_back(0.0);
  cnt.push_back(0);
  return (int)names.size() - 1;
}

cudaEvent_t Prof::ev() {
  if (!pool.empty()) {
    cudaEvent_t e = pool.back();
    pool.pop_back();
    return e;
  }
  cudaEvent_t e = nullptr;
  cudaEventCreate(&e);
  return e;
}

void Prof::begin(cudaStream_t st, const char* name, cudaEvent_t& a, int& c) {
  ++launches;
  if (!on) return;
  c = cls(name);
  a = ev();
  cudaEventRecord(a, st);
}

void Prof::end(cudaStream_t st, int c, cudaEvent_t a) {
  if (!on || c < 0) return;
  cudaEvent_t b = ev();
  cudaEventRecord(b, st);
  pending.push_back({c, a, b});
}

void Prof::collect() {
  if (pending.empty()) return;
  cudaEventSynchronize(pending.back().b);
  for (auto& r : pending) {
    float t = 0.f;
    if (cudaEventElapsedTime(&t, r.a, r.b) == cudaSuccess) {
      ms[r.cls] += t;
      cnt[r.cls] += 1;
    }
    pool.push_back(r.a);
    pool.push_back(r.b);
  }
  pending.clear();
}

void Prof::release() {
  collect();
  for (cudaEvent_t e : pool) cudaEventDestroy(e);
  pool.clear();
}

// One CTA per sum q: every thread adds its share of the block pairs
// (Neumaier), then a pair tree across the CTA.  With one CTA for all sums the
// chain of compensated FP64 additions, on one SM's FP64 pipe, took 34 us for
// 8 sums of 1216 blocks and 50 us for 9 (512 and 576 blocks in this form: 8-10).
__global__ void __launch_bounds__(128) k_finalize(const double* __restrict__ partials, int nblocks, int nq,
                                                  DevScalars* sc, int out0, int mode, double dxyz, double n4) {
  __shared__ double rs[4], rc[4];
  const int q = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double* lo = partials + (long long)nblocks * nq;
  Acc<double> a;
  for (int b = threadIdx.x; b < nblocks; b += 128) {
    a.add(__ldcg(partials + (long long)b * nq + q));
    a.c += __ldcg(lo + (long long)b * nq + q);
  }
  double s = a.s, c = a.c;
  warp_pair_sum(s, c);
  if (lane == 0) {
    rs[warp] = s;
    rc[warp] = c;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 4; ++w) pair_add(s, c, rs[w], rc[w]);
    const double v = s + c;
    sc->sums[out0 + q] = v;
    bool bad = !isfinite(v);
    if (mode == 2) {
      const double norm = v * dxyz;
      sc->norm = norm;
      sc->scale = norm > 0.0 ? sqrt(n4 / norm) : 1.0;
      bad |= !(norm > 0.0);
    }
    if (bad && mode != 3) atomicOr(&sc->flags, (unsigned)EP_FLAG_NONFINITE);
  }
}

__global__ void k_reset_scales(DevScalars* sc) {
  if (threadIdx.x < EP_NSLOTS) {
    sc->bscale[threadIdx.x] = 1.0;
    sc->bscale_f[threadIdx.x] = 1.0f;
  }
  if (threadIdx.x == 0) sc->den_scale = 1.0;
}
