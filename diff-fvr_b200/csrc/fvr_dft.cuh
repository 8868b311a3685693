// Small fixed-radix DFTs on registers (radix 2, 3, 4, 5), shared by the
// shared-memory line FFTs and the warp-level FFTs, with the mixed-radix plan
// and the Stockham butterfly of the former.
// Sign: forward e^{-2 pi i / r}, inverse e^{+2 pi i / r}; unnormalised.
#pragma once

#include "fvr_common.cuh"

namespace fvr {

template <typename T>
__device__ __forceinline__ Cx<T> mul_i(Cx<T> a, bool neg) {  // +i*a  or  -i*a
  return neg ? Cx<T>{a.y, -a.x} : Cx<T>{-a.y, a.x};
}

template <typename T, int R>
struct Dft;

template <typename T>
struct Dft<T, 2> {
  __device__ __forceinline__ static void run(Cx<T> (&v)[2], bool) {
    Cx<T> a = v[0];
    v[0] = cadd(a, v[1]);
    v[1] = csub(a, v[1]);
  }
};

template <typename T>
struct Dft<T, 4> {
  __device__ __forceinline__ static void run(Cx<T> (&v)[4], bool inv) {
    Cx<T> a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
    Cx<T> c = cadd(v[1], v[3]), d = csub(v[1], v[3]);
    Cx<T> id = mul_i(d, !inv);  // forward: -i d
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = cadd(b, id);
    v[3] = csub(b, id);
  }
};

template <typename T>
struct Dft<T, 3> {
  __device__ __forceinline__ static void run(Cx<T> (&v)[3], bool inv) {
    const T s3 = static_cast<T>(0.86602540378443864676372317075294);  // sqrt(3)/2
    Cx<T> t1 = cadd(v[1], v[2]), t2 = csub(v[1], v[2]);
    Cx<T> m{v[0].x - static_cast<T>(0.5) * t1.x, v[0].y - static_cast<T>(0.5) * t1.y};
    Cx<T> st{s3 * t2.x, s3 * t2.y};
    Cx<T> ist = mul_i(st, !inv);  // forward: -i s t2
    v[0] = cadd(v[0], t1);
    v[1] = cadd(m, ist);
    v[2] = csub(m, ist);
  }
};

template <typename T>
struct Dft<T, 5> {
  __device__ __forceinline__ static void run(Cx<T> (&v)[5], bool inv) {
    const T c1 = static_cast<T>(0.30901699437494742410229341718282);   // cos(2pi/5)
    const T c2 = static_cast<T>(-0.80901699437494742410229341718282);  // cos(4pi/5)
    const T s1 = static_cast<T>(0.95105651629515357211643933337938);   // sin(2pi/5)
    const T s2 = static_cast<T>(0.58778525229247312916870595463907);   // sin(4pi/5)
    Cx<T> t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
    Cx<T> t3 = csub(v[1], v[4]), t4 = csub(v[2], v[3]);
    Cx<T> a1{v[0].x + c1 * t1.x + c2 * t2.x, v[0].y + c1 * t1.y + c2 * t2.y};
    Cx<T> a2{v[0].x + c2 * t1.x + c1 * t2.x, v[0].y + c2 * t1.y + c1 * t2.y};
    Cx<T> b1{s1 * t3.x + s2 * t4.x, s1 * t3.y + s2 * t4.y};
    Cx<T> b2{s2 * t3.x - s1 * t4.x, s2 * t3.y - s1 * t4.y};
    Cx<T> ib1 = mul_i(b1, !inv), ib2 = mul_i(b2, !inv);  // forward: -i b
    v[0] = Cx<T>{v[0].x + t1.x + t2.x, v[0].y + t1.y + t2.y};
    v[1] = cadd(a1, ib1);
    v[4] = csub(a1, ib1);
    v[2] = cadd(a2, ib2);
    v[3] = csub(a2, ib2);
  }
};

constexpr int kMaxPass = 24;
// Largest prime factor of a transform length (direct DFT pass, O(n * p) work).
constexpr int kMaxPrime = 127;

struct FftPlan {
  int n;
  int npass;
  int radix[kMaxPass];
};

inline bool make_plan(int64_t n, FftPlan* plan) {
  if (n < 1 || n > 16384) return false;
  plan->n = static_cast<int>(n);
  plan->npass = 0;
  int64_t m = n;
  const int order[] = {4, 2, 3, 5, 7, 11, 13};
  for (int r : order) {
    while (m % r == 0) {
      if (plan->npass >= kMaxPass) return false;
      plan->radix[plan->npass++] = r;
      m /= r;
    }
  }
  // remaining odd prime factors up to kMaxPrime run as direct DFT passes
  for (int r = 17; r <= kMaxPrime && m > 1; r += 2) {
    while (m % r == 0) {
      if (plan->npass >= kMaxPass) return false;
      plan->radix[plan->npass++] = r;
      m /= r;
    }
  }
  return m == 1;
}

template <typename T, int R>
__device__ __forceinline__ void bfly(const Cx<T>* __restrict__ src, Cx<T>* __restrict__ dst, int j, int Ns, int n,
                                     const Cx<T>* __restrict__ tw, bool inv) {
  const int nb = n / R;
  const int k = j % Ns;
  Cx<T> v[R];
#pragma unroll
  for (int t = 0; t < R; ++t) v[t] = src[j + t * nb];
  if (Ns > 1) {
    const int step = n / (Ns * R);
#pragma unroll
    for (int t = 1; t < R; ++t) {
      Cx<T> w = tw[k * t * step];
      if (inv) w.y = -w.y;
      v[t] = cmul(v[t], w);
    }
  }
  Dft<T, R>::run(v, inv);
  const int idx = (j / Ns) * Ns * R + k;
#pragma unroll
  for (int t = 0; t < R; ++t) dst[idx + t * Ns] = v[t];
}

}  // namespace fvr
