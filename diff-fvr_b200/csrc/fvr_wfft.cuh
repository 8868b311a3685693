// Warp-level complex FFT of length N = 32 M (M = 2, 3, 4, 5) held in
// registers: lane l holds x[l + 32 m], m < M.  Four-step split N = M x 32:
// an M-point DFT per lane, a twiddle W_N^(l k2), then a 32-point radix-2
// decimation-in-frequency across the lanes.  Unnormalised; INV selects
// e^{+2 pi i / N}.
//
// A butterfly across lanes l and l ^ h for two registers (p, p + M/2) swaps
// one register against the partner's other one, so each lane then holds both
// operands of one butterfly: one shuffle and one butterfly per lane, where
// exchanging both registers takes two shuffles and computes every sum and
// difference in both lanes.  The swap trades lane bit h for the register bit,
// which leaves the frequencies in the order of wfft_elem.  An odd M's last
// register keeps the plain exchange.  (M = 4: 20 shuffles and about 170
// instructions a transform, 40 and 270 with the plain exchange.)
#pragma once

#include "fvr_dft.cuh"

namespace fvr {

__device__ __forceinline__ int brev4(int x) { return static_cast<int>(__brev(static_cast<unsigned>(x)) >> 28); }
__device__ __forceinline__ int brev5(int x) { return static_cast<int>(__brev(static_cast<unsigned>(x)) >> 27); }

// Transform element held by register `slot` of lane `lane`.
template <int M>
__device__ __forceinline__ int wfft_elem(int lane, int slot) {
  constexpr int MH = M / 2;
  if (M % 2 && slot == M - 1) return M - 1 + M * brev5(lane);
  const int hi = slot >= MH ? 1 : 0;
  return slot - MH * hi + MH * (lane >> 4) + M * (brev4(lane & 15) + 16 * hi);
}

// Position lane + 32 slot of transform element k.
template <int M>
__device__ __forceinline__ int wfft_pos(int k) {
  constexpr int MH = M / 2;
  const int q = k / M, k2 = k - q * M;
  if (M % 2 && k2 == M - 1) return brev5(q) + 32 * (M - 1);
  const int r = k2 >= MH ? 1 : 0;
  return 16 * r + brev4(q & 15) + 32 * (k2 - MH * r + MH * (q >> 4));
}

template <int M, bool INV>
struct WarpFft {
  Cx<float> stw[4];  // stage s (half size h = 16 >> s): W_{2h}^(l mod h), negated in the upper lanes (l & h)
  Cx<float> itw[M];  // W_N^(l k2)

  __device__ __forceinline__ void init(int lane) {
    constexpr float sgn = INV ? 1.f : -1.f;
#pragma unroll
    for (int s = 0; s < 4; ++s) {
      const int h = 16 >> s;
      float sn, cs;
      sincospif(static_cast<float>(lane % h) / static_cast<float>(h), &sn, &cs);
      stw[s] = lane & h ? Cx<float>{-cs, -sgn * sn} : Cx<float>{cs, sgn * sn};
    }
#pragma unroll
    for (int k = 0; k < M; ++k) {
      float sn, cs;
      sincospif(2.f * static_cast<float>(lane * k) / static_cast<float>(32 * M), &sn, &cs);
      itw[k] = Cx<float>{cs, sgn * sn};
    }
  }

  // Packed (FP32x2) sum and difference; each component rounds as the scalar form.
  static __device__ __forceinline__ Cx<float> add(Cx<float> a, Cx<float> b) {
    const float2 r = __fadd2_rn(make_float2(a.x, a.y), make_float2(b.x, b.y));
    return Cx<float>{r.x, r.y};
  }
  static __device__ __forceinline__ Cx<float> sub(Cx<float> a, Cx<float> b) {
    const float2 r = __ffma2_rn(make_float2(b.x, b.y), make_float2(-1.f, -1.f), make_float2(a.x, a.y));
    return Cx<float>{r.x, r.y};
  }

  // (keep - other) times the stage's twiddle; the sign makes it lower minus
  // upper operand in both lanes.
  __device__ __forceinline__ Cx<float> diff(Cx<float> keep, Cx<float> other, int s, bool upper) const {
    const Cx<float> d = sub(keep, other);
    if (s < 4) return cmul(d, stw[s]);
    return upper ? Cx<float>{-d.x, -d.y} : d;
  }

  __device__ __forceinline__ void run(Cx<float> (&x)[M], int lane) const {
    constexpr int MH = M / 2;
    Dft<float, M>::run(x, INV);
#pragma unroll
    for (int k = 1; k < M; ++k) x[k] = cmul(x[k], itw[k]);
#pragma unroll
    for (int s = 0; s < 5; ++s) {
      const int h = 16 >> s;
      const bool upper = (lane & h) != 0;
#pragma unroll
      for (int p = 0; p < MH; ++p) {
        const Cx<float> a = x[p], b = x[p + MH];
        const Cx<float> send = upper ? a : b, keep = upper ? b : a;
        Cx<float> v;
        v.x = __shfl_xor_sync(0xffffffffu, send.x, h);
        v.y = __shfl_xor_sync(0xffffffffu, send.y, h);
        x[p] = add(keep, v);
        x[p + MH] = diff(keep, v, s, upper);
      }
      if (M % 2) {
        Cx<float> v;
        v.x = __shfl_xor_sync(0xffffffffu, x[M - 1].x, h);
        v.y = __shfl_xor_sync(0xffffffffu, x[M - 1].y, h);
        const Cx<float> d = diff(x[M - 1], v, s, upper);
        x[M - 1] = upper ? d : add(x[M - 1], v);
      }
    }
  }
};

}  // namespace fvr
