// Image-similarity kernels of the registration loss, sm_100a: the
// edge-dominant gradient NCC (src/fvr/cone_beam_fvr.py:71-112) and the
// zero-mean image NCC it is mixed with
// (experiments/exp30_gpu_multistart_registration.py:120-134).
//
// For each image pair (pred a, target b) and channel: Sobel x / y responses
// (zero padding) on the interior [crop, H-crop) x [crop, W-crop), their NCC
// per direction, averaged; optionally the same on 3x3 box-blurred images
// (zero padding, divisor 9) weighted by w; optionally the NCC of the whole
// images.  Everything is expressed through five moments per combination
// -- S_u, S_v, S_uu, S_vv, S_uv -- so the forward pass is one stencil +
// reduction pass over the images and the adjoint is one stencil pass that
// applies the transposed Sobel and box filters to closed-form fields.
//
// Both passes march: a warp owns a strip of 64 columns (two per lane, the
// outer lanes are halo) and walks down 8 to 32 rows, keeping the last rows'
// horizontal sums in registers; horizontal neighbours come from the lane's
// other column or one shuffle.  The pair (a, b) goes through the filters as
// one packed f32x2 value.  No shared memory and no barriers.  Measured on 64
// candidates x two views of 256 x 256 (kernel times): an earlier form with
// 32 x 32 tiles in shared memory took 2 x 43 us (moments), 2 x 119 us
// (finalize, one CTA for all pairs) and 2 x 91 us (adjoint), the image NCC
// another 350 us as separate tensor operations; now 57, 9 and 66 us for both
// views and both similarities.  The moments and adjoint passes are bound by
// issued instructions (the images alone take 5 and 10 us at the copy
// bandwidth).  A CTA is one warp, so that an SM starts the next strip whenever
// one of its warps is done.
#include "fvr_common.cuh"

namespace fvr {

constexpr int kEdgeMom = 5;       // S_u, S_v, S_uu, S_vv, S_uv
constexpr int kEdgeCombos = 4;    // fine x, fine y, coarse x, coarse y
constexpr int kEdgeStats = kEdgeCombos * kEdgeMom;     // moments kept for the backward of the edge NCC
constexpr int kEdgeNM = kEdgeStats + kEdgeMom;         // ... and of the registration loss: the whole images'
constexpr int kEdgeMaxViews = 4;
constexpr int kMomCols = 60;      // columns it produces: 64 less two halo columns a side
constexpr int kGradCols = 56;     // ... four halo columns a side

struct EdgeArgs {
  const float* a[kEdgeMaxViews];  // per view [B][C][H][W]
  const float* b[kEdgeMaxViews];  // [Bt][C][H][W], Bt = 1 (broadcast) or B
  int Bt[kEdgeMaxViews];
  float* grad[kEdgeMaxViews];     // adjoint: [B][C][H][W]
  int views, B, Cch, H, W, crop;
  int coarse;        // 1: blurred scale enabled
  int nm;            // moments per pair in stats: kEdgeStats or kEdgeNM
  int rows;          // rows a CTA (one warp) produces
  int vec;           // 1: every row starts on an 8-byte boundary
  double base, ce, cn;  // out = base + sum over views (ce edge + cn ncc)
  float w;           // weight of the blurred scale
};

struct EdgeJob {
  const float *a, *b;
  int view, bi, ch;
  int rb, re;        // rows [rb, re) of this warp
  int strip;
};

// Pair p = (view, item, channel); job j of the pair = (row chunk, strip).
__device__ __forceinline__ EdgeJob edge_job(const EdgeArgs& e, int64_t pair, int job, int strips) {
  EdgeJob j;
  j.view = static_cast<int>(pair / (e.B * e.Cch));
  const int r = static_cast<int>(pair - static_cast<int64_t>(j.view) * e.B * e.Cch);
  j.bi = r / e.Cch;
  j.ch = r - j.bi * e.Cch;
  const int64_t plane = static_cast<int64_t>(e.H) * e.W;
  j.a = e.a[j.view] + (static_cast<int64_t>(j.bi) * e.Cch + j.ch) * plane;
  j.b = e.b[j.view] + (static_cast<int64_t>(e.Bt[j.view] == 1 ? 0 : j.bi) * e.Cch + j.ch) * plane;
  const int chunk = job / strips;
  j.strip = job - chunk * strips;
  j.rb = chunk * e.rows;
  j.re = min(e.H, j.rb + e.rows);
  return j;
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ float2 twice_plus(float2 a, float2 b) { return __ffma2_rn(a, make_float2(2.f, 2.f), b); }
__device__ __forceinline__ float2 shfl_up2(float2 v) {
  return make_float2(__shfl_up_sync(0xffffffffu, v.x, 1), __shfl_up_sync(0xffffffffu, v.y, 1));
}
__device__ __forceinline__ float2 shfl_down2(float2 v) {
  return make_float2(__shfl_down_sync(0xffffffffu, v.x, 1), __shfl_down_sync(0xffffffffu, v.y, 1));
}

// Walks down the rows of both images at columns c, c + 1, as (a, b) pairs,
// zero outside; two rows are in flight ahead of the one handed out.
struct RowReader {
  const float *a, *b;  // next row to load, at column c
  int r, H, W, c;
  bool vec, in0, in1;
  float2 n0[2], n1[2];

  __device__ __forceinline__ void load(float2 (&x)[2]) {
    x[0] = x[1] = make_float2(0.f, 0.f);
    if (r >= 0 && r < H) {
      if (vec) {  // W and c even: both columns are inside or neither
        if (in0) {
          const float2 u = __ldg(reinterpret_cast<const float2*>(a));
          const float2 v = __ldg(reinterpret_cast<const float2*>(b));
          x[0] = make_float2(u.x, v.x);
          x[1] = make_float2(u.y, v.y);
        }
      } else {
        if (in0) x[0] = make_float2(__ldg(a), __ldg(b));
        if (in1) x[1] = make_float2(__ldg(a + 1), __ldg(b + 1));
      }
    }
    ++r;
    a += W;
    b += W;
  }
  __device__ __forceinline__ void init(const EdgeArgs& e, const float* ia, const float* ib, int row, int col) {
    r = row;
    H = e.H;
    W = e.W;
    c = col;
    vec = e.vec != 0;
    in0 = c >= 0 && c < W;
    in1 = c + 1 >= 0 && c + 1 < W;
    const int64_t o = static_cast<int64_t>(row) * W + col;
    a = ia + o;  // read only where the row and the column are inside
    b = ib + o;
    load(n0);
    load(n1);
  }
  __device__ __forceinline__ void next(float2 (&x)[2]) {
    x[0] = n0[0];
    x[1] = n0[1];
    n0[0] = n1[0];
    n0[1] = n1[1];
    load(n1);
  }
};

// Horizontal parts of the filters at the lane's two columns: d = right - left
// (Sobel x), s = left + 2 mid + right (Sobel y), h = left + mid + right (box).
// The outermost column on each side of the warp comes out wrong (halo).
__device__ __forceinline__ void row_parts(const float2 (&x)[2], float2 (&d)[2], float2 (&s)[2], float2 (&h)[2]) {
  const float2 l = shfl_up2(x[1]), r = shfl_down2(x[0]);
  d[0] = sub2(x[1], l);
  d[1] = sub2(r, x[0]);
  const float2 t0 = add2(x[1], l), t1 = add2(r, x[0]);
  s[0] = twice_plus(x[0], t0);
  s[1] = twice_plus(x[1], t1);
  h[0] = add2(t0, x[0]);
  h[1] = add2(t1, x[1]);
}

// The last two rows' horizontal parts of the images and of the blurred
// images.  step() takes row t and gives the Sobel responses g of row t - 1
// and, with COARSE, those of the blurred images, gb, of row t - 2.
template <bool COARSE>
struct EdgeMarch {
  float2 d0[2], d1[2], s0[2], s1[2], h0[2], h1[2];      // rows t - 2, t - 1
  float2 bd0[2], bd1[2], bs0[2], bs1[2];                // blurred rows t - 3, t - 2

  __device__ __forceinline__ void init() {
#pragma unroll
    for (int j = 0; j < 2; ++j)
      d0[j] = d1[j] = s0[j] = s1[j] = h0[j] = h1[j] = bd0[j] = bd1[j] = bs0[j] = bs1[j] = make_float2(0.f, 0.f);
  }

  // in_row: row t - 1 lies in the image; in_col[j]: column j does.
  __device__ __forceinline__ void step(const float2 (&x)[2], bool in_row, const bool (&in_col)[2], float2 (&gx)[2],
                                       float2 (&gy)[2], float2 (&gbx)[2], float2 (&gby)[2]) {
    float2 d[2], s[2], h[2];
    row_parts(x, d, s, h);
    float2 bl[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      gx[j] = twice_plus(d1[j], add2(d0[j], d[j]));
      gy[j] = sub2(s[j], s0[j]);
      d0[j] = d1[j];
      d1[j] = d[j];
      s0[j] = s1[j];
      s1[j] = s[j];
      if (COARSE) {
        const float2 v = __fmul2_rn(add2(add2(h0[j], h1[j]), h[j]), make_float2(1.f / 9.f, 1.f / 9.f));
        bl[j] = in_row && in_col[j] ? v : make_float2(0.f, 0.f);
        h0[j] = h1[j];
        h1[j] = h[j];
      }
    }
    if (COARSE) {
      float2 bd[2], bs[2], unused[2];
      row_parts(bl, bd, bs, unused);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        gbx[j] = twice_plus(bd1[j], add2(bd0[j], bd[j]));
        gby[j] = sub2(bs[j], bs0[j]);
        bd0[j] = bd1[j];
        bd1[j] = bd[j];
        bs0[j] = bs1[j];
        bs1[j] = bs[j];
      }
    }
  }
};

// Sums 32 per-lane values over the warp; lane l returns the total of v[l].
// Each step halves the values a lane carries: 31 exchanges instead of 160.
__device__ __forceinline__ double warp_sum_each(double (&v)[32]) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const double send = up ? v[i] : v[i + o];
      const double keep = up ? v[i + o] : v[i];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
    }
  }
  return v[0];
}

// Moments of one strip of rows -> partial[pair][job][kEdgeNM] (fp64).  Products
// are summed per lane in f32 over two rows (four terms), then in fp64: 57 us for
// 64 candidates x two views of 256 x 256, and 54 with all 64 terms of a lane in
// f32, 64 with four warps to a CTA.  The
// whole images' mean may be large against their spread, so those moments are
// taken about a value of the lane's own first row and moved to zero in fp64.
template <bool COARSE, bool NCC>
__global__ void __launch_bounds__(32, 12) edge_moments_kernel(EdgeArgs e, int strips, int jobs,
                                                              double* __restrict__ partial) {
  const int64_t pair = blockIdx.x / jobs;
  const int job = static_cast<int>(blockIdx.x - pair * jobs);
  const int lane = threadIdx.x;
  const EdgeJob jb = edge_job(e, pair, job, strips);
  const int c = jb.strip * kMomCols - 2 + 2 * lane;
  const bool own = lane >= 1 && lane <= 30;
  bool in_img[2], in_edge[2], mine[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    in_img[j] = c + j >= 0 && c + j < e.W;
    mine[j] = own && in_img[j];
    in_edge[j] = own && c + j >= e.crop && c + j < e.W - e.crop;
  }
  float2 m1[kEdgeCombos] = {}, m2[kEdgeCombos] = {};  // (S_u, S_v), (S_uu, S_vv) of at most two rows
  float m3[kEdgeCombos] = {};                         // S_uv
  double sum[kEdgeNM] = {};                           // ... of all rows
  auto add = [&](int k, float2 g) {
    m1[k] = add2(m1[k], g);
    m2[k] = __ffma2_rn(g, g, m2[k]);
    m3[k] = fmaf(g.x, g.y, m3[k]);
  };
  float2 pivot = make_float2(0.f, 0.f), i1, i2;  // whole images: sums of (x - pivot), squares
  float i3;
  auto clear = [&] {
#pragma unroll
    for (int k = 0; k < kEdgeCombos; ++k) {
      m1[k] = m2[k] = make_float2(0.f, 0.f);
      m3[k] = 0.f;
    }
    i1 = i2 = make_float2(0.f, 0.f);
    i3 = 0.f;
  };
  auto flush = [&] {
#pragma unroll
    for (int k = 0; k < (COARSE ? kEdgeCombos : 2); ++k) {
      double* s = sum + k * kEdgeMom;
      s[0] += m1[k].x;
      s[1] += m1[k].y;
      s[2] += m2[k].x;
      s[3] += m2[k].y;
      s[4] += m3[k];
    }
    if (NCC) {
      double* s = sum + kEdgeStats;
      s[0] += i1.x;
      s[1] += i1.y;
      s[2] += i2.x;
      s[3] += i2.y;
      s[4] += i3;
    }
  };
  const int lo = max(jb.rb, e.crop), hi = min(jb.re, e.H - e.crop);  // interior rows of this job
  EdgeMarch<COARSE> march;
  march.init();
  const int t_end = jb.re + (COARSE ? 2 : 1);
  RowReader rows;
  rows.init(e, jb.a, jb.b, jb.rb - 2, c);
  int t = jb.rb - 2;
  auto row = [&] {
    float2 x[2];
    rows.next(x);
    if (NCC && t >= jb.rb && t < jb.re) {
      if (t == jb.rb) pivot = x[0];  // the lane's first column: the second may lie outside
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (mine[j]) {
          const float2 u = sub2(x[j], pivot);
          i1 = add2(i1, u);
          i2 = __ffma2_rn(u, u, i2);
          i3 = fmaf(u.x, u.y, i3);
        }
    }
    float2 gx[2], gy[2], gbx[2], gby[2];
    march.step(x, t - 1 >= 0 && t - 1 < e.H, in_img, gx, gy, gbx, gby);
    if (t - 1 >= lo && t - 1 < hi) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (in_edge[j]) {
          add(0, gx[j]);
          add(1, gy[j]);
        }
    }
    if (COARSE && t - 2 >= lo && t - 2 < hi) {
#pragma unroll
      for (int j = 0; j < 2; ++j)
        if (in_edge[j]) {
          add(2, gbx[j]);
          add(3, gby[j]);
        }
    }
    ++t;
  };
  while (t < t_end) {  // a row past the end adds nothing
    clear();
    row();
    row();
    flush();
  }
  double v[32];
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = 0.0;
#pragma unroll
  for (int k = 0; k < kEdgeStats; ++k) v[k] = sum[k];
  if (NCC) {
    const double n = static_cast<double>((mine[0] ? 1 : 0) + (mine[1] ? 1 : 0)) * (jb.re - jb.rb);
    const double pu = pivot.x, pv = pivot.y, su = sum[kEdgeStats], sv = sum[kEdgeStats + 1];
    double* im = v + kEdgeStats;
    im[0] = su + n * pu;
    im[1] = sv + n * pv;
    im[2] = sum[kEdgeStats + 2] + pu * (2.0 * su + n * pu);
    im[3] = sum[kEdgeStats + 3] + pv * (2.0 * sv + n * pv);
    im[4] = sum[kEdgeStats + 4] + pu * sv + pv * su + n * pu * pv;
  }
  const double s = warp_sum_each(v);
  if (lane < kEdgeNM) partial[(pair * jobs + job) * kEdgeNM + lane] = s;
}

// NCC of one combination from its moments over n pixels, denominator
// sqrt(max(S_uu S_vv, 1e-12)) of the centred sums.
__device__ __forceinline__ double edge_ncc(const double* m, double n) {
  const double suu = m[2] - m[0] * m[0] / n, svv = m[3] - m[1] * m[1] / n, suv = m[4] - m[0] * m[1] / n;
  return suv / sqrt(fmax(suu * svv, 1e-12));
}

// One CTA of NW warps per batch item: strip sums -> stats[pair][nm] in a fixed order,
// then out = base + sum over views (ce edge + cn ncc), edge = the channel mean
// of (1 - w) fine + w coarse.
template <int NW>
__global__ void __launch_bounds__(32 * NW) edge_finalize_kernel(EdgeArgs e, int jobs,
                                                               const double* __restrict__ partial,
                                                               double* __restrict__ stats, float* __restrict__ out,
                                                               double* __restrict__ value) {
  __shared__ double part[NW][kEdgeNM];
  const int bi = blockIdx.x, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const double n = static_cast<double>(e.H - 2 * e.crop) * static_cast<double>(e.W - 2 * e.crop);
  const double n_img = static_cast<double>(e.H) * static_cast<double>(e.W);
  double val = e.base;
  for (int v = 0; v < e.views; ++v) {
    double edge = 0.0, ncc = 0.0;
    for (int ch = 0; ch < e.Cch; ++ch) {
      const int64_t pair = (static_cast<int64_t>(v) * e.B + bi) * e.Cch + ch;
      if (lane < kEdgeNM) {
        double s = 0.0;
#pragma unroll 8
        for (int t = wid; t < jobs; t += NW) s += partial[(pair * jobs + t) * kEdgeNM + lane];
        part[wid][lane] = s;
      }
      __syncthreads();
      if (threadIdx.x < kEdgeNM) {
        double s = 0.0;
#pragma unroll
        for (int k = 0; k < NW; ++k) s += part[k][lane];
        part[0][lane] = s;
        if (lane < e.nm) stats[pair * e.nm + lane] = s;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        const double* st = part[0];
        const double fine = 0.5 * (edge_ncc(st, n) + edge_ncc(st + kEdgeMom, n));
        edge += e.coarse ? (1.0 - e.w) * fine +
                               e.w * 0.5 * (edge_ncc(st + 2 * kEdgeMom, n) + edge_ncc(st + 3 * kEdgeMom, n))
                         : fine;
        if (e.cn != 0.0) ncc += edge_ncc(st + kEdgeCombos * kEdgeMom, n_img);
      }
      __syncthreads();
    }
    val += e.ce * edge / e.Cch + e.cn * ncc / e.Cch;
  }
  if (threadIdx.x == 0) {
    if (out) out[bi] = static_cast<float>(val);
    if (value) value[bi] = val;
  }
}

// out[0] = mean of value[B], in a fixed order.
__global__ void edge_mean_kernel(const double* __restrict__ value, int B, float* __restrict__ out) {
  double s = 0.0;
  for (int i = threadIdx.x; i < B; i += 32) s += value[i];
  s = warp_sum(s);
  if (threadIdx.x == 0) out[0] = static_cast<float>(s / B);
}

// d out / d a (or d b with swap) of one strip of rows.  Interior gradient
// fields g_k(q) = alpha_k (v_k(q) - mean v_k) + beta_k (u_k(q) - mean u_k) on
// the interior, transposed Sobel, and for the blurred scale the transposed box
// filter; the fine and the coarse fields go through the transposed Sobel
// together as one f32x2 value.  Row t enters, row t - 4 leaves.  Sixteen
// warps an SM, 66 us (twelve warps, without spills: 69; CTAs of four warps: 71
// with twelve and 84 with sixteen).
template <bool COARSE, bool NCC>
__global__ void __launch_bounds__(32, 16) edge_grad_kernel(EdgeArgs e, int strips, int jobs,
                                                           const double* __restrict__ stats,
                                                           const float* __restrict__ g, int64_t g_stride,
                                                           double g_scale, int swap) {
  // alpha, beta, -mean u, -mean v, and what the means' rounding to float leaves of alpha mean v + beta mean u
  __shared__ float4 coef[kEdgeCombos + 1];
  __shared__ float rest[kEdgeCombos + 1];
  const int64_t pair = blockIdx.x / jobs;
  const int lane = threadIdx.x;
  const EdgeJob jb = edge_job(e, pair, static_cast<int>(blockIdx.x - pair * jobs), strips);
  if (threadIdx.x < kEdgeCombos + 1) {
    const int k = threadIdx.x;
    const bool kept = (k + 1) * kEdgeMom <= e.nm;
    const double none[kEdgeMom] = {0.0, 0.0, 0.0, 0.0, 0.0};
    const double* m = kept ? stats + pair * e.nm + k * kEdgeMom : none;
    // u = the differentiated image's response, v = the other one's
    const double su = swap ? m[1] : m[0], sv = swap ? m[0] : m[1];
    const double suu_raw = swap ? m[3] : m[2], svv_raw = swap ? m[2] : m[3];
    const bool whole = k == kEdgeCombos;
    const double n = whole ? static_cast<double>(e.H) * static_cast<double>(e.W)
                           : static_cast<double>(e.H - 2 * e.crop) * static_cast<double>(e.W - 2 * e.crop);
    const double suu = suu_raw - su * su / n, svv = svv_raw - sv * sv / n, suv = m[4] - m[0] * m[1] / n;
    const double prod = suu * svv, den = sqrt(fmax(prod, 1e-12));
    const double sw = k < 2 ? (e.coarse ? 1.0 - e.w : 1.0) : (e.coarse ? static_cast<double>(e.w) : 0.0);
    const double wk = static_cast<double>(g[g_stride * jb.bi]) * g_scale * (whole ? e.cn : e.ce * sw * 0.5) / e.Cch;
    const double al = wk / den, be = prod > 1e-12 ? -wk * suv * svv / (den * den * den) : 0.0;
    const double mu = su / n, mv = sv / n;
    const float fu = static_cast<float>(mu), fv = static_cast<float>(mv);
    coef[k] = make_float4(static_cast<float>(al), static_cast<float>(be), -fu, -fv);
    rest[k] = static_cast<float>(al * (fv - mv) + be * (fu - mu));
  }
  __syncwarp();
  const int c = jb.strip * kGradCols - 4 + 2 * lane;
  const bool own = lane >= 2 && lane <= 29;
  bool in_img[2], in_edge[2];
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    in_img[j] = c + j >= 0 && c + j < e.W;
    in_edge[j] = c + j >= e.crop && c + j < e.W - e.crop;
  }
  // alpha (v - mean v) + beta (u - mean u): centred first, since a mean may be large against the spread
  float4 cc[kEdgeCombos + 1];
  float kk[kEdgeCombos + 1];
#pragma unroll
  for (int k = 0; k <= kEdgeCombos; ++k) {
    cc[k] = coef[k];
    kk[k] = rest[k];
  }
  auto fields = [&](int k, const float2 (&x)[2], float (&f)[2]) {
    const float4 c = cc[k];
    const float k0 = kk[k];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const float2 d = add2(x[j], make_float2(c.z, c.w));
      f[j] = fmaf(c.x, d.y, fmaf(c.y, d.x, k0));
    }
  };
  float* out = e.grad[jb.view] + (static_cast<int64_t>(jb.bi) * e.Cch + jb.ch) * static_cast<int64_t>(e.H) * e.W;
  EdgeMarch<COARSE> march;
  march.init();
  const float2 zero = make_float2(0.f, 0.f);
  float fx1[2] = {0.f, 0.f}, fy1[2] = {0.f, 0.f};             // fine fields of row t - 2
  float2 e0[2] = {zero, zero}, e1[2] = {zero, zero};          // transposed Sobel x parts of rows t - 4, t - 3
  float2 q0[2] = {zero, zero}, q1[2] = {zero, zero};          // transposed Sobel y parts
  float h0[2] = {0.f, 0.f}, h1[2] = {0.f, 0.f};               // box parts of rows t - 5, t - 4
  float of[2] = {0.f, 0.f};                                   // fine gradient of row t - 4
  float im0[2] = {0.f, 0.f}, im1[2] = {0.f, 0.f}, im2[2] = {0.f, 0.f}, im3[2] = {0.f, 0.f};  // rows t - 4 .. t - 1
  const int64_t W = e.W;
  RowReader rows;
  rows.init(e, swap ? jb.b : jb.a, swap ? jb.a : jb.b, jb.rb - 4, c);
#pragma unroll 4
  for (int t = jb.rb - 4; t < jb.re + 4; ++t) {
    float2 x[2];
    rows.next(x);
    float2 gx[2], gy[2], gbx[2], gby[2];
    march.step(x, t - 1 >= 0 && t - 1 < e.H, in_img, gx, gy, gbx, gby);
    const bool rf = t - 1 >= e.crop && t - 1 < e.H - e.crop, rc = t - 2 >= e.crop && t - 2 < e.H - e.crop;
    float2 Fx[2], Fy[2];  // (fine, coarse) fields of row t - 2
    float vx[2], vy[2];
    fields(0, gx, vx);
    fields(1, gy, vy);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      Fx[j] = make_float2(fx1[j], 0.f);
      Fy[j] = make_float2(fy1[j], 0.f);
      const bool f_in = rf && in_edge[j];
      fx1[j] = f_in ? vx[j] : 0.f;
      fy1[j] = f_in ? vy[j] : 0.f;
    }
    if (COARSE) {
      fields(2, gbx, vx);
      fields(3, gby, vy);
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const bool c_in = rc && in_edge[j];
        Fx[j].y = c_in ? vx[j] : 0.f;
        Fy[j].y = c_in ? vy[j] : 0.f;
      }
    }
    float2 xl, xr, yl, yr;
    if (COARSE) {
      xl = shfl_up2(Fx[1]);
      xr = shfl_down2(Fx[0]);
      yl = shfl_up2(Fy[1]);
      yr = shfl_down2(Fy[0]);
    } else {
      xl = make_float2(__shfl_up_sync(0xffffffffu, Fx[1].x, 1), 0.f);
      xr = make_float2(__shfl_down_sync(0xffffffffu, Fx[0].x, 1), 0.f);
      yl = make_float2(__shfl_up_sync(0xffffffffu, Fy[1].x, 1), 0.f);
      yr = make_float2(__shfl_down_sync(0xffffffffu, Fy[0].x, 1), 0.f);
    }
    const float2 ev[2] = {sub2(xl, Fx[1]), sub2(Fx[0], xr)};
    const float2 qv[2] = {twice_plus(Fy[0], add2(yl, Fy[1])), twice_plus(Fy[1], add2(Fy[0], yr))};
    const bool r3 = t - 3 >= 0 && t - 3 < e.H;
    float of_new[2], gb[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      // (fine gradient, gradient w.r.t. the blurred image) of row t - 3
      const float2 o = add2(twice_plus(e1[j], add2(e0[j], ev[j])), sub2(q0[j], qv[j]));
      e0[j] = e1[j];
      e1[j] = ev[j];
      q0[j] = q1[j];
      q1[j] = qv[j];
      of_new[j] = o.x;
      gb[j] = r3 && in_img[j] ? o.y : 0.f;
    }
    float bt[2] = {0.f, 0.f};
    if (COARSE) {
      const float l = __shfl_up_sync(0xffffffffu, gb[1], 1), r = __shfl_down_sync(0xffffffffu, gb[0], 1);
      const float m = gb[0] + gb[1];
      const float h[2] = {l + m, m + r};
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        bt[j] = ((h0[j] + h1[j]) + h[j]) * (1.f / 9.f);
        h0[j] = h1[j];
        h1[j] = h[j];
      }
    }
    float res[2], vn[2];
    if (NCC) fields(kEdgeCombos, x, vn);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      res[j] = of[j] + bt[j];
      of[j] = of_new[j];
      if (NCC) {
        res[j] += im0[j];
        im0[j] = im1[j];
        im1[j] = im2[j];
        im2[j] = im3[j];
        im3[j] = vn[j];
      }
    }
    const int r = t - 4;
    if (r >= jb.rb && own) {
      float* o = out + r * W + c;
      if (e.vec) {
        if (in_img[0]) *reinterpret_cast<float2*>(o) = make_float2(res[0], res[1]);
      } else {
        if (in_img[0]) o[0] = res[0];
        if (in_img[1]) o[1] = res[1];
      }
    }
  }
}

static int edge_common(int64_t B, int64_t C, int64_t H, int64_t W, int64_t crop, float w, EdgeArgs* e) {
  if (B < 1 || C < 1 || H < 3 || W < 3 || crop < 0) return FVR_ERR_ARG;
  if (H - 2 * crop < 1 || W - 2 * crop < 1 || B * C > 65535 || H > 32768 || W > 32768) return FVR_ERR_ARG;
  e->B = (int)B;
  e->Cch = (int)C;
  e->H = (int)H;
  e->W = (int)W;
  e->crop = (int)crop;
  e->nm = kEdgeStats;
  e->coarse = (w > 0.f && W >= 96) ? 1 : 0;  // the reference tests the last dim (cone_beam_fvr.py:86, 107)
  e->w = w;
  e->vec = W % 2 == 0 ? 1 : 0;
  return FVR_OK;
}

static int edge_view(EdgeArgs* e, int v, const float* a, const float* b, int64_t Bt, float* grad) {
  if (!a || !b || (Bt != 1 && Bt != e->B)) return FVR_ERR_ARG;
  e->a[v] = a;
  e->b[v] = b;
  e->Bt[v] = (int)Bt;
  e->grad[v] = grad;
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(grad)) & 7)
    e->vec = 0;
  return FVR_OK;
}

static int64_t edge_jobs(int64_t H, int64_t W, int rows, int cols) { return cdiv64(H, rows) * cdiv64(W, cols); }

// Rows per warp.  A warp's time is its rows and about six more (halo, prologue,
// sums) whether it is alone on an SM or one of the twelve that fit, so the
// moments take the rows with the shortest waves x (rows + 6), a smaller count
// only for a tenth less of it.  8 / 12 / 16 / 24 / 32 rows, us: one 256^2 image
// 5.8 / 7.1 / 8.4 / 11.0 / 13.7, 16 images 12.8 / 9.5 / 11.2 / 13.1 / 16.1, 64
// images 36 / 33 / 30 / 29 / 33, 64 x two views with the image NCC 77 / 68 / 63 /
// 59 / 57.
constexpr int kMomSlots = 148 * 12, kGradSlots = 148 * 16;
static int edge_mom_rows(int64_t pairs, int64_t H, int64_t W) {
  int best = 32;
  int64_t cost = 0;
  for (int rows : {32, 24, 16, 12, 8}) {
    const int64_t c = cdiv64(pairs * edge_jobs(H, W, rows, kMomCols), kMomSlots) * (rows + 6);
    if (cost == 0 || 10 * c < 9 * cost) {
      best = rows;
      cost = c;
    }
  }
  return best;
}

// The adjoint has eight halo rows and sixteen warps an SM: the fewest rows whose
// warps are on the GPU together, else 32, which issue least.  One 256^2 image
// 9.8 / 11.4 / 12.3 / 15.2 / 18.0, 16 images 21 / 15 / 17 / 18 / 21, 64 images
// 58 / 47 / 44 / 41 / 42, 64 x two views with the image NCC 100 / 85 / 76 / 67 / 67.
static int edge_grad_rows(int64_t pairs, int64_t H, int64_t W) {
  for (int rows : {8, 12, 16, 24})
    if (pairs * edge_jobs(H, W, rows, kGradCols) <= kGradSlots) return rows;
  return 32;
}

// Strip records, then one fp64 value per item (for the batch mean).
static int64_t edge_ws_bytes(int64_t views, int64_t B, int64_t C, int64_t H, int64_t W) {
  const int64_t pairs = views * B * C;
  return (pairs * edge_jobs(H, W, edge_mom_rows(pairs, H, W), kMomCols) * kEdgeNM + B) * (int64_t)sizeof(double);
}

static int64_t edge_pairs(const EdgeArgs& e) { return static_cast<int64_t>(e.views) * e.B * e.Cch; }

template <typename K>
static int edge_grid(const EdgeArgs& e, int cols, K launch) {
  const int64_t jobs = edge_jobs(e.H, e.W, e.rows, cols);
  const int64_t n = edge_pairs(e) * jobs;
  if (n > 2147483647) return FVR_ERR_ARG;
  launch(static_cast<unsigned>(n), static_cast<int>(cdiv64(e.W, cols)), static_cast<int>(jobs));
  FVR_LAUNCH_CHECK();
  return FVR_OK;
}

static int edge_forward(EdgeArgs e, void* workspace, double* stats, float* out, bool mean, cudaStream_t s) {
  double* part = static_cast<double*>(workspace);
  e.rows = edge_mom_rows(edge_pairs(e), e.H, e.W);
  const int rc = edge_grid(e, kMomCols, [&](unsigned n, int strips, int jobs) {
    if (e.coarse && e.cn != 0.0) edge_moments_kernel<true, true><<<n, 32, 0, s>>>(e, strips, jobs, part);
    else if (e.coarse) edge_moments_kernel<true, false><<<n, 32, 0, s>>>(e, strips, jobs, part);
    else if (e.cn != 0.0) edge_moments_kernel<false, true><<<n, 32, 0, s>>>(e, strips, jobs, part);
    else edge_moments_kernel<false, false><<<n, 32, 0, s>>>(e, strips, jobs, part);
  });
  if (rc) return rc;
  const int jobs = (int)edge_jobs(e.H, e.W, e.rows, kMomCols);
  double* value = part + edge_pairs(e) * jobs * kEdgeNM;
  if (e.B == 1) mean = false;  // of one item
  const auto finalize = jobs > 32 ? edge_finalize_kernel<16> : edge_finalize_kernel<4>;
  finalize<<<static_cast<unsigned>(e.B), jobs > 32 ? 512 : 128, 0, s>>>(e, jobs, part, stats, mean ? nullptr : out,
                                                                        mean ? value : nullptr);
  FVR_LAUNCH_CHECK();
  if (mean) {
    edge_mean_kernel<<<1, 32, 0, s>>>(value, e.B, out);
    FVR_LAUNCH_CHECK();
  }
  return FVR_OK;
}

static int edge_backward(EdgeArgs e, const double* stats, const float* g, int64_t g_stride, double g_scale, int swap,
                         cudaStream_t s) {
  e.rows = edge_grad_rows(edge_pairs(e), e.H, e.W);
  return edge_grid(e, kGradCols, [&](unsigned n, int strips, int jobs) {
    if (e.coarse && e.cn != 0.0)
      edge_grad_kernel<true, true><<<n, 32, 0, s>>>(e, strips, jobs, stats, g, g_stride, g_scale, swap);
    else if (e.coarse)
      edge_grad_kernel<true, false><<<n, 32, 0, s>>>(e, strips, jobs, stats, g, g_stride, g_scale, swap);
    else if (e.cn != 0.0)
      edge_grad_kernel<false, true><<<n, 32, 0, s>>>(e, strips, jobs, stats, g, g_stride, g_scale, swap);
    else
      edge_grad_kernel<false, false><<<n, 32, 0, s>>>(e, strips, jobs, stats, g, g_stride, g_scale, swap);
  });
}

static int reg_loss_args(const float* const* imgs, const float* const* refs, const int64_t* ref_batch, int views,
                         float* const* grads, int64_t B, int64_t H, int64_t W, int64_t crop, float ms_weight,
                         float edge_weight, EdgeArgs* e) {
  if (!imgs || !refs || !ref_batch || views < 1 || views > kEdgeMaxViews) return FVR_ERR_ARG;
  int rc = edge_common(B, 1, H, W, crop, ms_weight, e);
  if (rc) return rc;
  e->views = views;
  e->nm = kEdgeNM;
  e->base = 1.0;
  e->ce = -static_cast<double>(edge_weight) / views;
  e->cn = -(1.0 - static_cast<double>(edge_weight)) / views;
  for (int v = 0; v < views; ++v)
    if ((rc = edge_view(e, v, imgs[v], refs[v], ref_batch[v], grads ? grads[v] : nullptr))) return rc;
  return FVR_OK;
}

}  // namespace fvr

using namespace fvr;

extern "C" {

int64_t fvr_edge_ncc_workspace(int64_t B, int64_t C, int64_t H, int64_t W, int64_t crop) {
  if (B < 1 || C < 1 || H - 2 * crop < 1 || W - 2 * crop < 1) return 0;
  return edge_ws_bytes(1, B, C, H, W);
}

int64_t fvr_edge_ncc_stats_count(void) { return kEdgeStats; }

int fvr_edge_ncc_forward(const float* a, const float* b, int64_t B, int64_t Bt, int64_t C, int64_t H, int64_t W,
                         int64_t crop, float ms_weight, int reduction_mean, void* workspace, int64_t ws_bytes,
                         double* stats, float* out, void* stream) {
  EdgeArgs e{};
  int rc = edge_common(B, C, H, W, crop, ms_weight, &e);
  if (rc) return rc;
  e.views = 1;
  e.ce = 1.0;
  if ((rc = edge_view(&e, 0, a, b, Bt, nullptr))) return rc;
  if (!workspace || !stats || !out) return FVR_ERR_ARG;
  if (ws_bytes < fvr_edge_ncc_workspace(B, C, H, W, crop)) return FVR_ERR_WORKSPACE;
  return edge_forward(e, workspace, stats, out, reduction_mean != 0, static_cast<cudaStream_t>(stream));
}

int fvr_edge_ncc_backward(const float* a, const float* b, int64_t B, int64_t Bt, int64_t C, int64_t H, int64_t W,
                          int64_t crop, float ms_weight, int reduction_mean, const double* stats, const float* g,
                          int64_t g_stride, int wrt_b, float* grad, void* stream) {
  EdgeArgs e{};
  int rc = edge_common(B, C, H, W, crop, ms_weight, &e);
  if (rc) return rc;
  if (!stats || !g || !grad) return FVR_ERR_ARG;
  e.views = 1;
  e.ce = 1.0;
  if ((rc = edge_view(&e, 0, a, b, Bt, grad))) return rc;
  return edge_backward(e, stats, g, g_stride, reduction_mean ? 1.0 / static_cast<double>(B) : 1.0, wrt_b != 0,
                       static_cast<cudaStream_t>(stream));
}

int64_t fvr_reg_loss_workspace(int64_t views, int64_t B, int64_t H, int64_t W) {
  if (views < 1 || B < 1 || H < 1 || W < 1) return 0;
  return edge_ws_bytes(views, B, 1, H, W);
}

int64_t fvr_reg_loss_stats_count(void) { return kEdgeNM; }

int fvr_reg_loss_forward(const float* const* imgs, const float* const* refs, const int64_t* ref_batch, int views,
                         int64_t B, int64_t H, int64_t W, int64_t crop, float ms_weight, float edge_weight,
                         void* workspace, int64_t ws_bytes, double* stats, float* out, void* stream) {
  EdgeArgs e{};
  const int rc = reg_loss_args(imgs, refs, ref_batch, views, nullptr, B, H, W, crop, ms_weight, edge_weight, &e);
  if (rc) return rc;
  if (!workspace || !stats || !out) return FVR_ERR_ARG;
  if (ws_bytes < fvr_reg_loss_workspace(views, B, H, W)) return FVR_ERR_WORKSPACE;
  return edge_forward(e, workspace, stats, out, false, static_cast<cudaStream_t>(stream));
}

int fvr_reg_loss_backward(const float* const* imgs, const float* const* refs, const int64_t* ref_batch, int views,
                          int64_t B, int64_t H, int64_t W, int64_t crop, float ms_weight, float edge_weight,
                          const double* stats, const float* g, int64_t g_stride, float* const* grads, void* stream) {
  if (!stats || !g || !grads) return FVR_ERR_ARG;
  for (int v = 0; v < views && v < kEdgeMaxViews; ++v)
    if (!grads[v]) return FVR_ERR_ARG;
  EdgeArgs e{};
  const int rc = reg_loss_args(imgs, refs, ref_batch, views, grads, B, H, W, crop, ms_weight, edge_weight, &e);
  if (rc) return rc;
  return edge_backward(e, stats, g, g_stride, 1.0, 0, static_cast<cudaStream_t>(stream));
}

}  // extern "C"
