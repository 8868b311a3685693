// PoU pinhole warp on a separable lattice and its adjoint, sm_100a.
//
// The pinhole lattice's rays agree per detector column (rx) and per detector
// row (ry) up to float rounding, so block b of pose n is sampled at image
// column (d_b rx[c] - cu) / ds + c0 by every pixel of detector column c and at
// image row (d_b ry[r] - cv) / ds + c0 by every pixel of row r: the bilinear
// warp is a 1-D interpolation along x followed by one along y, and its adjoint
// the two transposed ones in the other order.  Both kernels march down the
// detector rows with the column's image position in registers, so the
// position arithmetic (fp64), the column's two image loads and the x
// interpolation are paid once per image row instead of once per pixel.
#include "fvr_common.cuh"

namespace fvr {

struct SepArgs {
  const float* imgs;   // [B][N][P][P] block images
  const double* offs;  // [B][N][3]: d_b, cu, cv
  const float* rxc;    // [W] column ray coordinate
  const float* ryr;    // [Hd] row ray coordinate
  const float* ic;     // [Hd W] obliquity factor
  int B, N, P, Hd, W;
  double inv_ds, c_idx;
};

// Image position of a ray coordinate on a block axis: cell index clamped to
// [-2, P] (below -1 and from P on the sample misses the image) and fraction.
__device__ __forceinline__ int sep_cell(double scale, double off, float ray, int P, float& t) {
  const double p = fma(scale, static_cast<double>(ray), off);
  t = 0.f;
  if (!(p > -1.0)) return -2;  // NaN counts as a miss
  if (!(p < static_cast<double>(P))) return P;
  const double f = floor(p);
  t = static_cast<float>(p - f);
  return static_cast<int>(f);
}

// ----------------------------------------------------------------------------
// forward
// ----------------------------------------------------------------------------

constexpr int kSepCols = 4;       // detector columns per thread
constexpr int kSepBlocks = 32;    // blocks per round of the row table
constexpr int kSepRingRows = 36;  // image rows of the slab ring
constexpr int kSepStages = 4;     // slabs in the ring at most

__device__ __forceinline__ void cp_async16(float* dst, const float* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ float2 sub2(float2 x, float2 y) { return __ffma2_rn(y, make_float2(-1.f, -1.f), x); }
__device__ __forceinline__ float2 bcast(float x) { return make_float2(x, x); }

// out[n][r][c] = ic sum_b bilinear(imgs[b][n]).  A CTA owns RG detector rows x
// 4 columns per thread of one pose and runs over the blocks that touch its
// rows.  The image rows those detector rows sample are one contiguous piece of
// the block image, copied to shared memory up to three blocks ahead (read on
// demand, every image row cost a trip to memory: 567 us).  Per block a lane
// interpolates each image row at its columns once, blends neighbouring rows
// per detector row, and does both in f32x2 pairs.
// More rows reuse an image row more often, fewer leave more CTAs (the rule is
// at the launch).  Bound by dependent issue at 14 warps per SM.  64 blocks x 64
// poses x 256^2 pixels: 207 us, and 394 us for a kernel with one thread per
// pixel and the row pairs blended in shared memory; 8 blocks x 64 poses x
// 512^2 pixels: 95 and 429 us.
template <int RG>
__global__ void __launch_bounds__(128) pou_warp_sep_kernel(SepArgs a, int tiles, float* __restrict__ out) {
  constexpr int NC = kSepCols;
  extern __shared__ __align__(16) float ring[];  // [kSepRingRows * P]
  __shared__ int2 rows[kSepBlocks][RG];          // (iy, ty) of the band's detector rows per block
  __shared__ int list[kSepBlocks], first[kSepBlocks], count[kSepBlocks];  // live blocks and their image rows
  __shared__ double2 xmap[kSepBlocks];  // image column of a ray: xmap.x rx + xmap.y
  __shared__ int n_live, slot_rows;
  const int T = blockDim.x, n = blockIdx.y;
  const int band = blockIdx.x / tiles, tile = blockIdx.x - band * tiles;
  const int P = a.P, r0 = band * RG, c0 = tile * T * NC + threadIdx.x;
  const bool aligned = (P & 3) == 0 && (reinterpret_cast<uintptr_t>(a.imgs) & 15) == 0;
  float rx[NC];
#pragma unroll
  for (int j = 0; j < NC; ++j) rx[j] = c0 + T * j < a.W ? __ldg(a.rxc + c0 + T * j) : 0.f;
  float2 acc[RG][NC / 2];
#pragma unroll
  for (int r = 0; r < RG; ++r)
#pragma unroll
    for (int h = 0; h < NC / 2; ++h) acc[r][h] = bcast(0.f);
  for (int b0 = 0; b0 < a.B; b0 += kSepBlocks) {
    const int nb = min(kSepBlocks, a.B - b0);
    __syncthreads();  // the previous round's tables and slabs are no longer read
    for (int e = threadIdx.x; e < nb * RG; e += T) {
      const int k = e / RG, r = e - k * RG;
      const double* o = a.offs + 3 * (static_cast<int64_t>(b0 + k) * a.N + n);
      float t = 0.f;
      const int iy = r0 + r < a.Hd ? sep_cell(o[0] * a.inv_ds, a.c_idx - o[2] * a.inv_ds, __ldg(a.ryr + r0 + r), P, t)
                                   : -2;
      rows[k][r] = make_int2(iy >= P ? -2 : iy, __float_as_int(t));
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // blocks in increasing order, with the image rows they need
      const int k = threadIdx.x;
      int lo = 0x7fffffff, hi = -1;
      if (k < nb) {
        const double* o = a.offs + 3 * (static_cast<int64_t>(b0 + k) * a.N + n);
        xmap[k] = make_double2(o[0] * a.inv_ds, a.c_idx - o[1] * a.inv_ds);
      }
      if (k < nb)
        for (int r = 0; r < RG; ++r) {
          const int iy = rows[k][r].x;
          if (iy >= -1) {
            lo = min(lo, max(iy, 0));
            hi = max(hi, min(iy + 1, P - 1));
          }
        }
      const unsigned m = __ballot_sync(0xffffffffu, hi >= 0);
      const int need = hi >= 0 ? hi - lo + 1 : 0;
      const bool fits = aligned && need <= kSepRingRows;
      if (hi >= 0) {
        const int i = __popc(m & ((1u << k) - 1u));
        list[i] = k;
        first[i] = lo;
        count[i] = fits ? need : 0;  // 0: read from memory
      }
      const int most = __reduce_max_sync(0xffffffffu, fits ? need : 0);
      if (k == 0) {
        n_live = __popc(m);
        slot_rows = max(most, 1);
      }
    }
    __syncthreads();
    const int live = n_live, slot = slot_rows * P, stages = min(kSepStages, kSepRingRows / slot_rows);
    auto fetch = [&](int i) {
      if (i < live) {
        const int q = count[i] * (P >> 2);
        const float* src = a.imgs + (static_cast<int64_t>(b0 + list[i]) * a.N + n) * P * P + first[i] * P;
        float* dst = ring + (i % stages) * slot;
        for (int e = threadIdx.x; e < q; e += T) cp_async16(dst + 4 * e, src + 4 * e);
      }
      cp_async_commit();
    };
    for (int i = 0; i < stages - 1; ++i) fetch(i);
    for (int i = 0; i < live; ++i) {
      const double2 xm = xmap[list[i]];
      int ix[NC];
      float tj[NC];
      bool in0[NC], in1[NC];
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        ix[j] = sep_cell(xm.x, xm.y, rx[j], P, tj[j]);
        in0[j] = ix[j] >= 0 && ix[j] < P;
        in1[j] = ix[j] >= -1 && ix[j] + 1 < P;
      }
      // slab i has landed for every thread, and slab i - 1 is no longer read
      if (stages == 1) {
        __syncthreads();
        fetch(i);
        cp_async_wait<0>();
        __syncthreads();
      } else {
        if (stages == 2) cp_async_wait<0>();
        else if (stages == 3) cp_async_wait<1>();
        else cp_async_wait<2>();
        __syncthreads();
        fetch(i + stages - 1);
      }
      int cur = -3;                         // the march is in image cell `cur`
      float2 lo[NC / 2], hi[NC / 2], dv[NC / 2];  // x-interpolated rows cur and cur + 1, their difference
      auto march = [&](auto row) {
#pragma unroll
        for (int r = 0; r < RG; ++r) {
          const int2 e = rows[list[i]][r];
          if (e.x < -1) continue;
          if (e.x != cur) {
            if (e.x == cur + 1) {
#pragma unroll
              for (int h = 0; h < NC / 2; ++h) lo[h] = hi[h];
            } else {
              row(e.x, lo);
            }
            row(e.x + 1, hi);
#pragma unroll
            for (int h = 0; h < NC / 2; ++h) dv[h] = sub2(hi[h], lo[h]);
            cur = e.x;
          }
          const float2 ty = bcast(__int_as_float(e.y));
#pragma unroll
          for (int h = 0; h < NC / 2; ++h) acc[r][h] = __ffma2_rn(ty, dv[h], __fadd2_rn(acc[r][h], lo[h]));
        }
      };
      float v0[NC], v1[NC];  // columns outside the image keep their zeros
#pragma unroll
      for (int j = 0; j < NC; ++j) v0[j] = v1[j] = 0.f;
      auto interpolate = [&](const float* q, float2 (&v)[NC / 2]) {
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          if (in0[j] && fvr_checked(ix[j], P, kSiteWarpTap)) v0[j] = q[ix[j]];
          if (in1[j] && fvr_checked(ix[j] + 1, P, kSiteWarpTap)) v1[j] = q[ix[j] + 1];
        }
#pragma unroll
        for (int h = 0; h < NC / 2; ++h) {
          const float2 u0 = make_float2(v0[2 * h], v0[2 * h + 1]), u1 = make_float2(v1[2 * h], v1[2 * h + 1]);
          v[h] = __ffma2_rn(make_float2(tj[2 * h], tj[2 * h + 1]), sub2(u1, u0), u0);
        }
      };
      auto clear = [&](float2 (&v)[NC / 2]) {
#pragma unroll
        for (int h = 0; h < NC / 2; ++h) v[h] = bcast(0.f);
      };
      if (count[i] > 0) {
        const float* base = ring + (i % stages) * slot - first[i] * P;
        march([&](int y, float2 (&v)[NC / 2]) {
          if (y >= 0 && y < P) interpolate(base + y * P, v);
          else clear(v);
        });
      } else {
        const float* img = a.imgs + (static_cast<int64_t>(b0 + list[i]) * a.N + n) * P * P;
        march([&](int y, float2 (&v)[NC / 2]) {
          if (y >= 0 && y < P) interpolate(img + static_cast<int64_t>(y) * P, v);
          else clear(v);
        });
      }
    }
    cp_async_wait<0>();
  }
#pragma unroll
  for (int r = 0; r < RG; ++r) {
    if (r0 + r < a.Hd) {
      const int64_t q = static_cast<int64_t>(r0 + r) * a.W;
      const float v[NC] = {acc[r][0].x, acc[r][0].y, acc[r][1].x, acc[r][1].y};
#pragma unroll
      for (int j = 0; j < NC; ++j) {
        const int c = c0 + T * j;
        if (c < a.W) out[static_cast<int64_t>(n) * a.Hd * a.W + q + c] = v[j] * __ldg(a.ic + q + c);
      }
    }
  }
}

// The same for few poses, where the marching kernel's serial chain over the
// blocks shows (1 pose, 8 blocks, 256^2 pixels: 10.4 us): a CTA owns 4 rows x
// 32 columns, its 8 warps take every eighth block each and their sums meet in
// shared memory.  All taps of a block are independent loads.
constexpr int kSepFewRows = 4, kSepFewWarps = 8;

__global__ void __launch_bounds__(32 * kSepFewWarps) pou_warp_sep_few_kernel(SepArgs a, int tiles,
                                                                             float* __restrict__ out) {
  constexpr int RG = kSepFewRows;
  __shared__ float part[kSepFewWarps][RG][32];
  const int n = blockIdx.y, P = a.P, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int band = blockIdx.x / tiles, r0 = band * RG, c = (blockIdx.x - band * tiles) * 32 + lane;
  const float rx = c < a.W ? __ldg(a.rxc + c) : 0.f;
  const float ry = lane < RG && r0 + lane < a.Hd ? __ldg(a.ryr + r0 + lane) : 0.f;
  float acc[RG];
#pragma unroll
  for (int r = 0; r < RG; ++r) acc[r] = 0.f;
  for (int b = wid; b < a.B; b += kSepFewWarps) {
    const int64_t bn = static_cast<int64_t>(b) * a.N + n;
    const double* o = a.offs + 3 * bn;
    const double sc = __ldg(o) * a.inv_ds;
    float tx, ty;
    const int ix = sep_cell(sc, a.c_idx - __ldg(o + 1) * a.inv_ds, rx, P, tx);
    int iy = sep_cell(sc, a.c_idx - __ldg(o + 2) * a.inv_ds, ry, P, ty);  // lane r: detector row r
    if (lane >= RG || r0 + lane >= a.Hd) iy = -2;
    const float* img = a.imgs + bn * P * P;
    const bool x0 = ix >= 0 && ix < P, x1 = ix >= -1 && ix + 1 < P;
    float v[RG][4], t[RG];
#pragma unroll
    for (int r = 0; r < RG; ++r) {
      const int y = __shfl_sync(0xffffffffu, iy, r);
      t[r] = __shfl_sync(0xffffffffu, ty, r);
      const bool y0 = y >= 0 && y < P, y1 = y >= -1 && y + 1 < P;
      v[r][0] = x0 && y0 ? ldg_in(img, y * P + ix, P * P, kSiteWarpTap) : 0.f;
      v[r][1] = x1 && y0 ? ldg_in(img, y * P + ix + 1, P * P, kSiteWarpTap) : 0.f;
      v[r][2] = x0 && y1 ? ldg_in(img, (y + 1) * P + ix, P * P, kSiteWarpTap) : 0.f;
      v[r][3] = x1 && y1 ? ldg_in(img, (y + 1) * P + ix + 1, P * P, kSiteWarpTap) : 0.f;
    }
#pragma unroll
    for (int r = 0; r < RG; ++r) {
      const float lo = fmaf(tx, v[r][1] - v[r][0], v[r][0]), hi = fmaf(tx, v[r][3] - v[r][2], v[r][2]);
      acc[r] += fmaf(t[r], hi - lo, lo);
    }
  }
#pragma unroll
  for (int r = 0; r < RG; ++r) part[wid][r][lane] = acc[r];
  __syncthreads();
  if (wid < RG && r0 + wid < a.Hd && c < a.W) {
    float s = 0.f;
    for (int k = 0; k < kSepFewWarps; ++k) s += part[k][wid][lane];
    const int64_t q = static_cast<int64_t>(r0 + wid) * a.W + c;
    out[static_cast<int64_t>(n) * a.Hd * a.W + q] = s * __ldg(a.ic + q);
  }
}

// ----------------------------------------------------------------------------
// adjoint
// ----------------------------------------------------------------------------

constexpr int kSepBand = 8;      // image rows of a unit at most
constexpr int kSepPass = 128;    // detector columns of a march, four per lane
constexpr int kSepWide = 256;    // detector columns of a warp's G buffer

// Dynamic shared memory: column map (ix, tx) [Wp] (W rounded up to four), row fractions [Hd], first
// table position at or beyond each image index [P + 3] for columns and rows,
// the warps' G buffers.
__host__ __device__ constexpr int sep_padded(int W) { return (W + 3) / 4 * 4; }
__host__ __device__ constexpr int64_t sep_adj_gbuf_at(int P, int Hd, int W) {
  return (8LL * sep_padded(W) + 4LL * Hd + 8LL * (P + 3) + 15) / 16 * 16;
}
__host__ __device__ constexpr int64_t sep_adj_smem(int P, int Hd, int W, int warps) {
  return sep_adj_gbuf_at(P, Hd, W) + 4LL * warps * kSepBand * kSepWide;
}

struct SepGrad {
  const float* gout;  // [N][Hd W]
  const float4* gic;  // [N][Hd][Wp / 4]: gout ic, rows padded with zeros
  float* gimgs;       // [B][N][P][P]
  double* goffs;      // [3][B][N]: dL/d(d_b, cu, cv)
};

// first[i + 1] = first k with cell(k) >= i, for i = -1 .. P + 1; cells are
// non-decreasing in k.
template <typename F>
__device__ __forceinline__ void sep_first(int* first, int count, int P, F cell) {
  for (int k = threadIdx.x; k <= count; k += blockDim.x) {
    const int prev = k == 0 ? -2 : cell(k - 1), here = k == count ? P + 1 : cell(k);
    for (int i = prev + 1; i <= here; ++i)
      if (i >= -1) first[i + 1] = k;
  }
}

// gic[n][r][c] = g[n][r][c] ic[r][c] with the rows padded by zeros to a
// multiple of four columns: the adjoint reads every detector row once per
// block, as aligned 16-byte words whatever the detector's width.
__global__ void __launch_bounds__(256) pou_warp_sep_weigh_kernel(const float* __restrict__ g,
                                                                 const float* __restrict__ ic, int Hd, int W, int Wp,
                                                                 bool vec, float4* __restrict__ gic) {
  const int quads = Hd * (Wp / 4), q = blockIdx.x * 256 + threadIdx.x;
  if (q >= quads) return;
  const int row = q / (Wp / 4), c = 4 * (q - row * (Wp / 4));
  const float *gp = g + (static_cast<int64_t>(blockIdx.y) * Hd + row) * W + c, *ip = ic + static_cast<int64_t>(row) * W + c;
  float4 v;
  if (vec) {  // W a multiple of four, 16-byte aligned inputs
    const float4 a = __ldg(reinterpret_cast<const float4*>(gp)), b = __ldg(reinterpret_cast<const float4*>(ip));
    v = make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w);
  } else {
    v.x = __ldg(gp) * __ldg(ip);
    v.y = c + 1 < W ? __ldg(gp + 1) * __ldg(ip + 1) : 0.f;
    v.z = c + 2 < W ? __ldg(gp + 2) * __ldg(ip + 2) : 0.f;
    v.w = c + 3 < W ? __ldg(gp + 3) * __ldg(ip + 3) : 0.f;
  }
  gic[static_cast<int64_t>(blockIdx.y) * quads + q] = v;
}

// One CTA per (pose, block).  Its units are bands of image rows (those the
// detector reaches, split evenly over the warps) x groups of image columns
// whose detector columns fit a G buffer; a warp takes a unit and writes
// dL/dimgs there, every element once (nothing to clear, no atomics):
//   march down the detector rows of cell y0 - 1, y0, .. for 128 detector
//   columns at a time, four neighbours per lane in f32x2 pairs, keeping the cell's sums
//   A0 = sum g ic and A1 = sum ty g ic; leaving cell y gives G[y][c] =
//   (A0 - A1)(y) + A1(y - 1) and, with the image row's value and slope at the
//   column, the pose-offset sums;
//   then lane x gathers G[y][c] over its detector columns, weight 1 - |px(c) - x|.
// The sum of g ry dv/dpy comes from ry = (y + ty - oy) / scale: per cell
// (y - oy) A0 + A1, so no third sum is kept while marching.
// Bound by issue at 16 warps per SM (50 % issue active; three CTAs per SM
// spill: 974 us).  64 blocks x 64 poses x 256^2 pixels: 495 us, with the
// separate slice adjoint 1232 us against 1422 us for a gather along x of every
// detector row inside the slice-adjoint kernel; 8 blocks x 64 poses x 512^2
// pixels: 265 us against 1104 us for a scatter with atomics.
template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB) pou_warp_sep_adjoint_kernel(SepArgs a, SepGrad w) {
  constexpr int NW = THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[4][NW];
  // per thread: sums of g dv/dpx, g rx dv/dpx, g dv/dpy, g (y + ty - oy) dv/dpy (no registers held while marching)
  __shared__ double sums[4][THREADS];
  const int P = a.P, Hd = a.Hd, W = a.W, Wp = sep_padded(W);
  int2* cmap = reinterpret_cast<int2*>(smem);             // (ix, tx) per detector column, -2 in the padding
  float* rty = reinterpret_cast<float*>(cmap + Wp);       // ty per detector row, in march order
  int* cfirst = reinterpret_cast<int*>(rty + Hd);
  int* rfirst = cfirst + (P + 3);
  const int n = blockIdx.x, b = blockIdx.y;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t bn = static_cast<int64_t>(b) * a.N + n;
  const double* o = a.offs + 3 * bn;
  const double sc = o[0] * a.inv_ds, ox = a.c_idx - o[1] * a.inv_ds, oy = a.c_idx - o[2] * a.inv_ds;
  // march order: increasing image position
  const bool rev_c = sc * (static_cast<double>(__ldg(a.rxc + W - 1)) - static_cast<double>(__ldg(a.rxc))) < 0.0;
  const bool rev_r = sc * (static_cast<double>(__ldg(a.ryr + Hd - 1)) - static_cast<double>(__ldg(a.ryr))) < 0.0;
  int* rcell = reinterpret_cast<int*>(smem + sep_adj_gbuf_at(P, Hd, W));  // in the G buffers until they are used
#pragma unroll
  for (int k = 0; k < 4; ++k) sums[k][threadIdx.x] = 0.0;
  for (int c = threadIdx.x; c < Wp; c += THREADS) {
    float t = 0.f;
    const int i = c < W ? sep_cell(sc, ox, __ldg(a.rxc + c), P, t) : -2;
    cmap[c] = make_int2(i, __float_as_int(t));
  }
  for (int k = threadIdx.x; k < Hd; k += THREADS) rcell[k] = sep_cell(sc, oy, __ldg(a.ryr + (rev_r ? Hd - 1 - k : k)), P, rty[k]);
  __syncthreads();
  sep_first(cfirst, W, P, [&](int k) { return cmap[rev_c ? W - 1 - k : k].x; });
  sep_first(rfirst, Hd, P, [&](int k) { return rcell[k]; });
  __syncthreads();
  // detector columns whose cell lies in [i0, i1), as a range of c
  auto columns = [&](int i0, int i1, int& c0, int& c1) {
    const int f0 = cfirst[i0 + 1], f1 = cfirst[i1 + 1];
    c0 = rev_c ? W - f1 : f0;
    c1 = rev_c ? W - f0 : f1;
  };
  const float* img = a.imgs + bn * P * P;
  float* gimg = w.gimgs + bn * P * P;
  const float* gout = w.gout + static_cast<int64_t>(n) * Hd * W;
  // image rows that any detector row reaches: cells -1 .. P - 1 give rows cell, cell + 1
  int ya = P, yb = P;
  if (rfirst[0] < rfirst[P + 1]) {
    int lo = 0, hi = P;  // first row y with a detector row in cell y - 1 or y
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (rfirst[mid + 2] > rfirst[0]) hi = mid;
      else lo = mid + 1;
    }
    ya = lo;
    hi = P;  // first row y >= ya with no detector row in any cell >= y - 1
    while (lo < hi) {
      const int mid = (lo + hi) / 2;
      if (rfirst[mid] >= rfirst[P + 1]) hi = mid;
      else lo = mid + 1;
    }
    yb = lo;
  }
  for (int q = threadIdx.x; q < ya * P; q += THREADS) gimg[q] = 0.f;
  for (int q = yb * P + threadIdx.x; q < P * P; q += THREADS) gimg[q] = 0.f;
  // as many 32-column groups per unit as the G buffer takes
  const int groups = (P + 31) / 32;
  int gs = groups;
  for (; gs > 1; --gs) {
    bool fits = true;
    for (int g = 0; g < groups; g += gs) {
      int c0, c1;
      columns(32 * g - 1, min(P, 32 * (g + gs)), c0, c1);
      fits &= c1 - (c0 & ~3) <= kSepWide;
    }
    if (fits) break;
  }
  const int supers = (groups + gs - 1) / gs;
  const int nbands = yb > ya ? ((yb - ya + kSepBand - 1) / kSepBand + NW - 1) / NW * NW : 0;
  float* G = reinterpret_cast<float*>(smem + sep_adj_gbuf_at(P, Hd, W)) + wid * kSepBand * kSepWide;
  for (int u = wid; u < nbands * supers; u += NW) {
    const int sg = u / nbands, band = u - sg * nbands;
    const int y0 = ya + static_cast<int>(static_cast<int64_t>(band) * (yb - ya) / nbands);
    const int y1 = ya + static_cast<int>(static_cast<int64_t>(band + 1) * (yb - ya) / nbands);
    if (y0 >= y1) continue;
    const int x0 = 32 * gs * sg, x1 = min(P, x0 + 32 * gs);
    const int kr0 = rfirst[y0], kr1 = rfirst[y1 + 1];  // cells y0 - 1 .. y1 - 1
    int ca, cb;
    columns(x0 - 1, x1, ca, cb);
    float2 gsum[kSepBand / 2];  // rows 2 i, 2 i + 1
#pragma unroll
    for (int i = 0; i < kSepBand / 2; ++i) gsum[i] = bcast(0.f);
    if (ca >= cb || kr0 >= kr1) {  // nothing reaches this unit
      for (int x = x0 + lane; x < x1; x += 32)
        for (int y = y0; y < y1; ++y) gimg[y * P + x] = 0.f;
      continue;
    }
    const int cs = ca & ~3;  // 16-byte words of a detector row
    for (int kp = cs; kp < cb; kp += kSepWide) {  // several only for a single 32-column group
      const int ke = min(cb, kp + kSepWide);
      for (int sp = kp; sp < ke; sp += kSepPass) {
        const int c = sp + 4 * lane;
        const bool on = c < Wp;
        float2 tx[2], A0[2], A1[2], p0[2], p1[2], Lp[2], sx[2], v0[2], v1[2], fy[2], f1[2];
        int ix[4];
        bool in0[4], in1[4];  // image values ix, ix + 1 belong to the sums
        float tj[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int2 e = on ? cmap[c + j] : make_int2(-2, 0);
          // a column's sums belong to the unit that holds image column max(ix, 0)
          const bool own = c + j >= ca && c + j < ke && e.x >= -1 && max(e.x, 0) >= x0 && e.x < x1;
          ix[j] = e.x;
          tj[j] = __int_as_float(e.y);
          in0[j] = own && e.x >= 0;
          in1[j] = own && e.x + 1 < P;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          tx[h] = make_float2(tj[2 * h], tj[2 * h + 1]);
          A0[h] = A1[h] = p0[h] = p1[h] = Lp[h] = sx[h] = v0[h] = v1[h] = fy[h] = f1[h] = bcast(0.f);
        }
        auto load_image = [&](int y) {  // lanes outside keep their zeros
          const float* q = img + y * P;
          if (in0[0]) v0[0].x = ldg_in(q, ix[0], P, kSiteWarpTap);
          if (in0[1]) v0[0].y = ldg_in(q, ix[1], P, kSiteWarpTap);
          if (in0[2]) v0[1].x = ldg_in(q, ix[2], P, kSiteWarpTap);
          if (in0[3]) v0[1].y = ldg_in(q, ix[3], P, kSiteWarpTap);
          if (in1[0]) v1[0].x = ldg_in(q, ix[0] + 1, P, kSiteWarpTap);
          if (in1[1]) v1[0].y = ldg_in(q, ix[1] + 1, P, kSiteWarpTap);
          if (in1[2]) v1[1].x = ldg_in(q, ix[2] + 1, P, kSiteWarpTap);
          if (in1[3]) v1[1].y = ldg_in(q, ix[3] + 1, P, kSiteWarpTap);
        };
        const int step = rev_r ? -(Wp / 4) : Wp / 4;
        const float4* gq = w.gic + (static_cast<int64_t>(n) * Hd + (rev_r ? Hd - 1 - kr0 : kr0)) * (Wp / 4) + c / 4;
        float4 gn = make_float4(0.f, 0.f, 0.f, 0.f), gm = gn;  // the next two detector rows' values
        int kr = kr0;
        if (on) gn = __ldg(gq);
        gq += step;
        if (on && kr + 1 < kr1) gm = __ldg(gq);
        auto cell = [&](int kend) {
#pragma unroll
          for (int h = 0; h < 2; ++h) A0[h] = A1[h] = bcast(0.f);
          for (; kr < kend; ++kr) {
            const float2 ty = bcast(rty[kr]);
            const float2 g0 = make_float2(gn.x, gn.y), g1 = make_float2(gn.z, gn.w);
            gn = gm;
            gq += step;
            if (on && kr + 2 < kr1) gm = __ldg(gq);
            A0[0] = __fadd2_rn(A0[0], g0);
            A0[1] = __fadd2_rn(A0[1], g1);
            A1[0] = __ffma2_rn(ty, g0, A1[0]);
            A1[1] = __ffma2_rn(ty, g1, A1[1]);
          }
        };
        if (y0 > 0) {
          load_image(y0 - 1);
#pragma unroll
          for (int h = 0; h < 2; ++h) Lp[h] = __ffma2_rn(tx[h], sub2(v1[h], v0[h]), v0[h]);
        }
        cell(rfirst[y0 + 1]);
        for (int y = y0; y < y1; ++y) {
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            p0[h] = A0[h];
            p1[h] = A1[h];
          }
          load_image(y);
          cell(rfirst[y + 2]);
          const float2 yo = bcast(static_cast<float>(static_cast<double>(y - 1) - oy));
          float2 g[2];
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            g[h] = __fadd2_rn(sub2(A0[h], A1[h]), p1[h]);
            const float2 d = sub2(v1[h], v0[h]);
            const float2 L = __ffma2_rn(tx[h], d, v0[h]), D = sub2(L, Lp[h]);
            Lp[h] = L;
            sx[h] = __ffma2_rn(g[h], d, sx[h]);
            fy[h] = __ffma2_rn(p0[h], D, fy[h]);  // cell y - 1
            f1[h] = __ffma2_rn(__ffma2_rn(yo, p0[h], p1[h]), D, f1[h]);
          }
          *reinterpret_cast<float4*>(G + (y - y0) * kSepWide + (c - kp)) = make_float4(g[0].x, g[0].y, g[1].x, g[1].y);
        }
        if (y1 == P) {  // the last cell's lower row lies outside the image
          const float2 yo = bcast(static_cast<float>(static_cast<double>(P - 1) - oy));
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            const float2 D = sub2(bcast(0.f), Lp[h]);
            fy[h] = __ffma2_rn(A0[h], D, fy[h]);
            f1[h] = __ffma2_rn(__ffma2_rn(yo, A0[h], A1[h]), D, f1[h]);
          }
        }
        const float sj[4] = {sx[0].x, sx[0].y, sx[1].x, sx[1].y};
        float dx = 0.f, drx = 0.f;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (in0[j] || in1[j]) {
            dx += sj[j];
            drx = fmaf(sj[j], __ldg(a.rxc + c + j), drx);
          }
        sums[0][threadIdx.x] += static_cast<double>(dx);
        sums[1][threadIdx.x] += static_cast<double>(drx);
        sums[2][threadIdx.x] += static_cast<double>((fy[0].x + fy[0].y) + (fy[1].x + fy[1].y));
        sums[3][threadIdx.x] += static_cast<double>((f1[0].x + f1[0].y) + (f1[1].x + f1[1].y));
      }
      __syncwarp();
      for (int xg = x0; xg < x1; xg += 32) {
        const int x = xg + lane;
        if (kp == cs)
#pragma unroll
          for (int i = 0; i < kSepBand / 2; ++i) gsum[i] = bcast(0.f);
        int t0 = 0, t1 = 0;
        if (x < x1) columns(x - 1, x + 1, t0, t1);
        t1 = min(t1, ke);
        for (int k = max(t0, kp); k < t1; ++k) {
          const int2 e = cmap[k];
          const float t = __int_as_float(e.y);
          const float2 wt = bcast(e.x == x ? 1.f - t : t);
          const float* q = G + (k - kp);
#pragma unroll
          for (int i = 0; i < kSepBand / 2; ++i)
            if (fvr_checked((2 * i + 1) * kSepWide + k - kp, kSepBand * kSepWide, kSiteWarpFused))
              gsum[i] = __ffma2_rn(wt, make_float2(q[2 * i * kSepWide], q[(2 * i + 1) * kSepWide]), gsum[i]);
        }
        if (ke == cb && x < x1) {
#pragma unroll
          for (int i = 0; i < kSepBand / 2; ++i) {
            if (y0 + 2 * i < y1) gimg[(y0 + 2 * i) * P + x] = gsum[i].x;
            if (y0 + 2 * i + 1 < y1) gimg[(y0 + 2 * i + 1) * P + x] = gsum[i].y;
          }
        }
      }
      __syncwarp();
    }
  }
  // a block in the source plane (scale near 0) does not determine ry from the image row: sum g ry dv/dpy directly
  const bool direct = fabs(sc) < 1.0;
  double s_ry = sums[3][threadIdx.x];
  if (direct) {
    s_ry = 0.0;
    for (int64_t q = threadIdx.x; q < static_cast<int64_t>(Hd) * W; q += THREADS) {
      const int r = static_cast<int>(q / W), c = static_cast<int>(q - static_cast<int64_t>(r) * W);
      const float ry = __ldg(a.ryr + r);
      float ty;
      const int iy = sep_cell(sc, oy, ry, P, ty), ix = cmap[c].x;
      if (iy < -1 || iy >= P || ix < -1 || ix >= P) continue;
      const float tx = __int_as_float(cmap[c].y);
      auto at = [&](int y, int x) { return y >= 0 && y < P && x >= 0 && x < P ? __ldg(img + y * P + x) : 0.f; };
      const float D = (1.f - tx) * (at(iy + 1, ix) - at(iy, ix)) + tx * (at(iy + 1, ix + 1) - at(iy, ix + 1));
      s_ry += static_cast<double>(__ldg(gout + q) * __ldg(a.ic + q)) * static_cast<double>(ry) * static_cast<double>(D);
    }
  }
  const double mine[4] = {sums[0][threadIdx.x], sums[1][threadIdx.x], sums[2][threadIdx.x], s_ry};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    const double t = warp_sum(mine[k]);
    if (lane == 0) red[k][wid] = t;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double t[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k = 0; k < 4; ++k)
      for (int v = 0; v < NW; ++v) t[k] += red[k][v];
    const int64_t BN = static_cast<int64_t>(a.B) * a.N;
    w.goffs[bn] = a.inv_ds * (t[1] + (direct ? t[3] : t[3] / sc));
    w.goffs[BN + bn] = -a.inv_ds * t[0];
    w.goffs[2 * BN + bn] = -a.inv_ds * t[2];
  }
}

static int sep_args(const float* imgs, int64_t B, int64_t N, int64_t P, const double* offs, const float* rxc,
                    const float* ryr, const float* ic, int64_t H, int64_t W, double inv_ds, double c_idx, SepArgs* a) {
  if (!imgs || !offs || !rxc || !ryr || !ic || B < 1 || N < 1 || N > 65535 || B > 4096) return FVR_ERR_ARG;
  if (!fvr_pou_warp_sep_supported(P, H, W)) return FVR_ERR_UNSUPPORTED;
  *a = SepArgs{imgs, offs, rxc, ryr, ic, (int)B, (int)N, (int)P, (int)H, (int)W, inv_ds, c_idx};
  return FVR_OK;
}

template <int THREADS, int MINB>
static int sep_adjoint(const SepArgs& a, const SepGrad& w, cudaStream_t s) {
  const int64_t smem = sep_adj_smem(a.P, a.Hd, a.W, THREADS / 32);
  // the shared-memory opt-in is a per-device setting: made before every launch
  if (cudaFuncSetAttribute(pou_warp_sep_adjoint_kernel<THREADS, MINB>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(smem)) != cudaSuccess)
    return FVR_ERR_CUDA;
  pou_warp_sep_adjoint_kernel<THREADS, MINB>
      <<<dim3(static_cast<unsigned>(a.N), static_cast<unsigned>(a.B)), THREADS, smem, s>>>(a, w);
  FVR_LAUNCH_CHECK();
  return FVR_OK;
}

template <int RG>
static int sep_forward(const SepArgs& a, float* out, cudaStream_t s) {
  const int64_t smem = 4LL * kSepRingRows * a.P;
  if (smem > 48 * 1024 &&
      cudaFuncSetAttribute(pou_warp_sep_kernel<RG>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(smem)) != cudaSuccess)
    return FVR_ERR_CUDA;
  const int64_t warps = cdiv64(a.W, 32 * kSepCols), tiles = cdiv64(warps, 4), per = cdiv64(warps, tiles);
  const dim3 grid(static_cast<unsigned>(tiles * cdiv64(a.Hd, RG)), static_cast<unsigned>(a.N));
  pou_warp_sep_kernel<RG><<<grid, static_cast<unsigned>(32 * per), smem, s>>>(a, static_cast<int>(tiles), out);
  FVR_LAUNCH_CHECK();
  return FVR_OK;
}

}  // namespace fvr

using namespace fvr;

extern "C" {

int fvr_pou_warp_sep_supported(int64_t P, int64_t H, int64_t W) {
  return P >= 2 && P <= 512 && H >= 1 && W >= 1 && H <= 65535 && W <= 65535 ? 1 : 0;
}

int fvr_pou_warp_sep(const float* imgs, int64_t B, int64_t N, int64_t P, const double* offs, const float* rxc,
                     const float* ryr, const float* ic, int64_t H, int64_t W, double inv_ds, double c_idx, float* out,
                     void* stream) {
  SepArgs a;
  const int rc = sep_args(imgs, B, N, P, offs, rxc, ryr, ic, H, W, inv_ds, c_idx, &a);
  if (rc) return rc;
  if (!out) return FVR_ERR_ARG;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // rows per CTA by the CTAs that leaves (8 against 16 rows: 217 / 207 us at 1024 CTAs of 16 rows, 30 / 45 us at
  // 336); below two CTAs per SM the blocks are split over warps
  const int64_t tiles = N * cdiv64(W, 512);
  if (tiles * cdiv64(H, 16) >= 888) return sep_forward<16>(a, out, s);
  if (tiles * cdiv64(H, 8) >= 296) return sep_forward<8>(a, out, s);
  const int xt = static_cast<int>(cdiv64(W, 32));
  pou_warp_sep_few_kernel<<<dim3(static_cast<unsigned>(xt * cdiv64(H, kSepFewRows)), static_cast<unsigned>(N)),
                            32 * kSepFewWarps, 0, s>>>(a, xt, out);
  FVR_LAUNCH_CHECK();
  return FVR_OK;
}

int fvr_pou_warp_sep_adjoint_supported(int64_t P, int64_t H, int64_t W) {
  if (!fvr_pou_warp_sep_supported(P, H, W)) return 0;
  // the row cells are staged in the G buffers; two 256-thread CTAs and one of 512 threads fit an SM
  return 4 * H <= 4LL * 8 * kSepBand * kSepWide && sep_adj_smem((int)P, (int)H, (int)W, 16) <= 200 * 1024 ? 1 : 0;
}

int64_t fvr_pou_warp_sep_adjoint_workspace(int64_t N, int64_t H, int64_t W) {
  return N < 1 || H < 1 || W < 1 ? 0 : 4 * N * H * ((W + 3) / 4 * 4);
}

int fvr_pou_warp_sep_adjoint(const float* imgs, int64_t B, int64_t N, int64_t P, const double* offs, const float* rxc,
                             const float* ryr, const float* ic, int64_t H, int64_t W, double inv_ds, double c_idx,
                             const float* gout, void* workspace, int64_t ws_bytes, float* grad_imgs, double* goffs,
                             void* stream) {
  SepArgs a;
  const int rc = sep_args(imgs, B, N, P, offs, rxc, ryr, ic, H, W, inv_ds, c_idx, &a);
  if (rc) return rc;
  if (!gout || !grad_imgs || !goffs || !workspace || (reinterpret_cast<uintptr_t>(workspace) & 15)) return FVR_ERR_ARG;
  if (ws_bytes < fvr_pou_warp_sep_adjoint_workspace(N, H, W)) return FVR_ERR_WORKSPACE;
  if (!fvr_pou_warp_sep_adjoint_supported(P, H, W)) return FVR_ERR_UNSUPPORTED;
  float4* gic = static_cast<float4*>(workspace);
  const SepGrad w{gout, gic, grad_imgs, goffs};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int Wp = sep_padded((int)W);
  const bool vec = W % 4 == 0 && ((reinterpret_cast<uintptr_t>(gout) | reinterpret_cast<uintptr_t>(ic)) & 15) == 0;
  pou_warp_sep_weigh_kernel<<<dim3((unsigned)cdiv64(H * (Wp / 4), 256), (unsigned)N), 256, 0, s>>>(
      gout, ic, (int)H, (int)W, Wp, vec, gic);
  FVR_LAUNCH_CHECK();
  // 256 threads once two CTAs per SM can run, else all 16 warps on one (pose, block)
  if (B * N >= 296) return sep_adjoint<256, 2>(a, w, s);
  return sep_adjoint<512, 1>(a, w, s);
}

int fvr_pou_pinhole_supported(int64_t P, int64_t H, int64_t W) {
  return fvr_pou_image_supported(P) && fvr_pou_warp_sep_supported(P, H, W);
}

int fvr_pou_pinhole_forward(int dtype, const void* stencil, const float* scales, int64_t B, int64_t P,
                            const float* mats, int64_t N, const double* base12, double vscale, const float* centers,
                            const float* freqs, const float* rxc, const float* ryr, const float* ic, int64_t H,
                            int64_t W, double inv_ds, double c_idx, double* geo, double* offs, float* imgs, float* out,
                            void* stream) {
  if (!mats || !out) return FVR_ERR_ARG;
  if (!fvr_pou_pinhole_supported(P, H, W)) return FVR_ERR_UNSUPPORTED;
  int rc = fvr_pou_pose(mats, nullptr, N, base12, vscale, centers, B, geo, offs, stream);
  if (!rc) rc = fvr_pou_slice_image(dtype, stencil, scales, B, P, geo, N, freqs, imgs, stream);
  if (!rc) rc = fvr_pou_warp_sep(imgs, B, N, P, offs, rxc, ryr, ic, H, W, inv_ds, c_idx, out, stream);
  return rc;
}

// Workspace of the backward: weighed detector gradient | offset gradients |
// slice-adjoint records, each on a 256-byte boundary.
static int64_t pinhole_round(int64_t bytes) { return (bytes + 255) / 256 * 256; }

int64_t fvr_pou_pinhole_backward_workspace(int64_t B, int64_t N, int64_t H, int64_t W) {
  if (B < 1 || N < 1) return 0;
  return pinhole_round(fvr_pou_warp_sep_adjoint_workspace(N, H, W)) + pinhole_round(24 * B * N) +
         fvr_pou_slice_image_adjoint_workspace(B, N);
}

int fvr_pou_pinhole_backward(int dtype, const void* stencil, const float* scales, int64_t B, int64_t P,
                             const double* geo, const double* offs, int64_t N, const double* base12, double vscale,
                             const float* centers, const float* freqs, const float* imgs, const float* rxc,
                             const float* ryr, const float* ic, int64_t H, int64_t W, double inv_ds, double c_idx,
                             const float* gout, float* grad_imgs, void* workspace, int64_t ws_bytes, float* gmats,
                             void* stream) {
  if (!workspace || !grad_imgs || (reinterpret_cast<uintptr_t>(workspace) & 15) || !gmats || !offs) return FVR_ERR_ARG;
  if (!fvr_pou_pinhole_supported(P, H, W) || !fvr_pou_warp_sep_adjoint_supported(P, H, W)) return FVR_ERR_UNSUPPORTED;
  if (ws_bytes < fvr_pou_pinhole_backward_workspace(B, N, H, W)) return FVR_ERR_WORKSPACE;
  const int64_t gic_bytes = fvr_pou_warp_sep_adjoint_workspace(N, H, W);
  const int64_t part_bytes = fvr_pou_slice_image_adjoint_workspace(B, N);
  char* w = static_cast<char*>(workspace);
  double* goffs = reinterpret_cast<double*>(w + pinhole_round(gic_bytes));
  double* part = reinterpret_cast<double*>(reinterpret_cast<char*>(goffs) + pinhole_round(24 * B * N));
  int rc = fvr_pou_warp_sep_adjoint(imgs, B, N, P, offs, rxc, ryr, ic, H, W, inv_ds, c_idx, gout, workspace, gic_bytes,
                                    grad_imgs, goffs, stream);
  if (!rc)
    rc = fvr_pou_slice_image_adjoint(dtype, stencil, scales, B, P, geo, N, freqs, grad_imgs, part, part_bytes, stream);
  if (!rc)
    rc = fvr_pou_pose_backward(part, 1, goffs, nullptr, 0, geo, centers, B, N, base12, vscale, gmats, nullptr, stream);
  return rc;
}

}  // extern "C"

FVR_CHECK_ACCESSOR(check_word_pou_sep)
