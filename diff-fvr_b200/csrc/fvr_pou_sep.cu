// PoU pinhole warp on a separable lattice and its adjoint, sm_100a.
//
// The pinhole lattice's rays agree per detector column (rx) and per detector
// row (ry) up to float rounding, so block b of pose n is sampled at image
// column (d_b rx[c] - cu) / ds + c0 by every pixel of detector column c and at
// image row (d_b ry[r] - cv) / ds + c0 by every pixel of row r: the bilinear
// warp is a 1-D interpolation along x followed by one along y, and its adjoint
// the two transposed ones in the other order.  The kernels march down the
// detector rows: forward, the position arithmetic (fp64), a column's two image
// loads and its x interpolation are paid once per image row instead of once per
// pixel; the adjoint reduces the pixels to four weighted sums per image cell,
// which is all that the image gradient and the pose offsets need of them.
#include <type_traits>

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
// poses x 256^2 pixels: 203 us, and 394 us for a kernel with one thread per
// pixel and the row pairs blended in shared memory; 8 blocks x 64 poses x
// 512^2 pixels: 94 and 429 us.
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

constexpr int kSepBand = 8;             // image rows of a gather unit
constexpr int kSepPairs = 5;            // pairs of cell rows it reads (the last is half used)
constexpr int kSepPass = 128;           // detector columns of a march, four per lane
constexpr int kSepStepCols = 512;        // detector columns of a step: 18 cell rows of 512 or 34 of 256
constexpr int kSepBufBytes = 8 * (2 * kSepBand + 2) * kSepStepCols;  // cell-row sums of a CTA, 72 KB
static_assert(8 * (4 * kSepBand + 2) * (kSepStepCols / 2) <= kSepBufBytes, "four bands of half rows");

// Dynamic shared memory: column map (ix, tx) [Wp] (W rounded up to four), row fractions [Hd], first
// table position at or beyond each image index [P + 3] for columns and rows,
// the buffer of cell-row sums.
__host__ __device__ constexpr int sep_padded(int W) { return (W + 3) / 4 * 4; }
__host__ __device__ constexpr int64_t sep_adj_gbuf_at(int P, int Hd, int W) {
  return (8LL * sep_padded(W) + 4LL * Hd + 8LL * (P + 3) + 15) / 16 * 16;
}
__host__ __device__ constexpr int64_t sep_adj_smem(int P, int Hd, int W) {
  return sep_adj_gbuf_at(P, Hd, W) + kSepBufBytes;
}

struct SepGrad {
  const float* gout;  // [N][Hd W]
  const float4* gic;  // [poses of this launch][Hd][Wp / 4]: gout ic, rows padded with zeros
  float* gimgs;       // [B][poses of this launch][P][P]
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

// One CTA per (pose, block) of a range of poses (the pointers are those of its
// first pose, a.N is the pose count of the whole arrays; WHOLE: the range is all
// of them, and one index serves both images, worth 10 us).  A detector pixel lies in one cell of the block
// image, [x, x + 1) x [y, y + 1), at fractions (tx, ty); everything the adjoint
// needs of the pixels is four sums per cell, of g ic times the weights of the
// cell's four corners (each weight by itself: 1 - tx taken from sums of 1 and tx
// would cancel on samples next to the far side).  The CTA walks down the image rows that the detector reaches in
// steps of a few 8-row bands, over as many 32-column groups as its buffer holds
// the detector columns of:
//   its warps march down the detector rows of the step's cells, 128 detector
//   columns at a time, four neighbours per lane in f32x2 pairs: per cell row
//   and column A0 = sum (1 - ty) g ic and A1 = sum ty g ic, to the buffer;
//   then a warp takes a band of a group: lane x sums its cell's columns, S0, S1
//   = sum (1 - tx) A0, A1 and T0, T1 = sum tx A0, A1, and with S = S0 + S1(y - 1)
//   and T alike, dL/dimg[y][x] = S + T(x - 1); the pose-offset sums take the
//   image's differences over the cell.
// Every element of dL/dimgs is written once (nothing to clear, no atomics).
// The sums of g rx dv/dpx and g ry dv/dpy come from rx = (x + tx - ox) / scale
// and ry alike, in f32 relative to the integer next to ox, oy.
// Bound by issue.  64 blocks x 64 poses x 256^2 pixels: 444 us, against 495
// with bands marched by one warp each and the image's values and differences
// interpolated at every detector column (two loads and nine operations per
// image row and detector column); 8 blocks x 64 poses x 512^2 pixels: 138
// against 265.
template <int THREADS, int MINB, bool WHOLE>
__global__ void __launch_bounds__(THREADS, MINB) pou_warp_sep_adjoint_kernel(SepArgs a, SepGrad w) {
  constexpr int NW = THREADS / 32;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[4][NW];
  // per thread: sums of g dv/dpx, g (x + tx - ox) dv/dpx, g dv/dpy, g (y + ty - oy) dv/dpy (no registers held
  // while marching)
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
  int* rcell = reinterpret_cast<int*>(smem + sep_adj_gbuf_at(P, Hd, W));  // in the sum buffer until it is used
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
  float* gimg = w.gimgs + (WHOLE ? bn : static_cast<int64_t>(b) * gridDim.x + n) * P * P;
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
  // as many 32-column groups per step as have their detector columns in the buffer (one group: in column passes if
  // they are more); rows of half the length leave room for up to four bands, of which those that keep the warps
  // busiest are taken
  const int groups = (P + 31) / 32;
  int gs = groups, cols = 0;
  for (;; --gs) {
    cols = 0;
    for (int g = 0; g < groups; g += gs) {
      int c0, c1;
      columns(32 * g - 1, min(P, 32 * (g + gs)), c0, c1);
      cols = max(cols, c1 - (c0 & ~3));
    }
    if (gs == 1 || cols <= kSepStepCols) break;
  }
  const bool narrow = cols <= kSepStepCols / 2;
  int bands = 1;
  for (int v = 2; v <= (narrow ? 4 : 2); ++v) {
    const int r0 = (bands * gs + NW - 1) / NW, r1 = (v * gs + NW - 1) / NW;
    if (r1 * bands <= r0 * v) bands = v;
  }
  float* buf = reinterpret_cast<float*>(smem + sep_adj_gbuf_at(P, Hd, W));
  const int step = rev_r ? -(Wp / 4) : Wp / 4;
  // x0 - ox, y0 - 1 - oy relative to the nearest integer of ox, oy; what is left of them is applied at the end, in f64
  const double rox = rint(ox), roy = rint(oy);
  float dx = 0.f, drx = 0.f, fy = 0.f, f1 = 0.f;
  auto steps = [&](auto row_length) {
    constexpr int pitch = decltype(row_length)::value;
    for (int xc = 0; xc < P; xc += 32 * gs) {
      const int xe = min(P, xc + 32 * gs);
      int ca, cb;
      columns(xc - 1, xe, ca, cb);
      const int cs = ca & ~3;  // 16-byte words of a detector row
      for (int ys = ya; ys < yb; ys += bands * kSepBand) {
        const int rows = min(bands * kSepBand, yb - ys);  // cells ys - 1 .. ys + rows - 1
        // lane's cell (two rows a pair) and, lane = cell row, the cell left of the group: sums over columns
        float2 S0[kSepPairs], T0[kSepPairs], S1[kSepPairs], T1[kSepPairs];
        float L0, LT0, L1, LT1;
        for (int kp = cs; kp < max(cb, cs + 1); kp += pitch) {
          const int ke = min(cb, kp + pitch);
          const int passes = (ke - kp + kSepPass - 1) / kSepPass, parts = passes % 2 ? NW : passes % 4 ? NW / 2 : NW / 4;
          __syncthreads();
          for (int u = wid; u < passes * parts; u += NW) {
            const int pass = u / parts, part = u - pass * parts;
            int cell = (rows + 1) * part / parts;
            const int cell1 = (rows + 1) * (part + 1) / parts;
            if (cell >= cell1) continue;
            const int c = kp + kSepPass * pass + 4 * lane;
            const bool on = c < Wp, keep = c < kp + pitch;
            const int kr1 = rfirst[ys + cell1];
            int kr = rfirst[ys + cell], kend = rfirst[ys + cell + 1];
            const float4* gq =
                w.gic + (static_cast<int64_t>(n) * Hd + (rev_r ? Hd - 1 - kr : kr)) * (Wp / 4) + c / 4;
            float4* q = reinterpret_cast<float4*>(buf + 2 * cell * pitch + (c - kp));
            float4 nxt[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              nxt[j] = make_float4(0.f, 0.f, 0.f, 0.f);
              if (on && kr + j < kr1) nxt[j] = __ldg(gq + j * step);
            }
            float2 A0[2], A1[2];
            A0[0] = A0[1] = A1[0] = A1[1] = bcast(0.f);
            auto flush = [&] {
              if (keep) {
                q[0] = make_float4(A0[0].x, A0[0].y, A0[1].x, A0[1].y);
                q[pitch / 4] = make_float4(A1[0].x, A1[0].y, A1[1].x, A1[1].y);
              }
              q += pitch / 2;
              A0[0] = A0[1] = A1[0] = A1[1] = bcast(0.f);
              ++cell;
              kend = rfirst[ys + cell + 1];
            };
            for (; kr < kr1; kr += 4) {
              float4 cur[4];
              gq += 4 * step;
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                cur[j] = nxt[j];
                if (on && kr + 4 + j < kr1) nxt[j] = __ldg(gq + j * step);
              }
#pragma unroll
              for (int j = 0; j < 4; ++j) {
                if (kr + j < kr1) {
                  while (kr + j >= kend) flush();
                  const float2 ty = bcast(rty[kr + j]), uy = bcast(1.f - rty[kr + j]);
                  const float2 g0 = make_float2(cur[j].x, cur[j].y), g1 = make_float2(cur[j].z, cur[j].w);
                  A0[0] = __ffma2_rn(uy, g0, A0[0]);
                  A0[1] = __ffma2_rn(uy, g1, A0[1]);
                  A1[0] = __ffma2_rn(ty, g0, A1[0]);
                  A1[1] = __ffma2_rn(ty, g1, A1[1]);
                }
              }
            }
            while (cell < cell1) flush();
          }
          __syncthreads();
          for (int u = wid; u < gs * bands; u += NW) {
            const int band = u / gs, xg = xc + 32 * (u - band * gs), y0 = ys + band * kSepBand;
            const int nr = min(kSepBand, ys + rows - y0);
            if (nr <= 0 || xg >= P) continue;
            const int x = xg + lane;
            const bool in = x < P, right = x + 1 < P;
            if (kp == cs) {
#pragma unroll
              for (int i = 0; i < kSepPairs; ++i) S0[i] = T0[i] = S1[i] = T1[i] = bcast(0.f);
              L0 = LT0 = L1 = LT1 = 0.f;
            }
            float vi[kSepBand + 1], ri[kSepBand + 1];  // image rows y0 - 1 .. y0 + nr - 1 at x, x + 1
            {
              const float* q = img + (y0 - 1) * P + x;
              const bool last = ke == cb;
#pragma unroll
              for (int i = 0; i <= kSepBand; ++i) {
                const bool row = last && in && i <= nr && y0 + i > 0;
                vi[i] = row ? __ldg(q + i * P) : 0.f;
                ri[i] = row && right ? __ldg(q + i * P + 1) : 0.f;
              }
            }
            const float* bq = buf + 2 * band * kSepBand * pitch - kp;
            int t0 = 0, t1 = 0, l0, l1;
            if (in) columns(x, x + 1, t0, t1);
            t1 = min(t1, ke);
            for (int k = max(t0, kp); k < t1; ++k) {
              if (!fvr_checked(k - kp, pitch, kSiteWarpFused)) continue;
              const float tx = __int_as_float(cmap[k].y);
              const float2 t = bcast(tx), u = bcast(1.f - tx);
              const float* q = bq + k;
#pragma unroll
              for (int i = 0; i < kSepPairs; ++i) {
                const float2 v0 = make_float2(q[4 * i * pitch], q[(4 * i + 2) * pitch]);
                const float2 v1 = make_float2(q[(4 * i + 1) * pitch], q[(4 * i + 3) * pitch]);
                S0[i] = __ffma2_rn(u, v0, S0[i]);
                T0[i] = __ffma2_rn(t, v0, T0[i]);
                S1[i] = __ffma2_rn(u, v1, S1[i]);
                T1[i] = __ffma2_rn(t, v1, T1[i]);
              }
            }
            columns(xg - 1, xg, l0, l1);
            if (lane <= nr)
              for (int k = max(l0, kp); k < min(l1, ke); ++k) {
                const float t = __int_as_float(cmap[k].y), v0 = bq[2 * lane * pitch + k],
                            v1 = bq[(2 * lane + 1) * pitch + k];
                L0 += v0;
                L1 += v1;
                LT0 = fmaf(t, v0, LT0);
                LT1 = fmaf(t, v1, LT1);
              }
            if (ke < cb) continue;
            // this unit's sums: with x and y relative to the lane's cell and to cell row y0 - 1
            float ux = 0.f, urx = 0.f, uy = 0.f, ury = 0.f;
            // the left cell's S and T of image row y0 + lane - 1 (lane >= 1)
            const float up = __shfl_up_sync(0xffffffffu, L1, 1), upt = __shfl_up_sync(0xffffffffu, LT1, 1);
            const float LS = L0 + up, LT = LT0 + upt;
            if (xg == 0 && l0 < l1) {  // column -1 is no image column: its sums are taken here, image values 0 there
              const int y = y0 + lane - 1;  // row y of the cell
              const float v = lane <= nr && y >= 0 ? img[y * P] : 0.f;
              const float below = lane <= nr && y + 1 < P ? img[(y + 1) * P] : 0.f;
              if (lane >= 1 && lane <= nr) {
                dx = fmaf(LS, v, dx);
                drx = fmaf(fmaf(static_cast<float>(-1 - rox), LS, LT), v, drx);
              }
              if (lane < nr || (lane == nr && y0 + nr == P)) {
                const float D = below - v, p = (LT0 + LT1) * D;
                uy = p;
                ury = fmaf(static_cast<float>(lane), p, LT1 * D);
              }
            }
            float* gq = gimg + y0 * P + x;
            float vp = vi[0], rp = ri[0];
            auto at = [](const float2(&a)[kSepPairs], int i) { return i & 1 ? a[i / 2].y : a[i / 2].x; };
            auto row = [&](int i) {
              const float v = vi[i + 1], r = ri[i + 1], d = r - v;
              const float SG = at(S0, i + 1) + at(S1, i);
              const float TG = at(T0, i + 1) + at(T1, i);
              const float tl = __shfl_up_sync(0xffffffffu, TG, 1), t0l = __shfl_sync(0xffffffffu, LT, i + 1);
              if (in) gq[i * P] = SG + (lane == 0 ? t0l : tl);
              ux = fmaf(SG + TG, d, ux);
              urx = fmaf(TG, d, urx);
              const float Dv = v - vp, Dr = r - rp;  // cell y - 1, at x and x + 1
              const float p = fmaf(at(T0, i) + at(T1, i), Dr, (at(S0, i) + at(S1, i)) * Dv);
              uy += p;
              ury = fmaf(at(S1, i), Dv, fmaf(static_cast<float>(i), p, ury));
              ury = fmaf(at(T1, i), Dr, ury);
              vp = v;
              rp = r;
            };
            if (nr == kSepBand && y0 + nr < P) {
#pragma unroll
              for (int i = 0; i < kSepBand; ++i) row(i);
            } else {
#pragma unroll
              for (int i = 0; i < kSepBand; ++i)
                if (i < nr) {
                  row(i);
                  if (i + 1 == nr && y0 + nr == P) {  // the last cell's lower row lies outside the image
                    const float p = fmaf(at(T0, i + 1) + at(T1, i + 1), -rp, (at(S0, i + 1) + at(S1, i + 1)) * -vp);
                    uy += p;
                    ury = fmaf(at(S1, i + 1), -vp, fmaf(static_cast<float>(i + 1), p, ury));
                    ury = fmaf(at(T1, i + 1), -rp, ury);
                  }
                }
            }
            dx += ux;
            drx += fmaf(static_cast<float>(x - rox), ux, urx);
            fy += uy;
            f1 += fmaf(static_cast<float>(y0 - 1 - roy), uy, ury);
          }
        }
        sums[0][threadIdx.x] += static_cast<double>(dx);
        sums[1][threadIdx.x] += static_cast<double>(drx);
        sums[2][threadIdx.x] += static_cast<double>(fy);
        sums[3][threadIdx.x] += static_cast<double>(f1);
        dx = drx = fy = f1 = 0.f;
      }
    }
  };
  if (narrow) steps(std::integral_constant<int, kSepStepCols / 2>{});
  else steps(std::integral_constant<int, kSepStepCols>{});
  sums[1][threadIdx.x] += (rox - ox) * sums[0][threadIdx.x];
  sums[3][threadIdx.x] += (roy - oy) * sums[2][threadIdx.x];
  // a block in the source plane (scale near 0) does not determine rx and ry from the image position: the sums of
  // g rx dv/dpx and g ry dv/dpy directly
  const bool direct = fabs(sc) < 1.0;
  double s_rx = sums[1][threadIdx.x], s_ry = sums[3][threadIdx.x];
  if (direct) {
    s_rx = s_ry = 0.0;
    for (int64_t q = threadIdx.x; q < static_cast<int64_t>(Hd) * W; q += THREADS) {
      const int r = static_cast<int>(q / W), c = static_cast<int>(q - static_cast<int64_t>(r) * W);
      const float rx = __ldg(a.rxc + c), ry = __ldg(a.ryr + r);
      float ty;
      const int iy = sep_cell(sc, oy, ry, P, ty), ix = cmap[c].x;
      if (iy < -1 || iy >= P || ix < -1 || ix >= P) continue;
      const float tx = __int_as_float(cmap[c].y);
      auto at = [&](int y, int x) { return y >= 0 && y < P && x >= 0 && x < P ? __ldg(img + y * P + x) : 0.f; };
      const float v00 = at(iy, ix), v01 = at(iy, ix + 1), v10 = at(iy + 1, ix), v11 = at(iy + 1, ix + 1);
      const double g = static_cast<double>(__ldg(gout + q) * __ldg(a.ic + q));
      s_rx += g * static_cast<double>(rx) * static_cast<double>((1.f - ty) * (v01 - v00) + ty * (v11 - v10));
      s_ry += g * static_cast<double>(ry) * static_cast<double>((1.f - tx) * (v10 - v00) + tx * (v11 - v01));
    }
  }
  const double mine[4] = {sums[0][threadIdx.x], s_rx, sums[2][threadIdx.x], s_ry};
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
    w.goffs[bn] = a.inv_ds * (direct ? t[1] + t[3] : (t[1] + t[3]) / sc);
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

template <int THREADS, int MINB, bool WHOLE>
static int sep_adjoint(const SepArgs& a, const SepGrad& w, int64_t poses, cudaStream_t s) {
  const int64_t smem = sep_adj_smem(a.P, a.Hd, a.W);
  // the shared-memory opt-in is a per-device setting: made before every launch
  if (cudaFuncSetAttribute(pou_warp_sep_adjoint_kernel<THREADS, MINB, WHOLE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           static_cast<int>(smem)) != cudaSuccess)
    return FVR_ERR_CUDA;
  pou_warp_sep_adjoint_kernel<THREADS, MINB, WHOLE>
      <<<dim3(static_cast<unsigned>(poses), static_cast<unsigned>(a.B)), THREADS, smem, s>>>(a, w);
  FVR_LAUNCH_CHECK();
  return FVR_OK;
}

template <int RG>
static int sep_forward(const SepArgs& a, float* out, cudaStream_t s) {
  const int64_t smem = 4LL * kSepRingRows * a.P;
  if (smem > kSmemPlain &&  // a per-device setting: before every such launch
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
  // The most rows per CTA that leave 8 warps an SM, four rows down to 5 warps an SM, below that the blocks split over
  // warps.  16 / 8 / 4 rows / split, us (warps at 16 rows): 64 blocks x 256^2 pixels, 64 poses (2048) 202 / 207 / 254 /
  // 743, 32 poses 158 / 115 / 162 / 376, 16 poses 148 / 92 / 83 / 190, 8 poses 146 / 85 / 67 / 96, 4 poses 147 / 86 /
  // 63 / 49; 8 blocks x 512^2, 16 poses (2048) 28 / 32 / 37 / 134, 4 poses 20 / 14 / 13 / 36.
  const int64_t row_warps = N * cdiv64(W, 32 * kSepCols);
  if (row_warps * cdiv64(H, 16) >= 8 * 148) return sep_forward<16>(a, out, s);
  if (row_warps * cdiv64(H, 8) >= 8 * 148) return sep_forward<8>(a, out, s);
  if (row_warps * cdiv64(H, 4) >= 5 * 148) return sep_forward<4>(a, out, s);
  const int xt = static_cast<int>(cdiv64(W, 32));
  pou_warp_sep_few_kernel<<<dim3(static_cast<unsigned>(xt * cdiv64(H, kSepFewRows)), static_cast<unsigned>(N)),
                            32 * kSepFewWarps, 0, s>>>(a, xt, out);
  FVR_LAUNCH_CHECK();
  return FVR_OK;
}

int fvr_pou_warp_sep_adjoint_supported(int64_t P, int64_t H, int64_t W) {
  if (!fvr_pou_warp_sep_supported(P, H, W)) return 0;
  // the row cells are staged in the buffer of cell-row sums, beside which the tables have 72 KB
  return H <= 16384 && sep_adj_gbuf_at((int)P, (int)H, (int)W) <= 72 * 1024 ? 1 : 0;
}

int64_t fvr_pou_warp_sep_adjoint_workspace(int64_t N, int64_t H, int64_t W) {
  return N < 1 || H < 1 || W < 1 ? 0 : 4 * N * H * ((W + 3) / 4 * 4);
}

int fvr_pou_warp_sep_adjoint_poses(const float* imgs, int64_t B, int64_t N, int64_t P, const double* offs,
                                   const float* rxc, const float* ryr, const float* ic, int64_t H, int64_t W,
                                   double inv_ds, double c_idx, const float* gout, int64_t n0, int64_t count,
                                   void* workspace, int64_t ws_bytes, float* grad_imgs, double* goffs, void* stream) {
  SepArgs a;
  const int rc = sep_args(imgs, B, N, P, offs, rxc, ryr, ic, H, W, inv_ds, c_idx, &a);
  if (rc) return rc;
  if (!gout || !grad_imgs || !goffs || !workspace || (reinterpret_cast<uintptr_t>(workspace) & 15)) return FVR_ERR_ARG;
  if (n0 < 0 || count < 1 || count > N - n0) return FVR_ERR_ARG;
  if (ws_bytes < fvr_pou_warp_sep_adjoint_workspace(count, H, W)) return FVR_ERR_WORKSPACE;
  if (!fvr_pou_warp_sep_adjoint_supported(P, H, W)) return FVR_ERR_UNSUPPORTED;
  a.imgs += n0 * P * P;
  a.offs += 3 * n0;
  gout += n0 * H * W;
  float4* gic = static_cast<float4*>(workspace);
  const SepGrad w{gout, gic, grad_imgs, goffs + n0};
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int Wp = sep_padded((int)W);
  const bool vec = W % 4 == 0 && ((reinterpret_cast<uintptr_t>(gout) | reinterpret_cast<uintptr_t>(ic)) & 15) == 0;
  pou_warp_sep_weigh_kernel<<<dim3((unsigned)cdiv64(H * (Wp / 4), 256), (unsigned)count), 256, 0, s>>>(
      gout, ic, (int)H, (int)W, Wp, vec, gic);
  FVR_LAUNCH_CHECK();
  // 256 threads once two CTAs per SM can run, else all 16 warps on one (pose, block)
  if (B * count >= 296)
    return count == N ? sep_adjoint<256, 2, true>(a, w, count, s) : sep_adjoint<256, 2, false>(a, w, count, s);
  return count == N ? sep_adjoint<512, 1, true>(a, w, count, s) : sep_adjoint<512, 1, false>(a, w, count, s);
}

int fvr_pou_warp_sep_adjoint(const float* imgs, int64_t B, int64_t N, int64_t P, const double* offs, const float* rxc,
                             const float* ryr, const float* ic, int64_t H, int64_t W, double inv_ds, double c_idx,
                             const float* gout, void* workspace, int64_t ws_bytes, float* grad_imgs, double* goffs,
                             void* stream) {
  return fvr_pou_warp_sep_adjoint_poses(imgs, B, N, P, offs, rxc, ryr, ic, H, W, inv_ds, c_idx, gout, 0, N, workspace,
                                        ws_bytes, grad_imgs, goffs, stream);
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

// Workspace of the backward: weighed detector gradient of a chunk | offset
// gradients | slice-adjoint records, each on a 256-byte boundary.
static int64_t pinhole_round(int64_t bytes) { return (bytes + 255) / 256 * 256; }

int64_t fvr_pou_pinhole_backward_chunked_workspace(int64_t B, int64_t N, int64_t H, int64_t W, int64_t chunk) {
  if (B < 1 || N < 1 || chunk < 1) return 0;
  return pinhole_round(fvr_pou_warp_sep_adjoint_workspace(chunk < N ? chunk : N, H, W)) + pinhole_round(24 * B * N) +
         fvr_pou_slice_image_adjoint_workspace(B, N);
}

int64_t fvr_pou_pinhole_backward_workspace(int64_t B, int64_t N, int64_t H, int64_t W) {
  return fvr_pou_pinhole_backward_chunked_workspace(B, N, H, W, N);
}

// Poses are independent up to the pose gradients at the end: dL/dimgs is formed
// and reduced for `chunk` of them at a time.
int fvr_pou_pinhole_backward_chunked(int dtype, const void* stencil, const float* scales, int64_t B, int64_t P,
                                     const double* geo, const double* offs, int64_t N, const double* base12,
                                     double vscale, const float* centers, const float* freqs, const float* imgs,
                                     const float* rxc, const float* ryr, const float* ic, int64_t H, int64_t W,
                                     double inv_ds, double c_idx, const float* gout, int64_t chunk, float* grad_imgs,
                                     void* workspace, int64_t ws_bytes, float* gmats, void* stream) {
  if (!workspace || !grad_imgs || (reinterpret_cast<uintptr_t>(workspace) & 15) || !gmats || !offs || !geo || N < 1 ||
      chunk < 1)
    return FVR_ERR_ARG;
  if (!fvr_pou_pinhole_supported(P, H, W) || !fvr_pou_warp_sep_adjoint_supported(P, H, W)) return FVR_ERR_UNSUPPORTED;
  if (ws_bytes < fvr_pou_pinhole_backward_chunked_workspace(B, N, H, W, chunk)) return FVR_ERR_WORKSPACE;
  if (chunk > N) chunk = N;
  const int64_t gic_bytes = fvr_pou_warp_sep_adjoint_workspace(chunk, H, W);
  char* w = static_cast<char*>(workspace);
  double* goffs = reinterpret_cast<double*>(w + pinhole_round(gic_bytes));
  double* part = reinterpret_cast<double*>(reinterpret_cast<char*>(goffs) + pinhole_round(24 * B * N));
  int rc = FVR_OK;
  for (int64_t n0 = 0; n0 < N && !rc; n0 += chunk) {
    const int64_t count = chunk < N - n0 ? chunk : N - n0;
    rc = fvr_pou_warp_sep_adjoint_poses(imgs, B, N, P, offs, rxc, ryr, ic, H, W, inv_ds, c_idx, gout, n0, count,
                                        workspace, gic_bytes, grad_imgs, goffs, stream);
    if (!rc)  // records [pose][block][6]
      rc = fvr_pou_slice_image_adjoint(dtype, stencil, scales, B, P, geo + n0 * fvr_pou_geo_stride(), count, freqs,
                                       grad_imgs, part + 6 * B * n0, fvr_pou_slice_image_adjoint_workspace(B, count),
                                       stream);
  }
  if (!rc)
    rc = fvr_pou_pose_backward(part, 1, goffs, nullptr, 0, geo, centers, B, N, base12, vscale, gmats, nullptr, stream);
  return rc;
}

int fvr_pou_pinhole_backward(int dtype, const void* stencil, const float* scales, int64_t B, int64_t P,
                             const double* geo, const double* offs, int64_t N, const double* base12, double vscale,
                             const float* centers, const float* freqs, const float* imgs, const float* rxc,
                             const float* ryr, const float* ic, int64_t H, int64_t W, double inv_ds, double c_idx,
                             const float* gout, float* grad_imgs, void* workspace, int64_t ws_bytes, float* gmats,
                             void* stream) {
  return fvr_pou_pinhole_backward_chunked(dtype, stencil, scales, B, P, geo, offs, N, base12, vscale, centers, freqs,
                                          imgs, rxc, ryr, ic, H, W, inv_ds, c_idx, gout, N, grad_imgs, workspace,
                                          ws_bytes, gmats, stream);
}

}  // extern "C"

FVR_CHECK_ACCESSOR(check_word_pou_sep)
