// Parallel-beam image path on whole images in shared memory, sm_100a
// (src/fvr/torch_engine.py:236-253, 309-337): one CTA or two per image.
//
//  * tc_image_kernel: modulated slice -> inverse 2D FFT -> real part -> ReLU;
//  * tc_image_adjoint_kernel: ReLU mask -> 2D FFT of the image gradient ->
//    slice adjoint -> pose gradient;
//  * cncc_image_kernel: spectral NCC of an image pair and its image gradient,
//    both spectra from one complex transform (pred + i target), the gradient
//    by the inverse transform of the closed-form spectral gradient.
//
// All transforms use that the image side is real: the row pass runs over the
// rows 0 .. n0/2 of a Hermitian spectrum (or over pairs of real rows), the
// column pass over pairs of real columns (or over the columns 0 .. n1/2), so a
// transform is n0/2 + n1/2 lines.  A warp transforms a line on its own: copy to
// its scratch, Stockham passes, copy back.  While SMs are left over, a cluster
// of two CTAs shares an image: each takes half the lines of a pass and writes
// the results to the CTA that reads them next.
//
// As separate passes over memory an image step (render, image NCC, pose
// gradient) was 19 launches, ten of them line-FFT passes of 22 us for 64 images
// of 96 x 96; here it is five.  Kernels at that size: render 19 us, NCC with its
// image gradient 31 us, adjoint 24 us (288 us before; with one CTA an image 28,
// 39 and 33); bound by issue in the 128 CTAs, 32 warps each, and by the
// latency of a line's passes.
#include <cooperative_groups.h>

#include "fvr_dft.cuh"
#include "fvr_slice.cuh"

namespace fvr {

constexpr int kImgPasses = 8;

struct LinePlan {  // mixed-radix plan of one line length, per pass: n / radix, n / (Ns radix), 1 / Ns
  int n, npass, radix[kImgPasses], nb[kImgPasses], step[kImgPasses];
  float inv_ns[kImgPasses];
};

static bool line_plan(int64_t n, LinePlan* p) {
  FftPlan f;
  if (!make_plan(n, &f) || f.npass > kImgPasses) return false;
  p->n = f.n;
  p->npass = f.npass;
  int Ns = 1;
  for (int i = 0; i < f.npass; ++i) {
    p->radix[i] = f.radix[i];
    p->nb[i] = f.n / f.radix[i];
    p->step[i] = f.n / (Ns * f.radix[i]);
    p->inv_ns[i] = 1.f / static_cast<float>(Ns);
    Ns *= f.radix[i];
  }
  return true;
}

// j / Ns and j % Ns for 0 <= j < 4096 (inv = 1 / Ns; the quotient's distance
// from an integer is at least 0.5 / Ns, far above the float rounding).
__device__ __forceinline__ int quotient(int j, float inv) { return __float2int_rz((static_cast<float>(j) + 0.5f) * inv); }

// One radix-R Stockham pass of a line of n values by a warp.
template <int R, bool INV>
__device__ __forceinline__ void line_pass(const Cx<float>* src, Cx<float>* dst, int Ns, int n, int nb, int step,
                                          float inv_ns, const Cx<float>* tw, int lane) {
  for (int j = lane; j < nb; j += 32) {
    const int q = quotient(j, inv_ns), k = j - q * Ns;
    Cx<float> v[R];
#pragma unroll
    for (int t = 0; t < R; ++t) v[t] = src[j + t * nb];
    if (Ns > 1) {
#pragma unroll
      for (int t = 1; t < R; ++t) {
        Cx<float> w = tw[t * k * step];
        if (INV) w.y = -w.y;
        v[t] = cmul(v[t], w);
      }
    }
    Dft<float, R>::run(v, INV);
    Cx<float>* d = dst + q * Ns * R + k;
#pragma unroll
    for (int t = 0; t < R; ++t) d[t * Ns] = v[t];
  }
}

// The same for an odd radix without a register butterfly: the inputs are
// twiddled in place, then a lane forms outputs m and r - m together from the
// sums and differences of inputs t and r - t (a quarter of the products of the
// plain sum).
template <bool INV>
__device__ __forceinline__ void wide_pass(Cx<float>* src, Cx<float>* dst, int r, int Ns, int n, int nb, int step,
                                          float inv_ns, const Cx<float>* tw, int lane) {
  const float inv_nb = 1.f / static_cast<float>(nb);
  if (Ns > 1) {
    for (int e = nb + lane; e < n; e += 32) {
      const int t = quotient(e, inv_nb), j = e - t * nb, k = j - quotient(j, inv_ns) * Ns;
      Cx<float> w = tw[t * k * step];
      if (INV) w.y = -w.y;
      src[e] = cmul(src[e], w);
    }
    __syncwarp();
  }
  const int h = (r - 1) / 2;
  for (int e = lane; e < nb * (h + 1); e += 32) {
    const int m = quotient(e, inv_nb), j = e - m * nb, q = quotient(j, inv_ns), k = j - q * Ns, d = m * nb;
    const Cx<float> x0 = src[j];
    Cx<float> even = x0, odd{0.f, 0.f};
    int at = 0;
    for (int t = 1; t <= h; ++t) {
      at += d;
      if (at >= n) at -= n;
      const Cx<float> w = tw[at];  // (cos, -sin)
      const Cx<float> u = src[j + t * nb], v = src[j + (r - t) * nb];
      even.x = fmaf(u.x + v.x, w.x, even.x);
      even.y = fmaf(u.y + v.y, w.x, even.y);
      odd.x = fmaf(v.y - u.y, w.y, odd.x);
      odd.y = fmaf(u.x - v.x, w.y, odd.y);
    }
    if (INV) odd = Cx<float>{-odd.x, -odd.y};
    Cx<float>* o = dst + q * Ns * r + k;
    o[m * Ns] = cadd(even, odd);
    if (m > 0) o[(r - m) * Ns] = csub(even, odd);
  }
}

// Transforms the line in `a` (n values); the result is in the returned buffer.
template <bool INV>
__device__ __forceinline__ const Cx<float>* line_fft(Cx<float>* a, Cx<float>* b, const LinePlan& p,
                                                     const Cx<float>* tw, int lane) {
  Cx<float>*src = a, *dst = b;
  int Ns = 1;
  const int n = p.n;
  for (int i = 0; i < p.npass; ++i) {
    const int r = p.radix[i], nb = p.nb[i], step = p.step[i];
    const float inv_ns = p.inv_ns[i];
    __syncwarp();
    if (r == 4) line_pass<4, INV>(src, dst, Ns, n, nb, step, inv_ns, tw, lane);
    else if (r == 2) line_pass<2, INV>(src, dst, Ns, n, nb, step, inv_ns, tw, lane);
    else if (r == 3) line_pass<3, INV>(src, dst, Ns, n, nb, step, inv_ns, tw, lane);
    else if (r == 5) line_pass<5, INV>(src, dst, Ns, n, nb, step, inv_ns, tw, lane);
    else wide_pass<INV>(src, dst, r, Ns, n, nb, step, inv_ns, tw, lane);
    Cx<float>* t = src;
    src = dst;
    dst = t;
    Ns *= r;
  }
  __syncwarp();
  return src;
}

// Shared memory: the image [n0][n1 + 1] complex, the two twiddle tables, two
// line buffers per warp.
struct ImgShape {
  int n0, n1;
  LinePlan p0, p1;        // columns (length n0), rows (length n1)
  const float2 *tw0, *tw1;
};

__host__ __device__ constexpr int64_t img_smem(int64_t n0, int64_t n1, int warps) {
  return 8 * (n0 * (n1 + 1) + n0 + n1 + 2 * warps * (n0 > n1 ? n0 : n1));
}

struct ImgMem {
  Cx<float>*buf, *tw0, *tw1, *la, *lb;
};

template <int THREADS>
__device__ __forceinline__ ImgMem img_mem(unsigned char* smem, const ImgShape& s) {
  ImgMem m;
  const int nm = max(s.n0, s.n1), wid = threadIdx.x >> 5;
  m.buf = reinterpret_cast<Cx<float>*>(smem);
  m.tw0 = m.buf + s.n0 * (s.n1 + 1);
  m.tw1 = m.tw0 + s.n0;
  m.la = m.tw1 + s.n1 + 2 * wid * nm;
  m.lb = m.la + nm;
  for (int i = threadIdx.x; i < s.n0; i += THREADS) m.tw0[i] = Cx<float>{__ldg(&s.tw0[i].x), __ldg(&s.tw0[i].y)};
  for (int i = threadIdx.x; i < s.n1; i += THREADS) m.tw1[i] = Cx<float>{__ldg(&s.tw1[i].x), __ldg(&s.tw1[i].y)};
  return m;
}

// The CTAs of a cluster share an image (one CTA: all of it).  Of the columns of
// the half spectrum, kx = 0 .. n1/2, rank r takes [c0, c1) together with their
// mirrors n1 - kx, of the row pairs [p0, p1).  A pass writes a line's results
// into the buffer of the rank that reads them next, which holds nothing else
// there; a cluster barrier stands between passes.
struct ImgPart {
  int nr, rank, h, c0, c1, p0, p1, pc;  // pc: first row pair of rank 1
  int n_up;                             // own columns above n1 / 2

  __device__ __forceinline__ void init(int n0, int n1) {
    const auto cl = cooperative_groups::this_cluster();
    nr = static_cast<int>(cl.num_blocks());
    rank = static_cast<int>(cl.block_rank());
    h = n1 / 2;
    const int pairs = (n0 + 1) / 2;
    c0 = (h + 1) * rank / nr;
    c1 = (h + 1) * (rank + 1) / nr;
    p0 = pairs * rank / nr;
    p1 = pairs * (rank + 1) / nr;
    pc = nr > 1 ? pairs / nr : pairs;
    n_up = max(0, min(c1, (n1 + 1) / 2) - max(c0, 1));
  }
  __device__ __forceinline__ int cols() const { return c1 - c0 + n_up; }
  // natural index of own column e < cols()
  __device__ __forceinline__ int col(int e, int n1) const {
    return e < c1 - c0 ? c0 + e : n1 - max(c0, 1) - (e - (c1 - c0));
  }
  __device__ __forceinline__ int col_rank(int k, int n1) const {
    return nr > 1 && min(k, n1 - k) >= (h + 1) / nr ? 1 : 0;
  }
  __device__ __forceinline__ int row_rank(int y) const { return (y >> 1) >= pc ? 1 : 0; }
  // every rank's copy of a shared-memory array
  template <typename T>
  __device__ __forceinline__ void map(T* p, T* (&out)[2]) const {
    out[0] = out[1] = p;
    if (nr > 1) out[1 - rank] = cooperative_groups::this_cluster().map_shared_rank(p, 1 - rank);
  }
  __device__ __forceinline__ void sync() const {
    if (nr > 1) cooperative_groups::this_cluster().sync();
    else __syncthreads();
  }
};

// Inverse transform (unnormalised) of a Hermitian spectrum to a real image:
// the columns kx <= n1/2, then the rows two at a time as real and imaginary
// part of one line.  col(r, kx) gives the spectrum in an own column; it may
// read buffer columns kx and (n1 - kx) mod n1.  out(y, x, v) takes the image
// of the own row pairs.
template <int THREADS, typename F, typename O>
__device__ __forceinline__ void hermitian_to_real(const ImgShape& s, const ImgMem& m, const ImgPart& part, F col, O out) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, pitch = s.n1 + 1;
  Cx<float>* bufs[2];
  part.map(m.buf, bufs);
  for (int kx = part.c0 + wid; kx < part.c1; kx += (THREADS / 32)) {
    for (int r = lane; r < s.n0; r += 32) m.la[r] = col(r, kx);
    const Cx<float>* y = line_fft<true>(m.la, m.lb, s.p0, m.tw0, lane);
    for (int r = lane; r < s.n0; r += 32) bufs[part.row_rank(r)][r * pitch + kx] = y[r];
    __syncwarp();
  }
  part.sync();
  for (int t = part.p0 + wid; t < part.p1; t += (THREADS / 32)) {
    const bool two = 2 * t + 1 < s.n0;
    const Cx<float>* src = m.buf + 2 * t * pitch;
    for (int k = lane; k < s.n1; k += 32) {
      const int kk = k <= part.h ? k : s.n1 - k;
      const float sg = kk == 0 || 2 * kk == s.n1 ? 0.f : k <= part.h ? 1.f : -1.f;  // those are real
      const Cx<float> p = src[kk], q = two ? src[pitch + kk] : Cx<float>{0.f, 0.f};
      m.la[k] = Cx<float>{p.x - sg * q.y, sg * p.y + q.x};
    }
    const Cx<float>* z = line_fft<true>(m.la, m.lb, s.p1, m.tw1, lane);
    for (int x = lane; x < s.n1; x += 32) {
      out(2 * t, x, z[x].x);
      if (two) out(2 * t + 1, x, z[x].y);
    }
    __syncwarp();
  }
}

// ----------------------------------------------------------------------------
// image forward
// ----------------------------------------------------------------------------

struct TcImageArgs {
  SliceArgs sl;         // axes unused: formed from the pose here
  const float* poses;   // [C][6]
  int lateral;
  ImgShape sh;          // n0 = n1 = R
  double kappa;
};

template <int DT, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) tc_image_kernel(TcImageArgs a, float* __restrict__ img) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double ax[8];
  const int R = a.sl.R, pitch = R + 1, h = R / 2;
  const ImgMem m = img_mem<THREADS>(smem, a.sh);
  ImgPart part;
  part.init(R, R);
  const int c = blockIdx.x / part.nr, cols = part.cols();
  if (threadIdx.x == 0) slice_axes(a.poses + 6 * c, a.lateral, a.sl.sx, a.sl.sy, a.sl.sz, ax);
  __syncthreads();
  for (int q = threadIdx.x; q < R * cols; q += THREADS) {
    const int i = q / cols, jj = part.col(q - i * cols, R), j = jj + h < R ? jj + h : jj + h - R;
    Interp o;
    float sn, cs;
    slice_sample<DT, false>(a.sl, ax, __ldg(a.sl.lin + i), __ldg(a.sl.lin + j), o, sn, cs);
    const int ii = i < h ? i - h + R : i - h;  // ifftshift position
    m.buf[ii * pitch + jj] = Cx<float>{o.sr * cs - o.si * sn, o.sr * sn + o.si * cs};
  }
  part.sync();
  // Re ifft2(S) = ifft2 of S's Hermitian part
  const float scale = 1.f / (static_cast<float>(R) * static_cast<float>(R));
  float* out = img + static_cast<int64_t>(c) * R * R;
  hermitian_to_real<THREADS>(
      a.sh, m, part,
      [&](int r, int k) {
        const Cx<float> p = m.buf[r * pitch + k], q = m.buf[(r == 0 ? 0 : R - r) * pitch + (k == 0 ? 0 : R - k)];
        return Cx<float>{0.5f * (p.x + q.x), 0.5f * (p.y - q.y)};
      },
      [&](int y, int x, float z) {
        const float v = z * scale;
        out[y * R + x] = v > 0.f ? v : 0.f;
      });
}

// ----------------------------------------------------------------------------
// image adjoint
// ----------------------------------------------------------------------------

// Buffer use: the spectra of row pairs [ceil(R/2)][R + 1], then the half
// spectrum [R][R/2 + 1].
__host__ __device__ constexpr int64_t img_adjoint_smem(int64_t R, int warps) {
  return 8 * ((R + 1) / 2 * (R + 1) + R * (R / 2 + 1) + R + 2 * warps * R);
}

template <int DT, int THREADS>
__global__ void __launch_bounds__(THREADS, 1) tc_image_adjoint_kernel(TcImageArgs a, const float* __restrict__ img,
                                                                          const float* __restrict__ gout,
                                                                          float* __restrict__ grad) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double ax[8], red[8][(THREADS / 32)], sums[2][8];
  const int R = a.sl.R, half = R / 2, lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  ImgPart part;
  part.init(R, R);
  const int c = blockIdx.x / part.nr, cols = part.cols();
  const int zp = R + 1, gp = half + 1;
  Cx<float>* zr = reinterpret_cast<Cx<float>*>(smem);
  Cx<float>* gb = zr + (R + 1) / 2 * zp;
  Cx<float>* tw = gb + R * gp;
  Cx<float>*la = tw + R + 2 * wid * R, *lb = la + R;
  for (int i = threadIdx.x; i < R; i += THREADS)
    tw[i] = Cx<float>{__ldg(&a.sh.tw1[i].x), __ldg(&a.sh.tw1[i].y)};
  if (threadIdx.x == 0) slice_axes(a.poses + 6 * c, a.lateral, a.sl.sx, a.sl.sy, a.sl.sz, ax);
  Cx<float>* zrs[2];
  part.map(zr, zrs);
  part.sync();
  const float *im = img + static_cast<int64_t>(c) * R * R, *go = gout + static_cast<int64_t>(c) * R * R;
  // rows 2s and 2s + 1 of the masked gradient as real and imaginary part of one line
  for (int s = part.p0 + wid; s < part.p1; s += (THREADS / 32)) {
    const int y = 2 * s;
    for (int k = lane; k < R; k += 32) {
      const float u = __ldg(im + y * R + k) > 0.f ? __ldg(go + y * R + k) : 0.f;
      const float v = y + 1 < R && __ldg(im + (y + 1) * R + k) > 0.f ? __ldg(go + (y + 1) * R + k) : 0.f;
      la[k] = Cx<float>{u, v};
    }
    const Cx<float>* z = line_fft<false>(la, lb, a.sh.p1, tw, lane);
    for (int k = lane; k < R; k += 32) zrs[part.col_rank(k, R)][s * zp + k] = z[k];
    __syncwarp();
  }
  part.sync();
  const float scale = 1.f / (static_cast<float>(R) * static_cast<float>(R));
  for (int kx = part.c0 + wid; kx < part.c1; kx += (THREADS / 32)) {
    const int km = kx == 0 ? 0 : R - kx;
    for (int y = lane; y < R; y += 32) {
      const Cx<float> A = zr[(y >> 1) * zp + kx], B = zr[(y >> 1) * zp + km];
      la[y] = (y & 1) ? Cx<float>{0.5f * (A.y + B.y), 0.5f * (B.x - A.x)}
                      : Cx<float>{0.5f * (A.x + B.x), 0.5f * (A.y - B.y)};
    }
    const Cx<float>* z = line_fft<false>(la, lb, a.sh.p0, tw, lane);
    for (int y = lane; y < R; y += 32) gb[y * gp + kx] = Cx<float>{z[y].x * scale, z[y].y * scale};
    __syncwarp();
  }
  __syncthreads();
  // dL/dS = e^{-i phi} G and dL/dphi = Re(conj(G) i S) per sample
  double acc[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int q = threadIdx.x; q < R * cols; q += THREADS) {
    const int i = q / cols, kj = part.col(q - i * cols, R), j = kj + half < R ? kj + half : kj + half - R;
    const float ku = __ldg(a.sl.lin + i), kv = __ldg(a.sl.lin + j);
    Interp o;
    float sn, cs;
    slice_sample<DT, true>(a.sl, ax, ku, kv, o, sn, cs);
    const int ki = i < half ? i - half + R : i - half;
    Cx<float> g;  // G at frequency (ki, kj); G(-k) = conj G(k)
    if (kj <= half) {
      g = gb[ki * gp + kj];
    } else {
      g = gb[(ki == 0 ? 0 : R - ki) * gp + R - kj];
      g.y = -g.y;
    }
    const float shr = o.sr * cs - o.si * sn, shi = o.sr * sn + o.si * cs;
    const float ph = g.y * shr - g.x * shi;
    const float dr = cs * g.x + sn * g.y, di = cs * g.y - sn * g.x;
    const float e0 = dr * o.dxr + di * o.dxi, e1 = dr * o.dyr + di * o.dyi, e2 = dr * o.dzr + di * o.dzi;
    acc[0] += ku * e0;
    acc[1] += ku * e1;
    acc[2] += ku * e2;
    acc[3] += kv * e0;
    acc[4] += kv * e1;
    acc[5] += kv * e2;
    acc[6] += ku * ph;
    acc[7] += kv * ph;
  }
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const double v = warp_sum(acc[k]);
    if (lane == 0) red[k][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 8) {
    double t = 0.0;
    for (int w = 0; w < (THREADS / 32); ++w) t += red[threadIdx.x][w];
    double* p[2];
    part.map(&sums[part.rank][threadIdx.x], p);
    *p[0] = t;  // to rank 0
  }
  part.sync();
  if (part.rank == 0 && threadIdx.x == 0) {
    double r[8];
    for (int k = 0; k < 8; ++k) r[k] = part.nr > 1 ? sums[0][k] + sums[1][k] : sums[0][k];
    const double du[3] = {r[0], r[1], r[2]}, dv[3] = {r[3], r[4], r[5]};
    double ga[3];
    axes_vjp(a.poses + 6 * c, a.lateral, a.sl.sx, a.sl.sy, a.sl.sz, du, dv, ga);
    float* o = grad + 6 * c;
    for (int k = 0; k < 3; ++k) o[k] = static_cast<float>(ga[k]);
    o[3] = static_cast<float>(a.kappa * r[6]);
    o[4] = static_cast<float>(a.kappa * r[7]);
    o[5] = 0.f;
  }
}

// ----------------------------------------------------------------------------
// image spectral NCC
// ----------------------------------------------------------------------------

// Largest magnitude of n values over the CTA, as float bits (non-negative
// floats order as integers, infinity and NaN above them).
template <int THREADS>
__device__ __forceinline__ unsigned image_max(const float* p, int64_t n, unsigned* red) {
  unsigned m = 0u;
  for (int64_t i = threadIdx.x; i < n; i += THREADS) m = max(m, __float_as_uint(fabsf(__ldg(p + i))));
  m = __reduce_max_sync(0xffffffffu, m);
  __syncthreads();
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  m = 0u;
  for (int w = 0; w < THREADS / 32; ++w) m = max(m, red[w]);
  return m;
}

// Power of two that brings a largest magnitude (float bits) into [1, 2).
__device__ __forceinline__ float unit_scale(unsigned bits) {
  const int e = static_cast<int>(bits >> 23);
  return e == 255 || bits == 0u ? 1.f : ldexpf(1.f, 127 - max(e, 1));
}

// ncc[b] of pred[b] and target[b or 0] (both multiplied by the high-pass table,
// fftshift order, or unfiltered), and with grad the gradient of 1 - mean ncc.
// The pair shares one transform, whose rounding follows the larger of the two,
// so both are first scaled to one magnitude (exactly, by powers of two), and
// the spectrum of an image of zeros is taken as zero.
template <int THREADS>
__global__ void __launch_bounds__(THREADS, 1) cncc_image_kernel(ImgShape s, const float* __restrict__ pred,
                                                                    const float* __restrict__ target,
                                                                    int64_t t_stride, const float* __restrict__ hp,
                                                                    int B, double* __restrict__ ncc,
                                                                    float* __restrict__ grad) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double red[3][(THREADS / 32)];
  __shared__ float coef[2];
  __shared__ unsigned wmax[THREADS / 32];
  __shared__ double sums[2][3];
  const int n0 = s.n0, n1 = s.n1, pitch = n1 + 1;
  ImgPart part;
  part.init(n0, n1);
  const int b = blockIdx.x / part.nr, cols = part.cols();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t n = static_cast<int64_t>(n0) * n1;
  const ImgMem m = img_mem<THREADS>(smem, s);
  Cx<float>* bufs[2];
  part.map(m.buf, bufs);
  part.sync();
  const float *pp = pred + b * n, *tp = target + b * t_stride;
  const unsigned pmax = image_max<THREADS>(pp, n, wmax), tmax = image_max<THREADS>(tp, n, wmax);
  const float sp = unit_scale(pmax), st = unit_scale(tmax);
  for (int r = n0 * part.rank / part.nr + wid; r < n0 * (part.rank + 1) / part.nr; r += (THREADS / 32)) {
    for (int k = lane; k < n1; k += 32) m.la[k] = Cx<float>{sp * __ldg(pp + r * n1 + k), st * __ldg(tp + r * n1 + k)};
    const Cx<float>* y = line_fft<false>(m.la, m.lb, s.p1, m.tw1, lane);
    for (int k = lane; k < n1; k += 32) bufs[part.col_rank(k, n1)][r * pitch + k] = y[k];
    __syncwarp();
  }
  part.sync();
  for (int e = wid; e < cols; e += (THREADS / 32)) {
    const int c = part.col(e, n1);
    for (int r = lane; r < n0; r += 32) m.la[r] = m.buf[r * pitch + c];
    const Cx<float>* y = line_fft<false>(m.la, m.lb, s.p0, m.tw0, lane);
    for (int r = lane; r < n0; r += 32) m.buf[r * pitch + c] = y[r];
    __syncwarp();
  }
  __syncthreads();
  // Fp = (Z(k) + conj Z(-k)) / 2, Ft = (Z(k) - conj Z(-k)) / 2i; the squared
  // high-pass weight averaged over k and -k (the products are equal there)
  auto spectra = [&](int r, int k, Cx<float>& fp, Cx<float>& ft) {
    const int rm = r == 0 ? 0 : n0 - r, km = k == 0 ? 0 : n1 - k;
    const Cx<float> z = m.buf[r * pitch + k], y = m.buf[rm * pitch + km];
    fp = Cx<float>{0.5f * (z.x + y.x), 0.5f * (z.y - y.y)};
    ft = Cx<float>{0.5f * (z.y + y.y), 0.5f * (y.x - z.x)};
    if (pmax == 0u) fp = Cx<float>{0.f, 0.f};
    if (tmax == 0u) ft = Cx<float>{0.f, 0.f};
    if (!hp) return 1.f;
    const int h0 = n0 / 2, h1 = n1 / 2;  // frequency k sits at (k + n/2) mod n of the table
    const float u = __ldg(hp + ((r + h0) % n0) * n1 + (k + h1) % n1);
    const float v = __ldg(hp + ((rm + h0) % n0) * n1 + (km + h1) % n1);
    return 0.5f * (u * u + v * v);
  };
  float acc[3] = {0.f, 0.f, 0.f};
  const int rows = n0 / 2 + 1;
  for (int q = threadIdx.x; q < rows * cols; q += THREADS) {
    const int r = q / cols, k = part.col(q - r * cols, n1);
    Cx<float> fp, ft;
    const float w = spectra(r, k, fp, ft) * (r == 0 || 2 * r == n0 ? 1.f : 2.f);
    acc[0] = fmaf(w, fmaf(fp.x, ft.x, fp.y * ft.y), acc[0]);
    acc[1] = fmaf(w, fmaf(fp.x, fp.x, fp.y * fp.y), acc[1]);
    acc[2] = fmaf(w, fmaf(ft.x, ft.x, ft.y * ft.y), acc[2]);
  }
#pragma unroll
  for (int k = 0; k < 3; ++k) {
    const double v = warp_sum(static_cast<double>(acc[k]));
    if (lane == 0) red[k][wid] = v;
  }
  __syncthreads();
  if (threadIdx.x < 3) {
    double t = 0.0;
    for (int w = 0; w < (THREADS / 32); ++w) t += red[threadIdx.x][w];
    double* p[2];
    part.map(&sums[part.rank][threadIdx.x], p);
    for (int r = 0; r < part.nr; ++r) *p[r] = t;
  }
  part.sync();
  if (threadIdx.x == 0) {
    double t[3];
    for (int k = 0; k < 3; ++k) t[k] = part.nr > 1 ? sums[0][k] + sums[1][k] : sums[0][k];
    const double up = 1.0 / sp, ut = 1.0 / st;  // back to the images' own scales
    t[0] *= up * ut;
    t[1] *= up * up;
    t[2] *= ut * ut;
    const double e = sqrt(t[1] * t[2]);
    const double aa = 1.0 / (e + 1e-8);
    const double bb = e > 0.0 ? -t[0] * t[2] / (2.0 * e * (e + 1e-8) * (e + 1e-8)) : 0.0;
    if (part.rank == 0) ncc[b] = t[0] * aa;
    coef[0] = static_cast<float>(-aa / B * ut);
    coef[1] = static_cast<float>(-2.0 * bb / B * up);
  }
  if (!grad) return;
  __syncthreads();
  const float ca = coef[0], cb = coef[1];
  float* out = grad + b * n;
  hermitian_to_real<THREADS>(
      s, m, part,
      [&](int r, int k) {
        Cx<float> fp, ft;
        const float w = spectra(r, k, fp, ft);
        return Cx<float>{w * (ca * ft.x + cb * fp.x), w * (ca * ft.y + cb * fp.y)};
      },
      [&](int y, int x, float v) { out[y * n1 + x] = v; });
}

// loss = 1 - mean ncc, in a fixed order.
__global__ void cncc_mean_kernel(const double* __restrict__ ncc, int B, float* __restrict__ loss) {
  double s = 0.0;
  for (int i = threadIdx.x; i < B; i += 32) s += ncc[i];
  s = warp_sum(s);
  if (threadIdx.x == 0) *loss = static_cast<float>(1.0 - s / B);
}

// Largest dynamic shared memory a CTA may use beside the kernels' static part.
constexpr int64_t kImgSmemMax = 224 * 1024;

static bool img_shape(int64_t n0, int64_t n1, const void* tw0, const void* tw1, ImgShape* s) {
  if (n0 < 2 || n1 < 2 || n0 > 4096 || n1 > 4096) return false;
  s->n0 = static_cast<int>(n0);
  s->n1 = static_cast<int>(n1);
  s->tw0 = static_cast<const float2*>(tw0);
  s->tw1 = static_cast<const float2*>(tw1);
  return line_plan(n0, &s->p0) && line_plan(n1, &s->p1);
}

static int image_args(int dtype, const void* stencil, const float* scales, int64_t D, int64_t H, int64_t W,
                      const float* poses, int64_t C, int view, const float* lin, int64_t R, double kappa,
                      const void* tw, TcImageArgs* a) {
  Stencil st;
  const int rc = stencil_from(dtype, stencil, scales, D, H, W, &st);
  if (rc) return rc;
  if (!poses || !lin || !tw || C < 1 || C > 65535 || (view != 0 && view != 1)) return FVR_ERR_ARG;
  a->sl = SliceArgs{st, nullptr, lin, (int)R, kappa / 3.14159265358979323846, half_extent(W), half_extent(H),
                    half_extent(D), 0};
  a->poses = poses;
  a->lateral = view;
  a->kappa = kappa;
  if (!img_shape(R, R, tw, tw, &a->sh)) return FVR_ERR_UNSUPPORTED;
  return FVR_OK;
}

// Launches kernel<1024> where its line buffers fit, else kernel<512>, two CTAs
// to an image where that pays: a pair takes 0.67 (render) to 0.79 (NCC) of one
// CTA's time for 96 x 96 images, so it does while all pairs fit in one wave,
// and not at 150 images (three waves of pairs 213 us, two of single CTAs 210).
// The shared-memory opt-in is a per-device setting: made before every launch.
template <typename K, typename... A>
static int img_launch(K wide, int64_t wide_smem, K narrow, int64_t narrow_smem, int64_t images, cudaStream_t s,
                      A... args) {
  const bool w = wide_smem <= kImgSmemMax;
  const int64_t smem = w ? wide_smem : narrow_smem;
  const K k = w ? wide : narrow;
  int dev = 0, sms = 0;
  if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess ||
      cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
    return FVR_ERR_CUDA;
  const int64_t one = (images + sms - 1) / sms, two = (2 * images + sms - 1) / sms;
  const unsigned pair = 3 * two < 4 * one ? 2 : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(images) * pair);
  cfg.blockDim = dim3(w ? 1024 : 512);
  cfg.dynamicSmemBytes = static_cast<size_t>(smem);
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = pair;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k, args...) == cudaSuccess ? FVR_OK : FVR_ERR_CUDA;
}

}  // namespace fvr

using namespace fvr;

extern "C" {

int fvr_image_supported(int64_t n0, int64_t n1) {
  ImgShape s;
  return img_shape(n0, n1, nullptr, nullptr, &s) && img_smem(n0, n1, 16) <= kImgSmemMax &&
                 (n0 != n1 || img_adjoint_smem(n0, 16) <= kImgSmemMax)
             ? 1
             : 0;
}

int fvr_tc_image(int dtype, const void* stencil, const float* scales, int64_t D, int64_t H, int64_t W,
                 const float* poses, int64_t C, int view, const float* lin, int64_t R, double kappa, const void* tw,
                 float* img, void* stream) {
  TcImageArgs a;
  const int rc = image_args(dtype, stencil, scales, D, H, W, poses, C, view, lin, R, kappa, tw, &a);
  if (rc) return rc;
  if (!img) return FVR_ERR_ARG;
  if (!fvr_image_supported(R, R)) return FVR_ERR_UNSUPPORTED;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t w = img_smem(R, R, 32), n = img_smem(R, R, 16);
  switch (dtype) {
    case FVR_F32: return img_launch(tc_image_kernel<FVR_F32, 1024>, w, tc_image_kernel<FVR_F32, 512>, n, C, s, a, img);
    case FVR_BF16:
      return img_launch(tc_image_kernel<FVR_BF16, 1024>, w, tc_image_kernel<FVR_BF16, 512>, n, C, s, a, img);
    case FVR_F16: return img_launch(tc_image_kernel<FVR_F16, 1024>, w, tc_image_kernel<FVR_F16, 512>, n, C, s, a, img);
  }
  return FVR_ERR_DTYPE;
}

int fvr_tc_image_backward(int dtype, const void* stencil, const float* scales, int64_t D, int64_t H, int64_t W,
                          const float* poses, int64_t C, int view, const float* lin, int64_t R, double kappa,
                          const void* tw, const float* img, const float* gout, float* grad_poses, void* stream) {
  TcImageArgs a;
  const int rc = image_args(dtype, stencil, scales, D, H, W, poses, C, view, lin, R, kappa, tw, &a);
  if (rc) return rc;
  if (!img || !gout || !grad_poses) return FVR_ERR_ARG;
  if (!fvr_image_supported(R, R)) return FVR_ERR_UNSUPPORTED;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t w = img_adjoint_smem(R, 32), n = img_adjoint_smem(R, 16);
  switch (dtype) {
    case FVR_F32:
      return img_launch(tc_image_adjoint_kernel<FVR_F32, 1024>, w, tc_image_adjoint_kernel<FVR_F32, 512>, n, C, s, a,
                        img, gout, grad_poses);
    case FVR_BF16:
      return img_launch(tc_image_adjoint_kernel<FVR_BF16, 1024>, w, tc_image_adjoint_kernel<FVR_BF16, 512>, n, C, s, a,
                        img, gout, grad_poses);
    case FVR_F16:
      return img_launch(tc_image_adjoint_kernel<FVR_F16, 1024>, w, tc_image_adjoint_kernel<FVR_F16, 512>, n, C, s, a,
                        img, gout, grad_poses);
  }
  return FVR_ERR_DTYPE;
}

int64_t fvr_cncc_image_workspace(int64_t B) { return B < 1 ? 0 : 8 * B; }

int fvr_cncc_image(const float* pred, const float* target, int64_t B, int64_t Bt, int64_t n0, int64_t n1,
                   const float* hp, const void* tw0, const void* tw1, void* workspace, int64_t ws_bytes, float* loss,
                   float* grad, void* stream) {
  if (!pred || !target || !tw0 || !tw1 || !workspace || !loss || B < 1 || B > 65535 || (Bt != 1 && Bt != B))
    return FVR_ERR_ARG;
  if (ws_bytes < fvr_cncc_image_workspace(B)) return FVR_ERR_WORKSPACE;
  ImgShape s;
  if (!img_shape(n0, n1, tw0, tw1, &s) || img_smem(n0, n1, 16) > kImgSmemMax) return FVR_ERR_UNSUPPORTED;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  double* ncc = static_cast<double*>(workspace);
  const int rc = img_launch(cncc_image_kernel<1024>, img_smem(n0, n1, 32), cncc_image_kernel<512>,
                            img_smem(n0, n1, 16), B, st, s, pred, target, Bt == 1 ? (int64_t)0 : n0 * n1, hp, (int)B,
                            ncc, grad);
  if (rc) return rc;
  cncc_mean_kernel<<<1, 32, 0, st>>>(ncc, (int)B, loss);
  FVR_LAUNCH_CHECK();
  return FVR_OK;
}

}  // extern "C"

FVR_CHECK_ACCESSOR(check_word_image)
