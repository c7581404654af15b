// Gradient band-pass filter (reference bandpass_filter, FD2DGPU.cu:4125-4182, with the Gaussian
// filter of construct_gaussian_bandpass_filter, FD2DGPU.cu:4038-4077, as the reference calls it
// at :4135).  Off the time-stepping path: the reference applies it, when enabled, once per LSRTM
// iteration to the summed gradients (main.cpp:1074-1089, commented out in the shipped loop).
//
// What the reference computes for one image f [nx][nz] (z fastest):
//   F = FFT2(f) in double complex (cuFFT Z2Z, unnormalised), quadrant swap S, multiply every
//   element by the complex number (k, k) (GPU_lowpass builds make_cuDoubleComplex(k, k), not
//   (k, 0)), quadrant swap S again, inverse FFT2, divide by nx*nz, keep the real part.
// S exchanges quadrant (y, x) with (y + nx/2, x + nz/2) and (y, x + nz/2) with (y + nx/2, x) for
// y < nx/2, x < nz/2 (fft_shift / ifft_shift); for odd sizes the last row / column stay put.  S is
// an involution and the multiply is elementwise, so S (k F) S-swapped equals k(S(j)) F(j): the
// filter simply acts in natural frequency order as k' = k o S.  The result is therefore
//   out = Re(IFFT2((1 + i) k' F)) / (nx nz) = (Re g - Im g) / (nx nz),  g = IFFT2(k' F).
//
// Here each 1D transform of up to kFftMaxN points is one CTA's work in shared memory, by Bluestein's
// chirp-z method (Bluestein 1970): the benchmark grids are odd or prime (1201, 401, 601), so a DFT
// of any length becomes a circular convolution with a chirp, done by power-of-two FFTs of M >=
// 2n - 1 points.  Along x the forward transform, the filter and the inverse transform are one
// kernel (a column never leaves shared memory in between), so an image is read and written three
// times in all.  The filter and every table are computed on the device.  Two 1201 x 401
// host images on a B200: 80 (up to 180) -> 1.35 ms a call, 0.31 ms of it in kernels (k_fft_x 181 us: six radix-4
// passes of shared memory per transform set the pace), the rest copies.  Longer transforms take dense DFT products (k_dft_gemm) with
// tables built on the host: exact for any size, about 0.1 s a call.
#pragma once
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

namespace ds2d {

constexpr int kDftTile = 16;

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ void cmac(double2 &acc, double2 a, double2 b) {
  acc.x = fma(a.x, b.x, acc.x);
  acc.x = fma(-a.y, b.y, acc.x);
  acc.y = fma(a.x, b.y, acc.y);
  acc.y = fma(a.y, b.x, acc.y);
}

// Operand / result access of one DFT product C[m][n] = sum_k A[m][k] B[k][n].
struct DftArgs {
  int M, N, K;
  // A: real float [M][K] (lda), or complex [M][K] (lda); B: complex [K][N] (ldb)
  const float *a_real;
  const double2 *a, *b;
  long long lda, ldb;
  // epilogue: complex C [M][N] (ldc), optionally times (k, k) with k = filt[m][n] (ldf);
  // or the real part of C / scale as float into out_real [M][N] (ldo)
  double2 *c;
  long long ldc;
  const float *filt;
  long long ldf;
  float *out_real;
  long long ldo;
  double scale;
};

__global__ void __launch_bounds__(kDftTile *kDftTile) k_dft_gemm(DftArgs p) {
  __shared__ double2 As[kDftTile][kDftTile + 1], Bs[kDftTile][kDftTile + 1];
  const int tx = threadIdx.x % kDftTile, ty = threadIdx.x / kDftTile;
  const int m = blockIdx.y * kDftTile + ty, n = blockIdx.x * kDftTile + tx;
  double2 acc = make_double2(0.0, 0.0);
  for (int k0 = 0; k0 < p.K; k0 += kDftTile) {
    const int ka = k0 + tx, kb = k0 + ty;
    double2 av = make_double2(0.0, 0.0), bv = make_double2(0.0, 0.0);
    if (m < p.M && ka < p.K)
      av = p.a_real ? make_double2((double)p.a_real[(long long)m * p.lda + ka], 0.0)
                    : p.a[(long long)m * p.lda + ka];
    if (kb < p.K && n < p.N) bv = p.b[(long long)kb * p.ldb + n];
    As[ty][tx] = av;
    Bs[ty][tx] = bv;
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kDftTile; kk++) cmac(acc, As[ty][kk], Bs[kk][tx]);
    __syncthreads();
  }
  if (m >= p.M || n >= p.N) return;
  if (p.out_real) {  // GPU_divide then Z2R: real part / (nx nz), as float
    p.out_real[(long long)m * p.ldo + n] = (float)(acc.x / p.scale);
    return;
  }
  if (p.filt) {
    const double k = (double)p.filt[(long long)m * p.ldf + n];
    acc = cmul(acc, make_double2(k, k));
  }
  p.c[(long long)m * p.ldc + n] = acc;
}

// ---- Bluestein transforms ----------------------------------------------------------------------
constexpr int kFftMaxN = 4096;   // M = 2^13 points: 144 KB of shared memory
constexpr int kFftMaxLogM = 13;
constexpr int kFftT = 256;

struct FftPlan {
  int n, logm;               // transform length, log2 of the convolution length M
  const double2 *tw;         // [M / 4] exp(-2 pi i m / M)
  const double2 *chirp;      // [n] exp(-pi i j^2 / n)
  const double2 *spec;       // [M] FFT of the conjugate chirp, in the order fft_dif leaves
};

// Shared position of element i: one 16-byte element of padding per 8, so the passes with small
// strides spread over the banks.
__host__ __device__ __forceinline__ int fft_pos(int i) { return i + (i >> 3); }
inline size_t fft_smem(int logm) { return sizeof(double2) * (size_t)fft_pos(1 << logm); }

__device__ __forceinline__ double2 cadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 csub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }

// In-place forward FFT (decimation in frequency: natural order in, bit-reversed out), two radix-2
// stages per pass over the data; ends with a barrier.
__device__ __forceinline__ void fft_dif(double2 *x, const double2 *tw, int logm) {
  const int m = 1 << logm;
  int lh = logm;
  for (; lh >= 2; lh -= 2) {
    const int q = 1 << (lh - 2);
    for (int t = threadIdx.x; t < m / 4; t += kFftT) {
      const int j = t & (q - 1), i = ((t >> (lh - 2)) << lh) + j;
      double2 &p0 = x[fft_pos(i)], &p1 = x[fft_pos(i + q)], &p2 = x[fft_pos(i + 2 * q)], &p3 = x[fft_pos(i + 3 * q)];
      const double2 x0 = p0, x1 = p1, x2 = p2, x3 = p3;
      const double2 w = __ldg(tw + ((size_t)j << (logm - lh))), w2 = cmul(w, w);
      const double2 y0 = cadd(x0, x2), y1 = cadd(x1, x3);
      const double2 y2 = cmul(csub(x0, x2), w), d = cmul(csub(x1, x3), w);
      const double2 y3 = make_double2(d.y, -d.x);  // times -i
      p0 = cadd(y0, y1);
      p1 = cmul(csub(y0, y1), w2);
      p2 = cadd(y2, y3);
      p3 = cmul(csub(y2, y3), w2);
    }
    __syncthreads();
  }
  if (lh == 1) {
    for (int t = threadIdx.x; t < m / 2; t += kFftT) {
      double2 &p0 = x[fft_pos(2 * t)], &p1 = x[fft_pos(2 * t + 1)];
      const double2 a = p0, b = p1;
      p0 = cadd(a, b);
      p1 = csub(a, b);
    }
    __syncthreads();
  }
}

// In-place inverse FFT without the 1 / M (decimation in time: bit-reversed in, natural out).
__device__ __forceinline__ void fft_dit_inv(double2 *x, const double2 *tw, int logm) {
  const int m = 1 << logm;
  int lh = 2;
  if (logm & 1) {
    for (int t = threadIdx.x; t < m / 2; t += kFftT) {
      double2 &p0 = x[fft_pos(2 * t)], &p1 = x[fft_pos(2 * t + 1)];
      const double2 a = p0, b = p1;
      p0 = cadd(a, b);
      p1 = csub(a, b);
    }
    __syncthreads();
    lh = 3;
  }
  for (; lh <= logm; lh += 2) {
    const int q = 1 << (lh - 2);
    for (int t = threadIdx.x; t < m / 4; t += kFftT) {
      const int j = t & (q - 1), i = ((t >> (lh - 2)) << lh) + j;
      double2 &p0 = x[fft_pos(i)], &p1 = x[fft_pos(i + q)], &p2 = x[fft_pos(i + 2 * q)], &p3 = x[fft_pos(i + 3 * q)];
      const double2 w = cconj(__ldg(tw + ((size_t)j << (logm - lh)))), w2 = cmul(w, w);
      const double2 z0 = p0, z1 = cmul(p1, w2), z2 = p2, z3 = cmul(p3, w2);
      const double2 y0 = cadd(z0, z1), y1 = csub(z0, z1);
      const double2 y2 = cmul(cadd(z2, z3), w), d = cmul(csub(z2, z3), w);
      const double2 y3 = make_double2(-d.y, d.x);  // times i
      p0 = cadd(y0, y2);
      p2 = csub(y0, y2);
      p1 = cadd(y1, y3);
      p3 = csub(y1, y3);
    }
    __syncthreads();
  }
}

// Chirp-z transform of the n chirped inputs in x (zeros from n to M): x[k], times chirp[k] / M, is
// the DFT.  The caller has written x; starts and ends with a barrier.
__device__ __forceinline__ void bluestein(double2 *x, const FftPlan &p) {
  __syncthreads();
  fft_dif(x, p.tw, p.logm);
  for (int i = threadIdx.x; i < 1 << p.logm; i += kFftT) x[fft_pos(i)] = cmul(x[fft_pos(i)], __ldg(p.spec + i));
  __syncthreads();
  fft_dit_inv(x, p.tw, p.logm);
}

struct FftTables {
  int n, logm;
  double2 *tw, *chirp, *spec;
};
struct FftTables2 {
  FftTables t[2];
};
// Twiddles and chirps of the two directions (grid.y).
__global__ void __launch_bounds__(kFftT) k_fft_tables(FftTables2 a) {
  const FftTables &t = a.t[blockIdx.y];
  const int m = 1 << t.logm, i = blockIdx.x * kFftT + threadIdx.x;
  double s, c;
  if (i < m / 4) {
    sincospi(-2.0 * i / m, &s, &c);
    t.tw[i] = make_double2(c, s);
  }
  if (i < t.n) {  // j^2 mod 2n keeps the angle small
    sincospi(-(double)(((long long)i * i) % (2LL * t.n)) / t.n, &s, &c);
    t.chirp[i] = make_double2(c, s);
  }
}
__global__ void __launch_bounds__(kFftT) k_fft_spec(FftTables2 a) {
  extern __shared__ __align__(16) unsigned char fft_sm[];
  double2 *x = reinterpret_cast<double2 *>(fft_sm);
  const FftTables &t = a.t[blockIdx.x];
  const int m = 1 << t.logm;
  for (int i = threadIdx.x; i < m; i += kFftT) {
    const int j = i < t.n ? i : m - i < t.n ? m - i : -1;
    x[fft_pos(i)] = j >= 0 ? cconj(t.chirp[j]) : make_double2(0.0, 0.0);
  }
  __syncthreads();
  fft_dif(x, t.tw, t.logm);
  for (int i = threadIdx.x; i < m; i += kFftT) t.spec[i] = x[fft_pos(i)];
}

// The band-pass filter (gaussian_bandpass below, same arithmetic) before its normalisation, and
// the bits of its maximum.
__global__ void __launch_bounds__(256) k_bandpass_filter(int nx, int nz, int low, int high, float *f,
                                                         unsigned *fmax) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  float g = 0.f;
  if (i < (long long)nx * nz) {
    const int y = (int)(i / nz), x = (int)(i - (long long)y * nz);
    const int dx = x - nz / 2, dy = y - nx / 2;
    const float scale = __fdiv_rn((float)nz, (float)nx), sy = __fmul_rn(scale, (float)dy);
    const float dist = __fsqrt_rn(__fadd_rn((float)(dx * dx), __fmul_rn(sy, sy)));
    const float d2 = __fmul_rn(-dist, dist);
    g = low == 0 ? (float)exp(d2 / (2.0 * high * high))
                 : (float)(exp(d2 / (2.0 * high * high)) - exp(d2 / (2.0 * low * low)));
    if (g < 0) g = 0;
    f[i] = g;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) g = fmaxf(g, __shfl_xor_sync(0xffffffffu, g, o));
  if ((threadIdx.x & 31) == 0 && g > 0.f) atomicMax(fmax, __float_as_uint(g));
}

struct FftImages {
  float *img[2];       // [nx][nz]
  double2 *t[2];       // [nx][nz] work planes
  int nx, nz;
  const float *filt;   // [nx][nz], quadrant-centred, not normalised
  const unsigned *fmax;
};

// Forward along z: one CTA per row and image.
__global__ void __launch_bounds__(kFftT) k_fft_z(FftImages a, FftPlan p) {
  extern __shared__ __align__(16) unsigned char fft_sm[];
  double2 *x = reinterpret_cast<double2 *>(fft_sm);
  const float *src = a.img[blockIdx.y] + (size_t)blockIdx.x * a.nz;
  double2 *dst = a.t[blockIdx.y] + (size_t)blockIdx.x * a.nz;
  const int m = 1 << p.logm;
  for (int i = threadIdx.x; i < m; i += kFftT) {
    double2 v = make_double2(0.0, 0.0);
    if (i < p.n) {
      const double2 c = __ldg(p.chirp + i);
      const double f = src[i];
      v = make_double2(f * c.x, f * c.y);
    }
    x[fft_pos(i)] = v;
  }
  bluestein(x, p);
  const double sc = 1.0 / m;
  for (int i = threadIdx.x; i < p.n; i += kFftT) {
    const double2 v = cmul(x[fft_pos(i)], __ldg(p.chirp + i));
    dst[i] = make_double2(v.x * sc, v.y * sc);
  }
}

// Along x: forward transform, filter in natural frequency order times (k, k), inverse transform
// (the conjugate of a forward transform of the conjugate).  One CTA per column and image, in place.
__global__ void __launch_bounds__(kFftT) k_fft_x(FftImages a, FftPlan p) {
  extern __shared__ __align__(16) unsigned char fft_sm[];
  double2 *x = reinterpret_cast<double2 *>(fft_sm);
  double2 *col = a.t[blockIdx.y] + blockIdx.x;
  const int m = 1 << p.logm, nz = a.nz, hx = a.nx / 2, hz = nz / 2, z = blockIdx.x;
  for (int i = threadIdx.x; i < m; i += kFftT)
    x[fft_pos(i)] = i < p.n ? cmul(col[(size_t)i * nz], __ldg(p.chirp + i)) : make_double2(0.0, 0.0);
  bluestein(x, p);
  const double sc = 1.0 / m;
  const float fm = __uint_as_float(*a.fmax);
  for (int i = threadIdx.x; i < m; i += kFftT) {
    double2 v = make_double2(0.0, 0.0);
    if (i < p.n) {
      const double2 c = __ldg(p.chirp + i);
      const double2 g = cmul(x[fft_pos(i)], c);
      const bool swap = i < 2 * hx && z < 2 * hz;  // quadrant_swap
      const int jx = !swap ? i : i < hx ? i + hx : i - hx, jz = !swap ? z : z < hz ? z + hz : z - hz;
      const double k = (double)__fdiv_rn(a.filt[(size_t)jx * nz + jz], fm);
      const double2 h = cmul(make_double2(g.x * sc, g.y * sc), make_double2(k, k));
      v = cmul(cconj(h), c);
    }
    x[fft_pos(i)] = v;
  }
  bluestein(x, p);
  for (int i = threadIdx.x; i < p.n; i += kFftT) {
    const double2 v = cmul(x[fft_pos(i)], __ldg(p.chirp + i));
    col[(size_t)i * nz] = make_double2(v.x * sc, -v.y * sc);
  }
}

// Inverse along z, real part / (nx nz) into the image.
__global__ void __launch_bounds__(kFftT) k_fft_z_inv(FftImages a, FftPlan p) {
  extern __shared__ __align__(16) unsigned char fft_sm[];
  double2 *x = reinterpret_cast<double2 *>(fft_sm);
  const double2 *src = a.t[blockIdx.y] + (size_t)blockIdx.x * a.nz;
  float *dst = a.img[blockIdx.y] + (size_t)blockIdx.x * a.nz;
  const int m = 1 << p.logm;
  for (int i = threadIdx.x; i < m; i += kFftT)
    x[fft_pos(i)] = i < p.n ? cmul(cconj(src[i]), __ldg(p.chirp + i)) : make_double2(0.0, 0.0);
  bluestein(x, p);
  const double sc = 1.0 / m, n = (double)(a.nx * a.nz);
  for (int i = threadIdx.x; i < p.n; i += kFftT)
    dst[i] = (float)(cmul(x[fft_pos(i)], __ldg(p.chirp + i)).x * sc / n);
}

// Host side -----------------------------------------------------------------------------------

// construct_gaussian_bandpass_filter(filter, width = nz, height = nx, low, high) in the
// reference's own arithmetic (FD2DGPU.cu:4038-4077): float distance, double exponentials stored
// as float, negative values clamped to 0, normalised to a maximum of 1; low == 0 gives the
// low-pass form.  Indexed [ix][iz] like the images.
inline std::vector<float> gaussian_bandpass(int nx, int nz, int low, int high) {
  std::vector<float> f((size_t)nx * nz);
  const int cx = nz / 2, cy = nx / 2;
  float maxv = 0.0f;
  for (int y = 0; y < nx; y++)
    for (int x = 0; x < nz; x++) {
      const int dx = x - cx, dy = y - cy;
      const float scale = float(nz) / nx;
      const float dist = std::sqrt((float)(dx * dx) + (scale * dy) * (scale * dy));
      const float d2 = -dist * dist;
      float g;
      if (low == 0)
        g = (float)std::exp(d2 / (2.0 * high * high));
      else
        g = (float)(std::exp(d2 / (2.0 * high * high)) - std::exp(d2 / (2.0 * low * low)));
      if (g < 0) g = 0;
      f[(size_t)y * nz + x] = g;
      if (g > maxv) maxv = g;
    }
  for (float &v : f) v /= maxv;
  return f;
}

// The quadrant swap S of fft_shift / ifft_shift (FD2DGPU.cu:3922-3965) as an index map on
// [ix][iz] (an involution; for odd sizes the last row and column map to themselves).
inline size_t quadrant_swap(int nx, int nz, int ix, int iz) {
  const int hx = nx / 2, hz = nz / 2;
  if (ix < 2 * hx && iz < 2 * hz) {
    const int jx = ix < hx ? ix + hx : ix - hx;
    const int jz = iz < hz ? iz + hz : iz - hz;
    return (size_t)jx * nz + jz;
  }
  return (size_t)ix * nz + iz;
}

// DFT matrix W[j][k] = exp(sign 2 pi i (j k mod n) / n) in FP64.
inline std::vector<double2> dft_matrix(int n, int sign) {
  std::vector<double2> w((size_t)n * n);
  const double two_pi = 6.283185307179586476925286766559;
  for (int j = 0; j < n; j++)
    for (int k = 0; k < n; k++) {
      const long long m = ((long long)j * k) % n;
      const double a = sign * two_pi * (double)m / n;
      w[(size_t)j * n + k] = make_double2(std::cos(a), std::sin(a));
    }
  return w;
}

}  // namespace ds2d
