// FP32 ramp filter by FFT (sm_100a).
//
// The reference filters each zero-padded row with cuFFT (R2C, multiply by the
// spectrum of the fftshifted taps and 1/N, C2R; ReconstructionMachine.cu:
// 206-290, cuda_kernels.cuh:41-58). On the nch data samples that circular
// convolution is the linear one y[n] = sum_k h[|n-k|] x[k] when the transform
// is long enough. Evaluated as a Toeplitz product (k_toeplitz_f32) a row costs
// 2 nch^2 FLOP, 1.6 M at nch = 888, and the FP32 pipe bounds it; by FFT of
// N = 2048 it costs about 0.12 M.
//
// Precision. A line integral's row is large and smooth and its filtered row
// small (the ramp removes the mean), so an FFT of the row itself, whose
// rounding is relative to the row, is 4 times less exact than the Toeplitz
// product (measured). The transform therefore runs on the row's differences
// d[i] = x[i] - x[i-1], i = 0 .. nch (x = 0 outside), which are exact or
// rounded relative to the difference: y[n] = sum_i d[i] a[n - i] with the
// running sums a[m] = h[0] / 2 + h[1] + ... + h[m], a[-1-m] = -a[m] (the
// constant that makes them antisymmetric meets sum d = 0). Its kernel a acts
// like a Hilbert transform, whose spectrum is flat. Both rows of a pair meet the
// transform's rounding, which is relative to the 2-norm of what is transformed:
// each is scaled by a power of two that brings the norm of its differences near 1
// (a row scaled by its largest sample was, smooth beside a rough row, up to 45
// times less exact than the Toeplitz product; by the norm it is more exact than
// that); twiddles and spectrum are rounded from FP64.
// A row with a sample that is not finite or beyond 1e30 (where the transform's
// sums could overflow although the filtered row does not), and a row of few
// samples that are not 0 (a lone reading, the gradient of a small region), is
// summed as the Toeplitz product sums it: the product's error grows with the root
// of the terms, the transform's is spread over the whole row, and they cross at 25
// samples (N = 256) to 70 (N = 2048) and 90 (N = 4096; one sample: 3e-8 of the row
// against 1e-7). "Few" is 64, 96 from N = 1024, 128 at N = 4096.
//
// Two rows are one complex sequence d_a + i d_b: the kernel a is real, so the
// inverse transform is y_a + i y_b without any unpacking. N = 16 R2 R3 points
// run as three passes of radix 16, R2 and R3, 16 points per thread, T = N / 16
// threads per transform:
//   pass 1  (from global memory)  radix 16 over n1, twiddle
//   pass 2                        radix R2 over n2, twiddle
//   pass 3                        radix R3 over n3, times A / N, inverse radix R3
//   pass 2', pass 1'              the same backwards, to global memory
// in place in shared memory, so no pass reorders its data: the frequencies
// stay in digit-reversed order, in which the spectrum is stored. nch < N / 2,
// so the upper eight inputs and outputs of the first radix 16 do not exist: it
// is two radix-8 transforms. Real and imaginary parts are separate arrays with
// a pad of R3 words per k1 block and the 16-byte chunks of a radix-R3 group
// permuted, which makes every access of the five passes conflict-free.
//
// Bound by shared-memory wavefronts (67 % of the pipe) and issue (63 %) at 16 warps
// per SM, by registers: 64 rows of 888 channels, 2460 views, 0.83 ms (Toeplitz
// product 5.8).
#include "wfbp_internal.h"

#include <math.h>

#include <algorithm>
#include <vector>

namespace {

constexpr int FF_THREADS = 128;  // threads per CTA of the transforms with at most 128 threads
constexpr unsigned FF_BIG = 0x7149F2CAu;  // 1e30f

// N = 16 R2 R3
template <int N> struct FftShape;
template <> struct FftShape<256> { static constexpr int R2 = 1, R3 = 16; };
template <> struct FftShape<512> { static constexpr int R2 = 8, R3 = 4; };
template <> struct FftShape<1024> { static constexpr int R2 = 16, R3 = 4; };
template <> struct FftShape<2048> { static constexpr int R2 = 16, R3 = 8; };
template <> struct FftShape<4096> { static constexpr int R2 = 16, R3 = 16; };

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// a * w, or a * conj(w)
template <bool INV>
__device__ __forceinline__ float2 cmul(float2 a, float2 w) {
  return INV ? make_float2(fmaf(a.x, w.x, a.y * w.y), fmaf(a.y, w.x, -a.x * w.y))
             : make_float2(fmaf(a.x, w.x, -a.y * w.y), fmaf(a.y, w.x, a.x * w.y));
}
// a * (-i), or a * i
template <bool INV>
__device__ __forceinline__ float2 crot(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2& a0, float2& a1, float2& a2, float2& a3) {
  const float2 t0 = cadd(a0, a2), t1 = csub(a0, a2), t2 = cadd(a1, a3), t3 = crot<INV>(csub(a1, a3));
  a0 = cadd(t0, t2);
  a1 = cadd(t1, t3);
  a2 = csub(t0, t2);
  a3 = csub(t1, t3);
}

// v[k] = sum_j v[j] w8^(jk)
template <bool INV>
__device__ __forceinline__ void dft8(float2 (&v)[8]) {
  constexpr float h = 0.70710678118654752f;
  float2 e0 = v[0], e1 = v[2], e2 = v[4], e3 = v[6], o0 = v[1], o1 = v[3], o2 = v[5], o3 = v[7];
  dft4<INV>(e0, e1, e2, e3);
  dft4<INV>(o0, o1, o2, o3);
  o1 = INV ? make_float2(h * (o1.x - o1.y), h * (o1.x + o1.y)) : make_float2(h * (o1.x + o1.y), h * (o1.y - o1.x));
  o2 = crot<INV>(o2);
  o3 = INV ? make_float2(-h * (o3.x + o3.y), h * (o3.x - o3.y)) : make_float2(h * (o3.y - o3.x), -h * (o3.x + o3.y));
  v[0] = cadd(e0, o0);
  v[4] = csub(e0, o0);
  v[1] = cadd(e1, o1);
  v[5] = csub(e1, o1);
  v[2] = cadd(e2, o2);
  v[6] = csub(e2, o2);
  v[3] = cadd(e3, o3);
  v[7] = csub(e3, o3);
}

// exp(-2 pi i j / 16)
__device__ __forceinline__ constexpr float w16c(int j) {
  constexpr float c1 = 0.92387953251128674f, c2 = 0.70710678118654752f, c3 = 0.38268343236508977f;
  const float t[16] = {1, c1, c2, c3, 0, -c3, -c2, -c1, -1, -c1, -c2, -c3, 0, c3, c2, c1};
  return t[j & 15];
}
__device__ __forceinline__ float2 w16(int j) { return make_float2(w16c(j), w16c(j + 4)); }

template <bool INV>
__device__ __forceinline__ void dft16(float2 (&v)[16]) {
#pragma unroll
  for (int j = 0; j < 4; j++) dft4<INV>(v[j], v[j + 4], v[j + 8], v[j + 12]);
#pragma unroll
  for (int j = 1; j < 4; j++)
#pragma unroll
    for (int k = 1; k < 4; k++) v[j + 4 * k] = cmul<INV>(v[j + 4 * k], w16(j * k));
  float2 o[16];
#pragma unroll
  for (int k = 0; k < 4; k++) {
    dft4<INV>(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
#pragma unroll
    for (int m = 0; m < 4; m++) o[k + 4 * m] = v[4 * k + m];
  }
#pragma unroll
  for (int k = 0; k < 16; k++) v[k] = o[k];
}

template <int R, bool INV>
__device__ __forceinline__ void dft(float2 (&v)[R]) {
  if constexpr (R == 16) dft16<INV>(v);
  else if constexpr (R == 8) dft8<INV>(v);
  else if constexpr (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
}

// Barrier over the threads that share a transform (a warp holds whole
// transforms when T <= 32).
template <int T>
__device__ __forceinline__ void fft_sync() {
  if constexpr (T <= 32) __syncwarp();
  else __syncthreads();
}

// The 16-byte chunks of a group of R3 points are permuted by the group's index
// (n2; with two passes, R2 = 1, k1), so that the vector accesses of pass 3
// reach all banks: xor of the word within the group.
template <int R3>
__device__ __forceinline__ int chunk_xor(int group) {
  if constexpr (R3 == 8) return ((group >> 2) & 1) << 2;
  if constexpr (R3 == 16) return ((group >> 1) & 3) << 2;
  return 0;
}
// Word of point t = n2 R3 + n3 of block k1.
template <int R2, int R3, int BLK>
__device__ __forceinline__ int fft_word(int k1, int t) {
  return k1 * BLK + (t ^ chunk_xor<R3>(R2 > 1 ? t / R3 : k1));
}

// Sum over the threads of a transform, or of a warp where a transform takes several.
template <int T>
__device__ __forceinline__ unsigned reduce_add(unsigned v) {
  if constexpr (T >= 32) return __reduce_add_sync(0xffffffffu, v);
#pragma unroll
  for (int o = T / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// The power of two (biased exponent) that a row is divided by, from its eight
// differences in each thread: that of their 2-norm over the threads of a
// transform, or of a warp where a transform takes several (the row takes its
// warps' largest: at most sqrt(8) below its norm's); FF_OUT where a difference is
// not finite or FF_BIG or more. some: the thread's samples that are not 0 in, the
// transform's or warp's out.
constexpr unsigned FF_OUT = 255u;

template <int T>
__device__ __forceinline__ unsigned row_exponent(const float2 (&a)[8], float float2::*row, unsigned& some) {
  unsigned top = 0u;  // magnitudes order as their bits, NaN above all
#pragma unroll
  for (int j = 0; j < 8; j++) top = max(top, __float_as_uint(a[j].*row) & 0x7fffffffu);
  if constexpr (T >= 32) {
    top = __reduce_max_sync(0xffffffffu, top);
  } else {
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
  }
  const unsigned e = max(top >> 23, 1u);
  const float s = __uint_as_float((254u - min(e, 253u)) << 23);  // the largest times s is in [1, 2)
  float q = 0.0f;
  if (e - 80u < 94u) {  // the squares and s squared are in range
#pragma unroll
    for (int j = 0; j < 8; j++) q = fmaf(a[j].*row, a[j].*row, q);
    q *= s * s;
  } else {
#pragma unroll
    for (int j = 0; j < 8; j++) q = fmaf(a[j].*row * s, a[j].*row * s, q);
  }
  // at most 32 x 8 squares below 4 in units of 2^-7, and the samples, in one sum
  const unsigned sum = reduce_add<T>(((unsigned)(q * 128.0f) << 12) + some);
  some = sum & 0xfffu;
  return top >= FF_BIG ? FF_OUT : e + (unsigned)(max(31 - __clz((int)sum) - 19, 0) >> 1);
}

// y[n] = sum_k x[k] h[|n - k|] over the samples that are not 0, in order of k
// (the Toeplitz product's chain), for a thread's eight outputs.
template <int T>
__device__ __forceinline__ void direct_sum(const float* __restrict__ x, const float* __restrict__ taps, int nch, int t,
                                        float2 (&a)[8], float float2::*row) {
  float y[8];
#pragma unroll
  for (int j = 0; j < 8; j++) y[j] = 0.0f;
  auto add = [&](int k, float xk) {
#pragma unroll
    for (int j = 0; j < 8; j++) y[j] = fmaf(xk, __ldg(taps + abs(min(j * T + t, nch - 1) - k)), y[j]);
  };
  if constexpr (T >= 32) {  // a warp's threads are all of the same transform
    const int lane = t % 32;
    for (int k0 = 0; k0 < nch; k0 += 32) {
      const float xv = k0 + lane < nch ? __ldg(x + k0 + lane) : 0.0f;
      for (unsigned m = __ballot_sync(0xffffffffu, xv != 0.0f); m; m &= m - 1u) {
        const int b = __ffs((int)m) - 1;
        add(k0 + b, __shfl_sync(0xffffffffu, xv, b));
      }
    }
  } else {
    for (int k = 0; k < nch; k++) {
      const float xk = __ldg(x + k);
      if (xk != 0.0f) add(k, xk);
    }
  }
#pragma unroll
  for (int j = 0; j < 8; j++) a[j].*row = y[j];
}

// Rows of X [V][nr][nch] -> Y, rows as they are or (TR) in the backprojection
// layout Y[view][channel][nrp]. Rows 2 i and 2 i + 1 of a view are a pair (an
// odd view's last row is alone), so that a row's roundings do not depend on
// where a range of views begins. A CTA holds G transforms at a time and walks
// the pairs with the grid's stride: the twiddles of pass 1 stay in its
// threads' registers.
template <int N, bool TR>
__global__ void __launch_bounds__(N / 16 > FF_THREADS ? N / 16 : FF_THREADS, N / 16 > FF_THREADS ? 2 : 4)
k_filter_fft(const float* __restrict__ X, float* __restrict__ Y, const float* __restrict__ taps,
             const float2* __restrict__ spec, const float2* __restrict__ tw, int V, int nch, int nr, int nrp) {
  constexpr int R2 = FftShape<N>::R2, R3 = FftShape<N>::R3, T = N / 16;
  constexpr int CTA = T > FF_THREADS ? T : FF_THREADS, G = CTA / T;
  constexpr int PAD = R2 > 1 ? R3 : 0, BLK = T + PAD, PLANE = 16 * BLK + (R2 > 1 ? 0 : 16);
  constexpr int NW = CTA / 32;
  static_assert(T == R2 * R3, "N = 16 R2 R3");
  extern __shared__ float sm_fft[];
  __shared__ float2 s_tw2[R2 * R3];       // twiddles of pass 2, [k2][n3]
  __shared__ unsigned s_row[2][2][NW];    // exponents and counts of the pair's rows by warp, two buffers
  const int tid = threadIdx.x, g = tid / T, t = tid % T;
  float* re = sm_fft + (size_t)g * 2 * PLANE;
  float* im = re + PLANE;
  if constexpr (R2 > 1) {
    for (int e = tid; e < R2 * R3; e += CTA) s_tw2[e] = __ldg(tw + 16 * (e / R3) * (e % R3));
  }
  float2 tw1[16];
#pragma unroll
  for (int k = 1; k < 16; k++) tw1[k] = __ldg(tw + t * k);
  __syncthreads();

  const unsigned per_view = (unsigned)(nr + 1) / 2;
  const long pairs = (long)V * per_view, steps = (pairs + G - 1) / G;
  int buf = 0;
  for (long st = blockIdx.x; st < steps; st += gridDim.x, buf ^= 1) {
    const long pair = st * G + g;
    const long v = pairs < (1l << 31) ? (long)((unsigned)pair / per_view) : pair / per_view;
    const int r0 = 2 * (int)(pair - v * per_view);
    const long m = v * nr + r0;  // row of X
    const bool has_a = pair < pairs, has_b = has_a && r0 + 1 < nr;
    // ---- pass 1: points n = n1 T + t, n1 < 8 (the others are padding), minus
    // their left neighbours (from L1)
    float2 a[8];
    const float *xa = X + m * nch, *xb = xa + nch;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int n = j * T + t;
      a[j].x = has_a && n < nch ? __ldg(xa + n) : 0.0f;
      a[j].y = has_b && n < nch ? __ldg(xb + n) : 0.0f;
    }
    unsigned some_a = 0u, some_b = 0u;  // samples that are not 0
#pragma unroll
    for (int j = 0; j < 8; j++) {
      some_a += a[j].x != 0.0f ? 1u : 0u;
      some_b += a[j].y != 0.0f ? 1u : 0u;
    }
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const int n = j * T + t - 1;
      a[j].x -= has_a && n >= 0 && n < nch ? __ldg(xa + n) : 0.0f;
      a[j].y -= has_b && n >= 0 && n < nch ? __ldg(xb + n) : 0.0f;
    }
    unsigned exps = row_exponent<T>(a, &float2::x, some_a);  // row a's + 2^16 row b's, as the counts
    exps |= row_exponent<T>(a, &float2::y, some_b) << 16;
    unsigned some = some_a | some_b << 16;
    if constexpr (T > 32) {
      if (tid % 32 == 0) {
        s_row[buf][0][tid / 32] = exps;
        s_row[buf][1][tid / 32] = some;
      }
      __syncthreads();  // also: the previous step's pass 1' has read its points
      exps = some = 0u;
#pragma unroll
      for (int w = 0; w < T / 32; w++) {
        exps = __vmaxu2(exps, s_row[buf][0][g * (T / 32) + w]);
        some += s_row[buf][1][g * (T / 32) + w];
      }
    } else {
      __syncwarp();
    }
    const unsigned ea = exps & 0xffffu, eb = exps >> 16;  // the same for all threads of the transform
    const unsigned ca = some & 0xffffu, cb = some >> 16;
    // rows that are summed directly
    constexpr unsigned FEW = N > 2048 ? 128u : N > 512 ? 96u : 64u;
    const bool sum_a = ea == FF_OUT || ca - 1u < FEW, sum_b = eb == FF_OUT || cb - 1u < FEW;
    // powers of two: row times 2^(127 - e), result times 2^(e - 127); a row of zeros gives zeros
    const float sa = __uint_as_float((254u - ea) << 23), sb = __uint_as_float((254u - eb) << 23);
    const float ua = ca ? __uint_as_float(ea << 23) : 0.0f, ub = cb ? __uint_as_float(eb << 23) : 0.0f;
#pragma unroll
    for (int j = 0; j < 8; j++) {
      a[j].x = sum_a ? 0.0f : a[j].x * sa;
      a[j].y = sum_b ? 0.0f : a[j].y * sb;
    }
    {
      float2 o[8];
#pragma unroll
      for (int j = 0; j < 8; j++) o[j] = j ? cmul<false>(a[j], w16(j)) : a[j];
      dft8<false>(a);
      dft8<false>(o);
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const float2 e = k ? cmul<false>(a[k], tw1[2 * k]) : a[k], d = cmul<false>(o[k], tw1[2 * k + 1]);
        const int we = fft_word<R2, R3, BLK>(2 * k, t), wd = fft_word<R2, R3, BLK>(2 * k + 1, t);
        re[we] = e.x;
        im[we] = e.y;
        re[wd] = d.x;
        im[wd] = d.y;
      }
    }
    fft_sync<T>();
    // ---- pass 2
    if constexpr (R2 > 1) {
#pragma unroll
      for (int j = 0; j < 16 / R2; j++) {
        const int u = t + T * j, k1 = u / R3, n3 = u % R3;
        float2 v[R2];
#pragma unroll
        for (int k = 0; k < R2; k++) {
          const int w = fft_word<R2, R3, BLK>(k1, k * R3 + n3);
          v[k] = make_float2(re[w], im[w]);
        }
        dft<R2, false>(v);
#pragma unroll
        for (int k = 0; k < R2; k++) {
          const int w = fft_word<R2, R3, BLK>(k1, k * R3 + n3);
          const float2 x = k ? cmul<false>(v[k], s_tw2[k * R3 + n3]) : v[k];
          re[w] = x.x;
          im[w] = x.y;
        }
      }
      fft_sync<T>();
    }
    // ---- pass 3, the spectrum, pass 3 backwards
#pragma unroll
    for (int j = 0; j < 16 / R3; j++) {
      const int b = t + T * j, base = (b / R2) * BLK + (b % R2) * R3;
      const int cx = chunk_xor<R3>(R2 > 1 ? b % R2 : b);
      float2 v[R3];
#pragma unroll
      for (int c = 0; c < R3 / 4; c++) {
        const int w = base + ((4 * c) ^ cx);
        const float4 x = *reinterpret_cast<const float4*>(re + w), y = *reinterpret_cast<const float4*>(im + w);
        v[4 * c] = make_float2(x.x, y.x);
        v[4 * c + 1] = make_float2(x.y, y.y);
        v[4 * c + 2] = make_float2(x.z, y.z);
        v[4 * c + 3] = make_float2(x.w, y.w);
      }
      dft<R3, false>(v);
#pragma unroll
      for (int k = 0; k < R3; k += 2) {
        const float4 h = __ldg(reinterpret_cast<const float4*>(spec + b * R3 + k));
        v[k] = cmul<false>(v[k], make_float2(h.x, h.y));
        v[k + 1] = cmul<false>(v[k + 1], make_float2(h.z, h.w));
      }
      dft<R3, true>(v);
#pragma unroll
      for (int c = 0; c < R3 / 4; c++) {
        const int w = base + ((4 * c) ^ cx);
        *reinterpret_cast<float4*>(re + w) = make_float4(v[4 * c].x, v[4 * c + 1].x, v[4 * c + 2].x, v[4 * c + 3].x);
        *reinterpret_cast<float4*>(im + w) = make_float4(v[4 * c].y, v[4 * c + 1].y, v[4 * c + 2].y, v[4 * c + 3].y);
      }
    }
    fft_sync<T>();
    // ---- pass 2 backwards
    if constexpr (R2 > 1) {
#pragma unroll
      for (int j = 0; j < 16 / R2; j++) {
        const int u = t + T * j, k1 = u / R3, n3 = u % R3;
        float2 v[R2];
#pragma unroll
        for (int k = 0; k < R2; k++) {
          const int w = fft_word<R2, R3, BLK>(k1, k * R3 + n3);
          const float2 x = make_float2(re[w], im[w]);
          v[k] = k ? cmul<true>(x, s_tw2[k * R3 + n3]) : x;
        }
        dft<R2, true>(v);
#pragma unroll
        for (int k = 0; k < R2; k++) {
          const int w = fft_word<R2, R3, BLK>(k1, k * R3 + n3);
          re[w] = v[k].x;
          im[w] = v[k].y;
        }
      }
      fft_sync<T>();
    }
    // ---- pass 1 backwards: the samples n < N / 2
    {
      float2 o[8];
#pragma unroll
      for (int k = 0; k < 8; k++) {
        const int we = fft_word<R2, R3, BLK>(2 * k, t), wd = fft_word<R2, R3, BLK>(2 * k + 1, t);
        const float2 e = make_float2(re[we], im[we]), d = make_float2(re[wd], im[wd]);
        a[k] = k ? cmul<true>(e, tw1[2 * k]) : e;
        o[k] = cmul<true>(d, tw1[2 * k + 1]);
      }
      dft8<true>(a);
      dft8<true>(o);
#pragma unroll
      for (int j = 0; j < 8; j++) {
        a[j] = cadd(a[j], j ? cmul<true>(o[j], w16(j)) : o[j]);
        a[j].x *= ua;
        a[j].y *= ub;
      }
    }
    if (sum_a && has_a) direct_sum<T>(xa, taps, nch, t, a, &float2::x);
    if (sum_b && has_b) direct_sum<T>(xb, taps, nch, t, a, &float2::y);
    if constexpr (TR) {
      float* y = Y + (size_t)v * nch * nrp + r0;  // nrp is a multiple of 4, r0 even
      const bool both = has_b && (reinterpret_cast<uintptr_t>(Y) & 7) == 0;  // Y may be at any float
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int n = j * T + t;
        if (n < nch && both) {
          *reinterpret_cast<float2*>(y + (size_t)n * nrp) = a[j];
        } else if (n < nch) {
          if (has_a) y[(size_t)n * nrp] = a[j].x;
          if (has_b) y[(size_t)n * nrp + 1] = a[j].y;
        }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; j++) {
        const int n = j * T + t;
        if (n < nch && has_a) Y[m * nch + n] = a[j].x;
        if (n < nch && has_b) Y[(m + 1) * nch + n] = a[j].y;
      }
    }
    if constexpr (T <= 32) __syncwarp();  // pass 1' has read its points before the next step's pass 1 writes
  }
}

// tw[j] = exp(-2 pi i j / N), rounded from FP64.
__global__ void __launch_bounds__(256) k_filter_twiddles(int N, float2* __restrict__ tw) {
  const int j = blockIdx.x * 256 + threadIdx.x;
  double s, c;
  sincospi(-2.0 * (double)j / (double)N, &s, &c);
  tw[j] = make_float2((float)c, (float)s);
}

// A[f] / N, the spectrum of the running sums a of the symmetric taps. a's
// differences are h inside the window [-nch, nch) and -S / 2 at both its ends
// (S = H[0], the sum of all taps), so with w = 2 pi f / N and
// H[f] = h[0] + 2 sum_d h[d] cos(w d)
//   A[f] = (H[f] - S cos(w nch)) / (1 - exp(-i w)),  A[0] = 0,
// in FP64, stored at the place pass 3 has frequency f in: f = k1 + 16 k2 +
// 16 R2 k3 at (k1 R2 + k2) R3 + k3. One warp per frequency f <= N / 2
// (A[N - f] is its conjugate).
__global__ void __launch_bounds__(256)
k_filter_spectrum(const float* __restrict__ taps, int nch, int N, int R2, int R3, float2* __restrict__ spec) {
  const int f = blockIdx.x * 8 + threadIdx.x / 32, lane = threadIdx.x % 32;
  if (f > N / 2) return;
  const double step = 2.0 / (double)N;
  double acc = 0.0, sum = 0.0;
  for (int d = lane; d < nch; d += 32) {
    const int j = (int)(((long)f * d) % N);
    const double h = (d ? 2.0 : 1.0) * (double)__ldg(taps + d);
    acc += h * cospi((double)j * step);
    sum += h;
  }
  for (int o = 16; o > 0; o >>= 1) {
    acc += __shfl_xor_sync(0xffffffffu, acc, o);
    sum += __shfl_xor_sync(0xffffffffu, sum, o);
  }
  if (lane < 2) {
    // 1 / (1 - exp(-i w)) = (sin(w / 2) - i cos(w / 2)) / (2 sin(w / 2))
    double re = 0.0, im = 0.0;
    if (f) {
      const double num = (acc - sum * cospi((double)(((long)f * nch) % N) * step)) / (double)N;
      double s, c;
      sincospi((double)f / (double)N, &s, &c);
      re = 0.5 * num;
      im = -0.5 * num * c / s;
    }
    const int ff = lane ? (N - f) % N : f;
    const int k1 = ff % 16, k2 = (ff / 16) % R2, k3 = ff / (16 * R2);
    spec[(k1 * R2 + k2) * R3 + k3] = make_float2((float)re, (float)(lane ? -im : im));
  }
}

template <int N, bool TR>
cudaError_t launch_n(const float* x, float* y, const float* taps, const float2* spec, const float2* tw, int V,
                     int nch, int nr, int nrp, cudaStream_t s) {
  constexpr int R2 = FftShape<N>::R2, R3 = FftShape<N>::R3, T = N / 16;
  constexpr int CTA = T > FF_THREADS ? T : FF_THREADS, G = CTA / T;
  constexpr int PLANE = 16 * (T + (R2 > 1 ? R3 : 0)) + (R2 > 1 ? 0 : 16);
  constexpr int smem = G * 2 * PLANE * (int)sizeof(float);
  auto kern = k_filter_fft<N, TR>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 0, per_sm = 1;
  if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
  if ((e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, CTA, smem)) != cudaSuccess) return e;
  const long steps = ((long)V * ((nr + 1) / 2) + G - 1) / G;
  const unsigned grid = (unsigned)std::max(1L, std::min<long>(steps, (long)sms * std::max(per_sm, 1)));
  kern<<<grid, CTA, smem, s>>>(x, y, taps, spec, tw, V, nch, nr, nrp);
  return cudaGetLastError();
}

template <bool TR>
cudaError_t launch_by_size(const float* x, float* y, const float* taps, const float2* spec, const float2* tw, int N,
                           int V, int nch, int nr, int nrp, cudaStream_t s) {
  switch (N) {
    case 256: return launch_n<256, TR>(x, y, taps, spec, tw, V, nch, nr, nrp, s);
    case 512: return launch_n<512, TR>(x, y, taps, spec, tw, V, nch, nr, nrp, s);
    case 1024: return launch_n<1024, TR>(x, y, taps, spec, tw, V, nch, nr, nrp, s);
    case 2048: return launch_n<2048, TR>(x, y, taps, spec, tw, V, nch, nr, nrp, s);
    case 4096: return launch_n<4096, TR>(x, y, taps, spec, tw, V, nch, nr, nrp, s);
  }
  return cudaErrorInvalidValue;
}

void fft_radices(int N, int* r2, int* r3) {
  *r2 = N == 256 ? 1 : N == 512 ? 8 : 16;
  *r3 = N / (16 * *r2);
}

}  // namespace

int filter_fft_size(int nch) {
  for (int n = 256; n <= 4096; n *= 2)
    if (nch < n / 2) return n;
  return 0;
}

cudaError_t launch_filter_twiddles(int N, float2* tw, cudaStream_t s) {
  k_filter_twiddles<<<(unsigned)(N / 256), 256, 0, s>>>(N, tw);
  return cudaGetLastError();
}

cudaError_t launch_filter_spectrum(const float* d_taps, int nch, int N, float2* spec, cudaStream_t s) {
  int r2, r3;
  fft_radices(N, &r2, &r3);
  k_filter_spectrum<<<(unsigned)((N / 2 + 1 + 7) / 8), 256, 0, s>>>(d_taps, nch, N, r2, r3, spec);
  return cudaGetLastError();
}

cudaError_t launch_filter_fft(const float* x, float* y, const float* d_taps, const float2* spec, const float2* tw, int N,
                              int V, int nch, int nr, int nrp, bool transposed, cudaStream_t s) {
  if (nch >= N / 2 || V < 1) return cudaErrorInvalidValue;
  return transposed ? launch_by_size<true>(x, y, d_taps, spec, tw, N, V, nch, nr, nrp, s)
                    : launch_by_size<false>(x, y, d_taps, spec, tw, N, V, nch, nr, nrp, s);
}
