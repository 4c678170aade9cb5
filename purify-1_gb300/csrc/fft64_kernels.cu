// FP64 row and column passes of the padded-grid FFT (declared in fft_kernels.h).
//
// Bound by FP64 arithmetic (about 8 warp instructions a clock on the whole
// chip), so the passes do only the work that is needed: rows y0 ... y0+Ny-1 in
// the row pass, with Z S or S^H Z^H in its loads or stores, and radix-16 stages
// with every twiddle from a table (a third of the operations of radix-2
// stages).
// Measured on a 1024^2 grid, image 512^2 (us, cold caches): rows 43, columns 74
// (FP64 pipe 80% busy), against cuFFT's 2-D plan, 88 + 90, with a pad or crop of
// 5: pair of J = 6 1,204 -> 1,071.
// A pass neither starts before the kernel ahead of it is done nor lets the next
// one start early.  CTAs that come in early crowd onto the SMs that have room:
// with both, the pair above took 1,177 us (the gridding kernels run in order of
// decreasing work), and Phi^H of 2,000 visibilities at 256^2 84 instead of 54.
// A thread holds one radix-16 butterfly, or as many smaller ones as make 16
// values, in registers; a CTA holds 16 values a thread in shared memory between
// stages.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "device_kernels.h"
#include "fft_kernels.h"
#include "gridding_device.cuh"

namespace pg {
namespace {

// Values of one thread, and the stage radix: 16 while it divides what is left.
constexpr int kVals = 16;
template <int N, int Ns>
struct Radix64 {
  static constexpr int value = (N / Ns) % 16 == 0 ? 16 : N / Ns;
};
// Threads and lines per CTA.  Small CTAs even out the load of the SMs, whose
// FP64 units are what a pass waits for; a column pass takes two columns at
// least, a whole 32-byte sector of each row.
constexpr int line_threads(int N, bool cols) {
  return cols ? (N / 8 > 64 ? N / 8 : 64) : (N / 16 > 64 ? N / 16 : 64);
}
template <int N, bool COLS>
struct Lines {
  static constexpr int T = line_threads(N, COLS);
  static constexpr int V = T * kVals / N;
  // one 16-byte piece of padding in 16; the lines of a column pass 8 / V
  // pieces of the banks apart
  static constexpr int raw = N + N / 16;
  static constexpr int pad = COLS && V <= 8 ? (8 / V - raw % 8 + 8) % 8 : 0;
  static constexpr int stride = raw + pad;
  static constexpr size_t smem = sizeof(double2) * size_t(V) * stride;
};

__device__ __forceinline__ double2 cadd(double2 a, double2 b) {
  return make_double2(a.x + b.x, a.y + b.y);
}
__device__ __forceinline__ double2 csub(double2 a, double2 b) {
  return make_double2(a.x - b.x, a.y - b.y);
}
__device__ __forceinline__ double2 cmul64(double2 a, double2 w) {
  return make_double2(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
}
// v exp(-+ 2 pi i E / 16)
template <int E, bool INV>
__device__ __forceinline__ double2 root16(double2 v) {
  constexpr double c1 = 0.92387953251128675613, s1 = 0.38268343236508977173;
  constexpr double h = 0.70710678118654752440;
  if constexpr (E == 0) return v;
  if constexpr (E == 4) return INV ? make_double2(-v.y, v.x) : make_double2(v.y, -v.x);
  if constexpr (E == 2)
    return INV ? make_double2(h * (v.x - v.y), h * (v.x + v.y))
               : make_double2(h * (v.x + v.y), h * (v.y - v.x));
  if constexpr (E == 6)
    return INV ? make_double2(-h * (v.x + v.y), h * (v.x - v.y))
               : make_double2(h * (v.y - v.x), -h * (v.x + v.y));
  constexpr double c = E == 1 ? c1 : E == 3 ? s1 : -c1;
  constexpr double s = E == 1 ? -s1 : E == 3 ? -c1 : s1;  // forward
  return cmul64(v, make_double2(c, INV ? -s : s));
}
__device__ __forceinline__ void dft2(double2 &a, double2 &b) {
  const double2 t = csub(a, b);
  a = cadd(a, b);
  b = t;
}
template <bool INV>
__device__ __forceinline__ void dft4(double2 &a, double2 &b, double2 &c, double2 &d) {
  dft2(a, c);
  dft2(b, d);
  d = root16<4, INV>(d);
  dft2(a, b);
  dft2(c, d);
  const double2 t = b;  // natural order: a, c, b, d
  b = c;
  c = t;
}
// R-point transform in registers; output k is left at v[place<R>(k)].
template <int R>
__device__ __forceinline__ constexpr int place(int k) {
  return R == 16 ? 4 * (k % 4) + k / 4 : R == 8 ? 2 * (k % 4) + k / 4 : k;
}
template <int R, bool INV>
__device__ __forceinline__ void dft64(double2 *v) {
  if constexpr (R == 2) dft2(v[0], v[1]);
  if constexpr (R == 4) dft4<INV>(v[0], v[1], v[2], v[3]);
  if constexpr (R == 8) {
    dft4<INV>(v[0], v[2], v[4], v[6]);
    dft4<INV>(v[1], v[3], v[5], v[7]);
    v[3] = root16<2, INV>(v[3]);
    v[5] = root16<4, INV>(v[5]);
    v[7] = root16<6, INV>(v[7]);
#pragma unroll
    for (int p = 0; p < 4; ++p) dft2(v[2 * p], v[2 * p + 1]);
  }
  if constexpr (R == 16) {
#pragma unroll
    for (int q = 0; q < 4; ++q) dft4<INV>(v[q], v[q + 4], v[q + 8], v[q + 12]);
    v[5] = root16<1, INV>(v[5]);
    v[6] = root16<2, INV>(v[6]);
    v[7] = root16<3, INV>(v[7]);
    v[9] = root16<2, INV>(v[9]);
    v[10] = root16<4, INV>(v[10]);
    v[11] = root16<6, INV>(v[11]);
    v[13] = root16<3, INV>(v[13]);
    v[14] = root16<6, INV>(v[14]);
    v[15] = root16<9, INV>(v[15]);
#pragma unroll
    for (int p = 0; p < 4; ++p) dft4<INV>(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
  }
}

// Global loads and stores of the first and last stages: element n of line
// l0 + l.  Columns: rows y0 ... y0+Ny-1 alone are read (forward; the others
// are zero) or written (inverse).  Rows: forward reads the image, with the
// corrections, inverse writes it.  The loads go past L1: each value is read
// once, and the inverse column pass works in place, so nothing may be taken
// for read-only data.
template <bool COLS, bool INV>
__device__ __forceinline__ double2 load64(const Fft64Args &a, const double2 *in,
                                          int line, int n) {
  if constexpr (COLS) {
    if (!INV && (n < a.y0 || n >= a.y0 + a.Ny)) return make_double2(0, 0);
    return __ldcg(in + size_t(n) * a.Nu + line);
  } else {
    if (line >= a.Ny) return make_double2(0, 0);
    if constexpr (INV) return __ldcg(in + size_t(a.y0 + line) * a.Nu + n);
    const int i = n - a.x0;
    if (i < 0 || i >= a.Nx) return make_double2(0, 0);
    const double2 x = __ldcg(in + size_t(line) * a.Nx + i);
    const double s = a.su[i] * a.sv[line];
    return make_double2(s * x.x, s * x.y);
  }
}
template <bool COLS, bool INV>
__device__ __forceinline__ void store64(const Fft64Args &a, double2 *out, int line,
                                        int n, double2 x) {
  if constexpr (COLS) {
    if (!INV || (n >= a.y0 && n < a.y0 + a.Ny)) out[size_t(n) * a.Nu + line] = x;
  } else {
    if (line >= a.Ny) return;
    if constexpr (!INV) {
      out[size_t(a.y0 + line) * a.Nu + n] = x;
    } else {
      const int i = n - a.x0;
      if (i < 0 || i >= a.Nx) return;
      const double s = a.su[i] * a.sv[line];
      out[size_t(line) * a.Nx + i] = make_double2(s * x.x, s * x.y);
    }
  }
}

template <int N, bool COLS, bool INV, int Ns>
__device__ __forceinline__ void stage64(const Fft64Args &a, const double2 *in, double2 *out,
                                        double2 *sm, const double2 *__restrict__ tw, int line0) {
  using L = Lines<N, COLS>;
  constexpr int R = Radix64<N, Ns>::value, R0 = Radix64<N, 1>::value, Q = kVals / R, P = N / R;
  constexpr bool FIRST = Ns == 1, LAST = Ns * R == N;
  // the line fastest where a column pass meets global memory
  constexpr bool FAST = COLS && (FIRST || LAST);
  double2 v[Q][R];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int flat = int(threadIdx.x) + q * L::T;
    const int l = FAST ? flat % L::V : flat / P, j = FAST ? flat / L::V : flat % P;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int n = j + r * P;
      if constexpr (FIRST)
        v[q][r] = load64<COLS, INV>(a, in, line0 + l, n);
      else
        v[q][r] = sm[l * L::stride + n + n / 16];
    }
  }
  if constexpr (!FIRST) __syncthreads();  // every read of this stage is done
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const int flat = int(threadIdx.x) + q * L::T;
    const int l = FAST ? flat % L::V : flat / P, j = FAST ? flat / L::V : flat % P;
    const int k = j % Ns;
    if constexpr (!FIRST) {
#pragma unroll
      for (int r = 1; r < R; ++r) {
        double2 w = __ldg(tw + (Ns - R0) + (r - 1) * Ns + k);
        if (INV) w.y = -w.y;
        v[q][r] = cmul64(v[q][r], w);
      }
    }
    dft64<R, INV>(v[q]);
    const int d = (j / Ns) * Ns * R + k;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int n = d + r * Ns;
      if constexpr (LAST)
        store64<COLS, INV>(a, out, line0 + l, n, v[q][place<R>(r)]);
      else
        sm[l * L::stride + n + n / 16] = v[q][place<R>(r)];
    }
  }
  if constexpr (!LAST) {
    __syncthreads();
    stage64<N, COLS, INV, Ns * R>(a, in, out, sm, tw, line0);
  }
}

// One pass: `in` and `out` may be the same grid in a column pass (a CTA reads
// its columns before it writes them).
template <int N, bool COLS, bool INV>
__global__ void __launch_bounds__(Lines<N, COLS>::T, 512 / Lines<N, COLS>::T)
    fft64_kernel(const Fft64Args a, const double2 *in, double2 *out) {
  extern __shared__ double2 fft64_sm[];
  stage64<N, COLS, INV, 1>(a, in, out, fft64_sm,
                           static_cast<const double2 *>(COLS ? a.tw_v : a.tw_u),
                           int(blockIdx.x) * Lines<N, COLS>::V);
}

template <int N, bool COLS, bool INV>
cudaError_t launch64(const Fft64Args &a, const void *in, void *out, cudaStream_t s) {
  using L = Lines<N, COLS>;
  auto fn = fft64_kernel<N, COLS, INV>;
  if (L::smem > 48 * 1024) {
    const cudaError_t e =
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(L::smem));
    if (e != cudaSuccess) return e;
  }
  const int lines = COLS ? a.Nu : a.Ny;
  fn<<<(lines + L::V - 1) / L::V, L::T, L::smem, s>>>(a, static_cast<const double2 *>(in),
                                                      static_cast<double2 *>(out));
  return cudaGetLastError();
}

template <bool COLS, bool INV>
cudaError_t launch64_n(const Fft64Args &a, const void *in, void *out, cudaStream_t s) {
  switch (COLS ? a.Nv : a.Nu) {
    case 128: return launch64<128, COLS, INV>(a, in, out, s);
    case 256: return launch64<256, COLS, INV>(a, in, out, s);
    case 512: return launch64<512, COLS, INV>(a, in, out, s);
    case 1024: return launch64<1024, COLS, INV>(a, in, out, s);
    case 2048: return launch64<2048, COLS, INV>(a, in, out, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace

// Below 128 a pass is a few CTAs' latency: Phi at 64^2 39.2 us, cuFFT's plan 37.2
// (128^2: 35.1 and 43.3).
bool fft64_supported(int Nu, int Nv) {
  for (int n : {Nu, Nv})
    if (n < 128 || n > 2048 || (n & (n - 1)) != 0) return false;
  return true;
}

std::vector<double> fft64_twiddle_table(int N) {
  std::vector<double> t(2 * size_t(N), 0.0);
  auto radix = [&](int Ns) { return (N / Ns) % 16 == 0 ? 16 : N / Ns; };  // Radix64
  for (int Ns = radix(1); Ns < N; Ns *= radix(Ns))
    for (int r = 1; r < radix(Ns); ++r)
      for (int k = 0; k < Ns; ++k) {
        const double ang = -2.0 * M_PI * double(r) * double(k) / (double(Ns) * radix(Ns));
        const size_t e = 2 * (size_t(Ns - radix(1)) + size_t(r - 1) * Ns + k);
        t[e] = std::cos(ang);
        t[e + 1] = std::sin(ang);
      }
  return t;
}

cudaError_t launch_fft64_forward(const Fft64Args &a, const void *x, void *pad, void *work,
                                 cudaStream_t s) {
  if (!fft64_supported(a.Nu, a.Nv) || a.Nx <= 0 || a.Ny <= 0 || a.x0 < 0 || a.y0 < 0 ||
      a.x0 + a.Nx > a.Nu || a.y0 + a.Ny > a.Nv)
    return cudaErrorInvalidValue;
  const cudaError_t e = launch64_n<false, false>(a, x, pad, s);
  return e != cudaSuccess ? e : launch64_n<true, false>(a, pad, work, s);
}

cudaError_t launch_fft64_inverse(const Fft64Args &a, void *work, void *x, cudaStream_t s) {
  if (!fft64_supported(a.Nu, a.Nv) || a.Nx <= 0 || a.Ny <= 0 || a.x0 < 0 || a.y0 < 0 ||
      a.x0 + a.Nx > a.Nu || a.y0 + a.Ny > a.Nv)
    return cudaErrorInvalidValue;
  const cudaError_t e = launch64_n<true, true>(a, work, work, s);
  return e != cudaSuccess ? e : launch64_n<false, true>(a, work, x, s);
}

}  // namespace pg
