// RecursiveGaussianFilter / RecursiveGaussianAxisFilter
// (src/filters/recursive_gaussian.rs): the Young & van Vliet 3rd-order IIR
// approximation of the Gaussian.  The reference converts the whole largest
// region to f64 (P::to_f64), runs on every line along each axis a causal then
// an anticausal pass in place (recursive_gaussian.rs:56-130), and converts the
// requested region back (P::from_f64).  Here:
//   k_rec_lines  one thread per line: the causal pass, then the anticausal pass,
//                in an f64 scratch image; the first axis' kernel converts as it
//                reads the input, the last one's as it writes the requested
//                region (f32: round to nearest; u8: round half away from zero,
//                clamp to [0, 255], NaN -> 0)
//   k_rec_copy   conversions alone: the requested region where no axis is
//                filtered, and both ways around the passes of a few lines
// Reference rounding rounds every product and sum separately in the
// reference's order, bit for bit; FMA rounding uses fused multiply-adds (f64
// throughout either way: an f32 recursion drifts past 1e-5 of the reference
// once sigma reaches a few pixels).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "internal.hpp"
#include "pixel.cuh"

namespace itkg {
namespace {

constexpr int kT = 256;

struct RecGeom {
  int64_t n[3];        // largest region size (1 on missing axes)
  int64_t lo[3];       // largest region index
};

// An input or output image seen from the largest region: byte strides per axis,
// the address of the largest region's first voxel.
struct RecImage {
  char* at;
  int64_t p[3];
  int32_t dtype;
  int32_t pad_;
};

__device__ __forceinline__ double rec_read(const char* p, int dtype) {  // exact for every input type
  switch (dtype) {
    case ITKG_F32: return (double)*reinterpret_cast<const float*>(p);
    case ITKG_I16: return (double)to_f32(*reinterpret_cast<const int16_t*>(p));
    case ITKG_U8: return (double)to_f32(*reinterpret_cast<const uint8_t*>(p));
    case ITKG_BF16: return (double)to_f32(*reinterpret_cast<const __nv_bfloat16*>(p));
    default: return (double)to_f32(*reinterpret_cast<const __half*>(p));
  }
}

// v = B x + a1 y[-1] + a2 y[-2] + a3 y[-3]
template <bool REF>
__device__ __forceinline__ double rec_step(double x, double y1, double y2, double y3, double B, double a1,
                                           double a2, double a3) {
  if constexpr (REF) {
    // (((B x) + a1 y1) + a2 y2) + a3 y3, each product and sum rounded (recursive_gaussian.rs:63)
    double v = __dadd_rn(__dmul_rn(B, x), __dmul_rn(a1, y1));
    v = __dadd_rn(v, __dmul_rn(a2, y2));
    return __dadd_rn(v, __dmul_rn(a3, y3));
  } else {
    return fma(a3, y3, fma(a2, y2, fma(a1, y1, __dmul_rn(B, x))));
  }
}

__device__ __forceinline__ float out_f32(double v) { return __double2float_rn(v); }
__device__ __forceinline__ uint8_t out_u8_of(double v) {  // round half away from zero, clamp, NaN -> 0
  double r = round(v);
  r = fmin(fmax(r, 0.0), 255.0);
  return (uint8_t)r;
}

__device__ __forceinline__ void rec_write(char* p, int dtype, double v) {
  if (dtype == ITKG_U8) *reinterpret_cast<uint8_t*>(p) = out_u8_of(v);
  else *reinterpret_cast<float*>(p) = out_f32(v);
}

struct RecLines {
  RecGeom g;
  double* d;            // scratch: sample (x, y, z) at (z n1 + y) pitch + x
  int64_t pitch;        // doubles per row; even where rows are filtered (16-byte accesses)
  int32_t axis;
  int32_t pad_;
  RecImage in, out;     // FIRST / LAST
  int64_t in_step, out_step;  // their strides along the axis
  int64_t w0, w1;       // LAST: the requested samples of a line
  int64_t lo[3], hi[3]; // LAST: the requested region, from the largest one's first voxel
  double B, a1, a2, a3;
};

// Four samples of a line, p[0], p[s], ...; CONTIG: s = 1 and p on a 16-byte
// boundary.  n: how many exist (the rest repeat the last one that does).
template <bool CONTIG>
__device__ __forceinline__ void rec_load4(const double* p, int64_t s, int n, double (&v)[4]) {
  if (CONTIG && n == 4) {
    const double2 a = *reinterpret_cast<const double2*>(p), b = *reinterpret_cast<const double2*>(p + 2);
    v[0] = a.x, v[1] = a.y, v[2] = b.x, v[3] = b.y;
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = p[min(k, n - 1) * s];
  }
}

template <bool CONTIG>
__device__ __forceinline__ void rec_store4(double* p, int64_t s, int n, const double (&v)[4]) {
  if (CONTIG && n == 4) {
    *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
    *reinterpret_cast<double2*>(p + 2) = make_double2(v[2], v[3]);
  } else {
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (k < n) p[k * s] = v[k];
  }
}

// One line per thread.  axis 0: lines are rows (CONTIG); axis 1: stride pitch;
// axis 2: stride n1 pitch.  I: the type that counts a line's samples; 64 bits
// only for lines beyond 2^30 (256^3, three axes, reference and FMA rounding: 1501
// and 871 us in 32 bits, 1580 and 1053 in 64).
template <typename I, bool REF, bool FIRST, bool LAST, bool CONTIG>
__global__ void __launch_bounds__(32) k_rec_lines(const __grid_constant__ RecLines a) {
  const int64_t L = (int64_t)blockIdx.x * 32 + threadIdx.x;
  const int64_t n0 = a.g.n[0], n1 = a.g.n[1], n2 = a.g.n[2];
  int64_t c[3] = {0, 0, 0};  // the line's first voxel
  if (CONTIG) {
    c[1] = L % n1, c[2] = L / n1;
  } else {
    const int64_t q = L / n0;
    c[0] = L - q * n0, c[1] = a.axis == 1 ? 0 : q, c[2] = a.axis == 1 ? q : 0;
  }
  if (CONTIG ? L >= n1 * n2 : L >= n0 * (a.axis == 1 ? n2 : n1)) return;
  const I n = (I)(CONTIG ? n0 : a.axis == 1 ? n1 : n2);
  const int64_t s = CONTIG ? 1 : a.axis == 1 ? a.pitch : a.pitch * n1;
  double* const p = a.d + (c[2] * n1 + c[1]) * a.pitch + c[0];
  const int64_t is = a.in_step, os = a.out_step;
  const char* const ip = FIRST ? a.in.at + c[0] * a.in.p[0] + c[1] * a.in.p[1] + c[2] * a.in.p[2] : nullptr;
  char* const op = LAST ? a.out.at + c[0] * a.out.p[0] + c[1] * a.out.p[1] + c[2] * a.out.p[2] : nullptr;
  I w0 = 0, w1 = 0;  // samples to write
  if (LAST) {
    bool in = true;
#pragma unroll
    for (int d = 0; d < 3; ++d) in = in && (d == a.axis || (c[d] >= a.lo[d] && c[d] < a.hi[d]));
    if (in) w0 = (I)a.w0, w1 = (I)a.w1;
  }
  auto read = [&](I i, double (&v)[4]) {  // samples i .. i + 3 of the axis' input
    const int m = (int)min((I)4, n - i);
    if constexpr (FIRST) {
#pragma unroll
      for (int k = 0; k < 4; ++k) v[k] = rec_read(ip + (int64_t)(i + min(k, m - 1)) * is, a.in.dtype);
    } else {
      rec_load4<CONTIG>(p + i * s, s, m, v);
    }
  };
  double v[4], nx[4];
  read(0, v);
  double y1 = v[0], y2 = y1, y3 = y1;  // steady state of the first sample
  for (I i = 0; i < n; i += 4) {
    if (i + 4 < n) read(i + 4, nx);
    const int m = (int)min((I)4, n - i);
    double o[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (k < m) {
        o[k] = rec_step<REF>(v[k], y1, y2, y3, a.B, a.a1, a.a2, a.a3);
        y3 = y2;
        y2 = y1;
        y1 = o[k];
      } else {
        o[k] = 0.0;
      }
      v[k] = nx[k];
    }
    rec_store4<CONTIG>(p + i * s, s, m, o);
  }
  // backwards from the steady state of the last causal sample (y1), the last
  // group first
  y2 = y1;
  y3 = y1;
  const I top = (n - 1) / 4 * 4;
  rec_load4<CONTIG>(p + top * s, s, (int)(n - top), v);
  for (I i = top; i >= 0; i -= 4) {
    if (i >= 4) rec_load4<CONTIG>(p + (i - 4) * s, s, 4, nx);
    const int m = (int)min((I)4, n - i);
    double o[4];
#pragma unroll
    for (int k = 3; k >= 0; --k) {
      if (k < m) {
        o[k] = rec_step<REF>(v[k], y1, y2, y3, a.B, a.a1, a.a2, a.a3);
        y3 = y2;
        y2 = y1;
        y1 = o[k];
      } else {
        o[k] = 0.0;
      }
      v[k] = nx[k];
    }
    if constexpr (LAST) {
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (i + k >= w0 && i + k < w1) rec_write(op + (int64_t)(i + k) * os, a.out.dtype, o[k]);
    } else {
      rec_store4<CONTIG>(p + i * s, s, m, o);
    }
  }
}

using RecFn = void (*)(const RecLines);
template <typename I>
const RecFn kRecFns[2][2][2][2] = {  // [ref][first][last][axis 0]
    {{{k_rec_lines<I, false, false, false, false>, k_rec_lines<I, false, false, false, true>},
      {k_rec_lines<I, false, false, true, false>, k_rec_lines<I, false, false, true, true>}},
     {{k_rec_lines<I, false, true, false, false>, k_rec_lines<I, false, true, false, true>},
      {k_rec_lines<I, false, true, true, false>, k_rec_lines<I, false, true, true, true>}}},
    {{{k_rec_lines<I, true, false, false, false>, k_rec_lines<I, true, false, false, true>},
      {k_rec_lines<I, true, false, true, false>, k_rec_lines<I, true, false, true, true>}},
     {{k_rec_lines<I, true, true, false, false>, k_rec_lines<I, true, true, false, true>},
      {k_rec_lines<I, true, true, true, false>, k_rec_lines<I, true, true, true, true>}}}};
constexpr int64_t kMaxInt32Line = 1 << 30;  // i + 4 stays below 2^31

// Samples r .. r + m - 1 of the largest region, converted: between the images
// where no axis is filtered, to and from scratch (kRecF64) where conversions
// stay out of the line kernels.
constexpr int kRecF64 = -1;
__global__ void __launch_bounds__(kT) k_rec_copy(RecImage in, RecImage out, int64_t r0, int64_t r1, int64_t r2, int64_t m0,
                                                  int64_t m1, int64_t m2) {
  const int64_t i = (int64_t)blockIdx.x * kT + threadIdx.x;
  if (i >= m0) return;
  for (int64_t k = blockIdx.z; k < m2; k += gridDim.z)
    for (int64_t j = blockIdx.y; j < m1; j += gridDim.y) {
      const char* const p = in.at + (r0 + i) * in.p[0] + (r1 + j) * in.p[1] + (r2 + k) * in.p[2];
      char* const q = out.at + (r0 + i) * out.p[0] + (r1 + j) * out.p[1] + (r2 + k) * out.p[2];
      const double v = in.dtype == kRecF64 ? *reinterpret_cast<const double*>(p) : rec_read(p, in.dtype);
      if (out.dtype == kRecF64) *reinterpret_cast<double*>(q) = v;
      else rec_write(q, out.dtype, v);
    }
}

// The derivative users (edges.rs:686-950): stencils on the smoothed image `s`
// (a dense image of the requested region, m0 x m1 x m2, in the input's pixel
// type), clamped to that region, in f64 with every operation rounded in the
// reference's order.  kind: 0 gradient magnitude, 1 Laplacian, 2 derivative
// (axis, order), 3 gradient (one f32 component per axis), 4 2-D Hessian
// (f32 components h00, h11, h01).
template <typename Tp>
__device__ __forceinline__ double sval(const Tp* s, int64_t m0, int64_t m1, int64_t x, int64_t y, int64_t z) {
  return (double)s[(z * m1 + y) * m0 + x];
}

template <typename Tp>
__global__ void __launch_bounds__(kT) k_rec_deriv(const Tp* s, int64_t m0, int64_t m1, int64_t m2, int D, int kind,
                                                   int axis, int order, double h0, double h1, double h2, char* dst,
                                                   int64_t dp0, int64_t dp1, int64_t dp2, int out_u8) {
  const int64_t x = (int64_t)blockIdx.x * kT + threadIdx.x;
  if (x >= m0) return;
  const int64_t m[3] = {m0, m1, m2};
  const double h[3] = {h0, h1, h2};
  for (int64_t z = blockIdx.z; z < m2; z += gridDim.z)
    for (int64_t y = blockIdx.y; y < m1; y += gridDim.y) {
      const int64_t p[3] = {x, y, z};
      // s at p with coordinate a moved by off, clamped to the region
      auto get = [&](int a, int off) {
        int64_t q[3] = {p[0], p[1], p[2]};
        q[a] = q[a] + off < 0 ? 0 : (q[a] + off >= m[a] ? m[a] - 1 : q[a] + off);
        return sval(s, m0, m1, q[0], q[1], q[2]);
      };
      auto first = [&](int a) {  // (s[+1] - s[-1]) / (2 h)
        return __ddiv_rn(__dsub_rn(get(a, 1), get(a, -1)), __dmul_rn(2.0, h[a]));
      };
      auto second = [&](int a) {  // ((s[+1] - 2 s[0]) + s[-1]) / (h h)
        return __ddiv_rn(__dadd_rn(__dsub_rn(get(a, 1), __dmul_rn(2.0, get(a, 0))), get(a, -1)),
                         __dmul_rn(h[a], h[a]));
      };
      char* const o = dst + x * dp0 + y * dp1 + z * dp2;
      if (kind <= 2) {
        double v = 0.0;
        if (kind == 0) {
          for (int a = 0; a < D; ++a) {
            const double d = first(a);
            v = __dadd_rn(v, __dmul_rn(d, d));
          }
          v = __dsqrt_rn(v);
        } else if (kind == 1) {
          for (int a = 0; a < D; ++a) v = __dadd_rn(v, second(a));
        } else {
          v = order == 1 ? first(axis) : (order == 2 ? second(axis) : 0.0);
        }
        if (out_u8) *reinterpret_cast<uint8_t*>(o) = out_u8_of(v);
        else *reinterpret_cast<float*>(o) = __double2float_rn(v);
      } else if (kind == 3) {
        for (int a = 0; a < D; ++a) reinterpret_cast<float*>(o)[a] = __double2float_rn(first(a));
      } else {
        const double h00 = second(0), h11 = second(1);
        auto g2 = [&](int dx, int dy) {
          const int64_t xi = x + dx < 0 ? 0 : (x + dx >= m0 ? m0 - 1 : x + dx);
          const int64_t yi = y + dy < 0 ? 0 : (y + dy >= m1 ? m1 - 1 : y + dy);
          return sval(s, m0, m1, xi, yi, z);
        };
        const double num = __dadd_rn(__dsub_rn(__dsub_rn(g2(1, 1), g2(1, -1)), g2(-1, 1)), g2(-1, -1));
        const double h01 = __ddiv_rn(num, __dmul_rn(__dmul_rn(4.0, h0), h1));
        float* const f = reinterpret_cast<float*>(o);
        f[0] = __double2float_rn(h00);
        f[1] = __double2float_rn(h11);
        f[2] = __double2float_rn(h01);
      }
    }
}

// DifferenceOfGaussiansFilter (edges.rs:995-1006): s1 - s2 in f64, converted.
template <typename Tp>
__global__ void __launch_bounds__(kT) k_rec_sub(const Tp* s1, const Tp* s2, int64_t m0, int64_t m1, int64_t m2,
                                                 char* dst, int64_t dp0, int64_t dp1, int64_t dp2, int out_u8) {
  const int64_t x = (int64_t)blockIdx.x * kT + threadIdx.x;
  if (x >= m0) return;
  for (int64_t z = blockIdx.z; z < m2; z += gridDim.z)
    for (int64_t y = blockIdx.y; y < m1; y += gridDim.y) {
      const int64_t i = (z * m1 + y) * m0 + x;
      const double v = __dsub_rn((double)s1[i], (double)s2[i]);
      char* const o = dst + x * dp0 + y * dp1 + z * dp2;
      if (out_u8) *reinterpret_cast<uint8_t*>(o) = out_u8_of(v);
      else *reinterpret_cast<float*>(o) = __double2float_rn(v);
    }
}

// ZeroCrossingFilter (edges.rs:480-514) over the Laplacian image `l` (dense,
// the requested region): 1 where center * neighbour < 0 (f64; exact for f32
// and u8 values) for a neighbour along some axis, clamped to the region;
// else 0, in the pixel type.
template <typename Tp>
__global__ void __launch_bounds__(kT) k_rec_zero(const Tp* l, int64_t m0, int64_t m1, int64_t m2, int D, char* dst,
                                                  int64_t dp0, int64_t dp1, int64_t dp2, int out_u8) {
  const int64_t x = (int64_t)blockIdx.x * kT + threadIdx.x;
  if (x >= m0) return;
  const int64_t m[3] = {m0, m1, m2};
  for (int64_t z = blockIdx.z; z < m2; z += gridDim.z)
    for (int64_t y = blockIdx.y; y < m1; y += gridDim.y) {
      const int64_t p[3] = {x, y, z};
      const double c = sval(l, m0, m1, x, y, z);
      bool zc = false;
      for (int a = 0; a < D && !zc; ++a)
        for (int off = -1; off <= 1 && !zc; off += 2) {
          int64_t q[3] = {p[0], p[1], p[2]};
          q[a] = q[a] + off < 0 ? 0 : (q[a] + off >= m[a] ? m[a] - 1 : q[a] + off);
          zc = __dmul_rn(c, sval(l, m0, m1, q[0], q[1], q[2])) < 0.0;
        }
      char* const o = dst + x * dp0 + y * dp1 + z * dp2;
      if (out_u8) *reinterpret_cast<uint8_t*>(o) = zc ? 1 : 0;
      else *reinterpret_cast<float*>(o) = zc ? 1.0f : 0.0f;
    }
}

dim3 grid3(int64_t n0, int64_t n1, int64_t n2) {
  return dim3((unsigned)((n0 + kT - 1) / kT), (unsigned)std::min<int64_t>(std::max<int64_t>(n1, 1), 65535),
              (unsigned)std::min<int64_t>(std::max<int64_t>(n2, 1), 65535));
}

}  // namespace

// Host-side Young & van Vliet coefficients (recursive_gaussian.rs:33-49), f64,
// every operation in the reference's order.
void yvv_coeffs(double sigma, double out[4]) {
  if (!(sigma > 0.5)) sigma = 0.5;  // sigma.max(0.5); f64::max takes 0.5 over NaN
  const double q = sigma >= 2.5 ? 0.98711 * sigma - 0.96330 : 3.97156 - 4.14554 * std::sqrt(1.0 - 0.26891 * sigma);
  const double q2 = q * q;
  const double q3 = q2 * q;
  const double b0 = 1.57825 + 2.44413 * q + 1.4281 * q2 + 0.422205 * q3;
  const double b1 = 2.44413 * q + 2.85619 * q2 + 1.26661 * q3;
  const double b2 = -(1.4281 * q2 + 1.26661 * q3);
  const double b3 = 0.422205 * q3;
  out[0] = 1.0 - (b1 + b2 + b3) / b0;
  out[1] = b1 / b0;
  out[2] = b2 / b0;
  out[3] = b3 / b0;
}

itkg_status launch_recursive(const itkg_image& in, const itkg_region& largest, const itkg_region& requested,
                             double sigma, int axis, int rounding, const itkg_image& out, void* stream) {
  const int D = in.dim;
  const bool ref = rounding == ITKG_ROUND_REFERENCE;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  RecGeom g;
  for (int d = 0; d < 3; ++d) {
    g.n[d] = d < D ? (int64_t)largest.size[d] : 1;
    g.lo[d] = d < D ? largest.index[d] : 0;
  }
  if (g.n[0] * g.n[1] * g.n[2] == 0) return ITKG_SUCCESS;
  if (in.dtype != ITKG_F32 && in.dtype != ITKG_I16 && in.dtype != ITKG_U8 && in.dtype != ITKG_BF16 && in.dtype != ITKG_F16)
    return set_error(ITKG_ERROR_UNSUPPORTED, "input dtype %d not supported", in.dtype);
  RecLines a;
  std::memset(&a, 0, sizeof a);
  a.g = g;
  a.pitch = g.n[0] > 1 && axis <= 0 ? (g.n[0] + 1) / 2 * 2 : g.n[0];
  a.in.at = static_cast<char*>(in.data);
  a.out.at = static_cast<char*>(out.data);
  a.in.dtype = in.dtype;
  a.out.dtype = out.dtype;
  int axes[3], naxes = 0;  // lines of length <= 1 are left alone (recursive_gaussian.rs:98-100)
  for (int d = 0; d < 3; ++d) {
    a.in.p[d] = d < D ? in.pitch[d] : 0;
    a.out.p[d] = d < D ? out.pitch[d] : 0;
    if (d < D) {
      a.in.at += (g.lo[d] - in.region.index[d]) * in.pitch[d];
      a.out.at += (g.lo[d] - out.region.index[d]) * out.pitch[d];
      a.lo[d] = requested.index[d] - g.lo[d];
      a.hi[d] = a.lo[d] + (int64_t)requested.size[d];
      if ((axis < 0 || d == axis) && g.n[d] > 1) axes[naxes++] = d;
    } else {
      a.hi[d] = 1;
    }
  }
  itkg_status st = ITKG_SUCCESS;
  double* buf = nullptr;
  auto copy = [&](const RecImage& from, const RecImage& to, const int64_t* lo, const int64_t* hi) {
    k_rec_copy<<<grid3(hi[0] - lo[0], hi[1] - lo[1], hi[2] - lo[2]), kT, 0, s>>>(from, to, lo[0], lo[1], lo[2], hi[0] - lo[0],
                                                                              hi[1] - lo[1], hi[2] - lo[2]);
    note_launch("recursive_copy");
  };
  RecImage scratch;
  std::memset(&scratch, 0, sizeof scratch);
  const int64_t none[3] = {0, 0, 0};
  // One axis of few lines runs at the latency of its own f64 chain, which the
  // conversions on the same pipe hold up: they run apart, over the whole image.
  // (Up to four warps; they share no f64 pipe.)  30000 samples in one line,
  // reference rounding: 17.2 ms with them in the line kernel, 14.4 apart.
  const bool apart = naxes == 1 && g.n[0] * g.n[1] * g.n[2] / g.n[axes[0]] <= 128;
  if (naxes == 0) {
    copy(a.in, a.out, a.lo, a.hi);
  } else {
    st = scratch_alloc(reinterpret_cast<void**>(&buf), (size_t)(a.pitch * g.n[1] * g.n[2]) * sizeof(double), stream);
    if (st != ITKG_SUCCESS) return st;
    a.d = buf;
    scratch.at = reinterpret_cast<char*>(buf);
    scratch.dtype = kRecF64;
    scratch.p[0] = sizeof(double);
    scratch.p[1] = a.pitch * (int64_t)sizeof(double);
    scratch.p[2] = scratch.p[1] * g.n[1];
    if (apart) copy(a.in, scratch, none, g.n);
  }
  for (int i = 0; i < naxes; ++i) {
    const int d = axes[i];
    double c[4];
    yvv_coeffs(sigma / in.spacing[d], c);
    a.axis = d;
    a.in_step = a.in.p[d];
    a.out_step = a.out.p[d];
    a.w0 = a.lo[d], a.w1 = a.hi[d];
    a.B = c[0], a.a1 = c[1], a.a2 = c[2], a.a3 = c[3];
    const int64_t lines = g.n[0] * g.n[1] * g.n[2] / g.n[d];
    const unsigned blocks = (unsigned)((lines + 31) / 32);
    const auto& fns = g.n[d] > kMaxInt32Line ? kRecFns<int64_t> : kRecFns<int>;
    fns[ref ? 1 : 0][i == 0 && !apart][i + 1 == naxes && !apart][d == 0]<<<blocks, 32, 0, s>>>(a);
    note_launch(ref ? "recursive_lines_f64" : "recursive_lines_f64_fma");
  }
  if (apart) copy(scratch, a.out, a.lo, a.hi);
  {
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) st = set_error(ITKG_ERROR_CUDA, "recursive gaussian launch: %s", cudaGetErrorString(e));
  }
  scratch_free(buf, stream);
  if (st == ITKG_SUCCESS) set_last_kernel(ref ? "recursive_lines_f64" : "recursive_lines_f64_fma");
  return st;
}

itkg_status launch_recursive_derivative(const itkg_image& in, const itkg_region& largest,
                                        const itkg_region& requested, double sigma, double sigma2, int kind,
                                        int axis, int order, int rounding, const itkg_image& out, void* stream) {
  const int D = in.dim;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the smoothed image: RecursiveGaussianFilter::generate_region(requested) in the input's pixel type
  itkg_image sm;
  std::memset(&sm, 0, sizeof sm);
  sm.dim = D;
  sm.dtype = in.dtype;
  sm.components = 1;
  sm.location = ITKG_DEVICE;
  sm.region = requested;
  int64_t m[3] = {1, 1, 1};
  for (int d = 0; d < D; ++d) m[d] = (int64_t)requested.size[d], sm.spacing[d] = in.spacing[d];
  const int64_t esz = in.dtype == ITKG_U8 ? 1 : 4;
  sm.pitch[0] = esz;
  sm.pitch[1] = esz * m[0];
  sm.pitch[2] = esz * m[0] * m[1];
  const bool dog = kind == 5;
  const size_t sm_bytes = (size_t)(esz * m[0] * m[1] * m[2]);
  void* buf = nullptr;
  void* buf2 = nullptr;
  {
    itkg_status sa = scratch_alloc(&buf, sm_bytes, stream);
    if (sa == ITKG_SUCCESS && dog) sa = scratch_alloc(&buf2, sm_bytes, stream);
    if (sa != ITKG_SUCCESS) {
      scratch_free(buf, stream);
      return sa;
    }
  }
  sm.data = buf;
  itkg_status st = launch_recursive(in, largest, requested, sigma, -1, rounding, sm, stream);
  if (st == ITKG_SUCCESS && dog) {  // the second smoothing, then s1 - s2
    itkg_image sm2 = sm;
    sm2.data = buf2;
    st = launch_recursive(in, largest, requested, sigma2, -1, rounding, sm2, stream);
    if (st == ITKG_SUCCESS) {
      int64_t dp[3] = {0, 0, 0};
      for (int d = 0; d < 3; ++d) dp[d] = d < D ? out.pitch[d] : 0;
      char* dst = static_cast<char*>(out.data);
      for (int d = 0; d < D; ++d) dst += (requested.index[d] - out.region.index[d]) * out.pitch[d];
      const dim3 gr = grid3(m[0], m[1], m[2]);
      const int u8 = out.dtype == ITKG_U8 ? 1 : 0;
      if (in.dtype == ITKG_U8)
        k_rec_sub<uint8_t><<<gr, kT, 0, s>>>(static_cast<const uint8_t*>(buf), static_cast<const uint8_t*>(buf2), m[0],
                                             m[1], m[2], dst, dp[0], dp[1], dp[2], u8);
      else
        k_rec_sub<float><<<gr, kT, 0, s>>>(static_cast<const float*>(buf), static_cast<const float*>(buf2), m[0], m[1],
                                           m[2], dst, dp[0], dp[1], dp[2], u8);
      note_launch("recursive_difference");
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) st = set_error(ITKG_ERROR_CUDA, "recursive difference launch: %s", cudaGetErrorString(e));
    }
    scratch_free(buf, stream);
    scratch_free(buf2, stream);
    if (st == ITKG_SUCCESS) set_last_kernel("recursive_difference");
    return st;
  }
  if (st == ITKG_SUCCESS) {
    double h[3] = {1.0, 1.0, 1.0};
    for (int d = 0; d < D; ++d) h[d] = in.spacing[d];
    int64_t dp[3] = {0, 0, 0};
    for (int d = 0; d < 3; ++d) dp[d] = d < D ? out.pitch[d] : 0;
    char* dst = static_cast<char*>(out.data);
    for (int d = 0; d < D; ++d) dst += (requested.index[d] - out.region.index[d]) * out.pitch[d];
    const dim3 gr = grid3(m[0], m[1], m[2]);
    const int u8 = out.dtype == ITKG_U8 ? 1 : 0;
    // ZeroCrossingBasedEdgeDetectionFilter (edges.rs:1045-1052): the Laplacian
    // (kind 1) into a dense scratch image in the pixel type, then zero crossings
    const bool zero = kind == 6;
    void* lap = nullptr;
    if (zero) st = scratch_alloc(&lap, sm_bytes, stream);
    if (st == ITKG_SUCCESS) {
      char* const d1 = zero ? static_cast<char*>(lap) : dst;
      const int64_t p1[3] = {zero ? esz : dp[0], zero ? esz * m[0] : dp[1], zero ? esz * m[0] * m[1] : dp[2]};
      const int k1 = zero ? 1 : kind;
      if (in.dtype == ITKG_U8)
        k_rec_deriv<uint8_t><<<gr, kT, 0, s>>>(static_cast<const uint8_t*>(buf), m[0], m[1], m[2], D, k1, axis, order,
                                               h[0], h[1], h[2], d1, p1[0], p1[1], p1[2], u8);
      else
        k_rec_deriv<float><<<gr, kT, 0, s>>>(static_cast<const float*>(buf), m[0], m[1], m[2], D, k1, axis, order,
                                             h[0], h[1], h[2], d1, p1[0], p1[1], p1[2], u8);
      note_launch("recursive_derivative");
      if (zero) {
        if (in.dtype == ITKG_U8)
          k_rec_zero<uint8_t><<<gr, kT, 0, s>>>(static_cast<const uint8_t*>(lap), m[0], m[1], m[2], D, dst, dp[0],
                                                dp[1], dp[2], u8);
        else
          k_rec_zero<float><<<gr, kT, 0, s>>>(static_cast<const float*>(lap), m[0], m[1], m[2], D, dst, dp[0], dp[1],
                                              dp[2], u8);
        note_launch("recursive_zero_crossing");
      }
      const cudaError_t e = cudaGetLastError();
      if (e != cudaSuccess) st = set_error(ITKG_ERROR_CUDA, "recursive derivative launch: %s", cudaGetErrorString(e));
    }
    scratch_free(lap, stream);
  }
  scratch_free(buf, stream);
  if (st == ITKG_SUCCESS) set_last_kernel(kind == 6 ? "recursive_zero_crossing" : "recursive_derivative");
  return st;
}

}  // namespace itkg
