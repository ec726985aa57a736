// Per-axis passes for longer kernels (and for the casting passes of 2-D
// images): one pass of convolve_axis (src/filters/conv.rs:11-41) with the taps
// walked once per run of outputs.
//
// A thread makes M consecutive outputs along the pass axis for two lines (the
// two lanes of a packed register).  It reads each of the M + 2R inputs its run
// reaches once and adds it, times the tap, to every output it reaches: output
// m takes tap j - m from input j, so each output sums its taps in ascending
// order from zero exactly as the one-output-per-thread pass does, bit for bit
// in either rounding.  Inputs and taps beyond an output's window are never
// multiplied in (the first and last M - 1 inputs run as unrolled triangles),
// so an infinity or NaN reaches the same outputs as before.  The inputs of a
// run that ends past the request are clamped to the request's last tap
// (line_window.hpp): a pass's source ends there.  The M live taps
// sit in registers and shift by one per input.
//
//   k_lines_yz  passes along y and z: lanes on columns c and c + 32 of a
//               64-column strip, inputs straight from L1 / L2 (a block's warps
//               stack along the axis and share their windows in L1).
//   k_lines_x   passes along x: the tile is transposed through shared memory
//               ([x][64 rows], stride 66 floats: 8-byte stores and loads of
//               consecutive row pairs are conflict-free), then the same walk.
//
// Bound: the FP32 pipe (M packed FMAs per input against two 4-byte loads and
// one tap load), with the staging latency on top along x.  Measured on 192^3
// f32, radius 24, FMA rounding, per pass: x 27.4 us, y and z 20.7 us (the FMA
// pipe's floor is 8.6 us, the 57 MB of compulsory traffic 8.3 us); the
// one-output-per-thread pass, which issued a load, a clamp and 64-bit address
// arithmetic per tap, took 307 us.  Radius 12: x 22.9, y / z 14.9 us, against
// 94.7 and 66 us of the unrolled small-radius pass.
//
// Reference rounding with packed arithmetic: a packed mul / add pair is
// contracted to an FMA by ptxas, so the product is fma(x, w, -0), with the -0
// a kernel argument the compiler cannot fold (x * w rounded once, the sign of
// zero kept), and the sum a packed add: bit-identical to the scalar sequence
// and half its issue slots.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "f32x2.cuh"
#include "internal.hpp"
#include "line_window.hpp"
#include "pixel.cuh"

namespace itkg {
namespace {

constexpr int kM = kLineRun;   // outputs per thread
constexpr int kStrip = 64;     // lines per warp (two per lane)
constexpr int kRowPitch = 66;  // k_lines_x: floats per staged x position
constexpr int kMaxWarps = 8;
// Warps per block: 4, so that four blocks share an SM at 128 registers and one
// block's staging overlaps the others' arithmetic.  k_lines_x stages
// (16 warps + 2R) * 66 floats, so from R = 65 on fewer than four blocks fit and
// a block has 8 warps, as far as they fit 227 KB (R <= 360).
constexpr int kWarps = 4, kSmallR = 64, kBigR = 360;

template <bool REF>
__device__ __forceinline__ f2_t tap2(f2_t acc, f2_t x, f2_t w, f2_t nz) {
  if constexpr (REF) return add2(acc, fma2(x, w, nz));
  else return fma2(x, w, acc);
}

// The walk: load(j) gives input j (0 .. 2R + kM - 1) of the thread's two
// lines, called in ascending order.  W2[i] holds tap j - i while input j is
// added; w2[j] is tap j in both lanes.  Needs 2R >= kM - 1.
template <bool REF, typename Load>
__device__ __forceinline__ void walk(const f2_t* w2, int R, f2_t nz, f2_t (&acc)[kM], Load load) {
  f2_t W2[kM];
#pragma unroll
  for (int m = 0; m < kM; ++m) acc[m] = 0ull, W2[m] = 0ull;
  auto step = [&](int j, int live) {  // input j reaches outputs 0 .. live - 1
#pragma unroll
    for (int i = kM - 1; i > 0; --i) W2[i] = W2[i - 1];
    W2[0] = w2[j];
    const f2_t v = load(j);
#pragma unroll
    for (int m = 0; m < kM; ++m)
      if (m < live) acc[m] = tap2<REF>(acc[m], v, W2[m], nz);
  };
#pragma unroll
  for (int j = 0; j < kM - 1; ++j) step(j, j + 1);
  int j = kM - 1;
  const int je = 2 * R + 1;
  // (a whole turn of the tap window costs no register moves; shorter pieces
  // pay kM moves per piece)
#pragma unroll 1
  for (; j + kM <= je; j += kM) {
#pragma unroll
    for (int s = 0; s < kM; ++s) step(j + s, kM);
  }
#pragma unroll 1
  for (; j + 4 <= je; j += 4) {
#pragma unroll
    for (int s = 0; s < 4; ++s) step(j + s, kM);
  }
#pragma unroll 1
  for (; j < je; ++j) step(j, kM);
#pragma unroll
  for (int t = 0; t < kM - 1; ++t) {  // taps run out: outputs t + 1 .. kM - 1
    const f2_t v = load(je + t);
#pragma unroll
    for (int m = t + 1; m < kM; ++m) acc[m] = tap2<REF>(acc[m], v, W2[m - t - 1], nz);
  }
}

// The passes are programmatic dependents of each other: the next one's blocks
// may be scheduled as this one's retire (they wait here for it to complete
// before they touch memory), which hides its launch.
__device__ __forceinline__ void pdl_begin() {
  asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory");
  asm volatile("griddepcontrol.wait;\n" ::: "memory");
}

struct LineTaps2 {
  f2_t w2[kMaxParamTaps];  // tap k in both lanes
};

struct LinesArgs {
  AxisArgs a;
  float nz;      // -0 (see the file comment)
  int32_t runs;  // runs of kM outputs along the axis
};

// grid: x strips of 64 flattened columns, y groups of blockDim.y runs, z the
// remaining axis.  Input f32.  The last strip of a row is moved back to end
// with the row (FULL: rows of at least 64 columns), so that every lane's two
// columns exist and both loads share one address; the columns that the strip
// before it writes are not written again.
template <typename Tout, bool REF, bool FULL>
__global__ void __launch_bounds__(32 * kMaxWarps, 2) k_lines_yz(const __grid_constant__ LinesArgs p,
                                                                const __grid_constant__ LineTaps2 W) {
  const AxisArgs& a = p.a;
  pdl_begin();
  const int md = a.axis, od = 3 - md;
  const int64_t rowlen = a.out_size[0] * a.comps;
  const int64_t strip = (int64_t)blockIdx.x * kStrip;
  const int64_t c0 = (FULL ? min(strip, rowlen - kStrip) : strip) + threadIdx.x;
  const int run = blockIdx.y * blockDim.y + threadIdx.y;
  if (c0 >= rowlen || run >= p.runs) return;
  const bool one = c0 >= strip, two = FULL ? c0 + 32 >= strip : c0 + 32 < rowlen;  // columns to write
  const int d1 = FULL ? 32 : (two ? 32 : 0);  // the second column (the first again where there is none)
  const int64_t mp = md == 1 ? a.src_pitch[1] : a.src_pitch[2], op = od == 1 ? a.src_pitch[1] : a.src_pitch[2];
  const int64_t mo = md == 1 ? a.src_origin[1] : a.src_origin[2], oo = od == 1 ? a.src_origin[1] : a.src_origin[2];
  const int64_t m_at = (md == 1 ? a.out_index[1] : a.out_index[2]) + (int64_t)run * kM;
  const int64_t o_first = od == 1 ? a.out_index[1] : a.out_index[2];
  const int64_t on = od == 1 ? a.out_size[1] : a.out_size[2];
  const int64_t left = (md == 1 ? a.out_size[1] : a.out_size[2]) - (int64_t)run * kM;
  const int nv = (int)(left < kM ? left : kM);
  const f2_t nz = pack2(p.nz, p.nz);
  const LineWindow win = line_window(m_at, nv, a.radius, a.lo, a.hi);
  const int64_t dmp = md == 1 ? a.dst_pitch[1] : a.dst_pitch[2], dop = od == 1 ? a.dst_pitch[1] : a.dst_pitch[2];
  const int64_t dmo = md == 1 ? a.dst_origin[1] : a.dst_origin[2], doo = od == 1 ? a.dst_origin[1] : a.dst_origin[2];
  for (int64_t o = blockIdx.z; o < on; o += gridDim.z) {
    // a pointer that steps by one pitch from window entry to window entry
    const char* s = static_cast<const char*>(a.src) + (a.out_index[0] - a.src_origin[0]) * a.src_pitch[0] + c0 * 4 +
                    (o_first + o - oo) * op + (a.lo - mo + line_at(win, 0)) * mp;
    f2_t acc[kM];
    walk<REF>(W.w2, a.radius, nz, acc, [&](int j) {
      const float* const f = reinterpret_cast<const float*>(s);
      // (plain loads: the previous pass may write this memory while this block
      // waits in pdl_begin, and read-only loads ask for memory that nothing
      // writes during the kernel)
      const f2_t v = pack2(f[0], f[d1]);
      s += line_steps(win, j) ? mp : 0;
      return v;
    });
    char* d = static_cast<char*>(a.dst) + (a.out_index[0] - a.dst_origin[0]) * a.dst_pitch[0] +
              c0 * (int64_t)sizeof(Tout) + (o_first + o - doo) * dop + (m_at - dmo) * dmp;
#pragma unroll
    for (int m = 0; m < kM; ++m) {
      if (m < nv) {
        float lo, hi;
        unpack2(acc[m], lo, hi);
        Tout* const t = reinterpret_cast<Tout*>(d);
        if (one) t[0] = from_f32<Tout>(lo);
        if (two) t[32] = from_f32<Tout>(hi);
      }
      d += dmp;
    }
  }
}

// grid: x groups of blockDim.y runs along x, y (strided) groups of 64 lines.
// A line is one component of one row; line l is component l % comps of row
// l / comps.  Output f32.
template <typename Tin, bool REF>
__global__ void __launch_bounds__(32 * kMaxWarps, 2) k_lines_x(const __grid_constant__ LinesArgs p,
                                                               const __grid_constant__ LineTaps2 W) {
  extern __shared__ float tile[];  // [x position][kRowPitch]
  const AxisArgs& a = p.a;
  pdl_begin();
  const int warp = threadIdx.y, lane = threadIdx.x, nw = blockDim.y;
  const int64_t nlines = a.out_size[1] * a.out_size[2] * a.comps;
  const int64_t groups = (nlines + kStrip - 1) / kStrip;
  const int x_first = blockIdx.x * nw * kM;  // first output of the block
  const int64_t x_left = a.out_size[0] - x_first;
  const int span = (int)min((int64_t)nw * kM, x_left);  // outputs of the block inside the request
  const int width = nw * kM + 2 * a.radius;              // staged positions
  const LineWindow win = line_window(a.out_index[0] + x_first, span, a.radius, a.lo, a.hi);
  const f2_t nz = pack2(p.nz, p.nz);
  __shared__ int64_t s_src[kStrip], s_dst[kStrip];  // byte offsets of the group's lines
  const char* const src = static_cast<const char*>(a.src) + (a.lo - a.src_origin[0]) * a.src_pitch[0];
  char* const dst = static_cast<char*>(a.dst) + (a.out_index[0] + x_first - a.dst_origin[0]) * a.dst_pitch[0];
  for (int64_t g = blockIdx.y; g < groups; g += gridDim.y) {
    const int nl = (int)min((int64_t)kStrip, nlines - g * kStrip);  // lines of the group
    // (one 64-bit division chain per line and group, not per line and warp)
    for (int i = warp * 32 + lane; i < kStrip; i += nw * 32) {
      const int64_t l = g * kStrip + min(i, nl - 1);
      const int64_t row = l / a.comps, c = l - row * a.comps;
      const int64_t z = a.out_index[2] + row / a.out_size[1], y = a.out_index[1] + row % a.out_size[1];
      s_src[i] = c * (int64_t)sizeof(Tin) + (y - a.src_origin[1]) * a.src_pitch[1] + (z - a.src_origin[2]) * a.src_pitch[2];
      s_dst[i] = c * 4 + (y - a.dst_origin[1]) * a.dst_pitch[1] + (z - a.dst_origin[2]) * a.dst_pitch[2];
    }
    __syncthreads();
    // stage: warp w takes line pairs 2w, 2w + 1, then 2 (w + nw), ...; lanes
    // along x, four positions each: 16 loads in flight per thread (entries
    // past the tile repeat the window's last position and are dropped)
    static_assert(kStrip / 2 % 2 == 0, "whole quads of lines");
    for (int pr = 2 * warp; pr < kStrip / 2; pr += 2 * nw) {
      const char* sl[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) sl[i] = src + s_src[2 * pr + i];
      float* const t = tile + 2 * pr;
      for (int xb = lane; xb < width; xb += 128) {
        float v[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int64_t off = (int64_t)line_at(win, xb + 32 * q) * a.src_pitch[0];
#pragma unroll
          for (int i = 0; i < 4; ++i) v[q][i] = to_f32(*reinterpret_cast<const Tin*>(sl[i] + off));
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int x = xb + 32 * q;
          if (x < width) {
            *reinterpret_cast<float2*>(t + x * kRowPitch) = make_float2(v[q][0], v[q][1]);
            *reinterpret_cast<float2*>(t + x * kRowPitch + 2) = make_float2(v[q][2], v[q][3]);
          }
        }
      }
    }
    __syncthreads();
    f2_t acc[kM];
    const bool active = warp * kM < span;
    float* const t0 = tile + (warp * kM) * kRowPitch + 2 * lane;
    if (active)
      walk<REF>(W.w2, a.radius, nz, acc, [&](int j) { return *reinterpret_cast<const f2_t*>(t0 + j * kRowPitch); });
    __syncthreads();  // the staged inputs are free for the outputs
    if (active) {
#pragma unroll
      for (int m = 0; m < kM; ++m) *reinterpret_cast<f2_t*>(t0 + m * kRowPitch) = acc[m];
    }
    __syncthreads();
    for (int pr = warp; 2 * pr < nl; pr += nw) {
      char* const da = dst + s_dst[2 * pr];
      char* const db = dst + s_dst[2 * pr + 1];
      const bool two = 2 * pr + 1 < nl;
      const float* const t = tile + 2 * pr;
      for (int x = lane; x < span; x += 32) {
        const float2 v = *reinterpret_cast<const float2*>(t + x * kRowPitch);
        *reinterpret_cast<float*>(da + x * a.dst_pitch[0]) = v.x;
        if (two) *reinterpret_cast<float*>(db + x * a.dst_pitch[0]) = v.y;
      }
    }
    __syncthreads();
  }
}

using LinesFn = void (*)(const LinesArgs, const LineTaps2);

template <typename T>
LinesFn yz_fn(bool ref, bool full) {
  return ref ? (full ? k_lines_yz<T, true, true> : k_lines_yz<T, true, false>)
             : (full ? k_lines_yz<T, false, true> : k_lines_yz<T, false, false>);
}
template <typename T>
LinesFn x_fn(bool ref) { return ref ? k_lines_x<T, true> : k_lines_x<T, false>; }

// Warps per block: `runs` split evenly over the fewest blocks of at most `most`.
int warps_for(int64_t runs, int most) {
  const int64_t blocks = (runs + most - 1) / most;
  return (int)((runs + blocks - 1) / blocks);
}

// k_lines_x's dynamic shared memory for nw warps at radius R, and the most it
// takes.  Beside it the kernel has 1 KB of its own (line offsets), which counts
// against the 48 KB that need no opt-in.
constexpr size_t x_smem(int nw, int R) { return (size_t)(nw * kM + 2 * R) * kRowPitch * sizeof(float); }
constexpr int kMaxR = (kMaxParamTaps - 1) / 2;
constexpr size_t kXSmemMost = std::max(x_smem(kMaxWarps, kBigR), x_smem(kWarps, kMaxR));
static_assert(kXSmemMost + 2 * kStrip * sizeof(int64_t) <= 227 * 1024, "k_lines_x fits a block");

// The limit on dynamic shared memory is the kernel's, shared by every thread
// that launches it: set once per kernel and device, to the most that any call
// takes, so that no call lowers it under another's launch.
std::mutex g_x_mu;
std::vector<std::pair<const void*, int>> g_x_ready;
itkg_status prepare_x(const void* fn) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return set_error(ITKG_ERROR_CUDA, "cudaGetDevice: %s", cudaGetErrorString(e));
  std::lock_guard<std::mutex> lk(g_x_mu);
  for (const auto& r : g_x_ready)
    if (r.first == fn && r.second == dev) return ITKG_SUCCESS;
  e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kXSmemMost);
  if (e != cudaSuccess) return set_error(ITKG_ERROR_CUDA, "conv_lines smem: %s", cudaGetErrorString(e));
  g_x_ready.push_back({fn, dev});
  return ITKG_SUCCESS;
}

}  // namespace

itkg_status launch_conv_lines(const AxisArgs& a, const float* w, int in_dtype, int out_dtype, int rounding,
                              void* stream) {
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const bool ref = rounding == ITKG_ROUND_REFERENCE;
  const bool f32 = in_dtype == ITKG_F32 && out_dtype == ITKG_F32;
  const int64_t n = a.out_size[a.axis];
  const int64_t extent = a.hi - a.lo + 1;
  // window arithmetic in int32
  if (2 * a.radius < kM - 1 || extent > INT32_MAX / 2 || n > INT32_MAX / 2) return ITKG_ERROR_UNSUPPORTED;
  LineTaps2 W;
  for (int k = 0; k < 2 * a.radius + 1; ++k) W.w2[k] = splat2_host(w[k]);
  LinesArgs p;
  p.a = a;
  p.nz = -0.0f;
  p.runs = (int32_t)((n + kM - 1) / kM);
  LinesFn fn = nullptr;
  dim3 grid, block;
  size_t smem = 0;
  if (a.axis == 0) {
    if (out_dtype != ITKG_F32) return ITKG_ERROR_UNSUPPORTED;
    switch (in_dtype) {
      case ITKG_F32: fn = x_fn<float>(ref); break;
      case ITKG_I16: fn = x_fn<int16_t>(ref); break;
      case ITKG_U8: fn = x_fn<uint8_t>(ref); break;
      case ITKG_BF16: fn = x_fn<__nv_bfloat16>(ref); break;
      case ITKG_F16: fn = x_fn<__half>(ref); break;
      default: return ITKG_ERROR_UNSUPPORTED;
    }
    const int nw = warps_for(p.runs, a.radius > kSmallR && a.radius <= kBigR ? kMaxWarps : kWarps);
    const int64_t groups = (a.out_size[1] * a.out_size[2] * a.comps + kStrip - 1) / kStrip;
    block = dim3(32, (unsigned)nw);
    grid = dim3((unsigned)((p.runs + nw - 1) / nw), (unsigned)std::min<int64_t>(groups, 65535));
    smem = x_smem(nw, a.radius);
    const itkg_status st = prepare_x(reinterpret_cast<const void*>(fn));
    if (st != ITKG_SUCCESS) return st;
  } else {
    if (in_dtype != ITKG_F32) return ITKG_ERROR_UNSUPPORTED;
    const bool full = a.out_size[0] * a.comps >= kStrip;
    switch (out_dtype) {
      case ITKG_F32: fn = yz_fn<float>(ref, full); break;
      case ITKG_BF16: fn = yz_fn<__nv_bfloat16>(ref, full); break;
      case ITKG_F16: fn = yz_fn<__half>(ref, full); break;
      case ITKG_U8: fn = yz_fn<uint8_t>(ref, full); break;
      default: return ITKG_ERROR_UNSUPPORTED;
    }
    const int nw = warps_for(p.runs, kWarps);
    const int64_t strips = (a.out_size[0] * a.comps + kStrip - 1) / kStrip;
    const int64_t others = a.out_size[3 - a.axis];
    const int64_t gy = (p.runs + nw - 1) / nw;
    if (strips > INT32_MAX || gy > 65535) return ITKG_ERROR_UNSUPPORTED;
    block = dim3(32, (unsigned)nw);
    grid = dim3((unsigned)strips, (unsigned)gy, (unsigned)std::min<int64_t>(others, 65535));
  }
  // Radius 8 .. 12 between f32 images also has the unrolled pass of
  // conv_axis.cu, whose blocks are smaller: under 128 blocks (of the 152 SMs)
  // it is the faster one along x (512^2, reference rounding, radius 12: 6.9
  // against 8.4 us) and as fast along y; 97 x 61 x 73 has 140 blocks: 12.7
  // against 8.8 us.
  if (f32 && a.radius <= kMaxSmallRadius && (uint64_t)grid.x * grid.y * grid.z < 128) return ITKG_ERROR_UNSUPPORTED;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg;
  std::memset(&cfg, 0, sizeof cfg);
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaError_t e = cudaLaunchKernelEx(&cfg, fn, p, W);
  note_launch(ref ? "conv_lines_f32_ref" : "conv_lines_f32_fma");
  if (e == cudaSuccess) e = cudaGetLastError();
  if (e != cudaSuccess) return set_error(ITKG_ERROR_CUDA, "conv_lines launch: %s", cudaGetErrorString(e));
  return ITKG_SUCCESS;
}

}  // namespace itkg
