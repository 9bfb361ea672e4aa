// residual.cu — reprojection residual of the centred radial camera model over an unsorted
// observation list, and its hand-written vector-Jacobian product (adjoint).
//
// Model (crates/openmvg-ba/src/kernel/multi_view/self_calibration/model.rs:26-129): camera j has
// R_j = exp(rotvec_j), translation t_j and intrinsics (f, k1, k2); for observation i of camera j
// and point p, X_c = R_j X_p + t_j, n = (X_c.x / X_c.z, X_c.y / X_c.z), r^2 = |n|^2 and
//   residual_i = f (1 + k1 r^2 + k2 r^4) n - pixel_i            (pixels centred at the principal point)
// An observation is admissible when X_c.z > 64 eps max|X_c|, r^2 is inside the first radial turn
// (the first positive root of 1 + 3 k1 r^2 + 5 k2 r^4) and the distortion map has det > 1e-12
// (model.rs:26-75, 143-172); otherwise its residual is NaN and it adds nothing to the gradients.
//
// Adjoint of one observation with upstream gradient g (2 values) and J = d residual / d X_c:
//   a = J^T g;  d/dt += a;  d/dX_p += R^T a;  d/drotvec += Jl(rotvec)^T (R X_p x a)
//   d/df += (Jint[:,0] . g) / f;  d/dk1 += Jint[:,1] . g;  d/dk2 += Jint[:,2] . g
// where Jl is the left Jacobian of SO(3) (d exp(w) X / dw = -[exp(w) X]x Jl(w)) and Jint holds the
// model's intrinsic columns (log f, k1, k2) (model.rs:298-315).
//
// Determinism: observations arrive in any order, so gradients are reduced by key with integer
// atomics on per-output fixed-point values. A first pass records each output component's largest
// contribution magnitude (atomicMax on the float's bits, order independent); each component's
// power-of-two scale leaves ceil(log2 n) + 1 bits of headroom in a signed 64-bit accumulator; a second
// pass adds the scaled, rounded contributions (integer addition is associative, so the sum is the same
// in every run); a last pass converts and accumulates into the caller's gradient arrays. Resolution:
// 2^-(61 - ceil(log2 n)) of the component's largest term. The rotation's left Jacobian is the same for
// all of a camera's observations, so the passes reduce R X_p x a and the last one applies Jl^T.
//
// What bounds the passes is neither bytes nor flops but the number of separate lines their gathers and
// atomics touch: a lane has its own camera and point. So a camera's constants are one 64-byte row read
// in four 16-byte loads, the twelve contributions of an observation are handed over a warp's shared
// memory so that one instruction's lanes cover neighbouring accumulators (about 3 observations' lines
// instead of 32), and the first pass reads the current maximum and leaves out the atomic unless the
// contribution is larger. Measured at 10M unordered observations of 3,000 cameras and 2M points, per
// launch: first pass 931 -> 417 us, second 1,078 -> 521 us (a camera's 26 constants in as many scattered
// loads, an atomic's 32 lanes on 32 lines and one atomic per contribution in both passes before).
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <string>

#include "../../include/ba_cuda.h"
#include "ba_device.cuh"

namespace omvgba {
namespace residual {

constexpr int kThreads = 256;

// A camera's constants: one row of 16 values, 16-byte aligned. turn: the first radial turn (squared
// radius), infinite when there is none.
template <typename T>
struct __align__(16) CamRow {
  T R[9], t[3], f, k1, k2, turn;
};
constexpr size_t kCamScratch = 104;  // bytes of workspace reserved per camera

template <typename T>
__device__ __forceinline__ void rodrigues(const T w[3], T R[9], T Jl[9]) {
  const T t2 = w[0] * w[0] + w[1] * w[1] + w[2] * w[2];
  const T th = sqrt(t2);
  // a = sin(th)/th, b = (1 - cos th)/th^2 = 2 sin^2(th/2)/th^2, c = (th - sin th)/th^3
  T a, b, c;
  const T small = sizeof(T) == 4 ? T(0.1) : T(1e-3);
  if (th < small) {
    a = T(1) - t2 / T(6) + t2 * t2 / T(120);
    b = T(0.5) - t2 / T(24) + t2 * t2 / T(720);
    c = T(1) / T(6) - t2 / T(120) + t2 * t2 / T(5040);
  } else {
    const T s = sin(th), h = sin(T(0.5) * th);
    a = s / th;
    b = T(2) * h * h / t2;
    c = (th - s) / (t2 * th);
  }
  // K = [w]x, K^2 = w w^T - t2 I
  const T K[9] = {0, -w[2], w[1], w[2], 0, -w[0], -w[1], w[0], 0};
  for (int i = 0; i < 3; ++i)
    for (int j = 0; j < 3; ++j) {
      const T k2 = w[i] * w[j] - (i == j ? t2 : T(0));
      const T id = i == j ? T(1) : T(0);
      R[3 * i + j] = id + a * K[3 * i + j] + b * k2;
      Jl[3 * i + j] = id + b * K[3 * i + j] + c * k2;
    }
}

template <typename T>
__device__ __forceinline__ T radial_turn(T k1, T k2) {
  double turn = 0.0;
  return first_radial_turn_squared((double)k1, (double)k2, &turn) ? (T)turn : T(INFINITY);
}

// The row of camera j without its turn (infinite).
template <typename T>
__device__ __forceinline__ CamRow<T> make_row(const T* __restrict__ rotvec, const T* __restrict__ trans,
                                              const T* __restrict__ intr, uint64_t j) {
  CamRow<T> c;
  const T w[3] = {rotvec[3 * j], rotvec[3 * j + 1], rotvec[3 * j + 2]};
  T Jl[9];
  rodrigues(w, c.R, Jl);
  for (int k = 0; k < 3; ++k) c.t[k] = trans[3 * j + k];
  c.f = intr[3 * j];
  c.k1 = intr[3 * j + 1];
  c.k2 = intr[3 * j + 2];
  c.turn = T(INFINITY);
  return c;
}

// Residual, J = d residual / d X_c and the intrinsic columns (log f, k1, k2); false when the
// observation is inadmissible.
template <typename T>
__device__ __forceinline__ bool radial_eval(const CamRow<T>& c, T X, T Y, T Z, T ox, T oy, T r[2], T J[2][3],
                                            T Ji[2][3], T* radius2 = nullptr) {
  const T s = fmax(fmax(fabs(X), fabs(Y)), fabs(Z));
  if (!(isfinite(X) && isfinite(Y) && isfinite(Z)) || !(Z > T(64.0 * kEps) * s)) return false;
  if (!(c.f > T(0) && isfinite(c.f) && isfinite(c.k1) && isfinite(c.k2))) return false;
  const T iz = T(1) / Z;
  const T n0 = X * iz, n1 = Y * iz;
  const T r2 = n0 * n0 + n1 * n1;
  if (r2 >= c.turn && c.turn < T(INFINITY)) return false;
  if (radius2) *radius2 = r2;
  const T r4 = r2 * r2;
  const T dist = T(1) + c.k1 * r2 + c.k2 * r4;
  const T rd = c.k1 + T(2) * (c.k2 * r2);
  const T slope = dist + T(2) * r2 * rd;
  const T det = dist * slope;
  if (!isfinite(det) || det <= T(1e-12)) return false;
  const T p0 = c.f * dist * n0, p1 = c.f * dist * n1;
  const T dx = T(2) * n0 * rd, dy = T(2) * n1 * rd;
  const T nj00 = c.f * (dist + n0 * dx), nj01 = c.f * n0 * dy;
  const T nj10 = c.f * n1 * dx, nj11 = c.f * (dist + n1 * dy);
  J[0][0] = nj00 * iz;
  J[0][1] = nj01 * iz;
  J[0][2] = -(nj00 * n0 + nj01 * n1) * iz;
  J[1][0] = nj10 * iz;
  J[1][1] = nj11 * iz;
  J[1][2] = -(nj10 * n0 + nj11 * n1) * iz;
  r[0] = p0 - ox;
  r[1] = p1 - oy;
  Ji[0][0] = p0;
  Ji[0][1] = c.f * r2 * n0;
  Ji[0][2] = c.f * r4 * n0;
  Ji[1][0] = p1;
  Ji[1][1] = c.f * r2 * n1;
  Ji[1][2] = c.f * r4 * n1;
  return isfinite(r[0]) && isfinite(r[1]) && isfinite(J[0][0] + J[0][1] + J[0][2] + J[1][0] + J[1][1] + J[1][2]);
}

template <typename T>
__device__ __forceinline__ void camera_point(const CamRow<T>& c, const T* X, T xc[3], T rx[3]) {
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    rx[i] = c.R[3 * i] * X[0] + c.R[3 * i + 1] * X[1] + c.R[3 * i + 2] * X[2];
    xc[i] = rx[i] + c.t[i];
  }
}

// Points of a warp's lanes into `out` (96 values, lane l's at 3 l): three lanes share a point, so a load
// instruction touches about 11 points' lines instead of 32. p must be in range (0 stands in).
template <typename T>
__device__ __forceinline__ void warp_points(const T* __restrict__ points, uint32_t p, T* out) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int s = 0; s < 3; ++s) {
    const int at = 32 * s + lane, o = at / 3;
    const uint32_t q = __shfl_sync(0xffffffffu, p, o);
    out[at] = points[3 * (uint64_t)q + (at - 3 * o)];
  }
  __syncwarp();
}

// Forward pass: the camera constants are recomputed per observation, so the pass needs no scratch.
// An observation whose camera or point index is out of range (a negative int32 index reads as a
// large uint32) touches no camera or point and gets a NaN residual. The radial turn is a handful of FP64
// divisions and a root: it is formed only where 1 + 3 k1 s + 5 k2 s^2 could reach zero up to the
// observation's own radius.
template <typename T>
__global__ void k_forward(uint64_t n, const uint32_t* __restrict__ cam, const uint32_t* __restrict__ pt,
                          const T* __restrict__ pixel, const T* __restrict__ rotvec, const T* __restrict__ intr,
                          const T* __restrict__ trans, const T* __restrict__ points, uint64_t ncam, uint64_t npts,
                          T* __restrict__ residual) {
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const uint32_t j = cam[i], p = pt[i];
  T r[2] = {T(NAN), T(NAN)};
  if (j < ncam && p < npts) {
    const CamRow<T> c = make_row(rotvec, trans, intr, j);
    const T X[3] = {points[3 * (uint64_t)p], points[3 * (uint64_t)p + 1], points[3 * (uint64_t)p + 2]};
    T xc[3], rx[3], J[2][3], Ji[2][3], r2;
    camera_point(c, X, xc, rx);
    bool ok = radial_eval(c, xc[0], xc[1], xc[2], pixel[2 * i], pixel[2 * i + 1], r, J, Ji, &r2);
    if (ok && !(T(3) * fabs(c.k1) * r2 + T(5) * fabs(c.k2) * r2 * r2 < T(0.5))) {
      const T turn = radial_turn(c.k1, c.k2);
      ok = !(r2 >= turn && turn < T(INFINITY));
    }
    if (!ok) r[0] = r[1] = T(NAN);
  }
  residual[2 * i] = r[0];
  residual[2 * i + 1] = r[1];
}

// The same with every camera's row in shared memory, formed once per CTA: a persistent grid of CTAs
// walks the observations, pixels and residuals as 2-vectors. 16-byte chunk q of row j sits at chunk
// q ^ swizzle(j), so that lanes with different cameras spread over the banks.
template <typename T>
__device__ __forceinline__ uint32_t row_chunk(uint32_t j, uint32_t q) {
  constexpr uint32_t CH = sizeof(T);  // chunks of a row: 64 or 128 bytes
  return j * CH + (q ^ (sizeof(T) == 4 ? (j >> 1) & 3u : j & 7u));
}
template <typename T>
struct __align__(2 * sizeof(T)) Pair2 {
  T x, y;
};
template <typename T>
__global__ void __launch_bounds__(1024) k_forward_table(uint64_t n, const uint32_t* __restrict__ cam,
                                                        const uint32_t* __restrict__ pt, const T* __restrict__ pixel,
                                                        const T* __restrict__ rotvec, const T* __restrict__ intr,
                                                        const T* __restrict__ trans, const T* __restrict__ points,
                                                        uint32_t ncam, uint64_t npts, T* __restrict__ residual) {
  extern __shared__ uint4 table[];  // ncam rows of sizeof(T) chunks
  constexpr uint32_t CH = sizeof(T);
  union Row {
    CamRow<T> c;
    uint4 q[CH];
    __device__ Row() {}
  };
  for (uint32_t j = threadIdx.x; j < ncam; j += blockDim.x) {
    Row row;
    row.c = make_row(rotvec, trans, intr, j);
    row.c.turn = radial_turn(row.c.k1, row.c.k2);
#pragma unroll
    for (uint32_t q = 0; q < CH; ++q) table[row_chunk<T>(j, q)] = row.q[q];
  }
  __syncthreads();
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += step) {
    const uint32_t j = cam[i], p = pt[i];
    const Pair2<T> px = reinterpret_cast<const Pair2<T>*>(pixel)[i];
    T r[2] = {T(NAN), T(NAN)};
    if (j < ncam && p < npts) {
      const T X[3] = {points[3 * (uint64_t)p], points[3 * (uint64_t)p + 1], points[3 * (uint64_t)p + 2]};
      Row row;
#pragma unroll
      for (uint32_t q = 0; q < CH; ++q) row.q[q] = table[row_chunk<T>(j, q)];
      T xc[3], rx[3], J[2][3], Ji[2][3];
      camera_point(row.c, X, xc, rx);
      if (!radial_eval(row.c, xc[0], xc[1], xc[2], px.x, px.y, r, J, Ji)) r[0] = r[1] = T(NAN);
    }
    reinterpret_cast<Pair2<T>*>(residual)[i] = Pair2<T>{r[0], r[1]};
  }
}

// Fixed-point accumulation tables, one entry per output component (cameras: 9 = rotvec 3,
// translation 3, intrinsics 3; points: 3).
struct Accum {
  uint32_t* maxbits;  // largest |contribution| (float bits)
  unsigned long long* sum;
  uint64_t ncomp;
  uint32_t* bad_index;  // set when an observation's camera or point index is out of range
  int headroom;
};

constexpr int kCamComps = 9;
constexpr int kObsComps = kCamComps + 3;

// A component's scale 2^e from its largest contribution (bits, finite): 62 - headroom - E with the
// largest < 2^E.
__device__ __forceinline__ int scale_exponent(uint32_t bits, int headroom) {
  const int E = bits >= 0x00800000u ? (int)(bits >> 23) - 126 : (32 - __clz((int)bits)) - 149;
  return 62 - headroom - E;
}
__device__ __forceinline__ double exp2_int(int e) {  // 2^e, e in the range of normal doubles
  return __hiloint2double((e + 1023) << 20, 0);
}

// Clears the accumulators (words of 16 bytes) and forms the camera rows.
__global__ void k_vjp_setup(uint64_t ncam, const float* __restrict__ rotvec, const float* __restrict__ trans,
                            const float* __restrict__ intr, CamRow<float>* __restrict__ rows, uint4* clear,
                            uint64_t words) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x, first = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  for (uint64_t i = first; i < words; i += step) clear[i] = make_uint4(0, 0, 0, 0);
  for (uint64_t j = first; j < ncam; j += step) {
    CamRow<float> c = make_row(rotvec, trans, intr, j);
    c.turn = radial_turn(c.k1, c.k2);
    rows[j] = c;
  }
}

// One observation's contributions per lane; PASS 0 records maxima, PASS 1 adds fixed-point values. An
// observation whose camera or point index is out of range adds nothing anywhere and raises the
// bad-index word, which makes the finish pass write NaN into every gradient output. The warp's 32 x 12
// contributions go through shared memory: lane l of step s then takes contribution (32 s + l) % 12 of
// observation (32 s + l) / 12.
template <int PASS>
__global__ void __launch_bounds__(kThreads) k_vjp(uint64_t n, const uint32_t* __restrict__ cam,
                                                  const uint32_t* __restrict__ pt, const float* __restrict__ pixel,
                                                  const CamRow<float>* __restrict__ rows,
                                                  const float* __restrict__ points, const float* __restrict__ grad,
                                                  uint64_t ncam, uint64_t npts, Accum acc) {
  __shared__ float sv[kThreads / 32][kObsComps * 33];
  const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  const int lane = threadIdx.x & 31;
  float* mine = sv[threadIdx.x >> 5];
  uint32_t j = 0, p = 0;
  float v[kObsComps];
#pragma unroll
  for (int k = 0; k < kObsComps; ++k) v[k] = 0.0f;
  bool live = i < n;
  if (live) {
    j = cam[i];
    p = pt[i];
    if (j >= ncam || p >= npts) {
      if (PASS == 0) atomicOr(acc.bad_index, 1u);
      live = false;
      j = p = 0;
    }
  }
  if (npts > 0) warp_points(points, p, mine);
  if (live) {
    const float g0 = grad[2 * i], g1 = grad[2 * i + 1];
    if (!(g0 == 0.0f && g1 == 0.0f)) {
      CamRow<float> c;
      const float4* row = reinterpret_cast<const float4*>(rows + j);
#pragma unroll
      for (int q = 0; q < 4; ++q) reinterpret_cast<float4*>(&c)[q] = __ldg(row + q);
      const float X[3] = {mine[3 * lane], mine[3 * lane + 1], mine[3 * lane + 2]};
      float xc[3], rx[3], r[2], J[2][3], Ji[2][3];
      camera_point(c, X, xc, rx);
      if (radial_eval(c, xc[0], xc[1], xc[2], pixel[2 * i], pixel[2 * i + 1], r, J, Ji)) {
        float a[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) a[k] = J[0][k] * g0 + J[1][k] * g1;
        // rotation, before Jl^T: rx x a
        v[0] = rx[1] * a[2] - rx[2] * a[1];
        v[1] = rx[2] * a[0] - rx[0] * a[2];
        v[2] = rx[0] * a[1] - rx[1] * a[0];
#pragma unroll
        for (int k = 0; k < 3; ++k) v[3 + k] = a[k];
        v[6] = (Ji[0][0] * g0 + Ji[1][0] * g1) / c.f;
        v[7] = Ji[0][1] * g0 + Ji[1][1] * g1;
        v[8] = Ji[0][2] * g0 + Ji[1][2] * g1;
        // point: R^T a
#pragma unroll
        for (int k = 0; k < 3; ++k) v[9 + k] = c.R[k] * a[0] + c.R[3 + k] * a[1] + c.R[6 + k] * a[2];
      }
    }
  }
  __syncwarp();  // the points are read: their place takes the contributions
#pragma unroll
  for (int k = 0; k < kObsComps; ++k) mine[k * 33 + lane] = v[k];
  __syncwarp();
  // (32 s + l) / 12 and % 12 repeat every three steps, eight observations on
  uint32_t ou[3], ku[3];
#pragma unroll
  for (int u = 0; u < 3; ++u) {
    ou[u] = (32 * u + lane) / kObsComps;
    ku[u] = (32 * u + lane) % kObsComps;
  }
  uint32_t* const pt_max = acc.maxbits + (uint64_t)kCamComps * ncam;
  unsigned long long* const pt_sum = acc.sum + (uint64_t)kCamComps * ncam;
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    float val[3];
    uint32_t* mx[3];
    unsigned long long* sm[3];
    uint32_t bits[3];
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      const uint32_t o = 8 * t + ou[u], k = ku[u];
      const uint32_t oj = __shfl_sync(0xffffffffu, j, o), op = __shfl_sync(0xffffffffu, p, o);
      val[u] = mine[k * 33 + o];
      const bool cam_part = k < kCamComps;
      const uint64_t at = cam_part ? (uint64_t)oj * kCamComps + k : (uint64_t)op * 3 + (k - kCamComps);
      mx[u] = (cam_part ? acc.maxbits : pt_max) + at;
      if (PASS == 1) sm[u] = (cam_part ? acc.sum : pt_sum) + at;
      // an absent observation's values are zero: nothing to read or add
      bits[u] = val[u] != 0.0f ? (PASS == 0 ? *mx[u] : __ldg(mx[u])) : 0u;
    }
#pragma unroll
    for (int u = 0; u < 3; ++u) {
      if (val[u] == 0.0f) continue;
      if (PASS == 0) {
        const uint32_t b = isnan(val[u]) ? 0x7fc00000u : __float_as_uint(fabsf(val[u]));
        if (b > bits[u]) atomicMax(mx[u], b);  // a stale maximum only adds an atomic
      } else if (bits[u] < 0x7f800000u) {  // else a non-finite component: resolved in the finish pass
        const long long q = __double2ll_rn((double)val[u] * exp2_int(scale_exponent(bits[u], acc.headroom)));
        atomicAdd(sm[u], (unsigned long long)q);
      }
    }
  }
}

// Component k's sum as a double; NaN when a contribution was not finite or an index was out of range.
__device__ __forceinline__ double component_sum(const Accum& acc, uint64_t k, bool bad) {
  const uint32_t bits = acc.maxbits[k];
  if (bad || bits >= 0x7f800000u) return NAN;
  if (bits == 0u) return 0.0;
  return (double)(long long)acc.sum[k] * exp2_int(-scale_exponent(bits, acc.headroom));
}

__global__ void k_vjp_finish(Accum acc, uint64_t ncam, const float* __restrict__ rotvec, float* __restrict__ g_rot,
                             float* __restrict__ g_t, float* __restrict__ g_int, float* __restrict__ g_pt) {
  const uint64_t k = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
  if (k >= acc.ncomp) return;
  const bool bad = *acc.bad_index != 0u;
  if (k >= kCamComps * ncam) {
    g_pt[k - kCamComps * ncam] += (float)component_sum(acc, k, bad);
    return;
  }
  const uint64_t j = k / kCamComps, c = k - kCamComps * j;
  if (c < 3) {  // Jl^T times the summed R X_p x a
    const float w[3] = {rotvec[3 * j], rotvec[3 * j + 1], rotvec[3 * j + 2]};
    float R[9], Jl[9];
    rodrigues(w, R, Jl);
    double val = 0.0;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
      const float col = c == 0 ? Jl[3 * r] : (c == 1 ? Jl[3 * r + 1] : Jl[3 * r + 2]);
      const double s = component_sum(acc, kCamComps * j + r, bad);
      // a camera without contributions may have no finite Jl (its rotation vector is not finite)
      if (s != 0.0) val += (double)col * s;
    }
    g_rot[3 * j + c] += (float)val;
  } else {
    const float val = (float)component_sum(acc, k, bad);
    if (c < 6)
      g_t[3 * j + c - 3] += val;
    else
      g_int[3 * j + c - 6] += val;
  }
}

inline size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Workspace: camera rows, then the cleared region (maxima, sums, bad-index word).
struct VjpLayout {
  size_t pre, maxbits, sum, bad, total;
};
inline VjpLayout vjp_layout(uint64_t ncam, uint64_t npts) {
  VjpLayout l;
  const uint64_t ncomp = kCamComps * ncam + 3 * npts;
  l.pre = 0;
  l.maxbits = align256(kCamScratch * ncam);
  l.sum = l.maxbits + align256(sizeof(uint32_t) * ncomp);
  l.bad = l.sum + align256(sizeof(unsigned long long) * ncomp);
  l.total = l.bad + 256;
  return l;
}

inline unsigned grid_for(uint64_t n) { return (unsigned)((n + kThreads - 1) / kThreads); }

inline int ceil_log2(uint64_t n) {
  int b = 0;
  while ((1ull << b) < n && b < 63) ++b;
  return b;
}

int fail(omvgba_error* e, int code, const std::string& msg) {
  if (e) {
    e->code = code;
    e->detail = -1;
    std::strncpy(e->message, msg.c_str(), sizeof(e->message) - 1);
    e->message[sizeof(e->message) - 1] = 0;
  }
  return code;
}

int ok(omvgba_error* e) {
  if (e) {
    e->code = 0;
    e->detail = -1;
    e->message[0] = 0;
  }
  return OMVGBA_OK;
}

int cuda_status(omvgba_error* e) {
  cudaError_t st = cudaGetLastError();
  if (st != cudaSuccess) return fail(e, OMVGBA_CUDA_ERROR, std::string("CUDA error: ") + cudaGetErrorString(st));
  return ok(e);
}

// Which forward kernel: the shared-memory camera table pays for itself once every CTA of a persistent grid
// has many more observations than the table has rows (kTableObservations, 32 per camera), fits beside
// nothing else in an SM's shared memory, and needs pixels and residuals aligned for 2-vector access.
// Everything else recomputes the row per observation. Measured, recomputed -> table: 10M observations of
// 3,000 cameras FP32 228 -> 142 us, 1.2M of 500 cameras FP64 41 -> 29 us. At 8,000 observations the two
// are equal (a launch's latency).
constexpr uint64_t kTableObservations = 1u << 18;
constexpr size_t kTableMaxBytes = 200 * 1024;

template <typename T>
int forward(void* stream, uint64_t n, const uint32_t* cam, const uint32_t* pt, const T* pixel, uint64_t ncam,
            const T* rotvec, const T* trans, const T* intr, uint64_t npts, const T* points, T* residual,
            omvgba_error* err) {
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const bool aligned = ((reinterpret_cast<uintptr_t>(pixel) | reinterpret_cast<uintptr_t>(residual)) % (2 * sizeof(T))) == 0;
  // (the rows first: a caller that does not know its camera count may pass any bound, also one whose products wrap)
  if (aligned && ncam <= kTableMaxBytes / sizeof(CamRow<T>) && n >= kTableObservations && n >= 32 * ncam) {
    const size_t smem = (size_t)ncam * sizeof(CamRow<T>);
    const int threads = smem > kTableMaxBytes / 2 ? 1024 : 512;
    int dev = 0, sms = 0, per = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(k_forward_table<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTableMaxBytes);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_forward_table<T>, threads, smem);
    if (e != cudaSuccess) return cuda_status(err);
    const unsigned grid = (unsigned)std::min<uint64_t>((n + threads - 1) / threads, (uint64_t)sms * std::max(per, 1));
    k_forward_table<T><<<grid, threads, smem, st>>>(n, cam, pt, pixel, rotvec, intr, trans, points, (uint32_t)ncam, npts,
                                                     residual);
    return cuda_status(err);
  }
  k_forward<T><<<grid_for(n), kThreads, 0, st>>>(n, cam, pt, pixel, rotvec, intr, trans, points, ncam, npts,
                                                  residual);
  return cuda_status(err);
}

bool any_null(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if (!p) return true;
  return false;
}

}  // namespace residual
}  // namespace omvgba

using namespace omvgba::residual;

extern "C" {

uint64_t omvgba_residual_vjp_workspace_bytes(uint64_t observation_count, uint64_t camera_count,
                                             uint64_t point_count) {
  (void)observation_count;
  return vjp_layout(camera_count, point_count).total;
}

int32_t omvgba_residual_forward_f32(void* stream, uint64_t observation_count, const uint32_t* camera_index,
                                    const uint32_t* point_index, const float* pixel, uint64_t camera_count,
                                    const float* rotvec, const float* translation, const float* intrinsics,
                                    uint64_t point_count, const float* points, float* residual,
                                    omvgba_error* error) {
  if (observation_count == 0) return ok(error);
  if (any_null({camera_index, point_index, pixel, rotvec, translation, intrinsics, points, residual}))
    return fail(error, OMVGBA_INVALID_ARGUMENT, "null argument");
  return forward<float>(stream, observation_count, camera_index, point_index, pixel, camera_count, rotvec,
                        translation, intrinsics, point_count, points, residual, error);
}

int32_t omvgba_residual_forward_f64(void* stream, uint64_t observation_count, const uint32_t* camera_index,
                                    const uint32_t* point_index, const double* pixel, uint64_t camera_count,
                                    const double* rotvec, const double* translation, const double* intrinsics,
                                    uint64_t point_count, const double* points, double* residual,
                                    omvgba_error* error) {
  if (observation_count == 0) return ok(error);
  if (any_null({camera_index, point_index, pixel, rotvec, translation, intrinsics, points, residual}))
    return fail(error, OMVGBA_INVALID_ARGUMENT, "null argument");
  return forward<double>(stream, observation_count, camera_index, point_index, pixel, camera_count, rotvec,
                         translation, intrinsics, point_count, points, residual, error);
}

int32_t omvgba_residual_vjp_f32(void* stream, uint64_t observation_count, const uint32_t* camera_index,
                                const uint32_t* point_index, const float* pixel, uint64_t camera_count,
                                const float* rotvec, const float* translation, const float* intrinsics,
                                uint64_t point_count, const float* points, const float* grad_residual,
                                float* grad_rotvec, float* grad_translation, float* grad_intrinsics,
                                float* grad_points, void* workspace, uint64_t workspace_bytes,
                                omvgba_error* error) {
  if (observation_count == 0) return ok(error);
  if (any_null({camera_index, point_index, pixel, rotvec, translation, intrinsics, points, grad_residual,
                grad_rotvec, grad_translation, grad_intrinsics, grad_points, workspace}))
    return fail(error, OMVGBA_INVALID_ARGUMENT, "null argument");
  const VjpLayout l = vjp_layout(camera_count, point_count);
  if (workspace_bytes < l.total)
    return fail(error, OMVGBA_INVALID_ARGUMENT,
                "workspace too small: " + std::to_string(workspace_bytes) + " < " + std::to_string(l.total));
  if ((reinterpret_cast<uintptr_t>(workspace) & 255) != 0)
    return fail(error, OMVGBA_INVALID_ARGUMENT, "workspace must be 256-byte aligned");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(workspace);
  CamRow<float>* rows = reinterpret_cast<CamRow<float>*>(ws + l.pre);
  Accum acc{reinterpret_cast<uint32_t*>(ws + l.maxbits), reinterpret_cast<unsigned long long*>(ws + l.sum),
            kCamComps * camera_count + 3 * point_count, reinterpret_cast<uint32_t*>(ws + l.bad),
            ceil_log2(observation_count) + 1};
  const uint64_t words = (l.total - l.maxbits) / 16;
  k_vjp_setup<<<(unsigned)std::min<uint64_t>(4096, grid_for(std::max(words, camera_count))), kThreads, 0, st>>>(
      camera_count, rotvec, translation, intrinsics, rows, reinterpret_cast<uint4*>(ws + l.maxbits), words);
  k_vjp<0><<<grid_for(observation_count), kThreads, 0, st>>>(observation_count, camera_index, point_index, pixel, rows,
                                                             points, grad_residual, camera_count, point_count, acc);
  k_vjp<1><<<grid_for(observation_count), kThreads, 0, st>>>(observation_count, camera_index, point_index, pixel, rows,
                                                             points, grad_residual, camera_count, point_count, acc);
  k_vjp_finish<<<grid_for(acc.ncomp), kThreads, 0, st>>>(acc, camera_count, rotvec, grad_rotvec, grad_translation,
                                                         grad_intrinsics, grad_points);
  return cuda_status(error);
}

}  // extern "C"
