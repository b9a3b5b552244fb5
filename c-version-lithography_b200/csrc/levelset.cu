// WENO5-Godunov level-set kernels (source/utils/level_set_utils.cpp of the
// reference) as shared-memory-tiled stencils.
//
// Boundary handling: the reference edge-pads phi by 3 on both axes and
// der_weno5 pads by 3 more along the derivative axis; edge padding twice is
// edge padding once by 6, and after cropping the output pixel (i, j) reads
// phi[i][clamp(j-3 .. j+3)] and phi[clamp(i-3 .. i+3)][j]. The tile loader
// therefore clamps every halo index into the image.
#include <cuda_runtime.h>
#include <algorithm>
#include <cfloat>

#include "litho_internal.cuh"

namespace litho_b200 {

constexpr int LS_NT = 128;
constexpr int LS_H = 3;              // halo rows
constexpr int LS_HX = 4;             // halo columns on each side (3 used; keeps pairs aligned)
// A tile takes TXL threads along x, each of which computes blocks of 2 x 2 pixels: its width,
// the rows per pass of the CTA, and the width with halo.
constexpr int LS_WIDE = 32, LS_NARROW = 16;
constexpr int ls_tx(int txl) { return 2 * txl; }
constexpr int ls_ty(int txl) { return 2 * (LS_NT / txl); }
constexpr int ls_sw(int txl) { return ls_tx(txl) + 2 * LS_HX; }
constexpr int LS_ET = 256;           // threads of the elementwise and reduction kernels
// CTAs of tall tiles from which they are used (at least four per SM).
constexpr int LS_TALL_CTAS = 592;
static_assert(ls_sw(LS_WIDE) % 4 == 0 && ls_sw(LS_NARROW) % 4 == 0, "tile rows are 16-byte aligned");

__device__ __forceinline__ float2 f2(float a) { return make_float2(a, a); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, f2(-1.f), a); }
// Reciprocal within 1 ulp of a normal x (the callers keep x normal).
__device__ __forceinline__ float rcp_normal(float x) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float2 rcp2(float2 x) { return make_float2(rcp_normal(x.x), rcp_normal(x.y)); }

// sqrt(x), x >= 0, within 1 ulp, without the branches of the IEEE one.
__device__ __forceinline__ float sqrt_normal(float x) {
  float r;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// WENO5-JS one-sided derivatives (level_set_utils.cpp:45-113) of N neighbouring pixels along
// one axis, for the two lanes of packed FP32x2 arithmetic at once: D[i .. i + 5] are the
// undivided differences around pixel i (D[i + 2], D[i + 3] next to it). The results m[i]
// (minus) and p[i] (plus) are undivided too: the weights do not depend on the spacing.
//
// Minus of pixel i and plus of pixel i - 1 are the two mirrored stencils over the same five
// differences (window i), so they share the smoothness indicators, their normaliser and the
// products of the weights. With e_i = D_{i+1} - D_i and t_i = e_{i+1} - e_i the indicators
// of the triples T_i = (D_i, D_{i+1}, D_{i+2}), T_{i+1}, T_{i+2} are 13/12 t^2 + 1/4 q^2, with
//   q = t_i + 2 e_{i+1}, e_{i+1} + e_{i+2}, t_{i+2} - 2 e_{i+2},
// and the candidates are a difference plus multiples of its triple's two e. Two pixels take
// 127 packed instructions for their 8 derivatives; evaluated one stencil at a time they
// took 4 x 55.
//
// The indicators (scaled by 12/13, and eps with them) are divided by the window's max D^2
// before the weights, which are invariant under that; the scaled values stay inside FP32
// range. alpha_i = gamma_i / S_i^2 and sum(alpha_i d_i) / sum(alpha_i) are both multiplied
// by 10 S1^2 S2^2 S3^2: one division, of values in [1e-24, 1e8]. A window of differences
// below 1.1e-19, whose squares FP32 does not hold as normal numbers, counts as 1.1e-19: its
// weights only mix values of that size.
constexpr float WENO_TINY = 1.1e-19f;
template <int N>
__device__ __forceinline__ void weno5_chain(const float2 (&D)[N + 5], float2 (&m)[N], float2 (&p)[N]) {
  float2 e[N + 4], t[N + 3], t2[N + 3];
#pragma unroll
  for (int i = 0; i < N + 4; ++i) e[i] = sub2(D[i + 1], D[i]);
#pragma unroll
  for (int i = 0; i < N + 3; ++i) {
    t[i] = sub2(e[i + 1], e[i]);
    t2[i] = __fmul2_rn(t[i], t[i]);
  }
  auto cand = [&](float2 d, float ca, float2 ea, float cb, float2 eb) {
    return __ffma2_rn(f2(cb), eb, __ffma2_rn(f2(ca), ea, d));
  };
  // the triples' central candidates: of T_i from its left (two upwind) and right neighbour
  float2 cA[N + 2], cB[N + 2];
#pragma unroll
  for (int i = 1; i < N + 1; ++i) {
    cA[i] = cand(D[i + 1], 1.f / 6.f, e[i], 1.f / 3.f, e[i + 1]);
    cB[i + 1] = cand(D[i + 2], -1.f / 3.f, e[i + 1], -1.f / 6.f, e[i + 2]);
  }
  static_assert(N == 2, "three windows around D[2 .. 4]");
  const float2 mid = make_float2(fmaxf(fmaxf(fabsf(D[2].x), fabsf(D[3].x)), fmaxf(fabsf(D[4].x), WENO_TINY)),
                                 fmaxf(fmaxf(fabsf(D[2].y), fabsf(D[3].y)), fmaxf(fabsf(D[4].y), WENO_TINY)));
#pragma unroll
  for (int i = 0; i <= N; ++i) {
    // the largest |D| of the window: its three middle ones and two of (left, right) ends
    const float2 top = make_float2(
        i < 2 ? fmaxf(fmaxf(mid.x, fabsf(D[1].x)), fabsf(D[i ? 5 : 0].x)) : fmaxf(fmaxf(mid.x, fabsf(D[5].x)), fabsf(D[6].x)),
        i < 2 ? fmaxf(fmaxf(mid.y, fabsf(D[1].y)), fabsf(D[i ? 5 : 0].y)) : fmaxf(fmaxf(mid.y, fabsf(D[5].y)), fabsf(D[6].y)));
    const float2 inv = rcp2(__fmul2_rn(top, top));
    auto smooth = [&](float2 q, float2 tt) {
      return __ffma2_rn(__ffma2_rn(__fmul2_rn(q, q), f2(3.f / 13.f), tt), inv, f2(1e-6f * 12.f / 13.f));
    };
    const float2 s1 = smooth(__ffma2_rn(f2(2.f), e[i + 1], t[i]), t2[i]);
    const float2 s2 = smooth(__fadd2_rn(e[i + 1], e[i + 2]), t2[i + 1]);
    const float2 s3 = smooth(__ffma2_rn(f2(-2.f), e[i + 2], t[i + 2]), t2[i + 2]);
    const float2 p1 = __fmul2_rn(s2, s3), p2 = __fmul2_rn(s1, s3), p3 = __fmul2_rn(s1, s2);
    const float2 b1 = __fmul2_rn(p1, p1), b2 = __fmul2_rn(f2(6.f), __fmul2_rn(p2, p2)),
                 b3 = __fmul2_rn(p3, p3);
    auto blend = [&](float2 w1, float2 w3, float2 d1, float2 d2, float2 d3) {
      const float2 w = __fmul2_rn(f2(3.f), w3);
      const float2 num = __ffma2_rn(w, d3, __ffma2_rn(b2, d2, __fmul2_rn(w1, d1)));
      return __fmul2_rn(num, rcp2(__fadd2_rn(__fadd2_rn(w1, b2), w)));
    };
    if (i < N)
      m[i] = blend(b1, b3, cand(D[i + 2], -1.f / 3.f, e[i], 5.f / 6.f, e[i + 1]), cA[i + 1], cB[i + 2]);
    if (i > 0)
      p[i - 1] = blend(b3, b1, cand(D[i + 2], -5.f / 6.f, e[i + 2], 1.f / 3.f, e[i + 3]), cB[i + 1], cA[i]);
  }
}

// Godunov's one-sided slope along an axis for the sign of the normal speed
// (level_set_utils.cpp:180-213): of (minus, plus), max(m, 0) and -min(p, 0) where the
// speed is positive, max(-m, 0) and -min(-p, 0) where it is negative; the larger counts. Where
// the speed is zero the slope does not count, whatever it is (speed_times).
__device__ __forceinline__ float godunov(float sign, float m, float p) {
  return fmaxf(fmaxf(sign * m, -sign * p), 0.f);
}
__device__ __forceinline__ float speed_times(float speed, float length) {
  return speed == 0.f ? 0.f : speed * length;
}

// Tile rows y0 - LS_H .. , columns x0 - LS_HX ..: every index clamped into the image.
template <int SH, int SW>
__device__ __forceinline__ void load_tile(float (*t)[SW], const float* __restrict__ phi,
                                          int rows, int cols, int y0, int x0, bool vec4) {
  if (vec4 && x0 >= LS_HX && x0 - LS_HX + SW <= cols) {
    constexpr int Q = SW / 4;
    const float* base = phi + x0 - LS_HX;
#pragma unroll
    for (int i0 = 0; i0 < SH * Q; i0 += LS_NT) {
      const int i = i0 + (int)threadIdx.x;
      if (i < SH * Q) {
        const int ty = i / Q, c = 4 * (i - ty * Q);
        const float* row = base + (size_t)min(max(y0 - LS_H + ty, 0), rows - 1) * cols;
        *reinterpret_cast<float4*>(&t[ty][c]) = __ldg(reinterpret_cast<const float4*>(row + c));
      }
    }
    return;
  }
  // warp w loads tile rows w, w + 4, ...; each lane columns lane, lane + 32, ...
  constexpr int NC = (SW + 31) / 32;
  const int lane = threadIdx.x & 31;
  int xc[NC];
#pragma unroll
  for (int k = 0; k < NC; ++k) xc[k] = min(max(x0 - LS_HX + lane + 32 * k, 0), cols - 1);
  for (int ty = threadIdx.x >> 5; ty < SH; ty += LS_NT / 32) {
    const float* row = phi + (size_t)min(max(y0 - LS_H + ty, 0), rows - 1) * cols;
#pragma unroll
    for (int k = 0; k < NC; ++k)
      if (lane + 32 * k < SW) t[ty][lane + 32 * k] = __ldg(row + xc[k]);
  }
}

// _gradient_1d along x (level_set_utils.cpp:228-255) at global column x of row ly.
template <int SW>
__device__ __forceinline__ float grad_x(const float (*t)[SW], int ly, int lx, int x, int cols,
                                        float inv2d) {
  if (x == 0) return (-3.f * t[ly][lx] + 4.f * t[ly][lx + 1] - t[ly][lx + 2]) * inv2d;
  if (x == cols - 1) return (3.f * t[ly][lx] - 4.f * t[ly][lx - 1] + t[ly][lx - 2]) * inv2d;
  return (t[ly][lx + 1] - t[ly][lx - 1]) * inv2d;
}
template <int SW>
__device__ __forceinline__ float grad_y(const float (*t)[SW], int ly, int lx, int y, int rows,
                                        float inv2d) {
  if (y == 0) return (-3.f * t[ly][lx] + 4.f * t[ly + 1][lx] - t[ly + 2][lx]) * inv2d;
  if (y == rows - 1) return (3.f * t[ly][lx] - 4.f * t[ly - 1][lx] + t[ly - 2][lx]) * inv2d;
  return (t[ly + 1][lx] - t[ly - 1][lx]) * inv2d;
}

// b kappa |grad phi| (level_set_utils.cpp:257-278) from undivided differences (px, py two
// apart, the second ones differences of those): ix2 = 1 / (2 dx)^2, iy2 alike, kb = b ix2 iy2.
__device__ __forceinline__ float kappa_value(float px, float py, float pxx, float pxy, float pyy,
                                             float ix2, float iy2, float kb) {
  const float px2 = px * px, py2 = py * py;
  const float g2 = fmaf(px2, ix2, py2 * iy2);
  const float num = fmaf(pyy, px2, fmaf(-2.f * px * py, pxy, pxx * py2));
  return g2 > (float)DBL_EPSILON ? kb * num * rcp_normal(g2) : 0.f;
}

// The same at global (y, x) near the image border, where some differences are one-sided.
template <int SW>
__device__ __noinline__ float kappa_border(const float (*t)[SW], int ly, int lx, int y, int x,
                                           int rows, int cols, float dx, float dy, float b) {
  const float ix = 1.f / (2.f * dx), iy = 1.f / (2.f * dy);
  float pxy, pxx, pyy;
  // phi_x at (y, x) and its row/column neighbours used by the second derivatives.
  auto px_at = [&](int oy, int ox) { return grad_x(t, ly + oy, lx + ox, x + ox, cols, ix); };
  auto py_at = [&](int oy) { return grad_y(t, ly + oy, lx, y + oy, rows, iy); };
  const float px = px_at(0, 0);
  const float py = py_at(0);
  if (y == 0) pxy = (-3.f * px + 4.f * px_at(1, 0) - px_at(2, 0)) * iy;
  else if (y == rows - 1) pxy = (3.f * px - 4.f * px_at(-1, 0) + px_at(-2, 0)) * iy;
  else pxy = (px_at(1, 0) - px_at(-1, 0)) * iy;
  if (x == 0) pxx = (-3.f * px + 4.f * px_at(0, 1) - px_at(0, 2)) * ix;
  else if (x == cols - 1) pxx = (3.f * px - 4.f * px_at(0, -1) + px_at(0, -2)) * ix;
  else pxx = (px_at(0, 1) - px_at(0, -1)) * ix;
  if (y == 0) pyy = (-3.f * py + 4.f * py_at(1) - py_at(2)) * iy;
  else if (y == rows - 1) pyy = (3.f * py - 4.f * py_at(-1) + py_at(-2)) * iy;
  else pyy = (py_at(1) - py_at(-1)) * iy;
  const float g2 = px * px + py * py;
  const float num = pxx * py * py - 2.f * px * py * pxy + pyy * px * px;
  return g2 > (float)DBL_EPSILON ? b * __fdividef(num, g2) : 0.f;
}

// what: 0 = delta (+ habs), 1 = kappa term, 2 = normal = kappa - delta,
// 3 = RK2 stage 1: out = phi0 + dt N(phi0), 4 = RK2 stage 2:
// out = 0.5 phi0 + 0.5 (phi1 + dt N(phi1)), mask_out = out >= 0.
struct LsArgs {
  int rows, cols;
  const float* phi;   // field whose stencil is evaluated
  const float* phi0;  // stage 2: the step's starting phi
  const float* vn;
  float dx, dy, b;
  const float* dt;    // device scalar (stages)
  float* out;
  float* out2;        // habs (what 0) or mask (what 4)
  // Batched launches: image blockIdx.z of rows x cols images back to back; its dt at
  // dt[blockIdx.z * dt_stride]; its update window {y0, y1, x0, x1} (stages 3, 4 and what
  // 6, 8) at wins + 4 blockIdx.z, the whole image when wins is null.
  const int* wins;
  int dt_stride;
  int vec4, vec2;     // 16-byte loads of phi rows; 8-byte accesses of pixel pairs elsewhere
};

// Stencil modes 0-4. A CTA computes TX x (TY RPT) pixels from a tile in shared memory, each thread RPT blocks of 2 x 2 pixels: packed FP32x2 lanes are the two rows
// along x and the two columns along y, and neighbouring pixels of a block share their
// smoothness indicators and candidates (weno5_chain). The stencil is bound by FP32 issue
// (a packed instruction takes the issue port and the FMA pipe twice): 187 and 206 thread
// instructions per pixel in stages 1 and 2, 82 of them packed, against 422 and 443 for one pixel
// per thread. Stages of 16 images of 2048^2: 932 -> 488 us and 1005 -> 538 us (1.9 and 2.0 TB/s).
// Longer strips fed by cp.async one pass ahead removed the wait for the tile but cost as
// many instructions as they hid (1.24 against 1.23 ms per update at that stage), and scalar
// FFMA on blocks of 2 x 4 pixels ran out of registers and instruction cache (1.6 ms).
//
// DIV: every difference is divided by the spacing before any product of differences, as the
// reference does it. Products of undivided ones leave FP32's range when the spacing, and a
// signed distance with it, is far from 1: the curvature's are its third power, at a spacing of
// 1e-12 its error has doubled and at 1e-15 it is NaN. So DIV serves the spacings outside
// LS_NEAR .. LS_FAR, inside which the products of slopes from 1e-8 to 1e9 stay in range and
// the divisions would cost 3.6 % (16 images of 2048^2: 1136 us an update against 1096).
constexpr float LS_NEAR = 1.f / 4096, LS_FAR = 4096.f;
template <int WHAT, int RPT, bool WIN, bool DIV, int TXL>
__global__ void __launch_bounds__(LS_NT, RPT == 1 ? 6 : 7) levelset_kernel(LsArgs a) {
  constexpr int TY = ls_ty(TXL), SH = TY * RPT + 2 * LS_H, SW = ls_sw(TXL);
  __shared__ __align__(16) float t[SH][SW];
  const size_t img = (size_t)blockIdx.z * a.rows * a.cols;
  const float* phi = a.phi + img;
  float* out = a.out + img;
  int wy0 = 0, wy1 = 0, wx0 = 0, wx1 = 0;   // WIN: the image's update window
  if (WIN) {
    const int* w = a.wins + 4 * (size_t)blockIdx.z;
    wy0 = w[0]; wy1 = w[1]; wx0 = w[2]; wx1 = w[3];
  }
  const int x0 = blockIdx.x * ls_tx(TXL), y0 = blockIdx.y * (TY * RPT);
  const float* phi0 = a.phi0 ? a.phi0 + img : nullptr;
  const float* vn = a.vn ? a.vn + img : nullptr;
  float* out2 = a.out2 ? a.out2 + img : nullptr;
  const int lx = 2 * (threadIdx.x % TXL), x = x0 + lx;
  const bool pair = x + 1 < a.cols;       // both columns of the block lie in the image
  const bool v2 = pair && a.vec2;
  auto load2 = [&](const float* p, size_t i) -> float2 {
    if (v2) return __ldg(reinterpret_cast<const float2*>(p + i));
    return make_float2(__ldg(p + i), pair ? __ldg(p + i + 1) : 0.f);
  };
  auto store2 = [&](float* p, size_t i, float2 v) {
    if (v2) {
      *reinterpret_cast<float2*>(p + i) = v;
    } else {
      p[i] = v.x;
      if (pair) p[i + 1] = v.y;
    }
  };
  // The normal speed of a block, [row](x, x + 1), loaded one pass ahead of its use.
  float2 sp_n[2] = {f2(0.f), f2(0.f)};
  auto fetch = [&](int r) {
    const int y = y0 + 2 * (threadIdx.x / TXL) + r * TY;
    const size_t i = (size_t)y * a.cols + x;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (x < a.cols && y + h < a.rows) {
        if (WHAT != 1) sp_n[h] = load2(vn, i + (size_t)h * a.cols);
        // the starting phi, read at the end of the pass: its line into L2 by then
        if (WHAT == 4 && (threadIdx.x & 15) == 0)
          asm volatile("prefetch.global.L2 [%0];" ::"l"(phi0 + i + (size_t)h * a.cols));
      }
    }
  };
  fetch(0);
  load_tile<SH, SW>(t, phi, a.rows, a.cols, y0, x0, a.vec4 != 0);
  __syncthreads();
  const float idx = 1.f / a.dx, idy = 1.f / a.dy;
  const float ix2 = DIV ? 1.f : 0.25f * idx * idx, iy2 = DIV ? 1.f : 0.25f * idy * idy;
  const float kb = a.b * ix2 * iy2;
  const float dt = (WHAT >= 3) ? a.dt[(size_t)blockIdx.z * a.dt_stride] : 0.f;
  if (x >= a.cols) return;
#pragma unroll 1
  for (int r = 0; r < RPT; ++r) {
    const int ly = 2 * (threadIdx.x / TXL) + r * TY, y = y0 + ly;
    if (y >= a.rows) break;
    const bool two = y + 1 < a.rows;        // both rows lie in the image
    const size_t i0 = (size_t)y * a.cols + x, i1 = i0 + a.cols;
    float2 ph[2] = {f2(0.f), f2(0.f)};      // stage 2: the starting phi, used last
    if (WHAT == 4) {
      ph[0] = load2(phi0, i0);
      if (two) ph[1] = load2(phi0, i1);
    }
    const float* c = &t[ly + LS_H][lx + LS_HX];   // pixel (y, x)
    auto at2 = [&](int oy, int ox) { return *reinterpret_cast<const float2*>(c + oy * SW + ox); };
    const float2 sp[2] = {sp_n[0], sp_n[1]};
    if (r + 1 < RPT) fetch(r + 1);
    if (WIN && (y + 1 < wy0 || y >= wy1 || x + 1 < wx0 || x >= wx1)) {
      // Outside the update window the step keeps phi (stage 1) / the starting phi (stage 2).
      for (int h = 0; h < (two ? 2 : 1); ++h) {
        const size_t i = h ? i1 : i0;
        const float2 keep = WHAT == 3 ? at2(h, 0) : ph[h];
        if (WHAT == 4 && out2)
          store2(out2, i, make_float2(keep.x >= 0.f ? 1.f : 0.f, keep.y >= 0.f ? 1.f : 0.f));
        store2(out, i, keep);
      }
      continue;
    }
    // rows y, y + 1, columns x - 4 .. x + 5
    float ra[10], rb[10];
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const float2 p = at2(0, 2 * k - 4), q = at2(1, 2 * k - 4);
      ra[2 * k] = p.x; ra[2 * k + 1] = p.y;
      rb[2 * k] = q.x; rb[2 * k + 1] = q.y;
    }
    // columns x, x + 1, rows y - 3 .. y + 4
    float2 col[8];
#pragma unroll
    for (int k = 0; k < 8; ++k)
      col[k] = k == 3 ? make_float2(ra[4], ra[5]) : k == 4 ? make_float2(rb[4], rb[5]) : at2(k - 3, 0);
    float2 kap[2] = {f2(0.f), f2(0.f)};
    if (WHAT != 0) {
      if (x >= 2 && x + 1 < a.cols - 2 && y >= 2 && y + 1 < a.rows - 2) {
        // Every difference is central. d(y, x) = phi(y, x + 1) - phi(y, x - 1) of columns x
        // and x + 1 on the rows y - 1 .. y + 2; along x, d of x + 1 is also the step from x.
        // DIV: first and second differences are divided by the two spacings they span, and
        // kappa_value by 1.
        const float2 hx = f2(0.5f * idx), hy = f2(0.5f * idy);
        auto over = [](float2 d, float2 h) { return DIV ? __fmul2_rn(d, h) : d; };
        const float2 up = at2(-1, -2), un = at2(-1, 2), dp = at2(2, -2), dn = at2(2, 2);
        const float2 dm = over(make_float2(col[2].y - up.y, un.x - col[2].x), hx);   // row y - 1
        const float2 da = over(make_float2(ra[5] - ra[3], ra[6] - ra[4]), hx);       // row y
        const float2 db = over(make_float2(rb[5] - rb[3], rb[6] - rb[4]), hx);       // row y + 1
        const float2 dd = over(make_float2(col[5].y - dp.y, dn.x - col[5].x), hx);   // row y + 2
        const float2 ea = over(make_float2(ra[4] - ra[2], ra[7] - ra[5]), hx);       // of x - 1, x + 2
        const float2 eb = over(make_float2(rb[4] - rb[2], rb[7] - rb[5]), hx);
        const float2 pyA = over(sub2(col[4], col[2]), hy), pyB = over(sub2(col[5], col[3]), hy);
        const float2 pyyA = over(sub2(pyB, over(sub2(col[3], col[1]), hy)), hy);
        const float2 pyyB = over(sub2(over(sub2(col[6], col[4]), hy), pyA), hy);
        const float2 pxyA = over(sub2(db, dm), hy), pxyB = over(sub2(dd, da), hy);
        const float2 pxxA = over(make_float2(da.y - ea.x, ea.y - da.x), hx);
        const float2 pxxB = over(make_float2(db.y - eb.x, eb.y - db.x), hx);
        kap[0].x = kappa_value(da.x, pyA.x, pxxA.x, pxyA.x, pyyA.x, ix2, iy2, kb);
        kap[0].y = kappa_value(da.y, pyA.y, pxxA.y, pxyA.y, pyyA.y, ix2, iy2, kb);
        kap[1].x = kappa_value(db.x, pyB.x, pxxB.x, pxyB.x, pyyB.x, ix2, iy2, kb);
        kap[1].y = kappa_value(db.y, pyB.y, pxxB.y, pxyB.y, pyyB.y, ix2, iy2, kb);
      } else {
        for (int h = 0; h < (two ? 2 : 1); ++h) {
          kap[h].x = kappa_border(t, ly + h + LS_H, lx + LS_HX, y + h, x, a.rows, a.cols, a.dx,
                                  a.dy, a.b);
          if (pair)
            kap[h].y = kappa_border(t, ly + h + LS_H, lx + 1 + LS_HX, y + h, x + 1, a.rows, a.cols,
                                    a.dx, a.dy, a.b);
        }
      }
    }
    float2 del[2] = {f2(0.f), f2(0.f)};     // Vn |grad phi|
    if (WHAT != 1) {
      const float2 sg0 = make_float2(copysignf(1.f, sp[0].x), copysignf(1.f, sp[0].y));
      const float2 sg1 = make_float2(copysignf(1.f, sp[1].x), copysignf(1.f, sp[1].y));
      const float sx = DIV ? 1.f : idx, sy = DIV ? 1.f : idy;   // what the slopes still lack
      float2 g[2];
      {
        float2 D[7];
#pragma unroll
        for (int k = 0; k < 7; ++k) {
          D[k] = make_float2(ra[k + 2] - ra[k + 1], rb[k + 2] - rb[k + 1]);
          if (DIV) D[k] = __fmul2_rn(D[k], f2(idx));
        }
        float2 m[2], p[2];   // [column], lanes rows
        weno5_chain<2>(D, m, p);
        g[0] = make_float2(godunov(sg0.x, m[0].x, p[0].x) * sx, godunov(sg0.y, m[1].x, p[1].x) * sx);
        g[1] = make_float2(godunov(sg1.x, m[0].y, p[0].y) * sx, godunov(sg1.y, m[1].y, p[1].y) * sx);
      }
      {
        float2 D[7];
#pragma unroll
        for (int k = 0; k < 7; ++k) {
          D[k] = sub2(col[k + 1], col[k]);
          if (DIV) D[k] = __fmul2_rn(D[k], f2(idy));
        }
        float2 m[2], p[2];   // [row], lanes columns
        weno5_chain<2>(D, m, p);
        auto length = [&](float gx, float sgn, float mi, float pl) {
          const float gy = godunov(sgn, mi, pl) * sy;
          return sqrt_normal(fmaf(gx, gx, gy * gy));
        };
        del[0] = make_float2(speed_times(sp[0].x, length(g[0].x, sg0.x, m[0].x, p[0].x)),
                             speed_times(sp[0].y, length(g[0].y, sg0.y, m[0].y, p[0].y)));
        del[1] = make_float2(speed_times(sp[1].x, length(g[1].x, sg1.x, m[1].x, p[1].x)),
                             speed_times(sp[1].y, length(g[1].y, sg1.y, m[1].y, p[1].y)));
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (h && !two) break;
      const size_t i = h ? i1 : i0;
      float2 v;
      if (WHAT == 0) {
        v = del[h];
        if (out2) store2(out2, i, make_float2(fabsf(sp[h].x), fabsf(sp[h].y)));
      } else if (WHAT == 1) {
        v = kap[h];
      } else {
        const float2 n = sub2(kap[h], del[h]);
        if (WHAT == 2) {
          v = n;
        } else {
          const float2 here = col[3 + h];
          const float2 start = WHAT == 4 ? ph[h] : here;
          v = make_float2(here.x + dt * n.x, here.y + dt * n.y);
          if (WHAT == 4) v = make_float2(0.5f * start.x + 0.5f * v.x, 0.5f * start.y + 0.5f * v.y);
          if (WIN) {
            const bool in_y = y + h >= wy0 && y + h < wy1;
            if (!(in_y && x >= wx0 && x < wx1)) v.x = start.x;
            if (!(in_y && x + 1 >= wx0 && x + 1 < wx1)) v.y = start.y;
          }
          if (WHAT == 4 && out2)
            store2(out2, i, make_float2(v.x >= 0.f ? 1.f : 0.f, v.y >= 0.f ? 1.f : 0.f));
        }
      }
      store2(out, i, v);
    }
  }
}

// Elementwise modes: 6 speed restricted to the update window, 8 phi inside the window over
// phi0 outside (out may be phi0).
template <int WHAT>
__global__ void __launch_bounds__(LS_ET) window_kernel(LsArgs a) {
  const size_t img = (size_t)blockIdx.z * a.rows * a.cols;
  const int* w = a.wins + 4 * (size_t)blockIdx.z;
  const int wy0 = w[0], wy1 = w[1], wx0 = w[2], wx1 = w[3];
  const int x = blockIdx.x * 32 + threadIdx.x % 32;
  for (int r = 0; r < 4; ++r) {
    const int y = blockIdx.y * 32 + threadIdx.x / 32 + 8 * r;
    if (y < a.rows && x < a.cols) {
      const size_t i = img + (size_t)y * a.cols + x;
      const bool in = y >= wy0 && y < wy1 && x >= wx0 && x < wx1;
      if (WHAT == 6) a.out[i] = in ? a.vn[i] : 0.f;
      else a.out[i] = in ? a.phi[i] : a.phi0[i];
    }
  }
}

template <int WHAT, int RPT, bool DIV, int TXL = LS_WIDE>
static void ls_launch_t(cudaStream_t s, const LsArgs& a, int nimg) {
  constexpr int TX = ls_tx(TXL), TY = ls_ty(TXL) * RPT;
  const dim3 g((a.cols + TX - 1) / TX, (a.rows + TY - 1) / TY, nimg);
  if constexpr (WHAT >= 3) {
    if (a.wins) {
      levelset_kernel<WHAT, RPT, true, DIV, TXL><<<g, LS_NT, 0, s>>>(a);
      return;
    }
  }
  levelset_kernel<WHAT, RPT, false, DIV, TXL><<<g, LS_NT, 0, s>>>(a);
}

template <int WHAT, bool DIV>
static void ls_launch(cudaStream_t s, const LsArgs& a, int nimg) {
  // Images of one narrow tile, of whose wide one half the lanes would have no pixel.
  if (a.cols <= ls_tx(LS_NARROW)) return ls_launch_t<WHAT, 1, DIV, LS_NARROW>(s, a, nimg);
  // Tall tiles (fewer halo rows per pixel) where they fill the GPU, else one pass per CTA.
  constexpr int TX = ls_tx(LS_WIDE), TY = 4 * ls_ty(LS_WIDE);
  const long long tall = (long long)((a.cols + TX - 1) / TX) * ((a.rows + TY - 1) / TY) * nimg;
  if (tall >= LS_TALL_CTAS) ls_launch_t<WHAT, 4, DIV>(s, a, nimg);
  else ls_launch_t<WHAT, 1, DIV>(s, a, nimg);
}
template <int WHAT>
static void ls_launch(cudaStream_t s, const LsArgs& a, int nimg) {
  if (std::min(a.dx, a.dy) < LS_NEAR || std::max(a.dx, a.dy) > LS_FAR)
    ls_launch<WHAT, true>(s, a, nimg);
  else
    ls_launch<WHAT, false>(s, a, nimg);
}

cudaError_t launch_levelset(cudaStream_t s, int what, int rows, int cols, const float* phi,
                            const float* phi0, const float* vn, float dx, float dy, float b,
                            const float* dt, float* out, float* out2, int nimg,
                            const int* d_windows, int dt_stride) {
  if (nimg < 1 || nimg > 65535) return cudaErrorInvalidValue;
  auto aligned = [](const void* p, size_t n) { return reinterpret_cast<uintptr_t>(p) % n == 0; };
  LsArgs a{rows, cols, phi, phi0, vn, dx, dy, b, dt, out, out2, d_windows,
           dt_stride, cols % 4 == 0 && aligned(phi, 16),
           cols % 2 == 0 && aligned(phi0, 8) && aligned(vn, 8) && aligned(out, 8) && aligned(out2, 8)};
  const dim3 flat((cols + 31) / 32, (rows + 31) / 32, nimg);
  switch (what) {
    case 0: ls_launch<0>(s, a, nimg); break;
    case 1: ls_launch<1>(s, a, nimg); break;
    case 2: ls_launch<2>(s, a, nimg); break;
    case 3: ls_launch<3>(s, a, nimg); break;
    case 4: ls_launch<4>(s, a, nimg); break;
    case 6: window_kernel<6><<<flat, LS_ET, 0, s>>>(a); break;
    case 8: window_kernel<8><<<flat, LS_ET, 0, s>>>(a); break;
    default: return cudaErrorInvalidValue;
  }
  return cudaGetLastError();
}

// max |Vn| of image blockIdx.y and its dt = get_dt_normal_kappa (level_set_utils.cpp:280-288)
// in one launch: vd[2 i] = max |Vn|, vd[2 i + 1] = dt. The CTAs of an image join their
// maxima with an atomic on the float's bits (|Vn| >= 0 orders as integers), and the last of
// them to arrive (count[i]) computes dt. vd and count start at zero. A non-finite Vn raises
// *bad. Bound by HBM reads: four 16-byte loads in flight per thread (16 images of 2048^2:
// 111 us with one 4-byte load each, 47 us so), and no second launch for dt.
__global__ void __launch_bounds__(LS_ET) speed_dt_kernel(const float* __restrict__ v, size_t n, int vec,
                                                         float dx, float dy, float cfl, float b,
                                                         float* __restrict__ vd,
                                                         unsigned* __restrict__ count, int* bad) {
  __shared__ float sh[LS_ET / 32];
  v += (size_t)blockIdx.y * n;
  vd += 2 * (size_t)blockIdx.y;
  float m = 0.f, chk = 0.f;   // chk stays 0 exactly while every value is finite
  auto take = [&](float a) {
    m = fmaxf(m, fabsf(a));
    chk = __fmaf_rn(a, 0.f, chk);
  };
  const size_t stride = (size_t)gridDim.x * LS_ET, i0 = (size_t)blockIdx.x * LS_ET + threadIdx.x;
  if (vec) {
    const float4* v4 = reinterpret_cast<const float4*>(v);
    const size_t n4 = n / 4;
    auto take4 = [&](float4 a) { take(a.x); take(a.y); take(a.z); take(a.w); };
    size_t i = i0;
    for (; i + 3 * stride < n4; i += 4 * stride) {
      float4 a[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) a[q] = __ldg(v4 + i + q * stride);
#pragma unroll
      for (int q = 0; q < 4; ++q) take4(a[q]);
    }
    for (; i < n4; i += stride) take4(__ldg(v4 + i));
  } else {
    size_t i = i0;
    for (; i + 3 * stride < n; i += 4 * stride) {
      float a[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) a[q] = __ldg(v + i + q * stride);
#pragma unroll
      for (int q = 0; q < 4; ++q) take(a[q]);
    }
    for (; i < n; i += stride) take(__ldg(v + i));
  }
  if (chk != 0.f) atomicOr(bad, 1);   // also true for NaN
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < LS_ET / 32; ++w) m = fmaxf(m, sh[w]);
  atomicMax(reinterpret_cast<int*>(vd), __float_as_int(m));
  __threadfence();
  if (atomicAdd(count + blockIdx.y, 1u) != gridDim.x - 1) return;
  __threadfence();
  m = __int_as_float(atomicMax(reinterpret_cast<int*>(vd), 0));
  const double normal = (double)m / dx + (double)m / dy;
  const double kap = (double)b * (1.0 / ((double)dx * dx) + 1.0 / ((double)dy * dy)) * 2.0;
  const double den = normal + kap;
  vd[1] = den < 1e-9 ? 1e-3f : (float)(cfl / den);
}

cudaError_t launch_speed_dt(cudaStream_t s, const float* vn, size_t n, int nimg, float dx, float dy,
                            float cfl, float b, float* vd, unsigned* count, int* bad) {
  if (nimg < 1 || nimg > 65535) return cudaErrorInvalidValue;
  const int vec = n % 4 == 0 && reinterpret_cast<uintptr_t>(vn) % 16 == 0;
  // about 16 values per thread, and at most 8 CTAs per SM in all
  const size_t want = (n + 16 * LS_ET - 1) / (16 * LS_ET);
  const size_t cap = std::max<size_t>(1, 1184 / (size_t)nimg);
  const dim3 grid((unsigned)std::min(want, cap), nimg);
  speed_dt_kernel<<<grid, LS_ET, 0, s>>>(vn, n, vec, dx, dy, cfl, b, vd, count, bad);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- mask rendering
// render_levelset_mask (levelset_mask_renderer.cpp:7-33), Gray mode: phi (float32)
// upsampled by `scale` with pixel-centre bilinear interpolation and edge
// replication (the cv::resize INTER_LINEAR convention), then the fraction of each
// source pixel's scale x scale subpixels with phi >= 0. Upsampled coordinate X
// samples the source at u = (X + 0.5) / scale - 0.5: columns floor(u) and
// floor(u) + 1 with weights 1 - t and t, t = u - floor(u); before the first and
// from the last source column on the edge value is used alone (t = 0). The two
// passes are separable: rows first, then columns, each a product sum in FP32.
// nimg images of rows x cols lie back to back; one thread per source pixel.
__device__ __forceinline__ void bilinear_coord(int X, int n, double inv, int& i0, int& i1,
                                               float& w0, float& w1) {
  float u = (float)((X + 0.5) * inv - 0.5);
  int i = (int)floorf(u);
  float t = u - (float)i;
  if (i < 0) { i = 0; t = 0.f; }
  if (i >= n - 1) { i = n - 1; t = 0.f; }
  i0 = i;
  i1 = min(i + 1, n - 1);
  w0 = 1.f - t;
  w1 = t;
}

__global__ void render_gray_kernel(const float* __restrict__ phi, int rows, int cols, int nimg,
                                   int scale, float* __restrict__ mask) {
  const size_t per = (size_t)rows * cols;
  const size_t idx = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= per * nimg) return;
  const int img = (int)(idx / per);
  const int y = (int)((idx % per) / cols), x = (int)(idx % cols);
  const float* p = phi + (size_t)img * per;
  const double inv = 1.0 / scale;
  int inside = 0;
  for (int sy = 0; sy < scale; ++sy) {
    int r0, r1;
    float b0, b1;
    bilinear_coord(y * scale + sy, rows, inv, r0, r1, b0, b1);
    for (int sx = 0; sx < scale; ++sx) {
      int c0, c1;
      float a0, a1;
      bilinear_coord(x * scale + sx, cols, inv, c0, c1, a0, a1);
      const float h0 = __fadd_rn(__fmul_rn(p[(size_t)r0 * cols + c0], a0),
                                 __fmul_rn(p[(size_t)r0 * cols + c1], a1));
      const float h1 = __fadd_rn(__fmul_rn(p[(size_t)r1 * cols + c0], a0),
                                 __fmul_rn(p[(size_t)r1 * cols + c1], a1));
      const float v = __fadd_rn(__fmul_rn(h0, b0), __fmul_rn(h1, b1));
      inside += v >= 0.f;
    }
  }
  mask[idx] = (float)((double)inside / ((double)scale * scale));
}

__global__ void render_binary_kernel(const float* __restrict__ phi, size_t n,
                                     float* __restrict__ mask) {
  const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) mask[i] = phi[i] >= 0.f ? 1.f : 0.f;
}

cudaError_t launch_render_mask(cudaStream_t s, const float* phi, int rows, int cols, int nimg,
                               int gray, int scale, float* mask) {
  const size_t n = (size_t)rows * cols * nimg;
  const unsigned nb = (unsigned)((n + 255) / 256);
  if (gray)
    render_gray_kernel<<<nb, 256, 0, s>>>(phi, rows, cols, nimg, scale, mask);
  else
    render_binary_kernel<<<nb, 256, 0, s>>>(phi, n, mask);
  return cudaGetLastError();
}

}  // namespace litho_b200
