// LevelSetUtils::reinit_sdf (level_set_utils.cpp:290-319): two OpenCV
// distanceTransform(DIST_L2, 5) calls, i.e. the 5 x 5 chamfer distance with the float32
// weights a = 1, b = 1.4, c = 2.1969 of every pixel to the nearest pixel of the other
// class (inside: phi > level, or phi >= level when inclusive).
//
// OpenCV computes it by two raster passes, in which every row waits for the row before.
// Those passes minimise, over the feature pixels q, the chamfer norm of p - q: every
// vector is a combination of two neighbouring steps of the mask, and the steps of the
// forward pass and then those of the backward pass lie inside the box of p and q. The
// norm is the maximum of four linear functions of (|dx|, |dy|) (chamfer_norm), it grows
// with |dy|, and so only the nearest feature pixel of each column matters:
//   d(x, y) = min over x' of N(|x - x'|, g(x', y)),
// g the vertical distance in column x' to the other class of (x, y). All rows are then
// independent, and since N(k, .) >= k the search around x ends at k = d.
//
// Two kernels:
//   columns  32 columns x all rows per CTA: the class bits of the column, and for every
//            block of RI_RB rows the distances from it to the nearest row above and below
//            whose class differs from the adjacent row's (two words per column);
//   rows     one CTA per block of RI_RB rows: the signed vertical distance s of every
//            pixel (positive inside) from those words into shared memory, then the search
//            along each row: a thread takes two rows of a column as a packed FP32x2 pair,
//            both sides of x at once (the nearer of the two), the first RI_NEAR columns
//            one by one, then blocks of 32 columns by their bounds.
// The words of a block live in that block's own output rows (rows 0 and 1), which only
// its CTA reads and then overwrites: the transform needs no memory besides its output.
//
// The search is bound by issue and the min / max pipe (about 300 instructions a pixel on
// patterns of 18-57 pixels in 64-pixel cells: ncu 68 % issue active, the ALU pipe first),
// where the row-sequential form it replaces was bound by the latency of 2 rows steps of
// three barriers. Times with the printed mask, before -> after: 24 images of 1266^2 4.19 ->
// 0.55 ms, one 2048^2 image 8.5 -> 0.11 ms, 64 of 257^2 0.70 -> 0.12 ms; a single inside
// pixel, the longest searches: 84 images of 1266^2 7.9 -> 5.6 ms, one 16384^2 2020 -> 22 ms.
#include <cuda_runtime.h>

#include <algorithm>

#include "litho_internal.cuh"

namespace litho_b200 {

namespace {

constexpr int RI_RB = 8;        // rows per block
constexpr int RI_NEAR = 32;     // columns searched one by one on each side
constexpr int RI_PAD = RI_NEAR + 4;   // edge columns repeated on each side of a staged row
constexpr int RI_GRP = 8;       // 32-column blocks per group of the far search
constexpr float RI_FAR = 1e30f;       // no such row in the column
constexpr uint32_t RI_DMAX = (1u << 27) - 1;   // no such row; FP32 distances end at 2^24
constexpr size_t RI_SMEM = 220 * 1024;

// A block's word per column and side: class bits of four of its rows (bits 0-3), the
// class of the adjacent row outside the block (bit 4), and the distance from the block's
// border row to the nearest row of the other class beyond it (RI_DMAX: none, 0: the image
// ends at the block).
__device__ __forceinline__ uint32_t ri_word(uint32_t bits4, uint32_t cls, uint32_t dist) {
  return bits4 | cls << 4 | dist << 5;
}

constexpr int RI_CW = 16;        // warps of the columns kernel
constexpr int RI_CHUNK = 1024;   // words (32 rows each) staged at a time: 128 KiB

// Class bits of word w of a column: bit i is row 32 w + i (0 past the last row).
__device__ __forceinline__ uint32_t ri_load_word(const float* __restrict__ p, int rows, int cols,
                                                 int w, float level, int inclusive) {
  uint32_t b = 0;
  const int ny = min(32, rows - 32 * w);
  const float* q = p + (size_t)32 * w * cols;
  if (ny == 32) {
#pragma unroll
    for (int r = 0; r < 32; ++r) {
      const float v = __ldg(q + (size_t)r * cols);
      b |= (uint32_t)(inclusive ? v >= level : v > level) << r;
    }
  } else {
    for (int r = 0; r < ny; ++r) {
      const float v = __ldg(q + (size_t)r * cols);
      b |= (uint32_t)(inclusive ? v >= level : v > level) << r;
    }
  }
  return b;
}

// Pass 0 walks the staged chunks of words downwards and writes every block's word for the
// rows above it, pass 1 walks them upwards and writes the words for the rows below; the
// rows beyond the chunk are known by the nearest row of each class (carry). One chunk
// covers 32768 rows, and is then staged once for both passes.
__global__ void __launch_bounds__(32 * RI_CW)
reinit_columns_kernel(const float* __restrict__ phi, int rows, int cols, float level,
                      int inclusive, float* __restrict__ sdf) {
  extern __shared__ uint32_t ri_words[];   // [min(words, RI_CHUNK)][32]
  __shared__ int carry[2][32];             // nearest row of class 0, 1 beyond the chunk (-1: none)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane;
  const bool in = x < cols;
  const size_t img = (size_t)blockIdx.y * rows * cols;
  const float* p = phi + img + x;
  float* out = sdf + img + x;
  const int nw = (rows + 31) / 32, nch = (nw + RI_CHUNK - 1) / RI_CHUNK;
  const uint32_t last = rows % 32 ? (1u << (rows % 32)) - 1u : 0xffffffffu;
  for (int pass = 0; pass < 2; ++pass) {
    if (warp < 2) carry[warp][lane] = -1;
    for (int c = 0; c < nch; ++c) {
      const int w0 = (pass ? nch - 1 - c : c) * RI_CHUNK, w1 = min(nw, w0 + RI_CHUNK);
      if (pass == 0 || nch > 1)
        for (int w = w0 + warp; w < w1; w += RI_CW)
          ri_words[32 * (w - w0) + lane] = in ? ri_load_word(p, rows, cols, w, level, inclusive) : 0u;
      __syncthreads();
      // bits of word w that differ from class cls (rows of the image only)
      auto other = [&](int w, uint32_t cls) -> uint32_t {
        const uint32_t b = ri_words[32 * (w - w0) + lane];
        return (cls ? ~b : b) & (w == nw - 1 ? last : 0xffffffffu);
      };
      for (int w = w0 + warp; w < w1 && in; w += RI_CW) {
        const uint32_t W = ri_words[32 * (w - w0) + lane];
        const int ny = min(32, rows - 32 * w);
        // the class of the row next to the word and the nearest row beyond of the other one
        uint32_t wcls = 0;
        int wrow = -1;
        if (pass == 0 && w > 0) {
          wcls = w > w0 ? ri_words[32 * (w - 1 - w0) + lane] >> 31 : carry[1][lane] > carry[0][lane];
          int v = w - 1;
          while (v >= w0 && !other(v, wcls)) --v;
          wrow = v >= w0 ? 32 * v + 31 - __clz(other(v, wcls)) : carry[1 - wcls][lane];
        } else if (pass == 1 && w + 1 < nw) {
          const int a0 = carry[0][lane], a1 = carry[1][lane];
          wcls = w + 1 < w1 ? ri_words[32 * (w + 1 - w0) + lane] & 1u : a0 < 0 || (a1 >= 0 && a1 < a0);
          int v = w + 1;
          while (v < w1 && !other(v, wcls)) ++v;
          wrow = v < w1 ? 32 * v + __ffs(other(v, wcls)) - 1 : carry[1 - wcls][lane];
        }
        for (int r0 = 0; r0 < ny; r0 += RI_RB) {
          const int y0 = 32 * w + r0, rn = r0 + RI_RB;
          uint32_t cls = wcls, dist = 0;
          int row = wrow;
          if (pass == 0) {
            if (r0 > 0) {
              cls = (W >> (r0 - 1)) & 1u;
              const uint32_t o = (cls ? ~W : W) & ((1u << r0) - 1u);
              if (o) row = 32 * w + 31 - __clz(o);
              else if (w > 0 && wcls != cls) row = 32 * w - 1;
            }
            if (y0 > 0) dist = row >= 0 ? min((uint32_t)(y0 - row), RI_DMAX - 1) : RI_DMAX;
            out[(size_t)y0 * cols] = __uint_as_float(ri_word((W >> r0) & 15u, cls, dist));
          } else if (y0 + 1 < rows) {   // a block of one row has no row below
            if (rn < ny) {
              cls = (W >> rn) & 1u;
              const uint32_t o = other(w, cls) & (0xffffffffu << rn);
              if (o) row = 32 * w + __ffs(o) - 1;
              else if (w + 1 < nw && wcls != cls) row = 32 * w + 32;
            }
            if (y0 + RI_RB < rows)
              dist = row >= 0 ? min((uint32_t)(row - (y0 + RI_RB - 1)), RI_DMAX - 1) : RI_DMAX;
            out[(size_t)(y0 + 1) * cols] =
                __uint_as_float(ri_word((W >> (r0 + 4)) & 15u, cls, dist));
          }
        }
      }
      __syncthreads();
      if (nch > 1 && warp < 2) {   // class `warp`: its row of the chunk nearest to the next chunk
        const uint32_t cls = 1u - warp;
        int v = pass ? w0 : w1 - 1;
        while (v >= w0 && v < w1 && !other(v, cls)) v += pass ? 1 : -1;
        if (v >= w0 && v < w1)
          carry[warp][lane] = pass ? 32 * v + __ffs(other(v, cls)) - 1 : 32 * v + 31 - __clz(other(v, cls));
      }
      __syncthreads();
    }
  }
}

// Signed vertical distance (positive inside) of row r of a block of nv rows to the other
// class in its column, from the block's two words.
__device__ __forceinline__ float ri_vertical(uint32_t w0, uint32_t w1, int r, int nv) {
  const uint32_t bits = (w0 & 15u) | (w1 & 15u) << 4;
  const uint32_t c = (bits >> r) & 1u;
  const uint32_t o = (c ? ~bits : bits) & ((1u << nv) - 1u);
  uint32_t d = RI_DMAX;
  const uint32_t above = o & ((1u << r) - 1u), below = o >> (r + 1);
  if (above) d = r - (31 - __clz(above));
  else if (w0 >> 5) {
    // the row above the block is 1 beyond its border row; RI_DMAX stays the largest
    const uint32_t e = ((w0 >> 4) & 1u) != c ? 1u : w0 >> 5;
    if (e != RI_DMAX) d = e + r;
  }
  if (below) d = min(d, (uint32_t)__ffs(below));
  else if (w1 >> 5) {
    const uint32_t e = ((w1 >> 4) & 1u) != c ? 1u : w1 >> 5;
    if (e != RI_DMAX) d = min(d, e + (RI_RB - 1 - r));
  }
  const float f = d == RI_DMAX ? RI_FAR : (float)d;
  return c ? f : -f;
}

// Facets of the chamfer norm in (k, g), k, g >= 0: k + (c - 2) g, (c - b) k + (2b - c) g
// and the same with k and g exchanged.
constexpr double RI_B = 1.4f, RI_C = 2.1969f;
constexpr float RI_F1 = (float)(RI_C - 2.0), RI_F2 = (float)(RI_C - RI_B),
                RI_F3 = (float)(2.0 * RI_B - RI_C);
// d = min(d, N(k, max(g, 0))) for both rows of a pair: facets that grow with g stay below k
// at a negative g.
__device__ __forceinline__ float2 chamfer_norm(float k, float2 g) {
  const float2 kk = make_float2(k, k), c1 = make_float2(RI_F1, RI_F1),
               c2 = make_float2(RI_F2, RI_F2), c3 = make_float2(RI_F3, RI_F3);
  const float2 f1 = __ffma2_rn(c1, g, kk), f2 = __ffma2_rn(c3, g, __fmul2_rn(c2, kk));
  const float2 f3 = __ffma2_rn(c2, g, __fmul2_rn(c3, kk)), f4 = __ffma2_rn(c1, kk, g);
  return make_float2(fmaxf(fmaxf(fmaxf(f1.x, f2.x), f3.x), fmaxf(f4.x, k)),
                     fmaxf(fmaxf(fmaxf(f1.y, f2.y), f3.y), fmaxf(f4.y, k)));
}
__device__ __forceinline__ float2 min2(float2 a, float2 b) {
  return make_float2(fminf(a.x, b.x), fminf(a.y, b.y));
}
// The smallest distance that columns with bounds m = (min, max) of row 2p, (min, max) of
// row 2p + 1 offer the pair of signs sg.
__device__ __forceinline__ float2 ri_low(float4 m, float2 sg) {
  return make_float2(sg.x > 0.f ? m.x : -m.y, sg.y > 0.f ? m.z : -m.w);
}
__device__ __forceinline__ float4 ri_join(float4 a, float4 b) {
  return make_float4(fminf(a.x, b.x), fmaxf(a.y, b.y), fminf(a.z, b.z), fmaxf(a.w, b.w));
}

// G row pairs of a block are staged at a time, in descending order, so that the words
// (rows 0 and 1, in pair 0) are overwritten last.
template <int NT, int G>
__global__ void __launch_bounds__(NT)
reinit_rows_kernel(float* __restrict__ sdf_all, float* __restrict__ mask_all, int rows, int cols,
                   float dx) {
  extern __shared__ __align__(16) float2 ri_s[];   // [G][W] pairs (row 2p, row 2p + 1)
  const int W = cols + 2 * RI_PAD, nb = (cols + 31) / 32;
  const int ng = (nb + RI_GRP - 1) / RI_GRP;
  float4* bounds = reinterpret_cast<float4*>(ri_s + ((size_t)G * W + 1) / 2 * 2);   // [G][nb]
  float4* groups = bounds + G * nb;                                                 // [G][ng]
  const size_t img = (size_t)blockIdx.y * rows * cols;
  const int y0 = blockIdx.x * RI_RB, nv = min(RI_RB, rows - y0);
  float* sdf = sdf_all + img + (size_t)y0 * cols;
  float* mask = mask_all ? mask_all + img + (size_t)y0 * cols : nullptr;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int p0 = RI_RB / 2 - G; p0 >= 0; p0 -= G) {
    if (2 * p0 >= nv) continue;
    // ---- vertical distances of the pairs p0 .. p0 + G - 1
    for (int x = threadIdx.x; x < cols; x += NT) {
      const uint32_t w0 = __float_as_uint(sdf[x]);
      const uint32_t w1 = nv > 1 ? __float_as_uint(sdf[cols + x]) : 0u;
#pragma unroll
      for (int g = 0; g < G; ++g) {
        const int r = 2 * (p0 + g);
        float2 v = make_float2(0.f, 0.f);   // rows past the image end their search at once
        if (r < nv) v.x = ri_vertical(w0, w1, r, nv);
        if (r + 1 < nv) v.y = ri_vertical(w0, w1, r + 1, nv);
        float2* row = ri_s + g * W + RI_PAD;
        row[x] = v;
        // An edge column repeated further out offers distances of at least its own.
        if (x == 0)
          for (int k = 1; k <= RI_PAD; ++k) row[-k] = v;
        if (x == cols - 1)
          for (int k = 1; k <= RI_PAD; ++k) row[cols - 1 + k] = v;
      }
    }
    __syncthreads();
    // ---- (min, max) of every 32 columns, per row of a pair
    for (int i = warp; i < G * nb; i += NT / 32) {
      const int g = i / nb, b = i % nb;
      const float2 v = ri_s[g * W + RI_PAD + min(32 * b + lane, cols - 1)];
      float4 m = make_float4(v.x, v.x, v.y, v.y);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        m = ri_join(m, make_float4(__shfl_xor_sync(0xffffffffu, m.x, o),
                                   __shfl_xor_sync(0xffffffffu, m.y, o),
                                   __shfl_xor_sync(0xffffffffu, m.z, o),
                                   __shfl_xor_sync(0xffffffffu, m.w, o)));
      }
      if (lane == 0) bounds[i] = m;
    }
    __syncthreads();
    // and of every RI_GRP such blocks
    for (int i = threadIdx.x; i < G * ng; i += NT) {
      const int g = i / ng, b0 = (i % ng) * RI_GRP, b1 = min(b0 + RI_GRP, nb);
      float4 m = bounds[g * nb + b0];
      for (int b = b0 + 1; b < b1; ++b) m = ri_join(m, bounds[g * nb + b]);
      groups[i] = m;
    }
    __syncthreads();
    // ---- search along the rows
    for (int g = 0; g < G; ++g) {
      const int r = 2 * (p0 + g);
      if (r >= nv) break;
      const float2* row = ri_s + g * W + RI_PAD;
      for (int x = threadIdx.x; x < cols; x += NT) {
        const float2 s = row[x];
        const float2 sg = make_float2(s.x < 0.f ? -1.f : 1.f, s.y < 0.f ? -1.f : 1.f);
        float2 d = make_float2(fabsf(s.x), fabsf(s.y));
        int k = 1;
        for (; k <= RI_NEAR && fmaxf(d.x, d.y) > (float)k; k += 4) {
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 a = __fmul2_rn(row[x - k - u], sg), b = __fmul2_rn(row[x + k + u], sg);
            d = min2(d, chamfer_norm((float)(k + u), min2(a, b)));
          }
        }
        if (fmaxf(d.x, d.y) > (float)k) {
          // Far search: groups of blocks, blocks and columns outwards from x, each read only
          // where its bound is below the distances found so far.
          auto near_enough = [&](float dist, float4 m) {
            const float2 n = chamfer_norm(dist, ri_low(m, sg));
            return n.x < d.x || n.y < d.y;
          };
          auto visit = [&](int q0) {   // group q0; x may lie inside it
            const int b0 = q0 * RI_GRP, b1 = min(b0 + RI_GRP, nb);
            for (int b = b0; b < b1; ++b) {
              const int dist = max(max(32 * b - x, x - (32 * b + 31)), 0);
              if (!near_enough((float)dist, bounds[g * nb + b])) continue;
              const int xe = min(32 * b + 32, cols);
              float kf = (float)(32 * b - x);
              for (int q = 32 * b; q < xe; ++q, kf += 1.f)
                d = min2(d, chamfer_norm(fabsf(kf), __fmul2_rn(row[q], sg)));
            }
          };
          const int xg = x / (32 * RI_GRP);
          visit(xg);
          for (int j = 1; j < ng; ++j) {
            const int gl = xg - j, gr = xg + j;
            const float kl = gl >= 0 ? (float)(x - (32 * RI_GRP * (gl + 1) - 1)) : RI_FAR;
            const float kr = gr < ng ? (float)(32 * RI_GRP * gr - x) : RI_FAR;
            if (fminf(kl, kr) >= fmaxf(d.x, d.y)) break;   // and so is all that is further out
            if (gl >= 0 && near_enough(kl, groups[g * ng + gl])) visit(gl);
            if (gr < ng && near_enough(kr, groups[g * ng + gr])) visit(gr);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (r + h >= nv) break;
          const float e = h ? d.y : d.x;
          const bool inside = (h ? s.y : s.x) > 0.f;
          float v = e >= RI_FAR ? 3.402823466e38f : e * dx;   // no pixel of the other class
          if (!inside) v = -v;
          sdf[(size_t)(r + h) * cols + x] = v;
          if (mask) mask[(size_t)(r + h) * cols + x] = v >= 0.f ? 1.f : 0.f;
        }
      }
    }
    if (p0 > 0) __syncthreads();   // the staged pairs are replaced
  }
}

template <int G>
size_t ri_rows_smem(int cols) {
  const size_t W = cols + 2 * RI_PAD, nb = (cols + 31) / 32, ng = (nb + RI_GRP - 1) / RI_GRP;
  return ((G * W + 1) / 2 * 2) * sizeof(float2) + G * (nb + ng) * sizeof(float4);
}

template <int NT, int G>
cudaError_t ri_rows_launch(cudaStream_t s, int rows, int cols, float dx, float* sdf, float* mask,
                           int nimg) {
  const size_t smem = ri_rows_smem<G>(cols);
  if (smem > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(reinit_rows_kernel<NT, G>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
  }
  reinit_rows_kernel<NT, G><<<dim3((rows + RI_RB - 1) / RI_RB, nimg), NT, smem, s>>>(sdf, mask, rows,
                                                                                  cols, dx);
  return cudaGetLastError();
}

template <int NT>
cudaError_t ri_rows(cudaStream_t s, int rows, int cols, float dx, float* sdf, float* mask, int nimg) {
  // as many of the block's four row pairs at a time as shared memory holds
  if (ri_rows_smem<4>(cols) <= RI_SMEM) return ri_rows_launch<NT, 4>(s, rows, cols, dx, sdf, mask, nimg);
  if (ri_rows_smem<2>(cols) <= RI_SMEM) return ri_rows_launch<NT, 2>(s, rows, cols, dx, sdf, mask, nimg);
  return ri_rows_launch<NT, 1>(s, rows, cols, dx, sdf, mask, nimg);
}

}  // namespace

cudaError_t launch_reinit_sdf(cudaStream_t s, int rows, int cols, const float* phi, float level,
                              int inclusive, float dx, float* sdf, float* mask, int nimg,
                              int threads) {
  if (nimg < 1 || nimg > 65535 || rows < 1 || cols < 1) return cudaErrorInvalidValue;
  const size_t words = std::min<size_t>((rows + 31) / 32, RI_CHUNK) * 32 * sizeof(uint32_t);
  if (words > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(reinit_columns_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)words);
    if (e != cudaSuccess) return e;
  }
  reinit_columns_kernel<<<dim3((cols + 31) / 32, nimg), 32 * RI_CW, words, s>>>(
      phi, rows, cols, level, inclusive, sdf);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  if (threads <= 0) {
    // One CTA per SM (wide images): as many threads as fit (4096^2: 342 us, 377 us with
    // 512). Few row blocks: larger CTAs, whose rows are then the parallelism there is
    // (2048^2: 110 us with 512 threads, 121 with 256; 24 x 1266^2: 596 and 555).
    const long long ctas = (long long)((rows + RI_RB - 1) / RI_RB) * nimg;
    threads = ri_rows_smem<4>(cols) > RI_SMEM / 2 ? 1024 : ctas <= 592 ? 512 : 256;
  }
  switch (threads) {
    case 128: return ri_rows<128>(s, rows, cols, dx, sdf, mask, nimg);
    case 256: return ri_rows<256>(s, rows, cols, dx, sdf, mask, nimg);
    case 512: return ri_rows<512>(s, rows, cols, dx, sdf, mask, nimg);
    case 1024: return ri_rows<1024>(s, rows, cols, dx, sdf, mask, nimg);
    default: return cudaErrorInvalidValue;
  }
}

// A smooth test pattern (sin x cos y with a per-image phase) whose zero set crosses
// every row: the input of the timing of litho_ctx_autotune.
__global__ void chamfer_probe_kernel(float* __restrict__ p, int rows, int cols, int nimg) {
  const size_t n = (size_t)rows * cols * nimg;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % cols), y = (int)((i / cols) % rows), k = (int)(i / ((size_t)rows * cols));
    p[i] = sinf(0.031f * x + k) * cosf(0.027f * y) - 0.1f;
  }
}

cudaError_t launch_chamfer_probe(cudaStream_t s, float* p, int rows, int cols, int nimg) {
  chamfer_probe_kernel<<<1184, 256, 0, s>>>(p, rows, cols, nimg);
  return cudaGetLastError();
}

}  // namespace litho_b200
