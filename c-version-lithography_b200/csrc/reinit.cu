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
//            along each row: a thread takes two rows of a column, a warp a patch of columns
//            of all staged rows, both sides of x at once (the nearer of the two), the first
//            RI_NEAR columns one by one, then blocks of 32 columns by their bounds.
// The words of a block live in that block's own output rows (rows 0 and 1), which only
// its CTA reads and then overwrites: the transform needs no memory besides its output.
//
// The search is bound by issue and the min / max pipe (218 instructions a pixel on patterns
// of 18-57 pixels in 64-pixel cells: ncu 73 % issue active, the ALU pipe 66 %), where the
// row-sequential form it replaces was bound by the latency of 2 rows steps of three barriers.
// Times with the printed mask, row-sequential -> now: 24 images of 1266^2 4.19 -> 0.365 ms
// (rows 307 us, columns 54), one 2048^2 image 8.5 -> 0.060 ms, 64 of 257^2 0.70 -> 0.061 ms;
// a single inside pixel, long searches: 84 images of 1266^2 7.9 -> 5.0 ms, one 16384^2 2020 ->
// 19.5 ms. The longest ones, where every column on the way is nearer than the last, are those
// around one diagonal line across an otherwise empty image: batches that fill the GPU are slower
// with them than the row-sequential form was (84 images of 1266^2 8.0 -> 14.7 ms, 300 of 512^2
// 2.7 -> 4.6), smaller ones faster (one 2048^2 image 8.8 -> 1.0). So are images of a single block
// of rows (3 x 1000: 27 -> 32 us), of which one CTA does the search. Searching outwards from x
// helps sparse points (300 of 512^2, one pixel in 10^4: 2.9 -> 2.0 ms) and not the diagonal, and
// costs 4 to 12 % elsewhere in registers and steps.
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
template <bool INCL>
__device__ __forceinline__ uint32_t ri_load_word(const float* __restrict__ p, int rows, int cols,
                                                 int w, float level) {
  uint32_t b = 0;
  const int ny = min(32, rows - 32 * w);
  const float* q = p + (size_t)32 * w * cols;
  if (ny == 32) {
#pragma unroll 1
    for (int h = 0; h < 32; h += 16, q += (size_t)16 * cols) {   // 16 loads in flight
      uint32_t b16 = 0;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const float v = __ldg(q + (size_t)r * cols);
        if (INCL ? v >= level : v > level) b16 |= 1u << r;
      }
      b |= b16 << h;
    }
  } else {
    for (int r = 0; r < ny; ++r) {
      const float v = __ldg(q + (size_t)r * cols);
      if (INCL ? v >= level : v > level) b |= 1u << r;
    }
  }
  return b;
}

// Pass 0 goes down the chunks of words and writes every block's word for the rows above it,
// pass 1 goes up and writes the words for the rows below; one chunk covers 32768 rows, and is
// then staged once for both passes. A warp takes a run of words; the nearest row of either
// class beyond its run comes from the other warps' runs (near) and the chunks before (carry),
// and is then carried from block to block: the adjacent row is the nearer one, so that the
// other is the row sought. 24 images of 1266^2: 86 us with a search backwards from each word
// (divergent, 50 instructions a pixel), 54 us so.
template <bool INCL>
__global__ void __launch_bounds__(32 * RI_CW, 3)
reinit_columns_kernel(const float* __restrict__ phi, int rows, int cols, float level,
                      float* __restrict__ sdf) {
  extern __shared__ uint32_t ri_words[];   // [min(words, RI_CHUNK)][32]
  __shared__ int near[RI_CW][2][32];       // nearest row of class 0, 1 in a warp's run
  __shared__ int carry[2][32];             // and beyond the chunk
  constexpr int NONE[2] = {-1, 0x7fffffff};   // no such row above, below
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int x = blockIdx.x * 32 + lane;
  const bool in = x < cols;
  const size_t img = (size_t)blockIdx.y * rows * cols;
  const float* p = phi + img + x;
  float* out = sdf + img + x;
  const int nw = (rows + 31) / 32, nch = (nw + RI_CHUNK - 1) / RI_CHUNK;
  const uint32_t last = rows % 32 ? (1u << (rows % 32)) - 1u : 0xffffffffu;
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {
    auto nearer = [&](int a, int b) { return pass ? min(a, b) : max(a, b); };
    // the nearest of the rows of mask m in word w, or a
    auto row_of = [&](int w, uint32_t m, int a) {
      return m ? 32 * w + (pass ? __ffs(m) - 1 : 31 - __clz(m)) : a;
    };
    if (warp < 2) carry[warp][lane] = NONE[pass];
    for (int c = 0; c < nch; ++c) {
      const int w0 = (pass ? nch - 1 - c : c) * RI_CHUNK, w1 = min(nw, w0 + RI_CHUNK);
      const int per = (w1 - w0 + RI_CW - 1) / RI_CW;
      const int wa = min(w0 + warp * per, w1), wb = min(wa + per, w1);
      int a[2] = {NONE[pass], NONE[pass]};
      for (int w = wa; w < wb; ++w) {
        uint32_t& W = ri_words[32 * (w - w0) + lane];
        if (pass == 0 || nch > 1) W = in ? ri_load_word<INCL>(p, rows, cols, w, level) : 0u;
        const uint32_t b = W;
        a[0] = nearer(a[0], row_of(w, ~b & (w == nw - 1 ? last : 0xffffffffu), NONE[pass]));
        a[1] = nearer(a[1], row_of(w, b, NONE[pass]));
      }
      near[warp][0][lane] = a[0];
      near[warp][1][lane] = a[1];
      __syncthreads();
      a[0] = carry[0][lane];
      a[1] = carry[1][lane];
      for (int u = pass ? warp + 1 : 0; u < (pass ? RI_CW : warp); ++u) {
        a[0] = nearer(a[0], near[u][0][lane]);
        a[1] = nearer(a[1], near[u][1][lane]);
      }
      for (int i = wa; i < wb && in; ++i) {
        const int w = pass ? wa + wb - 1 - i : i;
        const uint32_t b = ri_words[32 * (w - w0) + lane];
        const uint32_t valid = w == nw - 1 ? last : 0xffffffffu;
        float* o = out + (size_t)(32 * w + pass) * cols;
#pragma unroll
        for (int e = 0; e < 32 / RI_RB; ++e) {
          const int r0 = RI_RB * (pass ? 32 / RI_RB - 1 - e : e);
          const int y0 = 32 * w + r0;
          if (y0 + pass < rows) {   // a block of one row has no row below
            const uint32_t cls = pass ? a[1] < a[0] : a[1] > a[0];
            const int far = pass ? max(a[0], a[1]) : min(a[0], a[1]);
            const int d = pass ? far - (y0 + RI_RB - 1) : y0 - far;
            uint32_t dist = far == NONE[pass] ? RI_DMAX : min((uint32_t)d, RI_DMAX - 1);
            if (pass ? y0 + RI_RB >= rows : y0 == 0) dist = 0;
            o[(size_t)r0 * cols] =
                __uint_as_float(ri_word((b >> (r0 + 4 * pass)) & 15u, cls, dist));
          }
          const uint32_t m = (uint32_t)((1u << RI_RB) - 1u) << r0;
          a[0] = row_of(w, ~b & valid & m, a[0]);
          a[1] = row_of(w, b & m, a[1]);
        }
      }
      __syncthreads();
      if (nch > 1) {
        if (warp < 2)
          for (int u = 0; u < RI_CW; ++u) carry[warp][lane] = nearer(carry[warp][lane], near[u][warp][lane]);
        __syncthreads();
      }
    }
  }
}

// Signed vertical distances (positive inside) of the rows of a block of nv rows to the other
// class in their column, from the block's two words: a row is 1 from the row before it when
// their classes differ, else 1 further than that row. Rows past the image: 0.
__device__ __forceinline__ void ri_vertical(uint32_t w0, uint32_t w1, int nv, float (&v)[RI_RB]) {
  const uint32_t bits = (w0 & 15u) | (w1 & 15u) << 4;
  const uint32_t diff = (bits ^ (bits >> 1)) & ((1u << (nv - 1)) - 1u);   // rows r and r + 1
  // the border row's distance beyond the block (class of the row there, word's distance)
  auto beyond = [](uint32_t w, uint32_t c) -> float {
    const uint32_t dist = w >> 5;
    if (dist == 0) return RI_FAR;
    if (((w >> 4) & 1u) != c) return 1.f;
    return dist == RI_DMAX ? RI_FAR : (float)dist;
  };
  float d = beyond(w0, bits & 1u);
  v[0] = d;
#pragma unroll
  for (int r = 1; r < RI_RB; ++r) {
    d = (diff >> (r - 1)) & 1u ? 1.f : d + 1.f;
    v[r] = d;
  }
  d = beyond(w1, bits >> (RI_RB - 1));   // a block cut by the image's end has none
#pragma unroll
  for (int r = RI_RB - 1; r >= 0; --r) {
    if (r < RI_RB - 1) d = (diff >> r) & 1u ? 1.f : d + 1.f;
    d = r < nv ? d : RI_FAR;
    const float m = fminf(v[r], d);
    v[r] = r < nv ? ((bits >> r) & 1u ? m : -m) : 0.f;
  }
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
// The same for one row and a compile-time k: its multiples are immediate operands.
__device__ __forceinline__ float chamfer_near(float k, float g) {
  const float f1 = __fmaf_rn(RI_F1, g, k), f2 = __fmaf_rn(RI_F3, g, RI_F2 * k);
  const float f3 = __fmaf_rn(RI_F2, g, RI_F3 * k), f4 = __fmaf_rn(RI_F1, k, g);
  return fmaxf(fmaxf(fmaxf(f1, f2), f3), fmaxf(f4, k));
}
__device__ __forceinline__ float redux_min(float v) {
  float r;
  asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
}
__device__ __forceinline__ float redux_max(float v) {
  float r;
  asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
  return r;
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

// Pairs of a staged row: with 8 modulo 16 the two row pairs that a half warp reads lie in
// different banks.
__host__ __device__ constexpr int ri_pitch(int cols) {
  return (cols + 2 * RI_PAD + 7) / 16 * 16 + 8;
}

// G row pairs of a block are staged at a time, in descending order, so that the words
// (rows 0 and 1, in pair 0) are overwritten last. A warp searches for a patch of 32 / G
// columns of these pairs: its lanes' distances, up to which the search runs, differ less
// over 8 x 8 pixels than over 32 x 2 (24 images of 1266^2: 464 us so far, 307 us with the patches,
// immediate multiples of k and the recurrence for the vertical distances).
template <int NT, int G>
__global__ void __launch_bounds__(NT)
reinit_rows_kernel(float* __restrict__ sdf_all, float* __restrict__ mask_all, int rows, int cols,
                   float dx) {
  extern __shared__ __align__(16) float2 ri_s[];   // [G][W] pairs (row 2p, row 2p + 1)
  const int W = ri_pitch(cols), nb = (cols + 31) / 32;
  const int ng = (nb + RI_GRP - 1) / RI_GRP;
  float4* bounds = reinterpret_cast<float4*>(ri_s + (size_t)G * W);   // [G][nb]
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
      float v[RI_RB];
      ri_vertical(w0, w1, nv, v);
#pragma unroll
      for (int p = 0; p < RI_RB / 2; ++p) {
        if (p < p0 || p >= p0 + G) continue;
        const float2 pv = make_float2(v[2 * p], v[2 * p + 1]);
        float2* row = ri_s + (p - p0) * W + RI_PAD;
        row[x] = pv;
        // An edge column repeated further out offers distances of at least its own.
        if (x == 0)
          for (int k = 1; k <= RI_PAD; ++k) row[-k] = pv;
        if (x == cols - 1)
          for (int k = 1; k <= RI_PAD; ++k) row[cols - 1 + k] = pv;
      }
    }
    __syncthreads();
    // ---- (min, max) of every 32 columns, per row of a pair
    for (int i = warp; i < G * nb; i += NT / 32) {
      const int g = i / nb, b = i % nb;
      const float2 v = ri_s[g * W + RI_PAD + min(32 * b + lane, cols - 1)];
      const float4 m = make_float4(redux_min(v.x), redux_max(v.x), redux_min(v.y), redux_max(v.y));
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
    {
      constexpr int PC = 32 / G;   // columns of a warp's patch
      const int g = lane / PC, r = 2 * (p0 + g);
      const float2* row = ri_s + g * W + RI_PAD;
      for (int x = warp * PC + lane % PC; x < cols; x += (NT / 32) * PC) {
        if (r >= nv) break;
        const float2 s = row[x];
        const float2 sg = make_float2(s.x < 0.f ? -1.f : 1.f, s.y < 0.f ? -1.f : 1.f);
        float2 d = make_float2(fabsf(s.x), fabsf(s.y));
#pragma unroll
        for (int k = 1; k <= RI_NEAR; k += 4) {
          if (!(fmaxf(d.x, d.y) > (float)k)) break;
#pragma unroll
          for (int u = 0; u < 4; ++u) {
            const float2 a = __fmul2_rn(row[x - k - u], sg), b = __fmul2_rn(row[x + k + u], sg);
            d.x = fminf(d.x, chamfer_near((float)(k + u), fminf(a.x, b.x)));
            d.y = fminf(d.y, chamfer_near((float)(k + u), fminf(a.y, b.y)));
          }
        }
        if (fmaxf(d.x, d.y) > (float)(RI_NEAR + 1)) {
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
  const size_t W = ri_pitch(cols), nb = (cols + 31) / 32, ng = (nb + RI_GRP - 1) / RI_GRP;
  return G * W * sizeof(float2) + G * (nb + ng) * sizeof(float4);
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
  auto columns = [&](auto kernel) -> cudaError_t {
    if (words > 48 * 1024) {
      const cudaError_t e = cudaFuncSetAttribute(
          kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)words);
      if (e != cudaSuccess) return e;
    }
    kernel<<<dim3((cols + 31) / 32, nimg), 32 * RI_CW, words, s>>>(phi, rows, cols, level, sdf);
    return cudaGetLastError();
  };
  const cudaError_t e = inclusive ? columns(reinit_columns_kernel<true>)
                                  : columns(reinit_columns_kernel<false>);
  if (e != cudaSuccess) return e;
  if (threads <= 0) {
    // One CTA per SM (wide images): as many threads as fit (4096^2: 195 us, 212 us with
    // 512). Few row blocks: larger CTAs, whose rows are then the parallelism there is
    // (4 x 1266^2: 84 us with 512 threads, 86 with 256 and 90 with 1024; 24 x 1266^2: 385, 365
    // and 442).
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
