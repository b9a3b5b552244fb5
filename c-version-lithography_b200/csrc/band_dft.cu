// Band-limited DFT passes of the SOCS imaging and its adjoint (FP32 SIMT path).
//
// Every SOCS kernel H_k is supported on a band S of Nr x Nc integer
// frequencies. Then (exactly, in exact arithmetic)
//   E_k(x)   = sum_{v in S} H_k(v) m(v) e^{2 pi i v.x/N},  m = DFT_N(M)|_S / N^2
//   I(x)     = sum_k w'_k |E_k(x)|^2 = sum_{d in D} c(d) e^{2 pi i d.x/N},  D = S - S
// and c(d) is obtained exactly from a Pr x Pc grid (Pr >= 2Nr-1, Pc >= 2Nc-1):
//   e_k(j) = sum_v H_k(v) m(v) e^{2 pi i v.j/P},  c(d) = DFT_P(sum_k w'_k |e_k|^2)(d)/(Pr Pc).
// The adjoint of source/utils/gradient.cpp:34-109 becomes
//   g'(d)    = DFT_N(dL/dI)|_D / N^2,   gamma(j) = sum_{d in D} g'(d) e^{2 pi i d.j/P}
//   Z_k(u)   = DFT_P(e_k gamma)(u)/(Pr Pc) = sum_v H_k(v) m(v) g'(u - v)
//   X(u)     = scale sum_k w'_k conj(H_k(u)) Z_k(u),  grad(y) = Re sum_{u in S} X(u) e^{2 pi i u.y/N}.
// So the full-resolution work is two K-independent separable passes per
// direction: a tile analysis (row DFT of a 128 x 128 tile, then its column
// contraction, giving one band partial per tile) and a row synthesis GEMM with
// a fused elementwise epilogue. The K-dependent work lives on the small grid.
#include <cuda_runtime.h>

#include <type_traits>

#include <algorithm>

#include <cuda_bf16.h>

#include "device_common.cuh"
#include "tc_ptx.cuh"

namespace litho_b200 {

// Asynchronous copies into shared memory (cp.async); ok = false zero-fills.
template <int BYTES>
__device__ __forceinline__ void cp_async(void* dst, const void* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(
                   static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
               "l"(src), "n"(BYTES), "r"(ok ? BYTES : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(LEFT) : "memory");
}

// Shared memory of a CTA (227 KiB) less the static sums of the epilogues.
constexpr size_t SMEM_CTA = 227 * 1024 - 256;

// ---------------------------------------------------------------- tile analysis
// For every 128 x 128 tile: R[y][f] = sum_x A[y][x] tw[f][x] (phase 1, f the real columns
// Re, Im of the column twiddles), then P[r][c] = sum_y T(r, y) R[y][c] (phase 2), each sum
// in increasing x or y with fmaf.
//
// Both phases are FP32 FMA work (about 120 per pixel and direction at a 35 x 35 band); what
// bounded them was latency: two CTAs per SM that loaded, waited and computed in turn (FMA
// pipe 30 % busy). The image block and twiddles of the next 32 columns are now fetched into
// registers while the current ones are multiplied (two shared buffers, one barrier per
// block), the row twiddles of phase 2 are copied asynchronously during phase 1 and kept for
// all rows, and phase 2 gives every thread RPT rows (with their conjugates when sym) x 2
// columns: 62 and 72 us (forward, adjoint) -> 45 and 45 at 2048^2. Bands whose row twiddles
// (1 KiB a row) do not fit beside the rest of a CTA's shared memory, from about 160 rows on,
// take them in equal pieces of `rows` rows (PIECES): only the first one is copied during phase 1.
constexpr int AT_NT = 256, AT_TM = 8, AT_BK = 32;
constexpr int AT_TILE = 128;             // rows, and columns of x per tile
constexpr int AT_AS = AT_TILE + 4;       // row stride of an image block [BK][128]

struct AnalysisArgs {
  const float* in;     // mode 0: A = in;  mode 1: A = (1 + cos(in)) / 2 (theta -> mask)
  float* mask_out;     // nullable (mode 1)
  int* flag;           // non-finite inputs raise flag[0]
  int N, mode;
  int vec4;            // rows are 16-byte aligned (N % 4 == 0 and an aligned base pointer)
  const float* tw;     // [2 * ncols][N] real rows (Re, Im of the column twiddles)
  int ncols;
  const float2* TY;    // [nr][N] row twiddles
  int nrows_out, nr, sym;
  int rows;            // PIECES: rows whose twiddles are staged at a time (a multiple of RPT)
  float2* part;        // [tiles][nrows_out][ncols]
};

// Row twiddles per shared row [y][ts]: every thread's RPT rows, an odd count (the copies of
// 32 consecutive y then fall into different banks).
__host__ __device__ constexpr int at_ts(int nr, int rpt) { return (nr + rpt - 1) / rpt * rpt | 1; }

template <int TN, int RPT, bool PIECES>
__global__ void __launch_bounds__(AT_NT, 2)
analysis_tile_kernel(AnalysisArgs a) {
  extern __shared__ __align__(16) float smem[];
  constexpr int BN = 16 * TN;              // real columns of this CTA
  constexpr int BS = BN + 1, RS = BN + 4;
  float* As = smem;                                    // [2][BK][AS]
  float* Bs = smem + 2 * AT_BK * AT_AS;                // [2][BK][BS]
  float* R = smem;                                     // [128][RS] (after phase 1)
  constexpr int P1 = 2 * AT_BK * (AT_AS + BS), P2 = AT_TILE * RS;
  float2* TYs = reinterpret_cast<float2*>(smem + ((P1 > P2 ? P1 : P2) + 3) / 4 * 4);   // [128][ts]
  const int rows = PIECES ? a.rows : a.nr;
  const int ts = at_ts(rows, RPT);
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  const int x0 = blockIdx.x * AT_TILE, y0 = blockIdx.y * AT_TILE;
  const int f0 = blockIdx.z * BN;
  const int Nn = 2 * a.ncols, N = a.N;
  const int nkt = (min(N - x0, AT_TILE) + AT_BK - 1) / AT_BK;
  pdl_trigger();
  // the row twiddles (constant tables), ready long before phase 2
  auto copy_rows = [&](int first) {
    for (int e = tid; e < AT_TILE * ts; e += AT_NT) {
      const int yy = e % AT_TILE, r = e / AT_TILE;
      const bool ok = first + r < a.nr && y0 + yy < N;
      cp_async<8>(TYs + yy * ts + r, a.TY + (ok ? (size_t)(first + r) * N + y0 + yy : 0), ok);
    }
    cp_async_commit();
  };
  copy_rows(0);
  float va[16], vb[2 * TN];
  // image block kt: rows (tid >> 3) + 32 q, columns 4 (tid & 7) ..; twiddle block kt: column
  // tid % 32 of the rows f tid / 32 + 8 q
  auto fetch_b = [&](int kt) {
    const int x = x0 + kt * AT_BK + (tid & 31);
#pragma unroll
    for (int q = 0; q < 2 * TN; ++q) {
      const int f = f0 + (tid >> 5) + 8 * q;
      vb[q] = f < Nn && x < N ? __ldg(a.tw + (size_t)f * N + x) : 0.f;
    }
  };
  auto fetch_a = [&](int kt) {
    const int x = x0 + kt * AT_BK + 4 * (tid & 7);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int y = y0 + (tid >> 3) + 32 * q;
      const float* p = a.in + (size_t)y * N + x;
      if (a.vec4 && y < N && x + 3 < N) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(p));
        va[4 * q] = t.x; va[4 * q + 1] = t.y; va[4 * q + 2] = t.z; va[4 * q + 3] = t.w;
      } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) va[4 * q + e] = (y < N && x + e < N) ? __ldg(p + e) : 0.f;
      }
    }
  };
  auto store_blocks = [&](int kt) {
    float* as = As + (kt & 1) * AT_BK * AT_AS;
    float* bs = Bs + (kt & 1) * AT_BK * BS;
    const int x = x0 + kt * AT_BK + 4 * (tid & 7);
    bool bad = false;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int yy = (tid >> 3) + 32 * q, y = y0 + yy;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        float v = va[4 * q + e];
        const bool in_range = y < N && x + e < N;
        bad |= !isfinite(v);   // 0 outside the image
        if (a.mode == 1) {
          v = in_range ? 0.5f * (1.f + cosf(v)) : 0.f;
          if (a.mask_out && in_range && blockIdx.z == 0) a.mask_out[(size_t)y * N + x + e] = v;
        }
        as[(4 * (tid & 7) + e) * AT_AS + yy] = v;
      }
    }
    if (bad) atomicOr(a.flag, 1);
#pragma unroll
    for (int q = 0; q < 2 * TN; ++q) bs[(tid & 31) * BS + (tid >> 5) + 8 * q] = vb[q];
  };
  fetch_b(0);
  pdl_wait();
  fetch_a(0);
  float acc[AT_TM][TN];
#pragma unroll
  for (int i = 0; i < AT_TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
  store_blocks(0);
  __syncthreads();
#pragma unroll 1
  for (int kt = 0; kt < nkt; ++kt) {
    if (kt + 1 < nkt) {
      fetch_a(kt + 1);
      fetch_b(kt + 1);
    }
    const float* as = As + (kt & 1) * AT_BK * AT_AS + ty * AT_TM;
    const float* bs = Bs + (kt & 1) * AT_BK * BS + tx;
#pragma unroll 4
    for (int kk = 0; kk < AT_BK; ++kk) {
      float av[AT_TM], bv[TN];
#pragma unroll
      for (int i = 0; i < AT_TM; i += 4) {
        const float4 t = *reinterpret_cast<const float4*>(as + kk * AT_AS + i);
        av[i] = t.x; av[i + 1] = t.y; av[i + 2] = t.z; av[i + 3] = t.w;
      }
#pragma unroll
      for (int j = 0; j < TN; ++j) bv[j] = bs[kk * BS + 16 * j];
#pragma unroll
      for (int i = 0; i < AT_TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
    if (kt + 1 < nkt) store_blocks(kt + 1);   // the other buffer: read before the last barrier
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < AT_TM; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) R[(ty * AT_TM + i) * RS + tx + 16 * j] = acc[i][j];
  cp_async_wait<0>();
  __syncthreads();
  // Phase 2: item (row group, column pair).
  const int c0 = f0 / 2, npairs = (min(BN / 2, a.ncols - c0) + 1) / 2;
  float2* out = a.part + (size_t)(blockIdx.y * gridDim.x + blockIdx.x) * a.nrows_out * a.ncols;
  for (int first = 0;; first += rows) {
    const int items = (min(rows, a.nr - first) + RPT - 1) / RPT * npairs;
    for (int it = tid; it < items; it += AT_NT) {
      const int r0 = it / npairs * RPT, cp = it % npairs, c = c0 + 2 * cp;
      float2 p[RPT][2], m[RPT][2];   // rows r, and (sym) their conjugates' rows -r
#pragma unroll
      for (int i = 0; i < RPT; ++i) p[i][0] = p[i][1] = m[i][0] = m[i][1] = make_float2(0.f, 0.f);
      const float2* t0 = TYs + r0;
      const float* rr = R + 4 * cp;
      if (!a.sym) {
#pragma unroll 4
        for (int yy = 0; yy < AT_TILE; ++yy) {
          const float4 rv = *reinterpret_cast<const float4*>(rr + yy * RS);
          const float2 ra = make_float2(rv.x, rv.y), rb = make_float2(rv.z, rv.w);
#pragma unroll
          for (int i = 0; i < RPT; ++i) {
            const float2 t = t0[yy * ts + i];
            cfma(p[i][0], t, ra);
            cfma(p[i][1], t, rb);
          }
        }
      } else {
#pragma unroll 2
        for (int yy = 0; yy < AT_TILE; ++yy) {
          const float4 rv = *reinterpret_cast<const float4*>(rr + yy * RS);
          const float2 ra = make_float2(rv.x, rv.y), rb = make_float2(rv.z, rv.w);
#pragma unroll
          for (int i = 0; i < RPT; ++i) {
            const float2 t = t0[yy * ts + i], tc = conjf2(t);
            cfma(p[i][0], t, ra);
            cfma(p[i][1], t, rb);
            cfma(m[i][0], tc, ra);
            cfma(m[i][1], tc, rb);
          }
        }
      }
#pragma unroll
      for (int i = 0; i < RPT; ++i) {
        const int r = first + r0 + i;
        if (r >= a.nr) break;
        float2* o = out + (size_t)(a.sym ? a.nr - 1 + r : r) * a.ncols + c;
        o[0] = p[i][0];
        if (c + 1 < a.ncols) o[1] = p[i][1];
        if (a.sym && r > 0) {
          o = out + (size_t)(a.nr - 1 - r) * a.ncols + c;
          o[0] = m[i][0];
          if (c + 1 < a.ncols) o[1] = m[i][1];
        }
      }
    }
    if (!PIECES || first + rows >= a.nr) break;
    __syncthreads();   // the rows in use have been read
    copy_rows(first + rows);
    cp_async_wait<0>();
    __syncthreads();
  }
}

template <int TN, int RPT, bool PIECES = false>
static cudaError_t analysis_tile_t(cudaStream_t s, AnalysisArgs a) {
  constexpr int BN = 16 * TN;
  constexpr size_t p1 = 2 * AT_BK * (AT_AS + BN + 1), p2 = AT_TILE * (BN + 4);
  constexpr size_t base = ((p1 > p2 ? p1 : p2) + 3) / 4 * 4 * sizeof(float);
  auto rows_smem = [](int rows) { return (size_t)AT_TILE * at_ts(rows, RPT) * sizeof(float2); };
  a.rows = a.nr;
  for (int pieces = 2; base + rows_smem(a.rows) > SMEM_CTA; ++pieces) {
    // no rule of its own for a tall band: pieces of the 32-column variant
    if constexpr (!PIECES) return analysis_tile_t<2, 2, true>(s, a);
    a.rows = ((a.nr + pieces - 1) / pieces + RPT - 1) / RPT * RPT;
  }
  const size_t smem = base + rows_smem(a.rows);
  cudaError_t e = cudaFuncSetAttribute(analysis_tile_kernel<TN, RPT, PIECES>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int t = (a.N + AT_TILE - 1) / AT_TILE;
  dim3 grid(t, t, (2 * a.ncols + BN - 1) / BN);
  return launch_pdl(analysis_tile_kernel<TN, RPT, PIECES>, grid, dim3(AT_NT), smem, s, a);
}

int analysis_tiles(int N) {
  const int t = (N + AT_TILE - 1) / AT_TILE;
  return t * t;
}

// Tile partials of sum_{y, x} T(a, y) A[y][x] tw(c, x) for every 128 x 128 tile:
// part[tile][a][c], tiles in row-major order of the tile grid (each tile's partials
// contiguous, so that the tensor-core epilogue writes them as one coalesced block).
// Tiles below which the columns are split over more CTAs, 8 columns each or 16: the split fills
// the SMs and repeats the loads and cosines of a tile. Evaluations with 35 x 35 frequencies, 8
// columns each / 16 / unsplit: 4 tiles 107 / 118 / 125 us, 25 tiles 121 / 133 / 137, 36 tiles 127 /
// 130 / 149, 49 tiles 129 / 135 / 156, 64 tiles 155 / 142 / 158; 81 tiles 161 / 145 / 163, 100
// tiles 167 / 168 / 162, 121 tiles 194 / 187 / 166. With 52 x 52 the first line lies between 36 and
// 49 tiles (160 / 164 and 188 / 171 us), with 21 x 21 at 49 (103 / 102).
constexpr int AT_SMALL = 32, AT_MID = 96;
cudaError_t launch_analysis(cudaStream_t s, int mode, const float* in, float* mask_out,
                            int* flag, const float* tw, int N, int ncols, const float2* TY,
                            int nrows_out, int nr, int sym, float2* part) {
  const int vec4 = (N % 4 == 0) && (reinterpret_cast<uintptr_t>(in) % 16 == 0);
  const AnalysisArgs a{in, mask_out, flag, N, mode, vec4, tw, ncols, TY, nrows_out, nr, sym, nr, part};
  const int n2 = 2 * ncols, tiles = analysis_tiles(N);
  if (tiles < AT_SMALL) return analysis_tile_t<1, 1>(s, a);
  if (tiles < AT_MID) return analysis_tile_t<2, 2>(s, a);
  if (n2 <= 32) return analysis_tile_t<2, 2>(s, a);
  if (n2 <= 48) return analysis_tile_t<3, 3>(s, a);
  if (n2 <= 64) return analysis_tile_t<4, 3>(s, a);
  if (n2 <= 80) return analysis_tile_t<5, 3>(s, a);
  if (n2 <= 96) return analysis_tile_t<6, 3>(s, a);
  return analysis_tile_t<8, 3>(s, a);
}

// out[o] = scale * sum_t part[t][o] in a fixed order: RT_G tile groups (group g sums
// tiles g, g + RT_G, ... in turn), then a fixed tree over the groups. A CTA covers
// RT_E consecutive entries, so each group's loads are coalesced.
constexpr int RT_E = 16, RT_G = 32;
__global__ void __launch_bounds__(RT_E * RT_G)
reduce_tiles_kernel(const float2* __restrict__ part, int tiles, int count, int trows,
                    float scale, float2* __restrict__ out) {
  pdl_trigger();
  pdl_wait();
  part += (size_t)blockIdx.y * tiles * count;   // image b of a batch: [b][tile][entry]
  out += (size_t)blockIdx.y * count;
  __shared__ float2 sh[RT_G][RT_E];
  const int e = threadIdx.x % RT_E, g = threadIdx.x / RT_E;
  const int o = blockIdx.x * RT_E + e;
  float2 v = make_float2(0.f, 0.f);
  if (o < count) {
#pragma unroll 8
    for (int t = g; t < tiles; t += RT_G) {
      const float2 p = __ldg(part + (size_t)t * count + o);
      v.x += p.x;
      v.y += p.y;
    }
  }
  sh[g][e] = v;
  __syncthreads();
#pragma unroll
  for (int h = RT_G / 2; h > 0; h >>= 1) {
    if (g < h) {
      sh[g][e].x += sh[g + h][e].x;
      sh[g][e].y += sh[g + h][e].y;
    }
    __syncthreads();
  }
  // Entry o of a tile block is (row, c) = (o / ncols, o % ncols), or with trows > 0
  // (column-major blocks of trows rows) (o % trows, o / trows); out is row-major.
  const int oo = trows > 0 ? (o % trows) * (count / trows) + o / trows : o;
  if (g == 0 && o < count) out[oo] = make_float2(sh[0][e].x * scale, sh[0][e].y * scale);
}

cudaError_t launch_reduce_tiles(cudaStream_t s, const float2* part, int tiles, int count,
                                float scale, float2* out, int batch, int trows) {
  return launch_pdl(reduce_tiles_kernel, dim3((count + RT_E - 1) / RT_E, batch),
                    dim3(RT_E * RT_G), 0, s, part, tiles, count, trows, scale, out);
}

// ---------------------------------------------------------------- row synthesis
// out[y][x] = sum_f AYt[f][y] * Bt[f][x], f < nf in order with fmaf, from operands stored
// with f as the slow index (row stride ld, a multiple of 4): 64 x 64 tiles, 4 x 4 pixels per
// thread. The whole inner dimension of both operands is copied asynchronously in two halves:
// one wait per half, no other barrier in the product, and several CTAs per SM overlap their
// copies, products and epilogues. The tile then goes through shared memory, so that every
// global access of the epilogue is a row of float4 and its code exists once. Half of the
// kernel's issue slots are the epilogue's (expf, division, sinf, FP64 sums), so the many
// warps of small thread tiles count for more than the FMAs per operand byte of large ones
// (8 x 8 pixels per thread: a 2048^2 CTM evaluation 215 us against 206). With 128 x 128 tiles
// and two barriers per 16 inner columns the two syntheses of 2048^2 took 48 and 47 us (FMA
// pipe 25 % busy), now 33 and 29; of 256^2 23 us, now 7. An inner dimension whose operands do
// not fit in shared memory (512 bytes per f: bands from 227 rows on) is taken in slices of ns
// (SLICES).
constexpr int SF_T = 64, SF_NT = 256, SF_SS = SF_T + 4;

template <class Epi, bool SLICES>
__global__ void __launch_bounds__(SF_NT)
synth_kernel(const float* __restrict__ AYt, const float* __restrict__ Bt, int N, int ld, int nf,
             int slice, Epi epi) {
  extern __shared__ __align__(16) float sf[];
  const int ns = SLICES ? slice : nf;
  float* As = sf;                   // [ns][64]
  float* Bs = sf + ns * SF_T;       // [ns][64]
  const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
  const int m0 = blockIdx.y * SF_T, n0 = blockIdx.x * SF_T;
  // rows f0 .. f1 - 1 of an operand, 64 floats from `first`: zeros past the row stride
  auto copy = [&](float* dst, const float* src, int f0, int f1, int first) {
    const int c = 4 * (tid % 16);
    const bool ok = first + c < ld;
    for (int f = f0 + tid / 16; f < f1; f += SF_NT / 16)
      cp_async<16>(dst + f * SF_T + c, ok ? src + (size_t)f * ld + first + c : src, ok);
  };
  pdl_trigger();
  int half = (ns + 1) / 2;
  copy(As, AYt, 0, half, m0);
  pdl_wait();   // the band operand comes from the previous kernel
  copy(Bs, Bt, 0, half, n0);
  cp_async_commit();
  copy(As, AYt, half, ns, m0);
  copy(Bs, Bt, half, ns, n0);
  cp_async_commit();
  // the epilogue's input lines into L2
  if (const float* img = epi.input()) {
    const int m = m0 + tid / 2, n = n0 + 32 * (tid % 2);
    if (tid < 2 * SF_T && m < N && n < N)
      asm volatile("prefetch.global.L2 [%0];" ::"l"(img + (size_t)m * N + n));
  }
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  auto multiply = [&](int f0, int f1) {
#pragma unroll 4
    for (int f = f0; f < f1; ++f) {
      const float4 a = *reinterpret_cast<const float4*>(As + f * SF_T + 4 * ty);
      const float4 b = *reinterpret_cast<const float4*>(Bs + f * SF_T + 4 * tx);
      const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
    }
  };
  cp_async_wait<1>();
  __syncthreads();
  multiply(0, half);
  cp_async_wait<0>();
  __syncthreads();
  multiply(half, ns);
  __syncthreads();
  for (int f0 = ns; SLICES && f0 < nf; f0 += ns) {   // the slices after the first
    const int n = min(ns, nf - f0);
    half = (n + 1) / 2;
    const float* At = AYt + (size_t)f0 * ld;
    const float* Bf = Bt + (size_t)f0 * ld;
    copy(As, At, 0, half, m0);
    copy(Bs, Bf, 0, half, n0);
    cp_async_commit();
    copy(As, At, half, n, m0);
    copy(Bs, Bf, half, n, n0);
    cp_async_commit();
    cp_async_wait<1>();
    __syncthreads();
    multiply(0, half);
    cp_async_wait<0>();
    __syncthreads();
    multiply(half, n);
    __syncthreads();
  }
  float* stage = sf;   // [64][SS], over the operands
#pragma unroll
  for (int i = 0; i < 4; ++i)
    *reinterpret_cast<float4*>(stage + (4 * ty + i) * SF_SS + 4 * tx) =
        make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  __syncthreads();
#pragma unroll 2
  for (int e = tid; e < SF_T * (SF_T / 4); e += SF_NT) {
    const int r = e / (SF_T / 4), c = 4 * (e % (SF_T / 4)), m = m0 + r, n = n0 + c;
    if (m < N && n < N)
      epi.store4(m, n, *reinterpret_cast<const float4*>(stage + r * SF_SS + c), min(4, N - n));
  }
  epi.template finish<SF_NT>();
}

int synth_ld(int N) { return (N + 3) / 4 * 4; }
int synth_blocks(int N) { return ((N + SF_T - 1) / SF_T) * ((N + SF_T - 1) / SF_T); }

template <class Epi>
static cudaError_t launch_synth(cudaStream_t s, const float* AYt, const float* Bt, int N, int nf,
                                const Epi& e, int* nblocks) {
  int ns = nf;   // equal slices
  for (int slices = 2; (size_t)2 * ns * SF_T * sizeof(float) > SMEM_CTA; ++slices)
    ns = (nf + slices - 1) / slices;
  const size_t smem = std::max((size_t)2 * ns * SF_T, (size_t)SF_T * SF_SS) * sizeof(float);
  const int t = (N + SF_T - 1) / SF_T;
  *nblocks = t * t;
  auto launch = [&](auto kernel) -> cudaError_t {
    const cudaError_t err =
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (err != cudaSuccess) return err;
    return launch_pdl(kernel, dim3(t, t, 1), dim3(SF_NT), smem, s, AYt, Bt, N, synth_ld(N), nf, ns, e);
  };
  return ns < nf ? launch(synth_kernel<Epi, true>) : launch(synth_kernel<Epi, false>);
}

cudaError_t launch_synth_resist(cudaStream_t s, const float* AYt, const float* Bt, int N, int nf,
                                const ResistEpilogue& ep, int* nblocks) {
  const int vec = N % 4 == 0 && aligned16(ep.aerial) && aligned16(ep.wafer) &&
                  aligned16(ep.target) && aligned16(ep.pe_window) && aligned16(ep.pen_window) &&
                  aligned16(ep.dldi);
  return launch_synth(s, AYt, Bt, N, nf, ResistEpi{ep, N, vec, 0.0, 0.0}, nblocks);
}

cudaError_t launch_synth_grad(cudaStream_t s, const float* AYt, const float* Bt, int N, int nf,
                              const GradEpilogue& ep, int* nblocks) {
  const int vec = N % 4 == 0 && aligned16(ep.grad_mask) && aligned16(ep.theta) &&
                  aligned16(ep.grad_theta);
  return launch_synth(s, AYt, Bt, N, nf, GradEpi{ep, N, vec, 0.0}, nblocks);
}

// ---------------------------------------------------------------- small-grid band stage
// Small tables (a few tens of KB for a 35 x 35 band) are staged in shared
// memory when they fit in SMEM_STAGE bytes; otherwise the kernels read them
// from global memory (L2-resident), with the same arithmetic.
constexpr size_t SMEM_STAGE = 200 * 1024;

// dst[i] = load(i) for i < n, the NT threads of the CTA striding through i: every
// thread issues B loads before its B shared-memory stores, so the global (L2)
// latencies of a staging pass overlap instead of adding up.
template <int NT, int B = 8, class T, class Load>
__device__ __forceinline__ void fill_batched(T* dst, int n, Load load) {
  for (int base = threadIdx.x; base < n; base += NT * B) {
    T v[B];
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int i = base + q * NT;
      if (i < n) v[q] = load(i);
    }
#pragma unroll
    for (int q = 0; q < B; ++q) {
      const int i = base + q * NT;
      if (i < n) dst[i] = v[q];
    }
  }
}

// Forward 1: grid (K, column chunks of W, batch). CTA (k, q) owns small-grid
// columns jc in [q W, q W + W): A = H_k m on the band, T = A ESc^T restricted to
// those columns (Nr x W) and e_k = ESr T (Pr x W); ik = w_k |e_k|^2. Columns are
// independent, so the split costs no recomputation. Every thread accumulates four
// adjacent columns, so one row operand from shared memory feeds four complex FMAs.
constexpr int BF_NT = 512;   // threads of the fields and Z kernels (more loads in flight while staging)
constexpr int BW_ONE = 8, BW_BATCH = 16;   // chunk widths (multiples of 4): one image, a batch
__host__ __device__ constexpr int even_up(int n) { return (n + 1) & ~1; }
__device__ __forceinline__ void cfma4(float2 (&acc)[4], float2 a, const float2* b4) {
  const float4 b01 = *reinterpret_cast<const float4*>(b4);
  const float4 b23 = *reinterpret_cast<const float4*>(b4 + 2);
  cfma(acc[0], a, make_float2(b01.x, b01.y));
  cfma(acc[1], a, make_float2(b01.z, b01.w));
  cfma(acc[2], a, make_float2(b23.x, b23.y));
  cfma(acc[3], a, make_float2(b23.z, b23.w));
}

// The small-grid tables are zero-padded DFTs of even length P = 2 n: for band frequency
// f, ES[f][j + n] = (-1)^f ES[f][j]. A transform over the P outputs folds into n:
// out[j] = Ev[j] + Od[j] and out[j + n] = Ev[j] - Od[j], Ev and Od the sums over the
// frequencies of even and odd f (each in increasing order), and a transform over the
// P inputs into n: out = sum_{j < n} ES[f][j] (in[j] + (-1)^f in[j + n]). Every kernel
// of a stage folds the same way with the same operation order, so chunked, whole-grid,
// batched and single-image launches stay bit-identical.
__device__ __forceinline__ float2 fold_sum(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 fold_diff(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

template <int W>
__global__ void __launch_bounds__(BF_NT)
band_fields_kernel(const float2* __restrict__ H, const float2* __restrict__ mband,
                   const float* __restrict__ w, int Nr, int Nc, int Pr, int Pc, int row0,
                   const float2* __restrict__ ESc_t, const float2* __restrict__ ESr_t,
                   int stage_tables, float2* __restrict__ e, float* __restrict__ ik) {
  static_assert(W % 4 == 0, "four columns per thread");
  constexpr int JB = W / 4;
  extern __shared__ __align__(16) float2 sm2[];
  const int k = blockIdx.x;
  const int j0 = blockIdx.y * W;
  const int cw = min(W, Pc - j0);
  {  // image b of a batch
    const size_t b = blockIdx.z;
    mband += b * Nr * Nc;
    e += b * gridDim.x * Pr * Pc;
    ik += b * gridDim.x * Pr * Pc;
  }
  float2* A = sm2;                      // [Nr][Nc]
  float2* T = A + even_up(Nr * Nc);     // [Nr][W]
  float2* esc = T + Nr * W;             // [Nc][W] (columns past cw are zero)
  float2* esr = esc + Nc * W;           // [Nr][Pr] (staged when stage_tables)
  pdl_trigger();
  fill_batched<BF_NT>(esc, Nc * W, [&](int i) {
    const int c = i / W, jj = i % W;
    return jj < cw ? ESc_t[(size_t)c * Pc + j0 + jj] : make_float2(0.f, 0.f);
  });
  const float2* ESR = ESr_t;
  if (stage_tables) {
    fill_batched<BF_NT>(esr, Nr * Pr, [&](int i) { return ESr_t[i]; });
    ESR = esr;
  }
  pdl_wait();
  fill_batched<BF_NT>(A, Nr * Nc, [&](int i) { return cmul(H[(size_t)k * Nr * Nc + i], mband[i]); });
  __syncthreads();
  for (int it = threadIdx.x; it < Nr * JB; it += BF_NT) {
    const int r = it / JB, jb = 4 * (it % JB);
    float2 acc[4] = {};
    for (int c = 0; c < Nc; ++c) cfma4(acc, A[r * Nc + c], esc + c * W + jb);
    *reinterpret_cast<float4*>(T + r * W + jb) = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
    *reinterpret_cast<float4*>(T + r * W + jb + 2) =
        make_float4(acc[2].x, acc[2].y, acc[3].x, acc[3].y);
  }
  __syncthreads();
  const float wk = w[k];
  // e_k rows jr and jr + Nr from the two parity classes of the band rows (fold_rows).
  const int r_even = row0 & 1;   // first r with row0 + r even
  for (int it = threadIdx.x; it < Nr * JB; it += BF_NT) {
    const int jr = it / JB, jb = 4 * (it % JB);
    float2 ev[4] = {}, od[4] = {};
    for (int r = r_even; r < Nr; r += 2) cfma4(ev, ESR[r * Pr + jr], T + r * W + jb);
    for (int r = 1 - r_even; r < Nr; r += 2) cfma4(od, ESR[r * Pr + jr], T + r * W + jb);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (jb + q >= cw) break;
      const float2 v[2] = {fold_sum(ev[q], od[q]), fold_diff(ev[q], od[q])};
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const size_t o = ((size_t)k * Pr + jr + h * Nr) * Pc + j0 + jb + q;
        e[o] = v[h];
        ik[o] = wk * (v[h].x * v[h].x + v[h].y * v[h].y);
      }
    }
  }
}

// C = A B over operands in shared memory: each thread owns an RT x 2 block of C (rows
// m0 .. m0 + RT - 1, columns 2p and 2p + 1) and adds the terms in k order with cfma, the
// operand order and summation order of the chunked kernels, so every element is
// bit-identical to theirs. Work items run pair-fastest: a warp's B loads are adjacent
// 16-byte words and its A loads one or two broadcast addresses. Column 2p takes A0, column
// 2p + 1 takes A1 (the same operand, or the two classes of a folded transform). The operands
// are read two k at a time, 16 bytes each: the shared-memory wavefronts, about as many as
// the FMAs with 8-byte A loads, are what bounds these products. A[m][k] is at A + m lda + k,
// B[k][n] at B + k ldb + n; lda and ldb even, all bases 16-byte aligned.
template <int RT, int NT, class Store>
__device__ __forceinline__ void cgemm_rt2(int M, int npairs, int Kd, const float2* __restrict__ A0,
                                          const float2* __restrict__ A1, int lda,
                                          const float2* __restrict__ B, int ldb, Store store) {
  const int rblocks = (M + RT - 1) / RT;
  for (int it = threadIdx.x; it < rblocks * npairs; it += NT) {
    const int m0 = (it / npairs) * RT, p = it % npairs;
    const float2* bp = B + 2 * p;
    int ro[RT];
#pragma unroll
    for (int i = 0; i < RT; ++i) ro[i] = min(m0 + i, M - 1) * lda;
    float2 acc[RT][2];
#pragma unroll
    for (int i = 0; i < RT; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
    int k = 0;
    for (; k + 1 < Kd; k += 2) {
      const float4 b = *reinterpret_cast<const float4*>(bp + k * ldb);
      const float4 c = *reinterpret_cast<const float4*>(bp + (k + 1) * ldb);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        const float4 a = *reinterpret_cast<const float4*>(A0 + ro[i] + k);
        cfma(acc[i][0], make_float2(a.x, a.y), make_float2(b.x, b.y));
        cfma(acc[i][0], make_float2(a.z, a.w), make_float2(c.x, c.y));
        const float4 d = A1 == A0 ? a : *reinterpret_cast<const float4*>(A1 + ro[i] + k);
        cfma(acc[i][1], make_float2(d.x, d.y), make_float2(b.z, b.w));
        cfma(acc[i][1], make_float2(d.z, d.w), make_float2(c.z, c.w));
      }
    }
    if (k < Kd) {
      const float4 b = *reinterpret_cast<const float4*>(bp + k * ldb);
#pragma unroll
      for (int i = 0; i < RT; ++i) {
        cfma(acc[i][0], A0[ro[i] + k], make_float2(b.x, b.y));
        cfma(acc[i][1], A1[ro[i] + k], make_float2(b.z, b.w));
      }
    }
#pragma unroll
    for (int i = 0; i < RT; ++i) {
      if (m0 + i < M) {
        store(m0 + i, 2 * p, acc[i][0]);
        store(m0 + i, 2 * p + 1, acc[i][1]);
      }
    }
  }
}

// C = A B folded over the output rows (the transform over P = 2 M outputs): output rows
// m and m + M of each column pair from Ev = sum over k of the parity class k0, k0 + 2,
// ... and Od = sum over the other class, each in increasing k with cfma, stored as
// Ev + Od (row m) and Ev - Od (row m + M). Each thread owns four rows x 2 columns. A[m][k] is
// at A + k lda + m (lda even): its four rows are two 16-byte words.
template <int NT, class Store>
__device__ __forceinline__ void fold_rows4(int M, int npairs, int Kd, int k0, const float2* __restrict__ A,
                                           int lda, const float2* __restrict__ B, int ldb, Store store) {
  const int rblocks = (M + 3) / 4;
  for (int it = threadIdx.x; it < rblocks * npairs; it += NT) {
    const int m0 = (it / npairs) * 4, p = it % npairs;
    float2 ev[4][2], od[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) ev[i][0] = ev[i][1] = od[i][0] = od[i][1] = make_float2(0.f, 0.f);
    auto term = [&](float2 (&acc)[4][2], int k) {
      const float4 b = *reinterpret_cast<const float4*>(B + k * ldb + 2 * p);
      const float4 a01 = *reinterpret_cast<const float4*>(A + k * lda + m0);
      const float4 a23 = *reinterpret_cast<const float4*>(A + k * lda + m0 + 2);
      const float2 av[4] = {make_float2(a01.x, a01.y), make_float2(a01.z, a01.w),
                            make_float2(a23.x, a23.y), make_float2(a23.z, a23.w)};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        cfma(acc[i][0], av[i], make_float2(b.x, b.y));
        cfma(acc[i][1], av[i], make_float2(b.z, b.w));
      }
    };
    // k0 = 1: the first term belongs to the odd class
    int k = 0;
    if (k0) term(od, k++);
    for (; k + 1 < Kd; k += 2) {
      term(ev, k);
      term(od, k + 1);
    }
    if (k < Kd) term(ev, k);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (m0 + i < M) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          store(m0 + i, 2 * p + h, fold_sum(ev[i][h], od[i][h]));
          store(m0 + i + M, 2 * p + h, fold_diff(ev[i][h], od[i][h]));
        }
      }
    }
  }
}

// Forward 1, whole small grid per CTA: grid (K, 1, batch), CTA (k, b) computes all of
// e_k = ESr (A ESc^T) (Pr x Pc) and ik = w_k |e_k|^2 for image b, every table staged
// once per CTA instead of once per column chunk. Same arithmetic as
// band_fields_kernel (bit-identical results), register-blocked: 4 rows x 2 columns of
// T and, folded over the row parity classes, 4 row pairs (jr, jr + Nr) x 2 columns of
// e_k per thread.
constexpr int BG_NT = 320;
__global__ void __launch_bounds__(BG_NT)
band_fields_whole_kernel(const float2* __restrict__ H, const float2* __restrict__ mband,
                         const float* __restrict__ w, int Nr, int Nc, int Pr, int Pc, int row0,
                         const float2* __restrict__ ESc_t, const float2* __restrict__ ESr_t,
                         float2* __restrict__ e, float* __restrict__ ik) {
  extern __shared__ __align__(16) float2 sm2[];
  const int k = blockIdx.x, NcE = even_up(Nc);
  {  // image b of a batch
    const size_t b = blockIdx.z;
    mband += b * Nr * Nc;
    e += b * gridDim.x * Pr * Pc;
    ik += b * gridDim.x * Pr * Pc;
  }
  float2* esc = sm2;                    // [Nc][Pc]
  float2* esr = esc + Nc * Pc;          // [Nr][Pr] (+ 2: the last rows' 16-byte reads)
  float2* T = esr + Nr * Pr + 2;        // [Nr][Pc]
  float2* A = T + Nr * Pc;              // [Nr][NcE]
  pdl_trigger();
  fill_batched<BG_NT>(esc, Nc * Pc, [&](int i) { return ESc_t[i]; });
  fill_batched<BG_NT>(esr, Nr * Pr, [&](int i) { return ESr_t[i]; });
  pdl_wait();
  fill_batched<BG_NT>(A, Nr * NcE, [&](int i) {
    const int r = i / NcE, c = i - r * NcE, o = r * Nc + min(c, Nc - 1);
    return cmul(H[(size_t)k * Nr * Nc + o], mband[o]);
  });
  __syncthreads();
  cgemm_rt2<4, BG_NT>(Nr, Pc / 2, Nc, A, A, NcE, esc, Pc,
                      [&](int r, int j, float2 v) { T[r * Pc + j] = v; });
  __syncthreads();
  const float wk = w[k];
  float2* ek = e + (size_t)k * Pr * Pc;
  float* ikk = ik + (size_t)k * Pr * Pc;
  fold_rows4<BG_NT>(Nr, Pc / 2, Nr, row0 & 1, esr, Pr, T, Pc, [&](int jr, int j, float2 v) {
    const size_t o = (size_t)jr * Pc + j;
    ek[o] = v;
    ikk[o] = wk * (v.x * v.x + v.y * v.y);
  });
}

static size_t fields_whole_smem(const BandGeom& g) {
  return (size_t)(g.Nc * g.Pc + g.Nr * g.Pr + 2 + g.Nr * g.Pc + g.Nr * even_up(g.Nc)) * sizeof(float2);
}

template <int W>
static size_t fields_smem(const BandGeom& g, bool staged) {
  return (size_t)(even_up(g.Nr * g.Nc) + g.Nr * W + g.Nc * W + (staged ? g.Nr * g.Pr : 0)) *
         sizeof(float2);
}
size_t band_fields_smem(const BandGeom& g) {
  return fields_smem<(BW_ONE > BW_BATCH ? BW_ONE : BW_BATCH)>(g, false);
}

// Forward 2: i[j] = sum_k ik[k][j] in k order.
__global__ void sum_k_kernel(const float* __restrict__ ik, int K, int n, float* __restrict__ iP) {
  pdl_trigger();
  pdl_wait();
  ik += (size_t)blockIdx.y * K * n;   // image b of a batch
  iP += (size_t)blockIdx.y * n;
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= n) return;
  float s = 0.f;
  for (int k = 0; k < K; ++k) s += ik[(size_t)k * n + j];
  iP[j] = s;
}

// Sum of a value over SPLIT adjacent lanes (a power of two dividing 32), added in a
// fixed order ((0 + 1) + (2 + 3) for 4); every lane of the warp must call it.
template <int SPLIT>
__device__ __forceinline__ float2 split_sum(float2 a) {
#pragma unroll
  for (int o = 1; o < SPLIT; o <<= 1) {
    a.x += __shfl_xor_sync(0xffffffffu, a.x, o);
    a.y += __shfl_xor_sync(0xffffffffu, a.y, o);
  }
  return a;
}

// Forward 3 (one CTA per band row dr >= 0): chat[dr][dc] = DFT_P(i)(dr, dc) / (Pr Pc)
// for dc in [-(Nc-1), Nc-1].
constexpr int BI_NT = 256;
__global__ void __launch_bounds__(BI_NT)
band_chat_kernel(const float* __restrict__ iP, int Nr, int Nc, int Pr, int Pc,
                 const float2* __restrict__ EDr_t, const float2* __restrict__ EDc, float inv,
                 float2* __restrict__ chat) {
  // Operands are staged with one parallel round trip; the products then run
  // from shared memory (the L2 latency chains of a per-thread loop dominated).
  extern __shared__ float2 sb[];
  const int nd = 2 * Nc - 1;
  float2* v = sb;                                    // [Pc]
  float2* ed = v + Pc;                               // [Pr]
  float2* edc = ed + Pr;                             // [Pc][nd]
  float* ip = reinterpret_cast<float*>(edc + Pc * nd);  // [Pr][Pc]
  const int dr = blockIdx.x;
  iP += (size_t)blockIdx.y * Pr * Pc;   // image b of a batch
  chat += (size_t)blockIdx.y * Nr * nd;
  pdl_trigger();
  fill_batched<BI_NT>(ed, Pr, [&](int jr) { return EDr_t[(size_t)(dr + Nr - 1) * Pr + jr]; });
  fill_batched<BI_NT>(edc, Pc * nd, [&](int i) { return EDc[i]; });
  pdl_wait();
  fill_batched<BI_NT>(ip, Pr * Pc, [&](int i) { return iP[i]; });
  __syncthreads();
  // Each output is summed by SPLIT adjacent lanes (terms sub, sub + SPLIT, ...), their
  // partial sums then added in a fixed order; whole warps iterate together.
  constexpr int SPLIT = 4, GROUPS = BI_NT / SPLIT;
  const int sub = threadIdx.x % SPLIT, grp = threadIdx.x / SPLIT;
  for (int base = 0; base < Pc; base += GROUPS) {
    const int jc = base + grp;
    float2 a = make_float2(0.f, 0.f);
    if (jc < Pc)
      for (int jr = sub; jr < Pr; jr += SPLIT) {
        const float i0 = ip[jr * Pc + jc];
        a.x = fmaf(ed[jr].x, i0, a.x); a.y = fmaf(-ed[jr].y, i0, a.y);
      }
    a = split_sum<SPLIT>(a);
    if (jc < Pc && sub == 0) v[jc] = a;
  }
  __syncthreads();
  for (int base = 0; base < nd; base += GROUPS) {
    const int dc = base + grp;
    float2 a = make_float2(0.f, 0.f);
    if (dc < nd)
      for (int jc = sub; jc < Pc; jc += SPLIT) cfma(a, v[jc], conjf2(edc[jc * nd + dc]));
    a = split_sum<SPLIT>(a);
    if (dc < nd && sub == 0) chat[(size_t)dr * nd + dc] = make_float2(a.x * inv, a.y * inv);
  }
}

// Four interleaved partial sums added as (0 + 1) + (2 + 3): the order split_sum<4>
// gives the lane sums of the per-row kernels.
__device__ __forceinline__ float2 sum4(const float2 (&a)[4]) {
  return make_float2((a[0].x + a[1].x) + (a[2].x + a[3].x), (a[0].y + a[1].y) + (a[2].y + a[3].y));
}

// Forward 3 with up to BC_DR band rows (per) per CTA: grid (ceil(Nr / per), batch). The tables and
// the image's small-grid intensity are staged once per BC_DR rows instead of once per
// row; one thread per pair of outputs keeps the four interleaved partial sums of
// band_chat_kernel and adds them in its order, so the results are bit-identical.
constexpr int BC_DR = 5;
// Rows per CTA (1 .. most) of the row-grouped small-grid kernels, whose CTAs take smem bytes. The
// rows of a CTA share the staging of its tables, but a grid below two CTAs per SM leaves SMs idle:
// few enough for BAND_CTAS CTAs. Where the tables leave room for one CTA per SM (bands from about
// 48 x 48 on), the count with the least waves x (rows + 2), the staging taking about as long as
// two rows. Evaluations of 300^2 images with 6 kernels, these rules / the first one for all bands /
// as many rows as leave 148 CTAs: 9 images of 58 x 58 frequencies 266 / 291 / 266 us, 16 images
// 317 / 318 / 346; 9 images of 40 x 64 231 / 252 / 231, 16 images of 52 x 52 288 / 288 / 303.
constexpr int BAND_CTAS = 296;
static int rows_per_cta(int rows, int batch, int most, size_t smem) {
  if (2 * (smem + 1024) <= 228 * 1024) {
    const long long per = ((long long)rows * batch + BAND_CTAS - 1) / BAND_CTAS;
    return (int)std::max<long long>(1, std::min<long long>(per, most));
  }
  int best = 1;
  long long cost = 0;
  for (int per = 1; per <= most; ++per) {
    const long long ctas = (long long)((rows + per - 1) / per) * batch;
    const long long c = (ctas + BAND_CTAS / 2 - 1) / (BAND_CTAS / 2) * (per + 2);
    if (per == 1 || c < cost) {
      best = per;
      cost = c;
    }
  }
  return best;
}
__global__ void __launch_bounds__(256)
band_chat_rows_kernel(const float* __restrict__ iP, int Nr, int Nc, int Pr, int Pc,
                      const float2* __restrict__ EDr_t, const float2* __restrict__ EDc, float inv,
                      int per, float2* __restrict__ chat) {
  extern __shared__ __align__(16) float2 sb[];
  const int nd = 2 * Nc - 1, ndE = even_up(nd);
  const int dr0 = blockIdx.x * per, nr = min(per, Nr - dr0);
  iP += (size_t)blockIdx.y * Pr * Pc;   // image b of a batch
  chat += (size_t)blockIdx.y * Nr * nd;
  float2* edc = sb;                                    // [Pc][ndE] (column nd zero)
  float2* ed = edc + Pc * ndE;                         // [BC_DR][Pr]
  float2* V = ed + BC_DR * Pr;                         // [BC_DR][Pc]
  float* ip = reinterpret_cast<float*>(V + BC_DR * Pc);  // [Pr][Pc]
  pdl_trigger();
  fill_batched<256>(ed, nr * Pr, [&](int i) {
    return EDr_t[(size_t)(dr0 + i / Pr + Nr - 1) * Pr + i % Pr];
  });
  fill_batched<256>(edc, Pc * ndE, [&](int i) {
    const int jc = i / ndE, dc = i % ndE;
    return dc < nd ? EDc[(size_t)jc * nd + dc] : make_float2(0.f, 0.f);
  });
  pdl_wait();
  fill_batched<256>(ip, Pr * Pc, [&](int i) { return iP[i]; });
  __syncthreads();
  // V[r][jc] = sum_jr conj(ed[r][jr]) ip[jr][jc], two columns per thread.
  const int pc2 = Pc / 2;
  for (int it = threadIdx.x; it < nr * pc2; it += 256) {
    const int r = it / pc2, jc = 2 * (it % pc2);
    float2 a0[4], a1[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) a0[s] = a1[s] = make_float2(0.f, 0.f);
    for (int jr0 = 0; jr0 < Pr; jr0 += 4) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int jr = jr0 + s;
        if (jr < Pr) {
          const float2 e = ed[r * Pr + jr];
          const float2 i2 = *reinterpret_cast<const float2*>(ip + jr * Pc + jc);
          a0[s].x = fmaf(e.x, i2.x, a0[s].x); a0[s].y = fmaf(-e.y, i2.x, a0[s].y);
          a1[s].x = fmaf(e.x, i2.y, a1[s].x); a1[s].y = fmaf(-e.y, i2.y, a1[s].y);
        }
      }
    }
    V[r * Pc + jc] = sum4(a0);
    V[r * Pc + jc + 1] = sum4(a1);
  }
  __syncthreads();
  // chat[dr][dc] = inv sum_jc V[r][jc] conj(EDc[jc][dc]), two outputs per thread.
  const int nd2 = ndE / 2;
  for (int it = threadIdx.x; it < nr * nd2; it += 256) {
    const int r = it / nd2, dc = 2 * (it % nd2);
    float2 a0[4], a1[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) a0[s] = a1[s] = make_float2(0.f, 0.f);
    for (int jc0 = 0; jc0 < Pc; jc0 += 4) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int jc = jc0 + s;
        if (jc < Pc) {
          const float2 v = V[r * Pc + jc];
          const float4 t = *reinterpret_cast<const float4*>(edc + jc * ndE + dc);
          cfma(a0[s], v, make_float2(t.x, -t.y));
          cfma(a1[s], v, make_float2(t.z, -t.w));
        }
      }
    }
    const float2 c0 = sum4(a0), c1 = sum4(a1);
    float2* out = chat + (size_t)(dr0 + r) * nd;
    out[dc] = make_float2(c0.x * inv, c0.y * inv);
    if (dc + 1 < nd) out[dc + 1] = make_float2(c1.x * inv, c1.y * inv);
  }
}

static size_t chat_rows_smem(const BandGeom& g) {
  const int ndE = even_up(2 * g.Nc - 1);
  return (size_t)(g.Pc * ndE + BC_DR * g.Pr + BC_DR * g.Pc) * sizeof(float2) +
         (size_t)g.Pr * g.Pc * sizeof(float);
}

static size_t chat_smem(const BandGeom& g) {
  const int nd = 2 * g.Nc - 1;
  return (size_t)(g.Pc + g.Pr + g.Pc * nd) * sizeof(float2) + (size_t)g.Pr * g.Pc * sizeof(float);
}

// Band -> image columns: Ut[2a + {0,1}][x] = kappa(a) sum_c coef[a][c] phase(c, x) for
// a 64-column x strip and 8 band rows per CTA (coefficients and phases staged).
// mode 0 (band S): phase = conj(TX[c][x]) (TX = e^{-2 pi i s_c x/N}), kappa = 1.
// mode 1 (difference set D, c in [0, 2nc-1), d = c - (nc-1)):
//   phase = d >= 0 ? conj(TX[d][x]) : TX[-d][x], kappa(a) = a > 0 ? 2 : 1 (Hermitian half).
// Rows 2*nrows .. kp-1 of Ut are zero.
// With img set (tensor-core path) the result goes
// straight into the split-BF16 operand image of the row synthesis instead of Ut:
// x tile x / 128 at img + (x / 128) * img_tile_bytes, hi of column f at
// sw128_offset(128, x % 128, f) and lo at sw128_offset(128, x % 128, kp + f).
//
// Both modes are summed over the nph = nc phase rows T_j = TX[j][x] = (t, u) as
// sum_j S_j t + D_j u. For a coefficient A of phase conj(T_j) and B of phase T_j,
// A conj(T_j) + B T_j = (A + B) t + (A.y - B.y, B.x - A.x) u, so
//   S_j = A + B, D_j = (A.y - B.y, B.x - A.x),
// with A = coef[a][j], B = 0 in mode 0 and A = coef[a][nc-1+j], B = coef[a][nc-1-j]
// (B = 0 for j = 0) in mode 1: each conjugate pair of the difference set costs one
// complex-by-real product pair instead of two complex products. Every output adds
// its terms in j order as fma(D, u, fma(S, t, acc)) per component, in every kernel
// below, so the batched and per-image expansions give bit-identical results.
constexpr int EX_X = 64, EX_NT = 256;
// Row stride of Ut ([kp][ut_ld], synth_ld).
__host__ __device__ __forceinline__ size_t ut_ld(int N) { return (size_t)((N + 3) / 4 * 4); }

// S_j and D_j of band row coef_row for phase row j, as (S.x, S.y, D.x, D.y).
__device__ __forceinline__ float4 expand_sd(const float2* __restrict__ coef_row, int mode, int nc,
                                            int j) {
  const float2 A = coef_row[mode ? nc - 1 + j : j];
  const float2 B = (mode && j > 0) ? coef_row[nc - 1 - j] : make_float2(0.f, 0.f);
  return make_float4(A.x + B.x, A.y + B.y, A.y - B.y, B.x - A.x);
}
// acc + S t + D u, lane by lane fma(D, u, fma(S, t, acc)) (packed FP32x2, the
// rounding of two scalar fmaf per lane).
__device__ __forceinline__ float2 sd_fma(float2 acc, float4 sd, float t, float u) {
  return __ffma2_rn(make_float2(sd.z, sd.w), make_float2(u, u),
                    __ffma2_rn(make_float2(sd.x, sd.y), make_float2(t, t), acc));
}
// Phase rows of an expansion: nc for the difference set, ncoef for the band S.
__host__ __device__ __forceinline__ int expand_nph(int mode, int ncoef, int nc) {
  return mode ? nc : ncoef;
}

// The accumulation and store of the expansion for one CTA of 8 PAIRS band rows, from
// its staged coefficient pairs sd [8 PAIRS][nph] and phases ph [nph][EX_X]. Each
// output is summed over j in order whatever PAIRS is.
template <int PAIRS>
__device__ __forceinline__ void expand_store(const float4* sd, const float2* ph, int nrows,
                                             int nph, int N, int mode, int kp, int a0, int x0,
                                             float* __restrict__ Ut, uint8_t* __restrict__ img,
                                             uint32_t img_tile_bytes) {
  // Thread (xx, rq): row pairs p of rows a0 + 2 (PAIRS rq + p) + {0, 1}, each pair the
  // four consecutive output columns f0 .. f0 + 3 of image row x, written as one 8- or
  // 16-byte store.
  constexpr int R = 8 * PAIRS;
  const int xx = threadIdx.x % EX_X, rq = threadIdx.x / EX_X;
  const int x = x0 + xx;
  float2 acc[2 * PAIRS];
#pragma unroll
  for (int i = 0; i < 2 * PAIRS; ++i) acc[i] = make_float2(0.f, 0.f);
  for (int j = 0; j < nph; ++j) {
    const float2 p = ph[j * EX_X + xx];
#pragma unroll
    for (int i = 0; i < 2 * PAIRS; ++i) acc[i] = sd_fma(acc[i], sd[(2 * PAIRS * rq + i) * nph + j], p.x, p.y);
  }
  if (x >= N) return;
#pragma unroll
  for (int q = 0; q < PAIRS; ++q) {
    const int ra = a0 + 2 * (PAIRS * rq + q), rb = ra + 1;
    const float ka = ra < nrows ? ((mode == 1 && ra > 0) ? 2.f : 1.f) : 0.f;
    const float kb = rb < nrows ? ((mode == 1 && rb > 0) ? 2.f : 1.f) : 0.f;
    const float4 v = make_float4(ka * acc[2 * q].x, ka * acc[2 * q].y, kb * acc[2 * q + 1].x,
                                 kb * acc[2 * q + 1].y);
    const int f0 = 2 * ra;
    if (f0 >= kp) continue;
    if (img) {
      uint8_t* tile = img + (size_t)(x / 128) * img_tile_bytes;
      const __nv_bfloat162 h01 = __floats2bfloat162_rn(v.x, v.y);
      const __nv_bfloat162 h23 = __floats2bfloat162_rn(v.z, v.w);
      const float2 f01 = __bfloat1622float2(h01), f23 = __bfloat1622float2(h23);
      const __nv_bfloat162 l01 = __floats2bfloat162_rn(v.x - f01.x, v.y - f01.y);
      const __nv_bfloat162 l23 = __floats2bfloat162_rn(v.z - f23.x, v.w - f23.y);
      uint2 hw, lw;
      hw.x = *reinterpret_cast<const uint32_t*>(&h01);
      hw.y = *reinterpret_cast<const uint32_t*>(&h23);
      lw.x = *reinterpret_cast<const uint32_t*>(&l01);
      lw.y = *reinterpret_cast<const uint32_t*>(&l23);
      *reinterpret_cast<uint2*>(tile + sw128_offset(128, x % 128, f0)) = hw;
      *reinterpret_cast<uint2*>(tile + sw128_offset(128, x % 128, kp + f0)) = lw;
    } else {
      float* o = Ut + (size_t)f0 * ut_ld(N) + x;
      o[0] = v.x;
      o[ut_ld(N)] = v.y;
      o[2 * ut_ld(N)] = v.z;
      o[3 * ut_ld(N)] = v.w;
    }
  }
  // Columns past the last row group are zero.
  if (blockIdx.y == gridDim.y - 1 && rq == 0) {
    for (int f = 2 * R * gridDim.y; f < kp; f += 4) {
      if (img) {
        uint8_t* tile = img + (size_t)(x / 128) * img_tile_bytes;
        *reinterpret_cast<uint2*>(tile + sw128_offset(128, x % 128, f)) = make_uint2(0u, 0u);
        *reinterpret_cast<uint2*>(tile + sw128_offset(128, x % 128, kp + f)) = make_uint2(0u, 0u);
      } else {
        for (int q = 0; q < 4; ++q) Ut[(size_t)(f + q) * ut_ld(N) + x] = 0.f;
      }
    }
  }
}

template <int PAIRS>
__global__ void __launch_bounds__(EX_NT)
expand_kernel(const float2* __restrict__ coef, int nrows, int ncoef, int ld,
              const float2* __restrict__ TX, int N, int mode, int nc, int kp,
              float* __restrict__ Ut, uint8_t* __restrict__ img, uint32_t img_tile_bytes) {
  constexpr int R = 8 * PAIRS;
  extern __shared__ __align__(16) float4 se[];
  const int nph = expand_nph(mode, ncoef, nc);
  float4* sd = se;                                         // [R][nph]
  float2* ph = reinterpret_cast<float2*>(se + R * nph);    // [nph][EX_X]
  const int x0 = blockIdx.x * EX_X, a0 = blockIdx.y * R;
  {  // image b of a batch
    const size_t b = blockIdx.z;
    coef += b * nrows * ld;
    if (img) img += b * ((N + 127) / 128) * (size_t)img_tile_bytes;
    else Ut += b * ut_ld(N) * kp;
  }
  pdl_trigger();
  fill_batched<EX_NT>(ph, nph * EX_X, [&](int i) {
    const int j = i / EX_X, x = x0 + i % EX_X;
    return x < N ? TX[(size_t)j * N + x] : make_float2(0.f, 0.f);
  });
  pdl_wait();
  fill_batched<EX_NT>(sd, R * nph, [&](int i) {
    const int r = i / nph, j = i % nph;
    return (a0 + r < nrows) ? expand_sd(coef + (size_t)(a0 + r) * ld, mode, nc, j)
                            : make_float4(0.f, 0.f, 0.f, 0.f);
  });
  __syncthreads();
  expand_store<PAIRS>(sd, ph, nrows, nph, N, mode, kp, a0, x0, Ut, img, img_tile_bytes);
}

// The expansion with every band row of an x strip in one CTA (up to 64 rows): all 256
// threads stage the tables, then thread (xp, rg), rg < ceil(nrows / 8), computes image
// rows x0 + 2 xp and x0 + 2 xp + 1 for the eight band rows 8 rg .. 8 rg + 7, so each
// step over j takes one 16-byte phase load and eight 16-byte broadcast loads of
// coefficient pairs for 32 packed FMAs. The pairs are staged transposed
// (sdT[j][8 groups]); rows past nrows are zero. Same operands, order and scale as
// expand_store: bit-identical results.
constexpr int EXR_X = 64, EXR_NT = 256;
__global__ void __launch_bounds__(EXR_NT)
expand_rows_kernel(const float2* __restrict__ coef, int nrows, int ncoef, int ld,
                   const float2* __restrict__ TX, int N, int mode, int nc, int kp,
                   float* __restrict__ Ut, uint8_t* __restrict__ img, uint32_t img_tile_bytes) {
  extern __shared__ __align__(16) float4 sr4[];
  const int groups = (nrows + 7) / 8, R = 8 * groups;
  const int nph = expand_nph(mode, ncoef, nc);
  float4* sdT = sr4;                                             // [nph][R]
  float2* ph = reinterpret_cast<float2*>(sr4 + nph * R);         // [nph][EXR_X]
  const int x0 = blockIdx.x * EXR_X;
  {  // image b of a batch
    const size_t b = blockIdx.z;
    coef += b * nrows * ld;
    if (img) img += b * ((N + 127) / 128) * (size_t)img_tile_bytes;
    else Ut += b * ut_ld(N) * kp;
  }
  pdl_trigger();
  fill_batched<EXR_NT>(ph, nph * EXR_X, [&](int i) {
    const int j = i / EXR_X, x = x0 + i % EXR_X;
    return x < N ? TX[(size_t)j * N + x] : make_float2(0.f, 0.f);
  });
  pdl_wait();
  // sdT[j][r] = the pair of band row r: coalesced reads of coef, a transposed store.
  for (int base = threadIdx.x; base < R * nph; base += EXR_NT * 4) {
    float4 v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = base + q * EXR_NT, r = i / nph;
      if (i < R * nph)
        v[q] = r < nrows ? expand_sd(coef + (size_t)r * ld, mode, nc, i % nph)
                         : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int i = base + q * EXR_NT;
      if (i < R * nph) sdT[(i % nph) * R + i / nph] = v[q];
    }
  }
  __syncthreads();
  const int xp = threadIdx.x % 32, rg = threadIdx.x / 32;
  if (rg >= groups) return;   // staging helpers only
  float2 acc[8][2];
#pragma unroll
  for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = make_float2(0.f, 0.f);
  for (int j = 0; j < nph; ++j) {
    const float4 p = *reinterpret_cast<const float4*>(ph + j * EXR_X + 2 * xp);
    const float4* cq = sdT + j * R + 8 * rg;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const float4 sd = cq[i];
      acc[i][0] = sd_fma(acc[i][0], sd, p.x, p.y);
      acc[i][1] = sd_fma(acc[i][1], sd, p.z, p.w);
    }
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int x = x0 + 2 * xp + h;
    if (x >= N) continue;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int ra = 8 * rg + 2 * q, rb = ra + 1;
      const float ka = ra < nrows ? ((mode == 1 && ra > 0) ? 2.f : 1.f) : 0.f;
      const float kb = rb < nrows ? ((mode == 1 && rb > 0) ? 2.f : 1.f) : 0.f;
      const float4 v = make_float4(ka * acc[2 * q][h].x, ka * acc[2 * q][h].y,
                                   kb * acc[2 * q + 1][h].x, kb * acc[2 * q + 1][h].y);
      const int f0 = 2 * ra;
      if (f0 >= kp) continue;
      if (img) {
        uint8_t* tile = img + (size_t)(x / 128) * img_tile_bytes;
        const __nv_bfloat162 h01 = __floats2bfloat162_rn(v.x, v.y);
        const __nv_bfloat162 h23 = __floats2bfloat162_rn(v.z, v.w);
        const float2 f01 = __bfloat1622float2(h01), f23 = __bfloat1622float2(h23);
        const __nv_bfloat162 l01 = __floats2bfloat162_rn(v.x - f01.x, v.y - f01.y);
        const __nv_bfloat162 l23 = __floats2bfloat162_rn(v.z - f23.x, v.w - f23.y);
        uint2 hw, lw;
        hw.x = *reinterpret_cast<const uint32_t*>(&h01);
        hw.y = *reinterpret_cast<const uint32_t*>(&h23);
        lw.x = *reinterpret_cast<const uint32_t*>(&l01);
        lw.y = *reinterpret_cast<const uint32_t*>(&l23);
        *reinterpret_cast<uint2*>(tile + sw128_offset(128, x % 128, f0)) = hw;
        *reinterpret_cast<uint2*>(tile + sw128_offset(128, x % 128, kp + f0)) = lw;
      } else {
        float* o = Ut + (size_t)f0 * ut_ld(N) + x;
      o[0] = v.x;
      o[ut_ld(N)] = v.y;
      o[2 * ut_ld(N)] = v.z;
      o[3 * ut_ld(N)] = v.w;
      }
    }
    // Columns past the last row group are zero.
    if (rg == 0) {
      for (int f = 2 * R; f < kp; f += 4) {
        if (img) {
          uint8_t* tile = img + (size_t)(x / 128) * img_tile_bytes;
          *reinterpret_cast<uint2*>(tile + sw128_offset(128, x % 128, f)) = make_uint2(0u, 0u);
          *reinterpret_cast<uint2*>(tile + sw128_offset(128, x % 128, kp + f)) = make_uint2(0u, 0u);
        } else {
          for (int q = 0; q < 4; ++q) Ut[(size_t)(f + q) * ut_ld(N) + x] = 0.f;
        }
      }
    }
  }
}

template <int PAIRS>
static cudaError_t launch_expand_t(cudaStream_t s, const float2* coef, int nrows, int ncoef,
                                   int ld, const float2* TX, int N, int mode, int nc, int kp,
                                   float* Ut, void* img, int batch) {
  constexpr int R = 8 * PAIRS;
  // Split-BF16 image tile: 128 rows x [hi | lo] of kp columns, in 64-column atoms.
  const uint32_t img_tile_bytes = (uint32_t)((2 * kp + 63) / 64) * 128u * 128u;
  const int nph = expand_nph(mode, ncoef, nc);
  const size_t smem = (size_t)R * nph * sizeof(float4) + (size_t)nph * EX_X * sizeof(float2);
  cudaError_t e = cudaFuncSetAttribute(expand_kernel<PAIRS>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  dim3 grid((N + EX_X - 1) / EX_X, (nrows + R - 1) / R, batch);
  return launch_pdl(expand_kernel<PAIRS>, grid, dim3(EX_NT), smem, s, coef, nrows, ncoef, ld, TX,
                    N, mode, nc, kp, Ut, static_cast<uint8_t*>(img), img_tile_bytes);
}

// Batches take 16 rows per CTA (fewer phase-table stagings, more reuse of each phase),
// single images 8 (more CTAs); the results are the same.
static cudaError_t launch_expand(cudaStream_t s, const float2* coef, int nrows, int ncoef, int ld,
                                 const float2* TX, int N, int mode, int nc, int kp, float* Ut,
                                 void* img, int batch) {
  if (batch >= 8 && nrows <= 64) {
    // Every band row of an x strip in one CTA (enough CTAs from 8 images on).
    const int R = 8 * ((nrows + 7) / 8);
    const uint32_t img_tile_bytes = (uint32_t)((2 * kp + 63) / 64) * 128u * 128u;
    const int nph = expand_nph(mode, ncoef, nc);
    const size_t smem = (size_t)nph * R * sizeof(float4) + (size_t)nph * EXR_X * sizeof(float2);
    cudaError_t e = cudaFuncSetAttribute(expand_rows_kernel,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    return launch_pdl(expand_rows_kernel, dim3((N + EXR_X - 1) / EXR_X, 1, batch),
                      dim3(EXR_NT), smem, s, coef, nrows, ncoef, ld, TX, N, mode, nc, kp, Ut,
                      static_cast<uint8_t*>(img), img_tile_bytes);
  }
  return batch >= 4 ? launch_expand_t<2>(s, coef, nrows, ncoef, ld, TX, N, mode, nc, kp, Ut, img, batch)
                    : launch_expand_t<1>(s, coef, nrows, ncoef, ld, TX, N, mode, nc, kp, Ut, img, batch);
}

static size_t z_whole_smem(const BandGeom& g);

// Whole small grid per CTA (width BW_WHOLE, or by default from 8 images on) where both
// whole-grid kernels' tables fit in shared memory.
static bool band_whole(const BandGeom& g, int batch, int width) {
  if (fields_whole_smem(g) > SMEM_STAGE || z_whole_smem(g) > SMEM_STAGE) return false;
  return width > 0 ? width == BW_WHOLE : batch >= 8;
}

cudaError_t launch_band_forward(cudaStream_t s, const Cache& c, Field& f, float* ik, float* iP,
                                float2* chat, float* Ut, void* img, int batch, int width) {
  const BandGeom& g = c.g;
  auto fields = [&](auto wtag) -> cudaError_t {
    constexpr int W = decltype(wtag)::value;
    const bool staged = fields_smem<W>(g, true) <= SMEM_STAGE;
    const size_t sm1 = fields_smem<W>(g, staged);
    cudaError_t e1 = cudaFuncSetAttribute(band_fields_kernel<W>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm1);
    if (e1 != cudaSuccess) return e1;
    return launch_pdl(band_fields_kernel<W>, dim3(g.K, (g.Pc + W - 1) / W, batch), dim3(BF_NT),
                      sm1, s, c.H, static_cast<const float2*>(f.mband), c.w, g.Nr, g.Nc, g.Pr,
                      g.Pc, g.row0, c.ESc_t, c.ESr_t, (int)staged, f.e, ik);
  };
  // Schedule: the autotuned one when set, else the whole small grid per CTA for large
  // batches (enough CTAs to fill the GPU) and column chunks otherwise.
  cudaError_t err;
  if (band_whole(g, batch, width)) {
    const size_t smw = fields_whole_smem(g);
    err = cudaFuncSetAttribute(band_fields_whole_kernel,
                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smw);
    if (err == cudaSuccess)
      err = launch_pdl(band_fields_whole_kernel, dim3(g.K, 1, batch), dim3(BG_NT), smw, s, c.H,
                       static_cast<const float2*>(f.mband), c.w, g.Nr, g.Nc, g.Pr, g.Pc, g.row0,
                       c.ESc_t, c.ESr_t, f.e, ik);
  } else {
    const bool wide = width > 0 ? width >= BW_BATCH : batch >= 4;
    err = wide ? fields(std::integral_constant<int, BW_BATCH>{})
               : fields(std::integral_constant<int, BW_ONE>{});
  }
  if (err != cudaSuccess) return err;
  const int n = g.Pr * g.Pc;
  err = launch_pdl(sum_k_kernel, dim3((n + 255) / 256, batch), dim3(256), 0, s,
                   static_cast<const float*>(ik), g.K, n, iP);
  if (err != cudaSuccess) return err;
  const int nd = 2 * g.Nc - 1;
  if (batch >= 4 && chat_rows_smem(g) <= SMEM_STAGE) {
    // BC_DR band rows per CTA (bit-identical to one row per CTA) once a batch fills the GPU.
    const size_t smc = chat_rows_smem(g);
    err = cudaFuncSetAttribute(band_chat_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smc);
    if (err != cudaSuccess) return err;
    const int per = rows_per_cta(g.Nr, batch, BC_DR, smc);
    err = launch_pdl(band_chat_rows_kernel, dim3((g.Nr + per - 1) / per, batch), dim3(256),
                     smc, s, static_cast<const float*>(iP), g.Nr, g.Nc, g.Pr, g.Pc, c.EDr_t, c.EDc,
                     1.f / ((float)g.Pr * (float)g.Pc), per, chat);
  } else {
    const size_t smc = chat_smem(g);
    err = cudaFuncSetAttribute(band_chat_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smc);
    if (err != cudaSuccess) return err;
    err = launch_pdl(band_chat_kernel, dim3(g.Nr, batch), dim3(BI_NT), smc, s,
                     static_cast<const float*>(iP), g.Nr, g.Nc, g.Pr, g.Pc, c.EDr_t, c.EDc,
                     1.f / ((float)g.Pr * (float)g.Pc), chat);
  }
  if (err != cudaSuccess) return err;
  return launch_expand(s, chat, g.Nr, nd, nd, c.TXDc, g.N, 1, g.Nc, g.kp_rows, Ut, img, batch);
}

// Adjoint 1 (one CTA per small-grid row jr):
//   wv[c] = sum_a EDr_t[a][jr] kappa(c) g'[a][c]   (a = dr + Nr - 1, c = dc >= 0)
//   gamma[jr][jc] = Re sum_c wv[c] EDc_t[c + Nc - 1][jc]   (gamma is real)
__global__ void __launch_bounds__(256)
band_gamma_kernel(const float2* __restrict__ gh, int Nr, int Nc, int Pr, int Pc,
                  const float2* __restrict__ EDr_t, const float2* __restrict__ EDc_t,
                  float* __restrict__ gam) {
  extern __shared__ float2 sg[];
  const int jr = blockIdx.x;
  const int na = 2 * Nr - 1;
  gh += (size_t)blockIdx.y * na * Nc;   // image b of a batch
  gam += (size_t)blockIdx.y * Pr * Pc;
  float2* wv = sg;               // [Nc]
  float2* edr = wv + Nc;         // [na]   column jr of EDr_t
  float2* ghs = edr + na;        // [na][Nc]
  float2* edc = ghs + na * Nc;   // [Nc][Pc] rows Nc-1 .. 2Nc-2 of EDc_t
  pdl_trigger();
  fill_batched<256>(edr, na, [&](int r) { return EDr_t[(size_t)r * Pr + jr]; });
  fill_batched<256>(edc, Nc * Pc, [&](int i) { return EDc_t[(size_t)(Nc - 1) * Pc + i]; });
  pdl_wait();
  fill_batched<256>(ghs, na * Nc, [&](int i) { return gh[i]; });
  __syncthreads();
  // SPLIT adjacent lanes per output, as in band_chat_kernel.
  constexpr int SPLIT = 4, GROUPS = 256 / SPLIT;
  const int sub = threadIdx.x % SPLIT, grp = threadIdx.x / SPLIT;
  for (int base = 0; base < Nc; base += GROUPS) {
    const int c = base + grp;
    float2 a = make_float2(0.f, 0.f);
    if (c < Nc)
      for (int r = sub; r < na; r += SPLIT) cfma(a, edr[r], ghs[r * Nc + c]);
    a = split_sum<SPLIT>(a);
    const float kc = c > 0 ? 2.f : 1.f;
    if (c < Nc && sub == 0) wv[c] = make_float2(kc * a.x, kc * a.y);
  }
  __syncthreads();
  for (int base = 0; base < Pc; base += GROUPS) {
    const int jc = base + grp;
    float acc = 0.f;
    if (jc < Pc)
      for (int c = sub; c < Nc; c += SPLIT) {
        const float2 t = edc[c * Pc + jc];
        acc = fmaf(wv[c].x, t.x, fmaf(-wv[c].y, t.y, acc));
      }
    acc = split_sum<SPLIT>(make_float2(acc, 0.f)).x;
    if (jc < Pc && sub == 0) gam[(size_t)jr * Pc + jc] = acc;
  }
}

// Adjoint 1 with up to BG_JR small-grid rows (per) per CTA: grid (ceil(Pr / per), batch). The
// tables and the image's g' are staged once per BG_JR rows; one thread per output (wv)
// or pair of outputs (gamma) keeps the four interleaved partial sums of
// band_gamma_kernel and adds them in its order, so the results are bit-identical.
constexpr int BG_JR = 10;
__global__ void __launch_bounds__(256)
band_gamma_rows_kernel(const float2* __restrict__ gh, int Nr, int Nc, int Pr, int Pc,
                       const float2* __restrict__ EDr_t, const float2* __restrict__ EDc_t, int per,
                       float* __restrict__ gam) {
  extern __shared__ __align__(16) float2 sg[];
  const int na = 2 * Nr - 1;
  const int jr0 = blockIdx.x * per, nj = min(per, Pr - jr0);
  gh += (size_t)blockIdx.y * na * Nc;   // image b of a batch
  gam += (size_t)blockIdx.y * Pr * Pc;
  float2* edc = sg;                  // [Nc][Pc] rows Nc-1 .. 2Nc-2 of EDc_t
  float2* ghs = edc + Nc * Pc;       // [na][Nc]
  float2* edr = ghs + na * Nc;       // [BG_JR][na]: EDr_t[a][jr0 + j]
  float2* wv = edr + BG_JR * na;     // [BG_JR][Nc]
  pdl_trigger();
  fill_batched<256>(edr, nj * na, [&](int i) {
    return EDr_t[(size_t)(i % na) * Pr + jr0 + i / na];
  });
  fill_batched<256>(edc, Nc * Pc, [&](int i) { return EDc_t[(size_t)(Nc - 1) * Pc + i]; });
  pdl_wait();
  fill_batched<256>(ghs, na * Nc, [&](int i) { return gh[i]; });
  __syncthreads();
  // wv[j][c] = kappa(c) sum_a EDr_t[a][jr] g'[a][c]
  for (int it = threadIdx.x; it < nj * Nc; it += 256) {
    const int j = it / Nc, c = it % Nc;
    float2 a[4];
#pragma unroll
    for (int s = 0; s < 4; ++s) a[s] = make_float2(0.f, 0.f);
    for (int r0 = 0; r0 < na; r0 += 4) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int r = r0 + s;
        if (r < na) cfma(a[s], edr[j * na + r], ghs[r * Nc + c]);
      }
    }
    const float2 v = sum4(a);
    const float kc = c > 0 ? 2.f : 1.f;
    wv[j * Nc + c] = make_float2(kc * v.x, kc * v.y);
  }
  __syncthreads();
  // gamma[jr][jc] = Re sum_c wv[j][c] EDc_t[c + Nc - 1][jc], two columns per thread
  const int pc2 = Pc / 2;
  for (int it = threadIdx.x; it < nj * pc2; it += 256) {
    const int j = it / pc2, jc = 2 * (it % pc2);
    float a0[4] = {0.f, 0.f, 0.f, 0.f}, a1[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c0 = 0; c0 < Nc; c0 += 4) {
#pragma unroll
      for (int s = 0; s < 4; ++s) {
        const int c = c0 + s;
        if (c < Nc) {
          const float2 w = wv[j * Nc + c];
          const float4 t = *reinterpret_cast<const float4*>(edc + c * Pc + jc);
          a0[s] = fmaf(w.x, t.x, fmaf(-w.y, t.y, a0[s]));
          a1[s] = fmaf(w.x, t.z, fmaf(-w.y, t.w, a1[s]));
        }
      }
    }
    float* out = gam + (size_t)(jr0 + j) * Pc + jc;
    out[0] = (a0[0] + a0[1]) + (a0[2] + a0[3]);
    out[1] = (a1[0] + a1[1]) + (a1[2] + a1[3]);
  }
}

static size_t gamma_rows_smem(const BandGeom& g) {
  const int na = 2 * g.Nr - 1;
  return (size_t)(g.Nc * g.Pc + na * g.Nc + BG_JR * na + BG_JR * g.Nc) * sizeof(float2);
}

static size_t gamma_smem(const BandGeom& g) {
  const int na = 2 * g.Nr - 1;
  return (size_t)(g.Nc + na + na * g.Nc + g.Nc * g.Pc) * sizeof(float2);
}

// Largest dynamic shared memory any small-grid kernel needs for this band
// (the per-kernel CTAs fall back to unstaged tables above their staging limit).
size_t band_max_smem(const BandGeom& g) {
  constexpr int WMAX = BW_ONE > BW_BATCH ? BW_ONE : BW_BATCH;
  size_t m = band_fields_smem(g);
  m = std::max(m, (size_t)(g.Pr * WMAX + g.Pc * WMAX) * sizeof(float2));
  m = std::max(m, chat_smem(g));
  m = std::max(m, gamma_smem(g));
  m = std::max(m, (size_t)(16 + EX_X) * (2 * g.Nc - 1) * sizeof(float2));   // expand, 16 rows
  return m;
}

// The folded input of the Z transform over the small-grid columns: entry i = jr Pc + jc
// of [Pr][Pc] holds, for jc < Nc, q(jr, jc) + q(jr, jc + Nc) and, for jc >= Nc,
// q(jr, jc - Nc) - q(jr, jc), where q = e_k gamma (products rounded on their own).
__device__ __forceinline__ float2 z_fold_q(const float2* __restrict__ ek,
                                           const float* __restrict__ gam, int Nc, int Pc, int i) {
  const int jr = i / Pc, jc = i % Pc, j = jc < Nc ? jc : jc - Nc;
  const size_t o0 = (size_t)jr * Pc + j, o1 = o0 + Nc;
  const float2 t0 = ek[o0], t1 = ek[o1];
  const float g0 = gam[o0], g1 = gam[o1];
  const float2 a = make_float2(__fmul_rn(t0.x, g0), __fmul_rn(t0.y, g0));
  const float2 b = make_float2(__fmul_rn(t1.x, g1), __fmul_rn(t1.y, g1));
  return jc < Nc ? fold_sum(a, b) : fold_diff(a, b);
}

// The staged product q = e_k gamma ([Pr][Pc], products by __fmul_rn) folded in place into
// the layout of z_fold_q, with the same operations; one thread per (jr, jc < Nc) pair.
__device__ __forceinline__ float2 z_product(const float2* __restrict__ ek,
                                            const float* __restrict__ gam, int i) {
  const float2 t = ek[i];
  const float g = gam[i];
  return make_float2(__fmul_rn(t.x, g), __fmul_rn(t.y, g));
}
template <int NT>
__device__ __forceinline__ void z_fold_inplace(float2* q, int Pr, int Nc, int Pc) {
  for (int i = threadIdx.x; i < Pr * Nc; i += NT) {
    const int jr = i / Nc, jc = i - jr * Nc;
    float2* row = q + jr * Pc;
    const float2 a = row[jc], b = row[jc + Nc];
    row[jc] = fold_sum(a, b);
    row[jc + Nc] = fold_diff(a, b);
  }
}

// Adjoint 2: grid (K, band column chunks of W, batch). CTA (k, q) owns band columns
// uc in [q W, q W + W): q_k = e_k gamma (Pr x Pc, staged), Z1 = q_k conj(ESc)
// restricted to those columns (Pr x W), Zk = conj(ESr_t) Z1 / (Pr Pc) (Nr x W); four
// adjacent columns per thread as in the fields kernel.
template <int W>
__global__ void __launch_bounds__(BF_NT)
band_z_kernel(const float2* __restrict__ e, const float* __restrict__ gam, int Nr, int Nc, int Pr,
              int Pc, int col0, const float2* __restrict__ ESc, const float2* __restrict__ ESr_t,
              int stage_tables, float inv, float2* __restrict__ Zk) {
  static_assert(W % 4 == 0, "four columns per thread");
  constexpr int JB = W / 4;
  extern __shared__ __align__(16) float2 sz[];
  const int k = blockIdx.x;
  const int u0 = blockIdx.y * W;
  const int uw = min(W, Nc - u0);
  {  // image b of a batch
    const size_t b = blockIdx.z;
    e += b * gridDim.x * Pr * Pc;
    gam += b * Pr * Pc;
    Zk += b * gridDim.x * Nr * Nc;
  }
  float2* Z1 = sz;                  // [Pr][W]
  float2* esc = Z1 + Pr * W;        // [Pc][W] (rows jc < Nc used; columns past uw are zero)
  float2* q = esc + Pc * W;         // [Pr][Pc]   (staged: folded, z_fold_q)
  float2* esr = q + Pr * Pc;        // [Nr][Pr]   (staged)
  const float2* ek = e + (size_t)k * Pr * Pc;
  pdl_trigger();
  fill_batched<BF_NT>(esc, Nc * W, [&](int i) {
    const int jc = i / W, uu = i % W;
    return uu < uw ? conjf2(ESc[(size_t)jc * Nc + u0 + uu]) : make_float2(0.f, 0.f);
  });
  const float2* ESR = ESr_t;
  if (stage_tables) {
    fill_batched<BF_NT>(esr, Nr * Pr, [&](int i) { return ESr_t[i]; });
    ESR = esr;
  }
  pdl_wait();
  if (stage_tables) {
    fill_batched<BF_NT>(q, Pr * Pc, [&](int i) { return z_product(ek, gam, i); });
    __syncthreads();
    z_fold_inplace<BF_NT>(q, Pr, Nc, Pc);
  }
  __syncthreads();
  // Columns u0 + jb + {0, 2} have the parity of col0, {1, 3} the other (u0, jb multiples
  // of 4): the even class takes the folded sums, the odd class the differences.
  const int cpar = col0 & 1;
  for (int it = threadIdx.x; it < Pr * JB; it += BF_NT) {
    const int jr = it / JB, jb = 4 * (it % JB);
    float2 acc[4] = {};
    for (int jc = 0; jc < Nc; ++jc) {
      float2 va, vb;
      if (stage_tables) {
        va = q[jr * Pc + (cpar ? Nc : 0) + jc];
        vb = q[jr * Pc + (cpar ? 0 : Nc) + jc];
      } else {
        const float2 vs = z_fold_q(ek, gam, Nc, Pc, jr * Pc + jc);
        const float2 vd = z_fold_q(ek, gam, Nc, Pc, jr * Pc + Nc + jc);
        va = cpar ? vd : vs;
        vb = cpar ? vs : vd;
      }
      const float4 b01 = *reinterpret_cast<const float4*>(esc + jc * W + jb);
      const float4 b23 = *reinterpret_cast<const float4*>(esc + jc * W + jb + 2);
      cfma(acc[0], va, make_float2(b01.x, b01.y));
      cfma(acc[1], vb, make_float2(b01.z, b01.w));
      cfma(acc[2], va, make_float2(b23.x, b23.y));
      cfma(acc[3], vb, make_float2(b23.z, b23.w));
    }
    *reinterpret_cast<float4*>(Z1 + jr * W + jb) = make_float4(acc[0].x, acc[0].y, acc[1].x, acc[1].y);
    *reinterpret_cast<float4*>(Z1 + jr * W + jb + 2) =
        make_float4(acc[2].x, acc[2].y, acc[3].x, acc[3].y);
  }
  __syncthreads();
  for (int it = threadIdx.x; it < Nr * JB; it += BF_NT) {
    const int ur = it / JB, jb = 4 * (it % JB);
    float2 acc[4] = {};
    for (int jr = 0; jr < Pr; ++jr) cfma4(acc, conjf2(ESR[ur * Pr + jr]), Z1 + jr * W + jb);
#pragma unroll
    for (int qq = 0; qq < 4; ++qq) {
      if (jb + qq >= uw) break;
      Zk[((size_t)k * Nr + ur) * Nc + u0 + jb + qq] =
          make_float2(acc[qq].x * inv, acc[qq].y * inv);
    }
  }
}

// Adjoint 2, whole small grid per CTA: grid (K, 1, batch), CTA (k, b) computes all of
// Zk for image b, every table staged once. Same arithmetic as band_z_kernel
// (bit-identical results); the band columns are padded to an even count with zero
// table columns, whose outputs are not stored.
constexpr int BZ_NT = 256;
__global__ void __launch_bounds__(BZ_NT)
band_z_whole_kernel(const float2* __restrict__ e, const float* __restrict__ gam, int Nr, int Nc,
                    int Pr, int Pc, int col0, const float2* __restrict__ ESc,
                    const float2* __restrict__ ESr_t, float inv, float2* __restrict__ Zk) {
  extern __shared__ __align__(16) float2 sz[];
  const int k = blockIdx.x;
  const int NcE = even_up(Nc);
  {  // image b of a batch
    const size_t b = blockIdx.z;
    e += b * gridDim.x * Pr * Pc;
    gam += b * Pr * Pc;
    Zk += b * gridDim.x * Nr * Nc;
  }
  // The second transform's table takes the place of the folded input, which is dead by
  // then: three CTAs per SM instead of two (384 CTAs for 16 images and 24 kernels fit at once).
  float2* esc = sz;                   // [Nc][NcE]
  float2* Z1 = esc + Nc * NcE;        // [Pr][NcE]
  float2* q = Z1 + Pr * NcE;          // [Pr][2][NcE]: folded sums, differences
  float2* esr = q;                    // [Nr][Pr]
  const float2* ek = e + (size_t)k * Pr * Pc;
  pdl_trigger();
  fill_batched<BZ_NT>(esc, Nc * NcE, [&](int i) {
    const int jc = i / NcE, u = i % NcE;
    return u < Nc ? conjf2(ESc[(size_t)jc * Nc + u]) : make_float2(0.f, 0.f);
  });
  pdl_wait();
  // q = e_k gamma (products rounded on their own) folded as it is read: column jc of row jr
  // holds q(jr, jc) + q(jr, jc + Nc), and NcE further on the difference.
  for (int base = threadIdx.x; base < Pr * Nc; base += BZ_NT * 4) {
    float2 t0[4], t1[4];
    float g0[4], g1[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = base + u * BZ_NT;
      if (i < Pr * Nc) {
        const int o = i / Nc * Pc + i % Nc;
        t0[u] = ek[o]; t1[u] = ek[o + Nc];
        g0[u] = gam[o]; g1[u] = gam[o + Nc];
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int i = base + u * BZ_NT;
      if (i < Pr * Nc) {
        const float2 a = make_float2(__fmul_rn(t0[u].x, g0[u]), __fmul_rn(t0[u].y, g0[u]));
        const float2 b = make_float2(__fmul_rn(t1[u].x, g1[u]), __fmul_rn(t1[u].y, g1[u]));
        float2* row = q + i / Nc * 2 * NcE + i % Nc;
        row[0] = fold_sum(a, b);
        row[NcE] = fold_diff(a, b);
      }
    }
  }
  __syncthreads();
  // Column 2p has the parity of col0: sums for an even class, differences for an odd one.
  const int off0 = (col0 & 1) ? NcE : 0;
  cgemm_rt2<5, BZ_NT>(Pr, NcE / 2, Nc, q + off0, q + NcE - off0, 2 * NcE, esc, NcE,
                      [&](int jr, int u, float2 v) { Z1[jr * NcE + u] = v; });
  __syncthreads();
  fill_batched<BZ_NT>(esr, Nr * Pr, [&](int i) { return conjf2(ESr_t[i]); });
  __syncthreads();
  float2* zk = Zk + (size_t)k * Nr * Nc;
  cgemm_rt2<3, BZ_NT>(Nr, NcE / 2, Pr, esr, esr, Pr, Z1, NcE, [&](int ur, int u, float2 v) {
    if (u < Nc) zk[(size_t)ur * Nc + u] = make_float2(v.x * inv, v.y * inv);
  });
}

static size_t z_whole_smem(const BandGeom& g) {
  const int NcE = even_up(g.Nc);
  return (size_t)(g.Nc * NcE + g.Pr * NcE + std::max(g.Pr * 2 * NcE, g.Nr * g.Pr)) * sizeof(float2);
}

// Adjoint 3: X[u] = scale sum_k w_k conj(H_k(u)) Z_k(u). Four lanes per u: lane j
// sums k = j, j + 4, ... in order (the loads of up to 8 of its k issued together),
// then the four partial sums are added in a fixed order.
constexpr int BX_SPLIT = 4;
__global__ void band_x_kernel(const float2* __restrict__ Zk, const float2* __restrict__ H,
                              const float* __restrict__ w, int K, int nb, float scale,
                              float2* __restrict__ X) {
  pdl_trigger();
  pdl_wait();
  Zk += (size_t)blockIdx.y * K * nb;   // image b of a batch
  X += (size_t)blockIdx.y * nb;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const int u = t / BX_SPLIT, j = t % BX_SPLIT;
  float2 acc = make_float2(0.f, 0.f);
  if (u < nb) {
    for (int k0 = j; k0 < K; k0 += 8 * BX_SPLIT) {
      float2 hv[8], zv[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int k = k0 + q * BX_SPLIT;
        if (k < K) {
          hv[q] = H[(size_t)k * nb + u];
          zv[q] = Zk[(size_t)k * nb + u];
        }
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int k = k0 + q * BX_SPLIT;
        if (k < K) {
          const float2 c = cmul(conjf2(hv[q]), zv[q]);
          acc.x = fmaf(w[k], c.x, acc.x);
          acc.y = fmaf(w[k], c.y, acc.y);
        }
      }
    }
  }
  // lanes 4u .. 4u + 3 are adjacent in one warp: (0 + 1) + (2 + 3)
#pragma unroll
  for (int o = 1; o < BX_SPLIT; o <<= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
  }
  if (u < nb && j == 0) X[u] = make_float2(acc.x * scale, acc.y * scale);
}

cudaError_t launch_band_adjoint(cudaStream_t s, const Cache& c, const Field& f, const float2* gh,
                                double scale, float* gam, float2* Zk, float2* X, float* Vt,
                                void* img, int batch, int width) {
  const BandGeom& g = c.g;
  cudaError_t e0;
  if (batch >= 4 && gamma_rows_smem(g) <= SMEM_STAGE) {
    // BG_JR small-grid rows per CTA (bit-identical to one row per CTA) for batches.
    const size_t smg = gamma_rows_smem(g);
    e0 = cudaFuncSetAttribute(band_gamma_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)smg);
    if (e0 != cudaSuccess) return e0;
    const int per = rows_per_cta(g.Pr, batch, BG_JR, smg);
    e0 = launch_pdl(band_gamma_rows_kernel, dim3((g.Pr + per - 1) / per, batch), dim3(256),
                    smg, s, gh, g.Nr, g.Nc, g.Pr, g.Pc, c.EDr_t, c.EDc_t, per, gam);
  } else {
    const size_t smg = gamma_smem(g);
    e0 = cudaFuncSetAttribute(band_gamma_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)smg);
    if (e0 != cudaSuccess) return e0;
    e0 = launch_pdl(band_gamma_kernel, dim3(g.Pr, batch), dim3(256), smg, s, gh, g.Nr, g.Nc, g.Pr,
                    g.Pc, c.EDr_t, c.EDc_t, gam);
  }
  if (e0 != cudaSuccess) return e0;
  auto zk = [&](auto wtag) -> cudaError_t {
    constexpr int W = decltype(wtag)::value;
    const size_t base = (size_t)(g.Pr * W + g.Pc * W) * sizeof(float2);
    const size_t full = base + (size_t)(g.Pr * g.Pc + g.Nr * g.Pr) * sizeof(float2);
    const int stage = full <= SMEM_STAGE;
    const size_t smz = stage ? full : base;
    cudaError_t e1 = cudaFuncSetAttribute(band_z_kernel<W>,
                                          cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smz);
    if (e1 != cudaSuccess) return e1;
    return launch_pdl(band_z_kernel<W>, dim3(g.K, (g.Nc + W - 1) / W, batch), dim3(BF_NT), smz, s,
                      static_cast<const float2*>(f.e), static_cast<const float*>(gam), g.Nr, g.Nc,
                      g.Pr, g.Pc, g.col0, c.ESc, c.ESr_t, stage, 1.f / ((float)g.Pr * (float)g.Pc),
                      Zk);
  };
  cudaError_t err;
  if (band_whole(g, batch, width)) {
    const size_t smw = z_whole_smem(g);
    err = cudaFuncSetAttribute(band_z_whole_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               (int)smw);
    if (err == cudaSuccess)
      err = launch_pdl(band_z_whole_kernel, dim3(g.K, 1, batch), dim3(BZ_NT), smw, s,
                       static_cast<const float2*>(f.e), static_cast<const float*>(gam), g.Nr,
                       g.Nc, g.Pr, g.Pc, g.col0, c.ESc, c.ESr_t, 1.f / ((float)g.Pr * (float)g.Pc),
                       Zk);
  } else {
    const bool wide = width > 0 ? width >= BW_BATCH : batch >= 4;
    err = wide ? zk(std::integral_constant<int, BW_BATCH>{})
               : zk(std::integral_constant<int, BW_ONE>{});
  }
  if (err != cudaSuccess) return err;
  const int nb = g.Nr * g.Nc;
  err = launch_pdl(band_x_kernel, dim3((nb * BX_SPLIT + 127) / 128, batch), dim3(128), 0, s,
                   static_cast<const float2*>(Zk), c.H, c.w, g.K, nb, (float)scale, X);
  if (err != cudaSuccess) return err;
  return launch_expand(s, X, g.Nr, g.Nc, g.Nc, c.TXSc, g.N, 0, g.Nc, g.kp_rows, Vt, img, batch);
}

// ---------------------------------------------------------------- FP64 partial sums
__global__ void sum_partials_kernel(const double* __restrict__ part, int n, int stride,
                                    double* __restrict__ out) {
  // One warp per component; lanes stride over blocks, then a fixed shuffle tree.
  pdl_trigger();
  pdl_wait();
  const int comp = blockIdx.x;
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 32) s += part[(size_t)i * stride + comp];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) out[comp] = s;
}

cudaError_t launch_sum_partials(cudaStream_t s, const double* part, int n, int stride,
                                double* out) {
  return launch_pdl(sum_partials_kernel, dim3(stride), dim3(32), 0, s, part, n, stride, out);
}

// The status words of a call (non-finite flag, wait code), handed to the host and cleared for
// the next call by one thread of the call's last kernel.
__device__ __forceinline__ void publish_status(double* status, double* host_status) {
  volatile long long* w = reinterpret_cast<volatile long long*>(status);
  *reinterpret_cast<volatile long long*>(host_status) = *w;
  *w = 0;
}

// Two partial sets in one launch: blocks [0, sa) sum a's components, the rest b's. With
// `status` it is the last kernel of its call: outputs and status go to pinned host memory.
__global__ void sum_partials2_kernel(const double* __restrict__ a, int na, int sa,
                                     double* __restrict__ out_a, const double* __restrict__ b,
                                     int nb, int sb, double* __restrict__ out_b, double* status,
                                     double* host_status) {
  pdl_trigger();
  pdl_wait();
  if (status && blockIdx.x == 0 && threadIdx.x == 0) publish_status(status, host_status);
  const bool first = (int)blockIdx.x < sa;
  const int comp = first ? blockIdx.x : blockIdx.x - sa;
  const double* part = first ? a : b;
  const int n = first ? na : nb, stride = first ? sa : sb;
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 32) s += part[(size_t)i * stride + comp];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (threadIdx.x == 0) (first ? out_a : out_b)[comp] = s;
}

cudaError_t launch_sum_partials2(cudaStream_t s, const double* a, int na, int sa, double* out_a,
                                 const double* b, int nb, int sb, double* out_b, double* status,
                                 double* host_status) {
  return launch_pdl(sum_partials2_kernel, dim3(sa + sb), dim3(32), 0, s, a, na, sa, out_a, b, nb,
                    sb, out_b, status, host_status);
}

// Per image b of a batch: out[b ldo ..][0..sa) from a + b na sa (sa components over na
// blocks) and [sa..sa+sb) from b + b nb sb, each in the fixed shuffle order. `status` as above.
__global__ void sum_partials_batch_kernel(const double* __restrict__ a, int na, int sa,
                                          const double* __restrict__ b, int nb, int sb,
                                          double* __restrict__ out, int ldo, double* status,
                                          double* host_status) {
  pdl_trigger();
  pdl_wait();
  if (status && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0)
    publish_status(status, host_status);
  const size_t img = blockIdx.y;
  const bool first = (int)blockIdx.x < sa;
  const int comp = first ? blockIdx.x : blockIdx.x - sa;
  const int n = first ? na : nb, stride = first ? sa : sb;
  const double* part = first ? a + img * na * sa : b + img * nb * sb;
  double v = 0.0;
  for (int i = threadIdx.x; i < n; i += 32) v += part[(size_t)i * stride + comp];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if (threadIdx.x == 0) out[img * ldo + blockIdx.x] = v;
}

cudaError_t launch_sum_partials_batch(cudaStream_t s, const double* a, int na, int sa,
                                      const double* b, int nb, int sb, double* out, int ldo,
                                      int batch, double* status, double* host_status) {
  return launch_pdl(sum_partials_batch_kernel, dim3(sa + sb, batch), dim3(32), 0, s, a, na, sa, b,
                    nb, sb, out, ldo, status, host_status);
}

// ---------------------------------------------------------------- results to the host
// The end of a call without such a sum kernel: the reduction header (nhead doubles) and
// `more` go to pinned host memory and the header is cleared for the next call. It stands in
// for a memset before the call and one or two copies after it, 3 us each with 3 to 13 us
// between them: imaging of 256^2 took 77 us with them and takes 71 us without, PE gradients of
// 16 masks of 512^2 212 and 191 us.
__global__ void publish_kernel(double* __restrict__ head, int nhead, double* __restrict__ host,
                               const double* __restrict__ more, int nmore,
                               double* __restrict__ host_more) {
  pdl_trigger();
  pdl_wait();
  if ((int)threadIdx.x < nhead) {
    host[threadIdx.x] = head[threadIdx.x];
    head[threadIdx.x] = 0.0;
  }
  for (int i = threadIdx.x; i < nmore; i += blockDim.x) host_more[i] = more[i];
}

cudaError_t launch_publish(cudaStream_t s, double* head, int nhead, double* host,
                           const double* more, int nmore, double* host_more) {
  return launch_pdl(publish_kernel, dim3(1), dim3(256), 0, s, head, nhead, host, more, nmore,
                    host_more);
}

// ---------------------------------------------------------------- field export
// B[r][x] = sum_c A[k][r][c] e^{2 pi i s_c x/N};  E[y][x] = sum_r e^{2 pi i s_r y/N} B[r][x].
__global__ void export_rows_kernel(const float2* __restrict__ H, const float2* __restrict__ mband,
                                   int k, int Nr, int Nc, int N, const float2* __restrict__ TXSc,
                                   float2* __restrict__ B) {
  const int r = blockIdx.y;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= N) return;
  float2 acc = make_float2(0.f, 0.f);
  for (int c = 0; c < Nc; ++c) {
    const float2 a = cmul(H[((size_t)k * Nr + r) * Nc + c], mband[(size_t)r * Nc + c]);
    cfma(acc, a, conjf2(TXSc[(size_t)c * N + x]));
  }
  B[(size_t)r * N + x] = acc;
}

__global__ void export_cols_kernel(const float2* __restrict__ B, int Nr, int N,
                                   const float2* __restrict__ TYS, float2* __restrict__ E) {
  const int y = blockIdx.y;
  const int x = blockIdx.x * blockDim.x + threadIdx.x;
  if (x >= N) return;
  float2 acc = make_float2(0.f, 0.f);
  for (int r = 0; r < Nr; ++r) cfma(acc, conjf2(TYS[(size_t)r * N + y]), B[(size_t)r * N + x]);
  E[(size_t)y * N + x] = acc;
}

cudaError_t launch_export_field(cudaStream_t s, const Cache& c, const Field& f, int k,
                                float2* tmp_rows, float2* out) {
  const BandGeom& g = c.g;
  export_rows_kernel<<<dim3((g.N + 127) / 128, g.Nr), 128, 0, s>>>(c.H, f.mband, k, g.Nr, g.Nc,
                                                                   g.N, c.TXSc, tmp_rows);
  export_cols_kernel<<<dim3((g.N + 127) / 128, g.N), 128, 0, s>>>(tmp_rows, g.Nr, g.N, c.TYS,
                                                                  out);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- PE loss and dL/dI
// Loss::pe_loss / background_penalty_loss partial sums (source/utils/loss.cpp:16-64)
// and, when dldi is set, the dL/dI of the pe_gradient* variants
// (source/utils/gradient.cpp:121-196) without the common 4 alpha.
constexpr int PL_NT = 256;
__global__ void __launch_bounds__(PL_NT)
pe_loss_kernel(const float* __restrict__ w, const float* __restrict__ t,
               const float* __restrict__ pe_win, const float* __restrict__ pen_win,
               float pe_weight, float penalty, float pen_thr, size_t n,
               float* __restrict__ dldi, double* __restrict__ partial) {
  __shared__ double sh[PL_NT / 32];
  double pe = 0.0, pen = 0.0;
  for (size_t i = (size_t)blockIdx.x * PL_NT + threadIdx.x; i < n; i += (size_t)gridDim.x * PL_NT) {
    const float W = w[i], T = t[i];
    const float pw = pe_win ? pe_win[i] : 1.f;
    const float r = W - T;
    pe += (double)r * (double)r * (double)pw;
    float s = pe_weight * r * pw;
    if (penalty != 0.f && T < 0.5f) {
      const float qw = pen_win ? pen_win[i] : pw;
      const float ex = fmaxf(W - pen_thr, 0.f);
      pen += (double)ex * (double)ex * (double)qw;
      s += penalty * ex * qw;
    }
    if (dldi) dldi[i] = s * W * (1.f - W);
  }
  const double a = block_sum<PL_NT>(pe, sh);
  const double b = block_sum<PL_NT>(pen, sh);
  if (threadIdx.x == 0) {
    partial[2 * blockIdx.x] = a;
    partial[2 * blockIdx.x + 1] = b;
  }
}

static int pe_blocks(size_t n) {
  int nb = (int)((n + PL_NT - 1) / PL_NT);
  return nb > 592 ? 592 : nb;
}

cudaError_t launch_pe_loss(cudaStream_t s, const float* w, const float* t, const float* pe_win,
                           const float* pen_win, float penalty, float pen_thr, size_t n,
                           double* partial, int* nblocks) {
  *nblocks = pe_blocks(n);
  pe_loss_kernel<<<*nblocks, PL_NT, 0, s>>>(w, t, pe_win, pen_win, 1.f, penalty, pen_thr, n,
                                            nullptr, partial);
  return cudaGetLastError();
}

cudaError_t launch_pe_dldi(cudaStream_t s, const float* w, const float* t, const float* pe_win,
                           const float* pen_win, float pe_weight, float penalty, float pen_thr,
                           size_t n, float* dldi, double* partial, int* nblocks) {
  *nblocks = pe_blocks(n);
  pe_loss_kernel<<<*nblocks, PL_NT, 0, s>>>(w, t, pe_win, pen_win, pe_weight, penalty, pen_thr,
                                            n, dldi, partial);
  return cudaGetLastError();
}

}  // namespace litho_b200
