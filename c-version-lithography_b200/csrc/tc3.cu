// Persistent, warp-specialised split-BF16 tensor-core passes (tcgen05, sm_100a).
//
// The per-tile kernels of tc2.cu run one 128 x 128 tile per CTA, two CTAs per SM,
// each CTA through its phases in order (operand copies, MMA, tensor-memory
// read-back, epilogue). The kernels here run one CTA per SM over a contiguous share
// of the work items (image z, tile row yt, tile column xt; images fastest, so
// consecutive items of a CTA share their tile's constant operand images, which
// stay in shared memory), with each phase in its own warps and the phases of
// neighbouring items overlapped:
//   * loader / epilogue warps move image data between global memory and shared or
//     tensor memory;
//   * one converged warp issues, by one elected lane, the bulk copies of the constant
//     operand images and every tcgen05.mma, and commits each MMA group to an mbarrier;
//   * the accumulators are double-buffered in tensor memory, so the epilogue of
//     item j runs while the MMAs of item j + 1 do.
// The roles hand buffers to each other through mbarriers (full / free per buffer,
// phase parity per use). Every wait is bounded and a whole warp's (pwait_warp): on
// expiry, or when another role has given up, the warp records a code in *err (first
// failure only) and leaves its loop; the MMA warp then waits (bounded) for its own
// copies and MMAs in flight, the tensor memory is released and the kernel returns.
//
// The syntheses compute the transposed accumulator D[x][y] (tensor-memory lane =
// image column x) so that the 32 lanes of a warp touch 32 consecutive pixels of an
// image row: every global access of the epilogues is a fully used 128-byte line,
// with no staging through shared memory. Per element the products and their order
// are those of the per-tile kernels (s2_mma_swapped), so images agree bit for bit.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <type_traits>

#include "device_common.cuh"
#include "tc_ptx.cuh"
#include "tc_split2.cuh"

namespace litho_b200 {

namespace {

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ uint8_t* align1024(uint8_t* p) {
  return reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(p) + 1023) &
                                    ~static_cast<uintptr_t>(1023));
}

// Bounded wait of a whole warp for the completion of the phase of `bar` with parity `parity`.
// Gives up when another role has failed (*fail) or after about 2^31 SM cycles (one second),
// then records `code` in *err (first failure wins) and returns false. Every lane gets the same
// answer: a lane that gave up alone would leave the others at the warp-wide instructions that
// follow (tcgen05.ld, shuffles, __syncwarp), which wait for it without a limit.
__device__ __forceinline__ bool pwait_warp(uint32_t bar, uint32_t parity, volatile int* fail,
                                           int* err, int code) {
  constexpr unsigned ALL = 0xffffffffu;
  if (__all_sync(ALL, tc::mbar_try_wait(bar, parity))) return true;
  const long long t0 = clock64();
  while (!__all_sync(ALL, tc::mbar_try_wait(bar, parity))) {
    if (__any_sync(ALL, *fail)) return false;
    if (__any_sync(ALL, clock64() - t0 > (1LL << 31))) {
      *fail = 1;
      atomicCAS(err, 0, code);
      return false;
    }
  }
  return true;
}

// This CTA's contiguous share [lo, hi) of `items` work items.
__device__ __forceinline__ void my_items(int items, int& lo, int& hi) {
  lo = (int)((long long)blockIdx.x * items / gridDim.x);
  hi = (int)((long long)(blockIdx.x + 1) * items / gridDim.x);
}
struct Item {
  int z, yt, xt;
};
// Item it of T x T tiles x B images, images fastest.
__device__ __forceinline__ Item item_at(int it, int T, int B) {
  Item r;
  r.z = it % B;
  const int t = it / B;
  r.xt = t % T;
  r.yt = t / T;
  return r;
}
// The item after it (no division: a role walks its items in order).
__device__ __forceinline__ Item item_next(Item it, int T, int B) {
  if (++it.z == B) {
    it.z = 0;
    if (++it.xt == T) {
      it.xt = 0;
      ++it.yt;
    }
  }
  return it;
}

// Per-item FP64 partial sums of the epilogue warps without a CTA barrier (a warp that
// leaves its loop on a failed wait must not strand the others): every warp adds its
// lanes' values in a fixed shuffle order and its lane 0 stores them in slot b = j & 3
// and arrives on red_bar[b] (count = epilogue warps); a collecting thread waits for
// the slot (bounded), adds the warps in order and writes the partials: in the fused kernel
// a TMEM warp before it frees the accumulator that item j + 1 needs; in the syntheses one
// warp in turn during its item j + 1 (collect2), which reads slot b before it reads the
// accumulator of item j + 2, and no warp reaches item j + 4, which writes slot b again,
// before every warp has read the accumulator of item j + 2 (the accumulators are
// double-buffered). Either way a slot is read before it is written again.
constexpr int EPI_SLOTS = 4;
template <int NV>
struct EpiSums {
  double v[EPI_SLOTS][16][NV];
};
template <int NP, int NV>
__device__ __forceinline__ void epi_put(EpiSums<NV>& sh, uint32_t red_bar, int b,
                                        const double (&v)[NP]) {
  double t[NV] = {};   // values past NP are zero
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    t[k] = v[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t[k] += __shfl_xor_sync(0xffffffffu, t[k], o);
  }
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int k = 0; k < NV; ++k) sh.v[b][threadIdx.x >> 5][k] = t[k];
    mbar_arrive(red_bar);
  }
}
// The slot's sums over nw warps, added in warp order (false when the wait gave up); a whole
// warp calls it, and every lane gets them.
template <int NV>
__device__ __forceinline__ bool epi_take(const EpiSums<NV>& sh, uint32_t red_bar, int b,
                                         uint32_t parity, int nw, volatile int* fail, int* err,
                                         int code, double (&out)[NV]) {
  if (!pwait_warp(red_bar, parity, fail, err, code)) return false;
#pragma unroll
  for (int k = 0; k < NV; ++k) {
    out[k] = 0.0;
    for (int w = 0; w < nw; ++w) out[k] += sh.v[b][w][k];
  }
  return true;
}

// s2_mma_swapped of two 128-row tiles for the kp that the pipelines take.
__device__ __forceinline__ void s2_mma_swapped_kp(uint32_t acc, uint32_t sa, uint32_t sb, int kp,
                                                  uint32_t idesc, uint32_t lead) {
  switch (kp) {
    case 16: return s2_mma_swapped<16>(acc, sa, 128, sb, 128, idesc, lead);
    case 32: return s2_mma_swapped<32>(acc, sa, 128, sb, 128, idesc, lead);
    case 48: return s2_mma_swapped<48>(acc, sa, 128, sb, 128, idesc, lead);
    case 64: return s2_mma_swapped<64>(acc, sa, 128, sb, 128, idesc, lead);
    case 80: return s2_mma_swapped<80>(acc, sa, 128, sb, 128, idesc, lead);
    case 96: return s2_mma_swapped<96>(acc, sa, 128, sb, 128, idesc, lead);
    case 112: return s2_mma_swapped<112>(acc, sa, 128, sb, 128, idesc, lead);
    default: return s2_mma_swapped<128>(acc, sa, 128, sb, 128, idesc, lead);
  }
}

// i modulo n for any i (the periodic layout).
__device__ __forceinline__ int wrapped(int i, int n) {
  i %= n;
  return i < 0 ? i + n : i;
}

// L2 prefetch of the row segment of this lane for a later item: the line holding row
// yb + lane, column x0 of image img (N x N floats), when columns x0 .. x0 + 31 lie
// inside the image and pf (N % 4 == 0, 16-byte aligned image base) holds.
__device__ __forceinline__ void prefetch_rows(const float* img, int N, int yb, int x0, bool pf) {
  const int y = yb + (int)(threadIdx.x & 31);
  if (pf && y < N && x0 + 32 <= N) tc::prefetch_l2_line(img + (size_t)y * N + x0);
}

// The sums of item j (slot j & 3) over nw warps into out[0 .. nv - 1], by the whole warp that
// collects item j (false when the wait gave up). Item j is collected by warp
// j % nw one item later, when every warp has normally stored its part, so that no warp
// waits for the others in the common case.
__device__ __forceinline__ bool collect2(const EpiSums<2>& sh, uint64_t* red_bar, int j, int nw,
                                         volatile int* fail, int* err, int code, double* out,
                                         int nv) {
  double t[2];
  if (!epi_take<2>(sh, tc::smem_u32(&red_bar[j & 3]), j & 3, (j >> 2) & 1, nw, fail, err, code,
                   t))
    return false;
  if ((threadIdx.x & 31) == 0) {
    out[0] = t[0];
    if (nv > 1) out[1] = t[1];
  }
  return true;
}

// R (tensor memory: lanes y = lane_base + lane, columns f) -> sR, the K-major
// [hi | lo] operand of stage 2 (rb rows f, K = y), for the 8-column groups u0, u0 + du,
// .. below nu (rows f from 8 nu on are left as they are: the columns of the product that
// they belong to are not used). The words (f, y & ~1) hold the pair of lanes y & ~1 and
// y | 1: for each pair of columns (f, f + 1) the even lane splits and stores column f (hi
// and lo word), the odd lane column f + 1, after one exchange of values between the two.
// acc: the accumulator's address with this warp's lane base.
__device__ __forceinline__ void r_to_operand(uint32_t acc, uint8_t* sR, int rb, int lane_base,
                                             int u0, int du, int nu) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t ye = ((uint32_t)lane_base + lane) & ~1u;
  const uint32_t odd = lane & 1u;
  // sw128_offset(rb, f, k) for f = 8 u + i + odd, k = ye (hi) or 128 + ye (lo): the
  // part that depends on f % 8, and the 1024-byte group u
  uint32_t off[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t f8 = 2u * i + odd;
    off[i] = (ye >> 6) * (uint32_t)rb * 128u + f8 * 128u + ((((ye & 63u) >> 3) ^ f8) << 4) +
             (ye & 7u) * 2u;
  }
  const uint32_t LO = 2u * (uint32_t)rb * 128u;   // k + 128: two atoms further
#pragma unroll 1
  for (int u = u0; u < nu; u += du) {
    float rv[8];
    tmem_ld8x(acc + (uint32_t)(8 * u), rv);
    uint8_t* sq = sR + (uint32_t)u * 1024u;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      // the even lane receives its partner's column i, the odd lane column i + 1
      const float got = __shfl_xor_sync(0xffffffffu, odd ? rv[i] : rv[i + 1], 1);
      uint32_t h2, l2;
      split_pair(odd ? got : rv[i], odd ? rv[i + 1] : got, h2, l2);
      uint8_t* w = sq + off[i >> 1];
      *reinterpret_cast<uint32_t*>(w) = h2;
      *reinterpret_cast<uint32_t*>(w + LO) = l2;
    }
  }
}

// Q (tensor memory: lanes n = 2 r + s, columns f = 2 c + t) -> the tile's partials
// P[r][c] of the band (see analysis_stages in tc2.cu): Re = Q[2r][2c] - Q[2r+1][2c+1],
// Im = Q[2r][2c+1] + Q[2r+1][2c]; with sym also the conjugate rows -r (from the odd
// lane of the pair), for the 8-column groups u0, u0 + du, .. below nu. The tile's block
// is stored column-major, P[c][row] at out + c nrows_out + row, so that a warp's store of
// one column touches two runs of consecutive rows instead of 32 rows ncols apart
// (reduce_tiles_kernel with trows = nrows_out reads this layout).
__device__ __forceinline__ void q_to_partials(uint32_t acc, float2* out, const Tc2Analysis& a,
                                              int lane_base, int u0, int du, int nu) {
  const int lane = threadIdx.x & 31;
  const int nn = lane_base + lane;
  const int r = nn >> 1, s = nn & 1;
  if (lane_base >= 2 * a.nr) return;   // none of this warp's lanes holds a row
  // the output row of this lane, or none
  float2* row = nullptr;
  if (r < a.nr) {
    if (!a.sym)
      row = s == 0 ? out + r : nullptr;
    else if (s == 0)
      row = out + (a.nr - 1 + r);
    else if (r >= 1)
      row = out + (a.nr - 1 - r);
  }
#pragma unroll 1
  for (int u = u0; u < nu; u += du) {
    float qv[8], pv[8];
    tmem_ld8x(acc + (uint32_t)(8 * u), qv);
#pragma unroll
    for (int i = 0; i < 8; ++i) pv[i] = __shfl_xor_sync(0xffffffffu, qv[i], 1);
    if (row == nullptr) continue;
    float2* rq = row + (size_t)(4 * u) * a.nrows_out;
    const int nc = a.ncols - 4 * u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (i >= nc) break;
      const float o0 = qv[2 * i], o1 = qv[2 * i + 1], p0 = pv[2 * i], p1 = pv[2 * i + 1];
      rq[(size_t)i * a.nrows_out] = s == 0 ? make_float2(o0 - p1, o1 + p0)
                                           : make_float2(p0 + o1, p1 - o0);
    }
  }
}

int sm_count() {
  static int count[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 148;
  if (!count[dev]) {
    int c = 0;
    if (cudaDeviceGetAttribute(&c, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || c <= 0)
      c = 148;
    count[dev] = c;
  }
  return count[dev];
}

}  // namespace

// =============================================================== tile analysis
// The partials of launch_analysis_tc2 (same products, same order, same layout
// part[image][yt][xt][row][c]) from a persistent pipeline:
//   warps 0-15  load the image tile (theta -> mask for mode 1), split it into the
//               [hi | lo] operand sA;
//   warp 24     (one elected lane) copies the TX tile (per xt) and the TY tile (per yt),
//               issues stage 1 R = sA . TX^T into accR[j & 1] and stage 2
//               Q = TY . R^T into accQ[j & 1];
//   warps 16-23 turn R into the stage-2 operand sR, and Q into the item's partials
//               (two warps per lane quarter, each taking every other 16-column group).
// Shared memory: TY 64 KiB | sA 64 KiB | TX | sR (BN x 128 split tiles, BN <= 96).
// Tensor memory: 512 columns, accR[b] at 128 b, accQ[b] at 256 + 128 b.
// A3_TMW TMEM warps: warps A3_LOADW + i and A3_LOADW + i + 4 share the lane quarter i
// of the accumulators and split its 16-column groups (even / odd).
constexpr int A3_LOADW = 16, A3_TMW = 8, A3_MMAW = A3_LOADW + A3_TMW;
constexpr int A3_NT = (A3_MMAW + 1) * 32;
// chunks of 8 pixels per loader thread, rows between a thread's chunks
constexpr int A3_CH = 2048 / (32 * A3_LOADW), A3_RS = 2 * A3_LOADW;

template <int BN, int MODE>
__global__ void __launch_bounds__(A3_NT, 1)
analysis_tc3_kernel(Tc2Analysis a, int T, int B, const uint8_t* __restrict__ txImg,
                    const uint8_t* __restrict__ tyImg, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 0 sA full (16 loader warps), 1-2 stage 1 done [b], 3 sR full (8 TMEM warps),
  // 4-5 stage 2 done [b], 6-7 accQ[b] free (8 TMEM warps), 8 TX landed, 9 TY landed
  __shared__ __align__(8) uint64_t bars[10];
  __shared__ uint32_t tmem_slot;
  __shared__ int fail;
  constexpr uint32_t TXB = s2_tile_bytes(BN, 128);
  uint8_t* smem = align1024(smem_raw);
  uint8_t* sA = smem + A2_A_BYTES;
  uint8_t* sR = smem + 2 * A2_A_BYTES + TXB;
  const uint32_t uTY = tc::smem_u32(smem), uA = tc::smem_u32(sA);
  const uint32_t uTX = uA + A2_A_BYTES, uR = tc::smem_u32(sR);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  auto bar = [&](int i) { return tc::smem_u32(&bars[i]); };
  int lo, hi;
  my_items(T * T * B, lo, hi);
  const int n = hi - lo;
  pdl_trigger();
  if (threadIdx.x == 0) {
    tc::mbar_init(bar(0), A3_LOADW);
    tc::mbar_init(bar(1), 1);
    tc::mbar_init(bar(2), 1);
    tc::mbar_init(bar(3), A3_TMW);
    tc::mbar_init(bar(4), 1);
    tc::mbar_init(bar(5), 1);
    tc::mbar_init(bar(6), A3_TMW);
    tc::mbar_init(bar(7), A3_TMW);
    tc::mbar_init(bar(8), 1);
    tc::mbar_init(bar(9), 1);
    fail = 0;
    tc::fence_mbar_init();
  }
  if (warp == A3_MMAW) tc::tmem_alloc(tc::smem_u32(&tmem_slot), 512);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* vfail = &fail;
  constexpr uint32_t idesc = tc::idesc_bf16(128, BN);

  if (warp < A3_LOADW) {
    // ------------------------------------------------------------ loaders
    pdl_wait();
    const int tid = threadIdx.x;
    // chunk i of a thread: row (tid >> 4) + A3_RS i, columns c8 .. c8 + 7 of the tile;
    // its hi part at so + 128 A3_RS i of sA, its lo part 32 KiB further (sw128_offset)
    const int r0 = tid >> 4, c8 = (tid & 15) * 8;
    const uint32_t so = sw128_offset(128, r0, c8);
    constexpr int HALF = A3_CH / 2;
    float v[A3_CH][8];
    // chunks i0 .. i0 + HALF - 1 of item it into v
    auto load_half = [&](const Item& it, int i0) {
      const int m0 = it.yt * 128 + r0, x = it.xt * 128 + c8;
      const float* img = a.in + (size_t)it.z * a.N * a.N + (size_t)m0 * a.N + x;
#pragma unroll
      for (int i = i0; i < i0 + HALF; ++i) {
        const int m = m0 + A3_RS * i;
        const float* pi = img + (size_t)(A3_RS * i) * a.N;
        if (a.vec4 && m < a.N && x + 7 < a.N) {
          const float4 p = __ldg(reinterpret_cast<const float4*>(pi));
          const float4 q = __ldg(reinterpret_cast<const float4*>(pi + 4));
          v[i][0] = p.x; v[i][1] = p.y; v[i][2] = p.z; v[i][3] = p.w;
          v[i][4] = q.x; v[i][5] = q.y; v[i][6] = q.z; v[i][7] = q.w;
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) v[i][e] = (m < a.N && x + e < a.N) ? __ldg(pi + e) : 0.f;
        }
      }
    };
    // chunks i0 .. i0 + HALF - 1 of item j: theta -> mask (mode 1), split into the hi /
    // lo words hw / lw of sA (stored by store_half); the non-finite inputs flagged in bad
    uint4 hw[HALF], lw[HALF];
    auto conv_half = [&](const Item& it, int i0, bool& bad) {
      const int m0 = it.yt * 128 + r0, x = it.xt * 128 + c8;
      float* mo = a.mask_out ? a.mask_out + (size_t)it.z * a.N * a.N + (size_t)m0 * a.N + x
                             : nullptr;
      const bool full = a.vec4 && it.yt * 128 + 127 < a.N && x + 7 < a.N;
#pragma unroll
      for (int i = i0; i < i0 + HALF; ++i) {
        const int m = m0 + A3_RS * i;
        float u[8];
        if (full) {
          // every input is finite exactly when chk stays 0
          float chk = 0.f;
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            chk = __fmaf_rn(v[i][e], 0.f, chk);
            u[e] = MODE == 1 ? 0.5f * (1.f + fast_cos(v[i][e])) : v[i][e];
          }
          bad |= chk != 0.f;
          if (mo) {
            float* po = mo + (size_t)(A3_RS * i) * a.N;
            *reinterpret_cast<float4*>(po) = make_float4(u[0], u[1], u[2], u[3]);
            *reinterpret_cast<float4*>(po + 4) = make_float4(u[4], u[5], u[6], u[7]);
          }
        } else {
#pragma unroll
          for (int e = 0; e < 8; ++e) {
            const bool in_range = m < a.N && x + e < a.N;
            u[e] = v[i][e];
            if (in_range) bad |= !isfinite(u[e]);
            if (MODE == 1) {
              u[e] = in_range ? 0.5f * (1.f + fast_cos(u[e])) : 0.f;
              if (mo && in_range) mo[(size_t)(A3_RS * i) * a.N + e] = u[e];
            }
          }
        }
        split_pair(u[0], u[1], hw[i - i0].x, lw[i - i0].x);
        split_pair(u[2], u[3], hw[i - i0].y, lw[i - i0].y);
        split_pair(u[4], u[5], hw[i - i0].z, lw[i - i0].z);
        split_pair(u[6], u[7], hw[i - i0].w, lw[i - i0].w);
      }
    };
    auto store_half = [&](int i0) {
#pragma unroll
      for (int i = i0; i < i0 + HALF; ++i) {
        *reinterpret_cast<uint4*>(sA + so + (uint32_t)(128 * A3_RS) * i) = hw[i - i0];
        *reinterpret_cast<uint4*>(sA + so + 32768u + (uint32_t)(128 * A3_RS) * i) = lw[i - i0];
      }
    };
    // The loads run half an item ahead of the conversion: the second half of item j
    // loads while the first half converts, the first half of item j + 1 while the
    // second half of item j converts. The first half is converted before the wait for
    // sA to become free, so that only its stores follow stage 1 of the previous item.
    // the input tile of item i + 2 is fetched into L2 during item i: 512 segments of 128
    // bytes, one per loader thread (row tid / 4, columns 32 (tid % 4) ..)
    const bool pf = a.N % 4 == 0 && reinterpret_cast<uintptr_t>(a.in) % 16 == 0;
    auto prefetch_item = [&](const Item& i) {
      const int y = i.yt * 128 + (tid >> 2), x = i.xt * 128 + 32 * (tid & 3);
      static_assert(A3_LOADW * 32 == 512, "one 128-byte segment per loader thread");
      if (pf && y < a.N && x + 32 <= a.N)
        tc::prefetch_l2_line(a.in + (size_t)i.z * a.N * a.N + (size_t)y * a.N + x);
    };
    Item cur = item_at(lo, T, B);
    if (n > 0) load_half(cur, 0);
    if (n > 1) prefetch_item(item_next(cur, T, B));
    for (int j = 0; j < n; ++j, cur = item_next(cur, T, B)) {
      if (j + 2 < n) prefetch_item(item_next(item_next(cur, T, B), T, B));
      load_half(cur, HALF);
      bool bad = false;
      conv_half(cur, 0, bad);
      // sA is free once stage 1 of the previous item has completed
      if (j > 0 && !pwait_warp(bar(1 + ((j - 1) & 1)), ((j - 1) >> 1) & 1, vfail, err, 11)) break;
      store_half(0);
      if (j + 1 < n) load_half(item_next(cur, T, B), 0);
      conv_half(cur, HALF, bad);
      store_half(HALF);
      if (bad) atomicOr(a.flag, 1);
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(0));
    }
  } else if (warp < A3_MMAW) {
    // ------------------------------------------------------------ TMEM warps
    pdl_wait();
    const int lane_base = (warp & 3) * 32;
    constexpr int DQ = A3_TMW / 4;
    const int u0 = (warp - A3_LOADW) / 4;   // first 8-column group of this warp
    const int nu = (2 * a.ncols + 7) / 8;
    const int count = a.nrows_out * a.ncols;
    Item prv = item_at(lo, T, B), cur = prv;   // items j - 1 and j
    for (int j = 0; j <= n; ++j) {
      if (j > 0) {
        prv = cur;
        cur = item_next(cur, T, B);
      }
      if (j < n && !pwait_warp(bar(1 + (j & 1)), (j >> 1) & 1, vfail, err, 12)) break;
      // stage 2 of the previous item done: sR is free and its Q is ready
      if (j > 0 && !pwait_warp(bar(4 + ((j - 1) & 1)), ((j - 1) >> 1) & 1, vfail, err, 13)) break;
      tc::fence_after();
      if (j < n) {
        r_to_operand(tmem + (uint32_t)((j & 1) * 128) + ((uint32_t)lane_base << 16), sR, BN,
                     lane_base, u0, DQ, nu);
        fence_async_smem();
        tc::fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(3));
      }
      if (j > 0) {
        // Q of the previous item -> its partials P[r][c] (see analysis_stages in tc2.cu)
        const int jp = j - 1;
        float2* out = a.part + (((size_t)prv.z * T + prv.yt) * T + prv.xt) * count;
        q_to_partials(tmem + 256u + (uint32_t)((jp & 1) * 128) + ((uint32_t)lane_base << 16), out,
                      a, lane_base, u0, DQ, nu);
        tc::fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(6 + (jp & 1)));
      }
    }
  } else {
    // ------------------------------------------------------------ MMA warp
    const uint32_t lead = tc::elect_one();
    int pxt = -1, pyt = -1;
    uint32_t ntx = 0, nty = 0;
    int m1 = 0, m2 = 0;
    // Issue order MMA1(0), MMA1(1), MMA2(0), MMA1(2), MMA2(1), ...: stage 1 of item j
    // is issued as soon as its operand sA is full, before stage 2 of item j - 1 waits
    // for its operand sR, so the tensor pipe runs stage 1 of the next item while the
    // TMEM warps build sR.
    Item it = item_at(lo, T, B), prv = it;
    for (int j = 0; j <= n; ++j) {
      if (j < n) {
        const bool newx = it.xt != pxt;
        if (newx) {
          // the TX tile in use is read by stage 1 of the previous item
          if (j > 0 && !pwait_warp(bar(1 + ((j - 1) & 1)), ((j - 1) >> 1) & 1, vfail, err, 14)) break;
          bulk_tile(uTX, txImg + (size_t)it.xt * TXB, TXB, bar(8), lead);
          ++ntx;
          pxt = it.xt;
        }
        if (!pwait_warp(bar(0), j & 1, vfail, err, 15)) break;
        if (newx && !pwait_warp(bar(8), (ntx - 1) & 1, vfail, err, 16)) break;
        tc::fence_after();
        s2_mma(tmem + (uint32_t)((j & 1) * 128), uA, 128, uTX, BN, 128, idesc, lead);
        tc::mma_commit(bar(1 + (j & 1)), lead);
        ++m1;
      }
      if (j > 0) {
        // stage 2 of item jj = j - 1
        const int jj = j - 1;
        const bool newy = prv.yt != pyt;
        if (newy) {
          if (jj > 0 && !pwait_warp(bar(4 + ((jj - 1) & 1)), ((jj - 1) >> 1) & 1, vfail, err, 17)) break;
          bulk_tile(uTY, tyImg + (size_t)prv.yt * A2_A_BYTES, A2_A_BYTES, bar(9), lead);
          ++nty;
          pyt = prv.yt;
        }
        if (!pwait_warp(bar(3), jj & 1, vfail, err, 18)) break;
        if (newy && !pwait_warp(bar(9), (nty - 1) & 1, vfail, err, 19)) break;
        if (jj >= 2 && !pwait_warp(bar(6 + (jj & 1)), ((jj - 2) >> 1) & 1, vfail, err, 20)) break;
        tc::fence_after();
        s2_mma(tmem + 256u + (uint32_t)((jj & 1) * 128), uTY, 128, uR, BN, 128, idesc, lead);
        tc::mma_commit(bar(4 + (jj & 1)), lead);
        ++m2;
        prv = item_next(prv, T, B);
      }
      if (j < n) it = item_next(it, T, B);
    }
    if (*vfail) {
      // nothing of this CTA may still be in flight when it exits
      if (ntx) tc::mbar_wait(bar(8), (ntx - 1) & 1);
      if (nty) tc::mbar_wait(bar(9), (nty - 1) & 1);
      if (m1) tc::mbar_wait(bar(1 + ((m1 - 1) & 1)), ((m1 - 1) >> 1) & 1);
      if (m2) tc::mbar_wait(bar(4 + ((m2 - 1) & 1)), ((m2 - 1) >> 1) & 1);
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == A3_MMAW) tc::tmem_dealloc(tmem, 512);
}

template <int BN, int MODE>
static cudaError_t analysis_tc3_m(cudaStream_t s, const Tc2Analysis& a, const void* tx,
                                  const void* ty, int* err, int batch) {
  const size_t smem = 2 * (size_t)A2_A_BYTES + 2 * (size_t)s2_tile_bytes(BN, 128) + 1024;
  cudaError_t e = cudaFuncSetAttribute(analysis_tc3_kernel<BN, MODE>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int T = (a.N + 127) / 128;
  const int items = T * T * batch;
  const int grid = items < sm_count() ? items : sm_count();
  return launch_pdl(analysis_tc3_kernel<BN, MODE>, dim3(grid), dim3(A3_NT), smem, s, a, T, batch,
                    static_cast<const uint8_t*>(tx), static_cast<const uint8_t*>(ty), err);
}
template <int BN>
static cudaError_t analysis_tc3_t(cudaStream_t s, const Tc2Analysis& a, const void* tx,
                                  const void* ty, int* err, int batch) {
  return a.mode == 1 ? analysis_tc3_m<BN, 1>(s, a, tx, ty, err, batch)
                     : analysis_tc3_m<BN, 0>(s, a, tx, ty, err, batch);
}

bool tc3_analysis_supported(int ncols, int nr) {
  return tc2_analysis_supported(ncols, nr) && tc2_analysis_rows(ncols) <= 96;
}

cudaError_t launch_analysis_tc3(cudaStream_t s, int mode, const float* in, float* mask_out,
                                int* flag, int N, int ncols, int nrows_out, int nr, int sym,
                                float2* part, const void* tx_img, const void* ty_img, int* err,
                                int batch) {
  // vector loads of the input and vector stores of the mask
  const int vec4 = (N % 4 == 0) && (reinterpret_cast<uintptr_t>(in) % 16 == 0) &&
                   (reinterpret_cast<uintptr_t>(mask_out) % 16 == 0);
  Tc2Analysis a{in, mask_out, flag, N, mode, vec4, ncols, nrows_out, nr, sym, part};
  switch (tc2_analysis_rows(ncols)) {
    case 16: return analysis_tc3_t<16>(s, a, tx_img, ty_img, err, batch);
    case 32: return analysis_tc3_t<32>(s, a, tx_img, ty_img, err, batch);
    case 48: return analysis_tc3_t<48>(s, a, tx_img, ty_img, err, batch);
    case 64: return analysis_tc3_t<64>(s, a, tx_img, ty_img, err, batch);
    case 80: return analysis_tc3_t<80>(s, a, tx_img, ty_img, err, batch);
    case 96: return analysis_tc3_t<96>(s, a, tx_img, ty_img, err, batch);
    default: return cudaErrorInvalidValue;
  }
}


// =============================================================== epilogue arithmetic
// Per pixel exactly the FAST arithmetic of ResistEpiT<true> / GradEpiT<true>
// (device_common.cuh); loss and norm terms are summed in FP32 over a thread's 32
// pixels of an item and in FP64 from there on.
struct S3Resist {
  ResistEpilogue p;
  __device__ __forceinline__ float sigmoid(float I) const {
    const float z = -p.alpha * (I - p.thr);
    return __fdividef(1.f, 1.f + __expf(z));
  }
  // Mode 1 at in-range pixel i (image offset included): the stores of aerial / wafer,
  // the loss terms into pe / pen, and dL/dI returned.
  __device__ __forceinline__ float dldi(size_t i, float I, float T, bool plain, float& pe,
                                        float& pen) const {
    if (p.aerial) p.aerial[i] = I;
    const float W = sigmoid(I);
    if (p.wafer) p.wafer[i] = W;
    const float r = W - T;
    if (plain) {
      pe += r * r;
      return p.pe_weight * r * W * (1.f - W);
    }
    const float pw = p.pe_window ? __ldg(p.pe_window + i) : 1.f;
    const float qw = p.pen_window ? __ldg(p.pen_window + i) : pw;
    pe += r * r * pw;
    float s = p.pe_weight * r * pw;
    if ((p.penalty != 0.f || p.loss_penalty_term) && T < 0.5f) {
      const float ex = fmaxf(W - p.pen_thr, 0.f);
      pen += ex * ex * qw;
      s += p.penalty * ex * qw;
    }
    return s * W * (1.f - W);
  }
  __host__ __device__ __forceinline__ bool plain() const {
    return p.pe_window == nullptr && p.pen_window == nullptr && p.penalty == 0.f &&
           !p.loss_penalty_term;
  }
};

// =============================================================== row synthesis
// out[y][x] = sum_f AY[y][f] Bt[x][f] with the theta-chain (KIND 0, GradEpilogue), the
// resist (KIND 1, ResistEpilogue) or the plain (KIND 2, GradEpilogue without theta: dPE/dM
// stored once or twice) epilogue, as launch_synth_grad_tc2 /
// launch_synth_resist_tc2, from a persistent pipeline:
//   warp 16      (one elected lane) copies the AY tile (per yt), double-buffers the band
//                operand tile Bt (per image and xt) and issues D[x][y] into acc[j & 1];
//   warps 0-15   run the epilogue of item j while the MMA of item j + 1 runs: warp w
//                takes lanes x = 32 (w % 4) + lane and rows y = 32 (w / 4) .. + 31.
// The FP64 partial of an item (squared gradient norm, or the two loss terms) is
// written to [image][yt][xt] as the per-tile kernels write theirs. Shared memory:
// AY | Bt[0] | Bt[1] (split tiles of 128 x kp). Tensor memory: acc[b] at 128 b.
constexpr int S3_EPIW = 16, S3_MMAW = 16;
constexpr int S3_NT = (S3_EPIW + 1) * 32;

template <int KIND>
__global__ void __launch_bounds__(S3_NT, 1)
synth_tc3_kernel(const uint8_t* __restrict__ Aimg, const uint8_t* __restrict__ Bimg, int N,
                 int kp, int T, int B, GradEpilogue g, S3Resist r, int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // 0-1 Bt[b] landed, 2 AY landed, 3-4 acc[b] full, 5-6 acc[b] free (epilogue warps)
  __shared__ __align__(8) uint64_t bars[7];
  __shared__ uint32_t tmem_slot;
  __shared__ int fail;
  __shared__ __align__(8) uint64_t red_bar[EPI_SLOTS];
  __shared__ EpiSums<2> red;
  const uint32_t tb = s2_tile_bytes(128, kp);
  uint8_t* smem = align1024(smem_raw);
  const uint32_t uAY = tc::smem_u32(smem);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  auto bar = [&](int i) { return tc::smem_u32(&bars[i]); };
  int lo, hi;
  my_items(T * T * B, lo, hi);
  const int n = hi - lo;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int i = 0; i < 5; ++i) tc::mbar_init(bar(i), 1);
    tc::mbar_init(bar(5), S3_EPIW);
    tc::mbar_init(bar(6), S3_EPIW);
    for (int i = 0; i < EPI_SLOTS; ++i) tc::mbar_init(tc::smem_u32(&red_bar[i]), S3_EPIW);
    fail = 0;
    tc::fence_mbar_init();
  }
  if (warp == S3_MMAW) tc::tmem_alloc(tc::smem_u32(&tmem_slot), 256);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot;
  volatile int* vfail = &fail;

  if (warp < S3_EPIW) {
    // ------------------------------------------------------------ epilogue warps
    pdl_wait();
    const int q = warp & 3, h = warp >> 2;
    const uint32_t lane_addr = (uint32_t)(32 * q) << 16;
    const float* src = KIND == 0 ? g.theta : KIND == 1 && r.p.mode == 1 ? r.p.target : nullptr;
    const bool plain = KIND == 1 && r.plain();
    // theta chain without the dPE/dM output: the CTM evaluation
    const bool lean = KIND == 0 && g.grad_mask == nullptr;
    // per-pixel input, coalesced along x: rows e0 .. e0 + 15 of item j into pre[]
    float pre[32];
    auto load_rows = [&](const Item& it, int e0) {
      const int x = it.xt * 128 + 32 * q + lane, yb = it.yt * 128 + 32 * h;
      const float* sp = src + (size_t)it.z * N * N + (size_t)yb * N + x;
      if (x < N && yb + 31 < N) {
#pragma unroll
        for (int e = e0; e < e0 + 16; ++e) pre[e] = __ldg(sp + e * N);
      } else {
#pragma unroll
        for (int e = e0; e < e0 + 16; ++e) pre[e] = (x < N && yb + e < N) ? __ldg(sp + e * N) : 0.f;
      }
    };
    Item it = item_at(lo, T, B);
    // the input rows of item i + 2 are fetched into L2 during item i
    const bool pf = src && N % 4 == 0 && reinterpret_cast<uintptr_t>(src) % 16 == 0;
    auto prefetch_item = [&](const Item& i) {
      prefetch_rows(src + (size_t)i.z * N * N, N, i.yt * 128 + 32 * h, i.xt * 128 + 32 * q, pf);
    };
    if (src && n > 0) {
      load_rows(it, 0);
      load_rows(it, 16);
    }
    if (n > 1) prefetch_item(item_next(it, T, B));
    const bool sums = KIND == 0 || (KIND == 1 && r.p.mode == 1);
    // the partial sums of item i: the squared norm (KIND 0) or the two loss terms
    auto sums_out = [&](const Item& i) {
      const size_t bid = ((size_t)i.z * T + i.yt) * T + i.xt;
      return KIND == 0 ? g.norm_partial + bid : r.p.loss_partial + 2 * bid;
    };
    Item ip = it;   // item j - 1
    int done = 0;   // items finished
    for (int j = 0; j < n; ++j, ip = it, it = item_next(it, T, B)) {
      const Item nxt = item_next(it, T, B);
      if (j + 2 < n) prefetch_item(item_next(nxt, T, B));
      const int x = it.xt * 128 + 32 * q + lane;
      const int yb = it.yt * 128 + 32 * h;
      const bool xin = x < N;
      const bool full = xin && yb + 31 < N;
      const size_t base = (size_t)it.z * N * N;
      if (!pwait_warp(bar(3 + (j & 1)), (j >> 1) & 1, vfail, err, 21)) break;
      tc::fence_after();
      float d[32];
      tc::tmem_ld32(tmem + (uint32_t)((j & 1) * 128) + lane_addr + (uint32_t)(32 * h), d);
      tc::fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(5 + (j & 1)));
      float s0 = 0.f, s1 = 0.f;
      // rows e0 .. e0 + 15; the inputs of the next item load into the rows just used
      auto rows = [&](int e0) {
        if (KIND == 2) {
          // dPE/dM alone (the second copy is the full chip's raw gradient)
          float* gp = g.grad_mask + base + (size_t)yb * N + x;
          float* cp = g.grad_copy ? g.grad_copy + base + (size_t)yb * N + x : nullptr;
          const int ny = xin ? N - yb : 0;
          if (full) {
#pragma unroll
            for (int e = e0; e < e0 + 16; ++e) gp[e * N] = d[e];
            if (cp) {
#pragma unroll
              for (int e = e0; e < e0 + 16; ++e) cp[e * N] = d[e];
            }
          } else {
#pragma unroll
            for (int e = e0; e < e0 + 16; ++e) {
              if (e < ny) {
                gp[e * N] = d[e];
                if (cp) cp[e * N] = d[e];
              }
            }
          }
        } else if (lean && full) {
          float* gp = g.grad_theta + base + (size_t)yb * N + x;
#pragma unroll
          for (int e = e0; e < e0 + 16; ++e) {
            const float gt = -0.5f * d[e] * fast_sin(pre[e]);
            s0 += gt * gt;
            gp[e * N] = gt;
          }
        } else {
#pragma unroll
          for (int e = e0; e < e0 + 16; ++e) {
            const int y = yb + e;
            const bool in = xin && y < N;
            const size_t i = base + (size_t)y * N + x;
            if (KIND == 0) {
              const float G = d[e];
              if (in && g.grad_mask) g.grad_mask[i] = G;
              if (in) {
                // pixels past the image edge are left out: the band operand's rows there
                // are not part of the image and may hold anything
                const float gt = -0.5f * G * fast_sin(pre[e]);
                s0 += gt * gt;
                g.grad_theta[i] = gt;
              }
            } else if (in) {
              const float I = d[e];
              if (r.p.mode == 0) {
                if (r.p.aerial) r.p.aerial[i] = I;
                if (r.p.wafer) r.p.wafer[i] = r.sigmoid(I);
              } else {
                r.p.dldi[i] = r.dldi(i, I, pre[e], plain, s0, s1);
              }
            }
          }
        }
        if (src && j + 1 < n) load_rows(nxt, e0);
      };
      rows(0);
      rows(16);
      if (sums) {
        const double v[2] = {(double)s0, (double)s1};
        if (KIND == 0) epi_put<1>(red, tc::smem_u32(&red_bar[j & 3]), j & 3, {v[0]});
        else epi_put<2>(red, tc::smem_u32(&red_bar[j & 3]), j & 3, v);
        // the sums of item j - 1, by one warp in turn
        if (j > 0 && warp == (j - 1) % S3_EPIW &&
            !collect2(red, red_bar, j - 1, S3_EPIW, vfail, err, 27, sums_out(ip), KIND == 0 ? 1 : 2))
          break;
      }
      done = j + 1;
    }
    // the sums of the last item
    if (sums && n > 0 && done == n && warp == (n - 1) % S3_EPIW)
      collect2(red, red_bar, n - 1, S3_EPIW, vfail, err, 28, sums_out(ip), KIND == 0 ? 1 : 2);
  } else if (warp == S3_MMAW) {
    // ------------------------------------------------------------ MMA warp
    const uint32_t lead = tc::elect_one();
    // the band operand image is written by the previous kernel of the stream
    pdl_wait();
    constexpr uint32_t idesc = tc::idesc_bf16(128, 128);
    auto bt_src = [&](const Item& it) { return Bimg + ((size_t)it.z * T + it.xt) * tb; };
    int pyt = -1;
    uint32_t nay = 0;
    int nb = 0, nm = 0;
    Item it = item_at(lo, T, B);
    if (n > 0) {
      bulk_tile(uAY + tb, bt_src(it), tb, bar(0), lead);
      nb = 1;
    }
    for (int j = 0; j < n; ++j, it = item_next(it, T, B)) {
      const bool newy = it.yt != pyt;
      if (newy) {
        // the AY tile in use is read by the previous item's MMA
        if (j > 0 && !pwait_warp(bar(3 + ((j - 1) & 1)), ((j - 1) >> 1) & 1, vfail, err, 22)) break;
        bulk_tile(uAY, Aimg + (size_t)it.yt * tb, tb, bar(2), lead);
        ++nay;
        pyt = it.yt;
      }
      if (!pwait_warp(bar(j & 1), (j >> 1) & 1, vfail, err, 23)) break;
      if (newy && !pwait_warp(bar(2), (nay - 1) & 1, vfail, err, 24)) break;
      if (j >= 2 && !pwait_warp(bar(5 + (j & 1)), ((j - 2) >> 1) & 1, vfail, err, 25)) break;
      tc::fence_after();
      s2_mma_swapped_kp(tmem + (uint32_t)((j & 1) * 128), uAY, uAY + (uint32_t)(1 + (j & 1)) * tb, kp,
                        idesc, lead);
      tc::mma_commit(bar(3 + (j & 1)), lead);
      ++nm;
      if (j + 1 < n) {
        // Bt[(j + 1) & 1] is read by the MMA of item j - 1
        if (j >= 1 && !pwait_warp(bar(3 + ((j - 1) & 1)), ((j - 1) >> 1) & 1, vfail, err, 26)) break;
        bulk_tile(uAY + (uint32_t)(1 + ((j + 1) & 1)) * tb, bt_src(item_next(it, T, B)), tb,
                  bar((j + 1) & 1), lead);
        ++nb;
      }
    }
    if (*vfail) {
      if (nb) tc::mbar_wait(bar((nb - 1) & 1), ((nb - 1) >> 1) & 1);
      if (nay) tc::mbar_wait(bar(2), (nay - 1) & 1);
      if (nm) tc::mbar_wait(bar(3 + ((nm - 1) & 1)), ((nm - 1) >> 1) & 1);
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == S3_MMAW) tc::tmem_dealloc(tmem, 256);
}

template <int KIND>
static cudaError_t synth_tc3_t(cudaStream_t s, const void* Aimg, const void* Bimg, int N, int kp,
                               const GradEpilogue& g, const ResistEpilogue& r, int* err,
                               int* nblocks, int batch) {
  const size_t smem = 3 * (size_t)s2_tile_bytes(128, kp) + 1024;
  cudaError_t e = cudaFuncSetAttribute(synth_tc3_kernel<KIND>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int T = (N + 127) / 128;
  const int items = T * T * batch;
  const int grid = items < sm_count() ? items : sm_count();
  *nblocks = T * T;
  return launch_pdl(synth_tc3_kernel<KIND>, dim3(grid), dim3(S3_NT), smem, s,
                    static_cast<const uint8_t*>(Aimg), static_cast<const uint8_t*>(Bimg), N, kp,
                    T, batch, g, S3Resist{r}, err);
}

bool tc3_synth_supported(int kp) { return kp % 16 == 0 && kp <= 128; }

cudaError_t launch_synth_grad_tc3(cudaStream_t s, const void* Aimg, const void* Bimg, int N,
                                  int kp, const GradEpilogue& ep, int* err, int* nblocks,
                                  int batch) {
  if (!ep.theta)
    return synth_tc3_t<2>(s, Aimg, Bimg, N, kp, ep, ResistEpilogue{}, err, nblocks, batch);
  return synth_tc3_t<0>(s, Aimg, Bimg, N, kp, ep, ResistEpilogue{}, err, nblocks, batch);
}

cudaError_t launch_synth_resist_tc3(cudaStream_t s, const void* Aimg, const void* Bimg, int N,
                                    int kp, const ResistEpilogue& ep, int* err, int* nblocks,
                                    int batch) {
  return synth_tc3_t<1>(s, Aimg, Bimg, N, kp, GradEpilogue{}, ep, err, nblocks, batch);
}

// =============================================================== fused resist + adjoint analysis
// The CTM evaluation's resist synthesis and the adjoint tile analysis of its dL/dI
// (launch_synth_resist_analysis_tc2: same loss partials, same adjoint partials) from a
// persistent pipeline. Per item j:
//   SMMA(j)   I^T = Ut . AYD^T into accI[j & 1] (transposed: lanes x);
//   epi(j)    warps 0-15: resist, loss terms, dL/dI, written as the split operand sA
//             (M = y, K = x) over Ut. sA is MN-major (mn_chunk_offset): a thread holds
//             rows y of its column x and writes them as 16-byte chunks, with no exchange
//             between lanes;
//   MMA1(j)   R = sA . TXD^T into accR; once done, Ut of item j + 1 takes sA's place and
//             SMMA(j + 1) is issued;
//   R(j)      warps 16-23: R -> sR;  MMA2(j)  Q = TYD . R^T into accQ;
//   Q(j)      warps 16-23, after R(j + 1): Q -> the item's adjoint partials.
// One set of 16 warps that did epi, R and Q in turn left half of the issue slots idle, and
// the MMA thread spent 3400 cycles on the 15 instructions of a synthesis (see elect_one); now
// R and Q run beside the next item's epilogue. 16 tiles of 2048^2: 216 us before, 184 us now; 12 of
// 1266^2 127 and 102, 16 micro tiles of 1280^2 with windows 146 and 101.
// Shared memory: sA / Ut | TXD (per xt) | TYD (per yt) | sR | AYD (per yt). TXD and sR hold the
// rf = 2 ncols rows f rounded to 8, TYD the rn = 2 nr rows n: the products read on to BN and
// 128 rows, into the tiles that follow, and their columns and lanes past rf and rn are not
// used. Where this does not fit (2 ncols or 2 nr above 80), AYD and TXD share one place: AYD is
// copied with every Ut, TXD once SMMA is done.
// Tensor memory: accI[b] at 128 b, accR at 256, accQ at 384.
constexpr int F3_EPIW = 16, F3_TMW = 8, F3_MMAW = F3_EPIW + F3_TMW;
constexpr int F3_NT = (F3_MMAW + 1) * 32;

__host__ __device__ constexpr uint32_t f3_rows(int ncols) { return (uint32_t)(2 * ncols + 7) / 8 * 8; }
// Dynamic shared memory of rf rows f, rn rows n and synthesis tiles of tb bytes: 1 KiB to align
// and, behind the last tile, 1 KiB for rows read past rf.
__host__ __device__ constexpr uint32_t f3_smem(uint32_t rf, uint32_t rn, uint32_t tb, bool res) {
  const uint32_t f = rf * 512u, x = A2_A_BYTES > tb ? A2_A_BYTES : tb;
  return x + (res ? f + tb : (f > tb ? f : tb)) + rn * 512u + f + 2048;
}
constexpr uint32_t F3_SMEM_MAX = 232448 - 2048;   // beside the static barriers and sums

// MODE 0: no window, no penalty, no image output (the CTM evaluation); 1: windows and
// penalty; 2: aerial / wafer outputs too. 16 micro tiles of 1280^2 with windows: 435 us when
// one epilogue served all modes and loaded each pixel's windows in turn, 101 us now (383 us with
// windows as images and both outputs); 12 tiles of 1266^2 (19 % of the tiles ragged) 102 us, 137
// when their edge left the packed arithmetic.
template <int BN, int MODE>
__global__ void __launch_bounds__(F3_NT, 1)
fused_tc3_kernel(const uint8_t* __restrict__ Aimg, const uint8_t* __restrict__ Bimg, int N,
                 int kp, int T, int B, S3Resist r, Tc2Analysis a, int res,
                 const uint8_t* __restrict__ txImg, const uint8_t* __restrict__ tyImg,
                 int* __restrict__ err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  // Ut, AYD, TXD, TYD landed; SMMA done [j & 1]; sA full (epilogue warps); MMA1 done; accR free
  // (TMEM warps); sR full (TMEM warps); MMA2 done; accQ free (TMEM warps). A phase of one item
  // completes only after every waiter has seen that of the item before.
  enum { UT, AY, TX, TY, SM, SM1, AFULL, M1, RFREE, SFULL, M2, QFREE, NBARS };
  __shared__ __align__(8) uint64_t bars[NBARS];
  __shared__ uint32_t tmem_slot;
  __shared__ int fail;
  __shared__ __align__(8) uint64_t red_bar[EPI_SLOTS];
  __shared__ EpiSums<2> red;
  const uint32_t rf = f3_rows(a.ncols), rn = f3_rows(a.nr);
  const uint32_t tb = s2_tile_bytes(128, kp);
  uint8_t* sA = align1024(smem_raw);
  const uint32_t uA = tc::smem_u32(sA), uUt = uA;
  const uint32_t uTXD = uA + (A2_A_BYTES > tb ? A2_A_BYTES : tb);
  const uint32_t uTYD = uTXD + (res || rf * 512u > tb ? rf * 512u : tb), uR = uTYD + rn * 512u;
  const uint32_t uAYD = res ? uR + rf * 512u : uTXD;
  uint8_t* sR = sA + (uR - uA);
  const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  auto bar = [&](int i) { return tc::smem_u32(&bars[i]); };
  int lo, hi;
  my_items(T * T * B, lo, hi);
  const int n = hi - lo;
  pdl_trigger();
  if (threadIdx.x == 0) {
    for (int i = 0; i < NBARS; ++i)
      tc::mbar_init(bar(i), i == AFULL ? F3_EPIW
                            : i == RFREE || i == SFULL || i == QFREE ? F3_TMW
                                                                     : 1);
    for (int i = 0; i < EPI_SLOTS; ++i) tc::mbar_init(tc::smem_u32(&red_bar[i]), F3_EPIW);
    fail = 0;
    tc::fence_mbar_init();
  }
  if (warp == F3_MMAW) tc::tmem_alloc(tc::smem_u32(&tmem_slot), 512);
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_slot;
  const uint32_t tR = tmem + 256u, tQ = tmem + 384u;
  volatile int* vfail = &fail;

  if (warp < F3_EPIW) {
    // ------------------------------------------------------------ epilogue warps
    pdl_wait();
    const int q = warp & 3, h = warp >> 2;
    const int lane_base = 32 * q;
    const uint32_t lane_addr = (uint32_t)lane_base << 16;
    const int xl = lane_base + lane;
    float pre[32];
    // the layout comes with a loss region only (MODE 1)
    const bool lay = MODE == 1 && r.p.layout != nullptr;
    auto prefetch = [&](const Item& it) {
      const int x = it.xt * 128 + xl, yb = it.yt * 128 + 32 * h;
      const float* tp;
      size_t step = N;
      int wrap = 32;   // row of the segment from which the layout starts again
      if (lay) {
        const int H = r.p.layout_h, W = r.p.layout_w;
        const int gy = wrapped(__ldg(r.p.origins + 2 * it.z) + yb, H);
        tp = r.p.layout + (size_t)gy * W + wrapped(__ldg(r.p.origins + 2 * it.z + 1) + x, W);
        step = W;
        wrap = H - gy;
      } else {
        tp = r.p.target + (size_t)it.z * N * N + (size_t)yb * N + x;
      }
      if (x < N && yb + 31 < N && wrap >= 32) {
#pragma unroll
        for (int e = 0; e < 32; ++e) pre[e] = __ldg(tp + e * step);
      } else if (lay) {
        const int H = r.p.layout_h;
#pragma unroll
        for (int e = 0; e < 32; ++e)
          pre[e] = (x < N && yb + e < N)
                       ? __ldg(tp + ((ptrdiff_t)e - (ptrdiff_t)((e + H - wrap) / H) * H) * (ptrdiff_t)step)
                       : 0.f;
      } else {
#pragma unroll
        for (int e = 0; e < 32; ++e) pre[e] = (x < N && yb + e < N) ? __ldg(tp + e * step) : 0.f;
      }
    };
    Item it = item_at(lo, T, B);
    if (n > 0) prefetch(it);
    for (int j = 0; j < n; ++j, it = item_next(it, T, B)) {
      const int x = it.xt * 128 + xl, yb = it.yt * 128 + 32 * h;
      const bool xin = x < N;
      const size_t base = (size_t)it.z * N * N;
      const uint32_t acc = tmem + (uint32_t)((j & 1) * 128) + lane_addr + (uint32_t)(32 * h);
      // rows 32 h + e0 .. + 15 of column xl: two 16-byte chunks of hi, two of lo
      auto store_a = [&](const float (&d)[16], int e0) {
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          uint4 h4, l4;
          split_pair(d[8 * c + 0], d[8 * c + 1], h4.x, l4.x);
          split_pair(d[8 * c + 2], d[8 * c + 3], h4.y, l4.y);
          split_pair(d[8 * c + 4], d[8 * c + 5], h4.z, l4.z);
          split_pair(d[8 * c + 6], d[8 * c + 7], h4.w, l4.w);
          uint8_t* w = sA + mn_chunk_offset((uint32_t)(32 * h + e0 + 8 * c), (uint32_t)xl);
          *reinterpret_cast<uint4*>(w) = h4;
          *reinterpret_cast<uint4*>(w + MN_LO) = l4;
        }
      };
      if (!pwait_warp(bar(SM + (j & 1)), (j >> 1) & 1, vfail, err, 31)) break;
      tc::fence_after();
      // d[e] becomes dL/dI at (yb + e0 + e, x), 0 outside the image.
      float s0 = 0.f, s1 = 0.f;
      bool bad;
      const int ny = xin ? N - yb : 0;   // rows e < ny lie in the image
      constexpr bool OUT = MODE == 2;
      if (MODE == 0) {
        // The window-free arithmetic of S3Resist::dldi on pixel pairs in packed FP32x2
        // (each lane rounded as the scalar operation, in the scalar order, so dL/dI is
        // the per-tile kernels' bit for bit; __expf and the reciprocal stay per lane).
        // Every dL/dI is non-finite exactly when its r is, and then so is the product
        // with 0 in chk. The loss terms are summed in two interleaved FP32 chains, at the
        // image edge in one of rounded squares (the FP64 losses of ragged images depend on
        // it in the ninth digit); past it r is 0, and with it dL/dI and the loss term.
        float2 chk = make_float2(0.f, 0.f), se = chk;
        const float2 na = make_float2(-r.p.alpha, -r.p.alpha);
        const float2 nt = make_float2(-r.p.thr, -r.p.thr);
        const float2 one = make_float2(1.f, 1.f), pw = make_float2(r.p.pe_weight, r.p.pe_weight);
        auto pixels = [&](auto edge) {
#pragma unroll
          for (int e0 = 0; e0 < 32; e0 += 16) {
            float d[16];
            tmem_ld16x(acc + (uint32_t)e0, d);
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
              const float2 z = __fmul2_rn(na, __fadd2_rn(make_float2(d[e], d[e + 1]), nt));
              const float2 den = __fadd2_rn(one, make_float2(__expf(z.x), __expf(z.y)));
              float2 W = make_float2(__fdividef(1.f, den.x), __fdividef(1.f, den.y));
              float2 rr = __fadd2_rn(W, make_float2(-pre[e0 + e], -pre[e0 + e + 1]));
              if (decltype(edge)::value) {
                // the accumulator there may hold anything
                if (e0 + e >= ny) rr.x = W.x = 0.f;
                if (e0 + e + 1 >= ny) rr.y = W.y = 0.f;
              }
              if (decltype(edge)::value && ny < 32)
                se.x = __fadd_rn(__fadd_rn(se.x, __fmul_rn(rr.x, rr.x)), __fmul_rn(rr.y, rr.y));
              else
                se = __ffma2_rn(rr, rr, se);
              const float2 g = __fmul2_rn(__fmul2_rn(__fmul2_rn(pw, rr), W),
                                          __fadd2_rn(one, make_float2(-W.x, -W.y)));
              chk = __ffma2_rn(g, make_float2(0.f, 0.f), chk);
              d[e] = g.x;
              d[e + 1] = g.y;
            }
            store_a(d, e0);
          }
        };
        // one branch for the warp: the tensor-memory accesses take all its lanes
        if (__all_sync(0xffffffffu, ny >= 32)) pixels(std::false_type{});
        else pixels(std::true_type{});
        s0 = se.x + se.y;
        bad = chk.x + chk.y != 0.f;
      } else {
        // Windows, penalty or image outputs: the scalar arithmetic, eight rows at a time so
        // that their window loads are in flight together.
        float chk = 0.f;
        int ry0 = 0, ry1 = 0;   // the rows e of the loss region
        if (r.p.region) {
          const int* R = r.p.region + 4 * it.z;
          const int x0 = __ldg(R + 2), x1 = __ldg(R + 3);
          ry0 = __ldg(R) - yb;
          ry1 = x >= x0 && x < x1 ? __ldg(R + 1) - yb : ry0;
        }
        const bool pen_on = r.p.penalty != 0.f || r.p.loss_penalty_term;
        if (MODE == 1 && r.p.region && __all_sync(0xffffffffu, ny >= 32)) {
          // The same arithmetic on pixel pairs where the windows come from the loss region and
          // no row is past the image: a window is 0 or 1, and 0 adds nothing to a sum. 16 micro
          // tiles of 1280^2: 120 us with the scalar form for them all, 100 us so.
          const int lo = max(ry0, 0), hi = min(ry1, 32);
          const uint32_t rm = hi > lo ? (0xffffffffu >> (32 - (hi - lo))) << lo : 0u;
          const float2 na = make_float2(-r.p.alpha, -r.p.alpha), nt = make_float2(-r.p.thr, -r.p.thr);
          const float2 one = make_float2(1.f, 1.f), pwt = make_float2(r.p.pe_weight, r.p.pe_weight);
          const float2 pen = make_float2(r.p.penalty, r.p.penalty);
          const float2 npt = make_float2(-r.p.pen_thr, -r.p.pen_thr);
          float2 ck = make_float2(0.f, 0.f);
#pragma unroll
          for (int e0 = 0; e0 < 32; e0 += 16) {
            float d[16];
            __syncwarp();
            tmem_ld16x(acc + (uint32_t)e0, d);
#pragma unroll
            for (int e = 0; e < 16; e += 2) {
              const float2 z = __fmul2_rn(na, __fadd2_rn(make_float2(d[e], d[e + 1]), nt));
              const float2 den = __fadd2_rn(one, make_float2(__expf(z.x), __expf(z.y)));
              const float2 W = make_float2(__fdividef(1.f, den.x), __fdividef(1.f, den.y));
              const float2 Tv = make_float2(pre[e0 + e], pre[e0 + e + 1]);
              const float2 rr = __fadd2_rn(W, make_float2(-Tv.x, -Tv.y));
              const bool inx = rm >> (e0 + e) & 1u, iny = rm >> (e0 + e + 1) & 1u;
              const float2 pw = make_float2(inx && (!r.p.region_main || Tv.x > 0.5f) ? 1.f : 0.f,
                                            iny && (!r.p.region_main || Tv.y > 0.5f) ? 1.f : 0.f);
              const float2 qw = make_float2(inx && pen_on && Tv.x < 0.5f ? 1.f : 0.f,
                                            iny && pen_on && Tv.y < 0.5f ? 1.f : 0.f);
              const float2 ep = __fadd2_rn(W, npt);
              const float2 ex = make_float2(fmaxf(ep.x, 0.f), fmaxf(ep.y, 0.f));
              const float2 r2 = __fmul2_rn(rr, rr), x2 = __fmul2_rn(ex, ex);
              s0 = __fmaf_rn(r2.y, pw.y, __fmaf_rn(r2.x, pw.x, s0));
              s1 = __fmaf_rn(x2.y, qw.y, __fmaf_rn(x2.x, qw.x, s1));
              const float2 sum =
                  __ffma2_rn(__fmul2_rn(pen, ex), qw, __fmul2_rn(__fmul2_rn(pwt, rr), pw));
              const float2 g = __fmul2_rn(__fmul2_rn(sum, W), __fadd2_rn(one, make_float2(-W.x, -W.y)));
              ck = __ffma2_rn(g, make_float2(0.f, 0.f), ck);
              d[e] = g.x;
              d[e + 1] = g.y;
            }
            store_a(d, e0);
          }
          chk = ck.x + ck.y;
        } else {
          const size_t i0 = base + (size_t)yb * N + x;
          const float* pwp = r.p.pe_window ? r.p.pe_window + i0 : nullptr;
          const float* qwp = r.p.pen_window ? r.p.pen_window + i0 : nullptr;
          float d[16];
#pragma unroll
          for (int e0 = 0; e0 < 32; e0 += 8) {
            if (e0 % 16 == 0) {
              __syncwarp();
              tmem_ld16x(acc + (uint32_t)e0, d);
            }
            float pw[8], qw[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              if (r.p.region) {
                const bool in = e0 + e >= ry0 && e0 + e < ry1;
                pw[e] = in && (!r.p.region_main || pre[e0 + e] > 0.5f) ? 1.f : 0.f;
                qw[e] = in ? 1.f : 0.f;   // used where T < 0.5
              } else {
                pw[e] = pwp && e0 + e < ny ? __ldg(pwp + (e0 + e) * N) : 1.f;
                qw[e] = qwp && e0 + e < ny ? __ldg(qwp + (e0 + e) * N) : pw[e];
              }
            }
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const float I = d[e0 % 16 + e], T = pre[e0 + e];
              const float W = r.sigmoid(I);
              const float rr = W - T;
              const bool in = e0 + e < ny;   // the accumulator past the edge may hold anything
              float sum = r.p.pe_weight * rr * pw[e];
              if (in) s0 += rr * rr * pw[e];
              if (pen_on && T < 0.5f) {
                const float ex = fmaxf(W - r.p.pen_thr, 0.f);
                if (in) s1 += ex * ex * qw[e];
                sum += r.p.penalty * ex * qw[e];
              }
              const float g = in ? sum * W * (1.f - W) : 0.f;
              if (OUT && in) {
                if (r.p.aerial) r.p.aerial[i0 + (size_t)(e0 + e) * N] = I;
                if (r.p.wafer) r.p.wafer[i0 + (size_t)(e0 + e) * N] = W;
              }
              chk = __fmaf_rn(g, 0.f, chk);
              d[e0 % 16 + e] = g;
            }
            if (e0 % 16) store_a(d, e0 - 8);
          }
        }
        bad = chk != 0.f;
      }
      tc::fence_before();
      fence_async_smem();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar(AFULL));
      if (bad) atomicOr(a.flag, 1);
      {
        const double v[2] = {(double)s0, (double)s1};
        const uint32_t rb = tc::smem_u32(&red_bar[j & 3]);
        if (MODE == 0) epi_put<1>(red, rb, j & 3, {v[0]});   // no penalty term
        else epi_put<2>(red, rb, j & 3, v);
      }
      if (j + 1 < n) prefetch(item_next(it, T, B));
    }
  } else if (warp < F3_MMAW) {
    // ------------------------------------------------------------ TMEM warps
    // Two warps per lane quarter, alternate 8-column groups. Iteration j: R(j), Q(j - 1).
    pdl_wait();
    const int lane_base = (warp & 3) * 32;
    const uint32_t lane_addr = (uint32_t)lane_base << 16;
    const int u0 = (warp - F3_EPIW) / 4;
    const int count = a.nrows_out * a.ncols;
    const int nu = (int)rf / 8;   // 8-column groups of the rows f
    Item it = item_at(lo, T, B), ip = it;
    for (int j = 0; j <= n; ++j, ip = it, it = item_next(it, T, B)) {
      if (j < n && !pwait_warp(bar(M1), j & 1, vfail, err, 33)) break;
      // MMA2(j - 1) has read sR and written Q(j - 1)
      if (j > 0 && !pwait_warp(bar(M2), (j - 1) & 1, vfail, err, 32)) break;
      tc::fence_after();
      if (j < n) {
        r_to_operand(tR + lane_addr, sR, (int)rf, lane_base, u0, F3_TMW / 4, nu);
        fence_async_smem();
        tc::fence_before();
        __syncwarp();
        // The loss sums of item j, by a warp without a share of Q, before it frees accR: their
        // slot is written again in item j + 4, and SMMA(j + 2) already follows MMA1(j + 1).
        if (warp == F3_MMAW - 1) {
          double t[2];
          if (epi_take<2>(red, tc::smem_u32(&red_bar[j & 3]), j & 3, (j >> 2) & 1, F3_EPIW, vfail,
                          err, 46, t) && lane == 0) {
            const size_t bid = ((size_t)it.z * T + it.yt) * T + it.xt;
            r.p.loss_partial[2 * bid] = t[0];
            r.p.loss_partial[2 * bid + 1] = t[1];
          }
        }
        if (lane == 0) {
          mbar_arrive(bar(RFREE));
          mbar_arrive(bar(SFULL));
        }
        __syncwarp();
      }
      if (j > 0) {
        q_to_partials(tQ + lane_addr,
                      a.part + (((size_t)ip.z * T + ip.yt) * T + ip.xt) * count, a, lane_base, u0,
                      F3_TMW / 4, nu);
        tc::fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(QFREE));
      }
    }
  } else if (warp == F3_MMAW) {
    // ------------------------------------------------------------ MMA warp
    const uint32_t lead = tc::elect_one();
    // the band operand image is written by the previous kernel of the stream
    pdl_wait();
    constexpr uint32_t idI = tc::idesc_bf16(128, 128), idA = tc::idesc_bf16(128, BN);
    constexpr uint32_t TXB = s2_tile_bytes(BN, 128);
    // copies of each operand so far, the tiles they hold and the last commit
    uint32_t nut = 0, nay = 0, ntx = 0, nty = 0, last_bar = 0, last_par = 0;
    int yay = -1, xtx = -1, yty = -1;
    auto commit = [&](int b, int par) {
      tc::mma_commit(bar(b), lead);
      last_bar = bar(b);
      last_par = (uint32_t)par & 1u;
    };
    // the operands of an item's synthesis, whose places the caller knows to be free
    auto load_ops = [&](const Item& it) {
      bulk_tile(uUt, Bimg + ((size_t)it.z * T + it.xt) * tb, tb, bar(UT), lead);
      ++nut;
      if (!res || it.yt != yay) {
        bulk_tile(uAYD, Aimg + (size_t)it.yt * tb, tb, bar(AY), lead);
        ++nay;
        yay = it.yt;
      }
    };
    Item it = item_at(lo, T, B), ip = it;   // items j and j - 1
    if (n > 0) load_ops(it);
    // Step j: SMMA(j), MMA2(j - 1), MMA1(j), then the copies for SMMA(j + 1).
    for (int j = 0; j <= n; ++j, ip = it, it = item_next(it, T, B)) {
      if (j < n) {
        if (!pwait_warp(bar(UT), j & 1, vfail, err, 35)) break;
        if (!pwait_warp(bar(AY), (nay - 1) & 1, vfail, err, 36)) break;
        tc::fence_after();
        // accI[j & 1] was read by epi(j - 2), before MMA1(j - 1) could start
        s2_mma_swapped_kp(tmem + (uint32_t)((j & 1) * 128), uAYD, uUt, kp, idI, lead);
        commit(SM + (j & 1), j >> 1);
        if (!res || it.xt != xtx) {
          // MMA1(j - 1) has read the TXD tile in use; shared, AYD must have been read too
          if (!res && !pwait_warp(bar(SM + (j & 1)), (j >> 1) & 1, vfail, err, 37)) break;
          bulk_tile_rows(uTXD, txImg + (size_t)it.xt * TXB, BN, (int)rf, bar(TX), lead);
          ++ntx;
          xtx = it.xt;
        }
      }
      if (j > 0) {
        const int i = j - 1;   // MMA2(i)
        if (ip.yt != yty) {
          if (i > 0 && !pwait_warp(bar(M2), (i - 1) & 1, vfail, err, 38)) break;
          bulk_tile_rows(uTYD, tyImg + (size_t)ip.yt * A2_A_BYTES, 128, (int)rn, bar(TY), lead);
          ++nty;
          yty = ip.yt;
        }
        if (!pwait_warp(bar(TY), (nty - 1) & 1, vfail, err, 39)) break;
        if (!pwait_warp(bar(SFULL), i & 1, vfail, err, 40)) break;
        if (i > 0 && !pwait_warp(bar(QFREE), (i - 1) & 1, vfail, err, 41)) break;
        tc::fence_after();
        s2_mma(tQ, uTYD, (int)rn, uR, (int)rf, 128, idA, lead);
        commit(M2, i);
      }
      if (j < n) {
        if (!pwait_warp(bar(TX), (ntx - 1) & 1, vfail, err, 42)) break;
        if (!pwait_warp(bar(AFULL), j & 1, vfail, err, 43)) break;
        if (j > 0 && !pwait_warp(bar(RFREE), (j - 1) & 1, vfail, err, 44)) break;
        tc::fence_after();
        s2_mma_amn(tR, uA, uTXD, (int)rf, idA | IDESC_A_MN, lead);
        commit(M1, j);
        if (j + 1 < n) {
          if (!pwait_warp(bar(M1), j & 1, vfail, err, 45)) break;
          load_ops(item_next(it, T, B));
        }
      }
    }
    if (*vfail) {
      // nothing of this CTA may still be in flight when it exits
      if (nut) tc::mbar_wait(bar(UT), (nut - 1) & 1);
      if (nay) tc::mbar_wait(bar(AY), (nay - 1) & 1);
      if (ntx) tc::mbar_wait(bar(TX), (ntx - 1) & 1);
      if (nty) tc::mbar_wait(bar(TY), (nty - 1) & 1);
      if (last_bar) tc::mbar_wait(last_bar, last_par);
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == F3_MMAW) tc::tmem_dealloc(tmem, 512);
}

template <int BN, int MODE>
static cudaError_t fused_tc3_m(cudaStream_t s, const void* Aimg, const void* Bimg, int N, int kp,
                               const ResistEpilogue& e, const Tc2Analysis& a, const void* tx,
                               const void* ty, int* err, int* nblocks, int batch) {
  const uint32_t tb = s2_tile_bytes(128, kp), rf = f3_rows(a.ncols), rn = f3_rows(a.nr);
  const bool res = f3_smem(rf, rn, tb, true) <= F3_SMEM_MAX;
  const size_t smem = f3_smem(rf, rn, tb, res);
  if (smem > F3_SMEM_MAX) return cudaErrorInvalidValue;
  cudaError_t r = cudaFuncSetAttribute(fused_tc3_kernel<BN, MODE>,
                                       cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (r != cudaSuccess) return r;
  const int T = (N + 127) / 128;
  const int items = T * T * batch;
  const int grid = items < sm_count() ? items : sm_count();
  *nblocks = T * T;
  return launch_pdl(fused_tc3_kernel<BN, MODE>, dim3(grid), dim3(F3_NT), smem, s,
                    static_cast<const uint8_t*>(Aimg), static_cast<const uint8_t*>(Bimg), N, kp, T,
                    batch, S3Resist{e}, a, (int)res, static_cast<const uint8_t*>(tx),
                    static_cast<const uint8_t*>(ty), err);
}
template <int BN>
static cudaError_t fused_tc3_t(cudaStream_t s, const void* Aimg, const void* Bimg, int N, int kp,
                               const ResistEpilogue& e, const Tc2Analysis& a, const void* tx,
                               const void* ty, int* err, int* nblocks, int batch) {
  const bool out = e.aerial || e.wafer;
  const bool plain = S3Resist{e}.plain() && !e.region;
  if (e.layout && (out || plain)) return cudaErrorInvalidValue;
  return out ? fused_tc3_m<BN, 2>(s, Aimg, Bimg, N, kp, e, a, tx, ty, err, nblocks, batch)
         : plain ? fused_tc3_m<BN, 0>(s, Aimg, Bimg, N, kp, e, a, tx, ty, err, nblocks, batch)
                 : fused_tc3_m<BN, 1>(s, Aimg, Bimg, N, kp, e, a, tx, ty, err, nblocks, batch);
}

bool tc3_fused_supported(int kp, int ncols, int nr) {
  if (!tc3_analysis_supported(ncols, nr) || !tc3_synth_supported(kp)) return false;
  return f3_smem(f3_rows(ncols), f3_rows(nr), s2_tile_bytes(128, kp), false) <= F3_SMEM_MAX;
}

cudaError_t launch_synth_resist_analysis_tc3(cudaStream_t s, const void* Aimg, const void* Bimg,
                                             int N, int kp, const ResistEpilogue& ep, int ncols,
                                             int nr, float2* part, int* flag, const void* tx_img,
                                             const void* ty_img, int* err, int* nblocks,
                                             int batch) {
  if (!tc3_fused_supported(kp, ncols, nr)) return cudaErrorInvalidValue;
  const Tc2Analysis a{nullptr, nullptr, flag, N, 0, 0, ncols, 2 * nr - 1, nr, 1, part};
  switch (tc2_analysis_rows(ncols)) {
    case 16: return fused_tc3_t<16>(s, Aimg, Bimg, N, kp, ep, a, tx_img, ty_img, err, nblocks, batch);
    case 32: return fused_tc3_t<32>(s, Aimg, Bimg, N, kp, ep, a, tx_img, ty_img, err, nblocks, batch);
    case 48: return fused_tc3_t<48>(s, Aimg, Bimg, N, kp, ep, a, tx_img, ty_img, err, nblocks, batch);
    case 64: return fused_tc3_t<64>(s, Aimg, Bimg, N, kp, ep, a, tx_img, ty_img, err, nblocks, batch);
    case 80: return fused_tc3_t<80>(s, Aimg, Bimg, N, kp, ep, a, tx_img, ty_img, err, nblocks, batch);
    case 96: return fused_tc3_t<96>(s, Aimg, Bimg, N, kp, ep, a, tx_img, ty_img, err, nblocks, batch);
    default: return cudaErrorInvalidValue;
  }
}

}  // namespace litho_b200
