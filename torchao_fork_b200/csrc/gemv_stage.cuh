// Staging of the activations of a decode GEMV (gemv_int8_fused.cu, gemv_int4_fused.cu) for 2 .. 16 rows, the rows in registers: x (* norm_w)
// -> per-row power-of-two scaling -> fp16 in shared memory, row scales, sums over a segment of k.
//
// The GEMVs of a batch are bound by this staging, not by their weights (which stream into the ring meanwhile): a CTA turns all
// activations into fp16 before its first product.  8 rows of 4096, from the end of the kernel in front: 4.4 us with the norm and 3.9 without
// (7.3 and 5.7 in loops over four rows at a time, with the values on their way through shared memory); one token of 8 sequences
// through four layers of int8: 341 us instead of 367.
// Here every load of a thread is in flight at once, the values stay in registers between the two passes, and where R sums are wanted over
// the lanes of a warp, every exchange halves the number of sums a lane still holds (R = 8: 9 exchanges instead of 40).  The sums
// are those of a butterfly per row, in the same order: same bits.
#pragma once
#include <cuda_fp16.h>

#include "common.cuh"
#include "per_device.h"

namespace ao {

// x[j] of the lanes that differ in the bits O, O / 2, .., 1 of their number, combined; what a lane ends with belongs to row
// (lane % (2 O)) * R / (2 O) + j, j < max(1, R / (2 O))
template <int R, int O, typename Op>
__device__ __forceinline__ void fold_rows(float (&x)[R], int lane, Op op) {
  int n = R / 2;
#pragma unroll
  for (int o = O; o; o >>= 1, n >>= 1) {
    if (n >= 1) {
      const bool up = (lane & o) != 0;
#pragma unroll
      for (int j = 0; j < R / 2; ++j) {
        if (j < n) {
          const float keep = up ? x[j + n] : x[j], send = up ? x[j] : x[j + n];
          x[j] = op(keep, __shfl_xor_sync(0xffffffffu, send, o));
        }
      }
    } else {
      x[0] = op(x[0], __shfl_xor_sync(0xffffffffu, x[0], o));
    }
  }
}

// Rows row0 .. row0 + R - 1 (below M), N chunks of 8 elements per row and thread, CT threads.  part: [16][CT / 32][2]; row_scale: [16].
// chunk(f, dn, sums) -> the fp16 words of a chunk with values f, dn the row's factor; what it leaves in sums[0 .. S) is added up over the
// SEG / 8 chunks of a segment and handed to done(segment, row, sums) by one lane per row.
// (Sixteen rows are two calls: their 64 registers of values and the rest do not fit 96.)
template <int R, int N, int CT, int S, int SEG, typename Chunk, typename Done>
__device__ __forceinline__ void stage_rows(const __nv_bfloat16* x, int64_t ldx, int64_t Kx, int row0, int M, const __nv_bfloat16* norm_w, float eps,
                                           int chunks_per_row, uint8_t* x_s, uint32_t x_row_bytes, float* part, float* row_scale, Chunk chunk, Done done) {
  constexpr int W = CT / 32;
  static_assert(W == 16 && (R == 4 || R == 8), "");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const auto add = [](float a, float b) { return a + b; };
  const auto larger = [](float a, float b) { return fmaxf(a, b); };
  uint4 wn[N], v[N][R];
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int64_t k0 = (int64_t)(i * CT + tid) * 8;
    wn[i] = make_uint4(0u, 0u, 0u, 0u);
    if (norm_w != nullptr && k0 < Kx) wn[i] = __ldg(reinterpret_cast<const uint4*>(norm_w + k0));   // not the work of the kernel in front
  }
  grid_dependency_wait();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int64_t k0 = (int64_t)(i * CT + tid) * 8;
#pragma unroll
    for (int m = 0; m < R; ++m) {
      v[i][m] = make_uint4(0u, 0u, 0u, 0u);
      if (row0 + m < M && k0 < Kx) v[i][m] = *reinterpret_cast<const uint4*>(x + (row0 + m) * ldx + k0);
    }
  }
  float ss[R], am[R];
#pragma unroll
  for (int m = 0; m < R; ++m) {
    ss[m] = am[m] = 0.f;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      uint4& w = v[i][m];
      float f[8];
      if (norm_w != nullptr) {
        unpack8(w, f);
#pragma unroll
        for (int e = 0; e < 8; ++e) ss[m] = fmaf(f[e], f[e], ss[m]);
        // bf16(x * w): the fp32 product of two bf16 is exact, so one packed multiply is the product rounded once
        const auto mul = [](uint32_t a, uint32_t b) {
          uint32_t d;
          asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
          return d;
        };
        w = make_uint4(mul(w.x, wn[i].x), mul(w.y, wn[i].y), mul(w.z, wn[i].z), mul(w.w, wn[i].w));
      }
      unpack8(w, f);
#pragma unroll
      for (int e = 0; e < 8; ++e) am[m] = fmaxf(am[m], fabsf(f[e]));
    }
  }
  constexpr int kOwn = 32 / R;   // lanes that end with the same row's numbers
  fold_rows<R, 16>(ss, lane, add);
  fold_rows<R, 16>(am, lane, larger);
  if (lane % kOwn == 0) *reinterpret_cast<float2*>(part + ((row0 + lane / kOwn) * W + warp) * 2) = make_float2(ss[0], am[0]);
  named_bar_sync(1, CT);
  // every warp adds the 16 partials of all rows: half a warp, half of the rows
  float t[R / 2], a[R / 2];
#pragma unroll
  for (int j = 0; j < R / 2; ++j) {
    const float2 p = *reinterpret_cast<const float2*>(part + ((row0 + (lane >> 4) * (R / 2) + j) * W + (lane & 15)) * 2);
    t[j] = p.x, a[j] = p.y;
  }
  fold_rows<R / 2, 8>(t, lane, add);
  fold_rows<R / 2, 8>(a, lane, larger);
  // 2^e brings the row's largest magnitude to [2^13, 2^14); below 2^-113 to less, as 2^-e has to be a number, which leaves every bf16 exact all the same
  int e = 0;
  if (a[0] > 0.f) e = max(-126, (int)((__float_as_uint(a[0]) >> 23) & 0xFF) - 127 - 13);
  const float up = __uint_as_float((uint32_t)(e + 127) << 23), own_dn = __uint_as_float((uint32_t)(127 - e) << 23);
  if (warp == 0 && lane % kOwn == 0)   // for the epilogue warp
    row_scale[row0 + lane / kOwn] = norm_w != nullptr ? up * rsqrtf(t[0] / (float)Kx + eps) : up;
  float dn[R];
#pragma unroll
  for (int m = 0; m < R; ++m) dn[m] = __shfl_sync(0xffffffffu, own_dn, m * kOwn);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const int ci = i * CT + tid;
    if (ci - lane >= chunks_per_row) continue;   // (the whole warp)
    float sums[S][R];
#pragma unroll
    for (int m = 0; m < R; ++m) {
      float f[8], own[S];
      unpack8(v[i][m], f);
      const uint4 w = chunk(f, dn[m], own);
      if (row0 + m < M && ci < chunks_per_row) *reinterpret_cast<uint4*>(x_s + (size_t)(row0 + m) * x_row_bytes + (size_t)ci * 16) = w;
#pragma unroll
      for (int s = 0; s < S; ++s) sums[s][m] = own[s];
    }
    constexpr int C = SEG / 8, kEach = R > C ? R / C : 1, kSame = C > R ? C / R : 1;   // lanes per segment; sums per lane, or lanes per sum
#pragma unroll
    for (int s = 0; s < S; ++s) fold_rows<R, C / 2>(sums[s], lane, add);
    if (ci < chunks_per_row && lane % kSame == 0) {
#pragma unroll
      for (int j = 0; j < kEach; ++j) {
        float own[S];
#pragma unroll
        for (int s = 0; s < S; ++s) own[s] = sums[s][j];
        done(ci / C, row0 + (lane % C) * R / C + j, own);
      }
    }
  }
}

// ---- k shared out over the CTAs of a cluster (SPLIT kernels) ----------------------------------------------------------------
// For activations that one CTA cannot hold, or takes long to stage.  Each CTA sums its part of a strip; those of the other ranks send theirs
// into shared memory of rank 0 (st.async), which has room for all its strips, adds them in rank order and finishes the strip: nobody waits to send.
constexpr int kMaxSplitStrips = 32;   // strips of a cluster
// Stages of the weight ring that have to fit beside the activations and the inbox.  With three the ring no longer covers the way from memory (int4
// 8192 x 28672, 8 rows 46 us and the GEMM 45 to 46, 16384 x 28672, 7 rows 82 and 78; int8 104 and 86); with four it does (40.5 at 7 rows; 73 at 6).
constexpr int kSplitStages = 4;

// Which products of 2 to 8 rows without a norm share k: a line for each kernel that the call would take otherwise (us, that kernel / halves or
// quarters of k).
//  - the GEMV over whole rows (they fit one CTA): 57344 activations.  int8, 8 rows of 3072 x 8192 12.1 / 8.7, of 8192 x 8192 19.1 / 16.0, 4 of
//    4096 x 14336 15.4 / 14.7; int4 10.3 / 8.3, 15.5 / 13.4, 15.9 / 13.4.  Below: int8, 8 rows of 5120 x 5120 9.9 / 10.0, 4 of 8192 x 8192 14.4 / 15.2;
//  - nothing fits, so a strip kernel or the GEMM: 3 rows (the kernels for up to 2 rows ask for less).  Int4 4096 x 14336, 8 rows 17.8 / 14.1, 8192 x 28672,
//    3 / 7 rows 45.2 / 38.7, 45.5 / 40.5 (the GEMM since 35.8: for groups of 128 and 256 ao_b200_int4_mm does not ask there); int8 17.7 / 16.4, 50.7 / 40.9, 50.8 / 45.5, 8 rows 50.8 / 49.4;
//  - the GEMM, which adds residuals: k of 8192.  Int4 3072 x 8192, 2 / 8 rows 14.9 / 7.6, 16.2 / 8.2, 8192 x 28672, 3 / 7 rows 45.5 / 38.2, 46 / 40.4; int8
//    15.7 / 8.1, 17.4 / 8.7, 48.4 / 40.1, 49.5 / 45.4, 28672 x 8192, 8 rows 49.7 / 44.7.  Below: int8 28672 x 4096, 8 rows 30 / 36.
// More rows are not split: twice the products per weight in CTAs with half the k (16 rows of 8192 x 8192: 26 us against the GEMM's 23).
enum class Instead { kWholeRows, kNothingFits, kGemm };
static inline bool share_k(int64_t M, int64_t Kp, Instead instead) {
  if (M < 2 || M > 8) return false;
  return instead == Instead::kWholeRows ? M * Kp >= 57344 : instead == Instead::kNothingFits ? M >= 3 : Kp >= 8192;
}

// at the start, by every thread: rank 0's epilogue warp makes the barriers of its `strips` strips; `bytes` arrive at each
__device__ __forceinline__ void split_begin(bool owner, int strips, uint64_t* in_full, uint32_t bytes, int lane) {
  if (owner) {
    if (lane < strips) {
      mbar_init(&in_full[lane], 1);
      fence_barrier_init();
      mbar_arrive_expect_tx(&in_full[lane], bytes);
    }
    __syncwarp();
  }
  asm volatile("barrier.cluster.arrive.release;" ::: "memory");
}
// before the first send, and before a thread leaves
__device__ __forceinline__ void split_meet() { asm volatile("barrier.cluster.wait.acquire;" ::: "memory"); }
// The epilogue warp's sums of strip li, scaled (each rank has scaled its part of a row by itself): false, and sent on, on the other ranks; all
// parts added on rank 0.  The wait is bounded: NaN after about two seconds, which the caller takes for sums that are to be done again.
template <int MT>
__device__ __forceinline__ bool split_sums(float4 (&sum)[MT], const float* row_scale, uint64_t* in_full, float4* inbox, int li, int rank, int ks, int lane) {
  const int c = lane & 3;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    const float r0 = row_scale[8 * mt + 2 * c], r1 = row_scale[8 * mt + 2 * c + 1];
    sum[mt] = make_float4(sum[mt].x * r0, sum[mt].y * r1, sum[mt].z * r0, sum[mt].w * r1);
  }
  if (rank != 0) {
#pragma unroll
    for (int mt = 0; mt < MT; ++mt) {
      uint32_t to, bar;
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(to) : "r"(smem_u32(inbox + ((li * (ks - 1) + rank - 1) * MT + mt) * 32 + lane)));
      asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(bar) : "r"(smem_u32(&in_full[li])));
      asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(to), "f"(sum[mt].x), "f"(sum[mt].y),
                   "f"(sum[mt].z), "f"(sum[mt].w), "r"(bar)
                   : "memory");
    }
    return false;
  }
  const long long t0 = clock64();
  bool here = true;
  while (here && !mbar_try_wait(&in_full[li], 0)) here = clock64() - t0 < 4000000000ll;
#pragma unroll
  for (int mt = 0; mt < MT; ++mt) {
    for (int r = 0; r + 1 < ks; ++r) {
      const float4 v = inbox[((li * (ks - 1) + r) * MT + mt) * 32 + lane];
      sum[mt] = make_float4(sum[mt].x + v.x, sum[mt].y + v.y, sum[mt].z + v.z, sum[mt].w + v.w);
    }
    if (!here) sum[mt] = make_float4(__int_as_float(0x7FFFFFFF), __int_as_float(0x7FFFFFFF), __int_as_float(0x7FFFFFFF), __int_as_float(0x7FFFFFFF));
  }
  return true;
}
// The sums of a strip (lane (g, c): rows g and g + 8, x and y, z and w; columns 2 c, 2 c + 1 of the M) where some are not finite, done again by the whole
// warp: an infinity has lost its sign against the weights' offset, or one rank's part has overflowed where the total does not.  weights(row, k, w): eight
// of them from k on, as fp32.  A row of x with infinities or NaN is decided by these alone; one without is added up in 64 bits and rounded to 32 once, a
// weight row at a time.  (Every row with an infinity: 8 rows of 4096 x 14336 0.23 ms, 7 of 8192 x 28672 about 1.5.)
template <typename Weights>
__device__ __forceinline__ float4 split_again(float4 sum, const __nv_bfloat16* x, int64_t ldx, int M, int64_t Kx, int lane, Weights&& weights) {
  const auto bad = [](float v) { return !(fabsf(v) < INFINITY); };
#pragma unroll 1
  for (int m = 0; m < M; ++m) {
    const bool mine = (lane & 3) == m >> 1;
    const bool low = mine && bad(m & 1 ? sum.y : sum.x), high = mine && bad(m & 1 ? sum.w : sum.z);
    if (!__any_sync(0xffffffffu, low || high)) continue;
    const __nv_bfloat16* row_x = x + m * ldx;
    double t = 0.0;               // of weight row lane & 15
    bool odd = false;             // the row of x has something that is not finite
    const auto top = [](uint32_t u) { return (u & 0x7F807F80u) + 0x00800080u; };   // the upper bit of a half: its exponent is all ones
#pragma unroll 1
    for (int64_t k0 = 0; k0 < Kx; k0 += 8 * 256) {
      uint4 v[8];
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int64_t k = k0 + i * 256 + 8 * lane;
        v[i] = make_uint4(0u, 0u, 0u, 0u);
        if (k < Kx) v[i] = *reinterpret_cast<const uint4*>(row_x + k);
      }
      uint32_t own = 0u;          // which of this lane's eight
#pragma unroll
      for (int i = 0; i < 8; ++i) own |= (((top(v[i].x) | top(v[i].y) | top(v[i].z) | top(v[i].w)) & 0x80008000u) != 0u ? 1u : 0u) << i;
      uint32_t at = __ballot_sync(0xffffffffu, own != 0u);
      odd = odd || at != 0u;
#pragma unroll 1
      for (; at != 0u; at &= at - 1) {
        const int src = __ffs(at) - 1;
#pragma unroll 1
        for (uint32_t left = __shfl_sync(0xffffffffu, own, src); left != 0u; left &= left - 1) {
          float f[8], w[8];
          const int64_t there = k0 + (__ffs(left) - 1) * 256 + 8 * src;
          unpack8(*reinterpret_cast<const uint4*>(row_x + there), f);
          weights(lane & 15, there, w);
#pragma unroll
          for (int e = 0; e < 8; ++e)
            if (bad(f[e])) t += (double)f[e] * (double)w[e];
        }
        if (__all_sync(0xffffffffu, t != t)) break;   // (NaN stays NaN)
      }
      if (__all_sync(0xffffffffu, t != t)) break;
    }
    if (!odd) {
#pragma unroll 1
      for (int row = 0; row < 16; ++row) {
        if (!__any_sync(0xffffffffu, (lane >> 2) == (row & 7) && (row < 8 ? low : high))) continue;
        double part = 0.0;
#pragma unroll 2
        for (int64_t k = 8 * lane; k < Kx; k += 256) {
          float f[8], w[8];
          unpack8(*reinterpret_cast<const uint4*>(row_x + k), f);
          weights(row, k, w);
#pragma unroll
          for (int e = 0; e < 8; ++e) part += (double)f[e] * (double)w[e];
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
        if ((lane & 15) == row) t = part;
      }
    }
    const float lo = __shfl_sync(0xffffffffu, (float)t, lane >> 2), hi = __shfl_sync(0xffffffffu, (float)t, (lane >> 2) + 8);
    if (low) (m & 1 ? sum.y : sum.x) = lo;
    if (high) (m & 1 ? sum.w : sum.z) = hi;
  }
  return sum;
}
// whether any of the sums that count is not finite, on any lane
__device__ __forceinline__ bool split_overflowed(const float4& s, int M, int lane) {
  const int m = 2 * (lane & 3);
  const bool low = fabsf(s.x) < INFINITY && fabsf(s.z) < INFINITY, high = fabsf(s.y) < INFINITY && fabsf(s.w) < INFINITY;
  return __any_sync(0xffffffffu, (m < M && !low) || (m + 1 < M && !high));
}
// Clusters of ks CTAs, one per SM, that run at the same time: the SMs of a GPC need not be a multiple of ks.  The same for every shape, so asked
// for once per kernel, ks and device.  (0 or less: none.)
static inline int split_clusters(const void* kern, cudaLaunchConfig_t cfg, int ks, int sms, NumberPerDevice (&at_once)[5]) {
  int device = -1;
  cudaGetDevice(&device);
  return at_once[ks].get(device, [&] {
    cfg.gridDim = dim3((unsigned)(sms / ks * ks));
    cfg.dynamicSmemBytes = 200 * 1024;
    cfg.numAttrs = 1;   // the cluster dimension
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) cudaGetLastError(), n = 0;
    return n > 0 ? n : -1;
  });
}

}  // namespace ao
