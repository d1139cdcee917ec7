// HQQ (half-quadratic quantization) qparam search for Int4WeightOnlyConfig(use_hqq=True).
//
// Reference: torchao/quantization/quant_primitives.py:1998-2111 (_choose_qparams_and_quantize_affine_hqq) with
// optimize_weights_proximal_legacy (:1915-1973) and _convert_to_affinequantized_format (:1981-1995), called from
// AffineQuantizedTensor.from_hp_to_intx (affine_quantized_tensor.py:252-288).  The reference runs ~15 eager tensor ops
// per iteration over an fp32 copy of the weight; here an iteration is ONE pass over the bf16 weight (a warp per
// group, everything else in registers), and the early-stop test (a mean over the WHOLE tensor, so the iteration count
// is global) reads per-block partial sums of the error.  Arithmetic: fp32 with explicit single roundings where the
// reference has op boundaries (W * scale, + zero, ...), i.e. the reference's CPU path; its CUDA path runs the same
// iteration in fp16, which this does not imitate.  The result feeds the same packed format as the tinygemm recipe.
#include "common.cuh"
#include "f32x2.h"

namespace ao {

constexpr int kHqqWarps = 8;

__device__ __forceinline__ float warp_sum_h(float v) {
#pragma unroll
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// lane l of the group's warp owns elements l + 32 j, j < G / 32 (coalesced 64-byte rows of bf16)
template <int G>
__device__ __forceinline__ void load_group(const __nv_bfloat16* w, int64_t group, int lane, float (&v)[G / 32]) {
  const __nv_bfloat16* p = w + group * G + lane;
#pragma unroll
  for (int j = 0; j < G / 32; ++j) v[j] = __bfloat162float(p[32 * j]);
}

// scale = (15 / (max - min)).clamp(max = 2e4), zero = round(-min * scale)          (:2052-2060)
template <int G>
__global__ void __launch_bounds__(kHqqWarps * 32) hqq_init_kernel(const __nv_bfloat16* __restrict__ w, int64_t n_groups,
                                                                  float* __restrict__ scale, float* __restrict__ zero) {
  const int lane = threadIdx.x & 31;
  const int64_t group = (int64_t)blockIdx.x * kHqqWarps + (threadIdx.x >> 5);
  if (group >= n_groups) return;
  float v[G / 32];
  load_group<G>(w, group, lane, v);
  float mn = v[0], mx = v[0];
#pragma unroll
  for (int j = 1; j < G / 32; ++j) {
    mn = fminf(mn, v[j]);
    mx = fmaxf(mx, v[j]);
  }
#pragma unroll
  for (int o = 16; o; o >>= 1) {
    mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (lane == 0) {
    const float s = fminf(__fdiv_rn(15.f, __fsub_rn(mx, mn)), 2e4f);  // constant group: 15 / 0 = inf -> 2e4
    scale[group] = s;
    zero[group] = rintf(__fmul_rn(-mn, s));
  }
}

// One proximal iteration (:1958-1962):
//   W_q = round(W * scale + zero).clamp(0, 15);  W_r = (W_q - zero) / scale
//   W_e = sign(d) * relu(|d| - (1 / beta) * |d| ^ (p - 1)),  d = W - W_r
//   zero <- mean(W_q - (W - W_e) * scale);  err_partial[block] = sum |W - W_r|
template <int G>
__global__ void __launch_bounds__(kHqqWarps * 32) hqq_step_kernel(const __nv_bfloat16* __restrict__ w, int64_t n_groups,
                                                                  const float* __restrict__ scale, float* __restrict__ zero,
                                                                  float inv_beta, float lp_m1, float* __restrict__ err_partial,
                                                                  const int* __restrict__ stop) {
  __shared__ float s_err[kHqqWarps];
  if (stop != nullptr && *reinterpret_cast<const volatile int*>(stop) != 0) return;  // ao_b200_hqq_solve: the early stop has fired
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t group = (int64_t)blockIdx.x * kHqqWarps + warp;
  float err = 0.f;
  if (group < n_groups) {
    float v[G / 32];
    load_group<G>(w, group, lane, v);
    const float s = scale[group], z = zero[group];
    float acc = 0.f;
#pragma unroll
    for (int j = 0; j < G / 32; ++j) {
      const float wq = fminf(fmaxf(rintf(__fadd_rn(__fmul_rn(v[j], s), z)), 0.f), 15.f);
      const float wr = __fdiv_rn(__fsub_rn(wq, z), s);
      const float d = __fsub_rn(v[j], wr), ad = fabsf(d);
      float we = 0.f;  // d = 0: pow = inf, relu(-inf) = 0, sign = 0
      if (ad > 0.f) we = copysignf(fmaxf(__fsub_rn(ad, __fmul_rn(inv_beta, powf(ad, lp_m1))), 0.f), d);
      acc += __fsub_rn(wq, __fmul_rn(__fsub_rn(v[j], we), s));
      err += ad;
    }
    acc = warp_sum_h(acc);
    if (lane == 0) zero[group] = __fdiv_rn(acc, (float)G);
  }
  err = warp_sum_h(err);
  if (lane == 0) s_err[warp] = err;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int i = 0; i < kHqqWarps; ++i) t += s_err[i];  // fixed order: the early-stop decision is reproducible
    err_partial[blockIdx.x] = t;
  }
}

// W_q = round(W * scale + zero).clamp(0, 15) (:1971); scale_ao = 1 / scale (:2078), zero_ao = (8 - zero) * scale_ao
// (:1981-1995), both cast to bf16 (:2101-2102)
template <int G>
__global__ void __launch_bounds__(kHqqWarps * 32) hqq_finalize_kernel(const __nv_bfloat16* __restrict__ w, int64_t n_groups,
                                                                      const float* __restrict__ scale,
                                                                      const float* __restrict__ zero, int32_t* __restrict__ q,
                                                                      __nv_bfloat16* __restrict__ scale_out,
                                                                      __nv_bfloat16* __restrict__ zero_out) {
  const int lane = threadIdx.x & 31;
  const int64_t group = (int64_t)blockIdx.x * kHqqWarps + (threadIdx.x >> 5);
  if (group >= n_groups) return;
  float v[G / 32];
  load_group<G>(w, group, lane, v);
  const float s = scale[group], z = zero[group];
  int32_t* qp = q + group * G + lane;
#pragma unroll
  for (int j = 0; j < G / 32; ++j) qp[32 * j] = (int32_t)fminf(fmaxf(rintf(__fadd_rn(__fmul_rn(v[j], s), z)), 0.f), 15.f);
  if (lane == 0) {
    const float si = __fdiv_rn(1.f, s);
    scale_out[group] = __float2bfloat16_rn(si);
    zero_out[group] = __float2bfloat16_rn(__fmul_rn(__fsub_rn(8.f, z), si));
  }
}

// ---- the whole search: chunks of iterations with the group in registers --------------------------------------------------
// The iterations of a group depend on no other group; only the early stop looks at all of them.  So a thread keeps 32
// weights of a group in registers through kHqqChunk iterations and leaves behind the zero point after each of them (`hist`)
// and the block's error of each (`err`); hqq_mean_kernel adds the errors up, and whoever comes next works out
// from the means which iteration was the last (hqq_last), so that iterations past the stop cost work but change nothing.
//
// Bound by the fp32 pipe and instruction issue: ten iterations of all groups of 4096 x 4096 take 95 us.  What keeps the arithmetic at eleven
// instructions per pair of weights and iteration:
//  - pairs of weights in one register pair (add, mul, fma .f32x2: the single operation's rounding in each half.  But a product whose one use is a sum
//    can come out as one fused operation (f32x2.h), so such a sum is a fused one already, with a factor of one);
//  - the group's smallest and largest weight bound every |d| and say whether anything is clamped, so that, as a rule, neither
//    the clamp nor the shrinkage is looked at per weight.  |d| - c |d|^(p - 1) is not positive for |d| <= c^(1 / (2 - p)) (p < 1), 0.17 at the
//    reference's constants, which is above most weights' error: powf runs only above that threshold (less a margin of 1e-3, thousands of
//    times powf's error);
//  - (q - z) / s is x = n r, r = rn(1 / s), corrected once, x + r (n - x s): the correctly rounded quotient by Markstein's theorem (IBM J. Res.
//    Dev. 34, 1990), as neither r nor the remainder leaves the normal range (s in [2e-38, 2e4], |n| >= 2^-24 or 0);
//  - 32 weights per thread, packed as they come: 16 registers, and half as many exchanges per weight as with 16.
// Same numbers as hqq_step_kernel, bit for bit: there lane l of 32 adds elements l + 32 j and the lanes meet in steps of 16, 8, 4, 2, 1;
// here thread r of L = G / 32 holds the elements of the lanes r, r + L, .. of it, so the first steps of that tree are its own.
// What keeps the iterations few: a group whose zero point comes out as it went in, bit for bit, while no |d| of it can pass the smallest threshold still
// to come, gives the same zero point and error in every iteration that follows, so it is at rest and its lanes take the next group.  A zero point
// moves by the mean rounding error and settles as soon as no weight crosses a rounding boundary on the way: of normal weights in groups of 32 / 64 / 128 / 256
// 2.4 / 3.4 / 4.8 / 6.7 iterations of 20 move it, and one more shows it.  (Groups that never rest, as with weights of spread 3, where powf decides: hqq_deal_kernel.)
// The search over 4096 x 4096, groups of 64, 20 iterations, in all its kernels: 199 us with all iterations of all groups, 109 without those at rest
// (groups of 32 / 128 / 256: 213 / 226 / 186 -> 120 / 127 / 135).  Taken back: groups put together anew among a block's warps after each iteration (155),
// rounds of two and three iterations over a block's list (141).
constexpr int kHqqChunk = 10;   // iterations per launch: bounds hist to 10 numbers per group
constexpr int kHqqMaxIters = 64, kHqqLaunches = (kHqqMaxIters + kHqqChunk - 1) / kHqqChunk;
constexpr int kHqqPer = 32;     // weights per thread
constexpr int kHqqThreads = 256, kHqqBlocks = 4;   // per block; per SM: 64 registers (with all iterations of all groups 207 us, 3 blocks of 80 220; 16 weights per thread and 4 blocks 228)
constexpr int kHqqShare = 512;  // groups of a block at a time, at most; a multiple of 8

struct HqqChunk {
  float inv_beta[kHqqChunk], threshold[kHqqChunk];
  float lp_m1;
  float least;                  // smallest threshold of this launch's iterations and of those that follow
  int first, count;             // iterations [first, first + count)
};

// number of the last iteration among the first n whose means are known: the first one that does not improve (:1956; up to it each mean is the best so
// far), else n - 1.  All lanes of a warp together: one look at a mean after the other was 20 dependent loads at the start of every block.
__device__ __forceinline__ int hqq_last(const double* __restrict__ mean, int n, bool& stopped) {
  for (int first = 0; first < n; first += 32) {
    const int i = first + (threadIdx.x & 31);
    const bool worse = i < n && !(mean[i] < (i == 0 ? 1e4 : mean[i - 1]));
    const uint32_t any = __ballot_sync(0xffffffffu, worse);
    if (any != 0) {
      stopped = true;
      return first + __ffs(any) - 1;
    }
  }
  stopped = false;
  return n - 1;
}

// sign(d) relu(|d| - c |d|^(p - 1)); out of line: sixteen inlined powf would not fit the instruction caches
__device__ __noinline__ float hqq_shrink(float d, float c, float lp_m1) {
  const float ad = fabsf(d);
  return copysignf(fmaxf(__fsub_rn(ad, __fmul_rn(c, powf(ad, lp_m1))), 0.f), d);
}

// sum of leaf(i) over the pairs of lanes i, i + O, i + 2 O, .. < I in the order of a tree whose last step adds neighbours O apart; leaf gives
// the pair's sums of W_q - (W - W_e) s and of |d|
template <int I, int O, typename Leaf>
__device__ __forceinline__ void hqq_tree(int i, Leaf&& leaf, F2& acc, float2& e) {
  if constexpr (O >= I) {
    leaf(i, acc, e);
  } else {
    F2 acc2;
    float2 e2;
    hqq_tree<I, 2 * O>(i, leaf, acc, e);
    hqq_tree<I, 2 * O>(i + O, leaf, acc2, e2);
    acc = f2_add(acc, acc2);
    e = make_float2(e.x + e2.x, e.y + e2.y);
  }
}

// How the launches deal out the groups: in equal contiguous shares, as long as most groups can come to rest (a block's lanes then go on without a gap), else in
// pieces of what a block holds at once, to whoever is through with the last one.
struct HqqDeal {
  int fine, next[kHqqLaunches];  // pieces; the next one of each launch
};
__host__ __device__ __forceinline__ int hqq_piece(int group_size) { return 8192 / group_size; }   // groups of 256 threads (and of what an error is kept of)
// what the group's smallest and largest weight say about all of it: how far |d| can go (half a step, or what the clamp cuts off; the margins are a hundred times
// the roundings of t + z and of the quotient).  t_lo, t_hi: both times the scale
__device__ __forceinline__ float hqq_bound(float t_lo, float t_hi, float z, float recip) {
  const float q_lo = __fadd_rn(t_lo, z), q_hi = __fadd_rn(t_hi, z);
  return (fmaxf(0.51f, fmaxf(-q_lo, q_hi - 15.f)) + (fabsf(z) + 16.f) * 1e-6f) * recip;
}

// Pieces, where more than one in 16 of a sample of groups, as they are at first, has a |d| that may pass the smallest threshold: those never rest, and in shares
// blocks end with few of their warps at work, and rows cost differently.  4096 x 4096, groups of 64, us, in launches of a block per piece without rest / in shares /
// in pieces: normal weights (rows of e^(0.3 normal) times) the spread 3 1362 / 1546 / 1340, 1 1035 / 1290 / 1085, 0.8 753 / 919 / 775, 0.6 468 / 524 /
// 462, 0.4 320 / 279 / 310, 0.02 198 / 109 / 128.
// One launch of one block; 8 threads per group, 128 groups.
__global__ void __launch_bounds__(1024) hqq_deal_kernel(const __nv_bfloat16* __restrict__ w, int64_t n_groups, int G, float least, HqqDeal* __restrict__ deal) {
  const int64_t step = (n_groups + 127) / 128, group = (threadIdx.x >> 3) * step;
  float mn = INFINITY, mx = -INFINITY;
  if (group < n_groups) {
    for (int i = threadIdx.x & 7; i < G / 8; i += 8) {
      float f[8];
      unpack8(ldg128(reinterpret_cast<const unsigned short*>(w) + group * G + 8 * i), f);
#pragma unroll
      for (int j = 0; j < 8; ++j) mn = fminf(mn, f[j]), mx = fmaxf(mx, f[j]);
    }
  }
#pragma unroll
  for (int o = 4; o; o >>= 1) mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o)), mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  const float s = fminf(__fdiv_rn(15.f, __fsub_rn(mx, mn)), 2e4f), z = rintf(__fmul_rn(-mn, s));
  const bool never = !(hqq_bound(__fmul_rn(mn, s), __fmul_rn(mx, s), z, __frcp_rn(s)) <= 0.999f * least);
  const int count = __syncthreads_count(group < n_groups && never), all = __syncthreads_count(group < n_groups);
  if (threadIdx.x == 0) deal->fine = 16 * count > all;
  if (threadIdx.x < kHqqLaunches) deal->next[threadIdx.x] = 0;
}

// A block takes contiguous groups, at most kHqqShare at a time; L lanes of a warp take one group, two iterations, and then the next one if theirs is over, each
// at its own count.  rest: per group, the error of a group that has come to rest, else -1 (written by a launch for the next).
template <int G>
__global__ void __launch_bounds__(kHqqThreads, kHqqBlocks) hqq_iterate_kernel(const __nv_bfloat16* __restrict__ w, int64_t n_groups, HqqChunk ch, int share, int64_t n_err,
                                                                              float* __restrict__ scale, float* __restrict__ hist, double* __restrict__ err,
                                                                              const double* __restrict__ mean, float* __restrict__ rest, HqqDeal* __restrict__ deal) {
  constexpr int L = G / kHqqPer, I = 32 / L, J = G / 32;   // threads per group; its lanes per thread; elements per lane
  constexpr float kMagic = 12582912.f;                     // 1.5 * 2^23: adding and subtracting it is rint up to 2^22, and beyond that the clamp decides
  constexpr int kAtRest = 256;
  __shared__ float s_err[kHqqChunk][kHqqShare], s_z[kHqqShare], s_es[kHqqShare], s_threshold[kHqqChunk], s_inv_beta[kHqqChunk];
  __shared__ short s_done[kHqqShare];                      // iterations whose results are there; + kAtRest: the others are as the last one
  __shared__ short s_todo[kHqqShare];
  __shared__ int s_n, s_next;                              // how many; the next ones to be fetched
  __shared__ int s_piece;
  bool stopped = false;
  if (ch.first > 0) hqq_last(mean, ch.first, stopped);
  if (stopped) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, part = lane % L;
  if (threadIdx.x < kHqqChunk) s_threshold[threadIdx.x] = ch.threshold[threadIdx.x], s_inv_beta[threadIdx.x] = ch.inv_beta[threadIdx.x];
#pragma unroll 1
  for (int64_t turn = blockIdx.x;; turn += gridDim.x) {
    const bool fine = deal->fine != 0;
    if (threadIdx.x == 0) {
      s_n = s_next = 0;
      if (fine) s_piece = atomicAdd(&deal->next[ch.first / kHqqChunk], 1);
    }
    __syncthreads();
    const int64_t piece = fine ? s_piece : turn, base = piece * (fine ? hqq_piece(G) : share);
    if (base >= n_groups) break;
    const int most = fine ? hqq_piece(G) : share, here = (int)(n_groups - base < most ? n_groups - base : most);
#pragma unroll 1
    for (int g0 = warp * 32; g0 < here; g0 += kHqqThreads) {
      const int g = g0 + lane;
      bool todo = g < here;
      if (todo && ch.first > 0) {
        const float e = rest[base + g];
        s_z[g] = hist[(int64_t)(kHqqChunk - 1) * n_groups + base + g];
        todo = e < 0.f;
        if (!todo) s_es[g] = e, s_done[g] = kAtRest;
      }
      const uint32_t any = __ballot_sync(0xffffffffu, todo);
      int at = 0;
      if (any != 0 && lane == 0) at = atomicAdd(&s_n, __popc(any));
      at = __shfl_sync(0xffffffffu, at, 0) + __popc(any & ((1u << lane) - 1u));
      if (todo) s_todo[at] = (short)g;
    }
    __syncthreads();
    const int n = s_n;
    uint32_t v[kHqqPer / 2];       // pair (j I + i) / 2: weights i L + 32 j (lower half) and (i + 1) L + 32 j of the thread's, bf16
#pragma unroll
    for (int k = 0; k < kHqqPer / 2; ++k) v[k] = 0u;
    float s = 1.f, z = 0.f, t_lo = 0.f, t_hi = 0.f;
    int g = 0, it = 0;
    bool moves = false;            // the lane has a group, which is neither at rest nor through
    auto weights = [&](int k) { return f2(__uint_as_float(v[k] << 16), __uint_as_float(v[k] & 0xFFFF0000u)); };
#pragma unroll 1
    for (;;) {
      const uint32_t idle = __ballot_sync(0xffffffffu, !moves);
      int next = n;                // lane 0 looks for its warp: other warps move s_next meanwhile, and all lanes have to come to the same answer
      if (idle != 0) {
        if (lane == 0 && *reinterpret_cast<volatile int*>(&s_next) < n) next = atomicAdd(&s_next, __popc(idle) / L);
        next = __shfl_sync(0xffffffffu, next, 0);
      }
      if (next < n) {
        const int at = next + __popc(idle & ((1u << lane) - 1u)) / L;
        const bool fresh = !moves && at < n;
        if (fresh) {
          g = s_todo[at], it = 0, moves = true;
          const unsigned short* wp = reinterpret_cast<const unsigned short*>(w) + (base + g) * G;
          if constexpr (L <= 2) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint4 x[L];
#pragma unroll
              for (int h = 0; h < L; ++h) x[h] = ldg128(wp + (c * L + h) * 8);
              if constexpr (L == 1) {
                v[4 * c] = x[0].x, v[4 * c + 1] = x[0].y, v[4 * c + 2] = x[0].z, v[4 * c + 3] = x[0].w;
              } else {
                const uint32_t half = part ? 0x7632u : 0x5410u;
#pragma unroll
                for (int h = 0; h < L; ++h) v[4 * c + 2 * h] = __byte_perm(x[h].x, x[h].y, half), v[4 * c + 2 * h + 1] = __byte_perm(x[h].z, x[h].w, half);
              }
            }
          } else {
#pragma unroll
            for (int j = 0; j < J; ++j)
#pragma unroll
              for (int i = 0; i < I; i += 2) v[(j * I + i) / 2] = (uint32_t)wp[32 * j + L * i + part] | ((uint32_t)wp[32 * j + L * (i + 1) + part] << 16);
          }
        }
        uint32_t lo2 = v[0], hi2 = v[0];
#pragma unroll
        for (int k = 1; k < kHqqPer / 2; ++k) {
          asm("min.bf16x2 %0, %0, %1;" : "+r"(lo2) : "r"(v[k]));
          asm("max.bf16x2 %0, %0, %1;" : "+r"(hi2) : "r"(v[k]));
        }
        float mn = fminf(__uint_as_float(lo2 << 16), __uint_as_float(lo2 & 0xFFFF0000u)), mx = fmaxf(__uint_as_float(hi2 << 16), __uint_as_float(hi2 & 0xFFFF0000u));
#pragma unroll
        for (int o = L / 2; o; o >>= 1) {
          mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        if (fresh) {
          if (ch.first == 0) {     // (:2052-2060), as in hqq_init_kernel
            s = fminf(__fdiv_rn(15.f, __fsub_rn(mx, mn)), 2e4f);
            z = rintf(__fmul_rn(-mn, s));
            if (part == 0) scale[base + g] = s;
          } else {
            s = scale[base + g], z = s_z[g];
          }
          t_lo = __fmul_rn(mn, s), t_hi = __fmul_rn(mx, s);
        }
      }
      if (!__any_sync(0xffffffffu, moves)) break;
      // (the minus signs ride along: -x = n (-r), its remainder n + (-x) s, and -(x + r rem) = (-r) rem + (-x), all rounded as without them)
      const float nr = -__frcp_rn(s);
      const F2 s2 = f2(s, s), ns2 = f2(-s, -s), nr2 = f2(nr, nr), one = f2(1.f, 1.f), minus = f2(-1.f, -1.f), magic = f2(kMagic, kMagic), no_magic = f2(-kMagic, -kMagic);
#pragma unroll 1
      for (int twice = 0; twice < 2; ++twice) {
        // (the compiler would keep all weights unpacked and multiplied beside the packed ones, and have no registers left)
#pragma unroll
        for (int k = 0; k < kHqqPer / 2; ++k) asm volatile("" : "+r"(v[k]));
        const float thr = s_threshold[it];
        const F2 z2 = f2(z, z), nz2 = f2(-z, -z);
        // no weight of the group is clamped, and no |d| is above the threshold
        const float q_lo = __fadd_rn(t_lo, z), q_hi = __fadd_rn(t_hi, z), bound = hqq_bound(t_lo, t_hi, z, -nr);
        const bool inside = __all_sync(0xffffffffu, !moves || (q_lo >= -0.5f && q_hi < 15.5f));
        const bool small = __all_sync(0xffffffffu, !moves || bound <= 0.999f * thr);
        auto quotients = [&](F2 f, bool clamp, F2& wq, F2& nt) {   // W_q, -W * scale and d = W - W_r of a pair
          nt = f2_mul(f, ns2);
          wq = f2_add(f2_add(f2_fma(nt, minus, z2), magic), no_magic);
          if (clamp) {
            const float2 q = f2_get(wq);
            wq = f2(fminf(fmaxf(q.x, 0.f), 15.f), fminf(fmaxf(q.y, 0.f), 15.f));
          }
          const F2 n = f2_add(wq, nz2), nx = f2_mul(n, nr2);
          return f2_get(f2_add(f, f2_fma(f2_fma(nx, s2, n), nr2, nx)));
        };
        auto lane_pair = [&](int i, F2& acc, float2& e, auto&& one) {   // J elements each, one after the other
#pragma unroll
          for (int j = 0; j < J; ++j) {
            F2 a;
            const float2 d = one((j * I + i) / 2, a);
            acc = j == 0 ? a : f2_add(acc, a);
            e = j == 0 ? make_float2(fabsf(d.x), fabsf(d.y)) : make_float2(e.x + fabsf(d.x), e.y + fabsf(d.y));
          }
        };
        F2 acc;
        float2 e;
        if (small && inside) {         // W_e = 0: mean of W_q - W * scale
          hqq_tree<I, 2>(0, [&](int i, F2& a, float2& b) {
            lane_pair(i, a, b, [&](int k, F2& x) {
              F2 wq, nt;
              const float2 d = quotients(weights(k), false, wq, nt);
              x = f2_fma(nt, one, wq);
              return d;
            });
          }, acc, e);
        } else if (small) {
          hqq_tree<I, 2>(0, [&](int i, F2& a, float2& b) {
            lane_pair(i, a, b, [&](int k, F2& x) {
              F2 wq, nt;
              const float2 d = quotients(weights(k), true, wq, nt);
              x = f2_fma(nt, one, wq);
              return d;
            });
          }, acc, e);
        } else {
          const float c = s_inv_beta[it];
          hqq_tree<I, 2>(0, [&](int i, F2& a, float2& b) {
            lane_pair(i, a, b, [&](int k, F2& x) {
              F2 wq, nt;
              const float2 d = quotients(weights(k), true, wq, nt), f = f2_get(weights(k)), t = f2_get(nt), q = f2_get(wq);
              float2 u = make_float2(-t.x, -t.y);              // (W - W_e) * scale
              if (fabsf(d.x) > thr) u.x = __fmul_rn(__fsub_rn(f.x, hqq_shrink(d.x, c, ch.lp_m1)), s);
              if (fabsf(d.y) > thr) u.y = __fmul_rn(__fsub_rn(f.y, hqq_shrink(d.y, c, ch.lp_m1)), s);
              x = f2(__fsub_rn(q.x, u.x), __fsub_rn(q.y, u.y));
              return d;
            });
          }, acc, e);
        }
        const float2 last = f2_get(acc);
        float sum = last.x + last.y, es = e.x + e.y;
#pragma unroll
        for (int o = L / 2; o; o >>= 1) {
          sum += __shfl_xor_sync(0xffffffffu, sum, o);
          es += __shfl_xor_sync(0xffffffffu, es, o);
        }
        if (moves) {
          const float next = __fmul_rn(sum, 1.f / (float)G);   // (a power of two: the quotient, rounded once too)
          const bool rests = __float_as_uint(next) == __float_as_uint(z) && bound <= 0.999f * ch.least;
          z = next;
          moves = !rests && it + 1 < ch.count;
          if (part == 0) {
            hist[(int64_t)it * n_groups + base + g] = z;
            s_err[it][g] = es;
            if (!moves) s_z[g] = z, s_es[g] = es, s_done[g] = (short)(it + 1 + (rests ? kAtRest : 0));
          }
          it += moves;
        }
      }
    }
    __syncthreads();
    // what a group at rest would have given in the iterations that were left out
#pragma unroll 1
    for (int g = threadIdx.x; g < (here + 7) / 8 * 8; g += kHqqThreads) {
      const bool in = g < here;
      const int done = in ? s_done[g] : kAtRest;
      const float e = in ? s_es[g] : 0.f, z = in ? s_z[g] : 0.f;
      for (int it = done & (kAtRest - 1); it < ch.count; ++it) {
        s_err[it][g] = e;
        if (in) hist[(int64_t)it * n_groups + base + g] = z;
      }
      if (in) rest[base + g] = done & kAtRest ? e : -1.f;
    }
    __syncthreads();
    // eight groups at a time in fp32, as the blocks of hqq_step_kernel; fixed order: the stop is reproducible
#pragma unroll 1
    for (int it = warp; it < ch.count; it += kHqqThreads / 32) {
      double sum = 0.0;
      for (int b = lane * 8; b < here; b += 256) {
        float f = 0.f;
#pragma unroll
        for (int i = 0; i < 8; ++i) f += s_err[it][b + i];
        sum += (double)f;
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) err[(int64_t)it * n_err + piece] = sum;
    }
    __syncthreads();
  }
}

// block i: mean[first + i] = sum of err[i][..] / numel, in double, fixed order
__global__ void __launch_bounds__(1024) hqq_mean_kernel(const double* __restrict__ err, int64_t n_err, int64_t n_groups, int share, int piece, double inv_numel, int first,
                                                        double* __restrict__ mean, const HqqDeal* __restrict__ deal) {
  __shared__ double s_sum[1024];
  bool stopped = false;
  if (first > 0) hqq_last(mean, first, stopped);
  if (stopped) return;
  const int most = deal->fine ? piece : share;
  const int64_t n_blocks = (n_groups + most - 1) / most;
  const double* e = err + blockIdx.x * n_err;
  double t = 0.0;
  for (int64_t i = threadIdx.x; i < n_blocks; i += 1024) t += e[i];
  s_sum[threadIdx.x] = t;
  __syncthreads();
  for (int o = 512; o; o >>= 1) {
    if ((int)threadIdx.x < o) s_sum[threadIdx.x] += s_sum[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) mean[first + blockIdx.x] = s_sum[0] * inv_numel;
}

// the zero points of the last iteration that ran
__device__ __forceinline__ const float* hqq_zero(const float* hist, int64_t n_groups, const double* mean, int iters) {
  bool stopped;
  return hist + (int64_t)(hqq_last(mean, iters, stopped) % kHqqChunk) * n_groups;
}

template <int G>
__global__ void __launch_bounds__(kHqqWarps * 32) hqq_plain_kernel(const __nv_bfloat16* __restrict__ w, int64_t n_groups, const float* __restrict__ scale,
                                                                   const float* __restrict__ hist, const double* __restrict__ mean, int iters,
                                                                   int32_t* __restrict__ q, __nv_bfloat16* __restrict__ scale_out,
                                                                   __nv_bfloat16* __restrict__ zero_out) {
  const float* zero = hqq_zero(hist, n_groups, mean, iters);
  const int lane = threadIdx.x & 31;
  const int64_t group = (int64_t)blockIdx.x * kHqqWarps + (threadIdx.x >> 5);
  if (group >= n_groups) return;
  float v[G / 32];
  load_group<G>(w, group, lane, v);
  const float s = scale[group], z = zero[group];
  int32_t* qp = q + group * G + lane;
#pragma unroll
  for (int j = 0; j < G / 32; ++j) qp[32 * j] = (int32_t)fminf(fmaxf(rintf(__fadd_rn(__fmul_rn(v[j], s), z)), 0.f), 15.f);
  if (lane == 0) {
    const float si = __fdiv_rn(1.f, s);
    scale_out[group] = __float2bfloat16_rn(si);
    zero_out[group] = __float2bfloat16_rn(__fmul_rn(__fsub_rn(8.f, z), si));
  }
}

// clamp(rint(w * s + z), 0, 15) of eight weights as a packed word.  The clamp commutes with rint at 0 and 15 (and takes NaN to 0 either way); rint of
// what is left is an add of 1.5 * 2^23, whose bits are a constant plus q: shifted and added up, eight of them are the word plus a constant.
// (Product and sum one weight at a time: as f32x2 they came out as one fused operation, and one word in a million differed.)
__device__ __forceinline__ uint32_t packed_word(const uint4& raw, float s, float z) {
  constexpr uint32_t kMagic = 0x4B400000u;  // 1.5 * 2^23
  const uint32_t w2[4] = {raw.x, raw.y, raw.z, raw.w};
  uint32_t word = 0;
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    float a = __uint_as_float(w2[p] << 16), b = __uint_as_float(w2[p] & 0xFFFF0000u);
    a = __fadd_rn(fminf(fmaxf(__fadd_rn(__fmul_rn(a, s), z), 0.f), 15.f), __uint_as_float(kMagic));
    b = __fadd_rn(fminf(fmaxf(__fadd_rn(__fmul_rn(b, s), z), 0.f), 15.f), __uint_as_float(kMagic));
    word += (__float_as_uint(a) - kMagic) << (4 * nib_slot(2 * p));
    word += (__float_as_uint(b) - kMagic) << (4 * nib_slot(2 * p + 1));
  }
  return word;
}

// the same straight into the strip-major storage (include/ao_b200.h): a warp takes (16-row strip, 64-k tile) after tile, thread = 16-byte
// lane chunk of it, and then one thread per (row, group) of the parameters; padding rows and columns are zero in both.  Bound by HBM: weights in,
// words out.  With the group size known to the compiler and one 32-bit division per tile: 19.9 us for 4096 x 4096, against 24.6 with 64-bit
// divisions by it in every thread.
template <int G>
__global__ void __launch_bounds__(256) hqq_packed_kernel(const __nv_bfloat16* __restrict__ w, int64_t N, int64_t K, int64_t Np, int64_t Kp,
                                                         const float* __restrict__ scale, const float* __restrict__ hist, const double* __restrict__ mean,
                                                         int iters, uint4* __restrict__ packed, uint32_t* __restrict__ sz) {
  constexpr int kHalves = G < 64 ? 2 : 1;   // groups per tile
  const float* zero = nullptr;
  const int64_t groups = K / G;
  const uint32_t k_tiles = (uint32_t)(Kp / 64), groups_p = (uint32_t)(Kp / G);
  const uint32_t tiles = (uint32_t)(Np / 16) * k_tiles;                 // < 2^32 by far: a tile is 2 KB of weights
  const int lane = threadIdx.x & 31, g = lane >> 2, c = lane & 3;
  for (uint64_t tile = (uint64_t)blockIdx.x * 8 + (threadIdx.x >> 5); tile < tiles; tile += (uint64_t)gridDim.x * 8) {
    const uint32_t strip = (uint32_t)tile / k_tiles, kt = (uint32_t)tile - strip * k_tiles;
    const int64_t row0 = (int64_t)strip * 16 + g, k0 = (int64_t)kt * 64 + 8 * c;
    uint4 raw[4];
    float s[2][kHalves], z[2][kHalves];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      raw[j] = make_uint4(0u, 0u, 0u, 0u);
      const int64_t row = row0 + 8 * (j & 1), k = k0 + 32 * (j >> 1);
      if (row < N && k < K) raw[j] = ldg128(w + row * K + k);
    }
    if (zero == nullptr) zero = hqq_zero(hist, N * (K / G), mean, iters);  // (while the first weights are on their way)
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
      for (int h = 0; h < kHalves; ++h) {
        const int64_t row = row0 + 8 * r, grp = (k0 + 32 * h) / G;
        const bool there = row < N && grp < groups;
        s[r][h] = there ? scale[row * groups + grp] : 0.f;              // (padding: 0 * 0 + 0)
        z[r][h] = there ? zero[row * groups + grp] : 0.f;
      }
    uint32_t words[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const bool there = row0 + 8 * (j & 1) < N && k0 + 32 * (j >> 1) < K;
      words[j] = there ? packed_word(raw[j], s[j & 1][(j >> 1) * (kHalves - 1)], z[j & 1][(j >> 1) * (kHalves - 1)]) : 0u;
    }
    packed[tile * 32 + lane] = make_uint4(words[0], words[1], words[2], words[3]);
  }
  if (zero == nullptr) zero = hqq_zero(hist, N * (K / G), mean, iters);
  const uint64_t params = (uint64_t)Np * groups_p;
  for (uint64_t o = (uint64_t)blockIdx.x * 256 + threadIdx.x; o < params; o += (uint64_t)gridDim.x * 256) {
    const uint32_t pair = (uint32_t)(o >> 4), strip = pair / groups_p, grp = pair - strip * groups_p;   // [strip][group][16 rows]
    const int64_t row = (int64_t)strip * 16 + (o & 15);
    uint32_t word = 0;
    if (row < N && grp < groups) {
      const float sc = scale[row * groups + grp], si = __fdiv_rn(1.f, sc);
      word = float_to_bf16_bits(si) | (float_to_bf16_bits(__fmul_rn(__fsub_rn(8.f, zero[row * groups + grp]), si)) << 16);
    }
    sz[o] = word;
  }
}

}  // namespace ao

#include <cmath>

using namespace ao;

#define AO_HQQ_DISPATCH(KERNEL, ...)                                                 \
  switch (group_size) {                                                              \
    case 32: KERNEL<32><<<grid, kHqqWarps * 32, 0, s>>>(__VA_ARGS__); break;         \
    case 64: KERNEL<64><<<grid, kHqqWarps * 32, 0, s>>>(__VA_ARGS__); break;         \
    case 128: KERNEL<128><<<grid, kHqqWarps * 32, 0, s>>>(__VA_ARGS__); break;       \
    case 256: KERNEL<256><<<grid, kHqqWarps * 32, 0, s>>>(__VA_ARGS__); break;       \
    default: return AO_B200_ERR_UNSUPPORTED;                                         \
  }

extern "C" int64_t ao_b200_hqq_blocks(int64_t n_groups) { return (n_groups + kHqqWarps - 1) / kHqqWarps; }

extern "C" int ao_b200_hqq_init(const void* w, int64_t n_groups, int group_size, float* scale, float* zero, void* stream) {
  AO_CHECK_ARG(w && scale && zero && n_groups > 0 && n_groups <= ((int64_t)1 << 31) * kHqqWarps);
  auto s = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)ao_b200_hqq_blocks(n_groups);
  AO_HQQ_DISPATCH(hqq_init_kernel, static_cast<const __nv_bfloat16*>(w), n_groups, scale, zero);
  return ao_launch_status();
}

extern "C" int ao_b200_hqq_step(const void* w, int64_t n_groups, int group_size, const float* scale, float* zero,
                                double beta, double lp_norm, float* err_partial, void* stream) {
  AO_CHECK_ARG(w && scale && zero && err_partial && n_groups > 0 && beta > 0.0);
  auto s = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)ao_b200_hqq_blocks(n_groups);
  const float inv_beta = (float)(1.0 / beta), lp_m1 = (float)(lp_norm - 1.0);
  AO_HQQ_DISPATCH(hqq_step_kernel, static_cast<const __nv_bfloat16*>(w), n_groups, scale, zero, inv_beta, lp_m1, err_partial, nullptr);
  return ao_launch_status();
}

// The reference's global early stop (:1964-1972) decided on the device: current = mean |W - W_r| of the iteration that
// just ran (per-block partial sums added in a fixed order, in double); the first iteration that does not improve on the
// best so far sets `stop`, which makes the remaining step launches return at once (its zero is kept, as in the reference).
// state: [double best][int stop][int iterations run]
__global__ void __launch_bounds__(256) hqq_judge_kernel(const float* __restrict__ err_partial, int64_t n_blocks, double inv_numel,
                                                        double* __restrict__ state) {
  __shared__ double s_sum[256];
  int* flags = reinterpret_cast<int*>(state + 1);
  if (*reinterpret_cast<volatile int*>(flags) != 0) return;
  double t = 0.0;
  for (int64_t i = threadIdx.x; i < n_blocks; i += 256) t += (double)err_partial[i];
  s_sum[threadIdx.x] = t;
  __syncthreads();
  for (int o = 128; o; o >>= 1) {
    if ((int)threadIdx.x < o) s_sum[threadIdx.x] += s_sum[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const double current = s_sum[0] * inv_numel;
    flags[1] += 1;
    if (current < state[0]) state[0] = current;
    else flags[0] = 1;
  }
}

__global__ void hqq_state_init_kernel(double* state) {
  state[0] = 1e4;
  reinterpret_cast<int*>(state + 1)[0] = 0;
  reinterpret_cast<int*>(state + 1)[1] = 0;
}

extern "C" int ao_b200_hqq_solve(const void* w, int64_t n_groups, int group_size, const float* scale, float* zero,
                                 double beta, double kappa, double lp_norm, int iters, float* err_partial, void* state,
                                 void* stream) {
  AO_CHECK_ARG(w && scale && zero && err_partial && state && n_groups > 0 && beta > 0.0 && kappa > 0.0 && iters >= 1);
  AO_CHECK_ARG(ao_aligned(state, 8));
  auto s = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)ao_b200_hqq_blocks(n_groups);
  hqq_state_init_kernel<<<1, 1, 0, s>>>(static_cast<double*>(state));  // best = 1e4 (:1956), stop = iterations = 0
  const double inv_numel = 1.0 / ((double)n_groups * (double)group_size);
  const float lp_m1 = (float)(lp_norm - 1.0);
  const int* stop = reinterpret_cast<const int*>(static_cast<const double*>(state) + 1);
  for (int it = 0; it < iters; ++it) {
    const float inv_beta = (float)(1.0 / beta);
    AO_HQQ_DISPATCH(hqq_step_kernel, static_cast<const __nv_bfloat16*>(w), n_groups, scale, zero, inv_beta, lp_m1, err_partial, stop);
    hqq_judge_kernel<<<1, 256, 0, s>>>(err_partial, (int64_t)grid, inv_numel, static_cast<double*>(state));
    beta *= kappa;
  }
  return ao_launch_status();
}

extern "C" int ao_b200_hqq_finalize(const void* w, int64_t n_groups, int group_size, const float* scale, const float* zero,
                                    int32_t* q, void* scale_out, void* zero_out, void* stream) {
  AO_CHECK_ARG(w && scale && zero && q && scale_out && zero_out && n_groups > 0);
  auto s = static_cast<cudaStream_t>(stream);
  const unsigned grid = (unsigned)ao_b200_hqq_blocks(n_groups);
  AO_HQQ_DISPATCH(hqq_finalize_kernel, static_cast<const __nv_bfloat16*>(w), n_groups, scale, zero, q,
                  static_cast<__nv_bfloat16*>(scale_out), static_cast<__nv_bfloat16*>(zero_out));
  return ao_launch_status();
}

static int64_t hqq_search_blocks(int64_t n_groups, int group_size) { return (n_groups * group_size + 8191) / 8192; }

// [mean double x kHqqMaxIters][err double kHqqChunk x blocks][scale][hist kHqqChunk x n_groups][rest][deal]
extern "C" int64_t ao_b200_hqq_search_workspace_bytes(int64_t n_groups, int group_size) {
  if (n_groups <= 0 || group_size < kHqqPer) return 0;
  return (kHqqMaxIters + kHqqChunk * hqq_search_blocks(n_groups, group_size)) * 8 + (2 + kHqqChunk) * n_groups * 4 + (int64_t)sizeof(HqqDeal);
}

extern "C" int ao_b200_hqq_search(const void* w, int64_t N, int64_t K, int group_size, double beta, double kappa, double lp_norm, int iters,
                                  void* workspace, int64_t workspace_bytes, int32_t* q, void* scale_out, void* zero_out, int64_t Np, int64_t Kp,
                                  void* packed, void* scale_and_zero, void* stream) {
  AO_CHECK_ARG(w && workspace && N > 0 && K > 0 && beta > 0.0 && kappa > 0.0 && iters >= 1 && iters <= kHqqMaxIters);
  if (!(group_size == 32 || group_size == 64 || group_size == 128 || group_size == 256)) return AO_B200_ERR_UNSUPPORTED;
  AO_CHECK_ARG(K % group_size == 0 && ao_aligned(w, 16) && ao_aligned(workspace, 8));
  AO_CHECK_ARG((q && scale_out && zero_out) || (packed && scale_and_zero));
  AO_CHECK_ARG(!packed || (scale_and_zero && Np % 16 == 0 && Np >= N && Kp % 64 == 0 && Kp % group_size == 0 && Kp >= K && ao_aligned(packed, 16) &&
                           ao_aligned(scale_and_zero, 4)));
  const int64_t n_groups = N * (K / group_size), blocks = hqq_search_blocks(n_groups, group_size);
  AO_CHECK_ARG(blocks <= 2147483647);
  if (workspace_bytes < ao_b200_hqq_search_workspace_bytes(n_groups, group_size)) return AO_B200_ERR_WORKSPACE;
  auto s = static_cast<cudaStream_t>(stream);
  auto wb = static_cast<const __nv_bfloat16*>(w);
  double* mean = static_cast<double*>(workspace);
  double* err = mean + kHqqMaxIters;
  float* scale = reinterpret_cast<float*>(err + kHqqChunk * blocks);
  float* hist = scale + n_groups;
  float* rest = hist + kHqqChunk * n_groups;
  HqqDeal* deal = reinterpret_cast<HqqDeal*>(rest + n_groups);
  // as many blocks as the chip holds at once; their groups in equal shares, as many times as it takes (hqq_iterate_kernel: or in pieces)
  const int64_t most = (int64_t)kHqqBlocks * kNumSMs, rounds = (n_groups + most * kHqqShare - 1) / (most * kHqqShare);
  int share = (int)((n_groups + rounds * most * 8 - 1) / (rounds * most * 8) * 8);
  if (share < hqq_piece(group_size)) share = hqq_piece(group_size);   // (a block's worth of threads, and what `blocks` counts)
  const unsigned grid = (unsigned)((n_groups + share - 1) / share < most ? (n_groups + share - 1) / share : most);
  float inv_beta[kHqqMaxIters], threshold[kHqqMaxIters];
  for (int i = 0; i < iters; ++i) {
    inv_beta[i] = (float)(1.0 / beta);
    threshold[i] = lp_norm < 1.0 ? (float)(0.999 * std::pow(1.0 / beta, 1.0 / (2.0 - lp_norm))) : 0.f;
    beta *= kappa;
  }
  for (int first = 0; first < iters; first += kHqqChunk) {
    HqqChunk ch;
    ch.first = first;
    ch.count = iters - first < kHqqChunk ? iters - first : kHqqChunk;
    ch.lp_m1 = (float)(lp_norm - 1.0);
    ch.least = threshold[first];
    for (int i = first; i < iters; ++i) ch.least = threshold[i] < ch.least ? threshold[i] : ch.least;
    if (first == 0) hqq_deal_kernel<<<1, 1024, 0, s>>>(wb, n_groups, group_size, ch.least, deal);
    for (int i = 0; i < ch.count; ++i) ch.inv_beta[i] = inv_beta[first + i], ch.threshold[i] = threshold[first + i];
    switch (group_size) {
      case 32: hqq_iterate_kernel<32><<<grid, kHqqThreads, 0, s>>>(wb, n_groups, ch, share, blocks, scale, hist, err, mean, rest, deal); break;
      case 64: hqq_iterate_kernel<64><<<grid, kHqqThreads, 0, s>>>(wb, n_groups, ch, share, blocks, scale, hist, err, mean, rest, deal); break;
      case 128: hqq_iterate_kernel<128><<<grid, kHqqThreads, 0, s>>>(wb, n_groups, ch, share, blocks, scale, hist, err, mean, rest, deal); break;
      default: hqq_iterate_kernel<256><<<grid, kHqqThreads, 0, s>>>(wb, n_groups, ch, share, blocks, scale, hist, err, mean, rest, deal); break;
    }
    hqq_mean_kernel<<<ch.count, 1024, 0, s>>>(err, blocks, n_groups, share, hqq_piece(group_size), 1.0 / ((double)n_groups * (double)group_size), first, mean, deal);
  }
  if (packed) {
    const int64_t tiles = (Np / 16) * (Kp / 64), want = (tiles + 7) / 8;
    const unsigned grid = (unsigned)(want < 148 * 16 ? want : 148 * 16);
    auto* out = static_cast<uint4*>(packed);
    auto* sz = static_cast<uint32_t*>(scale_and_zero);
    switch (group_size) {
      case 32: hqq_packed_kernel<32><<<grid, 256, 0, s>>>(wb, N, K, Np, Kp, scale, hist, mean, iters, out, sz); break;
      case 64: hqq_packed_kernel<64><<<grid, 256, 0, s>>>(wb, N, K, Np, Kp, scale, hist, mean, iters, out, sz); break;
      case 128: hqq_packed_kernel<128><<<grid, 256, 0, s>>>(wb, N, K, Np, Kp, scale, hist, mean, iters, out, sz); break;
      default: hqq_packed_kernel<256><<<grid, 256, 0, s>>>(wb, N, K, Np, Kp, scale, hist, mean, iters, out, sz); break;
    }
  }
  if (q) {
    const unsigned grid = (unsigned)ao_b200_hqq_blocks(n_groups);
    AO_HQQ_DISPATCH(hqq_plain_kernel, wb, n_groups, scale, hist, mean, iters, q, static_cast<__nv_bfloat16*>(scale_out),
                    static_cast<__nv_bfloat16*>(zero_out));
  }
  return ao_launch_status();
}
