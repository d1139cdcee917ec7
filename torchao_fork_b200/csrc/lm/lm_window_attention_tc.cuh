// Attention under a sliding window for prompt portions on tcgen05 / tensor memory: what window_attention_prompt_kernel computes
// (lm_window_attention_mma.cu; the same three bf16 parts of the fp32 weights, the same masks, keys and values), for tiles of 128
// rows of one sequence x one query head, 128 keys at a time.
//
//   S = Q K^T       128 x 128 fp32 in tensor memory, two buffers: the next tile's product runs while this tile's weights are made
//   P               exp2(s - m), split exactly into bf16 parts p1 + p2 + p3 and stored to tensor memory (p1, p2 over S, p3 beside
//                   it) as the A operand of
//   O += P V        three MMAs over the same values, 128 x dv fp32 in tensor memory
// m is the largest score so far when it grew by more than 2^8: O is rescaled only then (the weights stay below 256, their
// bf16 parts lose nothing), and sum and product carry the same factor.
//
// Key and value tiles lie in shared memory as [64 columns][128 rows][128 bytes, swizzled]: K-major for the keys, the same
// order read MN-major for the values, so both come as they are stored: a tile whose keys are neighbours in the step's rows or in
// the ring by one TMA copy per 64 columns, others (a boundary between the stores, the last tile of a run) by 16-byte
// asynchronous copies.  (16-byte copies for every tile took 5000 clocks a tile.)
//
// Bound by the tensor cores: 128 x 128 x (d + 3 dv) per tile, 2048 clocks at d = dv = 128, beside 1650 issue slots of the weights
// (two threads per row).  One CTA per SM; late tiles, which see the most keys, start first.
// Roles (416 threads): warps 0-7 weights and epilogue (lane quadrant = warp % 4, half of the columns = warp / 4), 8-11 loads,
// 12 MMA issue.  Every wait is bounded; a CTA that gives up writes NaN.
#pragma once
#include <cuda.h>

#include "lm_mma.cuh"

namespace lm {

constexpr int kTcRows = 128, kTcKeys = 128, kTcThreads = 13 * 32;
constexpr uint32_t kTcHeader = 4096;   // barriers, row exchange

struct WinPromptArgs {
  const float* qn;                         // [n][H][NM][d] fp32
  const __nv_bfloat16 *kn, *vn;            // step rows [n][G][NM][d], [n][G][dv]
  const __nv_bfloat16 *ring_k, *ring_v;    // [slots][ring][G][NM d], [slots][ring][G][dv]
  const __nv_bfloat16 *first_k, *first_v;  // [slots][first_rows][...]
  int ring, first_rows;
  const int32_t *slot, *pos, *back, *tile_first, *tile_count;
  int H, G, d, window, keep;
  float scale, lambda, out_scale, eps;
  int unit_rms;
  __nv_bfloat16* out;
  int64_t ld_out;
};
struct WinTcMaps {   // rows of the step's keys and values and of the rings, in boxes of 64 columns x 128 rows
  CUtensorMap step_k, step_v, ring_k, ring_v;
};

__device__ __forceinline__ uint32_t tc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_bar_init(uint64_t* b, uint32_t n) { asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(tc_smem(b)), "r"(n) : "memory"); }
__device__ __forceinline__ void tc_arrive(uint64_t* b) { asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc_smem(b)) : "memory"); }
__device__ __forceinline__ bool tc_try(uint64_t* b, uint32_t parity) {
  uint32_t ok;
  asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(tc_smem(b)), "r"(parity) : "memory");
  return ok != 0;
}
// bounded: false (and *dead set) after about two seconds or once another warp has given up.  Nobody leaves its loop then: the
// later waits return at once, so that everybody meets at the end.
__device__ __forceinline__ bool tc_wait(uint64_t* b, uint32_t parity, volatile int* dead) {
  if (tc_try(b, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 32; ++i)
      if (tc_try(b, parity)) return true;
    if (*dead != 0 || clock64() - t0 > 4000000000ll) {
      *dead = 1;
      return false;
    }
  }
}
__device__ __forceinline__ bool tc_elect() {
  uint32_t p;
  asm volatile("{\n\t.reg .b32 rx;\n\t.reg .pred px;\n\telect.sync rx|px, 0xffffffff;\n\tselp.u32 %0, 1, 0, px;\n\t}" : "=r"(p));
  return p != 0;
}
__device__ __forceinline__ void tc_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_commit(uint64_t* b) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(tc_smem(b)) : "memory");
}
__device__ __forceinline__ void tc_mma_ss(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d), "l"(a), "l"(b), "r"(idesc),
               "r"(acc)
               : "memory");
}
__device__ __forceinline__ void tc_mma_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a), "l"(b), "r"(idesc),
               "r"(acc)
               : "memory");
}
__device__ __forceinline__ void tc_ld32(uint32_t a, float* v) {
  uint32_t* d = reinterpret_cast<uint32_t*>(v);
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]),
        "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15]), "=r"(d[16]), "=r"(d[17]), "=r"(d[18]), "=r"(d[19]), "=r"(d[20]), "=r"(d[21]), "=r"(d[22]),
        "=r"(d[23]), "=r"(d[24]), "=r"(d[25]), "=r"(d[26]), "=r"(d[27]), "=r"(d[28]), "=r"(d[29]), "=r"(d[30]), "=r"(d[31])
      : "r"(a));
}
__device__ __forceinline__ void tc_ld16(uint32_t a, float* v) {
  uint32_t* d = reinterpret_cast<uint32_t*>(v);
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]),
                 "=r"(d[11]), "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15])
               : "r"(a));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_st16(uint32_t a, const uint32_t* d) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(a), "r"(d[0]), "r"(d[1]), "r"(d[2]),
               "r"(d[3]), "r"(d[4]), "r"(d[5]), "r"(d[6]), "r"(d[7]), "r"(d[8]), "r"(d[9]), "r"(d[10]), "r"(d[11]), "r"(d[12]), "r"(d[13]), "r"(d[14]), "r"(d[15])
               : "memory");
}
__device__ __forceinline__ void tc_pair_sync(int q) { asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory"); }  // the two warps of a lane quadrant
__device__ __forceinline__ float tc_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

template <int NM>
__global__ void __launch_bounds__(kTcThreads, 1) window_attention_tc_kernel(WinPromptArgs a, int dv, const __grid_constant__ WinTcMaps maps) {
  using T = __nv_bfloat16;
  extern __shared__ __align__(1024) unsigned char smem_tc[];
  uint64_t* kfull = reinterpret_cast<uint64_t*>(smem_tc);   // [2] keys of a tile are there
  uint64_t *kdone = kfull + 2, *vfull = kfull + 4, *vdone = kfull + 6, *sfull = kfull + 8, *pfull = kfull + 10, *odone = kfull + 12, *qfull = kfull + 13;
  uint32_t* tmem_s = reinterpret_cast<uint32_t*>(kfull + 14);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_s + 1);
  float* xmax = reinterpret_cast<float*>(smem_tc + 1024);   // [2 steps][2 halves][128 rows]
  float* xsum = xmax + 512;                                 // [2 halves][128 rows]
  const int d = a.d, G = a.G, KD = NM * d, kc = d / 8, kb = (d + 63) / 64, vb = (dv + 63) / 64;
  unsigned char* Ks = smem_tc + kTcHeader;                  // [2][kb][128][128 bytes]
  unsigned char* Vs = Ks + (size_t)2 * kb * 16384;          // [2][vb][128][128]
  unsigned char* Qs = Vs + (size_t)2 * vb * 16384;          // [NM][kc][128][16 bytes], no swizzle
  float* Os = reinterpret_cast<float*>(Qs + (size_t)NM * kc * 2048);  // [dv][128], two maps only
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // late tiles have the most keys: those of all heads start first
  const int turn = blockIdx.x / a.H, h = blockIdx.x - turn * a.H, g = h / (a.H / G);
  const int tile = gridDim.x / a.H - 1 - turn;
  const int first = a.tile_first[tile], count = min(a.tile_count[tile], kTcRows);
  const int pa = a.pos[first], back0 = a.back[first];
  const int p0 = pa - back0;                                // the first position the step brings of this sequence
  const int64_t seg_row0 = first - back0;
  const int lo = max(0, pa - a.window + 1);                 // the oldest key of the first row's window
  const int nf = min(a.keep, lo);                           // kept first positions that lie in front of it
  const int nk = nf + (pa + count - lo);                    // key index kk: the kept ones, then lo .. the last row's own position
  const int n_tiles = (nk + kTcKeys - 1) / kTcKeys, steps = NM * n_tiles;

  if (warp == 12) {
    if (lane < 2) {
      tc_bar_init(&kfull[lane], 4);
      tc_bar_init(&kdone[lane], 1);
      tc_bar_init(&vfull[lane], 4);
      tc_bar_init(&vdone[lane], 1);
      tc_bar_init(&sfull[lane], 1);
      tc_bar_init(&pfull[lane], 8);
    } else if (lane == 2) {
      tc_bar_init(odone, 1);
      tc_bar_init(qfull, 8);
      *dead = 0;
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(tmem_s)), "r"(512));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    tc_before();
  }
  __syncthreads();
  tc_after();
  const uint32_t tb = *reinterpret_cast<volatile uint32_t*>(tmem_s);
  // columns: S / p1, p2 [0, 128) and [128, 256); p3 [256, 320) and [320, 384); O [384, 384 + dv)
  const uint32_t col_o = tb + 384;

  if (warp == 12) {
    // ---- MMA issue ----
    const uint32_t idesc_s = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
    const uint32_t idesc_o = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | (((uint32_t)dv >> 3) << 17) | ((128u >> 4) << 24);  // B (values) MN-major
    const uint64_t kmaj = ((uint64_t)(2048u >> 4) << 16) | ((uint64_t)(128u >> 4) << 32) | (1ull << 46);   // chunks 2048 bytes apart, 8-row groups 128
    // swizzled rows of 128 bytes, 8-row groups 1024 bytes apart; MN-major: the next 64 columns 16384 bytes on
    const uint64_t swk = (1ull << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
    const uint64_t swmn = ((uint64_t)(16384u >> 4) << 16) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
    const uint32_t q0 = tc_smem(Qs) >> 4, k0 = tc_smem(Ks) >> 4, v0 = tc_smem(Vs) >> 4;
    auto scores = [&](int s) {
      const int b = s & 1, m = s / n_tiles;
      const bool ok = tc_wait(&kfull[b], (s >> 1) & 1, dead);
      tc_after();
      if (tc_elect()) {
        if (ok) {
          for (int ks = 0; ks < d / 16; ++ks)
            tc_mma_ss(tb + b * 128, kmaj | (q0 + (uint32_t)(m * kc + 2 * ks) * 128), swk | (k0 + (uint32_t)(b * kb + (ks >> 2)) * 1024 + (ks & 3) * 2), idesc_s, ks != 0);
        }
        tc_commit(&sfull[b]);
        tc_commit(&kdone[b]);
      }
      __syncwarp();
    };
    tc_wait(qfull, 0, dead);
    tc_after();
    scores(0);
    for (int s = 0; s < steps; ++s) {
      if (s + 1 < steps) scores(s + 1);
      const int b = s & 1;
      bool ok = tc_wait(&pfull[b], (s >> 1) & 1, dead);
      ok = tc_wait(&vfull[b], (s >> 1) & 1, dead) && ok;
      tc_after();
      if (tc_elect()) {
        if (ok) {
          const uint32_t fresh = s % n_tiles == 0 ? 0u : 1u;
#pragma unroll
          for (int part = 0; part < 3; ++part) {
            const uint32_t pa_ = part < 2 ? tb + b * 128 + part * 64 : tb + 256 + b * 64;
#pragma unroll
            for (int ks = 0; ks < 8; ++ks) tc_mma_ts(col_o, pa_ + 8 * ks, swmn | (v0 + (uint32_t)(b * vb) * 1024 + ks * 128), idesc_o, part || ks ? 1u : fresh);
          }
        }
        tc_commit(odone);
        tc_commit(&vdone[b]);
      }
      __syncwarp();
    }
    // the last arrival of the tensor core: nothing of this CTA may come after its shared memory has been given back
    tc_wait(&vdone[(steps - 1) & 1], ((steps - 1) >> 1) & 1, dead);
  } else if (warp >= 8) {
    // ---- loads ----
    const int64_t sl = a.slot[first];
    const T* ring_k = a.ring_k + (sl * a.ring * G + g) * KD;
    const T* ring_v = a.ring_v + (sl * a.ring * G + g) * dv;
    const T* first_k = a.first_k + (sl * a.first_rows * G + g) * KD;
    const T* first_v = a.first_v + (sl * a.first_rows * G + g) * dv;
    const T* step_k = a.kn + (seg_row0 * G + g) * KD;
    const T* step_v = a.vn + (seg_row0 * G + g) * dv;
    // copies of this lane: its row of every four, 16-byte chunk lane % 8 of every eight
    const int key0 = (warp - 8) * 32 + (lane >> 3), ch = lane & 7;
    auto load = [&](unsigned char* dst, uint64_t* full, int t, int cols, int64_t row, const T* step, const T* firsts, const T* ring, const CUtensorMap* step_map,
                    const CUtensorMap* ring_map, int col) {
      const int j0 = lo + (t * kTcKeys - nf), boxes = (cols + 63) / 64;   // first position of a tile without kept keys
      const bool in = t * kTcKeys >= nf && (t + 1) * kTcKeys <= nk;
      const bool by_step = in && j0 >= p0, by_ring = in && j0 >= a.first_rows && j0 + kTcKeys <= p0 && j0 % a.ring + kTcKeys <= a.ring;
      if (by_step || by_ring) {
        const CUtensorMap* map = by_step ? step_map : ring_map;
        const int y = by_step ? (int)(seg_row0 + (j0 - p0)) : (int)(sl * a.ring + j0 % a.ring);
        if (warp == 8 && tc_elect()) {
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(tc_smem(full)), "r"(boxes * 16384) : "memory");
          for (int k = 0; k < boxes; ++k)
            asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(tc_smem(dst + k * 16384)),
                         "l"(map), "r"(col + 64 * k), "r"(y), "r"(tc_smem(full))
                         : "memory");
        } else if (warp != 8 && lane == 0) {
          tc_arrive(full);
        }
        __syncwarp();
        return;
      }
#pragma unroll 1
      for (int kg = 0; kg < 8; ++kg) {
        const int key = key0 + 4 * kg, kk = t * kTcKeys + key;
        unsigned char* to = dst + key * 128 + ((ch ^ (key & 7)) * 16);
        if (kk < nk) {
          const int j = kk < nf ? kk : lo + (kk - nf);
          const T* src = (j >= p0 ? step + (int64_t)(j - p0) * row : (j < a.first_rows ? firsts + (int64_t)j * row : ring + (int64_t)(j % a.ring) * row)) + ch * 8;
          for (int c = ch * 8; c < cols; c += 64, to += 16384, src += 64) cp_async16(to, src);
        } else {   // weights of no key are zero, and so must be what they meet
          for (int c = ch * 8; c < cols; c += 64, to += 16384) *reinterpret_cast<uint4*>(to) = make_uint4(0, 0, 0, 0);
        }
      }
      cp_async_commit();
      cp_async_wait<0>();
      // visible to the tensor core (async proxy), then announced
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(full);
    };
    for (int s = 0; s < steps; ++s) {
      const int b = s & 1, m = s / n_tiles, t = s - m * n_tiles;
      if (s >= 2) tc_wait(&kdone[b], ((s >> 1) - 1) & 1, dead);
      load(Ks + (size_t)b * kb * 16384, &kfull[b], t, d, (int64_t)G * KD, step_k + m * d, first_k + m * d, ring_k + m * d, &maps.step_k, &maps.ring_k, g * KD + m * d);
      if (s >= 2) tc_wait(&vdone[b], ((s >> 1) - 1) & 1, dead);
      load(Vs + (size_t)b * vb * 16384, &vfull[b], t, dv, (int64_t)G * dv, step_v, first_v, ring_v, &maps.step_v, &maps.ring_v, g * dv);
    }
  } else {
    // ---- weights and epilogue: thread = (row, half of the columns) ----
    const int q = warp & 3, half = warp >> 2, row = q * 32 + lane;
    const uint32_t lane_col = (uint32_t)(32 * q) << 16;
    {
      // queries as bf16 operands (rows past the run are zero); a negative factor goes into their sign
      const float sign = a.scale < 0.f ? -1.f : 1.f;
#pragma unroll 4
      for (int c = half; c < NM * kc; c += 2) {
        uint4 o = make_uint4(0, 0, 0, 0);
        if (row < count) {
          const float4* src = reinterpret_cast<const float4*>(a.qn + ((int64_t)(first + row) * a.H + h) * KD + c * 8);
          const float4 x = src[0], y = src[1];
          o = make_uint4(pack_bf16(x.x * sign, x.y * sign), pack_bf16(x.z * sign, x.w * sign), pack_bf16(y.x * sign, y.y * sign), pack_bf16(y.z * sign, y.w * sign));
        }
        *reinterpret_cast<uint4*>(Qs + ((size_t)c * 128 + row) * 16) = o;
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) tc_arrive(qfull);
    }
    const float sl2 = fmaxf(fabsf(a.scale) * 1.44269504088896341f, 1e-30f);   // (never zero: -inf stays -inf)
    const int i = row < count ? pa + row : -1;   // the row's own position (-1: no row)
    const int w_lo = pa + 32 * q, w_hi = pa + min(count, 32 * q + 32) - 1;   // positions of this warp's rows
    const int blocks = dv / 16;
    float m_used = -INFINITY, l = 0.f;
    for (int s = 0; s < steps; ++s) {
      const int b = s & 1, mp = s / n_tiles, t = s - mp * n_tiles, kk0 = t * kTcKeys + half * 64;
      if (t == 0) m_used = -INFINITY, l = 0.f;
      tc_wait(&sfull[b], (s >> 1) & 1, dead);
      tc_after();
      float v[64];
      tc_ld32(tb + lane_col + b * 128 + half * 64, v);
      tc_ld32(tb + lane_col + b * 128 + half * 64 + 32, v + 32);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      // every key of this half is one of every row of this warp: contiguous, not in its future, inside the window
      const int j0 = lo + (kk0 - nf);
      const bool all = kk0 >= nf && kk0 + 64 <= nk && j0 + 63 <= w_lo && w_hi - j0 < a.window && count >= 32 * q + 32;
      if (!all) {
#pragma unroll
        for (int e = 0; e < 64; ++e) {
          const int kk = kk0 + e, j = kk < nf ? kk : j0 + e;
          if (!(kk < nk && j <= i && (i - j < a.window || j < a.keep))) v[e] = -INFINITY;
        }
      }
      float mx = fmaxf(v[0], v[1]);
#pragma unroll
      for (int e = 2; e < 64; e += 2) mx = fmaxf(mx, fmaxf(v[e], v[e + 1]));
      xmax[(b * 2 + half) * 128 + row] = mx;
      tc_before();
      tc_pair_sync(q);   // also: both halves have read S, which the parts overwrite
      tc_after();
      mx = fmaxf(mx, xmax[(b * 2 + (half ^ 1)) * 128 + row]);
      mx = mx == -INFINITY ? mx : mx * sl2;
      const bool grow = mx > m_used + 8.f || (m_used == -INFINITY && mx > m_used);
      float c = 1.f;
      if (grow) {
        c = m_used == -INFINITY ? 0.f : tc_exp2(m_used - mx);
        m_used = mx;
        l *= c;
      }
      if (t > 0 && __any_sync(0xffffffffu, grow)) {   // the same rows, hence the same answer in both halves' warps
        tc_wait(odone, (s - 1) & 1, dead);
        tc_after();
        for (int k = half; k < blocks; k += 2) {
          float o[16];
          tc_ld16(col_o + lane_col + k * 16, o);
#pragma unroll
          for (int e = 0; e < 16; ++e) o[e] *= c;
          tc_st16(col_o + lane_col + k * 16, reinterpret_cast<uint32_t*>(o));
        }
      }
      const float m = m_used == -INFINITY ? 0.f : m_used;
      // p = p1 + p2 + p3 exactly: the leading 8 bits, cut off twice.  In pieces of 32, so that the exponentials of one piece (8 clocks
      // a warp) run beside the splitting of another.
      const uint32_t to = lane_col + tb + b * 128 + half * 32, to3 = lane_col + tb + 256 + b * 64 + half * 32;
      float sum[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int e0 = 0; e0 < 64; e0 += 32) {
#pragma unroll
        for (int e = e0; e < e0 + 32; ++e) {
          v[e] = tc_exp2(fmaf(v[e], sl2, -m));
          sum[e & 3] += v[e];
        }
#pragma unroll
        for (int part = 0; part < 3; ++part) {
          uint32_t o[16];
#pragma unroll
          for (int k = 0; k < 16; ++k) {
            const uint32_t x = __float_as_uint(v[e0 + 2 * k]), y = __float_as_uint(v[e0 + 2 * k + 1]);
            o[k] = __byte_perm(x, y, 0x7632);
            if (part < 2) v[e0 + 2 * k] -= __uint_as_float(x & 0xFFFF0000u), v[e0 + 2 * k + 1] -= __uint_as_float(y & 0xFFFF0000u);
          }
          tc_st16((part < 2 ? to + part * 64 : to3) + e0 / 2, o);
        }
      }
      l += (sum[0] + sum[1]) + (sum[2] + sum[3]);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      tc_before();
      __syncwarp();
      if (lane == 0) tc_arrive(&pfull[b]);
      if (t < n_tiles - 1) continue;

      // ---- the map's result ----
      xsum[half * 128 + row] = l;
      tc_wait(odone, s & 1, dead);
      tc_after();
      tc_pair_sync(q);
      const float total = l + xsum[(half ^ 1) * 128 + row];
      const float norm = *dead ? NAN : (i >= 0 ? 1.f / total : 0.f);
      if (mp + 1 < NM) {   // the first map's result waits with the thread that made it
        for (int k = half; k < blocks; k += 2) {
          float o[16];
          tc_ld16(col_o + lane_col + k * 16, o);
#pragma unroll
          for (int e = 0; e < 16; ++e) Os[(k * 16 + e) * 128 + row] = o[e] * norm;
        }
        tc_before();
        tc_pair_sync(q);   // xsum is free again
        continue;
      }
      float k_out = a.out_scale;
      if (a.unit_rms) {
        float ss = 0.f;
        for (int k = half; k < blocks; k += 2) {
          float o[16];
          tc_ld16(col_o + lane_col + k * 16, o);
#pragma unroll
          for (int e = 0; e < 16; ++e) {
            float y = o[e] * norm;
            if (NM == 2) y = Os[(k * 16 + e) * 128 + row] - a.lambda * y;
            ss = fmaf(y, y, ss);
          }
        }
        tc_pair_sync(q);   // everybody has read xsum
        xsum[half * 128 + row] = ss;
        tc_pair_sync(q);
        k_out /= sqrtf((ss + xsum[(half ^ 1) * 128 + row]) / (float)dv + a.eps);
      }
      T* dst = a.out + (int64_t)(first + row) * a.ld_out + (int64_t)h * dv;
      const int align = a.ld_out % 8 == 0 && (reinterpret_cast<uintptr_t>(a.out) & 15) == 0 ? 8 : (a.ld_out % 2 == 0 ? 2 : 1);
      for (int k = half; k < blocks; k += 2) {
        float o[16];
        tc_ld16(col_o + lane_col + k * 16, o);
        uint32_t w[8];
#pragma unroll
        for (int e = 0; e < 16; ++e) {
          o[e] *= norm;
          if (NM == 2) o[e] = Os[(k * 16 + e) * 128 + row] - a.lambda * o[e];
        }
#pragma unroll
        for (int e = 0; e < 8; ++e) w[e] = pack_bf16(o[2 * e] * k_out, o[2 * e + 1] * k_out);
        if (i < 0) continue;
        T* to = dst + k * 16;
        if (align == 8) {
          reinterpret_cast<uint4*>(to)[0] = make_uint4(w[0], w[1], w[2], w[3]);
          reinterpret_cast<uint4*>(to)[1] = make_uint4(w[4], w[5], w[6], w[7]);
        } else if (align == 2) {
#pragma unroll
          for (int e = 0; e < 8; ++e) reinterpret_cast<uint32_t*>(to)[e] = w[e];
        } else {   // rows of odd length: every other row starts on an odd element
#pragma unroll
          for (int e = 0; e < 16; ++e) to[e] = __ushort_as_bfloat16((unsigned short)(w[e >> 1] >> (16 * (e & 1))));
        }
      }
    }
  }
  if (*dead) {
    for (int k = 0; k < 64; ++k) __nanosleep(100000);   // copies and MMAs that are still in flight
  }
  tc_before();
  __syncthreads();
  if (warp == 12) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(512));
  }
}

inline size_t win_tc_smem(int nm, int d, int dv) {
  return kTcHeader + (size_t)2 * ((d + 63) / 64 + (dv + 63) / 64) * 16384 + (size_t)nm * (d / 8) * 2048 + (nm == 2 ? (size_t)dv * 512 : 0);
}
// shapes of this kernel (bf16 storage): both tiles twice, the queries and, for two maps, a result have to fit shared memory
inline bool win_tc_ok(int nm, int d, int dv) { return d % 16 == 0 && dv % 16 == 0 && dv >= 16 && dv <= 128 && win_tc_smem(nm, d, dv) <= 226 * 1024; }

using TcEncode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline TcEncode tc_encode() {
  static TcEncode fn = []() -> TcEncode {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<TcEncode>(p);
  }();
  return fn;
}
// rows of `cols` bf16; how many there are is the caller's to know (the kernel only names rows that the arguments name)
inline bool tc_rows_map(CUtensorMap* map, const void* base, int64_t cols) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)1 << 31}, strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)kTcKeys}, steps[2] = {1, 1};
  return tc_encode()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides, box, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int NM>
int launch_win_tc(const WinPromptArgs& a, int dv, int n_tiles, cudaStream_t st) {
  auto kern = window_attention_tc_kernel<NM>;
  static bool set = false;   // per instantiation
  if (!set) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 226 * 1024) != cudaSuccess) return AO_B200_ERR_CUDA;
    set = true;
  }
  WinTcMaps maps;
  const int64_t kd = (int64_t)a.G * NM * a.d, vd = (int64_t)a.G * dv;
  if (tc_encode() == nullptr || !tc_rows_map(&maps.step_k, a.kn, kd) || !tc_rows_map(&maps.step_v, a.vn, vd) || !tc_rows_map(&maps.ring_k, a.ring_k, kd) ||
      !tc_rows_map(&maps.ring_v, a.ring_v, vd))
    return AO_B200_ERR_CUDA;
  if ((int64_t)n_tiles * a.H > 2147483647) return AO_B200_ERR_UNSUPPORTED;
  kern<<<(unsigned)n_tiles * (unsigned)a.H, kTcThreads, win_tc_smem(NM, a.d, dv), st>>>(a, dv, maps);
  return lm_launch_status();
}

}  // namespace lm
