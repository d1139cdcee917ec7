// Attention under a sliding window for prompt portions on tcgen05 / tensor memory: the computation of window_attention_prompt_kernel
// (lm_window_attention_mma.cu: the same bf16 queries and keys, the same masks, the fp32 weights as the same three bf16 parts that add up to
// them exactly, fp32 sums) for tiles of 128 consecutive rows of one sequence x one query head, 64 keys at a time.
//
//   S = Q K^T     128 x 64 fp32 in tensor memory
//   P             exp2(S - m) in fp32, cut into bf16 parts p1 + p2 + p3 (8 bits each, by truncation: exact) and stored to tensor memory
//                 as the A operand; p1 and p2 lie over S, which is in registers by then
//   O += P V      three products over the same values, 128 x dv fp32 in tensor memory
// m is a row's largest score when it last grew by more than 2^8; only then is O rescaled.  Weights stay below 2^8, and sum and product
// carry the same factor.
//
// The keys of a tile are shared out over the C CTAs of a cluster (their results meet in shared memory at the end, each CTA finishes 128 / C
// of the rows): late tiles have sixteen times the keys of early ones, and a short run has too few tiles to fill the chip.
//
// One step after the other: a product is waited for before anything that it read or wrote is touched again, so no hand-over depends on the
// order in which the tensor core retires its work, and nothing is in flight at the end.  What overlaps is two CTAs per SM (256 columns of
// tensor memory each): one makes weights while the other multiplies.  Queries, keys and values lie as [64 columns][rows][128 bytes, 16-byte
// pieces swizzled], which the tensor core reads K-major (queries, keys) or MN-major (values).  (Without swizzle the score product
// alone took 1340 clocks a step, twice what its operands need.)  Keys and values come by 16-byte cp.async, whole rows by neighbouring threads:
// the next keys while the weights meet the values, the next values during the next score product.
// Warps 0-7: loads, weights and results, two threads per row (lane quadrant = warp % 4, half of the columns = warp / 4); warp 8: products.
// Every wait is bounded; a CTA whose wait ran out goes on without waiting, so that all meet at the end, and marks its rows with NaN.
//
// Bound by the chain of a step (scores -> largest -> weights -> parts -> products): about 3600 clocks with two CTAs on the SM, of which the tensor core
// works 1170 for each (d = dv = 128); a CTA's start (queries, first keys) takes 6000 clocks more and its end (the peers' shares) 9000.  2048 rows x 16
// heads of 128 (four key heads): 8.5 steps a CTA, 60 us, tensor pipe active in 31 % of the clocks, against 308 us of window_attention_prompt_kernel; the same with
// all keys of a tile in one CTA 110 us (the last tiles alone took 95), with unswizzled operands 84 us.
// A warp's instructions follow one another at nearly five clocks each, so what counts is their number, about 740 per step at first: addresses once per map
// instead of once per load, the largest score three at a time, O to shared memory 32 columns at a time: 57.6 -> 55.8 us, 117 rows of two maps 20.5 -> 19.2,
// heads of 64 (keys in rows of 8 pieces, values drained 8 columns at a time) 2048 rows 50.7 -> 47.8, 200 rows of 8 heads 11.1 -> 10.3, of 96 55.3 -> 51.3.
// Launched while the kernel in front ends (nothing of memory is touched before the wait): in a series of calls 59.4 -> 56.7 us.  Letting the kernel behind
// start as early: 55.0, but 16 to 23 us calls up to 4 us more, as its CTAs take the places of the last ones of this.
// Taken back: four threads per row (16 warps for the weights: 70.0 us in place of 55.8); the next step's scores beside this one's weights (two score buffers,
// p3 in shared memory: 57.4 -> 56.6, small sizes up to 5 % more); an early and a late tile per cluster, in one wave (60.3).
#include "../f32x2.h"
#include "../per_device.h"
#include "lm_mma.cuh"
#include "lm_window_attention.cuh"

namespace lm {

namespace {

constexpr int kTcKeys = 64, kTcThreads = 288, kTcRowThreads = 256;
constexpr uint32_t kTcHeader = 4096;                  // barriers, row exchange
constexpr uint32_t kTcColumns = 256, kTcO = 128;      // columns 32 h ..: the scores of half h, then its p1 and p2, 16 each; 64 + 16 h ..: its p3; 128 ..: O
// Two CTAs per SM and no third one, which would wait for tensor memory, perhaps while its cluster waits for it
constexpr size_t kTcMinSmem = 80 * 1024;

__device__ __forceinline__ uint32_t tc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// bounded: false (and *dead set) after about two seconds
__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* dead) {
  const uint32_t at = tc_smem(bar);
  const long long t0 = clock64();
  for (;;) {
#pragma unroll 1
    for (int i = 0; i < 32; ++i) {
      uint32_t ok;
      asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(ok) : "r"(at), "r"(parity) : "memory");
      if (ok) return true;
    }
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
__device__ __forceinline__ void tc_arrive(int bar) { asm volatile("bar.arrive %0, %1;" ::"r"(bar), "n"(kTcThreads) : "memory"); }
__device__ __forceinline__ void tc_sync(int bar) { asm volatile("bar.sync %0, %1;" ::"r"(bar), "n"(kTcThreads) : "memory"); }
__device__ __forceinline__ void tc_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t tc_peer(uint32_t addr, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
__device__ __forceinline__ float tc_peer_f32(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr));
  return v;
}
__device__ __forceinline__ float4 tc_peer_f32x4(uint32_t addr) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
  return v;
}
__device__ __forceinline__ void tc_peer_set(uint32_t addr) { asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(1) : "memory"); }
__device__ __forceinline__ void tc_cp16(uint32_t smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem), "l"(gmem) : "memory");
}
// 32 lanes x 32 / 8 columns, thread = lane.  The load and its wait are one statement: nothing that uses the values can come between them.
__device__ __forceinline__ void tc_ld32(uint32_t a, uint32_t (&d)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,"
      "%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n\ttcgen05.wait::ld.sync.aligned;"
      : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7]), "=r"(d[8]), "=r"(d[9]), "=r"(d[10]), "=r"(d[11]),
        "=r"(d[12]), "=r"(d[13]), "=r"(d[14]), "=r"(d[15]), "=r"(d[16]), "=r"(d[17]), "=r"(d[18]), "=r"(d[19]), "=r"(d[20]), "=r"(d[21]), "=r"(d[22]),
        "=r"(d[23]), "=r"(d[24]), "=r"(d[25]), "=r"(d[26]), "=r"(d[27]), "=r"(d[28]), "=r"(d[29]), "=r"(d[30]), "=r"(d[31])
      : "r"(a)
      : "memory");
}
__device__ __forceinline__ void tc_ld8(uint32_t a, uint32_t (&d)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n\ttcgen05.wait::ld.sync.aligned;"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7])
               : "r"(a)
               : "memory");
}
__device__ __forceinline__ void tc_st8(uint32_t a, const uint32_t (&d)[8]) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(a), "r"(d[0]), "r"(d[1]), "r"(d[2]), "r"(d[3]), "r"(d[4]), "r"(d[5]),
               "r"(d[6]), "r"(d[7])
               : "memory");
}
__device__ __forceinline__ void tc_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
using ao::F2;
using ao::f2;
using ao::f2_add;
using ao::f2_fma;
using ao::f2_get;
__device__ __forceinline__ float tc_max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
__device__ __forceinline__ float tc_exp2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// descriptor of an operand in shared memory in rows of 128 swizzled bytes: 1024 bytes from 8 rows to the next 8; `lead` from 64 columns to the
// next 64 (MN-major only).  (In a cluster a CTA's own addresses carry its rank above bit 24; the descriptor wants the offset.)
__device__ __forceinline__ uint64_t tc_desc(uint32_t addr, uint32_t lead) {
  return ((uint64_t)((1024u >> 4) | (1u << 14) | (2u << 29)) << 32) | ((lead >> 4) << 16) | ((addr & 0x3FFFFu) >> 4);
}
// where 16-byte piece c of row r lies in a tile of `rows` rows
__device__ __forceinline__ uint32_t tc_at(int r, int c, int rows) { return (c >> 3) * (rows * 128) + r * 128 + (((c ^ r) & 7) << 4); }

// the row of key kk: the kept positions, then those from lo on, of which the step brings p0 and later ones (its rows from seg_row0 on)
__device__ __forceinline__ const __nv_bfloat16* win_row(const WinPromptArgs& a, int kk, int nf, int lo, int p0, int64_t seg_row0, int64_t slot, int g, int width,
                                                        const __nv_bfloat16* step, const __nv_bfloat16* kept, const __nv_bfloat16* ring) {
  const int j = kk < nf ? kk : lo + (kk - nf);
  return j >= p0 ? step + ((seg_row0 + (j - p0)) * a.G + g) * width
                 : (j < a.first_rows ? kept + ((slot * a.first_rows + j) * a.G + g) * width : ring + ((slot * a.ring + j % a.ring) * a.G + g) * width);
}
// two bf16, each zero where it is an infinity or NaN
__device__ __forceinline__ uint32_t finite_or_zero(uint32_t v) {
  if ((v & 0x7F80u) == 0x7F80u) v &= 0xFFFF0000u;
  if ((v & 0x7F800000u) == 0x7F800000u) v &= 0xFFFFu;
  return v;
}
// Values that are not finite, of a step in which some rows do not see all keys: a hidden key's weight is 0, and 0 times them is not.  So they are zero
// in the product (each thread looks at the pieces that it has loaded, which have landed) and are added afterwards to the rows that see their key.
// marks: [2][2], the step's keys that have such values; zero at first.  n: the how manieth such step this is.
__device__ __forceinline__ void hide_odd_values(unsigned char* values, int pieces, uint32_t* marks, int n) {
  const int wide = 32 - __clz(pieces - 1), c = threadIdx.x & ((1 << wide) - 1), rows = kTcRowThreads >> wide;
  if (threadIdx.x < 2) marks[2 * ((n + 1) & 1) + threadIdx.x] = 0u;   // (who reads these has done so before this step's scores)
  if (c >= pieces) return;
  const auto top = [](uint32_t v) { return (v & 0x7F807F80u) + 0x00800080u; };   // the upper bit of a half: its exponent is all ones
#pragma unroll 1
  for (int row = threadIdx.x >> wide; row < kTcKeys; row += rows) {
    uint4* at = reinterpret_cast<uint4*>(values + tc_at(row, c, kTcKeys));
    const uint4 v = *at;
    if (((top(v.x) | top(v.y) | top(v.z) | top(v.w)) & 0x80008000u) == 0u) continue;
    *at = make_uint4(finite_or_zero(v.x), finite_or_zero(v.y), finite_or_zero(v.z), finite_or_zero(v.w));
    atomicOr(&marks[2 * (n & 1) + (row >> 5)], 1u << (row & 31));
  }
}
// keys: those that hide_odd_values has marked; a row sees key kk where kk <= see_hi and (kk >= see_lo or kk < see_keep).  Whatever their weight, the
// sum is the infinity or NaN.  Columns [first_column, first_column + columns) of the row, at o_mine in tensor memory.  Out of line: the steps keep their registers.
__device__ __noinline__ void add_odd_values(const WinPromptArgs& a, uint64_t keys, int k0, int see_hi, int see_lo, int see_keep, int row, int lo, int nf, int g,
                                            uint32_t o_mine, int dv, int first_column, int columns) {
  const int back = a.back[row], p0 = a.pos[row] - back;
  const int64_t seg_row0 = row - back, slot = a.slot[row];
#pragma unroll 1
  for (int c = 0; c < columns; c += 8) {
    uint32_t o[8];
    tc_ld8(o_mine + c, o);
#pragma unroll 1
    for (uint64_t left = keys; left != 0; left &= left - 1) {
      const int kk = k0 + __ffsll((long long)left) - 1;
      if (kk > see_hi || (kk < see_lo && kk >= see_keep)) continue;
      const uint4 v = *reinterpret_cast<const uint4*>(win_row(a, kk, nf, lo, p0, seg_row0, slot, g, dv, a.vn, a.first_v, a.ring_v) + first_column + c);
      const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const float f = __uint_as_float(i & 1 ? w[i >> 1] & 0xFFFF0000u : w[i >> 1] << 16);
        if (!(fabsf(f) < INFINITY)) o[i] = __float_as_uint(__uint_as_float(o[i]) + f);
      }
    }
    __syncwarp();
    tc_st8(o_mine + c, o);
  }
  tc_st_wait();
}

// What a CTA's threads agree on, at the start of shared memory
struct TcShared {
  uint64_t s_ready, o_ready;   // a step's scores are in tensor memory; its values have been added
  uint32_t tmem;
  int dead;                    // a wait has run out
  uint32_t odd[4];             // CAREFUL: which of a step's 64 keys have a value that is not finite [2 steps][2]
  int again;                   // a result of the tile is not finite
};

// The tile, start to end.  CAREFUL (a second time): a value that is not finite has no part in rows that do not see its key.
template <int NM, int C, bool CAREFUL>
__device__ __forceinline__ void attend(const WinPromptArgs& a, int dv) {
  using T = __nv_bfloat16;
  extern __shared__ __align__(1024) unsigned char smem_tc[];
  TcShared& sh = *reinterpret_cast<TcShared*>(smem_tc);
  uint64_t *s_ready = &sh.s_ready, *o_ready = &sh.o_ready;
  volatile int* dead = &sh.dead;
  const uint32_t tb = *reinterpret_cast<volatile uint32_t*>(&sh.tmem);
  float* xch = reinterpret_cast<float*>(smem_tc + 1024);         // [2 halves][128 rows] largest score, at the end sum of weights
  float* row_m = reinterpret_cast<float*>(smem_tc + 2048);       // [128] what a row's weights are relative to, for the peers
  float* row_l = row_m + 128;                                    // [128] their sum
  const int d = a.d, G = a.G, KD = NM * d, kc = d / 8, vc = dv / 8, dvh = dv / 2, kb = (d + 63) / 64, vb = (dv + 63) / 64;
  unsigned char* Qs = smem_tc + kTcHeader;                       // [kb][128 rows][128 bytes], one map at a time
  unsigned char* Ks = Qs + kb * 16384;                           // [kb][64 keys][128 bytes]
  unsigned char* Vs = Ks + kb * 8192;                            // [vb][64 keys][128 bytes]
  const uint32_t pitch = dv * 4 + 16;
  unsigned char* Ob = smem_tc + kTcHeader;                       // [128 rows][pitch] O for the peers, where Q, K and V were
  float* Os = reinterpret_cast<float*>(Ob + max(kb * 24576 + vb * 8192, (int)(128 * pitch)));   // [128 / C rows][dv] first of two maps
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // late tiles have the most keys: those of all heads start first
  const int64_t turn = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) / C;
  const int rank = blockIdx.x % C;
  const int h = (int)(turn % a.H), tile = (int)(gridDim.x / C - 1 - turn / a.H), g = h / (a.H / G);
  const int first = a.tile_first[tile], count = min(a.tile_count[tile], kTcRows);
  const int pa = a.pos[first];
  const int lo = max(0, pa - a.window + 1);        // the oldest key of the first row's window
  const int nf = min(a.keep, lo);                  // kept first positions that lie in front of it
  const int nk = nf + (pa + count - lo);           // key index kk: the kept ones, then lo .. the last row's own position
  const int all = (nk + kTcKeys - 1) / kTcKeys, begin = (int)((int64_t)all * rank / C), steps = (int)((int64_t)all * (rank + 1) / C) - begin;   // this CTA's

  uint32_t parity = CAREFUL ? (uint32_t)(NM * steps) & 1u : 0u;   // of the step's barriers
  int hidings = 0;                                               // steps in which some rows did not see all keys
  bool ok = !CAREFUL || *dead == 0;                              // (a wait ran out before: nothing more is issued)

#pragma unroll 1
  for (int m = 0; m < NM; ++m) {
    if (warp == 8) {
      // ---- products ----
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (8u << 24);              // fp32 <- bf16 x bf16, 128 rows
      const uint32_t idesc_s = idesc | ((kTcKeys / 8u) << 17), idesc_o = idesc | (1u << 16) | ((uint32_t)vc << 17);   // values: MN-major
      const uint64_t q_desc = tc_desc(tc_smem(Qs), 0), k_desc = tc_desc(tc_smem(Ks), 0), v_desc = tc_desc(tc_smem(Vs), 8192);
#pragma unroll 1
      for (int t = 0; t < steps; ++t, parity ^= 1u) {
        tc_sync(1);                                        // keys (and, the first time, queries) are there; the parts before have been read
        tc_after();
        if (tc_elect() && ok) {
          for (int ks = 0; ks < kc / 2; ++ks)              // 16 columns each
            tc_mma_ss(tb, q_desc + (((ks >> 2) * 16384 + (ks & 3) * 32) >> 4), k_desc + (((ks >> 2) * 8192 + (ks & 3) * 32) >> 4), idesc_s, ks != 0);
          tc_commit(s_ready);
        }
        __syncwarp();
#pragma unroll 1
        for (int b = 0; b < 2; ++b) {                      // 16 keys of either half at a time: their parts (and the values) are there
          tc_sync(2 + b);
          tc_after();
          if (tc_elect() && ok) {
#pragma unroll
            for (int i = 0; i < 6; ++i) {
              const int part = i >> 1, half = i & 1;
              tc_mma_ts(tb + kTcO, part < 2 ? tb + half * 32 + part * 16 + b * 8 : tb + 64 + half * 16 + b * 8, v_desc + (2 * half + b) * (2048 >> 4), idesc_o,
                        t > 0 || b > 0 || i > 0);
            }
            if (b == 1) tc_commit(o_ready);
          }
          __syncwarp();
        }
        ok = ok && tc_wait(o_ready, parity, dead);
      }
    } else {
      // ---- loads, weights ----
      const int64_t seg_row0 = first - a.back[first], s = a.slot[first];
      const int p0 = pa - a.back[first];                   // the first position the step brings of this sequence
      // the threads of a row take its 16-byte pieces: 2, 4, 8 or 16 threads, as many as there are pieces, or the next power of two.  `src`: this thread's piece of
      // the first key's row (key index 0), were it among the step's own rows
      struct Pieces {
        int c, row0, rows;
        const T* src;
      };
      auto pieces_of = [&](int pieces, int width, int off, const T* step) {
        const int wide = 32 - __clz(pieces - 1), c = threadIdx.x & ((1 << wide) - 1), row0 = threadIdx.x >> wide;
        return Pieces{c < pieces ? c : -1, row0, kTcRowThreads >> wide, step + ((seg_row0 + (lo - nf - p0) + row0) * G + g) * width + off + c * 8};
      };
      auto load = [&](unsigned char* tile_at, int t, const Pieces& p, int width, int off, const T* step, const T* kept, const T* ring) {
        if (p.c < 0) return;
        const int k0 = (begin + t) * kTcKeys, j0 = lo + (k0 - nf);
        const uint32_t dst = tc_smem(tile_at) + tc_at(p.row0, p.c, kTcKeys);   // (rows a multiple of 8 apart: the same swizzle)
        if (k0 >= nf && j0 >= p0 && k0 + kTcKeys <= nk) {  // all from the step's own rows
          const T* src = p.src + (int64_t)k0 * (G * width);
          if (p.rows == 16) {
#pragma unroll
            for (int i = 0; i < 4; ++i) tc_cp16(dst + i * (16 * 128), src + (int64_t)i * 16 * (G * width));
          } else {
#pragma unroll 1
            for (int row = p.row0; row < kTcKeys; row += p.rows) tc_cp16(dst + (row - p.row0) * 128, src + (int64_t)(row - p.row0) * (G * width));
          }
          return;
        }
#pragma unroll 1
        for (int row = p.row0; row < kTcKeys; row += p.rows) {
          const int kk = k0 + row;
          const uint32_t at = tc_at(row, p.c, kTcKeys);
          if (kk < nk) {
            tc_cp16(tc_smem(tile_at) + at, win_row(a, kk, nf, lo, p0, seg_row0, s, g, width, step, kept, ring) + off + p.c * 8);
          } else {                                         // behind the last key: zero
            *reinterpret_cast<uint4*>(tile_at + at) = make_uint4(0, 0, 0, 0);
          }
        }
      };
      const Pieces kp = pieces_of(kc, KD, m * d, a.kn), vp = pieces_of(vc, dv, 0, a.vn);
      auto load_k = [&](int t) { load(Ks, t, kp, KD, m * d, a.kn, a.first_k, a.ring_k); };
      auto load_v = [&](int t) { load(Vs, t, vp, dv, 0, a.vn, a.first_v, a.ring_v); };
      // this thread's row of the tile and which keys it sees: kk <= see_hi and (kk >= see_lo or kk < see_keep)
      const int q = warp & 3, half = warp >> 2, r = q * 32 + lane;
      const uint32_t lanes = tb + ((uint32_t)(32 * q) << 16), mine = lanes + half * 32, o_mine = lanes + kTcO + half * dvh;
      float m_ref = -INFINITY, l = 0.f;
      if (steps > 0) {
        load_k(0);
        cp_async_commit();
        // the map's queries as bf16 (rows past the run are zero)
        const float* mine_q = a.qn + (((int64_t)(first + kp.row0) * a.H + h) * NM + m) * d + kp.c * 8;
        const int64_t next_q = (int64_t)kp.rows * a.H * NM * d;
        if (kp.c >= 0) {
#pragma unroll 4
          for (int row = kp.row0; row < kTcRows; row += kp.rows, mine_q += next_q) {
            float4 x = make_float4(0.f, 0.f, 0.f, 0.f), y = x;
            if (row < count) x = __ldg(reinterpret_cast<const float4*>(mine_q)), y = __ldg(reinterpret_cast<const float4*>(mine_q + 4));
            if (a.scale < 0.f) x = make_float4(-x.x, -x.y, -x.z, -x.w), y = make_float4(-y.x, -y.y, -y.z, -y.w);
            *reinterpret_cast<uint4*>(Qs + tc_at(row, kp.c, kTcRows)) = make_uint4(pack_bf16(x.x, x.y), pack_bf16(x.z, x.w), pack_bf16(y.x, y.y), pack_bf16(y.z, y.w));
          }
        }
        cp_async_wait<0>();
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        tc_before();
        tc_arrive(1);
        load_v(0);
        cp_async_commit();
      }
      const float to_log2 = fmaxf(fabsf(a.scale) * 1.4426950408889634f, 1e-37f);   // (the sign is the queries'; a hidden key stays -inf)
#pragma unroll 1
      for (int t = 0; t < steps; ++t, parity ^= 1u) {
        const int k0 = (begin + t) * kTcKeys;
        const bool plain = k0 + kTcKeys <= nk && (k0 + kTcKeys - 1 < nf || lo + (k0 + kTcKeys - 1 - nf) <= pa) &&
                           pa + count - 1 - (lo + max(k0 - nf, 0)) < a.window;   // every row sees every key of the step
        ok = ok && tc_wait(s_ready, parity, dead);
        tc_after();
        uint32_t x[32];
        tc_ld32(mine, x);
        // the row's largest score, in units of log2
        float top = -INFINITY;
        {
          const int base = k0 + half * 32;
          if (!plain) {
            const int hi = (r < count ? nf + (pa + r - lo) : -1) - base, low = nf + max(pa + r - a.window + 1 - lo, 0) - base;
            const int kept = nf + max(a.keep - lo, 0) - base;
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (!(i <= hi && (i >= low || i < kept))) x[i] = 0xFF800000u;
          }
#pragma unroll
          for (int i = 0; i < 32; i += 2) top = tc_max3(top, __uint_as_float(x[i]), __uint_as_float(x[i + 1]));
          top *= to_log2;
        }
        // (the two warps of a lane quadrant; the other's value of the step before has been read: both have passed o_ready since)
        xch[half * kTcRows + r] = top;
        asm volatile("bar.sync %0, 64;" ::"r"(4 + q) : "memory");
        top = fmaxf(top, xch[(half ^ 1) * kTcRows + r]);
        const bool grows = top > m_ref + 8.f;
        if (__any_sync(0xffffffffu, grows)) {
          const float f = grows ? tc_exp2(m_ref - top) : 1.f;
          m_ref = grows ? top : m_ref;
          l *= f;
          if (t > 0) {
            for (int c = 0; c < dvh; c += 8) {
              uint32_t o[8];
              tc_ld8(o_mine + c, o);
#pragma unroll
              for (int i = 0; i < 8; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
              tc_st8(o_mine + c, o);
            }
          }
        }
        const float m_use = m_ref == -INFINITY ? 0.f : m_ref;   // (a row that has seen no key yet)
        const F2 c2 = f2(to_log2, to_log2), nm2 = f2(-m_use, -m_use), minus = f2(-1.f, -1.f);
        F2 l2 = f2(0.f, 0.f);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
          uint32_t p[3][8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const float2 t = f2_get(f2_fma(f2(__uint_as_float(x[16 * b + 2 * i]), __uint_as_float(x[16 * b + 2 * i + 1])), c2, nm2));
            float2 w = make_float2(tc_exp2(t.x), tc_exp2(t.y));
            l2 = f2_add(l2, f2(w.x, w.y));
#pragma unroll
            for (int part = 0; part < 3; ++part) {
              const uint32_t u0 = __float_as_uint(w.x), u1 = __float_as_uint(w.y);
              p[part][i] = __byte_perm(u0, u1, 0x7632);    // the upper halves, side by side
              w = f2_get(f2_fma(f2(__uint_as_float(u0 & 0xFFFF0000u), __uint_as_float(u1 & 0xFFFF0000u)), minus, f2(w.x, w.y)));   // exact
            }
          }
          tc_st8(mine + b * 8, p[0]);
          tc_st8(mine + 16 + b * 8, p[1]);
          tc_st8(lanes + 64 + half * 16 + b * 8, p[2]);
          tc_st_wait();
          if (b == 0) {
            cp_async_wait<0>();                            // the step's values
            if (CAREFUL && !plain) hide_odd_values(Vs, vc, sh.odd, hidings);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          }
          tc_before();
          tc_arrive(2 + b);
        }
        const float2 ls = f2_get(l2);
        l += ls.x + ls.y;
        const bool more = t + 1 < steps;
        if (more) load_k(t + 1);                           // the product that read this step's keys is over
        cp_async_commit();
        ok = ok && tc_wait(o_ready, parity, dead);
        tc_after();
        if (CAREFUL && !plain) {   // (the marks are older than the products that o_ready stands for)
          const volatile uint32_t* mark = sh.odd + 2 * (hidings++ & 1);
          const uint64_t keys = mark[0] | ((uint64_t)mark[1] << 32);
          if (keys != 0) {
            add_odd_values(a, keys, k0, r < count ? nf + (pa + r - lo) : -1, nf + max(pa + r - a.window + 1 - lo, 0), nf + max(a.keep - lo, 0), first, lo, nf,
                           g, o_mine, dv, half * dvh, dvh);
            tc_before();
          }
        }
        if (more) {
          cp_async_wait<0>();
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          tc_before();
          tc_arrive(1);
          load_v(t + 1);
          cp_async_commit();
        }
      }
      // ---- this CTA's share to where the cluster reads it ----
      xch[half * kTcRows + r] = l;
      asm volatile("bar.sync 8, 256;" ::: "memory");       // (also: every warp is past the last product, which read Q, K and V)
      if (half == 0) {
        row_m[r] = m_ref;
        row_l[r] = l + xch[kTcRows + r];
      }
      float* dst = reinterpret_cast<float*>(Ob + r * pitch) + half * dvh;
      if (dvh == 64) {
#pragma unroll 1
        for (int c = 0; c < 64; c += 32) {
          uint32_t o[32];
          tc_ld32(o_mine + c, o);
#pragma unroll
          for (int i = 0; i < 32; i += 4)
            *reinterpret_cast<uint4*>(dst + c + i) = steps == 0 ? make_uint4(0u, 0u, 0u, 0u) : make_uint4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        }
      } else {
        for (int c = 0; c < dvh; c += 8) {
          uint32_t o[8];
          tc_ld8(o_mine + c, o);
          if (steps == 0) {
#pragma unroll
            for (int i = 0; i < 8; ++i) o[i] = 0u;
          }
          *reinterpret_cast<uint4*>(dst + c) = make_uint4(o[0], o[1], o[2], o[3]);
          *reinterpret_cast<uint4*>(dst + c + 4) = make_uint4(o[4], o[5], o[6], o[7]);
        }
      }
      tc_before();
    }
    tc_cluster_sync();
    // ---- rows rank * 128 / C ..: 2 C threads per row, four columns at a time ----
    if (warp < 8) {
      constexpr int per = 2 * C;
      const int rr = threadIdx.x / per, part = threadIdx.x % per, row = rank * (kTcRows / C) + rr;
      float top = -INFINITY, sum = 0.f;
      const uint32_t m_at = tc_smem(row_m + row), l_at = tc_smem(row_l + row), o_at = tc_smem(Ob) + row * pitch;
      float f[C], ls[C];                                   // what each share counts, and its sum of weights
#pragma unroll
      for (int c = 0; c < C; ++c) f[c] = tc_peer_f32(tc_peer(m_at, c)), ls[c] = tc_peer_f32(tc_peer(l_at, c));
#pragma unroll
      for (int c = 0; c < C; ++c) top = fmaxf(top, f[c]);
#pragma unroll
      for (int c = 0; c < C; ++c) {
        f[c] = top == -INFINITY ? 1.f : tc_exp2(f[c] - top);
        sum += f[c] * ls[c];
      }
      const float k = 1.f / sum;
      // U pieces of four columns at a time, all shares of them in flight: use(piece, the row's four results)
      constexpr int U = C >= 4 || NM == 2 ? 1 : 4 / C;   // (two maps, two pieces: 300 bytes of registers spilled, 2048 rows of 16 heads 133 us and not 111)
      auto results = [&](auto&& use) {
        for (int c0 = part; c0 < dv / 4; c0 += U * per) {
          float4 v[U][C];
#pragma unroll
          for (int u = 0; u < U; ++u)
#pragma unroll
            for (int c = 0; c < C; ++c)
              if (c0 + u * per < dv / 4) v[u][c] = tc_peer_f32x4(tc_peer(o_at + (c0 + u * per) * 16, c));
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const int c4 = c0 + u * per;
            if (c4 >= dv / 4) continue;
            float4 y = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int c = 0; c < C; ++c)
              y.x = fmaf(f[c], v[u][c].x, y.x), y.y = fmaf(f[c], v[u][c].y, y.y), y.z = fmaf(f[c], v[u][c].z, y.z), y.w = fmaf(f[c], v[u][c].w, y.w);
            y.x *= k, y.y *= k, y.z *= k, y.w *= k;
            if (NM == 2 && m == 1) {
              const float4 one = *reinterpret_cast<const float4*>(Os + (size_t)rr * dv + c4 * 4);
              y.x = one.x - a.lambda * y.x, y.y = one.y - a.lambda * y.y, y.z = one.z - a.lambda * y.z, y.w = one.w - a.lambda * y.w;
            }
            use(c4, y);
          }
        }
      };
      if (m + 1 < NM) {   // the first map's result waits with the thread that made it
        results([&](int c4, const float4& y) { *reinterpret_cast<float4*>(Os + (size_t)rr * dv + c4 * 4) = y; });
      } else {
        float mul = a.out_scale;
        if (a.unit_rms) {
          float ss = 0.f;
          results([&](int, const float4& y) { ss = fmaf(y.x, y.x, fmaf(y.y, y.y, fmaf(y.z, y.z, fmaf(y.w, y.w, ss)))); });
#pragma unroll
          for (int o = per / 2; o; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
          mul /= sqrtf(ss / (float)dv + a.eps);
        }
        T* dst = a.out + (int64_t)(first + row) * a.ld_out + (int64_t)h * dv;
        const bool wide = a.ld_out % 4 == 0 && reinterpret_cast<uintptr_t>(a.out) % 8 == 0, pairs = a.ld_out % 2 == 0;
        if (row < count) {
          bool finite = true;
          results([&](int c4, const float4& y) {
            if (!CAREFUL) finite = finite && fabsf(y.x * mul) < INFINITY && fabsf(y.y * mul) < INFINITY && fabsf(y.z * mul) < INFINITY && fabsf(y.w * mul) < INFINITY;
            const uint2 w = make_uint2(pack_bf16(y.x * mul, y.y * mul), pack_bf16(y.z * mul, y.w * mul));
            if (wide) {
              *reinterpret_cast<uint2*>(dst + c4 * 4) = w;
            } else if (pairs) {
              *reinterpret_cast<uint32_t*>(dst + c4 * 4) = w.x, *reinterpret_cast<uint32_t*>(dst + c4 * 4 + 2) = w.y;
            } else {   // rows of odd length: every other row starts on an odd element
              const uint32_t u[2] = {w.x, w.y};
#pragma unroll
              for (int i = 0; i < 4; ++i) dst[c4 * 4 + i] = __ushort_as_bfloat16((unsigned short)(u[i >> 1] >> (16 * (i & 1))));
            }
          });
          if (!finite) {
#pragma unroll
            for (int c = 0; c < C; ++c) tc_peer_set(tc_peer(tc_smem(&sh.again), c));
          }
        }
      }
    }
    tc_cluster_sync();   // the peers have read what lies here
  }
}

template <int NM, int C>
__device__ __noinline__ void attend_carefully(const WinPromptArgs& a, int dv) {
  attend<NM, C, true>(a, dv);
}

template <int NM, int C>
__global__ void __launch_bounds__(kTcThreads, 2) window_attention_tc_kernel(const __grid_constant__ WinPromptArgs a, int dv) {
  extern __shared__ __align__(1024) unsigned char smem_tc[];
  TcShared& sh = *reinterpret_cast<TcShared*>(smem_tc);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == 8) {
    if (lane == 0) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&sh.s_ready)) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(tc_smem(&sh.o_ready)) : "memory");
      sh.dead = sh.again = 0;
      sh.odd[0] = sh.odd[1] = sh.odd[2] = sh.odd[3] = 0u;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh.tmem)), "r"(kTcColumns));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    tc_before();
  }
  pdl_wait();
  __syncthreads();
  tc_after();
  attend<NM, C, false>(a, dv);
  // A hidden key's weight is 0, and 0 times a value that is not finite is not: where a result is not finite (on any CTA of the cluster, which has
  // told the others) the tile is done once more with an eye to that.  (Looking at the values of every step that hides keys: 2048 rows 62 us, not 60.)
  if (*reinterpret_cast<volatile int*>(&sh.again) != 0) attend_carefully<NM, C>(a, dv);
  if (*reinterpret_cast<volatile int*>(&sh.dead) != 0) {   // a wait ran out: all rows of the tile are marked, after the peers' results, and what is in
    const int64_t turn = ((int64_t)blockIdx.y * gridDim.x + blockIdx.x) / C;   // flight gets the time to land
    const int h = (int)(turn % a.H), tile = (int)(gridDim.x / C - 1 - turn / a.H);
    const int first = a.tile_first[tile];
    if (threadIdx.x < min(a.tile_count[tile], kTcRows))
      for (int c = 0; c < dv; ++c) a.out[(int64_t)(first + threadIdx.x) * a.ld_out + (int64_t)h * dv + c] = __ushort_as_bfloat16((unsigned short)0x7FFF);
    for (int i = 0; i < 64; ++i) __nanosleep(100000);
  }
  tc_before();
  __syncthreads();
  if (warp == 8) {
    tc_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(*reinterpret_cast<volatile uint32_t*>(&sh.tmem)), "r"(kTcColumns));
  }
}

template <int NM, int C>
int launch(const WinPromptArgs& a, int dv, int n_tiles, cudaStream_t st) {
  const size_t held = (size_t)((a.d + 63) / 64) * 24576 + (size_t)((dv + 63) / 64) * 8192, shares = (size_t)128 * (dv * 4 + 16);
  size_t smem = kTcHeader + (held > shares ? held : shares) + (NM == 2 ? (size_t)(kTcRows / C) * dv * 4 : 0);
  if (smem < kTcMinSmem) smem = kTcMinSmem;
  auto kern = window_attention_tc_kernel<NM, C>;
  static ao::OncePerDevice once;   // per instantiation
  if (!ao::dynamic_smem(once, kern, 113 * 1024)) return AO_B200_ERR_CUDA;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(n_tiles * C), (unsigned)a.H);
  cfg.blockDim = dim3(kTcThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  if (cudaLaunchKernelEx(&cfg, kern, a, dv) == cudaSuccess) return AO_B200_OK;
  return lm_launch_status();
}

// CTAs per tile.  Two from the 148 SMs' worth of CTAs on up to four times what the chip holds at once (2 x 148): beyond that whole tiles
// balance by themselves, and a share costs its 9000 clocks.  Fewer tiles: as many shares as fill the chip.  Two maps always share, as the
// first map's result of a whole tile would leave room for one CTA per SM only.
template <int NM>
int launch(const WinPromptArgs& a, int dv, int n_tiles, cudaStream_t st) {
  const int64_t tiles = (int64_t)n_tiles * a.H;
  if (tiles <= 37) return launch<NM, 8>(a, dv, n_tiles, st);
  if (tiles <= 74) return launch<NM, 4>(a, dv, n_tiles, st);
  if (tiles <= 592 || NM == 2) return launch<NM, 2>(a, dv, n_tiles, st);
  return launch<1, 1>(a, dv, n_tiles, st);
}

}  // namespace

int launch_win_tc(const WinPromptArgs& a, int n_maps, int dv, int n_tiles, cudaStream_t st) {
  return n_maps == 2 ? launch<2>(a, dv, n_tiles, st) : launch<1>(a, dv, n_tiles, st);
}

}  // namespace lm
