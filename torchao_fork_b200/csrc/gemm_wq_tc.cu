// Weight-only quantized linear for more than a few rows, int4 and int8: fused dequant + GEMM on tcgen05 / tensor memory.
//
//   y[m][n] = sum_k x[m][k] * W'[n][k]
//   int4   W' = bf16_rn((q - 8) * scale + zero): the arithmetic of the reference's tinygemm op (aten._weight_int4pack_mm, behind
//          torchao/dtypes/uintx/tensor_core_tiled_layout.py:_linear_bf16_act_uint4_weight_impl), one rounding per weight;
//   int4, few rows (DEFER)   W' unrounded: the affine is applied in fp32 to the sums over 128 k (or a group, if that is
//          smaller): y += s D + (z - 136 s) X with D = sum x (128 + q), X = sum x; results that are not finite (x with
//          infinities, NaN or values above 2^100, where D and X overflow) are added up weight by weight with W' as above;
//   int8   W' = q, the row scale applied to the bf16-rounded sum (torchao/dtypes/uintx/plain_layout.py:250-266).
//
// The tensor-core mapping is transposed so that the dequantized weights never touch shared memory:
//   MMA M (128 TMEM lanes)  = 128 weight rows (8 strips of the strip-major packed layout)
//   MMA N (16 .. 256)       = NT activation rows
//   A operand               = W' in TENSOR MEMORY, written by the dequant warps with tcgen05.st.16x128b: the 16-byte lane chunk
//                             of the packed layout holds rows g / g + 8 of a strip, which is that store's (lane, column) pattern
//   B operand               = activations in shared memory (no-swizzle K-major core matrices), one bulk copy per 128 k out of
//                             a copy of x that stage_x_kernel has put into that order (the k order inside a 32-k block is the
//                             store's: column 4 i + c holds k = 8 c + 2 i, 2 i + 1, so neither side shuffles); or, DIRECT, straight
//                             out of x by TMA (rows of 128 swizzled bytes, k in its own order), and the dequant warps turn the
//                             weights round to match (wq_turn_int4, wq_turn_int8), which takes no staging but 12 instructions a word
//   D                       = fp32 in tensor memory
//
// PAIR: two CTAs of a cluster work on 256 weight rows x NT activation rows with cta_group::2 MMAs: each dequantizes its own
// 128 rows and holds half of the activation tile, so the shared-memory and L2 traffic of the activations is halved.  (One CTA
// at NT = 256 would need 64 B/clk of shared-memory writes and as much in reads for B alone, of 128 B/clk.)
//
// Work split: units of (row block, row tile of x, 128 k; up to 128 rows 256 k), tile-major, dealt out contiguously and evenly to as many CTAs (or
// pairs) as there are SMs (small weights: tile by tile, wq_owners).  A tile whose K is shared between neighbours is summed by the one that arrives last, in CTA order
// (fp32 partial sums and tickets in the workspace; nobody waits for another CTA), so there is no last wave that is nearly
// empty and few row blocks still fill the chip.
//
// Roles (768 threads): warps 0-3 epilogue (warp = TMEM lane quadrant), 4-19 dequant (one strip each; two sets take
// alternate units), 20 weight producer (two TMA tensor copies per unit: 8 strips of weights, 8 strips of parameters),
// 21 activation producer, 22 and 23 MMA issue: the waits, the issue and the commit of a unit take one warp 600 clocks, so up to
// NT = 64 two warps take alternate units, each with accumulators of its own that the epilogue adds.  At the end all warps
// add up the tiles that this CTA was the last to reach.  Every wait is bounded: a CTA that gives up fills the rows of all its tiles with NaN
// (a shared tile then misses a ticket, so nobody else writes it) and returns once its copies and products in flight are over.
//
// Bound by the tensor cores from about 512 rows (8 MMAs of N = 256 take 1024 clocks per unit and pair, the dequant of a unit
// about 900 clocks per set of warps, two sets in flight), below that by the dequant -> MMA chain of a unit: conversions (all 16 warps at them at the
// same time, 440 clocks per 128 k and set) and, once per unit, the way over six barriers, about 700 clocks of each role.  Hence units of 256 k up to
// 128 rows: int4 28672 x 8192, 16 / 32 / 64 rows 46.9 / 47.7 / 49.5 -> 37.4 / 38.0 / 41.1 us, 14336 x 4096, 77 rows 26.1 -> 23.8, int8 28672 x 8192 and
// 14336 x 4096, 16 rows 49.5 -> 46.5, 23.3 -> 20.2; from 144 rows on they give nothing (int4 28672 x 8192, 200 rows 75.2 and 75.3; int8 14336 x 4096, 300 rows 40.2 and 42.5).  Measured,
// 14336 x 4096, int4 with groups of 128, M = 64 / 256 / 512 / 1000 / 2048: 22 / 37.6 / 54.2 / 94 / 174 us, the last 0.85 of 1634 TFLOP/s (one CTA
// per 128 x 256 tile with the whole K, activations multicast over 4 CTAs, run-time divisions and parameters read from global memory in
// the dequant loop: 29.9 / 36.5 / 67.0 / 128 / 225 us); int8 8192 x 8192, M = 32 / 512 / 2048: 24 / 63 / 227 us (44 / 66 / 244 us).
#include <cuda.h>
#include <cuda_bf16.h>

#include <cstdlib>
#include <mutex>

#include "common.cuh"
#include "f32x2.h"
#include "per_device.h"

namespace ao {

constexpr int kWqEpiWarps = 4, kWqDqWarps = 16;
constexpr int kWqBehind = 8;  // units (wq_gemm_kernel, t_early; 0, 4 and 16 measure the same, without the path 300 rows of 14336 x 4096 take 41.3 us, not 37.4)
constexpr int kWqBehindLong = 2;  // of 256 k: int4 28672 x 1280, 128 rows 22.9 us with 4 and 8, 19.9 with 2 and 1; 28672 x 2048, 64 rows 23.0 with 8, 20.2 with 4 and less
constexpr int kWqWProd = kWqEpiWarps + kWqDqWarps, kWqXProd = kWqWProd + 1, kWqMma = kWqXProd + 1;
constexpr int kWqThreads = (kWqMma + 2) * 32;  // 768
constexpr int kWqSlots = 4;                    // ring of A in tensor memory: 64 columns (128 k) each, or half as many of 256 k
constexpr int kWqMaxW = 16, kWqMaxX = 8;       // rings of weights and of tiles of x
constexpr int kWqPitch = 128 * 2 + 16;         // bytes of a row of the output tile in shared memory (rows land on distinct banks)
constexpr int kWqHeader = 1024;                // mbarriers, TMEM base, give-up flag
constexpr int kWqDirectRows = 512, kWqDirectN = 8192;  // from and up to which, at most, the GEMM reads the activations where they are (wq_plan)
constexpr int kWqLongNT = 128;                 // rows of a tile up to which a unit has 256 k (both sides: above)
constexpr int kWqMaxSplitTiles = 16;           // tiles per worker from which whole tiles are dealt out (imbalance <= 1/16)

struct WqParams {
  CUtensorMap wmap;          // weights: rows = strips, row = the strip's bytes; box = 8 strips x 128 k
  CUtensorMap smap;          // int4 scale / zero: rows = strips, row = 16 words per group; box = 8 strips x the unit's groups
  CUtensorMap xmap;          // DIRECT, activations: box = BR rows x 64 k, 128 bytes per row, 16-byte pieces swizzled; zeros past M and Kx
  const uint8_t* xt;         // staged activations [MT * ranks][KU][x_bytes]
  const uint32_t *packed, *sz;  // DEFER: what the maps show, for sums that are done again
  const __nv_bfloat16* scale8;
  __nv_bfloat16* y;
  const __nv_bfloat16* residual;  // y = bf16(residual + bf16(sum)); may be y itself
  float* part;               // shares of split tiles [workers][2][ranks][NT * 128]
  uint32_t* tickets;         // [tiles][ranks], zeroed by the staging kernel
  int64_t N_out, ldy, ld_res;
  int M, Kp, NT, BR, KU, MT, w_slots, x_slots, a_slots, n_mma, vec_store;
  uint32_t off_x, off_w;     // activation ring, weight ring
  long long wait_limit;      // clocks after which a wait gives up
  uint32_t x_bytes, x_sub;   // one unit of staged activations (and, DEFER, its sums), 128 k of it
  int quantum, base, rem;    // worker c owns units [first(c), first(c + 1)), first(c) = (c base + min(c, rem)) quantum
};

__host__ __device__ __forceinline__ int wq_first(int c, int base, int rem, int quantum) { return (c * base + (c < rem ? c : rem)) * quantum; }
__device__ __forceinline__ int wq_owner(int u, int base, int rem, int quantum) {
  const int v = u / quantum, big = rem * (base + 1);
  return v < big ? v / (base + 1) : rem + (v - big) / base;
}

// ---- staging: x -> bf16 units in the B operand's order ---------------------------------------------------------------
// piece (block b of BR rows, 128 k number ku; one or two make a unit): [16 chunks of 8 k][BR rows][8] and, SEG > 0, behind it fp32 sums [128 / SEG][16].
// Chunk 4 q + i holds of the 32-k quarter q the k = 8 c + 2 i + e at place 2 c + e.  A thread moves 32 k of one row: 64 bytes in,
// four 16-byte pieces out; a warp covers 8 rows x 128 k, so that every piece of 8 rows is one full 128-byte line.
// Rows >= M and columns >= Kx are zero.  Bound by HBM / L2: bytes of x in and out once; for few rows by the way there and back, which the GEMM's first
// weights are in if they ask first.  So the first piece is brought to L2 before the wait (which reads nothing: what the kernel in front writes meets it
// there), and a block takes no more threads and registers than a CTA of the GEMM leaves (768 x 80 of 65536), so that neither waits for the other's SM.
// In a chain, against blocks of 256 and no prefetch: int4 24 rows of 14336 x 4096 20.9 -> 19.8 us, 20 of 4096 x 4096 14.0 -> 13.4, 128 of 14336 x 4096 26.8 ->
// 25.7, int8 32 of 8192 x 8192 24.1 -> 23.4.  (The GEMM let go behind the loads instead of at once: 24 -> 26.2 us at 77 rows.)
constexpr int kStageThreads = 64;
template <int SEG>
__global__ void __launch_bounds__(kStageThreads, 16) stage_x_kernel(const __nv_bfloat16* __restrict__ x, int64_t M, int64_t Kx, int64_t ldx, uint32_t pieces, int BR, int KU,
                                                                    uint32_t x_bytes, uint8_t* __restrict__ xt, uint32_t* __restrict__ tickets, int n_tickets,
                                                                    bool settled) {
  // The GEMM behind reads weights and parameters without a wait of its own.  They may be the work of the kernel in front of this
  // one (quantize_, then a call), so it is let go only when that one is over and its writes are visible; at once where the caller
  // answers for the weights (settled), as a decode step does: 16 tokens of 8 sequences through four layers 5842 us, behind the wait 5968
  if (settled) grid_launch_dependents();
  const uint32_t gid = blockIdx.x * kStageThreads + threadIdx.x, step = gridDim.x * (kStageThreads / 32), groups = (uint32_t)BR / 8;
  const int lane = threadIdx.x & 31, row8 = lane >> 2, quarter = lane & 3;  // quarter: 32-k piece of the unit
  uint32_t w = gid >> 5;
  if (w < pieces) {
    const uint32_t rg = w / (uint32_t)KU, ku = w - rg * (uint32_t)KU;
    const int64_t m = (int64_t)rg * 8 + row8, k0 = (int64_t)ku * 128 + quarter * 32;
    if (m < M && k0 < Kx) asm volatile("prefetch.global.L2 [%0];" ::"l"(x + m * ldx + k0));
  }
  grid_dependency_wait();
  if (!settled) grid_launch_dependents();
  uint4 v[4];
  // a warp's piece: 8 rows x 128 k
  auto load = [&](uint32_t w) {
    const uint32_t rg = w / (uint32_t)KU, ku = w - rg * (uint32_t)KU;         // row group: 8 rows, block after block
    const int64_t m = (int64_t)rg * 8 + row8, k0 = (int64_t)ku * 128 + quarter * 32;
    const __nv_bfloat16* src = x + m * ldx + k0;
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      v[c] = make_uint4(0u, 0u, 0u, 0u);
      if (m < M && k0 + 8 * c < Kx) v[c] = *reinterpret_cast<const uint4*>(src + 8 * c);  // Kx % 8 == 0: all or nothing
    }
  };
  if (w < pieces) load(w);
  for (int i = (int)gid; i < n_tickets; i += gridDim.x * kStageThreads) tickets[i] = 0u;
  while (w < pieces) {
    const uint32_t rg = w / (uint32_t)KU, ku = w - rg * (uint32_t)KU, b = rg / groups, r = (rg - b * groups) * 8 + row8;
    uint8_t* unit = xt + ((int64_t)b * KU + ku) * x_bytes;
    uint8_t* dst = unit + ((int64_t)(quarter * 4) * BR + r) * 16;
    *reinterpret_cast<uint4*>(dst) = make_uint4(v[0].x, v[1].x, v[2].x, v[3].x);
    *reinterpret_cast<uint4*>(dst + (int64_t)BR * 16) = make_uint4(v[0].y, v[1].y, v[2].y, v[3].y);
    *reinterpret_cast<uint4*>(dst + (int64_t)BR * 32) = make_uint4(v[0].z, v[1].z, v[2].z, v[3].z);
    *reinterpret_cast<uint4*>(dst + (int64_t)BR * 48) = make_uint4(v[0].w, v[1].w, v[2].w, v[3].w);
    if constexpr (SEG > 0) {
      float s = 0.f;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float f[8];
        unpack8(v[c], f);
#pragma unroll
        for (int e = 0; e < 8; ++e) s += f[e];
      }
      if (SEG >= 64) s += __shfl_xor_sync(0xffffffffu, s, 1);
      if (SEG >= 128) s += __shfl_xor_sync(0xffffffffu, s, 2);
      if ((quarter * 32) % SEG == 0) reinterpret_cast<float*>(unit + (int64_t)BR * 256)[(quarter * 32 / SEG) * 16 + r] = s;
    }
    w += step;
    if (w < pieces) load(w);
  }
}

// DIRECT: nothing to stage, but the tickets (n >= 1 words); lets the GEMM go as stage_x_kernel does
__global__ void __launch_bounds__(kStageThreads, 16) clear_tickets_kernel(uint32_t* __restrict__ tickets, int n, bool settled) {
  if (settled) grid_launch_dependents();
  grid_dependency_wait();
  if (!settled) grid_launch_dependents();
  for (int i = blockIdx.x * kStageThreads + threadIdx.x; i < n; i += gridDim.x * kStageThreads) tickets[i] = 0u;
}

// ---- PTX wrappers ------------------------------------------------------------------------------------------------------
__device__ __forceinline__ void wq_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void wq_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ bool wq_elect_one() {
  uint32_t pred;
  asm volatile("{\n\t.reg .b32 rx;\n\t.reg .pred px;\n\telect.sync rx|px, 0xffffffff;\n\tselp.u32 %0, 1, 0, px;\n\t}" : "=r"(pred));
  return pred != 0;
}
// PAIR: both CTAs' barriers at this offset
template <bool PAIR>
__device__ __forceinline__ void wq_commit(uint64_t* bar) {
  if constexpr (PAIR)
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)), "h"((uint16_t)3)
                 : "memory");
  else
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// D(tmem, f32 [128 or 256][N]) (+)= A(tmem, bf16 [..][16]) * B(smem, bf16 [N][16])
template <bool PAIR>
__device__ __forceinline__ void wq_mma(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
  if constexpr (PAIR)
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem),
                 "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
  else
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem), "r"(a_tmem),
                 "l"(b_desc), "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void wq_st_16x128b_x8(uint32_t taddr, const uint32_t* r) {
  asm volatile("tcgen05.st.sync.aligned.16x128b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]),
               "r"(r[14]), "r"(r[15])
               : "memory");
}
// 16 lanes x 16 columns: thread l holds row l / 4 (d[0], d[1]; second 8 columns d[4], d[5]) and row l / 4 + 8 (d[2], d[3], d[6], d[7]),
// columns 2 (l % 4), + 1 of each 8
__device__ __forceinline__ void wq_ld_16x256b_x2(uint32_t taddr, uint32_t* d) {
  asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(d[0]), "=r"(d[1]), "=r"(d[2]), "=r"(d[3]), "=r"(d[4]), "=r"(d[5]), "=r"(d[6]), "=r"(d[7])
               : "r"(taddr));
}
__device__ __forceinline__ void wq_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// four 8 x 8 blocks of that shape, transposed: lanes 8 i .. 8 i + 7 give the row addresses of block i
__device__ __forceinline__ void wq_stmatrix_trans(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
  asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1,%2,%3,%4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {  // one rounding per product
  uint32_t d;
  asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ uint32_t add_bf16x2(uint32_t a, uint32_t b) {  // one rounding per sum
  uint32_t d;
  asm("add.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
  return d;
}
__device__ __forceinline__ void wq_tma_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(smem_u32(dst)), "l"(map),
               "r"(x), "r"(y), "r"(smem_u32(bar))
               : "memory");
}
// arrival on the leader CTA's barrier at this offset (PAIR), else on the own one.  (What it announces is in tensor memory or was
// written by the async proxy and is complete; .release.cluster here made every arrival wait about 1900 clocks.)
template <bool PAIR>
__device__ __forceinline__ void wq_arrive_leader(uint64_t* bar) {
  if constexpr (PAIR)
    asm volatile("{\n\t.reg .b32 ra;\n\tmapa.shared::cluster.u32 ra, %0, 0;\n\tmbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}" ::"r"(smem_u32(bar)) : "memory");
  else
    mbar_arrive(bar);
}
// bounded wait: false (and *dead set) after `limit` clocks, or as soon as another warp of the CTA has given up.  The lanes of a warp may
// answer differently then.  So roles of whole warps keep their answer and their place in the loops (their instructions are the
// warp's); what they must not do any more is announce: neither products nor arrivals that the other CTA of a pair would believe.
__device__ __forceinline__ bool wq_wait(uint64_t* bar, uint32_t parity, volatile int* dead, long long limit) {
  if (mbar_try_wait(bar, parity)) return true;
  const long long t0 = clock64();
  for (;;) {
    if (*dead != 0 || clock64() - t0 > limit) {
      *dead = 1;
      return false;
    }
#pragma unroll 1
    for (int i = 0; i < 32; ++i)
      if (mbar_try_wait(bar, parity)) return true;
  }
}
// barrier of the epilogue warps; true if any of them brings a failure
__device__ __forceinline__ bool wq_epi_sync(bool failed) {
  uint32_t any;
  asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.or.pred q, 1, %2, p;\n\tselp.u32 %0, 1, 0, q;\n\t}"
               : "=r"(any)
               : "r"((uint32_t)failed), "n"(kWqEpiWarps * 32)
               : "memory");
  return any != 0;
}
// DEFER: the sum of x W' for one weight row and one row of x, all from global memory.  w: the strip's words; sz: the row's
// parameters, 16 words apart per group; x: the row's pieces in the staged units
template <int G>
__device__ __forceinline__ float wq_exact(const uint32_t* w, const uint32_t* sz, const uint8_t* x, uint32_t x_bytes, int K, int g, int hrow) {
  float sum = 0.f;
#pragma unroll 1
  for (int k = 0; k < K; k += 8) {
    const int q4 = k >> 5, c = (k >> 3) & 3;
    const uint32_t szw = __ldg(sz + (int64_t)(k / G) * 16);
    uint32_t o[4];
    dequant_word(__ldg(w + (int64_t)(k >> 6) * 128 + (4 * g + c) * 4 + 2 * (q4 & 1) + hrow), __byte_perm(szw, 0, 0x1010), __byte_perm(szw, 0, 0x3232), o);
    const uint8_t* piece = x + (int64_t)(k >> 7) * x_bytes + (q4 & 3) * 4 * 256 + c * 4;  // chunks of 16 rows x 16 bytes
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const uint32_t xv = __ldcg(reinterpret_cast<const uint32_t*>(piece + i * 256));
      sum = fmaf(__uint_as_float(xv << 16), __uint_as_float(o[i] << 16), sum);
      sum = fmaf(__uint_as_float(xv & 0xFFFF0000u), __uint_as_float(o[i] & 0xFFFF0000u), sum);
    }
  }
  return sum;
}
// DEFER: eight results of row m of x that are not all finite.  D or X may have overflowed where the sum itself does not, or their difference
// may have lost an infinity's sign, so they are done again from the weights.  Rare, and slow (a row of 8192: milliseconds); out of line and
// asked for once per result, so that the roles' loops stay as they are (28672 x 8192, 16 rows: 45.1 us without it, 45.8 with it; staging that
// marks such rows and an epilogue that looks at every unit: 50)
template <int G>
__device__ __noinline__ uint4 wq_again(const WqParams& p, uint4 v, int m, int64_t n0) {
  uint32_t o[4] = {v.x, v.y, v.z, v.w};
#pragma unroll 1
  for (int e = 0; e < 8; ++e) {
    const int n = (int)n0 + e, r = n & 15;
    const uint32_t bits = float_to_bf16_bits(wq_exact<G>(p.packed + (int64_t)(n >> 4) * p.Kp * 2, p.sz + (int64_t)(n >> 4) * (p.Kp / G) * 16 + r,
                                                         p.xt + m * 16, p.x_sub, p.Kp, r & 7, r >> 3));
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (i == (e >> 1)) o[i] = e & 1 ? (o[i] & 0xFFFFu) | (bits << 16) : (o[i] & 0xFFFF0000u) | bits;
  }
  return make_uint4(o[0], o[1], o[2], o[3]);
}
// whether any of eight bf16 is an infinity or NaN
__device__ __forceinline__ bool any_inf_bf16(uint4 v) {
  const auto half = [](uint32_t w) { return (w & 0x7F80u) == 0x7F80u || (w & 0x7F800000u) == 0x7F800000u; };
  return half(v.x) || half(v.y) || half(v.z) || half(v.w);
}
// Between the four lanes c of a row group: lane c has of each of two words the weights k = 8 c + 2 i, + 1 (i = 0 .. 3, pair i at bits 4 i and 16 + 4 i)
// and gets those of k = 8 c' + 2 c, + 1 (c' = 0 .. 3, at bits 4 c' and 16 + 4 c'): the place of a pair in the word and the lane change roles, first
// their upper bits (bytes), then their lower ones (half bytes).
__device__ __forceinline__ void wq_turn_int4(uint32_t& a, uint32_t& b, int lane) {
  constexpr uint32_t kLow = 0x0F0F0F0Fu;
  const bool up = lane & 2, odd = lane & 1;
  uint32_t r = __shfl_xor_sync(0xffffffffu, __byte_perm(a, b, up ? 0x6420u : 0x7531u), 2);
  a = __byte_perm(a, r, up ? 0x3514u : 0x5240u);
  b = __byte_perm(b, r, up ? 0x3716u : 0x7260u);
  const uint32_t keep = odd ? ~kLow : kLow, s0 = odd ? 0u : 4u, s4 = 4u - s0;
  r = __shfl_xor_sync(0xffffffffu, ((a >> s0) & kLow) | ((b << s4) & ~kLow), 1);
  a = (a & keep) | ((r << s0) & ~keep);
  b = (b & keep) | ((r >> s4) & ~keep);
}
// the same for bytes: a has the pairs i = 0, 1, b has 2, 3; after it a has those of c' = 0, 1, b of c' = 2, 3
__device__ __forceinline__ void wq_turn_int8(uint32_t& a, uint32_t& b, int lane) {
  const bool up = lane & 2, odd = lane & 1;
  uint32_t r = __shfl_xor_sync(0xffffffffu, up ? a : b, 2);
  a = up ? r : a;
  b = up ? b : r;
  r = __shfl_xor_sync(0xffffffffu, __byte_perm(a, b, odd ? 0x5410u : 0x7632u), 1);
  a = __byte_perm(a, r, odd ? 0x3254u : 0x5410u);
  b = __byte_perm(b, r, odd ? 0x3276u : 0x7610u);
}
// ring position: slot and the parity of its current use
struct WqRing {
  int slot = 0;
  uint32_t use = 0;
  __device__ __forceinline__ void step(int by, int n) {
    slot += by;
    if (slot >= n) {
      slot -= n;
      use ^= 1u;
    }
  }
};

// ---- the GEMM ----------------------------------------------------------------------------------------------------------
// G == 0: int8.  Shared memory: header, output tile, activation ring (x_slots x x_bytes), weight ring (w_slots x [8 strips x 128 k]
// [8 strips x parameters]).
template <int G, bool DEFER, bool PAIR, bool DIRECT, bool EARLY, int KW>
__global__ void __launch_bounds__(kWqThreads, 1) wq_gemm_kernel(const __grid_constant__ WqParams p) {
  extern __shared__ __align__(1024) uint8_t wq_smem[];
  constexpr bool kI8 = (G == 0);
  constexpr int kTileB = kI8 ? 1024 : 512;                                // bytes of one (strip, 64-k) tile
  constexpr int kSegs = DEFER ? (G < 128 ? 128 / (G ? G : 128) : 1) : 1;  // accumulation segments per unit
  constexpr int kSzWords = kI8 ? 0 : (G < 128 ? 128 / (G ? G : 128) : 1) * 16;
  constexpr uint32_t kWBytes = 8 * 2 * kTileB, kSBytes = 8 * kSzWords * 4, kWSub = kWBytes + kSBytes, kWSlot = KW * kWSub;
  constexpr int kAllSegs = KW * kSegs;  // of a unit, KW times 128 k
  constexpr int kRanks = PAIR ? 2 : 1;
  uint64_t* wfull = reinterpret_cast<uint64_t*>(wq_smem);
  uint64_t* wempty = wfull + kWqMaxW;
  uint64_t* xfull = wempty + kWqMaxW;     // per slot of x: the tile has landed here
  uint64_t* xpeer = xfull + kWqMaxX;      // PAIR, leader: ... and in the second CTA
  uint64_t* xdone = xpeer + kWqMaxX;      // the MMAs on it have retired (DEFER: D is final)
  uint64_t* dread = xdone + kWqMaxX;      // DEFER: the epilogue has read D and the sums
  uint64_t* afull = dread + kWqMaxX;      // per slot of A: it is in tensor memory
  uint64_t* adone = afull + kWqSlots;     // the MMAs on it have retired
  uint64_t* dfull = adone + kWqSlots;     // accumulator buffers of a tile
  uint64_t* dempty = dfull + 2;
  uint32_t* tmem_base_s = reinterpret_cast<uint32_t*>(dempty + 2);
  volatile int* dead = reinterpret_cast<volatile int*>(tmem_base_s + 1);
  volatile int* s_last = dead + 1;        // [3]: this CTA was the last to reach its first / last tile; it finishes its last tile from its accumulators
  uint8_t* stage = wq_smem + kWqHeader;   // output tile [NT][kWqPitch]
  uint8_t* xring = wq_smem + p.off_x;
  uint8_t* wring = wq_smem + p.off_w;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int worker = blockIdx.x / kRanks, rank = blockIdx.x % kRanks;
  const int u0 = wq_first(worker, p.base, p.rem, p.quantum), u1 = wq_first(worker + 1, p.base, p.rem, p.quantum);
  const int KU = p.KU, NT = p.NT, x_slots = p.x_slots, a_slots = p.a_slots, n_mma = p.n_mma;
  const int d_bufs = NT <= 128 ? 2 : 1;
  auto wait = [&](uint64_t* bar, uint32_t parity) { return wq_wait(bar, parity, dead, p.wait_limit); };
  grid_launch_dependents();

  // the weights do not wait for the staging kernel (see there): their producer fills the ring while the others set up
  // (running positions: a division per unit is what paced the producers)
  const int t_first = u0 / KU, ku_first = u0 - t_first * KU;
  int w_ku = ku_first, w_mt = t_first % p.MT, w_strip = ((t_first / p.MT) * kRanks + rank) * 8;
  auto load_weights = [&](int slot) {
    const int ku = w_ku, strip = w_strip;
    if (++w_ku == KU) {
      w_ku = 0;
      if (++w_mt == p.MT) w_mt = 0, w_strip += kRanks * 8;
    }
    uint8_t* dst = wring + slot * kWSlot;
    mbar_arrive_expect_tx(&wfull[slot], kWSlot);
#pragma unroll
    for (int j = 0; j < KW; ++j) {  // (128 k past the end: zeros)
      wq_tma_2d(dst + j * kWSub, &p.wmap, (ku * KW + j) * 256, strip, &wfull[slot]);
      if constexpr (!kI8) wq_tma_2d(dst + j * kWSub + kWBytes, &p.smap, G == 256 ? ((ku * KW + j) >> 1) * 16 : (ku * KW + j) * kSzWords, strip, &wfull[slot]);
    }
  };
  if (warp == kWqWProd) {
    if (lane < p.w_slots) {
      mbar_init(&wfull[lane], 1);
      mbar_init(&wempty[lane], DEFER ? 8 + kWqEpiWarps : 8);  // DEFER: the epilogue reads the parameters
    }
    fence_barrier_init();
    __syncwarp();
    if (wq_elect_one())
      for (int i = 0; i < p.w_slots && u0 + i < u1; ++i) load_weights(i);
    __syncwarp();
  } else if (warp == kWqMma) {
    if (lane < x_slots) {
      mbar_init(&xfull[lane], 1);
      mbar_init(&xpeer[lane], 1);
      mbar_init(&xdone[lane], 1);
      mbar_init(&dread[lane], kWqEpiWarps);
    } else if (lane >= 8 && lane < 8 + kWqSlots) {
      mbar_init(&afull[lane - 8], 8 * kRanks);
      mbar_init(&adone[lane - 8], 1);
    } else if (lane >= 16 && lane < 18) {
      mbar_init(&dfull[lane - 16], n_mma);
      mbar_init(&dempty[lane - 16], kWqEpiWarps * kRanks);
      s_last[lane - 16] = 0;
    } else if (lane == 18) {
      *dead = 0;
      s_last[2] = 0;
    }
    fence_barrier_init();
    __syncwarp();
    if constexpr (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_s)), "r"(512));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_base_s)), "r"(512));
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    wq_fence_before();
  }
  __syncthreads();
  if constexpr (PAIR) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  wq_fence_after();
  const uint32_t tb = *reinterpret_cast<volatile uint32_t*>(tmem_base_s);
  // columns [0, 256): accumulators (DEFER: one per slot of x and segment, else [buffer][MMA warp]); [256, 512): A ring
  const uint32_t a_col0 = tb + 256;

  // fp32 sums of rows 32 q + 16 h .. + 15, columns c .. c + 15 (fragment order of wq_ld_16x256b_x2) -> output tile
  auto to_stage = [&](int q, int c, int h, const float* f, const uint32_t (&sc)[4]) {
    const uint32_t at = smem_u32(stage) + (uint32_t)(c + 8 * (lane >> 4) + (lane & 7)) * kWqPitch + (32 * q + 16 * h + 8 * ((lane >> 3) & 1)) * 2;
    uint32_t o[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // block i: column group i >> 1, row group i & 1
      const float a = f[4 * (i >> 1) + 2 * (i & 1)], b = f[4 * (i >> 1) + 2 * (i & 1) + 1];
      asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(o[i]) : "f"(b), "f"(a));
      // int8: mm result rounded to bf16, THEN multiplied by the row scale and rounded again (the product of two bf16 is exact in fp32, so a packed
      // multiply rounds it once, as a product in fp32 and a conversion do, with a quarter of the instructions: int8 8192 x 8192, 2048 rows 220.2 -> 217.7 us,
      // 14336 x 4096, 700 / 300 rows 70.5 -> 68.6, 40.0 -> 38.9)
      if constexpr (kI8) o[i] = mul_bf16x2(o[i], h ? sc[2 + (i & 1)] : sc[i & 1]);
    }
    wq_stmatrix_trans(at, o[0], o[1], o[2], o[3]);
  };
  // the row scales (int8) of a thread's four rows 32 q + lane / 4 + 8 i, each twice
  auto row_scales = [&](int nb, int q, uint32_t (&sc)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int64_t n = ((int64_t)nb * kRanks + rank) * 128 + 32 * q + (lane >> 2) + 8 * i;
      sc[i] = kI8 && n < p.N_out ? __bfloat16_as_ushort(p.scale8[n]) * 0x10001u : 0u;
    }
  };
  // output tile -> y: 16-byte pieces of 256-byte rows; `threads` threads, this one is number `th`
  auto copy_out = [&](int nb, int mt, int th, int threads) {
    const int64_t nbase = ((int64_t)nb * kRanks + rank) * 128;
    const int m0 = mt * NT, rows = min(NT, p.M - m0);
    const int col = th & 15;
    const int64_t n0 = nbase + col * 8;
    if (n0 >= p.N_out) return;
    __nv_bfloat16* dst = p.y + (int64_t)m0 * p.ldy + n0;
    const __nv_bfloat16* res = p.residual == nullptr ? nullptr : p.residual + (int64_t)m0 * p.ld_res + n0;
    const uint32_t src = smem_u32(stage) + col * 16;
    const bool vec = p.vec_store && n0 + 8 <= p.N_out;
#pragma unroll 4
    for (int m = th >> 4; m < rows; m += threads >> 4) {
      uint4 v = lds128(src + m * kWqPitch);
      if constexpr (DEFER)
        if (__builtin_expect(any_inf_bf16(v), 0)) v = wq_again<G>(p, v, m0 + m, n0);
      if (vec) {
        if (res != nullptr) {
          const uint4 r = *reinterpret_cast<const uint4*>(res + m * p.ld_res);
          v = make_uint4(add_bf16x2(r.x, v.x), add_bf16x2(r.y, v.y), add_bf16x2(r.z, v.z), add_bf16x2(r.w, v.w));
        }
        *reinterpret_cast<uint4*>(dst + m * p.ldy) = v;
      } else {
        const uint32_t vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int e = 0; e < 8; ++e) {
          if (n0 + e >= p.N_out) continue;
          __nv_bfloat16 o = __ushort_as_bfloat16((unsigned short)(vv[e >> 1] >> (16 * (e & 1))));
          if (res != nullptr) o = __float2bfloat16_rn(__bfloat162float(res[m * p.ld_res + e]) + __bfloat162float(o));
          dst[m * p.ldy + e] = o;
        }
      }
    }
  };
  // share of worker c in tile t: [NT / 16 column blocks][2 halves x 2 column groups][4 quadrants][32 lanes] float4
  auto share = [&](int c, int t) {
    const int slot = wq_first(c, p.base, p.rem, p.quantum) >= t * KU ? 0 : 1;  // its first tile, or its last
    return reinterpret_cast<float4*>(p.part) + (((int64_t)c * 2 + slot) * kRanks + rank) * NT * 32;
  };

  if (warp == kWqWProd) {
    // ---- weight producer ----
    if (wq_elect_one()) {
      WqRing w;
      w.use = 1;
      for (int u = u0 + p.w_slots; u < u1; ++u) {
        if (!wait(&wempty[w.slot], w.use ^ 1u)) break;
        load_weights(w.slot);
        w.step(1, p.w_slots);
      }
    }
    __syncwarp();
  } else if (warp == kWqXProd) {
    // ---- activation producer ----
    grid_dependency_wait();
    if (wq_elect_one()) {
      WqRing x;
      const int64_t tile_bytes = (int64_t)KU * p.x_bytes;
      const uint8_t* base = DIRECT ? nullptr : p.xt + rank * tile_bytes;
      int mt = t_first % p.MT, ku = ku_first;
      const uint8_t* src = DIRECT ? nullptr : base + mt * (kRanks * tile_bytes) + (int64_t)ku * p.x_bytes;
      for (int u = u0; u < u1; ++u) {
        if (!wait(DEFER ? &dread[x.slot] : &xdone[x.slot], x.use ^ 1u)) break;
        mbar_arrive_expect_tx(&xfull[x.slot], p.x_bytes);
        uint8_t* dst = xring + (uint32_t)x.slot * p.x_bytes;
        if constexpr (DIRECT) {
          const int row = (mt * kRanks + rank) * p.BR;
          wq_tma_2d(dst, &p.xmap, ku * 128, row, &xfull[x.slot]);
          wq_tma_2d(dst + p.BR * 128, &p.xmap, ku * 128 + 64, row, &xfull[x.slot]);
        } else {
          bulk_g2s(dst, src, p.x_bytes, &xfull[x.slot]);
          src += p.x_bytes;
        }
        x.step(1, x_slots);
        if (++ku == KU) {
          ku = 0;
          if (++mt == p.MT) mt = 0;
          if (!DIRECT) src = base + mt * (kRanks * tile_bytes);
        }
      }
    }
    __syncwarp();
  } else if (warp >= kWqMma) {
    const int mw = warp - kWqMma;
    WqRing x, a, d;
    if (PAIR && rank != 0) {
      // ---- the pair's second CTA: tells the first one that its half of the activations has landed ----
      bool ok = true;
      for (int u = u0; u < (mw == 0 ? u1 : u0); ++u) {
        ok = ok && wait(&xfull[x.slot], x.use);
        if (wq_elect_one() && ok) wq_arrive_leader<PAIR>(&xpeer[x.slot]);
        __syncwarp();
        x.step(1, x_slots);
      }
    } else {
      // ---- MMA issue: 8 x (M 128 / 256, N = NT, K 16) per unit, whole warp in uniform control flow ----
      x.step(mw, x_slots);
      a.step(mw, a_slots);
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)NT >> 3) << 17) | (((128u * kRanks) >> 4) << 24);
      // B tile: chunks of 8 k, `chunk` bytes from one to the next.  DIRECT: [64 k][BR rows][128 bytes], 1024 bytes from 8 rows to the next
      const uint32_t chunk = (uint32_t)p.BR * 16;
      const uint32_t desc_hi = DIRECT ? (1024u >> 4) | (1u << 14) | (2u << 29) : (128u >> 4) | (1u << 14);
      const uint32_t kstep = DIRECT ? 32u >> 4 : (2 * chunk) >> 4, khalf = DIRECT ? ((uint32_t)p.BR * 128 - 4 * 32) >> 4 : 0u;
      const uint32_t desc_lo = (DIRECT ? 0u : (chunk >> 4) << 16) | ((smem_u32(xring) & 0x3FFFFu) >> 4), xstep = p.x_bytes >> 4, xsub = p.x_sub >> 4;
      int u = u0;
      bool ok = true;
      while (u < (mw < n_mma ? u1 : u0)) {
        const int ue = min(u1, (u / KU + 1) * KU);  // the units of this tile
        if (!DEFER) ok = ok && wait(&dempty[d.slot], d.use ^ 1u);
        const uint32_t dcol = tb + d.slot * 128 + mw * 64;
        uint32_t acc = 0;
        // this warp's units: those whose number in the CTA's sequence is mw (mod n_mma)
        if (n_mma == 2 && ((u - u0) & 1) != mw) ++u;
        for (; u < ue; u += n_mma) {
          const bool ra = mbar_try_wait(&afull[a.slot], a.use), rx = mbar_try_wait(&xfull[x.slot], x.use);
          ok = ok && (ra || wait(&afull[a.slot], a.use)) && (rx || wait(&xfull[x.slot], x.use));
          if (PAIR) ok = ok && wait(&xpeer[x.slot], x.use);
          wq_fence_after();
          if (wq_elect_one() && ok) {
            const uint32_t b0 = desc_lo + (uint32_t)x.slot * xstep, a0 = a_col0 + a.slot * (64 * KW);
            const uint32_t d0 = DEFER ? tb + x.slot * (kAllSegs * 16) : dcol;
#pragma unroll
            for (int ks = 0; ks < 8 * KW; ++ks) {
              const uint64_t bdesc = ((uint64_t)desc_hi << 32) | (b0 + (ks & 7) * kstep + ((ks & 7) >= 4 ? khalf : 0u) + (ks >= 8 ? xsub : 0u));
              wq_mma<PAIR>(d0 + (DEFER ? ks / (8 / kSegs) * 16 : 0), a0 + 8 * ks, bdesc, idesc, DEFER ? (ks % (8 / kSegs) != 0) : (ks != 0 ? 1u : acc));
            }
            wq_commit<PAIR>(&adone[a.slot]);
            wq_commit<PAIR>(&xdone[x.slot]);
          }
          __syncwarp();
          acc = 1;
          x.step(n_mma, x_slots);
          a.step(n_mma, a_slots);
        }
        u = ue;
        if (!DEFER) {
          if (wq_elect_one() && ok) wq_commit<PAIR>(&dfull[d.slot]);
          __syncwarp();
          d.step(1, d_bufs);
        }
      }
    }
  } else if (warp >= kWqEpiWarps) {
    // ---- dequant: packed words -> bf16 -> tensor memory; 8 words (int4) of one strip per warp and unit ----
    const int dq = (warp - kWqEpiWarps) & 7, set = (warp - kWqEpiWarps) >> 3, qd = warp & 3, strip = 2 * qd + (dq >> 2);
    const uint32_t taddr0 = a_col0 + ((uint32_t)(32 * qd + 16 * (dq >> 2)) << 16);
    const uint32_t w0_u = smem_u32(wring) + strip * (2 * kTileB) + lane * 16;
    const uint32_t s0_u = smem_u32(wring) + kWBytes + strip * (kSzWords * 4) + (lane >> 2) * 4;
    WqRing w, a;
    w.step(set, p.w_slots);
    a.step(set, a_slots);
    // A weight slot of an odd ring is used by the two sets in turn, and a set must not look for its phase of `wfull` before the
    // other set's phase in between (unit u - w_slots) is over.  That unit has retired when the A slot is free, as long as w_slots >= a_slots:
    // so with a short odd ring the A slot is waited for first.  (A longer ring cannot be overtaken while one MMA warp keeps the
    // sets at most a_slots + 1 units apart; with two the ring is even.)
    const bool a_first = (p.w_slots & 1) && p.w_slots < a_slots + 2;
    // DEFER: the words of the next unit are fetched while this unit's store to tensor memory is on its way (28672 x 8192, 16 rows: 46.4 -> 44.1
    // us).  The others are bound by the conversions or the MMAs and do best announcing first (int8 8192 x 8192, 2048 rows: 217 against 223 us).
    constexpr int kWords = kI8 ? 16 : 8, kSzn = (kI8 || DEFER) ? 1 : kSzWords / 16;
    uint32_t wd[kWords], sz[kSzn][2];
    bool ok = true;
    auto words = [&](int j) {  // of the unit's j-th 128 k
      const uint32_t wt = w0_u + w.slot * kWSlot + j * kWSub, st = s0_u + w.slot * kWSlot + j * kWSub;
#pragma unroll
      for (int i = 0; i < kWords / 4; ++i) {
        const uint4 v = lds128(wt + i * 512);
        wd[4 * i] = v.x, wd[4 * i + 1] = v.y, wd[4 * i + 2] = v.z, wd[4 * i + 3] = v.w;
      }
      if constexpr (!kI8 && !DEFER) {
#pragma unroll
        for (int h = 0; h < kSzn; ++h) {
          sz[h][0] = lds32(st + h * 64);
          sz[h][1] = lds32(st + h * 64 + 32);
        }
      }
    };
    auto fetch = [&](int u) {
      if (u >= u1) return;
      if (a_first) ok = ok && wait(&adone[a.slot], a.use ^ 1u);
      ok = ok && wait(&wfull[w.slot], w.use);
      words(0);
    };
    fetch(u0 + set);
    for (int u = u0 + set; u < u1; u += 2) {
      uint32_t r[32];
      auto convert = [&]() {
        if constexpr (DIRECT) {  // x is in its own order, so the weights have to be
#pragma unroll
          for (int j = 0; j < kWords; j += kI8 ? 4 : 2) {
            if constexpr (kI8) {
              wq_turn_int8(wd[j], wd[j + 2], lane);
              wq_turn_int8(wd[j + 1], wd[j + 3], lane);
            } else {
              wq_turn_int4(wd[j], wd[j + 1], lane);
            }
          }
        }
        if constexpr (kI8) {
#pragma unroll
          for (int j = 0; j < 16; ++j) {  // 32-k quarters of the unit; lane chunk: words (row g, k 0-3), (g+8, k 0-3), (g, k 4-7), (g+8, k 4-7)
            const int q4 = j >> 2, hrow = j & 1, i0 = 2 * ((j >> 1) & 1);
            u8x4_to_bf16x2x2(wd[j], r[2 * (4 * q4 + i0) + hrow], r[2 * (4 * q4 + i0 + 1) + hrow]);
          }
        } else {
#pragma unroll
          for (int j = 0; j < 8; ++j) {  // word j: row g + 8 (j & 1), 32-k quarter j >> 1 of the unit
            const int q4 = j >> 1, hrow = j & 1;
            uint32_t o[4];
            if constexpr (DEFER) {
#pragma unroll
              for (int i = 0; i < 4; ++i) asm("lop3.b32 %0, %1, 0x000f000f, 0x43004300, 0xea;" : "=r"(o[i]) : "r"(wd[j] >> (4 * i)));  // 128 + q
            } else {
              const uint32_t szw = sz[q4 * kSzn / 4][hrow];
              dequant_word(wd[j], __byte_perm(szw, 0, 0x1010), __byte_perm(szw, 0, 0x3232), o);
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) r[2 * (4 * q4 + i) + hrow] = o[i];
          }
        }
      };
      convert();
      if constexpr (KW == 2) words(1);
      __syncwarp();
      if (lane == 0) mbar_arrive(&wempty[w.slot]);  // everything that this warp reads of the slot is in registers
      ok = ok && wait(&adone[a.slot], a.use ^ 1u);  // the MMAs that read this A slot have retired
      wq_fence_after();
      const uint32_t ta = taddr0 + a.slot * (64 * KW);
      wq_st_16x128b_x8(ta, r);
      wq_st_16x128b_x8(ta + 32, r + 16);
      if constexpr (KW == 2) {
        convert();
        wq_st_16x128b_x8(ta + 64, r);
        wq_st_16x128b_x8(ta + 96, r + 16);
      }
      uint64_t* full = &afull[a.slot];
      const bool announce = ok;
      w.step(2, p.w_slots);
      a.step(2, a_slots);
      if (DEFER && !a_first) fetch(u + 2);
      asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
      wq_fence_before();
      __syncwarp();
      if (lane == 0 && announce) wq_arrive_leader<PAIR>(full);
      if (!DEFER || a_first) fetch(u + 2);  // (a_first waits for MMAs: not before this unit is announced)
    }
  } else {
    // ---- epilogue ----
    grid_dependency_wait();
    const uint32_t lane_col = tb + ((uint32_t)(32 * warp) << 16);
    WqRing d, x, w;
    bool ok = true;
    // EARLY: this CTA's last tile, if it is shared with the next one alone and that one has more to do behind it: as a rule that one's share was there
    // long ago.  Then this one stays in tensor memory and all warps finish the tile, at the end: no store of NT * 512 bytes and its way back.
    int t_early = -1;
    if (EARLY && u1 % KU != 0) {
      const int t = u1 / KU;
      if (u0 <= t * KU && wq_first(worker + 2, p.base, p.rem, p.quantum) >= (t + 1) * KU + (KW == 2 ? kWqBehindLong : kWqBehind)) t_early = t;
    }
    for (int u = u0, t = u0 / KU; u < u1; ++t) {
      const int ue = min(u1, (t + 1) * KU), nb = t / p.MT, mt = t - nb * p.MT;
      const bool whole = u == t * KU && ue == (t + 1) * KU;
      float4* mine = share(worker, t) + warp * 32 + lane;
      uint32_t sc[4];
      row_scales(nb, warp, sc);
      if (whole) wq_epi_sync(false);  // the previous output tile has been copied out
      if constexpr (DEFER) {
        float acc[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] = 0.f;
        for (; u < ue; ++u) {
          const bool rw = mbar_try_wait(&wfull[w.slot], w.use), rx = mbar_try_wait(&xfull[x.slot], x.use), rd = mbar_try_wait(&xdone[x.slot], x.use);
          ok = ok && (rw || wait(&wfull[w.slot], w.use)) && (rx || wait(&xfull[x.slot], x.use)) && (rd || wait(&xdone[x.slot], x.use));
          wq_fence_after();
          // parameters of rows 32 warp + lane / 4 + 8 i, sums of columns 2 (lane % 4) + {0, 1, 8, 9}
          const uint32_t st0 = smem_u32(wring) + w.slot * kWSlot + kWBytes + 2 * warp * (kSzWords * 4) + (lane >> 2) * 4;
          const uint32_t xs0 = smem_u32(xring) + (uint32_t)x.slot * p.x_bytes + 16 * 256 + (lane & 3) * 8;
#pragma unroll
          for (int all = 0; all < kAllSegs; ++all) {
            const int sg = all % kSegs;
            const uint32_t st = st0 + all / kSegs * kWSub, xs = xs0 + all / kSegs * p.x_sub;
            uint32_t v[16];
            wq_ld_16x256b_x2(lane_col + (x.slot * kAllSegs + all) * 16, v);
            wq_ld_16x256b_x2(lane_col + (16u << 16) + (x.slot * kAllSegs + all) * 16, v + 8);
            float s[4], zt[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              const uint32_t szw = lds32(st + (i >> 1) * (kSzWords * 4) + sg * 64 + (i & 1) * 32);
              s[i] = __uint_as_float(szw << 16);
              zt[i] = fmaf(-136.f, s[i], __uint_as_float(szw & 0xFFFF0000u));
            }
            const float2 xa = lds64f(xs + sg * 64), xb = lds64f(xs + sg * 64 + 32);
            const float X[4] = {xa.x, xa.y, xb.x, xb.y};
            wq_ld_wait();
            const F2 x2[2] = {f2(X[0], X[1]), f2(X[2], X[3])};
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int e = 0; e < 8; e += 2) {  // e: column group e >> 2, row group (e >> 1) & 1, column e & 1
                const int r = 2 * h + ((e >> 1) & 1);
                const F2 part = f2_fma(f2(zt[r], zt[r]), x2[e >> 2], f2(acc[8 * h + e], acc[8 * h + e + 1]));
                const float2 y = f2_get(f2_fma(f2(s[r], s[r]), f2(__uint_as_float(v[8 * h + e]), __uint_as_float(v[8 * h + e + 1])), part));
                acc[8 * h + e] = y.x, acc[8 * h + e + 1] = y.y;
              }
          }
          wq_fence_before();
          __syncwarp();
          if (lane == 0) {
            mbar_arrive(&dread[x.slot]);
            mbar_arrive(&wempty[w.slot]);
          }
          x.step(1, x_slots);
          w.step(1, p.w_slots);
        }
        if (whole) {
          to_stage(warp, 0, 0, acc, sc);
          to_stage(warp, 0, 1, acc + 8, sc);
        } else {
#pragma unroll
          for (int i = 0; i < 4; ++i) __stcg(mine + i * 128, make_float4(acc[4 * i], acc[4 * i + 1], acc[4 * i + 2], acc[4 * i + 3]));
        }
      } else {
        ok = ok && wait(&dfull[d.slot], d.use);
        wq_fence_after();
        if (EARLY && t == t_early) {
          if (wq_epi_sync(!ok)) break;
          bool here = false;
          if (threadIdx.x == 0) {
            uint32_t arrived;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(arrived) : "l"(p.tickets + t * kRanks + rank) : "memory");
            here = arrived == 1u;
            if (here) s_last[2] = 1;
          }
          if (wq_epi_sync(here)) {
            wq_fence_before();
            break;
          }
        }
        // which accumulators hold something: both MMA warps', unless the tile has one unit here
        const bool two = n_mma == 2 && ue - u > 1;
        const uint32_t dcol = lane_col + d.slot * 128 + (n_mma == 2 && ue - u == 1 ? ((u - u0) & 1) * 64 : 0);
#pragma unroll 1
        for (int c = 0; c < NT; c += 16) {
          uint32_t v[16];
          float f[16];
          wq_ld_16x256b_x2(dcol + c, v);
          wq_ld_16x256b_x2(dcol + (16u << 16) + c, v + 8);
          if (two) {
            uint32_t v2[16];
            wq_ld_16x256b_x2(dcol + 64 + c, v2);
            wq_ld_16x256b_x2(dcol + (16u << 16) + 64 + c, v2 + 8);
            wq_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]) + __uint_as_float(v2[i]);
          } else {
            wq_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) f[i] = __uint_as_float(v[i]);
          }
          if (c + 16 >= NT) {
            wq_fence_before();
            __syncwarp();
            if (lane == 0) wq_arrive_leader<PAIR>(&dempty[d.slot]);
          }
          if (whole) {
            to_stage(warp, c, 0, f, sc);
            to_stage(warp, c, 1, f + 8, sc);
          } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) __stcg(mine + (c / 4 + i) * 128, make_float4(f[4 * i], f[4 * i + 1], f[4 * i + 2], f[4 * i + 3]));
          }
        }
        d.step(1, d_bufs);
        u = ue;
      }
      if (!whole) __threadfence();
      if (wq_epi_sync(!ok)) break;
      if (whole) {
        copy_out(nb, mt, threadIdx.x, kWqEpiWarps * 32);
      } else if (threadIdx.x == 0) {
        // a tile shared with neighbours: whoever arrives last adds all shares (below)
        const int c0 = wq_owner(t * KU, p.base, p.rem, p.quantum), c1 = wq_owner(t * KU + KU - 1, p.base, p.rem, p.quantum);
        if (atomicAdd(&p.tickets[t * kRanks + rank], 1u) == (uint32_t)(c1 - c0)) s_last[t == u0 / KU ? 0 : 1] = 1;
      }
    }
  }

  // ---- shared tiles that this CTA was the last to reach: all warps add the shares in CTA order and finish the rows ----
  __syncthreads();
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    if (s_last[k] == 0) continue;
    __threadfence();
    const int t = k == 0 ? u0 / KU : (u1 - 1) / KU, nb = t / p.MT, mt = t - nb * p.MT;
    const int c0 = wq_owner(t * KU, p.base, p.rem, p.quantum), c1 = wq_owner(t * KU + KU - 1, p.base, p.rem, p.quantum);
    for (int it = warp; it < NT / 2; it += kWqThreads / 32) {  // (column block, quadrant, half)
      const int h = it & 1, q = (it >> 1) & 3, c = (it >> 3) * 16;
      float f[8];
      uint32_t sc[4];
#pragma unroll
      for (int i = 0; i < 8; ++i) f[i] = 0.f;
      row_scales(nb, q, sc);
#pragma unroll 4
      for (int cc = c0; cc <= c1; ++cc) {
        const float4* src = share(cc, t) + (c / 4 + 2 * h) * 128 + q * 32 + lane;
        const float4 v0 = __ldcg(src), v1 = __ldcg(src + 128);
        f[0] += v0.x, f[1] += v0.y, f[2] += v0.z, f[3] += v0.w, f[4] += v1.x, f[5] += v1.y, f[6] += v1.z, f[7] += v1.w;
      }
      to_stage(q, c, h, f, sc);
    }
    __syncthreads();
    copy_out(nb, mt, threadIdx.x, kWqThreads);
    __syncthreads();
  }
  if (EARLY && s_last[2] != 0) {
    // the last tile: this CTA's share, the first, is its accumulators (which of them hold something: as in the epilogue), the next CTA's is the other
    wq_fence_after();
    __threadfence();
    const int t = u1 / KU, nb = t / p.MT, mt = t - nb * p.MT, held = u1 - t * KU;
    const bool two = n_mma == 2 && held > 1;
    const int q = warp & 3;                                // tensor memory: a warp reaches the lanes of its quadrant
    const uint32_t dcol = tb + ((uint32_t)(32 * q) << 16) + (d_bufs == 2 ? ((t - u0 / KU) & 1) * 128 : 0) + (n_mma == 2 && held == 1 ? ((t * KU - u0) & 1) * 64 : 0);
    const float4* other = share(worker + 1, t) + q * 32 + lane;
    uint32_t sc[4];
    row_scales(nb, q, sc);
    constexpr int kStep = kWqThreads / 128, kBatch = 3;    // (column block, half) pairs per round of the quadrant's warps; rounds with their loads in flight
#pragma unroll 1
    for (int it0 = warp >> 2; it0 < NT / 8; it0 += kStep * kBatch) {
      float4 w[kBatch][2];
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const float4* src = other + min(it0 + j * kStep, NT / 8 - 1) * 256;
        w[j][0] = __ldcg(src), w[j][1] = __ldcg(src + 128);
      }
#pragma unroll
      for (int j = 0; j < kBatch; ++j) {
        const int it = it0 + j * kStep, h = it & 1, c = (it >> 1) * 16;
        if (it >= NT / 8) break;
        uint32_t v[8], v2[8];
        float f[8];
        wq_ld_16x256b_x2(dcol + ((uint32_t)(16 * h) << 16) + c, v);
        if (two) wq_ld_16x256b_x2(dcol + ((uint32_t)(16 * h) << 16) + 64 + c, v2);
        wq_ld_wait();
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = two ? __uint_as_float(v[i]) + __uint_as_float(v2[i]) : __uint_as_float(v[i]);
        f[0] += w[j][0].x, f[1] += w[j][0].y, f[2] += w[j][0].z, f[3] += w[j][0].w;
        f[4] += w[j][1].x, f[5] += w[j][1].y, f[6] += w[j][1].z, f[7] += w[j][1].w;
        to_stage(q, c, h, f, sc);
      }
    }
    __syncthreads();
    copy_out(nb, mt, threadIdx.x, kWqThreads);
    __syncthreads();
  }

  // ---- teardown: nobody touches tensor memory any more ----
  if (*dead != 0) {
    grid_dependency_wait();  // (whoever had y before)
    for (int t = u0 / KU; t <= (u1 - 1) / KU; ++t) {
      const int nb = t / p.MT, m0 = (t - nb * p.MT) * NT, rows = min(NT, p.M - m0);
      const int64_t nbase = ((int64_t)nb * kRanks + rank) * 128;
      for (int i = threadIdx.x; i < rows * 128; i += kWqThreads) {
        const int64_t n = nbase + (i & 127);
        if (n < p.N_out) p.y[(int64_t)(m0 + (i >> 7)) * p.ldy + n] = __ushort_as_bfloat16((unsigned short)0x7FFF);
      }
    }
    for (int i = 0; i < 64; ++i) __nanosleep(100000);  // copies and MMAs of this CTA that are still in flight
  }
  wq_fence_before();
  __syncthreads();
  if constexpr (PAIR) asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
  if (warp == kWqMma) {
    wq_fence_after();
    if constexpr (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(512));
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tb), "r"(512));
  }
}

// ---- host ---------------------------------------------------------------------------------------------------------------
static int wq_sm_count() {
  static int n = 0;
  if (n == 0) {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    n = v > 0 ? v : kNumSMs;
  }
  return n;
}

// how one call is cut up; a pure function of the shape, so the workspace size is too
struct WqPlan {
  bool defer, pair, direct;
  int KW;  // 128 k per unit
  int NT, BR, MT, NB, KU, ranks, workers, quantum, base, rem;
  int64_t tiles, n_tickets;
  uint32_t x_bytes, x_sub;
  int64_t off_part, off_xt, bytes;  // [tickets][shares][staged activations]
};

static int kw_of(const WqPlan& w) { return !w.direct && w.NT <= kWqLongNT ? 2 : 1; }

// Small weights, up to 128 rows and a tile per SM: where an even deal leaves a worker fewer than ten units of 256 k, tiles are not cut where it happens to fall, if
// it costs less, but each goes to so many owners, with equally many of its units each (KU may grow by an eighth, of zeros, to divide).  The number of owners per tile; 0:
// dealt evenly.  In units, a worker that holds pieces of two tiles pays 10 to 13 beside its own (two drains, two shares out, tickets, and the tile that it finishes);
// owners of one tile 5 (two or three pairs of CTAs 7), and the adding up of a share of NT rows for each of them; one owner nothing.  (One unit takes an owner as long as two, which
// go to its two sets of dequant warps.)  us, units of 128 k evenly / of 256 k evenly / as here: int4, 17 rows, 4096 x 256 6.0 / 7.2 / 5.8, x 768 9.4 / 13.1 / 7.0, x 1280 11.4 /
// 13.8 / 8.0, x 2816 13.4 / 15.0 / 11.2, x 4096 14.7 / 13.5 / 11.6, 14336 x 1024 12.9 / 12.2 / 8.2, 128 rows, 4096 x 256 9.0 / 11.8 / 9.0, 8192 x 768 16.4 / 18.6 / 10.9, x 2304
// 20.4 / 20.2 / 15.9, 4096 x 4096 23.2 / 21.7 / 18.3; int8, 17 rows, 1024 x 768 9.7 / 14.2 / 7.2, 4096 x 2304 13.7 / 14.9 / 11.8, 100 rows 14336 x 2816 25.0 / 25.3 / 19.6; 8 rows with
// a residual, int4 4096 x 768 8.9 / 10.2 / 5.7.  Of 900 sizes of 17 to 128 rows 6 are 2 to 6 % slower than with units of 128 k, most of them int8 and dealt evenly; beyond ten units a
// worker an even deal was not slower than those (whole tiles are faster up to a tile per worker there too: int4 14336 x 4096, 128 rows 26.5 / 22.0, not taken here).
static int wq_owners(WqPlan& w, int sms) {
  if (w.KW != 2 || w.tiles > sms || w.tiles * w.KU >= 10 * (int64_t)sms) return 0;
  int64_t best = 160 * ((w.tiles * w.KU + sms - 1) / sms + (w.tiles * w.KU < 4 * (int64_t)sms ? 13 : 10));   // in 160ths of a unit
  int owners = 0, units = w.KU;
  for (int ku = w.KU; ku <= w.KU + (w.KU + 7) / 8; ++ku) {
    for (int s = 1; s <= ku && w.tiles * s <= sms; ++s) {
      const int64_t cost = s == 1 ? 160 * ku : 160 * (ku / s > 2 ? ku / s : 2) + (w.pair && s < 4 ? 1120 : 800) + s * (w.NT > 32 ? w.NT : 32);
      if (ku % s == 0 && cost < best) best = cost, owners = s, units = ku;
    }
  }
  w.KU = units;
  return owners;
}

static bool wq_plan(int64_t M, int64_t Np, int64_t Kp, bool int4, WqPlan& w) {
  if (M <= 0 || Np % 128 != 0 || Kp % 64 != 0 || M > ((int64_t)1 << 24)) return false;
  w.defer = int4 && M <= 16;
  w.pair = M > 32;
  w.ranks = w.pair ? 2 : 1;
  w.MT = (int)((M + 255) / 256);
  w.NT = (int)(((M + w.MT - 1) / w.MT + 15) / 16 * 16);
  // Staging takes time by M x K, reading in place (the weights turned round among the lanes) by the units, M x K x N.  Staged / in place, us: int8
  // 4096 x 14336, 1000 rows 102.4 / 97.5, 700 rows 74.8 / 72.1; int4 4096 x 14336, 700 / 1000 rows 72.0 / 67.3, 97.8 / 92.4; 6144 x 4096 and 4096 x 4096, 700 rows
  // 41.5 / 39.2, 34.9 / 33.4; int8 8192 x 8192, 2048 rows 217.5 / 215; but int4 14336 x 4096, 700 and 2048 rows 65.2 / 65.6, 166.4 / 166.3; 300 rows of 4096 x 14336
  // 40.6 / 42.7, 64 rows of 28672 x 8192 51.4 / 58.8, where the lanes' turn lengthens the way from a unit's weights to its product.  So it is with tiles of
  // fewer rows, whose products no longer cover the turn: int8 8192 x 8192, 528 / 600 rows (tiles of 176 / 208) 58.2 / 64.3, 66.5 / 70.5, 640 (224) 69.6 / 72.4, 700 (240)
  // 76.7 / 76.9, 4096 x 4096, 800 (208) 1.02 times, 640 (224) 0.98, 2048 x 8192, 528 0.99; int4 8192 x 8192, 528 1.03, 560 (192) 1.01, 4096 x 14336, 528 0.99
  const int64_t most = int4 ? (w.NT < 192 ? kWqDirectN / 2 : kWqDirectN) : (w.NT < 224 ? kWqDirectN / 4 : (w.NT < 240 ? kWqDirectN / 2 : kWqDirectN));
  w.direct = M >= kWqDirectRows && Np <= most;
  w.BR = w.NT / w.ranks;
  w.KW = kw_of(w);
  w.KU = (int)((Kp + 128 * w.KW - 1) / (128 * w.KW));
  w.NB = (int)((Np + 128 * w.ranks - 1) / (128 * w.ranks));
  w.tiles = (int64_t)w.NB * w.MT;
  if (w.tiles * w.KU > 2000000000) return false;
  const int sms = wq_sm_count() / w.ranks;
  w.quantum = w.tiles >= (int64_t)kWqMaxSplitTiles * sms ? w.KU : 1;
  int64_t parts = w.tiles * w.KU / w.quantum;
  w.workers = (int)(w.quantum > 1 ? sms : (parts / 2 < sms ? (parts + 1) / 2 : sms));
  const bool shared = w.quantum == 1;
  if (const int owners = wq_owners(w, sms)) {
    if (owners == 1) w.quantum = w.KU;
    parts = w.tiles * w.KU / w.quantum;
    w.workers = (int)w.tiles * owners;
  }
  w.base = (int)(parts / w.workers);
  w.rem = (int)(parts % w.workers);
  w.n_tickets = shared ? w.tiles * w.ranks : 0;
  w.x_sub = (uint32_t)w.BR * 256 + (w.defer ? 4 * 64 : 0);  // (the sums' space is that of the smallest group)
  w.x_bytes = w.KW * w.x_sub;
  auto up = [](int64_t v) { return (v + 255) / 256 * 256; };
  w.off_part = up(w.n_tickets * 4);
  w.off_xt = w.off_part + (!shared ? 0 : up((int64_t)w.workers * 2 * w.ranks * w.NT * 512));
  w.bytes = w.off_xt + up((int64_t)w.MT * w.ranks * w.KU * w.x_bytes);
  // (DIRECT too, where nobody writes the copy as a rule, 29 MB of 68 at int8 4096 x 14336, 1000 rows: wq_gemm may stage all the same.  The size is that of these rows;
  // fewer may need more, as shares go by NT: int4 4096 x 4096, 256 rows 41 MB, 257 rows 24 MB.)
  return true;
}

using WqEncode = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                              CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
static WqEncode wq_encode_fn() {
  static WqEncode fn = []() -> WqEncode {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) return nullptr;
    return reinterpret_cast<WqEncode>(p);
  }();
  return fn;
}
// rows of `row_bytes`, `pitch` apart (0: one behind the other), read in boxes of 8 rows x box elements
// or of box_rows, then swizzled as rows of 128 bytes
static bool wq_map(CUtensorMap* map, CUtensorMapDataType type, int elem, const void* base, int64_t row_bytes, int64_t rows, int box, int64_t pitch = 0,
                   int box_rows = 0) {
  const cuuint64_t dims[2] = {(cuuint64_t)(row_bytes / elem), (cuuint64_t)rows}, strides[1] = {(cuuint64_t)(pitch ? pitch : row_bytes)};
  const cuuint32_t boxes[2] = {(cuuint32_t)box, (cuuint32_t)(box_rows ? box_rows : 8)}, steps[2] = {1, 1};
  auto encode = [&]() {
    return wq_encode_fn()(map, type, 2, const_cast<void*>(base), dims, strides, boxes, steps, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          box_rows ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_NONE,
                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
  };
  if (encode()) return true;
  // a host thread that has not called the runtime yet has no current context, which the driver's encoder asks for
  int dev = 0;
  return cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess && encode();
}

// rings in shared and tensor memory of a call with groups of G (0: int8), a function of its plan too
struct WqRings {
  int n_mma, x_slots, w_slots, a_slots;
  uint32_t off_x, off_w, w_slot;  // activation ring, weight ring, bytes of a slot of weights
  bool early;
};
constexpr size_t kWqBudget = 226 * 1024;

static WqRings wq_rings(const WqPlan& w, int G) {
  WqRings r;
  r.n_mma = w.NT <= 64 ? 2 : 1;
  r.w_slot = (uint32_t)(w.KW * (8 * 2 * (G == 0 ? 1024 : 512) + (G == 0 ? 0 : 8 * (G < 128 ? 128 / G : 1) * 64)));
  // tiles of x in flight (an L2 round trip is about 850 clocks; DEFER: as many as there are accumulators); what they and the
  // output tile leave of shared memory holds weights in flight
  // (even where two MMA warps alternate)
  if (w.KW == 2) r.x_slots = w.x_bytes > 24 * 1024 ? 3 : (w.x_bytes > 9 * 1024 || (w.defer && G == 64) ? 4 : (w.defer && G == 32 ? 2 : 6));
  else r.x_slots = w.x_bytes > 24 * 1024 ? 3 : 5;   // (144 rows and more: 18 KB at least)
  const size_t unit = w.direct ? 1024 : 16;    // (rows of 128 swizzled bytes: eight of them have to lie as the hardware counts)
  r.off_x = (uint32_t)((kWqHeader + (size_t)w.NT * kWqPitch + unit - 1) / unit * unit);
  r.off_w = (uint32_t)((r.off_x + (size_t)r.x_slots * w.x_bytes + 127) / 128 * 128);
  r.w_slots = (int)((kWqBudget - r.off_w) / r.w_slot);
  if (r.w_slots > kWqMaxW) r.w_slots = kWqMaxW;
  if (r.n_mma == 2) r.w_slots &= ~1;           // two MMA warps let the two dequant sets drift apart: each set keeps slots of its own
  r.a_slots = w.KW == 2 ? kWqSlots / 2 : (r.w_slots == 3 ? 3 : kWqSlots);   // (see a_first in the kernel)
  // The last tile from the accumulators where every CTA has a tile's worth of units, so that a tile has two owners as a rule: 4096 x 4096, 2048 rows
  // 63.9 -> 57.1 us; 14336 x 4096 int4, 300 / 1000 rows 39.8 -> 36.2 / 94.0 -> 89.3; 28672 x 4096 int8, 32 / 77 / 300 rows 32.4 -> 30.9 / 37.7 -> 34.9 /
  // 74.6 -> 70.9.  With less a CTA its neighbour is not there yet or it has several, and the mere presence of the code costs 0.2 to 0.5 us
  // (14336 x 4096, 77 rows: 25.6 -> 25.8; 4096 x 4096 int8, 200 rows: 28.5 -> 29.0).
  r.early = !w.defer && (int64_t)w.base * w.quantum >= w.KU;
  return r;
}

template <int G, bool DEFER, bool PAIR, bool DIRECT, int KW>
static int wq_launch(WqParams& p, const WqPlan& w, cudaStream_t s) {
  const WqRings r = wq_rings(w, G);
  p.n_mma = r.n_mma;
  p.x_slots = r.x_slots;
  p.w_slots = r.w_slots;
  p.a_slots = r.a_slots;
  p.off_x = r.off_x;
  p.off_w = r.off_w;
  const size_t smem = r.off_w + (size_t)r.w_slots * r.w_slot;
  const bool early = r.early;
  auto kern = wq_gemm_kernel<G, DEFER, PAIR, DIRECT, false, KW>;
  static OncePerDevice once[2];
  if (early) kern = wq_gemm_kernel<G, DEFER, PAIR, DIRECT, !DEFER, KW>;
  if (!dynamic_smem(once[early], kern, (int)kWqBudget)) return AO_B200_ERR_CUDA;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(w.workers * w.ranks));
  cfg.blockDim = dim3(kWqThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = 2;
  at[1].val.clusterDim.y = 1;
  at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = PAIR ? 2 : 1;
  return cudaLaunchKernelEx(&cfg, kern, p) == cudaSuccess ? AO_B200_OK : AO_B200_ERR_CUDA;
}

template <int SEG>
static int wq_stage(const void* x, int64_t M, int64_t Kx, int64_t ldx, const WqPlan& w, uint8_t* xt, uint32_t* tickets, bool settled, cudaStream_t s) {
  const int ku = w.KU * w.KW;  // (whole units)
  const int64_t pieces = (int64_t)w.MT * w.ranks * (w.BR / 8) * ku;
  if (pieces > 0x7fffffff) return AO_B200_ERR_UNSUPPORTED;   // (2 KB of activations each)
  int64_t grid = (pieces + kStageThreads / 32 - 1) / (kStageThreads / 32);
  if (grid > 148 * 32) grid = 148 * 32;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kStageThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, stage_x_kernel<SEG>, static_cast<const __nv_bfloat16*>(x), M, Kx, ldx, (uint32_t)pieces, w.BR, ku, w.x_sub, xt, tickets,
                            (int)w.n_tickets, settled) == cudaSuccess
             ? AO_B200_OK
             : AO_B200_ERR_CUDA;
}

static int wq_clear(uint32_t* tickets, int64_t n, bool settled, cudaStream_t s) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)(n > 148 * kStageThreads ? 148 : (n + kStageThreads - 1) / kStageThreads + (n == 0)));
  cfg.blockDim = dim3(kStageThreads);
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, clear_tickets_kernel, tickets, (int)n, settled) == cudaSuccess ? AO_B200_OK : AO_B200_ERR_CUDA;
}

// x [M][ldx] bf16 (first Kx columns valid), y [M][ldy] bf16.  G == 0: int8 weights (`sz` is then the bf16 per-row scale)
static int wq_gemm(const void* x, int64_t M, int64_t Kx, int64_t ldx, const void* packed, const void* sz, int64_t Np, int64_t Kp, int G, void* y,
                   int64_t N_out, int64_t ldy, const void* residual, int64_t ld_res, void* workspace, int64_t workspace_bytes, cudaStream_t s) {
  WqPlan w;
  if (!wq_plan(M, Np, Kp, G != 0, w) || wq_encode_fn() == nullptr) return AO_B200_ERR_UNSUPPORTED;
  if (workspace == nullptr || workspace_bytes < w.bytes || !ao_aligned(workspace, 16)) return AO_B200_ERR_WORKSPACE;
  auto* ws = static_cast<uint8_t*>(workspace);
  WqParams p;
  const bool ok = G ? wq_map(&p.wmap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, packed, Kp * 8, Np / 16, 256) &&
                          wq_map(&p.smap, CU_TENSOR_MAP_DATA_TYPE_UINT32, 4, sz, Kp / G * 64, Np / 16, (G < 128 ? 128 / G : 1) * 16)
                    : wq_map(&p.wmap, CU_TENSOR_MAP_DATA_TYPE_INT64, 8, packed, Kp * 16, Np / 16, 256);
  if (!ok) return AO_B200_ERR_UNSUPPORTED;
  // Results may be written over the activations: then they are staged first (there is room: wq_plan), as where they are no tensor that the copy engine takes
  const auto x0 = reinterpret_cast<uintptr_t>(x), y0 = reinterpret_cast<uintptr_t>(y);
  const bool apart = x0 + ((M - 1) * ldx + Kx) * 2 <= y0 || y0 + ((M - 1) * ldy + N_out) * 2 <= x0;
  w.direct = w.direct && apart && wq_map(&p.xmap, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, x, Kx * 2, M, 64, ldx * 2, w.BR);
  p.tickets = reinterpret_cast<uint32_t*>(ws);
  p.part = reinterpret_cast<float*>(ws + w.off_part);
  p.xt = ws + w.off_xt;
  // about two seconds; the variable is there for the test of what a wait that runs out leaves behind
  static const long long limit = []() { const char* e = std::getenv("AO_B200_GEMM_WAIT_CLOCKS"); return e ? std::atoll(e) : 4000000000ll; }();
  p.wait_limit = limit;
  p.scale8 = G ? nullptr : static_cast<const __nv_bfloat16*>(sz);
  p.y = static_cast<__nv_bfloat16*>(y);
  p.N_out = N_out;
  p.ldy = ldy;
  p.residual = static_cast<const __nv_bfloat16*>(residual);
  p.ld_res = ld_res;
  p.vec_store = (ldy % 8 == 0 && ao_aligned(y, 16) && ld_res % 8 == 0 && ao_aligned(residual, 16)) ? 1 : 0;
  p.M = (int)M;
  p.Kp = (int)Kp;
  p.packed = static_cast<const uint32_t*>(packed);
  p.sz = static_cast<const uint32_t*>(sz);
  p.NT = w.NT;
  p.BR = w.BR;
  p.KU = w.KU;
  p.MT = w.MT;
  p.x_bytes = w.x_bytes;
  p.x_sub = w.x_sub;
  p.quantum = w.quantum;
  p.base = w.base;
  p.rem = w.rem;
  // Staging and GEMM go into the stream as neighbours: another thread's call on the same stream may use the same workspace, and
  // the host is free to run it between the two launches.
  static std::mutex together;
  std::lock_guard<std::mutex> lock(together);
  const bool settled = residual != nullptr;  // (ao_b200_mm_residual's contract)
  int rc;
  if (w.direct) rc = wq_clear(p.tickets, w.n_tickets, settled, s);
  else if (!w.defer) rc = wq_stage<0>(x, M, Kx, ldx, w, ws + w.off_xt, p.tickets, settled, s);
  else if (G == 32) rc = wq_stage<32>(x, M, Kx, ldx, w, ws + w.off_xt, p.tickets, settled, s);
  else if (G == 64) rc = wq_stage<64>(x, M, Kx, ldx, w, ws + w.off_xt, p.tickets, settled, s);
  else rc = wq_stage<128>(x, M, Kx, ldx, w, ws + w.off_xt, p.tickets, settled, s);
  if (rc != AO_B200_OK) return rc;
  switch (G) {
    case 0:
      if (w.direct) return wq_launch<0, false, true, true, 1>(p, w, s);
      if (w.KW == 2) return w.pair ? wq_launch<0, false, true, false, 2>(p, w, s) : wq_launch<0, false, false, false, 2>(p, w, s);
      return wq_launch<0, false, true, false, 1>(p, w, s);
#define AO_WQ(GG)                                                                                                              \
  case GG:                                                                                                                     \
    if (w.direct) return wq_launch<GG, false, true, true, 1>(p, w, s);                                                         \
    if (w.defer) return wq_launch<GG, true, false, false, 2>(p, w, s);                                                         \
    if (w.KW == 2) return w.pair ? wq_launch<GG, false, true, false, 2>(p, w, s) : wq_launch<GG, false, false, false, 2>(p, w, s); \
    return wq_launch<GG, false, true, false, 1>(p, w, s);
    AO_WQ(32)
    AO_WQ(64)
    AO_WQ(128)
    AO_WQ(256)
#undef AO_WQ
  }
  return AO_B200_ERR_UNSUPPORTED;
}

// bytes of the workspace for M rows (0: shape not handled by this kernel).  Its contents need not survive between calls.
int64_t int4_gemm_tc_workspace_bytes(int64_t M, int64_t Np, int64_t Kp) {
  WqPlan w;
  return wq_plan(M, Np, Kp, true, w) ? w.bytes : 0;
}
int64_t int8_gemm_tc_workspace_bytes(int64_t M, int64_t Np, int64_t Kp) {
  WqPlan w;
  return wq_plan(M, Np, Kp, false, w) ? w.bytes : 0;
}
// how a call of M rows is cut up (ao_b200_mm_plan)
bool gemm_tc_plan(int64_t M, int64_t Np, int64_t Kp, int G, ao_b200_mm_cut& c) {
  WqPlan w;
  if (!wq_plan(M, Np, Kp, G != 0, w)) return false;
  const WqRings r = wq_rings(w, G);
  c.rows_per_tile = w.NT;
  c.row_tiles = w.MT;
  c.tiles = w.tiles;
  c.unit_k = 128 * w.KW;
  c.units_per_tile = w.KU;
  c.pair = w.pair;
  c.defer = w.defer;
  c.in_place = w.direct;
  c.workers = w.workers;
  c.quantum = w.quantum;
  c.base = w.base;
  c.rem = w.rem;
  c.weight_slots = r.w_slots;
  c.activation_slots = r.x_slots;
  c.operand_slots = r.a_slots;
  c.issuers = r.n_mma;
  c.early = r.early;
  return true;
}

int int4_gemm_tc(const void* x, int64_t M, int64_t Kx, int64_t ldx, const void* packed, const void* sz, int64_t Np, int64_t Kp, int G, void* y,
                 int64_t N_out, int64_t ldy, const void* residual, int64_t ld_res, void* workspace, int64_t workspace_bytes, cudaStream_t s) {
  if (!(G == 32 || G == 64 || G == 128 || G == 256)) return AO_B200_ERR_UNSUPPORTED;
  return wq_gemm(x, M, Kx, ldx, packed, sz, Np, Kp, G, y, N_out, ldy, residual, ld_res, workspace, workspace_bytes, s);
}

// int8 weights: packed = strip-major biased int8 (Np % 128 == 0), scale bf16 [N_out]
int int8_gemm_tc(const void* x, int64_t M, int64_t Kx, int64_t ldx, const void* packed, const void* scale, int64_t Np, int64_t Kp, void* y, int64_t N_out,
                 int64_t ldy, const void* residual, int64_t ld_res, void* workspace, int64_t workspace_bytes, cudaStream_t s) {
  return wq_gemm(x, M, Kx, ldx, packed, scale, Np, Kp, 0, y, N_out, ldy, residual, ld_res, workspace, workspace_bytes, s);
}

}  // namespace ao
