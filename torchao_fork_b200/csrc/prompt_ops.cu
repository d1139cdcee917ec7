// What the Llama block does between its products for rows of a prompt, one pass each: rotation of queries and keys, SiLU * up (the
// norm is rmsnorm_kernel of decode_ops.cu).  As tensor operations these were ten passes and more over fp32 copies: 700 tokens through two
// Mistral-7B layers and the output product took 1956 us of which about 850 were such passes, now 1036 in all.  Bound by memory;
// 16 bytes per thread.  Each is launched while the kernel in front ends (launch_early) and waits for it
// before anything else: that forward 949 -> 918 us.  The roundings are those of the single operations: fp32 products rounded before they are added (no fused
// multiply-add), silu rounded to bf16 before its product.
#include <cassert>

#include <cuda_bf16.h>

#include "../../include/ao_b200.h"
#include "common.cuh"

namespace ao {
namespace {

__device__ __forceinline__ float lo_f(uint32_t v) { return __uint_as_float(v << 16); }
__device__ __forceinline__ float hi_f(uint32_t v) { return __uint_as_float(v & 0xFFFF0000u); }
__device__ __forceinline__ uint32_t pack_rn(float a, float b) { return float_to_bf16_bits(a) | (float_to_bf16_bits(b) << 16); }

__device__ __forceinline__ uint32_t rotate_pair(uint32_t x, uint32_t cs) {
  const float a = lo_f(x), b = hi_f(x), c = lo_f(cs), s = hi_f(cs);
  return pack_rn(__fsub_rn(__fmul_rn(a, c), __fmul_rn(b, s)), __fadd_rn(__fmul_rn(b, c), __fmul_rn(a, s)));
}
// x [B][T][H][8 n8] (any strides that are whole 16-byte pieces) -> y, packed; freqs [T][8 n8]: cos, sin of every pair
__global__ void __launch_bounds__(256) rotary_kernel(const uint4* __restrict__ x, int64_t sb, int64_t st, int64_t sh, const uint4* __restrict__ freqs,
                                                     uint4* __restrict__ y, int T, int H, int n8, int64_t total) {
  grid_dependency_wait();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= total) return;
  const int c = (int)(i % n8);
  const int64_t r = i / n8;
  const int h = (int)(r % H);
  const int64_t bt = r / H;
  const int t = (int)(bt % T);
  const uint4 v = x[bt / T * sb + t * st + h * sh + c], f = freqs[(int64_t)t * n8 + c];
  y[i] = make_uint4(rotate_pair(v.x, f.x), rotate_pair(v.y, f.y), rotate_pair(v.z, f.z), rotate_pair(v.w, f.w));
}

// Keys and values of a prompt into the cache: k rotated on the way, both to the rows pos[t] of [B][H][S][8 n8].  As a rotation into a buffer and two
// indexed stores (each with index arithmetic of its own) this was 27 us a layer for 700 tokens of 8 heads; what has to move takes 2.
__global__ void __launch_bounds__(256) kv_rows_kernel(const uint4* __restrict__ k, int64_t kb, int64_t kt, int64_t kh, const uint4* __restrict__ v, int64_t vb,
                                                      int64_t vt, int64_t vh, const uint4* __restrict__ freqs, const void* __restrict__ pos, bool pos64,
                                                      uint4* __restrict__ k_cache, uint4* __restrict__ v_cache, int T, int H, int S, int n8, int64_t total) {
  grid_dependency_wait();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= total) return;
  const int c = (int)(i % n8);
  const int64_t r = i / n8;
  const int h = (int)(r % H);
  const int64_t bt = r / H, b = bt / T;
  const int t = (int)(bt % T);
  int64_t p = pos64 ? static_cast<const int64_t*>(pos)[t] : static_cast<const int32_t*>(pos)[t];
  if (p < 0) p += S;
  assert(p >= 0 && p < S);  // a position that the cache does not have ends the program, as an indexed store does
  if (p < 0 || p >= S) return;
  const uint4 x = k[b * kb + t * kt + h * kh + c], f = freqs[(int64_t)t * n8 + c];
  const int64_t at = ((b * H + h) * S + p) * n8 + c;
  k_cache[at] = make_uint4(rotate_pair(x.x, f.x), rotate_pair(x.y, f.y), rotate_pair(x.z, f.z), rotate_pair(x.w, f.w));
  v_cache[at] = v[b * vb + t * vt + h * vh + c];
}
// Each key and value head for all query heads that share it, [heads][head] -> [heads][rep][head]: read once, both in one launch (two copies
// that read a head rep times: 19 us a layer for 704 positions of 8 heads, rep 4; 11.5 MB to write).
__global__ void __launch_bounds__(256) repeat_heads_kernel(const uint4* __restrict__ k, const uint4* __restrict__ v, uint4* __restrict__ k_out,
                                                           uint4* __restrict__ v_out, int64_t head, int64_t total, int rep) {
  grid_dependency_wait();
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= total) return;
  const uint4 x = (blockIdx.y == 0 ? k : v)[i];
  uint4* out = (blockIdx.y == 0 ? k_out : v_out) + i / head * head * rep + i % head;
  for (int r = 0; r < rep; ++r) out[r * head] = x;
}

__device__ __forceinline__ float silu_f(float g) { return __uint_as_float(float_to_bf16_bits(g / (1.f + expf(-g))) << 16); }
__device__ __forceinline__ uint32_t silu_mul_pair(uint32_t g, uint32_t u) { return pack_rn(silu_f(lo_f(g)) * lo_f(u), silu_f(hi_f(g)) * hi_f(u)); }
__global__ void __launch_bounds__(256) silu_mul_rows_kernel(const uint4* __restrict__ gate, const uint4* __restrict__ up, uint4* __restrict__ y, int64_t n8) {
  grid_dependency_wait();
  grid_launch_dependents();   // (a kernel that follows programmatically waits before it reads)
  const int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (i >= n8) return;
  const uint4 g = gate[i], u = up[i];
  y[i] = make_uint4(silu_mul_pair(g.x, u.x), silu_mul_pair(g.y, u.y), silu_mul_pair(g.z, u.z), silu_mul_pair(g.w, u.w));
}

}  // namespace
}  // namespace ao

extern "C" int ao_b200_rotary(const void* x, int64_t stride_b, int64_t stride_t, int64_t stride_h, const void* freqs_cis, void* y, int64_t B, int64_t T,
                              int64_t H, int64_t head_dim, void* stream) {
  AO_CHECK_ARG(x && freqs_cis && y && B > 0 && T > 0 && H > 0 && head_dim > 0 && head_dim % 8 == 0);
  AO_CHECK_ARG(stride_b % 8 == 0 && stride_t % 8 == 0 && stride_h % 8 == 0 && ao_aligned(x, 16) && ao_aligned(freqs_cis, 16) && ao_aligned(y, 16));
  const int64_t total = B * T * H * (head_dim / 8), blocks = (total + 255) / 256;
  if (T > 2147483647 || H > 2147483647 || blocks > 2147483647) return AO_B200_ERR_UNSUPPORTED;
  return ao::launch_early(ao::rotary_kernel, dim3((unsigned)blocks), 256, stream,
      static_cast<const uint4*>(x), stride_b / 8, stride_t / 8, stride_h / 8, static_cast<const uint4*>(freqs_cis), static_cast<uint4*>(y), (int)T, (int)H,
      (int)(head_dim / 8), total);
}

extern "C" int ao_b200_kv_rows(const void* k, int64_t k_stride_b, int64_t k_stride_t, int64_t k_stride_h, const void* v, int64_t v_stride_b, int64_t v_stride_t,
                               int64_t v_stride_h, const void* freqs_cis, const void* pos, int pos_bytes, void* k_cache, void* v_cache, int64_t B,
                               int64_t T, int64_t H, int64_t S, int64_t head_dim, void* stream) {
  AO_CHECK_ARG(k && v && freqs_cis && pos && k_cache && v_cache && B > 0 && T > 0 && H > 0 && S > 0 && head_dim > 0 && head_dim % 8 == 0);
  AO_CHECK_ARG(k_stride_b % 8 == 0 && k_stride_t % 8 == 0 && k_stride_h % 8 == 0 && v_stride_b % 8 == 0 && v_stride_t % 8 == 0 && v_stride_h % 8 == 0);
  AO_CHECK_ARG(ao_aligned(k, 16) && ao_aligned(v, 16) && ao_aligned(freqs_cis, 16) && ao_aligned(k_cache, 16) && ao_aligned(v_cache, 16));
  AO_CHECK_ARG((pos_bytes == 4 || pos_bytes == 8) && ao_aligned(pos, pos_bytes));
  const int64_t total = B * T * H * (head_dim / 8), blocks = (total + 255) / 256;
  if (T > 2147483647 || H > 2147483647 || S > 2147483647 || blocks > 2147483647) return AO_B200_ERR_UNSUPPORTED;
  return ao::launch_early(ao::kv_rows_kernel, dim3((unsigned)blocks), 256, stream,
      static_cast<const uint4*>(k), k_stride_b / 8, k_stride_t / 8, k_stride_h / 8, static_cast<const uint4*>(v), v_stride_b / 8, v_stride_t / 8, v_stride_h / 8,
      static_cast<const uint4*>(freqs_cis), pos, pos_bytes == 8, static_cast<uint4*>(k_cache), static_cast<uint4*>(v_cache), (int)T, (int)H, (int)S, (int)(head_dim / 8), total);
}

extern "C" int ao_b200_repeat_heads(const void* k, const void* v, void* k_out, void* v_out, int64_t heads, int64_t head_elements, int64_t rep, void* stream) {
  AO_CHECK_ARG(k && v && k_out && v_out && heads > 0 && head_elements > 0 && head_elements % 8 == 0 && rep > 0);
  AO_CHECK_ARG(ao_aligned(k, 16) && ao_aligned(v, 16) && ao_aligned(k_out, 16) && ao_aligned(v_out, 16));
  const int64_t head = head_elements / 8, total = heads * head, blocks = (total + 255) / 256;
  if (rep > 2147483647 || blocks > 2147483647) return AO_B200_ERR_UNSUPPORTED;
  return ao::launch_early(ao::repeat_heads_kernel, dim3((unsigned)blocks, 2), 256, stream,
      static_cast<const uint4*>(k), static_cast<const uint4*>(v), static_cast<uint4*>(k_out), static_cast<uint4*>(v_out), head, total, (int)rep);
}

extern "C" int ao_b200_silu_mul_rows(const void* gate, const void* up, void* y, int64_t count, void* stream) {
  AO_CHECK_ARG(gate && up && y && count > 0 && count % 8 == 0 && ao_aligned(gate, 16) && ao_aligned(up, 16) && ao_aligned(y, 16));
  const int64_t n8 = count / 8, blocks = (n8 + 255) / 256;
  if (blocks > 2147483647) return AO_B200_ERR_UNSUPPORTED;
  return ao::launch_early(ao::silu_mul_rows_kernel, dim3((unsigned)blocks), 256, stream, static_cast<const uint4*>(gate), static_cast<const uint4*>(up),
                          static_cast<uint4*>(y), n8);
}
