// What the two kernels behind ao_lm_window_attention_prompt share: lm_window_attention_tc.cu (tcgen05, the shapes of win_tc_ok) and
// lm_window_attention_mma.cu (mma.sync, the others).
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

namespace lm {

constexpr int kTcRows = 128;   // query rows of a tile of the tcgen05 kernel

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

// d and dv multiples of 16 (win_prompt_ok) up to 128: what fits two CTAs per SM, in shared memory and in tensor memory
inline bool win_tc_ok(int n_maps, int d, int dv) { return (n_maps == 1 || n_maps == 2) && d <= 128 && dv <= 128; }
int launch_win_tc(const WinPromptArgs& a, int n_maps, int dv, int n_tiles, cudaStream_t st);

}  // namespace lm
