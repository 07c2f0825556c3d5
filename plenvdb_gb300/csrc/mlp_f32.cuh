// The FP32 rgbnet kernels (mlp_f32.cu) as the rgbnet dispatch (mlp.cu) calls them.
#pragma once
#include "pvdb_internal.cuh"

namespace pvdb {

struct MlpArgs {
  const float* w0; const float* b0;
  const float* w1; const float* b1;
  const float* w2; const float* b2;
  int c0, dpe, din;  // din = c0 + dpe
};

// Flat parameter layout shared with the train step and the Python side:
// [w0 (128 x din), b0 (128), w1 (128 x 128), b1 (128), w2 (3 x 128), b2 (3)].
__host__ __device__ inline int64_t mlp_param_count(int din) {
  return int64_t(128) * din + 128 + 128 * 128 + 128 + 3 * 128 + 3;
}

// Row tiles of the FP32 kernels over `units` CTAs (or groups): `full` rounds of
// 128-row tiles, tile t to unit t % units, then 32-row tiles from row32. The
// remainder takes a further round of 128-row tiles when it would need more than
// three rounds of 32-row tiles.
struct TilePlan {
  int64_t full;
  int64_t row32;
};
__device__ __forceinline__ TilePlan tile_plan(int64_t M, int64_t units) {
  TilePlan p;
  const int64_t rounds = M / (128 * units);
  p.full = rounds * units;
  const int64_t rem = M - p.full * 128;
  if (rem > 3 * 32 * units) p.full += (rem + 127) / 128;
  p.row32 = p.full * 128;
  return p;
}

// CTAs of a backward's grid that have a row tile, and so a partial weight
// gradient (the others write none): the first ones.
__device__ __forceinline__ int active_parts(int64_t M, int grid, bool tensor_cores) {
  int64_t n;
  if (tensor_cores) {
    n = (M + 127) / 128;
  } else {
    const TilePlan p = tile_plan(M, grid);
    n = p.row32 < M ? (M - p.row32 + 31) / 32 : 0;
    n = p.full > n ? p.full : n;
  }
  return int(n < grid ? n : grid);
}

// rows: k0 [M, c0], ray [M], M = totals[1]; hpe [rays, 128]: the per-ray part
// of layer 0; out [M, 3]: sigmoid of the logits, times rw [M] when given.
int mlp_f32_forward(const MlpArgs& a, const float* k0, const int32_t* ray, const float* hpe,
                    const uint32_t* totals, float* out, const float* rw, cudaStream_t st);

// grad_k0 [M, c0] and per-CTA partial weight gradients wpart [grid][param count]
// in the flat layout; pe [rays, 32]: the per-ray PE.
int mlp_f32_backward(const MlpArgs& a, const float* k0, const int32_t* ray, const float* hpe,
                     const float* pe, const uint32_t* totals, const float* rgb,
                     const float* grad_rgb, float* grad_k0, float* wpart, int grid,
                     cudaStream_t st);

}  // namespace pvdb
