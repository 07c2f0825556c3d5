// The merged renderer's rows as the BF16 rgbnet reads them: trilinear features
// of a row from the per-voxel records, beside the pixel's part of its X row.
#pragma once
#include "pvdb_internal.cuh"
#include "tc.cuh"

namespace pvdb {

// 12-channel BF16 features per voxel of the allocated leaves; record nslots
// holds the empty row (every voxel outside them).
struct RowSource {
  GridView idx;                 // topology of the leaves
  int nslots;
  const __nv_bfloat16* colh;    // [nslots + 1][kHalfStride]
  const float* xyz;             // [M, 3] index-space positions
  const int32_t* pix;           // [M]
  const uint4* pex;             // [pixels][6]: the pixel's part of its X rows
};

// Slots of the 8 corners of the sample's cell (int() truncation,
// renderer.cu:271-300), nslots where a corner lies in no allocated leaf, and
// their scales.
__device__ __forceinline__ void cell_corners(const GridView& g, int nslots, const float xyz[3],
                                             int s[8], float sc[8]) {
  const int i = int(xyz[0]), j = int(xyz[1]), k = int(xyz[2]);
  corner_slots(g, i, j, k, s);
#pragma unroll
  for (int c = 0; c < 8; ++c) s[c] = s[c] < 0 ? nslots : s[c];
  corner_scales(xyz[0] - float(i), xyz[1] - float(j), xyz[2] - float(k), sc);
}

// Trilinear features from BF16 records (trigetColor, renderer.cu:303-310): per
// channel c0*s0, then the fma chain over corners 1..7; four corners in flight.
__device__ __forceinline__ void features12_bf16(const GridView& g, int nslots,
                                                const __nv_bfloat16* __restrict__ colh,
                                                const float xyz[3], float acc[12]) {
  int slot[8];
  float sc[8];
  cell_corners(g, nslots, xyz, slot, sc);
#pragma unroll
  for (int c0 = 0; c0 < 8; c0 += 4) {
    uint32_t w[4][8];
#pragma unroll
    for (int c = 0; c < 4; ++c) ld_nc32(colh + int64_t(slot[c0 + c]) * kHalfStride, w[c]);
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int q = 0; q < 12; ++q) {
        const float v = __uint_as_float(q & 1 ? w[c][q >> 1] & 0xFFFF0000u : w[c][q >> 1] << 16);
        acc[q] = c0 + c == 0 ? __fmul_rn(v, sc[0]) : __fmaf_rn(v, sc[c0 + c], acc[q]);
      }
  }
}

// A row's position and pixel; pixel -1 past the rows. Loaded well before the
// row is formed, since the feature loads wait for them (loaded in place, the
// forward over the 800x800 frame's rows took 921 us instead of 875).
struct RowPos {
  float xyz[3];
  int pix;
};
__device__ __forceinline__ RowPos load_row_pos(const RowSource& S, int64_t m, int64_t M) {
  RowPos r = {{0.f, 0.f, 0.f}, -1};
  if (m < M) {
#pragma unroll
    for (int a = 0; a < 3; ++a) r.xyz[a] = __ldg(S.xyz + m * 3 + a);
    r.pix = __ldg(S.pix + m);
  }
  return r;
}

// The row's X row ([k0 | PE | 1 | 0], 48 BF16 columns) as row `row` of the X
// tile at `tile`; zeros past the rows.
__device__ __forceinline__ void write_x_row(const RowSource& S, const RowPos& r, int row,
                                            uint8_t* tile) {
  uint4 c0 = make_uint4(0u, 0u, 0u, 0u), c1 = c0;
  const uint4* pe = S.pex + int64_t(max(r.pix, 0)) * 6;
  if (r.pix >= 0) {
    float acc[12];
    features12_bf16(S.idx, S.nslots, S.colh, r.xyz, acc);
    const uint4 p1 = __ldg(pe + 1);
    c0 = make_uint4(tc::pack_bf16(acc[0], acc[1]), tc::pack_bf16(acc[2], acc[3]),
                    tc::pack_bf16(acc[4], acc[5]), tc::pack_bf16(acc[6], acc[7]));
    c1 = make_uint4(tc::pack_bf16(acc[8], acc[9]), tc::pack_bf16(acc[10], acc[11]), p1.z, p1.w);
  }
  *reinterpret_cast<uint4*>(tile + tc::kmaj(row, 0, kRgbXK)) = c0;
  *reinterpret_cast<uint4*>(tile + tc::kmaj(row, 8, kRgbXK)) = c1;
#pragma unroll
  for (int cb = 2; cb < 6; ++cb)
    *reinterpret_cast<uint4*>(tile + tc::kmaj(row, 8 * cb, kRgbXK)) =
        r.pix >= 0 ? __ldg(pe + cb) : make_uint4(0u, 0u, 0u, 0u);
}

}  // namespace pvdb
