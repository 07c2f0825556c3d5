// Merged-VDB renderer (MGRenderer, plenvdb.h:933-1068; renderer.cu:122-424).
//
// Data: an index leaf store (voxel -> row id, 0 = empty; the voxels with a row
// are the active ones) plus per-row density and k0 features (FP32, or BF16
// features with FP32 density). Loading lays the density out per voxel of the
// allocated leaves, and 12-channel features too (if there is memory for them),
// with one more record that holds row 0 (every voxel outside the leaves): a
// trilinear corner is then one load at its slot, not a row id and a load behind it.
//
// Per frame:
//   k_render_march         a warp per 32 pixels: get_rays (renderer.cu:122-167)
//                          in the unit-cube frame, t += steplen before each
//                          sample, skip when isActive(rint(xyz)) is false,
//                          index-grid trilinear density (int() truncation,
//                          renderer.cu:271-300), raw2alpha, both thresholds,
//                          early stop at a colour sample once T < t_stop
//                          (renderer.cu:240-266); appends each colour sample's
//                          position, weight and pixel to the frame's rows
//   k_render_pe / k_render_x (BF16), k_render_k0 (FP32)
//                          per row: the trilinear features (renderer.cu:303-310)
//                          into the rgbnet's X tiles or k0 rows; with BF16
//                          features the BF16 rgbnet gathers them itself
//   rgbnet                 the MLP on all rows (PE part once per pixel), each
//                          row's w/(1+exp(-logit))
//   k_render_composite     per pixel: T*bg + the sum of its rows in sample
//                          order (final_render renderer.cu:112-119,
//                          deterministic instead of atomics); bg alone when the
//                          pixel has no colour sample (renderer.cu:325-329).
// The reference marches twice, counting the samples first. Here the rows need
// no order among the pixels: a warp takes rows from a counter for every batch
// of samples it has finished and links its batches, and the composite walks
// them. Where a row lies varies from run to run; its value and the order a
// pixel's rows are added in do not. A frame with more rows than the buffers
// hold is marched again after they have grown.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "pvdb_internal.cuh"
#include "render_rows.cuh"
#include "tc.cuh"

namespace pvdb {

struct MlpArgs {
  const float* w0; const float* b0;
  const float* w1; const float* b1;
  const float* w2; const float* b2;
  int c0, dpe, din;
};
int mlp_forward_rows(const MlpArgs& a, const float* k0rows, const int32_t* ray,
                     const float* viewdirs, int R, const uint32_t* need, const uint32_t* totals,
                     int64_t max_rows, const float* rw, float* out, float* hpe_buf, int precision,
                     void** blob, size_t* blob_cap, void** xt, size_t* xt_cap, uint32_t* err,
                     cudaStream_t st);
int mlp_tc_forward_gather(const float* w0, const float* b0, const float* w1, const float* b1,
                          const float* w2, const float* b2, int c0, int dpe, const RowSource& src,
                          const uint32_t* totals, float* out, const float* rw, void** blob,
                          size_t* blob_cap, uint32_t* err, cudaStream_t st);

struct RenderP {
  int H, W, inverse_y;
  float K[9];
  float c2w[16];
  float mn[3], mx[3];
  float wsm1[3];
  float near_, far_, stepdist, shift, interval, thr, bg, t_stop;
  int dcol;
  // index store: nslots = nleaf * 512 voxel slots; record nslots of the
  // per-voxel arrays holds row 0
  // (the leaf table holds -d for a block with no leaf, d the Chebyshev distance
  // in blocks to the nearest leaf)
  GridView idx;               // topology; values unused
  int nslots;
  const float* vden;          // [nslots + 1]
  const float* vcol;          // [nslots + 1][12] (features per voxel, storage 0)
  const __nv_bfloat16* vcolh; // [nslots + 1][kHalfStride] (features per voxel, storage 1)
  const int32_t* rows;        // [nslots] row id of every in-leaf voxel (features in rows)
  const float* col;           // [N*dcol] (features in rows, storage 0)
  const __nv_bfloat16* colh;  // [N*dcol] (features in rows, storage 1)
  int storage;
};

// The colour samples one warp of the march finished together.
struct RenderBatch {
  uint32_t row0;    // first row; pixel l's rows follow those of the pixels before it
  int32_t next;     // the warp's next batch, -1: none
  uint8_t cnt[32];  // rows per pixel of the warp
};

struct RenderW {
  uint32_t* n;       // [HW] colour samples per pixel
  float* T;          // [HW]
  uint32_t* totals;  // [1] rows, [2] batches, [3] the rgbnet's given-up waits
  int32_t* head;     // [warps] first batch of each warp, -1: none
  RenderBatch* batch;  // [bcap]
  int64_t bcap;
  float* viewdirs;   // [HW*3] (pixels with colour samples)
  float* rk0;        // [cap*dcol]
  float* rw;         // [cap]
  float* rxyz;       // [cap*3] index-space position
  int32_t* rpix;     // [cap]
  int64_t cap;
};

// The ray of pixel n (get_rays, renderer.cu:134-151) in the unit-cube frame.
struct PixelRay {
  float rd[3], len, steplen;
  float o[3], d[3];
};
__device__ __forceinline__ void pixel_ray(const RenderP& P, int n, PixelRay& r) {
  const float pi = float(n % P.W) + 0.5f, pj = float(n / P.W) + 0.5f;
  float dir[3];
  dir[0] = __fdiv_rn(pi - P.K[2], P.K[0]);
  if (P.inverse_y) {
    dir[1] = __fdiv_rn(pj - P.K[5], P.K[4]);
    dir[2] = 1.f;
  } else {
    dir[1] = -__fdiv_rn(pj - P.K[5], P.K[4]);
    dir[2] = -1.f;
  }
  for (int a = 0; a < 3; ++a)
    r.rd[a] = __fmaf_rn(dir[2], P.c2w[4 * a + 2], __fmaf_rn(dir[1], P.c2w[4 * a + 1],
                                                            __fmul_rn(dir[0], P.c2w[4 * a])));
  r.len = sqrtf(__fmaf_rn(r.rd[2], r.rd[2],
                          __fmaf_rn(r.rd[1], r.rd[1], __fmul_rn(r.rd[0], r.rd[0]))));
  r.steplen = __fdiv_rn(P.stepdist, r.len);
  for (int a = 0; a < 3; ++a) {
    const float ext = P.mx[a] - P.mn[a];
    r.o[a] = __fdiv_rn(P.c2w[4 * a + 3] - P.mn[a], ext);
    r.d[a] = __fdiv_rn(r.rd[a], ext);
  }
}

// advance: t after n additions of step, each rounded. While t stays between
// two powers of two its ulp u is fixed, so every addition adds the same
// multiple of u, su = (t + step) - t, and m of them add m su exactly; the one
// exception is a step whose remainder is exactly half an ulp (ties go to the
// even neighbour), which takes the additions one by one, as does a t near the
// next power of two.
__device__ __forceinline__ float half_ulp(float t) {
  return __uint_as_float((__float_as_uint(t) & 0x7F800000u) - (24u << 23));
}
__device__ __forceinline__ float next_pow2(float t) {
  return __uint_as_float((__float_as_uint(t) & 0x7F800000u) + 0x00800000u);
}
__device__ __forceinline__ bool steps_exact(float t, float step, float su) {
  return t > 1e-20f && t < 1e20f && su > 0.f && fabsf(step - su) != half_ulp(t);
}
__device__ __forceinline__ float advance(float t, float step, int n) {
  while (n > 0) {
    float t1 = __fadd_rn(t, step);
    --n;
    const float su = t1 - t;
    if (n > 0 && steps_exact(t, step, su)) {
      const float room = (next_pow2(t) - t1) / su * 0.999f - 1.f;
      const int m = room < float(n) ? int(room) : n;
      if (m > 0) {
        t1 = __fmaf_rn(float(m), su, t1);
        n -= m;
      }
    }
    t = t1;
  }
  return t;
}

// A warp marches 8 x 4 pixels. Of a ray's samples, few are active (17 of 295 on
// the 160^3 benchmark scene), and an active one costs several times the test of
// an inactive one, so the two are kept apart: each lane tests its own pixel's
// samples and lists up to kListed active ones; the warp then evaluates the
// listed samples of all its pixels, a sample a lane; and each lane takes its
// alphas in order. Where no leaf is near, the march only advances t until
// shortly before the faces of the empty region.
// (One lane a pixel evaluating samples as it met them, and eight lanes a pixel,
// both took 600 us on the 800x800 benchmark frame.)
constexpr int kListed = 16;
constexpr int kTileW = 8, kTileH = 4;
// Tiles per block of the march and the composite: one, so that a block's slots
// are given back when its own tile ends (a 397x301 FP32 frame 2.37 -> 2.24 ms
// against four; 800x800 the same).
constexpr int kTileWarps = 1;
constexpr uint8_t kNoRow = 255;

struct MarchList {
  float t[kListed][32];
  float alpha[kListed][32];    // then the weight
  uint8_t rank[kListed][32];   // row within the pixel's rows of the batch
  uint16_t entry[kListed * 32];  // 32 * index + lane of the e-th listed sample
};

__global__ void __launch_bounds__(32 * kTileWarps)
    k_render_march(RenderP P, RenderW Wk) {
  __shared__ MarchList lists[kTileWarps];
  MarchList& L = lists[threadIdx.x >> 5];
  const int warp = blockIdx.x * kTileWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int tiles_x = (P.W + kTileW - 1) / kTileW, tiles = tiles_x * ((P.H + kTileH - 1) / kTileH);
  if (warp >= tiles) return;
  const int px = (warp % tiles_x) * kTileW + lane % kTileW,
            py = (warp / tiles_x) * kTileH + lane / kTileW;
  const bool in_image = px < P.W && py < P.H;
  const int n = in_image ? py * P.W + px : 0;
  PixelRay r;
  pixel_ray(P, n, r);
  const float steplen = r.steplen;
  // get_tminmax against the unit cube (renderer.cu:50-64)
  const float vx = r.d[0] == 0.f ? float(1e-6) : r.d[0];
  const float vy = r.d[1] == 0.f ? float(1e-6) : r.d[1];
  const float vz = r.d[2] == 0.f ? float(1e-6) : r.d[2];
  const float ax = __fdiv_rn(1.f - r.o[0], vx), ay = __fdiv_rn(1.f - r.o[1], vy),
              az = __fdiv_rn(1.f - r.o[2], vz);
  const float bx = __fdiv_rn(-r.o[0], vx), by = __fdiv_rn(-r.o[1], vy),
              bz = __fdiv_rn(-r.o[2], vz);
  const float tmin = fmaxf(fminf(fmaxf(fmaxf(fminf(ax, bx), fminf(ay, by)), fminf(az, bz)), P.far_), P.near_);
  const float tmax = fmaxf(fminf(fminf(fminf(fmaxf(ax, bx), fmaxf(ay, by)), fmaxf(az, bz)), P.far_), P.near_);
  // the reference loops while t < tmax; the iteration bound (the sample count
  // of the [tmin,tmax] chord plus slack) only guards against a step that no
  // longer advances t (non-finite or vanishing steplen)
  const float nsteps_f = (tmax - tmin) / steplen;
  const int max_it =
      in_image && nsteps_f > 0.f && nsteps_f < 1e6f ? int(nsteps_f) + 4 : 0;
  // skips: the inverse of the voxels advanced per step, and the most steps a
  // skip may take: t's rounding (at most tmax 2^-23 per addition) stays below
  // a quarter of a step
  float inv[3];
#pragma unroll
  for (int a = 0; a < 3; ++a) inv[a] = 1.f / (r.d[a] * P.wsm1[a] * steplen);
  const float most = fminf(0.25f * steplen / (tmax * 1.2e-7f), 4096.f);
  float T = 1.f;
  uint32_t cnt = 0;
  float t = tmin;
  int it = 0;
  int32_t last = -1;  // the warp's last batch
  bool stop = false;
  for (;;) {
    // this pixel's next active samples
    int c = 0;
    while (c < kListed && !stop && t < tmax && it < max_it) {
      t = __fadd_rn(t, steplen);
      ++it;
      float p[3], xyz[3];
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        p[a] = __fmaf_rn(t, r.d[a], r.o[a]);
        xyz[a] = __fmul_rn(p[a], P.wsm1[a]);
      }
      if ((0.f > p[0]) | (0.f > p[1]) | (0.f > p[2]) | (1.f < p[0]) | (1.f < p[1]) | (1.f < p[2]))
        continue;
      const int ri = __float2int_rn(xyz[0]), rj = __float2int_rn(xyz[1]),
                rk = __float2int_rn(xyz[2]);
      const int leaf = leaf_of(P.idx, ri, rj, rk);
      if (leaf < 0) {
        // every sample whose rounded position stays in the blocks nearer than
        // the nearest leaf is inactive: the steps that keep it 0.01 voxel
        // (above the rounding of xyz) and one step inside their outer faces
        float steps = most;
        const int b[3] = {ri & ~7, rj & ~7, rk & ~7};
        const float out = -8.f * float(leaf + 1);  // the further blocks, in voxels
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const float face = float(b[a]) + (inv[a] > 0.f ? 7.49f + out : -0.49f - out);
          const float s = (face - xyz[a]) * inv[a];
          if (s < steps) steps = s;  // (an axis that does not advance gives inf or NaN)
        }
        const int skip = int(fmaxf(steps, 0.f)) - 1;
        t = advance(t, steplen, skip);
        it += max(skip, 0);
        continue;
      }
      const int v = vox_offset(ri, rj, rk);
      if (!((__ldg(P.idx.mask + leaf * 8 + (v >> 6)) >> (v & 63)) & 1ull)) continue;
      L.t[c][lane] = t;
      ++c;
    }
    // the listed samples of all pixels, pixel after pixel
    int end = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += x;
    }
    const int total = __shfl_sync(0xffffffffu, end, 31);
    if (total == 0) break;  // every pixel is done
    for (int i = 0; i < c; ++i) L.entry[end - c + i] = uint16_t(32 * i + lane);
    __syncwarp();
    for (int e0 = 0; e0 < total; e0 += 32) {
      const int e = e0 + lane;
      const int en = L.entry[min(e, total - 1)], i = en >> 5, l = en & 31;
      const float dx = __shfl_sync(0xffffffffu, r.d[0], l),
                  dy = __shfl_sync(0xffffffffu, r.d[1], l),
                  dz = __shfl_sync(0xffffffffu, r.d[2], l);
      const float te = L.t[i][l];
      const float xyz[3] = {__fmul_rn(__fmaf_rn(te, dx, r.o[0]), P.wsm1[0]),
                            __fmul_rn(__fmaf_rn(te, dy, r.o[1]), P.wsm1[1]),
                            __fmul_rn(__fmaf_rn(te, dz, r.o[2]), P.wsm1[2])};
      int slot[8];
      float sc[8];
      cell_corners(P.idx, P.nslots, xyz, slot, sc);
      float val[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) val[q] = __ldg(P.vden + slot[q]);
      float sig = __fmul_rn(val[0], sc[0]);
#pragma unroll
      for (int q = 1; q < 8; ++q) sig = __fmaf_rn(val[q], sc[q], sig);
      const float alpha = 1.f - powf(1.f + expf(sig + P.shift), -P.interval);
      if (e < total) L.alpha[i][l] = alpha;
    }
    __syncwarp();
    // each pixel's samples in order
    int k = 0;
    for (int i = 0; i < c; ++i) {
      uint8_t rank = kNoRow;
      const float alpha = L.alpha[i][lane];
      if (!stop && !(alpha <= P.thr)) {
        const float w = T * alpha;
        T = T * (1.f - alpha);
        if (!(w <= P.thr)) {
          L.alpha[i][lane] = w;
          rank = uint8_t(k++);
          stop = T < P.t_stop;
        }
      }
      L.rank[i][lane] = rank;
    }
    cnt += k;
    // rows for the colour samples
    int kend = k;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, kend, o);
      if (lane >= o) kend += x;
    }
    const int rows = __shfl_sync(0xffffffffu, kend, 31);
    if (rows == 0) continue;
    uint32_t row0 = 0, id = 0;
    if (lane == 0) {
      row0 = atomicAdd(Wk.totals + 1, uint32_t(rows));
      id = atomicAdd(Wk.totals + 2, 1u);
    }
    row0 = __shfl_sync(0xffffffffu, row0, 0);
    id = __shfl_sync(0xffffffffu, id, 0);
    if (id < Wk.bcap) {
      RenderBatch& B = Wk.batch[id];
      B.cnt[lane] = uint8_t(k);
      if (lane == 0) {
        B.row0 = row0;
        B.next = -1;
        if (last >= 0)
          Wk.batch[last].next = int32_t(id);
        else
          Wk.head[warp] = int32_t(id);
        last = int32_t(id);
      }
    }
    __syncwarp();
    const int64_t m0 = int64_t(row0) + kend - k;  // this pixel's first row
    for (int e0 = 0; e0 < total; e0 += 32) {
      const int e = e0 + lane;
      const int en = L.entry[min(e, total - 1)], i = en >> 5, l = en & 31;
      const int64_t ml = __shfl_sync(0xffffffffu, m0, l);
      const float dx = __shfl_sync(0xffffffffu, r.d[0], l),
                  dy = __shfl_sync(0xffffffffu, r.d[1], l),
                  dz = __shfl_sync(0xffffffffu, r.d[2], l);
      const int nl = __shfl_sync(0xffffffffu, n, l);
      const uint8_t rank = L.rank[i][l];
      const int64_t m = ml + rank;
      if (e >= total || rank == kNoRow || m >= Wk.cap) continue;
      const float te = L.t[i][l];
      Wk.rw[m] = L.alpha[i][l];
      Wk.rpix[m] = nl;
      Wk.rxyz[m * 3] = __fmul_rn(__fmaf_rn(te, dx, r.o[0]), P.wsm1[0]);
      Wk.rxyz[m * 3 + 1] = __fmul_rn(__fmaf_rn(te, dy, r.o[1]), P.wsm1[1]);
      Wk.rxyz[m * 3 + 2] = __fmul_rn(__fmaf_rn(te, dz, r.o[2]), P.wsm1[2]);
    }
    __syncwarp();
  }
  if (lane == 0 && last < 0) Wk.head[warp] = -1;
  if (in_image) {
    Wk.n[n] = cnt;
    Wk.T[n] = T;
    if (cnt)
#pragma unroll
      for (int a = 0; a < 3; ++a) Wk.viewdirs[n * 3 + a] = __fdiv_rn(r.rd[a], r.len);
  }
}

// The trilinear features of row m (trigetColor, renderer.cu:303-310): per
// channel c0*s0, then the fma chain over corners 1..7, at the position the
// march had (same arithmetic). CT = 12: vector loads of the per-voxel records;
// 0: any channel count up to 16, by row id.
template <int CT>
__device__ __forceinline__ void row_features(const RenderP& P, const RenderW& Wk, int64_t m,
                                             float* acc) {
  const float xyz[3] = {__ldg(Wk.rxyz + m * 3), __ldg(Wk.rxyz + m * 3 + 1),
                        __ldg(Wk.rxyz + m * 3 + 2)};
  if (CT == 12 && P.storage == 1) {
    features12_bf16(P.idx, P.nslots, P.vcolh, xyz, acc);
    return;
  }
  int slot[8];
  float sc[8];
  cell_corners(P.idx, P.nslots, xyz, slot, sc);
  if (CT == 12) {
    {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const float4* src = reinterpret_cast<const float4*>(P.vcol + int64_t(slot[c]) * 12);
        float v[12];
#pragma unroll
        for (int b = 0; b < 3; ++b) *reinterpret_cast<float4*>(v + 4 * b) = __ldg(src + b);
#pragma unroll
        for (int q = 0; q < 12; ++q)
          acc[q] = c == 0 ? __fmul_rn(v[q], sc[0]) : __fmaf_rn(v[q], sc[c], acc[q]);
      }
    }
    return;
  }
  int32_t id[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) id[c] = slot[c] == P.nslots ? 0 : __ldg(P.rows + slot[c]);
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    if (q >= P.dcol) break;
    float a = 0.f;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int64_t e = int64_t(id[c]) * P.dcol + q;
      const float v = P.storage == 0 ? __ldg(P.col + e) : __bfloat162float(P.colh[e]);
      a = c == 0 ? __fmul_rn(v, sc[0]) : __fmaf_rn(v, sc[c], a);
    }
    acc[q] = a;
  }
}

// FP32 rgbnet: the k0 rows.
template <int CT>
__global__ void __launch_bounds__(256)
    k_render_k0(RenderP P, RenderW Wk, int64_t M) {
  const int64_t m = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (m >= M) return;
  float acc[CT ? CT : 16];
  row_features<CT>(P, Wk, m, acc);
  if (CT == 12) {
    float4* dst = reinterpret_cast<float4*>(Wk.rk0 + m * 12);
#pragma unroll
    for (int b = 0; b < 3; ++b)
      dst[b] = make_float4(acc[4 * b], acc[4 * b + 1], acc[4 * b + 2], acc[4 * b + 3]);
  } else {
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (q < P.dcol) Wk.rk0[m * P.dcol + q] = acc[q < (CT ? CT : 16) ? q : 0];
  }
}

// BF16 rgbnet: the pixel's part of its X rows ([0 (dcol) | PE | 1 | 0], 48
// BF16 columns), for the pixels with colour samples; one thread per 8 columns.
__global__ void __launch_bounds__(192)
    k_render_pe(RenderP P, RenderW Wk, int npe, uint4* pex) {
  const int64_t e = blockIdx.x * 192ll + threadIdx.x;
  const int n = int(e / 6), cb = int(e % 6);
  if (n >= P.H * P.W || Wk.n[n] == 0) return;
  const int dpe = 3 + 6 * npe;
  const float v[3] = {Wk.viewdirs[n * 3], Wk.viewdirs[n * 3 + 1], Wk.viewdirs[n * 3 + 2]};
  uint32_t w[4];
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    float x2[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int q = 8 * cb + 2 * h + u - P.dcol;  // PE component (dvgo.py:354-355)
      float x = q == dpe ? 1.f : 0.f;
      if (q >= 0 && q < 3) {
        x = q == 0 ? v[0] : q == 1 ? v[1] : v[2];
      } else if (q >= 3 && q < dpe) {
        const int qq = q - 3, cs = qq / (3 * npe), rem = qq - cs * 3 * npe, a = rem / npe,
                  i = rem - a * npe;
        const float f = (a == 0 ? v[0] : a == 1 ? v[1] : v[2]) * float(1 << i);
        x = cs ? cosf(f) : sinf(f);
      }
      x2[u] = x;
    }
    w[h] = tc::pack_bf16(x2[0], x2[1]);
  }
  pex[e] = make_uint4(w[0], w[1], w[2], w[3]);
}

// BF16 rgbnet: row m of the X tiles, the features beside the pixel's part. The
// padding rows of the last tile are zero.
template <int CT>
__global__ void __launch_bounds__(256)
    k_render_x(RenderP P, RenderW Wk, int64_t M, const uint4* __restrict__ pex, uint8_t* xt) {
  const int64_t m = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (m >= (M + 127) / 128 * 128) return;
  uint4 row[6];
#pragma unroll
  for (int cb = 0; cb < 6; ++cb) row[cb] = make_uint4(0u, 0u, 0u, 0u);
  if (m < M) {
    const int n = Wk.rpix[m];
#pragma unroll
    for (int cb = CT == 12 ? 1 : 0; cb < 6; ++cb) row[cb] = __ldg(pex + int64_t(n) * 6 + cb);
    float acc[CT ? CT : 16];
    row_features<CT>(P, Wk, m, acc);
    if (CT == 12) {
      row[0] = make_uint4(tc::pack_bf16(acc[0], acc[1]), tc::pack_bf16(acc[2], acc[3]),
                          tc::pack_bf16(acc[4], acc[5]), tc::pack_bf16(acc[6], acc[7]));
      row[1].x = tc::pack_bf16(acc[8], acc[9]);
      row[1].y = tc::pack_bf16(acc[10], acc[11]);
    } else {
      uint32_t* w = reinterpret_cast<uint32_t*>(row);
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        if (q >= P.dcol) continue;
        const uint32_t b = tc::pack_bf16(acc[q < (CT ? CT : 16) ? q : 0], 0.f) & 0xFFFFu;
        w[q >> 1] = q & 1 ? (w[q >> 1] & 0x0000FFFFu) | (b << 16) : (w[q >> 1] & 0xFFFF0000u) | b;
      }
    }
  }
  uint8_t* tile = xt + (m >> 7) * int64_t(kRgbXTile);
#pragma unroll
  for (int cb = 0; cb < 6; ++cb)
    *reinterpret_cast<uint4*>(tile + tc::kmaj(int(m & 127), 8 * cb, kRgbXK)) = row[cb];
}

// A warp per warp of the march, a lane per pixel: adds the pixel's rows batch
// after batch, in sample order (part [M, 3]: the rows' contributions). A batch's
// rows are contiguous and come through shared memory (lanes reading their own
// rows from global memory, 12 bytes apart, took 118 us of the 800x800 frame);
// the next batch's header travels meanwhile.
__global__ void __launch_bounds__(32 * kTileWarps)
    k_render_composite(RenderP P, RenderW Wk, const float* __restrict__ part, float* image) {
  __shared__ float bufs[kTileWarps][kListed * 32 * 3];
  float* buf = bufs[threadIdx.x >> 5];
  const int warp = blockIdx.x * kTileWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int tiles_x = (P.W + kTileW - 1) / kTileW, tiles = tiles_x * ((P.H + kTileH - 1) / kTileH);
  if (warp >= tiles) return;
  const int px = (warp % tiles_x) * kTileW + lane % kTileW,
            py = (warp / tiles_x) * kTileH + lane / kTileW;
  const bool in_image = px < P.W && py < P.H;
  const int64_t n = in_image ? int64_t(py) * P.W + px : 0;
  int32_t b = Wk.head[warp];
  float acc[3];
  acc[0] = acc[1] = acc[2] = in_image && Wk.n[n] ? __fmul_rn(Wk.T[n], P.bg) : P.bg;
  uint32_t cnt = 0, row0 = 0;
  int32_t next = -1;
  if (b >= 0) {
    cnt = Wk.batch[b].cnt[lane];
    row0 = Wk.batch[b].row0;
    next = Wk.batch[b].next;
  }
  while (b >= 0) {
    uint32_t cnt_n = 0, row0_n = 0;
    int32_t next_n = -1;
    if (next >= 0) {
      cnt_n = Wk.batch[next].cnt[lane];
      row0_n = Wk.batch[next].row0;
      next_n = Wk.batch[next].next;
    }
    uint32_t end = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint32_t x = __shfl_up_sync(0xffffffffu, end, o);
      if (lane >= o) end += x;
    }
    const uint32_t rows = __shfl_sync(0xffffffffu, end, 31);
    const float* src = part + int64_t(row0) * 3;
    for (uint32_t q0 = lane; q0 < rows * 3; q0 += 16 * 32) {
      float v[16];
#pragma unroll
      for (uint32_t e = 0; e < 16; ++e) v[e] = q0 + 32 * e < rows * 3 ? __ldg(src + q0 + 32 * e) : 0.f;
#pragma unroll
      for (uint32_t e = 0; e < 16; ++e)
        if (q0 + 32 * e < rows * 3) buf[q0 + 32 * e] = v[e];
    }
    __syncwarp();
    const float* mine = buf + (end - cnt) * 3;
    for (uint32_t q = 0; q < cnt; ++q)
#pragma unroll
      for (int c = 0; c < 3; ++c) acc[c] = __fadd_rn(acc[c], mine[3 * q + c]);
    __syncwarp();
    b = next;
    cnt = cnt_n;
    row0 = row0_n;
    next = next_n;
  }
  if (in_image)
#pragma unroll
    for (int c = 0; c < 3; ++c) image[n * 3 + c] = acc[c];
}

// Per-voxel records of the leaves from the rows (row id rows[s]; slot
// nleaf * 512: row 0): density, and 12-channel features in FP32 or BF16
// (nearest even).
__global__ void k_fill_voxels(int64_t nslots, const int32_t* __restrict__ rows,
                              const float* __restrict__ den, const float* __restrict__ col,
                              float* vden, float* vcol, __nv_bfloat16* vcolh) {
  const int64_t s = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (s > nslots) return;
  const int64_t id = s < nslots ? rows[s] : 0;
  vden[s] = den[id];
  if (vcol)
    for (int q = 0; q < 12; ++q) vcol[s * 12 + q] = col[id * 12 + q];
  if (vcolh)
    for (int q = 0; q < kHalfStride; ++q)
      vcolh[s * kHalfStride + q] = __float2bfloat16_rn(q < 12 ? col[id * 12 + q] : 0.f);
}

__global__ void k_to_bf16(const float* __restrict__ src, __nv_bfloat16* dst, int64_t n) {
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i < n) dst[i] = __float2bfloat16_rn(src[i]);
}

__global__ void k_fill_rows(GridView g, int32_t* rows, const int32_t* __restrict__ dense, int rx,
                            int ry, int rz) {
  const int64_t s = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (s >= int64_t(g.nleaf) * kLeafVox) return;
  const int leaf = int(s >> 9), v = int(s & 511);
  const int x = g.origin[leaf * 3] + (v >> 6), y = g.origin[leaf * 3 + 1] + ((v >> 3) & 7),
            z = g.origin[leaf * 3 + 2] + (v & 7);
  rows[s] = (x < rx && y < ry && z < rz) ? dense[(int64_t(x) * ry + y) * rz + z] : 0;
}

}  // namespace pvdb

using namespace pvdb;

struct pvdb_renderer_s {
  int dcol, dpe, dhid, dout;
  bool flags[5] = {false, false, false, false, false};
  pvdb_grid_s* topo = nullptr;
  // 12 channels: per-voxel features; other counts, or no memory for them (an index
  // whose voxels share rows has far more voxels than rows): row ids and rows
  bool voxels = false;
  int32_t* d_rows = nullptr;
  float* d_vden = nullptr;
  float* d_col = nullptr;           // rows, or the per-voxel records
  __nv_bfloat16* d_colh = nullptr;  // rows, or the per-voxel records
  int64_t nrows = 0;
  int storage = 0;
  float* d_params = nullptr;  // [w0 (dhid x din), b0, w1, b1, w2 (3 x dhid), b2]
  int reso[3] = {0, 0, 0};
  float K[9], xyz_min[3], xyz_max[3];
  float near_ = 0, far_ = 1e9f, stepdist = 0, shift = 0, interval = 0, thr = 0, bg = 0, t_stop = 1e-3f;
  int inverse_y = 0, H = 0, W = 0;
  float c2w[16];
  // frame buffers
  uint32_t* d_n = nullptr;
  int32_t* d_head = nullptr;
  RenderBatch* d_batch = nullptr;
  int64_t batch_cap = 0;
  float* d_T = nullptr;
  float* d_viewdirs = nullptr;
  float* d_hpe = nullptr;
  float* d_image = nullptr;
  uint32_t* d_totals = nullptr;
  float* d_rk0 = nullptr;
  float* d_rw = nullptr;
  float* d_rxyz = nullptr;
  int32_t* d_rpix = nullptr;
  float* d_part = nullptr;
  int64_t rows_cap = 0;
  void* d_packed = nullptr;  // BF16 weight tiles of the tensor-core rgbnet
  size_t packed_cap = 0;
  void* d_xt = nullptr;      // BF16 X tiles of the rows (tensor-core rgbnet)
  size_t xt_cap = 0;
};

// Test hook (pvdb_debug_render_exact): buffers of exactly what is asked for, one row
// and one batch at first, so that a small frame outgrows them.
static std::atomic<int> g_dbg_exact{0};

static int renderer_grow_batches(pvdb_renderer_s* r, int64_t need) {
  if (need <= r->batch_cap) return PVDB_OK;
  const int64_t cap = g_dbg_exact ? need : need + need / 4 + 4096;
  dev_free(r->d_batch);
  r->d_batch = nullptr;
  r->batch_cap = 0;
  const int rc = dev_alloc((void**)&r->d_batch, size_t(cap) * sizeof(RenderBatch));
  if (!rc) r->batch_cap = cap;
  return rc;
}

// The leaf table with -d in the blocks that have no leaf, d the Chebyshev
// distance in blocks to the nearest one (two passes over half of the 26
// neighbours each).
static std::vector<int32_t> leaf_distances(const pvdb_grid_s* g) {
  const int L[3] = {g->ldim[0], g->ldim[1], g->ldim[2]};
  std::vector<int32_t> t = g->h_table;
  const int32_t none = -(std::max(L[0], std::max(L[1], L[2])) + 1);
  for (int32_t& v : t)
    if (v < 0) v = none;
  auto at = [&](int x, int y, int z) -> int32_t& { return t[(int64_t(x) * L[1] + y) * L[2] + z]; };
  auto relax = [&](int x, int y, int z, int sign) {
    int32_t& v = at(x, y, z);
    if (v >= 0) return;
    for (int q = 0; q < 13; ++q) {  // the neighbours before this one in the pass's order
      const int dx = sign * (q / 9 - 1), dy = sign * (q / 3 % 3 - 1), dz = sign * (q % 3 - 1);
      const int a = x + dx, b = y + dy, c = z + dz;
      if (a < 0 || b < 0 || c < 0 || a >= L[0] || b >= L[1] || c >= L[2]) continue;
      const int32_t w = at(a, b, c);
      v = std::max(v, w >= 0 ? -1 : w - 1);
    }
  };
  for (int x = 0; x < L[0]; ++x)
    for (int y = 0; y < L[1]; ++y)
      for (int z = 0; z < L[2]; ++z) relax(x, y, z, 1);
  for (int x = L[0] - 1; x >= 0; --x)
    for (int y = L[1] - 1; y >= 0; --y)
      for (int z = L[2] - 1; z >= 0; --z) relax(x, y, z, -1);
  return t;
}

static int renderer_grow_rows(pvdb_renderer_s* r, int64_t need) {
  if (need <= r->rows_cap) return PVDB_OK;
  const int64_t cap = g_dbg_exact ? need : std::max<int64_t>(need + need / 4, 1 << 20);
  void* ptrs[] = {r->d_rk0, r->d_rw, r->d_rxyz, r->d_rpix, r->d_part};
  for (void* p : ptrs) dev_free(p);
  r->d_rk0 = r->d_rw = r->d_rxyz = r->d_part = nullptr;
  r->d_rpix = nullptr;
  r->rows_cap = 0;
  int rc;
  if ((rc = dev_alloc((void**)&r->d_rk0, size_t(cap) * r->dcol * 4)) ||
      (rc = dev_alloc((void**)&r->d_rw, size_t(cap) * 4)) ||
      (rc = dev_alloc((void**)&r->d_rxyz, size_t(cap) * 12)) ||
      (rc = dev_alloc((void**)&r->d_rpix, size_t(cap) * 4)) ||
      (rc = dev_alloc((void**)&r->d_part, size_t(cap) * 12)))
    return rc;
  r->rows_cap = cap;
  return PVDB_OK;
}

// The status word of the rgbnet's bounded waits was set: some rows of that frame
// were not written. Cleared once it is reported.
static int wait_gave_up(pvdb_renderer_s* r, cudaStream_t st) {
  PVDB_CHECK_CUDA(cudaMemsetAsync(r->d_totals + 3, 0, 4, st));
  return set_error(PVDB_ERR_TIMEOUT,
                   "a tensor-core MMA wait timed out: the last rendered image is incomplete");
}

extern "C" {

int pvdb_debug_render_exact(int on) {
  g_dbg_exact.store(on);
  return PVDB_OK;
}

int pvdb_renderer_create(int32_t dcol, int32_t dpe, int32_t dhid, int32_t dout,
                         pvdb_renderer* out) {
  clear_error();
  PVDB_REQUIRE(out, "null argument");
  PVDB_REQUIRE(dcol > 0 && dcol <= 16, "dcol must be in 1..16");
  PVDB_REQUIRE(dpe == 3 || dpe == 9 || dpe == 15 || dpe == 21 || dpe == 27,
               "dpe must be 3*(1+2*pe) with pe in 0..4");
  PVDB_REQUIRE(dhid == 128, "dhid must be 128");
  PVDB_REQUIRE(dout == 3, "dout must be 3");
  pvdb_renderer_s* r = new pvdb_renderer_s();
  r->dcol = dcol;
  r->dpe = dpe;
  r->dhid = dhid;
  r->dout = dout;
  const size_t P = size_t(dhid) * (dcol + dpe) + dhid + size_t(dhid) * dhid + dhid + 3 * dhid + 3;
  int rc = dev_alloc((void**)&r->d_params, P * 4);
  if (!rc) rc = dev_alloc((void**)&r->d_totals, 64);
  if (!rc) {
    const cudaError_t e = cudaMemset(r->d_totals, 0, 64);
    if (e != cudaSuccess) rc = cuda_error(e, "renderer create");
  }
  if (rc) {
    pvdb_renderer_destroy(r);
    return rc;
  }
  *out = r;
  return PVDB_OK;
}

int pvdb_renderer_destroy(pvdb_renderer r) {
  if (!r) return PVDB_OK;
  pvdb_grid_destroy(r->topo);
  void* ptrs[] = {r->d_rows, r->d_vden, r->d_col, r->d_colh, r->d_params, r->d_n, r->d_head,
                  r->d_T, r->d_viewdirs, r->d_hpe, r->d_image, r->d_totals, r->d_batch,
                  r->d_rk0, r->d_rw, r->d_rxyz, r->d_rpix, r->d_part, r->d_packed, r->d_xt};
  for (void* p : ptrs) dev_free(p);
  delete r;
  return PVDB_OK;
}

int pvdb_renderer_load_data(pvdb_renderer r, const int32_t reso[3], const int32_t* index,
                            const float* density, const float* features, int64_t n_rows,
                            int32_t storage, int32_t mem) {
  clear_error();
  PVDB_REQUIRE(r && reso && index && density && features, "null argument");
  PVDB_REQUIRE(n_rows >= 1, "n_rows must be >= 1 (row 0 is the empty row)");
  PVDB_REQUIRE(storage == 0 || storage == 1, "storage must be 0 (FP32) or 1 (BF16 features)");
  const int64_t nvox = int64_t(reso[0]) * reso[1] * reso[2];
  std::vector<int32_t> idx_host;
  const int32_t* idx = index;
  if (mem == PVDB_MEM_DEVICE) {
    idx_host.resize(nvox);
    PVDB_CHECK_CUDA(cudaMemcpy(idx_host.data(), index, nvox * 4, cudaMemcpyDeviceToHost));
    idx = idx_host.data();
  }
  std::vector<uint8_t> active(nvox);
  for (int64_t q = 0; q < nvox; ++q) {
    PVDB_REQUIRE(idx[q] >= 0 && idx[q] < n_rows, "index row out of range");
    active[q] = idx[q] > 0;
  }
  pvdb_grid_destroy(r->topo);
  r->topo = nullptr;
  r->flags[0] = false;  // until everything below is in place
  int rc = pvdb_grid_create_from_mask(reso, 1, 0.f, active.data(), PVDB_MEM_HOST, &r->topo);
  if (rc) return rc;
  {
    const std::vector<int32_t> table = leaf_distances(r->topo);
    PVDB_CHECK_CUDA(cudaMemcpy(r->topo->d_table, table.data(), table.size() * 4,
                               cudaMemcpyHostToDevice));
  }
  dev_free(r->d_rows);
  dev_free(r->d_vden);
  dev_free(r->d_col);
  dev_free(r->d_colh);
  r->d_rows = nullptr;
  r->d_vden = r->d_col = nullptr;
  r->d_colh = nullptr;
  const int64_t ns = r->topo->nslots();
  const size_t nf = size_t(n_rows) * r->dcol;
  // device copies of the inputs, freed on every way out
  struct Temp {
    int32_t *dense = nullptr, *rows = nullptr;
    float *den = nullptr, *col = nullptr;
    ~Temp() {
      dev_free(dense);
      dev_free(rows);
      dev_free(den);
      dev_free(col);
    }
  } tmp;
  if ((rc = dev_alloc((void**)&tmp.rows, std::max<int64_t>(ns, 1) * 4)) ||
      (rc = dev_alloc((void**)&tmp.dense, nvox * 4)) ||
      (rc = dev_alloc((void**)&tmp.den, n_rows * 4)) ||
      (rc = dev_alloc((void**)&tmp.col, nf * 4)) ||
      (rc = dev_alloc((void**)&r->d_vden, (ns + 1) * 4)))
    return rc;
  bool voxels = r->dcol == 12;
  for (;;) {
    if (storage == 0)
      rc = dev_alloc((void**)&r->d_col, voxels ? size_t(ns + 1) * 48 : nf * 4);
    else
      rc = dev_alloc((void**)&r->d_colh, voxels ? size_t(ns + 1) * kHalfStride * 2 : nf * 2);
    if (!rc) break;
    if (!voxels || rc != PVDB_ERR_NOMEM) return rc;
    clear_error();
    voxels = false;
  }
  r->voxels = voxels;
  const cudaMemcpyKind kind = mem == PVDB_MEM_DEVICE ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  PVDB_CHECK_CUDA(cudaMemcpy(tmp.dense, index, nvox * 4, kind));
  PVDB_CHECK_CUDA(cudaMemcpy(tmp.den, density, n_rows * 4, kind));
  PVDB_CHECK_CUDA(cudaMemcpy(tmp.col, features, nf * 4, kind));
  if (ns) {
    k_fill_rows<<<ceil_div(ns, 256), 256>>>(r->topo->view(), tmp.rows, tmp.dense, reso[0], reso[1],
                                            reso[2]);
    PVDB_CHECK_LAUNCH("k_fill_rows");
  }
  k_fill_voxels<<<ceil_div(ns + 1, 256), 256>>>(ns, tmp.rows, tmp.den, tmp.col, r->d_vden,
                                                voxels ? r->d_col : nullptr,
                                                voxels ? r->d_colh : nullptr);
  PVDB_CHECK_LAUNCH("k_fill_voxels");
  if (!voxels) {
    if (storage == 0) {
      PVDB_CHECK_CUDA(cudaMemcpy(r->d_col, tmp.col, nf * 4, cudaMemcpyDeviceToDevice));
    } else {
      k_to_bf16<<<ceil_div(nf, 256), 256>>>(tmp.col, r->d_colh, int64_t(nf));
      PVDB_CHECK_LAUNCH("k_to_bf16");
    }
    r->d_rows = tmp.rows;
    tmp.rows = nullptr;
  }
  PVDB_CHECK_CUDA(cudaDeviceSynchronize());
  r->nrows = n_rows;
  r->storage = storage;
  for (int a = 0; a < 3; ++a) r->reso[a] = reso[a];
  r->flags[0] = true;
  return PVDB_OK;
}

int pvdb_renderer_load_params(pvdb_renderer r, const float* w0, const float* b0, const float* w1,
                              const float* b1, const float* w2, const float* b2) {
  clear_error();
  PVDB_REQUIRE(r && w0 && b0 && w1 && b1 && w2 && b2, "null argument");
  const int din = r->dcol + r->dpe, H = r->dhid;
  // the reference takes [in,out] row-major (run.py:98-104); store nn.Linear [out,in]
  std::vector<float> flat;
  flat.reserve(size_t(H) * din + H + size_t(H) * H + H + 3 * H + 3);
  for (int o = 0; o < H; ++o)
    for (int i = 0; i < din; ++i) flat.push_back(w0[size_t(i) * H + o]);
  flat.insert(flat.end(), b0, b0 + H);
  for (int o = 0; o < H; ++o)
    for (int i = 0; i < H; ++i) flat.push_back(w1[size_t(i) * H + o]);
  flat.insert(flat.end(), b1, b1 + H);
  for (int o = 0; o < 3; ++o)
    for (int i = 0; i < H; ++i) flat.push_back(w2[size_t(i) * 3 + o]);
  flat.insert(flat.end(), b2, b2 + 3);
  PVDB_CHECK_CUDA(cudaMemcpy(r->d_params, flat.data(), flat.size() * 4, cudaMemcpyHostToDevice));
  r->flags[1] = true;
  return PVDB_OK;
}

int pvdb_renderer_set_scene(pvdb_renderer r, const int32_t reso[3], const float K[9],
                            const float xyz_min[3], const float xyz_max[3]) {
  clear_error();
  PVDB_REQUIRE(r && reso && K && xyz_min && xyz_max, "null argument");
  for (int a = 0; a < 3; ++a) {
    r->reso[a] = reso[a];
    r->xyz_min[a] = xyz_min[a];
    r->xyz_max[a] = xyz_max[a];
  }
  std::memcpy(r->K, K, sizeof(r->K));
  r->flags[2] = true;
  return PVDB_OK;
}

int pvdb_renderer_set_kwargs(pvdb_renderer r, float near_, float far_, float stepdist,
                             float act_shift, float interval, float fast_color_thres, float bg,
                             int32_t inverse_y, int32_t h, int32_t w, float t_stop) {
  clear_error();
  PVDB_REQUIRE(r, "null renderer");
  PVDB_REQUIRE(h > 0 && w > 0 && int64_t(h) * w < (int64_t(1) << 31), "bad image size");
  PVDB_REQUIRE(stepdist > 0.f, "stepdist must be positive");
  (void)far_;
  r->near_ = near_;
  r->far_ = 1e9f;  // plenvdb.h:1008
  r->stepdist = stepdist;
  r->shift = act_shift;
  r->interval = interval;
  r->thr = fast_color_thres;
  r->bg = bg;
  r->inverse_y = inverse_y;
  r->t_stop = t_stop;
  if (h != r->H || w != r->W || !r->d_n) {
    const size_t HW = size_t(h) * w;
    void* ptrs[] = {r->d_n, r->d_head, r->d_T, r->d_viewdirs, r->d_hpe, r->d_image};
    for (void* p : ptrs) dev_free(p);
    r->d_n = nullptr;
    r->d_head = nullptr;
    r->d_T = r->d_viewdirs = r->d_hpe = r->d_image = nullptr;
    r->flags[3] = false;  // no frame, and no size that a later call could keep,
    r->H = r->W = 0;      // until all of them are there again
    int rc;
    if ((rc = dev_alloc((void**)&r->d_n, HW * 4)) || (rc = dev_alloc((void**)&r->d_head,
                        size_t(ceil_div(w, kTileW)) * ceil_div(h, kTileH) * 4)) ||
        (rc = dev_alloc((void**)&r->d_T, HW * 4)) ||
        (rc = dev_alloc((void**)&r->d_viewdirs, HW * 12)) ||
        (rc = dev_alloc((void**)&r->d_hpe, HW * (128 + 32) * 4)) ||
        (rc = dev_alloc((void**)&r->d_image, HW * 12)))
      return rc;
    r->H = h;
    r->W = w;
  }
  r->flags[3] = true;
  return PVDB_OK;
}

int pvdb_renderer_input_c2w(pvdb_renderer r, const float* c2w, int32_t mem, pvdb_stream s) {
  clear_error();
  PVDB_REQUIRE(r && c2w, "null argument");
  if (mem == PVDB_MEM_DEVICE) {
    PVDB_CHECK_CUDA(cudaMemcpyAsync(r->c2w, c2w, 64, cudaMemcpyDeviceToHost, as_stream(s)));
    PVDB_CHECK_CUDA(cudaStreamSynchronize(as_stream(s)));
  } else {
    std::memcpy(r->c2w, c2w, 64);
  }
  r->flags[4] = true;
  return PVDB_OK;
}

int pvdb_renderer_render(pvdb_renderer r, int32_t precision, pvdb_stream s) {
  clear_error();
  PVDB_REQUIRE(r, "null renderer");
  for (int q = 0; q < 5; ++q)
    if (!r->flags[q])
      return set_error(PVDB_ERR_STATE,
                       "render needs load_data, load_params, setScene, setKwargs and input_a_c2w");
  PVDB_REQUIRE(precision == 0 || precision == 1, "precision must be 0 (FP32) or 1 (BF16 rgbnet)");
  cudaStream_t st = as_stream(s);
  RenderP P{};
  P.H = r->H;
  P.W = r->W;
  P.inverse_y = r->inverse_y;
  std::memcpy(P.K, r->K, sizeof(P.K));
  std::memcpy(P.c2w, r->c2w, sizeof(P.c2w));
  for (int a = 0; a < 3; ++a) {
    P.mn[a] = r->xyz_min[a];
    P.mx[a] = r->xyz_max[a];
    P.wsm1[a] = float(r->reso[a] - 1);
  }
  P.near_ = r->near_;
  P.far_ = r->far_;
  P.stepdist = r->stepdist;
  P.shift = r->shift;
  P.interval = r->interval;
  P.thr = r->thr;
  P.bg = r->bg;
  P.t_stop = r->t_stop;
  P.dcol = r->dcol;
  P.idx = r->topo->view();
  P.nslots = int(r->topo->nslots());
  P.vden = r->d_vden;
  P.rows = r->d_rows;
  P.vcol = P.col = r->d_col;
  P.vcolh = P.colh = r->d_colh;
  P.storage = r->storage;
  RenderW Wk{};
  Wk.n = r->d_n;
  Wk.T = r->d_T;
  Wk.totals = r->d_totals;
  Wk.head = r->d_head;
  Wk.viewdirs = r->d_viewdirs;
  const int HW = r->H * r->W;
  const int tiles = ceil_div(r->W, kTileW) * ceil_div(r->H, kTileH);
  prof_begin_call();
  prof_mark(st, 0);
  int rc = renderer_grow_rows(r, 1);
  if (!rc) rc = renderer_grow_batches(r, g_dbg_exact ? 1 : tiles);
  if (rc) return rc;
  uint32_t total = 0;
  for (;;) {
    Wk.rw = r->d_rw;
    Wk.rxyz = r->d_rxyz;
    Wk.rpix = r->d_rpix;
    Wk.cap = r->rows_cap;
    Wk.batch = r->d_batch;
    Wk.bcap = r->batch_cap;
    PVDB_CHECK_CUDA(cudaMemsetAsync(r->d_totals, 0, 12, st));
    k_render_march<<<ceil_div(tiles, kTileWarps), 32 * kTileWarps, 0, st>>>(P, Wk);
    PVDB_CHECK_LAUNCH("k_render_march");
    uint32_t tot[3] = {0, 0, 0};
    PVDB_CHECK_CUDA(cudaMemcpyAsync(tot, r->d_totals + 1, 12, cudaMemcpyDeviceToHost, st));
    PVDB_CHECK_CUDA(cudaStreamSynchronize(st));
    // (this frame's rgbnet has not run: the word is an earlier frame's)
    if (tot[2]) return wait_gave_up(r, st);
    total = tot[0];
    if (int64_t(tot[0]) <= r->rows_cap && int64_t(tot[1]) <= r->batch_cap) break;
    // the counts do not depend on the buffers: one more march holds them
    if ((rc = renderer_grow_rows(r, tot[0])) || (rc = renderer_grow_batches(r, tot[1]))) return rc;
  }
  prof_mark(st, 1);
  prof_mark(st, 2);
  Wk.rk0 = r->d_rk0;
  MlpArgs a;
  const int din = r->dcol + r->dpe, H = r->dhid;
  a.w0 = r->d_params;
  a.b0 = a.w0 + size_t(H) * din;
  a.w1 = a.b0 + H;
  a.b1 = a.w1 + size_t(H) * H;
  a.w2 = a.b1 + H;
  a.b2 = a.w2 + 3 * H;
  a.c0 = r->dcol;
  a.dpe = r->dpe;
  a.din = din;
  // 12 BF16 channels a voxel and the BF16 rgbnet: the rgbnet gathers the features itself
  const bool gather = precision == 1 && r->voxels && r->storage == 1;
  uint4* pex = reinterpret_cast<uint4*>(r->d_hpe);  // 96 of the 640 bytes a pixel
  if (total) {
    const int64_t M = total;
    const int rgrid = ceil_div((M + 127) / 128 * 128, 256);
    if (precision == 1) {
      k_render_pe<<<ceil_div(int64_t(HW) * 6, 192), 192, 0, st>>>(P, Wk, (r->dpe - 3) / 6, pex);
      PVDB_CHECK_LAUNCH("k_render_pe");
      if (!gather) {
        const int64_t ntiles = (r->rows_cap + 127) / 128;
        if ((rc = dev_reserve(&r->d_xt, &r->xt_cap, size_t(ntiles) * kRgbXTile))) return rc;
        uint8_t* xt = static_cast<uint8_t*>(r->d_xt);
        if (r->voxels)
          k_render_x<12><<<rgrid, 256, 0, st>>>(P, Wk, M, pex, xt);
        else
          k_render_x<0><<<rgrid, 256, 0, st>>>(P, Wk, M, pex, xt);
        PVDB_CHECK_LAUNCH("k_render_x");
      }
    } else {
      if (r->voxels)
        k_render_k0<12><<<rgrid, 256, 0, st>>>(P, Wk, M);
      else
        k_render_k0<0><<<rgrid, 256, 0, st>>>(P, Wk, M);
      PVDB_CHECK_LAUNCH("k_render_k0");
    }
  }
  prof_mark(st, 3);
  if (total && gather) {
    const RowSource src{P.idx, P.nslots, P.vcolh, r->d_rxyz, r->d_rpix, pex};
    rc = mlp_tc_forward_gather(a.w0, a.b0, a.w1, a.b1, a.w2, a.b2, a.c0, a.dpe, src, r->d_totals,
                               r->d_part, r->d_rw, &r->d_packed, &r->packed_cap, r->d_totals + 3,
                               st);
    if (rc) return rc;
  } else if (total) {
    rc = mlp_forward_rows(a, r->d_rk0, r->d_rpix, r->d_viewdirs, HW, r->d_n, r->d_totals,
                          r->rows_cap, r->d_rw, r->d_part, r->d_hpe, precision, &r->d_packed,
                          &r->packed_cap, &r->d_xt, &r->xt_cap, r->d_totals + 3, st);
    if (rc) return rc;
  }
  prof_mark(st, 4);
  k_render_composite<<<ceil_div(tiles, kTileWarps), 32 * kTileWarps, 0, st>>>(P, Wk, r->d_part,
                                                                               r->d_image);
  PVDB_CHECK_LAUNCH("k_render_composite");
  prof_mark(st, 5);
  return PVDB_OK;
}

int pvdb_renderer_output(pvdb_renderer r, float* out, int32_t mem, pvdb_stream s) {
  clear_error();
  PVDB_REQUIRE(r && out, "null argument");
  PVDB_REQUIRE(r->d_image, "no image rendered");
  const size_t bytes = size_t(r->H) * r->W * 12;
  cudaStream_t st = as_stream(s);
  PVDB_CHECK_CUDA(cudaMemcpyAsync(out, r->d_image, bytes,
                                  mem == PVDB_MEM_DEVICE ? cudaMemcpyDeviceToDevice
                                                         : cudaMemcpyDeviceToHost,
                                  st));
  if (mem == PVDB_MEM_HOST) {
    uint32_t status = 0;
    PVDB_CHECK_CUDA(cudaMemcpyAsync(&status, r->d_totals + 3, 4, cudaMemcpyDeviceToHost, st));
    PVDB_CHECK_CUDA(cudaStreamSynchronize(st));
    if (status) return wait_gave_up(r, st);
  }
  return PVDB_OK;
}

int pvdb_renderer_views(pvdb_renderer r, float** image, int32_t** n_samples_total) {
  clear_error();
  PVDB_REQUIRE(r, "null renderer");
  if (image) *image = r->d_image;
  if (n_samples_total) *n_samples_total = (int32_t*)(r->d_totals + 1);
  return PVDB_OK;
}

}  // extern "C"
