// rgbnet in FP32 (the plain method): Linear(C0+Dpe -> 128) ReLU
// Linear(128 -> 128) ReLU Linear(128 -> 3), sigmoid (dvgo.py:91-107, :354-362),
// on the CUDA cores. Layer 0 is split into the per-row k0 part and a per-ray
// part hpe = W0[:,C0:]·PE(viewdir) + b0 (mlp.cu).
//
// Both kernels are bound by the FP32 FMA rate (128 per clock and SM). Every
// operand is a [feature][row] or [n][k] tile in shared memory with a row
// stride of 4 mod 32 words, so that it can be read in 16-byte loads along
// either index: along the output index (four outputs of one reduction step)
// or along the reduction index (four steps of one output). A warp's lanes are
// laid out 4 x 8 over its output block, which makes each of these loads at
// most 128 distinct bytes in distinct banks: one shared-memory cycle per warp
// (measured), against 8 for the 32 lanes' FMAs on 4 x 8 outputs.
//
// Work is handed out in tiles of 128 rows while that fills every SM, and the
// rest (or a batch too small for one round) in tiles of 32 rows, whose chain
// of dependent phases is a quarter as long.
#include <algorithm>

#include "mlp_f32.cuh"

namespace pvdb {

namespace {

constexpr int kW = 128;        // hidden width
constexpr int kLd = kW + 4;    // row stride of a 128-wide tile (4 mod 32 words)
constexpr int kPeStride = 32;  // PE floats per ray

__device__ __forceinline__ void bar_group(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Two FP32 FMAs in one instruction (each rounded as fmaf): half the issue slots
// and register reads of two fmaf. Row pairs come packed from 16-byte loads, the
// other factor is duplicated. In the forward's product loop it reached 108
// against 103 FMAs per clock and SM; in the backward's, beside its resident
// accumulators, the duplicates spilled and cost what they gave.
typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ f32x2 dup2(float v) {
  f32x2 d;
  asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
  return d;
}
__device__ __forceinline__ void unpack2(f32x2 v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}

// One step of a reduce-scatter over lanes that differ in `mask`: the first
// N/2 entries of v become the sums of the half this lane keeps.
template <int N>
__device__ __forceinline__ void scatter_step(float* v, int mask, bool hi) {
#pragma unroll
  for (int i = 0; i < N / 2; ++i) {
    const float send = hi ? v[i] : v[i + N / 2];
    const float keep = hi ? v[i + N / 2] : v[i];
    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
  }
}

// k0 rows [row][4*CQ] (zero past c0 and past M) and ray ids (-1 past M) of a tile.
template <int TR, int CQ>
__device__ __forceinline__ void load_rows(float* x, int32_t* rays, int t, int nt, int c0,
                                          const float* __restrict__ k0,
                                          const int32_t* __restrict__ ray, int64_t row0,
                                          int64_t M) {
  for (int i = t; i < TR * 4 * CQ; i += nt) {
    const int rr = i / (4 * CQ), q = i % (4 * CQ);
    const int64_t m = row0 + rr;
    x[i] = m < M && q < c0 ? __ldg(k0 + m * c0 + q) : 0.f;
  }
  for (int i = t; i < TR; i += nt) rays[i] = row0 + i < M ? __ldg(ray + row0 + i) : -1;
}

// Layer 0: h0[n][row] = relu(hpe[ray][n] + sum_q w0k[q][n] x[row][q]), the sum
// in q order from hpe. Thread t: feature t % 128, the rows of part t / 128.
template <int TR, int CQ, int NT>
__device__ __forceinline__ void layer0(float* h0, int ld, const float* w0k, const float* x,
                                       const int32_t* rays, const float* __restrict__ hpe, int t) {
  const int n = t & (kW - 1);
  constexpr int kRows = TR / (NT / kW);
  const int r0 = (t / kW) * kRows;
  float w[4 * CQ];
#pragma unroll
  for (int q = 0; q < 4 * CQ; ++q) w[q] = w0k[q * kW + n];
  constexpr int kB = kRows < 16 ? kRows : 16;  // rows whose hpe loads are in flight together
#pragma unroll 1
  for (int r = r0; r < r0 + kRows; r += kB) {
    float z[kB];
#pragma unroll
    for (int i = 0; i < kB; ++i) {
      const int ry = rays[r + i];
      z[i] = ry >= 0 ? __ldg(hpe + int64_t(ry) * kW + n) : 0.f;
    }
#pragma unroll
    for (int i = 0; i < kB; ++i)
#pragma unroll
      for (int b = 0; b < CQ; ++b) {
        const float4 v = *reinterpret_cast<const float4*>(x + (r + i) * 4 * CQ + 4 * b);
        z[i] = fmaf(w[4 * b], v.x, z[i]);
        z[i] = fmaf(w[4 * b + 1], v.y, z[i]);
        z[i] = fmaf(w[4 * b + 2], v.z, z[i]);
        z[i] = fmaf(w[4 * b + 3], v.w, z[i]);
      }
#pragma unroll
    for (int i = 0; i < kB; i += 4)
      *reinterpret_cast<float4*>(h0 + n * ld + r + i) =
          make_float4(fmaxf(z[i], 0.f), fmaxf(z[i + 1], 0.f), fmaxf(z[i + 2], 0.f),
                      fmaxf(z[i + 3], 0.f));
  }
}

// w0k[q][n] = w0[n][q] for the k0 columns, zero past c0.
template <int CQ>
__device__ __forceinline__ void load_w0k(float* w0k, const MlpArgs& a, int t, int nt) {
  for (int i = t; i < 4 * CQ * kW; i += nt) {
    const int q = i / kW, n = i % kW;
    w0k[i] = q < a.c0 ? __ldg(a.w0 + n * a.din + q) : 0.f;
  }
}

// Four floats of W1, which may be a view into a parameter buffer at any offset: in
// one load (VEC) only where it lies on a 16-byte boundary, which the launch looks
// at. (A choice in the kernel moved its schedule: 160^3 FP32 step 741 -> 747 us.)
template <bool VEC>
__device__ __forceinline__ float4 w1_quad(const float* w1) {
  if constexpr (VEC) return __ldg(reinterpret_cast<const float4*>(w1));
  return make_float4(__ldg(w1), __ldg(w1 + 1), __ldg(w1 + 2), __ldg(w1 + 3));
}

// ----------------------------------------------------------------- forward
// One CTA of 512 threads per SM: two groups of 256 share the transposed W1 and
// each takes its own tiles (named barriers), so one group's loads and layer 0
// run under the other's FMAs. Layer 1 per thread: 8 rows x 8 columns (128-row
// tiles), 4 x 4 (32-row tiles), each sum in k order.
// A row's logits are the same bits in either kind of tile (the renderer's rows
// lie anywhere): of each 64 columns the chain over columns 4 x .. 4 x + 3 and
// 32 + 4 x .. 32 + 4 x + 3 for x = 0..7, the chains' sum as a tree over bits 2, 1,
// 0 of x, then the two 64-column sums. In a 128-row tile a thread has the whole
// chain; in a 32-row tile lane x has its first half and lane x + 8 goes on from
// there. (Two chains of four instead, added in the thread, cost a 397x301 FP32
// frame 2237 -> 2304 us.)
constexpr int kFwdGroup = 256;
constexpr int kFwdThreads = 2 * kFwdGroup;

template <int CQ>
struct FwdGroupSmem {
  float h0[kW * kLd];  // relu(layer 0), [n][row]; 32-row tiles use a stride of 36
  float x[128 * 4 * CQ];  // k0 rows; then the logit partials [column warp][row][c]
  int32_t rays[128];
};
template <int CQ>
struct FwdSmem {
  float w1t[kW * kW];  // [k][n]
  float w0k[4 * CQ * kW];
  float w2[3 * kW];
  float b1[kW];
  float b2[4];
  FwdGroupSmem<CQ> g[2];
};

// RT, CT: 4-row and 4-column chunks per thread (2, 2: 128-row tiles; 1, 1: 32).
template <int RT, int CT, int CQ>
__device__ __forceinline__ void fwd_tile(FwdSmem<CQ>& S, FwdGroupSmem<CQ>& G, int bar, int t,
                                         const MlpArgs& a, const float* __restrict__ k0,
                                         const int32_t* __restrict__ ray,
                                         const float* __restrict__ hpe, int64_t row0, int64_t M,
                                         float* out, const float* rw) {
  constexpr int TR = RT == 2 ? 128 : 32;
  constexpr int ld = TR + 4;
  constexpr int kColWarps = 2;                // 64 columns each
  constexpr int kColLanes = RT == 2 ? 8 : 16;
  const int lane = t & 31, warp = t >> 5, tx = lane % kColLanes, ty = lane / kColLanes;
  const int cw = warp % kColWarps;
  // rows rb + 16 i + e, columns cb + 32 j + e
  const int rb = (warp / kColWarps) * (RT == 2 ? 32 : 8) + 4 * ty;
  const int cb = cw * 64 + 4 * tx;
  load_rows<TR, CQ>(G.x, G.rays, t, kFwdGroup, a.c0, k0, ray, row0, M);
  bar_group(bar, kFwdGroup);
  layer0<TR, CQ, kFwdGroup>(G.h0, ld, S.w0k, G.x, G.rays, hpe, t);
  bar_group(bar, kFwdGroup);
  f32x2 acc2[2 * RT][4 * CT];  // row pairs
#pragma unroll
  for (int i = 0; i < 2 * RT; ++i)
#pragma unroll
    for (int j = 0; j < 4 * CT; ++j) acc2[i][j] = 0;
#pragma unroll 4
  for (int k = 0; k < kW; ++k) {
    f32x2 av[2 * RT];
    float bv[4 * CT];
#pragma unroll
    for (int i = 0; i < RT; ++i)
      *reinterpret_cast<ulonglong2*>(av + 2 * i) =
          *reinterpret_cast<const ulonglong2*>(G.h0 + k * ld + rb + 16 * i);
#pragma unroll
    for (int j = 0; j < CT; ++j)
      *reinterpret_cast<float4*>(bv + 4 * j) =
          *reinterpret_cast<const float4*>(S.w1t + k * kW + cb + 32 * j);
#pragma unroll
    for (int j = 0; j < 4 * CT; ++j) {
      const f32x2 d = dup2(bv[j]);
#pragma unroll
      for (int i = 0; i < 2 * RT; ++i) acc2[i][j] = fma2(av[i], d, acc2[i][j]);
    }
  }
  // logits: this thread's columns, then the lanes of its rows (a reduce-scatter),
  // then the column warps
  float lg[12 * RT];
#pragma unroll
  for (int i = 0; i < 12 * RT; ++i) lg[i] = 0.f;
  auto add_columns = [&](float* l) {
#pragma unroll
    for (int j = 0; j < 4 * CT; ++j) {
      const int n = cb + 32 * (j >> 2) + (j & 3);
      const float b1 = S.b1[n];
      const float w[3] = {S.w2[n], S.w2[kW + n], S.w2[2 * kW + n]};
#pragma unroll
      for (int i = 0; i < 2 * RT; ++i) {
        float h[2];
        unpack2(acc2[i][j], h[0], h[1]);
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          h[e] = fmaxf(h[e] + b1, 0.f);
#pragma unroll
          for (int c = 0; c < 3; ++c)
            l[3 * (2 * i + e) + c] = fmaf(w[c], h[e], l[3 * (2 * i + e) + c]);
        }
      }
    }
  };
  add_columns(lg);
  float* red = G.x;
  int row = rb;
  bool mine = true;
  if (RT == 2) {
    scatter_step<24>(lg, 4, tx & 4);
    scatter_step<12>(lg, 2, tx & 2);
    scatter_step<6>(lg, 1, tx & 1);
    row += (tx & 4 ? 16 : 0) + (tx & 2) + (tx & 1);
  } else {
    // the chain goes on from the lane of the lower half
#pragma unroll
    for (int i = 0; i < 12; ++i) lg[i] = __shfl_xor_sync(0xffffffffu, lg[i], 8);
    add_columns(lg);
    scatter_step<12>(lg, 4, tx & 4);
    scatter_step<6>(lg, 2, tx & 2);
#pragma unroll
    for (int c = 0; c < 3; ++c) lg[c] += __shfl_xor_sync(0xffffffffu, lg[c], 1);
    row += (tx & 4 ? 2 : 0) + (tx & 2 ? 1 : 0);
    mine = (tx & 9) == 8;
  }
  if (mine) {
#pragma unroll
    for (int c = 0; c < 3; ++c) red[(cw * TR + row) * 3 + c] = lg[c];
  }
  bar_group(bar, kFwdGroup);
  for (int e = t; e < TR * 3; e += kFwdGroup) {
    float s = red[e];
#pragma unroll
    for (int w = 1; w < kColWarps; ++w) s += red[w * TR * 3 + e];
    s += S.b2[e % 3];
    if (row0 * 3 + e < M * 3)
      out[row0 * 3 + e] = __fdiv_rn(rw ? __ldg(rw + row0 + e / 3) : 1.f, 1.f + expf(-s));
  }
  bar_group(bar, kFwdGroup);  // the partials are read: the next tile's rows may land
}

template <int CQ, bool VEC>
__global__ void __launch_bounds__(kFwdThreads, 1)
    k_mlp_fwd_f32(MlpArgs a, const float* __restrict__ k0, const int32_t* __restrict__ ray,
                  const float* __restrict__ hpe, const uint32_t* __restrict__ totals, float* out,
                  const float* __restrict__ rw) {
  grid_dep_sync();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  FwdSmem<CQ>& S = *reinterpret_cast<FwdSmem<CQ>*>(smem_raw);
  const int64_t M = totals[1];
  const int64_t units = 2ll * gridDim.x;
  const TilePlan P = tile_plan(M, units);
  // unit u = blockIdx.x + gridDim.x * group: a small batch spreads over the SMs first
  if (int64_t(blockIdx.x) >= P.full && P.row32 + 32ll * blockIdx.x >= M) return;
  const int tid = threadIdx.x;
  for (int i = tid; i < kW * kW / 4; i += kFwdThreads) {
    const int n = i % kW, k = 4 * (i / kW);  // lanes along n: conflict-free stores
    const float4 v = w1_quad<VEC>(a.w1 + n * kW + k);
    S.w1t[k * kW + n] = v.x;
    S.w1t[(k + 1) * kW + n] = v.y;
    S.w1t[(k + 2) * kW + n] = v.z;
    S.w1t[(k + 3) * kW + n] = v.w;
  }
  load_w0k<CQ>(S.w0k, a, tid, kFwdThreads);
  for (int i = tid; i < 3 * kW; i += kFwdThreads) S.w2[i] = a.w2[i];
  if (tid < kW) S.b1[tid] = a.b1[tid];
  if (tid < 3) S.b2[tid] = a.b2[tid];
  __syncthreads();
  const int g = tid / kFwdGroup, t = tid % kFwdGroup;
  const int64_t u = int64_t(blockIdx.x) + int64_t(gridDim.x) * g;
  FwdGroupSmem<CQ>& G = S.g[g];
  for (int64_t i = u; i < P.full; i += units)
    fwd_tile<2, 2, CQ>(S, G, 1 + g, t, a, k0, ray, hpe, i * 128, M, out, rw);
  for (int64_t r = P.row32 + u * 32; r < M; r += units * 32)
    fwd_tile<1, 1, CQ>(S, G, 1 + g, t, a, k0, ray, hpe, r, M, out, rw);
}

// ---------------------------------------------------------------- backward
// One CTA of 512 threads per SM; per tile of TR rows (128 or 32):
//   h0 = relu(layer 0); h1 = relu(h0.W1^T + b1) in registers (the forward's
//   sums in the forward's order, so the ReLU masks are the forward's)
//   dl  = grad_rgb (1-y) y          dz1 = (dl.W2) [h1 > 0]
//   dW2 += dl^T.h1, db1 += sum dz1  (registers; lanes of a column reduced per tile)
//   dW1 += dz1^T.h0                 dz0 = (dz1.W1) [h0 > 0]
//   dW0|db0 += dz0^T.[k0|PE|1]      gk0 = dz0.W0k
// The weight gradients stay in registers over all the CTA's tiles; per-CTA
// partials are summed in CTA order afterwards, so they are deterministic for a
// given grid size.
constexpr int kBwdThreads = 512;

template <int CQ>
struct BwdSmem {
  static constexpr int kQ = CQ == 3 ? 40 : 48;  // columns of [k0 | PE | 1 | 0]
  float w1[kW * kLd];  // [n][k]
  float h0[kW * kLd];  // [k][row]; then [k0 | PE | 1]^T [q][row]
  float dz[kW * kLd];  // dz1 [n][row]; then dz0 [k][row]
  float x[128 * 4 * CQ];
  float w0k[4 * CQ * kW];
  float dl[128 * 4];
  float w2[3 * kW];
  float b1[kW];
  int32_t rays[128];
};

struct BwdIn {
  const float* __restrict__ k0;
  const int32_t* __restrict__ ray;
  const float* __restrict__ hpe;
  const float* __restrict__ pe;
  const float* __restrict__ rgb;
  const float* __restrict__ grad_rgb;
  float* grad_k0;
};

// The weight-gradient accumulators of a thread (warp w, lane = 8 ty + tx).
template <int CQ>
struct BwdAcc {
  static constexpr int kQJ = BwdSmem<CQ>::kQ / 8;
  float w1[4][8];    // dW1[16 (w / 2) + ty + 4 i][64 (w % 2) + tx + 8 j]
  float w0[2][kQJ];  // dW0[8 w + ty + 4 i][tx + 8 j]
  float m128[8];     // dW2 / db1 sums of two columns, from the 128-row tiles
  float m32[2];      // dW2 / db1 sums (two of a column's four), from the 32-row tiles
  float b2;          // warps 0..2: this lane's part of db2[warp]
};

template <int TR, int CQ>
__device__ __forceinline__ void bwd_tile(BwdSmem<CQ>& B, BwdAcc<CQ>& A, const MlpArgs& a,
                                         const BwdIn& in, int64_t row0, int64_t M) {
  constexpr int ld = TR + 4;
  constexpr int CJ = TR == 128 ? 8 : 2;          // columns per thread
  constexpr int kColWarps = TR == 128 ? 2 : 8;   // a warp: 16 rows x 8 CJ columns
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = lane & 7, ty = lane >> 3;
  const int rb = (warp / kColWarps) * 16 + 4 * ty;
  const int nb = (warp % kColWarps) * (8 * CJ);
  load_rows<TR, CQ>(B.x, B.rays, tid, kBwdThreads, a.c0, in.k0, in.ray, row0, M);
  for (int i = tid; i < TR * 3; i += kBwdThreads) {
    float d = 0.f;
    if (row0 * 3 + i < M * 3) {
      const float y = __ldg(in.rgb + row0 * 3 + i);
      d = __ldg(in.grad_rgb + row0 * 3 + i) * (1.f - y) * y;
    }
    B.dl[(i / 3) * 4 + i % 3] = d;
  }
  __syncthreads();
  layer0<TR, CQ, kBwdThreads>(B.h0, ld, B.w0k, B.x, B.rays, in.hpe, tid);
  if (warp < 3) {
    for (int r = lane; r < TR; r += 32) A.b2 += B.dl[r * 4 + warp];
  }
  __syncthreads();
  // ---- layer 1: columns n = nb + tx + 8 j, read along k
  float acc[4][CJ];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < CJ; ++j) acc[i][j] = 0.f;
#pragma unroll 1
  for (int k = 0; k < kW; k += 4) {
    float av[4][4];  // [k][row]
#pragma unroll
    for (int e = 0; e < 4; ++e)
      *reinterpret_cast<float4*>(av[e]) =
          *reinterpret_cast<const float4*>(B.h0 + (k + e) * ld + rb);
#pragma unroll
    for (int j = 0; j < CJ; ++j) {
      float bv[4];
      *reinterpret_cast<float4*>(bv) =
          *reinterpret_cast<const float4*>(B.w1 + (nb + tx + 8 * j) * kLd + k);
#pragma unroll
      for (int e = 0; e < 4; ++e)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[i][j] = fmaf(av[e][i], bv[e], acc[i][j]);
    }
  }
  // ---- dz1, and this tile's dW2 / db1 sums over the thread's four rows
  {
    float d[4][3];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float4 v = *reinterpret_cast<const float4*>(B.dl + (rb + i) * 4);
      d[i][0] = v.x;
      d[i][1] = v.y;
      d[i][2] = v.z;
    }
    float s[4 * CJ];
#pragma unroll
    for (int j = 0; j < CJ; ++j) {
      const int n = nb + tx + 8 * j;
      const float b1 = B.b1[n];
      const float w[3] = {B.w2[n], B.w2[kW + n], B.w2[2 * kW + n]};
      float z[4];
      float sc[3] = {0.f, 0.f, 0.f}, sb = 0.f;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float h = fmaxf(acc[i][j] + b1, 0.f);
        float g = 0.f;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          g = fmaf(d[i][c], w[c], g);
          sc[c] = fmaf(d[i][c], h, sc[c]);
        }
        z[i] = h > 0.f ? g : 0.f;
        sb += z[i];
      }
      *reinterpret_cast<float4*>(B.dz + n * ld + rb) = make_float4(z[0], z[1], z[2], z[3]);
#pragma unroll
      for (int c = 0; c < 3; ++c) s[4 * j + c] = sc[c];
      s[4 * j + 3] = sb;
    }
    // over the four ty: lane ty keeps a quarter of the values
    scatter_step<4 * CJ>(s, 16, ty & 2);
    scatter_step<2 * CJ>(s, 8, ty & 1);
    if (TR == 128) {
#pragma unroll
      for (int e = 0; e < 8; ++e) A.m128[e] += s[e];
    } else {
#pragma unroll
      for (int e = 0; e < 2; ++e) A.m32[e] += s[e];
    }
  }
  __syncthreads();
  // ---- dW1[n][k] += sum_row dz1[n][row] h0[k][row], read along the rows:
  // n = 16 (warp / 2) + ty + 4 i, k = 64 (warp % 2) + tx + 8 j
  {
    const float* za = B.dz + (16 * (warp >> 1) + ty) * ld;
    const float* hb = B.h0 + (64 * (warp & 1) + tx) * ld;
#pragma unroll 1
    for (int r = 0; r < TR; r += 4) {
      float av[4][4];  // [n][row]
#pragma unroll
      for (int i = 0; i < 4; ++i)
        *reinterpret_cast<float4*>(av[i]) = *reinterpret_cast<const float4*>(za + 4 * i * ld + r);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        float bv[4];
        *reinterpret_cast<float4*>(bv) = *reinterpret_cast<const float4*>(hb + 8 * j * ld + r);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int i = 0; i < 4; ++i) A.w1[i][j] = fmaf(av[i][e], bv[e], A.w1[i][j]);
      }
    }
  }
  // ---- dh0[row][k] = sum_n dz1[n][row] W1[n][k]; k in chunks of 4 (TR = 128:
  // two chunks, k = 64 (warp % 2) + 4 tx + 32 j + e) or 2 (TR = 32:
  // k = 16 (warp % 8) + 2 tx + e)
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < CJ; ++j) acc[i][j] = 0.f;
  const int kb = TR == 128 ? 64 * (warp & 1) + 4 * tx : 16 * (warp & 7) + 2 * tx;
#pragma unroll 4
  for (int n = 0; n < kW; ++n) {
    float av[4], bv[CJ];
    *reinterpret_cast<float4*>(av) = *reinterpret_cast<const float4*>(B.dz + n * ld + rb);
    if (TR == 128) {
#pragma unroll
      for (int j = 0; j < CJ / 4; ++j)
        *reinterpret_cast<float4*>(bv + 4 * j) =
            *reinterpret_cast<const float4*>(B.w1 + n * kLd + kb + 32 * j);
    } else {
      *reinterpret_cast<float2*>(bv) = *reinterpret_cast<const float2*>(B.w1 + n * kLd + kb);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < CJ; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
  }
  // dz0 = dh0 [h0 > 0]
#pragma unroll
  for (int j = 0; j < CJ; ++j) {
    const int k = TR == 128 ? kb + 32 * (j >> 2) + (j & 3) : kb + j;
    const float4 h = *reinterpret_cast<const float4*>(B.h0 + k * ld + rb);
    acc[0][j] = h.x > 0.f ? acc[0][j] : 0.f;
    acc[1][j] = h.y > 0.f ? acc[1][j] : 0.f;
    acc[2][j] = h.z > 0.f ? acc[2][j] : 0.f;
    acc[3][j] = h.w > 0.f ? acc[3][j] : 0.f;
  }
  __syncthreads();  // dz1 and h0 are read
#pragma unroll
  for (int j = 0; j < CJ; ++j) {
    const int k = TR == 128 ? kb + 32 * (j >> 2) + (j & 3) : kb + j;
    *reinterpret_cast<float4*>(B.dz + k * ld + rb) =
        make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
  }
  // [k0 | PE | 1 | 0]^T over h0 (PE rows are 32 floats; lanes along the rows)
  {
    float* xt = B.h0;
    const int r = tid & (TR - 1);
    const int ry = B.rays[r];
    for (int q = tid / TR; q < BwdSmem<CQ>::kQ; q += kBwdThreads / TR) {
      float v = 0.f;
      if (q < a.c0)
        v = B.x[r * 4 * CQ + q];
      else if (q < a.din)
        v = ry >= 0 ? __ldg(in.pe + int64_t(ry) * kPeStride + (q - a.c0)) : 0.f;
      else if (q == a.din)
        v = 1.f;
      xt[q * ld + r] = v;
    }
  }
  __syncthreads();
  // ---- dW0|db0[n][q] += sum_row dz0[n][row] x[q][row]: n = 8 warp + ty + 4 i, q = tx + 8 j
  {
    constexpr int QJ = BwdAcc<CQ>::kQJ;
    const float* za = B.dz + (8 * warp + ty) * ld;
    const float* xb = B.h0 + tx * ld;
#pragma unroll 1
    for (int r = 0; r < TR; r += 4) {
      float av[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
        *reinterpret_cast<float4*>(av[i]) = *reinterpret_cast<const float4*>(za + 4 * i * ld + r);
#pragma unroll
      for (int j = 0; j < QJ; ++j) {
        float bv[4];
        *reinterpret_cast<float4*>(bv) = *reinterpret_cast<const float4*>(xb + 8 * j * ld + r);
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int i = 0; i < 2; ++i) A.w0[i][j] = fmaf(av[i][e], bv[e], A.w0[i][j]);
      }
    }
  }
  // ---- gk0[row][q] = sum_n dz0[n][row] w0k[q][n]: a thread takes four rows,
  // half of the channels and every NS-th n; the NS lanes are then reduced
  {
    constexpr int NS = TR == 128 ? 8 : 32;
    constexpr int KQ = 2 * CQ;  // channels per thread
    const int ns = lane & (NS - 1);
    const int grp = warp * (32 / NS) + lane / NS;  // row group x channel half
    const int rg = grp % (TR / 4), q0 = (grp / (TR / 4)) * KQ;
    float v[4 * KQ];
#pragma unroll
    for (int e = 0; e < 4 * KQ; ++e) v[e] = 0.f;
#pragma unroll 4
    for (int n = ns; n < kW; n += NS) {
      const float4 z = *reinterpret_cast<const float4*>(B.dz + n * ld + 4 * rg);
#pragma unroll
      for (int q = 0; q < KQ; ++q) {
        const float w = B.w0k[(q0 + q) * kW + n];
        v[q] = fmaf(z.x, w, v[q]);
        v[KQ + q] = fmaf(z.y, w, v[KQ + q]);
        v[2 * KQ + q] = fmaf(z.z, w, v[2 * KQ + q]);
        v[3 * KQ + q] = fmaf(z.w, w, v[3 * KQ + q]);
      }
    }
    scatter_step<4 * KQ>(v, 1, ns & 1);
    scatter_step<2 * KQ>(v, 2, ns & 2);
    scatter_step<KQ>(v, 4, ns & 4);
#pragma unroll
    for (int o = 8; o < NS; o <<= 1)
#pragma unroll
      for (int e = 0; e < KQ / 2; ++e) v[e] += __shfl_xor_sync(0xffffffffu, v[e], o);
    const int64_t m = row0 + 4 * rg + 2 * (ns & 1) + ((ns >> 1) & 1);
    if (ns < 8 && m < M) {
#pragma unroll
      for (int e = 0; e < KQ / 2; ++e) {
        const int q = q0 + (ns & 4 ? KQ / 2 : 0) + e;
        if (q < a.c0) in.grad_k0[m * a.c0 + q] = v[e];
      }
    }
  }
  __syncthreads();
}

template <int CQ, bool VEC>
__global__ void __launch_bounds__(kBwdThreads, 1)
    k_mlp_bwd_f32(MlpArgs a, BwdIn in, const uint32_t* __restrict__ totals, float* wpart) {
  grid_dep_sync();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  BwdSmem<CQ>& B = *reinterpret_cast<BwdSmem<CQ>*>(smem_raw);
  const int64_t M = totals[1];
  const TilePlan P = tile_plan(M, gridDim.x);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, tx = lane & 7, ty = lane >> 3;
  float* pw0 = wpart + int64_t(blockIdx.x) * mlp_param_count(a.din);
  float* pb0 = pw0 + kW * a.din;
  float* pw1 = pb0 + kW;
  float* pb1 = pw1 + kW * kW;
  float* pw2 = pb1 + kW;
  float* pb2 = pw2 + 3 * kW;
  constexpr int QJ = BwdAcc<CQ>::kQJ;
  BwdAcc<CQ> A;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) A.w1[i][j] = 0.f;
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < QJ; ++j) A.w0[i][j] = 0.f;
#pragma unroll
  for (int e = 0; e < 8; ++e) A.m128[e] = 0.f;
  A.m32[0] = A.m32[1] = 0.f;
  A.b2 = 0.f;
  if (blockIdx.x >= active_parts(M, gridDim.x, false)) return;
  {
    for (int i = tid; i < kW * kW / 4; i += kBwdThreads) {
      const int n = i / (kW / 4), k = 4 * (i % (kW / 4));
      *reinterpret_cast<float4*>(B.w1 + n * kLd + k) = w1_quad<VEC>(a.w1 + n * kW + k);
    }
    load_w0k<CQ>(B.w0k, a, tid, kBwdThreads);
    for (int i = tid; i < 3 * kW; i += kBwdThreads) B.w2[i] = a.w2[i];
    if (tid < kW) B.b1[tid] = a.b1[tid];
    __syncthreads();
  }
  for (int64_t i = blockIdx.x; i < P.full; i += gridDim.x)
    bwd_tile<128, CQ>(B, A, a, in, i * 128, M);
  for (int64_t r = P.row32 + 32ll * blockIdx.x; r < M; r += 32ll * gridDim.x)
    bwd_tile<32, CQ>(B, A, a, in, r, M);
  // this CTA's partials
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j)
      pw1[(16 * (warp >> 1) + ty + 4 * i) * kW + 64 * (warp & 1) + tx + 8 * j] = A.w1[i][j];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int n = 8 * warp + ty + 4 * i;
#pragma unroll
    for (int j = 0; j < QJ; ++j) {
      const int q = tx + 8 * j;
      if (q < a.din)
        pw0[n * a.din + q] = A.w0[i][j];
      else if (q == a.din)
        pb0[n] = A.w0[i][j];
    }
  }
  // dW2 / db1: the row warps' sums of a column through shared memory, in warp
  // order. s[4 j + c] after the reduce-scatter over ty: 128-row tiles, lane ty
  // holds columns j = 2 ty', 2 ty' + 1 (c = 0..3 each); 32-row tiles, lane ty
  // holds column j = ty' / 2, entries 2 (ty' % 2) + {0, 1}; ty' = ty.
  float* part = B.h0;  // [10 row warps][4][128]
  __syncthreads();
  {
    const int nb = (warp & 1) * 64;
#pragma unroll
    for (int e = 0; e < 8; ++e) {
      const int s = ty * 8 + e;  // index among the 32 values (ty & 2 picks the upper half first)
      part[((warp >> 1) * 4 + (s & 3)) * kW + nb + tx + 8 * (s >> 2)] = A.m128[e];
    }
    const int nb32 = (warp & 7) * 16;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int s = ty * 2 + e;
      part[((8 + (warp >> 3)) * 4 + (s & 3)) * kW + nb32 + tx + 8 * (s >> 2)] = A.m32[e];
    }
  }
  __syncthreads();
  {
    const int c = tid / kW, n = tid % kW;
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 10; ++w) s += part[(w * 4 + c) * kW + n];
    if (c < 3)
      pw2[c * kW + n] = s;
    else
      pb1[n] = s;
  }
  if (warp < 3) {
    float s = A.b2;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) pb2[warp] = s;
  }
}

static_assert(sizeof(FwdSmem<4>) <= 227 * 1024 && sizeof(BwdSmem<4>) <= 227 * 1024,
              "one CTA's shared memory");

template <int CQ, bool VEC>
int fwd_launch(const MlpArgs& a, const float* k0, const int32_t* ray, const float* hpe,
               const uint32_t* totals, float* out, const float* rw, cudaStream_t st) {
  const auto kernel = k_mlp_fwd_f32<CQ, VEC>;
  PVDB_SMEM_ATTR(kernel, int(sizeof(FwdSmem<CQ>)));
  launch_k(kernel, num_sms(), kFwdThreads, sizeof(FwdSmem<CQ>), st, a, k0, ray, hpe, totals, out,
           rw);
  PVDB_CHECK_LAUNCH("k_mlp_fwd_f32");
  return PVDB_OK;
}

template <int CQ, bool VEC>
int bwd_launch(const MlpArgs& a, const BwdIn& in, const uint32_t* totals, float* wpart, int grid,
               cudaStream_t st) {
  const auto kernel = k_mlp_bwd_f32<CQ, VEC>;
  PVDB_SMEM_ATTR(kernel, int(sizeof(BwdSmem<CQ>)));
  launch_k(kernel, grid, kBwdThreads, sizeof(BwdSmem<CQ>), st, a, in, totals, wpart);
  PVDB_CHECK_LAUNCH("k_mlp_bwd_f32");
  return PVDB_OK;
}

bool on_16_bytes(const float* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

// Up to 12 k0 channels (at most 39 input columns) or up to 16 (43): the
// channel count padded to 12 or 16 with zeros.
int mlp_f32_forward(const MlpArgs& a, const float* k0, const int32_t* ray, const float* hpe,
                    const uint32_t* totals, float* out, const float* rw, cudaStream_t st) {
  const bool vec = on_16_bytes(a.w1);
  const auto launch = a.c0 <= 12 ? (vec ? fwd_launch<3, true> : fwd_launch<3, false>)
                                 : (vec ? fwd_launch<4, true> : fwd_launch<4, false>);
  return launch(a, k0, ray, hpe, totals, out, rw, st);
}

int mlp_f32_backward(const MlpArgs& a, const float* k0, const int32_t* ray, const float* hpe,
                     const float* pe, const uint32_t* totals, const float* rgb,
                     const float* grad_rgb, float* grad_k0, float* wpart, int grid,
                     cudaStream_t st) {
  const BwdIn in{k0, ray, hpe, pe, rgb, grad_rgb, grad_k0};
  const bool vec = on_16_bytes(a.w1);
  const auto launch = a.c0 <= 12 ? (vec ? bwd_launch<3, true> : bwd_launch<3, false>)
                                 : (vec ? bwd_launch<4, true> : bwd_launch<4, false>);
  return launch(a, in, totals, wpart, grid, st);
}

}  // namespace pvdb
