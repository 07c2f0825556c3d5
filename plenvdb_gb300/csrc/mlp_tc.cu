// rgbnet on the 5th-generation tensor cores (tcgen05), BF16 operands with FP32
// accumulation in TMEM — the BF16 path of the colour MLP (dvgo.py:99-107,
// :354-362; renderer.cu:83-119).
//
// Rows are processed in tiles of 128 (TMEM lane = tile row). Each row's input
// is X = [k0 (c0) | PE (dpe) | 1 | 0...], 48 BF16 columns, so layer 0 is one
// K=48 GEMM against W0f = [W0 | b0 | 0] (the bias rides on the ones column).
//
// Forward (k_mlp_fwd_tc), per tile:
//   L0  Z0 = X . W0f^T            3 MMAs (K=48)        H0 = relu(Z0)
//   L1  Z1 = H0 . W1^T            8 MMAs (K=128)       H1 = relu(Z1 + b1)
//   L2  Z2 = H1 . W2p^T           8 MMAs, N=16         rgb = sigmoid(Z2 + b2)
// X tiles are built beforehand and fetched with bulk copies, or (GATHER, the
// renderer's BF16 features) formed by the slot's own threads, a row a thread,
// while the tensor cores run the previous tile's layer 1: the rows are then
// never written out. A tile is a chain
// of three MMA batches and three epilogues, so the kernel is bound by that
// chain's latency and by how many chains an SM keeps going: one persistent CTA
// per SM shares the 48 KB of weights between four independent warpgroups, each
// with its own tile, 128 TMEM columns (Z0 and Z1 in turn, then H1 and Z2),
// barriers and issuing thread. Epilogues read TMEM with tcgen05.ld (thread =
// tile row), apply bias/activation in FP32 and store BF16: H0 into shared memory
// in the canonical layout the next MMA reads, H1 back into TMEM, from where L2
// takes its A operand (512 cycles a tile of shared-memory traffic less; 800x800
// frame 1496 -> 1480 us, 320^3 step 4831 -> 4807 us). Both in TMEM would take 192
// columns a tile, so two tiles in flight instead of four.
#include <algorithm>

#include "march.cuh"
#include "render_rows.cuh"
#include "tc.cuh"

namespace pvdb {

namespace {

constexpr int kW = 128;
constexpr int kFwdSlots = 4;                    // warpgroups, a tile in flight each
constexpr int kFwdThreads = 128 * kFwdSlots;
constexpr int kXK = kRgbXK;  // input columns of a row: k0 | PE | 1 | 0
// packed weight blob (bytes, canonical K-major BF16 tiles)
constexpr uint32_t kOffW0 = 0;                             // W0f  [128 n][48 q]
constexpr uint32_t kOffW1 = kOffW0 + 128 * kXK * 2;        // W1   [128 n][128 k]   12288
constexpr uint32_t kOffW2 = kOffW1 + 128 * 128 * 2;        // W2p  [16 c][128 k]    45056
constexpr uint32_t kPackFwdBytes = kOffW2 + 16 * 128 * 2;  // 49152
// shared-memory layout of the forward kernel
constexpr uint32_t kXTile = kRgbXTile;                // 12288 B: one X tile
constexpr uint32_t kSlotBytes = kXTile + 128 * 128 * 2;     // X [128 x 48], H [128 x 128] bf16
constexpr uint32_t kSmSlots = kPackFwdBytes;
constexpr uint32_t kSmB1 = kSmSlots + kFwdSlots * kSlotBytes;  // b1 f32[128]
constexpr uint32_t kSmB2 = kSmB1 + 128 * 4;                    // b2 f32[16]
constexpr uint32_t kSmBar = kSmB2 + 16 * 4;  // mbarriers: MMA, X per slot, then the weights
constexpr uint32_t kSmTmem = kSmBar + 8 * (2 * kFwdSlots + 1);  // TMEM base address (4 B)
constexpr uint32_t kSmFlag = kSmTmem + 4;                       // timeout flag per slot
constexpr uint32_t kSmFwdBytes = kSmFlag + 4 * kFwdSlots;
static_assert(kSlotBytes % 1024 == 0 && kSmFwdBytes <= 232448, "the forward CTA's shared memory");
constexpr uint32_t kTmemCols = 128 * kFwdSlots;
constexpr uint32_t kWaitIters = 1u << 22;

struct MlpArgsTc {
  const float* w0; const float* b0;
  const float* w1; const float* b1;
  const float* w2; const float* b2;
  int c0, dpe, din;
};

// FP32 nn.Linear weights -> BF16 canonical K-major tiles (one thread per
// element). The backward reads the same tiles, transposed through MN-major
// descriptors.
__global__ void k_pack(MlpArgsTc a, uint8_t* blob) {
  grid_dep_sync();
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  __nv_bfloat16* w0 = reinterpret_cast<__nv_bfloat16*>(blob + kOffW0);
  __nv_bfloat16* w1 = reinterpret_cast<__nv_bfloat16*>(blob + kOffW1);
  __nv_bfloat16* w2 = reinterpret_cast<__nv_bfloat16*>(blob + kOffW2);
  if (t < 128 * kXK) {  // W0f[n][q] = w0[n][q] (q < din), b0[n] (q == din), 0
    const int n = t / kXK, q = t % kXK;
    const float v = q < a.din ? a.w0[n * a.din + q] : q == a.din ? a.b0[n] : 0.f;
    w0[tc::kmaj(n, q, kXK) / 2] = __float2bfloat16_rn(v);
  }
  if (t < 128 * 128) {
    const int n = t / 128, k = t % 128;
    w1[tc::kmaj(n, k, 128) / 2] = __float2bfloat16_rn(a.w1[n * 128 + k]);
  }
  if (t < 16 * 128) {
    const int n = t / 128, k = t % 128;
    w2[tc::kmaj(n, k, 128) / 2] = __float2bfloat16_rn(n < 3 ? a.w2[n * 128 + k] : 0.f);
  }
}

// The rows' X tiles in global memory, tile after tile in the canonical BF16
// K-major layout the MMAs read (one 16-byte chunk per thread): the MLP
// kernels fetch a tile with one bulk copy.
__global__ void __launch_bounds__(256)
    k_build_x(MlpArgsTc a, const float* __restrict__ k0, const int32_t* __restrict__ ray,
              const float* __restrict__ pe, int pe_stride, const uint32_t* __restrict__ totals,
              uint8_t* xt) {
  grid_dep_sync();
  const int64_t M = totals[1];
  const int64_t nchunks = (M + 127) / 128 * (128 * 6);
  for (int64_t c = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; c < nchunks;
       c += int64_t(gridDim.x) * blockDim.x) {
    const int64_t tile = c / (128 * 6);
    const int w = int(c - tile * (128 * 6));
    const int r = w / 6, qb = (w % 6) * 8;
    const int64_t m = tile * 128 + r;
    float v[8];
    if (m < M) {
      const int64_t rr = __ldg(ray + m);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int qq = qb + e;
        v[e] = qq < a.c0 ? __ldg(k0 + m * a.c0 + qq)
               : qq < a.din ? __ldg(pe + rr * pe_stride + (qq - a.c0))
               : qq == a.din ? 1.f : 0.f;
      }
    } else {
#pragma unroll
      for (int e = 0; e < 8; ++e) v[e] = 0.f;
    }
    uint4 pk;
    pk.x = tc::pack_bf16(v[0], v[1]);
    pk.y = tc::pack_bf16(v[2], v[3]);
    pk.z = tc::pack_bf16(v[4], v[5]);
    pk.w = tc::pack_bf16(v[6], v[7]);
    *reinterpret_cast<uint4*>(xt + tile * kXTile + tc::kmaj(r, qb, kXK)) = pk;
  }
}

// Thread 0 starts the bulk copy of X tile `t` into shared buffer `b`.
__device__ __forceinline__ void x_fetch(uint8_t* sm_x, const uint8_t* xt, int64_t t,
                                        uint64_t* xbar) {
  tc::mbar_expect_tx(xbar, kXTile);
  tc::bulk_g2s(sm_x, xt + t * kXTile, kXTile, xbar);
}

// BF16 pair (lo, hi) of FP32 values, rounded to nearest even and clamped below
// at zero: relu and rounding in one instruction (the values of relu before
// rounding, up to the sign of a zero).
__device__ __forceinline__ uint32_t pack_relu_bf16(float lo, float hi) {
  uint32_t r;
  asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
  return r;
}

// relu(v + bias) of 8 consecutive columns as 8 BF16.
__device__ __forceinline__ uint4 relu_pack8(const float* v, const float* bias, int col) {
  float h[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) h[e] = bias ? v[e] + bias[col + e] : v[e];
  return make_uint4(pack_relu_bf16(h[0], h[1]), pack_relu_bf16(h[2], h[3]),
                    pack_relu_bf16(h[4], h[5]), pack_relu_bf16(h[6], h[7]));
}

// 32 FP32 values (+ bias, relu) -> 4 x 8 BF16 into a K-major tile (ktot columns).
__device__ __forceinline__ void store_relu32(uint8_t* tile, int row, int col0, int ktot,
                                             const float* v, const float* bias) {
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<uint4*>(tile + tc::kmaj(row, col0 + 8 * c, ktot)) =
        relu_pack8(v + 8 * c, bias, col0 + 8 * c);
}

// relu(Z [+ bias]) of this thread's row, 128 columns, as BF16 into the K-major
// tile, or (TO_TMEM) packed in pairs over the first 64 of the columns they were
// read from; the TMEM load of a chunk travels while the previous one is packed.
template <bool TO_TMEM>
__device__ __forceinline__ void epilogue_relu(uint32_t taddr, uint8_t* tile, int row,
                                              const float* bias) {
  uint32_t r[2][32];
  tc::tmem_ld16_issue(taddr, r[0]);
  tc::tmem_ld16_issue(taddr + 16, r[0] + 16);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    tc::tmem_wait_ld();
    if (j < 3) {
      tc::tmem_ld16_issue(taddr + 32 * (j + 1), r[(j + 1) & 1]);
      tc::tmem_ld16_issue(taddr + 32 * (j + 1) + 16, r[(j + 1) & 1] + 16);
    }
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[j & 1][i]);
    if (TO_TMEM) {
      // (columns 16 j .. 16 j + 15 were read before: the loads in flight are
      // those of columns 32 (j + 1) and up)
      uint32_t h[16];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const uint4 p = relu_pack8(v + 8 * c, bias, 32 * j + 8 * c);
        h[4 * c] = p.x; h[4 * c + 1] = p.y; h[4 * c + 2] = p.z; h[4 * c + 3] = p.w;
      }
      tc::tmem_st16_issue(taddr + 16 * j, h);
    } else {
      store_relu32(tile, row, 32 * j, 128, v, bias);
    }
  }
  if (TO_TMEM) tc::tmem_wait_st();
}

__device__ __forceinline__ void slot_sync(int slot) {
  asm volatile("bar.sync %0, 128;" ::"r"(1 + slot) : "memory");
}

// out [M, 3]: sigmoid(Z2 + b2), times rw [M] when given (a row's contribution to
// its pixel).
template <bool GATHER>
__global__ void __launch_bounds__(kFwdThreads, 1)
    k_mlp_fwd_tc(MlpArgsTc a, const uint8_t* __restrict__ blob, const uint8_t* __restrict__ xt,
                 RowSource src, const uint32_t* __restrict__ totals, float* out,
                 const float* __restrict__ rw, uint32_t* err) {
  grid_dep_sync();
  extern __shared__ __align__(1024) uint8_t sm[];
  const int64_t M = totals[1];
  const int64_t ntiles = (M + 127) / 128;
  if (blockIdx.x >= ntiles) return;
  const int tid = threadIdx.x, row = tid & 127;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0), slot = warp >> 2;
  const bool issuer = (warp & 3) == 0;  // the slot's warp that issues its MMAs
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + kSmBar);
  uint64_t* bar = bars + 2 * slot;       // this slot's MMAs
  uint64_t* xbar = bars + 2 * slot + 1;  // this slot's X tile
  uint64_t* wbar = bars + 2 * kFwdSlots;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kSmTmem);
  uint32_t* flag = reinterpret_cast<uint32_t*>(sm + kSmFlag) + slot;
  float* b1s = reinterpret_cast<float*>(sm + kSmB1);
  float* b2s = reinterpret_cast<float*>(sm + kSmB2);
  uint8_t* sx = sm + kSmSlots + slot * kSlotBytes;
  uint8_t* sh = sx + kXTile;
  // tile u, u + stride, ... per slot: the slots of different SMs come first
  const int64_t u = int64_t(blockIdx.x) + int64_t(gridDim.x) * slot;
  const int64_t stride = int64_t(gridDim.x) * kFwdSlots;
  if (tid < 128) b1s[tid] = a.b1[tid];
  if (tid < 16) b2s[tid] = tid < 3 ? a.b2[tid] : 0.f;
  if (tid == 0) {
    tc::mbar_init(wbar, 1);
    // the packed weights (48 KB) in one bulk copy, beside the first X tiles'
    tc::mbar_expect_tx(wbar, kPackFwdBytes);
    tc::bulk_g2s(sm, blob, kPackFwdBytes, wbar);
  }
  if (row == 0) {
    *flag = 0;
    tc::mbar_init(bar, 1);
    tc::mbar_init(xbar, 1);
    if (!GATHER && u < ntiles) x_fetch(sx, xt, u, xbar);
  }
  if (tid < 32) {
    tc::tmem_alloc(tmem_slot, kTmemCols);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t sbase = tc::smem_addr(sm);
  const uint32_t xb = tc::smem_addr(sx), hb = tc::smem_addr(sh);
  const uint32_t d = tmem + 128u * slot;                              // the slot's columns
  const uint32_t t_lane = d + (uint32_t(row & ~31) << 16);           // this warp's lanes
  const uint32_t id_n128 = tc::idesc_bf16(128, 128);
  const uint32_t id_n16 = tc::idesc_bf16(128, 16);
  uint32_t phase = 0, xph = 0;
  bool ok = true, x_out = false;
  // a wait that gives up flags the slot; its threads leave together after the
  // next slot barrier (what they read until then is in bounds, if wrong)
  auto wait = [&](uint64_t* b, uint32_t parity) {
    if (tc::mbar_wait(b, parity, kWaitIters)) return;
    atomicOr(flag, 1u);
    if (err) atomicOr(err, 2u);
  };
  auto slot_ok = [&]() {
    tc::fence_before();
    tc::fence_async_smem();
    slot_sync(slot);
    return *((volatile uint32_t*)flag) == 0;
  };
  if (GATHER && u < ntiles) {
    write_x_row(src, load_row_pos(src, u * 128 + row, M), row, sx);
    ok = slot_ok();
  }
  for (int64_t t = u; ok && t < ntiles; t += stride) {
    const bool more = t + stride < ntiles;
    RowPos next;
    if (GATHER) next = load_row_pos(src, (t + stride) * 128 + row, M);
    if (issuer) {
      if (!GATHER) wait(xbar, xph);
      if (t == u) wait(wbar, 0);
      tc::fence_after();
      if (tc::elect_one()) {
#pragma unroll
        for (int s = 0; s < 3; ++s)
          tc::mma_bf16(d, tc::make_desc(xb + 256 * s, 128, 768),
                       tc::make_desc(sbase + kOffW0 + 256 * s, 128, 768), id_n128, s > 0);
        tc::mma_commit(bar);
      }
      __syncwarp();
    }
    xph ^= 1u;
    wait(bar, phase);
    phase ^= 1u;
    tc::fence_after();
    // the X tile is read: the next one travels from here
    x_out = !GATHER && more;
    if (row == 0 && x_out) x_fetch(sx, xt, t + stride, xbar);
    // ---- H0 = relu(Z0)
    epilogue_relu<false>(t_lane, sh, row, nullptr);
    if (!(ok = slot_ok())) break;
    if (issuer) {
      tc::fence_after();
      if (tc::elect_one()) {
#pragma unroll
        for (int s = 0; s < 8; ++s)
          tc::mma_bf16(d, tc::make_desc(hb + 256 * s, 128, 2048),
                       tc::make_desc(sbase + kOffW1 + 256 * s, 128, 2048), id_n128, s > 0);
        tc::mma_commit(bar);
      }
      __syncwarp();
    }
    if (GATHER && more) write_x_row(src, next, row, sx);
    wait(bar, phase);
    phase ^= 1u;
    tc::fence_after();
    // ---- H1 = relu(Z1 + b1), over Z1's first 64 columns
    epilogue_relu<true>(t_lane, nullptr, row, b1s);
    if (!(ok = slot_ok())) break;
    if (issuer) {
      tc::fence_after();
      if (tc::elect_one()) {
#pragma unroll
        for (int s = 0; s < 8; ++s)
          tc::mma_bf16_ta(d + 64, d + 8 * s, tc::make_desc(sbase + kOffW2 + 256 * s, 128, 2048),
                          id_n16, s > 0);
        tc::mma_commit(bar);
      }
      __syncwarp();
    }
    wait(bar, phase);
    phase ^= 1u;
    tc::fence_after();
    // ---- logits
    float v[16];
    tc::tmem_ld16(t_lane + 64, v);
    const int64_t m = t * 128 + row;
    if (m < M) {
      const float w = rw ? __ldg(rw + m) : 1.f;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        const float lg = v[c] + b2s[c];
        out[m * 3 + c] = __fdiv_rn(w, 1.f + expf(-lg));
      }
    }
    if (!(ok = slot_ok())) break;
  }
  if (!ok) {
    // a wait gave up: give the MMAs and the X copy in flight one more bounded
    // wait before their TMEM and shared memory are released
    tc::mbar_wait(bar, phase ^ 1u, kWaitIters);
    if (x_out) tc::mbar_wait(xbar, xph, kWaitIters);
    tc::mbar_wait(wbar, 0, kWaitIters);
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (tid < 32) tc::tmem_dealloc(tmem, kTmemCols);
}

// ---------------------------------------------------------------- backward
// Per 128-row tile:
//   recompute  Z0 = X.W0f^T -> H0 = relu(Z0);  Z1 = H0.W1^T -> H1 = relu(Z1 + b1)
//   dl   = grad_rgb * y (1 - y)                       [128 x 3] (sigmoid backward)
//   dZ1  = (dl . W2) * [H1 > 0]
//   dZ0  = (dZ1 . W1) * [H0 > 0]
//   gk0  = dZ0 . W0k
//   dW2 += H1^T . dl      dW1|db1 += dZ1^T . [H0|1]   dW0|db0 += dZ0^T . X
// One persistent CTA per SM keeps two tiles in flight, in two slots with their
// own shared-memory tiles and TMEM columns: while the eight epilogue warps of
// one slot drain TMEM and write the next operand, the tensor cores run the
// other slot's MMAs. One elected thread of a seventeenth warp issues every
// MMA, in a fixed order (stage k of slot 0, then stage k of slot 1, tile pair
// after tile pair), so the weight-gradient accumulators, resident in TMEM
// across all the CTA's tiles, sum in an order fixed by the data: bitwise
// reproducible.
//   stage  MMAs (issuer)                                   epilogue (the slot's warps)
//   S0     Z0 = X.W0f^T                -> A                E0  H0 = relu(Z0)
//   S1     Z1 = H0.W1^T                -> A                E1  H1 = relu(Z1 + b1), dl
//   S2     dZ1' = dl.W2 -> A;  dW2 += H1^T.dl             E2  dZ1 = dZ1'*[H1 > 0], over H1
//   S3     dH0 = dZ1.W1 -> A;  dW1|db1 += dZ1^T.[H0|1]     E3  dZ0 = dH0*[H0 > 0], over dZ1
//   S4     gk0 = dZ0.W0k -> G; dW0|db0 += dZ0^T.X          E4  gk0 -> global
// dl has three nonzero columns of the MMA's 16; dZ1' is one K = 16 MMA whose
// B operand is W2's first 8 rows (rows 3..7 zero) followed, as the second
// 8 of K, by finite weights that meet dl's zero columns. E2 masks it with the
// relu of H1, which E1 keeps in registers. A ones column in H0 and in X turns
// the bias sums into one more MMA column. W1 and
// W0k are the forward's K-major weight tiles read through MN-major
// descriptors (no transposed copies). An epilogue signals the issuer through
// its slot's mbarrier (256 arrivals) after a proxy fence (its shared-memory
// writes feed the next MMAs) and a tcgen05 fence (its TMEM reads precede the
// next MMA into those columns). The X tiles rotate through three buffers
// (tile j in buffer j % 3): E4 of tile j, after S4 has read the buffer for the
// last time, starts the bulk copy of tile j + 3's X, so a copy has two tiles'
// time to land before S0 needs it. At the end the CTA writes its partial
// weight gradients in the flat parameter layout; the partials are summed over
// CTAs in a fixed order.
constexpr int kBwdEpiWarps = 8;             // per slot: 4 lane quarters x 2 column halves
constexpr int kBwdThreads = (2 * kBwdEpiWarps + 1) * 32;  // + the issuer warp: 544
constexpr int kBwdIssuer = 2 * kBwdEpiWarps;  // warp index of the issuer
constexpr int kBwdXBufs = 3;                // X tiles in flight: tile j uses buffer j % 3
constexpr uint32_t kSlH0 = 0;               // H0 [128 r][144 k], col 128 = 1
constexpr uint32_t kSlH1 = kSlH0 + 128 * 144 * 2;  // H1, then dZ1, then dZ0 [128 r][128 n]
constexpr uint32_t kSlDl = kSlH1 + 128 * 128 * 2;  // dl [128 r][16 c]
constexpr uint32_t kSlot = kSlDl + 128 * 16 * 2;   // 73728 B per slot
constexpr uint32_t kBX = 2 * kSlot;                // X x 3 [128 r][48 q]: k0 | PE | 1 | 0
// W2p rows 0..7 [8 c][128 k] (K-major, as in the blob): the B operand of
// dZ1 = dl . W2, read MN-major; its K = 16 reaches 2 KB past the rows, into
// W0f (finite values that meet dl's zero columns 8..15)
constexpr uint32_t kBW2 = kBX + kBwdXBufs * kXTile;
constexpr uint32_t kBW0f = kBW2 + 8 * 128 * 2;     // W0f [128 n][48 q]
constexpr uint32_t kBW1 = kBW0f + 128 * kXK * 2;   // W1  [128 n][128 k]
constexpr uint32_t kBB1 = kBW1 + 128 * 128 * 2;    // b1 f32[128]
constexpr uint32_t kBBar = kBB1 + 128 * 4;         // mma[2], epi[2], x[3], drain, weights
constexpr uint32_t kBTmem = kBBar + 80;
constexpr uint32_t kBFlag = kBTmem + 4;
constexpr uint32_t kBXIssued = kBFlag + 4;         // X copies started, per buffer
constexpr uint32_t kSmBwdBytes = kBXIssued + 12;
constexpr uint32_t kBwdWBytes = kOffW2;            // W0f and W1 of the blob (45056 B)
constexpr uint32_t kBwdW2Bytes = 8 * 128 * 2;      // W2p rows 0..7 of the blob
static_assert(kSlot % 1024 == 0, "slot tiles keep their alignment");
static_assert(kBW1 - kBW0f == kOffW1 - kOffW0 && kBwdWBytes % 16 == 0, "W0f, W1 as in the blob");
static_assert(kSmBwdBytes <= 232448, "backward CTA exceeds 227 KB of shared memory");
// TMEM columns: per slot A (128) and G (16); the resident weight-gradient sums
constexpr uint32_t kTA0 = 0;     // slot s: kTA0 + 128*s  (Z0, Z1, dH0)
constexpr uint32_t kTG0 = 256;   // slot s: kTG0 + 16*s   (grad k0)
constexpr uint32_t kTW2 = 288;   // dW2 [128 n x 16 c]
constexpr uint32_t kTW0 = 304;   // dW0|db0 [128 n x 48 q]
constexpr uint32_t kTW1 = 352;   // dW1|db1 [128 n x 144 k]
constexpr uint32_t kTmemBwdCols = 512;
static_assert(kTW1 + 144 <= kTmemBwdCols, "TMEM columns");

// 0xFFFF in each 16-bit half of a BF16 pair whose magnitude is nonzero: bit 15
// (bit 31) of (w & 0x7FFF7FFF) + 0x7FFF7FFF is set exactly when the low (high)
// half is nonzero, and a byte permute replicates those sign bits over their
// halves.
__device__ __forceinline__ uint32_t nonzero_mask_bf16x2(uint32_t w) {
  const uint32_t t = (w & 0x7FFF7FFFu) + 0x7FFF7FFFu;
  uint32_t m;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(m) : "r"(t), "r"(0u), "r"(0xBB99u));
  return m;
}

// relu mask of 8 BF16 activations (a uint4: a relu output is positive exactly
// when its magnitude is nonzero) applied to 8 FP32 values, as 8 BF16.
__device__ __forceinline__ uint4 mask_pack(const float* v, uint4 h) {
  return make_uint4(tc::pack_bf16(v[0], v[1]) & nonzero_mask_bf16x2(h.x),
                    tc::pack_bf16(v[2], v[3]) & nonzero_mask_bf16x2(h.y),
                    tc::pack_bf16(v[4], v[5]) & nonzero_mask_bf16x2(h.z),
                    tc::pack_bf16(v[6], v[7]) & nonzero_mask_bf16x2(h.w));
}

// Bounded wait that also gives up as soon as another role has (flag set).
__device__ __forceinline__ bool bwait(uint64_t* bar, uint32_t parity, uint32_t* flag,
                                      uint32_t* err, uint32_t spin_max) {
  for (uint32_t i = 0; i < spin_max; ++i) {
    if (tc::mbar_try(bar, parity)) return true;
    if ((i & 31u) == 31u && *((volatile uint32_t*)flag)) return false;
  }
  atomicOr(flag, 1u);
  if (err) atomicOr(err, 2u);
  return false;
}

// The slot's epilogue threads: results written to shared memory are made
// visible to the tensor cores, TMEM reads are ordered before the next MMA,
// then the thread arrives on the slot's epilogue barrier.
__device__ __forceinline__ void epi_done(uint64_t* bar) {
  tc::fence_async_smem();
  tc::fence_before();
  tc::mbar_arrive(bar);
}

__global__ void __launch_bounds__(kBwdThreads, 1)
    k_mlp_bwd_tc(MlpArgsTc a, const uint8_t* __restrict__ blob, const uint8_t* __restrict__ xt,
                 const uint32_t* __restrict__ totals, const float* __restrict__ rgb,
                 const float* __restrict__ grad_rgb, float* grad_k0, float* wpart, uint32_t* err,
                 uint32_t spin_max, int hold) {
  grid_dep_sync();
  extern __shared__ __align__(1024) uint8_t sm[];
  const int64_t M = totals[1];
  const int64_t ntiles = (M + 127) / 128;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);  // (uniform for the compiler too)
  const int64_t P = int64_t(kW) * a.din + kW + kW * kW + kW + 3 * kW + 3;
  float* pw0 = wpart + int64_t(blockIdx.x) * P;
  float* pb0 = pw0 + kW * a.din;
  float* pw1 = pb0 + kW;
  float* pb1 = pw1 + kW * kW;
  float* pw2 = pb1 + kW;
  float* pb2 = pw2 + 3 * kW;
  if (blockIdx.x >= ntiles) return;  // no partial either (active_parts)
  // this CTA's tiles: t_j = blockIdx.x + j * gridDim.x, j < nj; tile j goes to slot j & 1
  const int nj = int((ntiles - blockIdx.x + gridDim.x - 1) / gridDim.x);
  uint64_t* mbar = reinterpret_cast<uint64_t*>(sm + kBBar);  // [2] MMA stage done
  uint64_t* ebar = mbar + 2;                                  // [2] epilogue done
  uint64_t* xbar = mbar + 4;                                  // [3] X buffer landed
  uint64_t* dbar = mbar + 7;                                  // drain
  uint64_t* wbar = mbar + 8;                                  // weight tiles landed
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(sm + kBTmem);
  uint32_t* flag = reinterpret_cast<uint32_t*>(sm + kBFlag);
  uint32_t* xissued = reinterpret_cast<uint32_t*>(sm + kBXIssued);
  float* b1s = reinterpret_cast<float*>(sm + kBB1);
  if (tid < 128) b1s[tid] = a.b1[tid];
  if (tid < 256) {
    // H0 columns 128..143 of both slots: [1, 0 x 15] for every row
    const int s = tid >> 7, r = tid & 127;
    uint8_t* h0 = sm + s * kSlot + kSlH0;
    *reinterpret_cast<uint4*>(h0 + tc::kmaj(r, 128, 144)) =
        make_uint4(tc::pack_bf16(1.f, 0.f), 0u, 0u, 0u);
    *reinterpret_cast<uint4*>(h0 + tc::kmaj(r, 136, 144)) = make_uint4(0u, 0u, 0u, 0u);
  }
  if (tid == kBwdIssuer * 32) {
    *flag = 0;
    tc::mbar_init(mbar, 1);
    tc::mbar_init(mbar + 1, 1);
    tc::mbar_init(ebar, 32 * kBwdEpiWarps);
    tc::mbar_init(ebar + 1, 32 * kBwdEpiWarps);
    for (int b = 0; b < kBwdXBufs; ++b) tc::mbar_init(xbar + b, 1);
    tc::mbar_init(dbar, 1);
    tc::mbar_init(wbar, 1);
    // W0f and W1 of the forward's blob in one bulk copy
    tc::mbar_expect_tx(wbar, kBwdWBytes + kBwdW2Bytes);
    tc::bulk_g2s(sm + kBW0f, blob, kBwdWBytes, wbar);
    tc::bulk_g2s(sm + kBW2, blob + kOffW2, kBwdW2Bytes, wbar);
    // the X tiles of the first three tiles
    for (int b = 0; b < kBwdXBufs; ++b) {
      xissued[b] = b < nj ? 1u : 0u;
      if (b < nj) x_fetch(sm + kBX + b * kXTile, xt, blockIdx.x + int64_t(b) * gridDim.x, xbar + b);
    }
  }
  if (warp == kBwdIssuer) {
    tc::tmem_alloc(tmem_slot, kTmemBwdCols);
    tc::tmem_relinquish();
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t sb = tc::smem_addr(sm);
  float db2[3] = {0.f, 0.f, 0.f};
  int xdone = 0;  // X tiles the issuer saw land, in order: tile j in buffer j % kBwdXBufs
  bool wdone = false;             // the issuer saw the weight copy land

  if (warp == kBwdIssuer) {
    // ------------------------------------------------------------ MMA issuer
    // the whole warp waits, and goes on or leaves together; one elected lane issues
    if (!hold) {
      const uint32_t id_kk = tc::idesc_bf16(128, 128);               // A, B K-major
      const uint32_t id_kn = tc::idesc_bf16(128, 128, false, true);  // B MN-major
      const uint32_t id_g = tc::idesc_bf16(128, 16, false, true);    // grad k0
      const uint32_t id_w2 = tc::idesc_bf16(128, 16, true, true);    // H1^T . dl
      const uint32_t id_w1 = tc::idesc_bf16(128, 144, true, true);   // dZ1^T . [H0|1]
      const uint32_t id_w0 = tc::idesc_bf16(128, 48, true, true);    // dZ0^T . X
      uint32_t eph = 0u;  // bit s: parity of slot s's epilogue barrier
      bool w2_on = false, w1_on = false, w0_on = false;
      auto all_wait = [&](uint64_t* b, uint32_t parity) {
        return bool(__all_sync(0xffffffffu, bwait(b, parity, flag, err, spin_max)));
      };
      bool ok = wdone = all_wait(wbar, 0);
      for (int pair = 0; ok && 2 * pair < nj; ++pair) {
#pragma unroll
        for (int k = 0; k < 5; ++k) {
#pragma unroll 1
          for (int s = 0; ok && s < 2; ++s) {
            const int j = 2 * pair + s;
            if (j >= nj) continue;
            const int xb = j % kBwdXBufs;
            if (k == 0) {
              ok = all_wait(xbar + xb, (j / kBwdXBufs) & 1u);
              xdone += ok;
            } else {
              ok = all_wait(ebar + s, (eph >> s) & 1u);
              eph ^= 1u << s;
            }
            if (!ok) break;
            tc::fence_after();
            const uint32_t sl = sb + uint32_t(s) * kSlot;
            const uint32_t sx = sb + kBX + uint32_t(xb) * kXTile;
            const uint32_t tA = tmem + kTA0 + 128u * uint32_t(s);
            if (tc::elect_one()) {
              if (k == 0) {  // Z0 = X . W0f^T
#pragma unroll
                for (uint32_t q = 0; q < 3; ++q)
                  tc::mma_bf16(tA, tc::make_desc(sx + 256 * q, 128, 768),
                               tc::make_desc(sb + kBW0f + 256 * q, 128, 768), id_kk, q > 0);
              } else if (k == 1) {  // Z1 = H0 . W1^T
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                  tc::mma_bf16(tA, tc::make_desc(sl + kSlH0 + 256 * q, 128, 2304),
                               tc::make_desc(sb + kBW1 + 256 * q, 128, 2048), id_kk, q > 0);
              } else if (k == 2) {  // dZ1' = dl . W2 -> A;  dW2 += H1^T . dl
                tc::mma_bf16(tA, tc::make_desc(sl + kSlDl, 128, 256),
                             tc::make_desc(sb + kBW2, 2048, 128), id_kn, 0u);
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                  tc::mma_bf16(tmem + kTW2, tc::make_desc(sl + kSlH1 + 4096 * q, 2048, 128),
                               tc::make_desc(sl + kSlDl + 512 * q, 256, 128), id_w2,
                               (w2_on || q > 0) ? 1u : 0u);
              } else if (k == 3) {  // dH0 = dZ1 . W1;  dW1|db1 += dZ1^T . [H0|1]
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                  tc::mma_bf16(tA, tc::make_desc(sl + kSlH1 + 256 * q, 128, 2048),
                               tc::make_desc(sb + kBW1 + 4096 * q, 2048, 128), id_kn, q > 0);
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                  tc::mma_bf16(tmem + kTW1, tc::make_desc(sl + kSlH1 + 4096 * q, 2048, 128),
                               tc::make_desc(sl + kSlH0 + 4608 * q, 2304, 128), id_w1,
                               (w1_on || q > 0) ? 1u : 0u);
              } else {  // grad k0 = dZ0 . W0k;  dW0|db0 += dZ0^T . X
                const uint32_t tG = tmem + kTG0 + 16u * uint32_t(s);
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                  tc::mma_bf16(tG, tc::make_desc(sl + kSlH1 + 256 * q, 128, 2048),
                               tc::make_desc(sb + kBW0f + 1536 * q, 768, 128), id_g, q > 0);
#pragma unroll
                for (uint32_t q = 0; q < 8; ++q)
                  tc::mma_bf16(tmem + kTW0, tc::make_desc(sl + kSlH1 + 4096 * q, 2048, 128),
                               tc::make_desc(sx + 1536 * q, 768, 128), id_w0,
                               (w0_on || q > 0) ? 1u : 0u);
              }
              tc::mma_commit(mbar + s);
            }
            __syncwarp();
            w2_on = w2_on || k == 2;
            w1_on = w1_on || k == 3;
            w0_on = w0_on || k == 4;
          }
        }
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------- epilogues of slot s
    // warp (s, q4, half): TMEM lanes / tile rows 32*q4.., columns 64*half..
    const int s = warp / kBwdEpiWarps, w8 = warp % kBwdEpiWarps;
    const int q4 = w8 & 3, half = w8 >> 2;
    const int row = 32 * q4 + lane;
    const int c0 = 64 * half;
    const uint32_t tl = tmem + (uint32_t(32 * q4) << 16);
    const uint32_t tA = tl + kTA0 + 128u * uint32_t(s) + uint32_t(c0);
    const uint32_t tG = tl + kTG0 + 16u * uint32_t(s);
    uint8_t* h0 = sm + s * kSlot + kSlH0;
    uint8_t* h1 = sm + s * kSlot + kSlH1;
    uint8_t* dl = sm + s * kSlot + kSlDl;
    // 16-byte row stores only when every row starts on a 16-byte boundary
    const bool vec_k0 = (a.c0 & 3) == 0 && (reinterpret_cast<uintptr_t>(grad_k0) & 15u) == 0;
    uint32_t mph = 0;
    bool ok = true;
    for (int j = s; ok && j < nj; j += 2) {
      const int64_t mrow = (int64_t(blockIdx.x) + int64_t(j) * gridDim.x) * 128 + row;
      // sigmoid inputs of this row, read before the first wait
      float yv[3] = {0.f, 0.f, 0.f}, gv[3] = {0.f, 0.f, 0.f};
      if (mrow < M) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          yv[c] = __ldg(rgb + mrow * 3 + c);
          gv[c] = __ldg(grad_rgb + mrow * 3 + c);
        }
      }
      // ---- E0: H0 = relu(Z0) (the thread's 64 columns in one TMEM round trip)
      if (!(ok = bwait(mbar + s, mph, flag, err, spin_max))) break;
      mph ^= 1u;
      tc::fence_after();
      {
        uint32_t r[64];
#pragma unroll
        for (int q = 0; q < 4; ++q) tc::tmem_ld16_issue(tA + uint32_t(16 * q), r + 16 * q);
        tc::tmem_wait_ld();
#pragma unroll
        for (int g = 0; g < 8; ++g) {
          float v[8];
#pragma unroll
          for (int e = 0; e < 8; ++e) v[e] = __uint_as_float(r[8 * g + e]);
          *reinterpret_cast<uint4*>(h0 + tc::kmaj(row, c0 + 8 * g, 144)) =
              relu_pack8(v, nullptr, 0);
        }
      }
      epi_done(ebar + s);
      // ---- E1: H1 = relu(Z1 + b1); dl = grad_rgb * y * (1 - y)
      if (!(ok = bwait(mbar + s, mph, flag, err, spin_max))) break;
      mph ^= 1u;
      tc::fence_after();
      uint4 hp[8];  // this thread's 64 H1 values, then its dZ1 values, as BF16
#pragma unroll
      for (int cb = 0; cb < 64; cb += 32) {
        float v[32];
        tc::tmem_ld32(tA + uint32_t(cb), v);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          hp[cb / 8 + c] = relu_pack8(v + 8 * c, b1s, c0 + cb + 8 * c);
          *reinterpret_cast<uint4*>(h1 + tc::kmaj(row, c0 + cb + 8 * c, 128)) = hp[cb / 8 + c];
        }
      }
      // dl, in BF16 the A operand of dZ1' = dl . W2 and the B operand of dW2
      {
        float d[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) d[c] = gv[c] * (1.f - yv[c]) * yv[c];
        if (half == 0) {
#pragma unroll
          for (int c = 0; c < 3; ++c) db2[c] += d[c];
          *reinterpret_cast<uint4*>(dl + tc::kmaj(row, 0, 16)) =
              make_uint4(tc::pack_bf16(d[0], d[1]), tc::pack_bf16(d[2], 0.f), 0u, 0u);
          *reinterpret_cast<uint4*>(dl + tc::kmaj(row, 8, 16)) = make_uint4(0u, 0u, 0u, 0u);
        }
      }
      epi_done(ebar + s);
      // ---- E2: dZ1 = dZ1' * [H1 > 0] over H1 once the dW2 MMA has read it
      if (!(ok = bwait(mbar + s, mph, flag, err, spin_max))) break;
      mph ^= 1u;
      tc::fence_after();
#pragma unroll
      for (int cb = 0; cb < 64; cb += 32) {
        float v[32];
        tc::tmem_ld32(tA + uint32_t(cb), v);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(h1 + tc::kmaj(row, c0 + cb + 8 * c, 128)) =
              mask_pack(v + 8 * c, hp[cb / 8 + c]);
      }
      epi_done(ebar + s);
      // ---- E3: dZ0 = dH0 * [H0 > 0], over dZ1 (the thread's own H0 columns,
      // written by its E0, are read before the wait)
      uint4 hm[8];
#pragma unroll
      for (int g = 0; g < 8; ++g)
        hm[g] = *reinterpret_cast<const uint4*>(h0 + tc::kmaj(row, c0 + 8 * g, 144));
      if (!(ok = bwait(mbar + s, mph, flag, err, spin_max))) break;
      mph ^= 1u;
      tc::fence_after();
#pragma unroll
      for (int cb = 0; cb < 64; cb += 32) {
        float v[32];
        tc::tmem_ld32(tA + uint32_t(cb), v);
#pragma unroll
        for (int c = 0; c < 4; ++c)
          *reinterpret_cast<uint4*>(h1 + tc::kmaj(row, c0 + cb + 8 * c, 128)) =
              mask_pack(v + 8 * c, hm[cb / 8 + c]);
      }
      epi_done(ebar + s);
      // ---- E4: grad k0; the tile's X buffer is free again (S4 is done): it
      // takes the X tile of tile j + 3
      if (!(ok = bwait(mbar + s, mph, flag, err, spin_max))) break;
      mph ^= 1u;
      tc::fence_after();
      if (w8 == 0 && lane == 0 && j + kBwdXBufs < nj) {
        const int xb = j % kBwdXBufs;
        xissued[xb] += 1u;
        x_fetch(sm + kBX + xb * kXTile, xt, blockIdx.x + int64_t(j + kBwdXBufs) * gridDim.x,
                xbar + xb);
      }
      if (half == 0) {
        float v[16];
        tc::tmem_ld16(tG, v);
        if (mrow < M) {
          float* dst = grad_k0 + mrow * a.c0;
          if (vec_k0) {
#pragma unroll
            for (int b = 0; b < 4; ++b)
              if (4 * b < a.c0)
                reinterpret_cast<float4*>(dst)[b] =
                    make_float4(v[4 * b], v[4 * b + 1], v[4 * b + 2], v[4 * b + 3]);
          } else {
#pragma unroll
            for (int qq = 0; qq < 16; ++qq)
              if (qq < a.c0) dst[qq] = v[qq];
          }
        }
      }
      tc::fence_before();
    }
  }
  // ---------------------------------------------------------------- teardown
  __syncthreads();
  const bool failed = *((volatile uint32_t*)flag) != 0;
  if (warp == kBwdIssuer && tc::elect_one()) {
    // every MMA this thread issued completes before TMEM is released; copies
    // still in flight (a wait gave up) land before shared memory is released
    if (!hold) {
      tc::mma_commit(dbar);
      tc::mbar_wait(dbar, 0, spin_max);
    }
    if (!wdone) tc::mbar_wait(wbar, 0, spin_max);
    for (int b = 0; b < kBwdXBufs; ++b) {  // at most one copy per buffer is outstanding
      const uint32_t waits = uint32_t(xdone + kBwdXBufs - 1 - b) / kBwdXBufs;
      if (xissued[b] > waits) tc::mbar_wait(xbar + b, waits & 1u, spin_max);
    }
  }
  __syncthreads();
  // The dW1 and dW0|db0 rows are staged in shared memory (the slots' space,
  // free now) with odd row strides, so that thread n's row writes hit
  // distinct banks, and then written out row-major by consecutive threads:
  // coalesced stores, not one 32-byte sector per thread and store.
  constexpr int kS1 = kW + 1;   // dW1 row stride (floats)
  constexpr int kS0 = kXK + 1;  // dW0|db0 row stride
  float* s1 = reinterpret_cast<float*>(sm);
  float* s0 = s1 + kW * kS1;
  static_assert((kW * kS1 + kW * kS0) * 4 <= kBX, "staging fits in the slots");
  if (failed) {
    for (int64_t i = tid; i < P; i += kBwdThreads) pw0[i] = 0.f;
  } else if (warp < 8) {
    tc::fence_after();
    // partial gradients of this CTA: thread (q4, lane) holds row n = 32*q4 + lane
    const int q4 = warp & 3, half = warp >> 2;
    const int n = 32 * q4 + lane;
    const uint32_t tl = tmem + (uint32_t(32 * q4) << 16);
    float v[16];
    float* s1row = s1 + n * kS1;
    float* s0row = s0 + n * kS0;
    if (half == 0) {
      tc::tmem_ld16(tl + kTW2, v);
#pragma unroll
      for (int c = 0; c < 3; ++c) pw2[c * kW + n] = v[c];
#pragma unroll
      for (int j = 0; j < 2; ++j) {  // dW0|db0 columns 0..31
        tc::tmem_ld16(tl + kTW0 + 16 * j, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) s0row[16 * j + i] = v[i];
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // dW1 columns 0..63
        tc::tmem_ld16(tl + kTW1 + 16 * j, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) s1row[16 * j + i] = v[i];
      }
      tc::tmem_ld16(tl + kTW1 + 128, v);  // db1
      pb1[n] = v[0];
    } else {
      tc::tmem_ld16(tl + kTW0 + 32, v);  // dW0|db0 columns 32..47
#pragma unroll
      for (int i = 0; i < 16; ++i) s0row[32 + i] = v[i];
#pragma unroll
      for (int j = 4; j < 8; ++j) {  // dW1 columns 64..127
        tc::tmem_ld16(tl + kTW1 + 16 * j, v);
#pragma unroll
        for (int i = 0; i < 16; ++i) s1row[16 * j + i] = v[i];
      }
    }
  }
  __syncthreads();
  if (!failed) {
    for (int i = tid; i < kW * kW; i += kBwdThreads) pw1[i] = s1[(i >> 7) * kS1 + (i & 127)];
    for (int i = tid; i < kW * a.din; i += kBwdThreads) {
      const int n = i / a.din;
      pw0[i] = s0[n * kS0 + (i - n * a.din)];
    }
    if (tid < kW) pb0[tid] = s0[tid * kS0 + a.din];
  }

  if (!failed) {
    // db2: fixed-order sum of the per-row partials of both slots (the first X
    // buffer as scratch: no copy or MMA touches it any more)
    float* red = reinterpret_cast<float*>(sm + kBX);
    if (warp < 2 * kBwdEpiWarps && ((warp % kBwdEpiWarps) >> 2) == 0) {
      const int idx = (warp / kBwdEpiWarps) * 128 + 32 * (warp & 3) + lane;
      for (int c = 0; c < 3; ++c) red[c * 256 + idx] = db2[c];
    }
    __syncthreads();
    if (tid < 3) {
      float acc = 0.f;
      for (int i = 0; i < 256; ++i) acc += red[tid * 256 + i];
      pb2[tid] = acc;
    }
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  if (warp == kBwdIssuer) tc::tmem_dealloc(tmem, kTmemBwdCols);
}

}  // namespace

// Packs the FP32 weights into the BF16 tile blob (read by the forward and,
// transposed, by the backward).
int mlp_tc_pack(const float* w0, const float* b0, const float* w1, const float* b1,
                const float* w2, const float* b2, int c0, int dpe, void** blob,
                size_t* blob_cap, cudaStream_t st) {
  if (c0 > 16 || c0 + dpe + 1 > kXK)
    return set_error(PVDB_ERR_ARG, "the tensor-core rgbnet takes at most 16 k0 and 47 input channels");
  int rc = dev_reserve(blob, blob_cap, kPackFwdBytes);
  if (rc) return rc;
  MlpArgsTc a{w0, b0, w1, b1, w2, b2, c0, dpe, c0 + dpe};
  launch_k(k_pack, ceil_div(128 * 128, 256), 256, 0, st, a, static_cast<uint8_t*>(*blob));
  PVDB_CHECK_LAUNCH("k_pack");
  return PVDB_OK;
}

// The X tiles of rows k0rows [M, c0] (M = totals[1]) with the PE of each
// row's ray (pe [rays, pe_stride]); room for max_rows rows is reserved.
int mlp_tc_build_x(int c0, int dpe, const float* k0rows, const int32_t* ray, const float* pe,
                   int pe_stride, const uint32_t* totals, int64_t max_rows, void** xt,
                   size_t* xt_cap, cudaStream_t st) {
  if (c0 > 16 || c0 + dpe + 1 > kXK)
    return set_error(PVDB_ERR_ARG, "the tensor-core rgbnet takes at most 16 k0 and 47 input channels");
  const int64_t ntiles = (max_rows + 127) / 128;
  int rc = dev_reserve(xt, xt_cap, size_t(std::max<int64_t>(ntiles, 1)) * kXTile);
  if (rc) return rc;
  MlpArgsTc a{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, c0, dpe, c0 + dpe};
  const int grid = int(std::min<int64_t>(ceil_div(ntiles * 128 * 6, 256), int64_t(num_sms()) * 16));
  launch_k(k_build_x, std::max(grid, 1), 256, 0, st, a, k0rows, ray, pe, pe_stride, totals,
           static_cast<uint8_t*>(*xt));
  PVDB_CHECK_LAUNCH("k_build_x");
  return PVDB_OK;
}

// Forward over the rows (see mlp_tc_build_x for the inputs). packed: the blob
// already holds this call's weights; x_ready: the X tiles are already built.
int mlp_tc_forward_rows(const float* w0, const float* b0, const float* w1, const float* b1,
                        const float* w2, const float* b2, int c0, int dpe, const float* k0rows,
                        const int32_t* ray, const float* pe, int pe_stride, const uint32_t* totals,
                        int64_t max_rows, float* out, const float* rw, void** blob, size_t* blob_cap,
                        void** xt, size_t* xt_cap, uint32_t* err,
                        cudaStream_t st, int packed, int x_ready) {
  int rc = PVDB_OK;
  if (!packed && (rc = mlp_tc_pack(w0, b0, w1, b1, w2, b2, c0, dpe, blob, blob_cap, st)))
    return rc;
  if (!x_ready && (rc = mlp_tc_build_x(c0, dpe, k0rows, ray, pe, pe_stride, totals, max_rows, xt,
                                       xt_cap, st)))
    return rc;
  MlpArgsTc a{w0, b0, w1, b1, w2, b2, c0, dpe, c0 + dpe};
  PVDB_SMEM_ATTR(k_mlp_fwd_tc<false>, int(kSmFwdBytes));
  launch_k(k_mlp_fwd_tc<false>, num_sms(), kFwdThreads, kSmFwdBytes, st, a,
           static_cast<const uint8_t*>(*blob), static_cast<const uint8_t*>(*xt), RowSource{}, totals,
           out, rw, err);
  PVDB_CHECK_LAUNCH("k_mlp_fwd_tc");
  return PVDB_OK;
}

// The forward over the renderer's rows (12 BF16 feature channels, 27 PE
// values), X rows formed from src by the kernel itself.
int mlp_tc_forward_gather(const float* w0, const float* b0, const float* w1, const float* b1,
                          const float* w2, const float* b2, int c0, int dpe, const RowSource& src,
                          const uint32_t* totals, float* out, const float* rw, void** blob,
                          size_t* blob_cap, uint32_t* err, cudaStream_t st) {
  const int rc = mlp_tc_pack(w0, b0, w1, b1, w2, b2, c0, dpe, blob, blob_cap, st);
  if (rc) return rc;
  MlpArgsTc a{w0, b0, w1, b1, w2, b2, c0, dpe, c0 + dpe};
  PVDB_SMEM_ATTR(k_mlp_fwd_tc<true>, int(kSmFwdBytes));
  launch_k(k_mlp_fwd_tc<true>, num_sms(), kFwdThreads, kSmFwdBytes, st, a,
           static_cast<const uint8_t*>(*blob), nullptr, src, totals, out, rw, err);
  PVDB_CHECK_LAUNCH("k_mlp_fwd_tc<gather>");
  return PVDB_OK;
}

// Weight and k0 gradients of the rows; per-CTA partials go to wpart (grid x P
// floats), the caller sums them.
int mlp_tc_backward_rows(const float* w0, const float* b0, const float* w1, const float* b1,
                         const float* w2, const float* b2, int c0, int dpe, const float* k0rows,
                         const int32_t* ray, const float* pe, int pe_stride,
                         const uint32_t* totals, int64_t max_rows, const float* rgb,
                         const float* grad_rgb, float* grad_k0, float* wpart, int grid,
                         void** blob, size_t* blob_cap, void** xt, size_t* xt_cap, uint32_t* err,
                         cudaStream_t st, int packed, int x_ready) {
  int rc = PVDB_OK;
  if (!packed && (rc = mlp_tc_pack(w0, b0, w1, b1, w2, b2, c0, dpe, blob, blob_cap, st)))
    return rc;
  if (!x_ready && (rc = mlp_tc_build_x(c0, dpe, k0rows, ray, pe, pe_stride, totals, max_rows, xt,
                                       xt_cap, st)))
    return rc;
  MlpArgsTc a{w0, b0, w1, b1, w2, b2, c0, dpe, c0 + dpe};
  PVDB_SMEM_ATTR(k_mlp_bwd_tc, int(kSmBwdBytes));
  launch_k(k_mlp_bwd_tc, grid, kBwdThreads, kSmBwdBytes, st, a, static_cast<const uint8_t*>(*blob),
           static_cast<const uint8_t*>(*xt), totals, rgb, grad_rgb, grad_k0, wpart, err,
           debug_spin_limit(kWaitIters), debug_hold_first());
  PVDB_CHECK_LAUNCH("k_mlp_bwd_tc");
  return PVDB_OK;
}

}  // namespace pvdb
