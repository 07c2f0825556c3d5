// rgbnet: Linear(C0+Dpe -> 128) ReLU Linear(128 -> 128) ReLU Linear(128 -> 3),
// then sigmoid (dvgo.py:91-107, :354-362), evaluated on the colour rows of a
// march workspace. Layer 0 is split into the per-row k0 part and a per-ray
// part W0[:,C0:]·PE(viewdir) + b0 computed once per ray (the reference
// renderer hoists it the same way, renderer.cu:100-101).
//
// The FP32 kernels are in mlp_f32.cu, the BF16 tensor-core kernels in
// mlp_tc.cu; both leave per-CTA partial weight gradients that k_wgrad_reduce
// sums in CTA order, so the weight gradients are deterministic for a given
// grid size.
#include <algorithm>

#include "march.cuh"
#include "mlp_f32.cuh"

namespace pvdb {

constexpr int kW = 128;     // hidden width
constexpr int kMaxC0 = 16;  // k0 channels
constexpr int kMaxPe = 32;  // PE dims

// PE of a unit view direction (dvgo.py:354-355): [d, sin(d*2^i), cos(d*2^i)]
// with the frequencies innermost per axis: sin at 3 + a*npe + i, cos at
// 3 + 3*npe + a*npe + i.
// Per ray: pe[r][0:dpe] and (HPE) hpe[r][n] = b0[n] + sum_q w0[n][c0+q] * pe[r][q].
// A 128-thread block takes kPeRays rays, without those whose entry of `need`
// (NULL: all rays) is zero: each PE component is evaluated once, then thread n
// forms hpe[r][n] with its PE weights in registers, four rays at a time (the
// sums are chains of dependent FMAs; 16 rays a block keep a small batch spread
// over the SMs).
constexpr int kPeRays = 16;
template <bool HPE>
__global__ void __launch_bounds__(128)
    k_pe_hpe(const float* __restrict__ viewdirs, int R, int npe, MlpArgs a, float* pe_out,
             float* hpe, const uint32_t* __restrict__ need) {
  grid_dep_sync();
  __shared__ __align__(16) float pe_s[kPeRays][kMaxPe];
  __shared__ int list[kPeRays];
  __shared__ int count;
  const int n = threadIdx.x;
  const int r0 = blockIdx.x * kPeRays;
  if (n < 32) {
    const bool take = n < kPeRays && r0 + n < R && (!need || __ldg(need + r0 + n) != 0);
    const unsigned m = __ballot_sync(0xffffffffu, take);
    if (take) list[__popc(m & lanemask_lt())] = r0 + n;
    if (n == 0) count = __popc(m);
  }
  for (int e = n; e < kPeRays * kMaxPe; e += kW) (&pe_s[0][0])[e] = 0.f;
  __syncthreads();
  const int nr = count;
  for (int e = n; e < nr * a.dpe; e += kW) {
    const int rr = e / a.dpe, q = e - rr * a.dpe, r = list[rr];
    float v;
    if (q < 3) {
      v = viewdirs[r * 3 + q];
    } else {
      const int qq = q - 3, sc = qq / (3 * npe), rem = qq % (3 * npe), ax = rem / npe,
                i = rem % npe;
      const float x = viewdirs[r * 3 + ax] * float(1 << i);
      v = sc ? cosf(x) : sinf(x);
    }
    pe_s[rr][q] = v;
    pe_out[int64_t(r) * kMaxPe + q] = v;
  }
  if (!HPE) return;
  float w[kMaxPe];
#pragma unroll
  for (int q = 0; q < kMaxPe; ++q) w[q] = q < a.dpe ? __ldg(a.w0 + n * a.din + a.c0 + q) : 0.f;
  const float b = a.b0[n];
  __syncthreads();
  for (int rr = 0; rr < nr; rr += 4) {
    float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < kMaxPe; q += 4) {
      if (q >= a.dpe) break;  // (the padding columns are zero)
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const float4 p = *reinterpret_cast<const float4*>(&pe_s[rr + i][q]);
        s[i] = fmaf(w[q], p.x, s[i]);
        s[i] = fmaf(w[q + 1], p.y, s[i]);
        s[i] = fmaf(w[q + 2], p.z, s[i]);
        s[i] = fmaf(w[q + 3], p.w, s[i]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if (rr + i < nr) hpe[int64_t(list[rr + i]) * kW + n] = b + s[i];
  }
}

static int pe_launch(const float* viewdirs, int R, const MlpArgs& a, float* pe, float* hpe,
                     const uint32_t* need, cudaStream_t st) {
  const int npe = (a.dpe - 3) / 6;
  if (hpe)
    launch_k(k_pe_hpe<true>, ceil_div(R, kPeRays), kW, 0, st, viewdirs, R, npe, a, pe, hpe, need);
  else
    launch_k(k_pe_hpe<false>, ceil_div(R, kPeRays), kW, 0, st, viewdirs, R, npe, a, pe, hpe, need);
  PVDB_CHECK_LAUNCH("k_pe_hpe");
  return PVDB_OK;
}

// Sum of the per-CTA partials: eight interleaved running sums (partials c,
// c+8, ...) combined in a fixed order, so the loads of eight partials are in
// flight together and the result is the same on every run.
// Only the CTAs that had a tile wrote one (a batch smaller than the grid).
// 256 threads per 32 parameters: warp u sums the partials c = u, u+8, ... in
// increasing c, then the 8 warp sums combine as ((s0+s1)+(s2+s3))+((s4+s5)+(s6+s7)).
__global__ void __launch_bounds__(256)
    k_wgrad_reduce(const float* __restrict__ wpart, int grid, int tensor_cores,
                   const uint32_t* __restrict__ totals, int64_t P, float* out) {
  grid_dep_sync();
  const int nparts = active_parts(totals[1], grid, tensor_cores);
  __shared__ float part[8][33];
  const int u = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t i = blockIdx.x * 32ll + lane;
  float acc = 0.f;
  if (i < P)
    for (int c = u; c < nparts; c += 8) acc += __ldg(wpart + int64_t(c) * P + i);
  part[u][lane] = acc;
  __syncthreads();
  if (u == 0 && i < P)
    out[i] = ((part[0][lane] + part[1][lane]) + (part[2][lane] + part[3][lane])) +
             ((part[4][lane] + part[5][lane]) + (part[6][lane] + part[7][lane]));
}

__global__ void k_scatter_grads(const float* __restrict__ flat, int din, float* w0, float* b0,
                                float* w1, float* b1, float* w2, float* b2) {
  grid_dep_sync();
  const int64_t P = mlp_param_count(din);
  const int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (i >= P) return;
  int64_t o = i;
  const int64_t s0 = int64_t(kW) * din, s1 = kW, s2 = int64_t(kW) * kW, s3 = kW, s4 = 3 * kW;
  if (o < s0) { if (w0) w0[o] = flat[i]; return; }
  o -= s0;
  if (o < s1) { if (b0) b0[o] = flat[i]; return; }
  o -= s1;
  if (o < s2) { if (w1) w1[o] = flat[i]; return; }
  o -= s2;
  if (o < s3) { if (b1) b1[o] = flat[i]; return; }
  o -= s3;
  if (o < s4) { if (w2) w2[o] = flat[i]; return; }
  o -= s4;
  if (b2) b2[o] = flat[i];
}

// ------------------------------------------------------------------ host
static int mlp_grid() { return num_sms(); }

static int mlp_reserve(pvdb_march_s* m, int din) {
  int rc = dev_reserve((void**)&m->hpe, &m->hpe_cap,
                       size_t(m->max_rays) * (kW + kMaxPe) * 4);
  if (rc) return rc;
  const size_t P = size_t(mlp_param_count(din));
  return dev_reserve((void**)&m->wpart, &m->wpart_cap, (size_t(mlp_grid()) + 1) * P * 4);
}

int mlp_tc_pack(const float* w0, const float* b0, const float* w1, const float* b1,
                const float* w2, const float* b2, int c0, int dpe, void** blob,
                size_t* blob_cap, cudaStream_t st);
int mlp_tc_forward_rows(const float* w0, const float* b0, const float* w1, const float* b1,
                        const float* w2, const float* b2, int c0, int dpe, const float* k0rows,
                        const int32_t* ray, const float* pe, int pe_stride, const uint32_t* totals,
                        int64_t max_rows, float* out, const float* rw, void** blob, size_t* blob_cap,
                        void** xt, size_t* xt_cap, uint32_t* err,
                        cudaStream_t st, int packed, int x_ready);

// Inputs of the rgbnet that depend only on the rays and the weights: the
// per-ray PE (FP32 path: and hpe) and, BF16 path, the packed BF16 weight
// tiles of the forward and the backward. The train step runs this on a side
// stream while the march runs.
int mlp_prepare(pvdb_march_s* m, const MlpArgs& a, const float* viewdirs, int R, int precision,
                cudaStream_t st) {
  if (R <= 0) return PVDB_OK;
  int rc = mlp_reserve(m, a.din);
  if (rc) return rc;
  float* pe = m->hpe + size_t(m->max_rays) * kW;
  if ((rc = pe_launch(viewdirs, R, a, pe, precision == 1 ? nullptr : m->hpe, nullptr, st))) return rc;
  if (precision == 1)
    return mlp_tc_pack(a.w0, a.b0, a.w1, a.b1, a.w2, a.b2, a.c0, a.dpe, &m->mlp_packed,
                       &m->mlp_packed_cap, st);
  return PVDB_OK;
}

// The per-ray PE that mlp_prepare writes (stride floats per ray), and the X
// tiles of the tensor-core path reserved for the workspace's rows.
const float* mlp_pe_buffer(pvdb_march_s* m, int* stride) {
  *stride = kMaxPe;
  return m->hpe ? m->hpe + size_t(m->max_rays) * kW : nullptr;
}
int mlp_reserve_x(pvdb_march_s* m) {
  const int64_t ntiles = (m->slots + 127) / 128;
  return dev_reserve(&m->mlp_xt, &m->mlp_xt_cap, size_t(std::max<int64_t>(ntiles, 1)) * kRgbXTile);
}

// prepared: mlp_prepare already ran for these rays and weights; x_ready: the
// BF16 X tiles are already built (march_k0_x).
int mlp_forward_impl(pvdb_march_s* m, const MlpArgs& a, const float* k0rows,
                     const float* viewdirs, float* rgb, int precision, cudaStream_t st,
                     bool prepared, bool x_ready) {
  const int R = m->n_rays;
  if (R <= 0) return PVDB_OK;
  int rc = mlp_reserve(m, a.din);
  if (rc) return rc;
  float* hpe = m->hpe;
  float* pe = m->hpe + size_t(m->max_rays) * kW;
  if (!prepared && (rc = pe_launch(viewdirs, R, a, pe, precision == 1 ? nullptr : hpe, nullptr, st)))
    return rc;
  if (precision == 1)
    return mlp_tc_forward_rows(a.w0, a.b0, a.w1, a.b1, a.w2, a.b2, a.c0, a.dpe, k0rows,
                               m->w.r_ray, pe, kMaxPe, m->w.totals, m->slots, rgb, nullptr,
                               &m->mlp_packed, &m->mlp_packed_cap, &m->mlp_xt, &m->mlp_xt_cap,
                               m->w.totals + 3, st, prepared ? 1 : 0, x_ready ? 1 : 0);
  return mlp_f32_forward(a, k0rows, m->w.r_ray, hpe, m->w.totals, rgb, nullptr, st);
}

// Rows from the merged renderer; M = totals[1]; out [M, 3] gets each row's
// contribution rw / (1 + exp(-logit)). FP32: k0rows [M, c0], ray [M] ->
// viewdirs [R,3], hpe_buf holds R*(128+32) floats; the rays whose entry of
// `need` is zero have no row. BF16: the X tiles in *xt are already built.
int mlp_forward_rows(const MlpArgs& a, const float* k0rows, const int32_t* ray,
                     const float* viewdirs, int R, const uint32_t* need, const uint32_t* totals,
                     int64_t max_rows, const float* rw, float* out, float* hpe_buf, int precision,
                     void** blob, size_t* blob_cap, void** xt, size_t* xt_cap, uint32_t* err,
                     cudaStream_t st) {
  if (R <= 0) return PVDB_OK;
  if (precision == 1)
    return mlp_tc_forward_rows(a.w0, a.b0, a.w1, a.b1, a.w2, a.b2, a.c0, a.dpe, k0rows, ray,
                               nullptr, kMaxPe, totals, max_rows, out, rw, blob, blob_cap, xt,
                               xt_cap, err, st, 0, 1);
  float* pe = hpe_buf + size_t(R) * kW;
  const int rc = pe_launch(viewdirs, R, a, pe, hpe_buf, need, st);
  if (rc) return rc;
  return mlp_f32_forward(a, k0rows, ray, hpe_buf, totals, out, rw, st);
}

int mlp_tc_backward_rows(const float* w0, const float* b0, const float* w1, const float* b1,
                         const float* w2, const float* b2, int c0, int dpe, const float* k0rows,
                         const int32_t* ray, const float* pe, int pe_stride,
                         const uint32_t* totals, int64_t max_rows, const float* rgb,
                         const float* grad_rgb, float* grad_k0, float* wpart, int grid,
                         void** blob, size_t* blob_cap, void** xt, size_t* xt_cap, uint32_t* err,
                         cudaStream_t st, int packed, int x_ready);

// hpe/pe of the current forward must still be in the workspace; prepared: the
// BF16 backward tiles were packed by mlp_prepare.
int mlp_backward_impl(pvdb_march_s* m, const MlpArgs& a, const float* k0rows, const float* rgb,
                      const float* grad_rgb, float* grad_k0, float* grad_flat, int precision,
                      cudaStream_t st, bool prepared) {
  const int R = m->n_rays;
  const int64_t P = mlp_param_count(a.din);
  if (R <= 0) {
    PVDB_CHECK_CUDA(cudaMemsetAsync(grad_flat, 0, P * 4, st));
    return PVDB_OK;
  }
  int rc = mlp_reserve(m, a.din);
  if (rc) return rc;
  const int G = mlp_grid();
  if (precision == 1) {
    rc = mlp_tc_backward_rows(a.w0, a.b0, a.w1, a.b1, a.w2, a.b2, a.c0, a.dpe, k0rows, m->w.r_ray,
                              m->hpe + size_t(m->max_rays) * kW, kMaxPe, m->w.totals, m->slots,
                              rgb, grad_rgb, grad_k0, m->wpart, G, &m->mlp_packed,
                              &m->mlp_packed_cap, &m->mlp_xt, &m->mlp_xt_cap, m->w.totals + 3, st,
                              prepared ? 1 : 0, prepared ? 1 : 0);
    if (rc) return rc;
    launch_k(k_wgrad_reduce, ceil_div(P, 32), 256, 0, st, m->wpart, G, precision, m->w.totals,
             P, grad_flat);
    PVDB_CHECK_LAUNCH("k_wgrad_reduce");
    return PVDB_OK;
  }
  rc = mlp_f32_backward(a, k0rows, m->w.r_ray, m->hpe, m->hpe + size_t(m->max_rays) * kW,
                        m->w.totals, rgb, grad_rgb, grad_k0, m->wpart, G, st);
  if (rc) return rc;
  launch_k(k_wgrad_reduce, ceil_div(P, 32), 256, 0, st, m->wpart, G, precision, m->w.totals,
             P, grad_flat);
  PVDB_CHECK_LAUNCH("k_wgrad_reduce");
  return PVDB_OK;
}

int mlp_args_from(const pvdb_mlp_weights* w, MlpArgs& a) {
  PVDB_REQUIRE(w && w->w0 && w->b0 && w->w1 && w->b1 && w->w2 && w->b2, "null MLP weight");
  PVDB_REQUIRE(w->width == kW, "rgbnet width must be 128");
  PVDB_REQUIRE(w->c0 > 0 && w->c0 <= kMaxC0, "k0 channels must be in 1..16");
  PVDB_REQUIRE(w->pe >= 0 && w->pe <= 4, "viewbase_pe must be in 0..4");
  a.w0 = w->w0; a.b0 = w->b0; a.w1 = w->w1; a.b1 = w->b1; a.w2 = w->w2; a.b2 = w->b2;
  a.c0 = w->c0;
  a.dpe = 3 + 6 * w->pe;
  a.din = a.c0 + a.dpe;
  return PVDB_OK;
}

}  // namespace pvdb

using namespace pvdb;

extern "C" {

int pvdb_mlp_forward(pvdb_march m, const pvdb_mlp_weights* w, const float* k0,
                     const float* viewdirs, float* rgb, int32_t precision, pvdb_stream s) {
  clear_error();
  PVDB_REQUIRE(m && viewdirs && rgb, "null argument");
  PVDB_REQUIRE(m->has_fwd, "mlp before march forward");
  PVDB_REQUIRE(m->k0 && m->k0->C == w->c0, "k0 channels differ from the march's k0 grid");
  PVDB_REQUIRE(precision == 0 || precision == 1, "precision must be 0 or 1");
  MlpArgs a;
  int rc = mlp_args_from(w, a);
  if (rc) return rc;
  return mlp_forward_impl(m, a, k0 ? k0 : m->w.r_k0, viewdirs, rgb, precision, as_stream(s), false,
                          false);
}

int pvdb_mlp_backward(pvdb_march m, const pvdb_mlp_weights* w, const float* k0,
                      const float* viewdirs, const float* rgb, const float* grad_rgb,
                      pvdb_mlp_grads* g, float* grad_k0, int32_t precision, pvdb_stream s) {
  clear_error();
  PVDB_REQUIRE(m && viewdirs && rgb && grad_rgb && g && grad_k0, "null argument");
  PVDB_REQUIRE(m->has_fwd, "mlp before march forward");
  PVDB_REQUIRE(m->k0 && m->k0->C == w->c0, "k0 channels differ from the march's k0 grid");
  MlpArgs a;
  int rc = mlp_args_from(w, a);
  if (rc) return rc;
  PVDB_REQUIRE(precision == 0 || precision == 1, "precision must be 0 (fp32) or 1 (bf16)");
  cudaStream_t st = as_stream(s);
  // hpe/pe depend only on the weights and viewdirs: recompute them so the
  // backward does not rely on a preceding forward call of the same weights.
  rc = mlp_reserve(m, a.din);
  if (rc) return rc;
  if (m->n_rays > 0 &&
      (rc = pe_launch(viewdirs, m->n_rays, a, m->hpe + size_t(m->max_rays) * kW,
                      precision == 1 ? nullptr : m->hpe, nullptr, as_stream(s))))
    return rc;
  const int64_t P = mlp_param_count(a.din);
  float* flat = m->wpart + int64_t(mlp_grid()) * P;  // spare slot after the partials
  rc = mlp_backward_impl(m, a, k0 ? k0 : m->w.r_k0, rgb, grad_rgb, grad_k0, flat, precision, st,
                         false);
  if (rc) return rc;
  launch_k(k_scatter_grads, ceil_div(P, 256), 256, 0, st, flat, a.din, g->w0, g->b0, g->w1, g->b1,
           g->w2, g->b2);
  PVDB_CHECK_LAUNCH("k_scatter_grads");
  return PVDB_OK;
}

}  // extern "C"
