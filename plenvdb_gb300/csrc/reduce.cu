// Device-wide scan, stable LSD radix sort and the generic point backward
// (DensityVDB/ColorVDB backward, plenvdb.h:468-485, :557-573).
//
// Sizes may live on the device (n_dev != NULL): kernels are launched for the
// host-side maximum with a fixed, SM-count-sized grid and loop over the tiles
// that the device-side count actually needs, so the fused training step never
// synchronises with the host.
#include <algorithm>

#include <atomic>

#include "reduce.cuh"

namespace pvdb {

static int g_num_sms = 0;
int num_sms() {
  if (!g_num_sms) {
    int dev = 0, n = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    g_num_sms = n > 0 ? n : 148;
  }
  return g_num_sms;
}

__device__ __forceinline__ int64_t eff_size(int64_t n_max, const uint32_t* n_dev) {
  return n_dev ? min(n_max, (int64_t)*n_dev) : n_max;
}

// ------------------------------------------------------------------- scan
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;  // 4096

__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* total) {
  __shared__ uint32_t warp_sums[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  if (lane == 31) warp_sums[wid] = x;
  __syncthreads();
  if (wid == 0) {
    const int nw = blockDim.x >> 5;
    uint32_t s = lane < nw ? warp_sums[lane] : 0u;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      uint32_t y = __shfl_up_sync(0xffffffffu, s, o);
      if (lane >= o) s += y;
    }
    if (lane < nw) warp_sums[lane] = s;  // inclusive
  }
  __syncthreads();
  const uint32_t warp_excl = wid ? warp_sums[wid - 1] : 0u;
  if (total) *total = warp_sums[(blockDim.x >> 5) - 1];
  const uint32_t r = warp_excl + x - v;
  __syncthreads();
  return r;
}

__global__ void k_scan_reduce(const uint32_t* __restrict__ in, int64_t n_max,
                              const uint32_t* n_dev, uint32_t* partial) {
  grid_dep_sync();
  const int64_t n = eff_size(n_max, n_dev);
  const int64_t ntiles = (n + kScanTile - 1) / kScanTile;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t base = t * kScanTile + int64_t(threadIdx.x) * kScanItems;
    uint32_t s = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q)
      if (base + q < n) s += in[base + q];
    uint32_t tot;
    block_exclusive_scan(s, &tot);
    if (threadIdx.x == 0) partial[t] = tot;
  }
}

__global__ void k_scan_partials(uint32_t* partial, int64_t n_max, const uint32_t* n_dev,
                                uint32_t* total) {
  grid_dep_sync();
  __shared__ uint32_t carry_s;
  const int64_t n = eff_size(n_max, n_dev);
  const int64_t nb = (n + kScanTile - 1) / kScanTile;
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (int64_t base = 0; base < nb; base += blockDim.x) {
    const int64_t i = base + threadIdx.x;
    const uint32_t v = i < nb ? partial[i] : 0u;
    uint32_t tot;
    const uint32_t ex = block_exclusive_scan(v, &tot);
    const uint32_t c = carry_s;
    if (i < nb) partial[i] = c + ex;
    __syncthreads();
    if (threadIdx.x == 0) carry_s = c + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0 && total) *total = carry_s;
}

__global__ void k_scan_apply(const uint32_t* __restrict__ in, uint32_t* out, int64_t n_max,
                             const uint32_t* n_dev, const uint32_t* __restrict__ partial) {
  grid_dep_sync();
  const int64_t n = eff_size(n_max, n_dev);
  const int64_t ntiles = (n + kScanTile - 1) / kScanTile;
  for (int64_t t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const int64_t base = t * kScanTile + int64_t(threadIdx.x) * kScanItems;
    uint32_t v[kScanItems];
    uint32_t s = 0;
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
      v[q] = base + q < n ? in[base + q] : 0u;
      s += v[q];
    }
    uint32_t run = block_exclusive_scan(s, nullptr) + partial[t];
#pragma unroll
    for (int q = 0; q < kScanItems; ++q) {
      if (base + q < n) out[base + q] = run;
      run += v[q];
    }
  }
}

// Single-block scan for short inputs: 1024 threads walk the input in chunks
// of 8192 with a running carry (one launch instead of three). Each chunk goes
// through shared memory so that global loads and stores are coalesced; thread
// t scans elements 8t .. 8t+7 of the chunk (the padded index spreads them
// over the banks).
constexpr int kScan1Threads = 1024;
constexpr int kScan1Items = 8;
constexpr int64_t kScan1Max = 262144;  // inputs up to this length take the one-block path

__device__ __forceinline__ int scan1_pad(int i) { return i + (i >> 5); }

__global__ void __launch_bounds__(kScan1Threads)
    k_scan_single(const uint32_t* __restrict__ in, uint32_t* out, int64_t n_max,
                  const uint32_t* n_dev, uint32_t* total) {
  grid_dep_sync();
  constexpr int kChunk = kScan1Threads * kScan1Items;
  __shared__ uint32_t buf[kChunk + kChunk / 32];
  __shared__ uint32_t carry_s;
  const int64_t n = eff_size(n_max, n_dev);
  const int t = threadIdx.x;
  if (t == 0) carry_s = 0;
  __syncthreads();
  for (int64_t c0 = 0; c0 < n; c0 += kChunk) {
#pragma unroll
    for (int q = 0; q < kScan1Items; ++q) {
      const int e = q * kScan1Threads + t;
      buf[scan1_pad(e)] = c0 + e < n ? in[c0 + e] : 0u;
    }
    __syncthreads();
    uint32_t v[kScan1Items];
    uint32_t sum = 0;
#pragma unroll
    for (int q = 0; q < kScan1Items; ++q) {
      v[q] = buf[scan1_pad(t * kScan1Items + q)];
      sum += v[q];
    }
    uint32_t tot;
    uint32_t run = block_exclusive_scan(sum, &tot) + carry_s;
#pragma unroll
    for (int q = 0; q < kScan1Items; ++q) {
      buf[scan1_pad(t * kScan1Items + q)] = run;
      run += v[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kScan1Items; ++q) {
      const int e = q * kScan1Threads + t;
      if (c0 + e < n) out[c0 + e] = buf[scan1_pad(e)];
    }
    __syncthreads();
    if (t == 0) carry_s += tot;
    __syncthreads();
  }
  if (t == 0 && total) *total = carry_s;
}

int scan_exclusive_u32(const uint32_t* in, uint32_t* out, int64_t n, uint32_t* total,
                       uint32_t** partial, size_t* partial_cap, cudaStream_t st) {
  return scan_exclusive_u32_dev(in, out, n, nullptr, total, partial, partial_cap, st);
}

int scan_exclusive_u32_dev(const uint32_t* in, uint32_t* out, int64_t n_max,
                           const uint32_t* n_dev, uint32_t* total, uint32_t** partial,
                           size_t* partial_cap, cudaStream_t st) {
  if (n_max <= 0) {
    if (total) PVDB_CHECK_CUDA(cudaMemsetAsync(total, 0, 4, st));
    return PVDB_OK;
  }
  if (n_max <= kScan1Max) {
    launch_k(k_scan_single, 1, kScan1Threads, 0, st, in, out, n_max, n_dev, total);
    PVDB_CHECK_LAUNCH("k_scan_single");
    return PVDB_OK;
  }
  const int64_t nb = (n_max + kScanTile - 1) / kScanTile;
  int rc = dev_reserve((void**)partial, partial_cap, size_t(nb) * 4);
  if (rc) return rc;
  const int grid = int(std::min<int64_t>(nb, int64_t(num_sms()) * 8));
  launch_k(k_scan_reduce, grid, kScanThreads, 0, st, in, n_max, n_dev, *partial);
  launch_k(k_scan_partials, 1, 1024, 0, st, *partial, n_max, n_dev, total);
  launch_k(k_scan_apply, grid, kScanThreads, 0, st, in, out, n_max, n_dev, *partial);
  PVDB_CHECK_LAUNCHES("scan", 3);
  return PVDB_OK;
}

// ------------------------------------------------------------- radix sort
// Stable LSD radix sort, 8-bit digits, one kernel per digit pass ("onesweep"):
//   k_os_init     zeroes the per-pass tile status words, digit histograms and
//                 tile counters for the tiles the device-side count needs;
//   k_os_hist     builds the digit histograms of every pass in one read;
//   k_os_scatter  per pass: CTAs take 1024-key tiles in order from a counter,
//                 count the tile's digits, publish them, and find the tile's
//                 exclusive prefix per digit by looking back over the earlier
//                 tiles' published counts (decoupled look-back); then scatter
//                 stably (tile order, and (warp, round, lane) = index order
//                 inside a tile).
// A tile publishes its own count before it waits on anyone, and a tile only
// waits on tiles taken earlier (already running), so every wait ends; each is
// still bounded, and one that gives up sets an error flag.
constexpr int kRsWarps = kRsThreads / 32;
constexpr uint32_t kOsAgg = 0x40000000u;     // status: tile count published
constexpr uint32_t kOsPrefix = 0x80000000u;  // status: inclusive prefix published
constexpr uint32_t kOsValue = 0x3FFFFFFFu;
constexpr uint32_t kOsSpinMax = 1u << 24;

// Scratch words after the status array: ghist [npass][256], counters
// [npass], n, error flag.
struct OsLayout {
  int64_t ntiles_max;
  int npass;
  int64_t status, ghist, counters, n, err, words;
};
static OsLayout os_layout(int64_t n_max, int npass) {
  OsLayout L;
  L.ntiles_max = (n_max + kRsTile - 1) / kRsTile;
  L.npass = npass;
  L.status = 0;
  L.ghist = L.status + int64_t(npass) * L.ntiles_max * kRsBins;
  L.counters = L.ghist + int64_t(npass) * kRsBins;
  L.n = L.counters + npass;
  L.err = L.n + 1;
  L.words = L.err + 1;
  return L;
}

__global__ void k_os_init(int64_t n_max, const uint32_t* n_dev, int npass, int64_t ntiles_max,
                          uint32_t* scratch, OsLayout L) {
  grid_dep_sync();
  const int64_t n = eff_size(n_max, n_dev);
  const int64_t ntiles = (n + kRsTile - 1) / kRsTile;
  const int64_t per = ntiles * kRsBins;
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < int64_t(npass) * per;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int64_t p = i / per, r = i - p * per;
    scratch[L.status + p * ntiles_max * kRsBins + r] = 0u;
  }
  const int64_t t = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (t < int64_t(npass) * kRsBins) scratch[L.ghist + t] = 0u;
  if (t < npass) scratch[L.counters + t] = 0u;
  if (t == 0) {
    scratch[L.n] = uint32_t(n);
    scratch[L.err] = 0u;
  }
}

__global__ void __launch_bounds__(kRsThreads)
    k_os_hist(const uint32_t* __restrict__ keys, int npass, uint32_t* scratch, OsLayout L) {
  grid_dep_sync();
  __shared__ uint32_t h[4][kRsBins];
  const int64_t n = scratch[L.n];
  for (int q = threadIdx.x; q < 4 * kRsBins; q += blockDim.x) (&h[0][0])[q] = 0u;
  __syncthreads();
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const uint32_t k = keys[i];
    for (int p = 0; p < npass; ++p) atomicAdd(&h[p][(k >> (8 * p)) & 255u], 1u);
  }
  __syncthreads();
  for (int p = 0; p < npass; ++p) {
    const uint32_t c = h[p][threadIdx.x];
    if (c) atomicAdd(scratch + L.ghist + p * kRsBins + threadIdx.x, c);
  }
}

__global__ void __launch_bounds__(kRsThreads)
    k_os_scatter(const uint32_t* __restrict__ kin, const uint32_t* __restrict__ vin, int pass,
                 uint32_t* scratch, OsLayout L, uint32_t* kout, uint32_t* vout, uint32_t* err,
                 uint32_t spin_max, int hold_first) {
  grid_dep_sync();
  // an earlier pass gave up: its order is wrong, so this one does nothing
  if (*(volatile uint32_t*)err) return;
  __shared__ uint32_t wh[kRsWarps][kRsBins];
  __shared__ uint32_t gbase[kRsBins];
  __shared__ uint32_t tile_s;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, d = threadIdx.x;
  const int shift = 8 * pass;
  const int64_t n = scratch[L.n];
  const int64_t ntiles = (n + kRsTile - 1) / kRsTile;
  volatile uint32_t* status = scratch + L.status + int64_t(pass) * L.ntiles_max * kRsBins;
  const unsigned lt = lanemask_lt();
  // bucket bases of this pass: exclusive scan of the digit histogram
  {
    uint32_t tot;
    gbase[d] = block_exclusive_scan(scratch[L.ghist + pass * kRsBins + d], &tot);
  }
  for (;;) {
    if (threadIdx.x == 0) tile_s = atomicAdd(scratch + L.counters + pass, 1u);
    for (int q = threadIdx.x; q < kRsWarps * kRsBins; q += kRsThreads) (&wh[0][0])[q] = 0;
    __syncthreads();
    const int64_t t = tile_s;
    if (t >= ntiles) break;
    const int64_t wbase = t * kRsTile + int64_t(w) * (kRsRounds * 32);
    uint32_t key[kRsRounds];
#pragma unroll
    for (int r = 0; r < kRsRounds; ++r) {
      const int64_t i = wbase + r * 32 + lane;
      key[r] = i < n ? kin[i] : 0u;
    }
    // per-warp digit histogram
#pragma unroll
    for (int r = 0; r < kRsRounds; ++r) {
      const bool valid = wbase + r * 32 + lane < n;
      const uint32_t dg = valid ? ((key[r] >> shift) & 255u) : 256u;
      const unsigned peers = __match_any_sync(0xffffffffu, dg);
      if (valid && lane == __ffs(peers) - 1) wh[w][dg] += __popc(peers);
      __syncwarp();
    }
    __syncthreads();
    // thread d: tile count, publish, look back, publish the inclusive prefix
    {
      uint32_t cnt = 0;
#pragma unroll
      for (int q = 0; q < kRsWarps; ++q) cnt += wh[q][d];
      volatile uint32_t* my = status + t * kRsBins + d;
      if (t == 0) {
        if (!hold_first) *my = kOsPrefix | cnt;  // (the test hook withholds it)
      } else {
        *my = kOsAgg | cnt;
      }
      uint32_t acc = 0;
      for (int64_t tt = t - 1; tt >= 0; --tt) {
        uint32_t v = status[tt * kRsBins + d];
        for (uint32_t it = 0; v == 0u; ++it) {
          if (it >= spin_max) {
            atomicOr(err, 4u);
            v = kOsPrefix;  // give up: leave the positions wrong but finish
            break;
          }
          v = status[tt * kRsBins + d];
        }
        acc += v & kOsValue;
        if (v & kOsPrefix) break;
      }
      if (t > 0) *my = kOsPrefix | (acc + cnt);
      // per-warp exclusive offsets of this digit
      uint32_t run = gbase[d] + acc;
#pragma unroll
      for (int q = 0; q < kRsWarps; ++q) {
        const uint32_t c = wh[q][d];
        wh[q][d] = run;
        run += c;
      }
    }
    __syncthreads();
    // stable ranks and scatter
#pragma unroll
    for (int r = 0; r < kRsRounds; ++r) {
      const int64_t i = wbase + r * 32 + lane;
      const bool valid = i < n;
      const uint32_t dg = valid ? ((key[r] >> shift) & 255u) : 256u;
      const unsigned peers = __match_any_sync(0xffffffffu, dg);
      uint32_t pos = 0;
      if (valid) pos = wh[w][dg] + __popc(peers & lt);
      __syncwarp();
      if (valid && lane == __ffs(peers) - 1) wh[w][dg] += __popc(peers);
      __syncwarp();
      if (valid) {
        kout[pos] = key[r];
        vout[pos] = vin ? vin[i] : uint32_t(i);
      }
    }
    __syncthreads();
  }
}

int slot_key_bits(int64_t nslots) {
  int b = 1;
  while ((int64_t(1) << b) <= nslots) ++b;
  return b;
}

int radix_sort_pairs_dev(ReduceScratch& rs, int64_t n_max, const uint32_t* n_dev, int key_bits,
                         bool iota_vals, int* out_buf, cudaStream_t st, uint32_t** status) {
  *out_buf = 0;
  if (status) *status = nullptr;
  if (n_max <= 0) return PVDB_OK;
  const int npass = (key_bits + 7) / 8;
  if (npass < 1 || npass > 4) return set_error(PVDB_ERR_ARG, "radix sort takes 1..32 key bits");
  const OsLayout L = os_layout(n_max, npass);
  int rc = dev_reserve((void**)&rs.hist, &rs.hist_cap, size_t(L.words) * 4);
  if (rc) return rc;
  uint32_t* sc = rs.hist;
  uint32_t* errp = sc + L.err;
  if (status) *status = errp;
  const uint32_t spin = debug_spin_limit(kOsSpinMax);
  const int hold = debug_hold_first();
  const int g_init = int(std::min<int64_t>(
      std::max<int64_t>(ceil_div(int64_t(npass) * L.ntiles_max * kRsBins, 256), 1),
      int64_t(num_sms()) * 8));
  launch_k(k_os_init, g_init, 256, 0, st, n_max, n_dev, npass, L.ntiles_max, sc, L);
  PVDB_CHECK_LAUNCH("k_os_init");
  const int g_hist = int(std::min<int64_t>(ceil_div(n_max, kRsThreads), int64_t(num_sms()) * 4));
  launch_k(k_os_hist, g_hist, kRsThreads, 0, st, rs.keys[0], npass, sc, L);
  PVDB_CHECK_LAUNCH("k_os_hist");
  const int grid = int(std::min<int64_t>(L.ntiles_max, int64_t(num_sms()) * 4));
  int cur = 0;
  for (int p = 0; p < npass; ++p) {
    launch_k(k_os_scatter, grid, kRsThreads, 0, st, rs.keys[cur],
             (p == 0 && iota_vals) ? nullptr : rs.vals[cur], p, sc, L, rs.keys[cur ^ 1],
             rs.vals[cur ^ 1], errp, spin, hold);
    PVDB_CHECK_LAUNCH("k_os_scatter");
    cur ^= 1;
  }
  *out_buf = cur;
  return PVDB_OK;
}

int radix_sort_words(int64_t n_max, int key_bits) {
  return int(os_layout(n_max, (key_bits + 7) / 8).words);
}

int radix_sort_pairs(ReduceScratch& rs, int64_t n, int key_bits, bool iota_vals, int* out_buf,
                     cudaStream_t st, uint32_t** status) {
  return radix_sort_pairs_dev(rs, n, nullptr, key_bits, iota_vals, out_buf, st, status);
}

int scratch_reserve(ReduceScratch& rs, int64_t n) {
  if (rs.cap >= size_t(n) && rs.keys[0]) return PVDB_OK;
  for (int b = 0; b < 2; ++b) {
    dev_free(rs.keys[b]);
    dev_free(rs.vals[b]);
    rs.keys[b] = rs.vals[b] = nullptr;
  }
  rs.cap = 0;
  const size_t want = std::max<size_t>(size_t(n), 4096);
  int rc;
  for (int b = 0; b < 2; ++b) {
    if ((rc = dev_alloc((void**)&rs.keys[b], want * 4))) return rc;
    if ((rc = dev_alloc((void**)&rs.vals[b], want * 4))) return rc;
  }
  rs.cap = want;
  return PVDB_OK;
}

int reduce_reserve(pvdb_grid_s* g, int64_t n) { return scratch_reserve(g->red, n); }

void free_scratch(ReduceScratch& rs) {
  for (int b = 0; b < 2; ++b) {
    dev_free(rs.keys[b]);
    dev_free(rs.vals[b]);
    rs.keys[b] = rs.vals[b] = nullptr;
  }
  dev_free(rs.hist);
  dev_free(rs.partial);
  dev_free(rs.cells);
  dev_free(rs.rec);
  dev_free(rs.npts);
  dev_free(rs.mark);
  rs.hist = rs.partial = rs.npts = rs.mark = nullptr;
  rs.cells = nullptr;
  rs.rec = nullptr;
  rs.cap = rs.hist_cap = rs.partial_cap = rs.cells_cap = rs.rec_cap = 0;
  rs.epoch = 0;
}

// ------------------------------------------------- generic point backward
struct PointSrc {
  const float* xs;
  const float* ys;
  const float* zs;
  const float* g;
  int C;
  bool vec;  // 12-channel gradients on 16-byte boundaries
  __device__ __forceinline__ void pos(int64_t s, float& x, float& y, float& z) const {
    x = xs[s]; y = ys[s]; z = zs[s];
  }
  __device__ __forceinline__ float gd(int64_t s) const { return g[s]; }
  __device__ __forceinline__ bool has_c(int64_t) const { return true; }
  __device__ __forceinline__ float gc(int64_t s, int ch) const { return g[s * C + ch]; }
};

namespace {
std::atomic<uint32_t> g_dbg_spin{0};
std::atomic<int> g_dbg_hold{0};
}  // namespace

uint32_t debug_spin_limit(uint32_t builtin) {
  const uint32_t v = g_dbg_spin.load();
  return v ? v : builtin;
}

int debug_hold_first() { return g_dbg_hold.load() == 1 ? 1 : 0; }
int debug_hold_staging() { return g_dbg_hold.load() == 2 ? 1 : 0; }

int read_wait_status(const uint32_t* status, cudaStream_t st, const char* what) {
  uint32_t h = 0;
  if (status) PVDB_CHECK_CUDA(cudaMemcpyAsync(&h, status, 4, cudaMemcpyDeviceToHost, st));
  PVDB_CHECK_CUDA(cudaStreamSynchronize(st));
  if (h) return set_error(PVDB_ERR_TIMEOUT, what);
  return PVDB_OK;
}

__global__ void k_point_keys(GridView gv, const float* __restrict__ xs, const float* __restrict__ ys,
                             const float* __restrict__ zs, int64_t n, uint32_t* keys) {
  grid_dep_sync();
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (p >= n) return;
  emit_corner_keys(gv, xs[p], ys[p], zs[p], keys, p);
}

// The point backward sums, for every voxel, the contributions of its points in
// point order. A point touches the 8 corners of one cell, and a voxel's points
// are those of the 8 cells around it: sorting the points by cell (one key a
// point, not eight) and merging a voxel's 8 cells by point id gives the same
// order, so the same bits, as sorting the 8 n (slot, corner) pairs
// (noalloc.cu). Cells are (i, j, k) in [-1, 8 ldim): their keys are leaf-major
// over a lattice of one more leaf per axis. Points of a scalar grid with a zero
// gradient add nothing and are dropped first.
//   density, 2.4 M points of which 6% carry a gradient, 160^3: 1250 -> 96 us;
//   12 channels, 149 k points: 220 -> 88 us (kernel times)

// The merge of the up to 8 point lists around one voxel: list c is the points
// of the cell that has the voxel as corner c, at positions pos[c] .. end[c];
// ids(pos) gives a point's id. A few points are taken first and then
// loaded together: their loads do not wait for one another, only the sums do.

// A point as the sums read it: cell-relative position, gradient of up to 12
// channels (density: g[0]).
struct PointTerm {
  float u, v, w;
  float g[12];
};

__device__ __forceinline__ float corner_scale(const PointTerm& t, int corner) {
  int di, dj, dk;
  corner_delta(corner, di, dj, dk);
  return __fmul_rn(__fmul_rn(di ? t.u : 1.f - t.u, dj ? t.v : 1.f - t.v), dk ? t.w : 1.f - t.w);
}

template <bool SCALAR, int BATCH, class Ids, class Load>
__device__ __forceinline__ void merge_lists(const Ids& ids, const Load& load,
                                            const uint32_t first[8], const uint32_t end[8],
                                            float acc[12], bool& any) {
  uint32_t head[8], pos[8];
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    pos[c] = first[c];
    head[c] = first[c] < end[c] ? ids(first[c]) : kInvalidKey;
  }
#pragma unroll
  for (int q = 0; q < 12; ++q) acc[q] = 0.f;
  any = false;
  for (;;) {
    uint32_t s[BATCH], at[BATCH];
    int corner[BATCH];
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      s[b] = head[0];
#pragma unroll
      for (int c = 1; c < 8; ++c) s[b] = min(s[b], head[c]);
      at[b] = 0;
      corner[b] = 0;
      if (s[b] != kInvalidKey) {
#pragma unroll
        for (int c = 0; c < 8; ++c)
          if (head[c] == s[b]) {  // (a point is in one cell: exactly one list)
            corner[b] = c;
            at[b] = pos[c];
            ++pos[c];
            head[c] = pos[c] < end[c] ? ids(pos[c]) : kInvalidKey;
          }
      }
    }
    if (s[0] == kInvalidKey) return;
    PointTerm t[BATCH];
#pragma unroll
    for (int b = 0; b < BATCH; ++b)
      if (s[b] != kInvalidKey) load(s[b], at[b], t[b]);
#pragma unroll
    for (int b = 0; b < BATCH; ++b) {
      if (s[b] == kInvalidKey) break;
      if (SCALAR) {
        if (t[b].g[0] == 0.f) continue;
        acc[0] = __fadd_rn(acc[0], density_corner_term(t[b].g[0], t[b].u, t[b].v, t[b].w, corner[b]));
      } else {
        const float scale = corner_scale(t[b], corner[b]);
#pragma unroll
        for (int q = 0; q < 12; ++q) acc[q] = __fadd_rn(acc[q], __fmul_rn(t[b].g[q], scale));
      }
      any = true;
    }
  }
}

// Adds the merged lists' contributions into the voxel's gradient: density
// ((g*a)*b)*c per point with a nonzero gradient; features g*scale, channels in
// chunks of 12, the lists walked again per chunk. make_load(ch0, nch): the
// loader of that chunk.
// BATCH points are loaded together.
template <bool SCALAR, int BATCH, class Ids, class MakeLoad>
__device__ __forceinline__ void merge_voxel(int C, const Ids& ids, const MakeLoad& make_load,
                                            const uint32_t first[8], const uint32_t end[8],
                                            int64_t slot, float* grad, uint8_t* touched) {
  float acc[12];
  bool any;
  if (SCALAR) {
    merge_lists<true, BATCH>(ids, make_load(0, 1), first, end, acc, any);
    if (!any) return;
    grad[slot] = __fadd_rn(grad[slot], acc[0]);
  } else {
    for (int ch0 = 0; ch0 < C; ch0 += 12) {
      const int nch = min(12, C - ch0);
      merge_lists<false, BATCH>(ids, make_load(ch0, nch), first, end, acc, any);
      if (!any) return;
      float* dst = grad + slot * C + ch0;
#pragma unroll
      for (int q = 0; q < 12; ++q)
        if (q < nch) dst[q] = __fadd_rn(dst[q], acc[q]);
    }
  }
  if (touched) touched[slot >> 9] = 1;
}

// A voxel with more points than long_from is summed by a warp (merge_long): its
// thread would take them one after another, some 0.6 us each, twice what the pair
// sort's walk takes. A warp takes a voxel's points 12 times as fast but is a warp:
// where very many voxels are long, their threads together are faster, and their one
// longest voxel does not count. So 32 points up to 512 k points in the call, 128
// from 2 M. (160^3, 30 k points at 600 voxels: 384 us by threads, 98 by warps; 1.8 M
// points over the scene: 522 by threads, 669 by warps from 32 points on, 520 so.)
__device__ __forceinline__ uint32_t long_from(int64_t n) {
  return uint32_t(min(max(n >> 14, int64_t(32)), int64_t(128)));
}
constexpr uint32_t kLongLeast = 32;
struct LongVoxel {
  uint32_t first[8], end[8];
  uint32_t slot;
  __device__ __forceinline__ void set(const uint32_t f[8], const uint32_t e[8], int64_t s) {
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      first[c] = f[c];
      end[c] = e[c];
    }
    slot = uint32_t(s);
  }
};
// The most that n points have of them.
inline int64_t most_long_voxels(int64_t n) { return n * 8 / (kLongLeast + 1); }
// A warp's space to sum one.
struct alignas(16) LongWarp {
  uint32_t ids[8][32];   // the next points of each list
  uint32_t order[256];   // their merge: position | list << 29
  float term[12 * 33];   // [channel][point]
};

// merge_voxel by a warp, the same sums in the same order. The points are put in
// order first: up to kLongOnce at once, each counting the smaller ids among all;
// more in rounds, of the next 32 points of every list. What lies up to the smallest
// of the lists' last ids is complete, and ranked by counting the smaller ids of each
// list. Then 32 points at a time are loaded and multiplied by the lanes side by
// side, and a lane per channel adds them in order.
constexpr uint32_t kLongOnce = 128;
template <bool SCALAR, class Ids, class MakeLoad>
__device__ __forceinline__ void merge_long(LongWarp& S, const LongVoxel& V, int C, const Ids& ids,
                                           const MakeLoad& make_load, float* grad,
                                           uint8_t* touched) {
  const int lane = threadIdx.x & 31;
  for (int ch0 = 0; ch0 < (SCALAR ? 1 : C); ch0 += 12) {
    const int nch = SCALAR ? 1 : min(12, C - ch0);
    const auto load = make_load(ch0, nch);
    float acc = 0.f;
    // adds the points order[0 .. m - 1]
    const auto add_points = [&](uint32_t m) {
      PointTerm t;
      int corner = 0;
      const auto fetch = [&](uint32_t e) {
        if (e >= m) return;
        const uint32_t o = S.order[e], at = o & 0x1FFFFFFFu;
        corner = int(o >> 29);
        load(ids(at), at, t);
      };
      fetch(lane);
      for (uint32_t b = 0; b < m; b += 32) {
        // (x + -0 = x for every x: behind the last point, and for a zero gradient of a
        // scalar grid, which is left out of the sum)
        const bool in = b + lane < m;
        if (SCALAR) {
          S.term[lane] = !in || t.g[0] == 0.f
                             ? -0.f
                             : density_corner_term(t.g[0], t.u, t.v, t.w, corner);
        } else {
          const float scale = in ? corner_scale(t, corner) : 0.f;
#pragma unroll
          for (int q = 0; q < 12; ++q)
            S.term[q * 33 + lane] = in ? __fmul_rn(t.g[q], scale) : -0.f;
        }
        __syncwarp();
        fetch(b + 32 + lane);  // these travel while the lanes add
        if (lane < nch) {
          const float* row = S.term + lane * 33;
#pragma unroll
          for (int j = 0; j < 32; ++j) acc = __fadd_rn(acc, row[j]);
        }
        __syncwarp();
      }
    };
    uint32_t pos[8], total = 0, most = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      pos[c] = V.first[c];
      const uint32_t n = V.end[c] - pos[c];
      total += n;
      most = max(most, n);
    }
    if (total <= kLongOnce) {
      uint32_t* id = &S.ids[0][0];
      uint32_t* where = reinterpret_cast<uint32_t*>(S.term);
      for (uint32_t l = lane; l < most; l += 32) {
        uint32_t at = l;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t n = V.end[c] - pos[c];
          if (l < n) {
            id[at] = ids(pos[c] + l);
            where[at] = (pos[c] + l) | uint32_t(c) << 29;
          }
          at += n;
        }
      }
      if (lane < 3) id[total + lane] = kInvalidKey;  // to a whole group of four
      __syncwarp();
      uint32_t mine[kLongOnce / 32], rank[kLongOnce / 32];
#pragma unroll
      for (uint32_t j = 0; j < kLongOnce / 32; ++j) {
        mine[j] = lane + 32 * j < total ? id[lane + 32 * j] : 0u;
        rank[j] = 0;
      }
      for (uint32_t i = 0; i < total; i += 4) {
        const uint4 w = *reinterpret_cast<const uint4*>(id + i);
#pragma unroll
        for (uint32_t j = 0; j < kLongOnce / 32; ++j)
          rank[j] += (w.x < mine[j]) + (w.y < mine[j]) + (w.z < mine[j]) + (w.w < mine[j]);
      }
#pragma unroll
      for (uint32_t j = 0; j < kLongOnce / 32; ++j)
        if (lane + 32 * j < total) S.order[rank[j]] = where[lane + 32 * j];
      __syncwarp();  // (the terms may be written over `where`)
      add_points(total);
    } else {
      for (;;) {
        uint32_t id[8], rank[8], bound = kInvalidKey - 1u, live = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const uint32_t left = V.end[c] - pos[c];
          id[c] = uint32_t(lane) < left ? ids(pos[c] + lane) : kInvalidKey;
          S.ids[c][lane] = id[c];
          const uint32_t last = __shfl_sync(0xffffffffu, id[c], 31);
          if (left > 32) bound = min(bound, last);
          live |= uint32_t(left > 0) << c;
          rank[c] = 0;
        }
        if (!live) break;
        __syncwarp();
        for (uint32_t rest = live; rest; rest &= rest - 1) {
          const uint32_t* w = S.ids[__ffs(rest) - 1];
#pragma unroll
          for (int c = 0; c < 8; ++c) {  // (the own list: the lane)
            uint32_t lo = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1) lo += w[lo + step - 1] < id[c] ? step : 0;
            rank[c] += lo + (w[lo] < id[c]);
          }
        }
        uint32_t m = 0;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          const bool take = id[c] <= bound;
          if (take) S.order[rank[c]] = (pos[c] + lane) | uint32_t(c) << 29;
          const uint32_t taken = __popc(__ballot_sync(0xffffffffu, take));
          pos[c] += taken;
          m += taken;
        }
        __syncwarp();  // (the ids are read too: the next round may write them)
        add_points(m);
      }
    }
    if (lane < nch) {
      float* dst = grad + int64_t(V.slot) * C + ch0 + lane;
      *dst = __fadd_rn(*dst, acc);
    }
    __syncwarp();
  }
  if (touched && lane == 0) touched[V.slot >> 9] = 1;
}

// A point's term from the call's arrays.
struct ArrayLoad {
  const PointSrc& src;
  int ch0, nch;
  __device__ __forceinline__ void operator()(uint32_t s, uint32_t, PointTerm& t) const {
    float x, y, z;
    src.pos(s, x, y, z);
    t.u = x - float(ifloor(x));
    t.v = y - float(ifloor(y));
    t.w = z - float(ifloor(z));
    const float* gs = src.g + int64_t(s) * src.C + ch0;
    if (src.vec) {
#pragma unroll
      for (int b = 0; b < 3; ++b)
        *reinterpret_cast<float4*>(t.g + 4 * b) = __ldg(reinterpret_cast<const float4*>(gs) + b);
    } else {
#pragma unroll
      for (int q = 0; q < 12; ++q) t.g[q] = q < nch ? __ldg(gs + q) : 0.f;
    }
  }
};

// Cell lattice of a grid: ext[a] = ldim[a] + 1 leaves of cells per axis.
struct CellLattice {
  int ext[3];
};
__device__ __forceinline__ uint32_t lattice_key(const CellLattice& L, int i, int j, int k) {
  const unsigned a = unsigned(i) + 1u, b = unsigned(j) + 1u, c = unsigned(k) + 1u;
  if (a > unsigned(L.ext[0] - 1) * 8u || b > unsigned(L.ext[1] - 1) * 8u ||
      c > unsigned(L.ext[2] - 1) * 8u)
    return kInvalidKey;
  const unsigned x = a + 7u, y = b + 7u, z = c + 7u;
  return (((x >> 3) * L.ext[1] + (y >> 3)) * L.ext[2] + (z >> 3)) << 9 |
         unsigned(vox_offset(x, y, z));
}
// (also clears the count of the call's leaves, as k_point_compact does: a memset
// between the launches would hold up the ones behind it)
__global__ void k_point_cells(CellLattice L, PointSrc src, int64_t n, uint32_t* keys,
                              uint32_t* nleaves) {
  grid_dep_sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) *nleaves = 0;
  const int64_t p = blockIdx.x * int64_t(blockDim.x) + threadIdx.x;
  if (p >= n) return;
  float x, y, z;
  src.pos(p, x, y, z);
  keys[p] = lattice_key(L, ifloor(x), ifloor(y), ifloor(z));
}

// Scalar grids: the points with a gradient, in order, 2048 points a block.
constexpr int kPtItems = 8;
constexpr int kPtBlock = 256 * kPtItems;
__global__ void __launch_bounds__(256)
    k_point_count(const float* __restrict__ g, int64_t n, uint32_t* counts) {
  grid_dep_sync();
  const int64_t b0 = int64_t(blockIdx.x) * kPtBlock;
  uint32_t c = 0;
#pragma unroll
  for (int q = 0; q < kPtItems; ++q) {
    const int64_t p = b0 + q * 256 + threadIdx.x;
    c += p < n && !(__ldg(g + p) == 0.f);
  }
  uint32_t tot;
  block_exclusive_scan(c, &tot);
  if (threadIdx.x == 0) counts[blockIdx.x] = tot;
}
// Their cell keys and ids; with PAIRS the slots of their corners and the ids of the
// pairs, eight a point, and the number of those behind that of the points.
template <bool PAIRS>
__global__ void __launch_bounds__(256)
    k_point_compact(GridView g, CellLattice L, PointSrc src, int64_t n,
                    const uint32_t* __restrict__ offs, uint32_t* keys, uint32_t* ids,
                    uint32_t* npts, uint32_t* nleaves) {
  grid_dep_sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *nleaves = 0;
    if (PAIRS) npts[1] = npts[0] * 8;
  }
  __shared__ uint32_t wc[kPtItems][8];  // points of each 32-point group, then their offsets
  const int64_t b0 = int64_t(blockIdx.x) * kPtBlock;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t bal[kPtItems];
#pragma unroll
  for (int q = 0; q < kPtItems; ++q) {
    const int64_t p = b0 + q * 256 + threadIdx.x;
    bal[q] = __ballot_sync(0xffffffffu, p < n && !(__ldg(src.g + min(p, n - 1)) == 0.f));
    if (lane == 0) wc[q][w] = __popc(bal[q]);
  }
  __syncthreads();
  const uint32_t mine = threadIdx.x < 8 * kPtItems ? wc[threadIdx.x >> 3][threadIdx.x & 7] : 0u;
  const uint32_t ex = block_exclusive_scan(mine, nullptr);
  if (threadIdx.x < 8 * kPtItems) wc[threadIdx.x >> 3][threadIdx.x & 7] = ex;
  __syncthreads();
  const uint32_t base = offs[blockIdx.x];
#pragma unroll
  for (int q = 0; q < kPtItems; ++q) {
    if (!((bal[q] >> lane) & 1u)) continue;
    const int64_t p = b0 + q * 256 + threadIdx.x;
    const uint32_t o = base + wc[q][w] + __popc(bal[q] & lanemask_lt());
    float x, y, z;
    src.pos(p, x, y, z);
    if (PAIRS) {
      emit_corner_keys(g, x, y, z, keys, o);
#pragma unroll
      for (int c = 0; c < 8; ++c) ids[int64_t(o) * 8 + c] = uint32_t(p) * 8 + c;
    } else {
      keys[o] = lattice_key(L, ifloor(x), ifloor(y), ifloor(z));
      ids[o] = uint32_t(p);
    }
  }
}

// Thread per sorted point, set: the point's record (u, v, w and the density
// gradient; with VEC the 12 feature gradients behind it) in sorted order, its
// cell's entry of the table from the first and the last point of the cell, and
// the leaves holding the cell's corners flagged and listed, once each (mark: the
// call that listed a leaf last). The sums walk the leaves of this call, not all
// that were touched since the gradient was zeroed.
template <bool VEC>
__global__ void __launch_bounds__(256)
    k_point_group(GridView g, CellLattice L, PointSrc src, const uint32_t* __restrict__ skeys,
                  const uint32_t* __restrict__ svals, int64_t n_max, const uint32_t* n_dev,
                  uint2* cells, float4* rec, uint8_t* touched, uint32_t* mark, uint32_t epoch,
                  int32_t* list, uint32_t* count, uint32_t* nlong,
                  const uint32_t* __restrict__ status) {
  grid_dep_sync();
  if (*status) return;  // the sort gave up a wait: its order is wrong
  if (blockIdx.x == 0 && threadIdx.x == 0) *nlong = 0;
  const int64_t n = eff_size(n_max, n_dev);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const uint32_t key = skeys[i];
    if (key == kInvalidKey) continue;
    const bool first = i == 0 || skeys[i - 1] != key, last = i + 1 == n || skeys[i + 1] != key;
    const uint32_t s = svals[i];
    float x, y, z;
    src.pos(s, x, y, z);
    const int ci = ifloor(x), cj = ifloor(y), ck = ifloor(z);
    float4* dst = rec + i * (VEC ? 4 : 1);
    dst[0] = make_float4(x - float(ci), y - float(cj), z - float(ck),
                         src.C == 1 ? src.gd(s) : 0.f);
    if (VEC) {
      const float4* gs = reinterpret_cast<const float4*>(src.g + int64_t(s) * 12);
#pragma unroll
      for (int b = 0; b < 3; ++b) dst[1 + b] = __ldg(gs + b);
    }
    if (last) cells[key].y = uint32_t(i) + 1u;
    if (!first) continue;
    cells[key].x = uint32_t(i);
    int slots[8];
    corner_slots(g, ci, cj, ck, slots);
    int before = -1;  // (most cells lie in one leaf)
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int l = slots[c] < 0 ? -1 : slots[c] >> 9;
      if (l != before && l >= 0 && mark[l] != epoch && atomicExch(mark + l, epoch) != epoch) {
        touched[l] = 1;
        list[atomicAdd(count, 1u)] = l;
      }
      before = l;
    }
  }
}

// A sorted point's term from its record, and (without grouped features) the
// call's gradients.
template <bool VEC>
struct RecLoad {
  const float4* __restrict__ rec;
  const PointSrc& src;
  int ch0, nch;
  __device__ __forceinline__ void operator()(uint32_t s, uint32_t at, PointTerm& t) const {
    const float4* r = rec + int64_t(at) * (VEC ? 4 : 1);
    float4 p;
    if (VEC) {
      float4 g[3];
      ld_nc32(r, p, g[0]);
      ld_nc32(r + 2, g[1], g[2]);
#pragma unroll
      for (int b = 0; b < 3; ++b) *reinterpret_cast<float4*>(t.g + 4 * b) = g[b];
    } else {
      p = __ldg(r);
    }
    t.u = p.x;
    t.v = p.y;
    t.w = p.z;
    if (VEC) return;
    if (src.C == 1) {
      t.g[0] = p.w;
    } else {
      const float* gs = src.g + int64_t(s) * src.C + ch0;
#pragma unroll
      for (int q = 0; q < 12; ++q) t.g[q] = q < nch ? __ldg(gs + q) : 0.f;
    }
  }
};

// Thread per voxel of the listed leaves; neighbouring threads read neighbouring
// table entries and records. Long voxels are listed.
template <bool SCALAR, bool VEC>
__global__ void __launch_bounds__(kVoxelThreads, SCALAR ? 7 : VEC ? 6 : 4)
    k_point_gather(GridView g, CellLattice L, const int32_t* __restrict__ list,
                   const uint32_t* __restrict__ count, const uint32_t* __restrict__ svals,
                   const uint2* __restrict__ cells, const float4* __restrict__ rec, PointSrc src,
                   int64_t n_max, const uint32_t* n_dev, LongVoxel* longs, uint32_t* nlong,
                   const uint32_t* __restrict__ status) {
  grid_dep_sync();
  if (*status) return;
  const int64_t nv = int64_t(*count) * kLeafVox;
  const uint32_t most = long_from(eff_size(n_max, n_dev));
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < nv;
       i += int64_t(gridDim.x) * blockDim.x) {
    const int leaf = __ldg(list + (i >> 9)), vox = int(i & 511);
    const int vi = __ldg(g.origin + leaf * 3) + (vox >> 6),
              vj = __ldg(g.origin + leaf * 3 + 1) + ((vox >> 3) & 7),
              vk = __ldg(g.origin + leaf * 3 + 2) + (vox & 7);
    uint32_t first[8], end[8], points = 0;
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      int di, dj, dk;
      corner_delta(c, di, dj, dk);
      const uint2 e = __ldg(cells + lattice_key(L, vi - di, vj - dj, vk - dk));
      first[c] = e.x;
      end[c] = e.y;
      points += e.y - e.x;
    }
    if (!points) continue;
    const int64_t slot = int64_t(leaf) * kLeafVox + vox;
    if (points > most) {
      longs[atomicAdd(nlong, 1u)].set(first, end, slot);
      continue;
    }
    merge_voxel<SCALAR, SCALAR ? 4 : 2>(
        src.C, [&](uint32_t pos) { return __ldg(svals + pos); },
        [&](int ch0, int nch) { return RecLoad<VEC>{rec, src, ch0, nch}; }, first, end, slot,
        g.grad, nullptr);
  }
}

// A warp per long voxel (they lie side by side: a block of the gather's would have
// dozens, most blocks none); then the table's entries are cleared, thread per point.
template <bool SCALAR, bool VEC>
__global__ void __launch_bounds__(kVoxelThreads)
    k_point_long(GridView g, const LongVoxel* __restrict__ longs,
                 const uint32_t* __restrict__ nlong, const uint32_t* __restrict__ skeys,
                 const uint32_t* __restrict__ svals, const float4* __restrict__ rec, PointSrc src,
                 int64_t n_max, const uint32_t* n_dev, uint2* cells,
                 const uint32_t* __restrict__ status) {
  grid_dep_sync();
  if (*status) return;
  __shared__ LongWarp S[kVoxelThreads / 32];
  const uint32_t nl = *nlong, w = threadIdx.x >> 5;
  for (uint32_t k = w * gridDim.x + blockIdx.x; k < nl; k += gridDim.x * (kVoxelThreads / 32))
    merge_long<SCALAR>(
        S[w], longs[k], src.C, [&](uint32_t pos) { return __ldg(svals + pos); },
        [&](int ch0, int nch) { return RecLoad<VEC>{rec, src, ch0, nch}; }, g.grad, nullptr);
  const int64_t n = eff_size(n_max, n_dev);
  for (int64_t i = blockIdx.x * int64_t(blockDim.x) + threadIdx.x; i < n;
       i += int64_t(gridDim.x) * blockDim.x) {
    const uint32_t key = skeys[i];
    if (key != kInvalidKey && (i == 0 || skeys[i - 1] != key)) cells[key] = make_uint2(0u, 0u);
  }
}

// Up to kSmallPoints points: one block sorts (cell, point) words in shared
// memory, and a second kernel, eight threads per sorted point, takes a voxel at
// the first point of its first cell and finds its cells by binary search; two
// launches in place of the sort's seven and no table. The eight searches run
// side by side and four points are loaded at a time: a thread is alone with its
// latencies (203 rays' colour points 67 -> 59 us a call).
constexpr int kSmallPoints = 2048;
constexpr int kSmallBits = 11;
// points a thread loads together: the few threads leave the registers free
constexpr int kSmallBatch = 4;
constexpr uint64_t kNoPoint = ~0ull;
// 14 bits per coordinate (resolutions are at most 8192)
__device__ __forceinline__ uint64_t small_cell(const CellLattice& L, int i, int j, int k) {
  const unsigned a = unsigned(i) + 1u, b = unsigned(j) + 1u, c = unsigned(k) + 1u;
  if (a > unsigned(L.ext[0] - 1) * 8u || b > unsigned(L.ext[1] - 1) * 8u ||
      c > unsigned(L.ext[2] - 1) * 8u)
    return kNoPoint >> kSmallBits;
  return uint64_t(a) << 28 | uint64_t(b) << 14 | c;
}

__global__ void __launch_bounds__(1024)
    k_point_small_sort(CellLattice L, PointSrc src, int n, int size, uint64_t* out) {
  grid_dep_sync();
  __shared__ uint64_t w[kSmallPoints];
  for (int p = threadIdx.x; p < size; p += 1024) {
    uint64_t v = kNoPoint;
    if (p < n && !(src.C == 1 && __ldg(src.g + p) == 0.f)) {
      float x, y, z;
      src.pos(p, x, y, z);
      v = small_cell(L, ifloor(x), ifloor(y), ifloor(z)) << kSmallBits | uint64_t(p);
    }
    w[p] = v;
  }
  // bitonic: one compare per thread and step
  for (int k = 2; k <= size; k <<= 1)
    for (int j = k >> 1; j > 0; j >>= 1) {
      __syncthreads();
      const int a = threadIdx.x;
      if (a < size / 2) {
        const int lo = 2 * a - (a & (j - 1)), hi = lo + j;
        const uint64_t x = w[lo], y = w[hi];
        if ((x > y) == ((lo & k) == 0)) {
          w[lo] = y;
          w[hi] = x;
        }
      }
    }
  __syncthreads();
  for (int p = threadIdx.x; p < n; p += 1024) out[p] = w[p];
}

template <bool SCALAR>
__global__ void __launch_bounds__(kVoxelThreads)
    k_point_small_gather(GridView g, CellLattice L, const uint64_t* __restrict__ sorted, int n,
                         PointSrc src, uint8_t* touched) {
  grid_dep_sync();
  __shared__ __align__(16) uint64_t w[kSmallPoints];
  __shared__ LongVoxel longs[kVoxelThreads];
  __shared__ LongWarp S[kVoxelThreads / 32];
  __shared__ int nlong;
  if (threadIdx.x == 0) nlong = 0;
  const ulonglong2* s2 = reinterpret_cast<const ulonglong2*>(sorted);
#pragma unroll
  for (int b = 0; b < kSmallPoints / 256; ++b) {  // (the words behind n are not used)
    const int p = b * 128 + threadIdx.x;
    if (2 * p < n) reinterpret_cast<ulonglong2*>(w)[p] = __ldg(s2 + p);
  }
  __syncthreads();
  const int t = blockIdx.x * 128 + threadIdx.x, i = t >> 3, c = t & 7;
  // the voxel at corner c of point i's cell, if point i is the first of its cell
  int slot = -1, vi = 0, vj = 0, vk = 0;
  if (i < n) {
    const uint64_t cell = w[i] >> kSmallBits;
    if (cell != kNoPoint >> kSmallBits && (i == 0 || (w[i - 1] >> kSmallBits) != cell)) {
      int di, dj, dk;
      corner_delta(c, di, dj, dk);
      vi = int(cell >> 28) - 1 + di;
      vj = int(cell >> 14 & 0x3FFFu) - 1 + dj;
      vk = int(cell & 0x3FFFu) - 1 + dk;
      slot = slot_of(g, vi, vj, vk);
    }
  }
  const auto ids = [&](uint32_t pos) { return uint32_t(w[pos]) & (kSmallPoints - 1); };
  const auto make_load = [&](int ch0, int nch) { return ArrayLoad{src, ch0, nch}; };
  if (slot >= 0) {
    // the eight cells' lists: the binary searches of their first points, then of
    // their ends, side by side
    uint64_t want[8];
    uint32_t first[8], end[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      int ei, ej, ek;
      corner_delta(q, ei, ej, ek);
      want[q] = small_cell(L, vi - ei, vj - ej, vk - ek);
      first[q] = 0;
    }
#pragma unroll 1
    for (int step = kSmallPoints; step > 0; step >>= 1) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint32_t at = first[q] + step;
        if (at <= uint32_t(n) && (w[at - 1] >> kSmallBits) < want[q]) first[q] = at;
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) end[q] = first[q];
#pragma unroll 1
    for (int step = kSmallPoints; step > 0; step >>= 1) {
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const uint32_t at = end[q] + step;
        if (at <= uint32_t(n) && (w[at - 1] >> kSmallBits) <= want[q]) end[q] = at;
      }
    }
    bool owner = true;  // (another thread takes the voxel at its first cell with points)
    uint32_t points = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      owner = owner && (q >= c || end[q] == first[q]);
      points += end[q] - first[q];
    }
    if (owner && points > kLongLeast)
      longs[atomicAdd(&nlong, 1)].set(first, end, slot);
    else if (owner)
      merge_voxel<SCALAR, kSmallBatch>(src.C, ids, make_load, first, end, slot, g.grad, touched);
  }
  __syncthreads();
  for (int k = threadIdx.x >> 5; k < nlong; k += kVoxelThreads / 32)
    merge_long<SCALAR>(S[threadIdx.x >> 5], longs[k], src.C, ids, make_load, g.grad, touched);
}

// The form of the backward for n points. Up to kSmallPoints: one block's sort.
// Beyond, the sort by cell with a table over the lattice, where there are points
// enough for the leaves that it walks, voxel by voxel, and for the table; else the
// sort of the (slot, corner) pairs, whose cost is the points' alone. Points over
// all voxels are as fast either way at n = nslots / 40 to nslots / 20 (pairs and
// cells, us: 100^3 full 30 k points 100 and 99, 80 k 147 and 119; 256^3 full 600 k 610 and
// 619, 150 k 215 and 386; a scene at 400^3 (4.5 M slots) 150 k 194 and 212, 300 k 304 and
// 268), and below some 8192 points the fewer launches win (100^3 full, 5000: 77 and
// 87). The table takes at most 2 KB a point and 1 GiB.
constexpr int64_t kMaxCells = int64_t(1) << 27;
static bool points_by_cell(const pvdb_grid_s* g, int64_t ncells, int64_t n) {
  return n >= 8192 && n * 20 >= g->nslots() && n * 256 >= ncells && ncells <= kMaxCells;
}

// Scalar grids from this many points on: the pair sort, too, first drops the points
// without a gradient. Of the samples of rays through a scene one in 16 carries one
// (240^3, 58 k samples: 162 us without, 96 with it); where all do, the two more
// passes cost some 5 us (400^3, 50 k points: 124 and 122, 160^3 full 119 and 123).
constexpr int64_t kPairsCompact = 32768;

// The points of a scalar grid that have a gradient, in order: keys[0], vals[0] and
// npts of the grid's scratch (keys[1] and vals[1] are free until the sort's first pass).
template <bool PAIRS>
static int compact_points(pvdb_grid_s* g, const CellLattice& L, const PointSrc& src, int64_t n,
                          cudaStream_t st) {
  ReduceScratch& rs = g->red;
  int rc;
  if (!rs.npts && (rc = dev_alloc((void**)&rs.npts, 16))) return rc;
  const int nb = ceil_div(n, kPtBlock);
  uint32_t *counts = rs.vals[1], *offs = rs.keys[1];
  launch_k(k_point_count, nb, 256, 0, st, src.g, n, counts);
  PVDB_CHECK_LAUNCH("k_point_count");
  if ((rc = scan_exclusive_u32(counts, offs, nb, rs.npts, &rs.partial, &rs.partial_cap, st)))
    return rc;
  launch_k(k_point_compact<PAIRS>, nb, 256, 0, st, g->view(), L, src, n, offs, rs.keys[0],
           rs.vals[0], rs.npts, g->d_tcount);
  PVDB_CHECK_LAUNCH("k_point_compact");
  return PVDB_OK;
}

static int point_backward_pairs(pvdb_grid_s* g, const CellLattice& L, const PointSrc& src,
                                int64_t n, cudaStream_t st, uint32_t** status) {
  const int64_t nc = n * 8;
  int rc = reduce_reserve(g, nc);
  if (rc) return rc;
  g->tlist_valid = false;
  const bool compact = g->C == 1 && n >= kPairsCompact;
  const uint32_t* n_dev = nullptr;
  if (compact) {
    if ((rc = compact_points<true>(g, L, src, n, st))) return rc;
    n_dev = g->red.npts + 1;
  } else {
    launch_k(k_point_keys, ceil_div(n, 256), 256, 0, st, g->view(), src.xs, src.ys, src.zs, n,
             g->red.keys[0]);
    PVDB_CHECK_LAUNCH("k_point_keys");
  }
  int buf = 0;
  rc = radix_sort_pairs_dev(g->red, nc, n_dev, slot_key_bits(g->nslots()), !compact, &buf, st,
                            status);
  if (rc) return rc;
  const int grid = int(std::min<int64_t>(ceil_div(nc, 256), int64_t(num_sms()) * 16));
  launch_k(k_segment_reduce<PointSrc>, grid, 256, 0, st, g->red.keys[buf], g->red.vals[buf], nc,
           n_dev, src, g->C == 1 ? g->d_grad : nullptr, g->C == 1 ? nullptr : g->d_grad, g->C,
           g->d_touched, g->d_touched, *status);
  PVDB_CHECK_LAUNCH("k_segment_reduce");
  return PVDB_OK;
}

static int point_backward_small(pvdb_grid_s* g, const CellLattice& L, const PointSrc& src, int n,
                                cudaStream_t st) {
  int rc = reduce_reserve(g, 2 * kSmallPoints);
  if (rc) return rc;
  uint64_t* w = reinterpret_cast<uint64_t*>(g->red.keys[0]);
  int size = 64;
  while (size < n) size *= 2;
  launch_k(k_point_small_sort, 1, 1024, 0, st, L, src, n, size, w);
  PVDB_CHECK_LAUNCH("k_point_small_sort");
  launch_k(g->C == 1 ? k_point_small_gather<true> : k_point_small_gather<false>,
           ceil_div(int64_t(n) * 8, 128), 128, 0, st, g->view(), L, w, n, src, g->d_touched);
  PVDB_CHECK_LAUNCH("k_point_small_gather");
  return PVDB_OK;
}

// What the cell form keeps with the grid beyond the sort's scratch: given back when
// memory for the rest is missing, or when a call ends between the kernels that
// fill and clear the table.
static void free_cells(ReduceScratch& rs) {
  dev_free(rs.cells);
  dev_free(rs.rec);
  rs.cells = nullptr;
  rs.rec = nullptr;
  rs.cells_cap = rs.rec_cap = 0;
}

// The cell table, zeroed when it is new.
static int cell_table(pvdb_grid_s* g, int64_t ncells, cudaStream_t st) {
  ReduceScratch& rs = g->red;
  if (rs.cells_cap >= size_t(ncells) * 8) return PVDB_OK;
  int rc = dev_reserve((void**)&rs.cells, &rs.cells_cap, size_t(ncells) * 8);
  if (rc) return rc;
  const cudaError_t e = cudaMemsetAsync(rs.cells, 0, rs.cells_cap, st);
  if (e == cudaSuccess) return PVDB_OK;
  free_cells(rs);
  return cuda_error(e, "cell table");
}

static int point_backward_cells(pvdb_grid_s* g, const CellLattice& L, int64_t ncells,
                                const PointSrc& src, int64_t n, cudaStream_t st,
                                uint32_t** status) {
  ReduceScratch& rs = g->red;
  int rc = cell_table(g, ncells, st);
  if (rc || (rc = reduce_reserve(g, n))) return rc;
  // the records, then the list of the long voxels
  const size_t rec_bytes = size_t(n) * (src.vec ? 64 : 16);
  if ((rc = dev_reserve((void**)&rs.rec, &rs.rec_cap,
                        rec_bytes + size_t(most_long_voxels(n)) * sizeof(LongVoxel))))
    return rc;
  LongVoxel* longs = reinterpret_cast<LongVoxel*>(reinterpret_cast<char*>(rs.rec) + rec_bytes);
  if (!rs.npts && (rc = dev_alloc((void**)&rs.npts, 16))) return rc;
  if (!rs.mark) {
    rs.epoch = 0;
    if ((rc = dev_alloc((void**)&rs.mark, size_t(g->nleaf) * 4))) return rc;
  }
  if (rs.epoch + 1 <= 1) {  // new marks, or the last number is given out
    rs.epoch = 0;
    PVDB_CHECK_CUDA(cudaMemsetAsync(rs.mark, 0, size_t(g->nleaf) * 4, st));
  }
  ++rs.epoch;
  g->tlist_valid = false;  // d_tlist takes this call's leaves
  const int bits = slot_key_bits(ncells);
  const uint32_t* n_dev = nullptr;
  int buf = 0;
  if (g->C == 1) {
    if ((rc = compact_points<false>(g, L, src, n, st))) return rc;
    n_dev = rs.npts;
    rc = radix_sort_pairs_dev(rs, n, n_dev, bits, false, &buf, st, status);
  } else {
    launch_k(k_point_cells, ceil_div(n, 256), 256, 0, st, L, src, n, rs.keys[0], g->d_tcount);
    PVDB_CHECK_LAUNCH("k_point_cells");
    rc = radix_sort_pairs(rs, n, bits, true, &buf, st, status);
  }
  if (rc) return rc;
  const uint32_t *skeys = rs.keys[buf], *svals = rs.vals[buf];
  const int sgrid = int(std::min<int64_t>(ceil_div(n, 256), stride_grid()));
  struct Filled {  // the table, until k_point_long is launched
    ReduceScratch* rs;
    ~Filled() {
      if (rs) free_cells(*rs);
    }
  } filled{&rs};
  launch_k(src.vec ? k_point_group<true> : k_point_group<false>, sgrid, 256, 0, st, g->view(), L,
           src, skeys, svals, n, n_dev, rs.cells, rs.rec, g->d_touched, rs.mark, rs.epoch, g->d_tlist,
           g->d_tcount, rs.npts + 1, *status);
  PVDB_CHECK_LAUNCH("k_point_group");
  launch_k(g->C == 1 ? k_point_gather<true, false>
           : src.vec ? k_point_gather<false, true>
                     : k_point_gather<false, false>,
           voxel_grid(g), kVoxelThreads, 0, st, g->view(), L, g->d_tlist, g->d_tcount, svals, rs.cells,
           rs.rec, src, n, n_dev, longs, rs.npts + 1, *status);
  PVDB_CHECK_LAUNCH("k_point_gather");
  launch_k(g->C == 1 ? k_point_long<true, false>
           : src.vec ? k_point_long<false, true>
                     : k_point_long<false, false>,
           stride_grid(), kVoxelThreads, 0, st, g->view(), longs, rs.npts + 1, skeys, svals, rs.rec,
           src, n, n_dev, rs.cells, *status);
  PVDB_CHECK_LAUNCH("k_point_long");
  filled.rs = nullptr;
  return PVDB_OK;
}

}  // namespace pvdb

using namespace pvdb;

extern "C" int pvdb_debug_wait_limit(uint32_t spins, int32_t hold_first) {
  clear_error();
  g_dbg_spin.store(spins);
  g_dbg_hold.store(hold_first == 2 ? 2 : hold_first ? 1 : 0);
  return PVDB_OK;
}

extern "C" int pvdb_grid_sample_backward(pvdb_grid g, const float* xs, const float* ys,
                                         const float* zs, const float* grad_out, int64_t n,
                                         int32_t mem, pvdb_stream s) {
  clear_error();
  PVDB_REQUIRE(g, "null grid");
  PVDB_REQUIRE(n >= 0, "negative size");
  if (n == 0) return PVDB_OK;
  PVDB_REQUIRE(xs && ys && zs && grad_out, "null argument");
  PVDB_REQUIRE(n * 8 < int64_t(0xFFFFFFF0u), "too many points for one backward call");
  cudaStream_t st = as_stream(s);
  const float *dx = xs, *dy = ys, *dz = zs, *dg = grad_out;
  if (mem == PVDB_MEM_HOST) {
    int rc = dev_reserve(&g->d_stage, &g->stage_cap, size_t(n) * 4 * (3 + g->C));
    if (rc) return rc;
    float* b = (float*)g->d_stage;
    PVDB_CHECK_CUDA(cudaMemcpyAsync(b, xs, n * 4, cudaMemcpyHostToDevice, st));
    PVDB_CHECK_CUDA(cudaMemcpyAsync(b + n, ys, n * 4, cudaMemcpyHostToDevice, st));
    PVDB_CHECK_CUDA(cudaMemcpyAsync(b + 2 * n, zs, n * 4, cudaMemcpyHostToDevice, st));
    PVDB_CHECK_CUDA(cudaMemcpyAsync(b + 3 * n, grad_out, n * 4 * g->C, cudaMemcpyHostToDevice, st));
    dx = b; dy = b + n; dz = b + 2 * n; dg = b + 3 * n;
  }
  const PointSrc src{dx, dy, dz, dg, g->C, g->C == 12 && (reinterpret_cast<uintptr_t>(dg) & 15u) == 0};
  const CellLattice L{{g->ldim[0] + 1, g->ldim[1] + 1, g->ldim[2] + 1}};
  const int64_t ncells = int64_t(L.ext[0]) * L.ext[1] * L.ext[2] * kLeafVox;
  uint32_t* status = nullptr;
  int rc = PVDB_OK;
  if (n <= kSmallPoints) {
    rc = point_backward_small(g, L, src, int(n), st);
  } else {
    // the form that the points are better off with, and the other one if memory is
    // missing (all of it is reserved before anything is added)
    bool cells = points_by_cell(g, ncells, n);
    for (int attempt = 0;; ++attempt, cells = !cells) {
      rc = cells ? point_backward_cells(g, L, ncells, src, n, st, &status)
                 : point_backward_pairs(g, L, src, n, st, &status);
      if (rc != PVDB_ERR_NOMEM || attempt || (!cells && ncells > kMaxCells)) break;
      clear_error();
      if (cells) free_cells(g->red);
    }
  }
  if (rc) return rc;
  g->tlist_valid = false;  // new touched leaves
  // the call waits for its stream (as the reference's backward does) so that a
  // sort wait that gave up is reported, with the gradient left unchanged
  return read_wait_status(status, st, "a radix-sort look-back wait of the grid backward timed out");
}
