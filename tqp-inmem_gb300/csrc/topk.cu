// topk.cu - launchers of the warp-list top-k (topk.cuh) and tqpk_topk_stable.
#include <algorithm>

#include "topk.cuh"

namespace tqpk {

__device__ __forceinline__ bool ArraySource::get(int64_t i, uint64_t& k) const {
  if (i >= n) return false;
  const int64_t src = perm ? perm[i] : i;
  k = sort_key(keys, dt, src, desc);
  return true;
}

// Test hook (tqpk_debug_topk_barrier): the poll limit of the single-launch top-k's grid barrier and
// a number of arrivals it also waits for that never come.
static int g_tk_spin_limit = kSpinLimit;
static int g_tk_missing = 0;

// CTAs of k_tk_fused<Src> that fit on the device at once (the cooperative launch's limit).
template <class Src>
static int fused_capacity() {
  static int cap = -1;
  if (cap < 0) {
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_tk_fused<Src>, 256, 0) != cudaSuccess) {
      (void)cudaGetLastError();
      per_sm = 0;
    }
    cap = per_sm * num_sms();
  }
  return cap;
}

template <int R, class Src>
static int launch_r(const Src& src, int k, int grid, TopkOut O, cudaStream_t s) {
  (void)grid;
  // groups of G items (a multiple of 4), at most kTopkGroups of them
  int64_t G = 4;
  while (G * kTopkGroups < src.n) G <<= 1;
  const int ng = (int)std::max<int64_t>(1, (src.n + G - 1) / G);
  if constexpr (!Src::kStoredOrder) {
    if (R == 1 && G <= kTopkFusedMaxG && O.err && ng <= fused_capacity<Src>()) {
      // one cooperative launch: all ng CTAs resident together, so the grid barrier inside completes
      cudaLaunchConfig_t cfg = {};
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeCooperative;
      attr[0].val.cooperative = 1;
      cfg.gridDim = dim3(ng);
      cfg.blockDim = dim3(256);
      cfg.stream = s;
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      TQPK_CUDA(cudaLaunchKernelEx(&cfg, k_tk_fused<Src>, src, G, k, O, g_tk_spin_limit, g_tk_missing));
      return TQPK_OK;
    }
  }
  k_tk_group_best<Src><<<ng, 256, 0, s>>>(src, G, k, O);
  TQPK_CHECK_LAUNCH();
  k_tk_filter<R, Src><<<ng, 256, 0, s>>>(src, G, k, O);     // the same groups
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

template <class Src>
static int launch_src(const Src& src, int k, int grid, TopkOut O, cudaStream_t s) {
  if (k > 256) return TQPK_EUNSUPPORTED;
  if constexpr (Src::kStoredOrder) {
    return launch_r<1>(src, k, grid, O, s);          // stored columns use no warp lists
  } else {
    if (k <= 32) return launch_r<1>(src, k, grid, O, s);
    if (k <= 64) return launch_r<2>(src, k, grid, O, s);
    if (k <= 128) return launch_r<4>(src, k, grid, O, s);
    return launch_r<8>(src, k, grid, O, s);
  }
}

int topk_warp_launch(int kind, const void* src, int k, int grid, TopkOut O, cudaStream_t s) {
  if (kind == 0) return launch_src(*static_cast<const DenseSumSource*>(src), k, grid, O, s);
  return launch_src(*static_cast<const ArraySource*>(src), k, grid, O, s);
}

__global__ void k_topk_positions_to_perm(const int64_t* idx, const int64_t* count, const int64_t* perm_in,
                                         int64_t* perm_out, int64_t k) {
  const int64_t m = *count;
  for (int64_t j = threadIdx.x; j < k; j += blockDim.x) {
    if (j < m) perm_out[j] = perm_in ? perm_in[idx[j]] : idx[j];
  }
}

// Elements (cand[i], or i) whose key ties with the m-th of a top-k's entries, counted per 4096-element tile
// and then (WRITE) listed in input order; also how many of the entries come strictly before it.  A row of
// several keys is in the first k only if it is in the first k by the first key or ties with the k-th, so a
// sort with a limit looks at the later keys of these rows only.  Bound: one read of the key column.
struct TieCtl {
  unsigned long long less, ties;
};

template <bool WRITE>
__global__ void __launch_bounds__(kBlock) k_topk_ties(const void* __restrict__ keys, int dt, int desc,
                                                      const int64_t* __restrict__ cand, int64_t n,
                                                      const int64_t* __restrict__ top, int m, TieCtl* ctl,
                                                      int* __restrict__ tile_ties, int64_t* __restrict__ out) {
  __shared__ int s_cnt[kItems * (kBlock / 32)];      // ties of (step, warp), then their exclusive scan
  __shared__ int si[kBlock / 32 + 1];
  __shared__ int64_t sw[kBlock / 32 + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t t0 = blockIdx.x * (int64_t)kTile;
  uint64_t k[kItems];
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const int64_t i = t0 + j * kBlock + threadIdx.x;
    k[j] = i < n ? sort_key(keys, dt, cand ? cand[i] : i, desc) : 0;
  }
  const uint64_t cut = sort_key(keys, dt, top[m - 1], desc);
  uint32_t hits = 0;
#pragma unroll
  for (int j = 0; j < kItems; ++j)
    hits |= (uint32_t)(t0 + j * kBlock + threadIdx.x < n && k[j] == cut) << j;
  if (!WRITE) {
    int total;
    block_excl_scan<kBlock, int>(__popc(hits), total, si);
    if (threadIdx.x == 0) {
      tile_ties[blockIdx.x] = total;
      if (total) atomicAdd(&ctl->ties, (unsigned long long)total);
    }
    if (blockIdx.x == 0)
      for (int e = threadIdx.x; e < m; e += kBlock)
        if (sort_key(keys, dt, top[e], desc) < cut) atomicAdd(&ctl->less, 1ull);
    return;
  }
  int64_t before = 0, base;                          // the ties of the tiles before this one
  for (int t = threadIdx.x; t < (int)blockIdx.x; t += kBlock) before += tile_ties[t];
  block_excl_scan<kBlock, int64_t>(before, base, sw);
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const unsigned b = __ballot_sync(0xffffffffu, (hits >> j) & 1u);
    if (lane == 0) s_cnt[j * (kBlock / 32) + warp] = __popc(b);
  }
  __syncthreads();
  int total, mine = threadIdx.x < kItems * (kBlock / 32) ? s_cnt[threadIdx.x] : 0;
  mine = block_excl_scan<kBlock, int>(mine, total, si);
  if (threadIdx.x < kItems * (kBlock / 32)) s_cnt[threadIdx.x] = mine;
  __syncthreads();
#pragma unroll
  for (int j = 0; j < kItems; ++j) {
    const unsigned b = __ballot_sync(0xffffffffu, (hits >> j) & 1u);
    if ((hits >> j) & 1u) {
      const int64_t i = t0 + j * kBlock + threadIdx.x;
      out[base + s_cnt[j * (kBlock / 32) + warp] + __popc(b & ((1u << lane) - 1u))] = cand ? cand[i] : i;
    }
  }
}

}  // namespace tqpk

using namespace tqpk;

static int topk_ties(bool write, const void* keys, int32_t dt, int32_t desc, const int64_t* cand, int64_t n,
                     const int64_t* top, int64_t m, int64_t* out, int64_t* h_less, int64_t* h_ties, void* ws,
                     size_t ws_bytes, tqpk_stream stream) {
  if (n < 1 || m < 1 || m > 256 || m > n || !keys || !top || !ws) return TQPK_EINVAL;
  if (!dtype_size(dt)) return TQPK_EDTYPE;
  const int64_t tiles = (n + kTile - 1) / kTile;
  if (tiles > INT32_MAX) return TQPK_EUNSUPPORTED;
  WsCursor cur(ws, ws_bytes);
  TieCtl* ctl = cur.take<TieCtl>(1);
  int* base = cur.take<int>(tiles);
  if (!ctl || !base) return TQPK_ENOMEM;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (write) {
    k_topk_ties<true><<<(int)tiles, kBlock, 0, s>>>(keys, dt, desc ? 1 : 0, cand, n, top, (int)m, ctl, base, out);
    TQPK_CHECK_LAUNCH();
    return TQPK_OK;
  }
  TQPK_CUDA(cudaMemsetAsync(ctl, 0, sizeof(TieCtl), s));
  k_topk_ties<false><<<(int)tiles, kBlock, 0, s>>>(keys, dt, desc ? 1 : 0, cand, n, top, (int)m, ctl, base, nullptr);
  TQPK_CHECK_LAUNCH();
  TieCtl h;
  TQPK_CUDA(cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, s));
  TQPK_CUDA(cudaStreamSynchronize(s));
  *h_less = (int64_t)h.less;
  *h_ties = (int64_t)h.ties;
  return TQPK_OK;
}

extern "C" size_t tqpk_topk_ties_workspace_bytes(int64_t n) {
  return 512 + align_up((size_t)((std::max<int64_t>(n, 0) + kTile - 1) / kTile) * 4, 256);
}

extern "C" int tqpk_topk_ties(const void* d_keys, int32_t dt, int32_t desc, const int64_t* d_cand, int64_t n,
                              const int64_t* d_top, int64_t m, int64_t* h_less, int64_t* h_ties, void* ws,
                              size_t ws_bytes, tqpk_stream stream) {
  if (!h_less || !h_ties) return TQPK_EINVAL;
  return topk_ties(false, d_keys, dt, desc, d_cand, n, d_top, m, nullptr, h_less, h_ties, ws, ws_bytes, stream);
}

extern "C" int tqpk_topk_ties_write(const void* d_keys, int32_t dt, int32_t desc, const int64_t* d_cand, int64_t n,
                                    const int64_t* d_top, int64_t m, int64_t* d_out, void* ws, size_t ws_bytes,
                                    tqpk_stream stream) {
  if (!d_out) return TQPK_EINVAL;
  return topk_ties(true, d_keys, dt, desc, d_cand, n, d_top, m, d_out, nullptr, nullptr, ws, ws_bytes, stream);
}

// Test hook: the poll limit of the single-launch top-k's grid barrier, and arrivals it also waits
// for that never come (its bounded wait then runs out: TQPK_ETIMEOUT in the caller's error word).
// (kSpinLimit, 0) restores the defaults.  Not thread-safe; for tests only.
extern "C" int tqpk_debug_topk_barrier(int32_t spin_limit, int32_t missing) {
  if (spin_limit < 0 || spin_limit > kSpinLimit || missing < 0 || missing > 1024) return TQPK_EINVAL;
  g_tk_spin_limit = spin_limit;
  g_tk_missing = missing;
  return TQPK_OK;
}

extern "C" size_t tqpk_topk_workspace_bytes(int64_t n, int64_t k) {
  if (n < 0) n = 0;
  if (k <= 256) return topk_scratch_bytes(n, (int)std::max<int64_t>(k, 1)) + 1024;
  return sort_ws_bytes(n) + align_up((size_t)n * sizeof(int64_t), 256);
}

extern "C" int tqpk_topk_stable(const void* d_keys, int32_t dt, int32_t desc, const int64_t* d_perm_in, int64_t n,
                                int64_t k, int64_t* d_perm_out, void* ws, size_t ws_bytes, tqpk_stream stream) {
  if (n < 0 || k < 0 || (n > 0 && k > 0 && (!d_keys || !d_perm_out || !ws))) return TQPK_EINVAL;
  if (!dtype_size(dt)) return TQPK_EDTYPE;
  const int64_t m = std::min(n, k);
  if (m == 0) return TQPK_OK;
  if (ws_bytes < tqpk_topk_workspace_bytes(n, k)) return TQPK_ENOMEM;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (k > 256) {
    WsCursor full(ws, ws_bytes);
    int64_t* order = full.take<int64_t>(n);
    if (!order) return TQPK_ENOMEM;
    const SortKey key{d_keys, nullptr, dt, desc ? 1 : 0, 0, 0};
    int rc = sort_keys(&key, 1, d_perm_in, n, order, full.base + full.off, ws_bytes - full.off, s);
    if (rc) return rc;
    TQPK_CUDA(cudaMemcpyAsync(d_perm_out, order, m * sizeof(int64_t), cudaMemcpyDeviceToDevice, s));
    return TQPK_OK;
  }
  const int grid = topk_grid_size();
  WsCursor cur(ws, ws_bytes);
  unsigned* ticket = cur.take<unsigned>(64);
  int64_t* count = cur.take<int64_t>(4);
  int64_t* idx = cur.take<int64_t>(k);
  uint64_t* ck = cur.take<uint64_t>(topk_list_entries(n, (int)k));
  int64_t* ci = cur.take<int64_t>(topk_list_entries(n, (int)k));
  if (!ci) return TQPK_ENOMEM;
  TQPK_CUDA(cudaMemsetAsync(ticket, 0, 256, s));
  ArraySource src{d_keys, dt, d_perm_in, n, desc ? 1 : 0};
  TopkOut O{idx, count, ck, ci, ticket, nullptr, reinterpret_cast<unsigned long long*>(ticket + 8), ticket + 16};
  O.cap = topk_list_cap(n, (int)k);
  timing_before(KID_PIPE_TOPK, s);
  int rc = topk_warp_launch(1, &src, (int)k, grid, O, s);
  timing_after(KID_PIPE_TOPK, s);
  if (rc) return rc;
  k_topk_positions_to_perm<<<1, 256, 0, s>>>(idx, count, d_perm_in, d_perm_out, m);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}
