// keys.cu - group codes of arbitrary key tuples, and row gathers of string columns.
//
// The reference stacks the group-by key columns side by side, a 2-D string
// column contributing its w bytes as w columns (aggregate.py:291-311), then
// numbers the distinct rows of that stack (:313-333).  Key tuples that do not
// fit the dense mixed-radix slots or the packed 62-bit hash of groupby.cu
// (string keys, float keys, more than TQPK_MAX_KEYS keys) are numbered here:
//
//   1. k_key_insert: each row passing the mask hashes its key tuple and claims
//      or finds its entry of an open-addressing table (capacity a power of two
//      >= 2n).  An entry is one 64-bit word, (24-bit fingerprint << 40) |
//      (representative row + 1), claimed with one compare-and-swap; a
//      fingerprint match is confirmed by comparing the whole key tuple with
//      the representative row's, so distinct tuples never share a group.
//   2. A claimed entry is numbered by the same kernel (group ids in claim order).
//   3. The groups are ordered by key tuple with the library's stable radix sort
//      (sort_keys over the representative rows): one key per numeric column, one
//      per 8 bytes of a string column (big-endian words of the bytes, an int8
//      column's with the sign bit flipped, so unsigned word order is the byte
//      order of the reference's stacked columns).
//   4. k_key_codes: every row gets the rank of its group; d_reps[rank] is the
//      group's representative row.
//
// A dense group-by over the codes (domain [0, G)) then produces the groups in
// ascending key-tuple order, and the key outputs are gathered from the
// representative rows (tqpk_gather_rows for string keys).
#include "common.cuh"

namespace tqpk {

constexpr int kMaxEncKeys = TQPK_MAX_COLS;
constexpr uint64_t kRowMask = (1ull << 40) - 1;

struct KeyTuple {
  const void* col[kMaxEncKeys];
  int dt[kMaxEncKeys];
  int width[kMaxEncKeys];   // bytes per row of a string key, 0 for a 1-D key
  int n;
};

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  // splitmix64 finaliser (S. Vigna): a bijective avalanche of 64 bits
  z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
  z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
  return z ^ (z >> 31);
}

// The bits a key contributes to equality: integers by value, float64 with
// -0.0 folded onto +0.0 (torch.unique sees them equal).
__device__ __forceinline__ uint64_t key_bits(const void* p, int dt, int64_t row) {
  if (dt == TQPK_F64) {
    const uint64_t b = static_cast<const uint64_t*>(p)[row];
    return (b << 1) == 0 ? 0 : b;                     // -0.0 as +0.0, in integer instructions
  }
  return static_cast<uint64_t>(ld_int(p, dt, row));
}

__device__ __forceinline__ uint64_t key_hash(const KeyTuple& K, int64_t row) {
  uint64_t h = 0x9e3779b97f4a7c15ull;
  for (int k = 0; k < K.n; ++k) {
    const int w = K.width[k];
    if (w) {
      const uint8_t* s = static_cast<const uint8_t*>(K.col[k]) + row * w;
      for (int i = 0; i < w; i += 8) h = mix64(h ^ load_bytes8(s + i, w - i, i > 0 || row > 0));
    } else {
      h = mix64(h ^ key_bits(K.col[k], K.dt[k], row));
    }
  }
  return h;
}

__device__ __forceinline__ bool key_equal(const KeyTuple& K, int64_t a, int64_t b) {
  for (int k = 0; k < K.n; ++k) {
    const int w = K.width[k];
    if (w) {
      const uint8_t* x = static_cast<const uint8_t*>(K.col[k]) + a * w;
      const uint8_t* y = static_cast<const uint8_t*>(K.col[k]) + b * w;
      for (int i = 0; i < w; i += 8)
        if (load_bytes8(x + i, w - i, i > 0 || a > 0) != load_bytes8(y + i, w - i, i > 0 || b > 0)) return false;
    } else if (key_bits(K.col[k], K.dt[k], a) != key_bits(K.col[k], K.dt[k], b)) {
      return false;
    }
  }
  return true;
}

// Passing rows of a 1024-row tile are gathered first, so that hashing runs with full warps under a
// selective mask; a claimed entry is numbered at once (one counter update per 256 rows; a pass over the
// table that counted each occupied entry on one word took 19 us for 27.6 K groups, this kernel byte by byte
// 44 us for 128 K of 800 K rows).
constexpr int kKeyTile = 4 * kBlock;

__global__ void __launch_bounds__(kBlock) k_key_insert(const __grid_constant__ KeyTuple K, const uint8_t* mask, int64_t n,
                                                       uint64_t* __restrict__ table, int64_t cap,
                                                       int64_t* __restrict__ entry_of_row,
                                                       int64_t* __restrict__ gid_of_entry,
                                                       int64_t* __restrict__ rep_of_gid, unsigned long long* counter,
                                                       int* err) {
  __shared__ uint16_t s_row[kKeyTile];
  __shared__ int sw[kBlock / 32 + 1];
  __shared__ unsigned s_claims[kBlock / 32];
  __shared__ unsigned long long s_at;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool mask_vec = (reinterpret_cast<uintptr_t>(mask) & 3u) == 0;
  for (int64_t t0 = blockIdx.x * (int64_t)kKeyTile; t0 < n; t0 += (int64_t)gridDim.x * kKeyTile) {
    const int64_t r0[1] = {t0 + 4 * threadIdx.x};
    uint32_t bits = valid_rows<1>(r0, n);
    if (mask && bits) {
      uint8_t x[4];
      load_rows<uint8_t, 1>(mask, r0, n, mask_vec, x);
      bits &= bits_of<4>([&](int i) { return x[i] != 0; });
    }
    int total;
    int at = block_excl_scan<kBlock, int>(__popc(bits), total, sw);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if ((bits >> j) & 1u) s_row[at++] = (uint16_t)(4 * threadIdx.x + j);
      else if (r0[0] + j < n) entry_of_row[r0[0] + j] = -1;
    }
    __syncthreads();
    for (int i0 = 0; i0 < total; i0 += kBlock) {
      const int i = i0 + threadIdx.x;
      int64_t r = 0, found = -1;
      bool claimed = false;
      if (i < total) {
        r = t0 + s_row[i];
        const uint64_t h = key_hash(K, r);
        const uint64_t mine = ((h >> 40) << 40) | static_cast<uint64_t>(r + 1);
        int64_t p = static_cast<int64_t>(h & static_cast<uint64_t>(cap - 1));
        for (int64_t probe = 0; probe < cap; ++probe) {
          uint64_t e = table[p];
          if (e == 0) {
            e = atomicCAS(reinterpret_cast<unsigned long long*>(&table[p]), 0ull, (unsigned long long)mine);
            claimed = e == 0;
          }
          if (claimed || ((e >> 40) == (h >> 40) && key_equal(K, r, static_cast<int64_t>((e & kRowMask) - 1)))) {
            found = p;
            break;
          }
          p = (p + 1) & (cap - 1);
        }
        if (found < 0) set_error(err, TQPK_ENOMEM);   // cannot happen at capacity >= 2n; kept as a bound
        entry_of_row[r] = found;
      }
      const unsigned m = __ballot_sync(0xffffffffu, claimed);
      if (lane == 0) s_claims[warp] = __popc(m);
      __syncthreads();
      unsigned before = 0, all = 0;
#pragma unroll
      for (int w = 0; w < kBlock / 32; ++w) {
        before += w < warp ? s_claims[w] : 0;
        all += s_claims[w];
      }
      if (threadIdx.x == 0) s_at = all ? atomicAdd(counter, (unsigned long long)all) : 0;
      __syncthreads();
      if (claimed) {
        const int64_t g = (int64_t)s_at + before + __popc(m & ((1u << lane) - 1u));
        gid_of_entry[found] = g;
        rep_of_gid[g] = r;
      }
    }
    __syncthreads();
  }
}

__global__ void k_key_rank(const int64_t* __restrict__ perm, int64_t G, const int64_t* __restrict__ rep_of_gid,
                           int64_t* __restrict__ rank_of_gid, int64_t* __restrict__ reps_out) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < G; i += (int64_t)gridDim.x * blockDim.x) {
    rank_of_gid[perm[i]] = i;
    reps_out[i] = rep_of_gid[perm[i]];
  }
}

__global__ void k_key_codes(const int64_t* __restrict__ entry_of_row, int64_t n, const int64_t* __restrict__ gid_of_entry,
                            const int64_t* __restrict__ rank_of_gid, int32_t* __restrict__ codes) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t e = entry_of_row[r];
    codes[r] = e < 0 ? 0 : static_cast<int32_t>(rank_of_gid[gid_of_entry[e]]);
  }
}

// Word `word` of each row of an int8/uint8 [n, w] column as a sort key: bytes
// word*8 .. word*8+7 big-endian (an int8 column's with the sign bit of each
// byte flipped; zero past w), stored as int64 with its top bit flipped, so the
// library's int64 sort orders rows as the byte columns compare, most
// significant first.
__global__ void k_string_words(const uint8_t* __restrict__ src, int64_t n, int w, int word, uint8_t flip,
                               int64_t* __restrict__ out) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const uint8_t* s = src + r * w;
    uint64_t v = 0;
    for (int i = 0; i < 8; ++i) {
      const int c = word * 8 + i;
      v = (v << 8) | (c < w ? static_cast<uint64_t>(s[c] ^ flip) : 0ull);
    }
    out[r] = static_cast<int64_t>(v ^ (1ull << 63));
  }
}

// Rows of fewer than 16 bytes: a thread reads its row by words into shared memory, and the block writes its
// 256 rows, which lie one after another, 16 bytes at a time.  A byte per thread with a 64-bit division each
// took 57 us for 1.5 M rows of 15 bytes.
__global__ void __launch_bounds__(kBlock) k_gather_short_rows(const uint8_t* __restrict__ src, int w,
                                                              const int64_t* __restrict__ idx, int64_t n_idx,
                                                              int64_t n_src, uint8_t* __restrict__ dst, int vec) {
  extern __shared__ __align__(16) uint8_t stage[];
  for (int64_t j0 = blockIdx.x * (int64_t)kBlock; j0 < n_idx; j0 += (int64_t)gridDim.x * kBlock) {
    const int64_t j = j0 + threadIdx.x;
    if (j < n_idx) {
      const int64_t r = idx[j];
      const bool ok = r >= 0 && r < n_src;
      uint8_t* out = stage + threadIdx.x * w;
      for (int i = 0; i < w; i += 8) {
        const uint64_t x = ok ? load_bytes8(src + r * w + i, w - i, i > 0 || r > 0) : 0;
#pragma unroll
        for (int b = 0; b < 8; ++b)
          if (i + b < w) out[i + b] = (uint8_t)(x >> (8 * b));
      }
    }
    __syncthreads();
    const int64_t left = (n_idx - j0) * w;
    const int bytes = (int)(left < (int64_t)kBlock * w ? left : (int64_t)kBlock * w);
    uint8_t* o = dst + j0 * w;                    // 256 rows: a multiple of 16 bytes
    const int whole = vec ? bytes / 16 : 0;
    for (int i = threadIdx.x; i < whole; i += kBlock)
      reinterpret_cast<uint4*>(o)[i] = reinterpret_cast<const uint4*>(stage)[i];
    for (int i = whole * 16 + threadIdx.x; i < bytes; i += kBlock) o[i] = stage[i];
    __syncthreads();
  }
}

// Sixteen bytes of a column of `total` bytes from byte `at` on (those past its end: 0), by aligned words that
// lie in it, byte by byte at its ends.
__device__ __forceinline__ ulonglong2 load_bytes16(const uint8_t* col, int64_t at, int64_t total) {
  const uint8_t* s = col + at;
  const unsigned off = (unsigned)(reinterpret_cast<uintptr_t>(s) & 3u);
  if ((reinterpret_cast<uintptr_t>(s) & 15u) == 0 && at + 16 <= total) return *reinterpret_cast<const ulonglong2*>(s);
  if (at >= off && at - off + 20 <= total) {
    const unsigned* a = reinterpret_cast<const unsigned*>(s - off);
    const unsigned w0 = a[0], w1 = a[1], w2 = a[2], w3 = a[3], w4 = a[4];
    return make_ulonglong2(((uint64_t)__funnelshift_r(w1, w2, 8 * off) << 32) | __funnelshift_r(w0, w1, 8 * off),
                           ((uint64_t)__funnelshift_r(w3, w4, 8 * off) << 32) | __funnelshift_r(w2, w3, 8 * off));
  }
  uint64_t v[2] = {0, 0};
  const int m = total - at < 16 ? (int)(total - at) : 16;
#pragma unroll 1
  for (int i = 0; i < m; ++i) v[i >> 3] |= static_cast<uint64_t>(s[i]) << (8 * (i & 7));
  return make_ulonglong2(v[0], v[1]);
}

// Rows of 16 bytes and more: a thread makes 16 bytes of the output at a time, out of one row or two, so that
// consecutive threads read consecutive words of a row, and write them at once.  What bounds it: the rows'
// sectors.  In place of rows staged in shared memory a row per thread, whose byte stores met in one bank when the
// width was a multiple of 32 (750 K rows of 128 bytes 425 us, 64 bytes 122), or a byte per thread (247 and 119):
// 40 and 24.
constexpr int kChunkRow = 16, kWideRow = 4096;

__global__ void __launch_bounds__(kBlock) k_gather_chunks(const uint8_t* __restrict__ src, unsigned w,
                                                          const int64_t* __restrict__ idx, int64_t n_idx, int64_t n_src,
                                                          uint8_t* __restrict__ dst) {
  constexpr int U = 2;                             // chunks a thread has in flight
  const int64_t total = n_src * w;
  for (int64_t j0 = blockIdx.x * (int64_t)kBlock; j0 < n_idx; j0 += (int64_t)gridDim.x * kBlock) {
    const unsigned bytes = (unsigned)(n_idx - j0 < kBlock ? n_idx - j0 : kBlock) * w, chunks = bytes / 16;
    uint8_t* o = dst + j0 * w;                     // 256 rows: a multiple of 16 bytes
    for (unsigned c0 = threadIdx.x; c0 < chunks; c0 += U * kBlock) {
      unsigned at[U], left[U];                     // byte of the row the chunk starts at, and the row's bytes in it
      int64_t r0[U], r1[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const unsigned p = 16 * min(c0 + u * kBlock, chunks - 1), row = p / w;
        at[u] = p - row * w;
        left[u] = min(16u, w - at[u]);
        r0[u] = idx[j0 + row];
        r1[u] = left[u] < 16 ? idx[j0 + row + 1] : -1;
      }
      ulonglong2 a[U], b[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        a[u] = b[u] = make_ulonglong2(0, 0);
        if (r0[u] >= 0 && r0[u] < n_src) a[u] = load_bytes16(src, r0[u] * w + at[u], total);
        if (r1[u] >= 0 && r1[u] < n_src) b[u] = load_bytes16(src, r1[u] * w, total);
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (c0 + u * kBlock >= chunks) break;
        const unsigned m = 8 * left[u];            // bits of the first row
        ulonglong2 x = a[u];
        if (m < 64) {
          x.x = (x.x & ((1ull << m) - 1)) | (b[u].x << m);
          x.y = (b[u].y << m) | (b[u].x >> (64 - m));
        } else if (m < 128) {
          x.y = (m > 64 ? x.y & ((1ull << (m - 64)) - 1) : 0) | (b[u].x << (m - 64));
        }
        reinterpret_cast<ulonglong2*>(o)[c0 + u * kBlock] = x;
      }
    }
    for (unsigned i = chunks * 16 + threadIdx.x; i < bytes; i += kBlock) {
      const unsigned row = i / w;
      const int64_t r = idx[j0 + row];
      o[i] = r >= 0 && r < n_src ? src[r * w + (i - row * w)] : 0;
    }
  }
}

__global__ void k_gather_rows(const uint8_t* __restrict__ src, int64_t row_bytes, const int64_t* __restrict__ idx,
                              int64_t n_idx, int64_t n_src, uint8_t* __restrict__ dst, int* err) {
  const int64_t total = n_idx * row_bytes;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t j = i / row_bytes, b = i - j * row_bytes;
    const int64_t r = idx[j];
    if (r < 0 || r >= n_src) {
      set_error(err, TQPK_EINVAL);
      dst[i] = 0;
      continue;
    }
    dst[i] = src[r * row_bytes + b];
  }
}

static int64_t key_capacity(int64_t n) {
  int64_t c = 1024;
  while (c < 2 * n) c <<= 1;
  return c;
}

}  // namespace tqpk

using namespace tqpk;

extern "C" size_t tqpk_key_encode_workspace_bytes(int64_t n) {
  if (n < 0) n = 0;
  const int64_t cap = key_capacity(n);
  return align_up(cap * 8, 256) * 2 + align_up(n * 8, 256) * 5 + sort_ws_bytes(n, kMaxSortKeys) + 4096;
}

extern "C" int tqpk_key_encode(int32_t n_keys, const void* const* h_keys, const int32_t* h_dtypes,
                               const int32_t* h_widths, const uint8_t* d_mask, int64_t n, int32_t* d_codes,
                               int64_t* d_reps, int64_t* h_groups, void* d_ws, size_t ws_bytes,
                               tqpk_stream stream) {
  if (n_keys < 1 || n_keys > kMaxEncKeys || n < 0 || !h_keys || !h_dtypes || !h_widths || !h_groups) return TQPK_EINVAL;
  if (n >= (int64_t)kRowMask || n > (int64_t)INT32_MAX) return TQPK_EUNSUPPORTED;
  KeyTuple K{};
  K.n = n_keys;
  for (int k = 0; k < n_keys; ++k) {
    if (h_widths[k] < 0) return TQPK_EINVAL;
    if (h_widths[k] > 0 && dtype_size(h_dtypes[k]) != 1) return TQPK_EDTYPE;
    if (!dtype_size(h_dtypes[k])) return TQPK_EDTYPE;
    if (n > 0 && !h_keys[k]) return TQPK_EINVAL;
    K.col[k] = h_keys[k];
    K.dt[k] = h_dtypes[k];
    K.width[k] = h_widths[k];
  }
  *h_groups = 0;
  if (n == 0) return TQPK_OK;
  if (!d_codes || !d_reps || !d_ws) return TQPK_EINVAL;
  if (ws_bytes < tqpk_key_encode_workspace_bytes(n)) return TQPK_ENOMEM;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int64_t cap = key_capacity(n);
  WsCursor ws(d_ws, ws_bytes);
  uint64_t* table = ws.take<uint64_t>(cap);
  int64_t* gid_of_entry = ws.take<int64_t>(cap);
  int64_t* entry_of_row = ws.take<int64_t>(n);
  int64_t* rep_of_gid = ws.take<int64_t>(n);
  int64_t* rank_of_gid = ws.take<int64_t>(n);
  int64_t* perm_a = ws.take<int64_t>(n);
  int64_t* perm_b = ws.take<int64_t>(n);
  int* ctl = ws.take<int>(4);
  void* sort_ws = ws.take<char>(sort_ws_bytes(n, kMaxSortKeys));
  if (!sort_ws || !ctl) return TQPK_ENOMEM;
  unsigned long long* counter = reinterpret_cast<unsigned long long*>(ctl);   // ctl[0..1]
  int* err = ctl + 2;
  TQPK_CUDA(cudaMemsetAsync(table, 0, cap * 8, s));
  TQPK_CUDA(cudaMemsetAsync(ctl, 0, 16, s));
  k_key_insert<<<grid_for((n + 3) / 4, 8), kBlock, 0, s>>>(K, d_mask, n, table, cap, entry_of_row, gid_of_entry,
                                                           rep_of_gid, counter, err);
  TQPK_CHECK_LAUNCH();
  int64_t host[2] = {0, 0};
  TQPK_CUDA(cudaMemcpyAsync(host, ctl, 16, cudaMemcpyDeviceToHost, s));
  TQPK_CUDA(cudaStreamSynchronize(s));
  const int64_t G = host[0];
  const int e = static_cast<int>(host[1] & 0xffffffff);
  if (e) return e;
  *h_groups = G;
  if (G == 0) return TQPK_OK;
  // the groups by key tuple, each through its representative row; a tuple of more than kMaxSortKeys
  // words is sorted in runs of words, least significant run first
  int total = 0;
  for (int k = 0; k < n_keys; ++k) total += K.width[k] ? (K.width[k] + 7) / 8 : 1;
  int64_t* cur = nullptr;
  SortKey run[kMaxSortKeys];
  int m = 0, left = total;
  for (int k = n_keys - 1; k >= 0; --k) {
    const int nw = K.width[k] ? (K.width[k] + 7) / 8 : 1;
    for (int w = nw - 1; w >= 0; --w) {
      run[kMaxSortKeys - 1 - m++] = SortKey{K.col[k], rep_of_gid, K.dt[k], 0, K.width[k], w};
      if (--left == 0 || m == kMaxSortKeys) {
        int64_t* out = (cur == perm_a) ? perm_b : perm_a;
        const int rc = sort_keys(run + kMaxSortKeys - m, m, cur, G, out, sort_ws, sort_ws_bytes(n, kMaxSortKeys), s, true);
        if (rc) return rc;
        cur = out;
        m = 0;
      }
    }
  }
  k_key_rank<<<grid_for(G, 4), kBlock, 0, s>>>(cur, G, rep_of_gid, rank_of_gid, d_reps);
  TQPK_CHECK_LAUNCH();
  k_key_codes<<<grid_for(n, 8), kBlock, 0, s>>>(entry_of_row, n, gid_of_entry, rank_of_gid, d_codes);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

extern "C" int tqpk_gather_rows(const void* d_src, int64_t n_src, int64_t row_bytes, const int64_t* d_idx, int64_t n_idx,
                                void* d_dst, tqpk_stream stream) {
  if (n_src < 0 || n_idx < 0 || row_bytes <= 0) return TQPK_EINVAL;
  if (n_idx == 0) return TQPK_OK;
  if (!d_src || !d_idx || !d_dst) return TQPK_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if (row_bytes < kChunkRow) {
    k_gather_short_rows<<<grid_for(n_idx, 8), kBlock, (size_t)row_bytes * kBlock, s>>>(
        static_cast<const uint8_t*>(d_src), (int)row_bytes, d_idx, n_idx, n_src, static_cast<uint8_t*>(d_dst),
        aligned16(d_dst) ? 1 : 0);
    TQPK_CHECK_LAUNCH();
    return TQPK_OK;
  }
  if (row_bytes <= kWideRow && aligned16(d_dst)) {
    k_gather_chunks<<<grid_for(n_idx, 8), kBlock, 0, s>>>(static_cast<const uint8_t*>(d_src), (unsigned)row_bytes, d_idx,
                                                          n_idx, n_src, static_cast<uint8_t*>(d_dst));
    TQPK_CHECK_LAUNCH();
    return TQPK_OK;
  }
  k_gather_rows<<<grid_for(n_idx * row_bytes, 8), kBlock, 0, s>>>(static_cast<const uint8_t*>(d_src), row_bytes, d_idx,
                                                                  n_idx, n_src, static_cast<uint8_t*>(d_dst), nullptr);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

extern "C" int tqpk_string_words(const void* d_src, int64_t n, int32_t width, int32_t word, int32_t signed_bytes,
                                 int64_t* d_out, tqpk_stream stream) {
  if (n < 0 || width <= 0 || word < 0 || word * 8 >= width) return TQPK_EINVAL;
  if (n == 0) return TQPK_OK;
  if (!d_src || !d_out) return TQPK_EINVAL;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  k_string_words<<<grid_for(n, 8), kBlock, 0, s>>>(static_cast<const uint8_t*>(d_src), n, width, word,
                                                   signed_bytes ? 0x80u : 0u, d_out);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}
