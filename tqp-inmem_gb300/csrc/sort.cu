// sort.cu - kernel (b): stable LSD radix sort of (key, row) pairs over one or more keys.
//
// Reference: operators/sort.py:22-42 runs one stable torch.sort per key (last
// key first), permuting `perm` each time, then slices perm[:limit].
// sort_keys runs that whole loop: keys[0] is the most significant key, and the
// keys are sorted last to first, each key's digits least significant first.
// tqpk_argsort_stable is its one-key form.
//
// Every key has an order-preserving unsigned image (signed integers: sign bit
// flipped in their own width; float64: sign-magnitude flip with -0.0 -> +0.0
// and NaN as the largest value; eight bytes of a string row big-endian;
// descending: bitwise complement, which keeps ties stable).
//
//   hist : all 8-bit digit histograms of every key in one read of the key
//          columns; the last CTA of each key scans them into global digit
//          offsets and records which digits vary (a digit that holds every
//          row is no pass at all).
//   pass : launch p runs the p-th varying digit; launches beyond the last one
//          return at once, so the host never reads the digit masks.  A key's
//          first pass gathers the key through the rows' current order and
//          keeps it as a 32-bit word when its varying digits allow; the last
//          pass writes the int64 permutation itself.
//
// What bounds a pass: the tiles are L2-resident (8 B per row each way at 32-bit
// keys), so it is the chain load -> rank -> look-back -> scatter of one tile.
// Rows are ranked by match_any per warp, reordered by digit in shared memory
// and written as runs (a 4096-row tile has 16-row runs; the direct scatter
// they replace wrote 16 B per row to 32 places per warp store), and a digit's
// look-back reads eight predecessors at a time (one at a time, 129 tiles took
// ~15 of a pass's 23 us).
#include <algorithm>

#include "common.cuh"

namespace tqpk {

constexpr int kRadix = 256;
constexpr int kDigits = 8;                   // 8-bit digits of a 64-bit key
constexpr int kMaxPasses = kMaxSortKeys * kDigits;
constexpr int kHistThreads = 512;

struct SortKeySet {
  SortKey k[kMaxSortKeys];
  int n;
};

struct SortCtl {
  int err;
  unsigned mask[kMaxSortKeys];       // varying digits per key
  unsigned ticket[kMaxSortKeys];     // hist CTAs done
  unsigned tile_ctr[kMaxPasses];     // next tile of each pass
};

__host__ __device__ __forceinline__ int sort_key_digits(const SortKey& K) {
  if (K.width) return kDigits;
  switch (K.dt) {
    case TQPK_I8: case TQPK_U8: case TQPK_BOOL: return 1;
    case TQPK_I32: return 4;
  }
  return kDigits;
}

// The unsigned image of element e under key K.
__device__ __forceinline__ uint64_t sort_image(const SortKey& K, int64_t e) {
  const int64_t r = K.rows ? K.rows[e] : e;
  if (K.width) {                     // bytes word*8 .. word*8+7, big-endian, zero past the width
    const uint8_t* s = static_cast<const uint8_t*>(K.col) + r * K.width;
    const uint8_t flip = K.dt == TQPK_I8 ? 0x80u : 0u;   // int8 bytes order as signed values
    uint64_t w = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int c = K.word * 8 + i;
      w = (w << 8) | (c < K.width ? static_cast<uint64_t>(s[c] ^ flip) : 0ull);
    }
    return K.desc ? ~w : w;
  }
  switch (K.dt) {
    case TQPK_I8: { const unsigned v = static_cast<const uint8_t*>(K.col)[r] ^ 0x80u; return K.desc ? v ^ 0xffu : v; }
    case TQPK_U8:
    case TQPK_BOOL: { const unsigned v = static_cast<const uint8_t*>(K.col)[r]; return K.desc ? v ^ 0xffu : v; }
    case TQPK_I32: { const unsigned v = static_cast<const uint32_t*>(K.col)[r] ^ 0x80000000u; return K.desc ? ~v : v; }
  }
  return sort_key_bits(static_cast<const uint64_t*>(K.col)[r], K.dt == TQPK_F64, K.desc);
}

// Histograms of every digit of key blockIdx.y; the key's last CTA scans them.  An int64 key's high
// half is usually constant over long stretches, so a thread counts its repeats in a register.
__global__ void __launch_bounds__(kHistThreads) k_sort_hist(const __grid_constant__ SortKeySet S,
                                                            const int64_t* __restrict__ perm_in, int64_t n,
                                                            unsigned long long* __restrict__ hist,
                                                            int64_t* __restrict__ offsets, SortCtl* ctl) {
  __shared__ unsigned sh[kDigits * kRadix];
  __shared__ int s_last;
  const int key = blockIdx.y;
  const SortKey K = S.k[key];
  const int nd = sort_key_digits(K);
  for (int i = threadIdx.x; i < nd * kRadix; i += kHistThreads) sh[i] = 0;
  __syncthreads();
  unsigned hi_run = 0, hi_val = 0;
  auto flush_hi = [&]() {
    if (!hi_run) return;
#pragma unroll
    for (int d = 0; d < 4; ++d) atomicAdd(&sh[(4 + d) * kRadix + ((hi_val >> (8 * d)) & 255)], hi_run);
  };
  const int64_t stride = (int64_t)gridDim.x * kHistThreads;
#pragma unroll 4
  for (int64_t i = blockIdx.x * (int64_t)kHistThreads + threadIdx.x; i < n; i += stride) {
    const uint64_t u = sort_image(K, perm_in ? perm_in[i] : i);
    const unsigned lo = (unsigned)u;
    atomicAdd(&sh[lo & 255], 1u);
    if (nd > 1) {
#pragma unroll
      for (int d = 1; d < 4; ++d) atomicAdd(&sh[d * kRadix + ((lo >> (8 * d)) & 255)], 1u);
    }
    if (nd > 4) {
      const unsigned hi = (unsigned)(u >> 32);
      if (hi != hi_val || !hi_run) {
        flush_hi();
        hi_run = 0;
        hi_val = hi;
      }
      ++hi_run;
    }
  }
  if (nd > 4) flush_hi();
  __syncthreads();
  unsigned long long* H = hist + (size_t)key * kDigits * kRadix;
  for (int i = threadIdx.x; i < nd * kRadix; i += kHistThreads)
    if (sh[i]) atomicAdd(&H[i], (unsigned long long)sh[i]);
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(&ctl->ticket[key], 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  // warp d scans digit d: eight bins per lane
  const int d = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (d >= nd) return;
  unsigned long long c[8], sum = 0;
  bool all = false;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    c[q] = __ldcg(&H[d * kRadix + lane * 8 + q]);
    all = all || c[q] == (unsigned long long)n;
    sum += c[q];
  }
  unsigned long long run = warp_incl_scan(sum) - sum;
  int64_t* O = offsets + ((size_t)key * kDigits + d) * kRadix;
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    O[lane * 8 + q] = (int64_t)run;
    run += c[q];
  }
  if (!__any_sync(0xffffffffu, all) && lane == 0) atomicOr(&ctl->mask[key], 1u << d);
}

// Look-back status word: flag (2 bits) | pass number + 1 (10 bits) | value (52 bits).  The pass number
// makes a word of an earlier pass read as "not there yet", so the array is zeroed once per sort.
constexpr int kStValueBits = 52;
__device__ __forceinline__ uint64_t st_word(unsigned flag, unsigned epoch, uint64_t v) {
  return ((uint64_t)flag << 62) | ((uint64_t)epoch << kStValueBits) | v;
}
__device__ __forceinline__ uint64_t ld_relaxed(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_relaxed(uint64_t* p, uint64_t v) {
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Exclusive prefix of digit `d` before `tile`.  Only the words themselves are communicated, so
// relaxed accesses do; eight predecessors are read at a time.
__device__ __forceinline__ uint64_t radix_lookback(uint64_t* status, int64_t tile, int d, unsigned epoch, int* err) {
  uint64_t excl = 0;
  int64_t p = tile - 1;
  int spins = 0;
  while (p >= 0) {
    uint64_t w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) w[q] = p - q >= 0 ? ld_relaxed(&status[(p - q) * kRadix + d]) : 0;
    int used = 0;
    bool done = false, ready = true;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const unsigned flag = (unsigned)(w[q] >> 62);
      const unsigned ep = (unsigned)(w[q] >> kStValueBits) & 1023u;
      if (!done && ready && p - q >= 0) {
        if (flag == 0 || ep != epoch) {
          ready = false;
        } else {
          excl += w[q] & ((1ull << kStValueBits) - 1);
          ++used;
          done = flag == 2;
        }
      }
    }
    if (done) break;
    p -= used;
    if (!ready) {
      if (++spins > kSpinLimit) {
        set_error(err, TQPK_ETIMEOUT);
        break;
      }
      __nanosleep(32);
    }
  }
  return excl;
}

constexpr int kSortItems = 16;

template <int BLOCK, class V>
constexpr size_t pass_smem() {
  return (size_t)BLOCK * kSortItems * (8 + sizeof(V)) + kRadix * 12 + (BLOCK / 32) * kRadix * 4;
}

template <class V>
struct PassArgs {
  const int64_t* perm_in;    // element of position i (null: i)
  int64_t n;
  uint64_t* kbuf[2];
  V* vbuf[2];
  int64_t* perm_out;
  const int64_t* offsets;
  uint64_t* status;
  SortCtl* ctl;
  int p;                     // which varying digit, counted over all keys from the last key up
};

// V: type of a row's position among the n rows (uint32 below 2^32 rows).
template <int BLOCK, class V>
__global__ void __launch_bounds__(BLOCK) k_sort_pass(const __grid_constant__ SortKeySet S, const PassArgs<V> A) {
  constexpr int kTileN = BLOCK * kSortItems;
  constexpr int kWarps = BLOCK / 32;
  static_assert(BLOCK >= kRadix, "one thread per digit");
  extern __shared__ __align__(16) unsigned char smem[];
  uint64_t* s_key = reinterpret_cast<uint64_t*>(smem);
  V* s_val = reinterpret_cast<V*>(s_key + kTileN);
  int64_t* s_gbase = reinterpret_cast<int64_t*>(s_val + kTileN);
  unsigned* s_dbase = reinterpret_cast<unsigned*>(s_gbase + kRadix);
  unsigned(*wcnt)[kRadix] = reinterpret_cast<unsigned(*)[kRadix]>(s_dbase + kRadix);
  __shared__ unsigned s_tile;
  __shared__ unsigned s_ws[kRadix / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the p-th varying digit, keys from last to first
  int total = 0, key = -1, digit = 0;
  unsigned kmask = 0;
  for (int k = S.n - 1; k >= 0; --k) {
    const unsigned m = A.ctl->mask[k];
    const int c = __popc(m);
    if (key < 0 && A.p < total + c) {
      unsigned b = m;
      for (int q = A.p - total; q > 0; --q) b &= b - 1;
      key = k;
      kmask = m;
      digit = __ffs(b) - 1;
    }
    total += c;
  }
  const int64_t n = A.n;
  if (key < 0) {
    if (A.p == 0)                    // no digit varies: the order stays as it is
      for (int64_t i = blockIdx.x * (int64_t)BLOCK + threadIdx.x; i < n; i += (int64_t)gridDim.x * BLOCK)
        A.perm_out[i] = A.perm_in ? A.perm_in[i] : i;
    return;
  }
  const SortKey K = S.k[key];
  const bool first = (kmask & ((1u << digit) - 1u)) == 0;     // the key's first pass reads the column
  const bool keep = (kmask >> (digit + 1)) != 0;              // a later pass of the key reads kbuf
  const bool final_pass = A.p == total - 1;
  const bool low = (kmask >> 4) == 0, high = (kmask & 15u) == 0;
  const bool narrow = low || high;                            // the key is kept as its low or high half
  const int shift = 8 * (digit - (high ? 4 : 0));
  const int from = (A.p + 1) & 1, to = A.p & 1;
  const int64_t tiles = (n + kTileN - 1) / kTileN;
  const unsigned epoch = (unsigned)A.p + 1;
  const int64_t* off = A.offsets + ((size_t)key * kDigits + digit) * kRadix;
  const unsigned lt = (1u << lane) - 1u;
  while (true) {
    __syncthreads();
    if (threadIdx.x == 0) s_tile = atomicAdd(&A.ctl->tile_ctr[A.p], 1u);
    for (int i = threadIdx.x; i < kWarps * kRadix; i += BLOCK) (&wcnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    if (tile >= tiles) return;
    const int64_t tbase = tile * kTileN;
    const int64_t wbase = tbase + (int64_t)warp * (32 * kSortItems);
    uint64_t k[kSortItems];
    V v[kSortItems];
    unsigned rank[kSortItems];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
      const int64_t i = wbase + j * 32 + lane;
      v[j] = i >= n ? V(0) : A.p == 0 ? (V)i : A.vbuf[from][i];
    }
    if (first) {
#pragma unroll
      for (int j = 0; j < kSortItems; ++j) {
        // after an expired look-back a position may be left over from other data: it stays in bounds,
        // and the call reports the error
        const int64_t e = (int64_t)v[j] < n ? (int64_t)v[j] : n - 1;
        k[j] = 0;
        if (wbase + j * 32 + lane < n) k[j] = sort_image(K, A.perm_in ? A.perm_in[e] : e);
        if (high) k[j] >>= 32;
      }
    } else if (narrow) {
#pragma unroll
      for (int j = 0; j < kSortItems; ++j) {
        const int64_t i = wbase + j * 32 + lane;
        k[j] = i < n ? reinterpret_cast<const unsigned*>(A.kbuf[from])[i] : 0;
      }
    } else {
#pragma unroll
      for (int j = 0; j < kSortItems; ++j) {
        const int64_t i = wbase + j * 32 + lane;
        k[j] = i < n ? A.kbuf[from][i] : 0;
      }
    }
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
      const bool ok = wbase + j * 32 + lane < n;
      const unsigned d = ok ? (unsigned)(k[j] >> shift) & 255u : 256u + lane;   // out of range: a digit of its own
      const unsigned peers = __match_any_sync(0xffffffffu, d);
      unsigned base = 0;
      if (ok) base = wcnt[warp][d];
      __syncwarp();
      if (ok && lane == 31 - __clz(peers)) wcnt[warp][d] = base + __popc(peers);
      __syncwarp();
      rank[j] = base + __popc(peers & lt);
    }
    __syncthreads();
    // thread d owns digit d: warp prefixes, the tile's count (published at once), then the digits'
    // places inside the tile
    unsigned run = 0, inc = 0;
    if (threadIdx.x < kRadix) {
      const int d = threadIdx.x;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const unsigned c = wcnt[w][d];
        wcnt[w][d] = run;
        run += c;
      }
      st_relaxed(&A.status[tile * kRadix + d], st_word(tile == 0 ? 2 : 1, epoch, run));
      inc = warp_incl_scan(run);
      if (lane == 31) s_ws[warp] = inc;
    }
    __syncthreads();
    if (threadIdx.x < kRadix) {
      unsigned before = 0;
#pragma unroll
      for (int w = 0; w < kRadix / 32; ++w) before += w < warp ? s_ws[w] : 0;
      s_dbase[threadIdx.x] = before + inc - run;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
      if (wbase + j * 32 + lane < n) {
        const unsigned d = (unsigned)(k[j] >> shift) & 255u;
        const unsigned at = s_dbase[d] + wcnt[warp][d] + rank[j];
        s_key[at] = k[j];
        s_val[at] = v[j];
      }
    }
    if (threadIdx.x < kRadix) {
      const int d = threadIdx.x;
      const uint64_t excl = radix_lookback(A.status, tile, d, epoch, &A.ctl->err);
      if (tile > 0) st_relaxed(&A.status[tile * kRadix + d], st_word(2, epoch, excl + run));
      s_gbase[d] = off[d] + (int64_t)excl - (int64_t)s_dbase[d];
    }
    __syncthreads();
    const int count = (int)(n - tbase < kTileN ? n - tbase : kTileN);
    for (int i = threadIdx.x; i < count; i += BLOCK) {
      const uint64_t x = s_key[i];
      const V src = s_val[i];
      int64_t pos = s_gbase[(unsigned)(x >> shift) & 255u] + i;
      pos = pos < n ? pos : n - 1;             // in bounds also after an expired look-back
      if (keep) {
        if (narrow) reinterpret_cast<unsigned*>(A.kbuf[to])[pos] = (unsigned)x;
        else A.kbuf[to][pos] = x;
      }
      if (final_pass) {
        const int64_t e = (int64_t)src < n ? (int64_t)src : n - 1;
        A.perm_out[pos] = A.perm_in ? A.perm_in[e] : e;
      } else {
        A.vbuf[to][pos] = src;
      }
    }
  }
}

// Small sorts (n <= kSmallSort, e.g. the groups of an aggregate result): one CTA sorts (key, position)
// pairs with a bitonic network in shared memory, key by key from the last.  Ties fall to the smaller
// position, so the result is the stable order, and the host never waits.
constexpr int kSmallSort = 2048;

__global__ void __launch_bounds__(1024) k_sort_small(const __grid_constant__ SortKeySet S, const int64_t* perm_in,
                                                     int n, int64_t* perm_out) {
  __shared__ uint64_t sk[kSmallSort];
  __shared__ uint16_t si[kSmallSort];        // current order: si[i] is the position of the i-th row
  __shared__ uint16_t order[kSmallSort];
  int P = 1;
  while (P < n) P <<= 1;
  for (int i = threadIdx.x; i < n; i += blockDim.x) order[i] = static_cast<uint16_t>(i);
  __syncthreads();
  for (int key = S.n - 1; key >= 0; --key) {
    const SortKey K = S.k[key];
    for (int i = threadIdx.x; i < P; i += blockDim.x) {
      if (i < n) {
        const int pos = order[i];
        sk[i] = sort_image(K, perm_in ? perm_in[pos] : pos);
        si[i] = static_cast<uint16_t>(i);
      } else {
        sk[i] = ~0ull;
        si[i] = 0xffffu;
      }
    }
    __syncthreads();
    for (int k = 2; k <= P; k <<= 1) {
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int i = threadIdx.x; i < P; i += blockDim.x) {
          const int ixj = i ^ j;
          if (ixj > i) {
            const bool up = (i & k) == 0;
            const uint64_t ka = sk[i], kb = sk[ixj];
            const uint16_t ia = si[i], ib = si[ixj];
            const bool greater = ka > kb || (ka == kb && ia > ib);
            if (greater == up) {
              sk[i] = kb; sk[ixj] = ka;
              si[i] = ib; si[ixj] = ia;
            }
          }
        }
        __syncthreads();
      }
    }
    // order = old order through the sorted places (at most two rows per thread)
    uint16_t next[kSmallSort / 1024];
#pragma unroll
    for (int q = 0; q < kSmallSort / 1024; ++q) {
      const int i = threadIdx.x + q * 1024;
      next[q] = i < n ? order[si[i]] : 0;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kSmallSort / 1024; ++q) {
      const int i = threadIdx.x + q * 1024;
      if (i < n) order[i] = next[q];
    }
    __syncthreads();
  }
  for (int i = threadIdx.x; i < n; i += blockDim.x) perm_out[i] = perm_in ? perm_in[order[i]] : order[i];
}

// Tiles of 512 threads (8192 rows, 32-row runs) once they fill the SMs twice; 256 threads below.
constexpr int64_t kBigSort = int64_t(1) << 21;

static int64_t sort_tiles(int64_t n) {
  const int64_t t = (n >= kBigSort ? 512 : 256) * kSortItems;
  return n > 0 ? (n + t - 1) / t : 1;
}

size_t sort_ws_bytes(int64_t n, int nk) {
  const size_t m = (size_t)(n > 0 ? n : 1);
  const size_t vb = n < (int64_t(1) << 32) ? 4 : 8;
  size_t b = align_up(sizeof(SortCtl), 256);
  b += align_up((size_t)nk * kDigits * kRadix * 8, 256);            // histograms
  b += align_up((size_t)sort_tiles(n) * kRadix * 8, 256);           // look-back words
  b += align_up((size_t)nk * kDigits * kRadix * 8, 256);            // offsets
  b += 2 * align_up(m * 8, 256) + 2 * align_up(m * vb, 256);
  return b + 1024;
}

template <int BLOCK, class V>
static int run_passes(const SortKeySet& S, PassArgs<V> A, int max_passes, cudaStream_t s) {
  constexpr size_t smem = pass_smem<BLOCK, V>();
  static int per_sm = 0;
  if (!per_sm) {
    TQPK_CUDA(cudaFuncSetAttribute(k_sort_pass<BLOCK, V>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int o = 0;
    TQPK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_sort_pass<BLOCK, V>, BLOCK, smem));
    per_sm = std::max(o, 1);
  }
  const int64_t tiles = (A.n + BLOCK * kSortItems - 1) / (BLOCK * kSortItems);
  const int grid = (int)std::min<int64_t>(tiles, (int64_t)per_sm * num_sms());
  for (A.p = 0; A.p < max_passes; ++A.p) {
    timing_before(KID_SORT_PASS, s);
    k_sort_pass<BLOCK, V><<<grid, BLOCK, smem, s>>>(S, A);
    timing_after(KID_SORT_PASS, s);
    TQPK_CHECK_LAUNCH();
  }
  return TQPK_OK;
}

template <class V>
static int sort_large(const SortKeySet& S, const int64_t* perm_in, int64_t n, int64_t* perm_out, void* ws,
                      size_t ws_bytes, cudaStream_t s) {
  WsCursor cur(ws, ws_bytes);
  const size_t hist_words = (size_t)S.n * kDigits * kRadix;
  SortCtl* ctl = cur.take<SortCtl>(1);
  unsigned long long* hist = cur.take<unsigned long long>(hist_words);
  uint64_t* status = cur.take<uint64_t>((size_t)sort_tiles(n) * kRadix);
  const size_t zeroed = cur.off;
  int64_t* offsets = cur.take<int64_t>(hist_words);
  PassArgs<V> A{};
  A.kbuf[0] = cur.take<uint64_t>(n);
  A.kbuf[1] = cur.take<uint64_t>(n);
  A.vbuf[0] = cur.take<V>(n);
  A.vbuf[1] = cur.take<V>(n);
  if (!ctl || !hist || !status || !offsets || !A.kbuf[0] || !A.kbuf[1] || !A.vbuf[0] || !A.vbuf[1]) return TQPK_ENOMEM;
  TQPK_CUDA(cudaMemsetAsync(ws, 0, zeroed, s));
  const int gx = (int)std::max<int64_t>(1, std::min<int64_t>((n + kHistThreads * 16 - 1) / (kHistThreads * 16),
                                                             (int64_t)num_sms() * 2));
  k_sort_hist<<<dim3(gx, S.n), kHistThreads, 0, s>>>(S, perm_in, n, hist, offsets, ctl);
  TQPK_CHECK_LAUNCH();
  A.perm_in = perm_in;
  A.n = n;
  A.perm_out = perm_out;
  A.offsets = offsets;
  A.status = status;
  A.ctl = ctl;
  int max_passes = 0;
  for (int k = 0; k < S.n; ++k) max_passes += sort_key_digits(S.k[k]);
  const int rc = n >= kBigSort ? run_passes<512, V>(S, A, max_passes, s) : run_passes<256, V>(S, A, max_passes, s);
  if (rc) return rc;
  int err = 0;
  TQPK_CUDA(cudaMemcpyAsync(&err, &ctl->err, sizeof(int), cudaMemcpyDeviceToHost, s));
  TQPK_CUDA(cudaStreamSynchronize(s));
  return err;
}

// The stable order of elements perm_in[0..n) (null: 0..n-1) by keys[0], then keys[1], ...  perm_out must
// not overlap perm_in.  n > kSmallSort synchronises once (the look-back's error word).
int sort_keys(const SortKey* keys, int nk, const int64_t* perm_in, int64_t n, int64_t* perm_out, void* ws,
              size_t ws_bytes, cudaStream_t s) {
  if (nk < 1 || nk > kMaxSortKeys) return TQPK_EUNSUPPORTED;
  if (n == 0) return TQPK_OK;
  SortKeySet S{};
  S.n = nk;
  for (int k = 0; k < nk; ++k) S.k[k] = keys[k];
  if (n <= kSmallSort) {   // no workspace needed
    k_sort_small<<<1, 1024, 0, s>>>(S, perm_in, (int)n, perm_out);
    TQPK_CHECK_LAUNCH();
    return TQPK_OK;
  }
  if (!ws) return TQPK_EINVAL;
  if (ws_bytes < sort_ws_bytes(n, nk)) return TQPK_ENOMEM;
  if (sort_tiles(n) > INT32_MAX) return TQPK_EUNSUPPORTED;
  if (n < (int64_t(1) << 32)) return sort_large<uint32_t>(S, perm_in, n, perm_out, ws, ws_bytes, s);
  return sort_large<uint64_t>(S, perm_in, n, perm_out, ws, ws_bytes, s);
}

}  // namespace tqpk

using namespace tqpk;

extern "C" size_t tqpk_sort_workspace_bytes(int64_t n) { return sort_ws_bytes(n < 0 ? 0 : n); }

extern "C" int tqpk_argsort_stable(const void* d_keys, int32_t dt, int32_t desc, const int64_t* d_perm_in, int64_t n,
                                   int64_t* d_perm_out, void* ws, size_t ws_bytes, tqpk_stream stream) {
  if (n < 0 || (n > 0 && (!d_keys || !d_perm_out))) return TQPK_EINVAL;
  if (!dtype_size(dt)) return TQPK_EDTYPE;
  const SortKey key{d_keys, nullptr, dt, desc ? 1 : 0, 0, 0};
  return sort_keys(&key, 1, d_perm_in, n, d_perm_out, ws, ws_bytes, static_cast<cudaStream_t>(stream));
}

// Sort words of a key list (a [n, w] column is ceil(w/8) words, most significant first), or -1.
static int expand_keys(int32_t nk, const void* const* cols, const int32_t* dts, const int32_t* widths,
                       const int32_t* descs, SortKey* out, int* rc) {
  int m = 0;
  for (int k = 0; k < nk; ++k) {
    *rc = TQPK_EDTYPE;
    if (!dtype_size(dts[k]) || (widths[k] > 0 && dtype_size(dts[k]) != 1)) return -1;
    *rc = TQPK_EINVAL;
    if (widths[k] < 0) return -1;
    const int words = widths[k] > 0 ? (widths[k] + 7) / 8 : 1;
    *rc = TQPK_EUNSUPPORTED;
    if (words > kMaxSortKeys - m) return -1;
    for (int w = 0; w < words; ++w)
      out[m++] = SortKey{cols ? cols[k] : nullptr, nullptr, dts[k], descs && descs[k] ? 1 : 0, widths[k], w};
  }
  *rc = TQPK_OK;
  return m;
}

extern "C" size_t tqpk_argsort_keys_workspace_bytes(int64_t n, int32_t n_keys, const int32_t* dts,
                                                    const int32_t* widths) {
  if (n_keys < 1 || n_keys > kMaxSortKeys || !dts || !widths) return 0;
  SortKey keys[kMaxSortKeys];
  int rc;
  const int m = expand_keys(n_keys, nullptr, dts, widths, nullptr, keys, &rc);
  return m < 0 ? 0 : sort_ws_bytes(n < 0 ? 0 : n, m);
}

extern "C" int tqpk_argsort_keys(int32_t n_keys, const void* const* d_cols, const int32_t* dts, const int32_t* widths,
                                 const int32_t* descs, const int64_t* d_perm_in, int64_t n, int64_t* d_perm_out,
                                 void* ws, size_t ws_bytes, tqpk_stream stream) {
  if (n_keys < 1 || !d_cols || !dts || !widths || !descs || n < 0 || (n > 0 && !d_perm_out)) return TQPK_EINVAL;
  if (n_keys > kMaxSortKeys) return TQPK_EUNSUPPORTED;
  for (int k = 0; k < n_keys; ++k)
    if (n > 0 && !d_cols[k]) return TQPK_EINVAL;
  SortKey keys[kMaxSortKeys];
  int rc;
  const int m = expand_keys(n_keys, d_cols, dts, widths, descs, keys, &rc);
  if (m < 0) return rc;
  return sort_keys(keys, m, d_perm_in, n, d_perm_out, ws, ws_bytes, static_cast<cudaStream_t>(stream));
}
