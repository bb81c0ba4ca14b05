// sort.cu - kernel (b): stable LSD radix sort of (key, row) pairs over one or more keys.
//
// Reference: operators/sort.py:22-42 runs one stable torch.sort per key (last
// key first), permuting `perm` each time, then slices perm[:limit].
// sort_keys runs that whole loop: keys[0] is the most significant key, and the
// keys are sorted last to first, each key's digits least significant first.
// tqpk_argsort_stable is its one-key form, and waits for it beyond one CTA's rows.
//
// Up to 2048 rows are sorted by one CTA, up to 98304 by one cluster; more rows
// by the tiled passes below.
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
//   pass : a key gets at most four launches; launch q sorts by the q-th of its
//          four highest varying digits (fewer vary: the launch returns at once),
//          so the host never reads the digit masks.  The key's first pass gathers
//          the column through the rows' current order and keeps a 32-bit word of
//          it; the sort's last pass writes the int64 permutation itself.
//   fix  : a key of more than four varying digits (a price as float64 varies in
//          seven) is then ordered by its four highest digits.  Rows that agree in
//          those are already in order unless their low digits disagree with it,
//          which in real columns happens to a few neighbours: runs of up to 32
//          such rows are sorted in place.  A longer run raises a flag, and the
//          host, which waits for the sort anyway, sorts again with every digit
//          (as text is from the start).
//
// What bounds a pass: the tiles are L2-resident (8 B per row each way), so it is
// the chain load -> rank -> look-back -> write of one tile (about 1.5, 2, 3 and
// 2 us of a 4096-row tile's 9) and the instructions of the rank.  Rows are ranked
// per warp by eight ballots (match_any of 32 different digits was slower),
// reordered by digit in shared memory and written as runs, and a digit's
// look-back reads eight predecessors at a time.
#include <stddef.h>

#include <algorithm>

#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

namespace tqpk {

constexpr int kRadix = 256;
constexpr int kDigits = 8;                   // 8-bit digits of a 64-bit key
constexpr int kMaxPasses = kMaxSortKeys * kDigits;
constexpr int kHistThreads = 512;

struct SortKeySet {
  SortKey k[kMaxSortKeys];
  int n;
  int mixed;                         // the caller knows that the rows come in no order
};

struct SortCtl {
  int err;
  int redo;                          // a key's four highest digits did not order it: sort by every digit
  unsigned fixes[kMaxSortKeys];      // runs listed per key
  unsigned tile_ctr[kMaxPasses];     // next tile of each pass
  unsigned mask[kMaxSortKeys];       // varying digits per key
  unsigned ticket[kMaxSortKeys];     // hist CTAs done
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
    const int left = K.width - K.word * 8;
    // big-endian; read byte by byte, each load behind the last, it made a text key's set-up 12 us of 27.6 K
    // rows, as words ~4
    const uint64_t le = load_bytes8(static_cast<const uint8_t*>(K.col) + r * K.width + K.word * 8, left,
                                    K.word > 0 || r > 0);
    uint64_t w = ((uint64_t)__byte_perm((unsigned)le, 0, 0x0123) << 32) | __byte_perm((unsigned)(le >> 32), 0, 0x0123);
    if (K.dt == TQPK_I8)             // int8 bytes order as signed values
      w ^= left >= 8 ? 0x8080808080808080ull : 0x8080808080808080ull & ~(~0ull >> (8 * left));
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

constexpr int kSortBlock = 512;
constexpr int kSortWarps = kSortBlock / 32;
constexpr int kKeyPasses = 4;                // launches of a key: its four highest varying digits
constexpr int kFixRun = 32;                  // longest run of rows that k_sort_fix reorders

// Shared memory of a pass: the tile's keys (32-bit words, or 64-bit in the every-digit form) and
// positions, digit places, per-warp digit counts.
template <int ITEMS, class V, class K>
constexpr size_t pass_smem() {
  return (size_t)kSortBlock * ITEMS * (sizeof(K) + sizeof(V)) + kRadix * 12 + kSortWarps * kRadix * 4;
}

// The digits of `mask` a key is sorted by: the four highest varying ones, or all of them.
__device__ __forceinline__ unsigned sorted_digits(unsigned mask, bool every) {
  if (every) return mask;
  while (__popc(mask) > kKeyPasses) mask &= mask - 1;
  return mask;
}

template <class V>
struct PassArgs {
  SortKey key;
  const int64_t* perm_in;    // element of position i (null: i)
  int64_t n;
  void* kbuf[2];
  V* vbuf[2];
  int64_t* perm_out;
  const int64_t* offsets;    // of this key: [kDigits][kRadix]
  uint64_t* status;
  SortCtl* ctl;
  int k, nk;                 // this key's index, and the number of keys
  int q;                     // which of the key's digits
  unsigned every;            // bit k: key k is sorted by every varying digit
};

// How many passes run before key k's, and in all.
template <class V>
__device__ __forceinline__ void pass_counts(const PassArgs<V>& A, int& before, int& total) {
  before = 0;
  total = 0;
  for (int j = A.nk - 1; j >= 0; --j) {
    const int c = __popc(sorted_digits(A.ctl->mask[j], (A.every >> j) & 1u));
    total += c;
    if (j > A.k) before += c;
  }
}

// V: type of a row's position among the n rows (uint32 below 2^32 rows).  K: uint32, the key's four
// highest varying digits packed, or uint64, the whole key, when every digit is sorted by.
template <int ITEMS, class V, class K>
__global__ void __launch_bounds__(kSortBlock, 2) k_sort_pass(const __grid_constant__ PassArgs<V> A) {
  constexpr int kTileN = kSortBlock * ITEMS;
  constexpr bool kEvery = sizeof(K) == 8;
  extern __shared__ __align__(16) unsigned char smem[];
  K* s_key = reinterpret_cast<K*>(smem);
  V* s_val = reinterpret_cast<V*>(s_key + kTileN);
  int64_t* s_gbase = reinterpret_cast<int64_t*>(s_val + kTileN);
  unsigned* s_dbase = reinterpret_cast<unsigned*>(s_gbase + kRadix);
  unsigned(*wcnt)[kRadix] = reinterpret_cast<unsigned(*)[kRadix]>(s_dbase + kRadix);
  __shared__ unsigned s_tile;
  __shared__ unsigned s_ws[kRadix / 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned varying = A.ctl->mask[A.k];
  const unsigned digits = sorted_digits(varying, kEvery);
  const int64_t n = A.n;
  int before, total;
  pass_counts(A, before, total);
  if (A.q >= __popc(digits)) {
    if (total == 0 && A.k == 0 && A.q == 0)       // no digit varies: the order stays as it is
      for (int64_t i = blockIdx.x * (int64_t)kSortBlock + threadIdx.x; i < n; i += (int64_t)gridDim.x * kSortBlock)
        A.perm_out[i] = A.perm_in ? A.perm_in[i] : i;
    return;
  }
  const int p = before + A.q;
  unsigned left = digits;
  for (int q = A.q; q > 0; --q) left &= left - 1;
  const int digit = __ffs(left) - 1;
  const bool more = (left & (left - 1)) != 0;                 // a later pass of this key
  const bool keep = more || varying != digits;                // that pass, or k_sort_check, reads kbuf
  const bool final_pass = p == total - 1;
  const bool keep_row = !final_pass || varying != digits;
  // the 32-bit word of a key holds its sorted digits side by side
  const int shift = kEvery ? 8 * digit : 8 * A.q;
  const int from = (p + 1) & 1, to = p & 1;
  const int64_t tiles = (n + kTileN - 1) / kTileN;
  const unsigned epoch = (unsigned)p + 1;
  const int64_t* off = A.offsets + digit * kRadix;
  const unsigned lt = (1u << lane) - 1u;
  while (true) {
    __syncthreads();
    if (threadIdx.x == 0) s_tile = atomicAdd(&A.ctl->tile_ctr[p], 1u);
    for (int i = threadIdx.x; i < kSortWarps * kRadix; i += kSortBlock) (&wcnt[0][0])[i] = 0;
    __syncthreads();
    const int64_t tile = s_tile;
    if (tile >= tiles) return;
    const int64_t tbase = tile * kTileN;
    const int64_t wbase = tbase + (int64_t)warp * (32 * ITEMS);
    K k[ITEMS];
    V v[ITEMS];
    unsigned rank[ITEMS];
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const int64_t i = wbase + j * 32 + lane;
      v[j] = i >= n ? V(0) : p == 0 ? (V)i : A.vbuf[from][i];
    }
    if (A.q == 0) {
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        // after an expired look-back a position may be left over from other data: it stays in bounds,
        // and the call reports the error
        const int64_t e = (int64_t)v[j] < n ? (int64_t)v[j] : n - 1;
        k[j] = 0;
        if (wbase + j * 32 + lane < n) {
          const uint64_t u = sort_image(A.key, A.perm_in ? A.perm_in[e] : e);
          if (kEvery) {
            k[j] = (K)u;
          } else {
            unsigned w = 0, d = digits;
#pragma unroll
            for (int q = 0; q < kKeyPasses; ++q) {
              if (d) w |= ((unsigned)(u >> (8 * (__ffs(d) - 1))) & 255u) << (8 * q);
              d &= d - 1;
            }
            k[j] = (K)w;
          }
        }
      }
    } else {
      const K* in = static_cast<const K*>(A.kbuf[from]);
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const int64_t i = wbase + j * 32 + lane;
        k[j] = i < n ? in[i] : 0;
      }
    }
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
      const bool ok = wbase + j * 32 + lane < n;
      const unsigned d = (unsigned)(k[j] >> shift) & 255u;
      unsigned peers = __ballot_sync(0xffffffffu, ok);     // lanes of the warp with the same digit
#pragma unroll
      for (int b = 0; b < 8; ++b) {
        const bool set = (d >> b) & 1u;
        const unsigned m = __ballot_sync(0xffffffffu, set);
        peers &= set ? m : ~m;
      }
      const int leader = ok ? 31 - __clz(peers) : lane;
      unsigned old = 0;
      if (ok && lane == leader) old = atomicAdd(&wcnt[warp][d], (unsigned)__popc(peers));
      rank[j] = __shfl_sync(0xffffffffu, old, leader) + __popc(peers & lt);
      __syncwarp();
    }
    __syncthreads();
    // thread d owns digit d: warp prefixes, the tile's count (published at once), then the digits'
    // places inside the tile
    unsigned run = 0, inc = 0;
    if (threadIdx.x < kRadix) {
      const int d = threadIdx.x;
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) {
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
      unsigned below = 0;
#pragma unroll
      for (int w = 0; w < kRadix / 32; ++w) below += w < warp ? s_ws[w] : 0;
      s_dbase[threadIdx.x] = below + inc - run;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < ITEMS; ++j) {
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
#pragma unroll 4
    for (int i = threadIdx.x; i < count; i += kSortBlock) {
      const K x = s_key[i];
      const V src = s_val[i];
      int64_t pos = s_gbase[(unsigned)(x >> shift) & 255u] + i;
      pos = pos < n ? pos : n - 1;             // in bounds also after an expired look-back
      if (keep) static_cast<K*>(A.kbuf[to])[pos] = x;
      if (final_pass) {
        const int64_t e = (int64_t)src < n ? (int64_t)src : n - 1;
        A.perm_out[pos] = A.perm_in ? A.perm_in[e] : e;
      }
      if (keep_row) A.vbuf[to][pos] = src;
    }
  }
}

template <class V>
__device__ __forceinline__ int64_t pass_element(const PassArgs<V>& A, V v) {
  const int64_t e = (int64_t)v < A.n ? (int64_t)v : A.n - 1;
  return A.perm_in ? A.perm_in[e] : e;
}

// After the passes of a key that varies in more digits than it was sorted by: neighbours with one word
// are compared by the whole key.  The first pair of a run (rows of one word) found out of order puts
// the run's first row on the list that k_sort_fix works off (the free position buffer); a run longer
// than kFixRun sets ctl->redo.
template <class V>
__global__ void __launch_bounds__(kBlock) k_sort_check(const __grid_constant__ PassArgs<V> A) {
  const unsigned varying = A.ctl->mask[A.k];
  if (varying == sorted_digits(varying, false)) return;
  int before, total;
  pass_counts(A, before, total);
  const int at = (before + kKeyPasses - 1) & 1;
  const unsigned* word = static_cast<const unsigned*>(A.kbuf[at]);
  const V* pos = A.vbuf[at];
  V* list = A.vbuf[at ^ 1];
  const int64_t n = A.n;
  const int lane = threadIdx.x & 31;
  for (int64_t i0 = blockIdx.x * (int64_t)kBlock + (threadIdx.x & ~31); i0 < n; i0 += (int64_t)gridDim.x * kBlock) {
    const int64_t i = i0 + lane;
    const unsigned w = i < n ? word[i] : 0;
    const bool joins = i > 0 && i < n && word[i - 1] == w;
    const int below = __shfl_down_sync(0xffffffffu, (int)joins, 1);     // one shuffle, taken by all lanes
    const bool next = lane < 31 && below;
    uint64_t u = 0;
    if (joins || next) u = sort_image(A.key, pass_element(A, pos[i]));
    uint64_t prev = __shfl_up_sync(0xffffffffu, u, 1);
    if (joins && lane == 0) prev = sort_image(A.key, pass_element(A, pos[i - 1]));
    if (!joins || prev <= u) continue;
    // out of order: the run's first such pair if every pair before it in the run is in order
    int64_t head = i - 1;
    uint64_t x = prev;
    bool mine = true;
    while (head > 0 && word[head - 1] == w) {
      if (i - head >= kFixRun) {
        A.ctl->redo = 1;
        mine = false;
        break;
      }
      const uint64_t y = sort_image(A.key, pass_element(A, pos[head - 1]));
      if (y > x) {
        mine = false;
        break;
      }
      x = y;
      --head;
    }
    if (mine) list[atomicAdd(&A.ctl->fixes[A.k], 1u)] = (V)head;
  }
}

// Orders each listed run by the whole key: a stable insertion sort of at most kFixRun rows.
template <class V>
__global__ void __launch_bounds__(kBlock) k_sort_fix(const __grid_constant__ PassArgs<V> A) {
  const int64_t fixes = A.ctl->fixes[A.k];
  if (fixes == 0 || A.ctl->redo) return;
  int before, total;
  pass_counts(A, before, total);
  const int at = (before + kKeyPasses - 1) & 1;
  const unsigned* word = static_cast<const unsigned*>(A.kbuf[at]);
  V* pos = A.vbuf[at];
  const V* list = A.vbuf[at ^ 1];
  for (int64_t f = blockIdx.x * (int64_t)kBlock + threadIdx.x; f < fixes; f += (int64_t)gridDim.x * kBlock) {
    const int64_t i = (int64_t)list[f];
    const unsigned w = word[i];
    uint64_t key[kFixRun];
    V row[kFixRun];
    int m = 0;
    for (int64_t j = i; j < A.n && word[j] == w; ++j) {
      if (m == kFixRun) {
        A.ctl->redo = 1;
        m = 0;
        break;
      }
      const V v = pos[j];
      const uint64_t u = sort_image(A.key, pass_element(A, v));
      int b = m++;
      for (; b > 0 && key[b - 1] > u; --b) {
        key[b] = key[b - 1];
        row[b] = row[b - 1];
      }
      key[b] = u;
      row[b] = v;
    }
    for (int a = 0; a < m; ++a) {
      pos[i + a] = row[a];
      if (before + kKeyPasses == total) A.perm_out[i + a] = pass_element(A, row[a]);
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
  // every read before the first write: perm_out may be perm_in, or a key column
  int64_t row[kSmallSort / 1024];
#pragma unroll
  for (int q = 0; q < kSmallSort / 1024; ++q) {
    const int i = threadIdx.x + q * 1024;
    row[q] = i < n ? (perm_in ? perm_in[order[i]] : order[i]) : 0;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kSmallSort / 1024; ++q) {
    const int i = threadIdx.x + q * 1024;
    if (i < n) perm_out[i] = row[q];
  }
}

// Mid-size sorts (the groups of an aggregate, small tables): the rows live in the shared memory of one
// cluster of 16 CTAs for the whole sort, every key and digit of it in one launch.  As launches these
// sorts were 60 passes of seven tiles: each ~15 us of latency for 0.3 MB of rows, two synchronisations a
// key.  A pass here is rank, exchange of the CTAs' digit counts, and a scatter into the owning CTA's
// buffer (distributed shared memory), with two hardware cluster barriers and no look-back.  Digits are
// the 8-bit windows that start at the lowest varying bit not yet sorted by.  Text is first recoded: a byte
// becomes its rank among the values its position takes, in as few bits as those need (letters of a word
// list: 3-4 bits instead of the 7 that vary), which halves its passes; keys whose varying bits lie within 32
// of each other travel in one word with the position (27.6 K rows by four keys, 25-byte text among them: 166
// -> 129 us; a 24-bit integer key 28.8 -> 24.5).
constexpr int kClusterCtas = 16;
constexpr int kClusterThreads = 512;
constexpr int kClusterWarps = kClusterThreads / 32;
constexpr int kClusterItemsSmall = 4, kClusterItemsLarge = 12;
constexpr int64_t kClusterSort = (int64_t)kClusterCtas * kClusterThreads * kClusterItemsLarge;   // 98304 rows

template <int ITEMS>
struct ClusterSmem {
  static constexpr int kRows = kClusterThreads * ITEMS;
  uint64_t key[2][kRows];            // packed: the key's varying 32 bits above the position; else the key
  unsigned val[2][kRows];            // not packed: the position
  unsigned wcnt[kClusterWarps][kRadix];
  unsigned counts[2][kClusterCtas][kRadix];   // every CTA's digit counts, by pass parity
  unsigned base[kRadix];
  uint64_t bits[2][2];               // OR, AND of this CTA's keys, by key parity
  unsigned ws[kClusterWarps];
  unsigned seen[2][8][8];            // text: byte values at each of a word's positions in this CTA, by key parity
  unsigned values[8][8];             // the same over the cluster
  uint8_t rank[8][256];              // a value's place among them
  int width[8];                      // bits of a position's rank
  unsigned broken;                   // this CTA's word of cluster_broken
};

// Whether rows e0, e1 are out of order by keys[from..to).
__device__ __forceinline__ bool out_of_order(const SortKeySet& S, int from, int to, int64_t e0, int64_t e1) {
  for (int f = from; f < to; ++f) {
    const uint64_t a = sort_image(S.k[f], e0), b = sort_image(S.k[f], e1);
    if (a != b) return a > b;
  }
  return false;
}

// What this CTA's rows (and the row after them) say about the order the rows come in.  Bit 0: not the
// order of all the keys; bit 1: not the order of the keys behind the first column (from `rest` on).  The
// groups of an aggregate come in the order of their keys, and most reports sort them by a total and then
// those keys, or by the keys alone: then the first column's passes are the whole sort, or there are none.
// Rows in any other order say so within the first 512 of a CTA, and the CTA stops looking.
// 27.6 K groups by a count and then their three keys, two of them text: 129 us without, 47 with; 27.6 K
// random integers 25 us without, 27 with, 60 K 39.6 and 39.7.
template <int ITEMS>
__device__ __forceinline__ unsigned cluster_broken(const SortKeySet& S, int rest, const int64_t* perm_in, int n,
                                                   int first, int mine) {
  unsigned broken = rest < S.n ? 0 : 2;
  for (int j = 0; j < ITEMS && broken != 3; ++j) {
    const int i = j * kClusterThreads + threadIdx.x;
    bool all = false, later = false;
    if (i < mine && first + i + 1 < n) {
      const int64_t e0 = perm_in ? perm_in[first + i] : first + i, e1 = perm_in ? perm_in[first + i + 1] : first + i + 1;
      if (!(broken & 1)) all = out_of_order(S, 0, S.n, e0, e1);
      if (!(broken & 2)) later = out_of_order(S, rest, S.n, e0, e1);
    }
    if (__syncthreads_or(all)) broken |= 1;
    if (__syncthreads_or(later)) broken |= 2;
  }
  return broken;
}

// Recodes this CTA's rows' words of text (M.key[cur][i]) as the ranks of their bytes; returns the bits used.
template <int ITEMS>
__device__ __forceinline__ int cluster_recode(cg::cluster_group& cluster, ClusterSmem<ITEMS>& M, int cur, int mine,
                                              int parity, bool desc) {
  unsigned(*seen)[8] = M.seen[parity];
  if (threadIdx.x < 64) seen[threadIdx.x >> 3][threadIdx.x & 7] = 0;
  __syncthreads();
  for (int i = threadIdx.x; i < mine; i += kClusterThreads) {
    const uint64_t u = M.key[cur][i];
    unsigned known[8];
#pragma unroll
    for (int p = 0; p < 8; ++p)
      known[p] = *const_cast<volatile unsigned*>(&seen[p][((unsigned)(u >> (8 * p)) & 255u) >> 5]);
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      const unsigned b = (unsigned)(u >> (8 * p)) & 255u, bit = 1u << (b & 31);
      if (!(known[p] & bit)) atomicOr(&seen[p][b >> 5], bit);
    }
  }
  cluster.sync();
  if (threadIdx.x < 64) {
    unsigned m = 0;
#pragma unroll
    for (int c = 0; c < kClusterCtas; ++c) m |= cluster.map_shared_rank(&seen[0][0], c)[threadIdx.x];
    M.values[threadIdx.x >> 3][threadIdx.x & 7] = m;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 8 * 256; i += kClusterThreads) {
    const int p = i >> 8, b = i & 255;
    int r = __popc(M.values[p][b >> 5] & ((1u << (b & 31)) - 1u)), n_values = 0;
#pragma unroll
    for (int w = 0; w < 8; ++w) {
      const int c = __popc(M.values[p][w]);
      r += w < (b >> 5) ? c : 0;
      n_values += c;
    }
    M.rank[p][b] = (uint8_t)r;
    if (b == 0) M.width[p] = n_values > 1 ? 32 - __clz(n_values - 1) : 0;
  }
  __syncthreads();
  int total_bits = 0;
#pragma unroll
  for (int p = 0; p < 8; ++p) total_bits += M.width[p];
  const uint64_t full = total_bits >= 64 ? ~0ull : (1ull << total_bits) - 1ull;
  for (int i = threadIdx.x; i < mine; i += kClusterThreads) {
    const uint64_t u = M.key[cur][i];
    uint64_t w = 0;
    int at = 0;
#pragma unroll
    for (int p = 0; p < 8; ++p) {
      w |= (uint64_t)M.rank[p][(u >> (8 * p)) & 255u] << at;         // a zero-width position has rank 0
      at += M.width[p];
    }
    M.key[cur][i] = desc ? full - w : w;
  }
  return total_bits;
}

template <int ITEMS>
__global__ void __launch_bounds__(kClusterThreads) k_sort_cluster(const __grid_constant__ SortKeySet S,
                                                                  const int64_t* perm_in, int n,
                                                                  int64_t* perm_out) {
  extern __shared__ __align__(16) unsigned char raw[];
  ClusterSmem<ITEMS>& M = *reinterpret_cast<ClusterSmem<ITEMS>*>(raw);
  cg::cluster_group cluster = cg::this_cluster();
  const int cta = (int)cluster.block_rank();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  const unsigned R = ((unsigned)n + kClusterCtas - 1) / kClusterCtas;        // rows per CTA (<= kRows)
  const int mine = max(0, min((int)R, n - cta * (int)R));
  int cur = 0, pass = 0;
  for (int i = threadIdx.x; i < mine; i += kClusterThreads) M.val[0][i] = (unsigned)(cta * (int)R + i);
  int rest = 1;                      // the second column's first key
  while (rest < S.n && S.k[rest].word > 0) ++rest;
  const unsigned here = S.mixed ? 3 : cluster_broken<ITEMS>(S, rest, perm_in, n, cta * (int)R, mine);
  if (threadIdx.x == 0) M.broken = here;
  cluster.sync();                    // every CTA of the cluster runs before any writes to another
  const unsigned broken = __reduce_or_sync(0xffffffffu, *cluster.map_shared_rank(&M.broken, lane % kClusterCtas));
  const int sorted_from = !(broken & 1) ? 0 : !(broken & 2) ? rest : S.n;
  bool packed = false;               // where the positions are: in key, or in val
  for (int key = sorted_from - 1; key >= 0; --key) {
    SortKey K = S.k[key];
    const bool text = K.width > 0, desc = K.desc != 0;
    if (text) K.desc = 0;            // turned round after the recoding
    uint64_t any = 0, all = ~0ull;
    for (int i = threadIdx.x; i < mine; i += kClusterThreads) {
      const unsigned v = packed ? (unsigned)M.key[cur][i] : M.val[cur][i];
      const uint64_t u = sort_image(K, perm_in ? perm_in[v] : (int64_t)v);
      M.key[cur][i] = u;
      M.val[cur][i] = v;
      any |= u;
      all &= u;
    }
    uint64_t vary;                   // the same in every CTA, so all run the same passes
    if (text) {
      __syncthreads();
      const int bits = cluster_recode<ITEMS>(cluster, M, cur, mine, key & 1, desc);
      vary = bits >= 64 ? ~0ull : (1ull << bits) - 1ull;
    } else {
      if (threadIdx.x == 0) {
        M.bits[key & 1][0] = 0;
        M.bits[key & 1][1] = ~0ull;
      }
      __syncthreads();
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        any |= __shfl_xor_sync(0xffffffffu, any, o);
        all &= __shfl_xor_sync(0xffffffffu, all, o);
      }
      if (lane == 0) {
        atomicOr(reinterpret_cast<unsigned long long*>(&M.bits[key & 1][0]), (unsigned long long)any);
        atomicAnd(reinterpret_cast<unsigned long long*>(&M.bits[key & 1][1]), (unsigned long long)all);
      }
      cluster.sync();
      any = 0;
      all = ~0ull;
      if (lane < kClusterCtas) {
        const uint64_t* b = cluster.map_shared_rank(&M.bits[key & 1][0], lane);
        any = b[0];
        all = b[1];
      }
#pragma unroll
      for (int o = 16; o; o >>= 1) {
        any |= __shfl_xor_sync(0xffffffffu, any, o);
        all &= __shfl_xor_sync(0xffffffffu, all, o);
      }
      vary = any & ~all;
    }
    // varying bits within 32 of each other: one word of 32 key bits and the position, one remote store a row
    const int low = vary ? __ffsll((long long)vary) - 1 : 0;
    packed = (vary >> low) >> 32 == 0;
    if (packed) {
      __syncthreads();
      for (int i = threadIdx.x; i < mine; i += kClusterThreads)
        M.key[cur][i] = ((M.key[cur][i] >> low) << 32) | M.val[cur][i];
      vary = (vary >> low) << 32;
    }
    while (vary) {
      const int shift = __ffsll((long long)vary) - 1;
      vary = shift + 8 < 64 ? vary & (~0ull << (shift + 8)) : 0;
      for (int i = threadIdx.x; i < kClusterWarps * kRadix; i += kClusterThreads) (&M.wcnt[0][0])[i] = 0;
      __syncthreads();
      uint64_t k[ITEMS];
      unsigned v[ITEMS], rank[ITEMS];
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        const int i = warp * (32 * ITEMS) + j * 32 + lane;
        const bool ok = i < mine;
        k[j] = ok ? M.key[cur][i] : 0;
        v[j] = ok && !packed ? M.val[cur][i] : 0;
        const unsigned d = (unsigned)(k[j] >> shift) & 255u;
        unsigned peers = __ballot_sync(0xffffffffu, ok);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const bool set = (d >> b) & 1u;
          const unsigned m = __ballot_sync(0xffffffffu, set);
          peers &= set ? m : ~m;
        }
        const int leader = ok ? 31 - __clz(peers) : lane;
        unsigned old = 0;
        if (ok && lane == leader) old = atomicAdd(&M.wcnt[warp][d], (unsigned)__popc(peers));
        rank[j] = __shfl_sync(0xffffffffu, old, leader) + __popc(peers & lt);
        __syncwarp();
      }
      __syncthreads();
      // the tile's digit counts go to every CTA before the barrier (reading them after it cost a round trip)
      if (threadIdx.x < kRadix) {
        unsigned run = 0;
#pragma unroll
        for (int w = 0; w < kClusterWarps; ++w) {
          const unsigned c = M.wcnt[w][threadIdx.x];
          M.wcnt[w][threadIdx.x] = run;
          run += c;
        }
#pragma unroll
        for (int c = 0; c < kClusterCtas; ++c)
          cluster.map_shared_rank(&M.counts[pass & 1][cta][0], c)[threadIdx.x] = run;
      }
      cluster.sync();
      unsigned total = 0, before = 0, inc = 0;
      if (threadIdx.x < kRadix) {
#pragma unroll
        for (int c = 0; c < kClusterCtas; ++c) {
          const unsigned x = M.counts[pass & 1][c][threadIdx.x];
          before += c < cta ? x : 0;
          total += x;
        }
        inc = warp_incl_scan(total);
        if (lane == 31) M.ws[warp] = inc;
      }
      __syncthreads();
      if (threadIdx.x < kRadix) {
        unsigned below = 0;
#pragma unroll
        for (int w = 0; w < kRadix / 32; ++w) below += w < warp ? M.ws[w] : 0;
        M.base[threadIdx.x] = below + inc - total + before;
      }
      __syncthreads();
#pragma unroll
      for (int j = 0; j < ITEMS; ++j) {
        if (warp * (32 * ITEMS) + j * 32 + lane < mine) {
          const unsigned d = (unsigned)(k[j] >> shift) & 255u;
          const unsigned pos = M.base[d] + M.wcnt[warp][d] + rank[j];
          const unsigned owner = pos / R, at = pos - owner * R;
          cluster.map_shared_rank(&M.key[cur ^ 1][0], owner)[at] = k[j];
          if (!packed) cluster.map_shared_rank(&M.val[cur ^ 1][0], owner)[at] = v[j];
        }
      }
      cluster.sync();
      cur ^= 1;
      ++pass;
    }
    __syncthreads();
  }
  int64_t row[ITEMS];
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = j * kClusterThreads + threadIdx.x;
    row[j] = 0;
    if (i < mine) {
      const unsigned v = packed ? (unsigned)M.key[cur][i] : M.val[cur][i];
      row[j] = perm_in ? perm_in[v] : (int64_t)v;
    }
  }
  // no CTA leaves while another may still reach into it, and every read of perm_in and the key columns comes
  // before the first write: perm_out may be one of them
  cluster.sync();
#pragma unroll
  for (int j = 0; j < ITEMS; ++j) {
    const int i = j * kClusterThreads + threadIdx.x;
    if (i < mine) perm_out[cta * (int64_t)R + i] = row[j];
  }
}

// One cluster, where the device can hold one (launched is set), else nothing.
template <int ITEMS>
static int run_cluster(const SortKeySet& S, const int64_t* perm_in, int n, int64_t* perm_out, bool& launched,
                       cudaStream_t s) {
  constexpr size_t smem = sizeof(ClusterSmem<ITEMS>);
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = kClusterCtas;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.gridDim = dim3(kClusterCtas);
  cfg.blockDim = dim3(kClusterThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  static PerDevice resident;           // clusters the device holds at a time, plus one
  const int fits = resident.get([&] {
    int clusters = 0;
    if (cudaFuncSetAttribute(k_sort_cluster<ITEMS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess ||
        cudaFuncSetAttribute(k_sort_cluster<ITEMS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&clusters, k_sort_cluster<ITEMS>, &cfg) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
    }
    return clusters + 1;
  });
  launched = fits > 1;
  if (!launched) return TQPK_OK;
  TQPK_CUDA(cudaLaunchKernelEx(&cfg, k_sort_cluster<ITEMS>, S, perm_in, n, perm_out));
  ++g_launches;
  return TQPK_OK;
}

// Rows per thread of a pass.  All tiles of a sort of up to 1.2 M rows are resident at once at eight
// (two CTAs of 4096 rows per SM); larger sorts take twelve, whose longer runs and fewer look-backs
// cost less per row.
constexpr int kItemsSmall = 8, kItemsLarge = 12;
constexpr int64_t kLargeSort = int64_t(1200) << 10;

static int64_t sort_tiles(int64_t n) {
  const int64_t t = (n > kLargeSort ? kItemsLarge : kItemsSmall) * kSortBlock;
  return n > 0 ? (n + t - 1) / t : 1;
}

size_t sort_ws_bytes(int64_t n, int nk) {
  const size_t m = (size_t)(n > 0 ? n : 1);
  const size_t vb = n < (int64_t(1) << 32) ? 4 : 8;
  size_t b = align_up(sizeof(SortCtl), 256);
  b += align_up((size_t)nk * kDigits * kRadix * 8, 256);            // histograms
  // look-back words; just above kLargeSort the tiles are fewer than at it, and a workspace for n rows serves
  // any fewer
  b += align_up((size_t)std::max(sort_tiles(n), sort_tiles(std::min(n, kLargeSort))) * kRadix * 8, 256);
  b += align_up((size_t)nk * kDigits * kRadix * 8, 256);            // offsets
  b += 2 * align_up(m * 8, 256) + 2 * align_up(m * vb, 256);
  return b + 1024;
}

// The passes of one key.
template <int ITEMS, class V, class K>
static int run_key(PassArgs<V> A, cudaStream_t s) {
  constexpr size_t smem = pass_smem<ITEMS, V, K>();
  static PerDevice resident;           // CTAs per SM
  const int per_sm = resident.get([&] {
    int o = 0;
    if (cudaFuncSetAttribute(k_sort_pass<ITEMS, V, K>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
            cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, k_sort_pass<ITEMS, V, K>, kSortBlock, smem) != cudaSuccess) {
      (void)cudaGetLastError();
      return 0;
    }
    return std::max(o, 1);
  });
  if (per_sm <= 0) return TQPK_ECUDA;
  const int grid = (int)std::min<int64_t>(sort_tiles(A.n), (int64_t)per_sm * num_sms());
  const int nd = sort_key_digits(A.key);
  const int passes = sizeof(K) == 8 ? nd : std::min(nd, kKeyPasses);
  for (A.q = 0; A.q < passes; ++A.q) {
    timing_before(KID_SORT_PASS, s);
    k_sort_pass<ITEMS, V, K><<<grid, kSortBlock, smem, s>>>(A);
    timing_after(KID_SORT_PASS, s);
    TQPK_CHECK_LAUNCH();
  }
  if (passes == nd) return TQPK_OK;
  k_sort_check<V><<<grid_for(A.n, 8), kBlock, 0, s>>>(A);
  TQPK_CHECK_LAUNCH();
  k_sort_fix<V><<<num_sms(), kBlock, 0, s>>>(A);
  TQPK_CHECK_LAUNCH();
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
  A.perm_in = perm_in;
  A.n = n;
  A.perm_out = perm_out;
  A.status = status;
  A.ctl = ctl;
  A.nk = S.n;
  // four rows a thread for one key (0.8 M rows: 13 us, 18 with sixteen); several keys fill the SMs together
  const int64_t per_cta = (int64_t)kHistThreads * (S.n == 1 ? 4 : 16);
  const int gx = (int)std::max<int64_t>(1, std::min<int64_t>((n + per_cta - 1) / per_cta, (int64_t)num_sms() * 2));
  // eight letters of text rarely differ in the first four only: text is sorted by every digit
  for (int k = 0; k < S.n; ++k) A.every |= S.k[k].width ? 1u << k : 0u;
  for (int attempt = 0; attempt < 2; ++attempt) {
    if (attempt == 0) {
      TQPK_CUDA(cudaMemsetAsync(ws, 0, zeroed, s));
      k_sort_hist<<<dim3(gx, S.n), kHistThreads, 0, s>>>(S, perm_in, n, hist, offsets, ctl);
      TQPK_CHECK_LAUNCH();
    } else {                         // the masks and offsets stay
      A.every = ~0u;
      TQPK_CUDA(cudaMemsetAsync(ctl, 0, offsetof(SortCtl, mask), s));
      TQPK_CUDA(cudaMemsetAsync(status, 0, (size_t)sort_tiles(n) * kRadix * sizeof(uint64_t), s));
    }
    for (int k = S.n - 1; k >= 0; --k) {
      A.key = S.k[k];
      A.k = k;
      A.offsets = offsets + (size_t)k * kDigits * kRadix;
      const bool large = n > kLargeSort;
      const int rc = (A.every >> k) & 1u ? (large ? run_key<kItemsLarge, V, uint64_t>(A, s) : run_key<kItemsSmall, V, uint64_t>(A, s))
                                         : (large ? run_key<kItemsLarge, V, uint32_t>(A, s) : run_key<kItemsSmall, V, uint32_t>(A, s));
      if (rc) return rc;
    }
    int h[2] = {0, 0};               // [0] error, [1] a key needs every digit
    TQPK_CUDA(cudaMemcpyAsync(h, ctl, sizeof(h), cudaMemcpyDeviceToHost, s));
    TQPK_CUDA(cudaStreamSynchronize(s));
    if (h[0]) return h[0];
    if (!h[1]) return TQPK_OK;
  }
  return TQPK_ETIMEOUT;              // not reached: the second attempt sorts by every digit
}

// Whether perm_out shares memory with perm_in or a key column: the passes read both until the last one writes.
static bool sort_in_place(const SortKey* keys, int nk, const int64_t* perm_in, int64_t n, const int64_t* perm_out) {
  const uintptr_t o0 = reinterpret_cast<uintptr_t>(perm_out), o1 = o0 + (uintptr_t)n * 8;
  auto meets = [&](const void* p, uintptr_t bytes) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p);
    return p && a < o1 && o0 < a + bytes;
  };
  bool in = meets(perm_in, (uintptr_t)n * 8);
  for (int k = 0; k < nk && !in; ++k)
    in = meets(keys[k].col, (uintptr_t)n * (keys[k].width ? keys[k].width : dtype_size(keys[k].dt)));
  return in;
}

// Workspace of the exported sorts: sort_ws_bytes, and a permutation for an in-place call.
static size_t argsort_ws_bytes(int64_t n, int nk) {
  return sort_ws_bytes(n, nk) + (n > kSmallSort ? align_up((size_t)n * 8, 256) : 0);
}

// The stable order of elements perm_in[0..n) (null: 0..n-1) by keys[0], then keys[1], ...  perm_out may be
// perm_in (or a key column) given argsort_ws_bytes: the tiled passes then write to the workspace, and the order
// is copied out behind them.  n > kClusterSort synchronises once (the look-back's error word).  mixed: the rows
// are known to come in no order (entries of a hash table in the order they were claimed), so nothing looks for
// one.
int sort_keys(const SortKey* keys, int nk, const int64_t* perm_in, int64_t n, int64_t* perm_out, void* ws,
              size_t ws_bytes, cudaStream_t s, bool mixed) {
  if (nk < 1 || nk > kMaxSortKeys) return TQPK_EUNSUPPORTED;
  if (n == 0) return TQPK_OK;
  SortKeySet S{};
  S.n = nk;
  S.mixed = mixed;
  for (int k = 0; k < nk; ++k) S.k[k] = keys[k];
  if (n <= kSmallSort) {   // no workspace needed
    k_sort_small<<<1, 1024, 0, s>>>(S, perm_in, (int)n, perm_out);
    TQPK_CHECK_LAUNCH();
    return TQPK_OK;
  }
  if (!ws) return TQPK_EINVAL;
  if (ws_bytes < sort_ws_bytes(n, nk)) return TQPK_ENOMEM;
  if (n <= kClusterSort) {
    bool launched = false;
    const int rc = n <= kClusterCtas * kClusterThreads * kClusterItemsSmall
                       ? run_cluster<kClusterItemsSmall>(S, perm_in, (int)n, perm_out, launched, s)
                       : run_cluster<kClusterItemsLarge>(S, perm_in, (int)n, perm_out, launched, s);
    if (rc || launched) return rc;
  }
  if (sort_tiles(n) > INT32_MAX) return TQPK_EUNSUPPORTED;
  WsCursor cur(ws, ws_bytes);
  int64_t* order = perm_out;
  if (sort_in_place(keys, nk, perm_in, n, perm_out)) order = cur.take<int64_t>(n);
  if (!order) return TQPK_ENOMEM;
  void* rest = cur.base + cur.off;
  const int rc = n < (int64_t(1) << 32) ? sort_large<uint32_t>(S, perm_in, n, order, rest, ws_bytes - cur.off, s)
                                        : sort_large<uint64_t>(S, perm_in, n, order, rest, ws_bytes - cur.off, s);
  if (rc || order == perm_out) return rc;
  TQPK_CUDA(cudaMemcpyAsync(perm_out, order, (size_t)n * 8, cudaMemcpyDeviceToDevice, s));
  return TQPK_OK;
}

}  // namespace tqpk

using namespace tqpk;

extern "C" size_t tqpk_sort_workspace_bytes(int64_t n) { return argsort_ws_bytes(n < 0 ? 0 : n, 1); }

extern "C" int tqpk_argsort_stable(const void* d_keys, int32_t dt, int32_t desc, const int64_t* d_perm_in, int64_t n,
                                   int64_t* d_perm_out, void* ws, size_t ws_bytes, tqpk_stream stream) {
  if (n < 0 || (n > 0 && (!d_keys || !d_perm_out))) return TQPK_EINVAL;
  if (!dtype_size(dt)) return TQPK_EDTYPE;
  const SortKey key{d_keys, nullptr, dt, desc ? 1 : 0, 0, 0};
  const int rc = sort_keys(&key, 1, d_perm_in, n, d_perm_out, ws, ws_bytes, static_cast<cudaStream_t>(stream));
  // one launch or many, a sort beyond one CTA is complete when the call returns
  if (rc == TQPK_OK && n > kSmallSort) TQPK_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  return rc;
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

// Test hook: the form for 2^32 rows and more (8-byte positions) on any number of rows above the cluster's.
extern "C" int tqpk_debug_argsort_wide(int32_t n_keys, const void* const* d_cols, const int32_t* dts,
                                       const int32_t* widths, const int32_t* descs, const int64_t* d_perm_in, int64_t n,
                                       int64_t* d_perm_out, void* ws, size_t ws_bytes, tqpk_stream stream) {
  if (n_keys < 1 || n_keys > kMaxSortKeys || !d_cols || !dts || !widths || !descs || n <= kClusterSort || !d_perm_out || !ws)
    return TQPK_EINVAL;
  SortKeySet S{};
  int rc;
  S.n = expand_keys(n_keys, d_cols, dts, widths, descs, S.k, &rc);
  if (S.n < 0) return rc;
  return sort_large<uint64_t>(S, d_perm_in, n, d_perm_out, ws, ws_bytes, static_cast<cudaStream_t>(stream));
}

extern "C" size_t tqpk_argsort_keys_workspace_bytes(int64_t n, int32_t n_keys, const int32_t* dts,
                                                    const int32_t* widths) {
  if (n_keys < 1 || n_keys > kMaxSortKeys || !dts || !widths) return 0;
  SortKey keys[kMaxSortKeys];
  int rc;
  const int m = expand_keys(n_keys, nullptr, dts, widths, nullptr, keys, &rc);
  return m < 0 ? 0 : argsort_ws_bytes(n < 0 ? 0 : n, m);
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
