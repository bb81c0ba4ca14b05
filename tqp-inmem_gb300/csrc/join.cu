// join.cu - kernel (c): equi-join probe emitting (build_row, probe_row) pairs.
//
// Reference: operators/hashjoin.py:24-177 sorts the build keys, takes
// unique_consecutive + counts + an exclusive prefix, binary-searches every
// probe key (searchsorted), expands duplicates through a padded (m, lmax)
// arange matrix with masked_select / repeat_interleave (several host syncs),
// re-checks key equality and gathers the output columns.
//
// Here the build side is turned into a directory once:
//   DIRECT  dense key range (<= max(4*rows, 2^24) slots): dir[slot = key - min]
//           = a build row of that key.  That answers a unique build side, and a
//           semi or anti join of any.  Only a join that needs every build row of
//           a repeated key also gets the rows radix-sorted stably by key (csr,
//           ascending row inside a key) and run[slot] = the key's csr range.
//   SORTED  sparse keys: the same stable sort, plus the distinct keys and run
//           starts; the probe binary-searches the distinct keys (the
//           reference's searchsorted, on a deduplicated array).
// Probes with at most one output per probe row (unique build keys; semi, anti)
// are one single-pass kernel: warps read 128 consecutive rows at a time, the
// hits are placed in shared memory by block scan and written contiguously at the
// tile's decoupled look-back offset.  Repeated build keys take two kernels: the
// pairs of every tile are counted, then written at the scanned offsets, each
// thread finding its pair's probe row by a search in the tile's scan, so that
// consecutive threads write consecutive pairs.  Either way pairs come by
// ascending probe row, as the reference's do, then ascending build row (the
// reference sorts build keys with an unstable torch.sort, hashjoin.py:43, so its
// order of one key's duplicate build rows is not fixed; this is the stable one).
// Rows failing either side's filter mask are skipped in place: the inputs are
// never compacted, and the emitted ids index the original columns.
//
// Measured on the operators' plans (1.5 M orders, 6 M lines): a semi-join whose
// build side repeats its keys took 1003 us with the csr it never read; pairs of
// a key repeated four times (24 M) were written by one thread per probe row,
// 534 us of the probe.
#include <algorithm>

#include "common.cuh"

namespace tqpk {

struct JoinDir {
  int mode, wide;           // wide: 64-bit entries (2^32 - 1 build rows or more)
  int64_t key_min, slots, n_unique;
  const void* dir;          // DIRECT: a build row per slot, all ones = empty
  const void* run;          // DIRECT, repeated keys: (start, end) in csr per slot
  const int64_t* csr;       // build rows sorted by (key, row); null: dir holds the one row
  const int64_t* ukeys;     // SORTED: distinct keys
  const int64_t* ustart;    // SORTED: run starts (n_unique + 1 entries)
};

// A compaction leaves a negative status in its count when a look-back gave up.
__global__ void k_count_status(const int64_t* count, int* err) {
  if (*count < 0) set_error(err, (int)*count);
}

// dir[slot] = a build row of the key; *dup set when a key has two.  Four exchanges are in flight per thread.
template <class R>
__global__ void __launch_bounds__(kBlock) k_join_build_direct(const void* keys, int dt, RowFilter F, int64_t nb,
                                                              int64_t kmin, int kvec, R* __restrict__ dir, int* dup) {
  bool repeated = false;
  const int64_t groups = (nb + 3) >> 2;
  for (int64_t g = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; g < groups;
       g += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r0 = g << 2;
    int64_t valid = nb - r0;
    uint32_t b = valid >= 4 ? 0xfu : ((1u << valid) - 1);
    if (F.mask) {
      int64_t m[4];
      ld4_int(F.mask, TQPK_U8, r0, nb, F.mask_vec, m);
      b &= (m[0] != 0) | ((m[1] != 0) << 1) | ((m[2] != 0) << 2) | ((m[3] != 0) << 3);
    }
    if (!b) continue;
    int64_t x[4];
    ld4_int(keys, dt, r0, nb, kvec != 0, x);
    // of neighbouring rows with one key (a table stored by it) only the last is exchanged
    unsigned last = b;
#pragma unroll
    for (int j = 0; j < 3; ++j)
      if (((b >> j) & 3u) == 3u && x[j] == x[j + 1]) last &= ~(1u << j);
    repeated |= last != b;
    R old[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      old[j] = R(~R(0));
      if ((last >> j) & 1u) {
        if (sizeof(R) == 4) old[j] = (R)atomicExch(reinterpret_cast<unsigned*>(&dir[x[j] - kmin]), (unsigned)(r0 + j));
        else old[j] = (R)atomicExch(reinterpret_cast<unsigned long long*>(&dir[x[j] - kmin]), (unsigned long long)(r0 + j));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) repeated |= old[j] != R(~R(0));
  }
  // one store per CTA: a store per repeated row queued on the word (6 M rows of a key repeated four times: 50
  // us, 77 with a row count per key beside the directory)
  if (__syncthreads_or(repeated) && threadIdx.x == 0) *dup = 1;
}

// After the stable sort (csr[i] = i-th build row in (key, row) order): each run's range by slot (DIRECT,
// run zeroed before), or the head flags (SORTED).
template <class R>
__global__ void k_join_runs(const void* keys, int dt, const int64_t* csr, int64_t m, int64_t kmin, int direct,
                            int64_t slots, R* run, int64_t* head_flag_rows) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = ld_int(keys, dt, csr[i]);
    const bool head = (i == 0) || ld_int(keys, dt, csr[i - 1]) != k;
    if (direct) {
      const bool tail = i + 1 == m || ld_int(keys, dt, csr[i + 1]) != k;
      const int64_t slot = k - kmin;
      if (slot < 0 || slot >= slots) continue;          // keys changed since the plan was made: stay in bounds
      if (head) run[2 * slot] = (R)i;
      if (tail) run[2 * slot + 1] = (R)(i + 1);
    } else {
      head_flag_rows[i] = head ? 1 : 0;
    }
  }
}

// SORTED mode: distinct keys + run starts from the head flags (ordered).
__global__ void __launch_bounds__(kBlock) k_join_unique(const void* keys, int dt, const int64_t* csr,
                                                        const int64_t* head, int64_t m, int64_t* ukeys,
                                                        int64_t* ustart, int64_t* nu, uint64_t* status,
                                                        int* tile_ctr, int* err) {
  __shared__ int s_tile;
  __shared__ uint64_t s_excl;
  __shared__ int sw[kBlock / 32 + 1];
  if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr, 1);
  __syncthreads();
  const int64_t tile = s_tile;
  const int64_t i0 = tile * kTile + threadIdx.x * kItems;
  uint32_t bits = 0;
  for (int j = 0; j < kItems; ++j)
    if (i0 + j < m && head[i0 + j]) bits |= 1u << j;
  int total;
  const int excl = block_excl_scan<kBlock, int>(__popc(bits), total, sw);
  if (threadIdx.x < 32) {
    uint64_t e = lookback_warp(status, tile, (uint64_t)total, err);
    if (threadIdx.x == 0) s_excl = e;
  }
  __syncthreads();
  int64_t pos = (int64_t)s_excl + excl;
  while (bits) {
    const int j = __ffs(bits) - 1;
    bits &= bits - 1;
    ukeys[pos] = ld_int(keys, dt, csr[i0 + j]);
    ustart[pos] = i0 + j;
    ++pos;
  }
  if (tile == (int64_t)gridDim.x - 1 && threadIdx.x == 0) {
    *nu = (int64_t)(s_excl + total);
    ustart[s_excl + total] = m;
  }
}

// The distinct key at or after `key` in a sorted directory: its index when equal, else -1.
__device__ __forceinline__ int64_t join_find(const JoinDir& D, int64_t key) {
  int64_t lo = 0, hi = D.n_unique;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (D.ukeys[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo < D.n_unique && D.ukeys[lo] == key ? lo : -1;
}

// The csr range [first, first + count) of a probe key's build rows (a unique directory: first is the row).
__device__ __forceinline__ int64_t join_range(const JoinDir& D, int64_t key, int64_t& first) {
  if (D.mode != TQPK_JOIN_DIRECT) {
    const int64_t u = join_find(D, key);
    if (u < 0) return 0;
    first = D.ustart[u];
    return D.ustart[u + 1] - first;
  }
  const int64_t slot = key - D.key_min;
  if (slot < 0 || slot >= D.slots) return 0;
  if (!D.csr) {
    if (D.wide) {
      const uint64_t r = static_cast<const uint64_t*>(D.dir)[slot];
      first = (int64_t)r;
      return r != ~0ull;
    }
    const unsigned r = static_cast<const unsigned*>(D.dir)[slot];
    first = r;
    return r != ~0u;
  }
  if (D.wide) {
    const longlong2 q = static_cast<const longlong2*>(D.run)[slot];
    first = q.x;
    return q.y - q.x;
  }
  const uint2 q = static_cast<const uint2*>(D.run)[slot];
  first = q.x;
  return (int64_t)(q.y - q.x);
}


// Probes with at most one output per row.  dup (inner join of a build side not known to be unique):
// nothing is done when it is set.
template <int JT, bool DIRECT, class R>
__global__ void __launch_bounds__(kBlock) k_join_probe(JoinDir D, const void* pkeys, int pdt, RowFilter F, int64_t np,
                                                       int64_t* __restrict__ out_b, int64_t* __restrict__ out_p,
                                                       int64_t capacity, const int64_t* base_ptr, int64_t* total_out,
                                                       uint64_t* status, int* tile_ctr, const int* dup, int* err) {
  __shared__ int s_tile;
  __shared__ uint64_t s_excl;
  __shared__ int s_warp[kBlock / 32 + 1];
  __shared__ uint16_t s_p[kTile];                      // row of the tile, by output place
  __shared__ R s_b[JT == TQPK_JT_INNER ? kTile : 1];   // its build row
  if (dup && *dup) return;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) s_tile = atomicAdd(tile_ctr, 1);
  __syncthreads();
  const int64_t tile = s_tile;
  // warp w reads rows [512 w, 512 w + 512) of the tile, 128 consecutive rows a load
  const int64_t w0 = tile * kTile + warp * (32 * kItems);
  const bool kvec = ((reinterpret_cast<uintptr_t>(pkeys) & 15u) == 0);
  uint32_t hits = 0;
  R row[kItems];
  uint32_t live[kItems / 4];
  int64_t key[kItems];
#pragma unroll
  for (int q = 0; q < kItems / 4; ++q) {
    const int64_t g0 = w0 + 128 * q + 4 * lane;
    const int64_t valid = np - g0;
    uint32_t b = valid >= 4 ? 0xfu : (valid <= 0 ? 0u : ((1u << valid) - 1));
    if (F.mask && b) {
      int64_t m[4];
      ld4_int(F.mask, TQPK_U8, g0, np, F.mask_vec, m);
      b &= (m[0] != 0) | ((m[1] != 0) << 1) | ((m[2] != 0) << 2) | ((m[3] != 0) << 3);
    }
    live[q] = b;
  }
#pragma unroll
  for (int q = 0; q < kItems / 4; ++q) {
    int64_t x[4] = {0, 0, 0, 0};
    if (live[q]) ld4_int(pkeys, pdt, w0 + 128 * q + 4 * lane, np, kvec, x);
#pragma unroll
    for (int j = 0; j < 4; ++j) key[4 * q + j] = x[j];
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const bool on = (live[i / 4] >> (i & 3)) & 1u;
    row[i] = R(~R(0));
    if (DIRECT) {
      const int64_t slot = key[i] - D.key_min;
      if (on && slot >= 0 && slot < D.slots) row[i] = static_cast<const R*>(D.dir)[slot];
    } else if (on && join_find(D, key[i]) >= 0) {
      row[i] = 0;
    }
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const bool on = (live[i / 4] >> (i & 3)) & 1u;
    const bool hit = row[i] != R(~R(0));
    if (JT == TQPK_JT_ANTI ? on && !hit : hit) hits |= 1u << i;
  }
  // output places: the four 128-row steps' counts (at most 128 each) share one warp scan
  unsigned c = 0;
#pragma unroll
  for (int q = 0; q < kItems / 4; ++q) c |= __popc((hits >> (4 * q)) & 15u) << (8 * q);
  unsigned even = c & 0x00ff00ffu, odd = (c >> 8) & 0x00ff00ffu;
  const unsigned ie = warp_incl_scan(even), io = warp_incl_scan(odd);
  const unsigned te = __shfl_sync(0xffffffffu, ie, 31), to = __shfl_sync(0xffffffffu, io, 31);
  const unsigned step_total[4] = {te & 0xffffu, to & 0xffffu, te >> 16, to >> 16};
  const unsigned xe = ie - even, xo = io - odd;
  const unsigned before[4] = {xe & 0xffffu, xo & 0xffffu, xe >> 16, xo >> 16};
  const int wtotal = (int)(step_total[0] + step_total[1] + step_total[2] + step_total[3]);
  if (lane == 0) s_warp[warp] = wtotal;
  __syncthreads();
  int total = 0, wbase = 0;
#pragma unroll
  for (int w = 0; w < kBlock / 32; ++w) {
    if (w == warp) wbase = total;
    total += s_warp[w];
  }
  unsigned at0 = wbase;
#pragma unroll
  for (int q = 0; q < kItems / 4; ++q) {
    unsigned at = at0 + before[q];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if ((hits >> (4 * q + j)) & 1u) {
        s_p[at] = (uint16_t)(warp * (32 * kItems) + 128 * q + 4 * lane + j);
        if (JT == TQPK_JT_INNER) s_b[at] = row[4 * q + j];
        ++at;
      }
    }
    at0 += step_total[q];
  }
  if (threadIdx.x < 32) {
    uint64_t e = lookback_warp(status, tile, (uint64_t)total, err);
    if (threadIdx.x == 0) s_excl = e;
  }
  __syncthreads();
  const int64_t gbase = (base_ptr ? *base_ptr : 0) + (int64_t)s_excl;
  for (int i = threadIdx.x; i < total; i += kBlock) {
    if (gbase + i >= capacity) break;
    out_p[gbase + i] = tile * kTile + s_p[i];
    if (JT == TQPK_JT_INNER) out_b[gbase + i] = (int64_t)s_b[i];
    else if (JT == TQPK_JT_ANTI && out_b) out_b[gbase + i] = (int64_t)TQPK_NULL_INDEX;
  }
  if (tile == (int64_t)gridDim.x - 1 && threadIdx.x == 0) *total_out = gbase + total;
}

// ---- joins whose build key repeats: count the pairs of every tile, scan, write -------------------
constexpr int kPairRows = 4 * kBlock;        // probe rows per tile

struct PairCtl {
  unsigned done;          // counting CTAs finished
  int pad;
  int64_t total;          // pairs in all
};

// The join's extra conditions: a numeric predicate program over columns of both sides (bit c of
// probe_cols: column c is the probe side's).
struct PairCond {
  tqpk_predicate P;
  unsigned probe_cols;
  // The usual condition, one comparison of an integer column of each side (a second key): build <cmp> probe.
  int two_sided, cmp, build_dt, probe_dt;
  const void* build_col;
  const void* probe_col;
  const int64_t* vals;      // the build column's values in csr order (null: read by build row)
};

// What the counting pass of a join with conditions leaves for the writing one: per tile whether its threads
// took their own rows' pairs, then which of them hold (bit 16 j + t: pair t of a thread's row j) and where
// each row's build rows start (4-byte entries only).
struct PairKept {
  uint8_t* by_row;
  uint64_t* held;
  unsigned* first;
};

__global__ void k_pair_vals(const void* __restrict__ col, int dt, const int64_t* __restrict__ csr, int64_t m,
                            int64_t* __restrict__ vals) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x)
    vals[i] = ld_int(col, dt, csr[i]);
}

__device__ __forceinline__ bool pair_cmp(const PairCond& C, const tqpk_pred_insn& I, int64_t b, int64_t p) {
  const int64_t r = (C.probe_cols >> I.col) & 1u ? p : b;
  const void* col = C.P.cols[I.col];
  const int dt = C.P.dtypes[I.col];
  if (I.op == TQPK_P_MASK) return ld_int(col, TQPK_U8, r) != 0;
  if (I.op == TQPK_P_CMPCOL) {
    const int c2 = (int)I.lit_i;
    const int64_t r2 = (C.probe_cols >> c2) & 1u ? p : b;
    if (I.domain == TQPK_DOM_F64) return cmp_op<double>(I.cmp, ld_f64(col, dt, r), ld_f64(C.P.cols[c2], C.P.dtypes[c2], r2));
    return cmp_op<int64_t>(I.cmp, ld_int(col, dt, r), ld_int(C.P.cols[c2], C.P.dtypes[c2], r2));
  }
  if (I.domain == TQPK_DOM_F64) {
    const double x = ld_f64(col, dt, r);
    if (I.cmp != TQPK_ISCLOSE) return cmp_op<double>(I.cmp, x, I.lit_f);
    const double err = fabs(__dsub_rn(x, I.lit_f));
    return (x == I.lit_f) || (isfinite(err) && err <= I.lit_aux);
  }
  const int64_t x = ld_int(col, dt, r);
  if (I.domain == TQPK_DOM_F32) return cmp_op<float>(I.cmp, static_cast<float>(x), static_cast<float>(I.lit_f));
  return cmp_op<int64_t>(I.cmp, x, I.lit_i);
}

// The program for build row b and probe row p; the stack is a word of bits (at most 32 deep).
__device__ __forceinline__ bool pair_holds(const PairCond& C, int64_t b, int64_t p) {
  unsigned st = 0;
  for (int k = 0; k < C.P.n_insn; ++k) {
    const tqpk_pred_insn& I = C.P.insn[k];
    switch (I.op) {
      case TQPK_P_AND: st = ((st >> 1) & ~1u) | ((st >> 1) & st & 1u); break;
      case TQPK_P_OR: st = (st >> 1) | (st & 1u); break;
      case TQPK_P_NOT: st ^= 1u; break;
      case TQPK_P_TRUE: st = (st << 1) | 1u; break;
      case TQPK_P_FALSE: st <<= 1; break;
      default: st = (st << 1) | (pair_cmp(C, I, b, p) ? 1u : 0u); break;
    }
  }
  return st & 1u;
}

// Pass COUNT leaves each tile's pair count in tile_base; its last CTA scans them into offsets.  COND: only
// the pairs that satisfy C count (24 M pairs of a key repeated four times, one in four kept: materialising
// them, gathering the condition's columns and compacting took ~600 us).  What bounds it is the L1's handling
// of scattered lanes, about one a clock: the csr entry and the build column's value of every pair, in both
// passes, took 248 + 300 us.  So the usual condition's build column is laid out in csr order first, a row's
// values then come two to a load, and a tile whose rows have at most kRowPairs candidates each gives every
// thread its own four rows and keeps its verdicts for the writing pass.  Longer runs are spread over the
// block pair by pair, by a search in the tile's scan, in both passes; where the probe side has too few tiles
// for the GPU, gridDim.y CTAs share a tile's pairs, each a consecutive part of them (3000 x 3000 rows of one key
// with a second key, three tiles: 23.4 ms with one CTA a tile, which had to judge its pairs twice, 15.4 when they
// were written, gathered, filtered and compacted, now 0.49; 20 K probe rows of ordinary runs as before).
constexpr int kRowPairs = 16;

template <bool COUNT, bool COND>
__global__ void __launch_bounds__(kBlock) k_join_pairs(JoinDir D, const void* pkeys, int pdt, RowFilter F, int64_t np,
                                                       int kvec, int64_t* __restrict__ out_b,
                                                       int64_t* __restrict__ out_p, int64_t capacity,
                                                       int64_t* __restrict__ tile_base, PairCtl* ctl, PairKept W,
                                                       const __grid_constant__ PairCond C) {
  constexpr bool kRows = !COUNT || COND;
  __shared__ int64_t sw[kBlock / 32 + 1];
  __shared__ int64_t s_pre[kRows ? kPairRows : 1];     // pairs before each row of the tile
  __shared__ int64_t s_first[kRows ? kPairRows : 1];   // where its build rows start
  __shared__ int s_last;
  const int64_t tile = blockIdx.x;
  const int part = blockIdx.y, parts = gridDim.y;
  const int64_t slot = tile * parts + part;             // of tile_base
  const int64_t g0 = tile * kPairRows + 4 * threadIdx.x;
  if (!COUNT && COND && W.by_row[tile]) {
    if (part > 0) return;
    uint64_t held = W.held[tile * kBlock + threadIdx.x];
    const uint4 f4 = *reinterpret_cast<const uint4*>(&W.first[4 * (tile * kBlock + threadIdx.x)]);
    int64_t kept;
    int64_t at = tile_base[slot] + block_excl_scan<kBlock, int64_t>(__popcll(held), kept, sw);
    for (; held; held &= held - 1, ++at) {
      const int q = __ffsll((long long)held) - 1, j = q >> 4;
      const int64_t f = (int64_t)(j == 0 ? f4.x : j == 1 ? f4.y : j == 2 ? f4.z : f4.w) + (q & 15);
      if (at >= capacity) break;
      out_p[at] = g0 + j;
      out_b[at] = D.csr ? D.csr[f] : f;
    }
    return;
  }
  const int64_t valid = np - g0;
  uint32_t b = valid >= 4 ? 0xfu : (valid <= 0 ? 0u : ((1u << valid) - 1));
  if (F.mask && b) {
    int64_t m[4];
    ld4_int(F.mask, TQPK_U8, g0, np, F.mask_vec, m);
    b &= (m[0] != 0) | ((m[1] != 0) << 1) | ((m[2] != 0) << 2) | ((m[3] != 0) << 3);
  }
  int64_t x[4] = {0, 0, 0, 0}, first[4] = {0, 0, 0, 0}, cnt[4];
  if (b) ld4_int(pkeys, pdt, g0, np, kvec != 0, x);
  int64_t mine = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    cnt[j] = (b >> j) & 1u ? join_range(D, x[j], first[j]) : 0;
    mine += cnt[j];
  }
  int64_t total;
  int64_t excl = block_excl_scan<kBlock, int64_t>(mine, total, sw);
  // pair o of the tile: its probe row (the last one with s_pre <= o) and build row
  auto pair = [&](int64_t o, int& row, int64_t& build) {
    int lo = 0, hi = kPairRows;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      if (s_pre[mid] <= o) lo = mid; else hi = mid;
    }
    const int64_t f = s_first[lo] + (o - s_pre[lo]);
    row = lo;
    build = D.csr ? D.csr[f] : f;
  };
  __shared__ unsigned s_kept[2][kBlock / 32];
  const bool by_row = COUNT && COND && !__syncthreads_or(D.wide || cnt[0] > kRowPairs || cnt[1] > kRowPairs ||
                                                         cnt[2] > kRowPairs || cnt[3] > kRowPairs);
  if (COUNT && COND && threadIdx.x == 0 && part == 0) W.by_row[tile] = by_row;
  int64_t from = total * part / parts, to = total * (part + 1) / parts;       // this CTA's pairs of the tile
  if (by_row && part > 0) to = from = total = 0;
  if (by_row && part == 0) {
    uint64_t held = 0;
    int64_t pv[4] = {0, 0, 0, 0};
    if (b && C.two_sided) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (cnt[j]) pv[j] = ld_int(C.probe_col, C.probe_dt, g0 + j);
    }
    const int most = (int)max(max(cnt[0], cnt[1]), max(cnt[2], cnt[3]));
    for (int t = 0; C.vals && t < most; t += 2) {
      int64_t v[4][2];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int64_t* p = C.vals + first[j] + t;
        const int left = (int)cnt[j] - t;
        if (left >= 2 && (first[j] & 1) == 0) {
          const longlong2 a = *reinterpret_cast<const longlong2*>(p);
          v[j][0] = a.x;
          v[j][1] = a.y;
        } else {
          v[j][0] = left >= 1 ? p[0] : 0;
          v[j][1] = left >= 2 ? p[1] : 0;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int left = (int)cnt[j] - t;
        const uint64_t two = (left >= 1 && cmp_op<int64_t>(C.cmp, v[j][0], pv[j]) ? 1u : 0u) |
                             (left >= 2 && cmp_op<int64_t>(C.cmp, v[j][1], pv[j]) ? 2u : 0u);
        held |= two << (16 * j + t);
      }
    }
    for (int t = 0; !C.vals && t < most; ++t) {
      int64_t build[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) build[j] = t < cnt[j] ? (D.csr ? D.csr[first[j] + t] : first[j] + t) : -1;
      if (C.two_sided) {
        int64_t bv[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) bv[j] = build[j] >= 0 ? ld_int(C.build_col, C.build_dt, build[j]) : 0;
#pragma unroll
        for (int j = 0; j < 4; ++j)
          held |= (uint64_t)(build[j] >= 0 && cmp_op<int64_t>(C.cmp, bv[j], pv[j])) << (16 * j + t);
      } else {
#pragma unroll 1
        for (int j = 0; j < 4; ++j)
          if (build[j] >= 0) held |= (uint64_t)pair_holds(C, build[j], g0 + j) << (16 * j + t);
      }
    }
    W.held[tile * kBlock + threadIdx.x] = held;
    *reinterpret_cast<uint4*>(&W.first[4 * (tile * kBlock + threadIdx.x)]) =
        make_uint4((unsigned)first[0], (unsigned)first[1], (unsigned)first[2], (unsigned)first[3]);
    block_excl_scan<kBlock, int64_t>(__popcll(held), total, sw);
  } else {
    total = to - from;
  }
  if (kRows && !by_row) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      s_pre[4 * threadIdx.x + j] = excl;
      s_first[4 * threadIdx.x + j] = first[j];
      excl += cnt[j];
    }
    __syncthreads();
  }
  if (COUNT && COND && !by_row) {
    int64_t kept = 0;
    for (int64_t o = from + threadIdx.x; o < to; o += kBlock) {
      int row;
      int64_t build;
      pair(o, row, build);
      kept += pair_holds(C, build, tile * kPairRows + row) ? 1 : 0;
    }
    block_excl_scan<kBlock, int64_t>(kept, total, sw);
  }
  if (COUNT) {
    const int64_t slots = (int64_t)gridDim.x * parts;
    if (threadIdx.x == 0) {
      tile_base[slot] = total;
      __threadfence();
      s_last = atomicAdd(&ctl->done, 1u) == (unsigned)(slots - 1);
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    int64_t run = 0;
    for (int64_t t0 = 0; t0 < slots; t0 += 4 * kBlock) {
      int64_t c[4], sum = 0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int64_t t = t0 + 4 * threadIdx.x + q;
        c[q] = t < slots ? __ldcg(reinterpret_cast<const long long*>(&tile_base[t])) : 0;
        sum += c[q];
      }
      int64_t all;
      int64_t at = run + block_excl_scan<kBlock, int64_t>(sum, all, sw);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int64_t t = t0 + 4 * threadIdx.x + q;
        if (t < slots) tile_base[t] = at;
        at += c[q];
      }
      run += all;
    }
    if (threadIdx.x == 0) ctl->total = run;
    return;
  }
  int64_t base = tile_base[slot];
  if (!COND) {
    base -= from;
    for (int64_t o = from + threadIdx.x; o < to; o += kBlock) {
      if (base + o >= capacity) break;
      int row;
      int64_t build;
      pair(o, row, build);
      out_p[base + o] = tile * kPairRows + row;
      out_b[base + o] = build;
    }
    return;
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int64_t o0 = from; o0 < to; o0 += kBlock) {
    const int64_t o = o0 + threadIdx.x;
    int row = 0;
    int64_t build = 0;
    bool keep = false;
    if (o < to) {
      pair(o, row, build);
      keep = pair_holds(C, build, tile * kPairRows + row);
    }
    const unsigned m = __ballot_sync(0xffffffffu, keep);
    unsigned* kept = s_kept[((o0 - from) / kBlock) & 1];
    if (lane == 0) kept[warp] = __popc(m);
    __syncthreads();                 // two buffers: the next chunk's counts do not overwrite this one's
    int64_t at = base + __popc(m & ((1u << lane) - 1u));
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) {
      at += w < warp ? kept[w] : 0;
      base += kept[w];
    }
    if (keep && at < capacity) {
      out_p[at] = tile * kPairRows + row;
      out_b[at] = build;
    }
  }
}

// Column c of the rows idx[j], four rows per thread: their reads are all in flight before the first write
// (one row at a time, a thread waited for every column of it: 41 us for the six columns of 1.5 M joined rows).
constexpr int kGatherRows = 4;

template <class T>
__device__ __forceinline__ void gather_column(const void* in, void* out, const int64_t (&i)[kGatherRows], int64_t j0,
                                              int64_t n, unsigned null, T null_value) {
  const T* src = static_cast<const T*>(in);
  T v[kGatherRows];
#pragma unroll
  for (int u = 0; u < kGatherRows; ++u) v[u] = j0 + u * kBlock < n && !((null >> u) & 1u) ? src[i[u]] : null_value;
#pragma unroll
  for (int u = 0; u < kGatherRows; ++u)
    if (j0 + u * kBlock < n) static_cast<T*>(out)[j0 + u * kBlock] = v[u];
}

__global__ void __launch_bounds__(kBlock) k_gather(int ncols, const __grid_constant__ ColSet C,
                                                   const int64_t* __restrict__ idx, int64_t n, int null_aware) {
  for (int64_t t0 = blockIdx.x * (int64_t)(kGatherRows * kBlock); t0 < n;
       t0 += (int64_t)gridDim.x * (kGatherRows * kBlock)) {
    const int64_t j0 = t0 + threadIdx.x;
    int64_t i[kGatherRows];
    unsigned null = 0;
#pragma unroll
    for (int u = 0; u < kGatherRows; ++u) i[u] = j0 + u * kBlock < n ? idx[j0 + u * kBlock] : 0;
#pragma unroll
    for (int u = 0; u < kGatherRows; ++u) null |= (unsigned)(null_aware && i[u] == TQPK_NULL_INDEX) << u;
    for (int c = 0; c < ncols; ++c) {
      switch (C.size[c]) {
        case 1: gather_column<uint8_t>(C.in[c], C.out[c], i, j0, n, null, (uint8_t)(int8_t)TQPK_NULL_INDEX); break;
        case 4: gather_column<int32_t>(C.in[c], C.out[c], i, j0, n, null, TQPK_NULL_INDEX); break;
        case 8: gather_column<int64_t>(C.in[c], C.out[c], i, j0, n, null, TQPK_NULL_INDEX); break;
        default: gather_column<double>(C.in[c], C.out[c], i, j0, n, null, (double)TQPK_NULL_INDEX); break;
      }
    }
  }
}

// ---------------------------------------------------------------- host side
struct BuildLayout {
  int* hdr;            // [0] dup flag, [1] error, [2] tile counter
  int64_t* nu;         // distinct keys (SORTED)
  void* dir;           // one entry per slot (4 bytes, or 8 when wide)
  void* run;           // two entries per slot
  int64_t* csr;
  int64_t* rows;       // the passing build rows in row order (a masked build side)
  int64_t* ukeys;
  int64_t* ustart;
  int64_t* head;
  void* sort_ws;
  size_t sort_bytes;
  uint64_t* status;
};

// Entries are 4 bytes unless a plan says otherwise; wide plans have unique's bit 8 set.
constexpr int kWide = 256;
static bool is_wide(const tqpk_join_plan& p) { return (p.unique & kWide) != 0; }
static int uniqueness(const tqpk_join_plan& p) { return p.unique & ~kWide; }

static bool layout(const tqpk_join_plan& p, void* ws, size_t bytes, BuildLayout& L) {
  WsCursor c(ws, bytes);
  const int64_t m = p.nb_rows > 0 ? p.nb_rows : 1;
  const size_t e = is_wide(p) ? 8 : 4;
  const bool direct = p.mode == TQPK_JOIN_DIRECT;
  L.hdr = c.take<int>(64);
  L.nu = c.take<int64_t>(4);
  L.dir = c.take<char>(direct ? p.slots * e : 1);
  L.run = c.take<char>(direct ? 2 * p.slots * e : 1);
  L.csr = c.take<int64_t>(m);
  L.rows = c.take<int64_t>(m);
  L.ukeys = c.take<int64_t>(direct ? 1 : m);
  L.ustart = c.take<int64_t>(direct ? 1 : m + 1);
  L.head = c.take<int64_t>(direct ? 1 : m);
  L.status = c.take<uint64_t>((m + kTile - 1) / kTile + 1);
  // the rest: the sort's, or the compaction's of a masked build side, which goes by its rows before the mask
  const size_t used = align_up(c.off, 256);
  L.sort_bytes = bytes > used ? (bytes - used) / 256 * 256 : 0;
  L.sort_ws = c.take<char>(L.sort_bytes);
  return L.sort_ws != nullptr && L.sort_bytes >= sort_ws_bytes(m);
}

// nb: the build side's rows, those its mask drops among them (0: it has no mask).
static size_t layout_bytes(const tqpk_join_plan& p, int64_t nb) {
  const int64_t m = p.nb_rows > 0 ? p.nb_rows : 1;
  const size_t e = is_wide(p) ? 8 : 4;
  const bool direct = p.mode == TQPK_JOIN_DIRECT;
  size_t b = 256 + 256;
  b += direct ? align_up(p.slots * e, 256) + align_up(2 * p.slots * e, 256) : 512;
  b += 2 * align_up(m * 8, 256);
  b += direct ? 768 : align_up(m * 8, 256) + align_up((m + 1) * 8, 256) + align_up(m * 8, 256);
  b += align_up(((m + kTile - 1) / kTile + 1) * 8, 256);
  b += align_up(std::max(sort_ws_bytes(m), nb > 0 ? compact_status_bytes(nb) : 0), 256);
  return b + 2048;
}

// The directory a probe reads; pairs: of every build row of a key (the csr), when keys repeat.
static JoinDir make_dir(const tqpk_join_plan& p, const BuildLayout& L, bool pairs) {
  JoinDir D{};
  D.mode = p.mode;
  D.wide = is_wide(p) ? 1 : 0;
  D.key_min = p.key_min;
  D.slots = p.nb_rows > 0 ? p.slots : 0;
  D.n_unique = p.n_unique;
  D.dir = L.dir;
  D.run = L.run;
  D.csr = pairs && uniqueness(p) == 0 ? L.csr : nullptr;
  D.ukeys = L.ukeys;
  D.ustart = L.ustart;
  if (p.nb_rows == 0) D.mode = TQPK_JOIN_DIRECT;       // no slot at all
  return D;
}

template <int JT>
static int launch_probe(const JoinDir& D, const void* pkeys, int pdt, const RowFilter& F, int64_t np, int64_t* out_b,
                        int64_t* out_p, int64_t capacity, const int64_t* base, int64_t* total, uint64_t* status,
                        int* tile_ctr, const int* dup, int* err, cudaStream_t s) {
  const int64_t tiles = (np + kTile - 1) / kTile;
  timing_before(KID_JOIN_PROBE, s);
  if (D.mode != TQPK_JOIN_DIRECT) {
    if constexpr (JT != TQPK_JT_INNER)
      k_join_probe<JT, false, unsigned><<<(int)tiles, kBlock, 0, s>>>(D, pkeys, pdt, F, np, out_b, out_p, capacity, base,
                                                                      total, status, tile_ctr, dup, err);
  } else if (D.wide) {
    k_join_probe<JT, true, uint64_t><<<(int)tiles, kBlock, 0, s>>>(D, pkeys, pdt, F, np, out_b, out_p, capacity, base,
                                                                   total, status, tile_ctr, dup, err);
  } else {
    k_join_probe<JT, true, unsigned><<<(int)tiles, kBlock, 0, s>>>(D, pkeys, pdt, F, np, out_b, out_p, capacity, base,
                                                                   total, status, tile_ctr, dup, err);
  }
  timing_after(KID_JOIN_PROBE, s);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

struct ProbeLayout {
  int* ctl;              // [0] tile counter A, [1] error, [2] tile counter B, [3] a repeated build key
  int64_t* totals;
  PairCtl* pair;
  uint64_t* status_a;
  uint64_t* status_b;
  size_t zeroed;
  int64_t* tile_base;
  PairKept kept;         // joins with conditions
  int64_t* vals;
};

// CTAs that share a tile's pairs: two per SM in all while the tiles are fewer than that.
constexpr int64_t kMaxParts = 128, kPartSlots = 1024;       // at most tiles + kPartSlots places in tile_base
static dim3 pair_grid(int64_t tiles) {
  const int64_t want = std::min<int64_t>(2 * num_sms(), kPartSlots);
  const int64_t parts = tiles < want ? std::min(kMaxParts, (want + tiles - 1) / tiles) : 1;
  return dim3((unsigned)tiles, (unsigned)parts);
}

static bool probe_layout(int64_t np, void* pws, size_t bytes, ProbeLayout& W, int64_t cond_build_rows = -1) {
  const int64_t tiles = (np + kTile - 1) / kTile;
  WsCursor cur(pws, bytes);
  W.ctl = cur.take<int>(64);
  W.totals = cur.take<int64_t>(8);
  W.pair = cur.take<PairCtl>(1);
  W.status_a = cur.take<uint64_t>(tiles + 1);
  W.status_b = cur.take<uint64_t>(tiles + 1);
  W.zeroed = cur.off;
  const int64_t ptiles = (np + kPairRows - 1) / kPairRows;
  W.tile_base = cur.take<int64_t>(ptiles + kPartSlots + 1);
  if (cond_build_rows < 0) return W.tile_base != nullptr;
  W.kept.by_row = cur.take<uint8_t>(ptiles + 1);
  W.kept.held = cur.take<uint64_t>(ptiles * kBlock + 1);
  W.kept.first = cur.take<unsigned>(ptiles * kPairRows + 4);
  W.vals = cur.take<int64_t>(cond_build_rows + 2);
  return W.vals != nullptr;
}

// Pair counts of every tile of probe rows and their sum (W.pair->total), on the device.
static int count_pairs(const JoinDir& D, const void* pkeys, int pdt, const RowFilter& F, int64_t np,
                       const PairCond& C, const ProbeLayout& W, cudaStream_t s) {
  const int64_t tiles = (np + kPairRows - 1) / kPairRows;
  if (tiles > INT32_MAX) return TQPK_EUNSUPPORTED;
  auto kernel = C.P.n_insn ? k_join_pairs<true, true> : k_join_pairs<true, false>;
  kernel<<<pair_grid(tiles), kBlock, 0, s>>>(D, pkeys, pdt, F, np, aligned16(pkeys) ? 1 : 0, nullptr, nullptr, 0,
                                             W.tile_base, W.pair, W.kept, C);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

static int write_pairs(const JoinDir& D, const void* pkeys, int pdt, const RowFilter& F, int64_t np, const PairCond& C,
                       const ProbeLayout& W, int64_t* out_b, int64_t* out_p, int64_t capacity, cudaStream_t s) {
  const int64_t tiles = (np + kPairRows - 1) / kPairRows;
  auto kernel = C.P.n_insn ? k_join_pairs<false, true> : k_join_pairs<false, false>;
  timing_before(KID_JOIN_PROBE, s);
  kernel<<<pair_grid(tiles), kBlock, 0, s>>>(D, pkeys, pdt, F, np, aligned16(pkeys) ? 1 : 0, out_b, out_p, capacity,
                                             W.tile_base, W.pair, W.kept, C);
  timing_after(KID_JOIN_PROBE, s);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

}  // namespace tqpk

using namespace tqpk;

extern "C" int tqpk_join_plan_build(const void* keys, int32_t dt, const uint8_t* mask, int64_t nb, tqpk_join_plan* plan,
                                    void* scratch, tqpk_stream stream) {
  if (!plan || nb < 0 || (nb > 0 && !keys)) return TQPK_EINVAL;
  if (!is_int_dtype(dt)) return TQPK_EDTYPE;
  *plan = tqpk_join_plan{};
  int64_t mn = 0, mx = -1, rows = 0;
  const void* cols[1] = {keys};
  const int32_t dts[1] = {dt};
  int rc = key_ranges(nullptr, mask, nb, 1, cols, dts, &mn, &mx, &rows, scratch, static_cast<cudaStream_t>(stream));
  if (rc) return rc;
  plan->nb_rows = rows;
  plan->key_min = rows ? mn : 0;
  plan->key_max = rows ? mx : -1;
  const int64_t range = rows ? (mx - mn + 1) : 1;
  // direct addressing reads 4 B per slot of the key range (12 B when keys repeat; the workspace holds 12, and about
  // 40 per build row, as repeats show while the directory is filled); up to 2^24 slots
  // that is cheaper than a binary search per probe row even for a sparse build side (a filtered
  // dimension of 2 M keys joined by a 60 M-row fact table: 7.6 ms sorted, ~0.1 ms direct)
  const bool dense = rows == 0 || (range > 0 && range <= std::max<int64_t>(4 * rows, int64_t(1) << 24) &&
                                   range < (int64_t(1) << 31));
  plan->mode = dense ? TQPK_JOIN_DIRECT : TQPK_JOIN_SORTED;
  plan->slots = dense ? range : 0;
  plan->unique = 1 | (nb >= (int64_t)0xffffffffu ? kWide : 0);
  plan->ws_bytes = layout_bytes(*plan, mask ? nb : 0);
  return TQPK_OK;
}

extern "C" int tqpk_join_rows(tqpk_join_plan* plan, const void* keys, int32_t dt, const uint8_t* mask, int64_t nb,
                              void* ws, size_t ws_bytes, tqpk_stream stream) {
  if (!plan || nb < 0 || (nb > 0 && !keys)) return TQPK_EINVAL;
  if (!is_int_dtype(dt)) return TQPK_EDTYPE;
  if (!ws || ws_bytes < plan->ws_bytes) return TQPK_ENOMEM;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  BuildLayout L;
  if (!layout(*plan, ws, ws_bytes, L)) return TQPK_ENOMEM;
  plan->unique = is_wide(*plan) ? kWide : 0;
  if (plan->nb_rows == 0) return TQPK_OK;
  // Passing build rows in row order (all of them without a mask), then a stable sort by key -> CSR.
  if (mask) {
    ColSet C;
    C.n = 1;
    C.in[0] = nullptr;
    C.out[0] = L.rows;
    C.size[0] = 0;  // row ids
    int64_t* d_m = L.nu + 1;
    TQPK_CUDA(cudaMemsetAsync(L.rows, 0, plan->nb_rows * 8, s));   // row ids even if the compaction fails
    int rc = compact_launch(nullptr, mask, nb, C, d_m, L.sort_ws, L.sort_bytes, s);
    if (rc) return rc;
    k_count_status<<<1, 1, 0, s>>>(d_m, L.hdr + 1);   // a failed compaction's status joins the error word
    TQPK_CHECK_LAUNCH();
  }
  const SortKey by_key{keys, nullptr, dt, 0, 0, 0};
  int rc = sort_keys(&by_key, 1, mask ? L.rows : nullptr, plan->nb_rows, L.csr, L.sort_ws, L.sort_bytes, s);
  if (rc) return rc;
  const int direct = plan->mode == TQPK_JOIN_DIRECT;
  if (direct) TQPK_CUDA(cudaMemsetAsync(L.run, 0, 2 * plan->slots * (is_wide(*plan) ? 8 : 4), s));
  if (is_wide(*plan))
    k_join_runs<uint64_t><<<grid_for(plan->nb_rows, 8), kBlock, 0, s>>>(keys, dt, L.csr, plan->nb_rows, plan->key_min,
                                                                        direct, plan->slots, static_cast<uint64_t*>(L.run),
                                                                        L.head);
  else
    k_join_runs<unsigned><<<grid_for(plan->nb_rows, 8), kBlock, 0, s>>>(keys, dt, L.csr, plan->nb_rows, plan->key_min,
                                                                        direct, plan->slots, static_cast<unsigned*>(L.run),
                                                                        L.head);
  TQPK_CHECK_LAUNCH();
  if (!direct) {
    const int64_t tiles = (plan->nb_rows + kTile - 1) / kTile;
    TQPK_CUDA(cudaMemsetAsync(L.status, 0, (tiles + 1) * 8, s));
    TQPK_CUDA(cudaMemsetAsync(L.hdr + 2, 0, sizeof(int), s));
    k_join_unique<<<(int)tiles, kBlock, 0, s>>>(keys, dt, L.csr, L.head, plan->nb_rows, L.ukeys, L.ustart, L.nu,
                                                L.status, L.hdr + 2, L.hdr + 1);
    TQPK_CHECK_LAUNCH();
    int64_t nu = 0;
    TQPK_CUDA(cudaMemcpyAsync(&nu, L.nu, 8, cudaMemcpyDeviceToHost, s));
    TQPK_CUDA(cudaStreamSynchronize(s));
    plan->n_unique = nu;
  }
  int err = 0;
  TQPK_CUDA(cudaMemcpyAsync(&err, L.hdr + 1, sizeof(int), cudaMemcpyDeviceToHost, s));
  TQPK_CUDA(cudaStreamSynchronize(s));
  return err;
}

extern "C" int tqpk_join_directory(tqpk_join_plan* plan, const void* keys, int32_t dt, const uint8_t* mask, int64_t nb,
                                   void* ws, size_t ws_bytes, tqpk_stream stream) {
  if (!plan || nb < 0 || (nb > 0 && !keys)) return TQPK_EINVAL;
  if (!is_int_dtype(dt)) return TQPK_EDTYPE;
  if (!ws || ws_bytes < plan->ws_bytes) return TQPK_ENOMEM;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  BuildLayout L;
  if (!layout(*plan, ws, ws_bytes, L)) return TQPK_ENOMEM;
  TQPK_CUDA(cudaMemsetAsync(L.hdr, 0, 64 * sizeof(int), s));
  const int wide = plan->unique & kWide;
  if (plan->mode == TQPK_JOIN_SORTED) return tqpk_join_rows(plan, keys, dt, mask, nb, ws, ws_bytes, stream);
  plan->unique = (plan->nb_rows > 0 ? TQPK_JOIN_UNKNOWN : 1) | wide;
  TQPK_CUDA(cudaMemsetAsync(L.dir, 0xff, plan->slots * (wide ? 8 : 4), s));
  if (plan->nb_rows == 0) return TQPK_OK;
  const RowFilter F = make_filter(nullptr, mask);
  const int kvec = aligned16(keys) ? 1 : 0;
  if (wide)
    k_join_build_direct<uint64_t><<<grid_for((nb + 3) / 4, 8), kBlock, 0, s>>>(keys, dt, F, nb, plan->key_min, kvec,
                                                                              static_cast<uint64_t*>(L.dir), L.hdr);
  else
    k_join_build_direct<unsigned><<<grid_for((nb + 3) / 4, 8), kBlock, 0, s>>>(keys, dt, F, nb, plan->key_min, kvec,
                                                                              static_cast<unsigned*>(L.dir), L.hdr);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

extern "C" int tqpk_join_build(tqpk_join_plan* plan, const void* keys, int32_t dt, const uint8_t* mask, int64_t nb,
                               void* ws, size_t ws_bytes, tqpk_stream stream) {
  int rc = tqpk_join_directory(plan, keys, dt, mask, nb, ws, ws_bytes, stream);
  if (rc || uniqueness(*plan) != TQPK_JOIN_UNKNOWN) return rc;
  int dup = 0;
  TQPK_CUDA(cudaMemcpyAsync(&dup, ws, sizeof(dup), cudaMemcpyDeviceToHost, static_cast<cudaStream_t>(stream)));
  TQPK_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  if (dup) return tqpk_join_rows(plan, keys, dt, mask, nb, ws, ws_bytes, stream);
  plan->unique = (plan->unique & kWide) | 1;
  return TQPK_OK;
}

extern "C" size_t tqpk_join_probe_workspace_bytes(int64_t np) {
  const int64_t tiles = (np + kTile - 1) / kTile;
  return 2048 + 2 * align_up((size_t)(tiles + 1) * 8, 256) + align_up(((size_t)np / kPairRows + kPartSlots + 2) * 8, 256);
}

extern "C" size_t tqpk_join_pairs_workspace_bytes(const tqpk_join_plan* plan, int64_t np, int32_t with_cond) {
  if (!plan || np < 0) return 0;
  const size_t base = tqpk_join_probe_workspace_bytes(np), t = (size_t)np / kPairRows + 2;
  if (!with_cond) return base;
  return base + align_up(t, 256) + align_up(t * kBlock * 8, 256) + align_up(t * kPairRows * 4, 256) +
         align_up(((size_t)plan->nb_rows + 2) * 8, 256);
}

extern "C" int tqpk_join_probe(const tqpk_join_plan* plan, const void* build_ws, const void* pkeys, int32_t pdt,
                               const uint8_t* pmask, int64_t np, int32_t jt, int64_t* out_b, int64_t* out_p,
                               int64_t capacity, int64_t* h_count, void* pws, size_t pws_bytes, tqpk_stream stream) {
  if (!plan || !build_ws || np < 0 || (np > 0 && !pkeys) || !h_count || capacity < 0) return TQPK_EINVAL;
  if (jt < TQPK_JT_INNER || jt > TQPK_JT_OUTER) return TQPK_EINVAL;
  if ((jt == TQPK_JT_INNER || jt == TQPK_JT_OUTER) && capacity > 0 && !out_b) return TQPK_EINVAL;
  if (capacity > 0 && !out_p) return TQPK_EINVAL;
  if (!is_int_dtype(pdt)) return TQPK_EDTYPE;
  if (!pws || pws_bytes < tqpk_join_probe_workspace_bytes(np)) return TQPK_ENOMEM;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  BuildLayout L;
  if (!layout(*plan, const_cast<void*>(build_ws), plan->ws_bytes, L)) return TQPK_ENOMEM;
  const JoinDir D = make_dir(*plan, L, jt == TQPK_JT_INNER || jt == TQPK_JT_OUTER);
  ProbeLayout W;
  if (!probe_layout(np, pws, pws_bytes, W)) return TQPK_ENOMEM;
  *h_count = 0;
  if (np == 0) return TQPK_OK;
  TQPK_CUDA(cudaMemsetAsync(pws, 0, W.zeroed, s));
  const RowFilter F = make_filter(nullptr, pmask);
  int* dup = nullptr;
  int64_t* pair_total = W.totals;
  int rc;
  if (jt == TQPK_JT_INNER || jt == TQPK_JT_OUTER) {
    const bool one = D.mode == TQPK_JOIN_DIRECT && !D.csr;       // at most one build row per key
    if (uniqueness(*plan) == TQPK_JOIN_UNKNOWN) dup = L.hdr;
    if (plan->nb_rows > 0) {
      if (one) {
        rc = launch_probe<TQPK_JT_INNER>(D, pkeys, pdt, F, np, out_b, out_p, capacity, nullptr, W.totals, W.status_a,
                                         W.ctl, dup, W.ctl + 1, s);
      } else {
        pair_total = &W.pair->total;
        const PairCond none{};
        rc = count_pairs(D, pkeys, pdt, F, np, none, W, s);
        if (!rc && capacity > 0) rc = write_pairs(D, pkeys, pdt, F, np, none, W, out_b, out_p, capacity, s);
      }
      if (rc) return rc;
    }
    if (jt == TQPK_JT_OUTER) {
      rc = launch_probe<TQPK_JT_ANTI>(D, pkeys, pdt, F, np, out_b, out_p, capacity, pair_total, W.totals + 1,
                                      W.status_b, W.ctl + 2, dup, W.ctl + 1, s);
      if (rc) return rc;
    }
  } else if (jt == TQPK_JT_SEMI) {
    if (plan->nb_rows > 0) {
      rc = launch_probe<TQPK_JT_SEMI>(D, pkeys, pdt, F, np, nullptr, out_p, capacity, nullptr, W.totals, W.status_a,
                                      W.ctl, nullptr, W.ctl + 1, s);
      if (rc) return rc;
    }
  } else {
    rc = launch_probe<TQPK_JT_ANTI>(D, pkeys, pdt, F, np, nullptr, out_p, capacity, nullptr, W.totals, W.status_a,
                                    W.ctl, nullptr, W.ctl + 1, s);
    if (rc) return rc;
  }
  // one read: control words, totals and the pair total lie beside each other
  struct { int ctl[64]; int64_t totals[32]; PairCtl pair; } h;
  if (dup) TQPK_CUDA(cudaMemcpyAsync(W.ctl + 3, dup, sizeof(int), cudaMemcpyDeviceToDevice, s));
  TQPK_CUDA(cudaMemcpyAsync(&h, W.ctl, sizeof(h), cudaMemcpyDeviceToHost, s));
  TQPK_CUDA(cudaStreamSynchronize(s));
  if (h.ctl[1]) return h.ctl[1];
  if (dup && h.ctl[3]) {
    *h_count = -1;               // the build keys repeat: tqpk_join_rows first
    return TQPK_ECAPACITY;
  }
  *h_count = jt == TQPK_JT_OUTER ? h.totals[1] : pair_total == W.totals ? h.totals[0] : h.pair.total;
  return *h_count > capacity ? TQPK_ECAPACITY : TQPK_OK;
}

// The conditions of a call (null: none): numeric instructions only.
static int pair_cond(const tqpk_predicate* cond, uint32_t probe_cols, PairCond& C) {
  C = PairCond{};
  if (!cond) return TQPK_OK;
  const int rc = check_pred(cond);
  if (rc) return rc;
  for (int k = 0; k < cond->n_insn; ++k)
    if (cond->insn[k].op > TQPK_P_CMPCOL) return TQPK_EUNSUPPORTED;
  C.P = *cond;
  C.probe_cols = probe_cols;
  const tqpk_pred_insn& I = cond->insn[0];
  if (cond->n_insn == 1 && I.op == TQPK_P_CMPCOL && I.domain == TQPK_DOM_I64) {
    const int c1 = I.col, c2 = (int)I.lit_i;
    const bool p1 = (probe_cols >> c1) & 1u, p2 = (probe_cols >> c2) & 1u;
    const bool known = I.cmp >= TQPK_LT && I.cmp <= TQPK_NE;       // another operator holds for no pair
    if (known && p1 != p2 && is_int_dtype(cond->dtypes[c1]) && is_int_dtype(cond->dtypes[c2])) {
      const int bc = p1 ? c2 : c1, pc = p1 ? c1 : c2;
      static const int flipped[] = {TQPK_GT, TQPK_GE, TQPK_LT, TQPK_LE, TQPK_EQ, TQPK_NE};   // of LT, LE, GT, ...
      C.two_sided = 1;
      C.cmp = p1 ? flipped[I.cmp - TQPK_LT] : I.cmp;
      C.build_col = cond->cols[bc];
      C.build_dt = cond->dtypes[bc];
      C.probe_col = cond->cols[pc];
      C.probe_dt = cond->dtypes[pc];
    }
  }
  return TQPK_OK;
}

extern "C" int tqpk_join_count(const tqpk_join_plan* plan, const void* build_ws, const void* pkeys, int32_t pdt,
                               const uint8_t* pmask, int64_t np, const tqpk_predicate* cond, uint32_t probe_cols,
                               int64_t* h_count, void* pws, size_t pws_bytes, tqpk_stream stream) {
  if (!plan || !build_ws || np < 0 || (np > 0 && !pkeys) || !h_count) return TQPK_EINVAL;
  if (!is_int_dtype(pdt)) return TQPK_EDTYPE;
  PairCond C;
  int rc = pair_cond(cond, probe_cols, C);
  if (rc) return rc;
  if (!pws || pws_bytes < tqpk_join_pairs_workspace_bytes(plan, np, cond != nullptr)) return TQPK_ENOMEM;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  BuildLayout L;
  ProbeLayout W;
  if (!layout(*plan, const_cast<void*>(build_ws), plan->ws_bytes, L)) return TQPK_ENOMEM;
  if (!probe_layout(np, pws, pws_bytes, W, cond ? plan->nb_rows : -1)) return TQPK_ENOMEM;
  *h_count = 0;
  if (np == 0) return TQPK_OK;
  if (uniqueness(*plan) == TQPK_JOIN_UNKNOWN) {
    int dup = 0;
    TQPK_CUDA(cudaMemcpyAsync(&dup, L.hdr, sizeof(dup), cudaMemcpyDeviceToHost, s));
    TQPK_CUDA(cudaStreamSynchronize(s));
    if (dup) {
      *h_count = -1;             // the build keys repeat: tqpk_join_rows first
      return TQPK_ECAPACITY;
    }
  }
  TQPK_CUDA(cudaMemsetAsync(pws, 0, W.zeroed, s));
  const JoinDir D = make_dir(*plan, L, true);
  if (C.two_sided && D.csr && !D.wide && plan->nb_rows > 0) {
    k_pair_vals<<<grid_for(plan->nb_rows, 8), kBlock, 0, s>>>(C.build_col, C.build_dt, D.csr, plan->nb_rows, W.vals);
    TQPK_CHECK_LAUNCH();
    C.vals = W.vals;
  }
  rc = count_pairs(D, pkeys, pdt, make_filter(nullptr, pmask), np, C, W, s);
  if (rc) return rc;
  TQPK_CUDA(cudaMemcpyAsync(h_count, &W.pair->total, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  TQPK_CUDA(cudaStreamSynchronize(s));
  return TQPK_OK;
}

extern "C" int tqpk_join_write(const tqpk_join_plan* plan, const void* build_ws, const void* pkeys, int32_t pdt,
                               const uint8_t* pmask, int64_t np, const tqpk_predicate* cond, uint32_t probe_cols,
                               int64_t* out_b, int64_t* out_p, int64_t capacity, void* pws, size_t pws_bytes,
                               tqpk_stream stream) {
  if (!plan || !build_ws || np < 0 || (np > 0 && !pkeys) || capacity < 0) return TQPK_EINVAL;
  if (capacity > 0 && (!out_b || !out_p)) return TQPK_EINVAL;
  if (!is_int_dtype(pdt)) return TQPK_EDTYPE;
  PairCond C;
  const int rc = pair_cond(cond, probe_cols, C);
  if (rc) return rc;
  if (!pws || pws_bytes < tqpk_join_pairs_workspace_bytes(plan, np, cond != nullptr)) return TQPK_ENOMEM;
  if (np == 0 || capacity == 0) return TQPK_OK;
  BuildLayout L;
  ProbeLayout W;
  if (!layout(*plan, const_cast<void*>(build_ws), plan->ws_bytes, L)) return TQPK_ENOMEM;
  if (!probe_layout(np, pws, pws_bytes, W, cond ? plan->nb_rows : -1)) return TQPK_ENOMEM;
  return write_pairs(make_dir(*plan, L, true), pkeys, pdt, make_filter(nullptr, pmask), np, C, W, out_b, out_p,
                     capacity, static_cast<cudaStream_t>(stream));
}

extern "C" int tqpk_gather(int32_t ncols, const void* const* cols_in, const int32_t* dts, const int64_t* idx,
                           int64_t n_idx, int32_t null_aware, void* const* cols_out, tqpk_stream stream) {
  if (ncols < 0 || ncols > TQPK_MAX_COLS || n_idx < 0 || (n_idx > 0 && !idx)) return TQPK_EINVAL;
  if (n_idx == 0 || ncols == 0) return TQPK_OK;
  ColSet C;
  C.n = ncols;
  for (int c = 0; c < ncols; ++c) {
    const int sz = dtype_size(dts[c]);
    if (!sz) return TQPK_EDTYPE;
    if (!cols_in[c] || !cols_out[c]) return TQPK_EINVAL;
    C.in[c] = cols_in[c];
    C.out[c] = cols_out[c];
    C.size[c] = (dts[c] == TQPK_F64) ? 9 : sz;  // 9: float64 (null fill is -64.0)
  }
  k_gather<<<grid_for((n_idx + kGatherRows - 1) / kGatherRows, 8), kBlock, 0, static_cast<cudaStream_t>(stream)>>>(ncols, C, idx, n_idx, null_aware);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}
