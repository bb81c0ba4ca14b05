// filter.cu - kernel (a): predicate evaluation and stable stream compaction.
//
// Reference: operators/filter.py:14-204 evaluates a predicate tree with one
// ATen launch per tree node and stores a bool mask; IO/vortex_pipeline.py:58
// later compacts every consumer column with tensor[mask] (nonzero + gather,
// one host sync per column).  Here the whole predicate program runs in one
// pass with 128-bit loads over groups of four rows, and compaction of up to
// 16 columns is one single-pass kernel: per-thread popc of a 16-row mask, a
// block scan, and a decoupled look-back across 4096-row tiles so the output
// keeps row order (what tensor[mask] gives).
#include <stdio.h>

#include <algorithm>

#include <type_traits>

#include "common.cuh"

namespace tqpk {

thread_local int64_t g_launches = 0;

namespace {
struct Timing {
  int kid = KID_NONE;
  int n = 0;
  cudaEvent_t ev[2 * 4096];
  bool created = false;
};
Timing g_timing;
}  // namespace

void timing_before(int kid, cudaStream_t s) {
  if (g_timing.kid != kid || g_timing.n >= 4096) return;
  cudaEventRecord(g_timing.ev[2 * g_timing.n], s);
}
void timing_after(int kid, cudaStream_t s) {
  if (g_timing.kid != kid || g_timing.n >= 4096) return;
  cudaEventRecord(g_timing.ev[2 * g_timing.n + 1], s);
  ++g_timing.n;
}

int num_sms() {
  static int cached[64] = {0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 152;
  if (!cached[dev]) {
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || v <= 0) v = 152;
    cached[dev] = v;
  }
  return cached[dev];
}

// 4 Q rows per thread, four at a time 1024 rows apart (coalesced): a thread's loads of a column are all in
// flight, and type, operator and program are decided once for them.
template <int Q>
__global__ void __launch_bounds__(kBlock, Q == 1 ? 6 : 3) k_filter_mask(const __grid_constant__ tqpk_predicate P,
                                                                        int64_t n, uint8_t* __restrict__ mask,
                                                                        unsigned long long* count, int vec,
                                                                        int mask_vec) {
  unsigned local = 0;
  for (int64_t t0 = blockIdx.x * (int64_t)(4 * Q * kBlock); t0 < n; t0 += (int64_t)gridDim.x * (4 * Q * kBlock)) {
    int64_t r0[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) r0[q] = t0 + (q * kBlock + threadIdx.x) * 4;
    const uint32_t bits = eval_pred_rows<Q>(P, r0, n, vec);
    local += __popc(bits);
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const uint32_t b = (bits >> (4 * q)) & 0xfu;
      if (mask_vec && r0[q] + 4 <= n) {
        const uint32_t w = (b & 1u) | ((b & 2u) << 7) | ((b & 4u) << 14) | ((b & 8u) << 21);
        *reinterpret_cast<uint32_t*>(mask + r0[q]) = w;
      } else {
        for (int j = 0; j < 4 && r0[q] + j < n; ++j) mask[r0[q] + j] = (b >> j) & 1u;
      }
    }
  }
  if (count) {
    local = __reduce_add_sync(0xffffffffu, local);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(count, (unsigned long long)local);
  }
}

// Programs that search text (Contains, LIKE): the block takes 1024 rows through the program together, and a
// search stages their bytes 256 rows at a time in shared memory (coalesced), where each thread searches one row;
// the verdicts go back to the rows' owners as bits.  Searched in place, every byte of a warp's rows was a
// scattered load.  Equality and prefixes stop at their first different byte and stay in place.  Rows of up to
// kStagedRow bytes, which 48 KB hold beside the verdicts.  1.5 M rows, us in place / staged: a search without a
// hit on 25 bytes 44 / 25, 150 bytes 444 / 111, 188 bytes 473 / 174; one that hits early in every row, 25 bytes
// 37 / 30, 150 bytes 87 / 89, 188 bytes 83 / 120 (a predicate that keeps everything, so the line is not drawn by
// it).  Seven substrings in an IN list on 25 bytes 33 / 63, a prefix on 150 bytes 36 / 43.
// Rows of 64 or 128 bytes are staged a word apart, or the threads' bytes would meet in two banks or one (128 bytes,
// without a hit 784 us and in place 787, a word apart 120; 64 bytes 188, 393 and 65).  Multiples of 32 gain less
// (160 bytes 240 and 152) and lose as much where a hit comes early (95 and 116): staged by words, not 16 bytes.
constexpr int kStagedRow = 188;
__host__ __device__ __forceinline__ int64_t staged_pitch(int64_t stride) { return stride % 64 ? stride : stride + 4; }

__global__ void __launch_bounds__(kBlock) k_filter_text(const __grid_constant__ tqpk_predicate P, int64_t n,
                                                        uint8_t* __restrict__ mask, unsigned long long* count, int vec,
                                                        int mask_vec) {
  extern __shared__ __align__(16) int8_t stage[];
  __shared__ unsigned s_bits[4 * kBlock / 32];
  unsigned local = 0;
  for (int64_t t0 = blockIdx.x * (int64_t)(4 * kBlock); t0 < n; t0 += (int64_t)gridDim.x * (4 * kBlock)) {
    const int64_t r0[1] = {t0 + 4 * threadIdx.x};
    const uint32_t b = eval_pred_with<1>(P, r0, n, vec, [&](const tqpk_pred_insn& I) {
      if (I.op < TQPK_P_CONTAINS) return str_leaf4(P, I, r0[0], n);
      const int64_t stride = str_stride(P, I.col);
      const int8_t* base = static_cast<const int8_t*>(P.cols[I.col]);
      const bool apart = stride % 64 == 0 && P.widths[I.col] == stride && (reinterpret_cast<uintptr_t>(base) & 3u) == 0;
      const int pitch = (int)(apart ? staged_pitch(stride) : stride);
#pragma unroll 1
      for (int j = 0; j < 4; ++j) {
        const int64_t q0 = t0 + j * kBlock;
        const int rows = (int)(n - q0 < kBlock ? (n - q0 < 0 ? 0 : n - q0) : kBlock);
        __syncthreads();
        if (rows > 0) {                      // a substring's last row ends before its stride does
          const int bytes = (int)((rows - 1) * stride) + P.widths[I.col];
          const int8_t* s = base + q0 * stride;
          if (apart) {
            const unsigned words = (unsigned)stride / 4;           // of a row; one more between two
            for (unsigned i = threadIdx.x; i < words * rows; i += kBlock)
              reinterpret_cast<unsigned*>(stage)[i + i / words] = reinterpret_cast<const unsigned*>(s)[i];
          } else {
            const int whole = (reinterpret_cast<uintptr_t>(s) & 15u) == 0 ? bytes / 16 : 0;
            for (int i = threadIdx.x; i < whole; i += kBlock)
              reinterpret_cast<uint4*>(stage)[i] = reinterpret_cast<const uint4*>(s)[i];
            for (int i = whole * 16 + threadIdx.x; i < bytes; i += kBlock) stage[i] = s[i];
          }
        }
        __syncthreads();
        const bool ok = (int)threadIdx.x < rows && str_leaf(P, I, stage + (int)threadIdx.x * pitch);
        const unsigned m = __ballot_sync(0xffffffffu, ok);
        if ((threadIdx.x & 31) == 0) s_bits[(j * kBlock + threadIdx.x) >> 5] = m;
      }
      __syncthreads();
      return (s_bits[threadIdx.x >> 3] >> (4 * (threadIdx.x & 7))) & 0xfu;
    });
    local += __popc(b);
    if (mask_vec && r0[0] + 4 <= n) {
      *reinterpret_cast<uint32_t*>(mask + r0[0]) = (b & 1u) | ((b & 2u) << 7) | ((b & 4u) << 14) | ((b & 8u) << 21);
    } else {
      for (int j = 0; j < 4 && r0[0] + j < n; ++j) mask[r0[0] + j] = (b >> j) & 1u;
    }
  }
  if (count) {
    local = __reduce_add_sync(0xffffffffu, local);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(count, (unsigned long long)local);
  }
}

// Sixteen rows a thread from here on (four CTAs of 4096 rows per SM), four below, where more warps matter
// more than fewer instructions.
constexpr int64_t kManyRows = int64_t(5) << 19;

// Comparisons of columns of different types keep four rows a thread: sixteen of each do not fit the registers
// in the wider type, and a thread that takes them four at a time has too few loads in flight (6 M rows, int32
// against int64 29 us, uint8 against int64 25; 19 and 18 with four rows).
static bool many_rows(const tqpk_predicate* pred, int64_t n) {
  if (n < kManyRows) return false;
  for (int k = 0; pred && k < pred->n_insn; ++k) {
    const tqpk_pred_insn& I = pred->insn[k];
    if (I.op == TQPK_P_CMPCOL && pred->dtypes[I.col] != pred->dtypes[(int)I.lit_i]) return false;
  }
  return true;
}

// Control block of one compaction (zeroed before the launch).
struct CompactCtl {
  int tile_ctr;      // next tile to take
  int err;           // first error status of any CTA
  int finished;      // CTAs done
  int pad;
  int64_t kept;      // rows kept, written by the CTA of the last tile
};
constexpr size_t kCompactCtlBytes = 256;   // one WsCursor piece
static_assert(sizeof(CompactCtl) <= kCompactCtlBytes, "control block");

// Test hook (tqpk_debug_compact_wait): the poll limit of the look-back, and a tile whose CTA
// publishes nothing, so that its successors' waits run out.  Defaults: kSpinLimit, none.
static int g_dbg_spin_limit = kSpinLimit;
static int64_t g_dbg_stall_tile = -1;

// One 4096-row tile of k_compact: the tile's mask bits, its block scan, the look-back for its
// output offset, then the kept rows of every column in row order.
__device__ __forceinline__ void compact_tile(const tqpk_predicate& P, const RowFilter& F, int64_t n, const ColSet& C,
                                             uint64_t* status, CompactCtl* ctl, int spin_limit, int64_t tile,
                                             uint64_t& s_excl, int* sw) {
  const int64_t r0 = tile * kTile + threadIdx.x * kItems;
  uint32_t bits = 0;
#pragma unroll
  for (int q = 0; q < kItems / 4; ++q) bits |= filter4(F, P, r0 + 4 * q, n) << (4 * q);
  int total;
  const int excl = block_excl_scan<kBlock, int>(__popc(bits), total, sw);
  if (threadIdx.x < 32) {
    uint64_t e = lookback_warp(status, tile, (uint64_t)total, &ctl->err, spin_limit);
    if (threadIdx.x == 0) s_excl = e;
  }
  __syncthreads();
  const int64_t base = (int64_t)s_excl + excl;
  for (int c = 0; c < C.n; ++c) {
    int64_t pos = base;
    uint32_t b = bits;
    switch (C.size[c]) {
      case 1: {
        const uint8_t* in = static_cast<const uint8_t*>(C.in[c]);
        uint8_t* out = static_cast<uint8_t*>(C.out[c]);
        while (b) { int j = __ffs(b) - 1; b &= b - 1; out[pos++] = in[r0 + j]; }
        break;
      }
      case 4: {
        const uint32_t* in = static_cast<const uint32_t*>(C.in[c]);
        uint32_t* out = static_cast<uint32_t*>(C.out[c]);
        while (b) { int j = __ffs(b) - 1; b &= b - 1; out[pos++] = in[r0 + j]; }
        break;
      }
      case 8: {
        const uint64_t* in = static_cast<const uint64_t*>(C.in[c]);
        uint64_t* out = static_cast<uint64_t*>(C.out[c]);
        while (b) { int j = __ffs(b) - 1; b &= b - 1; out[pos++] = in[r0 + j]; }
        break;
      }
      default: {  // size 0: the row index itself (int64), for row-id compaction
        int64_t* out = static_cast<int64_t*>(C.out[c]);
        while (b) { int j = __ffs(b) - 1; b &= b - 1; out[pos++] = r0 + j; }
        break;
      }
    }
  }
  if (tile == (int64_t)gridDim.x - 1 && threadIdx.x == 0) ctl->kept = (int64_t)(s_excl + total);
}

__global__ void __launch_bounds__(kBlock) k_compact(const __grid_constant__ tqpk_predicate P, RowFilter F, int64_t n,
                                                    const __grid_constant__ ColSet C, int64_t* count,
                                                    uint64_t* status, CompactCtl* ctl, int spin_limit,
                                                    int64_t stall_tile) {
  __shared__ int s_tile;
  __shared__ uint64_t s_excl;
  __shared__ int sw[kBlock / 32 + 1];
  if (threadIdx.x == 0) s_tile = atomicAdd(&ctl->tile_ctr, 1);
  __syncthreads();
  const int64_t tile = s_tile;
  if (tile != stall_tile) compact_tile(P, F, n, C, status, ctl, spin_limit, tile, s_excl, sw);
  // The last CTA to finish writes the result: the kept-row count, or the error status (negative)
  // when any look-back gave up.  Every CTA's error write precedes its fence and its increment.
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&ctl->finished, 1) == (int)gridDim.x - 1) {
      __threadfence();
      const int e = *reinterpret_cast<volatile int*>(&ctl->err);
      const int64_t kept = *reinterpret_cast<volatile int64_t*>(&ctl->kept);
      *count = e ? (int64_t)e : kept;
    }
  }
}

// Min/max of up to four integer key columns over the rows passing a filter,
// plus the passing-row count.  out = [min0..min3, max0..max3].
// Range record blockIdx.x of kRangeWords words.
constexpr int kRangeWords = 16;
__global__ void k_init_range(int64_t* out) {
  out += blockIdx.x * kRangeWords;
  if (threadIdx.x < TQPK_MAX_KEYS) {
    out[threadIdx.x] = INT64_MAX;
    out[TQPK_MAX_KEYS + threadIdx.x] = INT64_MIN;
  }
  if (threadIdx.x == 0) out[2 * TQPK_MAX_KEYS] = 0;
}

// Min and max of 4 Q rows' keys where their bit is set, in the column's own width.
template <class T, int Q>
__device__ __forceinline__ void range_rows(const void* col, const int64_t (&r0)[Q], int64_t n, bool vec, uint32_t bits,
                                           int64_t& mn, int64_t& mx) {
  T x[4 * Q];
  load_rows<T, Q>(col, r0, n, vec, x);
  using W = std::conditional_t<sizeof(T) == 8, int64_t, int>;
  constexpr W kMost = sizeof(T) == 8 ? (W)INT64_MAX : (W)INT32_MAX, kLeast = -kMost - 1;
  W lo = kMost, hi = kLeast;
#pragma unroll
  for (int i = 0; i < 4 * Q; ++i) {
    lo = min(lo, (bits >> i) & 1u ? (W)x[i] : kMost);
    hi = max(hi, (bits >> i) & 1u ? (W)x[i] : kLeast);
  }
  mn = min(mn, (int64_t)lo);
  mx = max(mx, (int64_t)hi);
}

// 4 Q rows per thread and step, each column's type decided once for them, and one update per CTA: four rows
// at a time spent ~260 instructions on two one-byte keys, and an update per warp (9.7 K on the same words)
// queued.
template <int Q, bool PRED>
__global__ void __launch_bounds__(kBlock) k_key_range(const __grid_constant__ tqpk_predicate P, RowFilter F, int64_t n,
                                                      KeySet K, int64_t* out, unsigned long long* count, int vec) {
  __shared__ int64_t s_mn[TQPK_MAX_KEYS][kBlock / 32], s_mx[TQPK_MAX_KEYS][kBlock / 32];
  __shared__ unsigned s_cnt[kBlock / 32];
  int64_t mn[TQPK_MAX_KEYS], mx[TQPK_MAX_KEYS];
#pragma unroll
  for (int k = 0; k < TQPK_MAX_KEYS; ++k) { mn[k] = INT64_MAX; mx[k] = INT64_MIN; }
  unsigned cnt = 0;
  for (int64_t t0 = blockIdx.x * (int64_t)(4 * Q * kBlock); t0 < n; t0 += (int64_t)gridDim.x * (4 * Q * kBlock)) {
    int64_t r0[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) r0[q] = t0 + (q * kBlock + threadIdx.x) * 4;
    const uint32_t bits = filter_rows<Q, PRED>(F, P, r0, n);
    if (!bits) continue;
    cnt += __popc(bits);
#pragma unroll
    for (int k = 0; k < TQPK_MAX_KEYS; ++k) {
      if (k >= K.n) break;
      switch (K.dt[k]) {
        case TQPK_I64: range_rows<int64_t, Q>(K.col[k], r0, n, vec, bits, mn[k], mx[k]); break;
        case TQPK_I32: range_rows<int32_t, Q>(K.col[k], r0, n, vec, bits, mn[k], mx[k]); break;
        case TQPK_I8: range_rows<int8_t, Q>(K.col[k], r0, n, vec, bits, mn[k], mx[k]); break;
        default: range_rows<uint8_t, Q>(K.col[k], r0, n, vec, bits, mn[k], mx[k]); break;
      }
    }
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int k = 0; k < TQPK_MAX_KEYS; ++k) {
    if (k >= K.n) break;
    int64_t a = mn[k], z = mx[k];
#pragma unroll
    for (int o = 16; o; o >>= 1) {
      a = min(a, (int64_t)__shfl_xor_sync(0xffffffffu, (long long)a, o));
      z = max(z, (int64_t)__shfl_xor_sync(0xffffffffu, (long long)z, o));
    }
    if (lane == 0) {
      s_mn[k][warp] = a;
      s_mx[k][warp] = z;
    }
  }
  cnt = __reduce_add_sync(0xffffffffu, cnt);
  if (lane == 0) s_cnt[warp] = cnt;
  __syncthreads();
  if (warp) return;
  for (int k = 0; k < K.n; ++k) {
    int64_t a = lane < kBlock / 32 ? s_mn[k][lane] : INT64_MAX, z = lane < kBlock / 32 ? s_mx[k][lane] : INT64_MIN;
#pragma unroll
    for (int o = 4; o; o >>= 1) {
      a = min(a, (int64_t)__shfl_xor_sync(0xffffffffu, (long long)a, o));
      z = max(z, (int64_t)__shfl_xor_sync(0xffffffffu, (long long)z, o));
    }
    if (lane == 0 && a <= z) {
      atomicMin(reinterpret_cast<long long*>(&out[k]), (long long)a);
      atomicMax(reinterpret_cast<long long*>(&out[TQPK_MAX_KEYS + k]), (long long)z);
    }
  }
  unsigned c = lane < kBlock / 32 ? s_cnt[lane] : 0;
  c = __reduce_add_sync(0xffffffffu, c);
  if (lane == 0 && c) atomicAdd(count, (unsigned long long)c);
}

// ---------------------------------------------------------------- host side
bool pred_vec_ok(const tqpk_predicate* p) {
  if (!p) return true;
  for (int c = 0; c < p->n_cols; ++c)
    if (!aligned16(p->cols[c])) return false;
  return true;
}

int check_pred(const tqpk_predicate* p) {
  if (!p) return TQPK_OK;
  if (p->n_insn < 0 || p->n_insn > TQPK_MAX_PRED || p->n_cols < 0 || p->n_cols > TQPK_MAX_COLS) return TQPK_EINVAL;
  int depth = 0;
  for (int k = 0; k < p->n_insn; ++k) {
    const tqpk_pred_insn& I = p->insn[k];
    switch (I.op) {
      case TQPK_P_CMP:
      case TQPK_P_MASK:
        if (I.col < 0 || I.col >= p->n_cols || !p->cols[I.col]) return TQPK_EINVAL;
        if (!dtype_size(p->dtypes[I.col])) return TQPK_EDTYPE;
        if (I.op == TQPK_P_CMP && I.domain == TQPK_DOM_F64 && p->dtypes[I.col] != TQPK_F64 &&
            I.cmp == TQPK_ISCLOSE)
          return TQPK_EINVAL;
        if (I.op == TQPK_P_MASK && dtype_size(p->dtypes[I.col]) != 1) return TQPK_EDTYPE;
        ++depth;
        break;
      case TQPK_P_CMPCOL:
        if (I.col < 0 || I.col >= p->n_cols || !p->cols[I.col] || I.lit_i < 0 || I.lit_i >= p->n_cols ||
            !p->cols[I.lit_i] || I.cmp == TQPK_ISCLOSE)
          return TQPK_EINVAL;
        if (!dtype_size(p->dtypes[I.col]) || !dtype_size(p->dtypes[I.lit_i])) return TQPK_EDTYPE;
        ++depth;
        break;
      case TQPK_P_STRCMP:
      case TQPK_P_PREFIX:
      case TQPK_P_CONTAINS:
      case TQPK_P_LIKE2: {
        if (I.col < 0 || I.col >= p->n_cols || !p->cols[I.col]) return TQPK_EINVAL;
        if (dtype_size(p->dtypes[I.col]) != 1) return TQPK_EDTYPE;
        const int64_t w = p->widths[I.col];
        const uint64_t L = (uint64_t)I.lit_i;
        if (w <= 0 || p->strides[I.col] < 0 || (p->strides[I.col] > 0 && p->strides[I.col] < w)) return TQPK_EINVAL;
        bool ok;
        if (I.op == TQPK_P_STRCMP) {
          ok = (L & 0xffffffffu) + w <= TQPK_MAX_STRPOOL && I.cmp >= TQPK_LT && I.cmp <= TQPK_NE;
        } else if (I.op == TQPK_P_LIKE2) {
          ok = (L & 0xffff) + ((L >> 16) & 0xffff) <= TQPK_MAX_STRPOOL &&
               ((L >> 32) & 0xffff) + (L >> 48) <= TQPK_MAX_STRPOOL;
        } else {
          ok = (L & 0xffffffffu) + (L >> 32) <= TQPK_MAX_STRPOOL && (I.op != TQPK_P_PREFIX || (int64_t)(L >> 32) <= w);
        }
        if (!ok) return TQPK_EINVAL;
        ++depth;
        break;
      }
      case TQPK_P_TRUE:
      case TQPK_P_FALSE: ++depth; break;
      case TQPK_P_AND:
      case TQPK_P_OR:
        if (depth < 2) return TQPK_EINVAL;
        --depth;
        break;
      case TQPK_P_NOT:
        if (depth < 1) return TQPK_EINVAL;
        break;
      default: return TQPK_EINVAL;
    }
  }
  return (p->n_insn == 0 || depth == 1) ? TQPK_OK : TQPK_EINVAL;
}

bool spec_cols_vec(const tqpk_groupby_spec* S) {
  if (!S) return true;
  for (int c = 0; c < S->n_cols; ++c)
    if (!aligned16(S->cols[c])) return false;
  return true;
}

RowFilter make_filter(const tqpk_predicate* pred, const uint8_t* mask) {
  RowFilter F;
  F.mask = mask;
  F.use_pred = (pred != nullptr && mask == nullptr) ? 1 : 0;
  F.mask_vec = mask ? ((reinterpret_cast<uintptr_t>(mask) & 3u) == 0) : 0;
  F.pred_vec = pred_vec_ok(pred) ? 1 : 0;
  return F;
}

const tqpk_predicate* pred_or_empty(const tqpk_predicate* p) {
  static const tqpk_predicate empty = {};
  return p ? p : &empty;
}

int grid_for(int64_t work_items, int per_sm) {
  int64_t g = (work_items + kBlock - 1) / kBlock;
  int64_t cap = (int64_t)num_sms() * per_sm;
  if (g > cap) g = cap;
  return (int)(g < 1 ? 1 : g);
}

// The range record of the key columns K over the filtered rows, on the device (record initialised before).
static int launch_range(const tqpk_predicate* pred, const uint8_t* mask, int64_t n, const KeySet& K, bool vec,
                        int64_t* out, cudaStream_t s) {
  const RowFilter F = make_filter(pred, mask);
  const bool many = many_rows(F.use_pred ? pred : nullptr, n);
  auto kernel = F.use_pred ? (many ? k_key_range<4, true> : k_key_range<1, true>)
                           : (many ? k_key_range<4, false> : k_key_range<1, false>);
  kernel<<<grid_for((n + 3) / 4 / (many ? 4 : 1), 8), kBlock, 0, s>>>(
      *pred_or_empty(pred), F, n, K, out, reinterpret_cast<unsigned long long*>(out + 2 * TQPK_MAX_KEYS), vec ? 1 : 0);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

// Shared by the group-by and join planners: min/max of key columns over the
// filtered rows.  scratch holds 8 int64 + 1 counter; synchronises.
int key_ranges(const tqpk_predicate* pred, const uint8_t* mask, int64_t n, int nk, const void* const* cols,
               const int32_t* dts, int64_t* h_min, int64_t* h_max, int64_t* h_count, void* scratch,
               cudaStream_t s) {
  if (nk < 0 || nk > TQPK_MAX_KEYS || !scratch) return TQPK_EINVAL;
  if (n == 0) {  // no rows: empty ranges (min > max); empty tensors may carry null pointers
    for (int k = 0; k < nk; ++k) {
      h_min[k] = 0;
      h_max[k] = -1;
    }
    *h_count = 0;
    return TQPK_OK;
  }
  KeySet K;
  K.n = nk;
  bool vec = true;
  for (int k = 0; k < nk; ++k) {
    if (!cols[k] || !is_int_dtype(dts[k])) return cols[k] ? TQPK_EDTYPE : TQPK_EINVAL;
    K.col[k] = cols[k];
    K.dt[k] = dts[k];
    vec = vec && aligned16(cols[k]);
  }
  int64_t* out = static_cast<int64_t*>(scratch);
  k_init_range<<<1, 32, 0, s>>>(out);
  TQPK_CHECK_LAUNCH();
  const int rc = launch_range(pred, mask, n, K, vec, out, s);
  if (rc) return rc;
  int64_t host[2 * TQPK_MAX_KEYS + 1];
  TQPK_CUDA(cudaMemcpyAsync(host, out, sizeof(host), cudaMemcpyDeviceToHost, s));
  TQPK_CUDA(cudaStreamSynchronize(s));
  for (int k = 0; k < nk; ++k) {
    h_min[k] = host[k];
    h_max[k] = host[TQPK_MAX_KEYS + k];
  }
  *h_count = host[2 * TQPK_MAX_KEYS];
  return TQPK_OK;
}

// Stable compaction used inside the library (groups, join rows).
// Workspace of one compaction: the control block, then one status word per tile (both
// 256-byte aligned pieces, as compact_launch takes them).
size_t compact_status_bytes(int64_t n) { return kCompactCtlBytes + align_up(((n + kTile - 1) / kTile) * 8, 256); }

int compact_launch(const tqpk_predicate* pred, const uint8_t* mask, int64_t n, const ColSet& C, int64_t* d_count,
                   void* ws, size_t ws_bytes, cudaStream_t s) {
  const int64_t tiles = (n + kTile - 1) / kTile;
  WsCursor cur(ws, ws_bytes);
  CompactCtl* ctl = reinterpret_cast<CompactCtl*>(cur.take<unsigned char>(kCompactCtlBytes));
  uint64_t* status = cur.take<uint64_t>(tiles > 0 ? tiles : 1);
  if (!ctl || !status) return TQPK_ENOMEM;
  TQPK_CUDA(cudaMemsetAsync(ws, 0, cur.off, s));
  if (tiles == 0) {
    TQPK_CUDA(cudaMemsetAsync(d_count, 0, sizeof(int64_t), s));
    return TQPK_OK;
  }
  if (tiles > INT32_MAX) return TQPK_EUNSUPPORTED;
  RowFilter F = make_filter(pred, mask);
  k_compact<<<(int)tiles, kBlock, 0, s>>>(*pred_or_empty(pred), F, n, C, d_count, status, ctl, g_dbg_spin_limit,
                                          g_dbg_stall_tile);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

}  // namespace tqpk

using namespace tqpk;

extern "C" int tqpk_version(void) { return 1; }

extern "C" const char* tqpk_status_string(int status) {
  switch (status) {
    case TQPK_OK: return "ok";
    case TQPK_EINVAL: return "invalid argument";
    case TQPK_ENOMEM: return "workspace too small";
    case TQPK_ETIMEOUT: return "bounded device wait expired";
    case TQPK_EDTYPE: return "unsupported dtype";
    case TQPK_ECUDA: return "CUDA error";
    case TQPK_ECAPACITY: return "output capacity too small";
    case TQPK_EUNSUPPORTED: return "unsupported shape";
  }
  return "unknown status";
}

extern "C" int64_t tqpk_launch_count(void) { return g_launches; }

extern "C" int tqpk_timing_begin(int32_t kernel_id) {
  if (!g_timing.created) {
    for (int i = 0; i < 2 * 4096; ++i) TQPK_CUDA(cudaEventCreate(&g_timing.ev[i]));
    g_timing.created = true;
  }
  g_timing.kid = kernel_id;
  g_timing.n = 0;
  return TQPK_OK;
}

extern "C" int tqpk_timing_end(double* h_total_ms, int32_t* h_launches) {
  if (!h_total_ms || !h_launches) return TQPK_EINVAL;
  double total = 0.0;
  for (int i = 0; i < g_timing.n; ++i) {
    TQPK_CUDA(cudaEventSynchronize(g_timing.ev[2 * i + 1]));
    float ms = 0.f;
    TQPK_CUDA(cudaEventElapsedTime(&ms, g_timing.ev[2 * i], g_timing.ev[2 * i + 1]));
    total += ms;
  }
  *h_total_ms = total;
  *h_launches = g_timing.n;
  g_timing.kid = KID_NONE;
  g_timing.n = 0;
  return TQPK_OK;
}

extern "C" int tqpk_abi_sizes(int64_t* out, int n) {
  const int64_t sizes[] = {sizeof(tqpk_pred_insn), sizeof(tqpk_predicate), sizeof(tqpk_expr_insn), sizeof(tqpk_acc),
                           sizeof(tqpk_groupby_spec), sizeof(tqpk_gb_plan), sizeof(tqpk_join_plan)};
  const int k = (int)(sizeof(sizes) / sizeof(sizes[0]));
  for (int i = 0; i < n && i < k; ++i) out[i] = sizes[i];
  return k;
}

extern "C" int tqpk_filter_mask(const tqpk_predicate* h_pred, int64_t n, uint8_t* d_mask,
                                unsigned long long* d_count, tqpk_stream stream) {
  if (!h_pred || n < 0 || (n > 0 && !d_mask)) return TQPK_EINVAL;
  int rc = check_pred(h_pred);
  if (rc) return rc;
  if (n == 0) return TQPK_OK;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int mask_vec = (reinterpret_cast<uintptr_t>(d_mask) & 3u) == 0;
  timing_before(KID_FILTER_MASK, s);
  bool text = false;
  int64_t searched = 0;          // the widest text row that is searched, as staged
  for (int k = 0; k < h_pred->n_insn; ++k) {
    const tqpk_pred_insn& I = h_pred->insn[k];
    text = text || I.op >= TQPK_P_STRCMP;
    if (I.op >= TQPK_P_CONTAINS) searched = std::max(searched, staged_pitch(str_stride(*h_pred, I.col)));
  }
  if (searched > 0 && searched <= kStagedRow) {
    k_filter_text<<<grid_for((n + 3) / 4, 8), kBlock, (size_t)searched * kBlock, s>>>(
        *h_pred, n, d_mask, d_count, pred_vec_ok(h_pred) ? 1 : 0, mask_vec);
    timing_after(KID_FILTER_MASK, s);
    TQPK_CHECK_LAUNCH();
    return TQPK_OK;
  }
  // other programs with text stay four rows a thread: its bytes keep every warp busy
  const bool many = !text && many_rows(h_pred, n);
  auto kernel = many ? k_filter_mask<4> : k_filter_mask<1>;
  kernel<<<grid_for((n + 3) / 4 / (many ? 4 : 1), 8), kBlock, 0, s>>>(*h_pred, n, d_mask, d_count,
                                                                      pred_vec_ok(h_pred) ? 1 : 0, mask_vec);
  timing_after(KID_FILTER_MASK, s);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}

// Test hook: the poll limit of the compaction's look-back, and a tile whose CTA publishes nothing
// (its successors' bounded waits then run out and the call's count becomes TQPK_ETIMEOUT).
// (kSpinLimit or less, -1) restores the defaults.  Not thread-safe; for tests only.
extern "C" int tqpk_debug_compact_wait(int32_t spin_limit, int64_t stall_tile) {
  if (spin_limit < 0 || spin_limit > kSpinLimit || stall_tile < -1) return TQPK_EINVAL;
  g_dbg_spin_limit = spin_limit;
  g_dbg_stall_tile = stall_tile;
  return TQPK_OK;
}

// [min, max] of one integer column over all n rows (one host synchronisation); d_scratch holds
// 256 bytes.  An empty column gives min > max.
extern "C" int tqpk_key_range(const void* d_col, int32_t dtype, int64_t n, void* d_scratch, int64_t* h_min,
                              int64_t* h_max, tqpk_stream stream) {
  if (n < 0 || !d_scratch || !h_min || !h_max || (n > 0 && !d_col)) return TQPK_EINVAL;
  int64_t cnt = 0;
  const void* cols[1] = {d_col};
  const int32_t dts[1] = {dtype};
  return key_ranges(nullptr, nullptr, n, 1, cols, dts, h_min, h_max, &cnt, d_scratch,
                    static_cast<cudaStream_t>(stream));
}

// tqpk_key_range of several columns, each over its own rows, with one host synchronisation; d_scratch holds
// 128 bytes per column.
extern "C" int tqpk_key_ranges(int32_t n_cols, const void* const* d_cols, const int32_t* dtypes, const int64_t* rows,
                               void* d_scratch, int64_t* h_min, int64_t* h_max, tqpk_stream stream) {
  if (n_cols < 0 || n_cols > TQPK_MAX_COLS || !d_cols || !dtypes || !rows || !d_scratch || !h_min || !h_max)
    return TQPK_EINVAL;
  if (n_cols == 0) return TQPK_OK;
  for (int c = 0; c < n_cols; ++c) {
    if (rows[c] < 0 || (rows[c] > 0 && !d_cols[c])) return TQPK_EINVAL;
    if (!is_int_dtype(dtypes[c])) return TQPK_EDTYPE;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  int64_t* out = static_cast<int64_t*>(d_scratch);
  k_init_range<<<n_cols, 32, 0, s>>>(out);
  TQPK_CHECK_LAUNCH();
  for (int c = 0; c < n_cols; ++c) {
    if (rows[c] == 0) continue;
    KeySet K{};
    K.n = 1;
    K.col[0] = d_cols[c];
    K.dt[0] = dtypes[c];
    const int rc = launch_range(nullptr, nullptr, rows[c], K, aligned16(d_cols[c]), out + c * kRangeWords, s);
    if (rc) return rc;
  }
  int64_t host[TQPK_MAX_COLS * kRangeWords];
  TQPK_CUDA(cudaMemcpyAsync(host, out, (size_t)n_cols * kRangeWords * 8, cudaMemcpyDeviceToHost, s));
  TQPK_CUDA(cudaStreamSynchronize(s));
  for (int c = 0; c < n_cols; ++c) {
    h_min[c] = rows[c] ? host[c * kRangeWords] : 0;
    h_max[c] = rows[c] ? host[c * kRangeWords + TQPK_MAX_KEYS] : -1;
  }
  return TQPK_OK;
}

extern "C" size_t tqpk_compact_workspace_bytes(int64_t n) { return compact_status_bytes(n < 0 ? 0 : n); }

extern "C" int tqpk_compact(const tqpk_predicate* h_pred, const uint8_t* d_mask, int64_t n, int32_t ncols,
                            const void* const* h_cols_in, const int32_t* h_dtypes, void* const* h_cols_out,
                            int64_t* d_count, void* d_ws, size_t ws_bytes, tqpk_stream stream) {
  if (n < 0 || ncols < 0 || ncols > TQPK_MAX_COLS || !d_count || !d_ws) return TQPK_EINVAL;
  if (n == 0) {  // nothing to keep; empty tensors may carry null pointers
    TQPK_CUDA(cudaMemsetAsync(d_count, 0, sizeof(int64_t), static_cast<cudaStream_t>(stream)));
    return TQPK_OK;
  }
  if (!h_pred && !d_mask) return TQPK_EINVAL;
  int rc = check_pred(h_pred);
  if (rc) return rc;
  ColSet C;
  C.n = ncols;
  for (int c = 0; c < ncols; ++c) {
    const int sz = dtype_size(h_dtypes[c]);
    if (!sz && h_dtypes[c] != TQPK_ROWID) return TQPK_EDTYPE;
    if (n > 0 && ((sz && !h_cols_in[c]) || !h_cols_out[c])) return TQPK_EINVAL;
    C.in[c] = h_cols_in[c];
    C.out[c] = h_cols_out[c];
    C.size[c] = sz;
  }
  return compact_launch(d_mask ? nullptr : h_pred, d_mask, n, C, d_count, d_ws, ws_bytes,
                        static_cast<cudaStream_t>(stream));
}

namespace tqpk {
__global__ void k_mark_rows(const int64_t* __restrict__ idx, int64_t n_idx, uint8_t* __restrict__ flags, int64_t n) {
  for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < n_idx; j += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = idx[j];
    if (i >= 0 && i < n) flags[i] = 1;
  }
}
}  // namespace tqpk

// flags[idx[j]] = 1 for every j (indices outside [0, n) are skipped): the rows a set of
// join pairs touches, for the semi / anti / outer forms of a join with extra conditions.
extern "C" int tqpk_mark_rows(const int64_t* d_idx, int64_t n_idx, uint8_t* d_flags, int64_t n, tqpk_stream stream) {
  if (n_idx < 0 || n < 0 || (n_idx > 0 && (!d_idx || !d_flags))) return TQPK_EINVAL;
  if (n_idx == 0) return TQPK_OK;
  k_mark_rows<<<grid_for(n_idx, 4), kBlock, 0, static_cast<cudaStream_t>(stream)>>>(d_idx, n_idx, d_flags, n);
  TQPK_CHECK_LAUNCH();
  return TQPK_OK;
}
