// pmb_sort.cu — the sort strategy of the group-by: packed-key LSD radix sort + segmented reduce.
//
// The reference's A2 build sorts (u128 lane, row index) pairs with a stable 16-pass 8-bit LSD
// radix sort, marks segment starts and scans them into group ids on the CPU
// (crates/polars-metal-kernels/src/groupby_build_sort/gpu.rs:24-252,
// shaders/groupby_sort_u128_lane.metal:52-172, shaders/groupby_segments.metal:18-40; CPU
// statement groupby_build_sort/reference.rs:3-35). Here, for B200:
//   1. k_key_range   — per key column the range of its values (as order-preserving u64) and
//                      whether it has nulls; the host packs every key into only its significant
//                      bits (value - min), so most keys fit one 64-bit word and the sort runs
//                      ceil(bits / 8) passes instead of 16;
//   2. k_sort_encode — filter (the query's predicate), packed key + row index, compacted; and the
//                      digit histograms of every pass, in the same read;
//   3. k_sort_pass   — one stable 8-bit LSD pass per digit that is not constant (onesweep style:
//                      warp-level ranking through shared lane masks, per-digit decoupled look-back
//                      for the tile's global offsets, the tile reordered in shared memory so that
//                      the writes are coalesced);
//   4. k_seg_starts  — segment starts (key differs from its predecessor) compacted in order;
//   5. with the run-time compiler: k_chunk_bounds cuts the sorted rows at segment starts into
//      work items that fit a shared-memory table, and the partitioned strategy's aggregation
//      (pmb_jit_part_agg, then k_part_finalize) reduces every item's segments there; without it,
//      k_seg_reduce — one thread per group folds its rows into a group record and writes the
//      output row; groups of more than 256 rows go to k_seg_reduce_big (one CTA per group).
// Both use the hash path's records and finalisation, so every strategy gives identical results,
// exact float sums included. The order of the output groups is not specified.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <type_traits>
#include <vector>

#include "pmb_groupby.h"
#include "pmb_jit.h"

namespace {

constexpr int ST_NT = 256;              // threads of the sort kernels
constexpr int ST_PER = 16;              // rows per thread in an encode or segment tile
constexpr int ST_TILE = ST_NT * ST_PER;  // 4096 rows per tile
constexpr int RADIX = 256;
constexpr int MAX_PASSES = 16;
constexpr int BIG = 256;                // rows above which a group is reduced by a whole CTA
constexpr int BIG_NT = 128;

// packed-key layout of the sort: per key column an optional null bit, then (value - min) bits
struct SortKeyLayout {
  int n_keys;
  int words;  // 1 or 2
  int bits;   // total
  int col[PMB_MAX_KEYS];
  int null_off[PMB_MAX_KEYS];  // -1: no null bit
  int data_off[PMB_MAX_KEYS];
  int data_bits[PMB_MAX_KEYS];
  unsigned long long lo[PMB_MAX_KEYS];  // order-preserving u64 of the smallest valid value
  int dtype[PMB_MAX_KEYS];
  int elem[PMB_MAX_KEYS];
  const uint8_t* data[PMB_MAX_KEYS];
  const uint8_t* valid[PMB_MAX_KEYS];
};

struct RangeOut {
  unsigned long long lo[PMB_MAX_KEYS];
  unsigned long long hi[PMB_MAX_KEYS];
  unsigned int nulls[PMB_MAX_KEYS];
  unsigned int any[PMB_MAX_KEYS];
};

// order-preserving u64 of a key value: signed integers with the sign bit flipped, everything
// else (unsigned, bool, float bit patterns) as is; grouping only needs equality, the order just
// has to be consistent
__host__ __device__ __forceinline__ bool signed_dt(int dt) {
  return dt == PMB_I8 || dt == PMB_I16 || dt == PMB_I32 || dt == PMB_I64;
}
__device__ __forceinline__ unsigned long long ordered_bits(uint64_t b, int dt) {
  switch (dt) {
    case PMB_I8: return (unsigned long long)((long long)(int8_t)b) ^ 0x8000000000000000ULL;
    case PMB_I16: return (unsigned long long)((long long)(int16_t)b) ^ 0x8000000000000000ULL;
    case PMB_I32: return (unsigned long long)((long long)(int32_t)b) ^ 0x8000000000000000ULL;
    case PMB_I64: return b ^ 0x8000000000000000ULL;
    default: return b;
  }
}
__device__ __forceinline__ uint64_t from_ordered(unsigned long long o, int dt) {
  return signed_dt(dt) ? (o ^ 0x8000000000000000ULL) : o;
}

// Range of one key column in its own integer type: 16 bytes (V rows) per load, RU loads in flight
// per thread. Bound by DRAM; one row per load with four in flight read 12-byte keys at 2.7 TB/s
// (200M rows: 876 us).
constexpr int RU = 4;
template <typename T>
__device__ __forceinline__ void range_column(const T* __restrict__ d, const uint8_t* __restrict__ valid, int64_t n,
                                             T& lo, T& hi, unsigned& any, unsigned& nul) {
  constexpr int V = 16 / (int)sizeof(T);
  constexpr unsigned ALL = V == 16 ? 0xFFFFu : (1u << V) - 1u;
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t chunks = n / V;
  for (int64_t c0 = t0; c0 < chunks; c0 += RU * stride) {
    uint4 x[RU];
    unsigned ok[RU];
#pragma unroll
    for (int u = 0; u < RU; u++) {
      const int64_t c = c0 + u * stride;
      ok[u] = 0;
      x[u] = make_uint4(0u, 0u, 0u, 0u);
      if (c >= chunks) continue;
      x[u] = __ldcs(reinterpret_cast<const uint4*>(d) + c);
      if (!valid) ok[u] = ALL;
      else if (V == 16) ok[u] = reinterpret_cast<const uint16_t*>(valid)[c];
      else ok[u] = (valid[(c * V) >> 3] >> ((c * V) & 7)) & ALL;
      nul |= ok[u] != ALL;
    }
#pragma unroll
    for (int u = 0; u < RU; u++) {
      if (ok[u] == 0u) continue;
      any = 1u;
      T v[V];
      memcpy(v, &x[u], 16);
#pragma unroll
      for (int i = 0; i < V; i++) {
        if (!((ok[u] >> i) & 1u)) continue;
        lo = v[i] < lo ? v[i] : lo;
        hi = v[i] > hi ? v[i] : hi;
      }
    }
  }
  const int64_t r = chunks * V + t0;
  if (r < n) {
    if (pmb_valid_bit(valid, r)) {
      any = 1u;
      lo = d[r] < lo ? d[r] : lo;
      hi = d[r] > hi ? d[r] : hi;
    } else {
      nul = 1u;
    }
  }
}

// range of column (data, valid) of T, as order-preserving u64
template <typename T>
__device__ __forceinline__ void range_of(const uint8_t* data, const uint8_t* valid, int64_t n, int dtype,
                                         unsigned long long& lo, unsigned long long& hi, unsigned& any, unsigned& nul) {
  T l = std::is_signed<T>::value ? (T)(((unsigned long long)1 << (8 * sizeof(T) - 1)) - 1) : (T)~(T)0;
  T g = std::is_signed<T>::value ? (T)((unsigned long long)1 << (8 * sizeof(T) - 1)) : (T)0;
  range_column<T>(reinterpret_cast<const T*>(data), valid, n, l, g, any, nul);
  if (!any) return;
  lo = ordered_bits((uint64_t)l, dtype);
  hi = ordered_bits((uint64_t)g, dtype);
}

__global__ void __launch_bounds__(ST_NT) k_key_range(const __grid_constant__ SortKeyLayout L, int64_t n,
                                                     RangeOut* out) {
  for (int k = 0; k < L.n_keys; k++) {
    unsigned long long lo = ~0ULL, hi = 0;
    unsigned nul = 0, any = 0;
    const uint8_t* data = L.data[k];
    const uint8_t* valid = L.valid[k];
    const int dt = L.dtype[k];
    switch (dt) {
      case PMB_I8: range_of<int8_t>(data, valid, n, dt, lo, hi, any, nul); break;
      case PMB_I16: range_of<int16_t>(data, valid, n, dt, lo, hi, any, nul); break;
      case PMB_I32: range_of<int32_t>(data, valid, n, dt, lo, hi, any, nul); break;
      case PMB_I64: range_of<long long>(data, valid, n, dt, lo, hi, any, nul); break;
      case PMB_U8: range_of<uint8_t>(data, valid, n, dt, lo, hi, any, nul); break;
      case PMB_U16: range_of<uint16_t>(data, valid, n, dt, lo, hi, any, nul); break;
      case PMB_U32: case PMB_F32: range_of<uint32_t>(data, valid, n, dt, lo, hi, any, nul); break;
      case PMB_U64: case PMB_F64: range_of<unsigned long long>(data, valid, n, dt, lo, hi, any, nul); break;
      default:  // Bool
        for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
          if (!pmb_valid_bit(valid, r)) {
            nul = 1u;
            continue;
          }
          const unsigned long long o = pmb_load_bits(data, 0, r);
          lo = o < lo ? o : lo;
          hi = o > hi ? o : hi;
          any = 1u;
        }
        break;
    }
    for (int o = 16; o; o >>= 1) {
      const unsigned long long x = __shfl_xor_sync(0xffffffffu, lo, o), y = __shfl_xor_sync(0xffffffffu, hi, o);
      lo = x < lo ? x : lo;
      hi = y > hi ? y : hi;
      nul |= __shfl_xor_sync(0xffffffffu, nul, o);
      any |= __shfl_xor_sync(0xffffffffu, any, o);
    }
    if ((threadIdx.x & 31) == 0) {
      if (any) {
        atomicMin(&out->lo[k], lo);
        atomicMax(&out->hi[k], hi);
        atomicOr(&out->any[k], 1u);
      }
      if (nul) atomicOr(&out->nulls[k], 1u);
    }
  }
}

template <int W>
struct PKey {
  unsigned long long w[W];
};

template <int W>
__device__ __forceinline__ PKey<W> pack_sort_key(const SortKeyLayout& L, int64_t r) {
  PKey<W> k;
  for (int i = 0; i < W; i++) k.w[i] = 0;
  auto put = [&](int off, unsigned long long v, int bits) {
    if (bits == 0) return;
    const int wi = off >> 6, sh = off & 63;
    k.w[wi] |= v << sh;
    if (W > 1 && sh + bits > 64 && wi + 1 < W) k.w[wi + 1] |= v >> (64 - sh);
  };
  for (int c = 0; c < L.n_keys; c++) {
    if (!pmb_valid_bit(L.valid[c], r)) {
      put(L.null_off[c], 1ULL, 1);
      continue;
    }
    unsigned long long o = ordered_bits(pmb_load_bits(L.data[c], L.elem[c], r), L.dtype[c]);
    put(L.data_off[c], o - L.lo[c], L.data_bits[c]);
  }
  return k;
}

template <int W>
__device__ __forceinline__ unsigned digit_of(const PKey<W>& k, int shift) {
  const int wi = shift >> 6, sh = shift & 63;
  unsigned long long v = k.w[wi] >> sh;
  if (W > 1 && sh > 56 && wi + 1 < W) v |= k.w[wi + 1] << (64 - sh);
  return (unsigned)(v & 0xFF);
}

// hash of a packed key for the partitioned strategy: its top bits are the partition, its low 32
// bits the slot in the partition's shared-memory table
template <int W>
__device__ __forceinline__ unsigned long long part_hash(const PKey<W>& k) {
  unsigned long long h = pmb_fmix64(k.w[0]);
  if (W > 1) h = pmb_fmix64(h ^ (k.w[W - 1] + 0x9E3779B97F4A7C15ULL));
  return h;
}

// digit of a pass: key bits (sort strategy) or hash bits (partitioned strategy)
template <int W>
__device__ __forceinline__ unsigned pass_digit(const PKey<W>& k, int shift, bool hashed) {
  return hashed ? (unsigned)((part_hash<W>(k) >> shift) & 0xFFu) : digit_of<W>(k, shift);
}

struct EncodeParams {
  DQuery q;
  SortKeyLayout L;
  int passes;
  int64_t n;
  unsigned long long* keys;  // W words per key, word-major: word i of key j at keys[i * cap + j]
  uint64_t cap;
  unsigned int* idx;
  unsigned long long* lb;      // look-back states, one per tile, zeroed
  unsigned long long* ticket;
  unsigned long long* kept;    // rows that passed the filter
  unsigned int* hist;          // passes x 256
  unsigned int* status;
  int hashed;                  // digits of the key hash (partitioned strategy)
  int shift0;                  // bit of pass 0's digit; pass p uses shift0 + 8p
};

// exclusive offsets of a tile's ST_PER x 8 warp counts (item-major), in place, and their total: four
// counts to a lane of warp 0, which calls this whole
__device__ __forceinline__ unsigned scan_counts(unsigned int* cnt) {
  static_assert(ST_PER * (ST_NT / 32) == 128, "four counts per lane");
  const int lane = threadIdx.x & 31;
  uint4 c = reinterpret_cast<uint4*>(cnt)[lane];
  const unsigned sum = c.x + c.y + c.z + c.w;
  unsigned x = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += y;
  }
  const unsigned e = x - sum;
  reinterpret_cast<uint4*>(cnt)[lane] = make_uint4(e, e + c.x, e + c.x + c.y, e + c.x + c.y + c.z);
  return __shfl_sync(0xffffffffu, x, 31);
}

// Filter, pack and compact in row order (4096-row tiles, decoupled look-back), with the digit histograms
// of every pass. Without a predicate (PRED false) every row keeps its place: no verdicts, no look-back,
// four rows' keys packed before any is counted, so that their loads go out together. 200M rows of
// 12-byte keys: 2437 us with one thread scanning the tile's counts, a look-back for rows that all stay
// and a global count per partition, 1371 us now.
template <int W, bool PRED>
__global__ void __launch_bounds__(ST_NT) k_sort_encode(const __grid_constant__ EncodeParams E) {
  __shared__ unsigned int s_hist[MAX_PASSES][RADIX];
  __shared__ __align__(16) unsigned int s_cnt[ST_PER][ST_NT / 32];
  __shared__ long long s_tile;
  __shared__ unsigned long long s_base;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < E.passes * RADIX; i += ST_NT) (&s_hist[0][0])[i] = 0;
  if (PRED && tid == 0) s_tile = (long long)atomicAdd(E.ticket, 1ULL);
  __syncthreads();
  const long long tile = PRED ? s_tile : (long long)blockIdx.x;
  unsigned keep = 0;  // bit j: row j of this thread is kept
  if (PRED) {
    const TileCtx t{nullptr, nullptr, nullptr, 0};
    for (int j = 0; j < ST_PER; j++) {
      const int64_t r = tile * ST_TILE + (int64_t)j * ST_NT + tid;
      const bool k = r < E.n && eval_keep(E.q, t, r);
      const unsigned b = __ballot_sync(0xffffffffu, k);
      if (k) keep |= 1u << j;
      if (lane == 0) s_cnt[j][warp] = __popc(b);
    }
    __syncthreads();
    if (warp == 0) {
      const unsigned acc = scan_counts(&s_cnt[0][0]);
      const unsigned long long b = pmb_lookback_warp(E.lb, tile, acc, E.status);
      if (lane == 0) {
        s_base = b;
        if (tile == (long long)gridDim.x - 1) *E.kept = b + acc;
      }
    }
    __syncthreads();
  } else if (blockIdx.x == 0 && tid == 0) {
    *E.kept = (unsigned long long)E.n;
  }
  for (int j0 = 0; j0 < ST_PER; j0 += 4) {
    PKey<W> k[4];
    bool in[4];
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const int64_t r = tile * ST_TILE + (int64_t)(j0 + u) * ST_NT + tid;
      in[u] = PRED ? ((keep >> (j0 + u)) & 1u) != 0u : r < E.n;
      if (in[u]) k[u] = pack_sort_key<W>(E.L, r);
    }
#pragma unroll
    for (int u = 0; u < 4; u++) {
      const unsigned b = __ballot_sync(0xffffffffu, in[u]);
      if (!in[u]) continue;
      const int64_t r = tile * ST_TILE + (int64_t)(j0 + u) * ST_NT + tid;
      const unsigned long long h = E.hashed ? part_hash<W>(k[u]) : 0ULL;
      for (int p = 0; p < E.passes; p++) {
        const int sh = E.shift0 + 8 * p;
        atomicAdd(&s_hist[p][E.hashed ? (unsigned)(h >> sh) & 0xFFu : digit_of<W>(k[u], sh)], 1u);
      }
      const uint64_t pos = PRED ? s_base + s_cnt[j0 + u][warp] + __popc(b & ((1u << lane) - 1u)) : (uint64_t)r;
#pragma unroll
      for (int i = 0; i < W; i++) E.keys[(uint64_t)i * E.cap + pos] = k[u].w[i];
      E.idx[pos] = (unsigned)r;
    }
  }
  __syncthreads();
  for (int i = tid; i < E.passes * RADIX; i += ST_NT) {
    unsigned v = (&s_hist[0][0])[i];
    if (v) atomicAdd(&E.hist[i], v);
  }
}

struct PassParams {
  const unsigned long long* kin;
  unsigned long long* kout;
  const unsigned int* iin;
  unsigned int* iout;
  uint64_t cap;  // word stride of the key arrays
  int64_t n;
  int shift;
  const unsigned int* hist;      // this pass's 256 digit counts
  unsigned long long* lb;        // n_tiles x 256 look-back states (tile-major), zeroed
  unsigned long long* ticket;
  unsigned int* status;
  // values carried along instead of row numbers (PAY): element e of the pass's output row goes to
  // pay_out[e]; it comes from pay_in[e] by position, or (FIRST) from column data by the row number
  int n_pay;
  int pay_elem[PMB_MAX_COLS + 1];             // bytes of an output element: 8 or 4
  const uint8_t* pay_in[PMB_MAX_COLS + 1];    // null: the mask element (FIRST)
  int pay_src[PMB_MAX_COLS + 1];              // FIRST: bytes of the column's values (1, 2, 4, 8)
  uint8_t* pay_out[PMB_MAX_COLS + 1];
  int n_mask;                                 // the mask's bits, from these bitmaps
  const uint8_t* mask_bits[2 * PMB_MAX_COLS];
  int mask_pos[2 * PMB_MAX_COLS];
};

// Tile shape of a pass, for W-word keys: three (two) CTAs of 12 (16) warps fit an SM's shared memory
template <int W>
struct PassShape {
  static constexpr int NT = W == 1 ? 384 : 512;
  static constexpr int PER = W == 1 ? 10 : 6;
  static constexpr int CTAS = W == 1 ? 3 : 2;
  static constexpr int TILE = NT * PER, NW = NT / 32;
  static constexpr size_t SMEM = (size_t)TILE * (8 * W + 4) + (size_t)NW * RADIX * 8;
};

// exclusive prefix of one digit over the earlier tiles: LB_W predecessor states are read per step
// (independent loads, one L2 round trip), summed up to the nearest inclusive prefix
constexpr int LB_W = 4;
__device__ __forceinline__ unsigned long long digit_lookback(unsigned long long* lb, long long tile, unsigned count,
                                                             unsigned int* st) {
  const unsigned long long VAL = (1ULL << 62) - 1;
  if (tile == 0) return 0;
  unsigned long long excl = 0;
  long long t = tile - 1;
  uint32_t spins = 0;
  for (;;) {
    unsigned long long s[LB_W];
#pragma unroll
    for (int k = 0; k < LB_W; k++)
      s[k] = t - k >= 0 ? *((volatile unsigned long long*)&lb[(t - k) * RADIX]) : (2ULL << 62);
    bool done = false, miss = false;
    int used = 0;
#pragma unroll
    for (int k = 0; k < LB_W; k++) {
      if (done || miss) continue;
      const unsigned f = (unsigned)(s[k] >> 62);
      if (f == 0u) {
        miss = true;
      } else {
        excl += s[k] & VAL;
        used++;
        done = f == 2u;
      }
    }
    if (done) break;
    t -= used;
    if (miss && ++spins > PMB_SPIN_LIMIT) {
      atomicOr(st, PMB_ST_TIMEOUT);
      return 0;
    }
  }
  *((volatile unsigned long long*)&lb[tile * RADIX]) = (2ULL << 62) | (excl + count);
  return excl;
}

// One stable LSD pass over 8 bits at `shift` (onesweep: one read and one write of the pairs).
// Every warp counts its keys' digits with shared atomics as soon as they are loaded, so the tile's
// counts are published to the later tiles' look-backs before any ranking, and the counters, once
// scanned, are the keys' running positions in the tile: a key goes straight to its place in shared
// memory. The lanes of a round with the same digit find each other through a per-warp table of
// lane masks (one atomicOr; the way CUB's block radix ranking has as its atomic-or match):
// __match_any_sync and eight ballots per key both cost more issue slots.
// What bounds it: shared-memory atomics and accesses (42 shared wavefronts per 32 keys, the LSU data pipe at 67%
// of its peak over 20M pairs and DRAM at 27%; without any output or look-back the ranking alone takes 60% of
// the time), then the loads and look-backs that 36 warps an SM wait for. 100M 64-bit keys:
// 795 us (3.0 TB/s of the 6.4 a plain copy reaches); 256 threads x 16 keys with match_any, ranks
// held to the end and a look-back of one state per step took 1020 us. 128-bit keys, 20M: 259 us,
// against 552 us. Prefetching the next tile with bulk copies (persistent CTAs) took 900-960 us.
// With PAY a row takes its aggregated values with it through the passes instead of its number: the
// values move element by element through the tile's buffers to the places the keys went to.
enum { PAY_NONE = 0, PAY_FIRST = 1, PAY_NEXT = 2 };
template <int W, bool HASHED, int PAY = PAY_NONE>
__global__ void __launch_bounds__(PassShape<W>::NT, PassShape<W>::CTAS)
    k_sort_pass(const __grid_constant__ PassParams P) {
  constexpr int NT = PassShape<W>::NT, PER = PassShape<W>::PER, TILE = PassShape<W>::TILE, NW = PassShape<W>::NW;
  extern __shared__ __align__(16) unsigned char smem[];
  unsigned long long* s_key = reinterpret_cast<unsigned long long*>(smem);    // W x TILE
  unsigned int* s_idx = reinterpret_cast<unsigned int*>(s_key + W * TILE);   // TILE
  unsigned int(*s_off)[RADIX] = reinterpret_cast<unsigned int(*)[RADIX]>(s_idx + TILE);  // NW
  unsigned int(*s_lanes)[RADIX] = s_off + NW;                                            // NW
  __shared__ long long s_out[RADIX];  // output position of a digit's first key, less its tile position
  __shared__ uint2 s_scan[RADIX / 32];
  __shared__ long long s_tile;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) {
    const unsigned st = *reinterpret_cast<volatile unsigned int*>(P.status);
    const long long t = (long long)atomicAdd(P.ticket, 1ULL);
    s_tile = st & PMB_ST_TIMEOUT ? -1 : t;
  }
  for (int i = tid; i < 2 * NW * RADIX; i += NT) (&s_off[0][0])[i] = 0u;
  __syncthreads();
  const long long tile = s_tile;
  if (tile < 0) return;  // a wait gave up: the pass's input need not match its digit counts
  // warp-striped items: item j of lane l of warp w is tile element w * PER * 32 + j * 32 + l
  const int64_t e0 = (int64_t)tile * TILE + warp * (PER * 32) + lane;
  const unsigned lt = (1u << lane) - 1u;
  PKey<W> k[PER];
  unsigned ix[PER];
  unsigned short lps[PER];  // PAY: the keys' places in the tile
#pragma unroll
  for (int j = 0; j < PER; j++)
#pragma unroll
    for (int w = 0; w < W; w++) k[j].w[w] = e0 + j * 32 < P.n ? __ldcs(&P.kin[(uint64_t)w * P.cap + e0 + j * 32]) : 0ULL;
#pragma unroll
  for (int j = 0; j < PER; j++) ix[j] = PAY != PAY_NEXT && e0 + j * 32 < P.n ? __ldcs(&P.iin[e0 + j * 32]) : 0u;
  unsigned dg[(PER + 3) / 4];  // digits of the key hash, four to a register (a key's own digit is a shift away)
#pragma unroll
  for (int j = 0; j < (PER + 3) / 4; j++) dg[j] = 0u;
#pragma unroll
  for (int j = 0; HASHED && j < PER; j++) dg[j >> 2] |= pass_digit<W>(k[j], P.shift, true) << (8 * (j & 3));
  auto digit = [&](int j) { return HASHED ? (dg[j >> 2] >> (8 * (j & 3))) & 0xFFu : digit_of<W>(k[j], P.shift); };
#pragma unroll
  for (int j = 0; j < PER; j++)
    if (e0 + j * 32 < P.n) atomicAdd(&s_off[warp][digit(j)], 1u);
  __syncthreads();
  // thread d: the tile's count of digit d, published at once; then the tile-local exclusive scan
  // over the digits, and every warp's first position of the digit
  unsigned acc = 0, x = 0, gs = 0;  // gs: output position of the digit's first key, all tiles
  if (tid < RADIX) {
    unsigned c[NW];
#pragma unroll
    for (int w = 0; w < NW; w++) c[w] = s_off[w][tid];
#pragma unroll
    for (int w = 0; w < NW; w++) {
      const unsigned t = c[w];
      c[w] = acc;
      acc += t;
    }
    *((volatile unsigned long long*)&P.lb[tile * RADIX + tid]) = ((tile == 0 ? 2ULL : 1ULL) << 62) | acc;
    const unsigned hd = P.hist[tid];
    x = acc;
    gs = hd;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o), z = __shfl_up_sync(0xffffffffu, gs, o);
      if (lane >= o) {
        x += y;
        gs += z;
      }
    }
    if (lane == 31) s_scan[warp] = make_uint2(x, gs);
    asm volatile("bar.sync 1, 256;" ::: "memory");  // the RADIX threads of this scan
#pragma unroll
    for (int w = 0; w < RADIX / 32; w++)
      if (w < warp) {
        x += s_scan[w].x;
        gs += s_scan[w].y;
      }
    x -= acc;
    gs -= hd;
#pragma unroll
    for (int w = 0; w < NW; w++) s_off[w][tid] = c[w] + x;
  }
  __syncthreads();
  // the tile reordered by digit in shared memory, in item order (stable): the lanes of a round with
  // the same digit are ordered by lane, earlier rounds and warps come first
#pragma unroll
  for (int j = 0; j < PER; j++) {
    const bool in = e0 + j * 32 < P.n;
    const unsigned d = digit(j);
    if (in) atomicOr(&s_lanes[warp][d], 1u << lane);
    __syncwarp();
    const unsigned peers = s_lanes[warp][d], first = s_off[warp][d], below = __popc(peers & lt);
    __syncwarp();
    if (in) {
      if (below == 0u) {
        s_off[warp][d] = first + __popc(peers);
        s_lanes[warp][d] = 0u;
      }
      const unsigned lp = first + below;
#pragma unroll
      for (int w = 0; w < W; w++) s_key[w * TILE + lp] = k[j].w[w];
      if (PAY == PAY_NONE) s_idx[lp] = ix[j];
      else lps[j] = (unsigned short)lp;
    }
    __syncwarp();
  }
  if (tid < RADIX) {
    const unsigned long long pre = digit_lookback(P.lb + tid, tile, acc, P.status);
    s_out[tid] = (long long)gs + (long long)pre - (long long)x;
  }
  __syncthreads();
  const int valid = (int)min((long long)TILE, (long long)P.n - tile * TILE);
  unsigned dest[PER];  // PAY: output rows of the tile's places tid, tid + NT, ...
#pragma unroll
  for (int j = 0; j < PER; j++) {
    const int i = tid + j * NT;
    if (i >= valid) continue;
    PKey<W> kk;
#pragma unroll
    for (int w = 0; w < W; w++) kk.w[w] = s_key[w * TILE + i];
    const uint64_t g = (uint64_t)(s_out[pass_digit<W>(kk, P.shift, HASHED)] + i);
#pragma unroll
    for (int w = 0; w < W; w++) P.kout[(uint64_t)w * P.cap + g] = kk.w[w];
    if (PAY == PAY_NONE) P.iout[g] = s_idx[i];
    else dest[j] = (unsigned)g;
  }
  if (PAY != PAY_NONE) {
    // an 8-byte element goes through the keys' buffer, a 4-byte one through the row numbers'
    for (int el = 0; el < P.n_pay; el++) {
      const uint8_t* src = P.pay_in[el];
      if (P.pay_elem[el] == 8) {
        unsigned long long v[PER];
#pragma unroll
        for (int j = 0; j < PER; j++)
          v[j] = e0 + j * 32 < P.n
                     ? reinterpret_cast<const unsigned long long*>(src)[PAY == PAY_FIRST ? (int64_t)ix[j] : e0 + j * 32]
                     : 0ULL;
        __syncthreads();  // the buffer's last readers are done
#pragma unroll
        for (int j = 0; j < PER; j++)
          if (e0 + j * 32 < P.n) s_key[lps[j]] = v[j];
        __syncthreads();
        unsigned long long* out = reinterpret_cast<unsigned long long*>(P.pay_out[el]);
#pragma unroll
        for (int j = 0; j < PER; j++)
          if (tid + j * NT < valid) out[dest[j]] = s_key[tid + j * NT];
      } else {
        unsigned v[PER];
#pragma unroll
        for (int j = 0; j < PER; j++) {
          v[j] = 0u;
          if (e0 + j * 32 >= P.n) continue;
          if (PAY == PAY_NEXT) {
            v[j] = reinterpret_cast<const unsigned*>(src)[e0 + j * 32];
          } else if (src) {
            const int b = P.pay_src[el];
            v[j] = b == 4 ? reinterpret_cast<const unsigned*>(src)[ix[j]]
                          : b == 2 ? (unsigned)reinterpret_cast<const unsigned short*>(src)[ix[j]] : (unsigned)src[ix[j]];
          } else {
            for (int q = 0; q < P.n_mask; q++)
              v[j] |= ((P.mask_bits[q][ix[j] >> 3] >> (ix[j] & 7)) & 1u) << P.mask_pos[q];
          }
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < PER; j++)
          if (e0 + j * 32 < P.n) s_idx[lps[j]] = v[j];
        __syncthreads();
        unsigned* out = reinterpret_cast<unsigned*>(P.pay_out[el]);
#pragma unroll
        for (int j = 0; j < PER; j++)
          if (tid + j * NT < valid) out[dest[j]] = s_idx[tid + j * NT];
      }
    }
  }
}

struct StartsParams {
  const unsigned long long* keys;
  uint64_t cap;
  int64_t n;
  unsigned int* starts;  // n_groups + 1 entries (the last one = n)
  unsigned long long* lb;
  unsigned long long* ticket;
  unsigned long long* n_groups;
  unsigned int* status;
};

template <int W>
__global__ void __launch_bounds__(ST_NT) k_seg_starts(const __grid_constant__ StartsParams S) {
  __shared__ __align__(16) unsigned int s_cnt[ST_PER][ST_NT / 32];
  __shared__ long long s_tile;
  __shared__ unsigned long long s_base;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  if (tid == 0) s_tile = (long long)atomicAdd(S.ticket, 1ULL);
  __syncthreads();
  const long long tile = s_tile;
  bool head[ST_PER];
  for (int j = 0; j < ST_PER; j++) {
    const int64_t e = tile * ST_TILE + (int64_t)j * ST_NT + tid;
    bool hd = false;
    if (e < S.n) {
      hd = e == 0;
      for (int w = 0; w < W && !hd; w++) hd = S.keys[(uint64_t)w * S.cap + e] != S.keys[(uint64_t)w * S.cap + e - 1];
    }
    head[j] = hd;
    const unsigned b = __ballot_sync(0xffffffffu, hd);
    if (lane == 0) s_cnt[j][warp] = __popc(b);
  }
  __syncthreads();
  if (warp == 0) {
    const unsigned acc = scan_counts(&s_cnt[0][0]);
    const unsigned long long b = pmb_lookback_warp(S.lb, tile, acc, S.status);
    if (lane == 0) {
      s_base = b;
      if (tile == (long long)gridDim.x - 1) {
        *S.n_groups = b + acc;
        S.starts[b + acc] = (unsigned)S.n;
      }
    }
  }
  __syncthreads();
  for (int j = 0; j < ST_PER; j++) {
    const unsigned b = __ballot_sync(0xffffffffu, head[j]);
    if (head[j]) {
      const int64_t e = tile * ST_TILE + (int64_t)j * ST_NT + tid;
      S.starts[s_base + s_cnt[j][warp] + __popc(b & ((1u << lane) - 1u))] = (unsigned)e;
    }
  }
}

struct ReduceParams {
  DQuery q;
  RecInit ri;
  SortKeyLayout L;
  const unsigned long long* keys;
  uint64_t cap;
  const unsigned int* idx;
  const unsigned int* starts;
  const unsigned long long* n_groups;
  unsigned int* big;             // groups reduced by k_seg_reduce_big
  unsigned long long* big_n;
  unsigned int* status;
  uint8_t* out_data[PMB_MAX_OUT];
  uint8_t* out_valid[PMB_MAX_OUT];
};

__device__ __forceinline__ void store_bits(uint8_t* d, int bytes, int64_t p, uint64_t v) {
  switch (bytes) {
    case 0: break;
    case 1: d[p] = (uint8_t)v; break;
    case 2: reinterpret_cast<uint16_t*>(d)[p] = (uint16_t)v; break;
    case 4: reinterpret_cast<uint32_t*>(d)[p] = (uint32_t)v; break;
    default: reinterpret_cast<uint64_t*>(d)[p] = v; break;
  }
}

// key value of key column c from the packed sort key (false: null)
template <int W>
__device__ __forceinline__ bool unpack_sort_key(const SortKeyLayout& L, const PKey<W>& k, int c, uint64_t& v) {
  auto get = [&](int off, int bits) -> unsigned long long {
    if (bits == 0) return 0ULL;
    const int wi = off >> 6, sh = off & 63;
    unsigned long long x = k.w[wi] >> sh;
    if (W > 1 && sh + bits > 64 && wi + 1 < W) x |= k.w[wi + 1] << (64 - sh);
    return bits == 64 ? x : (x & ((1ULL << bits) - 1ULL));
  };
  if (L.null_off[c] >= 0 && get(L.null_off[c], 1)) return false;
  v = from_ordered(get(L.data_off[c], L.data_bits[c]) + L.lo[c], L.dtype[c]);
  return true;
}

// writes group p's output row from its record; `bitset` chooses how validity / bool bits are set
// (warp-wide for the one-thread-per-group kernel, atomic for the big-group kernel)
template <int W, bool WARP>
__device__ __forceinline__ void write_group(const ReduceParams& R, int64_t p, int64_t p_first, bool have,
                                           const PKey<W>& k, const uint8_t* rec) {
  const DQuery& q = R.q;
  int oc = 0;
  auto setbit = [&](uint8_t* words, bool bit) {
    if (WARP) {
      warp_set_bits(reinterpret_cast<unsigned int*>(words), p, p_first, bit);
    } else if (bit) {
      atomicOr(reinterpret_cast<unsigned int*>(words) + (p >> 5), 1u << (p & 31));
    }
  };
  for (int c = 0; c < q.n_keys; c++, oc++) {
    uint64_t v = 0;
    const bool valid = have && unpack_sort_key<W>(R.L, k, c, v);
    const int dt = R.L.dtype[c];
    if (have) store_bits(R.out_data[oc], pmb_dtype_bytes(dt), p, v);
    if (dt == PMB_BOOL) setbit(R.out_data[oc], have && valid && v);
    setbit(R.out_valid[oc], have && valid);
  }
  for (int a = 0; a < q.n_aggs; a++, oc++) {
    const DAggOut& A = q.agg[a];
    bool valid = true;
    uint64_t bits = 0;
    if (have) finalize_agg(q, A, rec, valid, bits);
    if (have) store_bits(R.out_data[oc], pmb_dtype_bytes(A.out_dtype), p, bits);
    if (A.out_dtype == PMB_BOOL) setbit(R.out_data[oc], have && valid && bits);
    setbit(R.out_valid[oc], have && valid);
  }
}

template <int W, int RW>
__global__ void __launch_bounds__(ST_NT) k_seg_reduce(const __grid_constant__ ReduceParams R) {
  const int64_t ng = (int64_t)*R.n_groups;
  const TileCtx t{nullptr, nullptr, nullptr, 0};
  uint64_t recw[RW];  // the group record, RW >= rec_bytes / 8
  uint8_t* rec = reinterpret_cast<uint8_t*>(recw);
  const int rw = R.q.rec_bytes / 8;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  // every lane of a warp runs the same number of iterations (warp-wide bit setting)
  const int64_t span = (ng + stride - 1) / stride * stride;
  for (int64_t g0 = (int64_t)blockIdx.x * blockDim.x; g0 < span; g0 += stride) {
    const int64_t g = g0 + threadIdx.x;
    const int64_t p_first = g0 + (threadIdx.x & ~31);
    bool have = g < ng;
    PKey<W> k{};
    if (have) {
      const unsigned s = R.starts[g], e = R.starts[g + 1];
      for (int i = 0; i < W; i++) k.w[i] = R.keys[(uint64_t)i * R.cap + s];
      if (e - s > (unsigned)BIG) {
        R.big[atomicAdd(R.big_n, 1ULL)] = (unsigned)g;
        have = false;
      } else {
        for (int w = 0; w < rw; w++) recw[w] = R.ri.w[w];
        for (unsigned i = s; i < e; i++) {
          const int64_t row = R.idx[i];
          fx_range_check(R.q, t, row, R.status);
          apply_row_private(R.q, t, rec, row);
        }
      }
    }
    write_group<W, true>(R, g, p_first, have, k, rec);
  }
}

// groups of more than BIG rows: one CTA each (persistent over the list); thread records are
// merged in shared memory by one thread
template <int W>
__global__ void __launch_bounds__(BIG_NT) k_seg_reduce_big(const __grid_constant__ ReduceParams R) {
  extern __shared__ __align__(16) unsigned char srec[];  // BIG_NT records
  const TileCtx t{nullptr, nullptr, nullptr, 0};
  const int rb = R.q.rec_bytes, rw = rb / 8;
  const unsigned long long nb = *R.big_n;
  uint8_t* mine = srec + (size_t)threadIdx.x * rb;
  for (unsigned long long b = blockIdx.x; b < nb; b += gridDim.x) {
    const unsigned g = R.big[b];
    const unsigned s = R.starts[g], e = R.starts[g + 1];
    for (int w = 0; w < rw; w++) reinterpret_cast<uint64_t*>(mine)[w] = R.ri.w[w];
    for (unsigned i = s + threadIdx.x; i < e; i += BIG_NT) {
      const int64_t row = R.idx[i];
      fx_range_check(R.q, t, row, R.status);
      apply_row_private(R.q, t, mine, row);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int j = 1; j < BIG_NT; j++) merge_private(R.q, srec, srec + (size_t)j * rb);
      PKey<W> k;
      for (int i = 0; i < W; i++) k.w[i] = R.keys[(uint64_t)i * R.cap + s];
      write_group<W, false>(R, g, g, true, k, srec);
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- partitioned strategy
// After the hash-digit passes the kept rows are ordered by partition (the top `pb` bits of the key
// hash), so every group's rows lie inside one partition; the
// partition starts are read off the sorted keys. k_part_agg: persistent CTAs take work items (runs of
// consecutive partitions) and aggregate one partition at a time in a shared-memory table (slot claim by a tag word, records in the global-record layout updated by
// apply_row_shared, values gathered by row index). At the end of each partition the occupied
// slots are compacted and written straight to the output columns (one atomic per partition for
// the output rows; validity words built in shared memory). No global hash table is involved.
constexpr int PA_NT = 1024;
constexpr int PA_R = 2;   // rows per thread and step
constexpr int PA_UC = 4;  // aggregated columns whose loads are issued together

struct PartParams {
  DQuery q;
  RecInit ri;
  SortKeyLayout L;
  const unsigned long long* keys;  // sorted packed keys, word-major (stride cap)
  uint64_t cap;
  const unsigned int* idx;         // their row indices
  int64_t m;                       // kept rows
  const unsigned long long* pstart;  // n_parts + 1: first row of every partition
  int64_t n_parts;
  int run;                         // partitions per work item
  int64_t n_items;
  int slots;                       // shared table slots
  int n_out;
  int stage_bytes;                 // one row's aggregated columns, staged per thread
  unsigned int used;               // columns the aggregates read (bit per column)
  int n_used;
  int32_t ucol[PMB_MAX_COLS];      // those columns, in order
  int32_t sdoff[PMB_MAX_COLS];     // a column's value in the stage
  int32_t svoff[PMB_MAX_COLS];     // its validity byte in the stage
  unsigned long long* ticket;
  unsigned long long* n_groups;    // output rows claimed
  int64_t out_cap;
  unsigned int* status;
  uint8_t* out_data[PMB_MAX_OUT];
  uint8_t* out_valid[PMB_MAX_OUT];
};

template <int W>
__device__ __forceinline__ PKey<W> pa_key(const PartParams& A, int64_t i) {
  PKey<W> k;
#pragma unroll
  for (int w = 0; w < W; w++) k.w[w] = A.keys[(uint64_t)w * A.cap + i];
  return k;
}
// shared-memory layout of k_part_agg for `slots` slots
struct PaLayout {
  size_t tag, key, rec, list, vb, db, stage, bytes;
};
__host__ __device__ inline PaLayout pa_layout(int slots, int W, int rec_bytes, int n_out, int stage_bytes) {
  PaLayout o;
  const size_t words = (size_t)slots / 32 + 2;
  o.tag = 0;
  o.key = ((size_t)slots * 4 + 15) & ~(size_t)15;
  o.rec = o.key + (size_t)slots * 8 * W;
  o.list = o.rec + (size_t)slots * rec_bytes;
  o.vb = (o.list + (size_t)slots * 2 + 15) & ~(size_t)15;
  o.db = o.vb + (size_t)n_out * words * 4;
  o.stage = (o.db + (size_t)PMB_MAX_KEYS * words * 4 + 15) & ~(size_t)15;
  o.bytes = o.stage + (size_t)PA_NT * stage_bytes;
  return o;
}

template <int W>
__global__ void __launch_bounds__(PA_NT, 1) k_part_agg(const __grid_constant__ PartParams A) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (*A.status & PMB_ST_TIMEOUT) return;  // the passes gave up: their row numbers need not be any
  const int S = A.slots, rb = A.q.rec_bytes, rw = rb / 8;
  const PaLayout Ly = pa_layout(S, W, rb, A.n_out, A.stage_bytes);
  unsigned int* tag = reinterpret_cast<unsigned int*>(smem + Ly.tag);  // 0 empty, 1 claimed, 2 key published
  unsigned long long* tkey = reinterpret_cast<unsigned long long*>(smem + Ly.key);  // W x S
  uint8_t* trec = smem + Ly.rec;
  unsigned short* list = reinterpret_cast<unsigned short*>(smem + Ly.list);
  const int nwords = S / 32 + 2;
  unsigned int* vb = reinterpret_cast<unsigned int*>(smem + Ly.vb);  // n_out x nwords
  unsigned int* db = reinterpret_cast<unsigned int*>(smem + Ly.db);  // n_keys x nwords (Bool keys)
  uint8_t* stage = smem + Ly.stage + (size_t)threadIdx.x * A.stage_bytes;
  __shared__ long long s_item;
  __shared__ unsigned long long s_base;
  __shared__ unsigned s_total;  // claimed slots of the current partition
  const int tid = threadIdx.x;
  bool has_fx = false;
  for (int f = 0; f < A.q.n_fields; f++) has_fx |= A.q.field[f].kind == F_SUM_FX;
  for (int i = tid; i < S; i += PA_NT) {
    tag[i] = 0u;
    for (int w = 0; w < rw; w++) reinterpret_cast<uint64_t*>(trec + (size_t)i * rb)[w] = A.ri.w[w];
  }
  for (int i = tid; i < (A.n_out + PMB_MAX_KEYS) * nwords; i += PA_NT) vb[i] = 0u;  // vb and db are adjacent
  if (tid == 0) s_total = 0u;
  for (;;) {
    __syncthreads();
    if (tid == 0) s_item = (long long)atomicAdd(A.ticket, 1ULL);
    __syncthreads();
    const long long it = s_item;
    if (it >= A.n_items) break;
    {
      // the item's partitions: rows [ps, pe)
      const int64_t ps = (int64_t)A.pstart[it * A.run], pe = (int64_t)A.pstart[min((long long)A.n_parts, (it + 1) * A.run)];
      for (int64_t b = ps; b < pe; b += (int64_t)PA_NT * PA_R) {
        // PA_R rows per thread; their key and row-index loads go out together
        PKey<W> k[PA_R];
        unsigned slot[PA_R], row[PA_R], probes[PA_R];
        bool pending[PA_R];
        int found[PA_R];
#pragma unroll
        for (int r = 0; r < PA_R; r++) {
          const int64_t i = b + (int64_t)r * PA_NT + tid;
          pending[r] = i < pe;
          found[r] = -1;
          probes[r] = 0;
          slot[r] = 0;
          row[r] = 0;
          if (pending[r]) {
            k[r] = pa_key<W>(A, i);
            row[r] = A.idx[i];
          }
        }
#pragma unroll
        for (int r = 0; r < PA_R; r++)
          if (pending[r]) slot[r] = (unsigned)(((part_hash<W>(k[r]) & 0xFFFFFFFFULL) * (unsigned long long)S) >> 32);
        // find or claim the keys' slots. A claimer publishes its key before the next barrier, so a
        // row that meets a slot being claimed tries that slot again after the barrier instead of
        // waiting for it (a wait could stall on a claimer in its own warp)
        for (int round = 0; round < 64; round++) {
          bool any = false;
#pragma unroll
          for (int r = 0; r < PA_R; r++) {
            while (pending[r]) {
              const unsigned sl = slot[r];
              unsigned tg = *reinterpret_cast<volatile unsigned int*>(&tag[sl]);
              if (tg == 0u) {
                if (atomicCAS(&tag[sl], 0u, 1u) == 0u) {
#pragma unroll
                  for (int w = 0; w < W; w++) tkey[(size_t)w * S + sl] = k[r].w[w];
                  __threadfence_block();
                  *reinterpret_cast<volatile unsigned int*>(&tag[sl]) = 2u;
                  list[atomicAdd(&s_total, 1u)] = (unsigned short)sl;  // the item's groups, in claim order
                  found[r] = (int)sl;
                  pending[r] = false;
                  break;
                }
                tg = *reinterpret_cast<volatile unsigned int*>(&tag[sl]);
              }
              if (tg != 2u) break;  // being claimed: this slot again after the barrier
              __threadfence_block();
              bool eq = true;
#pragma unroll
              for (int w = 0; w < W; w++) eq &= reinterpret_cast<volatile unsigned long long*>(tkey)[(size_t)w * S + sl] == k[r].w[w];
              if (eq) {
                found[r] = (int)sl;
                pending[r] = false;
                break;
              }
              slot[r] = sl + 1 == (unsigned)S ? 0u : sl + 1;
              if (++probes[r] >= (unsigned)S) {
                atomicOr(A.status, PMB_ST_OVERFLOW);  // the item has more groups than the table
                pending[r] = false;
              }
            }
            any |= pending[r];
          }
          if (!__syncthreads_or(any)) break;
        }
        // the rows' aggregated columns: the first PA_UC columns of both rows are loaded together,
        // then every row is staged (one copy of each value) and applied to its record
        uint64_t vals[PA_R][PA_UC];
        unsigned vmask[PA_R];
#pragma unroll
        for (int r = 0; r < PA_R; r++) {
          vmask[r] = 0u;
          if (pending[r]) atomicOr(A.status, PMB_ST_OVERFLOW);
#pragma unroll
          for (int u = 0; u < PA_UC; u++) {
            vals[r][u] = 0;
            if (found[r] >= 0 && u < A.n_used) {
              const DCol& C = A.q.col[A.ucol[u]];
              vals[r][u] = pmb_load_bits(C.data, C.elem, row[r]);
              if (C.valid && pmb_valid_bit(C.valid, row[r])) vmask[r] |= 1u << u;
            }
          }
        }
        auto put = [&](int c, uint64_t v, bool ok) {
          const DCol& C = A.q.col[c];
          uint8_t* d = stage + A.sdoff[c];
          switch (C.elem) {
            case 8: *reinterpret_cast<uint64_t*>(d) = v; break;
            case 4: *reinterpret_cast<uint32_t*>(d) = (uint32_t)v; break;
            case 2: *reinterpret_cast<uint16_t*>(d) = (uint16_t)v; break;
            default: *d = (uint8_t)v; break;
          }
          if (C.valid) stage[A.svoff[c]] = ok ? 1 : 0;
        };
#pragma unroll
        for (int r = 0; r < PA_R; r++) {
          if (found[r] < 0) continue;
#pragma unroll
          for (int u = 0; u < PA_UC; u++)
            if (u < A.n_used) put(A.ucol[u], vals[r][u], (vmask[r] >> u) & 1u);
          for (int u = PA_UC; u < A.n_used; u++) {
            const DCol& C = A.q.col[A.ucol[u]];
            put(A.ucol[u], pmb_load_bits(C.data, C.elem, row[r]), C.valid && pmb_valid_bit(C.valid, row[r]));
          }
          const TileCtx ts{stage, A.sdoff, A.svoff, 0};
          if (has_fx) fx_range_check(A.q, ts, 0, A.status);
          apply_row_shared(A.q, ts, trec + (size_t)found[r] * rb, 0);
        }
      }
      // the partition is complete: its groups (the claimed slots) go to the output
      __syncthreads();
      const unsigned total = s_total;
      if (tid == 0) s_base = total ? atomicAdd(A.n_groups, (unsigned long long)total) : 0ULL;
      __syncthreads();
      const unsigned long long base = s_base, a0 = base & ~31ULL;
      for (unsigned li = tid; li < total; li += PA_NT) {
        const unsigned long long p = base + li;
        if ((int64_t)p >= A.out_cap) {
          atomicOr(A.status, PMB_ST_OVERFLOW);
          continue;
        }
        const int sl = list[li];
        const unsigned rbit = (unsigned)(p - a0);
        PKey<W> k;
#pragma unroll
        for (int w = 0; w < W; w++) k.w[w] = tkey[(size_t)w * S + sl];
        const uint8_t* rec = trec + (size_t)sl * rb;
        int oc = 0;
        for (int c = 0; c < A.q.n_keys; c++, oc++) {
          uint64_t v = 0;
          const bool valid = unpack_sort_key<W>(A.L, k, c, v);
          const int dt = A.L.dtype[c];
          if (dt == PMB_BOOL) {
            if (valid && v) atomicOr(&db[c * nwords + (rbit >> 5)], 1u << (rbit & 31));
          } else {
            store_bits(A.out_data[oc], pmb_dtype_bytes(dt), (int64_t)p, v);
          }
          if (valid) atomicOr(&vb[oc * nwords + (rbit >> 5)], 1u << (rbit & 31));
        }
        for (int ag = 0; ag < A.q.n_aggs; ag++, oc++) {
          const DAggOut& Ag = A.q.agg[ag];
          bool valid = true;
          uint64_t bits = 0;
          finalize_agg(A.q, Ag, rec, valid, bits);
          store_bits(A.out_data[oc], pmb_dtype_bytes(Ag.out_dtype), (int64_t)p, bits);
          if (Ag.out_dtype == PMB_BOOL && valid && bits)
            atomicOr(reinterpret_cast<unsigned int*>(A.out_data[oc]) + (p >> 5), 1u << (p & 31));
          if (valid) atomicOr(&vb[oc * nwords + (rbit >> 5)], 1u << (rbit & 31));
        }
      }
      __syncthreads();
      // bitmap words into the outputs, then the table and the bitmaps are reset
      const int nw = total ? (int)((base - a0 + total + 31) / 32) : 0;
      for (int i = tid; i < A.n_out * nw; i += PA_NT) {
        const int oc = i / nw, w = i % nw;
        if ((int64_t)((a0 >> 5) + w) * 32 >= A.out_cap + 32) continue;
        const unsigned v = vb[oc * nwords + w];
        if (v) atomicOr(reinterpret_cast<unsigned int*>(A.out_valid[oc]) + (a0 >> 5) + w, v);
        vb[oc * nwords + w] = 0u;
        if (oc < A.q.n_keys && A.L.dtype[oc] == PMB_BOOL) {
          const unsigned d = db[oc * nwords + w];
          if (d) atomicOr(reinterpret_cast<unsigned int*>(A.out_data[oc]) + (a0 >> 5) + w, d);
          db[oc * nwords + w] = 0u;
        }
      }
      for (unsigned li = tid; li < total; li += PA_NT) {
        const int sl = list[li];
        tag[sl] = 0u;
        for (int w = 0; w < rw; w++) reinterpret_cast<uint64_t*>(trec + (size_t)sl * rb)[w] = A.ri.w[w];
      }
      if (tid == 0) s_total = 0u;  // every thread read it before the s_base barrier
      __syncthreads();
    }
  }
}

// First row of every partition of the m sorted keys (pstart[2^pb] = m), a binary search each: about 28
// dependent reads, all partitions at once. Counting the rows of 65,536 partitions in the encode pass cost
// a global atomic a row and the counts a trip through the host; reading the sorted keys for the places
// where the partition changes took 600 us for 200M rows, the searches 33 us.
template <int W>
__global__ void __launch_bounds__(ST_NT) k_part_starts(const unsigned long long* __restrict__ keys, uint64_t cap, int64_t m,
                                                       int pb, unsigned long long* __restrict__ pstart) {
  const long long q = (long long)blockIdx.x * ST_NT + threadIdx.x;
  if (q > (1LL << pb)) return;
  int64_t lo = 0, hi = m;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    PKey<W> k;
#pragma unroll
    for (int w = 0; w < W; w++) k.w[w] = keys[(uint64_t)w * cap + mid];
    if ((long long)(part_hash<W>(k) >> (64 - pb)) < q) lo = mid + 1;
    else hi = mid;
  }
  pstart[q] = (unsigned long long)lo;
}

// dense groups of the run-time compiled partitioned aggregation (packed keys, global-layout
// records) into the output columns, group g into output row g
struct PartFinParams {
  ReduceParams R;
  const unsigned long long* gkeys;  // word-major, stride gcap
  const uint8_t* grecs;
  uint64_t gcap;
};

template <int W>
__global__ void __launch_bounds__(ST_NT) k_part_finalize(const __grid_constant__ PartFinParams F) {
  const int64_t ng = (int64_t)*F.R.n_groups;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  // every lane of a warp runs the same number of iterations (warp-wide bit setting)
  const int64_t span = (ng + stride - 1) / stride * stride;
  for (int64_t g0 = (int64_t)blockIdx.x * blockDim.x; g0 < span; g0 += stride) {
    const int64_t g = g0 + threadIdx.x;
    const int64_t p_first = g0 + (threadIdx.x & ~31);
    const bool have = g < ng;
    PKey<W> k{};
    if (have)
      for (int w = 0; w < W; w++) k.w[w] = F.gkeys[(uint64_t)w * F.gcap + g];
    write_group<W, true>(F.R, g, p_first, have, k, have ? F.grecs + (uint64_t)g * F.R.q.rec_bytes : nullptr);
  }
}

// ---------------------------------------------------------------- dense groups in a wanted order
// A group-by whose result is then sorted by its keys: the dense groups' packed keys are rearranged
// into order keys (the sort columns' fields, most significant highest, then the other keys), sorted
// with the group numbers, and the records finalised in that order. A group is one contiguous record
// until then, so following the order costs two or three sectors a group; sorting the finished
// columns gathered one random 32-byte sector per group and column (49M groups of 9 columns:
// finalise 2.0 ms and gather 8.7 ms, 6.8 ms here), and needed the ranges and encode passes again.
struct GroupOrder {
  SortKeyLayout L;  // the packed keys' fields
  int null_off[PMB_MAX_KEYS];  // per key column, its fields in the order key (null_off -1: none)
  int data_off[PMB_MAX_KEYS];
  int desc[PMB_MAX_KEYS];
  int nulls_last[PMB_MAX_KEYS];
};

template <int W>
__device__ __forceinline__ unsigned long long key_field(const PKey<W>& k, int off, int bits) {
  if (bits == 0) return 0ULL;
  const int wi = off >> 6, sh = off & 63;
  unsigned long long v = k.w[wi] >> sh;
  if (W > 1 && sh + bits > 64 && wi + 1 < W) v |= k.w[wi + 1] << (64 - sh);
  return bits == 64 ? v : (v & ((1ULL << bits) - 1ULL));
}
template <int W>
__device__ __forceinline__ void put_field(PKey<W>& k, int off, unsigned long long v, int bits) {
  if (bits == 0) return;
  const int wi = off >> 6, sh = off & 63;
  k.w[wi] |= v << sh;
  if (W > 1 && sh + bits > 64 && wi + 1 < W) k.w[wi + 1] |= v >> (64 - sh);
}
__device__ __forceinline__ unsigned long long field_max(int bits) {
  return bits == 0 ? 0ULL : ~0ULL >> (64 - bits);
}

template <int W>
__global__ void __launch_bounds__(ST_NT) k_group_order(const __grid_constant__ GroupOrder O,
                                                       const unsigned long long* gkeys, uint64_t gcap, int64_t ng,
                                                       unsigned long long* okeys, uint64_t ocap, unsigned int* idx,
                                                       int passes, unsigned int* hist) {
  __shared__ unsigned int s_hist[MAX_PASSES * RADIX];
  for (int i = threadIdx.x; i < passes * RADIX; i += ST_NT) s_hist[i] = 0u;
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * ST_NT;
  for (int64_t g = (int64_t)blockIdx.x * ST_NT + threadIdx.x; g < ng; g += stride) {
    PKey<W> k, o;
    for (int w = 0; w < W; w++) {
      k.w[w] = gkeys[(uint64_t)w * gcap + g];
      o.w[w] = 0ULL;
    }
    for (int c = 0; c < O.L.n_keys; c++) {
      const bool null = O.L.null_off[c] >= 0 && key_field<W>(k, O.L.null_off[c], 1) != 0;
      if (O.null_off[c] >= 0) put_field<W>(o, O.null_off[c], null == (O.nulls_last[c] != 0) ? 1ULL : 0ULL, 1);
      if (null) continue;
      const unsigned long long v = key_field<W>(k, O.L.data_off[c], O.L.data_bits[c]);
      put_field<W>(o, O.data_off[c], O.desc[c] ? field_max(O.L.data_bits[c]) - v : v, O.L.data_bits[c]);
    }
    for (int w = 0; w < W; w++) okeys[(uint64_t)w * ocap + g] = o.w[w];
    idx[g] = (unsigned)g;
    for (int p = 0; p < passes; p++) atomicAdd(&s_hist[p * RADIX + digit_of<W>(o, 8 * p)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * RADIX; i += ST_NT) {
    const unsigned v = s_hist[i];
    if (v) atomicAdd(&hist[i], v);
  }
}

// output rows 0 .. m-1 = the groups at positions start .. start + m - 1 of the order
template <int W>
__global__ void __launch_bounds__(ST_NT) k_ordered_finalize(const __grid_constant__ PartFinParams F,
                                                            const __grid_constant__ GroupOrder O,
                                                            const unsigned long long* okeys, const unsigned int* idx,
                                                            int64_t start, int64_t m, const unsigned int* status) {
  if (status && (*status & PMB_ST_TIMEOUT)) return;  // the sort gave up: idx need not be an order
  // a warp's 32 records come into shared memory word by word, all lanes on the same few records, so
  // that every sector of a record is fetched once and all loads are in flight together (a lane walking
  // its own record took 6.8 ms for 49M groups, 1.1 TB/s)
  extern __shared__ __align__(16) unsigned long long s_rec[];
  const int lane = threadIdx.x & 31, rw = F.R.q.rec_bytes / 8;
  unsigned long long* mine = s_rec + (size_t)(threadIdx.x / 32) * 32 * rw;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  // every lane of a warp runs the same number of iterations (warp-wide bit setting)
  const int64_t span = (m + stride - 1) / stride * stride;
  for (int64_t p0 = (int64_t)blockIdx.x * blockDim.x; p0 < span; p0 += stride) {
    const int64_t p = p0 + threadIdx.x;
    const bool have = p < m;
    PKey<W> k{}, o{};
    const uint8_t* rec = nullptr;
    const unsigned g = have ? idx[start + p] : 0u;
    {
      int r = 0, c = lane;  // word c of record r
      while (c >= rw) {
        c -= rw;
        r++;
      }
      __syncwarp();  // the warp's reads of the previous records are done
      for (int w = 0; w < rw; w++) {
        const unsigned gr = __shfl_sync(0xffffffffu, g, r & 31);
        mine[w * 32 + lane] = *(reinterpret_cast<const unsigned long long*>(F.grecs + (uint64_t)gr * F.R.q.rec_bytes) + c);
        c += 32;
        while (c >= rw) {
          c -= rw;
          r++;
        }
      }
      __syncwarp();
    }
    if (have) {
      rec = reinterpret_cast<const uint8_t*>(mine + lane * rw);
      // one-word keys: the packed key back from the sorted order key (read in sequence); two-word
      // order keys are not sorted whole, the group's own packed key is fetched
      for (int w = 0; w < W; w++) (W == 1 ? o : k).w[w] = W == 1 ? okeys[start + p] : F.gkeys[(uint64_t)w * F.gcap + g];
      for (int c = 0; W == 1 && c < O.L.n_keys; c++) {
        const bool null = O.null_off[c] >= 0 && (key_field<W>(o, O.null_off[c], 1) != 0) == (O.nulls_last[c] != 0);
        if (null) {
          put_field<W>(k, O.L.null_off[c], 1ULL, 1);
          continue;
        }
        const unsigned long long v = key_field<W>(o, O.data_off[c], O.L.data_bits[c]);
        put_field<W>(k, O.L.data_off[c], O.desc[c] ? field_max(O.L.data_bits[c]) - v : v, O.L.data_bits[c]);
      }
    }
    write_group<W, true>(F.R, p, p0 + (threadIdx.x & ~31), have, k, rec);
  }
}

// whether the order names key columns only, each once (then the groups' packed keys decide it)
bool ordered_by_keys(const CompiledQuery& cq, const SortKeyLayout& L) {
  const pmb_sort_spec* s = cq.order;
  if (!s || !s->by || s->n_by < 1 || s->n_by > L.n_keys) return false;
  unsigned seen = 0;
  for (int i = 0; i < s->n_by; i++) {
    const int c = s->by[i];
    if (c < 0 || c >= L.n_keys || ((seen >> c) & 1u)) return false;
    if (pmb_is_float(L.dtype[c])) return false;  // packed as raw bits, which do not order
    seen |= 1u << c;
  }
  return !(s->drop_nulls && L.null_off[s->by[0]] >= 0);
}

template <int W>
int ordered_finalize(pmb_handle* h, const CompiledQuery& cq, const PartFinParams& F, int64_t ng, int64_t* rows) {
  const pmb_sort_spec& s = *cq.order;
  GroupOrder O;
  memset(&O, 0, sizeof(O));
  O.L = F.R.L;
  const int nk = O.L.n_keys;
  // fields from the least significant up: the keys the order does not name, then its columns backwards
  std::vector<int> cols;
  for (int c = 0; c < nk; c++) {
    bool named = false;
    for (int i = 0; i < s.n_by; i++) named |= s.by[i] == c;
    if (!named) cols.push_back(c);
  }
  for (int i = s.n_by - 1; i >= 0; i--) {
    cols.push_back(s.by[i]);
    O.desc[s.by[i]] = s.descending && s.descending[i];
    O.nulls_last[s.by[i]] = s.nulls_last && s.nulls_last[i];
  }
  int off = 0;
  for (int c : cols) {
    O.data_off[c] = off;
    off += O.L.data_bits[c];
    O.null_off[c] = O.L.null_off[c] >= 0 ? off : -1;
    off += O.L.null_off[c] >= 0;
  }
  const int passes = (off + 7) / 8;
  const uint64_t ocap = (uint64_t)ng;
  unsigned long long* k0 = (unsigned long long*)pmb_ws_alloc(h, (size_t)W * ng * 8 + 16);
  unsigned long long* k1 = (unsigned long long*)pmb_ws_alloc(h, (size_t)W * ng * 8 + 16);
  unsigned int* i0 = (unsigned int*)pmb_ws_alloc(h, (size_t)ng * 4 + 16);
  unsigned int* i1 = (unsigned int*)pmb_ws_alloc(h, (size_t)ng * 4 + 16);
  unsigned int* hist = (unsigned int*)pmb_ws_alloc(h, (size_t)MAX_PASSES * RADIX * 4);
  if (!k0 || !k1 || !i0 || !i1 || !hist) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (group order)");
  PMB_CUDA(h, cudaMemsetAsync(hist, 0, (size_t)MAX_PASSES * RADIX * 4, h->stream));
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((ng + ST_NT - 1) / ST_NT, (int64_t)h->sm_count * 8));
  pmb_kernel_begin(h, "group_order");
  k_group_order<W><<<blocks, ST_NT, 0, h->stream>>>(O, F.gkeys, F.gcap, ng, k0, ocap, i0, passes, hist);
  pmb_kernel_end(h);
  PMB_CUDA(h, cudaGetLastError());
  std::vector<unsigned int> hh;
  if (ng > PMB_SORT_NO_READBACK && passes > 0) {
    PMB_CUDA(h, cudaMemcpyAsync(h->pinned, hist, (size_t)passes * RADIX * 4, cudaMemcpyDeviceToHost, h->stream));
    PMB_CUDA(h, cudaStreamSynchronize(h->stream));
    hh.assign((const unsigned int*)h->pinned, (const unsigned int*)h->pinned + (size_t)passes * RADIX);
  }
  const int rc = pmb_sort_pairs(h, W, &k0, &k1, &i0, &i1, ocap, ng, passes, hist, hh.empty() ? nullptr : hh.data(), false,
                                &h->sort_status);
  if (rc) return rc;
  const int64_t start = s.offset >= 0 ? std::min<int64_t>(s.offset, ng) : std::max<int64_t>(0, ng + s.offset);
  const int64_t m = s.limit < 0 ? ng - start : std::min<int64_t>(s.limit, ng - start);
  if (m > 0) {
    const int fb = (int)std::max<int64_t>(1, std::min<int64_t>((m + ST_NT - 1) / ST_NT, (int64_t)h->sm_count * 16));
    pmb_kernel_begin(h, "ordered_finalize");
    const size_t fsmem = (size_t)ST_NT * F.R.q.rec_bytes;
    PMB_CUDA(h, cudaFuncSetAttribute(k_ordered_finalize<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fsmem));
    k_ordered_finalize<W><<<fb, ST_NT, fsmem, h->stream>>>(F, O, k0, i0, start, m, h->sort_status);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
  }
  *rows = m;
  return PMB_OK;
}

// the per-thread stage of k_part_agg: the aggregated columns' values (widest first, each aligned
// to its size), then one validity byte per nullable column; returns its bytes (a multiple of 8)
static int pa_stage(const DQuery& q, unsigned* used, int32_t* sdoff, int32_t* svoff) {
  *used = 0;
  for (int f = 0; f < q.n_fields; f++)
    if (q.field[f].kind != F_LEN) *used |= 1u << q.field[f].col;
  int off = 0;
  for (int e = 8; e >= 1; e /= 2)
    for (int c = 0; c < q.n_cols; c++)
      if (((*used >> c) & 1u) && std::max<int>(q.col[c].elem, 1) == e) {
        sdoff[c] = off;
        off += e;
      }
  for (int c = 0; c < q.n_cols; c++)
    if (((*used >> c) & 1u) && q.col[c].valid) svoff[c] = off++;
  return (off + 7) & ~7;
}

// run_part_agg's answer when the sort strategy should reduce its segments itself
constexpr int kSegReduce = -77;

// work-item boundaries for aggregating sorted rows in shared-memory tables: chunk c starts at the
// first segment start at or after c * chunk (m at the end), so no group is cut
__global__ void k_chunk_bounds(const unsigned int* __restrict__ starts, unsigned long long ng, int64_t m, int64_t chunk,
                               int64_t n_chunks, unsigned long long* __restrict__ out) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c > n_chunks) return;
  const int64_t x = c * chunk;
  if (c == n_chunks || x >= m) {
    out[c] = (unsigned long long)m;
    return;
  }
  unsigned long long lo = 0, hi = ng;
  while (lo < hi) {
    const unsigned long long mid = (lo + hi) >> 1;
    if ((int64_t)starts[mid] < x) lo = mid + 1;
    else hi = mid;
  }
  out[c] = lo < ng ? (unsigned long long)starts[lo] : (unsigned long long)m;
}

// float sums that left their fixed-point range: widen to the largest exponent seen (the sorted
// order does not depend on it); true when a column must switch to double-double instead
static bool widen_fx(CompiledQuery& cq, const unsigned int* st) {
  DQuery& q = cq.dq;
  for (int i = 0; i < q.n_fields; i++) {
    DField& f = q.field[i];
    if (f.kind != F_SUM_FX || st[4 + f.fx_slot] == 0) continue;
    const int e = (int)st[4 + f.fx_slot] - 1022 + 1;
    if (e > q.fx_e[f.fx_slot]) {
      f.fx = (int16_t)(f.fx - (e - q.fx_e[f.fx_slot]));
      q.fx_e[f.fx_slot] = (int16_t)e;
    }
  }
  return pmb_fx_to_dd(cq);
}

template <int W>
int run_sort(pmb_handle* h, CompiledQuery& cq, const SortKeyLayout& L, pmb_result* r, int64_t part_groups);

// The values that the partition passes carry: per element its column (-1: the mask of validity bits, bit
// c, and Bool values, bit 16 + c), its bytes, where it is now and where the next pass puts it.
struct Payload {
  int n = 0;
  int col[PMB_MAX_COLS + 1];
  int elem[PMB_MAX_COLS + 1];
  const uint8_t* cur[PMB_MAX_COLS + 1];
  uint8_t* buf[2][PMB_MAX_COLS + 1];
  bool mask = false;
  int row_bytes = 0;
  // the aggregation that reads them, compiled before the passes: no other kernel can take over afterwards
  // (the passes move no row numbers)
  cudaKernel_t kernel = nullptr;
  JitPlan plan;
  int ctas = 1;
};

// Carrying pays where the gathers by row number miss L2: a random read costs a whole DRAM access (42 G/s
// on 1.6 GB, whatever its width or cache hint), 400M of them 9.5 of the aggregation's 11.5 ms for 200M
// rows with two value columns. Every pass moves the values instead. Up to PAY_BYTES a row, and from
// PAY_MIN bytes of value columns (about half of L2) on.
constexpr int PAY_BYTES = 32;
constexpr int64_t PAY_MIN = 64LL << 20;
bool plan_payload(const DQuery& q, Payload* p) {
  unsigned used = 0;
  for (int f = 0; f < q.n_fields; f++)
    if (q.field[f].kind != F_LEN) used |= 1u << q.field[f].col;
  auto add = [&](int col, int elem) {
    p->col[p->n] = col;
    p->elem[p->n++] = elem;
    p->row_bytes += elem;
  };
  for (int c = 0; c < q.n_cols; c++) {
    if (!((used >> c) & 1u)) continue;
    if (q.col[c].elem) add(c, q.col[c].elem == 8 ? 8 : 4);
    p->mask |= q.col[c].valid != nullptr || q.col[c].elem == 0;
  }
  if (p->mask) add(-1, 4);
  return p->n > 0 && p->row_bytes <= PAY_BYTES && q.n_rows * p->row_bytes >= PAY_MIN;
}

// CTAs an SM of the run-time compiled aggregation: two where a row's carried values fit the 32 registers of
// their threads (pmb_jit_part.cuh has both sides' times), else one
inline int part_ctas(int W, const Payload& pay) { return W == 1 && pay.row_bytes <= 24 ? 2 : 1; }

// Partitions per work item: runs of them with half a table of rows on average (rows bound the groups; the
// hash spreads them, so a run stays far from the whole table), at least one each. Not by the rows of a
// partition rounded down: 1.9 of them as 1 would make runs of 0.95 of a table.
inline int part_run(int slots, int64_t n_parts, int64_t m) {
  return (int)std::max<int64_t>(1, std::min<int64_t>(n_parts, slots / 2 * n_parts / std::max<int64_t>(1, m)));
}

// the aggregation of the partitioned strategy over keys / row indices sorted by partition
template <int W>
int run_part_agg(pmb_handle* h, CompiledQuery& cq, const SortKeyLayout& L, pmb_result* r, const unsigned long long* keys,
                 const unsigned int* idx, uint64_t cap, int64_t m, const unsigned long long* pstart, int64_t n_parts,
                 int run, int slots, int64_t groups, unsigned long long* ctr, unsigned int* status,
                 int strategy = PMB_STRATEGY_PARTITIONED, const Payload* pay = nullptr) {
  DQuery& q = cq.dq;
  const int n_out = q.n_keys + q.n_aggs;
  PartParams A;
  memset(&A, 0, sizeof(A));
  for (size_t w = 0; w < cq.rec_init.size() && w < 48; w++) A.ri.w[w] = cq.rec_init[w];
  A.L = L;
  A.keys = keys;
  A.cap = cap;
  A.idx = idx;
  A.m = m;
  A.pstart = pstart;
  A.n_parts = n_parts;
  A.run = run;
  A.n_items = (n_parts + run - 1) / run;
  A.slots = slots;
  A.n_out = n_out;
  A.stage_bytes = pa_stage(q, &A.used, A.sdoff, A.svoff);
  for (int c = 0; c < q.n_cols; c++)
    if ((A.used >> c) & 1u) A.ucol[A.n_used++] = c;
  A.ticket = ctr + 1;
  A.n_groups = ctr + 2;
  A.status = status;
  const size_t smem = pa_layout(slots, W, q.rec_bytes, n_out, A.stage_bytes).bytes;
  PMB_CUDA(h, cudaFuncSetAttribute(k_part_agg<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  int64_t out_cap = std::min<int64_t>(std::max<int64_t>(m, 1), 2 * groups + 65536);
  // should the smaller tables of two CTAs not hold an item's groups, one CTA of the same kernel with the
  // whole table follows
  int ctas = pay ? pay->ctas : 1;
  for (int attempt = 0;; attempt++) {
    if (attempt >= 6) return pmb_fail(h, PMB_E_CUDA, "partitioned strategy did not converge");
    const WsMark mark = pmb_ws_mark(h);
    const size_t vbytes = (size_t)((out_cap + 31) / 32 * 4) + 16;
    for (int c = 0; c < n_out; c++) {
      const int dt = r->columns[c].dtype;
      const size_t dbytes = dt == PMB_BOOL ? vbytes : (size_t)out_cap * pmb_dtype_bytes(dt) + 16;
      A.out_data[c] = (uint8_t*)pmb_ws_alloc(h, dbytes);
      A.out_valid[c] = (uint8_t*)pmb_ws_alloc(h, vbytes);
      if (!A.out_data[c] || !A.out_valid[c]) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (outputs)");
      PMB_CUDA(h, cudaMemsetAsync(A.out_valid[c], 0, vbytes, h->stream));
      if (dt == PMB_BOOL) PMB_CUDA(h, cudaMemsetAsync(A.out_data[c], 0, vbytes, h->stream));
    }
    A.q = q;
    A.out_cap = out_cap;
    PMB_CUDA(h, cudaMemsetAsync(ctr + 1, 0, 16, h->stream));
    // (the first attempt finds the status of the passes, and a wait that gave up there ends it)
    if (attempt > 0) PMB_CUDA(h, cudaMemsetAsync(status, 0, 64, h->stream));
    unsigned long long ng = 0;
    unsigned int st[12] = {0};
    // the run-time compiled aggregation writes dense groups that a prebuilt kernel finalises;
    // without NVRTC (or for a signature it cannot take) the prebuilt kernel does both
    JitPlan J;
    cudaKernel_t jk = nullptr;
    if (pay) {
      J = pay->plan;
      jk = pay->kernel;
    } else if (m > 0 && pmb_jit_enabled(1LL << 40) && pmb_jit_part_kernel(h, cq, W, L.bits < 64, false, 1, &J, &jk) != PMB_OK) {
      jk = nullptr;  // the prebuilt kernel instead (the compile error stays readable in pmb_last_error)
    }
    unsigned long long* gkeys = nullptr;
    uint8_t* grecs = nullptr;
    if (jk) {
      gkeys = (unsigned long long*)pmb_ws_alloc(h, (size_t)W * out_cap * 8 + 16);
      grecs = (uint8_t*)pmb_ws_alloc(h, (size_t)out_cap * q.rec_bytes + 16);
      if (!gkeys || !grecs) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (groups)");
    }
    if (m > 0) {
      const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(A.n_items, h->sm_count));
      if (jk) {
        int jslots = slots, jrun = run;
        if (ctas == 2) {
          jslots = std::min(slots, (h->max_smem_optin / 2 - 1536) / (4 + 8 * W + J.srec + 2) & ~7);
          jrun = part_run(jslots, n_parts, m);
        }
        const int64_t jitems = (n_parts + jrun - 1) / jrun;
        JPartH JA;
        memset(&JA, 0, sizeof(JA));
        for (int c = 0; c < q.n_cols; c++) {
          JA.qp.col_data[c] = q.col[c].data;
          JA.qp.col_valid[c] = q.col[c].valid;
        }
        JA.qp.n_rows = q.n_rows;
        JA.qp.status = status;
        for (int f = 0; f < q.n_fields; f++)
          if (q.field[f].kind == F_SUM_FX) {
            JA.qp.fx[q.field[f].fx_slot] = q.field[f].fx;
            JA.qp.fx_e[q.field[f].fx_slot] = q.fx_e[q.field[f].fx_slot];
          }
        JA.keys = keys;
        JA.kcap = cap;
        JA.idx = idx;
        JA.pstart = A.pstart;
        JA.n_parts = n_parts;
        JA.run = jrun;
        JA.n_items = jitems;
        JA.slots = jslots;
        // More than the table's longest run of full slots, about ln(slots) / (a - 1 - ln(a)) of them at a load of a,
        // up to 0.85 (items have half a table on average, those of sorted rows at most 0.7 and one group). With
        // every slot tried, the rows of overflowing partitions took 33 ms (4.5M rows, 2.2M kept in 256 partitions by
        // a hint of 5000 groups), 8.7 ms so.
        JA.probes = (unsigned)std::max(256, jslots / 4);
        JA.ticket = A.ticket;
        JA.gkeys = gkeys;
        JA.grecs = grecs;
        JA.gcap = (unsigned long long)out_cap;
        JA.n_groups = A.n_groups;
        if (pay) {
          for (int e = 0; e < pay->n; e++)
            if (pay->col[e] < 0) JA.paymask = (const unsigned int*)pay->cur[e];
            else JA.pay[pay->col[e]] = pay->cur[e];
        }
        const size_t jsmem = (((size_t)jslots * 4 + 15) & ~(size_t)15) + (size_t)jslots * (8 * W + J.srec + 2);
        PMB_CUDA(h, cudaFuncSetAttribute((const void*)jk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)jsmem));
        void* args[] = {&JA};
        pmb_kernel_begin(h, "part_agg");
        PMB_CUDA(h, cudaLaunchKernel((const void*)jk, dim3((unsigned)std::max<int64_t>(1, std::min<int64_t>(jitems, (int64_t)h->sm_count * ctas))), dim3(J.nt), args, jsmem, h->stream));
        pmb_kernel_end(h);
      } else {
        pmb_kernel_begin(h, "part_agg");
        k_part_agg<W><<<grid, PA_NT, smem, h->stream>>>(A);
        pmb_kernel_end(h);
        PMB_CUDA(h, cudaGetLastError());
      }
      PMB_CUDA(h, cudaMemcpyAsync(&ng, ctr + 2, 8, cudaMemcpyDeviceToHost, h->stream));
      PMB_CUDA(h, cudaMemcpyAsync(st, status, sizeof(st), cudaMemcpyDeviceToHost, h->stream));
      PMB_CUDA(h, cudaStreamSynchronize(h->stream));
      if (jk && !(st[0] & (PMB_ST_TIMEOUT | PMB_ST_FXRANGE | PMB_ST_OVERFLOW)) && ng > 0) {
        PartFinParams F;
        memset(&F, 0, sizeof(F));
        F.R.q = q;
        F.R.L = L;
        F.R.n_groups = A.n_groups;
        for (int c = 0; c < n_out; c++) {
          F.R.out_data[c] = A.out_data[c];
          F.R.out_valid[c] = A.out_valid[c];
        }
        F.gkeys = gkeys;
        F.grecs = grecs;
        F.gcap = (uint64_t)out_cap;
        if (ordered_by_keys(cq, L)) {
          const WsMark order_mark = pmb_ws_mark(h);
          int64_t rows = 0;
          const int orc = ordered_finalize<W>(h, cq, F, (int64_t)ng, &rows);
          if (orc && orc != PMB_E_OOM) return orc;
          if (orc) {  // the order keys do not fit: the columns are sorted, whose keys may be narrower
            pmb_ws_release(h, order_mark);
          } else {
            ng = (unsigned long long)rows;
            cq.ordered = true;
          }
        }
        if (!cq.ordered) {
          const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)ng + ST_NT - 1) / ST_NT, (int64_t)h->sm_count * 16));
          pmb_kernel_begin(h, "part_finalize");
          k_part_finalize<W><<<blocks, ST_NT, 0, h->stream>>>(F);
          pmb_kernel_end(h);
          PMB_CUDA(h, cudaGetLastError());
        }
      }
    }
    if (st[0] & PMB_ST_TIMEOUT) return pmb_fail(h, PMB_E_TIMEOUT, "a bounded device wait timed out (partitioned)");
    if (st[0] & PMB_ST_FXRANGE) {
      if (widen_fx(cq, st)) return PMB_RETRY_DD;
      pmb_ws_release(h, mark);
      continue;
    }
    if (st[0] & PMB_ST_OVERFLOW) {
      pmb_ws_release(h, mark);
      if ((int64_t)ng > out_cap) {  // more groups than output rows: the exact upper bound next
        out_cap = std::max<int64_t>(m, 1);
        continue;
      }
      if (ctas > 1) {
        ctas = 1;
        continue;
      }
      // a partition had more groups than its table: the sort strategy instead (the sort's own
      // segment reduce when the caller is the sort)
      if (strategy == PMB_STRATEGY_SORT) return kSegReduce;
      PMB_CUDA(h, cudaMemsetAsync(ctr, 0, 64, h->stream));
      return run_sort<W>(h, cq, L, r, 0);
    }
    r->n_groups = (int64_t)ng;
    r->capacity = out_cap;
    r->strategy_used = strategy;
    for (int c = 0; c < n_out; c++) {
      r->columns[c].data = A.out_data[c];
      r->columns[c].validity = A.out_valid[c];
    }
    return PMB_OK;
  }
}

template <int W>
int run_sort(pmb_handle* h, CompiledQuery& cq, const SortKeyLayout& L, pmb_result* r, int64_t part_groups) {
  DQuery& q = cq.dq;
  const int64_t n = q.n_rows;
  const int n_out = q.n_keys + q.n_aggs;
  // partitioned strategy: the largest shared table that fits, and 2^8 or 2^16 partitions so that
  // a partition holds about a third of a table
  int pb = 0, slots = 0;
  if (part_groups > 0) {
    unsigned used;
    int32_t sd[PMB_MAX_COLS], sv[PMB_MAX_COLS];
    const int stage = pa_stage(q, &used, sd, sv);
    for (slots = 4096; slots >= 256; slots /= 2)
      if (pa_layout(slots, W, q.rec_bytes, n_out, stage).bytes + 2048 <= (size_t)h->max_smem_optin) break;
    if (slots < 256) return pmb_fail(h, PMB_E_UNSUPPORTED, "partitioned strategy: group record too large");
    // twice the estimate: an undersized partition count overflows tables (and falls back to the
    // sort), an oversized one costs one more pass
    pb = 2 * part_groups * 3 / slots + 1 <= 256 ? 8 : 16;
  }
  const int passes = part_groups > 0 ? pb / 8 : std::max(0, (L.bits + 7) / 8);
  const uint64_t cap = (uint64_t)n;
  unsigned long long* k0 = (unsigned long long*)pmb_ws_alloc(h, (size_t)W * cap * 8 + 16);
  unsigned long long* k1 = (unsigned long long*)pmb_ws_alloc(h, (size_t)W * cap * 8 + 16);
  unsigned int* i0 = (unsigned int*)pmb_ws_alloc(h, (size_t)cap * 4 + 16);
  unsigned int* i1 = (unsigned int*)pmb_ws_alloc(h, (size_t)cap * 4 + 16);
  unsigned int* hist = (unsigned int*)pmb_ws_alloc(h, (size_t)MAX_PASSES * RADIX * 4);
  const int64_t n_parts = part_groups > 0 ? (int64_t)1 << pb : 0;
  unsigned long long* pstart = n_parts ? (unsigned long long*)pmb_ws_alloc(h, (size_t)(n_parts + 1) * 8) : nullptr;
  if (n_parts && !pstart) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (partition offsets)");
  unsigned long long* ctr = (unsigned long long*)pmb_ws_alloc(h, 64);  // kept, ticket, n_groups, big_n
  unsigned int* status = (unsigned int*)pmb_ws_alloc(h, 64);
  const int64_t max_tiles = (n + ST_TILE - 1) / ST_TILE;
  const int64_t max_ptiles = (n + PassShape<W>::TILE - 1) / PassShape<W>::TILE;  // pass tiles
  unsigned long long* lb = (unsigned long long*)pmb_ws_alloc(
      h, (size_t)std::max<int64_t>({max_tiles, max_ptiles * RADIX, 1}) * 8);
  if (!k0 || !k1 || !i0 || !i1 || !hist || !ctr || !status || !lb)
    return pmb_fail(h, PMB_E_OOM, "workspace exhausted (sort buffers)");
  PMB_CUDA(h, cudaMemsetAsync(hist, 0, (size_t)MAX_PASSES * RADIX * 4, h->stream));
  PMB_CUDA(h, cudaMemsetAsync(ctr, 0, 64, h->stream));
  PMB_CUDA(h, cudaMemsetAsync(status, 0, 64, h->stream));
  {
    EncodeParams E;
    memset(&E, 0, sizeof(E));
    E.q = q;
    E.L = L;
    E.passes = passes;
    E.n = n;
    E.keys = k0;
    E.cap = cap;
    E.idx = i0;
    E.lb = lb;
    E.ticket = ctr + 1;
    E.kept = ctr;
    E.hist = hist;
    E.status = status;
    E.hashed = part_groups > 0;
    E.shift0 = part_groups > 0 ? 64 - pb : 0;
    PMB_CUDA(h, cudaMemsetAsync(lb, 0, (size_t)std::max<int64_t>(max_tiles, 1) * 8, h->stream));
    pmb_kernel_begin(h, "sort_encode");
    const auto encode = q.prog.n_ops > 0 ? k_sort_encode<W, true> : k_sort_encode<W, false>;
    encode<<<(unsigned)std::max<int64_t>(max_tiles, 1), ST_NT, 0, h->stream>>>(E);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
  }
  std::vector<unsigned int> hh((size_t)std::max(passes, 1) * RADIX);
  PMB_CUDA(h, cudaMemcpyAsync(h->pinned, ctr, 8, cudaMemcpyDeviceToHost, h->stream));
  PMB_CUDA(h, cudaMemcpyAsync(h->pinned + 8, status, 4, cudaMemcpyDeviceToHost, h->stream));
  if (passes) PMB_CUDA(h, cudaMemcpyAsync(h->pinned + 64, hist, (size_t)passes * RADIX * 4, cudaMemcpyDeviceToHost, h->stream));
  PMB_CUDA(h, cudaStreamSynchronize(h->stream));
  const unsigned long long kept = *(unsigned long long*)h->pinned;
  const unsigned int st0 = *(unsigned int*)(h->pinned + 8);
  memcpy(hh.data(), h->pinned + 64, (size_t)passes * RADIX * 4);
  if (st0 & PMB_ST_TIMEOUT) return pmb_fail(h, PMB_E_TIMEOUT, "a bounded device wait timed out (sort)");
  const int64_t m = (int64_t)kept;
  // LSD passes over the digits that are not the same for every key
  const int64_t tiles = (m + ST_TILE - 1) / ST_TILE;
  const int64_t ptiles = (m + PassShape<W>::TILE - 1) / PassShape<W>::TILE;
  constexpr size_t pass_smem = PassShape<W>::SMEM;
  // the partition passes carry the aggregated values when the run-time compiled aggregation can take
  // them and the buffers fit
  Payload pay;
  bool carry = part_groups > 0 && m > 1 && !h->no_carry && plan_payload(q, &pay) && pmb_jit_enabled(1LL << 40);
  if (carry) {
    const std::string keep_err = h->err;
    pay.ctas = part_ctas(W, pay);
    carry = pmb_jit_part_kernel(h, cq, W, L.bits < 64, true, pay.ctas, &pay.plan, &pay.kernel) == PMB_OK;
    h->carried = carry;
    const WsMark mark = pmb_ws_mark(h);
    for (int b = 0; carry && b < passes; b++)
      for (int e = 0; carry && e < pay.n; e++) {
        pay.buf[b][e] = (uint8_t*)pmb_ws_alloc(h, (size_t)m * pay.elem[e] + 16);
        carry = pay.buf[b][e] != nullptr;
      }
    if (!carry) pmb_ws_release(h, mark);
    h->err = keep_err;
  }
  const auto pass = part_groups > 0 ? k_sort_pass<W, true> : k_sort_pass<W, false>;
  PMB_CUDA(h, cudaFuncSetAttribute(pass, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pass_smem));
  if (h->fault_wait) PMB_CUDA(h, cudaMemsetAsync(status, PMB_ST_TIMEOUT, 1, h->stream));
  for (int p = 0; p < passes && m > 1; p++) {
    bool constant = false;
    for (int d = 0; d < RADIX; d++) constant |= hh[(size_t)p * RADIX + d] == (unsigned)m;
    if (constant && !carry) continue;
    PassParams P;
    P.n_pay = 0;
    P.kin = k0;
    P.kout = k1;
    P.iin = i0;
    P.iout = i1;
    P.cap = cap;
    P.n = m;
    P.shift = (part_groups > 0 ? 64 - pb : 0) + 8 * p;
    P.hist = hist + (size_t)p * RADIX;
    P.lb = lb;
    P.ticket = ctr + 1;
    P.status = status;
    PMB_CUDA(h, cudaMemsetAsync(lb, 0, (size_t)ptiles * RADIX * 8, h->stream));
    PMB_CUDA(h, cudaMemsetAsync(ctr + 1, 0, 8, h->stream));
    pmb_kernel_begin(h, "sort_pass");
    if (carry) {
      P.n_pay = pay.n;
      P.n_mask = 0;
      for (int e = 0; e < pay.n; e++) {
        const int c = pay.col[e];
        P.pay_elem[e] = pay.elem[e];
        P.pay_src[e] = c >= 0 ? q.col[c].elem : 0;
        P.pay_in[e] = p > 0 ? pay.cur[e] : c >= 0 ? q.col[c].data : nullptr;
        P.pay_out[e] = pay.buf[p][e];
        pay.cur[e] = pay.buf[p][e];
      }
      unsigned used = 0;
      for (int f = 0; f < q.n_fields; f++)
        if (q.field[f].kind != F_LEN) used |= 1u << q.field[f].col;
      for (int c = 0; c < q.n_cols; c++) {
        if (!((used >> c) & 1u)) continue;
        if (q.col[c].valid) {
          P.mask_bits[P.n_mask] = q.col[c].valid;
          P.mask_pos[P.n_mask++] = c;
        }
        if (q.col[c].elem == 0) {
          P.mask_bits[P.n_mask] = q.col[c].data;
          P.mask_pos[P.n_mask++] = 16 + c;
        }
      }
      const auto moving = p == 0 ? k_sort_pass<W, true, PAY_FIRST> : k_sort_pass<W, true, PAY_NEXT>;
      PMB_CUDA(h, cudaFuncSetAttribute(moving, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pass_smem));
      moving<<<(unsigned)ptiles, PassShape<W>::NT, pass_smem, h->stream>>>(P);
    } else {
      pass<<<(unsigned)ptiles, PassShape<W>::NT, pass_smem, h->stream>>>(P);
    }
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
    std::swap(k0, k1);
    std::swap(i0, i1);
  }
  if (part_groups > 0) {
    pmb_kernel_begin(h, "part_starts");
    k_part_starts<W><<<(unsigned)(n_parts / ST_NT + 1), ST_NT, 0, h->stream>>>(k0, cap, m, pb, pstart);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
    return run_part_agg<W>(h, cq, L, r, k0, i0, cap, m, pstart, n_parts, part_run(slots, n_parts, m), slots, part_groups, ctr, status,
                           PMB_STRATEGY_PARTITIONED, carry ? &pay : nullptr);
  }
  // segment starts
  unsigned int* starts = (unsigned int*)pmb_ws_alloc(h, (size_t)(m + 2) * 4);
  if (!starts) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (segment starts)");
  unsigned long long ng = 0;
  if (m > 0) {
    StartsParams S;
    S.keys = k0;
    S.cap = cap;
    S.n = m;
    S.starts = starts;
    S.lb = lb;
    S.ticket = ctr + 1;
    S.n_groups = ctr + 2;
    S.status = status;
    PMB_CUDA(h, cudaMemsetAsync(lb, 0, (size_t)tiles * 8, h->stream));
    PMB_CUDA(h, cudaMemsetAsync(ctr + 1, 0, 8, h->stream));
    pmb_kernel_begin(h, "seg_starts");
    k_seg_starts<W><<<(unsigned)tiles, ST_NT, 0, h->stream>>>(S);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
    unsigned int st = 0;
    PMB_CUDA(h, cudaMemcpyAsync(&ng, ctr + 2, 8, cudaMemcpyDeviceToHost, h->stream));
    PMB_CUDA(h, cudaMemcpyAsync(&st, status, 4, cudaMemcpyDeviceToHost, h->stream));
    PMB_CUDA(h, cudaStreamSynchronize(h->stream));
    if (st & PMB_ST_TIMEOUT) return pmb_fail(h, PMB_E_TIMEOUT, "a bounded device wait timed out (sort)");
  }
  // with the run-time compiler, the sorted rows are cut at segment starts into work items that fit
  // a shared-memory table, and the partitioned strategy's aggregation reduces them (values
  // gathered once per row, records in shared memory); otherwise thread-per-segment reduces below
  if (ng > 0 && pmb_jit_enabled(1LL << 40)) {
    unsigned used;
    int32_t sd[PMB_MAX_COLS], sv[PMB_MAX_COLS];
    const int stage = pa_stage(q, &used, sd, sv);
    int slots = 4096;
    for (; slots >= 256; slots /= 2)
      if (pa_layout(slots, W, q.rec_bytes, n_out, stage).bytes + 2048 <= (size_t)h->max_smem_optin) break;
    if (slots >= 256) {
      const int64_t chunk = (int64_t)(0.7 * slots);
      const int64_t n_chunks = (m + chunk - 1) / chunk;
      unsigned long long* bounds = (unsigned long long*)pmb_ws_alloc(h, (size_t)(n_chunks + 1) * 8);
      if (!bounds) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (segment chunks)");
      pmb_kernel_begin(h, "chunk_bounds");
      k_chunk_bounds<<<(unsigned)((n_chunks + 1 + 255) / 256), 256, 0, h->stream>>>(starts, ng, m, chunk, n_chunks, bounds);
      pmb_kernel_end(h);
      PMB_CUDA(h, cudaGetLastError());
      const WsMark mark = pmb_ws_mark(h);
      const int rc = run_part_agg<W>(h, cq, L, r, k0, i0, cap, m, bounds, n_chunks, 1, slots, (int64_t)ng, ctr, status,
                                     PMB_STRATEGY_SORT);
      if (rc != kSegReduce) return rc;
      pmb_ws_release(h, mark);
      PMB_CUDA(h, cudaMemcpyAsync(ctr + 2, &ng, 8, cudaMemcpyHostToDevice, h->stream));  // the group count again
    }
  }
  // outputs
  ReduceParams R;
  memset(&R, 0, sizeof(R));
  R.q = q;
  for (size_t w = 0; w < cq.rec_init.size() && w < 48; w++) R.ri.w[w] = cq.rec_init[w];
  R.L = L;
  R.cap = cap;
  R.idx = i0;
  R.starts = starts;
  R.n_groups = ctr + 2;
  R.big = (unsigned int*)pmb_ws_alloc(h, (size_t)(ng + 1) * 4);
  R.big_n = ctr + 3;
  R.status = status;
  if (!R.big) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (big groups)");
  const size_t vbytes = (size_t)((ng + 31) / 32 * 4) + 16;
  for (int c = 0; c < n_out; c++) {
    const int dt = r->columns[c].dtype;
    const size_t db = dt == PMB_BOOL ? vbytes : (size_t)ng * pmb_dtype_bytes(dt) + 16;
    R.out_data[c] = (uint8_t*)pmb_ws_alloc(h, db);
    R.out_valid[c] = (uint8_t*)pmb_ws_alloc(h, vbytes);
    if (!R.out_data[c] || !R.out_valid[c]) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (outputs)");
    PMB_CUDA(h, cudaMemsetAsync(R.out_valid[c], 0, vbytes, h->stream));
    if (dt == PMB_BOOL) PMB_CUDA(h, cudaMemsetAsync(R.out_data[c], 0, vbytes, h->stream));
  }
  for (int attempt = 0; ng > 0; attempt++) {
    R.keys = k0;
    PMB_CUDA(h, cudaMemsetAsync(ctr + 3, 0, 8, h->stream));
    PMB_CUDA(h, cudaMemsetAsync(status, 0, 64, h->stream));
    const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>(((int64_t)ng + ST_NT - 1) / ST_NT, (int64_t)h->sm_count * 16));
    pmb_kernel_begin(h, "seg_reduce");
    if (q.rec_bytes <= 96) k_seg_reduce<W, 12><<<blocks, ST_NT, 0, h->stream>>>(R);
    else if (q.rec_bytes <= 192) k_seg_reduce<W, 24><<<blocks, ST_NT, 0, h->stream>>>(R);
    else k_seg_reduce<W, 48><<<blocks, ST_NT, 0, h->stream>>>(R);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
    const size_t big_smem = (size_t)BIG_NT * q.rec_bytes;
    PMB_CUDA(h, cudaFuncSetAttribute(k_seg_reduce_big<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)big_smem));
    pmb_kernel_begin(h, "seg_reduce_big");
    k_seg_reduce_big<W><<<h->sm_count, BIG_NT, big_smem, h->stream>>>(R);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
    unsigned int st[12];
    PMB_CUDA(h, cudaMemcpyAsync(st, status, sizeof(st), cudaMemcpyDeviceToHost, h->stream));
    PMB_CUDA(h, cudaStreamSynchronize(h->stream));
    if (st[0] & PMB_ST_TIMEOUT) return pmb_fail(h, PMB_E_TIMEOUT, "a bounded device wait timed out (sort)");
    if (!(st[0] & PMB_ST_FXRANGE)) break;
    // a float sum left its fixed-point range: widen to the largest exponent seen; the sorted
    // order does not depend on it, so only the reduction runs again
    if (attempt >= 4) return pmb_fail(h, PMB_E_CUDA, "float-sum range did not converge");
    if (widen_fx(cq, st)) return PMB_RETRY_DD;
    R.q = q;
    for (int c = 0; c < n_out; c++) {
      PMB_CUDA(h, cudaMemsetAsync(R.out_valid[c], 0, vbytes, h->stream));
      if (r->columns[c].dtype == PMB_BOOL) PMB_CUDA(h, cudaMemsetAsync(R.out_data[c], 0, vbytes, h->stream));
    }
  }
  r->n_groups = (int64_t)ng;
  r->capacity = 0;
  r->strategy_used = PMB_STRATEGY_SORT;
  for (int c = 0; c < n_out; c++) {
    r->columns[c].data = R.out_data[c];
    r->columns[c].validity = R.out_valid[c];
  }
  return PMB_OK;
}

// the key columns as a layout (without fields)
void key_columns(const DQuery& q, SortKeyLayout& L) {
  memset(&L, 0, sizeof(L));
  L.n_keys = q.n_keys;
  for (int k = 0; k < q.n_keys; k++) {
    const DCol& C = q.col[q.key[k].col];
    L.col[k] = q.key[k].col;
    L.dtype[k] = C.dtype;
    L.elem[k] = C.elem;
    L.data[k] = C.data;
    L.valid[k] = C.valid;
  }
}

// cq.ranges from the key columns, unless an earlier step of the call has read them
int read_key_ranges(pmb_handle* h, CompiledQuery& cq, const SortKeyLayout& L) {
  if (cq.ranges.have) return PMB_OK;
  const int64_t n = cq.dq.n_rows;
  RangeOut* ro = (RangeOut*)pmb_ws_alloc(h, sizeof(RangeOut));
  if (!ro) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (key ranges)");
  PMB_CUDA(h, cudaMemsetAsync(ro, 0, sizeof(RangeOut), h->stream));
  PMB_CUDA(h, cudaMemsetAsync(ro->lo, 0xFF, sizeof(ro->lo), h->stream));
  const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + ST_NT - 1) / ST_NT, (int64_t)h->sm_count * 8));
  pmb_kernel_begin(h, "key_range");
  k_key_range<<<blocks, ST_NT, 0, h->stream>>>(L, n, ro);
  pmb_kernel_end(h);
  PMB_CUDA(h, cudaGetLastError());
  PMB_CUDA(h, cudaMemcpyAsync(h->pinned, ro, sizeof(RangeOut), cudaMemcpyDeviceToHost, h->stream));
  PMB_CUDA(h, cudaStreamSynchronize(h->stream));
  const RangeOut* got = reinterpret_cast<const RangeOut*>(h->pinned);
  memcpy(cq.ranges.lo, got->lo, sizeof(got->lo));
  memcpy(cq.ranges.hi, got->hi, sizeof(got->hi));
  memcpy(cq.ranges.nulls, got->nulls, sizeof(got->nulls));
  memcpy(cq.ranges.any, got->any, sizeof(got->any));
  cq.ranges.have = true;
  return PMB_OK;
}

}  // namespace

int pmb_groupby_sort(pmb_handle* h, CompiledQuery& cq, pmb_result* r, int64_t part_groups) {
  DQuery& q = cq.dq;
  if (q.n_rows > 0xFFFFFFF0LL) return pmb_fail(h, PMB_E_UNSUPPORTED, "sort strategy: more than 2^32 rows");
  if (q.rec_bytes > 384) return pmb_fail(h, PMB_E_UNSUPPORTED, "sort strategy: group record above 384 bytes");
  SortKeyLayout L;
  key_columns(q, L);
  const int rrc = read_key_ranges(h, cq, L);
  if (rrc) return rrc;
  const CompiledQuery::KeyRanges& got = cq.ranges;
  int off = 0;
  for (int k = 0; k < q.n_keys; k++) {
    L.null_off[k] = -1;
    if (got.nulls[k]) L.null_off[k] = off++;
    int bits = 0;
    if (got.any[k]) {
      L.lo[k] = got.lo[k];
      const unsigned long long span = got.hi[k] - got.lo[k];
      while (bits < 64 && (span >> bits) != 0) bits++;
    }
    L.data_off[k] = off;
    L.data_bits[k] = bits;
    off += bits;
  }
  L.bits = off;
  L.words = off > 64 ? 2 : 1;
  if (off > 128) return pmb_fail(h, PMB_E_UNSUPPORTED, "sort strategy: packed key above 128 bits");
  return L.words == 1 ? run_sort<1>(h, cq, L, r, part_groups) : run_sort<2>(h, cq, L, r, part_groups);
}

bool pmb_apply_packed_keys(CompiledQuery& cq) {
  DQuery& q = cq.dq;
  const CompiledQuery::KeyRanges& R = cq.ranges;
  DKey key[PMB_MAX_KEYS];
  int off = 0;
  for (int k = 0; k < q.n_keys; k++) {
    DKey& K = key[k] = q.key[k];
    int bits = 0;
    K.bias = 0;
    if (R.any[k]) {
      const unsigned long long span = R.hi[k] - R.lo[k];
      while (bits < 64 && (span >> bits) != 0) bits++;
      const int dt = q.col[K.col].dtype;
      K.bias = signed_dt(dt) ? (R.lo[k] ^ 0x8000000000000000ULL) : R.lo[k];
    }
    K.nullable = R.nulls[k] != 0;
    K.bits = (int8_t)bits;
    K.null_off = (int16_t)std::min(off, 63);
    off += K.nullable ? 1 : 0;
    K.data_off = (int16_t)std::min(off, 63);  // (a field without bits may start at 64)
    off += bits;
  }
  if (off > 64) return false;
  memcpy(q.key, key, sizeof(DKey) * q.n_keys);
  q.packed = (uint32_t)q.key_bits;
  q.key_bits = std::max(off, 1);
  return true;
}

// A nullable Int64 key is 65 bits wide by its type, two key columns 96 or more; their values mostly
// need far fewer. Packed into 64 bits they take the run-time compiled hash kernel, its sampled-key
// tables and the CTA-shared tier instead of the prebuilt 128-bit kernel, which has none of them
// (10M rows, nullable Int64 keys, 200K groups: 2524 us there). Below the run-time kernel's 2M rows the 64-bit
// prebuilt kernels have the sampled-key tables, which pay for the ranges (a pass and a wait, 20 to 60 us) where some
// key is frequent. Packed / not, us, one key, Zipf(1.0) and a quarter of the rows' number of groups: 20K rows 219 / 141,
// 193 / 126, 136 / 108; 60K 226 / 217, 201 / 167, 141 / 116; 200K 244 / 501, 217 / 317, 167 / 139; 1.9M 777 / 3971,
// 608 / 2080, 421 / 424. Hence PACK_ROWS.
constexpr int64_t PACK_ROWS = 100000;
int pmb_pack_wide_keys(pmb_handle* h, CompiledQuery& cq) {
  if (cq.dq.key_bits <= 64 || (cq.dq.n_rows < PACK_ROWS && !pmb_jit_enabled(cq.dq.n_rows)) || cq.dq.n_rows == 0) return PMB_OK;
  SortKeyLayout L;
  key_columns(cq.dq, L);
  const int rc = read_key_ranges(h, cq, L);
  if (rc) return rc;
  pmb_apply_packed_keys(cq);
  return PMB_OK;
}

// dst[i] = src[idx[i]], four rows of a thread in flight
__global__ void __launch_bounds__(ST_NT) k_gather_word(const unsigned long long* __restrict__ src,
                                                       const unsigned int* __restrict__ idx, int64_t n,
                                                       unsigned long long* __restrict__ dst, const unsigned int* status) {
  if (*status & PMB_ST_TIMEOUT) return;  // the passes gave up: idx need not be an order
  const int64_t stride = (int64_t)gridDim.x * ST_NT;
  for (int64_t i0 = (int64_t)blockIdx.x * ST_NT + threadIdx.x; i0 < n; i0 += 4 * stride) {
    unsigned long long v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = i0 + u * stride < n ? src[idx[i0 + u * stride]] : 0ULL;
#pragma unroll
    for (int u = 0; u < 4; u++)
      if (i0 + u * stride < n) dst[i0 + u * stride] = v[u];
  }
}

// Stable LSD sort of (key, row index) pairs for callers outside the group-by's own sort: the onesweep
// pass kernel over the 8-bit digits 0 .. n_passes-1 of W-word keys (word-major, stride cap).
// hist_host holds every pass's digit counts of all n keys (also at hist_dev); a digit that one value
// fills is skipped. On return *i is the order and, for one-word keys, *k the sorted keys (the inputs
// or the alternates). Two-word keys are sorted a word at a time, the second word fetched in the order
// of the first: a pass over 12-byte pairs takes half the time of one over 20-byte pairs (20M rows: 159
// against 316 us), the fetch less than one pass; their sorted keys are not returned. The second words
// are stored by row number; `permuted`: *i is not 0, 1, 2, ... already on entry. Without hist_host every
// digit gets its pass (one more pass of up to a million keys takes less than reading the counts back).
// The call does not wait: *status_dev (device; null before a call's first round) holds PMB_ST_TIMEOUT
// after the stream has got there, and then neither *i nor *k can be relied on: whatever follows an entry of
// *i to a row looks at the status first.
int pmb_sort_pairs(pmb_handle* h, int W, unsigned long long** k, unsigned long long** k_alt, unsigned int** i,
                   unsigned int** i_alt, uint64_t cap, int64_t n, int n_passes, const unsigned int* hist_dev,
                   const unsigned int* hist_host, bool permuted, unsigned int** status_dev) {
  if (W != 1 && W != 2) return pmb_fail(h, PMB_E_INVALID, "sort: key of 1 or 2 words");
  if (n_passes > MAX_PASSES) return pmb_fail(h, PMB_E_INVALID, "sort: more than 16 digit passes");
  if (n <= 1 || n_passes <= 0) return PMB_OK;
  const int64_t tiles = (n + PassShape<1>::TILE - 1) / PassShape<1>::TILE;
  const size_t lb_bytes = (size_t)tiles * RADIX * 8;
  // per pass a ticket and look-back states; small ones are cleared for all passes at once
  const size_t pass_bytes = lb_bytes + 64;
  const bool at_once = pass_bytes * n_passes <= (size_t)32 << 20;
  const size_t clear = at_once ? pass_bytes * n_passes : pass_bytes;
  uint8_t* zeroed = (uint8_t*)pmb_ws_alloc(h, clear + 64);
  if (!zeroed) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (sort passes)");
  // the status of an earlier round of the same call goes on being used
  unsigned int* status = *status_dev ? *status_dev : (unsigned int*)(zeroed + clear);
  if (at_once) PMB_CUDA(h, cudaMemsetAsync(zeroed, 0, clear + 64, h->stream));
  else PMB_CUDA(h, cudaMemsetAsync(zeroed + clear, 0, 64, h->stream));
  if (h->fault_wait) PMB_CUDA(h, cudaMemsetAsync(status, PMB_ST_TIMEOUT, 1, h->stream));
  PMB_CUDA(h, cudaFuncSetAttribute(k_sort_pass<1, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PassShape<1>::SMEM));
  unsigned long long* a = *k;       // the current word's keys, and where the next pass writes them
  unsigned long long* b = *k_alt;
  bool moved = permuted;            // the order differs from the rows'
  for (int p = 0; p < n_passes; p++) {
    if (p == 8) {
      a = *k + cap;
      b = *k_alt + cap;
    }
    bool constant = false;
    for (int d = 0; hist_host && d < RADIX; d++) constant |= hist_host[(size_t)p * RADIX + d] == (unsigned)n;
    if (constant) continue;
    uint8_t* z = zeroed + (at_once ? (size_t)p * pass_bytes : 0);
    if (!at_once) PMB_CUDA(h, cudaMemsetAsync(z, 0, pass_bytes, h->stream));
    if (p >= 8 && moved) {  // the second word in the order so far, once
      const int blocks = (int)std::max<int64_t>(1, std::min<int64_t>((n + 4 * ST_NT - 1) / (4 * ST_NT), (int64_t)h->sm_count * 8));
      pmb_kernel_begin(h, "sort_fetch");
      k_gather_word<<<blocks, ST_NT, 0, h->stream>>>(a, *i, n, b, status);
      pmb_kernel_end(h);
      PMB_CUDA(h, cudaGetLastError());
      std::swap(a, b);
      moved = false;
    }
    PassParams P;
    P.kin = a;
    P.kout = b;
    P.iin = *i;
    P.iout = *i_alt;
    P.cap = cap;
    P.n = n;
    P.shift = 8 * (p & 7);
    P.hist = hist_dev + (size_t)p * RADIX;
    P.ticket = (unsigned long long*)z;
    P.lb = (unsigned long long*)(z + 64);
    P.status = status;
    pmb_kernel_begin(h, "sort_pass");
    k_sort_pass<1, false><<<(unsigned)tiles, PassShape<1>::NT, PassShape<1>::SMEM, h->stream>>>(P);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
    std::swap(a, b);
    std::swap(*i, *i_alt);
    if (p < 8) moved = true;
  }
  if (W == 1) {
    *k = a;
    *k_alt = b;
  }
  *status_dev = status;
  return PMB_OK;
}

