// pmb_order.cu — the rows of a table sorted by some of its columns, on the device: a Sort over a
// GroupBy, top_k and bottom_k.
//
// The reference sorts on the CPU: its Sort plan runs the inner pipeline, then Polars'
// `df.sort(by, descending, nulls_last)` and the slice (python/polars_metal/_udf.py:684-721); only
// a single non-null Float32 column goes to an MLX sort, reversed and sliced on the host
// (_build_sort_fused, python/polars_metal/_udf.py:724-790). Here every dtype and any number of
// sort columns run on the GPU:
//   1. k_order_range  — per sort column the range of its values in Polars' order (as an unsigned
//                       integer) and its null count;
//   2. the sort columns are packed into keys of one or two 64-bit words: per column a null flag
//                       (when the column has nulls) above (value - min) or (max - value) bits, the
//                       most significant column highest. Columns that do not fit 128 bits go to
//                       further rounds, least significant first; every round is a stable sort of
//                       the previous round's order, so the rounds compose;
//                       A wide column of few distinct values (measurements of limited resolution)
//                       goes in as the value's rank among them (order_dict);
//   3. k_order_encode — keys of the rows in the current order, with the digit histograms;
//   4. pmb_sort_pairs — the group-by sort's LSD onesweep passes over the digits that vary;
//   5. k_order_gather — the slice of the sorted rows, a warp per 32 output rows so that each
//                       validity word is one ballot. Integer and Bool sort columns are decoded from
//                       the sorted keys when one round holds them all; the other columns are
//                       gathered by row index, without reading the validity of a column that
//                       k_order_range found to have no nulls.
// A small table takes k_order_small instead, which does all of it in one launch.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <vector>

#include "pmb_groupby.h"

namespace {

constexpr int OR_NT = 256;
constexpr int OR_PASSES = 16;   // 8-bit digits of a 128-bit key
constexpr int OR_RADIX = 256;

// Polars' order of a value as an unsigned integer: signed integers with the sign bit flipped;
// floats with -0.0 read as 0.0 and every NaN as one NaN above +inf, negative values' bits
// inverted and non-negative values' sign bit set; unsigned integers and Bool as they are
__device__ __forceinline__ unsigned long long order_key(uint64_t b, int dt) {
  switch (dt) {
    case PMB_I8: return (unsigned long long)(long long)(int8_t)b ^ 0x8000000000000000ULL;
    case PMB_I16: return (unsigned long long)(long long)(int16_t)b ^ 0x8000000000000000ULL;
    case PMB_I32: return (unsigned long long)(long long)(int32_t)b ^ 0x8000000000000000ULL;
    case PMB_I64: return b ^ 0x8000000000000000ULL;
    case PMB_F32: {
      uint32_t x = (uint32_t)b;
      if ((x & 0x7FFFFFFFu) > 0x7F800000u) x = 0x7FC00000u;
      if (x == 0x80000000u) x = 0u;
      return (x & 0x80000000u) ? (unsigned long long)(uint32_t)~x : (unsigned long long)(x | 0x80000000u);
    }
    case PMB_F64: {
      uint64_t x = b;
      if ((x & 0x7FFFFFFFFFFFFFFFULL) > 0x7FF0000000000000ULL) x = 0x7FF8000000000000ULL;
      if (x == 0x8000000000000000ULL) x = 0ULL;
      return (x >> 63) ? ~x : (x | 0x8000000000000000ULL);
    }
    default: return b;
  }
}

struct SortCols {
  int n;
  const uint8_t* data[PMB_MAX_KEYS];
  const uint8_t* valid[PMB_MAX_KEYS];
  int elem[PMB_MAX_KEYS];
  int dtype[PMB_MAX_KEYS];
};

struct OrderRange {
  unsigned long long lo[PMB_MAX_KEYS];
  unsigned long long hi[PMB_MAX_KEYS];
  unsigned long long nulls[PMB_MAX_KEYS];
  unsigned int any[PMB_MAX_KEYS];
  unsigned int distinct[PMB_MAX_KEYS];  // of RS_ROWS sampled rows: distinct values, and those that
  unsigned int f1[PMB_MAX_KEYS];        // occurred once
  unsigned int f2[PMB_MAX_KEYS];        // and twice
};

__device__ __forceinline__ unsigned long long warp_min64(unsigned long long v) {
  for (int o = 16; o; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ unsigned long long warp_max64(unsigned long long v) {
  for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// range and null count of one sort column: 16 bytes (V rows) per load, RU loads in flight. 20M rows of
// Float64 and Int32 with nulls took 172 us with a row per load (four in flight), 91 us so,
// the counts of nulls included.
constexpr int RU = 4;
template <typename T>
__device__ __forceinline__ void order_range_of(const uint8_t* data, const uint8_t* __restrict__ valid, int64_t n, int dtype,
                                               unsigned long long& lo, unsigned long long& hi, unsigned& any,
                                               unsigned long long& nul) {
  constexpr int V = 16 / (int)sizeof(T);
  constexpr unsigned ALL = V == 16 ? 0xFFFFu : (1u << V) - 1u;
  const T* __restrict__ d = reinterpret_cast<const T*>(data);
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
      x[u] = reinterpret_cast<const uint4*>(d)[c];
      if (!valid) ok[u] = ALL;
      else if (V == 16) ok[u] = reinterpret_cast<const uint16_t*>(valid)[c];
      else ok[u] = (valid[(c * V) >> 3] >> ((c * V) & 7)) & ALL;
      nul += V - __popc(ok[u]);
    }
#pragma unroll
    for (int u = 0; u < RU; u++) {
      if (ok[u] == 0u) continue;
      any = 1u;
      T v[V];
      memcpy(v, &x[u], 16);
#pragma unroll
      for (int i = 0; i < V; i++) {
        const unsigned long long o = order_key((uint64_t)v[i], dtype);
        if ((ok[u] >> i) & 1u) {
          lo = min(lo, o);
          hi = max(hi, o);
        }
      }
    }
  }
  const int64_t r = chunks * V + t0;
  if (r < n) {
    if (pmb_valid_bit(valid, r)) {
      const unsigned long long o = order_key((uint64_t)d[r], dtype);
      any = 1u;
      lo = min(lo, o);
      hi = max(hi, o);
    } else {
      nul++;
    }
  }
}

struct NullFlagCols {
  int n;
  const uint8_t* valid[PMB_MAX_OUT];  // null: no bitmap
};

// flags[c] = 1 when the bitmap of column c has a null among rows [0, n)
__device__ __forceinline__ void null_flags(const NullFlagCols& V, int64_t n, unsigned int* flags) {
  const int64_t t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t quads = n >> 7;  // whole 16-byte pieces (the bitmaps are 16-byte aligned)
  for (int c = 0; c < V.n; c++) {
    const uint8_t* v = V.valid[c];
    if (!v) continue;
    bool hole = false;
    for (int64_t i = t0; i < quads; i += stride) {
      const uint4 x = reinterpret_cast<const uint4*>(v)[i];
      hole |= (x.x & x.y & x.z & x.w) != 0xFFFFFFFFu;
    }
    for (int64_t r = quads * 128 + t0; r < n; r += stride) hole |= !((v[r >> 3] >> (r & 7)) & 1u);
    if (__any_sync(0xffffffffu, hole) && (threadIdx.x & 31) == 0) atomicOr(&flags[c], 1u);
  }
}

// Distinct values of a sort column among RS_ROWS rows spread over the table, by 32-bit fingerprint.
constexpr int RS_ROWS = 1024, RS_SLOTS = 2048;
__device__ void sample_column(const SortCols& C, int c, int64_t n, OrderRange* out) {
  __shared__ unsigned int s_fp[RS_SLOTS], s_num[RS_SLOTS];
  for (int i = threadIdx.x; i < RS_SLOTS; i += OR_NT) {
    s_fp[i] = 0u;
    s_num[i] = 0u;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < RS_ROWS; i += OR_NT) {
    const int64_t r = n / RS_ROWS * i;
    if (!pmb_valid_bit(C.valid[c], r)) continue;
    const unsigned long long hk = pmb_fmix64(order_key(pmb_load_bits(C.data[c], C.elem[c], r), C.dtype[c]));
    const unsigned fp = (unsigned)(hk >> 32) | 1u;
    unsigned s = (unsigned)hk & (RS_SLOTS - 1);
    for (int p = 0; p < RS_SLOTS; p++) {
      const unsigned cur = atomicCAS(&s_fp[s], 0u, fp);
      if (cur == 0u || cur == fp) {
        atomicAdd(&s_num[s], 1u);
        break;
      }
      s = (s + 1) & (RS_SLOTS - 1);
    }
  }
  __syncthreads();
  unsigned d = 0, f1 = 0, f2 = 0;
  for (int i = threadIdx.x; i < RS_SLOTS; i += OR_NT) {
    d += s_num[i] > 0;
    f1 += s_num[i] == 1;
    f2 += s_num[i] == 2;
  }
  if (d) atomicAdd(&out->distinct[c], d);
  if (f1) atomicAdd(&out->f1[c], f1);
  if (f2) atomicAdd(&out->f2[c], f2);
}

// the sort columns' ranges (blockIdx.y 0), which columns have nulls (blockIdx.y 1) and, with a third grid
// row, how many distinct values a sample of each has
__global__ void __launch_bounds__(OR_NT) k_order_range(const __grid_constant__ SortCols C, int64_t n, OrderRange* out,
                                                       const __grid_constant__ NullFlagCols V, unsigned int* flags) {
  if (blockIdx.y == 1) {
    null_flags(V, n, flags);
    return;
  }
  if (blockIdx.y == 2) {
    if (blockIdx.x < C.n) sample_column(C, blockIdx.x, n, out);
    return;
  }
  const int lane = threadIdx.x & 31;
  for (int c = 0; c < C.n; c++) {
    unsigned long long lo = ~0ULL, hi = 0, nul = 0;
    unsigned any = 0;
    const uint8_t* data = C.data[c];
    const uint8_t* valid = C.valid[c];
    const int dt = C.dtype[c];
    switch (dt) {  // the type's order is a constant in each
      case PMB_I8: order_range_of<uint8_t>(data, valid, n, PMB_I8, lo, hi, any, nul); break;
      case PMB_I16: order_range_of<uint16_t>(data, valid, n, PMB_I16, lo, hi, any, nul); break;
      case PMB_I32: order_range_of<uint32_t>(data, valid, n, PMB_I32, lo, hi, any, nul); break;
      case PMB_I64: order_range_of<unsigned long long>(data, valid, n, PMB_I64, lo, hi, any, nul); break;
      case PMB_U8: order_range_of<uint8_t>(data, valid, n, PMB_U8, lo, hi, any, nul); break;
      case PMB_U16: order_range_of<uint16_t>(data, valid, n, PMB_U16, lo, hi, any, nul); break;
      case PMB_U32: order_range_of<uint32_t>(data, valid, n, PMB_U32, lo, hi, any, nul); break;
      case PMB_U64: order_range_of<unsigned long long>(data, valid, n, PMB_U64, lo, hi, any, nul); break;
      case PMB_F32: order_range_of<uint32_t>(data, valid, n, PMB_F32, lo, hi, any, nul); break;
      case PMB_F64: order_range_of<unsigned long long>(data, valid, n, PMB_F64, lo, hi, any, nul); break;
      default:  // Bool
        for (int64_t r = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
          if (!pmb_valid_bit(valid, r)) {
            nul++;
            continue;
          }
          const unsigned long long o = pmb_load_bits(data, 0, r);
          lo = min(lo, o);
          hi = max(hi, o);
          any = 1;
        }
    }
    lo = warp_min64(lo);
    hi = warp_max64(hi);
    for (int o = 16; o; o >>= 1) nul += __shfl_xor_sync(0xffffffffu, nul, o);
    any = __any_sync(0xffffffffu, any);
    if (lane == 0) {
      if (any) {
        atomicMin(&out->lo[c], lo);
        atomicMax(&out->hi[c], hi);
        atomicOr(&out->any[c], 1u);
      }
      if (nul) atomicAdd(&out->nulls[c], nul);
    }
  }
}

// ---------------------------------------------------------------- ranks of few distinct values
// A float column of limited resolution takes 64 key bits for a few thousand values, eight of the eleven
// passes of 20M rows ordered by (float, int). Its distinct values are collected and ranked, and the ranks
// sorted instead: 14 bits, four passes of one-word keys, and the column itself read back from its sorted
// ranks instead of gathered.
// Every kernel reads the count from the device; the host reads it once, after the last.
constexpr int DICT_CTA = 16384;            // slots of a CTA's set
constexpr int DICT_MAX = DICT_CTA / 4 * 3; // distinct values at most
constexpr int DICT_SEEN = 65536;           // slots of the global set
constexpr int DICT_SLOTS = 16384;          // slots of the largest lookup table
constexpr int DICT_NT = 1024;

struct DictCtl {
  unsigned int count;  // distinct values so far
  unsigned int fail;   // too many, or two that the lookup table cannot tell apart
  unsigned int alias;  // some valid value's bits are not those of its order key (-0.0, NaN payloads)
};

struct DictCol {
  const uint8_t* data;
  const uint8_t* valid;
  int elem, dtype;
};

// the raw bits of the value whose order key is o (-0.0 reads 0.0, every NaN the same one)
__device__ __forceinline__ uint64_t dict_value(unsigned long long o, int dt) {
  switch (dt) {
    case PMB_I8: case PMB_I16: case PMB_I32: case PMB_I64: return o ^ 0x8000000000000000ULL;
    case PMB_F32: return (o & 0x80000000ULL) ? (o & 0x7FFFFFFFULL) : (uint64_t)(uint32_t)~(uint32_t)o;
    case PMB_F64: return (o >> 63) ? (o & 0x7FFFFFFFFFFFFFFFULL) : ~o;
    default: return o;
  }
}

// The distinct values (as order keys, none of them PMB_EMPTY64) of a column's valid rows: each CTA
// collects its rows' values in shared memory and adds them to the global set at the end, so that the rows
// wait for no global probe (with every CTA's first meeting of a value sent there at once, 20M rows of
// 10,000 values took 478 us, 165 us so). A column of too many values stops after some 12,000 rows
// of every CTA.
template <typename T>
__global__ void __launch_bounds__(DICT_NT) k_dict_collect(const DictCol c, int64_t n, unsigned long long* seen,
                                                          unsigned long long* list, DictCtl* ctl) {
  extern __shared__ unsigned long long s_seen[];
  __shared__ unsigned s_n, s_alias;
  for (int i = threadIdx.x; i < DICT_CTA; i += DICT_NT) s_seen[i] = PMB_EMPTY64;
  if (threadIdx.x == 0) s_n = s_alias = 0u;
  __syncthreads();
  const T* __restrict__ data = reinterpret_cast<const T*>(c.data);
  const bool fl = c.dtype == PMB_F32 || c.dtype == PMB_F64;
  constexpr int U = 4;
  const int64_t stride = (int64_t)gridDim.x * DICT_NT;
  for (int64_t r0 = (int64_t)blockIdx.x * DICT_NT + threadIdx.x; r0 < n; r0 += U * stride) {
    unsigned long long k[U], first[U];
    unsigned at[U];
    bool ok[U];
    T x[U];
#pragma unroll
    for (int u = 0; u < U; u++) {
      const int64_t r = r0 + u * stride;
      x[u] = r < n ? data[r] : (T)0;
      ok[u] = r < n && pmb_valid_bit(c.valid, r);
    }
    if (*reinterpret_cast<volatile unsigned int*>(&s_n) > DICT_MAX) break;
#pragma unroll
    for (int u = 0; u < U; u++) {
      k[u] = order_key((uint64_t)x[u], c.dtype);
      if (fl && ok[u] && dict_value(k[u], c.dtype) != (uint64_t)x[u]) s_alias = 1u;
      at[u] = (unsigned)pmb_fmix64(k[u]) & (DICT_CTA - 1);
      first[u] = *reinterpret_cast<volatile unsigned long long*>(&s_seen[at[u]]);
    }
#pragma unroll
    for (int u = 0; u < U; u++) {
      if (!ok[u] || first[u] == k[u]) continue;
      unsigned long long cur = first[u];
      unsigned s = at[u];
      for (int p = 0; p < DICT_CTA; p++) {
        if (cur == PMB_EMPTY64) {
          cur = atomicCAS(&s_seen[s], PMB_EMPTY64, k[u]);
          if (cur == PMB_EMPTY64) {
            atomicAdd(&s_n, 1u);
            break;
          }
        }
        if (cur == k[u]) break;
        s = (s + 1) & (DICT_CTA - 1);
        cur = *reinterpret_cast<volatile unsigned long long*>(&s_seen[s]);
      }
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    if (s_alias) ctl->alias = 1u;
    if (s_n > DICT_MAX) ctl->fail = 1u;
  }
  if (s_n > DICT_MAX) return;
  for (int i = threadIdx.x; i < DICT_CTA; i += DICT_NT) {
    const unsigned long long v = s_seen[i];
    if (v == PMB_EMPTY64) continue;
    unsigned s = (unsigned)(pmb_fmix64(v) >> 20) & (DICT_SEEN - 1);
    int p = 0;
    for (; p < 64; p++) {
      unsigned long long cur = __ldcg(&seen[s]);
      if (cur == PMB_EMPTY64) {
        cur = atomicCAS(&seen[s], PMB_EMPTY64, v);
        if (cur == PMB_EMPTY64) {
          const unsigned l = atomicAdd(&ctl->count, 1u);
          if (l < DICT_MAX) list[l] = v;
          else ctl->fail = 1u;
          break;
        }
      }
      if (cur == v) break;
      s = (s + 1) & (DICT_SEEN - 1);
    }
    if (p == 64) ctl->fail = 1u;  // a run of 64 in a set a fifth full: it holds too many
  }
}

// rank[i] += the values of part blockIdx.y that lie below value i (blockIdx.x * OR_NT + threadIdx.x)
constexpr int DICT_PARTS = 32;
__global__ void __launch_bounds__(OR_NT) k_dict_rank(const unsigned long long* __restrict__ list, const DictCtl* ctl,
                                                     unsigned int* rank) {
  __shared__ unsigned long long s_v[DICT_MAX / DICT_PARTS];
  if (ctl->fail) return;  // (the count may exceed DICT_MAX then)
  const int n = (int)ctl->count, i = blockIdx.x * OR_NT + threadIdx.x;
  if ((int)blockIdx.x * OR_NT >= n) return;
  const int part = (n + DICT_PARTS - 1) / DICT_PARTS, j0 = part * blockIdx.y, m = min(part, n - j0);
  for (int j = threadIdx.x; j < m; j += OR_NT) s_v[j] = list[j0 + j];
  __syncthreads();
  if (i >= n || m <= 0) return;
  const unsigned long long v = list[i];
  unsigned c = 0;
#pragma unroll 8
  for (int j = 0; j < m; j++) c += s_v[j] < v;
  if (c) atomicAdd(&rank[i], c);
}

// slots of the lookup table of n values: at most three quarters full
__host__ __device__ __forceinline__ int dict_slots(int n) {
  int s = 512;
  while (s / 4 * 3 < n) s *= 2;
  return s;
}
__device__ __forceinline__ unsigned dict_fp(unsigned long long hk) { return (unsigned)(hk >> 32) | 1u; }

// The lookup table: fingerprints by linear probing, and each one's rank. A lookup takes the first equal
// fingerprint from its first slot on, and every value looked up is in the table, so that the answer is
// right as long as no value met its own fingerprint on the way to its slot (the call sorts whole keys
// then). And the values' bits by rank, from which the sorted column is written.
__global__ void __launch_bounds__(OR_NT) k_dict_table(const unsigned long long* __restrict__ list,
                                                      const unsigned int* __restrict__ rank, DictCtl* ctl,
                                                      int dtype, unsigned int* fps, unsigned short* codes,
                                                      unsigned long long* values) {
  const int n = (int)ctl->count, i = blockIdx.x * OR_NT + threadIdx.x;
  if (i >= n || n > DICT_MAX || ctl->fail == 1u) return;
  values[rank[i]] = dict_value(list[i], dtype);
  const unsigned mask = (unsigned)dict_slots(n) - 1u;
  const unsigned long long hk = pmb_fmix64(list[i]);
  const unsigned fp = dict_fp(hk);
  unsigned s = (unsigned)hk & mask;
  for (unsigned p = 0; p <= mask; p++) {
    const unsigned cur = atomicCAS(&fps[s], 0u, fp);
    if (cur == 0u) {
      codes[s] = (unsigned short)rank[i];
      return;
    }
    if (cur == fp) break;
    s = (s + 1) & mask;
  }
  ctl->fail = 2u;
}

// one round's packed key: per column a null flag (null_off >= 0) and `data_bits` value bits
struct OrderLayout {
  int n;
  int bits;
  int null_off[PMB_MAX_KEYS];
  int data_off[PMB_MAX_KEYS];
  int data_bits[PMB_MAX_KEYS];
  int desc[PMB_MAX_KEYS];
  int nulls_last[PMB_MAX_KEYS];
  unsigned long long lo[PMB_MAX_KEYS];
  unsigned long long hi[PMB_MAX_KEYS];
  const uint8_t* data[PMB_MAX_KEYS];
  const uint8_t* valid[PMB_MAX_KEYS];
  int elem[PMB_MAX_KEYS];
  int dtype[PMB_MAX_KEYS];
  int dict;                 // the column that goes in by rank (-1: none)
  int dict_slots;
  const unsigned int* dict_fps;
  const unsigned short* dict_codes;
};

template <int W>
__device__ __forceinline__ void put_bits(unsigned long long (&k)[W], int off, unsigned long long v, int bits) {
  if (bits == 0) return;
  const int wi = off >> 6, sh = off & 63;
  k[wi] |= v << sh;
  if (W > 1 && sh + bits > 64 && wi + 1 < W) k[wi + 1] |= v >> (64 - sh);
}

template <int W>
__device__ __forceinline__ unsigned key_digit(const unsigned long long (&k)[W], int shift) {
  const int wi = shift >> 6, sh = shift & 63;
  return (unsigned)((k[wi] >> sh) & 0xFFu);  // digits are 8-bit aligned: never across words
}

constexpr int EU = 4;  // rows of a thread in flight
template <int E>
__device__ __forceinline__ void encode_load(const uint8_t* d, const unsigned (&r)[EU], uint64_t (&x)[EU]) {
#pragma unroll
  for (int u = 0; u < EU; u++) x[u] = pmb_load_bits(d, E, r[u]);
}

// DICT: the lookup table is copied into shared memory, and the CTAs have DICT_NT threads. 20M rows of
// (Float64, Int32): 274 us for the eleven digits of whole keys, 246 us for the four with ranks. Bound by
// the counting's shared atomics, many of one digit.
template <int W, bool DICT>
__global__ void __launch_bounds__(DICT ? DICT_NT : OR_NT) k_order_encode(const __grid_constant__ OrderLayout L, int64_t n,
                                                        const unsigned int* perm, unsigned long long* keys,
                                                        uint64_t cap, unsigned int* idx, int passes,
                                                        unsigned int* hist, const unsigned int* status) {
  if (perm && status && (*status & PMB_ST_TIMEOUT)) return;  // the round before gave up: perm need not be an order
  __shared__ unsigned int s_hist[OR_PASSES * OR_RADIX];
  extern __shared__ unsigned int s_fps[];
  unsigned short* s_codes = reinterpret_cast<unsigned short*>(s_fps + (DICT ? L.dict_slots : 0));
  for (int i = threadIdx.x; i < passes * OR_RADIX; i += blockDim.x) s_hist[i] = 0;
  if (DICT)
    for (int i = threadIdx.x; i < L.dict_slots; i += blockDim.x) {
      s_fps[i] = L.dict_fps[i];
      s_codes[i] = L.dict_codes[i];
    }
  __syncthreads();
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p0 < n; p0 += EU * stride) {
    unsigned r[EU];
    unsigned long long k[EU][W];
#pragma unroll
    for (int u = 0; u < EU; u++) {
      const int64_t pos = p0 + u * stride;
      r[u] = pos < n ? (perm ? perm[pos] : (unsigned)pos) : 0u;
#pragma unroll
      for (int i = 0; i < W; i++) k[u][i] = 0;
    }
    for (int c = 0; c < L.n; c++) {
      uint64_t x[EU];
      bool v[EU];
      const uint8_t* d = L.data[c];
      switch (L.elem[c]) {  // a column's rows are loaded before any is used
        case 0: encode_load<0>(d, r, x); break;
        case 1: encode_load<1>(d, r, x); break;
        case 2: encode_load<2>(d, r, x); break;
        case 4: encode_load<4>(d, r, x); break;
        default: encode_load<8>(d, r, x); break;
      }
#pragma unroll
      for (int u = 0; u < EU; u++) v[u] = pmb_valid_bit(L.valid[c], r[u]);
#pragma unroll
      for (int u = 0; u < EU; u++) {
        if (L.null_off[c] >= 0) put_bits<W>(k[u], L.null_off[c], (L.nulls_last[c] ? !v[u] : v[u]) ? 1ULL : 0ULL, 1);
        if (!v[u]) continue;
        unsigned long long o = order_key(x[u], L.dtype[c]);
        if (DICT && c == L.dict) {
          const unsigned long long hk = pmb_fmix64(o);
          const unsigned fp = dict_fp(hk), mask = (unsigned)L.dict_slots - 1u;
          unsigned s = (unsigned)hk & mask;
          for (unsigned p = 0; p < mask && s_fps[s] != fp; p++) s = (s + 1) & mask;
          o = s_codes[s];
        }
        put_bits<W>(k[u], L.data_off[c], L.desc[c] ? L.hi[c] - o : o - L.lo[c], L.data_bits[c]);
      }
    }
#pragma unroll
    for (int u = 0; u < EU; u++) {
      const int64_t pos = p0 + u * stride;
      if (pos >= n) break;
      keys[pos] = k[u][0];
      if (W > 1) keys[cap + r[u]] = k[u][W - 1];  // the second word by row (see pmb_sort_pairs)
      idx[pos] = r[u];
      for (int p = 0; p < passes; p++) atomicAdd(&s_hist[p * OR_RADIX + key_digit<W>(k[u], 8 * p)], 1u);
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < passes * OR_RADIX; i += blockDim.x) {
    const unsigned v = s_hist[i];
    if (v) atomicAdd(&hist[i], v);
  }
}

struct GatherCols {
  int n;
  const uint8_t* data[PMB_MAX_OUT];
  const uint8_t* valid[PMB_MAX_OUT];  // null: every row valid
  int elem[PMB_MAX_OUT];
  int dec[PMB_MAX_OUT];               // >= 0: decoded from the sorted keys, column dec of L
  int zero[PMB_MAX_OUT];              // an integer or Bool sort column: its null rows read 0
  uint8_t* out_data[PMB_MAX_OUT];
  unsigned int* out_valid[PMB_MAX_OUT];
  const unsigned long long* keys;     // the sorted one-word keys, with dec >= 0
  const unsigned long long* values;   // the bits by rank of the column that went in by rank
};

__device__ __forceinline__ unsigned long long get_bits(const unsigned long long* keys, uint64_t pos, int off, int bits) {
  if (bits == 0) return 0;
  const unsigned long long v = keys[pos] >> off;
  return bits == 64 ? v : (v & ((1ULL << bits) - 1ULL));
}

// the raw bits of an integer or Bool value from its order key
__device__ __forceinline__ uint64_t from_order_key(unsigned long long o, int dt) {
  switch (dt) {
    case PMB_I8: case PMB_I16: case PMB_I32: case PMB_I64: return o ^ 0x8000000000000000ULL;
    default: return o;
  }
}

constexpr int GU = 8;  // output words a warp fills per iteration: GU independent loads in flight

template <typename T>
__device__ __forceinline__ void gather_rows(const uint8_t* data, const int64_t (&r)[GU], const bool (&ok)[GU],
                                            uint64_t (&b)[GU]) {
  const T* __restrict__ d = reinterpret_cast<const T*>(data);
#pragma unroll
  for (int u = 0; u < GU; u++) b[u] = ok[u] ? (uint64_t)d[r[u]] : 0;
}

// Rows idx[start + p] (start + p without an order) for p < m of column blockIdx.y; a warp fills GU
// validity words (32 rows each) per iteration, loading the rows of all GU words before it writes any.
// Bound by one random 32-byte sector per row and column; with the columns one after another in a
// thread, four rows at a time, 20M rows of 4 columns took 1195 us, 965 us so.
__global__ void __launch_bounds__(OR_NT) k_order_gather(const __grid_constant__ GatherCols G,
                                                        const __grid_constant__ OrderLayout L, const unsigned int* idx,
                                                        int64_t start, int64_t m, const unsigned int* status) {
  if (idx && status && (*status & PMB_ST_TIMEOUT)) return;  // the sort gave up: idx need not be an order
  const int lane = threadIdx.x & 31;
  const int64_t warps = (int64_t)gridDim.x * (blockDim.x / 32);
  const int c = blockIdx.y, e = G.elem[c], k = G.dec[c];
  for (int64_t w0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / 32 * GU; w0 * 32 < m; w0 += warps * GU) {
    bool ok[GU], v[GU];
    uint64_t b[GU];
#pragma unroll
    for (int u = 0; u < GU; u++) ok[u] = (w0 + u) * 32 + lane < m;
    if (k >= 0) {
      // decoded: the null flag and the value field of the sorted key at position start + p
#pragma unroll
      for (int u = 0; u < GU; u++) {
        v[u] = ok[u];
        b[u] = 0;
        if (!ok[u]) continue;
        const uint64_t pos = (uint64_t)(start + (w0 + u) * 32 + lane);
        if (L.null_off[k] >= 0) {
          const bool flag = get_bits(G.keys, pos, L.null_off[k], 1) != 0;
          v[u] = L.nulls_last[k] ? !flag : flag;
        }
        const unsigned long long f = get_bits(G.keys, pos, L.data_off[k], L.data_bits[k]);
        const unsigned long long o = L.desc[k] ? L.hi[k] - f : L.lo[k] + f;
        if (v[u]) b[u] = k == L.dict ? G.values[o] : from_order_key(o, L.dtype[k]);
        else if (!G.zero[c]) b[u] = pmb_load_bits(G.data[c], e, idx[pos]);  // a float's bits under a null
      }
    } else {
      int64_t r[GU];
#pragma unroll
      for (int u = 0; u < GU; u++) {
        const int64_t p = start + (w0 + u) * 32 + lane;
        r[u] = ok[u] ? (idx ? (int64_t)idx[p] : p) : 0;
      }
      const uint8_t* d = G.data[c];
      switch (e) {
        case 0:
#pragma unroll
          for (int u = 0; u < GU; u++) b[u] = ok[u] ? (uint64_t)((d[r[u] >> 3] >> (r[u] & 7)) & 1u) : 0;
          break;
        case 1: gather_rows<uint8_t>(d, r, ok, b); break;
        case 2: gather_rows<uint16_t>(d, r, ok, b); break;
        case 4: gather_rows<uint32_t>(d, r, ok, b); break;
        default: gather_rows<unsigned long long>(d, r, ok, b); break;
      }
      const uint8_t* vb = G.valid[c];
#pragma unroll
      for (int u = 0; u < GU; u++) {
        v[u] = ok[u] && (vb == nullptr || ((vb[r[u] >> 3] >> (r[u] & 7)) & 1u));
        if (G.zero[c] && !v[u]) b[u] = 0;
      }
    }
#pragma unroll
    for (int u = 0; u < GU; u++) {
      const int64_t p = (w0 + u) * 32 + lane;
      if (ok[u]) {
        switch (e) {
          case 0: break;
          case 1: G.out_data[c][p] = (uint8_t)b[u]; break;
          case 2: reinterpret_cast<uint16_t*>(G.out_data[c])[p] = (uint16_t)b[u]; break;
          case 4: reinterpret_cast<uint32_t*>(G.out_data[c])[p] = (uint32_t)b[u]; break;
          default: reinterpret_cast<uint64_t*>(G.out_data[c])[p] = b[u]; break;
        }
      }
      const unsigned vw = __ballot_sync(0xffffffffu, v[u]);
      const unsigned dw = __ballot_sync(0xffffffffu, ok[u] && e == 0 && b[u]);
      if (lane == 0 && (w0 + u) * 32 < m) {
        G.out_valid[c][w0 + u] = vw;
        if (e == 0) reinterpret_cast<unsigned int*>(G.out_data[c])[w0 + u] = dw;
      }
    }
  }
}

// ---------------------------------------------------------------- small tables in one launch
// Up to SMALL_ROWS rows whose sort columns fit 128 key bits at their full widths: one CTA packs the
// keys, sorts them in shared memory and gathers the slice, in one launch without a read-back, where that is less
// than the general path's launches (ranges, encode, a pass per digit, gather) and its read-back (small_pays).
constexpr int SMALL_ROWS = 8192;
constexpr int SMALL_NT = 1024;

struct SmallOrder {
  OrderLayout L;  // fields at the columns' full widths
  GatherCols G;   // dec >= 0: an integer or Bool sort column (its null rows read 0)
  int W;
  int n, n2;      // rows; the next power of two (at least 64)
  int drop_nulls;
  long long offset, limit;
  unsigned long long* out_rows;  // rows written
};

template <int W>
__device__ __forceinline__ bool small_less(const unsigned long long* lo, const unsigned long long* hi,
                                           const unsigned short* ix, int a, int b) {
  if (W > 1 && hi[a] != hi[b]) return hi[a] < hi[b];
  if (lo[a] != lo[b]) return lo[a] < lo[b];
  return ix[a] < ix[b];  // rows with equal keys keep their order
}

template <int W>
__global__ void __launch_bounds__(SMALL_NT, 1) k_order_small(const __grid_constant__ SmallOrder S) {
  extern __shared__ __align__(16) unsigned long long smem_keys[];
  __shared__ int s_nulls;
  const int n = S.n, n2 = S.n2, tid = threadIdx.x, lane = tid & 31;
  unsigned long long* lo = smem_keys;
  unsigned long long* hi = smem_keys + n2;  // W == 2 only
  unsigned short* ix = reinterpret_cast<unsigned short*>(smem_keys + (size_t)W * n2);
  if (tid == 0) s_nulls = 0;
  __syncthreads();
  const OrderLayout& L = S.L;
  for (int r = tid; r < n2; r += SMALL_NT) {
    unsigned long long k[W];
    for (int i = 0; i < W; i++) k[i] = r < n ? 0ULL : ~0ULL;  // padding rows sort behind every row
    if (r < n) {
      for (int c = 0; c < L.n; c++) {
        const bool v = pmb_valid_bit(L.valid[c], r);
        if (L.null_off[c] >= 0) put_bits<W>(k, L.null_off[c], (L.nulls_last[c] ? !v : v) ? 1ULL : 0ULL, 1);
        if (!v) {
          if (c == 0 && S.drop_nulls) atomicAdd(&s_nulls, 1);
          continue;
        }
        const unsigned long long o = order_key(pmb_load_bits(L.data[c], L.elem[c], r), L.dtype[c]);
        put_bits<W>(k, L.data_off[c], L.desc[c] ? L.hi[c] - o : o - L.lo[c], L.data_bits[c]);
      }
    }
    lo[r] = k[0];
    if (W > 1) hi[r] = k[W - 1];
    ix[r] = (unsigned short)r;
  }
  __syncthreads();
  // bitonic network; a warp's 32 pairs of a step with j <= 32 lie in its own 64 elements, so those
  // steps need no CTA barrier among them
  for (int kk = 2; kk <= n2; kk <<= 1) {
    for (int j = kk >> 1; j > 0; j >>= 1) {
      for (int t = tid; t < n2 / 2; t += SMALL_NT) {
        const int a = 2 * t - (t & (j - 1)), b = a + j;
        const bool up = (a & kk) == 0;
        if (small_less<W>(lo, hi, ix, b, a) == up) {
          const unsigned long long x = lo[a];
          lo[a] = lo[b];
          lo[b] = x;
          if (W > 1) {
            const unsigned long long y = hi[a];
            hi[a] = hi[b];
            hi[b] = y;
          }
          const unsigned short z = ix[a];
          ix[a] = ix[b];
          ix[b] = z;
        }
      }
      if (j > 32 || j == 1) __syncthreads();
      else __syncwarp();
    }
  }
  const long long total = S.drop_nulls ? n - s_nulls : n;
  const long long start = S.offset >= 0 ? min(S.offset, total) : max(0LL, total + S.offset);
  const int m = (int)(S.limit < 0 ? total - start : min(S.limit, total - start));
  if (tid == 0) *S.out_rows = (unsigned long long)m;
  // a warp fills whole validity words; its columns' loads are independent
  const GatherCols& G = S.G;
  const int words = (m + 31) / 32;
  for (int w = tid / 32; w < words; w += SMALL_NT / 32) {
    const int p = w * 32 + lane;
    const bool in = p < m;
    const int r = in ? ix[start + p] : 0;
    for (int c = 0; c < G.n; c++) {
      const int e = G.elem[c];
      const bool v = in && pmb_valid_bit(G.valid[c], r);
      uint64_t b = in ? pmb_load_bits(G.data[c], e, r) : 0;
      if (G.dec[c] >= 0 && !v) b = 0;
      if (in) {
        switch (e) {
          case 0: break;
          case 1: G.out_data[c][p] = (uint8_t)b; break;
          case 2: reinterpret_cast<uint16_t*>(G.out_data[c])[p] = (uint16_t)b; break;
          case 4: reinterpret_cast<uint32_t*>(G.out_data[c])[p] = (uint32_t)b; break;
          default: reinterpret_cast<uint64_t*>(G.out_data[c])[p] = b; break;
        }
      }
      const unsigned vw = __ballot_sync(0xffffffffu, v);
      const unsigned dw = __ballot_sync(0xffffffffu, in && e == 0 && b);
      if (lane == 0) {
        G.out_valid[c][w] = vw;
        if (e == 0) reinterpret_cast<unsigned int*>(G.out_data[c])[w] = dw;
      }
    }
  }
}

// order keys of a dtype's smallest value, and the key bits of its whole range
void full_field(int dt, unsigned long long* lo, int* bits) {
  *lo = 0;
  *bits = pmb_dtype_bits(dt);
  if (pmb_is_signed(dt)) *lo = 0x8000000000000000ULL - (1ULL << (*bits - 1));
}

// Ranks cost 8 us a million rows (20M: 205 us for the set, the ranks and the table) and 50 us for a wait
// and small kernels; a pass costs 11 us a million rows. So they are tried where two passes and more are
// saved, DICT_GAIN rows of passes in all (260 us). 20M rows by (Float64 of 8,800 values, Int32): 4240 us
// with whole keys, 2380 us so. The sample misses rare values (8,800 look like 2,900 to 4,600), hence half
// of DICT_MAX as the most that it may promise: values that do not fit cost 115 us for nothing.
constexpr int64_t DICT_ROWS = 1 << 21, DICT_GAIN = 24000000;

int blocks_for(const pmb_handle* h, int64_t threads) {
  return (int)std::max<int64_t>(1, std::min<int64_t>((threads + OR_NT - 1) / OR_NT, (int64_t)h->sm_count * 8));
}

// The lookup table of a column's ranks, when it has at most DICT_MAX distinct values (else *count stays 0).
struct OrderDict {
  unsigned int count = 0;
  const unsigned int* fps = nullptr;
  const unsigned short* codes = nullptr;
  const unsigned long long* values = nullptr;
  bool alias = false;
};
int order_dict(pmb_handle* h, const DictCol& c, int64_t n, OrderDict* d) {
  const WsMark mark = pmb_ws_mark(h);
  // cleared together: control words, ranks, fingerprints
  const size_t zero = 64 + (size_t)DICT_MAX * 4 + (size_t)DICT_SLOTS * 4;
  static_assert(DICT_SLOTS / 4 * 3 >= DICT_MAX, "the lookup table's slots");
  uint8_t* z = (uint8_t*)pmb_ws_alloc(h, zero);
  unsigned long long* seen = (unsigned long long*)pmb_ws_alloc(h, (size_t)DICT_SEEN * 8);
  unsigned long long* list = (unsigned long long*)pmb_ws_alloc(h, (size_t)DICT_MAX * 8);
  unsigned short* codes = (unsigned short*)pmb_ws_alloc(h, (size_t)DICT_SLOTS * 2);
  unsigned long long* values = (unsigned long long*)pmb_ws_alloc(h, (size_t)DICT_MAX * 8);
  if (!z || !seen || !list || !codes || !values) {  // the keys go in whole
    pmb_ws_release(h, mark);
    return PMB_OK;
  }
  DictCtl* ctl = (DictCtl*)z;
  unsigned int* rank = (unsigned int*)(z + 64);
  unsigned int* fps = rank + DICT_MAX;
  PMB_CUDA(h, cudaMemsetAsync(z, 0, zero, h->stream));
  PMB_CUDA(h, cudaMemsetAsync(seen, 0xFF, (size_t)DICT_SEEN * 8, h->stream));
  const auto collect = c.elem == 8 ? k_dict_collect<unsigned long long> : k_dict_collect<uint32_t>;
  PMB_CUDA(h, cudaFuncSetAttribute(collect, cudaFuncAttributeMaxDynamicSharedMemorySize, DICT_CTA * 8));
  pmb_kernel_begin(h, "dict_collect");
  collect<<<(unsigned)h->sm_count, DICT_NT, DICT_CTA * 8, h->stream>>>(c, n, seen, list, ctl);
  pmb_kernel_end(h);
  pmb_kernel_begin(h, "dict_rank");
  k_dict_rank<<<dim3(DICT_MAX / OR_NT, DICT_PARTS), OR_NT, 0, h->stream>>>(list, ctl, rank);
  pmb_kernel_end(h);
  pmb_kernel_begin(h, "dict_table");
  k_dict_table<<<DICT_MAX / OR_NT, OR_NT, 0, h->stream>>>(list, rank, ctl, c.dtype, fps, codes, values);
  pmb_kernel_end(h);
  PMB_CUDA(h, cudaGetLastError());
  PMB_CUDA(h, cudaMemcpyAsync(h->pinned, ctl, sizeof(DictCtl), cudaMemcpyDeviceToHost, h->stream));
  PMB_CUDA(h, cudaStreamSynchronize(h->stream));
  const DictCtl* got = (const DictCtl*)h->pinned;
  if (got->fail || got->count > DICT_MAX) {
    pmb_ws_release(h, mark);
    return PMB_OK;
  }
  d->count = got->count;
  d->fps = fps;
  d->codes = codes;
  d->values = values;
  d->alias = got->alias != 0;
  return PMB_OK;
}

// Distinct values of a sort column from its sample (Chao's estimate: the seen ones and f1^2 / 2 f2)
double sampled_distinct(const OrderRange& g, int k) {
  const double f1 = g.f1[k], f2 = g.f2[k];
  return f1 == 0 ? g.distinct[k] : g.distinct[k] + f1 * f1 / (2 * std::max(f2, 0.5));
}

// Whether k_order_small beats the general path, whose time goes by its passes. Measured for sort_columns of three
// columns, us: k_order_small of one- / two-word keys 38 / 51 up to 1024 rows, 50 / 78 to 2048, 80 / 140 to 4096,
// 146 / 280 to 8192, whatever the values; the general path 44 where all rows have one key, 73 with one pass, 85 with
// two, 106 with four, 146 with eight, 165 with nine of two-word keys. The passes follow from the values'
// ranges, which only the general path reads: floats are taken to fill their types, integers 16 bits of them.
bool small_pays(const DCol* cols, const pmb_sort_spec& s, int64_t n, int full_bits) {
  if (n <= 1 || n > SMALL_ROWS || full_bits > 128) return false;
  static constexpr int us[4][2] = {{38, 51}, {50, 78}, {80, 140}, {146, 280}};
  int size = 0, bits = 0;
  while ((1024 << size) < n) size++;
  for (int k = 0; k < s.n_by; k++) {
    const DCol& d = cols[s.by[k]];
    bits += (pmb_is_float(d.dtype) ? pmb_dtype_bits(d.dtype) : std::min(pmb_dtype_bits(d.dtype), 16)) + (d.valid != nullptr);
  }
  return us[size][full_bits > 64] <= 62 + 11 * ((bits + 7) / 8);
}

// pmb_order_columns for a table that k_order_small takes
int order_small(pmb_handle* h, const DCol* cols, int n_cols, int64_t n, const pmb_sort_spec& s, const int* desc,
                const int* nlast, pmb_result* r) {
  SmallOrder S;
  memset(&S, 0, sizeof(S));
  S.n = (int)n;
  S.n2 = 64;
  while (S.n2 < S.n) S.n2 *= 2;
  S.drop_nulls = s.drop_nulls && cols[s.by[0]].valid;
  S.offset = s.offset;
  S.limit = s.limit;
  OrderLayout& L = S.L;
  GatherCols& G = S.G;
  L.n = s.n_by;
  G.n = n_cols;
  for (int c = 0; c < n_cols; c++) G.dec[c] = -1;
  int off = 0;
  for (int k = s.n_by - 1; k >= 0; k--) {  // the most significant column highest
    const DCol& d = cols[s.by[k]];
    L.data[k] = d.data;
    L.valid[k] = d.valid;
    L.elem[k] = d.elem;
    L.dtype[k] = d.dtype;
    L.desc[k] = desc[k];
    L.nulls_last[k] = nlast[k];
    full_field(d.dtype, &L.lo[k], &L.data_bits[k]);
    L.hi[k] = L.lo[k] + (L.data_bits[k] == 64 ? ~0ULL : (1ULL << L.data_bits[k]) - 1ULL);
    L.data_off[k] = off;
    off += L.data_bits[k];
    L.null_off[k] = d.valid ? off : -1;
    off += d.valid ? 1 : 0;
    if (!pmb_is_float(d.dtype)) G.dec[s.by[k]] = k;
  }
  L.bits = off;
  S.W = off > 64 ? 2 : 1;
  // rows of the slice: known here unless rows with a null first column are dropped
  int64_t start = s.offset >= 0 ? std::min<int64_t>(s.offset, n) : std::max<int64_t>(0, n + s.offset);
  int64_t m = s.limit < 0 ? n - start : std::min<int64_t>(s.limit, n - start);
  if (S.drop_nulls) m = n;
  const int64_t words = (m + 31) / 32;
  for (int c = 0; c < n_cols; c++) {
    const int e = cols[c].elem;
    G.data[c] = cols[c].data;
    G.valid[c] = cols[c].valid;
    G.elem[c] = e;
    G.out_data[c] = (uint8_t*)pmb_ws_alloc(h, (e ? (size_t)m * e : (size_t)words * 4) + 16);
    G.out_valid[c] = (unsigned int*)pmb_ws_alloc(h, (size_t)words * 4 + 16);
    if (!G.out_data[c] || !G.out_valid[c]) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (sort outputs)");
  }
  S.out_rows = (unsigned long long*)pmb_ws_alloc(h, 16);
  if (!S.out_rows) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (sort rows)");
  const int smem = S.n2 * (8 * S.W + 2);
  pmb_kernel_begin(h, "order_small");
  if (S.W == 1) {
    PMB_CUDA(h, cudaFuncSetAttribute(k_order_small<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_order_small<1><<<1, SMALL_NT, smem, h->stream>>>(S);
  } else {
    PMB_CUDA(h, cudaFuncSetAttribute(k_order_small<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    k_order_small<2><<<1, SMALL_NT, smem, h->stream>>>(S);
  }
  pmb_kernel_end(h);
  PMB_CUDA(h, cudaGetLastError());
  if (S.drop_nulls) {
    PMB_CUDA(h, cudaMemcpyAsync(h->pinned, S.out_rows, 8, cudaMemcpyDeviceToHost, h->stream));
    PMB_CUDA(h, cudaStreamSynchronize(h->stream));
    m = (int64_t) * (unsigned long long*)h->pinned;
  }
  r->n_groups = m;
  for (int c = 0; c < n_cols; c++) {
    r->columns[c].data = G.out_data[c];
    r->columns[c].validity = (uint8_t*)G.out_valid[c];
    r->columns[c].length = m;
    r->columns[c].on_device = 1;
  }
  return PMB_OK;
}

}  // namespace

int pmb_order_columns(pmb_handle* h, const DCol* cols, int n_cols, int64_t n, const pmb_sort_spec& s, pmb_result* r) {
  if (n_cols <= 0 || n_cols > PMB_MAX_OUT || r->n_columns != n_cols)
    return pmb_fail(h, PMB_E_INVALID, "sort: 1 to 32 columns");
  if (s.n_by <= 0 || s.n_by > PMB_MAX_KEYS || !s.by) return pmb_fail(h, PMB_E_INVALID, "sort: 1 to 8 sort columns");
  for (int k = 0; k < s.n_by; k++)
    if (s.by[k] < 0 || s.by[k] >= n_cols) return pmb_fail(h, PMB_E_INVALID, "sort: sort column index out of range");
  if (n > 0xFFFFFFFELL) return pmb_fail(h, PMB_E_UNSUPPORTED, "sort: more than 2^32 - 2 rows");
  for (int c = 0; c < n_cols; c++) r->columns[c].dtype = cols[c].dtype;
  const int nb = s.n_by;
  int desc[PMB_MAX_KEYS], nlast[PMB_MAX_KEYS];
  for (int k = 0; k < nb; k++) {
    desc[k] = s.descending ? (s.descending[k] != 0) : 0;
    nlast[k] = s.nulls_last ? (s.nulls_last[k] != 0) : 0;
  }
  if (s.drop_nulls) nlast[0] = 1;  // the first column's nulls last, then cut off
  int full_bits = 0;
  for (int k = 0; k < nb; k++) {
    const DCol& d = cols[s.by[k]];
    full_bits += pmb_dtype_bits(d.dtype) + (d.valid != nullptr);
  }
  if (small_pays(cols, s, n, full_bits)) return order_small(h, cols, n_cols, n, s, desc, nlast, r);
  // ranges and null counts of the sort columns
  SortCols C;
  memset(&C, 0, sizeof(C));
  C.n = nb;
  for (int k = 0; k < nb; k++) {
    const DCol& d = cols[s.by[k]];
    C.data[k] = d.data;
    C.valid[k] = d.valid;
    C.elem[k] = d.elem;
    C.dtype[k] = d.dtype;
  }
  OrderRange got;
  memset(&got, 0, sizeof(got));
  for (int k = 0; k < PMB_MAX_KEYS; k++) got.lo[k] = ~0ULL;
  // which columns have a null at all (a column without one is gathered without its bitmap)
  unsigned int has_null[PMB_MAX_OUT];
  for (int c = 0; c < n_cols; c++) has_null[c] = cols[c].valid != nullptr;
  if (n > 0) {
    OrderRange* ro = (OrderRange*)pmb_ws_alloc(h, sizeof(OrderRange) + PMB_MAX_OUT * 4);
    if (!ro) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (sort ranges)");
    unsigned int* flags = (unsigned int*)(ro + 1);
    PMB_CUDA(h, cudaMemsetAsync(ro, 0, sizeof(OrderRange) + PMB_MAX_OUT * 4, h->stream));
    PMB_CUDA(h, cudaMemsetAsync(ro->lo, 0xFF, sizeof(ro->lo), h->stream));
    NullFlagCols V;
    memset(&V, 0, sizeof(V));
    V.n = n_cols;
    for (int c = 0; c < n_cols; c++) V.valid[c] = cols[c].valid;
    pmb_kernel_begin(h, "order_range");
    k_order_range<<<dim3((unsigned)blocks_for(h, n), n >= DICT_ROWS ? 3 : 2), OR_NT, 0, h->stream>>>(C, n, ro, V, flags);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
    PMB_CUDA(h, cudaMemcpyAsync(h->pinned, ro, sizeof(got) + PMB_MAX_OUT * 4, cudaMemcpyDeviceToHost, h->stream));
    PMB_CUDA(h, cudaStreamSynchronize(h->stream));
    memcpy(&got, h->pinned, sizeof(got));
    memcpy(has_null, h->pinned + sizeof(got), (size_t)n_cols * 4);
  }
  // field widths; rounds of at most 128 bits, cut from the least significant column up
  int nbits[PMB_MAX_KEYS], dbits[PMB_MAX_KEYS];
  for (int k = 0; k < nb; k++) {
    nbits[k] = got.nulls[k] ? 1 : 0;
    int b = 0;
    if (got.any[k]) {
      const unsigned long long span = got.hi[k] - got.lo[k];
      while (b < 64 && (span >> b) != 0) b++;
    }
    dbits[k] = b;
  }
  // the widest column by rank
  int dict_col = -1;
  OrderDict dict;
  if (n >= DICT_ROWS) {
    int bits = 0;
    for (int k = 0; k < nb; k++) {
      bits += nbits[k] + dbits[k];
      const int e = cols[s.by[k]].elem;  // (narrower columns have too few bits to gain)
      if ((e == 4 || e == 8) && got.any[k] && got.hi[k] != PMB_EMPTY64 && (dict_col < 0 || dbits[k] > dbits[dict_col])) dict_col = k;
    }
    if (dict_col >= 0) {
      const double est = sampled_distinct(got, dict_col);
      int b = 1;
      while (b < 63 && (double)(1ULL << b) < 2 * est) b++;  // (a sample sees few of the rare values)
      const int saved = (bits + 7) / 8 - (bits - dbits[dict_col] + b + 7) / 8;
      if (est <= DICT_MAX / 2 && saved >= 2 && (int64_t)saved * n >= DICT_GAIN) {
        const DCol& d = cols[s.by[dict_col]];
        const int rc = order_dict(h, DictCol{d.data, d.valid, d.elem, d.dtype}, n, &dict);
        if (rc) return rc;
      }
      if (dict.count > 0) {
        got.lo[dict_col] = 0;
        got.hi[dict_col] = dict.count - 1;
        for (b = 0; ((dict.count - 1) >> b) != 0; b++) {}
        dbits[dict_col] = b;
      } else {
        dict_col = -1;
      }
    }
  }
  struct Round {
    int first, last, bits;
  };
  std::vector<Round> rounds;  // least significant first
  for (int end = nb - 1; end >= 0;) {
    int first = end, bits = nbits[end] + dbits[end];
    while (first > 0 && bits + nbits[first - 1] + dbits[first - 1] <= 128) {
      first--;
      bits += nbits[first] + dbits[first];
    }
    rounds.push_back({first, end, bits});
    end = first - 1;
  }
  const uint64_t cap = (uint64_t)std::max<int64_t>(n, 1);
  unsigned long long* k0 = (unsigned long long*)pmb_ws_alloc(h, (size_t)2 * cap * 8 + 16);
  unsigned long long* k1 = (unsigned long long*)pmb_ws_alloc(h, (size_t)2 * cap * 8 + 16);
  unsigned int* i0 = (unsigned int*)pmb_ws_alloc(h, (size_t)cap * 4 + 16);
  unsigned int* i1 = (unsigned int*)pmb_ws_alloc(h, (size_t)cap * 4 + 16);
  unsigned int* hist = (unsigned int*)pmb_ws_alloc(h, (size_t)OR_PASSES * OR_RADIX * 4);
  if (!k0 || !k1 || !i0 || !i1 || !hist) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (sort keys)");
  const unsigned int* perm = nullptr;  // the order so far (none: row order)
  std::vector<unsigned int> hh((size_t)OR_PASSES * OR_RADIX);
  OrderLayout L;  // the last round's layout
  memset(&L, 0, sizeof(L));
  int W = 1;
  for (const Round& rd : rounds) {
    if (rd.bits == 0 || n <= 1) continue;  // every key equal: the order stays
    memset(&L, 0, sizeof(L));
    L.n = rd.last - rd.first + 1;
    L.dict = dict_col >= rd.first && dict_col <= rd.last ? dict_col - rd.first : -1;
    L.dict_slots = L.dict >= 0 ? dict_slots((int)dict.count) : 0;
    L.dict_fps = dict.fps;
    L.dict_codes = dict.codes;
    int off = 0;
    for (int k = rd.last; k >= rd.first; k--) {  // the most significant column highest
      const int i = k - rd.first;
      const DCol& d = cols[s.by[k]];
      L.data[i] = d.data;
      L.valid[i] = d.valid;
      L.elem[i] = d.elem;
      L.dtype[i] = d.dtype;
      L.desc[i] = desc[k];
      L.nulls_last[i] = nlast[k];
      L.lo[i] = got.lo[k];
      L.hi[i] = got.hi[k];
      L.data_off[i] = off;
      L.data_bits[i] = dbits[k];
      off += dbits[k];
      L.null_off[i] = nbits[k] ? off : -1;
      off += nbits[k];
    }
    L.bits = off;
    W = off > 64 ? 2 : 1;
    const int passes = (off + 7) / 8;
    PMB_CUDA(h, cudaMemsetAsync(hist, 0, (size_t)OR_PASSES * OR_RADIX * 4, h->stream));
    pmb_kernel_begin(h, "order_encode");
    if (L.dict >= 0) {
      const int smem = L.dict_slots * 6;
      const auto encode = W == 1 ? k_order_encode<1, true> : k_order_encode<2, true>;
      PMB_CUDA(h, cudaFuncSetAttribute(encode, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
      static_assert(DICT_SLOTS * 6 <= 96 << 10, "two CTAs an SM");
      encode<<<h->sm_count * 2, DICT_NT, smem, h->stream>>>(L, n, perm, k0, cap, i0, passes, hist, h->sort_status);
    } else if (W == 1) {
      k_order_encode<1, false><<<blocks_for(h, n), OR_NT, 0, h->stream>>>(L, n, perm, k0, cap, i0, passes, hist, h->sort_status);
    } else {
      k_order_encode<2, false><<<blocks_for(h, n), OR_NT, 0, h->stream>>>(L, n, perm, k0, cap, i0, passes, hist, h->sort_status);
    }
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
    const bool counts = n > PMB_SORT_NO_READBACK;
    if (counts) {
      PMB_CUDA(h, cudaMemcpyAsync(h->pinned, hist, (size_t)passes * OR_RADIX * 4, cudaMemcpyDeviceToHost, h->stream));
      PMB_CUDA(h, cudaStreamSynchronize(h->stream));
      memcpy(hh.data(), h->pinned, (size_t)passes * OR_RADIX * 4);
    }
    const int rc = pmb_sort_pairs(h, W, &k0, &k1, &i0, &i1, cap, n, passes, hist, counts ? hh.data() : nullptr,
                                  perm != nullptr, &h->sort_status);
    if (rc) return rc;
    perm = i0;  // the next round reads the rows in this order (and rewrites i0 with the same values)
  }
  // the slice of the sorted rows (rows whose first sort column is null last, when dropped)
  const int64_t total = s.drop_nulls ? n - (int64_t)got.nulls[0] : n;
  const int64_t start = s.offset >= 0 ? std::min<int64_t>(s.offset, total) : std::max<int64_t>(0, total + s.offset);
  const int64_t m = s.limit < 0 ? total - start : std::min<int64_t>(s.limit, total - start);
  GatherCols G;
  memset(&G, 0, sizeof(G));
  G.n = n_cols;
  G.keys = k0;
  G.values = dict.values;
  for (int c = 0; c < n_cols; c++) G.dec[c] = -1;
  // one round sorted every column: integer and Bool sort columns come back out of the sorted keys
  // (float keys are canonical in the key, -0.0 and NaN payloads, so floats are gathered)
  if (rounds.size() == 1 && perm != nullptr) {
    for (int k = 0; k < nb; k++) {
      const int dt = cols[s.by[k]].dtype;
      if (dt == PMB_F32 || dt == PMB_F64) {
        // by rank, unless the ranks read a value's bits differently
        if (W == 1 && k == dict_col && !dict.alias) G.dec[s.by[k]] = k - rounds[0].first;
        continue;
      }
      if (W == 1) G.dec[s.by[k]] = k - rounds[0].first;  // (two-word keys are not sorted whole)
      G.zero[s.by[k]] = 1;
    }
  }
  const int64_t words = (m + 31) / 32;
  for (int c = 0; c < n_cols; c++) {
    const int e = cols[c].elem;
    const size_t db = e ? (size_t)m * e : (size_t)words * 4;
    G.data[c] = cols[c].data;
    G.valid[c] = has_null[c] ? cols[c].valid : nullptr;
    G.elem[c] = e;
    G.out_data[c] = (uint8_t*)pmb_ws_alloc(h, db + 16);
    G.out_valid[c] = (unsigned int*)pmb_ws_alloc(h, (size_t)words * 4 + 16);
    if (!G.out_data[c] || !G.out_valid[c]) return pmb_fail(h, PMB_E_OOM, "workspace exhausted (sort outputs)");
  }
  if (m > 0) {
    pmb_kernel_begin(h, "order_gather");
    const dim3 gb((unsigned)blocks_for(h, (words + GU - 1) / GU * 32), (unsigned)n_cols);
    k_order_gather<<<gb, OR_NT, 0, h->stream>>>(G, L, perm, start, m, h->sort_status);
    pmb_kernel_end(h);
    PMB_CUDA(h, cudaGetLastError());
  }
  r->n_groups = m;
  for (int c = 0; c < n_cols; c++) {
    r->columns[c].data = G.out_data[c];
    r->columns[c].validity = (uint8_t*)G.out_valid[c];
    r->columns[c].length = m;
    r->columns[c].on_device = 1;
  }
  return PMB_OK;
}

// the end of a sorted call: outputs, then the status of the sort's bounded waits
static int order_finish(pmb_handle* h, pmb_result* r, bool to_host) {
  unsigned int* st = reinterpret_cast<unsigned int*>(h->pinned);
  *st = 0;
  if (h->sort_status) PMB_CUDA(h, cudaMemcpyAsync(st, h->sort_status, 4, cudaMemcpyDeviceToHost, h->stream));
  const int rc = pmb_finish_outputs(h, r, to_host);
  if (rc) return rc;
  PMB_CUDA(h, cudaStreamSynchronize(h->stream));
  if (*st & PMB_ST_TIMEOUT) return pmb_fail(h, PMB_E_TIMEOUT, "a bounded device wait timed out (sort)");
  return PMB_OK;
}

extern "C" int pmb_sort_columns(pmb_handle* h, const pmb_column* cols, int32_t n_cols, const pmb_sort_spec* spec,
                                int32_t output_on_device, pmb_result** out) {
  if (!h) return PMB_E_INVALID;
  if (!out) return pmb_fail(h, PMB_E_INVALID, "out is NULL");
  *out = nullptr;
  if (!spec || !cols || n_cols <= 0 || n_cols > PMB_MAX_COLS)
    return pmb_fail(h, PMB_E_INVALID, "sort: a spec and 1 to 16 columns are required");
  const int64_t n = cols[0].length;
  for (int c = 0; c < n_cols; c++) {
    if (cols[c].length != n) return pmb_fail(h, PMB_E_INVALID, "sort: columns differ in length");
    if (cols[c].dtype < PMB_BOOL || cols[c].dtype > PMB_F64) return pmb_fail(h, PMB_E_INVALID, "unknown dtype");
  }
  PMB_CUDA(h, cudaSetDevice(h->device));
  int rc = pmb_ws_begin(h);
  if (rc) return rc;
  pmb_call_begin(h);
  DCol d[PMB_MAX_COLS];
  memset(d, 0, sizeof(d));
  for (int c = 0; c < n_cols; c++) pmb_expect_column(h, cols[c], n);
  for (int c = 0; c < n_cols; c++) {
    rc = pmb_stage_column(h, cols[c], n, &d[c]);
    if (rc) return rc;
  }
  pmb_result* r = pmb_result_new(n_cols);
  if (!r) return pmb_fail(h, PMB_E_OOM, "host allocation failed");
  rc = pmb_order_columns(h, d, n_cols, n, *spec, r);
  if (!rc) rc = order_finish(h, r, output_on_device == 0);
  if (rc) {
    pmb_result_free(r);
    return rc;
  }
  r->strategy_used = PMB_STRATEGY_SORT;
  pmb_call_end(h);
  *out = r;
  return PMB_OK;
}

static int groupby_sorted(pmb_handle* h, const pmb_query* q, const pmb_column* cols, int32_t n_cols,
                          const pmb_sort_spec* spec, pmb_result** out) {
  if (!h) return PMB_E_INVALID;
  if (!out) return pmb_fail(h, PMB_E_INVALID, "out is NULL");
  *out = nullptr;
  if (!q || !spec) return pmb_fail(h, PMB_E_INVALID, "a query and a sort spec are required");
  pmb_query qd = *q;
  qd.output_on_device = 1;
  pmb_result* g = nullptr;
  bool ordered = false;
  int rc = pmb_groupby_call(h, &qd, cols, n_cols, spec, &ordered, &g);
  if (rc) return rc;
  if (ordered) {
    rc = order_finish(h, g, q->output_on_device == 0);
    if (rc) {
      pmb_result_free(g);
      return rc;
    }
    pmb_call_end(h);
    *out = g;
    return PMB_OK;
  }
  // the group-by's device columns stay in the workspace; the sort's buffers follow them (no
  // workspace reset), and its launches add to the same call's statistics
  DCol d[PMB_MAX_OUT];
  memset(d, 0, sizeof(d));
  for (int c = 0; c < g->n_columns && c < PMB_MAX_OUT; c++) {
    d[c].data = (const uint8_t*)g->columns[c].data;
    d[c].valid = g->columns[c].validity;
    d[c].dtype = g->columns[c].dtype;
    d[c].elem = pmb_dtype_bytes(g->columns[c].dtype);
    // a key column without nulls has a bitmap of ones: no null bit in the sort key, nothing to read
    if (c < q->n_keys && cols[q->key_columns[c]].validity == nullptr) d[c].valid = nullptr;
  }
  pmb_result* r = pmb_result_new(g->n_columns);
  if (!r) {
    pmb_result_free(g);
    return pmb_fail(h, PMB_E_OOM, "host allocation failed");
  }
  rc = pmb_order_columns(h, d, g->n_columns, g->n_groups, *spec, r);
  r->strategy_used = g->strategy_used;
  r->rehash_count = g->rehash_count;
  r->capacity = g->capacity;
  pmb_result_free(g);
  if (!rc) rc = order_finish(h, r, q->output_on_device == 0);
  if (rc) {
    pmb_result_free(r);
    return rc;
  }
  pmb_call_end(h);
  *out = r;
  return PMB_OK;
}

extern "C" int pmb_groupby_sorted(pmb_handle* h, const pmb_query* q, const pmb_column* cols, int32_t n_cols,
                                  const pmb_sort_spec* spec, pmb_result** out) {
  return pmb_again_uncarried(h, [&] { return groupby_sorted(h, q, cols, n_cols, spec, out); });
}
