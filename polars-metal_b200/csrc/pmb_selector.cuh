// pmb_selector.cuh — device side of the strategy selector shared by its own kernels
// (pmb_learned.cu) and the sampling kernels every group-by starts with (pmb_groupby.cu): the
// 4096-row key sample, its sketch features, and the network of one query.
#pragma once

#include "pmb_groupby.h"

namespace {

constexpr int NF = PMB_SELECTOR_FEATURES;
constexpr int NH = PMB_SELECTOR_HIDDEN;
constexpr int NO = PMB_SELECTOR_OUTPUTS;
constexpr int NS = PMB_SELECTOR_STRATEGIES;  // outputs 0..NS-1: strategy scores; output NS: log2(groups)
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + NH * NF, OFF_W2 = OFF_B1 + NH, OFF_B2 = OFF_W2 + NH * NH,
              OFF_W3 = OFF_B2 + NH, OFF_B3 = OFF_W3 + NO * NH, N_PARAMS = OFF_B3 + NO;
static_assert(N_PARAMS == PMB_SELECTOR_PARAMS, "parameter layout");

constexpr int SAMPLE = 4096;
constexpr int F_NT = 1024;
constexpr int TSLOTS = 8192;  // sample counts: slots of a 32-bit key fingerprint and a count, dynamic smem
constexpr int HLL = 256;
constexpr int BUCKETS = 1024;

__device__ __forceinline__ float lg2p1(double x) { return (float)log2(x + 1.0); }

// sample i of query q (rows evenly spaced over the input): its key hash, never 0, or 0 when the
// filter drops the row or i is past the sample; `nul` tells whether a key column is null there.
// One thread per sample, so the sample's loads are all in flight at once.
__device__ __forceinline__ void sample_one(const DQuery& q, int i, unsigned long long& hv, unsigned char& nul) {
  hv = 0ULL;
  nul = 0;
  const int64_t n = q.n_rows;
  const int m = (int)(n < SAMPLE ? n : SAMPLE);
  if (i >= m) return;
  const TileCtx t{nullptr, nullptr, nullptr, 0};
  const int64_t r = (int64_t)((__int128)i * n / m);  // evenly spaced rows
  if (q.prog.n_ops > 0 && !eval_keep(q, t, r)) return;
  bool anynull = false;
  for (int k = 0; k < q.n_keys; k++) anynull |= !tc_isvalid(q, t, q.key[k].col, r);
  unsigned long long lo, hi = 0;
  if (q.key_bits > 64) {
    Key128 kk = pack_key128(q, t, r);
    lo = kk.lo;
    hi = kk.hi;
  } else {
    lo = pack_key64(q, t, r);
  }
  hv = pmb_fmix64(lo ^ pmb_fmix64(hi + 0x9E3779B97F4A7C15ULL)) | 1ULL;  // never 0 (empty)
  nul = anynull ? 1 : 0;
}

// the features of query q into out[NF] from its samples (hs, ns: SAMPLE entries written by
// sample_one); called by one whole CTA of F_NT threads with TSLOTS words of its dynamic shared memory
__device__ __forceinline__ void features_body(const DQuery& q, const unsigned long long* __restrict__ hs,
                                              const unsigned char* __restrict__ ns, float* out,
                                              unsigned long long* s_slot) {
  __shared__ unsigned int s_hll[HLL];
  __shared__ unsigned int s_bkt[BUCKETS];
  __shared__ unsigned int s_acc[16];
  __shared__ double s_z;
  __shared__ int s_zeros;
  const int tid = threadIdx.x;
  // fingerprints, then counts: two 32-bit tables, so that a count is a native shared add (a 64-bit one is
  // a compare-and-swap loop, on which the samples of a few keys queued for 40 us)
  unsigned int* s_fp = reinterpret_cast<unsigned int*>(s_slot);
  unsigned int* s_num = s_fp + TSLOTS;
  for (int i = tid; i < TSLOTS; i += F_NT) s_slot[i] = 0ULL;
  for (int i = tid; i < HLL; i += F_NT) s_hll[i] = 0u;
  for (int i = tid; i < BUCKETS; i += F_NT) s_bkt[i] = 0u;
  if (tid < 16) s_acc[tid] = 0u;
  __syncthreads();
  const int64_t n = q.n_rows;
  const int m = (int)(n < SAMPLE ? n : SAMPLE);
  const bool pred = q.prog.n_ops > 0;
  for (int i = tid; i < m; i += F_NT) {
    const unsigned long long h = hs[i];
    if (h == 0ULL) continue;  // dropped by the filter
    atomicAdd(&s_acc[0], 1u);  // kept
    if (ns[i]) atomicAdd(&s_acc[1], 1u);
    // HyperLogLog register: index from the top 8 bits, rank of the rest
    const unsigned reg = (unsigned)(h >> 56);
    const unsigned rank = (unsigned)__clzll((h << 8) | 0xFFULL) + 1u;
    atomicMax(&s_hll[reg], rank);
    atomicAdd(&s_bkt[(h >> 20) & (BUCKETS - 1)], 1u);
    // exact counts by 32-bit fingerprint (a collision among 4096 samples is rare and only blurs a
    // feature)
    const unsigned fp = (unsigned)(h >> 32) | 1u;
    unsigned s = (unsigned)(h >> 11) & (TSLOTS - 1);
    for (int p = 0; p < TSLOTS; p++) {
      unsigned cur = *reinterpret_cast<volatile unsigned int*>(&s_fp[s]);
      if (cur == 0u) cur = atomicCAS(&s_fp[s], 0u, fp);
      if (cur == 0u || cur == fp) {
        atomicAdd(&s_num[s], 1u);
        break;
      }
      s = (s + 1) & (TSLOTS - 1);
    }
  }
  __syncthreads();
  // frequency profile of the sample keys (per-thread counts, one shared atomic per warp and bin:
  // a shared atomic per key and bin serialised the CTA on ten addresses)
  unsigned cnt[7] = {0, 0, 0, 0, 0, 0, 0}, top = 0, btop = 0;
  for (int i = tid; i < TSLOTS; i += F_NT) {
    const unsigned c = s_num[i];
    if (!c) continue;
    cnt[0]++;  // distinct
    cnt[1] += c == 1;
    cnt[2] += c == 2;
    cnt[3] += c > 2 && c <= 4;
    cnt[4] += c > 4 && c <= 8;
    cnt[5] += c > 8;
    top = max(top, c);
  }
  for (int i = tid; i < BUCKETS; i += F_NT) {
    cnt[6] += s_bkt[i] != 0u;
    btop = max(btop, s_bkt[i]);
  }
#pragma unroll
  for (int i = 0; i < 7; i++) cnt[i] = __reduce_add_sync(0xffffffffu, cnt[i]);
  top = __reduce_max_sync(0xffffffffu, top);
  btop = __reduce_max_sync(0xffffffffu, btop);
  if ((tid & 31) == 0) {
#pragma unroll
    for (int i = 0; i < 6; i++) atomicAdd(&s_acc[2 + i], cnt[i]);
    atomicMax(&s_acc[8], top);
    atomicAdd(&s_acc[9], cnt[6]);
    atomicMax(&s_acc[10], btop);
  }
  // HyperLogLog sums by warp 0: the terms are powers of two
  if (tid < 32) {
    double z = 0.0;
    int zeros = 0;
    for (int i = tid; i < HLL; i += 32) {
      z += ldexp(1.0, -(int)s_hll[i]);
      zeros += s_hll[i] == 0;
    }
    for (int o = 16; o; o >>= 1) {
      z += __shfl_xor_sync(0xffffffffu, z, o);
      zeros += __shfl_xor_sync(0xffffffffu, zeros, o);
    }
    if (tid == 0) {
      s_z = z;
      s_zeros = zeros;
    }
  }
  __syncthreads();
  if (tid == 0) {
    const double kept = s_acc[0], mk = kept > 0 ? kept : 1.0;
    const double d = s_acc[2], f1 = s_acc[3], f2 = s_acc[4];
    // HyperLogLog estimate (Flajolet et al. 2007) with linear counting for small ranges
    const double z = s_z;
    const int zeros = s_zeros;
    double hll = (0.7213 / (1.0 + 1.079 / HLL)) * HLL * HLL / z;
    if (hll <= 2.5 * HLL && zeros) hll = HLL * log((double)HLL / zeros);
    const double neff = (double)n * (m > 0 ? kept / m : 0.0);
    const double gee = kept > 0 ? sqrt(neff / mk) * f1 + (d - f1) : 0.0;
    const double chao = d + f1 * f1 / (2.0 * (f2 > 0 ? f2 : 1.0));
    float* o = out;
    o[0] = lg2p1((double)n) / 32.f;
    o[1] = (q.packed ? (int)q.packed : q.key_bits) / 128.f;  // by the key's types
    o[2] = (float)(s_acc[1] / mk);
    o[3] = m > 0 ? (float)(kept / m) : 0.f;
    o[4] = (float)(d / mk);
    o[5] = (float)(f1 / mk);
    o[6] = (float)(f2 / mk);
    o[7] = (float)(s_acc[5] / mk);
    o[8] = (float)(s_acc[6] / mk);
    o[9] = (float)(s_acc[7] / mk);
    o[10] = (float)(s_acc[8] / mk);
    o[11] = s_acc[9] / (float)BUCKETS;
    o[12] = lg2p1(s_acc[10]) / 12.f;
    o[13] = lg2p1(hll) / 13.f;
    o[14] = lg2p1(gee) / 32.f;
    o[15] = lg2p1(chao) / 32.f;
    o[16] = lg2p1(neff) / 32.f;
    o[17] = q.rec_bytes / 256.f;
    o[18] = q.n_fields / 24.f;
    o[19] = q.n_aggs / 24.f;
    o[20] = pred ? 1.f : 0.f;
    o[21] = q.n_keys / 8.f;
    o[22] = (kept > 0 && d == kept) ? 1.f : 0.f;
    o[23] = 1.f;
  }
}

// The network for one query by a CTA of F_NT threads: the weights come into shared memory with
// coalesced loads (transposed, so that neighbouring units read neighbouring words), then unit j
// sums its inputs in the order of mlp_layers (the same fused multiply-adds, the same result).
constexpr int MLP_ROW = NH + 1;
constexpr int MLP_WORDS = (NF + NH) * MLP_ROW + NO * NH + 2 * NH + NO;
__device__ __forceinline__ void mlp_load(const float* __restrict__ P, float* w) {
  for (int i = threadIdx.x; i < NH * NF; i += F_NT) w[(i % NF) * MLP_ROW + i / NF] = P[OFF_W1 + i];
  float* w2 = w + NF * MLP_ROW;
  for (int i = threadIdx.x; i < NH * NH; i += F_NT) w2[(i % NH) * MLP_ROW + i / NH] = P[OFF_W2 + i];
  float* w3 = w2 + NH * MLP_ROW;
  for (int i = threadIdx.x; i < NO * NH; i += F_NT) w3[i] = P[OFF_W3 + i];
  float* b = w3 + NO * NH;
  for (int i = threadIdx.x; i < NH; i += F_NT) {
    b[i] = P[OFF_B1 + i];
    b[NH + i] = P[OFF_B2 + i];
  }
  if (threadIdx.x < NO) b[2 * NH + threadIdx.x] = P[OFF_B3 + threadIdx.x];
}
__device__ __forceinline__ void mlp_run(const float* w, const float* x, float* h1, float* h2, float* out) {
  const int j = threadIdx.x;
  const float *w2 = w + NF * MLP_ROW, *w3 = w2 + NH * MLP_ROW, *b = w3 + NO * NH;
  if (j < NH) {
    float a = b[j];
    for (int i = 0; i < NF; i++) a = fmaf(w[i * MLP_ROW + j], x[i], a);
    h1[j] = fmaxf(a, 0.f);
  }
  __syncthreads();
  if (j < NH) {
    float a = b[NH + j];
    for (int k = 0; k < NH; k++) a = fmaf(w2[k * MLP_ROW + j], h1[k], a);
    h2[j] = fmaxf(a, 0.f);
  }
  __syncthreads();
  if (j < NO) {
    float c = b[2 * NH + j];
    for (int k = 0; k < NH; k++) c = fmaf(w3[j * NH + k], h2[k], c);
    out[j] = c;
  }
}

}  // namespace
