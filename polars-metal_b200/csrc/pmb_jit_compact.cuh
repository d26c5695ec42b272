// pmb_jit_compact.cuh — the top-level filter's compaction compiled at run time for one query
// signature (NVRTC). This text follows pmb_device.cuh, the parameter block of pmb_jit_skeleton.cuh
// and a generated section that defines, for that signature and a tile of JC_TILE rows:
//   jc_issue   the bulk copies (TMA) of a whole tile's columns into a stage
//   jc_copy    plain copies of the partial last tile
//   jc_keep    the predicate of a row of a stage
//   jc_out     one warp's 32 consecutive output rows of every column, from a stage
//
// Persistent CTAs take tiles in ticket order: bulk copies into the CTA's stage, verdicts, look-back,
// output. A stage holds no registers, so an SM keeps seven tiles of 28-byte rows in flight. The kept
// rows of a tile are listed in shared memory; then every warp writes 32 output rows at a time from an
// output position that is a multiple of 32, so stores are whole aligned lines and a validity word is
// one ballot and one plain store (only a tile's first and last word are shared with its neighbours).
// What bounds it: DRAM and the tile's chain of round trips. With four rows per thread held in
// registers from the verdict to the scatter: 1288 us for 100M rows of 28 bytes (54% kept), 808 us
// here, against 666 us for the bytes alone at a copy's rate (20M rows under a profiler: DRAM 61% of its peak,
// reads 1.01 of the columns' bytes, 86% of the warps active, waiting at the tile's barriers). (Fetching the next tile ahead into a second stage was
// slower, 1.9 ms: a tile taken early publishes its count late, and every later look-back waits.)

#define JC_NT 256
#define JC_PER (JC_TILE / JC_NT)
#define JC_NC (JC_PER * (JC_NT / 32))  // warps' counts per tile

struct JCParams {
  const unsigned char* col_data[16];
  const unsigned char* col_valid[16];
  long long n_rows;
  unsigned long long* lb;      // look-back states, one per tile
  unsigned long long* ticket;  // tile ticket
  unsigned long long* n_out;   // rows kept (written by the last tile)
  unsigned int* status;
  unsigned char* out_data[16];
  unsigned int* out_valid[16];
};

// bits of 32 consecutive outputs at word w: the whole word when `full`, else OR-ed (zeroed before)
__device__ __forceinline__ void jc_word(unsigned int* words, long long w, unsigned bits, bool full) {
  if ((threadIdx.x & 31) == 0) {
    if (full) words[w] = bits;
    else if (bits) atomicOr(&words[w], bits);
  }
}

// the look-back of pmb_internal.cuh for a whole warp (NVRTC sees only this text)
__device__ __forceinline__ unsigned long long jc_lookback_warp(unsigned long long* status, long long tile,
                                                               unsigned long long count, unsigned int* st) {
  const unsigned long long VAL = (1ULL << 62) - 1;
  const int lane = threadIdx.x & 31;
  if (tile == 0) {
    if (lane == 0) atomicExch(&status[0], (2ULL << 62) | count);
    return 0;
  }
  if (lane == 0) atomicExch(&status[tile], (1ULL << 62) | count);
  unsigned long long excl = 0;
  long long top = tile - 1;
  unsigned spins = 0;
  for (;;) {
    const long long t = top - lane;
    const unsigned long long s = t >= 0 ? *((volatile unsigned long long*)&status[t]) : (2ULL << 62);
    const unsigned flag = (unsigned)(s >> 62);
    const unsigned incl = __ballot_sync(0xffffffffu, flag == 2u), none = __ballot_sync(0xffffffffu, flag == 0u);
    const int first = incl ? __ffs(incl) - 1 : 32;
    const unsigned need = first == 32 ? 0xffffffffu : (0xffffffffu >> (31 - first));
    if (none & need) {
      if (++spins > PMB_SPIN_LIMIT) {
        if (lane == 0) atomicOr(st, PMB_ST_TIMEOUT);
        return 0;
      }
      continue;
    }
    unsigned long long v = lane <= first ? (s & VAL) : 0ULL;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    excl += v;
    if (first < 32) break;
    top -= 32;
  }
  if (lane == 0) atomicExch(&status[tile], (2ULL << 62) | (excl + count));
  return excl;
}

extern "C" __global__ void __launch_bounds__(JC_NT) pmb_jit_compact(const __grid_constant__ JCParams P) {
  extern __shared__ __align__(128) unsigned char st[];  // the stage
  __shared__ unsigned long long bar;
  __shared__ long long s_tile;
  __shared__ unsigned short s_row[JC_TILE];  // the tile's kept rows, in order
  __shared__ unsigned s_cnt[JC_NC];
  __shared__ unsigned long long s_base;
  __shared__ int s_abort;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const unsigned lt = (1u << lane) - 1u;
  const long long n_tiles = (P.n_rows + JC_TILE - 1) / JC_TILE, n_full = P.n_rows / JC_TILE;
  const unsigned long long pol = pmb_policy_evict_first();
  // thread 0: the next tile into the stage
  auto take = [&]() {
    const long long t = (long long)atomicAdd(P.ticket, 1ULL);
    s_tile = t;
    if (t < n_full) jc_issue(P, st, t, &bar, pol);
  };
  if (tid == 0) {
    s_abort = 0;
    mbar_init(&bar, 1);
    mbar_fence_init();
    take();
  }
  __syncthreads();
  for (unsigned parity = 0;;) {
    const long long tile = s_tile;
    if (tile >= n_tiles) break;
    const int rows = (int)min((long long)JC_TILE, P.n_rows - tile * JC_TILE);
    if (rows == JC_TILE) {
      if (!mbar_wait_bounded(&bar, parity)) s_abort = 1;
      parity ^= 1u;
    } else {
      jc_copy(P, st, tile * JC_TILE, rows);
    }
    __syncthreads();
    if (s_abort) {  // (the copy that did not arrive has been waited for up to the limit)
      if (tid == 0) atomicOr(P.status, PMB_ST_TIMEOUT);
      return;
    }
    unsigned kept[JC_PER];  // ballots of the warp's rows
#pragma unroll
    for (int j = 0; j < JC_PER; j++) {
      const int lr = j * JC_NT + tid;
      kept[j] = __ballot_sync(0xffffffffu, lr < rows && jc_keep(st, lr));
      if (lane == 0) s_cnt[j * (JC_NT / 32) + warp] = (unsigned)__popc(kept[j]);
    }
    __syncthreads();
    // every warp scans the counts (JC_NC <= 32) and lists its rows
    const unsigned c = lane < JC_NC ? s_cnt[lane] : 0u;
    unsigned x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
      if (lane >= o) x += y;
    }
    const int total = (int)__shfl_sync(0xffffffffu, x, 31);
    x -= c;
#pragma unroll
    for (int j = 0; j < JC_PER; j++) {
      const unsigned first = __shfl_sync(0xffffffffu, x, j * (JC_NT / 32) + warp);
      if ((kept[j] >> lane) & 1u) s_row[first + __popc(kept[j] & lt)] = (unsigned short)(j * JC_NT + tid);
    }
    if (warp == 0) {
      const unsigned long long base = jc_lookback_warp(P.lb, tile, (unsigned long long)total, P.status);
      if (lane == 0) {
        s_base = base;
        if (tile == n_tiles - 1) *P.n_out = base + total;
      }
    }
    __syncthreads();
    const long long base = (long long)s_base;
    for (int i0 = warp * 32 - (int)(base & 31); i0 < total; i0 += JC_NT) {
      const int i = i0 + lane;
      const bool in = i >= 0 && i < total;
      jc_out(P, st, in ? s_row[i] : 0, in, base + i, (base + i0) >> 5, i0 >= 0 && i0 + 32 <= total);
    }
    __syncthreads();
    if (tid == 0) {
      fence_proxy_async();  // the CTA's reads of the stage come before the copies' writes
      take();
    }
    __syncthreads();
  }
}
