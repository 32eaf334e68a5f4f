// local_sort.cuh -- CTA-local completion of the batch sort.
//
// The device-wide sort (Trie::sort_unique) refines ties one 8-nibble chunk
// at a time.  Once every still-tied run of positions holds at most
// kSortLocalCap keys, one CTA per run finishes it in shared memory: per
// chunk, a stable block radix sort of (tie-group rank << 32 | chunk) on the
// digits that vary, until no ties are left or the key length breaks them.
// Results are identical to continuing device-wide: the order is
// lexicographic (terminator before nibble 0) and equal keys keep their batch
// order, so the last one is the kept occurrence.
#pragma once
#include "trie_kernels.cuh"

namespace gmpt {

constexpr int kSortLocalCap = 2048;
constexpr int kSortLocalThreads = 256;
// Runs by size, each with CTAs that fit it: up to 32 positions a warp
// (k_local_sort_warp), up to kSortSmallCap two warps, the rest eight.  Word
// keys leave tens of thousands of runs, most of a few positions: in CTAs of
// 256 threads each, 512K vocabulary keys took 1.95 ms, 0.60 so; the 1.7K-key runs
// of a 16M-key load 2.24 ms, 1.25 with their gathers in flight together.
constexpr int kSortSmallCap = 512, kSortSmallThreads = 64, kSortWarpCap = 32;
constexpr int kSortIptMax = 8;
static_assert(kSortLocalCap == kSortIptMax * kSortLocalThreads && kSortSmallCap == kSortIptMax * kSortSmallThreads, "");

// groups no larger than this are ordered by direct counting instead of radix passes
constexpr uint32_t kSortSmallGroup = 32;

template <int kCap, int kThreads>
struct LocalSortSmem {
  static constexpr int kWarps = kThreads / 32;
  uint64_t key[2][kCap];
  uint32_t val[2][kCap];
  union {
    uint16_t cnt[kWarps][256];  // radix pass: per-warp digit counts, then offsets (<= kCap)
    uint16_t gbeg[kCap];        // small-group pass: first position of every tied group
  };
  uint32_t warp_tmp[kWarps + 1];
  unsigned long long mask;
  uint32_t maxlen;
  uint32_t maxg;
  static_assert(kWarps * 256 == kCap, "gbeg shares the radix counters' space");
};

// block-wide exclusive scan of one value per thread
template <int kWarps>
__device__ __forceinline__ uint32_t cta_excl_scan(uint32_t v, uint32_t *tmp, uint32_t &total) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t incl = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    uint32_t u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) tmp[wid] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t run = 0;
    for (int w = 0; w < kWarps; ++w) {
      uint32_t c = tmp[w];
      tmp[w] = run;
      run += c;
    }
    tmp[kWarps] = run;
  }
  __syncthreads();
  total = tmp[kWarps];
  uint32_t r = tmp[wid] + incl - v;
  __syncthreads();
  return r;
}

// one stable pass on digit `shift` of key[src] -> key[src ^ 1]
template <int kCap, int kThreads>
__device__ __forceinline__ void cta_radix_pass(LocalSortSmem<kCap, kThreads> &L, int src, int m, int shift) {
  constexpr int kWarps = kThreads / 32, kDigits = 256 / kThreads;
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int i = threadIdx.x; i < kWarps * 256; i += kThreads) (&L.cnt[0][0])[i] = 0;
  static_assert(kCap < 65536, "digit offsets are 16-bit");
  __syncthreads();
  const unsigned lt = (1u << lane) - 1u;
  const int rounds = (m + kThreads - 1) / kThreads, base = wid * rounds * 32;  // a warp's share, in order
  uint32_t rk[kSortIptMax];
#pragma unroll
  for (int r = 0; r < kSortIptMax; ++r) {
    if (r >= rounds) break;
    int k = base + r * 32 + lane;
    bool ok = k < m;
    uint32_t d = ok ? (uint32_t)((L.key[src][k] >> shift) & 0xFF) : (256u + lane);
    unsigned peers = __match_any_sync(0xffffffffu, d);
    uint32_t old = ok ? L.cnt[wid][d] : 0;
    __syncwarp();
    if (ok && (int)lane == __ffs(peers) - 1) L.cnt[wid][d] = (uint16_t)(old + __popc(peers));
    __syncwarp();
    rk[r] = old + __popc(peers & lt);
  }
  __syncthreads();
  // digit-major exclusive offsets: thread t owns digits t * kDigits and on
  uint32_t tot = 0;
#pragma unroll
  for (int q = 0; q < kDigits; ++q)
    for (int w = 0; w < kWarps; ++w) tot += L.cnt[w][threadIdx.x * kDigits + q];
  uint32_t all;
  uint32_t run = cta_excl_scan<kWarps>(tot, L.warp_tmp, all);
#pragma unroll
  for (int q = 0; q < kDigits; ++q)
    for (int w = 0; w < kWarps; ++w) {
      uint32_t c = L.cnt[w][threadIdx.x * kDigits + q];
      L.cnt[w][threadIdx.x * kDigits + q] = (uint16_t)run;
      run += c;
    }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < kSortIptMax; ++r) {
    if (r >= rounds) break;
    int k = base + r * 32 + lane;
    if (k < m) {
      uint64_t kk = L.key[src][k];
      uint32_t d = (uint32_t)((kk >> shift) & 0xFF);
      uint32_t dst = L.cnt[wid][d] + rk[r];
      L.key[src ^ 1][dst] = kk;
      L.val[src ^ 1][dst] = L.val[src][k];
    }
  }
  __syncthreads();
}

// Runs of at most kSortWarpCap positions, a warp each: lane k holds position
// k's item; per chunk the lanes of a tied group are ranked by counting.
__global__ void __launch_bounds__(256) k_local_sort_warp(TrieView tv, const uint32_t *seg_start, const uint32_t *seg_end,
                                                         int runs, int c0, uint32_t *order, uint8_t *eqprev,
                                                         const uint64_t *koff, const uint32_t *klen) {
  constexpr unsigned kAll = 0xffffffffu;
  const int run = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (run >= runs) return;
  const uint32_t a = seg_start[run];
  const int m = (int)(seg_end[run] - a);
  if (m > kSortWarpCap || m < 2) return;
  const bool on = lane < m;
  uint32_t it = on ? order[a + lane] : 0u;
  uint32_t len = on ? klen[it] : 0u;
  const uint32_t maxlen = __reduce_max_sync(kAll, len);
  uint64_t ko = on ? koff[it] : 0ull;
  uint32_t group = on ? 0u : 1u;  // first position of the lane's tied group (lanes past m: one of their own)
  const int nchunks = (int)((maxlen + 7) / 8);
  // the last pass is the key length; a run whose keys all end before chunk c0
  // (longer keys elsewhere kept the batch sort going) still takes it
  for (int c = min(c0, nchunks); c <= nchunks; ++c) {
    const uint32_t ch = !on ? 0u : (c < nchunks ? key_chunk(tv.keys, ko, len, c) : len);
    // place inside the group: members with a smaller chunk, or an equal one and before this lane
    uint32_t less = 0, eq = 0;
    for (int j = 0; j < m; ++j) {
      const uint32_t gj = __shfl_sync(kAll, group, j), cj = __shfl_sync(kAll, ch, j);
      if (gj == group && cj < ch) ++less;
      if (gj == group && cj == ch && j < lane) ++eq;
    }
    const uint32_t g2 = group + less, dst = on ? g2 + eq : (uint32_t)lane;
    // lane dst takes this lane's item
    uint32_t from = 0;
    for (int j = 0; j < 32; ++j)
      if (__shfl_sync(kAll, dst, j) == (uint32_t)lane) from = (uint32_t)j;
    it = __shfl_sync(kAll, it, from);
    len = __shfl_sync(kAll, len, from);
    ko = __shfl_sync(kAll, ko, from);
    group = __shfl_sync(kAll, on ? g2 : (uint32_t)kSortWarpCap, from);
    const uint32_t gp = __shfl_up_sync(kAll, group, 1);
    if (!__any_sync(kAll, on && lane > 0 && gp == group)) break;  // no ties left
  }
  const uint32_t gp = __shfl_up_sync(kAll, group, 1);
  if (on) {
    order[a + lane] = it;
    eqprev[a + lane] = lane > 0 && gp == group ? 1 : 0;
  }
}

// seg_start / seg_end: position runs still tied before chunk c
// (runs of other sizes than (kMin, kCap] are another launch's)
template <int kMin, int kCap, int kThreads>
__global__ void __launch_bounds__(kThreads) k_local_sort(TrieView tv, const uint32_t *seg_start,
                                                         const uint32_t *seg_end, int c0, uint32_t *order,
                                                         uint8_t *eqprev, const uint64_t *koff, const uint32_t *klen) {
  constexpr int kWarps = kThreads / 32;
  extern __shared__ __align__(16) uint8_t smem_raw[];
  using Smem = LocalSortSmem<kCap, kThreads>;
  Smem &L = *reinterpret_cast<Smem *>(smem_raw);
  const uint32_t a = seg_start[blockIdx.x];
  const int m = (int)(seg_end[blockIdx.x] - a);
  if (m > kCap || m <= kMin) return;
  const int ipt = (m + kThreads - 1) / kThreads;  // items per thread
  if (threadIdx.x == 0) L.maxlen = 0;
  __syncthreads();
  for (int k = threadIdx.x; k < m; k += kThreads) {
    uint32_t it = order[a + k];
    L.val[0][k] = it;
    atomicMax(&L.maxlen, klen[it]);
  }
  __syncthreads();
  const int nchunks = (int)((L.maxlen + 7) / 8);
  // keys that all end before chunk c0 are still parted by their length
  const int first = min(c0, nchunks);
  int src = 0;
  // tied[k] == 1: item k equals item k-1 on everything compared so far
  // (all items start tied: they share the chunks before `first`)
  for (int c = first; c <= nchunks; ++c) {
    // group rank of each item = number of group starts before it
    // (thread t owns items [t * ipt, t * ipt + ipt))
    uint32_t starts = 0;
    uint8_t st[kSortIptMax], tp[kSortIptMax + 1];
#pragma unroll
    for (int r = 0; r <= kSortIptMax; ++r) {
      if (r > ipt) break;
      int k = threadIdx.x * ipt + r;  // r == ipt: the next thread's first item
      bool tied_prev;
      if (c == first)
        tied_prev = k > 0 && k < m;
      else
        tied_prev = k > 0 && k < m && L.key[src][k] == L.key[src][k - 1];
      tp[r] = tied_prev ? 1 : 0;
      if (r == ipt) break;
      st[r] = (k < m && !tied_prev) ? 1 : 0;
      starts += st[r];
    }
    uint32_t ngroups;
    uint32_t rank = cta_excl_scan<kWarps>(starts, L.warp_tmp, ngroups);
    if (ngroups == (uint32_t)m) break;  // every key distinct
    // build (rank, chunk) keys in the current order
    if (threadIdx.x == 0) {
      L.mask = 0;
      L.maxg = 0;
    }
    __syncthreads();
    uint64_t acc = 0, k0 = 0;
    uint16_t gid[kSortIptMax];
    // gathers of all items of the thread in flight together: offsets and
    // lengths, then the chunks (an item already alone in its group keeps its
    // place whatever its chunk: it gathers nothing)
    uint64_t ko[kSortIptMax];
    uint32_t kl[kSortIptMax];
#pragma unroll
    for (int r = 0; r < kSortIptMax; ++r) {
      const int k = threadIdx.x * ipt + r;
      const bool need = r < ipt && k < m && (tp[r] || tp[r + 1]);
      const uint32_t it = need ? L.val[src][k] : 0u;
      ko[r] = need ? koff[it] : 0ull;
      kl[r] = need ? klen[it] : 0u;
    }
    uint32_t ch[kSortIptMax];
#pragma unroll
    for (int r = 0; r < kSortIptMax; ++r)
      ch[r] = c < nchunks ? key_chunk(tv.keys, ko[r], kl[r], c) : kl[r];  // length 0: no load, chunk 0
#pragma unroll
    for (int r = 0; r < kSortIptMax; ++r) {
      const int k = threadIdx.x * ipt + r;
      gid[r] = 0;
      if (r >= ipt || k >= m) continue;
      rank += st[r];
      gid[r] = (uint16_t)(rank - 1);
      if (c > first && st[r]) L.gbeg[rank - 1] = (uint16_t)k;
      L.key[src][k] = ((uint64_t)(rank - 1) << 32) | ch[r];
    }
    if (c > first && threadIdx.x == 0) L.gbeg[ngroups] = (uint16_t)m;  // ngroups < m <= kSortLocalCap
    __syncthreads();
    if (c > first) {
      // Largest tied group: when every group is small (the usual tail, a
      // few pairs among singletons), each item finds its place in its group
      // by counting the members that order before it -- one pass instead
      // of one radix pass per varying byte of (rank, chunk).
      uint32_t gmax = 0;
#pragma unroll
      for (int r = 0; r < kSortIptMax; ++r) {
        const int k = threadIdx.x * ipt + r;
        if (r < ipt && k < m && st[r]) gmax = max(gmax, (uint32_t)(L.gbeg[gid[r] + 1] - L.gbeg[gid[r]]));
      }
      gmax = __reduce_max_sync(0xffffffffu, gmax);
      if ((threadIdx.x & 31) == 0 && gmax) atomicMax(&L.maxg, gmax);
      __syncthreads();
      if (L.maxg <= kSortSmallGroup) {
#pragma unroll
        for (int r = 0; r < kSortIptMax; ++r) {
          const int k = threadIdx.x * ipt + r;
          if (r >= ipt || k >= m) continue;
          const uint64_t key = L.key[src][k];
          const uint32_t b = L.gbeg[gid[r]], e = L.gbeg[gid[r] + 1];
          uint32_t pos = b;
          for (uint32_t j = b; j < e; ++j) {  // stable: equal chunks keep their order
            const uint64_t kj = L.key[src][j];
            pos += (kj < key || (kj == key && j < (uint32_t)k)) ? 1u : 0u;
          }
          L.key[src ^ 1][pos] = key;
          L.val[src ^ 1][pos] = L.val[src][k];
        }
        src ^= 1;
        __syncthreads();
        continue;
      }
    }
    k0 = L.key[src][0];
    for (int k = threadIdx.x; k < m; k += kThreads) acc |= L.key[src][k] ^ k0;
    for (int o = 16; o; o >>= 1) acc |= __shfl_xor_sync(0xffffffffu, acc, o);
    if ((threadIdx.x & 31) == 0 && acc) atomicOr(&L.mask, (unsigned long long)acc);
    __syncthreads();
    uint64_t mask = L.mask;
    {
      // nibbles that vary move to the low end of every key when that saves
      // digit passes (the order and the equalities between keys are kept;
      // the keys are rebuilt from scratch for the next chunk)
      uint64_t nmask = 0;
      int nv = 0, bytes = 0;
      for (int k = 0; k < 16; ++k)
        if ((mask >> (4 * k)) & 0xFull) {
          nmask |= 0xFull << (4 * k);
          ++nv;
        }
      for (int b = 0; b < 8; ++b) bytes += ((mask >> (8 * b)) & 0xFFull) ? 1 : 0;
      if ((4 * nv + 7) / 8 < bytes) {
        for (int k = threadIdx.x; k < m; k += kThreads) {
          const uint64_t x = L.key[src][k];
          uint64_t out = 0;
          for (int q = 15; q >= 0; --q)
            if ((nmask >> (4 * q)) & 0xFull) out = (out << 4) | ((x >> (4 * q)) & 0xFull);
          L.key[src][k] = out;
        }
        mask = nv >= 16 ? ~0ull : ((1ull << (4 * nv)) - 1);
        __syncthreads();
      }
    }
    for (int shift = 0; shift < 64; shift += 8) {
      if (((mask >> shift) & 0xFF) == 0) continue;
      cta_radix_pass<kCap, kThreads>(L, src, m, shift);
      src ^= 1;
    }
  }
  // final ties are exact duplicates (every chunk and the length equal)
  __syncthreads();
  for (int k = threadIdx.x; k < m; k += kThreads) {
    order[a + k] = L.val[src][k];
    eqprev[a + k] = (k > 0 && L.key[src][k] == L.key[src][k - 1]) ? 1 : 0;
  }
}

// positions of each still-tied run (called with the sort_flags scan)
__global__ void k_sort_runs(const unsigned long long *flags, const unsigned long long *pos, const uint8_t *eqprev,
                            int n, uint32_t *seg_start, uint32_t *seg_end) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  unsigned long long f = flags[p];
  if (!(f & 1ull)) return;
  uint32_t seg = (uint32_t)(pos[p] >> 32) + (uint32_t)(f >> 32) - 1u;
  if (f >> 32) seg_start[seg] = (uint32_t)p;
  if (!eqprev[p + 1]) seg_end[seg] = (uint32_t)p + 1;
}

// longest run; the runs are counted in the high half of *total
__global__ void k_run_max(const uint32_t *start, const uint32_t *end, const unsigned long long *total, uint32_t *out) {
  const uint32_t S = (uint32_t)(*total >> 32);
  uint32_t v = 0;
  for (uint32_t s = blockIdx.x * blockDim.x + threadIdx.x; s < S; s += gridDim.x * blockDim.x)
    v = max(v, end[s] - start[s]);
  const uint32_t w = __reduce_max_sync(0xffffffffu, v);
  if ((threadIdx.x & 31) == 0 && w) atomicMax(out, w);
}

}  // namespace gmpt
