// grid_hash.cuh -- PhaseHC of a small or middle dirty list inside one
// cooperative launch: k_hash_grid (a hash call's whole pass) and k_block (the
// hash phases of a persistent block update) share it.
//
// A pass over a few thousand nodes is a chain of latencies, not throughput:
// level after level as separate launches cost the host round trip that sizes
// them, a launch gap each, and the slowest node of every level.  Here the
// only order kept is child before parent:
//   1. every leaf (and extension over a clean branch) is hashed; every dirty
//      branch counts its dirty branch children and tells them who it is
//   2. while many branches are ready (no dirty child left), a wave hashes them
//      a pair of lanes each and makes parents ready; then a warp takes each
//      ready branch, hashes it with the extension above it, and the warp that
//      finishes a parent's last child goes on to the parent, up to the root.
// No warp waits for another inside a phase; phases end at a grid barrier with
// a bounded wait.
//
// A hash call of 7.7K dirty nodes of a 1M-key trie takes 141 us so, 178 as a
// launch per nibble depth; of 3.8K nodes of random keys 109 and 180 (larger
// lists at kGridHashMax); an Ethereum block of 275 accounts (19K keys), with a
// grid barrier per depth instead, took 626 us, 429 so.
#pragma once
#include "trie_kernels.cuh"

namespace gmpt {

constexpr int kGridThreads = 512;  // one CTA per SM at 128 registers
constexpr int kGridMaxTs = 64;

// Control block of one cooperative launch.  Zeroed before its first use; a
// completed launch leaves the counters as the next one needs them.
struct GridCtl {
  uint64_t barrier_ns;           // longest grid-barrier wait before giving up
  uint32_t bar_count, bar_gen;   // grid barrier
  uint32_t status;               // 1: a barrier gave up; 2: stopped on bad input
  uint32_t ready[3];             // ready branches per wave, rotating
  uint32_t n_ts, pad;            // phase timeline of CTA 0 (globaltimer, ns)
  uint64_t ts[kGridMaxTs];
};

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// A barrier wait longer than GridCtl::barrier_ns (2 s unless the trie's
// "block_barrier_ns" option says otherwise) gives up: the CTA raises
// ERR_BARRIER and leaves the kernel, and so does every CTA at its next
// barrier.  A hash call then hashes its list again level by level, a block
// update ends with an error.

// Grid-wide barrier of a cooperative launch (all CTAs co-resident).
// Returns false when this CTA must stop.
__device__ inline bool grid_barrier(GridCtl *D, Counters *ctr) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    volatile uint32_t *vgen = &D->bar_gen;
    const uint32_t g = *vgen;
    __threadfence();
    const uint32_t arrived = atomicAdd(&D->bar_count, 1u);
    if (arrived == gridDim.x - 1) {
      atomicExch(&D->bar_count, 0u);
      __threadfence();
      atomicAdd(&D->bar_gen, 1u);
    } else {
      const uint64_t t0 = global_ns();
      const uint64_t limit = D->barrier_ns;
      uint32_t spins = 0;
      while (*vgen == g) {
        __nanosleep(32);
        if ((++spins & 63) == 0 && global_ns() - t0 > limit) {
          ok = 0;
          break;
        }
      }
    }
    if (!ok) {
      set_error(ctr, ERR_BARRIER);
      atomicOr(&D->status, 1u);
    } else if (*reinterpret_cast<volatile uint32_t *>(&D->status) & 1u) {
      ok = 0;  // another CTA gave up earlier
    }
    __threadfence();
    s_ok = ok;
    if (blockIdx.x == 0 && D->n_ts < kGridMaxTs) D->ts[D->n_ts++] = global_ns();
  }
  __syncthreads();
  return s_ok != 0;
}

// How a grid's threads see the work.  Warps are numbered CTA-fastest
// (consecutive warp ids sit on different SMs, the first 4 x SMs on different
// schedulers).  Latency-bound items (a key's descent) go to warp j % W, lane
// j / W: a few hundred use one lane in each of many warps.  A thread per
// node's permutation costs its scheduler the same whether one lane or all
// work, so those use one warp per scheduler until its lanes are full.
struct GridPlace {
  int lane, W, gw, t_spread, T;
  __device__ __forceinline__ GridPlace() {
    T = gridDim.x * blockDim.x;
    lane = threadIdx.x & 31;
    W = T >> 5;
    gw = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
    t_spread = lane * W + gw;
  }
  // warps that hash n nodes a thread each
  __device__ __forceinline__ uint32_t dense(uint32_t n) const {
    return min((uint32_t)W, max(4u * gridDim.x, (n + 31u) / 32u));
  }
};

// Branch f has `kids` dirty branches below it: note it, or list it as ready.
__device__ __forceinline__ void list_ready(const TrieView &tv, uint32_t f, uint32_t at, uint32_t *ready, uint32_t cap) {
  if (at < cap)
    ready[at] = f;
  else
    set_error(tv.ctr, ERR_INTERNAL);
}
__device__ __forceinline__ void branch_pending(const TrieView &tv, uint32_t f, uint32_t kids, uint32_t *ready,
                                               uint32_t cap, uint32_t *n_ready) {
  tv.full_pend[f] = kids;
  if (kids == 0) list_ready(tv, f, atomicAdd(n_ready, 1u), ready, cap);
}

// The dirty branch below child slot word r (straight, or under its
// extension), or kNoNode.
__device__ __forceinline__ uint32_t dirty_branch_below(const TrieView &tv, uint32_t r) {
  if (ref_kind(r) == KIND_SHORT) r = __ldcg(tv.short_child + ref_idx(r));
  if (ref_kind(r) != KIND_FULL) return kNoNode;
  return __ldcg(tv.full_epoch + ref_idx(r)) == tv.gen ? ref_idx(r) : kNoNode;
}

// Whether a dirty short node is hashed in step 1; an extension over a dirty
// branch is left to that branch (recorded in full_ext).
__device__ __forceinline__ bool short_first(const TrieView &tv, uint32_t s) {
  if (__ldcg(tv.short_dead + s)) return false;
  const uint32_t c = __ldcg(tv.short_child + s);
  if (ref_kind(c) == KIND_FULL && __ldcg(tv.full_epoch + ref_idx(c)) == tv.gen) {
    tv.full_ext[ref_idx(c)] = s;
    return false;
  }
  return true;
}

// The branch above one whose task (with its extension) starts at nibble depth
// `top`, or kNoNode at a root.  full_par is written in step 1 for every dirty
// branch that is not a root's: whatever is dirty has a dirty parent.
__device__ __forceinline__ uint32_t parent_branch(const TrieView &tv, uint32_t par, uint32_t top) {
  return top != 0 && par < tv.cap_full ? par : kNoNode;
}

// A ready branch is hashed: one child less for the branch above it (par, when
// the hashed nodes start at depth top > 0), which is listed when that was the
// last.  The caller has fenced the hash.
__device__ __forceinline__ void child_done(const TrieView &tv, uint32_t par, uint32_t top, uint32_t at0, uint32_t *next,
                                           uint32_t *ready, uint32_t cap) {
  const uint32_t p = parent_branch(tv, par, top);
  if (p != kNoNode && atomicSub(&tv.full_pend[p], 1u) == 1u) list_ready(tv, p, at0 + atomicAdd(next, 1u), ready, cap);
}

// A wave of n ready branches, a pair of lanes each: the even lane writes the
// message into its column, both permute (keccak_f1600_pair), then the same for
// the extension above.  Branches of more than kPairBlocks blocks (a long value:
// its serial blocks are shorter a warp each) or below 32 bytes are left to the
// whole warp, an extension of more than one block to the even lane.
// A thread each, a wave of 2^13 branches of 10 children with their extensions
// took 38 us; a pair each, 31 (2.9 us a permutation against 4.9).
constexpr uint32_t kPairBlocks = 12;

__device__ inline void wave_by_pairs(const TrieView &tv, const GridPlace &g, const uint32_t *list, uint32_t n,
                                     uint32_t at0, uint32_t *next, uint32_t *ready, uint32_t cap, uint32_t *stage,
                                     uint8_t *wmsg, const CoopLanes &cl) {
  constexpr unsigned kAll = 0xffffffffu;
  const bool odd = g.lane & 1;
  const int even = g.lane & ~1;
  const uint32_t S = blockDim.x;
  uint32_t *st = stage - (odd ? 1 : 0);  // the pair's column
  const uint32_t wd = g.dense(2 * n);
  if ((uint32_t)g.gw >= wd) return;
  for (uint32_t j0 = (uint32_t)g.gw; j0 < n; j0 += 16 * wd) {  // items j0 + pair * wd
    const uint32_t j = j0 + (uint32_t)(g.lane >> 1) * wd;
    const uint32_t f = j < n ? __ldcg(list + j) : kNoNode;
    const bool on = f != kNoNode;
    const uint32_t *chp = tv.full_child + (size_t)(on ? f : 0) * 17;
    uint32_t present = 0;
    bool regular = on;
    if (on && !odd) {
      uint32_t ch[17];
#pragma unroll
      for (int k = 0; k < 17; ++k) ch[k] = __ldcg(chp + k);
      const bool any_raw = __ldcg(&tv.ctr->raw_nodes) != 0;
#pragma unroll
      for (int k = 0; k < 17; ++k) {
        const uint32_t kd = ref_kind(ch[k]);
        present |= (kd != KIND_NULL ? 1u : 0u) << k;
        regular = regular && kd != KIND_VALUE;
        if (any_raw && kd != KIND_NULL && kd != KIND_VALUE)
          regular = regular && __ldcg((kd == KIND_FULL ? tv.full_hlen : tv.short_hlen) + ref_idx(ch[k])) == 32;
      }
      regular = regular && present < (1u << 16) && present != 0;
    }
    uint32_t body = 17u + 32u * __popc(present);
    if (on && !odd && !regular) {
      body = 0;
#pragma unroll 1
      for (int k = 0; k < 17; ++k) {
        const EncItem it = child_item<true>(tv, __ldcg(chp + k));
        body += it.pren + it.blen;
      }
    }
    uint64_t hdr;
    uint32_t hn;
    rlp_head(body, 0xc0, 0xf7, hdr, hn);
    const uint32_t total = body + hn;
    const bool pair = __shfl_sync(kAll, on && total >= 32 && total < kPairBlocks * 136, even);
    const unsigned other = __ballot_sync(kAll, on && !pair && !odd);
    // the branch
    BranchWriter<true> bw(st, S, hdr, hn, present);
    ItemWriter<true> iw(st, S, hdr, hn);
    uint32_t a[25], h[4] = {0, 0, 0, 0};
#pragma unroll
    for (int i = 0; i < 25; ++i) a[i] = 0;
    bool going = pair;
    uint32_t blocks = 0;
    while (__any_sync(kAll, going)) {
      bool last = false;
      if (going && !odd) last = regular ? bw.fill(tv, chp) : iw.fill(tv, chp);
      __syncwarp();
      last = __shfl_sync(kAll, last, even);
      if (going) {
        ++blocks;
#pragma unroll
        for (int i = 0; i < 17; ++i) a[i] ^= st[(2 * i + (odd ? 1 : 0)) * S];
      }
      keccak_f1600_pair(a, odd);
      __syncwarp();  // the column is read before it is written again
      if (going && last) {
#pragma unroll
        for (int i = 0; i < 4; ++i) h[i] = a[i];
      }
      if (going && !last && !odd) regular ? bw.next() : iw.next();
      going = going && !last;
    }
    uint32_t e = kNoNode, top = 0;
    if (pair) {
      uint32_t *o = reinterpret_cast<uint32_t *>(tv.full_hash + (size_t)f * 32);
#pragma unroll
      for (int i = 0; i < 4; ++i) o[2 * i + (odd ? 1 : 0)] = h[i];
      if (!odd) {
        tv.full_hlen[f] = 32;
        e = ext_above(tv, f);
        top = e != kNoNode ? __ldcg(tv.short_depth + e) : __ldcg(tv.full_depth + f);
      }
    }
    __syncwarp();  // an extension of more blocks than one reads both lanes' halves back (hash_node below)
    // the extension above: [header][key][0xa0][hash], one block
    EncItem key{0, 0, 0, nullptr, 0};
    if (e != kNoNode) key = compact_item(tv, __ldcg(tv.short_key + e), __ldcg(tv.short_klen + e));
    const uint32_t payload = key.pren + key.blen + 33;
    rlp_head(payload, 0xc0, 0xf7, hdr, hn);
    const bool one = e != kNoNode && payload + hn <= 135;
    const bool one_pair = __shfl_sync(kAll, one, even);
    if (__any_sync(kAll, one)) {
      uint32_t hx[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) hx[i] = __shfl_xor_sync(kAll, h[i], 1);
      if (one) {  // even lane: h has the low halves, hx the high ones
        WordWriter o(st, S);
        o.bytes((uint32_t)hdr, hn);
        o.bytes8(key.pre, key.pren);
        write_nibbles(o, key.body, key.blen);
        o.bytes(0xa0u, 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          o.word(h[i]);
          o.word(hx[i]);
        }
        o.bytes(0x01u, 1);
        o.bytes(0u, 3);  // at least the pending bytes
        for (uint32_t w = o.w; w < 34; ++w) st[w * S] = 0;
        st[33 * S] |= 0x80000000u;
      }
      __syncwarp();
#pragma unroll
      for (int i = 0; i < 25; ++i) a[i] = i < 17 && one_pair ? st[(2 * i + (odd ? 1 : 0)) * S] : 0u;
      keccak_f1600_pair(a, odd);
      __syncwarp();
      const uint32_t ee = __shfl_sync(kAll, e, even);
      if (one_pair) {
        uint32_t *o = reinterpret_cast<uint32_t *>(tv.short_hash + (size_t)ee * 32);
#pragma unroll
        for (int i = 0; i < 4; ++i) o[2 * i + (odd ? 1 : 0)] = a[i];
        if (!odd) tv.short_hlen[ee] = 32;
      }
    }
    if (e != kNoNode && !one) hash_node<true, false>(tv, e, stage, S);
    if (tv.account && pair && !odd) {
      atomicAdd(&tv.ctr->enc_bytes, (unsigned long long)total + (one ? payload + hn : 0u));
      atomicAdd(&tv.ctr->keccak_blocks, (unsigned long long)blocks + (one ? 1u : 0u));
      atomicAdd(&tv.ctr->hashed, one ? 2u : 1u);
    }
    __threadfence();  // both lanes' halves before the parent's count
    __syncwarp();
    if (pair && !odd) child_done(tv, __ldcg(tv.full_par + f), top, at0, next, ready, cap);
    for (unsigned m = other; m; m &= m - 1) {
      const uint32_t fi = __shfl_sync(kAll, f, __ffs(m) - 1);
      const uint32_t t = hash_full_warp<true>(tv, fi, child_word(tv, fi, g.lane), wmsg, cl, kNoNode, nullptr);
      __threadfence();
      __syncwarp();
      if (g.lane == 0) child_done(tv, __ldcg(tv.full_par + fi), t, at0, next, ready, cap);
      __syncwarp();
    }
  }
}

// Hash the nd dirty nodes of dl.  ready: room for every dirty branch (`cap`
// entries; a trie left half built by a put that ran out of nodes could ask
// for more, which is an error and not a write past the end).
// warp_max: up to this many nodes or ready branches are hashed a warp each.
// Returns false when a barrier gave up.  *waves counts the waves.
__device__ inline bool hash_grid(const TrieView &tv, DirtyList dl, uint32_t nd, uint32_t *ready, uint32_t cap,
                                 GridCtl *D, uint32_t warp_max, uint32_t *stage, uint8_t *wmsg, uint32_t *waves) {
  const GridPlace g;
  const CoopLanes cl = coop_lanes(g.lane);
  if (nd <= warp_max) {
    for (uint32_t j = (uint32_t)g.gw; j < nd; j += (uint32_t)g.W) {
      const uint32_t r = __ldcg(dl.ref + j), idx = ref_idx(r);
      if (ref_kind(r) == KIND_FULL) {
        if (__ldcg(tv.full_dead + idx)) continue;
        const uint32_t c =
            g.lane < 16 ? dirty_branch_below(tv, __ldcg(tv.full_child + (size_t)idx * 17 + g.lane)) : kNoNode;
        if (c != kNoNode) tv.full_par[c] = idx;
        const unsigned kids = __ballot_sync(0xffffffffu, c != kNoNode);
        if (g.lane == 0) branch_pending(tv, idx, __popc(kids), ready, cap, &D->ready[0]);
      } else {
        // every lane asks (same words), lane 0's note of an extension stands
        if (short_first(tv, idx)) hash_short_warp<true>(tv, idx, wmsg, cl, false, 0, 0);
      }
      __syncwarp();
    }
  } else {
    const uint32_t wd = g.dense(nd);
    for (uint32_t j = (uint32_t)g.gw < wd ? g.lane * wd + g.gw : nd; j < nd; j += 32 * wd) {
      const uint32_t r = __ldcg(dl.ref + j), idx = ref_idx(r);
      if (ref_kind(r) == KIND_FULL) {
        if (__ldcg(tv.full_dead + idx)) continue;
        const uint32_t *ch = tv.full_child + (size_t)idx * 17;
        uint32_t kids = 0;
#pragma unroll 4
        for (int k = 0; k < 16; ++k) {
          const uint32_t c = dirty_branch_below(tv, __ldcg(ch + k));
          if (c != kNoNode) {
            tv.full_par[c] = idx;
            ++kids;
          }
        }
        branch_pending(tv, idx, kids, ready, cap, &D->ready[0]);
      } else if (short_first(tv, idx)) {
        hash_node<true, false>(tv, idx, stage, blockDim.x);
      }
    }
  }
  if (!grid_barrier(D, tv.ctr)) return false;
  if (g.t_spread == 0) atomicExch(&tv.ctr->n_dirty, 0u);  // every CTA has read it
  uint32_t base = 0, k = 0;
  while (true) {
    // ready[k % 3] is this wave's count, [(k + 1) % 3] collects the next
    // one's, and [(k + 2) % 3], last read a barrier ago, is cleared for the
    // one after
    const uint32_t n = min(__ldcg(&D->ready[k % 3]), cap - base);
    if (n == 0) break;
    uint32_t *next = &D->ready[(k + 1) % 3];
    if (g.t_spread == 0) D->ready[(k + 2) % 3] = 0;
    ++*waves;
    const bool climb = n <= warp_max;
    if (climb) {
      for (uint32_t j = (uint32_t)g.gw; j < n; j += (uint32_t)g.W) {
        uint32_t f = __ldcg(ready + base + j);
        uint32_t r = child_word(tv, f, g.lane);
        while (true) {
          // the parent's slots are loaded while this branch is hashed
          const uint32_t par = __ldcg(tv.full_par + f);
          uint32_t r_par = 0;
          const uint32_t top = hash_full_warp<true>(tv, f, r, wmsg, cl, par < tv.cap_full ? par : kNoNode, &r_par);
          const uint32_t p = parent_branch(tv, par, top);
          if (p == kNoNode) break;
          __threadfence();  // this child's hash before its parent's count
          __syncwarp();
          uint32_t left = 0;
          if (g.lane == 0) left = atomicSub(&tv.full_pend[p], 1u);
          left = __shfl_sync(0xffffffffu, left, 0);
          if (left != 1) break;  // another child is still to come
          __threadfence();       // the other children's hashes, before reading them
          f = p;
          r = r_par;
        }
        __syncwarp();
      }
    } else {
      wave_by_pairs(tv, g, ready + base, n, base + n, next, ready, cap, stage, wmsg, cl);
    }
    if (!grid_barrier(D, tv.ctr)) return false;
    if (climb) break;
    base += n;
    ++k;
  }
  // counters as the next pass finds them: nothing reads them after the last
  // barrier (a climb leaves its own wave's count, a finished chain of waves zeros)
  if (g.t_spread == 0) D->ready[0] = D->ready[1] = D->ready[2] = 0;
  return true;
}

// One hash call's whole pass over the nd nodes of the dirty list.
__global__ void __launch_bounds__(kGridThreads, 1) k_hash_grid(TrieView tv, DirtyList dl, uint32_t nd, uint32_t *ready,
                                                              uint32_t cap, GridCtl *D, uint32_t warp_max) {
  extern __shared__ __align__(16) uint32_t smem[];  // kStageWords message words per thread, a window per warp
  uint8_t *wmsg = reinterpret_cast<uint8_t *>(smem + kStageWords * blockDim.x) + (threadIdx.x >> 5) * kWarpMsgBytes;
  uint32_t waves = 0;
  hash_grid(tv, dl, nd, ready, cap, D, warp_max, smem + threadIdx.x, wmsg, &waves);
}

}  // namespace gmpt
