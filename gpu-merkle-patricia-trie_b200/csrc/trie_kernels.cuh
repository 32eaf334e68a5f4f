// trie_kernels.cuh -- sm_100a kernels of the batched MPT update path.
//
// Pipeline of one PhaseNU batch (puts_2phase_with_valuehp,
// mpt-with-compress/include/mpt/gpu_mpt.cuh:1262-1399):
//   k_stage        key/value records into trie-owned arenas, key validation
//   k_sort_*       lexicographic sort of the batch by 8-nibble chunks with
//                  segment refinement; last occurrence of a key wins
//   k_walk         per unique key: read-only descent from the root, marks
//                  the path dirty, overwrites values of keys that exist,
//                  and finds where new keys attach (anchor)
//   k_items_*      new keys + one "pseudo" item per short node that must be
//                  split, in key order, which groups them by anchor (or
//                  nearly: k_item_runs)
//   k_level_*      level-synchronous construction of the compressed
//                  subtries of every group (branch / extension / leaf)
//   k_hash_level   fused RLP encode + Keccak-256 of every dirty node of one
//                  nibble depth, deepest first (PhaseHC)
// The reference instead expands every key into one 240-byte FullNode per
// nibble and recompresses (K:3655, K:4025, K:4643); building the compressed
// form directly from the sorted batch writes each node once.
#pragma once
#include "common.cuh"
#include "keccak.cuh"

namespace gmpt {

// ---------------------------------------------------------------------------
// dirty list

struct DirtyList {
  uint32_t *ref;
  uint16_t *depth;
};

__device__ __forceinline__ void dirty_push(Counters *c, DirtyList d, uint32_t ref, uint32_t depth) {
  uint32_t i = warp_alloc(&c->n_dirty, 1);
  d.ref[i] = ref;
  d.depth[i] = (uint16_t)depth;
}

// First visitor of a node in this hash generation appends it to the dirty
// list.  Reads go through L2 (ld.cg): under LockNU the node may have been
// created by another SM during this launch.
__device__ __forceinline__ void mark_full(const TrieView &tv, DirtyList d, uint32_t f, uint32_t gen) {
  if (__ldcg(tv.full_epoch + f) != gen) {
    if (atomicExch(&tv.full_epoch[f], gen) != gen)
      dirty_push(tv.ctr, d, make_ref(KIND_FULL, f), __ldcg(tv.full_depth + f));
  }
}

__device__ __forceinline__ void mark_short(const TrieView &tv, DirtyList d, uint32_t s, uint32_t gen) {
  if (__ldcg(tv.short_epoch + s) != gen) {
    if (atomicExch(&tv.short_epoch[s], gen) != gen)
      dirty_push(tv.ctr, d, make_ref(KIND_SHORT, s), __ldcg(tv.short_depth + s));
  }
}

__device__ __forceinline__ void write_slot(const TrieView &tv, uint64_t slot, uint32_t ref) {
  if (is_root_slot(slot))
    tv.roots[slot_trie(slot)] = ref;
  else
    tv.full_child[(slot >> 5) * 17 + (slot & 31)] = ref;
}

__device__ __forceinline__ uint32_t new_full(const TrieView &tv, DirtyList d, uint32_t depth, uint32_t gen) {
  uint32_t f = warp_alloc(&tv.ctr->n_full, 1);
  if (f >= tv.cap_full) {
    set_error(tv.ctr, ERR_CAPACITY);
    return 0xFFFFFFFFu;
  }
  uint32_t *ch = tv.full_child + (size_t)f * 17;
#pragma unroll
  for (int i = 0; i < 17; ++i) ch[i] = 0;
  tv.full_depth[f] = (uint16_t)depth;
  tv.full_epoch[f] = gen;
  tv.full_hlen[f] = 0;
  tv.full_dead[f] = 0;
  tv.full_ext[f] = kNoNode;
  dirty_push(tv.ctr, d, make_ref(KIND_FULL, f), depth);
  return f;
}

__device__ __forceinline__ uint32_t new_short(const TrieView &tv, DirtyList d, uint64_t key_off, uint32_t klen,
                                              uint32_t child, uint32_t depth, uint32_t gen) {
  uint32_t s = warp_alloc(&tv.ctr->n_short, 1);
  if (s >= tv.cap_short) {
    set_error(tv.ctr, ERR_CAPACITY);
    return 0xFFFFFFFFu;
  }
  tv.short_key[s] = key_off;
  tv.short_klen[s] = klen;
  tv.short_child[s] = child;
  tv.short_depth[s] = (uint16_t)depth;
  tv.short_epoch[s] = gen;
  tv.short_dead[s] = 0;
  tv.short_claim[s] = 0;
  tv.short_hlen[s] = 0;
  dirty_push(tv.ctr, d, make_ref(KIND_SHORT, s), depth);
  return s;
}

// ---------------------------------------------------------------------------
// staging

// A batch where it lies (caller's device arrays, or copies made for a host
// batch), and where its bytes go.
struct StageIn {
  const uint8_t *keys;   // key stream; the arena's own copy when copy_keys is off
  const uint8_t *vals;
  const int *ki;
  const int64_t *vi;
  const uint64_t *hp;    // or null
  const int *tid;        // or null
  int64_t kbytes, vbytes;
  uint64_t key_base, val_base, vid_base;  // key_base is 8-byte aligned, val_base 16
  int copy_keys, copy_vals;  // copy the stream into the arena (its source is aligned alike)
  int check_stream;          // the key stream is checked whole (hex keys)
};

__device__ __forceinline__ void stage_error(Counters *c, uint32_t bits) {
  set_error(c, bits);
  c->stage_bad = 1;
}

// Eight nibble bytes: any of 17 or more, and how many 16s.
__device__ __forceinline__ void check_nibbles8(uint64_t x, uint32_t &bad, uint32_t &terms) {
  const uint64_t hi = x & 0x1010101010101010ull;  // bit 4 set: 16..31
  bad |= (x & 0xE0E0E0E0E0E0E0E0ull) != 0 || (x & ((hi >> 4) * 0x0Full)) != 0;
  terms += __popcll(hi);
}

// Stage a batch in one pass: copy the key and value streams into the arenas
// (64 bytes in flight per thread), check the key stream as it
// goes by -- no byte > 16, and exactly as many 16s as keys that end in one (so
// none is interior, given that the index pairs tile the stream; k_stage_keys
// looks at batches that do not) -- and build the per-key and value records.
// Grid-stride, counters reduced per CTA.
// Bound by HBM.  Separate copies, record and check launches read the key
// stream twice and cost a 16K-key put eight operations before its insert;
// 16M YCSB keys: 1.36 ms, now 1.11 (5.9 GB: 5.3 TB/s).
__global__ void __launch_bounds__(256) k_stage(TrieView tv, StageIn in, int n, uint64_t *koff, uint32_t *klen) {
  uint32_t terms = 0, gaps = 0, lmax = 0, vmax = 0, sterms = 0, sbad = 0;
  const int64_t T = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  // streams: whole words, then the tail bytes and 64 zero bytes
  // behind them (8-byte loads may read past a key's or a value's last byte)
  if (in.copy_keys || in.check_stream) {
    const int64_t nv = in.kbytes / 8;
    const uint64_t *src = reinterpret_cast<const uint64_t *>(in.keys);
    uint64_t *dst = reinterpret_cast<uint64_t *>(const_cast<uint8_t *>(tv.keys) + in.key_base);
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {  // the usual source: 16 bytes a load
      const int64_t np = nv / 2;
      const ulonglong2 *s2 = reinterpret_cast<const ulonglong2 *>(src);
      const bool even = (in.key_base & 15) == 0;
      for (int64_t w = t0; w < np; w += 4 * T) {
        ulonglong2 x[4];
#pragma unroll
        for (int k = 0; k < 4; ++k)
          if (w + k * T < np) x[k] = s2[w + k * T];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          if (w + k * T >= np) continue;
          uint64_t *d = dst + 2 * (w + k * T);
          if (in.copy_keys && even) {
            *reinterpret_cast<ulonglong2 *>(d) = x[k];
          } else if (in.copy_keys) {
            d[0] = x[k].x;
            d[1] = x[k].y;
          }
          check_nibbles8(x[k].x, sbad, sterms);
          check_nibbles8(x[k].y, sbad, sterms);
        }
      }
      if (t0 == 0 && (nv & 1)) {
        const uint64_t x = src[nv - 1];
        if (in.copy_keys) dst[nv - 1] = x;
        check_nibbles8(x, sbad, sterms);
      }
    } else {
      for (int64_t w = t0; w < nv; w += T) {
        const uint64_t x = src[w];
        if (in.copy_keys) dst[w] = x;
        check_nibbles8(x, sbad, sterms);
      }
    }
    if (t0 < (in.kbytes & 7)) {
      const uint8_t b = in.keys[8 * nv + t0];
      if (in.copy_keys) reinterpret_cast<uint8_t *>(dst)[8 * nv + t0] = b;
      sbad |= b > 16;
      sterms += b == 16;
    }
  }
  if (in.copy_vals) {
    const int64_t nv = in.vbytes / 16;
    const uint4 *src = reinterpret_cast<const uint4 *>(in.vals);
    uint4 *dst = reinterpret_cast<uint4 *>(const_cast<uint8_t *>(tv.vals) + in.val_base);
    for (int64_t w = t0; w < nv; w += 4 * T) {
      uint4 x[4];
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (w + k * T < nv) x[k] = __ldcs(src + w + k * T);
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (w + k * T < nv) dst[w + k * T] = x[k];
    }
    if (t0 < (in.vbytes & 15)) reinterpret_cast<uint8_t *>(dst)[16 * nv + t0] = in.vals[16 * nv + t0];
  }
  if (t0 < 64) const_cast<uint8_t *>(tv.keys)[in.key_base + in.kbytes + t0] = 0;
  // records
  for (int64_t i = t0; i < n; i += T) {
    if (in.tid && (uint32_t)in.tid[i] >= tv.n_tries) stage_error(tv.ctr, ERR_BAD_TRIE);
    int ks = in.ki[2 * i], ke = in.ki[2 * i + 1];
    bool bad = ks < 0 || ke < ks || (int64_t)ke >= in.kbytes;  // index pair outside the key stream
    if (bad) ks = ke = 0;
    int len = ke - ks + 1;
    if (len > kMaxKeyNibbles) {
      stage_error(tv.ctr, ERR_KEY_TOO_LONG);
      bad = true;
    }
    bool term = false;
    if (!bad) {
      const uint8_t last = in.keys[ke];
      if (last > 16) bad = true;
      term = last == 16;
    }
    const bool gap = (i == 0) ? (ks != 0) : (ks != in.ki[2 * i - 1] + 1);
    terms += (term && !bad) ? 1u : 0u;
    gaps |= gap ? 1u : 0u;
    if (bad) {
      stage_error(tv.ctr, ERR_BAD_KEY);
      len = 1;  // keep later stages in bounds
    }
    koff[i] = in.key_base + (uint64_t)ks;
    klen[i] = (uint32_t)len;
    lmax = max(lmax, (uint32_t)len);
    int64_t vs = in.vi[2 * i], ve = in.vi[2 * i + 1];
    if (vs < 0 || ve < vs - 1 || ve >= in.vbytes || ve - vs + 1 > 0x7FFFFFFF) {  // empty values allowed
      stage_error(tv.ctr, ERR_BAD_KEY);
      vs = 0;
      ve = -1;
    }
    const uint64_t vid = in.vid_base + (uint64_t)i;
    vmax = max(vmax, (uint32_t)(ve - vs + 1));
    tv.rec[vid] = ValueRec{in.val_base + (uint64_t)vs, (uint32_t)(ve - vs + 1), 0u};
    tv.rec_hp[vid] = in.hp ? in.hp[i] : 0ull;
  }
  __shared__ uint32_t red[6][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  terms = __reduce_add_sync(0xffffffffu, terms);
  gaps = __reduce_or_sync(0xffffffffu, gaps);
  lmax = __reduce_max_sync(0xffffffffu, lmax);
  vmax = __reduce_max_sync(0xffffffffu, vmax);
  sterms = __reduce_add_sync(0xffffffffu, sterms);
  sbad = __reduce_or_sync(0xffffffffu, sbad);
  if (lane == 0) {
    red[0][warp] = terms;
    red[1][warp] = gaps;
    red[2][warp] = lmax;
    red[3][warp] = vmax;
    red[4][warp] = sterms;
    red[5][warp] = sbad;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t t = 0, g = 0, m = 0, v = 0, st = 0, sb = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      t += red[0][w];
      g |= red[1][w];
      m = max(m, red[2][w]);
      v = max(v, red[3][w]);
      st += red[4][w];
      sb |= red[5][w];
    }
    if (t) atomicAdd(&tv.ctr->key_terms, t);
    if (g) atomicOr(&tv.ctr->noncontig, 1u);
    if (m) atomicMax(&tv.ctr->max_klen, m);
    if (v) atomicMax(&tv.ctr->max_vlen, v);
    if (st) atomicAdd(&tv.ctr->stream_terms, (unsigned long long)st);
    if (sb) atomicOr(&tv.ctr->bad_byte, 1u);
  }
}

// Raw key bytes (the caller skips the hex conversion, util/utils.cuh:340-349
// key_bytes_to_hex).  A pair (s, e) is a key of e - s + 1 bytes, e = s - 1
// the empty key; its hex form is 2 * bytes + 1 nibbles.
__device__ __forceinline__ int raw_key_len(const int *ki, int i, int64_t raw_bytes) {
  const int s = ki[2 * i], e = ki[2 * i + 1];
  const bool bad = s < 0 || e < s - 1 || (int64_t)e >= raw_bytes || 2ll * (e - s + 1) + 1 > kMaxKeyNibbles;
  return bad ? -1 : e - s + 1;
}

// Hex length of every key into flags (for the offset scan); a malformed pair
// sets ERR_BAD_KEY and counts as the empty key so later stages stay in bounds.
__global__ void k_raw_lens(TrieView tv, const int *ki, int n, int64_t raw_bytes, unsigned long long *flags) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int len = raw_key_len(ki, i, raw_bytes);
  if (len < 0) set_error(tv.ctr, ERR_BAD_KEY);
  flags[i] = 2ull * (uint64_t)max(len, 0) + 1ull;
}

// Expand every key to nibbles (high, low per byte) + terminator 16 at hex
// offset pos[i] of `out`, and rewrite its index pair (in place) to the hex
// range.  A warp takes 32 keys and walks them with a byte per lane, so loads
// and stores are coalesced (a key per thread, byte after byte, took 76 us for
// 300K 20-byte keys; this takes 23).
__global__ void __launch_bounds__(256) k_raw_expand(const uint8_t *raw, int *ki, const unsigned long long *pos, int n,
                                                    int64_t raw_bytes, uint8_t *out) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int i0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31, i = i0 + lane;
  const int len = i < n ? max(raw_key_len(ki, i, raw_bytes), 0) : 0;
  const int s = i < n ? ki[2 * i] : 0;
  const unsigned long long p = i < n ? pos[i] : 0ull;
  for (int k = 0; k < 32 && i0 + k < n; ++k) {
    const int kl = __shfl_sync(kAll, len, k), ks = __shfl_sync(kAll, s, k);
    uint8_t *o = out + __shfl_sync(kAll, p, k);
    for (int b = lane; b < kl; b += 32) {
      const uint8_t x = raw[ks + b];
      o[2 * b] = x >> 4;
      o[2 * b + 1] = x & 15;
    }
    if (lane == 0) o[2 * kl] = 16;
  }
  if (i < n) {
    ki[2 * i] = (int)p;
    ki[2 * i + 1] = (int)(p + 2 * (uint64_t)len);
  }
}

// Verdict on a staged hex-key batch: one whose index pairs tile the stream is
// checked whole (k_stage), the others key by key here.  (The host reports
// the reason when it reads the counters.)
__global__ void k_stage_keys(TrieView tv, const uint64_t *koff, const uint32_t *klen, int n) {
  if (!__ldcg(&tv.ctr->noncontig)) {
    if (blockIdx.x == 0 && threadIdx.x == 0 &&
        (__ldcg(&tv.ctr->bad_byte) || __ldcg(&tv.ctr->stream_terms) != __ldcg(&tv.ctr->key_terms)))
      tv.ctr->stage_bad = 1;
    return;
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint8_t *k = tv.keys + koff[i];
    int len = (int)klen[i];
    uint64_t acc = 0;
    for (int j = 0; j < len - 1; j += 8) acc |= load_u64_unaligned(k + j) & low_mask64(min(8, len - 1 - j));
    if (acc & 0xF0F0F0F0F0F0F0F0ull) stage_error(tv.ctr, ERR_BAD_KEY);
  }
}

// ---------------------------------------------------------------------------
// sort + dedup (chunked MSD refinement over LSD radix passes)

__device__ __forceinline__ uint32_t key_chunk(const uint8_t *keys, uint64_t off, uint32_t len, int c) {
  uint32_t start = (uint32_t)c * 8;
  if (start >= len) return 0;
  uint64_t x = load_u64_unaligned(keys + off + start);
  uint32_t rem = len - start;
  if (rem < 8) x &= (1ull << (8 * rem)) - 1;  // zero bytes beyond the key
  return pack_nibbles8(x);
}

// *differs = 1 when some key's chunk c is not key 0's (a chunk every key of
// the batch shares needs no sort pass: YCSB keys all begin with "user")
__global__ void k_chunk_shared(const uint8_t *keys, const uint64_t *koff, const uint32_t *klen, int n, int c,
                               uint32_t *differs) {
  // once one warp has found a difference the rest have nothing to add: they
  // read the flag and leave instead of queueing atomics on one address
  if (__any_sync(0xffffffffu, __ldcg(differs) != 0u)) return;  // the whole warp leaves
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool d = i < n && key_chunk(keys, koff[i], klen[i], c) != key_chunk(keys, koff[0], klen[0], c);
  if (__any_sync(0xffffffffu, d) && (threadIdx.x & 31) == 0 && !__ldcg(differs)) atomicOr(differs, 1u);
}

// active = tied with a neighbour; packed: low = active, high = segment start
__global__ void k_sort_flags(const uint8_t *eqprev, int n, unsigned long long *flags) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  uint32_t tl = eqprev[p], tr = eqprev[p + 1];
  uint32_t active = (tl | tr) ? 1u : 0u;
  uint32_t start = (active && !tl) ? 1u : 0u;
  flags[p] = (unsigned long long)active | ((unsigned long long)start << 32);
}

// c >= 0: key chunk c; c == -1: key length; c == -2: trie id (forest batches)
__global__ void k_sort_build(TrieView tv, const unsigned long long *flags, const unsigned long long *pos,
                             const uint32_t *order, const uint64_t *koff, const uint32_t *klen, int n, int c,
                             uint32_t *act, uint64_t *skey, uint32_t *sval, const int *tid) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  unsigned long long f = flags[p];
  if (!(f & 1ull)) return;
  unsigned long long q = pos[p];
  uint32_t k = (uint32_t)q;
  uint32_t seg = (uint32_t)(q >> 32) + (uint32_t)(f >> 32) - 1u;
  uint32_t it = order[p];
  uint32_t ch = c >= 0 ? key_chunk(tv.keys, koff[it], klen[it], c) : (c == -1 ? klen[it] : (uint32_t)tid[it]);
  act[k] = (uint32_t)p;
  skey[k] = ((uint64_t)seg << 32) | ch;
  sval[k] = it;
}

__global__ void k_sort_scatter(const uint32_t *act, const uint64_t *skey, const uint32_t *sval, int K,
                               uint32_t *order, uint8_t *eqprev) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  uint32_t p = act[k];
  order[p] = sval[k];
  eqprev[p] = (k > 0 && skey[k] == skey[k - 1]) ? 1 : 0;
}

__global__ void k_init_order(uint32_t *order, uint8_t *eqprev, int n) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > n) return;
  if (p < n) order[p] = (uint32_t)p;
  eqprev[p] = (p > 0 && p < n) ? 1 : 0;
}

// keep the last of every run of equal keys
__global__ void k_keep_flags(const uint8_t *eqprev, int n, unsigned long long *flags) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  flags[p] = eqprev[p + 1] ? 0ull : 1ull;
}

__global__ void k_keep_scatter(const unsigned long long *flags, const unsigned long long *pos,
                               const uint32_t *order, int n, uint32_t *uord) {
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  if (flags[p]) uord[(uint32_t)pos[p]] = order[p];
}

// ---------------------------------------------------------------------------
// mixed read/write batches (puts_*_with_read, gpu_mpt.cuh:684-765 and
// 1609-1713).  The sort leaves equal keys (same trie) in runs, in batch
// order; p is a sorted position, order[p] its batch index, rw[i] = 1 for a
// write.  A read takes the last write before it in its run, else the trie
// as it was before the batch; each run keeps its last write for the insert.

__global__ void k_rw_sorted_flags(const uint8_t *eqprev, const uint32_t *order, const uint8_t *rw, int n,
                                  unsigned long long *is_write, unsigned long long *is_head) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  is_write[p] = rw[order[p]] ? 1ull : 0ull;
  is_head[p] = eqprev[p] ? 0ull : 1ull;
}

// sorted slots -> order / eqprev as the full-key sort leaves them
__global__ void k_rw_groups(const uint64_t *skey, const uint32_t *sval, int n, uint32_t *order, uint8_t *eqprev) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > n) return;
  if (p < n) order[p] = sval[p];
  eqprev[p] = (p > 0 && p < n && skey[p] == skey[p - 1]) ? 1 : 0;
}

// the kept writes' key records, for a key-order sort of them alone
__global__ void k_rw_gather(const uint32_t *kept, int m, const uint64_t *koff, const uint32_t *klen, const int *tid,
                            uint64_t *koff_out, uint32_t *klen_out, int *tid_out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint32_t i = kept[j];
  koff_out[j] = koff[i];
  klen_out[j] = klen[i];
  if (tid) tid_out[j] = tid[i];
}

__global__ void k_rw_map(const uint32_t *order, const uint32_t *kept, int m, uint32_t *uord) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < m) uord[j] = kept[order[j]];
}

// Key bytes of the kept writes of a mixed batch, moved together to the start
// of the batch's region of the key arena (the reads' keys are referenced by
// nothing once the reads are answered).  sizes -> scan -> copy out -> copy
// back -> offsets.
__global__ void k_rw_kept_sizes(const uint32_t *kept, int m, const uint32_t *klen, unsigned long long *sizes) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < m) sizes[j] = klen[kept[j]];
}

__global__ void k_rw_kept_copy(const uint8_t *keys, const uint64_t *koff, const uint32_t *klen, const uint32_t *kept,
                               const unsigned long long *offs, int m, uint8_t *out) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint32_t i = kept[j];
  const uint8_t *src = keys + koff[i];
  uint8_t *dst = out + offs[j];
  for (uint32_t b = 0; b < klen[i]; ++b) dst[b] = src[b];
}

__global__ void k_rw_kept_offsets(const uint32_t *kept, const unsigned long long *offs, int m, uint64_t base,
                                  uint64_t *koff) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < m) koff[kept[j]] = base + offs[j];
}

__global__ void k_rw_read_flags(TrieView tv, const uint8_t *rw, int n, unsigned long long *is_read) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (rw[i] > 1) set_error(tv.ctr, ERR_BAD_FLAG);
  is_read[i] = rw[i] ? 0ull : 1ull;
}

// wpos[k] = sorted position of the k-th write in sorted order
__global__ void k_rw_wpos(const unsigned long long *is_write, const unsigned long long *wrank, int n, uint32_t *wpos) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  if (is_write[p]) wpos[wrank[p]] = (uint32_t)p;
}

__device__ __forceinline__ int64_t lookup(const TrieView &tv, uint32_t root, const uint8_t *kb, uint32_t len);

__global__ void k_rw_resolve(TrieView tv, const uint32_t *order, const uint8_t *rw, const unsigned long long *is_head,
                             const unsigned long long *heads_before, const unsigned long long *wrank,
                             const uint32_t *wpos, const unsigned long long *n_writes, const unsigned long long *rrank,
                             const uint64_t *koff, const uint32_t *klen, const int *tid, uint64_t vid_base, int n,
                             uint64_t *out_hp, int *out_len, unsigned long long *keep) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const uint32_t i = order[p];
  // run id of a sorted position: heads up to and including it, minus one
  auto run = [&](uint32_t q) { return heads_before[q] + is_head[q]; };
  const unsigned long long k = wrank[p];  // writes before p in sorted order
  const unsigned long long nw = *n_writes;
  if (rw[i]) {
    keep[p] = (k + 1 >= nw || run(wpos[k + 1]) != run(p)) ? 1ull : 0ull;
    return;
  }
  keep[p] = 0ull;
  int64_t vid = -1;
  if (k > 0) {
    const uint32_t q = wpos[k - 1];
    if (run(q) == run(p)) vid = (int64_t)(vid_base + order[q]);
  }
  if (vid < 0) {
    const uint32_t tr = tid ? (uint32_t)tid[i] : 0u;
    vid = tr < tv.n_tries ? lookup(tv, tv.roots[tr], tv.keys + koff[i], klen[i]) : -1;
  }
  const unsigned long long r = rrank[i];
  out_hp[r] = vid < 0 ? 0ull : tv.rec_hp[vid];
  out_len[r] = vid < 0 ? 0 : (int)tv.rec[vid].len;
}

// ---------------------------------------------------------------------------
// walk (PhaseNU against an existing trie)

enum : uint8_t { W_EXISTS = 0, W_NEW = 1, W_SPLIT = 2, W_ERROR = 3 };

// anchor code: kind(2) | index(30) | child(5)  (37 bits, shifted left 27
// in the item sort key; the low 27 bits hold the rank)
__device__ __forceinline__ uint64_t code_full(uint32_t f, uint32_t c) {
  return (1ull << 35) | ((uint64_t)f << 5) | c;
}
__device__ __forceinline__ uint64_t code_short(uint32_t s) { return (2ull << 35) | ((uint64_t)s << 5) | 31u; }
// the root word of trie t (kind 0)
__device__ __forceinline__ uint64_t code_root(uint32_t t) { return (uint64_t)t << 5; }
__device__ __forceinline__ uint64_t code_slot(uint64_t slot) {
  return is_root_slot(slot) ? code_root(slot_trie(slot)) : code_full((uint32_t)(slot >> 5), (uint32_t)(slot & 31));
}

// nibble order used by the sort: terminator (16) sorts before 0
__device__ __forceinline__ int sym_rank(uint8_t b) { return b == 16 ? -1 : (int)b; }

struct WalkOut {
  uint8_t *status;
  uint64_t *code;
  uint32_t *d0;
  uint64_t *slot;
  uint32_t *short_id;
  uint8_t *after;
  // pseudo items
  uint32_t *p_short;
  uint32_t *p_d0;
  uint64_t *p_slot;
  uint32_t *p_amin;
  uint32_t *p_max;
};

// Thread per kWalkWays unique keys advancing together, so each thread keeps
// several independent pointer chases in flight (the walk is latency bound).
constexpr int kWalkWays = 4;

__global__ void __launch_bounds__(256, 2) k_walk(TrieView tv, DirtyList dl, const uint32_t *uord, int m,
                                                 const uint64_t *koff, const uint32_t *klen, uint64_t vid_base,
                                                 WalkOut wo, const int *tid) {
  const int nthreads = gridDim.x * blockDim.x;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t gen = tv.gen;
  uint32_t ref[kWalkWays], x[kWalkWays], len[kWalkWays], item[kWalkWays];
  uint64_t slot[kWalkWays];
  bool act[kWalkWays];
#pragma unroll
  for (int w = 0; w < kWalkWays; ++w) {
    const int j = t + w * nthreads;
    act[w] = j < m;
    item[w] = act[w] ? uord[j] : 0;
    len[w] = act[w] ? klen[item[w]] : 0;
    const uint32_t tr = (act[w] && tid) ? (uint32_t)tid[item[w]] : 0u;
    ref[w] = act[w] ? tv.roots[tr] : 0u;
    x[w] = 0;
    slot[w] = root_slot(tr);
  }
  for (int round = 0; round < kMaxKeyNibbles + 2; ++round) {
    bool any = false;
#pragma unroll
    for (int w = 0; w < kWalkWays; ++w) {
      if (!act[w]) continue;
      const int j = t + w * nthreads;
      const uint8_t *kb = tv.keys + koff[item[w]];
      const uint32_t kind = ref_kind(ref[w]), idx = ref_idx(ref[w]);
      if (kind == KIND_NULL) {
        wo.status[j] = W_NEW;
        wo.code[j] = code_slot(slot[w]);
        wo.d0[j] = x[w];
        wo.slot[j] = slot[w];
        act[w] = false;
        continue;
      }
      if (kind == KIND_FULL) {
        mark_full(tv, dl, idx, gen);
        if (x[w] >= len[w]) {
          wo.status[j] = W_ERROR;
          set_error(tv.ctr, ERR_BAD_KEY);
          act[w] = false;
          continue;
        }
        const uint32_t c = kb[x[w]];
        slot[w] = ((uint64_t)idx << 5) | c;
        ref[w] = tv.full_child[(size_t)idx * 17 + c];
        ++x[w];
        any = true;
        continue;
      }
      if (kind == KIND_SHORT) {
        const uint8_t *sk = tv.keys + tv.short_key[idx];
        const uint32_t sl = tv.short_klen[idx];
        const uint32_t lim = min(sl, len[w] - x[w]);
        const uint32_t mm = (uint32_t)match_nibbles(sk, kb + x[w], (int)lim);
        if (mm == sl) {
          mark_short(tv, dl, idx, gen);
          ref[w] = tv.short_child[idx];
          x[w] += sl;
          any = true;
          continue;
        }
        act[w] = false;
        if (mm == len[w] - x[w]) {  // key ends inside a stored key: prefix
          wo.status[j] = W_ERROR;
          set_error(tv.ctr, ERR_BAD_KEY);
          continue;
        }
        wo.status[j] = W_SPLIT;
        wo.code[j] = code_short(idx);
        wo.d0[j] = x[w];
        wo.slot[j] = slot[w];
        wo.short_id[j] = idx;
        wo.after[j] = sym_rank(kb[x[w] + mm]) > sym_rank(sk[mm]) ? 1 : 0;
        // the first diverger claims the split and creates the pseudo item
        const uint32_t ep = tv.epoch;
        if (tv.short_claim[idx] != ep) {
          if (atomicExch(&tv.short_claim[idx], ep) != ep) {
            const uint32_t p = atomicAdd(&tv.ctr->n_pseudo, 1u);
            wo.p_short[p] = idx;
            wo.p_d0[p] = x[w];
            wo.p_slot[p] = slot[w];
            wo.p_amin[p] = 0xFFFFFFFFu;
            wo.p_max[p] = 0;
            tv.short_pseudo[idx] = p;
            tv.short_dead[idx] = 1;
          }
        }
        continue;
      }
      // value node
      act[w] = false;
      if (x[w] == len[w]) {
        atomicMax(&tv.value_vid[idx], (unsigned long long)(vid_base + item[w]));
        wo.status[j] = W_EXISTS;
      } else {
        wo.status[j] = W_ERROR;
        set_error(tv.ctr, ERR_BAD_KEY);
      }
    }
    if (!any) break;
  }
}

__global__ void k_pseudo_ranks(TrieView tv, const WalkOut wo, int m) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  if (wo.status[j] != W_SPLIT) return;
  uint32_t p = tv.short_pseudo[wo.short_id[j]];
  if (wo.after[j]) atomicMin(&wo.p_amin[p], (uint32_t)j);
  atomicMax(&wo.p_max[p], (uint32_t)j);
}

// Where a pseudo item (a short node re-inserted as a key ending in its old
// child) goes in key order: just before the first key that sorts after the
// short node's key, else after the last diverger.  Both are divergers of that
// short node alone, so a key has at most one pseudo item on either side.
__global__ void k_pseudo_place(TrieView tv, const WalkOut wo, int m, uint32_t *before, uint32_t *after) {
  const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= min(tv.ctr->n_pseudo, (uint32_t)m)) return;
  if (wo.p_amin[p] != 0xFFFFFFFFu)
    before[wo.p_amin[p]] = p + 1;
  else
    after[wo.p_max[p]] = p + 1;
}

// items at and around key j
__global__ void k_item_counts(const uint8_t *status, const uint32_t *before, const uint32_t *after, int m,
                              unsigned long long *flags) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint8_t st = status[j];
  flags[j] = (st == W_NEW || st == W_SPLIT ? 1ull : 0ull) + (before[j] ? 1ull : 0ull) + (after[j] ? 1ull : 0ull);
}

// the items of a build: key ending in `ref`, anchored at `code` / `slot` from nibble d0 on
struct ItemArrays {
  uint64_t *base;
  uint32_t *len, *ref, *d0;
  uint64_t *slot, *code;
};

__device__ __forceinline__ void put_pseudo(const TrieView &tv, const WalkOut &wo, const ItemArrays &it, uint64_t i,
                                           uint32_t p) {
  const uint32_t s = wo.p_short[p], d0 = wo.p_d0[p];
  it.base[i] = tv.short_key[s] - d0;
  it.len[i] = d0 + tv.short_klen[s];
  it.ref[i] = tv.short_child[s];
  it.d0[i] = d0;
  it.slot[i] = wo.p_slot[p];
  it.code[i] = code_short(s);
}

// new keys (status NEW / SPLIT) and pseudo items, in key order
__global__ void k_items_place(TrieView tv, const WalkOut wo, const uint32_t *before, const uint32_t *after,
                              const unsigned long long *pos, int m, const uint32_t *uord, const uint64_t *koff,
                              const uint32_t *klen, uint64_t vid_base, ItemArrays it) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  const uint8_t st = wo.status[j];
  uint64_t i = pos[j];
  if (before[j]) put_pseudo(tv, wo, it, i++, before[j] - 1);
  if (st == W_NEW || st == W_SPLIT) {
    const uint32_t item = uord[j];
    uint32_t v = warp_alloc(&tv.ctr->n_value, 1);
    if (v >= tv.cap_value) {
      set_error(tv.ctr, ERR_CAPACITY);
      v = 0;
    }
    tv.value_vid[v] = vid_base + item;
    it.base[i] = koff[item];
    it.len[i] = klen[item];
    it.ref[i] = make_ref(KIND_VALUE, v);
    it.d0[i] = wo.d0[j];
    it.slot[i] = wo.slot[j];
    it.code[i] = wo.code[j];
    ++i;
  }
  if (after[j]) put_pseudo(tv, wo, it, i, after[j] - 1);
}

// Runs of split groups among the *total items in key order: as many as split
// nodes when every group is in one piece.  A group comes in pieces when keys
// anchored deeper, below the split extension's branch, sort between its own;
// the groups are then sorted by anchor.
__global__ void k_item_runs(const uint64_t *code, const unsigned long long *total, unsigned long long *runs) {
  const uint64_t T = *total;
  uint32_t c = 0;
  for (uint64_t i = blockIdx.x * blockDim.x + threadIdx.x; i < T; i += (uint64_t)gridDim.x * blockDim.x)
    c += (code[i] >> 35) == 2ull && (i == 0 || code[i - 1] != code[i]) ? 1u : 0u;
  c = __reduce_add_sync(0xffffffffu, c);
  if ((threadIdx.x & 31) == 0 && c) atomicAdd(runs, (unsigned long long)c);
}

// sort keys (anchor, position) of the items
__global__ void k_item_keys(const uint64_t *code, int T, uint64_t *key, uint32_t *id) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T) return;
  key[i] = (code[i] << 27) | (uint64_t)i;
  id[i] = (uint32_t)i;
}

// Empty trie: every unique key is a new item of the single root group, already
// in sorted order (no walk, no grouping sort).  Value node j = vbase + j.
__global__ void k_items_bulk(TrieView tv, const uint32_t *uord, int m, const uint64_t *koff, const uint32_t *klen,
                             uint64_t vid_base, uint32_t vbase, uint64_t *sb_base, uint32_t *sb_len,
                             uint32_t *sb_ref, uint32_t *sb_d0, uint64_t *sb_slot, uint64_t *sb_code,
                             const int *tid) {
  int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= m) return;
  if (j == 0) atomicAdd(&tv.ctr->n_value, (uint32_t)m);
  uint32_t item = uord[j];
  uint32_t v = vbase + (uint32_t)j;
  tv.value_vid[v] = vid_base + item;
  sb_base[j] = koff[item];
  sb_len[j] = klen[item];
  sb_ref[j] = make_ref(KIND_VALUE, v);
  sb_d0[j] = 0;
  const uint32_t tr = tid ? (uint32_t)tid[item] : 0u;
  sb_slot[j] = root_slot(tr);
  sb_code[j] = code_root(tr);
}

// items in anchor order
__global__ void k_items_gather(const ItemArrays it, const uint32_t *order, int T, ItemArrays out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T) return;
  const uint32_t s = order[i];
  out.base[i] = it.base[s];
  out.len[i] = it.len[s];
  out.ref[i] = it.ref[s];
  out.d0[i] = it.d0[s];
  out.slot[i] = it.slot[s];
  out.code[i] = it.code[s];
}

// group starts and adjacent LCPs
__global__ void k_items_lcp(TrieView tv, const uint64_t *sb_base, const uint32_t *sb_len, const uint32_t *sb_d0,
                            const uint64_t *sb_code, int T, uint16_t *lcp) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T) return;
  if (i == 0 || sb_code[i] != sb_code[i - 1]) {
    lcp[i] = kLcpInf;
    return;
  }
  uint32_t d0 = sb_d0[i];
  uint32_t la = sb_len[i - 1], lb = sb_len[i];
  uint32_t lim = min(la, lb);
  uint32_t m = d0 + (uint32_t)match_nibbles(tv.keys + sb_base[i - 1] + d0, tv.keys + sb_base[i] + d0, (int)(lim - d0));
  if (m >= lim) {  // equal keys or one is a prefix of the other
    set_error(tv.ctr, ERR_BAD_KEY);
    m = lim - 1;
  }
  lcp[i] = (uint16_t)m;
}

// ---------------------------------------------------------------------------
// level-synchronous subtrie construction

struct SegArrays {
  uint32_t *start, *end, *depth, *D, *branch;
  uint64_t *slot;
};

struct SortedItems {
  const uint64_t *base;
  const uint32_t *len;
  const uint32_t *ref;
  const uint32_t *d0;
  const uint64_t *slot;
  const uint64_t *code;
  const uint16_t *lcp;
};

// leaf for item i whose path is consumed up to nibble depth x
__device__ __forceinline__ void make_leaf(const TrieView &tv, DirtyList dl, const SortedItems &si, uint32_t i,
                                          uint32_t x, uint64_t slot, uint32_t gen) {
  uint32_t len = si.len[i];
  uint32_t child = si.ref[i];
  if (x < len) {
    uint32_t s = new_short(tv, dl, si.base[i] + x, len - x, child, x, gen);
    if (s == 0xFFFFFFFFu) return;
    write_slot(tv, slot, make_ref(KIND_SHORT, s));
  } else {
    write_slot(tv, slot, child);
  }
}

// groups -> leaves (singletons) or first-level segments
// kflags bits: 0 keep, 1 child/segment start, 2 child/segment end
__global__ void k_groups_init(TrieView tv, DirtyList dl, SortedItems si, int T, uint32_t gen, uint8_t *kflags,
                              unsigned long long *flags) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T) return;
  bool gs = (i == 0) || si.code[i] != si.code[i - 1];
  bool ge = (i + 1 == T) || si.code[i + 1] != si.code[i];
  if (gs && ge) {
    make_leaf(tv, dl, si, i, si.d0[i], si.slot[i], gen);
    kflags[i] = 0;
    flags[i] = 0;
    return;
  }
  kflags[i] = 1 | (gs ? 2 : 0) | (ge ? 4 : 0);
  flags[i] = 1ull | ((unsigned long long)(gs ? 1 : 0) << 32);
}

__global__ void k_groups_scatter(SortedItems si, const uint8_t *kflags, const unsigned long long *pos, int T,
                                 uint32_t *act, uint32_t *aseg, SegArrays sg) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= T) return;
  uint8_t f = kflags[i];
  if (!(f & 1)) return;
  unsigned long long q = pos[i];
  uint32_t k = (uint32_t)q;
  uint32_t s = (uint32_t)(q >> 32) + ((f & 2) ? 1u : 0u) - 1u;
  act[k] = (uint32_t)i;
  aseg[k] = s;
  if (f & 2) {
    sg.start[s] = (uint32_t)i;
    sg.depth[s] = si.d0[i];
    sg.slot[s] = si.slot[i];
    sg.D[s] = 0xFFFFFFFFu;
  }
  if (f & 4) sg.end[s] = (uint32_t)i + 1;
}

// D[s] = min LCP over the interior boundaries of segment s
__global__ void k_level_min(SortedItems si, const uint32_t *act, const uint32_t *aseg, int K, SegArrays sg) {
  __shared__ uint32_t s_first;
  __shared__ uint32_t wmin[32];
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  bool ok = k < K;
  uint32_t s = ok ? aseg[k] : 0xFFFFFFFFu;
  uint32_t v = 0xFFFFFFFFu;
  if (ok) {
    uint32_t i = act[k];
    if (i != sg.start[s]) v = si.lcp[i];
  }
  if (threadIdx.x == 0) s_first = s;
  __syncthreads();
  int same = __syncthreads_and(!ok || s == s_first);
  if (same) {
    uint32_t w = __reduce_min_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) wmin[threadIdx.x >> 5] = w;
    __syncthreads();
    if (threadIdx.x == 0) {
      uint32_t b = wmin[0];
      for (int i = 1; i < (int)(blockDim.x >> 5); ++i) b = min(b, wmin[i]);
      if (b != 0xFFFFFFFFu && s_first != 0xFFFFFFFFu) atomicMin(&sg.D[s_first], b);
    }
    return;
  }
  unsigned peers = __match_any_sync(0xffffffffu, s);
  uint32_t w = __reduce_min_sync(peers, v);
  if (ok && (int)(threadIdx.x & 31) == __ffs(peers) - 1 && w != 0xFFFFFFFFu) atomicMin(&sg.D[s], w);
}

// one branch (+ extension) per segment
__global__ void k_level_nodes(TrieView tv, DirtyList dl, SortedItems si, int S, SegArrays sg, uint32_t gen) {
  int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= S) return;
  uint32_t D = sg.D[s];
  uint32_t d = sg.depth[s];
  uint32_t i0 = sg.start[s];
  if (D == 0xFFFFFFFFu || D < d || D >= si.len[i0]) {
    set_error(tv.ctr, ERR_INTERNAL);
    sg.branch[s] = 0xFFFFFFFFu;
    return;
  }
  uint32_t f = new_full(tv, dl, D, gen);
  sg.branch[s] = f;
  if (f == 0xFFFFFFFFu) return;
  uint32_t top = make_ref(KIND_FULL, f);
  if (D > d) {
    uint32_t e = new_short(tv, dl, si.base[i0] + d, D - d, top, d, gen);
    if (e == 0xFFFFFFFFu) return;
    top = make_ref(KIND_SHORT, e);
  }
  write_slot(tv, sg.slot[s], top);
}

// children of every branch: leaves now, larger children become segments of
// the next level
__global__ void k_level_children(TrieView tv, DirtyList dl, SortedItems si, const uint32_t *act,
                                 const uint32_t *aseg, int K, SegArrays sg, uint32_t gen, uint8_t *kflags,
                                 uint8_t *knib, unsigned long long *flags) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  uint32_t i = act[k];
  uint32_t s = aseg[k];
  uint32_t D = sg.D[s];
  uint32_t f = sg.branch[s];
  if (f == 0xFFFFFFFFu) {
    kflags[k] = 0;
    flags[k] = 0;
    return;
  }
  bool cs = (i == sg.start[s]) || si.lcp[i] == D;
  bool ce = (i + 1 == sg.end[s]) || si.lcp[i + 1] == D;
  // only the first item of a child run names the child slot: the other
  // items skip the gather of their key's nibble
  uint8_t nib = cs ? tv.keys[si.base[i] + D] : 0;
  uint64_t slot = ((uint64_t)f << 5) | nib;
  if (cs && ce) {
    make_leaf(tv, dl, si, i, D + 1, slot, gen);
    kflags[k] = 0;
    flags[k] = 0;
    return;
  }
  kflags[k] = 1 | (cs ? 2 : 0) | (ce ? 4 : 0);
  knib[k] = nib;
  flags[k] = 1ull | ((unsigned long long)(cs ? 1 : 0) << 32);
}

__global__ void k_level_scatter(const uint32_t *act, const uint32_t *aseg, const uint8_t *kflags,
                                const uint8_t *knib, const unsigned long long *pos, int K, SegArrays cur,
                                uint32_t *nact, uint32_t *naseg, SegArrays nxt) {
  int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= K) return;
  uint8_t f = kflags[k];
  if (!(f & 1)) return;
  unsigned long long q = pos[k];
  uint32_t nk = (uint32_t)q;
  uint32_t ns = (uint32_t)(q >> 32) + ((f & 2) ? 1u : 0u) - 1u;
  uint32_t i = act[k];
  uint32_t s = aseg[k];
  nact[nk] = i;
  naseg[nk] = ns;
  if (f & 2) {
    nxt.start[ns] = i;
    nxt.depth[ns] = cur.D[s] + 1;
    nxt.slot[ns] = ((uint64_t)cur.branch[s] << 5) | knib[k];
    nxt.D[ns] = 0xFFFFFFFFu;
  }
  if (f & 4) nxt.end[ns] = i + 1;
}

// ---------------------------------------------------------------------------
// PhaseHC: dirty nodes with nothing dirty below them first, then the branches
// by nibble depth, deepest first; an extension over a dirty branch is hashed
// in that branch's level

// Keccak blocks a dirty branch's encoding is expected to take, minus one,
// capped at kHashClasses - 1: children counted as 33-byte references, and a
// value in slot 16 (a key that ends at the branch) by its length, which can
// be kilobytes.  Branches of a level are binned by it, so the lanes of a warp
// need the same number of permutations and none idles through another's extra
// ones.
constexpr uint32_t kHashClasses = 8;

__device__ __forceinline__ uint32_t full_bytes(const TrieView &tv, uint32_t idx) {
  const uint32_t *c = tv.full_child + (size_t)idx * 17;
  uint32_t cnt = 0;
#pragma unroll
  for (int k = 0; k < 16; ++k) cnt += c[k] != 0u ? 1u : 0u;
  uint32_t bytes = 20u + 32u * cnt;
  const uint32_t v = c[16];
  if (ref_kind(v) == KIND_VALUE) bytes += 3u + load_rec(tv, tv.value_vid[ref_idx(v)]).len;
  return bytes;
}

__device__ __forceinline__ uint32_t full_class(const TrieView &tv, uint32_t idx) {
  return min(full_bytes(tv, idx) / 136u, kHashClasses - 1u);
}

// Leaves (short nodes over a value) depend on nothing below them, so every
// dirty leaf is hashed in one launch ahead of the levels, whatever its
// depth; the levels then hold only branches and extensions.  Leaves are
// ordered by their exact Keccak block count (minus one, capped at
// kLeafClasses - 1) over the whole batch, so a warp's 32 leaves need the
// same number of permutations.  Ordering inside one 128-node CTA alone left
// about half of the lanes idle with values of up to kilobytes (1 to 31
// blocks), and hashing leaves level by level made deep tries a chain of
// small launches, each as long as its slowest leaf.
//
// An extension over a dirty branch has one input, that branch's hash, so it
// belongs to the branch's level, not to one of its own: in a level hashed a
// warp per branch the warp goes on to it (full_ext names it), in a level
// hashed a thread per node it is listed behind the level's branches.  Keys
// whose branches sit below one-nibble extensions (ASCII digits, words) would
// otherwise take two levels per character: a 16K-key update of a 1M-key trie
// ran 21 launches, now 12.  An extension over a clean branch (what a split or
// a delete leaves above an untouched subtree) has no dirty input and goes
// with the leaves.
constexpr uint32_t kLeafClasses = 32;
// bins: the kLeafClasses leaf bins, one bin of dead short nodes (LockNU's
// splits leave many), then per nibble depth kHashClasses bins of branches,
// longest first, and one of the extensions right above those branches; a
// level is one contiguous range of the sorted dirty list
constexpr uint32_t kDeadBin = kLeafClasses;
constexpr uint32_t kBinsPerDepth = kHashClasses + 1;

__host__ __device__ __forceinline__ uint32_t level_bin(uint32_t depth) { return kLeafClasses + 1u + depth * kBinsPerDepth; }

// The extension above branch f that f's task hashes, or kNoNode.  full_ext
// may be left from an earlier pass; an extension still in the trie whose
// child is f is f's parent, and is dirty whenever f is.
__device__ __forceinline__ uint32_t ext_above(const TrieView &tv, uint32_t f) {
  const uint32_t e = __ldcg(tv.full_ext + f);
  if (e == kNoNode) return kNoNode;
  return (__ldcg(tv.short_child + e) == make_ref(KIND_FULL, f) && !__ldcg(tv.short_dead + e)) ? e : kNoNode;
}

// Bin of a dirty node at nibble depth `depth`.  Inside a launch the classes
// run longest first, so the CTAs of the slowest nodes start in the first wave
// instead of forming the last one.  Records the extension above a dirty
// branch in full_ext.
__device__ __forceinline__ uint32_t dirty_bin(const TrieView &tv, uint32_t r, uint32_t depth, bool leaf_classes) {
  const uint32_t idx = ref_idx(r);
  if (ref_kind(r) == KIND_FULL) return level_bin(depth) + kHashClasses - 1u - full_class(tv, idx);
  if (tv.short_dead[idx]) return kDeadBin;
  const uint32_t ch = tv.short_child[idx];
  if (ref_kind(ch) == KIND_FULL && tv.full_epoch[ref_idx(ch)] == tv.gen) {
    tv.full_ext[ref_idx(ch)] = idx;
    return level_bin(depth + tv.short_klen[idx]) + kHashClasses;
  }
  if (!leaf_classes) return kLeafClasses - 1u;
  uint32_t bytes = tv.short_klen[idx] / 2u + 8u;
  bytes += ref_kind(ch) == KIND_VALUE ? load_rec(tv, tv.value_vid[ref_idx(ch)]).len : 33u;
  return kLeafClasses - 1u - min(bytes / 136u, kLeafClasses - 1u);
}

// Histogram of the dirty list over the bins (nbins of them, covering every
// depth a node can have).  Leaves are classed by block count only when
// `leaf_classes` is set (a batch held values long enough for a leaf to take
// two or more Keccak blocks).  Counts are aggregated per warp: one shared
// atomic per distinct bin, not one per node (a load's millions of leaves
// share one bin and would queue on its address).
__global__ void k_dirty_hist(TrieView tv, const uint32_t *ref, const uint16_t *depth, int n, uint32_t *bins,
                             int nbins, int leaf_classes, uint16_t *bin_of) {
  extern __shared__ uint32_t h[];
  for (int b = threadIdx.x; b < nbins; b += blockDim.x) h[b] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int i0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31); i0 < n; i0 += gridDim.x * blockDim.x) {
    const int i = i0 + lane;
    uint32_t b = 0xFFFFFFFFu;
    if (i < n) {
      b = min(dirty_bin(tv, ref[i], depth[i], leaf_classes != 0), (uint32_t)nbins - 1u);
      bin_of[i] = (uint16_t)b;
    }
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    if (i < n && lane == __ffs(peers) - 1) atomicAdd(&h[b], (uint32_t)__popc(peers));
  }
  __syncthreads();
  for (int b = threadIdx.x; b < nbins; b += blockDim.x)
    if (h[b]) atomicAdd(&bins[b], h[b]);
}

// Scatter of the dirty list into its bins, 256 entries per CTA pass.  Counts
// are aggregated per warp (match_any) and then per CTA in a shared table of
// the bins the pass touches, so a hot bin (a level of millions of leaves)
// takes one global atomic per CTA pass instead of one per warp.
__global__ void __launch_bounds__(256) k_dirty_scatter(const uint32_t *ref, const uint16_t *bin_of, int n,
                                                       uint32_t *cursor, uint32_t *out, Counters *ctr) {
  constexpr uint32_t kEmpty = 0xFFFFFFFFu;
  __shared__ uint32_t tbin[256], tcnt[256], tbase[256];
  const int lane = threadIdx.x & 31;
  for (int c0 = blockIdx.x * 256; c0 < n; c0 += gridDim.x * 256) {
    tbin[threadIdx.x] = kEmpty;
    tcnt[threadIdx.x] = 0;
    __syncthreads();
    const int i = c0 + threadIdx.x;
    const bool ok = i < n;
    const uint32_t r = ok ? ref[i] : 0u;
    const uint32_t b = ok ? bin_of[i] : kEmpty;
    const unsigned peers = __match_any_sync(0xffffffffu, b);
    const int leader = __ffs(peers) - 1;
    uint32_t slot = 0, off = 0, claimed = 0;
    if (ok && lane == leader) {
      slot = (b * 0x9E3779B1u) >> 24;  // at most 256 bins per pass: a free slot exists
      for (int probe = 0; probe < 256; ++probe) {
        const uint32_t prev = atomicCAS(&tbin[slot], kEmpty, b);
        if (prev == kEmpty || prev == b) {
          claimed = 1;
          break;
        }
        slot = (slot + 1) & 255u;
      }
      // no slot of this bin (cannot happen with <= 256 bins per pass): report
      // it and leave the entries out rather than count them in another bin
      if (claimed)
        off = atomicAdd(&tcnt[slot], (uint32_t)__popc(peers));
      else
        set_error(ctr, ERR_INTERNAL);
    }
    slot = __shfl_sync(0xffffffffu, slot, leader);
    off = __shfl_sync(0xffffffffu, off, leader);
    claimed = __shfl_sync(0xffffffffu, claimed, leader);
    __syncthreads();
    if (tbin[threadIdx.x] != kEmpty) tbase[threadIdx.x] = atomicAdd(&cursor[tbin[threadIdx.x]], tcnt[threadIdx.x]);
    __syncthreads();
    if (ok && claimed) out[tbase[slot] + off + __popc(peers & ((1u << lane) - 1u))] = r;
    __syncthreads();
  }
}

// one message item: <= 8 prefix bytes, then a body read from memory
struct EncItem {
  uint64_t pre;
  uint32_t pren;
  uint32_t nib;  // body holds nibbles, packed in pairs
  const uint8_t *body;
  uint32_t blen;
};

__device__ __forceinline__ int be_size(uint64_t v) {
  int s = 1;
  while (v >>= 8) ++s;
  return s;
}

// RLP header bytes (tag small/large) for a payload of `size`, little-endian
__device__ __forceinline__ void rlp_head(uint64_t size, uint32_t small_tag, uint32_t large_tag, uint64_t &pre,
                                         uint32_t &pren) {
  if (size < 56) {
    pre = small_tag + size;
    pren = 1;
    return;
  }
  int s = be_size(size);
  pre = large_tag + (uint32_t)s;
  for (int k = 0; k < s; ++k) pre |= ((size >> (8 * (s - 1 - k))) & 0xFF) << (8 * (1 + k));
  pren = 1 + s;
}

// Loads of node fields and message bytes.  kCoh = true inside a persistent
// launch, where the data may have been written earlier in the same launch by
// another SM, before a grid barrier (fence, arrive, wait, fence): ordinary
// loads then see those writes, but the non-coherent read-only path
// (ld.global.nc) is not used for them.  Key nibbles are staged by an earlier
// launch and stay on the read-only path in both modes.
template <bool kCoh, typename T>
__device__ __forceinline__ T ldn(const T *p) {
  return *p;
}

template <bool kCoh>
__device__ __forceinline__ uint64_t ld8(const uint8_t *p) {
  if constexpr (kCoh)
    return load_u64_unaligned_cg(p);
  else
    return load_u64_unaligned(p);
}

// the item a parent writes for child `r` (node.cuh:437-450 / 548-557;
// rlp.cuh:132-155 write_bytes; a value node's "hash" is its raw value)
template <bool kCoh = false>
__device__ __forceinline__ EncItem child_item(const TrieView &tv, uint32_t r) {
  EncItem it{0, 0, 0, nullptr, 0};
  uint32_t kind = ref_kind(r), idx = ref_idx(r);
  if (kind == KIND_NULL) {
    it.pre = 0x80;
    it.pren = 1;
    return it;
  }
  const uint8_t *h;
  uint32_t hl;
  if (kind == KIND_VALUE) {
    unsigned long long vid = ldn<kCoh>(tv.value_vid + idx);
    const ValueRec rc = load_rec(tv, vid);
    h = tv.vals + rc.off;
    hl = rc.len;
  } else {
    if (kind == KIND_FULL) {
      h = tv.full_hash + (size_t)idx * 32;
      hl = ldn<kCoh>(tv.full_hlen + idx);
    } else {
      h = tv.short_hash + (size_t)idx * 32;
      hl = ldn<kCoh>(tv.short_hlen + idx);
    }
    if (tv.geth_mode && hl < 32) {  // go-ethereum embeds small nodes
      it.body = h;
      it.blen = hl;
      return it;
    }
  }
  it.body = h;
  it.blen = hl;
  if (hl == 1 && ldn<kCoh>(h) < 0x80) return it;  // single byte is its own encoding
  rlp_head(hl, 0x80, 0xb7, it.pre, it.pren);
  return it;
}

// compact (hex-prefix) key item: utils.cuh:361-396 hex_to_compact
__device__ __forceinline__ EncItem compact_item(const TrieView &tv, uint64_t koff, uint32_t klen) {
  EncItem it{0, 0, 1, nullptr, 0};
  const uint8_t *k = tv.keys + koff;
  uint32_t term = (klen > 0 && k[klen - 1] == 16) ? 1 : 0;
  uint32_t ln = klen - term;
  uint32_t odd = ln & 1;
  uint32_t clen = ln / 2 + 1;
  uint32_t flag = (term << 5) | (odd ? (0x10u | k[0]) : 0u);
  it.body = k + odd;
  it.blen = clen - 1;
  if (clen == 1) {  // one byte < 0x80: written as itself
    it.pre = flag;
    it.pren = 1;
    return it;
  }
  uint64_t h;
  uint32_t hn;
  rlp_head(clen, 0x80, 0xb7, h, hn);
  it.pre = h | ((uint64_t)flag << (8 * hn));
  it.pren = hn + 1;
  return it;
}

// 16 nibble bytes -> 8 bytes (hi << 4 | lo)
__device__ __forceinline__ uint64_t pack_pairs8(const uint8_t *p) {
  uint64_t r = 0;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    uint64_t x = load_u64_unaligned(p + 8 * h);
    uint64_t z = ((x & 0x000F000F000F000Full) << 4) | ((x >> 8) & 0x000F000F000F000Full);
    z = (z | (z >> 8)) & 0x0000FFFF0000FFFFull;
    z = (z | (z >> 16)) & 0x00000000FFFFFFFFull;
    r |= z << (32 * h);
  }
  return r;
}

template <bool kCoh = false>
__device__ __forceinline__ EncItem node_item(const TrieView &tv, bool full, uint32_t idx, int item,
                                             uint64_t payload) {
  EncItem it{0, 0, 0, nullptr, 0};
  if (item == 0) {
    rlp_head(payload, 0xc0, 0xf7, it.pre, it.pren);
    return it;
  }
  if (full) return child_item<kCoh>(tv, ldn<kCoh>(tv.full_child + (size_t)idx * 17 + (item - 1)));
  if (item == 1) return compact_item(tv, ldn<kCoh>(tv.short_key + idx), ldn<kCoh>(tv.short_klen + idx));
  return child_item<kCoh>(tv, ldn<kCoh>(tv.short_child + idx));
}

// Thread per dirty node: RLP-encode straight into the sponge, Keccak-256 if
// the encoding is >= 32 bytes, else keep it raw (gpu_mpt_kernels.cuh:2885-3045
// semantics; cpu_mpt.cuh:380-496).
__device__ __forceinline__ void prefetch_l1(const void *p) {
  asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// One thread's message, written front to back as 32-bit words: word w goes
// to st[w * stride], each once.  Bytes pending for the next word are the top
// `pb` bytes of `prev`, so a whole source word costs one funnel shift and one
// store whatever the byte position is.
struct WordWriter {
  uint32_t *st;
  uint32_t stride;
  uint32_t w = 0, pb = 0, prev = 0;
  __device__ __forceinline__ WordWriter(uint32_t *s, uint32_t n) : st(s), stride(n) {}
  __device__ __forceinline__ void word(uint32_t v) {
    st[w * stride] = __funnelshift_l(prev, v, 8 * pb);
    ++w;
    prev = v;
  }
  // the low n (0..4) bytes of v
  __device__ __forceinline__ void bytes(uint32_t v, uint32_t n) {
    const uint32_t t = __funnelshift_l(prev, v, 8 * pb);  // pending bytes, then v
    const uint32_t have = pb + n;
    if (have >= 4) {
      st[w * stride] = t;
      ++w;
      pb = have - 4;
      prev = v << (8 * (4 - n));  // n >= 1 here: its last bytes on top
    } else {
      pb = have;
      prev = have ? t << (8 * (4 - have)) : 0u;
    }
  }
  // the low n (0..8) bytes of v
  __device__ __forceinline__ void bytes8(uint64_t v, uint32_t n) {
    bytes((uint32_t)v, min(n, 4u));
    if (n > 4) bytes((uint32_t)(v >> 32), n - 4);
  }
};

// Four aligned 8-byte words covering bytes from `src` on, and the funnel that
// takes unaligned 32-bit words out of them.  Loading four at a time keeps a
// gather's L2 round trips to one per 32 bytes.
struct SrcWords {
  const uint2 *q;
  uint32_t sh, skew;
  bool up;
  __device__ __forceinline__ explicit SrcWords(const uint8_t *src) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(src);
    q = reinterpret_cast<const uint2 *>(a & ~uintptr_t(7));
    skew = (uint32_t)(a & 7);
    sh = 8 * (skew & 3);
    up = (skew & 4) != 0;
  }
  // unaligned 32-bit words 0 and 1 from aligned words c, d
  __device__ __forceinline__ uint2 pair(uint2 c, uint2 d) const {
    const uint32_t x0 = up ? c.y : c.x, x1 = up ? d.x : c.y, x2 = up ? d.y : d.x;
    return make_uint2(__funnelshift_r(x0, x1, sh), __funnelshift_r(x1, x2, sh));
  }
};

// n bytes at src (any alignment) appended to the message.  An aligned word is
// read only if the n bytes reach into it.
template <bool kCoh>
__device__ __forceinline__ void write_body(WordWriter &o, const uint8_t *src, uint32_t n) {
  const SrcWords s(src);
  const uint32_t words = (n + s.skew + 7) / 8;
  auto ld = [&](uint32_t j) -> uint2 {
    if (j >= words) return make_uint2(0u, 0u);
    if constexpr (kCoh)
      return s.q[j];
    else
      return __ldg(s.q + j);
  };
  uint2 c = ld(0);
  for (uint32_t j = 0; 8 * j < n; j += 4) {
    const uint2 d[4] = {ld(j + 1), ld(j + 2), ld(j + 3), ld(j + 4)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t at = 8 * (j + k);
      const uint2 v = s.pair(c, d[k]);
      c = d[k];
      if (at + 8 <= n) {
        o.word(v.x);
        o.word(v.y);
      } else if (at < n) {
        const uint32_t r = n - at;  // 1..7
        o.bytes(v.x, min(r, 4u));
        if (r > 4) o.bytes(v.y, r - 4);
      }
    }
  }
}

// Four bytes from eight nibble bytes (first nibble of a byte is its high half).
__device__ __forceinline__ uint32_t pack_pairs4(uint2 v) {
  return __byte_perm((v.x << 4) | (v.x >> 8), (v.y << 4) | (v.y >> 8), 0x6420);
}

// n bytes packed from 2n nibbles at src appended to the message.
__device__ __forceinline__ void write_nibbles(WordWriter &o, const uint8_t *src, uint32_t n) {
  const SrcWords s(src);
  const uint32_t words = (2 * n + s.skew + 7) / 8;
  auto ld = [&](uint32_t j) { return j < words ? __ldg(s.q + j) : make_uint2(0u, 0u); };
  uint2 c = ld(0);
  for (uint32_t j = 0; 4 * j < n; j += 4) {
    const uint2 d[4] = {ld(j + 1), ld(j + 2), ld(j + 3), ld(j + 4)};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const uint32_t at = 4 * (j + k);
      const uint32_t v = pack_pairs4(s.pair(c, d[k]));
      c = d[k];
      if (at + 4 <= n)
        o.word(v);
      else if (at < n)
        o.bytes(v, n - at);
    }
  }
}

// Staging words (32-bit) per thread: a block, and what one branch child (gap
// bytes, tag and hash) can run past its end.
constexpr uint32_t kStageWords = 34 + 14;

// Message of a regular branch, block by block: 0x80 per empty slot, 0xa0 + 32
// hash bytes per child, then the Keccak padding (rlp.cuh:132-155,
// node.cuh:46-112).  A child at a time: its hash in two 16-byte loads, eight
// funnel-shifted words out; what the last child writes past a block moves to
// the front of the next.
template <bool kCoh>
struct BranchWriter {
  WordWriter o;
  uint32_t left;
  int prev = -1;
  bool done = false;
  __device__ __forceinline__ BranchWriter(uint32_t *st, uint32_t stride, uint64_t hdr, uint32_t hn, uint32_t present)
      : o(st, stride), left(present) {
    o.bytes((uint32_t)hdr, hn);
  }
  // stage the next block; true: it is the last one
  __device__ __forceinline__ bool fill(const TrieView &tv, const uint32_t *chp) {
    while (o.w < 34 && !done) {
      const int k = left ? __ffs(left) - 1 : 17;  // next child, or the end
      left &= left - 1;
      uint32_t gap = (uint32_t)(k - prev - 1);
      prev = k;
      if (k < 17) {
        const uint32_t r = ldn<kCoh>(chp + k);
        const uint4 *h = reinterpret_cast<const uint4 *>(
            (ref_kind(r) == KIND_FULL ? tv.full_hash : tv.short_hash) + (size_t)ref_idx(r) * 32);
        const uint4 x = ldn<kCoh>(h), y = ldn<kCoh>(h + 1);
        for (; gap >= 4; gap -= 4) o.word(0x80808080u);
        // gap (0..3) empty slots, then the child's tag
        o.bytes((0x80808080u & ((1u << (8 * gap)) - 1u)) | (0xa0u << (8 * gap)), gap + 1);
        o.word(x.x), o.word(x.y), o.word(x.z), o.word(x.w);
        o.word(y.x), o.word(y.y), o.word(y.z), o.word(y.w);
      } else {
        for (; gap >= 4; gap -= 4) o.word(0x80808080u);
        o.bytes((0x80808080u & ((1u << (8 * gap)) - 1u)) | (0x01u << (8 * gap)), gap + 1);
        o.bytes(0u, o.pb ? 4 - o.pb : 0u);  // whole words from here on
        done = true;
      }
    }
    const bool last = done && o.w <= 34;
    if (last) {
      for (uint32_t w = o.w; w < 34; ++w) o.st[w * o.stride] = 0;
      o.st[33 * o.stride] |= 0x80000000u;
    }
    return last;
  }
  // after a block that was not the last
  __device__ __forceinline__ void next() {
    for (uint32_t w = 34; w < o.w; ++w) o.st[(w - 34) * o.stride] = o.st[w * o.stride];
    o.w -= 34;
  }
};

// Message of any branch, block by block: its items one after another (values
// of up to kilobytes, children below 32 bytes).
template <bool kCoh>
struct ItemWriter {
  WordWriter o;
  EncItem cur;
  uint32_t item = 0, off = 0;  // item 0: the list header, then the 17 slots
  bool pre = true, done = false;
  __device__ __forceinline__ ItemWriter(uint32_t *st, uint32_t stride, uint64_t hdr, uint32_t hn)
      : o(st, stride), cur{hdr, hn, 0, nullptr, 0} {}
  __device__ __forceinline__ bool fill(const TrieView &tv, const uint32_t *chp) {
    while (o.w < 34 && !done) {
      if (pre) {
        pre = false;
        o.bytes8(cur.pre, cur.pren);
      } else if (off < cur.blen) {
        const uint32_t n = min(cur.blen - off, 32u);
        write_body<kCoh>(o, cur.body + off, n);
        off += n;
      } else if (++item <= 17) {
        cur = child_item<kCoh>(tv, ldn<kCoh>(chp + item - 1));
        off = 0;
        pre = true;
      } else {
        o.bytes(0x01u, 1);
        o.bytes(0u, o.pb ? 4 - o.pb : 0u);
        done = true;
      }
    }
    const bool last = done && o.w <= 34;
    if (last) {
      for (uint32_t w = o.w; w < 34; ++w) o.st[w * o.stride] = 0;
      o.st[33 * o.stride] |= 0x80000000u;
    }
    return last;
  }
  __device__ __forceinline__ void next() {
    for (uint32_t w = 34; w < o.w; ++w) o.st[(w - 34) * o.stride] = o.st[w * o.stride];
    o.w -= 34;
  }
};

// Encode + hash one dirty node; `stage` is this thread's column of the
// message block in shared memory (kStageWords 32-bit words, word w at
// stage[w * stride]).
//
// Bound by the integer pipe (one permutation per 136 bytes), so the encoders
// around it are kept to few instructions per byte: whole words through one
// funnel shift, a branch child's hash in two 16-byte loads.  16M-key YCSB
// load: 16.7M one-block leaves 6.08 -> 5.12 ms (3.26 G permutations/s, 0.81
// of the register-only rate; random value gathers are the rest), 5.1M
// branches of two or three children 1.96 -> 1.56 ms, their extensions 1.28 ms
// (0.97 of it).
template <bool kCoh, bool full>
__device__ __forceinline__ void hash_node(const TrieView &tv, uint32_t idx, uint32_t *stage, uint32_t stride) {
  const bool dead = ldn<kCoh>((full ? tv.full_dead : tv.short_dead) + idx) != 0;
  // a short node's fields, loaded together
  uint64_t skey = 0;
  uint32_t sklen = 0, schild = 0;
  if (!full) {
    skey = ldn<kCoh>(tv.short_key + idx);
    sklen = ldn<kCoh>(tv.short_klen + idx);
    schild = ldn<kCoh>(tv.short_child + idx);
  }
  if (dead) return;  // unlinked by a split or a delete
  // depth 0 holds exactly the roots of the forest's tries; go-ethereum
  // hashes a root whatever its size
  bool force = tv.geth_mode && (full ? ldn<kCoh>(tv.full_depth + idx) : ldn<kCoh>(tv.short_depth + idx)) == 0;
  int nitems = full ? 18 : 3;
  // pass 1: payload size (all child loads issued together)
  uint64_t payload = 0;
  EncItem it1{0, 0, 0, nullptr, 0}, it2{0, 0, 0, nullptr, 0};  // short: key, child
  const uint32_t *chp = tv.full_child + (size_t)idx * 17;
  // branch whose children are all hashed nodes (32-byte references) and whose
  // value slot is empty: its encoding is regular and is generated child by
  // child.  While no node of the tries has had an encoding below 32 bytes
  // (raw_nodes) the children's lengths need no look: a gather of one byte per
  // child, which costs a sector each.
  uint32_t present = 0;
  bool regular = full;
  if (full) {
    uint32_t ch[17];
#pragma unroll
    for (int k = 0; k < 17; ++k) ch[k] = ldn<kCoh>(chp + k);
    const bool any_raw = __ldcg(&tv.ctr->raw_nodes) != 0;
#pragma unroll
    for (int k = 0; k < 17; ++k) {
      const uint32_t kd = ref_kind(ch[k]);
      present |= (kd != KIND_NULL ? 1u : 0u) << k;
      regular = regular && kd != KIND_VALUE;
    }
    regular = regular && present < (1u << 16);
    payload = 17u + 32u * __popc(present);
    if (any_raw || !regular) {
      payload = 0;
#pragma unroll
      for (int k = 0; k < 17; ++k) {
        const EncItem it = child_item<kCoh>(tv, ch[k]);
        payload += it.pren + it.blen;
        const uint32_t kd = ref_kind(ch[k]);
        if (kd == KIND_VALUE) {  // a key ending here: its value (up to kilobytes) closes the encoding
          prefetch_l1(it.body);
          if (it.blen > 120) prefetch_l1(it.body + 128);
        }
        if (kd != KIND_NULL) regular = regular && it.blen == 32 && it.pren == 1;
      }
    }
  } else {
    prefetch_l1(tv.keys + skey);
    it2 = child_item<kCoh>(tv, schild);
    if (ref_kind(schild) == KIND_VALUE) {
      prefetch_l1(it2.body);
      if (it2.blen > 120) prefetch_l1(it2.body + 128);
    }
    it1 = compact_item(tv, skey, sklen);
    payload = it1.pren + it1.blen + it2.pren + it2.blen;
  }
  uint64_t hdr;
  uint32_t hn;
  rlp_head(payload, 0xc0, 0xf7, hdr, hn);
  uint64_t total = payload + hn;
  bool raw = total < 32 && !force;
  Sponge sp;
  sp.reset(stage, stride);
  if (!full && total <= 135) {
    // One-block short node (every leaf with a value up to ~100 bytes, every
    // extension): header, key, child, padding, permuted once.
    WordWriter o(stage, stride);
    o.bytes((uint32_t)hdr, hn);  // at most two bytes here
    o.bytes8(it1.pre, it1.pren);
    write_nibbles(o, it1.body, it1.blen);
    o.bytes((uint32_t)it2.pre, it2.pren);
    write_body<kCoh>(o, it2.body, it2.blen);
    if (raw) {
      const uint32_t z = total == 0 ? 0u : (uint32_t)total;
      o.bytes(0u, 4);  // flush the pending bytes
      for (uint32_t w = o.w; w < 8; ++w) stage[w * stride] = 0;
      uint64_t keep[4];
#pragma unroll
      for (int w = 0; w < 4; ++w) {
        keep[w] = sp.word(w);
        const int left = (int)z - 8 * w;
        keep[w] = left >= 8 ? keep[w] : (left <= 0 ? 0ull : (keep[w] & ((1ull << (8 * left)) - 1)));
      }
#pragma unroll
      for (int w = 0; w < 4; ++w) sp.a[w] = keep[w];
    } else {
      o.bytes(0x01u, 1);
      o.bytes(0u, 3);  // at least the pending bytes; position 135 is inside the block
      for (uint32_t w = o.w; w < 34; ++w) stage[w * stride] = 0;
      stage[33 * stride] |= 0x80000000u;
      sp.absorb();
    }
  } else if (regular) {
    BranchWriter<kCoh> bw(stage, stride, hdr, hn, present);
    while (true) {
      const bool last = bw.fill(tv, chp);
      sp.absorb();
      if (last) break;
      bw.next();
    }
  } else {
  // pass 2: stream
  int item = 0;
  EncItem cur{hdr, hn, 0, nullptr, 0};
  uint32_t off = 0;
  bool pre_pending = true, last = false;
  while (true) {
    while (!sp.full()) {
      if (pre_pending) {
        pre_pending = false;
        if (cur.pren) sp.push(cur.pre, cur.pren);
        continue;
      }
      if (off < cur.blen) {
        const uint32_t room = 17u - sp.w;  // whole words left in this block
        if (!cur.nib && cur.blen - off >= 8u * room) {
          // the item (a long value) covers the rest of the block: whole
          // words straight from memory, the loads independent of each other
          // (the partial word carried in acc keeps its length)
          const uint8_t *src = cur.body + off;
          const uint32_t ca = 8u * sp.accn;
#pragma unroll 4
          for (uint32_t i = 0; i < room; ++i) {
            const uint64_t x = ld8<kCoh>(src + 8u * i);
            if (ca == 0) {
              sp.emit(x);
            } else {
              sp.emit(sp.acc | (x << ca));
              sp.acc = x >> (64u - ca);
            }
          }
          off += 8u * room;
          continue;
        }
        uint32_t nb = min(8u, cur.blen - off);
        uint64_t v = cur.nib ? pack_pairs8(cur.body + 2 * off) : ld8<kCoh>(cur.body + off);
        sp.push(v & low_bytes_mask(nb), nb);
        off += nb;
        continue;
      }
      if (++item == nitems) {
        sp.pad();
        last = true;
        break;
      }
      cur = node_item<kCoh>(tv, full, idx, item, payload);
      off = 0;
      pre_pending = true;
    }
    if (raw) break;
    // a long body (a value of up to kilobytes) streams through many blocks:
    // start the loads of the next two lines of it before the permutation,
    // so they arrive while it runs (addresses stay inside the body)
    if (cur.body && !cur.nib && off < cur.blen) {
      const uint32_t rest = cur.blen - off - 1;
      prefetch_l1(cur.body + off + min(128u, rest));
      prefetch_l1(cur.body + off + min(256u, rest));
    }
    sp.absorb();
    if (last) break;
  }
  }
  if (tv.account) {  // accounting (timing mode): encoding bytes and absorbed blocks of this pass
    unsigned am = __activemask();
    unsigned long long eb = __reduce_add_sync(am, (uint32_t)total);
    unsigned long long kb = __reduce_add_sync(am, raw ? 0u : (uint32_t)((total + 1 + 135) / 136));
    uint32_t nh = __popc(am);
    if ((int)(threadIdx.x & 31) == __ffs(am) - 1) {
      atomicAdd(&tv.ctr->enc_bytes, eb);
      atomicAdd(&tv.ctr->keccak_blocks, kb);
      atomicAdd(&tv.ctr->hashed, nh);
    }
  }
  uint8_t *hout = (full ? tv.full_hash : tv.short_hash) + (size_t)idx * 32;
  uint64_t *o = reinterpret_cast<uint64_t *>(hout);
  if (raw && full) {  // a short node's is in sp.a already
#pragma unroll
    for (int w = 0; w < 4; ++w) {
      uint64_t v = sp.word(w);
      int keep = (int)total - 8 * w;
      sp.a[w] = keep >= 8 ? v : (keep <= 0 ? 0ull : (v & ((1ull << (8 * keep)) - 1)));
    }
  }
  reinterpret_cast<ulonglong2 *>(o)[0] = make_ulonglong2(sp.a[0], sp.a[1]);
  reinterpret_cast<ulonglong2 *>(o)[1] = make_ulonglong2(sp.a[2], sp.a[3]);
  (full ? tv.full_hlen : tv.short_hlen)[idx] = raw ? (uint8_t)total : 32;
  if (raw) tv.ctr->raw_nodes = 1;
}

// Message buffer of one warp for the warp-cooperative hashing (8 Keccak blocks).
constexpr int kWarpMsgBytes = 8 * 136;

// Up to 32 bytes of a message item, in four little-endian words.
struct Bytes32 {
  uint64_t w[4];
};

// One lane's item of a message: at most 8 prefix bytes in pre (a string's or a
// list's header: 5 for a length of 32 bits), and a body that is in registers
// when it has at most 32 bytes (a node's hash, a short value), else in memory.
struct WarpItem {
  uint64_t pre = 0;
  uint32_t pren = 0, blen = 0;
  Bytes32 body{};
  const uint8_t *far = nullptr;  // body of more than 32 bytes
};

// Header of a child node's item once its hash (or encoding below 32 bytes) is
// in the body.
__device__ __forceinline__ void node_head(const TrieView &tv, WarpItem &it) {
  if (tv.geth_mode && it.blen < 32) return;                         // go-ethereum embeds small nodes
  if (it.blen == 1 && (uint8_t)it.body.w[0] < 0x80) return;         // single byte is its own encoding
  rlp_head(it.blen, 0x80, 0xb7, it.pre, it.pren);
}

// The item a branch (or a short node) writes for child `r`: child_item with
// the bytes of hashes and short values already loaded, every load of a lane
// issued before the first is used.
template <bool kCoh>
__device__ __forceinline__ WarpItem warp_child_item(const TrieView &tv, uint32_t r) {
  WarpItem it;
  const uint32_t kind = ref_kind(r), idx = ref_idx(r);
  if (kind == KIND_NULL) {
    it.pre = 0x80;
    it.pren = 1;
    return it;
  }
  if (kind == KIND_VALUE) {
    const unsigned long long vid = ldn<kCoh>(tv.value_vid + idx);
    const ValueRec rc = load_rec(tv, vid);
    const uint8_t *v = tv.vals + rc.off;
    it.blen = rc.len;
    if (rc.len > 32) {
      it.far = v;
    } else {
#pragma unroll
      for (uint32_t w = 0; w < 4; ++w)
        if (8 * w < rc.len) it.body.w[w] = ld8<kCoh>(v + 8 * w);
    }
  } else {
    const bool full = kind == KIND_FULL;
    const ulonglong2 *h = reinterpret_cast<const ulonglong2 *>((full ? tv.full_hash : tv.short_hash) + (size_t)idx * 32);
    const ulonglong2 a = __ldcg(h), b = __ldcg(h + 1);
    it.blen = __ldcg((full ? tv.full_hlen : tv.short_hlen) + idx);
    it.body = Bytes32{{a.x, a.y, b.x, b.y}};
    node_head(tv, it);
    return it;
  }
  if (it.blen == 1 && (uint8_t)it.body.w[0] < 0x80) return it;  // single byte is its own encoding
  rlp_head(it.blen, 0x80, 0xb7, it.pre, it.pren);
  return it;
}

// Bytes [0, n) of v at message position p, clipped to the window [lo, hi).
__device__ __forceinline__ void put_prefix(uint8_t *msg, uint32_t lo, uint32_t hi, uint64_t v, uint32_t n, uint32_t p) {
  for (uint32_t q = 0; q < n; ++q)
    if (p + q >= lo && p + q < hi) msg[p + q - lo] = (uint8_t)(v >> (8 * q));
}

// A body held in registers (at most 32 bytes) at position p, clipped.
__device__ __forceinline__ void put_body32(uint8_t *msg, uint32_t lo, uint32_t hi, const Bytes32 &b, uint32_t n,
                                           uint32_t p) {
  if (p + n <= lo || p >= hi) return;
  if (p >= lo && p + n <= hi) {
    uint8_t *m = msg + (p - lo);
#pragma unroll
    for (uint32_t j = 0; j < 32; ++j)
      if (j < n) m[j] = (uint8_t)(b.w[j >> 3] >> (8 * (j & 7)));
  } else {  // across a window's edge (behind a long value)
#pragma unroll
    for (uint32_t w = 0; w < 4; ++w) put_prefix(msg, lo, hi, b.w[w], n > 8 * w ? min(8u, n - 8 * w) : 0u, p + 8 * w);
  }
}

// The warp copies a long body (n bytes at src, message position p), clipped:
// whole aligned 8-byte words of the window where it covers them (unaligned
// loads, all lanes' in flight together), single bytes at the two ends.
template <bool kCoh>
__device__ __forceinline__ void put_far(uint8_t *msg, uint32_t lo, uint32_t hi, const uint8_t *src, uint32_t n,
                                        uint32_t p, int lane) {
  const uint32_t a = max(p, lo) - lo, z = min(p + n, hi) - lo;  // window range
  if (p + n <= lo || p >= hi) return;
  const uint8_t *s0 = src + ((int64_t)lo - (int64_t)p);  // byte of window offset 0 (read only inside [a, z))
  const uint32_t wa = (a + 7) & ~7u, wz = z & ~7u;
  if (wa >= wz) {
    for (uint32_t j = a + lane; j < z; j += 32) msg[j] = ldn<kCoh>(s0 + j);
    return;
  }
  uint64_t *m64 = reinterpret_cast<uint64_t *>(msg);
  for (uint32_t j = wa + 8u * lane; j < wz; j += 256) m64[j >> 3] = ld8<kCoh>(s0 + j);
  if (a + lane < wa) msg[a + lane] = ldn<kCoh>(s0 + a + lane);
  if (wz + lane < z) msg[wz + lane] = ldn<kCoh>(s0 + wz + lane);
}

// Zero the blocks [b0, b0 + wb) of a message in the warp's window.
__device__ __forceinline__ void window_clear(uint64_t *m64, uint32_t wb, int lane) {
  for (uint32_t w = lane; w < wb * 17; w += 32) m64[w] = 0;
  __syncwarp();
}

// Keccak padding (0x01 after the message, 0x80 on the last byte) of the bytes
// in the window [lo, lo + 136 wb) of a `total`-byte message of nblk blocks;
// nothing else writes these bytes.
__device__ __forceinline__ void put_padding(uint8_t *msg, uint32_t lo, uint32_t wb, uint32_t total, uint32_t nblk) {
  const uint32_t end = nblk * 136 - 1;
  if (total >= lo && total < lo + wb * 136) msg[total - lo] = total == end ? 0x81 : 0x01;
  if (total != end && end < lo + wb * 136) msg[end - lo] = 0x80;
}

// Absorb the window's wb blocks into the warp-spread state.
__device__ __forceinline__ uint64_t window_absorb(uint64_t a, const uint64_t *m64, uint32_t wb, const CoopLanes &cl,
                                                  int lane) {
  for (uint32_t bb = 0; bb < wb; ++bb) {
    if (lane < 17) a ^= m64[bb * 17 + lane];
    a = keccak_f1600_warp(a, cl);
  }
  __syncwarp();  // the next window reuses the buffer
  return a;
}

// Store a node's 32-byte hash (a: the warp-spread state) or, below 32 bytes,
// its encoding (the zero-padded window); returns lane l's word of it for
// l < 4.
__device__ __forceinline__ uint64_t store_hash(const TrieView &tv, uint64_t *o, uint8_t *hlen, bool raw, uint64_t a,
                                               const uint64_t *m64, uint32_t total, uint32_t nblk, int lane) {
  const uint64_t v = raw ? m64[lane & 3] : a;
  if (lane < 4) o[lane] = v;
  if (lane == 0) *hlen = raw ? (uint8_t)total : 32;
  if (lane == 0 && raw) tv.ctr->raw_nodes = 1;
  if (lane == 0 && tv.account) {
    atomicAdd(&tv.ctr->enc_bytes, (unsigned long long)total);
    atomicAdd(&tv.ctr->keccak_blocks, (unsigned long long)(raw ? 0u : nblk));
    atomicAdd(&tv.ctr->hashed, 1u);
  }
  __syncwarp();
  return v;
}

// Warp-cooperative encode + hash of short node idx (a leaf, or an extension).
// known: the child's hash (hw: lane l < 4 holds word l, hl bytes) comes from
// the caller, which has just computed it.  All 32 lanes call it alike.
template <bool kCoh>
__device__ __forceinline__ void hash_short_warp(const TrieView &tv, uint32_t idx, uint8_t *msg, const CoopLanes &cl,
                                                bool known, uint64_t hw, uint32_t hl) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint64_t ko = ldn<kCoh>(tv.short_key + idx);
  const uint32_t klen = ldn<kCoh>(tv.short_klen + idx);
  const uint32_t child = ldn<kCoh>(tv.short_child + idx);
  const bool dead = ldn<kCoh>(tv.short_dead + idx) != 0;
  const bool force = tv.geth_mode && ldn<kCoh>(tv.short_depth + idx) == 0;
  if (dead) return;  // unlinked by a split or a delete
  const EncItem key = compact_item(tv, ko, klen);
  WarpItem it;
  if (known) {
    it.blen = hl;
#pragma unroll
    for (int w = 0; w < 4; ++w) it.body.w[w] = __shfl_sync(kAll, hw, w);
    node_head(tv, it);
  } else {
    it = warp_child_item<kCoh>(tv, child);
  }
  const uint32_t payload = key.pren + key.blen + it.pren + it.blen;
  uint64_t hdr;
  uint32_t hn;
  rlp_head(payload, 0xc0, 0xf7, hdr, hn);
  const uint32_t total = payload + hn;
  const bool raw = total < 32 && !force;
  const uint32_t nblk = raw ? 1u : (total + 1 + 135) / 136;
  const uint32_t pk = hn + key.pren, pc = pk + key.blen;  // key body, child item
  uint64_t *m64 = reinterpret_cast<uint64_t *>(msg);
  uint64_t a = 0;
  for (uint32_t b0 = 0; b0 < nblk; b0 += kWarpMsgBytes / 136) {
    const uint32_t wb = min((uint32_t)(kWarpMsgBytes / 136), nblk - b0);
    const uint32_t lo = b0 * 136, hi = lo + wb * 136;
    window_clear(m64, wb, lane);
    if (lane == 31) put_prefix(msg, lo, hi, hdr, hn, 0);
    if (lane == 30) put_prefix(msg, lo, hi, key.pre, key.pren, hn);
    if (lane == 29) put_prefix(msg, lo, hi, it.pre, it.pren, pc);
    for (uint32_t j = lane; j < key.blen; j += 32)
      if (pk + j >= lo && pk + j < hi) msg[pk + j - lo] = (uint8_t)((key.body[2 * j] << 4) | key.body[2 * j + 1]);
    if (it.far) {
      put_far<kCoh>(msg, lo, hi, it.far, it.blen, pc + it.pren, lane);
    } else {
      const uint32_t q = pc + it.pren + lane;
      const uint64_t w = lane < 16 ? (lane < 8 ? it.body.w[0] : it.body.w[1])
                                   : (lane < 24 ? it.body.w[2] : it.body.w[3]);
      if ((uint32_t)lane < it.blen && q >= lo && q < hi) msg[q - lo] = (uint8_t)(w >> (8 * (lane & 7)));
    }
    if (lane == 28 && !raw) put_padding(msg, lo, wb, total, nblk);
    __syncwarp();
    if (raw) break;  // under 32 bytes: the window holds the whole encoding
    a = window_absorb(a, m64, wb, cl, lane);
  }
  store_hash(tv, reinterpret_cast<uint64_t *>(tv.short_hash + (size_t)idx * 32), tv.short_hlen + idx, raw, a, m64,
             total, nblk, lane);
}

// This lane's child slot word of branch f (lane < 17).
__device__ __forceinline__ uint32_t child_word(const TrieView &tv, uint32_t f, int lane) {
  return lane < 17 ? __ldcg(tv.full_child + (size_t)f * 17 + lane) : 0u;
}

// Warp-cooperative encode + hash of branch node idx and of the extension
// above it, for levels with few nodes or for branches of many blocks, where
// one thread's serial chain is the latency.  Lane k < 17 loads the item of
// child k (slot word r); a scan gives every item its place, and the message
// is built window by window (kWarpMsgBytes, 8 blocks) in the warp's shared
// buffer -- every lane its own item's bytes at once, long values by all
// lanes -- and absorbed with the warp-spread permutation.  All 32 lanes call
// it with the same idx.  Returns the nibble depth where the hashed nodes
// start (0: a root).  up: the branch above (or kNoNode); *r_up gets this
// lane's slot word of it.
// Bound by latency: the serial permutations (2.2 us each, 4 for 16 children),
// before them three dependent loads (node, children, the extension's key),
// each step's loads issued together and none behind a branch.  Building item
// after item (one L2 round trip each) took a 16-child branch 15-17 us per
// level of a 1M-key trie; this form takes 10-11.
template <bool kCoh>
__device__ __forceinline__ uint32_t hash_full_warp(const TrieView &tv, uint32_t idx, uint32_t r, uint8_t *msg,
                                                   const CoopLanes &cl, uint32_t up, uint32_t *r_up) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const uint32_t kind = ref_kind(r);
  const bool node = kind == KIND_FULL || kind == KIND_SHORT, full = kind == KIND_FULL;
  // 1. the node's own words (node 0 stands in where there is none to load)
  const bool dead = ldn<kCoh>(tv.full_dead + idx) != 0;
  const uint32_t depth = ldn<kCoh>(tv.full_depth + idx);
  const uint32_t ext = __ldcg(tv.full_ext + idx);
  // 2. its children's hashes, the extension, the parent's slots
  const size_t ci = node ? ref_idx(r) : 0;
  const ulonglong2 *hp = reinterpret_cast<const ulonglong2 *>((full ? tv.full_hash : tv.short_hash) + ci * 32);
  const ulonglong2 h0 = __ldcg(hp), h1 = __ldcg(hp + 1);
  const uint32_t hl = __ldcg((full ? tv.full_hlen : tv.short_hlen) + ci);
  const uint32_t ei = ext != kNoNode ? ext : 0u;
  const uint64_t eko = __ldcg(tv.short_key + ei);
  const uint32_t eklen = __ldcg(tv.short_klen + ei), echild = __ldcg(tv.short_child + ei);
  const uint32_t edepth = __ldcg(tv.short_depth + ei);
  const bool edead = __ldcg(tv.short_dead + ei) != 0;
  if (r_up) *r_up = up != kNoNode ? child_word(tv, up, lane) : 0u;
  if (dead) return depth;  // unlinked by a delete: nothing to hash
  // 3. the extension's key (full_ext checked as ext_above does): an
  // extension's key has no terminator; up to 32 packed bytes, one per lane
  const bool has_ext = ext != kNoNode && !edead && echild == make_ref(KIND_FULL, idx);
  const uint32_t eodd = eklen & 1u, ebytes = eklen / 2;
  const bool ext_fits = has_ext && ebytes <= 32;
  const uint8_t *ek = tv.keys + (ext_fits ? eko : 0);
  const bool ebyte_on = ext_fits && (uint32_t)lane < ebytes;
  const uint32_t ek0 = __ldg(ek);
  const uint32_t ehi = __ldg(ek + (ebyte_on ? eodd + 2 * lane : 0)), elo = __ldg(ek + (ebyte_on ? eodd + 2 * lane + 1 : 0));
  WarpItem it;
  if (node) {
    it.blen = hl;
    it.body = Bytes32{{h0.x, h0.y, h1.x, h1.y}};
    node_head(tv, it);
  } else if (lane < 17) {
    it = warp_child_item<kCoh>(tv, r);  // an empty slot or a value
  }
  const bool force = tv.geth_mode && depth == 0;
  const uint32_t sz = it.pren + it.blen;
  uint32_t incl = sz;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t v = __shfl_up_sync(kAll, incl, o);
    if (lane >= o) incl += v;
  }
  const uint32_t payload = __shfl_sync(kAll, incl, 31);
  uint64_t hdr;
  uint32_t hn;
  rlp_head(payload, 0xc0, 0xf7, hdr, hn);
  const uint32_t total = payload + hn;
  const bool raw = total < 32 && !force;
  const uint32_t nblk = raw ? 1u : (total + 1 + 135) / 136;
  const uint32_t my_off = hn + incl - sz;  // message offset of this lane's item
  const unsigned far = __ballot_sync(kAll, it.far != nullptr);
  uint64_t *m64 = reinterpret_cast<uint64_t *>(msg);
  uint64_t a = 0, hw = 0;  // this lane's word of the state; of the branch's hash
  bool in_ext = false;     // one absorb site for both messages (instruction fetch)
  for (uint32_t b0 = 0;;) {
    const uint32_t wb = in_ext ? 1u : min((uint32_t)(kWarpMsgBytes / 136), nblk - b0);
    window_clear(m64, wb, lane);
    if (!in_ext) {
      const uint32_t lo = b0 * 136, hi = lo + wb * 136;
      if (lane == 31) put_prefix(msg, lo, hi, hdr, hn, 0);
      if (lane == 30 && !raw) put_padding(msg, lo, wb, total, nblk);
      put_prefix(msg, lo, hi, it.pre, it.pren, my_off);
      if (!it.far) put_body32(msg, lo, hi, it.body, it.blen, my_off + it.pren);
      for (unsigned m = far; m; m &= m - 1) {
        const int k = __ffs(m) - 1;
        const uint8_t *src = reinterpret_cast<const uint8_t *>(
            __shfl_sync(kAll, reinterpret_cast<unsigned long long>(it.far), k));
        const uint32_t n = __shfl_sync(kAll, it.blen, k), p = __shfl_sync(kAll, my_off + it.pren, k);
        put_far<kCoh>(msg, lo, hi, src, n, p, lane);
      }
    } else {
      // [list header][key header + flag][key bytes][0xa0][hash]: 35 to 70
      // bytes; the compact key is itself when one byte, else a string
      const uint32_t kpren = ebytes == 0 ? 1u : 2u, ep = kpren + ebytes + 33;
      const uint32_t en = ep < 56 ? 1u : 2u, kp = en + kpren, bp = kp + ebytes;
      const uint32_t flag = eodd ? 0x10u | ek0 : 0u;
      if (lane == 31) {
        msg[0] = (uint8_t)(ep < 56 ? 0xc0 + ep : 0xf8);
        if (en == 2) msg[1] = (uint8_t)ep;
      }
      if (lane == 30) {
        if (ebytes) msg[en] = (uint8_t)(0x80 + ebytes + 1);
        msg[kp - 1] = (uint8_t)flag;
      }
      if (lane == 29) put_padding(msg, 0, 1, en + ep, 1);
      if (lane == 28) msg[bp] = 0xa0;
      if (ebyte_on) msg[kp + lane] = (uint8_t)((ehi << 4) | elo);
      if (lane < 4) {
#pragma unroll
        for (int j = 0; j < 8; ++j) msg[bp + 1 + 8 * lane + j] = (uint8_t)(hw >> (8 * j));
      }
    }
    __syncwarp();
    if (in_ext || !raw) a = window_absorb(a, m64, wb, cl, lane);
    if (in_ext) {
      const uint32_t ep = (ebytes == 0 ? 1u : 2u) + ebytes + 33;
      store_hash(tv, reinterpret_cast<uint64_t *>(tv.short_hash + (size_t)ext * 32), tv.short_hlen + ext, false, a, m64,
                 (ep < 56 ? 1u : 2u) + ep, 1, lane);
      return edepth;
    }
    b0 += wb;
    if (b0 < nblk) continue;
    hw = store_hash(tv, reinterpret_cast<uint64_t *>(tv.full_hash + (size_t)idx * 32), tv.full_hlen + idx, raw, a, m64,
                    total, nblk, lane);
    if (!has_ext) return depth;
    if (!ext_fits || raw) {
      hash_short_warp<kCoh>(tv, ext, msg, cl, true, hw, raw ? total : 32u);
      return edepth;
    }
    in_ext = true;
    a = 0;
  }
}

// A warp per node (4 per CTA): a level's branches when it has few, or its
// branches of many blocks, each with the extension above it; or a few leaves.
__global__ void __launch_bounds__(128) k_hash_warp(TrieView tv, const uint32_t *refs, int count) {
  extern __shared__ uint64_t msg_all[];  // one message window per warp
  const int j = blockIdx.x * 4 + (threadIdx.x >> 5);
  if (j >= count) return;  // whole warps leave together
  uint8_t *msg = reinterpret_cast<uint8_t *>(msg_all) + (threadIdx.x >> 5) * kWarpMsgBytes;
  const CoopLanes cl = coop_lanes(threadIdx.x & 31);
  const uint32_t r = refs[j];
  if (ref_kind(r) == KIND_FULL)
    hash_full_warp<false>(tv, ref_idx(r), child_word(tv, ref_idx(r), threadIdx.x & 31), msg, cl, kNoNode, nullptr);
  else
    hash_short_warp<false>(tv, ref_idx(r), msg, cl, false, 0, 0);
}

// Thread per node of one launch's list, which the bins order by Keccak block
// count, so the lanes of a warp permute together.  (Ordering each CTA's nodes
// again before encoding cost a barrier behind four dependent gathers: leaf
// launch of a 1M-key load 0.76 of the integer pipe.)
constexpr int kHashLevelThreads = 128;

#ifndef GMPT_HASH_CTAS
#define GMPT_HASH_CTAS 6
#endif
template <bool kFull>
__device__ __forceinline__ void hash_level_thread(const TrieView &tv, const uint32_t *refs, int count) {
  extern __shared__ uint32_t stage_all[];
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < count) hash_node<false, kFull>(tv, ref_idx(refs[t]), stage_all + threadIdx.x, blockDim.x);
}

// Six 128-thread CTAs per SM (at most 85 registers): the permutation keeps
// its 25 lanes in registers; a few encoder temporaries spill, and the extra
// resident warps hide more of the child / record gathers (measured faster
// than five CTAs at 96 registers without spills).
// The level kernel at the register budget of six resident CTAs per SM (the
// throughput form), and with the whole register file open to one CTA per
// SM: a level too small to fill the SMs is as long as the serial Keccak
// chain of its longest node, which the wider form schedules with more
// permutation state in flight.
template <bool kFull>
__global__ void __launch_bounds__(kHashLevelThreads, GMPT_HASH_CTAS) k_hash_level(TrieView tv, const uint32_t *refs,
                                                                                 int count) {
  hash_level_thread<kFull>(tv, refs, count);
}

template <bool kFull>
__global__ void __launch_bounds__(kHashLevelThreads, 1) k_hash_level_wide(TrieView tv, const uint32_t *refs, int count) {
  hash_level_thread<kFull>(tv, refs, count);
}

// ---------------------------------------------------------------------------
// gets (gpu_mpt_kernels.cuh:2267-2340)

// Record id of key kb[0..len), or -1.  A chain of dependent loads (a slot per
// level, then the leaf's fields, its key and its record); a leaf's fields are
// loaded together and its key compared 32 nibbles at a time.
__device__ __forceinline__ int64_t lookup(const TrieView &tv, uint32_t root, const uint8_t *kb, uint32_t len) {
  uint32_t ref = root;
  uint32_t x = 0;
  for (uint32_t guard = 0; guard <= len + 1; ++guard) {
    uint32_t kind = ref_kind(ref), idx = ref_idx(ref);
    if (kind == KIND_NULL) return -1;
    if (kind == KIND_VALUE) return x == len ? (int64_t)tv.value_vid[idx] : -1;
    if (kind == KIND_FULL) {
      if (x >= len) return -1;
      uint32_t c = kb[x];
      if (c > 16) return -1;
      ref = tv.full_child[(size_t)idx * 17 + c];
      ++x;
      continue;
    }
    const uint32_t sl = tv.short_klen[idx], child = tv.short_child[idx];
    const uint8_t *sk = tv.keys + tv.short_key[idx];
    if (len - x < sl) return -1;
    if (!equal_nibbles(sk, kb + x, sl)) return -1;
    x += sl;
    ref = child;
  }
  return -1;
}

__global__ void k_gets(TrieView tv, const uint8_t *keys, const int *idx, int n, int64_t keys_bytes,
                       uint64_t *out_hp, int *out_len, int64_t *out_vid, const int *tid) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int ks = idx[2 * i], ke = idx[2 * i + 1];
  int len = ke - ks + 1;
  const uint32_t tr = tid ? (uint32_t)tid[i] : 0u;
  bool ok = ks >= 0 && len > 0 && (int64_t)ke < keys_bytes && tr < tv.n_tries;
  int64_t vid = ok ? lookup(tv, tv.roots[tr], keys + ks, (uint32_t)len) : -1;
  if (out_vid) out_vid[i] = vid;
  if (vid < 0) {
    out_hp[i] = 0;
    out_len[i] = 0;
  } else {
    out_hp[i] = tv.rec_hp[vid];
    out_len[i] = (int)tv.rec[vid].len;
  }
}

// Root bytes of trie ids[i] (or trie first + i when ids is null) into out[33 i ..]:
// 32 bytes (zero-padded) and the length (0 = empty trie).  Warp per trie.
__global__ void k_roots(TrieView tv, const int *ids, int first, int n, uint8_t *out) {
  const int i = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5);
  if (i >= n) return;
  const int t = threadIdx.x & 31;
  const uint32_t tr = ids ? (uint32_t)ids[i] : (uint32_t)(first + i);
  out += 33 * (size_t)i;
  uint32_t r = tr < tv.n_tries ? tv.roots[tr] : 0u;
  uint32_t kind = ref_kind(r), idx = ref_idx(r);
  uint32_t len = 0;
  const uint8_t *h = nullptr;
  if (kind == KIND_FULL) {
    h = tv.full_hash + (size_t)idx * 32;
    len = tv.full_hlen[idx];
  } else if (kind == KIND_SHORT) {
    h = tv.short_hash + (size_t)idx * 32;
    len = tv.short_hlen[idx];
  } else if (kind == KIND_VALUE) {
    unsigned long long vid = tv.value_vid[idx];
    const ValueRec rc = tv.rec[vid];
    h = tv.vals + rc.off;
    len = min(32u, rc.len);
  }
  out[t] = (h && (uint32_t)t < len) ? h[t] : 0;
  if (t == 0) out[32] = (uint8_t)len;
}

}  // namespace gmpt
