// block_update.cuh -- one persistent launch that updates many tries of a
// forest and hashes them: the Ethereum block shape, where every touched
// account's storage trie is updated and hashed first, its new root is
// written into the account's value, and then the state trie is updated and
// hashed.
//
// The reference runs one MPT object per trie and one puts_latching + one
// hash_onepass (several kernel launches, host synchronisation between them)
// per trie (gpu_mpt.cuh:554-615, 1162-1191).  Here a block is:
//   k_block_stage  copy + validate the key/value streams into the arenas and
//                  build the value records (an ordinary launch, so the arena
//                  bytes are read-only for the next one)
//   k_block        cooperative persistent kernel, for stage 0 then stage 1:
//                    [stage 1 only] patch: value bytes of key i at
//                      patch_off[i] := root of trie patch_trie[i]
//                    LockNU insert of the stage's keys into their tries
//                    hash what they made dirty (hash_grid: leaves, then
//                    every branch once its children are done)
//                  with a grid barrier between phases, then the roots asked
//                  for are written out.
// Both launches plus the descriptor / counter copies are captured once as a
// CUDA graph and replayed per block; sizes come from the device-side
// descriptor, so the graph is rebuilt only when a buffer or pool moves.
#pragma once
#include "grid_hash.cuh"
#include "latch_kernels.cuh"
#include "trie_kernels.cuh"

namespace gmpt {

struct BlockDesc {
  // set by the host for every launch; copying it in also zeroes the fields
  // below that the kernels fill
  int32_t n, n0, n_out, pad0;      // keys; stage 0 = [0, n0), stage 1 = [n0, n)
  int64_t kbytes, vbytes;          // stream lengths
  uint64_t key_base, val_base, vid_base;
  uint32_t gen, pad1;              // dirty generation of stage 0 (stage 1: gen + 1)
  uint32_t warp_max;               // hash_grid's warp_max
  uint32_t max_klen;               // filled by k_block_stage: the longest key
  // the block where it lies (the caller's device arrays, or copies of host
  // arrays); the streams are 8-byte aligned
  const uint8_t *keys;             // key stream (nibble bytes)
  const uint8_t *vals;             // value stream
  const int *kidx;                 // [2n] inclusive pairs; must tile the stream
  const int64_t *vidx;             // [2n]
  const int *tid;                  // [n] trie of each key (null: trie 0)
  const int *patch_trie;           // [n] -1 = no patch (null: none)
  const int *patch_off;            // [n] byte offset of the 32-byte root in the value
  const int *out_ids;              // [n_out] tries whose roots are reported (pinned host memory)
  uint8_t *out;                    // [n_out * 33] root bytes + length (pinned host memory)
  GridCtl ctl;                     // barrier_ns set, the rest zero
  // filled by k_block_stage
  uint32_t stream_terms, key_terms, noncontig, bad;  // bad: BLOCK_BAD_* bits
  // filled by k_block
  uint32_t levels[2], dirty[2];    // hash waves and dirty nodes of each stage
};

enum : uint32_t { BLOCK_BAD_KEY = 1, BLOCK_BAD_TRIE = 2, BLOCK_BAD_PATCH = 4, BLOCK_BAD_VALUE = 8 };

struct BlockBufs {
  uint64_t *koff;          // [n] staged key offsets
  uint32_t *klen;          // [n]
  uint32_t *ready;         // branches whose dirty children are hashed
  BlockDesc *desc;
};

// Word w of a stream of n bytes, zero past its end.  A last partial word is
// taken byte by byte: the stream may be the caller's array, of which no byte
// past the end is read.
__device__ __forceinline__ uint64_t stream_word(const uint8_t *src, int64_t n, int64_t w) {
  if (8 * w + 8 <= n) return reinterpret_cast<const uint64_t *>(src)[w];
  uint64_t x = 0;
  for (int64_t b = 8 * w; b < n; ++b) x |= (uint64_t)src[b] << (8 * (b - 8 * w));
  return x;
}

// Copy the streams into the arenas (8-byte words; 64 zero bytes follow each
// stream), validate keys and pairs, and build the value records.  Grid-stride;
// every thread runs to the end.
__global__ void __launch_bounds__(kGridThreads) k_block_stage(TrieView tv, BlockBufs bb) {
  BlockDesc *D = bb.desc;
  const int n = D->n, n0 = D->n0;
  const int64_t kb = D->kbytes, vb = D->vbytes;
  const uint64_t key_base = D->key_base, val_base = D->val_base, vid_base = D->vid_base;
  const int64_t T = (int64_t)gridDim.x * blockDim.x, t0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int *kidx = D->kidx, *tid = D->tid, *patch_trie = D->patch_trie, *patch_off = D->patch_off;
  const int64_t *vidx = D->vidx;
  const uint8_t *keys = D->keys;
  if (t0 == 0) D->ctl.ts[D->ctl.n_ts++] = global_ns();
  uint32_t terms = 0, bad = 0, kterms = 0, gap = 0, lmax = 0;
  {
    uint64_t *dst = reinterpret_cast<uint64_t *>(const_cast<uint8_t *>(tv.keys) + key_base);
    const int64_t words = (kb + 7) / 8 + 8;
    for (int64_t w = t0; w < words; w += T) {
      const uint64_t x = stream_word(keys, kb, w);
      if (x & 0xE0E0E0E0E0E0E0E0ull) bad |= BLOCK_BAD_KEY;  // >= 32
      const uint64_t hi = x & 0x1010101010101010ull;        // 16..31
      if (x & ((hi >> 4) * 0x0Full)) bad |= BLOCK_BAD_KEY;  // 17..31
      terms += __popcll(hi);
      dst[w] = x;
    }
  }
  {
    uint64_t *dst = reinterpret_cast<uint64_t *>(const_cast<uint8_t *>(tv.vals) + val_base);
    const uint8_t *vals = D->vals;
    const int64_t words = (vb + 7) / 8 + 8;
    for (int64_t w = t0; w < words; w += T) dst[w] = stream_word(vals, vb, w);
  }
  for (int64_t i = t0; i < n; i += T) {
    int ks = kidx[2 * i], ke = kidx[2 * i + 1];
    bool badk = ks < 0 || ke < ks || (int64_t)ke >= kb || ke - ks + 1 > kMaxKeyNibbles;
    if (!badk) {
      const uint8_t last = keys[ke];
      if (last > 16) badk = true;
      kterms += last == 16 ? 1u : 0u;
    }
    if (i == 0 ? ks != 0 : ks != kidx[2 * i - 1] + 1) gap = 1;
    if (i + 1 == n && (int64_t)ke + 1 != kb) gap = 1;
    if (badk) {
      bad |= BLOCK_BAD_KEY;
      ks = ke = 0;
    }
    bb.koff[i] = key_base + (uint64_t)ks;
    bb.klen[i] = (uint32_t)(ke - ks + 1);
    lmax = max(lmax, (uint32_t)(ke - ks + 1));
    if (tid && (uint32_t)tid[i] >= tv.n_tries) bad |= BLOCK_BAD_TRIE;
    int64_t vs = vidx[2 * i], ve = vidx[2 * i + 1];
    if (vs < 0 || ve < vs - 1 || ve >= vb) {
      bad |= BLOCK_BAD_VALUE;
      vs = 0;
      ve = -1;
    }
    const int pt = patch_trie ? patch_trie[i] : -1;
    if (pt >= 0 && ((uint32_t)pt >= tv.n_tries || i < n0 || patch_off[i] < 0 ||
                    (int64_t)patch_off[i] + 32 > ve - vs + 1))
      bad |= BLOCK_BAD_PATCH;
    const uint64_t vid = vid_base + (uint64_t)i;
    tv.rec[vid] = ValueRec{val_base + (uint64_t)vs, (uint32_t)(ve - vs + 1), 0u};
    tv.rec_hp[vid] = 0;
  }
  terms = __reduce_add_sync(0xffffffffu, terms);
  kterms = __reduce_add_sync(0xffffffffu, kterms);
  bad = __reduce_or_sync(0xffffffffu, bad);
  gap = __reduce_or_sync(0xffffffffu, gap);
  lmax = __reduce_max_sync(0xffffffffu, lmax);
  if ((threadIdx.x & 31) == 0) {
    if (terms) atomicAdd(&D->stream_terms, terms);
    if (kterms) atomicAdd(&D->key_terms, kterms);
    if (bad) atomicOr(&D->bad, bad);
    if (gap) atomicOr(&D->noncontig, 1u);
    if (lmax) atomicMax(&D->max_klen, lmax);
  }
}

// 33 bytes for the root of trie tr (warp-wide: lane b writes byte b)
__device__ __forceinline__ void write_root(const TrieView &tv, uint32_t tr, uint8_t *out, int lane) {
  const uint32_t r = tr < tv.n_tries ? __ldcg(tv.roots + tr) : 0u;
  const uint32_t kind = ref_kind(r), idx = ref_idx(r);
  const uint8_t *h = nullptr;
  uint32_t len = 0;
  if (kind == KIND_FULL) {
    h = tv.full_hash + (size_t)idx * 32;
    len = __ldcg(tv.full_hlen + idx);
  } else if (kind == KIND_SHORT) {
    h = tv.short_hash + (size_t)idx * 32;
    len = __ldcg(tv.short_hlen + idx);
  }
  out[lane] = (h && (uint32_t)lane < len) ? __ldcg(h + lane) : 0;
  if (lane == 0) out[32] = (uint8_t)len;
}

__global__ void __launch_bounds__(kGridThreads, 1) k_block(TrieView tv0, DirtyList dl, BlockBufs bb, uint32_t retry_limit) {
  extern __shared__ __align__(16) uint32_t smem[];  // kStageWords message words per thread, a window per warp
  BlockDesc *D = bb.desc;
  const int n = D->n, n0 = D->n0, n_out = D->n_out;
  const uint64_t vid_base = D->vid_base;
  const int t = blockIdx.x * blockDim.x + threadIdx.x, T = gridDim.x * blockDim.x;
  TrieView tv = tv0;
  if (t == 0) D->ctl.ts[D->ctl.n_ts++] = global_ns();
  const GridPlace g;
  // this warp's message buffer for hash_full_warp, after the staging words
  uint8_t *wmsg = reinterpret_cast<uint8_t *>(smem + kStageWords * blockDim.x) + (threadIdx.x >> 5) * kWarpMsgBytes;
  // staging outcome: every CTA reads the same words, so all leave together
  if (D->bad || D->noncontig || D->stream_terms != D->key_terms) {
    if (t == 0) atomicOr(&D->ctl.status, 2u);
    return;
  }
  for (int s = 0; s < 2; ++s) {
    const int i0 = s ? n0 : 0, i1 = s ? n : n0;
    tv.gen = D->gen + (uint32_t)s;
    if (s == 1) {
      // stage-1 values take the roots their stage-0 tries just got
      for (int i = n0 + t; i < n && D->patch_trie; i += T) {
        const int pt = D->patch_trie[i];
        if (pt < 0) continue;
        uint8_t *dst = const_cast<uint8_t *>(tv.vals) + tv.rec[vid_base + (uint64_t)i].off + D->patch_off[i];
        const uint32_t r = __ldcg(tv.roots + pt);
        const uint32_t kind = ref_kind(r), idx = ref_idx(r);
        const uint8_t *h = kind == KIND_FULL ? tv.full_hash + (size_t)idx * 32
                                             : (kind == KIND_SHORT ? tv.short_hash + (size_t)idx * 32 : nullptr);
        const uint32_t hl =
            kind == KIND_FULL ? __ldcg(tv.full_hlen + idx) : (kind == KIND_SHORT ? __ldcg(tv.short_hlen + idx) : 0u);
        for (uint32_t b = 0; b < 32; ++b) dst[b] = (h && b < hl) ? __ldcg(h + b) : 0;
      }
    }
    // insert (LockNU; the patched bytes are only read after the next barrier)
    const int span = T * kLatchWays;
    for (int base = i0; base < i1; base += span)
      latch_keys(tv, dl, bb.koff + base, bb.klen + base, min(span, i1 - base), vid_base + (uint64_t)base, retry_limit,
                 D->tid ? D->tid + base : nullptr, g.t_spread, T);
    if (!grid_barrier(&D->ctl, tv.ctr)) return;
    const uint32_t nd = __ldcg(&tv.ctr->n_dirty);
    uint32_t waves = 0;
    if (!hash_grid(tv, dl, nd, bb.ready, tv.cap_full, &D->ctl, D->warp_max, smem + threadIdx.x, wmsg, &waves)) return;
    if (t == 0) {
      D->levels[s] = waves;
      D->dirty[s] = nd;
    }
    if (!grid_barrier(&D->ctl, tv.ctr)) return;  // the cleared counters are seen by every CTA
  }
  // roots asked for: one warp each
  for (int w = t >> 5; w < n_out; w += T >> 5) write_root(tv, (uint32_t)D->out_ids[w], D->out + 33 * (size_t)w, g.lane);
  __syncthreads();
  if (t == 0 && D->ctl.n_ts < kGridMaxTs) D->ctl.ts[D->ctl.n_ts++] = global_ns();
}

}  // namespace gmpt
