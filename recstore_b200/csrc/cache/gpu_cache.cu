// Set-associative LRU embedding cache in HBM with the Query / Replace / Update / Dump contract of the
// cache the reference vendors from HugeCTR (src/storage/gpu_cache/nv_gpu_cache.cu:392-531 get_kernel,
// 700-852 insert_replace_kernel, 970-1074 update_kernel, 1155-1226 dump_kernel; API
// gpu_cache_api.hpp:27-50; torch wrapper src/framework/pytorch/recstore_gpu_cache.h:31-106).
//
// Layout: `nsets` sets of 32 slots; a warp probes a set with one 256-byte coalesced load (one key per
// lane) and a ballot.  Differences from the reference kernel shape (1 key per warp, 2 keys per
// 64-thread block, a per-set mutex even on reads):
//   * each warp walks a strided list of keys and keeps the next key's set line in flight while it
//     copies the current row, so many keys are in flight per SM;
//   * the hit path takes no lock: it reads keys / values and stamps the slot's counter with a relaxed store (a
//     stale stamp only makes LRU slightly approximate).  Every slot carries a sequence number that a writer makes
//     odd before it touches the slot's key or values and even again afterwards; Query reads it before and after
//     the row copy and reports the key as a MISS when it was odd or changed, so a Query that overlaps a Replace /
//     Update of the same slot on another stream never returns a torn or wrong-key row as a hit;
//   * Replace / Update take a per-set lock with a BOUNDED spin; on give-up the key is skipped and
//     RS_DEV_WAIT_TIMEOUT is recorded.
// Semantics kept: Query writes hit rows in place, leaves miss rows untouched, appends (position,
// key) of every miss in arbitrary order with a device-side count, bumps the global clock; Replace
// inserts into an empty slot or evicts the smallest stamp and refreshes the stamp when the key is
// already cached; Update overwrites values of cached keys only; Dump enumerates the keys of a set range.
#include "common/rs_common.h"
#include "kv/hash_table.cuh"

namespace {
using rs::ht_hash;

constexpr unsigned long long kEmptyKey = 0xFFFFFFFFFFFFFFFFull;
constexpr int kWays = 32;

struct CacheView {
  unsigned long long* keys;   // [nsets * 32]
  unsigned* stamps;           // [nsets * 32]
  unsigned* vers;             // [nsets * 32] slot sequence numbers (odd while a writer is inside)
  unsigned char* dirty;       // [nsets * 32] 1 = the row was changed in the cache and the backing store is behind
  float* values;              // [nsets * 32, dim]
  int* locks;                 // [nsets]
  unsigned* clock;            // global LRU clock
  unsigned long long nsets;
  int dim;
};

__device__ __forceinline__ void copy_row(float* __restrict__ dst, const float* __restrict__ src, int dim, int lane) {
  for (int v = lane; v < (dim >> 2); v += 32) reinterpret_cast<float4*>(dst)[v] = reinterpret_cast<const float4*>(src)[v];
}

__global__ void cache_init_kernel(CacheView c) {
  const unsigned long long i = static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < c.nsets * kWays) {
    c.keys[i] = kEmptyKey;
    c.stamps[i] = 0;
    c.vers[i] = 0;
    c.dirty[i] = 0;
  }
  if (i < c.nsets) c.locks[i] = 0;
  if (i == 0) *c.clock = 0;
}

__global__ void cache_tick_kernel(unsigned* clock, int* miss_count) {
  atomicAdd(clock, 1u);
  if (miss_count) *miss_count = 0;
}

// Eight lanes per key: each compares four of the 32 tags of the key's set (one 32-byte load), so a warp probes four keys per
// step and keeps four steps (16 keys) in flight; the set of a key, a 64-bit remainder, is worked out by one lane and not by
// all that probe it.  Hits are validated like a seqlock reader (version, key, row, version again), in three phases over the
// 16 keys, so that the warp pays three dependent round trips and two fences per 16 keys.  Misses are gathered over the warp
// and appended with one atomicAdd: a counter bumped once per missing key serialises the whole grid on one L2 address when the
// hit rate is low.  Bound by latency; a warp per key, four keys in flight, took 45 us for 65,536 keys x 32 floats
// at 47 % hits, this form 19 us.
constexpr int kProbeLanes = 8;
constexpr int kProbeSteps = 4;
constexpr int kProbeKeys = 32 / kProbeLanes * kProbeSteps;    // keys per warp and pass

__device__ __forceinline__ void load_tags(unsigned long long (&t)[4], const unsigned long long* p) {
  asm volatile("ld.global.cg.v4.u64 {%0,%1,%2,%3}, [%4];" : "=l"(t[0]), "=l"(t[1]), "=l"(t[2]), "=l"(t[3]) : "l"(p) : "memory");
}
// Index of `key` among the four tags of this lane, or -1.
__device__ __forceinline__ int match_tags(const unsigned long long (&t)[4], unsigned long long key) {
  return t[0] == key ? 0 : t[1] == key ? 1 : t[2] == key ? 2 : t[3] == key ? 3 : -1;
}

__global__ void __launch_bounds__(256) cache_query_kernel(CacheView c, const long long* __restrict__ keys, long long n,
                                                          float* __restrict__ out, long long* __restrict__ miss_index,
                                                          long long* __restrict__ miss_keys, int* __restrict__ miss_count) {
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, l = lane & (kProbeLanes - 1), sub = lane / kProbeLanes;
  const long long nwarps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const unsigned now = *c.clock;
  for (long long i0 = (static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kProbeKeys; i0 < n;
       i0 += nwarps * kProbeKeys) {
    unsigned long long my_key = kEmptyKey, my_set = 0;
    if (lane < kProbeKeys && i0 + lane < n) {
      my_key = static_cast<unsigned long long>(keys[i0 + lane]);
      my_set = ht_hash(my_key) % c.nsets;
    }
    unsigned long long key[kProbeSteps], slot[kProbeSteps], tags[kProbeSteps][4];
#pragma unroll
    for (int u = 0; u < kProbeSteps; ++u) {
      const int j = u * (32 / kProbeLanes) + sub;
      key[u] = __shfl_sync(kAll, my_key, j);
      slot[u] = __shfl_sync(kAll, my_set, j) * kWays;        // first slot of the set, for now
      if (key[u] != kEmptyKey) load_tags(tags[u], c.keys + slot[u] + l * 4);
    }
    unsigned v0[kProbeSteps];
    bool hit[kProbeSteps];
#pragma unroll
    for (int u = 0; u < kProbeSteps; ++u) {
      const int w = key[u] != kEmptyKey ? match_tags(tags[u], key[u]) : -1;
      const unsigned m = (__ballot_sync(kAll, w >= 0) >> (sub * kProbeLanes)) & ((1u << kProbeLanes) - 1u);
      hit[u] = m != 0;
      const int from = hit[u] ? __ffs(m) - 1 : 0;
      const int way = __shfl_sync(kAll, l * 4 + (w < 0 ? 0 : w), from, kProbeLanes);
      if (hit[u]) slot[u] += way;
      v0[u] = hit[u] ? *reinterpret_cast<volatile unsigned*>(&c.vers[slot[u]]) : 1u;
    }
    __threadfence();
    unsigned long long k0[kProbeSteps];
#pragma unroll
    for (int u = 0; u < kProbeSteps; ++u) {
      k0[u] = kEmptyKey;
      if (hit[u]) k0[u] = *reinterpret_cast<volatile unsigned long long*>(&c.keys[slot[u]]);
    }
    if (out != nullptr) {
      // rows through L2, never from a possibly stale L1 line: the version check only vouches for what L2 holds
      for (int v = l; v < (c.dim >> 2); v += kProbeLanes) {
        float4 x[kProbeSteps];
#pragma unroll
        for (int u = 0; u < kProbeSteps; ++u)
          if (hit[u]) x[u] = __ldcg(reinterpret_cast<const float4*>(c.values + slot[u] * c.dim) + v);
#pragma unroll
        for (int u = 0; u < kProbeSteps; ++u)
          if (hit[u]) reinterpret_cast<float4*>(out + (i0 + u * (32 / kProbeLanes) + sub) * c.dim)[v] = x[u];
      }
    }
    __threadfence();
    bool my_miss = false;
#pragma unroll
    for (int u = 0; u < kProbeSteps; ++u) {
      bool valid = false;
      if (hit[u]) {
        const unsigned v1 = *reinterpret_cast<volatile unsigned*>(&c.vers[slot[u]]);
        valid = (v0[u] & 1u) == 0u && v1 == v0[u] && k0[u] == key[u];
      }
      // every lane of the key must have seen the same even version (they read it on their own)
      const unsigned ok = (__ballot_sync(kAll, valid) >> (sub * kProbeLanes)) & ((1u << kProbeLanes) - 1u);
      valid = ok == (1u << kProbeLanes) - 1u;
      if (valid && l == 0 && c.stamps[slot[u]] != now) c.stamps[slot[u]] = now;
      const int from = (lane - u * (32 / kProbeLanes)) * kProbeLanes;          // key `lane` was probed by these lanes
      const bool theirs = __shfl_sync(kAll, static_cast<int>(valid), from & 31) != 0;
      if (lane / (32 / kProbeLanes) == u) my_miss = !theirs && my_key != kEmptyKey;   // (padding: neither a hit nor a miss)
    }
    const unsigned misses = __ballot_sync(kAll, my_miss);
    if (misses) {
      int base = 0;
      if (lane == 0) base = atomicAdd(miss_count, __popc(misses));
      base = __shfl_sync(kAll, base, 0);
      if (my_miss) {
        const int at = base + __popc(misses & ((1u << lane) - 1u));
        miss_index[at] = i0 + lane;
        miss_keys[at] = static_cast<long long>(my_key);
      }
    }
  }
}

__device__ __forceinline__ bool lock_set(int* lock, int lane) {
  int ok = 0;
  if (lane == 0) {
    for (int spin = 0; spin < (1 << 20); ++spin) {
      if (atomicCAS(lock, 0, 1) == 0) { ok = 1; break; }
      __nanosleep(32);
    }
    __threadfence();
  }
  return __shfl_sync(0xffffffffu, ok, 0) != 0;
}
__device__ __forceinline__ void unlock_set(int* lock, int lane) {
  __syncwarp();
  if (lane == 0) {
    __threadfence();
    atomicExch(lock, 0);
  }
}

// mode 0: Replace (insert or evict LRU, refresh stamp when present); mode 1: Update (present keys only).
// Eight lanes per key, four keys per warp.  A write is a chain of about eight dependent memory round trips (lock, tags, version,
// row, version, unlock and the fences between them), so what counts is how many keys are in such a chain at once: a warp per
// key and 32 warps per SM took 81 us for 65,536 present keys x 32 floats, this form 49 us.  Sets are locked by TRYING: a key whose set is
// taken stays pending while the other keys of the warp go on, and no lane ever waits while it holds a lock.  The number of
// tries is bounded; a key that never got its set is skipped and RS_DEV_WAIT_TIMEOUT recorded.
__global__ void __launch_bounds__(256, 8) cache_write_kernel(CacheView c, const long long* __restrict__ keys, long long n,
                                                          const float* __restrict__ values, int mode,
                                                          unsigned long long* status) {
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kPer = 32 / kProbeLanes;
  const int lane = threadIdx.x & 31, l = lane & (kProbeLanes - 1), sub = lane / kProbeLanes;
  const unsigned wm = ((1u << kProbeLanes) - 1u) << (sub * kProbeLanes);
  const long long nwarps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const unsigned now = *c.clock;
  for (long long i0 = (static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kPer; i0 < n; i0 += nwarps * kPer) {
    const long long i = i0 + sub;
    const unsigned long long key = i < n ? static_cast<unsigned long long>(keys[i]) : kEmptyKey;
    const unsigned long long set = ht_hash(key) % c.nsets;
    bool todo = key != kEmptyKey;
    float4 ahead = make_float4(0.f, 0.f, 0.f, 0.f);      // the row's first piece, on its way before the set is locked
    if (todo && l < (c.dim >> 2)) ahead = reinterpret_cast<const float4*>(values + i * c.dim)[l];
    for (int spin = 0; spin < (1 << 20) && __any_sync(kAll, todo); ++spin) {
      int got = 0;
      if (todo && l == 0) got = atomicCAS(&c.locks[set], 0, 1) == 0;
      got = __shfl_sync(kAll, got, 0, kProbeLanes);
      if (got) {
        todo = false;
        __threadfence();
        unsigned long long tags[4];
        load_tags(tags, c.keys + set * kWays + l * 4);
        const int w = match_tags(tags, key);
        const unsigned hits = __ballot_sync(wm, w >= 0) >> (sub * kProbeLanes);
        const bool hit = hits != 0;
        int way = -1;
        if (hit) {
          way = __shfl_sync(wm, l * 4 + (w < 0 ? 0 : w), __ffs(hits) - 1, kProbeLanes);
        } else if (mode == 0) {
          // the first empty way, or the least recently stamped one
          const int e = match_tags(tags, kEmptyKey);
          const unsigned empty = __ballot_sync(wm, e >= 0) >> (sub * kProbeLanes);
          if (empty) {
            way = __shfl_sync(wm, l * 4 + (e < 0 ? 0 : e), __ffs(empty) - 1, kProbeLanes);
          } else {
            unsigned long long best = ~0ull;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              const unsigned st = *reinterpret_cast<volatile unsigned*>(&c.stamps[set * kWays + l * 4 + q]);
              const unsigned long long mine = (static_cast<unsigned long long>(st) << 5) | static_cast<unsigned>(l * 4 + q);
              best = mine < best ? mine : best;
            }
#pragma unroll
            for (int o = kProbeLanes / 2; o > 0; o >>= 1) {
              const unsigned long long other = __shfl_xor_sync(wm, best, o);
              best = other < best ? other : best;
            }
            way = static_cast<int>(best & 31);
          }
        }
        if (way >= 0) {
          const unsigned long long slot = set * kWays + way;
          if (!hit || mode == 1) {            // (Replace of a cached key only refreshes its stamp)
            // sequence number odd -> key and values change -> even again (readers discard what they copied meanwhile)
            if (l == 0) {
              atomicAdd(&c.vers[slot], 1u);
              __threadfence();
            }
            __syncwarp(wm);
            for (int v = l; v < (c.dim >> 2); v += kProbeLanes)
              reinterpret_cast<float4*>(c.values + slot * c.dim)[v] = v == l ? ahead : reinterpret_cast<const float4*>(values + i * c.dim)[v];
            if (l == 0 && !hit) *reinterpret_cast<volatile unsigned long long*>(&c.keys[slot]) = key;
            __threadfence();
            __syncwarp(wm);
            if (l == 0) atomicAdd(&c.vers[slot], 1u);
          }
          if (l == 0 && mode == 0) c.stamps[slot] = now;
        }
        __syncwarp(wm);
        if (l == 0) {
          __threadfence();
          atomicExch(&c.locks[set], 0);
        }
      }
      __syncwarp();
      if (__any_sync(kAll, todo)) __nanosleep(32);
    }
    if (todo && l == 0 && status) atomicOr(status, (unsigned long long)RS_DEV_WAIT_TIMEOUT);
  }
}

// Replace that hands the evicted rows back (write-back caches) and never evicts a row stamped at or after
// `protect_from` (rows of the step in flight and of the batches already announced).  Dirty evicted rows go to
// evict_keys / evict_values (cursor evict_count); a key that finds its set full of protected rows is not inserted and is
// reported in refused_keys (cursor refused_count): the caller serves it from the backing store.
__global__ void __launch_bounds__(256) cache_replace_evict_kernel(CacheView c, const long long* __restrict__ keys, const int* n_dev,
                                                                  long long n_cap, const float* __restrict__ values, unsigned protect_from,
                                                                  long long* __restrict__ evict_keys, float* __restrict__ evict_values,
                                                                  int* evict_count, long long* __restrict__ refused_keys,
                                                                  int* refused_count, unsigned long long* status) {
  const int lane = threadIdx.x & 31;
  const long long warp = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long nwarps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const unsigned now = *c.clock;
  const long long n = n_dev ? min(static_cast<long long>(*n_dev), n_cap) : n_cap;
  for (long long i = warp; i < n; i += nwarps) {
    const unsigned long long key = static_cast<unsigned long long>(keys[i]);
    if (key == kEmptyKey) continue;
    const unsigned long long set = ht_hash(key) % c.nsets;
    if (!lock_set(&c.locks[set], lane)) {
      if (lane == 0 && status) atomicOr(status, (unsigned long long)RS_DEV_WAIT_TIMEOUT);
      if (lane == 0 && refused_keys) refused_keys[atomicAdd(refused_count, 1)] = static_cast<long long>(key);
      continue;
    }
    const unsigned long long line = *reinterpret_cast<volatile unsigned long long*>(&c.keys[set * kWays + lane]);
    const unsigned hit = __ballot_sync(0xffffffffu, line == key);
    if (hit) {                                   // already cached (brought in by a step in between): only refresh the stamp
      if (lane == 0) c.stamps[set * kWays + (__ffs(hit) - 1)] = now;
      unlock_set(&c.locks[set], lane);
      continue;
    }
    int way = -1;
    bool evicting = false;
    const unsigned empty = __ballot_sync(0xffffffffu, line == kEmptyKey);
    if (empty) {
      way = __ffs(empty) - 1;
    } else {
      const unsigned st = *reinterpret_cast<volatile unsigned*>(&c.stamps[set * kWays + lane]);
      unsigned long long best = (static_cast<unsigned long long>(st) << 5) | lane;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other < best ? other : best;
      }
      if (static_cast<unsigned>(best >> 5) < protect_from) { way = static_cast<int>(best & 31); evicting = true; }
    }
    if (way < 0) {                               // every way holds a protected row
      if (lane == 0 && refused_keys) refused_keys[atomicAdd(refused_count, 1)] = static_cast<long long>(key);
      unlock_set(&c.locks[set], lane);
      continue;
    }
    const unsigned long long slot = set * kWays + way;
    if (evicting && c.dirty[slot] && evict_keys) {
      int pos = 0;
      if (lane == 0) pos = atomicAdd(evict_count, 1);
      pos = __shfl_sync(0xffffffffu, pos, 0);
      copy_row(evict_values + static_cast<long long>(pos) * c.dim, c.values + slot * c.dim, c.dim, lane);
      const unsigned long long old = __shfl_sync(0xffffffffu, line, way);
      if (lane == 0) evict_keys[pos] = static_cast<long long>(old);
    }
    if (lane == 0) {
      atomicAdd(&c.vers[slot], 1u);
      __threadfence();
    }
    __syncwarp();
    copy_row(c.values + slot * c.dim, values + i * c.dim, c.dim, lane);
    if (lane == 0) {
      *reinterpret_cast<volatile unsigned long long*>(&c.keys[slot]) = key;
      c.stamps[slot] = now;
      c.dirty[slot] = 0;
    }
    __threadfence();
    __syncwarp();
    if (lane == 0) atomicAdd(&c.vers[slot], 1u);
    unlock_set(&c.locks[set], lane);
  }
}

// Optimizer step on cached rows, in place.  A cached row is [D weights | state | padding] (dim = D + 4).  keys are distinct;
// grad [n, D] and norm [n] (sum of squares over the key's occurrences).  optimizer 0: w -= lr * g; 1 (row-wise Adagrad):
// state += norm / D, w -= lr * g / (sqrt(state) + eps).  A key that is not cached is appended to missing (cursor
// missing_count) with its index, for the caller to apply on the backing store.
__global__ void __launch_bounds__(256) cache_apply_kernel(CacheView c, const long long* __restrict__ keys, const int* n_dev, long long n_cap,
                                                          const float* __restrict__ grad, const float* __restrict__ norm, int D, float lr,
                                                          float eps, int optimizer, long long* __restrict__ missing_index,
                                                          int* missing_count) {
  const int lane = threadIdx.x & 31;
  const long long warp = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long nwarps = static_cast<long long>(gridDim.x) * (blockDim.x >> 5);
  const long long n = n_dev ? min(static_cast<long long>(*n_dev), n_cap) : n_cap;
  for (long long i = warp; i < n; i += nwarps) {
    const unsigned long long key = static_cast<unsigned long long>(keys[i]);
    if (key == kEmptyKey) continue;
    const unsigned long long set = ht_hash(key) % c.nsets;
    const unsigned long long line = c.keys[set * kWays + lane];
    const unsigned hit = __ballot_sync(0xffffffffu, line == key);
    if (!hit) {
      if (lane == 0 && missing_index) missing_index[atomicAdd(missing_count, 1)] = i;
      continue;
    }
    const unsigned long long slot = set * kWays + (__ffs(hit) - 1);
    float* row = c.values + slot * c.dim;
    if (lane == 0) {
      atomicAdd(&c.vers[slot], 1u);
      __threadfence();
    }
    __syncwarp();
    float scale = -lr;
    if (optimizer == 1) {
      const float stt = row[D] + (norm ? norm[i] : 0.f) / static_cast<float>(D);
      scale = -lr / (sqrtf(stt) + eps);
      __syncwarp();
      if (lane == 0) row[D] = stt;
    }
    for (int v = lane; v < (D >> 2); v += 32) {
      float4 w = reinterpret_cast<float4*>(row)[v];
      const float4 g = __ldg(reinterpret_cast<const float4*>(grad + i * D) + v);
      w.x += scale * g.x; w.y += scale * g.y; w.z += scale * g.z; w.w += scale * g.w;
      reinterpret_cast<float4*>(row)[v] = w;
    }
    if (lane == 0) c.dirty[slot] = 1;
    __threadfence();
    __syncwarp();
    if (lane == 0) atomicAdd(&c.vers[slot], 1u);
  }
}

__global__ void cache_set_clock_kernel(unsigned* clock, unsigned v) { *clock = v; }

// Every dirty row of the set range -> (keys, values), dirty bits cleared: a flush for checkpoints.
__global__ void __launch_bounds__(256) cache_flush_dirty_kernel(CacheView c, long long* __restrict__ keys_out, float* __restrict__ values_out,
                                                                int* count) {
  const int lane = threadIdx.x & 31;
  const unsigned long long warp = static_cast<unsigned long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const unsigned long long nwarps = static_cast<unsigned long long>(gridDim.x) * (blockDim.x >> 5);
  for (unsigned long long slot = warp; slot < c.nsets * kWays; slot += nwarps) {
    if (c.keys[slot] == kEmptyKey || !c.dirty[slot]) continue;
    int pos = 0;
    if (lane == 0) pos = atomicAdd(count, 1);
    pos = __shfl_sync(0xffffffffu, pos, 0);
    if (lane == 0) { keys_out[pos] = static_cast<long long>(c.keys[slot]); c.dirty[slot] = 0; }
    copy_row(values_out + static_cast<long long>(pos) * c.dim, c.values + slot * c.dim, c.dim, lane);
  }
}

__global__ void cache_dump_kernel(CacheView c, unsigned long long set_begin, unsigned long long set_end,
                                  long long* __restrict__ keys_out, unsigned long long* count) {
  const unsigned long long i = set_begin * kWays + static_cast<unsigned long long>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= set_end * kWays) return;
  const unsigned long long k = c.keys[i];
  if (k == kEmptyKey) return;
  keys_out[atomicAdd(count, 1ull)] = static_cast<long long>(k);
}

struct CacheOwned {
  CacheView v;
};
}  // namespace

// num_items is rounded up to a multiple of 32; dim must be a multiple of 4.
RS_API int rs_cache_create(unsigned long long num_items, int dim, void** handle) {
  RS_REQUIRE(handle && num_items > 0 && dim > 0 && dim % 4 == 0, "rs_cache_create: bad argument (dim %% 4 == 0)");
  CacheOwned* h = new CacheOwned();
  CacheView& v = h->v;
  v.nsets = (num_items + kWays - 1) / kWays;
  v.dim = dim;
  const unsigned long long slots = v.nsets * kWays;
  RS_CUDA(cudaMalloc(&v.keys, slots * sizeof(unsigned long long)));
  RS_CUDA(cudaMalloc(&v.stamps, slots * sizeof(unsigned)));
  RS_CUDA(cudaMalloc(&v.vers, slots * sizeof(unsigned)));
  RS_CUDA(cudaMalloc(&v.dirty, slots));
  RS_CUDA(cudaMalloc(&v.values, slots * static_cast<size_t>(dim) * sizeof(float)));
  RS_CUDA(cudaMalloc(&v.locks, v.nsets * sizeof(int)));
  RS_CUDA(cudaMalloc(&v.clock, sizeof(unsigned)));
  cache_init_kernel<<<static_cast<unsigned>((slots + 255) / 256), 256>>>(v);
  RS_LAUNCH_CHECK();
  RS_CUDA(cudaDeviceSynchronize());
  *handle = h;
  return RS_OK;
}
RS_API int rs_cache_destroy(void* handle) {
  if (!handle) return RS_OK;
  CacheOwned* h = static_cast<CacheOwned*>(handle);
  cudaFree(h->v.keys); cudaFree(h->v.stamps); cudaFree(h->v.vers); cudaFree(h->v.dirty); cudaFree(h->v.values); cudaFree(h->v.locks); cudaFree(h->v.clock);
  delete h;
  return RS_OK;
}
RS_API unsigned long long rs_cache_capacity(void* handle) { return static_cast<CacheOwned*>(handle)->v.nsets * kWays; }
RS_API unsigned long long rs_cache_num_sets(void* handle) { return static_cast<CacheOwned*>(handle)->v.nsets; }

// out: [n, dim] (hit rows written, miss rows untouched); miss_index / miss_keys: [n]; miss_count: device int.
RS_API int rs_cache_query(void* handle, const long long* keys, long long n, float* out, long long* miss_index,
                          long long* miss_keys, int* miss_count, cudaStream_t stream) {
  RS_REQUIRE(handle && keys && miss_index && miss_keys && miss_count, "rs_cache_query: null argument");   // out == null: probe only
  CacheView& v = static_cast<CacheOwned*>(handle)->v;
  cache_tick_kernel<<<1, 1, 0, stream>>>(v.clock, miss_count);
  RS_LAUNCH_CHECK();
  if (n == 0) return RS_OK;
  long long warps = (n + kProbeKeys - 1) / kProbeKeys;
  if (warps > 148 * 64) warps = 148 * 64;
  cache_query_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, stream>>>(v, keys, n, out, miss_index, miss_keys, miss_count);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
RS_API int rs_cache_replace(void* handle, const long long* keys, long long n, const float* values,
                            unsigned long long* status, cudaStream_t stream) {
  RS_REQUIRE(handle && keys && values, "rs_cache_replace: null argument");
  if (n == 0) return RS_OK;
  CacheView& v = static_cast<CacheOwned*>(handle)->v;
  const long long per = 32 / kProbeLanes;
  long long warps = (n + per - 1) / per;
  if (warps > 148 * 64) warps = 148 * 64;
  cache_write_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, stream>>>(v, keys, n, values, 0, status);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
RS_API int rs_cache_update(void* handle, const long long* keys, long long n, const float* values,
                           unsigned long long* status, cudaStream_t stream) {
  RS_REQUIRE(handle && keys && values, "rs_cache_update: null argument");
  if (n == 0) return RS_OK;
  CacheView& v = static_cast<CacheOwned*>(handle)->v;
  const long long per = 32 / kProbeLanes;
  long long warps = (n + per - 1) / per;
  if (warps > 148 * 64) warps = 148 * 64;
  cache_write_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, stream>>>(v, keys, n, values, 1, status);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
// keys_out must hold (set_end - set_begin) * 32 entries; count: device counter, zeroed here.
RS_API int rs_cache_dump(void* handle, unsigned long long set_begin, unsigned long long set_end, long long* keys_out,
                         unsigned long long* count, cudaStream_t stream) {
  RS_REQUIRE(handle && keys_out && count, "rs_cache_dump: null argument");
  CacheView& v = static_cast<CacheOwned*>(handle)->v;
  RS_REQUIRE(set_begin <= set_end && set_end <= v.nsets, "rs_cache_dump: set range [%llu, %llu) outside [0, %llu)",
             set_begin, set_end, v.nsets);
  RS_CUDA(cudaMemsetAsync(count, 0, sizeof(unsigned long long), stream));
  const unsigned long long slots = (set_end - set_begin) * kWays;
  if (slots == 0) return RS_OK;
  cache_dump_kernel<<<static_cast<unsigned>((slots + 255) / 256), 256, 0, stream>>>(v, set_begin, set_end, keys_out, count);
  RS_LAUNCH_CHECK();
  return RS_OK;
}

// ---- write-back cache verbs (the HBM tier of a table whose backing store is host memory)
// keys may be bounded by a device count n_dev (<= n_cap).  evict_* / refused_* outputs hold up to n_cap entries; their
// counters are NOT cleared here (one pair of counters can collect over several calls).
RS_API int rs_cache_replace_evict(void* handle, const long long* keys, const int* n_dev, long long n_cap, const float* values,
                                  unsigned protect_from, long long* evict_keys, float* evict_values, int* evict_count,
                                  long long* refused_keys, int* refused_count, unsigned long long* status, cudaStream_t stream) {
  RS_REQUIRE(handle && keys && values, "rs_cache_replace_evict: null argument");
  RS_REQUIRE(!evict_keys || (evict_values && evict_count), "rs_cache_replace_evict: eviction output needs values and a counter");
  RS_REQUIRE(!refused_keys || refused_count, "rs_cache_replace_evict: refusal output needs a counter");
  if (n_cap == 0) return RS_OK;
  CacheView& v = static_cast<CacheOwned*>(handle)->v;
  long long warps = n_cap < 148 * 32 ? n_cap : 148 * 32;
  cache_replace_evict_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, stream>>>(v, keys, n_dev, n_cap, values, protect_from,
                                                                                        evict_keys, evict_values, evict_count,
                                                                                        refused_keys, refused_count, status);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
// D: weights per row; the cache was created with dim >= D + 1 (state at column D).
RS_API int rs_cache_apply(void* handle, const long long* keys, const int* n_dev, long long n_cap, const float* grad, const float* norm,
                          int D, float lr, float eps, int optimizer, long long* missing_index, int* missing_count, cudaStream_t stream) {
  RS_REQUIRE(handle && keys && grad, "rs_cache_apply: null argument");
  CacheView& v = static_cast<CacheOwned*>(handle)->v;
  RS_REQUIRE(D % 4 == 0 && D > 0 && D + 1 <= v.dim, "rs_cache_apply: rows of %d weights need a cache of at least %d columns (has %d)", D, D + 1, v.dim);
  RS_REQUIRE(!missing_index || missing_count, "rs_cache_apply: the missing list needs a counter");
  if (n_cap == 0) return RS_OK;
  long long warps = n_cap < 148 * 32 ? n_cap : 148 * 32;
  cache_apply_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, stream>>>(v, keys, n_dev, n_cap, grad, norm, D, lr, eps, optimizer,
                                                                                missing_index, missing_count);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
RS_API int rs_cache_set_clock(void* handle, unsigned value, cudaStream_t stream) {
  RS_REQUIRE(handle, "rs_cache_set_clock: null handle");
  cache_set_clock_kernel<<<1, 1, 0, stream>>>(static_cast<CacheOwned*>(handle)->v.clock, value);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
// keys_out / values_out: room for the whole capacity; count: device int, cleared here.
RS_API int rs_cache_flush_dirty(void* handle, long long* keys_out, float* values_out, int* count, cudaStream_t stream) {
  RS_REQUIRE(handle && keys_out && values_out && count, "rs_cache_flush_dirty: null argument");
  CacheView& v = static_cast<CacheOwned*>(handle)->v;
  RS_CUDA(cudaMemsetAsync(count, 0, sizeof(int), stream));
  cache_flush_dirty_kernel<<<148 * 4, 256, 0, stream>>>(v, keys_out, values_out, count);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
// Query variant that does not advance the clock (the caller sets it with rs_cache_set_clock) and may skip the row copy
// (out == null: probe: stamps the hits, lists the misses).
RS_API int rs_cache_query_noclock(void* handle, const long long* keys, long long n, float* out, long long* miss_index,
                                  long long* miss_keys, int* miss_count, cudaStream_t stream) {
  RS_REQUIRE(handle && keys && miss_index && miss_keys && miss_count, "rs_cache_query_noclock: null argument");
  CacheView& v = static_cast<CacheOwned*>(handle)->v;
  RS_CUDA(cudaMemsetAsync(miss_count, 0, sizeof(int), stream));
  if (n == 0) return RS_OK;
  long long warps = (n + kProbeKeys - 1) / kProbeKeys;
  if (warps > 148 * 64) warps = 148 * 64;
  cache_query_kernel<<<static_cast<unsigned>((warps + 7) / 8), 256, 0, stream>>>(v, keys, n, out, miss_index, miss_keys, miss_count);
  RS_LAUNCH_CHECK();
  return RS_OK;
}

// out[missing_index[i]] = retrieved[i]  (the reference's merge_op, src/framework/pytorch/merge.cu:6-18)
namespace {
__global__ void merge_rows_kernel(float* __restrict__ out, const float* __restrict__ retrieved,
                                  const long long* __restrict__ missing_index, long long n, int dim) {
  const long long i = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const int lane = threadIdx.x & 31;
  const long long d = missing_index[i];
  if ((dim & 3) == 0) {
    for (int v = lane; v < (dim >> 2); v += 32)
      reinterpret_cast<float4*>(out + d * dim)[v] = reinterpret_cast<const float4*>(retrieved + i * dim)[v];
  } else {
    for (int v = lane; v < dim; v += 32) out[d * dim + v] = retrieved[i * dim + v];
  }
}
// dst[i] = key in [start, end) ? hbm[key - start] : host_table[key]   (uva_cache_query_op,
// src/framework/pytorch/recstore_pytorch.cu:12-37); host_table is device-accessible host memory.
__global__ void range_cache_query_kernel(float* __restrict__ dst, const long long* __restrict__ ids, long long n, int dim,
                                         const float* __restrict__ hbm, const float* __restrict__ host_table, long long start,
                                         long long end, long long host_rows, unsigned long long* status) {
  const long long i = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const int lane = threadIdx.x & 31;
  const long long k = ids[i];
  const float* src;
  bool host = false;
  if (k >= start && k < end) src = hbm + (k - start) * dim;
  else if (k >= 0 && k < host_rows) { src = host_table + k * dim; host = true; }
  else {
    if (lane == 0 && status) atomicOr(status, (unsigned long long)RS_DEV_OOB_ROW);
    return;
  }
  // Host rows are written by the CPU between kernels: they are read around the GPU's caches, every time.
  if ((dim & 3) == 0) {
    for (int v = lane; v < (dim >> 2); v += 32)
      reinterpret_cast<float4*>(dst + i * dim)[v] = host ? __ldcv(reinterpret_cast<const float4*>(src) + v) : reinterpret_cast<const float4*>(src)[v];
  } else {
    for (int v = lane; v < dim; v += 32) dst[i * dim + v] = host ? __ldcv(src + v) : src[v];
  }
}
}  // namespace

RS_API int rs_merge_rows(float* out, const float* retrieved, const long long* missing_index, long long n, int dim,
                         cudaStream_t stream) {
  RS_REQUIRE(out && retrieved && missing_index, "rs_merge_rows: null argument");
  if (n == 0) return RS_OK;
  merge_rows_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(out, retrieved, missing_index, n, dim);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
RS_API int rs_range_cache_query(float* dst, const long long* ids, long long n, int dim, const float* hbm,
                                const float* host_table, long long start, long long end, long long host_rows,
                                unsigned long long* status, cudaStream_t stream) {
  RS_REQUIRE(dst && ids && hbm && host_table, "rs_range_cache_query: null argument");
  if (n == 0) return RS_OK;
  range_cache_query_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(dst, ids, n, dim, hbm, host_table, start,
                                                                                   end, host_rows, status);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
