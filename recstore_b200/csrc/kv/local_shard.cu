// Lookup, get and put on a shard whose keys all live on the calling GPU (one rank): no buckets, no exchange windows.
//
// The multi-GPU verbs (comm/shard_exchange.cu) fold duplicate keys, send keys to their owners, and send rows back through
// windows; with one rank each of those passes only moves data around the same HBM.  Here ONE kernel resolves the keys (row
// number, or find-or-insert in the shard's hash table) and copies the rows; the optimizer then takes the occurrences as they
// are (ops/embedding.cu folds equal rows on its way).  Lookup + Adagrad update of 262,144 keys x 32 at Zipf 1.1: 182 -> 62 us;
// lookup + update + get of 32,768 keys on a hash-table shard: 184 -> 42 us.  Results are those of the exchange path: gets and lookups of reference's
// PS shard (src/ps/base/cache_ps_impl.h:60-140) with first-touch insertion.
#include "common/row_vec.cuh"
#include "common/rs_common.h"
#include "kv/hash_table.cuh"
#include "kv/key_init.cuh"

namespace {

struct LocalShardArgs {
  float* weight;
  long long local_rows;
  const long long* ids;        // [n]; negative = padding: a zero row, nothing inserted
  long long n;
  int D;
  float* out;                  // [n, D] or null
  long long* rows;             // [n] row of every id or -1, or null
  unsigned char* found;        // [n] or null (get): 0 for an absent key or a row that starts with a NaN, which reads as zeros
  const float* values;         // put: rows to store, or null
  float* state;                // put: optimizer state to reset, or null
  int use_hash, find_only, refuse_reserved;
  rs::HashTableView ht;
  float init_scale;
  unsigned char* row_init;
  unsigned long long* status;
};

__device__ __forceinline__ void load_16(rs::RowVec<8>& r, const float* p) {
  const float4 a = __ldg(reinterpret_cast<const float4*>(p)), b = __ldg(reinterpret_cast<const float4*>(p) + 1);
  r.v[0] = a.x; r.v[1] = a.y; r.v[2] = a.z; r.v[3] = a.w; r.v[4] = b.x; r.v[5] = b.y; r.v[6] = b.z; r.v[7] = b.w;
}
__device__ __forceinline__ void load_16(rs::RowVec<4>& r, const float* p) { rs::row_load_nc(r, p); }

// A warp takes `kpw` consecutive ids (32, fewer when the batch would leave SMs without work).  Every lane resolves one of them, so
// up to 32 hash probes are in flight per warp (bound by these chains of dependent loads: 17 us for 262,144 dense rows of 32
// floats, 16 us for 32,768 hashed ones from cold caches); its sub-warps of L lanes then copy the rows, U of them in flight each.
template <int V, int L>
__global__ void __launch_bounds__(128) local_shard_kernel(const LocalShardArgs a, const int kpw) {
  constexpr int G = 32 / L;
  constexpr int U = V == 8 ? 4 : 8;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, l = lane & (L - 1), g = lane / L;
  const unsigned wm = L == 32 ? kAll : ((1u << (L & 31)) - 1u) << (g * L);
  const long long i0 = (static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5)) * kpw;
  if (i0 >= a.n) return;
  const int m = static_cast<int>(min(static_cast<long long>(kpw), a.n - i0));
  const int nvec = a.D / V;

  // flags of this lane's id
  enum { kFresh = 1, kFormula = 2, kAbsent = 4 };
  long long key = -1, row = -1;
  int fl = 0;
  if (lane < m) {
    key = a.ids[i0 + lane];
    if (key < 0) {
      if (a.refuse_reserved && static_cast<unsigned long long>(key) >= rs::kHtTomb && a.status)
        atomicOr(a.status, (unsigned long long)RS_DEV_BAD_ARG);
    } else if (a.use_hash) {
      if (a.find_only) {
        row = rs::ht_find(a.ht, static_cast<unsigned long long>(key));
        if (row < 0) fl |= kAbsent;
      } else {
        bool ins = false, full = false;
        row = rs::ht_insert(a.ht, static_cast<unsigned long long>(key), &ins, &full);
        if (full && a.status) atomicOr(a.status, (unsigned long long)RS_DEV_TABLE_FULL);
        if (ins) fl |= kFresh | kFormula;
      }
      // A key that another thread inserted a moment ago may not hold its initial value yet: such a reader computes the same
      // value from the key instead of reading the row.
      if (row >= 0 && !(fl & kFresh) && *reinterpret_cast<volatile unsigned char*>(a.row_init + row) == 0) fl |= kFormula;
    } else if (key < a.local_rows) {
      row = key;
    } else if (a.status) {
      atomicOr(a.status, (unsigned long long)RS_DEV_OOB_ROW);
    }
    if (a.rows) a.rows[i0 + lane] = row;
  }
  if (a.use_hash) {
    __threadfence();                           // the flag bytes above before the rows below
    __syncwarp();
  }
  if (a.values == nullptr && a.out == nullptr && !__any_sync(kAll, fl & kFresh)) return;   // rows resolved, nothing to move

  for (int j0 = 0; j0 < m; j0 += G * U) {
    long long r[U], k[U];
    int f[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = (j0 + u * G + g) & 31;
      r[u] = __shfl_sync(kAll, row, j);
      f[u] = __shfl_sync(kAll, fl, j);
      k[u] = a.use_hash ? __shfl_sync(kAll, key, j) : 0;
    }
    bool drop[U];
#pragma unroll
    for (int u = 0; u < U; ++u) drop[u] = false;
    for (int v = l; v - l < nvec; v += L) {     // (all lanes of a sub-warp make the same number of steps)
      rs::RowVec<V> x[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = j0 + u * G + g;
        rs::row_zero(x[u]);
        if (j >= m || v >= nvec) continue;
        if (a.values) {
          if (r[u] >= 0) load_16(x[u], a.values + (i0 + j) * a.D + v * V);
        } else if (r[u] >= 0 && !(f[u] & kFormula) && a.out) {
          rs::row_load_cg(x[u], a.weight + r[u] * a.D + v * V);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = j0 + u * G + g;
        if (a.found && v == l) {                // first step: lane 0 of the sub-warp holds the row's first element
          const float first = __shfl_sync(wm, x[u].v[0], 0, L);
          drop[u] = (f[u] & kAbsent) || (first != first && !(f[u] & kFormula));
          if (l == 0 && j < m) a.found[i0 + j] = drop[u] ? 0 : 1;
        }
        if (j >= m || v >= nvec) continue;
        float* const at = a.weight + r[u] * a.D + v * V;
        if (a.values) {
          if (r[u] >= 0) rs::row_store(at, x[u]);
          continue;
        }
        if (r[u] >= 0 && (f[u] & kFormula)) {
#pragma unroll
          for (int e = 0; e < V; ++e) x[u].v[e] = rs::key_init_value(static_cast<unsigned long long>(k[u]), v * V + e, a.init_scale);
          if (f[u] & kFresh) rs::row_store(at, x[u]);                  // first touch: the row keeps it
        }
        if (drop[u]) rs::row_zero(x[u]);
        if (a.out) rs::row_store(a.out + (i0 + j) * a.D + v * V, x[u]);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int j = j0 + u * G + g;
      const bool wrote = j < m && r[u] >= 0 && (a.values != nullptr || (f[u] & kFresh));
      __syncwarp(wm);
      if (wrote && l == 0) {
        if (a.values && a.state) a.state[r[u]] = 0.f;
        if (a.row_init) {
          __threadfence();
          *reinterpret_cast<volatile unsigned char*>(a.row_init + r[u]) = 1;
        }
      }
    }
  }
}

}  // namespace

// One launch for every verb of a one-rank shard.
//   lookup: out + rows;  get: out + found, find_only;  put: values (+ state, row_init);  resolve only: rows, nothing else.
// ht null: ids are row numbers below local_rows (others: zero row, RS_DEV_OOB_ROW).  refuse_reserved: the keys -1 and -2 set
// RS_DEV_BAD_ARG, as they do where duplicates are folded.
RS_API int rs_shard_local(float* weight, long long local_rows, const long long* ids, long long n, int D, float* out, long long* rows,
                          unsigned char* found, const float* values, float* state, const rs::HashTableView* ht, int find_only,
                          int refuse_reserved, float init_scale, unsigned char* row_init, unsigned long long* status,
                          cudaStream_t stream) {
  RS_REQUIRE(weight && (ids || n == 0) && n >= 0 && D > 0 && D % 4 == 0 && local_rows >= 0, "rs_shard_local: bad argument");
  RS_REQUIRE(!ht || row_init, "rs_shard_local: the hash-table shard needs its row_init bytes");
  RS_REQUIRE(!found || out, "rs_shard_local: found flags come with the rows");
  if (n == 0) return RS_OK;
  LocalShardArgs a;
  memset(&a, 0, sizeof(a));
  a.weight = weight; a.local_rows = local_rows; a.ids = ids; a.n = n; a.D = D; a.out = out; a.rows = rows; a.found = found;
  a.values = values; a.state = state; a.use_hash = ht != nullptr; a.find_only = find_only; a.refuse_reserved = refuse_reserved;
  if (ht) a.ht = *ht;
  a.init_scale = init_scale; a.row_init = row_init; a.status = status;
  // Ids per warp: 32 once every SM has sixteen warps, fewer in a small batch, but one for every sub-warp.
  auto launch = [&](auto kern, int L) -> int {
    int kpw = 32;
    while (kpw > 32 / L && n < 148ll * 16 * kpw) kpw >>= 1;
    const long long grid = (n + 4 * kpw - 1) / (4 * kpw);
    RS_REQUIRE(grid < (1ll << 31), "rs_shard_local: too many ids");
    kern<<<static_cast<unsigned>(grid), 128, 0, stream>>>(a, kpw);
    return RS_OK;
  };
  int rc;
  if (rs::row_wide(weight, D)) {
    if (D <= 32) rc = launch(local_shard_kernel<8, 4>, 4);
    else if (D <= 64) rc = launch(local_shard_kernel<8, 8>, 8);
    else if (D <= 128) rc = launch(local_shard_kernel<8, 16>, 16);
    else rc = launch(local_shard_kernel<8, 32>, 32);
  } else {
    if (D <= 32) rc = launch(local_shard_kernel<4, 8>, 8);
    else rc = launch(local_shard_kernel<4, 32>, 32);
  }
  if (rc != RS_OK) return rc;
  RS_LAUNCH_CHECK();
  return RS_OK;
}
