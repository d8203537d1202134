// Fused embedding forward and backward for model-parallel embedding shards on sm_100a.
//
// Forward (rs_emb_forward): for every (local table, sample) bag it resolves the ids to rows of
// the shard (direct index or hash-table probe), sum-pools the rows (optional per-sample
// weights) and stores the pooled vector STRAIGHT INTO THE DESTINATION RANK'S BUFFER through a
// peer pointer: destination rank = sample / B_local, address = dst[rank] + (sample % B_local) *
// row_stride + dst_col[table].  With peer windows mapped over NVLink this is the table-wise
// all-to-all of the reference (nn.EmbeddingBag per table, src/executable/dlrm/dlrm_model.py:
// 255-314, followed by all_to_all_single, extend_distributed.py:389-426) done by the gather
// kernel itself, with no pack/unpack and no collective call.  It also replaces the plain
// gather kernels uva_cache_query / UVAQueryKernel / LookupKernel
// (src/framework/pytorch/recstore_pytorch.cu:12-37, src/storage/gpu_cache/gpu_cache_nohash.cu:
// 2-12, static_hash_table.cu:223-268).
//
// Backward (rs_emb_backward): consumes per-bag gradients (as pushed by the peers into this
// rank's gradient window), counting-sorts each 256-occurrence group by row in shared memory so
// that equal rows are adjacent, sums every run in registers and applies SGD or row-wise Adagrad in
// place with one vector atomic per run.  Semantics follow the reference optimizers
// (src/python/pytorch/recstore/DistOpt.py:511-557): state[row] += sum over occurrences of
// mean(g^2); W[row] -= lr * sum over occurrences of g / (sqrt(state[row]) + eps), with the
// state read after all occurrences of the step were accumulated (hence two passes).
//
// No kernel here traps: out-of-range ids set RS_DEV_OOB_ROW in the status word and are skipped.
#include <cuda_bf16.h>
#include <cstdlib>
#include "common/row_vec.cuh"
#include "common/rs_common.h"
#include "comm/flags.cuh"
#include "kv/hash_table.cuh"

namespace {

struct EmbFwdArgs {
  const float* weight;
  const long long* table_base;   // [T] first row of each local table inside `weight`
  const long long* table_rows;   // [T] number of rows of each local table
  const long long* indices;      // [nnz]
  const long long* offsets;      // [T*B + 1] or null when hotness is fixed per table
  const int* hotness;            // [T] used when offsets == null
  const long long* hot_base;     // [T] start of table t's ids inside `indices` when offsets == null
  const float* psw;              // optional per-sample weights [nnz]
  int T, B, D, B_local;
  void* const* dst;              // [world] destination base pointers
  long long dst_row_stride;      // elements
  const int* dst_col;            // [T] element offset of the table's feature inside a destination row
  int out_bf16;
  long long* row_idx;            // optional [nnz]: resolved row per id (-1 if invalid)
  int* occ2bag;                  // optional [nnz]
  int use_hash;
  rs::HashTableView ht;
  unsigned long long* status;
  // Row-sharded tables (a table spread cyclically over the ranks, this rank holding ids with id % id_div == id_rem at
  // local row id / id_div): the ids of a bag arrive from the sample's rank in a fixed-capacity region of `hotness`
  // slots, of which only counts[bag] are filled.
  const int* counts;             // [T*B] or null
  int id_div, id_rem;            // 1, 0 for whole tables
  // Occurrence list for the backward pass, compacted: positions come from an atomic cursor instead of the id's index
  // (the regions above are mostly holes).  Null = write at the id's own index.
  int* occ_cursor;
  rs::FlagWait wait;             // optional: wait for the source rank's keys before reading a bag
  rs::FlagSignal sig;            // optional: publish "my pooled rows have landed" when the grid is done
};

constexpr int kMaxChunks = 4;  // D <= 512

template <int NC>
__device__ __forceinline__ void store_pooled(const EmbFwdArgs& a, int t, int b, const float4 (&acc)[NC], int lane, int nvec) {
  const int dst_rank = b / a.B_local;
  const long long off = static_cast<long long>(b - dst_rank * a.B_local) * a.dst_row_stride + a.dst_col[t];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int v = lane + c * 32;
    if (v < nvec) {
      if (a.out_bf16) {
        __nv_bfloat16* d = reinterpret_cast<__nv_bfloat16*>(a.dst[dst_rank]) + off;
        __nv_bfloat162 lo = __floats2bfloat162_rn(acc[c].x, acc[c].y);
        __nv_bfloat162 hi = __floats2bfloat162_rn(acc[c].z, acc[c].w);
        uint2 o;
        o.x = *reinterpret_cast<uint32_t*>(&lo);
        o.y = *reinterpret_cast<uint32_t*>(&hi);
        *(reinterpret_cast<uint2*>(d) + v) = o;
      } else {
        float* d = reinterpret_cast<float*>(a.dst[dst_rank]) + off;
        *(reinterpret_cast<float4*>(d) + v) = acc[c];
      }
    }
  }
}

// Bags of a row-sharded table (fixed-capacity regions filled by the peers, compact occurrence list): one warp per block of
// 32 consecutive bags of one table; lane i resolves the metadata of bag i.
template <int NC>
__device__ __forceinline__ void emb_fwd_body(const EmbFwdArgs& a, long long blk) {
  const int lane = threadIdx.x & 31;
  const int blocks_per_table = (a.B + 31) >> 5;
  const int t = static_cast<int>(blk / blocks_per_table);
  const int b0 = static_cast<int>(blk % blocks_per_table) << 5;
  const int nb = min(32, a.B - b0);
  const long long base = a.table_base[t];
  const long long nrows = a.table_rows[t];
  const int nvec = a.D >> 2;

  if (a.wait.my_flags != nullptr) {
    // The bags of this warp come from one source rank (two when the block of 32 straddles a boundary).
    const int s0 = b0 / a.B_local, s1 = (b0 + nb - 1) / a.B_local;
    for (int src = s0; src <= s1; ++src) rs::flag_wait_one_warp(a.wait, src);
  }
  long long beg = 0, end = 0;
  if (lane < nb) {
    const long long bag = static_cast<long long>(t) * a.B + b0 + lane;
    if (a.offsets) {
      beg = a.offsets[bag];
      end = a.offsets[bag + 1];
    } else {
      const int h = a.hotness[t];
      beg = a.hot_base[t] + static_cast<long long>(b0 + lane) * h;
      end = beg + (a.counts ? min(max(__ldcv(a.counts + bag), 0), h) : h);
    }
  }
  const bool sharded = a.id_div > 1;
  auto resolve = [&](long long id) -> long long {
    if (a.use_hash) return rs::ht_find(a.ht, static_cast<unsigned long long>(id));
    if (!sharded) {
      if (id >= 0 && id < nrows) return base + id;
    } else if (id >= 0 && id % a.id_div == a.id_rem && id / a.id_div < nrows) {
      return base + id / a.id_div;
    }
    if (a.status) atomicOr(a.status, (unsigned long long)RS_DEV_OOB_ROW);
    return -1;
  };
  for (int j = 0; j < nb; ++j) {
    const long long jb = __shfl_sync(0xffffffffu, beg, j);
    const long long je = __shfl_sync(0xffffffffu, end, j);
    const long long bag = static_cast<long long>(t) * a.B + b0 + j;
    float4 acc[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) acc[c] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (long long i0 = jb; i0 < je; i0 += 32) {
      const int n = static_cast<int>(min(32ll, je - i0));
      long long my_row = -1;
      float my_w = 1.f;
      long long opos = i0;                        // where this chunk's occurrences are recorded
      if (a.occ_cursor != nullptr) {
        int p = 0;
        if (lane == 0) p = atomicAdd(a.occ_cursor, n);
        opos = __shfl_sync(0xffffffffu, p, 0);
      }
      if (lane < n) {
        const long long id = a.counts ? __ldcv(a.indices + i0 + lane) : a.indices[i0 + lane];   // pushed by a peer: not through L1
        my_row = resolve(id);
        if (a.psw) my_w = a.psw[i0 + lane];
        if (a.row_idx) a.row_idx[opos + lane] = my_row;
        if (a.occ2bag) a.occ2bag[opos + lane] = static_cast<int>(bag);
      }
      for (int k0 = 0; k0 < n; k0 += 4) {
        long long r[4];
        float w[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          r[u] = __shfl_sync(0xffffffffu, my_row, (k0 + u) & 31);
          w[u] = __shfl_sync(0xffffffffu, my_w, (k0 + u) & 31);
          if (k0 + u >= n) r[u] = -1;
        }
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          const int v = lane + c * 32;
          if (v < nvec) {
            float4 x[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
              x[u] = r[u] >= 0 ? __ldg(reinterpret_cast<const float4*>(a.weight + r[u] * a.D) + v)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int u = 0; u < 4; ++u) {
              acc[c].x += w[u] * x[u].x; acc[c].y += w[u] * x[u].y;
              acc[c].z += w[u] * x[u].z; acc[c].w += w[u] * x[u].w;
            }
          }
        }
      }
    }
    store_pooled<NC>(a, t, b0 + j, acc, lane, nvec);
  }
}

template <int NC>
__global__ void __launch_bounds__(256) emb_fwd_sharded_kernel(const EmbFwdArgs a) {
  // Warps loop over the blocks of 32 bags, so the grid can be a single resident wave (see launch_emb_fwd).
  const int warps_per_block = blockDim.x >> 5;
  const long long total = static_cast<long long>(a.T) * ((a.B + 31) >> 5);
  const long long stride = static_cast<long long>(gridDim.x) * warps_per_block;
  for (long long blk = static_cast<long long>(blockIdx.x) * warps_per_block + (threadIdx.x >> 5); blk < total; blk += stride)
    emb_fwd_body<NC>(a, blk);
  rs::flag_publish_when_grid_done(a.sig);   // (no-op without a signal) every thread arrives here
}

// Bags a sub-warp of L lanes takes at once: as many as its lanes can describe while their ids stay near one id per lane of a
// warp, one bag from 17 ids on, never more than `cap`, except that four one-id bags are one batch of loads anyway (and fewer
// CTAs leave a GEMM beside a small lookup more SMs).
template <int L> __device__ __forceinline__ int bags_per_task(long long h, int cap) {
  if (h <= 1 && cap < 4) cap = 4;
  int nb = h <= 1 ? L : (h >= 17 ? 1 : 1 << (31 - __clz(static_cast<int>(32 / h))));
  nb = nb < L ? nb : L;
  return nb < cap ? nb : cap;
}

// Lookup of whole tables.  A sub-warp of L lanes takes a task: up to L consecutive bags of one table, fewer where bags hold
// several ids (see bags_per_task), so a table with 100 ids per bag spreads over as many sub-warps as it has bags.  Tasks are
// numbered table after table; a warp finds the tables of its tasks in a running sum over the tables' task counts, 32 tables
// per step.  Bags with one id each take the short way: all rows of a task in groups of U loads, straight to their places.
// Otherwise the ids of the task's bags, which lie one after another, are walked in chunks of L with U rows in flight and a
// bag is stored when its last id has been added.
// Bound by issue slots and rows in flight (skewed ids hit L2): at 128 floats half a warp per row, 32-byte loads and 16-byte
// bf16 stores.  The form before it (a warp per 32 bags whatever they held, 16-byte loads by a warp per row, destination
// worked out per row) took 180 us for 65,536 x 26 one-id bags at Zipf 1.2 and 342 us for 8,192 x 26 bags of 214 ids a
// sample, there with one table's 256 warps still running long after the others had ended; this one 122 and 106 us (436 MB of
// bf16 rows written in the first case: 66 us at 6.65 TB/s).
template <int V, int L, int NC>
__global__ void __launch_bounds__(256, 3) emb_pool_kernel(const EmbFwdArgs a, const int nb_cap) {
  constexpr int G = 32 / L;
  constexpr int U = V * NC <= 8 ? 4 : 2;
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, l = lane & (L - 1), g = lane / L;
  const unsigned wm = L == 32 ? kAll : ((1u << (L & 31)) - 1u) << (g * L);
  const unsigned stride = gridDim.x * (blockDim.x >> 5) * G;
  const int nvec = a.D / V;
  const int esz = a.out_bf16 ? 2 : 4;

  int jag_nb = 0;
  if (a.offsets) {
    const long long bags = static_cast<long long>(a.T) * a.B;
    jag_nb = bags_per_task<L>((a.offsets[bags] - a.offsets[0] + bags - 1) / bags, nb_cap);
  }
  // Lane i: bags per task and running task count of table tab0 + i.
  int tab0 = 0, my_nb = 1;
  unsigned my_end = 0;
  auto load_tables = [&](int first, unsigned before) {
    tab0 = first;
    const int t = first + lane;
    my_nb = 1;
    unsigned n = 0;
    if (t < a.T) {
      my_nb = a.offsets ? jag_nb : bags_per_task<L>(a.hotness[t], nb_cap);
      n = static_cast<unsigned>((a.B + my_nb - 1) / my_nb);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(kAll, n, o);
      if (lane >= o) n += y;
    }
    my_end = before + n;
  };
  load_tables(0, 0);
  unsigned before = 0;                                   // tasks of the tables below tab0

  for (unsigned base = (blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * G;; base += stride) {
    const unsigned task = base + g;
    // Tables of the warp's tasks.  They ascend, so a step to the next 32 tables is never taken back; a warp whose tasks lie
    // on both sides of such a step serves the lower ones first.
    bool todo = true;
    bool more = true;
    while (more) {
      const unsigned last = __shfl_sync(kAll, my_end, 31);
      const bool here = todo && task < last;
      int pos = 0;
#pragma unroll
      for (int st = 16; st > 0; st >>= 1) {
        const unsigned c = __shfl_sync(kAll, my_end, pos + st - 1);
        if (c <= task) pos += st;
      }
      const unsigned prev = __shfl_sync(kAll, my_end, pos > 0 ? pos - 1 : 0);
      const int nb = __shfl_sync(kAll, my_nb, pos);
      if (here) {
        todo = false;
        const int t = tab0 + pos;
        const int b0 = static_cast<int>((task - (pos > 0 ? prev : before)) * static_cast<unsigned>(nb));
        const int n = min(nb, a.B - b0);
        const long long tbase = a.table_base[t], nrows = a.table_rows[t];
        long long beg = 0, end = 0;
        if (l < n) {
          if (a.offsets) {
            const long long bag = static_cast<long long>(t) * a.B + b0 + l;
            beg = a.offsets[bag];
            end = a.offsets[bag + 1];
          } else {
            const int h = a.hotness[t];
            beg = a.hot_base[t] + static_cast<long long>(b0 + l) * h;
            end = beg + h;
          }
        }
        auto resolve = [&](long long id) -> long long {
          if (a.use_hash) return rs::ht_find(a.ht, static_cast<unsigned long long>(id));
          if (id >= 0 && id < nrows) return tbase + id;
          if (a.status) atomicOr(a.status, (unsigned long long)RS_DEV_OOB_ROW);
          return -1;
        };
        // Where the bags go: all to one rank (one base for the task) unless the task straddles two ranks' samples.
        const int col = a.dst_col[t];
        const int rank0 = b0 / a.B_local;
        const bool one_rank = (b0 + n - 1) < (rank0 + 1) * static_cast<long long>(a.B_local);
        char* const dst0 = reinterpret_cast<char*>(a.dst[rank0]) +
                           ((b0 - rank0 * static_cast<long long>(a.B_local)) * a.dst_row_stride + col) * esz;
        auto place = [&](int j) -> char* {
          if (one_rank) return dst0 + j * (a.dst_row_stride * esz);
          const int r = (b0 + j) / a.B_local;
          return reinterpret_cast<char*>(a.dst[r]) + ((b0 + j - r * static_cast<long long>(a.B_local)) * a.dst_row_stride + col) * esz;
        };
        auto store = [&](int j, const rs::RowVec<V> (&x)[NC]) {
          char* const d = place(j);
          const bool al = (reinterpret_cast<uintptr_t>(d) & 15) == 0;
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            const int v = l + c * L;
            if (v < nvec) {
              if (a.out_bf16) rs::row_store_bf16(reinterpret_cast<__nv_bfloat16*>(d) + v * V, x[c], al);
              else rs::row_store(reinterpret_cast<float*>(d) + v * V, x[c]);
            }
          }
        };
        const int bag0 = t * a.B + b0;                    // (T * B < 2^31, checked on the host)
        if (a.psw == nullptr && __all_sync(wm, l >= n || end - beg == 1)) {
          long long my_row = -1;
          if (l < n) {
            my_row = resolve(a.indices[beg]);
            if (a.row_idx) a.row_idx[beg] = my_row;
            if (a.occ2bag) a.occ2bag[beg] = bag0 + l;
          }
          for (int j0 = 0; j0 < n; j0 += U) {
            rs::RowVec<V> x[U][NC];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const long long r = __shfl_sync(wm, my_row, (j0 + u) & (L - 1), L);
#pragma unroll
              for (int c = 0; c < NC; ++c) {
                rs::row_zero(x[u][c]);
                const int v = l + c * L;
                if (j0 + u < n && r >= 0 && v < nvec) rs::row_load_nc(x[u][c], a.weight + r * a.D + v * V);
              }
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
              if (j0 + u < n) store(j0 + u, x[u]);
          }
        } else {
          rs::RowVec<V> acc[NC];
#pragma unroll
          for (int c = 0; c < NC; ++c) rs::row_zero(acc[c]);
          const long long i_begin = __shfl_sync(wm, beg, 0, L), i_end = __shfl_sync(wm, end, n - 1, L);
          int j = 0;                                      // bag being summed and the end of its ids
          long long j_end = __shfl_sync(wm, end, 0, L);
          auto close = [&]() {
            store(j, acc);
#pragma unroll
            for (int c = 0; c < NC; ++c) rs::row_zero(acc[c]);
            ++j;
            j_end = __shfl_sync(wm, end, j & (L - 1), L);
          };
          for (long long i0 = i_begin; i0 < i_end; i0 += L) {
            const int m = static_cast<int>(min(static_cast<long long>(L), i_end - i0));
            long long my_row = -1;
            float my_w = 1.f;
            // lane l's id belongs to the first bag that ends behind it
            int mine = 0;
#pragma unroll
            for (int st = L / 2; st > 0; st >>= 1) {
              const long long e = __shfl_sync(wm, end, min(mine + st, n) - 1, L);
              if (mine + st <= n - 1 && e <= i0 + l) mine += st;
            }
            if (l < m) {
              my_row = resolve(a.indices[i0 + l]);
              if (a.psw) my_w = a.psw[i0 + l];
              if (a.row_idx) a.row_idx[i0 + l] = my_row;
              if (a.occ2bag) a.occ2bag[i0 + l] = bag0 + mine;
            }
            for (int k0 = 0; k0 < m; k0 += U) {
              rs::RowVec<V> x[U][NC];
              float w[U];
#pragma unroll
              for (int u = 0; u < U; ++u) {
                const long long r = __shfl_sync(wm, my_row, (k0 + u) & (L - 1), L);
                w[u] = __shfl_sync(wm, my_w, (k0 + u) & (L - 1), L);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                  rs::row_zero(x[u][c]);
                  const int v = l + c * L;
                  if (k0 + u < m && r >= 0 && v < nvec) rs::row_load_nc(x[u][c], a.weight + r * a.D + v * V);
                }
              }
#pragma unroll
              for (int u = 0; u < U; ++u) {
                if (k0 + u >= m) break;
                while (j < n - 1 && i0 + k0 + u >= j_end) close();
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                  for (int e = 0; e < V; ++e) acc[c].v[e] = fmaf(w[u], x[u][c].v[e], acc[c].v[e]);
              }
            }
          }
          while (j < n) close();                          // the last bag with ids, and the empty ones after it
        }
      }
      __syncwarp();
      // Another 32 tables when a task of this warp lies behind these.
      more = __any_sync(kAll, todo && task >= last) && tab0 + 32 < a.T;
      if (more) {
        before = last;
        load_tables(tab0 + 32, before);
      }
    }
    // The last table's count is known once it is loaded: a warp none of whose tasks exist is done.
    if (!__any_sync(kAll, !todo)) break;
  }
  rs::flag_publish_when_grid_done(a.sig);   // (no-op without a signal) every thread arrives here
}

// ------------------------------------------------------------------ backward
struct EmbBwdArgs {
  float* weight;
  float* state;                  // [rows] row-wise Adagrad accumulator (null for SGD)
  const long long* row_idx;      // [nnz] resolved rows (-1 = skip)
  const int* occ2bag;            // [nnz] or null (bag == occurrence)
  long long nnz;
  const void* grad;              // per-bag gradients
  const int* grad_col;           // [T] element offset of the table's slice inside a gradient row, or null
  long long grad_row_stride;     // elements between samples
  const float* gnorm;            // optional [B, gnorm_stride]: sum of squares of each bag gradient
  int gnorm_stride;
  int B, D, grad_bf16;
  const float* psw;
  float lr, eps;
  int optimizer;                 // 0 = SGD, 1 = row-wise Adagrad
  long long total_rows;
  unsigned long long* status;
  const int* nnz_dev;            // optional: the live number of occurrences (<= nnz) as counted on the device
  rs::FlagWait wait;             // optional: wait for the peers' gradient pushes first
};

__device__ __forceinline__ long long live_nnz(const EmbBwdArgs& a) {
  if (a.nnz_dev == nullptr) return a.nnz;
  const long long n = *reinterpret_cast<const volatile int*>(a.nnz_dev);
  return n < a.nnz ? n : a.nnz;
}

constexpr int kStateMax = 1024;  // occurrences a CTA of the state pass folds
constexpr int kApplyThreads = 512;   // threads of an apply CTA (128 in small batches) ...
constexpr int kApplyPer = 2;     // ... and the occurrences each of them takes at most
constexpr int kApplyMax = kApplyThreads * kApplyPer;

// Sample and table of occurrence i.  32-bit arithmetic wherever the bag number allows it: a 64-bit division costs more
// than the rest of the address computation.
__device__ __forceinline__ void bag_of(const EmbBwdArgs& a, long long i, int& t, int& b) {
  if (a.occ2bag) {
    const unsigned bag = static_cast<unsigned>(a.occ2bag[i]);
    t = static_cast<int>(bag / static_cast<unsigned>(a.B));
    b = static_cast<int>(bag - static_cast<unsigned>(t) * static_cast<unsigned>(a.B));
  } else if (i < a.B) {
    t = 0;
    b = static_cast<int>(i);
  } else {
    t = static_cast<int>(i / a.B);
    b = static_cast<int>(i % a.B);
  }
}

// Pass 1 of row-wise Adagrad: state[row] += w^2 * |g_bag|^2 / D for every occurrence.
// A CTA folds up to 1,024 occurrences before it touches the state: the lanes of a warp that hold the same row add up in
// registers, one lane per row and warp adds to a shared-memory hash, and one global atomic per distinct row of the CTA
// follows.  Without the first fold the float adds in shared memory, compare-and-swap loops, are serialised by the hot rows of
// a skewed id stream (49 us for 1.70 M occurrences at Zipf 1.2); without the second the global atomics on the hottest row are
// (33 us for 262,144 occurrences at Zipf 1.1), and its sum becomes a chain of thousands of fp32 roundings.  With both: 36 and
// 13 us.
struct StateFold {
  unsigned long long key[2 * kStateMax];
  float val[2 * kStateMax];
};
__device__ __forceinline__ void state_fold_clear(StateFold& f, int slots) {
  for (int s = threadIdx.x; s < slots; s += blockDim.x) {
    f.key[s] = ~0ull;
    f.val[s] = 0.f;
  }
  __syncthreads();
}
// One value per lane and round of a warp, summed over equal rows and added to the fold; row < 0: nothing to add.
// `narrow`: rows fit into 32 bits (the match of 64-bit values costs twice as much).
__device__ __forceinline__ void state_fold_insert(StateFold& f, int slots, long long row, float v);
template <int R>
__device__ __forceinline__ void state_fold_add(StateFold& f, int slots, const long long (&row)[R], float (&v)[R], bool narrow) {
  unsigned peers[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    peers[r] = narrow ? __match_any_sync(0xffffffffu, static_cast<unsigned>(row[r]))
                      : __match_any_sync(0xffffffffu, static_cast<unsigned long long>(row[r]));
  rs::warp_sum_peers(peers, v);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (row[r] >= 0 && static_cast<int>(threadIdx.x & 31) == __ffs(peers[r]) - 1) state_fold_insert(f, slots, row[r], v[r]);
}
__device__ __forceinline__ void state_fold_insert(StateFold& f, int slots, long long row, float v) {
  unsigned s = static_cast<unsigned>(rs::ht_hash(static_cast<unsigned long long>(row))) & (slots - 1);
  for (int p = 0; p < slots; ++p) {
    const unsigned long long prev = atomicCAS(&f.key[s], ~0ull, static_cast<unsigned long long>(row));
    if (prev == ~0ull || prev == static_cast<unsigned long long>(row)) {
      atomicAdd(&f.val[s], v);
      return;
    }
    s = (s + 1) & (slots - 1);
  }
}
__device__ __forceinline__ void state_fold_flush(const StateFold& f, int slots, float* state) {
  __syncthreads();
  for (int s = threadIdx.x; s < slots; s += blockDim.x)
    if (f.key[s] != ~0ull) atomicAdd(&state[f.key[s]], f.val[s]);
}

// With precomputed bag norms: one thread per occurrence, `rounds` (at most 4) of them per thread.
__global__ void __launch_bounds__(256) emb_state_norm_kernel(const EmbBwdArgs a, const int rounds) {
  __shared__ StateFold f;
  const long long nnz = live_nnz(a);
  const long long i0 = static_cast<long long>(blockIdx.x) * 256 * rounds;
  if (i0 >= nnz) return;                       // whole block past the live occurrences
  rs::flag_wait_all(a.wait);
  const int slots = 512 * rounds;
  state_fold_clear(f, slots);
  const float inv_d = 1.f / static_cast<float>(a.D);
  long long row[4];
  float v[4];
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const long long i = i0 + r * 256 + threadIdx.x;
    row[r] = -1;
    v[r] = 0.f;
    if (r < rounds && i < nnz) {
      row[r] = a.row_idx[i];
      if (row[r] < 0 || row[r] >= a.total_rows) {
        row[r] = -1;
      } else {
        int t, b;
        bag_of(a, i, t, b);
        const float w = a.psw ? a.psw[i] : 1.f;
        v[r] = w * w * a.gnorm[static_cast<long long>(b) * a.gnorm_stride + t] * inv_d;
      }
    }
  }
  const bool narrow = a.total_rows < 0xffffffffll;
  if (rounds > 1) {
    state_fold_add(f, slots, row, v, narrow);
  } else {
    const long long row1[1] = {row[0]};
    float v1[1] = {v[0]};
    state_fold_add(f, slots, row1, v1, narrow);
  }
  state_fold_flush(f, slots, a.state);
}

// Without norms a warp takes `opw` consecutive occurrences per round (32, fewer when the batch would leave SMs without work):
// its sub-warps compute the squared norms, U gradient rows of each in flight.
template <int V, int L, int NC, bool BF16>
__global__ void __launch_bounds__(256) emb_state_kernel(const EmbBwdArgs a, const int opw, const int rounds) {
  constexpr int G = 32 / L;
  constexpr int U = V * NC <= 8 ? 4 : 2;
  __shared__ StateFold f;
  const long long nnz = live_nnz(a);
  const long long c0 = static_cast<long long>(blockIdx.x) * 8 * opw * rounds;
  if (c0 >= nnz) return;
  rs::flag_wait_all(a.wait);
  const int slots = 16 * opw * rounds;
  state_fold_clear(f, slots);
  const int lane = threadIdx.x & 31, l = lane & (L - 1), g = lane / L;
  const int nvec = a.D / V;
  for (int rd = 0; rd < rounds; ++rd) {
    const long long i = c0 + (rd * 8 + (threadIdx.x >> 5)) * opw + lane;
    long long row = -1, goff = 0;
    float w = 1.f, v = 0.f;
    if (lane < opw && i < nnz) {
      row = a.row_idx[i];
      if (row < 0 || row >= a.total_rows) {
        row = -1;
      } else {
        int t, b;
        bag_of(a, i, t, b);
        goff = b * a.grad_row_stride + (a.grad_col ? a.grad_col[t] : 0);
        if (a.psw) w = a.psw[i];
      }
    }
    const bool wide = V == 4 || __all_sync(0xffffffffu, (goff & 7) == 0);
    for (int j0 = 0; j0 < opw; j0 += G * U) {
      rs::RawVec<V, BF16> x[U][NC];
      bool on[U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int j = (j0 + u * G + g) & 31;
        const long long go = __shfl_sync(0xffffffffu, goff, j);
        on[u] = __shfl_sync(0xffffffffu, row, j) >= 0 && j0 + u * G + g < opw;
        if (on[u]) {
#pragma unroll
          for (int c = 0; c < NC; ++c) x[u][c].load(a.grad, go + static_cast<long long>(min(l + c * L, nvec - 1)) * V, wide);
        }
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        float sq = 0.f;
        if (on[u]) {
#pragma unroll
          for (int c = 0; c < NC; ++c) {
            if (l + c * L < nvec) {
              const rs::RowVec<V> h = x[u][c].get();
#pragma unroll
              for (int e = 0; e < V; ++e) sq += h.v[e] * h.v[e];
            }
          }
        }
#pragma unroll
        for (int o = L / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
        // occurrence j0 + u * G + k lies in sub-warp k; lane j keeps the norm of occurrence j
        const int k = lane - j0 - u * G;
        const float got = __shfl_sync(0xffffffffu, sq, (k & (G - 1)) * L);
        if (k >= 0 && k < G) v = got;
      }
    }
    const long long row1[1] = {row};
    float v1[1] = {v * (w * w / static_cast<float>(a.D))};
    state_fold_add(f, slots, row1, v1, a.total_rows < 0xffffffffll);
  }
  state_fold_flush(f, slots, a.state);
}

// Apply pass: one CTA per `gs` occurrences (1,024 at most, fewer when that leaves SMs without work).  They are counting-sorted by row
// in shared memory (hash slot -> count -> exclusive scan -> position), so equal rows sit next to each other, together with
// their factor -lr * w / (sqrt(state) + eps): one state read and one root per occurrence, by the thread that owns it, and
// none in the loop over the rows.  Every sub-warp then owns an equal share of the sorted positions, whatever the skew of the
// ids: it streams their gradients with U loads in flight, sums runs of equal rows in registers and issues one vector
// atomic per unit and run.  A row that straddles warps or groups simply receives several atomics; the larger the group the
// fewer of them meet on the hot rows, which the L2 takes one after another.
// Bound by latency (sort, then gradients) and by those atomics: 16-byte bf16 loads by half a warp per 128-float row.  The
// form before it (256 occurrences, a warp per row, state read and root inside the loop, 32 % of the warps resident) took
// 278 us for 1.70 M occurrences x 128 at Zipf 1.2; this one 141 us (436 MB of gradients: 66 us), 231 us with groups of 256.
template <int V, int L, int NC, bool BF16>
__global__ void __launch_bounds__(kApplyThreads) emb_apply_kernel(const EmbBwdArgs a, const int gs) {
  constexpr int kPer = kApplyPer;
  const int threads = blockDim.x, warps = threads >> 5;
  // the hash is dead once the positions are known; the sorted arrays take its place
  __shared__ __align__(16) unsigned char s_mem[2 * kApplyMax * 12 > kApplyMax * 20 ? 2 * kApplyMax * 12 : kApplyMax * 20];
  __shared__ int s_warp_sum[kApplyThreads / 32];
  long long* const s_key = reinterpret_cast<long long*>(s_mem);                        // [2 gs]
  int* const s_cnt = reinterpret_cast<int*>(s_mem + 2 * kApplyMax * 8);                // [2 gs] occurrences per slot, then offsets
  long long* const s_goff = reinterpret_cast<long long*>(s_mem);                       // sorted: gradient offset
  long long* const s_row = reinterpret_cast<long long*>(s_mem + kApplyMax * 8);        // sorted: row
  float* const s_coef = reinterpret_cast<float*>(s_mem + kApplyMax * 16);              // sorted: factor of the gradient

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const long long g0 = static_cast<long long>(blockIdx.x) * gs;
  const long long nnz = live_nnz(a);
  if (g0 >= nnz) return;                       // whole group past the live occurrences
  rs::flag_wait_all(a.wait);
  const int slots = 2 * gs;
  for (int s = tid; s < slots; s += threads) {
    s_key[s] = -1;
    s_cnt[s] = 0;
  }
  long long row[kPer], goff[kPer];
  float coef[kPer];
  bool narrow = false;
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    const int at = q * threads + tid;
    row[q] = -1;
    goff[q] = 0;
    coef[q] = -a.lr;
    if (at < gs && g0 + at < nnz) {
      row[q] = a.row_idx[g0 + at];
      if (row[q] >= a.total_rows) {
        if (a.status) atomicOr(a.status, (unsigned long long)RS_DEV_OOB_ROW);
        row[q] = -1;
      }
    }
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    if (row[q] < 0) continue;
    const long long occ = g0 + q * threads + tid;
    int t, b;
    bag_of(a, occ, t, b);
    goff[q] = b * a.grad_row_stride + (a.grad_col ? a.grad_col[t] : 0);
    if (a.optimizer == 1) coef[q] = -a.lr / (sqrtf(__ldcv(&a.state[row[q]])) + a.eps);
    if (a.psw) coef[q] *= a.psw[occ];
    narrow = narrow || (goff[q] & 7) != 0;
  }
  const bool wide = !__syncthreads_or(V == 8 && narrow);   // (also: the slots are cleared)
  int slot[kPer], rank[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    slot[q] = -1;
    rank[q] = 0;
    if (row[q] < 0) continue;
    unsigned s = static_cast<unsigned>(rs::ht_hash(static_cast<unsigned long long>(row[q]))) & (slots - 1);
    for (int p = 0; p < slots; ++p) {
      const long long prev = static_cast<long long>(atomicCAS(reinterpret_cast<unsigned long long*>(&s_key[s]),
                                                               static_cast<unsigned long long>(-1ll),
                                                               static_cast<unsigned long long>(row[q])));
      if (prev == -1 || prev == row[q]) {
        slot[q] = static_cast<int>(s);
        rank[q] = atomicAdd(&s_cnt[s], 1);
        break;
      }
      s = (s + 1) & (slots - 1);
    }
  }
  __syncthreads();
  // exclusive scan of the slot counts: 2 * kPer neighbouring slots per thread, warp shuffles, then the warp totals
  int total = 0;
  {
    constexpr int kScan = 2 * kPer;
    int c[kScan], sum = 0;
#pragma unroll
    for (int q = 0; q < kScan; ++q) {
      c[q] = kScan * tid + q < slots ? s_cnt[kScan * tid + q] : 0;
      sum += c[q];
    }
    int incl = sum;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp_sum[warp] = incl;
    __syncthreads();
    int excl = incl - sum;
    for (int q = 0; q < warps; ++q) {
      excl += q < warp ? s_warp_sum[q] : 0;
      total += s_warp_sum[q];
    }
#pragma unroll
    for (int q = 0; q < kScan; ++q) {
      if (kScan * tid + q < slots) s_cnt[kScan * tid + q] = excl;
      excl += c[q];
    }
  }
  __syncthreads();
  int pos[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) pos[q] = slot[q] >= 0 ? s_cnt[slot[q]] + rank[q] : -1;
  __syncthreads();                              // the hash has been read for the last time
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
    if (pos[q] < 0) continue;
    s_goff[pos[q]] = goff[q];
    s_row[pos[q]] = row[q];
    s_coef[pos[q]] = coef[q];
  }
  __syncthreads();

  constexpr int G = 32 / L;
  constexpr int U = V * NC <= 8 ? 4 : 2;
  const int l = lane & (L - 1);
  const int nvec = a.D / V;
  const int share = gs / (warps * G);
  const int p_begin = (warp * G + lane / L) * share;
  const int p_end = min(total, p_begin + share);
  long long cur = -1;
  rs::RowVec<V> acc[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) rs::row_zero(acc[c]);

  auto flush = [&]() {
    if (cur < 0) return;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int v = l + c * L;
      if (v < nvec) rs::row_atomic_add(a.weight + cur * a.D + static_cast<long long>(v) * V, acc[c]);
      rs::row_zero(acc[c]);
    }
  };

  for (int p0 = p_begin; p0 < p_end; p0 += U) {
    rs::RawVec<V, BF16> x[U][NC];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const long long go = s_goff[min(p0 + u, p_end - 1)];   // past the end: re-read the last valid position, ignored below
#pragma unroll
      for (int c = 0; c < NC; ++c) x[u][c].load(a.grad, go + static_cast<long long>(min(l + c * L, nvec - 1)) * V, wide);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (p0 + u >= p_end) break;
      const long long r = s_row[p0 + u];
      if (r != cur) {
        flush();
        cur = r;
      }
      const float k = s_coef[p0 + u];
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        const rs::RowVec<V> h = x[u][c].get();
#pragma unroll
        for (int e = 0; e < V; ++e) acc[c].v[e] = fmaf(k, h.v[e], acc[c].v[e]);
      }
    }
  }
  if (G > 1) {
    // A hot row fills whole sub-warps: equal rows at the ends of neighbouring sub-warps are added up towards the first of
    // them, which alone sends.
    __syncwarp();
#pragma unroll
    for (int o = 1; o < G; o <<= 1) {
      const long long theirs = __shfl_down_sync(0xffffffffu, cur, o * L);
      const bool join = lane + o * L < 32 && cur >= 0 && theirs == cur;
#pragma unroll
      for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int e = 0; e < V; ++e) {
          const float y = __shfl_down_sync(0xffffffffu, acc[c].v[e], o * L);
          if (join) acc[c].v[e] += y;
        }
    }
    const long long before = __shfl_up_sync(0xffffffffu, cur, L);
    if (lane >= L && before == cur) cur = -1;
  }
  flush();
}

// Plain row gather / scatter used by the PS get / put verbs: out[i] = W[rows[i]] (zeros when rows[i] < 0).
__global__ void rows_gather_kernel(const float* __restrict__ w, const long long* __restrict__ rows, long long n, int D,
                                   float* __restrict__ out) {
  const long long i = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const int lane = threadIdx.x & 31;
  const long long r = rows[i];
  for (int v = lane; v < (D >> 2); v += 32) {
    const float4 x = r >= 0 ? __ldg(reinterpret_cast<const float4*>(w + r * D) + v) : make_float4(0.f, 0.f, 0.f, 0.f);
    *(reinterpret_cast<float4*>(out + i * D) + v) = x;
  }
}
__global__ void rows_scatter_kernel(float* __restrict__ w, const long long* __restrict__ rows, long long n, int D,
                                    const float* __restrict__ in) {
  const long long i = static_cast<long long>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= n) return;
  const int lane = threadIdx.x & 31;
  const long long r = rows[i];
  if (r < 0) return;
  for (int v = lane; v < (D >> 2); v += 32)
    *(reinterpret_cast<float4*>(w + r * D) + v) = __ldg(reinterpret_cast<const float4*>(in + i * D) + v);
}

}  // namespace

namespace {
int launch_emb_fwd(const EmbFwdArgs& a, cudaStream_t stream) {
  if (a.T == 0 || a.B == 0) return RS_OK;
  // Four warps per CTA: at 64 registers per thread such a CTA still fits on an SM beside one persistent GEMM CTA, so the
  // lookup and its NVLink pushes really run at the same time as the MLP that is launched beside them.
  static const int wpb = [] { const char* e = getenv("RECSTORE_EMB_FWD_WARPS"); return (e && e[0] == '8') ? 8 : 4; }();
  // RECSTORE_EMB_FWD_CTAS_PER_SM=c (0 = no limit, the default): at most c CTAs per SM, the warps looping over the bags.
  // The hardware hands out the CTAs of a later kernel only once every CTA of the earlier one has been placed, so a lookup
  // with thousands of CTAs holds back the GEMMs launched beside it on another stream until its last wave; a grid that is
  // resident as a whole does not.
  static const int per_sm = [] { const char* e = getenv("RECSTORE_EMB_FWD_CTAS_PER_SM"); return e ? atoi(e) : 0; }();
  const long long bags = static_cast<long long>(a.T) * a.B;
  if (a.counts || a.occ_cursor || a.id_div > 1 || a.wait.my_flags || bags >= (1ll << 31)) {
    const long long nblocks = static_cast<long long>(a.T) * ((a.B + 31) / 32);
    long long grid = (nblocks + wpb - 1) / wpb;
    if (per_sm > 0 && grid > 148ll * per_sm) grid = 148ll * per_sm;
    RS_REQUIRE(grid < (1ll << 31), "rs_emb_forward: too many bags");
    if (a.D <= 128) emb_fwd_sharded_kernel<1><<<static_cast<unsigned>(grid), wpb * 32, 0, stream>>>(a);
    else if (a.D <= 256) emb_fwd_sharded_kernel<2><<<static_cast<unsigned>(grid), wpb * 32, 0, stream>>>(a);
    else emb_fwd_sharded_kernel<4><<<static_cast<unsigned>(grid), wpb * 32, 0, stream>>>(a);
    RS_LAUNCH_CHECK();
    return RS_OK;
  }
  // How many bags share a sub-warp is settled on the device (it depends on the ids per bag); the host caps it so that a small
  // batch still gives every SM sixteen warps, and sizes the grid for one-id bags: longer ones mean more tasks, over which
  // the warps loop.
  auto launch = [&](auto kern, int L) {
    const int G = 32 / L;
    int cap = L;
    while (cap > 1 && bags / cap < 148ll * 16 * G) cap >>= 1;
    const long long tasks = static_cast<long long>(a.T) * ((a.B + cap - 1) / cap);
    long long grid = (tasks + wpb * G - 1) / (wpb * G);
    if (per_sm > 0 && grid > 148ll * per_sm) grid = 148ll * per_sm;
    kern<<<static_cast<unsigned>(grid), wpb * 32, 0, stream>>>(a, cap);
  };
#define RS_LAUNCH_POOL(V, L, NC) launch(emb_pool_kernel<V, L, NC>, L)
  RS_ROW_DISPATCH(rs::row_wide(a.weight, a.D), a.D, RS_LAUNCH_POOL);
#undef RS_LAUNCH_POOL
  RS_LAUNCH_CHECK();
  return RS_OK;
}
}  // namespace

RS_API int rs_emb_forward(const float* weight, const long long* table_base, const long long* table_rows,
                          const long long* indices, const long long* offsets, const int* hotness,
                          const long long* hot_base, const float* psw, int T, int B, int D, int B_local,
                          void* const* dst, long long dst_row_stride, const int* dst_col, int out_bf16,
                          long long* row_idx, int* occ2bag, const rs::HashTableView* ht,
                          unsigned long long* status, cudaStream_t stream) {
  RS_REQUIRE(weight && table_base && table_rows && indices && dst && dst_col, "rs_emb_forward: null argument");
  RS_REQUIRE(offsets || (hotness && hot_base), "rs_emb_forward: need offsets or fixed hotness");
  RS_REQUIRE(D % 4 == 0 && D > 0 && D <= 128 * kMaxChunks, "rs_emb_forward: D=%d must be a multiple of 4, <= 512", D);
  RS_REQUIRE(T >= 0 && B >= 0 && B_local > 0, "rs_emb_forward: bad sizes");
  EmbFwdArgs a;
  memset(&a, 0, sizeof(a));
  a.weight = weight; a.table_base = table_base; a.table_rows = table_rows; a.indices = indices;
  a.offsets = offsets; a.hotness = hotness; a.hot_base = hot_base; a.psw = psw;
  a.T = T; a.B = B; a.D = D; a.B_local = B_local; a.dst = dst; a.dst_row_stride = dst_row_stride;
  a.dst_col = dst_col; a.out_bf16 = out_bf16; a.row_idx = row_idx; a.occ2bag = occ2bag;
  a.use_hash = ht != nullptr;
  if (ht) a.ht = *ht;
  a.status = status;
  a.id_div = 1; a.id_rem = 0;
  return launch_emb_fwd(a, stream);
}

// The same lookup with the extras of the multi-GPU engine.
//   counts / id_div / id_rem / occ_cursor: bags of a row-sharded table (see EmbFwdArgs); occ_cursor must be zero on entry.
//   wait_flags ... wait_channel:  each warp first waits (bounded) for the flag of the rank its bags come from.
//   sig_flags_of ... sig_channel: when the whole grid is done its last block publishes this rank's next epoch on the
//                                  channel to every rank (data then flag, one launch).  sig_done: a zeroed device counter.
RS_API int rs_emb_forward_ex(const float* weight, const long long* table_base, const long long* table_rows,
                             const long long* indices, const int* hotness, const long long* hot_base, int T, int B, int D,
                             int B_local, void* const* dst, long long dst_row_stride, const int* dst_col, int out_bf16,
                             long long* row_idx, int* occ2bag, unsigned long long* status,
                             const int* counts, int id_div, int id_rem, int* occ_cursor,
                             const void* wait_flags, const unsigned* counters, unsigned long long timeout_ns, int wait_channel,
                             void* const* sig_flags_of, unsigned* sig_done, int sig_channel, int world, int me,
                             cudaStream_t stream) {
  RS_REQUIRE(weight && table_base && table_rows && indices && dst && dst_col && hotness && hot_base, "rs_emb_forward_ex: null argument");
  RS_REQUIRE(D % 4 == 0 && D > 0 && D <= 128 * kMaxChunks, "rs_emb_forward_ex: D=%d must be a multiple of 4, <= 512", D);
  RS_REQUIRE(T >= 0 && B >= 0 && B_local > 0 && id_div >= 1 && id_rem >= 0 && id_rem < id_div, "rs_emb_forward_ex: bad sizes");
  RS_REQUIRE(world >= 1 && world <= 32 && me >= 0 && me < world, "rs_emb_forward_ex: bad rank / world");
  RS_REQUIRE((!wait_flags && !sig_flags_of) || counters, "rs_emb_forward_ex: flags need the epoch counters");
  RS_REQUIRE(!sig_flags_of || sig_done, "rs_emb_forward_ex: a signal needs its done counter");
  EmbFwdArgs a;
  memset(&a, 0, sizeof(a));
  a.weight = weight; a.table_base = table_base; a.table_rows = table_rows; a.indices = indices;
  a.hotness = hotness; a.hot_base = hot_base;
  a.T = T; a.B = B; a.D = D; a.B_local = B_local; a.dst = dst; a.dst_row_stride = dst_row_stride;
  a.dst_col = dst_col; a.out_bf16 = out_bf16; a.row_idx = row_idx; a.occ2bag = occ2bag;
  a.status = status;
  a.counts = counts; a.id_div = id_div; a.id_rem = id_rem; a.occ_cursor = occ_cursor;
  a.wait.my_flags = reinterpret_cast<const uint32_t*>(wait_flags); a.wait.sig_counters = counters;
  a.wait.timeout_ns = timeout_ns; a.wait.status = status; a.wait.world = world; a.wait.channel = wait_channel;
  a.sig.flags_of = reinterpret_cast<uint32_t* const*>(sig_flags_of); a.sig.sig_counters = const_cast<unsigned*>(counters);
  a.sig.done = sig_done; a.sig.world = world; a.sig.me = me; a.sig.channel = sig_channel;
  if ((T == 0 || B == 0) && sig_flags_of) return rs::set_error(RS_ERR_INVALID, "rs_emb_forward_ex: an empty lookup cannot carry the signal");
  return launch_emb_fwd(a, stream);
}

// optimizer: 0 SGD (one launch), 1 row-wise Adagrad (two launches: state pass, apply pass).
// gnorm (optional): precomputed sum of squares of every bag gradient, [B, gnorm_stride] fp32 indexed
// [sample, local table]; saves the state pass a full read of the gradients.
namespace {
int emb_backward_impl(float* weight, float* state, long long total_rows, const long long* row_idx,
                      const int* occ2bag, long long nnz, const void* grad, const int* grad_col,
                      long long grad_row_stride, const float* gnorm, int gnorm_stride, int B, int D,
                      int grad_bf16, const float* psw, float lr, float eps, int optimizer,
                      unsigned long long* status, const int* nnz_dev, const rs::FlagWait& wait, cudaStream_t stream);
}  // namespace

RS_API int rs_emb_backward(float* weight, float* state, long long total_rows, const long long* row_idx,
                           const int* occ2bag, long long nnz, const void* grad, const int* grad_col,
                           long long grad_row_stride, const float* gnorm, int gnorm_stride, int B, int D,
                           int grad_bf16, const float* psw, float lr, float eps, int optimizer,
                           unsigned long long* status, cudaStream_t stream) {
  rs::FlagWait w;
  memset(&w, 0, sizeof(w));
  return emb_backward_impl(weight, state, total_rows, row_idx, occ2bag, nnz, grad, grad_col, grad_row_stride, gnorm, gnorm_stride,
                           B, D, grad_bf16, psw, lr, eps, optimizer, status, nullptr, w, stream);
}

// The same update with the extras of the multi-GPU engine: nnz_dev (optional) is the live occurrence count on the device
// (nnz is then the capacity of the lists and sizes the grids); wait_flags (optional) makes the first kernel wait, bounded,
// until every rank's flag on `wait_channel` has reached this rank's own epoch (the peers' gradient pushes have landed).
RS_API int rs_emb_backward_ex(float* weight, float* state, long long total_rows, const long long* row_idx,
                              const int* occ2bag, long long nnz, const void* grad, const int* grad_col,
                              long long grad_row_stride, const float* gnorm, int gnorm_stride, int B, int D,
                              int grad_bf16, float lr, float eps, int optimizer, unsigned long long* status,
                              const int* nnz_dev, const void* wait_flags, const unsigned* counters, unsigned long long timeout_ns,
                              int wait_channel, int world, cudaStream_t stream) {
  rs::FlagWait w;
  memset(&w, 0, sizeof(w));
  w.my_flags = reinterpret_cast<const uint32_t*>(wait_flags); w.sig_counters = counters; w.timeout_ns = timeout_ns;
  w.status = status; w.world = world; w.channel = wait_channel;
  RS_REQUIRE(!wait_flags || (counters && world >= 1 && world <= 32), "rs_emb_backward_ex: bad flag arguments");
  return emb_backward_impl(weight, state, total_rows, row_idx, occ2bag, nnz, grad, grad_col, grad_row_stride, gnorm, gnorm_stride,
                           B, D, grad_bf16, nullptr, lr, eps, optimizer, status, nnz_dev, w, stream);
}

namespace {
int emb_backward_impl(float* weight, float* state, long long total_rows, const long long* row_idx,
                      const int* occ2bag, long long nnz, const void* grad, const int* grad_col,
                      long long grad_row_stride, const float* gnorm, int gnorm_stride, int B, int D,
                      int grad_bf16, const float* psw, float lr, float eps, int optimizer,
                      unsigned long long* status, const int* nnz_dev, const rs::FlagWait& wait, cudaStream_t stream) {
  RS_REQUIRE(weight && row_idx && grad, "rs_emb_backward: null argument");
  RS_REQUIRE(optimizer == 0 || (optimizer == 1 && state), "rs_emb_backward: row-wise Adagrad needs a state tensor");
  RS_REQUIRE(D % 4 == 0 && D > 0 && D <= 128 * kMaxChunks, "rs_emb_backward: D=%d must be a multiple of 4, <= 512", D);
  RS_REQUIRE(B > 0, "rs_emb_backward: B must be positive");
  if (nnz == 0) return RS_OK;
  EmbBwdArgs a;
  a.weight = weight; a.state = state; a.row_idx = row_idx; a.occ2bag = occ2bag; a.nnz = nnz; a.grad = grad;
  a.grad_col = grad_col; a.grad_row_stride = grad_row_stride; a.gnorm = gnorm; a.gnorm_stride = gnorm_stride;
  a.B = B; a.D = D; a.grad_bf16 = grad_bf16;
  a.psw = psw; a.lr = lr; a.eps = eps; a.optimizer = optimizer; a.total_rows = total_rows; a.status = status;
  a.nnz_dev = nnz_dev; a.wait = wait;
  RS_REQUIRE(nnz < (1ll << 36), "rs_emb_backward: too many occurrences");
  // 8-float units need rows and gradients that start on their boundaries (the offsets inside the gradient buffer are
  // looked at in the kernel, they are device values).
  const bool wide = rs::row_wide(weight, D) && (reinterpret_cast<uintptr_t>(grad) & (grad_bf16 ? 15 : 31)) == 0;
  if (optimizer == 1) {
    // As many occurrences per CTA as keep every SM busy, 1,024 at most: the fewer atomics a hot row gets, the more exact its sum.
    if (gnorm) {
      const int rounds = nnz >= 1024 * 148 ? 4 : nnz >= 512 * 148 ? 2 : 1;
      emb_state_norm_kernel<<<static_cast<unsigned>((nnz + 256 * rounds - 1) / (256 * rounds)), 256, 0, stream>>>(a, rounds);
    } else {
      auto launch = [&](auto kern, int L) {
        int opw = 32, rounds = nnz >= 1024 * 148 ? 4 : nnz >= 512 * 148 ? 2 : 1;
        while (opw > 32 / L && nnz < 8ll * opw * 296) opw >>= 1;
        kern<<<static_cast<unsigned>((nnz + 8 * opw * rounds - 1) / (8 * opw * rounds)), 256, 0, stream>>>(a, opw, rounds);
      };
#define RS_LAUNCH_STATE(V, L, NC)                                 \
  do {                                                            \
    if (grad_bf16) launch(emb_state_kernel<V, L, NC, true>, L);   \
    else launch(emb_state_kernel<V, L, NC, false>, L);            \
  } while (0)
      RS_ROW_DISPATCH(wide, D, RS_LAUNCH_STATE);
#undef RS_LAUNCH_STATE
    }
    RS_LAUNCH_CHECK();
  }
  // The largest group that still gives every SM two CTAs, never less than one position per sub-warp.  CTAs of 512 threads
  // once a batch fills them; below, the barriers of the sort cost more than the warps gain (3,072 rows of 400: 15.5 us).
  auto launch = [&](auto kern, int L) {
    const int threads = nnz >= 296ll * kApplyThreads ? kApplyThreads : 128;
    // bf16 gradients come from the DLRM engine, which runs this pass beside the GEMMs of the bottom MLP: a GEMM CTA needs an SM
    // for itself, so a small batch must not put a CTA on each (600 x 10 occurrences: 375 CTAs made the step 3 us longer
    // than 24 did, although the pass itself is 4 us shorter).
    const int least = grad_bf16 ? 128 : (threads / 32) * (32 / L);
    int gs = threads * kApplyPer;
    while (gs > least && nnz < 296ll * gs) gs >>= 1;
    kern<<<static_cast<unsigned>((nnz + gs - 1) / gs), threads, 0, stream>>>(a, gs);
  };
#define RS_LAUNCH_APPLY(V, L, NC)                                 \
  do {                                                            \
    if (grad_bf16) launch(emb_apply_kernel<V, L, NC, true>, L);   \
    else launch(emb_apply_kernel<V, L, NC, false>, L);            \
  } while (0)
  RS_ROW_DISPATCH(wide, D, RS_LAUNCH_APPLY);
#undef RS_LAUNCH_APPLY
  RS_LAUNCH_CHECK();
  return RS_OK;
}

}  // namespace

RS_API int rs_rows_gather(const float* weight, const long long* rows, long long n, int D, float* out,
                          cudaStream_t stream) {
  RS_REQUIRE(weight && rows && out && D % 4 == 0, "rs_rows_gather: bad argument");
  if (n == 0) return RS_OK;
  rows_gather_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(weight, rows, n, D, out);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
RS_API int rs_rows_scatter(float* weight, const long long* rows, long long n, int D, const float* in,
                           cudaStream_t stream) {
  RS_REQUIRE(weight && rows && in && D % 4 == 0, "rs_rows_scatter: bad argument");
  if (n == 0) return RS_OK;
  rows_scatter_kernel<<<static_cast<unsigned>((n + 7) / 8), 256, 0, stream>>>(weight, rows, n, D, in);
  RS_LAUNCH_CHECK();
  return RS_OK;
}
