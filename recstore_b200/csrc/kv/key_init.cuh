// Initial value of a row that the hash-table shard sees for the first time: uniform in [-scale, scale), a function of the key
// and the column only, so a table does not depend on the order in which its keys arrive.
#pragma once
#include "kv/hash_table.cuh"

namespace rs {
__device__ __forceinline__ float key_init_value(unsigned long long key, int col, float scale) {
  const unsigned long long h = ht_hash(key * 0x9E3779B97F4A7C15ull + static_cast<unsigned long long>(col) + 1ull);
  return (static_cast<float>(h >> 40) * (1.0f / 16777216.0f) * 2.f - 1.f) * scale;
}
}  // namespace rs
