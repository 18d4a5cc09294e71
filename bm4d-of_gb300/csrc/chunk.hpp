// chunk.hpp -- sizes of the chunks of groups that the filter and the aggregation
// take at a time (host arithmetic of runtime.cu).
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace bm4dof {

constexpr size_t kChunkBytes = (size_t)2 << 30;        // 16 GiB gave the same times and held 14 GiB more
constexpr size_t kBatchChunkBytes = (size_t)512 << 20; // per sequence of a batch

// Bytes that a chunk's terms, weights and bin lists may take in a single run.
//   env_mb   BM4DOF_SLOT_MB, in MiB (0: not set): a fifth of it.  Callers tuned the
//            value with 1.3 to 2.8 times the bytes a group and 10 launches a chunk
//            (6 now); the golden cases' chunk test holds both.
//   usable   device memory that the context holds or could take (0: unknown): a 16th
//   limit    the context's memory limit (0: none): a quarter, or, where the other
//            buffers leave no room for that (tight), a 32nd
inline size_t chunk_bytes(double env_mb, size_t usable, size_t limit, bool tight)
{
	size_t b = kChunkBytes;
	if (env_mb > 0.0) b = (size_t)(env_mb * 1048576.0) / 5;
	if (usable) b = std::min(b, usable / 16);
	if (limit) b = std::min(b, limit / (tight ? 32 : 4));
	return b;
}

// Groups per chunk: at least one, at most all G; slot numbers and positions in the
// bins' lists (np * entries a group, entries per member) fit 32 bits.
inline long long chunk_groups(size_t bytes, size_t per_group, unsigned np, unsigned entries, long long G)
{
	long long n = (long long)(bytes / per_group);
	n = std::min(n, (1ll << 28) / np);
	n = std::min(n, (long long)UINT32_MAX / ((long long)np * entries));
	return std::max(1ll, std::min(n, G));
}

}  // namespace bm4dof
