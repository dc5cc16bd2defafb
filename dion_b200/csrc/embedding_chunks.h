// Index arithmetic of the embedding backward (embedding_ops.cu), in 32-bit integers up to
// 2^31 - 257 positions: no sum here may pass 2^31.
#pragma once

#ifdef __CUDACC__
#define DION_HD __host__ __device__ __forceinline__
#else
#define DION_HD static inline
#endif

namespace dion {

constexpr int kEmbChunk = 64;        // sorted positions per chunk, doubled until 1024 chunks suffice

DION_HD int emb_chunk(long long n) {
  long long chunk = kEmbChunk;
  while ((n + chunk - 1) / chunk > 1024) chunk *= 2;
  return (int)chunk;
}
DION_HD int emb_num_chunks(long long n, int chunk) { return (int)((n + chunk - 1) / chunk); }

// Chunk c is [c * chunk, emb_chunk_end(c * chunk, chunk, n)).
DION_HD int emb_chunk_end(int p0, int chunk, int n) { return n - p0 > chunk ? p0 + chunk : n; }

// Middle of [lo, hi) for the binary search.
DION_HD int emb_mid(int lo, int hi) { return lo + ((hi - lo) >> 1); }

}  // namespace dion
