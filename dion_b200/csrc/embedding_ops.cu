// Backward of the token embedding for sm_100a: the weight gradient GW[v] = sum of the rows of DY
// whose token id is v, written exactly once per row (zeros where the id does not occur), with a
// result that does not depend on scheduling.  It replaces what the reference gets from the stock
// dense embedding backward under its compiler (models/gpt_model.py:298-307: `nn.Embedding`), which
// zero-fills the [V, C] gradient and scatters into it with atomics.
//
// Three launches and the sort, no host synchronisation, scratch supplied by the caller:
//   1. keys[i] = id (V for ids outside [0, V)), vals[i] = i as 32-bit integers;
//   2. a stable radix sort of the (key, position) pairs over just the bits an id needs
//      (CUB's device-wide sort; 16 bits for a 50 K vocabulary instead of the 64 of a sort of the
//      id tensor itself), so that every id's positions are consecutive and ascending;
//   3. starts[v] = first sorted index whose key is >= v, one thread per v (binary search) - the
//      run of row v is [starts[v], starts[v+1]);
//      In the same launch one block per chunk of sorted positions (64 up to 65536 tokens) sums the
//      parts of runs longer than a chunk that lie in it.  Such a run covers the first or the last
//      position of every chunk it meets, so a chunk has two slots; the block counts the run's
//      positions on either side itself, one read per thread (bisecting for its ends: 134 instead of
//      114 us for 131072 skewed tokens and 512 rows of 256; as a launch of its own behind the
//      starts: 121, and 21 instead of 17 us for 512 tokens);
//   4. one warp per row of GW sums the run in fp32 in position order, or its parts in chunk order,
//      or writes zeros.
// Real token streams have ids that occur thousands of times per batch, and vocabularies are often
// ordered by frequency, so that the longest runs are neighbours: with each of them summed by the
// block of its row, 32768 tokens of rank-one-over-frequency text (768 columns) took 919 us, all but
// a few of them in the first block.
#include <cub/device/device_radix_sort.cuh>

#include "common.cuh"
#include "embedding_chunks.h"

namespace dion {

enum : int { DT_F32 = 0, DT_BF16 = 1 };

// 8 consecutive elements as floats (callers guarantee 8-element alignment).
__device__ __forceinline__ void emb_load8(const void* p, int dt, long long i, float (&v)[8]) {
  if (dt == DT_F32) {
    const float4* q = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(p) + i);
    const float4 a = q[0], b = q[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else {
    const uint4 u = *reinterpret_cast<const uint4*>(reinterpret_cast<const __nv_bfloat16*>(p) + i);
    const float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z),
                 d = unpack_bf16x2(u.w);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y; v[4] = c.x; v[5] = c.y; v[6] = d.x; v[7] = d.y;
  }
}

__global__ void __launch_bounds__(256)
emb_keys_kernel(const long long* __restrict__ ids, int* __restrict__ keys, int* __restrict__ vals,
                int n, int V) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i >= n) return;
  const long long t = ids[i];
  keys[i] = (t >= 0 && t < V) ? static_cast<int>(t) : V;
  vals[i] = i;
}

constexpr int kEmbWarps = 8;

// acc += the rows perm[j] of DY for j in [j0, j1), columns [c8*8, c8*8+8), four loads in flight.
__device__ __forceinline__ void emb_sum_run(const void* __restrict__ DY, int dy_dt,
                                            const int* __restrict__ perm, int j0, int j1, int C,
                                            int c8, float (&acc)[8]) {
  int j = j0;
  for (; j + 4 <= j1; j += 4) {
    float v[4][8];
#pragma unroll
    for (int u = 0; u < 4; ++u) emb_load8(DY, dy_dt, (long long)perm[j + u] * C + c8 * 8, v[u]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int e = 0; e < 8; ++e) acc[e] += v[u][e];
  }
  for (; j < j1; ++j) {
    float v[8];
    emb_load8(DY, dy_dt, (long long)perm[j] * C + c8 * 8, v);
#pragma unroll
    for (int e = 0; e < 8; ++e) acc[e] += v[e];
  }
}

// The first `chunks` blocks: part[2 * c + slot][C] = sum over the positions of chunk c that belong to
// the long run covering its first (slot 0) or its last position (slot 1, if that is another run).
// The others: starts[v] for a row v per thread.
__global__ void __launch_bounds__(kEmbWarps * 32)
emb_starts_parts_kernel(const int* __restrict__ sorted, int* __restrict__ starts,
                        const int* __restrict__ perm, const void* __restrict__ DY, int dy_dt,
                        float* __restrict__ part, int n, int C, int V, int chunk, int chunks) {
  extern __shared__ __align__(16) float emb_part[];          // [kEmbWarps][C]
  if ((int)blockIdx.x >= chunks) {
    const int v = ((int)blockIdx.x - chunks) * (kEmbWarps * 32) + threadIdx.x;
    if (v > V) return;
    int lo = 0, hi = n;                      // first index with sorted[idx] >= v
    while (lo < hi) {
      const int mid = emb_mid(lo, hi);
      if (sorted[mid] < v) lo = mid + 1; else hi = mid;
    }
    starts[v] = lo;
    return;
  }
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int p0 = blockIdx.x * chunk, p1 = emb_chunk_end(p0, chunk, n);
  const int first = sorted[p0], last = sorted[p1 - 1];
  for (int slot = 0; slot < 2; ++slot) {
    const int v = slot == 0 ? first : last;
    if (v >= V || (slot == 1 && first == last)) continue;    // ids outside the table sort last
    // The run's positions among the `chunk` on either side of the one it covers, and in this chunk.
    const int p = slot == 0 ? p0 : p1 - 1;
    const int from = p > chunk ? p - chunk : 0, to = n - p > chunk ? p + chunk : n - 1;
    int near = 0, inside = 0;
    for (int i0 = from; i0 <= to; i0 += kEmbWarps * 32) {
      const int i = i0 + (int)threadIdx.x;
      const bool here = i <= to && sorted[i] == v;
      near += __syncthreads_count(here);
      inside += __syncthreads_count(here && i >= p0 && i < p1);
    }
    if (near <= chunk) continue;                             // the same in every thread
    const int lo = slot == 0 ? p0 : p1 - inside, hi = lo + inside;
    const int seg = (hi - lo + kEmbWarps - 1) / kEmbWarps;
    const int j0 = lo + w * seg < hi ? lo + w * seg : hi, j1 = j0 + seg < hi ? j0 + seg : hi;
    for (int c8 = lane; c8 < C / 8; c8 += 32) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      emb_sum_run(DY, dy_dt, perm, j0, j1, C, c8, acc);
#pragma unroll
      for (int q = 0; q < 8; ++q) emb_part[(size_t)w * C + c8 * 8 + q] = acc[q];
    }
    __syncthreads();
    float* out = part + (size_t)(2 * blockIdx.x + slot) * C;
    for (int c = threadIdx.x; c < C; c += kEmbWarps * 32) {
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < kEmbWarps; ++q) t += emb_part[(size_t)q * C + c];
      out[c] = t;
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kEmbWarps * 32)
embedding_bwd_kernel(const int* __restrict__ starts, const int* __restrict__ perm,
                     const void* __restrict__ DY, int dy_dt, const float* __restrict__ part,
                     float* __restrict__ GW, int C, int V, int chunk) {
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (long long v = blockIdx.x * kEmbWarps + w; v < V; v += gridDim.x * kEmbWarps) {
    const int s = starts[v], e = starts[v + 1];
    const bool parts = e - s > chunk;
    // The first chunk holds the run in slot 0 only if the run covers its first position.
    const int c0 = s / chunk, c1 = (e - 1) / chunk;
    for (int c8 = lane; c8 < C / 8; c8 += 32) {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (parts) {
        const float* p = part + c8 * 8;
        emb_load8(p, DT_F32, (long long)(2 * c0 + (s % chunk != 0)) * C, acc);
        int c = c0 + 1;
        for (; c + 3 <= c1; c += 4) {
          float u[4][8];
#pragma unroll
          for (int q = 0; q < 4; ++q) emb_load8(p, DT_F32, (long long)(2 * (c + q)) * C, u[q]);
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int x = 0; x < 8; ++x) acc[x] += u[q][x];
        }
        for (; c <= c1; ++c) {
          float u[8];
          emb_load8(p, DT_F32, (long long)(2 * c) * C, u);
#pragma unroll
          for (int x = 0; x < 8; ++x) acc[x] += u[x];
        }
      } else {
        emb_sum_run(DY, dy_dt, perm, s, e, C, c8, acc);
      }
      float4* q = reinterpret_cast<float4*>(GW + v * C + c8 * 8);
      q[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
      q[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
    }
  }
}

static inline int key_bits(long long V) {   // bits needed for the values 0 .. V
  int b = 1;
  while ((1LL << b) <= V) ++b;
  return b;
}

}  // namespace dion

using namespace dion;
static inline cudaStream_t S(void* s) { return static_cast<cudaStream_t>(s); }

// Bytes of temporary storage the sort of n (key, position) pairs needs.
DION_EXPORT long long dion_embedding_sort_bytes(long long n, long long V) {
  if (n <= 0) return 0;
  size_t bytes = 0;
  const int* kin = nullptr;
  int* kout = nullptr;
  if (cub::DeviceRadixSort::SortPairs(nullptr, bytes, kin, kout, kin, kout, static_cast<int>(n), 0,
                                      key_bits(V)) != cudaSuccess)
    return -1;
  return static_cast<long long>(bytes);
}

// Rows of C floats that the partial sums of n tokens need.
DION_EXPORT long long dion_embedding_part_rows(long long n) {
  if (n <= 0) return 0;
  return 2LL * emb_num_chunks(n, emb_chunk(n));
}

// ids: int64 [n].  DY: [n, C] fp32 or bf16 (dy_dt).  GW: fp32 [V, C], needs no initialisation.
// Scratch: keys, vals int32 [2n] each (unsorted then sorted halves), starts int32 [V+1], temp of
// at least dion_embedding_sort_bytes(n, V) bytes, part fp32 [dion_embedding_part_rows(n), C], 16-byte
// aligned.  Limits: n, V < 2^31; 8*C*4 bytes of shared
// memory (C <= 7168); C a multiple of 8.
DION_EXPORT int dion_embedding_bwd(const void* ids, const void* DY, int dy_dt, float* GW,
                                   long long n, int C, long long V, int* keys, int* vals,
                                   int* starts, void* temp, long long temp_bytes, float* part,
                                   void* stream) {
  if (V <= 0) return 0;
  if (C % 8 || n < 0 || n >= (1LL << 31) - 256 || V >= (1LL << 31) - 256) return -2;
  const size_t smem = (size_t)kEmbWarps * C * sizeof(float);
  if (smem > 224 * 1024) return -2;
  const int ni = static_cast<int>(n), Vi = static_cast<int>(V);
  if (ni > 0) {
    emb_keys_kernel<<<(ni + 255) / 256, 256, 0, S(stream)>>>(static_cast<const long long*>(ids),
                                                            keys, vals, ni, Vi);
    size_t bytes = static_cast<size_t>(temp_bytes);
    if (cub::DeviceRadixSort::SortPairs(temp, bytes, keys, keys + ni, vals, vals + ni, ni, 0,
                                        key_bits(V), S(stream)) != cudaSuccess)
      return -4;
  }
  // The same limit in every call: a smaller one, set by another thread, could come between it and
  // the launch.
  constexpr size_t kMost = (size_t)kEmbWarps * 7168 * sizeof(float);
  if (smem > kMost ||
      (smem > 48 * 1024 &&
       cudaFuncSetAttribute(emb_starts_parts_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                            (int)kMost) != cudaSuccess))
    return -3;
  const int chunk = emb_chunk(n);
  const int chunks = ni > chunk ? emb_num_chunks(n, chunk) : 0;   // else no run is longer than a chunk
  emb_starts_parts_kernel<<<chunks + Vi / (kEmbWarps * 32) + 1, kEmbWarps * 32, chunks ? smem : 0,
                            S(stream)>>>(keys + ni, starts, vals + ni, DY, dy_dt, part, ni, C, Vi,
                                         chunk, chunks);
  const int groups = (Vi + kEmbWarps - 1) / kEmbWarps;
  const int cap = 148 * 8;
  embedding_bwd_kernel<<<groups < cap ? groups : cap, kEmbWarps * 32, 0, S(stream)>>>(
      starts, vals + ni, DY, dy_dt, part, GW, C, Vi, chunk);
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
