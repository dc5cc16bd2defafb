// Transformer blocks of the GPT without gradients (sampling, scoring) for sm_100a: two host calls
// per block issue all of its kernels but the attention.
//
// A block of a short prompt is a dozen kernels of 2 to 9 us; issued one by one through the Python
// front end they cost 400 us of host time per block, 4.8 ms for twelve, against 0.8 ms of device
// time.  Here the host side of a block is this file: one kernel rounds the block's six fp32
// weights to bf16 (one after the other, q/k/v stacked for one product), the products run on the
// tcgen05 kernels of ns_gemm2_sm100.cu / ns_gemm_sm100.cu (relu^2 in the epilogue where the two-CTA
// kernel takes them), the norms and RoPE on those of model_ops.cu.  The entry points of the other
// libraries are given by address.
#include "common.cuh"
#include "tmap_cache.h"

namespace dion {

constexpr int kCastMax = 6;
struct CastArgs {
  const void* src[kCastMax];
  long long end8[kCastMax];   // running totals of 8-element groups
  int n;
  int dt;                     // 0 fp32, 1 bf16
};

// dst = the sources one after the other, rounded to bf16; every size is a multiple of 8 and every
// address 16-byte aligned.  Bound by memory: 6 bytes an element for fp32, two groups in flight per
// thread.
__global__ void __launch_bounds__(256)
infer_cast_kernel(const CastArgs a, __nv_bfloat16* dst) {
  const long long total = a.end8[a.n - 1];
  const long long step = (long long)gridDim.x * 256;
  for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += 2 * step) {
    uint4 out[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long j = i + h * step;
      if (j >= total) break;
      int t = 0;
      long long begin = 0;
#pragma unroll
      for (int q = 0; q < kCastMax - 1; ++q)
        if (q < a.n - 1 && j >= a.end8[q]) { t = q + 1; begin = a.end8[q]; }
      const void* src = a.src[0];
#pragma unroll
      for (int q = 1; q < kCastMax; ++q)
        if (t == q) src = a.src[q];
      if (a.dt == 0) {
        const float4* s = reinterpret_cast<const float4*>(src) + 2 * (j - begin);
        const float4 x = __ldg(s), y = __ldg(s + 1);
        out[h] = make_uint4(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w), pack_bf16x2(y.x, y.y),
                            pack_bf16x2(y.z, y.w));
      } else {
        out[h] = __ldg(reinterpret_cast<const uint4*>(src) + (j - begin));
      }
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
      if (i + h * step < total) reinterpret_cast<uint4*>(dst)[i + h * step] = out[h];
  }
}

}  // namespace dion

using namespace dion;

typedef int (*Gemm2Fn)(const void*, long long, long long, int, const void*, long long, long long,
                       int, void*, long long, long long, const void*, long long, long long, int,
                       int, int, int, float, float, const float*, int, int, int, const void*, int,
                       int, int*, void*, const void*);
typedef int (*GemmFn)(const void*, long long, long long, int, const void*, long long, long long,
                      int, void*, long long, long long, const void*, long long, long long, void*,
                      long long, long long, void*, int, int, int, int, float, float, const float*,
                      int, int, int, const void*, int, int, int, int*, void*, const void*);
typedef int (*NormFn)(const void*, int, const void*, int, void*, void*, int, float*, long long, int,
                      float, void*);
typedef int (*RopeFn)(const void*, const void*, long long, const void*, const void*, void*, void*,
                      float*, int, int, int, int, float, void*);
typedef int (*Relu2Fn)(const void*, void*, int, long long, void*);

struct DionInferGemm {
  const void* tiles;
  int n_tiles;
  int bn;          // 0: two-CTA kernel, else BN of the single-CTA kernel
};

// One forward pass: mirrored by models/inference.py.
struct DionInfer {
  Gemm2Fn gemm2;      // dion_ns_gemm2_ex
  GemmFn gemm;        // dion_ns_gemm_ex
  NormFn norm;        // dion_rmsnorm_fwd
  RopeFn rope;        // dion_rope_qknorm_fwd
  Relu2Fn relu2;      // dion_relu2_fwd
  void* x0;           // residual stream, fp32 [rows, C]
  void* x1;           // the same after the attention
  void* h;            // normalized stream, bf16 [rows, C]
  void* w;            // bf16 weights of the current block
  void* qkv;          // bf16 [rows, 3C]
  void* qo;           // bf16 [rows, C]
  void* ko;
  void* o;            // bf16 [rows, C]: what is added to the stream
  void* act;          // bf16 [rows, F]
  float* rstd;        // fp32 [2 * rows * H]
  int* status;
  int B, T, H, D, F, w_dt, sms;
  float eps_x, eps_qk;
  DionInferGemm cfg[4];   // qkv, attention projection, MLP in, MLP out
};

// Y [rows, N] = X [rows, K] W[N, K]^T; relu2: squared positive part.
static int product(const DionInfer* p, int which, const void* X, const __nv_bfloat16* W, void* Y,
                   int N, int K, int relu2, void* stream) {
  const DionInferGemm& g = p->cfg[which];
  const int rows = p->B * p->T;
  const long long sx = (long long)rows * K, sw = (long long)N * K, sy = (long long)rows * N;
  if (g.bn == 0)
    return p->gemm2(X, K, sx, 0, W, K, sw, 0, Y, N, sy, nullptr, 0, 0, 1, rows, N, K, 1.f, 0.f,
                    nullptr, 0, 0, 0, g.tiles, g.n_tiles, relu2 ? 1 : 0, p->status, stream, nullptr);
  const int rc = p->gemm(X, K, sx, 0, W, K, sw, 0, Y, N, sy, nullptr, 0, 0, nullptr, 0, 0, nullptr, 1,
                         rows, N, K, 1.f, 0.f, nullptr, 0, 0, 0, g.tiles, g.n_tiles, g.bn, p->sms,
                         p->status, stream, nullptr);
  if (rc != 0 || !relu2) return rc;
  return p->relu2(Y, Y, 1, sy, stream);
}

// Rounds the block's weights into w, projects h to q, k and v, applies RoPE and the QK norm.
DION_EXPORT int dion_infer_block_in(const DionInfer* p, const void* wq, const void* wk,
                                    const void* wv, const void* wo, const void* wfc,
                                    const void* wpr, const void* cos, const void* sin,
                                    void* stream) {
  const int C = p->H * p->D;
  const long long cc = (long long)C * C / 8, cf = (long long)C * p->F / 8;
  CastArgs a;
  const void* src[kCastMax] = {wq, wk, wv, wo, wfc, wpr};
  long long end = 0;
  for (int i = 0; i < kCastMax; ++i) {
    if (reinterpret_cast<uintptr_t>(src[i]) & 15) return -10;
    a.src[i] = src[i];
    a.end8[i] = end += i < 4 ? cc : cf;
  }
  a.n = kCastMax;
  a.dt = p->w_dt;
  const long long blocks = (end + 511) / 512;
  infer_cast_kernel<<<(unsigned)(blocks < 8 * p->sms ? blocks : 8 * p->sms), 256, 0,
                      static_cast<cudaStream_t>(stream)>>>(a, static_cast<__nv_bfloat16*>(p->w));
  if (cudaGetLastError() != cudaSuccess) return -1;
  const __nv_bfloat16* w = static_cast<const __nv_bfloat16*>(p->w);
  int rc = product(p, 0, p->h, w, p->qkv, 3 * C, C, 0, stream);
  if (rc != 0) return rc;
  const __nv_bfloat16* q = static_cast<const __nv_bfloat16*>(p->qkv);
  return p->rope(q, q + C, 3LL * C, cos, sin, p->qo, p->ko, p->rstd, p->B, p->T, p->H, p->D,
                 p->eps_qk, stream);
}

// The block behind the attention's result y (bf16 [rows, C]): projection, residual and norm, MLP,
// residual and norm.  x0 and h are the next block's input.
DION_EXPORT int dion_infer_block_out(const DionInfer* p, const void* y, void* stream) {
  const int C = p->H * p->D, F = p->F;
  const long long rows = (long long)p->B * p->T;
  const __nv_bfloat16* wo = static_cast<const __nv_bfloat16*>(p->w) + 3LL * C * C;
  const __nv_bfloat16* wfc = wo + (long long)C * C;
  const __nv_bfloat16* wpr = wfc + (long long)C * F;
  int rc = product(p, 1, y, wo, p->o, C, C, 0, stream);
  if (rc == 0)
    rc = p->norm(p->x0, 0, p->o, 1, p->x1, p->h, 1, p->rstd, rows, C, p->eps_x, stream);
  if (rc == 0) rc = product(p, 2, p->h, wfc, p->act, F, C, 1, stream);
  if (rc == 0) rc = product(p, 3, p->act, wpr, p->o, C, F, 0, stream);
  if (rc == 0)
    rc = p->norm(p->x1, 0, p->o, 1, p->x0, p->h, 1, p->rstd, rows, C, p->eps_x, stream);
  return rc;
}

// ---------------------------------------------------------------------------------------------
// Short prompts: the whole stack of blocks from one host call (dion_infer_stack)
// ---------------------------------------------------------------------------------------------
// A block of GPT-160M has 28 MB of fp32 weights and, for 128 rows, 1.8 GFLOP: 4.4 us of memory, 1 us
// of tensor cores.  Rounded to bf16 by one kernel (11 us) and multiplied by four tcgen05 products of 6
// to 24 CTAs (12 us each) it took 80 us with its norms, RoPE and attention.  Here
//   * a product reads its fp32 weights itself and rounds them on the way to the tensor cores, with K
//     split over the CTAs of a cluster, so that about one CTA per SM streams weights;
//   * the norms are folded into the products: a row's scale commutes with the product, so the
//     product takes bf16(x) and its epilogue multiplies by 1 / rms, whose sum of squares the
//     epilogue that wrote x left behind (one partial sum per column tile);
//   * residual, relu^2 and the rounding of the stream ride in the epilogues, RoPE and the norm of
//     queries and keys in the attention;
//   * launches are programmatic: the next kernel's CTAs start beside the present one's and fetch
//     their weights, which nothing in the stack writes, before they wait for it to end.
namespace dion {

constexpr int kSkThreads = 160;      // warp 0: X and MMA; warps 1 to 4: weights and epilogue
constexpr int kSkABytes = 128 * 128; // a 64-wide K slab of 128 rows, bf16
constexpr int kSkRing = 4;           // slabs of X in shared memory

enum : int { kSkStore = 0, kSkRelu2 = 1, kSkResidual = 2 };

struct SkinnyArgs {
  const void *w0, *w1, *w2;   // [n_per_w, K] each, stacked to N rows
  int n_per_w;
  int w_dt;              // 0 fp32, 1 bf16
  int rows, N, K;
  int slabs;             // K slabs per CTA of a cluster (its share of K)
  const float* ss;       // partial sums of squares of the input rows [rows, parts], or null
  int parts;
  float eps;
  int epi;
  __nv_bfloat16* Y;      // [rows, N] (kSkStore, kSkRelu2)
  float* x;              // [rows, N] fp32 stream, updated in place (kSkResidual)
  __nv_bfloat16* xb;     // its rounded copy
  float* ss_out;         // [rows, gridDim.y] partial sums of squares of the new stream
  int* status;
};

__device__ __forceinline__ uint32_t sk_cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void sk_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float4 sk_ld_cluster(uint32_t local, uint32_t rank) {
  uint32_t a;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(local), "r"(rank));
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a));      // volatile: stays behind the cluster barrier
  return v;
}
// Y[rows, N] = X[rows, K] W^T for one tile of 128 rows x BN columns per cluster: grid (splits, column
// tiles, row tiles), cluster (splits, 1, 1); CTA s of a cluster takes K slabs [s * slabs, ...), SLABS
// at most.  A CTA's weights are all requested at once, into registers (96 to 128 of them), so nothing
// but the memory's latency is waited for; the partial results meet through distributed shared
// memory, each CTA finishing its part of the rows.
template <int BN, int SLABS>
__global__ void __launch_bounds__(kSkThreads)
skinny_kernel(const __grid_constant__ CUtensorMap map_x, const SkinnyArgs p) {
  constexpr int kRing = SLABS < kSkRing ? SLABS : kSkRing;
  constexpr int kBBytes = BN * 128;
  constexpr int kPitch = BN + 4;       // fp32 row of the partial result
  constexpr int kLanes = BN / 4;       // lanes that share a row of the result
  extern __shared__ uint8_t sk_smem[];
  uint8_t* a_buf = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(sk_smem) + 1023) &
                                              ~static_cast<uintptr_t>(1023));
  uint8_t* b_buf = a_buf + kRing * kSkABytes;
  __shared__ __align__(8) uint64_t x_bar[kRing], e_bar[kRing];
  __shared__ __align__(8) uint64_t conv_bar, done_bar;
  __shared__ uint32_t tmem_slot;
  __shared__ int sk_ok;
  __shared__ float rms_inv[128];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int splits = (int)gridDim.x;
  const int rank = (int)sk_cluster_rank();
  const int total_slabs = (p.K + 63) / 64;
  const int s0 = rank * p.slabs;
  const int ns = total_slabs - s0 < p.slabs ? total_slabs - s0 : p.slabs;   // 1 to SLABS
  const int n0 = blockIdx.y * BN;
  const int row0 = blockIdx.z * 128;
  let_next_kernel_start();

  float4 w[BN / 16][SLABS][2];
  const int t = (int)threadIdx.x - 32;     // 0..127 in warps 1 to 4
  if (warp > 0) {
    // ---- weights: eight lanes take 64 elements of a row ----
#pragma unroll
    for (int j = 0; j < BN / 16; ++j) {
      const int n = n0 + (t >> 3) + 16 * j;
      const int which = (n >= p.n_per_w) + (n >= 2 * p.n_per_w);
      const void* base = which == 0 ? p.w0 : which == 1 ? p.w1 : p.w2;
      const long long at = (long long)(n - which * p.n_per_w) * p.K + s0 * 64 + (t & 7) * 8;
#pragma unroll
      for (int s = 0; s < SLABS; ++s) {
        w[j][s][0] = w[j][s][1] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (s < ns && n < p.N && (s0 + s) * 64 + (t & 7) * 8 < p.K) {   // K is a multiple of 8
          if (p.w_dt == 0) {
            const float4* src = reinterpret_cast<const float4*>(static_cast<const float*>(base) + at + s * 64);
            w[j][s][0] = __ldg(src);
            w[j][s][1] = __ldg(src + 1);
          } else {
            w[j][s][0] = __ldg(reinterpret_cast<const float4*>(
                static_cast<const __nv_bfloat16*>(base) + at + s * 64));
          }
        }
      }
    }
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRing; ++s) {
      mbar_init(&x_bar[s], 1);
      mbar_init(&e_bar[s], 1);
    }
    mbar_init(&conv_bar, 4);
    mbar_init(&done_bar, 1);
    sk_ok = 1;
    fence_barrier_init();
    fence_proxy_async();
    prefetch_tmap(&map_x);
  }
  if (warp == 0) {
    tmem_alloc(&tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  // The rows this CTA finishes: rank * per + t / kLanes + kStep * i; those of the first batch have
  // their old stream requested long before it is needed.
  constexpr int kStep = 128 / kLanes, kBatch = 2;
  const int per = ((128 + splits - 1) / splits + 15) / 16 * 16;
  const int n = n0 + t % kLanes * 4;         // N is a multiple of 8
  float4 old[kBatch];
  auto finishes = [&](int rr) { return rr < per && rank * per + rr < 128; };
  auto stream_at = [&](int rr) {
    return reinterpret_cast<float4*>(p.x + (long long)(row0 + rank * per + rr) * p.N + n);
  };
  auto request_old = [&](int rr0) {
#pragma unroll
    for (int u = 0; u < kBatch; ++u) {
      const int rr = rr0 + u * kStep;
      if (p.epi == kSkResidual && finishes(rr) && row0 + rank * per + rr < p.rows && n < p.N)
        old[u] = *stream_at(rr);
    }
  };

  if (warp == 0) {
    if (lane == 0) {
      wait_for_previous_kernel();
      auto load = [&](int s) {
        mbar_expect_tx(&x_bar[s % kRing], kSkABytes);
        tma_load_3d(a_buf + (s % kRing) * kSkABytes, &map_x, &x_bar[s % kRing], (s0 + s) * 64, row0, 0);
      };
      int loaded = 0;
      for (; loaded < ns && loaded < kRing; ++loaded) load(loaded);
      constexpr uint32_t idesc = make_idesc_bf16(128, BN, 0, 0);
      bool ok = mbar_wait_bounded(&conv_bar, 0);
      int s = 0;
      for (; s < ns && ok; ++s) {
        if (!mbar_wait_bounded(&x_bar[s % kRing], (s / kRing) & 1)) {
          ok = false;
          break;
        }
        tc_fence_after();
        const uint32_t sa = smem_u32(a_buf + (s % kRing) * kSkABytes);
        const uint32_t sb = smem_u32(b_buf + s * kBBytes);
#pragma unroll
        for (int k = 0; k < 4; ++k)
          tc_mma_bf16(tmem, make_smem_desc(sa + k * 32, 16, 1024),
                      make_smem_desc(sb + k * 32, 16, 1024), idesc, (s | k) != 0 ? 1u : 0u);
        tc_commit(&e_bar[s % kRing]);
        if (loaded < ns) {      // the slab's place is free once these products have read it
          ok = mbar_wait_bounded(&e_bar[s % kRing], (s / kRing) & 1);
          if (ok) load(loaded++);
        }
      }
      if (ok) {
        tc_commit(&done_bar);
      } else {
        atomicExch(p.status, kStatusTimeoutFull);
        sk_ok = 0;
        for (; s < loaded; ++s)      // copies in flight land before the CTA exits
          mbar_wait_bounded(&x_bar[s % kRing], (s / kRing) & 1);
        mbar_arrive(&done_bar);
      }
    }
    __syncwarp();
  } else {
    // ---- rounded into the operand layout ----
#pragma unroll
    for (int j = 0; j < BN / 16; ++j) {
      const int r = (t >> 3) + 16 * j;
#pragma unroll
      for (int s = 0; s < SLABS; ++s) {
        if (s >= ns) break;
        const float4 a = w[j][s][0], b = w[j][s][1];
        const uint4 o = p.w_dt == 0
                            ? make_uint4(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w),
                                         pack_bf16x2(b.x, b.y), pack_bf16x2(b.z, b.w))
                            : make_uint4(__float_as_uint(a.x), __float_as_uint(a.y),
                                         __float_as_uint(a.z), __float_as_uint(a.w));
        *reinterpret_cast<uint4*>(b_buf + s * kBBytes + r * 128 + (((t & 7) ^ (r & 7)) << 4)) = o;
      }
    }
    fence_proxy_async();
    __syncwarp();
    if (lane == 0) mbar_arrive(&conv_bar);
    wait_for_previous_kernel();    // from here on, what the preceding kernels wrote is read and written
    request_old(t / kLanes);
    if (p.ss != nullptr) {  // 1 / rms of every row of the tile
      float sum = 0.f;
      if (row0 + t < p.rows) {
        const float* ss = p.ss + (long long)(row0 + t) * p.parts;
#pragma unroll 8
        for (int i = 0; i < p.parts; ++i) sum += ss[i];
      }
      rms_inv[t] = rsqrtf(sum / (float)p.K + p.eps);
    }

    // ---- this CTA's share of the sum, from TMEM to shared memory (X has been read) ----
    if (!mbar_wait_bounded(&done_bar, 0)) {
      if (lane == 0) atomicExch(p.status, kStatusTimeoutTmemFull);
      sk_ok = 0;
    }
    __syncwarp();
    tc_fence_after();
    const int lane_grp = warp & 3;
    float4* mine = reinterpret_cast<float4*>(a_buf + (size_t)(lane_grp * 32 + lane) * kPitch * 4);
#pragma unroll
    for (int half = 0; half < BN / 32; ++half) {
      float v[32];
      tmem_ld_32x32(tmem + (static_cast<uint32_t>(lane_grp * 32) << 16) + half * 32, v);
      tmem_ld_wait();
#pragma unroll
      for (int q = 0; q < 8; ++q)
        mine[half * 8 + q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
    tc_fence_before();
  }
  __syncthreads();
  sk_cluster_sync();      // every CTA of the cluster has written its partial result
  if (warp > 0 && sk_ok) {
    const int q = t % kLanes;
    for (int rr0 = t / kLanes; rr0 < per; rr0 += kStep * kBatch) {
      float4 part[kBatch][8];
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int rr = rr0 + u * kStep;
        const uint32_t at = smem_u32(a_buf + (size_t)(rank * per + rr) * kPitch * 4 + q * 16);
#pragma unroll
        for (int s = 0; s < 8; ++s)
          if (s < splits && finishes(rr)) part[u][s] = sk_ld_cluster(at, (uint32_t)s);
      }
      if (rr0 != t / kLanes) request_old(rr0);
#pragma unroll
      for (int u = 0; u < kBatch; ++u) {
        const int rr = rr0 + u * kStep;
        if (!finishes(rr)) continue;           // the same for a whole warp
        const int g = row0 + rank * per + rr;
        const bool live = g < p.rows, in = live && n < p.N;
        float4 a = part[u][0];
#pragma unroll
        for (int s = 1; s < 8; ++s) {
          if (s < splits) {
            a.x += part[u][s].x; a.y += part[u][s].y; a.z += part[u][s].z; a.w += part[u][s].w;
          }
        }
        if (p.ss != nullptr) {
          const float r = rms_inv[rank * per + rr];
          a.x *= r; a.y *= r; a.z *= r; a.w *= r;
        }
        if (p.epi == kSkResidual) {
          float sq = 0.f;
          if (in) {
            float4 x = old[u];
            const float2 lo = unpack_bf16x2(pack_bf16x2(a.x, a.y));
            const float2 hi = unpack_bf16x2(pack_bf16x2(a.z, a.w));
            x.x += lo.x; x.y += lo.y; x.z += hi.x; x.w += hi.y;
            *stream_at(rr) = x;
            *reinterpret_cast<uint2*>(p.xb + (long long)g * p.N + n) =
                make_uint2(pack_bf16x2(x.x, x.y), pack_bf16x2(x.z, x.w));
            sq = x.x * x.x + x.y * x.y + x.z * x.z + x.w * x.w;
          }
#pragma unroll
          for (int o = kLanes / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(0xffffffffu, sq, o);
          if (q == 0 && live) p.ss_out[(long long)g * gridDim.y + blockIdx.y] = sq;
        } else if (in) {
          if (p.epi == kSkRelu2) {
            a.x = fmaxf(a.x, 0.f); a.y = fmaxf(a.y, 0.f); a.z = fmaxf(a.z, 0.f); a.w = fmaxf(a.w, 0.f);
            a.x *= a.x; a.y *= a.y; a.z *= a.z; a.w *= a.w;
          }
          *reinterpret_cast<uint2*>(p.Y + (long long)g * p.N + n) =
              make_uint2(pack_bf16x2(a.x, a.y), pack_bf16x2(a.z, a.w));
        }
      }
    }
  }
  sk_cluster_sync();      // nobody leaves while its partial result may still be read
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, BN);
  }
}

// The stream's entry: bf16 copy and sum of squares of every row; one warp a row.
__global__ void __launch_bounds__(256)
stream_in_kernel(const float* __restrict__ x, __nv_bfloat16* xb, float* ss, int rows, int C) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  float s = 0.f;
  for (int c = lane * 4; c < C; c += 128) {
    const float4 v = *reinterpret_cast<const float4*>(x + (long long)row * C + c);
    s += v.x * v.x + v.y * v.y + v.z * v.z + v.w * v.w;
    *reinterpret_cast<uint2*>(xb + (long long)row * C + c) =
        make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) ss[row] = s;
}

// ---- causal attention of short sequences ------------------------------------------------------
// One CTA per 64 queries of a head; keys and values pass through shared memory in chunks of 128. Four
// warps take the first 64 keys of every chunk for 16 queries each, four more the other 64; scores and
// running softmax stay in registers, and the two halves are joined at the end.
// Queries and keys get their RoPE and RMS norm on the way in, in the arithmetic of
// rope_qknorm_fwd_kernel; a key is then rotated once per 64 queries.  24 CTAs for 128 tokens of 12
// heads: a chain of latencies of a few us whatever computes the products, so these are warp-level
// MMAs, which need no TMEM and no second trip of the probabilities through memory.
__device__ __forceinline__ void mma_16816(float* c, const uint32_t* a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    const float2 x = unpack_bf16x2(w[e]);
    f[2 * e] = x.x;
    f[2 * e + 1] = x.y;
  }
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  return make_uint4(pack_bf16x2(f[0], f[1]), pack_bf16x2(f[2], f[3]), pack_bf16x2(f[4], f[5]),
                    pack_bf16x2(f[6], f[7]));
}

constexpr int kAttThreads = 256, kAttChunk = 128;
template <int D>
__host__ __device__ constexpr int att_smem() { return (64 + 2 * kAttChunk) * (D + 8) * 2; }

template <int D>
__global__ void __launch_bounds__(kAttThreads)
short_attention_kernel(const __nv_bfloat16* __restrict__ qkv, const __nv_bfloat16* __restrict__ cs,
                       const __nv_bfloat16* __restrict__ sn, __nv_bfloat16* __restrict__ y, int T,
                       int H, float eps, float scale_log2) {
  constexpr int P = D + 8;      // row pitch: fragments of eight rows fall into different banks
  constexpr int KC = kAttChunk, HALF = D / 2, TPV = D / 16, VPP = kAttThreads / TPV;
  extern __shared__ __align__(16) uint8_t at_smem[];
  __nv_bfloat16* qs = reinterpret_cast<__nv_bfloat16*>(at_smem);
  __nv_bfloat16* ks = qs + 64 * P;
  __nv_bfloat16* vs = ks + KC * P;
  const int warp = (threadIdx.x >> 5) & 3, lane = threadIdx.x & 31;
  const int part = threadIdx.x >> 7;       // which 64 keys of a chunk
  const int h = blockIdx.y, b = blockIdx.z;
  const int q0 = blockIdx.x * 64;
  const int C = H * D;
  const long long ld = 3LL * C;
  const __nv_bfloat16* base = qkv + (long long)b * T * ld + h * D;
  const int r_lo = q0 + warp * 16 + (lane >> 2), r_hi = r_lo + 8, cc = (lane & 3) * 2;
  let_next_kernel_start();
  wait_for_previous_kernel();

  // Rows [first, first + n) of a section of qkv, rotated and normalized, into `dst`.
  const int sub = (int)threadIdx.x % TPV;
  auto rotate_in = [&](__nv_bfloat16* dst, const __nv_bfloat16* src, int first, int n) {
#pragma unroll 2
    for (int r = (int)threadIdx.x / TPV; r < n; r += VPP) {
      const int tok = first + r;
      uint4 u1 = make_uint4(0u, 0u, 0u, 0u), u2 = u1, uc = u1, us = u1;
      if (tok < T) {
        const __nv_bfloat16* x = src + (long long)tok * ld;
        u1 = *reinterpret_cast<const uint4*>(x + sub * 8);
        u2 = *reinterpret_cast<const uint4*>(x + HALF + sub * 8);
        uc = __ldg(reinterpret_cast<const uint4*>(cs + (long long)tok * HALF + sub * 8));
        us = __ldg(reinterpret_cast<const uint4*>(sn + (long long)tok * HALF + sub * 8));
      }
      float x1[8], x2[8], c[8], s[8];
      unpack8(u1, x1); unpack8(u2, x2); unpack8(uc, c); unpack8(us, s);
      float ss = 0.f;
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const float a = x1[e] * c[e] + x2[e] * s[e], d = x2[e] * c[e] - x1[e] * s[e];
        x1[e] = a;
        x2[e] = d;
        ss += a * a + d * d;
      }
#pragma unroll
      for (int o = TPV / 2; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
      const float g = rsqrtf(ss / (float)D + eps);
#pragma unroll
      for (int e = 0; e < 8; ++e) { x1[e] *= g; x2[e] *= g; }
      *reinterpret_cast<uint4*>(dst + r * P + sub * 8) = pack8(x1);
      *reinterpret_cast<uint4*>(dst + r * P + HALF + sub * 8) = pack8(x2);
    }
  };

  uint32_t qf[D / 16][4];
  float o[D / 8][4];
#pragma unroll
  for (int d = 0; d < D / 8; ++d)
#pragma unroll
    for (int e = 0; e < 4; ++e) o[d][e] = 0.f;
  float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};

  const int keys = q0 + 64 < T ? q0 + 64 : T;      // later keys are masked for every query here
  for (int c0 = 0; c0 < keys; c0 += KC) {
    const int blocks = (keys - c0 < KC ? keys - c0 + 63 : KC) / 64;    // of 64 keys
    __syncthreads();
#pragma unroll 4
    for (int e = threadIdx.x; e < blocks * 64 * (D / 8); e += kAttThreads) {
      const int r = e / (D / 8), c = (e - r * (D / 8)) * 8, key = c0 + r;
      uint4 vv = make_uint4(0u, 0u, 0u, 0u);
      if (key < T) vv = *reinterpret_cast<const uint4*>(base + 2 * C + (long long)key * ld + c);
      *reinterpret_cast<uint4*>(vs + r * P + c) = vv;
    }
    if (c0 == 0) rotate_in(qs, base, q0, 64);
    rotate_in(ks, base + C, c0, blocks * 64);
    __syncthreads();
    if (c0 == 0) {
#pragma unroll
      for (int d = 0; d < D / 16; ++d) {
        const __nv_bfloat16* lo = qs + (r_lo - q0) * P + d * 16 + cc;
        const __nv_bfloat16* hi = lo + 8 * P;
        qf[d][0] = *reinterpret_cast<const uint32_t*>(lo);
        qf[d][1] = *reinterpret_cast<const uint32_t*>(hi);
        qf[d][2] = *reinterpret_cast<const uint32_t*>(lo + 8);
        qf[d][3] = *reinterpret_cast<const uint32_t*>(hi + 8);
      }
    }
    if (part < blocks) {
      const int kb = part, key0 = c0 + kb * 64;
      float s[8][4];
#pragma unroll
      for (int n = 0; n < 8; ++n) {
#pragma unroll
        for (int e = 0; e < 4; ++e) s[n][e] = 0.f;
#pragma unroll
        for (int d = 0; d < D / 16; ++d) {
          const __nv_bfloat16* kp = ks + (kb * 64 + n * 8 + (lane >> 2)) * P + d * 16 + cc;
          mma_16816(s[n], qf[d], *reinterpret_cast<const uint32_t*>(kp),
                    *reinterpret_cast<const uint32_t*>(kp + 8));
        }
      }
      if (key0 >= q0) {      // the block on the diagonal
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (key0 + n * 8 + cc + (e & 1) > ((e & 2) ? r_hi : r_lo)) s[n][e] = -INFINITY;
      }
#pragma unroll
      for (int half = 0; half < 2; ++half) {
        float mx = m[half];
#pragma unroll
        for (int n = 0; n < 8; ++n) mx = fmaxf(mx, fmaxf(s[n][2 * half], s[n][2 * half + 1]));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 1));
        mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 2));
        if (mx == -INFINITY) mx = 0.f;         // all of these keys come after the query
        const float corr = exp2f((m[half] - mx) * scale_log2);
        m[half] = mx;
        float sum = 0.f;
#pragma unroll
        for (int n = 0; n < 8; ++n)
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            const float x = exp2f((s[n][2 * half + e] - mx) * scale_log2);
            s[n][2 * half + e] = x;
            sum += x;
          }
        l[half] = l[half] * corr + sum;
#pragma unroll
        for (int d = 0; d < D / 8; ++d) {
          o[d][2 * half] *= corr;
          o[d][2 * half + 1] *= corr;
        }
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {      // 16 keys at a time
        const uint32_t a[4] = {pack_bf16x2(s[2 * j][0], s[2 * j][1]),
                               pack_bf16x2(s[2 * j][2], s[2 * j][3]),
                               pack_bf16x2(s[2 * j + 1][0], s[2 * j + 1][1]),
                               pack_bf16x2(s[2 * j + 1][2], s[2 * j + 1][3])};
#pragma unroll
        for (int d = 0; d < D / 16; ++d) {
          const int key = kb * 64 + j * 16 + ((lane >> 3) & 1) * 8 + (lane & 7);
          const uint32_t addr = smem_u32(vs + key * P + d * 16 + (lane >> 4) * 8);
          uint32_t f[4];
          asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
                       : "=r"(f[0]), "=r"(f[1]), "=r"(f[2]), "=r"(f[3])
                       : "r"(addr)
                       : "memory");
          mma_16816(o[2 * d], a, f[0], f[1]);
          mma_16816(o[2 * d + 1], a, f[2], f[3]);
        }
      }
    }
  }
  // The second half of the keys hands over (m, l, o); a query without keys there brings m = -inf or
  // l = 0.  Key 0 is in the first half, so its m is finite.
  __syncthreads();
  float* mine = reinterpret_cast<float*>(at_smem) + (size_t)(warp * 32 + lane) * (D / 2 + 5);
  if (part == 1) {
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      mine[half] = m[half];
      mine[2 + half] = l[half];
    }
#pragma unroll
    for (int d = 0; d < D / 8; ++d)
#pragma unroll
      for (int e = 0; e < 4; ++e) mine[4 + d * 4 + e] = o[d][e];
  }
  __syncthreads();
  if (part == 1) return;
#pragma unroll
  for (int half = 0; half < 2; ++half) {
    const float m2 = mine[half], mx = fmaxf(m[half], m2);
    const float c1 = exp2f((m[half] - mx) * scale_log2), c2 = exp2f((m2 - mx) * scale_log2);
    float sum = l[half] * c1 + mine[2 + half] * c2;
    sum += __shfl_xor_sync(0xffffffffu, sum, 1);
    sum += __shfl_xor_sync(0xffffffffu, sum, 2);
    const float inv = 1.f / sum;
    const int r = half ? r_hi : r_lo;
    if (r < T) {
#pragma unroll
      for (int d = 0; d < D / 8; ++d)
        *reinterpret_cast<uint32_t*>(y + ((long long)b * T + r) * C + h * D + d * 8 + cc) =
            pack_bf16x2((o[d][2 * half] * c1 + mine[4 + d * 4 + 2 * half] * c2) * inv,
                        (o[d][2 * half + 1] * c1 + mine[4 + d * 4 + 2 * half + 1] * c2) * inv);
    }
  }
}

}  // namespace dion

// The blocks' weights and buffers; mirrored by models/inference.py.
struct DionStack {
  NormFn norm;
  const void* const* weights;   // host array: q, k, v, projection, MLP in, MLP out of every block
  const void* const* cos;       // host arrays: bf16 [T, D / 2] of every block
  const void* const* sin;
  float* x;                     // fp32 [rows, C]: embedded tokens, overwritten
  void* h;                      // bf16 [rows, C]: the result
  void* xb;                     // bf16 [rows, C]
  void* qkv;                    // bf16 [rows, 3 C]
  void* y;                      // bf16 [rows, C]
  void* act;                    // bf16 [rows, F]
  float* ss;                    // fp32 [rows, C / 32]
  float* rstd;                  // fp32 [rows]
  int* status;
  int blocks, B, T, H, D, F, w_dt;
  float eps_x, eps_qk;
};

namespace dion {

typedef CUresult (*EncodeTiledFnI)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static int map_rows(CUtensorMap* map, const void* ptr, int rows, int cols) {
  static EncodeTiledFnI enc = [] {
    void* sym = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      sym = nullptr;
    return reinterpret_cast<EncodeTiledFnI>(sym);
  }();
  if (!enc) return -1;
  const cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, 1};
  const cuuint64_t strides[2] = {(cuuint64_t)cols * 2, (cuuint64_t)cols * 2 * (cuuint64_t)rows};
  const cuuint32_t box[3] = {64, 128, 1};
  return encode_bf16_3d(enc, map, ptr, dims, strides, box);
}

// Launch with leave to start before the preceding kernel has ended (see wait_for_previous_kernel).
template <class Kernel, class... Args>
static int launch_early(Kernel kernel, dim3 grid, int threads, int dyn, int cluster,
                        cudaStream_t stream, const Args&... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads, 1, 1);
  cfg.dynamicSmemBytes = dyn;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = cluster > 0 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, args...) != cudaSuccess) {
    cudaGetLastError();
    return -22;
  }
  return 0;
}

template <int BN, int SLABS>
static int launch_skinny(const CUtensorMap& mx, const SkinnyArgs& a, int splits, cudaStream_t stream) {
  constexpr int kRing = SLABS < kSkRing ? SLABS : kSkRing;
  constexpr int kOperands = kRing * kSkABytes + SLABS * BN * 128, kPart = 128 * (BN + 4) * 4;
  constexpr int kDyn = (kOperands > kPart ? kOperands : kPart) + 1024;
  static const bool configured =
      cudaFuncSetAttribute(skinny_kernel<BN, SLABS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           kDyn) == cudaSuccess;
  if (!configured) return -21;
  return launch_early(skinny_kernel<BN, SLABS>,
                      dim3(splits, (a.N + BN - 1) / BN, (a.rows + 127) / 128), kSkThreads, kDyn,
                      splits, stream, mx, a);
}

// 64-column tiles where they make enough CTAs (they read X half as often), else 32; K split over
// as few CTAs as bring the grid to 132, none of them empty, and as hold a CTA's share of K in
// registers (256 elements for 64 columns, 512 for 32).  -> columns, or 0 where K is too long.
static int sk_shape(int rows, int N, int K, int* splits, int* slabs) {
  const int total = (K + 63) / 64, tiles_m = (rows + 127) / 128;
  int best_bn = 0, best_ctas = 0;
  for (int bn = 64; bn >= 32; bn /= 2) {
    for (int s = 1; s <= 8 && best_ctas < 132; ++s) {
      const int per = (total + s - 1) / s;
      if (per > (bn == 64 ? 4 : 8) || per * (s - 1) >= total) continue;
      const int ctas = (N + bn - 1) / bn * tiles_m * s;
      if (ctas > best_ctas) {
        best_ctas = ctas; best_bn = bn; *splits = s; *slabs = per;
      }
    }
  }
  return best_bn;
}

static int skinny(const CUtensorMap& mx, SkinnyArgs& a, cudaStream_t s) {
  int splits = 1;
  const int bn = sk_shape(a.rows, a.N, a.K, &splits, &a.slabs);
  if (bn == 64) {
    switch (a.slabs) {
      case 1: return launch_skinny<64, 1>(mx, a, splits, s);
      case 2: return launch_skinny<64, 2>(mx, a, splits, s);
      case 3: return launch_skinny<64, 3>(mx, a, splits, s);
      default: return launch_skinny<64, 4>(mx, a, splits, s);
    }
  }
  if (bn == 32) {
    switch (a.slabs) {
      case 1: return launch_skinny<32, 1>(mx, a, splits, s);
      case 2: return launch_skinny<32, 2>(mx, a, splits, s);
      case 3: case 4: return launch_skinny<32, 4>(mx, a, splits, s);
      case 5: case 6: return launch_skinny<32, 6>(mx, a, splits, s);
      default: return launch_skinny<32, 8>(mx, a, splits, s);
    }
  }
  return -20;
}

template <int D>
static int launch_attention(const DionStack* p, int block, cudaStream_t s) {
  static const bool configured =
      cudaFuncSetAttribute(short_attention_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           att_smem<D>()) == cudaSuccess;
  if (!configured) return -21;
  const float scale_log2 = 1.4426950408889634f / sqrtf((float)D);   // log2(e) / sqrt(D)
  return launch_early(short_attention_kernel<D>, dim3((p->T + 63) / 64, p->H, p->B), kAttThreads,
                      att_smem<D>(),
                      0, s, static_cast<const __nv_bfloat16*>(p->qkv),
                      static_cast<const __nv_bfloat16*>(p->cos[block]),
                      static_cast<const __nv_bfloat16*>(p->sin[block]),
                      static_cast<__nv_bfloat16*>(p->y), p->T, p->H, p->eps_qk, scale_log2);
}

}  // namespace dion

// All blocks of the stack for `rows` = B * T rows: x -> h, the normalized stream.  Widths up to C =
// 1024, F = 4096 (a CTA's share of K has to fit its registers), head dimensions 32, 64 and 128.
DION_EXPORT int dion_infer_stack(const DionStack* p, void* stream) {
  const int C = p->H * p->D, rows = p->B * p->T;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  if ((p->D != 32 && p->D != 64 && p->D != 128) || C > 4096 || p->F > 4096 || p->F % 8 ||
      p->H > 65535 || p->B > 65535)
    return -10;
  CUtensorMap m_x, m_y, m_act;
  if (map_rows(&m_x, p->xb, rows, C) != 0 || map_rows(&m_y, p->y, rows, C) != 0 ||
      map_rows(&m_act, p->act, rows, p->F) != 0)
    return -11;
  stream_in_kernel<<<(rows + 7) / 8, 256, 0, s>>>(p->x, static_cast<__nv_bfloat16*>(p->xb), p->ss,
                                                  rows, C);
  if (cudaGetLastError() != cudaSuccess) return -12;
  int splits, slabs;
  const int bn_proj = sk_shape(rows, C, C, &splits, &slabs), bn_out = sk_shape(rows, C, p->F, &splits, &slabs);
  if (bn_proj == 0 || bn_out == 0) return -20;
  SkinnyArgs a = {};
  a.w_dt = p->w_dt; a.rows = rows; a.status = p->status; a.eps = p->eps_x;
  a.x = p->x; a.xb = static_cast<__nv_bfloat16*>(p->xb); a.ss_out = p->ss;
  for (int b = 0; b < p->blocks; ++b) {
    const void* const* w = p->weights + 6 * b;
    // q, k, v
    a.w0 = w[0]; a.w1 = w[1]; a.w2 = w[2]; a.n_per_w = C; a.N = 3 * C; a.K = C;
    a.ss = p->ss; a.parts = b == 0 ? 1 : (C + bn_out - 1) / bn_out;
    a.epi = kSkStore; a.Y = static_cast<__nv_bfloat16*>(p->qkv);
    int rc = skinny(m_x, a, s);
    if (rc == 0)
      rc = p->D == 32 ? launch_attention<32>(p, b, s)
           : p->D == 64 ? launch_attention<64>(p, b, s) : launch_attention<128>(p, b, s);
    if (rc != 0) return rc;
    // projection and residual
    a.w0 = w[3]; a.N = C; a.ss = nullptr; a.epi = kSkResidual;
    rc = skinny(m_y, a, s);
    if (rc != 0) return rc;
    // MLP
    a.w0 = w[4]; a.n_per_w = a.N = p->F; a.ss = p->ss; a.parts = (C + bn_proj - 1) / bn_proj;
    a.epi = kSkRelu2; a.Y = static_cast<__nv_bfloat16*>(p->act);
    rc = skinny(m_x, a, s);
    if (rc != 0) return rc;
    a.w0 = w[5]; a.n_per_w = a.N = C; a.K = p->F; a.ss = nullptr; a.epi = kSkResidual;
    rc = skinny(m_act, a, s);
    if (rc != 0) return rc;
  }
  return p->norm(p->x, 0, nullptr, 0, nullptr, p->h, 1, p->rstd, rows, C, p->eps_x, stream);
}

// ---- next-token logits ------------------------------------------------------------------------
// out[r][n] = float(bf16(h[r] . bf16(W[n]))) for a handful of rows r: the weights of the output head
// are read once as they are (154 MB in fp32 for GPT-160M's 50304 words, 24 us of memory; rounded to
// bf16 and multiplied by the library 46 us).  One warp takes NV words at a time, a lane four
// consecutive elements of every 128, with all their loads in flight.
namespace dion {

template <int R, int NV>
__global__ void __launch_bounds__(256)
head_kernel(const __nv_bfloat16* __restrict__ h, long long h_stride, const void* __restrict__ W,
            int w_dt, float* __restrict__ out, int V, int C) {
  constexpr int CH = 8;                 // C <= 1024
  const int lane = threadIdx.x & 31;
  float x[R][CH][4];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const int k = c * 128 + lane * 4;
#pragma unroll
      for (int e = 0; e < 4; ++e) x[r][c][e] = 0.f;
      if (k < C) {
        const uint2 u = *reinterpret_cast<const uint2*>(h + r * h_stride + k);
        const float2 lo = unpack_bf16x2(u.x), hi = unpack_bf16x2(u.y);
        x[r][c][0] = lo.x; x[r][c][1] = lo.y; x[r][c][2] = hi.x; x[r][c][3] = hi.y;
      }
    }
  const int warps = gridDim.x * 8;
  for (int n0 = (blockIdx.x * 8 + (threadIdx.x >> 5)) * NV; n0 < V; n0 += warps * NV) {
    float4 w[NV][CH];
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const int k = c * 128 + lane * 4;
        w[v][c] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k < C && n0 + v < V) {
          const long long at = (long long)(n0 + v) * C + k;
          if (w_dt == 0) {
            w[v][c] = __ldg(reinterpret_cast<const float4*>(static_cast<const float*>(W) + at));
          } else {
            const uint2 u =
                __ldg(reinterpret_cast<const uint2*>(static_cast<const __nv_bfloat16*>(W) + at));
            const float2 lo = unpack_bf16x2(u.x), hi = unpack_bf16x2(u.y);
            w[v][c] = make_float4(lo.x, lo.y, hi.x, hi.y);
          }
        }
      }
    float acc[NV][R];
#pragma unroll
    for (int v = 0; v < NV; ++v) {
#pragma unroll
      for (int r = 0; r < R; ++r) acc[v][r] = 0.f;
#pragma unroll
      for (int c = 0; c < CH; ++c) {
        const float2 lo = unpack_bf16x2(pack_bf16x2(w[v][c].x, w[v][c].y));
        const float2 hi = unpack_bf16x2(pack_bf16x2(w[v][c].z, w[v][c].w));
#pragma unroll
        for (int r = 0; r < R; ++r)
          acc[v][r] += lo.x * x[r][c][0] + lo.y * x[r][c][1] + hi.x * x[r][c][2] + hi.y * x[r][c][3];
      }
    }
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int r = 0; r < R; ++r) {
        float a = acc[v][r];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if (lane == 0 && n0 + v < V)
          out[(long long)r * V + n0 + v] = __bfloat162float(__float2bfloat16(a));
      }
  }
}

}  // namespace dion

// h: `rows` (1 to 4) vectors of C bf16, h_stride elements apart; W [V, C]; C a multiple of 4 up to
// 1024, 16-byte aligned weights, 8-byte aligned h.
DION_EXPORT int dion_infer_head(const void* h, long long h_stride, const void* W, int w_dt, float* out,
                                int rows, int V, int C, int sms, void* stream) {
  if (rows <= 0 || V <= 0) return 0;
  if (rows > 4 || C <= 0 || C > 1024 || (C & 3) || (h_stride & 3) ||
      (reinterpret_cast<uintptr_t>(W) & 15) || (reinterpret_cast<uintptr_t>(h) & 7))
    return -10;
  const __nv_bfloat16* hp = static_cast<const __nv_bfloat16*>(h);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int grid = 2 * sms;
  switch (rows) {
    case 1: head_kernel<1, 4><<<grid, 256, 0, s>>>(hp, h_stride, W, w_dt, out, V, C); break;
    case 2: head_kernel<2, 2><<<grid, 256, 0, s>>>(hp, h_stride, W, w_dt, out, V, C); break;
    case 3: head_kernel<3, 2><<<grid, 256, 0, s>>>(hp, h_stride, W, w_dt, out, V, C); break;
    default: head_kernel<4, 1><<<grid, 256, 0, s>>>(hp, h_stride, W, w_dt, out, V, C);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -1;
}
