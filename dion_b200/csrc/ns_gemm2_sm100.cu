// Two-CTA (cta_group::2) variant of the Newton-Schulz GEMM for sm_100a:
//
//     C[b] = alpha * s_b^pa * A[b] * op(B[b]) + beta * s_b^pb * D[b]
//
// A pair of CTAs on neighbouring SMs (a cluster of two) computes one 256x256 output tile with
// tcgen05.mma.cta_group::2 (UMMA 256x256x16).  Each CTA stages only its own 128 rows of A and its
// own 128 of the 256 columns of B per 64-wide K slab (32 KB instead of the 48 KB a lone CTA needs
// for a 128x256 tile), which takes the shared-memory traffic per MMA cycle below the SM's
// bandwidth - the limit the single-CTA kernel in ns_gemm_sm100.cu runs into.  Loads are plain TMA
// (cp.async.bulk.tensor with .cta_group::2 so that both CTAs' transfers complete on the leader's
// barrier; no multicast).  The leader CTA's MMA thread issues the instructions for the pair and
// releases stages / publishes accumulators in both CTAs with a cluster-multicast tcgen05.commit.
// Each CTA drains its own half (128 TMEM lanes) of the accumulator in its epilogue warps, 64 or 32
// columns at a time through shared memory: D arrives by TMA (each group's next sub-tile is in flight),
// each thread combines its row in place in the swizzled buffer, and the buffer leaves by TMA store.
// In symmetric mode only tiles on or above the diagonal are computed; the warps of an off-diagonal
// tile also store their registers at the mirrored position, 64 bytes of a row at a time.
//
// Operand layouts and the epilogue arithmetic are the same as in the single-CTA kernel.  All waits
// are bounded; the epilogue threads meet at a barrier that also ANDs their wait results, so a
// timeout makes all of them leave together.
#include "common.cuh"
#include "tmap_cache.h"

namespace dion {

constexpr int BM2 = 128;   // rows per CTA (256 per pair)
constexpr int BN2 = 256;   // columns per pair (128 loaded by each CTA)
constexpr int BK2 = 64;
// Groups of four warps drain a tile in turn, each through two sub-tile buffers of its own: a buffer is
// written again only after its store has read it and, with D, the next D has arrived, so that one D
// sub-tile is always in flight.  A sub-tile is a chain of latencies (D, TMEM, arithmetic, barrier,
// store): one group takes 4.7 us a tile (7.2 with D), more than the 3.3 us that K = 768 multiplies
// for, two take 3.6 (5.3).  The mirrored copy of symmetric tiles doubles the instructions, so these
// have four groups on half as wide sub-tiles: polynomial 64 x 768^3 66.5 -> 59.4 us, Gram 48 x 768^3 48 ->
// 44 us.  Plain tiles gain nothing from that (update of 64 matrices 768 x 3072: 213 us either way).
// With 32 KB per operand stage:
//   plain       5 stages + 4 buffers of 128 x 64
//   symmetric   5 stages + 8 buffers of 128 x 32
constexpr int kABytes2 = BM2 * BK2 * 2;          // 16 KB
constexpr int kBBytes2 = (BN2 / 2) * BK2 * 2;    // 16 KB
constexpr int kStageBytes2 = kABytes2 + kBBytes2;
// The composed forms (see dion_ns_compose2) are kernels of their own, so that the vectors that
// their addends are scaled with cost the others no registers.
enum : int { kAddScalar = 0, kAddDiag = 1, kAddVector = 2 };
template <int STAGES, int BUFS, int COLS, int GROUPS, int ADD, bool SYM>
struct Cfg2 {
  static constexpr int kStages = STAGES, kDC = BUFS, kCols = COLS, kGroups = GROUPS, kAdd = ADD;
  static constexpr bool kSym = SYM;
  static constexpr int kThreads = 64 + GROUPS * 128;   // producer, MMA, groups of four warps
  static constexpr int kBufBytes = BM2 * COLS * 2;     // a sub-tile: two boxes of 64 rows
  static constexpr int kDynBytes = STAGES * kStageBytes2 + BUFS * kBufBytes + 1024;
};
using CfgPlain = Cfg2<5, 4, 64, 2, kAddScalar, false>;
using CfgSym = Cfg2<5, 8, 32, 4, kAddScalar, true>;
using CfgSymDiag = Cfg2<5, 8, 32, 4, kAddDiag, true>;
using CfgPlainVec = Cfg2<5, 4, 64, 2, kAddVector, false>;
constexpr uint32_t kTmemCols2 = 2 * BN2;

// Epilogue forms: C = alpha*acc + beta*D | relu(alpha*acc)^2 | alpha*acc * 2*sqrt(D).
enum : int { kEpiAxpby = 0, kEpiRelu2 = 1, kEpiMul2Sqrt = 2 };

struct Gemm2Args {
  int batch, M, N, K;
  const __nv_bfloat16* D;
  long long ldd, strideD;
  __nv_bfloat16* C;
  long long ldc, strideC;
  float alpha, beta;
  const float* scale;
  int alpha_pow, beta_pow;
  int sym;
  const int2* tiles;  // (tile_m, tile_n) in units of 256 x 256
  int tiles_per_mat;
  int total_tiles;
  int* status;
  int epi;      // kEpi*
  // ---- optional coupling to other GPUs (same meaning as in GemmArgs of ns_gemm_sm100.cu) ----
  // Gating: rows [s*rows_per_src, (s+1)*rows_per_src) of the gated operands were stored into
  // this GPU's memory by rank s, which then raised wait_flags[s] to *seq_ptr.
  const int* wait_flags;
  const int* seq_ptr;
  int n_src;
  int rows_per_src;
  int wait_a, wait_b, wait_k;
  // scale = 1 / (sqrt(sum_s scale_partials[b*n_src + s]) * scale_mult + scale_eps)
  const float* scale_partials;
  float scale_mult, scale_eps;
  // Output rows go to their owners instead of C: row r of matrix b is stored at
  // remote_c[r / rows_per_dst] + ((remote_slot + b) * rows_per_dst + r % rows_per_dst) * ldc.
  long long remote_c[8];
  int rows_per_dst;
  int remote_slot;
  // cols_per_dst > 0: split by columns instead: element (r, c) of matrix b goes to
  // remote_c[c / cols_per_dst] + ((remote_slot + b) * M + r) * cols_per_dst + c % cols_per_dst
  // (a multiple of 8 columns, so a 16-byte piece has one destination).
  int cols_per_dst;
  // ---- composed forms: symmetric matrices kept as bf16 off the diagonal and fp32 on it ----
  // kAddVector: D is scaled by beta * row_vec[b*M + row], or by beta * col_vec[b*N + column].
  // kAddDiag:   row_vec as above (null: ones).  With diag_out the diagonal leaves there as
  //             result + diag_add and is stored as zero in C; with col_vec too, the right operand's
  //             (and D's) diagonal is bf16(col_vec) and what the rounding took is added back.  With
  //             `patch` (dense [batch, M, M]) the diagonal of that matrix becomes bf16(patch_vec).
  const float* row_vec;
  const float* col_vec;
  float* diag_out;
  float diag_add;
  __nv_bfloat16* patch;
  const float* patch_vec;
};

__device__ __forceinline__ int ld_acquire_sys2(const int* p) {
  int v;
  asm volatile("ld.acquire.sys.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ float ld_volatile_f32_2(const float* p) {
  float v;
  asm volatile("ld.volatile.global.f32 %0, [%1];" : "=f"(v) : "l"(p) : "memory");
  return v;
}
// Barrier over the 128 threads of an epilogue group without a predicate (barriers 5 to 8).
__device__ __forceinline__ void epi_barrier_plain(int group) {
  asm volatile("barrier.cta.sync.aligned %0, 128;" ::"r"(5 + group) : "memory");
}

__device__ __forceinline__ uint32_t cluster_ctarank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_id_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%clusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t num_clusters_x() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%nclusterid.x;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// shared::cluster address of `local_addr` (a shared::cta address) in the CTA with rank `rank`.
__device__ __forceinline__ uint32_t map_to_cta(uint32_t local_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr)
               : "memory");
}
// TMA load whose completion is counted on a barrier that may live in the peer CTA of the pair.
__device__ __forceinline__ void tma_load_3d_pair(void* smem_dst, const CUtensorMap* map,
                                                 uint32_t bar_cluster_addr, int x, int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1, {%3, %4, %5}], [%2];" ::"r"(smem_u32(smem_dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(bar_cluster_addr), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void tmem_alloc_pair(uint32_t* smem_result, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                   smem_u32(smem_result)),
               "r"(ncols)
               : "memory");
}
__device__ __forceinline__ void tmem_relinquish_pair() {
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc_pair(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols)
               : "memory");
}
// Arrives on the barrier at the same shared-memory offset in both CTAs of the pair once all
// tcgen05.mma issued so far have completed.
__device__ __forceinline__ void tc_commit_pair(uint64_t* bar) {
  const uint16_t mask = 3;
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 "
      "[%0], %1;" ::"r"(smem_u32(bar)),
      "h"(mask)
      : "memory");
}
__device__ __forceinline__ void tc_mma_bf16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc,
                                                 uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n"
      ".reg .pred p;\n"
      "setp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n"
      "}\n" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
      : "memory");
}

// Bounded wait with cluster-scope acquire (the arrivals come from both CTAs of the pair).
__device__ __forceinline__ bool mbar_wait_bounded_cluster(uint64_t* bar, uint32_t parity) {
  WaitBudget budget;
  for (;;) {
    uint32_t ok;
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n"
        "}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (budget.spent()) return false;
  }
}

// TMA store of one box from shared memory (bulk-group completion).
__device__ __forceinline__ void tma_store_3d(const CUtensorMap* map, const void* smem_src, int x,
                                             int y, int z) {
  asm volatile(
      "cp.async.bulk.tensor.3d.global.shared::cta.bulk_group [%0, {%2, %3, %4}], [%1];" ::"l"(
          reinterpret_cast<uint64_t>(map)),
      "r"(smem_u32(smem_src)), "r"(x), "r"(y), "r"(z)
      : "memory");
}
__device__ __forceinline__ void bulk_commit_group() {
  asm volatile("cp.async.bulk.commit_group;" ::: "memory");
}
// Waits until all but the latest N committed stores have read their shared memory.
template <int N>
__device__ __forceinline__ void bulk_wait_group_read() {
  asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void bulk_wait_group_all() {
  asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
}
// Barrier over the 128 threads of an epilogue group (barriers 1 to 4) that also ANDs a predicate.
__device__ __forceinline__ bool epi_barrier_and(int group, bool mine) {
  uint32_t out;
  asm volatile(
      "{\n"
      ".reg .pred p, q;\n"
      "setp.ne.u32 q, %1, 0;\n"
      "barrier.cta.red.and.pred.aligned p, %2, 128, q;\n"
      "selp.u32 %0, 1, 0, p;\n"
      "}\n"
      : "=r"(out)
      : "r"((uint32_t)mine), "r"(1 + group)
      : "memory");
  return out != 0;
}

__device__ __forceinline__ float ipow2(float s, int p) {
  float r = 1.f;
  for (int i = 0; i < p; ++i) r *= s;
  return r;
}

template <bool A_MN, bool B_MN, class CFG>
__global__ void __launch_bounds__(CFG::kThreads, 1)
ns_gemm2_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_d,
                const Gemm2Args p) {
  constexpr int kStages2 = CFG::kStages, kDC = CFG::kDC;
  constexpr int kEpiGroups = CFG::kGroups, kSubCols = CFG::kCols, kNSub = BN2 / kSubCols;
  constexpr int kEpiBufBytes = CFG::kBufBytes;
  constexpr int kGDC = CFG::kDC / kEpiGroups;       // buffers per group
  static_assert(kGDC >= 2 && kNSub % kEpiGroups == 0, "");
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) &
                                             ~static_cast<uintptr_t>(1023));
  __shared__ __align__(8) uint64_t full_bar[kStages2];    // used in the leader CTA
  __shared__ __align__(8) uint64_t empty_bar[kStages2];   // one copy per CTA
  __shared__ __align__(8) uint64_t tfull_bar[2];          // one copy per CTA
  __shared__ __align__(8) uint64_t tempty_bar[2];         // used in the leader CTA
  __shared__ __align__(8) uint64_t dfull_bar[kDC];        // D sub-tiles, one copy per CTA
  __shared__ uint32_t tmem_base_slot;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();  // 0 = leader
  const int num_kb = (p.K + BK2 - 1) / BK2;
  const int first_tile = (int)cluster_id_x();
  const int tile_step = (int)num_clusters_x();
  let_next_kernel_start();

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages2; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 8 * kEpiGroups);  // every epilogue warp of both CTAs
    }
    for (int a = 0; a < kDC; ++a) mbar_init(&dfull_bar[a], 1);
    fence_barrier_init();
    fence_proxy_async();
    prefetch_tmap(&map_a);
    prefetch_tmap(&map_b);
    prefetch_tmap(&map_c);
    if (p.D) prefetch_tmap(&map_d);
  }
  if (warp == 1) {
    tmem_alloc_pair(&tmem_base_slot, kTmemCols2);
    tmem_relinquish_pair();
  }
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();  // barriers of both CTAs are initialised before anyone signals them
  tc_fence_after();
  const uint32_t tmem_base = tmem_base_slot;

  if (warp == 0) {
    // ------------------------------ TMA producer (both CTAs) ------------------------------
    if (lane == 0) {
      uint32_t stage = 0, phase = 0;
      bool ok = true;
      uint32_t ready_mask = 0;
      wait_for_previous_kernel();
      const int seq = p.wait_flags ? *p.seq_ptr : 0;
      // Waits (bounded) until every source rank owning rows [r0, r1] has delivered.
      auto sources_ready = [&](int r0, int r1) -> bool {
        for (int src = r0 / p.rows_per_src; src <= r1 / p.rows_per_src && src < p.n_src; ++src) {
          if (ready_mask & (1u << src)) continue;
          if (!flag_wait_bounded(p.wait_flags + src, seq)) {
            report_peer_timeout(p.status, src, seq, ld_acquire_sys2(p.wait_flags + src));
            return false;
          }
          ready_mask |= 1u << src;
          // peer stores (generic proxy) must be visible to the TMA reads (async proxy)
          asm volatile("fence.proxy.async;" ::: "memory");
        }
        return true;
      };
      for (int t = first_tile; t < p.total_tiles && ok; t += tile_step) {
        const int b = t / p.tiles_per_mat;
        const int2 tt = p.tiles[t - b * p.tiles_per_mat];
        const int row0 = tt.x * 256 + (int)cta * BM2;          // this CTA's rows of A
        const int col0 = tt.y * BN2 + (int)cta * (BN2 / 2);    // this CTA's columns of B
        if (p.wait_flags) {
          // Gate this CTA's share of the tile on the ranks that own its operand rows.
          if (p.wait_a && row0 < p.M) {
            const int r1 = row0 + BM2 - 1 < p.M ? row0 + BM2 - 1 : p.M - 1;
            ok = sources_ready(row0, r1);
          }
          if (ok && p.wait_b && col0 < p.N) {
            const int r1 = col0 + BN2 / 2 - 1 < p.N ? col0 + BN2 / 2 - 1 : p.N - 1;
            ok = sources_ready(col0, r1);
          }
          if (!ok) break;
        }
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded(&empty_bar[stage], phase ^ 1)) {
            atomicExch(p.status, kStatusTimeoutEmpty);
            ok = false;
            break;
          }
          if (p.wait_flags && p.wait_k) {
            // K-slab gating: rows [kb*BK2, +BK2) of MN-major operands belong to these sources.
            const int k1 = kb * BK2 + BK2 - 1 < p.K ? kb * BK2 + BK2 - 1 : p.K - 1;
            if (!sources_ready(kb * BK2, k1)) {
              ok = false;
              break;
            }
          }
          uint8_t* sa = smem + stage * kStageBytes2;
          uint8_t* sb = sa + kABytes2;
          const uint32_t bar = map_to_cta(smem_u32(&full_bar[stage]), 0);
          if (cta == 0) mbar_expect_tx(&full_bar[stage], 2 * kStageBytes2);
          if (!A_MN) {
            tma_load_3d_pair(sa, &map_a, bar, kb * BK2, row0, b);
          } else {
#pragma unroll
            for (int c = 0; c < BM2 / 64; ++c)
              tma_load_3d_pair(sa + c * (BK2 * 128), &map_a, bar, row0 + c * 64, kb * BK2, b);
          }
          if (!B_MN) {
            tma_load_3d_pair(sb, &map_b, bar, kb * BK2, col0, b);
          } else {
#pragma unroll
            for (int c = 0; c < (BN2 / 2) / 64; ++c)
              tma_load_3d_pair(sb + c * (BK2 * 128), &map_b, bar, col0 + c * 64, kb * BK2, b);
          }
          if (++stage == kStages2) {
            stage = 0;
            phase ^= 1;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ------------------------------ MMA issuer (leader CTA only) --------------------------
    if (lane == 0 && cta == 0) {
      constexpr uint32_t idesc = make_idesc_bf16(256, BN2, A_MN ? 1 : 0, B_MN ? 1 : 0);
      uint32_t stage = 0, phase = 0;
      uint32_t aslot = 0, aphase = 0;
      bool ok = true;
      for (int t = first_tile; t < p.total_tiles && ok; t += tile_step) {
        if (!mbar_wait_bounded_cluster(&tempty_bar[aslot], aphase ^ 1)) {
          atomicExch(p.status, kStatusTimeoutTmemEmpty);
          break;
        }
        tc_fence_after();
        const uint32_t d_tmem = tmem_base + aslot * BN2;
        for (int kb = 0; kb < num_kb; ++kb) {
          if (!mbar_wait_bounded_cluster(&full_bar[stage], phase)) {
            atomicExch(p.status, kStatusTimeoutFull);
            ok = false;
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(smem + stage * kStageBytes2);
          const uint32_t sb = sa + kABytes2;
#pragma unroll
          for (int k = 0; k < BK2 / 16; ++k) {
            const uint64_t da = A_MN ? make_smem_desc(sa + k * 2048, BK2 * 128, 1024)
                                     : make_smem_desc(sa + k * 32, 16, 1024);
            const uint64_t db = B_MN ? make_smem_desc(sb + k * 2048, BK2 * 128, 1024)
                                     : make_smem_desc(sb + k * 32, 16, 1024);
            tc_mma_bf16_pair(d_tmem, da, db, idesc, (kb | k) != 0 ? 1u : 0u);
          }
          tc_commit_pair(&empty_bar[stage]);
          if (++stage == kStages2) {
            stage = 0;
            phase ^= 1;
          }
        }
        if (!ok) break;
        tc_commit_pair(&tfull_bar[aslot]);
        aslot ^= 1;
        if (aslot == 0) aphase ^= 1;
      }
    }
  } else {
    // ------------------------------ epilogue (both CTAs) ----------------------------------
    // The 128 x 256 half-tile of this CTA is drained in sub-tiles of 64 or 32 columns, in turn by the
    // groups of warps.  D arrives by TMA into a shared-memory buffer (prefetched), each thread
    // combines its row in place, and the buffer leaves by TMA store; with `sym`, off-diagonal tiles
    // are also stored at the mirrored position.  g counts the sub-tiles of this group.
    const int grp = (warp - 2) >> 2;
    const int lane_grp = warp & 3;
    const int row_in_tile = lane_grp * 32 + lane;
    const bool elected = (warp == 2 + 4 * grp && lane == 0);
    const bool has_d = p.D != nullptr;
    const int epi = p.epi;
    constexpr uint32_t kBoxBytes = kEpiBufBytes / 2;
    // Position of 16-byte piece c of row r in a box: r * row bytes + (c ^ swizzle(r)) * 16.
    auto swizzle = [](uint32_t r) { return kSubCols == 64 ? r & 7u : (r >> 1) & 3u; };
    const uint32_t row_off = (uint32_t)(row_in_tile >> 6) * kBoxBytes +
                             (uint32_t)(row_in_tile & 63) * (kSubCols * 2);
    const uint32_t row_sw = swizzle(row_in_tile);
    uint8_t* dc_base = smem + kStages2 * kStageBytes2 + grp * kGDC * kEpiBufBytes;
    uint64_t* dfull = dfull_bar + grp * kGDC;
    wait_for_previous_kernel();

    // Iterator over the sub-tiles this group will process, in order (used for the D prefetch).
    // Only the last column of tiles can be narrower than 256 columns.
    int pf_t = first_tile, pf_s = grp;
    auto pf_skip = [&]() {   // to the next sub-tile of this group that exists
      while (pf_t < p.total_tiles) {
        const int2 tt = p.tiles[pf_t % p.tiles_per_mat];
        if (pf_s < kNSub && tt.y * BN2 + pf_s * kSubCols < p.N) break;
        pf_s = grp;
        pf_t += tile_step;
      }
    };
    auto pf_valid = [&]() { return pf_t < p.total_tiles; };
    auto pf_coords = [&](int& b, int& r0, int& c0) {
      b = pf_t / p.tiles_per_mat;
      const int2 tt = p.tiles[pf_t - b * p.tiles_per_mat];
      r0 = tt.x * 256 + (int)cta * BM2;
      c0 = tt.y * BN2 + pf_s * kSubCols;
    };
    auto pf_advance = [&]() {
      pf_s += kEpiGroups;
      pf_skip();
    };
    if (elected && has_d) pf_skip();
    uint32_t d_issued = 0;  // D sub-tiles requested so far (elected thread)
    auto issue_d = [&](uint32_t g) {
      d_issued = g + 1;
      int b, r0, c0;
      pf_coords(b, r0, c0);
      const uint32_t buf = g % kGDC;
      uint8_t* dst = dc_base + buf * kEpiBufBytes;
      mbar_expect_tx(&dfull[buf], kEpiBufBytes);
      tma_load_3d(dst, &map_d, &dfull[buf], c0, r0, b);
      tma_load_3d(dst + kBoxBytes, &map_d, &dfull[buf], c0, r0 + 64, b);
    };
    if (elected && has_d) {
      for (uint32_t g0 = 0; g0 < kGDC && pf_valid(); ++g0) {
        issue_d(g0);
        pf_advance();
      }
    }

    uint32_t aslot = 0, aphase = 0;
    uint32_t g = 0;  // running sub-tile count of this group
    bool ok = true;
    bool all_sources_ready = false;
    const bool remote = p.remote_c[0] != 0;
    const int epi_tid = ((warp - 2) & 3) * 32 + lane;   // 0..127
    for (int t = first_tile; t < p.total_tiles && ok; t += tile_step) {
      const int b = t / p.tiles_per_mat;
      const int2 tt = p.tiles[t - b * p.tiles_per_mat];
      bool mine_ok = __all_sync(0xffffffffu, mbar_wait_bounded(&tfull_bar[aslot], aphase));
      if (!mine_ok && lane == 0) atomicExch(p.status, kStatusTimeoutTmemFull);
      tc_fence_after();
      float sc = 1.f;
      if (p.scale != nullptr) sc = p.scale[b];
      if (p.scale_partials != nullptr && mine_ok) {
        // The norm needs every source's partial sum: wait for all of them once.
        if (!all_sources_ready) {
          int fine = 1;
          if (lane == 0) {
            const int seq = *p.seq_ptr;
            for (int src = 0; src < p.n_src && fine; ++src) {
              if (!flag_wait_bounded(p.wait_flags + src, seq)) {
                report_peer_timeout(p.status, src, seq, ld_acquire_sys2(p.wait_flags + src));
                fine = 0;
              }
            }
          }
          fine = __shfl_sync(0xffffffffu, fine, 0);
          if (!fine) mine_ok = false;
          all_sources_ready = true;
        }
        float ss = 0.f;
        for (int src = 0; src < p.n_src; ++src)
          ss += ld_volatile_f32_2(p.scale_partials + (long long)b * p.n_src + src);
        sc = 1.f / (sqrtf(ss) * p.scale_mult + p.scale_eps);
      }
      const float alpha = p.alpha * ipow2(sc, p.alpha_pow);
      const float beta = p.beta * ipow2(sc, p.beta_pow);
      const int row0 = tt.x * 256 + (int)cta * BM2;
      const bool mirror = p.sym && tt.y > tt.x;
      const int row = row0 + row_in_tile;
      float row_beta = beta;
      if (CFG::kAdd != kAddScalar && p.row_vec != nullptr)
        row_beta = row < p.M ? beta * p.row_vec[(long long)b * p.M + row] : 0.f;
      int nsub = (p.N - tt.y * BN2 + kSubCols - 1) / kSubCols;
      nsub = nsub > kNSub ? kNSub : nsub;
      // After this group's last read of the accumulator: hand the TMEM slot back to the MMA thread.
      auto release_accumulator = [&]() {
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(map_to_cta(smem_u32(&tempty_bar[aslot]), 0));
      };
      if (grp >= nsub && mine_ok) release_accumulator();   // a narrow tile: nothing to drain here
      if (grp >= nsub) ok = epi_barrier_and(grp, mine_ok);
#pragma unroll 1
      for (int s = grp; s < nsub; s += kEpiGroups, ++g) {
        const int c0 = tt.y * BN2 + s * kSubCols;
        // kAddDiag: a tile on the diagonal leaves exactly symmetric (products of matrices that
        // commute but for their rounding are not), by blocks of a warp's 32 rows x 32 columns.
        const bool diag_tile = CFG::kAdd == kAddDiag && tt.x == tt.y;
        const bool on_diag = diag_tile && c0 == row - lane;
        const bool above = diag_tile && c0 > row - lane;
        const uint32_t buf = g % kGDC;
        uint8_t* dc = dc_base + buf * kEpiBufBytes;
        if (elected && has_d) {
          // The stores of sub-tile g-1 have read their buffers: the next D may land there.
          bulk_wait_group_read<0>();
          if (mine_ok && g > 0 && pf_valid()) {
            issue_d(g + kGDC - 1);
            pf_advance();
          }
        }
        if (has_d && mine_ok) {
          mine_ok = __all_sync(0xffffffffu,
                               mbar_wait_bounded(&dfull[buf], (g / kGDC) & 1));
          if (!mine_ok && lane == 0) atomicExch(p.status, kStatusTimeoutFull);
        }
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(lane_grp * 32) << 16) +
                               aslot * BN2 + s * kSubCols;
        if (mine_ok) {
          // 32 columns at a time: everything is requested first, and the form is chosen once, so
          // that a warp has many instructions in flight.
#pragma unroll
          for (int half = 0; half < kSubCols / 32; ++half) {
            const int ch = c0 + half * 32;
            float v[32];
            tmem_ld_32x32(taddr + half * 32, v);
            auto cell = [&](int q) {
              return reinterpret_cast<uint4*>(dc + row_off +
                                              (((uint32_t)(half * 4 + q) ^ row_sw) << 4));
            };
            uint4 d[4];
            if (has_d) {
#pragma unroll
              for (int q = 0; q < 4; ++q) d[q] = *cell(q);
            }
            tmem_ld_wait();
            if (half == kSubCols / 32 - 1 && s + kEpiGroups >= nsub) release_accumulator();
            // f(i, D's element) for every element i of the row piece
            auto with_d = [&](auto f) {
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const uint32_t w[4] = {d[q].x, d[q].y, d[q].z, d[q].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                  const float2 x = unpack_bf16x2(w[e]);
                  f(q * 8 + 2 * e, x.x);
                  f(q * 8 + 2 * e + 1, x.y);
                }
              }
            };
            if (CFG::kAdd == kAddVector && p.col_vec != nullptr) {
              float cv[32];   // N is a multiple of 8
#pragma unroll
              for (int q = 0; q < 8; ++q) {
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (ch + q * 4 < p.N)
                  x = *reinterpret_cast<const float4*>(p.col_vec + (long long)b * p.N + ch + q * 4);
                cv[q * 4] = x.x; cv[q * 4 + 1] = x.y; cv[q * 4 + 2] = x.z; cv[q * 4 + 3] = x.w;
              }
              with_d([&](int i, float x) { v[i] = alpha * v[i] + beta * cv[i] * x; });
            } else if (CFG::kAdd != kAddScalar) {
              with_d([&](int i, float x) { v[i] = alpha * v[i] + row_beta * x; });
            } else if (has_d && !CFG::kSym && epi == kEpiMul2Sqrt) {
              with_d([&](int i, float x) { v[i] = alpha * v[i] * (2.f * sqrtf(x)); });
            } else if (has_d) {
              with_d([&](int i, float x) { v[i] = alpha * v[i] + beta * x; });
            } else if (!CFG::kSym && epi == kEpiRelu2) {
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                const float t = fmaxf(alpha * v[i], 0.f);
                v[i] = t * t;
              }
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] *= alpha;
            }
            if (CFG::kAdd == kAddDiag && on_diag && p.diag_out != nullptr) {
              float mine = 0.f;
#pragma unroll
              for (int i = 0; i < 32; ++i) {
                if (i == lane) {
                  mine = v[i];
                  v[i] = 0.f;
                }
              }
              if (row < p.M) {
                const long long at = (long long)b * p.M + row;
                mine += p.diag_add;
                if (p.col_vec != nullptr) {
                  const float f = p.col_vec[at];
                  mine += row_beta * (f - __bfloat162float(__float2bfloat16(f)));
                }
                p.diag_out[at] = mine;
                if (p.patch != nullptr)
                  p.patch[at * p.M + row] = __float2bfloat16(p.patch_vec[at]);
              }
            }
            uint32_t pk[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) pk[i] = pack_bf16x2(v[2 * i], v[2 * i + 1]);
#pragma unroll
            for (int q = 0; q < 4; ++q)
              *cell(q) = make_uint4(pk[4 * q], pk[4 * q + 1], pk[4 * q + 2], pk[4 * q + 3]);
            if (CFG::kSym && (mirror || above)) {
              // Mirrored copy, two columns at a time: neighbouring lanes swap so that each holds
              // one column of its own and the other's row, 64 bytes of C's row per half-warp.
              const int c = ch + (lane & 1), r2 = row & ~1;
              const uint32_t sel = (lane & 1) ? 0x3276u : 0x5410u;
              uint8_t* dst = reinterpret_cast<uint8_t*>(p.C + (long long)b * p.strideC +
                                                        (long long)c * p.ldc + r2);
              const long long step = 4 * p.ldc;   // two rows of C in bytes
              const bool whole = ch + 32 <= p.N && row - lane + 32 <= p.M;
#pragma unroll
              for (int i = 0; i < 16; ++i) {
                const uint32_t w =
                    __byte_perm(pk[i], __shfl_xor_sync(0xffffffffu, pk[i], 1), sel);
                if (whole || (c + 2 * i < p.N && r2 + 1 < p.M))
                  *reinterpret_cast<uint32_t*>(dst + i * step) = w;
                else if (c + 2 * i < p.N && r2 < p.M)
                  *reinterpret_cast<uint16_t*>(dst + i * step) = (uint16_t)w;
              }
            }
          }
          if (CFG::kAdd == kAddDiag && on_diag) {
            // Below the diagonal of this 32 x 32 block: the elements above it.
            __syncwarp();
            uint8_t* blk = dc + (row_off - (uint32_t)(lane * kSubCols * 2));
            auto cell2 = [&](uint32_t r, uint32_t c) {
              return reinterpret_cast<uint16_t*>(blk + r * (kSubCols * 2) +
                                                 (((c >> 3) ^ swizzle(r)) << 4) + (c & 7) * 2);
            };
#pragma unroll 4
            for (int c = 0; c < 31; ++c)
              if (c < lane) *cell2(lane, c) = *cell2(c, lane);
          }
          fence_proxy_async();
        }
        // No D: sub-tile g+1 overwrites what the store of g+1-kGDC reads.
        if (elected && !has_d) bulk_wait_group_read<kGDC - 2>();
        // Every epilogue thread reaches this barrier (all waits above are bounded); it also
        // tells whether any of them gave up.
        ok = epi_barrier_and(grp, mine_ok);
        if (!ok) break;
        if (remote) {
          // Rows leave for the ranks that own them: 16-byte stores over NVLink, eight
          // consecutive threads per 128-byte row segment of the (swizzled) sub-tile.
          constexpr int kChunks = kSubCols / 8;
          const int chunk = epi_tid % kChunks;
          if (c0 + chunk * 8 < p.N) {
#pragma unroll
            for (int i = 0; i < kChunks; ++i) {
              const int rr = epi_tid / kChunks + (128 / kChunks) * i;     // row of the 128-row half-tile
              const int grow = row0 + rr;
              if (grow < p.M) {
                const uint8_t* src = dc + (uint32_t)(rr >> 6) * kBoxBytes +
                                     (uint32_t)(rr & 63) * (kSubCols * 2) +
                                     (((uint32_t)chunk ^ swizzle(rr)) << 4);
                __nv_bfloat16* out;
                if (p.cols_per_dst > 0) {
                  const int col = c0 + chunk * 8;
                  const int dst = col / p.cols_per_dst;
                  out = reinterpret_cast<__nv_bfloat16*>(p.remote_c[dst]) +
                        ((long long)(p.remote_slot + b) * p.M + grow) * p.cols_per_dst +
                        (col - dst * p.cols_per_dst);
                } else {
                  const int dst = grow / p.rows_per_dst;
                  out = reinterpret_cast<__nv_bfloat16*>(p.remote_c[dst]) +
                        ((long long)(p.remote_slot + b) * p.rows_per_dst +
                         (grow - dst * p.rows_per_dst)) * p.ldc + c0 + chunk * 8;
                }
                *reinterpret_cast<uint4*>(out) = *reinterpret_cast<const uint4*>(src);
              }
            }
          }
          fence_proxy_async();
          epi_barrier_plain(grp);   // the buffer has been read: it may take another D sub-tile
          continue;
        }
        if (elected) {
          if (CFG::kAdd == kAddDiag) {   // boxes of 32 rows; none below the diagonal
#pragma unroll
            for (int w = 0; w < 4; ++w)
              if (row0 + w * 32 < p.M && !(diag_tile && c0 < row0 + w * 32))
                tma_store_3d(&map_c, dc + w * (kEpiBufBytes / 4), c0, row0 + w * 32, b);
          } else {
            if (row0 < p.M) tma_store_3d(&map_c, dc, c0, row0, b);
            if (row0 + 64 < p.M) tma_store_3d(&map_c, dc + kBoxBytes, c0, row0 + 64, b);
          }
          bulk_commit_group();
        }
      }
      aslot ^= 1;
      if (aslot == 0) aphase ^= 1;
    }
    if (elected) {
      bulk_wait_group_all();
      // After a timeout: let the D copies still in flight land before the CTA exits.
      if (!ok)
        for (uint32_t x = g; x < d_issued; ++x)
          mbar_wait_bounded(&dfull[x % kGDC], (x / kGDC) & 1);
    }
  }

  // Nobody leaves while the peer may still read this CTA's shared memory or signal its barriers.
  tc_fence_before();
  __syncthreads();
  cluster_sync_all();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc_pair(tmem_base, kTmemCols2);
  }
}

}  // namespace dion

// ---------------------------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------------------------
namespace dion {

typedef CUresult (*EncodeTiledFn2)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                   const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                   const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                   CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

static EncodeTiledFn2 get_encode_fn2() {
  static EncodeTiledFn2 fn = nullptr;
  if (fn) return fn;
  void* sym = nullptr;
  cudaDriverEntryPointQueryResult qres;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &sym, cudaEnableDefault, &qres) !=
          cudaSuccess ||
      qres != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn2>(sym);
  return fn;
}

static int make_map2(CUtensorMap* map, const void* ptr, int batch, int rows, int cols,
                     long long ld, long long batch_stride, int box_cols, int box_rows) {
  EncodeTiledFn2 enc = get_encode_fn2();
  if (!enc) return -1;
  cuuint64_t dims[3] = {(cuuint64_t)cols, (cuuint64_t)rows, (cuuint64_t)batch};
  cuuint64_t strides[2] = {(cuuint64_t)ld * 2, (cuuint64_t)batch_stride * 2};
  if (batch == 1) strides[1] = (cuuint64_t)ld * 2 * (cuuint64_t)rows;
  cuuint32_t box[3] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows, 1};
  return encode_bf16_3d(enc, map, ptr, dims, strides, box);  // cached when opted in
}

template <bool A_MN, bool B_MN, class CFG>
static int launch2(const CUtensorMap& ma, const CUtensorMap& mb, const CUtensorMap& mc,
                   const CUtensorMap& md, const Gemm2Args& args, cudaStream_t stream) {
  static bool configured = false;
  static int max_clusters = 0;
  auto kernel = ns_gemm2_kernel<A_MN, B_MN, CFG>;
  constexpr int kDynBytes2 = CFG::kDynBytes;
  if (!configured) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDynBytes2) !=
        cudaSuccess)
      return -3;
    cudaLaunchConfig_t probe = {};
    probe.gridDim = dim3(2 * 74, 1, 1);
    probe.blockDim = dim3(CFG::kThreads, 1, 1);
    probe.dynamicSmemBytes = kDynBytes2;
    cudaLaunchAttribute pattr[1];
    pattr[0].id = cudaLaunchAttributeClusterDimension;
    pattr[0].val.clusterDim.x = 2;
    pattr[0].val.clusterDim.y = 1;
    pattr[0].val.clusterDim.z = 1;
    probe.attrs = pattr;
    probe.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &probe) != cudaSuccess || n <= 0) {
      cudaGetLastError();
      return -5;
    }
    max_clusters = n;
    configured = true;
  }
  int clusters = args.total_tiles < max_clusters ? args.total_tiles : max_clusters;
  if (clusters <= 0) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * clusters, 1, 1);
  cfg.blockDim = dim3(CFG::kThreads, 1, 1);
  cfg.dynamicSmemBytes = kDynBytes2;
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // CTAs may start as those of the preceding kernel leave their SMs, set up and wait for it to end:
  // the launch gap, the ramp and the other kernel's last wave overlap.  Five iterations on 6 x 1000 x
  // 1536: 328 -> 286 us, 48 x 192 x 768 201 -> 166, 4 x 1024^2 266 -> 230, 12 x 768 x 3072 444 -> 428; 24 x
  // 2048^2 as before.  Launches that wait for other GPUs start in order.
  cfg.numAttrs = args.wait_flags == nullptr && args.scale_partials == nullptr &&
                 args.remote_c[0] == 0 ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kernel, ma, mb, mc, md, args) != cudaSuccess) {
    cudaGetLastError();
    return -4;
  }
  return 0;
}

template <class CFG>
static int launch2_mode(int a_mn, int b_mn, const CUtensorMap& ma, const CUtensorMap& mb,
                        const CUtensorMap& mc, const CUtensorMap& md, const Gemm2Args& args,
                        cudaStream_t stream) {
  switch ((a_mn ? 2 : 0) | (b_mn ? 1 : 0)) {
    case 0: return launch2<false, false, CFG>(ma, mb, mc, md, args, stream);
    case 1: return launch2<false, true, CFG>(ma, mb, mc, md, args, stream);
    case 2: return launch2<true, false, CFG>(ma, mb, mc, md, args, stream);
    default: return launch2<true, true, CFG>(ma, mb, mc, md, args, stream);
  }
}

}  // namespace dion

// Optional cross-GPU coupling of one launch; see the matching fields of Gemm2Args (the layout is
// shared with DionGemmExtra of ns_gemm_sm100.cu so that one host structure serves both kernels).
struct DionGemm2Extra {
  const int* wait_flags;
  const int* seq_ptr;
  int n_src, rows_per_src, wait_a, wait_b, wait_k;
  const float* scale_partials;
  float scale_mult, scale_eps;
  long long remote_c[8];
  int rows_per_dst, remote_slot;
  int cols_per_dst;
};

// Same contract as dion_ns_gemm_ex (ns_gemm_sm100.cu) for the features it has: bf16 output,
// optional D, per-batch scale, symmetric mode, gating on peer flags, norm from partial sums and
// rows stored to their owners (then C may be null); `tiles` holds (tile_m, tile_n) pairs in units
// of 256 x 256.
DION_EXPORT int dion_ns_gemm2_ex(const void* A, long long lda, long long strideA, int a_mn,
                                 const void* B, long long ldb, long long strideB, int b_mn, void* C,
                                 long long ldc, long long strideC, const void* D, long long ldd,
                                 long long strideD, int batch, int M, int N, int K, float alpha,
                                 float beta, const float* scale, int alpha_pow, int beta_pow,
                                 int sym, const void* tiles, int tiles_per_mat, int epi,
                                 int* status, void* stream, const DionGemm2Extra* ex) {
  using namespace dion;
  if (batch <= 0 || M <= 0 || N <= 0 || K <= 0) return 0;
  const bool remote = ex != nullptr && ex->remote_c[0] != 0;
  if ((lda & 7) || (ldb & 7) || (strideA & 7) || (strideB & 7) ||
      (reinterpret_cast<uintptr_t>(A) & 15) || (reinterpret_cast<uintptr_t>(B) & 15) ||
      (C == nullptr && !remote))
    return -10;
  CUtensorMap ma, mb;
  if (!a_mn) {
    if (make_map2(&ma, A, batch, M, K, lda, strideA, BK2, BM2) != 0) return -12;
  } else {
    if (make_map2(&ma, A, batch, K, M, lda, strideA, 64, BK2) != 0) return -12;
  }
  if (!b_mn) {
    if (make_map2(&mb, B, batch, N, K, ldb, strideB, BK2, BN2 / 2) != 0) return -13;
  } else {
    if (make_map2(&mb, B, batch, K, N, ldb, strideB, 64, BK2) != 0) return -13;
  }
  // C leaves (and D arrives) through TMA in boxes of 64 rows.
  if (C && ((ldc & 7) || (strideC & 7) || (reinterpret_cast<uintptr_t>(C) & 15))) return -11;
  if (D && ((ldd & 7) || (strideD & 7) || (reinterpret_cast<uintptr_t>(D) & 15))) return -11;
  if (remote && (sym || (ldc & 7) || (N & 7) || (D == nullptr && C == nullptr))) return -15;
  CUtensorMap mc, md;
  // A map needs some valid tensor even where the kernel never uses it (no D / remote output).
  const void* c_for_map = C ? C : D;
  const int sub_cols = sym ? CfgSym::kCols : CfgPlain::kCols;
  if (make_map2(&mc, c_for_map, batch, M, N, C ? ldc : ldd, C ? strideC : strideD, sub_cols,
                64) != 0)
    return -14;
  if (make_map2(&md, D ? D : C, batch, M, N, D ? ldd : ldc, D ? strideD : strideC, sub_cols,
                64) != 0)
    return -14;
  Gemm2Args a;
  a.batch = batch; a.M = M; a.N = N; a.K = K;
  a.D = static_cast<const __nv_bfloat16*>(D); a.ldd = ldd; a.strideD = strideD;
  a.C = static_cast<__nv_bfloat16*>(C); a.ldc = ldc; a.strideC = strideC;
  a.alpha = alpha; a.beta = beta; a.scale = scale; a.alpha_pow = alpha_pow; a.beta_pow = beta_pow;
  a.sym = sym;
  a.tiles = static_cast<const int2*>(tiles); a.tiles_per_mat = tiles_per_mat;
  a.total_tiles = tiles_per_mat * batch;
  a.status = status;
  a.wait_flags = nullptr; a.seq_ptr = nullptr; a.n_src = 0; a.rows_per_src = 1;
  a.wait_a = a.wait_b = a.wait_k = 0;
  a.scale_partials = nullptr; a.scale_mult = 1.f; a.scale_eps = 0.f;
  for (int i = 0; i < 8; ++i) a.remote_c[i] = 0;
  a.rows_per_dst = 1; a.remote_slot = 0; a.cols_per_dst = 0;
  a.row_vec = a.col_vec = a.patch_vec = nullptr; a.diag_out = nullptr; a.diag_add = 0.f;
  a.patch = nullptr;
  if (ex != nullptr) {
    if (ex->n_src > 8 || ex->n_src < 0) return -14;
    if ((ex->wait_flags != nullptr || ex->scale_partials != nullptr) &&
        (ex->seq_ptr == nullptr || ex->rows_per_src <= 0))
      return -16;
    a.wait_flags = ex->wait_flags; a.seq_ptr = ex->seq_ptr; a.n_src = ex->n_src;
    a.rows_per_src = ex->rows_per_src; a.wait_a = ex->wait_a; a.wait_b = ex->wait_b;
    a.wait_k = ex->wait_k;
    a.scale_partials = ex->scale_partials; a.scale_mult = ex->scale_mult;
    a.scale_eps = ex->scale_eps;
    for (int i = 0; i < 8; ++i) a.remote_c[i] = ex->remote_c[i];
    a.rows_per_dst = ex->rows_per_dst > 0 ? ex->rows_per_dst : 1;
    a.remote_slot = ex->remote_slot;
    if (ex->cols_per_dst < 0 || (ex->cols_per_dst & 7)) return -16;
    a.cols_per_dst = ex->remote_c[0] != 0 ? ex->cols_per_dst : 0;
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  a.epi = epi;
  if (epi == kEpiMul2Sqrt && D == nullptr) return -16;
  if (epi == kEpiRelu2 && D != nullptr) return -16;
  if (sym) return launch2_mode<CfgSym>(a_mn, b_mn, ma, mb, mc, md, a, s);
  return launch2_mode<CfgPlain>(a_mn, b_mn, ma, mb, mc, md, a, s);
}

DION_EXPORT int dion_ns_gemm2(const void* A, long long lda, long long strideA, int a_mn,
                              const void* B, long long ldb, long long strideB, int b_mn, void* C,
                              long long ldc, long long strideC, const void* D, long long ldd,
                              long long strideD, int batch, int M, int N, int K, float alpha,
                              float beta, const float* scale, int alpha_pow, int beta_pow, int sym,
                              const void* tiles, int tiles_per_mat, int epi, int* status,
                              void* stream) {
  return dion_ns_gemm2_ex(A, lda, strideA, a_mn, B, ldb, strideB, b_mn, C, ldc, strideC, D, ldd,
                          strideD, batch, M, N, K, alpha, beta, scale, alpha_pow, beta_pow, sym,
                          tiles, tiles_per_mat, epi, status, stream, nullptr);
}

// Whole Newton-Schulz iteration from one host call: for every coefficient triple (a, b, c)
//   A  = s^2 * X X^T            (wide / square; X^T X for tall matrices), symmetric
//   B  = b * A + c * A A        symmetric
//   X' = s * (a * X + B X)      (X B for tall matrices)
// with the input scale s applied in the first iteration only, ping-ponging between the buffers
// X (X2 from the second iteration on, when given: X is then only read) and Xalt.  All operands are
// dense [batch, rows, cols] bf16.  The result of the last
// iteration lies in Xalt when `iters` is odd, else in X (X2).  This only saves the host the 3 * iters
// trips through the Python front end; the launches are the same as issued one by one.
DION_EXPORT int dion_ns_iterate2(void* X, void* Xalt, void* X2, void* A, void* Bm, int batch, int m,
                                 int n, const float* coeffs, int iters, const float* scale,
                                 const void* tiles_gg, int n_tiles_gg, const void* tiles_mn,
                                 int n_tiles_mn, int* status, void* stream) {
  const int tall = m > n;
  const int g = tall ? n : m;
  const long long sx = (long long)m * n, sg = (long long)g * g;
  void* cur = X;
  void* nxt = Xalt;
  for (int it = 0; it < iters; ++it) {
    const float a = coeffs[3 * it], b = coeffs[3 * it + 1], c = coeffs[3 * it + 2];
    const float* sc = (it == 0) ? scale : nullptr;
    const int p2 = sc ? 2 : 0, p1 = sc ? 1 : 0;
    // Gram matrix: wide X [g, K=n] against itself; tall X read as [K=m, g] on both sides.
    int rc = dion_ns_gemm2(cur, n, sx, tall, cur, n, sx, tall, A, g, sg, nullptr, 0, 0, batch, g, g,
                           tall ? m : n, 1.f, 0.f, sc, p2, 0, 1, tiles_gg, n_tiles_gg, 0, status,
                           stream);
    if (rc != 0) return rc;
    rc = dion_ns_gemm2(A, g, sg, 0, A, g, sg, 0, Bm, g, sg, A, g, sg, batch, g, g, g, c, b, nullptr,
                       0, 0, 1, tiles_gg, n_tiles_gg, 0, status, stream);
    if (rc != 0) return rc;
    if (tall) {  // X' = a X + X B, B symmetric: given as [N, K]
      rc = dion_ns_gemm2(cur, n, sx, 0, Bm, g, sg, 0, nxt, n, sx, cur, n, sx, batch, m, n, g, 1.f, a,
                         sc, p1, p1, 0, tiles_mn, n_tiles_mn, 0, status, stream);
    } else {     // X' = a X + B X, X given as [K, N]
      rc = dion_ns_gemm2(Bm, g, sg, 0, cur, n, sx, 1, nxt, n, sx, cur, n, sx, batch, m, n, g, 1.f, a,
                         sc, p1, p1, 0, tiles_mn, n_tiles_mn, 0, status, stream);
    }
    if (rc != 0) return rc;
    void* t = cur; cur = nxt; nxt = it == 0 && X2 != nullptr ? X2 : t;
  }
  return 0;
}

namespace dion {

// One product of the composed form; every operand is dense (leading dimension = its columns).
struct ComposedProduct {
  const void* A; int a_rows, a_cols, a_mn;
  const void* B; int b_rows, b_cols, b_mn;
  void* C;
  const void* D;
  int M, N, K;
  float alpha, beta;
  const float* scale;
  int alpha_pow, beta_pow, sym;
  const float *row_vec, *col_vec;
  float* diag_out;
  float diag_add;
  void* patch;
  const float* patch_vec;
  const void* tiles; int n_tiles;
};

static int composed_product(const ComposedProduct& q, int batch, int* status, cudaStream_t stream) {
  CUtensorMap ma, mb, mc, md;
  const long long sa = (long long)q.a_rows * q.a_cols, sb = (long long)q.b_rows * q.b_cols;
  const long long sc = (long long)q.M * q.N;
  if (make_map2(&ma, q.A, batch, q.a_rows, q.a_cols, q.a_cols, sa, q.a_mn ? 64 : BK2,
                q.a_mn ? BK2 : BM2) != 0)
    return -12;
  if (make_map2(&mb, q.B, batch, q.b_rows, q.b_cols, q.b_cols, sb, q.b_mn ? 64 : BK2,
                q.b_mn ? BK2 : BN2 / 2) != 0)
    return -13;
  const int sub_cols = !q.sym ? CfgPlainVec::kCols : q.D ? CfgSymDiag::kCols : CfgSym::kCols;
  const int box_rows = q.sym && q.D ? 32 : 64;   // see the stores of kAddDiag
  if (make_map2(&mc, q.C, batch, q.M, q.N, q.N, sc, sub_cols, box_rows) != 0) return -14;
  if (make_map2(&md, q.D ? q.D : q.C, batch, q.M, q.N, q.N, sc, sub_cols, 64) != 0) return -14;
  Gemm2Args a = {};
  a.batch = batch; a.M = q.M; a.N = q.N; a.K = q.K;
  a.D = static_cast<const __nv_bfloat16*>(q.D); a.ldd = q.N; a.strideD = sc;
  a.C = static_cast<__nv_bfloat16*>(q.C); a.ldc = q.N; a.strideC = sc;
  a.alpha = q.alpha; a.beta = q.beta; a.scale = q.scale;
  a.alpha_pow = q.alpha_pow; a.beta_pow = q.beta_pow; a.sym = q.sym;
  a.tiles = static_cast<const int2*>(q.tiles); a.tiles_per_mat = q.n_tiles;
  a.total_tiles = q.n_tiles * batch;
  a.status = status; a.epi = kEpiAxpby;
  a.rows_per_src = 1; a.rows_per_dst = 1;
  a.row_vec = q.row_vec; a.col_vec = q.col_vec;
  a.diag_out = q.diag_out; a.diag_add = q.diag_add;
  a.patch = static_cast<__nv_bfloat16*>(q.patch); a.patch_vec = q.patch_vec;
  if (q.sym && q.D == nullptr) return launch2_mode<CfgSym>(q.a_mn, q.b_mn, ma, mb, mc, md, a, stream);
  if (q.sym) return launch2<false, false, CfgSymDiag>(ma, mb, mc, md, a, stream);
  return q.b_mn ? launch2<false, true, CfgPlainVec>(ma, mb, mc, md, a, stream)
                : launch2<false, false, CfgPlainVec>(ma, mb, mc, md, a, stream);
}

}  // namespace dion

// The same loop as dion_ns_iterate2 with the steps of a group composed on the small matrix:
//   A = s^2 X X^T;  Q = a I + b A + c A A;  with a second step:  A = Q A Q,  Q = (a I + b A + c A A) Q;
//   X = s Q X.
// All of these are polynomials of one symmetric matrix, so every small product is computed as a
// half.  With g = min(m, n), rho = max(m, n) / g and products counted in g^3, a group of two costs
// 3 rho + 5 where two plain steps cost 6 rho + 2: 17 against 26 at rho = 4, 53 against 98 at 16,
// the same at rho = 1.
// Z and Q are kept as bf16 off the diagonal and fp32 on it, and every small result is exactly
// symmetric.  With a bf16 diagonal the rounding of Q alone doubled the result's error, with rounding
// that differs above and below the diagonal it was a quarter larger; so it is smaller than the plain
// loop's (which rounds X, A and B in every step): 0.6-0.9 of it on gradients, on spectra with a few
// dominant directions and on decaying ones, from g = 512 and rho = 2.  Three steps in one group are
// not: the rounding that a dominant direction leaves in A grows by the square of each step's slope
// at zero (66, 16, ...) and diverges.
// A group has one or two steps.  `work` holds three matrices [batch, g, g] bf16, `vecs` three vectors
// [batch, g] fp32.  Buffers X, X2, Xalt as in dion_ns_iterate2, one swap a group; the result lies in
// Xalt after an odd number of groups, else in X (X2).
DION_EXPORT int dion_ns_compose2(void* X, void* Xalt, void* X2, void* work, float* vecs, int batch,
                                 int m, int n, const float* coeffs, const int* groups, int n_groups,
                                 const float* scale, const void* tiles_gg, int n_tiles_gg,
                                 const void* tiles_mn, int n_tiles_mn, int* status, void* stream) {
  using namespace dion;
  const int tall = m > n;
  const int g = tall ? n : m;
  if (batch <= 0 || m <= 0 || n <= 0) return 0;
  if ((m & 7) || (n & 7) || (reinterpret_cast<uintptr_t>(X) & 15)) return -10;
  const size_t mat = (size_t)batch * g * g;
  __nv_bfloat16* w = static_cast<__nv_bfloat16*>(work);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // C = alpha * Y B + beta * row_vec D, symmetric, all operands [g, g]
  auto small = [&](const void* Y, const void* B, void* C, const void* D, float alpha, float beta,
                   const float* row_vec, const float* col_vec, float* diag_out, float diag_add,
                   void* patch, const float* patch_vec) {
    ComposedProduct q = {Y, g, g, 0, B, g, g, 0, C, D, g, g, g, alpha, beta, nullptr, 0, 0, 1,
                         row_vec, col_vec, diag_out, diag_add, patch, patch_vec, tiles_gg, n_tiles_gg};
    return composed_product(q, batch, status, s);
  };
  void* cur = X;
  void* nxt = Xalt;
  for (int gr = 0, at = 0; gr < n_groups; ++gr) {
    const float* sc = gr == 0 ? scale : nullptr;
    if (groups[gr] != 1 && groups[gr] != 2) return -10;
    void* A = w;
    void* Q = w + mat;        // off the diagonal, with `q` on it
    void* Y = w + 2 * mat;    // first Q A, then the second step's Z, with `y` on its diagonal
    float* q = vecs;
    float* y = vecs + (size_t)batch * g;
    float* h = vecs + 2 * (size_t)batch * g;
    // Gram matrix: wide X [g, K = n] against itself; tall X read as [K = m, g] on both sides.
    ComposedProduct gram = {cur, m, n, tall, cur, m, n, tall, A, nullptr, g, g, tall ? m : n,
                            1.f, 0.f, sc, sc ? 2 : 0, 0, 1, nullptr, nullptr, nullptr, 0.f,
                            nullptr, nullptr, tiles_gg, n_tiles_gg};
    int rc = composed_product(gram, batch, status, s);
    if (rc != 0) return rc;
    const float* co = coeffs + 3 * at;
    at += groups[gr];
    rc = small(A, A, Q, A, co[2], co[1], nullptr, nullptr, q, co[0], nullptr, nullptr);
    if (rc != 0) return rc;
    if (groups[gr] == 2) {
      rc = small(Q, A, Y, A, 1.f, 1.f, q, nullptr, nullptr, 0.f, nullptr, nullptr);    // Q A
      if (rc == 0)
        rc = small(Q, Y, A, Y, 1.f, 1.f, q, nullptr, nullptr, 0.f, nullptr, nullptr);  // Q A Q
      // On the way Q gets its diagonal back, rounded, to be read as a whole matrix below.
      if (rc == 0) rc = small(A, A, Y, A, co[5], co[4], nullptr, nullptr, y, co[3], Q, q);
      if (rc == 0) rc = small(Y, Q, A, Q, 1.f, 1.f, y, q, h, 0.f, nullptr, nullptr);   // Z Q
      if (rc != 0) return rc;
      Q = A;
      q = h;
    }
    ComposedProduct up = {Q, g, g, 0, cur, m, n, 1, nxt, cur, m, n, g, 1.f, 1.f, sc, sc ? 1 : 0,
                          sc ? 1 : 0, 0, q, nullptr, nullptr, 0.f, nullptr, nullptr, tiles_mn,
                          n_tiles_mn};
    if (tall) {    // X' = X Q, Q symmetric: given as [N, K]
      up.A = cur; up.a_rows = m; up.a_cols = n;
      up.B = Q; up.b_rows = g; up.b_cols = g; up.b_mn = 0;
      up.row_vec = nullptr; up.col_vec = q;
    }
    rc = composed_product(up, batch, status, s);
    if (rc != 0) return rc;
    void* t = cur; cur = nxt; nxt = gr == 0 && X2 != nullptr ? X2 : t;
  }
  return 0;
}

namespace dion {

// M[b][i][i] += a for a dense bf16 batch [batch, g, g], rounded once more.
__global__ void __launch_bounds__(256)
add_diagonal_kernel(__nv_bfloat16* M, int batch, int g, float a) {
  const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
  if (i >= (long long)batch * g) return;
  __nv_bfloat16* x = M + i * g + i % g;
  *x = __float2bfloat16(__bfloat162float(*x) + a);
}

}  // namespace dion

// Gram form of the loop from one host call: R = s^2 X X^T (X^T X for tall X); for every (a, b, c):
//   Z = a I + b R + c R R,  Q = Z Q (Q = Z in the first),  R = (Z R) Z,
// where reset[it] != 0 first applies Q to X and forms R anew.  R is not brought forward where nothing
// reads it again.  `work` holds five matrices [batch, g, g]; the results go to and fro between Y0 and
// Y1, X is only read.  Returns 0 or 1, the buffer that holds the result, or an error below zero.
// 24 launches for five steps: issued one by one from Python they take 0.5 ms, more than the
// products of anything up to 8 x 1024 x 2048.
DION_EXPORT int dion_ns_gram2(const void* X, void* Y0, void* Y1, void* work, int batch, int m, int n,
                              const float* coeffs, const int* reset, int iters, const float* scale,
                              const void* tiles_sym, int n_tiles_sym, const void* tiles_gg,
                              int n_tiles_gg, const void* tiles_mn, int n_tiles_mn, int* status,
                              void* stream) {
  using namespace dion;
  const int tall = m > n;
  const int g = tall ? n : m;
  if (batch <= 0 || m <= 0 || n <= 0 || iters <= 0) return -10;
  const long long sx = (long long)m * n, sg = (long long)g * g;
  const size_t mat = (size_t)batch * g * g;
  __nv_bfloat16* w = static_cast<__nv_bfloat16*>(work);
  void *R = w, *T = w + mat, *zq[3] = {w + 2 * mat, w + 3 * mat, w + 4 * mat};
  int qi = -1;                       // the one of zq that holds Q
  const void* cur = X;
  void* out[2] = {Y0, Y1};
  int which = 0;
  const float* sc = scale;           // X itself is unnormalized until Q has been applied to it
  auto small = [&](const void* A, const void* B, int b_kn, void* C, const void* D, float alpha,
                   float beta, int sym) {
    return dion_ns_gemm2(A, g, sg, 0, B, g, sg, b_kn, C, g, sg, D, D ? g : 0, D ? sg : 0, batch, g, g,
                         g, alpha, beta, nullptr, 0, 0, sym, sym ? tiles_sym : tiles_gg,
                         sym ? n_tiles_sym : n_tiles_gg, 0, status, stream);
  };
  auto gram = [&]() {
    return dion_ns_gemm2(cur, n, sx, tall, cur, n, sx, tall, R, g, sg, nullptr, 0, 0, batch, g, g,
                         tall ? m : n, 1.f, 0.f, sc, sc ? 2 : 0, 0, 1, tiles_sym, n_tiles_sym, 0,
                         status, stream);
  };
  auto apply = [&]() {
    const void* Q = zq[qi];
    int rc;
    if (tall)
      rc = dion_ns_gemm2(cur, n, sx, 0, Q, g, sg, 0, out[which], n, sx, nullptr, 0, 0, batch, m, n, g,
                         1.f, 0.f, sc, sc ? 1 : 0, 0, 0, tiles_mn, n_tiles_mn, 0, status, stream);
    else
      rc = dion_ns_gemm2(Q, g, sg, 0, cur, n, sx, 1, out[which], n, sx, nullptr, 0, 0, batch, m, n, g,
                         1.f, 0.f, sc, sc ? 1 : 0, 0, 0, tiles_mn, n_tiles_mn, 0, status, stream);
    cur = out[which];
    which ^= 1;
    sc = nullptr;
    qi = -1;
    return rc;
  };
  int rc = gram();
  for (int it = 0; it < iters && rc == 0; ++it) {
    if (reset[it] && qi >= 0) {
      rc = apply();
      if (rc == 0) rc = gram();
      if (rc != 0) break;
    }
    const float a = coeffs[3 * it], b = coeffs[3 * it + 1], c = coeffs[3 * it + 2];
    const int zi = (qi + 1) % 3;
    void* Z = zq[zi];
    rc = small(R, R, 0, Z, R, c, b, 1);
    if (rc != 0) break;
    add_diagonal_kernel<<<(unsigned)(((long long)batch * g + 255) / 256), 256, 0,
                          static_cast<cudaStream_t>(stream)>>>(static_cast<__nv_bfloat16*>(Z), batch,
                                                               g, a);
    if (cudaGetLastError() != cudaSuccess) return -4;
    if (qi < 0) {
      qi = zi;
    } else {
      const int next = 3 - qi - zi;
      rc = small(Z, zq[qi], 1, zq[next], nullptr, 1.f, 0.f, 0);
      if (rc != 0) break;
      qi = next;
    }
    if (it + 1 < iters && !reset[it + 1]) {
      rc = small(Z, R, 0, T, nullptr, 1.f, 0.f, 0);          // Z R   (R symmetric, so R^T = R)
      if (rc == 0) rc = small(T, Z, 0, R, nullptr, 1.f, 0.f, 1);   // (Z R) Z  (Z symmetric)
    }
  }
  if (rc == 0) rc = apply();
  return rc != 0 ? (rc < 0 ? rc : -4) : which ^ 1;
}
