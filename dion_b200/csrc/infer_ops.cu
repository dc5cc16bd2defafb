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
