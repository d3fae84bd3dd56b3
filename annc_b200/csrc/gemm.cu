// GEMM dispatcher, the kn4 converters and the KPFusedBatchMatMulAddSigmoid twin.
#include <cuda_bf16.h>

#include <cstdlib>
#include <cstring>

#include "common.h"
#include "gemm.h"
#include "kn4.h"

namespace annc {
namespace gemm {

static int validate(const annc_gemm_desc& d) {
  ANNC_REQUIRE(d.a && d.b && d.c, ANNC_ERR_INVALID_ARGUMENT, "gemm: null operand");
  ANNC_REQUIRE(d.m >= 0 && d.n >= 0 && d.k >= 0 && d.batch >= 1, ANNC_ERR_INVALID_ARGUMENT,
               "gemm: bad extents");
  ANNC_REQUIRE(d.activation >= ANNC_ACT_NONE && d.activation <= ANNC_ACT_SIGMOID,
               ANNC_ERR_INVALID_ARGUMENT, "gemm: bad activation");
  ANNC_REQUIRE(d.b_format == ANNC_B_PLAIN || d.b_format == ANNC_B_KN4, ANNC_ERR_INVALID_ARGUMENT,
               "gemm: bad b_format");
  ANNC_REQUIRE(d.b_format == ANNC_B_PLAIN || !d.trans_b, ANNC_ERR_INVALID_ARGUMENT,
               "gemm: kn4 B cannot be transposed");
  ANNC_REQUIRE(d.math >= ANNC_MATH_AUTO && d.math <= ANNC_MATH_BF16, ANNC_ERR_INVALID_ARGUMENT,
               "gemm: bad math mode");
  return ANNC_OK;
}

// Pair kernel (256 x 256 tiles per two SMs, persistent; few tiles are cut in halves) or single-CTA kernel
// (128 x 128 tiles, one or two per SM, or split K inside a cluster).  With its TMA-store epilogue the pair
// kernel wins from 20 tiles on, except where the single one
//   * splits K (at most 74 tiles of one product, K from 225 on): us pair / single 300 x 3000 x 704 1.18 times,
//     2600 x 260 x 1024 1.29, 1024 x 1100 x 4096 1.48 times its time, and 1.02 at K = 256; at K = 128, unsplit, 0.89;
//   * takes the product in one round (at most 148 tiles) and the pair kernel has more tiles than it can
//     cut (more than 37 on 74 pairs): 300 x 5000 1.09 to 1.12, 2048 x 1100 1.12 to 1.15 from K = 128 to 4096.
// Otherwise, pair / single over 40 products and batches each at K = 64 to 4096, with and without an addend:
// up to 37 pair tiles 0.80 to 1.00, more than 148 single tiles 0.53 to 0.75 (149 to 222, two rounds; 10 x [520 x
// 300 x 64], 60 pair tiles for 150 of them, 1.06) and 0.85 to 1.00 (more, two per SM).  Below 20 pair tiles K is split nearly always (1024^3 17.7 / 14.6).
// A narrow C pays for 256 columns of multiplications: from n = 64 on that still hides under the memory
// traffic when K is short and the rows fill every pair (65536 x 64 x 256 24 / 28).
// Its general epilogue (beta * C, rows not of whole 16-byte pieces) is slow per tile and needs a long
// main loop to hide in.
static bool use_pair(const annc_gemm_desc& d, int math) {
  if (!pair_supported(d, math)) return false;
  if (math == ANNC_MATH_BF16 || (d.io_flags & (ANNC_IO_SOFTMAX | ANNC_IO_PAIR))) return true;
  if (!tc_supported(d, math)) return true;
  if (d.io_flags & ANNC_IO_SINGLE) return false;
  const long long pair_tiles = ((d.m + 255) / 256) * ((d.n + 255) / 256) * d.batch;
  if (d.m >= 256 && d.n >= 192 && d.k >= 1024 && pair_tiles >= 74) return true;
  if (!pair_stores_by_tma(d)) return false;
  const long long single_tiles = ((d.m + 127) / 128) * ((d.n + 127) / 128) * d.batch;
  const bool single_splits = d.batch == 1 && single_tiles * 2 <= 148 && d.k > 224;
  if (d.n >= 192 && d.m >= 192 && pair_tiles >= 20 && !single_splits && (single_tiles > 148 || pair_tiles <= 37)) return true;
  return d.n >= 64 && d.k <= 512 && pair_tiles >= 148;
}

// AUTO: tensor cores (TF32) when the shape fits a tcgen05 kernel, else CUDA cores.
static int pick_math(const annc_gemm_desc& d) {
  if (d.math == ANNC_MATH_FP32) return ANNC_MATH_FP32;
  const int want = d.math == ANNC_MATH_AUTO ? ANNC_MATH_TF32 : d.math;
  if (d.math == ANNC_MATH_AUTO && (d.io_flags & ~ANNC_IO_SINGLE) == 0 && (d.m < 64 || d.n < 16 || d.k < 32))
    return ANNC_MATH_FP32;  // tiny shapes stay on the CUDA cores
  return (tc_supported(d, want) || pair_supported(d, want)) ? want : ANNC_MATH_FP32;
}

const char* route_name(const annc_gemm_desc& d) {
  const int math = pick_math(d);
  switch (math) {
    case ANNC_MATH_TF32: return use_pair(d, math) ? "tcgen05_pair_tf32" : "tcgen05_tf32";
    case ANNC_MATH_BF16: return "tcgen05_pair_bf16";
    default: return "simt_fp32";
  }
}

namespace {

__global__ void kn4_convert_kernel(const float* src, float* dst, long long K, long long N,
                                   int to_packed) {
  const long long total = K * N;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride) {
    const long long k = e / N, n = e - k * N;
    const long long o = kn4::offset(K, N, k, n);
    if (to_packed) dst[o] = src[e];
    else dst[e] = src[o];
  }
}

// Between kn4 and [K,N], or from kn4 to [N,K] (the K-major layout the TMA route likes best), N % 4 ==
// 0: a block moves a tile of 128 (k) x 32 (n).  A thread reads 16-byte pieces of one panel (a piece never straddles
// two), whose place it works out once; for [N,K] the tile turns in shared memory (rows of 129
// floats: neither side conflicts).  Bound by memory: 2048 x 4096 in 8 to 13 us (of which 10 at the copy rate from DRAM), 38 us with one element
// and one 64-bit place computation per thread and step.
enum Relay { RELAY_KN = 0, RELAY_NK = 1, RELAY_PACK = 2 /* [K,N] -> kn4 */ };
constexpr int kRelayK = 128, kRelayN = 32;
struct RelayParams {
  const float* src;
  float* dst;
  int K, N;
  // k-chunks: 352 rows each (len0 if there is only one) up to k_uniform, then the two that share the rest
  int k_uniform, k_split, len0;
};
template <int MODE>
__global__ void __launch_bounds__(256) kn4_relay_kernel(RelayParams p) {
  constexpr bool TRANSPOSED = MODE == RELAY_NK;
  __shared__ float tile[TRANSPOSED ? kRelayN : 1][kRelayK + 1];
  const int n0 = blockIdx.x * kRelayN, k0 = blockIdx.y * kRelayK;
  const int c = threadIdx.x & 7, kk = threadIdx.x >> 3;
  const int n = n0 + 4 * c;
  if (n < p.N) {
    const kn4::Chunk nc = kn4::axis_chunk(p.N, kn4::kTileN, n);
    const kn4::Panel pn = kn4::panel_of(nc.len, n - nc.start);
    const int term = (int)(nc.start + pn.start), width = (int)pn.width, in0 = n - term;
    float4 v[kRelayK / 32];  // all on their way before the first is stored
    long long to[kRelayK / 32];
#pragma unroll
    for (int i = 0; i < kRelayK / 32; ++i) {
      const int k = k0 + kk + 32 * i;
      if (k >= p.K) continue;
      int start, len;
      if (k < p.k_uniform) {
        start = k / (int)kn4::kTileK * (int)kn4::kTileK;
        len = p.len0;
      } else if (k < p.k_split) {
        start = p.k_uniform;
        len = p.k_split - p.k_uniform;
      } else {
        start = p.k_split;
        len = p.K - p.k_split;
      }
      const long long packed = (long long)start * p.N + (long long)len * term + (long long)(k - start) * width + in0;
      const long long plain = (long long)k * p.N + n;
      to[i] = MODE == RELAY_PACK ? packed : plain;
      v[i] = __ldg(reinterpret_cast<const float4*>(p.src + (MODE == RELAY_PACK ? plain : packed)));
    }
#pragma unroll
    for (int i = 0; i < kRelayK / 32; ++i) {
      const int k = k0 + kk + 32 * i;
      if (k >= p.K) continue;
      if (TRANSPOSED) {
        tile[4 * c][kk + 32 * i] = v[i].x;
        tile[4 * c + 1][kk + 32 * i] = v[i].y;
        tile[4 * c + 2][kk + 32 * i] = v[i].z;
        tile[4 * c + 3][kk + 32 * i] = v[i].w;
      } else {
        *reinterpret_cast<float4*>(p.dst + to[i]) = v[i];
      }
    }
  }
  if (!TRANSPOSED) return;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  for (int r = threadIdx.x >> 5; r < kRelayN && n0 + r < p.N; r += 8) {
#pragma unroll
    for (int i = 0; i < kRelayK / 32; ++i) {
      const int k = k0 + lane + 32 * i;
      if (k < p.K) p.dst[(long long)(n0 + r) * p.K + k] = tile[r][lane + 32 * i];
    }
  }
}

__global__ void cast_bf16_kernel(const float* __restrict__ src, __nv_bfloat16* __restrict__ dst,
                                 long long n) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride)
    dst[i] = __float2bfloat16_rn(src[i]);
}

// [K,N] fp32 -> [N,K] bf16 through a 32 x 32 shared-memory tile.
__global__ void __launch_bounds__(256)
bf16_weight_kernel(const float* __restrict__ src, long long ldb, __nv_bfloat16* __restrict__ dst,
                   long long K, long long N) {
  __shared__ float tile[32][33];
  const long long k0 = (long long)blockIdx.y * 32, n0 = (long long)blockIdx.x * 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int r = ty; r < 32; r += 8)
    tile[r][tx] = (k0 + r < K && n0 + tx < N) ? src[(k0 + r) * ldb + n0 + tx] : 0.f;
  __syncthreads();
  for (int r = ty; r < 32; r += 8)
    if (n0 + r < N && k0 + tx < K) dst[(n0 + r) * K + k0 + tx] = __float2bfloat16_rn(tile[tx][r]);
}

}  // namespace

// Re-laying a kn4 B into a buffer of 4*K*N bytes, 16-byte aligned.  relaid_desc() says whether that pays off
// for this descriptor and returns the descriptor of the equivalent plain-layout GEMM, whose `b` the
// caller sets to that buffer, together with the form the weight has to take there (1 = [N,K], 2 =
// [K,N]); relay_kn4() runs the conversion.  Kept apart so that a caller that owns a cache of constants
// converts once (`kept`: then only the products count, not the pass over the weight).
int relaid_desc(const annc_gemm_desc& d, bool kept, annc_gemm_desc* plain) {
  if (d.b_format != ANNC_B_KN4 || d.batch != 1 || (d.n & 3) || d.m < 64) return 0;
  if (reinterpret_cast<uintptr_t>(d.b) & 15) return 0;  // the packed weight is read in 16-byte pieces
  if (d.k >= (1LL << 31) || d.n >= (1LL << 31) || (d.k + kRelayK - 1) / kRelayK > 65535) return 0;
  *plain = d;
  plain->b = nullptr;
  plain->b_format = ANNC_B_PLAIN;
  plain->ldb = d.n;
  plain->workspace = nullptr;
  plain->workspace_bytes = 0;
  // The CUDA cores take the packed form as it lies, at a place computation per element: only long K (with
  // fewer than 16 columns) pays for the pass over the weight.  __layout_matmul, us packed / re-laid: 64 x 16 x 64
  // 13 / 16, 64 rows of 8 columns K = 1024 13.5 / 15.9, 2048 20.6 / 16.4; 4000 rows 512 15.6 / 16.5, 1024 24.9 / 22.6.
  if (!kept && pick_math(*plain) == ANNC_MATH_FP32 && d.k * (d.m >= 2048 ? 2 : 1) < 2048) return 0;
  // Re-laid as [N,K] the weight takes the K-major TMA route (one 16 KB box per stage), the
  // fastest one; [K,N] is the fallback when K rows would not be 16-byte pitched.
  if ((d.k & 3) == 0 && (d.k + 31) / 32 <= 65535) {
    annc_gemm_desc t = *plain;
    t.trans_b = 1;
    t.ldb = d.k;
    if (pair_supported(t, ANNC_MATH_TF32) && use_pair(t, ANNC_MATH_TF32)) {
      *plain = t;
      return 1;
    }
  }
  if (!tc_supported(*plain, ANNC_MATH_TF32)) return 0;
  return 2;
}

static RelayParams relay_params(const float* src, float* dst, long long k, long long n) {
  constexpr int tk = (int)kn4::kTileK;
  RelayParams p{src, dst, (int)k, (int)n, (int)k, (int)k, k < tk ? (int)k : tk};
  if (k >= tk && k % tk != 0) {  // the first of the last two chunks, as kn4::axis_chunk cuts them
    p.k_uniform = (int)(k / tk - 1) * tk;
    p.k_split = p.k_uniform + (int)kn4::axis_chunk(k, tk, p.k_uniform).len;
  }
  return p;
}
static dim3 relay_grid(long long k, long long n) {
  return dim3((unsigned)((n + kRelayN - 1) / kRelayN), (unsigned)((k + kRelayK - 1) / kRelayK));
}

void relay_kn4(const float* packed, float* ws, long long k, long long n, int form, cudaStream_t s) {
  const RelayParams p = relay_params(packed, ws, k, n);
  if (form == 1) kn4_relay_kernel<RELAY_NK><<<relay_grid(k, n), 256, 0, s>>>(p);
  else kn4_relay_kernel<RELAY_KN><<<relay_grid(k, n), 256, 0, s>>>(p);
}

// kn4 <-> [K,N], any extents: 16-byte pieces where they exist (2048 x 4096: 9 us against 54 us one element
// at a time), except for small matrices with enough rows that a block's threads walk several in turn
// (128 x 256 2.2 us / 2.0 us; 200 x 256 2.2 / 2.3, 64 x 512 1.9 / 2.0).
static void convert_kn4(const float* src, float* dst, long long k, long long n, bool pack, cudaStream_t s) {
  const bool pieces = n % 4 == 0 && n < (1LL << 31) && (k <= 64 || k * n > 32768) && (k + kRelayK - 1) / kRelayK <= 65535 &&
                      ((reinterpret_cast<uintptr_t>(src) | reinterpret_cast<uintptr_t>(dst)) & 15) == 0;
  if (pieces) {
    const RelayParams p = relay_params(src, dst, k, n);
    if (pack) kn4_relay_kernel<RELAY_PACK><<<relay_grid(k, n), 256, 0, s>>>(p);
    else kn4_relay_kernel<RELAY_KN><<<relay_grid(k, n), 256, 0, s>>>(p);
    return;
  }
  long long g = (k * n + 255) / 256;
  if (g > 148 * 32) g = 148 * 32;
  kn4_convert_kernel<<<(unsigned)g, 256, 0, s>>>(src, dst, k, n, pack ? 1 : 0);
}

static bool unpack_kn4_into_workspace(const annc_gemm_desc& d, cudaStream_t s, annc_gemm_desc* plain) {
  if (!d.workspace || (reinterpret_cast<uintptr_t>(d.workspace) & 15) ||
      d.workspace_bytes < (size_t)d.k * (size_t)d.n * sizeof(float))
    return false;
  const int form = relaid_desc(d, /*kept=*/false, plain);
  if (!form) return false;
  plain->b = static_cast<const float*>(d.workspace);
  relay_kn4(d.b, static_cast<float*>(d.workspace), d.k, d.n, form, s);
  return true;
}

}  // namespace gemm
}  // namespace annc

using namespace annc;

extern "C" {

int annc_gemm_run(const annc_gemm_desc* desc, void* stream) {
  ANNC_REQUIRE(desc, ANNC_ERR_INVALID_ARGUMENT, "gemm: null descriptor");
  ANNC_TRY(gemm::validate(*desc));
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  const int math = gemm::pick_math(*desc);
  if (desc->math != ANNC_MATH_AUTO && desc->math != math)
    return fail(ANNC_ERR_UNSUPPORTED, "gemm: shape not supported by the requested math mode");
  if (math == ANNC_MATH_FP32) {
    if ((desc->io_flags & ~ANNC_IO_SINGLE) != 0)
      return fail(ANNC_ERR_UNSUPPORTED, "gemm: io_flags need a tensor-core route this shape does not fit");
    return gemm::run_simt(*desc, s);
  }
  annc_gemm_desc plain;
  if (gemm::unpack_kn4_into_workspace(*desc, s, &plain))
    return gemm::use_pair(plain, math) ? gemm::run_pair(plain, math, s) : gemm::run_tc(plain, math, s);
  return gemm::use_pair(*desc, math) ? gemm::run_pair(*desc, math, s) : gemm::run_tc(*desc, math, s);
}

const char* annc_gemm_kernel_name(const annc_gemm_desc* desc) {
  if (!desc) return "";
  return gemm::route_name(*desc);
}

int annc_cast_bf16_dev(const float* src, void* dst_bf16, int64_t n, void* stream) {
  ANNC_REQUIRE(src && dst_bf16 && n >= 0, ANNC_ERR_INVALID_ARGUMENT, "cast: bad arguments");
  if (n == 0) return ANNC_OK;
  long long g = (n + 255) / 256;
  if (g > 148 * 16) g = 148 * 16;
  gemm::cast_bf16_kernel<<<(unsigned)g, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      src, static_cast<__nv_bfloat16*>(dst_bf16), n);
  ANNC_CUDA(cudaGetLastError());
  return ANNC_OK;
}

int annc_bf16_weight_dev(const float* b_kn, int64_t ldb, void* b_nk_bf16, int64_t k, int64_t n,
                         void* stream) {
  ANNC_REQUIRE(b_kn && b_nk_bf16 && k >= 1 && n >= 1 && ldb >= n, ANNC_ERR_INVALID_ARGUMENT,
               "bf16 weight: bad arguments");
  dim3 grid((unsigned)((n + 31) / 32), (unsigned)((k + 31) / 32));
  ANNC_REQUIRE(grid.y <= 65535, ANNC_ERR_UNSUPPORTED, "bf16 weight: k too large");
  gemm::bf16_weight_kernel<<<grid, 256, 0, static_cast<cudaStream_t>(stream)>>>(
      b_kn, ldb, static_cast<__nv_bfloat16*>(b_nk_bf16), k, n);
  ANNC_CUDA(cudaGetLastError());
  return ANNC_OK;
}

int annc_kn4_pack_dev(const float* b_kn, float* b_packed, int64_t k, int64_t n, void* stream) {
  ANNC_REQUIRE(b_kn && b_packed && b_kn != b_packed, ANNC_ERR_INVALID_ARGUMENT, "kn4: bad buffers");
  if (k * n <= 0) return ANNC_OK;
  gemm::convert_kn4(b_kn, b_packed, k, n, true, static_cast<cudaStream_t>(stream));
  ANNC_CUDA(cudaGetLastError());
  return ANNC_OK;
}

int annc_kn4_unpack_dev(const float* b_packed, float* b_kn, int64_t k, int64_t n, void* stream) {
  ANNC_REQUIRE(b_kn && b_packed && b_kn != b_packed, ANNC_ERR_INVALID_ARGUMENT, "kn4: bad buffers");
  if (k * n <= 0) return ANNC_OK;
  gemm::convert_kn4(b_packed, b_kn, k, n, false, static_cast<cudaStream_t>(stream));
  ANNC_CUDA(cudaGetLastError());
  return ANNC_OK;
}

int64_t annc_kn4_offset(int64_t K, int64_t N, int64_t k, int64_t n) {
  if (k < 0 || n < 0 || k >= K || n >= N) return -1;
  return kn4::offset(K, N, k, n);
}

int annc_KPFusedBatchMatMulAddSigmoid(const annc_tensor* lhs, const annc_tensor* rhs,
                                      const annc_tensor* bias, annc_alloc_fn alloc, void* ctx) {
  ANNC_REQUIRE(lhs && rhs && bias && alloc, ANNC_ERR_INVALID_ARGUMENT, "null argument");
  ANNC_REQUIRE(lhs->rank == 3, ANNC_ERR_INVALID_ARGUMENT, "lhs must be rank 3");
  ANNC_REQUIRE(rhs->rank == 2 || rhs->rank == 3, ANNC_ERR_INVALID_ARGUMENT, "rhs must be rank 2 or 3");
  ANNC_REQUIRE(bias->rank <= 3, ANNC_ERR_INVALID_ARGUMENT, "bias rank must be <= 3");
  const int64_t batch = lhs->dims[0], m = lhs->dims[1], k = lhs->dims[2];
  const bool rhs_batched = rhs->rank == 3;
  ANNC_REQUIRE(!rhs_batched || rhs->dims[0] == batch, ANNC_ERR_INVALID_ARGUMENT,
               "lhs/rhs batch mismatch");
  ANNC_REQUIRE(rhs->dims[rhs_batched ? 1 : 0] == k, ANNC_ERR_INVALID_ARGUMENT,
               "lhs/rhs contracting dim mismatch");
  const int64_t n = rhs->dims[rhs_batched ? 2 : 1];
  const int64_t out_dims[3] = {batch, m, n};
  float* out = static_cast<float*>(alloc(ctx, 0, ANNC_F32, 3, out_dims));
  // BuildBiasInfo (fused_batchmatmul_add_sigmoid.cc:197-214)
  int64_t bd[3] = {1, 1, 1};
  for (int i = 0; i < bias->rank; ++i) bd[3 - bias->rank + i] = bias->dims[i];
  ANNC_REQUIRE((bd[0] == 1 || bd[0] == batch) && (bd[1] == 1 || bd[1] == m) &&
                   (bd[2] == 1 || bd[2] == n),
               ANNC_ERR_INVALID_ARGUMENT, "bias shape is not broadcast-compatible");
  gemm::BiasBroadcast bb;
  bb.s2 = bd[2] == 1 ? 0 : 1;
  bb.s1 = bd[1] == 1 ? 0 : bd[2];
  bb.s0 = bd[0] == 1 ? 0 : bd[1] * bd[2];
  if (batch * m * n == 0) return ANNC_OK;
  ANNC_REQUIRE(out, ANNC_ERR_INTERNAL, "output allocation failed");
  Call call;
  annc_gemm_desc d;
  memset(&d, 0, sizeof(d));
  d.m = m;
  d.n = n;
  d.k = k;
  d.batch = batch;
  d.lda = k;
  d.ldb = n;
  d.ldc = n;
  d.stride_a = m * k;
  d.stride_b = rhs_batched ? k * n : 0;
  d.stride_c = m * n;
  d.alpha = 1.0f;
  d.beta = 0.0f;
  d.a = call.in((const float*)lhs->data, (size_t)numel(*lhs));
  d.b = call.in((const float*)rhs->data, (size_t)numel(*rhs));
  d.bias = call.in((const float*)bias->data, (size_t)numel(*bias));
  d.c = call.out(out, (size_t)(batch * m * n));
  d.activation = ANNC_ACT_SIGMOID;
  d.math = ANNC_MATH_FP32;  // the reference test asks for 1e-5
  if (call.status() != ANNC_OK) return call.status();
  ANNC_TRY(gemm::run_simt(d, call.stream(), &bb));
  return call.finish();
}

}  // extern "C"
