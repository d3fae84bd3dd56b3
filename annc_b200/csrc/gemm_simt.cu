// fp32 GEMM on the CUDA cores: the route for shapes the tensor-core kernel does
// not take (tiny or unaligned problems, transposed A, fp32-exact requests such
// as KPFusedBatchMatMulAddSigmoid whose reference tolerance is 1e-5).
// Register-tiled blocks with packed fp32x2 multiply-adds, strided batch on blockIdx.z.
#include "common.h"
#include "gemm.h"
#include "kn4.h"
#include "pdl.cuh"
#include "tc_ptx.cuh"

namespace annc {
namespace gemm {
namespace {

__device__ __forceinline__ float apply_act(float v, int act) {
  if (act == ANNC_ACT_RELU) return fmaxf(v, 0.0f);
  if (act == ANNC_ACT_SIGMOID) return __fdiv_rn(1.0f, 1.0f + expf(-v));
  return v;
}

// Two independent fp32 multiply-adds in one instruction; each half rounds like fmaf.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(unsigned long long v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
  asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

// Block tile BM x BN, k-steps of BK, TM x TN outputs per thread (TM as packed pairs); every output
// is one chain of fmaf over ascending k.  Both operands sit k-major in shared memory, two stages;
// the next k-step's global loads are in registers while this one is multiplied.  An operand whose
// k runs along the row is transposed on its way into shared memory.  A thread's rows and columns
// are groups of four, BM / (TM / 4) and BN / (TN / 4) apart, so that its shared-memory reads are
// 16 bytes wide and free of conflicts.  The finished tile goes through shared memory, so that the
// epilogue is one short loop over rows of 16-byte pieces: a small product is bound by the fetch of
// instructions that run once, and unrolled over the accumulators the epilogue was most of the code.
// Bound by instruction issue and, at small k, by the load latency of the first stages.  256 x
// [50 x 128] x [128 x 256] with bias and sigmoid: 80 us with the former tile (64 x 64, 4 x 4
// scalar multiply-adds and scalar loads per thread), 34 us now; pairs along n 41 us (twice as many
// values to double), 8 x 8 outputs per thread 36 us and 47 us with a batched B.  1 x 2048 x 2048:
// 228 us, 19 us with k split over a cluster.
//   KC: the operand's k is contiguous ([m,k] A, [n,k] B), else its m / n is ([k,m], [k,n], kn4).
//   VEC: 16-byte loads (bases and pitches allow them and no piece straddles an edge), else one
//   float at a time.  Idx: 64-bit where n or k needs it.
//   ranks > 1 (few tiles): the CTAs of a cluster along z share one tile and split its k range; each
//   leaves its partial tile in shared memory and rank r adds, for the rows i with i % ranks == r, the
//   ranks' parts in rank order (deterministic) before the epilogue.
template <int ROWS, int BK, int THREADS, bool KC, bool VEC, typename Idx>
struct OperandTile {
  static constexpr int PER = ROWS * BK / 4 / THREADS;  // pieces of four elements per thread
  static_assert(ROWS * BK / 4 % THREADS == 0, "every thread loads whole pieces");
  float4 r[PER];

  // Stage k0 of the operand into registers.  `x0` first row of the tile along m / n, `lim` its extent.
  __device__ __forceinline__ void load(const float* __restrict__ p, long long ld, Idx x0, Idx lim, Idx k0, Idx kdim,
                                       bool kn4_fmt) {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = threadIdx.x + i * THREADS;
      const Idx x = x0 + (KC ? e / (BK / 4) : (e % (ROWS / 4)) * 4);
      const Idx k = k0 + (KC ? (e % (BK / 4)) * 4 : e / (ROWS / 4));
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (x < lim && k < kdim) {
        const float* q = p + (KC ? x * ld + k : kn4_fmt ? kn4::offset(kdim, lim, k, x) : k * ld + x);
        if (VEC) {  // kn4: n % 4 == 0, four aligned columns never straddle a panel
          const float4 t = __ldg(reinterpret_cast<const float4*>(q));
          v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
        } else {
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            if (KC ? k + c < kdim : x + c < lim)
              v[c] = __ldg(!KC && kn4_fmt ? p + kn4::offset(kdim, lim, k, x + c) : q + c);
          }
        }
      }
      r[i] = make_float4(v[0], v[1], v[2], v[3]);
    }
  }
  // LD: floats between two k rows of the stage.
  template <int LD>
  __device__ __forceinline__ void store(float* __restrict__ s) const {
#pragma unroll
    for (int i = 0; i < PER; ++i) {
      const int e = threadIdx.x + i * THREADS;
      if (KC) {
        const int x = e / (BK / 4), k = (e % (BK / 4)) * 4;
        s[(k + 0) * LD + x] = r[i].x;
        s[(k + 1) * LD + x] = r[i].y;
        s[(k + 2) * LD + x] = r[i].z;
        s[(k + 3) * LD + x] = r[i].w;
      } else {
        const int k = e / (ROWS / 4), x = (e % (ROWS / 4)) * 4;
        *reinterpret_cast<float4*>(s + k * LD + x) = r[i];
      }
    }
  }
};

struct SimtArgs {
  annc_gemm_desc d;
  int bias_mode;  // 0: bias[n]; 1: the numpy-style broadcast strides below
  long long bias_s0, bias_s1, bias_s2;
  int ranks;      // CTAs of a cluster along z that share a tile
  int vec_c;      // 16-byte stores of C are possible
};

template <int BM, int BN, int BK, int TM, int TN, bool A_KC, bool B_KC, bool VEC, typename Idx>
__global__ void __launch_bounds__(BM * BN / (TM * TN), BM == 64 ? 4 : 8) sgemm_simt_kernel(SimtArgs args) {
  constexpr int THREADS = BM * BN / (TM * TN);
  constexpr int TX = BN / TN;  // threads along n
  constexpr int LDA = BM + 4, LDB = BN + 4;
  constexpr int RG = TM / 4, CG = TN / 4;  // groups of four rows / columns
  constexpr int LDP = BN + 4;              // finished (or partial) tile
  constexpr int STAGES = 2 * BK * (LDA + LDB), PART = BM * LDP;
  __shared__ __align__(16) float smem[STAGES > PART ? STAGES : PART];
  auto As = reinterpret_cast<float(*)[BK * LDA]>(smem);
  auto Bs = reinterpret_cast<float(*)[BK * LDB]>(smem + 2 * BK * LDA);
  const annc_gemm_desc& d = args.d;
  const Idx M = (Idx)d.m, N = (Idx)d.n, K = (Idx)d.k;
  const int ranks = args.ranks;
  const int rank = ranks > 1 ? (int)blockIdx.z : 0;  // of the cluster (one batch then)
  const long long bz = ranks > 1 ? 0 : blockIdx.z;
  const Idx k_per = ranks > 1 ? (K + ranks * BK - 1) / (ranks * BK) * BK : K;
  const Idx k_first = rank * k_per;
  const Idx k_end = min(K, k_first + k_per);
  const float* A = d.a + bz * d.stride_a;
  const float* B = d.b + bz * d.stride_b;
  const Idx m0 = (Idx)blockIdx.y * BM, n0 = (Idx)blockIdx.x * BN;
  const bool kn4_fmt = !B_KC && d.b_format == ANNC_B_KN4;
  const int tx = threadIdx.x % TX, ty = threadIdx.x / TX;

  // rows in pairs: A's pairs come out of shared memory as they are, only B's values are doubled
  unsigned long long acc[TM / 2][TN];
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;  // two +0.0f

  OperandTile<BM, BK, THREADS, A_KC, VEC, Idx> ta;
  OperandTile<BN, BK, THREADS, B_KC, VEC, Idx> tb;
  int cur = 0;
#pragma unroll 1
  for (Idx k0 = k_first - BK; k0 < k_end; k0 += BK) {  // round -1 only loads
    const bool next = k0 + BK < k_end;
    if (next) {
      ta.load(A, d.lda, m0, M, k0 + BK, K, false);
      tb.load(B, d.ldb, n0, N, k0 + BK, K, kn4_fmt);
    }
    if (k0 >= k_first) {
      // k rows past the end are zero in both operands; a short last stage ends at a multiple of 4
      const int kn = (int)min((Idx)BK, (k_end - k0 + 3) & ~(Idx)3);
#pragma unroll 1
      for (int k4 = 0; k4 < kn; k4 += 4) {
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) {
          unsigned long long a[TM / 2];
          float b[TN];
#pragma unroll
          for (int g = 0; g < RG; ++g) {
            const ulonglong2 v =
                *reinterpret_cast<const ulonglong2*>(&As[cur][(k4 + kk) * LDA + g * (BM / RG) + ty * 4]);
            a[2 * g] = v.x; a[2 * g + 1] = v.y;
          }
#pragma unroll
          for (int g = 0; g < CG; ++g) {
            const float4 v = *reinterpret_cast<const float4*>(&Bs[cur][(k4 + kk) * LDB + g * (BN / CG) + tx * 4]);
            b[4 * g] = v.x; b[4 * g + 1] = v.y; b[4 * g + 2] = v.z; b[4 * g + 3] = v.w;
          }
#pragma unroll
          for (int j = 0; j < TN; ++j) {
            const unsigned long long b2 = pack2(b[j], b[j]);
#pragma unroll
            for (int i = 0; i < TM / 2; ++i) fma2(acc[i][j], a[i], b2);
          }
        }
      }
    }
    if (next) {
      cur ^= 1;
      ta.template store<LDA>(As[cur]);
      tb.template store<LDB>(Bs[cur]);
      __syncthreads();
    }
  }

  __syncthreads();  // the stages become the finished tile
#pragma unroll
  for (int i = 0; i < TM / 2; ++i)
#pragma unroll
    for (int g = 0; g < CG; ++g) {
      float lo[4], hi[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) unpack2(acc[i][4 * g + j], lo[j], hi[j]);
      float* q = smem + ((i / 2) * (BM / RG) + ty * 4 + (i & 1) * 2) * LDP + g * (BN / CG) + tx * 4;
      *reinterpret_cast<float4*>(q) = make_float4(lo[0], lo[1], lo[2], lo[3]);
      *reinterpret_cast<float4*>(q + LDP) = make_float4(hi[0], hi[1], hi[2], hi[3]);
    }
  if (ranks > 1) tc::cluster_sync_all();
  else __syncthreads();

  float* C = d.c + bz * d.stride_c;
  const float* Add = d.addend ? d.addend + bz * d.stride_addend : nullptr;
  const float* bias = d.bias ? d.bias + bz * args.bias_s0 : nullptr;
  const long long bs1 = args.bias_mode ? args.bias_s1 : 0, bs2 = args.bias_mode ? args.bias_s2 : 1;
  const uint32_t part = tc::smem_u32(smem);
#pragma unroll 1
  for (int e = threadIdx.x; e < BM / ranks * (BN / 4); e += THREADS) {
    const int lm = rank + ranks * (e / (BN / 4)), ln = (e % (BN / 4)) * 4;
    const Idx gm = m0 + lm, gn = n0 + ln;
    if (gm >= M || gn >= N) continue;
    float v[4];
    if (ranks > 1) {
      v[0] = v[1] = v[2] = v[3] = 0.f;
      for (int r = 0; r < ranks; ++r) {
        float4 t;
        asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(t.x), "=f"(t.y), "=f"(t.z), "=f"(t.w)
                     : "r"(tc::mapa_u32(part + (uint32_t)((lm * LDP + ln) * sizeof(float)), (uint32_t)r))
                     : "memory");
        v[0] += t.x; v[1] += t.y; v[2] += t.z; v[3] += t.w;
      }
    } else {
      const float4 t = *reinterpret_cast<const float4*>(smem + lm * LDP + ln);
      v[0] = t.x; v[1] = t.y; v[2] = t.z; v[3] = t.w;
    }
    float* c = C + gm * d.ldc + gn;
    const float* add = Add ? Add + gm * d.ld_addend + gn : nullptr;
    const float* bp = bias ? bias + gm * bs1 + gn * bs2 : nullptr;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (gn + j >= N) continue;
      v[j] = d.alpha * v[j];
      if (d.beta != 0.f) v[j] += d.beta * c[j];
      if (add) v[j] += add[j];
      if (bp) v[j] += bp[j * bs2];
      v[j] = apply_act(v[j], d.activation);
    }
    if (args.vec_c && gn + 3 < N) {
      *reinterpret_cast<float4*>(c) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (gn + j < N) c[j] = v[j];
    }
  }
  if (ranks > 1) tc::cluster_sync_all();  // nobody leaves while a peer may still read its part
}

// n == 1 with row-major A: one warp per output row (a GEMV with the GEMM epilogue).
__global__ void __launch_bounds__(256) sgemm_n1_kernel(annc_gemm_desc d) {
  pdl_trigger();
  pdl_wait();
  const int lane = threadIdx.x & 31;
  const long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (i >= d.m) return;
  const float* a = d.a + i * d.lda;
  float s = 0.f;
  for (long long k = lane; k < d.k; k += 32) s = fmaf(a[k], d.b[k], s);
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) {
    float v = d.alpha * s;
    if (d.beta != 0.f) v += d.beta * d.c[i * d.ldc];
    if (d.addend) v += d.addend[i * d.ld_addend];
    if (d.bias) v += d.bias[0];
    d.c[i * d.ldc] = apply_act(v, d.activation);
  }
}

// Four sigmoids, out of line: unrolled into a kernel they fill the instruction cache of a loop that
// hardly ever takes them.
__device__ __noinline__ float4 sigmoid4(float4 v) {
  return make_float4(apply_act(v.x, ANNC_ACT_SIGMOID), apply_act(v.y, ANNC_ACT_SIGMOID),
                     apply_act(v.z, ANNC_ACT_SIGMOID), apply_act(v.w, ANNC_ACT_SIGMOID));
}

// k <= 16 with row-major A and B (the first DLRM layer, 13 dense features): the work is
// writing C.  A thread keeps its four columns of B in registers, every value doubled; 16 rows of A
// sit k-major in shared memory, so that one 16-byte read brings four rows of a k and a packed
// multiply-add does two rows of a column.  Every output row is written with coalesced 16-byte
// stores.  65536 x 512 x 13: 54 us with scalar multiply-adds on one row at a time and the sigmoid
// inlined, 37 us; 4096 x 512 x 13: 16 us with 64 rows a block, 5 us.
constexpr int SK_ROWS = 16, SK_MAXK = 16;
template <int K>
__global__ void __launch_bounds__(128) sgemm_smallk_kernel(annc_gemm_desc d) {
  __shared__ __align__(16) float As[K][SK_ROWS];
  const long long m0 = (long long)blockIdx.x * SK_ROWS;
  const long long col = ((long long)blockIdx.y * 128 + threadIdx.x) * 4;
  constexpr int PER = (SK_ROWS * K + 127) / 128;
  float t_a[PER];  // all loads of the block are out before the first is used
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = threadIdx.x + 128 * i, r = e / K, k = e - r * K;
    t_a[i] = (r < SK_ROWS && m0 + r < d.m && k < d.k) ? __ldg(d.a + (m0 + r) * d.lda + k) : 0.f;
  }
  unsigned long long w[K][4];
#pragma unroll
  for (int k = 0; k < K; ++k) {
    float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
    if (k < d.k && col < d.n) t = __ldg(reinterpret_cast<const float4*>(d.b + k * d.ldb + col));
    w[k][0] = pack2(t.x, t.x);
    w[k][1] = pack2(t.y, t.y);
    w[k][2] = pack2(t.z, t.z);
    w[k][3] = pack2(t.w, t.w);
  }
  float4 bias = make_float4(0.f, 0.f, 0.f, 0.f);
  if (d.bias && col < d.n) bias = __ldg(reinterpret_cast<const float4*>(d.bias + col));
#pragma unroll
  for (int i = 0; i < PER; ++i) {
    const int e = threadIdx.x + 128 * i, r = e / K;
    if (r < SK_ROWS) As[e - r * K][r] = t_a[i];
  }
  __syncthreads();
  if (col >= d.n) return;
  const int rows = (int)(d.m - m0 < SK_ROWS ? d.m - m0 : SK_ROWS);
#pragma unroll 1
  for (int r = 0; r < rows; r += 4) {
    unsigned long long acc[2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;  // two +0.0f
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(&As[k][r]);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        fma2(acc[0][j], a.x, w[k][j]);
        fma2(acc[1][j], a.y, w[k][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      if (r + i >= rows) break;
      float v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float lo, hi;
        unpack2(acc[i >> 1][j], lo, hi);
        v[j] = d.alpha * ((i & 1) ? hi : lo);
      }
      float* crow = d.c + (m0 + r + i) * d.ldc + col;
      if (d.beta != 0.f) {
        const float4 o = *reinterpret_cast<const float4*>(crow);
        v[0] += d.beta * o.x; v[1] += d.beta * o.y; v[2] += d.beta * o.z; v[3] += d.beta * o.w;
      }
      if (d.addend) {
        const float4 a4 = __ldg(reinterpret_cast<const float4*>(d.addend + (m0 + r + i) * d.ld_addend + col));
        v[0] += a4.x; v[1] += a4.y; v[2] += a4.z; v[3] += a4.w;
      }
      float4 o = make_float4(v[0] + bias.x, v[1] + bias.y, v[2] + bias.z, v[3] + bias.w);
      if (d.activation == ANNC_ACT_RELU)
        o = make_float4(fmaxf(o.x, 0.0f), fmaxf(o.y, 0.0f), fmaxf(o.z, 0.0f), fmaxf(o.w, 0.0f));
      else if (d.activation == ANNC_ACT_SIGMOID) o = sigmoid4(o);
      *reinterpret_cast<float4*>(crow) = o;
    }
  }
}

static bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

template <int BM, int BN, int BK, int TM, int TN, bool VEC, typename Idx = int>
cudaError_t launch_tile(const SimtArgs& a, dim3 grid, cudaStream_t s) {
  const bool ak = !a.d.trans_a, bk = a.d.trans_b != 0;
  auto kernel = ak ? (bk ? sgemm_simt_kernel<BM, BN, BK, TM, TN, true, true, VEC, Idx>
                         : sgemm_simt_kernel<BM, BN, BK, TM, TN, true, false, VEC, Idx>)
                   : (bk ? sgemm_simt_kernel<BM, BN, BK, TM, TN, false, true, VEC, Idx>
                         : sgemm_simt_kernel<BM, BN, BK, TM, TN, false, false, VEC, Idx>);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(BM * BN / (TM * TN));
  cfg.stream = s;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = a.ranks;
  cfg.attrs = attr;
  cfg.numAttrs = a.ranks > 1 ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, a);
}

// 64 x 64 tiles of 8 x 4 outputs per thread when they fill the SMs at least once, else 32 x 32
// tiles of 4 x 4 (few rows or columns, small products: more blocks, less padding), with K split
// over clusters of up to 8 CTAs while the tiles leave SMs idle and every rank keeps two k-steps.
int launch_simt(SimtArgs& a, cudaStream_t s) {
  const annc_gemm_desc& d = a.d;
  const bool huge = d.n >= (1LL << 31) - 64 || d.k >= (1LL << 31) - 64;  // 64-bit indices
  const long long big = ((d.m + 63) / 64) * ((d.n + 63) / 64) * d.batch;
  const bool wide = big >= 148 && d.n > 32 && d.m > 32 && !huge;
  const int bm = wide ? 64 : 32, bn = bm;
  const long long gx = (d.n + bn - 1) / bn, gy = (d.m + bm - 1) / bm;
  const bool many = d.batch > 1;
  const bool vec_a = aligned16(d.a) && (d.lda & 3) == 0 && (!many || (d.stride_a & 3) == 0) &&
                     ((d.trans_a ? d.m : d.k) & 3) == 0;
  const bool vec_b = aligned16(d.b) && (!many || (d.stride_b & 3) == 0) && ((d.trans_b ? d.k : d.n) & 3) == 0 &&
                     (d.b_format == ANNC_B_KN4 || (d.ldb & 3) == 0);
  a.vec_c = aligned16(d.c) && (d.ldc & 3) == 0 && (!many || (d.stride_c & 3) == 0);
  a.ranks = 1;
  if (!wide && !many)
    while (a.ranks < 8 && gx * gy * a.ranks * 2 <= 148 * 4 && d.k >= 32 * a.ranks * 4) a.ranks *= 2;
  // blockIdx.y and .z are limited to 65535: walk tall products and long batches in slabs.
  for (long long b0 = 0; b0 < d.batch; b0 += 65535) {
    const long long nb = d.batch - b0 < 65535 ? d.batch - b0 : 65535;
    for (long long y0 = 0; y0 < gy; y0 += 65535) {
      const long long ny = gy - y0 < 65535 ? gy - y0 : 65535;
      SimtArgs e = a;
      e.d.batch = nb;
      e.d.m = d.m - y0 * bm < ny * bm ? d.m - y0 * bm : ny * bm;
      e.d.a = d.a + b0 * d.stride_a + y0 * bm * (d.trans_a ? 1 : d.lda);
      e.d.b = d.b + b0 * d.stride_b;
      e.d.c = d.c + b0 * d.stride_c + y0 * bm * d.ldc;
      if (d.addend) e.d.addend = d.addend + b0 * d.stride_addend + y0 * bm * d.ld_addend;
      if (d.bias && a.bias_mode) e.d.bias = d.bias + b0 * a.bias_s0 + y0 * bm * a.bias_s1;
      const dim3 grid((unsigned)gx, (unsigned)ny, (unsigned)(a.ranks > 1 ? a.ranks : nb));
      if (wide && vec_a && vec_b) ANNC_CUDA((launch_tile<64, 64, 16, 8, 4, true>(e, grid, s)));
      else if (wide) ANNC_CUDA((launch_tile<64, 64, 16, 8, 4, false>(e, grid, s)));
      else if (huge) ANNC_CUDA((launch_tile<32, 32, 32, 4, 4, false, long long>(e, grid, s)));
      else if (vec_a && vec_b) ANNC_CUDA((launch_tile<32, 32, 32, 4, 4, true>(e, grid, s)));
      else ANNC_CUDA((launch_tile<32, 32, 32, 4, 4, false>(e, grid, s)));
    }
  }
  return ANNC_OK;
}

}  // namespace

int run_simt(const annc_gemm_desc& d, cudaStream_t s, const BiasBroadcast* bb) {
  if (d.m <= 0 || d.n <= 0 || d.batch <= 0) return ANNC_OK;
  if (d.n == 1 && d.batch == 1 && !d.trans_a && !bb && d.b_format == ANNC_B_PLAIN &&
      (d.trans_b || d.ldb == 1)) {
    const dim3 grid((unsigned)((d.m + 7) / 8));
    if (early_launch(d)) return launch_pdl(sgemm_n1_kernel, grid, dim3(256), 0, s, d) == cudaSuccess ? ANNC_OK : cuda_fail(cudaGetLastError(), "sgemm_n1_kernel");
    sgemm_n1_kernel<<<grid, 256, 0, s>>>(d);
    ANNC_CUDA(cudaGetLastError());
    return ANNC_OK;
  }
  if ((d.m + 63) / 64 > 65535) return fail(ANNC_ERR_UNSUPPORTED, "simt gemm: more than 4M rows");
  // With an addend a thread waits for each row's part of it in turn, which small products do not hide:
  // 200 x 512 x 13 6.8 us, 5.3 us in tiles; 1000 x 512 x 13 7.1 / 5.9; 500 x 2048 x 13 7.2 / 7.8.
  const bool small_add = d.addend && d.m * d.n <= (1 << 19);
  if (d.k <= SK_MAXK && d.k >= 1 && d.m >= 64 && !small_add && d.batch == 1 && !d.trans_a && !d.trans_b && !bb &&
      d.b_format == ANNC_B_PLAIN && (d.n & 3) == 0 && (d.ldb & 3) == 0 && (d.ldc & 3) == 0 &&
      aligned16(d.b) && aligned16(d.c) && (!d.bias || aligned16(d.bias)) &&
      (!d.addend || (aligned16(d.addend) && (d.ld_addend & 3) == 0)) &&
      (d.n / 4 + 127) / 128 <= 65535) {
    dim3 grid((unsigned)((d.m + SK_ROWS - 1) / SK_ROWS), (unsigned)((d.n / 4 + 127) / 128));
    // One build per K, for its registers and multiply-adds: 65536 x 512 with K = 9 28.7 us, 36 in the build for
    // 13; with K = 13 36 us, 37.5 us in that for 16.  14 and 15 take 16, whose index arithmetic is shifts:
    // 200 x 512 x 15 3.9 us, 4.8 us in a build of its own.
    static void (*const kernels[])(annc_gemm_desc) = {
        sgemm_smallk_kernel<8>,  sgemm_smallk_kernel<9>,  sgemm_smallk_kernel<10>, sgemm_smallk_kernel<11>,
        sgemm_smallk_kernel<12>, sgemm_smallk_kernel<13>, sgemm_smallk_kernel<SK_MAXK>};
    kernels[d.k <= 8 ? 0 : d.k <= 13 ? d.k - 8 : 6]<<<grid, 128, 0, s>>>(d);
    ANNC_CUDA(cudaGetLastError());
    return ANNC_OK;
  }
  SimtArgs args;
  args.d = d;
  args.bias_mode = bb ? 1 : 0;
  args.bias_s0 = bb ? bb->s0 : 0;
  args.bias_s1 = bb ? bb->s1 : 0;
  args.bias_s2 = bb ? bb->s2 : 0;
  // A batch whose B is shared and whose A and C slabs follow one another is one tall product: no
  // tile is left part empty by a slab's last rows (50 of 64).
  annc_gemm_desc& e = args.d;
  if (e.batch > 1 && e.stride_b == 0 && !e.trans_a && e.stride_a == e.m * e.lda && e.stride_c == e.m * e.ldc &&
      (!e.addend || e.stride_addend == e.m * e.ld_addend) &&
      (!e.bias || !bb || (bb->s0 == 0 && bb->s1 == 0))) {
    e.m *= e.batch;
    e.batch = 1;
  }
  return launch_simt(args, s);
}

}  // namespace gemm
}  // namespace annc
