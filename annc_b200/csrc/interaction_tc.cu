// DLRM dot interaction on the tensor cores (TF32): out[b] = [ Z[b,0,:] | strict lower
// triangle of Z[b] Z[b]^T | 0 padding ], Z f32[batch, F, 64].
//
// A tile is SPT = 128 / F consecutive samples = R = SPT * F rows of the [batch*F, 64]
// matrix.  One TMA box per 32-float half of the rows lands in a 128-byte-swizzled stage;
// the same stage is both the A and the B operand of UMMA 128x128x8 (kind::tf32, both
// K-major), eight instructions per tile, so the 128x128 accumulator holds every pairwise
// dot product of the tile's rows and the wanted ones are the diagonal F x F blocks.
// Rows R..127 of a stage are never written; whatever they hold only reaches accumulator
// rows and columns that are not read.
//
// Persistent CTAs (one per SM): warp 0 TMA producer over a 5-stage ring, warp 1 MMA
// issuer with two TMEM accumulators in ping-pong, warps 2-9 two epilogue groups of four
// warps, group g taking the tiles that use accumulator g.  A lane holds one accumulator row, of
// which the columns below the diagonal of its sample's block are one run of the output row: it
// drops them there in a shared-memory image of the tile's output (row offsets are triangular
// numbers, 32 in a row of which differ modulo 32: no bank conflicts), and one bulk copy sends the
// image off while the next tile is worked on.  Row 0 of every sample comes from global memory
// unrounded; the products are TF32 x TF32 with fp32 sums.
// Bound by HBM (F*64*4 bytes read and (64 + F(F-1)/2)*4 written per sample).  65536 x 27: 86 us (85 at the copy rate); 140 us
// with two stages and an epilogue that went through a copy of the whole accumulator and wrote
// the output one float per thread, a division's worth of index work each.
// All mbarrier waits are bounded (tc_ptx.cuh).
#include <cstring>

#include "common.h"
#include "pdl.cuh"
#include "tc_host.h"
#include "tc_ptx.cuh"

namespace annc {
namespace {

using namespace annc::tc;

constexpr int ID = 64;              // embedding dim
constexpr int I_STAGES = 5;
constexpr int I_BOX = 128 * 128;    // bytes reserved per 32-float half (128 rows x 128 B)
constexpr int I_STAGE = 2 * I_BOX;
constexpr int I_THREADS = 320;     // producer, MMA issuer, two epilogue groups of 128
// Row-0 floats each epilogue thread carries per tile: samples_per_tile * 64 / 128, rounded up
// to the template instance (2 covers F >= 26, the DLRM case; 32 covers F = 2).
// Output image of a tile: spt rows of 64 + F(F-1)/2 floats rounded up to four; largest for F = 2.
constexpr int I_IMG = 64 * 68 * 4;
constexpr size_t I_SMEM = 1024 + (size_t)I_STAGES * I_STAGE + 2 * I_IMG + 256;

__device__ int g_inter_error = 0;

struct InterParams {
  const float* z;
  float* out;
  long long batch, out_stride;
  int F, spt, rows, tri;
  int img_row;  // floats per row of the output image: 64 + tri, rounded up to four
  int bulk;     // the output rows are 16-byte aligned: bulk copies
  long long tiles;
};

__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void epi_sync(int group) {  // the 128 threads of one epilogue group
  asm volatile("bar.sync %0, 128;" ::"r"(group + 1) : "memory");
}

template <int ROW0_PER_THREAD>
__global__ void __launch_bounds__(I_THREADS, 1)
dot_interaction_tc_kernel(const __grid_constant__ CUtensorMap tmap, InterParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  uint8_t* gen = smem_raw + (base - raw);
  float* img_all = reinterpret_cast<float*>(gen + I_STAGES * I_STAGE);
  const uint32_t bars = base + I_STAGES * I_STAGE + 2 * I_IMG;
  const uint32_t bar_full = bars, bar_empty = bars + 8 * I_STAGES;
  const uint32_t bar_tfull = bars + 16 * I_STAGES, bar_tempty = bar_tfull + 16;
  uint32_t* tmem_slot =
      reinterpret_cast<uint32_t*>(gen + I_STAGES * I_STAGE + 2 * I_IMG + 16 * I_STAGES + 32);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* epi_fail_all = reinterpret_cast<volatile int*>(tmem_slot + 2);  // one word per group

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&tmap);
    for (int s = 0; s < I_STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1);
      mbar_init(bar_empty + 8 * s, 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(bar_tfull + 8 * b, 1);
      mbar_init(bar_tempty + 8 * b, 4);  // one arrival per epilogue warp
    }
    *abort_flag = 0;
    epi_fail_all[0] = 0;
    epi_fail_all[1] = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // padding inside the image rows: zero for good
  const int img_pad = p.img_row - ID - p.tri;
  for (int e = threadIdx.x; e < 2 * p.spt * img_pad; e += I_THREADS) {
    const int row = e / img_pad, g = row / p.spt;
    img_all[g * (I_IMG / 4) + (row - g * p.spt) * p.img_row + ID + p.tri + (e - row * img_pad)] = 0.f;
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)), "r"(256u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  const uint32_t box_bytes = (uint32_t)p.rows * 128u;
  // Launched while the kernel before it drains: nothing above touches what that one reads or writes.
  pdl_trigger();
  pdl_wait();

  if (*reinterpret_cast<volatile int*>(&g_inter_error) != 0) {  // an earlier launch gave up
  } else if (warp == 0) {
    if (lane == 0) {
      long long li = 0;
      for (long long t = blockIdx.x; t < p.tiles; t += gridDim.x, ++li) {
        const int s = (int)(li % I_STAGES);
        const uint32_t ph = (uint32_t)(li / I_STAGES) & 1u;
        if (!mbar_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, &g_inter_error)) break;
        const uint32_t st = base + s * I_STAGE;
        mbar_expect_tx(bar_full + 8 * s, 2 * box_bytes);
        tma_load_2d(st, &tmap, 0, (int)(t * p.rows), bar_full + 8 * s);
        tma_load_2d(st + I_BOX, &tmap, 32, (int)(t * p.rows), bar_full + 8 * s);
      }
    }
  } else if (warp == 1) {
    if (lane == 0) {
      const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | (16u << 17) | (8u << 24);
      long long li = 0;
      for (long long t = blockIdx.x; t < p.tiles; t += gridDim.x, ++li) {
        const int s = (int)(li % I_STAGES), buf = (int)(li & 1);
        const uint32_t ph = (uint32_t)(li / I_STAGES) & 1u, tph = (uint32_t)(li >> 1) & 1u;
        if (!mbar_wait(bar_tempty + 8 * buf, tph ^ 1u, abort_flag, &g_inter_error)) break;
        if (!mbar_wait(bar_full + 8 * s, ph, abort_flag, &g_inter_error)) break;
        tc_fence_after();
        const uint32_t st = base + s * I_STAGE;
#pragma unroll
        for (int kk = 0; kk < 8; ++kk) {
          const uint32_t a = st + (kk >> 2) * I_BOX + (kk & 3) * 32;
          const uint64_t d = smem_desc(a, 16, 1024, 2);
          umma_tf32(tmem_base + buf * 128, d, d, idesc, kk != 0 ? 1u : 0u);
        }
        umma_commit(bar_empty + 8 * s);
        umma_commit(bar_tfull + 8 * buf);
      }
    }
  } else {
    const int group = (warp - 2) >> 2;                // accumulator and tiles of this group
    const int q = warp & 3, te = (threadIdx.x - 64) & 127;
    float* img = img_all + group * (I_IMG / 4);
    volatile int* epi_fail = epi_fail_all + group;
    const int row_lo = 32 * q;
    // columns this warp's rows need: the diagonal blocks of the samples they belong to
    int c_lo = 0, c_hi = 0;
    if (row_lo < p.rows) {
      const int row_hi = min(row_lo + 31, p.rows - 1);
      c_lo = (row_lo / p.F) * p.F;
      c_hi = (row_hi / p.F + 1) * p.F;
    }
    // this lane's accumulator row: feature fi of sample fs; it keeps the columns first .. first + fi - 1
    const int row = row_lo + lane;
    const int fs = row / p.F, first = fs * p.F, fi = row < p.rows ? row - first : 0;
    float* const my_img = img + fs * p.img_row + ID + fi * (fi - 1) / 2;
    long long li = group;
    for (long long t = blockIdx.x + (long long)group * gridDim.x; t < p.tiles;
         t += 2LL * gridDim.x, li += 2) {
      const int buf = group;
      const uint32_t tph = (uint32_t)(li >> 1) & 1u;
      const long long b0 = t * p.spt;
      const int samples = (int)min((long long)p.spt, p.batch - b0);
      float row0[ROW0_PER_THREAD];
#pragma unroll
      for (int r = 0; r < ROW0_PER_THREAD; ++r) {  // unrounded copy of Z[b, 0, :]
        const int idx = te + 128 * r;
        const int s = idx / ID, col = idx - s * ID;
        row0[r] = s < samples ? p.z[(b0 + s) * p.F * ID + col] : 0.f;
      }
      // All four warps leave together: a warp that gave up still joins the barrier.
      const bool ok = __all_sync(0xffffffffu, mbar_wait(bar_tfull + 8 * buf, tph, abort_flag,
                                                        &g_inter_error)) != 0;
      if (!ok) *epi_fail = 1;
      if (te == 0) bulk_wait_read<0>();  // the image of the group's last tile has been read
      epi_sync(group);
      if (*epi_fail) break;  // written before the barrier by epilogue warps only: same answer for all
      tc_fence_after();
#pragma unroll 1
      for (int c0 = c_lo & ~31; c0 < c_hi; c0 += 32) {  // warp-uniform
        uint32_t r[32];
        tmem_ld32(tmem_base + buf * 128 + ((uint32_t)row_lo << 16) + (uint32_t)c0, r);
        tmem_ld_wait();
        const int d = c0 - first;
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if ((unsigned)(d + j) < (unsigned)fi) my_img[d + j] = __uint_as_float(r[j]);
      }
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar_tempty + 8 * buf);  // accumulator may be overwritten
#pragma unroll
      for (int r = 0; r < ROW0_PER_THREAD; ++r) {
        const int idx = te + 128 * r;
        const int s = idx / ID, col = idx - s * ID;
        if (s < p.spt) img[s * p.img_row + col] = row0[r];
      }
      if (p.bulk) fence_proxy_async();
      epi_sync(group);
      if (p.bulk) {
        if (te == 0) {
          const uint32_t src = smem_u32(img);
          const uint32_t row_bytes = (uint32_t)p.img_row * 4u;
          if (p.out_stride == p.img_row) {
            bulk_store(p.out + b0 * p.out_stride, src, (uint32_t)samples * row_bytes);
          } else {
            for (int s = 0; s < samples; ++s)
              bulk_store(p.out + (b0 + s) * p.out_stride, src + (uint32_t)s * row_bytes, row_bytes);
          }
          bulk_commit();
        }
      } else {
        const int w = ID + p.tri;
        for (int e = te; e < samples * w; e += 128) {
          const int s = e / w;
          p.out[(b0 + s) * p.out_stride + (e - s * w)] = img[s * p.img_row + (e - s * w)];
        }
      }
      // zeros behind the part the image holds
      const int have = p.bulk ? p.img_row : ID + p.tri;
      const int pad = (int)p.out_stride - have;
      for (int e = te; e < samples * pad; e += 128) {
        const int s = e / pad;
        p.out[(b0 + s) * p.out_stride + have + (e - s * pad)] = 0.f;
      }
    }
    if (te == 0) bulk_wait_all();  // the copies read this CTA's shared memory
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(256u)
                 : "memory");
  }
}

}  // namespace

// Launch; returns ANNC_ERR_UNSUPPORTED when the shape does not fit this kernel.
int dot_interaction_tc(const float* z, int64_t batch, int F, int dim, int64_t z_stride, float* out,
                       int64_t out_stride, cudaStream_t s) {
  if (dim != ID || F < 2 || F > 32 || z_stride != (int64_t)F * ID ||
      (reinterpret_cast<uintptr_t>(z) & 15) != 0 || batch * F >= (1LL << 31) ||
      out_stride >= (1 << 20))
    return ANNC_ERR_UNSUPPORTED;
  static bool attr_set_dev[kMaxDevices] = {};
  bool& attr_set = attr_set_dev[device_slot()];
  if (!attr_set) {
    ANNC_CUDA(cudaFuncSetAttribute(dot_interaction_tc_kernel<2>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)I_SMEM));
    ANNC_CUDA(cudaFuncSetAttribute(dot_interaction_tc_kernel<8>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)I_SMEM));
    ANNC_CUDA(cudaFuncSetAttribute(dot_interaction_tc_kernel<32>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)I_SMEM));
    attr_set = true;
  }
  InterParams p;
  memset(&p, 0, sizeof(p));
  p.z = z;
  p.out = out;
  p.batch = batch;
  p.out_stride = out_stride;
  p.F = F;
  p.spt = 128 / F;
  p.rows = p.spt * F;
  p.tri = F * (F - 1) / 2;
  p.tiles = (batch + p.spt - 1) / p.spt;
  p.img_row = (ID + p.tri + 3) & ~3;
  p.bulk = out_stride % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0;
  CUtensorMap tm;
  ANNC_TRY(tc::make_map(&tm, z, batch * F, ID, ID, p.rows, false));
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const unsigned grid = (unsigned)(p.tiles < sms ? p.tiles : sms);
  // Launched early at every size: us with the product that writes z before it, without / with, batch 200 12.1 / 11.6,
  // 4096 18.8 / 16.5, 65536 125 / 121.  Row-sharded steps, whose pooling kernel runs beside it, lose nothing either:
  // one rank, four issue orders, batch 65536 1327 to 1442 / 1323 to 1437, 16384 366 to 412 / 366 to 413.
  const int need = (p.spt * ID + 127) / 128;
  if (need <= 2) ANNC_CUDA(launch_pdl(dot_interaction_tc_kernel<2>, dim3(grid), dim3(I_THREADS), I_SMEM, s, tm, p));
  else if (need <= 8) ANNC_CUDA(launch_pdl(dot_interaction_tc_kernel<8>, dim3(grid), dim3(I_THREADS), I_SMEM, s, tm, p));
  else ANNC_CUDA(launch_pdl(dot_interaction_tc_kernel<32>, dim3(grid), dim3(I_THREADS), I_SMEM, s, tm, p));
  ANNC_CUDA(cudaGetLastError());
  return ANNC_OK;
}

int dot_interaction_error_flag(int* flag) {
  ANNC_CUDA(cudaMemcpyFromSymbol(flag, g_inter_error, sizeof(int)));
  return ANNC_OK;
}

}  // namespace annc
