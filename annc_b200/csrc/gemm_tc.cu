// TF32 GEMM on the 5th-generation tensor cores (tcgen05) for sm_100a.
//
//   C[M,N] = act(alpha * A[M,K] * B + beta * C + addend + bias)
//
// One CTA computes a 128 x 128 tile of C with UMMA 128x128x8 (kind::tf32), fp32
// accumulators in 128 TMEM columns.  Shared memory holds a ring of stages, each one
// 128 x 32 floats of A and 32 x 128 floats of B, both in the 128-byte-swizzle
// layout the UMMA shared-memory descriptors name (A and a K-major B: SWIZZLE_128B;
// an N-major B: SWIZZLE_128B_BASE32B).
//
//   warp 0      A tiles (and B when it is stored [N,K] or [K,N]) by TMA, cp.async.bulk.tensor
//               without multicast, completion counted on the stage's "full" mbarrier
//   warp 1      TMEM allocation, tcgen05.mma issue by one thread, tcgen05.commit on
//               the stage's "empty" mbarrier and, after the last k-step, on "done"
//   warps 2-5   B loader when B is stored in the kn4 prepacked layout:
//               16-byte cp.async from global straight into the N-major swizzled
//               stage (the packed layout is consumed as it lies in memory, no
//               unpacked copy is made); then the epilogue: tcgen05.ld of the
//               accumulator rows, alpha/beta/addend/bias/activation in registers,
//               16-byte stores.
//
// fp32 operands are fed unchanged to kind::tf32, which reads the upper 19 bits.
// With 3 stages (96 KB) two CTAs fit one SM, so one CTA's epilogue overlaps the other's
// main loop; small grids run 6 stages with one CTA per SM.  Every mbarrier wait is bounded: when a wait runs out the CTA
// raises a device flag (read by annc_gemm_check), leaves its loops, frees its TMEM
// and returns.
#include <cuda.h>

#include <cstdint>
#include <cstring>

#include "common.h"
#include "gemm.h"
#include "kn4.h"
#include "pdl.cuh"
#include "tc_host.h"
#include "tc_ptx.cuh"

namespace annc {
namespace gemm {
namespace {

constexpr int BM = 128, BN = 128, BK = 32;
// 3 stages (96 KB): two CTAs share an SM and hide each other's prologue and epilogue;
// 6 stages (192 KB): one CTA per SM with a deeper ring, for grids that cannot fill the
// SMs twice and would otherwise wait on memory latency.
constexpr int A_BYTES = BM * BK * 4;  // 16 KB
constexpr int B_BYTES = BN * BK * 4;  // 16 KB
constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
constexpr int NUM_THREADS = 192;      // 6 warps
constexpr int LOADER_THREADS = 128;   // warps 2..5
constexpr int TMEM_COLS = 128;
constexpr size_t smem_bytes(int stages) { return 1024 + (size_t)stages * STAGE_BYTES + 256; }

// B sources: [N,K] by TMA (K-major operand), [K,N] by TMA (N-major operand, four
// 32-column boxes per stage), kn4-packed by the cp.async loader (N-major operand).
enum BMode { B_TMA_NK = 0, B_TMA_KN = 1, B_KN4 = 2 };

struct TcParams {
  int M, N, K;
  int b_mode;
  const float* B;
  long long ldb;
  float* C;
  long long ldc;
  const float* addend;
  long long ld_addend;
  const float* bias;
  float alpha, beta;
  int act;
  int batched;    // A (and B when b_batched) are rank-3 tensor maps, batch = blockIdx.z
  int b_batched;
  long long stride_c, stride_addend;
  int split;      // > 1: the CTAs of a cluster (1, 1, split) share one tile and split its K range
};

__device__ int g_gemm_error = 0;  // 1: an mbarrier wait ran out

using namespace annc::tc;

// Four sigmoids, out of line: they would fill the instruction cache of an epilogue that hardly ever
// takes them.
__device__ __noinline__ float4 sigmoid4(float4 v) {
  return make_float4(__fdiv_rn(1.0f, 1.0f + expf(-v.x)), __fdiv_rn(1.0f, 1.0f + expf(-v.y)),
                     __fdiv_rn(1.0f, 1.0f + expf(-v.z)), __fdiv_rn(1.0f, 1.0f + expf(-v.w)));
}

// ---------------------------------------------------------------- kernel
template <int STAGES>
// (80 registers in the two-per-SM form, although shared memory is what limits it to two: a block then
// still fits beside four blocks of the row exchange's pooling kernel)
__global__ void __launch_bounds__(NUM_THREADS, STAGES <= 3 ? 4 : 1)
gemm_tf32_tcgen05_kernel(const __grid_constant__ CUtensorMap tmap_a,
                         const __grid_constant__ CUtensorMap tmap_b, TcParams p) {
  extern __shared__ uint8_t smem_raw[];
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;  // stages need 1024-byte alignment
  uint8_t* gen_base = smem_raw + (base - raw);
  const uint32_t bars = base + STAGES * STAGE_BYTES;
  // barrier block: full[STAGES], empty[STAGES], done, then tmem base word and abort word
  const uint32_t bar_full = bars, bar_empty = bars + 8 * STAGES, bar_done = bars + 16 * STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(gen_base + STAGES * STAGE_BYTES + 16 * STAGES + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
  // Split K: cluster rank c of `split` takes the k-steps [it0, it0 + KT); every CTA keeps its
  // partial tile in shared memory and the ranks add them, each for its share of the rows, in
  // rank order (deterministic) through distributed shared memory before the epilogue.
  const int KT_all = (p.K + BK - 1) / BK;
  const int crank = p.split > 1 ? (int)cluster_ctarank() : 0;
  const int per = (KT_all + p.split - 1) / (p.split > 1 ? p.split : 1);
  const int it0 = p.split > 1 ? min(KT_all, crank * per) : 0;
  const int KT = p.split > 1 ? min(KT_all, it0 + per) - it0 : KT_all;
  const int zb = p.split > 1 ? 0 : (int)blockIdx.z;  // batch index (no batches under split K)
  const bool b_by_loader = p.b_mode == B_KN4;
  const bool b_n_major = p.b_mode != B_TMA_NK;

  if (threadIdx.x == 0) {
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(bar_full + 8 * s, 1 + (b_by_loader ? LOADER_THREADS : 0));
      mbar_init(bar_empty + 8 * s, 1);
    }
    mbar_init(bar_done, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;
  // Launched while the kernel before it drains: what is above needs nothing of that kernel, what follows
  // waits for its end.
  pdl_trigger();
  pdl_wait();
  // A CTA of an earlier wave (or launch) gave up on a wait: do not start, fail fast.  (The
  // CTAs of a split-K cluster always run to their cluster barriers.)
  const bool poisoned = p.split <= 1 && *reinterpret_cast<volatile int*>(&g_gemm_error) != 0;

  bool done = false;  // warps 2..5: the accumulator is complete and sits in shared memory
  constexpr int LD = BN + 4;
  if (poisoned) {
  } else if (warp == 0) {
    // ---------------- TMA producer
    if (lane == 0) {
      for (int li = 0; li < KT; ++li) {
        const int it = it0 + li;
        const int s = li % STAGES;
        const uint32_t ph = (uint32_t)(li / STAGES) & 1u;
        if (!mbar_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, &g_gemm_error)) break;
        const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_BYTES;
        mbar_expect_tx(bar_full + 8 * s, b_by_loader ? A_BYTES : STAGE_BYTES);
        const int bz = zb;
        if (p.batched) tma_load_3d(sa, &tmap_a, it * BK, m0, bz, bar_full + 8 * s);
        else tma_load_2d(sa, &tmap_a, it * BK, m0, bar_full + 8 * s);
        if (p.b_mode == B_TMA_NK) {
          if (p.b_batched) tma_load_3d(sb, &tmap_b, it * BK, n0, bz, bar_full + 8 * s);
          else tma_load_2d(sb, &tmap_b, it * BK, n0, bar_full + 8 * s);
        } else if (p.b_mode == B_TMA_KN) {
#pragma unroll
          for (int j = 0; j < BN / 32; ++j) {  // one 32-column x BK-row box per block
            if (p.b_batched)
              tma_load_3d(sb + j * (BK * 128), &tmap_b, n0 + 32 * j, it * BK, bz, bar_full + 8 * s);
            else
              tma_load_2d(sb + j * (BK * 128), &tmap_b, n0 + 32 * j, it * BK, bar_full + 8 * s);
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer
    if (lane == 0) {
      // instruction descriptor: D fp32, A/B tf32, A K-major, B K- or N-major, N, M
      const uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((b_n_major ? 1u : 0u) << 16) |
                             ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(BM >> 4) << 24);
      bool ok = true;
      for (int it = 0; it < KT && ok; ++it) {  // local k-step
        const int s = it % STAGES;
        const uint32_t ph = (uint32_t)(it / STAGES) & 1u;
        ok = mbar_wait(bar_full + 8 * s, ph, abort_flag, &g_gemm_error);
        if (!ok) break;
        fence_proxy_async();
        tc_fence_after();
        const uint32_t sa = base + s * STAGE_BYTES, sb = sa + A_BYTES;
#pragma unroll
        for (int kk = 0; kk < BK / 8; ++kk) {
          // A, K-major: rows of 128 bytes, 8-row groups 1024 bytes apart; a k-step of 8
          // tf32 is 32 bytes along the row.
          const uint64_t ad = smem_desc(sa + kk * 32, 16, 1024, 2);
          // B, K-major ([N,K] source): same shape as A.  B, N-major ([K,N] / kn4 source):
          // 32-column blocks of BK rows x 128 bytes, blocks 4096 bytes apart (leading
          // offset), 4-row k groups 512 bytes apart (stride offset); a k-step of 8 rows
          // starts 1024 bytes after the previous one.
          const uint64_t bd = b_n_major ? smem_desc(sb + kk * 1024, BK * 128, 512, 1)
                                          : smem_desc(sb + kk * 32, 16, 1024, 2);
          umma_tf32(tmem_base, ad, bd, idesc, (it | kk) != 0 ? 1u : 0u);
        }
        umma_commit(bar_empty + 8 * s);
      }
      if (ok) umma_commit(bar_done);
    }
  } else {
    // ---------------- B loader (warps 2..5), then epilogue
    const int lt = threadIdx.x - 64;  // 0..127
    if (b_by_loader) {
      // The stage's 1024 16-byte chunks are numbered panel piece by panel piece (a piece =
      // the part of a kn4 panel inside this tile's 128 columns), row-major inside a piece,
      // which is the order the packed buffer stores them: chunk e = i * 128 + lt, so every
      // warp-wide cp.async reads 512 contiguous bytes.  The mapping e -> (row, column,
      // panel terms) does not depend on the k-step and is worked out once per thread.
      int a_kl[BK / 4], a_term[BK / 4], a_w[BK / 4], a_in[BK / 4];
      uint32_t a_dst[BK / 4];
#pragma unroll
      for (int i = 0; i < BK / 4; ++i) { a_kl[i] = 0; a_term[i] = 0; a_w[i] = -1; a_in[i] = 0; a_dst[i] = 0; }
      {
        const int tile_end = n0 + BN;
        const int n_end = p.N < tile_end ? p.N : tile_end;
        int cum = 0, col = n0;
        while (col < tile_end) {
          int wc, term = 0, w = -1, in0 = 0;  // wc: chunks of this piece per k-row
          if (col < n_end) {
            const kn4::Chunk nc = kn4::axis_chunk(p.N, kn4::kTileN, col);
            const kn4::Panel pn = kn4::panel_of(nc.len, col - nc.start);
            const int pend = (int)(nc.start + pn.start + pn.width);
            const int piece_end = pend < n_end ? pend : n_end;
            wc = (piece_end - col) / 4;
            term = (int)(nc.start + pn.start);
            w = (int)pn.width;
            in0 = (int)(col - nc.start - pn.start);
          } else {
            wc = (tile_end - col) / 4;  // columns past N: zero-filled
          }
          if (wc <= 0) break;  // cannot happen for N % 4 == 0; never spin
#pragma unroll
          for (int i = 0; i < BK / 4; ++i) {
            const int e = i * LOADER_THREADS + lt - cum;
            if (e >= 0 && e < BK * wc) {
              const int kl = e / wc, ci = e - kl * wc;
              const int c = (col - n0) / 4 + ci;
              a_kl[i] = kl;
              a_term[i] = term;
              a_w[i] = w;
              a_in[i] = in0 + 4 * ci;
              // 32-column block, row, then the 32-byte unit XOR (row % 4) and the 16-byte half
              a_dst[i] = (uint32_t)(c >> 3) * (BK * 128) + (uint32_t)kl * 128u +
                         (uint32_t)(((((c & 7) >> 1) ^ (kl & 3)) << 5) | ((c & 1) << 4));
            }
          }
          cum += BK * wc;
          col += 4 * wc;
        }
      }
      // K chunks: 352 rows each up to `k_uniform`, then the two chunks that share the
      // remainder (kn4.h); all in 32-bit arithmetic, the element offset in 64-bit.
      constexpr int TK = (int)kn4::kTileK;
      int k_uniform = p.K, k_split = p.K, len0 = p.K < TK ? p.K : TK;
      if (p.K >= TK && p.K % TK != 0) {
        k_uniform = (p.K / TK - 1) * TK;
        const int res = p.K - k_uniform;
        int first = (res / 2) / 12 * 12;
        if (res - first > first + 1) first += 12;
        k_split = k_uniform + first;
      }
      for (int li = 0; li < KT; ++li) {
        const int it = it0 + li;
        const int s = li % STAGES;
        const uint32_t ph = (uint32_t)(li / STAGES) & 1u;
        if (!mbar_wait(bar_empty + 8 * s, ph ^ 1u, abort_flag, &g_gemm_error)) break;
        const uint32_t sb = base + s * STAGE_BYTES + A_BYTES;
#pragma unroll
        for (int i = 0; i < BK / 4; ++i) {
          const int k = it * BK + a_kl[i];
          const bool ok = a_w[i] > 0 && k < p.K;
          const float* src = p.B;
          if (ok) {
            int start, len;
            if (k < k_uniform) {
              start = k / TK * TK;
              len = len0;
            } else if (k < k_split) {
              start = k_uniform;
              len = k_split - k_uniform;
            } else {
              start = k_split;
              len = p.K - k_split;
            }
            src = p.B + ((long long)start * p.N + (long long)len * a_term[i] +
                         (long long)((k - start) * a_w[i] + a_in[i]));
          }
          cp_async16(sb + a_dst[i], src, ok ? 16u : 0u);
        }
        cp_async_arrive_noinc(bar_full + 8 * s);
      }
      cp_async_wait_all();
    }
    // epilogue: warp w may touch TMEM lanes 32 (w % 4) .. 32 (w % 4) + 31
    const int q = warp & 3;
    done = __all_sync(0xffffffffu, mbar_wait(bar_done, 0, abort_flag, &g_gemm_error)) != 0;
    tc_fence_after();
    if (done) {
      // Phase 1: this warp's 32 x 128 accumulator slab, scaled by alpha, goes to shared
      // memory (the stage ring is idle once `done` has fired), rows padded to 132 floats.
      float* slab = reinterpret_cast<float*>(gen_base) + (size_t)q * 32 * LD;
      const uint32_t trow = tmem_base + ((uint32_t)(q * 32) << 16);
      constexpr int CW = STAGES <= 3 ? 32 : 64;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += CW) {
        uint32_t r[CW / 32][32];
        if (KT > 0) {
          tmem_ld32(trow + (uint32_t)c0, r[0]);
          if (CW == 64) tmem_ld32(trow + (uint32_t)c0 + 32u, r[CW / 32 - 1]);
          tmem_ld_wait();
        } else {  // a split-K rank without k-steps contributes zeros
#pragma unroll
          for (int j = 0; j < CW; ++j) r[j >> 5][j & 31] = 0u;
        }
#pragma unroll
        for (int j = 0; j < CW; j += 4) {
          const uint32_t* rj = &r[j >> 5][j & 31];
          *reinterpret_cast<float4*>(slab + lane * LD + c0 + j) =
              make_float4(p.alpha * __uint_as_float(rj[0]), p.alpha * __uint_as_float(rj[1]),
                          p.alpha * __uint_as_float(rj[2]), p.alpha * __uint_as_float(rj[3]));
        }
      }
      __syncwarp();
    }
    tc_fence_before();
  }
  // Split K: every rank's partial tile is in its shared memory now.
  if (p.split > 1) {
    __syncwarp();
    cluster_sync_all();
  }
  if (warp >= 2) {
    const int q = warp & 3;
    if (done) {
      const float* slab = reinterpret_cast<const float*>(gen_base) + (size_t)q * 32 * LD;
      const uint32_t slab_s = base + (uint32_t)((size_t)q * 32 * LD * sizeof(float));
      // Phase 2: one output row per instruction, the 32 lanes cover its 128 columns with
      // 16-byte accesses, so C, the addend and the bias are read and written coalesced.
      // Under split K rank c takes the rows rr with rr % split == c and adds the ranks'
      // partial rows in rank order.  Two rows go together: their reads of C, the addend and
      // the partial tiles are all out before the first is used.  One row at a time, behind
      // ordered volatile loads, paid the memory latency for every row: 512 x 1024 x 1024 with an
      // addend 12.7 us against 11.1 us, 1024^3 17.0 / 14.6, 2000 x 500 x 400 13.5 / 11.1 (four
      // rows: 11.7, 14.3, 11.0, but 200 x 256 x 512 8.9 against 7.6).
      constexpr int RB = 2;
      const int col = n0 + lane * 4;
      const bool vec = col + 3 < p.N && ((p.ldc & 3) == 0) && ((reinterpret_cast<uintptr_t>(p.C) & 15) == 0);
      const bool add_vec = col + 3 < p.N && p.addend && ((p.ld_addend & 3) == 0) &&
                           ((reinterpret_cast<uintptr_t>(p.addend) & 15) == 0);
      // four columns of a row, those past the edge read as zero
      auto load4 = [&](const float* q4, bool wide) {
        float4 t = make_float4(0.f, 0.f, 0.f, 0.f);
        if (wide) return *reinterpret_cast<const float4*>(q4);
        if (col < p.N) t.x = q4[0];
        if (col + 1 < p.N) t.y = q4[1];
        if (col + 2 < p.N) t.z = q4[2];
        if (col + 3 < p.N) t.w = q4[3];
        return t;
      };
      float4 bias4 = make_float4(0.f, 0.f, 0.f, 0.f);
      if (p.bias) bias4 = load4(p.bias + col, false);
      const int rows_here = col < p.N ? min(32, p.M - (m0 + q * 32)) : 0;
      const int rstep = p.split > 1 ? p.split : 1;
      const long long row0 = m0 + q * 32;
      const bool reads_rows = p.beta != 0.f || p.addend;
#pragma unroll 1
      for (int rr0 = crank; rr0 < rows_here; rr0 += rstep * RB) {
        float4 v[RB], old[RB], add[RB];
#pragma unroll
        for (int i = 0; i < RB; ++i) {
          const int rr = rr0 + i * rstep;
          if (reads_rows && rr < rows_here) {
            if (p.beta != 0.f) old[i] = load4(p.C + zb * p.stride_c + (row0 + rr) * p.ldc + col, vec);
            if (p.addend) add[i] = load4(p.addend + zb * p.stride_addend + (row0 + rr) * p.ld_addend + col, add_vec);
          }
        }
        if (p.split > 1) {
#pragma unroll
          for (int i = 0; i < RB; ++i) v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int r = 0; r < p.split; r += 2) {  // (split is even) four partial pieces in flight
            float4 t[2][RB];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
              const uint32_t peer = mapa_u32(slab_s, (uint32_t)(r + h));
#pragma unroll
              for (int i = 0; i < RB; ++i) {
                const int rr = min(rr0 + i * rstep, 31);
                // volatile keeps it behind the cluster barrier; no memory clobber, so that the
                // loads are issued back to back
                asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
                             : "=f"(t[h][i].x), "=f"(t[h][i].y), "=f"(t[h][i].z), "=f"(t[h][i].w)
                             : "r"(peer + (uint32_t)((rr * LD + lane * 4) * sizeof(float))));
              }
            }
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int i = 0; i < RB; ++i) {
                v[i].x += t[h][i].x; v[i].y += t[h][i].y; v[i].z += t[h][i].z; v[i].w += t[h][i].w;
              }
          }
        } else {
#pragma unroll
          for (int i = 0; i < RB; ++i)
            v[i] = *reinterpret_cast<const float4*>(slab + min(rr0 + i, 31) * LD + lane * 4);
        }
#pragma unroll
        for (int i = 0; i < RB; ++i) {
          const int rr = rr0 + i * rstep;
          if (rr >= rows_here) break;
          float* crow = p.C + zb * p.stride_c + (row0 + rr) * p.ldc + col;
          float o[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
          if (p.beta != 0.f) {
            o[0] += p.beta * old[i].x; o[1] += p.beta * old[i].y; o[2] += p.beta * old[i].z; o[3] += p.beta * old[i].w;
          }
          if (p.addend) {
            o[0] += add[i].x; o[1] += add[i].y; o[2] += add[i].z; o[3] += add[i].w;
          }
          o[0] += bias4.x; o[1] += bias4.y; o[2] += bias4.z; o[3] += bias4.w;
          if (p.act == ANNC_ACT_RELU) {
#pragma unroll
            for (int e = 0; e < 4; ++e) o[e] = fmaxf(o[e], 0.0f);
          } else if (p.act == ANNC_ACT_SIGMOID) {
            const float4 t = sigmoid4(make_float4(o[0], o[1], o[2], o[3]));
            o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
          }
          if (vec) {
            *reinterpret_cast<float4*>(crow) = make_float4(o[0], o[1], o[2], o[3]);
          } else {
#pragma unroll
            for (int e = 0; e < 4; ++e)
              if (col + e < p.N) crow[e] = o[e];
          }
        }
      }
    }
  }
  // Nobody leaves while a peer may still read its partial tile.
  if (p.split > 1) {
    __syncwarp();
    cluster_sync_all();
  }
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base),
                 "r"((uint32_t)TMEM_COLS)
                 : "memory");
  }
}

// ---------------------------------------------------------------- host side
bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; }

// Clusters of `size` CTAs of the six-stage kernel (one CTA per SM) that the device holds at once.
int max_clusters(int size) {
  static int known[kMaxDevices][4] = {};
  int& n = known[device_slot()][size == 2 ? 1 : size == 4 ? 2 : 3];
  if (n == 0) {
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)size;
    cfg.gridDim = dim3(1, 1, (unsigned)size);
    cfg.blockDim = dim3(NUM_THREADS);
    cfg.dynamicSmemBytes = smem_bytes(6);
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int got = 0;
    if (cudaOccupancyMaxActiveClusters(&got, gemm_tf32_tcgen05_kernel<6>, &cfg) != cudaSuccess || got < 1) {
      cudaGetLastError();
      got = 148 / size / 2;
    }
    n = got;
  }
  return n;
}

}  // namespace

bool tc_supported(const annc_gemm_desc& d, int math) {
  if (math != ANNC_MATH_TF32 || (d.io_flags & ~ANNC_IO_SINGLE) != 0) return false;
  if (d.trans_a || d.batch < 1 || d.batch > 65535) return false;
  if (d.batch > 1) {  // strided batch: rank-3 tensor maps need 16-byte batch pitches
    if (d.b_format != ANNC_B_PLAIN || (d.stride_a & 3) || (d.stride_b & 3) || d.stride_a <= 0 ||
        d.stride_c <= 0 || (d.stride_c & 3) || (d.addend && (d.stride_addend & 3)))
      return false;
  }
  if (d.m < 64 || d.n < 16 || d.k < 32) return false;
  if (d.m > 128LL * 65535 || d.n > (1LL << 30) || d.k > (1LL << 30)) return false;
  if (!al16(d.a) || (d.lda & 3) || (d.k & 3)) return false;  // TMA: 16-byte base and pitch
  if (d.b_format == ANNC_B_KN4) return (d.n & 3) == 0 && al16(d.b);
  if (d.trans_b) return al16(d.b) && (d.ldb & 3) == 0;       // [N,K] by TMA
  return al16(d.b) && (d.ldb & 3) == 0 && (d.n & 3) == 0;    // [K,N] by 16-byte cp.async
}

int run_tc(const annc_gemm_desc& d, int math, cudaStream_t s) {
  if (!tc_supported(d, math)) return fail(ANNC_ERR_UNSUPPORTED, "tcgen05 gemm: unsupported shape");
  static bool attr_set_dev[kMaxDevices] = {};
  bool& attr_set = attr_set_dev[device_slot()];
  if (!attr_set) {
    ANNC_CUDA(cudaFuncSetAttribute(gemm_tf32_tcgen05_kernel<3>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(3)));
    ANNC_CUDA(cudaFuncSetAttribute(gemm_tf32_tcgen05_kernel<6>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(6)));
    attr_set = true;
  }
  CUtensorMap ta, tb;
  const bool batched = d.batch > 1, b_batched = batched && d.stride_b > 0;
  if (batched) ANNC_TRY(make_map3(&ta, d.a, d.batch, d.m, d.k, d.lda, d.stride_a, BM, false));
  else ANNC_TRY(make_map(&ta, d.a, d.m, d.k, d.lda, BM, false));
  TcParams p;
  memset(&p, 0, sizeof(p));
  p.batched = batched;
  p.b_batched = b_batched;
  p.stride_c = batched ? d.stride_c : 0;
  p.stride_addend = batched ? d.stride_addend : 0;
  p.M = (int)d.m;
  p.N = (int)d.n;
  p.K = (int)d.k;
  if (d.b_format == ANNC_B_KN4) {
    p.b_mode = B_KN4;
    tb = ta;
  } else if (d.trans_b) {
    p.b_mode = B_TMA_NK;
    if (b_batched) ANNC_TRY(make_map3(&tb, d.b, d.batch, d.n, d.k, d.ldb, d.stride_b, BN, false));
    else ANNC_TRY(make_map(&tb, d.b, d.n, d.k, d.ldb, BN, false));
  } else {
    p.b_mode = B_TMA_KN;
    if (b_batched) ANNC_TRY(make_map3(&tb, d.b, d.batch, d.k, d.n, d.ldb, d.stride_b, BK, true));
    else ANNC_TRY(make_map(&tb, d.b, d.k, d.n, d.ldb, BK, true));
  }
  p.B = d.b;
  p.ldb = d.ldb;
  p.C = d.c;
  p.ldc = d.ldc;
  p.addend = d.addend;
  p.ld_addend = d.ld_addend;
  p.bias = d.bias;
  p.alpha = d.alpha;
  p.beta = d.beta;
  p.act = d.activation;
  dim3 grid((unsigned)((d.n + BN - 1) / BN), (unsigned)((d.m + BM - 1) / BM), (unsigned)d.batch);
  const long long ctas = (long long)grid.x * grid.y * grid.z;
  // Few tiles and a long K: a cluster of 2, 4 or 8 CTAs shares each tile and splits its K range,
  // so that a 512 x 1024 x 1024 product occupies 128 SMs instead of 32.
  const int kt_all = (int)((d.k + BK - 1) / BK);
  // All clusters have to be resident at once: one more round costs more than the split gives
  // (192 x 1024 x 1024, 16 tiles: 14.5 us in clusters of 8, of which 15 fit, 10.0 us in clusters of 4; 128 x 2304 x 1024 16.5 / 10.1).
  int split = 1;
  if (d.batch == 1 && ctas * 2 <= 148 && kt_all >= 8) {
    while (split < 8 && ctas <= max_clusters(split * 2) && kt_all / (split * 2) >= 2) split *= 2;
  }
  p.split = split;
  if (split > 1) grid.z = (unsigned)split;
  const bool deep = split > 1 || ctas <= 148 * 3 / 2;
  cudaLaunchConfig_t cfg;
  memset(&cfg, 0, sizeof(cfg));
  cfg.gridDim = grid;
  cfg.blockDim = dim3(NUM_THREADS);
  cfg.dynamicSmemBytes = smem_bytes(deep ? 6 : 3);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  cfg.attrs = attr;
  if (split > 1) {
    cudaLaunchAttribute& a = attr[cfg.numAttrs++];
    a.id = cudaLaunchAttributeClusterDimension;
    a.val.clusterDim.x = 1;
    a.val.clusterDim.y = 1;
    a.val.clusterDim.z = (unsigned)split;
  }
  if (early_launch(d)) attr[cfg.numAttrs++] = pdl_attribute();
  ANNC_CUDA(deep ? cudaLaunchKernelEx(&cfg, gemm_tf32_tcgen05_kernel<6>, ta, tb, p)
                 : cudaLaunchKernelEx(&cfg, gemm_tf32_tcgen05_kernel<3>, ta, tb, p));
  ANNC_CUDA(cudaGetLastError());
  return ANNC_OK;
}

int* gemm_error_word() {
  static int* addr_dev[kMaxDevices] = {};
  int*& addr = addr_dev[device_slot()];
  if (!addr) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_gemm_error) == cudaSuccess) addr = static_cast<int*>(p);
  }
  return addr;
}

int read_error_flag(int* flag) {
  ANNC_CUDA(cudaMemcpyFromSymbol(flag, g_gemm_error, sizeof(int)));
  return ANNC_OK;
}

}  // namespace gemm
}  // namespace annc

namespace annc { int dot_interaction_error_flag(int* flag); }

// Sets the device-side error word of the tensor-core kernels (what a CTA does when a bounded
// wait runs out), so that the host-side reporting can be exercised without a kernel that
// actually gives up.  annc_gemm_check and the custom calls report it; 0 clears it.
extern "C" int annc_gemm_debug_set_error_word(int value) {
  ANNC_CUDA(cudaMemcpyToSymbol(annc::gemm::g_gemm_error, &value, sizeof(int)));
  return ANNC_OK;
}

extern "C" int annc_gemm_check(void* stream, int* timed_out) {
  if (!timed_out) return annc::fail(ANNC_ERR_INVALID_ARGUMENT, "null argument");
  ANNC_CUDA(cudaStreamSynchronize(static_cast<cudaStream_t>(stream)));
  int a = 0, b = 0;
  ANNC_TRY(annc::gemm::read_error_flag(&a));
  ANNC_TRY(annc::dot_interaction_error_flag(&b));
  *timed_out = (a | b) ? 1 : 0;
  return ANNC_OK;
}
