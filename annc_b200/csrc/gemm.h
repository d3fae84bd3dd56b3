// Internal interface of the GEMM core.
#pragma once

#include <cuda_runtime.h>

#include "annc_b200.h"

namespace annc {
namespace gemm {

// bias[b*s0 + i*s1 + j*s2]: the numpy-style broadcast of
// KPFusedBatchMatMulAddSigmoid (fused_batchmatmul_add_sigmoid.cc:197-214).
struct BiasBroadcast {
  long long s0, s1, s2;
};

// CUDA-core fp32 route; takes every shape, both transposes and the kn4 B format.
int run_simt(const annc_gemm_desc& d, cudaStream_t s, const BiasBroadcast* bb = nullptr);

// Whether a product's blocks may take their places while the kernel before it on the stream drains (pdl.cuh).
// us back to back, without / with: 200 x 512 x 256 7.3 / 6.3, 512 x 1024 x 1024 9.8 / 9.2, 4096 x 512 x 416 11.2 / 10.4,
// 65536 x 64 x 256 23.7 / 22.2, 1024 x 2048 x 2048 28.3 / 27.3; to trigger behind the main loop instead of before
// it is the same.  Less of it as a product gets longer, but none lost: 8192 x 4096 x 2048 254 / 251, BF16 256 x 1024 x 4096
// 28.7 / 26.4, 16384 x 512 x 1024 26.6 / 23.5, 2048 x 1024 x 8192 51.8 / 49.3, 16384 x 1024 x 8192 253 / 247 (runs
// of one side 1 % apart), and the three layers of which that is the first 283 / 276.  Not beside another stream's kernel that needs the room, which is what ANNC_IO_SINGLE is for, and
// not where C is added to (600 x 2048 x 128 11.6 / 13.1, 256 x 5120 x 512 16.0 / 17.8, 1024 x 2048 x 2048 32.6 / 34.4).
inline bool early_launch(const annc_gemm_desc& d) { return !(d.io_flags & ANNC_IO_SINGLE) && d.beta == 0.f; }

// tcgen05 route: whether the descriptor fits, and the launch.
bool tc_supported(const annc_gemm_desc& d, int math);
int run_tc(const annc_gemm_desc& d, int math, cudaStream_t s);

// Persistent CTA-pair tcgen05 kernel (TF32 with fp32 operands, BF16 with bf16 operands).
bool pair_supported(const annc_gemm_desc& d, int math);
int run_pair(const annc_gemm_desc& d, int math, cudaStream_t s);
// Whether its epilogue for this descriptor stores by TMA (no beta * C or softmax, aligned rows).
bool pair_stores_by_tma(const annc_gemm_desc& d);
// How many of its `tiles` 256 x 256 tiles it takes whole on a chip of so many SM pairs; the rest of
// the last round is cut in halves (and only then the kernel's tile width is a run-time value).
long long pair_whole_tiles(const annc_gemm_desc& d, int math, long long tiles, long long pairs);

// A kn4-packed B re-laid into a 16-byte aligned buffer of 4*K*N bytes: relaid_desc returns 0 when that
// does not pay off, else the form the weight takes there (1 = [N,K], 2 = [K,N]) and fills `plain`
// with the equivalent plain-layout descriptor but for `b`; relay_kn4 runs the conversion (`kept`: once
// for many products).
int relaid_desc(const annc_gemm_desc& d, bool kept, annc_gemm_desc* plain);
void relay_kn4(const float* packed, float* ws, long long k, long long n, int form, cudaStream_t s);
// Device-side error word of the tensor-core kernels (a bounded wait that ran out).
int read_error_flag(int* flag);

// Picks the route the way annc_gemm_run does; returns a static name.
const char* route_name(const annc_gemm_desc& d);

}  // namespace gemm
}  // namespace annc
