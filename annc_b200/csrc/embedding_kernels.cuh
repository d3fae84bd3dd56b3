// Device kernels of the embedding path: segment prepass, bag (gather + segment
// reduce, with the fused uint64 hash-bucket modulo), the atomic route for
// unsorted segment ids, single-row gathers, and the helpers of the
// unique / non-zero ops.  HBM-bound: every table row is read once with 16-byte
// loads, every output row is written once.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.h"
#include "emb_device.cuh"
#include "pdl.cuh"

namespace annc {
namespace emb {

constexpr int kMaxTables = 120;         // tables per grouped launch: BagParams is 7.7 KB of the 32 KB
                                        // parameter space, the per-table marks fit the 512-byte header
constexpr int kErrRow = 1;              // row index outside its table
constexpr int kErrSegment = 2;          // segment id outside [0, batch)

// Head of the bag workspace (512 bytes), then int32 offsets[num_tables][batch + 1].
struct BagHeader {
  int err_bits;
  int any_unsorted;          // some table of the call is marked below
  int pad;
  int next_chunks;           // lookup-granular kernel: warps' worth of chunks handed out so far
  int unsorted[kMaxTables];  // per table: segment ids were seen to decrease
};
static_assert(sizeof(BagHeader) <= 512, "header layout");
constexpr size_t kHeaderBytes = 512;

__device__ __forceinline__ void mark_unsorted(BagHeader* hdr, int t) {
  hdr->unsorted[t] = 1;
  hdr->any_unsorted = 1;
}

struct BagTableDev {
  const float* table;
  const void* ids;
  const int64_t* seg;  // slice_input
  float* out;
  unsigned long long num_buckets;
  unsigned long long magic;  // floor((2^64 - 1) / num_buckets): reciprocal for the exact modulo
  const int* given_off;      // caller-supplied bag offsets [batch + 1] (then `seg` is not read)
  int rows;                  // (local) table rows and lookups: both below 2^31
  int nnz;
};
static_assert(sizeof(BagTableDev) == 64, "BagParams size is budgeted on 64-byte table entries");

struct BagParams {
  BagTableDev t[kMaxTables];
  int num_tables;
  int id_kind;  // 0 i32 rows, 1 i64 rows, 2 u64 fingerprints
  int combiner;
  int col;
  long long ncols;
  long long batch;
  long long dim;
  long long out_stride;
  int shard_count;  // row sharding: this rank owns rows r with r % shard_count == shard_rank,
  int shard_rank;   // stored at local row r / shard_count (the reference's mod-partition rule)
  int skip_empty;   // row sharding: bags without a lookup owned by this rank are not written
};

// ---- prepass: CSR offsets from the (sorted) segment column --------------------
// Thread i in [0, nnz] looks at the boundary between lookups i-1 and i and writes
// offsets[s] = i for every segment s in (seg[i-1], seg[i]] (empty bags included),
// with virtual seg[-1] = -1 and seg[nnz] = batch.  A decrease marks the table
// unsorted; ids outside [0, batch) set kErrSegment.
__global__ void bag_prepass_kernel(BagParams p, BagHeader* hdr, int* offsets) {
  const int t = blockIdx.y;
  const BagTableDev& T = p.t[t];
  if (T.given_off) return;
  int* off = offsets + (long long)t * (p.batch + 1);
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i <= T.nnz; i += stride) {
    long long prev = (i == 0) ? -1 : T.seg[(i - 1) * p.ncols + p.col];
    long long cur = (i == T.nnz) ? p.batch : T.seg[i * p.ncols + p.col];
    if (i < T.nnz && (cur < 0 || cur >= p.batch)) {
      atomicOr(&hdr->err_bits, kErrSegment);
      cur = cur < 0 ? 0 : p.batch;
    }
    if (prev < -1) prev = -1;
    if (prev > p.batch) prev = p.batch;
    if (cur < prev) {
      if (i < T.nnz) mark_unsorted(hdr, t);
      continue;
    }
    for (long long s = prev + 1; s <= cur; ++s) off[s] = (int)i;
  }
}

// Same boundary walk for the common two-column index matrix (sample, position): every
// thread reads its whole 16-byte row, so a warp reads 512 contiguous bytes, and takes the
// previous lookup's segment id from its neighbour lane.
__global__ void __launch_bounds__(256)
bag_prepass2_kernel(BagParams p, BagHeader* hdr, int* offsets) {
  const int t = blockIdx.y;
  const BagTableDev& T = p.t[t];
  if (T.given_off) return;
  int* off = offsets + (long long)t * (p.batch + 1);
  const int lane = threadIdx.x & 31;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long n_round = (T.nnz + 1 + 31) / 32 * 32;  // whole warps walk the loop together
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n_round; i += stride) {
    long long cur = p.batch;
    if (i < T.nnz) {
      const longlong2 v = __ldg(reinterpret_cast<const longlong2*>(T.seg) + i);
      cur = p.col == 0 ? v.x : v.y;
    }
    long long prev = __shfl_up_sync(0xffffffffu, cur, 1);
    if (lane == 0) prev = (i == 0) ? -1 : (i - 1 < T.nnz ? T.seg[(i - 1) * 2 + p.col] : p.batch);
    if (i > T.nnz) continue;
    if (i < T.nnz && (cur < 0 || cur >= p.batch)) {
      atomicOr(&hdr->err_bits, kErrSegment);
      cur = cur < 0 ? 0 : p.batch;
    }
    if (prev < -1) prev = -1;
    if (prev > p.batch) prev = p.batch;
    if (cur < prev) {
      if (i < T.nnz) mark_unsorted(hdr, t);
      continue;
    }
    for (long long s = prev + 1; s <= cur; ++s) off[s] = (int)i;
  }
}

// Row sharding.  Returns the local row, or -2 when another rank owns the row.  Rows below
// 2^32 (every real table) take 32-bit arithmetic.
constexpr long long kNotMine = -2;
__device__ __forceinline__ long long shard_row(long long r, int shard_count, int shard_rank) {
  if (shard_count <= 1 || r < 0) return r;
  if ((unsigned long long)r <= 0xffffffffull) {
    const unsigned b = (unsigned)r, q = b / (unsigned)shard_count;
    return (b - q * (unsigned)shard_count == (unsigned)shard_rank) ? (long long)q : kNotMine;
  }
  if ((int)(r % shard_count) != shard_rank) return kNotMine;
  return r / shard_count;
}
// Owner rank of row r >= 0 under the same rule.
__device__ __forceinline__ int shard_owner(long long r, int shard_count) {
  if ((unsigned long long)r <= 0xffffffffull) return (int)((unsigned)r % (unsigned)shard_count);
  return (int)(r % shard_count);
}

// Position of the k-th (0-based) set bit of m; k must be below popc(m).
__device__ __forceinline__ int kth_set_bit(unsigned m, int k) {
  int pos = 0;
  int c = __popc(m & 0xffffu);
  if (k >= c) { k -= c; pos += 16; m >>= 16; }
  c = __popc(m & 0xffu);
  if (k >= c) { k -= c; pos += 8; m >>= 8; }
  c = __popc(m & 0xfu);
  if (k >= c) { k -= c; pos += 4; m >>= 4; }
  c = __popc(m & 0x3u);
  if (k >= c) { k -= c; pos += 2; m >>= 2; }
  if (k >= (int)(m & 1u)) pos += 1;
  return pos;
}

// ---- bag kernel: LANES lanes own one bag; each lane owns VPL float4 columns -----
// Rows are added in lookup order into a zero accumulator, the order of the
// reference's scalar loop, so sums are bit-identical for sorted input.  Four
// row loads are in flight per group.  For an unsorted table the group writes the
// zero row and clears the bag's counter; the scatter kernels then do the work.
// SHARDED (row sharding): the lookups this rank owns are first compacted inside the group
// (lookup order kept), so that the four loads in flight are all real ones, and with
// skip_empty a bag without an owned lookup is left unwritten (its owner knows from the
// bag's ids which ranks contribute, see bag_owner_mask_kernel).
template <int LANES, int VPL, bool SHARDED>
__global__ void __launch_bounds__(256, VPL == 1 ? 5 : 3)
bag_reduce_kernel(BagParams p, BagHeader* hdr, int* offsets) {
  constexpr int GROUPS_PER_WARP = 32 / LANES;
  const int lane_in_warp = threadIdx.x & 31;
  const int lane = lane_in_warp % LANES;
  const unsigned gmask =
      (LANES == 32) ? 0xffffffffu : (((1u << LANES) - 1u) << ((lane_in_warp / LANES) * LANES));
  const long long group =
      ((long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) * GROUPS_PER_WARP +
      lane_in_warp / LANES;
  const long long total = (long long)p.num_tables * p.batch;
  if (group >= total) return;
  const int t = (int)(group / p.batch);
  const long long s = group - (long long)t * p.batch;
  const BagTableDev& T = p.t[t];
  int* off = offsets + (long long)t * (p.batch + 1);
  const int* roff = T.given_off ? T.given_off : off;
  float* orow = T.out + s * p.out_stride;

  float4 acc[VPL];
#pragma unroll
  for (int v = 0; v < VPL; ++v) acc[v] = make_float4(0.f, 0.f, 0.f, 0.f);

  if (hdr->unsorted[t]) {
#pragma unroll
    for (int v = 0; v < VPL; ++v)
      *reinterpret_cast<float4*>(orow + (v * LANES + lane) * 4) = acc[v];
    __syncwarp(gmask);
    if (lane == 0) off[s] = 0;  // becomes the bag's lookup counter
    return;
  }

  const int start = roff[s], end = roff[s + 1];
  if (!SHARDED && p.skip_empty && start == end) return;  // exchange: an empty part is not written
  int owned = 0;  // SHARDED: lookups of this bag that belong to this rank (group-uniform)
  for (int base = start; base < end; base += LANES) {
    int my = -1;  // local row (tables have fewer than 2^31 rows), -1 = skip
    bool mine = false;
    if (base + lane < end) {
      const long long r64 = shard_row(load_row_id(T.ids, p.id_kind, base + lane, T.num_buckets, T.magic),
                                      p.shard_count, p.shard_rank);
      mine = r64 != kNotMine;
      if (r64 != kNotMine && (r64 < 0 || r64 >= T.rows)) atomicOr(&hdr->err_bits, kErrRow);
      else if (r64 != kNotMine) my = (int)r64;
    }
    int n = min(LANES, end - base);
    if (SHARDED) {
      const int shift = (lane_in_warp / LANES) * LANES;
      owned += __popc(__ballot_sync(gmask, mine) >> shift & (LANES == 32 ? 0xffffffffu : ((1u << LANES) - 1u)));
      const unsigned bal = (__ballot_sync(gmask, my >= 0) >> shift) &
                           (LANES == 32 ? 0xffffffffu : ((1u << LANES) - 1u));
      n = __popc(bal);
      const int src = lane < n ? kth_set_bit(bal, lane) : lane;
      const int comp = __shfl_sync(gmask, my, src, LANES);
      my = lane < n ? comp : -1;
    }
    for (int j = 0; j < n; j += 4) {
      int r[4];
      float4 v[4][VPL];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        r[q] = __shfl_sync(gmask, my, (j + q) % LANES, LANES);
        if (j + q >= n) r[q] = -1;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (r[q] >= 0) {
          const float* src = T.table + (long long)r[q] * p.dim;
#pragma unroll
          for (int w = 0; w < VPL; ++w) v[q][w] = ldg4(src + (w * LANES + lane) * 4);
        }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (r[q] >= 0) {
#pragma unroll
          for (int w = 0; w < VPL; ++w) add4(acc[w], v[q][w]);
        }
      }
    }
  }
  if (SHARDED && p.skip_empty && owned == 0) return;
  if (p.combiner == 1 && end > start) {
    const float inv = __fdiv_rn(1.0f, (float)(end - start));
#pragma unroll
    for (int w = 0; w < VPL; ++w) {
      acc[w].x = __fmul_rn(acc[w].x, inv);
      acc[w].y = __fmul_rn(acc[w].y, inv);
      acc[w].z = __fmul_rn(acc[w].z, inv);
      acc[w].w = __fmul_rn(acc[w].w, inv);
    }
  }
#pragma unroll
  for (int w = 0; w < VPL; ++w)
    *reinterpret_cast<float4*>(orow + (w * LANES + lane) * 4) = acc[w];
}

// Which ranks contribute to each bag under row sharding: mask[t][s] has bit g set when bag s
// of table t has at least one lookup whose row r satisfies r % shard_count == g (in or out
// of range: the rule the senders use to decide whether they write the bag).  Half a warp per
// bag; `off` are the bag offsets of the table (given_off).
__global__ void __launch_bounds__(256)
bag_owner_mask_kernel(BagParams p, unsigned* mask) {
  const int lane = threadIdx.x & 15;
  const unsigned gmask = 0xffffu << (threadIdx.x & 16);
  const long long group = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
  const long long total = (long long)p.num_tables * p.batch;
  if (group >= total) return;
  const int t = (int)(group / p.batch);
  const long long s = group - (long long)t * p.batch;
  const BagTableDev& T = p.t[t];
  const int start = T.given_off[s], end = T.given_off[s + 1];
  unsigned m = 0;
  for (int i = start + lane; i < end; i += 16) {
    const long long r = load_row_id(T.ids, p.id_kind, i, T.num_buckets, T.magic);
    if (r >= 0) m |= 1u << shard_owner(r, p.shard_count);  // a negative row is nobody's
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) m |= __shfl_xor_sync(gmask, m, o, 16);
  if (lane == 0) mask[group] = m;
}

// Any dim (not a multiple of 4, or unaligned tables): one warp per bag, lanes
// stride over the columns; same summation order.
__global__ void __launch_bounds__(256)
bag_reduce_generic_kernel(BagParams p, BagHeader* hdr, int* offsets) {
  const int lane = threadIdx.x & 31;
  const long long group = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const long long total = (long long)p.num_tables * p.batch;
  if (group >= total) return;
  const int t = (int)(group / p.batch);
  const long long s = group - (long long)t * p.batch;
  const BagTableDev& T = p.t[t];
  int* off = offsets + (long long)t * (p.batch + 1);
  float* orow = T.out + s * p.out_stride;
  if (hdr->unsorted[t]) {
    for (long long c = lane; c < p.dim; c += 32) orow[c] = 0.f;
    __syncwarp();
    if (lane == 0) off[s] = 0;
    return;
  }
  const int* roff = T.given_off ? T.given_off : off;
  const int start = roff[s], end = roff[s + 1];
  const float inv = (p.combiner == 1 && end > start) ? __fdiv_rn(1.0f, (float)(end - start)) : 1.0f;
  if (p.shard_count > 1 && p.skip_empty) {
    bool any = false;
    for (int i = start + lane; i < end; i += 32)
      any = any || shard_row(load_row_id(T.ids, p.id_kind, i, T.num_buckets, T.magic), p.shard_count,
                             p.shard_rank) != kNotMine;
    if (!__any_sync(0xffffffffu, any)) return;
  }
  for (long long c0 = 0; c0 < p.dim; c0 += 32) {
    const long long c = c0 + lane;
    float acc = 0.f;
    for (int i = start; i < end; ++i) {
      long long r = shard_row(load_row_id(T.ids, p.id_kind, i, T.num_buckets, T.magic), p.shard_count,
                              p.shard_rank);
      if (r == kNotMine) continue;
      if (r < 0 || r >= T.rows) {
        if (lane == 0 && c0 == 0) atomicOr(&hdr->err_bits, kErrRow);
        continue;
      }
      if (c < p.dim) acc = __fadd_rn(acc, __ldg(T.table + r * p.dim + c));
    }
    if (c < p.dim) orow[c] = (p.combiner == 1 && end > start) ? __fmul_rn(acc, inv) : acc;
  }
}

// ---- lookup-granular bag kernel ------------------------------------------------------
// The same pooling without a prepass.  A group of LANES lanes takes a chunk of consecutive
// lookups of a table, tile by tile (LANES lookups, one per lane: ids and segment ids read with
// coalesced loads, the hash-bucket modulo applied by the lane that read the id) and owns the
// bags whose first lookup lies in the chunk; it follows its last bag past the chunk until the
// segment id changes.  Bag boundaries inside a tile are one ballot; rows are added in lookup
// order into a zero accumulator (the reference's order, bit-identical sums).  Bags without
// lookups are zero-filled by the group that owns the next bag (the first bag's owner fills from
// 0, the last bag's owner to the end).  A decrease of the segment ids marks the table unsorted:
// bag_stream_reset_kernel then clears its output and the atomic route below redoes it.
//
// For bags of a few lookups, and for callers that leave it a share of the SMs' block slots; bag_list_kernel
// below takes the others (the line between them: stream_shape_for).
//
// What bounds it: the instructions per lookup and the latency of the row loads.  So the loop
// is an unrolled pipeline: DEPTH - 1 row loads are out before a row is added, across tile borders
// too, the ids of the next tile are already under way, and what only a bag's start needs (its
// number, gaps of empty bags) is kept out of the loop.  Measured, 26 tables x 1 M rows x dim 64,
// batch 16384, 4.47 M lookups: 248 us with the former loop (two loads, then two adds; ids of a
// tile fetched at its start), 189 us now; 26 x 2,100 lookups: 100 us -> 18 us.  Choices at
// that size: DEPTH 2 with 64 registers 202 us, DEPTH 4 with 80 216 us, 64 bytes per lane 289 us,
// groups that drift apart 414 us.  The registers are its limit: at 64 it spills 54 bytes (dim 64; 68 at dim
// 128).
// The chunk length comes from the launch (stream_chunk): short for few lookups, so that they
// spread over all SMs, long enough for a batch that fills the chip several times.
//
// A warp starts on the chunks of its own number and takes its next ones from a counter in the
// header (asked for a chunk ahead), because the blocks do not all start together: beside the
// bottom MLP of a model step most of them wait for registers, and with a fixed share each they ran
// as a second wave (1230 us instead of 650 us on a first pass at batch 65536).
//
// A row has VPL 16-byte vectors per lane; FULL says that LANES * VPL vectors are exactly a row
// (otherwise the lanes past the row end load and store nothing).
struct StreamChunks {
  int first[kMaxTables + 1];  // table t owns the chunks [first[t], first[t + 1]); a table without
                              // lookups gets one chunk per 1024 bags to zero
  int chunk;                  // lookups per chunk of bag_stream_kernel, a multiple of LANES
  int list_chunk[kMaxTables]; // ... per chunk of table t of bag_list_kernel, a multiple of eight up to kBagChunk.  (A
                              // length per table costs the other kernel 3 to 8 % at dim 100.)
};

template <int LANES, int VPL, int DEPTH, bool FULL, int MINB>
__global__ void __launch_bounds__(256, MINB)
bag_stream_kernel(BagParams p, StreamChunks sc, BagHeader* hdr) {
  constexpr int GROUPS_PER_WARP = 32 / LANES;
  constexpr int STEPS = LANES < 8 ? LANES : 8;  // unrolled lookups
  static_assert(STEPS % DEPTH == 0, "the row buffers rotate a whole number of times per round");
  constexpr unsigned kAll = 0xffffffffu;
  constexpr unsigned kLaneMask = LANES == 32 ? kAll : ((1u << LANES) - 1u);
  constexpr int kNoBag = -3;  // a lookup whose segment id is out of range is added nowhere
  __shared__ int s_first[kMaxTables + 1];
  // Bags of the last two tiles' lookups: lookup i at i % (2 * LANES).  Read at bag starts only.
  __shared__ int s_key[256 / LANES][2 * LANES];
  constexpr int kRing = 2 * LANES - 1;
  for (int i = threadIdx.x; i <= p.num_tables; i += blockDim.x) s_first[i] = sc.first[i];
  __syncthreads();
  const int batch = (int)p.batch, ncols = (int)p.ncols, dim = (int)p.dim, out_stride = (int)p.out_stride;
  const int lane = threadIdx.x % LANES;
  const int shift = (int)(threadIdx.x & 31) / LANES * LANES;
  int* const keys = s_key[threadIdx.x / LANES];
  bool col_ok[VPL];
#pragma unroll
  for (int w = 0; w < VPL; ++w) col_ok[w] = FULL || (w * LANES + lane) * 4 < dim;

  // The groups of a warp work side by side on consecutive chunks and stay in step: every loop
  // below has the same trip count for the whole warp (a group that has finished has no rows left
  // to load), otherwise the groups drift apart and are executed one after the other.
  // Chunks are handed out in order, so the whole grid works through one table after the other and
  // ends together.
  unsigned gc_next = (blockIdx.x * 8 + (threadIdx.x >> 5)) * GROUPS_PER_WARP;
  while (gc_next < (unsigned)s_first[p.num_tables]) {
    const unsigned gc0 = gc_next;
    if ((threadIdx.x & 31) == 0)
      gc_next = (gridDim.x * 8 + (unsigned)atomicAdd(&hdr->next_chunks, 1)) * GROUPS_PER_WARP;
    const unsigned gc = gc0 + (threadIdx.x & 31) / LANES;
    const bool have = gc < (unsigned)s_first[p.num_tables];
    int lo = 0, hi = p.num_tables - 1;  // table of chunk gc: last t with first[t] <= gc
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((unsigned)s_first[mid] <= gc) lo = mid;
      else hi = mid - 1;
    }
    const int t = lo;
    const BagTableDev& T = p.t[t];
    const int n = have ? T.nnz : 0;
    const float* __restrict__ tab = T.table + lane * 4;
    float* __restrict__ outp = T.out + lane * 4;

    // rows [a, b) of the output <- 0 (bags without lookups)
    auto zero_fill = [&](int a, int b) {
      for (int s = a; s < b; ++s) {
        float* o = outp + (long long)s * out_stride;
#pragma unroll
        for (int w = 0; w < VPL; ++w)
          if (col_ok[w]) __stcs(reinterpret_cast<float4*>(o + w * LANES * 4), make_float4(0.f, 0.f, 0.f, 0.f));
      }
    };
    const long long chunk = (long long)(gc - (unsigned)s_first[t]);
    if (have && n == 0)  // a table without lookups: every bag is empty
      zero_fill((int)min(chunk * 1024, (long long)batch), (int)min((chunk + 1) * 1024, (long long)batch));

    // ---- the tile being added and the raw ids of the tile after it
    int base = n > 0 ? (int)chunk * sc.chunk : 0;  // below nnz < 2^31
    const int chunk_end = (int)min((long long)n, (long long)base + sc.chunk);
    long long raw_seg = 0;
    unsigned long long raw_id = 0;
    // Ids and outputs pass through once: they leave L2 to the table rows (evict-first).
    auto load_raw = [&](int b) {
      if (b < n - lane) {
        const int i = b + lane;
        raw_seg = __ldcs(reinterpret_cast<const long long*>(T.seg) + (long long)i * ncols + p.col);
        if (p.id_kind == 0) raw_id = (unsigned long long)(long long)__ldcs((const int*)T.ids + i);
        else raw_id = __ldcs((const unsigned long long*)T.ids + i);
      }
    };
    int row = -1;
    int to = 0;              // the tile's lookups before `to` can belong to this group's bags
    unsigned smask = 0;      // bag starts among them
    bool open = false;       // a bag is open after the tile
    bool more = n > 0;       // there is a tile after this one
    // The tile at `base` from its raw ids (a group without one: no rows).
    auto decode = [&]() {
      const bool in = more && base < n - lane;
      int k = kNoBag, r = -1;
      if (in) {
        if (raw_seg < 0 || raw_seg >= batch) atomicOr(&hdr->err_bits, kErrSegment);
        else k = (int)raw_seg;
        const long long r64 = p.id_kind == 2 ? (long long)fast_mod_u64(raw_id, T.num_buckets, T.magic) : (long long)raw_id;
        if (r64 < 0 || r64 >= T.rows) atomicOr(&hdr->err_bits, kErrRow);
        else r = (int)r64;
      }
      if (more) keys[(base + lane) & kRing] = k;
      __syncwarp();
      const int pk = keys[(base + lane - 1) & kRing];
      const bool starts = in && k != pk;
      const unsigned all = (__ballot_sync(kAll, starts) >> shift) & kLaneMask;
      const int tile_n = min(LANES, n - base);
      const bool inside = base < chunk_end;
      const int first = all ? __ffs(all) - 1 : tile_n;
      const int from = open ? 0 : (inside ? first : tile_n);
      const int end = inside ? tile_n : (open ? first : 0);
      const bool mine = more && lane >= from && lane < end;
      row = mine ? r : -1;
      smask = more && end > from ? (all & (kLaneMask >> (LANES - end))) : 0u;
      // lookups whose segment id is not the previous one or its successor: unsorted segment ids,
      // or empty bags in between (the owner of the next bag zeroes them)
      const bool odd = mine && starts && k >= 0 && pk >= -1 && k != pk + 1;
      unsigned gaps = __ballot_sync(kAll, odd);
      if (gaps) {
        if (odd && k < pk) mark_unsorted(hdr, t);
        gaps = (gaps >> shift) & kLaneMask;
        while (gaps) {
          const int i = base + __ffs(gaps) - 1;
          gaps &= gaps - 1;
          zero_fill(keys[(i - 1) & kRing] + 1, keys[i & kRing]);
        }
        __syncwarp();
      }
      if (more) {
        to = end;
        open = open || smask != 0;
        // the table ends here, the open bag ended, or no bag starts in the rest of the chunk
        more = !(base >= n - LANES || (inside ? (!open && base >= chunk_end - LANES) : end < tile_n));
      }
    };

    float4 acc[VPL];
#pragma unroll
    for (int v = 0; v < VPL; ++v) acc[v] = make_float4(0.f, 0.f, 0.f, 0.f);
    int bag = kNoBag;    // bag being summed
    int bag_start = 0;   // its first lookup (the mean's count)
    float4 v[DEPTH][VPL];  // rows on their way
    int vr[DEPTH];         // their numbers (negative: none)

    auto issue = [&](int slot, int j) {
      vr[slot] = __shfl_sync(kAll, row, j, LANES);
      if (vr[slot] >= 0) {
        const float* src = tab + (long long)vr[slot] * dim;
#pragma unroll
        for (int w = 0; w < VPL; ++w)
          if (col_ok[w]) v[slot][w] = ldg4(src + w * LANES * 4);
      }
    };
    auto flush = [&](int end) {
      if (bag >= 0) {
        if (p.combiner == 1) {
          const float inv = __fdiv_rn(1.0f, (float)(end - bag_start));
#pragma unroll
          for (int w = 0; w < VPL; ++w) {
            acc[w].x = __fmul_rn(acc[w].x, inv);
            acc[w].y = __fmul_rn(acc[w].y, inv);
            acc[w].z = __fmul_rn(acc[w].z, inv);
            acc[w].w = __fmul_rn(acc[w].w, inv);
          }
        }
        float* o = outp + (long long)bag * out_stride;
#pragma unroll
        for (int w = 0; w < VPL; ++w)
          if (col_ok[w]) __stcs(reinterpret_cast<float4*>(o + w * LANES * 4), acc[w]);
      }
    };

    if (lane == 0) {
      int before = -1;  // before the first lookup: bags 0 .. key - 1 are empty
      if (base > 0) {
        const long long ps = __ldcs(reinterpret_cast<const long long*>(T.seg) + (long long)(base - 1) * ncols + p.col);
        before = (ps < 0 || ps >= batch) ? kNoBag : (int)ps;
      }
      keys[(base - 1) & kRing] = before;
    }
    load_raw(base);
    decode();
    if (more) load_raw(base + LANES);
#pragma unroll
    for (int k = 0; k < DEPTH - 1; ++k) issue(k, k);
    bool go_on = true;
    while (go_on) {
      unsigned sm = smask;       // bag starts of the tile, the next lookup's bit first
      const int tile = base;
#pragma unroll 1
      for (int j = 0; j < LANES; j += STEPS) {
#pragma unroll
        for (int k = 0; k < STEPS; ++k) {
          // a row load goes out before the row loaded DEPTH - 1 steps ago is added; the last of a
          // tile's are those of the next tile
          if (k + DEPTH - 1 < STEPS || j + STEPS < LANES) {
            issue((k + DEPTH - 1) % DEPTH, j + k + DEPTH - 1);
          } else {
            if (k + DEPTH - 1 == STEPS) {
              go_on = __any_sync(kAll, more);
              if (go_on) {
                if (more) base += LANES;
                decode();
                if (more) load_raw(base + LANES);
              } else {
                row = -1;
              }
            }
            issue((k + DEPTH - 1) % DEPTH, k + DEPTH - 1 - STEPS);
          }
          if (sm & (1u << k)) {
            const int i = tile + j + k;
            flush(i);
#pragma unroll
            for (int w = 0; w < VPL; ++w) acc[w] = make_float4(0.f, 0.f, 0.f, 0.f);
            bag = keys[i & kRing];
            bag_start = i;
          }
          if (vr[k % DEPTH] >= 0) {
#pragma unroll
            for (int w = 0; w < VPL; ++w) add4(acc[w], v[k % DEPTH][w]);
          }
        }
        sm >>= STEPS;
      }
    }
    if (open) {
      flush(base + to);
      // the table's last lookup: bags after its bag are empty
      if (base + to == n && bag >= 0) zero_fill(bag + 1, batch);
    }
    gc_next = __shfl_sync(kAll, gc_next, 0);  // also: the ring is free for the next chunk
  }
  pdl_trigger();
}

// ---- the same by lists of bags ---------------------------------------------------------
// A warp takes a chunk of consecutive lookups of a table and
// owns the bags whose first lookup lies in it; it follows its last bag past the chunk.
//
// First the whole warp decodes a window, the chunk and up to kBagAhead lookups behind it, one lookup
// per lane: ids and segment ids by coalesced evict-first loads, the hash-bucket modulo, the rows'
// addresses into shared memory; one ballot over the bag starts of a tile of 32 makes the list of the
// chunk's bags.  Bags without lookups are zero-filled by the owner of the next bag (the first bag's
// owner fills from 0, the last bag's owner to the end).  A decrease of the segment ids marks the table
// unsorted: bag_stream_reset_kernel then clears its output and the atomic route below redoes it.
//
// Then the warp's groups of LANES lanes take bags from the list, each the next one when it has
// finished its own: a round loads Q rows of every group's bag and adds them in lookup order into a
// zero accumulator (the reference's order, bit-identical sums).  All groups run the same rounds; only
// a finished bag's store and the fetch of the next one are conditional.
//
// What bounds it: the instructions per lookup and the latency of ids and rows; DRAM is at 40 to 55 %.
// Hence: an address, not a row number, in shared memory (computed once, by the lane that decoded it);
// a row of zeros for what is not to be added, so that loads and packed adds need no guards (predicated
// packed adds are made of twice the instructions); rare ids behind one vote per tile.  The kernel above,
// in which every step asks whether a bag begins, and this one, us:
// 539 / 479 for 17.9 M lookups over 26 tables of up to 1 M rows of dim 64, 198 / 180 for 4.5 M over 26
// x 1 M rows, 173 / 144 for 64 x 50 K rows of dim 128 in bags of 25, 12.0 / 9.1 for 26 tables x 2,100
// lookups, 137 / 133 for 6 tables of dim 256.  Tried, us for 4.1 M lookups of dim 64 (this kernel: 127):
// row copies into a ring in shared memory 168, and 358 past L1, whose hits keep the popular rows off their L2
// slices; a warp per bag 179; groups over fixed shares of the chunk 167; windows of 160 lookups 140; two
// 16-byte loads per row and lane instead of one of 32 138.  Ids of eight tiles at a time: 191 instead of 180.
// Chunks are handed out as above.
constexpr int kBagWindow = 256;                   // lookups decoded at a time
constexpr int kBagAhead = 32;                     // of these behind the chunk: the end of its last bag
constexpr int kBagChunk = kBagWindow - kBagAhead;

// F floats of a row (4 or 8), one load of 16 or 32 aligned bytes, as packed pairs; each half of an add rounds
// like __fadd_rn.
template <int F>
struct RowPiece {
  static_assert(F == 4 || F == 8, "16 or 32 bytes");
  unsigned long long v[F / 2];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int k = 0; k < F / 2; ++k) v[k] = 0ull;
  }
  __device__ __forceinline__ void load(const char* p) {
    if (F == 8) {
      asm("ld.global.nc.v4.b64 {%0, %1, %2, %3}, [%4];"
          : "=l"(v[0]), "=l"(v[1]), "=l"(v[F / 2 - 2]), "=l"(v[F / 2 - 1])
          : "l"(p));
    } else {
      const ulonglong2 a = __ldg(reinterpret_cast<const ulonglong2*>(p));
      v[0] = a.x;
      v[1] = a.y;
    }
  }
  __device__ __forceinline__ void add(const RowPiece& o) {
#pragma unroll
    for (int k = 0; k < F / 2; ++k) asm("add.rn.f32x2 %0, %0, %1;" : "+l"(v[k]) : "l"(o.v[k]));
  }
  __device__ __forceinline__ float4 four(int h) const {
    float4 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v[2 * h]));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.z), "=f"(f.w) : "l"(v[2 * h + 1]));
    return f;
  }
};

// What stands for the rows that are not added, behind a bag's end or out of range: adding +0 changes no sum
// that began at +0.
__device__ __align__(32) float g_zero_row[512];

template <int LANES, int F, int VPL, int Q, int MINB>
__global__ void __launch_bounds__(256, MINB)
bag_list_kernel(BagParams p, StreamChunks sc, BagHeader* hdr) {
  constexpr int GROUPS = 32 / LANES;
  constexpr int TILES = 4;  // tiles of 32 lookups whose ids are on their way together
  constexpr unsigned kAll = 0xffffffffu;
  constexpr int kNoBag = -3;  // a lookup whose segment id is out of range is added nowhere
  using Vec = RowPiece<F>;
  __shared__ int s_first[kMaxTables + 1];
  __shared__ unsigned long long s_row[8][kBagWindow + Q];  // where the rows of the decoded lookups are
  // The chunk's bags: number, first lookup and the one behind the last, counted from the window's start
  // (an entry before the first: the one whose end the first bag writes).
  struct BagEntry {
    int bag;
    unsigned short first, end;
  };
  __shared__ __align__(8) BagEntry s_bag[8][kBagChunk + 2];
  for (int i = threadIdx.x; i <= p.num_tables; i += blockDim.x) s_first[i] = sc.first[i];
  __syncthreads();
  const int batch = (int)p.batch;
  const unsigned pitch = (unsigned)p.dim * 4u;                                // bytes of a table row
  const unsigned long long opitch = (unsigned long long)p.out_stride * 4ull;  // between two output rows
  const unsigned long long spitch = (unsigned long long)p.ncols * 8ull;       // between two segment ids
  const int warp = threadIdx.x >> 5, wl = threadIdx.x & 31;
  const int lane = wl % LANES, group = wl / LANES;
  unsigned long long* const rows = s_row[warp];
  const unsigned long long nothing = reinterpret_cast<unsigned long long>(g_zero_row);
  BagEntry* const bags = s_bag[warp] + 1;
  // Lane l holds the floats F l .. F l + F - 1 of every block of F * LANES; a lane past the row's end reads
  // its start instead and writes nothing.  (dim is a multiple of F.)
  bool col_ok[VPL];
  int col[VPL];  // bytes
#pragma unroll
  for (int w = 0; w < VPL; ++w) {
    const int c = (w * LANES + lane) * F;
    col_ok[w] = c < (int)p.dim;
    col[w] = col_ok[w] ? c * 4 : 0;
  }

  unsigned gc_next = blockIdx.x * 8 + warp;
  while (gc_next < (unsigned)s_first[p.num_tables]) {
    const unsigned gc = gc_next;
    if (wl == 0) gc_next = gridDim.x * 8 + (unsigned)atomicAdd(&hdr->next_chunks, 1);
    int lo = 0, hi = p.num_tables - 1;  // table of chunk gc: last t with first[t] <= gc
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if ((unsigned)s_first[mid] <= gc) lo = mid;
      else hi = mid - 1;
    }
    const int t = lo;
    const BagTableDev& T = p.t[t];
    const int n = T.nnz;
    char* const outp = reinterpret_cast<char*>(T.out);
    const unsigned long long tab = reinterpret_cast<unsigned long long>(T.table);
    const char* const segs = reinterpret_cast<const char*>(T.seg + p.col);

    auto store = [&](char* o, const Vec& a, int w, bool mean, float inv) {
#pragma unroll
      for (int h = 0; h < F / 4; ++h) {
        float4 f = a.four(h);
        if (mean) {
          f.x = __fmul_rn(f.x, inv);
          f.y = __fmul_rn(f.y, inv);
          f.z = __fmul_rn(f.z, inv);
          f.w = __fmul_rn(f.w, inv);
        }
        if (col_ok[w]) __stcs(reinterpret_cast<float4*>(o + col[w] + 16 * h), f);
      }
    };
    // rows [a, b) of the output <- 0 (bags without lookups), by the whole warp
    auto zero_fill = [&](int a, int b) {
      Vec z;
      z.zero();
      for (int s = a + group; s < b; s += GROUPS) {
#pragma unroll
        for (int w = 0; w < VPL; ++w) store(outp + (unsigned)s * opitch, z, w, false, 1.f);
      }
    };
    const long long chunk = (long long)(gc - (unsigned)s_first[t]);
    if (n == 0) {  // a table without lookups: every bag is empty
      zero_fill((int)min(chunk * 1024, (long long)batch), (int)min((chunk + 1) * 1024, (long long)batch));
      gc_next = __shfl_sync(kAll, gc_next, 0);
      continue;
    }
    const int base = (int)(chunk * sc.list_chunk[t]);  // below nnz < 2^31
    const int own = (int)min((long long)sc.list_chunk[t], (long long)n - base);

    int before = -1;  // segment of the lookup before the next tile
    if (base > 0) {
      const unsigned long long ps = __ldcs(reinterpret_cast<const unsigned long long*>(segs + (unsigned)(base - 1) * spitch));
      before = ps < (unsigned long long)batch ? (int)ps : kNoBag;
    }
    Vec acc[VPL];
#pragma unroll
    for (int w = 0; w < VPL; ++w) acc[w].zero();
    // The chunk's window, and then windows of the lookups behind it while its last bag goes on: one group
    // (`holder`) has that bag and `counted` lookups of it in its accumulator.
    int from = base, mine = own, window = min(own + kBagAhead, n - base);
    int holder = -1, counted = 0, last = kNoBag;
    int listed, end;  // bags in the list; lookup behind the last one, from the window's start
    bool open;        // ... which goes on behind the window
#pragma unroll 1
    while (true) {
      listed = 0;
      end = -1;
      const char* const seg0 = segs + ((unsigned)from + wl) * spitch;
      const char* const id0 = reinterpret_cast<const char*>(T.ids) + (unsigned long long)((unsigned)from + wl) * (p.id_kind == 0 ? 4u : 8u);
#pragma unroll 1
      for (int t0 = 0; t0 < window; t0 += 32 * TILES) {
        unsigned long long seg[TILES], id[TILES];
#pragma unroll
        for (int k = 0; k < TILES; ++k) seg[k] = id[k] = ~0ull;
        // Ids and outputs pass through once: they leave L2 to the table rows (evict-first).
#pragma unroll
        for (int k = 0; k < TILES; ++k)
          if (t0 + 32 * k + wl < window)
            seg[k] = __ldcs(reinterpret_cast<const unsigned long long*>(seg0 + (unsigned)(t0 + 32 * k) * spitch));
        if (p.id_kind == 0) {
#pragma unroll
          for (int k = 0; k < TILES; ++k)
            if (t0 + 32 * k + wl < window) id[k] = (unsigned long long)(long long)__ldcs(reinterpret_cast<const int*>(id0) + (t0 + 32 * k));
        } else {
#pragma unroll
          for (int k = 0; k < TILES; ++k)
            if (t0 + 32 * k + wl < window) id[k] = __ldcs(reinterpret_cast<const unsigned long long*>(id0) + (t0 + 32 * k));
        }
        if (p.id_kind == 2) {
          if (T.num_buckets < (1ull << 31)) {
#pragma unroll
            for (int k = 0; k < TILES; ++k) id[k] = fast_mod_u64_small(id[k], (unsigned)T.num_buckets, T.magic);
          } else {
#pragma unroll
            for (int k = 0; k < TILES; ++k) id[k] = fast_mod_u64(id[k], T.num_buckets, T.magic);
          }
        }
#pragma unroll
        for (int k = 0; k < TILES; ++k) {
          if (t0 + 32 * k >= window) break;
          const int j = t0 + 32 * k + wl;
          const bool seg_ok = seg[k] < (unsigned long long)batch, row_ok = id[k] < (unsigned long long)T.rows;
          const int key = seg_ok ? (int)seg[k] : kNoBag;
          rows[j] = row_ok ? tab + (unsigned long long)(unsigned)id[k] * pitch : nothing;
          int pk = __shfl_up_sync(kAll, key, 1);
          if (wl == 0) pk = before;
          before = __shfl_sync(kAll, key, 31);
          const bool in = j < window, starts = in && key != pk;
          const unsigned all = __ballot_sync(kAll, starts);
          const int rest = mine - (t0 + 32 * k);  // lookups of the chunk from this tile on
          const unsigned mask = rest >= 32 ? all : rest <= 0 ? 0u : all & ((1u << rest) - 1u);
          const bool lists = (mask >> wl) & 1u;
          if (lists) {
            BagEntry* e = bags + listed + __popc(mask & ((1u << wl) - 1u));
            e->bag = key;
            e->first = (unsigned short)j;
            e[-1].end = (unsigned short)j;
          }
          listed += __popc(mask);
          if (all != mask && end < 0) end = t0 + 32 * k + __ffs(all ^ mask) - 1;
          // Rare: ids out of range, and lookups whose segment id is not the previous one or its successor:
          // unsorted segment ids, or empty bags in between.
          if (__any_sync(kAll, in && (!seg_ok || !row_ok || (starts && key != pk + 1)))) {
            if (in && !seg_ok) atomicOr(&hdr->err_bits, kErrSegment);
            if (in && !row_ok) atomicOr(&hdr->err_bits, kErrRow);
            const bool odd = lists && key != pk + 1 && key >= 0 && pk >= -1;
            unsigned gaps = __ballot_sync(kAll, odd);
            if (__any_sync(kAll, odd && key < pk)) {  // unsorted: its output is cleared and redone anyway
              if (wl == 0) mark_unsorted(hdr, t);
              gaps = 0;
            }
            while (gaps) {
              const int src = __ffs(gaps) - 1;
              gaps &= gaps - 1;
              zero_fill(__shfl_sync(kAll, pk, src) + 1, __shfl_sync(kAll, key, src));
            }
          }
        }
      }
      open = end < 0 && from + window < n;  // the last bag goes on behind the window
      if (end < 0) end = window;
      if (holder >= 0) {
        listed = 1;
        if (wl == 0) {
          bags[0].bag = last;
          bags[0].first = 0;
        }
      }
      if (listed == 0) break;  // the bag that crosses the chunk began before it
      if (wl == 0) bags[listed - 1].end = (unsigned short)end;
      if (wl < Q) rows[window + wl] = nothing;  // a round may read past the last lookup
      __syncwarp();

      // b: this group's bag in the list, e; next: the first one nobody has taken; r: where the rows of its
      // next lookups are, `left` of them
      int b = holder < 0 ? group : (group == holder ? 0 : 1);
      int next = holder < 0 ? GROUPS : 1;
      int left = 0;
      BagEntry e{kNoBag, 0, 0};
      const unsigned long long* r = rows;
      bool holds = false;
      if (b < listed) {
        e = bags[b];
        r = rows + e.first;
        left = e.end - e.first;
      }
#pragma unroll 1
      while (__any_sync(kAll, b < listed)) {
        Vec v[Q][VPL];
        unsigned long long row[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) row[q] = r[q];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          if (q >= left) row[q] = nothing;
#pragma unroll
          for (int w = 0; w < VPL; ++w) v[q][w].load(reinterpret_cast<const char*>(row[q]) + col[w]);
        }
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
          for (int w = 0; w < VPL; ++w) acc[w].add(v[q][w]);
        left -= Q;
        r += left > 0 ? Q : 0;
        const bool done = left <= 0 && b < listed;
        const unsigned mask = __ballot_sync(kAll, done);
        if (done) {
          holds = open && b == listed - 1;  // its bag stays in the accumulator
          if (!holds) {
            if (e.bag >= 0) {
              char* o = outp + (unsigned)e.bag * opitch;
              const bool mean = p.combiner == 1;
              const float inv = mean ? __fdiv_rn(1.0f, (float)(counted + (int)e.end - (int)e.first)) : 1.0f;
#pragma unroll
              for (int w = 0; w < VPL; ++w) store(o, acc[w], w, mean, inv);
            }
#pragma unroll
            for (int w = 0; w < VPL; ++w) acc[w].zero();
          }
          b = next + __popc(mask & ((1u << (group * LANES)) - 1u)) / LANES;
          if (b < listed) {
            e = bags[b];
            r = rows + e.first;
            left = e.end - e.first;
          }
        }
        next += __popc(mask) / LANES;
      }
      last = bags[listed - 1].bag;
      if (!open) break;
      counted += end - (int)bags[listed - 1].first;
      holder = (__ffs(__ballot_sync(kAll, holds)) - 1) / LANES;
      before = last;
      from += window;
      window = min(32 * TILES, n - from);
      mine = 0;
      __syncwarp();
    }
    // the table's last lookup: bags after its bag are empty
    if (listed > 0 && last >= 0 && from + end == n) zero_fill(last + 1, batch);
    __syncwarp();
    gc_next = __shfl_sync(kAll, gc_next, 0);
  }
  pdl_trigger();
}

// The kernels for tables marked unsorted.  They follow every call, sorted or not (the host does
// not know), so their cost on sorted tables is what matters: one grid over all marked tables
// that leaves after one load, launched while the kernel before it drains (pdl_wait holds until
// that kernel has finished and its writes are visible).

// Zeroes the output and the per-bag counters for the atomic route.
__global__ void __launch_bounds__(256)
bag_stream_reset_kernel(BagParams p, BagHeader* hdr, int* offsets) {
  pdl_wait();
  pdl_trigger();
  if (!*(volatile int*)&hdr->any_unsorted) return;
  const long long stride = (long long)gridDim.x * blockDim.x;
  const long long total = p.batch * p.dim;
  for (int t = 0; t < p.num_tables; ++t) {
    if (!hdr->unsorted[t]) continue;
    const BagTableDev& T = p.t[t];
    int* counts = offsets + (long long)t * (p.batch + 1);
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride) {
      const long long s = e / p.dim, c = e - s * p.dim;
      T.out[s * p.out_stride + c] = 0.f;
      if (c == 0) counts[s] = 0;
    }
  }
}

// Atomic scatter (sum order not defined; within 1e-5 rel).
__global__ void __launch_bounds__(256)
bag_scatter_kernel(BagParams p, BagHeader* hdr, int* offsets) {
  pdl_wait();
  pdl_trigger();
  if (!*(volatile int*)&hdr->any_unsorted) return;
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (int t = 0; t < p.num_tables; ++t) {
    if (!hdr->unsorted[t]) continue;
    const BagTableDev& T = p.t[t];
    int* counts = offsets + (long long)t * (p.batch + 1);
    for (long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < T.nnz;
         i += warps) {
      long long seg = T.seg[i * p.ncols + p.col];
      long long r = shard_row(load_row_id(T.ids, p.id_kind, i, T.num_buckets, T.magic), p.shard_count,
                              p.shard_rank);
      if (seg < 0 || seg >= p.batch) continue;  // flagged by the prepass
      if (lane == 0) atomicAdd(&counts[seg], 1);  // bag length counts every rank's lookups
      if (r == kNotMine) continue;
      if (r < 0 || r >= T.rows) {
        if (lane == 0) atomicOr(&hdr->err_bits, kErrRow);
        continue;
      }
      float* orow = T.out + seg * p.out_stride;
      for (long long c = lane; c < p.dim; c += 32) atomicAdd(orow + c, __ldg(T.table + r * p.dim + c));
    }
  }
}

__global__ void __launch_bounds__(256)
bag_scatter_mean_kernel(BagParams p, BagHeader* hdr, int* offsets) {
  pdl_wait();
  if (!*(volatile int*)&hdr->any_unsorted) return;
  const long long total = p.batch * p.dim;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (int t = 0; t < p.num_tables; ++t) {
    if (!hdr->unsorted[t]) continue;
    const BagTableDev& T = p.t[t];
    const int* counts = offsets + (long long)t * (p.batch + 1);
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride) {
      const long long s = e / p.dim, c = e - s * p.dim;
      const int n = counts[s];
      if (n > 0) {
        float* q = T.out + s * p.out_stride + c;
        *q = __fmul_rn(*q, __fdiv_rn(1.0f, (float)n));
      }
    }
  }
}

// ---- max segment id (+1 = batch of the reference) ------------------------------
__global__ void seg_max_kernel(const int64_t* seg, long long nnz, long long ncols, int col,
                               long long* out_max) {
  long long m = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += stride) {
    long long v = seg[i * ncols + col];
    m = v > m ? v : m;
  }
  for (int o = 16; o > 0; o >>= 1) {
    long long w = __shfl_xor_sync(0xffffffffu, m, o);
    m = w > m ? w : m;
  }
  if ((threadIdx.x & 31) == 0 && m > 0) atomicMax(out_max, m);
}

// What the segment-reduce operator needs on the host before it can allocate its output, in the one
// pass that has to be waited for: the largest segment id, whether the ids are sorted (then the
// atomic route need not follow) and whether every id and row is in range (then nothing has to be
// read back afterwards).  Posted to the host by the block that ends last.
constexpr int kScanUnsorted = 4;  // beside kErrRow and kErrSegment
struct SegScan {
  long long max_seg;
  int flags;
  int blocks_done;
};
// Up to kSegScanOne lookups go to one block, which needs no cleared SegScan and clears the bag header on the
// way: 2,700 lookups without the memset before it and the copy behind it (0.8 and 2.4 us and 6 us of gaps).
constexpr int kSegScanThreads = 512;
constexpr long long kSegScanOne = 8 * kSegScanThreads;
__global__ void __launch_bounds__(kSegScanThreads)
seg_scan_kernel(const int64_t* seg, const void* ids, int id_kind, long long nnz, long long ncols, int col,
                long long rows, BagHeader* hdr, SegScan* out, PostBox box) {
  constexpr int WARPS = kSegScanThreads / 32;
  __shared__ long long s_max[WARPS];
  __shared__ int s_flags[WARPS];
  long long m = 0;
  int flags = 0;
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < nnz; i += stride) {
    const long long v = seg[i * ncols + col];
    const long long before = i > 0 ? seg[(i - 1) * ncols + col] : -1;
    const long long r = load_row_id(ids, id_kind, i, 1, 0);
    if (v < 0) flags |= kErrSegment;
    else if (v < before) flags |= kScanUnsorted;
    if (r < 0 || r >= rows) flags |= kErrRow;
    m = v > m ? v : m;
  }
  if (gridDim.x == 1)
    for (int e = threadIdx.x; e < (int)(kHeaderBytes / sizeof(int)); e += kSegScanThreads) reinterpret_cast<int*>(hdr)[e] = 0;
  for (int o = 16; o > 0; o >>= 1) {
    const long long w = __shfl_xor_sync(0xffffffffu, m, o);
    m = w > m ? w : m;
  }
  flags = (int)__reduce_or_sync(0xffffffffu, (unsigned)flags);
  if ((threadIdx.x & 31) == 0) {
    s_flags[threadIdx.x >> 5] = flags;
    s_max[threadIdx.x >> 5] = m;
  }
  __syncthreads();
  if (threadIdx.x != 0) return;
  for (int w = 1; w < WARPS; ++w) {
    m = s_max[w] > m ? s_max[w] : m;
    flags |= s_flags[w];
  }
  if (gridDim.x > 1) {
    if (flags) atomicOr(&out->flags, flags);
    if (m > 0) atomicMax(&out->max_seg, m);
    __threadfence();
    if (atomicAdd(&out->blocks_done, 1) != (int)gridDim.x - 1) return;
    __threadfence();
    m = *(volatile long long*)&out->max_seg;
    flags = *(volatile int*)&out->flags;
  } else {
    out->max_seg = m;
    out->flags = flags;
  }
  if (box.words) post_result(box, flags, m);
}

__global__ void store_i32_kernel(int* p, int v) { *p = v; }

// ---- single-row gathers ---------------------------------------------------------
// out[i,:] = skip(i) ? 0 : table[row(i),:]; one warp per output row.
// mode 0: KPFusedEmbeddingWithHashBucket (row = fp % num_buckets, empty -> zeros)
// mode 1: bounded variant (row outside [0, rows) -> zeros)
// mode 2: sparse_embedding2 (valid = lo <= id < hi; out = m * table[valid ? id : dflt])
struct GatherParams {
  const float* table;
  const void* ids;
  const unsigned char* empty;
  float* out;
  long long n, rows, dim;
  unsigned long long num_buckets;
  long long lo, hi, dflt;
  int mode;
  int ids64;
};

__global__ void __launch_bounds__(256) row_gather_kernel(GatherParams g, int* err) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  const bool vec = (g.dim % 4 == 0) && ((((uintptr_t)g.table) | ((uintptr_t)g.out)) % 16 == 0);
  for (long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < g.n;
       i += warps) {
    long long row = -1;
    float scale = 1.0f;
    bool use_scale = false;
    if (g.mode == 2) {
      long long id = g.ids64 ? ((const long long*)g.ids)[i] : (long long)((const int*)g.ids)[i];
      const bool valid = id >= g.lo && id < g.hi;
      row = valid ? id : g.dflt;
      scale = valid ? 1.0f : 0.0f;
      use_scale = true;
      if (row < 0 || row >= g.rows) {
        if (lane == 0) atomicOr(err, kErrRow);
        row = -1;
      }
    } else if (!(g.empty && g.empty[i])) {
      unsigned long long b = ((const unsigned long long*)g.ids)[i] % g.num_buckets;
      row = (long long)b;
      if (row < 0 || row >= g.rows) {
        if (g.mode == 0 && lane == 0) atomicOr(err, kErrRow);
        row = -1;
      }
    }
    float* o = g.out + i * g.dim;
    const float* src = row >= 0 ? g.table + row * g.dim : nullptr;
    if (vec) {
      for (long long c = lane * 4; c < g.dim; c += 128) {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (src) v = ldg4(src + c);
        if (use_scale) {
          v.x = __fmul_rn(scale, v.x);
          v.y = __fmul_rn(scale, v.y);
          v.z = __fmul_rn(scale, v.z);
          v.w = __fmul_rn(scale, v.w);
        }
        *reinterpret_cast<float4*>(o + c) = v;
      }
    } else {
      for (long long c = lane; c < g.dim; c += 32) {
        float v = src ? __ldg(src + c) : 0.f;
        o[c] = use_scale ? __fmul_rn(scale, v) : v;
      }
    }
  }
}

// KPFusedSparseDynamicStitch: table = id % N, row = id / N.
struct StitchParams {
  const float* const* tables;  // device array [N]
  const long long* table_rows; // device array [N]
  const long long* x;
  float* out;
  long long n, dim;
  int num_partitions;
};

__global__ void __launch_bounds__(256) stitch_kernel(StitchParams g, int* err) {
  const int lane = threadIdx.x & 31;
  const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long i = (long long)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); i < g.n;
       i += warps) {
    const long long id = g.x[i];
    const long long t = id % g.num_partitions;
    const long long r = id / g.num_partitions;
    float* o = g.out + i * g.dim;
    if (id < 0 || !(r < g.table_rows[t])) {
      if (lane == 0) atomicOr(err, kErrRow);
      for (long long c = lane; c < g.dim; c += 32) o[c] = 0.f;
      continue;
    }
    const float* src = g.tables[t] + r * g.dim;
    const bool vec = (g.dim % 4 == 0) && ((((uintptr_t)src) | ((uintptr_t)o)) % 16 == 0);
    if (vec) {
      for (long long c = lane * 4; c < g.dim; c += 128)
        *reinterpret_cast<float4*>(o + c) = ldg4(src + c);
    } else {
      for (long long c = lane; c < g.dim; c += 32) o[c] = __ldg(src + c);
    }
  }
}

// ---- first-appearance unique (KPFusedGather, segment order of the Nonzero op) ---
// Open-addressing table of int64 keys; the empty marker is INT64_MIN, a key equal
// to the marker lives in the extra last slot.  first[slot] = smallest position
// that holds the key.
constexpr long long kEmptyKey = (long long)0x8000000000000000ull;

__device__ __forceinline__ unsigned long long mix64(unsigned long long x) {
  x ^= x >> 33;
  x *= 0xff51afd7ed558ccdull;
  x ^= x >> 33;
  x *= 0xc4ceb9fe1a85ec53ull;
  x ^= x >> 33;
  return x;
}

__device__ __forceinline__ long long find_or_insert(long long* keys, long long cap, long long key) {
  if (key == kEmptyKey) return cap;  // dedicated slot
  unsigned long long h = mix64((unsigned long long)key) & (unsigned long long)(cap - 1);
  for (long long probe = 0; probe < cap; ++probe) {
    // A popular key is nearly always there already: a load (not an atomic, which the thousands of
    // lookups of one key would queue up for) settles it.  Keys never change once set.  300 K keys,
    // 5 % of them one key: 27 us with an unconditional exchange and minimum, 17 us.
    long long old = __ldcg(keys + h);
    if (old == key) return (long long)h;
    if (old == kEmptyKey) old = atomicCAS((unsigned long long*)&keys[h], (unsigned long long)kEmptyKey,
                              (unsigned long long)key);
    if (old == kEmptyKey || old == key) return (long long)h;
    h = (h + 1) & (unsigned long long)(cap - 1);
  }
  return -1;  // table full: cannot happen with cap >= 2 * n
}

// (The kernels from here to unique_inverse_kernel start while the one before them drains: 300 K keys, the whole call,
// 90 us -> 88 us.)
__global__ void unique_init_kernel(long long* keys, int* first, long long cap, int* total_err) {
  pdl_trigger();
  const long long stride = (long long)gridDim.x * blockDim.x;
  if (blockIdx.x == 0 && threadIdx.x < 3) total_err[threadIdx.x] = 0;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i <= cap; i += stride) {
    keys[i] = kEmptyKey;
    first[i] = 0x7fffffff;
  }
}

// `rows` >= 0: keys outside [0, rows) raise kErrRow.
__global__ void unique_insert_kernel(const int64_t* src, long long n, long long ncols, int col,
                                     long long* keys, int* first, long long cap, int* slot_of, long long rows,
                                     int* err) {
  pdl_trigger();
  pdl_wait();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const long long key = src[i * ncols + col];
    if (rows >= 0 && (key < 0 || key >= rows)) atomicOr(err, kErrRow);
    const long long slot = find_or_insert(keys, cap, key);
    slot_of[i] = (int)slot;
    if (slot >= 0 && __ldcg(first + slot) > (int)i) atomicMin(&first[slot], (int)i);  // it only falls
  }
}

// Position i holds the first appearance of its key.
__device__ __forceinline__ int is_first(const int* slot_of, const int* first, long long i, long long n) {
  if (i >= n) return 0;
  const int slot = slot_of[i];
  return slot >= 0 && __ldcg(first + slot) == (int)i ? 1 : 0;
}
// First appearances per tile of kScanTile positions.  The block that ends last adds the tiles up and posts
// the number of keys: the caller allocates its outputs while the kernels below still run (300 K keys: the
// device waited 23 us for a copy, a synchronize and the allocations before).
// total_err: {number of keys, error bits, blocks that are done}.
__global__ void __launch_bounds__(kScanThreads)
unique_count_kernel(const int* slot_of, const int* first, long long n, int* tile_sums, int* total_err, PostBox box) {
  __shared__ bool s_last;
  pdl_trigger();
  pdl_wait();
  const long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) s += is_first(slot_of, first, base + k, n);
  int total;
  block_exclusive_scan(s, &total);
  if (threadIdx.x == 0) {
    tile_sums[blockIdx.x] = total;
    __threadfence();
    s_last = atomicAdd(total_err + 2, 1) == (int)gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!s_last) return;
  s = 0;
  for (int t = threadIdx.x; t < (int)gridDim.x; t += kScanThreads) s += __ldcg(tile_sums + t);
  block_exclusive_scan(s, &total);
  if (threadIdx.x == 0) {
    total_err[0] = total;
    if (box.words) post_result(box, total_err[1], total);
  }
}
// Writes unique keys in first-appearance order and turns first[slot] into the key's rank.  (The
// rank is at most the first position, so no later position of the key takes it for its own.)  A
// block adds up the tiles before it by itself unless `scanned` says that tile_sums already holds
// their running sums.
__global__ void __launch_bounds__(kScanThreads)
unique_emit_kernel(const int64_t* src, long long n, long long ncols, int col, const int* slot_of, int* first,
                   const int* tile_sums, int scanned, long long* out_unique) {
  pdl_trigger();
  pdl_wait();
  int before = 0;
  if (scanned) {
    before = tile_sums[blockIdx.x];
  } else {
    int part = 0;
    for (int t = threadIdx.x; t < (int)blockIdx.x; t += kScanThreads) part += tile_sums[t];
    block_exclusive_scan(part, &before);
  }
  const long long base = (long long)blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int flag[kScanItems], s = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) s += flag[k] = is_first(slot_of, first, base + k, n);
  int rank = block_exclusive_scan(s, nullptr) + before;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    if (!flag[k]) continue;
    const long long i = base + k;
    if (out_unique) out_unique[rank] = src[i * ncols + col];
    first[slot_of[i]] = rank++;
  }
}

// inverse[i] = rank of key i; optionally as int64 (segment column for the bag kernels).
__global__ void unique_inverse_kernel(const int* slot_of, const int* first, long long n,
                                      int* inverse32, long long* inverse64) {
  pdl_wait();
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
    const int r = slot_of[i] >= 0 ? first[slot_of[i]] : 0;
    if (inverse32) inverse32[i] = r;
    if (inverse64) inverse64[i] = r;
  }
}

// out[u,:] = table[unique[u],:] (keys outside the table, reported before, are left out); the keys
// themselves go to out_keys on the way.  LANES lanes take four rows at a time, so that four row
// loads are out before the first store: 150 K rows of dim 64 in 17 us, 30 us with a warp and one
// load per row.
template <int LANES>
__global__ void __launch_bounds__(256)
unique_rows_kernel(const float* __restrict__ table, long long rows, int dim, int vec,
                   const long long* __restrict__ unique, long long nu, float* __restrict__ out,
                   long long* __restrict__ out_keys) {
  constexpr int R = 4;
  const int lane = threadIdx.x % LANES;
  const long long groups = (long long)gridDim.x * (256 / LANES);
  for (long long u0 = ((long long)blockIdx.x * (256 / LANES) + threadIdx.x / LANES) * R; u0 < nu; u0 += groups * R) {
    long long r[R];
#pragma unroll
    for (int k = 0; k < R; ++k) {
      r[k] = u0 + k < nu ? unique[u0 + k] : -1;
      if (out_keys && lane == k % LANES && u0 + k < nu) out_keys[u0 + k] = r[k];
      if (r[k] >= rows) r[k] = -1;
    }
    if (vec) {
      for (int c = lane * 4; c < dim; c += LANES * 4) {
        float4 v[R];
#pragma unroll
        for (int k = 0; k < R; ++k)
          if (r[k] >= 0) v[k] = ldg4(table + r[k] * dim + c);
#pragma unroll
        for (int k = 0; k < R; ++k)
          if (r[k] >= 0) __stcs(reinterpret_cast<float4*>(out + (u0 + k) * dim + c), v[k]);
      }
    } else {
      for (int c = lane; c < dim; c += LANES) {
        float v[R];
#pragma unroll
        for (int k = 0; k < R; ++k)
          if (r[k] >= 0) v[k] = __ldg(table + r[k] * dim + c);
#pragma unroll
        for (int k = 0; k < R; ++k)
          if (r[k] >= 0) out[(u0 + k) * dim + c] = v[k];
      }
    }
  }
}

// ---- non-zero compaction of the Nonzero op --------------------------------------
// dense f32[nseg, dim] (already scaled for mean); flag = value != 0.
__global__ void nonzero_flag_kernel(const float* dense, long long total, int* flag) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride)
    flag[e] = dense[e] != 0.0f ? 1 : 0;
}

__global__ void nonzero_emit_kernel(const float* dense, long long total, long long dim, int rank,
                                    const long long* seg_order, const int* flag, const int* pos,
                                    int* out_indices, float* out_values) {
  const long long stride = (long long)gridDim.x * blockDim.x;
  for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < total; e += stride) {
    if (!flag[e]) continue;
    const long long u = e / dim, d = e - u * dim;
    const int o = pos[e];
    out_indices[(long long)o * rank] = (int)seg_order[u];
    if (rank == 2) out_indices[(long long)o * 2 + 1] = (int)d;
    out_values[o] = dense[e];
  }
}

}  // namespace emb
}  // namespace annc
