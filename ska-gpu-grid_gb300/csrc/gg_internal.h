// Host-side launcher interfaces between the C ABI (gg_api.cu) and the
// kernel translation units.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

#include "gg_types.h"

namespace gg {

// process-wide count of kernel launches made by the library
void count_launch(int n = 1);
// records msg as the calling thread's gg_last_error() and returns code
int set_error(int code, const char *msg);

// One job of a binning pass.  Visibilities of all jobs of a batch live in one
// global index space: job j owns global indices [vis_base, vis_base+npts) and
// global uv tiles [tile_base, tile_base+ntiles).
struct BinJob {
  const void *uv;
  const void *vals;
  const int *gcf_index;  // per-visibility table index, or null
  int64_t vis_base;
  int64_t npts;
  int tile_base, ntiles;  // ntiles = ntx * ntx * n_gcf bins
  int N, S, G, log2G, log2T, ntx, P;
  int uv_f64;
  int n_gcf;
  int off;  // cells by which the uv tiles start before the grid (0: clamped)
  int rec;  // format of its sorted records, kRec*
};

// Sorted records: packed (main*G+sub) pairs (gather, gg_bin), window_record,
// regtile_record or regtile_table_record.
enum { kRecPacked = 0, kRecWindow = 1, kRecRegtile = 2, kRecTables = 3 };

struct BinBuffers {
  const BinJob *jobs;      // device [njobs]
  BinJob one;              // the job, if it is the only one
  const int64_t *vis_base; // device [njobs+1]
  const int *tile_base;    // device [njobs+1]
  int njobs;
  int64_t total_vis;       // sum of npts
  int total_tiles;         // sum of ntiles
  int vals_bytes;          // 8 (complex64) or 16 (complex128)
  int P;                   // polarisations (uniform over the batch)
  int *rank;               // [total_vis] rank in the tile (-1: dropped)
  int *counts;             // [total_tiles+1], zeroed by the caller: histogram,
                           // then block-local offsets
  int *scan_tmp;           // scan_tmp_ints; the first word zeroed by the caller
  int *block_off;          // scan_tmp + kScanHead: offsets of the scan's blocks
  int *bookmarks;          // [total_tiles+2]: exclusive offsets; the word at
                           // total_tiles+1 (zeroed by the caller) is set when
                           // input declared sorted is not (records left
                           // unwritten)
  int2 *sorted_idx;        // [total_vis + pad]
  void *sorted_vals;       // [P][vstride]
  int64_t vstride;
  int *order;              // [total_vis] or null
  int *flags;
  int input_sorted;
  int *kept_pos;           // [total_vis+1] (input_sorted only)
  // one value per visibility, complex64: {record, value} in sorted_idx
  int aos;
};

// Sorted record of the moving-window kernel: both main cells in one word
// (offset by 64 so that clamped mains stay positive; 16 bits each hold
// img_dim up to 32768 plus the support) and the sub-kernel index.
constexpr int kWinMainBias = 64;
__host__ __device__ inline int2 window_record(int mx, int sx, int my, int sy, int G) {
  return make_int2((int)(((unsigned)(my + kWinMainBias) << 16) | (unsigned)(mx + kWinMainBias)),
                   sy * G + sx);
}

// Sorted record of the register-tile kernel, for a main cell at (fx, fy) in
// its 8-cell tile: the byte offset of the footprint's first tap, seen from
// the sub-grid's first cell, in the table in shared memory, and the cell (fy
// alone for support 8, fy | fx << 8 for 16).  Table rows are regtile_row bytes
// long, their first tap at byte regtile_pad.
__host__ __device__ constexpr int regtile_row(int S) { return S == 8 ? 80 : 96; }
__host__ __device__ constexpr int regtile_pad(int S) { return S == 8 ? 32 : 0; }
__host__ __device__ inline int2 regtile_record(int fx, int sx, int fy, int sy, int G, int S) {
  const int row = regtile_row(S);
  return make_int2((sy * G + sx) * S * row + regtile_pad(S) - 4 * fx - row * fy,
                   S == 8 ? fy : fy | fx << 8);
}

// The same for tables in global memory ([G*G][S][S] complex entries).
__host__ __device__ inline int2 regtile_table_record(int fx, int sx, int fy, int sy, int G, int S) {
  return make_int2((((sy * G + sx) * S - fy) * S - fx) * 8, fy | fx << 8);
}

// index step only (vis2ints)
cudaError_t launch_vis2ints(int uv_f64, const void *uv, int64_t npts, int G,
                            int2 *packed, int *flags, cudaStream_t s);
// words before the block offsets in a scan's scratch
constexpr int kScanHead = 8;
// ints of scratch for a scan of n entries
size_t scan_tmp_ints(int64_t n);

// Work items for the moving-window kernel: every non-empty tile of job j
// (global tiles tile_base..) is cut into slices of at most `chunk` sorted
// visibilities.  Items of jobs of S-class c go to items + c*class_cap,
// counted in counters[c].
// records per work item of each support class (index: class of the job)
constexpr int kMaxClasses = 4;
struct ClassChunks {
  int c[kMaxClasses];
};
// Merge slots per support class (cap 0 or base null: none).  A tile of a job
// with a complex64 grid that is cut into more than one item gets slot
// heavy_counters[c]++ of its class: every one of its items carries the slot,
// and desc[slot] = {job, tile-local bin}.  A slot index beyond the class's
// cap (the host sizes cap so that this cannot happen) raises FLAG_BOUNDS and
// leaves the tile on the plain reduction.
struct ClassSlots {
  MergeSlots m[kMaxClasses];
};
struct ItemBuffers {
  WorkItem *items;         // null: no items
  const JobDesc *jobs;
  const int *job_class;
  int nclasses;
  ClassChunks chunks;
  int64_t class_cap;
  int *counters;           // [kMaxClasses], zeroed by the caller
  int *heavy_counters;     // [kMaxClasses], zeroed by the caller
  ClassSlots slots;
};
// count, scan, scatter; leaves bookmarks = exclusive offsets [total_tiles+1],
// and makes the work items when given
cudaError_t run_binning(const BinBuffers &b, const ItemBuffers *items, cudaStream_t s);
// Number of merge slots a class needs at most: tiles with more than `chunk`
// records, at most vis / (chunk + 1) of them.
inline int merge_slot_cap(int64_t vis, int chunk, int64_t tiles) {
  int64_t c = vis / ((int64_t)chunk + 1) + 1;
  if (c > tiles) c = tiles;
  return (int)c;
}
// Rounds every slot of the class once into its job's grid (after the
// class's window kernel): cell values that are nonzero are reduced into the
// output with the grid's layout, cells outside the grid skipped.
cudaError_t launch_merge_finalize(const MergeSlots &m, const int *heavy_counter,
                                  const JobDesc *jobs, int S, int T, int P, int sm_count,
                                  cudaStream_t s);
// ORs `bits` (1 << FLAG_*) into flags[FLAG_*] on the stream: the host-side
// injection behind gg_debug_inject_device_flags.
cudaError_t launch_inject_flags(int *flags, int bits, cudaStream_t s);
// Up to kMaxZero ranges of device memory (4-byte aligned) to clear.
constexpr int kMaxZero = 8;
struct ZeroRanges {
  void *p[kMaxZero];
  size_t bytes[kMaxZero];
  int n;
  void add(void *q, size_t b) {
    p[n] = q;
    bytes[n++] = b;
  }
};
// Copies `bytes` (a multiple of 16, dst 16-byte aligned; 0: none) from host
// memory to dst on the stream through kernel parameters, 16 KB per launch
// (nothing waits on a copy engine, and src may be rewritten once the call
// returns), and clears the ranges.
cudaError_t launch_setup(void *dst, const void *src, size_t bytes, const ZeroRanges &zero,
                         cudaStream_t s);
// clears the output grids of `njobs` jobs in `chunks` pieces of kZeroChunk
constexpr size_t kZeroChunk = 64 << 10;
cudaError_t launch_zero_jobs(const JobDesc *jobs, int njobs, int chunks, int sm_count,
                             cudaStream_t s);
// flags of a context (device int32[64], see gg_read_flags)
int *context_flags(gg_context *c);
// Makes the batched calls of a context use `flags` (device int32[64], the
// caller zeroes words 0..7) instead of its own flag words, until reset with
// null: the request server gives every batch in flight its own words, read
// back after the batch's output copies while the slot runs its next batch.
void context_set_batch_flags(gg_context *c, int *flags);
// consumes one pending injection of gg_debug_inject_device_flags: returns
// its bits (0: none pending)
int injected_device_flags();
// gg_read_flags without a context: flags of the last allocation-free call on
// the current device (gg_noalloc.cu); synchronises the stream
int noalloc_read_flags(void *stream, int32_t out[4]);

// ---- gridding launches ----------------------------------------------------
struct GridLaunch {
  const JobDesc *jobs;     // device [njobs]
  int njobs;
  int S;                   // support of every job in this launch
  int accum;               // GG_ACC_*
  int vals_f64;
  int gauss;
  int wphase;              // scatter: the reference's COMPUTE_GCF factor
  float sigma;             // GAUSS: uniform over the launch
  int G;                   // oversampling, uniform over the launch
  int tile;                // uv tile side, uniform over the launch
  int group_warps;         // moving window: warps per sub-grid (0: by support)
  int accumulate;          // gather: add into the grid instead of storing
  int P;
  int *flags;
  const int *holes;        // binned methods: bookmarks[total_tiles + 1]
  int sm_count;
  // scatter: global visibility space
  const int64_t *vis_base; // device [njobs+1]
  int64_t total_vis;
  // window: work queue
  const WorkItem *items;
  const int *nitems;
  int *item_next;
  int64_t max_items;
  MergeSlots merge;        // the class's FP64 merge slots (base null: none)
  // gather: global tiles of the jobs in this launch
  const int *tile_base;    // device [njobs+1]
  int total_tiles;
};

// Degridding (adjoint of the gridder): one launch per job
struct DegridLaunch {
  const void *grid;        // device: P planes of N*N complex (grid_f64: double)
  void *vals;              // device: npts*P complex out (vals_f64: double)
  const void *uv;          // device: npts (u,v) pairs (uv_f64: double)
  const void *gcf;         // device: n_gcf tables [G*G][S][S] of the values' type; null: Gaussian
  const int *gcf_index;    // device, optional: table of each visibility
  int64_t npts;
  int N, S, G, P, n_gcf;
  int uv_f64, grid_f64, vals_f64;
  int planar;              // grid layout: planar (1) or interleaved (0)
  int gauss;               // GCF computed on the fly (separable Gaussian)
  int compensated;         // FP32 values: two-sum (hi, lo) lane sums
  float sigma;
  int *flags;
  int sm_count;
};
cudaError_t launch_degrid(const DegridLaunch &d, cudaStream_t s);
// centred inverse 2-D FFT of P interleaved planes in place (cuFFT, loaded at
// first use); 0 on success, else a message in err.  Synchronises s.
int image_inverse_fft(void *grid, int64_t N, int P, bool f64, int sm_count, cudaStream_t s,
                      std::string &err);

// Register-tile moving window (gg_regtile.cu): FP32 values, support 8 or 16;
// one GCF table per launch (its copy fills the CTA's shared memory), or any
// number of them in global memory.
struct RegTileLaunch {
  const JobDesc *jobs;
  const WorkItem *items;
  const int *nitems;
  int *item_next;
  const int2 *idx;         // sorted records (regtile_record); {record, value}
                           // pairs of 16 bytes when vals is null
  const float2 *vals;      // sorted values, P planes of vstride
  int64_t vstride;
  int tables;              // tables read per item from the jobs' (gcf ignored)
  const unsigned *any_imag;  // whether any of those has imaginary parts
  const float2 *gcf;       // [G*G][S][S]
  int S, G, P;
  int compensated;
  int gauss;               // factors computed from sigma instead of gcf
  float sigma;
  int64_t max_items;       // upper bound of *nitems
  int sm_count;
  MergeSlots merge;        // base null: none
  int overlap;             // table fill while the binning ends (launch_overlapped)
};
cudaError_t launch_regtile(const RegTileLaunch &g, cudaStream_t s);
// JobDesc::gcf_info of the tables of a class's jobs (`tables` in all), and whether
// any of them has imaginary parts; both zeroed before.
cudaError_t launch_table_info(const JobDesc *jobs, int njobs, int S, int G, int64_t tables,
                              unsigned *any_imag, cudaStream_t s);
// Support 32 with the on-the-fly Gaussian, FP32 values (gg_septile.cu): one
// launch over the 16x16 output blocks of all jobs of a class.
struct SepTileLaunch {
  const JobDesc *jobs;     // the class's jobs, blk0 set
  int njobs;
  int total_blocks;
  int *next;               // zeroed counter of claimed blocks
  const int2 *idx;         // sorted records (window_record); {record, value}
                           // pairs of 16 bytes when vals is null
  const float2 *vals;      // sorted values, P planes of vstride
  int64_t vstride;
  int G, P;
  int compensated;
  int accumulate;          // add into the grid instead of storing
  float sigma;
  int sm_count;
  int64_t vis;             // visibilities of the class
  int overlap;             // follow each other by launch_overlapped
  // what sep_plan_kernel finds: a bit for every block that is summed as a whole,
  // and the dense ones {block, first unit, units, units done} with a merge slot
  // of P * 256 sums each; dense_count (slots taken << 32 | units) zeroed by the
  // caller
  unsigned *mask;
  int4 *dense;
  double2 *slots;
  unsigned long long *dense_count;
  int dense_cap;           // septile_dense_cap
  int dense_min, dense_unit, chunk;  // set by launch_septile
};
// More records than this make a block of support 32 dense: half a resident
// warp's share of all the visits that records pay to blocks (9 a record), so that
// no block keeps one warp much longer than the others; from 1024 records on.
inline int septile_dense_min(int64_t vis, int sm_count) {
  const int64_t half = 9 * vis / ((int64_t)sm_count * 32);
  return (int)(half > 1024 ? half : 1024);
}
// Dense blocks that there can be.
inline int64_t septile_dense_cap(int64_t vis, int64_t blocks, int sm_count) {
  const int64_t most = 9 * vis / septile_dense_min(vis, sm_count) + 1;
  return most < blocks ? most : blocks;
}
cudaError_t launch_septile(const SepTileLaunch &g, cudaStream_t s);
// Gather by output block (gg_gathertile.cu): FP32 values, support 8 or 16, one
// GCF table per launch.
struct GatherTileLaunch {
  const JobDesc *jobs;     // the class's jobs, blk0 set
  int njobs;
  int total_blocks;
  int *next;               // zeroed counter of claimed blocks
  const int2 *idx;         // sorted records (window_record); {record, value}
                           // pairs of 16 bytes when vals is null
  const float2 *vals;      // sorted values, P planes of vstride
  int64_t vstride;
  const float2 *gcf;       // [G*G][S][S]
  int S, G, P;
  int compensated;
  int accumulate;          // add each finished cell into the grid
  int gauss;               // factors computed from sigma instead of gcf
  float sigma;
  int sm_count;
  int overlap;             // table fill while the binning ends (launch_overlapped)
};
cudaError_t launch_gathertile(const GatherTileLaunch &g, cudaStream_t s);
size_t gathertile_smem_bytes(int S, int G);
inline int64_t septile_blocks(int64_t N) {
  const int64_t b = (N + kSepBlock - 1) / kSepBlock;
  return b * b;
}
size_t regtile_smem_bytes(int S, int G);

cudaError_t launch_scatter(const GridLaunch &g, cudaStream_t s);
cudaError_t launch_window(const GridLaunch &g, cudaStream_t s);
// one warp waiting on an mbarrier nobody completes (bounded-wait self-test)
cudaError_t launch_selftest_wait(int *flags, cudaStream_t s);
// test hook: the next n device allocations of the library fail (NOMEM);
// returns true (and consumes one) when the current allocation must fail
bool injected_alloc_failure();
// Row-doubled copy of ntab consecutive [G*G][S][S] GCF tables for the
// moving-window kernel: dst[s][b][a] = src[s][b mod S][a] for b < 2S, s over
// all ntab*G*G sub-kernels (elem_bytes 8 or 16).  With dst_real (complex64
// tables only) the real parts are written there too, and *has_imag (zeroed
// by the caller) is set when any imaginary part is nonzero.
cudaError_t launch_gcf_double_rows(const void *src, void *dst, int S, int G, int ntab,
                                   int elem_bytes, cudaStream_t s,
                                   float *dst_real = nullptr, int *has_imag = nullptr);
inline size_t gcf_double_rows_bytes(int S, int G, int elem_bytes) {
  return (size_t)elem_bytes * G * G * 2 * S * S;
}
cudaError_t launch_gather(const GridLaunch &g, cudaStream_t s);
// compensated scatter with complex64 output: out = fl(hi + lo)
cudaError_t launch_comp_finalize(float *out, const float *lo, int64_t n,
                                 cudaStream_t s);
// substitute inputs of the DEBUG1 footprint mode: vals[n*P+p] = (1, n),
// gcf = (1, 0) everywhere
cudaError_t launch_count_inputs(void *vals, int vals_f64, int64_t npts, int P,
                                void *gcf, int64_t gcf_elems, cudaStream_t s);
// smem bytes the window kernel needs (for occupancy sizing)
size_t window_smem_bytes(int S, int accum, int vals_f64, int T, int group_warps, int gauss);

}  // namespace gg
