// Index step and uv-tile binning on the device.
//
// Replaces, for the binned methods, the reference's host-side qsort by uv tile
// (comp_grid, grid.cu:256-276, dispatch grid.cu:467-475), vis2ints
// (grid_gpu.cu:352-365) and set_bookmarks (grid_gpu.cu:366-390):
//
//   bin_count    index step per visibility (bit-exact with grid.cu:159-163),
//                global uv-tile key, tile histogram, rank in the tile
//   scan         exclusive prefix sum of the histogram
//   bin_finish   places every kept visibility's record and values at its
//                sorted position, so the gridding kernels stream each tile
//                contiguously; writes the bookmarks; makes the work items
//
// Four launches with the set-up; they had been up to ten, a quarter of the time
// of a 10 k visibility call.
//
// All kernels work on a batch of jobs sharing one global visibility index
// space and one global tile space; a single job is a batch of one.
#include <algorithm>
#include <climits>
#include <cstring>

#include "gg_kernels.cuh"

namespace gg {

__device__ __forceinline__ int find_job64(const int64_t *base, int njobs,
                                          int64_t g) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}
__device__ __forceinline__ int find_job32(const int *base, int njobs, int g) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (base[mid] <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// Contiguous slice [w0, w1) of the visibilities for this warp (multiples of
// 32 apart), walked 32 at a time: the job of the slice's first visibility is
// found once, where a grid-stride walk would search the job table (dependent
// loads) on every step.
struct WarpSlice {
  int64_t w0, w1;
  __device__ WarpSlice(int64_t total) : WarpSlice(total, blockIdx.x, gridDim.x) {}
  __device__ WarpSlice(int64_t total, int64_t block, int64_t nblocks) {
    const int64_t nwarps = nblocks * (blockDim.x >> 5);
    const int64_t wid = block * (blockDim.x >> 5) + (threadIdx.x >> 5);
    const int64_t per = ((total + nwarps - 1) / nwarps + 31) & ~(int64_t)31;
    w0 = min(total, wid * per);
    w1 = min(total, w0 + per);
  }
};
// What a binning pass is compiled for: one job, described by the kernel's
// parameters, with float or double coordinates, or any jobs.
enum { kBinMany = 0, kBinOneF32 = 1, kBinOneF64 = 2 };

// f(job, s, e) for the visibilities [s, e) of each job in the slice: what a job
// has in common is loaded once, not for every visibility
template <int KIND, class F>
__device__ __forceinline__ void for_jobs(const BinBuffers &b, const WarpSlice &ws, F f) {
  if (ws.w0 >= ws.w1) return;
  if constexpr (KIND != kBinMany) {
    f(b.one, ws.w0, ws.w1);
    return;
  }
  int j = find_job64(b.vis_base, b.njobs, ws.w0);
  for (int64_t s = ws.w0; s < ws.w1; ++j) {
    const int64_t e = min(ws.w1, b.vis_base[j + 1]);
    if (e <= s) continue;  // an empty job
    const BinJob J = b.jobs[j];
    f(J, s, e);
    s = e;
  }
}

// entries of a scan block, and of one of its threads
constexpr int kScanPer = 8, kScanBlock = 2048;

// index step of visibility n of a uv array of either precision
__device__ __forceinline__ bool uv_index(const void *uv, int uv_f64, int64_t n,
                                         int G, int &mx, int &sx, int &my,
                                         int &sy) {
  if (uv_f64) {
    double2 c = __ldg((const double2 *)uv + n);
    bool a = index_step(c.x, G, mx, sx);
    bool b = index_step(c.y, G, my, sy);
    return a && b;
  }
  float2 c = __ldg((const float2 *)uv + n);
  bool a = index_step(c.x, G, mx, sx);
  bool b = index_step(c.y, G, my, sy);
  return a && b;
}

__global__ void __launch_bounds__(256)
    vis2ints_kernel(int uv_f64, const void *uv, int64_t npts, int G,
                    int2 *packed, int *flags) {
  for (int64_t n = blockIdx.x * 256ll + threadIdx.x; n < npts;
       n += (int64_t)gridDim.x * 256) {
    int mx, sx, my, sy;
    if (uv_index(uv, uv_f64, n, G, mx, sx, my, sy)) {
      packed[n] = make_int2(mx * G + sx, my * G + sy);
    } else {
      packed[n] = make_int2(INT_MIN, INT_MIN);
      atomicAdd(&flags[FLAG_INDEX], 1);
    }
  }
}

// resident CTAs per SM of the two passes over the visibilities of one job:
// both wait on loads and atomics, and 42 registers a thread hold a visibility
// and the next one's loads without spills (4.19 M visibilities, both passes
// and the tiles: 6 CTAs 384 us of the whole call, 8 CTAs 396; two or four
// visibilities a lane at once 396-409; the next one's loads ahead 387 -> 362).
// The passes over many jobs hold the job's fields too and spill at 42: 5 CTAs
// for the first and 4 for the other (256 jobs, whole call, 4.50 ms; 6 and 6
// 4.66, 6 and 5 4.63, 5 and 5 4.64, 6 and 3 4.55).
constexpr int kBinCtas = 6;

// Index step and tile of visibility n of a job at (u, v) = c.
//  * a visibility whose oversample index falls outside [0,G) would address
//    outside the GCF table in the reference; it is dropped and counted (bad)
//  * a visibility whose footprint misses the grid contributes nothing and is
//    dropped silently (the reference skips all of its taps, grid.cu:174-176)
//  * mains left/right of the grid are clamped into the edge tile (all of their
//    on-grid taps still lie inside that tile's window region), unless the
//    tiles start before the grid
// Returns the global tile, -1 when dropped.
template <class T2>
__device__ __forceinline__ int vis_tile(const BinJob &J, T2 c, int64_t n, int &mx, int &sx,
                                        int &my, int &sy, bool &bad) {
  const bool okx = index_step(c.x, J.G, mx, sx), oky = index_step(c.y, J.G, my, sy);
  bool ok = okx && oky && (unsigned)sx < (unsigned)J.G && (unsigned)sy < (unsigned)J.G;
  int gi = 0;
  if (ok && J.gcf_index) {
    gi = __ldg(J.gcf_index + n);
    ok = (unsigned)gi < (unsigned)J.n_gcf;
  }
  bad = !ok;
  const int h = J.S >> 1;
  if (!ok || mx + h < 0 || mx - h + 1 >= J.N || my + h < 0 || my - h + 1 >= J.N) return -1;
  const int cx = (J.off ? mx + J.off : min(max(mx, 0), J.N - 1)) >> J.log2T;
  const int cy = (J.off ? my + J.off : min(max(my, 0), J.N - 1)) >> J.log2T;
  return J.tile_base + (cy * J.ntx + cx) * J.n_gcf + gi;
}

template <class T> __device__ __forceinline__ T load_or_zero(const T *p, bool on) {
  T v{};
  if (on) v = __ldg(p);
  return v;
}

// Pass 1.  Every visibility of every job: its tile, and its rank among the
// visibilities of its tile (-1: dropped).  The rank comes from the histogram's
// own atomics, one for each run of equal tiles in a warp's 32 visibilities
// (tracks stay in a tile for many samples): the scattering pass then needs no
// second round of claims.  The tile itself is not kept: working it out again
// costs less than 8 bytes of traffic a visibility.
template <class T2>
__device__ __forceinline__ void bin_count_job(const BinBuffers &b, const BinJob &J, int64_t s,
                                              int64_t e) {
  const int lane = threadIdx.x & 31;
  const T2 *uv = static_cast<const T2 *>(J.uv) - J.vis_base;
  T2 c = load_or_zero(uv + s + lane, s + lane < e);
  for (int64_t g = s + lane; g - lane < e; g += 32) {
    const T2 next = load_or_zero(uv + g + 32, g + 32 < e);
    int key = -1, mx, sx, my, sy;
    bool bad = false;
    if (g < e) key = vis_tile(J, c, g - J.vis_base, mx, sx, my, sy, bad);
    c = next;
    const unsigned badm = __ballot_sync(0xffffffffu, bad);
    if (badm && lane == 0) atomicAdd(&b.flags[FLAG_INDEX], __popc(badm));
    // runs of equal keys: the first lane of each claims for all
    const int prev = __shfl_up_sync(0xffffffffu, key, 1);
    const bool head = lane == 0 || key != prev;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int first = 31 - __clz(heads & (0xffffffffu >> (31 - lane)));
    const unsigned after = lane == 31 ? 0u : heads >> (lane + 1);
    int start = 0;
    if (head && key >= 0) start = atomicAdd(&b.counts[key], after ? __ffs(after) : 32 - lane);
    start = __shfl_sync(0xffffffffu, start, first);
    if (g < e) {
      b.rank[g] = key >= 0 ? start + lane - first : -1;
      if (b.kept_pos) b.kept_pos[g] = key >= 0 ? 1 : 0;
    }
  }
}

template <int KIND>
__global__ void __launch_bounds__(256, KIND == kBinMany ? 5 : kBinCtas)
    bin_count_kernel(const __grid_constant__ BinBuffers b) {
  after_predecessor();
  for_jobs<KIND>(b, WarpSlice(b.total_vis), [&](const BinJob &J, int64_t s, int64_t e) {
    if (KIND == kBinOneF64 || (KIND == kBinMany && J.uv_f64)) bin_count_job<double2>(b, J, s, e);
    else bin_count_job<float2>(b, J, s, e);
  });
}

// first sorted position of tile t: the scan's block-local sum and its block's
// offset
__device__ __forceinline__ int tile_first(const BinBuffers &b, int t) {
  return b.counts[t] + b.block_off[t / kScanBlock];
}

// Pass 3, one part.  Sorted record of every kept visibility at the first
// position of its tile + its rank (input_sorted: the number of kept
// visibilities before it, which keeps input order; a visibility landing
// outside its own tile's range proves the input was not tile-sorted), and its
// values (one plane per polarisation; with `aos` the one value beside the
// record, one 16-byte store instead of two of 8).
template <class T2>
__device__ __forceinline__ void bin_scatter_job(const BinBuffers &b, const BinJob &J, int64_t s,
                                                int64_t e) {
  const int lane = threadIdx.x & 31;
  const T2 *uv = static_cast<const T2 *>(J.uv) - J.vis_base;
  const bool v32 = b.vals_bytes == 8;
  const float2 *vals = static_cast<const float2 *>(J.vals) - J.vis_base * b.P;  // if v32
  // the next visibility's coordinates, rank and value are loaded meanwhile
  const bool on = s + lane < e;
  T2 c = load_or_zero(uv + s + lane, on);
  int rank = on ? b.rank[s + lane] : -1;
  float2 v8 = load_or_zero(vals + (s + lane) * b.P, on && v32);
  for (int64_t g = s + lane; g < e; g += 32) {
    const bool more = g + 32 < e;
    const T2 c0 = c;
    const int rank0 = rank;
    const float2 v0 = v8;
    c = load_or_zero(uv + g + 32, more);
    rank = more ? b.rank[g + 32] : -1;
    v8 = load_or_zero(vals + (g + 32) * b.P, more && v32);
    if (rank0 < 0) continue;
    int mx, sx, my, sy;
    bool bad;
    const int64_t n = g - J.vis_base;
    const int key = vis_tile(J, c0, n, mx, sx, my, sy, bad);
    int pos;
    if (b.input_sorted) {
      pos = b.kept_pos[g];
      if (pos < tile_first(b, key) || pos >= tile_first(b, key + 1)) {
        atomicOr(&b.flags[FLAG_UNSORTED], 1);
        b.bookmarks[b.total_tiles + 1] = 1;  // this call's records have holes
        continue;
      }
    } else {
      pos = tile_first(b, key) + rank0;
    }
    int2 rec;
    if (J.rec == kRecPacked) rec = make_int2(mx * J.G + sx, my * J.G + sy);
    else if (J.rec == kRecRegtile)
      rec = regtile_record(mx & (kRegTile - 1), sx, my & (kRegTile - 1), sy, J.G, J.S);
    else if (J.rec == kRecTables)
      rec = regtile_table_record(mx & (kRegTile - 1), sx, my & (kRegTile - 1), sy, J.G, J.S);
    else rec = window_record(mx, sx, my, sy, J.G);
    if (b.aos) {
      reinterpret_cast<float4 *>(b.sorted_idx)[pos] =
          make_float4(__int_as_float(rec.x), __int_as_float(rec.y), v0.x, v0.y);
    } else {
      b.sorted_idx[pos] = rec;
      if (v32) {
        float2 *o = (float2 *)b.sorted_vals;
        o[pos] = v0;
        for (int p = 1; p < b.P; ++p) o[p * b.vstride + pos] = __ldg(vals + g * b.P + p);
      } else {
        const double2 *v = (const double2 *)J.vals + n * b.P;
        double2 *o = (double2 *)b.sorted_vals;
        for (int p = 0; p < b.P; ++p) o[p * b.vstride + pos] = __ldg(v + p);
      }
    }
    if (b.order) b.order[pos] = (int)g;
  }
}
template <int KIND>
__device__ __forceinline__ void bin_scatter_part(const BinBuffers &b, int64_t block,
                                                 int64_t nblocks) {
  const WarpSlice ws(b.total_vis, block, nblocks);
  for_jobs<KIND>(b, ws, [&](const BinJob &J, int64_t s, int64_t e) {
    if (KIND == kBinOneF64 || (KIND == kBinMany && J.uv_f64)) bin_scatter_job<double2>(b, J, s, e);
    else bin_scatter_job<float2>(b, J, s, e);
  });
}

// ---- exclusive scan ---------------------------------------------------------
constexpr int kScanThreads = kScanBlock / kScanPer;

// Exclusive prefix of a block's kScanBlock entries (v: this thread's kScanPer,
// replaced by their prefixes); returns the block's total.
__device__ __forceinline__ int scan_in_block(int (&v)[kScanPer]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ int wsum[kScanThreads / 32];
  __shared__ int total;
  int s = 0;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) {
    int t = v[i];
    v[i] = s;
    s += t;
  }
  int incl = s;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  __syncthreads();  // an earlier call's sums were read
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int x = lane < kScanThreads / 32 ? wsum[lane] : 0;
    int xi = x;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      int y = __shfl_up_sync(0xffffffffu, xi, o);
      if (lane >= o) xi += y;
    }
    if (lane < kScanThreads / 32) wsum[lane] = xi - x;
    if (lane == 31) total = xi;
  }
  __syncthreads();
  const int off = wsum[warp] + incl - s;
#pragma unroll
  for (int i = 0; i < kScanPer; ++i) v[i] += off;
  return total;
}

__device__ __forceinline__ void scan_load(const int *d, int64_t n, int64_t base,
                                          int (&v)[kScanPer]) {
  if (base + kScanPer <= n) {
    const int4 a = *reinterpret_cast<const int4 *>(d + base);
    const int4 c = *reinterpret_cast<const int4 *>(d + base + 4);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = c.x; v[5] = c.y; v[6] = c.z; v[7] = c.w;
  } else {
#pragma unroll
    for (int i = 0; i < kScanPer; ++i) v[i] = base + i < n ? d[base + i] : 0;
  }
}
__device__ __forceinline__ void scan_store(int *d, int64_t n, int64_t base,
                                           const int (&v)[kScanPer]) {
  if (base + kScanPer <= n) {
    *reinterpret_cast<int4 *>(d + base) = make_int4(v[0], v[1], v[2], v[3]);
    *reinterpret_cast<int4 *>(d + base + 4) = make_int4(v[4], v[5], v[6], v[7]);
  } else {
#pragma unroll
    for (int i = 0; i < kScanPer; ++i)
      if (base + i < n) d[base + i] = v[i];
  }
}

// Block-local exclusive prefixes of d in place; block_off[b] = the sum of the
// blocks before b, worked out by the block that finishes last (ticket, zeroed
// by the caller, counts them): one launch, and nothing waits.  The readers add
// d[i] and block_off[i / kScanBlock].
__global__ void __launch_bounds__(kScanThreads)
    scan_kernel(int *d, int64_t n, int *block_off, int *ticket) {
  __shared__ bool last;
  after_predecessor();
  const int64_t base = blockIdx.x * (int64_t)kScanBlock + threadIdx.x * kScanPer;
  int v[kScanPer];
  scan_load(d, n, base, v);
  const int total = scan_in_block(v);
  scan_store(d, n, base, v);
  if (threadIdx.x == 0) {
    block_off[blockIdx.x] = total;
    __threadfence();
    last = atomicAdd(ticket, 1) == (int)gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  int carry = 0;
  for (int64_t b0 = 0; b0 < gridDim.x; b0 += kScanBlock) {
    const int64_t at = b0 + threadIdx.x * kScanPer;
#pragma unroll
    for (int i = 0; i < kScanPer; ++i)
      v[i] = at + i < gridDim.x ? __ldcg(block_off + at + i) : 0;
    const int sum = scan_in_block(v);
#pragma unroll
    for (int i = 0; i < kScanPer; ++i)
      if (at + i < gridDim.x) block_off[at + i] = v[i] + carry;
    carry += sum;
  }
}

// the block offsets added in place
__global__ void __launch_bounds__(kScanThreads)
    scan_add_kernel(int *d, int64_t n, const int *boff) {
  int add = boff[blockIdx.x];
  int64_t base = blockIdx.x * (int64_t)kScanBlock;
  for (int i = threadIdx.x; i < kScanBlock; i += kScanThreads)
    if (base + i < n) d[base + i] += add;
}

static int64_t cdiv(int64_t a, int64_t b) { return (a + b - 1) / b; }

size_t scan_tmp_ints(int64_t n) {
  return (size_t)cdiv(n, kScanBlock) + kScanHead;
}

// tmp: the ticket (zeroed by the caller) in its first word, block offsets from
// kScanHead on
static cudaError_t scan_local(int *d, int64_t n, int *tmp, cudaStream_t s) {
  count_launch();
  return launch_overlapped(scan_kernel, (unsigned)cdiv(n, kScanBlock), kScanThreads, 0, s, true,
                           d, n, tmp + kScanHead, tmp);
}

// ---- driver -----------------------------------------------------------------
static unsigned grid_for(int64_t n) {
  int64_t b = cdiv(n, 256);
  return (unsigned)(b < 1 ? 1 : (b > 152 * 64 ? 152 * 64 : b));
}

cudaError_t launch_vis2ints(int uv_f64, const void *uv, int64_t npts, int G,
                            int2 *packed, int *flags, cudaStream_t s) {
  if (npts <= 0) return cudaSuccess;
  vis2ints_kernel<<<grid_for(npts), 256, 0, s>>>(uv_f64, uv, npts, G, packed,
                                                 flags);
  count_launch();
  return cudaGetLastError();
}

// ---- work items ---------------------------------------------------------------

// inclusive warp prefix sum
__device__ __forceinline__ int warp_incl_sum(int v, int lane) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

// Pass 3, the other part.  The final bookmarks, and the work items of the
// moving window: every non-empty tile cut into slices of at most its class's
// records.  A tile cut into several items gets a merge slot, cleared here.
__device__ __forceinline__ void bin_tiles_part(const BinBuffers &b, const ItemBuffers &it,
                                               int block, int nblocks) {
  const int lane = threadIdx.x & 31;
  for (int64_t base = (int64_t)block * 256 + (threadIdx.x & ~31); base <= b.total_tiles;
       base += (int64_t)nblocks * 256) {
    const int t = (int)(base + lane);
    int s0 = 0, e0 = 0;
    if (t <= b.total_tiles) {
      s0 = tile_first(b, t);
      b.bookmarks[t] = s0;
      if (t < b.total_tiles) e0 = tile_first(b, t + 1);
    }
    const bool full = t < b.total_tiles && e0 > s0;
    if (!it.items || !__any_sync(0xffffffffu, full)) continue;  // most tiles are empty
    int k = 0, j = 0, cls = 0, chunk = 1;
    if (full) {
      j = b.njobs == 1 ? 0 : find_job32(b.tile_base, b.njobs, t);
      cls = it.job_class[j];
      chunk = it.chunks.c[cls];
      k = (e0 - s0 + chunk - 1) / chunk;
    }
    for (int c = 0; c < it.nclasses; ++c) {
      const int kc = cls == c ? k : 0;
      if (!__any_sync(0xffffffffu, kc > 0)) continue;
      const int incl = warp_incl_sum(kc, lane);
      int start = 0;
      if (lane == 31) start = atomicAdd(&it.counters[c], incl);
      start = __shfl_sync(0xffffffffu, start, 31);
      // a merge slot for a tile cut into several items (complex64 grids of
      // classes with slots)
      const MergeSlots &ms = it.slots.m[c];
      int slot = -1;
      if (ms.base != nullptr) {  // uniform over the warp
        const int need = kc > 1 && !it.jobs[j].out_f64 ? 1 : 0;
        const unsigned needs = __ballot_sync(0xffffffffu, need);
        if (needs) {
          int h0 = 0;
          if (lane == 0) h0 = atomicAdd(&it.heavy_counters[c], __popc(needs));
          h0 = __shfl_sync(0xffffffffu, h0, 0);
          if (need) {
            slot = h0 + __popc(needs & ((1u << lane) - 1));
            if (slot >= ms.cap) {
              atomicOr(&b.flags[FLAG_BOUNDS], 1);
              slot = -1;
            } else {
              ms.desc[slot] = make_int4(j, t - b.tile_base[j], kc, 0);
            }
          }
          for (unsigned left = needs; left; left &= left - 1) {
            const int sl = __shfl_sync(0xffffffffu, slot, __ffs(left) - 1);
            if (sl < 0) continue;
            double2 *const cells = ms.base + (size_t)sl * ms.cells;
            for (int i = lane; i < ms.cells; i += 32) cells[i] = make_double2(0.0, 0.0);
          }
        }
      }
      if (kc) {
        WorkItem *dst = it.items + c * it.class_cap + start + (incl - kc);
        const JobDesc &J = it.jobs[j];
        const int local = t - b.tile_base[j], tile = J.n_gcf > 1 ? local / J.n_gcf : local;
        WorkItem w;
        w.job = j;
        w.bin = local;
        w.slot = slot;
        w.ox = (tile % J.ntx) * J.T - J.off - J.S / 2 + 1;
        w.oy = (tile / J.ntx) * J.T - J.off - J.S / 2 + 1;
        w.pad_ = 0;
        for (int i = 0; i < kc; ++i) {
          w.start = s0 + i * chunk;
          w.end = min(e0, s0 + (i + 1) * chunk);
          dst[i] = w;
        }
      }
    }
  }
}

// Pass 3: both parts side by side, the tiles' blocks first.
template <int KIND>
__global__ void __launch_bounds__(256, KIND == kBinMany ? 4 : kBinCtas)
    bin_finish_kernel(const __grid_constant__ BinBuffers b, const __grid_constant__ ItemBuffers it,
                      int tile_blocks) {
  after_predecessor();
  if ((int)blockIdx.x < tile_blocks) bin_tiles_part(b, it, blockIdx.x, tile_blocks);
  else bin_scatter_part<KIND>(b, (int64_t)blockIdx.x - tile_blocks, (int64_t)gridDim.x - tile_blocks);
}

cudaError_t run_binning(const BinBuffers &b, const ItemBuffers *items, cudaStream_t s) {
  cudaError_t e;
  const int kind = b.njobs > 1 ? kBinMany : b.one.uv_f64 ? kBinOneF64 : kBinOneF32;
  auto count = kind == kBinMany     ? bin_count_kernel<kBinMany>
               : kind == kBinOneF64 ? bin_count_kernel<kBinOneF64>
                                    : bin_count_kernel<kBinOneF32>;
  auto finish = kind == kBinMany     ? bin_finish_kernel<kBinMany>
                : kind == kBinOneF64 ? bin_finish_kernel<kBinOneF64>
                                     : bin_finish_kernel<kBinOneF32>;
  if (b.total_vis > 0) {
    count_launch();
    if ((e = launch_overlapped(count, grid_for(b.total_vis), 256, 0, s, true, b)) !=
        cudaSuccess)
      return e;
  }
  if ((e = scan_local(b.counts, (int64_t)b.total_tiles + 1, b.scan_tmp, s)) != cudaSuccess)
    return e;
  if (b.input_sorted && b.total_vis > 0) {
    // the ticket once more; the tiles' block offsets lie before this scan's
    int *const tmp = b.scan_tmp + scan_tmp_ints((int64_t)b.total_tiles + 1);
    if ((e = cudaMemsetAsync(tmp, 0, sizeof(int), s)) != cudaSuccess) return e;
    if ((e = scan_local(b.kept_pos, b.total_vis, tmp, s)) != cudaSuccess) return e;
    scan_add_kernel<<<(unsigned)cdiv(b.total_vis, kScanBlock), kScanThreads, 0, s>>>(
        b.kept_pos, b.total_vis, tmp + kScanHead);
    count_launch();
  }
  ItemBuffers it{};
  if (items) it = *items;
  for (int c = 0; c < kMaxClasses; ++c)
    if (it.slots.m[c].cap <= 0) it.slots.m[c].base = nullptr;
  const unsigned tiles = grid_for(cdiv((int64_t)b.total_tiles + 1, 4));
  const unsigned vis = b.total_vis > 0 ? grid_for(b.total_vis) : 0;
  count_launch();
  return launch_overlapped(finish, tiles + vis, 256, 0, s, true, b, it, (int)tiles);
}

// ---- FP64 merge slots of tiles cut into several work items ---------------------

// one CTA per slot (grid-stride over slots): cells of the slot's R x R
// sub-grid (P planes), origin at the tile's corner minus the halo
__global__ void __launch_bounds__(256)
    merge_finalize_kernel(MergeSlots m, const int *count, const JobDesc *jobs, int S, int T,
                          int P) {
  const int n = min(*count, m.cap);
  const int R = T + S - 1, H = S / 2;
  for (int sl = blockIdx.x; sl < n; sl += gridDim.x) {
    const int4 d = m.desc[sl];
    const JobDesc &J = jobs[d.x];
    const int tile = J.n_gcf > 1 ? d.y / J.n_gcf : d.y;
    const int ox = (tile % J.ntx) * T - J.off - H + 1, oy = (tile / J.ntx) * T - J.off - H + 1;
    const double2 *src = m.base + (size_t)sl * m.cells;
    for (int i = threadIdx.x; i < P * R * R; i += 256) {
      const double2 v = src[i];
      if (v.x == 0.0 && v.y == 0.0) continue;
      const int p = i / (R * R), c = i - p * R * R;
      const int gx = ox + c % R, gy = oy + c / R;
      if ((unsigned)gx < (unsigned)J.N && (unsigned)gy < (unsigned)J.N)
        out_red(J, (size_t)gy * J.N + gx, p, P, v.x, v.y);
    }
  }
}

cudaError_t launch_merge_finalize(const MergeSlots &m, const int *heavy_counter,
                                  const JobDesc *jobs, int S, int T, int P, int sm_count,
                                  cudaStream_t s) {
  if (!m.base || m.cap <= 0) return cudaSuccess;
  merge_finalize_kernel<<<sm_count * 8, 256, 0, s>>>(m, heavy_counter, jobs, S, T, P);
  count_launch();
  return cudaGetLastError();
}

__global__ void inject_flags_kernel(int *flags, int bits) {
  for (int f = 0; f < 4; ++f)
    if (bits & (1 << f)) atomicOr(&flags[f], 1);
}

cudaError_t launch_inject_flags(int *flags, int bits, cudaStream_t s) {
  inject_flags_kernel<<<1, 1, 0, s>>>(flags, bits);
  count_launch();
  return cudaGetLastError();
}

// ---- set-up: table upload through kernel parameters, and clearing ----------------
// A launch carries its parameters with it (copied by the driver at the call),
// so tables sent this way never wait on a copy engine behind the bulk
// transfers of other streams, and the host buffer is free once the call
// returns.
constexpr int kUploadChunk = 16384;  // bytes per launch (parameters: up to 32 KB)
constexpr int kUploadSmall = 2048;   // a job or two: no 16 KB of parameters
template <int BYTES> struct SetupParams {
  uint4 *dst;
  int n16;  // 16-byte words in this chunk
  ZeroRanges zero;
  uint4 data[BYTES / 16];
};

__device__ __forceinline__ void zero_range(void *p, size_t bytes, size_t i, size_t stride) {
  if ((reinterpret_cast<uintptr_t>(p) | bytes) % 16 == 0) {
    uint4 *const q = static_cast<uint4 *>(p);
    for (; i < bytes / 16; i += stride) q[i] = make_uint4(0, 0, 0, 0);
  } else {
    int *const q = static_cast<int *>(p);
    for (; i < bytes / 4; i += stride) q[i] = 0;
  }
}

template <int BYTES>
__global__ void __launch_bounds__(256) setup_kernel(const __grid_constant__ SetupParams<BYTES> p) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const size_t i = blockIdx.x * 256 + threadIdx.x, stride = (size_t)gridDim.x * 256;
  for (int k = (int)i; k < p.n16; k += (int)stride) p.dst[k] = p.data[k];
  for (int r = 0; r < p.zero.n; ++r) zero_range(p.zero.p[r], p.zero.bytes[r], i, stride);
}
// the same without a table: its launch carries no table
__global__ void __launch_bounds__(256) clear_kernel(const __grid_constant__ ZeroRanges z) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const size_t i = blockIdx.x * 256 + threadIdx.x, stride = (size_t)gridDim.x * 256;
  for (int r = 0; r < z.n; ++r) zero_range(z.p[r], z.bytes[r], i, stride);
}

template <int BYTES>
static void upload_chunk(char *dst, const char *src, size_t n, const ZeroRanges &zero,
                         unsigned blocks, cudaStream_t s) {
  static thread_local SetupParams<BYTES> p;  // 16 KB: off the stack
  p.dst = reinterpret_cast<uint4 *>(dst);
  p.n16 = (int)(n / 16);
  p.zero = zero;
  memcpy(p.data, src, n);
  setup_kernel<BYTES><<<blocks, 256, 0, s>>>(p);
  count_launch();
}

cudaError_t launch_setup(void *dst, const void *src, size_t bytes, const ZeroRanges &zero,
                         cudaStream_t s) {
  if (bytes % 16 || (uintptr_t)dst % 16) return cudaErrorInvalidValue;
  size_t clear = 0;
  for (int r = 0; r < zero.n; ++r) clear += zero.bytes[r];
  // 4 KB a block, up to eight blocks on each of 152 SMs
  const unsigned blocks = (unsigned)std::min<size_t>(152 * 8, 1 + clear / 4096);
  if (bytes == 0) {
    if (zero.n > 0) {
      clear_kernel<<<blocks, 256, 0, s>>>(zero);
      count_launch();
    }
    return cudaGetLastError();
  }
  char *const d = static_cast<char *>(dst);
  const char *const h = static_cast<const char *>(src);
  if (bytes <= kUploadSmall) {
    upload_chunk<kUploadSmall>(d, h, bytes, zero, blocks, s);
    return cudaGetLastError();
  }
  for (size_t o = 0; o < bytes; o += kUploadChunk)
    upload_chunk<kUploadChunk>(d + o, h + o, std::min<size_t>(kUploadChunk, bytes - o),
                               o == 0 ? zero : ZeroRanges{}, o == 0 ? blocks : 1, s);
  return cudaGetLastError();
}

// The output grids of a batch's jobs [j0, j1), kZeroChunk bytes at a time
// (JobDesc::blk0 numbers the chunks of the jobs of a class): one launch where
// a memset for each of 256 jobs took twice the time.
__global__ void __launch_bounds__(256)
    zero_jobs_kernel(const JobDesc *jobs, int njobs, int chunks) {
  for (int c = blockIdx.x; c < chunks; c += gridDim.x) {
    int j = 0, e = njobs - 1;
    while (j < e) {
      const int mid = (j + e + 1) >> 1;
      if (__ldg(&jobs[mid].blk0) <= c) j = mid; else e = mid - 1;
    }
    const JobDesc &J = jobs[j];
    const size_t bytes = (size_t)(J.out_f64 ? 16 : 8) * J.P * J.N * J.N;
    const size_t o = (size_t)(c - J.blk0) * kZeroChunk;
    zero_range(static_cast<char *>(J.out) + o, min(kZeroChunk, bytes - o), threadIdx.x, 256);
  }
}

cudaError_t launch_zero_jobs(const JobDesc *jobs, int njobs, int chunks, int sm_count,
                             cudaStream_t s) {
  if (chunks <= 0) return cudaSuccess;
  zero_jobs_kernel<<<std::min(chunks, sm_count * 8), 256, 0, s>>>(jobs, njobs, chunks);
  count_launch();
  return cudaGetLastError();
}

// ---- DEBUG1 footprint inputs --------------------------------------------------
__global__ void count_inputs_kernel(void *vals, int vals_f64, int64_t npts,
                                    int P, void *gcf, int64_t gcf_elems) {
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
       i < npts * P; i += stride) {
    int64_t n = i / P;
    if (vals_f64) ((double2 *)vals)[i] = make_double2(1.0, (double)n);
    else ((float2 *)vals)[i] = make_float2(1.f, (float)n);
  }
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
       i < gcf_elems; i += stride) {
    if (vals_f64) ((double2 *)gcf)[i] = make_double2(1.0, 0.0);
    else ((float2 *)gcf)[i] = make_float2(1.f, 0.f);
  }
}

cudaError_t launch_count_inputs(void *vals, int vals_f64, int64_t npts, int P,
                                void *gcf, int64_t gcf_elems, cudaStream_t s) {
  count_inputs_kernel<<<grid_for(npts * P > gcf_elems ? npts * P : gcf_elems),
                        256, 0, s>>>(vals, vals_f64, npts, P, gcf, gcf_elems);
  count_launch();
  return cudaGetLastError();
}

}  // namespace gg
