// Gridding with the on-the-fly Gaussian at support 32, FP32 values: every
// 16x16 block of output cells is summed in the registers of one warp.
//
// The factor of a tap is the product of two 1-D factors, so a record costs a
// block two vectors instead of a 32x32 table, and a support-32 footprint
// covers a large share of any block it touches.  Lane (c, h) of a warp holds
// the columns 2c, 2c+1 and the rows 2h, 2h+1, 8+2h, 9+2h of its block.  The
// visibilities that reach a block have their main cells in a 48x48
// neighbourhood: 6x6 uv tiles of 8 cells, which are 6 contiguous ranges of the
// sorted records, one for each row of tiles.  Each of them costs
//   * v * gx for two columns: one 8-byte load of column factors, padded with
//     zeros so that columns outside the footprint get zero;
//   * 8 packed multiply-adds by four row factors, two 8-byte loads.  The
//     first range reaches only the rows 0..7 and the last only 8..15: groups
//     of records that lie in one of them take one load and 4 multiply-adds.
// Both loads read a copy of the padded factors shifted to the alignment of the
// footprint (two copies).  Shared memory returns 8 bytes a lane and cycle
// also for broadcasts, so the shape of a lane's cells decides: 2 x 4 takes 5
// cycles for 10 packed operations, 1 x 8 took 7 for 9.
// Nothing moves, and the cells of most blocks are summed by one warp and stored
// once: no atomics, no cleared grid.  9 blocks visit a record, 45 % of their multiply-adds are
// inside its footprint; the moving window's shared-memory sub-grid cost a
// read-modify-write of each of the 1024 taps of (nearly) every record.
//
// A value that is not finite would reach cells outside its footprint through
// the zeros: a block whose sums are not finite is summed again cell by cell.
//
// Compensated sums: every cell's sum starts at a number so large that no term leads
// out of its binade, which makes what an addition rounds off exact to work out
// (exact_add2), two records at once; the sums are moved to a larger one when they
// come to need it.
//
// Few blocks (small grids), compensated sums: the warps of a CTA share a
// block, every warp takes every WARPS-th group of 32 records, and the partial
// (hi, lo) sums are added by TwoSum in shared memory.
//
// sep_plan_kernel looks at the blocks first.  Those that no record reaches it clears
// itself (on a grid that is added into they stay as they are), so that a warp
// does not pay a claim for each: 10 k visibilities on 8192^2 311 -> 217 us.  Dense
// ones, with more records than half a resident warp's share of all visits, are cut
// into units of 512 records (4096 for a CTA) that merge their sums in FP64, the
// last one storing them: a block would be one warp's walk through all its records.
// 1.05 M visibilities on 4096^2, nine tenths of them 4 cells rms around the
// centre: 38.8 -> 0.80 ms (the moving window 2.8); 4.19 M 100 cells rms around it
// 12.2 -> 2.6 (7.2).  Without dense blocks the two kernels cost 2 to 4 %: 1.05 M uniform ones
// on 4096^2 583 -> 605 us.
//
// Bound by the FMA pipe.  16.8 M visibilities of a uniform disk on 8192^2, whole
// call, and error against 64 bits: the moving window's shared-memory sub-grid 25.3
// ms, 7.3e-8; this kernel 8.0 ms, 6.1e-8 (8 groups of two unrolled; 4 8.1, 16
// 9.5; three CTAs per SM, which spill, 8.25; one record at once 9.8).  Four records
// at once take 7.1 ms, but in random order into a complex128 grid have 6.3e-8 where
// the moving window has 5.9e-8; runs of 16 summed plainly 4.95 ms with 9.3e-8 and
// 9.2e-8: not taken.
#include <algorithm>
#include <climits>
#include <type_traits>

#include "gg_kernels.cuh"

namespace gg {

namespace {

constexpr int kSepS = 32, kSepB = kSepBlock;  // support, block side
constexpr int kSepWarps = 8;
constexpr int kSepRow = 64;  // floats of a padded factor row: tap 0 at 16

constexpr int kSepAt = 2;  // records added at once
constexpr int kSepStage = 32;  // staged records of a warp: a group

// shared memory: factors [G][2][64] (copy c holds the row from its entry c
// on), a staging block per warp, and the partial sums of a shared block
__host__ __device__ constexpr size_t sep_factor_floats(int G) { return (size_t)G * 2 * kSepRow; }

__device__ __forceinline__ float2 lds64(uint32_t a) {
  float2 v;
  asm("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a));
  return v;
}

__device__ __noinline__ void sep_store_f64(const JobDesc &J, size_t cell, int plane, int P,
                                           bool accumulate, double dr, double di) {
  if (accumulate)
    out_red(J, cell, plane, P, dr, di);
  else
    grid_store<double>((double *)J.out, cell, plane, P, (size_t)J.N * J.N, J.planar, dr, di);
}
__device__ __forceinline__ void sep_store_f32(const JobDesc &J, size_t cell, int plane, int P,
                                              bool accumulate, float fr, float fi) {
  const size_t NN = (size_t)J.N * J.N;
  if (accumulate) {
    if (J.planar) {
      red_add((float *)J.out + plane * NN + cell, fr);
      red_add((float *)J.out + ((size_t)P + plane) * NN + cell, fi);
    } else {
      red_add_v2((float *)J.out + 2 * (plane * NN + cell), fr, fi);
    }
  } else if (J.planar) {
    grid_store<float>((float *)J.out, cell, plane, P, NN, true, fr, fi);
  } else {
    reinterpret_cast<float2 *>(J.out)[plane * NN + cell] = make_float2(fr, fi);
  }
}

// hi + lo into a cell of the grid
__device__ __forceinline__ void sep_store(const JobDesc &J, int gx, int gy, int plane, int P,
                                          bool accumulate, const float2 h, const float2 l) {
  if (gx >= J.N || gy >= J.N) return;
  // a grid that is added into: its other cells stay as they are
  if (accumulate && h.x == 0.f && h.y == 0.f && l.x == 0.f && l.y == 0.f) return;
  const size_t cell = (size_t)gy * J.N + gx;
  // FP64 sums only for a complex128 grid: the FP64 pipe is narrow
  if (J.out_f64)
    sep_store_f64(J, cell, plane, P, accumulate, (double)h.x + (double)l.x,
                  (double)h.y + (double)l.y);
  else
    sep_store_f32(J, cell, plane, P, accumulate, __fadd_rn(h.x, l.x), __fadd_rn(h.y, l.y));
}

// hi + lo exactly into a cell of a dense block's merge slot
__device__ __forceinline__ void sep_merge(double2 *cell, const float2 h, const float2 l) {
  const double dr = (double)h.x + (double)l.x, di = (double)h.y + (double)l.y;
  if (dr != 0.0) red_add(&cell->x, dr);
  if (di != 0.0) red_add(&cell->y, di);
}

// sorted record k and its value in a plane
__device__ __forceinline__ void sep_record(const SepTileLaunch &p, int k, int plane, int2 &q,
                                           float2 &v) {
  if (p.vals) {
    q = p.idx[k];
    v = p.vals[plane * p.vstride + k];
  } else {
    const float4 t = reinterpret_cast<const float4 *>(p.idx)[k];
    q = make_int2(__float_as_int(t.x), __float_as_int(t.y));
    v = make_float2(t.z, t.w);
  }
}

// main cells and sub-kernel of a sorted record (window_record)
__device__ __forceinline__ void sep_decode(const int2 q, int log2G, int &mx, int &my, int &sx,
                                           int &sy) {
  mx = (int)((unsigned)q.x & 0xffffu) - kWinMainBias;
  my = (int)((unsigned)q.x >> 16) - kWinMainBias;
  sx = q.y & ((1 << log2G) - 1);
  sy = q.y >> log2G;
}

// the job of a block
__device__ __forceinline__ const JobDesc &sep_job(const SepTileLaunch &p, int blk) {
  int j = 0, e = p.njobs - 1;
  while (j < e) {
    const int mid = (j + e + 1) >> 1;
    if (p.jobs[mid].blk0 <= blk) j = mid; else e = mid - 1;
  }
  return p.jobs[j];
}
// first cell of a job's block
__device__ __forceinline__ void sep_origin(const JobDesc &J, int blk, int &x0, int &y0) {
  const int nb = (J.N + kSepB - 1) / kSepB, b = blk - J.blk0;
  x0 = (b % nb) * kSepB;
  y0 = (b / nb) * kSepB;
}
// the sorted records of the r-th row of tiles that reaches a block (tiles start
// kSepOff before the grid)
__device__ __forceinline__ int2 sep_range(const JobDesc &J, int x0, int y0, int r) {
  const int bx = x0 / kSepTile, by = y0 / kSepTile + r;
  if (by >= J.ntx) return make_int2(0, 0);
  const int *const bm = J.bookmarks + by * J.ntx;
  return make_int2(bm[bx], bm[min(bx + 6, J.ntx)]);
}

// A block whose packed sums are not finite: its cells from those of its records
// [t0, t1) whose footprints cover them.
template <bool COMP>
__device__ __noinline__ void sep_redo(const SepTileLaunch &p, const JobDesc &J, int x0, int y0,
                                      int plane, const float *gt, int t0, int t1, double2 *slot,
                                      int tid, int nt) {
  constexpr int H = kSepS / 2;
  for (int c = tid; c < kSepB * kSepB; c += nt) {
    const int x = x0 + c % kSepB, y = y0 + c / kSepB;
    u64 run = 0ull, hi = 0ull, lo = 0ull;
    auto merge = [&]() {
      u64 e;
      hi = two_sum2(hi, run, e);
      lo = add2(lo, e);
      run = 0ull;
    };
    int t = 0;  // of the range's first record
    for (int r = 0; r < 6; ++r) {
      const int2 range = sep_range(J, x0, y0, r);
      const int first = range.x + max(0, t0 - t), last = min(range.y, range.x + (t1 - t));
      t += range.y - range.x;
      for (int k = first; k < last; ++k) {
        int2 q;
        float2 v;
        sep_record(p, k, plane, q, v);
        int mx, my, sx, sy;
        sep_decode(q, J.log2G, mx, my, sx, sy);
        const int a = x - (mx - H + 1), b = y - (my - H + 1);
        if ((unsigned)a >= (unsigned)kSepS || (unsigned)b >= (unsigned)kSepS) continue;
        const float gx = gt[sx * 2 * kSepRow + 16 + a], gy = gt[sy * 2 * kSepRow + 16 + b];
        run = fma2(mul2(pk2(v.x, v.y), pk2(gx, gx)), pk2(gy, gy), run);
        if (COMP) merge();
      }
    }
    const float2 h = upk2(COMP ? hi : run), l = upk2(lo);
    if (slot) sep_merge(slot + c, h, l);
    else sep_store(J, x, y, plane, p.P, p.accumulate, h, l);
  }
}

// zeros into a block of the grid
__device__ __forceinline__ void sep_clear(const SepTileLaunch &p, int blk, int lane) {
  const JobDesc &J = sep_job(p, blk);
  const int N = J.N, P = p.P;
  int x0, y0;
  sep_origin(J, blk, x0, y0);
  const int x = x0 + lane % kSepB, y = y0 + lane / kSepB;
  const size_t NN = (size_t)N * N, cell = (size_t)y * N + x;
  if (!J.planar && !J.out_f64) {
    float2 *const out = static_cast<float2 *>(J.out) + cell;
    for (int plane = 0; plane < P; ++plane)
#pragma unroll
      for (int i = 0; i < kSepB / 2; ++i)
        if (x < N && y + 2 * i < N) out[plane * NN + (size_t)(2 * i) * N] = make_float2(0.f, 0.f);
    return;
  }
  for (int plane = 0; plane < P; ++plane)
    for (int i = 0; i < kSepB / 2; ++i)
      sep_store(J, x, y + 2 * i, plane, P, false, make_float2(0.f, 0.f), make_float2(0.f, 0.f));
}

// What there is to do, 32 blocks a CTA.  Blocks that no record reaches are cleared
// here (or left, if the grid is added into); of the others a bit is set in `mask`,
// except that those with more than dense_min records are cut into units of
// dense_unit, each block with a merge slot that is cleared here.
__global__ void __launch_bounds__(256) sep_plan_kernel(const __grid_constant__ SepTileLaunch p) {
  __shared__ unsigned s_empty, s_dense;
  __shared__ int s_slot[32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, blk0 = blockIdx.x * 32;
  after_predecessor();
  if (warp == 0) {
    const int blk = min(blk0 + lane, p.total_blocks - 1);
    const bool valid = blk0 + lane < p.total_blocks;
    const JobDesc &J = sep_job(p, blk);
    int x0, y0, records = 0, slot = -1;
    sep_origin(J, blk, x0, y0);
#pragma unroll
    for (int r = 0; r < 6; ++r) {
      const int2 range = sep_range(J, x0, y0, r);
      records += range.y - range.x;
    }
    if (valid && records > p.dense_min) {
      const int units = (records + p.dense_unit - 1) / p.dense_unit;
      // slots and units are given out together: first units ascend with the slots
      const u64 old = atomicAdd(p.dense_count, (1ull << 32) | (u64)units);
      if ((old >> 32) < (u64)p.dense_cap) {
        slot = (int)(old >> 32);
        p.dense[slot] = make_int4(blk, (int)(unsigned)old, units, 0);
      }
    }
    s_slot[lane] = slot;
    const unsigned reached = __ballot_sync(0xffffffffu, valid && records > 0 && slot < 0);
    const unsigned dense = __ballot_sync(0xffffffffu, slot >= 0);
    const unsigned empty = __ballot_sync(0xffffffffu, valid && records == 0);
    if (lane == 0) {
      p.mask[blockIdx.x] = reached;
      s_dense = dense;
      s_empty = p.accumulate ? 0u : empty;
    }
  }
  __syncthreads();
  const int cells = p.P * kSepB * kSepB;
  for (unsigned d = s_dense; d; d &= d - 1) {
    double2 *const to = p.slots + (size_t)s_slot[__ffs(d) - 1] * cells;
    for (int i = threadIdx.x; i < cells; i += 256) to[i] = make_double2(0.0, 0.0);
  }
  // every eighth empty block a warp
  unsigned e = s_empty;
  for (int n = 0; e; ++n, e &= e - 1)
    if ((n & 7) == warp) sep_clear(p, blk0 + __ffs(e) - 1, lane);
}

// DENSE: the units of the dense blocks; else the blocks that are summed as a whole
template <bool COMP, bool SHARE, bool DENSE>
__global__ void __launch_bounds__(32 * kSepWarps, COMP ? 2 : 3)
    septile_kernel(const __grid_constant__ SepTileLaunch p) {
  constexpr int H = kSepS / 2, NT = 32 * kSepWarps;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  float *const gt = reinterpret_cast<float *>(smem);
  // factor offsets and values of a group
  float4 *const rec = reinterpret_cast<float4 *>(gt + sep_factor_floats(p.G)) + warp * kSepStage;
  float4 *const part = reinterpret_cast<float4 *>(gt + sep_factor_floats(p.G)) +
                       kSepWarps * kSepStage;
  // padded factors: entry i of a row is tap i - 16, zero outside
  const float inv = 1.0f / (2.0f * p.sigma * p.sigma);
  for (int i = tid; i < p.G * 2 * kSepRow; i += NT) {
    const int s = i / (2 * kSepRow), ap = i % kSepRow + i / kSepRow % 2 - 16;
    const float x = (float)(ap - H + 1) - (float)s / (float)p.G;
    gt[i] = (unsigned)ap < (unsigned)kSepS ? expf(-(x * x) * inv) : 0.f;
  }
  after_predecessor();
  __syncthreads();

  const int c = lane & 7, h = lane >> 3;
  const uint32_t ax = smem_addr(gt) + 8 * c, ay = smem_addr(gt) + 8 * h;
  auto row = [&](int k) { return 2 * h + (k >> 1 & 1) + 8 * (k >> 2); };
  // units, or chunks of p.chunk blocks, are spread over the SMs first, then claimed,
  // one ahead (two ahead, the last ones waited behind others: 10 % on tracks)
  const int dense = DENSE ? min((int)(*p.dense_count >> 32), p.dense_cap) : 0;
  int total = (p.total_blocks + p.chunk - 1) / p.chunk;
  if constexpr (DENSE) total = dense > 0 ? p.dense[dense - 1].y + p.dense[dense - 1].z : 0;
  const int workers = SHARE ? (int)gridDim.x : (int)gridDim.x * kSepWarps;
  __shared__ int s_share;
  auto share = [&](int x) {  // the first lane's (thread's) x
    if constexpr (SHARE) {
      if (tid == 0) s_share = x;
      __syncthreads();
      x = s_share;
      __syncthreads();
      return x;
    }
    return __shfl_sync(0xffffffffu, x, 0);
  };
  const bool leader = SHARE ? tid == 0 : lane == 0;
  auto claim_one = [&]() { return leader ? atomicAdd(p.next + DENSE, 1) + workers : 0; };
  int unit = SHARE ? (int)blockIdx.x : (int)(blockIdx.x + warp * gridDim.x);
  if (unit >= total) return;  // no one waits for this worker
  // a chunk's blocks that are summed; alone, a block tells by its records
  auto chunk_mask = [&]() {
    return DENSE || p.chunk == 1
               ? 1u
               : p.mask[unit * p.chunk >> 5] >> (unit * p.chunk & 31) & ((1u << p.chunk) - 1);
  };
  unsigned mask = chunk_mask();
  int claim = claim_one();
  auto advance = [&]() {  // false: nothing left
    unit = share(claim);
    if (unit >= total) return false;
    mask = chunk_mask();
    claim = claim_one();
    return true;
  };
  while (true) {
    int entry = 0, first = 0, blk;  // of a dense block; its records from `first` on
    if constexpr (DENSE) {
      int hi = dense - 1;
      while (entry < hi) {
        const int mid = (entry + hi + 1) >> 1;
        if (p.dense[mid].y <= unit) entry = mid; else hi = mid - 1;
      }
      blk = p.dense[entry].x;
      first = (unit - p.dense[entry].y) * p.dense_unit;
    } else {
      while (mask == 0)
        if (!advance()) return;
      blk = unit * p.chunk + __ffs(mask) - 1;
      mask &= mask - 1;
    }
    const JobDesc &J = sep_job(p, blk);
    int x0, y0;
    sep_origin(J, blk, x0, y0);
    const int log2G = J.log2G;
    // lane r < 6: the r-th row of tiles
    int beg = 0, end = 0;
    if (lane < 6) {
      const int2 range = sep_range(J, x0, y0, lane);
      beg = range.x;
      end = range.y;
    }
    // the ranges as one list: record t of it is record t + shift[r] of the
    // sorted ones, r the last range with start[r] <= t
    int sum = end - beg;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    const int start = sum - (end - beg), shift = beg - start;  // of range `lane`
    const int records = __shfl_sync(0xffffffffu, sum, 5);
    const int first_end = __shfl_sync(0xffffffffu, sum, 0);
    const int last_beg = __shfl_sync(0xffffffffu, start, 5);
    if constexpr (!DENSE) {
      if (records == 0 || (records > p.dense_min && !(p.mask[blk >> 5] >> (blk & 31) & 1))) continue;
    }
    const int last = DENSE ? min(records, first + p.dense_unit) : records;
    for (int plane = 0; plane < p.P; ++plane) {
      double2 *const slot =
          DENSE ? p.slots + ((size_t)entry * p.P + plane) * (kSepB * kSepB) : nullptr;
      // cell k: column 2c + (k & 1), row 2h + (k >> 1 & 1) + 8 (k >> 2).  Plain
      // sums, or sums from `base` on and their remainders.
      u64 sum[8], lo[COMP ? 8 : 1];
      u64 base = 0ull;
      float room = 0.f, bound = 0.f;  // that `base` is good for, and of the sums
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        sum[k] = 0ull;
        if constexpr (COMP) lo[k] = 0ull;
      }
      // the next terms add up to `more` at most: bound the sums by what they are
      // (sums of random signs stay far below those of magnitudes), and if they
      // and the terms need it move them to a larger base
      auto make_room = [&](float more) {
        if constexpr (COMP) {
          unsigned top = 0;
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const float2 t = upk2(sub2(sum[k], base));
            top = max(top, max(finite_magnitude(t.x), finite_magnitude(t.y)));
          }
          bound = __uint_as_float(__reduce_max_sync(0xffffffffu, top)) + more;
          if (room > 0.f && 4.f * bound <= room) return;
          const float b = sum_base(16.f * bound);
          const u64 b2 = pk2(b, b);
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            const u64 t = sub2(sum[k], base), n = add2(t, b2);
            lo[k] = add2(lo[k], sub2(t, sub2(n, b2)));
            sum[k] = n;
          }
          base = b2;
          room = b * (1.f / 1.5f);
        }
      };
      // the list in groups of 32
      int2 q = make_int2(0, 0);
      float2 v = make_float2(0.f, 0.f);
      int n = 0;
      auto fetch = [&](int g) {
        const int t = first + 32 * g + lane;
        n = min(32, last - first - 32 * g);
        if (n <= 0) return;
        int k = t + __shfl_sync(0xffffffffu, shift, 0);
#pragma unroll
        for (int r = 1; r < 6; ++r) {
          const int s0 = __shfl_sync(0xffffffffu, start, r);
          const int sh = __shfl_sync(0xffffffffu, shift, r);
          if (t >= s0) k = t + sh;
        }
        if (lane < n) sep_record(p, k, plane, q, v);
      };
      int g = SHARE ? warp : 0;
      fetch(g);
      while (n > 0) {
        const int m = n, at_group = first + 32 * g;
        __syncwarp();  // the previous group was read
        int2 at = make_int2(0, 0);
        if (lane < m) {
          int mx, my, sx, sy;
          sep_decode(q, log2G, mx, my, sx, sy);
          // entries of the padded rows at the block's first column and row
          const int ix = x0 - (mx - H + 1) + 16, iy = y0 - (my - H + 1) + 16;
          at = make_int2(((sx * 2 + (ix & 1)) * kSepRow + (ix & ~1)) * 4,
                         ((sy * 2 + (iy & 1)) * kSepRow + (iy & ~1)) * 4);
        } else {
          v = make_float2(0.f, 0.f);
        }
        rec[lane] = make_float4(__int_as_float(at.x), __int_as_float(at.y), v.x, v.y);
        if constexpr (COMP) {
          const unsigned top = __reduce_max_sync(
              0xffffffffu, max(finite_magnitude(v.x), finite_magnitude(v.y)));
          const float more = (float)m * __uint_as_float(top);  // factors are at most 1
          bound += more;
          if (!(2.f * bound <= room)) make_room(more);
        }
        g += SHARE ? kSepWarps : 1;
        fetch(g);
        __syncwarp();
        // kSepAt records at once into the cells [K0, K1)
        auto group = [&](auto k0, auto k1) {
          constexpr int K0 = decltype(k0)::value, K1 = decltype(k1)::value;
          constexpr bool LOW = K0 == 0, HIGH = K1 == 8;
          auto add = [&](const float4 *o) {
            u64 w[2][kSepAt];
            float2 g0[kSepAt], g1[kSepAt];
#pragma unroll
            for (int r = 0; r < kSepAt; ++r) {
              const float4 t = o[r];
              const float2 gx = lds64(ax + __float_as_uint(t.x));
              if constexpr (LOW) g0[r] = lds64(ay + __float_as_uint(t.y));
              if constexpr (HIGH) g1[r] = lds64(ay + __float_as_uint(t.y) + 32);
              const u64 vv = pk2(t.z, t.w);
              w[0][r] = mul2(vv, pk2(gx.x, gx.x));
              w[1][r] = mul2(vv, pk2(gx.y, gx.y));
            }
#pragma unroll
            for (int k = K0; k < K1; ++k) {
              auto terms = [&](u64 a) {
#pragma unroll
                for (int r = 0; r < kSepAt; ++r) {
                  const float2 gy = k < 4 ? g0[r] : g1[r];
                  const float g = k & 2 ? gy.y : gy.x;
                  a = fma2(w[k & 1][r], pk2(g, g), a);
                }
                return a;
              };
              const u64 n = terms(sum[k]);
              // what the sum lost of them, see exact_add2
              if constexpr (COMP) lo[k] = add2(lo[k], terms(sub2(sum[k], n)));
              sum[k] = n;
            }
          };
          if (m == 32) {
#pragma unroll 8
            for (int i = 0; i < 32; i += kSepAt) add(rec + i);
          } else {
#pragma unroll 1
            for (int i = 0; i < m; i += kSepAt) add(rec + i);
          }
        };
        using std::integral_constant;
        if (at_group + m <= first_end)
          group(integral_constant<int, 0>(), integral_constant<int, 4>());
        else if (at_group >= last_beg)
          group(integral_constant<int, 4>(), integral_constant<int, 8>());
        else
          group(integral_constant<int, 0>(), integral_constant<int, 8>());
      }
      if constexpr (COMP) {
#pragma unroll
        for (int k = 0; k < 8; ++k) sum[k] = sub2(sum[k], base);
      }
      bool bad = false;
      if constexpr (SHARE) {
        // cell (x, y) of warp w at part[w][16 y + x]
        __syncthreads();  // the previous block's partial sums were read
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          const float2 a = upk2(sum[k]);
          float2 l = make_float2(0.f, 0.f);
          if constexpr (COMP) l = upk2(lo[k]);
          part[warp * 256 + row(k) * 16 + 2 * c + (k & 1)] = make_float4(a.x, a.y, l.x, l.y);
        }
        __syncthreads();
        u64 sh = 0ull, sl = 0ull;
        for (int w = 0; w < kSepWarps; ++w) {
          const float4 t = part[w * 256 + tid];
          if constexpr (COMP) {
            u64 e;
            sh = two_sum2(sh, pk2(t.x, t.y), e);
            sl = add2(sl, add2(e, pk2(t.z, t.w)));
          } else {
            sh = add2(sh, pk2(t.x, t.y));
          }
        }
        const float2 z = upk2(fma2(sh, 0ull, 0ull));
        bad = __syncthreads_or(!(z.x == 0.f && z.y == 0.f));
        if (bad) sep_redo<COMP>(p, J, x0, y0, plane, gt, first, last, slot, tid, NT);
        else if (DENSE) sep_merge(slot + tid, upk2(sh), upk2(sl));
        else
          sep_store(J, x0 + (tid & 15), y0 + (tid >> 4), plane, p.P, p.accumulate, upk2(sh),
                    upk2(sl));
      } else {
        u64 z = 0ull;
#pragma unroll
        for (int k = 0; k < 8; ++k) z = fma2(sum[k], 0ull, z);
        const float2 zf = upk2(z);
        bad = __any_sync(0xffffffffu, !(zf.x == 0.f && zf.y == 0.f));
        if (!bad) {
#pragma unroll
          for (int k = 0; k < 8; ++k) {
            float2 l = make_float2(0.f, 0.f);
            if constexpr (COMP) l = upk2(lo[k]);
            const int x = 2 * c + (k & 1), y = row(k);
            if (DENSE) sep_merge(slot + y * kSepB + x, upk2(sum[k]), l);
            else sep_store(J, x0 + x, y0 + y, plane, p.P, p.accumulate, upk2(sum[k]), l);
          }
        } else {
          sep_redo<COMP>(p, J, x0, y0, plane, gt, first, last, slot, lane, 32);
        }
      }
    }
    if constexpr (DENSE) {
      // the last of a dense block's units stores the merged sums
      __threadfence();
      if constexpr (SHARE) __syncthreads();
      int done = 0;
      if (leader) done = atomicAdd(&p.dense[entry].w, 1) + 1;
      if (share(done) == p.dense[entry].z) {
        __threadfence();
        const double2 *const from = p.slots + (size_t)entry * p.P * (kSepB * kSepB);
        for (int i = SHARE ? tid : lane; i < p.P * kSepB * kSepB; i += SHARE ? NT : 32) {
          const double2 v = __ldcg(from + i);
          const int plane = i / (kSepB * kSepB), x = x0 + i % kSepB, y = y0 + i / kSepB % kSepB;
          if (x >= J.N || y >= J.N || (p.accumulate && v.x == 0.0 && v.y == 0.0)) continue;
          const size_t cell = (size_t)y * J.N + x;
          if (J.out_f64) sep_store_f64(J, cell, plane, p.P, p.accumulate, v.x, v.y);
          else sep_store_f32(J, cell, plane, p.P, p.accumulate, (float)v.x, (float)v.y);
        }
      }
    }
    if (DENSE && !advance()) return;
  }
}

template <bool COMP, bool SHARE, bool DENSE>
cudaError_t sep_launch(const SepTileLaunch &g, cudaStream_t s) {
  const size_t smem = sep_factor_floats(g.G) * 4 + kSepWarps * kSepStage * sizeof(float4) +
                      (SHARE ? kSepWarps * 256 * sizeof(float4) : 0);
  auto kern = septile_kernel<COMP, SHARE, DENSE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, 32 * kSepWarps, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const int64_t most = DENSE ? INT_MAX : (g.total_blocks + g.chunk - 1) / g.chunk;
  const int64_t blocks = std::min<int64_t>((int64_t)g.sm_count * per_sm, most);
  count_launch();
  return launch_overlapped(kern, (unsigned)blocks, 32 * kSepWarps, smem, s, g.overlap, g);
}

// Units of dense blocks first.  One kernel for both took 9 % longer where no block is
// dense (1.05 M uniform visibilities on 4096^2, 668 and 614 us).
template <bool COMP, bool SHARE> cudaError_t sep_launches(const SepTileLaunch &g, cudaStream_t s) {
  const cudaError_t e = sep_launch<COMP, SHARE, true>(g, s);
  return e != cudaSuccess ? e : sep_launch<COMP, SHARE, false>(g, s);
}

}  // namespace

cudaError_t launch_septile(const SepTileLaunch &launch, cudaStream_t s) {
  SepTileLaunch g = launch;
  if (g.total_blocks < 1) return cudaSuccess;
  // a block a warp while that gives every resident warp a few blocks
  const bool share = g.compensated && g.total_blocks < (int64_t)g.sm_count * 24 * 4;
  g.dense_unit = share ? 4096 : 512;
  g.dense_min = share ? std::max(2 * 4096, 8 * septile_dense_min(g.vis, g.sm_count))
                      : septile_dense_min(g.vis, g.sm_count);
  count_launch();
  // Blocks claimed one by one go to different SMs at the same time and share
  // their records in L2; where blocks have a few records each and most none,
  // eight at once.
  g.chunk = !share && 9 * g.vis < 16 * (int64_t)g.total_blocks ? 8 : 1;
  const cudaError_t e = launch_overlapped(sep_plan_kernel, (unsigned)((g.total_blocks + 31) / 32),
                                          256, 0, s, g.overlap, g);
  if (e != cudaSuccess) return e;
  return !g.compensated ? sep_launches<false, false>(g, s)
         : share        ? sep_launches<true, true>(g, s)
                        : sep_launches<true, false>(g, s);
}

}  // namespace gg
