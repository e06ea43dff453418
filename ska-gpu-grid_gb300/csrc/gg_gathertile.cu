// Gather gridding by 16x16 output block, FP32 values and supports 8 and 16 (the
// reference's GATHER method, grid_kernel_gather, grid_gpu.cu:391-503): every
// cell is summed in a register of the one lane that owns it and stored once --
// no atomics, no cleared grid.
//
// A warp owns a block; lane (c, h) holds its columns c, c + 8 and its rows
// 4h .. 4h+3.  The visibilities that reach the block have their main cells in
// 4x4 uv tiles of 8 cells, 4 contiguous ranges of the sorted records.  They are
// tested 32 at a time, one per lane, and those whose footprint meets the block
// are put in a shared buffer that every lane then reads as broadcasts.  (The
// 32-cell tile kernel had each of 8 warps test every record of 9 tiles and
// visited what it kept with a quarter of its lanes at work.)
//
//  * Table without imaginary parts: its real parts in shared memory, every
//    sub-kernel behind 15 rows of zeros, so the four rows of a lane are read
//    at fixed offsets and rows outside the footprint read zero; columns outside
//    get the value replaced by zero.  The row length puts the four row groups
//    that a warp reads in distinct banks.
//  * With imaginary parts: complex entries, no zeros (they would not fit for
//    support 16); rows outside get the value replaced by zero too.
//  * A block whose sums are not finite is summed again cell by cell, only from
//    the records whose footprints cover the cell (zero times a value or entry
//    that is not finite would spread).
//  * Compensated sums: runs of at most kGtRun records are summed plainly, then
//    added into (hi, lo) by TwoSum.
//  * Few blocks (small grids): the warps of a CTA share a block and add their
//    (hi, lo) sums by TwoSum in shared memory.
//
// Bound by instruction issue (76 % of active cycles; 54 % of the FMA pipe's and of
// the shared-memory wavefronts).  1.05 M visibilities of support 8 on 4096^2, whole call: 858 us
// by 32-cell tiles, 251 now.
#include <algorithm>

#include "gg_kernels.cuh"

namespace gg {

namespace {

constexpr int kGtB = kGatBlock;  // block side
constexpr int kGtWarps = 16;
// records summed plainly.  Errors against 64 bits with 16 / 8 / 4, where gather_kernel
// has 5.7e-8, 6.0e-8 and 7.3e-8: 1 M random ones of support 8 on 800^2 6.2e-8 /
// 5.0e-8 / 4.3e-8, on 200^2 6.4e-8 / 5.1e-8 / 4.3e-8, 1.05 M of tracks on 4096^2
// 6.4e-8 / 5.4e-8 / 4.6e-8 (whole calls of that 221 / 251 / 318 us).
constexpr int kGtRun = 8;
constexpr int kGtStage = 36;  // a group of 32 and zeros for the read-ahead

template <int S> struct GtCfg {
  // real parts: rows of ROW floats, 15 rows of zeros before each sub-kernel
  // (and behind the last)
  static constexpr int ROW = S + 2;
  static constexpr int ROWS = S + 15;
  static constexpr int PADX = 16;  // floats before and behind: columns outside
};
__host__ __device__ constexpr size_t gt_real_floats(int S, int G) {
  return (size_t)(G * G * (S + 15) + 15) * (S + 2) + 2 * 16;
}
__host__ __device__ constexpr size_t gt_table_bytes(int S, int G) {
  const size_t re = gt_real_floats(S, G) * 4, cx = (size_t)G * G * S * S * 8;
  return ((re > cx ? re : cx) + 15) & ~(size_t)15;
}

template <int OFF> __device__ __forceinline__ float lds(uint32_t a) {
  float v;
  asm("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
  return v;
}
template <int OFF> __device__ __forceinline__ float2 lds2(uint32_t a) {
  float2 v;
  asm("ld.shared.v2.f32 {%0, %1}, [%2+%3];" : "=f"(v.x), "=f"(v.y) : "r"(a), "n"(OFF));
  return v;
}
template <int I, int N, class F> __device__ __forceinline__ void gt_for(F &&f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    gt_for<I + 1, N>(f);
  }
}

__device__ __noinline__ void gt_store_f64(const JobDesc &J, size_t cell, int plane, int P,
                                          bool accumulate, const float2 h, const float2 l) {
  const size_t NN = (size_t)J.N * J.N;
  const double dr = (double)h.x + (double)l.x, di = (double)h.y + (double)l.y;
  if (!accumulate)
    grid_store<double>((double *)J.out, cell, plane, P, NN, J.planar, dr, di);
  else if (J.out_f64)  // into the present value, rounded once
    grid_add<double>((double *)J.out, cell, plane, P, NN, J.planar, dr, di);
  else
    grid_add<float>((float *)J.out, cell, plane, P, NN, J.planar, dr, di);
}

// (hi, lo) into a cell of the grid
__device__ __forceinline__ void gt_store(const JobDesc &J, int gx, int gy, int plane, int P,
                                         bool accumulate, const float2 h, const float2 l) {
  if (gx >= J.N || gy >= J.N) return;
  const size_t cell = (size_t)gy * J.N + gx, NN = (size_t)J.N * J.N;
  // FP64 sums only where the grid or its present value needs them: the FP64
  // pipe is so narrow that adding every cell in it took half of the kernel's
  // time (284 -> 212 us with the ranges joined into one list)
  if (accumulate || J.out_f64) {
    gt_store_f64(J, cell, plane, P, accumulate, h, l);
  } else {
    const float2 v = make_float2(__fadd_rn(h.x, l.x), __fadd_rn(h.y, l.y));
    if (J.planar) grid_store<float>((float *)J.out, cell, plane, P, NN, true, v.x, v.y);
    else reinterpret_cast<float2 *>(J.out)[plane * NN + cell] = v;
  }
}

// sorted record k and its value in a plane
__device__ __forceinline__ void gt_record(const GatherTileLaunch &p, int k, int plane, int2 &q,
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

// entry (a, b) of a sub-kernel
template <int S>
__device__ __forceinline__ float2 gt_entry(const unsigned char *table, bool cplx, int sub, int a,
                                           int b) {
  using C = GtCfg<S>;
  if (cplx) return reinterpret_cast<const float2 *>(table)[(sub * S + b) * S + a];
  const float *t = reinterpret_cast<const float *>(table);
  return make_float2(t[(sub * C::ROWS + 15 + b) * C::ROW + C::PADX + a], 0.f);
}

template <int S, bool COMP>
__device__ __noinline__ void gt_redo(const GatherTileLaunch &p, const JobDesc &J, int x0, int y0,
                                     int plane, const unsigned char *table, bool cplx, int tid,
                                     int nt) {
  for (int c = tid; c < kGtB * kGtB; c += nt) {
    const int x = x0 + c % kGtB, y = y0 + c / kGtB;
    u64 run = 0ull, hi = 0ull, lo = 0ull;
    int since = 0;
    auto merge = [&]() {
      u64 e;
      hi = two_sum2(hi, run, e);
      lo = add2(lo, e);
      run = 0ull;
      since = 0;
    };
    const int bx = x0 / kRegTile, by = y0 / kRegTile;
    for (int r = 0; r < 4 && by + r < J.ntx; ++r) {
      const int *const bm = J.bookmarks + (by + r) * J.ntx;
      for (int k = bm[bx]; k < bm[min(bx + 4, J.ntx)]; ++k) {
        int2 q;
        float2 v;
        gt_record(p, k, plane, q, v);
        const int a = x - ((int)((unsigned)q.x & 0xffffu) - kWinMainBias - S / 2 + 1);
        const int b = y - ((int)((unsigned)q.x >> 16) - kWinMainBias - S / 2 + 1);
        if ((unsigned)a >= (unsigned)S || (unsigned)b >= (unsigned)S) continue;
        const float2 g = gt_entry<S>(table, cplx, q.y, a, b);
        run = fma2(pk2(v.x, v.y), pk2(g.x, g.x), run);
        if (cplx) run = fma2(pk2(-v.y, v.x), pk2(g.y, g.y), run);
        if (COMP && ++since == kGtRun) merge();
      }
    }
    if (COMP) merge();
    gt_store(J, x, y, plane, p.P, p.accumulate, upk2(COMP ? hi : run), upk2(lo));
  }
}

// the CTA's blocks, for a table with (CX) or without imaginary parts
template <int S, bool COMP, bool SHARE, bool CX>
__device__ __forceinline__ void gt_blocks(const GatherTileLaunch &p, unsigned char *smem) {
  using C = GtCfg<S>;
  constexpr int H = S / 2, NT = 32 * kGtWarps;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  unsigned char *const after = smem + gt_table_bytes(S, p.G);
  // footprint places and sub-kernels, and values, of a group and the zeros
  // behind it
  int2 *const off = reinterpret_cast<int2 *>(after) + warp * kGtStage;
  float2 *const val = reinterpret_cast<float2 *>(after) + (kGtWarps + warp) * kGtStage;
  float4 *const part = reinterpret_cast<float4 *>(after + 16 * kGtWarps * kGtStage);
  const int c = lane & 7, h = lane >> 3;
  // a lane's first entry, seen from the block's first cell
  const uint32_t mine = smem_addr(smem) +
                        (CX ? 8 * (4 * h * S + c) : 4 * ((15 + 4 * h) * C::ROW + C::PADX + c));
  const int workers = SHARE ? (int)gridDim.x : (int)gridDim.x * kGtWarps;
  int blk = SHARE ? (int)blockIdx.x : (int)(blockIdx.x + warp * gridDim.x);
  __shared__ int s_next;
  while (blk < p.total_blocks) {
    int next = 0;
    if (SHARE ? tid == 0 : lane == 0) next = atomicAdd(p.next, 1) + workers;
    int j = 0;
    {
      int e = p.njobs - 1;
      while (j < e) {
        const int mid = (j + e + 1) >> 1;
        if (p.jobs[mid].blk0 <= blk) j = mid; else e = mid - 1;
      }
    }
    const JobDesc &J = p.jobs[j];
    const int nb = (J.N + kGtB - 1) / kGtB, b = blk - J.blk0;
    const int x0 = (b % nb) * kGtB, y0 = (b / nb) * kGtB;
    const int bx = x0 / kRegTile, by = y0 / kRegTile;  // tiles start kRegOff before the grid
    // lane r < 4: the r-th row of tiles
    int beg = 0, end = 0;
    if (lane < 4 && by + lane < J.ntx) {
      const int *const bm = J.bookmarks + (by + lane) * J.ntx;
      beg = bm[bx];
      end = bm[min(bx + 4, J.ntx)];
    }
    // the ranges as one list: record t of it is record t + shift[r] of the
    // sorted ones, r the last range with start[r] <= t
    int sum = end - beg;
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += y;
    }
    int start[4], shift[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      start[r] = __shfl_sync(0xffffffffu, sum - (end - beg), r);
      shift[r] = __shfl_sync(0xffffffffu, beg, r) - start[r];
    }
    const int records = __shfl_sync(0xffffffffu, sum, 3), groups = (records + 31) / 32;
    for (int plane = 0; plane < p.P; ++plane) {
      // cell (u, k): column c + 8u, row 4h + k
      u64 run[2][4], hi[COMP ? 2 : 1][4], lo[COMP ? 2 : 1][4];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
          run[u][k] = 0ull;
          if constexpr (COMP) hi[u][k] = lo[u][k] = 0ull;
        }
      int since = 0;  // records in the running sums
      auto merge = [&]() {
        if constexpr (COMP) {
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              u64 e;
              hi[u][k] = two_sum2(hi[u][k], run[u][k], e);
              lo[u][k] = add2(lo[u][k], e);
              run[u][k] = 0ull;
            }
        }
        since = 0;
      };
      int2 q = make_int2(0, 0);
      float2 v = make_float2(0.f, 0.f);
      bool have = false;
      auto fetch = [&](int g) {
        have = false;
        const int t = 32 * g + lane;
        have = t < records;
        int k = t + shift[0];
#pragma unroll
        for (int r = 1; r < 4; ++r)
          if (t >= start[r]) k = t + shift[r];
        if (have) gt_record(p, k, plane, q, v);
      };
      for (int g = SHARE ? warp : 0; g < groups; g += SHARE ? kGtWarps : 1) {
        if (g == (SHARE ? warp : 0)) fetch(g);
        // keep the records whose footprints meet the block
        const int fx = (int)((unsigned)q.x & 0xffffu) - kWinMainBias - H + 1 - x0;
        const int fy = (int)((unsigned)q.x >> 16) - kWinMainBias - H + 1 - y0;
        const bool keep = have && fx < kGtB && fx + S > 0 && fy < kGtB && fy + S > 0;
        const unsigned kept = __ballot_sync(0xffffffffu, keep);
        const int m = __popc(kept);
        __syncwarp();  // the previous group was read
        if (keep) {
          const int at = __popc(kept & ((1u << lane) - 1));
          // byte offset of the entry under the block's first cell, and fx, fy
          // (-15..15, biased)
          const int e = CX ? 8 * ((q.y * S - fy) * S - fx)
                           : 4 * ((q.y * C::ROWS - fy) * C::ROW - fx);
          off[at] = make_int2(e, (fx + 16) | (fy + 16) << 8);
          val[at] = v;
        }
        if (lane < 4) {  // read ahead: no footprint, no value
          off[m + lane] = make_int2(0, 16 | 16 << 8);
          val[m + lane] = make_float2(0.f, 0.f);
        }
        fetch(g + (SHARE ? kGtWarps : 1));
        __syncwarp();
        // the entries of a record are loaded while the previous one is added
        struct Taps {
          float g[2][4], h[CX ? 2 : 1][4];
          float2 v;
          bool in[2], row[CX ? 4 : 1];
        } a, b;
        auto load = [&](Taps &t, const int2 o, int i) {
          t.v = val[i];
          const int ox = (o.y & 0xff) - 16, oy = (o.y >> 8) - 16;
#pragma unroll
          for (int u = 0; u < 2; ++u) t.in[u] = (unsigned)(c + 8 * u - ox) < (unsigned)S;
          const uint32_t e = mine + (uint32_t)o.x;
          if constexpr (CX) {
#pragma unroll
            for (int k = 0; k < 4; ++k) t.row[k] = (unsigned)(4 * h + k - oy) < (unsigned)S;
          }
          gt_for<0, 4>([&](auto K) {
            constexpr int k = decltype(K)::value;
            gt_for<0, 2>([&](auto U) {
              constexpr int u = decltype(U)::value;
              if constexpr (CX) {
                // entries outside the sub-kernel may lie outside the table
                float2 w = make_float2(0.f, 0.f);
                if (t.in[u] && t.row[k]) w = lds2<8 * (k * S + 8 * u)>(e);
                t.g[u][k] = w.x;
                t.h[u][k] = w.y;
              } else {
                t.g[u][k] = lds<4 * (k * C::ROW + 8 * u)>(e);
              }
            });
          });
        };
        auto add = [&](const Taps &t) {
#pragma unroll
          for (int u = 0; u < 2; ++u) {
            const u64 w = t.in[u] ? pk2(t.v.x, t.v.y) : 0ull;
#pragma unroll
            for (int k = 0; k < 4; ++k) run[u][k] = fma2(w, pk2(t.g[u][k], t.g[u][k]), run[u][k]);
            if constexpr (CX) {
              const u64 z = t.in[u] ? pk2(-t.v.y, t.v.x) : 0ull;
#pragma unroll
              for (int k = 0; k < 4; ++k)
                run[u][k] = fma2(z, pk2(t.h[u][k], t.h[u][k]), run[u][k]);
            }
          }
        };
        load(a, off[0], 0);
        int2 o = off[1];
        for (int i0 = 0; i0 < m; i0 += kGtRun) {
          const int i1 = min(m, i0 + kGtRun);
          if (since + i1 - i0 > kGtRun) merge();
#pragma unroll 1
          for (int i = i0; i < i1; i += 2) {
            load(b, o, i + 1);
            o = off[i + 2];
            add(a);
            load(a, o, i + 2);
            o = off[i + 3];
            add(b);
          }
          since += i1 - i0;
        }
      }
      merge();
      if constexpr (SHARE) {
        // cell (x, y) of warp w at part[w][16 y + x]
        __syncthreads();  // the previous block's partial sums were read
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            const float2 s = upk2(COMP ? hi[u][k] : run[u][k]);
            float2 l = make_float2(0.f, 0.f);
            if constexpr (COMP) l = upk2(lo[u][k]);
            part[warp * 256 + (4 * h + k) * 16 + c + 8 * u] = make_float4(s.x, s.y, l.x, l.y);
          }
        __syncthreads();
        u64 sh = 0ull, sl = 0ull;
        if (tid < 256)
          for (int w = 0; w < kGtWarps; ++w) {
            const float4 t = part[w * 256 + tid];
            u64 e;
            sh = two_sum2(sh, pk2(t.x, t.y), e);
            sl = add2(sl, add2(e, pk2(t.z, t.w)));
          }
        const float2 z = upk2(fma2(sh, 0ull, 0ull));
        if (!__syncthreads_or(!(z.x == 0.f && z.y == 0.f))) {
          if (tid < 256)
            gt_store(J, x0 + (tid & 15), y0 + (tid >> 4), plane, p.P, p.accumulate, upk2(sh),
                     upk2(sl));
        } else {
          gt_redo<S, COMP>(p, J, x0, y0, plane, smem, CX, tid, NT);
        }
      } else {
        u64 z = 0ull;
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
          for (int k = 0; k < 4; ++k) {
            if constexpr (COMP) z = fma2(hi[u][k], 0ull, z);
            else z = fma2(run[u][k], 0ull, z);
          }
        const float2 zf = upk2(z);
        if (!__any_sync(0xffffffffu, !(zf.x == 0.f && zf.y == 0.f))) {
#pragma unroll
          for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
              float2 l = make_float2(0.f, 0.f);
              if constexpr (COMP) l = upk2(lo[u][k]);
              gt_store(J, x0 + c + 8 * u, y0 + 4 * h + k, plane, p.P, p.accumulate,
                       upk2(COMP ? hi[u][k] : run[u][k]), l);
            }
        } else {
          gt_redo<S, COMP>(p, J, x0, y0, plane, smem, CX, lane, 32);
        }
      }
    }
    if constexpr (SHARE) {
      if (tid == 0) s_next = next;
      __syncthreads();
      blk = s_next;
      __syncthreads();
    } else {
      blk = __shfl_sync(0xffffffffu, next, 0);
    }
  }
}

template <int S, bool COMP, bool SHARE>
__global__ void __launch_bounds__(32 * kGtWarps, 1)
    gathertile_kernel(const __grid_constant__ GatherTileLaunch p) {
  using C = GtCfg<S>;
  constexpr int NT = 32 * kGtWarps;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x, n = p.G * p.G * S * S;
  float *const re = reinterpret_cast<float *>(smem);
  int imag = 0;
  if (!p.overlap) after_predecessor();
  float *const g1 = reinterpret_cast<float *>(smem + gt_table_bytes(S, p.G));
  if (p.gauss) {
    gauss_fill(g1, S, p.G, p.sigma, tid, NT);
  } else {
#pragma unroll 4
    for (int i = tid; i < n; i += NT) imag |= __ldg(p.gcf + i).y != 0.f;
  }
  const bool cplx = __syncthreads_or(imag);
  if (cplx) {
    for (int i = tid; i < n; i += NT) reinterpret_cast<float2 *>(smem)[i] = __ldg(p.gcf + i);
  } else {
    const int nf = (int)gt_real_floats(S, p.G);
    for (int i = tid; i < nf; i += NT) {
      const int e = i - C::PADX, row = e / C::ROW, a = e - row * C::ROW;
      const int sub = row / C::ROWS, b = row % C::ROWS - 15;
      float g = 0.f;
      if (e >= 0 && a < S && b >= 0 && sub < p.G * p.G) {
        if (p.gauss) {
          const int sy = sub / p.G, sx = sub - sy * p.G;
          g = g1[sx * S + a] * g1[sy * S + b];
        } else {
          g = __ldg(p.gcf + (sub * S + b) * S + a).x;
        }
      }
      re[i] = g;
    }
  }
  if (p.overlap) after_predecessor();
  __syncthreads();
  // zeros behind the staged groups are written with each group
  if (cplx) gt_blocks<S, COMP, SHARE, true>(p, smem);
  else gt_blocks<S, COMP, SHARE, false>(p, smem);
}

size_t gt_smem(int S, int G, bool share) {
  return gt_table_bytes(S, G) + 16 * kGtWarps * kGtStage + (share ? kGtWarps * 256 * 16 : 0);
}

template <int S, bool COMP, bool SHARE>
cudaError_t gt_launch(const GatherTileLaunch &g, cudaStream_t s) {
  const size_t smem = gt_smem(S, g.G, SHARE);
  auto kern = gathertile_kernel<S, COMP, SHARE>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  const int blocks = std::min(g.sm_count, g.total_blocks);
  if (blocks < 1) return cudaSuccess;
  count_launch();
  return launch_overlapped(kern, (unsigned)blocks, 32 * kGtWarps, smem, s, g.overlap, g);
}

}  // namespace

size_t gathertile_smem_bytes(int S, int G) { return gt_smem(S, G, true); }

cudaError_t launch_gathertile(const GatherTileLaunch &g, cudaStream_t s) {
  // plain sums stay one sequence of additions
  const bool share = g.compensated && g.total_blocks < g.sm_count * kGtWarps * 2;
#define GG_GT(SV)                                                                         \
  return g.compensated ? (share ? gt_launch<SV, true, true>(g, s)                         \
                                : gt_launch<SV, true, false>(g, s))                       \
                       : gt_launch<SV, false, false>(g, s)
  switch (g.S) {
    case 8: GG_GT(8);
    case 16: GG_GT(16);
  }
#undef GG_GT
  return cudaErrorInvalidValue;
}

}  // namespace gg
