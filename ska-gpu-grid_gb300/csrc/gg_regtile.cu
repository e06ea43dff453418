// Moving-window gridding with the sub-grid of an 8-cell uv tile held in
// registers (the reference's MOVING_WINDOW method, grid_kernel_window,
// grid_gpu.cu:504-673, for FP32 values and supports 8 and 16).
//
// The visibilities of one 8x8 tile touch an R x R sub-grid, R = S + 7: 15x15
// or 23x23 cells.  A warp takes a work item (a slice of a tile's sorted
// records) and owns every cell of it: lane (lx, ly) of an LX x LY arrangement
// holds the cells x = LX i + lx, y = LY j + ly, 8 cells for support 8 and 18
// for support 16.  No cell ever moves, so a record costs its table loads and
// its multiply-adds whether or not it moves the footprint: the shared-memory
// sub-grid of window_kernel costs a read-modify-write of every tap at each
// move, and on uv tracks most records move.
//
//  * Rows.  A footprint of S rows starting at fy in 0..7 covers, of the S + 8
//    rows a lane owns, exactly S / LY: the rows j in [8/LY, S/LY) always, and
//    of each pair (j, j + S/LY), j < 8/LY, the first when fy <= LY j + ly and
//    the second otherwise.  The records of a block are therefore put in order
//    of fy (a counting sort of up to kRtBlock records in shared memory): while
//    fy stays the same a lane adds to one cell of each pair, and the two change
//    places when fy passes their row (plain sums: a running sum goes to the
//    right cell when fy changes).
//  * Columns.  Support 8: table rows sit behind eight zeros in shared memory,
//    so the four columns of a lane are read at fixed offsets and those outside
//    the footprint read zero.  Support 16, whose table reads would bind: of
//    its three columns the middle one is always inside and the outer two are
//    complementary, so they share one load, and one of them gets the value
//    replaced by zero.  The row length puts the LY rows that a warp reads in
//    distinct banks.
//  * Products by zero turn a value (or table entry) that is not finite into
//    NaN in cells its footprint does not cover.  A sub-grid that is not finite
//    at the end of its item is therefore summed again cell by cell, only
//    inside footprints.
//  * Compensated sums: every cell's sum starts at a power of two and a half so
//    large that the item's terms do not lead out of its binade, which makes
//    what an addition rounds off exact to work out (exact_add2): three packed
//    operations a term, taken two at a time, where a TwoSum of each takes eight.
//    No term is ever added to another plainly.  Runs of 16 summed plainly
//    between TwoSums, as it was, take one and a half, but made the error of
//    the sums larger than window_kernel's (in the listed sizes below up to 1.3
//    times; now 0.54 to 0.87 times).
//  * The records of a block are fetched while the previous block (also of the
//    previous plane or item) is summed.
//  * Real and imaginary parts of the table are kept apart; an item of a table
//    without imaginary parts never touches the second half.
//
// The whole table lives in each CTA's shared memory (2 x 98 KB for support 16
// at oversampling 8), hence one CTA per SM and one table per launch.  Several
// tables, or one that does not fit, are read from global memory by
// regtile_tables_kernel, complex entries as the caller keeps them, their
// imaginary parts only if any table of the class has some (1.05 M records of
// support 16 and 16 real tables on 2048^2: 372 us, as complex ones 421,
// window_kernel 420; what the tables are like costs 5 us to find out).  There the
// planes of an item are units of their own, next to each other, and the warps
// that sum them keep in step (where their number divides the CTA's warps), so
// that all but the first find a record's sub-kernel (2 KB for support 16) in L1.
// 524 k records of 4 planes and 32 tables of support 16 on 2048^2, whole call,
// and error against 64 bits: window_kernel 878 us, 9.2e-8; plain runs of 16 735,
// 1.2e-7; now 825, 8.0e-8 (with 12 warps a CTA instead of 8, whose registers
// spill, 910; two records at once 850).
//
// Bound by the FMA pipe, its latency and issue: 256 mixed jobs, support 8 / 16, 54 % of
// the pipe's cycles and 65 / 61 % of the issue slots, with 12 warps an SM for
// support 16 (8 warps without spills: the same for large jobs, 93 instead of 78 us
// for 100 k records on 777^2; 16 of 128 registers: 5 % slower; four records at once:
// 3.5 % faster, but in random order less exact than window_kernel).  Whole calls
// against window_kernel, us, and errors against 64 bits:
//   4.19 M records of support 8 on 4096^2     576 -> 369   5.4e-8 -> 4.6e-8
//   10 k of support 8 on 256^2                 86 -> 32    8.0e-8 -> 4.2e-8
//   100 k of support 16 on 777^2              125 -> 79    7.3e-8 -> 5.3e-8
//   256 mixed jobs, 45 M records             6491 -> 5327  7.8e-8 -> 5.6e-8
// (plain runs of 16: 356, 32, 68 and 4429 us with 7.1e-8, 7.5e-8, 9.1e-8, 9.0e-8).
#include <algorithm>

#include "gg_kernels.cuh"

namespace gg {

namespace {

// records between barriers of the warps that keep in step, and the most that
// are summed in a plain run (GG_ACC_PLAIN)
constexpr int kRtRun = 16;
// records sorted together: four per lane
constexpr int kRtBlock = 128;
// staged records: every fy's share is padded to an even number, and two more
// are read ahead
constexpr int kRtStage = kRtBlock + 8 + 2;

// GT: tables read from global memory (complex entries as the caller has them)
template <int S, bool GT> struct RtCfg {
  static constexpr int LX = S == 8 && !GT ? 4 : 8, LY = 32 / LX;
  static constexpr int NX = (S + 8) / LX, NY = (S + 8) / LY, R = S + kRegTile - 1;
  static constexpr int Q = S / LY;      // rows of a footprint per lane
  static constexpr int PAIRS = 8 / LY;  // rows j < PAIRS alternate with j + Q
  // columns behind zeros (every column loaded), or a shared load of the first
  // and last column, which are complementary
  static constexpr bool PADX = S == 8 && !GT;
  static constexpr int NL = PADX ? NX : NX - 1;  // loads per row
  static constexpr int WARPS = S == 8 ? 16 : GT ? 8 : 12;
  static constexpr int ENTRY = GT ? 8 : 4;    // bytes of a table entry
  static constexpr int ROW = GT ? 8 * S : regtile_row(S);  // of a table row
  static constexpr int PAD = GT ? 0 : regtile_pad(S);      // before its first tap
  static constexpr int SUB = S * ROW;
};

// floats of one table (a row behind the last: the zeros after its taps)
__host__ __device__ constexpr int rt_table_floats(int S, int G) {
  return (G * G * S + 1) * (regtile_row(S) / 4);
}

template <int OFF> __device__ __forceinline__ float lds(uint32_t a) {
  float v;
  asm("ld.shared.f32 %0, [%1+%2];" : "=f"(v) : "r"(a), "n"(OFF));
  return v;
}

// compile-time loop
template <int I, int N, class F> __device__ __forceinline__ void rt_for(F &&f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>{});
    rt_for<I + 1, N>(f);
  }
}

// sorted record k and its value in a plane
__device__ __forceinline__ void rt_record(const RegTileLaunch &p, int k, int plane, int2 &q,
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

// the table of a bin (uv tile * n_gcf + table)
template <int S> __device__ __forceinline__ const float2 *rt_table(const JobDesc &J, int bin) {
  return reinterpret_cast<const float2 *>(J.gcf) +
         (size_t)(J.n_gcf > 1 ? bin % J.n_gcf : 0) * J.G * J.G * S * S;
}

__device__ __forceinline__ TableInfo rt_info(const JobDesc &J, int bin) {
  return J.gcf_info[J.n_gcf > 1 ? bin % J.n_gcf : 0];
}

// The sub-grid of an item whose packed sums are not finite, cell by cell and
// only from the records whose footprints cover the cell.
template <int S, bool COMP, bool GT>
__device__ __noinline__ void rt_redo(const RegTileLaunch &p, const WorkItem &w, int plane,
                                     const float *tr, bool cplx, double2 *slot) {
  using C = RtCfg<S, GT>;
  constexpr int R = C::R;
  const JobDesc &J = p.jobs[w.job];
  const float *const ti = tr + rt_table_floats(S, p.G);
  const float2 *const gt = rt_table<S>(J, w.bin);
  for (int c = threadIdx.x & 31; c < R * R; c += 32) {
    const int x = c % R, y = c / R;
    const int gx = w.ox + x, gy = w.oy + y;
    if ((unsigned)gx >= (unsigned)J.N || (unsigned)gy >= (unsigned)J.N) continue;
    u64 run = 0ull, hi = 0ull, lo = 0ull;
    auto merge = [&]() {
      u64 e;
      hi = two_sum2(hi, run, e);
      lo = add2(lo, e);
      run = 0ull;
    };
    for (int k = w.start; k < w.end; ++k) {
      int2 q;
      float2 v;
      rt_record(p, k, plane, q, v);
      const int fy = q.y & 0xff;
      const int fx = C::PADX ? (-(q.x + fy * C::ROW - C::PAD) & 31) >> 2 : q.y >> 8;
      if ((unsigned)(x - fx) >= (unsigned)S || (unsigned)(y - fy) >= (unsigned)S) continue;
      const int at = (q.x + y * C::ROW) / C::ENTRY + x;
      float2 g;
      if constexpr (GT) g = __ldg(gt + at);
      else g = make_float2(tr[at], cplx ? ti[at] : 0.f);
      run = fma2(pk2(v.x, v.y), pk2(g.x, g.x), run);
      if (cplx) run = fma2(pk2(-v.y, v.x), pk2(g.y, g.y), run);
      if (COMP) merge();
    }
    const float2 h = upk2(COMP ? hi : run), l = upk2(lo);
    if (slot) {
      red_add(&slot[c].x, (double)h.x + (double)l.x);
      red_add(&slot[c].y, (double)h.y + (double)l.y);
    } else if (J.out_f64) {
      out_red(J, (size_t)gy * J.N + gx, plane, p.P, (double)h.x + (double)l.x,
              (double)h.y + (double)l.y);
    } else {
      out_red(J, (size_t)gy * J.N + gx, plane, p.P, (double)__fadd_rn(h.x, l.x),
              (double)__fadd_rn(h.y, l.y));
    }
  }
}

// A warp's share of the launch's units: one plane of an item each, the planes
// of an item next to each other (they read the same records and table rows).
// GT: CX says whether any table of the class has imaginary parts (the products of
// a table without them are then complex too, with the same finite sums: a choice
// for every item cost 4 to 13 %).  cplx: whether the launch's table has, or CX.
template <int S, bool COMP, bool GT, bool CX>
__device__ __forceinline__ void rt_items(const RegTileLaunch &p, const float *tr, float4 *stage,
                                         bool cplx, float gmax) {
  using C = RtCfg<S, GT>;
  constexpr int LX = C::LX, LY = C::LY, NX = C::NX, NY = C::NY, R = C::R, Q = C::Q,
                PAIRS = C::PAIRS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int lx = lane % LX, ly = lane / LX;
  const uint32_t tab = smem_addr(tr) + lx * 4 + ly * C::ROW;
  const uint32_t im_off = 4u * rt_table_floats(S, p.G);
  const int P = p.P, total = *p.nitems * P;
  const int first = gridDim.x * C::WARPS;
  // GT: the warps that sum the planes of an item keep in step (a barrier every
  // few records), so that one of them finds in L1 what another has loaded
  const bool grouped = GT && P > 1 && C::WARPS % P == 0;
  const int group = grouped ? warp / P : 0, member = grouped ? warp - group * P : 0;
  auto in_step = [&]() {
    if (grouped) asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "r"(32 * P) : "memory");
  };

  // The first units are spread over the SMs (the planes of an item stay
  // together); later ones are claimed ahead: while a unit is summed, the range
  // of the next is in registers and its first records, the range of the one
  // after and a further claim are on their way.
  int unit = P == 1 ? blockIdx.x + warp * gridDim.x : blockIdx.x * C::WARPS + warp;
  // of a group, the first warp claims an item
  __shared__ int s_claim[GT ? C::WARPS : 1];
  auto claim_one = [&]() {
    if (grouped) return lane == 0 && member == 0 ? (atomicAdd(p.item_next, 1) * P + first) : 0;
    return lane == 0 ? atomicAdd(p.item_next, 1) + first : 0;
  };
  auto claimed = [&](int c) {
    if (!grouped) return __shfl_sync(0xffffffffu, c, 0);
    if (lane == 0 && member == 0) s_claim[group] = c;
    in_step();
    c = s_claim[group] + member;
    in_step();  // all have read it
    return c;
  };
  auto range = [&](int it) {
    return it < total ? *reinterpret_cast<const int4 *>(p.items + (P == 1 ? it : it / P))
                      : make_int4(0, 0, 0, 0);
  };
  constexpr int PER = kRtBlock / 32;
  int2 pk[PER];
  float2 pv[PER];
  auto fetch = [&](int k0, int end, int plane) {
#pragma unroll
    for (int u = 0; u < PER; ++u) {
      const int k = k0 + u * 32 + lane;
      if (k < end) rt_record(p, k, plane, pk[u], pv[u]);
    }
  };
  if (unit >= total) return;  // the whole warp; no barrier follows
  int claim = claim_one();
  int4 cur = range(unit);  // {job, bin, start, end}
  fetch(cur.z, cur.w, P == 1 ? 0 : unit % P);
  int next = claimed(claim);
  claim = claim_one();
  int4 nxt = range(next);
  while (true) {
    const int next2 = claimed(claim);
    claim = claim_one();
    const int4 nxt2 = range(next2);
    const int item = P == 1 ? unit : unit / P, plane = unit - item * P;
    const int4 tail = reinterpret_cast<const int4 *>(p.items + item)[1];  // {slot, ox, oy}
    const JobDesc &J = p.jobs[cur.x];
    const int N = J.N;
    const bool other = J.out_f64 || J.planar;
    float2 *const out = static_cast<float2 *>(J.out);
    const char *gt = nullptr;  // this lane's entry under the sub-grid's first cell
    float factor_max = gmax;
    if constexpr (GT) {
      gt = reinterpret_cast<const char *>(rt_table<S>(J, cur.y)) + lx * 8 + ly * C::ROW;
      if constexpr (COMP) factor_max = __uint_as_float(rt_info(J, cur.y).top);
    }
    do {  // once; `break` ends the unit
      // Cells.  Compensated: sums in hi from `base` on and their remainders in
      // lo; of a pair, the cell that the current fy selects at j, the other at
      // j + Q.  Plain: sums in hi, and in run the running sums of the rows that
      // the current fy selects or every footprint covers.
      u64 hi[NX][NY], lo[COMP ? NX : 1][COMP ? NY : 1], run[COMP ? 1 : NX][COMP ? 1 : Q];
      u64 base = 0ull;
      float room = 0.f;  // bound on the item's sums that `base` is good for
      auto clear = [&]() {
#pragma unroll
        for (int i = 0; i < NX; ++i) {
#pragma unroll
          for (int j = 0; j < NY; ++j) {
            hi[i][j] = base;
            if constexpr (COMP) lo[i][j] = 0ull;
          }
          if constexpr (!COMP) {
#pragma unroll
            for (int j = 0; j < Q; ++j) run[i][j] = 0ull;
          }
        }
      };
      if constexpr (!COMP) clear();
      // a base for the terms of a block: room for twice what the item would take
      // if all its values were this large, and the sums moved when a later
      // block needs more
      auto rebase = [&](float need) {
        const float b = sum_base(2.f * need);
        const u64 old = base;
        base = pk2(b, b);
        if (room == 0.f) {
          clear();
        } else {
#pragma unroll
          for (int i = 0; i < NX; ++i)
#pragma unroll
            for (int j = 0; j < NY; ++j) {
              const u64 t = sub2(hi[i][j], old), n = add2(t, base);
              lo[i][j] = add2(lo[i][j], sub2(t, sub2(n, base)));
              hi[i][j] = n;
            }
        }
        room = b * (1.f / 1.5f);
      };
      // compensated: the cells of fy = f to the first place of their pairs (the
      // second of a pair is selected once fy > LY j + ly)
      int at_fy = 0;
      auto select = [&](int f) {
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) {
          if (min(at_fy, f) >= LY * (j + 1) || max(at_fy, f) <= LY * j) continue;
          const bool change = (LY * j + ly < at_fy) != (LY * j + ly < f);
          auto exchange = [&](u64 &a, u64 &b) {
            const u64 t = change ? b : a;
            b = change ? a : b;
            a = t;
          };
#pragma unroll
          for (int i = 0; i < NX; ++i) {
            exchange(hi[i][j], hi[i][j + Q]);
            exchange(lo[i][j], lo[i][j + Q]);
          }
        }
        at_fy = f;
      };
      // plain: the running sums of the alternating rows into the cells of fy = f
      auto merge_pairs = [&](int f) {
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) {
          const bool low = f <= LY * j + ly;
#pragma unroll
          for (int i = 0; i < NX; ++i) {
            hi[i][j] = add2(hi[i][j], low ? run[i][j] : 0ull);
            hi[i][j + Q] = add2(hi[i][j + Q], low ? 0ull : run[i][j]);
            run[i][j] = 0ull;
          }
        }
      };
      // those of the rows that every footprint covers
      auto merge_rest = [&]() {
#pragma unroll
        for (int j = PAIRS; j < Q; ++j)
#pragma unroll
          for (int i = 0; i < NX; ++i) {
            hi[i][j] = add2(hi[i][j], run[i][j]);
            run[i][j] = 0ull;
          }
      };
      // one staged record: its table entries (h: imaginary parts) and value
      struct Taps {
        float g[Q][C::NL], h[Q][C::NL];
        float vr, vi;
        bool left;  // the first column, not the last, is in the footprint
      };
      // the factors of one of a lane's rows
      auto load_row = [&](Taps &t, const float4 q, auto cx, auto JJ) {
        constexpr int j = decltype(JJ)::value;
        const int at = __float_as_int(q.y);
        const int fy = C::PADX ? at : at & 0xff;
        const bool left = at < (lx + 1) << 8;
        if constexpr (GT) {
          const char *a = gt + __float_as_int(q.x);
          if (j < PAIRS && fy > ly + LY * j) a += C::SUB;
          const int side = left ? 0 : C::ROW;
          rt_for<0, C::NL>([&](auto II) {
            constexpr int i = decltype(II)::value;
            const char *const e = (i == 0 ? a + side : a) + (j * LY * C::ROW + i * LX * 8);
            if constexpr (decltype(cx)::value) {
              const float2 w = __ldg(reinterpret_cast<const float2 *>(e));
              t.g[j][i] = w.x;
              t.h[j][i] = w.y;
            } else {
              t.g[j][i] = __ldg(reinterpret_cast<const float *>(e));
            }
          });
        } else {
          uint32_t a = tab + (uint32_t)__float_as_int(q.x);
          if (j < PAIRS && fy > ly + LY * j) a += C::SUB;
          const uint32_t side = C::PADX || left ? 0 : 64;
          rt_for<0, C::NL>([&](auto II) {
            constexpr int i = decltype(II)::value;
            constexpr int OFF = j * LY * C::ROW + i * LX * 4;
            const uint32_t ai = !C::PADX && i == 0 ? a + side : a;
            t.g[j][i] = lds<OFF>(ai);
            if constexpr (decltype(cx)::value) t.h[j][i] = lds<OFF>(ai + im_off);
          });
        }
      };
      auto load_value = [&](Taps &t, const float4 q) {
        t.vr = q.z;
        t.vi = q.w;
        t.left = __float_as_int(q.y) < (lx + 1) << 8;
      };
      auto load = [&](Taps &t, const float4 q, auto cx) {
        load_value(t, q);
        rt_for<0, Q>([&](auto JJ) { load_row(t, q, cx, JJ); });
      };
      // a value in the outer columns, of which the footprint covers one
      auto at_column = [&](u64 v, bool left, auto II) {
        constexpr int i = decltype(II)::value;
        if constexpr (C::PADX || (i > 0 && i < NX - 1)) return v;
        else return (i == 0) == left ? v : 0ull;
      };
      // terms va ga + vb gb into the sums of row j, column i
      auto add_two = [&](auto JJ, auto II, u64 va, u64 ga, u64 vb, u64 gb) {
        constexpr int j = decltype(JJ)::value, i = decltype(II)::value;
        if constexpr (COMP) exact_add2(hi[i][j], lo[i][j], va, ga, vb, gb);
        else run[i][j] = fma2(vb, gb, fma2(va, ga, run[i][j]));
      };
      auto add = [&](const Taps &t, auto cx) {
        const u64 v = pk2(t.vr, t.vi), w = pk2(-t.vi, t.vr);
        rt_for<0, Q>([&](auto JJ) {
          constexpr int j = decltype(JJ)::value;
          rt_for<0, NX>([&](auto II) {
            constexpr int i = decltype(II)::value, l = C::PADX || (i > 0 && i < NX - 1) ? i : 0;
            const u64 vi = at_column(v, t.left, II), g2 = pk2(t.g[j][l], t.g[j][l]);
            if constexpr (decltype(cx)::value)
              add_two(JJ, II, vi, g2, at_column(w, t.left, II), pk2(t.h[j][l], t.h[j][l]));
            else run[i][j] = fma2(vi, g2, run[i][j]);
          });
        });
      };
      // the staged records of a block in order of fy, cnt[f] of them (bytes;
      // even numbers) for each.  Compensated, two at a time by tables without
      // imaginary parts: a row's factors of the next two are loaded once it has
      // been added.
      auto add_block_by_two = [&](u64 cnt) {
        constexpr std::false_type cx{};
        Taps a, b;
        load(a, stage[0], cx);
        load(b, stage[1], cx);
        const float4 *st = stage + 2;
#pragma unroll 1
        for (int f = 0; f < 8; ++f) {
          int left = (int)(cnt >> (8 * f)) & 0xff;
          if (left == 0) continue;
          select(f);
#pragma unroll 1
          do {
            const int m = GT ? min(left, kRtRun) : left;
            const float4 *const end = st + m;
            left -= m;
            in_step();
#pragma unroll 1
            do {
              const float4 qa = st[0], qb = st[1];
              const u64 va = pk2(a.vr, a.vi), vb = pk2(b.vr, b.vi);
              rt_for<0, Q>([&](auto JJ) {
                constexpr int j = decltype(JJ)::value;
                rt_for<0, NX>([&](auto II) {
                  constexpr int i = decltype(II)::value, l = C::PADX || (i > 0 && i < NX - 1) ? i : 0;
                  add_two(JJ, II, at_column(va, a.left, II), pk2(a.g[j][l], a.g[j][l]),
                          at_column(vb, b.left, II), pk2(b.g[j][l], b.g[j][l]));
                });
                load_row(a, qa, cx, JJ);
                load_row(b, qb, cx, JJ);
              });
              load_value(a, qa);
              load_value(b, qb);
              st += 2;
            } while (st != end);
          } while (left > 0);
        }
      };
      // Compensated, a table in shared memory: two at a time without imaginary parts,
      // else one, and nothing loaded ahead, so that the rows that fy selects are the
      // same for a whole share and registers suffice.  For support 16 without
      // imaginary parts add_block_by_two takes 1 % less time.  add_block for complex
      // tables, 6 % faster for them, made the real ones 2 to 5 % slower (386 instead
      // of 369 us for 4.19 M records of support 8).
      auto add_share = [&](const float4 *st, const float4 *end, int f, auto cx) {
        constexpr bool CXR = decltype(cx)::value;
        constexpr int N2 = CXR ? 1 : 2;
        uint32_t at[PAIRS];
#pragma unroll
        for (int j = 0; j < PAIRS; ++j) at[j] = tab + (f > ly + LY * j ? C::SUB : 0);
        const int left_below = (lx + 1) << 8;
#pragma unroll 1
        do {
          float4 q[N2];
          uint32_t side[N2];
          bool left[N2];
#pragma unroll
          for (int r = 0; r < N2; ++r) {
            q[r] = st[r];
            left[r] = __float_as_int(q[r].y) < left_below;
            side[r] = __float_as_uint(q[r].x) + (C::PADX || left[r] ? 0 : 64);
          }
          rt_for<0, Q>([&](auto JJ) {
            constexpr int j = decltype(JJ)::value;
            const uint32_t row = j < PAIRS ? at[j < PAIRS ? j : 0] : tab;
            float g[N2][C::NL], h[N2][C::NL];
#pragma unroll
            for (int r = 0; r < N2; ++r)
              rt_for<0, C::NL>([&](auto II) {
                constexpr int i = decltype(II)::value;
                constexpr int OFF = j * LY * C::ROW + i * LX * 4;
                const uint32_t a =
                    row + (!C::PADX && i == 0 ? side[r] : __float_as_uint(q[r].x));
                g[r][i] = lds<OFF>(a);
                if constexpr (CXR) h[r][i] = lds<OFF>(a + im_off);
              });
            rt_for<0, NX>([&](auto II) {
              constexpr int i = decltype(II)::value, l = C::PADX || (i > 0 && i < NX - 1) ? i : 0;
              const u64 va = at_column(pk2(q[0].z, q[0].w), left[0], II);
              const u64 ga = pk2(g[0][l], g[0][l]);
              if constexpr (CXR)
                add_two(JJ, II, va, ga, at_column(pk2(-q[0].w, q[0].z), left[0], II),
                        pk2(h[0][l], h[0][l]));
              else
                add_two(JJ, II, va, ga, at_column(pk2(q[1].z, q[1].w), left[1], II),
                        pk2(g[1][l], g[1][l]));
            });
          });
          st += N2;
        } while (st != end);
      };
      auto add_shares = [&](u64 cnt, auto cx) {
        const float4 *st = stage;
#pragma unroll 1
        for (int f = 0; f < 8; ++f) {
          const float4 *const end = st + ((int)(cnt >> (8 * f)) & 0xff);
          if (st == end) continue;
          select(f);
          add_share(st, end, f, cx);
          st = end;
        }
      };
      // The others one at a time, the table entries of one loaded while the
      // previous one is added.
      auto add_block = [&](u64 cnt, auto cx) {
        Taps a, b;
        load(a, stage[0], cx);
        float4 q = stage[1];
        int since = 0;
        const float4 *st = stage + 2;
#pragma unroll 1
        for (int f = 0; f < 8; ++f) {
          int left = (int)(cnt >> (8 * f)) & 0xff;
          if constexpr (COMP)
            if (left > 0) select(f);
#pragma unroll 1
          while (left > 0) {
            const int m = min(left, kRtRun);
            const float4 *const end = st + m;
            in_step();
#pragma unroll 1
            while (st != end) {
              load(b, q, cx);
              q = st[0];
              add(a, cx);
              load(a, q, cx);
              q = st[1];
              add(b, cx);
              st += 2;
            }
            left -= m;
            if constexpr (!COMP) {
              merge_pairs(f);
              since += m;
              if (PAIRS < Q && since >= kRtRun) {
                merge_rest();
                since = 0;
              }
            }
          }
        }
        if constexpr (!COMP && PAIRS < Q) merge_rest();
      };
      for (int k0 = cur.z; k0 < cur.w; k0 += kRtBlock) {
        const int n = min(kRtBlock, cur.w - k0);
        // counting sort by fy: counters of 8 bits, one 64-bit word for all
        // eight (at most 128 records)
        u64 mine = 0ull;
#pragma unroll
        for (int u = 0; u < PER; ++u)
          if (u * 32 + lane < n) mine += 1ull << (8 * (pk[u].y & 7));
        if constexpr (COMP) {
          unsigned top = 0;
#pragma unroll
          for (int u = 0; u < PER; ++u)
            if (u * 32 + lane < n) top = max(top, max(finite_magnitude(pv[u].x), finite_magnitude(pv[u].y)));
          top = __reduce_max_sync(0xffffffffu, top);
          // twice the sum of the item's terms, were all of them as large
          const float need = (cplx ? 4.f : 2.f) * (float)(cur.w - cur.z + 8) *
                             (__uint_as_float(top) * factor_max);
          if (room == 0.f || !(need <= room)) rebase(need);
        }
        u64 incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const u64 y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        const u64 all = __shfl_sync(0xffffffffu, incl, 31);
        const u64 even = (all + 0x0101010101010101ull) & 0xfefefefefefefefeull;
        const u64 starts = even * 0x0101010101010100ull;  // sums of the lower bytes
        u64 at = starts + (incl - mine);
        __syncwarp();  // the previous block's records were all read
        if (lane < 8) {  // the zero behind an odd share
          const int c = (int)(all >> (8 * lane)) & 0xff;
          if (c & 1)
            stage[((int)(starts >> (8 * lane)) & 0xff) + c] =
                make_float4(__int_as_float(C::PAD), 0.f, 0.f, 0.f);
        } else if (lane < 10) {  // two zeros behind the last
          const int e = ((int)(starts >> 56) & 0xff) + ((int)(even >> 56) & 0xff);
          stage[e + lane - 8] = make_float4(__int_as_float(C::PAD), 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int u = 0; u < PER; ++u)
          if (u * 32 + lane < n) {
            const int sh = 8 * (pk[u].y & 7);
            stage[(int)(at >> sh) & 0xff] =
                make_float4(__int_as_float(pk[u].x), __int_as_float(pk[u].y), pv[u].x, pv[u].y);
            at += 1ull << sh;
          }
        if (k0 + kRtBlock < cur.w) fetch(k0 + kRtBlock, cur.w, plane);
        else fetch(nxt.z, nxt.w, P == 1 ? 0 : next % P);
        __syncwarp();
        if constexpr (!COMP) {
          if (cplx) add_block(even, std::true_type{});
          else add_block(even, std::false_type{});
        } else if constexpr (GT) {
          if constexpr (CX) add_block(even, std::true_type{});
          else add_block_by_two(even);
        } else if (cplx) {
          add_shares(even, std::true_type{});
        } else {
          if constexpr (S == 8) add_shares(even, std::false_type{});
          else add_block_by_two(even);
        }
      }
      const int ox = tail.y, oy = tail.z;
      double2 *const slot = COMP && p.merge.base && tail.x >= 0
                                ? p.merge.base + (size_t)tail.x * p.merge.cells + plane * R * R
                                : nullptr;
      if constexpr (COMP) select(0);
      u64 z = 0ull;
#pragma unroll
      for (int i = 0; i < NX; ++i)
#pragma unroll
        for (int j = 0; j < NY; ++j) {
          if constexpr (COMP) hi[i][j] = sub2(hi[i][j], base);
          z = fma2(hi[i][j], 0ull, z);
        }
      const float2 zf = upk2(z);
      if (__any_sync(0xffffffffu, !(zf.x == 0.f && zf.y == 0.f))) {
        rt_redo<S, COMP, GT>(p, p.items[item], plane, tr, GT ? rt_info(J, cur.y).imag : cplx,
                             slot);
        break;
      }
      if (!slot && !other) {
        // complex64 interleaved grid: hi + lo rounded once
        float2 *const row0 = out + (size_t)plane * N * N;
        const bool inside = ox >= 0 && oy >= 0 && ox + R <= N && oy + R <= N;
#pragma unroll
        for (int j = 0; j < NY; ++j) {
          const int gy = oy + LY * j + ly;
          float2 *const row = row0 + ((ptrdiff_t)gy * N + ox + lx);
          const bool yin = inside || (unsigned)gy < (unsigned)N;
#pragma unroll
          for (int i = 0; i < NX; ++i) {
            float2 v;
            if constexpr (COMP) v = upk2(add2(hi[i][j], lo[i][j]));
            else v = upk2(hi[i][j]);
            if ((v.x != 0.f || v.y != 0.f) && yin &&
                (inside || (unsigned)(ox + lx + LX * i) < (unsigned)N))
              red_add_v2(reinterpret_cast<float *>(row + LX * i), v.x, v.y);
          }
        }
        break;
      }
#pragma unroll
      for (int j = 0; j < NY; ++j)
#pragma unroll
        for (int i = 0; i < NX; ++i) {
          const int x = LX * i + lx, y = LY * j + ly;
          const int gx = ox + x, gy = oy + y;
          const float2 h = upk2(hi[i][j]);
          float2 l = make_float2(0.f, 0.f);
          if constexpr (COMP) l = upk2(lo[i][j]);
          if (h.x == 0.f && h.y == 0.f && l.x == 0.f && l.y == 0.f) continue;
          // merge slot and complex128 grid: hi + lo exactly
          double dr = (double)h.x + (double)l.x, di = (double)h.y + (double)l.y;
          if (slot) {
            red_add(&slot[y * R + x].x, dr);
            red_add(&slot[y * R + x].y, di);
          } else if ((unsigned)gx < (unsigned)N && (unsigned)gy < (unsigned)N) {
            if (!J.out_f64) {
              dr = (double)__fadd_rn(h.x, l.x);
              di = (double)__fadd_rn(h.y, l.y);
            }
            out_red(J, (size_t)gy * N + gx, plane, p.P, dr, di);
          }
        }
    } while (false);
    // the last unit of a cut tile rounds the merged sums into the grid
    if (COMP && p.merge.base && tail.x >= 0) {
      __threadfence();
      __syncwarp();
      int4 *const d = p.merge.desc + tail.x;
      int done = 0;
      if (lane == 0) done = atomicAdd(&d->w, 1) + 1;
      if (__shfl_sync(0xffffffffu, done == d->z * P, 0)) {
        __threadfence();
        const double2 *const src = p.merge.base + (size_t)tail.x * p.merge.cells;
#pragma unroll 4
        for (int i = lane; i < p.P * R * R; i += 32) {
          const double2 v = __ldcg(src + i);
          if (v.x == 0.0 && v.y == 0.0) continue;
          const int plane = i / (R * R), c = i - plane * R * R;
          const int gx = tail.y + c % R, gy = tail.z + c / R;
          if ((unsigned)gx < (unsigned)N && (unsigned)gy < (unsigned)N)
            out_red(J, (size_t)gy * N + gx, plane, p.P, v.x, v.y);
        }
      }
    }
    if (next >= total) return;
    unit = next;
    cur = nxt;
    next = next2;
    nxt = nxt2;
  }
}

// tables read from global memory, any number of them.  Both forms are launched
// (the flag is on the device) and one of them returns at once: as two branches
// of one kernel, the complex form of support 8 took 15 % longer.
template <int S, bool COMP, bool CX>
__global__ void __launch_bounds__(32 * RtCfg<S, true>::WARPS, 1)
    regtile_tables_kernel(const __grid_constant__ RegTileLaunch p) {
  extern __shared__ __align__(16) unsigned char smem[];
  after_predecessor();
  float4 *const stage = reinterpret_cast<float4 *>(smem) + (threadIdx.x >> 5) * kRtStage;
  if ((*p.any_imag != 0) == CX) rt_items<S, COMP, true, CX>(p, nullptr, stage, CX, 0.f);
}

template <int S, bool COMP>
__global__ void __launch_bounds__(32 * RtCfg<S, false>::WARPS, 1)
    regtile_kernel(const __grid_constant__ RegTileLaunch p) {
  using C = RtCfg<S, false>;
  constexpr int NT = 32 * C::WARPS, RF = C::ROW / 4, PF = C::PAD / 4;
  extern __shared__ __align__(16) unsigned char smem[];
  const int tid = threadIdx.x;
  const int nf = rt_table_floats(S, p.G), rows = p.G * p.G * S;
  float *const tr = reinterpret_cast<float *>(smem), *const ti = tr + nf;
  float4 *const stage = reinterpret_cast<float4 *>(smem + 8 * (size_t)nf) + (tid >> 5) * kRtStage;

  // tables: from the caller's [G*G][S][S], or the Gaussian's factors (expf as
  // everywhere; their product rounds as the on-the-fly factor does)
  int imag = 0;
  __shared__ unsigned s_top;  // largest magnitude in the table (the Gaussian's: at most 1)
  unsigned top = __float_as_uint(1.f);
  if (COMP && !p.gauss) {
    top = 0;
    if (tid == 0) s_top = 0;
    __syncthreads();
  }
  if (!p.overlap) after_predecessor();
  if (p.gauss) {
    float *g1 = reinterpret_cast<float *>(smem + 8 * (size_t)nf);
    gauss_fill(g1, S, p.G, p.sigma, tid, NT);
    __syncthreads();
    for (int i = tid; i < nf; i += NT) {
      const int row = i / RF, c = i - row * RF - PF;
      float g = 0.f;
      if ((unsigned)c < (unsigned)S && row < rows) {
        const int sub = row / S, b = row % S, sy = sub / p.G, sx = sub - sy * p.G;
        g = g1[sx * S + c] * g1[sy * S + b];
      }
      tr[i] = g;
    }
  } else {
#pragma unroll 4
    for (int i = tid; i < nf; i += NT) {
      const int row = i / RF, c = i - row * RF - PF;
      float2 v = make_float2(0.f, 0.f);
      if ((unsigned)c < (unsigned)S && row < rows) v = __ldg(p.gcf + row * S + c);
      tr[i] = v.x;
      ti[i] = v.y;
      imag |= v.y != 0.f;
      if constexpr (COMP) top = max(top, max(finite_magnitude(v.x), finite_magnitude(v.y)));
    }
    if constexpr (COMP) {
      top = __reduce_max_sync(0xffffffffu, top);
      if ((tid & 31) == 0) atomicMax(&s_top, top);
    }
  }
  if (p.overlap) after_predecessor();
  const bool cplx = __syncthreads_or(imag);
  if (COMP && !p.gauss) top = s_top;
  rt_items<S, COMP, false, true>(p, tr, stage, cplx, __uint_as_float(top));
}

constexpr int kInfoChunk = 1024;  // entries of a table that a block looks at

// What regtile_tables_kernel needs to know of every table of a class (blockIdx.y:
// jobs, those that share a stack of tables once): compensated sums choose their
// base by the largest magnitude, and a class of tables without imaginary parts
// takes half the products.
__global__ void __launch_bounds__(256)
    table_info_kernel(const JobDesc *jobs, int njobs, int entries, unsigned *any_imag) {
  after_predecessor();
  const int chunk = min(entries, kInfoChunk);
  for (int j = blockIdx.y; j < njobs; j += gridDim.y) {
    const JobDesc &J = jobs[j];
    if (!J.gcf_info_owner) continue;
    const int64_t chunks = (int64_t)J.n_gcf * (entries / chunk);
    for (int64_t c = blockIdx.x; c < chunks; c += gridDim.x) {
      const float2 *const t = static_cast<const float2 *>(J.gcf) + c * chunk;
      unsigned top = 0;
      bool imag = false;
#pragma unroll 4
      for (int i = threadIdx.x; i < chunk; i += 256) {
        const float2 v = __ldg(t + i);
        imag = imag || v.y != 0.f;
        top = max(top, max(finite_magnitude(v.x), finite_magnitude(v.y)));
      }
      top = __reduce_max_sync(0xffffffffu, top);
      imag = __any_sync(0xffffffffu, imag);
      if ((threadIdx.x & 31) == 0) {
        TableInfo *const info = J.gcf_info + c / (entries / chunk);
        atomicMax(&info->top, top);
        if (imag) {
          atomicOr(&info->imag, 1u);
          atomicOr(any_imag, 1u);
        }
      }
    }
  }
}

template <int S, bool GT>
cudaError_t rt_launch(void (*kern)(RegTileLaunch), const RegTileLaunch &g, cudaStream_t s) {
  constexpr int warps = RtCfg<S, GT>::WARPS;
  const size_t smem = GT ? warps * kRtStage * sizeof(float4) : regtile_smem_bytes(S, g.G);
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  const int64_t blocks = std::max<int64_t>(1, std::min<int64_t>(g.sm_count, g.max_items * g.P));
  count_launch();
  return launch_overlapped(kern, (unsigned)blocks, 32 * warps, smem, s, g.overlap, g);
}

template <int S, bool COMP> cudaError_t rt_launches(const RegTileLaunch &g, cudaStream_t s) {
  if (!g.tables) return rt_launch<S, false>(regtile_kernel<S, COMP>, g, s);
  const cudaError_t e = rt_launch<S, true>(regtile_tables_kernel<S, COMP, false>, g, s);
  return e != cudaSuccess ? e : rt_launch<S, true>(regtile_tables_kernel<S, COMP, true>, g, s);
}

}  // namespace

size_t regtile_smem_bytes(int S, int G) {
  const int warps = S == 8 ? RtCfg<8, false>::WARPS : RtCfg<16, false>::WARPS;
  return 8 * (size_t)rt_table_floats(S, G) + (size_t)warps * kRtStage * sizeof(float4);
}

cudaError_t launch_table_info(const JobDesc *jobs, int njobs, int S, int G, int64_t tables,
                              unsigned *any_imag, cudaStream_t s) {
  const int entries = G * G * S * S;
  const int64_t chunks = tables * ((entries + kInfoChunk - 1) / kInfoChunk);
  const int y = std::min(njobs, 1024), x = (int)std::min<int64_t>(chunks, std::max(1, 2048 / y));
  count_launch();
  return launch_overlapped(table_info_kernel, dim3(x, y), 256, 0, s, true, jobs, njobs, entries,
                           any_imag);
}

cudaError_t launch_regtile(const RegTileLaunch &g, cudaStream_t s) {
  switch (g.S) {
    case 8: return g.compensated ? rt_launches<8, true>(g, s) : rt_launches<8, false>(g, s);
    case 16: return g.compensated ? rt_launches<16, true>(g, s) : rt_launches<16, false>(g, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gg
