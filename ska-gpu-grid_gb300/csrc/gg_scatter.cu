// Scatter gridding (the reference's default method, grid_kernel
// grid_gpu.cu:95-173 and grid_kernel_small_gcf :254-327), rebuilt for sm_103a.
//
// Every tap is added into the grid in HBM/L2 by the memory system itself:
// native red.global.add.v2.f32 (one 8-byte complex per tap) or
// red.global.add.f64, instead of the reference's CAS retry loops
// (atomicAddWrap, grid_gpu.cu:53-90; the FP32 path there is always a CAS
// loop).  The small-support kernel's unsynchronised += (grid_gpu.cu:309-310)
// is a data race and has no counterpart here.
//
// A warp takes an equal share of the visibilities, 32 consecutive ones at a
// time: every lane loads one (u,v) as a 128-bit vector, performs the FP64 index
// step once, and parks the footprint's place, the sub-kernel and the values in
// shared memory; then the warp walks the visibilities with its lanes spread
// over the S*S taps, so its reductions hit consecutive cells of a footprint
// row.  Nothing waits for the other warps (256 visibilities a CTA, between
// barriers, left its last round three quarters empty).
//
// What binds: FP32 values, the L2's reductions by 32-byte sector (1 M
// visibilities of support 8 on 2048^2: 22 sectors each, 190 G/s of the 190 G/s
// that coalesced reductions reach; 190 -> 134 us once a visibility cost 83
// warp instructions instead of 156, 121 with equal shares).  FP64 values, the
// FP64 pipe: 16 multiplications a visibility of support 16 and lane when the
// table has no imaginary parts (32 operations before), one reduction per
// component with every sector touched once (262,144 visibilities on 1024^2,
// whole call: 605 us before, 305 now; of the difference 191 us by the products,
// 52 by equal shares, 57 by four factors instead of eight ahead and twice the
// warps; the multiplications alone take 215).
//
// Compensated mode (complex64 output): the hi grid is updated with
// atom.global.v2.f32.add, which returns the previous value; two_sum of
// (previous, term) is the exact rounding error, reduced into a lo grid that
// a final pass folds into the output.  With complex128 output the FP32 terms
// are reduced with red.global.add.f64, which is at least as accurate.
#include "gg_kernels.cuh"

namespace gg {

constexpr int kScatterThreads = 256;
// resident on an SM (FP64 values, support 16, the case below: 2 CTAs 362 us of
// the whole call, 3 324, 4 305, 5 310).  FP32 values, plain sums, several planes,
// 524 k visibilities of support 8 on 1024^2: two 160 us with 4, 152 with 5 and
// 159 with 6, four 290, 278 and 272; one 90, 95 and 98.
constexpr int kScatterCtas = 4, kScatterCtasPlanes = 5;
// Compensated sums wait for the previous value of every tap: more warps hide
// it, until those on the same cells get in each other's way, which takes longer
// on small footprints.  us with 4 / 5 / 6 CTAs, on tracks: support 4, 1 M
// visibilities 212 / 198 / 179, 4 M 715 / 657 / 574; support 8, 100 k 58 / 60 / 57,
// 1 M 317 / 300 / 298, 3 M 855 / 799 / 809; support 16, 262 k 286 / 275 / 325, 1 M
// 995 / 942 / 934, 4.19 M 4270 / 4012 / 3613; support 32, 300 k 1264 / 1088 /
// 1193, 2 M 8515 / 7301 / 6634.
constexpr int kScatterCtasComp = 5, kScatterCtasLarge = 6;
constexpr int64_t kScatterLarge = 1 << 21;  // visibilities, supports 16 and 32

__device__ __forceinline__ int find_job_v(const int64_t *base, int njobs,
                                          int64_t g) {
  int lo = 0, hi = njobs - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (__ldg(base + mid) <= g) lo = mid; else hi = mid - 1;
  }
  return lo;
}

// neither infinite nor NaN, without the FP64 pipe
__device__ __forceinline__ bool finite_bits(double x) {
  return (__double2hiint(x) & 0x7ff00000) != 0x7ff00000;
}

template <int S, class ACC, int GK, int CTAS>
__global__ void __launch_bounds__(kScatterThreads, CTAS)
    scatter_kernel(KParams kp) {
  constexpr bool GAUSS = GK == 1, WPHASE = GK == 2;
  using VT = typename ACC::VT;
  using VT2 = typename vec2_of<VT>::type;
  constexpr int NT = kScatterThreads, H = S / 2;
  extern __shared__ __align__(16) unsigned char smem[];
  // grid cell of the footprint's first tap, sub-kernel (of all tables), the
  // tap's column and row + 64 (16 bits each), job * 2 + inside the grid (-1:
  // skip)
  int4 *rec = reinterpret_cast<int4 *>(smem);
  VT2 *sval = reinterpret_cast<VT2 *>(smem + NT * sizeof(int4));  // [NT][P]
  float *g1 = reinterpret_cast<float *>(smem + NT * sizeof(int4) +
                                        (size_t)NT * kp.P * sizeof(VT2));
  // WPHASE: the per-visibility factor, beside the record
  float2 *sfac = reinterpret_cast<float2 *>(smem + NT * sizeof(int4) +
                                            (size_t)NT * kp.P * sizeof(VT2) + 64 * S * 4);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int P = kp.P;
  if constexpr (GAUSS) gauss_fill(g1, S, kp.G, kp.sigma, tid, NT);
  const int64_t vb0 = kp.njobs > 1 ? __ldg(kp.vis_base) : 0;
  constexpr bool F64 = std::is_same<VT, double>::value;
  constexpr int TAPS = (S * S + 31) / 32;    // of a lane
  constexpr int ROWS = S < 32 ? 32 / S : 1;  // rows between them
  const int lx = lane % S, ly = lane / S;
  // the current job
  int job = -1, N = 0, lane_cell = 0, step = 0;
  bool planar = false, f64 = false, native = false;
  size_t NN = 0;
  char *out = nullptr;
  float *lo = nullptr;
  const VT2 *gcf = nullptr;

  if constexpr (GAUSS) __syncthreads();
  const int64_t nwarps = (int64_t)gridDim.x * (NT / 32), wid = blockIdx.x * (NT / 32) + warp;
  const int64_t end = kp.total_vis * (wid + 1) / nwarps;
  for (int64_t c0 = kp.total_vis * wid / nwarps; c0 < end; c0 += 32) {
    __syncwarp();  // the previous 32 fully consumed
    {
      const int64_t t = c0 + lane;
      int4 r = make_int4(0, 0, 0, -1);
      if (t < end) {
        int j = 0;
        int64_t n = t;
        if (kp.njobs > 1) {
          const int64_t g = t + vb0;
          j = find_job_v(kp.vis_base, kp.njobs, g);
          n = g - __ldg(kp.vis_base + j);
        }
        const JobDesc &J = kp.jobs[j];
        int mx, sx, my, sy;
        bool ok;
        if (J.uv_f64) {
          double2 c = __ldg(reinterpret_cast<const double2 *>(J.uv) + n);
          ok = index_step(c.x, J.G, mx, sx) & index_step(c.y, J.G, my, sy);
        } else {
          float2 c = __ldg(reinterpret_cast<const float2 *>(J.uv) + n);
          ok = index_step(c.x, J.G, mx, sx) & index_step(c.y, J.G, my, sy);
        }
        if (ok && ((unsigned)sx >= (unsigned)J.G || (unsigned)sy >= (unsigned)J.G)) {
          ok = false;
          atomicAdd(&kp.flags[FLAG_INDEX], 1);
        } else if (!ok) {
          atomicAdd(&kp.flags[FLAG_INDEX], 1);
        }
        int tab = 0;
        if (ok && J.gcf_index) {
          tab = __ldg(J.gcf_index + n);
          if ((unsigned)tab >= (unsigned)J.n_gcf) {
            ok = false;
            atomicAdd(&kp.flags[FLAG_INDEX], 1);
          }
        }
        if (ok && mx + H >= 0 && mx - H + 1 < J.N && my + H >= 0 && my - H + 1 < J.N) {
          const int fx = mx - H + 1, fy = my - H + 1;
          const bool inside = fx >= 0 && fy >= 0 && fx + S <= J.N && fy + S <= J.N;
          r = make_int4(fy * J.N + fx, tab * J.G * J.G + sy * J.G + sx,
                        (fx + 64) | ((fy + 64) << 16), 2 * j + inside);
          const VT2 *v = reinterpret_cast<const VT2 *>(J.vals) + n * P;
          for (int p = 0; p < P; ++p) sval[tid * P + p] = __ldg(v + p);
          if constexpr (WPHASE) {
            // (T, w) at the centre offset S(S-1)/2-1 of the table
            const VT2 tw = __ldg(reinterpret_cast<const VT2 *>(J.gcf) + (S * (S - 1) / 2 - 1));
            double u, vv;
            if (J.uv_f64) {
              const double2 c = __ldg(reinterpret_cast<const double2 *>(J.uv) + n);
              u = c.x;
              vv = c.y;
            } else {
              const float2 c = __ldg(reinterpret_cast<const float2 *>(J.uv) + n);
              u = c.x;
              vv = c.y;
            }
            sfac[tid] = wphase_factor(u, vv, mx, sx, my, sy, J.G, (double)tw.x, (double)tw.y);
          }
        }
      }
      rec[tid] = r;
    }
    __syncwarp();
    // Lane l takes the taps l, l + 32, ... of a visibility: their places in
    // the footprint are the same for all, and so are the table offsets.  The
    // job's fields stay in registers while the job does.
    for (int q = tid - lane; q < tid - lane + 32; ++q) {
      const int4 r = rec[q];
      if (r.w < 0) continue;
      if (r.w >> 1 != job) {
        job = r.w >> 1;
        const JobDesc &J = kp.jobs[job];
        N = J.N;
        planar = J.planar;
        f64 = J.out_f64;
        out = static_cast<char *>(J.out);
        gcf = reinterpret_cast<const VT2 *>(J.gcf);
        lo = J.lo;
        lane_cell = ly * N + lx;
        step = ROWS * N;
        NN = (size_t)N * N;
        native = !planar && f64 == std::is_same<VT, double>::value &&
                 !std::is_same<ACC, AccComp>::value;
      }
      const bool inside = r.w & 1;
      const VT2 *const g0 = gcf + (int64_t)r.y * (S * S);
      const int cell0 = r.x + lane_cell;
      // factor of the tap at column x, row y; false: off the grid
      auto factor_at = [&](int x, int y, auto &g) {
        if (!inside) {
          const int fx = (r.z & 0xffff) - 64, fy = (int)((unsigned)r.z >> 16) - 64;
          if ((unsigned)(fx + x) >= (unsigned)N || (unsigned)(fy + y) >= (unsigned)N) return false;
        }
        if constexpr (GAUSS) {
          const int sub = r.y & (kp.G * kp.G - 1), sy = sub / kp.G, sx = sub - sy * kp.G;
          g.x = (VT)(g1[sx * S + x] * g1[sy * S + y]);
          g.y = (VT)0;
        } else if constexpr (WPHASE) {
          g.x = (VT)sfac[q].x;
          g.y = (VT)sfac[q].y;
        } else {
          g = __ldg(g0 + y * S + x);
        }
        return true;
      };
      // of this lane's tap k; false also: no such tap
      auto factor = [&](int k, VT &gr, VT &gi) {
        if (S * S % 32 != 0 && lane + 32 * k >= S * S) return false;
        VT2 g;
        if (!factor_at(lx, ly + k * ROWS, g)) return false;
        gr = g.x;
        gi = g.y;
        return true;
      };
      // the Gaussian's factor is real: an infinite component of a value stays
      // in its own component of the grid
      auto product = [&](const VT2 v, VT gr, VT gi, VT &tr, VT &ti) {
        if constexpr (GAUSS) {
          tr = v.x * gr;
          ti = v.y * gr;
        } else {
          cmul<VT>(v.x, v.y, gr, gi, tr, ti);
        }
      };
      // from a lane's first part to its part k, in doubles
      auto part_step = [&](int k) -> int64_t {
        if constexpr (S == 32) return 2 * ((int64_t)(k >> 1) * N + 16 * (k & 1));
        return 2 * (int64_t)k * (S < 16 ? 16 / S : 1) * N;
      };
      for (int p = 0; p < P; ++p) {
        const VT2 v = sval[q * P + p];
        if constexpr (F64) if (native) {
          // Complex128 grid: a lane takes one component of a tap, so that a
          // warp's reductions cover whole sectors (a reduction of the real
          // parts and one of the imaginary parts touched every sector twice).
          // FP64 products bind: a tap without an imaginary part takes one per
          // component instead of two (unless 0 * v matters), decided for the
          // whole warp, as a choice per tap would compute both.
          constexpr int PARTS = (S * S * 2 + 31) / 32, U = PARTS < 4 ? PARTS : 4;
          constexpr int PROWS = S < 16 ? 16 / S : 1;  // rows between a lane's parts
          const int px = (lane >> 1) % S, py = (lane >> 1) / S, im = lane & 1;
          // component = a * re(g) + b * im(g)
          const double va = im ? v.y : v.x, vb = im ? v.x : -v.y;
          double *const cell = reinterpret_cast<double *>(out) +
                               2 * (p * NN + (size_t)(r.x + py * N + px)) + im;
#pragma unroll 1
          for (int k0 = 0; k0 < PARTS; k0 += U) {
            double2 g[U];
            bool on[U];
            bool full = !GAUSS && (!finite_bits(va) || !finite_bits(vb));
#pragma unroll
            for (int k = 0; k < U; ++k) {
              // S = 32: two parts per row
              const int x = S == 32 ? px + 16 * ((k0 + k) & 1) : px;
              const int y = S == 32 ? (k0 + k) >> 1 : py + (k0 + k) * PROWS;
              g[k] = make_double2(0.0, 0.0);
              on[k] = factor_at(x, y, g[k]);
              full = full || (((unsigned)__double2hiint(g[k].y) << 1) | __double2loint(g[k].y)) != 0;
            }
            if (__any_sync(0xffffffffu, full)) {
#pragma unroll
              for (int k = 0; k < U; ++k)
                if (on[k]) red_add(cell + part_step(k0 + k), va * g[k].x + vb * g[k].y);
            } else {
#pragma unroll
              for (int k = 0; k < U; ++k)
                if (on[k]) red_add(cell + part_step(k0 + k), va * g[k].x);
            }
          }
          continue;
        }
        if (!F64 && native) {
          // complex64 grid
          float *const cell = reinterpret_cast<float *>(out) + 2 * (p * NN + (size_t)cell0);
#pragma unroll 4
          for (int k = 0; k < TAPS; ++k) {
            VT gr, gi, tr, ti;
            if (!factor(k, gr, gi)) continue;
            product(v, gr, gi, tr, ti);
            red_add_v2(cell + 2 * (int64_t)(k * step), (float)tr, (float)ti);
          }
          continue;
        }
#pragma unroll 2
        for (int k = 0; k < TAPS; ++k) {
          VT gr, gi, tr, ti;
          if (!factor(k, gr, gi)) continue;
          product(v, gr, gi, tr, ti);
          const size_t c = p * NN + (size_t)(cell0 + k * step);
          if constexpr (std::is_same<ACC, AccComp>::value) {
            if (!f64) {
              float *const hi = reinterpret_cast<float *>(out);
              float er, ei, s;
              if (planar) {
                float o = atomicAdd(hi + c, (float)tr);
                two_sum(o, (float)tr, s, er);
                o = atomicAdd(hi + (size_t)P * NN + c, (float)ti);
                two_sum(o, (float)ti, s, ei);
                if (er != 0.f) red_add(lo + c, er);
                if (ei != 0.f) red_add(lo + (size_t)P * NN + c, ei);
              } else {
                float2 o = atom_add_v2(hi + 2 * c, (float)tr, (float)ti);
                two_sum(o.x, (float)tr, s, er);
                two_sum(o.y, (float)ti, s, ei);
                if (er != 0.f || ei != 0.f) red_add_v2(lo + 2 * c, er, ei);
              }
              continue;
            }
          }
          if (f64)
            grid_red<double>((double *)out, c, 0, P, NN, planar, (double)tr, (double)ti);
          else
            grid_red<float>((float *)out, c, 0, P, NN, planar, (double)tr, (double)ti);
        }
      }
    }
  }
}

template <int S, class ACC, int GK, int CTAS>
static cudaError_t scatter_launch(const KParams &kp, int sm_count, cudaStream_t s) {
  using VT2 = typename vec2_of<typename ACC::VT>::type;
  size_t smem = kScatterThreads * sizeof(int4) +
                (size_t)kScatterThreads * kp.P * sizeof(VT2) + 64 * S * 4 +
                (GK == 2 ? kScatterThreads * sizeof(float2) : 0);
  auto kern = scatter_kernel<S, ACC, GK, CTAS>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kScatterThreads, smem);
  if (e != cudaSuccess) return e;
  if (per_sm < 1) return cudaErrorInvalidConfiguration;
  const int64_t chunks = (kp.total_vis + 31) / 32;  // at least four a warp
  int64_t grid = (int64_t)sm_count * per_sm;
  if (grid > chunks) grid = chunks;
  if (grid < 1) return cudaSuccess;
  kern<<<(unsigned)grid, kScatterThreads, smem, s>>>(kp);
  count_launch();
  return cudaGetLastError();
}

template <int S>
static cudaError_t scatter_dispatch(const GridLaunch &g, const KParams &kp,
                                    cudaStream_t s) {
  // GCF source: 0 table, 1 Gaussian on the fly, 2 COMPUTE_GCF phase factor
  const int gk = g.wphase ? 2 : (g.gauss ? 1 : 0);
#define GG_SC(ACCT, CTAS)                                                      \
  return gk == 2 ? scatter_launch<S, ACCT, 2, CTAS>(kp, g.sm_count, s)         \
                 : (gk == 1 ? scatter_launch<S, ACCT, 1, CTAS>(kp, g.sm_count, s) \
                            : scatter_launch<S, ACCT, 0, CTAS>(kp, g.sm_count, s))
  if (g.vals_f64) GG_SC(AccF64, kScatterCtas);
  if (g.accum == GG_ACC_COMPENSATED) {
    if constexpr (S <= 8) {
      GG_SC(AccComp, kScatterCtasLarge);
    } else {
      if (g.total_vis >= kScatterLarge) GG_SC(AccComp, kScatterCtasLarge);
      GG_SC(AccComp, kScatterCtasComp);
    }
  }
  if (g.P > 1) GG_SC(AccF32, kScatterCtasPlanes);
  GG_SC(AccF32, kScatterCtas);
#undef GG_SC
}

cudaError_t launch_scatter(const GridLaunch &g, cudaStream_t s) {
  KParams kp{};
  kp.jobs = g.jobs;
  kp.flags = g.flags;
  kp.njobs = g.njobs;
  kp.vis_base = g.vis_base;
  kp.total_vis = g.total_vis;
  kp.P = g.P;
  kp.T = g.tile;
  kp.G = g.G;
  kp.sigma = g.sigma;
  switch (g.S) {
    case 4: return scatter_dispatch<4>(g, kp, s);
    case 8: return scatter_dispatch<8>(g, kp, s);
    case 16: return scatter_dispatch<16>(g, kp, s);
    case 32: return scatter_dispatch<32>(g, kp, s);
  }
  return cudaErrorInvalidValue;
}

__global__ void comp_finalize_kernel(float *out, const float *lo, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    out[i] = __fadd_rn(out[i], lo[i]);
}

cudaError_t launch_comp_finalize(float *out, const float *lo, int64_t n,
                                 cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  int64_t b = (n + 255) / 256;
  if (b > 152 * 16) b = 152 * 16;
  comp_finalize_kernel<<<(unsigned)b, 256, 0, s>>>(out, lo, n);
  count_launch();
  return cudaGetLastError();
}

}  // namespace gg
