// Degridding: the adjoint of the gridder.  The reference has no degridder;
// this one keeps its gridder's conventions (grid.cu:157-191 for the index
// step, the tap window (-S/2, S/2] and the table entry of a tap) so that
// degridding with the same table is the exact adjoint of gridding:
//
//   vals[n][p] = sum over the on-grid taps of n of grid[p][y][x] * conj(w)
//
// and <grid(v), g> = <v, degrid(g)> for <a, b> = sum conj(a) b.
//
// Each visibility is summed by S lanes, one footprint column each (32/S
// visibilities per warp), so no atomics and no binning are needed: the lanes
// of a visibility read contiguous cells of one row per step, and
// consecutive visibilities on a uv track read overlapping footprints
// through L1/L2.
//  * The index step is done for 32 visibilities at once, one per lane, and
//    handed round by shuffles (every lane of a visibility had repeated it).
//  * Rows are taken four at a time: their cells and factors are loaded, then
//    summed.  Factors without imaginary parts, as a warp sees them, take one
//    packed multiply-add per tap instead of two.
//  * FP32 values with GG_ACC_COMPENSATED: every tap by a table with imaginary
//    parts, and every two taps by one without together with what their own sum
//    lost, are added into a two-sum (hi, lo) pair, which the reduction over the
//    lanes carries; else plain FP32 sums.  FP64 values: FP64 sums.
//  * The reduction splits the components first: one lane of a pair goes on with
//    the real, the other with the imaginary parts, which halves its shuffles.
//
// 4.19 M visibilities of support 8 from a 4096^2 grid: 664 us with a two-sum for
// every tap and the index step in every lane, 372 now.  Errors against 64 bits
// of that case: 3.6e-8 and 3.1e-8 (rms, relative).  Runs of four taps summed
// plainly take 328 us, but 4.7e-8: not taken.  With the table in shared memory
// (one CTA of 1024 threads): 6 % less above 1.5 M visibilities, more below: not
// taken.
#include <type_traits>

#include "gg_kernels.cuh"

namespace gg {

namespace {

__device__ __forceinline__ bool uv_step(const void *uv, int uv_f64, int64_t n, int G, int &mx,
                                        int &sx, int &my, int &sy) {
  if (uv_f64) {
    const double2 c = __ldg(reinterpret_cast<const double2 *>(uv) + n);
    const bool a = index_step(c.x, G, mx, sx);
    const bool b = index_step(c.y, G, my, sy);
    return a && b;
  }
  const float2 c = __ldg(reinterpret_cast<const float2 *>(uv) + n);
  const bool a = index_step(c.x, G, mx, sx);
  const bool b = index_step(c.y, G, my, sy);
  return a && b;
}

// running sum of one lane's component in the reduction: plain, or (hi, lo)
template <typename VT, bool COMP> struct LaneSum {
  VT h = 0, l = 0;
  // adds the partner lane's pair (hi sums two-summed, lo sums added)
  __device__ __forceinline__ void merge(VT oh, VT ol) {
    if constexpr (COMP) {
      float s, e;
      two_sum(h, oh, s, e);
      h = s;
      l = __fadd_rn(__fadd_rn(l, ol), e);
    } else {
      h += oh;
    }
  }
  __device__ __forceinline__ void merge_lane(int o) {
    const VT oh = __shfl_xor_sync(0xffffffffu, h, o);
    const VT ol = COMP ? __shfl_xor_sync(0xffffffffu, l, o) : (VT)0;
    merge(oh, ol);
  }
  __device__ __forceinline__ VT value() const {
    if constexpr (COMP) return __fadd_rn(h, l);
    return h;
  }
};

constexpr int kDegridCtas = 4;  // resident on an SM

template <int S, typename VT, typename GT, int GK, bool COMP>
__global__ void __launch_bounds__(256, kDegridCtas) degrid_kernel(const __grid_constant__ DegridLaunch d) {
  using VT2 = typename vec2_of<VT>::type;
  using GT2 = typename vec2_of<GT>::type;
  constexpr bool F32 = std::is_same<VT, float>::value;
  constexpr int VPW = 32 / S;          // visibilities per warp step
  constexpr int R = 4;                 // rows at a time
  __shared__ float g1[GK == 1 ? 64 * S : 1];
  if constexpr (GK == 1) {
    gauss_fill(g1, S, d.G, d.sigma, threadIdx.x, blockDim.x);
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, sl = lane % S, sv = lane / S;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const size_t NN = (size_t)d.N * d.N;
  const int N = d.N, GG = d.G * d.G;
  const VT2 *const tabs = reinterpret_cast<const VT2 *>(d.gcf) + sl;
  const u64 minus_one = pk2(-1.f, -1.f);
  // Few visibilities: every warp an equal share, in steps of VPW (160 k of
  // support 8: 20.4 -> 17.9 us, 10 k of support 16 24 -> 9.8).  From four groups
  // of 32 a warp on, the groups go round the warps: neighbouring ones share
  // cells (1 M: the same; 4.19 M: 344 us, in shares 387).
  const bool shares = d.npts < nwarps * 32 * 4;
  const int64_t steps = (d.npts + VPW - 1) / VPW;
  const int64_t end = shares ? min(d.npts, steps * (warp + 1) / nwarps * VPW) : d.npts;
  const int64_t stride = shares ? 32 : nwarps * 32;
  for (int64_t base = shares ? steps * warp / nwarps * VPW : warp * 32; base < end;
       base += stride) {
    // one visibility per lane: first cell of its footprint and sub-kernel (of
    // all tables; -1: dropped)
    int fx = 0, fy = 0, sub = -1;
    if (base + lane < end) {
      int sx, sy, mx, my, tab = 0;
      bool ok = uv_step(d.uv, d.uv_f64, base + lane, d.G, mx, sx, my, sy) &&
                (unsigned)sx < (unsigned)d.G && (unsigned)sy < (unsigned)d.G;
      if (ok && d.gcf_index) {
        tab = __ldg(d.gcf_index + base + lane);
        ok = (unsigned)tab < (unsigned)d.n_gcf;
      }
      if (ok) {
        fx = mx - S / 2 + 1;
        fy = my - S / 2 + 1;
        sub = tab * GG + sy * d.G + sx;
      } else {
        atomicAdd(&d.flags[FLAG_INDEX], 1);
      }
    }
#pragma unroll 1
    for (int it = 0; it < S && base + it * VPW < end; ++it) {
      const int src = it * VPW + sv;
      const int x0 = __shfl_sync(0xffffffffu, fx, src), y0 = __shfl_sync(0xffffffffu, fy, src);
      const int k = __shfl_sync(0xffffffffu, sub, src);
      const bool inside = k >= 0 && x0 >= 0 && y0 >= 0 && x0 + S <= N && y0 + S <= N;
      const bool all_in = __all_sync(0xffffffffu, inside);
      // cells of this lane's column; rows off the grid are not read
      const bool col = k >= 0 && (unsigned)(x0 + sl) < (unsigned)N;
      const int64_t cell0 = (int64_t)y0 * N + (x0 + sl);
      const VT2 *const w0 = tabs + (int64_t)(k < 0 ? 0 : k) * (S * S);
      const int sy = GK == 1 ? (k < 0 ? 0 : k / d.G) : 0;
      const float gx = GK == 1 ? g1[(k < 0 ? 0 : k - sy * d.G) * S + sl] : 0.f;
      for (int p = 0; p < d.P; ++p) {
        u64 run = 0ull, hi = 0ull, lo = 0ull;  // FP32: plain, or (hi, lo)
        auto put = [&](u64 t) {
          u64 e;
          hi = two_sum2(hi, t, e);
          lo = add2(lo, e);
        };
        VT re = 0, im = 0;                     // FP64
        bool force = false;
        rows:
#pragma unroll 1
        for (int b0 = 0; b0 < S; b0 += R) {
          VT2 c[R], w[R];
          auto load = [&](auto checked, auto planar) {
            const GT *const g = reinterpret_cast<const GT *>(d.grid);
#pragma unroll
            for (int b = 0; b < R; ++b) {
              const int64_t at = cell0 + (int64_t)(b0 + b) * N;
              const bool on = !decltype(checked)::value ||
                              (col && (unsigned)(y0 + b0 + b) < (unsigned)N);
              c[b].x = c[b].y = (VT)0;
              if constexpr (decltype(planar)::value) {
                if (on) {
                  c[b].x = (VT)__ldg(g + (size_t)p * NN + at);
                  c[b].y = (VT)__ldg(g + (size_t)(d.P + p) * NN + at);
                }
              } else if (on) {
                const GT2 v = __ldg(reinterpret_cast<const GT2 *>(g) + (size_t)p * NN + at);
                c[b].x = (VT)v.x;
                c[b].y = (VT)v.y;
              }
              if constexpr (GK == 1) {
                w[b].x = on ? (VT)(gx * g1[sy * S + b0 + b]) : (VT)0;
                w[b].y = (VT)0;
              } else {
                w[b].x = w[b].y = (VT)0;
                if (on) w[b] = __ldg(w0 + (b0 + b) * S);
              }
            }
          };
          if (d.planar) {
            if (all_in) load(std::false_type{}, std::true_type{});
            else load(std::true_type{}, std::true_type{});
          } else {
            if (all_in) load(std::false_type{}, std::false_type{});
            else load(std::true_type{}, std::false_type{});
          }
          // any factor with an imaginary part: both products
          bool full = force;
          if constexpr (GK != 1) {
#pragma unroll
            for (int b = 0; b < R; ++b) full = full || w[b].y != (VT)0;
          }
          auto sum = [&](auto real) {
#pragma unroll
            for (int b = 0; b < R; ++b) {
              // grid * conj(w)
              if constexpr (F32) {
                const u64 c1 = pk2(c[b].x, c[b].y), g1 = pk2(w[b].x, w[b].x);
                if constexpr (!COMP) {
                  run = fma2(c1, g1, run);
                  if constexpr (!decltype(real)::value)
                    run = fma2(pk2(c[b].y, -c[b].x), pk2(w[b].y, w[b].y), run);
                } else if constexpr (decltype(real)::value) {
                  if (b & 1) continue;
                  // two taps t, and what their sum lost: of -t + c1 g1 + c2 g2 only
                  // the first addition rounds to the size of a tap
                  const u64 c2 = pk2(c[b + 1].x, c[b + 1].y), g2 = pk2(w[b + 1].x, w[b + 1].x);
                  const u64 t = fma2(c2, g2, mul2(c1, g1));
                  put(t);
                  lo = add2(lo, fma2(c2, g2, fma2(c1, g1, mul2(t, minus_one))));
                } else {
                  put(fma2(pk2(c[b].y, -c[b].x), pk2(w[b].y, w[b].y), mul2(c1, g1)));
                }
              } else {
                re += c[b].x * w[b].x;
                im += c[b].y * w[b].x;
                if constexpr (!decltype(real)::value) {
                  re += c[b].y * w[b].y;
                  im -= c[b].x * w[b].y;
                }
              }
            }
          };
          if (__any_sync(0xffffffffu, full)) sum(std::false_type{});
          else sum(std::true_type{});
        }
        // a sum that is not finite (0 * c matters then): both products
        if (GK != 1 && !force) {
          bool fine;
          if constexpr (F32) {
            const float2 z = upk2(fma2(COMP ? hi : run, 0ull, 0ull));
            fine = z.x == 0.f && z.y == 0.f;
          } else {
            fine = re - re == 0.0 && im - im == 0.0;
          }
          if (!__all_sync(0xffffffffu, fine)) {
            run = hi = lo = 0ull;
            re = im = 0;
            force = true;
            goto rows;
          }
        }
        // even lanes go on with the real, odd ones with the imaginary parts
        const bool odd = sl & 1;
        LaneSum<VT, COMP> t;
        VT oh, ol = 0;
        if constexpr (F32) {
          const float2 h = upk2(COMP ? hi : run), l = upk2(lo);
          t.h = odd ? h.y : h.x;
          t.l = odd ? l.y : l.x;
          oh = odd ? h.x : h.y;
          ol = odd ? l.x : l.y;
        } else {
          t.h = odd ? im : re;
          oh = odd ? re : im;
        }
        oh = __shfl_xor_sync(0xffffffffu, oh, 1);
        if constexpr (COMP) ol = __shfl_xor_sync(0xffffffffu, ol, 1);
        t.merge(oh, ol);
#pragma unroll
        for (int o = 2; o < S; o <<= 1) t.merge_lane(o);
        if (sl < 2 && base + src < end)
          reinterpret_cast<VT *>(d.vals)[2 * ((size_t)(base + src) * d.P + p) + sl] = t.value();
      }
    }
  }
}

template <int S, typename VT, typename GT>
cudaError_t degrid_kinds(const DegridLaunch &d, unsigned blocks, cudaStream_t s) {
  constexpr bool F32 = std::is_same<VT, float>::value;
  if (d.gauss) {
    if (F32 && d.compensated) degrid_kernel<S, VT, GT, 1, F32><<<blocks, 256, 0, s>>>(d);
    else degrid_kernel<S, VT, GT, 1, false><<<blocks, 256, 0, s>>>(d);
  } else {
    if (F32 && d.compensated) degrid_kernel<S, VT, GT, 0, F32><<<blocks, 256, 0, s>>>(d);
    else degrid_kernel<S, VT, GT, 0, false><<<blocks, 256, 0, s>>>(d);
  }
  count_launch();
  return cudaGetLastError();
}

template <int S>
cudaError_t degrid_types(const DegridLaunch &d, unsigned blocks, cudaStream_t s) {
  if (d.vals_f64)
    return d.grid_f64 ? degrid_kinds<S, double, double>(d, blocks, s)
                      : degrid_kinds<S, double, float>(d, blocks, s);
  return d.grid_f64 ? degrid_kinds<S, float, double>(d, blocks, s)
                    : degrid_kinds<S, float, float>(d, blocks, s);
}

}  // namespace

cudaError_t launch_degrid(const DegridLaunch &d, cudaStream_t s) {
  if (d.npts <= 0) return cudaSuccess;
  // a step for every warp, until the resident CTAs are reached
  const int64_t steps = (d.npts + 32 / d.S - 1) / (32 / d.S), b = (steps + 7) / 8;
  const int64_t cap = (int64_t)d.sm_count * kDegridCtas;
  const unsigned blocks = (unsigned)(b < 1 ? 1 : (b > cap ? cap : b));
  switch (d.S) {
    case 4: return degrid_types<4>(d, blocks, s);
    case 8: return degrid_types<8>(d, blocks, s);
    case 16: return degrid_types<16>(d, blocks, s);
    case 32: return degrid_types<32>(d, blocks, s);
  }
  return cudaErrorInvalidValue;
}

}  // namespace gg
