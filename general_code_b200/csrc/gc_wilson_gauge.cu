// On-axis Wilson loops W(R,T) in the temporal gauge (sm_100a).
//
// Reference: wilson_loop (wilson_loops.h:1047-1074) averages, over x and the
// spatial directions nu, the loop
//     Re Tr[S(x,R) L(x+R nu,T) S(x+T t,R)^dag L(x,T)^dag] / N
// with time lines L(x,T) = U_t(x) U_t(x+t) ... U_t(x+(T-1)t) and space lines
// S(x,R) = U_nu(x) ... U_nu(x+(R-1)nu).
//
// The loop is gauge invariant. With G(s,t) the time line of spatial site s
// from slice 0 up to slice t (G(s,0) = 1, G(s,t+1) = G(s,t) U_t(s,t)),
// continued past the last slice with the periodic links (G(s,Lt+j) =
// W(s) G(s,j), W(s) the line over the whole extent), every time line is
// L(s;t0,T) = G(s,t0)^dag G(s,t0+T) when the temporal links are unitary, and
// the loop becomes
//     Re Tr[S'(x,R) S'(x+T t,R)^dag] / N,
//     S'(s,t,R) = G(s,t) S(s,t,R) G(s+R nu,t)^dag
//               = U'_nu(s,t) ... U'_nu(s+(R-1)nu,t),
//     U'_nu(s,t) = G(s,t) U_nu(s,t) G(s+nu,t)^dag
// with the transformed links on the slices 0 .. Lt-1 and, for the loops that
// pass the last slice, on T_max further ones. A loop then costs one 9-element
// trace instead of two matrix products (the T walk of the exact recursion in
// gc_wilson.cu), and each space line one product per R. (Two cuts of Lt
// slices each, with the second for the loops that pass the first, took 2 Lt
// lines per column instead of Lt + T_max: at SU(3) 32^4 FP64 a third more
// shared memory and products.)
//
// The identity needs unitary temporal links. The lines kernel measures the
// unitarity defects d = max |U_t U_t^dag - 1| of the lattice's temporal links
// and raises a flag when a block's links (32 columns) exceed the form's
// tolerance in the mean (FP64: 1e-14, a few roundings) or one of them exceeds
// 1e-12 (a time slab: 1e-14); mixed: when one exceeds 1e-6 (FP32 rounding of
// the 12-real links is 2.6e-7); for 12-real links the transform kernel checks
// the spatial links as well. (The mean, since W averages over all loops and every link enters as
// many of them: one link past 1e-14 in a configuration, as an
// orthonormalisation of nearly parallel rows leaves it, took the exact
// product for all loops, 21 ms instead of 5.8 for the spatial loops of SU(3)
// 24^4 FP64, for a difference below 1e-18.)
// Both W kernels are launched and read the flag on the device: the exact
// product (gc_wilson.cu) computes when it is raised, this form when it is
// not, and the reduction sums the partials of the one that ran; no host
// synchronisation, so the sequence can be captured in a graph. With a
// defect d per link a loop differs from the reference's product of links by at
// most about 2 T d (the two time lines), well inside the parity tolerances.
//
// Kernels:
//   gauge_lines_kernel      thread per spatial site: G(s,t), W(s) and the
//                           defect (FP64, stored as FP64 fields)
//   gauge_transform_kernel  thread per (extended site, spatial nu): U'_nu,
//                           computed in FP64, stored in the lattice's link
//                           format
//   wilson_corr_kernel      (gc_wilson_corr.cu) fundamental loops as
//                           correlations of the lines' elements along t
//   wilson_gram_kernel      (gc_wilson_gram.cu) FP64 fundamental loops of long
//                           T ranges, and the GEVP loops, as FP64 matrix
//                           products
//   wilson_gauge_reg_kernel mixed SU(3), and
//   wilson_gauge_q_kernel   SU(2) fundamental loops of few slices and T: one
//                           column per thread, the lines of its four start
//                           slices in registers (gauge_short_applies has the line)
//   wilson_gauge_kernel     the adjoint loops (|Tr|^2 is no bilinear form of
//                           the lines): block = `cols` columns (s, nu) over
//                           all slices, the transformed space lines in shared
//                           memory, extended by one link per R; a thread per
//                           (column unit, 1, 2 or 4 start slices) adds its
//                           loops for every T into a per-thread slot
// The last three sum their per-thread slots over the block in fixed order; one
// partial per (block, R, T), and the fixed-order tree over blocks of
// gc_wilson.cu finishes.
#include "gc_internal.cuh"
#include "gc_kernels.h"
#include "gc_pair.cuh"
#include "gc_rows01.cuh"
#include "gc_wcol.cuh"

#include <algorithm>
#include <type_traits>

namespace gc {

namespace {

template <int NC> struct F64Store;
template <> struct F64Store<3> {
  using type = StoreF64SU3;
};
template <> struct F64Store<2> {
  using type = StoreF64SU2;
};

// max_ij |(U U^dag - 1)_ij|
__device__ __forceinline__ double unitarity_defect(const SU3<double> &u) {
  double d = 0.0;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = i; j < 3; j++) {
      double re = 0.0, im = 0.0;
#pragma unroll
      for (int k = 0; k < 3; k++) {
        re = fma(u.e[i][k].re, u.e[j][k].re, re);
        re = fma(u.e[i][k].im, u.e[j][k].im, re);
        im = fma(u.e[i][k].im, u.e[j][k].re, im);
        im = fma(-u.e[i][k].re, u.e[j][k].im, im);
      }
      if (i == j)
        re -= 1.0;
      d = fmax(d, fmax(fabs(re), fabs(im)));
    }
  return d;
}
// SU(2) quaternion a0 + i a.sigma: U U^dag = |a|^2 1
__device__ __forceinline__ double unitarity_defect(const SU2<double> &u) {
  return fabs(dot4(u.a0, u.a0, u.a1, u.a1, u.a2, u.a2, u.a3, u.a3) - 1.0);
}

__device__ __forceinline__ double row_sum(const SU3<double> &u) {
  return (u.e[0][0].re + u.e[0][1].re) + u.e[0][2].re;
}
__device__ __forceinline__ double row_sum(const SU2<double> &u) { return u.a0; }

// The temporal link the gauge lines are built from. FP64 links are unitary to
// rounding. An FP32 link's last projection step leaves its singular values
// 1 - O(d^2) (d the defect before that step, up to 2e-5), a shrink of up to a
// few 1e-10 with one sign; through G^dag G != 1 it entered every transformed
// link, and W's error against FP64 grew linearly in R and T (3.4e-8 at 24^4,
// R,T = 12, against 4.3e-9 for the exact product). One FP64 Newton-Schulz
// step (SU(2): a / |a|) makes the link unitary to FP64 rounding; it moves
// the link by that shrink only, well inside the FP32 rounding of the stored
// link.
template <class Store>
__device__ __forceinline__ typename Store::template M<double> gauge_time_link(
    const typename Store::template M<double> &u) {
  if constexpr (Store::kBytes == 48 || Store::kBytes == 72)
    return ns_step(u);
  else if constexpr (Store::kBytes == 16)
    return proj(u);
  else
    return u;
}

// The stored SU(3) lines are made unitary once more: G^dag stands for G^-1,
// and over a long time extent the links' and the products' rounding adds up
// (1e-14 at Lt = 40, in the loops' values as well; W's error against 64 bits
// at 24^4 FP64 9e-15 -> 9e-16). A quaternion's norm does not drift that way.
__device__ __forceinline__ SU3<double> stored_line(const SU3<double> &G) { return polar_step(G); }
__device__ __forceinline__ SU2<double> stored_line(const SU2<double> &G) { return G; }
//
// The chain over t is serial: the next two links are loaded ahead. Where the
// columns alone leave most of the chip idle (a 16^3 slice has 4096) a column's
// slices are split into kLinesSegs segments of warps: each multiplies its own
// slices' links and keeps the partial lines, the segments' products meet in
// shared memory, and each then puts the product of the earlier segments in
// front of its partial lines. Four segments against one: 7.3 / 12.8 us at
// SU(2) 16^4 FP64, 30.4 / 29.5 at SU(3) 24^4 FP64, 82 / 73 at SU(3) 32^4
// mixed, so below 8192 columns only.
constexpr int kLinesCols = 32;

// Records of the line fields, read back by the thread that wrote them (not
// through the read-only path of the link loads).
__device__ __forceinline__ SU3<double> line_back(const void *f, size_t V, int site, SU3<double> *) {
  const double2 *p = reinterpret_cast<const double2 *>(f) + site;
  SU3<double> m;
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 v = p[k * V];
    m.e[k / 3][k % 3] = {v.x, v.y};
  }
  return m;
}
__device__ __forceinline__ SU2<double> line_back(const void *f, size_t V, int site, SU2<double> *) {
  const double2 *p = reinterpret_cast<const double2 *>(f) + site;
  const double2 a = p[0], b = p[V];
  return {a.x, a.y, b.x, b.y};
}

//
// MAPPED: the loops' time axis is a spatial axis of the lattice; g is the
// lattice with its axes reordered (the columns' three, then the time axis),
// which the lines and transformed links are stored on, and map gives the
// strides of the links' own site order.
template <bool MAPPED>
__device__ __forceinline__ int own_site(const Geom &g, const AxisMap &map, int site) {
  if (!MAPPED)
    return site;
  int x[4];
  site_coords(g, site, x);
  return x[0] * map.stride[0] + x[1] * map.stride[1] + x[2] * map.stride[2] + x[3] * map.stride[3];
}

template <class Store, int kLinesSegs, bool MAPPED>
__global__ void __launch_bounds__(kLinesCols *kLinesSegs)
    gauge_lines_kernel(const __grid_constant__ Geom g, const __grid_constant__ AxisMap map,
                       const void *Ut, void *GL, void *W, double tol, double most, int *flag) {
  wait_previous();
  using GS = typename F64Store<Store::NC>::type;
  using MD = typename Store::template M<double>;
  __shared__ MD total[kLinesSegs][kLinesCols];
  __shared__ double defects[kLinesSegs];
  const int c = threadIdx.x % kLinesCols, seg = threadIdx.x / kLinesCols;
  const int s = blockIdx.x * kLinesCols + c;
  const bool active = s < g.Vs;
  const size_t V = g.V;
  const int Lt = g.L[3], len = (Lt + kLinesSegs - 1) / kLinesSegs;
  const int t0 = min(Lt, seg * len), t1 = min(Lt, t0 + len);
  double dmax = 0.0, dsum = 0.0;
  MD G = unit(MD());
  if (active && t0 < t1) {
    const int base = own_site<MAPPED>(g, map, s), step = MAPPED ? map.stride[3] : g.Vs;
    auto link = [&](int t) {
      return Store::template load<double>(Ut, V, base + min(t, t1 - 1) * step);
    };
    MD u = link(t0), next = link(t0 + 1);
#pragma unroll 1
    for (int t = t0; t < t1; t++) {
      const MD after = link(t + 2);
      GS::template store<double>(GL, V, s + t * g.Vs, seg ? G : stored_line(G));
      const double d = unitarity_defect(u);
      dmax = fmax(dmax, d);
      dsum += d;
      G = mul(G, gauge_time_link<Store>(u));
      u = next;
      next = after;
    }
  }
  total[seg][c] = G;
  // (0 x G: NaN when a link was, whose defect's maximum may have dropped it)
  const double sum = warp_sum(fma(0.0, row_sum(G), dsum));
  if (c == 0)
    defects[seg] = sum;
  if (!(dmax <= most))
    *flag = 1;
  __syncthreads();
  if (threadIdx.x == 0) { // the mean over the block's links
    double mean = 0.0;
    for (int q = 0; q < kLinesSegs; q++)
      mean += defects[q];
    if (!(mean <= tol * min(kLinesCols, g.Vs - s) * Lt))
      *flag = 1;
  }
  if (!active)
    return;
  if (kLinesSegs == 1)
    GS::template store<double>(W, g.Vs, s, stored_line(G));
  if (seg == 0)
    return;
  MD before = total[0][c];
#pragma unroll 1
  for (int q = 1; q < seg; q++)
    before = mul(before, total[q][c]);
#pragma unroll 2
  for (int t = t0; t < t1; t++)
    GS::template store<double>(
        GL, V, s + t * g.Vs,
        stored_line(mul(before, line_back(GL, V, s + t * g.Vs, (MD *)nullptr))));
  if (seg == kLinesSegs - 1)
    GS::template store<double>(W, g.Vs, s, stored_line(mul(before, G)));
}

// U'_nu(s,te) = G(s,te) U_nu(s,te mod Lt) G(s+nu,te)^dag on the slices te of
// the extended lattice (sites [0, NE Vs), plane stride NE Vs), stored as Out;
// thread per (site, nu). Nothing where the lines raised the flag (the loops are
// not computed from these links then).
template <class Store, class Out, bool MAPPED>
__global__ void __launch_bounds__(128)
    gauge_transform_kernel(const __grid_constant__ Geom g, const __grid_constant__ AxisMap map,
                           const __grid_constant__ Fields4 U, const void *GL, const void *W,
                           const __grid_constant__ Fields4 UE, int NE, double tol, int *flag) {
  wait_previous();
  if (*flag != 0)
    return;
  using GS = typename F64Store<Store::NC>::type;
  using MD = typename Store::template M<double>;
  const int esite = blockIdx.x * blockDim.x + threadIdx.x;
  const int VE = NE * g.Vs;
  if (esite >= VE)
    return;
  const int nu = blockIdx.y;
  const bool past = esite >= g.V; // a slice past the last one
  const int site = past ? esite - g.V : esite;
  int x[4];
  site_coords(g, site, x);
  const int off = step_off(g, sel4(x, nu), nu, +1);
  const size_t V = g.V;
  const MD u = Store::template load<double>(U.f[nu], V, own_site<MAPPED>(g, map, site));
  // 12-real links: the transformed link's third row is rebuilt from its first
  // two, which holds for links in SU(3) only
  if (Out::kBytes == 48 && !past && !(unitarity_defect(u) <= tol))
    *flag = 1;
  MD a = mul(GS::template load<double>(GL, V, site), u);
  MD b = GS::template load<double>(GL, V, site + off);
  if (past) {
    const int s = site % g.Vs;
    a = mul(GS::template load<double>(W, g.Vs, s), a);
    b = mul(GS::template load<double>(W, g.Vs, s + off), b);
  }
  Out::template store<double>(UE.f[nu], VE, esite, mul_ad(a, b));
}

// The adjoint loops. Shared memory of one block: per-thread loop sums
// red[nt][threads] (FP64),
// then the space lines, one slot per (slice, column unit) over the NE slices.
// KS > 1: a thread owns KS consecutive start slices t0 = KS row + m, m < KS
// (KS divides Lt), and one shared-memory load of
// a top space line S(t) serves the loops of all of them that end on t
// (T = t - t0 - m): nt + KS - 1 loads for KS nt loops, the sums of the last
// KS values of T kept in registers. KS = 1: a thread owns the slices
// row + k rows and loads one line per loop.
// SLAB compiles in the check that a start is counted (t0 < tstarts, a time
// slab). A top line past the last slice belongs to an uncounted loop: its slot
// is clamped.
template <class Store, class CT, int KS, bool SLAB>
__global__ void __launch_bounds__(256)
    wilson_gauge_kernel(const __grid_constant__ Geom g, const __grid_constant__ Fields4 U,
                        int NE, int rmin, int rmax, int tmin, int tmax, int cols, int rows,
                        double *partials, const int *flag, int tstarts) {
  wait_previous();
  // the exact product runs instead when a temporal link failed the check
  if (flag && *flag != 0)
    return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  constexpr int LANES = wilson_lanes(Store::NC, sizeof(CT));
  using LL = LaneLoad<Store, CT, LANES>;
  using M = typename LL::M;
  using CS = ColSet<M>;
  const int Lt = g.L[3];
  const int nt = tmax - tmin + 1;
  const int nthreads = blockDim.x;
  const int cs = wilson_col_stride(cols, LANES);
  const int units = cs / LANES;
  const int nslots = NE * units;
  using Acc = double;
  Acc *red = reinterpret_cast<Acc *>(smem_raw); // [nt][nthreads]
  unsigned char *sa = smem_raw + ((sizeof(Acc) * nt * nthreads + 15) & ~(size_t)15);

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, nwarps = nthreads >> 5;
  const int u = tid % units;
  const int row = tid / units;
  const int nu = blockIdx.y;
  const int s0 = column_base(g, blockIdx.x, cols, nu) + LANES * u;
  const bool active = (row < rows) && (s0 < g.Vs);
  const bool lane1 = LANES == 2 && active && (LANES * u + 1 < cols) && (s0 + 1 < g.Vs);
  const int s1 = lane1 ? s0 + 1 : s0;
  const int kt = Lt / rows;
  const int Ln = sel4(g.L, nu), stn = sel4(g.stride, nu);
  const int xn0 = (s0 / stn) % Ln, xn1 = (s1 / stn) % Ln;
  const size_t VE = (size_t)NE * g.Vs;
  const int ne = (rmax - rmin + 1) * nt;
  double *part = partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * ne;

#pragma unroll 1
  for (int R = 1; R <= rmax; R++) {
    // extend the space lines by the link at x + (R-1) nu: the thread's start
    // slices, and its share of the slices past the last one
    if (active) {
      const int l0 = s0 + ((xn0 + R - 1) % Ln - xn0) * stn;
      const int l1 = s1 + ((xn1 + R - 1) % Ln - xn1) * stn;
#pragma unroll 1
      for (int k = 0; k < kt + (NE - Lt + rows - 1) / rows; k++) {
        const int t = k >= kt ? Lt + row + (k - kt) * rows : KS > 1 ? KS * row + k : row + k * rows;
        if (t >= NE)
          break;
        const int i = t * units + u;
        const M la = LL::load(U.f[nu], VE, l0 + t * g.Vs, l1 + t * g.Vs);
        CS::store(sa, nslots, i, R == 1 ? la : mul(CS::load(sa, nslots, i), la));
      }
    }
    __syncthreads();
    if (R >= rmin && KS > 1) {
      const int t0 = KS * row;
      M a[KS];
#pragma unroll
      for (int m = 0; m < KS; m++)
        a[m] = active ? CS::load(sa, nslots, (t0 + m) * units + u) : unit(M());
      int tt = min(t0 + tmin, NE - 1);
      Acc acc[KS]; // acc[m]: the sum for T index j - m
#pragma unroll
      for (int m = 0; m < KS; m++)
        acc[m] = Acc(0);
      // One step of the sweep: the loops of all starts that end on top line
      // b (index j), then the completed sum of T index j - KS + 1.
      auto step = [&](int j, const M &b) {
        if (active) {
#pragma unroll
          for (int m = 0; m < KS; m++)
            if (j - m >= 0 && j - m < nt && (!SLAB || t0 + m < tstarts)) // T = tmin + j - m
              acc[m] += gauge_trace<true>(a[m], b, lane1);
        }
        if (j - (KS - 1) >= 0) // T index j - KS + 1 has all KS starts
          red[(size_t)(j - (KS - 1)) * nthreads + tid] = acc[KS - 1];
#pragma unroll
        for (int m = KS - 1; m > 0; m--)
          acc[m] = acc[m - 1];
        acc[0] = Acc(0);
      };
      // two top lines in flight (b0, b1 alternate): the next line's load is
      // issued before the current line's traces (past the last step the
      // clamped slot's line is unused; inactive threads use no line)
      const int nsteps = nt + KS - 1;
      M b0, b1;
      if (active)
        b0 = CS::load(sa, nslots, tt * units + u);
#pragma unroll 1
      for (int j = 0; j < nsteps; j += 2) {
        tt = min(tt + 1, NE - 1);
        if (active)
          b1 = CS::load(sa, nslots, tt * units + u);
        step(j, b0);
        tt = min(tt + 1, NE - 1);
        if (active)
          b0 = CS::load(sa, nslots, tt * units + u);
        if (j + 1 < nsteps)
          step(j + 1, b1);
      }
    } else if (R >= rmin) {
#pragma unroll 1
      for (int k = 0; k < kt; k++) {
        const int t0 = row + k * rows;
        const M a = active ? CS::load(sa, nslots, t0 * units + u) : unit(M());
        int tt = min(t0 + tmin, NE - 1);
#pragma unroll 1
        for (int T = 0; T < nt; T++) {
          const Acc v =
              (active && (!SLAB || t0 < tstarts)) ? gauge_trace<true>(a, CS::load(sa, nslots, tt * units + u), lane1) : Acc(0);
          Acc *r = red + (size_t)T * nthreads + tid;
          *r = (k == 0) ? v : *r + v;
          tt = min(tt + 1, NE - 1);
        }
      }
    }
    if (R >= rmin) {
      __syncthreads();
      // fixed-order sum over the block's threads: warp w takes T = w, w +
      // nwarps, ...; each lane sums a strided subset, then a warp tree
#pragma unroll 1
      for (int T = warp; T < nt; T += nwarps) {
        double v = 0.0;
        for (int i = lane; i < nthreads; i += 32)
          v += double(red[(size_t)T * nthreads + i]);
        v = warp_sum(v);
        if (lane == 0)
          part[(R - rmin) * nt + T] = v;
      }
    }
    __syncthreads();
  }
}

// Shared-memory record of an FP32 SU(3) space line for the one-column kernel
// below: rows 0 and 1 (row 2 = conj(row0 x row1) is rebuilt where a trace
// needs it), 48 bytes moved as three 16-byte vectors at immediate offsets, in
// the element order of the stored links (StoreF32SU3). Consecutive threads
// hold consecutive records (a 12-word stride), so each quarter-warp phase of a
// 16-byte access covers the 32 banks once.
struct Rows01Set {
  static constexpr int kBytes = 48;
  __device__ __forceinline__ static void store(unsigned char *set, int i, const SU3<float> &m) {
    float4 *p = reinterpret_cast<float4 *>(set + (size_t)kBytes * i);
    p[0] = make_float4(m.e[0][0].re, m.e[0][0].im, m.e[0][1].re, m.e[0][1].im);
    p[1] = make_float4(m.e[0][2].re, m.e[0][2].im, m.e[1][0].re, m.e[1][0].im);
    p[2] = make_float4(m.e[1][1].re, m.e[1][1].im, m.e[1][2].re, m.e[1][2].im);
  }
  // rows 0 and 1 (row 2 not set)
  __device__ __forceinline__ static SU3<float> load(const unsigned char *set, int i) {
    const float4 *p = reinterpret_cast<const float4 *>(set + (size_t)kBytes * i);
    const float4 a = p[0], b = p[1], c = p[2];
    SU3<float> m;
    m.e[0][0] = {a.x, a.y};
    m.e[0][1] = {a.z, a.w};
    m.e[0][2] = {b.x, b.y};
    m.e[1][0] = {b.z, b.w};
    m.e[1][1] = {c.x, c.y};
    m.e[1][2] = {c.z, c.w};
    return m;
  }
};

// The fundamental loops of the mixed SU(3) form with one column per thread
// and KS consecutive start slices t0 = KS row + m whose space lines stay in
// registers from one R to the next. The trace sweep reads each top line once for the KS starts, as in
// wilson_gauge_kernel, but the lines are not lane-packed, so KS = 4 starts
// fit in the registers: twice the loops per shared-memory byte of the
// two-column, two-start form. Each R the thread extends its own starts' lines
// in registers (and stores them for the other threads' sweeps) and its share
// of the lines past slice KS rows - 1 in shared memory. Lines are products of
// SU(3) links, so they are computed and kept in shared memory as rows 0 and 1
// (48 bytes a line instead of 72; 72 instead of 108 multiply-adds a product),
// and row 2 is rebuilt where a trace needs it. Compiled for 16 warps per SM
// (128 registers, a few spilled): 8 warps at 175 registers took a fifth more.
// Bound by the FMA pipe's operands and the latency of the sweep (0.6
// instructions per cycle and scheduler). With one set of Lt + T_max lines
// instead of two cuts of Lt: 24^3 x 48, T <= 12, 1.42 -> 1.34 ms (a size that
// wilson_corr_kernel has now, 1.04 ms at T <= 24).
// Partials, block sums and the per-thread FP32 loop sums as
// wilson_gauge_kernel.
template <int KS, bool SLAB>
__global__ void __launch_bounds__(256, 2)
    wilson_gauge_reg_kernel(const __grid_constant__ Geom g, const __grid_constant__ Fields4 U,
                            int NE, int rmin, int rmax, int tmin, int tmax, int cols, int rows,
                            double *partials, const int *flag, int tstarts) {
  wait_previous();
  if (flag && *flag != 0)
    return;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nt = tmax - tmin + 1;
  const int nthreads = blockDim.x;
  float *red = reinterpret_cast<float *>(smem_raw); // [nt][nthreads]
  unsigned char *sa = smem_raw + ((sizeof(float) * nt * nthreads + 15) & ~(size_t)15);

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, nwarps = nthreads >> 5;
  const int u = tid % cols;
  const int row = tid / cols;
  const int nu = blockIdx.y;
  const int s0 = column_base(g, blockIdx.x, cols, nu) + u;
  const bool active = (row < rows) && (s0 < g.Vs);
  const int t0 = KS * row;
  const void *f = U.f[nu];
  const int Ln = sel4(g.L, nu), stn = sel4(g.stride, nu);
  const int xn = (s0 / stn) % Ln;
  const size_t VE = (size_t)NE * g.Vs;
  const int ne = (rmax - rmin + 1) * nt;
  double *part = partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * ne;

  SU3<float> a[KS];
#pragma unroll 1
  for (int R = 1; R <= rmax; R++) {
    // extend the lines by the link at x + (R-1) nu
    if (active) {
      const int l = s0 + ((xn + R - 1) % Ln - xn) * stn;
#pragma unroll
      for (int m = 0; m < KS; m++) {
        const int t = t0 + m;
        if (t >= NE)
          break;
        const SU3<float> lo = StoreF32SU3::load<float>(f, VE, l + t * g.Vs);
        if (R == 1) {
          a[m] = lo;
        } else {
          // rows 0 and 1 of the product; row 2 rebuilt for the traces
          a[m] = mul01(a[m], lo);
          rebuild_row2(a[m]);
        }
        Rows01Set::store(sa, t * cols + u, a[m]);
      }
#pragma unroll 1
      for (int t = KS * rows + row; t < NE; t += rows) {
        const int i = t * cols + u;
        const SU3<float> lx = StoreF32SU3::load<float>(f, VE, l + t * g.Vs);
        Rows01Set::store(sa, i, R == 1 ? lx : mul01(Rows01Set::load(sa, i), lx));
      }
    }
    __syncthreads();
    if (R >= rmin) {
      int tt = min(t0 + tmin, NE - 1);
      float acc[KS]; // acc[m]: the sum for T index j - m
#pragma unroll
      for (int m = 0; m < KS; m++)
        acc[m] = 0.f;
      // the loops of all starts that end on top line b (index j), then the
      // completed sum of T index j - KS + 1
      auto step = [&](int j, const SU3<float> &b) {
        if (active) {
#pragma unroll
          for (int m = 0; m < KS; m++)
            if (j - m >= 0 && j - m < nt && (!SLAB || t0 + m < tstarts)) // T = tmin + j - m
              acc[m] += gauge_trace<false>(a[m], b, false);
        }
        if (j - (KS - 1) >= 0)
          red[(size_t)(j - (KS - 1)) * nthreads + tid] = acc[KS - 1];
#pragma unroll
        for (int m = KS - 1; m > 0; m--)
          acc[m] = acc[m - 1];
        acc[0] = 0.f;
      };
      // two top lines in flight (b0, b1 alternate)
      const int nsteps = nt + KS - 1;
      SU3<float> b0, b1;
      if (active)
        b0 = Rows01Set::load(sa, tt * cols + u);
#pragma unroll 1
      for (int j = 0; j < nsteps; j += 2) {
        tt = min(tt + 1, NE - 1);
        if (active)
          b1 = Rows01Set::load(sa, tt * cols + u);
        rebuild_row2(b0);
        step(j, b0);
        tt = min(tt + 1, NE - 1);
        if (active)
          b0 = Rows01Set::load(sa, tt * cols + u);
        if (j + 1 < nsteps) {
          rebuild_row2(b1);
          step(j + 1, b1);
        }
      }
      __syncthreads();
      // fixed-order sum over the block's threads (as wilson_gauge_kernel)
#pragma unroll 1
      for (int T = warp; T < nt; T += nwarps) {
        double v = 0.0;
        for (int i = lane; i < nthreads; i += 32)
          v += double(red[(size_t)T * nthreads + i]);
        v = warp_sum(v);
        if (lane == 0)
          part[(R - rmin) * nt + T] = v;
      }
    }
    __syncthreads();
  }
}

// Shared-memory records of SU(2) space lines (quaternions) for the SU(2)
// one-column kernel: FP32 one 16-byte vector per slot; FP64 two planes of
// 16-byte (a0, a1) and (a2, a3) pairs. A quarter-warp phase of 8 consecutive
// slots reads 128 contiguous bytes of a plane: conflict-free when the block's
// columns are a multiple of 8.
template <class T> struct QuatSet;
template <> struct QuatSet<float> {
  static constexpr int kBytes = 16;
  __device__ __forceinline__ static void store(unsigned char *set, int, int i,
                                               const SU2<float> &q) {
    reinterpret_cast<float4 *>(set)[i] = make_float4(q.a0, q.a1, q.a2, q.a3);
  }
  __device__ __forceinline__ static SU2<float> load(const unsigned char *set, int, int i) {
    const float4 v = reinterpret_cast<const float4 *>(set)[i];
    return {v.x, v.y, v.z, v.w};
  }
};
template <> struct QuatSet<double> {
  static constexpr int kBytes = 32;
  __device__ __forceinline__ static void store(unsigned char *set, int nslots, int i,
                                               const SU2<double> &q) {
    double2 *p = reinterpret_cast<double2 *>(set);
    p[i] = make_double2(q.a0, q.a1);
    p[nslots + i] = make_double2(q.a2, q.a3);
  }
  __device__ __forceinline__ static SU2<double> load(const unsigned char *set, int nslots,
                                                     int i) {
    const double2 *p = reinterpret_cast<const double2 *>(set);
    const double2 a = p[i], b = p[nslots + i];
    return {a.x, a.y, b.x, b.y};
  }
};

// The fundamental SU(2) loops with one column per thread and KS consecutive
// start slices whose space lines stay in registers. The sweep runs over T:
// each step loads one line into a register window and adds the KS loops of
// that T, with no checks and no moves. Per-thread sums in the compute type
// (FP32 for the mixed form), block and grid sums in FP64. SLAB: starts are
// checked (t0 < tstarts: a time slab, or 4 does not divide Lt).
template <class Store, class CT, int KS, bool SLAB>
__global__ void __launch_bounds__(256)
    wilson_gauge_q_kernel(const __grid_constant__ Geom g, const __grid_constant__ Fields4 U,
                          int NE, int rmin, int rmax, int tmin, int tmax, int cols, int rows,
                          double *partials, const int *flag, int tstarts) {
  wait_previous();
  if (flag && *flag != 0)
    return;
  using Q = SU2<CT>;
  using QS = QuatSet<CT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int nt = tmax - tmin + 1;
  const int nthreads = blockDim.x;
  const int nslots = NE * cols;
  CT *red = reinterpret_cast<CT *>(smem_raw); // [nt][nthreads]
  unsigned char *sa = smem_raw + ((sizeof(CT) * nt * nthreads + 15) & ~(size_t)15);

  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, nwarps = nthreads >> 5;
  const int u = tid % cols;
  const int row = tid / cols;
  const int nu = blockIdx.y;
  const int s0 = column_base(g, blockIdx.x, cols, nu) + u;
  const bool active = (row < rows) && (s0 < g.Vs);
  const int t0 = KS * row;
  const void *f = U.f[nu];
  const int Ln = sel4(g.L, nu), stn = sel4(g.stride, nu);
  const int xn = (s0 / stn) % Ln;
  const size_t VE = (size_t)NE * g.Vs;
  const int ne = (rmax - rmin + 1) * nt;
  double *part = partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * ne;

  Q a[KS];
#pragma unroll 1
  for (int R = 1; R <= rmax; R++) {
    if (active) {
      const int l = s0 + ((xn + R - 1) % Ln - xn) * stn;
#pragma unroll
      for (int m = 0; m < KS; m++) {
        const int t = t0 + m;
        if (SLAB && t >= NE)
          break;
        const Q lo = Store::template load<CT>(f, VE, l + t * g.Vs);
        a[m] = R == 1 ? lo : mul(a[m], lo);
        QS::store(sa, nslots, t * cols + u, a[m]);
      }
#pragma unroll 1
      for (int t = KS * rows + row; t < NE; t += rows) {
        const int i = t * cols + u;
        const Q lx = Store::template load<CT>(f, VE, l + t * g.Vs);
        QS::store(sa, nslots, i, R == 1 ? lx : mul(QS::load(sa, nslots, i), lx));
      }
    }
    __syncthreads();
    if (R >= rmin) {
      // T-major sweep: the thread's sum for T index q is its KS loops of
      // starts t0 + m ending on the lines of relative index p = q + m
      // (slice t0 + tmin + p). A window of W = KS + 1 lines in registers
      // holds relative index p in w[p % W]; step q (unrolled by W, so every
      // slot index is a constant) loads the line p = q + KS that step q + 1
      // needs and adds the KS dot products of step q. Inactive threads load
      // nothing (zero lines) and write zero sums.
      constexpr int W = KS + 1;
      if (!active) {
#pragma unroll
        for (int m = 0; m < KS; m++)
          a[m] = Q{CT(0), CT(0), CT(0), CT(0)};
      }
      Q w[W];
      int tp = min(t0 + tmin, NE - 1); // slice of the next line to load
#pragma unroll
      for (int m = 0; m < KS; m++) {
        w[m] = active ? QS::load(sa, nslots, tp * cols + u) : a[0];
        tp = min(tp + 1, NE - 1);
      }
#pragma unroll 1
      for (int q0 = 0; q0 < nt; q0 += W) {
#pragma unroll
        for (int r = 0; r < W; r++) {
          if (q0 + r < nt) {
            w[(r + KS) % W] = active ? QS::load(sa, nslots, tp * cols + u) : a[0];
            tp = min(tp + 1, NE - 1);
            CT d[KS];
#pragma unroll
            for (int m = 0; m < KS; m++) {
              const Q &b = w[(r + m) % W];
              d[m] = (!SLAB || t0 + m < tstarts) ? dot4(a[m].a0, b.a0, a[m].a1, b.a1, a[m].a2, b.a2, a[m].a3, b.a3) : CT(0);
            }
#pragma unroll
            for (int k = 1; k < KS; k *= 2)
#pragma unroll
              for (int m = 0; m + k < KS; m += 2 * k)
                d[m] += d[m + k];
            red[(size_t)(q0 + r) * nthreads + tid] = d[0];
          }
        }
      }
      __syncthreads();
#pragma unroll 1
      for (int T = warp; T < nt; T += nwarps) {
        double v = 0.0;
        for (int i = lane; i < nthreads; i += 32)
          v += double(red[(size_t)T * nthreads + i]);
        v = warp_sum(v);
        if (lane == 0)
          part[(R - rmin) * nt + T] = v;
      }
    }
    __syncthreads();
  }
}

// The fixed-order tree over blocks (as reduce_partials_kernel in
// gc_wilson.cu) over the partials of whichever method ran.
__global__ void __launch_bounds__(256)
    reduce_select_kernel(const double *partials, int blocks_exact, int blocks_gauge,
                         const int *flag, int nr, int nt, double scale, double *out) {
  wait_previous();
  __shared__ double sh[256];
  const int e = blockIdx.x;
  const int nblocks = *flag ? blocks_exact : blocks_gauge;
  const int nentries = nr * nt;
  double s = 0.0;
  for (int b = threadIdx.x; b < nblocks; b += blockDim.x)
    s += partials[(size_t)b * nentries + e];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const int ir = e / nt, it = e % nt;
    out[it * nr + ir] = sh[0] * scale;
  }
}

// Which kernel takes the fundamental loops (whole W calls in us):
// wilson_corr_kernel unless
//   - the sequences are short, so that a thread's sums over its warp cost as
//     much as its products: the one-column kernels (four starts per thread)
//     take Lt x (T values) below a bound
//       SU(3) mixed, one column / correlation: 32^3 x 6 T <= 3 260 / 346, 32^3
//       x 8 T <= 4 316 / 371, 32^3 x 10 T <= 5 453 / 436, 24^4 T <= 2 407 /
//       369; on small lattices the correlation's blocks fill more of the chip:
//       12^3 x 8 87 / 71, 16^3 x 8 109 / 98, 24^3 x 8 134 / 144
//       SU(2) mixed: 32^3 x 8 T <= 4 101 / 125, 24^4 T <= 5 127 / 135, T <= 6
//       134 / 135, 32^4 T <= 6 370 / 346, 20^4 T <= 10 108 / 108
//       SU(2) FP64: 16^4 T <= 2 65 / 76, T <= 8 78 / 80, 24^4 T <= 6 211 / 187
//   - FP64 with a T range that one window does not cover (its 12 T values take
//     48 registers; a second window reads the lines again): the Gram matrix
//       SU(3), Gram matrix / correlation: 32^4 T <= 8 2248 / 2116, T <= 12
//       2868 / 2613, T <= 13 2914 / 3340, T <= 16 2966 / 3370; SU(2) 24^4 T <=
//       12 276 / 221, 32^4 T <= 12 812 / 629, T <= 16 802 / 792, 48^4 T <= 24
//       5710 / 6557
//     (these with one FP32 chain of the correlation's mixed form; with its short
//     sums, 5 to 17% slower, calls on either side of the line still meet: SU(3)
//     32^3 x 10 T <= 4 / 5 686 / 702, 24^3 x 8 T <= 3 / 4 212 / 230, SU(2) 24^4 T
//     <= 7 / 8 128 / 122)
// (q kernel: at most 32 threads per column, so that a block of 8 columns fits)
constexpr int kStarts = 4;
int start_rows(int Lt) { return (Lt + kStarts - 1) / kStarts; }
bool gauge_short_applies(const Geom &g, int nt, int nc, int ct_bytes) {
  const int work = g.L[3] * nt;
  if (nc == 2)
    return start_rows(g.L[3]) <= 32 && work < (ct_bytes == 4 ? 192 : 144);
  return ct_bytes == 4 && start_rows(g.L[3]) <= 64 && work <= 40 && g.Vs > 8192;
}
bool gauge_corr_applies(int tmax, int ct_bytes) { return ct_bytes == 4 || tmax <= 12; }

int largest_divisor_upto_g(int n, int cap) {
  for (int d = cap < n ? cap : n; d > 1; d--)
    if (n % d == 0)
      return d;
  return 1;
}

} // namespace

// The fundamental loops: wilson_gram_kernel's shape. The adjoint loops: every
// start slice of a column has a thread (rows = Lt up to 64; beyond, the largest
// divisor of Lt up to 64 with Lt/rows slices each), about 128 threads per block.
WilsonPlan wilson_gauge_plan(const Geom &g, int tmin, int tmax, int nc, int ct_bytes,
                             int units_req, bool adjoint, int tstarts) {
  const int Lt = g.L[3], NE = Lt + wilson_gauge_ext(g, tmax, tstarts);
  if (tstarts <= 0 || tstarts > Lt)
    tstarts = Lt;
  WilsonPlan p{};
  const int nt = tmax - tmin + 1;
  const bool few = gauge_short_applies(g, nt, nc, ct_bytes);
  if (!adjoint && !few && gauge_corr_applies(tmax, ct_bytes)) {
    p = wilson_corr_plan(g, tstarts, tmin, tmax, nc, ct_bytes, units_req);
    if (p.fits || units_req > 0)
      return p;
  }
  if (!adjoint && few && nc == 2) {
    // the SU(2) one-column kernel: four starts per thread, by default the
    // largest power of two (at least 8) of columns with at most 192 threads
    // per block (48^4 mixed: 5.15 ms with 16 columns of 12 threads, 5.47 ms
    // with 8)
    p.kernel = 2;
    p.starts = kStarts;
    p.rows = start_rows(Lt);
    int units = units_req;
    if (units <= 0)
      for (units = 8; 2 * units * p.rows <= 192;)
        units *= 2;
    p.cols_per_block = units;
    p.threads = wilson_threads(units, p.rows, 1);
    p.blocks = ((g.Vs + units - 1) / units) * 3;
    p.smem = ((size_t)nt * p.threads * ct_bytes + 15) / 16 * 16 +
             (size_t)(ct_bytes == 4 ? 16 : 32) * NE * units;
    p.fits = p.threads <= 256 && p.smem <= 200 * 1024;
    if (p.fits || units_req > 0)
      return p;
  }
  if (!adjoint && few && nc == 3) {
    // the mixed SU(3) one-column kernel: by default the largest power of two
    // of columns with at most 128 threads per block (of 8, 16 and 32 columns
    // 2-15% faster than twice or half, 10-50% than a quarter)
    p.kernel = 3;
    p.starts = kStarts;
    p.rows = start_rows(Lt);
    int units = units_req;
    if (units <= 0)
      for (units = 1; 2 * units * p.rows <= 128;)
        units *= 2;
    p.cols_per_block = units;
    p.threads = wilson_threads(units, p.rows, 1);
    p.blocks = ((g.Vs + units - 1) / units) * 3;
    p.smem = ((size_t)nt * p.threads * sizeof(float) + 15) / 16 * 16 +
             (size_t)Rows01Set::kBytes * NE * units;
    p.fits = p.threads <= 256 && p.smem <= 200 * 1024;
    if (p.fits || units_req > 0)
      return p;
  }
  if (!adjoint)
    return wilson_gram_plan(g, tstarts, tmax, nc, units_req, false);
  p = WilsonPlan{};
  const int ncomp = (nc == 3) ? 18 : 4;
  const int lanes = wilson_lanes(nc, ct_bytes);
  // consecutive start slices per thread (a divisor of Lt): 2 for SU(3) (its
  // registers hold two lane-packed matrices) and on SU(2) lattices that leave the
  // chip idle otherwise, 4 on larger SU(2) lattices (quaternions are small). SU(2)
  // calls in us with 2 / 4 starts: FP64 12^4 R,T <= 6 56 / 69, 16^3 x 4 54 / 67,
  // 16^4 R,T <= 8 75 / 90, 20^4 117 / 138, 16^3 x 32 102 / 102, 24^4 R,T <= 6 179 /
  // 165; mixed 16^4 70 / 79, 10^3 x 48 60 / 65, 16^3 x 32 101 / 90, 20^4 105 / 96
  p.starts = 1;
  const bool four = nc == 2 && g.V > (ct_bytes == 8 ? 160000 : 65536);
  for (int ks : {four ? 4 : 2, 2})
    if (p.starts == 1 && Lt % ks == 0 && Lt / ks <= 64)
      p.starts = ks;
  p.rows = p.starts > 1 ? Lt / p.starts : largest_divisor_upto_g(Lt, 64);
  // (about 128 threads: at SU(3) 32^4 the paired kernel took 5.5, 4.6, 3.8,
  // 3.1, 3.1 ms mixed with 1, 2, 4, 8, 16 column units of 16 threads; wider
  // blocks coalesce the extension's link loads)
  const int units = units_req > 0 ? units_req : std::max(1, 128 / p.rows);
  p.cols_per_block = units * lanes;
  p.threads = wilson_threads(p.cols_per_block, p.rows, lanes);
  p.blocks = ((g.Vs + p.cols_per_block - 1) / p.cols_per_block) * 3;
  p.smem = ((size_t)nt * p.threads * sizeof(double) + 15) / 16 * 16 +
           (size_t)ncomp * NE * wilson_col_stride(p.cols_per_block, lanes) * ct_bytes;
  p.fits = p.threads <= 256 && p.smem <= 200 * 1024;
  return p;
}

int wilson_gauge_ext(const Geom &g, int tmax, int tstarts) {
  return tstarts > 0 && tstarts < g.L[3] ? 0 : tmax;
}

bool wilson_gauge_applies(const Geom &g, int tmin, int tmax, int nc, int ct_bytes, bool adjoint,
                          int tstarts) {
  const int Lt = g.L[3];
  const bool slab = tstarts > 0 && tstarts < Lt;
  return Lt >= 2 && tmax <= (slab ? Lt - tstarts : Lt / 2) &&
         wilson_gauge_plan(g, tmin, tmax, nc, ct_bytes, 0, adjoint, tstarts).fits;
}

double wilson_gauge_tolerance(int ct_bytes) { return ct_bytes == 8 ? 1e-14 : 1e-6; }

namespace {
size_t align256(size_t n) { return (n + 255) / 256 * 256; }
} // namespace

size_t wilson_gauge_lines_bytes(const Geom &g, int nc) {
  const size_t line = nc == 3 ? 144 : 32;
  return align256(line * g.V) + align256(line * g.Vs);
}

size_t wilson_gauge_bytes(const Geom &g, int nc, int link_bytes, int ext) {
  return wilson_gauge_lines_bytes(g, nc) +
         3 * align256((size_t)link_bytes * (g.L[3] + ext) * g.Vs);
}

GaugeLinks wilson_gauge_links(void *base, const Geom &g, int nc, int link_bytes, int ext,
                              void *links) {
  GaugeLinks l{};
  const size_t line = nc == 3 ? 144 : 32;
  char *p = static_cast<char *>(base);
  l.G = p;
  p += align256(line * g.V);
  l.W = p;
  p = links ? static_cast<char *>(links) : p + align256(line * g.Vs);
  l.NE = g.L[3] + ext;
  for (int d = 0; d < 3; d++) {
    l.U.f[d] = p;
    p += align256((size_t)link_bytes * l.NE * g.Vs);
  }
  l.U.f[3] = nullptr;
  return l;
}

namespace {

template <class Store, class CT, bool MAPPED>
int launch_gauge_lines(const Geom &g, const AxisMap &map, const void *Ut, const GaugeLinks &l,
                       int *flag, cudaStream_t s) {
  const double tol = wilson_gauge_tolerance((int)sizeof(CT));
  // (a time slab counts the loops of a few start slices, which links of those
  // slices enter more often than the mean says)
  const bool slab = l.NE == g.L[3];
  const double most = sizeof(CT) == 8 && !slab ? 100 * tol : tol;
  const int blocks = (g.Vs + kLinesCols - 1) / kLinesCols;
  if (g.Vs < 8192)
    launch_chained(gauge_lines_kernel<Store, 4, MAPPED>, blocks, 4 * kLinesCols, 0, s, g, map, Ut,
                   l.G, l.W, tol, most, flag);
  else
    launch_chained(gauge_lines_kernel<Store, 1, MAPPED>, blocks, kLinesCols, 0, s, g, map, Ut, l.G,
                   l.W, tol, most, flag);
  return launch_check("gauge_lines_kernel");
}

template <class Store, class Out, class CT, bool MAPPED>
int launch_gauge_links(const Geom &g, const AxisMap &map, const Fields4 &U, const GaugeLinks &l,
                       const Fields4 &out, int ndir, int *flag, cudaStream_t s) {
  launch_chained(gauge_transform_kernel<Store, Out, MAPPED>,
                 dim3((l.NE * g.Vs + 127) / 128, ndir), 128, 0, s, g, map, U, l.G, l.W, out, l.NE, wilson_gauge_tolerance((int)sizeof(CT)),
                 flag);
  return launch_check("gauge_transform_kernel");
}

} // namespace

template <class Store, class CT>
int launch_wilson_gauge_prep(const Geom &g, const Fields4 &U, const GaugeLinks &l, int *flag,
                             cudaStream_t s) {
  cudaError_t e = cudaMemsetAsync(flag, 0, sizeof(int), s);
  if (e != cudaSuccess)
    return launch_check("gauge flag reset");
  const int rc = launch_gauge_lines<Store, CT, false>(g, AxisMap{}, U.f[3], l, flag, s);
  return rc ? rc : launch_gauge_links<Store, Store, CT, false>(g, AxisMap{}, U, l, l.U, 3, flag, s);
}

template <class Store, class CT>
int launch_wilson_gauge_second(const Geom &g, const Fields4 &U2, const GaugeLinks &l,
                               const Fields4 &out, int *flag, cudaStream_t s) {
  return launch_gauge_links<Store, Store, CT, false>(g, AxisMap{}, U2, l, out, 3, flag, s);
}

template <class Store, class CT>
int launch_axis_gauge_lines(const Geom &g, const AxisMap &map, const void *Ut,
                            const GaugeLinks &l, int *flag, cudaStream_t s) {
  return launch_gauge_lines<Store, CT, true>(g, map, Ut, l, flag, s);
}

template <class Store, class CT>
int launch_axis_gauge_links(const Geom &g, const AxisMap &map, const Fields4 &F,
                            const GaugeLinks &l, int *flag, cudaStream_t s) {
  return launch_gauge_links<Store, typename InterStore<Store>::type, CT, true>(g, map, F, l, l.U, 2,
                                                                              flag, s);
}

template <class Store, class CT>
int launch_wilson_gauge_kernel(const Geom &g, const GaugeLinks &l, int rmin, int rmax, int tmin,
                               int tmax, bool adjoint, const int *flag, double *partials,
                               int *blocks, cudaStream_t s, int units = 0, int tstarts = 0,
                               int ndir = 3) {
  const int nr = rmax - rmin + 1, nt = tmax - tmin + 1;
  // every start slice (on tmax further slices), or the start slices
  // [0, tstarts) of a time slab
  const int Lt = g.L[3];
  const bool slab = tstarts > 0 && tstarts < Lt;
  if (!slab)
    tstarts = Lt;
  if (tmax > (slab ? Lt - tstarts : Lt / 2))
    return plan_error(slab ? "wilson_gauge_kernel: time_max above Lt - t_starts"
                           : "wilson_gauge_kernel: time_max above Lt/2");
  if (nr * nt > kWilsonMaxEntries)
    return plan_error("wilson_gauge_kernel: too many (R,T) entries");
  const WilsonPlan p =
      wilson_gauge_plan(g, tmin, tmax, Store::NC, (int)sizeof(CT), units, adjoint, tstarts);
  if (!adjoint && p.kernel == 1)
    return launch_wilson_gram<Store, CT>(g, l, nullptr, rmin, rmax, tmin, tmax, flag, partials,
                                         blocks, s, units, tstarts, ndir);
  if (!adjoint && p.kernel == 4)
    return launch_wilson_corr<Store, CT>(g, l, rmin, rmax, tmin, tmax, flag, partials, blocks, s,
                                         units, tstarts, ndir);
  if (!p.fits || l.NE < tstarts + tmax)
    return plan_error("wilson_gauge_kernel: block shape does not fit");
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(s, &cap);
  const bool capturing = cap != cudaStreamCaptureStatusNone;
  auto go = [&](auto k_all, auto k_slab) {
    // (the start-slice checks of a t-slab compiled in only where they are used)
    auto kernel = slab ? k_slab : k_all;
    int r = allow_large_smem(kernel, p.smem, capturing);
    if (r)
      return r;
    launch_chained(kernel, dim3(p.blocks / 3, ndir), p.threads, p.smem, s, g, l.U, l.NE, rmin, rmax,
                   tmin, tmax, p.cols_per_block, p.rows, partials, flag, tstarts);
    return GC_OK;
  };
  if constexpr (Store::NC == 2) {
    if (p.kernel == 2) {
      auto k_all = wilson_gauge_q_kernel<Store, CT, kStarts, false>;
      auto k_some = wilson_gauge_q_kernel<Store, CT, kStarts, true>;
      const int rc = go(Lt % kStarts ? k_some : k_all, k_some);
      *blocks = p.blocks / 3 * ndir;
      return rc ? rc : launch_check("wilson_gauge_q_kernel");
    }
  }
  if constexpr (std::is_same<Store, StoreF32SU3>::value) {
    if (p.kernel == 3) {
      auto k_all = wilson_gauge_reg_kernel<kStarts, false>;
      auto k_some = wilson_gauge_reg_kernel<kStarts, true>;
      const int rc = go(Lt % kStarts ? k_some : k_all, k_some);
      *blocks = p.blocks / 3 * ndir;
      return rc ? rc : launch_check("wilson_gauge_reg_kernel");
    }
  }
  constexpr int K4 = Store::NC == 2 ? 4 : 2;
  const int rc = p.starts == 4   ? go(wilson_gauge_kernel<Store, CT, K4, false>,
                                      wilson_gauge_kernel<Store, CT, K4, true>)
                 : p.starts == 2 ? go(wilson_gauge_kernel<Store, CT, 2, false>,
                                      wilson_gauge_kernel<Store, CT, 2, true>)
                                 : go(wilson_gauge_kernel<Store, CT, 1, false>,
                                      wilson_gauge_kernel<Store, CT, 1, true>);
  if (rc)
    return rc;
  *blocks = p.blocks / 3 * ndir;
  return launch_check("wilson_gauge_kernel");
}

int launch_reduce_select(const double *partials, int blocks_exact, int blocks_gauge,
                         const int *flag, int nr, int nt, double scale, double *out_dev,
                         cudaStream_t s) {
  launch_chained(reduce_select_kernel, nr * nt, 256, 0, s, partials, blocks_exact, blocks_gauge,
                 flag, nr, nt, scale, out_dev);
  return launch_check("reduce_select_kernel");
}

template <class Store, class CT>
int launch_wilson_auto(const Geom &g, const Fields4 &U, const GaugeLinks &l, int rmin, int rmax,
                       int tmin, int tmax, bool adjoint, const int *flag, double *partials,
                       double *out_dev, cudaStream_t s, int units, int tstarts,
                       const Fields4 *second, const Fields4 *second_links) {
  if (tstarts <= 0 || tstarts > g.L[3])
    tstarts = g.L[3];
  int b_exact = 0, b_gauge = 0;
  int rc = launch_wilson_exact_gated<Store, CT>(g, U, second, rmin, rmax, tmin, tmax, adjoint,
                                                flag, partials, &b_exact, s, tstarts);
  if (rc)
    return rc;
  rc = second ? launch_wilson_gram<Store, CT>(g, l, second_links, rmin, rmax, tmin, tmax, flag,
                                              partials, &b_gauge, s, units, tstarts)
              : launch_wilson_gauge_kernel<Store, CT>(g, l, rmin, rmax, tmin, tmax, adjoint, flag,
                                                      partials, &b_gauge, s, units, tstarts);
  if (rc)
    return rc;
  const int nr = rmax - rmin + 1, nt = tmax - tmin + 1;
  // average over the loops counted: every site, or the tstarts slices (GEVP
  // counts every loop twice: the / (6 V) of wilson_loops.h:910)
  return launch_reduce_select(partials, b_exact, b_gauge, flag, nr, nt,
                              wilson_scale((long long)g.Vs * tstarts, Store::NC, adjoint) /
                                  (second ? 2.0 : 1.0),
                              out_dev, s);
}

size_t wilson_auto_partials_count(const Geom &g, int nr, int tmin, int tmax, int nc, int units,
                                  int tstarts) {
  int blocks = 0;
  for (int ct : {4, 8})
    for (bool adj : {false, true})
      blocks = std::max(blocks,
                        wilson_gauge_plan(g, tmin, tmax, nc, ct, units, adj, tstarts).blocks);
  const int nt = tmax - tmin + 1;
  return std::max<size_t>(wilson_partials_count(g, nr, nt, nc), (size_t)blocks * nr * nt);
}

// Kernels of the axis loops. Mixed SU(3) lines are full products there (planar
// APE sums need not project onto the group), which the one-column kernel of few
// slices does not have.
static WilsonPlan axis_loops_plan(const Geom &g, int tmin, int tmax, int nc, int ct_bytes) {
  WilsonPlan p = wilson_gauge_plan(g, tmin, tmax, nc, ct_bytes);
  if (p.kernel != 3)
    return p;
  p = wilson_corr_plan(g, g.L[3], tmin, tmax, nc, ct_bytes, 0);
  return p.fits ? p : wilson_gram_plan(g, g.L[3], tmax, nc, 0, false);
}

size_t axis_loops_partials(const Geom &g, int nr, int tmin, int tmax, int nc, int ct_bytes) {
  return (size_t)axis_loops_plan(g, tmin, tmax, nc, ct_bytes).blocks / 3 * 2 * nr *
         (tmax - tmin + 1);
}

bool axis_loops_apply(const Geom &g, int tmax, int nc, int ct_bytes) {
  return g.L[3] >= 2 && tmax <= g.L[3] / 2 && axis_loops_plan(g, 1, tmax, nc, ct_bytes).fits;
}

template <class Store, class CT>
int launch_axis_loops(const Geom &g, const GaugeLinks &l, int rmin, int rmax, int tmin, int tmax,
                      const int *flag, double *partials, double scale, double *out_dev,
                      cudaStream_t s) {
  int blocks = 0, rc;
  if constexpr (std::is_same<Store, StoreF32SU3>::value) {
    const WilsonPlan p = axis_loops_plan(g, tmin, tmax, 3, 4);
    rc = p.kernel == 4
             ? launch_wilson_corr<StoreF32SU3Full, float>(g, l, rmin, rmax, tmin, tmax, flag,
                                                          partials, &blocks, s, 0, g.L[3], 2)
             : launch_wilson_gram<StoreF32SU3Full, float>(g, l, nullptr, rmin, rmax, tmin, tmax,
                                                          flag, partials, &blocks, s, 0, g.L[3],
                                                          2);
  } else {
    rc = launch_wilson_gauge_kernel<Store, CT>(g, l, rmin, rmax, tmin, tmax, false, flag, partials,
                                               &blocks, s, 0, 0, 2);
  }
  return rc ? rc
            : launch_reduce_wilson(partials, blocks, rmax - rmin + 1, tmax - tmin + 1, scale,
                                   out_dev, s);
}

// Times one launch of the gauge W kernel of a lattice with `units` column
// units per block (the autotuner's candidate), from prepared transformed
// links; partials must hold wilson_auto_partials_count(.., units) doubles.
template <class Store, class CT>
int time_wilson_gauge(const Geom &g, const GaugeLinks &l, int rmin, int rmax, int tmin, int tmax,
                      int units, double *partials, cudaStream_t s, float *ms) {
  const WilsonPlan p = wilson_gauge_plan(g, tmin, tmax, Store::NC, (int)sizeof(CT), units);
  if (!p.fits)
    return GC_ERR_ARG;
  int blocks = 0;
  int rc = launch_wilson_gauge_kernel<Store, CT>(g, l, rmin, rmax, tmin, tmax, false, nullptr,
                                                 partials, &blocks, s, units);
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 3 && rc == GC_OK; rep++) {
    cudaEventRecord(e0, s);
    rc = launch_wilson_gauge_kernel<Store, CT>(g, l, rmin, rmax, tmin, tmax, false, nullptr,
                                               partials, &blocks, s, units);
    cudaEventRecord(e1, s);
    cudaEventSynchronize(e1);
    float t = 0;
    cudaEventElapsedTime(&t, e0, e1);
    best = std::min(best, t);
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  *ms = best;
  return rc;
}

#define GC_INSTANTIATE_WG(STORE, CT)                                                         \
  template int launch_wilson_gauge_prep<STORE, CT>(const Geom &, const Fields4 &,            \
                                                   const GaugeLinks &, int *, cudaStream_t); \
  template int launch_wilson_auto<STORE, CT>(const Geom &, const Fields4 &,                  \
                                             const GaugeLinks &, int, int, int, int, bool,   \
                                             const int *, double *, double *, cudaStream_t,  \
                                             int, int, const Fields4 *, const Fields4 *);    \
  template int launch_wilson_gauge_second<STORE, CT>(const Geom &, const Fields4 &,          \
                                                     const GaugeLinks &, const Fields4 &,    \
                                                     int *, cudaStream_t);                   \
  template int launch_axis_gauge_lines<STORE, CT>(const Geom &, const AxisMap &, const void *, \
                                                  const GaugeLinks &, int *, cudaStream_t);  \
  template int launch_axis_gauge_links<STORE, CT>(const Geom &, const AxisMap &,             \
                                                  const Fields4 &, const GaugeLinks &,       \
                                                  int *, cudaStream_t);                      \
  template int launch_axis_loops<STORE, CT>(const Geom &, const GaugeLinks &, int, int, int,  \
                                            int, const int *, double *, double, double *,     \
                                            cudaStream_t);                                   \
  template int time_wilson_gauge<STORE, CT>(const Geom &, const GaugeLinks &, int, int, int, \
                                            int, int, double *, cudaStream_t, float *);

GC_INSTANTIATE_WG(StoreF64SU3, double)
GC_INSTANTIATE_WG(StoreF64SU2, double)
GC_INSTANTIATE_WG(StoreF32SU3, float)
GC_INSTANTIATE_WG(StoreF32SU2, float)

} // namespace gc
