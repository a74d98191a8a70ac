// Fundamental on-axis loops of the temporal gauge by FP64 matrix instructions
// (sm_100a). gc_wilson_gauge.cu has the gauge and the transformed links.
//
// With the transformed space lines S'(s,t,R) written as rows of 18 (SU(3)) or
// 4 (SU(2) quaternions) reals, the loops of all start and end slices of one R
// are the Gram matrix
//     C_R[t0][t1] = sum over columns s and directions of
//                   sum_k S'(s,t0,R)_k S'(s,t1,R)_k ,
// and W(R,T) is the sum of its diagonal t1 - t0 = T: a matrix product with
// 18 (or 4) x columns as the inner dimension. mma.sync.m8n8k4.f64 computes it
// in FP64 (in both forms: the FP32 lines are exact in FP64, so the mixed
// form's sums are FP64 from the first product on). The instruction runs at
// 37 TFLOP/s here where separate FP64 fused multiply-adds reach 28 (their
// operands do not fit the register ports), and one 8-byte load of a fragment
// per lane serves up to eight of them: of the 8 x 8 tiles of C only those
// within T <= T_max of the diagonal are computed, and the fragment of a tile
// of slices is the same register as left operand and as right operand.
//
// A block owns `cols` columns (s, nu) on all NE slices. Per R: each thread
// extends its slots' lines by one transformed link (in the compute type; the
// line lives in shared memory as FP64), a barrier, the warps multiply (a warp
// per column pair and group of up to four tiles of start slices) and leave
// the tiles' sums over their start tiles in shared memory, a barrier, and the
// diagonals are summed over rows and warps in fixed order into the block's
// partial. The fixed-order tree over blocks of gc_wilson.cu finishes.
//
// Bound: the FP64 pipe, which the matrix instructions share with the FP64
// form's products (64% busy at SU(3) 24^4 FP64, the matrix instructions alone
// 46%): the blocks' extension and multiplication phases
// overlap only between the four blocks of an SM, and of the computed tiles
// T_max / (8 nd) lies within the band (0.5 at T <= 12, 0.67 at T <= 16). FP64,
// R,T <= L/2, whole W call: SU(3) 32^4 5.93 -> 2.97 ms, SU(2) 48^4 10.1 -> 5.74
// ms. Where one window of T fits a thread's registers, gc_wilson_corr.cu is
// faster (the rule is in gc_wilson_gauge.cu).
//
// GEVP (wilson_gevp_indexed, wilson_loops.h:1202-1233): a second set of
// lines, C = S2 S1^T + S1 S2^T.
#include "gc_internal.cuh"
#include "gc_kernels.h"
#include "gc_rows01.cuh"
#include "gc_wcol.cuh"

#include <algorithm>
#include <type_traits>

namespace gc {

namespace {

constexpr int kGramThreads = 128;
// Tiles of a warp task: up to kND tiles of end slices per start tile and pass,
// and as many tiles of start slices as keep the accumulators within kTiles
// (48 registers).
constexpr int kND = 4, kTiles = 12;
__host__ __device__ constexpr int start_tiles(int nd) { return nd >= 4 ? 3 : 4; }
static_assert(3 * kND <= kTiles && 4 * 3 <= kTiles, "accumulators");

__device__ __forceinline__ void dmma(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1},{%2},{%3},{%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}

// Layout of a set of lines in shared memory (in double2 units) and the inner
// dimension. A unit is what one run of matrix instructions consumes: a pair of
// SU(3) columns (36 reals a slice: nine steps of four) or one SU(2) column
// (one step). Fragment loads read, per half warp, four slices x four reals
// (strides of 36 and 4 doubles: all banks once); the extension's 16-byte
// accesses go over consecutive columns, whose stride is 2 (pairs, 9 within a
// pair) or 1 modulo 8 vectors: conflict-free as well.
template <int NC> struct GramSet;
template <> struct GramSet<3> {
  static constexpr int kColsPerUnit = 2, kSteps = 9, kSlice = 18;
  __host__ __device__ static int stride(int slices) { return slices * 18 + (10 - slices * 18 % 8) % 8; }
  __device__ static int record(int c, int t, int st) { return (c >> 1) * st + t * 18 + (c & 1) * 9; }
};
template <> struct GramSet<2> {
  static constexpr int kColsPerUnit = 1, kSteps = 1, kSlice = 2;
  __host__ __device__ static int stride(int slices) { return slices * 2 + 1; }
  __device__ static int record(int c, int t, int st) { return c * st + t * 2; }
};

__device__ __forceinline__ void put(double2 *p, const SU3<double> &m) {
#pragma unroll
  for (int k = 0; k < 9; k++)
    p[k] = make_double2(m.e[k / 3][k % 3].re, m.e[k / 3][k % 3].im);
}
__device__ __forceinline__ void put(double2 *p, const SU3<float> &m) {
#pragma unroll
  for (int k = 0; k < 9; k++)
    p[k] = make_double2(double(m.e[k / 3][k % 3].re), double(m.e[k / 3][k % 3].im));
}
template <class T> __device__ __forceinline__ void put(double2 *p, const SU2<T> &q) {
  p[0] = make_double2(double(q.a0), double(q.a1));
  p[1] = make_double2(double(q.a2), double(q.a3));
}
// line <- line u
template <class Store, class T> __device__ __forceinline__ void extend(double2 *p, const SU3<T> &u) {
  SU3<T> a;
  if constexpr (Store::kBytes == 48) {
    // products of SU(3) links: rows 0 and 1, row 2 rebuilt
#pragma unroll
    for (int k = 0; k < 6; k++)
      a.e[k / 3][k % 3] = {T(p[k].x), T(p[k].y)};
    a = mul01(a, u);
    rebuild_row2(a);
    put(p, a);
  } else {
#pragma unroll
    for (int k = 0; k < 9; k++)
      a.e[k / 3][k % 3] = {T(p[k].x), T(p[k].y)};
    put(p, mul(a, u));
  }
}
template <class Store, class T> __device__ __forceinline__ void extend(double2 *p, const SU2<T> &u) {
  const double2 v = p[0], w = p[1];
  put(p, mul(SU2<T>{T(v.x), T(v.y), T(w.x), T(w.y)}, u));
}

// Tiles of 8 slices: n0 of start slices, nd of end slices per start tile
// (t1 - t0 up to tmax), and the slots of a column they touch.
struct GramTiles {
  int n0, nd, slices, groups;
};
__host__ __device__ inline GramTiles gram_tiles(int tstarts, int tmax) {
  GramTiles t;
  t.n0 = (tstarts + 7) / 8;
  t.nd = (tmax + 7) / 8 + 1;
  t.slices = 8 * (t.n0 + t.nd - 1);
  t.groups = (t.n0 + start_tiles(t.nd) - 1) / start_tiles(t.nd);
  return t;
}

// One warp task: the tiles (i0 + m, i0 + m + d0 + d), m < MT, d < ND, summed
// over the units sub, sub + nsub, ... and over the start tiles, into E.
// f1 / f2: the lane's first fragment element of unit 0 (slice 8 i0 + lane / 4,
// real lane % 4) in the sets of the end / start lines.
template <class GS, int MT, int ND, bool GEVP>
__device__ __forceinline__ void gram_task(const double *f1, const double *f2, int unit_stride,
                                          int sub, int nsub, int units, int d0, int first_start,
                                          int tstarts, double *e, bool add) {
  constexpr int kTile = 16 * GS::kSlice; // doubles from one tile to the next
  double acc[MT][ND][2];
#pragma unroll
  for (int m = 0; m < MT; m++)
#pragma unroll
    for (int d = 0; d < ND; d++)
      acc[m][d][0] = acc[m][d][1] = 0.0;
  const int db = d0 * kTile;
  if (!GEVP && d0 == 0) {
    // the start tiles' fragments are the first of the end tiles'; the next
    // step's are loaded while the current ones are multiplied
    constexpr int NB = MT + ND - 1;
    double b[2][NB];
    auto load = [&](double (&x)[NB], const double *p) {
#pragma unroll
      for (int j = 0; j < NB; j++)
        x[j] = p[j * kTile];
    };
    auto mma = [&](const double (&x)[NB]) {
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int d = 0; d < ND; d++)
          dmma(acc[m][d], x[m], x[m + d]);
    };
    if (GS::kSteps == 1) {
#pragma unroll 1
      for (int unit = sub; unit < units; unit += nsub) {
        load(b[0], f1 + (size_t)unit * unit_stride);
        mma(b[0]);
      }
    } else {
#pragma unroll 1
      for (int unit = sub; unit < units; unit += nsub) {
        const double *p = f1 + (size_t)unit * unit_stride;
        load(b[0], p);
#pragma unroll
        for (int k = 0; k < GS::kSteps; k++) {
          if (k + 1 < GS::kSteps)
            load(b[(k + 1) & 1], p + 4 * (k + 1));
          mma(b[k & 1]);
        }
      }
    }
  } else {
    auto run = [&](const double *p1, const double *p2) {
      double a[MT], b[MT + ND - 1];
#pragma unroll
      for (int j = 0; j < MT + ND - 1; j++)
        b[j] = p1[db + j * kTile];
#pragma unroll
      for (int m = 0; m < MT; m++)
        a[m] = p2[m * kTile];
#pragma unroll
      for (int m = 0; m < MT; m++)
#pragma unroll
        for (int d = 0; d < ND; d++)
          dmma(acc[m][d], a[m], b[m + d]);
    };
#pragma unroll 1
    for (int unit = sub; unit < units; unit += nsub) {
      const double *p1 = f1 + (size_t)unit * unit_stride, *p2 = f2 + (size_t)unit * unit_stride;
#pragma unroll 1
      for (int k = 0; k < GS::kSteps; k++) {
        run(p1 + 4 * k, p2 + 4 * k);
        if (GEVP)
          run(p2 + 4 * k, p1 + 4 * k);
      }
    }
  }
  // sum over the start tiles (rows past the last start do not count); the lane
  // holds row lane / 4, columns 2 (lane % 4), + 1 of each tile
#pragma unroll
  for (int d = 0; d < ND; d++) {
    double e0 = 0.0, e1 = 0.0;
#pragma unroll
    for (int m = 0; m < MT; m++)
      if (first_start + 8 * m < tstarts) {
        e0 += acc[m][d][0];
        e1 += acc[m][d][1];
      }
    if (add) {
      e0 += e[8 * d];
      e1 += e[8 * d + 1];
    }
    e[8 * d] = e0;
    e[8 * d + 1] = e1;
  }
}

template <class Store, class CT, bool GEVP>
__global__ void __launch_bounds__(kGramThreads, 4)
    wilson_gram_kernel(const __grid_constant__ Geom g, const __grid_constant__ Fields4 U,
                       const __grid_constant__ Fields4 U2, int NE, int rmin, int rmax, int tmin,
                       int tmax, int cols, double *partials, const int *flag, int tstarts) {
  wait_previous();
  // the exact product runs instead when a link failed the check
  if (flag && *flag != 0)
    return;
  using GS = GramSet<Store::NC>;
  extern __shared__ __align__(16) double2 gram_smem[];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int nwarps = kGramThreads / 32;
  const int nt = tmax - tmin + 1;
  const GramTiles tl = gram_tiles(tstarts, tmax);
  const int st = GS::stride(tl.slices), units = cols / GS::kColsPerUnit;
  double2 *lines = gram_smem;               // [units][st]
  double2 *lines2 = lines + (GEVP ? units * st : 0);
  const int W = 8 * tl.nd;
  double *E = reinterpret_cast<double *>(lines2 + units * st) + warp * 8 * W; // [warp][8][W]

  const int nu = blockIdx.y;
  const int c = tid % cols, trow = tid / cols, tstep = kGramThreads / cols;
  const int s = column_base(g, blockIdx.x, cols, nu) + c;
  const bool active = s < g.Vs;
  const int Ln = sel4(g.L, nu), stn = sel4(g.stride, nu);
  const int xn = (s / stn) % Ln;
  const size_t VE = (size_t)NE * g.Vs;
  // slices the loops touch (a slab's lattice may have more than its tiles hold)
  const int nslots = min(NE, tstarts + tmax);
  double *part = partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (rmax - rmin + 1) * nt;
  // the warp's tasks: a group of start tiles and every nsub-th unit, or, with
  // more groups than warps, every nwarps-th group and all units
  const int nsub = max(1, nwarps / tl.groups);
  const int group0 = tl.groups < nwarps ? warp % tl.groups : warp;
  const int sub = tl.groups < nwarps ? warp / tl.groups : 0;
  const int per = (tl.n0 + tl.groups - 1) / tl.groups; // start tiles of a group
  const int r = lane >> 2;

  // a line's link of this R, and the lines of the thread's slots
  // trow, trow + tstep, ...: the first kPre links are loaded before the matrix
  // instructions of the R before, the others kBatch at a time
  using Raw = RawLink<Store, CT>;
  constexpr int kPre = Raw::kPre, kBatch = Raw::kBatch;
  Raw pre[kPre > 0 ? kPre : 1];
  auto site = [&](int R) { return s + ((xn + R - 1) % Ln - xn) * stn; };
  auto apply = [&](const Raw &x, int t, double2 *set, int R) {
    double2 *p = set + GS::record(c, t, st);
    if (R == 1)
      put(p, x.link());
    else
      extend<Store>(p, x.link());
  };
  auto fetch = [&](int R) {
    if (!active)
      return;
    const int l = site(R);
#pragma unroll
    for (int i = 0; i < kPre; i++)
      if (trow + i * tstep < nslots)
        pre[i].load(U.f[nu], VE, l + (trow + i * tstep) * g.Vs);
  };
  auto extend_from = [&](const void *f, int first, double2 *set, int R) {
    const int l = site(R);
#pragma unroll 1
    for (int t = trow + first * tstep; t < nslots; t += kBatch * tstep) {
      Raw x[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; j++)
        if (t + j * tstep < nslots)
          x[j].load(f, VE, l + (t + j * tstep) * g.Vs);
#pragma unroll
      for (int j = 0; j < kBatch; j++)
        if (t + j * tstep < nslots)
          apply(x[j], t + j * tstep, set, R);
    }
  };
  fetch(1);

  // columns past the lattice count as zero lines
  for (int i = tid; i < (GEVP ? 2 : 1) * units * st; i += kGramThreads)
    lines[i] = make_double2(0.0, 0.0);
  __syncthreads();

#pragma unroll 1
  for (int R = 1; R <= rmax; R++) {
    if (active) {
#pragma unroll
      for (int i = 0; i < kPre; i++)
        if (trow + i * tstep < nslots)
          apply(pre[i], trow + i * tstep, lines, R);
      if (GEVP)
        extend_from(U2.f[nu], 0, lines2, R);
      extend_from(U.f[nu], kPre, lines, R);
    }
    __syncthreads();
    // (issued here: the matrix instructions hide their latency)
    if (R < rmax)
      fetch(R + 1);
    if (R < rmin)
      continue; // (the extension's slots are the thread's own)
    // the warp's rows of E are its own until the barrier below
#pragma unroll 1
    for (int group = group0; group < tl.groups && sub < nsub; group += nwarps) {
      const int i0 = group * per, mt = min(per, tl.n0 - i0);
      const int lane0 = (8 * i0 + r) * 2 * GS::kSlice + (lane & 3);
      const double *f1 = reinterpret_cast<const double *>(lines) + lane0;
      const double *f2 = reinterpret_cast<const double *>(lines2) + lane0;
#pragma unroll 1
      for (int d0 = 0; d0 < tl.nd; d0 += kND) {
        const int dn = min(kND, tl.nd - d0);
        double *e = E + r * W + 8 * d0 + 2 * (lane & 3);
        // (compile-time tile counts: with run-time checks on every tile the
        // warp issued twelve instructions per matrix instruction)
        auto go = [&](auto MT, auto ND) {
          gram_task<GS, decltype(MT)::value, decltype(ND)::value, GEVP>(
              f1, f2, 2 * st, sub, nsub, units, d0, 8 * i0 + r, tstarts, e, group != group0);
        };
        using std::integral_constant;
        auto rows = [&](auto MT) {
          switch (dn) {
          case 1: go(MT, integral_constant<int, 1>()); break;
          case 2: go(MT, integral_constant<int, 2>()); break;
          case 3: go(MT, integral_constant<int, 3>()); break;
          default:
            if constexpr (decltype(MT)::value <= start_tiles(kND))
              go(MT, integral_constant<int, kND>());
          }
        };
        switch (mt) {
        case 1: rows(integral_constant<int, 1>()); break;
        case 2: rows(integral_constant<int, 2>()); break;
        case 3: rows(integral_constant<int, 3>()); break;
        default: rows(integral_constant<int, 4>()); break;
        }
      }
    }
    __syncthreads();
    // W(R,T): the diagonal T of the rows' tiles, over the warps
    const double *E0 = reinterpret_cast<const double *>(lines2 + units * st);
    const int used = min(nwarps, nsub * tl.groups); // warps that had a task
#pragma unroll 1
    for (int i = tid; i < (8 * nt + 31) / 32 * 32; i += kGramThreads) {
      const int T = tmin + i / 8, row = i & 7;
      double v = 0.0;
      if (T <= tmax)
        for (int w = 0; w < used; w++)
          v += E0[w * 8 * W + row * W + row + T];
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
        v += __shfl_xor_sync(0xffffffffu, v, o);
      if (row == 0 && T <= tmax)
        part[(R - rmin) * nt + T - tmin] = v;
    }
  }
}

size_t gram_smem_bytes(int nc, int cols, int tstarts, int tmax, bool gevp) {
  const GramTiles t = gram_tiles(tstarts, tmax);
  const size_t set = nc == 3 ? (size_t)(cols / 2) * GramSet<3>::stride(t.slices)
                             : (size_t)cols * GramSet<2>::stride(t.slices);
  return (gevp ? 2 : 1) * set * 16 + (size_t)kGramThreads / 32 * 8 * 8 * t.nd * 8;
}

} // namespace

// Columns per block: a power of two up to 32 (SU(3): at least a pair).
WilsonPlan wilson_gram_plan(const Geom &g, int tstarts, int tmax, int nc, int cols_req,
                            bool gevp) {
  WilsonPlan p{};
  const size_t want = 72 * 1024; // three blocks on an SM
  int cols = cols_req;
  if (cols <= 0) {
    cols = nc == 3 ? 8 : 16;
    while (cols > (nc == 3 ? 2 : 1) && gram_smem_bytes(nc, cols, tstarts, tmax, gevp) > want)
      cols /= 2;
  }
  p.cols_per_block = cols;
  p.kernel = 1;
  p.rows = 8; // (the autotuner's bound on columns: 256 / rows)
  p.threads = kGramThreads;
  p.blocks = ((g.Vs + cols - 1) / cols) * 3;
  p.smem = gram_smem_bytes(nc, cols, tstarts, tmax, gevp);
  p.fits = cols <= 32 && (cols & (cols - 1)) == 0 && (nc == 2 || cols >= 2) &&
           p.smem <= 200 * 1024;
  return p;
}

template <class Store, class CT>
int launch_wilson_gram(const Geom &g, const GaugeLinks &l, const Fields4 *second, int rmin,
                       int rmax, int tmin, int tmax, const int *flag, double *partials,
                       int *blocks, cudaStream_t s, int cols, int tstarts, int ndir) {
  const WilsonPlan p = wilson_gram_plan(g, tstarts, tmax, Store::NC, cols, second != nullptr);
  if (!p.fits || l.NE < tstarts + tmax)
    return plan_error("wilson_gram_kernel: block shape does not fit");
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(s, &cap);
  auto go = [&](auto kernel) {
    const int rc = allow_large_smem(kernel, p.smem, cap != cudaStreamCaptureStatusNone);
    if (!rc)
      launch_chained(kernel, dim3(p.blocks / 3, ndir), p.threads, p.smem, s, g, l.U,
                     second ? *second : l.U, l.NE, rmin, rmax, tmin, tmax, p.cols_per_block,
                     partials, flag, tstarts);
    return rc;
  };
  int rc;
  if constexpr (Store::kBytes == 72) // (the spatial loops' links: no GEVP)
    rc = go(wilson_gram_kernel<Store, CT, false>);
  else
    rc = second ? go(wilson_gram_kernel<Store, CT, true>)
                : go(wilson_gram_kernel<Store, CT, false>);
  *blocks = p.blocks / 3 * ndir;
  return rc ? rc : launch_check("wilson_gram_kernel");
}

#define GC_INSTANTIATE_GRAM(STORE, CT)                                                        \
  template int launch_wilson_gram<STORE, CT>(const Geom &, const GaugeLinks &,                \
                                             const Fields4 *, int, int, int, int, const int *, \
                                             double *, int *, cudaStream_t, int, int, int);

GC_INSTANTIATE_GRAM(StoreF64SU3, double)
GC_INSTANTIATE_GRAM(StoreF64SU2, double)
GC_INSTANTIATE_GRAM(StoreF32SU3, float)
GC_INSTANTIATE_GRAM(StoreF32SU3Full, float)
GC_INSTANTIATE_GRAM(StoreF32SU2, float)

} // namespace gc
