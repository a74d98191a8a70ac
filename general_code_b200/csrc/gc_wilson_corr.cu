// Fundamental on-axis loops of the temporal gauge as correlations along time
// (sm_100a). gc_wilson_gauge.cu has the gauge and the transformed links,
// gc_corr.cuh the correlation.
//
// A block owns `cols` columns (s, nu) on all NE slices; the space lines lie in
// shared memory as sequences over t, one per (element, column). Per R: each
// thread extends its slots' lines by one transformed link, a barrier, a thread
// per sequence correlates it, the warps' sums are left in shared memory, a
// barrier, and the sums over the warps (in order) are the block's partial. The
// fixed-order tree over blocks of gc_wilson.cu finishes.
//
// Against a thread that keeps the lines of four start slices and reads the end
// lines (18 reals for 72 multiply-adds, 4 for 16), a sequence's window makes
// the same products from a quarter (SU(3) T <= 16) to a sixth (SU(2) T <= 24)
// of the shared-memory reads, and a block's sums are one warp reduction per 32
// sequences instead of a pass over per-thread values in shared memory; against
// the FP64 matrix instructions (gc_wilson_gram.cu) it computes only the band.
// Bound: instruction issue (SU(3) mixed 32^4: 74% of the slots, FMA pipe 49%,
// 24 warps on an SM; SU(2) 48^4 77% and 51%; SU(3) FP64 24^4 shared-memory
// wavefronts 66%, FP64 pipe 49%). R,T <= L/2, whole W calls: SU(3) mixed 32^4
// 2.70 -> 1.84 ms, 24^4 0.75 -> 0.50, 18 x 20 x 22 x 26 0.48 -> 0.29; SU(2)
// mixed 48^4 5.16 -> 3.52; SU(3) FP64 24^4 0.80 -> 0.74. (The mixed figures with
// the short FP32 sums of gc_corr.cuh; the shares were taken with one chain over
// all starts, 5-17% faster.)
//
// 8 SU(3) columns a block (144 sequences, five warps, five blocks on an SM): 16
// with nine warps took 1.86 ms at 32^4. A warp stays on 8 columns, four slices
// at a time, so that its link loads and its writes move whole 128-byte rows and
// cover the banks once; with the column changing between slots the index
// arithmetic was a third of the instructions (SU(2) 48^4 3.21 ms). One link at
// a time for SU(3): three in flight spill at this occupancy (2.12 ms).
#include "gc_corr.cuh"
#include "gc_internal.cuh"
#include "gc_kernels.h"
#include "gc_rows01.cuh"
#include "gc_wcol.cuh"

#include <algorithm>
#include <type_traits>

namespace gc {

namespace {

// T values of a thread's window: their sums (FP32 two sets) and the window take
// 3 J registers (FP64 4 J). More spill: 24 for SU(2) 48^4, T <= 24, 3.86 ms
// against 3.57 in two windows of 12; 20 for SU(3) 32^4, T <= 16, 1.95 ms against
// 1.90. (24 with four blocks on an SM does not, and takes 3.43 ms, but 32^3 x 40,
// T <= 20, 0.64 ms against 0.60.)
constexpr int corr_jmax(int nc, size_t ct_bytes) { return ct_bytes == 8 ? 12 : nc == 2 ? 20 : 16; }
// Starts of one pass: equal shares of tstarts, whole vectors.
__device__ __forceinline__ int corr_pass(int tstarts, int V) {
  const int n = (tstarts + kCorrPass - 1) / kCorrPass;
  return ((tstarts + n - 1) / n + V - 1) / V * V;
}
template <class Store> constexpr int corr_elems() { return Store::NC == 3 ? 18 : 4; }

// A line's elements as sequences: element k of column c at (k cols + c) st.
template <class T> __device__ __forceinline__ void put_seq(T *p, int es, const SU3<T> &m) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    p[(2 * k) * es] = m.e[k / 3][k % 3].re;
    p[(2 * k + 1) * es] = m.e[k / 3][k % 3].im;
  }
}
template <class T> __device__ __forceinline__ void put_seq(T *p, int es, const SU2<T> &q) {
  p[0] = q.a0;
  p[es] = q.a1;
  p[2 * es] = q.a2;
  p[3 * es] = q.a3;
}
template <class T> __device__ __forceinline__ SU3<T> get_seq(const T *p, int es, SU3<T> *) {
  SU3<T> a;
#pragma unroll
  for (int k = 0; k < 9; k++)
    a.e[k / 3][k % 3] = {p[(2 * k) * es], p[(2 * k + 1) * es]};
  return a;
}
template <class T> __device__ __forceinline__ SU2<T> get_seq(const T *p, int es, SU2<T> *) {
  return {p[0], p[es], p[2 * es], p[3 * es]};
}
template <class Store, class T, class M>
__device__ __forceinline__ void extend_seq(T *p, int es, const M &u) {
  if constexpr (Store::kBytes == 48) {
    // products of SU(3) links: rows 0 and 1, row 2 rebuilt
    SU3<float> a;
#pragma unroll
    for (int k = 0; k < 6; k++)
      a.e[k / 3][k % 3] = {p[(2 * k) * es], p[(2 * k + 1) * es]};
    a = mul01(a, u);
    rebuild_row2(a);
    put_seq(p, es, a);
  } else {
    put_seq(p, es, mul(get_seq(p, es, (M *)nullptr), u));
  }
}

template <class Store, class CT> constexpr int corr_batch() {
  return Store::NC == 2 ? 4 : 1;
}

template <class Store, class CT>
__global__ void __launch_bounds__(Store::NC == 3 ? 160 : 128, Store::NC == 2 || sizeof(CT) == 4 ? 5 : 4)
    wilson_corr_kernel(const __grid_constant__ Geom g, const __grid_constant__ Fields4 U, int NE,
                       int rmin, int rmax, int tmin, int tmax, int cols, double *partials,
                       const int *flag, int tstarts) {
  wait_previous();
  // the exact product runs instead when a link failed the check
  if (flag && *flag != 0)
    return;
  constexpr int K = corr_elems<Store>(), V = CorrVec<CT>::V, kBatch = corr_batch<Store, CT>();
  constexpr int JMAX = corr_jmax(Store::NC, sizeof(CT));
  using Raw = RawLink<Store, CT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int nt = tmax - tmin + 1;
  const int nslots = min(NE, tstarts + tmax); // slices the loops touch
  const CorrRange cr = corr_range(tmin, tmax, V, JMAX);
  const int pass = corr_pass(tstarts, V);
  const int st = corr_stride(cr, nslots, tstarts, V), es = cols * st, nred = cr.n * cr.J;
  CT *seq = reinterpret_cast<CT *>(smem_raw);                 // [K][cols][st]
  double *red = reinterpret_cast<double *>(seq + (size_t)K * es); // [nwarps][nred]

  const int nu = blockIdx.y;
  const int base = column_base(g, blockIdx.x, cols, nu);
  const int Ln = sel4(g.L, nu), stn = sel4(g.stride, nu);
  const size_t VE = (size_t)NE * g.Vs;
  const void *f = U.f[nu];
  double *part = partials + ((size_t)blockIdx.y * gridDim.x + blockIdx.x) * (rmax - rmin + 1) * nt;

  // the thread's column and slices t0, t0 + tstep, ...: a warp extends 8
  // columns x 4 slices at a time
  const int cg = cols >> 3;
  const int c = (warp & (cg - 1)) * 8 + (lane & 7);
  const int t0 = warp / cg * 4 + (lane >> 3), tstep = nwarps / cg * 4;
  const int s = base + c, tend = s < g.Vs ? nslots : 0;
  const int xn = (s / stn) % Ln;
  CT *own = seq + c * st;
  // columns past the lattice and elements past the last slice count as zeros
  for (int i = tid; i < K * es; i += blockDim.x)
    seq[i] = CT(0);
  __syncthreads();

  int l = s, pos = xn; // the column's link of this R, its coordinate
#pragma unroll 1
  for (int R = 1; R <= rmax; R++) {
#pragma unroll 1
    for (int t = t0; t < tend; t += kBatch * tstep) {
      Raw x[kBatch];
#pragma unroll
      for (int j = 0; j < kBatch; j++)
        if (t + j * tstep < tend)
          x[j].load(f, VE, l + (t + j * tstep) * g.Vs);
#pragma unroll
      for (int j = 0; j < kBatch; j++)
        if (t + j * tstep < tend) {
          CT *p = own + t + j * tstep;
          if (R == 1)
            put_seq(p, es, x[j].link());
          else
            extend_seq<Store>(p, es, x[j].link());
        }
    }
    l += stn;
    if (++pos == Ln) {
      pos = 0;
      l -= Ln * stn;
    }
    __syncthreads();
    if (R >= rmin) {
      const CT *mine = seq + min(tid, K * cols - 1) * st;
      const bool valid = tid < K * cols;
#pragma unroll 1
      for (int ch = 0; ch < cr.n; ch++) {
        const int T = cr.first + ch * cr.J;
        auto run = [&](auto jj) {
          constexpr int J = decltype(jj)::value;
          auto part = [&](int t, int n, bool more) {
            CT acc[J];
#pragma unroll
            for (int j = 0; j < J; j++)
              acc[j] = CT(0);
            if (valid) {
              if (T == 1)
                correlate<CT, J, true>(mine + t, T, n, acc);
              else
                correlate<CT, J, false>(mine + t, T, n, acc);
            }
            corr_warp_sum<CT, J>(acc, lane, red + warp * nred + ch * J, more);
          };
          if constexpr (sizeof(CT) == 8)
            part(0, tstarts, false);
          else
#pragma unroll 1
            for (int t = 0; t < tstarts; t += pass)
              part(t, min(pass, tstarts - t), t > 0);
        };
        using std::integral_constant;
        switch (cr.J) {
        case 4: run(integral_constant<int, 4>()); break;
        case 8: run(integral_constant<int, 8>()); break;
        case 12: run(integral_constant<int, 12>()); break;
        case 16:
          if constexpr (JMAX >= 16)
            run(integral_constant<int, 16>());
          break;
        case 20:
          if constexpr (JMAX >= 20)
            run(integral_constant<int, 20>());
        }
      }
    }
    __syncthreads();
    if (R >= rmin)
      for (int i = tid; i < nt; i += blockDim.x) {
        double v = 0.0;
        for (int w = 0; w < nwarps; w++)
          v += red[w * nred + tmin - cr.first + i];
        part[(R - rmin) * nt + i] = v;
      }
  }
}

} // namespace

WilsonPlan wilson_corr_plan(const Geom &g, int tstarts, int tmin, int tmax, int nc, int ct_bytes,
                            int cols_req) {
  WilsonPlan p{};
  const int V = 16 / ct_bytes, K = nc == 3 ? 18 : 4;
  const CorrRange cr = corr_range(tmin, tmax, V, corr_jmax(nc, ct_bytes));
  const int st = corr_stride(cr, tstarts + tmax, tstarts, V);
  auto shape = [&](int cols) {
    p.cols_per_block = cols;
    p.threads = (K * cols + 31) / 32 * 32;
    p.smem = (size_t)K * cols * st * ct_bytes + (size_t)p.threads / 32 * cr.n * cr.J * 8;
  };
  shape(cols_req > 0 ? cols_req : nc == 3 ? 8 : 32);
  if (cols_req <= 0)
    while (p.cols_per_block > 8 && p.smem > 72 * 1024)
      shape(p.cols_per_block / 2);
  p.kernel = 4;
  p.rows = 8; // (the autotuner's bound on columns: 256 / rows)
  p.blocks = ((g.Vs + p.cols_per_block - 1) / p.cols_per_block) * 3;
  p.fits = p.cols_per_block >= 8 && (p.cols_per_block & (p.cols_per_block - 1)) == 0 &&
           p.threads <= (nc == 3 ? 160 : 128) && p.smem <= 200 * 1024;
  return p;
}

template <class Store, class CT>
int launch_wilson_corr(const Geom &g, const GaugeLinks &l, int rmin, int rmax, int tmin, int tmax,
                       const int *flag, double *partials, int *blocks, cudaStream_t s, int cols,
                       int tstarts, int ndir) {
  const WilsonPlan p =
      wilson_corr_plan(g, tstarts, tmin, tmax, Store::NC, (int)sizeof(CT), cols);
  if (!p.fits || l.NE < tstarts + tmax)
    return plan_error("wilson_corr_kernel: block shape does not fit");
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(s, &cap);
  int rc = allow_large_smem(wilson_corr_kernel<Store, CT>, p.smem,
                            cap != cudaStreamCaptureStatusNone);
  if (rc)
    return rc;
  launch_chained(wilson_corr_kernel<Store, CT>, dim3(p.blocks / 3, ndir), p.threads, p.smem, s, g,
                 l.U, l.NE, rmin, rmax, tmin, tmax, p.cols_per_block, partials, flag, tstarts);
  *blocks = p.blocks / 3 * ndir;
  return launch_check("wilson_corr_kernel");
}

#define GC_INSTANTIATE_CORR(STORE, CT)                                                         \
  template int launch_wilson_corr<STORE, CT>(const Geom &, const GaugeLinks &, int, int, int,  \
                                             int, const int *, double *, int *, cudaStream_t,  \
                                             int, int, int);

GC_INSTANTIATE_CORR(StoreF64SU3, double)
GC_INSTANTIATE_CORR(StoreF64SU2, double)
GC_INSTANTIATE_CORR(StoreF32SU3, float)
GC_INSTANTIATE_CORR(StoreF32SU3Full, float)
GC_INSTANTIATE_CORR(StoreF32SU2, float)

} // namespace gc
