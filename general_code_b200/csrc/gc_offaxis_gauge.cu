// Off-axis Wilson loops in the temporal gauge (sm_100a): the loops of
// gc_offaxis.cu (reference wilson_offaxis / wilson_offaxis_adjoint,
// lib/cpu/include/wilson_loops.h:313-663) from the transformed links of
// gc_wilson_gauge.cu.
//
// In the temporal gauge a time line is 1, so a loop of the space line S' (the
// product of the transformed links along its steps) is
// Re Tr[S'(x + T t) S'(x)^dag]: one trace instead of the two products of the
// exact walk. The lines are needed on the Lt start slices and, for the loops
// that pass the last one, on tmax further slices.
//
// The lines themselves cost more than their loops then (5 links and 6 loops
// per line at r, T <= 6). Many are equal step for step (the reference counts
// an orientation twice, and permutations repeat symmetric patterns), and many
// begin alike: as a tree with a node per step the 678 lines of r <= 6 (4473
// links) are 550 distinct lines and 1140 products (gc_offaxis_tree.h builds the
// tree). A block walks a part of
// the tree in depth-first order for its columns: a thread owns one line slot
// (column, slice), keeps the current product in registers and the
// products that a later branch continues on a short private stack (the
// largest branch is walked last, so the stack holds at most log2 of the nodes).
// The link of the next node is loaded while the current one is multiplied
// and its loops are summed.
//
// A finished line goes to shared memory (two buffers, one barrier per line),
// each thread adds the traces of the loops that start on its slot, and the
// per-thread values of one line are summed over the block in fixed order
// behind the next line's barrier; the grid sums the blocks as elsewhere.
//
// Bound: instruction issue at 20 warps per SM (57% of the issue slots; 28% of
// the FMA pipe; 3.3 TB/s from L2 at 16^4). r, T <= 6 at SU(3) 24^4, mixed
// 31.9 -> 12.3 ms, FP64 55.8 -> 21.4 ms; SU(2) mixed 10.8 -> 4.8 ms against
// the exact walk of every line (gc_offaxis.cu), which stays for T > Lt/2 and
// for links off the group.
#include "gc_internal.cuh"
#include "gc_kernels.h"
#include "gc_rows01.cuh"
#include "gc_wcol.cuh"

#include <algorithm>
#include <type_traits>

namespace gc {

namespace {

// A line slot's matrix in shared memory: planes of 16-byte vectors (and one
// of 8 bytes for the 18 reals of an FP32 SU(3) matrix) over the block's slots.
template <class M> struct SlotSet;
template <> struct SlotSet<SU3<double>> {
  static constexpr int kBytes = 144;
  __device__ __forceinline__ static void store(unsigned char *p, int n, int i,
                                               const SU3<double> &m) {
    double2 *q = reinterpret_cast<double2 *>(p) + i;
#pragma unroll
    for (int k = 0; k < 9; k++)
      q[k * n] = make_double2(m.e[k / 3][k % 3].re, m.e[k / 3][k % 3].im);
  }
  __device__ __forceinline__ static SU3<double> load(const unsigned char *p, int n, int i) {
    const double2 *q = reinterpret_cast<const double2 *>(p) + i;
    SU3<double> m;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      const double2 v = q[k * n];
      m.e[k / 3][k % 3] = {v.x, v.y};
    }
    return m;
  }
};
template <> struct SlotSet<SU3<float>> {
  static constexpr int kBytes = 72;
  __device__ __forceinline__ static void store(unsigned char *p, int n, int i,
                                               const SU3<float> &m) {
    float4 *q = reinterpret_cast<float4 *>(p) + i;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const cx<float> a = m.e[2 * k / 3][2 * k % 3], b = m.e[(2 * k + 1) / 3][(2 * k + 1) % 3];
      q[k * n] = make_float4(a.re, a.im, b.re, b.im);
    }
    reinterpret_cast<float2 *>(p + 64 * (size_t)n)[i] = make_float2(m.e[2][2].re, m.e[2][2].im);
  }
  __device__ __forceinline__ static SU3<float> load(const unsigned char *p, int n, int i) {
    const float4 *q = reinterpret_cast<const float4 *>(p) + i;
    SU3<float> m;
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float4 v = q[k * n];
      m.e[2 * k / 3][2 * k % 3] = {v.x, v.y};
      m.e[(2 * k + 1) / 3][(2 * k + 1) % 3] = {v.z, v.w};
    }
    const float2 v = reinterpret_cast<const float2 *>(p + 64 * (size_t)n)[i];
    m.e[2][2] = {v.x, v.y};
    return m;
  }
};
template <class T> struct SlotSet<SU2<T>> {
  static constexpr int kBytes = 4 * sizeof(T);
  using V = typename V2<T>::type;
  __device__ __forceinline__ static void store(unsigned char *p, int n, int i, const SU2<T> &m) {
    V *q = reinterpret_cast<V *>(p) + i;
    q[0] = V{m.a0, m.a1};
    q[n] = V{m.a2, m.a3};
  }
  __device__ __forceinline__ static SU2<T> load(const unsigned char *p, int n, int i) {
    const V *q = reinterpret_cast<const V *>(p) + i;
    const V a = q[0], b = q[n];
    return {a.x, a.y, b.x, b.y};
  }
};

// P <- P u or P u^dag, and the first factor. FP32 SU(3) products keep rows 0
// and 1 (gc_rows01.cuh); finish() rebuilds row 2 for the traces.
template <class M> struct LineOps {
  __device__ __forceinline__ static M first(const M &u, bool back) { return back ? adjoint(u) : u; }
  __device__ __forceinline__ static M extend(const M &P, const M &u, bool back) {
    return back ? mul_ad(P, u) : mul(P, u);
  }
  __device__ __forceinline__ static void finish(M &) {}
};
template <> struct LineOps<SU3<float>> {
  using M = SU3<float>;
  __device__ __forceinline__ static M first(const M &u, bool back) { return back ? adjoint(u) : u; }
  __device__ __forceinline__ static M extend(const M &P, const M &u, bool back) {
    return back ? mul_ad01(P, u) : mul01(P, u);
  }
  __device__ __forceinline__ static void finish(M &P) { rebuild_row2(P); }
};

// Slot i of a column is slice i of the extended lattice; the loops of a start
// slot i < Lt end on slot i + T.
__host__ __device__ inline int gauge_slots(int Lt, int tmax) { return Lt + tmax; }

struct GaugeShape {
  int cols, threads;
  size_t smem;
};
GaugeShape gauge_shape(const Geom &g, int nc, int ct_bytes, int tmin, int tmax, bool adjoint) {
  GaugeShape f{};
  const int n = gauge_slots(g.L[3], tmax), nt = tmax - tmin + 1;
  const size_t mat = (nc == 3 ? 18 : 4) * (size_t)ct_bytes;
  const size_t acc = (!adjoint && ct_bytes == 4) ? 4 : 8;
  auto set = [&](int cols) {
    f.cols = cols;
    f.threads = (n * cols + 31) / 32 * 32;
    f.smem = 2 * (size_t)f.threads * (mat + nt * acc);
  };
  // about 160 threads per block (FP32 about 256), a power of two of columns:
  // their links share the 32-byte sectors
  const int want = ct_bytes == 4 ? 320 : 160;
  int cols = 1;
  while (2 * cols * n <= want && 2 * cols <= 32)
    cols *= 2;
  set(cols);
  if (f.threads > 512 || f.smem > 200 * 1024)
    f.cols = 0;
  return f;
}

template <class Store, class CT, bool ADJ>
__global__ void __launch_bounds__(512)
    offaxis_gauge_kernel(const __grid_constant__ Geom g, const __grid_constant__ Fields4 U,
                         int NE, const OffaxisNode *__restrict__ nodes,
                         const int *__restrict__ chunk_nodes, int line0, int nlines, int tmin,
                         int tmax, int cols, double *partials, const int *flag) {
  wait_previous();
  if (*flag != 0)
    return;
  using M = typename Store::template M<CT>;
  using SS = SlotSet<M>;
  using Acc = GAcc<ADJ, CT>;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int Lt = g.L[3], nt = tmax - tmin + 1;
  const int nth = blockDim.x, tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31, nwarps = nth >> 5;
  unsigned char *lines = smem_raw; // [2][SS::kBytes * nth]
  Acc *red = reinterpret_cast<Acc *>(smem_raw + 2 * (size_t)SS::kBytes * nth); // [2][nt][nth]
  const int c = tid % cols, slot = tid / cols;
  const int s = blockIdx.x * cols + c;
  const bool active = slot < gauge_slots(Lt, tmax) && s < g.Vs;
  const bool starts = active && slot < Lt; // loops start on this slot
  const int x0 = s % g.L[0], x1 = (s / g.L[0]) % g.L[1], x2 = s / (g.L[0] * g.L[1]);
  const size_t VE = (size_t)NE * g.Vs;
  const int toff = slot * g.Vs;
  for (int i = tid; i < 2 * nt * nth; i += nth)
    red[i] = Acc(0);

  // the link of a node, seen from this slot
  auto link = [&](const int4 &d) {
    int y0 = x0 + d.x, y1 = x1 + d.y, y2 = x2 + d.z;
    y0 -= y0 >= g.L[0] ? g.L[0] : 0;
    y1 -= y1 >= g.L[1] ? g.L[1] : 0;
    y2 -= y2 >= g.L[2] ? g.L[2] : 0;
    return y0 + g.L[0] * (y1 + g.L[1] * y2) + toff;
  };
  auto field = [&](int axis) { return axis == 0 ? U.f[0] : axis == 1 ? U.f[1] : U.f[2]; };

  const int n0 = chunk_nodes[blockIdx.y], n1 = chunk_nodes[blockIdx.y + 1];
  const int4 *desc = reinterpret_cast<const int4 *>(nodes);
  M P, stack[kTreeStack];
  int done = 0, prev = -1; // lines finished by this block, the last one
  int4 d = __ldg(desc + 2 * n0);
  int ops = __ldg(reinterpret_cast<const int *>(desc + 2 * n0 + 1));
  M u;
  if (active)
    u = Store::template load<CT>(field(ops & 0xff), VE, link(d));
#pragma unroll 1
  for (int n = n0; n < n1; n++) {
    const int line = d.w;
    const bool back = (ops >> 8) & 1;
    const int from = (signed char)(ops >> 16), push = ops >> 24;
    if (active) {
      if (from == -2) {
        P = LineOps<M>::first(u, back);
      } else {
        if (from >= 0)
          P = stack[from];
        P = LineOps<M>::extend(P, u, back);
      }
      if (push >= 0)
        stack[push] = P;
    }
    if (n + 1 < n1) {
      d = __ldg(desc + 2 * n + 2);
      ops = __ldg(reinterpret_cast<const int *>(desc + 2 * n + 3));
      if (active)
        u = Store::template load<CT>(field(ops & 0xff), VE, link(d));
    }
    if (line < 0)
      continue;
    M a = P;
    LineOps<M>::finish(a);
    unsigned char *buf = lines + (done & 1) * (size_t)SS::kBytes * nth;
    Acc *r = red + (done & 1) * (size_t)nt * nth;
    if (active)
      SS::store(buf, nth, tid, a);
    __syncthreads();
    // the previous line's sums (its values were written before this barrier)
    if (prev >= 0) {
      const Acc *rp = red + ((done & 1) ^ 1) * (size_t)nt * nth;
#pragma unroll 1
      for (int T = warp; T < nt; T += nwarps) {
        double v = 0.0;
        for (int i = lane; i < nth; i += 32)
          v += double(rp[(size_t)T * nth + i]);
        v = warp_sum(v);
        if (lane == 0)
          partials[((size_t)blockIdx.x * nlines + prev - line0) * nt + T] = v;
      }
    }
    if (starts) {
#pragma unroll 2
      for (int T = tmin; T <= tmax; T++)
        r[(size_t)(T - tmin) * nth + tid] =
            gauge_trace<ADJ>(a, SS::load(buf, nth, tid + T * cols), false);
    }
    prev = line;
    done++;
  }
  __syncthreads();
  if (prev >= 0) {
    const Acc *rp = red + ((done & 1) ^ 1) * (size_t)nt * nth;
#pragma unroll 1
    for (int T = warp; T < nt; T += nwarps) {
      double v = 0.0;
      for (int i = lane; i < nth; i += 32)
        v += double(rp[(size_t)T * nth + i]);
      v = warp_sum(v);
      if (lane == 0)
        partials[((size_t)blockIdx.x * nlines + prev - line0) * nt + T] = v;
    }
  }
}

} // namespace

int offaxis_gauge_blocks(const Geom &g, int nc, int ct_bytes, int tmin, int tmax, bool adjoint) {
  if (g.L[3] < 2 || tmax > g.L[3] / 2)
    return 0;
  const GaugeShape f = gauge_shape(g, nc, ct_bytes, tmin, tmax, adjoint);
  return f.cols ? (g.Vs + f.cols - 1) / f.cols : 0;
}

template <class Store, class CT>
int launch_offaxis_gauge(const Geom &g, const GaugeLinks &l, const OffaxisNode *nodes,
                         const int *chunk_nodes, int chunk0, int nchunks,
                         int line0, int nlines, int tmin, int tmax, bool adjoint,
                         double *partials, const int *flag, cudaStream_t s) {
  const GaugeShape f = gauge_shape(g, Store::NC, (int)sizeof(CT), tmin, tmax, adjoint);
  if (!f.cols || tmax > g.L[3] / 2 || l.NE < g.L[3] + tmax)
    return plan_error("offaxis_gauge_kernel: block shape does not fit");
  const dim3 grid((g.Vs + f.cols - 1) / f.cols, nchunks);
  auto go = [&](auto kernel) {
    const int rc = allow_large_smem(kernel, f.smem);
    if (!rc)
      launch_chained(kernel, grid, f.threads, f.smem, s, g, l.U, l.NE, nodes, chunk_nodes + chunk0,
                     line0, nlines, tmin, tmax, f.cols, partials, flag);
    return rc;
  };
  const int rc = adjoint ? go(offaxis_gauge_kernel<Store, CT, true>)
                         : go(offaxis_gauge_kernel<Store, CT, false>);
  return rc ? rc : launch_check("offaxis_gauge_kernel");
}

#define GC_INSTANTIATE_OG(STORE, CT)                                                         \
  template int launch_offaxis_gauge<STORE, CT>(                                              \
      const Geom &, const GaugeLinks &, const OffaxisNode *, const int *, int, int, int, int,  \
      int, int, bool, double *, const int *, cudaStream_t);

GC_INSTANTIATE_OG(StoreF64SU3, double)
GC_INSTANTIATE_OG(StoreF64SU2, double)
GC_INSTANTIATE_OG(StoreF32SU3, float)
GC_INSTANTIATE_OG(StoreF32SU2, float)

} // namespace gc
