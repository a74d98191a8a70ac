// Polyakov loops and their correlators (sm_100a).
//
// Reference (lib/cpu/include/polyakov_loops.h):
//   get_polyakov_loop            :10-22  P(s) = U_t(s,0) U_t(s,1) ... U_t(s,Lt-1)
//   polyakov_loop                :24-41  mean over spatial sites of tr_real P
//   polyakov_loop_correlator_color_average  :83-145
//       C(D) = (1/Vs) sum_s Re[ tr P(s) conj(tr P(s+D)) ],  tr = Tr / N
//   polyakov_loop_correlator_singlet        :147-206
//       C(D) = (1/Vs) sum_s Re Tr[ P(s) P(s+D)^dag ] / N
// for the offsets D = (Dx,Dy,Dz) with |D| <= D_max that the reference visits
// (Dx >= 0 when Dy and Dz are both non-zero), stored at
// (Dz+D_max)(2D_max+1)^2 + (Dy+D_max)(2D_max+1) + Dx+D_max; other entries 0.
//
// polyakov_lines_kernel: thread per spatial site, the Lt time links of the
// site's column read in order (coalesced across threads), the product kept
// in the compute type and stored in FP64 as element planes
// (SU(3): 9 double2 planes, SU(2): 2 double2 planes, Vs entries each, and one
// plane of normalised traces), with
// fixed-order block sums of Re Tr P for the loop itself.
// The correlators are sums over components k (double2 planes: 9 for SU(3)
// singlets, 2 for SU(2), 1 for the traces) of products p_k(s) . p_k(s + D).
// polyakov_rows_kernel: a block holds a few rows (y, z) of one slice and the
// rows they meet for a run of dy at one dz in shared memory; a thread sums one
// component and one dy over x for all dx of its tile, eight sites and the
// tile's accumulators in registers, so that a load serves six
// multiply-adds.
// C(-D) = C(D), so only dx >= 0 is computed. polyakov_correlator_kernel, one
// block per offset with every operand read from L2 for one multiply-add pair,
// serves lattices whose rows do not fit. Fixed-order sums throughout.
#include "gc_internal.cuh"
#include "gc_kernels.h"

#include <algorithm>
#include <type_traits>

namespace gc {

namespace {

// FP64 element planes of the Polyakov lines (SU(3): 9 planes, SU(2): 2).
__device__ __forceinline__ void line_store(double2 *lines, int Vs, int s, const SU3<double> &m) {
#pragma unroll
  for (int k = 0; k < 9; k++)
    lines[(size_t)k * Vs + s] = make_double2(m.e[k / 3][k % 3].re, m.e[k / 3][k % 3].im);
}
__device__ __forceinline__ void line_store(double2 *lines, int Vs, int s, const SU2<double> &m) {
  lines[s] = make_double2(m.a0, m.a1);
  lines[(size_t)Vs + s] = make_double2(m.a2, m.a3);
}
__device__ __forceinline__ void line_load(const double2 *lines, int Vs, int s, SU3<double> &m) {
#pragma unroll
  for (int k = 0; k < 9; k++) {
    const double2 v = __ldg(lines + (size_t)k * Vs + s);
    m.e[k / 3][k % 3] = {v.x, v.y};
  }
}
__device__ __forceinline__ void line_load(const double2 *lines, int Vs, int s, SU2<double> &m) {
  const double2 a = __ldg(lines + s), b = __ldg(lines + (size_t)Vs + s);
  m = {a.x, a.y, b.x, b.y};
}

// tr P = Tr P / N: SU(3) complex, SU(2) the real a0 (the quaternion trace).
__device__ __forceinline__ double2 norm_trace(const SU3<double> &m) {
  return make_double2((m.e[0][0].re + m.e[1][1].re + m.e[2][2].re) / 3.0,
                      (m.e[0][0].im + m.e[1][1].im + m.e[2][2].im) / 3.0);
}
__device__ __forceinline__ double2 norm_trace(const SU2<double> &m) {
  return make_double2(m.a0, 0.0);
}

template <class T> __device__ __forceinline__ SU3<double> to_double(const SU3<T> &a) {
  return convert(a, (SU3<double> *)nullptr);
}
template <class T> __device__ __forceinline__ SU2<double> to_double(const SU2<T> &a) {
  return convert(a, (SU2<double> *)nullptr);
}

__device__ __forceinline__ double block_sum(double v, double *sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if (threadIdx.x < w)
      sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  return sh[0];
}

template <class Store, class CT>
__global__ void __launch_bounds__(256)
    polyakov_lines_kernel(const __grid_constant__ Geom g, const void *Ut, double2 *lines,
                          double *partials) {
  wait_previous();
  using M = typename Store::template M<CT>;
  using MD = typename Store::template M<double>;
  __shared__ double sh[256];
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  double tr = 0.0;
  if (s < g.Vs) {
    const size_t V = g.V;
    M A = Store::template load<CT>(Ut, V, s);
#pragma unroll 1
    for (int t = 1; t < g.L[3]; t++)
      A = mul(A, Store::template load<CT>(Ut, V, s + t * g.Vs));
    const MD P = to_double(A);
    line_store(lines, g.Vs, s, P);
    const double2 ntr = norm_trace(P);
    lines[(size_t)(Store::NC == 3 ? 9 : 2) * g.Vs + s] = ntr; // the trace's own plane
    tr = ntr.x;
  }
  const double b = block_sum(tr, sh);
  if (threadIdx.x == 0)
    partials[blockIdx.x] = b;
}

// offsets[i] = (Dx, Dy, Dz, place) of the i-th visited offset.
template <class MD, bool SINGLET>
__global__ void __launch_bounds__(256)
    polyakov_correlator_kernel(const __grid_constant__ Geom g, const double2 *lines,
                               const int4 *offsets, double scale, double *out) {
  __shared__ double sh[256];
  const int4 off = offsets[blockIdx.x];
  const int Lx = g.L[0], Ly = g.L[1], Lz = g.L[2];
  // shifts as non-negative residues
  const int dx = ((off.x % Lx) + Lx) % Lx, dy = ((off.y % Ly) + Ly) % Ly,
            dz = ((off.z % Lz) + Lz) % Lz;
  double acc = 0.0;
#pragma unroll 1
  for (int s = threadIdx.x; s < g.Vs; s += blockDim.x) {
    const int x = s % Lx, y = (s / Lx) % Ly, z = s / (Lx * Ly);
    int x2 = x + dx, y2 = y + dy, z2 = z + dz;
    x2 -= (x2 >= Lx) ? Lx : 0;
    y2 -= (y2 >= Ly) ? Ly : 0;
    z2 -= (z2 >= Lz) ? Lz : 0;
    const int s2 = x2 + Lx * (y2 + Ly * z2);
    MD a, b;
    line_load(lines, g.Vs, s, a);
    line_load(lines, g.Vs, s2, b);
    if (SINGLET) {
      // multiply_conj_tr: Re Tr(a b^dag) / N
      acc += conj_tr(a, b);
    } else {
      const double2 p = norm_trace(a), q = norm_trace(b);
      acc += fma(p.y, q.y, p.x * q.x); // Re(p conj(q))
    }
  }
  const double sum = block_sum(acc, sh);
  if (threadIdx.x == 0)
    out[off.w] = sum * scale;
}

constexpr int kRowsY = 4;   // rows of a block
constexpr int kRowsDy = 8;  // dy values of a block
constexpr int kRowsX = 8;   // sites of a thread's tile

// Shared rows: element (row, k, x) at row * NP * sx + k * sx + x, sx = 1 mod 8,
// so that lanes (k fastest, then dy) read consecutive banks.
__host__ __device__ inline int rows_sx(int Lx) { return (Lx + 6) / 8 * 8 + 1; }
constexpr int rows_groups(int NP) { return NP == 9 ? 4 : 16; } // thread groups over (row, x tile)

__device__ __forceinline__ void copy_async(double2 *smem, const double2 *global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(smem)),
               "l"(global)
               : "memory");
}

// Bound by shared-memory loads: a tile of 8 sites makes 24 of them for DXT = 9
// and they serve 144 FP64 fma; on 32^3, D = 8, SU(3) singlet, 280 us with the
// load/store pipe 67% busy and the FP64 pipe 27% (the form with a block per
// offset reads 18 operands from L2 for 18 fma). 6 or 9 dy a block, or 8 thread
// groups, measured no better; so did copies without cp.async (worse).
// partials[row tile][dz][dy][dx]: dz = dz0 + blockIdx.y / nch, dy = -D +
// kRowsDy (blockIdx.y % nch) + i, dx = DXT blockIdx.z + j. p: NP planes.
template <int NP, int DXT>
__global__ void __launch_bounds__(NP * kRowsDy * rows_groups(NP))
    polyakov_rows_kernel(const __grid_constant__ Geom g, const double2 *__restrict__ p, int D,
                         int dz0, int nch, double *partials) {
  wait_previous();
  extern __shared__ __align__(16) double2 rows[];
  constexpr int NG = rows_groups(NP), nth = NP * kRowsDy * NG;
  const int Lx = g.L[0], Ly = g.L[1], Lz = g.L[2], sx = rows_sx(Lx);
  const int tid = threadIdx.x;
  const int k = tid % NP, dyi = tid / NP % kRowsDy, group = tid / (NP * kRowsDy);
  const int ny = (Ly + kRowsY - 1) / kRowsY;
  const int y0 = blockIdx.x % ny * kRowsY, z = blockIdx.x / ny;
  const int dz = dz0 + (int)blockIdx.y / nch, dy0 = -D + (int)blockIdx.y % nch * kRowsDy;
  // the dy of this run nearest to 0 (nothing may lie within the sphere)
  const int near = dy0 > 0 ? dy0 : dy0 + kRowsDy - 1 < 0 ? dy0 + kRowsDy - 1 : 0;
  // and the dx of this tile that lie within it for the nearest dy
  const int room = D * D - near * near - dz * dz;
  int need = 0;
  while (need < DXT && ((int)blockIdx.z * DXT + need) * ((int)blockIdx.z * DXT + need) <= room)
    need++;
  if (need == 0)
    return;
  const int yrows = min(kRowsY, Ly - y0);
  // rows 0 .. kRowsY-1: y0 + r at z; then y0 + dy0 + r at z + dz
  const int nb = kRowsY + kRowsDy - 1;
  const int z2 = ((z + dz) % Lz + Lz) % Lz;
  // (a warp per component and every kStep-th row, by asynchronous copies: all
  // of a warp's rows are in flight, and no division per row)
  constexpr int nwarps = nth / 32, kStep = nwarps / NP;
  static_assert(nth % 32 == 0 && nwarps % NP == 0, "warps per component");
  const int kk = (tid >> 5) % NP, first = (tid >> 5) / NP;
  auto copy_rows = [&](int row0, int count, int y, int zz) {
    const double2 *q = p + (size_t)kk * g.Vs + (size_t)Lx * Ly * zz;
    y = ((y + first) % Ly + Ly) % Ly;
    for (int r = first; r < count; r += kStep) {
      double2 *dst = rows + ((row0 + r) * NP + kk) * sx;
      for (int x = tid & 31; x < Lx; x += 32)
        copy_async(dst + x, q + Lx * y + x);
      for (y += kStep; y >= Ly;)
        y -= Ly;
    }
  };
  copy_rows(0, kRowsY, y0, z);
  copy_rows(kRowsY, nb, y0 + dy0, z2);
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  double acc[DXT];
#pragma unroll
  for (int j = 0; j < DXT; j++)
    acc[j] = 0.0;
  const int nx = (Lx + kRowsX - 1) / kRowsX;
  const int dx0 = (int)blockIdx.z * DXT % Lx;
#pragma unroll 1
  for (int item = group; item < yrows * nx; item += NG) {
    const int r = item / nx, x0 = item % nx * kRowsX;
    const int a = (r * NP + k) * sx + x0, b = ((kRowsY + r + dyi) * NP + k) * sx;
    double2 u[kRowsX];
    if (x0 + kRowsX <= Lx) {
#pragma unroll
      for (int i = 0; i < kRowsX; i++)
        u[i] = rows[a + i];
    } else {
#pragma unroll
      for (int i = 0; i < kRowsX; i++)
        u[i] = x0 + i < Lx ? rows[a + i] : make_double2(0.0, 0.0);
    }
    int x = x0 + dx0;
    x = x >= Lx ? x - Lx : x;
    int v = b + x;
#pragma unroll
    for (int w = 0; w < kRowsX + DXT - 1; w++) {
      if (w >= kRowsX + need - 1)
        break;
      const double2 q = rows[v];
      v = v + 1 == b + Lx ? b : v + 1;
#pragma unroll
      for (int i = 0; i < kRowsX; i++)
        if (w - i >= 0 && w - i < DXT)
          acc[w - i] = fma(u[i].y, q.y, fma(u[i].x, q.x, acc[w - i]));
    }
  }
  __syncthreads();
  // sum over components and groups, in order
  double *red = reinterpret_cast<double *>(rows);
#pragma unroll
  for (int j = 0; j < DXT; j++)
    red[j * nth + tid] = acc[j];
  __syncthreads();
  const int ndx = gridDim.z * DXT;
  for (int e = tid; e < kRowsDy * DXT; e += nth) {
    const int i = e / DXT, j = e % DXT;
    double v = 0.0;
    for (int q = 0; q < NG; q++)
      for (int kk = 0; kk < NP; kk++)
        v += red[j * nth + (q * kRowsDy + i) * NP + kk];
    partials[((size_t)blockIdx.x * gridDim.y * kRowsDy + blockIdx.y * kRowsDy + i) * ndx +
             blockIdx.z * DXT + j] = v;
  }
}

size_t rows_smem(const Geom &g, int NP, int DXT) {
  const size_t rows = (size_t)(2 * kRowsY + kRowsDy - 1) * NP * rows_sx(g.L[0]) * 16;
  return std::max(rows, (size_t)NP * kRowsDy * rows_groups(NP) * DXT * 8);
}

} // namespace

template <class Store, class CT>
int launch_polyakov_lines(const Geom &g, const Fields4 &U, double2 *lines, double *partials,
                          double *out_dev, cudaStream_t s) {
  const int nb = (g.Vs + 255) / 256;
  launch_chained(polyakov_lines_kernel<Store, CT>, nb, 256, 0, s, g, U.f[3], lines, partials);
  int rc = launch_check("polyakov_lines_kernel");
  if (rc)
    return rc;
  if (!out_dev)
    return GC_OK;
  return launch_reduce_sum(partials, nb, 1.0 / (double)g.Vs, out_dev, s);
}

int launch_polyakov_correlator(const Geom &g, int nc, const double2 *lines, const int4 *offsets,
                               int noffsets, bool singlet, double *out_dev, cudaStream_t s) {
  if (noffsets <= 0)
    return GC_OK;
  const double scale = 1.0 / (double)g.Vs;
  if (nc == 3) {
    if (singlet)
      polyakov_correlator_kernel<SU3<double>, true>
          <<<noffsets, 256, 0, s>>>(g, lines, offsets, scale, out_dev);
    else
      polyakov_correlator_kernel<SU3<double>, false>
          <<<noffsets, 256, 0, s>>>(g, lines, offsets, scale, out_dev);
  } else {
    if (singlet)
      polyakov_correlator_kernel<SU2<double>, true>
          <<<noffsets, 256, 0, s>>>(g, lines, offsets, scale, out_dev);
    else
      polyakov_correlator_kernel<SU2<double>, false>
          <<<noffsets, 256, 0, s>>>(g, lines, offsets, scale, out_dev);
  }
  return launch_check("polyakov_correlator_kernel");
}

PolyakovRows polyakov_rows_plan(const Geom &g, int nc, bool singlet, int D) {
  PolyakovRows r{};
  const int NP = singlet ? (nc == 3 ? 9 : 2) : 1;
  r.ndxt = (D + 1 + 8) / 9;
  r.dxt = (D + 1 + r.ndxt - 1) / r.ndxt;
  r.nch = (2 * D + 1 + kRowsDy - 1) / kRowsDy;
  r.row_tiles = (g.L[1] + kRowsY - 1) / kRowsY * g.L[2];
  r.entries = r.nch * kRowsDy * r.ndxt * r.dxt;
  r.dz_per_launch = (int)std::min<size_t>(
      2 * D + 1, std::max<size_t>(1, ((size_t)8 << 20) / ((size_t)r.row_tiles * r.entries)));
  // SU(3) FP64, us per call, this form against a block per offset: 8^3 x 4,
  // D = 2: 49 / 48; 12^3 x 4, D = 3: 52 / 62; 32^3 x 8, D = 8: 339 / 606, D =
  // 16: 1850 / 3217; 48^3 x 8, D = 12: 3031 / 5678; SU(2) 32^3 x 8, D = 8: 149
  // / 267. So it is taken wherever its rows fit the shared memory (SU(3): Lx
  // up to 89) and its partial sums stay below 256 MB.
  r.fits = rows_smem(g, NP, r.dxt) <= 200 * 1024 && (size_t)r.dz_per_launch * r.nch < 65536 &&
           (size_t)r.row_tiles * r.entries <= (size_t)32 << 20;
  return r;
}

int launch_polyakov_rows(const Geom &g, int nc, bool singlet, const double2 *lines, int D,
                         const PolyakovRows &r, int dz0, int ndz, double *partials,
                         double *out_dev, cudaStream_t s) {
  // (the traces' plane follows the components')
  const double2 *p = singlet ? lines : lines + (size_t)(nc == 3 ? 9 : 2) * g.Vs;
  const dim3 grid(r.row_tiles, ndz * r.nch, r.ndxt);
  auto go = [&](auto np, auto dxt) {
    constexpr int NP = decltype(np)::value, DXT = decltype(dxt)::value;
    const size_t smem = rows_smem(g, NP, DXT);
    const int rc = allow_large_smem(polyakov_rows_kernel<NP, DXT>, smem);
    if (!rc)
      launch_chained(polyakov_rows_kernel<NP, DXT>, grid, NP * kRowsDy * rows_groups(NP), smem, s,
                     g, p, D, dz0, r.nch, partials);
    return rc;
  };
  using std::integral_constant;
  auto tiles = [&](auto np) {
    switch (r.dxt) {
    case 1: return go(np, integral_constant<int, 1>());
    case 2: return go(np, integral_constant<int, 2>());
    case 3: return go(np, integral_constant<int, 3>());
    case 4: return go(np, integral_constant<int, 4>());
    case 5: return go(np, integral_constant<int, 5>());
    case 6: return go(np, integral_constant<int, 6>());
    case 7: return go(np, integral_constant<int, 7>());
    case 8: return go(np, integral_constant<int, 8>());
    default: return go(np, integral_constant<int, 9>());
    }
  };
  int rc = singlet ? (nc == 3 ? tiles(integral_constant<int, 9>())
                              : tiles(integral_constant<int, 2>()))
                   : tiles(integral_constant<int, 1>());
  if (!rc)
    rc = launch_check("polyakov_rows_kernel");
  if (rc)
    return rc;
  const double scale = 1.0 / ((double)g.Vs * (singlet && nc == 3 ? 3.0 : 1.0));
  return launch_reduce_rows(partials, r.row_tiles, ndz * r.entries, scale, out_dev, s);
}

#define GC_INSTANTIATE_P(STORE, CT)                                                      \
  template int launch_polyakov_lines<STORE, CT>(const Geom &, const Fields4 &, double2 *, \
                                                double *, double *, cudaStream_t);

GC_INSTANTIATE_P(StoreF64SU3, double)
GC_INSTANTIATE_P(StoreF64SU2, double)
GC_INSTANTIATE_P(StoreF32SU3, float)
GC_INSTANTIATE_P(StoreF32SU2, float)

} // namespace gc
