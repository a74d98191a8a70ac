// Internal device-side types: lattice geometry, structure-of-arrays link
// storage, and the launch helpers shared by the kernels.
//
// Device layout (one "field" = one link direction, or one decorated-link
// field of HYP, or one line field): component planes, each V sites long, so
// that consecutive threads (consecutive sites) read consecutive 16-byte
// vectors.
//   FP64 SU(3): 9 planes of double2, plane k = element (k/3, k%3)   144 B/link
//   FP64 SU(2): 2 planes of double2: (a0,a1), (a2,a3)               32 B/link
//   FP32 SU(3): 3 planes of float4: (u00,u01), (u02,u10), (u11,u12); the
//               third row is rebuilt in registers as conj(row0 x row1)
//                                                                   48 B/link
//   FP32 SU(2): 1 plane of float4: (a0,a1,a2,a3)                   16 B/link
#pragma once

#include "gc_algebra.cuh"
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace gc {

struct Geom {
  int L[4];      // Lx, Ly, Lz, Lt
  int stride[4]; // 1, Lx, Lx*Ly, Lx*Ly*Lz
  int V;         // sites
  int Vs;        // spatial sites (Lx*Ly*Lz)
  unsigned inv[3]; // reciprocals of L[0..2] (set_reciprocals)
};

// floor(2^32 / L): umulhi(n, inv) is n / L or one less for every n < 2^32
// (L = 1: 2^32 - 1, the same), so that the divisions of site_coords by run-time
// extents take five instructions each instead of about 25 and three
// conversions.
inline void set_reciprocals(Geom &g) {
  for (int d = 0; d < 3; d++)
    g.inv[d] = g.L[d] > 1 ? (unsigned)((1ull << 32) / (unsigned)g.L[d]) : 0xffffffffu;
}

// n / d and n % d for 0 <= n, inv = floor(2^32 / d)
__host__ __device__ __forceinline__ int div_rem(int n, int d, unsigned inv, int *rem) {
#if defined(__CUDA_ARCH__)
  int q = (int)__umulhi((unsigned)n, inv);
#else
  int q = (int)(((unsigned long long)(unsigned)n * inv) >> 32);
#endif
  int r = n - q * d;
  if (r >= d) {
    q++;
    r -= d;
  }
  *rem = r;
  return q;
}

__host__ __device__ inline void site_coords(const Geom &g, int site, int x[4]) {
  const int r = div_rem(site, g.L[0], g.inv[0], &x[0]);
  x[3] = div_rem(div_rem(r, g.L[1], g.inv[1], &x[1]), g.L[2], g.inv[2], &x[2]);
}

// a[d] for a direction d known only at run time, as selects (a dynamically
// indexed array would be placed in local memory).
__host__ __device__ __forceinline__ int sel4(const int a[4], int d) {
  return d == 0 ? a[0] : d == 1 ? a[1] : d == 2 ? a[2] : a[3];
}

// Offset of a one-step move in direction mu (+1 or -1) from coordinate xm.
__host__ __device__ inline int step_off(const Geom &g, int xm, int mu, int dir) {
  const int L = sel4(g.L, mu), st = sel4(g.stride, mu);
  if (dir > 0)
    return (xm == L - 1) ? -(L - 1) * st : st;
  return (xm == 0) ? (L - 1) * st : -st;
}

// Offset of an n-step forward move (n >= 0, any size) from coordinate xm.
__host__ __device__ inline int fwd_off(const Geom &g, int xm, int mu, int n) {
  int xn = (xm + n) % sel4(g.L, mu);
  return (xn - xm) * sel4(g.stride, mu);
}

// ------------------------------------------------------------- storage
struct StoreF64SU3 {
  static constexpr int NC = 3;
  static constexpr int kBytes = 144;
  template <class CT> using M = SU3<CT>;
  template <class CT>
  __device__ __forceinline__ static SU3<CT> load(const void *f, size_t V,
                                                 int site) {
    const double2 *p = reinterpret_cast<const double2 *>(f) + site;
    SU3<CT> u;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      double2 v = __ldg(p + k * V);
      u.e[k / 3][k % 3] = {CT(v.x), CT(v.y)};
    }
    return u;
  }
  template <class CT>
  __device__ __forceinline__ static void store(void *f, size_t V, int site,
                                               const SU3<CT> &u) {
    double2 *p = reinterpret_cast<double2 *>(f) + site;
#pragma unroll
    for (int k = 0; k < 9; k++)
      p[k * V] = make_double2(double(u.e[k / 3][k % 3].re),
                              double(u.e[k / 3][k % 3].im));
  }
};

struct StoreF64SU2 {
  static constexpr int NC = 2;
  static constexpr int kBytes = 32;
  template <class CT> using M = SU2<CT>;
  template <class CT>
  __device__ __forceinline__ static SU2<CT> load(const void *f, size_t V,
                                                 int site) {
    const double2 *p = reinterpret_cast<const double2 *>(f) + site;
    double2 a = __ldg(p), b = __ldg(p + V);
    return {CT(a.x), CT(a.y), CT(b.x), CT(b.y)};
  }
  template <class CT>
  __device__ __forceinline__ static void store(void *f, size_t V, int site,
                                               const SU2<CT> &u) {
    double2 *p = reinterpret_cast<double2 *>(f) + site;
    p[0] = make_double2(double(u.a0), double(u.a1));
    p[V] = make_double2(double(u.a2), double(u.a3));
  }
};

struct StoreF32SU3 {
  static constexpr int NC = 3;
  static constexpr int kBytes = 48;
  template <class CT> using M = SU3<CT>;
  template <class CT>
  __device__ __forceinline__ static SU3<CT> load(const void *f, size_t V,
                                                 int site) {
    const float4 *p = reinterpret_cast<const float4 *>(f) + site;
    float4 a = __ldg(p), b = __ldg(p + V), c = __ldg(p + 2 * V);
    SU3<CT> u;
    u.e[0][0] = {CT(a.x), CT(a.y)};
    u.e[0][1] = {CT(a.z), CT(a.w)};
    u.e[0][2] = {CT(b.x), CT(b.y)};
    u.e[1][0] = {CT(b.z), CT(b.w)};
    u.e[1][1] = {CT(c.x), CT(c.y)};
    u.e[1][2] = {CT(c.z), CT(c.w)};
#pragma unroll
    for (int j = 0; j < 3; j++) {
      const int a1 = (j + 1) % 3, b1 = (j + 2) % 3;
      u.e[2][j] = cross_conj(u.e[0][a1], u.e[1][b1], u.e[0][b1], u.e[1][a1]);
    }
    return u;
  }
  template <class CT>
  __device__ __forceinline__ static void store(void *f, size_t V, int site,
                                               const SU3<CT> &u) {
    float4 *p = reinterpret_cast<float4 *>(f) + site;
    p[0] = make_float4(float(u.e[0][0].re), float(u.e[0][0].im),
                       float(u.e[0][1].re), float(u.e[0][1].im));
    p[V] = make_float4(float(u.e[0][2].re), float(u.e[0][2].im),
                       float(u.e[1][0].re), float(u.e[1][0].im));
    p[2 * V] = make_float4(float(u.e[1][1].re), float(u.e[1][1].im),
                           float(u.e[1][2].re), float(u.e[1][2].im));
  }
};

// FP32 SU(3) with all 18 reals: 9 planes of float2 (element (k/3, k%3)).
// Used for fields that may hold matrices that are not in SU(3) -- HYP's
// decorated links, whose projection (six Newton-Schulz steps, as in the
// reference) need not converge -- where rebuilding the third row would
// change the matrix.
struct StoreF32SU3Full {
  static constexpr int NC = 3;
  static constexpr int kBytes = 72;
  template <class CT> using M = SU3<CT>;
  template <class CT>
  __device__ __forceinline__ static SU3<CT> load(const void *f, size_t V,
                                                 int site) {
    const float2 *p = reinterpret_cast<const float2 *>(f) + site;
    SU3<CT> u;
#pragma unroll
    for (int k = 0; k < 9; k++) {
      float2 v = __ldg(p + k * V);
      u.e[k / 3][k % 3] = {CT(v.x), CT(v.y)};
    }
    return u;
  }
  template <class CT>
  __device__ __forceinline__ static void store(void *f, size_t V, int site,
                                               const SU3<CT> &u) {
    float2 *p = reinterpret_cast<float2 *>(f) + site;
#pragma unroll
    for (int k = 0; k < 9; k++)
      p[k * V] = make_float2(float(u.e[k / 3][k % 3].re), float(u.e[k / 3][k % 3].im));
  }
};

struct StoreF32SU2 {
  static constexpr int NC = 2;
  static constexpr int kBytes = 16;
  template <class CT> using M = SU2<CT>;
  template <class CT>
  __device__ __forceinline__ static SU2<CT> load(const void *f, size_t V,
                                                 int site) {
    float4 a = __ldg(reinterpret_cast<const float4 *>(f) + site);
    return {CT(a.x), CT(a.y), CT(a.z), CT(a.w)};
  }
  template <class CT>
  __device__ __forceinline__ static void store(void *f, size_t V, int site,
                                               const SU2<CT> &u) {
    reinterpret_cast<float4 *>(f)[site] =
        make_float4(float(u.a0), float(u.a1), float(u.a2), float(u.a3));
  }
};

// Storage of HYP's decorated-link fields for a link storage type: the same,
// except that 12-real SU(3) becomes the full 18-real form.
template <class Store> struct InterStore {
  using type = Store;
};
template <> struct InterStore<StoreF32SU3> {
  using type = StoreF32SU3Full;
};
// Bytes per link of HYP's decorated-link fields.
inline size_t inter_link_bytes(int nc, int prec) {
  if (nc == 3)
    return prec == 0 ? 144 : 72;
  return prec == 0 ? 32 : 16;
}

// Conversion between compute types (identity when equal).
template <class TO, class FROM>
__host__ __device__ __forceinline__ SU3<TO> convert(const SU3<FROM> &a, SU3<TO> *) {
  SU3<TO> b;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      b.e[i][j] = {TO(a.e[i][j].re), TO(a.e[i][j].im)};
  return b;
}
template <class TO, class FROM>
__host__ __device__ __forceinline__ SU2<TO> convert(const SU2<FROM> &a, SU2<TO> *) {
  return {TO(a.a0), TO(a.a1), TO(a.a2), TO(a.a3)};
}

// Set of per-direction field pointers passed to kernels by value.
struct Fields4 {
  void *f[4];
};

// Launch-status helper used by all host launchers.
int launch_check(const char *what);
// Records a launch-planning error (returned by the launcher as GC_ERR_ARG).
int plan_error(const char *what);

// Launches of one chain on a stream. A kernel launched by launch_chained is
// set up while the memory of the one before it drains: its blocks start when
// that kernel's have exited and wait (wait_previous, the first statement of
// every kernel launched this way) until its writes are visible. Saves about 2.4 us a
// launch (an APE step, us: SU(2) mixed 16^4 6.4 -> 3.9, SU(3) mixed 16^4 18.8 ->
// 16.1, 32^4 215 -> 212.6). Letting the next kernel start
// earlier (a trigger at the blocks' start) measured the same. Under stream
// capture the launch is an ordinary one: the batch, which captures its chains,
// puts multi-job kernels between these that do not wait this way, and such edges
// of a graph have not been measured.
__device__ __forceinline__ void wait_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
}
template <class... P, class... A>
inline void launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem,
                           cudaStream_t s, A &&...args) {
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(s, &cap);
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = cap == cudaStreamCaptureStatusNone ? 1 : 0;
  cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...); // (errors: launch_check)
}

} // namespace gc
