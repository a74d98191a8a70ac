// Loops of the temporal gauge as correlations of the space lines' elements
// along time (sm_100a; used by gc_wilson_corr.cu).
//
// With the line S'(t) of a column written as K reals (18 for SU(3), 4 for a
// quaternion), Re Tr[S'(t + T) S'(t)^dag] = sum_k s_k(t) s_k(t + T), so each
// element is a sequence in t whose autocorrelation is wanted at T_min ..
// T_max. A thread takes one sequence: it slides a window of J + V elements
// along t in registers (V = 16 bytes' worth, rotated by unrolling, so that no
// element moves) and adds V starts' products for J values of T per 16-byte
// load. No shared-memory operand is read twice and no product is computed for
// a T that is not wanted (beyond rounding the range up to J).
#pragma once

#include "gc_internal.cuh"
#include "gc_rows01.cuh"

namespace gc {

namespace {

template <class CT> struct CorrVec;
template <> struct CorrVec<float> {
  static constexpr int V = 4;
  __device__ __forceinline__ static void load(const float *p, float (&e)[4]) {
    const float4 v = *reinterpret_cast<const float4 *>(p);
    e[0] = v.x;
    e[1] = v.y;
    e[2] = v.z;
    e[3] = v.w;
  }
};
template <> struct CorrVec<double> {
  static constexpr int V = 2;
  __device__ __forceinline__ static void load(const double *p, double (&e)[2]) {
    const double2 v = *reinterpret_cast<const double2 *>(p);
    e[0] = v.x;
    e[1] = v.y;
  }
};

// acc += part, two FP32 numbers per instruction (SU(3) 32^4 1900 -> 1840 us, SU(2)
// 48^4 3580 -> 3520)
template <int J> __device__ __forceinline__ void add_pairs(float (&acc)[J], const float (&part)[J]) {
#pragma unroll
  for (int j = 0; j < J; j += 2) {
    const float2 v = __fadd2_rn(make_float2(acc[j], acc[j + 1]), make_float2(part[j], part[j + 1]));
    acc[j] = v.x;
    acc[j + 1] = v.y;
  }
}
template <int J> __device__ __forceinline__ void add_pairs(double (&)[J], const double (&)[J]) {}

// acc[j] += sum_{t < tstarts} s[t] s[t + T + j], j < J (a multiple of V). s is
// 16-byte aligned, T = 1 modulo V; reads s up to the vector of index
// tstarts - 1 + T + J - 1 (finite values there). OWN (T = 1): the starts are
// the window's first vector. FP32 sums the products of eight starts (two
// vectors) at a time and adds those sums.
template <class CT, int J, bool OWN>
__device__ __forceinline__ void correlate(const CT *s, int T, int tstarts, CT (&acc)[J]) {
  using CV = CorrVec<CT>;
  constexpr int V = CV::V, N = J / V + 1;
  constexpr bool kGroups = sizeof(CT) == 4;
  static_assert(J % V == 0, "whole vectors");
  const CT *b = s + (T - 1);
  CT w[N][V];
#pragma unroll
  for (int i = 0; i < N - 1; i++)
    CV::load(b + i * V, w[i]);
  const int full = tstarts / V;
  CT part[J];
#pragma unroll 1
  for (int q = 0; q < full; q += N) {
#pragma unroll
    for (int r = 0; r < N; r++) {
      if (q + r >= full) {
        if (kGroups && r % 2 == 1)
          add_pairs(acc, part);
        break;
      }
      CV::load(b + (q + r + N - 1) * V, w[(r + N - 1) % N]);
      CT a[V];
      if (OWN) {
#pragma unroll
        for (int m = 0; m < V; m++)
          a[m] = w[r][m];
      } else {
        CV::load(s + (q + r) * V, a);
      }
#pragma unroll
      for (int m = 0; m < V; m++)
#pragma unroll
        for (int j = 0; j < J; j++) {
          const CT x = w[(r + (m + 1 + j) / V) % N][(m + 1 + j) % V];
          if (!kGroups)
            acc[j] = GC_FMA(a[m], x, acc[j]);
          else
            part[j] = r % 2 == 0 && m == 0 ? a[m] * x : GC_FMA(a[m], x, part[j]);
        }
      if (kGroups && (r % 2 == 1 || r == N - 1))
        add_pairs(acc, part);
    }
  }
  if (tstarts % V) { // the starts that do not fill a vector
    CT a[V];
    CV::load(s + full * V, a);
#pragma unroll
    for (int i = 0; i < N; i++)
      CV::load(b + (full + i) * V, w[i]);
#pragma unroll
    for (int m = 0; m < V - 1; m++)
      if (m < tstarts % V)
#pragma unroll
        for (int j = 0; j < J; j++)
          acc[j] = GC_FMA(a[m], w[(m + 1 + j) / V][(m + 1 + j) % V], acc[j]);
  }
}

// The lanes with `bit` keep the upper half of v, the others the lower half,
// each with its partner's values added.
template <int N, class T>
__device__ __forceinline__ void corr_halve(const T (&v)[N], T (&h)[N / 2], int lane, int bit) {
  const bool up = lane & bit;
#pragma unroll
  for (int j = 0; j < N / 2; j++) {
    const T keep = up ? v[j + N / 2] : v[j], give = up ? v[j] : v[j + N / 2];
    h[j] = keep + __shfl_xor_sync(0xffffffffu, give, bit);
  }
}

// Sum of acc over the warp in a fixed order, into out[0 .. J - 1] (written
// by the lanes that hold them; added to what they wrote before with `more`): two halvings in the compute type (a
// sum of four lanes' values), the other eight in FP64.
template <class CT, int J>
__device__ __forceinline__ void corr_warp_sum(const CT (&acc)[J], int lane, double *out,
                                              bool more) {
  static_assert(J % 4 == 0, "quarters");
  CT h[J / 2], q[J / 4];
  corr_halve<J>(acc, h, lane, 16);
  corr_halve<J / 2>(h, q, lane, 8);
  double d[J / 4];
#pragma unroll
  for (int j = 0; j < J / 4; j++)
    d[j] = double(q[j]);
  out += ((lane & 16) ? J / 2 : 0) + ((lane & 8) ? J / 4 : 0);
  if constexpr (J % 8 == 0) {
    double e[J / 8];
    corr_halve<J / 4>(d, e, lane, 4);
    out += (lane & 4) ? J / 8 : 0;
#pragma unroll
    for (int j = 0; j < J / 8; j++) {
      e[j] += __shfl_xor_sync(0xffffffffu, e[j], 2);
      e[j] += __shfl_xor_sync(0xffffffffu, e[j], 1);
      if ((lane & 3) == 0)
        out[j] = more ? out[j] + e[j] : e[j];
    }
  } else {
#pragma unroll
    for (int j = 0; j < J / 4; j++) {
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
        d[j] += __shfl_xor_sync(0xffffffffu, d[j], o);
      if ((lane & 7) == 0)
        out[j] = more ? out[j] + d[j] : d[j];
    }
  }
}

// Starts that the FP32 sums of one pass take, at most; FP64 adds the passes. With
// the groups of eight in correlate the FP32 sums stay short however long the
// time extent is. On links of constant phase, whose products all round alike, W
// misses the exact value by 7e-8 (rms over the phase, Lt = 48 and 240; one chain
// over all starts 2e-7 and 1.7e-6, sums of four loops in FP32 3e-8). W calls,
// one chain / this / one pass of 32 / of 16 starts, us: SU(3) 32^4 T <= 16 1755
// / 1840 / 1830 / 2015, SU(2) 48^4 T <= 24 2930 / 3520 / 3300 / 3590.
constexpr int kCorrPass = 64;

// A range of T in chunks of J: T = first + i J, i < n (first = 1 modulo V,
// first <= tmin).
struct CorrRange {
  int first, J, n;
};
__host__ __device__ inline CorrRange corr_range(int tmin, int tmax, int V, int jmax) {
  CorrRange r;
  r.first = tmin - (tmin - 1) % V;
  const int want = tmax - r.first + 1;
  r.n = (want + jmax - 1) / jmax;
  r.J = ((want + r.n - 1) / r.n + 3) / 4 * 4;
  return r;
}
// Elements of a sequence: all that correlate reads, a stride that is an odd
// number of 16-byte vectors (so that 8 sequences' vectors, and 8 columns x V
// slices of a write, cover the banks once).
__host__ __device__ inline int corr_stride(const CorrRange &r, int nslots, int tstarts, int V) {
  int n = (tstarts + V - 1) / V * V + r.first - 1 + r.n * r.J;
  n = n > nslots ? n : nslots;
  return ((n + V - 1) / V | 1) * V;
}

} // namespace

} // namespace gc
