// Group algebra for SU(2) (quaternion a0 + i a.sigma) and SU(3) (3x3 complex),
// usable on host and device, templated on the arithmetic type (double/float).
//
// Semantics follow the reference's matrix types (lib/cpu/include/matrix.h):
//   mul(A,B)      = A*B        su2 :93-98,  su3 :348-350
//   mul_ad(A,B)   = A*B^dag    ("A ^ B")  su2 :99-104,  su3 :352-354
//   mul_da(A,B)   = A^dag*B    ("A % B")  su2 :105-110, su3 :356-358
//   conj_tr(A,B)  = Re Tr(A B^dag)/N  ("multiply_conj_tr") su2 :54-56, su3 :260-262
//   proj(A)       su2 :74-77 (a/|a|); su3 :279-292 (6 x [Newton-Schulz step,
//                 determinant phase fix])
// The quaternion product formulas and the projection iteration are the
// algebra itself and therefore have the same form as the reference's.
#pragma once

#include <cmath>

#if defined(__CUDACC__)
#define GC_HD __host__ __device__ __forceinline__
#else
#define GC_HD inline
#endif

// Fused multiply-add on the device; a*b+c on the host (the host generator is
// built without FMA instructions, where fma() would be a slow library call).
#if defined(__CUDA_ARCH__)
#define GC_FMA(a, b, c) fma((a), (b), (c))
#else
#define GC_FMA(a, b, c) ((a) * (b) + (c))
#endif

namespace gc {

template <class T> struct cx {
  T re, im;
};

// Every product-sum below is an explicit fused multiply-add chain: left to
// the compiler, `a*b + c*d` may be contracted into either fma(a, b, c*d) or
// fma(c, d, a*b) depending on the surrounding code, so the same function
// inlined into two kernels could round differently. Written out, one
// function rounds one way everywhere (the batch, serving and single-lattice
// paths give bitwise equal results).
template <class T> GC_HD cx<T> cmul(cx<T> a, cx<T> b) {
  return {GC_FMA(-a.im, b.im, a.re * b.re), GC_FMA(a.im, b.re, a.re * b.im)};
}
// conj(a) * b
template <class T> GC_HD cx<T> cmulc(cx<T> a, cx<T> b) {
  return {GC_FMA(a.im, b.im, a.re * b.re), GC_FMA(-a.im, b.re, a.re * b.im)};
}
// a * conj(b)
template <class T> GC_HD cx<T> cmul_c(cx<T> a, cx<T> b) {
  return {GC_FMA(a.im, b.im, a.re * b.re), GC_FMA(-a.re, b.im, a.im * b.re)};
}
template <class T> GC_HD cx<T> cadd(cx<T> a, cx<T> b) {
  return {a.re + b.re, a.im + b.im};
}
template <class T> GC_HD cx<T> csub(cx<T> a, cx<T> b) {
  return {a.re - b.re, a.im - b.im};
}

// ----------------------------------------------------------------- SU(2)
template <class T> struct SU2 {
  T a0, a1, a2, a3;
  static constexpr int N = 2;
};

template <class T> GC_HD SU2<T> unit(SU2<T>) { return {T(1), T(0), T(0), T(0)}; }

// sum of four products p0 + s1 p1 + s2 p2 + s3 p3 as one fused chain
template <class T> GC_HD T dot4(T x0, T y0, T x1, T y1, T x2, T y2, T x3, T y3) {
  return GC_FMA(x3, y3, GC_FMA(x2, y2, GC_FMA(x1, y1, x0 * y0)));
}
template <class T> GC_HD SU2<T> mul(const SU2<T> &A, const SU2<T> &B) {
  return {dot4(A.a0, B.a0, -A.a1, B.a1, -A.a2, B.a2, -A.a3, B.a3),
          dot4(A.a0, B.a1, B.a0, A.a1, A.a3, B.a2, -A.a2, B.a3),
          dot4(A.a0, B.a2, B.a0, A.a2, A.a1, B.a3, -A.a3, B.a1),
          dot4(A.a0, B.a3, B.a0, A.a3, A.a2, B.a1, -A.a1, B.a2)};
}
template <class T> GC_HD SU2<T> mul_ad(const SU2<T> &A, const SU2<T> &B) {
  return {dot4(A.a0, B.a0, A.a1, B.a1, A.a2, B.a2, A.a3, B.a3),
          dot4(-A.a0, B.a1, B.a0, A.a1, -A.a3, B.a2, A.a2, B.a3),
          dot4(-A.a0, B.a2, B.a0, A.a2, -A.a1, B.a3, A.a3, B.a1),
          dot4(-A.a0, B.a3, B.a0, A.a3, -A.a2, B.a1, A.a1, B.a2)};
}
template <class T> GC_HD SU2<T> mul_da(const SU2<T> &A, const SU2<T> &B) {
  return {dot4(A.a0, B.a0, A.a1, B.a1, A.a2, B.a2, A.a3, B.a3),
          dot4(A.a0, B.a1, -B.a0, A.a1, -A.a3, B.a2, A.a2, B.a3),
          dot4(A.a0, B.a2, -B.a0, A.a2, -A.a1, B.a3, A.a3, B.a1),
          dot4(A.a0, B.a3, -B.a0, A.a3, -A.a2, B.a1, A.a1, B.a2)};
}
template <class T> GC_HD SU2<T> scale(const SU2<T> &A, T s) {
  return {A.a0 * s, A.a1 * s, A.a2 * s, A.a3 * s};
}
template <class T> GC_HD SU2<T> add(const SU2<T> &A, const SU2<T> &B) {
  return {A.a0 + B.a0, A.a1 + B.a1, A.a2 + B.a2, A.a3 + B.a3};
}
template <class T> GC_HD T conj_tr(const SU2<T> &A, const SU2<T> &B) {
  return dot4(A.a0, B.a0, A.a1, B.a1, A.a2, B.a2, A.a3, B.a3);
}
template <class T> GC_HD T tr_real(const SU2<T> &A) { return A.a0; }
template <class T> GC_HD SU2<T> adjoint(const SU2<T> &A) {
  return {A.a0, -A.a1, -A.a2, -A.a3};
}
// a / |a| by four divisions, as the reference writes it (the seeded
// configuration generator keeps this form, so that its links stay bit for
// bit those of the committed fixtures).
template <class T> GC_HD SU2<T> proj_div(const SU2<T> &A) {
  const T rho = sqrt(dot4(A.a0, A.a0, A.a1, A.a1, A.a2, A.a2, A.a3, A.a3));
  return {A.a0 / rho, A.a1 / rho, A.a2 / rho, A.a3 / rho};
}
// a / |a| as a times one reciprocal (four divisions cost more than the
// link's loads in FP64: SU(2) APE at 48^4 0.365 -> 0.311 ms per step; each
// element within an ulp of the quotient).
template <class T> GC_HD SU2<T> proj(const SU2<T> &A) {
  const T inv = T(1) / sqrt(dot4(A.a0, A.a0, A.a1, A.a1, A.a2, A.a2, A.a3, A.a3));
  return {A.a0 * inv, A.a1 * inv, A.a2 * inv, A.a3 * inv};
}

// ----------------------------------------------------------------- SU(3)
// Row-major: e[i][j] is the element in row i, column j.
template <class T> struct SU3 {
  cx<T> e[3][3];
  static constexpr int N = 3;
};

template <class T> GC_HD SU3<T> unit(SU3<T>) {
  SU3<T> U;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      U.e[i][j] = {i == j ? T(1) : T(0), T(0)};
  return U;
}

// The complex multiply-accumulates below are written as explicit fused
// multiply-add chains (one rounding per term instead of a product and an add).
// This is a different but equally accurate rounding order from the
// reference's separate product and sum.
template <class T> GC_HD SU3<T> mul(const SU3<T> &A, const SU3<T> &B) {
  SU3<T> C;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      T re = A.e[i][0].re * B.e[0][j].re;
      T im = A.e[i][0].re * B.e[0][j].im;
      re = GC_FMA(-A.e[i][0].im, B.e[0][j].im, re);
      im = GC_FMA(A.e[i][0].im, B.e[0][j].re, im);
#pragma unroll
      for (int k = 1; k < 3; k++) {
        re = GC_FMA(A.e[i][k].re, B.e[k][j].re, re);
        re = GC_FMA(-A.e[i][k].im, B.e[k][j].im, re);
        im = GC_FMA(A.e[i][k].re, B.e[k][j].im, im);
        im = GC_FMA(A.e[i][k].im, B.e[k][j].re, im);
      }
      C.e[i][j] = {re, im};
    }
  return C;
}
// A * B^dag : C_ij = sum_k A_ik conj(B_jk)
template <class T> GC_HD SU3<T> mul_ad(const SU3<T> &A, const SU3<T> &B) {
  SU3<T> C;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      T re = A.e[i][0].re * B.e[j][0].re;
      T im = A.e[i][0].im * B.e[j][0].re;
      re = GC_FMA(A.e[i][0].im, B.e[j][0].im, re);
      im = GC_FMA(-A.e[i][0].re, B.e[j][0].im, im);
#pragma unroll
      for (int k = 1; k < 3; k++) {
        re = GC_FMA(A.e[i][k].re, B.e[j][k].re, re);
        re = GC_FMA(A.e[i][k].im, B.e[j][k].im, re);
        im = GC_FMA(A.e[i][k].im, B.e[j][k].re, im);
        im = GC_FMA(-A.e[i][k].re, B.e[j][k].im, im);
      }
      C.e[i][j] = {re, im};
    }
  return C;
}
// A^dag * B : C_ij = sum_k conj(A_ki) B_kj
template <class T> GC_HD SU3<T> mul_da(const SU3<T> &A, const SU3<T> &B) {
  SU3<T> C;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      T re = A.e[0][i].re * B.e[0][j].re;
      T im = A.e[0][i].re * B.e[0][j].im;
      re = GC_FMA(A.e[0][i].im, B.e[0][j].im, re);
      im = GC_FMA(-A.e[0][i].im, B.e[0][j].re, im);
#pragma unroll
      for (int k = 1; k < 3; k++) {
        re = GC_FMA(A.e[k][i].re, B.e[k][j].re, re);
        re = GC_FMA(A.e[k][i].im, B.e[k][j].im, re);
        im = GC_FMA(A.e[k][i].re, B.e[k][j].im, im);
        im = GC_FMA(-A.e[k][i].im, B.e[k][j].re, im);
      }
      C.e[i][j] = {re, im};
    }
  return C;
}
template <class T> GC_HD SU3<T> scale(const SU3<T> &A, T s) {
  SU3<T> C;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      C.e[i][j] = {A.e[i][j].re * s, A.e[i][j].im * s};
  return C;
}
template <class T> GC_HD SU3<T> add(const SU3<T> &A, const SU3<T> &B) {
  SU3<T> C;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      C.e[i][j] = cadd(A.e[i][j], B.e[i][j]);
  return C;
}
template <class T> GC_HD SU3<T> adjoint(const SU3<T> &A) {
  SU3<T> C;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      C.e[i][j] = {A.e[j][i].re, -A.e[j][i].im};
  return C;
}
// Re Tr(A B^dag) / 3
template <class T> GC_HD T conj_tr(const SU3<T> &A, const SU3<T> &B) {
  T s = T(0);
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      s = GC_FMA(A.e[i][j].im, B.e[i][j].im, GC_FMA(A.e[i][j].re, B.e[i][j].re, s));
  return s / T(3);
}
template <class T> GC_HD T tr_real(const SU3<T> &A) {
  return (A.e[0][0].re + A.e[1][1].re + A.e[2][2].re) / T(3);
}
// a*b - c*d for complex numbers, as fused chains
template <class T> GC_HD cx<T> cmul_sub(cx<T> a, cx<T> b, cx<T> c, cx<T> d) {
  T re = a.re * b.re;
  T im = a.re * b.im;
  re = GC_FMA(-a.im, b.im, re);
  im = GC_FMA(a.im, b.re, im);
  re = GC_FMA(-c.re, d.re, re);
  re = GC_FMA(c.im, d.im, re);
  im = GC_FMA(-c.re, d.im, im);
  im = GC_FMA(-c.im, d.re, im);
  return {re, im};
}
// conj(a*b - c*d), as fused chains: an element of conj(row x row), the third
// row of an SU(3) matrix from its first two
template <class T> GC_HD cx<T> cross_conj(cx<T> a, cx<T> b, cx<T> c, cx<T> d) {
  T re = a.re * b.re;
  T im = c.re * d.im;
  re = GC_FMA(-a.im, b.im, re);
  im = GC_FMA(c.im, d.re, im);
  re = GC_FMA(-c.re, d.re, re);
  im = GC_FMA(-a.re, b.im, im);
  re = GC_FMA(c.im, d.im, re);
  im = GC_FMA(-a.im, b.re, im);
  return {re, im};
}
// acc + a*b (complex)
template <class T> GC_HD cx<T> cmadd(cx<T> acc, cx<T> a, cx<T> b) {
  T re = GC_FMA(a.re, b.re, acc.re);
  T im = GC_FMA(a.re, b.im, acc.im);
  re = GC_FMA(-a.im, b.im, re);
  im = GC_FMA(a.im, b.re, im);
  return {re, im};
}
template <class T> GC_HD cx<T> det(const SU3<T> &m) {
  // cofactor expansion along the first column
  cx<T> c0 = cmul_sub(m.e[1][1], m.e[2][2], m.e[2][1], m.e[1][2]);
  cx<T> c1 = cmul_sub(m.e[0][1], m.e[2][2], m.e[2][1], m.e[0][2]);
  cx<T> c2 = cmul_sub(m.e[0][1], m.e[1][2], m.e[1][1], m.e[0][2]);
  cx<T> d = cmul(m.e[0][0], c0);
  d = cmadd(d, {-m.e[1][0].re, -m.e[1][0].im}, c1);
  d = cmadd(d, m.e[2][0], c2);
  return d;
}

// One Newton-Schulz step toward the unitary polar factor,
// A <- 3/2 A - 1/2 (A A^dag) A, followed by the determinant phase fix
// A <- (1 - (det A - 1)/3) A.  H = A A^dag is Hermitian: its upper triangle
// is computed and mirrored. The factor -1/2 is folded into H (exact: a power
// of two), so B = 3/2 A + (-H/2) A is one fused chain per element.
// H = -1/2 A A^dag (Hermitian; entries below the diagonal mirrored).
template <class T> GC_HD void ns_gram(const SU3<T> &A, cx<T> H[3][3]) {
#pragma unroll
  for (int i = 0; i < 3; i++) {
    T d = A.e[i][0].re * A.e[i][0].re;
    d = GC_FMA(A.e[i][0].im, A.e[i][0].im, d);
    d = GC_FMA(A.e[i][1].re, A.e[i][1].re, d);
    d = GC_FMA(A.e[i][1].im, A.e[i][1].im, d);
    d = GC_FMA(A.e[i][2].re, A.e[i][2].re, d);
    d = GC_FMA(A.e[i][2].im, A.e[i][2].im, d);
    H[i][i] = {T(-0.5) * d, T(0)};
#pragma unroll
    for (int j = i + 1; j < 3; j++) {
      T re = A.e[i][0].re * A.e[j][0].re;
      T im = A.e[i][0].im * A.e[j][0].re;
      re = GC_FMA(A.e[i][0].im, A.e[j][0].im, re);
      im = GC_FMA(-A.e[i][0].re, A.e[j][0].im, im);
#pragma unroll
      for (int k = 1; k < 3; k++) {
        re = GC_FMA(A.e[i][k].re, A.e[j][k].re, re);
        re = GC_FMA(A.e[i][k].im, A.e[j][k].im, re);
        im = GC_FMA(A.e[i][k].im, A.e[j][k].re, im);
        im = GC_FMA(-A.e[i][k].re, A.e[j][k].im, im);
      }
      H[i][j] = {T(-0.5) * re, T(-0.5) * im};
      H[j][i] = {T(-0.5) * re, T(0.5) * im};
    }
  }
}

// B = 3/2 A + H A with H from ns_gram, then the determinant phase fix.
template <class T> GC_HD SU3<T> ns_finish(const SU3<T> &A, const cx<T> H[3][3]) {
  SU3<T> B;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      cx<T> s = {T(1.5) * A.e[i][j].re, T(1.5) * A.e[i][j].im};
#pragma unroll
      for (int k = 0; k < 3; k++) {
        if (i == k) { // H_ii is real
          s.re = GC_FMA(H[i][i].re, A.e[k][j].re, s.re);
          s.im = GC_FMA(H[i][i].re, A.e[k][j].im, s.im);
        } else {
          s = cmadd(s, H[i][k], A.e[k][j]);
        }
      }
      B.e[i][j] = s;
    }
  cx<T> dt = det(B);
  const T third = T(1) / T(3);
  cx<T> c = {GC_FMA(-third, dt.re - T(1), T(1)), -third * dt.im};
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++)
      B.e[i][j] = cmul(c, B.e[i][j]);
  return B;
}

// One polar step without the determinant, 3/2 A - 1/2 A A^dag A: a matrix
// with unitarity defect d becomes unitary to O(d^2), its phase unchanged.
template <class T> GC_HD SU3<T> polar_step(const SU3<T> &A) {
  cx<T> H[3][3];
  ns_gram(A, H);
  SU3<T> B;
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int j = 0; j < 3; j++) {
      // A + (1/2 - A A^dag / 2) A: the small part is added last
      const T h = H[i][i].re + T(0.5);
      cx<T> s = {h * A.e[i][j].re, h * A.e[i][j].im};
#pragma unroll
      for (int k = 0; k < 3; k++)
        if (i != k)
          s = cmadd(s, H[i][k], A.e[k][j]);
      B.e[i][j] = cadd(A.e[i][j], s);
    }
  return B;
}
template <class T> GC_HD SU3<T> ns_step(const SU3<T> &A) {
  cx<T> H[3][3];
  ns_gram(A, H);
  return ns_finish(A, H);
}

template <class T> GC_HD SU3<T> proj(const SU3<T> &A) {
  SU3<T> B = ns_step(A);
#pragma unroll 1
  for (int it = 0; it < 5; it++)
    B = ns_step(B);
  return B;
}

// The same six-step iteration, leaving early once a step changes no element
// by more than tol. The iteration converges quadratically (the error after a
// step of size d is O(d^2)), so the remaining steps would change the result
// by O(tol^2) plus rounding; an input that needs all six steps gets all six.
// The first two steps are always taken (inputs of smearing steps are never
// converged that early), so the check runs only after steps 3, 4 and 5.
template <class T> GC_HD SU3<T> proj(const SU3<T> &A, T tol) {
  SU3<T> B = ns_step(ns_step(A));
#pragma unroll 1
  for (int it = 0; it < 4; it++) {
    SU3<T> N = ns_step(B);
    if (it == 3) { // the sixth and last step
      B = N;
      break;
    }
    T d = T(0);
#pragma unroll
    for (int i = 0; i < 3; i++)
#pragma unroll
      for (int j = 0; j < 3; j++) {
        d = fmax(d, fabs(N.e[i][j].re - B.e[i][j].re));
        d = fmax(d, fabs(N.e[i][j].im - B.e[i][j].im));
      }
    B = N;
    if (d <= tol)
      break;
  }
  return B;
}
template <class T> GC_HD SU2<T> proj(const SU2<T> &A, T) { return proj(A); }

// ---- SU(3) projection in the algebra generated by A^dag A
//
// The projection's limit is U = z A (A^dag A)^(-1/2) with z the cube root of
// 1/phase(det A). A Newton-Schulz step on the matrix costs about 250
// multiply-adds with its determinant; here the inverse square root is found
// as a polynomial instead. With m = tr(A^dag A)/3 and the traceless
// E = 1 - A^dag A / m, Cayley-Hamilton gives E^3 = q E + d (q = tr E^2 / 2,
// d = det E), so every power series in E is x0 + x1 E + x2 E^2: the series of
// (1 - E)^(-1/2) through E^5 starts it and each Newton step
// x += x r / 2, r = 1 - (1 - E) x^2, acts on three scalars (about 30
// multiply-adds). det(1 - E) = 1 - q - d gives |det A|, and z follows from
// three-term Newton steps on a complex number. About 340 multiply-adds plus
// 30 per Newton step, against 250 per step of the matrix iteration (three to
// six of them).
//
// The reference takes exactly six matrix steps, which reach the limit only
// for sums not too far from a multiple of an SU(3) matrix. The steps act on
// the three singular values and the determinant's phase alone, so where they
// converge is a property of four numbers, and polar_parts (U = z Y) answers
// (returns true) only inside a region where the six steps end within 1e-14 of the
// limit: 0.25 <= m <= 1.001, p m >= 0.24 with p = det(1 - E), and a phase
// below 0.7 (checked over 30 million singular values and phases up to the
// region's edge: 4e-15). Inside it the polynomial's own loops may not converge
// either: where one singular value is 1.52 to 1.535 times the rms and the others
// are equal, E reaches -1.36, the series starts near its zero at -1.366, and
// eight Newton steps (a factor 1.5 each from there) do not reach the root. A
// loop that ends at its cap answers false as well (3 million matrices with a
// singular value from 1 to 1.535 times the rms: 2.3e-15 in FP64, 1.4e-6 in
// FP32; at the cap the error was 0.45). Sums of SU(3) matrices with weights that
// add to one have m <= 1; of HYP's level-1 sums at plaquette 0.6 less than 1% lie outside,
// of APE sums none (of sums of random matrices 82% and 74%). Elsewhere the result
// is not set and the caller takes the reference's steps.
GC_HD double gc_rsqrt(double x) {
#if defined(__CUDA_ARCH__)
  return rsqrt(x);
#else
  return 1.0 / sqrt(x);
#endif
}
GC_HD float gc_rsqrt(float x) {
#if defined(__CUDA_ARCH__)
  return rsqrtf(x);
#else
  return 1.0f / sqrtf(x);
#endif
}
// Newton steps stop once the residual is below `value`: the step taken from
// there leaves 3/8 r^2 (inverse square root) or 2/9 r^2 (cube root). None is
// taken where the starting series is exact to rounding: q = |E|^2 / 2 below
// `series`, |w - 1| below `cube`.
template <class T> struct PolarTol;
template <> struct PolarTol<double> {
  static constexpr double value = 1e-8, series = 2e-6, cube = 5e-6;
};
template <> struct PolarTol<float> {
  static constexpr float value = 2e-4f, series = 2e-3f, cube = 4e-3f;
};

template <class T> GC_HD bool polar_parts(const SU3<T> &A, SU3<T> &Y, cx<T> &z) {
  // H = A^dag A: diagonal h, off-diagonal (0,1), (0,2), (1,2)
  T h[3];
  cx<T> o[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    T s = A.e[0][j].re * A.e[0][j].re;
    s = GC_FMA(A.e[0][j].im, A.e[0][j].im, s);
#pragma unroll
    for (int k = 1; k < 3; k++) {
      s = GC_FMA(A.e[k][j].re, A.e[k][j].re, s);
      s = GC_FMA(A.e[k][j].im, A.e[k][j].im, s);
    }
    h[j] = s;
  }
#pragma unroll
  for (int p = 0; p < 3; p++) {
    const int i = p == 2 ? 1 : 0, j = p == 0 ? 1 : 2;
    T re = A.e[0][i].re * A.e[0][j].re;
    T im = A.e[0][i].re * A.e[0][j].im;
    re = GC_FMA(A.e[0][i].im, A.e[0][j].im, re);
    im = GC_FMA(-A.e[0][i].im, A.e[0][j].re, im);
#pragma unroll
    for (int k = 1; k < 3; k++) {
      re = GC_FMA(A.e[k][i].re, A.e[k][j].re, re);
      re = GC_FMA(A.e[k][i].im, A.e[k][j].im, re);
      im = GC_FMA(A.e[k][i].re, A.e[k][j].im, im);
      im = GC_FMA(-A.e[k][i].im, A.e[k][j].re, im);
    }
    o[p] = {re, im};
  }
  const T m = ((h[0] + h[1]) + h[2]) * (T(1) / T(3));
  const T rs = gc_rsqrt(m), im = rs * rs;
  // E = 1 - H / m and F = E^2
  const T e0 = GC_FMA(-im, h[0], T(1)), e1 = GC_FMA(-im, h[1], T(1)),
          e2 = GC_FMA(-im, h[2], T(1));
  const cx<T> a = {-im * o[0].re, -im * o[0].im}, b = {-im * o[1].re, -im * o[1].im},
              c = {-im * o[2].re, -im * o[2].im};
  const T aa = GC_FMA(a.im, a.im, a.re * a.re), bb = GC_FMA(b.im, b.im, b.re * b.re),
          cc = GC_FMA(c.im, c.im, c.re * c.re);
  const T f0 = GC_FMA(e0, e0, aa + bb), f1 = GC_FMA(e1, e1, aa + cc),
          f2 = GC_FMA(e2, e2, bb + cc);
  const T q = T(0.5) * ((f0 + f1) + f2);
  // det E = e0 e1 e2 + 2 Re(a c conj(b)) - e0 |c|^2 - e1 |b|^2 - e2 |a|^2
  const cx<T> ac = cmul(a, c);
  T d = GC_FMA(e0, e1, -aa) * e2;
  d = GC_FMA(-e0, cc, d);
  d = GC_FMA(-e1, bb, d);
  d = GC_FMA(T(2) * ac.re, b.re, d);
  d = GC_FMA(T(2) * ac.im, b.im, d);
  const cx<T> D = det(A);
  // the region of the comment above (false for NaN and infinities)
  const T p = (T(1) - q) - d;
  if (!(m >= T(0.25) && m <= T(1.001) && p * m >= T(0.24) && fabs(D.im) <= T(0.84) * D.re))
    return false;
  // (1 - E)^(-1/2): 1 + E/2 + 3/8 E^2 + 5/16 E^3 + 35/128 E^4 + 63/256 E^5
  const T c5 = T(63.0 / 256.0);
  T x0 = GC_FMA(GC_FMA(c5, q, T(0.3125)), d, T(1));
  T x1 = GC_FMA(T(35.0 / 128.0), d, GC_FMA(GC_FMA(c5, q, T(0.3125)), q, T(0.5)));
  T x2 = GC_FMA(c5, d, GC_FMA(T(35.0 / 128.0), q, T(0.375)));
  // (the series' error is 0.23 |E|^6: below T's rounding it needs no step)
  T rn = T(0);
#pragma unroll 1
  for (int it = 0; it < 8 && q > PolarTol<T>::series; it++) {
    // s = x^2, r = 1 - s + E s
    const T z3 = T(2) * (x1 * x2), z4 = x2 * x2;
    const T s0 = GC_FMA(d, z3, x0 * x0);
    const T s1 = GC_FMA(d, z4, GC_FMA(q, z3, T(2) * (x0 * x1)));
    const T s2 = GC_FMA(q, z4, GC_FMA(x1, x1, T(2) * (x0 * x2)));
    const T r0 = GC_FMA(d, s2, T(1) - s0);
    const T r1 = GC_FMA(q, s2, s0 - s1);
    const T r2 = s1 - s2;
    rn = fabs(r0) + (fabs(r1) + fabs(r2));
    // x += x r / 2
    const T p3 = GC_FMA(x1, r2, x2 * r1), p4 = x2 * r2;
    const T p0 = GC_FMA(d, p3, x0 * r0);
    const T p1 = GC_FMA(d, p4, GC_FMA(q, p3, GC_FMA(x0, r1, x1 * r0)));
    const T p2 = GC_FMA(q, p4, GC_FMA(x0, r2, GC_FMA(x1, r1, x2 * r0)));
    x0 = GC_FMA(T(0.5), p0, x0);
    x1 = GC_FMA(T(0.5), p1, x1);
    x2 = GC_FMA(T(0.5), p2, x2);
    if (!(rn > PolarTol<T>::value))
      break;
  }
  // z: z^3 w = 1 with w = det A / |det A|, |det A|^2 = m^3 (1 - q - d)
  const T wn = (rs * im) * gc_rsqrt(p);
  const cx<T> w = {D.re * wn, D.im * wn};
  const cx<T> w1 = {GC_FMA(D.re, wn, T(-1)), w.im};
  // (1 + t)^(-1/3) = 1 - t/3 + 2/9 t^2
  const cx<T> t = {GC_FMA(T(2.0 / 9.0), w1.re, T(-1.0 / 3.0)), T(2.0 / 9.0) * w1.im};
  z = cmul(t, w1);
  z.re += T(1);
  // (error 0.17 |w1|^3)
  T gn = T(0);
#pragma unroll 1
  for (int it = 0; it < 8 && fabs(w1.re) + fabs(w1.im) > PolarTol<T>::cube; it++) {
    const cx<T> r = cmul(cmul(cmul(z, z), z), w);
    const cx<T> g = {T(1) - r.re, -r.im}; // 1 - z^3 w
    const cx<T> u = {GC_FMA(T(1.0 / 3.0), g.re, T(1)), T(1.0 / 3.0) * g.im};
    z = cmul(z, u);
    gn = fabs(g.re) + fabs(g.im);
    if (!(gn > PolarTol<T>::value))
      break;
  }
  // a loop ended at its cap (see above)
  if (rn > PolarTol<T>::value || gn > PolarTol<T>::value)
    return false;
  // X = rs (x0 + x1 E + x2 F); F off the diagonal: -e2 a + b conj(c),
  // -e1 b + a c, -e0 c + conj(a) b. FP32: the factor rs x0 goes to z, so that
  // polar_finish (FP64) multiplies Y by a number that is not 1. With z = 1 on a
  // smooth field U would be Y, on the grid of FP32, where an update below half a
  // rounding has no effect, and the common error of Y's scalars would stay in
  // every link (mean of U U^dag - 1 after 20 APE steps 1e-9, against 5e-11).
  if constexpr (sizeof(T) == 4) {
    const T ix = T(1) / x0, scale = rs * x0;
    x0 = T(1);
    x1 *= ix;
    x2 *= ix;
    z.re *= scale;
    z.im *= scale;
  } else {
    x0 *= rs;
    x1 *= rs;
    x2 *= rs;
  }
  const cx<T> bc = cmul_c(b, c), ab = cmulc(a, b);
  const T X0 = GC_FMA(x2, f0, GC_FMA(x1, e0, x0)), X1 = GC_FMA(x2, f1, GC_FMA(x1, e1, x0)),
          X2 = GC_FMA(x2, f2, GC_FMA(x1, e2, x0));
  const T ka = GC_FMA(-x2, e2, x1), kb = GC_FMA(-x2, e1, x1), kc = GC_FMA(-x2, e0, x1);
  const cx<T> Xa = {GC_FMA(x2, bc.re, ka * a.re), GC_FMA(x2, bc.im, ka * a.im)};
  const cx<T> Xb = {GC_FMA(x2, ac.re, kb * b.re), GC_FMA(x2, ac.im, kb * b.im)};
  const cx<T> Xc = {GC_FMA(x2, ab.re, kc * c.re), GC_FMA(x2, ab.im, kc * c.im)};
#pragma unroll
  for (int i = 0; i < 3; i++) {
    // row i of A X: the small terms first, so that one product and sum is
    // rounded at full size
    const cx<T> r0 = A.e[i][0], r1 = A.e[i][1], r2 = A.e[i][2];
    const cx<T> y0 = cmadd(cmul_c(r1, Xa), r2, {Xb.re, -Xb.im});
    const cx<T> y1 = cmadd(cmul(r0, Xa), r2, {Xc.re, -Xc.im});
    const cx<T> y2 = cmadd(cmul(r0, Xb), r1, Xc);
    Y.e[i][0] = {GC_FMA(r0.re, X0, y0.re), GC_FMA(r0.im, X0, y0.im)};
    Y.e[i][1] = {GC_FMA(r1.re, X1, y1.re), GC_FMA(r1.im, X1, y1.im)};
    Y.e[i][2] = {GC_FMA(r2.re, X2, y2.re), GC_FMA(r2.im, X2, y2.im)};
  }
  return true;
}

// z y, rounded once at full size where z is nearly real
template <class T> GC_HD cx<T> cphase(cx<T> z, cx<T> y) {
  return {GC_FMA(z.re, y.re, -z.im * y.im), GC_FMA(z.re, y.im, z.im * y.re)};
}
template <class T> GC_HD bool polar_su3(const SU3<T> &A, SU3<T> &U) {
  cx<T> z;
  if (!polar_parts(A, U, z))
    return false;
#pragma unroll
  for (int k = 0; k < 9; k++)
    U.e[k / 3][k % 3] = cphase(z, U.e[k / 3][k % 3]);
  return true;
}

// Newton-Schulz steps from B while its unitarity defect max|A A^dag - 1|
// (read off the step's own Gram matrix) exceeds tol, at most max_steps of
// them; *steps receives the number taken. The mixed-precision projection
// takes these in FP32 and then one step in FP64 (ns_step<double>): a step
// maps a defect d to O(d^2) (A = U(1 + E) becomes U(1 - 3/2 E^2 + ...),
// d = 2|E|), so from d <= 2e-5 the FP64 step lands below 1e-9, under the
// FP32 rounding of the stored link, and removes the FP32 rounding of the
// iterate. Together at most six steps, like the reference's projection.
template <class T> GC_HD SU3<T> ns_until(SU3<T> B, T tol, int max_steps, int *steps) {
  int n = 0;
#pragma unroll 1
  while (n < max_steps) {
    cx<T> H[3][3];
    ns_gram(B, H);
    // A A^dag = -2 H
    T d = T(0);
#pragma unroll
    for (int i = 0; i < 3; i++) {
      d = fmax(d, fabs(T(-2) * H[i][i].re - T(1)));
#pragma unroll
      for (int j = i + 1; j < 3; j++)
        d = fmax(d, fmax(fabs(H[i][j].re), fabs(H[i][j].im)) * T(2));
    }
    if (d <= tol)
      break;
    B = ns_finish(B, H);
    n++;
  }
  *steps = n;
  return B;
}

// The FP32 parts of polar_parts, U = z Y, made unitary with determinant 1 to FP64
// accuracy and rounded to FP32 once: with G = U U^dag and the determinant's
// phase, U += (-(G - 1)/2 - i Im(det U)/3) U to first order; the defect is a few
// 1e-7, so the second order is below 1e-12. Rows 0 and 1, and row 2 with ROW2
// (the 12-real links rebuild it).
template <bool ROW2> GC_HD SU3<float> polar_finish(const SU3<float> &Y, cx<float> z) {
  const cx<double> zd = {double(z.re), double(z.im)};
  SU3<double> U;
#pragma unroll
  for (int k = 0; k < 9; k++)
    U.e[k / 3][k % 3] = cphase(zd, {double(Y.e[k / 3][k % 3].re), double(Y.e[k / 3][k % 3].im)});
  cx<double> c[3][3];
#pragma unroll
  for (int i = 0; i < 3; i++)
#pragma unroll
    for (int k = i; k < 3; k++) {
      if (i == 2 && !ROW2)
        continue;
      double re = i == k ? GC_FMA(U.e[i][0].re, U.e[k][0].re, -1.0) : U.e[i][0].re * U.e[k][0].re;
      re = GC_FMA(U.e[i][0].im, U.e[k][0].im, re);
#pragma unroll
      for (int j = 1; j < 3; j++) {
        re = GC_FMA(U.e[i][j].re, U.e[k][j].re, re);
        re = GC_FMA(U.e[i][j].im, U.e[k][j].im, re);
      }
      if (i == k) {
        c[i][i] = {-0.5 * re, 0.0};
        continue;
      }
      double im = U.e[i][0].im * U.e[k][0].re;
      im = GC_FMA(-U.e[i][0].re, U.e[k][0].im, im);
#pragma unroll
      for (int j = 1; j < 3; j++) {
        im = GC_FMA(U.e[i][j].im, U.e[k][j].re, im);
        im = GC_FMA(-U.e[i][j].re, U.e[k][j].im, im);
      }
      c[i][k] = {-0.5 * re, -0.5 * im};
      c[k][i] = {c[i][k].re, -c[i][k].im};
    }
  // Im det = Im sum_j (row0 x row1)_j row2_j
  double di = 0.0;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const int a = (j + 1) % 3, b = (j + 2) % 3;
    const cx<double> x = cmul_sub(U.e[0][a], U.e[1][b], U.e[0][b], U.e[1][a]);
    di = GC_FMA(x.re, U.e[2][j].im, di);
    di = GC_FMA(x.im, U.e[2][j].re, di);
  }
  const double ph = di * (-1.0 / 3.0);
  SU3<float> R;
#pragma unroll
  for (int i = 0; i < (ROW2 ? 3 : 2); i++) {
    c[i][i].im = ph;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      cx<double> s = cmadd(U.e[i][j], c[i][0], U.e[0][j]);
      s = cmadd(s, c[i][1], U.e[1][j]);
      s = cmadd(s, c[i][2], U.e[2][j]);
      R.e[i][j] = {float(s.re), float(s.im)};
    }
  }
  return R;
}

// Gram-Schmidt reunitarisation: rows 0 and 1 orthonormalised, row 2 =
// conj(row0 x row1). Used by the configuration generator (not on the
// reference path).
template <class T> GC_HD SU3<T> reunitarize_gs(const SU3<T> &A) {
  SU3<T> U;
  T n0 = T(0);
  for (int j = 0; j < 3; j++)
    n0 += A.e[0][j].re * A.e[0][j].re + A.e[0][j].im * A.e[0][j].im;
  n0 = T(1) / sqrt(n0);
  for (int j = 0; j < 3; j++)
    U.e[0][j] = {A.e[0][j].re * n0, A.e[0][j].im * n0};
  // p = <u0, a1> = sum conj(u0_j) a1_j
  cx<T> p = {T(0), T(0)};
  for (int j = 0; j < 3; j++)
    p = cadd(p, cmulc(U.e[0][j], A.e[1][j]));
  cx<T> r[3];
  T n1 = T(0);
  for (int j = 0; j < 3; j++) {
    r[j] = csub(A.e[1][j], cmul(p, U.e[0][j]));
    n1 += r[j].re * r[j].re + r[j].im * r[j].im;
  }
  n1 = T(1) / sqrt(n1);
  for (int j = 0; j < 3; j++)
    U.e[1][j] = {r[j].re * n1, r[j].im * n1};
  // row2 = conj(row0 x row1)
  for (int j = 0; j < 3; j++) {
    int a = (j + 1) % 3, b = (j + 2) % 3;
    cx<T> c = csub(cmul(U.e[0][a], U.e[1][b]), cmul(U.e[0][b], U.e[1][a]));
    U.e[2][j] = {c.re, -c.im};
  }
  return U;
}

} // namespace gc
