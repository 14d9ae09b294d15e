// Shared device-side definitions for the two-electron engine.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// One primitive pair of a shell pair (Gaussian product theorem data).
//   p = alpha_a + alpha_b, ip = 1/p, P = (alpha_a A + alpha_b B) / p,
//   Kp = sqrt(2 pi^(5/2)) c_a c_b exp(-alpha_a alpha_b / p |A-B|^2) / p
// so that the primitive-quartet prefactor 2 pi^(5/2) K_ab K_cd / (p q sqrt(p+q)) is
// Kp_ab * Kp_cd * rsqrt(p+q)  (c_a, c_b: normalised contraction coefficients).
struct __align__(16) PrimPair {
  double p, Kp, Px, Py, Pz, ip;
};

// Primitive pairs of shell pairs in blocked columns, as the class kernels read their kets: 32
// consecutive shell pairs are a block, primitive pair k of the block is a row of three
// 512-byte pieces, (p, Kp), (Px, Py), (Pz, ip) of its 32 pairs.  The lanes of a warp hold
// nearly consecutive kets, so one 16-byte load of all lanes touches 4 lines or a few more; from
// an array of PrimPair it touched 32, and the L1 wavefronts of such loads, not FP64, bounded
// the s and p classes (77 % of the LSU data pipe, 38 % of the FP64 pipe).
constexpr int kPrimRow = 96;   // double2 per row
struct PrimCols {
  const double2 *p;
};
__device__ __forceinline__ PrimCols operator+(PrimCols c, int k) { return PrimCols{c.p + kPrimRow * k}; }
__device__ __forceinline__ PrimPair prim_at(const PrimPair *c, int k) { return c[k]; }
#ifdef __CUDACC__
__device__ __forceinline__ PrimPair prim_at(PrimCols c, int k) {
  const double2 *r = c.p + kPrimRow * k;
  const double2 a = __ldg(r), b = __ldg(r + 32), d = __ldg(r + 64);
  return PrimPair{a.x, a.y, b.x, b.y, d.x, d.y};
}
#endif

// Boys function F_m(T), m = 0..L, in FP64.
//  T <  BOYS_TMAX: 8th-order Taylor expansion of F_L about the nearest tabulated point
//                 (grid step 0.1, F_{n}'(T) = -F_{n+1}(T)), then downward recursion
//                 F_m = (2T F_{m+1} + e^-T) / (2m+1).
//  T >= BOYS_TMAX: F_0 = sqrt(pi/T)/2 (erf(sqrt T) = 1 to 2e-17 there), then upward
//                 recursion F_{m+1} = ((2m+1) F_m - e^-T) / (2T); T^(-1/2) from rsqrt.
// Table layout (up to T = 52, which the rows below need): tab[i * BOYS_NORD + n] = F_n(0.1 i), i =
// 0..BOYS_NT-1, followed by
// tab[BOYS_NT * BOYS_NORD + i] = exp(-0.1 i).
#define BOYS_TMAX 36.0
#define BOYS_NT 521
#define BOYS_NORD 32
#define BOYS_NTAYLOR 8
#define BOYS_TABLE_SIZE (BOYS_NT * BOYS_NORD + BOYS_NT)

// e^x for |x| <= 0.05 from its degree-9 Taylor polynomial (remainder < 3e-20 relative).
__device__ __forceinline__ double exp_small(double x) {
  double ex = 1.0 / 362880.0;
  ex = fma(x, ex, 1.0 / 40320.0);
  ex = fma(x, ex, 1.0 / 5040.0);
  ex = fma(x, ex, 1.0 / 720.0);
  ex = fma(x, ex, 1.0 / 120.0);
  ex = fma(x, ex, 1.0 / 24.0);
  ex = fma(x, ex, 1.0 / 6.0);
  ex = fma(x, ex, 0.5);
  ex = fma(x, ex, 1.0);
  return fma(x, ex, 1.0);
}

template <int L>
__device__ __forceinline__ void boys_eval(double T, const double* __restrict__ tab, double* F) {
  if (T < BOYS_TMAX) {
    const int i = __double2int_rn(T * 10.0);
    const double x = (double)i * 0.1 - T;   // -(T - T_i)
    const double* row = tab + i * BOYS_NORD + L;
    double f = __ldg(row + BOYS_NTAYLOR);
#pragma unroll
    for (int k = BOYS_NTAYLOR; k >= 1; --k) f = __ldg(row + k - 1) + x * f * (1.0 / k);
    F[L] = f;
    if (L > 0) {
      const double e = __ldg(tab + BOYS_NT * BOYS_NORD + i) * exp_small(x);
      const double t2 = 2.0 * T;
#pragma unroll
      for (int m = L - 1; m >= 0; --m) F[m] = (t2 * F[m + 1] + e) * (1.0 / (2 * m + 1));
    }
  } else {
    // F_0 = (sqrt(pi) / 2) T^(-1/2) and 1 / (2T) from one reciprocal square root
    const double r = rsqrt(T);
    F[0] = 0.88622692545275801 * r;
    if (L > 0) {
      const double e = exp(-T);
      const double i2t = 0.5 * r * r;
#pragma unroll
      for (int m = 0; m < L; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) * i2t;
    }
  }
}

// ---- rows of the class kernels ----
// What a kernel of total angular momentum L reads per primitive quartet: Taylor coefficients
// about the points T_i = i / 8 (x = T_i - T, |x| <= 1/16), ten doubles a row, 16-byte aligned and
// read as five double2:
//   L = 1 : F_k(T_i) / k!,  k = 0..9: F_0 is the polynomial and F_1 = -dF_0/dT its derivative in x
//   else  : F_{L+k}(T_i) / k!,  k = 0..8, then e^{-T_i}; F_L is the polynomial, the lower orders
//           follow from F_m = (2T F_{m+1} + e^-T) / (2m+1) with e^-T = e^{-T_i} e^x
// (truncation below 4e-17 of F_L).  Rows 0 .. 8 boys_tmax(L) are points; one more, the far row,
// serves every larger T, where F_n = c_n T^(-n-1/2) with c_n = sqrt(pi)/2 (2n-1)!!/2^n to 3e-17:
// its "values" are the c_n (class_boys).
__host__ __device__ constexpr double boys_tmax(int L) {
  return L == 1 ? 40.0 : L == 2 ? 44.0 : L == 3 ? 47.0 : L == 4 ? 50.0 : L == 5 ? 52.0 : 36.0;
}
__host__ __device__ constexpr double boys_tfar(int L) { return boys_tmax(L) + 0.125; }
#define BOYS_SROW (BOYS_NTAYLOR + 2)
#define BOYS_MAXL 12
__host__ __device__ constexpr int boys_nrows(int L) { return 8 * (int)boys_tmax(L) + 2; }
__host__ __device__ constexpr int boys_rows_size(int L) { return boys_nrows(L) * BOYS_SROW; }
__host__ __device__ constexpr int boys_rows_off(int L) { return L == 0 ? 0 : boys_rows_off(L - 1) + boys_rows_size(L - 1); }

#ifdef __CUDACC__
// Copy the rows of L (rows_g: kBoysRows, the rows of every L one after the other, constants
// of the module written by gen_eri.py) to shared memory with 16-byte asynchronous copies.
// Every CTA of a class kernel pays this once, so it bounds the short launches: with the
// coefficients scaled in each CTA instead (up to eight divisions per entry and an exp per
// row) a 21-class build of one water in 6-31G(d) took 1.97 ms, 1.53 ms with the copy.  The
// caller synchronises the block before it reads the rows.
template <int L>
__device__ __forceinline__ void load_boys(const double *__restrict__ rows_g, double *s) {
  static_assert(L >= 0 && L <= BOYS_MAXL, "rows of this L are not in the table");
  const double *src = rows_g + boys_rows_off(L);
  for (int k = threadIdx.x; k < boys_rows_size(L) / 2; k += blockDim.x) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(s + 2 * k);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(dst), "l"(src + 2 * k) : "memory");
  }
  asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
}
#else
// The rows of L from the table, for host builds of the class code: F at T_i = i / 8 by Taylor
// expansion about the nearest table point.
template <int L>
inline void stage_boys(const double *tab, double *s) {
  static_assert(boys_rows_size(L) <= BOYS_NT * BOYS_SROW, "rows fit the table's size");
  constexpr int base = L == 1 ? 0 : L, nc = L == 1 ? 10 : BOYS_NTAYLOR + 1;
  for (int i = 0; i < boys_nrows(L); ++i) {
    double *row = s + i * BOYS_SROW;
    const bool far = i == boys_nrows(L) - 1;
    const int at = (10 * i + 4) / 8;                       // nearest point 0.1 at
    const double dx = -(double)(10 * i - 8 * at) / 80.0;   // 0.1 at - T_i
    double inv_fact = 1.0, c = 0.88622692545275801;        // sqrt(pi) / 2
    for (int k = 0; k < base; ++k) c *= 0.5 * (2 * k + 1);
    for (int k = 0; k < BOYS_SROW; ++k) {
      if (k >= 2) inv_fact /= (double)k;
      if (k >= nc) {
        row[k] = far ? 0.0 : exp(-0.125 * (double)i);
      } else if (far) {   // c_L, and for L = 1 the derivative c_1 = c_0 / 2
        row[k] = k == 0 ? c : (L == 1 && k == 1) ? 0.5 * c : 0.0;
      } else {
        double f = 0.0;
        for (int j = 8; j >= 0; --j) f = tab[at * BOYS_NORD + base + k + j] + (j < 8 ? dx * f / (j + 1) : 0.0);
        row[k] = f * inv_fact;
      }
    }
  }
}
#endif

// Row values at T (below boys_tfar): F[0..L], with t2 = 2T in the recursion.  The row index comes
// from the low word of 8 T + 1.5 2^52, whose addition rounds to the nearest integer.
template <int L>
__device__ __forceinline__ void boys_row_eval(double T, double t2, const double *rows, double *F) {
  static_assert(BOYS_NTAYLOR == 8 && BOYS_SROW == 10, "row layout read as five double2");
#ifdef __CUDA_ARCH__
  const double u = fma(T, 8.0, 6755399441055744.0);
  const int i = __double2loint(u);
  const double x = fma(u - 6755399441055744.0, 0.125, -T);
#else
  const int i = __double2int_rn(T * 8.0);
  const double x = (double)i * 0.125 - T;
#endif
  const double2 *row = reinterpret_cast<const double2 *>(rows + i * BOYS_SROW);
  const double2 c01 = row[0], c23 = row[1], c45 = row[2], c67 = row[3], c89 = row[4];
  if constexpr (L == 1) {
    double f = c89.y, d = f;   // value and derivative by Horner's rule
    f = fma(x, f, c89.x);
    d = fma(x, d, f);
    f = fma(x, f, c67.y);
    d = fma(x, d, f);
    f = fma(x, f, c67.x);
    d = fma(x, d, f);
    f = fma(x, f, c45.y);
    d = fma(x, d, f);
    f = fma(x, f, c45.x);
    d = fma(x, d, f);
    f = fma(x, f, c23.y);
    d = fma(x, d, f);
    f = fma(x, f, c23.x);
    d = fma(x, d, f);
    f = fma(x, f, c01.y);
    d = fma(x, d, f);
    F[0] = fma(x, f, c01.x);
    F[1] = d;
  } else {
    double f = c89.x;
    f = fma(x, f, c67.y);
    f = fma(x, f, c67.x);
    f = fma(x, f, c45.y);
    f = fma(x, f, c45.x);
    f = fma(x, f, c23.y);
    f = fma(x, f, c23.x);
    f = fma(x, f, c01.y);
    f = fma(x, f, c01.x);
    F[L] = f;
    if constexpr (L > 1) {
      const double e = c89.y * exp_small(x);
#pragma unroll
      for (int m = L - 1; m >= 0; --m) F[m] = fma(t2, F[m + 1], e) * (1.0 / (2 * m + 1));
    }
  }
}

// x^(-1/2) for positive normal x: the hardware's approximation (20 bits or more) and one step
// of the third-order iteration y (1 + e/2 + 3 e^2/8), e = 1 - x y^2 (the binomial series of
// (1 - e)^(-1/2); error 5 e^3/16 < 1e-17).  Without the special cases of rsqrt(), so without
// its branch.
__device__ __forceinline__ double class_rsqrt(double x) {
#ifdef __CUDA_ARCH__
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x * y, y, 1.0);
  return fma(y * e, fma(0.375, e, 0.5), y);
#else
  return rsqrt(x);
#endif
}

// Boys values of the class kernels for exponents p, q (s = p + q, m = p q) at squared distance
// R2: returns y and G[0..L] with  F_n(T) (-2 rho)^n (p+q)^(-1/2) = y (-2 m y^2)^n G[n].
// Near (T < boys_tmax): y = s^(-1/2), so m y^2 = rho, and G = F(T).  Far: y = (m R2)^(-1/2), so
// m y^2 = 1 / R2, and G[n] = c_n: F_n = c_n T^(-n-1/2) with T = m R2 / s leaves exactly that.
// One reciprocal square root serves both and the far values are a row of the table, so near and
// far lanes go together.  The generated code evaluates the rows of
// all primitive quartets it has at hand without a branch between them, so their chains
// overlap; when all of a lane's are far, it takes the constants and skips the rows.  Measured
// with the blocked columns above, (H2O)_32 cc-pVDZ, against one branch per primitive quartet
// and PrimPair arrays: (ss|ss) 5.16 -> 4.21 ms, (ps|ss) 10.37 -> 9.02, (pp|ss) 2.82 -> 2.19,
// (ds|ss) 2.73 -> 2.09, the build 54.5 -> 49.3 ms (without the skip (ss|ss) took 5.67).
struct ClassArg {
  double y, T;
  bool far;
};
template <int L>
__device__ __forceinline__ ClassArg class_arg(double s, double m, double R2) {
  ClassArg c;
  const double z = m * R2;
  c.far = !(z < boys_tmax(L) * s);   // also where z or s is not a number: its row is in the table
  c.y = class_rsqrt(c.far ? z : s);
  c.T = c.far ? boys_tfar(L) : z * (c.y * c.y);
  return c;
}
template <int L>
__device__ __forceinline__ void class_rows(const ClassArg &c, const double *rows, double *G) {
  boys_row_eval<L>(c.T, c.far ? 2.0 : 2.0 * c.T, rows, G);
}
// the far row's values, without reading it
template <int L>
__device__ __forceinline__ void class_far(double *G) {
  double c = 0.88622692545275801;   // sqrt(pi) / 2
#pragma unroll
  for (int n = 0; n <= L; ++n) {
    G[n] = c;
    c *= 0.5 * (2 * n + 1);
  }
}

// F_0..F_L at any T from the same rows (kernels whose Boys values are a small part)
template <int L>
__device__ __forceinline__ void boys_eval_sm(double T, const double *rows, double *F) {
  if (T < boys_tmax(L)) {
    boys_row_eval<L>(T, 2.0 * T, rows, F);
  } else {
    // F_0 = (sqrt(pi) / 2) T^(-1/2) and 1 / (2T) from one reciprocal square root
    const double r = rsqrt(T);
    F[0] = 0.88622692545275801 * r;
    if (L > 0) {
      const double e = L <= 5 ? 0.0 : exp(-T);   // below 4e-17 of (2m+1) F_m past boys_tmax up to L = 5
      const double i2t = 0.5 * r * r;
#pragma unroll
      for (int m = 0; m < L; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) * i2t;
    }
  }
}

template <int LA, int LB, int LC, int LD>
struct EriClass;
