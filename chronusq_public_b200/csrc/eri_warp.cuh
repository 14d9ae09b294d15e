// Index helpers and the 1D Hermite expansion shared by the kernels that put a warp on a
// quartet or pair: the tensor-core class kernels (eri_tc.cuh) and the Schwarz bounds of the
// high pair classes (k_schwarz_warp in engine_impl.cuh).
#pragma once
#include "eri_common.cuh"

namespace warpmd {

__host__ __device__ constexpr int ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int nherm(int n) { return (n + 1) * (n + 2) * (n + 3) / 6; }
__host__ __device__ constexpr int nfun(int l) { return l > 1 ? 2 * l + 1 : ncart(l); }

// index of Hermite / Cartesian triple (t,u,v) in the "by total, CCA within total" order
__device__ __forceinline__ int hidx(int t, int u, int v) {
  const int n = t + u + v;
  const int i = n - t;
  return (n * (n + 1) * (n + 2)) / 6 + (i * (i + 1)) / 2 + v;
}
// decode Cartesian index k of angular momentum l (CCA order) into exponents
__device__ __forceinline__ void cart_of(int l, int k, int &x, int &y, int &z) {
  int i = 0;
  while ((i + 1) * (i + 2) / 2 <= k) ++i;
  const int j = k - i * (i + 1) / 2;
  x = l - i;
  y = i - j;
  z = j;
}
__device__ __forceinline__ void herm_of(int h, int &t, int &u, int &v) {
  int n = 0;
  while (nherm(n) <= h) ++n;
  cart_of(n, h - nherm(n - 1), t, u, v);
}

template <int LA, int LB>
struct PairDims {
  static constexpr int NE = (LA + 1) * (LB + 1) * (LA + LB + 1);  // E[i][j][t] per direction
};

// 1D Hermite coefficients E[i][j][t], i<=la, j<=lb, t<=i+j for one direction, by lanes.
// Layout: ((i*(lb+1)) + j)*(la+lb+1) + t.  Built serially by one lane (tiny).
template <int LA, int LB, typename T>
__device__ __forceinline__ void build_E1(T *E, T PA, T PB, T o2p) {
  constexpr int NT = LA + LB + 1;
#pragma unroll
  for (int k = 0; k < (LA + 1) * (LB + 1) * NT; ++k) E[k] = T(0);
  E[0] = T(1);
  // grow j at i = 0
#pragma unroll
  for (int j = 1; j <= LB; ++j)
#pragma unroll
    for (int t = 0; t <= j; ++t) {
      const T *prev = E + (0 * (LB + 1) + (j - 1)) * NT;
      T v = PB * (t <= j - 1 ? prev[t] : T(0));
      if (t > 0) v += o2p * prev[t - 1];
      if (t + 1 <= j - 1) v += T(t + 1) * prev[t + 1];
      E[(0 * (LB + 1) + j) * NT + t] = v;
    }
#pragma unroll
  for (int i = 1; i <= LA; ++i)
#pragma unroll
    for (int j = 0; j <= LB; ++j) {
      const T *prev = E + ((i - 1) * (LB + 1) + j) * NT;
      const int tm = i - 1 + j;
#pragma unroll
      for (int t = 0; t <= i + j; ++t) {
        T v = (t <= tm ? PA * prev[t] : T(0));
        if (t > 0 && t - 1 <= tm) v += o2p * prev[t - 1];
        if (t + 1 <= tm) v += T(t + 1) * prev[t + 1];
        E[(i * (LB + 1) + j) * NT + t] = v;
      }
    }
}

// Transform axis `ax` of a 4-index block from Cartesian to spherical (pure shells).
// in: dims d[0..3] (row-major), out: same with d[ax] -> 2l+1.  Lanes over output.
template <typename T>
__device__ __forceinline__ void sph_axis(const T *in, T *out, const int *d, int ax, int l, const double *C,
                                         int lane) {
  int nout[4] = {d[0], d[1], d[2], d[3]};
  const int ns = 2 * l + 1, nc = ncart(l);
  nout[ax] = ns;
  int inner = 1;
  for (int k = ax + 1; k < 4; ++k) inner *= d[k];
  int outer = 1;
  for (int k = 0; k < ax; ++k) outer *= d[k];
  const int total = outer * ns * inner;
  for (int e = lane; e < total; e += 32) {
    const int in_i = e % inner;
    const int m = (e / inner) % ns;
    const int o = e / (inner * ns);
    T s = T(0);
    for (int k = 0; k < nc; ++k) {
      const double c = C[m * nc + k];
      if (c != 0.0) s += T(c) * in[(o * nc + k) * inner + in_i];
    }
    out[e] = s;
  }
}

// Shared memory of a warp in k_schwarz_warp, (ab|ab) of one pair class.
template <int LA, int LB>
struct WarpDims {
  static constexpr int L = 2 * (LA + LB);
  static constexpr int HP = nherm(LA + LB), HL = nherm(L);
  static constexpr int NCAB = ncart(LA) * ncart(LB);
  static constexpr int NE = PairDims<LA, LB>::NE;
  static constexpr int NW = HP * NCAB, NC = NCAB * NCAB, NBUF = NW > NC ? NW : NC;
  // doubles per warp: E of bra and ket (3 directions), R (2 levels), W, C
  static constexpr int SMEM = 6 * NE + 2 * HL + 2 * NBUF;
};

}  // namespace warpmd
