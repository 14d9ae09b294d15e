// One-electron integrals S, T, V on the device (the reference computes them on the host
// with Libint's OneEDriver, src/aointegrals/aointegrals_builders.cpp:27-133, 337-467).
//
// McMurchie-Davidson, one warp per shell pair (kernels below):
//   S_ab  = sum_prims K (pi/p)^(3/2) Ex^{ax bx}_0 Ey^{ay by}_0 Ez^{az bz}_0
//   T_ab  = sum over directions of T1D_x S1D_y S1D_z with
//           T1D_ij = -2 b^2 S1D_{i,j+2} + b (2j+1) S1D_{ij} - j(j-1)/2 S1D_{i,j-2}
//   V_ab  = -sum_C Z_C (2 pi/p) K sum_tuv E^{ab}_{tuv} R_{tuv}(p, P - C)
// with K = c_a c_b exp(-a b/p |A-B|^2), S1D_ij = E^{ij}_0 sqrt(pi/p), then the Cartesian
// blocks are transformed to real solid harmonics for pure (L > 1) shells.
#pragma once
#include <type_traits>

#include "eri_common.cuh"

#define OE_MAXL 3

struct OneEShells {
  const int *L, *nprim, *poff, *bf;
  const double *alpha, *coef;
  const double3 *center;
};

// Molecule layout for batches: shell -> molecule, per-molecule output offset / leading
// dimension and charge range.  For one molecule: xoff = 0, ld = caller's, all charges.
struct OneEMols {
  const int *shmol;
  const long long *xoff;
  const int *nbf;
  const int *coff;   // charges of molecule m: [coff[m], coff[m+1])
  int batch;
};

// ---- class kernels: one warp per shell pair of one class (LA LB) ----
//
// What bounds them is the nuclear attraction: primitive pairs x nuclei Boys functions and R
// recursions (21 M for (H2O)_24 in cc-pVDZ).  The lanes of a warp split them: C lanes over
// the nuclei, 32 / C groups over the primitive pairs (charge_lanes picks C for the pair).
// A lane sums R_tuv over its nuclei, applies its primitive pair's expansion coefficients to
// the sum once, and the warp adds its Cartesian blocks up at the end.  LA and LB are
// template arguments so that every array index is a constant and the intermediates stay in
// registers.  (H2O)_24 cc-pVDZ, S, T, V and the dipole matrices: 277 us, of which the
// nuclear attraction of the s and p pairs is two thirds; with one thread per pair, run-time
// angular momenta and so arrays in local memory it took 18.8 ms.
#ifdef __CUDACC__
#define OE_LANES 32
__device__ __forceinline__ double oe_warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
#define OE_SYNCWARP() __syncwarp()
#define OE_SYNCBLOCK() __syncthreads()
#define OE_SHARED __shared__
#define OE_GRID gridDim.x
#define OE_BOUNDS __launch_bounds__(32 * OE_WARPS)
#else   // a host build runs a kernel body as one thread: one lane
#define OE_LANES 1
inline double oe_warp_sum(double x) { return x; }
#define OE_SYNCWARP()
#define OE_SYNCBLOCK()
#define OE_SHARED static
#define OE_GRID 1
#define OE_BOUNDS
#endif
#define OE_WARPS 4   // warps (shell pairs in flight) per block

// exponents of Cartesian component k of angular momentum l <= 3 (order of oe_cart)
__host__ __device__ constexpr int oe_row(int k) { return (k >= 1) + (k >= 3) + (k >= 6); }
__host__ __device__ constexpr int oe_cz(int k) { return k - oe_row(k) * (oe_row(k) + 1) / 2; }
__host__ __device__ constexpr int oe_cx(int l, int k) { return l - oe_row(k); }
__host__ __device__ constexpr int oe_cy(int k) { return oe_row(k) - oe_cz(k); }
__host__ __device__ constexpr int oe_ncart(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int oe_nherm(int n) { return (n + 1) * (n + 2) * (n + 3) / 6; }
__host__ __device__ constexpr int oe_herm(int t, int u, int v) {
  return ((t + u + v) * (t + u + v + 1) * (t + u + v + 2)) / 6 + ((u + v) * (u + v + 1)) / 2 + v;
}

// E[(i * (JB + 1) + j) * (LA + JB + 1) + t], i <= LA, j <= JB, t <= i + j
template <int LA, int JB>
__device__ __forceinline__ void oe_expand(double (&E)[(LA + 1) * (JB + 1) * (LA + JB + 1)], double PA, double PB,
                                          double o2p) {
  constexpr int NT = LA + JB + 1;
  E[0] = 1.0;
#pragma unroll
  for (int j = 1; j <= JB; ++j)
#pragma unroll
    for (int t = 0; t <= JB; ++t) {
      if (t > j) continue;
      double v = t < j ? PB * E[(j - 1) * NT + t] : 0.0;
      if (t > 0) v += o2p * E[(j - 1) * NT + t - 1];
      if (t + 1 < j) v += (t + 1) * E[(j - 1) * NT + t + 1];
      E[j * NT + t] = v;
    }
#pragma unroll
  for (int i = 1; i <= LA; ++i)
#pragma unroll
    for (int j = 0; j <= JB; ++j)
#pragma unroll
      for (int t = 0; t <= LA + JB; ++t) {
        if (t > i + j) continue;
        const int from = ((i - 1) * (JB + 1) + j) * NT;
        double v = t < i + j ? PA * E[from + t] : 0.0;
        if (t > 0) v += o2p * E[from + t - 1];
        if (t + 1 < i + j) v += (t + 1) * E[from + t + 1];
        E[(i * (JB + 1) + j) * NT + t] = v;
      }
}

// one primitive pair of shells a and b
struct OePrim {
  double be, p, o2p, K;   // exponent on b, p = sum, 1 / (2 p), c_a c_b exp(-mu AB^2)
  double3 P;
};
__device__ __forceinline__ OePrim oe_prim(const OneEShells &sh, int a, int b, const double3 &A, const double3 &B,
                                          int i, int j) {
  const double al = sh.alpha[sh.poff[a] + i], be = sh.alpha[sh.poff[b] + j];
  const double ABx = A.x - B.x, ABy = A.y - B.y, ABz = A.z - B.z;
  OePrim q;
  q.be = be;
  q.p = al + be;
  q.o2p = 0.5 / q.p;
  q.K = sh.coef[sh.poff[a] + i] * sh.coef[sh.poff[b] + j] *
        exp(-al * be / q.p * (ABx * ABx + ABy * ABy + ABz * ABz));
  q.P.x = (al * A.x + be * B.x) / q.p;
  q.P.y = (al * A.y + be * B.y) / q.p;
  q.P.z = (al * A.z + be * B.z) / q.p;
  return q;
}

// Cartesian overlap and kinetic blocks of the lane's share of the primitive pairs
template <int LA, int LB>
__device__ __forceinline__ void oe_overlap_kinetic(const OneEShells &sh, int a, int b, int lane, double *Sc,
                                                   double *Tc) {
  constexpr int NCA = oe_ncart(LA), NCB = oe_ncart(LB), JB = LB + 2, NT = LA + JB + 1;
  const double3 A = sh.center[a], B = sh.center[b];
#pragma unroll
  for (int k = 0; k < NCA * NCB; ++k) Sc[k] = Tc[k] = 0.0;
  const int nb = sh.nprim[b], n = sh.nprim[a] * nb;
  for (int q = lane; q < n; q += OE_LANES) {
    const OePrim w = oe_prim(sh, a, b, A, B, q / nb, q % nb);
    // 1D overlaps and kinetic factors of every (i, j)
    double s1[3][(LA + 1) * (LB + 1)], t1[3][(LA + 1) * (LB + 1)];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double E[(LA + 1) * (JB + 1) * NT];
      const double Pd = d == 0 ? w.P.x : d == 1 ? w.P.y : w.P.z, Ad = d == 0 ? A.x : d == 1 ? A.y : A.z,
                   Bd = d == 0 ? B.x : d == 1 ? B.y : B.z;
      oe_expand<LA, JB>(E, Pd - Ad, Pd - Bd, w.o2p);
#pragma unroll
      for (int i = 0; i <= LA; ++i)
#pragma unroll
        for (int j = 0; j <= LB; ++j) {
          const double s = E[(i * (JB + 1) + j) * NT];
          double t = -2.0 * w.be * w.be * E[(i * (JB + 1) + j + 2) * NT] + w.be * (2 * j + 1) * s;
          if (j >= 2) t -= 0.5 * j * (j - 1) * E[(i * (JB + 1) + (j >= 2 ? j - 2 : 0)) * NT];
          s1[d][i * (LB + 1) + j] = s;
          t1[d][i * (LB + 1) + j] = t;
        }
    }
    const double r = sqrt(3.141592653589793 / w.p), pre = w.K * r * r * r;
#pragma unroll
    for (int ka = 0; ka < NCA; ++ka)
#pragma unroll
      for (int kb = 0; kb < NCB; ++kb) {
        const int x = oe_cx(LA, ka) * (LB + 1) + oe_cx(LB, kb), y = oe_cy(ka) * (LB + 1) + oe_cy(kb),
                  z = oe_cz(ka) * (LB + 1) + oe_cz(kb);
        const double sx = s1[0][x], sy = s1[1][y], sz = s1[2][z];
        Sc[ka * NCB + kb] += pre * sx * sy * sz;
        Tc[ka * NCB + kb] += pre * (t1[0][x] * sy * sz + sx * t1[1][y] * sz + sx * sy * t1[2][z]);
      }
  }
}

// Cartesian dipole blocks <a| r_k - O_k |b> of the lane's share of the primitive pairs, by
// the McMurchie-Davidson first moment (Helgaker, Jorgensen & Olsen eq. 9.5.43): the moment's
// 1D factor is sqrt(pi/p) (E^{ij}_1 + (P - O) E^{ij}_0), the other two are overlaps.
template <int LA, int LB>
__device__ __forceinline__ void oe_dipole(const OneEShells &sh, int a, int b, const double3 &O, int lane, double *Dx,
                                          double *Dy, double *Dz) {
  constexpr int NCA = oe_ncart(LA), NCB = oe_ncart(LB), NT = LA + LB + 1;
  const double3 A = sh.center[a], B = sh.center[b];
#pragma unroll
  for (int k = 0; k < NCA * NCB; ++k) Dx[k] = Dy[k] = Dz[k] = 0.0;
  const int nb = sh.nprim[b], n = sh.nprim[a] * nb;
  for (int q = lane; q < n; q += OE_LANES) {
    const OePrim w = oe_prim(sh, a, b, A, B, q / nb, q % nb);
    double s1[3][(LA + 1) * (LB + 1)], m1[3][(LA + 1) * (LB + 1)];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      double E[(LA + 1) * (LB + 1) * NT];
      const double Pd = d == 0 ? w.P.x : d == 1 ? w.P.y : w.P.z, Ad = d == 0 ? A.x : d == 1 ? A.y : A.z,
                   Bd = d == 0 ? B.x : d == 1 ? B.y : B.z, Od = d == 0 ? O.x : d == 1 ? O.y : O.z;
      oe_expand<LA, LB>(E, Pd - Ad, Pd - Bd, w.o2p);
#pragma unroll
      for (int ij = 0; ij < (LA + 1) * (LB + 1); ++ij) {
        const double e1 = ij > 0 ? E[ij * NT + (NT > 1 ? 1 : 0)] : 0.0;
        s1[d][ij] = E[ij * NT];
        m1[d][ij] = e1 + (Pd - Od) * E[ij * NT];
      }
    }
    const double r = sqrt(3.141592653589793 / w.p), pre = w.K * r * r * r;
#pragma unroll
    for (int ka = 0; ka < NCA; ++ka)
#pragma unroll
      for (int kb = 0; kb < NCB; ++kb) {
        const int x = oe_cx(LA, ka) * (LB + 1) + oe_cx(LB, kb), y = oe_cy(ka) * (LB + 1) + oe_cy(kb),
                  z = oe_cz(ka) * (LB + 1) + oe_cz(kb);
        Dx[ka * NCB + kb] += pre * m1[0][x] * s1[1][y] * s1[2][z];
        Dy[ka * NCB + kb] += pre * s1[0][x] * m1[1][y] * s1[2][z];
        Dz[ka * NCB + kb] += pre * s1[0][x] * s1[1][y] * m1[2][z];
      }
  }
}

// Lanes that split the nuclei of one primitive pair (a power of two): the fewest lane steps,
// with one step's worth for the expansion of each primitive pair.
__device__ __forceinline__ int charge_lanes(int nprims, int ncharge) {
  int best = 1;
#ifdef __CUDACC__
  int cost = 0x7fffffff;
  for (int c = 1; c <= OE_LANES; c <<= 1) {
    const int groups = OE_LANES / c, k = ((nprims + groups - 1) / groups) * ((ncharge + c - 1) / c + 1);
    if (k < cost) cost = k, best = c;
  }
#endif
  return best;
}

// Cartesian nuclear-attraction block of the lane's share of (primitive pairs) x (nuclei
// [c_beg, c_end)).  `rows`: the Boys rows of LA + LB in shared memory.
template <int LA, int LB>
__device__ __forceinline__ void oe_attraction(const OneEShells &sh, int a, int b, int c_beg, int c_end,
                                              const double *__restrict__ Zc, const double3 *__restrict__ Rc,
                                              const double *rows, int lane, double *Vc) {
  constexpr int NCA = oe_ncart(LA), NCB = oe_ncart(LB), L = LA + LB, NH = oe_nherm(L), NT = L + 1;
  const double3 A = sh.center[a], B = sh.center[b];
#pragma unroll
  for (int k = 0; k < NCA * NCB; ++k) Vc[k] = 0.0;
  const int nb = sh.nprim[b], n = sh.nprim[a] * nb;
  const int C = charge_lanes(n, c_end - c_beg), groups = OE_LANES / C;
  for (int q = lane / C; q < n; q += groups) {
    const OePrim w = oe_prim(sh, a, b, A, B, q / nb, q % nb);
    double H[NH];
#pragma unroll
    for (int h = 0; h < NH; ++h) H[h] = 0.0;
    for (int c = c_beg + lane % C; c < c_end; c += C) {
      const double X = w.P.x - Rc[c].x, Y = w.P.y - Rc[c].y, Z = w.P.z - Rc[c].z;
      double F[L + 1], R[NH];
      boys_eval_sm<L>(w.p * (X * X + Y * Y + Z * Z), rows, F);
      double f = Zc[c];
#pragma unroll
      for (int m = 0; m <= L; ++m) {
        F[m] *= f;
        f *= -2.0 * w.p;
      }
      // R^{(m)}_{tuv}, m = L .. 0, in place: a triple of total N needs only totals below N of
      // the level before, so the totals are taken from the highest down
      R[0] = F[L];
#pragma unroll
      for (int m = L - 1; m >= 0; --m) {
#pragma unroll
        for (int N = L; N >= 1; --N) {
          if (N > L - m) continue;
#pragma unroll
          for (int i = 0; i <= L; ++i)
#pragma unroll
            for (int v = 0; v <= L; ++v) {
              if (i > N || v > i) continue;
              const int t = N - i, u = i - v;
              double r;
              if (t > 0) {
                r = X * R[oe_herm(t - 1, u, v)];
                if (t > 1) r += (t - 1) * R[oe_herm(t - 2, u, v)];
              } else if (u > 0) {
                r = Y * R[oe_herm(t, u - 1, v)];
                if (u > 1) r += (u - 1) * R[oe_herm(t, u - 2, v)];
              } else {
                r = Z * R[oe_herm(t, u, v - 1)];
                if (v > 1) r += (v - 1) * R[oe_herm(t, u, v - 2)];
              }
              R[oe_herm(t, u, v)] = r;
            }
        }
        R[0] = F[m];
      }
#pragma unroll
      for (int h = 0; h < NH; ++h) H[h] += R[h];
    }
    double Ex[(LA + 1) * (LB + 1) * NT], Ey[(LA + 1) * (LB + 1) * NT], Ez[(LA + 1) * (LB + 1) * NT];
    oe_expand<LA, LB>(Ex, w.P.x - A.x, w.P.x - B.x, w.o2p);
    oe_expand<LA, LB>(Ey, w.P.y - A.y, w.P.y - B.y, w.o2p);
    oe_expand<LA, LB>(Ez, w.P.z - A.z, w.P.z - B.z, w.o2p);
    const double pre = -2.0 * 3.141592653589793 / w.p * w.K;
#pragma unroll
    for (int ka = 0; ka < NCA; ++ka)
#pragma unroll
      for (int kb = 0; kb < NCB; ++kb) {
        const int ax = oe_cx(LA, ka), ay = oe_cy(ka), az = oe_cz(ka), bx = oe_cx(LB, kb), by = oe_cy(kb),
                  bz = oe_cz(kb);
        double s = 0.0;
#pragma unroll
        for (int t = 0; t <= L; ++t)
#pragma unroll
          for (int u = 0; u <= L; ++u)
#pragma unroll
            for (int v = 0; v <= L; ++v) {
              if (t > ax + bx || u > ay + by || v > az + bz) continue;
              s += Ex[(ax * (LB + 1) + bx) * NT + t] * Ey[(ay * (LB + 1) + by) * NT + u] *
                   Ez[(az * (LB + 1) + bz) * NT + v] * H[oe_herm(t, u, v)];
            }
        Vc[ka * NCB + kb] += pre * s;
      }
  }
}

// Cartesian block M[ka * ncb + kb] of shell pair (a, b) to real solid harmonics for pure
// (L > 1) shells, stored at rows a0.., columns b0.. of out and, transposed, at rows b0..,
// columns a0.. (column-major, leading dimension ld), by the lanes of a warp.
__device__ __forceinline__ void oe_store_pair(const double *M, int la, int lb, int a0, int b0, double *out, int ld) {
  const int nca = oe_ncart(la), ncb = oe_ncart(lb), na = la > 1 ? 2 * la + 1 : nca, nb = lb > 1 ? 2 * lb + 1 : ncb;
  const double *Ca = la == 2 ? kSph2 : kSph3, *Cb = lb == 2 ? kSph2 : kSph3;
  for (int e = threadIdx.x % OE_LANES; e < na * nb; e += OE_LANES) {
    const int i = e / nb, j = e % nb;
    if (a0 == b0 && j > i) continue;   // a shell with itself: one value for (i, j) and (j, i)
    double s = 0.0;
    for (int ka = la > 1 ? 0 : i; ka < (la > 1 ? nca : i + 1); ++ka)
      for (int kb = lb > 1 ? 0 : j; kb < (lb > 1 ? ncb : j + 1); ++kb)
        s += (la > 1 ? Ca[i * nca + ka] : 1.0) * (lb > 1 ? Cb[j * ncb + kb] : 1.0) * M[ka * ncb + kb];
    out[(size_t)(a0 + i) + (size_t)(b0 + j) * ld] = s;
    out[(size_t)(b0 + j) + (size_t)(a0 + i) * ld] = s;
  }
}

// The warp's sum of the lanes' Cartesian blocks M, stored.  `blk`: the block's doubles of
// shared memory, the warp's own.
template <int LA, int LB>
__device__ __forceinline__ void oe_store_block(const double *M, double *blk, int lane, int a0, int b0, double *out,
                                               int ld) {
  OE_SYNCWARP();   // the block before has been read
#pragma unroll
  for (int k = 0; k < oe_ncart(LA) * oe_ncart(LB); ++k) {
    const double s = oe_warp_sum(M[k]);
    if (k % OE_LANES == lane) blk[k] = s;
  }
  OE_SYNCWARP();
  oe_store_pair(blk, LA, LB, a0, b0, out, ld);
}

// S, T and V of the shell pairs (a of LA, b of LB) pairs[0 .. npairs), a warp per pair in
// turn.  `boys`: the finished Boys rows of the module (a host build: the table they are made
// from).
template <int LA, int LB>
__global__ void OE_BOUNDS
    k_one_e_class(OneEShells sh, const int2 *__restrict__ pairs, long long npairs, int ncharge,
                  const double *__restrict__ Zc, const double3 *__restrict__ Rc, const double *__restrict__ boys,
                  double *S0, double *T0, double *V0, int ld, OneEMols om) {
  constexpr int NC = oe_ncart(LA) * oe_ncart(LB);
  __align__(16) OE_SHARED double rows[boys_rows_size(LA + LB)];
  OE_SHARED double blocks[OE_WARPS][NC];
#ifdef __CUDACC__
  load_boys<LA + LB>(boys, rows);
#else
  stage_boys<LA + LB>(boys, rows);
#endif
  OE_SYNCBLOCK();
  const int lane = threadIdx.x % OE_LANES, warp = threadIdx.x / OE_LANES, warps = blockDim.x / OE_LANES;
  for (long long ip = (long long)blockIdx.x * warps + warp; ip < npairs; ip += (long long)OE_GRID * warps) {
    const int a = pairs[ip].x, b = pairs[ip].y;
    double *S = S0, *T = T0, *V = V0;
    int c_beg = 0, c_end = ncharge;
    if (om.batch) {
      const int m = om.shmol[a];
      S += om.xoff[m];
      T += om.xoff[m];
      V += om.xoff[m];
      ld = om.nbf[m];
      c_beg = om.coff[m];
      c_end = om.coff[m + 1];
    }
    const int a0 = sh.bf[a], b0 = sh.bf[b];
    double *blk = blocks[warp];
    {
      double Sc[NC], Tc[NC];
      oe_overlap_kinetic<LA, LB>(sh, a, b, lane, Sc, Tc);
      oe_store_block<LA, LB>(Sc, blk, lane, a0, b0, S, ld);
      oe_store_block<LA, LB>(Tc, blk, lane, a0, b0, T, ld);
    }
    double Vc[NC];
    oe_attraction<LA, LB>(sh, a, b, c_beg, c_end, Zc, Rc, rows, lane, Vc);
    oe_store_block<LA, LB>(Vc, blk, lane, a0, b0, V, ld);
  }
}

// Dipole matrices of the shell pairs (a of LA, b of LB): D0 holds the x, y and z matrices at
// D0, D0 + ld * nbf and D0 + 2 * ld * nbf.
template <int LA, int LB>
__global__ void OE_BOUNDS
    k_dipole_class(OneEShells sh, const int2 *__restrict__ pairs, long long npairs, double3 O, double *D0, int ld,
                   int nbf) {
  constexpr int NC = oe_ncart(LA) * oe_ncart(LB);
  OE_SHARED double blocks[OE_WARPS][NC];
  const int lane = threadIdx.x % OE_LANES, warp = threadIdx.x / OE_LANES, warps = blockDim.x / OE_LANES;
  for (long long ip = (long long)blockIdx.x * warps + warp; ip < npairs; ip += (long long)OE_GRID * warps) {
    const int a = pairs[ip].x, b = pairs[ip].y;
    double Dx[NC], Dy[NC], Dz[NC];
    oe_dipole<LA, LB>(sh, a, b, O, lane, Dx, Dy, Dz);
    double *blk = blocks[warp];
    const int a0 = sh.bf[a], b0 = sh.bf[b];
    oe_store_block<LA, LB>(Dx, blk, lane, a0, b0, D0, ld);
    oe_store_block<LA, LB>(Dy, blk, lane, a0, b0, D0 + (size_t)ld * nbf, ld);
    oe_store_block<LA, LB>(Dz, blk, lane, a0, b0, D0 + (size_t)2 * ld * nbf, ld);
  }
}

#ifndef __CUDACC__
// ---- host builds: the class code for a shell pair of run-time angular momenta ----
// Boys values of a run-time L from the table
__device__ __forceinline__ void boys_eval_rt(int L, double T, const double *__restrict__ tab, double *F) {
  if (T < BOYS_TMAX) {
    const int i = __double2int_rn(T * 10.0);
    const double x = (double)i * 0.1 - T;
    const double *row = tab + i * BOYS_NORD + L;
    double f = row[BOYS_NTAYLOR];
    for (int k = BOYS_NTAYLOR; k >= 1; --k) f = row[k - 1] + x * f / k;
    F[L] = f;
    const double e = exp(-T);
    for (int m = L - 1; m >= 0; --m) F[m] = (2.0 * T * F[m + 1] + e) / (2 * m + 1);
  } else {
    F[0] = 0.5 * sqrt(3.141592653589793 / T);
    const double e = exp(-T);
    for (int m = 0; m < L; ++m) F[m + 1] = ((2 * m + 1) * F[m] - e) / (2.0 * T);
  }
}

// f(LA, LB as integral constants) of the pair's angular momenta, L[x] >= L[y]
template <int LA = 0, int LB = 0, typename F>
inline void oe_host_class(int la, int lb, F f) {
  if (la == LA && lb == LB) f(std::integral_constant<int, LA>{}, std::integral_constant<int, LB>{});
  else if constexpr (LB < LA) oe_host_class<LA, LB + 1>(la, lb, f);
  else if constexpr (LA < OE_MAXL) oe_host_class<LA + 1, 0>(la, lb, f);
}
// S, T, V of shell pair pairs[blockIdx.x], shells in either order
inline void k_one_e(OneEShells sh, const int2 *pairs, long long, int ncharge, const double *Zc, const double3 *Rc,
                    const double *boys, double *S, double *T, double *V, int ld, OneEMols om) {
  const unsigned ip = blockIdx.x;
  int2 ab = pairs[ip];
  if (sh.L[ab.x] < sh.L[ab.y]) ab = int2{ab.y, ab.x};
  blockIdx.x = 0;
  oe_host_class(sh.L[ab.x], sh.L[ab.y], [&](auto la, auto lb) {
    k_one_e_class<la.value, lb.value>(sh, &ab, 1, ncharge, Zc, Rc, boys, S, T, V, ld, om);
  });
  blockIdx.x = ip;
}
// Cartesian dipole blocks of shell pair (a, b), shells in either order
inline void oe_dipole_pair(const OneEShells &sh, int a, int b, double3 O, double Dc[3][100]) {
  const bool swap = sh.L[a] < sh.L[b];
  const int x = swap ? b : a, y = swap ? a : b;
  double M[3][100];
  oe_host_class(sh.L[x], sh.L[y],
                [&](auto la, auto lb) { oe_dipole<la.value, lb.value>(sh, x, y, O, 0, M[0], M[1], M[2]); });
  const int nx = oe_ncart(sh.L[x]), ny = oe_ncart(sh.L[y]);
  for (int k = 0; k < 3; ++k)
    for (int i = 0; i < nx; ++i)
      for (int j = 0; j < ny; ++j) Dc[k][swap ? j * nx + i : i * ny + j] = M[k][i * ny + j];
}
#endif
