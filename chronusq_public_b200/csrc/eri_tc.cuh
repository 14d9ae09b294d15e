// Shell quartets of high angular momentum on the FP64 tensor cores, one warp per quartet.
//
// McMurchie-Davidson as in the generated per-thread code:
//   W[h][cd] = sum_k (-1)^|k| R[h + k] E_ket[cd][k]      per primitive quartet, summed over kets
//   V[ab][cd] = sum_h E_bra[ab][h] W[h][cd]              per bra primitive pair
// with the Hermite expansions E of a primitive pair already in the reference's (spherical)
// functions: k_expansions writes them once per geometry, rows of functions, columns of
// Hermite triples padded to a multiple of four (ExpansionDims).
//
// What bounds these classes is the FP64 tensor pipe: an m8n8k4 step takes it 16 cycles, and
// the padding of the tiles is part of the count.  So everything else is arranged to cost few
// instructions per primitive quartet:
//  - the 32 lanes evaluate the Boys functions and R recursions of up to NB primitive quartets
//    at once, of as many list entries as it takes, one lane each, into shared memory;
//  - W is computed transposed, W^T[cd][h] = E_ket R: its accumulator fragment (row cd,
//    columns 2t, 2t + 1 of a tile of h) is, column by column, the A fragment of the second
//    product V^T[cd][ab] = W^T E_bra^T when that product takes h in the order 2t + i, so W
//    never leaves the registers;
//  - V^T stays in registers over a quartet's primitives and goes through shared memory once,
//    to the digest.
// Measured (B200, 1965 MHz), the kernel that walked one primitive quartet at a time with its
// Boys values on every lane -> this one: (H2O)_32 cc-pVDZ (dp|pp) 7.57 -> 3.38 ms, (dp|dp) 2.57 ->
// 0.60, (dd|pp) 1.80 -> 0.54, (dd|ds) 1.05 -> 0.38, (dd|dp) 1.02 -> 0.27; (H2O)_5 cc-pVTZ
// (fd|dp) 0.98 -> 0.20, (ff|ff) 0.61 -> 0.20.
//
// The sign (-1)^|k| = (-1)^|h| (-1)^|h + k| is put on R (its argument is Q - P instead of
// P - Q) and on the columns of E_bra.
#pragma once
#include "eri_common.cuh"

namespace warpmd {

// Expansion table of one primitive pair of class (LA LB): NS rows of HP doubles.
template <int LA, int LB>
struct ExpansionDims {
  static constexpr int NS = nfun(LA) * nfun(LB), H = nherm(LA + LB);
  static constexpr int HP = (H + 3) / 4 * 4;
  static constexpr int SIZE = NS * HP;
};

template <int LA, int LB, int LC, int LD>
struct TcDims {
  using B = ExpansionDims<LA, LB>;
  using K = ExpansionDims<LC, LD>;
  static constexpr int L = LA + LB + LC + LD, HL = nherm(L);
  static constexpr int MT = (K::NS + 7) / 8;      // tiles of cd (rows of W^T and V^T)
  static constexpr int NT = (B::NS + 7) / 8;      // tiles of ab (columns of V^T)
  static constexpr int HT = (B::H + 7) / 8;       // tiles of h
  static constexpr int KT = K::HP / 4;            // steps of k
  // tiles of h held at a time, so that W^T and V^T fit the registers beside the rest
  static constexpr int HB0 = (44 - MT * NT) / MT;
  static constexpr int HB = HB0 < 1 ? 1 : (HB0 > HT ? HT : HB0);
  // primitive quartets evaluated at once and the stride of their R columns: odd, so that the
  // lanes' columns and a column's triples fall in different banks; entry HL is zero (padding)
  static constexpr int NB = L <= 5 ? 32 : L <= 8 ? 16 : 8;
  static constexpr int HLS = (HL + 1) | 1;
  static constexpr int NQ = B::NS * K::NS;
  static constexpr int NSA = nfun(LA), NSB = nfun(LB), NSC = nfun(LC), NSD = nfun(LD);
  // staged density blocks of the digest: (d,c), (b,a), (b,d), (a,c), (b,c), (a,d)
  static constexpr int NXS = NSC * NSD + NSA * NSB + NSB * NSD + NSA * NSC + NSB * NSC + NSA * NSD;
  static constexpr int WARP_DOUBLES = NB * HLS + NQ + NXS;
};

// total t + u + v of Hermite triple h
__host__ __device__ constexpr int herm_total(int h) {
  int n = 0;
  while (nherm(n) <= h) ++n;
  return n;
}

}  // namespace warpmd

// Expansion tables of the primitive pairs of shell pairs [beg, end), all of class (LA LB), a
// warp per shell pair in turn.  out: the table of primitive pair prim0.
template <int LA, int LB>
__global__ void __launch_bounds__(128) k_expansions(Pairs P, Shells S, int beg, int end, int prim0,
                                                    double *__restrict__ out) {
  using D = warpmd::ExpansionDims<LA, LB>;
  constexpr int NE = warpmd::PairDims<LA, LB>::NE, NTE = LA + LB + 1;
  constexpr int NCA = warpmd::ncart(LA), NCB = warpmd::ncart(LB), NB = warpmd::nfun(LB);
  __shared__ double E[4][3 * NE];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int pair = beg + blockIdx.x * 4 + wid; pair < end; pair += gridDim.x * 4) {
    const int2 ab = P.sh[pair];
    const double3 A = S.center[ab.x], B = S.center[ab.y];
    const int p0 = P.poff[pair], np = P.np[pair];
    for (int i = p0; i < p0 + np; ++i) {
      const PrimPair p = P.prim[i];
      __syncwarp();
      if (lane < 3) {
        const double Pc = lane == 0 ? p.Px : lane == 1 ? p.Py : p.Pz, Ac = lane == 0 ? A.x : lane == 1 ? A.y : A.z,
                     Bc = lane == 0 ? B.x : lane == 1 ? B.y : B.z;
        warpmd::build_E1<LA, LB, double>(E[wid] + lane * NE, Pc - Ac, Pc - Bc, 0.5 * p.ip);
      }
      __syncwarp();
      const double *Ex = E[wid], *Ey = Ex + NE, *Ez = Ey + NE;
      for (int e = lane; e < D::SIZE; e += 32) {
        const int row = e / D::HP, h = e % D::HP, ia = row / NB, ib = row % NB;
        double s = 0.0;
        if (h < D::H) {
          int t, u, v;
          warpmd::herm_of(h, t, u, v);
          for (int ka = LA > 1 ? 0 : ia; ka < (LA > 1 ? NCA : ia + 1); ++ka) {
            const double ca = LA > 1 ? (LA == 2 ? kSph2 : kSph3)[ia * NCA + ka] : 1.0;
            if (ca == 0.0) continue;
            int ax, ay, az;
            warpmd::cart_of(LA, ka, ax, ay, az);
            for (int kb = LB > 1 ? 0 : ib; kb < (LB > 1 ? NCB : ib + 1); ++kb) {
              const double cb = LB > 1 ? (LB == 2 ? kSph2 : kSph3)[ib * NCB + kb] : 1.0;
              if (cb == 0.0) continue;
              int bx, by, bz;
              warpmd::cart_of(LB, kb, bx, by, bz);
              if (t > ax + bx || u > ay + by || v > az + bz) continue;
              s += ca * cb * Ex[(ax * (LB + 1) + bx) * NTE + t] * Ey[(ay * (LB + 1) + by) * NTE + u] *
                   Ez[(az * (LB + 1) + bz) * NTE + v];
            }
          }
        }
        out[(size_t)(i - prim0) * D::SIZE + e] = s;
      }
    }
  }
}

// One FP64 tensor-core step D += A B on an 8x8x4 tile (mma.sync m8n8k4 .f64).  Fragments:
// a = A[g][t], b = B[t][g], d[i] = D[g][2t+i] with g = lane / 4, t = lane % 4.
__device__ __forceinline__ void dmma_884(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

// R_tuv, t + u + v <= L, from fac[n] = R^n_000, by the downward recursion in place: a triple
// of total N at level n needs totals N - 1 and N - 2 of level n + 1 only, so the totals are
// taken from the highest down.  Up to L = 5 the column stays in registers until it is done.
template <int L>
__device__ __forceinline__ void hermite_column(const double (&fac)[L + 1], double X, double Y, double Z, double *col) {
  constexpr int HL = warpmd::nherm(L);
  double reg[L <= 5 ? HL : 1];
  auto at = [&](int i) -> double & {
    if constexpr (L <= 5) return reg[i];
    else return col[i];
  };
  at(0) = fac[L];
#pragma unroll
  for (int n = L - 1; n >= 0; --n) {
#pragma unroll
    for (int N = L; N >= 1; --N) {
      if (N > L - n) continue;
#pragma unroll
      for (int i = 0; i <= L; ++i)
#pragma unroll
        for (int v = 0; v <= L; ++v) {
          if (i > N || v > i) continue;
          const int t = N - i, u = i - v;
          const int here = (N * (N + 1) * (N + 2)) / 6 + (i * (i + 1)) / 2 + v;
          // the triple with one less in its first non-zero direction, and with two less
          const int s1 = ((N - 1) * N * (N + 1)) / 6, s2 = ((N - 2) * (N - 1) * N) / 6;
          double r;
          if (t > 0) {
            r = X * at(s1 + (i * (i + 1)) / 2 + v);
            if (t > 1) r += (t - 1) * at(s2 + (i * (i + 1)) / 2 + v);
          } else if (u > 0) {
            r = Y * at(s1 + ((i - 1) * i) / 2 + v);
            if (u > 1) r += (u - 1) * at(s2 + ((i - 2) * (i - 1)) / 2 + v);
          } else {
            r = Z * at(s1 + ((i - 1) * i) / 2 + v - 1);
            if (v > 1) r += (v - 1) * at(s2 + ((i - 2) * (i - 1)) / 2 + v - 2);
          }
          at(here) = r;
        }
    }
    at(0) = fac[n];
  }
  if constexpr (L <= 5) {
#pragma unroll
    for (int h = 0; h < HL; ++h) col[h] = reg[h];
  }
  col[HL] = 0.0;
}

// The same by the four lanes sub = 0..3 of a column, in step, with the recursion of each triple
// from a table: rec[h] = a | b << 10 | d << 20 | m << 22 for R_h = P_d R_a + m R_b (d = 0, 1,
// 2 for x, y, z).  For L > 8, whose unrolled form would be tens of thousands of
// instructions.  Every lane of the warp calls it.
template <int L>
__device__ __forceinline__ void hermite_column4(const double (&fac)[L + 1], double X, double Y, double Z, double *col,
                                                int sub, const int *rec) {
  if (sub == 0) {
    col[0] = fac[L];
    col[warpmd::nherm(L)] = 0.0;
  }
#pragma unroll
  for (int n = L - 1; n >= 0; --n) {
#pragma unroll 1
    for (int N = L - n; N >= 1; --N) {
      const int beg = (N * (N + 1) * (N + 2)) / 6, cnt = ((N + 1) * (N + 2)) / 2;
      __syncwarp();   // the totals above have read this one's old values
      for (int j = sub; j < cnt; j += 4) {
        const int r = rec[beg + j], d = (r >> 20) & 3;
        col[beg + j] = (d == 0 ? X : d == 1 ? Y : Z) * col[r & 1023] + (double)(r >> 22) * col[(r >> 10) & 1023];
      }
    }
    __syncwarp();
    if (sub == 0) col[0] = fac[n];
  }
}

// Expansion tables of a class's bra and ket pair classes: primitive pair i's table is at
// table + (i - prim0) * SIZE.
struct Expansions {
  const double *bra, *ket;
  int bra0, ket0;
};

// Warps claim `take` consecutive list entries at a time; lane q holds entry q's data.  A claim
// of several fills the lanes of the R phase; one of too many leaves warps idle at the end.
// take = 0: a quarter of a warp's share of the list, at most 8, at least 2 unless the list is
// shorter than kTakeTwo.  Measured, ms at 1 / 2 / 4 / 8 / 16: (dp|pp) of (H2O)_32 cc-pVDZ, 1.2 M
// entries, 4.56 / 3.82 / 3.51 / 3.38 / 3.38; (dp|dp) of (H2O)_11, 22 k, 0.092 / 0.084 / 0.082 /
// 0.105 / 0.166; (ff|dd) of (H2O)_5 cc-pVTZ, 1040, 0.121 / 0.095 / 0.127 / 0.199 / 0.359; (dd|dd)
// of (H2O)_11, 358, 0.025 / 0.031 / 0.041 / 0.066 / 0.113.
constexpr long long kTakeTwo = 512;
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128) k_eri_tc(const uint2 *__restrict__ ql, const long long *__restrict__ range, int blk,
                                                Pairs P, Shells S, Expansions X, const double *__restrict__ rows_g,
                                                DigestGroups dg, unsigned long long *__restrict__ qhead, int take) {
  using D = warpmd::TcDims<LA, LB, LC, LD>;
  constexpr int L = D::L, MT = D::MT, NT = D::NT, HT = D::HT, KT = D::KT, HB = D::HB, NBR = D::NB;
  constexpr int NSAB = D::B::NS, NSCD = D::K::NS, HPB = D::B::HP, HPK = D::K::HP;
  extern __shared__ __align__(16) double smem[];
  __shared__ int s_rec[L > 8 ? D::HL : 1];   // recursion table of hermite_column4
  if constexpr (L > 8) {
    for (int k = threadIdx.x; k < D::HL; k += blockDim.x) {
      int t, u, v, a = 0, b = 0, d = 0, m = 0;
      warpmd::herm_of(k, t, u, v);
      if (t > 0) {
        a = warpmd::hidx(t - 1, u, v);
        if (t > 1) b = warpmd::hidx(t - 2, u, v), m = t - 1;
      } else if (u > 0) {
        d = 1;
        a = warpmd::hidx(t, u - 1, v);
        if (u > 1) b = warpmd::hidx(t, u - 2, v), m = u - 1;
      } else if (v > 0) {
        d = 2;
        a = warpmd::hidx(t, u, v - 1);
        if (v > 1) b = warpmd::hidx(t, u, v - 2), m = v - 1;
      }
      s_rec[k] = a | (b << 10) | (d << 20) | (m << 22);
    }
  }
  // s_sum[(n * KT + kt) * 32 + lane]: R index of h + k for the lane's B fragment of tile (n, kt)
  __shared__ short s_sum[HT * KT * 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < HT * KT * 32; e += blockDim.x) {
    const int l = e & 31, h = (e >> 5) / KT * 8 + (l >> 2), k = (e >> 5) % KT * 4 + (l & 3);
    int idx = D::HL;
    if (h < D::B::H && k < D::K::H) {
      int t1, u1, v1, t2, u2, v2;
      warpmd::herm_of(h, t1, u1, v1);
      warpmd::herm_of(k, t2, u2, v2);
      idx = warpmd::hidx(t1 + t2, u1 + u2, v1 + v2);
    }
    s_sum[e] = (short)idx;
  }
  __syncthreads();
  double *Rw = smem + (size_t)wid * D::WARP_DOUBLES, *V = Rw + NBR * D::HLS, *Xs = V + D::NQ;
  const int g = lane >> 2, t = lane & 3;
  unsigned odd = 0;   // bit 2 n + i: triple 8 n + 2 t + i has an odd total
#pragma unroll
  for (int n = 0; n < HT; ++n)
#pragma unroll
    for (int i = 0; i < 2; ++i) odd |= (unsigned)(warpmd::herm_total(8 * n + 2 * t + i) & 1) << (2 * n + i);
  const double *rows = rows_g + boys_rows_off(L);
  const long long beg = range[2 * blk], end = range[2 * blk + 1];
  if (take <= 0) {
    const long long warps = (long long)gridDim.x * (blockDim.x >> 5);
    take = (int)min(8ll, max((end - beg) >= kTakeTwo ? 2ll : 1ll, (end - beg) / (4 * warps)));
  }
  for (;;) {
    unsigned long long c0 = 0;
    if (lane == 0) c0 = atomicAdd(qhead + blk, (unsigned long long)take);
    c0 = __shfl_sync(0xffffffffu, c0, 0);
    const long long first = beg + (long long)c0;
    if (first >= end) return;
    const int nq = (int)min((long long)take, end - first);
    // lane q: entry q
    const uint2 e = ql[first + min(lane, nq - 1)];
    const int2 ab = P.sh[e.x], cd = P.sh[e.y];
    const int nk = P.np[e.y], pb = P.poff[e.x], pk = P.poff[e.y];
    const int np = lane < nq ? P.np[e.x] * nk : 0;
    const int a0 = S.bf[ab.x], b0 = S.bf[ab.y], c0f = S.bf[cd.x], d0 = S.bf[cd.y], mol = S.mol[ab.x];
    const int deg = (ab.x == ab.y ? 1 : 2) * (cd.x == cd.y ? 1 : 2) * (e.x == e.y ? 1 : 2);
    unsigned total;
    const int pre = (int)warp_excl_scan((unsigned)np, total);
    double vt[MT][NT][2];
#pragma unroll
    for (int m = 0; m < MT; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n) vt[m][n][0] = vt[m][n][1] = 0.0;
    for (int base = 0; base < (int)total; base += NBR) {
      // the lane's primitive quartet: entry q, bra primitive pair ib, ket primitive pair ik
      // (four lanes to a column when L > 8)
      const int slot = L > 8 ? lane >> 2 : min(lane, NBR - 1);
      const int m = min(base + slot, (int)total - 1);
      int q = 0;
#pragma unroll
      for (int s = 16; s > 0; s >>= 1) {
        const int cand = q + s;
        const int pc = __shfl_sync(0xffffffffu, pre, cand & 31);
        if (cand < nq && pc <= m) q = cand;
      }
      const int qnk = __shfl_sync(0xffffffffu, nk, q), local = m - __shfl_sync(0xffffffffu, pre, q);
      const int ib = local / qnk, ik = local - ib * qnk;
      const int bi = __shfl_sync(0xffffffffu, pb, q) + ib, ki = __shfl_sync(0xffffffffu, pk, q) + ik;
      __syncwarp();   // the round before has been read
      if (L > 8 || lane < NBR) {
        const PrimPair bp = P.prim[bi], kp = P.prim[ki];
        const double pq = bp.p + kp.p, rpq = rsqrt(pq), rho = bp.p * kp.p * (rpq * rpq);
        const double x = kp.Px - bp.Px, y = kp.Py - bp.Py, z = kp.Pz - bp.Pz;
        double F[L + 1];
        boys_eval_sm<L>(rho * (x * x + y * y + z * z), rows, F);
        double f = bp.Kp * kp.Kp * rpq;
#pragma unroll
        for (int n = 0; n <= L; ++n) {
          F[n] *= f;
          f *= -2.0 * rho;
        }
        if constexpr (L > 8) hermite_column4<L>(F, x, y, z, Rw + slot * D::HLS, lane & 3, s_rec);
        else hermite_column<L>(F, x, y, z, Rw + slot * D::HLS);
      }
      __syncwarp();
      const int cnt = min(NBR, (int)total - base);
      for (int l = 0; l < cnt;) {
        // kets [ik, ik + run) of one entry's bra primitive pair
        const int from = L > 8 ? 4 * l : l;
        const int qq = __shfl_sync(0xffffffffu, q, from), kk = __shfl_sync(0xffffffffu, ik, from);
        const int nkq = __shfl_sync(0xffffffffu, nk, qq), run = min(nkq - kk, cnt - l);
        const double *eb = X.bra + (size_t)(__shfl_sync(0xffffffffu, bi, from) - X.bra0) * D::B::SIZE;
        const double *ek = X.ket + (size_t)(__shfl_sync(0xffffffffu, ki, from) - X.ket0) * D::K::SIZE;
        const double *col0 = Rw + l * D::HLS;
#pragma unroll
        for (int h0 = 0; h0 < HT; h0 += HB) {
          double w[MT][HB][2];
#pragma unroll
          for (int mt = 0; mt < MT; ++mt)
#pragma unroll
            for (int n = 0; n < HB; ++n) w[mt][n][0] = w[mt][n][1] = 0.0;
          const double *ekj = ek, *col = col0;
          for (int j = 0; j < run; ++j, ekj += D::K::SIZE, col += D::HLS) {
#pragma unroll
            for (int kt = 0; kt < KT; ++kt) {
              double a[MT];
#pragma unroll
              for (int mt = 0; mt < MT; ++mt)
                a[mt] = 8 * mt + g < NSCD ? __ldg(ekj + (8 * mt + g) * HPK + 4 * kt + t) : 0.0;
#pragma unroll
              for (int n = 0; n < HB; ++n) {
                if (h0 + n >= HT) continue;
                const double b = col[s_sum[((h0 + n) * KT + kt) * 32 + lane]];
#pragma unroll
                for (int mt = 0; mt < MT; ++mt) dmma_884(w[mt][n], a[mt], b);
              }
            }
          }
#pragma unroll
          for (int n = 0; n < HB; ++n) {
            if (h0 + n >= HT) continue;
            const int h = 8 * (h0 + n) + 2 * t;
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) {
              double2 b = make_double2(0.0, 0.0);
              if (8 * nt + g < NSAB && h < HPB)
                b = __ldg(reinterpret_cast<const double2 *>(eb + (8 * nt + g) * HPB + h));
              if ((odd >> (2 * (h0 + n))) & 1u) b.x = -b.x;
              if ((odd >> (2 * (h0 + n) + 1)) & 1u) b.y = -b.y;
#pragma unroll
              for (int mt = 0; mt < MT; ++mt) {
                dmma_884(vt[mt][nt], w[mt][n][0], b.x);
                dmma_884(vt[mt][nt], w[mt][n][1], b.y);
              }
            }
          }
        }
        l += run;
        const int done = base + l;   // primitive quartets of the claim evaluated so far
        if (done != __shfl_sync(0xffffffffu, pre, qq) + __shfl_sync(0xffffffffu, np, qq)) continue;
        // entry qq is complete: V[ab][cd] to shared memory, then its digest
        __syncwarp();
#pragma unroll
        for (int mt = 0; mt < MT; ++mt)
#pragma unroll
          for (int nt = 0; nt < NT; ++nt)
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int c = 8 * mt + g, a = 8 * nt + 2 * t + i;
              if (c < NSCD && a < NSAB) V[a * NSCD + c] = vt[mt][nt][i];
              vt[mt][nt][i] = 0.0;
            }
        digest_warp<LA, LB, LC, LD>(V, Xs, dg, __shfl_sync(0xffffffffu, a0, qq), __shfl_sync(0xffffffffu, b0, qq),
                                    __shfl_sync(0xffffffffu, c0f, qq), __shfl_sync(0xffffffffu, d0, qq),
                                    __shfl_sync(0xffffffffu, mol, qq), (double)__shfl_sync(0xffffffffu, deg, qq),
                                    lane);
      }
    }
  }
}
