// Internals of the cqgpu engine shared by its translation units: device data layout,
// the screening / ERI / digest kernels (templates), the context structure and the
// class-kernel launchers.  engine.cu holds the C ABI; eri_part.cu instantiates the
// class kernels, a share of the quartet classes per translation unit, so that they
// compile in parallel.
#pragma once
#include <cuda_runtime.h>
#include <cub/device/device_scan.cuh>

#include <algorithm>
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <numeric>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/cqgpu.h"
#include "eri_common.cuh"
#include "_gen/eri_classes.cuh"
#include "_gen/eri_gc_classes.cuh"
#include "eri_warp.cuh"

#define CQG_MAXL 3
#ifndef CQG_NPART
#define CQG_NPART 8          // translation units the class kernels are compiled in (eri_part.cu)
#endif
#define CQG_NPC ((CQG_MAXL + 1) * (CQG_MAXL + 2) / 2)       // pair classes
#define CQG_NQC (CQG_NPC * (CQG_NPC + 1) / 2)                // quartet classes
#define CQG_MAXG 4
#define CQG_NBUCKET 16   // ket buckets of a (molecule, pair class): the primitive-count bucket of the pair's group

static_assert(CQG_NQC <= 55, "class table");

// ------------------------------------------------------------------ class tables ---
static_assert(CQG_GEN_MAXL == CQG_MAXL, "generated ERI code must match CQG_MAXL");
static const int kPairClass[10][2] = {{0, 0}, {1, 0}, {1, 1}, {2, 0}, {2, 1}, {2, 2},
                                      {3, 0}, {3, 1}, {3, 2}, {3, 3}};
static inline int pair_class_of(int la, int lb) {  // la >= lb
  return la * (la + 1) / 2 + lb;
}
static inline int nfun(int l) { return l > 1 ? 2 * l + 1 : (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int nfun_c(int l) { return l > 1 ? 2 * l + 1 : (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int ncart_c(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int nherm_c(int n) { return (n + 1) * (n + 2) * (n + 3) / 6; }

// Members a sibling group of a pair class holds at most (larger families are split into
// groups of this size): s-s pairs 4 (two s shells of one contraction on each centre, or the
// three distinct pairs of one centre's two), p-s and d-s pairs 2, every other class 1 (not
// grouped: the classes whose sibling pairs keep one orientation, L_a > L_b, or are
// symmetric in a and b, s-s).
__host__ __device__ constexpr int sibling_cap(int la, int lb) {
  return (la == 0 && lb == 0) ? 4 : ((la == 1 || la == 2) && lb == 0) ? 2 : 1;
}

// Sibling-group quartet classes (generated sibling form EriClassGC<.., MB, MK>, MB and MK
// the member caps of the bra and ket pair classes).
template <int LA, int LB, int LC, int LD>
struct EriGroup {
  static constexpr bool ok = false;
  static constexpr int MB = 1, MK = 1;
};
#define CQG_GC_TRAIT(A, B, C, D, MB_, MK_)                                                            \
  template <>                                                                                       \
  struct EriGroup<A, B, C, D> {                                                                     \
    static constexpr bool ok = true;                                                                \
    static constexpr int MB = MB_, MK = MK_;                                                        \
    static_assert(MB_ == sibling_cap(A, B) && MK_ == sibling_cap(C, D), "member caps of the class"); \
  };
CQG_GC_EACH(CQG_GC_TRAIT)
#undef CQG_GC_TRAIT

__host__ __device__ constexpr int pair_class_c(int la, int lb) { return la * (la + 1) / 2 + lb; }
// quartet class index (bra pair class i >= ket pair class j, k = i(i+1)/2 + j)
__host__ __device__ constexpr int qclass_index(int la, int lb, int lc, int ld) {
  return pair_class_c(la, lb) * (pair_class_c(la, lb) + 1) / 2 + pair_class_c(lc, ld);
}

// quartet class k <-> (bra pair class i, ket pair class j), i >= j, k = i(i+1)/2 + j
static inline void qclass_split(int k, int &i, int &j) {
  i = 0;
  while ((i + 1) * (i + 2) / 2 <= k) ++i;
  j = k - i * (i + 1) / 2;
}

// ------------------------------------------------------------------ device data ---
struct Shells {
  const double3 *center;
  const int *bf;     // first basis function of the shell within its molecule
  const int *mol;    // molecule of the shell
  // the shell's functions in the internal order of the per-thread classes: component k is
  // function pf.x + k pf.y of its molecule.  Shells of one angular momentum are together,
  // component by component: the lanes of a warp hold kets of one class at one bra, and their
  // exchange blocks X(c, a), Gh(c, a) then lie in a few lines of column a (for (H2O)_32 cc-pVDZ,
  // 8 for a p component instead of up to 32 of the 48 of a column)
  const int2 *pf;
};

// Per-molecule layout: a context holds nmol >= 1 molecules (a batch).  Matrices of
// molecule m are packed at offset xoff[m] with leading dimension nbf[m]; with a single
// molecule the caller's matrices are used in place (xoff[0] = 0, leading dimension ldx).
struct Mols {
  int nmol;
  const int *shoff;              // first (global) shell of molecule m
  const int *nsh;                // shells of molecule m
  const long long *Moff;         // offset of molecule m's nsh_m x nsh_m block-norm matrix
  const long long *xoff;         // offset of molecule m's matrices in packed storage
  const int *nbf;                // basis functions of molecule m
  const int *foff;               // basis functions of the molecules before m
  const int *pos;                // [foff[m] + r]: internal position of function r (Shells.pf)
  const int *fsh;                // [foff[m] + r]: shell of function r within the molecule
  // [Moff[m] + y + x nsh]: pair index of shells (x, y) of molecule m in their internal
  // orientation, -1 for the other order
  const int *pidx;
  const unsigned char *active;   // molecule m takes part in the call
  const int *molbk;              // [m][ket pair class][bucket + 1]: first pair of each bucket
  const int *molgbk;             // the same in group index space: first group of each bucket
};
struct Pairs {
  const int2 *sh;       // (shell a, shell b), internal orientation L_a >= L_b
  const double *Q;      // Schwarz bound
  const int *poff;      // first primitive pair
  const int *np;        // number of primitive pairs (after primitive screening)
  const int *kk;        // nprim(a) * nprim(b) of the contracted shells (model count)
  const PrimPair *prim;
  const double2 *cols;  // the same primitive pairs in blocked columns (PrimCols): pair i's are
  const int *coff;      // column i % 32 of the rows from coff[i]
  // Sibling groups: pairs whose shells have the same centres, angular momenta and
  // exponents (segmented copies of one general contraction) and differ only in their
  // contraction coefficients.  The members of a group are consecutive pairs, led by the
  // first.  Group g (group index space, in pair order) is led by pair glead[g]; gQ[g] is
  // the largest Q of its members and Qc[i] that of pair i's group (non-increasing within a
  // primitive bucket, so it serves the coarse range searches).
  const double *Qc;
  const int *glead;
  const double *gQ;
  // Per pair (meaningful for leaders): gsz members (0 for the other members), and the
  // group's unit-coefficient primitive pairs gprim[gpoff .. gpoff + gnp) (the union of the
  // members' screened primitive pairs) with the members' coefficient products
  // gw[gwoff + m * gnp + i], m < the member cap of the pair class (zero rows past gsz).
  const int *gsz;
  const int *gpoff;
  const int *gnp;
  const int *gwoff;
  const PrimPair *gprim;
  const double *gw;
  // Member masks of the sibling-group list entries (bit 4 i + j: bra member i with ket
  // member j), parallel to the quartet list.
  const unsigned short *qmask;
};
struct DigestGroups {
  const double *X[CQG_MAXG];
  double *G[CQG_MAXG];
  double sJ[CQG_MAXG];
  double sK[CQG_MAXG];
  int ng;
  int ldx;                        // leading dimension of X when nmol == 1
  int batch;                      // matrices are packed per molecule (Mols.xoff / nbf)
  const long long *xoff;
  const int *nbf;
  // for the per-thread classes: X and Gh in the internal order (leading dimension nbf), and the
  // Coulomb blocks by shell pair, component k of pair i of class c at joff[c] + k jn[c] + i -
  // jbeg[c]: the kets of a warp are nearly consecutive pairs
  const double *XP[CQG_MAXG];
  double *GP[CQG_MAXG];
  const double *DP[CQG_MAXG];
  double *JP[CQG_MAXG];
  long long joff[CQG_NPC];
  int jn[CQG_NPC], jbeg[CQG_NPC];
};

// base pointers and leading dimensions of molecule m's X and Gh
__device__ __forceinline__ void mol_view(const DigestGroups &dg, int g, int m, const double *&X, double *&G,
                                         size_t &ldx, size_t &ldg) {
  if (dg.batch) {
    const long long o = dg.xoff[m];
    X = dg.X[g] + o;
    G = dg.G[g] + o;
    ldx = ldg = (size_t)dg.nbf[m];
  } else {
    X = dg.X[g];
    G = dg.G[g];
    ldx = dg.ldx;
    ldg = (size_t)dg.nbf[0];
  }
}

// ------------------------------------------------------------------ kernels ---
// Schwarz: Q(ab) = sqrt(max_ij |(ij|ij)|) for pairs [beg, end) of one class, 2^ls lanes per
// pair, each with a share of the bra's primitive pairs.
template <int LA, int LB>
__global__ void __launch_bounds__(128) k_schwarz(Pairs P, Shells S, const double *__restrict__ boys_g,
                                                 int beg, int end, int ls, double *__restrict__ Qout) {
  __shared__ __align__(16) double boys[boys_rows_size(2 * (LA + LB))];
  load_boys<2 * (LA + LB)>(boys_g, boys);
  __syncthreads();
  const int t = blockIdx.x * blockDim.x + threadIdx.x, sub = t & ((1 << ls) - 1);
  const int i = min(beg + (t >> ls), end - 1);
  constexpr int NA = nfun_c(LA), NB = nfun_c(LB), NAB = NA * NB;
  int2 s = P.sh[i];
  double3 A = S.center[s.x], B = S.center[s.y];
  double out[NAB * NAB];
  const PrimPair *pp = P.prim + P.poff[i];
  const int np = P.np[i], b0 = (np * sub) >> ls, b1 = (np * (sub + 1)) >> ls;
  EriClass<LA, LB, LA, LB>::template run<double>(pp + b0, b1 - b0, pp, np, A, B, A, B, boys, out);
  double mx = 0.0;
#pragma unroll
  for (int ij = 0; ij < NAB; ++ij) {
    double v = out[ij * NAB + ij];
    for (int o = (1 << ls) >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    mx = fmax(mx, fabs(v));
  }
  if (sub == 0 && beg + (t >> ls) < end) Qout[i] = sqrt(mx);
}

// Block norms M(s1,s2) = max over matrices of max|X_i(block)|, and input checks.
struct XList {
  const double *X[8];
  double *P[8];   // the same in the internal order (Shells.pf), written here
  int n;
};
// Thread (s1, s2) of molecule blockIdx.z: the block of rows s1, columns s2.  Besides the norm
// and the checks it writes everything a call reads of the block later: the matrices in the
// internal order, and where (s2, s1) is a shell pair, the pair's norm and Coulomb blocks.
static __global__ void k_blocknorm(XList xl, int ldx, Mols mols, Shells S, const int *__restrict__ sz,
                                   const int *__restrict__ shL, double *__restrict__ M, double *__restrict__ MT,
                                   double *__restrict__ Mpair, DigestGroups dg, int *__restrict__ flags,
                                   double *__restrict__ Mmax, double sym_tol) {
  const int mol = blockIdx.z;
  const int nsh = mols.nsh[mol];
  const int s1 = blockIdx.x * blockDim.x + threadIdx.x;
  const int s2 = blockIdx.y;
  if (s2 >= nsh) return;   // whole blocks
  double mx = 0.0;
  if (s1 < nsh) {
    double *Mm = M + mols.Moff[mol], *MTm = MT + mols.Moff[mol];
    const int pair = mols.pidx[mols.Moff[mol] + s1 + (size_t)s2 * nsh];
    if (mols.active[mol]) {
      const int g1 = mols.shoff[mol] + s1, g2 = mols.shoff[mol] + s2;
      const int r0 = S.bf[g1], c0 = S.bf[g2], nr = sz[g1], nc = sz[g2], n = mols.nbf[mol];
      if (mols.nmol > 1) ldx = n;
      const long long xo = mols.nmol > 1 ? mols.xoff[mol] : 0;
      const int2 p1 = S.pf[g1], p2 = S.pf[g2];
      int bad = 0, asym = 0;
      for (int m = 0; m < xl.n; ++m) {
        const double *X = xl.X[m] + xo;
        double *P = xl.P[m] + xo;
        for (int c = 0; c < nc; ++c)
          for (int r = 0; r < nr; ++r) {
            double v = X[(size_t)(r0 + r) + (size_t)(c0 + c) * ldx];
            double t = X[(size_t)(c0 + c) + (size_t)(r0 + r) * ldx];
            if (!isfinite(v)) bad = 1;
            double av = fabs(v);
            mx = fmax(mx, av);
            if (fabs(v - t) > sym_tol * fmax(1.0, av)) asym = 1;
            P[(size_t)(p1.x + r * p1.y) + (size_t)(p2.x + c * p2.y) * n] = v;
          }
      }
      if (bad) atomicOr(flags + 0, 1);
      if (asym) atomicOr(flags + 1, 1);
      if (pair >= 0) {   // a = s2 (columns), b = s1 (rows)
        const int cls = pair_class_c(shL[g2], shL[g1]);
        for (int g = 0; g < dg.ng; ++g) {
          if (dg.sJ[g] == 0.0) continue;
          const double *X = dg.X[g] + xo;
          double *D = const_cast<double *>(dg.DP[g]) + dg.joff[cls] + (pair - dg.jbeg[cls]);
          for (int c = 0; c < nc; ++c)
            for (int r = 0; r < nr; ++r)
              D[(size_t)(c * nr + r) * dg.jn[cls]] = X[(size_t)(r0 + r) + (size_t)(c0 + c) * ldx];
        }
      }
    }
    Mm[(size_t)s1 + (size_t)s2 * nsh] = mx;
    MTm[(size_t)s2 + (size_t)s1 * nsh] = mx;   // transposed copy: M(s1, .) as a contiguous column
    if (pair >= 0) Mpair[pair] = mx;
  }
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  // non-negative doubles order like their bit patterns
  if ((threadIdx.x & 31) == 0 && mx > 0.0)
    atomicMax((unsigned long long *)Mmax, (unsigned long long)__double_as_longlong(mx));
}

// One screening task = (class block, bra pair).  Blocks are listed in task order.
struct BlockTable {
  int nblk;
  int task_beg[CQG_NQC + 1];   // first task of each block
  int bra_beg[CQG_NQC];        // first bra pair (global index) of the block
  int ket_beg[CQG_NQC];        // first ket pair (global index) of the block
  int ket_n[CQG_NQC];          // number of ket pairs of the block's ket class
  int diag[CQG_NQC];           // bra class == ket class
  int ket_class[CQG_NQC];      // pair class of the ket
  int grouped[CQG_NQC];        // tasks are bra sibling groups
  int gbra_beg[CQG_NQC];       // first bra group (group index) of a grouped block
  int min_members[CQG_NQC];    // grouped: member quartets a sibling entry holds at least
};

__device__ __forceinline__ int find_block(const BlockTable &bt, int task) {
  int b = 0;
  while (b + 1 < bt.nblk && bt.task_beg[b + 1] <= task) ++b;
  return b;
}

// number of ket pairs (from the start of the Q-descending ket list) that can pass
__device__ __forceinline__ int coarse_range(const double *__restrict__ Q, int kb, int kn, double cut) {
  // first index with Q < cut
  int lo = 0, hi = kn;
  while (lo < hi) {
    int mid = (lo + hi) >> 1;
    if (Q[kb + mid] >= cut) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Density-weighted Schwarz bound of a quartet: max of the six shell-block norms of the
// density times Q_ab Q_cd (contract.h:112-131).  The four norms that pair a bra shell with
// a ket shell are read from the transposed copy MT, where M(s1, .) and M(s2, .) are the
// contiguous columns s1 and s2 (one pair of columns per bra pair, so they stay in L1);
// m12 = M(s1, s2) is the bra's own, the same for every ket, and mcd = M(s3, s4) the ket's
// own, read from the per-pair copy Mpair (consecutive kets: a coalesced load).
__device__ __forceinline__ double quartet_bound(const double *__restrict__ col1, const double *__restrict__ col2,
                                                double m12, double mcd, int shoff, int2 cd, double qab, double qcd) {
  const int s3 = cd.x - shoff, s4 = cd.y - shoff;
  double m = fmax(m12, col1[s4]);
  m = fmax(m, col2[s4]);
  m = fmax(m, mcd);
  m = fmax(m, col1[s3]);
  m = fmax(m, col2[s3]);
  return m * qab * qcd;
}

// Per-block screening tallies in blkacc[kBlkAcc * blk + ...]: model primitive quartets
// (sum of Ka Kb Kc Kd) and executed primitive quartets of the FP64 and FP32 lists, then the
// number of contracted quartets of each (a sibling-group entry holds several).
constexpr int kBlkAcc = 6;

// The quartet list is laid out by virtual task v = part * ntask + task, part 0 / 1 = the
// FP64 / FP32 pair entries (one quartet each), part 2 / 3 = the FP64 / FP32 sibling-group
// entries; work list vb = part * CQG_NQC + class is the range of one part of one class.
constexpr int kListParts = 4;
#define CQG_NLIST (kListParts * CQG_NQC)
constexpr int kRangeThreads = 256;   // k_block_ranges: one thread per work list
static_assert(CQG_NLIST <= kRangeThreads, "k_block_ranges needs a thread per work list");

// exclusive prefix sum over the warp's lanes and the warp's total
__device__ __forceinline__ unsigned warp_excl_scan(unsigned x, unsigned &total) {
  const int lane = threadIdx.x & 31;
  unsigned v = x;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  total = __shfl_sync(0xffffffffu, v, 31);
  return v - x;
}

// Count (FILL=false) or write (FILL=true) the passing quartets of each task.  One warp
// per task; ket pairs scanned in ascending order, survivors compacted in lane order so the
// list is deterministic.  Quartets whose bound is below `cut32` go to the FP32 parts; the
// rest to the FP64 parts.  Counts cnt[v], offsets off[v] per virtual task v.
//
// In a grouped block a task is one bra sibling group and each lane takes one ket group:
// every member quartet (bra member i, ket member j) gets the exact test above.  A pair of
// groups with at least bt.min_members[blk] member quartets becomes one sibling entry (bra
// leader, ket leader) per precision, with the mask of its members that passed at that
// precision; the members of a smaller pair of groups become pair entries of their own.  So
// the contracted quartets, their count and their precision are those of the pair-level
// lists.  In a diagonal block (bra class = ket class) ket group <= bra group, and within one
// group ket member <= bra member, so every unordered pair of pairs is taken once.
//
// Tasks take the class's bra pairs (groups) from the last: the pairs are ordered by
// primitive-count bucket, so each class list starts with its heaviest quartets and the
// work queues hand out the light ones at the end of a launch.
struct ScreenTally {
  unsigned long long km64 = 0, ke64 = 0, km32 = 0, ke32 = 0, nq64 = 0, nq32 = 0;
};

// Survivor-mask cache between the two screening passes: the count pass stores, per task and
// per 32-ket step, the FP64 and FP32 survivor ballots (one uint2) at the task's slot in
// `masks`; the fill pass reads them instead of testing the bounds again.  A task whose
// steps do not fit in the buffer gets slot -1 and the fill pass tests its bounds itself.
static_assert(CQG_NBUCKET <= 32, "screen_pair_task searches one bucket per lane");
constexpr long long kMaskStepsInitial = 1ll << 22;   // 32 MiB; grown to what a call used
constexpr long long kMaskStepsMax = 1ll << 28;       // 2 GiB
struct MaskCache {
  uint2 *masks;
  unsigned long long *head;   // next free step (zeroed before the count pass)
  long long *slot;            // per task: first step, or -1
  long long cap;              // steps the buffer holds
};

template <bool FILL>
__device__ __forceinline__ void screen_pair_task(const BlockTable &bt, int blk, int t, int task, const Pairs &P,
                                                 const double *__restrict__ M, const double *__restrict__ MT,
                                                 const double *__restrict__ Mpair, const Mols &mols,
                                                 const int *__restrict__ shmol, double mm, double thresh,
                                                 double cut32, const bool (&dop)[kListParts],
                                                 const long long (&base)[kListParts], long long (&cpart)[kListParts],
                                                 uint2 *__restrict__ qlist, long long cap, const MaskCache &mc,
                                                 ScreenTally &ty) {
  const int lane = threadIdx.x & 31;
  const int bra = bt.bra_beg[blk] + t;
  const double qb = P.Q[bra];
  if (!(qb * mm > 0.0)) {
    if (!FILL && lane == 0) mc.slot[task] = -1;
    return;
  }
  const double cut = thresh / (qb * mm) * (1.0 - 1e-12);
  const int2 ab = P.sh[bra];
  const int mol = shmol[ab.x];
  if (!mols.active[mol]) {
    if (!FILL && lane == 0) mc.slot[task] = -1;
    return;
  }
  const int nsh = mols.nsh[mol], shoff = mols.shoff[mol];
  const double *Mm = M + mols.Moff[mol];
  const double *col1 = MT + mols.Moff[mol] + (size_t)(ab.x - shoff) * nsh;
  const double *col2 = MT + mols.Moff[mol] + (size_t)(ab.y - shoff) * nsh;
  const double m12 = Mm[(ab.x - shoff) + (size_t)(ab.y - shoff) * nsh];
  const int *bkt = mols.molbk + ((size_t)mol * CQG_NPC + bt.ket_class[blk]) * (CQG_NBUCKET + 1);
  const unsigned long long kkb = (unsigned long long)P.kk[bra], npb = (unsigned long long)P.np[bra];
  const unsigned below = (1u << lane) - 1u;
  // coarse range of every bucket at once: lane b < CQG_NBUCKET searches bucket b
  int my_kb = 0, my_kend = 0;
  if (lane < CQG_NBUCKET) {
    const int kb = bkt[lane], ke = bkt[lane + 1];
    int kend = kb;
    if (ke > kb) {
      kend = kb + coarse_range(P.Qc, kb, ke - kb, cut);
      if (bt.diag[blk]) kend = min(kend, bra + 1);   // unique pairs of pairs: ket <= bra
    }
    my_kb = kb;
    my_kend = max(kend, kb);
  }
  // the task's slot in the mask cache: the count pass reserves one step per 32 kets
  long long slot = -1;
  if (!FILL) {
    unsigned steps;
    warp_excl_scan((unsigned)((my_kend - my_kb + 31) >> 5), steps);
    if (lane == 0) {
      if (steps > 0) {
        const unsigned long long s0 = atomicAdd(mc.head, (unsigned long long)steps);
        slot = (long long)(s0 + steps) <= mc.cap ? (long long)s0 : -1;
      }
      mc.slot[task] = slot;
    }
    slot = __shfl_sync(0xffffffffu, slot, 0);
  } else {
    slot = mc.slot[task];
  }
  long long step = 0;
  for (int bk = 0; bk < CQG_NBUCKET; ++bk) {
    const int kb = __shfl_sync(0xffffffffu, my_kb, bk), kend = __shfl_sync(0xffffffffu, my_kend, bk);
    for (int k0 = kb; k0 < kend; k0 += 32, ++step) {
      const int ket = k0 + lane;
      unsigned b64, b32;
      if (FILL && slot >= 0) {   // survivors from the count pass
        const uint2 m = mc.masks[slot + step];
        b64 = m.x;
        b32 = m.y;
      } else {
        bool hi = false, lo = false;
        if (ket < kend) {
          const double bnd = quartet_bound(col1, col2, m12, Mpair[ket], shoff, P.sh[ket], qb, P.Q[ket]);
          const bool pass = bnd >= thresh;
          lo = pass && bnd < cut32;
          hi = pass && !lo;
        }
        b64 = __ballot_sync(0xffffffffu, hi);
        b32 = __ballot_sync(0xffffffffu, lo);
        if (!FILL && slot >= 0 && lane == 0) mc.masks[slot + step] = make_uint2(b64, b32);
      }
      const bool hi = (b64 >> lane) & 1u, lo = (b32 >> lane) & 1u;
      if (FILL) {
        if (hi && dop[0]) {
          const long long pos = base[0] + cpart[0] + __popc(b64 & below);
          if (pos < cap) qlist[pos] = make_uint2((unsigned)bra, (unsigned)ket);
        }
        if (lo && dop[1]) {
          const long long pos = base[1] + cpart[1] + __popc(b32 & below);
          if (pos < cap) qlist[pos] = make_uint2((unsigned)bra, (unsigned)ket);
        }
      } else {
        if (hi) {
          ty.km64 += (unsigned long long)P.kk[ket];
          ty.ke64 += (unsigned long long)P.np[ket];
        }
        if (lo) {
          ty.km32 += (unsigned long long)P.kk[ket];
          ty.ke32 += (unsigned long long)P.np[ket];
        }
      }
      cpart[0] += __popc(b64);
      cpart[1] += __popc(b32);
    }
  }
  if (!FILL) {   // the bra's factors are common to the task's quartets
    ty.km64 *= kkb;
    ty.ke64 *= npb;
    ty.km32 *= kkb;
    ty.ke32 *= npb;
    ty.nq64 = (unsigned long long)cpart[0];
    ty.nq32 = (unsigned long long)cpart[1];
  }
}

template <bool FILL>
__device__ __forceinline__ void screen_group_task(const BlockTable &bt, int blk, int t, const Pairs &P,
                                                  const double *__restrict__ MT, const double *__restrict__ Mpair,
                                                  const Mols &mols, const int *__restrict__ shmol, double mm,
                                                  double thresh, double cut32, const bool (&dop)[kListParts],
                                                  const long long (&base)[kListParts],
                                                  long long (&cpart)[kListParts], uint2 *__restrict__ qlist,
                                                  unsigned short *__restrict__ qmask, long long cap,
                                                  ScreenTally &ty) {
  const int lane = threadIdx.x & 31;
  const int gbra = bt.gbra_beg[blk] + t;
  const int bra = P.glead[gbra];
  const int mb = P.gsz[bra];
  const int min_members = bt.min_members[blk];
  const double qb = P.gQ[gbra];
  if (!(qb * mm > 0.0)) return;
  const double cut = thresh / (qb * mm) * (1.0 - 1e-12);
  const double tcut = thresh * (1.0 - 1e-12);   // margin for the rounding of the Q products
  const int mol = shmol[P.sh[bra].x];
  if (!mols.active[mol]) return;
  const int nsh = mols.nsh[mol], shoff = mols.shoff[mol];
  const double *MTm = MT + mols.Moff[mol];
  const int *bkt = mols.molgbk + ((size_t)mol * CQG_NPC + bt.ket_class[blk]) * (CQG_NBUCKET + 1);
  const unsigned below = (1u << lane) - 1u;
  for (int bk = 0; bk < CQG_NBUCKET; ++bk) {
    const int kb = bkt[bk], ke = bkt[bk + 1];
    if (ke <= kb) continue;
    int kend = kb + coarse_range(P.gQ, kb, ke - kb, cut);
    if (bt.diag[blk]) kend = min(kend, gbra + 1);   // ket group <= bra group
    for (int k0 = kb; k0 < kend; k0 += 32) {
      const int kx = k0 + lane;   // ket group
      int ket = 0;
      unsigned m64 = 0, m32 = 0;  // member masks, bit 4 i + j
      bool sib = false;
      if (kx < kend) {
        ket = P.glead[kx];
        const int mk = P.gsz[ket];
        const bool same = bt.diag[blk] && kx == gbra;
        sib = mb * mk > 1 && (same ? mb * (mb + 1) / 2 : mb * mk) >= min_members;
        const double qk = P.gQ[kx];
        for (int i = 0; i < mb; ++i) {
          const int bi = bra + i;
          const double qi = P.Q[bi];
          // the bound of each member quartet is at most Mmax Q_i Q_j: skip the six norms where
          // that already falls short (the groups' coarse range holds their largest Q)
          if (qi * qk * mm < tcut) continue;
          const int2 abi = P.sh[bi];
          const double *c1 = MTm + (size_t)(abi.x - shoff) * nsh;
          const double *c2 = MTm + (size_t)(abi.y - shoff) * nsh;
          const double mi = Mpair[bi];
          const int jmax = same ? min(mk, i + 1) : mk;
          for (int j = 0; j < jmax; ++j) {
            const int kj = ket + j;
            const double qj = P.Q[kj];
            if (qi * qj * mm < tcut) continue;
            const double bnd = quartet_bound(c1, c2, mi, Mpair[kj], shoff, P.sh[kj], qi, qj);
            if (bnd < thresh) continue;
            const unsigned bit = 1u << (4 * i + j);
            if (bnd < cut32) m32 |= bit; else m64 |= bit;
            if (!FILL) {
              const unsigned long long kq = (unsigned long long)P.kk[bi] * (unsigned long long)P.kk[kj];
              // executed primitive quartets of a member quartet evaluated on its own
              const unsigned long long eq =
                  sib ? 0ull : (unsigned long long)P.np[bi] * (unsigned long long)P.np[kj];
              if (bnd < cut32) {
                ty.km32 += kq;
                ty.ke32 += eq;
              } else {
                ty.km64 += kq;
                ty.ke64 += eq;
              }
            }
          }
        }
        if (!FILL) {
          if (sib) {   // a sibling entry evaluates the groups' shared primitive pairs once
            const unsigned long long gq = (unsigned long long)P.gnp[bra] * (unsigned long long)P.gnp[ket];
            if (m64) ty.ke64 += gq;
            if (m32) ty.ke32 += gq;
          }
          ty.nq64 += (unsigned long long)__popc(m64);
          ty.nq32 += (unsigned long long)__popc(m32);
        }
      }
      // pair entries (one per member quartet) of parts 0 and 1: several per lane
      const unsigned n0 = sib ? 0u : (unsigned)__popc(m64), n1 = sib ? 0u : (unsigned)__popc(m32);
      unsigned t0, t1;
      const unsigned e0 = warp_excl_scan(n0, t0), e1 = warp_excl_scan(n1, t1);
      // sibling entries of parts 2 and 3: at most one per lane
      const unsigned b2 = __ballot_sync(0xffffffffu, sib && m64), b3 = __ballot_sync(0xffffffffu, sib && m32);
      if (FILL) {
#pragma unroll
        for (int p = 0; p < 2; ++p) {
          unsigned m = p == 0 ? (sib ? 0u : m64) : (sib ? 0u : m32);
          if (!m || !dop[p]) continue;
          long long pos = base[p] + cpart[p] + (p == 0 ? e0 : e1);
          while (m) {   // member quartets in bit order
            const int bit = __ffs(m) - 1;
            m &= m - 1;
            if (pos < cap) qlist[pos] = make_uint2((unsigned)(bra + (bit >> 2)), (unsigned)(ket + (bit & 3)));
            ++pos;
          }
        }
        if (sib && m64 && dop[2]) {
          const long long pos = base[2] + cpart[2] + __popc(b2 & below);
          if (pos < cap) {
            qlist[pos] = make_uint2((unsigned)bra, (unsigned)ket);
            qmask[pos] = (unsigned short)m64;
          }
        }
        if (sib && m32 && dop[3]) {
          const long long pos = base[3] + cpart[3] + __popc(b3 & below);
          if (pos < cap) {
            qlist[pos] = make_uint2((unsigned)bra, (unsigned)ket);
            qmask[pos] = (unsigned short)m32;
          }
        }
      }
      cpart[0] += t0;
      cpart[1] += t1;
      cpart[2] += __popc(b2);
      cpart[3] += __popc(b3);
    }
  }
}

// Four CTAs of 256 threads per SM (64 registers; a few bytes of spills): the latency-bound
// screening runs 3.54 -> 3.02 ms per (H2O)_32 build against three CTAs at 80 registers.
template <bool FILL>
__global__ void __launch_bounds__(256, 4) k_quartets(BlockTable bt, int ntask, Pairs P, const double *__restrict__ M,
                                                  const double *__restrict__ MT, const double *__restrict__ Mpair,
                                                  Mols mols, const int *__restrict__ shmol,
                                                  const double *__restrict__ Mmax, double thresh,
                                                  double cut32, long long *__restrict__ cnt,
                                                  const long long *__restrict__ off, uint2 *__restrict__ qlist,
                                                  unsigned short *__restrict__ qmask,
                                                  unsigned long long *__restrict__ blkacc, long long vt0,
                                                  long long vt1, long long obase, long long cap, MaskCache mc) {
  const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (warp >= ntask) return;
  // fill pass: only the parts (virtual tasks part * ntask + warp) inside the chunk
  bool dop[kListParts];
  bool any = false;
#pragma unroll
  for (int p = 0; p < kListParts; ++p) {
    const long long v = (long long)p * ntask + warp;
    dop[p] = !FILL || (v >= vt0 && v < vt1);
    any = any || dop[p];
  }
  if (FILL && !any) return;
  const int blk = find_block(bt, warp);
  const int t = bt.task_beg[blk + 1] - 1 - warp;   // heaviest bra first
  long long base[kListParts], cpart[kListParts];
#pragma unroll
  for (int p = 0; p < kListParts; ++p) {
    base[p] = FILL ? off[(long long)p * ntask + warp] - obase : 0;
    cpart[p] = 0;
  }
  ScreenTally ty;
  const double mm = *Mmax;
  if (bt.grouped[blk])
    screen_group_task<FILL>(bt, blk, t, P, MT, Mpair, mols, shmol, mm, thresh, cut32, dop, base, cpart, qlist,
                            qmask, cap, ty);
  else
    screen_pair_task<FILL>(bt, blk, t, warp, P, M, MT, Mpair, mols, shmol, mm, thresh, cut32, dop, base, cpart,
                           qlist, cap, mc, ty);
  if (!FILL) {
    for (int o = 16; o > 0; o >>= 1) {
      ty.km64 += __shfl_xor_sync(0xffffffffu, ty.km64, o);
      ty.ke64 += __shfl_xor_sync(0xffffffffu, ty.ke64, o);
      ty.km32 += __shfl_xor_sync(0xffffffffu, ty.km32, o);
      ty.ke32 += __shfl_xor_sync(0xffffffffu, ty.ke32, o);
    }
    if (bt.grouped[blk]) {   // pair tasks count whole warps already
      for (int o = 16; o > 0; o >>= 1) {
        ty.nq64 += __shfl_xor_sync(0xffffffffu, ty.nq64, o);
        ty.nq32 += __shfl_xor_sync(0xffffffffu, ty.nq32, o);
      }
    }
    if (lane == 0) {
#pragma unroll
      for (int p = 0; p < kListParts; ++p) cnt[(long long)p * ntask + warp] = cpart[p];
      unsigned long long *acc = blkacc + kBlkAcc * blk;
      if (ty.nq64) {
        atomicAdd(acc + 0, ty.km64);
        atomicAdd(acc + 1, ty.ke64);
        atomicAdd(acc + 4, ty.nq64);
      }
      if (ty.nq32) {
        atomicAdd(acc + 2, ty.km32);
        atomicAdd(acc + 3, ty.ke32);
        atomicAdd(acc + 5, ty.nq32);
      }
    }
  }
}

// Ranges [beg, end) of the quartet list per work list vb = part * nblk + block from the
// per-task counts and offsets (virtual task part * ntask + task).
static __global__ void k_block_ranges(BlockTable bt, int ntask, const long long *__restrict__ cnt,
                               const long long *__restrict__ off, long long *__restrict__ range, long long cap,
                               int *__restrict__ flags) {
  int vb = threadIdx.x;
  const long long nv = (long long)kListParts * ntask;
  if (vb == 0 && ntask > 0 && off[nv - 1] + cnt[nv - 1] > cap) flags[2] = 1;   // list overflow
  if (vb >= kListParts * bt.nblk) return;
  const int part = vb / bt.nblk, b = vb % bt.nblk;
  const long long t0 = (long long)part * ntask + bt.task_beg[b], t1 = (long long)part * ntask + bt.task_beg[b + 1];
  long long beg = 0, end = 0;
  if (t1 > t0) {
    beg = off[t0];
    end = off[t1 - 1] + cnt[t1 - 1];
  } else if (t0 > 0) {
    beg = end = off[t0 - 1] + cnt[t0 - 1];
  }
  range[2 * vb] = min(beg, cap);
  range[2 * vb + 1] = min(end, cap);
}

// The scan of the counts and the ranges by one block, for lists of few tasks (one launch
// instead of the three of the device-wide scan).
constexpr int kScanThreads = 1024, kScanMax = 32 * kScanThreads;
static __global__ void __launch_bounds__(kScanThreads) k_scan_ranges(BlockTable bt, int ntask,
                                                                     const long long *__restrict__ cnt,
                                                                     long long *off, long long *__restrict__ range,
                                                                     long long cap, int *__restrict__ flags) {
  __shared__ long long part[32];
  const int nv = kListParts * ntask, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (nv + kScanThreads - 1) / kScanThreads, v0 = min(nv, (int)threadIdx.x * per), v1 = min(nv, v0 + per);
  long long sum = 0;
  for (int v = v0; v < v1; ++v) sum += cnt[v];
  long long inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const long long y = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += y;
  }
  if (lane == 31) part[warp] = inc;
  __syncthreads();
  long long before = inc - sum;
  for (int w = 0; w < warp; ++w) before += part[w];
  for (int v = v0; v < v1; ++v) {
    off[v] = before;
    before += cnt[v];
  }
  __syncthreads();   // block-wide: the offsets written above are read below
  const int vb = threadIdx.x;
  if (vb == 0 && ntask > 0 && off[nv - 1] + cnt[nv - 1] > cap) flags[2] = 1;   // list overflow
  if (vb >= kListParts * bt.nblk) return;
  const int p = vb / bt.nblk, b = vb % bt.nblk;
  const int t0 = p * ntask + bt.task_beg[b], t1 = p * ntask + bt.task_beg[b + 1];
  long long beg = 0, end = 0;
  if (t1 > t0) {
    beg = off[t0];
    end = off[t1 - 1] + cnt[t1 - 1];
  } else if (t0 > 0) {
    beg = end = off[t0 - 1] + cnt[t0 - 1];
  }
  range[2 * vb] = min(beg, cap);
  range[2 * vb + 1] = min(end, cap);
}

__device__ __forceinline__ double warp_sum(double x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// J/K digest of one quartet (contract.h:145-171), half of the updates:
//   COULOMB : Gh(a,b) += sJ sum_cd X(d,c) v ;  Gh(c,d) += sJ sum_ab X(b,a) v
//   EXCHANGE: Gh(a,c) += sK X(b,d) v ; Gh(b,d) += sK X(a,c) v ; Gh(a,d) += sK X(b,c) v ;
//             Gh(b,c) += sK X(a,d) v
// with v = (ab|cd) * degeneracy, sK = 0.5 * scale_K; the other half is Gh^T (added in
// k_finalize).  All lanes of the warp call this; `valid` lanes hold a quartet, and when
// every lane shares the bra pair (`bra_uniform`) the Gh(a,b) sums are reduced across the
// warp before one atomic per element.
// Exchange updates go to Gh(c, a), Gh(d, b), Gh(d, a), Gh(c, b) and X is read in the same
// orientation (both are symmetric in the end, k_finalize adds (Gh + Gh^T) / 2), so the bra
// index, the same across a bra-uniform warp, is the column.  What bounds this part is the
// number of lines a warp's loads and atomics touch: hence the internal order of X and Gh and
// the Coulomb blocks by pair: (ps|ps) 5.69 -> 4.69 ms, (pp|ps) 4.20 -> 3.83, (ds|ps) 3.44 -> 3.00
// per (H2O)_32 cc-pVDZ build, before the stripes of eri_jk_list.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void digest(const double *v, double deg, int bra, int ket, const Pairs &P, const Shells &S,
                                       const DigestGroups &dg, bool valid, bool bra_uniform) {
  constexpr int NA = nfun_c(LA), NB = nfun_c(LB), NC = nfun_c(LC), ND = nfun_c(LD);
  constexpr int CB = pair_class_c(LA, LB), CK = pair_class_c(LC, LD);
  const int lane = threadIdx.x & 31;
  const int2 ab = P.sh[bra], cd = P.sh[ket];
  const int2 pa = S.pf[ab.x], pb = S.pf[ab.y], pc = S.pf[cd.x], pd = S.pf[cd.y];
  const int mol = dg.batch ? S.mol[ab.x] : 0;
  const size_t n = (size_t)dg.nbf[mol];
  const long long xo = dg.batch ? dg.xoff[mol] : 0;
  for (int g = 0; g < dg.ng; ++g) {
    const double sJ = dg.sJ[g] * deg;
    const double sK = 0.5 * dg.sK[g] * deg;
    if (dg.sJ[g] != 0.0) {
      const long long jb = dg.joff[CB] + (bra - dg.jbeg[CB]), jk = dg.joff[CK] + (ket - dg.jbeg[CK]);
      const int nb = dg.jn[CB], nk = dg.jn[CK];
      const double *__restrict__ D = dg.DP[g];
      double *J = dg.JP[g];
      double xdc[NC * ND], xba[NA * NB];
#pragma unroll
      for (int k = 0; k < NC * ND; ++k) xdc[k] = valid ? __ldg(D + jk + (long long)k * nk) : 0.0;
#pragma unroll
      for (int k = 0; k < NA * NB; ++k) xba[k] = valid ? __ldg(D + jb + (long long)k * nb) : 0.0;
#pragma unroll
      for (int k = 0; k < NA * NB; ++k) {
        double s = 0.0;
#pragma unroll
        for (int q = 0; q < NC * ND; ++q) s += xdc[q] * v[k * NC * ND + q];
        s *= sJ;
        if (bra_uniform) {
          s = warp_sum(s);
          if (lane == 0) atomicAdd(J + jb + (long long)k * nb, s);
        } else if (valid) {
          atomicAdd(J + jb + (long long)k * nb, s);
        }
      }
      if (valid) {
#pragma unroll
        for (int q = 0; q < NC * ND; ++q) {
          double s = 0.0;
#pragma unroll
          for (int k = 0; k < NA * NB; ++k) s += xba[k] * v[k * NC * ND + q];
          atomicAdd(J + jk + (long long)q * nk, sJ * s);
        }
      }
    }
    if (dg.sK[g] != 0.0 && valid) {
      // columns a and b, rows c and d, of X and Gh in the internal order
      const double *__restrict__ X = dg.XP[g] + xo;
      double *G = dg.GP[g] + xo;
      auto at = [&](int2 row, int r, int2 col, int c) {
        return (size_t)(row.x + r * row.y) + (size_t)(col.x + c * col.y) * n;
      };
      double xbd[NB * ND], xac[NA * NC], xbc[NB * NC], xad[NA * ND];
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int d = 0; d < ND; ++d) xbd[b * ND + d] = __ldg(X + at(pd, d, pb, b));
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int c = 0; c < NC; ++c) xac[a * NC + c] = __ldg(X + at(pc, c, pa, a));
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int c = 0; c < NC; ++c) xbc[b * NC + c] = __ldg(X + at(pc, c, pb, b));
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int d = 0; d < ND; ++d) xad[a * ND + d] = __ldg(X + at(pd, d, pa, a));
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          double s = 0.0;
#pragma unroll
          for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int d = 0; d < ND; ++d) s += xbd[b * ND + d] * v[((a * NB + b) * NC + c) * ND + d];
          atomicAdd(G + at(pc, c, pa, a), sK * s);
        }
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          double s = 0.0;
#pragma unroll
          for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int c = 0; c < NC; ++c) s += xac[a * NC + c] * v[((a * NB + b) * NC + c) * ND + d];
          atomicAdd(G + at(pd, d, pb, b), sK * s);
        }
#pragma unroll
      for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int d = 0; d < ND; ++d) {
          double s = 0.0;
#pragma unroll
          for (int b = 0; b < NB; ++b)
#pragma unroll
            for (int c = 0; c < NC; ++c) s += xbc[b * NC + c] * v[((a * NB + b) * NC + c) * ND + d];
          atomicAdd(G + at(pd, d, pa, a), sK * s);
        }
#pragma unroll
      for (int b = 0; b < NB; ++b)
#pragma unroll
        for (int c = 0; c < NC; ++c) {
          double s = 0.0;
#pragma unroll
          for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int d = 0; d < ND; ++d) s += xad[a * ND + d] * v[((a * NB + b) * NC + c) * ND + d];
          atomicAdd(G + at(pc, c, pb, b), sK * s);
        }
    }
  }
}

template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ int eri_jk_one(const uint2 *__restrict__ ql, long long i, long long wfirst, long long end,
                                          const Pairs &P, const Shells &S, const double *boys,
                                          const DigestGroups &dg, int ls);

// Per-thread class kernel: persistent grid over the class's quartet range; the Boys rows
// of this class are staged in shared memory once per block.  T is the arithmetic type of
// everything after the (FP64) Boys values; the digest accumulates in FP64.
// Threads per block of the per-thread class kernels (each block stages its own copy of the
// Boys rows in shared memory).  128 and 256 measure within 2 % of each other on (H2O)_32
// cc-pVDZ; 512 caps registers at 128 and spills in the p/d classes.
#ifndef CQG_ERI_THREADS
#define CQG_ERI_THREADS 128
#endif
constexpr int kEriThreads = CQG_ERI_THREADS;

// Work queue: the class's quartet range [beg, end) is consumed in chunks of `chunk`
// quartets (a multiple of 32), each claimed by one warp with an atomic add on the list's
// head counter qhead[blk] (zeroed before the launch), so warps that drew cheap quartets
// take more chunks instead of idling at the tail of a static split.
//
// A quartet's primitive quartets are a serial chain of its lane (64 x 64 of them for four
// 1s or 2s shells of oxygen: 0.25 ms), which bounds the launches that do not fill the GPU.
// So 2^ls lanes share a quartet:
//  - as many as a list shorter than a quarter of the GPU's lanes leaves for each (the other
//    classes' launches run beside it), and
//  - while the warp draws heavy bras, as many as bring a lane's share of bra x heaviest ket
//    to kLaneWork primitive quartets per quartet the list has for each lane: a longer chain
//    than that ends before the list does.  The bra is that of the list's first quartet, then
//    that of the warp's last chunk (lists are sorted heaviest bra first).
// Sharing has a price, fewer quartets per digest, so longer lists do without.  Measured:
// one water in 6-31G(d) 390 -> 259 us, O2 UHF cc-pVDZ 1120 -> 282 us, (H2O)_5 6-31G(d) 733 ->
// 626 us; with every list that leaves a lane idle shared, (H2O)_5 took 819 us.
struct LaneShare {
  int lanes;    // lanes the class can have resident on the GPU
  int nk_max;   // primitive pairs of the class's heaviest ket
};
constexpr int kLaneWork = 256;
// A long list is claimed in kStripes interleaved stripes: in plain order the whole GPU works on a
// handful of bras at a time, and the atomics of all warps meet in their few columns of Gh, in a
// few L2 slices.  (H2O)_32 cc-pVDZ build 47.6 -> 44.7 ms with 8 stripes, 45.0 with 32 or 128; the
// heaviest bras still come first within the first stripe.
constexpr unsigned kStripes = 8, kStripeMin = 1u << 13;
template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ void eri_jk_list(const uint2 *__restrict__ ql, const long long *__restrict__ range, int blk,
                                            const Pairs &P, const Shells &S, const double *__restrict__ boys_g,
                                            const DigestGroups &dg, unsigned long long *__restrict__ qhead,
                                            int chunk, LaneShare share) {
  __shared__ __align__(16) double boys[boys_rows_size(LA + LB + LC + LD)];
  load_boys<LA + LB + LC + LD>(boys_g, boys);
  __syncthreads();
  const long long beg = range[2 * blk], end = range[2 * blk + 1];
  if (beg >= end) return;
  const int lane = threadIdx.x & 31;
  int ls0 = 0;
  while (ls0 < 5 && ((end - beg) << (ls0 + 3)) <= share.lanes) ++ls0;
  const int target = (int)min((long long)INT_MAX, kLaneWork * max(1ll, (end - beg) / share.lanes));
  int nb = P.np[ql[beg].x];
  // stripes of `per` claims of `chunk` entries (claims of one list: fewer than 2^31)
  const unsigned nch = (unsigned)((end - beg + chunk - 1) / chunk), per = (nch + kStripes - 1) / kStripes;
  const bool striped = ls0 == 0 && nb * share.nk_max <= target && nch >= kStripeMin;
  for (;;) {
    int ls = ls0;
    while (ls < 5 && ((nb * share.nk_max) >> ls) > target) ++ls;
    if (striped) ls = 0;
    const int step = 32 >> ls, take = ls ? step : chunk;
    unsigned long long c0 = 0;
    if (lane == 0) c0 = atomicAdd(qhead + blk, (unsigned long long)(striped ? 1 : take));
    c0 = __shfl_sync(0xffffffffu, c0, 0);
    if (striped) {
      const unsigned t = (unsigned)c0;
      if (t >= per * kStripes) return;
      c0 = (unsigned long long)(t % kStripes * per + t / kStripes) * chunk;
    }
    const long long cfirst = beg + (long long)c0;
    if (cfirst >= end) {
      if (striped) continue;   // past the end of the last stripe
      return;                  // the whole list is claimed
    }
    const long long cend = min(cfirst + (long long)take, end);
    for (long long wfirst = cfirst; wfirst < cend; wfirst += step)
      nb = eri_jk_one<LA, LB, LC, LD, T>(ql, wfirst + (lane >> ls), wfirst, cend, P, S, boys, dg, ls);
    nb = __shfl_sync(0xffffffffu, nb, 0);
  }
}

template <int LA, int LB, int LC, int LD, typename T>
__global__ void __launch_bounds__(kEriThreads) k_eri_jk(const uint2 *__restrict__ ql, const long long *__restrict__ range,
                                                int blk, Pairs P, Shells S, const double *__restrict__ boys_g,
                                                DigestGroups dg, unsigned long long *__restrict__ qhead, int chunk,
                                                LaneShare share) {
  eri_jk_list<LA, LB, LC, LD, T>(ql, range, blk, P, S, boys_g, dg, qhead, chunk, share);
}

// Classes whose kernel is compiled for MB resident CTAs per SM (launch bounds with a
// minimum block count; the other classes keep the compiler's own register choice).
// Measured on (H2O)_32 cc-pVDZ: (ps|ps) at 4 against 3 CTAs 4.3 % faster, at 5 4.26 -> 5.79 ms;
// (ds|ps) at 3 against 2 2.8 %, at 4 2.67 -> 3.00 ms; (pp|ss) 2.23 ms at 5, 2.35 at 4; (ds|ss) 1.97
// ms at 4, 2.28 at the compiler's 3 (1.92 at 5, but 0.37 instead of 0.33 ms on (H2O)_11); (ps|ss)
// 7.53 ms at 5, 7.75 at 4, 8.18 at 6; (ss|ss) 3.75 ms at 4, 4.00 at 3 (168 registers), 4.01 at 5;
// (dp|ss) 1.06 ms at 4, 1.13 at 3; (pp|ps) 3.32 ms at the compiler's 2, 3.36 at 3.  They are bound
// by the latency of their chains and loads, up to the registers that spill.
template <int LA, int LB, int LC, int LD>
struct EriMinBlocks {
  static constexpr int v = 0;
};
template <>
struct EriMinBlocks<1, 0, 1, 0> {
  static constexpr int v = 4;
};
template <>
struct EriMinBlocks<1, 1, 0, 0> {
  static constexpr int v = 5;
};
template <>
struct EriMinBlocks<2, 0, 1, 0> {
  static constexpr int v = 3;
};
template <>
struct EriMinBlocks<0, 0, 0, 0> {
  static constexpr int v = 4;
};
template <>
struct EriMinBlocks<2, 0, 0, 0> {
  static constexpr int v = 4;
};
template <>
struct EriMinBlocks<1, 0, 0, 0> {
  static constexpr int v = 5;
};
template <>
struct EriMinBlocks<2, 1, 0, 0> {
  static constexpr int v = 4;
};

template <int LA, int LB, int LC, int LD, typename T, int MB>
__global__ void __launch_bounds__(kEriThreads, MB) k_eri_jk_mb(const uint2 *__restrict__ ql,
                                                       const long long *__restrict__ range, int blk, Pairs P,
                                                       Shells S, const double *__restrict__ boys_g, DigestGroups dg,
                                                       unsigned long long *__restrict__ qhead, int chunk,
                                                       LaneShare share) {
  eri_jk_list<LA, LB, LC, LD, T>(ql, range, blk, P, S, boys_g, dg, qhead, chunk, share);
}

// One list entry (pair quartet) per 2^ls lanes with the class's per-thread code and its
// digest.  With ls > 0 the lanes of a quartet take equal parts of its bra and, past the bra's
// primitive pairs, of its ket, and their integrals are summed before the first of them
// digests.  Returns the primitive pairs of the lane's bra.
template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ int eri_jk_plain(const uint2 e, const bool valid, const Pairs &P, const Shells &S,
                                            const double *boys, const DigestGroups &dg, int ls) {
  constexpr int NA = nfun_c(LA), NB = nfun_c(LB), NC = nfun_c(LC), ND = nfun_c(LD);
  const int2 ab = P.sh[e.x], cd = P.sh[e.y];
  const int nb = P.np[e.x], nk = P.np[e.y];
  double v[NA * NB * NC * ND];
  if (valid) {
    const double3 A = S.center[ab.x], B = S.center[ab.y], C = S.center[cd.x], D = S.center[cd.y];
    PrimCols bp = {P.cols + (size_t)P.coff[e.x] * kPrimRow + (e.x & 31)},
             kp = {P.cols + (size_t)P.coff[e.y] * kPrimRow + (e.y & 31)};
    int nb1 = nb, nk1 = nk;
    if (ls) {
      const int s = threadIdx.x & ((1 << ls) - 1);
      int lb = 0;   // bra parts 2^lb <= nb, ket parts 2^(ls - lb)
      while (lb < ls && (2 << lb) <= nb) ++lb;
      const int lk = ls - lb, sb = s >> lk, sk = s & ((1 << lk) - 1);
      const int b0 = (nb * sb) >> lb, k0 = (nk * sk) >> lk;
      nb1 = ((nb * (sb + 1)) >> lb) - b0;
      nk1 = ((nk * (sk + 1)) >> lk) - k0;
      bp = bp + b0;
      kp = kp + k0;
    }
    if constexpr (sizeof(T) == sizeof(double)) {
      EriClass<LA, LB, LC, LD>::template run<double>(bp, nb1, kp, nk1, A, B, C, D, boys, v);
    } else {
      T vt[NA * NB * NC * ND];
      EriClass<LA, LB, LC, LD>::template run<T>(bp, nb1, kp, nk1, A, B, C, D, boys, vt);
#pragma unroll
      for (int k = 0; k < NA * NB * NC * ND; ++k) v[k] = (double)vt[k];
    }
  } else {
#pragma unroll
    for (int k = 0; k < NA * NB * NC * ND; ++k) v[k] = 0.0;
  }
  for (int o = (1 << ls) >> 1; o > 0; o >>= 1) {
#pragma unroll
    for (int k = 0; k < NA * NB * NC * ND; ++k) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
  }
  const unsigned bra0 = __shfl_sync(0xffffffffu, e.x, 0);
  const bool uniform = __all_sync(0xffffffffu, e.x == bra0);
  const double deg = (ab.x == ab.y ? 1.0 : 2.0) * (cd.x == cd.y ? 1.0 : 2.0) * (e.x == e.y ? 1.0 : 2.0);
  digest<LA, LB, LC, LD>(v, deg, (int)e.x, (int)e.y, P, S, dg, valid && (threadIdx.x & ((1 << ls) - 1)) == 0,
                         uniform);
  return nb;
}

// One sibling-group entry per lane: the generated sibling form evaluates the MB x MK member
// quartets (bra members leader e.x + i, ket members e.y + j) from one pass over the groups'
// primitive pairs, then each member quartet of the entry's mask is digested as a quartet of
// its own.
template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ void eri_jk_group(const uint2 e, const bool valid, const unsigned mask, const Pairs &P,
                                             const Shells &S, const double *boys, const DigestGroups &dg) {
  constexpr int NA = nfun_c(LA), NB = nfun_c(LB), NC = nfun_c(LC), ND = nfun_c(LD);
  constexpr int NQ = NA * NB * NC * ND;
  constexpr int MB = EriGroup<LA, LB, LC, LD>::MB, MK = EriGroup<LA, LB, LC, LD>::MK;
  const int mb = P.gsz[e.x], mk = P.gsz[e.y];
  double v[MB * MK * NQ];
  if (valid) {
    const int2 ab = P.sh[e.x], cd = P.sh[e.y];
    const double3 A = S.center[ab.x], B = S.center[ab.y], C = S.center[cd.x], D = S.center[cd.y];
    const PrimPair *bp = P.gprim + P.gpoff[e.x], *kp = P.gprim + P.gpoff[e.y];
    const double *bw = P.gw + P.gwoff[e.x], *kw = P.gw + P.gwoff[e.y];
    if constexpr (sizeof(T) == sizeof(double)) {
      EriClassGC<LA, LB, LC, LD, MB, MK>::template run<double>(bp, bw, P.gnp[e.x], kp, kw, P.gnp[e.y], A, B, C, D,
                                                               boys, v);
    } else {
      T vt[MB * MK * NQ];
      EriClassGC<LA, LB, LC, LD, MB, MK>::template run<T>(bp, bw, P.gnp[e.x], kp, kw, P.gnp[e.y], A, B, C, D, boys,
                                                          vt);
#pragma unroll
      for (int k = 0; k < MB * MK * NQ; ++k) v[k] = (double)vt[k];
    }
  } else {
#pragma unroll
    for (int k = 0; k < MB * MK * NQ; ++k) v[k] = 0.0;
  }
  const unsigned bra0 = __shfl_sync(0xffffffffu, e.x, 0);
  const bool uniform = __all_sync(0xffffffffu, e.x == bra0);
#pragma unroll
  for (int i = 0; i < MB; ++i) {
#pragma unroll
    for (int j = 0; j < MK; ++j) {
      const bool mv = valid && ((mask >> (4 * i + j)) & 1u);
      if (!__any_sync(0xffffffffu, mv)) continue;
      // members past the group's size are never in the mask; their lanes address the leader
      const int pa = i < mb ? (int)e.x + i : (int)e.x;
      const int pc = j < mk ? (int)e.y + j : (int)e.y;
      const int2 ab = P.sh[pa], cd = P.sh[pc];
      const double deg = (ab.x == ab.y ? 1.0 : 2.0) * (cd.x == cd.y ? 1.0 : 2.0) * (pa == pc ? 1.0 : 2.0);
      digest<LA, LB, LC, LD>(v + (i * MK + j) * NQ, deg, pa, pc, P, S, dg, mv, uniform);
    }
  }
}

template <int LA, int LB, int LC, int LD, typename T>
__device__ __forceinline__ int eri_jk_one(const uint2 *__restrict__ ql, long long i, long long wfirst, long long end,
                                          const Pairs &P, const Shells &S, const double *boys,
                                          const DigestGroups &dg, int ls) {
  const bool valid = i < end;
  const uint2 e = ql[valid ? i : wfirst];
  return eri_jk_plain<LA, LB, LC, LD, T>(e, valid, P, S, boys, dg, ls);
}

// Sibling-group list of class (LA LB|LC LD): the work queue and persistent grid of
// k_eri_jk, one entry (bra group, ket group, member mask) per thread, NT threads per CTA
// (64 lets one more CTA of these register-heavy kernels reside on an SM).
template <int LA, int LB, int LC, int LD, typename T, int NT>
__global__ void __launch_bounds__(NT) k_eri_gc(const uint2 *__restrict__ ql, const long long *__restrict__ range,
                                                int blk, Pairs P, Shells S, const double *__restrict__ boys_g,
                                                DigestGroups dg, unsigned long long *__restrict__ qhead, int chunk) {
  __shared__ __align__(16) double boys[boys_rows_size(LA + LB + LC + LD)];
  load_boys<LA + LB + LC + LD>(boys_g, boys);
  __syncthreads();
  const long long beg = range[2 * blk], end = range[2 * blk + 1];
  const int lane = threadIdx.x & 31;
  for (;;) {
    unsigned long long c0 = 0;
    if (lane == 0) c0 = atomicAdd(qhead + blk, (unsigned long long)chunk);
    c0 = __shfl_sync(0xffffffffu, c0, 0);
    const long long cfirst = beg + (long long)c0;
    if (cfirst >= end) return;   // the whole list is claimed
    const long long cend = min(cfirst + (long long)chunk, end);
    for (long long wfirst = cfirst; wfirst < cend; wfirst += 32) {
      const long long i = wfirst + lane;
      const bool valid = i < cend;
      const uint2 e = ql[valid ? i : wfirst];
      const unsigned mask = valid ? (unsigned)P.qmask[i] : 0u;
      eri_jk_group<LA, LB, LC, LD, T>(e, valid, mask, P, S, boys, dg);
    }
  }
}

// ---------------------------------------------- a warp on a quartet or a pair ---
// J/K digest of one quartet by a warp: V [a][b][c][d] in shared memory, lanes spread over the
// elements of Gh (the same updates as digest()).  Xs: shared memory for the density blocks.
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void digest_warp(const double *V, double *Xs, const DigestGroups &dg, int a0, int b0, int c0,
                                            int d0, int mol, double deg, int lane) {
  constexpr int NA = nfun_c(LA), NB = nfun_c(LB), NC = nfun_c(LC), ND = nfun_c(LD);
  // staged blocks: X(d,c) [NC*ND], X(b,a) [NA*NB], X(b,d), X(a,c), X(b,c), X(a,d)
  double *xdc = Xs, *xba = xdc + NC * ND, *xbd = xba + NA * NB, *xac = xbd + NB * ND;
  double *xbc = xac + NA * NC, *xad = xbc + NB * NC;
  for (int g = 0; g < dg.ng; ++g) {
    const double *Xv;
    double *G;
    size_t ld, n;
    mol_view(dg, g, mol, Xv, G, ld, n);
    const double *__restrict__ Xm = Xv;
    const double sJ = dg.sJ[g] * deg, sK = 0.5 * dg.sK[g] * deg;
    __syncwarp();
    for (int k = lane; k < NC * ND; k += 32) xdc[k] = __ldg(Xm + (d0 + k % ND) + (c0 + k / ND) * ld);
    for (int k = lane; k < NA * NB; k += 32) xba[k] = __ldg(Xm + (b0 + k % NB) + (a0 + k / NB) * ld);
    for (int k = lane; k < NB * ND; k += 32) xbd[k] = __ldg(Xm + (b0 + k / ND) + (d0 + k % ND) * ld);
    for (int k = lane; k < NA * NC; k += 32) xac[k] = __ldg(Xm + (a0 + k / NC) + (c0 + k % NC) * ld);
    for (int k = lane; k < NB * NC; k += 32) xbc[k] = __ldg(Xm + (b0 + k / NC) + (c0 + k % NC) * ld);
    for (int k = lane; k < NA * ND; k += 32) xad[k] = __ldg(Xm + (a0 + k / ND) + (d0 + k % ND) * ld);
    __syncwarp();
    // every update is written with the index that varies fastest across lanes as the
    // row (k_finalize symmetrises Gh), so a warp's atomics fall on consecutive addresses
    if (dg.sJ[g] != 0.0) {
      for (int k = lane; k < NA * NB; k += 32) {
        const int a = k / NB, b = k % NB;
        double s = 0.0;
        for (int cd = 0; cd < NC * ND; ++cd) s += xdc[cd] * V[k * NC * ND + cd];
        atomicAdd(G + (b0 + b) + (a0 + a) * n, sJ * s);
      }
      for (int k = lane; k < NC * ND; k += 32) {
        const int c = k / ND, d = k % ND;
        double s = 0.0;
        for (int ab2 = 0; ab2 < NA * NB; ++ab2) s += xba[ab2] * V[ab2 * NC * ND + k];
        atomicAdd(G + (d0 + d) + (c0 + c) * n, sJ * s);
      }
    }
    if (dg.sK[g] != 0.0) {
      for (int k = lane; k < NA * NC; k += 32) {   // G(a,c) += X(b,d) v
        const int a = k / NC, c = k % NC;
        double s = 0.0;
        for (int b = 0; b < NB; ++b)
          for (int d = 0; d < ND; ++d) s += xbd[b * ND + d] * V[((a * NB + b) * NC + c) * ND + d];
        atomicAdd(G + (c0 + c) + (a0 + a) * n, sK * s);
      }
      for (int k = lane; k < NB * ND; k += 32) {   // G(b,d) += X(a,c) v
        const int b = k / ND, d = k % ND;
        double s = 0.0;
        for (int a = 0; a < NA; ++a)
          for (int c = 0; c < NC; ++c) s += xac[a * NC + c] * V[((a * NB + b) * NC + c) * ND + d];
        atomicAdd(G + (d0 + d) + (b0 + b) * n, sK * s);
      }
      for (int k = lane; k < NA * ND; k += 32) {   // G(a,d) += X(b,c) v
        const int a = k / ND, d = k % ND;
        double s = 0.0;
        for (int b = 0; b < NB; ++b)
          for (int c = 0; c < NC; ++c) s += xbc[b * NC + c] * V[((a * NB + b) * NC + c) * ND + d];
        atomicAdd(G + (d0 + d) + (a0 + a) * n, sK * s);
      }
      for (int k = lane; k < NB * NC; k += 32) {   // G(b,c) += X(a,d) v
        const int b = k / NC, c = k % NC;
        double s = 0.0;
        for (int a = 0; a < NA; ++a)
          for (int d = 0; d < ND; ++d) s += xad[a * ND + d] * V[((a * NB + b) * NC + c) * ND + d];
        atomicAdd(G + (c0 + c) + (b0 + b) * n, sK * s);
      }
    }
  }
}

// Schwarz bounds of the pair classes whose (ab|ab) is a warp class: Q(i) = sqrt(max |(ab|ab)|)
// for pairs [beg, end), a warp per pair (set-up only).
template <int LA, int LB>
__global__ void __launch_bounds__(128) k_schwarz_warp(Pairs P, Shells S, const double *__restrict__ boys, int beg,
                                                      int end, double *__restrict__ Qout) {
  using WD = warpmd::WarpDims<LA, LB>;
  constexpr int L = WD::L;
  extern __shared__ double smem[];
  // decode tables: Hermite (t,u,v) of index h and Cartesian exponents of the pair, packed 4
  // bits per exponent
  __shared__ int s_h[WD::HP];
  __shared__ int s_cab[WD::NCAB];
  // s_rec[h], h >= 1: the downward recursion R^n_h = P_d R^{n+1}_a + m R^{n+1}_b of Hermite
  // triple h, packed as a | b << 10 | d << 20 | m << 22 (d = 0, 1, 2 for x, y, z)
  __shared__ int s_rec[WD::HL];
  for (int k = threadIdx.x; k < WD::HL; k += blockDim.x) {
    int t, u, v;
    warpmd::herm_of(k, t, u, v);
    if (k < WD::HP) s_h[k] = t | (u << 4) | (v << 8);
    int a = 0, b = 0, d = 0, m = 0;
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
  for (int k = threadIdx.x; k < WD::NCAB; k += blockDim.x) {
    int x0, y0, z0, x1, y1, z1;
    warpmd::cart_of(LA, k / warpmd::ncart(LB), x0, y0, z0);
    warpmd::cart_of(LB, k % warpmd::ncart(LB), x1, y1, z1);
    s_cab[k] = x0 | (y0 << 4) | (z0 << 8) | (x1 << 12) | (y1 << 16) | (z1 << 20);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  double *Eb = smem + (size_t)wid * WD::SMEM, *Ek = Eb + 3 * WD::NE, *Ra = Ek + 3 * WD::NE, *Rb = Ra + WD::HL;
  double *W = Rb + WD::HL, *Cc = W + WD::NBUF;
  for (int i = beg + blockIdx.x * (blockDim.x >> 5) + wid; i < end; i += gridDim.x * (blockDim.x >> 5)) {
    const int2 ab = P.sh[i];
    const double3 A = S.center[ab.x], B = S.center[ab.y];
    const PrimPair *pp = P.prim + P.poff[i];
    const int np = P.np[i];
    // E coefficients of a primitive pair, one direction per lane
    auto expand = [&](double *E, const PrimPair &p) {
      if (lane < 3) {
        const double Pc = lane == 0 ? p.Px : (lane == 1 ? p.Py : p.Pz);
        const double Ac = lane == 0 ? A.x : (lane == 1 ? A.y : A.z);
        const double Bc = lane == 0 ? B.x : (lane == 1 ? B.y : B.z);
        warpmd::build_E1<LA, LB, double>(E + lane * WD::NE, Pc - Ac, Pc - Bc, 0.5 * p.ip);
      }
    };
    __syncwarp();
    for (int k = lane; k < WD::NC; k += 32) Cc[k] = 0.0;
    for (int ib = 0; ib < np; ++ib) {
      const PrimPair bp = pp[ib];
      __syncwarp();
      expand(Eb, bp);
      for (int k = lane; k < WD::NW; k += 32) W[k] = 0.0;
      for (int ik = 0; ik < np; ++ik) {
        const PrimPair kp = pp[ik];
        __syncwarp();
        expand(Ek, kp);
        const double pq = bp.p + kp.p;
        const double rpq = rsqrt(pq);
        const double rho = bp.p * kp.p * (rpq * rpq);
        const double X = bp.Px - kp.Px, Y = bp.Py - kp.Py, Z = bp.Pz - kp.Pz;
        double F[L + 1];
        boys_eval<L>(rho * (X * X + Y * Y + Z * Z), boys, F);
        double f = bp.Kp * kp.Kp * rpq;
#pragma unroll
        for (int n = 0; n <= L; ++n) {
          F[n] *= f;
          f *= -2.0 * rho;
        }
        // R^{(n)}_{tuv}, n = L .. 0, ping-pong between Ra and Rb; level L in Ra when L even
        double *prev = (L % 2 == 0) ? Rb : Ra;
        double *cur = (L % 2 == 0) ? Ra : Rb;
        if (lane == 0) cur[0] = F[L];
#pragma unroll
        for (int n = L - 1; n >= 0; --n) {
          double *t_ = prev;
          prev = cur;
          cur = t_;
          __syncwarp();
          const int cnt = warpmd::nherm(L - n);
          for (int h = lane; h < cnt; h += 32) {
            double val = F[n];
            if (h > 0) {
              const int r = s_rec[h];
              const int dr = (r >> 20) & 3;
              const double pd = dr == 0 ? X : (dr == 1 ? Y : Z);
              val = pd * prev[r & 1023] + (double)(r >> 22) * prev[(r >> 10) & 1023];
            }
            cur[h] = val;
          }
        }
        __syncwarp();
        const double *R = cur;  // level 0
        // W[tuv][cd] += sum (-1)^(tau+nu+phi) E^cd R
        for (int e2 = lane; e2 < WD::NW; e2 += 32) {
          const int hc = s_h[e2 / WD::NCAB], cc = s_cab[e2 % WD::NCAB];
          const int t = hc & 15, u = (hc >> 4) & 15, v = hc >> 8;
          const int cx = cc & 15, cy = (cc >> 4) & 15, cz = (cc >> 8) & 15;
          const int dx = (cc >> 12) & 15, dy = (cc >> 16) & 15, dz = cc >> 20;
          constexpr int NT = LA + LB + 1;
          const double *ex = Ek + (cx * (LB + 1) + dx) * NT;
          const double *ey = Ek + WD::NE + (cy * (LB + 1) + dy) * NT;
          const double *ez = Ek + 2 * WD::NE + (cz * (LB + 1) + dz) * NT;
          double s = 0.0;
          for (int a1 = 0; a1 <= cx + dx; ++a1)
            for (int a2 = 0; a2 <= cy + dy; ++a2) {
              const double exy = ((a1 + a2) & 1 ? -1.0 : 1.0) * ex[a1] * ey[a2];
              for (int a3 = 0; a3 <= cz + dz; ++a3)
                s += exy * ((a3 & 1) ? -ez[a3] : ez[a3]) * R[warpmd::hidx(t + a1, u + a2, v + a3)];
            }
          W[e2] += s;
        }
      }
      __syncwarp();
      // C[ab][cd] += sum_tuv E^ab_tuv W[tuv][cd]
      for (int e2 = lane; e2 < WD::NC; e2 += 32) {
        const int cc = s_cab[e2 / WD::NCAB], c = e2 % WD::NCAB;
        const int ax = cc & 15, ay = (cc >> 4) & 15, az = (cc >> 8) & 15;
        const int bx = (cc >> 12) & 15, by = (cc >> 16) & 15, bz = cc >> 20;
        constexpr int NT = LA + LB + 1;
        const double *ex = Eb + (ax * (LB + 1) + bx) * NT;
        const double *ey = Eb + WD::NE + (ay * (LB + 1) + by) * NT;
        const double *ez = Eb + 2 * WD::NE + (az * (LB + 1) + bz) * NT;
        double s = 0.0;
        for (int a1 = 0; a1 <= ax + bx; ++a1)
          for (int a2 = 0; a2 <= ay + by; ++a2) {
            const double exy = ex[a1] * ey[a2];
            for (int a3 = 0; a3 <= az + bz; ++a3) s += exy * ez[a3] * W[warpmd::hidx(a1, a2, a3) * WD::NCAB + c];
          }
        Cc[e2] += s;
      }
    }
    __syncwarp();
    // Cartesian -> spherical on pure axes (L > 1), ping-pong Cc <-> W
    double *src = Cc, *dst = W;
    {
      int d[4] = {warpmd::ncart(LA), warpmd::ncart(LB), warpmd::ncart(LA), warpmd::ncart(LB)};
      const int ls[4] = {LA, LB, LA, LB};
#pragma unroll
      for (int ax = 0; ax < 4; ++ax) {
        if (ls[ax] < 2) continue;
        warpmd::sph_axis<double>(src, dst, d, ax, ls[ax], ls[ax] == 2 ? kSph2 : kSph3, lane);
        d[ax] = 2 * ls[ax] + 1;
        double *t_ = src;
        src = dst;
        dst = t_;
        __syncwarp();
      }
    }
    constexpr int NAB = warpmd::nfun(LA) * warpmd::nfun(LB);
    double mx = 0.0;
    for (int k = lane; k < NAB; k += 32) mx = fmax(mx, fabs(src[k * NAB + k]));
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) Qout[i] = sqrt(mx);
  }
}

#include "eri_tc.cuh"

// AX += 0.5 (Gh + Gh^T) of group g, molecule blockIdx.z of the context; Gh = G plus GP, which is
// in the internal order, plus the Coulomb sums of the shell pairs, JP.
static __global__ void k_finalize(DigestGroups dg, int g, Mols mols, const int *__restrict__ bf,
                                  const int *__restrict__ sz, const int *__restrict__ shL, double *__restrict__ AX0,
                                  int ldax) {
  __shared__ double tile[32][33];
  const int mol = blockIdx.z;
  const int n = mols.nbf[mol];
  if (!mols.active[mol] || (int)(blockIdx.x * 32) >= n || (int)(blockIdx.y * 32) >= n) return;
  const double *G = dg.G[g], *GP = dg.GP[g];
  double *AX = AX0;
  if (mols.nmol > 1) {
    G += mols.xoff[mol];
    GP += mols.xoff[mol];
    AX += mols.xoff[mol];
    ldax = n;
  }
  const int *pos = mols.pos + mols.foff[mol], *fsh = mols.fsh + mols.foff[mol];
  const int nsh = mols.nsh[mol], shoff = mols.shoff[mol];
  const int *pidx = mols.pidx + mols.Moff[mol];
  const bool coulomb = dg.sJ[g] != 0.0;
  auto gh = [&](int r, int c) {
    double v = G[(size_t)r + (size_t)c * n] + GP[(size_t)pos[r] + (size_t)pos[c] * n];
    if (coulomb) {
      const int y = fsh[r], x = fsh[c], pair = pidx[y + (size_t)x * nsh];
      if (pair >= 0) {
        const int gx = shoff + x, gy = shoff + y, cls = pair_class_c(shL[gx], shL[gy]);
        const int k = (c - bf[gx]) * sz[gy] + (r - bf[gy]);
        v += dg.JP[g][dg.joff[cls] + (size_t)k * dg.jn[cls] + (pair - dg.jbeg[cls])];
      }
    }
    return v;
  };
  int bx = blockIdx.x * 32, by = blockIdx.y * 32;
  int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  for (int k = ty; k < 32; k += 8) {
    int rr = by + tx, cc = bx + k;
    tile[k][tx] = (rr < n && cc < n) ? gh(rr, cc) : 0.0;  // tile[k][tx] = Gh(by+tx, bx+k)
  }
  __syncthreads();
  for (int k = ty; k < 32; k += 8) {
    int r = bx + tx, c = by + k;
    if (r < n && c < n) AX[(size_t)r + (size_t)c * ldax] += 0.5 * (gh(r, c) + tile[tx][k]);  // Gh(c, r)
  }
}

// FMA throughput probe (roofline denominator): independent dependent-FMA chains.
template <typename T>
__global__ void k_fma_probe(T *out, int iters, T seed) {
  T a0 = seed + threadIdx.x, a1 = a0 + 1, a2 = a0 + 2, a3 = a0 + 3, a4 = a0 + 4, a5 = a0 + 5, a6 = a0 + 6, a7 = a0 + 7;
  const T m = T(0.999999), c = T(1e-7);
  for (int i = 0; i < iters; ++i) {
#pragma unroll
    for (int k = 0; k < 16; ++k) {
      a0 = a0 * m + c; a1 = a1 * m + c; a2 = a2 * m + c; a3 = a3 * m + c;
      a4 = a4 * m + c; a5 = a5 * m + c; a6 = a6 * m + c; a7 = a7 * m + c;
    }
  }
  T s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
  if (s == T(-12345.0)) out[0] = s;
}

// ------------------------------------------------------------------ host side ---
#define CUCHK(call)                                                                \
  do {                                                                             \
    cudaError_t _e = (call);                                                       \
    if (_e != cudaSuccess) {                                                       \
      ctx->err = std::string(#call) + ": " + cudaGetErrorString(_e);               \
      return CQG_ERR_CUDA;                                                         \
    }                                                                              \
  } while (0)

// Device memory of the contexts, from a process-wide pool (engine.cu): *bytes is rounded up to
// the block's size.  A block may be handed to another context, on any stream, as soon as it
// is given back, so it is given back only when the device has finished with it.
cudaError_t cqg_pool_alloc(void **p, size_t *bytes, int *device);
void cqg_pool_free(void *p, size_t bytes, int device);

template <typename T>
struct DevBuf {
  T *p = nullptr;
  size_t n = 0, bytes = 0;
  int device = 0;
  // At least m elements; a larger buffer replaces the old one (contents are not kept) after
  // the device has finished with it.
  cudaError_t reserve(size_t m) {
    if (m <= n) return cudaSuccess;
    if (p) {
      const cudaError_t e = cudaDeviceSynchronize();
      if (e != cudaSuccess) return e;
      release();
    }
    const size_t want = std::max<size_t>(m, 1);
    size_t b = want * sizeof(T);
    void *q = nullptr;
    const cudaError_t e = cqg_pool_alloc(&q, &b, &device);
    if (e != cudaSuccess) return e;
    p = (T *)q;
    n = want;
    bytes = b;
    return cudaSuccess;
  }
  // gives the buffer back; the device has finished with it
  void release() {
    if (p) cqg_pool_free(p, bytes, device);
    p = nullptr;
    n = bytes = 0;
  }
};

// Side streams of the class launches besides the caller's.  One build is 21 launches in
// double zeta, 55 in triple zeta; in series each waits for the last warp of the one before.
// With seven side streams the tails overlap: one water in 6-31G(d) 1.53 -> 0.39 ms, O2 UHF
// cc-pVDZ 3.09 -> 1.12 ms, (H2O)_11 cc-pVDZ 7.3 -> 4.9 ms, (H2O)_5 cc-pVTZ 25.8 -> 21.7 ms;
// (H2O)_32, whose lists fill the GPU by themselves, within 1 %.
constexpr int kSideStreams = 7;
struct SideStreams {
  int device = 0;
  unsigned long long *host = nullptr;   // pinned: the call state as read back (kStateRead words)
  cudaEvent_t read = nullptr;
  cudaStream_t st[kSideStreams] = {};
  cudaEvent_t done[kSideStreams] = {}, fork = nullptr;
};

// words of the call state: flags, Mmax, mask-cache head, tallies, ranges | work-queue heads
constexpr int kStateRead = 4 + kBlkAcc * CQG_NQC + 2 * CQG_NLIST, kStateWords = kStateRead + CQG_NLIST + 1;

struct cqg_ctx {
  int device = 0;
  std::string err;
  double thresh = 1e-14;
  int policy = CQG_PREC_FP64;
  double fp32_cutoff = 0.0;
  int timing = 0;
  long long list_budget = 1LL << 32;   // quartets held in the list at once (8 B each: 32 GiB)
  int nsm = 148;                       // multiprocessors of the device
  // launch shapes per (precision, class) work list: persistent CTAs per SM and, for the
  // tensor-core classes, warps per CTA (0 = default); set by the autotuner
  int shape_cta[CQG_NLIST] = {0};
  int shape_wpb[CQG_NLIST] = {0};
  // entries a warp claims from the list's work queue at a time, in units of 32 for the
  // per-thread classes and at most 32 for the tensor-core ones (0 = default: 32, and a number
  // that follows the list's length)
  int shape_qpw[CQG_NLIST] = {0};
  // kernel form of a list whose class has both: 0 = per-thread, 1 = tensor-core
  int shape_var[CQG_NLIST] = {0};
  // 0: one launch per class list; 1 or 2: the lists of that tier's classes go through one
  // class-fused persistent kernel (eri_fused.cu); set by the autotuner or cqg_set_fusion
  int fused_tier = 0;
  int used_cta = 0;   // CTAs per SM of the last class launch (the autotuner's record of a default)
  double fusion_ms[3] = {0.0, 0.0, 0.0};   // autotuner's times of the three forms (ms)
  // Per-call state, one buffer: zeroed by one memset, and read back by one copy up to `range`.
  DevBuf<unsigned long long> d_state;
  int *p_flags = nullptr;                  // non-finite, asymmetric, list overflow
  double *p_Mmax = nullptr;
  unsigned long long *p_mhead = nullptr;   // MaskCache::head
  unsigned long long *p_blkacc = nullptr;  // screening tallies, kBlkAcc per class
  long long *p_range = nullptr;            // [begin, end) of every work list
  unsigned long long *p_qhead = nullptr;   // work-queue head of every work list, then the fused one
  int autotune_pending = 0;
  long long graph_capacity = 0;        // > 0: sync-free contraction for CUDA-graph capture
  bool class_possible[CQG_NQC] = {false};
  // molecules of the context (a batch when nmol > 1)
  int nmol = 0, max_nsh = 0, max_nbf = 0;
  long long packed = 0, Mtotal = 0;
  std::vector<int> hshmol, m_shoff, m_nsh, m_nbf;
  std::vector<long long> m_xoff, m_Moff;
  std::vector<unsigned char> h_active;
  DevBuf<int> d_shmol, d_mshoff, d_mnsh, d_mnbf, d_molbk;
  DevBuf<long long> d_mxoff, d_mMoff;
  DevBuf<unsigned char> d_active;
  // basis
  int nshell = 0, nbf = 0, maxl = 0;
  std::vector<int> hL, hbf, hsz, hnprim, hpoff;
  std::vector<double> halpha, hcoef, hcent;
  std::vector<double> Qmat;  // nshell x nshell
  // pairs, by class
  int pc_beg[CQG_NPC + 1] = {0};
  int bucket_beg[CQG_NPC][CQG_NBUCKET + 1];
  std::vector<int2> pair_sh;
  std::vector<double> pair_Q;
  DevBuf<double3> d_center;
  DevBuf<int> d_bf, d_sz;
  DevBuf<int2> d_pair_sh;
  DevBuf<double> d_pair_Q;
  DevBuf<int> d_pair_poff, d_pair_np, d_pair_kk;
  DevBuf<int> d_shL, d_shnp, d_shpoff;
  DevBuf<double> d_alpha, d_coef;
  DevBuf<double> d_oe;       // host-mode staging of S, T, V
  DevBuf<double> d_charges;  // Z then R (3 per charge)
  int launches = 0;
  DevBuf<PrimPair> d_prim;
  DevBuf<double2> d_cols;
  DevBuf<int2> d_pf;                   // internal order of the basis functions (Shells.pf, Mols.pos)
  DevBuf<int> d_pos, d_mfoff, d_pidx, d_fsh;
  DevBuf<double> d_XP;                 // per call: X in the internal order, Coulomb blocks of X by pair
  DevBuf<int> d_pair_coff;
  DevBuf<int> d_setup;                 // cqg_set_basis: group members, primitive-pair counts
  const double *boys = nullptr;        // kBoysTable (boys_eval) and kBoysRows (load_boys) on the context's
  const double *boys_rows = nullptr;   // device: module constants, valid as long as its CUDA context
  // Hermite expansion tables (k_expansions) of each pair class's primitive pairs: offset in
  // d_exp and index of the class's first primitive pair
  DevBuf<double> d_exp;
  size_t exp_off[CQG_NPC] = {0};
  int exp_prim0[CQG_NPC] = {0};
  bool exp_have[CQG_NPC] = {false};   // the class's tables are those of the current basis
  int pc_prim[CQG_NPC + 1] = {0};   // first primitive pair of each pair class
  int pc_np_max[CQG_NPC] = {0};   // most primitive pairs of a pair, per class
  // per-call scratch
  DevBuf<double> d_M, d_Mpair;
  DevBuf<long long> d_cnt, d_off;
  DevBuf<unsigned char> d_scan_tmp;
  DevBuf<uint2> d_qlist;
  DevBuf<double> d_G, d_X, d_AX, d_Gscratch;
  BlockTable bt;                      // the active table (bt_pair or bt_group)
  int ntask = 0;
  BlockTable bt_pair, bt_group;       // pair tasks everywhere / bra-group tasks for the sibling classes
  int ntask_pair = 0, ntask_group = 0;
  // sibling groups (Pairs): on = the sibling classes get sibling-entry lists
  int siblings = 0;
  // grouped classes: smallest number of member quartets of a pair of groups that makes a
  // sibling entry (smaller ones become pair entries); set from the sibling form's size
  int sibling_min[CQG_NQC] = {0};
  std::vector<int> pair_gsz, glead;
  std::vector<double> pair_Qc, gQ;
  int gc_beg[CQG_NPC + 1] = {0};      // first group of each pair class
  std::vector<int> fam;               // shell families (siblings.h)
  bool groups_ready = false;          // the group arrays of the current basis are on the device
  DevBuf<int> d_molgbk, d_gsz, d_gpoff, d_gnp, d_gwoff, d_glead;
  DevBuf<double> d_pair_Qc, d_gQ, d_gw;
  DevBuf<PrimPair> d_gprim;
  DevBuf<unsigned short> d_qmask;     // member masks, parallel to d_qlist
  // survivor-mask cache of the screening passes (MaskCache): steps, head, per-task slots
  DevBuf<uint2> d_masks;
  DevBuf<long long> d_mslot;
  long long mask_steps_used = 0;      // steps the last count pass asked for
  // buffers that a contraction outgrew while graph mode was on: captured launches hold their
  // addresses, so they stay the context's own until graph mode or the basis ends
  struct Retired {
    void *p;
    size_t bytes;
    int device;
  };
  std::vector<Retired> retired;
  SideStreams *side = nullptr;   // leased on first use (ClassStreams in engine.cu)
  // classes, most work first, as the last uncaptured contraction counted it (a captured one
  // launches in this order)
  int class_order[CQG_NQC];
  cudaEvent_t ev[4 + 2 * CQG_NQC + 2] = {};   // made when timing is first switched on
  bool events = false;
  cqg_stats stats;
  double *oe_table = nullptr;   // device address of the fixed charge table (cqg_one_e_noalloc)
};

static inline Pairs make_pairs(cqg_ctx *ctx);
static inline Shells make_shells(cqg_ctx *ctx);

// classes that have the tensor-core kernel only (same rule as gen_eri.WARP_CLASSES)
__host__ __device__ constexpr bool is_warp_class(int la, int lb, int lc, int ld) {
  return ncart_c(la) * ncart_c(lb) * ncart_c(lc) * ncart_c(ld) > 150 || la + lb + lc + ld >= 6;
}

// Per-thread classes whose live state overflows one thread's 255 registers (their
// generated code spills to local memory): they also get the tensor-core kernel, and the
// autotuner times both forms on the class's list and keeps the faster one.
__host__ __device__ constexpr bool is_variant_class(int la, int lb, int lc, int ld) {
  const int k = ((la * 4 + lb) * 4 + lc) * 4 + ld;
  return !is_warp_class(la, lb, lc, ld) &&
         (k == ((1 * 4 + 1) * 4 + 1) * 4 + 1 || k == ((2 * 4 + 0) * 4 + 1) * 4 + 1 ||   // (pp|pp), (ds|pp)
          k == ((2 * 4 + 0) * 4 + 2) * 4 + 0 || k == ((2 * 4 + 1) * 4 + 1) * 4 + 0 ||   // (ds|ds), (dp|ps)
          k == ((2 * 4 + 1) * 4 + 2) * 4 + 0 || k == ((2 * 4 + 2) * 4 + 0) * 4 + 0 ||   // (dp|ds), (dd|ss)
          k == ((2 * 4 + 2) * 4 + 1) * 4 + 0 || k == ((3 * 4 + 0) * 4 + 1) * 4 + 0 ||   // (dd|ps), (fs|ps)
          k == ((3 * 4 + 0) * 4 + 1) * 4 + 1 || k == ((3 * 4 + 0) * 4 + 2) * 4 + 0 ||   // (fs|pp), (fs|ds)
          k == ((3 * 4 + 1) * 4 + 1) * 4 + 0 || k == ((3 * 4 + 2) * 4 + 0) * 4 + 0);    // (fp|ps), (fd|ss)
}

// Of those, the classes whose FP64 list starts on the tensor-core kernel: (H2O)_5 cc-pVTZ,
// per-thread against tensor-core form, (fs|pp) 0.64 / 0.24 ms, (fs|ds) 0.30 / 0.27; the others
// are faster per thread ((pp|pp) 1.79 / 3.07 ms on (H2O)_32 cc-pVDZ, (dp|ds) 1.59 / 1.96, (ds|pp)
// 2.18 / 5.07), whose tiles would be mostly padding.
__host__ __device__ constexpr bool is_tensor_first(int la, int lb, int lc, int ld) {
  return la == 3 && lb == 0 && ((lc == 1 && ld == 1) || (lc == 2 && ld == 0));
}

// Dynamic shared memory above the default 48 KB, asked for once per kernel and device.
template <typename K>
static cudaError_t allow_smem(K kernel, size_t bytes, int device, std::atomic<bool> (&done)[64]) {
  const int slot = (device >= 0 && device < 64) ? device : 0;
  if (done[slot].load(std::memory_order_relaxed)) return cudaSuccess;
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) done[slot].store(true, std::memory_order_relaxed);
  return e;
}

// The tensor-core kernel over list blk.  Warps per CTA: as many as 200 KB of shared memory
// hold, at most four; CTAs per SM: what fits, so that each persistent CTA is resident.
template <int LA, int LB, int LC, int LD>
static cudaError_t launch_tc(cqg_ctx *ctx, int blk, long long n, cudaStream_t st, const DigestGroups &dg) {
  if (n == 0) return cudaSuccess;   // n < 0: count unknown on the host (graph mode)
  using D = warpmd::TcDims<LA, LB, LC, LD>;
  static std::atomic<bool> allowed[64];
  constexpr size_t per_warp = sizeof(double) * D::WARP_DOUBLES;
  constexpr int wpb_max = (int)(200u * 1024u / per_warp) < 1 ? 1 : (int)(200u * 1024u / per_warp) > 4 ? 4 : (int)(200u * 1024u / per_warp);
  cudaError_t e = allow_smem(&k_eri_tc<LA, LB, LC, LD>, per_warp * wpb_max, ctx->device, allowed);
  if (e != cudaSuccess) return e;
  const int wpb = ctx->shape_wpb[blk] > 0 ? std::min(wpb_max, ctx->shape_wpb[blk]) : wpb_max;
  const int cta = ctx->shape_cta[blk] > 0 ? ctx->shape_cta[blk]
                                          : std::max(1, (int)(220u * 1024u / (per_warp * wpb + 1024)));
  ctx->used_cta = cta;
  const long long cap = (long long)ctx->nsm * cta;
  const int blocks = (int)(n > 0 ? std::min<long long>((n + wpb - 1) / wpb, cap) : cap);
  const int bc = pair_class_c(LA, LB), kc = pair_class_c(LC, LD);
  if (!ctx->exp_have[bc] || !ctx->exp_have[kc]) return cudaErrorInvalidValue;   // no tables to read
  const Expansions X = {ctx->d_exp.p + ctx->exp_off[bc], ctx->d_exp.p + ctx->exp_off[kc], ctx->exp_prim0[bc],
                        ctx->exp_prim0[kc]};
  const int take = std::min(32, ctx->shape_qpw[blk]);
  k_eri_tc<LA, LB, LC, LD><<<blocks, 32 * wpb, per_warp * wpb, st>>>(ctx->d_qlist.p, ctx->p_range, blk,
                                                                    make_pairs(ctx), make_shells(ctx), X,
                                                                    ctx->boys_rows, dg, ctx->p_qhead, take);
  return cudaGetLastError();
}

template <int LA, int LB>
static cudaError_t launch_schwarz(cqg_ctx *ctx, Pairs P, Shells S, int beg, int end, double *Q, cudaStream_t st) {
  int n = end - beg;
  if (n <= 0) return cudaSuccess;
  if constexpr (is_warp_class(LA, LB, LA, LB)) {
    static std::atomic<bool> allowed[64];
    constexpr size_t per_warp = sizeof(double) * warpmd::WarpDims<LA, LB>::SMEM;
    constexpr int wpb = per_warp * 4 <= 200u * 1024u ? 4 : per_warp * 2 <= 200u * 1024u ? 2 : 1;
    cudaError_t e = allow_smem(&k_schwarz_warp<LA, LB>, per_warp * wpb, ctx->device, allowed);
    if (e != cudaSuccess) return e;
    k_schwarz_warp<LA, LB><<<std::min((n + wpb - 1) / wpb, ctx->nsm * 16), 32 * wpb, per_warp * wpb, st>>>(
        P, S, ctx->boys, beg, end, Q);
    return cudaGetLastError();
  } else {
    int ls = 0;   // up to a lane per primitive pair of the class's longest bra
    while (ls < 5 && (2 << ls) <= ctx->pc_np_max[pair_class_c(LA, LB)]) ++ls;
    k_schwarz<LA, LB><<<(unsigned)((((long long)n << ls) + 127) / 128), 128, 0, st>>>(P, S, ctx->boys_rows, beg, end, ls,
                                                                                  Q);
    return cudaGetLastError();
  }
}

// Expansion tables of pair class (LA LB)
template <int LA, int LB>
static cudaError_t launch_expansions(cqg_ctx *ctx) {
  constexpr int c = pair_class_c(LA, LB);
  const int beg = ctx->pc_beg[c], n = ctx->pc_beg[c + 1] - beg;
  if (n <= 0 || !ctx->exp_have[c]) return cudaSuccess;
  k_expansions<LA, LB><<<std::min((n + 3) / 4, ctx->nsm * 16), 128>>>(
      make_pairs(ctx), make_shells(ctx), beg, beg + n, ctx->exp_prim0[c], ctx->d_exp.p + ctx->exp_off[c]);
  return cudaGetLastError();
}

static inline MaskCache make_mask_cache(cqg_ctx *ctx) {
  MaskCache mc;
  mc.masks = ctx->d_masks.p;
  mc.head = ctx->p_mhead;
  mc.slot = ctx->d_mslot.p;
  mc.cap = (long long)ctx->d_masks.n;
  return mc;
}

static inline Pairs make_pairs(cqg_ctx *ctx) {
  Pairs P;
  P.sh = ctx->d_pair_sh.p;
  P.Q = ctx->d_pair_Q.p;
  P.poff = ctx->d_pair_poff.p;
  P.np = ctx->d_pair_np.p;
  P.kk = ctx->d_pair_kk.p;
  P.prim = ctx->d_prim.p;
  P.cols = ctx->d_cols.p;
  P.coff = ctx->d_pair_coff.p;
  P.Qc = ctx->d_pair_Qc.p;
  P.glead = ctx->d_glead.p;
  P.gQ = ctx->d_gQ.p;
  P.gsz = ctx->d_gsz.p;
  P.gpoff = ctx->d_gpoff.p;
  P.gnp = ctx->d_gnp.p;
  P.gwoff = ctx->d_gwoff.p;
  P.gprim = ctx->d_gprim.p;
  P.gw = ctx->d_gw.p;
  P.qmask = ctx->d_qmask.p;
  return P;
}
static inline Shells make_shells(cqg_ctx *ctx) {
  Shells S;
  S.center = ctx->d_center.p;
  S.bf = ctx->d_bf.p;
  S.mol = ctx->d_shmol.p;
  S.pf = ctx->d_pf.p;
  return S;
}
static inline Mols make_mols(cqg_ctx *ctx) {
  Mols M;
  M.nmol = ctx->nmol;
  M.shoff = ctx->d_mshoff.p;
  M.nsh = ctx->d_mnsh.p;
  M.Moff = ctx->d_mMoff.p;
  M.xoff = ctx->d_mxoff.p;
  M.nbf = ctx->d_mnbf.p;
  M.foff = ctx->d_mfoff.p;
  M.pos = ctx->d_pos.p;
  M.fsh = ctx->d_fsh.p;
  M.pidx = ctx->d_pidx.p;
  M.active = ctx->d_active.p;
  M.molbk = ctx->d_molbk.p;
  M.molgbk = ctx->d_molgbk.p;
  return M;
}

// CTAs of `kernel` (128 threads, static shared memory) resident on one SM: the default grid of
// the class kernels.  A persistent CTA beyond the resident ones starts only when a first one
// has drained the queue: it copies its Boys rows and finds no work.  (With the copy
// of load_boys: 8.59 -> 7.35 ms per (H2O)_11 cc-pVDZ build against twelve CTAs per SM.)  The count belongs to the kernel and the device
// and is asked for once.
template <typename K>
static int resident_ctas(K kernel, int threads, int device, std::atomic<int> (&known)[64]) {
  const int slot = (device >= 0 && device < 64) ? device : 0;
  int n = known[slot].load(std::memory_order_relaxed);
  if (n == 0) {
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, threads, 0) != cudaSuccess || n < 1) n = 1;
    known[slot].store(n, std::memory_order_relaxed);
  }
  return n;
}

typedef cudaError_t (*eri_launcher)(cqg_ctx *, int blk, long long n, cudaStream_t st, const DigestGroups &dg);

// One launch of the sibling-group kernel of class (LA LB|LC LD) over list blk: CTAs of 64
// threads when the list's schedule gives 2 warps per CTA, else 128.
template <int LA, int LB, int LC, int LD, typename T>
static cudaError_t launch_gc(cqg_ctx *ctx, int blk, long long n, cudaStream_t st, const DigestGroups &dg) {
  if (n == 0) return cudaSuccess;   // n < 0: count unknown on the host (graph mode)
  const int nt = ctx->shape_wpb[blk] == 2 ? 64 : kEriThreads;
  const int cta = ctx->shape_cta[blk] > 0 ? ctx->shape_cta[blk] : 4;
  ctx->used_cta = cta;
  const long long cap = (long long)ctx->nsm * cta;
  const long long nb = n > 0 ? std::min<long long>((n + nt - 1) / nt, cap) : cap;
  const int chunk = 32 * (ctx->shape_qpw[blk] > 0 ? ctx->shape_qpw[blk] : 1);
  if (nt == 64)
    k_eri_gc<LA, LB, LC, LD, T, 64><<<(unsigned)nb, 64, 0, st>>>(ctx->d_qlist.p, ctx->p_range, blk,
                                                                make_pairs(ctx), make_shells(ctx), ctx->boys_rows,
                                                                dg, ctx->p_qhead, chunk);
  else
    k_eri_gc<LA, LB, LC, LD, T, kEriThreads><<<(unsigned)nb, kEriThreads, 0, st>>>(
        ctx->d_qlist.p, ctx->p_range, blk, make_pairs(ctx), make_shells(ctx), ctx->boys_rows, dg, ctx->p_qhead,
        chunk);
  return cudaGetLastError();
}

// Class-fused schedule (eri_fused.cu): whether class (la lb|lc ld) belongs to the fused
// kernel of `tier` (1: (ss|ss) and (ps|ss), 2: every per-thread class up to (dd|dd)), and one
// launch of that kernel over the current list ranges.
bool cqg_fused_member(int tier, int la, int lb, int lc, int ld);
cudaError_t cqg_launch_fused(cqg_ctx *ctx, int tier, cudaStream_t st, const DigestGroups &dg);

template <int LA, int LB, int LC, int LD, typename T>
static cudaError_t launch_eri(cqg_ctx *ctx, int blk, long long n, cudaStream_t st, const DigestGroups &dg) {
  if (n == 0) return cudaSuccess;   // n < 0: count unknown on the host (graph mode)
  if constexpr (is_warp_class(LA, LB, LC, LD)) {   // FP32 lists too: the tensor form is FP64 throughout
    return launch_tc<LA, LB, LC, LD>(ctx, blk, n, st, dg);
  } else {
    if constexpr (is_variant_class(LA, LB, LC, LD)) {
      if (ctx->shape_var[blk] == 1) return launch_tc<LA, LB, LC, LD>(ctx, blk, n, st, dg);
    }
    constexpr int mb = EriMinBlocks<LA, LB, LC, LD>::v;
    auto kernel = [] {
      if constexpr (mb > 0) return &k_eri_jk_mb<LA, LB, LC, LD, T, mb>;
      else return &k_eri_jk<LA, LB, LC, LD, T>;
    }();
    static std::atomic<int> known[64];
    const int resident = resident_ctas(kernel, kEriThreads, ctx->device, known);
    const LaneShare share = {ctx->nsm * resident * kEriThreads, ctx->pc_np_max[pair_class_c(LC, LD)]};
    const int cta = ctx->shape_cta[blk] > 0 ? ctx->shape_cta[blk] : resident;
    ctx->used_cta = cta;
    const long long cap = (long long)ctx->nsm * cta;
    // up to 32 lanes per quartet (eri_jk_list)
    const long long nb = n > 0 ? std::min<long long>((32 * n + kEriThreads - 1) / kEriThreads, cap) : cap;
    const int chunk = 32 * (ctx->shape_qpw[blk] > 0 ? ctx->shape_qpw[blk] : 1);
    kernel<<<(unsigned)nb, kEriThreads, 0, st>>>(ctx->d_qlist.p, ctx->p_range, blk, make_pairs(ctx), make_shells(ctx),
                                                 ctx->boys_rows, dg, ctx->p_qhead, chunk, share);
    return cudaGetLastError();
  }
}

