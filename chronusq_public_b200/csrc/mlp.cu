// Kernels of the learned initial-density model: a small MLP trained and evaluated on the
// GPU with BF16 operands and FP32 accumulation.
//
//   k_gemm_bf16 : C[m][n] (+)= sum_k A(m,k) B(n,k), A and B BF16 with arbitrary strides
//                 (transposes are strides), on the tensor cores: mma.sync m16n8k16 BF16 x
//                 BF16 -> FP32 over block tiles that come through a ring of asynchronous
//                 copies; optional fused epilogue Z = C + bias (FP32) and Y = SiLU(Z) (BF16).
//                 or, backward, dZ = C * SiLU'(Z) (BF16, the next GEMMs' operand) and its column sums
//   k_gemm_parts: C[m][n] += sum_k A(m,k) B(n,k), the parts of a split K added with atomics (the
//                 gradient of a layer's input)
//   k_dz_colsum : a layer's dZ in BF16, through SiLU' for the hidden ones, and db[n] = sum_m dZ[m][n]
//   k_mse       : masked squared error, its gradient, and the loss sum
//   k_adam      : Adam step on FP32 master weights, BF16 copy for the next pass, all tensors of
//                 the network in one launch
//   k_silu_bwd, k_to_bf16 : the elementwise parts alone (cqg_mlp_silu_bwd, cqg_mlp_to_bf16)
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>
#include <utility>

#include "../../include/cqgpu.h"

namespace {

constexpr int GM = 128, GN = 128, GK = 32;   // large block tile, k per tile

__device__ __forceinline__ float silu(float z) { return z / (1.0f + __expf(-z)); }
__device__ __forceinline__ float silu_grad(float z) {
  const float s = 1.0f / (1.0f + __expf(-z));
  return s * (1.0f + z * (1.0f - s));
}

// D += A B for one 16 x 8 x 16 tile (A row-major 16 x 16, B column-major 16 x 8, BF16
// operands, FP32 accumulators).  Fragments (g = lane / 4, t = lane % 4):
//   a[0] = A[g][2t..2t+1], a[1] = A[g+8][2t..], a[2] = A[g][2t+8..], a[3] = A[g+8][2t+8..]
//   b[0] = B[2t..2t+1][g], b[1] = B[2t+8..2t+9][g]
//   d[0..1] = D[g][2t..2t+1], d[2..3] = D[g+8][2t..2t+1]
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// How an operand tile lies in shared memory: as [row][k] (k contiguous in memory, or any
// strides, staged element by element) or as [k][row] (rows contiguous); ldmatrix, transposing
// for the second, gives the same fragments from either.
enum { TILE_K = 0, TILE_R = 1, TILE_ANY = 2 };
constexpr int GP = GK + 8;   // padded row of a [row][k] tile: 80 bytes, no ldmatrix bank conflicts

__device__ __forceinline__ void cp_async16(unsigned dst, const void *src, int bytes) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void ldmatrix_x4(uint32_t (&r)[4], unsigned addr, bool trans) {
  if (trans)
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
  else
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr));
}

// A thread's 16-byte copies of one operand's tiles, ROWS rows from r0 x GK of k, of
// X(r, k) = X[r * sr + k * sk] (zero outside nrows x K).  Addresses and row bounds are worked
// out once: the products of a training step are short, and five tiles' worth of index
// arithmetic before the first copy was a third of their time.
template <int ROWS, int NT>
struct TileCopy {
  static constexpr int NC = ROWS * (GK / 8) / NT;
  const __nv_bfloat16 *src[NC];
  long long step;    // elements from one tile to the next
  unsigned dst[NC];  // offset in the tile
  int most[NC], k[NC], mul;
  __device__ __forceinline__ TileCopy(const __nv_bfloat16 *X, long long sr, long long sk, int r0, int nrows, int kb,
                                      int mode) {
    const bool kin = mode == TILE_K;
    step = kin ? GK : GK * sk;
    mul = kin ? 2 : 16;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int e = c * NT + threadIdx.x;
      const int r = r0 + (kin ? e / (GK / 8) : e % (ROWS / 8) * 8);
      k[c] = kin ? e % (GK / 8) * 8 : e / (ROWS / 8);
      dst[c] = 2 * (kin ? (r - r0) * GP + k[c] : k[c] * (ROWS + 8) + r - r0);
      most[c] = max(0, min(16, (nrows - r) * (kin ? 16 : 2)));
      src[c] = most[c] ? X + r * sr + (kb + k[c]) * sk : X;
    }
  }
  // tile kt of k [kb + kt * GK, ...), `left` = K - that
  __device__ __forceinline__ void start(unsigned tile, int kt, int left) const {
#pragma unroll
    for (int c = 0; c < NC; ++c) {
      const int bytes = min(most[c], max(0, (left - k[c]) * mul));
      cp_async16(tile + dst[c], bytes ? src[c] + kt * step : src[c], bytes);
    }
  }
};

// The same tile, [row][k], for operands that 16-byte copies cannot take; complete on return.
template <int ROWS, int NT>
__device__ __forceinline__ void stage_any(const __nv_bfloat16 *__restrict__ X, long long sr, long long sk, int r0,
                                          int nrows, int k0, int K, __nv_bfloat16 *S) {
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  const bool k_fast = sk <= sr;   // the smaller stride across threads
  constexpr int U = 8;            // loads in flight
#pragma unroll 1
  for (int e0 = threadIdx.x; e0 < ROWS * GK; e0 += NT * U) {
    __nv_bfloat16 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * NT;
      const int r = r0 + (k_fast ? e / GK : e % ROWS), k = k0 + (k_fast ? e % GK : e / ROWS);
      v[u] = (r < nrows && k < K) ? X[(long long)r * sr + (long long)k * sk] : zero;
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int e = e0 + u * NT;
      S[(k_fast ? e / GK : e % ROWS) * GP + (k_fast ? e % GK : e / ROWS)] = v[u];
    }
  }
}

// One product of a launch.  split: the block reduces k in [z kchunk, (z + 1) kchunk) and adds
// its partial tile to C with atomics (C zeroed by the caller), no epilogue.  dact: the
// epilogue is the backward step through the layer below, Y = bf16(value * SiLU'(dact)) and its
// column sums added to db; C is not written.
struct Gemm {
  const __nv_bfloat16 *A, *B;
  long long sam, sak, sbn, sbk, ldc, ldy;
  float *C;
  const float *bias, *dact;
  float *db;
  __nv_bfloat16 *Y;
  int M, N, K, kchunk, nbn, nbm, nbz;
  unsigned char amode, bmode, act, accumulate, split, pairs;   // pairs: C, Y and dact take 2-wide accesses
  __host__ int blocks() const { return nbn * nbm * nbz; }
};

// Block tile BM x BN (BM, BN multiples of 32), warps of 32 x WN output each (WN = 64 or 32):
// (BM / 32) x (BN / WN) warps; per 16-wide k step a warp issues 2 x (WN / 8) tensor-core
// tiles.  128 x 128 with 8 warps of 32 x 64 for large problems, 64 x 64 with 4 warps of
// 32 x 32 when the large tiles would leave most of the 148 SMs idle.  A training step's
// products (2048 x 256 x 256) are chains of load latencies, not arithmetic: tiles of 32 k come
// through a ring of STAGES asynchronous copies, and two products (the weight gradients of two
// layers, or one with the gradient of its layer's input) share a launch, the first `blocks0`
// blocks for g0.
// Measured, 2048 rows, width 256: a layer forward 17 us cold (9.1 us back to back) from one
// synchronous tile at a time before.
template <int BM, int BN, int WN, int STAGES>
__global__ void __launch_bounds__((BM / 32) * (BN / WN) * 32, BM == 64 ? 3 : 2)
    k_gemm_bf16(const __grid_constant__ Gemm g0, const __grid_constant__ Gemm g1, int blocks0) {
  constexpr int NWM = BM / 32, NJ = WN / 8, NT = NWM * (BN / WN) * 32;
  constexpr int ASZ = BM * GP, BSZ = BN * GP;   // [k][row] tiles, GK x (rows + 8), fit as well
  static_assert(GK * (BM + 8) <= ASZ && GK * (BN + 8) <= BSZ, "tile buffers");
  extern __shared__ __align__(16) __nv_bfloat16 tiles[];
  const bool first = (int)blockIdx.x < blocks0;
  const Gemm p = first ? g0 : g1;
  const int blk = first ? blockIdx.x : blockIdx.x - blocks0;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp % NWM) * 32, wn = (warp / NWM) * WN;
  const int M = p.M, N = p.N, K = p.K;
  const int n0 = blk % p.nbn * BN, m0 = blk / p.nbn % p.nbm * BM, z = blk / (p.nbn * p.nbm);
  const int g = lane >> 2, t = lane & 3;
  float acc[2][NJ][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  const int kb = p.split ? z * p.kchunk : 0, ke = p.split ? min(K, kb + p.kchunk) : K;
  const int nkt = (ke - kb + GK - 1) / GK;
  const __nv_bfloat16 *A = p.A, *B = p.B;
  const long long sam = p.sam, sak = p.sak, sbn = p.sbn, sbk = p.sbk;
  const int amode = p.amode, bmode = p.bmode;
  const TileCopy<BM, NT> ca(A, sam, sak, m0, M, kb, amode);
  const TileCopy<BN, NT> cb(B, sbn, sbk, n0, N, kb, bmode);
  auto issue = [&](int kt) {
    if (kt < nkt) {
      __nv_bfloat16 *As = tiles + (kt % STAGES) * (ASZ + BSZ), *Bs = As + ASZ;
      const int k0 = kb + kt * GK;
      if (amode != TILE_ANY)
        ca.start((unsigned)__cvta_generic_to_shared(As), kt, ke - k0);
      else
        stage_any<BM, NT>(A, sam, sak, m0, M, k0, ke, As);
      if (bmode != TILE_ANY)
        cb.start((unsigned)__cvta_generic_to_shared(Bs), kt, ke - k0);
      else
        stage_any<BN, NT>(B, sbn, sbk, n0, N, k0, ke, Bs);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
#pragma unroll 1
  for (int kt = 0; kt < STAGES - 1; ++kt) issue(kt);
  // the lane's ldmatrix row and column within a 16 x 16 block of either kind of tile
  const int j8 = lane >> 3, l8 = lane & 7;
  const bool at = amode == TILE_R, bt = bmode == TILE_R;
#pragma unroll 1
  for (int kt = 0; kt < nkt; ++kt) {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
    __syncthreads();   // tile kt is here, and tile kt - 1 has been used by every warp
    issue(kt + STAGES - 1);
    const __nv_bfloat16 *As = tiles + (kt % STAGES) * (ASZ + BSZ), *Bs = As + ASZ;
#pragma unroll
    for (int ks = 0; ks < GK; ks += 16) {
      uint32_t af[2][4], bf[NJ][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const __nv_bfloat16 *q = at ? As + (ks + l8 + (j8 >> 1) * 8) * (BM + 8) + wm + i * 16 + (j8 & 1) * 8
                                    : As + (wm + i * 16 + l8 + (j8 & 1) * 8) * GP + ks + (j8 >> 1) * 8;
        ldmatrix_x4(af[i], (unsigned)__cvta_generic_to_shared(q), at);
      }
#pragma unroll
      for (int j = 0; j < NJ; j += 2) {
        const __nv_bfloat16 *q = bt ? Bs + (ks + l8 + (j8 & 1) * 8) * (BN + 8) + wn + j * 8 + (j8 >> 1) * 8
                                    : Bs + (wn + j * 8 + l8 + (j8 >> 1) * 8) * GP + ks + (j8 & 1) * 8;
        uint32_t r[4];
        ldmatrix_x4(r, (unsigned)__cvta_generic_to_shared(q), bt);
        bf[j][0] = r[0];
        bf[j][1] = r[1];
        bf[j + 1][0] = r[2];
        bf[j + 1][1] = r[3];
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) mma_16816(acc[i][j], af[i], bf[j]);
    }
  }
  float *C = p.C;
  __nv_bfloat16 *Y = p.Y;
  const long long ldc = p.ldc, ldy = p.ldy;
  const bool pairs = p.pairs;
  if (p.split) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int m = m0 + wm + i * 16 + g + h * 8, n = n0 + wn + j * 8 + 2 * t;
          if (m >= M || n >= N) continue;
          float *c = C + m * ldc + n;
          if (pairs && n + 1 < N) {
            atomicAdd(reinterpret_cast<float2 *>(c), make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]));
          } else {
            atomicAdd(c, acc[i][j][2 * h]);
            if (n + 1 < N) atomicAdd(c + 1, acc[i][j][2 * h + 1]);
          }
        }
    return;
  }
  // the other epilogues from shared memory, four rows of two neighbouring columns a thread at
  // a time: short code (unrolled over the accumulators, instruction misses were 2 us of a
  // launch) with its loads in flight
  constexpr int SP = BN + 8, CG = BN / 2, RSTEP = NT / CG, U = 4;
  static_assert(BM * SP * 4 <= STAGES * (ASZ + BSZ) * 2 && BM % (RSTEP * U) == 0, "epilogue tile");
  float *S = reinterpret_cast<float *>(tiles);
  asm volatile("cp.async.wait_group 0;\n" ::: "memory");
  __syncthreads();
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int h = 0; h < 2; ++h)
        *reinterpret_cast<float2 *>(S + (wm + i * 16 + g + h * 8) * SP + wn + j * 8 + 2 * t) =
            make_float2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
  __syncthreads();
  const int c2 = threadIdx.x % CG * 2, n = n0 + c2;
  if (n >= N) return;
  const bool two = n + 1 < N, both = pairs && two;
  const float *bias = p.bias, *dact = p.dact;
  const bool act = p.act;
  const float *src = dact ? dact : p.accumulate ? C : nullptr;   // the activation's argument, or what C holds
  const long long lds = dact ? ldy : ldc;
  const float b0 = bias ? bias[n] : 0.f, b1 = bias && two ? bias[n + 1] : 0.f;
  float s0 = 0.f, s1 = 0.f;
#pragma unroll 1
  for (int r0 = threadIdx.x / CG; r0 < min(BM, M - m0); r0 += RSTEP * U) {
    float2 d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * RSTEP;
      d[u] = make_float2(0.f, 0.f);
      if (src && m0 + r < M) {
        const float *q = src + (m0 + r) * lds + n;
        if (both)
          d[u] = *reinterpret_cast<const float2 *>(q);
        else
          d[u] = make_float2(q[0], two ? q[1] : 0.f);
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * RSTEP;
      if (m0 + r >= M) break;
      const float2 v = *reinterpret_cast<const float2 *>(S + r * SP + c2);
      const float z0 = v.x + b0 + (dact ? 0.f : d[u].x), z1 = v.y + b1 + (dact ? 0.f : d[u].y);
      __nv_bfloat16 y0, y1;
      if (dact) {
        y0 = __float2bfloat16(z0 * silu_grad(d[u].x));
        y1 = __float2bfloat16(z1 * silu_grad(d[u].y));
        s0 += __bfloat162float(y0);
        s1 += __bfloat162float(y1);
      } else {
        float *c = C + (m0 + r) * ldc + n;
        if (both) {
          *reinterpret_cast<float2 *>(c) = make_float2(z0, z1);
        } else {
          c[0] = z0;
          if (two) c[1] = z1;
        }
        if (!Y) continue;
        y0 = __float2bfloat16(act ? silu(z0) : z0);
        y1 = __float2bfloat16(act ? silu(z1) : z1);
      }
      __nv_bfloat16 *y = Y + (m0 + r) * ldy + n;
      if (both) {
        *reinterpret_cast<__nv_bfloat162 *>(y) = __halves2bfloat162(y0, y1);
      } else {
        y[0] = y0;
        if (two) y[1] = y1;
      }
    }
  }
  if (dact) {
    atomicAdd(p.db + n, s0);
    if (two) atomicAdd(p.db + n + 1, s1);
  }
}

// Rows [r0, r0 + 64) x k [k0, k0 + 32) of X(r, k) = X[r * sr + k * sk] into S[row][k] (zero outside
// nrows x K).  Rows or k contiguous and 16-byte aligned: 8-element loads; anything else element
// by element.
constexpr int kPartTile = 64;
static_assert(148 * kPartTile * kPartTile == CQG_MLP_DX_MAX, "fewer than 148 tiles (k_parts) are split");
__device__ __forceinline__ void stage_part(const __nv_bfloat16 *__restrict__ X, long long sr, long long sk, int r0,
                                           int nrows, int k0, int K, bool vec_k, bool vec_r,
                                           __nv_bfloat16 (*S)[GP]) {
  const int tid = threadIdx.x, nth = blockDim.x;
  const __nv_bfloat16 zero = __float2bfloat16(0.f);
  if (vec_k) {                 // sk == 1, sr % 8 == 0, K % 8 == 0, X 16-byte aligned
    for (int e = tid; e < kPartTile * (GK / 8); e += nth) {
      const int rr = e / (GK / 8), kv = (e % (GK / 8)) * 8;
      const int r = r0 + rr, k = k0 + kv;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (r < nrows && k < K) v = *reinterpret_cast<const uint4 *>(X + (long long)r * sr + k);
      *reinterpret_cast<uint4 *>(&S[rr][kv]) = v;
    }
  } else if (vec_r) {          // sr == 1, sk % 8 == 0, nrows % 8 == 0, X 16-byte aligned
    for (int e = tid; e < GK * (kPartTile / 8); e += nth) {
      const int kk = e / (kPartTile / 8), rv = (e % (kPartTile / 8)) * 8;
      const int r = r0 + rv, k = k0 + kk;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (r < nrows && k < K) v = *reinterpret_cast<const uint4 *>(X + r + (long long)k * sk);
      const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
      for (int i = 0; i < 8; ++i) S[rv + i][kk] = h[i];
    }
  } else if (sk <= sr) {       // k varies fastest across threads
    for (int e = tid; e < kPartTile * GK; e += nth) {
      const int rr = e / GK, kk = e % GK;
      const int r = r0 + rr, k = k0 + kk;
      S[rr][kk] = (r < nrows && k < K) ? X[(long long)r * sr + (long long)k * sk] : zero;
    }
  } else {                     // rows vary fastest across threads
    for (int e = tid; e < kPartTile * GK; e += nth) {
      const int kk = e / kPartTile, rr = e % kPartTile;
      const int r = r0 + rr, k = k0 + kk;
      S[rr][kk] = (r < nrows && k < K) ? X[(long long)r * sr + (long long)k * sk] : zero;
    }
  }
}

// C[m][n] += sum_k A(m,k) B(n,k) over k [blockIdx.z kchunk, + kchunk), 64 x 64 tiles of four
// warps, one tile of k in shared memory at a time, C zeroed by the caller: the gradient of a
// layer's input when its product is split.  The parts of one element add up in the order in
// which their blocks finish, and the next dZ is that sum in BF16: a last bit that differs turns
// one BF16 rounding in some 2^16, 2^-8 of an element, and the layers below multiply it.  Which
// order is usual depends on how long the blocks run.  Measured, 2048 rows, width 256, four of
// these products in a pass, median of the largest relative change of a weight gradient: two
// runs of the layer-by-layer pass with this kernel 1.0e-5; cqg_mlp_backward with it against
// that pass 1.6e-5; with k_gemm_bf16 and atomics 3.7e-5 to 4.6e-5, its blocks being three times
// as fast; with the parts in any one fixed order 3.2e-5 to 7.4e-5.  (Against 64 bits all are
// the same, 1e-3: BF16 operands.)  So the products that are split keep this kernel, 17 us each
// where k_gemm_bf16 takes 9, and a training step keeps its gradients.
__global__ void __launch_bounds__(128)
    k_gemm_parts(const __nv_bfloat16 *__restrict__ A, long long sam, long long sak, const __nv_bfloat16 *__restrict__ B,
                 long long sbn, long long sbk, float *__restrict__ C, long long ldc, int M, int N, int K, int kchunk) {
  constexpr int NJ = 4;
  __shared__ __align__(16) __nv_bfloat16 As[kPartTile][GP];
  __shared__ __align__(16) __nv_bfloat16 Bs[kPartTile][GP];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp % 2) * 32, wn = (warp / 2) * 32;
  const int m0 = blockIdx.y * kPartTile, n0 = blockIdx.x * kPartTile;
  const int g = lane >> 2, t = lane & 3;
  const bool a16 = (reinterpret_cast<uintptr_t>(A) & 15) == 0, b16 = (reinterpret_cast<uintptr_t>(B) & 15) == 0;
  const bool avk = a16 && sak == 1 && sam % 8 == 0 && K % 8 == 0;
  const bool avr = a16 && !avk && sam == 1 && sak % 8 == 0 && M % 8 == 0;
  const bool bvk = b16 && sbk == 1 && sbn % 8 == 0 && K % 8 == 0;
  const bool bvr = b16 && !bvk && sbn == 1 && sbk % 8 == 0 && N % 8 == 0;
  float acc[2][NJ][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  const int kb = blockIdx.z * kchunk, ke = min(K, kb + kchunk);
  for (int k0 = kb; k0 < ke; k0 += GK) {
    stage_part(A, sam, sak, m0, M, k0, ke, avk, avr, As);
    stage_part(B, sbn, sbk, n0, N, k0, ke, bvk, bvr, Bs);
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < GK; ks += 16) {
      uint32_t af[2][4], bf[NJ][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = wm + i * 16 + g;
        af[i][0] = *reinterpret_cast<const uint32_t *>(&As[r][ks + 2 * t]);
        af[i][1] = *reinterpret_cast<const uint32_t *>(&As[r + 8][ks + 2 * t]);
        af[i][2] = *reinterpret_cast<const uint32_t *>(&As[r][ks + 2 * t + 8]);
        af[i][3] = *reinterpret_cast<const uint32_t *>(&As[r + 8][ks + 2 * t + 8]);
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int c = wn + j * 8 + g;
        bf[j][0] = *reinterpret_cast<const uint32_t *>(&Bs[c][ks + 2 * t]);
        bf[j][1] = *reinterpret_cast<const uint32_t *>(&Bs[c][ks + 2 * t + 8]);
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) mma_16816(acc[i][j], af[i], bf[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int m = m0 + wm + i * 16 + g + (q >> 1) * 8, n = n0 + wn + j * 8 + 2 * t + (q & 1);
        if (m < M && n < N) atomicAdd(C + m * ldc + n, acc[i][j][q]);
      }
}

__global__ void k_silu_bwd(const float *__restrict__ dY, const float *__restrict__ Z, __nv_bfloat16 *__restrict__ dZ,
                           long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) dZ[i] = __float2bfloat16(dY[i] * silu_grad(Z[i]));
}

__global__ void k_to_bf16(const float *__restrict__ x, __nv_bfloat16 *__restrict__ y, long long n) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i < n) y[i] = __float2bfloat16(x[i]);
}

// dZ = dY in BF16, times SiLU'(Z) where Z is given (dY null: `in` holds dZ already), and its
// column sums, db[n] += sum_m dZ[m][n] (db zeroed by the caller).  A block takes 32 columns x
// kColRows rows, a warp one row at a time (coalesced); one atomic per column and block.  The two
// as kernels of their own took 4 + 17 us per layer of 2048 x 256.
constexpr int kColRows = 64;
__global__ void __launch_bounds__(256) k_dz_colsum(const float *__restrict__ dY,
                                                   const float *__restrict__ Z,
                                                   const __nv_bfloat16 *__restrict__ in,
                                                   __nv_bfloat16 *__restrict__ out, int M, int N,
                                                   float *__restrict__ db) {
  __shared__ float part[8][33];
  const int c = threadIdx.x & 31, rg = threadIdx.x >> 5;
  const int n = blockIdx.y * 32 + c;
  const int m0 = blockIdx.x * kColRows, m1 = (int)min((long long)M, (long long)m0 + kColRows);
  float s = 0.f;
  if (n < N) {
#pragma unroll 4
    for (int m = m0 + rg; m < m1; m += 8) {
      const long long e = (long long)m * N + n;
      __nv_bfloat16 v;
      if (in) {
        v = in[e];
      } else {
        v = __float2bfloat16(Z ? dY[e] * silu_grad(Z[e]) : dY[e]);
        out[e] = v;
      }
      s += __bfloat162float(v);
    }
  }
  part[rg][c] = s;
  __syncthreads();
  if (rg == 0 && n < N) {
    float t = 0.f;
#pragma unroll
    for (int k = 0; k < 8; ++k) t += part[k][c];
    atomicAdd(db + n, t);
  }
}

// loss = sum mask*(pred-target)^2 / count ; dpred = 2 mask (pred-target) / count
__global__ void k_mse(const float *__restrict__ pred, const float *__restrict__ target, const float *__restrict__ mask,
                      long long n, float inv_count, float *__restrict__ dpred, float *__restrict__ loss) {
  __shared__ float red[256];
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  float l = 0.f;
  if (i < n) {
    const float w = mask ? mask[i] : 1.f;
    const float d = pred[i] - target[i];
    dpred[i] = 2.f * w * d * inv_count;
    l = w * d * d * inv_count;
  }
  red[threadIdx.x] = l;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicAdd(loss, red[0]);
}

// One Adam step of up to kAdamTensors tensors (blockIdx.y), bias-corrected, decoupled weight
// decay folded into the gradient, with an optional BF16 copy.  The learning rate and the two
// bias corrections 1 - b^step come from device memory when `hyper` is given (a captured step
// is then replayed with a schedule that changes from step to step).
constexpr int kAdamTensors = 16;
struct AdamTensors {
  float *w[kAdamTensors], *m1[kAdamTensors], *m2[kAdamTensors];
  const float *g[kAdamTensors];
  __nv_bfloat16 *wbf[kAdamTensors];
  long long n[kAdamTensors];
  float wd[kAdamTensors];
};
__global__ void __launch_bounds__(256) k_adam(AdamTensors ts, const float *__restrict__ hyper, float lr, float bc1,
                                              float bc2, float b1, float b2, float eps) {
  const int k = blockIdx.y;
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= ts.n[k]) return;
  if (hyper) {
    lr = hyper[0];
    bc1 = hyper[1];
    bc2 = hyper[2];
  }
  float *w = ts.w[k], *m1 = ts.m1[k], *m2 = ts.m2[k];
  const float w0 = w[i], gi = ts.g[k][i] + ts.wd[k] * w0;
  const float a = b1 * m1[i] + (1.f - b1) * gi;
  const float b = b2 * m2[i] + (1.f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = b;
  const float w1 = w0 - lr * (a / bc1) / (sqrtf(b / bc2) + eps);
  w[i] = w1;
  if (ts.wbf[k]) ts.wbf[k][i] = __float2bfloat16(w1);
}

// Shared memory above the default 48 KB, asked for once per kernel and device.
template <typename K>
cudaError_t allow_tiles(K kernel, int bytes, std::atomic<bool> (&done)[64]) {
  int device = 0;
  cudaError_t e = cudaGetDevice(&device);
  if (e != cudaSuccess) return e;
  const int slot = device < 64 ? device : 0;
  if (device < 64 && done[slot].load(std::memory_order_relaxed)) return cudaSuccess;
  e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
  if (e == cudaSuccess) done[slot].store(true, std::memory_order_relaxed);
  return e;
}

constexpr int kBigStages = 4, kSmallStages = 6;
constexpr int kBigSmem = kBigStages * (GM + GN) * GP * 2, kSmallSmem = kSmallStages * (64 + 64) * GP * 2;

Gemm gemm_of(const void *A, long long sam, long long sak, const void *B, long long sbn, long long sbk, float *C,
             long long ldc, int M, int N, int K) {
  // 16-byte copies need 16-byte aligned rows (of k or of rows)
  auto mode = [](const void *p, long long sr, long long sk) {
    if ((reinterpret_cast<uintptr_t>(p) & 15) != 0) return TILE_ANY;
    return sk == 1 && sr % 8 == 0 ? TILE_K : sr == 1 && sk % 8 == 0 ? TILE_R : TILE_ANY;
  };
  Gemm g = {};
  g.A = (const __nv_bfloat16 *)A;
  g.B = (const __nv_bfloat16 *)B;
  g.sam = sam;
  g.sak = sak;
  g.sbn = sbn;
  g.sbk = sbk;
  g.amode = mode(A, sam, sak);
  g.bmode = mode(B, sbn, sbk);
  g.C = C;
  g.ldc = ldc;
  g.M = M;
  g.N = N;
  g.K = K;
  return g;
}

// Two waves of 148 SMs or more of large tiles.
bool big_tiles(int M, int N) { return (long long)((N + GN - 1) / GN) * ((M + GM - 1) / GM) >= 296; }

void set_pairs(Gemm &g) {
  auto aligned = [](const void *p, int bytes) { return (reinterpret_cast<uintptr_t>(p) & (bytes - 1)) == 0; };
  g.pairs = (!g.C || (g.ldc % 2 == 0 && aligned(g.C, 8))) && (!g.Y || (g.ldy % 2 == 0 && aligned(g.Y, 4))) &&
            (!g.dact || (g.ldy % 2 == 0 && aligned(g.dact, 8)));
}

void tile_by(Gemm &g, int bm, int bn) {
  g.nbn = (g.N + bn - 1) / bn;
  g.nbm = (g.M + bm - 1) / bm;
  g.nbz = 1;
}

// Few 64 x 64 output tiles and a long reduction (weight gradients: K = batch rows): K split so
// that about two waves of blocks run, in parts of `least` or more; the part, or 0 for one.
int k_parts(int M, int N, int K, int least) {
  const long long tiles = (long long)((N + 63) / 64) * ((M + 63) / 64);
  if (tiles >= 148 || K < 128) return 0;
  const int splits = (int)std::min<long long>(std::min<long long>((296 + tiles - 1) / tiles, K / least), 64);
  return splits > 1 ? ((K + splits - 1) / splits + GK - 1) / GK * GK : 0;
}

void split_k(Gemm &g) {
  g.kchunk = k_parts(g.M, g.N, g.K, GK);
  if (g.kchunk > 0) {
    g.split = 1;
    g.nbz = (g.K + g.kchunk - 1) / g.kchunk;
  }
}

cqg_status launch_big(const Gemm &g, cudaStream_t st) {
  static std::atomic<bool> allowed[64];
  if (allow_tiles(&k_gemm_bf16<GM, GN, 64, kBigStages>, kBigSmem, allowed) != cudaSuccess) return CQG_ERR_CUDA;
  k_gemm_bf16<GM, GN, 64, kBigStages><<<g.blocks(), 256, kBigSmem, st>>>(g, g, g.blocks());
  return CQG_OK;
}

cqg_status launch_small(const Gemm &g, const Gemm *second, cudaStream_t st) {
  static std::atomic<bool> allowed[64];
  if (allow_tiles(&k_gemm_bf16<64, 64, 32, kSmallStages>, kSmallSmem, allowed) != cudaSuccess) return CQG_ERR_CUDA;
  const int n = g.blocks() + (second ? second->blocks() : 0);
  k_gemm_bf16<64, 64, 32, kSmallStages><<<n, 128, kSmallSmem, st>>>(g, second ? *second : g, g.blocks());
  return CQG_OK;
}

inline unsigned nblk(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

extern "C" {

cqg_status cqg_mlp_gemm_bf16(const void *A, long long sam, long long sak, const void *B, long long sbn, long long sbk,
                             float *C, long long ldc, int M, int N, int K, const float *bias, void *Y, long long ldy,
                             int act, int accumulate, void *stream) {
  if (!A || !B || !C || M < 0 || N < 0 || K < 0) return CQG_ERR_BAD_ARG;
  if (M == 0 || N == 0) return CQG_OK;
  cudaStream_t st = (cudaStream_t)stream;
  Gemm g = gemm_of(A, sam, sak, B, sbn, sbk, C, ldc, M, N, K);
  g.bias = bias;
  g.Y = (__nv_bfloat16 *)Y;
  g.ldy = ldy;
  g.act = act != 0;
  g.accumulate = accumulate != 0;
  set_pairs(g);
  const bool big = big_tiles(M, N);
  if ((M + (big ? GM : 64) - 1) / (big ? GM : 64) > 65535) return CQG_ERR_BAD_ARG;
  cqg_status s;
  if (big) {
    tile_by(g, GM, GN);
    s = launch_big(g, st);
  } else {
    tile_by(g, 64, 64);
    if (!bias && !Y) split_k(g);
    if (g.split && !accumulate &&
        cudaMemset2DAsync(C, ldc * sizeof(float), 0, N * sizeof(float), M, st) != cudaSuccess)
      return CQG_ERR_CUDA;
    s = launch_small(g, nullptr, st);
  }
  if (s != CQG_OK) return s;
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_silu_bwd(const float *dY, const float *Z, void *dZ, long long n, void *stream) {
  if (n <= 0) return CQG_OK;
  k_silu_bwd<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(dY, Z, (__nv_bfloat16 *)dZ, n);
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_to_bf16(const float *x, void *y, long long n, void *stream) {
  if (n <= 0) return CQG_OK;
  k_to_bf16<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(x, (__nv_bfloat16 *)y, n);
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_colsum(const void *dZ, int M, int N, float *db, void *stream) {
  if (N <= 0) return CQG_OK;
  if (cudaMemsetAsync(db, 0, (size_t)N * sizeof(float), (cudaStream_t)stream) != cudaSuccess) return CQG_ERR_CUDA;
  if (M <= 0) return CQG_OK;
  if ((M + 255) / 256 > 65535 || (N + 31) / 32 > 65535) return CQG_ERR_BAD_ARG;
  dim3 grid((M + kColRows - 1) / kColRows, (N + 31) / 32);
  k_dz_colsum<<<grid, 256, 0, (cudaStream_t)stream>>>(nullptr, nullptr, (const __nv_bfloat16 *)dZ, nullptr, M, N, db);
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_mse(const float *pred, const float *target, const float *mask, long long n, float inv_count,
                       float *dpred, float *loss, void *stream) {
  if (n <= 0) return CQG_OK;
  k_mse<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(pred, target, mask, n, inv_count, dpred, loss);
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_adam_tensors(int nt, float *const *w, const float *const *g, float *const *m1, float *const *m2,
                                const long long *n, const float *weight_decay, void *const *wbf, const float *hyper,
                                float lr, float b1, float b2, float eps, int step, void *stream) {
  if (nt <= 0 || !w || !g || !m1 || !m2 || !n || !weight_decay || !wbf || (!hyper && step < 1))
    return CQG_ERR_BAD_ARG;
  for (int k = 0; k < nt; ++k)
    if (n[k] <= 0) return CQG_ERR_BAD_ARG;
  const float bc1 = hyper ? 1.f : 1.f - powf(b1, (float)step), bc2 = hyper ? 1.f : 1.f - powf(b2, (float)step);
  for (int k0 = 0; k0 < nt; k0 += kAdamTensors) {
    AdamTensors ts = {};
    const int m = std::min(kAdamTensors, nt - k0);
    long long most = 0;
    for (int k = 0; k < m; ++k) {
      ts.w[k] = w[k0 + k];
      ts.g[k] = g[k0 + k];
      ts.m1[k] = m1[k0 + k];
      ts.m2[k] = m2[k0 + k];
      ts.wbf[k] = (__nv_bfloat16 *)wbf[k0 + k];
      ts.n[k] = n[k0 + k];
      ts.wd[k] = weight_decay[k0 + k];
      most = std::max(most, ts.n[k]);
    }
    k_adam<<<dim3(nblk(most, 256), m), 256, 0, (cudaStream_t)stream>>>(ts, hyper, lr, bc1, bc2, b1, b2, eps);
  }
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_adam(float *w, const float *g, float *m1, float *m2, long long n, float lr, float b1, float b2,
                        float eps, int step, float weight_decay, void *wbf, void *stream) {
  if (step < 1) return CQG_ERR_BAD_ARG;
  return cqg_mlp_adam_tensors(1, &w, &g, &m1, &m2, &n, &weight_decay, &wbf, nullptr, lr, b1, b2, eps, step, stream);
}

cqg_status cqg_mlp_adam_dev(float *w, const float *g, float *m1, float *m2, long long n, const float *hyper,
                            float b1, float b2, float eps, float weight_decay, void *wbf, void *stream) {
  if (!hyper) return CQG_ERR_BAD_ARG;
  return cqg_mlp_adam_tensors(1, &w, &g, &m1, &m2, &n, &weight_decay, &wbf, hyper, 0.f, b1, b2, eps, 0, stream);
}

cqg_status cqg_mlp_forward(int nl, const int *dims, int M, const void *X, const void *const *W, const float *const *b,
                           float *const *Z, void *const *Y, void *stream) {
  if (nl <= 0 || !dims || M < 0 || !X || !W || !b || !Z || !Y) return CQG_ERR_BAD_ARG;
  const void *h = X;
  for (int i = 0; i < nl; ++i) {
    const int K = dims[i], N = dims[i + 1];
    const bool last = i == nl - 1;
    const cqg_status st = cqg_mlp_gemm_bf16(h, K, 1, W[i], K, 1, Z[i], N, M, N, K, b[i], last ? nullptr : Y[i], N,
                                            last ? 0 : 1, 0, stream);
    if (st != CQG_OK) return st;
    h = Y[i];
  }
  return CQG_OK;
}

cqg_status cqg_mlp_backward(int nl, const int *dims, int M, const float *dout, const void *const *H,
                            const float *const *Z, const void *const *W, void *dZ0, void *dZ1, float *dX,
                            float *grads, void *stream) {
  if (nl <= 0 || !dims || M < 0 || !dout || !H || !Z || !W || !dZ0 || !dZ1 || !dX || !grads) return CQG_ERR_BAD_ARG;
  if ((M + GM - 1) / GM > 65535) return CQG_ERR_BAD_ARG;   // as cqg_mlp_gemm_bf16
  cudaStream_t st = (cudaStream_t)stream;
  long long nw = 0, nb = 0;
  for (int i = 0; i < nl; ++i) {
    if (dims[i] <= 0 || dims[i + 1] <= 0) return CQG_ERR_BAD_ARG;
    nw += (long long)dims[i] * dims[i + 1];
    nb += dims[i + 1];
  }
  // weight gradients of the layers, then bias gradients: all are added into zeros
  if (cudaMemsetAsync(grads, 0, (size_t)(nw + nb) * sizeof(float), st) != cudaSuccess) return CQG_ERR_CUDA;
  if (M == 0) return CQG_OK;
  float *gw = grads + nw, *gb = grads + nw + nb;
  __nv_bfloat16 *dZ = (__nv_bfloat16 *)dZ0, *next = (__nv_bfloat16 *)dZ1;
  auto launch_dz = [&](const float *dY, const float *z, __nv_bfloat16 *out, int N) {
    k_dz_colsum<<<dim3((M + kColRows - 1) / kColRows, (N + 31) / 32), 256, 0, st>>>(dY, z, nullptr, out, M, N, gb);
  };
  const int nout = dims[nl];
  gb -= nout;
  if ((nout + 31) / 32 > 65535) return CQG_ERR_BAD_ARG;
  launch_dz(dout, nullptr, dZ, nout);
  // a weight gradient waits for the next one, and both go in one launch: their blocks together
  // fill the GPU, and each dZ stays until the launch after that
  Gemm waiting = {};
  bool waits = false;
  for (int i = nl - 1; i >= 0; --i) {
    const int K = dims[i], N = dims[i + 1];
    gw -= (long long)K * N;
    // dW[n][k] = sum_m dZ[m][n] h[m][k]
    Gemm w = gemm_of(dZ, 1, N, H[i], 1, K, gw, K, N, K, M);
    w.accumulate = 1;
    set_pairs(w);
    const bool wbig = big_tiles(N, K);
    tile_by(w, wbig ? GM : 64, wbig ? GN : 64);
    if (!wbig) split_k(w);
    cqg_status s = CQG_OK;
    if (wbig) {
      if (waits) s = launch_small(waiting, nullptr, st);
      waits = false;
      if (s == CQG_OK) s = launch_big(w, st);
    } else if (waits) {
      s = launch_small(waiting, &w, st);
      waits = false;
    } else {
      waiting = w;
      waits = true;
    }
    if (s == CQG_OK && i > 0) {
      // dh[m][k] = sum_n dZ[m][n] W[n][k], through the SiLU of the layer below: the next dZ
      gb -= K;
      const int part = big_tiles(M, K) ? 0 : k_parts(M, K, N, 2 * GK);
      if (part > 0) {
        if (cudaMemsetAsync(dX, 0, (size_t)M * K * sizeof(float), st) != cudaSuccess) return CQG_ERR_CUDA;
        const dim3 grid((K + kPartTile - 1) / kPartTile, (M + kPartTile - 1) / kPartTile, (N + part - 1) / part);
        k_gemm_parts<<<grid, 128, 0, st>>>(dZ, N, 1, (const __nv_bfloat16 *)W[i], 1, K, dX, K, M, K, N, part);
        launch_dz(dX, Z[i - 1], next, K);
      } else {
        Gemm x = gemm_of(dZ, N, 1, W[i], 1, K, nullptr, K, M, K, N);
        x.dact = Z[i - 1];
        x.Y = next;
        x.ldy = K;
        x.db = gb;
        set_pairs(x);
        const bool xbig = big_tiles(M, K);
        tile_by(x, xbig ? GM : 64, xbig ? GN : 64);
        if (xbig) {
          s = launch_big(x, st);
        } else if (waits) {
          s = launch_small(x, &waiting, st);
          waits = false;
        } else {
          s = launch_small(x, nullptr, st);
        }
      }
    }
    if (s != CQG_OK) return s;
    std::swap(dZ, next);
  }
  if (waits) {
    const cqg_status s = launch_small(waiting, nullptr, st);
    if (s != CQG_OK) return s;
  }
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

}  // extern "C"
