// Kernels of the learned initial-density model: a small MLP trained and evaluated on the
// GPU with BF16 operands and FP32 accumulation.
//
//   k_gemm_bf16 : C[m][n] (+)= sum_k A(m,k) B(n,k), A and B BF16 with arbitrary strides
//                 (transposes are strides), on the tensor cores: mma.sync m16n8k16 BF16 x
//                 BF16 -> FP32 over block tiles that come through a ring of asynchronous
//                 copies; optional fused epilogue Z = C + bias (FP32) and Y = SiLU(Z) (BF16)
//   k_gemm_parts: the same product with K split over blocks, their parts added with atomics
//   k_silu_bwd  : dZ = dY * SiLU'(Z)  (BF16 out, the next GEMM's operand)
//   k_colsum    : db[n] = sum_m dZ[m][n]
//   k_mse       : masked squared error, its gradient, and the loss sum
//   k_adam      : Adam step on FP32 master weights, BF16 copy for the next pass
//   k_to_bf16   : FP32 -> BF16
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>
#include <atomic>

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
  __device__ __forceinline__ TileCopy(const __nv_bfloat16 *X, long long sr, long long sk, int r0, int nrows, int mode) {
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
      src[c] = most[c] ? X + r * sr + k[c] * sk : X;
    }
  }
  // tile kt, of k from kt * GK; `left` = K - that
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

struct Gemm {
  const __nv_bfloat16 *A, *B;
  long long sam, sak, sbn, sbk, ldc, ldy;
  float *C;
  const float *bias;
  __nv_bfloat16 *Y;
  int M, N, K, nbn;
  unsigned char amode, bmode, act, accumulate, pairs;   // pairs: C and Y take 2-wide accesses
};

// Block tile BM x BN (BM, BN multiples of 32), warps of 32 x WN output each (WN = 64 or 32):
// (BM / 32) x (BN / WN) warps; per 16-wide k step a warp issues 2 x (WN / 8) tensor-core
// tiles.  128 x 128 with 8 warps of 32 x 64 for large problems, 64 x 64 with 4 warps of
// 32 x 32 when the large tiles would leave most of the 148 SMs idle.  A training step's
// products (2048 x 256 x 256) are chains of load latencies, not arithmetic: tiles of 32 k come
// through a ring of STAGES asynchronous copies.  Measured, 2048 rows, width 256: a layer forward
// 9.1 us, 17 us with one synchronous tile at a time.
template <int BM, int BN, int WN, int STAGES>
__global__ void __launch_bounds__((BM / 32) * (BN / WN) * 32, BM == 64 ? 3 : 2)
    k_gemm_bf16(const __grid_constant__ Gemm p) {
  constexpr int NWM = BM / 32, NJ = WN / 8, NT = NWM * (BN / WN) * 32;
  constexpr int ASZ = BM * GP, BSZ = BN * GP;   // [k][row] tiles, GK x (rows + 8), fit as well
  static_assert(GK * (BM + 8) <= ASZ && GK * (BN + 8) <= BSZ, "tile buffers");
  extern __shared__ __align__(16) __nv_bfloat16 tiles[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int wm = (warp % NWM) * 32, wn = (warp / NWM) * WN;
  const int M = p.M, N = p.N, K = p.K;
  const int n0 = (int)blockIdx.x % p.nbn * BN, m0 = (int)blockIdx.x / p.nbn * BM;
  const int g = lane >> 2, t = lane & 3;
  float acc[2][NJ][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.f;
  const int nkt = (K + GK - 1) / GK;
  const __nv_bfloat16 *A = p.A, *B = p.B;
  const long long sam = p.sam, sak = p.sak, sbn = p.sbn, sbk = p.sbk;
  const int amode = p.amode, bmode = p.bmode;
  const TileCopy<BM, NT> ca(A, sam, sak, m0, M, amode);
  const TileCopy<BN, NT> cb(B, sbn, sbk, n0, N, bmode);
  auto issue = [&](int kt) {
    if (kt < nkt) {
      __nv_bfloat16 *As = tiles + (kt % STAGES) * (ASZ + BSZ), *Bs = As + ASZ;
      const int k0 = kt * GK;
      if (amode != TILE_ANY)
        ca.start((unsigned)__cvta_generic_to_shared(As), kt, K - k0);
      else
        stage_any<BM, NT>(A, sam, sak, m0, M, k0, K, As);
      if (bmode != TILE_ANY)
        cb.start((unsigned)__cvta_generic_to_shared(Bs), kt, K - k0);
      else
        stage_any<BN, NT>(B, sbn, sbk, n0, N, k0, K, Bs);
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
  // the epilogue from shared memory, four rows of two neighbouring columns a thread at
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
  const float *bias = p.bias;
  const bool act = p.act, accumulate = p.accumulate;
  const float b0 = bias ? bias[n] : 0.f, b1 = bias && two ? bias[n + 1] : 0.f;
#pragma unroll 1
  for (int r0 = threadIdx.x / CG; r0 < min(BM, M - m0); r0 += RSTEP * U) {
    float2 d[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int r = r0 + u * RSTEP;
      d[u] = make_float2(0.f, 0.f);
      if (accumulate && m0 + r < M) {
        const float *q = C + (m0 + r) * ldc + n;
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
      const float z0 = v.x + b0 + d[u].x, z1 = v.y + b1 + d[u].y;
      float *c = C + (m0 + r) * ldc + n;
      if (both) {
        *reinterpret_cast<float2 *>(c) = make_float2(z0, z1);
      } else {
        c[0] = z0;
        if (two) c[1] = z1;
      }
      if (!Y) continue;
      const __nv_bfloat16 y0 = __float2bfloat16(act ? silu(z0) : z0), y1 = __float2bfloat16(act ? silu(z1) : z1);
      __nv_bfloat16 *y = Y + (m0 + r) * ldy + n;
      if (both) {
        *reinterpret_cast<__nv_bfloat162 *>(y) = __halves2bfloat162(y0, y1);
      } else {
        y[0] = y0;
        if (two) y[1] = y1;
      }
    }
  }
}

// Rows [r0, r0 + 64) x k [k0, k0 + 32) of X(r, k) = X[r * sr + k * sk] into S[row][k] (zero outside
// nrows x K).  Rows or k contiguous and 16-byte aligned: 8-element loads; anything else element
// by element.
constexpr int kPartTile = 64;
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
// warps, one tile of k in shared memory at a time, C zeroed by the caller: the backward pass's
// products that are split.  The parts of one element add up in the order in which their
// blocks finish.  For the gradient of a layer's input that order is seen: the next dZ is the sum
// in BF16, a last bit that differs turns one BF16 rounding in some 2^16, 2^-8 of an element, and
// the layers below multiply it.  Which order is usual depends on how long the blocks run, on
// the launches around them and on where the buffers lie.  Measured, 2048 rows, width 256, four
// of these products in a pass, median of the largest relative change of a weight gradient
// between two processes on the same inputs: 1e-6 to 1.3e-5 for this kernel in the layer-by-layer
// pass; 1.4e-5 to 2e-5 with the whole pass in one call, the weight gradients of two layers in a
// launch and SiLU' with the column sums in another; 2.5e-5 and more with the sum in one fixed
// order or in blocks of k_gemm_bf16.  So the backward pass keeps this kernel (17 us a product
// where k_gemm_bf16 takes 9) and its launches, and training runs keep their gradients.
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

// db[n] += sum over rows [blockIdx.y * 256, +256) of dZ[m][n]: 32 columns x 8 row groups
// per block (a warp reads 32 consecutive columns of one row), partial sums reduced in shared
// memory, one atomic per column and block (db zeroed by the caller).
__global__ void __launch_bounds__(256) k_colsum(const __nv_bfloat16 *__restrict__ dZ, int M, int N,
                                                float *__restrict__ db) {
  __shared__ float part[8][33];
  const int c = threadIdx.x & 31, rg = threadIdx.x >> 5;
  const int n = blockIdx.x * 32 + c;
  const int m0 = blockIdx.y * 256, m1 = min(M, m0 + 256);
  float s = 0.f;
  if (n < N)
    for (int m = m0 + rg; m < m1; m += 8) s += __bfloat162float(dZ[(long long)m * N + n]);
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

__global__ void k_adam(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m1,
                       float *__restrict__ m2, long long n, float lr, float b1, float b2, float eps, float bc1,
                       float bc2, float wd, __nv_bfloat16 *__restrict__ wbf) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i] + wd * w[i];
  const float a = b1 * m1[i] + (1.f - b1) * gi;
  const float b = b2 * m2[i] + (1.f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = b;
  const float upd = lr * (a / bc1) / (sqrtf(b / bc2) + eps);
  w[i] -= upd;
  if (wbf) wbf[i] = __float2bfloat16(w[i]);
}

// The same step with the learning rate and the two bias corrections read from device memory
// (hyper = {lr, 1 - b1^step, 1 - b2^step}), so that a captured training step can be replayed
// with a schedule that changes from step to step.
__global__ void k_adam_dev(float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m1,
                           float *__restrict__ m2, long long n, const float *__restrict__ hyper, float b1, float b2,
                           float eps, float wd, __nv_bfloat16 *__restrict__ wbf) {
  const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float lr = hyper[0], bc1 = hyper[1], bc2 = hyper[2];
  const float gi = g[i] + wd * w[i];
  const float a = b1 * m1[i] + (1.f - b1) * gi;
  const float b = b2 * m2[i] + (1.f - b2) * gi * gi;
  m1[i] = a;
  m2[i] = b;
  w[i] -= lr * (a / bc1) / (sqrtf(b / bc2) + eps);
  if (wbf) wbf[i] = __float2bfloat16(w[i]);
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
  g.pairs = g.ldc % 2 == 0 && aligned(g.C, 8) && (!g.Y || (g.ldy % 2 == 0 && aligned(g.Y, 4)));
}

// Few 64 x 64 output tiles and a long reduction (weight gradients: K = batch rows): K split so
// that about two waves of blocks run, in parts of 64 or more; the part, or 0 for one.
int k_parts(int M, int N, int K) {
  const long long tiles = (long long)((N + 63) / 64) * ((M + 63) / 64);
  if (tiles >= 148 || K < 4 * GK) return 0;
  const int splits = (int)std::min<long long>(std::min<long long>((296 + tiles - 1) / tiles, K / (2 * GK)), 64);
  return splits > 1 ? ((K + splits - 1) / splits + GK - 1) / GK * GK : 0;
}

template <int BM, int BN, int WN, int STAGES>
cqg_status launch_gemm(Gemm &g, cudaStream_t st) {
  static std::atomic<bool> allowed[64];
  constexpr int smem = STAGES * (BM + BN) * GP * 2;
  if (allow_tiles(&k_gemm_bf16<BM, BN, WN, STAGES>, smem, allowed) != cudaSuccess) return CQG_ERR_CUDA;
  g.nbn = (g.N + BN - 1) / BN;
  k_gemm_bf16<BM, BN, WN, STAGES><<<g.nbn * ((g.M + BM - 1) / BM), (BM / 32) * (BN / WN) * 32, smem, st>>>(g);
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
  const bool big = big_tiles(M, N);
  if ((M + (big ? GM : 64) - 1) / (big ? GM : 64) > 65535) return CQG_ERR_BAD_ARG;
  const int part = big || bias || Y ? 0 : k_parts(M, N, K);
  if (part > 0) {
    if (!accumulate && cudaMemset2DAsync(C, ldc * sizeof(float), 0, N * sizeof(float), M, st) != cudaSuccess)
      return CQG_ERR_CUDA;
    const dim3 grid((N + kPartTile - 1) / kPartTile, (M + kPartTile - 1) / kPartTile, (K + part - 1) / part);
    k_gemm_parts<<<grid, 128, 0, st>>>((const __nv_bfloat16 *)A, sam, sak, (const __nv_bfloat16 *)B, sbn, sbk, C, ldc, M,
                                       N, K, part);
  } else {
    Gemm g = gemm_of(A, sam, sak, B, sbn, sbk, C, ldc, M, N, K);
    g.bias = bias;
    g.Y = (__nv_bfloat16 *)Y;
    g.ldy = ldy;
    g.act = act != 0;
    g.accumulate = accumulate != 0;
    set_pairs(g);
    const cqg_status s = big ? launch_gemm<GM, GN, 64, 4>(g, st) : launch_gemm<64, 64, 32, 6>(g, st);
    if (s != CQG_OK) return s;
  }
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
  if ((M + 255) / 256 > 65535) return CQG_ERR_BAD_ARG;
  dim3 grid((N + 31) / 32, (M + 255) / 256);
  k_colsum<<<grid, 256, 0, (cudaStream_t)stream>>>((const __nv_bfloat16 *)dZ, M, N, db);
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_mse(const float *pred, const float *target, const float *mask, long long n, float inv_count,
                       float *dpred, float *loss, void *stream) {
  if (n <= 0) return CQG_OK;
  k_mse<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(pred, target, mask, n, inv_count, dpred, loss);
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_adam(float *w, const float *g, float *m1, float *m2, long long n, float lr, float b1, float b2,
                        float eps, int step, float weight_decay, void *wbf, void *stream) {
  if (n <= 0 || step < 1) return CQG_ERR_BAD_ARG;
  const float bc1 = 1.f - powf(b1, (float)step), bc2 = 1.f - powf(b2, (float)step);
  k_adam<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(w, g, m1, m2, n, lr, b1, b2, eps, bc1, bc2, weight_decay,
                                                         (__nv_bfloat16 *)wbf);
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
}

cqg_status cqg_mlp_adam_dev(float *w, const float *g, float *m1, float *m2, long long n, const float *hyper,
                            float b1, float b2, float eps, float weight_decay, void *wbf, void *stream) {
  if (n <= 0 || !hyper) return CQG_ERR_BAD_ARG;
  k_adam_dev<<<nblk(n, 256), 256, 0, (cudaStream_t)stream>>>(w, g, m1, m2, n, hyper, b1, b2, eps, weight_decay,
                                                             (__nv_bfloat16 *)wbf);
  return cudaGetLastError() == cudaSuccess ? CQG_OK : CQG_ERR_CUDA;
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

}  // extern "C"
