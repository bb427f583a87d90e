// Gated delta rule: what surrounds the loop over the chunks (delta_rule.cu), in both directions, and the gated norm of its output.
//
// For a chunk of 64 tokens of one head, with G the running sum of the log decays from the chunk's start and D_ij = exp(G_i - G_j) for j <= i:
//
//     A_ij = beta_i (k_i . k_j) D_ij  (j < i),   T = (I + A)^-1,   u = T (beta v),   w = T (beta e^G k),
//     P_ij = (q_i . k_j) D_ij  (j <= i),   qg = e^G q,   kd = e^(G_last - G) k,   a = e^(G_last)
//
// One CTA of 256 threads makes one chunk: rows are read as the model has them (bf16 or fp32, any row and head strides; queries and keys are
// normalised here when asked to), everything between stays in shared memory, and only what the loop reads is written.  The backward kernel
// takes the loop's gradients (partial sums over slices of d_v, added here in their order) to the gradients of q, k, v, g and beta:
//
//     R_u = T^t du,  R_w = T^t dw,  dA = -(R_u u^t + R_w w^t) below the diagonal,  M = beta_i dA D,  N = dP D:
//     dv = beta R_u,   dq = N k + e^G dqg,   dk = beta e^G R_w + (M + M^t) k + N^t q + e^(G_last - G) dkd,   and row and column sums for G, beta
//
// All products are fp32 FMAs, as the framework operations that they replace were: 4 x 4 results per thread and operands as they lie in memory
// (rows of shared memory padded by four numbers, so that eight lanes' 16-byte reads fall on different banks).  A chunk of 128-wide heads is 2 MFMA
// forward and 4 MFMA backward, 0.12 and 0.23 ms of this GPU's FMA rate per 2048 chunks; two CTAs per SM cover the barriers and the triangular
// solve.  Measured for 4 x 4096 tokens, 8 heads of 128: 0.37 ms forward; 0.99 ms backward, of which 1.1 GB of partial sums are a part.  The
// framework operations that did this moved every 64 MB intermediate through memory some hundred times: a training pass of two such layers,
// recomputed in its backward pass, went from 36.9 to 23.9 ms.
#include "common.cuh"

namespace lvb {
namespace dchunk {

constexpr int kC = 64;
constexpr int kThreads = 256;
constexpr int kLd = kC + 4;  // row stride of a [64, 64] tile

template <typename T>
__device__ __forceinline__ float4 load4(const T* p);
template <>
__device__ __forceinline__ float4 load4<float>(const float* p) {
  return __ldg(reinterpret_cast<const float4*>(p));
}
template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
  const uint2 w = __ldg(reinterpret_cast<const uint2*>(p));
  const float2 a = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(w.x)), b = __bfloat1622float2(reinterpret_cast<const __nv_bfloat162&>(w.y));
  return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) { *reinterpret_cast<uint2*>(p) = make_uint2(pack_bf16x2(v.x, v.y), pack_bf16x2(v.z, v.w)); }

__device__ __forceinline__ float dot4(float4 a, float4 b) { return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w))); }
__device__ __forceinline__ float4 scale4(float4 a, float s) { return make_float4(a.x * s, a.y * s, a.z * s, a.w * s); }
__device__ __forceinline__ float4 fma4(float4 a, float s, float4 c) {
  return make_float4(fmaf(a.x, s, c.x), fmaf(a.y, s, c.y), fmaf(a.z, s, c.z), fmaf(a.w, s, c.w));
}

// Thread (ty, tx) of 16 x 16; a warp covers 4 x 8 of them.
struct Place {
  int ty, tx;
  __device__ Place() {
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    ty = (w >> 1) * 4 + (l >> 3);
    tx = (w & 1) * 8 + (l & 7);
  }
};

// acc[i][j] += sum_k X[ty + 16 i][k] Y[tx + 16 j][k]
template <int K>
__device__ __forceinline__ void gemm_nt(float (&acc)[4][4], const float* X, int ldx, const float* Y, int ldy, Place t) {
#pragma unroll 4
  for (int k = 0; k < K; k += 4) {
    float4 x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[i] = *reinterpret_cast<const float4*>(X + (t.ty + 16 * i) * ldx + k);
      y[i] = *reinterpret_cast<const float4*>(Y + (t.tx + 16 * i) * ldy + k);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        acc[i][j] = fmaf(x[i].x, y[j].x, acc[i][j]);
        acc[i][j] = fmaf(x[i].y, y[j].y, acc[i][j]);
        acc[i][j] = fmaf(x[i].z, y[j].z, acc[i][j]);
        acc[i][j] = fmaf(x[i].w, y[j].w, acc[i][j]);
      }
  }
}

// acc[i][j] += sum_k X[ty + 16 i][k] Y[k][4 tx + j], X zero above the diagonal
__device__ __forceinline__ void gemm_nn_lower(float (&acc)[4][4], const float* X, const float* Y, int ldy, Place t) {
  const int end = min(kC, (t.ty & ~3) + 4 + 48);  // rows ty + 16 i of this warp's 4 x 8 threads end at (ty | 3) + 48
#pragma unroll 2
  for (int k = 0; k < end; k += 4) {
    float4 x[4], y[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      x[i] = *reinterpret_cast<const float4*>(X + (t.ty + 16 * i) * kLd + k);
      y[i] = *reinterpret_cast<const float4*>(Y + (k + i) * ldy + 4 * t.tx);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const float xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
#pragma unroll
      for (int kk = 0; kk < 4; ++kk) {
        acc[i][0] = fmaf(xs[kk], y[kk].x, acc[i][0]);
        acc[i][1] = fmaf(xs[kk], y[kk].y, acc[i][1]);
        acc[i][2] = fmaf(xs[kk], y[kk].z, acc[i][2]);
        acc[i][3] = fmaf(xs[kk], y[kk].w, acc[i][3]);
      }
    }
  }
}

// acc[i][j] += sum_k X[k][4 ty + i] Y[k][4 tx + j]; kLower: X is zero above the diagonal (k < 4 ty)
template <bool kLower>
__device__ __forceinline__ void gemm_tn(float (&acc)[4][4], const float* X, const float* Y, int ldy, Place t) {
  const int begin = kLower ? 4 * (t.ty & ~3) : 0;  // the same for a warp
#pragma unroll 4
  for (int k = begin; k < kC; ++k) {
    const float4 x = *reinterpret_cast<const float4*>(X + k * kLd + 4 * t.ty);
    const float4 y = *reinterpret_cast<const float4*>(Y + k * ldy + 4 * t.tx);
    const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      acc[i][0] = fmaf(xs[i], y.x, acc[i][0]);
      acc[i][1] = fmaf(xs[i], y.y, acc[i][1]);
      acc[i][2] = fmaf(xs[i], y.z, acc[i][2]);
      acc[i][3] = fmaf(xs[i], y.w, acc[i][3]);
    }
  }
}

__device__ __forceinline__ void clear(float (&acc)[4][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
}

struct Rows {  // element (b, l, h, 0) at p + b sb + l sl + h sh
  const void* p;
  long long sb, sl, sh;
};
struct Gate {  // one number per (b, l, h)
  const float* p;
  long long sb, sl, sh;
};

struct Shape {
  int L, H, N, DV, normalize;
  float scale;  // of the queries
};

template <typename T>
__device__ __forceinline__ const T* row_ptr(const Rows& r, int b, int l, int h) {
  return reinterpret_cast<const T*>(r.p) + b * r.sb + l * r.sl + h * r.sh;
}

// One warp: row l of r (zeros past the end) times `scale`, divided by its 2-norm when asked to, as numbers 4 lane .. 4 lane + 3 of every
// 128; inv: the reciprocal of the norm
template <typename T, int DK>
__device__ __forceinline__ float4 unit_row(const Rows& r, const Shape& s, int b, int l, int h, float scale, float* inv) {
  const int lane = threadIdx.x & 31;
  float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
  if (l < s.L && 4 * lane < DK) x = load4<T>(row_ptr<T>(r, b, l, h) + 4 * lane);
  float n = 1.f;
  if (s.normalize) {
    n = 1.f / fmaxf(sqrtf(warp_sum(dot4(x, x))), 1e-12f);
    x = scale4(x, n);
  }
  *inv = n;
  return scale4(x, scale);
}

// s_G[i]: running sum of the log decays (zeros past the end), s_beta[i]; the first 64 threads, then a barrier by the caller
__device__ __forceinline__ void load_gates(const Gate& g, const Gate& beta, const Shape& s, int b, int l0, int h, float* s_G, float* s_beta) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x, la = l0 + 2 * lane;
    const float x0 = la < s.L ? g.p[b * g.sb + la * g.sl + h * g.sh] : 0.f, x1 = la + 1 < s.L ? g.p[b * g.sb + (la + 1) * g.sl + h * g.sh] : 0.f;
    float sum = x0 + x1;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float up = __shfl_up_sync(0xffffffffu, sum, o);
      if (lane >= o) sum += up;
    }
    const float before = __shfl_up_sync(0xffffffffu, sum, 1);
    const float base = lane > 0 ? before : 0.f;
    s_G[2 * lane] = base + x0;
    s_G[2 * lane + 1] = (base + x0) + x1;
  } else if (threadIdx.x < 96) {
    const int i = threadIdx.x - 32, l = l0 + i;
    s_beta[i] = l < s.L ? beta.p[b * beta.sb + l * beta.sl + h * beta.sh] : 0.f;
  }
}

struct Fwd {
  Rows q, k, v;
  Gate g, beta;
  Shape s;
  float *w, *qg, *kd, *P, *u, *a, *T;  // T may be null
};

template <typename T, int DK>
__global__ void __launch_bounds__(kThreads, 2) chunk_fwd_kernel(const Fwd p) {
  constexpr int ldk = DK + 4;
  extern __shared__ __align__(16) float smem[];
  float* sK = smem;
  float* sQ = sK + kC * ldk;
  float* sT = sQ + kC * ldk;   // A, then T
  float* sV = sT + kC * kLd;
  float* sG = sV + kC * kLd;
  float* sBeta = sG + kC;
  const Shape& s = p.s;
  const int n = blockIdx.x % s.N, bh = blockIdx.x / s.N, b = bh / s.H, h = bh % s.H;
  const int l0 = n * kC;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Place t;
  const size_t chunk = blockIdx.x;

  load_gates(p.g, p.beta, s, b, l0, h, sG, sBeta);
  for (int r = warp; r < kC; r += kThreads / 32) {
    float inv;
    const float4 q = unit_row<T, DK>(p.q, s, b, l0 + r, h, s.scale, &inv), k = unit_row<T, DK>(p.k, s, b, l0 + r, h, 1.f, &inv);
    if (4 * lane < DK) {
      store4(sQ + r * ldk + 4 * lane, q);
      store4(sK + r * ldk + 4 * lane, k);
    }
  }
  __syncthreads();
  {
    float acc[4][4];
    clear(acc);
    gemm_nt<DK>(acc, sK, ldk, sK, ldk, t);
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = t.ty + 16 * i, c = t.tx + 16 * j;
        sT[r * kLd + c] = c < r ? acc[i][j] * sBeta[r] * expf(sG[r] - sG[c]) : 0.f;
      }
    clear(acc);
    gemm_nt<DK>(acc, sQ, ldk, sK, ldk, t);
    float* P = p.P + chunk * kC * kC;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = t.ty + 16 * i, c = t.tx + 16 * j;
        P[r * kC + c] = c <= r ? acc[i][j] * expf(sG[r] - sG[c]) : 0.f;
      }
  }
  __syncthreads();
  if (warp < 2) {
    // T: column `col` of the inverse by forward substitution, in registers
    const int col = threadIdx.x;
    float x[kC];
#pragma unroll
    for (int r = 0; r < kC; ++r) {
      float c0 = r == col ? 1.f : 0.f, c1 = 0.f, c2 = 0.f, c3 = 0.f;
#pragma unroll
      for (int k = 0; k < r; k += 4) {
        const float4 a = *reinterpret_cast<const float4*>(sT + r * kLd + k);  // zeros from the diagonal on
        c0 = fmaf(-a.x, x[k], c0);
        if (k + 1 < r) c1 = fmaf(-a.y, x[k + 1], c1);
        if (k + 2 < r) c2 = fmaf(-a.z, x[k + 2], c2);
        if (k + 3 < r) c3 = fmaf(-a.w, x[k + 3], c3);
      }
      x[r] = (c0 + c1) + (c2 + c3);
    }
    asm volatile("bar.sync 1, 64;" ::: "memory");  // both warps have read A
#pragma unroll
    for (int r = 0; r < kC; ++r) sT[r * kLd + col] = x[r];
  } else {
    // meanwhile: qg, kd, and e^G k in place (kd is made from k before)
    const float G_last = sG[kC - 1];
    for (int r = warp - 2; r < kC; r += kThreads / 32 - 2) {
      if (4 * lane < DK) {
        const size_t at = (chunk * kC + r) * DK + 4 * lane;
        const float e = expf(sG[r]);
        const float4 k = *reinterpret_cast<const float4*>(sK + r * ldk + 4 * lane);
        store4(p.qg + at, scale4(*reinterpret_cast<const float4*>(sQ + r * ldk + 4 * lane), e));
        store4(p.kd + at, scale4(k, expf(G_last - sG[r])));
        store4(sK + r * ldk + 4 * lane, scale4(k, e));
      }
    }
    if (threadIdx.x == 64) p.a[chunk] = expf(G_last);
  }
  __syncthreads();
  {
    // T as the solution has it, for the backward pass; T beta in place for the products
    float* Tg = p.T ? p.T + chunk * kC * kC : nullptr;
    for (int i = threadIdx.x; i < kC * kC / 4; i += kThreads) {
      const int r = i / (kC / 4), c = 4 * (i % (kC / 4));
      float4 x = *reinterpret_cast<const float4*>(sT + r * kLd + c);
      if (Tg) store4(Tg + r * kC + c, x);
      x.x *= sBeta[c]; x.y *= sBeta[c + 1]; x.z *= sBeta[c + 2]; x.w *= sBeta[c + 3];
      store4(sT + r * kLd + c, x);
    }
  }
  __syncthreads();
#pragma unroll 1
  for (int c0 = 0; c0 < DK; c0 += kC) {
    float acc[4][4];
    clear(acc);
    gemm_nn_lower(acc, sT, sK + c0, ldk, t);
#pragma unroll
    for (int i = 0; i < 4; ++i) store4(p.w + (chunk * kC + t.ty + 16 * i) * DK + c0 + 4 * t.tx, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
  }
#pragma unroll 1
  for (int c0 = 0; c0 < s.DV; c0 += kC) {
    if (c0 > 0) __syncthreads();  // the previous tile has been read
    for (int i = threadIdx.x; i < kC * kC / 4; i += kThreads) {
      const int r = i / (kC / 4), c = 4 * (i % (kC / 4));
      const float4 x = l0 + r < s.L ? load4<T>(row_ptr<T>(p.v, b, l0 + r, h) + c0 + c) : make_float4(0.f, 0.f, 0.f, 0.f);
      store4(sV + r * kLd + c, x);
    }
    __syncthreads();
    float acc[4][4];
    clear(acc);
    gemm_nn_lower(acc, sT, sV, kLd, t);
#pragma unroll
    for (int i = 0; i < 4; ++i) store4(p.u + (chunk * kC + t.ty + 16 * i) * s.DV + c0 + 4 * t.tx, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
  }
}

struct Bwd {
  Rows q, k, v;
  Gate g, beta;
  Shape s;
  const float *w, *P, *u, *a, *T;                // of the forward pass
  const float *dw, *dqg, *dkd, *dP, *da, *du;    // [slices, chunks, ...] but du
  int slices;
  void *dq, *dk, *dv;                            // [B, L, H, .] contiguous, of the inputs' type
  float *dg, *dbeta;                             // [B, L, H]
};

__device__ __forceinline__ float4 sum_slices(const float* p, size_t stride, int slices) {
  float4 x = __ldg(reinterpret_cast<const float4*>(p));
  for (int i = 1; i < slices; ++i) {
    const float4 y = __ldg(reinterpret_cast<const float4*>(p + i * stride));
    x.x += y.x; x.y += y.y; x.z += y.z; x.w += y.w;
  }
  return x;
}

template <typename T, int DK>
__global__ void __launch_bounds__(kThreads, 2) chunk_bwd_kernel(const Bwd p) {
  constexpr int ldk = DK + 4;
  constexpr int kHalves = DK / kC;
  extern __shared__ __align__(16) float smem[];
  float* sK = smem;                 // k; dq in the end
  float* sT = sK + kC * ldk;        // T; a half of q
  float* sX = sT + kC * kLd;        // du or dw and their products; M + M^t
  float* sY = sX + kC * kLd;        // u or w; N
  float* sDk = sT;                  // dk in the end (room of sT and sX)
  float* sG = sY + kC * kLd;
  float* sBeta = sG + kC;
  float* sRow = sBeta + kC;         // [2][64] sums along rows that go to G
  float* sCol = sRow + 2 * kC;      // [4][64] sums along columns
  float* sB = sCol + 4 * kC;        // [2][64] to beta
  float* sDG = sB + 2 * kC;
  float* sLast = sDG + kC;          // [8] what goes to G_last, a number per warp
  const Shape& s = p.s;
  const int n = blockIdx.x % s.N, bh = blockIdx.x / s.N, b = bh / s.H, h = bh % s.H;
  const int l0 = n * kC;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const Place t;
  const size_t chunk = blockIdx.x, chunks = gridDim.x;
  const size_t tile_k = static_cast<size_t>(kC) * DK, tile_c = kC * kC;

  load_gates(p.g, p.beta, s, b, l0, h, sG, sBeta);
  for (int r = warp; r < kC; r += kThreads / 32) {
    float inv;
    const float4 k = unit_row<T, DK>(p.k, s, b, l0 + r, h, 1.f, &inv);
    if (4 * lane < DK) store4(sK + r * ldk + 4 * lane, k);
  }
  for (int i = threadIdx.x; i < kC * kC / 4; i += kThreads) {
    const int r = i / (kC / 4), c = 4 * (i % (kC / 4));
    store4(sT + r * kLd + c, __ldg(reinterpret_cast<const float4*>(p.T + chunk * tile_c + r * kC + c)));
  }
  float dA[4][4];              // rows ty + 16 i, columns tx + 16 j
  float dk[kHalves][4][4];     // rows 4 ty + i, columns 64 half + 4 tx + j
  float to_beta[4] = {0.f, 0.f, 0.f, 0.f}, to_G[4] = {0.f, 0.f, 0.f, 0.f};  // rows 4 ty + i
  clear(dA);

  // ---- values: R_u, dv
#pragma unroll 1
  for (int c0 = 0; c0 < s.DV; c0 += kC) {
    __syncthreads();
    for (int i = threadIdx.x; i < kC * kC / 4; i += kThreads) {
      const int r = i / (kC / 4), c = 4 * (i % (kC / 4));
      const size_t at = (chunk * kC + r) * s.DV + c0 + c;
      store4(sX + r * kLd + c, __ldg(reinterpret_cast<const float4*>(p.du + at)));
      store4(sY + r * kLd + c, __ldg(reinterpret_cast<const float4*>(p.u + at)));
    }
    __syncthreads();
    float R[4][4];
    clear(R);
    gemm_tn<true>(R, sT, sX, kLd, t);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 4 * t.ty + i, l = l0 + r;
      const float4 x = make_float4(R[i][0], R[i][1], R[i][2], R[i][3]);
      store4(sX + r * kLd + 4 * t.tx, x);
      if (l < s.L) {
        const int c = c0 + 4 * t.tx;
        to_beta[i] += dot4(x, load4<T>(row_ptr<T>(p.v, b, l, h) + c));
        store4(reinterpret_cast<T*>(p.dv) + ((static_cast<size_t>(b) * s.L + l) * s.H + h) * s.DV + c, scale4(x, sBeta[r]));
      }
    }
    __syncthreads();
    gemm_nt<kC>(dA, sX, kLd, sY, kLd, t);
  }
  // ---- keys: R_w
#pragma unroll
  for (int hf = 0; hf < kHalves; ++hf) {
    __syncthreads();
    for (int i = threadIdx.x; i < kC * kC / 4; i += kThreads) {
      const int r = i / (kC / 4), c = 4 * (i % (kC / 4));
      const size_t at = (chunk * kC + r) * DK + hf * kC + c;
      store4(sX + r * kLd + c, sum_slices(p.dw + at, chunks * tile_k, p.slices));
      store4(sY + r * kLd + c, __ldg(reinterpret_cast<const float4*>(p.w + at)));
    }
    __syncthreads();
    clear(dk[hf]);
    gemm_tn<true>(dk[hf], sT, sX, kLd, t);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 4 * t.ty + i;
      const float4 x = make_float4(dk[hf][i][0], dk[hf][i][1], dk[hf][i][2], dk[hf][i][3]);
      store4(sX + r * kLd + 4 * t.tx, x);
      const float e = expf(sG[r]), at_k = e * dot4(x, *reinterpret_cast<const float4*>(sK + r * ldk + hf * kC + 4 * t.tx));
      to_beta[i] += at_k;
      to_G[i] += sBeta[r] * at_k;
#pragma unroll
      for (int j = 0; j < 4; ++j) dk[hf][i][j] *= sBeta[r] * e;
    }
    __syncthreads();
    gemm_nt<kC>(dA, sX, kLd, sY, kLd, t);
  }
  // ---- scores: M, N and their sums
  float row_G[4] = {0.f, 0.f, 0.f, 0.f}, row_B[4] = {0.f, 0.f, 0.f, 0.f}, col_G[4] = {0.f, 0.f, 0.f, 0.f};
  {
    float kk[4][4];
    clear(kk);
    gemm_nt<DK>(kk, sK, ldk, sK, ldk, t);
    __syncthreads();  // sX, sY have been read
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int r = t.ty + 16 * i, c = t.tx + 16 * j;
        float N = 0.f;
        if (c <= r) {
          const float D = expf(sG[r] - sG[c]);
          const size_t at = chunk * tile_c + r * kC + c;
          float dP = __ldg(p.dP + at);
          for (int sl = 1; sl < p.slices; ++sl) dP += __ldg(p.dP + sl * chunks * tile_c + at);
          N = dP * D;
          const float x = dP * __ldg(p.P + at);
          row_G[i] += x;
          col_G[j] += x;
          if (c < r) {
            const float m = -dA[i][j] * D, y = m * kk[i][j];
            row_B[i] += y;
            row_G[i] += sBeta[r] * y;
            col_G[j] += sBeta[r] * y;
            sX[r * kLd + c] = m * sBeta[r];
            sX[c * kLd + r] = m * sBeta[r];
          } else {
            sX[r * kLd + c] = 0.f;
          }
        }
        sY[r * kLd + c] = N;
      }
  }
  {
    // sums along rows: 8 lanes, 2 warps; along columns: 4 lanes, 4 warps
#pragma unroll
    for (int i = 0; i < 4; ++i) {
#pragma unroll
      for (int o = 1; o < 8; o <<= 1) {
        row_G[i] += __shfl_xor_sync(0xffffffffu, row_G[i], o);
        row_B[i] += __shfl_xor_sync(0xffffffffu, row_B[i], o);
        to_G[i] += __shfl_xor_sync(0xffffffffu, to_G[i], o);
        to_beta[i] += __shfl_xor_sync(0xffffffffu, to_beta[i], o);
      }
#pragma unroll
      for (int o = 8; o < 32; o <<= 1) col_G[i] += __shfl_xor_sync(0xffffffffu, col_G[i], o);
      if ((lane & 7) == 0) {
        sRow[(warp & 1) * kC + t.ty + 16 * i] = row_G[i];
        sB[(warp & 1) * kC + t.ty + 16 * i] = row_B[i];
      }
      if (lane < 8) sCol[(warp >> 1) * kC + t.tx + 16 * i] = col_G[i];
    }
    __syncthreads();
    // the other order of rows
#pragma unroll
    for (int i = 0; i < 4; ++i)
      if ((lane & 7) == 0) {
        sRow[(warp & 1) * kC + 4 * t.ty + i] += to_G[i];
        sB[(warp & 1) * kC + 4 * t.ty + i] += to_beta[i];
      }
  }
  // ---- dk += (M + M^t) k + N^t q
#pragma unroll
  for (int hf = 0; hf < kHalves; ++hf) gemm_tn<false>(dk[hf], sX, sK + hf * kC, ldk, t);
#pragma unroll
  for (int hf = 0; hf < kHalves; ++hf) {
    __syncthreads();
    for (int r = warp; r < kC; r += kThreads / 32) {  // the norm needs the whole row
      float inv;
      const float4 q = unit_row<T, DK>(p.q, s, b, l0 + r, h, s.scale, &inv);
      if (4 * lane >= hf * kC && 4 * lane < (hf + 1) * kC) store4(sT + r * kLd + 4 * lane - hf * kC, q);
    }
    __syncthreads();
    gemm_tn<true>(dk[hf], sY, sT, kLd, t);
  }
  // ---- dq = N k
  float dq[kHalves][4][4];
#pragma unroll
  for (int hf = 0; hf < kHalves; ++hf) {
    clear(dq[hf]);
    gemm_nn_lower(dq[hf], sY, sK + hf * kC, ldk, t);
  }
  __syncthreads();
#pragma unroll
  for (int hf = 0; hf < kHalves; ++hf)
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      store4(sK + (t.ty + 16 * i) * ldk + hf * kC + 4 * t.tx, make_float4(dq[hf][i][0], dq[hf][i][1], dq[hf][i][2], dq[hf][i][3]));
      store4(sDk + (4 * t.ty + i) * ldk + hf * kC + 4 * t.tx, make_float4(dk[hf][i][0], dk[hf][i][1], dk[hf][i][2], dk[hf][i][3]));
    }
  __syncthreads();
  // ---- rows: the terms of qg and kd, the norms, and what goes to G
  const float G_last = sG[kC - 1];
  float last = 0.f;
  for (int r = warp; r < kC; r += kThreads / 32) {
    const int l = l0 + r;
    float inv_q, inv_k;
    float4 q = unit_row<T, DK>(p.q, s, b, l, h, 1.f, &inv_q), k = unit_row<T, DK>(p.k, s, b, l, h, 1.f, &inv_k);
    float4 gq = make_float4(0.f, 0.f, 0.f, 0.f), gk = gq, xq = gq, xk = gq;
    const float eq = expf(sG[r]), ek = expf(G_last - sG[r]);
    if (4 * lane < DK) {
      const size_t at = chunk * tile_k + r * DK + 4 * lane;
      xq = sum_slices(p.dqg + at, chunks * tile_k, p.slices);
      xk = sum_slices(p.dkd + at, chunks * tile_k, p.slices);
      gq = scale4(fma4(xq, eq, *reinterpret_cast<const float4*>(sK + r * ldk + 4 * lane)), s.scale);  // to the row before its scale
      gk = fma4(xk, ek, *reinterpret_cast<const float4*>(sDk + r * ldk + 4 * lane));
    }
    const float at_q = warp_sum(dot4(xq, q)) * eq * s.scale, at_k = warp_sum(dot4(xk, k)) * ek;
    if (lane == 0) sDG[r] = at_q - at_k;
    last += at_k;
    if (s.normalize) {  // x / max(|x|, 1e-12)
      const float pq = warp_sum(dot4(gq, q)), pk = warp_sum(dot4(gk, k));
      gq = scale4(inv_q < 0.999e12f ? fma4(q, -pq, gq) : gq, inv_q);
      gk = scale4(inv_k < 0.999e12f ? fma4(k, -pk, gk) : gk, inv_k);
    }
    if (l < s.L && 4 * lane < DK) {
      const size_t at = ((static_cast<size_t>(b) * s.L + l) * s.H + h) * DK + 4 * lane;
      store4(reinterpret_cast<T*>(p.dq) + at, gq);
      store4(reinterpret_cast<T*>(p.dk) + at, gk);
    }
  }
  if (lane == 0) sLast[warp] = last;
  __syncthreads();
  if (warp == 0) {
    float at_last = 0.f;
    for (int i = 0; i < kThreads / 32; ++i) at_last += sLast[i];
    float da = p.da[chunk];
    for (int i = 1; i < p.slices; ++i) da += p.da[i * chunks + chunk];
    at_last += da * p.a[chunk];
    float x[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 2 * lane + i;
      x[i] = sDG[r] + (sRow[r] + sRow[kC + r]) - ((sCol[r] + sCol[kC + r]) + (sCol[2 * kC + r] + sCol[3 * kC + r])) + (r == kC - 1 ? at_last : 0.f);
    }
    float sum = x[0] + x[1];  // the gradient of a step is the sum over the running sums that it is in
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const float down = __shfl_down_sync(0xffffffffu, sum, o);
      if (lane + o < 32) sum += down;
    }
    const float after = __shfl_down_sync(0xffffffffu, sum, 1);
    x[1] += lane < 31 ? after : 0.f;
    x[0] += x[1];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int r = 2 * lane + i, l = l0 + r;
      if (l < s.L) {
        const size_t at = (static_cast<size_t>(b) * s.L + l) * s.H + h;
        p.dg[at] = x[i];
        p.dbeta[at] = sB[r] + sB[kC + r];
      }
    }
  }
}

// ---- y = o rsqrt(mean(o^2) + eps) weight silu(gate): o [B, H, N, 64, dv] fp32, gate and y [B, L, H, dv]; a warp per row
struct Norm {
  const float* o;
  const void* gate;
  const float* weight;
  void* y;
  int B, L, H, N, DV;
  float eps;
  // backward
  const void* dy;
  float *d_o, *dw_part;  // dw_part [gridDim.x, dv]
  void* dgate;
};

template <typename T>
__global__ void __launch_bounds__(256) out_norm_fwd_kernel(const Norm p) {
  const int lane = threadIdx.x & 31;
  const long long row = (blockIdx.x * 256ll + threadIdx.x) >> 5, rows = static_cast<long long>(p.B) * p.L * p.H;
  if (row >= rows) return;
  const int h = static_cast<int>(row % p.H);
  const long long bl = row / p.H;
  const int l = static_cast<int>(bl % p.L), b = static_cast<int>(bl / p.L);
  const float* o = p.o + ((static_cast<long long>(b) * p.H + h) * p.N * kC + l) * p.DV;
  float ss = 0.f;
  for (int c = 4 * lane; c < p.DV; c += 128) {
    const float4 x = load4<float>(o + c);
    ss += dot4(x, x);
  }
  const float r = rsqrtf(warp_sum(ss) / static_cast<float>(p.DV) + p.eps);
  for (int c = 4 * lane; c < p.DV; c += 128) {
    const float4 x = load4<float>(o + c), z = load4<T>(reinterpret_cast<const T*>(p.gate) + row * p.DV + c), w = load4<float>(p.weight + c);
    store4(reinterpret_cast<T*>(p.y) + row * p.DV + c,
           make_float4(x.x * r * w.x * (z.x / (1.f + expf(-z.x))), x.y * r * w.y * (z.y / (1.f + expf(-z.y))),
                       x.z * r * w.z * (z.z / (1.f + expf(-z.z))), x.w * r * w.w * (z.w / (1.f + expf(-z.w)))));
  }
}

constexpr int kMaxNorm = 4;  // dv <= 512: 4 numbers per lane and 128

template <typename T>
__global__ void __launch_bounds__(256) out_norm_bwd_kernel(const Norm p) {
  __shared__ float s_part[8][128 * kMaxNorm];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const long long rows = static_cast<long long>(p.B) * p.N * kC * p.H;  // with the padding of the last chunk, whose gradients are zeros
  float4 acc[kMaxNorm];
#pragma unroll
  for (int i = 0; i < kMaxNorm; ++i) acc[i] = make_float4(0.f, 0.f, 0.f, 0.f);
  for (long long n = blockIdx.x * 8ll + warp; n < rows; n += gridDim.x * 8ll) {
    const int h = static_cast<int>(n % p.H);
    const long long bl = n / p.H;
    const int l = static_cast<int>(bl % (p.N * kC)), b = static_cast<int>(bl / (p.N * kC));
    const long long at_o = ((static_cast<long long>(b) * p.H + h) * p.N * kC + l) * p.DV;
    const long long at = ((static_cast<long long>(b) * p.L + l) * p.H + h) * p.DV;
    float4 x[kMaxNorm], gy[kMaxNorm];
    float ss = 0.f, gx = 0.f;
    if (l < p.L) {
#pragma unroll
      for (int i = 0; i < kMaxNorm; ++i) {
        const int c = 4 * lane + 128 * i;
        if (c < p.DV) {
          x[i] = load4<float>(p.o + at_o + c);
          ss += dot4(x[i], x[i]);
        }
      }
    }
    const float r = rsqrtf(warp_sum(ss) / static_cast<float>(p.DV) + p.eps);
#pragma unroll
    for (int i = 0; i < kMaxNorm; ++i) {
      const int c = 4 * lane + 128 * i;
      gy[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (c < p.DV && l < p.L) {
        const float4 z4 = load4<T>(reinterpret_cast<const T*>(p.gate) + at + c), d4 = load4<T>(reinterpret_cast<const T*>(p.dy) + at + c), w4 = load4<float>(p.weight + c);
        const float z[4] = {z4.x, z4.y, z4.z, z4.w}, d[4] = {d4.x, d4.y, d4.z, d4.w}, w[4] = {w4.x, w4.y, w4.z, w4.w};
        const float xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w};
        float dz[4], g[4], dw[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float sg = 1.f / (1.f + expf(-z[j])), silu = z[j] * sg, hat = xs[j] * r;
          dz[j] = d[j] * hat * w[j] * (sg * (1.f + z[j] * (1.f - sg)));
          dw[j] = d[j] * silu * hat;
          g[j] = d[j] * silu * w[j];
        }
        store4(reinterpret_cast<T*>(p.dgate) + at + c, make_float4(dz[0], dz[1], dz[2], dz[3]));
        acc[i].x += dw[0]; acc[i].y += dw[1]; acc[i].z += dw[2]; acc[i].w += dw[3];
        gy[i] = make_float4(g[0], g[1], g[2], g[3]);
        gx += dot4(gy[i], x[i]);
      }
    }
    const float m = warp_sum(gx) * r * r * r / static_cast<float>(p.DV);
#pragma unroll
    for (int i = 0; i < kMaxNorm; ++i) {
      const int c = 4 * lane + 128 * i;
      if (c < p.DV) store4(p.d_o + at_o + c, l < p.L ? fma4(x[i], -m, scale4(gy[i], r)) : gy[i]);
    }
  }
#pragma unroll
  for (int i = 0; i < kMaxNorm; ++i) store4(&s_part[warp][128 * i + 4 * lane], acc[i]);
  __syncthreads();
  for (int c = threadIdx.x; c < p.DV; c += 256) {
    float x = 0.f;
    for (int i = 0; i < 8; ++i) x += s_part[i][c];
    p.dw_part[static_cast<size_t>(blockIdx.x) * p.DV + c] = x;
  }
}

template <int DK>
constexpr int fwd_bytes() { return (2 * kC * (DK + 4) + 2 * kC * kLd + 2 * kC) * 4; }
template <int DK>
constexpr int bwd_bytes() { return (kC * (DK + 4) + 3 * kC * kLd + (2 + 2 + 4 + 2 + 1) * kC + 8) * 4; }

template <typename T, int DK>
int launch_fwd(const Fwd& p, int blocks, cudaStream_t st) {
  auto kern = chunk_fwd_kernel<T, DK>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, fwd_bytes<DK>()) != cudaSuccess) return kErrCuda;
  kern<<<blocks, kThreads, fwd_bytes<DK>(), st>>>(p);
  return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
}
template <typename T, int DK>
int launch_bwd(const Bwd& p, int blocks, cudaStream_t st) {
  auto kern = chunk_bwd_kernel<T, DK>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bwd_bytes<DK>()) != cudaSuccess) return kErrCuda;
  kern<<<blocks, kThreads, bwd_bytes<DK>(), st>>>(p);
  return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
}

// Rows are read 4 numbers at a time
bool rows_ok(const void* p, long long sb, long long sl, long long sh, bool bf16) {
  return ((sb | sl | sh) & 3) == 0 && (reinterpret_cast<uintptr_t>(p) & (bf16 ? 7 : 15)) == 0;
}

}  // namespace dchunk
}  // namespace lvb

using namespace lvb;
using namespace lvb::dchunk;

// strides: 15 numbers, (batch, position, head) of q, k, v (in elements; rows contiguous, multiples of 4), g and beta.  q, k [B, L, H, DK] and v
// [B, L, H, DV] are bf16 or fp32 by `bf16`, g (log decay) and beta fp32.  N = ceil(L / 64); w, qg, kd [B, H, N, 64, DK], P and T (may be null)
// [B, H, N, 64, 64], u [B, H, N, 64, DV], a [B, H, N], all fp32.  normalize: q and k are divided by their 2-norms (at least 1e-12).
extern "C" int lvb_delta_chunks_fwd(const void* q, const void* k, const void* v, const float* g, const float* beta, const long long* strides, float* w,
                                    float* qg, float* kd, float* P, float* u, float* a, float* T, int B, int L, int H, int DK, int DV, int bf16,
                                    int normalize, float scale, void* stream) {
  if (B <= 0 || L <= 0 || H <= 0 || DV <= 0 || DV % kC != 0 || (DK != 64 && DK != 128)) return kErrBadArg;
  const long long* x = strides;
  if (!rows_ok(q, x[0], x[1], x[2], bf16) || !rows_ok(k, x[3], x[4], x[5], bf16) || !rows_ok(v, x[6], x[7], x[8], bf16)) return kErrBadArg;
  const int N = (L + kC - 1) / kC;
  Fwd p{{q, x[0], x[1], x[2]}, {k, x[3], x[4], x[5]}, {v, x[6], x[7], x[8]}, {g, x[9], x[10], x[11]}, {beta, x[12], x[13], x[14]},
        {L, H, N, DV, normalize, scale}, w, qg, kd, P, u, a, T};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int blocks = B * H * N;
  if (bf16) return DK == 128 ? launch_fwd<__nv_bfloat16, 128>(p, blocks, st) : launch_fwd<__nv_bfloat16, 64>(p, blocks, st);
  return DK == 128 ? launch_fwd<float, 128>(p, blocks, st) : launch_fwd<float, 64>(p, blocks, st);
}

// The gradients of lvb_delta_chunks_fwd's inputs.  dw, dqg, dkd, dP, da: [slices, ...] partial sums, du complete; dq, dk [B, L, H, DK] and dv
// [B, L, H, DV] of the inputs' type, dg and dbeta [B, L, H] fp32.
extern "C" int lvb_delta_chunks_bwd(const void* q, const void* k, const void* v, const float* g, const float* beta, const long long* strides,
                                    const float* w, const float* P, const float* u, const float* a, const float* T, const float* dw, const float* dqg,
                                    const float* dkd, const float* dP, const float* da, const float* du, int slices, void* dq, void* dk, void* dv,
                                    float* dg, float* dbeta, int B, int L, int H, int DK, int DV, int bf16, int normalize, float scale, void* stream) {
  if (B <= 0 || L <= 0 || H <= 0 || DV <= 0 || DV % kC != 0 || (DK != 64 && DK != 128) || slices <= 0) return kErrBadArg;
  const long long* x = strides;
  if (!rows_ok(q, x[0], x[1], x[2], bf16) || !rows_ok(k, x[3], x[4], x[5], bf16) || !rows_ok(v, x[6], x[7], x[8], bf16)) return kErrBadArg;
  const int N = (L + kC - 1) / kC;
  Bwd p{{q, x[0], x[1], x[2]}, {k, x[3], x[4], x[5]}, {v, x[6], x[7], x[8]}, {g, x[9], x[10], x[11]}, {beta, x[12], x[13], x[14]},
        {L, H, N, DV, normalize, scale}, w, P, u, a, T, dw, dqg, dkd, dP, da, du, slices, dq, dk, dv, dg, dbeta};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  const int blocks = B * H * N;
  if (bf16) return DK == 128 ? launch_bwd<__nv_bfloat16, 128>(p, blocks, st) : launch_bwd<__nv_bfloat16, 64>(p, blocks, st);
  return DK == 128 ? launch_bwd<float, 128>(p, blocks, st) : launch_bwd<float, 64>(p, blocks, st);
}

// y [B, L, H, DV] = o rsqrt(mean(o^2) + eps) weight silu(gate); o [B, H, ceil(L / 64), 64, DV] fp32, gate and y bf16 or fp32, weight fp32 [DV]
extern "C" int lvb_delta_out_norm_fwd(const float* o, const void* gate, const float* weight, void* y, int B, int L, int H, int DV, float eps, int bf16,
                                      void* stream) {
  if (B <= 0 || L <= 0 || H <= 0 || DV <= 0 || (DV & 3) != 0) return kErrBadArg;
  Norm p{o, gate, weight, y, B, L, H, (L + kC - 1) / kC, DV, eps, nullptr, nullptr, nullptr, nullptr};
  const long long rows = static_cast<long long>(B) * L * H;
  const unsigned grid = static_cast<unsigned>((rows + 7) / 8);
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (bf16) out_norm_fwd_kernel<__nv_bfloat16><<<grid, 256, 0, st>>>(p);
  else out_norm_fwd_kernel<float><<<grid, 256, 0, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
}

// d_o (zeros in the padding of the last chunk), dgate, and dw_part [blocks, DV] whose sum over the blocks is the weight's gradient; DV <= 512
extern "C" int lvb_delta_out_norm_bwd(const float* o, const void* gate, const float* weight, const void* dy, float* d_o, void* dgate, float* dw_part,
                                      int blocks, int B, int L, int H, int DV, float eps, int bf16, void* stream) {
  if (B <= 0 || L <= 0 || H <= 0 || DV <= 0 || (DV & 3) != 0 || DV > 128 * kMaxNorm || blocks <= 0) return kErrBadArg;
  Norm p{o, gate, weight, nullptr, B, L, H, (L + kC - 1) / kC, DV, eps, dy, d_o, dw_part, dgate};
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (bf16) out_norm_bwd_kernel<__nv_bfloat16><<<blocks, 256, 0, st>>>(p);
  else out_norm_bwd_kernel<float><<<blocks, 256, 0, st>>>(p);
  return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
}
