// RMSNorm / LayerNorm forward and backward (bf16 activations, fp32 math).
//
// Covers hnn.RmsNorm / hnn.LayerNorm and Gemma's (1 + w) variant
// (src/levanter/layers/normalization.py:38-48, src/levanter/models/gemma.py:279-291), per-head
// qk-norm (rows = tokens*heads, dim = head_size) and the residual-add that precedes every
// pre-norm block: h = x + residual is written once and normalised in the same pass.
//
// Launch shape: blockDim = (TX, TY): TX threads cooperate on one row, TY rows per block.
// Every thread moves 16-byte vectors (8 bf16).  dim must be a multiple of 8.
#include "common.cuh"

namespace lvb {
namespace norm {

constexpr int kMaxThreads = 512;
constexpr int kFewRows = 1024;  // up to here a block per row beats a warp per row: fewer warps than the SMs' schedulers hold twice
constexpr int kMaxVecPerThread = 4;  // backward keeps dw partials in registers: dim <= 512 * 4 * 8

struct Vec8 {
  float v[8];
};

__device__ __forceinline__ Vec8 load8(const __nv_bfloat16* p) {
  uint4 w = *reinterpret_cast<const uint4*>(p);
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
  Vec8 o;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 f = __bfloat1622float2(h[j]);
    o.v[2 * j] = f.x;
    o.v[2 * j + 1] = f.y;
  }
  return o;
}
__device__ __forceinline__ Vec8 unpack8(const uint4& w) {
  const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&w);
  Vec8 o;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    float2 f = __bfloat1622float2(h[j]);
    o.v[2 * j] = f.x;
    o.v[2 * j + 1] = f.y;
  }
  return o;
}
__device__ __forceinline__ void store8(__nv_bfloat16* p, const Vec8& a) {
  uint4 o;
  o.x = pack_bf16x2(a.v[0], a.v[1]);
  o.y = pack_bf16x2(a.v[2], a.v[3]);
  o.z = pack_bf16x2(a.v[4], a.v[5]);
  o.w = pack_bf16x2(a.v[6], a.v[7]);
  *reinterpret_cast<uint4*>(p) = o;
}
__device__ __forceinline__ Vec8 loadw8(const void* w, int wf32, int col, float offset) {
  Vec8 o;
  if (w == nullptr) {
#pragma unroll
    for (int j = 0; j < 8; ++j) o.v[j] = 1.f;
    return o;
  }
  if (wf32) {
    // two 16-byte loads (col is a multiple of 8 and the array 16-byte aligned): eight scalar loads per vector made the
    // weight reads, not the activations, the busiest traffic of the load/store unit
    const float4* p = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(w) + col);
    const float4 lo = __ldg(p), hi = __ldg(p + 1);
    o.v[0] = lo.x + offset; o.v[1] = lo.y + offset; o.v[2] = lo.z + offset; o.v[3] = lo.w + offset;
    o.v[4] = hi.x + offset; o.v[5] = hi.y + offset; o.v[6] = hi.z + offset; o.v[7] = hi.w + offset;
  } else {
    o = load8(reinterpret_cast<const __nv_bfloat16*>(w) + col);
#pragma unroll
    for (int j = 0; j < 8; ++j) o.v[j] += offset;
  }
  return o;
}

// Sum over the TX threads of a row.  TX is a power of two up to 32 (rows never straddle warps then) or a multiple of 32, where shared memory joins
// the warps behind one barrier: a caller that comes here again takes the other half of the scratch (2 * reduce_floats).
__host__ __device__ inline int reduce_floats(int TX, int TY) { return TX > 32 ? TY * (TX >> 5) * 2 : 0; }

template <int N>
__device__ __forceinline__ void row_reduce(float (&val)[N], float* scratch, int TX) {
  const int tx = threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o < TX) {
#pragma unroll
      for (int i = 0; i < N; ++i) val[i] += __shfl_xor_sync(0xffffffffu, val[i], o);
    }
  if (TX > 32) {
    const int nw = TX >> 5;
    float* s = scratch + threadIdx.y * (nw * N);
    if ((tx & 31) == 0) {
#pragma unroll
      for (int i = 0; i < N; ++i) s[(tx >> 5) * N + i] = val[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) {  // at most 16 warps
      float v = (tx & 15) < nw ? s[(tx & 15) * N + i] : 0.f;
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      val[i] = v;
    }
  }
}

template <bool LN>
__global__ void norm_fwd_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual,
                                const void* __restrict__ w, const void* __restrict__ b, int wf32,
                                __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out,
                                float* __restrict__ rstd_out, float* __restrict__ mean_out, int rows, int dim,
                                float eps, float w_offset) {
  extern __shared__ float scratch[];
  const int TX = blockDim.x;
  const int row0 = blockIdx.x * blockDim.y + threadIdx.y;
  const int nvec = dim >> 3;
  // rows beyond the end still take part in the block-wide barriers of row_reduce
  const bool active = row0 < rows;
  const size_t base = static_cast<size_t>(active ? row0 : 0) * dim;
  float acc[2] = {0.f, 0.f};
  if (active) {
    for (int i = threadIdx.x; i < nvec; i += TX) {
      Vec8 a = load8(x + base + i * 8);
      if (residual != nullptr) {
        Vec8 r = load8(residual + base + i * 8);
#pragma unroll
        for (int j = 0; j < 8; ++j) a.v[j] += r.v[j];
        if (h_out != nullptr) {
          store8(h_out + base + i * 8, a);
          a = load8(h_out + base + i * 8);  // normalise exactly what later layers will read
        }
      }
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        acc[0] += a.v[j];
        acc[1] += a.v[j] * a.v[j];
      }
    }
  }
  row_reduce<2>(acc, scratch, TX);
  const float mean = LN ? acc[0] / dim : 0.f;
  const float var = LN ? fmaxf(acc[1] / dim - mean * mean, 0.f) : acc[1] / dim;
  const float rstd = rsqrtf(var + eps);
  if (!active) return;
  if (threadIdx.x == 0) {
    if (rstd_out != nullptr) rstd_out[row0] = rstd;
    if (LN && mean_out != nullptr) mean_out[row0] = mean;
  }
  const __nv_bfloat16* src = (residual != nullptr && h_out != nullptr) ? h_out : x;
  for (int i = threadIdx.x; i < nvec; i += TX) {
    Vec8 a = load8(src + base + i * 8);
    if (residual != nullptr && h_out == nullptr) {
      Vec8 r = load8(residual + base + i * 8);
#pragma unroll
      for (int j = 0; j < 8; ++j) a.v[j] += r.v[j];
    }
    Vec8 ww = loadw8(w, wf32, i * 8, w_offset);
    Vec8 o;
#pragma unroll
    for (int j = 0; j < 8; ++j) o.v[j] = (a.v[j] - mean) * rstd * ww.v[j];
    if (b != nullptr) {
      Vec8 bb = loadw8(b, wf32, i * 8, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) o.v[j] += bb.v[j];
    }
    store8(y + base + i * 8, o);
  }
}

// Forward with one 16-byte vector per thread (dim <= 4096): the row, the residual and the weights are all on their way before anything waits,
// and a row over up to 16 warps costs one barrier.  For few rows, where a warp per row leaves the chip idle and its chain of loads, sums and
// stores is the whole time (8 to 256 rows of 4096: 9.4 to 11 us there, 2.4 to 2.9 here), and for every dim that the warp form below does not have
// (8192 x 768: 8.9 us, 15.3 in passes over memory).
template <bool LN>
__global__ void __launch_bounds__(kMaxThreads)
norm_fwd_row_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual, const void* __restrict__ w,
                    const void* __restrict__ b, int wf32, __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out,
                    float* __restrict__ rstd_out, float* __restrict__ mean_out, int rows, int dim, float eps, float w_offset) {
  extern __shared__ float scratch[];
  chain_wait();
  const int col = threadIdx.x * 8;
  const int row = blockIdx.x * blockDim.y + threadIdx.y;
  const bool active = row < rows && col < dim;  // the others take part in the sums
  const size_t at = static_cast<size_t>(row) * dim + col;
  Vec8 a{}, ww{}, bb{};
  if (active) {
    const uint4 v = *reinterpret_cast<const uint4*>(x + at);
    uint4 r{};
    if (residual != nullptr) r = *reinterpret_cast<const uint4*>(residual + at);
    ww = loadw8(w, wf32, col, w_offset);
    if (b != nullptr) bb = loadw8(b, wf32, col, 0.f);
    a = unpack8(v);
    if (residual != nullptr) {
      const Vec8 rr = unpack8(r);
      uint4 h;
      h.x = pack_bf16x2(a.v[0] + rr.v[0], a.v[1] + rr.v[1]);
      h.y = pack_bf16x2(a.v[2] + rr.v[2], a.v[3] + rr.v[3]);
      h.z = pack_bf16x2(a.v[4] + rr.v[4], a.v[5] + rr.v[5]);
      h.w = pack_bf16x2(a.v[6] + rr.v[6], a.v[7] + rr.v[7]);
      if (h_out != nullptr) {
        *reinterpret_cast<uint4*>(h_out + at) = h;
        a = unpack8(h);  // normalise exactly what later layers will read
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j) a.v[j] += rr.v[j];
      }
    }
  }
  float acc[2] = {0.f, 0.f};
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    acc[0] += a.v[j];
    acc[1] += a.v[j] * a.v[j];
  }
  row_reduce<2>(acc, scratch, blockDim.x);
  if (!active) return;
  const float mean = LN ? acc[0] / dim : 0.f;
  const float var = LN ? fmaxf(acc[1] / dim - mean * mean, 0.f) : acc[1] / dim;
  const float rstd = rsqrtf(var + eps);
  if (threadIdx.x == 0) {
    if (rstd_out != nullptr) rstd_out[row] = rstd;
    if (LN && mean_out != nullptr) mean_out[row] = mean;
  }
  Vec8 o;
#pragma unroll
  for (int j = 0; j < 8; ++j) o.v[j] = (a.v[j] - mean) * rstd * ww.v[j] + bb.v[j];
  store8(y + at, o);
}

// Forward with one warp per row and the row held in registers (packed bf16: VPL 16-byte vectors per lane): every load of the
// row is issued before anything waits, the row is read from memory once, and the reduction is five shuffles with no
// block-wide barrier.  For dim = 256 * VPL, VPL in {1, 2, 4, 8, 16} (256 ... 4096).
template <bool LN, int VPL, bool RES>
__global__ void __launch_bounds__(128, 3)
norm_fwd_warp_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ residual, const void* __restrict__ w,
                     const void* __restrict__ b, int wf32, __nv_bfloat16* __restrict__ y, __nv_bfloat16* __restrict__ h_out,
                     float* __restrict__ rstd_out, float* __restrict__ mean_out, int rows, float eps, float w_offset) {
  constexpr int dim = 256 * VPL;
  const int lane = threadIdx.x & 31;
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (row >= rows) return;
  const size_t base = static_cast<size_t>(row) * dim;
  uint4 v[VPL];
#pragma unroll
  for (int s = 0; s < VPL; ++s) v[s] = *reinterpret_cast<const uint4*>(x + base + (lane + 32 * s) * 8);
  if constexpr (RES) {
    uint4 r[VPL];
#pragma unroll
    for (int s = 0; s < VPL; ++s) r[s] = *reinterpret_cast<const uint4*>(residual + base + (lane + 32 * s) * 8);
#pragma unroll
    for (int s = 0; s < VPL; ++s) {
      const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&v[s]);
      const __nv_bfloat162* c = reinterpret_cast<const __nv_bfloat162*>(&r[s]);
      uint4 o;
      uint32_t* ow = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float2 fa = __bfloat1622float2(a[j]), fc = __bfloat1622float2(c[j]);
        ow[j] = pack_bf16x2(fa.x + fc.x, fa.y + fc.y);  // normalise exactly what later layers will read
      }
      v[s] = o;
      if (h_out != nullptr) *reinterpret_cast<uint4*>(h_out + base + (lane + 32 * s) * 8) = o;
    }
  }
  float s1 = 0.f, s2 = 0.f;
#pragma unroll
  for (int s = 0; s < VPL; ++s) {
    const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&v[s]);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(a[j]);
      s1 += f.x + f.y;
      s2 += f.x * f.x + f.y * f.y;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  const float mean = LN ? s1 / dim : 0.f;
  const float var = LN ? fmaxf(s2 / dim - mean * mean, 0.f) : s2 / dim;
  const float rstd = rsqrtf(var + eps);
  if (lane == 0) {
    if (rstd_out != nullptr) rstd_out[row] = rstd;
    if (LN && mean_out != nullptr) mean_out[row] = mean;
  }
#pragma unroll
  for (int s = 0; s < VPL; ++s) {
    const int col = (lane + 32 * s) * 8;
    const __nv_bfloat162* a = reinterpret_cast<const __nv_bfloat162*>(&v[s]);
    const Vec8 ww = loadw8(w, wf32, col, w_offset);
    Vec8 o;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(a[j]);
      o.v[2 * j] = (f.x - mean) * rstd * ww.v[2 * j];
      o.v[2 * j + 1] = (f.y - mean) * rstd * ww.v[2 * j + 1];
    }
    if (b != nullptr) {
      const Vec8 bb = loadw8(b, wf32, col, 0.f);
#pragma unroll
      for (int j = 0; j < 8; ++j) o.v[j] += bb.v[j];
    }
    store8(y + base + col, o);
  }
}

// Backward.  Each block walks rows blockIdx.x * TY + ty, += gridDim.x * TY, with the next rows on their way into a ring of shared memory (every
// thread copies and reads its own vectors, so the ring needs no barrier), and keeps its share of dw (and db) in registers; a block's shares are
// added in shared memory and go to part[block][dim], which norm_bwd_reduce_kernel sums in a fixed order.  What bounds it is the instructions
// per element (444 per vector of eight while weights were read and widened twice a row and offsets made anew; about 250 now), then memory:
// 8192 x 4096 with a residual's gradient 94 -> 69 us (3.9 TB/s), 8192 x 768 with a mean 26 -> 16, 96000 x 128 28 -> 18.  The sum of the shares was
// 47 us for 7104 shares of 128 (four blocks, one share per thread row) and is 5.6; for 888 of 768, 14 -> 5.9 for both dw and db.
//   dx = rstd * (g - mean(g) - xhat * mean(g * xhat))        (LN)
//   dx = rstd * (g - xhat * mean(g * xhat))                   (RMS)      with g = dy * w
// If dres_in is given it is added to dx (gradient arriving through the residual stream).
template <int VPT>
__host__ __device__ constexpr int ring_rows() { return VPT == 1 ? 4 : VPT == 2 ? 3 : 2; }

__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

template <bool LN, bool DB, int VPT>
__global__ void __launch_bounds__(kMaxThreads, VPT == 1 ? 2 : 1)
norm_bwd_kernel(const __nv_bfloat16* __restrict__ dy, const __nv_bfloat16* __restrict__ x, const void* __restrict__ w, int wf32,
                const float* __restrict__ rstd_in, const float* __restrict__ mean_in, const __nv_bfloat16* __restrict__ dres_in,
                __nv_bfloat16* __restrict__ dx, float* __restrict__ dw_part, float* __restrict__ db_part, int rows, int dim, float w_offset) {
  extern __shared__ __align__(16) float scratch[];
  constexpr int kRing = ring_rows<VPT>();
  const int TX = blockDim.x, TY = blockDim.y, threads = TX * TY;
  const int nvec = dim >> 3;
  const int half = reduce_floats(TX, TY);
  float* sum = scratch + (2 * half + 3) / 4 * 4;  // [TY][TX][8] in the end, over the ring
  uint4* ring = reinterpret_cast<uint4*>(sum) + threadIdx.y * TX + threadIdx.x;  // [kRing][2 or 3][VPT][threads]
  const int kinds = dres_in != nullptr ? 3 : 2;
  float dw_acc[VPT][8], db_acc[DB ? VPT : 1][8];
#pragma unroll
  for (int s = 0; s < VPT; ++s)
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      dw_acc[s][j] = 0.f;
      if (DB) db_acc[DB ? s : 0][j] = 0.f;
    }
  const int row_stride = gridDim.x * TY;
  const int first = blockIdx.x * TY + threadIdx.y;
  const int iters = (rows + row_stride - 1) / row_stride;
  Vec8 ww[VPT];
#pragma unroll
  for (int s = 0; s < VPT; ++s)
    if (threadIdx.x + s * TX < nvec) ww[s] = loadw8(w, wf32, (threadIdx.x + s * TX) * 8, w_offset);
    else ww[s] = Vec8{};
  // offsets of this thread's first vector in the row that is fetched and in the row that is worked on
  const long long step = static_cast<long long>(row_stride) * dim;
  long long at_in = static_cast<long long>(first) * dim + threadIdx.x * 8, at_out = at_in;
  int row_in = first, slot_in = 0, slot = 0;
  const int slot_size = kinds * VPT * threads;
  auto fetch = [&]() {  // one group of copies per row, empty ones past the end
    if (row_in < rows) {
      uint4* dst = ring + slot_in * slot_size;
#pragma unroll
      for (int s = 0; s < VPT; ++s)
        if (threadIdx.x + s * TX < nvec) {
          cp_async16(dst + s * threads, dy + at_in + s * TX * 8);
          cp_async16(dst + (VPT + s) * threads, x + at_in + s * TX * 8);
          if (dres_in != nullptr) cp_async16(dst + (2 * VPT + s) * threads, dres_in + at_in + s * TX * 8);
        }
    }
    row_in += row_stride;
    at_in += step;
    slot_in = slot_in + 1 == kRing ? 0 : slot_in + 1;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float rstd = first < rows ? __ldg(rstd_in + first) : 0.f, mean = LN && first < rows ? __ldg(mean_in + first) : 0.f;
#pragma unroll
  for (int it = 0; it < kRing - 1; ++it) fetch();
  for (int it = 0; it < iters; ++it) {
    const int row = first + it * row_stride;
    const float my_rstd = rstd, my_mean = mean;
    const int next = row + row_stride;
    rstd = next < rows ? __ldg(rstd_in + next) : 0.f;
    mean = LN && next < rows ? __ldg(mean_in + next) : 0.f;
    fetch();  // into the place of the previous row
    asm volatile("cp.async.wait_group %0;" ::"n"(kRing - 1) : "memory");
    const uint4* src = ring + slot * slot_size;
    slot = slot + 1 == kRing ? 0 : slot + 1;
    const bool active = row < rows;
    float gw[VPT][8], xh[VPT][8];
    float acc[2] = {0.f, 0.f};
#pragma unroll
    for (int s = 0; s < VPT; ++s) {
      if (active && threadIdx.x + s * TX < nvec) {
        const Vec8 g = unpack8(src[s * threads]), a = unpack8(src[(VPT + s) * threads]);
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          xh[s][j] = (LN ? a.v[j] - my_mean : a.v[j]) * my_rstd;
          gw[s][j] = g.v[j] * ww[s].v[j];
          if (LN) acc[0] += gw[s][j];
          acc[1] += gw[s][j] * xh[s][j];
          dw_acc[s][j] += g.v[j] * xh[s][j];
          if (DB) db_acc[DB ? s : 0][j] += g.v[j];
        }
      }
    }
    if (LN) {
      row_reduce<2>(acc, scratch + (it & 1) * half, TX);
    } else {
      float one[1] = {acc[1]};
      row_reduce<1>(one, scratch + (it & 1) * half, TX);
      acc[1] = one[0];
    }
    const float m1 = LN ? acc[0] / dim * my_rstd : 0.f;
    const float m2 = acc[1] / dim * my_rstd;
    if (active) {
#pragma unroll
      for (int s = 0; s < VPT; ++s) {
        if (threadIdx.x + s * TX < nvec) {
          Vec8 o;
#pragma unroll
          for (int j = 0; j < 8; ++j) o.v[j] = my_rstd * gw[s][j] - (LN ? m1 + xh[s][j] * m2 : xh[s][j] * m2);
          if (dres_in != nullptr) {
            const Vec8 r = unpack8(src[(2 * VPT + s) * threads]);
#pragma unroll
            for (int j = 0; j < 8; ++j) o.v[j] += r.v[j];
          }
          store8(dx + at_out + s * TX * 8, o);
        }
      }
    }
    at_out += step;
  }
#pragma unroll
  for (int which = 0; which < (DB ? 2 : 1); ++which) {
    float* part = which == 0 ? dw_part : db_part;
    if (part == nullptr) continue;
#pragma unroll
    for (int s = 0; s < VPT; ++s) {
      float v[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = which == 0 ? dw_acc[s][j] : db_acc[DB ? s : 0][j];
      if (TY > 1) {
        __syncthreads();
        float4* mine = reinterpret_cast<float4*>(sum + (threadIdx.y * TX + threadIdx.x) * 8);
        mine[0] = make_float4(v[0], v[1], v[2], v[3]);
        mine[1] = make_float4(v[4], v[5], v[6], v[7]);
        __syncthreads();
        if (threadIdx.y == 0)
          for (int t = 1; t < TY; ++t)
#pragma unroll
            for (int j = 0; j < 8; ++j) v[j] += sum[(t * TX + threadIdx.x) * 8 + j];
      }
      const int i = threadIdx.x + s * TX;
      if (threadIdx.y == 0 && i < nvec) {
        float4* p = reinterpret_cast<float4*>(part + static_cast<size_t>(blockIdx.x) * dim + i * 8);
        p[0] = make_float4(v[0], v[1], v[2], v[3]);
        p[1] = make_float4(v[4], v[5], v[6], v[7]);
      }
    }
  }
}

// out[c] = sum over the blocks' shares, for dw and (blockIdx.y = 1) db.  A block owns 32 columns; its 32 thread rows each sum every 32nd
// share, four loads at a time, and are added in a fixed order.
__global__ void __launch_bounds__(1024)
norm_bwd_reduce_kernel(const float* __restrict__ part_w, const float* __restrict__ part_b, void* __restrict__ out_w, void* __restrict__ out_b, int out_bf16,
                       int nparts, int dim) {
  __shared__ float sm[32][33];
  const float* part = blockIdx.y == 0 ? part_w : part_b;
  void* out = blockIdx.y == 0 ? out_w : out_b;
  if (out == nullptr) return;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int c = blockIdx.x * 32 + tx;
  float a[4] = {0.f, 0.f, 0.f, 0.f};
  if (c < dim) {
    int r = ty;
    for (; r + 96 < nparts; r += 128)
#pragma unroll
      for (int j = 0; j < 4; ++j) a[j] += part[static_cast<size_t>(r + 32 * j) * dim + c];
    for (; r < nparts; r += 32) a[0] += part[static_cast<size_t>(r) * dim + c];
  }
  sm[ty][tx] = (a[0] + a[1]) + (a[2] + a[3]);
  __syncthreads();
  const float v = warp_sum(sm[tx][ty]);  // warp ty: the column ty of this block
  const int col = blockIdx.x * 32 + ty;
  if (tx == 0 && col < dim) {
    if (out_bf16) reinterpret_cast<__nv_bfloat16*>(out)[col] = __float2bfloat16(v);
    else reinterpret_cast<float*>(out)[col] = v;
  }
}

// Column sums of x [rows, cols] (a bias's gradient): a block takes 256 columns, a lane eight of them, and every eighth row of its share of the
// rows; part[share][cols] is summed by norm_bwd_reduce_kernel.  Bound by reading x once: 8192 x 3072 takes 9 us with the sum of the shares, a widened
// copy of x and its sum took 55.
__global__ void __launch_bounds__(256)
col_sum_kernel(const __nv_bfloat16* __restrict__ x, long long ld, float* __restrict__ part, int rows, int cols, int rows_per_share) {
  __shared__ __align__(16) float sm[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + lane * 8;
  const int begin = blockIdx.y * rows_per_share, end = min(rows, begin + rows_per_share);
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  if (col < cols) {
    const __nv_bfloat16* p = x + col;
    int r = begin + warp;
    for (; r + 24 < end; r += 32) {
      uint4 v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = __ldg(reinterpret_cast<const uint4*>(p + (r + 8 * j) * ld));
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const Vec8 a = unpack8(v[j]);
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] += a.v[i];
      }
    }
    for (; r < end; r += 8) {
      const Vec8 a = load8(p + r * ld);
#pragma unroll
      for (int i = 0; i < 8; ++i) acc[i] += a.v[i];
    }
  }
#pragma unroll
  for (int i = 0; i < 8; i += 4) *reinterpret_cast<float4*>(&sm[warp][lane * 8 + i]) = make_float4(acc[i], acc[i + 1], acc[i + 2], acc[i + 3]);
  __syncthreads();
  const int c = blockIdx.x * 256 + threadIdx.x;
  if (c < cols) {
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) s += sm[w][threadIdx.x];
    part[static_cast<size_t>(blockIdx.y) * cols + c] = s;
  }
}

// dW[o, c] = sum over the rows of dy[r, o] x[r, c] for a few outputs o (a head's decay or gate, a router): a tensor-core tile would be one CTA that
// walks all rows (8 outputs of 1024 columns over 16384 rows: 101 us), while reading x once takes 6.  A lane holds eight columns by eight outputs, a
// block of eight warps 256 columns of its share of the rows; part[share][o][c] is summed by norm_bwd_reduce_kernel.  blockIdx.z: eight outputs.
__global__ void __launch_bounds__(256)
few_outputs_dw_kernel(const __nv_bfloat16* __restrict__ dy, long long ldy, const __nv_bfloat16* __restrict__ x, long long ldx, float* __restrict__ part,
                      int rows, int outputs, int cols, int rows_per_share) {
  __shared__ __align__(16) float sm[8][256];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 256 + lane * 8, o0 = blockIdx.z * 8;
  const int begin = blockIdx.y * rows_per_share, end = min(rows, begin + rows_per_share);
  float acc[8][8];
#pragma unroll
  for (int o = 0; o < 8; ++o)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[o][j] = 0.f;
  if (col < cols) {
#pragma unroll 2
    for (int r = begin + warp; r < end; r += 8) {
      const Vec8 a = unpack8(__ldg(reinterpret_cast<const uint4*>(x + r * ldx + col)));
      const Vec8 g = unpack8(__ldg(reinterpret_cast<const uint4*>(dy + r * ldy + o0)));
#pragma unroll
      for (int o = 0; o < 8; ++o)
#pragma unroll
        for (int j = 0; j < 8; ++j) acc[o][j] = fmaf(g.v[o], a.v[j], acc[o][j]);
    }
  }
  const int c = blockIdx.x * 256 + threadIdx.x;
#pragma unroll
  for (int o = 0; o < 8; ++o) {
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 8; j += 4)
      *reinterpret_cast<float4*>(&sm[warp][lane * 8 + j]) = make_float4(acc[o][j], acc[o][j + 1], acc[o][j + 2], acc[o][j + 3]);
    __syncthreads();
    if (c < cols) {
      float s = 0.f;
#pragma unroll
      for (int w = 0; w < 8; ++w) s += sm[w][threadIdx.x];
      part[(static_cast<size_t>(blockIdx.y) * outputs + o0 + o) * cols + c] = s;
    }
  }
}

// TX threads per row: one vector each where 512 threads allow it, whole warps (or a power of two below one); TY rows per block of about 256
inline void pick_block(int dim, int& TX, int& TY) {
  const int nvec = dim >> 3;
  TX = 8;
  while (TX < nvec && TX < 32) TX <<= 1;
  if (nvec > 32) TX = (nvec + 31) / 32 * 32;
  if (TX > kMaxThreads) TX = kMaxThreads;
  TY = TX >= 256 ? 1 : 256 / TX;
}

}  // namespace norm
}  // namespace lvb

// y = norm(x (+ residual)) * (w + w_offset) (+ b).  layer_norm: 0 = RMS, 1 = LayerNorm.
// h_out (optional) receives x + residual.  rstd_out / mean_out are fp32 [rows] (saved for backward).
extern "C" int lvb_norm_fwd(const void* x, const void* residual, const void* w, const void* b, int w_is_f32, void* y,
                            void* h_out, float* rstd_out, float* mean_out, int rows, int dim, float eps,
                            float w_offset, int layer_norm, void* stream) {
  using namespace lvb;
  using namespace lvb::norm;
  if (rows <= 0 || dim <= 0 || (dim & 7)) return kErrBadArg;
  int TX, TY;
  pick_block(dim, TX, TY);
  dim3 block(TX, TY);
  dim3 grid((rows + TY - 1) / TY);
  size_t smem = sizeof(float) * 2 * reduce_floats(TX, TY);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto R = reinterpret_cast<const __nv_bfloat16*>(residual);
  auto Y = reinterpret_cast<__nv_bfloat16*>(y);
  auto H = reinterpret_cast<__nv_bfloat16*>(h_out);
  {
    const int vpl = dim / 256;
    const bool by_warp = dim % 256 == 0 && (vpl == 1 || vpl == 2 || vpl == 4 || vpl == 8 || vpl == 16);
    if ((dim >> 3) <= TX && (!by_warp || rows <= kFewRows)) {
      auto kern = layer_norm ? norm_fwd_row_kernel<true> : norm_fwd_row_kernel<false>;
      return launch_chained(kern, grid, block, smem, s, X, R, w, b, w_is_f32, Y, H, rstd_out, mean_out, rows, dim, eps, w_offset) == cudaSuccess ? kErrOk : kErrCuda;
    }
    if (by_warp) {
      const dim3 wgrid((rows + 3) / 4);
#define LVB_NORM_WARP(LNV, V)                                                                                                  \
  if (R != nullptr)                                                                                                            \
    norm_fwd_warp_kernel<LNV, V, true><<<wgrid, 128, 0, s>>>(X, R, w, b, w_is_f32, Y, H, rstd_out, mean_out, rows, eps, w_offset); \
  else                                                                                                                         \
    norm_fwd_warp_kernel<LNV, V, false><<<wgrid, 128, 0, s>>>(X, R, w, b, w_is_f32, Y, H, rstd_out, mean_out, rows, eps, w_offset)
#define LVB_NORM_WARP_V(LNV)                                                                                                   \
  switch (vpl) {                                                                                                               \
    case 1: LVB_NORM_WARP(LNV, 1); break;                                                                                      \
    case 2: LVB_NORM_WARP(LNV, 2); break;                                                                                      \
    case 4: LVB_NORM_WARP(LNV, 4); break;                                                                                      \
    case 8: LVB_NORM_WARP(LNV, 8); break;                                                                                      \
    default: LVB_NORM_WARP(LNV, 16); break;                                                                                    \
  }
      if (layer_norm) { LVB_NORM_WARP_V(true) } else { LVB_NORM_WARP_V(false) }
#undef LVB_NORM_WARP_V
#undef LVB_NORM_WARP
      return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
    }
  }
  if (layer_norm)
    norm_fwd_kernel<true><<<grid, block, smem, s>>>(X, R, w, b, w_is_f32, Y, H, rstd_out, mean_out, rows, dim, eps, w_offset);
  else
    norm_fwd_kernel<false><<<grid, block, smem, s>>>(X, R, w, b, w_is_f32, Y, H, rstd_out, mean_out, rows, dim, eps, w_offset);
  return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
}

namespace lvb {
namespace norm {
inline int vpt_room(int vpt) { return vpt <= 1 ? 1 : vpt <= 2 ? 2 : 4; }
}  // namespace norm
}  // namespace lvb

// Backward of lvb_norm_fwd.  x is the normalised input (x + residual if a residual was added).  scratch: fp32 [2 * nparts * dim], 16-byte
// aligned, where nparts = lvb_norm_bwd_parts(rows, dim); dw / db are [dim], bf16 with out_bf16 and fp32 otherwise (either may be null).
extern "C" int lvb_norm_bwd_parts(int rows, int dim) {
  using namespace lvb::norm;
  int TX, TY;
  pick_block(dim, TX, TY);
  // as many blocks as an SM's registers hold (64 per thread; one block of wide rows), and two rows per thread row, so that few rows do not make
  // as many shares
  const int blocks = (rows + 2 * TY - 1) / (2 * TY);
  const int cap = lvb::num_sms() * ((dim >> 3) > kMaxThreads ? 1 : 1024 / (TX * TY));
  return blocks < cap ? blocks : cap;
}

extern "C" int lvb_norm_bwd(const void* dy, const void* x, const void* w, int w_is_f32, const float* rstd,
                            const float* mean, const void* dres_in, void* dx, void* dw, void* db, int out_bf16, float* scratch,
                            int rows, int dim, float w_offset, int layer_norm, void* stream) {
  using namespace lvb;
  using namespace lvb::norm;
  if (rows <= 0 || dim <= 0 || (dim & 7)) return kErrBadArg;
  int TX, TY;
  pick_block(dim, TX, TY);
  if ((dim >> 3) > TX * kMaxVecPerThread) return kErrTooLarge;
  const int nparts = lvb_norm_bwd_parts(rows, dim);
  dim3 block(TX, TY);
  const int base = sizeof(float) * ((2 * reduce_floats(TX, TY) + 3) / 4 * 4);
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  float* dw_part = dw != nullptr ? scratch : nullptr;
  float* db_part = db != nullptr ? scratch + static_cast<size_t>(nparts) * dim : nullptr;
  auto DY = reinterpret_cast<const __nv_bfloat16*>(dy);
  auto X = reinterpret_cast<const __nv_bfloat16*>(x);
  auto DR = reinterpret_cast<const __nv_bfloat16*>(dres_in);
  auto DX = reinterpret_cast<__nv_bfloat16*>(dx);
  const int vpt = ((dim >> 3) + TX - 1) / TX;
  auto go = [&](auto kern, int ring) {
    const int smem = base + ring * (dres_in != nullptr ? 3 : 2) * vpt_room(vpt) * TX * TY * 16;
    // the same limit from every call (four vectors, three kinds, two rows are 192 KB): another thread may be about to launch a wider row
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess) return kErrCuda;
    kern<<<nparts, block, smem, s>>>(DY, X, w, w_is_f32, rstd, mean, DR, DX, dw_part, db_part, rows, dim, w_offset);
    return kErrOk;
  };
  int rc;
#define LVB_NORM_BWD(LN, DB)                                                      \
  if (vpt <= 1) rc = go(norm_bwd_kernel<LN, DB, 1>, ring_rows<1>());              \
  else if (vpt <= 2) rc = go(norm_bwd_kernel<LN, DB, 2>, ring_rows<2>());         \
  else rc = go(norm_bwd_kernel<LN, DB, 4>, ring_rows<4>())
  if (layer_norm) { LVB_NORM_BWD(true, true); } else if (db != nullptr) { LVB_NORM_BWD(false, true); } else { LVB_NORM_BWD(false, false); }
#undef LVB_NORM_BWD
  if (rc != kErrOk) return rc;
  if (dw != nullptr || db != nullptr)
    norm_bwd_reduce_kernel<<<dim3((dim + 31) / 32, db != nullptr ? 2 : 1), 1024, 0, s>>>(dw_part, db_part, dw, db, out_bf16, nparts, dim);
  return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
}

// Shares of the rows that lvb_col_sum works on: about four blocks per SM, at least 32 rows each.
extern "C" int lvb_col_sum_shares(int rows, int cols) {
  const int wanted = 4 * lvb::num_sms() / ((cols + 255) / 256), most = (rows + 31) / 32;
  return wanted < 1 ? 1 : wanted < most ? wanted : most;
}

// out[c] = sum over the rows of x[r, c], fp32 sums, stored as bf16 or fp32.  x: row stride ld, cols and ld multiples of 8, 16-byte aligned;
// scratch: fp32 [lvb_col_sum_shares(rows, cols), cols].
extern "C" int lvb_col_sum(const void* x, long long ld, void* out, int out_bf16, float* scratch, int rows, int cols, void* stream) {
  using namespace lvb;
  using namespace lvb::norm;
  if (rows <= 0 || cols <= 0 || (cols & 7) || (ld & 7) || (reinterpret_cast<uintptr_t>(x) & 15)) return kErrBadArg;
  int shares = lvb_col_sum_shares(rows, cols);
  const int per = (rows + shares - 1) / shares;
  shares = (rows + per - 1) / per;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  col_sum_kernel<<<dim3((cols + 255) / 256, shares), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(x), ld, scratch, rows, cols, per);
  norm_bwd_reduce_kernel<<<dim3((cols + 31) / 32, 1), 1024, 0, s>>>(scratch, nullptr, out, nullptr, out_bf16, shares, cols);
  return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
}

// Shares of the rows that lvb_few_outputs_dw works on: about two blocks per SM, at least 64 rows each.
extern "C" int lvb_few_outputs_dw_shares(int rows, int outputs, int cols) {
  const int wanted = 2 * lvb::num_sms() / ((cols + 255) / 256 * (outputs / 8 > 0 ? outputs / 8 : 1)), most = (rows + 63) / 64;
  return wanted < 1 ? 1 : wanted < most ? wanted : most;
}

// dw[outputs, cols] = dy[rows, outputs]^T x[rows, cols], fp32 sums stored as bf16 or fp32; outputs, cols and the row strides multiples of 8, the
// pointers 16-byte aligned.  scratch: fp32 [lvb_few_outputs_dw_shares(...), outputs, cols].
extern "C" int lvb_few_outputs_dw(const void* dy, long long ldy, const void* x, long long ldx, void* dw, int out_bf16, float* scratch, int rows, int outputs,
                                  int cols, void* stream) {
  using namespace lvb;
  using namespace lvb::norm;
  if (rows <= 0 || outputs <= 0 || cols <= 0 || ((outputs | cols | ldy | ldx) & 7) || ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dy)) & 15))
    return kErrBadArg;
  int shares = lvb_few_outputs_dw_shares(rows, outputs, cols);
  const int per = (rows + shares - 1) / shares;
  shares = (rows + per - 1) / per;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  few_outputs_dw_kernel<<<dim3((cols + 255) / 256, shares, outputs / 8), 256, 0, s>>>(reinterpret_cast<const __nv_bfloat16*>(dy), ldy,
                                                                                     reinterpret_cast<const __nv_bfloat16*>(x), ldx, scratch, rows, outputs, cols, per);
  const int dim = outputs * cols;
  norm_bwd_reduce_kernel<<<dim3((dim + 31) / 32, 1), 1024, 0, s>>>(scratch, nullptr, dw, nullptr, out_bf16, shares, dim);
  return cudaGetLastError() == cudaSuccess ? kErrOk : kErrCuda;
}
