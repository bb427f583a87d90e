// Token sampling: per row, greedy arg-max when the temperature is 0, otherwise a categorical draw from softmax(z / T) by
// the Gumbel-max trick, plus the log-probability of the chosen token (src/levanter/layers/sampler.py:35-81).
//
// A cluster of up to eight CTAs makes a single pass over a row: each thread keeps an online log-sum-exp (running max, scaled
// sum, eight logits at a time), the best perturbed score z/T + g and the best raw score, and the first CTA merges the eight
// results over distributed shared memory; the noise g = -log(-log(u)) comes from a counter-based
// hash of (row seed, vocabulary index), so a row's draw depends only on its own seed, never on what else is in the batch.
// Ties go to the lower index, which keeps the choice independent of the block size.
#include <cooperative_groups.h>

#include "common.cuh"

namespace lvb {
namespace sampler {

constexpr int kThreads = 256;

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__device__ __forceinline__ float gumbel(unsigned long long seed, int idx) {
  const unsigned long long h = mix64(seed ^ (static_cast<unsigned long long>(idx) * 0x9E3779B97F4A7C15ull));
  const float u = (static_cast<float>(h >> 40) + 0.5f) * (1.0f / 16777216.0f);  // (0, 1)
  return -__logf(-__logf(u));
}

struct Acc {
  float m, s;        // online log-sum-exp of z / T
  float best;        // best perturbed score
  int best_idx;
  float zbest;       // z / T at best_idx
};

__device__ __forceinline__ void merge(Acc& a, const Acc& b) {
  const float m = fmaxf(a.m, b.m);
  a.s = (a.m == -INFINITY ? 0.f : a.s * __expf(a.m - m)) + (b.m == -INFINITY ? 0.f : b.s * __expf(b.m - m));
  a.m = m;
  if (b.best > a.best || (b.best == a.best && b.best_idx < a.best_idx)) {
    a.best = b.best;
    a.best_idx = b.best_idx;
    a.zbest = b.zbest;
  }
}

template <typename T>
__global__ void __launch_bounds__(kThreads) sample_kernel(const T* __restrict__ logits, long long row_stride, int vocab,
                                                          const float* __restrict__ temps, const long long* __restrict__ seeds,
                                                          int* __restrict__ tokens, float* __restrict__ logprobs) {
  namespace cg = cooperative_groups;
  const cg::cluster_group cluster = cg::this_cluster();
  const int parts = static_cast<int>(cluster.num_blocks()), part = static_cast<int>(cluster.block_rank());
  chain_wait();
  const int row = blockIdx.x / parts;
  const T* z = logits + static_cast<long long>(row) * row_stride;
  const float t = temps[row];
  const bool greedy = (t == 0.f);
  const float inv_t = greedy ? 1.f : 1.f / t;
  const unsigned long long seed = static_cast<unsigned long long>(seeds[row]);
  Acc a{-INFINITY, 0.f, -INFINITY, 0x7fffffff, 0.f};
  auto visit = [&](float v, int i) {
    v *= inv_t;
    if (v > a.m) { a.s = a.s * __expf(a.m - v) + 1.f; a.m = v; }
    else if (v > -INFINITY) a.s += __expf(v - a.m);
    const float score = greedy ? v : v + gumbel(seed, i);
    if (score > a.best) { a.best = score; a.best_idx = i; a.zbest = v; }
  };
  auto visit8 = [&](const uint4& w, int i) {
    float v[8];
    const uint32_t u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u[j]));
      v[2 * j] = f.x * inv_t;
      v[2 * j + 1] = f.y * inv_t;
    }
    const float m = fmaxf(fmaxf(fmaxf(v[0], v[1]), fmaxf(v[2], v[3])), fmaxf(fmaxf(v[4], v[5]), fmaxf(v[6], v[7])));
    if (m > a.m) { a.s *= __expf(a.m - m); a.m = m; }
#pragma unroll
    for (int j = 0; j < 8; ++j) a.s += v[j] > -INFINITY ? __expf(v[j] - a.m) : 0.f;
    if (greedy) {
      if (m > a.best) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (v[j] > a.best) { a.best = v[j]; a.best_idx = i + j; a.zbest = v[j]; }
      }
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float score = v[j] + gumbel(seed, i + j);
        if (score > a.best) { a.best = score; a.best_idx = i + j; a.zbest = v[j]; }
      }
    }
  };
  int done = 0;
  if constexpr (sizeof(T) == 2) {
    // 16-byte loads (8 logits) when the row starts on a 16-byte boundary, four under way at a time
    if ((reinterpret_cast<uintptr_t>(z) & 15) == 0) {
      const int nvec = vocab / 8;
      const int end = static_cast<int>(static_cast<long long>(nvec) * (part + 1) / parts);
      const uint4* zv = reinterpret_cast<const uint4*>(z);
      int c = static_cast<int>(static_cast<long long>(nvec) * part / parts) + threadIdx.x;
      for (; c + 3 * kThreads < end; c += 4 * kThreads) {
        uint4 w[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) w[j] = __ldg(zv + c + j * kThreads);
#pragma unroll
        for (int j = 0; j < 4; ++j) visit8(w[j], (c + j * kThreads) * 8);
      }
      for (; c < end; c += kThreads) visit8(__ldg(zv + c), c * 8);
      done = nvec * 8;
    }
  }
  for (int i = done + part * kThreads + threadIdx.x; i < vocab; i += parts * kThreads) {
    float v;
    if constexpr (sizeof(T) == 2) v = __bfloat162float(z[i]); else v = z[i];
    visit(v, i);
  }
  __shared__ Acc sm[kThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    Acc b;
    b.m = __shfl_xor_sync(0xffffffffu, a.m, o);
    b.s = __shfl_xor_sync(0xffffffffu, a.s, o);
    b.best = __shfl_xor_sync(0xffffffffu, a.best, o);
    b.best_idx = __shfl_xor_sync(0xffffffffu, a.best_idx, o);
    b.zbest = __shfl_xor_sync(0xffffffffu, a.zbest, o);
    merge(a, b);
  }
  if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = a;
  __syncthreads();
  Acc r = sm[0];
  if (threadIdx.x == 0) {
    for (int w = 1; w < kThreads / 32; ++w) merge(r, sm[w]);
    sm[0] = r;
  }
  if (parts > 1) {
    cluster.sync();
    if (part == 0 && threadIdx.x == 0)
      for (int p = 1; p < parts; ++p) merge(r, *cluster.map_shared_rank(&sm[0], p));
    cluster.sync();  // the others' shared memory has been read
  }
  if (part == 0 && threadIdx.x == 0) {
    tokens[row] = r.best_idx;
    logprobs[row] = r.zbest - (r.m + __logf(r.s));
  }
}

// CTAs per row.  One CTA needs 60 us for 128256 logits, whatever the number of rows up to two per SM (it is bound by its own chain of logits); eight
// need 9.5 for one row, 14 for 64, 35 for 256 (65 before).  More rows than CTAs that fit at once gain nothing from a split, and a part below 4096
// logits is less than one round of loads.
inline int parts_for(int rows, int vocab) {
  int parts = 8;
  while (parts > 1 && (vocab / parts < 4096 || static_cast<long long>(rows) * parts > 2048)) parts >>= 1;
  return parts;
}

template <typename T>
int launch(const T* logits, long long row_stride, int rows, int vocab, const float* temps, const long long* seeds, int* tokens, float* logprobs,
           cudaStream_t s) {
  const int parts = parts_for(rows, vocab);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(rows) * parts);
  cfg.blockDim = dim3(kThreads);
  cfg.stream = s;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = parts;
  attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, sample_kernel<T>, logits, row_stride, vocab, temps, seeds, tokens, logprobs) == cudaSuccess ? kErrOk : kErrCuda;
}

}  // namespace sampler
}  // namespace lvb

// logits: [rows, vocab] fp32 (is_bf16 = 0) or bf16 with row stride `row_stride` elements; temps fp32 [rows];
// seeds int64 [rows]; tokens int32 [rows]; logprobs fp32 [rows].
extern "C" int lvb_sample(const void* logits, int is_bf16, long long row_stride, int rows, int vocab, const float* temps,
                          const long long* seeds, int* tokens, float* logprobs, void* stream) {
  using namespace lvb;
  using namespace lvb::sampler;
  if (rows <= 0 || vocab <= 0) return kErrBadArg;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  if (is_bf16)
    return launch(reinterpret_cast<const __nv_bfloat16*>(logits), row_stride, rows, vocab, temps, seeds, tokens, logprobs, s);
  return launch(reinterpret_cast<const float*>(logits), row_stride, rows, vocab, temps, seeds, tokens, logprobs, s);
}
