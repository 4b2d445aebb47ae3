// Multi-tensor LAMB: every parameter tensor of the model in three launches.
// Stands in for apex.optimizers.FusedLAMB, which the reference's BERT driver
// imports (examples/BertPretraining/run_pretraining_conef.py:42,449-450) and
// which is not available without apex.
//   launch 1: squared global gradient norm (for clipping)
//   launch 2: moments, update direction u = m_hat / (sqrt(v_hat) + eps) + wd * p,
//             written over the gradient; squared norms of p and u per tensor
//   launch 3: p -= lr * trust * u with trust = |p| / |u| (1 when either is 0)
#include "common.cuh"

constexpr int L_THREADS = 512;
// All kernels are bound by memory: 28 bytes per element are unavoidable (p, g, m, v in; p, m, v out), the update
// direction that passes through the gradient adds 8.  A CTA of the two update kernels takes a slice of L_SLICE
// elements of a chunk: with one CTA per 65,536-element chunk the four matrices and two feed-forward blocks of a
// BERT-large layer (12.6 M elements, 192 chunks) were 1.3 CTAs per SM with one 4-byte load per array and thread in
// flight.  Slices give ten CTAs per SM, 16-byte accesses where pointers and chunk starts are aligned, and shorter
// sums.  Measured on that layer, us: stage 1 110 -> 52 (its 28 bytes per element at 6.7 TB/s, the copy rate),
// stage 2 78 -> 20.  The norm of all gradients keeps a CTA per chunk (10 us either way): with eight times the atomics
// on one sum the results were further from 64 bits than at one CTA per chunk (6.2e-8 against 4.9e-8 relative).
constexpr int L_SLICE = 8192;

struct LambSlice { long long lo, hi; };
__device__ __forceinline__ LambSlice lamb_slice(long long chunk, int chunk_elems, int parts, int part, long long numel) {
  const long long c0 = chunk * chunk_elems, c1 = min(c0 + (long long)chunk_elems, numel);
  LambSlice s;
  s.lo = min(c0 + (long long)part * L_SLICE, c1);
  s.hi = min(s.lo + (long long)L_SLICE, c1);
  return s;
}

__global__ void __launch_bounds__(L_THREADS)
k_lamb_gnorm(const ConefLambTensor* __restrict__ tensors, const int2* __restrict__ chunks, int chunk_elems,
             float* __restrict__ norms) {
  __shared__ float scratch[33];
  const int2 c = chunks[blockIdx.x];
  const ConefLambTensor T = tensors[c.x];
  const long long lo = (long long)c.y * chunk_elems;
  const LambSlice S = {lo, min(lo + (long long)chunk_elems, T.numel)};      // one CTA and one atomic per chunk
  float s = 0.f;
  long long i = S.lo;
  if (((reinterpret_cast<uintptr_t>(T.g + S.lo)) & 15) == 0) {
    const long long hi4 = S.lo + ((S.hi - S.lo) & ~3LL);
#pragma unroll 4
    for (long long k = S.lo + 4LL * threadIdx.x; k < hi4; k += 4LL * L_THREADS) {
      const float4 g = *reinterpret_cast<const float4*>(T.g + k);
      s = fmaf(g.x, g.x, s); s = fmaf(g.y, g.y, s); s = fmaf(g.z, g.z, s); s = fmaf(g.w, g.w, s);
    }
    i = hi4;
  }
  for (i += threadIdx.x; i < S.hi; i += L_THREADS) { const float g = T.g[i]; s = fmaf(g, g, s); }
  s = block_sum(s, scratch);
  if (threadIdx.x == 0) atomicAdd(&norms[0], s);
}

struct LambCoef { float beta1, beta2, eps, bc1, bc2, gmul, wd; };

// one element: the moments in place, the update direction into g
__device__ __forceinline__ void lamb_element(const LambCoef& K, float p, float& g, float& m, float& v, float& pn,
                                             float& un) {
  const float gs = g * K.gmul;
  m = K.beta1 * m + (1.f - K.beta1) * gs;
  v = K.beta2 * v + (1.f - K.beta2) * gs * gs;
  const float u = (m / K.bc1) / (sqrtf(v / K.bc2) + K.eps) + K.wd * p;
  g = u;
  pn = fmaf(p, p, pn);
  un = fmaf(u, u, un);
}

// The moments go through the caches marked for early eviction: nothing reads them again in this step, while
// p and the update direction are read by the next kernel, which starts with the slices that were written last.
__global__ void __launch_bounds__(L_THREADS, 3)
k_lamb_stage1(const ConefLambTensor* __restrict__ tensors, const int2* __restrict__ chunks, int chunk_elems, int parts,
              float* __restrict__ norms, float beta1, float beta2, float eps, float bc1, float bc2,
              float grad_scale, float max_grad_norm) {
  __shared__ float scratch[33];
  const int2 c = chunks[blockIdx.x / parts];
  const ConefLambTensor T = tensors[c.x];
  const LambSlice S = lamb_slice(c.y, chunk_elems, parts, blockIdx.x % parts, T.numel);
  // gradient un-scaling and global-norm clipping folded into one factor
  float gmul = 1.f / grad_scale;
  if (max_grad_norm > 0.f) {
    const float gn = sqrtf(norms[0]) * gmul;
    if (gn > max_grad_norm) gmul *= max_grad_norm / gn;
  }
  const LambCoef K = {beta1, beta2, eps, bc1, bc2, gmul, T.weight_decay};
  float pn = 0.f, un = 0.f;
  long long i = S.lo;
  const bool vec = ((reinterpret_cast<uintptr_t>(T.p + S.lo) | reinterpret_cast<uintptr_t>(T.g + S.lo) |
                     reinterpret_cast<uintptr_t>(T.m + S.lo) | reinterpret_cast<uintptr_t>(T.v + S.lo)) & 15) == 0;
  if (vec) {
    const long long hi4 = S.lo + ((S.hi - S.lo) & ~3LL);
    for (long long k = S.lo + 4LL * threadIdx.x; k < hi4; k += 4LL * L_THREADS) {
      float4 g = *reinterpret_cast<const float4*>(T.g + k);
      const float4 p = *reinterpret_cast<const float4*>(T.p + k);
      float4 m = __ldcs(reinterpret_cast<const float4*>(T.m + k));
      float4 v = __ldcs(reinterpret_cast<const float4*>(T.v + k));
      lamb_element(K, p.x, g.x, m.x, v.x, pn, un);
      lamb_element(K, p.y, g.y, m.y, v.y, pn, un);
      lamb_element(K, p.z, g.z, m.z, v.z, pn, un);
      lamb_element(K, p.w, g.w, m.w, v.w, pn, un);
      __stcs(reinterpret_cast<float4*>(T.m + k), m);
      __stcs(reinterpret_cast<float4*>(T.v + k), v);
      *reinterpret_cast<float4*>(T.g + k) = g;
    }
    i = hi4;
  }
  for (i += threadIdx.x; i < S.hi; i += L_THREADS) {
    float g = T.g[i], m = T.m[i], v = T.v[i];
    lamb_element(K, T.p[i], g, m, v, pn, un);
    T.m[i] = m;
    T.v[i] = v;
    T.g[i] = g;
  }
  pn = block_sum(pn, scratch);
  un = block_sum(un, scratch);
  if (threadIdx.x == 0) {
    atomicAdd(&norms[1 + 2 * c.x], pn);
    atomicAdd(&norms[2 + 2 * c.x], un);
  }
}

__global__ void __launch_bounds__(L_THREADS)
k_lamb_stage2(const ConefLambTensor* __restrict__ tensors, const int2* __restrict__ chunks, int chunk_elems, int parts,
              const float* __restrict__ norms, float lr) {
  const int b = gridDim.x - 1 - blockIdx.x;      // backwards: the slices stage 1 wrote last are still in L2
  const int2 c = chunks[b / parts];
  const ConefLambTensor T = tensors[c.x];
  const LambSlice S = lamb_slice(c.y, chunk_elems, parts, b % parts, T.numel);
  const float pn = sqrtf(norms[1 + 2 * c.x]), un = sqrtf(norms[2 + 2 * c.x]);
  const float trust = (pn > 0.f && un > 0.f) ? pn / un : 1.f;
  const float step = lr * trust;
  long long i = S.lo;
  if (((reinterpret_cast<uintptr_t>(T.p + S.lo) | reinterpret_cast<uintptr_t>(T.g + S.lo)) & 15) == 0) {
    const long long hi4 = S.lo + ((S.hi - S.lo) & ~3LL);
#pragma unroll 4
    for (long long k = S.lo + 4LL * threadIdx.x; k < hi4; k += 4LL * L_THREADS) {
      float4 p = *reinterpret_cast<const float4*>(T.p + k);
      const float4 u = *reinterpret_cast<const float4*>(T.g + k);
      p.x -= step * u.x; p.y -= step * u.y; p.z -= step * u.z; p.w -= step * u.w;
      *reinterpret_cast<float4*>(T.p + k) = p;
    }
    i = hi4;
  }
  for (i += threadIdx.x; i < S.hi; i += L_THREADS) T.p[i] -= step * T.g[i];
}

extern "C" int conef_lamb_step(const ConefLambTensor* tensors, int ntensors, const int2* chunks, int nchunks,
                               int chunk_elems, float* norms, float lr, float beta1, float beta2, float eps,
                               int step, int bias_correction, float grad_scale, float max_grad_norm,
                               cudaStream_t stream) {
  if (ntensors <= 0 || nchunks <= 0) return 0;
  CONEF_CUDA(cudaMemsetAsync(norms, 0, sizeof(float) * (size_t)(1 + 2 * ntensors), stream));
  const int parts = chunk_elems > L_SLICE ? (chunk_elems + L_SLICE - 1) / L_SLICE : 1;
  if ((long long)nchunks * parts > 0x7fffffffLL) { conef_set_error("lamb_step: %d chunks are too many", nchunks); return 2; }
  const int grid = nchunks * parts;
  if (max_grad_norm > 0.f) {
    k_lamb_gnorm<<<nchunks, L_THREADS, 0, stream>>>(tensors, chunks, chunk_elems, norms);
    CONEF_CHECK_LAUNCH("k_lamb_gnorm");
  }
  float bc1 = 1.f, bc2 = 1.f;
  if (bias_correction) {
    bc1 = 1.f - powf(beta1, (float)step);
    bc2 = 1.f - powf(beta2, (float)step);
  }
  k_lamb_stage1<<<grid, L_THREADS, 0, stream>>>(tensors, chunks, chunk_elems, parts, norms, beta1, beta2, eps, bc1, bc2,
                                                 grad_scale, max_grad_norm);
  CONEF_CHECK_LAUNCH("k_lamb_stage1");
  k_lamb_stage2<<<grid, L_THREADS, 0, stream>>>(tensors, chunks, chunk_elems, parts, norms, lr);
  CONEF_CHECK_LAUNCH("k_lamb_stage2");
  return 0;
}

// ---------------------------------------------------------------------------
// Allocation-free variant (declared in conef_noalloc.h): the norm scratch lives in
// static device memory instead of a caller-provided buffer.
#include "conef_noalloc.h"

static __device__ __align__(256) float g_lamb_scratch[1 + 2 * CONEF_NOALLOC_MAX_TENSORS];

// In host code the array's name is only a handle; kernels need its device address,
// looked up once per device with that device current.
static float* g_lamb_scratch_addr[64] = {nullptr};

extern "C" int conef_lamb_step_noalloc(const ConefLambTensor* tensors, int ntensors, const int2* chunks,
                                       int nchunks, int chunk_elems, float lr, float beta1, float beta2,
                                       float eps, int step, int bias_correction, float grad_scale,
                                       float max_grad_norm, cudaStream_t stream) {
  if (ntensors <= 0 || nchunks <= 0) return 0;
  if (ntensors > CONEF_NOALLOC_MAX_TENSORS) {
    conef_set_error("conef_lamb_step_noalloc: %d tensors exceed the built-in scratch of %d tensors; "
                    "use conef_lamb_step with a caller-provided buffer", ntensors, CONEF_NOALLOC_MAX_TENSORS);
    return 2;
  }
  int dev = -1;
  CONEF_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) { conef_set_error("conef_lamb_step_noalloc: unsupported device index %d", dev); return 2; }
  if (g_lamb_scratch_addr[dev] == nullptr) {
    float* addr = nullptr;
    CONEF_CUDA(cudaGetSymbolAddress((void**)&addr, g_lamb_scratch));
    g_lamb_scratch_addr[dev] = addr;
  }
  // the same memset and kernels as the entry point with a caller-provided buffer: the accumulators
  // this call uses are cleared first, the rest of the array keeps old values
  return conef_lamb_step(tensors, ntensors, chunks, nchunks, chunk_elems, g_lamb_scratch_addr[dev], lr, beta1, beta2,
                         eps, step, bias_correction, grad_scale, max_grad_norm, stream);
}

// ---------------------------------------------------------------------------
// Multi-tensor SGD with momentum: one launch over all tensors (the same tensor / chunk tables as LAMB; `v` is
// unused).  torch.optim.SGD semantics: g += weight_decay p; buf = first ? g : momentum buf + (1 - dampening) g;
// update = nesterov ? g + momentum buf : buf; p -= lr update.  PyTorch's foreach path is about fifteen launches
// and three passes over parameters, gradients and buffers; this is one pass (read p, g, buf; write p, buf).
__global__ void __launch_bounds__(L_THREADS)
k_sgd_step(const ConefLambTensor* __restrict__ tensors, const int2* __restrict__ chunks, int chunk_elems, float lr,
           float momentum, float dampening, int nesterov, int first) {
  const int2 c = chunks[blockIdx.x];
  const ConefLambTensor T = tensors[c.x];
  const long long lo = (long long)c.y * chunk_elems;
  const long long hi = min(lo + (long long)chunk_elems, T.numel);
  const float wd = T.weight_decay;
  const bool vec = ((reinterpret_cast<uintptr_t>(T.p) | reinterpret_cast<uintptr_t>(T.g) |
                     reinterpret_cast<uintptr_t>(T.m)) & 15) == 0 && (lo & 3) == 0;
  long long i = lo;
  if (vec) {
    const long long hi4 = lo + ((hi - lo) & ~3LL);
    for (i = lo + 4LL * threadIdx.x; i < hi4; i += 4LL * L_THREADS) {
      float4 p = *reinterpret_cast<const float4*>(T.p + i);
      const float4 g4 = *reinterpret_cast<const float4*>(T.g + i);
      float4 b = momentum != 0.f && !first ? *reinterpret_cast<const float4*>(T.m + i) : make_float4(0.f, 0.f, 0.f, 0.f);
      float* pp = reinterpret_cast<float*>(&p);
      const float* gp = reinterpret_cast<const float*>(&g4);
      float* bp = reinterpret_cast<float*>(&b);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float g = fmaf(wd, pp[k], gp[k]);
        float u = g;
        if (momentum != 0.f) {
          bp[k] = first ? g : fmaf(momentum, bp[k], (1.f - dampening) * g);
          u = nesterov ? fmaf(momentum, bp[k], g) : bp[k];
        }
        pp[k] = fmaf(-lr, u, pp[k]);
      }
      *reinterpret_cast<float4*>(T.p + i) = p;
      if (momentum != 0.f) *reinterpret_cast<float4*>(T.m + i) = b;
    }
    i = hi4;
  }
  for (i += threadIdx.x; i < hi; i += L_THREADS) {
    const float g = fmaf(wd, T.p[i], T.g[i]);
    float u = g;
    if (momentum != 0.f) {
      const float b = first ? g : fmaf(momentum, T.m[i], (1.f - dampening) * g);
      T.m[i] = b;
      u = nesterov ? fmaf(momentum, b, g) : b;
    }
    T.p[i] = fmaf(-lr, u, T.p[i]);
  }
}

extern "C" int conef_sgd_step(const ConefLambTensor* tensors, int ntensors, const int2* chunks, int nchunks,
                              int chunk_elems, float lr, float momentum, float dampening, int nesterov, int first,
                              cudaStream_t stream) {
  if (ntensors <= 0 || nchunks <= 0) return 0;
  k_sgd_step<<<nchunks, L_THREADS, 0, stream>>>(tensors, chunks, chunk_elems, lr, momentum, dampening, nesterov, first);
  CONEF_CHECK_LAUNCH("k_sgd_step");
  return 0;
}
