// CUDA-core (fp32 FFMA) kernels for every phase of the predictive-coding train step.
// They handle any shape (ragged, tiny terminal widths, unaligned leading dimensions) and
// are the path for layers outside the tensor-core run.  One launch covers a whole range
// of layers: blockIdx.z selects the layer, blockIdx.x/y the output tile; CTAs outside a
// layer's own tile grid return at once.
#pragma once
#include <cuda_bf16.h>

#include <type_traits>

#include "dpc_math.cuh"

namespace dpc
{
constexpr int NTHREADS = 256;

// mode of a weight update
enum
{
  WG_LEARN = 0, // UpdateWeights: g = fe (or e_above for Simple), rate lr, optimizer
  WG_DFA = 1,   // DirectFeedbackUpdate: g = fe (holds proj), rate fl, plain accumulate
  // or-ed in: only store the raw sum g^T zin in the layer's gradient staging buffer g_W; the
  // update is applied later by apply_gradients_kernel (after a sum over batch shards)
  WG_GRAD_ONLY = 2
};
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool valid)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(valid ? 4 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool valid)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(valid ? 16 : 0)
               : "memory");
}

__device__ __forceinline__ bool aligned16(const void* p)
{
  return (reinterpret_cast<uintptr_t>(p) & 15) == 0;
}

__device__ __forceinline__ void block_energy_add(float local, double* energy)
{
  __shared__ float warp_sums[NTHREADS / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    local += __shfl_xor_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0)
    warp_sums[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    float s = 0.0f;
#pragma unroll
    for (int w = 0; w < NTHREADS / 32; ++w)
      s += warp_sums[w];
    atomicAdd(energy, (double)(0.5f * s));
  }
}

// ---------------------------------------------------------------------------------------
// Row split over a thread-block cluster.  The reductions over the batch below (Psi update, bias
// column sums) give one block a strip of columns and all rows, which fills the GPU when a launch
// covers thousands of layers but not when it covers four.  Such launches go out as clusters of R
// CTAs along z: CTA r of a cluster takes every R-th group of rows, leaves its partial sums in its
// own shared memory, and CTA 0 adds the others' in rank order through distributed shared memory
// (a fixed order: the result does not depend on timing).  Without the cluster attribute R is 1.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t rows_cluster_rank()
{
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t rows_cluster_size()
{
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void rows_cluster_sync()
{
  asm volatile("barrier.cluster.arrive.release.aligned;\n"
               "barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the float at the same shared-memory address in CTA `rank` of the cluster
__device__ __forceinline__ float rows_cluster_load(const float* own, uint32_t rank)
{
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(own);
  uint32_t ra;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(ra) : "memory");
  return v;
}

// ---------------------------------------------------------------------------------------
// Forward pass of narrow layers (at most 16 output units: the heads, e.g. 1024 -> 10).  The tiled
// kernel below gives such a layer one column of 64 x 64 tiles, i.e. batch/64 CTAs that each walk
// all of K: latency-bound (96 us for 4096 x 10 x 1024 against 3 us of traffic).  Here a warp owns
// one batch row: its lanes stride over K with 16-byte loads of the row and of the (L1-resident)
// weight rows, the partial dot products are reduced by shuffles, and lane 2j finishes output unit
// j with the same epilogue as the tiled kernel.  Needs size % 4 == 0 and 16-byte aligned z, W.
// ---------------------------------------------------------------------------------------
// Sums a[0..15] over the 32 lanes with 16 shuffles instead of 80: each step a lane hands the half
// of its values that its partner keeps to the partner and adds the partner's to the half it
// keeps.  Returns the total of a[(lane >> 1) & 15] (lanes 2n and 2n + 1 both end with unit n).
__device__ __forceinline__ float warp_reduce16(float (&a)[16], int lane)
{
#pragma unroll
  for (int w = 8; w >= 1; w >>= 1)
  {
    const bool upper = (lane & (2 * w)) != 0;
#pragma unroll
    for (int i = 0; i < w; ++i)
    {
      const float send = upper ? a[i] : a[i + w];
      const float keep = upper ? a[i + w] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, 2 * w);
    }
  }
  return a[0] + __shfl_xor_sync(0xffffffffu, a[0], 1);
}

// A block stages the weights once (SMEM; zeros fill chunks of 512 columns and an even number of rows) or reads them through
// L1, and its warps take pairs of rows (RPW; single rows where the batch has few) in turn, a lane 16 of each 512 elements:
// the copies of the next two chunks are under way meanwhile.  Two units at a time: a unit alone is one chain of additions.
// SIMPLE: SimplePC layers, whose operand is f(z).
// What bounds it: instructions (950 a warp and row of 1024 with tanh, half of them the activation) on few SMs -- 20 beside
// a tensor launch take 80 us for 4096 rows, where the head must fit in --, one memory latency after another on many.  Alone,
// us, rows that each began with their loads and then read the weights through L2 / this: 4096 x 1024 -> 10 12.3 / 9.8, as
// SimplePC 15.4 / 13.9, 4096 x 2048 -> 16 32 / 19, 1024 x 512 -> 10 6.6 / 5.1, 256 x 256 -> 10 6.7 / 4.1.
constexpr int kHeadRing = 2;
template <int RPW>
constexpr int kHeadRingFloats = (NTHREADS / 32) * kHeadRing * RPW * 512;
template <int RPW, bool SIMPLE, bool SMEM>
__global__ void __launch_bounds__(NTHREADS, 2)
    narrow_forward_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers, int batch,
                          int flags, double* energy)
{
  const int li = first + blockIdx.z;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0)
    return;
  extern __shared__ __align__(16) float head_smem[];
  const int N = L.next_size, K = L.size, KP = (K + 511) & ~511;
  constexpr bool simple = SIMPLE;
  const dpc_layer* Lup = (li + 1 < n_layers) ? &layers[li + 1] : nullptr;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr int WARPS = NTHREADS / 32, CH = 4; // a chunk: four 16-byte pieces a lane
  const int chunks = KP / 512, stride = gridDim.x * WARPS * RPW;
  float* head_w = head_smem + kHeadRingFloats<RPW>;
  if (SMEM)
    for (int i = threadIdx.x; i < ((N + 1) & ~1) * (KP / 4); i += NTHREADS)
    {
      const int j = i / (KP / 4), k = 4 * (i - j * (KP / 4));
      const bool in = j < N && k < K;
      cp_async16(&head_w[4 * i], in ? L.W + (size_t)j * K + k : L.W, in);
    }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // a lane copies and reads its own pieces: no barrier
  float* ring = head_smem + (warp * kHeadRing * RPW) * 512 + lane * 4;
  int slot = 0, fm = (blockIdx.x * WARPS + warp) * RPW, fc = 0; // the chunk to copy next
  auto fetch = [&](int to)
  {
    if (fm < batch)
    {
#pragma unroll
      for (int r = 0; r < RPW; ++r)
#pragma unroll
        for (int i = 0; i < CH; ++i)
        {
          const int k = fc * 512 + lane * 4 + i * 128;
          const bool in = fm + r < batch && k < K;
          cp_async16(ring + (to * RPW + r) * 512 + i * 128, in ? L.z + (size_t)(fm + r) * K + k : L.z, in);
        }
      if (++fc == chunks)
        fc = 0, fm += stride;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int m0 = fm;
#pragma unroll
  for (int q = 0; q < kHeadRing; ++q)
    fetch(q);
  if (SMEM)
  {
    asm volatile("cp.async.wait_group %0;" ::"n"(kHeadRing) : "memory");
    __syncthreads();
  }
  float esum = 0.0f;
  const bool next_ce = Lup && (Lup->flags & DPC_LAYER_SOFTMAX_CE);
  const bool do_err = (flags & DPC_FWD_ERR_NEXT) && Lup && !next_ce;
  const bool do_fe =
      (flags & DPC_FWD_FE) && Lup && !simple && !(next_ce && (flags & DPC_FWD_ERR_NEXT));
  const bool do_copy = (flags & DPC_FWD_COPY_NEXT) && Lup;
  const bool do_ce = next_ce && (flags & DPC_FWD_ERR_NEXT) && (flags & DPC_FWD_CE);
  for (; m0 < batch; m0 += stride)
  {
    float acc[RPW][16];
#pragma unroll
    for (int r = 0; r < RPW; ++r)
#pragma unroll
      for (int j = 0; j < 16; ++j)
        acc[r][j] = 0.0f;
    for (int kc = 0; kc < K; kc += 512)
    {
      asm volatile("cp.async.wait_group %0;" ::"n"(kHeadRing - 1) : "memory");
      float4 zv[RPW][CH];
#pragma unroll
      for (int r = 0; r < RPW; ++r)
#pragma unroll
        for (int i = 0; i < CH; ++i)
          zv[r][i] = *reinterpret_cast<const float4*>(ring + (slot * RPW + r) * 512 + i * 128);
      __syncwarp();
      fetch(slot);
      slot = slot + 1 == kHeadRing ? 0 : slot + 1;
      if (simple)
      {
        // the operand is f(z), kept for the weight update (src/layers/SimplePCLayer.cpp:146-150)
#pragma unroll
        for (int r = 0; r < RPW; ++r)
#pragma unroll
          for (int i = 0; i < CH; i += 2)
          {
            const float in[8] = {zv[r][i].x,     zv[r][i].y,     zv[r][i].z,     zv[r][i].w,
                                 zv[r][i + 1].x, zv[r][i + 1].y, zv[r][i + 1].z, zv[r][i + 1].w};
            float f[8], d[8];
            act_many<false>(L.act, in, f, d);
#pragma unroll
            for (int q = 0; q < 2; ++q)
            {
              const int k = kc + lane * 4 + (i + q) * 128;
              const bool in_range = m0 + r < batch && k < K;
              zv[r][i + q] = in_range ? make_float4(f[4 * q], f[4 * q + 1], f[4 * q + 2], f[4 * q + 3])
                                      : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
              if (in_range)
                *reinterpret_cast<float4*>(L.zF + (size_t)(m0 + r) * K + k) = zv[r][i + q];
            }
          }
      }
#pragma unroll
      for (int j = 0; j < 16; j += 2)
      {
        if (j < N)
        {
#pragma unroll
          for (int i = 0; i < CH; ++i)
          {
            const int k = kc + lane * 4 + i * 128;
            float4 wv[2];
#pragma unroll
            for (int h = 0; h < 2; ++h)
              if (SMEM)
                wv[h] = *reinterpret_cast<const float4*>(&head_w[(j + h) * KP + k]);
              else
                wv[h] = j + h < N && k < K ? __ldg(reinterpret_cast<const float4*>(L.W + (size_t)(j + h) * K + k))
                                           : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int h = 0; h < 2; ++h)
#pragma unroll
              for (int r = 0; r < RPW; ++r)
              {
                acc[r][j + h] = fmaf(zv[r][i].x, wv[h].x, acc[r][j + h]);
                acc[r][j + h] = fmaf(zv[r][i].y, wv[h].y, acc[r][j + h]);
                acc[r][j + h] = fmaf(zv[r][i].z, wv[h].z, acc[r][j + h]);
                acc[r][j + h] = fmaf(zv[r][i].w, wv[h].w, acc[r][j + h]);
              }
          }
        }
      }
    }
#pragma unroll
    for (int r = 0; r < RPW; ++r)
    {
      // lanes 2n and 2n+1 end with the sum of output unit n; the even one finishes it
      const float mine = warp_reduce16(acc[r], lane);
      const int m = m0 + r, n = lane >> 1;
      float out_pre = 0.0f, out_mu = 0.0f;
      if (m < batch && !(lane & 1) && n < N)
      {
        const size_t o = (size_t)m * N + n;
        const float pre = L.a * mine + L.b[n];
        float mu, d = 1.0f;
        if (simple)
          mu = pre;
        else if (do_fe)
          act_both(L.act, pre, mu, d);
        else
          mu = act_fwd(L.act, pre);
        if (!simple && (L.flags & DPC_LAYER_RESIDUAL))
          mu += L.z[o];
        out_pre = pre, out_mu = mu;
        if (!(flags & DPC_FWD_TRANSIENT))
        {
          const bool no_mu = do_copy && (flags & DPC_FWD_NO_MU);
          if (L.preact && !(no_mu && (flags & DPC_FWD_NO_PREACT)))
            L.preact[o] = pre;
          if (!no_mu)
            L.mu[o] = mu;
        }
        if (do_copy)
          Lup->z[o] = mu;
        float e = 0.0f;
        if (do_err)
        {
          e = (do_copy ? mu : Lup->z[o]) - mu;
          Lup->e[o] = e;
          esum += e * e;
        }
        else if (do_fe)
          e = Lup->e[o];
        if (do_fe)
          L.fe[o] = e * d;
      }
      if (do_ce)
      {
        // Softmax cross-entropy error of the layer above (softmax_ce_kernel and feedback_error_kernel in
        // their order of operations): unit j moves to lane j.
        const float logit = __shfl_sync(0xffffffffu, out_mu, 2 * lane & 31);
        const float pre = __shfl_sync(0xffffffffu, out_pre, 2 * lane & 31);
        const bool in = lane < N;
        float mx = in ? logit : -INFINITY;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        float s = in ? expf(logit - mx) : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          s += __shfl_xor_sync(0xffffffffu, s, o);
        if (in && m < batch)
        {
          const size_t o = (size_t)m * N + lane;
          const float p = expf(logit - mx) / s;
          const float z = do_copy ? logit : Lup->z[o];
          esum -= 2.0f * z * logf(p + 1e-8f); // (halved with the Gaussian energies)
          const float e = z - p;
          Lup->e[o] = e;
          if ((flags & DPC_FWD_FE) && !simple)
            L.fe[o] = e * act_deriv(L.act, pre);
        }
      }
    }
  }
  if (flags & DPC_FWD_ENERGY)
    block_energy_add(do_err || do_ce ? esum : 0.0f, energy);
}

// ---------------------------------------------------------------------------------------
// Elementwise / skinny kernels (grouped over layers with blockIdx.y = layer in range).
// ---------------------------------------------------------------------------------------

// The forward epilogue for a layer whose prediction is cached (clamped input layer):
// no GEMM, preact/mu are read from memory.
__global__ void cached_forward_kernel(const dpc_layer* __restrict__ layers, int first,
                                      int n_layers, int batch, int flags, double* energy)
{
  const int li = first + blockIdx.y;
  const dpc_layer L = layers[li];
  const dpc_layer* Lup = (li + 1 < n_layers) ? &layers[li + 1] : nullptr;
  float esum = 0.0f;
  if (L.next_size > 0 && Lup)
  {
    const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
    const bool next_ce = (Lup->flags & DPC_LAYER_SOFTMAX_CE) != 0;
    const bool do_err = (flags & DPC_FWD_ERR_NEXT) && !next_ce;
    const bool do_fe = (flags & DPC_FWD_FE) && !simple && !(next_ce && (flags & DPC_FWD_ERR_NEXT));
    const bool do_copy = (flags & DPC_FWD_COPY_NEXT) != 0;
    const size_t total = (size_t)batch * L.next_size;
    // the pass of a settling step: errors (and feedback errors), 16 bytes at a time
    if (do_err && !do_copy && total % 4 == 0 && aligned16(L.mu) && aligned16(Lup->z) && aligned16(Lup->e) &&
        (!do_fe || (aligned16(L.fe) && aligned16(L.preact))))
    {
      const size_t n4 = total / 4;
      for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n4;
           i += (size_t)gridDim.x * blockDim.x)
      {
        const float4 mu = reinterpret_cast<const float4*>(L.mu)[i];
        const float4 z = reinterpret_cast<const float4*>(Lup->z)[i];
        const float4 e = make_float4(z.x - mu.x, z.y - mu.y, z.z - mu.z, z.w - mu.w);
        reinterpret_cast<float4*>(Lup->e)[i] = e;
        esum += e.x * e.x, esum += e.y * e.y, esum += e.z * e.z, esum += e.w * e.w;
        if (do_fe)
        {
          const float4 p = reinterpret_cast<const float4*>(L.preact)[i];
          reinterpret_cast<float4*>(L.fe)[i] =
              make_float4(e.x * act_deriv(L.act, p.x), e.y * act_deriv(L.act, p.y), e.z * act_deriv(L.act, p.z),
                          e.w * act_deriv(L.act, p.w));
        }
      }
    }
    else
      for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
           o += (size_t)gridDim.x * blockDim.x)
      {
        const float mu = L.mu[o];
        if (do_copy)
          Lup->z[o] = mu;
        float e = 0.0f;
        if (do_err)
        {
          e = (do_copy ? mu : Lup->z[o]) - mu;
          Lup->e[o] = e;
          esum += e * e;
        }
        else if (do_fe)
          e = Lup->e[o];
        if (do_fe)
          L.fe[o] = e * act_deriv(L.act, L.preact[o]);
      }
  }
  if (flags & DPC_FWD_ENERGY)
    block_energy_add(esum, energy);
}

// e = z - mu_below (+ energy), src/backend/CPUBackend.cpp:602-629.
__global__ void error_kernel(const dpc_layer* __restrict__ layers, int li, int batch,
                             int with_energy, double* energy)
{
  const dpc_layer L = layers[li];
  const dpc_layer Lb = layers[li - 1];
  const size_t total = (size_t)batch * L.size;
  float esum = 0.0f;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
  {
    const float e = L.z[o] - Lb.mu[o];
    L.e[o] = e;
    esum += e * e;
  }
  if (with_energy)
    block_energy_add(esum, energy);
}

// Softmax cross-entropy error, one warp per batch row:
// e = z - softmax(mu_below), E = -sum z*log(p + 1e-8)   (CPUBackend.cpp:658-695).
__global__ void softmax_ce_kernel(const dpc_layer* __restrict__ layers, int li, int batch,
                                  int with_energy, double* energy)
{
  const dpc_layer L = layers[li];
  const float* mu = layers[li - 1].mu;
  const int n = L.size;
  const int warps = blockDim.x >> 5, lane = threadIdx.x & 31;
  float row_energy = 0.0f;
  for (int r = blockIdx.x * warps + (threadIdx.x >> 5); r < batch; r += gridDim.x * warps)
  {
    const float* mrow = mu + (size_t)r * n;
    const float* zrow = L.z + (size_t)r * n;
    float* erow = L.e + (size_t)r * n;
    float mx = -INFINITY;
    for (int j = lane; j < n; j += 32)
      mx = fmaxf(mx, mrow[j]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float s = 0.0f;
    for (int j = lane; j < n; j += 32)
      s += expf(mrow[j] - mx);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      s += __shfl_xor_sync(0xffffffffu, s, o);
    for (int j = lane; j < n; j += 32)
    {
      const float p = expf(mrow[j] - mx) / s;
      const float z = zrow[j];
      row_energy -= z * logf(p + 1e-8f);
      erow[j] = z - p;
    }
  }
  if (with_energy)
  {
    // block_energy_add halves its input (Gaussian energy); cross-entropy is not halved.
    block_energy_add(2.0f * row_energy, energy);
  }
}

// fe[l] = e[l+1] * f'(preact[l])
__global__ void feedback_error_kernel(const dpc_layer* __restrict__ layers, int first,
                                      int n_layers, int batch)
{
  const int li = first + blockIdx.y;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0 || (L.flags & DPC_LAYER_INPUT_ACT))
    return;
  const float* e_up = layers[li + 1].e;
  const size_t total = (size_t)batch * L.next_size;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    L.fe[o] = e_up[o] * act_deriv(L.act, L.preact[o]);
}

// ePC: fe[l] = src * f'(preact[l]) with an explicit source (terminal error or adj[l+1]).
__global__ void epc_source_kernel(const dpc_layer* __restrict__ layers, int li, int batch,
                                  const float* __restrict__ src)
{
  const dpc_layer L = layers[li];
  const size_t total = (size_t)batch * L.next_size;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    L.fe[o] = src[o] * act_deriv(L.act, L.preact[o]);
}

// ePC: z[l] = mu[l-1] + e[l]   (src/layers/FullPCLayer.cpp:574-582)
__global__ void epc_reconstruct_kernel(const dpc_layer* __restrict__ layers, int li, int batch)
{
  const dpc_layer L = layers[li];
  const float* mu = layers[li - 1].mu;
  const size_t total = (size_t)batch * L.size;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    L.z[o] = mu[o] + L.e[o];
}

// z -= ir*e for layers of the range that have no weights or no upper neighbour.
__global__ void relax_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers,
                             int batch, int only_weightless)
{
  const int li = first + blockIdx.y;
  const dpc_layer L = layers[li];
  if (only_weightless && L.next_size > 0 && li + 1 < n_layers)
    return;
  const size_t total = (size_t)batch * L.size;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    L.z[o] -= L.ir * L.e[o];
}

// DFA projection: fe[l] = (e_T · Psi[l+1]^T) * f'(preact[l])   (K = terminal_size).
// One thread per output unit j with its Psi row in registers; a block covers rows_per_block (at most
// DFA_ROWS) batch rows whose terminal errors sit in shared memory, so preact/fe stream through
// coalesced.
constexpr int DFA_ROWS = 32;
__global__ void dfa_proj_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers,
                                int batch, const float* __restrict__ eT, int from_output,
                                int rows_per_block)
{
  const int li = first + blockIdx.z;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  const dpc_layer Lup = layers[li + 1];
  if (L.next_size <= 0 || Lup.Psi == nullptr)
    return;
  const int TS = L.terminal_size, n = L.next_size;
  const int b0 = blockIdx.y * rows_per_block;
  if (b0 >= batch || (int)(blockIdx.x * blockDim.x) >= n)
    return;
  __shared__ __align__(16) float es[DFA_ROWS][16];
  for (int kc = 0; kc < TS; kc += 16)
  {
    const int kn = min(16, TS - kc);
    __syncthreads();
    for (int idx = threadIdx.x; idx < rows_per_block * 16; idx += blockDim.x)
    {
      const int r = idx >> 4, k = idx & 15;
      es[r][k] = (b0 + r < batch && k < kn) ? eT[(size_t)(b0 + r) * TS + kc + k] : 0.0f;
    }
    __syncthreads();
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j < n)
    {
      float psi[16];
      const float* pr = Lup.Psi + (size_t)j * Lup.psi_stride + kc;
#pragma unroll
      for (int k = 0; k < 16; ++k)
        psi[k] = k < kn ? pr[k] : 0.0f;
      const bool last = kc + 16 >= TS;
#pragma unroll 4
      for (int r = 0; r < rows_per_block; ++r)
      {
        if (b0 + r >= batch)
          break;
        float acc = 0.0f;
#pragma unroll
        for (int k4 = 0; k4 < 16; k4 += 4)
        {
          const float4 e4 = *reinterpret_cast<const float4*>(&es[r][k4]);
          acc = fmaf(e4.x, psi[k4], acc);
          acc = fmaf(e4.y, psi[k4 + 1], acc);
          acc = fmaf(e4.z, psi[k4 + 2], acc);
          acc = fmaf(e4.w, psi[k4 + 3], acc);
        }
        const size_t o = (size_t)(b0 + r) * n + j;
        if (kc > 0)
          acc += L.fe[o];
        if (last)
          acc *= (from_output && act_has_output_deriv(L.act))
                     ? act_deriv_from_output(L.act, Lup.z[o])
                     : act_deriv(L.act, L.preact[o]);
        L.fe[o] = acc;
      }
    }
  }
}

// The tensor-core path's bf16 "hi"/"mid" operand copies of the feedback errors of the layers
// [run_first, run_first + run_count): layer l has its hi plane at fe + 2 (l - run_first) * elems
// and its mid plane elems further on.  fe == NULL: no copies.  only != 0: the fp32 tensor of
// those layers is not kept at all (nothing reads it), the copies are the feedback error.
struct FePlanes
{
  __nv_bfloat16* fe;
  int run_first, run_count, only;
  long long elems;
};
__device__ __forceinline__ __nv_bfloat16* fe_plane_of(const FePlanes& P, int li)
{
  return (P.fe && li >= P.run_first && li < P.run_first + P.run_count)
             ? P.fe + 2 * (long long)(li - P.run_first) * P.elems
             : nullptr;
}

// Rows per block of the aligned kernel: its per-thread rows of Psi are strided 4-byte loads that
// cost as much L2 traffic as 32 rows of useful data, so a block amortises them over up to 128 rows
// (the host picks fewer when that would leave SMs without a block).
constexpr int DFA4_ROWS = 128;
// The same projection, four output units per thread with 128-bit accesses, for the common aligned case: next_size a multiple of 4, terminal_size <= 4*TS4, 16-byte aligned rows.
template <int TS4>
__global__ void __launch_bounds__(64)
    dfa_proj4_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers, int batch,
                     const float* __restrict__ eT, int from_output, int rows_per_block,
                     FePlanes planes)
{
  const int li = first + blockIdx.z;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  const dpc_layer Lup = layers[li + 1];
  if (L.next_size <= 0 || Lup.Psi == nullptr)
    return;
  const int TS = L.terminal_size, n = L.next_size;
  const int b0 = blockIdx.y * rows_per_block; // rows_per_block <= DFA4_ROWS
  const int j = (blockIdx.x * 64 + threadIdx.x) * 4;
  if (b0 >= batch || (int)(blockIdx.x * 256) >= n)
    return;
  __shared__ __align__(16) float es[DFA4_ROWS][TS4 * 4];
  for (int idx = threadIdx.x; idx < rows_per_block * TS4 * 4; idx += 64)
  {
    const int r = idx / (TS4 * 4), k = idx - r * (TS4 * 4);
    es[r][k] = (b0 + r < batch && k < TS) ? eT[(size_t)(b0 + r) * TS + k] : 0.0f;
  }
  __syncthreads();
  if (j >= n)
    return;
  float psi[4][TS4 * 4];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < TS4 * 4; ++k)
      psi[c][k] = k < TS ? Lup.Psi[(size_t)(j + c) * Lup.psi_stride + k] : 0.0f;
  const bool out_d = from_output && act_has_output_deriv(L.act);
  const float* src = out_d ? Lup.z : L.preact;
  const int rows = min(rows_per_block, batch - b0);
  __nv_bfloat16* hi = fe_plane_of(planes, li);
  const bool keep_fp32 = !(hi && planes.only);
#pragma unroll 8
  for (int r = 0; r < rows; ++r)
  {
    const size_t o = (size_t)(b0 + r) * n + j;
    const float4 s4 = *reinterpret_cast<const float4*>(src + o);
    float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k4 = 0; k4 < TS4; ++k4)
    {
      const float4 e4 = *reinterpret_cast<const float4*>(&es[r][k4 * 4]);
#pragma unroll
      for (int c = 0; c < 4; ++c)
      {
        acc[c] = fmaf(e4.x, psi[c][k4 * 4], acc[c]);
        acc[c] = fmaf(e4.y, psi[c][k4 * 4 + 1], acc[c]);
        acc[c] = fmaf(e4.z, psi[c][k4 * 4 + 2], acc[c]);
        acc[c] = fmaf(e4.w, psi[c][k4 * 4 + 3], acc[c]);
      }
    }
    const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
    float out[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
      out[c] = acc[c] * (out_d ? act_deriv_from_output(L.act, sv[c]) : act_deriv(L.act, sv[c]));
    if (keep_fp32)
      *reinterpret_cast<float4*>(L.fe + o) = make_float4(out[0], out[1], out[2], out[3]);
    if (hi)
    {
      const __nv_bfloat162 h0 = __floats2bfloat162_rn(out[0], out[1]);
      const __nv_bfloat162 h1 = __floats2bfloat162_rn(out[2], out[3]);
      const __nv_bfloat162 m0 =
          __floats2bfloat162_rn(out[0] - __low2float(h0), out[1] - __high2float(h0));
      const __nv_bfloat162 m1 =
          __floats2bfloat162_rn(out[2] - __low2float(h1), out[3] - __high2float(h1));
      uint2 hv, mv;
      hv.x = *reinterpret_cast<const uint32_t*>(&h0), hv.y = *reinterpret_cast<const uint32_t*>(&h1);
      mv.x = *reinterpret_cast<const uint32_t*>(&m0), mv.y = *reinterpret_cast<const uint32_t*>(&m1);
      *reinterpret_cast<uint2*>(hi + o) = hv;
      *reinterpret_cast<uint2*>(hi + planes.elems + o) = mv;
    }
  }
}

// The aligned projection for wide layers (next_size a multiple of 128) when there are enough
// rows to fill the GPU with blocks of 128 columns x at least 128 rows: the 128 rows of Psi a
// block needs come in through shared memory with coalesced loads ONCE per block (the kernel above
// re-reads them with strided loads for every 128 batch rows), lane l of every warp owns columns
// 4l..4l+3, warp w the batch rows w, w+8, ...: every access of a warp is one whole row segment.
template <int TS4>
__global__ void __launch_bounds__(256)
    dfa_proj128_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers, int batch,
                       const float* __restrict__ eT, int from_output, int rows_per_block,
                       FePlanes planes)
{
  const int li = first + blockIdx.y;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  const dpc_layer Lup = layers[li + 1];
  if (L.next_size <= 0 || Lup.Psi == nullptr)
    return;
  const int TS = L.terminal_size, n = L.next_size;
  const int j0 = blockIdx.x * 128;
  if (j0 >= n)
    return;
  constexpr int KC = TS4 * 4, ROWS = 128;
  __shared__ __align__(16) float es[ROWS][KC];
  __shared__ float ps[128][KC + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int idx = threadIdx.x; idx < 128 * KC; idx += 256)
  {
    const int r = idx / KC, k = idx - r * KC;
    ps[r][k] = k < TS ? Lup.Psi[(size_t)(j0 + r) * Lup.psi_stride + k] : 0.0f;
  }
  __syncthreads();
  float psi[4][KC];
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < KC; ++k)
      psi[c][k] = ps[4 * lane + c][k];
  const bool out_d = from_output && act_has_output_deriv(L.act);
  const float* src = out_d ? Lup.z : L.preact;
  __nv_bfloat16* hi = fe_plane_of(planes, li);
  const bool keep_fp32 = !(hi && planes.only);
  const int j = j0 + 4 * lane;
  const int b_begin = blockIdx.z * rows_per_block, b_end = min(batch, b_begin + rows_per_block);
  for (int b0 = b_begin; b0 < b_end; b0 += ROWS)
  {
    __syncthreads();
    for (int idx = threadIdx.x; idx < ROWS * KC; idx += 256)
    {
      const int r = idx / KC, k = idx - r * KC;
      es[r][k] = (b0 + r < b_end && k < TS) ? eT[(size_t)(b0 + r) * TS + k] : 0.0f;
    }
    __syncthreads();
    const int rows = min(ROWS, b_end - b0);
#pragma unroll 4
    for (int r = warp; r < rows; r += 8)
    {
      const size_t o = (size_t)(b0 + r) * n + j;
      const float4 s4 = *reinterpret_cast<const float4*>(src + o);
      float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int k4 = 0; k4 < TS4; ++k4)
      {
        const float4 e4 = *reinterpret_cast<const float4*>(&es[r][k4 * 4]);
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
          acc[c] = fmaf(e4.x, psi[c][k4 * 4], acc[c]);
          acc[c] = fmaf(e4.y, psi[c][k4 * 4 + 1], acc[c]);
          acc[c] = fmaf(e4.z, psi[c][k4 * 4 + 2], acc[c]);
          acc[c] = fmaf(e4.w, psi[c][k4 * 4 + 3], acc[c]);
        }
      }
      const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
      float out[4];
#pragma unroll
      for (int c = 0; c < 4; ++c)
        out[c] = acc[c] * (out_d ? act_deriv_from_output(L.act, sv[c]) : act_deriv(L.act, sv[c]));
      if (keep_fp32)
        *reinterpret_cast<float4*>(L.fe + o) = make_float4(out[0], out[1], out[2], out[3]);
      if (hi)
      {
        const __nv_bfloat162 h0 = __floats2bfloat162_rn(out[0], out[1]);
        const __nv_bfloat162 h1 = __floats2bfloat162_rn(out[2], out[3]);
        const __nv_bfloat162 m0 =
            __floats2bfloat162_rn(out[0] - __low2float(h0), out[1] - __high2float(h0));
        const __nv_bfloat162 m1 =
            __floats2bfloat162_rn(out[2] - __low2float(h1), out[3] - __high2float(h1));
        uint2 hv, mv;
        hv.x = *reinterpret_cast<const uint32_t*>(&h0), hv.y = *reinterpret_cast<const uint32_t*>(&h1);
        mv.x = *reinterpret_cast<const uint32_t*>(&m0), mv.y = *reinterpret_cast<const uint32_t*>(&m1);
        *reinterpret_cast<uint2*>(hi + o) = hv;
        *reinterpret_cast<uint2*>(hi + planes.elems + o) = mv;
      }
    }
  }
}

// Adam step counters: t += 1 once per UpdateWeights (src/backend/cuda/CUDABackendOptimizer.cu:20-31).
__global__ void bump_counters_kernel(const dpc_layer* __restrict__ layers, int first, int count,
                                     int n_layers)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count)
    return;
  const int li = first + i;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0 || li + 1 >= n_layers)
    return;
  if (L.opt != DPC_OPT_SGD && L.t)
    *L.t += 1;
  if (!(L.flags & DPC_LAYER_INPUT_ACT) && L.opt_psi != DPC_OPT_SGD && L.t_Psi)
    *L.t_Psi += 1;
}

// Rates and decays of a layer's updates, from the raw sums over `batch` rows.
// dfa: the direct-feedback update, decay_w: which decays the weights
__device__ __forceinline__ Sgd weight_sgd(const dpc_layer& L, int batch, bool dfa, bool decay_w)
{
  const float Bf = (float)batch;
  const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
  const bool decays = dfa ? decay_w && L.lmbda > 0.0f && L.fl != 0.0f : L.lmbda > 0.0f;
  return Sgd{dfa ? L.fl * L.a / Bf : simple ? L.lr / Bf : L.a * L.lr / Bf, decays ? 1.0f - L.lmbda : 1.0f};
}
__device__ __forceinline__ Sgd bias_sgd(const dpc_layer& L, int batch)
{
  return Sgd{L.lr / (float)batch, 1.0f};
}
__device__ __forceinline__ float psi_rate(const dpc_layer& L)
{
  return (L.flags & DPC_LAYER_FULLPC_PSI) ? L.fl * L.a : L.fl;
}
__device__ __forceinline__ Sgd psi_sgd(const dpc_layer& L, int batch)
{
  const bool decays = !(L.flags & DPC_LAYER_FULLPC_PSI) && L.psi_decay > 0.0f;
  return Sgd{psi_rate(L) / (float)batch, decays ? 1.0f - L.psi_decay : 1.0f};
}
// (of adam_update: AdamW's decay, or below zero)
__device__ __forceinline__ float weight_wd(const dpc_layer& L)
{
  return L.opt == DPC_OPT_ADAMW ? L.lr * L.lmbda : -1.0f;
}
__device__ __forceinline__ float psi_wd(const dpc_layer& L)
{
  const bool own = !(L.flags & DPC_LAYER_FULLPC_PSI) && L.psi_decay >= 0.0f;
  return L.opt_psi == DPC_OPT_ADAMW ? psi_rate(L) * (own ? L.psi_decay : L.lmbda) : -1.0f;
}

// b (+)= rate * s for one output unit (or s into the staging buffer): what follows the column sum.
__device__ __forceinline__ void bias_apply(const dpc_layer& L, int j, float s, int batch, int grad_only)
{
  if (grad_only)
    L.g_b[j] = s;
  else if (L.opt == DPC_OPT_SGD)
    L.b[j] = bias_sgd(L, batch)(L.b[j], s);
  else
  {
    float m = L.m_b[j], v = L.v_b[j];
    L.b[j] = adam_update(L.b[j], -s, m, v, adam_step_size(L.lr, *L.t), -1.0f);
    L.m_b[j] = m;
    L.v_b[j] = v;
  }
}

// Bias update from the column sums of the local gradient: a lane per output unit,
// summing the batch in row order like CPUBackend::SumRows (CPUBackend.cpp:243-248).
// Layers whose feedback error exists only as bf16 planes (see FePlanes) are summed by whole
// blocks instead: 32 row groups x 8 threads of 8 columns each (16-byte loads of both planes,
// hi + mid = fe to 2^-17), then a fixed-order reduction over the row groups in shared memory.
constexpr int kBiasBlockRows = 256;
__global__ void bias_update_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers,
                                   int batch, int grad_only, FePlanes planes)
{
  const int li = first + blockIdx.y;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0)
    return;
  const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
  const float* g = simple ? layers[li + 1].e : L.fe;
  const int n = L.next_size;
  const __nv_bfloat16* hi = (!simple && planes.only) ? fe_plane_of(planes, li) : nullptr;
  // Summed by whole blocks: the plane-only layers, and fp32 gradients of large batches (the
  // one-thread-per-column loop below keeps the reference's row order for the small cases).
  const bool wide = n % 64 == 0 && blockDim.x == 256 &&
                    (hi || (batch >= kBiasBlockRows && ((uintptr_t)g % 16) == 0));
  const uint32_t R = rows_cluster_size(), rank = rows_cluster_rank();
  if (wide)
  {
    __shared__ float part[32][65];
    __shared__ float mine[64];
    const int rg = threadIdx.x >> 3, c8 = (threadIdx.x & 7) * 8;
    for (int j0 = blockIdx.x * 64; j0 < n; j0 += gridDim.x * 64)
    {
      float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
      if (hi)
      {
        for (int b = rg + 32 * (int)rank; b < batch; b += 32 * (int)R)
        {
          const size_t o = (size_t)b * n + j0 + c8;
          const uint4 h = *reinterpret_cast<const uint4*>(hi + o);
          const uint4 m = *reinterpret_cast<const uint4*>(hi + planes.elems + o);
          const uint32_t hw[4] = {h.x, h.y, h.z, h.w}, mw[4] = {m.x, m.y, m.z, m.w};
#pragma unroll
          for (int q = 0; q < 4; ++q)
          {
            // a bf16 is the upper half of the fp32 with the same value
            acc[2 * q] += __uint_as_float(hw[q] << 16) + __uint_as_float(mw[q] << 16);
            acc[2 * q + 1] += __uint_as_float(hw[q] & 0xffff0000u) + __uint_as_float(mw[q] & 0xffff0000u);
          }
        }
      }
      else
      {
#pragma unroll 4
        for (int b = rg + 32 * (int)rank; b < batch; b += 32 * (int)R)
        {
          const size_t o = (size_t)b * n + j0 + c8;
          const float4 x = *reinterpret_cast<const float4*>(g + o);
          const float4 y = *reinterpret_cast<const float4*>(g + o + 4);
          acc[0] += x.x, acc[1] += x.y, acc[2] += x.z, acc[3] += x.w;
          acc[4] += y.x, acc[5] += y.y, acc[6] += y.z, acc[7] += y.w;
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 8; ++q)
        part[rg][c8 + q] = acc[q];
      __syncthreads();
      float s = 0.0f;
      if (threadIdx.x < 64)
      {
        for (int r = 0; r < 32; ++r)
          s += part[r][threadIdx.x];
        if (R > 1 && rank != 0)
          mine[threadIdx.x] = s;
      }
      if (R > 1)
      {
        rows_cluster_sync();
        if (rank == 0 && threadIdx.x < 64)
          for (uint32_t r = 1; r < R; ++r)
            s += rows_cluster_load(&mine[threadIdx.x], r);
        rows_cluster_sync(); // `mine` of the other CTAs may be rewritten (or go away) only now
      }
      if (threadIdx.x < 64 && rank == 0)
        bias_apply(L, j0 + threadIdx.x, s, batch, grad_only);
    }
    return;
  }
  if (rank != 0)
    return; // (a row-split launch over a layer that takes the column sums: one CTA does them)
  // Column sums in row order (the reference's), 32 columns at a time: seven warps copy groups of rows into shared memory,
  // three buffers ahead, the other one adds them up, a chain of dependent additions and nothing else.  It bounds the
  // kernel, with the barrier of a group: 784-(91x4)-100 at batch 3584 281 -> 45 us a launch, 3072-(37x3)-16 at batch 768
  // 204 -> 178 a step (76 us where all warps copied and seven then waited for the sums).
  constexpr int STAGES = 4, ROWS = 64, AT_ONCE = 16;
  __shared__ __align__(16) float stage[STAGES][ROWS][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int j0 = blockIdx.x * 32; j0 < n; j0 += gridDim.x * 32)
  {
    const int j = j0 + lane;
    auto copy = [&](int b0)
    {
      float* to = &stage[b0 / ROWS % STAGES][0][lane];
#pragma unroll
      for (int r = warp - 1; r < ROWS; r += 7)
        if (b0 + r < batch && j < n)
          cp_async4(to + r * 32, g + (size_t)(b0 + r) * n + j, true);
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float s = 0.0f;
    if (warp > 0)
#pragma unroll 1
      for (int q = 0; q < STAGES - 1; ++q)
        copy(q * ROWS);
#pragma unroll 1
    for (int b0 = -ROWS; b0 < batch; b0 += ROWS)
    {
      if (warp > 0)
      {
        if (b0 >= 0)
          copy(b0 + (STAGES - 1) * ROWS);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory"); // the next group of rows
      }
      else if (b0 >= 0)
      {
        const int rows = min(ROWS, batch - b0);
        const float* p = &stage[b0 / ROWS % STAGES][0][lane];
        float v[2][AT_ONCE]; // (what is added next is read before these are)
        auto read = [&](float (&x)[AT_ONCE], int r)
        {
#pragma unroll
          for (int q = 0; q < AT_ONCE; ++q)
            x[q] = p[(r + q) * 32];
        };
        auto add = [&](const float (&x)[AT_ONCE], int count)
        {
#pragma unroll
          for (int q = 0; q < AT_ONCE; ++q)
            if (q < count)
              s += x[q];
        };
        read(v[0], 0);
#pragma unroll
        for (int r = 0; r < ROWS; r += 2 * AT_ONCE)
        {
          read(v[1], r + AT_ONCE);
          add(v[0], rows - r);
          if (r + 2 * AT_ONCE < ROWS)
            read(v[0], r + 2 * AT_ONCE);
          add(v[1], rows - r - AT_ONCE);
        }
      }
      __syncthreads();
    }
    if (warp == 0 && j < n)
      bias_apply(L, j, s, batch, grad_only);
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
  }
}

// `step`: adam_step_size of the layer (two powers and a root: once per thread, not per element)
__device__ __forceinline__ float psi_step(const dpc_layer& L, int grad_only)
{
  return grad_only || L.opt_psi == DPC_OPT_SGD ? 0.0f : adam_step_size(psi_rate(L), *L.t_Psi);
}
__device__ __forceinline__ void psi_apply(const dpc_layer& L, int row, int k, float sum, int batch,
                                          int grad_only, float step)
{
  const size_t o = (size_t)row * L.psi_stride + k;
  if (grad_only)
    L.g_Psi[o] = sum;
  else if (L.opt_psi == DPC_OPT_SGD)
    L.Psi[o] = psi_sgd(L, batch)(L.Psi[o], sum);
  else
  {
    float m = L.m_Psi[o], v = L.v_Psi[o];
    L.Psi[o] = adam_update(L.Psi[o], -sum, m, v, step, psi_wd(L));
    L.m_Psi[o] = m;
    L.v_Psi[o] = v;
  }
}

// sum over the batch of zin[b][col + c] * g[b][k] for c < 4, k < KC: the common core of the Psi
// update and of the weight update of a narrow layer.  A block owns 128 columns of zin, lane l of
// every warp the columns 4l..4l+3 (one 16-byte load per batch row: a warp reads a whole 512-byte row
// segment), warp w the batch rows w, w+8, ...; the rows of g (at most KC wide, ldg apart) of 128
// batch rows at a time sit in shared memory.  The eight warps' partial sums are added in a fixed
// tree order through shared memory, then the CTAs of a row-split cluster in rank order.  Returns
// true in the threads that end up with the sums (warp 0 of CTA 0 of the cluster).
// What bounds it: bytes in flight.  A lane copies its pieces of the warp's next eight rows ahead (it alone reads them: no
// barrier), also across groups of 128 rows, and the next group's rows of g are read before this one's products (four rows in
// registers, drained at every group, took 500 us for 512 layers of 1024 x 512 instead of 302, the reads take 161).
template <int KC>
constexpr int kOuterFloats = 2 * 128 * KC + 8 * 8 * 128; // rows of g, twice; eight rows a warp, then the partial sums
template <int KC>
__device__ __forceinline__ bool batch_outer4(const float* __restrict__ zin, int s, int col,
                                             const float* __restrict__ g, int ldg, int TS,
                                             int batch, float (&acc)[4][KC], float* smem)
{
  constexpr int ROWS = 128, D = 8, PER = ROWS * KC / 256;
  static_assert(4 * 4 * KC * 32 <= 8 * D * 128, "the partial sums fit where the rows were");
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float(*part)[4 * KC][32] = reinterpret_cast<float(*)[4 * KC][32]>(smem + 2 * ROWS * KC);
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < KC; ++k)
      acc[c][k] = 0.0f;
  const uint32_t R = rows_cluster_size(), rank = rows_cluster_rank();
  const int stride = (int)R * ROWS;
  float* ring = smem + 2 * ROWS * KC + warp * D * 128 + lane * 4;
  int fb = (int)rank * ROWS, fr = warp; // the row to copy next: group and row in it
  auto fetch = [&](int to)
  {
    if (fb + fr < batch)
    {
      cp_async16(ring + to * 128, zin + (size_t)(fb + fr) * s + col, true);
      fr += 8;
      if (fr >= ROWS)
        fb += stride, fr = warp;
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int q = 0; q < D; ++q)
    fetch(q);
  float next[PER];
  auto read_g = [&](int b0)
  {
#pragma unroll
    for (int q = 0; q < PER; ++q)
    {
      const int idx = threadIdx.x + 256 * q, r = idx / KC, k = idx - r * KC;
      next[q] = (b0 + r < batch && k < TS) ? g[(size_t)(b0 + r) * ldg + k] : 0.0f;
    }
  };
  read_g((int)rank * ROWS);
  int slot = 0;
  float* es = smem;
  for (int b0 = (int)rank * ROWS; b0 < batch; b0 += stride)
  {
#pragma unroll
    for (int q = 0; q < PER; ++q)
      es[threadIdx.x + 256 * q] = next[q];
    __syncthreads();
    read_g(b0 + stride);
    const int rows = min(ROWS, batch - b0);
#pragma unroll 2
    for (int r = warp; r < rows; r += 8)
    {
      asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
      const float4 z4 = *reinterpret_cast<const float4*>(ring + slot * 128);
      __syncwarp();
      fetch(slot);
      slot = (slot + 1) & (D - 1);
      const float zv[4] = {z4.x, z4.y, z4.z, z4.w};
#pragma unroll
      for (int k4 = 0; k4 < KC; k4 += 4)
      {
        const float4 e4 = *reinterpret_cast<const float4*>(es + r * KC + k4);
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
          acc[c][k4] = fmaf(zv[c], e4.x, acc[c][k4]);
          acc[c][k4 + 1] = fmaf(zv[c], e4.y, acc[c][k4 + 1]);
          acc[c][k4 + 2] = fmaf(zv[c], e4.z, acc[c][k4 + 2]);
          acc[c][k4 + 3] = fmaf(zv[c], e4.w, acc[c][k4 + 3]);
        }
      }
    }
    es = es == smem ? smem + ROWS * KC : smem; // (the barrier of the group in between guards it)
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // tree over the warps: (w, w+4), then (w, w+2), then (0, 1)
#pragma unroll
  for (int half = 4; half >= 1; half >>= 1)
  {
    __syncthreads();
    if (warp >= half && warp < 2 * half)
    {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int k = 0; k < KC; ++k)
          part[warp - half][c * KC + k][lane] = acc[c][k];
    }
    __syncthreads();
    if (warp < half)
    {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int k = 0; k < KC; ++k)
          acc[c][k] += part[warp][c * KC + k][lane];
    }
  }
  if (R > 1)
  {
    // (part[0] was last read by this same warp 0 in the tree above)
    if (rank != 0 && warp == 0)
    {
#pragma unroll
      for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int k = 0; k < KC; ++k)
          part[0][c * KC + k][lane] = acc[c][k];
    }
    rows_cluster_sync();
    if (rank == 0 && warp == 0)
    {
      for (uint32_t r = 1; r < R; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c)
#pragma unroll
          for (int k = 0; k < KC; ++k)
            acc[c][k] += rows_cluster_load(&part[0][c * KC + k][lane], r);
    }
    rows_cluster_sync(); // nobody leaves while CTA 0 may still read its shared memory
  }
  return rank == 0 && warp == 0;
}

// The Psi update for the common aligned case (layer width a multiple of 128, at most KC terminal
// units, KC = 12 or 16): a block owns 128 rows of Psi (= 128 columns of z).
template <int KC>
__global__ void __launch_bounds__(256, 2)
    psi_update4_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers, int batch,
                       const float* __restrict__ eT, int grad_only)
{
  const int li = first + blockIdx.y;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0 || L.Psi == nullptr || (L.flags & DPC_LAYER_INPUT_ACT))
    return;
  const int TS = L.terminal_size, s = L.size;
  if ((int)blockIdx.x * 128 >= s)
    return;
  __shared__ __align__(16) float smem[kOuterFloats<KC>];
  const int col = blockIdx.x * 128 + (threadIdx.x & 31) * 4;
  float acc[4][KC];
  if (!batch_outer4<KC>(L.z, s, col, eT, TS, TS, batch, acc, smem))
    return;
  const float step = psi_step(L, grad_only);
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < KC; ++k)
      if (k < TS)
        psi_apply(L, col + c, k, acc[c][k], batch, grad_only, step);
}

// State update of a layer below a narrow one (at most KC <= 16 units above, own width a multiple of
// 128: the layer under a head, e.g. z[4096 x 1024] += ir (a fe[4096 x 10] W[10 x 1024] - e)).  The
// product has a K of 10: the tiled kernel spends its time on tile bookkeeping.  Here lane l of
// every warp keeps the weights of columns 4l..4l+3 in registers, a block owns 128 columns and
// `rows_per_block` batch rows, warp w the rows w, w+8, ...; the rows of the feedback error go
// through shared memory 128 at a time.  Same arithmetic per element as GemmEpilogue::state.
// PLAIN: no momentum, no residual term.  What bounds it: latency times bytes in flight, so eight rows a warp (PLAIN, else
// four) are under way as copies into shared memory (one row, because the next one's loads could not pass this one's
// stores, took 117 us of 4096 x 1024 on the 20 SMs beside a tensor launch, four in registers 71, this 65; SimplePC, which
// forms tanh' too, 105 with four in registers, 88).
template <bool PLAIN>
constexpr int kHeadStateRing = PLAIN ? 8 : 4; // rows a warp has under way
constexpr int kHeadStateSmem = 8 * 4 * 4 * 128 * 4;
template <int KC, bool PLAIN>
__global__ void __launch_bounds__(256, 2)
    narrow_state_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers, int batch,
                        int rows_per_block)
{
  const int li = first + blockIdx.z;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0)
    return;
  const dpc_layer* Lup = &layers[li + 1];
  const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
  const bool residual = (L.flags & DPC_LAYER_RESIDUAL) != 0;
  const int K = L.next_size, s = L.size;
  if ((int)blockIdx.x * 128 >= s)
    return;
  const float* g = simple ? Lup->e : L.fe;
  constexpr int ROWS = 128, D = kHeadStateRing<PLAIN>, PIECES = PLAIN ? 2 : 4;
  __shared__ __align__(16) float gs[ROWS][KC];
  extern __shared__ __align__(16) float state_ring[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int col = blockIdx.x * 128 + lane * 4;
  const int b_begin = blockIdx.y * rows_per_block;
  const int b_end = min(batch, b_begin + rows_per_block);
  // a lane copies and reads its own pieces of the warp's rows: no barrier
  float* ring = state_ring + warp * D * PIECES * 128 + lane * 4;
  int fr = b_begin + warp; // the row to copy next
  auto fetch = [&](int to)
  {
    if (fr < b_end)
    {
      const size_t o = (size_t)fr * s + col;
      float* d = ring + to * PIECES * 128;
      cp_async16(d, L.e + o, true);
      cp_async16(d + 128, L.z + o, true);
      if (!PLAIN && !simple && L.v)
        cp_async16(d + 256, L.v + o, true);
      if (!PLAIN && !simple && residual)
        cp_async16(d + 384, Lup->e + o, true);
    }
    fr += 8;
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
#pragma unroll
  for (int q = 0; q < D; ++q)
    fetch(q);
  float w[4][KC];
#pragma unroll
  for (int k = 0; k < KC; ++k)
  {
    float4 w4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (k < K)
      w4 = *reinterpret_cast<const float4*>(L.W + (size_t)k * s + col);
    w[0][k] = w4.x, w[1][k] = w4.y, w[2][k] = w4.z, w[3][k] = w4.w;
  }
  int slot = 0;
  for (int b0 = b_begin; b0 < b_end; b0 += ROWS)
  {
    __syncthreads();
    for (int idx = threadIdx.x; idx < ROWS * KC; idx += 256)
    {
      const int r = idx / KC, k = idx - r * KC;
      gs[r][k] = (b0 + r < b_end && k < K) ? g[(size_t)(b0 + r) * K + k] : 0.0f;
    }
    __syncthreads();
    const int rows = min(ROWS, b_end - b0);
    for (int r = warp; r < rows; r += 8)
    {
      asm volatile("cp.async.wait_group %0;" ::"n"(D - 1) : "memory");
      const float* piece = ring + slot * PIECES * 128;
      const float4 e4 = *reinterpret_cast<const float4*>(piece);
      const float4 z4 = *reinterpret_cast<const float4*>(piece + 128);
      float4 v4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), u4 = v4;
      if (!PLAIN && !simple && L.v)
        v4 = *reinterpret_cast<const float4*>(piece + 256);
      if (!PLAIN && !simple && residual)
        u4 = *reinterpret_cast<const float4*>(piece + 384);
      __syncwarp();
      fetch(slot);
      slot = (slot + 1) & (D - 1);
      const size_t o = (size_t)(b0 + r) * s + col;
      float acc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
      for (int k4 = 0; k4 < KC; k4 += 4)
      {
        const float4 g4 = *reinterpret_cast<const float4*>(&gs[r][k4]);
#pragma unroll
        for (int c = 0; c < 4; ++c)
        {
          acc[c] = fmaf(g4.x, w[c][k4], acc[c]);
          acc[c] = fmaf(g4.y, w[c][k4 + 1], acc[c]);
          acc[c] = fmaf(g4.z, w[c][k4 + 2], acc[c]);
          acc[c] = fmaf(g4.w, w[c][k4 + 3], acc[c]);
        }
      }
      float zz[4] = {z4.x, z4.y, z4.z, z4.w};
      const float ee[4] = {e4.x, e4.y, e4.z, e4.w};
      float vv[4] = {v4.x, v4.y, v4.z, v4.w};
      const float uu[4] = {u4.x, u4.y, u4.z, u4.w};
      float dd[4];
      if (simple)
        act_deriv4(L.act, zz, dd);
#pragma unroll
      for (int c = 0; c < 4; ++c)
      {
        // (said which product is fused: the compiler shares the subtraction of both branches in one instance, not in others)
        if (simple)
          zz[c] += L.ir * fmaf(acc[c], dd[c], -ee[c]);
        else
        {
          const float fb = fmaf(L.a, acc[c], -ee[c]);
          if (!PLAIN && L.v)
          {
            vv[c] = L.momentum_beta * vv[c] + (1.0f - L.momentum_beta) * fb;
            zz[c] += L.ir * vv[c];
          }
          else
            zz[c] += L.ir * fb;
          if (!PLAIN && residual)
            zz[c] += L.ir * uu[c];
        }
      }
      if (!PLAIN && !simple && L.v)
        *reinterpret_cast<float4*>(L.v + o) = make_float4(vv[0], vv[1], vv[2], vv[3]);
      *reinterpret_cast<float4*>(L.z + o) = make_float4(zz[0], zz[1], zz[2], zz[3]);
    }
  }
}

// One entry of a weight update from the raw sum over the batch.
__device__ __forceinline__ void weight_apply(const dpc_layer& L, size_t o, float sum, int batch,
                                             int mode, int flags, float step)
{
  if (mode & WG_GRAD_ONLY)
    L.g_W[o] = sum;
  else if (mode == WG_LEARN && L.opt != DPC_OPT_SGD)
  {
    float mm = L.m_W[o], vv = L.v_W[o];
    L.W[o] = adam_update(L.W[o], -1.0f * L.a * sum, mm, vv, step, weight_wd(L));
    L.m_W[o] = mm;
    L.v_W[o] = vv;
  }
  else
    L.W[o] = weight_sgd(L, batch, mode == WG_DFA, (flags & 1) != 0)(L.W[o], sum);
}

// Weight update of a narrow layer (at most KC <= 16 output units, input width a multiple of 128:
// the heads, e.g. W[10 x 1024] += alpha fe^T z over a batch of 4096).  The tiled kernel gives such
// a layer size/64 blocks that each walk the whole batch; here the batch is split over warps and
// over the CTAs of a cluster as in the Psi update, whose shape this product shares.
template <int KC>
__global__ void __launch_bounds__(256, 2)
    narrow_weight_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers, int batch,
                         int flags, int mode)
{
  const int li = first + blockIdx.y;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0)
    return;
  const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
  const int base_mode = mode & ~WG_GRAD_ONLY;
  if (base_mode == WG_DFA && (li + 1 >= n_layers || layers[li + 1].Psi == nullptr))
    return; // DirectFeedbackUpdate is a no-op unless the layer above owns feedback weights
  const int M = L.next_size, s = L.size;
  if ((int)blockIdx.x * 128 >= s)
    return;
  const float* g = (simple && base_mode == WG_LEARN) ? layers[li + 1].e : L.fe;
  const float* zin = simple ? L.zF : L.z;
  __shared__ __align__(16) float smem[kOuterFloats<KC>];
  const int col = blockIdx.x * 128 + (threadIdx.x & 31) * 4;
  float acc[4][KC];
  if (!batch_outer4<KC>(zin, s, col, g, M, M, batch, acc, smem))
    return;
  const float step = mode == WG_LEARN && L.opt != DPC_OPT_SGD ? adam_step_size(L.lr, *L.t) : 0.0f;
#pragma unroll
  for (int c = 0; c < 4; ++c)
#pragma unroll
    for (int k = 0; k < KC; ++k)
      if (k < M)
        weight_apply(L, (size_t)k * s + col + c, acc[c][k], batch, mode, flags, step);
}

// Feedback-weight update Psi[l] (+)= (fl*a/B) z[l]^T e_T.  A block of 256 threads owns 32 rows of Psi (= 32 columns of z)
// and 16 terminal columns: thread (g, q, i) adds up the batch rows b = g, g+4, ... for columns i, i+16 and terminal
// columns 4q .. 4q+3, the four row groups are then summed in a fixed order through shared memory.  64 batch rows at a
// time come into shared memory two buffers ahead.  What bounds it: the copies, element by element where rows are not
// aligned, and the reads of shared memory.  (Blocks of 64 columns that walked the batch once for every 16 terminal
// columns kept few SMs busy: 784-(91x4)-100 at batch 3584 1049 -> 113 us, 784-(500x3)-100
// at batch 2000 603 -> 55; with 16 columns a block 109 and 89.)
__global__ void __launch_bounds__(256)
    psi_update_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers, int batch,
                      const float* __restrict__ eT, int grad_only)
{
  const int li = first + blockIdx.y;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0 || L.Psi == nullptr || (L.flags & DPC_LAYER_INPUT_ACT))
    return;
  const int TS = L.terminal_size, s = L.size;
  constexpr int ROWS = 64, GROUPS = 4, COLS = 32, STAGES = 3;
  const int i0 = blockIdx.x * COLS, kc = blockIdx.z * 16;
  if (i0 >= s || kc >= TS)
    return;
  __shared__ __align__(16) float es[STAGES][ROWS][16], zs[STAGES][ROWS][COLS];
  __shared__ float part[GROUPS][COLS][17];
  const int tid = threadIdx.x, i = tid & 15, q = (tid >> 4) & 3, g = tid >> 6;
  const int kn = min(16, TS - kc), width = min(COLS, s - i0);
  const bool vec_z = s % 4 == 0 && aligned16(L.z), vec_e = TS % 4 == 0 && aligned16(eT);
  // 64 rows from b0 of `count` columns (a multiple of 4 where they are copied by fours), zeros beyond
  auto rows_of = [&](auto per_row, auto fours, float* to, const float* from, int ld, int b0, int count)
  {
    constexpr int PER_ROW = decltype(per_row)::value, W = decltype(fours)::value ? 4 : 1, PER = PER_ROW / W;
    const int c = tid % PER * W;
#pragma unroll
    for (int u = 0; u < ROWS * PER / 256; ++u)
    {
      const int r = tid / PER + u * (256 / PER);
      const bool in = b0 + r < batch && c < count;
      const float* src = in ? from + (size_t)(b0 + r) * ld + c : from;
      if (W == 4)
        cp_async16(to + r * PER_ROW + c, src, in);
      else
        cp_async4(to + r * PER_ROW + c, src, in);
    }
  };
  auto copy = [&](int b0, int buf)
  {
    if (b0 < batch)
    {
      const std::integral_constant<int, COLS> columns;
      const std::integral_constant<int, 16> terminals;
      if (vec_z)
        rows_of(columns, std::true_type(), &zs[buf][0][0], L.z + i0, s, b0, width);
      else
        rows_of(columns, std::false_type(), &zs[buf][0][0], L.z + i0, s, b0, width);
      if (vec_e)
        rows_of(terminals, std::true_type(), &es[buf][0][0], eT + kc, TS, b0, kn);
      else
        rows_of(terminals, std::false_type(), &es[buf][0][0], eT + kc, TS, b0, kn);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  float acc[2][4] = {};
#pragma unroll 1
  for (int u = 0; u < STAGES - 1; ++u)
    copy(u * ROWS, u);
  const float step = psi_step(L, grad_only);
  int buf = 0;
#pragma unroll 1
  for (int b0 = 0; b0 < batch; b0 += ROWS, buf = buf + 1 == STAGES ? 0 : buf + 1)
  {
    asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
    __syncthreads(); // this buffer has landed, and everybody is done with the one that is filled now
    copy(b0 + (STAGES - 1) * ROWS, buf == 0 ? STAGES - 1 : buf - 1);
    const int rows = min(ROWS, batch - b0);
#pragma unroll 4
    for (int r = g; r < rows; r += GROUPS)
    {
      const float4 e4 = *reinterpret_cast<const float4*>(&es[buf][r][4 * q]);
#pragma unroll
      for (int c = 0; c < 2; ++c)
      {
        const float zv = zs[buf][r][i + 16 * c];
        acc[c][0] = fmaf(zv, e4.x, acc[c][0]);
        acc[c][1] = fmaf(zv, e4.y, acc[c][1]);
        acc[c][2] = fmaf(zv, e4.z, acc[c][2]);
        acc[c][3] = fmaf(zv, e4.w, acc[c][3]);
      }
    }
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
  for (int c = 0; c < 2; ++c)
#pragma unroll
    for (int k = 0; k < 4; ++k)
      part[g][i + 16 * c][4 * q + k] = acc[c][k];
  __syncthreads();
  const int k = tid & 15;
  for (int row = tid >> 4; row < width && k < kn; row += 16)
    psi_apply(L, i0 + row, kc + k, ((part[0][row][k] + part[1][row][k]) + part[2][row][k]) + part[3][row][k], batch,
              grad_only, step);
}

// Applies staged gradients (the raw sums that the WG_GRAD_ONLY weight kernel and the grad_only
// bias / Psi kernels left in g_W, g_b, g_Psi, possibly summed over batch shards since) with
// exactly the formulas of the fused updates above; `batch` is the batch the sums cover (the
// global one).  which = WG_LEARN: W, b and Psi; WG_DFA: W only (DirectFeedbackUpdate);
// 2: W only with the learn-step formulas (b and Psi are updated by their own fused kernels).
__global__ void apply_gradients_kernel(const dpc_layer* __restrict__ layers, int first,
                                       int n_layers, int batch, int which, int flags)
{
  const int li = first + blockIdx.y;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0)
    return;
  const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
  const size_t nW = (size_t)L.next_size * L.size;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nthr = (size_t)gridDim.x * blockDim.x;
  if (which == WG_DFA)
  {
    if (layers[li + 1].Psi == nullptr)
      return;
    const Sgd update = weight_sgd(L, batch, true, (flags & 1) != 0);
    for (size_t o = tid; o < nW; o += nthr)
      L.W[o] = update(L.W[o], L.g_W[o]);
    return;
  }
  if (L.opt == DPC_OPT_SGD)
  {
    const Sgd update = weight_sgd(L, batch, false, false), bias = bias_sgd(L, batch);
    for (size_t o = tid; o < nW; o += nthr)
      L.W[o] = update(L.W[o], L.g_W[o]);
    if (which != 2)
      for (size_t j = tid; j < (size_t)L.next_size; j += nthr)
        L.b[j] = bias(L.b[j], L.g_b[j]);
  }
  else
  {
    const float step = adam_step_size(L.lr, *L.t), lr_wd = weight_wd(L), alpha = -1.0f * L.a;
    for (size_t o = tid; o < nW; o += nthr)
    {
      float mm = L.m_W[o], vv = L.v_W[o];
      L.W[o] = adam_update(L.W[o], alpha * L.g_W[o], mm, vv, step, lr_wd);
      L.m_W[o] = mm;
      L.v_W[o] = vv;
    }
    if (which != 2)
      for (size_t j = tid; j < (size_t)L.next_size; j += nthr)
      {
        float m = L.m_b[j], v = L.v_b[j];
        L.b[j] = adam_update(L.b[j], -L.g_b[j], m, v, step, -1.0f);
        L.m_b[j] = m;
        L.v_b[j] = v;
      }
  }
  if (L.Psi == nullptr || simple || which == 2)
    return;
  const int TS = L.terminal_size;
  const size_t nP = (size_t)L.size * TS;
  if (L.opt_psi == DPC_OPT_SGD)
  {
    const Sgd update = psi_sgd(L, batch);
    for (size_t q = tid; q < nP; q += nthr)
    {
      const size_t o = (q / TS) * L.psi_stride + q % TS;
      L.Psi[o] = update(L.Psi[o], L.g_Psi[o]);
    }
  }
  else
  {
    const float step = adam_step_size(psi_rate(L), *L.t_Psi), lr_wd = psi_wd(L);
    for (size_t q = tid; q < nP; q += nthr)
    {
      const size_t o = (q / TS) * L.psi_stride + q % TS;
      float m = L.m_Psi[o], v = L.v_Psi[o];
      L.Psi[o] = adam_update(L.Psi[o], -L.g_Psi[o], m, v, step, lr_wd);
      L.m_Psi[o] = m;
      L.v_Psi[o] = v;
    }
  }
}

// Row centring of W: subtract each row's mean (src/backend/CPUBackend.cpp:250-272).
__global__ void center_rows_kernel(const dpc_layer* __restrict__ layers, int first, int n_layers)
{
  const int li = first + blockIdx.y;
  if (li + 1 >= n_layers)
    return;
  const dpc_layer L = layers[li];
  if (L.next_size <= 0)
    return;
  __shared__ float red[32];
  for (int r = blockIdx.x; r < L.next_size; r += gridDim.x)
  {
    float* row = L.W + (size_t)r * L.size;
    float s = 0.0f;
    for (int c = threadIdx.x; c < L.size; c += blockDim.x)
      s += row[c];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0)
      red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x < 32)
    {
      float t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0f;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        t += __shfl_xor_sync(0xffffffffu, t, o);
      if (threadIdx.x == 0)
        red[0] = t;
    }
    __syncthreads();
    const float mean = red[0] / (float)L.size;
    for (int c = threadIdx.x; c < L.size; c += blockDim.x)
      row[c] -= mean;
    __syncthreads();
  }
}
} // namespace dpc
