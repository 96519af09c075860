// Convolutional predictive coding (SimpleConvPCLayer / SimpleConvPCNetwork of the reference):
// implicit-GEMM kernels on the CUDA cores.  No im2col buffer, no repack: the gathers that
// the reference materialises (Im2Col, Col2Im, RepackForBatchedGemm) happen while a tile is
// fetched, and bias, activation, error, gated error, state update and energy are epilogues.
//
// Layouts are the reference's: z, e [B, C, H, W]; W [O, C*kH*kW] (row index (c*kH+ky)*kW+kx);
// b [O]; preact, mu [B, O, oH, oW].
#include <algorithm>
#include <cstring>

#include "dpc_conv_internal.h"
#include "dpc_math.cuh"

namespace dpc
{
namespace conv
{
constexpr int TM = 64, TN = 64, TK = 16, THREADS = 256, PADC = 4;

enum ConvOp
{
  C_FWD = 0, // preact[o, (b,p)] = sum_k W[o,k] * col(z)[k,(b,p)]       M=O    N=B*oH*oW K=C*kH*kW
  C_BWD = 1  // dz[c, (b,y,x)]   = sum_k W^T[c,k=(o,ky,kx)] * g gathered  M=C    N=B*H*W   K=O*kH*kW
};

struct Tile
{
  float a[TK][TM + PADC];
  float b[TK][TN + PADC];
};

__device__ __forceinline__ void block_energy(float local, double* energy)
{
  __shared__ float warp_sums[THREADS / 32];
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
    for (int w = 0; w < THREADS / 32; ++w)
      s += warp_sums[w];
    atomicAdd(energy, (double)(0.5f * s));
  }
}

template <int OP>
__global__ void __launch_bounds__(THREADS)
    conv_gemm_kernel(const dpc_conv_layer L, float* __restrict__ z_up, float* __restrict__ e_up,
                     int batch, int flags, double* energy, int k_chunk,
                     float* __restrict__ split_out = nullptr)
{
  const int C = L.in_c, O = L.out_c, H = L.in_h, Wd = L.in_w, kH = L.k_h, kW = L.k_w;
  const int oH = L.out_h, oW = L.out_w, P = oH * oW, HW = H * Wd, KK = kH * kW;
  const int rows = C * KK;
  int M, N, K;
  if (OP == C_FWD)
    M = O, N = batch * P, K = rows;
  else
    M = C, N = batch * HW, K = O * KK;
  const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
  // k_chunk > 0: the reduction is split over blockIdx.z and the partial sums are added
  // atomically into a zeroed buffer (preact for the forward product, `split_out` for the state
  // update); a second kernel applies the epilogue.
  int k_begin = 0, k_end = K;
  if (k_chunk > 0)
  {
    k_begin = blockIdx.z * k_chunk;
    k_end = min(K, k_begin + k_chunk);
  }

  __shared__ Tile tile;
  const int t = threadIdx.x;
  const int tx = t & 15, ty = t >> 4;

  // ---- per-thread invariants of the B-operand gather: 4 consecutive n, one k per pass
  const int bn = n0 + ((t & 15) << 2);
  int nb[4], ny[4], nx[4]; // image and (already offset) pixel origin
#pragma unroll
  for (int j = 0; j < 4; ++j)
  {
    const int n = bn + j;
    if (n >= N)
    {
      nb[j] = -1, ny[j] = nx[j] = 0;
      continue;
    }
    if (OP == C_FWD)
    {
      const int b = n / P, p = n - b * P;
      const int oy = p / oW, ox = p - oy * oW;
      nb[j] = b, ny[j] = oy * L.s_h - L.p_h, nx[j] = ox * L.s_w - L.p_w;
    }
    else
    {
      const int b = n / HW, q = n - b * HW;
      const int y = q / Wd, x = q - y * Wd;
      nb[j] = b, ny[j] = y + L.p_h, nx[j] = x + L.p_w;
    }
  }

  float ra[4], rb[4];
  auto fetch = [&](int k0)
  {
    // A operand: row = t>>2, 4 consecutive k
    {
      const int m = m0 + (t >> 2);
      const int kb = k0 + ((t & 3) << 2);
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        const int k = kb + j;
        float v = 0.0f;
        if (m < M && k < k_end)
        {
          if (OP == C_FWD)
            v = L.W[(size_t)m * rows + k];
          else
          {
            const int o = k / KK, r = k - o * KK;
            v = L.W[(size_t)o * rows + m * KK + r];
          }
        }
        ra[j] = v;
      }
    }
    // B operand: k = t>>4, 4 consecutive n
    {
      const int k = k0 + (t >> 4);
      int q0 = 0, q1 = 0, q2 = 0; // FWD: (c, ky, kx); BWD: (o, ky, kx)
      const bool kin = k < k_end;
      if (kin)
      {
        q0 = k / KK;
        const int r = k - q0 * KK;
        q1 = r / kW, q2 = r - q1 * kW;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        float v = 0.0f;
        if (kin && nb[j] >= 0)
        {
          if (OP == C_FWD)
          {
            const int iy = ny[j] + q1, ix = nx[j] + q2;
            if (iy >= 0 && iy < H && ix >= 0 && ix < Wd)
              v = L.z[(((size_t)nb[j] * C + q0) * H + iy) * Wd + ix];
          }
          else
          {
            const int ty2 = ny[j] - q1, tx2 = nx[j] - q2;
            if (ty2 >= 0 && tx2 >= 0)
            {
              const int oy = ty2 / L.s_h, ox = tx2 / L.s_w;
              if (oy * L.s_h == ty2 && ox * L.s_w == tx2 && oy < oH && ox < oW)
                v = L.g[(((size_t)nb[j] * O + q0) * oH + oy) * oW + ox];
            }
          }
        }
        rb[j] = v;
      }
    }
  };
  auto stash = [&]()
  {
    const int r = t >> 2, kq = (t & 3) << 2;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      tile.a[kq + j][r] = ra[j];
    *reinterpret_cast<float4*>(&tile.b[t >> 4][(t & 15) << 2]) =
        make_float4(rb[0], rb[1], rb[2], rb[3]);
  };

  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j)
      acc[i][j] = 0.0f;

  if (k_begin < k_end)
  {
    fetch(k_begin);
    stash();
    __syncthreads();
    for (int k0 = k_begin; k0 < k_end; k0 += TK)
    {
      const bool more = k0 + TK < k_end;
      if (more)
        fetch(k0 + TK);
#pragma unroll
      for (int k = 0; k < TK; ++k)
      {
        const float4 av = *reinterpret_cast<const float4*>(&tile.a[k][ty * 4]);
        const float4 bv = *reinterpret_cast<const float4*>(&tile.b[k][tx * 4]);
        const float a4[4] = {av.x, av.y, av.z, av.w};
        const float b4[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            acc[i][j] = fmaf(a4[i], b4[j], acc[i][j]);
      }
      __syncthreads();
      if (more)
      {
        stash();
        __syncthreads();
      }
    }
  }

  // ------------------------------------------------------------------ epilogues
  if (k_chunk > 0)
  {
    float* dst = OP == C_FWD ? L.preact : split_out;
    const int PP = OP == C_FWD ? P : HW; // pixels per (image, channel) plane of the output
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
      const int m = m0 + ty * 4 + i;
      if (m >= M)
        continue;
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        const int n = n0 + tx * 4 + j;
        if (n >= N)
          continue;
        const int b = n / PP, q = n - b * PP;
        atomicAdd(&dst[((size_t)b * M + m) * PP + q], acc[i][j]);
      }
    }
    return;
  }
  if (OP == C_FWD)
  {
    float esum = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
      const int m = m0 + ty * 4 + i;
      if (m >= M)
        continue;
      const float bias = L.b[m];
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        const int n = n0 + tx * 4 + j;
        if (n >= N)
          continue;
        const int b = n / P, p = n - b * P;
        const size_t o = ((size_t)b * O + m) * P + p;
        const float pre = acc[i][j] + bias;
        float mu, d;
        act_both(L.act, pre, mu, d);
        L.preact[o] = pre;
        L.mu[o] = mu;
        if (flags & DPC_CONV_COPY_NEXT)
          z_up[o] = mu;
        if (flags & DPC_CONV_ERR_NEXT)
        {
          const float e = ((flags & DPC_CONV_COPY_NEXT) ? mu : z_up[o]) - mu;
          e_up[o] = e;
          esum += e * e;
          L.g[o] = e * d;
        }
      }
    }
    if (flags & DPC_CONV_ENERGY)
      block_energy(esum, energy);
  }
  else
  {
#pragma unroll
    for (int i = 0; i < 4; ++i)
    {
      const int m = m0 + ty * 4 + i;
      if (m >= M)
        continue;
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        const int n = n0 + tx * 4 + j;
        if (n >= N)
          continue;
        const int b = n / HW, q = n - b * HW;
        const size_t o = ((size_t)b * C + m) * HW + q;
        L.z[o] += L.ir * (acc[i][j] - L.e[o]);
      }
    }
  }
}

// Second half of a split forward product: preact holds the raw sums; bias, activation, the
// error of the layer above, the gated error and the energy as in the fused epilogue.
__global__ void conv_forward_finish_kernel(const dpc_conv_layer L, float* __restrict__ z_up,
                                           float* __restrict__ e_up, int batch, int flags,
                                           double* energy)
{
  const int P = L.out_h * L.out_w;
  const size_t total = (size_t)batch * L.out_c * P;
  float esum = 0.0f;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
  {
    const int oc = (int)((o / P) % L.out_c);
    const float pre = L.preact[o] + L.b[oc];
    float mu, d;
    act_both(L.act, pre, mu, d);
    L.preact[o] = pre;
    L.mu[o] = mu;
    if (flags & DPC_CONV_COPY_NEXT)
      z_up[o] = mu;
    if (flags & DPC_CONV_ERR_NEXT)
    {
      const float e = ((flags & DPC_CONV_COPY_NEXT) ? mu : z_up[o]) - mu;
      e_up[o] = e;
      esum += e * e;
      L.g[o] = e * d;
    }
  }
  if (flags & DPC_CONV_ENERGY)
    block_energy(esum, energy);
}

// Second half of a split state update: z += ir*(dz - e) with dz = the summed partials.
__global__ void conv_state_finish_kernel(const dpc_conv_layer L, const float* __restrict__ dz,
                                         int batch)
{
  const size_t total = (size_t)batch * L.in_c * L.in_h * L.in_w;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    L.z[o] += L.ir * (dz[o] - L.e[o]);
}

// A clamped layer whose prediction is cached: no convolution, preact/mu are read back.
__global__ void conv_cached_forward_kernel(const dpc_conv_layer L, float* __restrict__ z_up,
                                           float* __restrict__ e_up, int batch, int flags,
                                           double* energy)
{
  const size_t total = (size_t)batch * L.out_c * L.out_h * L.out_w;
  float esum = 0.0f;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
  {
    const float mu = L.mu[o];
    if (flags & DPC_CONV_COPY_NEXT)
      z_up[o] = mu;
    if (flags & DPC_CONV_ERR_NEXT)
    {
      const float e = ((flags & DPC_CONV_COPY_NEXT) ? mu : z_up[o]) - mu;
      e_up[o] = e;
      esum += e * e;
      L.g[o] = e * act_deriv(L.act, L.preact[o]);
    }
  }
  if (flags & DPC_CONV_ENERGY)
    block_energy(esum, energy);
}

// g = e_above * mu with mu still holding the prediction: what the reference's weight update
// reads when no state update came after the last CalculateState
// (src/layers/SimpleConvPCLayer.cpp:414 with mu from :279-285).
__global__ void conv_gate_with_prediction_kernel(const dpc_conv_layer L,
                                                 const float* __restrict__ e_up, int batch)
{
  const size_t total = (size_t)batch * L.out_c * L.out_h * L.out_w;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    L.g[o] = e_up[o] * L.mu[o];
}

// z -= ir*e for a layer without weights (the terminal layer when it is not clamped).
__global__ void conv_relax_kernel(const dpc_conv_layer L, int batch)
{
  const size_t total = (size_t)batch * L.in_c * L.in_h * L.in_w;
  for (size_t o = (size_t)blockIdx.x * blockDim.x + threadIdx.x; o < total;
       o += (size_t)gridDim.x * blockDim.x)
    L.z[o] -= L.ir * L.e[o];
}

// Weight and bias gradients of a range of layers in one launch: dW[o, r] = sum_(b,p) g[o,(b,p)]
// col(z)[r,(b,p)] and db[o] = sum_(b,p) g[o,(b,p)], raw sums added atomically into zeroed g_W, g_b.
// A block takes one 64 x 64 tile and one slice of the batch x pixel reduction of one layer; all layers
// together fill the GPU, where one after the other each was a latency-bound launch (91 us for the four
// layers of a 32x32x3 network at batch 128, 97 us more for bias sums of their own).  The
// (image, pixel) of a k advances by additions, with a multiplication for the row instead of divisions.
struct GradGroup
{
  int layer, first, tiles_n, tiles, chunk; // first block, column tiles, tiles, k per slice
};
struct GradGroups
{
  GradGroup g[16];
  int count;
};
__global__ void __launch_bounds__(THREADS)
    conv_gradient_kernel(const dpc_conv_layer* __restrict__ layers, const GradGroups G, int batch)
{
  int gi = 0;
  while (gi + 1 < G.count && (int)blockIdx.x >= G.g[gi + 1].first)
    ++gi;
  const GradGroup D = G.g[gi];
  const dpc_conv_layer& L = layers[D.layer];
  const int C = L.in_c, O = L.out_c, H = L.in_h, Wd = L.in_w, kW = L.k_w, oW = L.out_w;
  const int P = L.out_h * oW, KK = L.k_h * kW, rows = C * KK;
  const int local = blockIdx.x - D.first, tile_i = local % D.tiles, slice = local / D.tiles;
  const int n0 = (tile_i % D.tiles_n) * TN, m0 = (tile_i / D.tiles_n) * TM;
  const int k_begin = slice * D.chunk, k_end = min(batch * P, k_begin + D.chunk);
  const float* __restrict__ g = L.g;
  const float* __restrict__ z = L.z;
  // p / oW as a multiplication, exact while p * oW < 2^32
  const unsigned by_row = oW > 1 && (unsigned long long)P * oW < 0x100000000ull
                              ? (unsigned)((0x100000000ull + oW - 1) / oW)
                              : 0u;
  __shared__ Tile tile;
  const int t = threadIdx.x, tx = t & 15, ty = t >> 4;
  // B operand: k = t>>4, four consecutive n = (c, ky, kx)
  int zc[4], dy[4], dx[4];
#pragma unroll
  for (int j = 0; j < 4; ++j)
  {
    const int n = n0 + ((t & 15) << 2) + j;
    const int c = n / KK, r = n - c * KK;
    zc[j] = n < rows ? c * H * Wd : -1;
    dy[j] = r / kW - L.p_h, dx[j] = r - (r / kW) * kW - L.p_w;
  }
  // A operand: row t>>2, four consecutive k
  const int am = m0 + (t >> 2);
  int ka = k_begin + ((t & 3) << 2), kb = k_begin + (t >> 4);
  int ab = ka / P, ap = ka - ab * P, bb = kb / P, bp = kb - bb * P;
  const bool vec = P % 4 == 0 && (reinterpret_cast<uintptr_t>(g) & 15) == 0;
  float ra[4], rb[4], bsum = 0.0f;
  auto fetch = [&]()
  {
    if (am < O && vec && ka + 3 < k_end)
    {
      const float4 v = *reinterpret_cast<const float4*>(g + ((size_t)ab * O + am) * P + ap);
      ra[0] = v.x, ra[1] = v.y, ra[2] = v.z, ra[3] = v.w;
    }
    else
    {
      int b = ab, p = ap;
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        ra[j] = am < O && ka + j < k_end ? g[((size_t)b * O + am) * P + p] : 0.0f;
        if (++p == P)
          p = 0, ++b;
      }
    }
    const int oy = by_row ? (int)__umulhi((unsigned)bp, by_row) : bp / oW, ox = bp - oy * oW;
    const float* zi = z + (size_t)bb * C * H * Wd;
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      const int iy = oy * L.s_h + dy[j], ix = ox * L.s_w + dx[j];
      rb[j] = kb < k_end && zc[j] >= 0 && (unsigned)iy < (unsigned)H && (unsigned)ix < (unsigned)Wd
                  ? zi[zc[j] + iy * Wd + ix]
                  : 0.0f;
    }
    ka += TK, kb += TK;
    for (ap += TK; ap >= P; ap -= P)
      ++ab;
    for (bp += TK; bp >= P; bp -= P)
      ++bb;
  };
  auto stash = [&]()
  {
    const int r = t >> 2, kq = (t & 3) << 2;
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      tile.a[kq + j][r] = ra[j];
      bsum += ra[j];
    }
    *reinterpret_cast<float4*>(&tile.b[t >> 4][(t & 15) << 2]) = make_float4(rb[0], rb[1], rb[2], rb[3]);
  };
  float acc[4][4] = {};
  fetch();
  stash();
  __syncthreads();
  for (int k0 = k_begin; k0 < k_end; k0 += TK)
  {
    const bool more = k0 + TK < k_end;
    if (more)
      fetch();
#pragma unroll
    for (int k = 0; k < TK; ++k)
    {
      const float4 av = *reinterpret_cast<const float4*>(&tile.a[k][ty * 4]);
      const float4 bv = *reinterpret_cast<const float4*>(&tile.b[k][tx * 4]);
      const float a4[4] = {av.x, av.y, av.z, av.w};
      const float b4[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[i][j] = fmaf(a4[i], b4[j], acc[i][j]);
    }
    __syncthreads();
    if (more)
    {
      stash();
      __syncthreads();
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
  {
    const int m = m0 + ty * 4 + i;
    if (m >= O)
      continue;
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      const int n = n0 + tx * 4 + j;
      if (n < rows)
        atomicAdd(&L.g_W[(size_t)m * rows + n], acc[i][j]);
    }
  }
  if (n0 == 0)
  {
    bsum += __shfl_xor_sync(0xffffffffu, bsum, 1);
    bsum += __shfl_xor_sync(0xffffffffu, bsum, 2);
    if ((t & 3) == 0 && am < O)
      atomicAdd(&L.g_b[am], bsum);
  }
}

// Zeroes the sums that the gradient launch adds into.  blockIdx.y = layer.
__global__ void conv_zero_sums_kernel(const dpc_conv_layer* __restrict__ layers, int first)
{
  const dpc_conv_layer& L = layers[first + blockIdx.y];
  const size_t nW = L.out_c > 0 ? (size_t)L.out_c * L.in_c * L.k_h * L.k_w : 0;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  for (size_t o = tid; o < nW; o += (size_t)gridDim.x * blockDim.x)
    L.g_W[o] = 0.0f;
  for (int j = (int)tid; j < L.out_c; j += gridDim.x * blockDim.x)
    L.g_b[j] = 0.0f;
}

// SGD / Adam / AdamW on W and b from the raw sums in g_W, g_b
// (src/layers/SimpleConvPCLayer.cpp:424-556: SGD rate lr/B with decay (1-lambda) first;
// Adam-type gradients are -(1/B) * sum).
// blockIdx.y = layer.
__global__ void conv_apply_kernel(const dpc_conv_layer* __restrict__ layers, int first, int batch)
{
  const dpc_conv_layer L = layers[first + blockIdx.y];
  if (L.out_c <= 0)
    return;
  const size_t nW = (size_t)L.out_c * L.in_c * L.k_h * L.k_w;
  const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t nthr = (size_t)gridDim.x * blockDim.x;
  const float Bf = (float)batch;
  if (L.opt == DPC_OPT_SGD)
  {
    const float alpha = L.lr / Bf;
    const float decay = L.lmbda > 0.0f ? 1.0f - L.lmbda : 1.0f;
    for (size_t o = tid; o < nW; o += nthr)
    {
      float w = L.W[o];
      if (decay != 1.0f)
        w *= decay;
      L.W[o] = fmaf(alpha, L.g_W[o], w);
    }
    for (size_t j = tid; j < (size_t)L.out_c; j += nthr)
      L.b[j] = fmaf(alpha, L.g_b[j], L.b[j]);
    return;
  }
  const float step = adam_step_size(L.lr, *L.t + 1); // (the counter itself moves on afterwards)
  const float lr_wd = L.opt == DPC_OPT_ADAMW ? L.lr * L.lmbda : -1.0f;
  const float gs = -1.0f / Bf;
  for (size_t o = tid; o < nW; o += nthr)
  {
    float m = L.m_W[o], v = L.v_W[o];
    L.W[o] = adam_update(L.W[o], gs * L.g_W[o], m, v, step, lr_wd);
    L.m_W[o] = m;
    L.v_W[o] = v;
  }
  for (size_t j = tid; j < (size_t)L.out_c; j += nthr)
  {
    float m = L.m_b[j], v = L.v_b[j];
    L.b[j] = adam_update(L.b[j], gs * L.g_b[j], m, v, step, -1.0f);
    L.m_b[j] = m;
    L.v_b[j] = v;
  }
}

__global__ void conv_bump_counter_kernel(const dpc_conv_layer* __restrict__ layers, int first)
{
  const dpc_conv_layer& L = layers[first + threadIdx.x];
  if (L.out_c > 0 && L.opt != DPC_OPT_SGD)
    *L.t += 1;
}

// Row centring of W [O, C*kH*kW] (src/backend/CPUBackend.cpp:250-272): one block per row.
__global__ void conv_center_rows_kernel(const dpc_conv_layer* __restrict__ layers, int first)
{
  const dpc_conv_layer& L = layers[first + blockIdx.y];
  if ((int)blockIdx.x >= L.out_c)
    return;
  const int rows = L.in_c * L.k_h * L.k_w;
  float* row = L.W + (size_t)blockIdx.x * rows;
  float s = 0.0f;
  for (int c = threadIdx.x; c < rows; c += blockDim.x)
    s += row[c];
  __shared__ float red[32];
#pragma unroll
  for (int w = 16; w > 0; w >>= 1)
    s += __shfl_xor_sync(0xffffffffu, s, w);
  if ((threadIdx.x & 31) == 0)
    red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    float tsum = 0.0f;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w)
      tsum += red[w];
    red[0] = tsum;
  }
  __syncthreads();
  const float mean = red[0] / (float)rows;
  for (int c = threadIdx.x; c < rows; c += blockDim.x)
    row[c] -= mean;
}
} // namespace conv
} // namespace dpc

using namespace dpc;
using namespace dpc::conv;

namespace
{
// How many ways to split a reduction of length K over CTAs when the tile grid alone does not
// fill the GPU (returns 1 for "do not split"); k_chunk comes back as a multiple of TK.
int choose_split(int tiles, long long K, int sm_count, int* k_chunk)
{
  int splits = 1;
  if (tiles < sm_count && K >= 8 * TK)
    splits = (int)std::min<long long>((2LL * sm_count + tiles - 1) / tiles, K / (2 * TK));
  if (splits <= 1)
  {
    *k_chunk = 0;
    return 1;
  }
  long long chunk = (K + splits - 1) / splits;
  chunk = (chunk + TK - 1) / TK * TK;
  *k_chunk = (int)chunk;
  return (int)((K + chunk - 1) / chunk);
}

int conv_check_launch(dpc_ctx* ctx, const char* what)
{
  ctx->launches += 1;
  cudaError_t err = cudaPeekAtLastError();
  if (err != cudaSuccess)
    return cuda_fail(cudaGetLastError(), what);
  return DPC_OK;
}

inline int cdiv_i(long long a, long long b)
{
  return (int)((a + b - 1) / b);
}

int elem_grid(const dpc_conv_plan* p, size_t elems)
{
  size_t blocks = (elems + 1023) / 1024;
  const size_t cap = (size_t)p->ctx->sm_count * 8;
  return (int)std::max<size_t>(1, std::min(blocks, cap));
}

int validate(const dpc_conv_layer* l, int n)
{
  if (n < 2)
    return fail(DPC_ERR_INVALID, "a network needs at least two layers");
  for (int i = 0; i < n; ++i)
  {
    const dpc_conv_layer& L = l[i];
    if (L.in_c <= 0 || L.in_h <= 0 || L.in_w <= 0 || !L.z || !L.e)
      return fail(DPC_ERR_INVALID, "conv layer " + std::to_string(i) + ": bad input shape or state");
    if (L.out_c > 0)
    {
      if (L.k_h <= 0 || L.k_w <= 0 || L.s_h <= 0 || L.s_w <= 0 || L.p_h < 0 || L.p_w < 0)
        return fail(DPC_ERR_INVALID, "conv layer " + std::to_string(i) + ": bad kernel geometry");
      const int oh = (L.in_h + 2 * L.p_h - L.k_h) / L.s_h + 1;
      const int ow = (L.in_w + 2 * L.p_w - L.k_w) / L.s_w + 1;
      if (oh != L.out_h || ow != L.out_w || oh <= 0 || ow <= 0)
        return fail(DPC_ERR_INVALID, "conv layer " + std::to_string(i) + ": output size mismatch");
      if (!L.W || !L.b || !L.preact || !L.mu || !L.g || !L.g_W || !L.g_b)
        return fail(DPC_ERR_INVALID, "conv layer " + std::to_string(i) + ": missing tensors");
      if (L.opt != DPC_OPT_SGD && (!L.m_W || !L.v_W || !L.m_b || !L.v_b || !L.t))
        return fail(DPC_ERR_INVALID, "conv layer " + std::to_string(i) + ": missing Adam state");
      if (i + 1 >= n)
        return fail(DPC_ERR_INVALID, "the last layer must have out_c = 0");
      const dpc_conv_layer& U = l[i + 1];
      if (U.in_c != L.out_c || U.in_h != L.out_h || U.in_w != L.out_w)
        return fail(DPC_ERR_INVALID, "conv layer " + std::to_string(i) +
                                         ": output shape differs from the next layer's input");
    }
    else if (i + 1 != n)
      return fail(DPC_ERR_INVALID, "only the last layer may have out_c = 0");
  }
  return DPC_OK;
}

// The layer table on the device.
int upload_layers(dpc_conv_plan* p)
{
  if (!p->d)
    DPC_CUDA(cudaMalloc(&p->d, sizeof(dpc_conv_layer) * p->n));
  DPC_CUDA(cudaMemcpyAsync(p->d, p->h.data(), sizeof(dpc_conv_layer) * p->n, cudaMemcpyHostToDevice,
                           p->ctx->stream));
  return DPC_OK;
}

int check_layer(dpc_conv_plan* p, int layer)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  if (layer < 0 || layer >= p->n)
    return fail(DPC_ERR_INVALID, "layer out of range");
  return DPC_OK;
}
} // namespace

int dpc_conv_plan_create(dpc_ctx* ctx, const dpc_conv_layer* layers, int n_layers, int batch,
                         dpc_conv_plan** out)
{
  if (!ctx || !layers || !out || batch <= 0)
    return fail(DPC_ERR_INVALID, "bad argument");
  int rc = validate(layers, n_layers);
  if (rc != DPC_OK)
    return rc;
  DPC_CUDA(cudaSetDevice(ctx->device));
  auto* p = new dpc_conv_plan();
  p->ctx = ctx, p->n = n_layers, p->batch = batch;
  p->h.assign(layers, layers + n_layers);
  if (cudaMalloc(&p->energy, sizeof(double)) != cudaSuccess ||
      cudaMallocHost(&p->energy_host, sizeof(double)) != cudaSuccess)
  {
    delete p;
    return cuda_fail(cudaGetLastError(), "conv plan allocation");
  }
  cudaMemsetAsync(p->energy, 0, sizeof(double), ctx->stream);
  if ((rc = upload_layers(p)) != DPC_OK)
  {
    dpc_conv_plan_destroy(p);
    return rc;
  }
  for (int i = 0; i < n_layers; ++i)
    p->scratch_floats += (size_t)batch * layers[i].in_c * layers[i].in_h * layers[i].in_w;
  if (cudaMalloc(&p->scratch, p->scratch_floats * sizeof(float)) != cudaSuccess)
  {
    const cudaError_t e = cudaGetLastError();
    dpc_conv_plan_destroy(p);
    return cuda_fail(e, "conv plan scratch allocation");
  }
  if ((rc = conv_res_init(p)) < 0)
  {
    dpc_conv_plan_destroy(p);
    return rc;
  }
  *out = p;
  return DPC_OK;
}

int dpc_conv_plan_update(dpc_conv_plan* p, const dpc_conv_layer* layers, int n_layers)
{
  if (!p || !layers || n_layers != p->n)
    return fail(DPC_ERR_INVALID, "bad argument");
  int rc = validate(layers, n_layers);
  if (rc != DPC_OK)
    return rc;
  // new rates only: see dpc_plan_update
  bool structure = false;
  for (int i = 0; i < n_layers && !structure; ++i)
  {
    dpc_conv_layer a = p->h[i], b = layers[i];
    for (dpc_conv_layer* q : {&a, &b})
      q->lr = q->ir = q->lmbda = 0.0f;
    structure = memcmp(&a, &b, sizeof(dpc_conv_layer)) != 0;
  }
  if (!structure)
  {
    p->h.assign(layers, layers + n_layers);
    DPC_CUDA(cudaMemcpyAsync(p->d, p->h.data(), sizeof(dpc_conv_layer) * n_layers,
                             cudaMemcpyHostToDevice, p->ctx->stream));
    return DPC_OK;
  }
  DPC_CUDA(cudaStreamSynchronize(p->ctx->stream));
  p->h.assign(layers, layers + n_layers);
  if ((rc = upload_layers(p)) != DPC_OK)
    return rc;
  conv_res_free(p);
  rc = conv_res_init(p);
  return rc < 0 ? rc : DPC_OK;
}

int dpc_conv_plan_destroy(dpc_conv_plan* p)
{
  if (!p)
    return DPC_OK;
  cudaSetDevice(p->ctx->device);
  cudaStreamSynchronize(p->ctx->stream);
  conv_res_free(p);
  cudaFree(p->d);
  if (p->energy)
    cudaFree(p->energy);
  if (p->energy_host)
    cudaFreeHost(p->energy_host);
  if (p->scratch)
    cudaFree(p->scratch);
  delete p;
  return DPC_OK;
}

int dpc_conv_forward(dpc_conv_plan* p, int layer, int flags)
{
  int rc = check_layer(p, layer);
  if (rc != DPC_OK)
    return rc;
  const dpc_conv_layer& L = p->h[layer];
  if (L.out_c <= 0)
    return DPC_OK;
  const dpc_conv_layer& U = p->h[layer + 1];
  cudaStream_t st = p->ctx->stream;
  const size_t outs = (size_t)p->batch * L.out_c * L.out_h * L.out_w;
  if (flags & DPC_CONV_CACHED)
  {
    if (!(flags & (DPC_CONV_COPY_NEXT | DPC_CONV_ERR_NEXT | DPC_CONV_ENERGY)))
      return DPC_OK;
    conv_cached_forward_kernel<<<elem_grid(p, outs), THREADS, 0, st>>>(L, U.z, U.e, p->batch,
                                                                      flags, p->energy);
    return conv_check_launch(p->ctx, "conv cached forward kernel");
  }
  const long long N = (long long)p->batch * L.out_h * L.out_w;
  dim3 grid(cdiv_i(N, TN), cdiv_i(L.out_c, TM), 1);
  int k_chunk = 0;
  const int splits = choose_split((int)(grid.x * grid.y), (long long)L.in_c * L.k_h * L.k_w,
                                  p->ctx->sm_count, &k_chunk);
  if (splits > 1)
  {
    grid.z = splits;
    DPC_CUDA(cudaMemsetAsync(L.preact, 0, outs * sizeof(float), st));
    conv_gemm_kernel<C_FWD><<<grid, THREADS, 0, st>>>(L, U.z, U.e, p->batch, flags, p->energy,
                                                     k_chunk);
    if ((rc = conv_check_launch(p->ctx, "conv forward kernel (split)")) != DPC_OK)
      return rc;
    conv_forward_finish_kernel<<<elem_grid(p, outs), THREADS, 0, st>>>(L, U.z, U.e, p->batch, flags,
                                                                      p->energy);
    return conv_check_launch(p->ctx, "conv forward finish kernel");
  }
  conv_gemm_kernel<C_FWD><<<grid, THREADS, 0, st>>>(L, U.z, U.e, p->batch, flags, p->energy, 0);
  return conv_check_launch(p->ctx, "conv forward kernel");
}

int dpc_conv_update_state(dpc_conv_plan* p, int layer)
{
  int rc = check_layer(p, layer);
  if (rc != DPC_OK)
    return rc;
  const dpc_conv_layer& L = p->h[layer];
  cudaStream_t st = p->ctx->stream;
  const size_t ins = (size_t)p->batch * L.in_c * L.in_h * L.in_w;
  if (L.out_c <= 0 || layer + 1 >= p->n)
  {
    conv_relax_kernel<<<elem_grid(p, ins), THREADS, 0, st>>>(L, p->batch);
    return conv_check_launch(p->ctx, "conv relax kernel");
  }
  float* scratch = p->scratch;
  for (int i = 0; i < layer; ++i)
    scratch += (size_t)p->batch * p->h[i].in_c * p->h[i].in_h * p->h[i].in_w;
  const long long N = (long long)p->batch * L.in_h * L.in_w;
  dim3 grid(cdiv_i(N, TN), cdiv_i(L.in_c, TM), 1);
  int k_chunk = 0;
  const int splits = choose_split((int)(grid.x * grid.y), (long long)L.out_c * L.k_h * L.k_w,
                                  p->ctx->sm_count, &k_chunk);
  if (splits > 1)
  {
    grid.z = splits;
    DPC_CUDA(cudaMemsetAsync(scratch, 0, ins * sizeof(float), st));
    conv_gemm_kernel<C_BWD><<<grid, THREADS, 0, st>>>(L, nullptr, nullptr, p->batch, 0, p->energy,
                                                     k_chunk, scratch);
    if ((rc = conv_check_launch(p->ctx, "conv state update kernel (split)")) != DPC_OK)
      return rc;
    conv_state_finish_kernel<<<elem_grid(p, ins), THREADS, 0, st>>>(L, scratch, p->batch);
    return conv_check_launch(p->ctx, "conv state finish kernel");
  }
  conv_gemm_kernel<C_BWD><<<grid, THREADS, 0, st>>>(L, nullptr, nullptr, p->batch, 0, p->energy, 0);
  return conv_check_launch(p->ctx, "conv state update kernel");
}

// The layers of a settling pass do not depend on each other and a launch of a small batch leaves most
// SMs idle: side by side, the longest layer first.  16-32-64 channels of 3x3 taps on 32x32 pixels at
// batch 4, 8 passes (a state too large for image segments): 1.31 -> 0.91 ms a step.
static int conv_side_by_side(dpc_conv_plan* p, int first, int count, const std::function<int(int)>& one)
{
  std::vector<std::pair<double, Job>> work;
  for (int i = first; i < first + count; ++i)
  {
    const dpc_conv_layer& L = p->h[i];
    work.emplace_back((double)L.out_c * L.out_h * L.out_w * L.in_c * L.k_h * L.k_w, [=] { return one(i); });
  }
  std::stable_sort(work.begin(), work.end(), [](const auto& a, const auto& b) { return a.first > b.first; });
  std::vector<Job> jobs;
  for (auto& w : work)
    jobs.push_back(w.second);
  return run_side_by_side(p->ctx, jobs);
}

int dpc_conv_forward_range(dpc_conv_plan* p, int first, int count, int flags)
{
  int rc = check_layer(p, first);
  if (rc != DPC_OK || (rc = check_layer(p, first + count - 1)) != DPC_OK)
    return rc;
  if (flags & DPC_CONV_COPY_NEXT)
    return fail(DPC_ERR_INVALID, "dpc_conv_forward_range: a sweep's layers follow one another");
  const bool cached_first = (flags & DPC_CONV_CACHED) != 0;
  const int rest = flags & ~DPC_CONV_CACHED;
  return conv_side_by_side(p, first, count, [=](int i)
                           { return dpc_conv_forward(p, i, cached_first && i == first ? flags : rest); });
}

int dpc_conv_update_state_range(dpc_conv_plan* p, int first, int count)
{
  int rc = check_layer(p, first);
  if (rc != DPC_OK || (rc = check_layer(p, first + count - 1)) != DPC_OK)
    return rc;
  return conv_side_by_side(p, first, count, [=](int i) { return dpc_conv_update_state(p, i); });
}

int dpc_conv_gate_with_prediction(dpc_conv_plan* p, int layer)
{
  int rc = check_layer(p, layer);
  if (rc != DPC_OK)
    return rc;
  const dpc_conv_layer& L = p->h[layer];
  if (L.out_c <= 0)
    return DPC_OK;
  const size_t outs = (size_t)p->batch * L.out_c * L.out_h * L.out_w;
  conv_gate_with_prediction_kernel<<<elem_grid(p, outs), THREADS, 0, p->ctx->stream>>>(
      L, p->h[layer + 1].e, p->batch);
  return conv_check_launch(p->ctx, "conv gate kernel");
}

int dpc_conv_update_weights(dpc_conv_plan* p, int layer, int center_rows)
{
  return dpc_conv_update_weights_range(p, layer, 1, center_rows);
}

int dpc_conv_update_weights_range(dpc_conv_plan* p, int first, int count, int center_rows)
{
  int rc = check_layer(p, first);
  if (rc != DPC_OK || (rc = check_layer(p, first + count - 1)) != DPC_OK)
    return rc;
  cudaStream_t st = p->ctx->stream;
  while (count > 0)
  {
    const int c = std::min(count, 16);
    GradGroups G = {};
    int blocks = 0, adam = 0, max_o = 0;
    size_t max_w = 0;
    // every layer's reduction is split so that the layers together give about four blocks per SM
    double total = 0.0;
    for (int i = first; i < first + c; ++i)
    {
      const dpc_conv_layer& L = p->h[i];
      if (L.out_c > 0)
        total += (double)cdiv_i((long long)L.in_c * L.k_h * L.k_w, TN) * cdiv_i(L.out_c, TM) * p->batch *
                 L.out_h * L.out_w;
    }
    for (int i = first; i < first + c; ++i)
    {
      const dpc_conv_layer& L = p->h[i];
      if (L.out_c <= 0)
        continue;
      const int rows = L.in_c * L.k_h * L.k_w;
      const long long K = (long long)p->batch * L.out_h * L.out_w;
      GradGroup& g = G.g[G.count++];
      g.layer = i, g.first = blocks;
      g.tiles_n = cdiv_i(rows, TN), g.tiles = g.tiles_n * cdiv_i(L.out_c, TM);
      long long chunk = (long long)(total / (4.0 * p->ctx->sm_count)) + 1;
      chunk = std::min(std::max<long long>(chunk, 4 * TK), K);
      g.chunk = cdiv_i(chunk, TK) * TK;
      blocks += g.tiles * cdiv_i(K, g.chunk);
      adam |= L.opt != DPC_OPT_SGD;
      max_w = std::max(max_w, (size_t)L.out_c * rows);
      max_o = std::max(max_o, L.out_c);
    }
    if (G.count > 0)
    {
      conv_zero_sums_kernel<<<dim3(elem_grid(p, max_w), c), THREADS, 0, st>>>(p->d, first);
      if ((rc = conv_check_launch(p->ctx, "conv zero sums kernel")) != DPC_OK)
        return rc;
      conv_gradient_kernel<<<blocks, THREADS, 0, st>>>(p->d, G, p->batch);
      if ((rc = conv_check_launch(p->ctx, "conv gradient kernel")) != DPC_OK)
        return rc;
      conv_apply_kernel<<<dim3(elem_grid(p, max_w), c), THREADS, 0, st>>>(p->d, first, p->batch);
      if ((rc = conv_check_launch(p->ctx, "conv apply kernel")) != DPC_OK)
        return rc;
      if (adam)
      {
        conv_bump_counter_kernel<<<1, c, 0, st>>>(p->d, first);
        if ((rc = conv_check_launch(p->ctx, "conv counter kernel")) != DPC_OK)
          return rc;
      }
      if (center_rows)
      {
        conv_center_rows_kernel<<<dim3(max_o, c), 128, 0, st>>>(p->d, first);
        if ((rc = conv_check_launch(p->ctx, "conv center rows kernel")) != DPC_OK)
          return rc;
      }
    }
    first += c, count -= c;
  }
  return DPC_OK;
}

int dpc_conv_energy_reset(dpc_conv_plan* p)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  DPC_CUDA(cudaMemsetAsync(p->energy, 0, sizeof(double), p->ctx->stream));
  return DPC_OK;
}

int dpc_conv_energy_read(dpc_conv_plan* p, double* out)
{
  const int rc = dpc_conv_energy_fetch(p);
  return rc == DPC_OK ? dpc_conv_energy_wait(p, out) : rc;
}

int dpc_conv_energy_fetch(dpc_conv_plan* p)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  DPC_CUDA(cudaMemcpyAsync(p->energy_host, p->energy, sizeof(double), cudaMemcpyDeviceToHost,
                           p->ctx->stream));
  return DPC_OK;
}

int dpc_conv_energy_wait(dpc_conv_plan* p, double* out)
{
  if (!p || !out)
    return fail(DPC_ERR_INVALID, "bad argument");
  DPC_CUDA(cudaStreamSynchronize(p->ctx->stream));
  *out = *p->energy_host;
  return DPC_OK;
}
