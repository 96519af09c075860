// Image-resident train step of convolutional networks (SimpleConvPCLayer / SimpleConvPCNetwork).
//
// As in the dense networks (dpc_resident.cu) the images of a batch meet only in the weight updates.
// One CTA keeps one image's beliefs, errors and gated errors in shared memory -- 170 KB for a
// 32x32x3 network of 32-64-128 channels -- and walks projection, settling steps and energy in one
// launch; the weights stream from L2.  The launches it replaces took 430 us per settling step of
// that network at batch 128 (the transposed convolution alone 209 us: a gather over all taps of
// which stride 2 wastes three in four, with integer divisions per element); this kernel takes 36 us
// (433 us for a segment of ten, 73 of which are loads, the input layer and a closing pass).
//
// Both products are implicit GEMMs on the tensor cores with separable addresses: the operand of
// (k, pixel) sits at koff[k] + base[pixel], with zero borders around the planes instead of tests.
//   forward   out[o][p]  = sum_k W[o][k] z[koff[k] + base[p]]
//   state     dz[c][q]   = sum_k W'[c][k] g[koff[k] + base[q]], one product per stride-parity class
//             of input pixels: only the taps that hit an output pixel are in its k range
// A warp owns 16 or 32 output channels x 8..32 pixels (mma.m16n8k8 on tf32, three passes hi*lo + lo*hi
// + hi*hi with fp32 accumulation: the fp32 scheme of the tensor-core kernels of dpc_tc.cu).  The
// weights come in fragment order (conv_pack_kernel, once per weight update), so a lane's four elements
// are one 16-byte load, kDepth of them in flight.  mma.sync and not tcgen05: the products
// of one image are 16..128 x 64..256 x 64..576, far below a 128-row tile.
// Layers whose output is one pixel (dense heads) are dot products on the CUDA cores.
// What bounds it: the SM's load path -- every task reads its weight fragments again, 16 bytes a lane per
// k step -- and behind it the tensor pipe.  32x32x3 network at batch 128, 10 steps: 4.57 -> 0.70 ms a step.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "dpc_conv_internal.h"
#include "dpc_math.cuh"

namespace dpc
{
namespace conv
{
namespace
{
constexpr int kThreads = 512, kWarps = kThreads / 32, kMaxLayers = 16;
constexpr size_t kSmemLimit = 227 * 1024, kStatic = 4 * 1024;
constexpr int kDepth = 4; // weight loads in flight; the packed steps and the koff table are padded to it

struct RcLayer // per weight layer l; "up" is layer l + 1, the state it predicts
{
  int C, HW, O, P;               // input channels and pixels, outputs, output pixels
  int zoff, zplane, zpix;        // state l: first float, floats per channel, pixel table
  int uoff, uplane, upix;        // the same of state l + 1
  int eoff;                      // errors of state l + 1 (l = 0: none kept, z - mu0)
  int goff, gplane, gpix;        // gated errors of this layer's outputs (l = 0: none kept)
  int boff;                      // bias
  int dense;                     // one output pixel, no padding
  int vec;                       // ... and rows of W that can be read 16 bytes at a time
  int ffirst, fcount;            // forward tasks
};

struct __align__(16) RcTask
{
  int w, ks;     // float4 offset into the packed weights, steps of 8 along K (dense: first output/column)
  int ktab;      // koff table
  int ntab;      // pixel table: base, pixel index pairs
  int m0, count; // first output row, pixels of the tile (dense: outputs or columns)
  int shape;     // 8 x (16-row tiles) + (8-pixel tiles)
  int what;      // layer << 2 | op
};
enum
{
  OP_FORWARD = 0,
  OP_STATE = 1,
  OP_DENSE_FORWARD = 2,
  OP_DENSE_STATE = 3
};

struct RcPack // one (layer, role, class): how its weights are arranged
{
  int layer, w, ks, mblocks, M, mstride, aoff; // aoff: table of K source offsets, -1: zero
};

struct RcParams
{
  const dpc_conv_layer* layers;
  const RcLayer* rl;
  const RcTask* tasks;          // forward (by layer), then state; copied to shared memory
  const unsigned short* order;  // both lists again, longest tasks first
  const unsigned short* table;  // pixel tables
  const uint2* koff;            // per step and lane % 4: byte offsets of its two k
  const float4* packed;
  int nw, batch;
  int nf, nb, table_vecs, koff_vecs;
  int zfloats, mu0, efloat, gfloat, xoff, xfloats; // regions, in floats
  int tab_at, koff_at, task_at, order_at, bias_at, bias_n;  // further regions, float offsets
  int ops, steps, top_clamped;
  double* energy;
};

// The tensor core reads the leading 11 significant bits of a tf32 operand: x itself serves as its high
// part, and the remainder is exact (its own trailing bits, 2^-21 of |x|, are not read).
__device__ __forceinline__ uint32_t tf32_rest(float x)
{
  return __float_as_uint(x - __uint_as_float(__float_as_uint(x) & 0xffffe000u));
}
__device__ __forceinline__ float lds(uint32_t address)
{
  float v;
  asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(address));
  return v;
}

__device__ __forceinline__ void mma8(float (&c)[4], const float4& a, uint32_t b0, uint32_t b1)
{
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, "
               "{%8,%9}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(__float_as_uint(a.x)), "r"(__float_as_uint(a.y)), "r"(__float_as_uint(a.z)),
                 "r"(__float_as_uint(a.w)), "r"(b0), "r"(b1));
}

// acc[i][j]: rows m0 + 16 i + lane/4 (+8), pixels 8 j + 2 (lane % 4) (+1) of the task's tile
template <int MT, int NTL>
__device__ __forceinline__ void mma_tile(float (&acc)[MT][NTL][4], const RcTask& t, const float4* packed,
                                         const unsigned short* T, const uint2* koff, const float* sm,
                                         int lane)
{
  const int g = lane >> 2, c = lane & 3;
  uint32_t base[NTL];
  float cor[MT][NTL][4]; // the two small products: chains of their own
#pragma unroll
  for (int j = 0; j < NTL; ++j)
  {
    const int n = 8 * j + g;
    base[j] = (uint32_t)__cvta_generic_to_shared(sm + T[t.ntab + 2 * (n < t.count ? n : 0)]);
  }
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        acc[i][j][q] = cor[i][j][q] = 0.0f;
  if (t.ks == 0)
    return;
  // (the loads of the last kDepth steps run past the task's weights, inside the buffer)
  const float4* A[MT];
#pragma unroll
  for (int i = 0; i < MT; ++i)
    A[i] = packed + t.w + lane + i * t.ks * 32;
  const uint2* K = koff + t.ktab + c;
  float4 ring[kDepth][MT];
#pragma unroll
  for (int u = 0; u < kDepth; ++u)
#pragma unroll
    for (int i = 0; i < MT; ++i)
      ring[u][i] = A[i][u * 32];
  // operand values one step ahead, their offsets two (the table has two steps of zeros at its end)
  float next[NTL][2];
  uint2 k = K[0];
#pragma unroll
  for (int j = 0; j < NTL; ++j)
    next[j][0] = lds(base[j] + k.x), next[j][1] = lds(base[j] + k.y);
  k = K[4];
  for (int s = 0; s < t.ks; s += kDepth)
  {
#pragma unroll
    for (int i = 0; i < MT; ++i)
      A[i] += kDepth * 32;
#pragma unroll
    for (int u = 0; u < kDepth; ++u)
    {
      uint32_t bh[NTL][2], bl[NTL][2];
#pragma unroll
      for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int h = 0; h < 2; ++h)
        {
          bh[j][h] = __float_as_uint(next[j][h]);
          bl[j][h] = tf32_rest(next[j][h]);
        }
#pragma unroll
      for (int j = 0; j < NTL; ++j)
        next[j][0] = lds(base[j] + k.x), next[j][1] = lds(base[j] + k.y);
      k = K[4 * u + 8];
      float4 lo[MT];
#pragma unroll
      for (int i = 0; i < MT; ++i)
      {
        const float4 h = ring[u][i];
        lo[i] = make_float4(__uint_as_float(tf32_rest(h.x)), __uint_as_float(tf32_rest(h.y)),
                            __uint_as_float(tf32_rest(h.z)), __uint_as_float(tf32_rest(h.w)));
      }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NTL; ++j)
        {
          mma8(cor[i][j], ring[u][i], bl[j][0], bl[j][1]);
          mma8(acc[i][j], ring[u][i], bh[j][0], bh[j][1]);
        }
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NTL; ++j)
          mma8(cor[i][j], lo[i], bh[j][0], bh[j][1]);
#pragma unroll
      for (int i = 0; i < MT; ++i)
        ring[u][i] = A[i][u * 32];
    }
    K += 4 * kDepth;
  }
#pragma unroll
  for (int i = 0; i < MT; ++i)
#pragma unroll
    for (int j = 0; j < NTL; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q)
        acc[i][j][q] += cor[i][j][q];
}

// Activation and derivative of N values with one dispatch.
template <int N>
__device__ __forceinline__ void act_rows(int act, const float (&z)[N], float (&f)[N], float (&d)[N])
{
#define DPC_ACT_ROWS(A)                                                                           \
  case A:                                                                                         \
    _Pragma("unroll") for (int j = 0; j < N; ++j) act_both(A, z[j], f[j], d[j]);                  \
    break;
  switch (act)
  {
    DPC_ACT_ROWS(DPC_ACT_RELU)
    DPC_ACT_ROWS(DPC_ACT_GELU)
    DPC_ACT_ROWS(DPC_ACT_SIGMOID)
    DPC_ACT_ROWS(DPC_ACT_ESIGMOID)
    DPC_ACT_ROWS(DPC_ACT_TANH)
    DPC_ACT_ROWS(DPC_ACT_HARD_TANH)
  default:
#pragma unroll
    for (int j = 0; j < N; ++j)
      f[j] = z[j], d[j] = 1.0f;
  }
#undef DPC_ACT_ROWS
}

__global__ void __launch_bounds__(kThreads, 1) conv_resident_kernel(const RcParams P)
{
  extern __shared__ __align__(16) float sm[];
  __shared__ RcLayer rl[kMaxLayers];
  __shared__ float s_ir[kMaxLayers + 1];
  __shared__ int s_act[kMaxLayers];
  __shared__ float red[kWarps];
  __shared__ int next_task[2];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nw = P.nw;
  float* mu0 = sm + P.mu0;
  const unsigned short* T = reinterpret_cast<const unsigned short*>(sm + P.tab_at);
  const uint2* koff = reinterpret_cast<const uint2*>(sm + P.koff_at);
  const RcTask* tasks = reinterpret_cast<const RcTask*>(sm + P.task_at);
  const unsigned short* order = reinterpret_cast<const unsigned short*>(sm + P.order_at);
  float* bias = sm + P.bias_at;

  for (int i = tid; i < P.table_vecs; i += kThreads)
    reinterpret_cast<int4*>(sm + P.tab_at)[i] = __ldg(reinterpret_cast<const int4*>(P.table) + i);
  for (int i = tid; i < P.koff_vecs; i += kThreads)
    reinterpret_cast<int4*>(sm + P.koff_at)[i] = __ldg(reinterpret_cast<const int4*>(P.koff) + i);
  for (int i = tid; i < 2 * (P.nf + P.nb); i += kThreads)
    reinterpret_cast<int4*>(sm + P.task_at)[i] = __ldg(reinterpret_cast<const int4*>(P.tasks) + i);
  for (int i = tid; i < P.nf + P.nb; i += kThreads)
    reinterpret_cast<unsigned short*>(sm + P.order_at)[i] = __ldg(P.order + i);
  for (int l = tid; l <= nw; l += kThreads)
  {
    if (l < nw)
    {
      rl[l] = P.rl[l];
      s_act[l] = P.layers[l].act;
    }
    s_ir[l] = P.layers[l].ir;
  }
  if (tid < 2)
    next_task[tid] = 0;
  __syncthreads();
  for (int l = 0; l < nw; ++l)
    for (int i = tid; i < rl[l].O; i += kThreads)
      bias[rl[l].boff + i] = P.layers[l].b[i];
  double esum = 0.0;

  for (int img = blockIdx.x; img < P.batch; img += gridDim.x)
  {
    __syncthreads();
    for (int i = tid; i < P.zfloats; i += kThreads)
      sm[i] = 0.0f;
    bool pred = false; // this forward pass stores predictions in global memory
    int mode = 0;      // what a finished forward sum does: 0 errors, 1 sweep, 2 the input layer
    // ------------------------------------------------------------ finishing of single values
    auto finish_forward = [&](int l, int m, int p, float sum, float& local)
    {
      const RcLayer& L = rl[l];
      const float pre = sum + bias[L.boff + m];
      float mu, d;
      act_both(s_act[l], pre, mu, d);
      if (pred)
      {
        const size_t o = ((size_t)img * L.O + m) * L.P + p;
        P.layers[l].preact[o] = pre;
        P.layers[l].mu[o] = mu;
      }
      float* zu = sm + L.uoff + m * L.uplane + T[L.upix + p];
      if (mode == 2)
        mu0[m * L.P + p] = mu;
      else if (mode == 1)
        *zu = mu;
      else
      {
        const float e = *zu - mu;
        sm[L.eoff + m * L.P + p] = e;
        sm[L.goff + m * L.gplane + T[L.gpix + p]] = e * d;
        local += e * e;
      }
    };
    auto finish_state = [&](int l, int m, int q, float dz)
    {
      const RcLayer& L = rl[l];
      float* z = sm + L.zoff + m * L.zplane + T[L.zpix + q];
      const float zv = *z;
      const float e = l == 1 ? zv - mu0[m * L.HW + q] : sm[rl[l - 1].eoff + m * L.HW + q];
      *z = zv + s_ir[l] * (dz - e);
    };
    auto run_tile = [&](const RcTask& t, auto shape, float& local)
    {
      constexpr int MT = decltype(shape)::value / 8, NTL = decltype(shape)::value % 8;
      float acc[MT][NTL][4];
      mma_tile<MT, NTL>(acc, t, P.packed, T, koff, sm, lane);
      // Addresses are worked out once per pixel and shared by the rows of the lane; the activation is
      // dispatched once per pixel.  (One call per element took half the kernel's instructions.)
      const int l = t.what >> 2, g = lane >> 2, c = lane & 3;
      const RcLayer& L = rl[l];
      constexpr int ROWS = 2 * MT; // rows m0 + g + 8 r
      if ((t.what & 3) == OP_STATE)
      {
        const float* err = sm + (l == 1 ? P.mu0 : rl[l - 1].eoff);
        const float ir = s_ir[l];
#pragma unroll
        for (int j = 0; j < NTL; ++j)
#pragma unroll
          for (int b = 0; b < 2; ++b)
          {
            const int n = 8 * j + 2 * c + b;
            if (n >= t.count)
              continue;
            const int q = T[t.ntab + 2 * n + 1];
            float* z = sm + L.zoff + T[L.zpix + q] + (t.m0 + g) * L.zplane;
            const float* e = err + q + (t.m0 + g) * L.HW;
#pragma unroll
            for (int r = 0; r < ROWS; ++r)
              if (t.m0 + g + 8 * r < L.C)
              {
                const float zv = z[8 * r * L.zplane], ev = e[8 * r * L.HW];
                z[8 * r * L.zplane] = zv + ir * (acc[r >> 1][j][2 * (r & 1) + b] - (l == 1 ? zv - ev : ev));
              }
          }
        return;
      }
#pragma unroll
      for (int j = 0; j < NTL; ++j)
#pragma unroll
        for (int b = 0; b < 2; ++b)
        {
          const int n = 8 * j + 2 * c + b;
          if (n >= t.count)
            continue;
          const int p = T[t.ntab + 2 * n + 1];
          float pre[ROWS], mu[ROWS], d[ROWS];
#pragma unroll
          for (int r = 0; r < ROWS; ++r)
            pre[r] = acc[r >> 1][j][2 * (r & 1) + b] + bias[L.boff + min(t.m0 + g + 8 * r, L.O - 1)];
          act_rows<ROWS>(s_act[l], pre, mu, d);
          float* zu = sm + L.uoff + T[L.upix + p];
          float* gz = sm + L.goff + (l > 0 ? T[L.gpix + p] : 0);
#pragma unroll
          for (int r = 0; r < ROWS; ++r)
          {
            const int m = t.m0 + g + 8 * r;
            if (m >= L.O)
              continue;
            if (pred)
            {
              const size_t o = ((size_t)img * L.O + m) * L.P + p;
              P.layers[l].preact[o] = pre[r];
              P.layers[l].mu[o] = mu[r];
            }
            if (mode == 2)
              mu0[m * L.P + p] = mu[r];
            else if (mode == 1)
              zu[m * L.uplane] = mu[r];
            else
            {
              const float e = zu[m * L.uplane] - mu[r];
              sm[L.eoff + m * L.P + p] = e;
              gz[m * L.gplane] = e * d[r];
              local += e * e;
            }
          }
        }
    };
    auto run_task = [&](const RcTask& t, float& local)
    {
      const int l = t.what >> 2;
      switch (t.what & 3)
      {
      case OP_DENSE_FORWARD:
      {
        const RcLayer& L = rl[l];
        const int K = L.C * L.HW;
        const float* W = P.layers[l].W + (size_t)t.m0 * K;
        const float* z = sm + L.zoff;
        float s = 0.0f;
        if (L.vec)
        {
#pragma unroll 4
          for (int k = lane * 4; k < K; k += 128)
          {
            const float4 w = *reinterpret_cast<const float4*>(W + k);
            const float4 v = *reinterpret_cast<const float4*>(z + k);
            s = fmaf(v.x, w.x, s), s = fmaf(v.y, w.y, s);
            s = fmaf(v.z, w.z, s), s = fmaf(v.w, w.w, s);
          }
        }
        else
#pragma unroll 4
          for (int k = lane; k < K; k += 32)
            s = fmaf(z[k], W[k], s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0)
          finish_forward(l, t.m0, 0, s, local);
        break;
      }
      case OP_DENSE_STATE:
      {
        const RcLayer& L = rl[l];
        const int K = L.C * L.HW;
        for (int r = t.m0 + lane; r < t.m0 + t.count; r += 32)
        {
          float dz = 0.0f;
#pragma unroll 8
          for (int o = 0; o < L.O; ++o)
            dz = fmaf(sm[L.goff + o * L.gplane], P.layers[l].W[(size_t)o * K + r], dz);
          const int m = r / L.HW;
          finish_state(l, m, r - m * L.HW, dz);
        }
        break;
      }
      default:
        switch (t.shape)
        {
        case 18:
          run_tile(t, std::integral_constant<int, 18>(), local);
          break;
        case 17:
          run_tile(t, std::integral_constant<int, 17>(), local);
          break;
        case 12:
          run_tile(t, std::integral_constant<int, 12>(), local);
          break;
        case 10:
          run_tile(t, std::integral_constant<int, 10>(), local);
          break;
        default:
          run_tile(t, std::integral_constant<int, 9>(), local);
        }
      }
    };
    // Tasks [first, first + count) of the cost-ordered list go to whichever warp is free.
    auto run_list = [&](int slot, int first, int count, float& local)
    {
      for (;;)
      {
        int q = 0;
        if (lane == 0)
          q = atomicAdd(&next_task[slot], 1);
        q = __shfl_sync(0xffffffffu, q, 0);
        if (q >= count)
          break;
        run_task(tasks[order[first + q]], local);
      }
    };
    // Layer 1's error against the cached prediction of the clamped image; global: it and the first
    // layer's gated error go to memory (nothing on the chip reads them).
    auto first_error = [&](bool store, float& local)
    {
      const RcLayer& L = rl[0];
      for (int i = tid; i < L.O * L.P; i += kThreads)
      {
        const int m = i / L.P, p = i - m * L.P;
        const float e = sm[L.uoff + m * L.uplane + T[L.upix + p]] - mu0[i];
        local += e * e;
        if (store)
        {
          const size_t o = (size_t)img * L.O * L.P + i;
          P.layers[1].e[o] = e;
          P.layers[0].g[o] = e * act_deriv(s_act[0], P.layers[0].preact[o]);
        }
      }
    };

    // ------------------------------------------------------------ the clamped image
    if (P.ops & DPC_ROWS_FIRST)
    {
      for (int i = tid; i < P.xfloats; i += kThreads)
        sm[P.xoff + i] = 0.0f;
      __syncthreads();
      const RcLayer& L = rl[0];
      const float* x = P.layers[0].z + (size_t)img * L.C * L.HW;
      for (int i = tid; i < L.C * L.HW; i += kThreads)
      {
        const int c = i / L.HW, p = i - c * L.HW;
        sm[L.zoff + c * L.zplane + T[L.zpix + p]] = x[i];
      }
      __syncthreads();
      mode = 2, pred = true;
      float none = 0.0f;
      for (int t = L.ffirst + warp; t < L.ffirst + L.fcount; t += kWarps)
        run_task(tasks[t], none);
      mode = 0, pred = false;
      __syncthreads();
    }
    else
    {
      for (int i = tid; i < rl[0].O * rl[0].P; i += kThreads)
        mu0[i] = P.layers[0].mu[(size_t)img * rl[0].O * rl[0].P + i];
      __syncthreads(); // the belief planes are clear before the loop below fills them
    }
    // errors and gated errors (their borders stay zero); the image shared their memory
    for (int i = tid; i < P.gfloat; i += kThreads)
      sm[P.efloat + i] = 0.0f;
    for (int l = 0; l < nw; ++l)
    {
      const RcLayer& L = rl[l];
      const bool load = l + 1 == nw ? (P.top_clamped || !(P.ops & (DPC_ROWS_SWEEP | DPC_ROWS_ZERO_Z)))
                                    : !(P.ops & (DPC_ROWS_SWEEP | DPC_ROWS_ZERO_Z));
      if (!load)
        continue;
      const float* z = P.layers[l + 1].z + (size_t)img * L.O * L.P;
      for (int i = tid; i < L.O * L.P; i += kThreads)
      {
        const int m = i / L.P, p = i - m * L.P;
        sm[L.uoff + m * L.uplane + T[L.upix + p]] = z[i];
      }
    }
    __syncthreads();

    // ------------------------------------------------------------ projection
    if (P.ops & DPC_ROWS_SWEEP)
    {
      pred = (P.ops & DPC_ROWS_SWEEP_PRED) != 0;
      mode = 1;
      float none = 0.0f;
      for (int l = 0; l < nw; ++l)
      {
        const RcLayer& L = rl[l];
        const bool copy = !(l + 1 == nw && P.top_clamped);
        if (!copy)
          break;
        if (l == 0)
          for (int i = tid; i < L.O * L.P; i += kThreads)
          {
            const int m = i / L.P, p = i - m * L.P;
            sm[L.uoff + m * L.uplane + T[L.upix + p]] = mu0[i];
          }
        else
          for (int t = L.ffirst + warp; t < L.ffirst + L.fcount; t += kWarps)
            run_task(tasks[t], none);
        __syncthreads();
      }
      mode = 0, pred = false;
    }
    // ------------------------------------------------------------ settling and the closing energy
    const bool closing = (P.ops & DPC_ROWS_ENERGY_LAST) != 0;
    for (int t = 0; t < P.steps + (closing ? 1 : 0); ++t)
    {
      const bool energy = t == P.steps, last = energy || (!closing && t + 1 == P.steps);
      pred = energy ? (P.ops & DPC_ROWS_PRED_CLOSE) != 0 : last && (P.ops & DPC_ROWS_PRED_LAST) != 0;
      float local = 0.0f;
      const int f1 = rl[0].fcount; // the input layer's tasks come first in the list
      run_list(0, f1, P.nf - f1, local);
      if (last)
        first_error(true, local);
      if (energy)
      {
        esum += (double)local;
        break;
      }
      __syncthreads();
      if (tid == 0)
        next_task[0] = 0;
      run_list(1, P.nf, P.nb, local);
      if (!P.top_clamped)
      {
        const RcLayer& L = rl[nw - 1];
        for (int i = tid; i < L.O * L.P; i += kThreads)
        {
          const int m = i / L.P, p = i - m * L.P;
          float* z = sm + L.uoff + m * L.uplane + T[L.upix + p];
          *z -= s_ir[nw] * (nw == 1 ? *z - mu0[i] : sm[L.eoff + i]);
        }
      }
      __syncthreads();
      if (tid == 0)
        next_task[1] = 0;
    }
    __syncthreads();
    if (tid < 2)
      next_task[tid] = 0;
    // ------------------------------------------------------------ back to memory
    const bool passes = P.steps > 0 || closing;
    for (int l = 0; l < nw; ++l)
    {
      const RcLayer& L = rl[l];
      const size_t o = (size_t)img * L.O * L.P;
      const bool st_z = (P.ops & DPC_ROWS_STORE_Z) && !(l + 1 == nw && P.top_clamped);
      for (int i = tid; i < L.O * L.P; i += kThreads)
      {
        const int m = i / L.P, p = i - m * L.P;
        if (st_z)
          P.layers[l + 1].z[o + i] = sm[L.uoff + m * L.uplane + T[L.upix + p]];
        if (passes && l > 0)
        {
          P.layers[l + 1].e[o + i] = sm[L.eoff + i];
          P.layers[l].g[o + i] = sm[L.goff + m * L.gplane + T[L.gpix + p]];
        }
      }
    }
    if (passes)
    {
      float* e0 = P.layers[0].e + (size_t)img * rl[0].C * rl[0].HW;
      for (int i = tid; i < rl[0].C * rl[0].HW; i += kThreads)
        e0[i] = 0.0f;
    }
  }
  if (P.ops & DPC_ROWS_ENERGY_LAST)
  {
    float s = (float)esum;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0)
      red[warp] = s;
    __syncthreads();
    if (tid == 0)
    {
      double t = 0.0;
      for (int w = 0; w < kWarps; ++w)
        t += (double)red[w];
      atomicAdd(P.energy, 0.5 * t);
    }
  }
}

// Weights of one (layer, role, class) into fragment order: block = (group, 16-row block).
__global__ void conv_pack_kernel(const dpc_conv_layer* __restrict__ layers, const RcPack* __restrict__ packs,
                                 const int* __restrict__ aoff, float4* __restrict__ out)
{
  const RcPack G = packs[blockIdx.y];
  if ((int)blockIdx.x >= G.mblocks)
    return;
  const float* W = layers[G.layer].W;
  float4* dst = out + G.w + (size_t)blockIdx.x * G.ks * 32;
  for (int i = threadIdx.x + blockIdx.z * blockDim.x; i < G.ks * 32; i += blockDim.x * gridDim.z)
  {
    const int s = i >> 5, lane = i & 31, m = blockIdx.x * 16 + (lane >> 2), k = 8 * s + (lane & 3);
    const int a0 = aoff[G.aoff + k], a1 = aoff[G.aoff + k + 4];
    float v[4];
    v[0] = a0 >= 0 && m < G.M ? W[a0 + m * G.mstride] : 0.0f;
    v[1] = a0 >= 0 && m + 8 < G.M ? W[a0 + (m + 8) * G.mstride] : 0.0f;
    v[2] = a1 >= 0 && m < G.M ? W[a1 + m * G.mstride] : 0.0f;
    v[3] = a1 >= 0 && m + 8 < G.M ? W[a1 + (m + 8) * G.mstride] : 0.0f;
    dst[i] = make_float4(v[0], v[1], v[2], v[3]);
  }
}

struct ResState
{
  RcParams P = {};
  size_t smem = 0;
  void* dev = nullptr;
  float4* packed = nullptr;
  RcPack* packs = nullptr;
  int* aoff = nullptr;
  int n_packs = 0, max_mblocks = 0;
};

inline int up4(int v)
{
  return (v + 3) & ~3;
}
inline int cdiv(int a, int b)
{
  return (a + b - 1) / b;
}

struct Builder
{
  std::vector<RcLayer> rl;
  std::vector<RcTask> ft, bt;
  std::vector<unsigned short> table;
  std::vector<uint2> koffs;
  std::vector<RcPack> packs;
  std::vector<int> aoff;
  size_t packed = 0; // float4s
  bool ok = true;

  int put(long long v)
  {
    if (v < 0 || v > 65535)
      ok = false;
    table.push_back((unsigned short)v);
    return (int)table.size() - 1;
  }
  // Weights of one product: K source offsets in k order, rows mstride apart.
  int add_pack(int layer, int M, int mstride, const std::vector<int>& src)
  {
    RcPack g = {};
    g.layer = layer, g.M = M, g.mstride = mstride;
    g.ks = cdiv((int)src.size(), 8 * kDepth) * kDepth, g.mblocks = M > 16 ? 2 * cdiv(M, 32) : 1;
    g.w = (int)packed, g.aoff = (int)aoff.size();
    packed += (size_t)g.mblocks * g.ks * 32;
    aoff.insert(aoff.end(), src.begin(), src.end());
    aoff.resize(g.aoff + 8 * (size_t)g.ks, -1);
    packs.push_back(g);
    return (int)packs.size() - 1;
  }
  // Tiles of one product.  koff, pixels (base, index): operand addresses.
  void add_tiles(std::vector<RcTask>& list, int what, int pack, const std::vector<long long>& koff,
                 const std::vector<std::pair<long long, int>>& pixels, int want)
  {
    const RcPack g = packs[pack];
    const int ktab = (int)koffs.size();
    auto offset = [&](int k) { return k < (int)koff.size() ? (unsigned)(4 * koff[k]) : 0u; };
    for (int s = 0; s < g.ks + 2; ++s)
      for (int c = 0; c < 4; ++c)
        koffs.push_back(make_uint2(offset(8 * s + c), offset(8 * s + c + 4)));
    const int ntab = (int)table.size();
    for (const auto& p : pixels)
      put(p.first), put(p.second);
    // the widest tiles that still leave `want` tasks: per step a 32 x 16 tile reads and splits a third
    // of what three 16 x 8 tiles do per product
    const int count = (int)pixels.size();
    const int shapes[5] = {18, 12, 17, 10, 9};
    int shape = 9;
    for (int q : shapes)
      if ((q < 16 || g.M > 16) && 8 * (q % 8) < count + 8 &&
          cdiv(g.M, 16 * (q / 8)) * cdiv(count, 8 * (q % 8)) >= want)
      {
        shape = q;
        break;
      }
    if (g.M > 16 && shape < 16 && shape != 12)
      shape = cdiv(g.M, 32) * cdiv(count, 8) * 2 >= want ? 17 : shape;
    const int mt = shape / 8, ntl = shape % 8;
    for (int m = 0; m < g.M; m += 16 * mt)
      for (int n = 0; n < count; n += 8 * ntl)
      {
        RcTask t = {};
        t.w = g.w + m / 16 * g.ks * 32, t.ks = g.ks;
        t.ktab = ktab, t.ntab = ntab + 2 * n;
        t.m0 = m, t.count = std::min(8 * ntl, count - n);
        t.shape = shape, t.what = what;
        list.push_back(t);
      }
  }
};
} // namespace
} // namespace conv

using namespace conv;

void conv_res_free(dpc_conv_plan* p)
{
  auto* s = static_cast<ResState*>(p->res);
  if (!s)
    return;
  cudaFree(s->dev);
  cudaFree(s->packed);
  delete s;
  p->res = nullptr;
}

int conv_res_init(dpc_conv_plan* p)
{
  p->res = nullptr;
  if (getenv("DPC_DISABLE_RESIDENT"))
    return 1;
  const int nw = p->n - 1;
  if (nw > kMaxLayers)
    return 1;
  Builder B;
  B.rl.resize(nw);
  size_t weights = 0, shared = 0;
  std::vector<int> low_y(nw + 1, 0), low_x(nw + 1, 0), zpitch(nw + 1), zrows(nw + 1);
  std::vector<int> glow_y(nw, 0), glow_x(nw, 0), gpitch(nw, 0), grows(nw, 0);
  auto dense = [&](int l)
  {
    const dpc_conv_layer& L = p->h[l];
    return L.out_h == 1 && L.out_w == 1 && L.p_h == 0 && L.p_w == 0 && L.k_h == L.in_h && L.k_w == L.in_w;
  };
  // ---- planes with borders
  for (int l = 0; l <= nw; ++l)
  {
    const dpc_conv_layer& L = p->h[l];
    zpitch[l] = L.in_w, zrows[l] = L.in_h;
    if (l == nw || dense(l))
      continue;
    low_y[l] = L.p_h, low_x[l] = L.p_w;
    zrows[l] = std::max(L.in_h + L.p_h, (L.out_h - 1) * L.s_h + L.k_h);
    zpitch[l] = std::max(L.in_w + L.p_w, (L.out_w - 1) * L.s_w + L.k_w);
    if (l == 0)
      continue;
    // gated errors: every tap of every input pixel, (y + p - ky) / s, must fall into the plane
    auto extent = [](int in, int pad, int k, int s, int out, int& low, int& size)
    {
      int lo = 0, hi = out - 1;
      for (int y = 0; y < in; ++y)
      {
        const int r = (y + pad) % s, n = r < k ? (k - r + s - 1) / s : 0, q = (y + pad - r) / s;
        if (n > 0)
          lo = std::min(lo, q - (n - 1)), hi = std::max(hi, q);
      }
      low = -lo, size = hi - lo + 1;
    };
    extent(L.in_h, L.p_h, L.k_h, L.s_h, L.out_h, glow_y[l], grows[l]);
    extent(L.in_w, L.p_w, L.k_w, L.s_w, L.out_w, glow_x[l], gpitch[l]);
  }
  // ---- shared memory: Z of layers 1.. | mu0 | E, G (before them: the padded image) | tables
  RcParams P = {};
  size_t at = 0;
  std::vector<size_t> zoff(nw + 1);
  for (int l = 1; l <= nw; ++l)
  {
    zoff[l] = at;
    at += up4(p->h[l].in_c * zrows[l] * zpitch[l]);
  }
  P.zfloats = (int)at;
  P.mu0 = (int)at;
  at += up4(p->h[0].out_c * p->h[0].out_h * p->h[0].out_w);
  P.efloat = P.xoff = (int)at;
  zoff[0] = at;
  P.xfloats = up4(p->h[0].in_c * zrows[0] * zpitch[0]);
  size_t eg = at;
  for (int l = 0; l < nw; ++l)
  {
    const dpc_conv_layer& L = p->h[l];
    RcLayer& q = B.rl[l];
    q.C = L.in_c, q.HW = L.in_h * L.in_w, q.O = L.out_c, q.P = L.out_h * L.out_w;
    const size_t bytes = sizeof(float) * (size_t)L.out_c * L.in_c * L.k_h * L.k_w;
    weights += bytes;
    q.dense = dense(l);
    if (l > 0 && !q.dense)
      shared += bytes;
    q.vec = (q.C * q.HW) % 4 == 0 && (reinterpret_cast<uintptr_t>(L.W) & 15) == 0;
    if (q.dense && l > 0)
      gpitch[l] = grows[l] = 1;
    if (l > 0)
    {
      q.eoff = (int)eg;
      eg += up4(q.O * q.P);
      q.gplane = grows[l] * gpitch[l];
      q.goff = (int)eg;
      eg += up4(q.O * q.gplane);
    }
    q.boff = P.bias_n;
    P.bias_n += q.O;
  }
  P.gfloat = (int)(eg - at);
  at = std::max(eg, at + (size_t)P.xfloats);
  // A block reads the weights of every layer above the first from L2 in each pass, whatever the batch, where
  // the phase kernels share them between images and split them over the SMs.  Segments / phase kernels,
  // geometric means over random networks (8 to 28 pixels a side, 3 to 10 passes) by KB of weights in
  // the layers between the first and the dense heads:
  //            <= 100    100-200   200-300   300-450   450-1200  1200-4000
  //   1-4      0.52      0.80      0.77      1.35      1.78      1.79      images
  //   6-12     0.44      0.86      1.09      1.01      1.36      -
  //   16-64    0.27      0.58      0.56      0.72      0.60      0.96
  // (109-109-109 channels of 3x3 taps on 12x12 pixels, 8 images: 487/250 us, 411 before there were segments.)
  // A single image pays for its heads too: 87 channels on 8x8 pixels and 37 outputs, 805 KB, 340/291 us.
  // All weights together, at 128 images: 0-4 MB 0.35, 4-6 MB 0.34, 6-10 MB 0.54; at 32-64 images 0.61, 0.63, 1.05.
  const size_t first = sizeof(float) * (size_t)p->h[0].out_c * p->h[0].in_c * p->h[0].k_h * p->h[0].k_w;
  if (at * sizeof(float) > kSmemLimit || weights > (4u << 20) || (shared > 300 * 1024 && p->batch <= 12) ||
      (weights - first > 768 * 1024 && p->batch == 1))
    return 1;
  // ---- pixel tables
  auto plane_table = [&](int h, int w, int pitch, int ly, int lx)
  {
    const int first = (int)B.table.size();
    for (int y = 0; y < h; ++y)
      for (int x = 0; x < w; ++x)
        B.put((y + ly) * pitch + x + lx);
    return first;
  };
  std::vector<int> zpix(nw + 1);
  for (int l = 0; l <= nw; ++l)
    zpix[l] = plane_table(p->h[l].in_h, p->h[l].in_w, zpitch[l], low_y[l], low_x[l]);
  for (int l = 0; l < nw; ++l)
  {
    RcLayer& q = B.rl[l];
    q.zoff = (int)zoff[l], q.zplane = zrows[l] * zpitch[l], q.zpix = zpix[l];
    q.uoff = (int)zoff[l + 1], q.uplane = zrows[l + 1] * zpitch[l + 1], q.upix = zpix[l + 1];
    if (l > 0)
      q.gpix = plane_table(p->h[l].out_h, p->h[l].out_w, gpitch[l], glow_y[l], glow_x[l]);
  }
  // ---- tasks
  for (int l = 0; l < nw; ++l)
  {
    const dpc_conv_layer& L = p->h[l];
    RcLayer& q = B.rl[l];
    const int kk = L.k_h * L.k_w, rows = L.in_c * kk;
    q.ffirst = (int)B.ft.size();
    if (q.dense)
      for (int o = 0; o < q.O; ++o)
      {
        RcTask t = {};
        t.m0 = o, t.count = 1, t.ks = rows / 16, t.shape = 9, t.what = l << 2 | OP_DENSE_FORWARD;
        B.ft.push_back(t);
      }
    else
    {
      std::vector<int> src(rows);
      std::vector<long long> koff(rows);
      for (int c = 0, k = 0; c < L.in_c; ++c)
        for (int y = 0; y < L.k_h; ++y)
          for (int x = 0; x < L.k_w; ++x, ++k)
            src[k] = k, koff[k] = c * q.zplane + y * zpitch[l] + x;
      std::vector<std::pair<long long, int>> px;
      for (int y = 0; y < L.out_h; ++y)
        for (int x = 0; x < L.out_w; ++x)
          px.push_back({(long long)q.zoff + y * L.s_h * zpitch[l] + x * L.s_w, y * L.out_w + x});
      B.add_tiles(B.ft, l << 2 | OP_FORWARD, B.add_pack(l, q.O, rows, src), koff, px, kWarps);
    }
    q.fcount = (int)B.ft.size() - q.ffirst;
    if (l == 0)
      continue;
    if (q.dense)
    {
      for (int r = 0; r < rows; r += 128)
      {
        RcTask t = {};
        t.m0 = r, t.count = std::min(128, rows - r), t.ks = q.O / 2, t.shape = 9;
        t.what = l << 2 | OP_DENSE_STATE;
        B.bt.push_back(t);
      }
      continue;
    }
    const int classes = std::min(L.s_h, L.in_h) * std::min(L.s_w, L.in_w);
    for (int ry = 0; ry < L.s_h; ++ry)
      for (int rx = 0; rx < L.s_w; ++rx)
      {
        const int ny = ry < L.k_h ? cdiv(L.k_h - ry, L.s_h) : 0, nx = rx < L.k_w ? cdiv(L.k_w - rx, L.s_w) : 0;
        std::vector<std::pair<long long, int>> px;
        for (int y = 0; y < L.in_h; ++y)
          for (int x = 0; x < L.in_w; ++x)
            if ((y + L.p_h) % L.s_h == ry && (x + L.p_w) % L.s_w == rx)
            {
              const int qy = (y + L.p_h - ry) / L.s_h, qx = (x + L.p_w - rx) / L.s_w;
              const bool taps = ny > 0 && nx > 0;
              px.push_back({taps ? (long long)q.goff + (qy - (ny - 1) + glow_y[l]) * gpitch[l] + qx -
                                       (nx - 1) + glow_x[l]
                                 : q.goff,
                            y * L.in_w + x});
            }
        if (px.empty())
          continue;
        std::vector<int> src;
        std::vector<long long> koff;
        for (int j = 0; j < ny; ++j)
          for (int i = 0; i < nx; ++i)
            for (int o = 0; o < q.O; ++o)
            {
              src.push_back(o * rows + (ry + L.s_h * j) * L.k_w + rx + L.s_w * i);
              koff.push_back((long long)o * q.gplane + (ny - 1 - j) * gpitch[l] + nx - 1 - i);
            }
        B.add_tiles(B.bt, l << 2 | OP_STATE, B.add_pack(l, q.C, kk, src), koff, px,
                    std::max(2, kWarps / classes));
      }
  }
  if (!B.ok || B.ft.size() + B.bt.size() > 4096)
    return 1;
  // longest tasks first within each list (the input layer's stay in front)
  std::vector<unsigned short> order(B.ft.size() + B.bt.size());
  std::vector<RcTask> tasks = B.ft;
  tasks.insert(tasks.end(), B.bt.begin(), B.bt.end());
  for (size_t i = 0; i < order.size(); ++i)
    order[i] = (unsigned short)i;
  auto longer = [&](unsigned short a, unsigned short b)
  {
    auto cost = [](const RcTask& t) { return t.ks * ((t.shape / 8) * (t.shape % 8) * 3 + 2); };
    return cost(tasks[a]) > cost(tasks[b]);
  };
  std::stable_sort(order.begin() + B.rl[0].fcount, order.begin() + B.ft.size(), longer);
  std::stable_sort(order.begin() + B.ft.size(), order.end(), longer);
  while (B.table.size() % 8)
    B.table.push_back(0);
  order.resize((order.size() + 7) & ~(size_t)7);
  P.tab_at = (int)at;
  at += B.table.size() / 2;
  while (B.koffs.size() % 2)
    B.koffs.push_back(make_uint2(0, 0));
  P.koff_at = (int)at;
  at += 2 * B.koffs.size();
  P.task_at = (int)at;
  at += tasks.size() * (sizeof(RcTask) / 4);
  P.order_at = (int)at;
  at += order.size() / 2;
  P.bias_at = (int)at;
  at += up4(P.bias_n);
  if (at * sizeof(float) + kStatic > kSmemLimit)
    return 1;

  std::vector<unsigned char> host;
  auto put = [&](const void* src, size_t len)
  {
    const size_t here = host.size();
    host.resize((here + len + 15) & ~(size_t)15, 0);
    if (len)
      memcpy(host.data() + here, src, len);
    return here;
  };
  const size_t o_rl = put(B.rl.data(), sizeof(RcLayer) * nw), o_t = put(tasks.data(), sizeof(RcTask) * tasks.size());
  const size_t o_o = put(order.data(), 2 * order.size()), o_tab = put(B.table.data(), 2 * B.table.size());
  const size_t o_k = put(B.koffs.data(), sizeof(uint2) * B.koffs.size());
  const size_t o_p = put(B.packs.data(), sizeof(RcPack) * B.packs.size());
  const size_t o_a = put(B.aoff.data(), sizeof(int) * B.aoff.size());
  auto* st = new ResState();
  p->res = st;
  if (cudaMalloc(&st->dev, host.size()) != cudaSuccess ||
      cudaMalloc(&st->packed, (B.packed + 32 * kDepth) * sizeof(float4)) != cudaSuccess ||
      cudaMemcpyAsync(st->dev, host.data(), host.size(), cudaMemcpyHostToDevice, p->ctx->stream) != cudaSuccess)
  {
    conv_res_free(p);
    return cuda_fail(cudaGetLastError(), "image-resident plan tables");
  }
  auto* base = static_cast<unsigned char*>(st->dev);
  st->packs = reinterpret_cast<RcPack*>(base + o_p);
  st->aoff = reinterpret_cast<int*>(base + o_a);
  st->n_packs = (int)B.packs.size();
  for (const auto& g : B.packs)
    st->max_mblocks = std::max(st->max_mblocks, g.mblocks);
  P.layers = p->d;
  P.rl = reinterpret_cast<RcLayer*>(base + o_rl);
  P.tasks = reinterpret_cast<RcTask*>(base + o_t);
  P.order = reinterpret_cast<unsigned short*>(base + o_o);
  P.table = reinterpret_cast<unsigned short*>(base + o_tab);
  P.koff = reinterpret_cast<uint2*>(base + o_k);
  P.koff_vecs = (int)(B.koffs.size() / 2);
  P.packed = st->packed;
  P.nw = nw, P.batch = p->batch;
  P.nf = (int)B.ft.size(), P.nb = (int)B.bt.size();
  P.table_vecs = (int)(B.table.size() / 8);
  P.energy = p->energy;
  st->P = P;
  st->smem = at * sizeof(float);
  return DPC_OK;
}
} // namespace dpc

using namespace dpc;

int dpc_conv_images_available(dpc_conv_plan* p)
{
  return p && p->res ? 1 : 0;
}

int dpc_conv_images_segment(dpc_conv_plan* p, int ops, int steps, int top_clamped)
{
  if (!p || !p->res || steps < 0)
    return fail(DPC_ERR_INVALID, "dpc_conv_images_segment: not an image-resident plan, or a bad step count");
  auto* st = static_cast<conv::ResState*>(p->res);
  static thread_local int configured = -1;
  if (configured != p->ctx->device)
  {
    DPC_CUDA(cudaFuncSetAttribute(conv::conv_resident_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(conv::kSmemLimit - conv::kStatic)));
    configured = p->ctx->device;
  }
  cudaStream_t s = p->ctx->stream;
  if (st->n_packs > 0)
  {
    conv::conv_pack_kernel<<<dim3(st->max_mblocks, st->n_packs, 4), 256, 0, s>>>(p->d, st->packs, st->aoff,
                                                                             st->packed);
    p->ctx->launches += 1;
  }
  conv::RcParams P = st->P;
  P.ops = ops, P.steps = steps, P.top_clamped = top_clamped;
  conv::conv_resident_kernel<<<std::min(p->batch, p->ctx->sm_count), conv::kThreads, st->smem, s>>>(P);
  p->ctx->launches += 1;
  const cudaError_t err = cudaPeekAtLastError();
  return err == cudaSuccess ? DPC_OK : cuda_fail(cudaGetLastError(), "image-resident kernel");
}
