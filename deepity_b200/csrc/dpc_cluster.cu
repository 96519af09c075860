// Row segments on thread-block clusters.
//
// Between two weight updates a step is row-local (dpc_resident.cu).  There one block keeps a row group's state and as
// many weights as fit beside it; the others come from L2 on every pass, 1000 cycles per batch of loads along a sum that
// may be one chain.  Here a cluster of C blocks owns the rows and ALL weights stay in its shared memory: block r holds
// its share of every layer's output rows (for the predictions) and, once more, its share of the input columns (for the
// state updates), so a sum is formed whole, in one order, by the lane that finishes its element -- no partial sums in
// shared memory, no pass that adds them, two barriers a settling pass.  What the next phase of the other blocks reads
// (beliefs or f(z), gated errors or errors) is stored to all of them through distributed shared memory.
//
//   forward        lane = output and a slice of K: 16-byte reads of rows whose pitch is 4 x odd floats (no bank conflict)
//   state update   lane = input column and a slice of the output rows: neighbouring lanes read neighbouring floats
//   input layer    once a segment: its rows stream through the space that the weights take afterwards
//
// Sums are one ascending chain where ordered_sums() asks for it (slices: 1 lane an output), else up to four lanes share
// an output.  The same tasks serve the sweep and every pass: a belief that the sweep produced has an error of exactly
// zero in the passes that follow.
//
// What bounds a pass: the longest chain, which takes 30 to 50 cycles for four multiply-adds of the 16 that these need, or
// reads of shared memory (6 cycles a quad of 32 outputs and one row); then two dependent elementwise stretches of 600
// cycles and two barriers (50 cycles, 250 to 700 of a cluster).  us a step, segments of single blocks / of clusters:
// 100-300-200-77-10, AdamW, ReLU, batch 50, T 6 180 / 130 (a pass 24 000 / 10 000 cycles), 784-222-222-10 at batch 73
// 224 / 114; phase kernels / clusters: 16-448-448-16, SimplePC, ReLU, batch 23, T 16 303 / 110, 345-345-345-10 prediction
// at batch 6 101 / 59.  With two outputs a lane (half the operand reads) the same step took 155, with three or four quads
// ahead 131.
#include <algorithm>
#include <array>
#include <atomic>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "dpc_internal.h"
#include "dpc_math.cuh"
#include "dpc_tcgen05.cuh"

namespace dpc
{
namespace
{
using namespace ptx; // shared-memory addresses and cluster barriers: dpc_tcgen05.cuh
constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kMaxLayers = 96;
constexpr size_t kSmemLimit = 227 * 1024, kStatic = 7 * 1024; // per block; of it static

struct SegLayer // one per weight layer and block of the cluster, built on the host
{
  int K, N;
  int zoff, noff;   // offsets of layers l and l+1 in a row's state (multiples of 4)
  int o0, o1;       // outputs of this block
  int c0, c1;       // input columns of this block (l > 0): its outputs of the layer below
  int fpitch, foff; // rows [o0, o1) of W in shared memory
  int bpitch, boff; // columns [c0, c1)
  int f0, f1;       // forward tasks of the layer alone (sweep, logits)
  int vec;          // rows of W in global memory can be read 16 bytes at a time
  int lanes_k;      // ordered networks, layer alone: lanes along K, the narrow heads' order of additions
};

enum
{
  T_DOT = 0,
  T_LANES = 1, // forward: lanes along K, one output after the other
  T_PLAIN = 2  // no sum: outputs of the input layer, whose prediction is cached; a last layer that relaxes
};
struct __align__(16) SegTask
{
  int w, x, first;              // first weight in shared memory; first operand element; state element of lane 0
  int other;                    // residual layers: the elements below (forward) or above (state), from `first`
  unsigned short pitch, len, slice; // pitch of the weights; elements to walk; elements per lane of an output
  short row0, layer, j0;        // first row; forward: the weights' layer, state: the elements' layer; lane 0's unit
  unsigned char units, lg, kind, pad; // outputs; log2 of the lanes that share one; T_*
};
static_assert(sizeof(SegTask) == 32 && sizeof(SegLayer) == 64, "copied 16 bytes at a time");

struct SegParams
{
  const dpc_layer* layers;
  // per block of the cluster: SegLayer[nw] | forward tasks (sorted by layer) | state tasks | layer of each quad (short)
  const int4* table;
  int table_vecs, a_ft, a_bt, a_lq; // size of a block's table in 16-byte units, byte offsets of its parts
  const int2* counts;               // tasks of each block: forward, state
  int n, batch, S, C;               // layers, rows, floats of a row's state (layers 1..n-1), blocks of a cluster
  int R, groups;                    // rows of a group, groups
  int N1p, K0p;                     // padded widths of layer 1 and of the input
  int region;                       // floats of shared memory for the weights
  int kc, rows0, lg0, slice0;       // input layer: columns of a step, rows of the widest block, lanes an output,
  int one_row0;                     // tasks of one row instead of RT
  int ops, steps;
  int simple, has_v, ce, one_block, top_clamped, top_down_off, top_n;
  double* energy;
};

struct SegConst // what a finished sum of layer l needs, one 16-byte read
{
  float a, ir, beta;
  int kind; // activation, | 256: residual
  __device__ __forceinline__ int act() const { return kind & 255; }
  __device__ __forceinline__ bool residual() const { return (kind & 256) != 0; }
};
struct SegPointers
{
  const float *W, *b;
  float *z, *e, *mu, *preact;
};

__device__ __forceinline__ void copy16(float* dst, const float* src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src)
{
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_commit()
{
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <int N>
__device__ __forceinline__ void copies_wait()
{
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

__device__ __forceinline__ float4 shared4(uint32_t p)
{
  float4 v;
  asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(p));
  return v;
}

// The operands of four steps of a lane's sums -- one output (or column) x RT rows -- and their multiply-adds.  A chain of
// them costs 16 cycles a quad as long as the operands are there: those of the next U quads are read before the
// multiply-adds of these U (288 elements of one warp, cycles a quad: 34 -> 20 with one row, 40 -> 26 with two, 71 -> 45
// with four).  With many warps the reads bound it: 4 cycles a quad of weights, 2 one of operands that all lanes share.
template <int RT>
struct Quad
{
  float w[4];
  float4 x[RT];
  __device__ __forceinline__ void row(uint32_t wp, uint32_t xp, int S, int k)
  {
    const float4 v = shared4(wp + 4 * k);
    w[0] = v.x, w[1] = v.y, w[2] = v.z, w[3] = v.w;
    operands(xp, S, k);
  }
  __device__ __forceinline__ void column(uint32_t wp, int pitch, uint32_t xp, int S, int n)
  {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      asm volatile("ld.shared.f32 %0, [%1];" : "=f"(w[j]) : "r"(wp + 4 * (n + j) * pitch));
    operands(xp, S, n);
  }
  __device__ __forceinline__ void operands(uint32_t xp, int S, int k)
  {
#pragma unroll
    for (int r = 0; r < RT; ++r)
      x[r] = shared4(xp + 4 * (r * S + k));
  }
  __device__ __forceinline__ void multiply(float (&acc)[RT]) const
  {
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int r = 0; r < RT; ++r)
        acc[r] = fmaf(j == 0 ? x[r].x : j == 1 ? x[r].y : j == 2 ? x[r].z : x[r].w, w[j], acc[r]);
  }
};
template <int RT>
constexpr int kAhead = RT <= 2 ? 2 : 1;

// acc += sum of `quads` quads that load(quad, first element) fetches
template <int RT, typename Load>
__device__ __forceinline__ void dot(float (&acc)[RT], int quads, Load load)
{
  constexpr int U = kAhead<RT>;
  Quad<RT> a[U], b[U];
  auto fetch = [&](Quad<RT> (&f)[U], int q)
  {
#pragma unroll
    for (int u = 0; u < U; ++u)
      load(f[u], 4 * (q + u));
  };
  auto multiply = [&](const Quad<RT> (&f)[U])
  {
#pragma unroll
    for (int u = 0; u < U; ++u)
      f[u].multiply(acc);
  };
  int q = 0;
  if (quads >= U)
  {
    fetch(a, 0);
#pragma unroll 1
    for (; q + 3 * U <= quads; q += 2 * U)
    {
      fetch(b, q + U);
      multiply(a);
      fetch(a, q + 2 * U);
      multiply(b);
    }
    if (q + 2 * U <= quads)
    {
      fetch(b, q + U);
      multiply(a);
      multiply(b);
      q += 2 * U;
    }
    else
    {
      multiply(a);
      q += U;
    }
  }
#pragma unroll 1
  for (; q < quads; ++q)
  {
    load(a[0], 4 * q);
    a[0].multiply(acc);
  }
}

// acc[r] += sum over len elements (a multiple of 4) of x[r][k] w[k]
template <int RT>
__device__ __forceinline__ void dot_row(float (&acc)[RT], const float* w, const float* x, int S, int len)
{
  dot<RT>(acc, len >> 2, [w = smem_u32(w), x = smem_u32(x), S](Quad<RT>& q, int k) { q.row(w, x, S, k); });
}

// acc[r] += sum over len rows of w of g[r][n] w[n][this column]
template <int RT>
__device__ __forceinline__ void dot_column(float (&acc)[RT], const float* w, int pitch, const float* g, int S, int len)
{
  dot<RT>(acc, len >> 2, [w = smem_u32(w), g = smem_u32(g), pitch, S](Quad<RT>& q, int n) { q.column(w, pitch, g, S, n); });
#pragma unroll 1
  for (int n = len & ~3; n < len; ++n)
#pragma unroll
    for (int r = 0; r < RT; ++r)
      acc[r] = fmaf(g[r * S + n], w[n * pitch], acc[r]);
}

// Sums of the 1 << lg lanes that share an output, in all of them.
template <int V>
__device__ __forceinline__ void add_slices(float (&acc)[V], int lg)
{
  for (int bit = 16; bit >= 32 >> lg; bit >>= 1)
#pragma unroll
    for (int v = 0; v < V; ++v)
      acc[v] += __shfl_xor_sync(0xffffffffu, acc[v], bit);
}

template <int RT>
__global__ void __launch_bounds__(kThreads, 1) cluster_rows_kernel(const SegParams P)
{
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(16) SegConst lc[kMaxLayers];
  __shared__ SegPointers ptr[kMaxLayers];
  __shared__ float red[kWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = P.S, R = P.R, nw = P.n - 1, C = P.C; // nw weight layers
  const int rank = C > 1 ? (int)cluster_ctarank() : 0;
  const bool simple = P.simple != 0;

  // ---- shared memory: weights | table | bias | Z E G(or f(z)) [V] | mu0 d0 | top mu, d
  float* Ws = sm;
  unsigned char* tab = reinterpret_cast<unsigned char*>(Ws + P.region);
  const SegLayer* sl = reinterpret_cast<const SegLayer*>(tab);
  const SegTask* ftab = reinterpret_cast<const SegTask*>(tab + P.a_ft);
  const SegTask* btab = reinterpret_cast<const SegTask*>(tab + P.a_bt);
  const short* layer_of = reinterpret_cast<const short*>(tab + P.a_lq);
  float* bias = reinterpret_cast<float*>(tab + 16 * (size_t)P.table_vecs);
  float* Z = bias + S;
  float* E = Z + R * S;
  float* Gb = E + R * S; // gated errors; SimplePC: f(z), the forward operand
  float* Vb = Gb + R * S;
  float* mu0 = Vb + (P.has_v ? R * S : 0);
  float* d0 = mu0 + R * P.N1p;
  float* topmu = d0 + R * P.N1p;
  const int NT = P.top_n, NTp = (NT + 3) & ~3;
  float* topd = topmu + R * NTp;

  for (int i = tid; i < P.table_vecs; i += kThreads)
    reinterpret_cast<int4*>(tab)[i] = __ldg(P.table + (size_t)rank * P.table_vecs + i);
  const int2 tasks = __ldg(P.counts + rank);
  for (int l = tid; l <= nw; l += kThreads)
  {
    const dpc_layer& L = P.layers[l];
    ptr[l] = SegPointers{L.W, L.b, L.z, L.e, L.mu, L.preact};
    lc[l] = SegConst{L.a, L.ir, L.momentum_beta, L.act | ((L.flags & DPC_LAYER_RESIDUAL) ? 256 : 0)};
  }
  __syncthreads();

  auto barrier = [&]
  {
    if (C > 1)
      cluster_sync_all();
    else
      __syncthreads();
  };
  // a value that the other blocks read too
  auto publish = [&](float* p, float v)
  {
    *p = v;
    const uint32_t at = smem_u32(p);
    for (int q = 1; q < C; ++q)
      asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(mapa_u32(at, (uint32_t)((rank + q) & (C - 1)))), "f"(v)
                   : "memory");
  };
  auto load_weights = [&]
  {
    for (int l = 1; l < nw; ++l)
    {
      const SegLayer L = sl[l];
      const float* W = ptr[l].W;
      const int Kp = (L.K + 3) & ~3;
      for (int r = L.o0 + warp; r < L.o1; r += kWarps)
      {
        const float* src = W + (size_t)r * L.K;
        float* dst = Ws + L.foff + (r - L.o0) * L.fpitch;
        if (L.vec)
          for (int c = lane * 4; c < L.K; c += 128)
            copy16(dst + c, src + c);
        else
          for (int c = lane; c < Kp; c += 32)
            if (c < L.K)
              copy4(dst + c, src + c);
            else
              dst[c] = 0.0f;
      }
      const int columns = L.c1 - L.c0;
      if (columns <= 0)
        continue;
      // (a warp's lanes take several rows where the columns are few)
      const int units = L.vec ? columns / 4 : columns;
      int lgw = 5;
      while (lgw > 0 && (1 << lgw) >= 2 * units)
        --lgw;
      const int per = 32 >> lgw, sub = lane >> lgw, at = lane & ((1 << lgw) - 1);
      for (int r = warp * per + sub; r < L.N; r += kWarps * per)
      {
        const float* src = W + (size_t)r * L.K + L.c0;
        float* dst = Ws + L.boff + r * L.bpitch;
        if (L.vec)
          for (int c = at; c < units; c += 1 << lgw)
            copy16(dst + 4 * c, src + 4 * c);
        else
          for (int c = at; c < units; c += 1 << lgw)
            copy4(dst + c, src + c);
      }
    }
    copies_commit();
  };

  const bool first = P.ops & DPC_ROWS_FIRST;
  for (int i = tid; i < S; i += kThreads)
  {
    const int l = layer_of[i >> 2] - 1, j = i - sl[l].noff;
    bias[i] = j < sl[l].N ? ptr[l].b[j] : 0.0f;
  }
  if (!first)
    load_weights();
  double esum = 0.0;

  for (int grp = (int)blockIdx.x / C; grp < P.groups; grp += (int)gridDim.x / C)
  {
    const int row0 = grp * R;
    const int rows = min(R, P.batch - row0);
    __syncthreads();

    // ---------------------------------------------------------------- beliefs (every block: all of them)
    {
      const bool zeros = P.ops & (DPC_ROWS_SWEEP | DPC_ROWS_ZERO_Z), load_e = (P.ops & DPC_ROWS_LOAD_E) != 0;
      for (int i = tid; i < S; i += kThreads)
      {
        const int l = layer_of[i >> 2], j = i - sl[l - 1].noff, N = sl[l - 1].N;
        const bool load_z = j < N && (!zeros || (P.top_clamped && l == nw));
        const float* v_from = P.has_v && !(P.ops & DPC_ROWS_ZERO_V) && j < N ? P.layers[l].v : nullptr;
        const size_t o = (size_t)row0 * N + j;
        constexpr int U = 4; // rows whose loads are in flight together
        for (int r0 = 0; r0 < R; r0 += U)
        {
          float z[U], e[U], v[U];
#pragma unroll
          for (int u = 0; u < U; ++u)
          {
            const int r = r0 + u;
            const size_t at = o + (size_t)r * N;
            z[u] = load_z && r < rows ? ptr[l].z[at] : 0.0f;
            e[u] = load_e && j < N && r < rows ? ptr[l].e[at] : 0.0f;
            v[u] = v_from && r < rows ? v_from[at] : 0.0f;
          }
#pragma unroll
          for (int u = 0; u < U; ++u)
          {
            if (r0 + u >= R)
              break;
            const int t = (r0 + u) * S + i;
            Z[t] = z[u], E[t] = e[u];
            Gb[t] = simple && l < nw && j < N ? act_fwd(lc[l].act(), z[u]) : 0.0f;
            if (P.has_v)
              Vb[t] = v[u];
          }
        }
      }
    }
    // ---------------------------------------------------------------- the clamped input layer
    {
      const SegLayer L = sl[0];
      const dpc_layer& D = P.layers[0];
      const int No = L.o1 - L.o0;
      if (first)
      {
        float* X = Ws; // the rows, then two steps of the weights
        float* ring = Ws + R * P.K0p;
        const int cp = P.kc | 4;
        const float* W = ptr[0].W + (size_t)L.o0 * L.K;
        auto load_step = [&](int k0, int buffer)
        {
          const int width = min(P.kc, L.K - k0);
          float* dst = ring + buffer * P.rows0 * cp;
          int lgw = 5; // lanes of a row
          while (lgw > 0 && (1 << lgw) >= 2 * (L.vec ? width / 4 : width))
            --lgw;
          const int per = 32 >> lgw, sub = lane >> lgw, at = lane & ((1 << lgw) - 1);
          for (int r = warp * per + sub; r < No; r += kWarps * per)
          {
            const float* src = W + (size_t)r * L.K + k0;
            if (L.vec)
              for (int c = at * 4; c < width; c += 4 << lgw)
                copy16(dst + r * cp + c, src + c);
            else
              for (int c = at; c < ((width + 3) & ~3); c += 1 << lgw)
                if (c < width)
                  copy4(dst + r * cp + c, src + c);
                else
                  dst[r * cp + c] = 0.0f;
          }
        };
        if (!L.lanes_k)
          load_step(0, 0);
        copies_commit();
        for (int k = tid, it = 0; k < P.K0p; k += kThreads, ++it)
        {
          constexpr int U = 4; // rows whose loads are in flight together
          for (int r0 = 0; r0 < R; r0 += U)
          {
            float v[U];
            const float* from = D.z + (size_t)(row0 + r0) * L.K + k;
#pragma unroll
            for (int u = 0; u < U; ++u)
              v[u] = r0 + u < rows && k < L.K ? from[(size_t)u * L.K] : 0.0f;
#pragma unroll
            for (int u = 0; u < U; ++u)
            {
              if (r0 + u >= R)
                break;
              if (simple && r0 + u < rows && k < L.K)
              {
                v[u] = act_fwd(lc[0].act(), v[u]);
                if (it % C == rank)
                  D.zF[(size_t)(row0 + r0 + u) * L.K + k] = v[u];
              }
              X[(r0 + u) * P.K0p + k] = v[u];
            }
          }
        }
        if (L.lanes_k)
        {
          __syncthreads();
          for (int t = warp; t < No * R; t += kWarps)
          {
            const int g = t / R, r = t - g * R;
            float acc = 0.0f;
#pragma unroll 4
            for (int k = lane * 4; k < L.K; k += 128)
            {
              const float4 w = *reinterpret_cast<const float4*>(W + (size_t)g * L.K + k);
              const float4 v = *reinterpret_cast<const float4*>(X + r * P.K0p + k);
              acc = fmaf(v.x, w.x, acc);
              acc = fmaf(v.y, w.y, acc);
              acc = fmaf(v.z, w.z, acc);
              acc = fmaf(v.w, w.w, acc);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
              acc += __shfl_xor_sync(0xffffffffu, acc, o);
            if (lane == 0)
              mu0[r * P.N1p + L.o0 + g] = acc;
          }
          __syncthreads();
        }
        else
        {
          const int lg = P.lg0, per = 32 >> lg, o = lane & (per - 1), s = lane >> (5 - lg);
          const int blocks = (No + per - 1) >> (5 - lg);
          auto step_sums = [&](auto rows_a_task, int step, int k0)
          {
            constexpr int T = decltype(rows_a_task)::value;
            const int rbs = R / T;
            const int width = min(P.kc, P.K0p - k0);
            const int from = s * P.slice0, len = max(0, min(width - from, P.slice0));
            for (int t = warp; t < blocks * rbs; t += kWarps)
            {
              const int b = t / rbs, rb = (t - b * rbs) * T, j = b * per + o;
              float* m = mu0 + rb * P.N1p + L.o0 + j;
              float acc[T];
#pragma unroll
              for (int r = 0; r < T; ++r)
                acc[r] = step > 0 && s == 0 && j < No ? m[r * P.N1p] : 0.0f;
              dot_row<T>(acc, ring + (step & 1) * P.rows0 * cp + min(j, No - 1) * cp + from,
                         X + rb * P.K0p + k0 + from, P.K0p, len);
              __syncwarp();
              add_slices<T>(acc, lg);
              if (s == 0 && j < No)
#pragma unroll
                for (int r = 0; r < T; ++r)
                  m[r * P.N1p] = acc[r];
            }
          };
          for (int k0 = 0, step = 0; k0 < L.K; k0 += P.kc, ++step)
          {
            if (k0 + P.kc < L.K)
              load_step(k0 + P.kc, (step + 1) & 1);
            copies_commit();
            copies_wait<1>();
            __syncthreads();
            if (RT > 1 && P.one_row0)
              step_sums(std::integral_constant<int, 1>(), step, k0);
            else
              step_sums(std::integral_constant<int, RT>(), step, k0);
            __syncthreads();
          }
        }
        load_weights(); // (the rows and steps are done with)
        for (int i = tid; i < R * No; i += kThreads)
        {
          const int r = i / No, c = L.o0 + i - r * No;
          const float pre = lc[0].a * mu0[r * P.N1p + c] + bias[L.noff + c];
          float mu = pre, d = 1.0f;
          if (!simple)
            act_both(lc[0].act(), pre, mu, d); // (a residual layer is never the first)
          mu0[r * P.N1p + c] = mu;
          d0[r * P.N1p + c] = d;
          if (r < rows)
          {
            const size_t o = (size_t)(row0 + r) * L.N + c;
            D.mu[o] = mu;
            if (D.preact)
              D.preact[o] = pre;
          }
        }
      }
      else
        for (int i = tid; i < R * No; i += kThreads)
        {
          const int r = i / No, c = L.o0 + i - r * No;
          const size_t o = (size_t)(row0 + r) * L.N + c;
          mu0[r * P.N1p + c] = r < rows ? D.mu[o] : 0.0f;
          d0[r * P.N1p + c] = (r < rows && !simple) ? act_deriv(lc[0].act(), D.preact[o]) : 1.0f;
        }
    }
    copies_wait<0>();
    barrier();

    // What a lane has of a task: its output (or column), its slice of the sum, and which rows it finishes -- the lanes
    // of an output take them in turn.
    struct Lane
    {
      int unit, s;
      bool mine[RT];
    };
    auto lane_of = [&](const SegTask& t)
    {
      Lane q;
      const int o = lane & ((32 >> t.lg) - 1);
      q.s = lane >> (5 - t.lg);
      q.unit = min(o, t.units - 1);
#pragma unroll
      for (int r = 0; r < RT; ++r)
        q.mine[r] = o < t.units && (r & ((1 << t.lg) - 1)) == q.s;
      return q;
    };
    // Predictions (and derivatives) of a forward task, from their sums or from the clamped input layer's cache; the same
    // in all lanes of an output.  All rows together: one after the other their dependent instructions took 650 cycles each.
    auto predict = [&](const SegTask& t, const Lane& q, bool pred, float (&mu)[RT], float (&d)[RT])
    {
      const int l = t.layer;
      if (t.kind == T_PLAIN)
      {
        const int m = t.row0 * P.N1p + t.j0 + q.unit;
#pragma unroll
        for (int r = 0; r < RT; ++r)
          mu[r] = mu0[m + r * P.N1p], d[r] = d0[m + r * P.N1p];
        return;
      }
      const SegConst c = lc[l];
      const float b = bias[t.first + q.unit];
      const float* x = (simple ? Gb : Z) + t.x;
      float pre[RT];
#pragma unroll
      for (int r = 0; r < RT; ++r)
        pre[r] = 0.0f;
      if (t.kind == T_DOT)
      {
        const int from = q.s * t.slice;
        dot_row<RT>(pre, Ws + t.w + q.unit * t.pitch + from, x + from, S, max(0, min(t.len - from, (int)t.slice)));
        __syncwarp();
        add_slices<RT>(pre, t.lg);
      }
      else
        for (int g = 0; g < t.units; ++g) // lanes along K
        {
          float sum[RT];
#pragma unroll
          for (int r = 0; r < RT; ++r)
            sum[r] = 0.0f;
          const float* w = Ws + t.w + g * t.pitch;
#pragma unroll 2
          for (int k = lane * 4; k < t.len; k += 128)
          {
            Quad<RT> f;
            f.row(smem_u32(w), smem_u32(x), S, k);
            f.multiply(sum);
          }
          __syncwarp();
          add_slices<RT>(sum, 5);
#pragma unroll
          for (int r = 0; r < RT; ++r)
            pre[r] = lane == g ? sum[r] : pre[r];
        }
#pragma unroll
      for (int r = 0; r < RT; ++r)
        pre[r] = c.a * pre[r] + b, mu[r] = pre[r], d[r] = 1.0f;
      if (!simple)
      {
        act_many<true>(c.act(), pre, mu, d);
        if (c.residual())
#pragma unroll
          for (int r = 0; r < RT; ++r)
            mu[r] += Z[(t.row0 + r) * S + t.first + q.unit + t.other];
      }
      if (pred)
      {
        const int N = sl[l].N;
        float* const to_mu = ptr[l].mu + (size_t)(row0 + t.row0) * N + t.j0 + q.unit;
        float* const to_pre = ptr[l].preact ? ptr[l].preact + (to_mu - ptr[l].mu) : nullptr;
#pragma unroll
        for (int r = 0; r < RT; ++r)
          if (q.mine[r] && t.row0 + r < rows)
          {
            to_mu[(size_t)r * N] = mu[r];
            if (to_pre)
              to_pre[(size_t)r * N] = pre[r];
          }
      }
    };
    // softmax cross-entropy error of the top layer from its logits, all of them in this block (one warp per row)
    auto ce_error = [&](bool energy)
    {
      const int to = sl[nw - 1].noff;
      if (sl[nw - 1].o1 <= sl[nw - 1].o0)
        return;
      __syncthreads();
      for (int r = warp; r < R; r += kWarps)
      {
        const float* m = topmu + r * NTp;
        float mx = -INFINITY, s = 0.0f, en = 0.0f;
        for (int j = lane; j < NT; j += 32)
          mx = fmaxf(mx, m[j]);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        for (int j = lane; j < NT; j += 32)
          s += expf(m[j] - mx);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
          s += __shfl_xor_sync(0xffffffffu, s, o);
        for (int j = lane; j < NT; j += 32)
        {
          const int t = r * S + to + j;
          const float p = expf(m[j] - mx) / s;
          const float z = Z[t];
          en -= z * logf(p + 1e-8f);
          const float e = z - p;
          if (simple)
            publish(E + t, e);
          else
          {
            E[t] = e;
            publish(Gb + t, e * topd[r * NTp + j]);
          }
        }
        if (energy && r < rows)
          esum += 2.0 * (double)en; // (halved at the end; cross-entropy is not)
      }
    };

    // ---------------------------------------------------------------- forward sweep
    if (P.ops & DPC_ROWS_SWEEP)
      for (int l = 0; l < nw; ++l)
      {
        const bool top = l + 1 == nw, copy = !(top && P.top_clamped);
#pragma unroll 1
        for (int q = sl[l].f0 + warp; q < sl[l].f1; q += kWarps)
        {
          const SegTask t = ftab[q];
          const Lane p = lane_of(t);
          float mu[RT], d[RT], f[RT];
          predict(t, p, (P.ops & DPC_ROWS_SWEEP_PRED) != 0, mu, d);
          if (simple && !top)
          {
            float unused[RT];
            act_many<false>(lc[l + 1].act(), mu, f, unused);
          }
#pragma unroll
          for (int r = 0; r < RT; ++r)
          {
            if (!p.mine[r])
              continue;
            const int at = (t.row0 + r) * S + t.first + p.unit, m = (t.row0 + r) * NTp + t.j0 + p.unit;
            if (copy)
            {
              if (simple)
              {
                Z[at] = mu[r];
                if (!top)
                  publish(Gb + at, f[r]);
              }
              else
                publish(Z + at, mu[r]);
            }
            if (top && P.ce)
              topmu[m] = mu[r], topd[m] = d[r];
            else if (top && (P.ops & DPC_ROWS_TERMINAL))
            {
              const float e = Z[at] - mu[r];
              if (simple)
                publish(E + at, e);
              else
                E[at] = e;
            }
          }
        }
        if (top && P.ce && (P.ops & DPC_ROWS_TERMINAL))
          ce_error(false);
        barrier();
      }

    // Settling steps, then the closing passes (one loop: the code of a pass exists once).
    // err: errors (and gated errors) are recomputed; else the gated errors are refreshed from the
    // errors that are there.
    const int refresh_at = (P.ops & DPC_ROWS_REFRESH) ? P.steps : -1;
    const int preact_at = (P.ops & DPC_ROWS_PREACT) ? P.steps + (refresh_at >= 0) : -1;
    const int energy_at =
        (P.ops & DPC_ROWS_ENERGY_LAST) ? P.steps + (refresh_at >= 0) + (preact_at >= 0) : -1;
    const int passes = P.steps + (refresh_at >= 0) + (preact_at >= 0) + (energy_at >= 0);
    // (most blocks have one task a warp and phase: it stays in registers)
    const SegTask first_f = ftab[min(warp, max(tasks.x - 1, 0))], first_b = btab[min(warp, max(tasks.y - 1, 0))];
#pragma unroll 1
    for (int t = 0; t < passes; ++t)
    {
      const bool settles = t < P.steps, last = t + 1 == P.steps;
      const bool err = settles || t == energy_at;
      const bool gate = settles || t == refresh_at || (t == energy_at && (P.ops & DPC_ROWS_GATE_LAST));
      const bool energy = settles ? (P.ops & DPC_ROWS_ENERGY_EACH) != 0 : t == energy_at;
      const bool pred = settles ? last && (P.ops & DPC_ROWS_PRED_LAST)
                                : t == preact_at || (P.ops & DPC_ROWS_PRED_CLOSE) != 0;
      float local = 0.0f;
      SegTask task = first_f;
#pragma unroll 1
      for (int q = warp; q < tasks.x;)
      {
        const Lane p = lane_of(task);
        const bool ce_top = P.ce && task.layer + 1 == nw;
        const bool errors = err && !ce_top, gates = gate && !simple && !(err && ce_top);
        int at[RT];
        float z[RT], mu[RT], d[RT], e[RT];
#pragma unroll
        for (int r = 0; r < RT; ++r)
        {
          at[r] = (task.row0 + r) * S + task.first + p.unit;
          z[r] = Z[at[r]], e[r] = E[at[r]];
        }
        predict(task, p, pred, mu, d);
        if (ce_top)
        {
          const int m = task.row0 * NTp + task.j0;
#pragma unroll
          for (int r = 0; r < RT; ++r)
            if (p.mine[r])
              topmu[m + (r) * NTp + p.unit] = mu[r], topd[m + (r) * NTp + p.unit] = d[r];
        }
#pragma unroll
        for (int r = 0; r < RT; ++r)
        {
          e[r] = errors ? z[r] - mu[r] : e[r];
          if (errors && p.mine[r] && task.row0 + r < rows)
            local += e[r] * e[r];
        }
#pragma unroll
        for (int r = 0; r < RT; ++r)
        {
          if (!p.mine[r])
            continue;
          if (errors && (!simple || !settles))
            E[at[r]] = e[r];
          if (gates && !settles)
            Gb[at[r]] = e[r] * d[r];
          if (settles && (simple ? errors : gates))
            publish((simple ? E : Gb) + at[r], simple ? e[r] : e[r] * d[r]);
        }
        if ((q += kWarps) < tasks.x)
          task = ftab[q];
      }
      if (energy)
        esum += (double)local;
      if (err && P.ce)
        ce_error(energy);
      barrier();
      if (!settles)
        continue;
      const bool refresh_f = simple && !(last && !(P.ops & DPC_ROWS_ENERGY_LAST));
      task = first_b;
#pragma unroll 1
      for (int q = warp; q < tasks.y;)
      {
        if (!(task.kind == T_PLAIN && P.top_clamped))
        {
          const Lane p = lane_of(task);
          const int l = task.layer;
          const SegConst c = lc[l];
          int at[RT];
          float z[RT], e[RT], f[RT], u[RT], m[RT], acc[RT];
#pragma unroll
          for (int r = 0; r < RT; ++r)
          {
            at[r] = (task.row0 + r) * S + task.first + p.unit;
            z[r] = Z[at[r]], e[r] = E[at[r]];
            f[r] = simple ? Gb[at[r]] : 0.0f;
            u[r] = c.residual() ? E[at[r] + task.other] : 0.0f;
            m[r] = P.has_v ? Vb[at[r]] : 0.0f;
            acc[r] = 0.0f;
          }
          if (task.kind == T_DOT)
          {
            const int from = p.s * task.slice;
            dot_column<RT>(acc, Ws + task.w + from * task.pitch + p.unit, task.pitch, (simple ? E : Gb) + task.x + from,
                           S, max(0, min(task.len - from, (int)task.slice)));
            __syncwarp();
            add_slices<RT>(acc, task.lg);
          }
          if (l == nw || (P.top_down_off && l == nw - 1))
#pragma unroll
            for (int r = 0; r < RT; ++r)
              z[r] -= c.ir * e[r];
          else if (simple)
          {
            float d[RT];
            if (act_has_output_deriv(c.act()))
#pragma unroll
              for (int r = 0; r < RT; ++r)
                d[r] = act_deriv_from_output(c.act(), f[r]);
            else
            {
              float unused[RT];
              act_many<true>(c.act(), z, unused, d);
            }
#pragma unroll
            for (int r = 0; r < RT; ++r)
              z[r] += c.ir * (acc[r] * d[r] - e[r]);
          }
          else
          {
#pragma unroll
            for (int r = 0; r < RT; ++r)
            {
              float fb = c.a * acc[r] - e[r];
              if (P.has_v)
              {
                // (which product is fused: as in the segments of single blocks, as in the phase kernels)
                fb = P.one_block ? fmaf(c.beta, m[r], (1.0f - c.beta) * fb) : fmaf(1.0f - c.beta, fb, c.beta * m[r]);
                m[r] = fb;
              }
              z[r] += c.ir * fb;
              if (c.residual())
                z[r] += c.ir * u[r];
            }
          }
          if (refresh_f && l < nw)
          {
            float unused[RT];
            act_many<false>(c.act(), z, f, unused);
          }
#pragma unroll
          for (int r = 0; r < RT; ++r)
          {
            if (!p.mine[r])
              continue;
            if (P.has_v && l < nw && !(P.top_down_off && l == nw - 1))
              Vb[at[r]] = m[r];
            if (simple)
              Z[at[r]] = z[r];
            if (!simple || (refresh_f && l < nw))
              publish((simple ? Gb : Z) + at[r], simple ? f[r] : z[r]);
          }
        }
        if ((q += kWarps) < tasks.y)
          task = btab[q];
      }
      barrier();
    }
    if (P.ops & DPC_ROWS_LOGITS)
    {
      // the top belief becomes the prediction below it
      const int l = nw - 1;
      for (int q = sl[l].f0 + warp; q < sl[l].f1; q += kWarps)
      {
        const SegTask t = ftab[q];
        const Lane p = lane_of(t);
        float mu[RT], d[RT];
        predict(t, p, true, mu, d);
#pragma unroll
        for (int r = 0; r < RT; ++r)
          if (p.mine[r])
            Z[(t.row0 + r) * S + t.first + p.unit] = mu[r];
      }
      __syncthreads();
    }

    // ---------------------------------------------------------------- back to memory, what this block finished
    for (int i = tid; i < S; i += kThreads)
    {
      const int l = layer_of[i >> 2], j = i - sl[l - 1].noff, N = sl[l - 1].N;
      if (j < sl[l - 1].o0 || j >= sl[l - 1].o1)
        continue;
      const dpc_layer& L = P.layers[l];
      const bool st_z = (P.ops & DPC_ROWS_STORE_Z) && !(l == nw && P.top_clamped);
      const bool st_e = (P.ops & DPC_ROWS_STORE_E) || ((P.ops & DPC_ROWS_TERMINAL) && l == nw);
      float* fe = (P.ops & DPC_ROWS_STORE_G) && !simple ? P.layers[l - 1].fe : nullptr;
      float* zf = simple && l < nw && (P.ops & DPC_ROWS_STORE_Z) ? L.zF : nullptr;
      float* v = P.has_v && (P.ops & DPC_ROWS_STORE_V) ? L.v : nullptr;
      for (int r = 0; r < rows; ++r)
      {
        const size_t m = (size_t)(row0 + r) * N + j;
        const int o = r * S + i;
        if (st_z)
          ptr[l].z[m] = Z[o];
        if (st_e)
          ptr[l].e[m] = E[o];
        if (fe)
          fe[m] = Gb[o];
        if (zf)
          zf[m] = Gb[o];
        if (v)
          v[m] = Vb[o];
      }
    }
    if (P.ops & DPC_ROWS_STORE_E)
    {
      float* e0 = P.layers[0].e + (size_t)row0 * sl[0].K;
      for (int i = rank * kThreads + tid; i < rows * sl[0].K; i += kThreads * C)
        e0[i] = 0.0f;
    }
  }
  if (P.ops & (DPC_ROWS_ENERGY_EACH | DPC_ROWS_ENERGY_LAST))
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

struct SegState
{
  SegParams P = {};
  int RT = 1;
  size_t smem = 0;
  void* dev = nullptr; // tables and task counts
};

inline int up4(int v)
{
  return (v + 3) & ~3;
}
// a multiple of 4 that is an odd one
inline int odd4(int v)
{
  return up4(v) | 4;
}

auto kernel_of(int RT)
{
  return RT == 1 ? cluster_rows_kernel<1> : RT == 2 ? cluster_rows_kernel<2> : cluster_rows_kernel<4>;
}

// Clusters of C blocks that run at once with most of the shared memory each; 0: none.
int resident_clusters(const dpc_ctx* ctx, int C)
{
  if (C == 1)
    return ctx->sm_count;
  static std::atomic<int> known[16][5]; // value + 1
  const int lg = C == 2 ? 1 : C == 4 ? 2 : C == 8 ? 3 : 4;
  std::atomic<int>& k = known[ctx->device & 15][lg];
  if (const int v = k.load())
    return v - 1;
  int n = 0;
  auto kern = cluster_rows_kernel<1>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(ctx->sm_count / C * C));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemLimit - kStatic;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)C, 1, 1};
  cfg.attrs = attr, cfg.numAttrs = 1;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmemLimit - kStatic)) !=
          cudaSuccess ||
      (C > 8 && cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
      cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess)
  {
    cudaGetLastError();
    n = 0;
  }
  k.store(n + 1);
  return n;
}

// A way to lay a plan out: C blocks a cluster, R rows a group, RT of them a task.
struct Layout
{
  int C = 0, R = 0, RT = 0;
  double cycles = 0.0; // estimate of a step of eight passes
  size_t smem = 0;
  std::vector<unsigned char> host; // tables of the blocks, then their task counts
  SegParams P = {};
};

// one_block: the plan has the segments of dpc_resident.cu, whose order of additions an ordered network keeps; else that
// of the phase kernels.  Without `tables` the tasks are counted, which is all that the estimate needs.
bool lay_out(const dpc_plan* p, int C, int R, int RT, bool exact, bool one_block, bool has_v, int S, bool tables,
             Layout& out)
{
  const int nw = p->n - 1, rbs = R / RT;
  const bool ce = (p->h[p->n - 1].flags & DPC_LAYER_SOFTMAX_CE) != 0;
  const bool simple = (p->h[0].flags & DPC_LAYER_INPUT_ACT) != 0;
  const int N1p = up4(p->h[0].next_size), K0p = up4(p->h[0].size), NTp = up4(p->h[nw - 1].next_size);
  auto share = [&](int N) { return std::min(N, up4((N + C - 1) / C)); };
  auto outputs = [&](int l) { return l + 1 == nw && ce ? p->h[l].next_size : share(p->h[l].next_size); };
  // Lanes of an output: the longest sums are shared first, while every warp still has one task at most.
  std::vector<int> lanes[2] = {std::vector<int>(nw, 0), std::vector<int>(nw, 0)}; // forward, state: log2 by layer
  for (int state = 0; state < 2 && !exact; ++state)
  {
    std::vector<int>& lg = lanes[state];
    auto len = [&](int l) { return state ? p->h[l].next_size : p->h[l].size; };
    auto tasks = [&](int l, int g) { return ((state ? outputs(l - 1) : outputs(l)) + (32 >> g) - 1) / (32 >> g) * rbs; };
    int total = 0;
    for (int l = 1; l < nw; ++l)
      total += tasks(l, 0);
    for (;;)
    {
      int longest = 0;
      for (int l = 1; l < nw; ++l)
        if (lg[l] < 2 && len(l) >> lg[l] >= 32 && (!longest || len(l) >> lg[l] > len(longest) >> lg[longest]))
          longest = l;
      if (!longest || total - tasks(longest, lg[longest]) + tasks(longest, lg[longest] + 1) > kWarps)
        break;
      total += tasks(longest, lg[longest] + 1) - tasks(longest, lg[longest]);
      ++lg[longest];
    }
  }
  const int rows0 = outputs(0);
  int lg0 = 0;
  while (!exact && lg0 < 2 && (rows0 + (16 >> lg0) - 1) / (16 >> lg0) * R <= kWarps)
    ++lg0;

  std::vector<int> counts;
  size_t region = 0, most_ft = 0, most_bt = 0;
  double forward = 0.0, state = 0.0, sweep = 0.0;
  std::vector<std::vector<SegLayer>> layers(tables ? C : 1, std::vector<SegLayer>(nw));
  std::vector<std::vector<SegTask>> ft(C), bt(C);
  for (int r = 0; r < C; ++r)
  {
    std::vector<SegLayer>& mine = layers[tables ? r : 0];
    size_t at = 0;
    int off = 0, nf = 0, nb = 0; // tasks
    std::array<double, kWarps> warp_f{}, warp_b{};
    double reads_f = 0.0, reads_b = 0.0;
    auto cost = [&](int len, int lg) // cycles of a task alone, and of its shared-memory reads
    {
      const double quads = len / 4.0 / (1 << lg);
      return std::make_pair(quads * (RT == 1 ? 20 : RT == 2 ? 26 : 45) + 600 + 60.0 * RT, quads * (4 + 2.1 * RT));
    };
    for (int l = 0; l < nw; ++l)
    {
      const dpc_layer& L = p->h[l];
      SegLayer& q = mine[l];
      q.K = L.size, q.N = L.next_size;
      q.noff = off, q.zoff = l ? mine[l - 1].noff : 0;
      off += up4(q.N);
      const int each = share(q.N);
      const bool whole = l + 1 == nw && ce;
      q.o0 = whole ? (r ? q.N : 0) : std::min(q.N, r * each);
      q.o1 = whole ? q.N : std::min(q.N, (r + 1) * each);
      q.c0 = l ? mine[l - 1].o0 : 0, q.c1 = l ? mine[l - 1].o1 : 0;
      q.vec = L.size % 4 == 0 && ((uintptr_t)L.W % 16) == 0;
      // (the shapes of the narrow forward kernel)
      q.lanes_k = exact && q.N <= 16 && q.K % 4 == 0 && q.K >= 128 && ((uintptr_t)L.z % 16) == 0 && q.vec &&
                  (!simple || (!one_block && L.opt == DPC_OPT_SGD && ((uintptr_t)L.zF % 16) == 0));
      q.fpitch = odd4(q.K), q.bpitch = odd4(std::max(1, q.c1 - q.c0));
      if (l)
      {
        q.foff = (int)at, at += (size_t)(q.o1 - q.o0) * q.fpitch;
        q.boff = (int)at, at += (size_t)(q.c1 > q.c0 ? q.N : 0) * q.bpitch;
      }
    }
    auto forward_tasks = [&](int l, int kind)
    {
      SegLayer& q = mine[l];
      const int lg = kind == T_DOT ? lanes[0][l] : 0, per = kind == T_LANES ? 2 : 32 >> lg;
      q.f0 = nf;
      q.f1 = nf += (q.o1 - q.o0 + per - 1) / per * rbs;
      for (int b = q.o0; tables && b < q.o1; b += per)
        for (int rb = 0; rb < rbs; ++rb)
        {
          SegTask t = {};
          t.kind = (unsigned char)kind;
          t.units = (unsigned char)std::min(per, q.o1 - b), t.lg = (unsigned char)lg;
          t.w = q.foff + (b - q.o0) * q.fpitch, t.pitch = (unsigned short)q.fpitch;
          t.x = q.zoff + rb * RT * S, t.len = (unsigned short)up4(q.K);
          t.slice = (unsigned short)(lg ? odd4((up4(q.K) + (1 << lg) - 1) >> lg) : up4(q.K));
          t.first = q.noff + b, t.row0 = (short)(rb * RT), t.layer = (short)l, t.j0 = (short)b;
          t.other = q.zoff - q.noff;
          ft[r].push_back(t);
        }
    };
    // Tasks of a settling pass; the input layer's outputs, which have no sums, after the others: a second task of some
    // warps.  Behind them the tasks of layers that are formed in another order when they are alone: the phase kernels
    // take a narrow head with the layers below it in one launch.
    for (int k = 1; k <= nw; ++k)
    {
      const int l = k % nw;
      const SegLayer& q = mine[l];
      const bool alone = one_block || nw == 2;
      forward_tasks(l, l == 0 ? T_PLAIN : q.lanes_k && alone ? T_LANES : T_DOT);
      const auto c = l == 0 ? std::make_pair(400 + 60.0 * RT, 10.0) : cost(q.K, lanes[0][l]);
      for (int t = q.f0; t < q.f1; ++t)
        warp_f[t % kWarps] += c.first, reads_f += c.second;
      sweep = std::max(sweep, c.first * ((q.f1 - q.f0 + kWarps - 1) / kWarps));
    }
    counts.push_back(nf);
    for (int l = 1; l < nw; ++l)
      if (mine[l].lanes_k && !one_block && nw > 2)
        forward_tasks(l, T_LANES);
    for (int l = 1; l <= nw; ++l)
    {
      const bool relax = l == nw;
      const int c0 = mine[l - 1].o0, c1 = mine[l - 1].o1, off_l = mine[l - 1].noff;
      const int lg = relax ? 0 : lanes[1][l], per = 32 >> lg;
      const int end = nb + (c1 - c0 + per - 1) / per * rbs;
      if (!relax)
      {
        const auto c = cost(mine[l].N, lg);
        for (int t = nb; t < end; ++t)
          warp_b[t % kWarps] += c.first, reads_b += c.second;
      }
      nb = end;
      for (int b = c0; tables && b < c1; b += per)
        for (int rb = 0; rb < rbs; ++rb)
        {
          SegTask t = {};
          t.kind = relax ? T_PLAIN : T_DOT;
          t.units = (unsigned char)std::min(per, c1 - b), t.lg = (unsigned char)lg;
          if (!relax)
          {
            const SegLayer& q = mine[l];
            t.w = q.boff + b - c0, t.pitch = (unsigned short)q.bpitch;
            t.x = q.noff + rb * RT * S, t.len = (unsigned short)q.N;
            t.slice = (unsigned short)(lg ? odd4((q.N + (1 << lg) - 1) >> lg) : q.N);
            t.other = q.noff - q.zoff;
          }
          t.first = off_l + b, t.row0 = (short)(rb * RT), t.layer = (short)l, t.j0 = (short)b;
          bt[r].push_back(t);
        }
    }
    counts.push_back(nb);
    region = std::max(region, at);
    most_ft = std::max(most_ft, (size_t)nf), most_bt = std::max(most_bt, (size_t)nb);
    forward = std::max({forward, reads_f, *std::max_element(warp_f.begin(), warp_f.end())});
    state = std::max({state, reads_b, *std::max_element(warp_b.begin(), warp_b.end())});
  }
  // the rows and two steps of the input layer's weights share the space with the weights
  auto round16 = [](size_t b) { return (b + 15) & ~(size_t)15; };
  const size_t a_ft = round16(sizeof(SegLayer) * nw), a_bt = a_ft + sizeof(SegTask) * most_ft,
               a_lq = a_bt + sizeof(SegTask) * most_bt, table = round16(a_lq + sizeof(short) * (S / 4));
  const size_t fixed = table + kStatic +
                       sizeof(float) * (S + (size_t)R * S * (has_v ? 4 : 3) + 2 * (size_t)R * N1p + 2 * (size_t)R * NTp);
  if (fixed >= kSmemLimit)
    return false;
  const size_t left = (kSmemLimit - fixed) / sizeof(float) & ~(size_t)3;
  if (region > left || (size_t)R * K0p >= left)
    return false;
  // columns of a step: a few dozen KB of loads in flight, fewer steps of short rows
  int kc = (int)std::min<size_t>((left - (size_t)R * K0p) / (2 * (size_t)rows0), 256) / 8 * 8 - 4;
  kc = std::min(kc, K0p);
  if (kc < 12 && kc < K0p)
    return false;
  region = std::max(region, (size_t)R * K0p + 2 * (size_t)rows0 * (kc | 4));
  region = (region + 3) & ~(size_t)3;
  if (region > left)
    return false;

  out.C = C, out.R = R, out.RT = RT;
  out.smem = fixed + region * sizeof(float);
  const double sync = C > 1 ? 350 + 60 * C : 80;
  // (the whole region, the input layer's steps included: the rule below was measured with it)
  out.cycles = 6000 + region * sizeof(float) / 50.0 + (double)rows0 * K0p * 4 / 50.0 + R * (K0p + S) / 100.0 +
               nw * (sweep + sync) + 8 * (forward + state + 2 * sync);

  if (!tables)
    return true;
  SegParams& P = out.P;
  P = SegParams{};
  P.table_vecs = (int)(table / 16), P.a_ft = (int)a_ft, P.a_bt = (int)a_bt, P.a_lq = (int)a_lq;
  P.n = p->n, P.batch = p->batch, P.S = S, P.C = C, P.R = R, P.groups = (p->batch + R - 1) / R;
  P.N1p = N1p, P.K0p = K0p, P.region = (int)region;
  P.kc = kc, P.rows0 = rows0, P.lg0 = lg0, P.slice0 = lg0 ? odd4((kc + (1 << lg0) - 1) >> lg0) : kc;
  // (tasks of RT rows where these leave no warp idle)
  P.one_row0 = (rows0 + (32 >> lg0) - 1) / (32 >> lg0) * rbs < kWarps;
  P.simple = simple, P.has_v = has_v, P.ce = ce, P.one_block = one_block, P.top_n = p->h[nw - 1].next_size;
  out.host.assign(table * C + sizeof(int) * counts.size(), 0);
  for (int r = 0; r < C; ++r)
  {
    unsigned char* t = out.host.data() + r * table;
    memcpy(t, layers[r].data(), sizeof(SegLayer) * nw);
    memcpy(t + a_ft, ft[r].data(), sizeof(SegTask) * ft[r].size());
    memcpy(t + a_bt, bt[r].data(), sizeof(SegTask) * bt[r].size());
    short* lq = reinterpret_cast<short*>(t + a_lq);
    for (int l = 0; l < nw; ++l)
      for (int c = 0; c < layers[r][l].N; c += 4)
        lq[(layers[r][l].noff + c) / 4] = (short)(l + 1);
  }
  memcpy(out.host.data() + table * C, counts.data(), sizeof(int) * counts.size());
  return true;
}
} // namespace

void cluster_plan_free(dpc_plan* p)
{
  auto* s = static_cast<SegState*>(p->seg);
  if (!s)
    return;
  cudaFree(s->dev);
  delete s;
  p->seg = nullptr;
}

int cluster_plan_init(dpc_plan* p)
{
  p->seg = nullptr;
  if (getenv("DPC_DISABLE_RESIDENT") || getenv("DPC_DISABLE_CLUSTERS"))
    return 1;
  const int n = p->n, nw = n - 1;
  if (n > kMaxLayers || p->run.count > 0 || tc_extra_layer(p, 0))
    return 1;
  int S = 0, longest = 0;
  size_t weights = 0;
  bool has_v = false;
  const bool exact = ordered_sums(p);
  for (int l = 0; l < nw; ++l)
  {
    const dpc_layer& L = p->h[l];
    if (l > 0)
      weights += (size_t)L.size * L.next_size, longest = std::max({longest, L.size, L.next_size});
    if (L.next_size <= 0 || L.next_size > 8192 || (l > 0 && L.size > 16384) ||
        ((L.flags ^ p->h[0].flags) & DPC_LAYER_INPUT_ACT) || (l == 0 && (L.flags & DPC_LAYER_RESIDUAL)) ||
        (L.flags & DPC_LAYER_SOFTMAX_CE) || (l > 0 && tc_extra_layer(p, l)) ||
        // (one block forms a softmax error, others the beliefs below it)
        (l + 1 == nw && (L.flags & DPC_LAYER_RESIDUAL) && (p->h[nw].flags & DPC_LAYER_SOFTMAX_CE)))
      return 1;
    has_v |= L.v != nullptr && l > 0;
    S += up4(L.next_size);
  }
  const char* force = getenv("DPC_CLUSTER_SIZE");
  const bool streams = res_plan_streams(p), either = p->res && !force; // single blocks can, too
  // (cheap answers first: weights that fit no cluster, held twice; what the rule below turns down by the network's shape)
  if (8 * weights > 16 * kSmemLimit || (either && !exact && !streams && (weights < 16000 || longest < 48)))
    return 1;
  auto estimate = [&](int C, int R, int RT, Layout& x)
  { return lay_out(p, C, R, RT, exact, p->res != nullptr, has_v, S, false, x); };
  // The best layout of clusters of C blocks, so many of them at once.  (One group of rows a cluster: weights that are loaded
  // again for the next group are what phase kernels do better.)
  auto choose = [&](int C, int clusters, Layout& best)
  {
    const int rows = (p->batch + clusters - 1) / clusters;
    for (int RT = 1; RT <= 4 && RT < 2 * rows; RT *= 2)
    {
      Layout x;
      const int R = (rows + RT - 1) / RT * RT;
      if (R <= 64 && estimate(C, R, RT, x) && (best.C == 0 || x.cycles < best.cycles))
        best = x;
    }
  };
  Layout best;
  if (!force || atoi(force) == 1)
    choose(1, p->ctx->sm_count, best);
  // Sliced segments that fit one block leave it only for clusters with one row each.  Where these are no faster than one
  // block, the device need not be asked how many clusters it holds (1 ms in a process's first plan).
  bool ask = !(either && !exact && !streams);
  for (int C = 2; C <= 16 && !ask; C *= 2)
  {
    Layout x;
    ask = p->batch <= p->ctx->sm_count / C && estimate(C, 1, 1, x) && (best.C == 0 || x.cycles < best.cycles);
  }
  if (!ask)
    return 1;
  for (int C = 2; C <= 16; C *= 2)
    if (!force || atoi(force) == C)
      if (const int clusters = resident_clusters(p->ctx, C))
        choose(C, clusters, best);
  if (best.C == 0)
    return 1;
  // Against the segments of single blocks, us a step: ordered sums are one chain either way, and gain where it was read
  // from L2 (784-441-441-10, SimplePC, ReLU, batch 25, T 11 401 / 141, 784-(77x7)-10 165 / 116) or the input layer's was
  // (3072-(53x3)-10 182 / 159), little where it is short (100-(47x3)-10 60 / 69, 100-(28x30)-10 141 / 161) or many rows
  // share a cluster (3072-74-10 at batch 460 398 / 412).  Sliced ones gain where a block reads weights from L2 on every
  // pass (202-202-202-10 at batch 167 171 / 121, 100-(273x4)-10 268 / 117) or blocks were left over (784-(58x6)-10 at
  // batch 3 110 / 89; 784-(76x4)-10 at batch 153 125 / 146, 784-(40x23)-10 at batch 19 136 / 146).
  if (either && (exact ? best.C == 1 && longest < 64 && p->h[0].size < 2048 : !streams && !(best.R == 1 && best.C > 1)))
    return 1;
  // With one row a cluster almost all that fits gains, against phase kernels 1.1 to 3.  With several the rows share a
  // cluster's few warps, and every layer of a sweep and every pass pays a barrier of the cluster's size, so the more a
  // step takes by the estimate and the shorter its sums, the less is gained; single blocks and phase kernels spread rows
  // over the SMs.  SimplePC networks, with one segment a step instead of three, gain longer against phase kernels.  Lines
  // from 8000 random networks (0.98 to 1.0 of the others' speed in the mean where they lie).  Beyond them, others /
  // clusters: phase kernels 784-(64x20)-10, Adam, batch 80, T 10 241 / 367, 784-(128x9)-37, ReLU, batch 51 132 / 194,
  // 48-(48x18)-10, Adam, batch 320 194 / 274; single blocks 784-(32x44)-10 at batch 79 231 / 395, 188-(188x3)-37,
  // SimplePC, batch 192 112 / 161, 100-(320x2)-2, SimplePC, batch 128 202 / 315, with ordered sums 100-(80x5)-10,
  // SimplePC, Adam, batch 512 157 / 245.
  struct Limit
  {
    double few, many; // cycles that two or three rows a cluster may take, and more rows
    int longest;      // by sums shorter than this
  };
  const bool simple = p->h[0].flags & DPC_LAYER_INPUT_ACT;
  const Limit limit = p->res ? (exact ? Limit{70e3, 50e3, 100} : Limit{longest < 46 ? 100e3 : 180e3, 65e3, 200})
                             : (simple ? Limit{155e3, 155e3, 150} : Limit{120e3, 90e3, 150});
  if (!force && !(p->res && exact && streams) &&
      ((best.R > 8 && (p->res || !simple)) || (!p->res && !exact && !simple && best.R > 2) ||
       (best.R > 1 && longest < limit.longest && best.cycles > (best.R < 4 ? limit.few : limit.many)) ||
       (p->res && exact && longest < 40 && best.cycles > limit.few)))
    return 1;
  // Networks of a head on a wide layer: their passes are the head's alone, and the wide layer's one product is what phase
  // kernels spread over all SMs.  Multiply-adds of a block for it, in millions, and others / clusters in us:
  // 0.5 784-1280-10, ReLU, batch 48 212 / 177;  1.9 1960-1960-2, ReLU, batch 48 159 / 327;  4.2 1026-512-2, batch 1024
  // 436 / 568;  4.8 784-768-16, batch 878 314 / 451;  SimplePC, which has one segment a step:  1.9 784-1190-10, Adam, batch
  // 256 476 / 324;  6.3 3072-512-10, batch 320 376 / 496.  (0.86 of the others' speed in the mean of 115 random networks
  // beyond the line, 1.4 in 1685 before it.)
  const dpc_layer& L0 = p->h[0];
  const double product = 1.0 * best.R * std::min(L0.next_size, up4((L0.next_size + best.C - 1) / best.C)) * L0.size;
  if (!force && nw == 2 && product > (simple ? 3.5e6 : 1.2e6))
    return 1;
  if (!lay_out(p, best.C, best.R, best.RT, exact, p->res != nullptr, has_v, S, true, best))
    return 1;
  auto* st = new SegState();
  if (cudaMalloc(&st->dev, best.host.size()) != cudaSuccess ||
      cudaMemcpyAsync(st->dev, best.host.data(), best.host.size(), cudaMemcpyHostToDevice, p->ctx->stream) !=
          cudaSuccess)
  {
    cudaFree(st->dev);
    delete st;
    return cuda_fail(cudaGetLastError(), "tables of the cluster segments");
  }
  st->P = best.P;
  st->P.table = static_cast<const int4*>(st->dev);
  st->P.counts = reinterpret_cast<const int2*>(static_cast<char*>(st->dev) + (size_t)best.P.table_vecs * 16 * best.C);
  st->P.layers = p->d;
  st->P.energy = p->energy;
  st->RT = best.RT;
  st->smem = best.smem;
  p->seg = st;
  return DPC_OK;
}

int cluster_segment(dpc_plan* p, int ops, int steps, int top_clamped, int top_down_off)
{
  const auto* st = static_cast<const SegState*>(p->seg);
  SegParams P = st->P;
  P.ops = ops, P.steps = steps;
  P.top_clamped = top_clamped, P.top_down_off = top_down_off;
  auto kern = kernel_of(st->RT);
  const int which = st->RT >> 1;
  static thread_local int configured[3] = {-1, -1, -1};
  if (configured[which] != p->ctx->device)
  {
    DPC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)(kSmemLimit - kStatic)));
    DPC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    configured[which] = p->ctx->device;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(std::min(P.groups, resident_clusters(p->ctx, P.C)) * P.C));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = st->smem - kStatic;
  cfg.stream = p->ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)P.C, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = P.C > 1 ? 1 : 0;
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, P);
  p->ctx->launches += 1;
  return err == cudaSuccess ? DPC_OK : cuda_fail(err, "cluster segment kernel");
}
} // namespace dpc

using namespace dpc;

int dpc_rows_clusters(dpc_plan* p)
{
  return p && p->seg ? static_cast<const SegState*>(p->seg)->P.C : 0;
}
