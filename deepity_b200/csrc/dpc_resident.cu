// Row-resident train step of small dense networks.
//
// Within a step the batch rows meet only in the weight updates: a forward sweep, any number of
// settling steps, the refresh before learning and the closing energy are all row-local.  For a
// network whose weights fit (or nearly fit) one SM's shared memory, a launch per phase is pure
// latency -- a settling step of a 784-128-128-10 network at batch 64 is 2 MFLOP and took 44 us in
// three launches.  Here one CTA owns R rows and walks all phases between two weight updates by
// itself ("segment"): weights in shared memory (layer by layer, as many as fit, the others streamed
// from L2), beliefs, errors and gated errors of its rows in shared memory, no launch and no global
// traffic inside the settling loop, only barriers of the CTA.
//
// Measured: 784-128-128-10 at batch 64, 20 steps, 879 -> 113 us a step (about 2.5 us a settling pass: 1600 and
// 900 cycles of sums, two elementwise phases of 1000 that are chains of latencies); ordered sums with streamed
// weights, 100-300-200-77-10 at batch 50 with AdamW, 6 steps, 750 -> 183 us.
//
// A pass is a list of warp tasks that leave partial sums in shared memory, a barrier, and an
// elementwise pass that adds them in a fixed order and finishes (activation, error, gated error, or
// the state update); all layers of a settling pass are independent (Jacobi) and share one list.
//   forward, resident weights   lane = output, walking a slice of K: no reduction, no idle epilogue
//                               lanes (lanes along K with a shuffle reduction spend 300 instructions
//                               on 8 outputs of a 128-wide row, and a settling step is bound by issue
//                               slots).  Row pitch 4 x odd floats, so the lanes' 16-byte reads of
//                               neighbouring rows meet no bank conflict.
//   forward, streamed weights   lanes along K (coalesced), G outputs x R rows, halving reduction
//   state update                lane = 4 (or 1) input columns, walking a slice of the output rows
//
// The same tasks, i.e. the same order of additions, serve the sweep and every later pass: a belief
// that the sweep produced has an error of exactly zero afterwards (Adam-type updates rely on it).
// Networks with an Adam-type optimizer ("exact") go further: an update m / (sqrt(v) + eps) turns a
// rounding difference of a near-zero gradient into a step of full size, so every sum there has ONE
// order -- ascending, one accumulator, as the phase kernels have it -- and no slices.  So do networks
// whose activation has a kink, where such a difference flips a derivative between 0 and 1.
#include <algorithm>
#include <cstdlib>
#include <cstring>

#include "dpc_internal.h"
#include "dpc_math.cuh"

namespace dpc
{
namespace
{
constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kMaxLayers = 96;
constexpr size_t kSmemLimit = 227 * 1024, kStatic = 4 * 1024; // per block; of it static

struct ResLayer // one per weight layer, built on the host
{
  int K, N;
  int zoff, noff;    // offsets of layers l and l+1 in a row's state (multiples of 4)
  int ldw, woff;     // row pitch and offset of W in shared memory
  int rrows;         // rows of W that are resident (the first ones); the others are streamed
  int lanes_k;       // exact networks: lanes along K, the narrow heads' order of additions
  int vec;           // rows of W in global memory can be read 16 bytes at a time
  int kw;            // columns per lane of a state task: 4 or 1
  int fpart, fslice; // forward partial sums: offset, length of a slice of K
  int bpart, bslices; // state partial sums: offset, slices of the output rows
  int pad[2];
};

// Four neighbouring floats of a row's state (they belong to one layer).
struct __align__(16) ResQuad
{
  int fpart, bpart;       // their partial sums of slice 0, row 0 (row pitch `pitch`)
  short fslices, bslices; // slices of the prediction from below / of the feedback from above
  short layer, valid;     // layer 1 .. n-1; columns that exist (the rest is padding)
  int col, pitch;         // first column inside the layer, padded width of the layer
  int down, up;           // state offsets of the same columns in the layer below / above (residuals)
};

// One warp task, everything its lanes need in two 16-byte reads.  Offsets in floats.
struct __align__(16) ResTask
{
  int w, ldw;     // first weight and row pitch: in the resident weights, or in the layer's W
  int x, len;     // first operand element of the first row; K (forward) or output rows (state) to walk
  int out, pitch; // first partial sum of the first row, distance to the next row's
  int lanes;      // lanes (resident forward: outputs, state: column groups) that exist
  int kind;       // layer << 4 | T_*
  int w2, len2;   // state: streamed rows that follow the resident ones in the same sum
  int pad[2];
};
enum
{
  T_STREAM = 1, // weights in global memory
  T_VEC = 2,    // forward: rows readable 16 bytes at a time; state: 4 columns per lane
  T_LANES = 4   // forward: lanes along K
};

struct ResParams
{
  const dpc_layer* layers;
  // one table in global memory, copied to shared memory as it is:
  //   ResLayer[nw] | ResQuad[S / 4] | forward tasks (sorted by layer) | state tasks
  const int4* table;
  int table_vecs, a_quad, a_ft, a_bt; // its size in 16-byte units, byte offsets of the parts
  int n, batch, S;                    // layers, rows, floats of one row's state (layers 1..n-1)
  int nf, nb;                         // task counts
  int N1p, K0p;                       // padded width of layer 1 and of the input
  int ks0, kslice0;                   // input layer: slices of K and their length
  int wfloats;                        // resident weights
  int groups;                         // row groups
  int ops, steps;
  int exact;                          // one order of additions everywhere
  int simple, has_v, ce, top_clamped, top_down_off, top_n;
  double* energy;
};

template <int R>
constexpr int kRowsPerTask = R >= 4 ? 4 : R;

template <int V>
__device__ __forceinline__ float reduce_values(float (&a)[V], int lane)
{
  // the lanes exchange halves: after log2(V) steps lane i holds a partial sum of value
  // i >> (5 - log2 V), the remaining steps add the lanes that hold the same one
  int bit = 16;
#pragma unroll
  for (int w = V / 2; w >= 1; w >>= 1)
  {
    const bool upper = (lane & bit) != 0;
#pragma unroll
    for (int i = 0; i < w; ++i)
    {
      const float send = upper ? a[i] : a[i + w];
      const float keep = upper ? a[i + w] : a[i];
      a[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
    }
    bit >>= 1;
  }
  float s = a[0];
#pragma unroll
  for (; bit >= 1; bit >>= 1)
    s += __shfl_xor_sync(0xffffffffu, s, bit);
  return s;
}

// Streamed weights: acc[r * G + g] += sum over this lane's k in [k0, k1) of x[r][k] * W[row g][k]
template <int R, int G>
__device__ __forceinline__ void dot_streamed(float (&acc)[R * G], const float* __restrict__ W, int ldw,
                                             int rows_left, const float* x, int xs, int k0, int k1,
                                             int lane, bool vec)
{
  const float* row[G];
#pragma unroll
  for (int g = 0; g < G; ++g)
    row[g] = W + (size_t)min(g, rows_left - 1) * ldw;
  if (vec)
    for (int k = k0 + lane * 4; k < k1; k += 128)
    {
      float4 w[G];
#pragma unroll
      for (int g = 0; g < G; ++g)
        w[g] = *reinterpret_cast<const float4*>(row[g] + k);
#pragma unroll
      for (int r = 0; r < R; ++r)
      {
        const float4 v = *reinterpret_cast<const float4*>(x + r * xs + k);
#pragma unroll
        for (int g = 0; g < G; ++g)
        {
          float s = acc[r * G + g];
          s = fmaf(v.x, w[g].x, s);
          s = fmaf(v.y, w[g].y, s);
          s = fmaf(v.z, w[g].z, s);
          acc[r * G + g] = fmaf(v.w, w[g].w, s);
        }
      }
    }
  else
#pragma unroll 2
    for (int k = k0 + lane; k < k1; k += 32)
    {
      float w[G];
#pragma unroll
      for (int g = 0; g < G; ++g)
        w[g] = row[g][k];
#pragma unroll
      for (int r = 0; r < R; ++r)
      {
        const float v = x[r * xs + k];
#pragma unroll
        for (int g = 0; g < G; ++g)
          acc[r * G + g] = fmaf(v, w[g], acc[r * G + g]);
      }
    }
}

// Partial sums of the input layer, read once a segment from L2: tasks of G outputs x R rows x a slice of K, lanes
// along K, the loads of two strips (four of single elements) in flight together.  A function that is called: its
// registers are not the loop's.
template <int R, int G>
__device__ __noinline__ void input_sums(const float* __restrict__ W, int K, int N, const float* X, int xs, int slices,
                                        int slice, float* part, int warp, int lane, bool vec)
{
  constexpr int V = R * G, LPV = 32 / V;
  for (int t = warp; t < (N + G - 1) / G * slices; t += kWarps)
  {
    const int g0 = t / slices * G, k0 = (t - t / slices * slices) * slice, k1 = min(K, k0 + slice);
    const float* row[G];
#pragma unroll
    for (int g = 0; g < G; ++g)
      row[g] = W + (size_t)min(g0 + g, N - 1) * K;
    float acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i)
      acc[i] = 0.0f;
    auto strips = [&](auto width, auto count, int k) // `count` strips of 32 `width` elements from k
    {
      constexpr int E = decltype(width)::value, C = decltype(count)::value;
      float w[C][G][E];
#pragma unroll
      for (int q = 0; q < C; ++q)
#pragma unroll
        for (int g = 0; g < G; ++g)
          if constexpr (E == 4)
          {
            const float4 v = *reinterpret_cast<const float4*>(row[g] + k + q * 128);
            w[q][g][0] = v.x, w[q][g][1] = v.y, w[q][g][2] = v.z, w[q][g][3] = v.w;
          }
          else
            w[q][g][0] = row[g][k + q * 32];
#pragma unroll
      for (int q = 0; q < C; ++q)
#pragma unroll
        for (int r = 0; r < R; ++r)
        {
          float v[E];
          const float* x = X + r * xs + k + q * 32 * E;
          if constexpr (E == 4)
          {
            const float4 t4 = *reinterpret_cast<const float4*>(x);
            v[0] = t4.x, v[1] = t4.y, v[2] = t4.z, v[3] = t4.w;
          }
          else
            v[0] = *x;
#pragma unroll
          for (int g = 0; g < G; ++g)
#pragma unroll
            for (int j = 0; j < E; ++j)
              acc[r * G + g] = fmaf(v[j], w[q][g][j], acc[r * G + g]);
        }
    };
    using std::integral_constant;
    if (vec)
    {
      int k = k0 + lane * 4;
      if (V < 32) // (else the sums take the registers)
#pragma unroll 1
        for (; k + 128 < k1; k += 256)
          strips(integral_constant<int, 4>(), integral_constant<int, 2>(), k);
#pragma unroll 1
      for (; k < k1; k += 128)
        strips(integral_constant<int, 4>(), integral_constant<int, 1>(), k);
    }
    else
    {
      int k = k0 + lane;
#pragma unroll 1
      for (; k + 96 < k1; k += 128)
        strips(integral_constant<int, 1>(), integral_constant<int, 4>(), k);
#pragma unroll 1
      for (; k < k1; k += 32)
        strips(integral_constant<int, 1>(), integral_constant<int, 1>(), k);
    }
    __syncwarp();
    const float v = reduce_values<V>(acc, lane);
    if (lane % LPV == 0)
      part[t * V + lane / LPV] = v;
  }
}

// Resident weights: this lane's output over `len` inputs (walked four at a time, zero-padded).
template <int RT>
__device__ __forceinline__ void dot_resident(const float* w, const float* x, int S, int len, float* out,
                                             int pitch, bool valid)
{
  float acc[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r)
    acc[r] = 0.0f;
#pragma unroll 4
  for (int k = 0; k < len; k += 4)
  {
    const float4 wv = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
    for (int r = 0; r < RT; ++r)
    {
      const float4 v = *reinterpret_cast<const float4*>(x + r * S + k);
      acc[r] = fmaf(v.x, wv.x, acc[r]);
      acc[r] = fmaf(v.y, wv.y, acc[r]);
      acc[r] = fmaf(v.z, wv.z, acc[r]);
      acc[r] = fmaf(v.w, wv.w, acc[r]);
    }
  }
  if (valid)
#pragma unroll
    for (int r = 0; r < RT; ++r)
      out[r * pitch] = acc[r];
}

// The same for rows of W in global memory.
template <int RT>
__device__ __forceinline__ void dot_rows(const float* __restrict__ w, const float* x, int S, int len,
                                         float* out, int pitch, bool valid, bool vec)
{
  float acc[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r)
    acc[r] = 0.0f;
  int k = 0;
  if (vec)
  {
#pragma unroll 8
    for (; k < len; k += 4)
    {
      const float4 wv = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
      for (int r = 0; r < RT; ++r)
      {
        const float4 v = *reinterpret_cast<const float4*>(x + r * S + k);
        acc[r] = fmaf(v.x, wv.x, acc[r]);
        acc[r] = fmaf(v.y, wv.y, acc[r]);
        acc[r] = fmaf(v.z, wv.z, acc[r]);
        acc[r] = fmaf(v.w, wv.w, acc[r]);
      }
    }
  }
  else
#pragma unroll 8
    for (; k < len; ++k)
    {
      const float wv = w[k];
#pragma unroll
      for (int r = 0; r < RT; ++r)
        acc[r] = fmaf(x[r * S + k], wv, acc[r]);
    }
  if (valid)
#pragma unroll
    for (int r = 0; r < RT; ++r)
      out[r * pitch] = acc[r];
}

// The same for the input layer's rows, which may be long.  A lane's sum is one chain over its row, and each batch of
// loads costs the latency of L2 (1000 cycles): 16 loads in flight, 32 where they are single elements (32 rows of 1971
// elements that are not 16-byte aligned 108 -> 33 us).  A function that is called: its registers are not the loop's.
template <int RT>
__device__ __noinline__ void dot_input(const float* __restrict__ w, const float* x, int S, int len,
                                       float* out, int pitch, bool valid, bool vec)
{
  float acc[RT];
#pragma unroll
  for (int r = 0; r < RT; ++r)
    acc[r] = 0.0f;
  auto quads = [&](auto count, int k)
  {
    constexpr int C = decltype(count)::value;
    float4 wv[C];
#pragma unroll
    for (int q = 0; q < C; ++q)
      wv[q] = *reinterpret_cast<const float4*>(w + k + 4 * q);
#pragma unroll
    for (int q = 0; q < C; ++q)
#pragma unroll
      for (int r = 0; r < RT; ++r)
      {
        const float4 v = *reinterpret_cast<const float4*>(x + r * S + k + 4 * q);
        acc[r] = fmaf(v.x, wv[q].x, acc[r]);
        acc[r] = fmaf(v.y, wv[q].y, acc[r]);
        acc[r] = fmaf(v.z, wv[q].z, acc[r]);
        acc[r] = fmaf(v.w, wv[q].w, acc[r]);
      }
  };
  auto singles = [&](auto count, int k)
  {
    constexpr int C = decltype(count)::value;
    float wv[C];
#pragma unroll
    for (int q = 0; q < C; ++q)
      wv[q] = w[k + q];
#pragma unroll
    for (int q = 0; q < C; ++q)
#pragma unroll
      for (int r = 0; r < RT; ++r)
        acc[r] = fmaf(x[r * S + k + q], wv[q], acc[r]);
  };
  int k = 0;
  if (vec)
  {
#pragma unroll 1
    for (; k + 64 <= len; k += 64)
      quads(std::integral_constant<int, 16>(), k);
#pragma unroll 1
    for (; k + 16 <= len; k += 16)
      quads(std::integral_constant<int, 4>(), k);
#pragma unroll 1
    for (; k < len; k += 4)
      quads(std::integral_constant<int, 1>(), k);
  }
  else
  {
#pragma unroll 1
    for (; k + 32 <= len; k += 32)
      singles(std::integral_constant<int, 32>(), k);
#pragma unroll 1
    for (; k + 8 <= len; k += 8)
      singles(std::integral_constant<int, 8>(), k);
#pragma unroll 1
    for (; k < len; ++k)
      singles(std::integral_constant<int, 1>(), k);
  }
  if (valid)
#pragma unroll
    for (int r = 0; r < RT; ++r)
      out[r * pitch] = acc[r];
}

// One state task: sums over `len` rows of W for this lane's KW columns.
template <int RT, int KW, int UNROLL>
__device__ __forceinline__ void state_sum(float (&acc)[RT][KW], const float* w, int ldw, int len,
                                          const float* g, int S)
{
  int n = 0;
  // (streamed rows: the loads of 4 UNROLL rows are in flight together)
#pragma unroll UNROLL
  for (; n + 4 <= len; n += 4, w += 4 * (size_t)ldw)
  {
    float wv[4][KW];
#pragma unroll
    for (int j = 0; j < 4; ++j)
    {
      if constexpr (KW == 4)
      {
        const float4 v = *reinterpret_cast<const float4*>(w + j * (size_t)ldw);
        wv[j][0] = v.x, wv[j][1] = v.y, wv[j][2] = v.z, wv[j][3] = v.w;
      }
      else
        wv[j][0] = w[j * (size_t)ldw];
    }
#pragma unroll
    for (int r = 0; r < RT; ++r)
    {
      const float4 v = *reinterpret_cast<const float4*>(g + r * S + n);
#pragma unroll
      for (int c = 0; c < KW; ++c)
      {
        acc[r][c] = fmaf(v.x, wv[0][c], acc[r][c]);
        acc[r][c] = fmaf(v.y, wv[1][c], acc[r][c]);
        acc[r][c] = fmaf(v.z, wv[2][c], acc[r][c]);
        acc[r][c] = fmaf(v.w, wv[3][c], acc[r][c]);
      }
    }
  }
  for (; n < len; ++n, w += ldw)
#pragma unroll
    for (int c = 0; c < KW; ++c)
    {
      const float wv = w[c];
#pragma unroll
      for (int r = 0; r < RT; ++r)
        acc[r][c] = fmaf(g[r * S + n], wv, acc[r][c]);
    }
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src)
{
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

__device__ __forceinline__ void get4(float (&v)[4], const float* p)
{
  const float4 t = *reinterpret_cast<const float4*>(p);
  v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
}
__device__ __forceinline__ void put4(float* p, const float (&v)[4])
{
  *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
}
// Sum of `slices` partial sums, four neighbours at once, in slice order; four slices are read at a time.
__device__ __forceinline__ void sum4(float (&v)[4], const float* p, int slices, int stride)
{
  get4(v, p);
#pragma unroll 1
  for (int s = 1; s < slices; s += 4)
  {
    float t[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      get4(t[q], p + min(s + q, slices - 1) * stride);
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (s + q < slices)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          v[j] += t[q][j];
  }
}
// Activation and derivative of four values with one dispatch.
__device__ __forceinline__ void act4(int act, const float (&z)[4], float (&f)[4], float (&d)[4])
{
#define DPC_ACT4(A)                                                                               \
  case A:                                                                                         \
    _Pragma("unroll") for (int j = 0; j < 4; ++j) act_both(A, z[j], f[j], d[j]);                  \
    break;
  switch (act)
  {
    DPC_ACT4(DPC_ACT_RELU)
    DPC_ACT4(DPC_ACT_GELU)
    DPC_ACT4(DPC_ACT_SIGMOID)
    DPC_ACT4(DPC_ACT_ESIGMOID)
    DPC_ACT4(DPC_ACT_TANH)
    DPC_ACT4(DPC_ACT_HARD_TANH)
  default:
#pragma unroll
    for (int j = 0; j < 4; ++j)
      f[j] = z[j], d[j] = 1.0f;
  }
#undef DPC_ACT4
}
// f'(z) of four values whose f(z) is known, with one dispatch (one per value was a quarter of the elementwise
// phase of a state update).
__device__ __forceinline__ void deriv4(int act, const float (&z)[4], const float (&f)[4], float (&d)[4])
{
#define DPC_DERIV4(A)                                                                             \
  case A:                                                                                         \
    _Pragma("unroll") for (int j = 0; j < 4; ++j) d[j] = act_deriv_from_output(A, f[j]);          \
    break;
  switch (act)
  {
    DPC_DERIV4(DPC_ACT_TANH)
    DPC_DERIV4(DPC_ACT_SIGMOID)
    DPC_DERIV4(DPC_ACT_RELU)
    DPC_DERIV4(DPC_ACT_LINEAR)
    DPC_DERIV4(DPC_ACT_HARD_TANH)
  default:
    act_deriv4(act, z, d);
  }
#undef DPC_DERIV4
}

struct LayerConst // what a finished sum of layer l needs, one 16-byte read
{
  float a, ir, beta;
  int kind; // activation, | 256: residual
  __device__ __forceinline__ int act() const { return kind & 255; }
  __device__ __forceinline__ bool residual() const { return (kind & 256) != 0; }
};

template <int R>
__global__ void __launch_bounds__(kThreads, 1) resident_kernel(const ResParams P)
{
  constexpr int RT = kRowsPerTask<R>;
  constexpr int G = R == 8 ? 4 : 8, V = R * G, LPV = 32 / V; // outputs per group, lanes per value
  extern __shared__ __align__(16) float sm[];
  __shared__ __align__(16) LayerConst lc[kMaxLayers];
  __shared__ const float* sW[kMaxLayers];
  __shared__ float red[kWarps];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int S = P.S, nw = P.n - 1; // nw weight layers
  const bool simple = P.simple != 0;

  // ---- shared memory: weights | table | bias | Z E G(or f(z)) [V] | mu0 d0 | top mu, d | X / partials
  float* Ws = sm;
  unsigned char* tab = reinterpret_cast<unsigned char*>(Ws + P.wfloats);
  const ResLayer* sl = reinterpret_cast<const ResLayer*>(tab);
  const ResQuad* quad = reinterpret_cast<const ResQuad*>(tab + P.a_quad);
  const ResTask* ftab = reinterpret_cast<const ResTask*>(tab + P.a_ft);
  const ResTask* btab = reinterpret_cast<const ResTask*>(tab + P.a_bt);
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
  float* X = topd + R * NTp; // input rows; later the partial sums of the tasks

  for (int i = tid; i < P.table_vecs; i += kThreads)
    reinterpret_cast<int4*>(tab)[i] = __ldg(P.table + i);
  for (int l = tid; l <= nw; l += kThreads)
  {
    const dpc_layer& L = P.layers[l];
    sW[l] = L.W;
    lc[l] = LayerConst{L.a, L.ir, L.momentum_beta, L.act | ((L.flags & DPC_LAYER_RESIDUAL) ? 256 : 0)};
  }
  __syncthreads();
  for (int l = 1; l < nw; ++l)
  {
    const ResLayer L = sl[l];
    if (L.rrows == 0)
      continue;
    const float* src = sW[l];
    float* dst = Ws + L.woff;
    for (int r = warp; r < L.rrows; r += kWarps)
      if (L.vec)
        for (int c = lane * 4; c < L.K; c += 128)
          cp_async16(dst + r * L.ldw + c, src + (size_t)r * L.K + c);
      else
        for (int c = lane; c < L.ldw; c += 32)
          dst[r * L.ldw + c] = c < L.K ? src[(size_t)r * L.K + c] : 0.0f;
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  // Elementwise passes: a thread takes four neighbouring elements of a row at a time (most networks:
  // one quad per thread, whose table entry then stays in registers).
  const int S4 = S >> 2, nq = R * S4;
  const int own_r = tid / S4, own_i = tid - own_r * S4;
  const ResQuad own = quad[own_i];
  auto for_quads = [&](auto&& f)
  {
    if (tid >= nq)
      return;
    int i = own_i, r = own_r;
    ResQuad q = own;
    for (int idx = tid;;)
    {
      f(q, i, r);
      idx += kThreads;
      if (idx >= nq)
        break;
      r = idx / S4, i = idx - r * S4;
      q = quad[i];
    }
  };
  for (int i = tid; i < S; i += kThreads)
  {
    const ResQuad q = quad[i >> 2];
    bias[i] = (i & 3) < q.valid ? P.layers[q.layer - 1].b[q.col + (i & 3)] : 0.0f;
  }

  const bool first = P.ops & DPC_ROWS_FIRST;
  double esum = 0.0;

  for (int grp = blockIdx.x; grp < P.groups; grp += gridDim.x)
  {
    const int row0 = grp * R;
    const int rows = min(R, P.batch - row0);
    __syncthreads();

    // ---------------------------------------------------------------- beliefs
    for_quads([&](const ResQuad& q, int i, int r)
              {
                const int l = q.layer;
                const dpc_layer& L = P.layers[l];
                const size_t o = (size_t)(row0 + r) * sl[l - 1].N + q.col;
                const bool load_z =
                    (P.top_clamped && l == nw) || !(P.ops & (DPC_ROWS_SWEEP | DPC_ROWS_ZERO_Z));
                const bool load_v = P.has_v && !(P.ops & DPC_ROWS_ZERO_V) && L.v;
                float z[4], e[4], v[4], f[4], d[4];
#pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                  const bool in = r < rows && j < q.valid;
                  z[j] = in && load_z ? L.z[o + j] : 0.0f;
                  e[j] = in && (P.ops & DPC_ROWS_LOAD_E) ? L.e[o + j] : 0.0f;
                  v[j] = in && load_v ? L.v[o + j] : 0.0f;
                  f[j] = 0.0f;
                }
                if (simple && l < nw)
                  act4(lc[l].act(), z, f, d);
                const int t = r * S + 4 * i;
                put4(Z + t, z);
                put4(E + t, e);
                put4(Gb + t, f);
                if (P.has_v)
                  put4(Vb + t, v);
              });
    // ---------------------------------------------------------------- the clamped input layer
    {
      const ResLayer L = sl[0];
      const dpc_layer& D = P.layers[0];
      if (first)
      {
        for (int r = 0; r < R; ++r)
          for (int k = tid; k < P.K0p; k += kThreads)
          {
            float v = 0.0f;
            if (r < rows && k < L.K)
            {
              const size_t o = (size_t)(row0 + r) * L.K + k;
              v = D.z[o];
              if (simple)
              {
                v = act_fwd(lc[0].act(), v);
                D.zF[o] = v;
              }
            }
            X[r * P.K0p + k] = v;
          }
        __syncthreads();
        float* part = X + R * P.K0p;
        if (P.exact && !L.lanes_k)
        {
          // one ascending sum per output: lane = output
          constexpr int RBS = R / RT;
          for (int t = warp; t < (L.N + 31) / 32 * RBS; t += kWarps)
          {
            const int c = t / RBS * 32 + lane, rb = t % RBS * RT;
            dot_input<RT>(sW[0] + (size_t)min(c, L.N - 1) * L.K, X + rb * P.K0p, P.K0p, L.K,
                         part + (c / G) * V + rb * G + c % G, G, c < L.N, L.vec != 0);
          }
        }
        else
          input_sums<R, G>(sW[0], L.K, L.N, X, P.K0p, P.ks0, P.kslice0, part, warp, lane, L.vec != 0);
        __syncthreads();
        for (int i = tid; i < R * L.N; i += kThreads)
        {
          const int r = i / L.N, c = i - r * L.N;
          float v = 0.0f;
          for (int s = 0; s < P.ks0; ++s)
            v += part[((c / G) * P.ks0 + s) * V + r * G + c % G];
          const float pre = lc[0].a * v + bias[L.noff + c];
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
        for (int i = tid; i < R * L.N; i += kThreads)
        {
          const int r = i / L.N, c = i - r * L.N;
          const size_t o = (size_t)(row0 + r) * L.N + c;
          mu0[r * P.N1p + c] = r < rows ? D.mu[o] : 0.0f;
          d0[r * P.N1p + c] = (r < rows && !simple) ? act_deriv(lc[0].act(), D.preact[o]) : 1.0f;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();

    // One forward task: partial sums of up to 32 outputs x RT rows (resident) or G x R (streamed).
    auto forward_task = [&](const ResTask& t)
    {
      const float* x = (simple ? Gb : Z) + t.x;
      float* out = X + t.out;
      const bool stream = t.kind & T_STREAM;
      if (!(t.kind & T_LANES))
      {
        const int row = min(lane, t.lanes - 1) * t.ldw;
        if (!stream)
          dot_resident<RT>(Ws + t.w + row, x, S, t.len, out + lane, t.pitch, lane < t.lanes);
        else
          dot_rows<RT>(sW[t.kind >> 4] + t.w + row, x, S, t.len, out + lane, t.pitch, lane < t.lanes,
                       (t.kind & T_VEC) != 0);
        return;
      }
      float acc[V];
#pragma unroll
      for (int i = 0; i < V; ++i)
        acc[i] = 0.0f;
      dot_streamed<R, G>(acc, (stream ? sW[t.kind >> 4] : Ws) + t.w, t.ldw, t.lanes, x, S, 0, t.len, lane,
                         (t.kind & T_VEC) != 0);
      const float v = reduce_values<V>(acc, lane);
      const int idx = lane / LPV, r = idx / G, c = idx % G;
      if (lane % LPV == 0 && c < t.lanes)
        out[r * t.pitch + c] = v;
    };
    auto state_of = [&](const ResTask& t)
    {
      const float* g = (simple ? E : Gb) + t.x;
      if (lane >= t.lanes)
        return;
      const int k = (t.kind & T_VEC) ? lane * 4 : lane;
      float* out = X + t.out + k;
      auto run = [&](auto kw)
      {
        constexpr int KW = decltype(kw)::value;
        float acc[RT][KW] = {};
        if (t.len > 0)
          state_sum<RT, KW, 2>(acc, Ws + t.w + k, t.ldw, t.len, g, S);
        if (t.len2 > 0)
          state_sum<RT, KW, RT == 1 ? 6 : RT == 2 ? 4 : 2>(acc, sW[t.kind >> 4] + t.w2 + k, sl[t.kind >> 4].K, t.len2, g + t.len, S);
#pragma unroll
        for (int r = 0; r < RT; ++r)
#pragma unroll
          for (int c = 0; c < KW; ++c)
            out[r * t.pitch + c] = acc[r][c];
      };
      if (t.kind & T_VEC)
        run(std::integral_constant<int, 4>());
      else
        run(std::integral_constant<int, 1>());
    };
    // Prediction of the four elements of quad q (layer l + 1) in row r, from the partial sums or the
    // clamped input layer's cache; padding comes out as zero.
    auto predict = [&](const ResQuad& q, int i4, int r, bool pred, float (&mu)[4], float (&d)[4])
    {
      const int l = q.layer - 1;
      if (l == 0)
      {
        get4(mu, mu0 + r * P.N1p + q.col);
        get4(d, d0 + r * P.N1p + q.col);
      }
      else
      {
        float pre[4], b[4];
        sum4(pre, X + q.fpart + r * q.pitch, q.fslices, R * q.pitch);
        get4(b, bias + 4 * i4);
        const LayerConst C = lc[l];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          pre[j] = C.a * pre[j] + b[j];
        if (simple)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            mu[j] = pre[j], d[j] = 1.0f;
        else
        {
          act4(C.act(), pre, mu, d);
          if (C.residual())
          {
            float z[4];
            get4(z, Z + r * S + q.down);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              mu[j] += z[j];
          }
        }
        if (pred && r < rows)
        {
          const dpc_layer& D = P.layers[l];
          const size_t o = (size_t)(row0 + r) * sl[l].N + q.col;
#pragma unroll
          for (int j = 0; j < 4; ++j)
            if (j < q.valid)
            {
              D.mu[o + j] = mu[j];
              if (D.preact)
                D.preact[o + j] = pre[j];
            }
        }
      }
#pragma unroll
      for (int j = 1; j < 4; ++j)
        if (j >= q.valid)
          mu[j] = d[j] = 0.0f;
    };
    // softmax cross-entropy error of the top layer from its logits (one warp per row)
    auto ce_error = [&](bool energy)
    {
      for (int r = warp; r < R; r += kWarps)
      {
        const float* m = topmu + r * NTp;
        const int to = sl[nw - 1].noff;
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
          const float p = expf(m[j] - mx) / s;
          const float z = Z[r * S + to + j];
          en -= z * logf(p + 1e-8f);
          const float e = z - p;
          E[r * S + to + j] = e;
          if (!simple)
            Gb[r * S + to + j] = e * topd[r * NTp + j];
        }
        if (energy && r < rows)
          esum += 2.0 * (double)en; // (halved at the end; cross-entropy is not)
      }
      __syncthreads();
    };

    // ---------------------------------------------------------------- forward sweep
    if (P.ops & DPC_ROWS_SWEEP)
    {
      int f = 0; // the task list is sorted by layer
      for (int l = 0; l < nw; ++l)
      {
        const ResLayer& L = sl[l];
        if (l > 0)
        {
          int t = f;
          while (t < P.nf && (ftab[t].kind >> 4) == l)
            ++t;
          for (int q = f + warp; q < t; q += kWarps)
            forward_task(ftab[q]);
          f = t;
          __syncthreads();
        }
        const bool copy = !(l + 1 == nw && P.top_clamped);
        const int n4 = (L.N + 3) >> 2;
        for (int idx = tid; idx < R * n4; idx += kThreads)
        {
          const int r = idx / n4, i = (L.noff >> 2) + idx - r * n4, o = r * S + 4 * i;
          const ResQuad q = quad[i];
          float mu[4], d[4];
          predict(q, i, r, (P.ops & DPC_ROWS_SWEEP_PRED) != 0, mu, d);
          if (copy)
          {
            put4(Z + o, mu);
            if (simple && l + 1 < nw)
            {
              float f4[4], d4[4];
              act4(lc[l + 1].act(), mu, f4, d4);
              put4(Gb + o, f4);
            }
          }
          if (l + 1 == nw) // the top prediction feeds the terminal error
          {
            put4(topmu + r * NTp + q.col, mu);
            put4(topd + r * NTp + q.col, d);
          }
        }
        __syncthreads();
      }
      if (P.ops & DPC_ROWS_TERMINAL)
      {
        if (P.ce)
          ce_error(false);
        else
        {
          const int to = sl[nw - 1].noff;
          for (int i = tid; i < R * NT; i += kThreads)
          {
            const int r = i / NT, c = i - r * NT;
            E[r * S + to + c] = Z[r * S + to + c] - topmu[r * NTp + c];
          }
          __syncthreads();
        }
      }
    }

    // Settling steps, then the closing passes.  One loop, so that the code of a pass -- activations of
    // four values in every kind -- exists once: with a copy per use the passes waited for instructions.
    // err: errors (and gated errors) are recomputed; else the gated errors are refreshed from the
    // errors that are there.
    const int refresh_at = (P.ops & DPC_ROWS_REFRESH) ? P.steps : -1;
    const int preact_at = (P.ops & DPC_ROWS_PREACT) ? P.steps + (refresh_at >= 0) : -1;
    const int energy_at =
        (P.ops & DPC_ROWS_ENERGY_LAST) ? P.steps + (refresh_at >= 0) + (preact_at >= 0) : -1;
    const int passes = P.steps + (refresh_at >= 0) + (preact_at >= 0) + (energy_at >= 0);
#pragma unroll 1
    for (int t = 0; t < passes; ++t)
    {
      const bool settles = t < P.steps, last = t + 1 == P.steps;
      const bool err = settles || t == energy_at;
      const bool gate = settles || t == refresh_at || (t == energy_at && (P.ops & DPC_ROWS_GATE_LAST));
      const bool energy = settles ? (P.ops & DPC_ROWS_ENERGY_EACH) != 0 : t == energy_at;
      const bool pred = settles ? last && (P.ops & DPC_ROWS_PRED_LAST)
                                : t == preact_at || (P.ops & DPC_ROWS_PRED_CLOSE) != 0;
      for (int q = warp; q < P.nf; q += kWarps)
        forward_task(ftab[q]);
      __syncthreads();
      float local = 0.0f;
      for_quads([&](const ResQuad& q, int i, int r)
                {
                  const int o = r * S + 4 * i;
                  float mu[4], d[4], e[4];
                  predict(q, i, r, pred, mu, d);
                  const bool ce_top = P.ce && q.layer == nw;
                  if (ce_top)
                  {
                    put4(topmu + r * NTp + q.col, mu);
                    put4(topd + r * NTp + q.col, d);
                  }
                  if (err && !ce_top)
                  {
                    float z[4];
                    get4(z, Z + o);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                      e[j] = z[j] - mu[j];
                      if (r < rows)
                        local += e[j] * e[j];
                    }
                    put4(E + o, e);
                  }
                  else
                    get4(e, E + o);
                  if (gate && !simple && !(err && ce_top))
                  {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                      e[j] *= d[j];
                    put4(Gb + o, e);
                  }
                });
      if (energy)
        esum += (double)local;
      __syncthreads();
      if (err && P.ce)
        ce_error(energy);
      if (!settles)
        continue;
      for (int q = warp; q < P.nb; q += kWarps)
        state_of(btab[q]);
      __syncthreads();
      const bool refresh_f = simple && !(last && !(P.ops & DPC_ROWS_ENERGY_LAST));
      for_quads([&](const ResQuad& q, int i, int r)
                {
                  const int l = q.layer, o = r * S + 4 * i;
                  if (l == nw && P.top_clamped)
                    return;
                  const LayerConst C = lc[l];
                  float z[4], e[4];
                  get4(z, Z + o);
                  get4(e, E + o);
                  if (l == nw || (P.top_down_off && l == nw - 1))
                  {
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                      z[j] -= C.ir * e[j];
                    put4(Z + o, z);
                    return;
                  }
                  float dz[4];
                  sum4(dz, X + q.bpart + r * q.pitch, q.bslices, R * q.pitch);
                  if (simple)
                  {
                    float f[4], d[4];
                    get4(f, Gb + o);
                    deriv4(C.act(), z, f, d);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                      z[j] += C.ir * (dz[j] * d[j] - e[j]);
                  }
                  else
                  {
                    float fb[4], u[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                      fb[j] = C.a * dz[j] - e[j];
                    if (P.has_v)
                    {
                      const float beta = C.beta;
                      float v[4];
                      get4(v, Vb + o);
#pragma unroll
                      for (int j = 0; j < 4; ++j)
                        fb[j] = beta * v[j] + (1.0f - beta) * fb[j];
                      put4(Vb + o, fb);
                    }
                    if (C.residual())
                      get4(u, E + r * S + q.up);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                    {
                      z[j] += C.ir * fb[j];
                      if (C.residual())
                        z[j] += C.ir * u[j];
                    }
                  }
#pragma unroll
                  for (int j = 1; j < 4; ++j)
                    if (j >= q.valid)
                      z[j] = 0.0f;
                  put4(Z + o, z);
                  if (refresh_f)
                  {
                    float f[4], d[4];
                    act4(C.act(), z, f, d);
                    put4(Gb + o, f);
                  }
                });
      __syncthreads();
    }
    if (P.ops & DPC_ROWS_LOGITS)
    {
      // the top belief becomes the prediction below it
      const int l = nw - 1;
      if (l > 0)
      {
        for (int t = warp; t < P.nf; t += kWarps)
          if ((ftab[t].kind >> 4) == l)
            forward_task(ftab[t]);
        __syncthreads();
      }
      const int n4 = NTp >> 2;
      for (int idx = tid; idx < R * n4; idx += kThreads)
      {
        const int r = idx / n4, i = (sl[l].noff >> 2) + idx - r * n4;
        float mu[4], d[4];
        predict(quad[i], i, r, true, mu, d);
        put4(Z + r * S + 4 * i, mu);
      }
      __syncthreads();
    }

    // ---------------------------------------------------------------- back to memory
    for_quads([&](const ResQuad& q, int i, int r)
              {
                if (r >= rows)
                  return;
                const int l = q.layer, o = r * S + 4 * i;
                const dpc_layer& L = P.layers[l];
                const size_t m = (size_t)(row0 + r) * sl[l - 1].N + q.col;
                const bool st_z = (P.ops & DPC_ROWS_STORE_Z) && !(l == nw && P.top_clamped);
                const bool st_e =
                    (P.ops & DPC_ROWS_STORE_E) || ((P.ops & DPC_ROWS_TERMINAL) && l == nw);
                float* fe = (P.ops & DPC_ROWS_STORE_G) && !simple ? P.layers[l - 1].fe : nullptr;
                float* zf = simple && l < nw && (P.ops & DPC_ROWS_STORE_Z) ? L.zF : nullptr;
                float* v = P.has_v && (P.ops & DPC_ROWS_STORE_V) ? L.v : nullptr;
                for (int j = 0; j < q.valid; ++j)
                {
                  if (st_z)
                    L.z[m + j] = Z[o + j];
                  if (st_e)
                    L.e[m + j] = E[o + j];
                  if (fe)
                    fe[m + j] = Gb[o + j];
                  if (zf)
                    zf[m + j] = Gb[o + j];
                  if (v)
                    v[m + j] = Vb[o + j];
                }
              });
    if (P.ops & DPC_ROWS_STORE_E)
    {
      float* e0 = P.layers[0].e + (size_t)row0 * sl[0].K;
      for (int i = tid; i < rows * sl[0].K; i += kThreads)
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

struct ResState
{
  ResParams P = {};
  int R = 1;
  size_t smem = 0;
  bool streams = false;
  void* dev = nullptr; // tables
};

inline int up4(int v)
{
  return (v + 3) & ~3;
}

// Tables for groups of R rows; 1 when they do not fit the shared memory.
int build(dpc_plan* p, int R, int S, bool has_v, bool exact)
{
  const int nw = p->n - 1, G = R == 8 ? 4 : 8, RT = std::min(R, 4), rbs = R / RT;
  std::vector<ResLayer> rl(nw);
  int off = 0;
  for (int l = 0; l < nw; ++l)
  {
    const dpc_layer& L = p->h[l];
    ResLayer& q = rl[l];
    q = ResLayer{};
    q.K = L.size, q.N = L.next_size;
    q.noff = off;
    q.zoff = l ? rl[l - 1].noff : 0;
    off += up4(q.N);
    q.vec = L.size % 4 == 0 && ((uintptr_t)L.W % 16) == 0;
    q.ldw = up4(L.size) | 4; // 4 x odd: lanes that read 16 bytes of neighbouring rows share no bank
    q.woff = q.rrows = 0;
    // (the shapes of the narrow forward kernel)
    q.lanes_k = exact && q.N <= 16 && q.K % 4 == 0 && q.K >= 128 && !(L.flags & DPC_LAYER_INPUT_ACT) &&
                ((uintptr_t)L.z % 16) == 0 && q.vec;
  }
  const int N1p = up4(rl[0].N), K0p = up4(rl[0].K), NTp = up4(rl[nw - 1].N);
  const int ng0 = (rl[0].N + G - 1) / G;
  int ks0 = exact ? 1 : std::max(1, std::min(2 * kWarps / std::max(ng0, 1), (K0p + 127) / 128));
  const int kslice0 = ((K0p + ks0 - 1) / ks0 + 3) & ~3;
  ks0 = (K0p + kslice0 - 1) / kslice0;

  std::vector<ResTask> ft, bt;
  size_t fparts = 0, bparts = 0;
  // Slices: a settling pass has one list for all layers, so a layer's tasks get its share of the warps
  // (rounded down: one round for all), a slice being worth its overhead from 16 inputs or output rows
  // on; halved while the partial sums of all layers take more than 32 KB.
  auto tasks = [&](int shift)
  {
    ft.clear(), bt.clear();
    fparts = bparts = 0;
    double fw = 0.0, bw = 0.0;
    for (int l = 1; l < nw; ++l)
    {
      ResLayer& q = rl[l];
      q.kw = q.K >= 96 && (q.rrows == q.N || q.vec) ? 4 : 1;
      fw += (double)((q.N + 31) / 32) * q.K;
      bw += (double)((q.K + 32 * q.kw - 1) / (32 * q.kw)) * q.kw * q.N;
    }
    for (int l = 1; l < nw; ++l)
    {
      ResLayer& q = rl[l];
      const int np = up4(q.N), kp = up4(q.K);
      q.fpart = (int)fparts;
      int s = 1;
      if (!exact)
      {
        const int blks = (q.N + 31) / 32;
        const double share = (double)blks * q.K / fw;
        s = std::max(1, std::min({(int)(kWarps * share / (blks * rbs) + 0.01), q.K / 16, 16}) >> shift);
      }
      q.fslice = ((q.K + s - 1) / s + 3) & ~3;
      s = q.rrows > 0 ? (q.K + q.fslice - 1) / q.fslice : 1;
      // forward: resident rows, then streamed ones
      for (int part = 0; part < 2; ++part)
      {
        const int n0 = part ? q.rrows : 0, n1 = part ? q.N : q.rrows;
        const bool lanes = q.lanes_k || (part && !exact);
        ResTask t = {};
        t.ldw = part ? q.K : q.ldw, t.pitch = np;
        t.kind = l << 4 | (part ? T_STREAM : 0) | (lanes ? T_LANES : 0) | (q.vec ? T_VEC : 0);
        if (lanes)
          for (int b = n0; b < n1; b += G)
          {
            t.w = (part ? 0 : q.woff) + b * t.ldw, t.x = q.zoff, t.len = q.K;
            t.out = q.fpart + b, t.lanes = n1 - b;
            ft.push_back(t);
          }
        else
          for (int rb = 0; rb < rbs; ++rb)
            for (int k = 0; k < (part ? 1 : s); ++k)
              for (int b = n0; b < n1; b += 32)
              {
                t.w = (part ? 0 : q.woff) + b * t.ldw + k * q.fslice;
                t.x = q.zoff + rb * RT * S + k * q.fslice;
                t.len = std::min(q.K - k * q.fslice, part ? q.K : q.fslice);
                t.out = q.fpart + (k * R + rb * RT) * np + b, t.lanes = std::min(32, n1 - b);
                ft.push_back(t);
              }
      }
      fparts += (size_t)s * R * np;
      // state: slices of the resident and of the streamed rows; exact: one sum over both
      const int cols = 32 * q.kw, blks = (q.K + cols - 1) / cols;
      q.bpart = (int)bparts;
      int slice = q.N;
      if (!exact)
      {
        const double share = (double)blks * q.kw * q.N / bw;
        const int want =
            std::max(1, std::min({(int)(kWarps * share / (blks * rbs) + 0.01), q.N / 8, 16}) >> shift);
        slice = ((q.N + want - 1) / want + 3) & ~3;
      }
      std::vector<std::pair<int, int>> cuts; // row ranges
      if (exact)
        cuts.push_back({0, q.N});
      else
        for (int part = 0; part < 2; ++part)
          for (int n = part ? q.rrows : 0; n < (part ? q.N : q.rrows); n += slice)
            cuts.push_back({n, std::min(n + slice, part ? q.N : q.rrows)});
      q.bslices = (int)cuts.size();
      for (int rb = 0; rb < rbs; ++rb)
        for (int k = 0; k < q.bslices; ++k)
          for (int b = 0; b < blks; ++b)
          {
            const int n0 = cuts[k].first, n1 = cuts[k].second;
            ResTask t = {};
            t.ldw = q.ldw;
            t.w = q.woff + n0 * q.ldw + b * cols;
            t.len = std::max(0, std::min(n1, q.rrows) - n0);
            t.w2 = (n0 + t.len) * q.K + b * cols;
            t.len2 = n1 - n0 - t.len;
            t.x = q.noff + rb * RT * S + n0;
            t.out = q.bpart + (k * R + rb * RT) * kp + b * cols, t.pitch = kp;
            t.lanes = std::min(32, (q.K - b * cols + q.kw - 1) / q.kw);
            t.kind = l << 4 | (q.kw == 4 ? T_VEC : 0);
            bt.push_back(t);
          }
      bparts += (size_t)q.bslices * R * kp;
    }
    return std::max(fparts, bparts) * sizeof(float) <= 32 * 1024;
  };
  auto fit_tasks = [&]()
  {
    for (int shift = 0; !tasks(shift) && shift < 4; ++shift)
      ;
  };
  auto round16 = [](size_t b) { return (b + 15) & ~(size_t)15; };
  auto table_bytes = [&]()
  {
    return round16(sizeof(ResLayer) * nw) + sizeof(ResQuad) * (S / 4) +
           sizeof(ResTask) * (std::max<size_t>(ft.size(), 1) + std::max<size_t>(bt.size(), 1));
  };
  auto others = [&]()
  {
    const size_t x = std::max({(size_t)R * K0p + (size_t)ng0 * ks0 * R * G, fparts, bparts});
    const size_t f = table_bytes() / sizeof(float) + S + (size_t)R * S * (has_v ? 4 : 3) +
                     2 * (size_t)R * N1p + 2 * (size_t)R * NTp + x;
    return f * sizeof(float) + kStatic;
  };
  // residency: smallest layers first, against what is left beside everything else; one that does not
  // fit whole keeps as many blocks of 32 rows as do
  for (int l = 1; l < nw; ++l)
    rl[l].rrows = rl[l].N;
  fit_tasks();
  size_t o = others();
  for (int l = 1; l < nw; ++l)
    rl[l].rrows = 0;
  fit_tasks();
  o = std::max(o, others()) + 4096; // (a layer in two parts has a few tasks and sums more)
  if (o > kSmemLimit)
    return 1;
  const size_t left = (kSmemLimit - o) / sizeof(float);
  size_t used = 0;
  std::vector<int> order;
  for (int l = 1; l < nw; ++l)
    order.push_back(l);
  std::sort(order.begin(), order.end(), [&](int a, int b)
            { return (size_t)rl[a].N * rl[a].ldw < (size_t)rl[b].N * rl[b].ldw; });
  for (int l : order)
  {
    const int fit = (int)std::min<size_t>((left - used) / rl[l].ldw, (size_t)rl[l].N);
    rl[l].rrows = fit == rl[l].N ? fit : fit / 32 * 32;
    rl[l].woff = (int)used;
    used += (size_t)rl[l].rrows * rl[l].ldw;
  }
  fit_tasks();
  o = others() + used * sizeof(float);
  if (o > kSmemLimit)
    return 1;
  std::vector<ResQuad> quads(S / 4);
  for (int l = 0; l < nw; ++l)
    for (int c = 0; c < rl[l].N; c += 4)
    {
      ResQuad& q = quads[(rl[l].noff + c) / 4];
      q = ResQuad{};
      q.layer = (short)(l + 1), q.col = c, q.valid = (short)std::min(4, rl[l].N - c);
      q.pitch = up4(rl[l].N);
      q.down = rl[l].zoff + c; // residual layers are square
      q.up = l + 1 < nw ? rl[l + 1].noff + c : 0;
      q.fpart = rl[l].fpart + c;
      // (columns of streamed rows, and heads walked along K, have one sum)
      q.fslices = l == 0 ? 0
                  : c < rl[l].rrows && !rl[l].lanes_k ? (short)((rl[l].K + rl[l].fslice - 1) / rl[l].fslice)
                                                      : 1;
      if (l + 1 < nw)
      {
        const ResLayer& U = rl[l + 1];
        q.bpart = U.bpart + c;
        q.bslices = (short)U.bslices;
      }
    }
  std::vector<unsigned char> host(table_bytes(), 0);
  size_t at = 0;
  auto put = [&](const void* src, size_t len)
  {
    const size_t here = at;
    if (len)
      memcpy(host.data() + at, src, len);
    at += round16(len);
    return (int)here;
  };
  auto* st = new ResState();
  ResParams& P = st->P;
  put(rl.data(), sizeof(ResLayer) * nw);
  P.a_quad = put(quads.data(), sizeof(ResQuad) * quads.size());
  P.nf = (int)ft.size(), P.nb = (int)bt.size();
  ft.resize(std::max<size_t>(ft.size(), 1)); // (a network of one weight layer has no tasks)
  bt.resize(std::max<size_t>(bt.size(), 1));
  P.a_ft = put(ft.data(), sizeof(ResTask) * ft.size());
  P.a_bt = put(bt.data(), sizeof(ResTask) * bt.size());
  P.table_vecs = (int)(at / 16);
  if (cudaMalloc(&st->dev, host.size()) != cudaSuccess ||
      cudaMemcpyAsync(st->dev, host.data(), host.size(), cudaMemcpyHostToDevice, p->ctx->stream) != cudaSuccess)
  {
    cudaFree(st->dev);
    delete st;
    return cuda_fail(cudaGetLastError(), "row-resident plan tables");
  }
  P.table = static_cast<const int4*>(st->dev);
  P.layers = p->d;
  P.top_n = rl[nw - 1].N;
  P.n = p->n, P.batch = p->batch, P.S = S;
  P.N1p = N1p, P.K0p = K0p, P.ks0 = ks0, P.kslice0 = kslice0;
  P.wfloats = (int)((used + 3) & ~(size_t)3);
  P.groups = (p->batch + R - 1) / R;
  P.simple = (p->h[0].flags & DPC_LAYER_INPUT_ACT) ? 1 : 0;
  P.has_v = has_v ? 1 : 0;
  P.exact = exact ? 1 : 0;
  P.energy = p->energy;
  for (int l = 1; l < nw; ++l)
    st->streams |= rl[l].rrows < rl[l].N;
  st->R = R;
  st->smem = o;
  p->res = st;
  return DPC_OK;
}
} // namespace

void res_plan_free(dpc_plan* p)
{
  auto* s = static_cast<ResState*>(p->res);
  if (!s)
    return;
  cudaFree(s->dev);
  delete s;
  p->res = nullptr;
}

bool res_plan_streams(const dpc_plan* p)
{
  return p->res && static_cast<const ResState*>(p->res)->streams;
}

// Which plans run here: by shape only.  Plans with tensor-core layers do not; the others do while
// re-reading the weights once per pass and row group from L2 costs less than the launches it saves.
int res_plan_init(dpc_plan* p)
{
  p->res = nullptr;
  if (getenv("DPC_DISABLE_RESIDENT"))
    return 1;
  const int n = p->n, nw = n - 1;
  if (n > kMaxLayers || p->run.count > 0 || tc_extra_layer(p, 0))
    return 1;
  size_t wbytes = 0;
  int S = 0;
  int longest = 0;
  bool has_v = false;
  const bool exact = ordered_sums(p);
  for (int l = 0; l < nw; ++l)
  {
    const dpc_layer& L = p->h[l];
    if (L.next_size <= 0 || L.next_size > 8192 || (l > 0 && L.size > 16384) ||
        ((L.flags ^ p->h[0].flags) & DPC_LAYER_INPUT_ACT) || (l == 0 && (L.flags & DPC_LAYER_RESIDUAL)))
      return 1;
    if (l > 0)
    {
      wbytes += sizeof(float) * (size_t)L.size * L.next_size;
      longest = std::max(longest, std::max(L.size, L.next_size));
    }
    has_v |= L.v != nullptr && l > 0;
    S += up4(L.next_size);
    if ((L.flags & DPC_LAYER_SOFTMAX_CE) || (l > 0 && tc_extra_layer(p, l)))
      return 1;
  }
  const size_t w0 = sizeof(float) * (size_t)p->h[0].size * p->h[0].next_size;
  int R = 1;
  while (R < 8 && (p->batch + R - 1) / R > p->ctx->sm_count)
    R *= 2;
  // Weights above the first layer that pay, against the phase kernels.  A segment's time grows with all
  // weights of a pass, a phase kernel's with the longest sum of one of its layers (`longest`), since it
  // takes the layers side by side.  Measured, segments / phase kernels in us a step of a DKP network with
  // 10 settling steps at batch 50, 300, 1000:
  //   sliced    64-512-310-10 (647 KB)  245/416  437/566  737/930    64-640-500-10  320/482  674/730  1090/1265
  //             64-(128x10)-10 (596 KB) 263/283  418/383  747/698    64-(64x38)-10  413/372  720/561  1434/993
  //             64-800-700-10  478/572, 1851/1242 at batch 600       64-(300x4)-10  368/335  628/558  1178/1040
  //   ordered   64-256-256-10 (272 KB)  207/302  318/349  526/550    64-384-256-10  291/340  393/386  752/649
  //             64-384-384-10 (605 KB)  399/368  576/456  2946/1246  64-512-310-10  429/415  621/566  1211/930
  const double limit_kb = exact ? (R == 1 ? 100 + 1.0 * longest : 60 + 0.85 * longest)
                                : (R == 1 ? 300 + 2.5 * longest : 100 + 2.5 * longest);
  // The input layer's weights, read once a step by every block.  Segments / phase kernels, geometric means by
  // their size, batch <= 148 and 149 to 592:       SimplePC ordered  sliced      feedback ordered  sliced
  //   0.9-2.5 MB                                    0.39 / 0.46      0.27 / 0.33     0.79 / 0.94    0.50 / 0.56
  //   2.5-4 MB                                      0.43 / 0.69      0.25 / 0.32     0.91 / 0.90    0.47 / 0.60
  //   4-8 MB                                        0.45 / 0.53      0.24 / 0.40     0.88 / 1.14    0.48 / 0.67
  // Feedback networks with ordered sums lose first: 1.12 at 593 to 1184 rows and 0.9-2 MB, 1.45 at 2.5-4.
  // The line is where they reach the phase kernels' time; the others would go on.
  if (wbytes > limit_kb * 1024 || w0 > 2560 * 1024)
    return 1;
  // Batches of more than one group of 8 rows per SM: a block walks its groups one after the other, reading
  // the streamed weights and those of the input layer again for each, while the phase kernels fill the GPU
  // better the larger the batch.  A network with feedback weights opens three segments a step, each with
  // weights and state to load, a SimplePC network one or two, and the input layer's weights are read once a
  // step: a quarter of the others' weight.  Limits on rounds x (input layer / 4 + others) in KB, from 3412
  // random networks (batch 200 to 4096, 2 to 20 settling steps).  Geometric means of segments / phase kernels
  // beyond one round were 1.10 (feedback, ordered sums; slowest 1.78) and 1.05 (sliced), 0.88 and 0.80
  // (SimplePC); within the limits 1.03, 1.01, 0.85 and 0.79.  Segments / phase kernels in us a step:
  //   ordered   DKP 784-(91x4)-100 at batch 3584, 2 steps 2043/1868    Full 400-256-256-2 at 3747, 6 steps 1551/870
  //             SimplePC 717-287-100 at 2816, 4 steps 952/697, 1500-85-85-85-10 at 2217, 12 steps 534/804 (kept)
  const long long rounds = ((long long)(p->batch + R - 1) / R + p->ctx->sm_count - 1) / p->ctx->sm_count;
  const bool feedback = !(p->h[0].flags & DPC_LAYER_INPUT_ACT);
  const double round_kb = exact ? (feedback ? 200 : 800) : (feedback ? 800 : 1600);
  if (rounds > 1 && rounds * (w0 / 4 + wbytes) > round_kb * 1024)
    return 1;
  for (; R >= 1; R /= 2)
  {
    const int rc = build(p, R, S, has_v, exact);
    if (rc <= 0)
      return rc;
  }
  return 1;
}

template <int R>
static int launch(dpc_plan* p, const ResState* st, const ResParams& P)
{
  static thread_local int configured = -1;
  if (configured != p->ctx->device)
  {
    DPC_CUDA(cudaFuncSetAttribute(resident_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)(kSmemLimit - kStatic)));
    configured = p->ctx->device;
  }
  const int grid = std::min(P.groups, p->ctx->sm_count);
  resident_kernel<R><<<grid, kThreads, st->smem - kStatic, p->ctx->stream>>>(P);
  p->ctx->launches += 1;
  const cudaError_t err = cudaPeekAtLastError();
  return err == cudaSuccess ? DPC_OK : cuda_fail(cudaGetLastError(), "row-resident kernel");
}
} // namespace dpc

using namespace dpc;

int dpc_rows_available(dpc_plan* p)
{
  return p && p->res ? 1 : 0;
}

int dpc_rows_segment(dpc_plan* p, int ops, int steps, int top_clamped, int top_down_off)
{
  if (!p || !(p->res || p->seg) || steps < 0)
    return fail(DPC_ERR_INVALID, "dpc_rows_segment: not a row-resident plan, or a bad step count");
  if (p->seg)
    return cluster_segment(p, ops, steps, top_clamped, top_down_off);
  const auto* st = static_cast<const ResState*>(p->res);
  ResParams P = st->P;
  P.ops = ops, P.steps = steps;
  P.top_clamped = top_clamped, P.top_down_off = top_down_off;
  P.ce = (p->h[p->n - 1].flags & DPC_LAYER_SOFTMAX_CE) ? 1 : 0;
  switch (st->R)
  {
  case 1:
    return launch<1>(p, st, P);
  case 2:
    return launch<2>(p, st, P);
  case 4:
    return launch<4>(p, st, P);
  default:
    return launch<8>(p, st, P);
  }
}
