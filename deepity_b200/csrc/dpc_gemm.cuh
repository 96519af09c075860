// CUDA-core (fp32 FFMA) products of every phase, any shape, with the fused predictive-coding epilogues.
#pragma once
#include "dpc_simt.cuh"

namespace dpc
{
enum GemmOp
{
  OP_FWD = 0, // mu = f(a z W^T + b)             M=B  N=next K=size
  OP_FB = 1,  // z += ir (a fe W - e)            M=B  N=size K=next
  OP_WG = 2   // W += alpha g^T zin              M=next N=size K=B
};
// mode of OP_FB
enum
{
  FB_STATE = 0,  // UpdateState
  FB_ADJOINT = 1 // ePC ComputeAdjoint + UpdateErrorEPC (fe holds src * f'(preact))
};

// The output tiles of a launch, as runs of neighbouring layers with equally many (deep networks have few: one for each
// shape; 240 are 3.9 KB of parameters, which a launch takes as fast as 0.5 KB).  The last parameter of a kernel: the
// others and the first runs then come in with the same line of the constant cache.
struct TileRun
{
  int start, per;       // its first tile, tiles of a layer
  unsigned inverse;     // (2^32 - 1) / per
  unsigned short layer; // its first layer, from the list's
  unsigned short kind;
};
constexpr int kListRuns = 240;
struct TileList
{
  int first, layers, runs;
  TileRun run[kListRuns];
};
// Layer of tile t, which becomes the index within the layer.
__device__ __forceinline__ int tile_layer(const TileList& T, int& t, bool& kind)
{
  if (T.layers == 1) // (the steps of a sweep, one short launch after another)
  {
    kind = T.run[0].kind != 0;
    return T.first;
  }
  int lo = 0;
  for (int hi = T.runs; hi - lo > 1;)
  {
    const int mid = (lo + hi) >> 1;
    if (T.run[mid].start <= t)
      lo = mid;
    else
      hi = mid;
  }
  const TileRun& r = T.run[lo];
  t -= r.start;
  int layer = (int)__umulhi((unsigned)t, r.inverse); // t / per or one less
  t -= layer * r.per;
  if (t >= r.per)
    ++layer, t -= r.per;
  kind = r.kind != 0;
  return T.first + r.layer + layer;
}

// Four neighbouring values of a row, of which `left` exist.
__device__ __forceinline__ void load4(float (&v)[4], const float* p, bool vec, int left)
{
  if (vec)
  {
    const float4 t = *reinterpret_cast<const float4*>(p);
    v[0] = t.x, v[1] = t.y, v[2] = t.z, v[3] = t.w;
  }
  else
#pragma unroll
    for (int j = 0; j < 4; ++j)
      v[j] = j < left ? p[j] : 0.0f;
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4], bool vec, int left)
{
  if (vec)
    *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
  else
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (j < left)
        p[j] = v[j];
}

// The fused epilogue of four neighbouring outputs (m, n .. n + 3).  vec: every tensor it touches can be
// accessed 16 bytes at a time.
template <int OP>
struct GemmEpilogue
{
  dpc_layer L;
  float *up_z, *up_e;
  bool vec, simple, do_err, do_fe, do_copy, store_pre, store_mu;
  int N, flags, mode, batch;
  float step;
  const float* epc_src;

  __device__ __forceinline__ GemmEpilogue(const dpc_layer& layer, const dpc_layer* Lup, int batch_, int flags_,
                                          int mode_, const float* src)
      : L(layer), up_z(Lup ? Lup->z : nullptr), up_e(Lup ? Lup->e : nullptr), flags(flags_), mode(mode_),
        batch(batch_), epc_src(src)
  {
    simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
    N = OP == OP_FWD ? L.next_size : L.size;
    const bool next_ce = Lup && (Lup->flags & DPC_LAYER_SOFTMAX_CE);
    do_err = (flags & DPC_FWD_ERR_NEXT) && Lup && !next_ce;
    do_fe = (flags & DPC_FWD_FE) && Lup && !simple && !(next_ce && (flags & DPC_FWD_ERR_NEXT));
    do_copy = (flags & DPC_FWD_COPY_NEXT) && Lup;
    const bool transient = (flags & DPC_FWD_TRANSIENT) != 0, no_mu = do_copy && (flags & DPC_FWD_NO_MU);
    store_pre = !transient && L.preact && !(no_mu && (flags & DPC_FWD_NO_PREACT));
    store_mu = !transient && !no_mu;
    auto at = [](const void* p) { return reinterpret_cast<uintptr_t>(p); };
    const uintptr_t all = OP == OP_FWD
                              ? at(L.b) | at(L.z) | at(L.preact) | at(L.mu) | at(L.fe) | at(up_z) | at(up_e)
                          : OP == OP_FB ? at(L.z) | at(L.e) | at(L.v) | at(up_e) | at(L.adj) | at(src)
                                        : at(L.W) | at(L.g_W) | at(L.m_W) | at(L.v_W);
    vec = N % 4 == 0 && (all & 15) == 0;
  }
  // (the Adam step size, two powers and a root: once per thread)
  __device__ __forceinline__ void prepare()
  {
    step = OP == OP_WG && mode == WG_LEARN && L.opt != DPC_OPT_SGD ? adam_step_size(L.lr, *L.t) : 0.0f;
  }

  // Tensors whose values at an output the epilogue starts from, fetched while the product is formed.
  static constexpr int kPre = OP == OP_WG ? 3 : 2;
  __device__ __forceinline__ const float* pre(int i) const
  {
    if (OP == OP_FWD)
      return i == 0 ? (do_err ? (do_copy ? nullptr : up_z) : do_fe ? up_e : nullptr)
                    : !simple && (L.flags & DPC_LAYER_RESIDUAL) ? L.z : nullptr;
    if (OP == OP_FB)
      return i == 0 ? L.e : mode == FB_ADJOINT ? nullptr : L.z;
    const bool adam = mode == WG_LEARN && L.opt != DPC_OPT_SGD;
    return mode & WG_GRAD_ONLY ? nullptr : i == 0 ? L.W : !adam ? nullptr : i == 1 ? L.m_W : L.v_W;
  }

  // x: what pre() names; returns the sum of the squared errors
  __device__ __forceinline__ float forward(int m, int n, const float (&sum)[4], const float (&b)[4],
                                           const float (&x)[kPre][4]) const
  {
    const size_t o = (size_t)m * N + n;
    const int left = N - n;
    float pre[4], mu[4], d[4], e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      pre[j] = L.a * sum[j] + b[j], mu[j] = pre[j], d[j] = 1.0f, e[j] = x[0][j];
    if (!simple)
    {
      if (do_fe)
        act_many<true>(L.act, pre, mu, d);
      else
        act_many<false>(L.act, pre, mu, d);
      if (L.flags & DPC_LAYER_RESIDUAL)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          mu[j] += x[1][j];
    }
    if (store_pre)
      store4(L.preact + o, pre, vec, left);
    if (store_mu)
      store4(L.mu + o, mu, vec, left);
    float energy = 0.0f;
    if (do_copy)
      store4(up_z + o, mu, vec, left);
    if (do_err)
    {
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        e[j] = (do_copy ? mu[j] : e[j]) - mu[j];
        if (j < left)
          energy += e[j] * e[j];
      }
      store4(up_e + o, e, vec, left);
    }
    if (do_fe)
    {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        e[j] *= d[j];
      store4(L.fe + o, e, vec, left);
    }
    return energy;
  }

  __device__ __forceinline__ void state(int m, int n, const float (&sum)[4], const float (&x)[kPre][4]) const
  {
    const size_t o = (size_t)m * N + n;
    const int left = N - n;
    float z[4], e[4];
#pragma unroll
    for (int j = 0; j < 4; ++j)
      e[j] = x[0][j], z[j] = x[1][j];
    if (mode == FB_ADJOINT)
    {
      // ePC: adjoint of this layer and the error update driven by it.  `flags` carries the
      // hop scale (+1 or -1) as float bits with bit 0 replaced by the clamp flag.
      const float scale = __int_as_float(flags & ~1);
      float adj[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
        adj[j] = (L.a * scale) * sum[j];
      if (L.flags & DPC_LAYER_RESIDUAL)
      {
        float s[4];
        load4(s, epc_src + o, vec, left);
#pragma unroll
        for (int j = 0; j < 4; ++j)
          adj[j] += scale * s[j];
      }
      store4(L.adj + o, adj, vec, left);
      if (!(flags & 1))
      {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          e[j] = (1.0f - L.ir) * e[j] - L.ir * adj[j];
        store4(L.e + o, e, vec, left);
      }
      return;
    }
    if (simple)
    {
      float d[4];
      act_deriv4(L.act, z, d);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        z[j] += L.ir * (sum[j] * d[j] - e[j]);
    }
    else
    {
      const bool residual = (L.flags & DPC_LAYER_RESIDUAL) != 0;
      float fb[4], v[4], u[4];
      if (L.v)
        load4(v, L.v + o, vec, left);
      if (residual)
        load4(u, up_e + o, vec, left);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        fb[j] = L.a * sum[j] - e[j];
      if (L.v)
      {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          fb[j] = fmaf(1.0f - L.momentum_beta, fb[j], L.momentum_beta * v[j]);
        store4(L.v + o, fb, vec, left);
      }
#pragma unroll
      for (int j = 0; j < 4; ++j)
        z[j] += L.ir * fb[j];
      if (residual)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          z[j] += L.ir * u[j];
    }
    store4(L.z + o, z, vec, left);
  }

  __device__ __forceinline__ void weights(int m, int n, const float (&sum)[4], const float (&x)[kPre][4]) const
  {
    const size_t o = (size_t)m * N + n;
    const int left = N - n;
    if (mode & WG_GRAD_ONLY)
    {
      store4(L.g_W + o, sum, vec, left);
      return;
    }
    float w[4];
    if (mode == WG_LEARN && L.opt != DPC_OPT_SGD)
    {
      // adam_update, its roundings spelled out as they always were here: of b2 v + (1 - b2) g^2 the compiler fuses one
      // product in this kernel and the other in those of bias and Psi, and an update of a near-zero gradient is
      // sensitive to which (an epoch of 16 AdamW steps ends 3 % apart)
      const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f, lr_wd = weight_wd(L);
      float mm[4], vv[4];
#pragma unroll
      for (int j = 0; j < 4; ++j)
      {
        const float g = -1.0f * L.a * sum[j];
        mm[j] = fmaf(b1, x[1][j], (1.0f - b1) * g);
        vv[j] = fmaf(b2, x[OP == OP_WG ? 2 : 0][j], (1.0f - b2) * (g * g));
        w[j] = lr_wd >= 0.0f ? fmaf(-lr_wd, x[0][j], x[0][j]) : x[0][j];
        w[j] -= step * mm[j] / (sqrtf(vv[j]) + eps);
      }
      store4(L.m_W + o, mm, vec, left);
      store4(L.v_W + o, vv, vec, left);
    }
    else
    {
      const Sgd update = weight_sgd(L, batch, mode == WG_DFA, (flags & 1) != 0);
#pragma unroll
      for (int j = 0; j < 4; ++j)
        w[j] = update(x[0][j], sum[j]);
    }
    store4(L.W + o, w, vec, left);
  }
};

// f(z) of four values of SimplePC's operand that this thread copied, in place; kept as last fed to the
// products for the weight update (src/layers/SimplePCLayer.cpp:146-150) by the first column of tiles.
__device__ __forceinline__ void feed4(const dpc_layer& L, float* p, int r, int k, int M, int K, bool vec, bool keep)
{
  if (r >= M || k >= K)
    return;
  float z[4], f[4], d[4];
  load4(z, p, true, 4);
  act_many<false>(L.act, z, f, d);
#pragma unroll
  for (int j = 1; j < 4; ++j)
    if (k + j >= K)
      f[j] = 0.0f;
  store4(p, f, true, 4);
  if (keep && L.zF)
    store4(L.zF + (size_t)r * K + k, f, vec && aligned16(L.zF), K - k);
}

// The grouped GEMM kernel: T x T output tiles, one CTA of W warps each; every output is one ascending sum over K
// whatever the tile (a belief that the sweep produced has an error of exactly zero in the passes that follow).
//   T = 32, W = 4: 8 x 32 outputs a warp, 2 x 4 per lane        few tiles: all schedulers of an SM on one
//   T = 32, W = 2: 16 x 32, 4 x 4 per lane                      several tiles an SM: fewer shared-memory reads
//   T = 64, W = 4: 32 x 32, 8 x 4 per lane                       many: half the operand traffic too
// Steps of 64, 32 and 16 K, twice as many with LONG: a step's copies, wait and barrier cost about 600 cycles beside the
// 25 a K of a lone 32 x 32 tile (1 600 cycles per 32 K as steps of 32, 1 150 as steps of 128).
// Operands come through a cp.async ring, 16 bytes at a time where rows start on 16-byte boundaries, else element
// by element; a warp reads contiguous bytes of few rows either way.  What bounds it: with several tiles an SM reads
// of shared memory (24, 16 and 12 cycles per k and 32 x 32 outputs, against 8 of the multiply-adds), else
// latencies: hence the operands of the next four k are read before the multiply-adds of these, what the epilogue
// starts from comes through shared memory with the operands, and there is one short copy of each loop (launches
// start with cold instruction caches).  us, 32 x 32 tiles of 2 x 2 outputs per thread before / now: 784 -> 256 at
// batch 256 22 / 19, 116 -> 116 at batch 64 7.1 / 5.5, six 445-wide layers at batch 48 24.7 / 16.5, three 403-wide
// ones at batch 512 67 / 44, thirteen 153-wide ones at batch 1421 68 / 56 and their weights 240 / 125.
template <int T_, int W_, bool LONG>
struct GemmTile
{
  static constexpr int T = T_, W = W_;
  static constexpr int BK = (T == 64 ? 16 : W == 4 ? 64 : 32) * (LONG ? 2 : 1), PITCH = BK + 4; // (the lanes' 16-byte reads share no bank)
  static constexpr int THREADS = 32 * W, TM = T == 32 ? 8 / W : 8;
  static constexpr int STAGES = T == 64 ? (LONG ? 3 : 4) : W == 4 || LONG ? 2 : 3, OPERAND = T * PITCH, SLOT = 2 * OPERAND;
  static constexpr int bytes(int pre) { return (STAGES * SLOT + (T == 32 ? pre : 0) * T * T) * (int)sizeof(float); }
};

// H lines of W contiguous elements from (h0, c0) of a matrix with `lines` lines of `width`, zeros beyond it.
template <int W, int H, int PITCH, int THREADS>
__device__ __forceinline__ void copy_tile(float* dst, const float* __restrict__ P, int ld, int h0, int lines, int c0,
                                          int width, bool vec)
{
  const int tid = threadIdx.x;
  if (vec)
  {
    constexpr int PER = THREADS / (W / 4); // lines per round
    const int c = tid % (W / 4) * 4, h = tid / (W / 4);
#pragma unroll
    for (int q = 0; q < H / PER; ++q)
    {
      const bool in = c0 + c < width && h0 + h + q * PER < lines;
      cp_async16(dst + (h + q * PER) * PITCH + c, in ? P + (size_t)(h0 + h + q * PER) * ld + c0 + c : P, in);
    }
  }
  else
  {
    constexpr int PER = THREADS / W;
    const int c = tid % W, h = tid / W;
#pragma unroll
    for (int q = 0; q < H / PER; ++q)
    {
      const bool in = c0 + c < width && h0 + h + q * PER < lines;
      cp_async4(dst + (h + q * PER) * PITCH + c, in ? P + (size_t)(h0 + h + q * PER) * ld + c0 + c : P, in);
    }
  }
}

template <int OP, typename C>
__global__ void __launch_bounds__(C::THREADS, C::T == 32 ? 20 / C::W : 4)
    pc_gemm_kernel(const dpc_layer* __restrict__ layers, int n_layers, int batch, int flags, int mode, double* energy,
                   const float* __restrict__ epc_src, const __grid_constant__ TileList list)
{
  constexpr int T = C::T, W = C::W, BK = C::BK, PITCH = C::PITCH, THREADS = C::THREADS, TM = C::TM, STAGES = C::STAGES;
  constexpr bool A_K = OP != OP_WG, B_K = OP == OP_FWD; // K contiguous in memory, else the tile's rows
  using Epilogue = GemmEpilogue<OP>;
  constexpr int PRE = T == 32 ? Epilogue::kPre : 0; // (64 x 64 tiles: others on the SM hide it)
  extern __shared__ __align__(16) float sm[]; // C::bytes(Epilogue::kPre)
  float* pre = sm + STAGES * C::SLOT;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int t = blockIdx.x;
  bool kind;
  const int li = tile_layer(list, t, kind);
  const dpc_layer* Lup = li + 1 < n_layers ? &layers[li + 1] : nullptr;
  Epilogue E(layers[li], Lup, batch, flags, mode, epc_src);
  const dpc_layer& L = E.L;
  const int base_mode = OP == OP_WG ? mode & ~WG_GRAD_ONLY : mode;
  const bool up_error = E.simple && base_mode == (OP == OP_WG ? (int)WG_LEARN : (int)FB_STATE);
  const int M = OP == OP_WG ? L.next_size : batch, N = E.N;
  const int K = OP == OP_FWD ? L.size : OP == OP_FB ? L.next_size : batch;
  const float* A = OP == OP_FWD ? L.z : up_error ? E.up_e : L.fe;
  const float* B = OP != OP_WG ? L.W : E.simple ? L.zF : L.z;
  const int lda = OP == OP_FWD ? L.size : L.next_size, ldb = L.size;
  const bool vec_a = aligned16(A) && lda % 4 == 0, vec_b = aligned16(B) && ldb % 4 == 0;
  const int nt = (N + T - 1) / T;
  const int m0 = t / nt * T, n0 = (t - t / nt * nt) * T;

  auto load = [&](int k0, int slot)
  {
    if (k0 < K)
    {
      float* dst = sm + slot * C::SLOT;
      if (A_K)
        copy_tile<BK, T, PITCH, THREADS>(dst, A, lda, m0, M, k0, K, vec_a);
      else
        copy_tile<T, BK, T, THREADS>(dst, A, lda, k0, K, m0, M, vec_a);
      dst += C::OPERAND;
      if (B_K)
        copy_tile<BK, T, PITCH, THREADS>(dst, B, ldb, n0, N, k0, K, vec_b);
      else
        copy_tile<T, BK, T, THREADS>(dst, B, ldb, k0, K, n0, N, vec_b);
    }
  };

  // This lane's outputs: rows am(i), columns bn(j).  K-major operands: every fourth row, every eighth column, whose
  // 16-byte reads along K fall into distinct banks; else neighbours.
  const int lm = lane >> 3, ln = lane & 7;
  const int wm = T == 32 ? 32 / W * warp : 32 * (warp >> 1), wn = T == 32 ? 0 : 32 * (warp & 1);
  auto am = [&](int i) { return wm + (A_K ? lm + 4 * i : lm * TM + i); };
  auto bn = [&](int j) { return wn + (B_K ? ln + 8 * j : 4 * ln + j); };
  float acc[TM][4] = {};
  struct Fragment // the lane's operands of four k
  {
    float a[4][TM], b[4][4];
  };
  auto read = [&](Fragment& f, const float* a, const float* b, int k)
  {
    if (A_K)
#pragma unroll
      for (int i = 0; i < TM; ++i)
      {
        const float4 v = *reinterpret_cast<const float4*>(a + am(i) * PITCH + k);
        f.a[0][i] = v.x, f.a[1][i] = v.y, f.a[2][i] = v.z, f.a[3][i] = v.w;
      }
    else
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int i = 0; i < TM; i += 2)
        {
          const float2 v = *reinterpret_cast<const float2*>(a + (k + q) * T + am(0) + i);
          f.a[q][i] = v.x, f.a[q][i + 1] = v.y;
        }
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (B_K)
      {
        const float4 v = *reinterpret_cast<const float4*>(b + bn(j) * PITCH + k);
        f.b[0][j] = v.x, f.b[1][j] = v.y, f.b[2][j] = v.z, f.b[3][j] = v.w;
      }
      else
      {
        const float4 v = *reinterpret_cast<const float4*>(b + (k + j) * T + bn(0));
        f.b[j][0] = v.x, f.b[j][1] = v.y, f.b[j][2] = v.z, f.b[j][3] = v.w;
      }
  };
  auto multiply = [&](const Fragment& f)
  {
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
      for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          acc[i][j] = fmaf(f.a[q][i], f.b[q][j], acc[i][j]);
  };

  const int column = n0 + tid % (T / 4) * 4; // of all quads that this thread finishes
  float bias[4] = {};
  int slot = 0, fill = 0;
#pragma unroll 1
  for (int k0 = -(STAGES - 1) * BK; k0 < K; k0 += BK)
  {
    float* a = sm + slot * C::SLOT;
    const float* b = a + C::OPERAND;
    if (k0 >= 0)
    {
      asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
      if (OP == OP_FWD && E.simple)
      {
        // SimplePC multiplies f(z)
        if (!vec_a)
          __syncthreads(); // (copied element by element by other threads)
        constexpr int PER = THREADS / (BK / 4);
        const int k = tid % (BK / 4) * 4, r = tid / (BK / 4);
#pragma unroll 1
        for (int q = 0; q < T / PER; ++q)
          feed4(L, a + (r + q * PER) * PITCH + k, m0 + r + q * PER, k0 + k, M, K, vec_a, n0 == 0);
      }
      __syncthreads(); // the step has landed, and everybody is done with the slot that is refilled now
    }
    load(k0 + (STAGES - 1) * BK, fill);
    fill = fill + 1 == STAGES ? 0 : fill + 1;
    if (k0 == -BK)
    {
#pragma unroll
      for (int i = 0; i < PRE; ++i)
        if (const float* p = E.pre(i))
          copy_tile<T, T, T, THREADS>(pre + i * T * T, p, N, m0, M, n0, N, aligned16(p) && N % 4 == 0);
      if (OP == OP_FWD && column < N)
        load4(bias, L.b + column, E.vec, N - column);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    if (k0 < 0)
      continue;
    if (T == 64)
    {
#pragma unroll 2
      for (int k = 0; k < BK; k += 4)
      {
        Fragment f;
        read(f, a, b, k);
        multiply(f);
      }
    }
    else
    {
      Fragment f0, f1;
      read(f0, a, b, 0);
      const int left = K - k0;
#pragma unroll 1
      for (int k = 0; k < BK && k < left; k += 8)
      {
        read(f1, a, b, k + 4);
        multiply(f0);
        read(f0, a, b, k + 8); // (at the step's end the padding behind it, unused)
        multiply(f1);
      }
    }
    slot = slot + 1 == STAGES ? 0 : slot + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  // sums to shared memory as rows of T, then four neighbours per thread
#pragma unroll
  for (int i = 0; i < TM; ++i)
    if (B_K)
#pragma unroll
      for (int j = 0; j < 4; ++j)
        sm[am(i) * T + bn(j)] = acc[i][j];
    else
      *reinterpret_cast<float4*>(sm + am(i) * T + bn(0)) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  E.prepare();
  __syncthreads();
  float esum = 0.0f;
#pragma unroll 1
  for (int q = tid; q < T * T / 4; q += THREADS)
  {
    const int m = m0 + q / (T / 4);
    if (m >= M || column >= N)
      break;
    float s[4], x[Epilogue::kPre][4] = {};
    load4(s, sm + 4 * q, true, 4);
#pragma unroll
    for (int i = 0; i < Epilogue::kPre; ++i)
      if (const float* p = E.pre(i))
      {
        if (PRE > 0)
          load4(x[i], pre + i * T * T + 4 * q, true, 4);
        else
          load4(x[i], p + (size_t)m * N + column, E.vec, N - column);
      }
    if (OP == OP_FWD)
      esum += E.forward(m, column, s, bias, x);
    else if (OP == OP_FB)
      E.state(m, column, s, x);
    else
      E.weights(m, column, s, x);
  }
  if (OP == OP_FWD && (flags & DPC_FWD_ENERGY))
  {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
      esum += __shfl_xor_sync(0xffffffffu, esum, o);
    __syncthreads();
    if (lane == 0)
      sm[warp] = esum;
    __syncthreads();
    if (tid == 0)
    {
      float s = 0.0f;
      for (int w = 0; w < THREADS / 32; ++w)
        s += sm[w];
      atomicAdd(energy, (double)(0.5f * s));
    }
  }
}
} // namespace dpc
