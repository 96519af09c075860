// Sums over the batch of a learning phase, for layers outside the tensor-core kernels of networks whose sums
// may be split: weight gradients g^T z, bias gradients (column sums of g) and feedback-weight gradients
// z^T e_T, each with its update.
#pragma once
#include "dpc_gemm.cuh"

namespace dpc
{
// One launch for all of them.  A CTA owns a 32 x 32 tile of one product; its eight warps take every eighth
// group of eight batch rows, each warp all 1024 outputs (8 x 4 per lane, three 16-byte shared-memory reads
// per 32 multiply-adds), with a cp.async ring of its own, so that the row loop holds no barrier.  The CTAs of
// a cluster (R along x) split the groups further where a launch would leave SMs idle.  Partial sums meet
// through shared memory, first the warps', then the cluster's, in a fixed order.
//
// What bounds it: such a launch has few outputs and a batch of rows to walk, so it is the chain of row loads
// and the shared-memory reads of one SM.  (A tile that walked the whole batch step by step with 2 x 2 outputs
// per thread took 0.5 us per 16 rows, beside kernels of their own for bias and Psi.)  A step of 22 layers of 45
// units at batch 2167 769 -> 560 us, of 784-(256x8)-10 at batch 256 302 -> 268; the learn phase of
// 32-32-2 at batch 715 38 -> 6 us.  Weights of twelve tiles an SM and more are left to pc_gemm_kernel (weights_by_gemm
// in dpc_core.cu).
constexpr int BP_T = 32, BP_ROWS = 8, BP_WARPS = 8, BP_STAGES = 3;
constexpr int BP_SLOT = 2 * BP_ROWS * BP_T; // floats: rows of g, rows of z

struct BatchTiles
{
  int sums;      // their bias sums and the Psi sums of all layers are among them
  TileList list; // kind: the weight sums of these layers are
};

__device__ __forceinline__ float4 rows_cluster_load4(const float* own, uint32_t rank)
{
  const uint32_t a = (uint32_t)__cvta_generic_to_shared(own);
  uint32_t ra;
  float4 v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(ra) : "r"(a), "r"(rank));
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(ra)
               : "memory");
  return v;
}

__global__ void __launch_bounds__(32 * BP_WARPS, 2)
    batch_product_kernel(const dpc_layer* __restrict__ layers, int batch, int flags, int mode,
                         const float* __restrict__ eT, const __grid_constant__ BatchTiles T)
{
  const uint32_t R = rows_cluster_size(), rank = rows_cluster_rank();
  int t = (int)(blockIdx.x / R);
  bool weights;
  const int li = tile_layer(T.list, t, weights);
  const dpc_layer L = layers[li];
  const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
  const int base_mode = mode & ~WG_GRAD_ONLY;
  const int N = L.size, nt = (N + BP_T - 1) / BP_T;
  const int mt = weights ? (L.next_size + BP_T - 1) / BP_T : 0;
  int m0 = t / nt;
  const int n0 = (t - m0 * nt) * BP_T;
  const bool psi = m0 >= mt;
  m0 = (psi ? m0 - mt : m0) * BP_T;
  const int M = psi ? L.terminal_size : L.next_size; // also the row pitch of A
  const float* A = psi ? eT : simple && base_mode == WG_LEARN ? layers[li + 1].e : L.fe;
  const float* B = simple ? L.zF : L.z;
  const bool vecA = aligned16(A) && M % 4 == 0, vecB = aligned16(B) && N % 4 == 0;
  const bool bias = T.sums && !psi && n0 == 0;

  __shared__ __align__(16) float sm[BP_WARPS * BP_STAGES * BP_SLOT];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float* ring = sm + warp * (BP_STAGES * BP_SLOT);
  const int groups = (batch + BP_ROWS - 1) / BP_ROWS, stride = BP_WARPS * (int)R;
  auto copy = [&](float* dst, const float* G, int ld, int c0, bool vec, int r0)
  {
    if (vec)
    {
#pragma unroll
      for (int q = 0; q < BP_ROWS * BP_T / 128; ++q)
      {
        const int r = q * 4 + (lane >> 3), c = (lane & 7) * 4;
        const bool in = r0 + r < batch && c0 + c < ld;
        cp_async16(dst + r * BP_T + c, in ? G + (size_t)(r0 + r) * ld + c0 + c : G, in);
      }
    }
    else
    {
#pragma unroll
      for (int r = 0; r < BP_ROWS; ++r)
      {
        const bool in = r0 + r < batch && c0 + lane < ld;
        cp_async4(dst + r * BP_T + lane, in ? G + (size_t)(r0 + r) * ld + c0 + lane : G, in);
      }
    }
  };
  auto load = [&](int g, int slot)
  {
    if (g < groups)
    {
      float* dst = ring + slot * BP_SLOT;
      copy(dst, A, M, m0, vecA, g * BP_ROWS);
      copy(dst + BP_ROWS * BP_T, B, N, n0, vecB, g * BP_ROWS);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  // This lane's outputs: 8 rows from mg, 4 columns from ng; 4 rows where the tile has 16 at most (a tile of
  // ten terminal units): reads of shared memory bound the loop, 12 floats a row and lane then become 8.
  const bool narrow = M - m0 <= BP_T / 2;
  const int mg = (lane >> 3) * (narrow ? 4 : 8), ng = (lane & 7) * 4;
  float acc[8][4] = {}, bsum = 0.0f;
  const int g0 = (int)rank * BP_WARPS + warp;
#pragma unroll
  for (int q = 0; q < BP_STAGES - 1; ++q)
    load(g0 + q * stride, q);
  // What this thread will update -- a quad of outputs, row q / 8, columns 4 (q % 8).., of its CTA's share of the
  // tile, and a bias -- fetched while the sums are formed.
  const int share = 32 * BP_WARPS / (int)R, q = (int)rank * share + (int)threadIdx.x;
  const int m = m0 + (q >> 3), n = n0 + (q & 7) * 4;
  const bool mine = (int)threadIdx.x < share && m < M && n < N, grad_only = (mode & WG_GRAD_ONLY) != 0;
  const bool my_bias = bias && rank == 0 && threadIdx.x < BP_T && m0 + (int)threadIdx.x < M;
  const bool vec = N % 4 == 0 && aligned16(L.W) && aligned16(L.g_W);
  float old[4] = {}, old_bias = 0.0f;
  if (mine && !grad_only)
  {
    if (!psi)
      load4(old, L.W + (size_t)m * N + n, vec, N - n);
    else
#pragma unroll
      for (int j = 0; j < 4; ++j)
        old[j] = n + j < N ? L.Psi[(size_t)(n + j) * L.psi_stride + m] : 0.0f;
  }
  if (my_bias && !grad_only)
    old_bias = L.b[m0 + threadIdx.x];
  int slot = 0;
  for (int g = g0; g < groups; g += stride)
  {
    asm volatile("cp.async.wait_group %0;" ::"n"(BP_STAGES - 2) : "memory");
    __syncwarp(); // the group has landed for all lanes, and all are done with the slot refilled now
    load(g + (BP_STAGES - 1) * stride, slot == 0 ? BP_STAGES - 1 : slot - 1);
    const float* a = ring + slot * BP_SLOT;
    const float* b = a + BP_ROWS * BP_T;
    auto rows = [&](auto count)
    {
      constexpr int TM = decltype(count)::value;
#pragma unroll
      for (int k = 0; k < BP_ROWS; ++k)
      {
        float av[TM];
#pragma unroll
        for (int i = 0; i < TM; i += 4)
        {
          const float4 a4 = *reinterpret_cast<const float4*>(a + k * BP_T + mg + i);
          av[i] = a4.x, av[i + 1] = a4.y, av[i + 2] = a4.z, av[i + 3] = a4.w;
        }
        const float4 b4 = *reinterpret_cast<const float4*>(b + k * BP_T + ng);
        const float bv[4] = {b4.x, b4.y, b4.z, b4.w};
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j)
            acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      }
    };
    if (narrow)
      rows(std::integral_constant<int, 4>());
    else
      rows(std::integral_constant<int, 8>());
    if (bias)
#pragma unroll
      for (int k = 0; k < BP_ROWS; ++k)
        bsum += a[k * BP_T + lane];
    slot = slot + 1 == BP_STAGES ? 0 : slot + 1;
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();

  // ---- the warps' sums, then the cluster's
  constexpr int TILE = BP_T * BP_T;
  float* bpart = sm + BP_WARPS * TILE;  // [warps][32]
  float* cta = bpart + BP_WARPS * BP_T; // this CTA's sums: [32][32], then the bias's [32]
  static_assert(BP_WARPS * (TILE + BP_T) + TILE + BP_T <= BP_WARPS * BP_STAGES * BP_SLOT, "sums fit the rings");
#pragma unroll
  for (int i = 0; i < 8; ++i)
    if (i < 4 || !narrow)
      *reinterpret_cast<float4*>(sm + warp * TILE + (mg + i) * BP_T + ng) =
          make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
  if (bias)
    bpart[warp * BP_T + lane] = bsum;
  __syncthreads();
  const int busy = min(BP_WARPS, groups - (int)rank * BP_WARPS); // warps that had rows
  float4 s = *reinterpret_cast<const float4*>(sm + 4 * threadIdx.x);
#pragma unroll
  for (int w = 1; w < BP_WARPS; ++w)
    if (w < busy)
    {
      const float4 v = *reinterpret_cast<const float4*>(sm + w * TILE + 4 * threadIdx.x);
      s.x += v.x, s.y += v.y, s.z += v.z, s.w += v.w;
    }
  float bs = 0.0f;
  if (bias && threadIdx.x < BP_T)
    for (int w = 0; w < busy; ++w)
      bs += bpart[w * BP_T + threadIdx.x];
  if (R > 1)
  {
    *reinterpret_cast<float4*>(cta + 4 * threadIdx.x) = s;
    if (bias && threadIdx.x < BP_T)
      cta[TILE + threadIdx.x] = bs;
    rows_cluster_sync();
    // every CTA finishes its share of the tile; the first one the bias too (all loads before the first use)
    if ((int)threadIdx.x < share)
    {
      float4 v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        if (r < (int)R)
          v[r] = rows_cluster_load4(cta + 4 * q, r);
      s = v[0];
#pragma unroll
      for (int r = 1; r < 8; ++r)
        if (r < (int)R)
          s.x += v[r].x, s.y += v[r].y, s.z += v[r].z, s.w += v[r].w;
    }
    if (bias && rank == 0 && threadIdx.x < BP_T)
    {
      float v[8];
#pragma unroll
      for (int r = 1; r < 8; ++r)
        if (r < (int)R)
          v[r] = rows_cluster_load(cta + TILE + threadIdx.x, r);
#pragma unroll
      for (int r = 1; r < 8; ++r)
        if (r < (int)R)
          bs += v[r];
    }
    rows_cluster_sync(); // nobody leaves while its sums may still be read
  }
  // (every optimizer of these networks is SGD)
  if (my_bias)
    (grad_only ? L.g_b : L.b)[m0 + threadIdx.x] = grad_only ? bs : bias_sgd(L, batch)(old_bias, bs);
  if (!mine)
    return;
  float out[4] = {s.x, s.y, s.z, s.w};
  if (!grad_only)
  {
    const Sgd update = psi ? psi_sgd(L, batch) : weight_sgd(L, batch, mode == WG_DFA, (flags & 1) != 0);
#pragma unroll
    for (int j = 0; j < 4; ++j)
      out[j] = update(old[j], out[j]);
  }
  if (!psi)
    store4((grad_only ? L.g_W : L.W) + (size_t)m * N + n, out, vec, N - n);
  else
  {
    float* dst = grad_only ? L.g_Psi : L.Psi;
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (n + j < N)
        dst[(size_t)(n + j) * L.psi_stride + m] = out[j];
  }
}
} // namespace dpc
