// The sequential forward sweep over layers of 256 or 512 units on clusters; part of dpc_tc.cu.
//
// Rows of the batch are independent of each other, so a cluster can walk all layers with a few rows by itself.  Its
// beliefs never leave shared memory on the dependent path: block r of H / 128 forms outputs 128 r .. 128 r + 127 of every
// layer for the cluster's 8, 16 or 32 rows -- D[output][row], so that the weights are the 128-row operand A of
// tcgen05.mma and the beliefs the operand B -- and hands them, as operands of the next layer, to the other blocks: with
// st.async, or where a block's 128 k are whole 128-byte rows (32 rows) as bulk copies, either way counted in bytes on a
// barrier of their source.  A block multiplies its own half of K first.  Weights stream
// through a TMA ring that does not wait for anything of the chain.
//
//   beliefs      [k][rows], 128 bytes a k: the rows' bf16 "hi" values, then their "mid" values, one MN-major block
//                (128-byte swizzle), or up to 32 fp32 values (TF32: swizzle of 32-byte units); two buffers
//   products     two sums, one per half of K, that the epilogue adds: the K-split tiles' order of additions, so that their
//                bits stay (the errors right after a sweep are its rounding against the settling passes': another order
//                of the same accuracy moved those of 512 layers by 1e-3).  bf16 planes: x_hi w_hi and x_mid w_hi onto one
//                accumulator, x_hi w_mid onto another; TF32: one pass
//   fp32 beliefs and operand planes in global memory are written beside the next layer's multiplications
//
// What bounds a layer, in cycles of 512 units and 32 rows (bf16; 9 500 in all, 7 300 with TF32): 96 multiplications (40 each
// where nothing else reads shared memory), tensor memory -> activation -> own shared memory 1 500, waits for the other
// blocks' outputs 700 (between blocks 15 to 20 bytes a cycle leave an SM whichever instruction moves them; sent without an
// order of the targets they took 1 550) and for weights 1 200 (a layer's 256 KB an SM at 30 bytes a cycle).
// us, tiles that publish their rows in global memory -> this: 512 layers of 512 units at batch 1024 4202 -> 2845; 12 of
// them with TF32 88 -> 60; 24 of 512 at batch 256 168 -> 100; 8 of 256 units at batch 256 44 -> 19, 29 residual ones
// 203 -> 66; 24 of 256 at batch 2048 150 -> 90.
#pragma once

template <int ROWS>
constexpr int kSweepThreads = 32 * (2 + ROWS / 2 + (ROWS == 32 ? 1 : 0)); // weights, multiplications, epilogue, copies

template <bool TF32, int ROWS>
__global__ void __launch_bounds__(kSweepThreads<ROWS>, 1)
    cluster_sweep_kernel(const __grid_constant__ CUtensorMap mapW, const TcParams P, int H, int stages, int target_bias)
{
  constexpr int STAGE_BYTES = 32768, KB = 64; // a stage: 128 outputs x 64 k, both planes
  constexpr int GROUPS = ROWS / 8;            // of four epilogue warps
  constexpr bool BULK = ROWS == 32;
  constexpr int HALF = ROWS < 16 ? 16 : ROWS; // columns of the "hi" values (N of an instruction is a multiple of 16)
  constexpr uint32_t COLUMNS = 4 * HALF;      // tensor memory: "hi" and "mid" sums of each half of K
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  uint8_t* zbuf = smem; // two buffers of H x 128 bytes
  uint8_t* ring = smem + 2 * H * 128;
  uint64_t* full = reinterpret_cast<uint64_t*>(ring + stages * STAGE_BYTES);
  uint64_t* empty = full + 8;
  uint64_t* tfull = empty + 8;
  uint64_t* zfull = tfull + 1;  // [buffer][source]: its part of the next layer's operand is there
  uint64_t* slab = zfull + 8;   // [buffer][quarter]: all groups have written their rows of 32 outputs
  uint32_t* tmem_holder = reinterpret_cast<uint32_t*>(slab + 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_holder + 2); // as in pc_tc_kernel
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int blocks = H / 128;
  const uint32_t rank = cluster_ctarank();
  const int row0 = (int)(blockIdx.x / blocks) * ROWS, j0 = 128 * (int)rank;
  constexpr int SOURCE_KB = 128 / KB; // k blocks of a source

  if (threadIdx.x == 0)
  {
    for (int s = 0; s < 8; ++s)
    {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tfull, 1);
    for (int b = 0; b < 2; ++b)
      for (int q = 0; q < 4; ++q)
        mbar_init(&zfull[4 * b + q], q == (int)rank ? 4 * GROUPS : 1);
    for (int q = 0; q < 8; ++q)
      mbar_init(&slab[q], GROUPS);
    *abort_flag = 0;
    *reinterpret_cast<volatile long long*>(abort_flag + 2) = P.wait_cycles;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1)
  {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_holder)),
                 "r"(COLUMNS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // The block whose outputs are multiplied i-th: the own half of K first, each half in ascending order.
  auto source = [&](int i) { return blocks == 2 ? (int)rank ^ i : (((int)rank & 2) ^ (i & 2)) | (i & 1); };
  // Eight rows of one k as operand values: two 16-byte chunks at these offsets of a buffer.
  auto chunk = [](int k, int rows8, int half)
  {
    return TF32 ? k * 128 + ((rows8 ^ (k & 3)) << 5) + (half << 4)
                : k * 128 + (((half * (HALF >> 3) + rows8) ^ (k & 7)) << 4);
  };
  auto operands = [](const float* v, uint4 (&q)[2])
  {
    const float4 a = make_float4(v[0], v[1], v[2], v[3]), b = make_float4(v[4], v[5], v[6], v[7]);
    if (TF32)
    {
      q[0] = *reinterpret_cast<const uint4*>(&a);
      q[1] = *reinterpret_cast<const uint4*>(&b);
    }
    else
      split8(a, b, q[0], q[1]);
  };
  // the first layer's input, by every block
  {
    const float* z = P.layers[P.first].z + (size_t)row0 * H;
    for (int i = threadIdx.x; i < H * GROUPS; i += blockDim.x)
    {
      const int k = i & (H - 1), r8 = i / H;
      float v[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        v[r] = z[(size_t)(8 * r8 + r) * H + k];
      uint4 q[2];
      operands(v, q);
      *reinterpret_cast<uint4*>(zbuf + chunk(k, r8, 0)) = q[0];
      *reinterpret_cast<uint4*>(zbuf + chunk(k, r8, 1)) = q[1];
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  }
  tc_fence_before();
  cluster_sync_all();
  tc_fence_after();
  const uint32_t tmem = *tmem_holder;

  if (warp == 0)
  {
    // ---------------------------------------------------------------- weights
    if (lane == 0)
    {
      int s = 0;
      uint32_t phase = 1;
      bool alive = true;
      for (int l = 0; l < P.count && alive; ++l)
      {
        const int layer = P.first + l - P.run_first;
        for (int i = 0; i < blocks * SOURCE_KB; ++i)
        {
          const int kb = SOURCE_KB * source(i / SOURCE_KB) + i % SOURCE_KB;
          if (!mbar_wait(&empty[s], phase, abort_flag))
          {
            alive = false;
            break;
          }
          uint8_t* to = ring + s * STAGE_BYTES;
          mbar_expect_tx(&full[s], STAGE_BYTES);
          for (int half = 0; half < 2; ++half)
            if (TF32)
              tma_load_3d(to + half * 16384, &mapW, &full[s], kb * KB + 32 * half, j0, layer);
            else
              tma_load_3d(to + half * 16384, &mapW, &full[s], kb * KB, j0, 2 * layer + half);
          if (++s == stages)
            s = 0, phase ^= 1;
        }
      }
    }
  }
  else if (warp == 1)
  {
    // ---------------------------------------------------------------- multiplications (the warp together, one lane issues)
    constexpr uint32_t FMT = TF32 ? 2u : 1u;
    constexpr uint32_t BASE = (1u << 4) | (FMT << 7) | (FMT << 10) | (1u << 16) | ((uint32_t)(128 >> 4) << 24);
    constexpr uint32_t ONE = BASE | ((uint32_t)(HALF >> 3) << 17);
    constexpr uint32_t BYTES = BULK ? 128 * 128 : 128 * 4 * ROWS;
    const uint64_t da0 = make_desc(smem_u32(ring), 16, 1024, 2);
    const uint64_t db0 = make_desc(smem_u32(zbuf), 8192, TF32 ? 512 : 1024, TF32 ? 1 : 2);
    const int half_kb = blocks * SOURCE_KB / 2;
    int s = 0;
    uint32_t phase = 0;
    bool alive = true;
    for (int l = 0; l < P.count && alive; ++l)
    {
      uint64_t* ready = zfull + 4 * (l & 1);
      if (lane == 0)
        for (int q = 1; l > 0 && q < blocks; ++q)
          mbar_expect_tx(&ready[(rank + q) & (blocks - 1)], BYTES + 16 * target_bias);
      __syncwarp();
      for (int i = 0; i < blocks * SOURCE_KB; ++i)
      {
        const int kb = SOURCE_KB * source(i / SOURCE_KB) + i % SOURCE_KB;
        // A layer's first multiplications overwrite the sums.  What orders them behind this block's epilogue of the layer
        // below, which loads them, is its own part of the operand: with two blocks, and for the even ones of four, that is
        // also the part that is multiplied first; the odd ones of four begin with another block's, which may be here while
        // their own epilogue still loads (a block whose weights came late), so all wait for both.
        if (l > 0 && i == 0)
          alive = __all_sync(0xffffffffu, mbar_wait_cluster(&ready[rank], ((l - 1) >> 1) & 1, abort_flag));
        if (l > 0 && i % SOURCE_KB == 0)
        {
          alive = alive && __all_sync(0xffffffffu, mbar_wait_cluster(&ready[kb / SOURCE_KB], ((l - 1) >> 1) & 1, abort_flag));
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        }
        alive = alive && __all_sync(0xffffffffu, mbar_wait(&full[s], phase, abort_flag));
        if (!alive)
          break;
        tc_fence_after();
        const uint32_t sum = tmem + (uint32_t)(i < half_kb ? 0 : 2 * HALF);
        const uint64_t da = da0 + (uint64_t)(s * (STAGE_BYTES >> 4));
        const uint64_t db = db0 + (uint64_t)(((l & 1) * H + kb * KB) * (128 >> 4));
#pragma unroll
        for (int ks = 0; ks < (TF32 ? 8 : 4); ++ks)
        {
          const uint32_t more = ks > 0 || i % half_kb != 0;
          if (TF32)
            tc_mma_tf32(sum, da + (uint64_t)((ks >> 2) * (16384 >> 4) + (ks & 3) * (32 >> 4)),
                              db + (uint64_t)(ks * (1024 >> 4)), ONE, more);
          else
          {
            const uint64_t wh = da + (uint64_t)(ks * (32 >> 4)), bh = db + (uint64_t)(ks * (2048 >> 4));
            tc_mma_bf16(sum, wh, bh, ONE, more);
            tc_mma_bf16(sum, wh, bh + (uint64_t)((2 * HALF) >> 4), ONE, 1);
            tc_mma_bf16(sum + HALF, wh + (uint64_t)(16384 >> 4), bh, ONE, more);
          }
        }
        tc_commit(&empty[s]);
        if (++s == stages)
          s = 0, phase ^= 1;
      }
      if (alive)
        tc_commit(tfull);
    }
  }
  else if (BULK && warp == 2 + 4 * GROUPS)
  {
    // ---------------------------------------------------------------- copies to the other blocks, first all of this
    // block's outputs to the one that multiplies them right behind its own (the copies leave in this order)
    if (lane == 0)
    {
      bool alive = true;
      for (int l = 0; l + 1 < P.count && alive; ++l)
      {
        const int buffer = (l + 1) & 1;
        for (int b = 1; b < blocks && alive; ++b)
        {
          const uint32_t to = rank ^ (uint32_t)b;
          const uint32_t ready = mapa_u32(smem_u32(&zfull[4 * buffer + rank]), to);
          for (int q = 0; q < 4; ++q)
          {
            if (b == 1 && !mbar_wait(&slab[4 * buffer + q], (l >> 1) & 1, abort_flag))
            {
              alive = false;
              break;
            }
            const uint32_t from = smem_u32(zbuf + (buffer * H + j0 + 32 * q) * 128);
            asm volatile(
                "cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                    mapa_u32(from, to)),
                "r"(from), "r"(32u * 128u), "r"(ready)
                : "memory");
          }
        }
      }
    }
  }
  else
  {
    // ---------------------------------------------------------------- epilogue: a lane an output, eight rows
    const int quarter = warp & 3, grp = (warp - 2) >> 2, j = j0 + 32 * quarter + lane, r0 = 8 * grp;
    const uint32_t taddr = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)r0;
    float z[8]; // this output of the layer below (residual layers are square)
#pragma unroll
    for (int r = 0; r < 8; ++r)
      z[r] = P.layers[P.first].z[(size_t)(row0 + r0 + r) * H + j];
    for (int l = 0; l < P.count; ++l)
    {
      FwdMeta M;
      load_fwd_meta(P, P.first + l, M);
      const float bias = M.b[j];
      const bool no_mu = (P.flags & DPC_FWD_NO_MU) && !((P.flags & (1 << 10)) && l == 0);
      const bool store_pre = M.preact && !(no_mu && (P.flags & DPC_FWD_NO_PREACT));
      if (!__all_sync(0xffffffffu, mbar_wait(tfull, l & 1, abort_flag))) // (the warp gives up as a whole)
        break;
      tc_fence_after();
      float pre[8], half1[8]; // the two halves of K, each "hi" + "mid"
      tc_ld8(taddr, pre);
      tc_ld8(taddr + (uint32_t)(2 * HALF), half1);
      if (!TF32)
      {
        float m[8];
        tc_ld8(taddr + (uint32_t)HALF, m);
#pragma unroll
        for (int r = 0; r < 8; ++r)
          pre[r] += m[r];
        tc_ld8(taddr + (uint32_t)(3 * HALF), m);
#pragma unroll
        for (int r = 0; r < 8; ++r)
          half1[r] += m[r];
      }
#pragma unroll
      for (int r = 0; r < 8; ++r)
        pre[r] += half1[r];
      tc_fence_before(); // (arriving at ready[rank] below says that the sums have been loaded)
      float f[8], d[8];
#pragma unroll
      for (int r = 0; r < 8; ++r)
        pre[r] = M.a * pre[r] + bias;
      act_many<false>(M.act, pre, f, d);
#pragma unroll
      for (int r = 0; r < 8; ++r)
        z[r] = (M.flags & DPC_LAYER_RESIDUAL) ? f[r] + z[r] : f[r];
      uint4 out[2];
      operands(z, out);
      if (l + 1 < P.count)
      {
        uint8_t* next = zbuf + ((l + 1) & 1) * H * 128;
        uint64_t* ready = &zfull[4 * ((l + 1) & 1) + rank];
#pragma unroll
        for (int half = 0; half < 2; ++half)
          *reinterpret_cast<uint4*>(next + chunk(j, grp, half)) = out[half];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncwarp();
        if (lane == 0)
        {
          mbar_arrive(ready);
          if (BULK)
            mbar_arrive(&slab[4 * ((l + 1) & 1) + quarter]);
        }
        if (!BULK)
        {
          // to the block that multiplies this one's outputs right behind its own first
#pragma unroll
          for (int half = 0; half < 2; ++half)
          {
            const uint32_t at = smem_u32(next + chunk(j, grp, half));
            for (int b = 1; b < blocks; ++b)
            {
              const uint32_t to = rank ^ (uint32_t)b;
              asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 "
                           "[%0], {%1, %2, %3, %4}, [%5];" ::"r"(mapa_u32(at, to)),
                           "r"(out[half].x), "r"(out[half].y), "r"(out[half].z), "r"(out[half].w),
                           "r"(mapa_u32(smem_u32(ready), to))
                           : "memory");
            }
          }
        }
        __syncwarp();
      }
      // off the dependent path: beliefs, their planes and what the flags ask for
      const size_t o = (size_t)(row0 + r0) * H + j;
#pragma unroll
      for (int r = 0; r < 8; ++r)
      {
        M.up_z[o + (size_t)r * H] = z[r];
        if (!no_mu)
          M.mu[o + (size_t)r * H] = z[r];
        if (store_pre)
          M.preact[o + (size_t)r * H] = pre[r];
      }
      if (!TF32 && M.upz_hi)
      {
        // even lanes take two neighbouring outputs of the even rows, odd ones of the odd rows
        const bool odd = lane & 1;
#pragma unroll
        for (int half = 0; half < 2; ++half)
        {
          const uint32_t w[4] = {out[half].x, out[half].y, out[half].z, out[half].w};
          __nv_bfloat16* plane = M.upz_hi + (half ? P.act_elems : 0) + (size_t)(row0 + r0) * H + (j & ~1);
#pragma unroll
          for (int u = 0; u < 4; ++u) // rows 2u and 2u + 1 in the halves of a word
          {
            const uint32_t other = __shfl_xor_sync(0xffffffffu, w[u], 1);
            const uint32_t two = odd ? __byte_perm(other, w[u], 0x7632) : __byte_perm(w[u], other, 0x5410);
            *reinterpret_cast<uint32_t*>(plane + (size_t)(2 * u + (odd ? 1 : 0)) * H) = two;
          }
        }
      }
    }
  }

  // ------------------------------------------------------------------ teardown
  tc_fence_before();
  __syncthreads(); // whichever role gave up, all have ended and start no more copies
  if (threadIdx.x == 0 && *abort_flag)
  {
    atomicExch(P.error_flag, 1);
    // weights and other blocks' outputs that nobody waited for land before the shared memory goes away
    const long long t0 = clock64();
    while (clock64() - t0 < 2000000LL)
    {
    }
  }
  __syncwarp();
  cluster_sync_all(); // no block leaves while another may still store to its shared memory
  if (warp == 1)
  {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(COLUMNS) : "memory");
  }
}

// DPC_OK, or 1: not for this plan.
template <bool TF32>
int launch_cluster_sweep(dpc_plan* p, TcState* st, const CUtensorMap& w, const TcParams& P)
{
  const int H = p->run.width, B = p->batch, blocks = H / 128;
  if (getenv("DPC_DISABLE_CLUSTER_SWEEP") || (H != 256 && H != 512) || st->trace)
    return 1;
  // Where the tiles would split K (their bits stay).  Larger batches fill the SMs with tiles; several waves of clusters
  // took as long (24 layers of 512 units at batch 4096 453 us, a launch a layer 425).
  if (2 * (B / TBM) * (H / 64) > p->ctx->sm_count || getenv("DPC_DISABLE_KSPLIT"))
    return 1;
  // As few rows a cluster as there are SMs for, so that every layer's epilogue and exchange are short.
  int rows = 8;
  while (rows < 32 && (B / rows) * blocks > p->ctx->sm_count * 7 / 8)
    rows *= 2;
  const int stages = (232448 - 1024 - 512 - 2 * H * 128) / 32768;
  const int smem = 2 * H * 128 + stages * 32768 + 1024 + 512;
  if (smem > st->max_smem)
    return 1;
  auto kern = rows == 32   ? cluster_sweep_kernel<TF32, 32>
              : rows == 16 ? cluster_sweep_kernel<TF32, 16>
                           : cluster_sweep_kernel<TF32, 8>;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(B / rows * blocks));
  cfg.blockDim = dim3((unsigned)(rows == 32 ? kSweepThreads<32> : rows == 16 ? kSweepThreads<16> : kSweepThreads<8>));
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = p->ctx->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim = {(unsigned)blocks, 1, 1};
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  // One wave of clusters or none: how many run at once depends on how the SMs are grouped (33 of four blocks where 148 SMs
  // would hold 37).  24 layers of 512 units with TF32, tiles / clusters: batch 1024 174 / 117 us, 1152, 36 clusters,
  // 174 / 230.
  struct Known
  {
    int device = -1, clusters = 0;
  };
  static thread_local Known known[2][3];
  Known& at_once = known[H / 512][rows / 16];
  if (at_once.device != p->ctx->device)
  {
    DPC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448));
    DPC_CUDA(cudaOccupancyMaxActiveClusters(&at_once.clusters, kern, &cfg));
    at_once.device = p->ctx->device;
  }
  if (B / rows > at_once.clusters)
    return 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, w, P, H, stages, st->chain_target_bias);
  p->ctx->launches += 1;
  return e == cudaSuccess ? DPC_OK : cuda_fail(e, "cluster sweep launch");
}
