// Context, memory, CUDA graphs, plans and the phase entry points of the dpc_* C ABI.
#include <cstdio>
#include <functional>
#include <cstring>
#include <string>
#include <type_traits>

#include "dpc_internal.h"
#include "dpc_batch.cuh"

namespace dpc
{
static thread_local std::string g_error;

void set_error(const std::string& msg)
{
  g_error = msg;
}
int fail(int code, const std::string& msg)
{
  g_error = msg;
  return code;
}
int cuda_fail(cudaError_t err, const char* what)
{
  g_error = std::string(what) + ": " + cudaGetErrorString(err);
  return err == cudaErrorNoDevice || err == cudaErrorInsufficientDriver ? DPC_ERR_NO_DEVICE
                                                                         : DPC_ERR_CUDA;
}

static int check_launch(dpc_ctx* ctx, const char* what)
{
  ctx->launches += 1;
  cudaError_t err = cudaPeekAtLastError();
  if (err != cudaSuccess)
    return cuda_fail(cudaGetLastError(), what);
  return DPC_OK;
}

// How many CTAs of a cluster share the batch rows of one block's columns in the batch reductions
// (Psi update, bias column sums): doubled while the launch has fewer than four CTAs per SM (a CTA's
// time is one chain of dependent row loads: more, shorter chains hide more latency) and every CTA
// keeps at least `min_rows` rows.  1 for launches over many layers.
static int row_split(const dpc_ctx* ctx, long long blocks, int batch, int min_rows)
{
  int R = 1;
  while (R < 8 && blocks * R < 4LL * ctx->sm_count && batch / (2 * R) >= min_rows)
    R *= 2;
  return R;
}

// kern<<<(grid.x, grid.y, R), threads, 0, st>>> as clusters of R CTAs along z (R = 1: a plain launch)
template <typename... KArgs, typename... Args>
static void launch_row_split(void (*kern)(KArgs...), dim3 grid, int threads, int R, cudaStream_t st,
                             Args... args)
{
  if (R <= 1)
  {
    kern<<<grid, threads, 0, st>>>(args...);
    return;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid.x, grid.y, (unsigned)R);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = (unsigned)R;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, args...); // an error stays pending for check_launch()
}

static int check_range(dpc_plan* p, int first, int count)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  if (first < 0 || count < 0 || first + count > p->n)
    return fail(DPC_ERR_INVALID, "layer range out of bounds");
  return DPC_OK;
}

static inline int cdiv(int a, int b)
{
  return (a + b - 1) / b;
}

// The tiles of layers [first, end), of which layer i has tiles(i) of kind(i); end becomes the first layer that is left
// for another launch, where the layers are more runs than a list holds.
template <typename Tiles, typename Kind>
static int list_tiles(TileList& T, int first, int& end, Tiles tiles, Kind kind)
{
  T.first = first, T.runs = 0;
  int total = 0;
  for (int i = first; i < end; ++i)
  {
    const int n = tiles(i);
    const bool k = kind(i);
    if (T.runs == 0 || n != T.run[T.runs - 1].per || k != (T.run[T.runs - 1].kind != 0))
    {
      if (T.runs == kListRuns)
      {
        end = i;
        break;
      }
      // (runs without tiles are never looked up)
      T.run[T.runs++] = TileRun{total, n, n > 0 ? ~0u / n : 0u, (unsigned short)(i - first), (unsigned short)k};
    }
    total += n;
  }
  T.layers = end - first;
  return total;
}

// A product of layers [first, first+count) in one launch.
template <int OP>
static int launch_gemm(dpc_plan* p, int first, int count, int flags, int mode, const float* epc_src = nullptr)
{
  const int sm = p->ctx->sm_count;
  auto tiles_of = [&](int i, int T)
  {
    const dpc_layer& L = p->h[i];
    const int M = OP == OP_WG ? L.next_size : p->batch, N = OP == OP_FWD ? L.next_size : L.size;
    // (DirectFeedbackUpdate is a no-op unless the layer above owns feedback weights)
    const bool any = L.next_size > 0 && (OP != OP_WG || (mode & ~WG_GRAD_ONLY) != WG_DFA ||
                                         (i + 1 < p->n && p->h[i + 1].Psi));
    return any ? cdiv(M, T) * cdiv(N, T) : 0;
  };
  long long tiles = 0, tiles64 = 0, aligned = 0;
  bool vec = true; // rows can be copied 16 bytes at a time
  for (int i = first; i < first + count; ++i)
  {
    tiles += tiles_of(i, 32), tiles64 += tiles_of(i, 64);
    vec &= p->h[i].size % 4 == 0 && p->h[i].next_size % 4 == 0;
    const int K = OP == OP_FWD ? p->h[i].size : OP == OP_FB ? p->h[i].next_size : p->batch;
    if (p->h[i].size % 4 == 0 && (OP == OP_FWD || p->h[i].next_size % 4 == 0) && K >= 128)
      aligned += tiles_of(i, 32);
  }
  // us, W = 4 / W = 2 / T = 64, by 32 x 32 tiles an SM:  0.9 (445 wide, batch 48) 16.5 / 24 / -,  1.4 (784 x 256
  // weights) 31 / 26 / -,  3 (512 wide, batch 210) 25 / 22 / -,  3.7 (512 wide, batch 1089) 28 / 25 / -,  4.2 (403
  // wide, batch 512: rows that are copied element by element, by twice the threads) 44 / 49 / 59, state 35 / 34 / 40,
  // 7.3 (45 layers of 374 at batch 48, 1.8 tiles of 64 an SM) 51 / 43 / 36
  // 64 x 64 from six 32 x 32 tiles an SM already in forward products of SimplePC layers, which apply the activation to
  // their operand once for each column of tiles (two layers of 256 and one of 100, batch 1500: 1480 / 1340 us a step of
  // 20 passes with esigmoid, 1310 / 1260 with tanh; at batch 1400, 5.9 tiles an SM, 1060 / 1233).
  // Not 64 x 64 where layers are narrower than that and most of a tile is padding (20 passes over 400 layers of 32 at
  // batch 300 1440 / 1000 us a step on 64 x 64 / 32 x 32 tiles, 140 of 96 at batch 20 518 / 367).
  const bool feeds = OP == OP_FWD && (p->h[first].flags & DPC_LAYER_INPUT_ACT);
  const bool large =
      (4 * tiles64 >= 7LL * sm || (feeds && tiles64 > sm && tiles > 6LL * sm)) && 8 * tiles64 <= 3 * tiles;
  // Long steps, where most tiles have rows that are copied 16 bytes at a time and sums of 128 or more, and the tiles of
  // a kernel are at most one wave with the shared memory they take (76 KB, 43 KB; 64 x 64 tiles in any number).  us a
  // step, short / long: thirteen layers of 812 at batch 4 637 / 593, three of 768 at batch 128 649 / 615, twelve of 300
  // at batch 60 294 / 277; two warps: three of 320 at batch 900 1018 / 963; 64 x 64: fourteen of 1024 at batch 100
  // 1211 / 1165.  Four layers of 208 at batch 1000, 4.5 tiles an SM on four warps, 471 / 512; ten of 512 at batch 170,
  // 6.5 tiles on two, 634 / 657; six of 445 at batch 48, copied element by element, 196 / 208; 400 of 32 at batch 300
  // 932 / 1092.
  const bool long_steps = 2 * aligned > tiles;
  const bool two_warps = tiles >= (OP == OP_WG ? sm : vec ? 3LL * sm : 6LL * sm);
  for (int f = first, end; f < first + count; f = end)
  {
    TileList T;
    end = first + count;
    const int blocks = list_tiles(
        T, f, end, [&](int i) { return tiles_of(i, large ? 64 : 32); }, [](int) { return false; });
    if (blocks == 0)
      continue;
    auto go = [&](auto tile)
    {
      using C = decltype(tile);
      constexpr int bytes = C::bytes(GemmEpilogue<OP>::kPre);
      auto kern = pc_gemm_kernel<OP, C>;
      // (more than 48 KB have to be asked for, once a device)
      static thread_local int configured = -1;
      if (configured != p->ctx->device)
      {
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess)
          return;
        configured = p->ctx->device;
      }
      kern<<<blocks, C::THREADS, bytes, p->ctx->stream>>>(p->d, p->n, p->batch, flags, mode, p->energy, epc_src, T);
    };
    if (large && long_steps)
      go(GemmTile<64, 4, true>());
    else if (large)
      go(GemmTile<64, 4, false>());
    else if (two_warps)
      long_steps && tiles <= 5LL * sm ? go(GemmTile<32, 2, true>()) : go(GemmTile<32, 2, false>());
    else if (long_steps && tiles <= 2LL * sm)
      go(GemmTile<32, 4, true>());
    else
      go(GemmTile<32, 4, false>());
    const int rc = check_launch(p->ctx, "grouped GEMM kernel");
    if (rc != DPC_OK)
      return rc;
  }
  return DPC_OK;
}

// Networks with an Adam-type optimizer or an activation with a kink turn a rounding difference into a whole
// step (an update m / (sqrt(v) + eps), a derivative that flips between 0 and 1).  Sums over the width keep one
// ascending order in all kernels of theirs.  Their sums over the batch stay on the kernels that have always formed
// them -- some split the rows, over warps and clusters, in an order that a shape and a GPU fix -- and off
// batch_product_kernel.
bool ordered_sums(const dpc_plan* p)
{
  for (const dpc_layer& L : p->h)
    if (L.next_size > 0 && (L.opt != DPC_OPT_SGD || (L.Psi && L.opt_psi != DPC_OPT_SGD) || L.act == DPC_ACT_RELU ||
                            L.act == DPC_ACT_HARD_TANH))
      return true;
  return false;
}

static int elem_blocks(const dpc_plan* p, size_t max_elems)
{
  size_t blocks = (max_elems + 1023) / 1024; // 256 threads x 4 elements each
  size_t cap = (size_t)p->ctx->sm_count * 8;
  if (blocks > cap)
    blocks = cap;
  return (int)std::max<size_t>(blocks, 1);
}

constexpr int kMaxZ = 32768; // layers per launch (gridDim.y/z limit is 65535)
} // namespace dpc

using namespace dpc;

// The C linkage of every dpc_* definition below comes from its declaration in
// deepity_b200.h.
const char* dpc_last_error(void)
{
  return g_error.c_str();
}

const char* dpc_version(void)
{
  return "deepity_b200 0.1 (sm_100a)";
}

int dpc_create(int device, dpc_ctx** out)
{
  if (!out)
    return fail(DPC_ERR_INVALID, "dpc_create: null out");
  int n = 0;
  cudaError_t err = cudaGetDeviceCount(&n);
  if (err != cudaSuccess || n == 0)
  {
    cudaGetLastError();
    return fail(DPC_ERR_NO_DEVICE, "no CUDA device available (this library has no CPU fallback)");
  }
  if (device < 0 || device >= n)
    return fail(DPC_ERR_INVALID, "dpc_create: device index out of range");
  DPC_CUDA(cudaSetDevice(device));
  auto* ctx = new dpc_ctx();
  ctx->device = device;
  cudaDeviceProp prop;
  DPC_CUDA(cudaGetDeviceProperties(&prop, device));
  ctx->sm_count = prop.multiProcessorCount;
  DPC_CUDA(cudaStreamCreateWithFlags(&ctx->stream, cudaStreamNonBlocking));
  // streams that consecutive single tensor-core layers of one phase fork to (see dispatch_range)
  if (!getenv("DPC_DISABLE_LAYER_STREAMS"))
  {
    bool ok = cudaEventCreateWithFlags(&ctx->fork_ev, cudaEventDisableTiming) == cudaSuccess;
    for (int s = 0; s < dpc_ctx::kSide && ok; ++s)
      ok = cudaStreamCreateWithFlags(&ctx->side[s], cudaStreamNonBlocking) == cudaSuccess &&
           cudaEventCreateWithFlags(&ctx->join_ev[s], cudaEventDisableTiming) == cudaSuccess;
    if (!ok)
    {
      const cudaError_t e = cudaGetLastError();
      dpc_destroy(ctx);
      return cuda_fail(e, "creating the per-layer streams");
    }
  }
  *out = ctx;
  return DPC_OK;
}

int dpc_destroy(dpc_ctx* ctx)
{
  if (!ctx)
    return DPC_OK;
  cudaSetDevice(ctx->device);
  for (int s = 0; s < dpc_ctx::kSlots; ++s)
  {
    if (ctx->execs[s])
      cudaGraphExecDestroy(ctx->execs[s]);
    if (ctx->graphs[s])
      cudaGraphDestroy(ctx->graphs[s]);
  }
  if (ctx->stream)
  {
    cudaStreamSynchronize(ctx->stream);
    cudaStreamDestroy(ctx->stream);
  }
  for (int s = 0; s < dpc_ctx::kSide; ++s)
  {
    if (ctx->side[s])
    {
      cudaStreamSynchronize(ctx->side[s]);
      cudaStreamDestroy(ctx->side[s]);
    }
    if (ctx->join_ev[s])
      cudaEventDestroy(ctx->join_ev[s]);
  }
  if (ctx->fork_ev)
    cudaEventDestroy(ctx->fork_ev);
  delete ctx;
  return DPC_OK;
}

int dpc_set_precision(dpc_ctx* ctx, int precision)
{
  if (!ctx || (precision != DPC_PRECISION_FP32 && precision != DPC_PRECISION_TF32 &&
               precision != DPC_PRECISION_MIXED))
    return fail(DPC_ERR_INVALID, "dpc_set_precision: bad argument");
  ctx->precision = precision;
  return DPC_OK;
}

int dpc_get_precision(dpc_ctx* ctx)
{
  return ctx ? ctx->precision : DPC_ERR_INVALID;
}

void* dpc_stream(dpc_ctx* ctx)
{
  return ctx ? (void*)ctx->stream : nullptr;
}

int64_t dpc_launch_count(dpc_ctx* ctx)
{
  return ctx ? ctx->launches : 0;
}

int dpc_alloc(dpc_ctx* ctx, size_t bytes, void** out)
{
  if (!ctx || !out)
    return fail(DPC_ERR_INVALID, "dpc_alloc: null argument");
  DPC_CUDA(cudaSetDevice(ctx->device));
  DPC_CUDA(cudaMalloc(out, bytes ? bytes : 16));
  return DPC_OK;
}

int dpc_free(dpc_ctx* ctx, void* ptr)
{
  if (!ctx)
    return fail(DPC_ERR_INVALID, "dpc_free: null context");
  if (ptr)
    DPC_CUDA(cudaFree(ptr));
  return DPC_OK;
}

int dpc_zero(dpc_ctx* ctx, void* ptr, size_t bytes)
{
  if (!ctx || (!ptr && bytes))
    return fail(DPC_ERR_INVALID, "dpc_zero: null argument");
  DPC_CUDA(cudaMemsetAsync(ptr, 0, bytes, ctx->stream));
  return DPC_OK;
}

int dpc_copy_d2d(dpc_ctx* ctx, void* dst, const void* src, size_t bytes)
{
  if (!ctx)
    return fail(DPC_ERR_INVALID, "null context");
  DPC_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, ctx->stream));
  return DPC_OK;
}

int dpc_copy_h2d(dpc_ctx* ctx, void* dst, const void* host_src, size_t bytes)
{
  if (!ctx)
    return fail(DPC_ERR_INVALID, "null context");
  DPC_CUDA(cudaMemcpyAsync(dst, host_src, bytes, cudaMemcpyHostToDevice, ctx->stream));
  return DPC_OK;
}

int dpc_host_is_pageable(const void* host_ptr)
{
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, host_ptr) != cudaSuccess)
  {
    cudaGetLastError();
    return 1;
  }
  return a.type == cudaMemoryTypeUnregistered ? 1 : 0;
}

int dpc_copy_d2h(dpc_ctx* ctx, void* host_dst, const void* src, size_t bytes)
{
  if (!ctx)
    return fail(DPC_ERR_INVALID, "null context");
  DPC_CUDA(cudaMemcpyAsync(host_dst, src, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  return DPC_OK;
}

int dpc_copy_h2d_sync(dpc_ctx* ctx, void* dst, const void* host_src, size_t bytes)
{
  int rc = dpc_copy_h2d(ctx, dst, host_src, bytes);
  if (rc != DPC_OK)
    return rc;
  DPC_CUDA(cudaStreamSynchronize(ctx->stream));
  return DPC_OK;
}

int dpc_copy_d2h_sync(dpc_ctx* ctx, void* host_dst, const void* src, size_t bytes)
{
  int rc = dpc_copy_d2h(ctx, host_dst, src, bytes);
  if (rc != DPC_OK)
    return rc;
  DPC_CUDA(cudaStreamSynchronize(ctx->stream));
  return DPC_OK;
}

int dpc_alloc_host(dpc_ctx* ctx, size_t bytes, void** out)
{
  if (!ctx || !out)
    return fail(DPC_ERR_INVALID, "dpc_alloc_host: null argument");
  DPC_CUDA(cudaMallocHost(out, bytes ? bytes : 16));
  return DPC_OK;
}

int dpc_free_host(dpc_ctx* ctx, void* ptr)
{
  (void)ctx;
  if (ptr)
    DPC_CUDA(cudaFreeHost(ptr));
  return DPC_OK;
}

int dpc_sync(dpc_ctx* ctx)
{
  if (!ctx)
    return fail(DPC_ERR_INVALID, "null context");
  DPC_CUDA(cudaStreamSynchronize(ctx->stream));
  return DPC_OK;
}

namespace dpc
{
__global__ void gather_rows_kernel(const float* __restrict__ src, const int64_t* __restrict__ index,
                                   int64_t first, int rows, int64_t cols, float* __restrict__ dst,
                                   int vec)
{
  const int64_t per_row = vec ? cols / 4 : cols;
  const int64_t total = (int64_t)rows * per_row;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x)
  {
    const int64_t r = i / per_row, c = i - r * per_row;
    const int64_t s = index[first + r];
    if (vec)
      reinterpret_cast<float4*>(dst + r * cols)[c] =
          __ldg(reinterpret_cast<const float4*>(src + s * cols) + c);
    else
      dst[r * cols + c] = src[s * cols + c];
  }
}
} // namespace dpc

int dpc_gather_rows(dpc_ctx* ctx, const float* src_dev, const int64_t* index_dev, int64_t first,
                    int rows, int64_t cols, float* dst_dev)
{
  if (!ctx || !src_dev || !index_dev || !dst_dev || rows < 0 || cols <= 0 || first < 0)
    return fail(DPC_ERR_INVALID, "dpc_gather_rows: bad argument");
  if (rows == 0)
    return DPC_OK;
  const int vec = cols % 4 == 0 && ((uintptr_t)src_dev % 16) == 0 && ((uintptr_t)dst_dev % 16) == 0;
  const int64_t total = (int64_t)rows * (vec ? cols / 4 : cols);
  const int blocks = (int)std::min<int64_t>((total + 255) / 256, (int64_t)ctx->sm_count * 16);
  dpc::gather_rows_kernel<<<blocks, 256, 0, ctx->stream>>>(src_dev, index_dev, first, rows, cols,
                                                          dst_dev, vec);
  return check_launch(ctx, "gather_rows kernel");
}

int dpc_graph_begin(dpc_ctx* ctx, int slot)
{
  if (!ctx || slot < 0 || slot >= dpc_ctx::kSlots)
    return fail(DPC_ERR_INVALID, "dpc_graph_begin: bad slot");
  if (ctx->capturing_slot >= 0)
    return fail(DPC_ERR_STATE, "dpc_graph_begin: a capture is already open");
  DPC_CUDA(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal));
  ctx->capturing_slot = slot;
  ctx->launches_at_begin = ctx->launches;
  return DPC_OK;
}

int dpc_graph_end(dpc_ctx* ctx, int slot)
{
  if (!ctx || slot != ctx->capturing_slot)
    return fail(DPC_ERR_STATE, "dpc_graph_end: slot does not match the open capture");
  ctx->capturing_slot = -1;
  // Recorded launches run when the graph is replayed, not now.
  ctx->graph_kernels[slot] = ctx->launches - ctx->launches_at_begin;
  ctx->launches = ctx->launches_at_begin;
  cudaGraph_t graph = nullptr;
  DPC_CUDA(cudaStreamEndCapture(ctx->stream, &graph));
  if (ctx->execs[slot])
    cudaGraphExecDestroy(ctx->execs[slot]);
  if (ctx->graphs[slot])
    cudaGraphDestroy(ctx->graphs[slot]);
  ctx->execs[slot] = nullptr;
  ctx->graphs[slot] = graph;
  DPC_CUDA(cudaGraphInstantiate(&ctx->execs[slot], graph, 0));
  return DPC_OK;
}

int dpc_graph_launch(dpc_ctx* ctx, int slot)
{
  if (!ctx || slot < 0 || slot >= dpc_ctx::kSlots || !ctx->execs[slot])
    return fail(DPC_ERR_STATE, "dpc_graph_launch: nothing captured in this slot");
  DPC_CUDA(cudaGraphLaunch(ctx->execs[slot], ctx->stream));
  ctx->launches += ctx->graph_kernels[slot];
  return DPC_OK;
}

int dpc_graph_drop(dpc_ctx* ctx, int slot)
{
  if (!ctx || slot < 0 || slot >= dpc_ctx::kSlots)
    return fail(DPC_ERR_INVALID, "dpc_graph_drop: bad slot");
  if (ctx->execs[slot])
    cudaGraphExecDestroy(ctx->execs[slot]);
  if (ctx->graphs[slot])
    cudaGraphDestroy(ctx->graphs[slot]);
  ctx->execs[slot] = nullptr;
  ctx->graphs[slot] = nullptr;
  return DPC_OK;
}

// ------------------------------------------------------------------------------ plans
static int validate_layers(const dpc_layer* layers, int n, int batch)
{
  if (!layers || n < 2 || batch <= 0)
    return fail(DPC_ERR_INVALID, "plan: need at least two layers and a positive batch");
  for (int i = 0; i < n; ++i)
  {
    const dpc_layer& L = layers[i];
    if (L.size <= 0 || !L.z || !L.e)
      return fail(DPC_ERR_INVALID, "plan: layer " + std::to_string(i) + " lacks z/e or size");
    if (i + 1 < n)
    {
      if (L.next_size != layers[i + 1].size)
        return fail(DPC_ERR_INVALID, "plan: next_size of layer " + std::to_string(i) +
                                         " does not match the size of the layer above");
      if (!L.W || !L.b || !L.mu)
        return fail(DPC_ERR_INVALID, "plan: layer " + std::to_string(i) + " lacks W/b/mu");
      const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
      if (!simple && (!L.preact || !L.fe))
        return fail(DPC_ERR_INVALID, "plan: layer " + std::to_string(i) + " lacks preact/fe");
      if (simple && !L.zF)
        return fail(DPC_ERR_INVALID, "plan: SimplePC layer " + std::to_string(i) + " lacks zF");
      if ((L.flags & DPC_LAYER_RESIDUAL) && L.size != L.next_size)
        return fail(DPC_ERR_INVALID, "plan: residual layer must be square");
      if (L.opt != DPC_OPT_SGD && (!L.m_W || !L.v_W || !L.m_b || !L.v_b || !L.t))
        return fail(DPC_ERR_INVALID, "plan: Adam state missing on layer " + std::to_string(i));
      if (L.Psi && L.opt_psi != DPC_OPT_SGD && (!L.m_Psi || !L.v_Psi || !L.t_Psi))
        return fail(DPC_ERR_INVALID, "plan: Psi Adam state missing on layer " + std::to_string(i));
      // (the last layer of a layer-sharded block is not the terminal: only the stride is checked)
      if (L.Psi && (L.psi_stride < L.terminal_size || L.terminal_size <= 0))
        return fail(DPC_ERR_INVALID, "plan: terminal_size / psi_stride mismatch on layer " +
                                         std::to_string(i));
    }
    else if (L.next_size != 0)
      return fail(DPC_ERR_INVALID, "plan: the last layer must be weight-less (next_size 0)");
  }
  return DPC_OK;
}

int dpc_plan_create(dpc_ctx* ctx, const dpc_layer* layers, int n_layers, int batch,
                    dpc_plan** out)
{
  if (!ctx || !out)
    return fail(DPC_ERR_INVALID, "dpc_plan_create: null argument");
  int rc = validate_layers(layers, n_layers, batch);
  if (rc != DPC_OK)
    return rc;
  auto* p = new dpc_plan();
  p->ctx = ctx;
  p->n = n_layers;
  p->batch = batch;
  p->h.assign(layers, layers + n_layers);
  p->e_terminal = layers[n_layers - 1].e;
  p->init_precision = ctx->precision;
  cudaError_t err = cudaMalloc(&p->d, sizeof(dpc_layer) * n_layers);
  if (err == cudaSuccess)
    err = cudaMalloc(&p->energy, 2 * sizeof(double));
  if (err == cudaSuccess)
    err = cudaMallocHost(&p->energy_host, 2 * sizeof(double));
  if (err == cudaSuccess)
    err = cudaMemcpyAsync(p->d, p->h.data(), sizeof(dpc_layer) * n_layers, cudaMemcpyHostToDevice, ctx->stream);
  if (err == cudaSuccess)
    err = cudaMemsetAsync(p->energy, 0, 2 * sizeof(double), ctx->stream);
  if (err != cudaSuccess)
  {
    dpc_plan_destroy(p);
    return cuda_fail(err, "dpc_plan_create");
  }
  rc = tc_plan_init(p);
  if (rc >= 0)
    rc = res_plan_init(p);
  if (rc >= 0)
    rc = cluster_plan_init(p);
  if (rc < 0)
  {
    dpc_plan_destroy(p);
    return rc;
  }
  *out = p;
  return DPC_OK;
}

int dpc_plan_update(dpc_plan* p, const dpc_layer* layers, int n_layers)
{
  if (!p || n_layers != p->n)
    return fail(DPC_ERR_INVALID, "dpc_plan_update: layer count differs from the plan");
  int rc = validate_layers(layers, n_layers, p->batch);
  if (rc != DPC_OK)
    return rc;
  // New rates only (an epoch loop with a decaying learning rate): every kernel reads them from the
  // table, so a stream-ordered copy is all there is to do.
  bool structure = p->init_precision != p->ctx->precision;
  for (int i = 0; i < n_layers && !structure; ++i)
  {
    dpc_layer a = p->h[i], b = layers[i];
    for (dpc_layer* q : {&a, &b})
      q->lr = q->ir = q->fl = q->lmbda = q->psi_decay = q->momentum_beta = 0.0f;
    structure = memcmp(&a, &b, sizeof(dpc_layer)) != 0;
  }
  if (!structure)
  {
    p->h.assign(layers, layers + n_layers);
    DPC_CUDA(cudaMemcpyAsync(p->d, p->h.data(), sizeof(dpc_layer) * n_layers, cudaMemcpyHostToDevice,
                             p->ctx->stream));
    return DPC_OK;
  }
  // f(z) of SimplePC layers, as last fed to the products, survives in zF
  for (int i = 0; i < n_layers; ++i)
    if (layers[i].zF && layers[i].zF == p->h[i].zF && layers[i].size == p->h[i].size &&
        (rc = tc_zf_need(p, i, 1)) != DPC_OK)
      return rc;
  DPC_CUDA(cudaStreamSynchronize(p->ctx->stream));
  if (p->e_terminal == p->h[p->n - 1].e)
    p->e_terminal = layers[n_layers - 1].e;
  p->h.assign(layers, layers + n_layers);
  DPC_CUDA(cudaMemcpyAsync(p->d, p->h.data(), sizeof(dpc_layer) * n_layers, cudaMemcpyHostToDevice,
                           p->ctx->stream));
  tc_plan_free(p);
  res_plan_free(p);
  cluster_plan_free(p);
  p->init_precision = p->ctx->precision;
  rc = tc_plan_init(p);
  if (rc >= 0)
    rc = res_plan_init(p);
  if (rc >= 0)
    rc = cluster_plan_init(p);
  return rc < 0 ? rc : DPC_OK;
}

int dpc_plan_destroy(dpc_plan* p)
{
  if (!p)
    return DPC_OK;
  tc_plan_free(p);
  res_plan_free(p);
  cluster_plan_free(p);
  if (p->d)
    cudaFree(p->d);
  if (p->energy)
    cudaFree(p->energy);
  if (p->energy_host)
    cudaFreeHost(p->energy_host);
  delete p;
  return DPC_OK;
}

int dpc_plan_set_terminal_error(dpc_plan* p, const float* e_terminal_dev)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  p->e_terminal = e_terminal_dev ? e_terminal_dev : p->h[p->n - 1].e;
  return DPC_OK;
}

int dpc_plan_set_chain_trace(dpc_plan* p, void* trace_dev)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  tc_set_chain_trace(p, static_cast<unsigned long long*>(trace_dev));
  return DPC_OK;
}

int dpc_plan_tensor_run(dpc_plan* p, int* first, int* count)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  if (first)
    *first = p->run.first;
  if (count)
    *count = p->run.count;
  return DPC_OK;
}

int dpc_plan_describe(dpc_plan* p, char* buf, int buf_bytes)
{
  if (!p || !buf || buf_bytes <= 0)
    return fail(DPC_ERR_INVALID, "dpc_plan_describe: null argument");
  const std::string d = tc_describe(p);
  snprintf(buf, (size_t)buf_bytes, "%s", d.c_str());
  return DPC_OK;
}

int dpc_plan_invalidate(dpc_plan* p, int first, int count, int what)
{
  int rc = check_range(p, first, count);
  if (rc != DPC_OK)
    return rc;
  if (what & DPC_WROTE_Z)
    tc_touch(p, 0, first, count);
  if (what & DPC_WROTE_FE)
    tc_touch(p, 1, first, count);
  if (what & DPC_WROTE_W)
    tc_touch(p, 2, first, count);
  if (what & DPC_WROTE_ZF)
    tc_zf_written(p, first, count);
  if (what & DPC_REPLAYED)
    tc_replayed(p);
  for (int i = std::max(first, 1); (what & DPC_WROTE_E) && i < first + count; ++i)
    if (p->h[i - 1].flags & DPC_LAYER_INPUT_ACT)
      tc_touch(p, 1, i - 1, 1);
  return DPC_OK;
}

int dpc_plan_sync_operands(dpc_plan* p)
{
  return dpc_plan_sync_operands_of(p, DPC_WROTE_Z | DPC_WROTE_FE | DPC_WROTE_W);
}

int dpc_plan_sync_operands_of(dpc_plan* p, int what)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  return tc_sync_planes(p, what);
}

int dpc_plan_sync_input_activations(dpc_plan* p, int first, int count)
{
  const int rc = check_range(p, first, count);
  return rc == DPC_OK ? tc_zf_need(p, first, count) : rc;
}

int dpc_plan_set_wait_limit(dpc_plan* p, double milliseconds, int sweep_target_bias)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  cudaDeviceProp prop;
  DPC_CUDA(cudaGetDeviceProperties(&prop, p->ctx->device));
  // clock64() counts SM clocks; take the maximum clock so the limit is never shorter than asked
  const long long cycles =
      milliseconds > 0.0 ? (long long)(milliseconds * 1e-3 * (double)prop.clockRate * 1e3) : 0;
  tc_set_wait_limit(p, cycles, sweep_target_bias);
  return DPC_OK;
}

// ------------------------------------------------------------------------------ phases
// The CUDA-core kernels write the fp32 tensors only: tell the tensor-core path which of its
// operand planes have gone stale.
static void wrote(dpc_plan* p, int kind, int first, int count)
{
  if (p->run.count > 0 && count > 0)
    tc_touch(p, kind, first, count);
}
enum
{
  K_Z = 0,
  K_FE = 1,
  K_W = 2
};

static FePlanes fe_planes(dpc_plan* p)
{
  FePlanes P;
  void* base = nullptr;
  tc_fe_planes(p, &base, &P.run_first, &P.run_count, &P.elems, &P.only);
  P.fe = static_cast<__nv_bfloat16*>(base);
  return P;
}

// Whether the layer's forward pass runs on the narrow-head kernel: at most 16 output units and rows
// that can be read 16 bytes at a time.
static bool narrow_forward(const dpc_plan* p, int layer)
{
  const dpc_layer& L = p->h[layer];
  return L.next_size > 0 && L.next_size <= 16 && L.size % 4 == 0 && L.size >= 128 && ((uintptr_t)L.z % 16) == 0 &&
         ((uintptr_t)L.W % 16) == 0 &&
         // SimplePC layers under an Adam-type optimizer keep the grouped kernel's order of additions
         (!(L.flags & DPC_LAYER_INPUT_ACT) || (L.opt == DPC_OPT_SGD && ((uintptr_t)L.zF % 16) == 0));
}

template <int RPW, bool SIMPLE, bool SMEM>
static int launch_narrow_forward(dpc_plan* p, int f, int c, int flags, int blocks, size_t weights)
{
  auto kern = narrow_forward_kernel<RPW, SIMPLE, SMEM>;
  const size_t smem = sizeof(float) * kHeadRingFloats<RPW> + (SMEM ? weights : 0);
  static thread_local int configured = -1; // (the limit is an attribute of a device)
  if (configured != p->ctx->device)
  {
    DPC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 232448 - 1024));
    configured = p->ctx->device;
  }
  kern<<<dim3(blocks, 1, c), NTHREADS, smem, p->ctx->stream>>>(p->d, f, p->n, p->batch, flags, p->energy);
  return check_launch(p->ctx, "narrow forward kernel");
}

static int narrow_forward_simt(dpc_plan* p, int f, int c, int flags, bool simple)
{
  size_t weights = 0;
  for (int i = f; i < f + c; ++i)
    if (p->h[i].next_size > 0)
      weights = std::max(weights, sizeof(float) * (cdiv(p->h[i].next_size, 2) * 2) * ((size_t)cdiv(p->h[i].size, 512) * 512));
  const bool staged = weights <= 160 * 1024; // (beside the ring)
  // Single rows where pairs would leave SMs without a block (batch 256 x 256 -> 10: 4.1 us in 32 blocks); from 256 blocks of
  // pairs two to four a warp, which share a copy of the weights (four from 64 blocks on: 16.7 us instead of 9.8 for 4096 x
  // 1024 -> 10 alone, the same beside a tensor launch).
  const int pair_blocks = cdiv(p->batch, 16);
  if ((long long)pair_blocks * c < 64)
  {
    const int blocks = cdiv(p->batch, 8);
    if (!staged)
      return simple ? launch_narrow_forward<2, true, false>(p, f, c, flags, pair_blocks, 0)
                    : launch_narrow_forward<2, false, false>(p, f, c, flags, pair_blocks, 0);
    return simple   ? launch_narrow_forward<1, true, true>(p, f, c, flags, blocks, weights)
                    : launch_narrow_forward<1, false, true>(p, f, c, flags, blocks, weights);
  }
  const int turns = (int)std::min<long long>(4, std::max<long long>(1, (long long)pair_blocks * c / 128));
  const int blocks = cdiv(pair_blocks, turns);
  if (!staged)
    return simple ? launch_narrow_forward<2, true, false>(p, f, c, flags, blocks, 0)
                  : launch_narrow_forward<2, false, false>(p, f, c, flags, blocks, 0);
  return simple ? launch_narrow_forward<2, true, true>(p, f, c, flags, blocks, weights)
                : launch_narrow_forward<2, false, true>(p, f, c, flags, blocks, weights);
}

static int forward_simt(dpc_plan* p, int first, int count, int flags)
{
  cudaStream_t st = p->ctx->stream;
  if ((flags & DPC_FWD_CE) && count > 1 && first + count == p->n - 1)
  {
    // the head's kernel forms the softmax error, so the head does not share a grouped launch
    const int rc = forward_simt(p, first, count - 1, flags & ~DPC_FWD_CE);
    return rc == DPC_OK ? forward_simt(p, p->n - 2, 1, flags) : rc;
  }
  for (int f = first; f < first + count; f += kMaxZ)
  {
    const int c = std::min(kMaxZ, first + count - f);
    if (flags & DPC_FWD_CACHED)
    {
      size_t mx = 0;
      for (int i = f; i < f + c; ++i)
        mx = std::max(mx, (size_t)p->batch * std::max(p->h[i].next_size, 0));
      dim3 grid(elem_blocks(p, mx), c);
      cached_forward_kernel<<<grid, NTHREADS, 0, st>>>(p->d, f, p->n, p->batch, flags, p->energy);
    }
    else
    {
      // heads (at most 16 output units) with vector-loadable rows: one warp per batch row
      bool narrow = true;
      for (int i = f; i < f + c && narrow; ++i)
        narrow = p->h[i].next_size <= 0 || (narrow_forward(p, i) && ((p->h[i].flags ^ p->h[f].flags) & DPC_LAYER_INPUT_ACT) == 0);
      const bool simple = (p->h[f].flags & DPC_LAYER_INPUT_ACT) != 0;
      if (narrow)
      {
        const int rc = narrow_forward_simt(p, f, c, flags, simple);
        if (rc != DPC_OK)
          return rc;
        continue;
      }
      else
      {
        const int rc = launch_gemm<OP_FWD>(p, f, c, flags, 0);
        if (rc != DPC_OK)
          return rc;
        continue;
      }
    }
    int rc = check_launch(p->ctx, "forward kernel");
    if (rc != DPC_OK)
      return rc;
  }
  const bool simple = (p->h[first].flags & DPC_LAYER_INPUT_ACT) != 0;
  if (simple && !(flags & DPC_FWD_CACHED))
    tc_zf_written(p, first, count);
  if ((flags & DPC_FWD_FE) || (simple && (flags & DPC_FWD_ERR_NEXT)))
    wrote(p, K_FE, first, count);
  if (flags & DPC_FWD_COPY_NEXT)
    wrote(p, K_Z, first + 1, count);
  return DPC_OK;
}

// Runs the jobs side by side: job 0 (the largest, by convention) on the context's stream, the others
// on up to three streams that fork from it and join it (inside a graph capture: parallel branches).
// The launches of one phase are independent of each other, and most of them leave SMs idle -- a head,
// a cached input layer, a bias sum beside the tensor-core run -- so one after the other they would add
// their latencies.
int dpc::run_side_by_side(dpc_ctx* ctx, const std::vector<Job>& jobs)
{
  int rc = DPC_OK;
  if (jobs.size() < 2 || !ctx->fork_ev)
  {
    for (size_t q = 0; q < jobs.size() && rc == DPC_OK; ++q)
      rc = jobs[q]();
    return rc;
  }
  cudaStream_t main_stream = ctx->stream;
  const int used = std::min((int)jobs.size() - 1, dpc_ctx::kSide);
  bool forked = cudaEventRecord(ctx->fork_ev, main_stream) == cudaSuccess;
  for (int s = 0; s < used && forked; ++s)
    forked = cudaStreamWaitEvent(ctx->side[s], ctx->fork_ev, 0) == cudaSuccess;
  if (!forked)
    return cuda_fail(cudaGetLastError(), "fork of the per-layer streams");
  for (size_t q = 0; q < jobs.size() && rc == DPC_OK; ++q)
  {
    const int lane = (int)q % (used + 1);
    ctx->stream = lane == 0 ? main_stream : ctx->side[lane - 1];
    rc = jobs[q]();
  }
  ctx->stream = main_stream;
  // join whatever happened: a capture must not end with a stream still forked
  bool joined = true;
  for (int s = 0; s < used; ++s)
    joined &= cudaEventRecord(ctx->join_ev[s], ctx->side[s]) == cudaSuccess &&
              cudaStreamWaitEvent(main_stream, ctx->join_ev[s], 0) == cudaSuccess;
  if (rc != DPC_OK)
    return rc;
  return joined ? DPC_OK : cuda_fail(cudaGetLastError(), "join of the per-layer streams");
}

// Splits [first, first+count) into what the tensor-core path takes (the part inside the run as
// one piece, single layers outside it that fit the CTA-pair kernels one by one) and maximal
// pieces for the CUDA-core kernels.  A piece the tensor-core entry point declines (returns 1)
// goes to the CUDA-core kernels too.  run_first: the run comes first in the list.
template <typename TcFn, typename SimtFn>
static std::vector<Job> pieces_of(dpc_plan* p, int first, int count, TcFn tc, SimtFn simt, bool run_first)
{
  const int end = first + count;
  const int run0 = p->run.first, run1 = p->run.first + p->run.count;
  std::vector<Job> jobs;
  int i = first;
  while (i < end)
  {
    int j = i + 1;
    const bool in_run = p->run.count > 0 && i >= run0 && i < run1;
    if (in_run || tc_extra_layer(p, i))
    {
      if (in_run)
        j = std::min(end, run1);
      Job job = [=]
      {
        const int rc = tc(i, j - i);
        return rc > 0 ? simt(i, j - i) : rc;
      };
      if (in_run && run_first)
        jobs.insert(jobs.begin(), job);
      else
        jobs.push_back(job);
    }
    else
    {
      while (j < end && !(p->run.count > 0 && j >= run0 && j < run1) && !tc_extra_layer(p, j))
        ++j;
      jobs.push_back([=] { return simt(i, j - i); });
    }
    i = j;
  }
  return jobs;
}

// `independent`: the layers of the range neither read what another layer of the range writes nor
// write the same tensors (true of a settle pass, a state update and a weight update; not of a
// sweep): the pieces run side by side.
template <typename TcFn, typename SimtFn>
static int dispatch_range(dpc_plan* p, int first, int count, TcFn tc, SimtFn simt, bool independent = false)
{
  const std::vector<Job> jobs = pieces_of(p, first, count, tc, simt, independent);
  if (independent)
    return run_side_by_side(p->ctx, jobs);
  int rc = DPC_OK;
  for (size_t q = 0; q < jobs.size() && rc == DPC_OK; ++q)
    rc = jobs[q]();
  return rc;
}

int dpc_forward(dpc_plan* p, int first, int count, int flags)
{
  int rc = check_range(p, first, count);
  if (rc != DPC_OK)
    return rc;
  const bool head_cached = ((flags & DPC_FWD_CACHED) && first + count >= p->n - 1) ||
                           ((flags & DPC_FWD_CACHED_FIRST) && first == p->n - 2);
  if ((flags & DPC_FWD_CE) && (head_cached || !dpc_plan_fused_cross_entropy(p)))
    return fail(DPC_ERR_INVALID, "DPC_FWD_CE: the head's forward kernel does not run, use dpc_error");
  if (flags & DPC_FWD_CACHED)
    return forward_simt(p, first, count, flags);
  const bool cached_first = (flags & DPC_FWD_CACHED_FIRST) && count > 0;
  flags &= ~DPC_FWD_CACHED_FIRST;
  const bool independent = !(flags & DPC_FWD_COPY_NEXT);
  const int skip = cached_first ? 1 : 0;
  std::vector<Job> jobs = pieces_of(
      p, first + skip, count - skip, [=](int f, int c) { return tc_forward(p, f, c, flags); },
      [=](int f, int c) { return forward_simt(p, f, c, flags); }, independent);
  if (cached_first)
  {
    // (transient passes: a refresh recomputes the feedback error of this clamped layer before anyone
    // reads it, so a settling step computes the error alone)
    const int keep = (flags & DPC_FWD_TRANSIENT) && (flags & DPC_FWD_ERR_NEXT) ? ~DPC_FWD_FE : ~0;
    const Job cached = [=] { return forward_simt(p, first, 1, (flags & keep) | DPC_FWD_CACHED); };
    // beside the others; in a sweep before them
    jobs.insert(independent ? jobs.end() : jobs.begin(), cached);
  }
  if (independent)
    return run_side_by_side(p->ctx, jobs);
  for (size_t q = 0; q < jobs.size() && rc == DPC_OK; ++q)
    rc = jobs[q]();
  return rc;
}

int dpc_plan_fused_cross_entropy(dpc_plan* p)
{
  if (!p || p->n < 2 || !(p->h[p->n - 1].flags & DPC_LAYER_SOFTMAX_CE))
    return 0;
  const int head = p->n - 2;
  auto tensor = [&](int l)
  { return (p->run.count > 0 && l >= p->run.first && l < p->run.first + p->run.count) || tc_extra_layer(p, l); };
  // where the head shares the grouped launch of other layers, a launch of its own would cost more than the
  // two small kernels it replaces: only above the (clamped, separate) input layer or a tensor-core layer
  return head >= 1 && narrow_forward(p, head) && !tensor(head) && (head == 1 || tensor(head - 1)) ? 1 : 0;
}

int dpc_plan_state_from_prediction(dpc_plan* p)
{
  return p && tc_run_ready(p) && p->run.first <= 1 && p->run.first + p->run.count > 1 && p->h[0].mu &&
                 (uintptr_t)p->h[0].mu % 32 == 0 && !(p->h[1].flags & DPC_LAYER_SOFTMAX_CE)
             ? 1
             : 0;
}

int dpc_project_forward(dpc_plan* p, int first, int count, int skip_last_copy)
{
  return dpc_project_forward_ex(p, first, count, skip_last_copy, 0);
}

int dpc_project_forward_ex(dpc_plan* p, int first, int count, int skip_last_copy, int extra)
{
  extra &= DPC_FWD_NO_MU | DPC_FWD_NO_PREACT;
  int rc = check_range(p, first, count);
  if (rc != DPC_OK)
    return rc;
  int i0 = first;
  // The part of the sweep inside the tensor-core run goes out as one persistent launch.
  if (p->run.count > 0 && first <= p->run.first && first + count >= p->run.first + p->run.count &&
      !(skip_last_copy && p->run.first + p->run.count + 1 == p->n))
  {
    for (int i = first; i < p->run.first; ++i)
      if ((rc = dpc_forward(p, i, 1, DPC_FWD_COPY_NEXT | (i == first ? 0 : extra))) != DPC_OK)
        return rc;
    // (the chain kernel itself keeps mu of the sweep's very first layer when it starts there)
    rc = tc_project_forward(p, p->run.first, p->run.count,
                            DPC_FWD_COPY_NEXT | extra | (p->run.first == first ? (1 << 10) : 0));
    if (rc < 0)
      return rc;
    i0 = rc == DPC_OK ? p->run.first + p->run.count : p->run.first;
  }
  for (int i = i0; i < first + count; ++i)
  {
    if (p->h[i].next_size <= 0)
      continue;
    int flags = DPC_FWD_COPY_NEXT | (i == first ? 0 : extra);
    if (skip_last_copy && i + 2 == p->n)
      flags = 0;
    rc = dpc_forward(p, i, 1, flags);
    if (rc != DPC_OK)
      return rc;
  }
  return DPC_OK;
}

int dpc_error(dpc_plan* p, int layer, int with_energy)
{
  int rc = check_range(p, layer, 1);
  if (rc != DPC_OK)
    return rc;
  if (layer == 0)
    return fail(DPC_ERR_INVALID, "dpc_error: the input layer has no prediction below it");
  const dpc_layer& L = p->h[layer];
  cudaStream_t st = p->ctx->stream;
  if (p->h[layer - 1].flags & DPC_LAYER_INPUT_ACT)
    wrote(p, K_FE, layer - 1, 1);
  if (L.flags & DPC_LAYER_SOFTMAX_CE)
  {
    int blocks = std::min(cdiv(p->batch, NTHREADS / 32), p->ctx->sm_count * 8);
    softmax_ce_kernel<<<blocks, NTHREADS, 0, st>>>(p->d, layer, p->batch, with_energy, p->energy);
  }
  else
  {
    error_kernel<<<elem_blocks(p, (size_t)p->batch * L.size), NTHREADS, 0, st>>>(
        p->d, layer, p->batch, with_energy, p->energy);
  }
  return check_launch(p->ctx, "error kernel");
}

int dpc_feedback_error(dpc_plan* p, int first, int count)
{
  int rc = check_range(p, first, count);
  if (rc != DPC_OK || count == 0)
    return rc;
  for (int f = first; f < first + count; f += kMaxZ)
  {
    const int c = std::min(kMaxZ, first + count - f);
    size_t mx = 0;
    for (int i = f; i < f + c; ++i)
      mx = std::max(mx, (size_t)p->batch * std::max(p->h[i].next_size, 0));
    dim3 grid(elem_blocks(p, mx), c);
    feedback_error_kernel<<<grid, NTHREADS, 0, p->ctx->stream>>>(p->d, f, p->n, p->batch);
    if ((rc = check_launch(p->ctx, "feedback_error kernel")) != DPC_OK)
      return rc;
  }
  wrote(p, K_FE, first, count);
  return DPC_OK;
}

// Largest output width of layers [f, f+c) when every one of them is "narrow above" (1..16 output
// units, an input width that is a multiple of 128, 16-byte aligned tensors, a batch of at least 256
// rows: the layer under a head on a large batch), else 0.  Such layers have kernels of their own
// for the state update and the weight update (narrow_state_kernel, narrow_weight_kernel).
static int narrow_above(const dpc_plan* p, int f, int c)
{
  if (p->batch < 256)
    return 0;
  int widest = 0;
  for (int i = f; i < f + c; ++i)
  {
    const dpc_layer& L = p->h[i];
    const bool simple = (L.flags & DPC_LAYER_INPUT_ACT) != 0;
    const float* g = simple ? (i + 1 < p->n ? p->h[i + 1].e : nullptr) : L.fe;
    const float* zin = simple ? L.zF : L.z;
    if (L.next_size <= 0 || L.next_size > 16 || L.size % 128 != 0 || !g || !zin || !L.W || !L.z ||
        !L.e || ((uintptr_t)zin % 16) != 0 || ((uintptr_t)L.W % 16) != 0 || ((uintptr_t)L.z % 16) != 0 ||
        ((uintptr_t)L.e % 16) != 0 || (L.v && ((uintptr_t)L.v % 16) != 0) ||
        (i + 1 < p->n && p->h[i + 1].e && ((uintptr_t)p->h[i + 1].e % 16) != 0))
      return 0;
    widest = std::max(widest, L.next_size);
  }
  return widest;
}

static int update_state_simt(dpc_plan* p, int first, int count)
{
  cudaStream_t st = p->ctx->stream;
  wrote(p, K_Z, first, count);
  for (int f = first; f < first + count; f += kMaxZ)
  {
    const int c = std::min(kMaxZ, first + count - f);
    // Layers whose upper neighbour does not exist are handled by the relax kernel below.
    int cg = (f + c == p->n) ? c - 1 : c;
    int narrow_kc = cg > 0 ? narrow_above(p, f, cg) : 0;
    if (narrow_kc > 0)
    {
      // layers under a narrow one (the heads): 128 columns x a share of the batch rows per block
      int mxs = 0;
      bool plain = true; // no momentum, no residual term
      for (int i = f; i < f + cg; ++i)
      {
        mxs = std::max(mxs, p->h[i].size);
        plain = plain && ((p->h[i].flags & DPC_LAYER_INPUT_ACT) || (!p->h[i].v && !(p->h[i].flags & DPC_LAYER_RESIDUAL)));
      }
      const int gx = cdiv(mxs, 128);
      int rpb = cdiv(p->batch, 32) * 32;
      while (rpb > 32 && (long long)gx * cg * cdiv(p->batch, rpb) < p->ctx->sm_count)
        rpb = cdiv(rpb / 2, 32) * 32;
      dim3 grid(gx, cdiv(p->batch, rpb), cg);
      auto kern = narrow_kc <= 12 ? (plain ? narrow_state_kernel<12, true> : narrow_state_kernel<12, false>)
                                  : (plain ? narrow_state_kernel<16, true> : narrow_state_kernel<16, false>);
      static thread_local int configured[4] = {-1, -1, -1, -1};
      int& device = configured[2 * (narrow_kc <= 12) + plain];
      if (device != p->ctx->device)
      {
        DPC_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kHeadStateSmem));
        device = p->ctx->device;
      }
      kern<<<grid, 256, kHeadStateSmem, st>>>(p->d, f, p->n, p->batch, rpb);
      int rc = check_launch(p->ctx, "narrow update_state kernel");
      if (rc != DPC_OK)
        return rc;
    }
    else if (cg > 0)
    {
      const int rc = launch_gemm<OP_FB>(p, f, cg, 0, FB_STATE);
      if (rc != DPC_OK)
        return rc;
    }
    bool any_weightless = false;
    size_t mx = 0;
    for (int i = f; i < f + c; ++i)
      if (p->h[i].next_size <= 0 || i + 1 >= p->n)
      {
        any_weightless = true;
        mx = std::max(mx, (size_t)p->batch * p->h[i].size);
      }
    if (any_weightless)
    {
      dim3 grid(elem_blocks(p, mx), c);
      relax_kernel<<<grid, NTHREADS, 0, st>>>(p->d, f, p->n, p->batch, 1);
      int rc = check_launch(p->ctx, "relax kernel");
      if (rc != DPC_OK)
        return rc;
    }
  }
  return DPC_OK;
}

int dpc_update_state(dpc_plan* p, int first, int count)
{
  return dpc_update_state_ex(p, first, count, first + count, 0);
}

int dpc_update_state_ex(dpc_plan* p, int first, int count, int relax_from, int flags)
{
  int rc = check_range(p, first, count);
  if (rc != DPC_OK)
    return rc;
  const int end = first + count;
  relax_from = std::min(std::max(relax_from, first), end);
  const bool from_mu = (flags & DPC_STATE_FIRST_MU) != 0;
  if (from_mu && (first != 1 || relax_from == first || !dpc_plan_state_from_prediction(p)))
    return fail(DPC_ERR_INVALID, "DPC_STATE_FIRST_MU: the range does not start at a tensor-core layer 1");
  std::vector<Job> jobs = pieces_of(
      p, first, relax_from - first,
      [=](int f, int c) { return tc_update_state(p, f, c, (flags & DPC_STATE_FEED) != 0, from_mu && f == first); },
      [=](int f, int c) { return update_state_simt(p, f, c); }, true);
  for (int i = relax_from; i < end; ++i)
    jobs.push_back([=] { return dpc_relax(p, i); });
  return run_side_by_side(p->ctx, jobs);
}

int dpc_epc_reconstruct(dpc_plan* p, int layer)
{
  int rc = check_range(p, layer, 1);
  if (rc != DPC_OK)
    return rc;
  if (layer == 0)
    return fail(DPC_ERR_INVALID, "dpc_epc_reconstruct: the input layer has nothing below it");
  wrote(p, K_Z, layer, 1);
  epc_reconstruct_kernel<<<elem_blocks(p, (size_t)p->batch * p->h[layer].size), NTHREADS, 0,
                           p->ctx->stream>>>(p->d, layer, p->batch);
  return check_launch(p->ctx, "epc_reconstruct kernel");
}

int dpc_epc_adjoint(dpc_plan* p, int layer, int from_terminal, float scale, int clamped)
{
  int rc = check_range(p, layer, 1);
  if (rc != DPC_OK)
    return rc;
  const dpc_layer& L = p->h[layer];
  if (layer + 1 >= p->n || L.next_size <= 0 || !L.adj || !L.fe || !L.preact)
    return fail(DPC_ERR_INVALID, "dpc_epc_adjoint: layer has no weights, no adjoint buffer or no "
                                 "upper neighbour");
  const float* src = from_terminal ? p->h[p->n - 1].e : p->h[layer + 1].adj;
  if (!src)
    return fail(DPC_ERR_INVALID, "dpc_epc_adjoint: the layer above has no adjoint buffer");
  cudaStream_t st = p->ctx->stream;
  wrote(p, K_FE, layer, 1);
  epc_source_kernel<<<elem_blocks(p, (size_t)p->batch * L.next_size), NTHREADS, 0, st>>>(
      p->d, layer, p->batch, src);
  if ((rc = check_launch(p->ctx, "epc_source kernel")) != DPC_OK)
    return rc;
  // hop scale travels as float bits with the lowest mantissa bit replaced by the clamp flag
  // (scale is +1 or -1, whose lowest mantissa bit is zero)
  union
  {
    float f;
    int i;
  } u;
  u.f = scale;
  const int packed = (u.i & ~1) | (clamped ? 1 : 0);
  return launch_gemm<OP_FB>(p, layer, 1, packed, FB_ADJOINT, src);
}

int dpc_relax(dpc_plan* p, int layer)
{
  int rc = check_range(p, layer, 1);
  if (rc != DPC_OK)
    return rc;
  dim3 grid(elem_blocks(p, (size_t)p->batch * p->h[layer].size), 1);
  wrote(p, K_Z, layer, 1);
  relax_kernel<<<grid, NTHREADS, 0, p->ctx->stream>>>(p->d, layer, p->n, p->batch, 0);
  return check_launch(p->ctx, "relax kernel");
}

// Whether a layer is on the tensor-core path.
static bool tc_piece(dpc_plan* p, int i)
{
  return (p->run.count > 0 && i >= p->run.first && i < p->run.first + p->run.count) || tc_extra_layer(p, i);
}

// Batch products (dpc_batch.cuh) of layers [first, first+count), for networks whose sums may be split.
// weights: the weight sums of the layers for which it holds; with_sums (learn): their bias sums and the Psi
// sums of all layers too.
template <typename F>
static int launch_batch_products(dpc_plan* p, int first, int count, int mode, int flags, F weights, bool with_sums)
{
  bool tensor = p->run.count > 0;
  for (int i = 0; i < p->n && !tensor; ++i)
    tensor = tc_extra_layer(p, i);
  for (int f = first, end; f < first + count; f = end)
  {
    // DirectFeedbackUpdate is a no-op unless the layer above owns feedback weights
    auto sums = [&](int i)
    { return weights(i) && ((mode & ~WG_GRAD_ONLY) != WG_DFA || (i + 1 < p->n && p->h[i + 1].Psi)); };
    auto tiles_of = [&](int i)
    {
      const dpc_layer& L = p->h[i];
      const bool psi = with_sums && L.Psi && !(L.flags & DPC_LAYER_INPUT_ACT);
      return L.next_size <= 0 ? 0
                              : ((sums(i) ? cdiv(L.next_size, BP_T) : 0) + (psi ? cdiv(L.terminal_size, BP_T) : 0)) *
                                    cdiv(L.size, BP_T);
    };
    BatchTiles T;
    T.sums = with_sums;
    end = first + count;
    const int tiles = list_tiles(T.list, f, end, tiles_of, weights);
    if (tiles == 0)
      continue;
    // CTAs of a cluster that share a tile's batch rows: two groups of rows or more for each warp; beside
    // tensor-core launches, which wait where clusters take the SMs, eight (us a step with two / eight:
    // 784-(256x8)-10 at batch 256 274 / 267, at batch 512 245 / 235; with 32 / eight, i.e. single CTAs / pairs at
    // batch 1024: 512-(512x12)-10 515 / 511, in tf32 mode 466 / 458, 768-(768x6)-10 498 / 490).
    const int rows = BP_WARPS * BP_ROWS * (tensor ? 8 : 2);
    int R = 1;
    while (R < 8 && (long long)tiles * R < 2LL * p->ctx->sm_count && p->batch >= 2 * R * rows)
      R *= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(tiles * R));
    cfg.blockDim = dim3(32 * BP_WARPS);
    cfg.stream = p->ctx->stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim = {(unsigned)R, 1, 1};
    cfg.attrs = attr;
    cfg.numAttrs = R > 1 ? 1 : 0;
    cudaLaunchKernelEx(&cfg, batch_product_kernel, (const dpc_layer*)p->d, p->batch, flags, mode,
                       (const float*)p->e_terminal, T);
    const int rc = check_launch(p->ctx, "batch product kernel");
    if (rc != DPC_OK)
      return rc;
  }
  return DPC_OK;
}

// Before the weight sums of layers outside the tensor-core kernels: the operand of SimplePC layers is brought
// up to date, and the weights' operand planes are about to be behind.
static int weight_sums_begin(dpc_plan* p, int first, int count, int mode)
{
  if (!(mode & WG_GRAD_ONLY))
    wrote(p, K_W, first, count);
  return tc_zf_need(p, first, count);
}

// Whether the weight sums of layers [first, first+count) outside the tensor-core path are left to pc_gemm_kernel in a
// network whose sums may be split: where there are tiles for every SM several times over, no batch has to be split,
// and 64 x 64 outputs take half the operand traffic of batch_product_kernel's 32 x 32 (which costs 1.3 us a tile and SM
// however few the rows).  us a step, batch products / pc_gemm_kernel, by 32 x 32 tiles an SM and the 64 x 64 ones' area
// over theirs:  5.6, 1.0 (784-999-10, batch 16, 500, 2100) 221 / 220, 334 / 371, 629 / 781;  8.0, 1.3 (24 layers of 200,
// batch 16, 500) 302 / 291, 658 / 699;  10.8, 1.0 (100 layers of 128, batch 16, 500, 2100) 627 / 616, 1132 / 1096,
// 2779 / 2735;  10.8, 1.0 (three of 865, SimplePC, batch 192) 606 / 617;  11.2, 1.09 (four layers of 736, batch 48,
// 500) 248 / 236, 703 / 719;  13.8, 1.0 (eight of 512, batch 100, 2100) 389 / 381, 2339 / 2299;  20, 1.3 (60 of 200,
// batch 48, 500) 685 / 667, 1403 / 1444;  97, 1.0 (fourteen of 1024, batch 16, 1000) 889 / 738, 7720 / 7380.
static bool weights_by_gemm(dpc_plan* p, int first, int count)
{
  long long tiles = 0, tiles64 = 0;
  for (int i = first; i < first + count; ++i)
    if (p->h[i].next_size > 0 && !tc_piece(p, i))
    {
      const int M = p->h[i].next_size, N = p->h[i].size;
      tiles += (long long)cdiv(M, 32) * cdiv(N, 32), tiles64 += (long long)cdiv(M, 64) * cdiv(N, 64);
    }
  return tiles >= 12LL * p->ctx->sm_count && (p->batch <= 64 || 80 * tiles64 <= 21 * tiles);
}

static int weight_gemm_simt(dpc_plan* p, int first, int count, int mode, int flags)
{
  const int ready = weight_sums_begin(p, first, count, mode);
  if (ready != DPC_OK)
    return ready;
  if (!ordered_sums(p))
    return weights_by_gemm(p, first, count)
               ? launch_gemm<OP_WG>(p, first, count, flags, mode)
               : launch_batch_products(p, first, count, mode, flags, [](int) { return true; }, false);
  for (int f = first; f < first + count; f += kMaxZ)
  {
    const int c = std::min(kMaxZ, first + count - f);
    const int narrow_kc = narrow_above(p, f, c);
    bool staged_ok = true;
    for (int i = f; i < f + c; ++i)
      staged_ok &= !(mode & WG_GRAD_ONLY) || (p->h[i].g_W != nullptr);
    if (narrow_kc > 0 && staged_ok)
    {
      // heads on a large batch: the batch split over warps and the CTAs of a cluster
      int mxs = 0;
      for (int i = f; i < f + c; ++i)
        mxs = std::max(mxs, p->h[i].size);
      dim3 g(cdiv(mxs, 128), c);
      const int R = row_split(p->ctx, (long long)g.x * c, p->batch, 256);
      if (narrow_kc <= 12)
        launch_row_split(narrow_weight_kernel<12>, g, 256, R, p->ctx->stream, p->d, f, p->n,
                         p->batch, flags, mode);
      else
        launch_row_split(narrow_weight_kernel<16>, g, 256, R, p->ctx->stream, p->d, f, p->n,
                         p->batch, flags, mode);
      int rc = check_launch(p->ctx, "narrow weight kernel");
      if (rc != DPC_OK)
        return rc;
      continue;
    }
    const int rc = launch_gemm<OP_WG>(p, f, c, flags, mode);
    if (rc != DPC_OK)
      return rc;
  }
  return DPC_OK;
}

// The DFA projection over layers [first, first+count): four-units-per-thread kernel where the
// shapes allow it, the general kernel elsewhere.
static int launch_dfa_group(dpc_plan* p, int i, int c, int from_output, bool v, const FePlanes& planes);
static int launch_dfa_proj(dpc_plan* p, int first, int count, int from_output)
{
  wrote(p, K_FE, first, count);
  const FePlanes planes = fe_planes(p);
  auto vec_ok = [&](int i)
  {
    const dpc_layer& L = p->h[i];
    return L.next_size > 0 && L.next_size % 4 == 0 && L.terminal_size <= 16 &&
           ((uintptr_t)L.fe % 16 == 0) && ((uintptr_t)L.preact % 16 == 0) &&
           (i + 1 >= p->n || (uintptr_t)p->h[i + 1].z % 16 == 0);
  };
  std::vector<Job> jobs;
  int i = first;
  while (i < first + count)
  {
    const bool v = vec_ok(i);
    int j = i + 1;
    while (j < first + count && j - i < kMaxZ && vec_ok(j) == v &&
           (!v || p->h[j].terminal_size == p->h[i].terminal_size))
      ++j;
    const int c = j - i;
    // (the layer under the terminal has no feedback weights above it: nothing to do)
    bool any = false;
    for (int k = i; k < j; ++k)
      any |= p->h[k].next_size > 0 && k + 1 < p->n && p->h[k + 1].Psi != nullptr;
    if (any)
      jobs.push_back([=] { return launch_dfa_group(p, i, c, from_output, v, planes); });
    i = j;
  }
  return run_side_by_side(p->ctx, jobs);
}

static int launch_dfa_group(dpc_plan* p, int i, int c, int from_output, bool v, const FePlanes& planes)
{
  cudaStream_t st = p->ctx->stream;
  const int j = i + c;
  int mxn = 1;
  for (int k = i; k < j; ++k)
    mxn = std::max(mxn, p->h[k].next_size);
  bool wide = v;
  for (int k = i; k < j && wide; ++k)
    wide = p->h[k].next_size <= 0 || p->h[k].next_size % 128 == 0;
  const int ts4 = cdiv(std::max(p->h[i].terminal_size, 1), 4);
  const long long strips = (long long)cdiv(mxn, 128) * c;
  // rows per block of the other two: 32, fewer while SMs are left without a block (the rows of a block
  // follow one another: 8 blocks of 32 rows took 24 us for 100-300-200-77-10 at batch 50)
  auto few_rows = [&](int blocks)
  {
    int rpb = 32;
    while (rpb > 4 && (long long)blocks * cdiv(p->batch, rpb) < p->ctx->sm_count)
      rpb /= 2;
    return rpb;
  };
  if (wide && ts4 <= 4)
  {
    // blocks of 128 columns x the whole batch, or a share of it while there are fewer than four blocks
    // per SM: FullPCN 3072-(1024x4)-10 at batch 4096 has 32 strips
    int rpb = cdiv(p->batch, 32) * 32;
    while (rpb > 32 && strips * cdiv(p->batch, rpb) < 4 * p->ctx->sm_count)
      rpb = cdiv(rpb / 2, 32) * 32;
    dim3 grid(cdiv(mxn, 128), c, cdiv(p->batch, rpb));
    if (ts4 <= 1)
      dfa_proj128_kernel<1><<<grid, 256, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb, planes);
    else if (ts4 == 2)
      dfa_proj128_kernel<2><<<grid, 256, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb, planes);
    else if (ts4 == 3)
      dfa_proj128_kernel<3><<<grid, 256, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb, planes);
    else
      dfa_proj128_kernel<4><<<grid, 256, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb, planes);
  }
  else if (v)
  {
    int rpb = DFA4_ROWS;
    if (cdiv(mxn, 256) * cdiv(p->batch, rpb) * c < 4 * p->ctx->sm_count)
      rpb = few_rows(cdiv(mxn, 256) * c);
    dim3 grid(cdiv(mxn, 256), cdiv(p->batch, rpb), c);
    if (ts4 <= 1)
      dfa_proj4_kernel<1><<<grid, 64, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb, planes);
    else if (ts4 == 2)
      dfa_proj4_kernel<2><<<grid, 64, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb, planes);
    else if (ts4 == 3)
      dfa_proj4_kernel<3><<<grid, 64, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb, planes);
    else
      dfa_proj4_kernel<4><<<grid, 64, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb, planes);
  }
  else
  {
    const int rpb = few_rows(cdiv(mxn, 128) * c);
    dim3 grid(cdiv(mxn, 128), cdiv(p->batch, rpb), c);
    dfa_proj_kernel<<<grid, 128, 0, st>>>(p->d, i, p->n, p->batch, p->e_terminal, from_output, rpb);
  }
  int rc = check_launch(p->ctx, "dfa_proj kernel");
  if (rc != DPC_OK)
    return rc;
  if (v && planes.fe)
    tc_fe_written(p, i, c); // this kernel wrote the operand copies itself
  return DPC_OK;
}

int dpc_direct_feedback(dpc_plan* p, int first, int count, int decay_w)
{
  int rc = check_range(p, first, count);
  if (rc != DPC_OK || count == 0)
    return rc;
  // Only layers with an upper neighbour can take part.
  if (first + count == p->n)
    count -= 1;
  if (count <= 0)
    return DPC_OK;
  if ((rc = launch_dfa_proj(p, first, count, (decay_w & DPC_DFA_FROM_OUTPUT) ? 1 : 0)) != DPC_OK)
    return rc;
  decay_w &= DPC_DFA_DECAY_W;
  const int flags = decay_w ? 1 : 0;
  return dispatch_range(
      p, first, count, [&](int f, int c) { return tc_weight_gemm(p, f, c, WG_DFA, decay_w); },
      [&](int f, int c) { return weight_gemm_simt(p, f, c, WG_DFA, flags); }, /*independent=*/true);
}

// Psi update (or its raw sums) of layers [f, f+c): the 128-columns-per-block kernel when every
// layer of the launch that has feedback weights is a multiple of 128 wide with at most 16
// terminal units, the general kernel otherwise.
static int launch_psi_range(dpc_plan* p, int f, int c, int max_size, int grad_only, bool fast)
{
  cudaStream_t st = p->ctx->stream;
  int ts = 0;
  for (int i = f; i < f + c && i < p->n; ++i)
    if (p->h[i].next_size > 0 && p->h[i].Psi != nullptr)
      ts = std::max(ts, p->h[i].terminal_size);
  if (fast && ts > 0)
  {
    dim3 g(std::max(1, cdiv(max_size, 128)), c);
    const int R = row_split(p->ctx, (long long)g.x * c, p->batch, 256);
    if (ts <= 12)
      launch_row_split(psi_update4_kernel<12>, g, 256, R, st, p->d, f, p->n, p->batch,
                       p->e_terminal, grad_only);
    else
      launch_row_split(psi_update4_kernel<16>, g, 256, R, st, p->d, f, p->n, p->batch,
                       p->e_terminal, grad_only);
  }
  else
  {
    dim3 g(std::max(1, cdiv(max_size, 32)), c, std::max(1, cdiv(ts, 16)));
    psi_update_kernel<<<g, 256, 0, st>>>(p->d, f, p->n, p->batch, p->e_terminal, grad_only);
  }
  return check_launch(p->ctx, grad_only ? "psi gradient kernel" : "psi_update kernel");
}

static void psi_jobs(dpc_plan* p, int f, int c, int grad_only, std::vector<Job>& jobs)
{
  auto has_psi = [&](int i)
  { return p->h[i].next_size > 0 && p->h[i].Psi != nullptr && !(p->h[i].flags & DPC_LAYER_INPUT_ACT); };
  auto fits = [&](int i) { return !has_psi(i) || (p->h[i].size % 128 == 0 && p->h[i].terminal_size <= 16); };
  bool all = true, adam = false;
  for (int i = f; i < f + c && i < p->n; ++i)
    all &= fits(i), adam |= has_psi(i) && p->h[i].opt_psi != DPC_OPT_SGD;
  // Layers of both kinds: each run with its kernel (Adam-type updates keep one order of additions for
  // all, that of the general kernel).
  int i = f;
  while (i < f + c)
  {
    const bool fast = all || (!adam && fits(i));
    int j = i, mx = 0;
    while (j < f + c && (all || adam || fits(j) == fits(i)))
      mx = std::max(mx, p->h[j].size), ++j;
    jobs.push_back([=] { return launch_psi_range(p, i, j - i, mx, grad_only, fast); });
    i = j;
  }
}

// Bias update (or its raw sums) of layers [f, f+c).
static int launch_bias_update(dpc_plan* p, int f, int c, int grad_only)
{
  int max_next = 0;
  for (int i = f; i < f + c; ++i)
    max_next = std::max(max_next, p->h[i].next_size);
  const int rc = tc_fe_need(p, f, c);
  if (rc != DPC_OK)
    return rc;
  const FePlanes fp = fe_planes(p);
  // 256 threads: blocks of 64 columns where the feedback error is read from its planes or the batch is
  // large, of 32 columns elsewhere (a block takes several where the layer's own kind differs).  The CTAs of a cluster
  // share the batch; 1024 rows each or more beside tensor-core products (us a step with 256 / 1024: 512-(512x12)-10 at
  // batch 1024 523 / 515, in tf32 mode 470 / 462, 768-(768x6)-10 501 / 492), 256 where the order may not change.
  const bool by_blocks = fp.only || p->batch >= kBiasBlockRows;
  dim3 gb(std::max(1, cdiv(max_next, by_blocks ? 64 : 32)), c);
  launch_row_split(bias_update_kernel, gb, 256,
                   by_blocks ? row_split(p->ctx, (long long)gb.x * c, p->batch, ordered_sums(p) ? 256 : 1024) : 1,
                   p->ctx->stream, p->d, f, p->n, p->batch, grad_only, fp);
  return check_launch(p->ctx, "bias_update kernel");
}

// Jobs of a learn phase (grad_only: the raw sums): the weight sums of tensor-core pieces by `tc`, the others',
// bias and Psi sums by the kernels of this file.
template <typename TcFn>
static std::vector<Job> learn_jobs(dpc_plan* p, int first, int count, int grad_only, TcFn tc)
{
  const int mode = WG_LEARN | (grad_only ? WG_GRAD_ONLY : 0);
  auto simt = [=](int f, int c) { return weight_gemm_simt(p, f, c, mode, 0); };
  std::vector<Job> jobs;
  if (ordered_sums(p))
  {
    jobs = pieces_of(p, first, count, tc, simt, true);
    bool psi = false;
    for (int i = first; i < first + count; ++i)
      psi |= p->h[i].Psi != nullptr && !(p->h[i].flags & DPC_LAYER_INPUT_ACT);
    for (int f = first; f < first + count; f += kMaxZ)
    {
      const int c = std::min(kMaxZ, first + count - f);
      jobs.push_back([=] { return launch_bias_update(p, f, c, grad_only); });
      if (psi)
        psi_jobs(p, f, c, grad_only, jobs);
    }
    return jobs;
  }
  // Psi of tensor-core layers: strips of 128 columns x the whole batch where there are enough of them; tiles that
  // share the batch else, in one launch with the sums of the other layers (a 32 x 32 tile of ten terminal units
  // multiplies 1.6 times what it keeps).  us a step, strips / tiles: 40 layers of 512 at batch 1024 (160 strips)
  // 1272 / 1254, 150 of 256 at batch 512 (300) 1813 / 1801, 155 of 512 (620) 4183 / 4149 with runs 50 apart, 300 of
  // 512 (1200) 7860 / 7895.
  long long strips = 0;
  for (int i = first; i < first + count; ++i)
    if (tc_piece(p, i) && p->h[i].Psi && p->h[i].size % 128 == 0 && p->h[i].terminal_size <= 16)
      strips += p->h[i].size / 128;
  const bool by_strips = strips >= 4LL * p->ctx->sm_count, by_gemm = weights_by_gemm(p, first, count);
  auto sums = [=](int f, int c)
  {
    for (int i = f; i < f + c && !by_gemm; ++i)
      if (const int rc = tc_piece(p, i) ? DPC_OK : weight_sums_begin(p, i, 1, mode))
        return rc;
    return launch_batch_products(p, f, c, mode, 0, [=](int i) { return !by_gemm && !tc_piece(p, i); }, true);
  };
  for (int i = first, j; i < first + count; i = j)
  {
    const bool t = tc_piece(p, i);
    for (j = i + 1; j < first + count && j - i < kMaxZ && tc_piece(p, j) == t;)
      ++j;
    const int f = i, c = j - i;
    if (t)
    {
      // (a piece that `tc` declines gets its weight sums from `simt`)
      const std::vector<Job> own = pieces_of(p, f, c, tc, simt, true);
      jobs.insert(jobs.begin(), own.begin(), own.end());
      jobs.push_back([=] { return launch_bias_update(p, f, c, grad_only); });
      if (by_strips)
        psi_jobs(p, f, c, grad_only, jobs);
    }
    else
    {
      if (by_gemm)
      {
        jobs.insert(jobs.begin(), [=] { return simt(f, c); });
        jobs.push_back([=] { return launch_bias_update(p, f, c, grad_only); });
      }
      if (by_strips)
        jobs.push_back([=] { return sums(f, c); });
    }
  }
  if (!by_strips)
    jobs.push_back([=] { return sums(first, count); });
  return jobs;
}

int dpc_update_weights(dpc_plan* p, int first, int count, int center_rows)
{
  int rc = check_range(p, first, count);
  if (rc != DPC_OK || count == 0)
    return rc;
  if (first + count == p->n)
    count -= 1;
  if (count <= 0)
    return DPC_OK;
  bool any_adam = false;
  int max_next = 0;
  for (int i = first; i < first + count; ++i)
  {
    const dpc_layer& L = p->h[i];
    any_adam |= L.opt != DPC_OPT_SGD || (L.Psi && L.opt_psi != DPC_OPT_SGD);
    max_next = std::max(max_next, L.next_size);
  }
  if (any_adam)
  {
    bump_counters_kernel<<<cdiv(count, 256), 256, 0, p->ctx->stream>>>(p->d, first, count, p->n);
    if ((rc = check_launch(p->ctx, "bump_counters kernel")) != DPC_OK)
      return rc;
  }
  // the feedback-error planes are read by two of the jobs below: bring them up to date before the fork
  if ((rc = tc_fe_need(p, first, count)) != DPC_OK)
    return rc;
  const std::vector<Job> jobs = learn_jobs(
      p, first, count, 0,
      [=](int f, int c) -> int
      {
        bool all_sgd = true, all_staged = true;
        for (int i = f; i < f + c; ++i)
        {
          all_sgd &= p->h[i].opt == DPC_OPT_SGD;
          all_staged &= p->h[i].g_W != nullptr;
        }
        if (all_sgd)
          return tc_weight_gemm(p, f, c, WG_LEARN);
        if (!all_staged)
          return 1;
        // Adam-type optimizers: tensor-core product into the staging buffer, then the
        // optimizer as an elementwise kernel over W (b and Psi follow below as usual).
        int r = tc_weight_gemm(p, f, c, WG_LEARN | WG_GRAD_ONLY);
        if (r != DPC_OK)
          return r;
        size_t max_w = 1;
        for (int i = f; i < f + c; ++i)
          max_w = std::max(max_w, (size_t)p->h[i].next_size * p->h[i].size);
        for (int g = f; g < f + c; g += kMaxZ)
        {
          const int cc = std::min(kMaxZ, f + c - g);
          dim3 grid(elem_blocks(p, max_w), cc);
          wrote(p, K_W, g, cc);
          apply_gradients_kernel<<<grid, NTHREADS, 0, p->ctx->stream>>>(p->d, g, p->n, p->batch, 2, 0);
          if ((r = check_launch(p->ctx, "apply_gradients kernel")) != DPC_OK)
            return r;
        }
        return DPC_OK;
      });
  if ((rc = run_side_by_side(p->ctx, jobs)) != DPC_OK)
    return rc;
  for (int f = first; center_rows && f < first + count; f += kMaxZ)
  {
    const int c = std::min(kMaxZ, first + count - f);
    dim3 gc(std::min(max_next, 1024), c);
    wrote(p, K_W, f, c);
    center_rows_kernel<<<gc, 256, 0, p->ctx->stream>>>(p->d, f, p->n);
    if ((rc = check_launch(p->ctx, "center_rows kernel")) != DPC_OK)
      return rc;
  }
  return DPC_OK;
}

static int staging_ready(dpc_plan* p, int first, int count, int which)
{
  for (int i = first; i < first + count; ++i)
  {
    const dpc_layer& L = p->h[i];
    if (L.next_size <= 0)
      continue;
    if (!L.g_W || (which == 0 && (!L.g_b || (L.Psi && !(L.flags & DPC_LAYER_INPUT_ACT) && !L.g_Psi))))
      return fail(DPC_ERR_INVALID, "layer has no gradient staging buffers");
  }
  return DPC_OK;
}

int dpc_weight_gradients(dpc_plan* p, int first, int count, int which)
{
  int rc = check_range(p, first, count);
  if (rc != DPC_OK || count == 0)
    return rc;
  if (which != 0 && which != 1)
    return fail(DPC_ERR_INVALID, "which must be 0 (learn) or 1 (direct feedback)");
  if (first + count == p->n)
    count -= 1;
  if (count <= 0)
    return DPC_OK;
  if ((rc = staging_ready(p, first, count, which)) != DPC_OK)
    return rc;
  if (which == 1)
  {
    if ((rc = launch_dfa_proj(p, first, count, 0)) != DPC_OK)
      return rc;
    return dispatch_range(
        p, first, count,
        [&](int f, int c) { return tc_weight_gemm(p, f, c, WG_DFA | WG_GRAD_ONLY); },
        [&](int f, int c) { return weight_gemm_simt(p, f, c, WG_DFA | WG_GRAD_ONLY, 0); },
        /*independent=*/true);
  }
  if ((rc = tc_fe_need(p, first, count)) != DPC_OK)
    return rc;
  return run_side_by_side(
      p->ctx, learn_jobs(p, first, count, 1,
                         [=](int f, int c) { return tc_weight_gemm(p, f, c, WG_LEARN | WG_GRAD_ONLY); }));
}

int dpc_apply_gradients(dpc_plan* p, int first, int count, int which, int global_batch, int option)
{
  int rc = check_range(p, first, count);
  if (rc != DPC_OK || count == 0)
    return rc;
  if ((which != 0 && which != 1) || global_batch <= 0)
    return fail(DPC_ERR_INVALID, "bad which / global_batch");
  if (first + count == p->n)
    count -= 1;
  if (count <= 0)
    return DPC_OK;
  if ((rc = staging_ready(p, first, count, which)) != DPC_OK)
    return rc;
  cudaStream_t st = p->ctx->stream;
  bool any_adam = false;
  int max_next = 0;
  size_t max_w = 1;
  for (int i = first; i < first + count; ++i)
  {
    const dpc_layer& L = p->h[i];
    any_adam |= L.opt != DPC_OPT_SGD || (L.Psi && L.opt_psi != DPC_OPT_SGD);
    max_next = std::max(max_next, L.next_size);
    max_w = std::max(max_w, (size_t)std::max(L.next_size, 0) * L.size);
  }
  if (which == 0 && any_adam)
  {
    bump_counters_kernel<<<cdiv(count, 256), 256, 0, st>>>(p->d, first, count, p->n);
    if ((rc = check_launch(p->ctx, "bump_counters kernel")) != DPC_OK)
      return rc;
  }
  for (int f = first; f < first + count; f += kMaxZ)
  {
    const int c = std::min(kMaxZ, first + count - f);
    dim3 grid(elem_blocks(p, max_w), c);
    wrote(p, K_W, f, c);
    apply_gradients_kernel<<<grid, NTHREADS, 0, st>>>(p->d, f, p->n, global_batch, which, option ? 1 : 0);
    if ((rc = check_launch(p->ctx, "apply_gradients kernel")) != DPC_OK)
      return rc;
    if (which == 0 && option)
    {
      dim3 gc(std::min(max_next, 1024), c);
      center_rows_kernel<<<gc, 256, 0, st>>>(p->d, f, p->n);
      if ((rc = check_launch(p->ctx, "center_rows kernel")) != DPC_OK)
        return rc;
    }
  }
  return DPC_OK;
}

int dpc_energy_reset(dpc_plan* p)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  DPC_CUDA(cudaMemsetAsync(p->energy, 0, sizeof(double), p->ctx->stream));
  return DPC_OK;
}

int dpc_energy_read(dpc_plan* p, double* out)
{
  if (!p || !out)
    return fail(DPC_ERR_INVALID, "null argument");
  const int rc = dpc_energy_fetch(p);
  return rc == DPC_OK ? dpc_energy_wait(p, out) : rc;
}

int dpc_energy_fetch(dpc_plan* p)
{
  if (!p)
    return fail(DPC_ERR_INVALID, "null plan");
  DPC_CUDA(cudaMemcpyAsync(p->energy_host, p->energy, 2 * sizeof(double), cudaMemcpyDeviceToHost,
                           p->ctx->stream));
  return DPC_OK;
}

int dpc_energy_wait(dpc_plan* p, double* out)
{
  if (!p || !out)
    return fail(DPC_ERR_INVALID, "null argument");
  DPC_CUDA(cudaStreamSynchronize(p->ctx->stream));
  *out = *p->energy_host;
  if (*reinterpret_cast<int*>(p->energy_host + 1) != 0)
  {
    DPC_CUDA(cudaMemsetAsync(p->status(), 0, sizeof(int), p->ctx->stream));
    return fail(DPC_ERR_TIMEOUT, "a tensor-core kernel gave up waiting on a pipeline barrier");
  }
  return DPC_OK;
}
