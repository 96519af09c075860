// Shared by dpc_conv.cu (phase kernels, C ABI) and dpc_conv_resident.cu (image-resident segments).
#pragma once
#include <vector>

#include "dpc_internal.h"

struct dpc_conv_plan
{
  dpc_ctx* ctx = nullptr;
  int n = 0, batch = 0;
  std::vector<dpc_conv_layer> h;
  dpc_conv_layer* d = nullptr; // device copy of the table
  double* energy = nullptr;
  double* energy_host = nullptr;
  float* scratch = nullptr; // sums of split state updates, one buffer per layer
  size_t scratch_floats = 0;
  void* res = nullptr; // image-resident path state, owned by dpc_conv_resident.cu
};

namespace dpc
{
// DPC_OK: the plan has image-resident segments, 1: it does not (negative: a CUDA call failed).
int conv_res_init(dpc_conv_plan* plan);
void conv_res_free(dpc_conv_plan* plan);
} // namespace dpc
