// Flat C functions over the plugin's device primitives (b200_backend.h), for tests that call its kernels without the
// reference's host: host buffers in, host buffers out.
#include <initializer_list>

#include "b200_backend.h"

extern "C" __attribute__((visibility("default"))) int plugin_matmul(
    int trans_a, int trans_b, int M, int N, int K, float alpha, const float* a, size_t na, int lda, const float* b,
    size_t nb, int ldb, float beta, float* c, size_t nc, int ldc, int allow_tf32, int calls)
{
  b200::Ctx* ctx = b200::create();
  if (!ctx)
    return 1;
  float* A = b200::allocate(ctx, na);
  float* B = b200::allocate(ctx, nb);
  float* C = b200::allocate(ctx, nc);
  const bool ok = A && B && C;
  if (ok)
  {
    if (allow_tf32 >= 0)
      b200::set_allow_tf32(ctx, allow_tf32 != 0);
    b200::copy_from_host(ctx, A, a, na);
    b200::copy_from_host(ctx, B, b, nb);
    b200::copy_from_host(ctx, C, c, nc);
    for (int i = 0; i < calls; ++i)
      b200::sgemm(ctx, trans_a != 0, trans_b != 0, M, N, K, alpha, A, lda, B, ldb, beta, C, ldc);
    b200::copy_to_host(ctx, c, C, nc);
  }
  for (float* p : {A, B, C})
    b200::release(ctx, p);
  b200::destroy(ctx);
  return ok ? 0 : 2;
}
