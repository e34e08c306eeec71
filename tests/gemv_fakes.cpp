// Host-only program around bk_gemv.cu: the CUDA runtime and the other kernels' launchers are fakes that record which of them a call goes to.  Reads lines
// "K rows columns" and prints for each the launches of 8 columns, and "dense" where the lane order takes the dense tile kernel.
#include <stdarg.h>
#include <stdio.h>

#include "../bunker_b200/csrc/bk_internal.h"

static BkContext g_ctx_fake;
static int g_groups, g_dense;
BkContext& bk_ctx() { return g_ctx_fake; }
int32_t bk_fail(int32_t code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vfprintf(stderr, fmt, ap);
  va_end(ap);
  return code;
}
bool bk_gemv_mma_fits(int K, int) { return K < 8192; }
int32_t bk_gemv_mma_launch(void*, int, int, int, bool, int*) { return g_groups++, BK_OK; }
int32_t bk_gemv_umma_launch(void*, int, bool lanes) { return g_dense += lanes, BK_OK; }

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return g_groups++, cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t*, const void*, void**) { return g_groups++, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { return *a = cudaFuncAttributes(), cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t) { return *p = (void*)(1 << 20), cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
}

int main() {
  g_ctx_fake.ready = true;
  g_ctx_fake.sm_count = 148;
  g_ctx_fake.smem_optin = 232448;
  int K, rows, B;
  while (scanf("%d %d %d", &K, &rows, &B) == 3) {
    bkGemvArgs a = {};
    a.K = K; a.B = B; a.n_segs = 1; a.prologue = BK_PRO_Q8; a.x = 1 << 20; a.order = BK_GEMV_ORDER_LANES;
    a.segs[0].W = a.segs[0].out = 1 << 20;
    a.segs[0].n_rows = a.segs[0].ld_out = rows;
    a.segs[0].epilogue = BK_EPI_F32;
    g_groups = g_dense = 0;
    if (bkGemvQ4K(&a) != BK_OK) return 1;
    if (g_dense) printf("dense\n");
    else printf("%d\n", g_groups);
  }
  return 0;
}
