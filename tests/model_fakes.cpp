// Host-only program around bk_model.cu: the CUDA runtime and the library's other translation units are fakes that record what the
// model asks for.  Usage: model_fakes STEP_MODE PLAN_RC [MAX_LEN STEPS]  -- the result of finishing the step plan, and a longer cache with
// steps taken one by one; prints "key value" lines.
#include <stdarg.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>

#include "../bunker_b200/csrc/bk_internal.h"

static BkContext g_ctx_fake;
static int g_plan_rc, g_plans, g_plan_launches, g_gemvs, g_graphs, g_graph_launches;
static int g_plan_graphs, g_plan_steps, g_captured_from;   // a graph that holds a plan launch, launches of one
static std::map<cudaGraphExec_t, bool> g_is_plan;
static uint64_t g_next = 1 << 20;
static char g_err[256];

BkContext& bk_ctx() { return g_ctx_fake; }
int32_t bk_fail(int32_t code, const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_err, sizeof(g_err), fmt, ap);
  va_end(ap);
  return code;
}

// ---- the rest of the library ----
int32_t bk_comm_info(uint64_t, int*, int*) { return BK_ERR_COMM; }
int32_t bk_comm_push_desc(uint64_t, int, BkPush*) { return BK_ERR_COMM; }
int32_t bk_comm_reduce_desc(uint64_t, int, BkReduce*) { return BK_ERR_COMM; }
int32_t bk_comm_argmax_merge(uint64_t, int, int, uint64_t, uint64_t, int, uint64_t, uint64_t, uint64_t, uint64_t, int, int) { return BK_ERR_COMM; }
int32_t bk_gdn_launch(const bkGdnArgs&) { return BK_OK; }
int32_t bk_attn_launch(const bkAttnArgs&, int, int) { return BK_OK; }
int32_t bk_gemv_launch(const bkGemvArgs&) { return g_gemvs++, BK_OK; }
int32_t bk_gemv_launch_tp(const bkGemvArgs&, const BkPush*, const BkReduce*, int*) { return g_gemvs++, BK_OK; }
int32_t bk_argmax_launch(uint64_t, int32_t, int32_t, uint64_t, uint64_t, uint64_t, uint64_t, uint64_t, int32_t, int32_t, uint64_t) { return BK_OK; }
int32_t bk_quant_rows_launch(uint64_t, uint64_t, int32_t, int32_t, float, uint64_t, int32_t, const BkReduce*) { return BK_OK; }
bool bk_gemv_mma_fits(int, int) { return true; }
bool bk_tile_split(int, int, int, bool) { return false; }
bool bk_gemv_dense_lanes(int, int, int) { return false; }
bool bk_gemv_auto_tile(int, int) { return false; }
int32_t bk_plan_create(uint64_t* out, const BkPlanDims&) { return g_plans++, *out = 77, BK_OK; }
void bk_plan_add_layer(uint64_t, const BkPlanLayer&) {}
int32_t bk_plan_finish(uint64_t, uint64_t, uint64_t, uint64_t, int) { return g_plan_rc; }
int32_t bk_plan_launch(uint64_t, int, const BkStepIO&) { return g_plan_launches++, BK_OK; }
int32_t bk_plan_reset(uint64_t) { return BK_OK; }
void bk_plan_destroy(uint64_t) { g_plans--; }
extern "C" {
uint64_t bkArgmaxScratchBytes(int32_t) { return 64; }
uint64_t bkAttnScratchBytes(int32_t, int32_t, int32_t, int32_t, int32_t) { return 64; }
int32_t bkAttnPlan(int32_t, int32_t, int32_t, int32_t* split_len, int32_t*) { return *split_len = 64, BK_OK; }
int32_t bkEmbedQ4K(uint64_t, int32_t, uint64_t, int32_t, uint64_t) { return BK_OK; }
int32_t bkRopeTables(int32_t, int32_t, double, float*, float*) { return BK_OK; }

// ---- the CUDA runtime ----
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { *p = (void*)g_next; g_next += (n + 255) / 256 * 256; return cudaSuccess; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(1, n); return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) { *d = h; return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return g_captured_from = g_plan_launches, cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)1; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
  *e = (cudaGraphExec_t)(uintptr_t)(++g_graphs);
  g_plan_graphs += g_is_plan[*e] = g_plan_launches > g_captured_from;
  return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t) { return g_graph_launches++, g_plan_steps += g_is_plan[e], cudaSuccess; }
}

int main(int argc, char** argv) {
  if (argc < 3) return 2;
  g_ctx_fake.ready = true;
  g_ctx_fake.sm_count = 148;
  g_plan_rc = atoi(argv[2]);
  bkModelConfig c;
  memset(&c, 0, sizeof(c));
  c.hidden = 256; c.n_layers = 2; c.full_attn_interval = 2; c.vocab = 300; c.gdn_k_heads = 1; c.gdn_v_heads = 2; c.attn_q_heads = 2; c.attn_kv_heads = 1;
  c.head_dim = 256; c.rot_dim = 64; c.intermediate = 512; c.max_len = argc > 3 ? atoi(argv[3]) : 64; c.batch = 1; c.tp_size = 1; c.eps = 1e-6f; c.rope_theta = 1e7;
  uint64_t m = 0;
  if (bkModelCreate(&c, &m) != BK_OK) return 3;
  auto q4k = [](uint64_t n, uint64_t k) { return n * (k / 256) * 144; };
  std::map<std::string, uint64_t> t = {{"embed.weight", q4k(300, 256)}, {"final.norm.weight", 512}};
  for (int l = 0; l < 2; l++) {
    const std::string p = "model.layers." + std::to_string(l) + ".";
    t[p + "input_layernorm.weight"] = t[p + "post_attention_layernorm.weight"] = 512;
    t[p + "mlp.gate_proj.weight"] = t[p + "mlp.up_proj.weight"] = q4k(512, 256);
    t[p + "mlp.down_proj.weight"] = q4k(256, 512);
  }
  const std::string g = "model.layers.0.linear_attn.", a = "model.layers.1.self_attn.";
  t[g + "in_proj_qkv.weight"] = q4k(512, 256); t[g + "in_proj_z.weight"] = q4k(256, 256); t[g + "in_proj_a.weight"] = t[g + "in_proj_b.weight"] = q4k(2, 256);
  t[g + "conv1d.weight"] = 512 * 8; t[g + "A_log"] = 8; t[g + "dt_bias"] = 4; t[g + "norm.weight"] = 512; t[g + "out_proj.weight"] = q4k(256, 256);
  t[a + "q_proj.weight"] = q4k(1024, 256); t[a + "k_proj.weight"] = t[a + "v_proj.weight"] = q4k(256, 256); t[a + "q_norm.weight"] = t[a + "k_norm.weight"] = 512;
  t[a + "o_proj.weight"] = q4k(256, 512);
  for (auto& kv : t)
    if (bkModelSetTensor(m, kv.first.c_str(), g_next += 1 << 20, kv.second) != BK_OK) return 4;
  if (bkModelSetStepMode(m, atoi(argv[1])) != BK_OK) return 5;
  const int rc = bkModelFinalize(m);
  printf("finalize %d\nplans %d\n", rc, g_plans);
  if (rc != BK_OK) return printf("error %s\n", g_err), 0;
  g_plan_launches = g_gemvs = 0;
  int32_t tok = 5, id = 0;
  const int step = bkDecodeStep(m, &tok, &id, nullptr), eager = bkDecodeStepEager(m);
  printf("step %d\neager %d\ngraphs %d\ngraph_launches %d\nplan_launches %d\ngemvs %d\n", step, eager, g_graphs, g_graph_launches, g_plan_launches, g_gemvs);
  if (argc > 4) {
    bkModelReset(m);
    g_graph_launches = g_plan_steps = g_plan_launches = 0;
    int first_chain = -1, back = 0;   // the first position off the plan; positions that went back to it
    for (int i = 0; i < atoi(argv[4]); i++) {
      const int before = g_plan_steps + g_plan_launches;
      if ((i & 1 ? bkDecodeStep(m, &tok, nullptr, nullptr) : bkDecodeRun(m, 1)) != BK_OK) return 6;
      const bool plan = g_plan_steps + g_plan_launches > before;
      if (!plan && first_chain < 0) first_chain = i;
      back += plan && first_chain >= 0;
    }
    int32_t kernels = 0;
    bkModelInfo(m, nullptr, nullptr, &kernels, nullptr);
    printf("plan_graphs %d\nfirst_chain %d\nback %d\n", g_plan_graphs, first_chain, back);
  }
  bkModelDestroy(m);
  printf("plans_left %d\n", g_plans);
  return 0;
}
