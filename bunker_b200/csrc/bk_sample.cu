// bk_sample.cu -- temperature / top-k / top-p sampling over f32 logits, deterministic and reproducible on a host.
//
// bunker only has the greedy tail (buildArgmax + buildArgmaxComb, prototypes/decode.ts:749-791); this is the sampling
// step that stands beside it.  Per sequence:
//   1. the top_k (<= 64) largest logits, ties to the lower index, in descending order (exact selection);
//   2. p_i = exp((l_i - l_0) / T) with the library's own exp, summed in that order;
//   3. nucleus: the shortest prefix whose running sum reaches top_p * total;
//   4. u in [0,1) from a counter-based hash of (seed, step, sequence); the first i whose running sum exceeds u * prefix
//      total is the token.
//
// Selection.  Every candidate is a 64-bit key, unique and totally ordered: the logit's bits made monotonic above the
// complement of its index.  A cluster of one to eight CTAs per sequence runs a radix selection over 11-bit digits from the top:
// histogram of the digit among the keys that share the prefix chosen so far (shared memory per CTA, added up over
// distributed shared memory), then the digit in which the top_k-th key lies.  As soon as the keys at or above that
// prefix fit the candidate list, they are collected, and each finds its rank by counting the larger ones.  Ordinary logits
// need one digit (two reads of the row, the second from L2); equal or clustered logits take further digits, at most six.
// What bounds it: two passes over V floats by the cluster's SMs plus four cluster barriers.  Measured at V = 151936,
// top_k = 40, one sequence: 774 us with top_k rounds of a full scan by one CTA, 15.6 us like this.  One pick or two are rounds of a
// full scan all the same (sample_rounds_kernel; bkSample has the rule).
#include <math.h>

#include "bk_common.cuh"
#include "bk_internal.h"

namespace {

constexpr int kSampleMaxK = 64;

BK_DEVINL unsigned long long splitmix64(unsigned long long x) {
  x += 0x9E3779B97F4A7C15ull;
  x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
  x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
  return x ^ (x >> 31);
}

constexpr int kSampleThreads = 1024;
constexpr int kDigitBits = 11, kBins = 1 << kDigitBits;
constexpr int kListMax = 2048;       // candidates collected before the ranking

// larger key = earlier candidate; 0 is no candidate (a NaN).  -0 compares equal to +0, so it takes +0's key.
BK_DEVINL unsigned long long cand_key(float v, int i) {
  if (v != v) return 0ull;
  uint32_t u = __float_as_uint(v == 0.0f ? 0.0f : v);
  u = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
  return ((unsigned long long)u << 32) | (uint32_t)~i;
}
template <int CTAS>
BK_DEVINL void cluster_sync() {
  if (CTAS == 1) {
    __syncthreads();
    return;
  }
  asm volatile("barrier.cluster.arrive;" ::: "memory");
  asm volatile("barrier.cluster.wait;" ::: "memory");
}
// the same shared-memory object in CTA `rank` of the cluster
template <typename T>
BK_DEVINL uint32_t cluster_addr(const T* p, int rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_u32(p)), "r"(rank));
  return r;
}
BK_DEVINL uint32_t ld_cluster_u32(uint32_t a) {
  uint32_t v;
  asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
BK_DEVINL unsigned long long ld_cluster_u64(uint32_t a) {
  unsigned long long v;
  asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
  return v;
}

struct SampleParams {
  const float* logits;
  int V;
  float temperature;
  int top_k;
  float top_p;
  unsigned long long seed;
  const int32_t* step_dev;
  unsigned int step_add;
  int32_t* idx_out;
  float* val_out;
};

// The top_k largest logits of sequence b lie in cv / ci; pr: room for their weights.  By all threads of a CTA.
BK_DEVINL void pick_token(const SampleParams& p, int b, int top_k, const float* cv, const int* ci, float* pr) {
  const int tid = threadIdx.x;
  __syncthreads();
  if (p.temperature > 0.0f && tid < top_k) pr[tid] = bk_expf(__fmul_rn(__fsub_rn(cv[tid], cv[0]), __fdiv_rn(1.0f, p.temperature)));
  __syncthreads();
  if (tid == 0) {
    int pick = 0;
    if (top_k <= 0) {
      p.idx_out[b] = 0;
      if (p.val_out) p.val_out[b] = -INFINITY;
      return;
    }
    if (p.temperature > 0.0f && top_k > 1) {
      float total = 0.0f;
      for (int i = 0; i < top_k; i++) total = __fadd_rn(total, pr[i]);
      const float need = __fmul_rn(p.top_p, total);
      int m = top_k;
      float run = 0.0f;
      for (int i = 0; i < top_k; i++) {
        run = __fadd_rn(run, pr[i]);
        if (run >= need) {
          m = i + 1;
          break;
        }
      }
      float prefix_sum = 0.0f;
      for (int i = 0; i < m; i++) prefix_sum = __fadd_rn(prefix_sum, pr[i]);
      const unsigned int step = (p.step_dev ? (unsigned int)p.step_dev[b] : 0u) + p.step_add;
      const unsigned long long h = splitmix64(splitmix64(p.seed ^ ((unsigned long long)step << 20)) + (unsigned long long)b);
      const float u = __fmul_rn((float)(unsigned int)(h >> 40), 5.9604644775390625e-8f);   // 24 bits -> [0,1)
      const float target = __fmul_rn(u, prefix_sum);
      pick = m - 1;
      run = 0.0f;
      for (int i = 0; i < m; i++) {
        run = __fadd_rn(run, pr[i]);
        if (run > target) {
          pick = i;
          break;
        }
      }
    }
    p.idx_out[b] = ci[pick];
    if (p.val_out) p.val_out[b] = cv[pick];
  }
}

// One pick or two: one CTA per sequence, round r finds the candidate that follows round r-1's (larger logit first, then lower index).
// A round is one pass over the row in two comparisons a logit.
BK_DEVINL bool before(float v, int i, float w, int j) { return v > w || (v == w && i < j); }
BK_DEVINL void warp_first(float& v, int& i) {
  for (int off = 16; off >= 1; off >>= 1) {
    const float ov = __shfl_xor_sync(0xffffffffu, v, off);
    const int oi = __shfl_xor_sync(0xffffffffu, i, off);
    if (before(ov, oi, v, i)) {
      v = ov;
      i = oi;
    }
  }
}
__global__ void __launch_bounds__(kSampleThreads) sample_rounds_kernel(const __grid_constant__ SampleParams p) {
  __shared__ float sv[32], cv[kSampleMaxK], pr[kSampleMaxK];
  __shared__ int si[32], ci[kSampleMaxK];
  bk_pdl_trigger();
  const int b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, V = p.V;
  const float* l = p.logits + (size_t)b * V;
  bk_pdl_wait();
  float last_v = INFINITY;
  int last_i = -1, top_k = p.top_k;
  for (int r = 0; r < top_k; r++) {
    float v = -INFINITY;
    int at = 0x7fffffff;
    for (int i = tid; i < V; i += kSampleThreads) {
      const float x = __ldcg(l + i);   // (a NaN is before nothing)
      if (before(x, i, v, at) && before(last_v, last_i, x, i)) {
        v = x;
        at = i;
      }
    }
    warp_first(v, at);
    if (lane == 0) {
      sv[warp] = v;
      si[warp] = at;
    }
    __syncthreads();
    v = sv[lane];
    at = si[lane];
    warp_first(v, at);
    __syncthreads();
    if (at == 0x7fffffff) {   // fewer than top_k logits that are not NaN
      top_k = r;
      break;
    }
    if (tid == 0) {
      cv[r] = v;
      ci[r] = at;
    }
    last_v = v;
    last_i = at;
  }
  pick_token(p, b, top_k, cv, ci, pr);
}

template <int CTAS>
__global__ void __cluster_dims__(CTAS, 1, 1) __launch_bounds__(kSampleThreads) sample_kernel(const __grid_constant__ SampleParams p) {
  __shared__ unsigned int hist[kBins];
  __shared__ unsigned long long list[kListMax];
  __shared__ unsigned int n_list;
  __shared__ unsigned int wsum[32];
  __shared__ unsigned long long s_prefix;   // digits chosen so far (decided by CTA 0, read by the others)
  __shared__ unsigned int s_need, s_count;  // keys still wanted inside the prefix; keys at or above the chosen digit
  __shared__ float cv[kSampleMaxK], pr[kSampleMaxK];
  __shared__ int ci[kSampleMaxK];
  bk_pdl_trigger();
  const int rank = blockIdx.x % CTAS, b = blockIdx.x / CTAS, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, V = p.V;
  int top_k = p.top_k;
  const float* l = p.logits + (size_t)b * V;
  const int per = ((V + CTAS - 1) / CTAS + 3) & ~3;
  const int lo = min(V, rank * per), hi = min(V, lo + per);
  if (tid == 0) {
    n_list = 0;
    s_prefix = 0;
    s_need = top_k;
  }
  bk_pdl_wait();
  // the keys this thread looks at, in any order; four consecutive logits per load where the row allows it
  const bool vec = ((reinterpret_cast<uintptr_t>(l) & 15) == 0) && (V & 3) == 0;
  auto for_each = [&](auto&& f) {
    if (vec) {
      for (int i = lo + 4 * tid; i < hi; i += 4 * kSampleThreads) {
        const float4 v = __ldcg(reinterpret_cast<const float4*>(l + i));
        f(cand_key(v.x, i));
        f(cand_key(v.y, i + 1));
        f(cand_key(v.z, i + 2));
        f(cand_key(v.w, i + 3));
      }
    } else {
      for (int i = lo + tid; i < hi; i += kSampleThreads) f(cand_key(__ldcg(l + i), i));
    }
  };
  unsigned long long prefix = 0;
  int shift = 64;              // bits below the prefix
  unsigned long long cut = 1;  // collect the keys >= cut
  while (true) {
    const int bits = min(kDigitBits, shift), next = shift - bits;
    for (int i = tid; i < kBins; i += kSampleThreads) hist[i] = 0;
    __syncthreads();
    for_each([&](unsigned long long key) {
      if (key != 0 && (shift == 64 || (key >> shift) == prefix)) atomicAdd(&hist[(unsigned int)(key >> next) & ((1u << bits) - 1u)], 1u);
    });
    cluster_sync<CTAS>();
    if (rank == 0) {
      // thread t owns bins kBins-1-2t and kBins-2-2t (largest first); running count from the top
      unsigned int c0 = 0, c1 = 0;
      const int b0 = kBins - 1 - 2 * tid, b1 = b0 - 1;
      for (int r = 0; r < CTAS; r++) {
        c0 += ld_cluster_u32(cluster_addr(&hist[b0], r));
        c1 += ld_cluster_u32(cluster_addr(&hist[b1], r));
      }
      unsigned int run = c0 + c1;
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned int o = __shfl_up_sync(0xffffffffu, run, off);
        if (lane >= off) run += o;
      }
      if (lane == 31) wsum[warp] = run;
      __syncthreads();
      unsigned int base = 0;
      for (int w = 0; w < warp; w++) base += wsum[w];
      const unsigned int before = base + run - c0 - c1, need = s_need;
      unsigned int total = 0;
      for (int w = 0; w < 32; w++) total += wsum[w];
      __syncthreads();
      // the bin in which the need-th key lies, or bin 0 when there are fewer keys than that
      const bool here = before < need && before + c0 + c1 >= need, short_ = total < need && tid == kSampleThreads - 1;
      if (here || short_) {
        const bool first = here && before + c0 >= need;
        s_prefix = (s_prefix << bits) | (unsigned long long)(short_ ? 0 : first ? b0 : b1);
        s_count = short_ ? total : before + c0 + (first ? 0u : c1);
        s_need = short_ ? need : need - (first ? before : before + c0);
      }
    }
    cluster_sync<CTAS>();
    const int decided = 0;
    prefix = ld_cluster_u64(cluster_addr(&s_prefix, decided));
    // keys above this prefix are fewer than top_k, so the list holds what it says if the chosen digit's bin is small
    const unsigned int count = ld_cluster_u32(cluster_addr(&s_count, decided));
    shift = next;
    if (count <= (unsigned int)(kListMax - kSampleMaxK) || shift == 0) {
      cut = shift == 64 ? 1ull : (prefix << shift);
      if (cut == 0) cut = 1;
      break;
    }
  }
  // collect into CTA 0's list
  const uint32_t n_addr = cluster_addr(&n_list, 0), list_addr = cluster_addr(list, 0);
  for_each([&](unsigned long long key) {
    if (key >= cut) {
      unsigned int at;
      asm volatile("atom.shared::cluster.add.u32 %0, [%1], 1;" : "=r"(at) : "r"(n_addr) : "memory");
      if (at < (unsigned int)kListMax) asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(list_addr + 8 * at), "l"(key) : "memory");
    }
  });
  cluster_sync<CTAS>();
  if (rank != 0) return;
  const int n = min((int)n_list, kListMax);
  for (int i = tid; i < n; i += kSampleThreads) {
    const unsigned long long key = list[i];
    int r = 0;
    for (int j = 0; j < n; j++) r += list[j] > key;
    if (r < top_k) {
      ci[r] = (int)~(uint32_t)key;
      cv[r] = l[(int)~(uint32_t)key];
    }
  }
  if (n < top_k) top_k = n;   // fewer than top_k logits that are not NaN
  pick_token(p, b, top_k, cv, ci, pr);
}

}  // namespace

extern "C" int32_t bkSample(uint64_t logits, int32_t V, int32_t B, float temperature, int32_t top_k, float top_p, uint64_t seed,
                            uint64_t step_dev, uint32_t step_add, uint64_t idx, uint64_t val) {
  BK_REQUIRE_INIT();
  BK_ARG(logits && idx && V > 0 && B > 0, "bkSample: bad arguments");
  BK_ARG(top_k >= 1 && top_k <= kSampleMaxK, "bkSample: top_k=%d outside 1..%d", top_k, kSampleMaxK);
  BK_ARG(temperature >= 0.0f && top_p > 0.0f && top_p <= 1.0f, "bkSample: temperature=%g top_p=%g", (double)temperature, (double)top_p);
  SampleParams p = {bk_ptr<float>(logits), V, temperature, top_k, top_p, (unsigned long long)seed, bk_ptr<int32_t>(step_dev), step_add, bk_ptr<int32_t>(idx), bk_ptr<float>(val)};
  // CTAs per sequence: a short row is one CTA's (V 4,096, one sequence: 5 us with one, 7 with eight); a longer one takes as many as still
  // leave each CTA an SM of its own -- beyond that the clusters wait for one another (V 32,000, top_k 40, 64 sequences: 22 us with one, 15
  // with two, 23 with four, 39 with eight) -- and eight only where rows are long and sequences few (64,000, one sequence: 12.5 us, with four
  // 13.6; 151,936: 15.6 and 20.4).
  const int sms = bk_ctx().sm_count;
  const int ctas = V <= 8192 ? 1 : V > 40000 && B <= 8 ? 8 : B <= sms / 4 ? 4 : B <= sms / 2 ? 2 : 1;
  // Rounds of a full pass where the two passes of the selection, or its barriers, cost more: top_k 1 of 64 sequences, V 151,936: 23 us against
  // 29; of one, V 16,000: 5 against 7 (V 64,000: 11 against 9); top_k 2 of 200, V 151,936: 86 against 90 (top_k 3: 124 against 90).
  const bool rounds = top_k * ctas <= 2 || (top_k == 1 && V <= 32768);
  if (rounds) BK_CUDA(bk_launch_pdl(sample_rounds_kernel, dim3(B), dim3(kSampleThreads), 0, p));
  else if (ctas == 1) BK_CUDA(bk_launch_pdl(sample_kernel<1>, dim3(B), dim3(kSampleThreads), 0, p));
  else if (ctas == 2) BK_CUDA(bk_launch_pdl(sample_kernel<2>, dim3(2u * B), dim3(kSampleThreads), 0, p));
  else if (ctas == 4) BK_CUDA(bk_launch_pdl(sample_kernel<4>, dim3(4u * B), dim3(kSampleThreads), 0, p));
  else BK_CUDA(bk_launch_pdl(sample_kernel<8>, dim3(8u * B), dim3(kSampleThreads), 0, p));
  BK_CHECK_LAUNCH();
  return BK_OK;
}
