// bk_attn.cu -- split-KV flash-decode GQA attention over a bf16 KV cache.
//
// Replaces bunker's single-tile decode attention (emitFA2Attn, src/emitters.ts:188-226;
// buildFA2Attn, prototypes/decode.ts:427-468), whose cache is capped at 128 rows and
// replicated per query head.  Here the cache is per KV head, [B][Hkv][max_len][256],
// and a (batch, KV head) pair is cut into splits of split_len rows, one CTA each, so
// every SM streams K/V.  The same kernel applies the q/k head RMSNorm and the partial
// rotary (emitQNorm/emitKNorm/emitRoPE/emitRoPEK, src/emitters.ts:123-183) and appends
// the new K/V row, so one launch replaces five of the reference's.
//
// Per split: scores for all rows (each K row is read once for the G query heads of
// the group), exact max, p = exp(s-m), then o = sum p*V with each V row read once.
// The CTA that finishes a (batch, KV head) last merges its splits and applies the sigmoid output gate.
// Orders are fixed (see the CPU oracle): lane l owns dims [8l,8l+8); row jj of a
// split belongs to warp jj mod 8; warps and splits are added in ascending order.
#include "bk_common.cuh"
#include "bk_internal.h"

#include <algorithm>

namespace {

constexpr int kW = 8;        // warps per split CTA
constexpr int kHD = 256;     // head dim (8 per lane)
constexpr int kMaxSplits = 1024;

struct AttnParams {
  const uint16_t* qg;
  const uint16_t* k;
  const uint16_t* v;
  const uint16_t* q_norm_w;
  const uint16_t* k_norm_w;
  const float* cos_t;
  const float* sin_t;
  uint16_t* k_cache;
  uint16_t* v_cache;
  const int32_t* pos;
  uint16_t* out;
  uint8_t* out_q8;
  int out_q8_layout;
  float *part_ml, *part_o;   // partials of all entries: (m, l) pairs, and 256 sums 16-byte aligned
  unsigned int* counters;    // splits done per (entry, KV head); they reset themselves
  const uint16_t* gate;
  int B, Hq, Hkv, rot_half, max_len, split_len, max_splits, fused;
  int splits_first;   // the grid is (split, KV head, entry), not (KV head, entry, split)
  int settled;  // cache rows of earlier steps and pos[] are not outputs of the immediately preceding launch
  int n_seq;    // > 0: prompt columns.  Entry b of the launch is token b / n_seq of sequence b mod n_seq: it reads that
                // sequence's cache, and its own K/V row has already been appended (attn_append_kernel)
  float scale;
  unsigned long long* trace;
};

__device__ __forceinline__ void bf16x8_to_f32(uint4 v, float (&y)[8]) {
  y[0] = __uint_as_float(v.x << 16);
  y[1] = __uint_as_float(v.x & 0xffff0000u);
  y[2] = __uint_as_float(v.y << 16);
  y[3] = __uint_as_float(v.y & 0xffff0000u);
  y[4] = __uint_as_float(v.z << 16);
  y[5] = __uint_as_float(v.z & 0xffff0000u);
  y[6] = __uint_as_float(v.w << 16);
  y[7] = __uint_as_float(v.w & 0xffff0000u);
}

// head RMSNorm*(1+w) -> bf16 -> rotary on the first 2*rot_half dims, result in `stage`.  x and w: the row and the norm weights, 8 dims a lane;
// c and s: the lane's of the first 32 angles, which the caller has requested.
__device__ __forceinline__ float first_angles(const float* row, int rot_half) { return (threadIdx.x & 31) < rot_half ? row[threadIdx.x & 31] : 0.0f; }
__device__ __forceinline__ void norm_rope_256(uint4 xr, uint4 wr, float c, float s, const float* cos_row, const float* sin_row, int rot_half, uint16_t* stage) {
  const int lane = threadIdx.x & 31;
  float x[8], wv[8];
  bf16x8_to_f32(xr, x);
  bf16x8_to_f32(wr, wv);
  float acc = 0.0f;
#pragma unroll
  for (int e = 0; e < 8; e++) acc = fmaf(x[e], x[e], acc);
  acc = bk_warp_sum(acc);
  float rstd = bk_rcp_sqrt(__fadd_rn(__fdiv_rn(acc, (float)kHD), 1e-6f));
#pragma unroll
  for (int e = 0; e < 8; e++)
    stage[lane * 8 + e] = bk_f32_to_bf16(__fmul_rn(__fmul_rn(x[e], rstd), __fadd_rn(1.0f, wv[e])));
  __syncwarp();
  for (int i = lane; i < rot_half; i += 32) {
    if (i >= 32) {
      c = cos_row[i];
      s = sin_row[i];
    }
    float x1 = bk_bf16_to_f32(stage[i]), x2 = bk_bf16_to_f32(stage[i + rot_half]);
    uint16_t r1 = bk_f32_to_bf16(__fsub_rn(__fmul_rn(x1, c), __fmul_rn(x2, s)));
    uint16_t r2 = bk_f32_to_bf16(__fadd_rn(__fmul_rn(x2, c), __fmul_rn(x1, s)));
    stage[i] = r1;
    stage[i + rot_half] = r2;
  }
  __syncwarp();
}

// One level of a warp's xor butterfly over N values at once: a lane keeps half of its values and sends the other half to its partner
// `off` lanes away.  SWAPPED: the lanes with that bit set hold the two halves exchanged, so there is nothing to select; otherwise
// they do not.  The additions are the butterfly's, so the bits are too.
template <int N, bool SWAPPED>
__device__ __forceinline__ void butterfly_level(float (&v)[N], int off) {
  const bool upper = threadIdx.x & off;
#pragma unroll
  for (int i = 0; i < N / 2; i++) {
    const float send = !SWAPPED && upper ? v[i] : v[i + N / 2], keep = !SWAPPED && upper ? v[i + N / 2] : v[i];
    v[i] = __fadd_rn(keep, __shfl_xor_sync(0xffffffffu, send, off));
  }
}

// the sigmoid gate of a head, 8 dims a lane
__device__ __forceinline__ uint4 head_gate(const AttnParams& p, int b, int h) {
  const int lane = threadIdx.x & 31;
  return *reinterpret_cast<const uint4*>(p.fused ? p.qg + ((size_t)b * p.Hq + h) * 2 * kHD + kHD + lane * 8 : p.gate + ((size_t)b * p.Hq + h) * kHD + lane * 8);
}
// out = (O/L) * sigmoid(gate) of this lane's dims
__device__ void store_head_warp(const AttnParams& p, int b, int h, const float (&O)[8], float L, uint4 gate) {
  const int lane = threadIdx.x & 31;
  float gf[8];
  bf16x8_to_f32(gate, gf);
  uint32_t o[4];
#pragma unroll
  for (int e = 0; e < 8; e += 2) {
    float v0 = __fmul_rn(__fdiv_rn(O[e], L), bk_sigmoidf(gf[e]));
    float v1 = __fmul_rn(__fdiv_rn(O[e + 1], L), bk_sigmoidf(gf[e + 1]));
    o[e >> 1] = bk_f32x2_to_bf16x2(v0, v1);
  }
  *reinterpret_cast<uint4*>(p.out + ((size_t)b * p.Hq + h) * kHD + lane * 8) = make_uint4(o[0], o[1], o[2], o[3]);
  if (p.out_q8) {  // four lanes hold one 32-value block
    float y[8];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      y[2 * e] = __uint_as_float(o[e] << 16);
      y[2 * e + 1] = __uint_as_float(o[e] & 0xffff0000u);
    }
    if (p.out_q8_layout >= BK_Q8_TILE) bk_tile_store<8>(p.out_q8, p.Hq * kHD, p.B, b, (h * kHD + lane * 8) >> 5, y, (lane & 3) * 8, p.out_q8_layout == BK_Q8_TILE32);
    else if (p.out_q8_layout == BK_Q8_STAGED) bk_staged_store<8>(p.out_q8, p.Hq * kHD, p.B, b, (h * kHD + lane * 8) >> 5, y, (lane & 3) * 8);
    else bk_q8_1_store<8>(p.out_q8 + ((((size_t)b * p.Hq + h) * kHD + lane * 8) >> 5) * 36, y, (lane & 3) * 8);
  }
}

// Merge the splits of one (batch, q head) by one warp; lane l owns output dims [8l, 8l+8).  w_s: ns floats of shared memory private to the warp.  M = max m_s; w_s =
// exp(m_s - M); L = fma(w_s, l_s, L) and O = fma(w_s, o_s, O) in ascending s; out = (O/L) * sigmoid(gate).  As little code as there can be (see launch_split).
__device__ void combine_head_warp(const AttnParams& p, int b, int h, int ns, float* w_s, uint4 gate) {
  const int lane = threadIdx.x & 31;
  const float* sc_ml = p.part_ml + ((size_t)b * p.Hq + h) * p.max_splits * 2;
  const float* sc_o = p.part_o + ((size_t)b * p.Hq + h) * p.max_splits * kHD;
  float m = -INFINITY;
  for (int s = lane; s < ns; s += 32) {
    float ms = __ldcg(sc_ml + 2 * s);
    w_s[s] = ms;
    m = fmaxf(m, ms);
  }
  const float M = bk_warp_max(m);
  for (int s = lane; s < ns; s += 32) w_s[s] = bk_expf(__fsub_rn(w_s[s], M));
  __syncwarp();
  float L = 0.0f, O[8];
#pragma unroll
  for (int e = 0; e < 8; e++) O[e] = 0.0f;
#pragma unroll 4
  for (int s = 0; s < ns; s++) {
    const float w = w_s[s];
    L = fmaf(w, __ldcg(sc_ml + 2 * s + 1), L);
    const float4 a = __ldcg(reinterpret_cast<const float4*>(sc_o + (size_t)s * kHD + lane * 8));
    const float4 c = __ldcg(reinterpret_cast<const float4*>(sc_o + (size_t)s * kHD + lane * 8) + 1);
    O[0] = fmaf(w, a.x, O[0]); O[1] = fmaf(w, a.y, O[1]); O[2] = fmaf(w, a.z, O[2]); O[3] = fmaf(w, a.w, O[3]);
    O[4] = fmaf(w, c.x, O[4]); O[5] = fmaf(w, c.y, O[5]); O[6] = fmaf(w, c.z, O[6]); O[7] = fmaf(w, c.w, O[7]);
  }
  store_head_warp(p, b, h, O, L, gate);
}

// The same for many splits, all threads of a CTA for the heads of one (batch, KV head).  wl: G * ns pairs of shared memory; where a head has more than one warp they then take its sums.
// Bound: latency of L2, with one CTA at work.  The heads' dims are spread over all eight warps, so that 64 values a thread (32 where 80 registers
// are all there are) are on their way at a time, the first of them while the weights are made.  With a head a warp and four splits requested
// together the whole kernel took, us, so now: one head, 141 splits 25.7, 14.4, 157 splits 26.2, 16.3; 4 heads on 4, 40 splits 14.1, 11.7; 16 on 2, 63 splits 20.9,
// 19.9.  Few splits leave a head to its warp (V = 8), which then meets nobody: 8 heads on 8, 8 sequences, four
// splits of 128 12.7, 12.1.
template <int G, int V>   // V: dims of a thread
__device__ __forceinline__ void merge_splits(const AttnParams& p, int b, int kvh, int ns, float2* wl, float* l_s) {
  constexpr int T = kHD / V, U = (G == 1 || (G <= 4 && V == 8) ? 32 : 64) / V;   // threads of a head, splits requested together
  constexpr int kHeads = kW * 32 / T, kPasses = (G + kHeads - 1) / kHeads;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, col = tid % T * V;
  const float* src = nullptr;
  float o[U][V];
  auto request = [&](int s0) {
#pragma unroll
    for (int i = 0; i < U; i++)
      if (s0 + i < ns) {
        const float* at = src + (size_t)(s0 + i) * kHD;
        if constexpr (V >= 4) {
#pragma unroll
          for (int e = 0; e < V; e += 4) *reinterpret_cast<float4*>(o[i] + e) = __ldcg(reinterpret_cast<const float4*>(at + e));
        } else if constexpr (V == 2) {
          *reinterpret_cast<float2*>(o[i]) = __ldcg(reinterpret_cast<const float2*>(at));
        } else {
          o[i][0] = __ldcg(at);
        }
      }
  };
  auto enter = [&](int g) {
    src = p.part_o + ((size_t)b * p.Hq + kvh * G + min(g, G - 1)) * p.max_splits * kHD + col;
    if (g < G) request(0);
  };
  enter(tid / T);
  uint4 gate = make_uint4(0, 0, 0, 0);
  if (warp < G) {
    gate = head_gate(p, b, kvh * G + warp);
    const float2* ml = reinterpret_cast<const float2*>(p.part_ml) + ((size_t)b * p.Hq + kvh * G + warp) * p.max_splits;
    float2* mine = wl + warp * ns;
    float m = -INFINITY;
    for (int s = lane; s < ns; s += 32) {
      const float2 v = __ldcg(ml + s);
      mine[s] = v;
      m = fmaxf(m, v.x);
    }
    const float M = bk_warp_max(m);
    for (int s = lane; s < ns; s += 32) mine[s].x = bk_expf(__fsub_rn(mine[s].x, M));
  }
  if (T > 32) __syncthreads();
  else __syncwarp();
  float L[kPasses], O[kPasses][V];
#pragma unroll
  for (int pass = 0; pass < kPasses; pass++) {
    const int g = pass * kHeads + tid / T;
    if (pass) enter(g);
    L[pass] = 0.0f;
#pragma unroll
    for (int e = 0; e < V; e++) O[pass][e] = 0.0f;
    if (g < G) {
#pragma unroll 1
      for (int s0 = 0; s0 < ns; s0 += U) {
        if (s0) request(s0);
#pragma unroll
        for (int i = 0; i < U; i++)
          if (s0 + i < ns) {
            const float2 w = wl[g * ns + s0 + i];
            L[pass] = fmaf(w.x, w.y, L[pass]);
#pragma unroll
            for (int e = 0; e < V; e++) O[pass][e] = fmaf(w.x, o[i][e], O[pass][e]);
          }
      }
    }
  }
  if constexpr (V == 8) {
    if (warp < G) store_head_warp(p, b, kvh * G + warp, O[0], L[0], gate);
  } else {
    __syncthreads();   // the weights have been read
    float* sums = reinterpret_cast<float*>(wl);
#pragma unroll
    for (int pass = 0; pass < kPasses; pass++) {
      const int g = pass * kHeads + tid / T;
      if (g < G) {
#pragma unroll
        for (int e = 0; e < V; e++) sums[g * kHD + col + e] = O[pass][e];
        if (col == 0) l_s[g] = L[pass];
      }
    }
    __syncthreads();
    if (warp < G) {
      float out[8];
#pragma unroll
      for (int e = 0; e < 8; e++) out[e] = sums[warp * kHD + lane * 8 + e];
      store_head_warp(p, b, kvh * G + warp, out, l_s[warp], gate);
    }
  }
}

// dynamic shared memory layout (bytes):
//   q_st  : 8*256 bf16                 4096
//   k_st  : 256 bf16                    512   (the row this launch appends)
//   v_st  : 256 bf16                    512
//   m_s   : 8 f32 (+8 spare)             64
//   l_s   : kW*8 f32                    256
//   s_s   : split_len * heads (rounded up to a power of two) f32: the score, then p
//   o_s   : kW*8*256 f32              65536   (the rings of rows, then the warps' sums, then the split merge)
// One CTA per (split, KV head, batch).  Every warp streams its K rows and then its V rows through a ring of its own in shared memory,
// 8 or 16 rows of 512 bytes, by asynchronous copies: a lane copies and reads back its own 16 bytes of a row, so nothing has to be
// synchronised until the sums take the ring's place, the copies of the first V rows run under the scores and the softmax, and 16 warps keep 64 or 128 KB on the way.  (Rows in
// registers, three of a warp on their way, 200 instructions per K row and V row: 8 sequences, 32,768 rows, 8 heads per KV head 209 us = 0.39 of
// the copy rate, 6 heads and 4 KV heads 330 us, 4 and 1 90 us.  Now 139, 236 and 62 us; 163 instructions,
// 58 % of the issue slots, and what is waited for are results of the instruction before: FMAs of one chain, shuffles.)  Rows of the
// cache that were written in earlier steps do not depend on the kernel running just before this one, so (p.settled) the first rows are
// requested before the dependency wait.  The CTA that finishes a (batch, KV head) last merges the splits.
// Two CTAs per SM (at most 128 registers): with one CTA of 8 warps an SM cannot hide the latency of the per-row
// shuffle reductions and the stream stalls.
// Prompt columns: every column's K row (head norm + RoPE at its own position, the arithmetic of the decode step) and V
// row go into its sequence's cache before the attention launch, since a later token of the same pass attends to them.
// One warp per (KV head, column).
__global__ void __launch_bounds__(32) attn_append_kernel(const AttnParams p) {
  bk_pdl_trigger();
  __shared__ __align__(16) uint16_t k_st[kHD];
  const int kvh = blockIdx.x, b = blockIdx.y, lane = threadIdx.x;
  bk_pdl_wait();
  const int pos = __ldcg(p.pos + b);
  const int cb = b % p.n_seq;
  uint16_t* Kb = p.k_cache + ((size_t)cb * p.Hkv + kvh) * (size_t)p.max_len * kHD;
  uint16_t* Vb = p.v_cache + ((size_t)cb * p.Hkv + kvh) * (size_t)p.max_len * kHD;
  const float *cr = p.cos_t + (size_t)pos * p.rot_half, *sr = p.sin_t + (size_t)pos * p.rot_half;
  norm_rope_256(*reinterpret_cast<const uint4*>(p.k + ((size_t)b * p.Hkv + kvh) * kHD + lane * 8), *reinterpret_cast<const uint4*>(p.k_norm_w + lane * 8),
                first_angles(cr, p.rot_half), first_angles(sr, p.rot_half), cr, sr, p.rot_half, k_st);
  __syncwarp();
  *reinterpret_cast<uint4*>(Kb + (size_t)pos * kHD + lane * 8) = *reinterpret_cast<const uint4*>(k_st + lane * 8);
  *reinterpret_cast<uint4*>(Vb + (size_t)pos * kHD + lane * 8) =
      *reinterpret_cast<const uint4*>(p.v + ((size_t)b * p.Hkv + kvh) * kHD + lane * 8);
}

constexpr int kRows = 4;      // rows requested together

// kBatches: batches of rows of a warp on their way or in use; MANY: the merge for many splits
template <int G, int kBatches, bool MANY>
__global__ void __launch_bounds__(kW * 32, G == 1 ? 3 : 2) attn_split_kernel(const AttnParams p) {
  static_assert(kRows * kBatches * kHD * 2 <= 8 * kHD * 4, "a warp's ring is its part of o_s");
  constexpr int GP = G <= 1 ? 1 : G <= 2 ? 2 : G <= 4 ? 4 : 8;   // heads, up to a power of two
  bk_pdl_trigger();
  bk_stamp(p.trace, 0);
  extern __shared__ __align__(16) uint8_t smem[];
  uint16_t* q_st = reinterpret_cast<uint16_t*>(smem);
  uint16_t* k_st = q_st + 8 * kHD;
  uint16_t* v_st = k_st + kHD;
  float* m_s = reinterpret_cast<float*>(v_st + kHD);
  float* l_s = m_s + 16;
  float* s_s = l_s + kW * 8;
  float* o_s = reinterpret_cast<float*>(s_s + (size_t)p.split_len * GP);
  __shared__ int s_last;

  const bool splits_first = p.splits_first;
  const int split = splits_first ? blockIdx.x : blockIdx.z, kvh = splits_first ? blockIdx.y : blockIdx.x, b = splits_first ? blockIdx.z : blockIdx.y;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, tid = threadIdx.x;
  const int cb = p.n_seq > 0 ? b % p.n_seq : b;   // whose cache
  uint16_t* Kb = p.k_cache + ((size_t)cb * p.Hkv + kvh) * (size_t)p.max_len * kHD;
  uint16_t* Vb = p.v_cache + ((size_t)cb * p.Hkv + kvh) * (size_t)p.max_len * kHD;
  const int j0 = split * p.split_len;

  // rows of this warp: jj = warp + 8*i, i < nr; its stream is nb batches of K rows, then as many of V rows
  uint4* const ring = reinterpret_cast<uint4*>(o_s + (size_t)warp * 8 * kHD) + lane;   // this lane's 16 bytes of a row: ring[32 * slot]
  const uint16_t* const Kw = Kb + (size_t)(j0 + warp) * kHD + lane * 8;
  const uint16_t* const Vw = Vb + (size_t)(j0 + warp) * kHD + lane * 8;
  int pos = 0, ns = 0, nr = 0, nb = 0, np = 0;   // np: rows that come from the cache
  bool mine = false;                             // row np is the one at pos, which this launch may append
  auto set_pos = [&](int at) {
    pos = at;
    ns = min(pos + 1, j0 + p.split_len) - j0;   // <= 0: nothing to do for this split
    nr = max(0, (ns - warp + 7) >> 3);
    nb = (nr + kRows - 1) / kRows;
    mine = nr > 0 && j0 + warp + 8 * (nr - 1) == pos;
    np = nr - (mine ? 1 : 0);
  };
  auto copy = [&](uint32_t dst, const uint16_t* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
  };
  // request batch q; own: the row at pos comes from shared memory, once it is there
  auto request = [&](int q, bool own) {
    if (q < 2 * nb) {
      const bool is_v = q >= nb;
      const int i = kRows * (is_v ? q - nb : q);
      const uint16_t* src = (is_v ? Vw : Kw) + (uint32_t)i * (8 * kHD);
      uint4* dst = ring + 32 * kRows * (q % kBatches);
      if (i + kRows <= np) {
#pragma unroll
        for (int e = 0; e < kRows; e++) copy(smem_u32(dst) + e * 512, src + e * (8 * kHD));
      } else {
#pragma unroll 1
        for (int e = 0; e < kRows && i + e < nr; e++) {
          if (i + e < np) copy(smem_u32(dst) + e * 512, src + e * (8 * kHD));
          else if (own) dst[32 * e] = *reinterpret_cast<const uint4*>((is_v ? v_st : k_st) + lane * 8);
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  if (p.settled) {
    set_pos(p.pos[b]);
    for (int q = 0; q < kBatches; q++) request(q, false);
  }
  uint4 wrow = make_uint4(0, 0, 0, 0);
  if (p.fused && (warp < G || warp == kW - 1)) wrow = *reinterpret_cast<const uint4*>((warp < G ? p.q_norm_w : p.k_norm_w) + lane * 8);
  bk_pdl_wait();
  bk_stamp(p.trace, 2);
  uint4 xrow = make_uint4(0, 0, 0, 0);   // this warp's query head: it does not wait for the position
  if (warp < G) xrow = *reinterpret_cast<const uint4*>(p.qg + ((size_t)b * p.Hq + kvh * G + warp) * (p.fused ? 2 : 1) * kHD + lane * 8);
  // What the query heads and the new row wait for is requested ahead of the cache's rows, and of those only the first batch: a warp gives out
  // requests no faster than the SM takes them in, so with all four (two CTAs, 128 KB) the heads were ready 2.8 us after the start, with one 1.8.  8
  // sequences, 6 heads, 4 KV heads, 450 rows 14.0 -> 13.5 us, 1,600 rows 22.3 -> 21.3; with two 13.7 and 21.5, with none 13.7 and 21.6.
  float cos0 = 0.0f, sin0 = 0.0f;
  uint4 krow = make_uint4(0, 0, 0, 0), vrow = krow, kw = wrow;
  bool rest = false;   // the batches after the first have not been requested yet
  {
    // The position is taken (again) after the wait: the kernel that advances it may be only a few launches back and
    // still have been running when the early part above read it.  A changed value discards the early loads.
    const int pos_now = __ldcg(p.pos + b);
    if (p.fused && pos_now >= j0 && (warp < G || warp == kW - 1)) {
      cos0 = first_angles(p.cos_t + (size_t)pos_now * p.rot_half, p.rot_half);
      sin0 = first_angles(p.sin_t + (size_t)pos_now * p.rot_half, p.rot_half);
      if (p.n_seq == 0 && warp == kW - 1 && pos_now < j0 + p.split_len) {
        krow = *reinterpret_cast<const uint4*>(p.k + ((size_t)b * p.Hkv + kvh) * kHD + lane * 8);
        vrow = *reinterpret_cast<const uint4*>(p.v + ((size_t)b * p.Hkv + kvh) * kHD + lane * 8);
        if (G == kW) kw = *reinterpret_cast<const uint4*>(p.k_norm_w + lane * 8);
      }
    }
    if (!p.settled || pos_now != pos) {
      asm volatile("cp.async.wait_all;" ::: "memory");
      set_pos(pos_now);
      request(0, false);
      rest = true;
    }
  }
  if (ns <= 0) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    return;
  }
  const int nsplits = (pos + p.split_len) / p.split_len;
  const bool owner = pos >= j0 && pos < j0 + ns;

  // ---- phase 0: q (and, in the split that owns row pos, k/v append) ----
  if (p.fused) {
    const float* cr = p.cos_t + (size_t)pos * p.rot_half;
    const float* sr = p.sin_t + (size_t)pos * p.rot_half;
    if (p.n_seq == 0 && warp == kW - 1 && owner) {
      norm_rope_256(krow, kw, cos0, sin0, cr, sr, p.rot_half, k_st);
      *reinterpret_cast<uint4*>(Kb + (size_t)pos * kHD + lane * 8) = *reinterpret_cast<const uint4*>(k_st + lane * 8);
      *reinterpret_cast<uint4*>(Vb + (size_t)pos * kHD + lane * 8) = vrow;
      *reinterpret_cast<uint4*>(v_st + lane * 8) = vrow;
    }
    if (warp < G) norm_rope_256(xrow, wrow, cos0, sin0, cr, sr, p.rot_half, q_st + warp * kHD);
  } else {
    if (warp < G) *reinterpret_cast<uint4*>(q_st + warp * kHD + lane * 8) = xrow;
  }
  if ((!p.fused || p.n_seq > 0) && warp == kW - 1 && owner) {   // the row is in the cache
    *reinterpret_cast<uint4*>(k_st + lane * 8) = *reinterpret_cast<const uint4*>(Kb + (size_t)pos * kHD + lane * 8);
    *reinterpret_cast<uint4*>(v_st + lane * 8) = *reinterpret_cast<const uint4*>(Vb + (size_t)pos * kHD + lane * 8);
  }
  if (rest)
    for (int q = 1; q < kBatches; q++) request(q, false);
  __syncthreads();   // q and the row at pos are in shared memory
  bk_stamp(p.trace, 3);
  if (mine) {   // left out of the first requests
    const int q = np / kRows, e = np % kRows;
    if (q < kBatches) ring[32 * (kRows * q + e)] = *reinterpret_cast<const uint4*>(k_st + lane * 8);
    if (q + nb < kBatches) ring[32 * (kRows * (q + nb) + e)] = *reinterpret_cast<const uint4*>(v_st + lane * 8);
  }

  // ---- phase 1: scores ----
  {
    // query heads in pairs {q_g[d], q_g+1[d]}: one packed FMA advances the dot products of two heads (each its own
    // chain over d, as before)
    // The 5 levels of the warp's butterfly halve what a lane still holds, the scores of four rows: with heads a power of two in number
    // first a row's heads, then the rows, otherwise the rows first, so that 4 rows of 8 heads take 31 shuffles (one by one 36).  A
    // lane takes what the first levels halve in an order of its own, g ^ hsel or r ^ rsel, so that in each of them it keeps the first half
    // and sends the second.
    constexpr bool kHeadsFirst = G == GP;
    constexpr int kTurn = GP <= 2 && kBatches > 2 ? 2 : 1, R = kRows * kTurn;   // batches, rows scored together: eight where they have few heads (latency, not work)
    constexpr int HB = GP == 8 ? 3 : GP == 4 ? 2 : GP == 2 ? 1 : 0, RB = kTurn + 1, kPlain = 5 - HB - RB;   // levels that halve heads, rows, nothing
    const int hsel = kHeadsFirst ? lane >> (5 - HB) : (lane >> kPlain) & (GP - 1);   // the head and the row whose score this lane ends up with
    const int rsel = kHeadsFirst ? (lane >> kPlain) & (R - 1) : lane >> 3;
    const int swap = kHeadsFirst ? hsel : 0;
    constexpr int GH = (G + 1) / 2;
    float2 qp[GH][8];
#pragma unroll
    for (int g = 0; g < G; g += 2) {
      float q0[8], q1[8];
      bf16x8_to_f32(*reinterpret_cast<const uint4*>(q_st + (g ^ swap) * kHD + lane * 8), q0);
      if (g + 1 < G) bf16x8_to_f32(*reinterpret_cast<const uint4*>(q_st + ((g + 1) ^ swap) * kHD + lane * 8), q1);
#pragma unroll
      for (int d = 0; d < 8; d++) qp[g >> 1][d] = make_float2(q0[d], g + 1 < G ? q1[d] : 0.0f);
    }
#pragma unroll 1
    for (int q = 0; q < nb; q += kTurn) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kBatches - kTurn) : "memory");   // batches q and, of two, q + 1 have landed
      // this lane's part of the dot products of row r ^ rsel (a row past the last is whatever the ring holds: its scores are not stored)
      auto dots = [&](int r, float (&pa)[GP]) {
        float kf[8];
        bf16x8_to_f32(ring[32 * ((kRows * q + (r ^ rsel)) % (kRows * kBatches))], kf);
        float2 a2[GH];
#pragma unroll
        for (int g = 0; g < GH; g++) a2[g] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int d = 0; d < 8; d++)
#pragma unroll
          for (int g = 0; g < GH; g++) a2[g] = bk_fma2(qp[g][d], make_float2(kf[d], kf[d]), a2[g]);
#pragma unroll
        for (int g = 0; g < GP; g++) pa[g] = g / 2 >= GH ? 0.0f : g & 1 ? a2[g / 2 < GH ? g / 2 : 0].y : a2[g / 2 < GH ? g / 2 : 0].x;
      };
      float s1;
      if constexpr (kHeadsFirst) {
        float y[R];
#pragma unroll
        for (int r = 0; r < R; r++) {
          float pa[GP];
          dots(r, pa);
          if constexpr (GP == 8) {
            butterfly_level<8, true>(pa, 16);
            butterfly_level<4, true>(reinterpret_cast<float(&)[4]>(pa), 8);
            butterfly_level<2, true>(reinterpret_cast<float(&)[2]>(pa), 4);
          } else if constexpr (GP == 4) {
            butterfly_level<4, true>(pa, 16);
            butterfly_level<2, true>(reinterpret_cast<float(&)[2]>(pa), 8);
          } else if constexpr (GP == 2) {
            butterfly_level<2, true>(pa, 16);
          }
          y[r] = pa[0];
        }
        if constexpr (kTurn == 2) butterfly_level<8, true>(y, 16 >> HB);
        butterfly_level<4, true>(reinterpret_cast<float(&)[4]>(y), (1 << kPlain) * 2);
        butterfly_level<2, true>(reinterpret_cast<float(&)[2]>(y), 1 << kPlain);
        s1 = y[0];
      } else {
        float lo[GP], hi[GP];   // rows 0, 1 of the lane's order, plus what their partners have of them
        auto two_rows = [&](int r, float (&v)[GP]) {   // rows r and r + 2
          float w[GP];
          dots(r, v);
          dots(r + 2, w);
#pragma unroll
          for (int g = 0; g < G; g++) v[g] = __fadd_rn(v[g], __shfl_xor_sync(0xffffffffu, w[g], 16));
        };
        two_rows(0, lo);
        two_rows(1, hi);
#pragma unroll
        for (int g = 0; g < G; g++) lo[g] = __fadd_rn(lo[g], __shfl_xor_sync(0xffffffffu, hi[g], 8));
        if constexpr (GP == 8) {
          butterfly_level<8, false>(lo, 4);
          butterfly_level<4, false>(reinterpret_cast<float(&)[4]>(lo), 2);
          butterfly_level<2, false>(reinterpret_cast<float(&)[2]>(lo), 1);
        } else {
          butterfly_level<4, false>(lo, 4);
          butterfly_level<2, false>(reinterpret_cast<float(&)[2]>(lo), 2);
        }
        s1 = lo[0];
      }
#pragma unroll
      for (int off = (1 << kPlain) >> 1; off >= 1; off >>= 1) s1 = __fadd_rn(s1, __shfl_xor_sync(0xffffffffu, s1, off));
      const int i = kRows * q + rsel;
      if ((lane & ((1 << kPlain) - 1)) == 0 && i < nr) s_s[(size_t)(warp + 8 * i) * GP + hsel] = __fmul_rn(s1, p.scale);
      request(q + kBatches, true);
      if (kTurn == 2 && q + 1 < nb) request(q + 1 + kBatches, true);   // (else batch q + 1 is the first of the V rows)
    }
  }
  __syncthreads();
  bk_stamp(p.trace, 4);

  // ---- phase 2: exact max per head, p = exp(s - m) in place ----
  {
    constexpr int kStep = kW * 32 / GP;
    const int g = tid & (GP - 1);
    float m = -INFINITY;
    for (int jj = tid / GP; jj < ns; jj += kStep) m = fmaxf(m, s_s[(size_t)jj * GP + g]);
#pragma unroll
    for (int off = GP; off < 32; off <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, off));
    if (lane < GP) l_s[warp * 8 + lane] = m;  // l_s doubles as the cross-warp max buffer
    __syncthreads();
    if (tid < GP) {
      float mm = l_s[tid];
#pragma unroll
      for (int w = 1; w < kW; w++) mm = fmaxf(mm, l_s[w * 8 + tid]);
      m_s[tid] = mm;
    }
    __syncthreads();
    const float mg = m_s[g];
    for (int jj = tid / GP; jj < ns; jj += kStep) s_s[(size_t)jj * GP + g] = g < G ? bk_expf(__fsub_rn(s_s[(size_t)jj * GP + g], mg)) : 0.0f;
  }
  __syncthreads();

  // ---- phase 3: o = sum p * V ----
  {
    float2 acc[G][4];   // dims (2i, 2i+1) side by side: one packed FMA per pair
    float lw = 0.0f;    // of head lane mod GP
#pragma unroll
    for (int g = 0; g < G; g++) {
#pragma unroll
      for (int e = 0; e < 4; e++) acc[g][e] = make_float2(0.0f, 0.0f);
    }
#pragma unroll 1
    for (int q = 0; q < nb; q++) {
      asm volatile("cp.async.wait_group %0;" ::"n"(kBatches - 1) : "memory");   // batch nb + q has landed
      const uint4* rows = ring + 32 * kRows * ((nb + q) % kBatches);
#pragma unroll
      for (int r = 0; r < kRows; r++) {
        const int i = kRows * q + r;
        if (i < nr) {   // warp-uniform
          float vf[8];
          bf16x8_to_f32(rows[32 * r], vf);
          const float* ps = s_s + (size_t)(warp + 8 * i) * GP;
          lw = __fadd_rn(lw, ps[lane & (GP - 1)]);
          float pp[GP];
          if constexpr (GP >= 4) {
#pragma unroll
            for (int g = 0; g < GP; g += 4) *reinterpret_cast<float4*>(pp + g) = *reinterpret_cast<const float4*>(ps + g);
          } else if constexpr (GP == 2) {
            *reinterpret_cast<float2*>(pp) = *reinterpret_cast<const float2*>(ps);
          } else pp[0] = ps[0];
#pragma unroll
          for (int g = 0; g < G; g++)
#pragma unroll
            for (int d = 0; d < 4; d++) acc[g][d] = bk_fma2(make_float2(pp[g], pp[g]), make_float2(vf[2 * d], vf[2 * d + 1]), acc[g][d]);
        }
      }
      request(nb + q + kBatches, true);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();   // a lane's sums go over other lanes' bytes of the ring, which those have read by now
#pragma unroll
    for (int g = 0; g < G; g++) {   // over this warp's ring
      float4* d = reinterpret_cast<float4*>(o_s + ((size_t)(warp * 8 + g)) * kHD + lane * 8);
      d[0] = make_float4(acc[g][0].x, acc[g][0].y, acc[g][1].x, acc[g][1].y);
      d[1] = make_float4(acc[g][2].x, acc[g][2].y, acc[g][3].x, acc[g][3].y);
    }
    if (lane < G) l_s[warp * 8 + lane] = lw;
  }
  __syncthreads();
  bk_stamp(p.trace, 6);

  if (nsplits == 1) {   // nothing to merge with: the partials need not leave the CTA
    if (warp < G) {
      const uint4 gate = head_gate(p, b, kvh * G + warp);
      float L = l_s[warp], O[8];
#pragma unroll
      for (int w = 1; w < kW; w++) L = __fadd_rn(L, l_s[w * 8 + warp]);
#pragma unroll
      for (int e = 0; e < 8; e += 4) {
        float4 o = *reinterpret_cast<const float4*>(o_s + (size_t)warp * kHD + lane * 8 + e);
#pragma unroll
        for (int w = 1; w < kW; w++) {
          const float4 t = *reinterpret_cast<const float4*>(o_s + ((size_t)(w * 8 + warp)) * kHD + lane * 8 + e);
          o = make_float4(__fadd_rn(o.x, t.x), __fadd_rn(o.y, t.y), __fadd_rn(o.z, t.z), __fadd_rn(o.w, t.w));
        }
        O[e] = o.x; O[e + 1] = o.y; O[e + 2] = o.z; O[e + 3] = o.w;
      }
      const float w = bk_expf(__fsub_rn(m_s[warp], m_s[warp]));   // the merge of one split, operation for operation
      L = fmaf(w, L, 0.0f);
#pragma unroll
      for (int e = 0; e < 8; e++) O[e] = fmaf(w, O[e], 0.0f);
      store_head_warp(p, b, kvh * G + warp, O, L, gate);
    }
    bk_stamp(p.trace, 5);
    return;
  }
  // ---- cross-warp sums in warp order, partial out ----
  float *sc_ml = p.part_ml, *sc_o = p.part_o;
  for (int idx = tid; idx < G * kHD; idx += kW * 32) {
    const int g = idx >> 8, d = idx & 255;
    float o = o_s[(size_t)g * kHD + d];
#pragma unroll
    for (int w = 1; w < kW; w++) o = __fadd_rn(o, o_s[((size_t)(w * 8 + g)) * kHD + d]);
    sc_o[(((size_t)b * p.Hq + kvh * G + g) * p.max_splits + split) * kHD + d] = o;
  }
  if (tid < G) {
    float l = l_s[tid];
#pragma unroll
    for (int w = 1; w < kW; w++) l = __fadd_rn(l, l_s[w * 8 + tid]);
    size_t o = (((size_t)b * p.Hq + kvh * G + tid) * p.max_splits + split) * 2;
    sc_ml[o] = m_s[tid];
    sc_ml[o + 1] = l;
  }

  // ---- the CTA that completes this (batch, KV head) merges its splits ----
  __threadfence();
  __syncthreads();
  bk_stamp(p.trace, 7);
  unsigned int* cnt = p.counters + b * p.Hkv + kvh;
  if (tid == 0) {
    const unsigned int done = atomicAdd(cnt, 1u);
    s_last = (done == (unsigned int)(nsplits - 1));
  }
  __syncthreads();
  if (s_last) {
    __threadfence();
    if constexpr (!MANY) {
      if (warp < G) combine_head_warp(p, b, kvh * G + warp, nsplits, o_s + warp * kMaxSplits, head_gate(p, b, kvh * G + warp));
    } else {
      constexpr int V = G <= 2 ? G : G <= 4 || kBatches != 2 ? 4 : 8;
      if (V < 8 && nsplits <= 8) merge_splits<G, 8>(p, b, kvh, nsplits, reinterpret_cast<float2*>(o_s), l_s);
      else merge_splits<G, V>(p, b, kvh, nsplits, reinterpret_cast<float2*>(o_s), l_s);
    }
    if (tid == 0) *cnt = 0;
  }
  bk_stamp(p.trace, 5);
}

size_t attn_smem_bytes(int split_len, int heads) {
  const int gp = heads <= 1 ? 1 : heads <= 2 ? 2 : heads <= 4 ? 4 : 8;
  return 4096 + 1024 + 64 + 256 + (size_t)split_len * gp * 4 + (size_t)kW * 8 * kHD * 4;
}

template <int G, int kBatches, bool MANY>
int32_t launch_split_as(const AttnParams& p, dim3 grid, size_t smem) {
  static size_t configured = 0;
  if (smem > configured) {
    BK_CUDA(cudaFuncSetAttribute(attn_split_kernel<G, kBatches, MANY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    configured = smem;
  }
  BK_CUDA(bk_launch_pdl(attn_split_kernel<G, kBatches, MANY>, grid, dim3(kW * 32), smem, p));
  BK_CHECK_LAUNCH();
  return BK_OK;
}

// Two batches of rows on their way where the splits are short or two CTAs an SM hold all of them, else four.  There more requests bring no more bytes, but
// the query heads come later behind them and some CTAs run far ahead of others (24 heads on 4, four / two batches, us: 8 sequences, 900 rows, 256 splits of 128
// 17.6 / 17.1, 2,000 rows, 256 of 256 25.1 / 24.2, 600 rows, 320 of 64 21.0 / 19.7; but 5 sequences, 9,000 rows, 360 of 512 60.1 / 67.3).
// One or two heads per KV head leave room for three CTAs an SM, which many splits want (16 sequences, 8 heads on 8, 560 rows, 384 splits 18.5 us, two an SM
// 25.4).  What two an SM hold gets two at most, by shared memory that it does not use: three make an uneven spread, since the launch before still holds
// some SMs (6 sequences, 8 heads on 8, 1,100 rows, 288 splits 18.2 us, so 15.2; 16 on 8, 450 rows 16.3, so 13.9).
// The grid walks the splits last: a second wave is then made of last splits, which are short (8 sequences, 24 heads on 4, 320 splits of 64: 600 rows 20.2 us, so
// 19.0, 577 rows 19.3, so 17.4), and prompt columns of a sequence read the same rows at the same time.
// Settled rows (the steps of a model) are requested while the launch before still runs, and of those four batches are better; a single wave of them walks the
// splits first; and a launch of at most eight splits, or of many heads, takes the kernel with the short merge, since code is cold in a step.  24 layers, 8
// sequences, splits of 64, up to five of them: each of the three is worth 4 to 7 us of 1,135 a step; up to 15 of them: the short merge 1,158, the other 1,184.
template <int G, int kBatches>
int32_t launch_split_batches(const AttnParams& p, dim3 grid, size_t smem, int nsplit) {
  return nsplit > 8 && (!p.settled || G <= 4) ? launch_split_as<G, kBatches, true>(p, grid, smem) : launch_split_as<G, kBatches, false>(p, grid, smem);
}
template <int G>
int32_t launch_split(AttnParams& p, int nsplit) {
  const bool two_an_sm = (long long)nsplit * p.Hkv * p.B <= 2 * bk_ctx().sm_count;
  size_t smem = attn_smem_bytes(p.split_len, G);
  if (two_an_sm) smem = std::max<size_t>(smem, bk_ctx().smem_optin / 3);
  p.splits_first = p.settled && two_an_sm;
  const dim3 grid = p.splits_first ? dim3(nsplit, p.Hkv, p.B) : dim3(p.Hkv, p.B, nsplit);
  if (!p.settled && (p.split_len <= 128 || (p.split_len <= 256 && two_an_sm))) return launch_split_batches<G, 2>(p, grid, smem, nsplit);
  return launch_split_batches<G, 4>(p, grid, smem, nsplit);
}

}  // namespace

extern "C" {

int32_t bkAttnPlan(int32_t n_rows, int32_t B, int32_t Hkv, int32_t* split_len, int32_t* warps) {
  BK_REQUIRE_INIT();
  BK_ARG(n_rows > 0 && B > 0 && Hkv > 0 && split_len, "bkAttnPlan: bad arguments");
  // enough splits for about two CTAs per SM, rows per split a multiple of 64 in [64, 512]
  int target = (2 * bk_ctx().sm_count + B * Hkv - 1) / (B * Hkv);
  int len = (n_rows + target - 1) / target;
  len = ((len + 63) / 64) * 64;
  if (len < 64) len = 64;
  if (len > 512) len = 512;
  *split_len = len;
  if (warps) *warps = kW;
  return BK_OK;
}

uint64_t bkAttnScratchBytes(int32_t B, int32_t Hq, int32_t HD, int32_t max_len, int32_t split_len) {
  if (split_len <= 0) return 0;
  uint64_t ms = (uint64_t)(max_len + split_len - 1) / split_len;
  return (uint64_t)B * Hq * ms * (uint64_t)(HD + 2) * 4 + (uint64_t)B * Hq * 4;  // partials + completion counters
}

int32_t bkAttnDecode(const bkAttnArgs* args) {
  BK_REQUIRE_INIT();
  BK_ARG(args != nullptr, "bkAttnDecode: args is null");
  BK_ARG(args->out_q8_layout == BK_Q8_BLOCKS || args->out_q8_layout == BK_Q8_STAGED, "bkAttnDecode: out_q8_layout %d", args->out_q8_layout);
  return bk_attn_launch(*args, 0, 0);
}

}  // extern "C"

// n_seq > 0: the B entries are prompt columns of n_seq sequences (entry b = token b / n_seq of sequence b mod n_seq,
// pos[b] its position): one launch appends every column's K/V row, a second one attends -- the same arithmetic per
// column as B / n_seq decode steps.  layout_B > 0: the scratch buffer was sized for that many entries (launches with
// different B then share one buffer).
int32_t bk_attn_launch(const bkAttnArgs& args, int n_seq, int layout_B) {
  bkAttnArgs a = args;
  BK_ARG(layout_B == 0 || layout_B >= a.B, "attention: scratch laid out for %d entries, %d given", layout_B, a.B);
  BK_ARG(n_seq >= 0 && (n_seq == 0 || (a.B % n_seq == 0 && a.fused_norm_rope)), "attention: %d columns of %d sequences", a.B, n_seq);
  BK_ARG(a.HD == kHD, "bkAttnDecode: head_dim %d unsupported (256 only)", a.HD);
  BK_ARG(a.B > 0 && a.Hq > 0 && a.Hkv > 0 && a.Hq % a.Hkv == 0 && a.Hq / a.Hkv <= 8,
         "bkAttnDecode: bad head counts B=%d Hq=%d Hkv=%d (group size 1..8)", a.B, a.Hq, a.Hkv);
  BK_ARG(a.max_len > 0 && a.max_pos >= 0 && a.max_pos < a.max_len, "bkAttnDecode: max_pos=%d outside cache of %d rows",
         a.max_pos, a.max_len);
  BK_ARG(a.qg && a.k_cache && a.v_cache && a.pos && a.out && a.scratch, "bkAttnDecode: null pointer");
  BK_ARG(((a.qg | a.k_cache | a.v_cache | a.out) & 15) == 0, "bkAttnDecode: pointers must be 16-byte aligned");
  if (a.fused_norm_rope) {
    BK_ARG(a.k && a.v && a.q_norm_w && a.k_norm_w && a.cos_t && a.sin_t, "bkAttnDecode: fused mode needs k, v, norm weights and tables");
    BK_ARG(((a.k | a.v | a.q_norm_w | a.k_norm_w) & 15) == 0, "bkAttnDecode: pointers must be 16-byte aligned");
    BK_ARG(a.rot_half > 0 && 2 * a.rot_half <= kHD, "bkAttnDecode: rot_half=%d", a.rot_half);
  } else {
    BK_ARG(a.gate != 0, "bkAttnDecode: gate is null");
  }
  int split_len = a.split_len;
  if (split_len <= 0) {
    int32_t rc = bkAttnPlan(a.max_pos + 1, a.B, a.Hkv, &split_len, nullptr);
    if (rc) return rc;
  }
  BK_ARG(split_len % 8 == 0 && split_len <= 2048, "bkAttnDecode: split_len=%d must be a multiple of 8, at most 2048", split_len);
  int max_splits = (a.max_len + split_len - 1) / split_len;
  BK_ARG(max_splits <= kMaxSplits, "bkAttnDecode: %d splits exceed the limit of %d", max_splits, kMaxSplits);
  int nsplit = (a.max_pos + split_len) / split_len;
  AttnParams p;
  p.qg = bk_ptr<uint16_t>(a.qg);
  p.k = bk_ptr<uint16_t>(a.k);
  p.v = bk_ptr<uint16_t>(a.v);
  p.q_norm_w = bk_ptr<uint16_t>(a.q_norm_w);
  p.k_norm_w = bk_ptr<uint16_t>(a.k_norm_w);
  p.cos_t = bk_ptr<float>(a.cos_t);
  p.sin_t = bk_ptr<float>(a.sin_t);
  p.k_cache = bk_ptr<uint16_t>(a.k_cache);
  p.v_cache = bk_ptr<uint16_t>(a.v_cache);
  p.pos = bk_ptr<int32_t>(a.pos);
  p.out = bk_ptr<uint16_t>(a.out);
  p.out_q8 = bk_ptr<uint8_t>(a.out_q8);
  p.out_q8_layout = a.out_q8_layout;
  p.gate = bk_ptr<uint16_t>(a.gate);
  p.B = a.B;
  p.Hq = a.Hq;
  p.Hkv = a.Hkv;
  p.rot_half = a.rot_half;
  p.max_len = a.max_len;
  p.split_len = split_len;
  p.max_splits = max_splits;
  p.fused = a.fused_norm_rope;
  p.scale = a.scale;
  p.trace = bk_trace_slot();
  p.settled = n_seq ? 0 : a.cache_is_settled;
  p.n_seq = n_seq;
  {
    // The scratch buffer: the partials of layout_B entries, then the completion counters, which must stay where they are from launch to
    // launch.  The sums are read 16 bytes at a time: they lie behind the pairs (8 bytes each) or, where an odd number of
    // pairs would leave them off the boundary, in front of them.
    const size_t n = (size_t)(layout_B ? layout_B : a.B) * a.Hq * max_splits;
    const bool pairs_first = ((a.scratch + n * 8) & 15) == 0;
    BK_ARG(pairs_first || (a.scratch & 15) == 0, "bkAttnDecode: scratch must be 16-byte aligned");
    float* base = bk_ptr<float>(a.scratch);
    p.part_ml = pairs_first ? base : base + n * kHD;
    p.part_o = pairs_first ? base + n * 2 : base;
    p.counters = reinterpret_cast<unsigned int*>(base + n * (kHD + 2));
  }
  if (n_seq) {
    BK_CUDA(bk_launch_pdl(attn_append_kernel, dim3(a.Hkv, a.B), dim3(32), 0, p));
    BK_CHECK_LAUNCH();
  }
  int32_t rc;
  switch (a.Hq / a.Hkv) {
    case 1: rc = launch_split<1>(p, nsplit); break;
    case 2: rc = launch_split<2>(p, nsplit); break;
    case 3: rc = launch_split<3>(p, nsplit); break;
    case 4: rc = launch_split<4>(p, nsplit); break;
    case 5: rc = launch_split<5>(p, nsplit); break;
    case 6: rc = launch_split<6>(p, nsplit); break;
    case 7: rc = launch_split<7>(p, nsplit); break;
    default: rc = launch_split<8>(p, nsplit); break;
  }
  if (rc) return rc;
  return BK_OK;
}
