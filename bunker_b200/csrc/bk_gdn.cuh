// bk_gdn.cuh -- the fused conv1d + gated-DeltaNet step body (emitConv1d + emitGDN, src/emitters.ts:48-120;
// buildGDNDecode, prototypes/decode.ts:314-388), the per-op kernels of one token (bk_ops.cu).
#pragma once
#include "bk_common.cuh"
#include "bk_internal.h"

namespace {

// ---- fused conv1d + gated DeltaNet step ------------------------------------------
// One CTA of 512 threads per (batch, value head).  Thread (r = t>>7, j = t&127)
// has rows 32r..32r+31 of column j of the 128x128 state, in registers or (more than
// two heads an SM) in shared memory: one read and one write of the state per step.  Column sums over the 128 rows use the four
// row groups in order ((g0+g1)+g2)+g3.
struct GdnParams {
  const uint16_t* qkv;
  const uint16_t* z;
  const float* a;
  const float* b;
  const uint16_t* conv_w;
  const uint16_t* cs_in;
  uint16_t* cs_new;
  const float* A_log;
  const uint16_t* dt_bias;
  const float* norm_w;
  const float* S_in;
  float* S_new;
  uint16_t* out;
  float* o_raw;
  uint16_t* conv_out;
  uint8_t* out_q8;
  int out_q8_layout;
  int B, Hk, Hv, apply_conv;
  int T;      // tokens per sequence (gdn_step_body<kGdnMulti>)
  int early;  // state / conv state / weights are not outputs of the immediately preceding launch
  unsigned long long* trace;
};

// Two builds of this body.  gdn_step_kernel: launched with 576 threads when the grid has at most one CTA per SM; the
// two extra warps only keep a second CTA of this grid off the SM (register file), so no SM finishes last with two.
// gdn_step_kernel_x2: 64 registers, two CTAs per SM, for grids larger than the SM count (batch 8: 256 CTAs, one wave).
// gdn_step_kernel_x3: the state in shared memory instead of registers, three CTAs per SM, for grids of more than one such wave.  Bound: the
// state, 128 KB a head in and out, and while a CTA goes through its chain of norms and sums it neither loads nor stores.  In the step, us, two /
// three CTAs an SM: 13 sequences of 32 heads 17.1 / 13.4, 16 19.8 / 15.3, 32 35.2 / 26.6 (5.1 TB/s), 64 67.5 / 51.9, 8 of 48 heads 14.3 / 11.3.  (Quarter
// heads, eight CTAs of 128 threads an SM and the norm's sums through a cluster: as slow as two whole ones.  One CTA an SM that walks the heads
// behind a ring of copies: 34.5 us for 32 sequences, the chain of a head being 4.9.)
enum { kGdnOne, kGdnMulti, kGdnShared };
constexpr uint32_t kGdnHeadBytes = 128 * 128 * 4;
struct GdnSmem {
  float s_q[128], s_k[128], s_v[128], s_o[128];
  float s_part[4][128];
  float s_scal[4];  // q scale, k rstd, decay, beta
};

// kGdnMulti: a few tokens one after the other (T of them), the state and the three conv taps in registers between them.
// kGdnShared: the state comes by one bulk copy into `state`, and what is read twice of it is scaled by the decay twice.
template <int MODE>
__device__ __forceinline__ void gdn_step_body(const GdnParams& p, GdnSmem& sm, const int hv, const int b, float* state = nullptr, uint64_t* bar = nullptr, int* status = nullptr) {
  constexpr int D = 128;
  constexpr bool MULTI = MODE == kGdnMulti, SHARED = MODE == kGdnShared;
  float (&s_q)[D] = sm.s_q;
  float (&s_k)[D] = sm.s_k;
  float (&s_v)[D] = sm.s_v;
  float (&s_o)[D] = sm.s_o;
  float (&s_part)[4][D] = sm.s_part;
  float (&s_scal)[4] = sm.s_scal;
  bk_pdl_trigger();
  bk_stamp(p.trace, 0);
  const int t = threadIdx.x;
  const int ratio = p.Hv / p.Hk, hk = hv / ratio;
  const int keydim = p.Hk * D, C = 2 * keydim + p.Hv * D;
  const int warp = t >> 5, lane = t & 31;
  const bool active = t < 4 * D;            // threads beyond 512 only occupy registers (see the launch)
  const int r = active ? t >> 7 : 0, j = t & 127;
  const int which = t >> 7, ci = t & 127;
  int ch = 0;
  if (which == 0) ch = hk * D + ci;
  else if (which == 1) ch = keydim + hk * D + ci;
  else ch = 2 * keydim + hv * D + ci;
  const float* S = p.S_in + (((size_t)b * p.Hv + hv) * D + 32 * r) * D + j;
  float* Sn = p.S_new + (((size_t)b * p.Hv + hv) * D + 32 * r) * D + j;

  // State, conv taps and per-head constants do not come from the kernel that runs just before this one
  // (p.early != 0 asserts that), so they are requested before the dependency wait and arrive while the
  // projection GEMV is still finishing.
  float sd[SHARED ? 1 : 32];
  uint16_t h0 = 0, h1 = 0, h2 = 0;
  uint2 cw = make_uint2(0, 0);
  float alog = 0.0f, dtb = 0.0f, nw = 0.0f;
  auto load_static = [&]() {
    if (SHARED) {
      if (t == 0) {
        mbar_expect_tx(smem_u32(bar), kGdnHeadBytes);
        bulk_g2s(smem_u32(state), p.S_in + ((size_t)b * p.Hv + hv) * (D * D), kGdnHeadBytes, smem_u32(bar));
      }
    } else if (active) {
#pragma unroll
      for (int i = 0; i < 32; i++) sd[SHARED ? 0 : i] = S[(size_t)i * D];
    }
    if (t < 3 * D && p.apply_conv) {
      const uint16_t* st = p.cs_in + (size_t)b * 3 * C;
      h0 = st[ch];
      h1 = st[C + ch];
      h2 = st[2 * C + ch];
      cw = *reinterpret_cast<const uint2*>(p.conv_w + 4 * (size_t)ch);
    }
    if (t == 3 * D) {
      alog = p.A_log[hv];
      dtb = bk_bf16_to_f32(p.dt_bias[hv]);
    }
    if (t < D) nw = p.norm_w[t];
  };
  if (p.early) load_static();
  bk_pdl_wait();
  bk_stamp(p.trace, 2);
  if (!p.early) load_static();

  const int T = MULTI ? p.T : 1;   // rows tk*B + b of the per-token inputs and outputs
  for (int tk = 0; tk < T; tk++) {
    const size_t row = (size_t)tk * p.B + b;
    const bool last = !MULTI || tk == T - 1;
    float zv = 0.0f;
    if (t < D) zv = bk_bf16_to_f32(p.z[(row * p.Hv + hv) * D + t]);
    if (t < 3 * D) {
      uint16_t hx = p.qkv[row * C + ch];
      float val;
      if (p.apply_conv) {
        float w0 = __uint_as_float(cw.x << 16), w1 = __uint_as_float(cw.x & 0xffff0000u);
        float w2 = __uint_as_float(cw.y << 16), w3 = __uint_as_float(cw.y & 0xffff0000u);
        float raw = __fadd_rn(__fadd_rn(__fmul_rn(w0, bk_bf16_to_f32(h0)), __fmul_rn(w1, bk_bf16_to_f32(h1))),
                              __fadd_rn(__fmul_rn(w2, bk_bf16_to_f32(h2)), __fmul_rn(w3, bk_bf16_to_f32(hx))));
        uint16_t ob = bk_f32_to_bf16(__fmul_rn(raw, bk_sigmoidf(raw)));
        val = bk_bf16_to_f32(ob);
        // q/k channels are shared by `ratio` value heads: the first of them writes
        if (which == 2 || hv % ratio == 0) {
          if (last) {
            uint16_t* d = p.cs_new + (size_t)b * 3 * C;
            d[ch] = h1;
            d[C + ch] = h2;
            d[2 * C + ch] = hx;
          }
          if (p.conv_out) p.conv_out[row * C + ch] = ob;
        }
        if (MULTI) {
          h0 = h1;
          h1 = h2;
          h2 = hx;
        }
      } else {
        val = bk_bf16_to_f32(hx);
      }
      if (which == 0) s_q[ci] = val;
      else if (which == 1) s_k[ci] = val;
      else s_v[ci] = val;
    } else if (t == 3 * D) {
      // gates on an otherwise idle warp, overlapping the conv above
      float sp = bk_softplusf(__fadd_rn(p.a[row * p.Hv + hv], dtb));
      s_scal[2] = bk_expf(-__fmul_rn(bk_expf(alog), sp));
      s_scal[3] = bk_sigmoidf(p.b[row * p.Hv + hv]);
    }
    __syncthreads();
    if (warp < 2) {
      const float* src = warp == 0 ? s_q : s_k;
      float acc = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; e++) acc = fmaf(src[lane * 4 + e], src[lane * 4 + e], acc);
      acc = bk_warp_sum(acc);
      float rr = bk_rcp_sqrt(__fadd_rn(acc, 1e-6f));
      if (lane == 0) s_scal[warp] = (warp == 0) ? __fmul_rn(rr, 0.088388347648318441f) : rr;
    }
    __syncthreads();
    if (t < D) s_q[t] = __fmul_rn(s_q[t], s_scal[0]);
    else if (t < 2 * D) s_k[t - D] = __fmul_rn(s_k[t - D], s_scal[1]);
    __syncthreads();

    const float decay = s_scal[2], beta = s_scal[3];
    float acc = 0.0f;
    const float* st = state + 32 * r * D + j;
    if constexpr (SHARED) {
      mbar_wait_bounded(smem_u32(bar), 0, status);
#pragma unroll 16
      for (int i = 0; i < 32; i++) acc = fmaf(s_k[32 * r + i], __fmul_rn(st[i * D], decay), acc);
      s_part[r][j] = acc;
    } else if (active) {
#pragma unroll
      for (int i = 0; i < 32; i++) {
        sd[i] = __fmul_rn(sd[i], decay);
        acc = fmaf(s_k[32 * r + i], sd[i], acc);
      }
      s_part[r][j] = acc;
    }
    __syncthreads();
    float kS = __fadd_rn(__fadd_rn(__fadd_rn(s_part[0][j], s_part[1][j]), s_part[2][j]), s_part[3][j]);
    float delta = __fmul_rn(__fsub_rn(s_v[j], kS), beta);
    __syncthreads();
    acc = 0.0f;
    if constexpr (SHARED) {
#pragma unroll 16
      for (int i = 0; i < 32; i++) {
        const float v = fmaf(s_k[32 * r + i], delta, __fmul_rn(st[i * D], decay));
        Sn[(size_t)i * D] = v;
        acc = fmaf(s_q[32 * r + i], v, acc);
      }
      s_part[r][j] = acc;
    } else if (active) {
#pragma unroll
      for (int i = 0; i < 32; i++) {
        sd[i] = fmaf(s_k[32 * r + i], delta, sd[i]);
        if (last) Sn[(size_t)i * D] = sd[i];
        acc = fmaf(s_q[32 * r + i], sd[i], acc);
      }
      s_part[r][j] = acc;
    }
    __syncthreads();
    if (t < D) {
      float o = __fadd_rn(__fadd_rn(__fadd_rn(s_part[0][t], s_part[1][t]), s_part[2][t]), s_part[3][t]);
      s_o[t] = o;
      if (p.o_raw) p.o_raw[(row * p.Hv + hv) * D + t] = o;
    }
    __syncthreads();
    if (warp == 0) {
      float a2 = 0.0f;
#pragma unroll
      for (int e = 0; e < 4; e++) a2 = fmaf(s_o[lane * 4 + e], s_o[lane * 4 + e], a2);
      a2 = bk_warp_sum(a2);
      if (lane == 0) s_scal[0] = bk_rcp_sqrt(__fadd_rn(__fdiv_rn(a2, (float)D), 1e-6f));
    }
    __syncthreads();
    if (t < D) {
      float zs = __fmul_rn(zv, bk_sigmoidf(zv));
      float ow = __fmul_rn(__fmul_rn(s_o[t], s_scal[0]), nw);
      const uint16_t ob = bk_f32_to_bf16(__fmul_rn(ow, zs));
      p.out[(row * p.Hv + hv) * D + t] = ob;
      if (p.out_q8) {  // warp w of the first four holds block w of this head
        const float y[1] = {bk_bf16_to_f32(ob)};
        if (p.out_q8_layout >= BK_Q8_TILE) bk_tile_store<1>(p.out_q8, p.Hv * D, p.B * T, (int)row, hv * 4 + warp, y, lane, p.out_q8_layout == BK_Q8_TILE32);
        else if (p.out_q8_layout == BK_Q8_STAGED) bk_staged_store<1>(p.out_q8, p.Hv * D, p.B * T, (int)row, hv * 4 + warp, y, lane);
        else bk_q8_1_store<1>(p.out_q8 + ((row * p.Hv + hv) * 4 + warp) * 36, y, lane);
      }
    }
    if (!last) __syncthreads();   // s_scal[0] and s_o are rewritten by the next token
  }
  bk_stamp(p.trace, 5);
}

// ---- several tokens per sequence -----------------------------------------------------------
// Only the recurrence itself is serial.  Convolution, norms and gates of all tokens come first (gdn_prepare_kernel, one warp per
// token and head), then the recurrence, four CTAs per value head (32 columns of the state each, in registers for all tokens),
// then the gated norm (gdn_finish_kernel).  Per token the recurrence is two chains of 32 dependent FMAs and two barriers of
// four warps, 0.3 us; as one CTA per head that did everything token after token it took 2.7 us.  64 tokens, 32 value heads: 150 us
// as one launch, 40 us as three (7 + 24 + 5 us of kernels).  The operations and their order are those of gdn_step_body.
struct GdnTokens {
  GdnParams g;
  int T;            // tokens per sequence of this launch
  int t0, t_all;    // its first token, and the tokens of all launches
  int paired;       // (in the padding: of 232 bytes instead of 224, each of the three launches took the host 0.35 us longer)
  float *qn, *kn;   // [T*B][Hk][128] normalised; paired: [(T+1)*B][Hk][128] pairs {q of the token before, k of the token} at kn
  float* v;         // [T*B][Hv][128]
  float2* gates;    // [T*B][Hv] decay, beta
  float* o;         // [T*B][Hv][128]
};
__host__ __device__ inline size_t gdn_row_floats(int Hk, int Hv) { return (size_t)Hk * 256 + (size_t)Hv * 258; }   // (paired: and Hk * 256 once for every sequence)

// four values of a caller's buffer, which need not be aligned to them
__device__ __forceinline__ uint2 gdn_ld4(const uint16_t* p) {
  if ((reinterpret_cast<uintptr_t>(p) & 7) == 0) return *reinterpret_cast<const uint2*>(p);
  return make_uint2((uint32_t)p[0] | (uint32_t)p[1] << 16, (uint32_t)p[2] | (uint32_t)p[3] << 16);
}
__device__ __forceinline__ void gdn_st4(uint16_t* p, uint2 v) {
  if ((reinterpret_cast<uintptr_t>(p) & 7) == 0) {
    *reinterpret_cast<uint2*>(p) = v;
    return;
  }
  p[0] = (uint16_t)v.x;
  p[1] = (uint16_t)(v.x >> 16);
  p[2] = (uint16_t)v.y;
  p[3] = (uint16_t)(v.y >> 16);
}

// one warp per (row, head): heads 0..Hk-1 of q, of k, then the value heads; lane: channels 4 lane .. 4 lane + 3
__global__ void __launch_bounds__(128) gdn_prepare_kernel(const GdnTokens w) {
  bk_pdl_trigger();
  bk_pdl_wait();
  const GdnParams& p = w.g;
  const int lane = threadIdx.x & 31, heads = 2 * p.Hk + p.Hv, C = heads * 128;
  const int item = blockIdx.x * 4 + (threadIdx.x >> 5), row = item / heads, head = item - row * heads;
  if (row >= w.T * p.B) return;
  const int tk = w.t0 + row / p.B, b = row - row / p.B * p.B;
  const int ch = head * 128 + 4 * lane;
  auto taps = [&](int t) {   // the channels' raw values at token t; before token 0 the conv state
    const uint16_t* src = t >= 0 ? p.qkv + ((size_t)t * p.B + b) * C + ch : p.cs_in + ((size_t)b * 3 + t + 3) * C + ch;
    return gdn_ld4(src);
  };
  float x[4];
  const uint2 hx = taps(tk);
  if (p.apply_conv) {
    const uint2 h[3] = {taps(tk - 3), taps(tk - 2), taps(tk - 1)};
    auto at = [](const uint2& v, int e) { return e & 1 ? __uint_as_float((e < 2 ? v.x : v.y) & 0xffff0000u) : __uint_as_float((e < 2 ? v.x : v.y) << 16); };
    uint32_t ob[4];
#pragma unroll
    for (int e = 0; e < 4; e++) {
      const uint2 cw = *reinterpret_cast<const uint2*>(p.conv_w + 4 * (size_t)(ch + e));
      const float w0 = __uint_as_float(cw.x << 16), w1 = __uint_as_float(cw.x & 0xffff0000u);
      const float w2 = __uint_as_float(cw.y << 16), w3 = __uint_as_float(cw.y & 0xffff0000u);
      const float raw = __fadd_rn(__fadd_rn(__fmul_rn(w0, at(h[0], e)), __fmul_rn(w1, at(h[1], e))),
                                  __fadd_rn(__fmul_rn(w2, at(h[2], e)), __fmul_rn(w3, at(hx, e))));
      ob[e] = bk_f32_to_bf16(__fmul_rn(raw, bk_sigmoidf(raw)));
      x[e] = bk_bf16_to_f32((uint16_t)ob[e]);
    }
    if (p.conv_out) gdn_st4(p.conv_out + ((size_t)tk * p.B + b) * C + ch, make_uint2(ob[0] | ob[1] << 16, ob[2] | ob[3] << 16));
    if (tk == w.t_all - 1) {
      uint16_t* d = p.cs_new + (size_t)b * 3 * C + ch;
      gdn_st4(d, h[1]);
      gdn_st4(d + C, h[2]);
      gdn_st4(d + 2 * C, hx);
    }
  } else {
    x[0] = __uint_as_float(hx.x << 16);
    x[1] = __uint_as_float(hx.x & 0xffff0000u);
    x[2] = __uint_as_float(hx.y << 16);
    x[3] = __uint_as_float(hx.y & 0xffff0000u);
  }
  if (head >= 2 * p.Hk) {
    const int hv = head - 2 * p.Hk;
    const size_t o = (size_t)row * p.Hv + hv, in = ((size_t)tk * p.B + b) * p.Hv + hv;
    reinterpret_cast<float4*>(w.v + o * 128)[lane] = make_float4(x[0], x[1], x[2], x[3]);
    if (lane == 0) {
      const float sp = bk_softplusf(__fadd_rn(p.a[in], bk_bf16_to_f32(p.dt_bias[hv])));
      w.gates[o] = make_float2(bk_expf(-__fmul_rn(bk_expf(p.A_log[hv]), sp)), bk_sigmoidf(p.b[in]));
    }
    return;
  }
  float acc = 0.0f;
#pragma unroll
  for (int e = 0; e < 4; e++) acc = fmaf(x[e], x[e], acc);
  float f = bk_rcp_sqrt(__fadd_rn(bk_warp_sum(acc), 1e-6f));
  if (head < p.Hk) f = __fmul_rn(f, 0.088388347648318441f);
  if (w.paired) {
    const bool is_q = head < p.Hk;
    float* dst = w.kn + ((size_t)(row + (is_q ? p.B : 0)) * p.Hk + head - (is_q ? 0 : p.Hk)) * 256 + 8 * lane + (is_q ? 0 : 1);
#pragma unroll
    for (int e = 0; e < 4; e++) dst[2 * e] = __fmul_rn(x[e], f);
    return;
  }
  float* dst = head < p.Hk ? w.qn + ((size_t)row * p.Hk + head) * 128 : w.kn + ((size_t)row * p.Hk + head - p.Hk) * 128;
  reinterpret_cast<float4*>(dst)[lane] = make_float4(__fmul_rn(x[0], f), __fmul_rn(x[1], f), __fmul_rn(x[2], f), __fmul_rn(x[3], f));
}

// CTA (4 hv + quarter, b): warp r has rows 32r..32r+31 of column 32 quarter + lane.  Dynamic shared memory: per token kn and qn
// [256], v of the quarter [32]; then the gates.  The loop has no global load and one barrier a token: the sums over the warps
// of token t's outputs are formed after token t+1's barrier.
__host__ __device__ inline size_t gdn_recur_smem(int T) { return (size_t)T * (256 + 32 + 2) * 4; }
__global__ void __launch_bounds__(128) gdn_recur_kernel(const GdnTokens w) {
  extern __shared__ __align__(16) float gdn_tok[];
  __shared__ float part[2][2][4][32];   // [parity of the token][sum][warp][column]
  bk_pdl_trigger();
  const GdnParams& p = w.g;
  const int t = threadIdx.x, lane = t & 31, r = t >> 5, hv = blockIdx.x >> 2, b = blockIdx.y, hk = hv / (p.Hv / p.Hk), T = w.T;
  const int col = (blockIdx.x & 3) * 32 + lane;
  const size_t so = (((size_t)b * p.Hv + hv) * 128 + 32 * r) * 128 + col;
  float s[32];
  auto load_state = [&]() {
#pragma unroll
    for (int i = 0; i < 32; i++) s[i] = p.S_in[so + (size_t)i * 128];
  };
  if (p.early) load_state();
  bk_pdl_wait();
  if (!p.early) load_state();
  float* kq = gdn_tok;
  float* vs = gdn_tok + T * 256;
  float2* gs = reinterpret_cast<float2*>(vs + T * 32);
  auto copy16 = [](float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  };
  for (int i = t; i < T * 64; i += 128) {
    const int tk = i >> 6, q = i & 63;
    copy16(kq + i * 4, (q < 32 ? w.kn : w.qn) + (((size_t)tk * p.B + b) * p.Hk + hk) * 128 + (q & 31) * 4);
  }
  for (int i = t; i < T * 8; i += 128) copy16(vs + i * 4, w.v + (((size_t)(i >> 3) * p.B + b) * p.Hv + hv) * 128 + (blockIdx.x & 3) * 32 + (i & 7) * 4);
  for (int i = t; i < T; i += 128) gs[i] = __ldcg(w.gates + ((size_t)i * p.B + b) * p.Hv + hv);
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* out = w.o + ((size_t)b * p.Hv + hv) * 128 + col;
  const size_t out_step = (size_t)p.B * p.Hv * 128;
  auto finish = [&](int tk) {   // output of token tk
    if (r == 0) {
      const float(*q)[32] = part[tk & 1][1];
      out[tk * out_step] = __fadd_rn(__fadd_rn(__fadd_rn(q[0][lane], q[1][lane]), q[2][lane]), q[3][lane]);
    }
  };
#pragma unroll 1
  for (int tk = 0; tk < T; tk++) {
    const float4* k4 = reinterpret_cast<const float4*>(kq + tk * 256) + 8 * r;
    const float2 gate = gs[tk];
    const float v = vs[tk * 32 + lane];
    float4 k[8];
#pragma unroll
    for (int i = 0; i < 8; i++) k[i] = k4[i];
    float acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; i++) s[i] = __fmul_rn(s[i], gate.x);
#pragma unroll
    for (int i = 0; i < 8; i++) {
      acc = fmaf(k[i].x, s[4 * i], acc);
      acc = fmaf(k[i].y, s[4 * i + 1], acc);
      acc = fmaf(k[i].z, s[4 * i + 2], acc);
      acc = fmaf(k[i].w, s[4 * i + 3], acc);
    }
    float(*pp)[4][32] = part[tk & 1];
    pp[0][r][lane] = acc;
    __syncthreads();
    const float kS = __fadd_rn(__fadd_rn(__fadd_rn(pp[0][0][lane], pp[0][1][lane]), pp[0][2][lane]), pp[0][3][lane]);
    const float delta = __fmul_rn(__fsub_rn(v, kS), gate.y);
    if (tk > 0) finish(tk - 1);
    acc = 0.0f;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const float4 q = k4[32 + i];
      s[4 * i] = fmaf(k[i].x, delta, s[4 * i]);
      s[4 * i + 1] = fmaf(k[i].y, delta, s[4 * i + 1]);
      s[4 * i + 2] = fmaf(k[i].z, delta, s[4 * i + 2]);
      s[4 * i + 3] = fmaf(k[i].w, delta, s[4 * i + 3]);
      acc = fmaf(q.x, s[4 * i], acc);
      acc = fmaf(q.y, s[4 * i + 1], acc);
      acc = fmaf(q.z, s[4 * i + 2], acc);
      acc = fmaf(q.w, s[4 * i + 3], acc);
    }
    pp[1][r][lane] = acc;
  }
  __syncthreads();
  finish(T - 1);
#pragma unroll
  for (int i = 0; i < 32; i++) p.S_new[so + (size_t)i * 128] = s[i];
}

// The same recurrence where the grid leaves a warp or two to a scheduler and latency is all there is.  A token's output q.S and the next token's
// k.S both read the state that the token leaves, as it is and decayed: the two chains are one chain of packed FMAs, {q, k'} * {S, S g'}, and
// there is one of 32 links a token instead of two.  The pairs {q, k'} come from gdn_prepare_kernel.  In a pass of 64 tokens, 32 value heads 31.8 ->
// 25.0 us, of 17 tokens 14.8 -> 9.0.
__host__ __device__ inline size_t gdn_recur_pair_smem(int T) { return (size_t)(T + 1) * 1024 + (size_t)T * (32 + 2) * 4; }
__global__ void __launch_bounds__(128) gdn_recur_pair_kernel(const GdnTokens w) {
  extern __shared__ __align__(16) float gdn_tok[];
  __shared__ float2 part[2][4][32];   // [parity of the token][warp][column]: output of the token before, k.S of the token
  bk_pdl_trigger();
  const GdnParams& p = w.g;
  const int t = threadIdx.x, lane = t & 31, r = t >> 5, hv = blockIdx.x >> 2, b = blockIdx.y, hk = hv / (p.Hv / p.Hk), T = w.T;
  const int col = (blockIdx.x & 3) * 32 + lane;
  const size_t so = (((size_t)b * p.Hv + hv) * 128 + 32 * r) * 128 + col;
  float2 s[32];   // the state after a token, and that times the next token's decay
  auto load_state = [&]() {
#pragma unroll
    for (int i = 0; i < 32; i++) s[i].y = p.S_in[so + (size_t)i * 128];
  };
  if (p.early) load_state();
  bk_pdl_wait();
  if (!p.early) load_state();
  float* kq = gdn_tok;
  float* vs = gdn_tok + (T + 1) * 256;
  float2* gs = reinterpret_cast<float2*>(vs + T * 32);
  auto copy16 = [](float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
  };
  for (int i = t; i < (T + 1) * 64; i += 128) copy16(kq + i * 4, w.kn + (((size_t)(i >> 6) * p.B + b) * p.Hk + hk) * 256 + (i & 63) * 4);
  for (int i = t; i < T * 8; i += 128) copy16(vs + i * 4, w.v + (((size_t)(i >> 3) * p.B + b) * p.Hv + hv) * 128 + (blockIdx.x & 3) * 32 + (i & 7) * 4);
  for (int i = t; i < T; i += 128) gs[i] = __ldcg(w.gates + ((size_t)i * p.B + b) * p.Hv + hv);
  asm volatile("cp.async.commit_group;" ::: "memory");
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncthreads();
  float* out = w.o + ((size_t)b * p.Hv + hv) * 128 + col;
  const size_t out_step = (size_t)p.B * p.Hv * 128;
  auto pairs = [&](int entry) { return reinterpret_cast<const float4*>(kq + entry * 256) + 16 * r; };   // {q, k, q, k} of two rows each
  float4 u[16], v[16];
#pragma unroll
  for (int i = 0; i < 16; i++) {
    u[i] = pairs(0)[i];
    v[i] = pairs(1)[i];
  }
  float2 gate = gs[0], acc = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int i = 0; i < 32; i++) {
    s[i].y = __fmul_rn(s[i].y, gate.x);
    acc.y = fmaf(i & 1 ? u[i >> 1].w : u[i >> 1].y, s[i].y, acc.y);
  }
  auto sum4 = [](float a, float c, float d, float e) { return __fadd_rn(__fadd_rn(__fadd_rn(a, c), d), e); };
  // token tk: its keys are in `now`, its queries and the next token's keys in `next`.  A warp gets every pair in all its lanes, 64 cycles of the
  // shared memory's return path a token and warp: what comes after `next` is requested along the chain, into what it has used of `now`.
  auto token = [&](int tk, float4 (&now)[16], const float4 (&next)[16]) {
    float2(*pp)[32] = part[tk & 1];
    pp[r][lane] = acc;
    const float4* after = pairs(min(tk + 2, T));
    const float decay = tk + 1 < T ? gs[tk + 1].x : 1.0f, beta = gate.y, vv = vs[tk * 32 + lane];
    if (tk + 1 < T) gate = gs[tk + 1];
    __syncthreads();
    const float2 p0 = pp[0][lane], p1 = pp[1][lane], p2 = pp[2][lane], p3 = pp[3][lane];
    const float delta = __fmul_rn(__fsub_rn(vv, sum4(p0.y, p1.y, p2.y, p3.y)), beta);
    if (tk > 0 && r == (tk & 3)) out[(tk - 1) * out_step] = sum4(p0.x, p1.x, p2.x, p3.x);
    acc = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < 32; i++) {
      s[i].x = fmaf(i & 1 ? now[i >> 1].w : now[i >> 1].y, delta, s[i].y);
      s[i].y = __fmul_rn(s[i].x, decay);
      acc = bk_fma2(i & 1 ? make_float2(next[i >> 1].z, next[i >> 1].w) : make_float2(next[i >> 1].x, next[i >> 1].y), s[i], acc);
      if (i & 1) now[i >> 1] = after[i >> 1];
    }
  };
#pragma unroll 1
  for (int tk = 0; tk < T; tk += 2) {
    token(tk, u, v);
    if (tk + 1 < T) token(tk + 1, v, u);
  }
  part[T & 1][r][lane] = acc;
  __syncthreads();
  if (r == 0) out[(T - 1) * out_step] = sum4(part[T & 1][0][lane].x, part[T & 1][1][lane].x, part[T & 1][2][lane].x, part[T & 1][3][lane].x);
#pragma unroll
  for (int i = 0; i < 32; i++) p.S_new[so + (size_t)i * 128] = s[i].x;
}

// one warp per (row, value head)
__global__ void __launch_bounds__(128) gdn_finish_kernel(const GdnTokens w) {
  bk_pdl_trigger();
  const GdnParams& p = w.g;
  const int lane = threadIdx.x & 31, item = blockIdx.x * 4 + (threadIdx.x >> 5), row = item / p.Hv, hv = item - row * p.Hv;
  bk_pdl_wait();
  if (row >= w.T * p.B) return;
  const size_t orow = (size_t)w.t0 * p.B + row;   // row of the outputs
  const uint2 zz = gdn_ld4(p.z + (orow * p.Hv + hv) * 128 + 4 * lane);
  const float4 o4 = __ldcg(reinterpret_cast<const float4*>(w.o + (size_t)item * 128) + lane);
  const float o[4] = {o4.x, o4.y, o4.z, o4.w}, n[4] = {p.norm_w[4 * lane], p.norm_w[4 * lane + 1], p.norm_w[4 * lane + 2], p.norm_w[4 * lane + 3]};
  const float z[4] = {__uint_as_float(zz.x << 16), __uint_as_float(zz.x & 0xffff0000u), __uint_as_float(zz.y << 16), __uint_as_float(zz.y & 0xffff0000u)};
  if (p.o_raw)
    for (int e = 0; e < 4; e++) p.o_raw[(orow * p.Hv + hv) * 128 + 4 * lane + e] = o[e];
  float a2 = 0.0f;
#pragma unroll
  for (int e = 0; e < 4; e++) a2 = fmaf(o[e], o[e], a2);
  const float rstd = bk_rcp_sqrt(__fadd_rn(__fdiv_rn(bk_warp_sum(a2), 128.0f), 1e-6f));
  uint32_t ob[4];
  float y[4];
#pragma unroll
  for (int e = 0; e < 4; e++) {
    ob[e] = bk_f32_to_bf16(__fmul_rn(__fmul_rn(__fmul_rn(o[e], rstd), n[e]), __fmul_rn(z[e], bk_sigmoidf(z[e]))));
    y[e] = bk_bf16_to_f32((uint16_t)ob[e]);
  }
  gdn_st4(p.out + (orow * p.Hv + hv) * 128 + 4 * lane, make_uint2(ob[0] | ob[1] << 16, ob[2] | ob[3] << 16));
  if (p.out_q8) {   // eight lanes hold one 32-value block
    const int blk = hv * 4 + (lane >> 3), cols = p.B * w.t_all;
    if (p.out_q8_layout >= BK_Q8_TILE) bk_tile_store<4>(p.out_q8, p.Hv * 128, cols, (int)orow, blk, y, (lane & 7) * 4, p.out_q8_layout == BK_Q8_TILE32);
    else if (p.out_q8_layout == BK_Q8_STAGED) bk_staged_store<4>(p.out_q8, p.Hv * 128, cols, (int)orow, blk, y, (lane & 7) * 4);
    else bk_q8_1_store<4>(p.out_q8 + (orow * p.Hv * 4 + blk) * 36, y, (lane & 7) * 4);
  }
}

}  // namespace
