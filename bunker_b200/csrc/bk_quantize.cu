// bk_quantize.cu -- f32 / bf16 weight rows -> Q4_K superblocks on the device: the quantiser behind the weight loader.
//
// bunker uploads its safetensors weights as they are, bf16 (loadWeights, prototypes/decode.ts:64-76); the Q4_K model
// served here needs them quantised once at load time.  Half a warp per 256-weight superblock, lane l of it holding weights
// [16l, 16l+16) (half of sub-block l/2).  The arithmetic is the CPU oracle's, operation for operation:
//   sub-block:  lo = min(min x, 0), scale = (max x - lo) / 15, mn = 0 - lo
//   superblock: d = f16_rn(max scale / 63), dmin = f16_rn(max mn / 63), sc = floor(scale * (1/d) + 0.5) (<= 63),
//               m = floor(mn * (1/dmin) + 0.5) (<= 63)
//   weight:     q = clamp(floor((x + dmin*m) / (d*sc) + 0.5), 0, 15)
// Output layout: bytes [0,2) d, [2,4) dmin, [4,16) the twelve 6-bit scale/min bytes, [16,144) quants, every 32 bytes
// serving sub-blocks 2p (low nibbles) and 2p+1 (high nibbles).
#include "bk_common.cuh"
#include "bk_internal.h"

namespace {

constexpr int kQWarps = 8;   // warps of a CTA, two superblocks each

// floor(t / dl + 0.5) clamped to 0..15, the division and the addition each rounded once.  The quotient is first formed
// with the approximate reciprocal (relative error below 2^-21): unless it lies within kTieBand of a rounding boundary
// the integer is already the exact one.
constexpr float kTieBand = 2e-5f;
BK_DEVINL int quant4_exact(float t, float dl) { return max(0, min(15, (int)floorf(__fadd_rn(__fdiv_rn(t, dl), 0.5f)))); }

BK_DEVINL float2 add2_rd(float2 a, float2 b) {   // rounding down
  unsigned long long ra, rb, rd;
  asm("mov.b64 %0, {%1, %2};" : "=l"(ra) : "f"(a.x), "f"(a.y));
  asm("mov.b64 %0, {%1, %2};" : "=l"(rb) : "f"(b.x), "f"(b.y));
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(rd) : "l"(ra), "l"(rb));
  float2 d;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(rd));
  return d;
}

// 16 lanes per superblock, 16 weights each (half a sub-block): two superblocks per warp share the scalar work, and a
// superblock leaves through shared memory as 16-byte stores.  Issue-bound, the half-rate minima and maxima above all: 17408 x
// 5120 bf16 took 123 us with eight IEEE divisions per thread and byte stores (1.86 TB/s), 78 us with one weight at a time, 73 us with
// two (3.1 TB/s).
template <bool BF16>
__global__ void __launch_bounds__(kQWarps * 32) quantize_q4k_kernel(const void* x, size_t n_superblocks, uint8_t* out) {
  __shared__ __align__(16) uint8_t stage[kQWarps][2 * 144];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, half = lane >> 4, l = lane & 15;
  const size_t first = ((size_t)blockIdx.x * kQWarps + warp) * 2;
  if (first >= n_superblocks) return;   // whole warps leave together
  const size_t sb_idx = min(first + half, n_superblocks - 1);   // a last odd superblock is computed twice and stored once
  float v[16];
  if (BF16) {
    const uint4* src = reinterpret_cast<const uint4*>(reinterpret_cast<const uint16_t*>(x) + sb_idx * 256 + l * 16);
#pragma unroll
    for (int k = 0; k < 2; k++) {
      const uint4 r = __ldcs(src + k);
      v[8 * k + 0] = __uint_as_float(r.x << 16); v[8 * k + 1] = __uint_as_float(r.x & 0xffff0000u);
      v[8 * k + 2] = __uint_as_float(r.y << 16); v[8 * k + 3] = __uint_as_float(r.y & 0xffff0000u);
      v[8 * k + 4] = __uint_as_float(r.z << 16); v[8 * k + 5] = __uint_as_float(r.z & 0xffff0000u);
      v[8 * k + 6] = __uint_as_float(r.w << 16); v[8 * k + 7] = __uint_as_float(r.w & 0xffff0000u);
    }
  } else {
    const float4* src = reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + sb_idx * 256 + l * 16);
#pragma unroll
    for (int k = 0; k < 4; k++) {
      const float4 r = __ldcs(src + k);
      v[4 * k] = r.x; v[4 * k + 1] = r.y; v[4 * k + 2] = r.z; v[4 * k + 3] = r.w;
    }
  }
  float lo = v[0], hi = v[0];
#pragma unroll
  for (int e = 1; e < 16; e++) {
    lo = fminf(lo, v[e]);
    hi = fmaxf(hi, v[e]);
  }
  lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, 1));   // the two lanes of a sub-block
  hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, 1));
  if (lo > 0.0f) lo = 0.0f;
  float scale = __fdiv_rn(__fsub_rn(hi, lo), 15.0f);
  if (!(scale > 0.0f)) scale = 0.0f;
  const float mn = __fsub_rn(0.0f, lo);   // 0 - lo, not -lo: a zero minimum stays +0 (its sign would reach the f16 dmin)
  float max_scale = scale, max_min = mn;
#pragma unroll
  for (int off = 2; off <= 8; off <<= 1) {
    max_scale = fmaxf(max_scale, __shfl_xor_sync(0xffffffffu, max_scale, off));
    max_min = fmaxf(max_min, __shfl_xor_sync(0xffffffffu, max_min, off));
  }
  uint16_t dh, mh;
  asm("cvt.rn.f16.f32 %0, %1;" : "=h"(dh) : "f"(__fdiv_rn(max_scale, 63.0f)));
  asm("cvt.rn.f16.f32 %0, %1;" : "=h"(mh) : "f"(__fdiv_rn(max_min, 63.0f)));
  const float d = bk_f16_to_f32(dh), dm = bk_f16_to_f32(mh);
  const float inv_d = d > 0.0f ? __fdiv_rn(1.0f, d) : 0.0f, inv_dm = dm > 0.0f ? __fdiv_rn(1.0f, dm) : 0.0f;
  const int sc = min(63, (int)floorf(__fadd_rn(__fmul_rn(scale, inv_d), 0.5f)));
  const int m6 = min(63, (int)floorf(__fadd_rn(__fmul_rn(mn, inv_dm), 0.5f)));
  const float dl = __fmul_rn(d, (float)sc), ml = __fmul_rn(dm, (float)m6);
  uint32_t q[4] = {0u, 0u, 0u, 0u};   // sixteen 4-bit quants, one per byte
  if (dl > 0.0f) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(dl));
    // floor without conversions: y + 1.5 * 2^23 rounded down has floor(y) in its low bits, and the clamp to 0..15 is one of floats
    float off_tie = 0.0f;   // largest distance of a fraction from 1/2
    uint32_t t[16];
    const float2 ml2 = make_float2(ml, ml), r2 = make_float2(r, r), half2 = make_float2(0.5f, 0.5f);
#pragma unroll
    for (int e = 0; e < 16; e += 2) {   // two weights per instruction
      const float2 y = bk_fma2(bk_add2(make_float2(v[e], v[e + 1]), ml2), r2, half2);
      const float2 f = add2_rd(y, make_float2(12582912.0f, 12582912.0f));
      const float2 fl = bk_add2(f, make_float2(-12582912.0f, -12582912.0f));
      const float2 o = bk_add2(bk_fma2(fl, make_float2(-1.0f, -1.0f), y), make_float2(-0.5f, -0.5f));
      off_tie = fmaxf(off_tie, fmaxf(fabsf(o.x), fabsf(o.y)));
      t[e] = __float_as_uint(fminf(fmaxf(f.x, 12582912.0f), 12582927.0f));
      t[e + 1] = __float_as_uint(fminf(fmaxf(f.y, 12582912.0f), 12582927.0f));
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
      q[k] = __byte_perm(__byte_perm(t[4 * k], t[4 * k + 1], 0x0040), __byte_perm(t[4 * k + 2], t[4 * k + 3], 0x0040), 0x5410);
    const bool near_tie = off_tie > 0.5f - kTieBand;
    if (near_tie) {
      q[0] = q[1] = q[2] = q[3] = 0u;
#pragma unroll
      for (int e = 0; e < 16; e++) q[e >> 2] |= (uint32_t)quant4_exact(__fadd_rn(v[e], ml), dl) << (8 * (e & 3));
    }
  }
  // quant bytes: lanes 4p, 4p+1 hold sub-block 2p (low nibbles), lanes 4p+2, 4p+3 sub-block 2p+1 (high nibbles) of the
  // same 32 bytes
  uint32_t hn[4];
#pragma unroll
  for (int k = 0; k < 4; k++) hn[k] = __shfl_down_sync(0xffffffffu, q[k], 2);
  uint8_t* sb = stage[warp] + half * 144;
  if ((l & 2) == 0)
    *reinterpret_cast<uint4*>(sb + 16 + (l >> 2) * 32 + (l & 1) * 16) =
        make_uint4(q[0] | (hn[0] << 4), q[1] | (hn[1] << 4), q[2] | (hn[2] << 4), q[3] | (hn[3] << 4));
  // header: sub-block j's scale and min sit in lane 2j; lanes 0..3 assemble bytes j, j+4, j+8 of the twelve
  const int j = (lane & 16) + 2 * (l & 3);
  const int sc_lo = __shfl_sync(0xffffffffu, sc, j), sc_hi = __shfl_sync(0xffffffffu, sc, j + 8);
  const int m_lo = __shfl_sync(0xffffffffu, m6, j), m_hi = __shfl_sync(0xffffffffu, m6, j + 8);
  if (l < 4) {
    sb[4 + l] = (uint8_t)(sc_lo | ((sc_hi >> 4) << 6));
    sb[8 + l] = (uint8_t)(m_lo | ((m_hi >> 4) << 6));
    sb[12 + l] = (uint8_t)((sc_hi & 0x0f) | ((m_hi & 0x0f) << 4));
  }
  if (l == 0) *reinterpret_cast<uint32_t*>(sb) = (uint32_t)dh | ((uint32_t)mh << 16);
  __syncwarp();
  const int n16 = first + 1 < n_superblocks ? 18 : 9;
  if (lane < n16) reinterpret_cast<uint4*>(out + first * 144)[lane] = reinterpret_cast<const uint4*>(stage[warp])[lane];
}

}  // namespace

extern "C" int32_t bkQuantizeQ4K(uint64_t x, int32_t dtype, int64_t n_rows, int32_t K, uint64_t out) {
  BK_REQUIRE_INIT();
  BK_ARG(dtype == BK_DTYPE_F32 || dtype == BK_DTYPE_BF16, "bkQuantizeQ4K: dtype %d (BK_DTYPE_F32 or BK_DTYPE_BF16)", dtype);
  BK_ARG(n_rows > 0 && K > 0 && K % 256 == 0, "bkQuantizeQ4K: bad shape rows=%lld K=%d (K a multiple of 256)", (long long)n_rows, K);
  BK_ARG(x && out && (x & 15) == 0 && (out & 15) == 0, "bkQuantizeQ4K: null or misaligned pointer");
  const size_t nsb = (size_t)n_rows * (K / 256);
  const unsigned grid = (unsigned)((nsb + 2 * kQWarps - 1) / (2 * kQWarps));
  if (dtype == BK_DTYPE_BF16)
    quantize_q4k_kernel<true><<<grid, kQWarps * 32, 0, bk_ctx().stream>>>(bk_ptr<void>(x), nsb, bk_ptr<uint8_t>(out));
  else
    quantize_q4k_kernel<false><<<grid, kQWarps * 32, 0, bk_ctx().stream>>>(bk_ptr<void>(x), nsb, bk_ptr<uint8_t>(out));
  BK_CHECK_LAUNCH();
  return BK_OK;
}
